// generated by gen_plans.py -- do not edit
#include "launch_x.cuh"
namespace dwcu {
void launch_x_18_0(const XArgs &, cudaStream_t);
void launch_x_50_0(const XArgs &, cudaStream_t);
void launch_x_105_0(const XArgs &, cudaStream_t);
void launch_x_180_0(const XArgs &, cudaStream_t);
void launch_x_280_0(const XArgs &, cudaStream_t);
void launch_x_405_0(const XArgs &, cudaStream_t);
void launch_x_576_0(const XArgs &, cudaStream_t);
void launch_x_784_0(const XArgs &, cudaStream_t);
void launch_x_1080_0(const XArgs &, cudaStream_t);
void launch_x_1470_0(const XArgs &, cudaStream_t);
void launch_x_2016_0(const XArgs &, cudaStream_t);
void launch_x_18_0(const XArgs &a, cudaStream_t st) { launch_x_t<Rad<2, 3, 3>, 8, 16>(a, st); }
void launch_x_50_0(const XArgs &a, cudaStream_t st) { launch_x_t<Rad<2, 5, 5>, 16, 8>(a, st); }
void launch_x_105_0(const XArgs &a, cudaStream_t st) { launch_x_t<Rad<5, 3, 7>, 16, 8>(a, st); }
void launch_x_105_1(const XArgs &a, cudaStream_t st) { if (x_iteration_op(a.op)) launch_x_iter_t<Rad<3, 5, 7>, 16, 8>(a, st); else launch_x_105_0(a, st); }
void launch_x_180_0(const XArgs &a, cudaStream_t st) { launch_x_t<Rad<3, 10, 6>, 32, 4>(a, st); }
void launch_x_180_1(const XArgs &a, cudaStream_t st) { if (x_iteration_op(a.op)) launch_x_iter_t<Rad<5, 6, 6>, 32, 4>(a, st); else launch_x_180_0(a, st); }
void launch_x_280_0(const XArgs &a, cudaStream_t st) { launch_x_t<Rad<2, 14, 10>, 32, 4>(a, st); }
void launch_x_280_1(const XArgs &a, cudaStream_t st) { if (x_iteration_op(a.op)) launch_x_iter_t<Rad<7, 4, 10>, 32, 4>(a, st); else launch_x_280_0(a, st); }
void launch_x_405_0(const XArgs &a, cudaStream_t st) { launch_x_t<Rad<5, 9, 9>, 64, 1>(a, st); }
void launch_x_405_1(const XArgs &a, cudaStream_t st) { if (x_iteration_op(a.op)) launch_x_iter_t<Rad<3, 15, 9>, 64, 1>(a, st); else launch_x_405_0(a, st); }
void launch_x_576_0(const XArgs &a, cudaStream_t st) { launch_x_t<Rad<6, 12, 8>, 96, 1>(a, st); }
void launch_x_576_1(const XArgs &a, cudaStream_t st) { if (x_iteration_op(a.op)) launch_x_iter_t<Rad<8, 12, 6>, 96, 1>(a, st); else launch_x_576_0(a, st); }
void launch_x_784_0(const XArgs &a, cudaStream_t st) { launch_x_t<Rad<7, 14, 8>, 128, 1>(a, st); }
void launch_x_784_1(const XArgs &a, cudaStream_t st) { if (x_iteration_op(a.op)) launch_x_iter_t<Rad<8, 14, 7>, 128, 1>(a, st); else launch_x_784_0(a, st); }
void launch_x_1080_0(const XArgs &a, cudaStream_t st) { launch_x_t<Rad<6, 15, 12>, 96, 1>(a, st); }
void launch_x_1080_1(const XArgs &a, cudaStream_t st) { if (x_iteration_op(a.op)) launch_x_iter_t<Rad<8, 15, 9>, 128, 1>(a, st); else launch_x_1080_0(a, st); }
void launch_x_1470_0(const XArgs &a, cudaStream_t st) { launch_x_t<Rad<7, 15, 14>, 128, 1>(a, st); }
void launch_x_1470_1(const XArgs &a, cudaStream_t st) { if (x_iteration_op(a.op)) launch_x_iter_t<Rad<7, 14, 15>, 128, 1>(a, st); else launch_x_1470_0(a, st); }
void launch_x_2016_0(const XArgs &a, cudaStream_t st) { launch_x_t<Rad<9, 16, 14>, 160, 1>(a, st); }
void launch_x_2016_1(const XArgs &a, cudaStream_t st) { if (x_iteration_op(a.op)) launch_x_iter_t<Rad<9, 14, 16>, 160, 1>(a, st); else launch_x_2016_0(a, st); }
}  // namespace dwcu

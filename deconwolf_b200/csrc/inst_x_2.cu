// generated by gen_plans.py -- do not edit
#include "launch_x.cuh"
namespace dwcu {
void launch_x_4_0(const XArgs &, cudaStream_t);
void launch_x_27_0(const XArgs &, cudaStream_t);
void launch_x_64_0(const XArgs &, cudaStream_t);
void launch_x_126_0(const XArgs &, cudaStream_t);
void launch_x_210_0(const XArgs &, cudaStream_t);
void launch_x_320_0(const XArgs &, cudaStream_t);
void launch_x_450_0(const XArgs &, cudaStream_t);
void launch_x_648_0(const XArgs &, cudaStream_t);
void launch_x_882_0(const XArgs &, cudaStream_t);
void launch_x_1176_0(const XArgs &, cudaStream_t);
void launch_x_1575_0(const XArgs &, cudaStream_t);
void launch_x_4_0(const XArgs &a, cudaStream_t st) { launch_x_t<Rad<2, 2, 1>, 4, 32>(a, st); }
void launch_x_27_0(const XArgs &a, cudaStream_t st) { launch_x_t<Rad<3, 9, 1>, 4, 32>(a, st); }
void launch_x_64_0(const XArgs &a, cudaStream_t st) { launch_x_t<Rad<4, 4, 4>, 16, 8>(a, st); }
void launch_x_126_0(const XArgs &a, cudaStream_t st) { launch_x_t<Rad<3, 7, 6>, 32, 4>(a, st); }
void launch_x_126_1(const XArgs &a, cudaStream_t st) { if (x_iteration_op(a.op)) launch_x_iter_t<Rad<3, 6, 7>, 32, 4>(a, st); else launch_x_126_0(a, st); }
void launch_x_210_0(const XArgs &a, cudaStream_t st) { launch_x_t<Rad<3, 10, 7>, 32, 4>(a, st); }
void launch_x_210_1(const XArgs &a, cudaStream_t st) { if (x_iteration_op(a.op)) launch_x_iter_t<Rad<5, 6, 7>, 32, 4>(a, st); else launch_x_210_0(a, st); }
void launch_x_320_0(const XArgs &a, cudaStream_t st) { launch_x_t<Rad<8, 4, 10>, 32, 4>(a, st); }
void launch_x_320_1(const XArgs &a, cudaStream_t st) { if (x_iteration_op(a.op)) launch_x_iter_t<Rad<2, 16, 10>, 32, 4>(a, st); else launch_x_320_0(a, st); }
void launch_x_450_0(const XArgs &a, cudaStream_t st) { launch_x_t<Rad<5, 10, 9>, 64, 1>(a, st); }
void launch_x_450_1(const XArgs &a, cudaStream_t st) { if (x_iteration_op(a.op)) launch_x_iter_t<Rad<6, 15, 5>, 96, 1>(a, st); else launch_x_450_0(a, st); }
void launch_x_648_0(const XArgs &a, cudaStream_t st) { launch_x_t<Rad<6, 12, 9>, 96, 1>(a, st); }
void launch_x_648_1(const XArgs &a, cudaStream_t st) { if (x_iteration_op(a.op)) launch_x_iter_t<Rad<6, 9, 12>, 96, 1>(a, st); else launch_x_648_0(a, st); }
void launch_x_882_0(const XArgs &a, cudaStream_t st) { launch_x_t<Rad<7, 14, 9>, 128, 1>(a, st); }
void launch_x_882_1(const XArgs &a, cudaStream_t st) { if (x_iteration_op(a.op)) launch_x_iter_t<Rad<9, 14, 7>, 128, 1>(a, st); else launch_x_882_0(a, st); }
void launch_x_1176_0(const XArgs &a, cudaStream_t st) { launch_x_t<Rad<7, 14, 12>, 128, 1>(a, st); }
void launch_x_1176_1(const XArgs &a, cudaStream_t st) { if (x_iteration_op(a.op)) launch_x_iter_t<Rad<6, 14, 14>, 128, 1>(a, st); else launch_x_1176_0(a, st); }
void launch_x_1575_0(const XArgs &a, cudaStream_t st) { launch_x_t<Rad<7, 15, 15>, 128, 1>(a, st); }
void launch_x_1575_1(const XArgs &a, cudaStream_t st) { if (x_iteration_op(a.op)) launch_x_iter_t<Rad<15, 15, 7>, 256, 1>(a, st); else launch_x_1575_0(a, st); }
}  // namespace dwcu

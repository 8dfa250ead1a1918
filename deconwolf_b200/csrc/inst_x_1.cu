// generated by gen_plans.py -- do not edit
#include "launch_x.cuh"
namespace dwcu {
void launch_x_3_0(const XArgs &, cudaStream_t);
void launch_x_25_0(const XArgs &, cudaStream_t);
void launch_x_63_0(const XArgs &, cudaStream_t);
void launch_x_125_0(const XArgs &, cudaStream_t);
void launch_x_200_0(const XArgs &, cudaStream_t);
void launch_x_315_0(const XArgs &, cudaStream_t);
void launch_x_448_0(const XArgs &, cudaStream_t);
void launch_x_640_0(const XArgs &, cudaStream_t);
void launch_x_864_0(const XArgs &, cudaStream_t);
void launch_x_1152_0(const XArgs &, cudaStream_t);
void launch_x_1568_0(const XArgs &, cudaStream_t);
void launch_x_3_0(const XArgs &a, cudaStream_t st) { launch_x_t<Rad<3, 1, 1>, 4, 32>(a, st); }
void launch_x_25_0(const XArgs &a, cudaStream_t st) { launch_x_t<Rad<5, 5, 1>, 8, 16>(a, st); }
void launch_x_63_0(const XArgs &a, cudaStream_t st) { launch_x_t<Rad<7, 9, 1>, 8, 16>(a, st); }
void launch_x_125_0(const XArgs &a, cudaStream_t st) { launch_x_t<Rad<5, 5, 5>, 32, 4>(a, st); }
void launch_x_200_0(const XArgs &a, cudaStream_t st) { launch_x_t<Rad<5, 5, 8>, 32, 4>(a, st); }
void launch_x_200_1(const XArgs &a, cudaStream_t st) { if (x_iteration_op(a.op)) launch_x_iter_t<Rad<5, 10, 4>, 32, 4>(a, st); else launch_x_200_0(a, st); }
void launch_x_315_0(const XArgs &a, cudaStream_t st) { launch_x_t<Rad<5, 9, 7>, 64, 1>(a, st); }
void launch_x_315_1(const XArgs &a, cudaStream_t st) { if (x_iteration_op(a.op)) launch_x_iter_t<Rad<7, 9, 5>, 64, 1>(a, st); else launch_x_315_0(a, st); }
void launch_x_448_0(const XArgs &a, cudaStream_t st) { launch_x_t<Rad<4, 14, 8>, 64, 1>(a, st); }
void launch_x_448_1(const XArgs &a, cudaStream_t st) { if (x_iteration_op(a.op)) launch_x_iter_t<Rad<7, 8, 8>, 64, 1>(a, st); else launch_x_448_0(a, st); }
void launch_x_640_0(const XArgs &a, cudaStream_t st) { launch_x_t<Rad<8, 8, 10>, 96, 1>(a, st); }
void launch_x_640_1(const XArgs &a, cudaStream_t st) { if (x_iteration_op(a.op)) launch_x_iter_t<Rad<8, 10, 8>, 96, 1>(a, st); else launch_x_640_0(a, st); }
void launch_x_864_0(const XArgs &a, cudaStream_t st) { launch_x_t<Rad<8, 12, 9>, 96, 1>(a, st); }
void launch_x_864_1(const XArgs &a, cudaStream_t st) { if (x_iteration_op(a.op)) launch_x_iter_t<Rad<6, 16, 9>, 96, 1>(a, st); else launch_x_864_0(a, st); }
void launch_x_1152_0(const XArgs &a, cudaStream_t st) { launch_x_t<Rad<8, 12, 12>, 96, 1>(a, st); }
void launch_x_1152_1(const XArgs &a, cudaStream_t st) { if (x_iteration_op(a.op)) launch_x_iter_t<Rad<6, 16, 12>, 96, 1>(a, st); else launch_x_1152_0(a, st); }
void launch_x_1568_0(const XArgs &a, cudaStream_t st) { launch_x_t<Rad<8, 14, 14>, 128, 1>(a, st); }
void launch_x_1568_1(const XArgs &a, cudaStream_t st) { if (x_iteration_op(a.op)) launch_x_iter_t<Rad<7, 16, 14>, 128, 1>(a, st); else launch_x_1568_0(a, st); }
}  // namespace dwcu

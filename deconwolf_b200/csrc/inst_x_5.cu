// generated by gen_plans.py -- do not edit
#include "launch_x.cuh"
namespace dwcu {
void launch_x_7_0(const XArgs &, cudaStream_t);
void launch_x_32_0(const XArgs &, cudaStream_t);
void launch_x_75_0(const XArgs &, cudaStream_t);
void launch_x_140_0(const XArgs &, cudaStream_t);
void launch_x_225_0(const XArgs &, cudaStream_t);
void launch_x_343_0(const XArgs &, cudaStream_t);
void launch_x_490_0(const XArgs &, cudaStream_t);
void launch_x_686_0(const XArgs &, cudaStream_t);
void launch_x_945_0(const XArgs &, cudaStream_t);
void launch_x_1260_0(const XArgs &, cudaStream_t);
void launch_x_1680_0(const XArgs &, cudaStream_t);
void launch_x_7_0(const XArgs &a, cudaStream_t st) { launch_x_t<Rad<7, 1, 1>, 4, 32>(a, st); }
void launch_x_32_0(const XArgs &a, cudaStream_t st) { launch_x_t<Rad<2, 4, 4>, 8, 16>(a, st); }
void launch_x_75_0(const XArgs &a, cudaStream_t st) { launch_x_t<Rad<3, 5, 5>, 16, 8>(a, st); }
void launch_x_140_0(const XArgs &a, cudaStream_t st) { launch_x_t<Rad<4, 7, 5>, 32, 4>(a, st); }
void launch_x_140_1(const XArgs &a, cudaStream_t st) { if (x_iteration_op(a.op)) launch_x_iter_t<Rad<4, 5, 7>, 32, 4>(a, st); else launch_x_140_0(a, st); }
void launch_x_225_0(const XArgs &a, cudaStream_t st) { launch_x_t<Rad<5, 5, 9>, 32, 4>(a, st); }
void launch_x_225_1(const XArgs &a, cudaStream_t st) { if (x_iteration_op(a.op)) launch_x_iter_t<Rad<5, 9, 5>, 32, 4>(a, st); else launch_x_225_0(a, st); }
void launch_x_343_0(const XArgs &a, cudaStream_t st) { launch_x_t<Rad<7, 7, 7>, 64, 1>(a, st); }
void launch_x_490_0(const XArgs &a, cudaStream_t st) { launch_x_t<Rad<5, 14, 7>, 96, 1>(a, st); }
void launch_x_490_1(const XArgs &a, cudaStream_t st) { if (x_iteration_op(a.op)) launch_x_iter_t<Rad<7, 10, 7>, 96, 1>(a, st); else launch_x_490_0(a, st); }
void launch_x_686_0(const XArgs &a, cudaStream_t st) { launch_x_t<Rad<7, 14, 7>, 128, 1>(a, st); }
void launch_x_686_1(const XArgs &a, cudaStream_t st) { if (x_iteration_op(a.op)) launch_x_iter_t<Rad<7, 7, 14>, 64, 1>(a, st); else launch_x_686_0(a, st); }
void launch_x_945_0(const XArgs &a, cudaStream_t st) { launch_x_t<Rad<7, 15, 9>, 128, 1>(a, st); }
void launch_x_945_1(const XArgs &a, cudaStream_t st) { if (x_iteration_op(a.op)) launch_x_iter_t<Rad<9, 15, 7>, 160, 1>(a, st); else launch_x_945_0(a, st); }
void launch_x_1260_0(const XArgs &a, cudaStream_t st) { launch_x_t<Rad<7, 15, 12>, 128, 1>(a, st); }
void launch_x_1260_1(const XArgs &a, cudaStream_t st) { if (x_iteration_op(a.op)) launch_x_iter_t<Rad<6, 15, 14>, 128, 1>(a, st); else launch_x_1260_0(a, st); }
void launch_x_1680_0(const XArgs &a, cudaStream_t st) { launch_x_t<Rad<8, 15, 14>, 128, 1>(a, st); }
void launch_x_1680_1(const XArgs &a, cudaStream_t st) { if (x_iteration_op(a.op)) launch_x_iter_t<Rad<8, 14, 15>, 128, 1>(a, st); else launch_x_1680_0(a, st); }
}  // namespace dwcu

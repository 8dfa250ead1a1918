// generated by gen_plans.py -- do not edit
#include "launch_x.cuh"
namespace dwcu {
void launch_x_21_0(const XArgs &, cudaStream_t);
void launch_x_56_0(const XArgs &, cudaStream_t);
void launch_x_112_0(const XArgs &, cudaStream_t);
void launch_x_192_0(const XArgs &, cudaStream_t);
void launch_x_294_0(const XArgs &, cudaStream_t);
void launch_x_432_0(const XArgs &, cudaStream_t);
void launch_x_600_0(const XArgs &, cudaStream_t);
void launch_x_810_0(const XArgs &, cudaStream_t);
void launch_x_1125_0(const XArgs &, cudaStream_t);
void launch_x_1512_0(const XArgs &, cudaStream_t);
void launch_x_2048_0(const XArgs &, cudaStream_t);
void launch_x_21_0(const XArgs &a, cudaStream_t st) { launch_x_t<Rad<3, 7, 1>, 4, 32>(a, st); }
void launch_x_56_0(const XArgs &a, cudaStream_t st) { launch_x_t<Rad<2, 4, 7>, 8, 16>(a, st); }
void launch_x_112_0(const XArgs &a, cudaStream_t st) { launch_x_t<Rad<4, 4, 7>, 16, 8>(a, st); }
void launch_x_112_1(const XArgs &a, cudaStream_t st) { if (x_iteration_op(a.op)) launch_x_iter_t<Rad<2, 8, 7>, 16, 8>(a, st); else launch_x_112_0(a, st); }
void launch_x_192_0(const XArgs &a, cudaStream_t st) { launch_x_t<Rad<4, 8, 6>, 32, 4>(a, st); }
void launch_x_192_1(const XArgs &a, cudaStream_t st) { if (x_iteration_op(a.op)) launch_x_iter_t<Rad<4, 6, 8>, 32, 4>(a, st); else launch_x_192_0(a, st); }
void launch_x_294_0(const XArgs &a, cudaStream_t st) { launch_x_t<Rad<6, 7, 7>, 64, 1>(a, st); }
void launch_x_294_1(const XArgs &a, cudaStream_t st) { if (x_iteration_op(a.op)) launch_x_iter_t<Rad<7, 7, 6>, 64, 1>(a, st); else launch_x_294_0(a, st); }
void launch_x_432_0(const XArgs &a, cudaStream_t st) { launch_x_t<Rad<6, 9, 8>, 64, 1>(a, st); }
void launch_x_432_1(const XArgs &a, cudaStream_t st) { if (x_iteration_op(a.op)) launch_x_iter_t<Rad<4, 12, 9>, 64, 1>(a, st); else launch_x_432_0(a, st); }
void launch_x_600_0(const XArgs &a, cudaStream_t st) { launch_x_t<Rad<5, 12, 10>, 64, 1>(a, st); }
void launch_x_600_1(const XArgs &a, cudaStream_t st) { if (x_iteration_op(a.op)) launch_x_iter_t<Rad<6, 10, 10>, 64, 1>(a, st); else launch_x_600_0(a, st); }
void launch_x_810_0(const XArgs &a, cudaStream_t st) { launch_x_t<Rad<6, 15, 9>, 96, 1>(a, st); }
void launch_x_810_1(const XArgs &a, cudaStream_t st) { if (x_iteration_op(a.op)) launch_x_iter_t<Rad<9, 10, 9>, 96, 1>(a, st); else launch_x_810_0(a, st); }
void launch_x_1125_0(const XArgs &a, cudaStream_t st) { launch_x_t<Rad<5, 15, 15>, 128, 1>(a, st); }
void launch_x_1125_1(const XArgs &a, cudaStream_t st) { if (x_iteration_op(a.op)) launch_x_iter_t<Rad<15, 15, 5>, 128, 1>(a, st); else launch_x_1125_0(a, st); }
void launch_x_1512_0(const XArgs &a, cudaStream_t st) { launch_x_t<Rad<9, 14, 12>, 128, 1>(a, st); }
void launch_x_1512_1(const XArgs &a, cudaStream_t st) { if (x_iteration_op(a.op)) launch_x_iter_t<Rad<9, 12, 14>, 128, 1>(a, st); else launch_x_1512_0(a, st); }
void launch_x_2048_0(const XArgs &a, cudaStream_t st) { launch_x_t<Rad<8, 16, 16>, 160, 1>(a, st); }
void launch_x_2048_1(const XArgs &a, cudaStream_t st) { if (x_iteration_op(a.op)) launch_x_iter_t<Rad<16, 16, 8>, 256, 1>(a, st); else launch_x_2048_0(a, st); }
}  // namespace dwcu

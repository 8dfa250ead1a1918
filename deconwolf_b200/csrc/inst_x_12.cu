// generated by gen_plans.py -- do not edit
#include "launch_x.cuh"
namespace dwcu {
void launch_x_16_0(const XArgs &, cudaStream_t);
void launch_x_49_0(const XArgs &, cudaStream_t);
void launch_x_100_0(const XArgs &, cudaStream_t);
void launch_x_175_0(const XArgs &, cudaStream_t);
void launch_x_270_0(const XArgs &, cudaStream_t);
void launch_x_400_0(const XArgs &, cudaStream_t);
void launch_x_567_0(const XArgs &, cudaStream_t);
void launch_x_768_0(const XArgs &, cudaStream_t);
void launch_x_1050_0(const XArgs &, cudaStream_t);
void launch_x_1440_0(const XArgs &, cudaStream_t);
void launch_x_1960_0(const XArgs &, cudaStream_t);
void launch_x_16_0(const XArgs &a, cudaStream_t st) { launch_x_t<Rad<2, 2, 4>, 4, 32>(a, st); }
void launch_x_49_0(const XArgs &a, cudaStream_t st) { launch_x_t<Rad<7, 7, 1>, 8, 16>(a, st); }
void launch_x_100_0(const XArgs &a, cudaStream_t st) { launch_x_t<Rad<4, 5, 5>, 32, 4>(a, st); }
void launch_x_100_1(const XArgs &a, cudaStream_t st) { if (x_iteration_op(a.op)) launch_x_iter_t<Rad<5, 5, 4>, 32, 4>(a, st); else launch_x_100_0(a, st); }
void launch_x_175_0(const XArgs &a, cudaStream_t st) { launch_x_t<Rad<5, 5, 7>, 32, 4>(a, st); }
void launch_x_175_1(const XArgs &a, cudaStream_t st) { if (x_iteration_op(a.op)) launch_x_iter_t<Rad<5, 7, 5>, 32, 4>(a, st); else launch_x_175_0(a, st); }
void launch_x_270_0(const XArgs &a, cudaStream_t st) { launch_x_t<Rad<3, 10, 9>, 32, 4>(a, st); }
void launch_x_270_1(const XArgs &a, cudaStream_t st) { if (x_iteration_op(a.op)) launch_x_iter_t<Rad<5, 6, 9>, 32, 4>(a, st); else launch_x_270_0(a, st); }
void launch_x_400_0(const XArgs &a, cudaStream_t st) { launch_x_t<Rad<5, 10, 8>, 64, 1>(a, st); }
void launch_x_400_1(const XArgs &a, cudaStream_t st) { if (x_iteration_op(a.op)) launch_x_iter_t<Rad<4, 10, 10>, 64, 1>(a, st); else launch_x_400_0(a, st); }
void launch_x_567_0(const XArgs &a, cudaStream_t st) { launch_x_t<Rad<7, 9, 9>, 64, 1>(a, st); }
void launch_x_567_1(const XArgs &a, cudaStream_t st) { if (x_iteration_op(a.op)) launch_x_iter_t<Rad<9, 7, 9>, 96, 1>(a, st); else launch_x_567_0(a, st); }
void launch_x_768_0(const XArgs &a, cudaStream_t st) { launch_x_t<Rad<8, 12, 8>, 96, 1>(a, st); }
void launch_x_768_1(const XArgs &a, cudaStream_t st) { if (x_iteration_op(a.op)) launch_x_iter_t<Rad<6, 16, 8>, 96, 1>(a, st); else launch_x_768_0(a, st); }
void launch_x_1050_0(const XArgs &a, cudaStream_t st) { launch_x_t<Rad<7, 15, 10>, 128, 1>(a, st); }
void launch_x_1050_1(const XArgs &a, cudaStream_t st) { if (x_iteration_op(a.op)) launch_x_iter_t<Rad<10, 15, 7>, 160, 1>(a, st); else launch_x_1050_0(a, st); }
void launch_x_1440_0(const XArgs &a, cudaStream_t st) { launch_x_t<Rad<8, 15, 12>, 128, 1>(a, st); }
void launch_x_1440_1(const XArgs &a, cudaStream_t st) { if (x_iteration_op(a.op)) launch_x_iter_t<Rad<8, 12, 15>, 128, 1>(a, st); else launch_x_1440_0(a, st); }
void launch_x_1960_0(const XArgs &a, cudaStream_t st) { launch_x_t<Rad<10, 14, 14>, 160, 1>(a, st); }
void launch_x_1960_1(const XArgs &a, cudaStream_t st) { if (x_iteration_op(a.op)) launch_x_iter_t<Rad<14, 14, 10>, 256, 1>(a, st); else launch_x_1960_0(a, st); }
}  // namespace dwcu

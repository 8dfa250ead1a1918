// generated by gen_plans.py -- do not edit
#include "launch_x.cuh"
namespace dwcu {
void launch_x_10_0(const XArgs &, cudaStream_t);
void launch_x_40_0(const XArgs &, cudaStream_t);
void launch_x_84_0(const XArgs &, cudaStream_t);
void launch_x_150_0(const XArgs &, cudaStream_t);
void launch_x_245_0(const XArgs &, cudaStream_t);
void launch_x_375_0(const XArgs &, cudaStream_t);
void launch_x_512_0(const XArgs &, cudaStream_t);
void launch_x_729_0(const XArgs &, cudaStream_t);
void launch_x_980_0(const XArgs &, cudaStream_t);
void launch_x_1344_0(const XArgs &, cudaStream_t);
void launch_x_1792_0(const XArgs &, cudaStream_t);
void launch_x_10_0(const XArgs &a, cudaStream_t st) { launch_x_t<Rad<2, 5, 1>, 4, 32>(a, st); }
void launch_x_40_0(const XArgs &a, cudaStream_t st) { launch_x_t<Rad<4, 2, 5>, 8, 16>(a, st); }
void launch_x_84_0(const XArgs &a, cudaStream_t st) { launch_x_t<Rad<2, 7, 6>, 16, 8>(a, st); }
void launch_x_150_0(const XArgs &a, cudaStream_t st) { launch_x_t<Rad<3, 10, 5>, 32, 4>(a, st); }
void launch_x_150_1(const XArgs &a, cudaStream_t st) { if (x_iteration_op(a.op)) launch_x_iter_t<Rad<5, 6, 5>, 32, 4>(a, st); else launch_x_150_0(a, st); }
void launch_x_245_0(const XArgs &a, cudaStream_t st) { launch_x_t<Rad<5, 7, 7>, 64, 1>(a, st); }
void launch_x_245_1(const XArgs &a, cudaStream_t st) { if (x_iteration_op(a.op)) launch_x_iter_t<Rad<7, 7, 5>, 64, 1>(a, st); else launch_x_245_0(a, st); }
void launch_x_375_0(const XArgs &a, cudaStream_t st) { launch_x_t<Rad<5, 15, 5>, 96, 1>(a, st); }
void launch_x_375_1(const XArgs &a, cudaStream_t st) { if (x_iteration_op(a.op)) launch_x_iter_t<Rad<5, 5, 15>, 64, 1>(a, st); else launch_x_375_0(a, st); }
void launch_x_512_0(const XArgs &a, cudaStream_t st) { launch_x_t<Rad<8, 8, 8>, 64, 1>(a, st); }
void launch_x_512_1(const XArgs &a, cudaStream_t st) { if (x_iteration_op(a.op)) launch_x_iter_t<Rad<4, 16, 8>, 64, 1>(a, st); else launch_x_512_0(a, st); }
void launch_x_729_0(const XArgs &a, cudaStream_t st) { launch_x_t<Rad<9, 9, 9>, 96, 1>(a, st); }
void launch_x_980_0(const XArgs &a, cudaStream_t st) { launch_x_t<Rad<7, 14, 10>, 128, 1>(a, st); }
void launch_x_980_1(const XArgs &a, cudaStream_t st) { if (x_iteration_op(a.op)) launch_x_iter_t<Rad<10, 14, 7>, 160, 1>(a, st); else launch_x_980_0(a, st); }
void launch_x_1344_0(const XArgs &a, cudaStream_t st) { launch_x_t<Rad<8, 14, 12>, 128, 1>(a, st); }
void launch_x_1344_1(const XArgs &a, cudaStream_t st) { if (x_iteration_op(a.op)) launch_x_iter_t<Rad<8, 12, 14>, 128, 1>(a, st); else launch_x_1344_0(a, st); }
void launch_x_1792_0(const XArgs &a, cudaStream_t st) { launch_x_t<Rad<8, 16, 14>, 160, 1>(a, st); }
void launch_x_1792_1(const XArgs &a, cudaStream_t st) { if (x_iteration_op(a.op)) launch_x_iter_t<Rad<8, 14, 16>, 128, 1>(a, st); else launch_x_1792_0(a, st); }
}  // namespace dwcu

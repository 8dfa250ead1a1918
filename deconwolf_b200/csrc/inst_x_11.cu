// generated by gen_plans.py -- do not edit
#include "launch_x.cuh"
namespace dwcu {
void launch_x_15_0(const XArgs &, cudaStream_t);
void launch_x_48_0(const XArgs &, cudaStream_t);
void launch_x_98_0(const XArgs &, cudaStream_t);
void launch_x_168_0(const XArgs &, cudaStream_t);
void launch_x_256_0(const XArgs &, cudaStream_t);
void launch_x_392_0(const XArgs &, cudaStream_t);
void launch_x_560_0(const XArgs &, cudaStream_t);
void launch_x_756_0(const XArgs &, cudaStream_t);
void launch_x_1024_0(const XArgs &, cudaStream_t);
void launch_x_1400_0(const XArgs &, cudaStream_t);
void launch_x_1920_0(const XArgs &, cudaStream_t);
void launch_x_15_0(const XArgs &a, cudaStream_t st) { launch_x_t<Rad<3, 5, 1>, 4, 32>(a, st); }
void launch_x_48_0(const XArgs &a, cudaStream_t st) { launch_x_t<Rad<4, 2, 6>, 8, 16>(a, st); }
void launch_x_98_0(const XArgs &a, cudaStream_t st) { launch_x_t<Rad<2, 7, 7>, 16, 8>(a, st); }
void launch_x_98_1(const XArgs &a, cudaStream_t st) { if (x_iteration_op(a.op)) launch_x_iter_t<Rad<7, 2, 7>, 16, 8>(a, st); else launch_x_98_0(a, st); }
void launch_x_168_0(const XArgs &a, cudaStream_t st) { launch_x_t<Rad<4, 7, 6>, 32, 4>(a, st); }
void launch_x_168_1(const XArgs &a, cudaStream_t st) { if (x_iteration_op(a.op)) launch_x_iter_t<Rad<4, 6, 7>, 32, 4>(a, st); else launch_x_168_0(a, st); }
void launch_x_256_0(const XArgs &a, cudaStream_t st) { launch_x_t<Rad<4, 8, 8>, 32, 4>(a, st); }
void launch_x_256_1(const XArgs &a, cudaStream_t st) { if (x_iteration_op(a.op)) launch_x_iter_t<Rad<8, 4, 8>, 32, 4>(a, st); else launch_x_256_0(a, st); }
void launch_x_392_0(const XArgs &a, cudaStream_t st) { launch_x_t<Rad<4, 14, 7>, 64, 1>(a, st); }
void launch_x_392_1(const XArgs &a, cudaStream_t st) { if (x_iteration_op(a.op)) launch_x_iter_t<Rad<7, 8, 7>, 64, 1>(a, st); else launch_x_392_0(a, st); }
void launch_x_560_0(const XArgs &a, cudaStream_t st) { launch_x_t<Rad<4, 14, 10>, 96, 1>(a, st); }
void launch_x_560_1(const XArgs &a, cudaStream_t st) { if (x_iteration_op(a.op)) launch_x_iter_t<Rad<7, 8, 10>, 96, 1>(a, st); else launch_x_560_0(a, st); }
void launch_x_756_0(const XArgs &a, cudaStream_t st) { launch_x_t<Rad<6, 14, 9>, 96, 1>(a, st); }
void launch_x_756_1(const XArgs &a, cudaStream_t st) { if (x_iteration_op(a.op)) launch_x_iter_t<Rad<7, 12, 9>, 96, 1>(a, st); else launch_x_756_0(a, st); }
void launch_x_1024_0(const XArgs &a, cudaStream_t st) { launch_x_t<Rad<8, 16, 8>, 128, 1>(a, st); }
void launch_x_1024_1(const XArgs &a, cudaStream_t st) { if (x_iteration_op(a.op)) launch_x_iter_t<Rad<8, 8, 16>, 128, 1>(a, st); else launch_x_1024_0(a, st); }
void launch_x_1400_0(const XArgs &a, cudaStream_t st) { launch_x_t<Rad<10, 14, 10>, 160, 1>(a, st); }
void launch_x_1400_1(const XArgs &a, cudaStream_t st) { if (x_iteration_op(a.op)) launch_x_iter_t<Rad<10, 10, 14>, 160, 1>(a, st); else launch_x_1400_0(a, st); }
void launch_x_1920_0(const XArgs &a, cudaStream_t st) { launch_x_t<Rad<8, 16, 15>, 160, 1>(a, st); }
void launch_x_1920_1(const XArgs &a, cudaStream_t st) { if (x_iteration_op(a.op)) launch_x_iter_t<Rad<10, 16, 12>, 160, 1>(a, st); else launch_x_1920_0(a, st); }
}  // namespace dwcu

// generated by gen_plans.py -- do not edit
#include "launch_x.cuh"
namespace dwcu {
void launch_x_5_0(const XArgs &, cudaStream_t);
void launch_x_28_0(const XArgs &, cudaStream_t);
void launch_x_70_0(const XArgs &, cudaStream_t);
void launch_x_128_0(const XArgs &, cudaStream_t);
void launch_x_216_0(const XArgs &, cudaStream_t);
void launch_x_324_0(const XArgs &, cudaStream_t);
void launch_x_480_0(const XArgs &, cudaStream_t);
void launch_x_672_0(const XArgs &, cudaStream_t);
void launch_x_896_0(const XArgs &, cudaStream_t);
void launch_x_1200_0(const XArgs &, cudaStream_t);
void launch_x_1600_0(const XArgs &, cudaStream_t);
void launch_x_5_0(const XArgs &a, cudaStream_t st) { launch_x_t<Rad<5, 1, 1>, 4, 32>(a, st); }
void launch_x_28_0(const XArgs &a, cudaStream_t st) { launch_x_t<Rad<4, 7, 1>, 4, 32>(a, st); }
void launch_x_70_0(const XArgs &a, cudaStream_t st) { launch_x_t<Rad<2, 7, 5>, 16, 8>(a, st); }
void launch_x_128_0(const XArgs &a, cudaStream_t st) { launch_x_t<Rad<4, 4, 8>, 16, 8>(a, st); }
void launch_x_128_1(const XArgs &a, cudaStream_t st) { if (x_iteration_op(a.op)) launch_x_iter_t<Rad<2, 8, 8>, 16, 8>(a, st); else launch_x_128_0(a, st); }
void launch_x_216_0(const XArgs &a, cudaStream_t st) { launch_x_t<Rad<3, 9, 8>, 32, 4>(a, st); }
void launch_x_216_1(const XArgs &a, cudaStream_t st) { if (x_iteration_op(a.op)) launch_x_iter_t<Rad<4, 6, 9>, 32, 4>(a, st); else launch_x_216_0(a, st); }
void launch_x_324_0(const XArgs &a, cudaStream_t st) { launch_x_t<Rad<6, 9, 6>, 64, 1>(a, st); }
void launch_x_324_1(const XArgs &a, cudaStream_t st) { if (x_iteration_op(a.op)) launch_x_iter_t<Rad<3, 12, 9>, 64, 1>(a, st); else launch_x_324_0(a, st); }
void launch_x_480_0(const XArgs &a, cudaStream_t st) { launch_x_t<Rad<4, 15, 8>, 64, 1>(a, st); }
void launch_x_480_1(const XArgs &a, cudaStream_t st) { if (x_iteration_op(a.op)) launch_x_iter_t<Rad<5, 12, 8>, 64, 1>(a, st); else launch_x_480_0(a, st); }
void launch_x_672_0(const XArgs &a, cudaStream_t st) { launch_x_t<Rad<6, 14, 8>, 96, 1>(a, st); }
void launch_x_672_1(const XArgs &a, cudaStream_t st) { if (x_iteration_op(a.op)) launch_x_iter_t<Rad<7, 12, 8>, 96, 1>(a, st); else launch_x_672_0(a, st); }
void launch_x_896_0(const XArgs &a, cudaStream_t st) { launch_x_t<Rad<8, 16, 7>, 128, 1>(a, st); }
void launch_x_896_1(const XArgs &a, cudaStream_t st) { if (x_iteration_op(a.op)) launch_x_iter_t<Rad<8, 14, 8>, 128, 1>(a, st); else launch_x_896_0(a, st); }
void launch_x_1200_0(const XArgs &a, cudaStream_t st) { launch_x_t<Rad<8, 15, 10>, 128, 1>(a, st); }
void launch_x_1200_1(const XArgs &a, cudaStream_t st) { if (x_iteration_op(a.op)) launch_x_iter_t<Rad<10, 12, 10>, 128, 1>(a, st); else launch_x_1200_0(a, st); }
void launch_x_1600_0(const XArgs &a, cudaStream_t st) { launch_x_t<Rad<10, 16, 10>, 160, 1>(a, st); }
void launch_x_1600_1(const XArgs &a, cudaStream_t st) { if (x_iteration_op(a.op)) launch_x_iter_t<Rad<10, 10, 16>, 160, 1>(a, st); else launch_x_1600_0(a, st); }
}  // namespace dwcu

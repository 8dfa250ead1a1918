// generated by gen_plans.py -- do not edit
#include "launch_x.cuh"
namespace dwcu {
void launch_x_20_0(const XArgs &, cudaStream_t);
void launch_x_54_0(const XArgs &, cudaStream_t);
void launch_x_108_0(const XArgs &, cudaStream_t);
void launch_x_189_0(const XArgs &, cudaStream_t);
void launch_x_288_0(const XArgs &, cudaStream_t);
void launch_x_420_0(const XArgs &, cudaStream_t);
void launch_x_588_0(const XArgs &, cudaStream_t);
void launch_x_800_0(const XArgs &, cudaStream_t);
void launch_x_1120_0(const XArgs &, cudaStream_t);
void launch_x_1500_0(const XArgs &, cudaStream_t);
void launch_x_2025_0(const XArgs &, cudaStream_t);
void launch_x_20_0(const XArgs &a, cudaStream_t st) { launch_x_t<Rad<4, 5, 1>, 4, 32>(a, st); }
void launch_x_54_0(const XArgs &a, cudaStream_t st) { launch_x_t<Rad<6, 9, 1>, 8, 16>(a, st); }
void launch_x_108_0(const XArgs &a, cudaStream_t st) { launch_x_t<Rad<4, 3, 9>, 16, 8>(a, st); }
void launch_x_108_1(const XArgs &a, cudaStream_t st) { if (x_iteration_op(a.op)) launch_x_iter_t<Rad<3, 4, 9>, 16, 8>(a, st); else launch_x_108_0(a, st); }
void launch_x_189_0(const XArgs &a, cudaStream_t st) { launch_x_t<Rad<3, 9, 7>, 32, 4>(a, st); }
void launch_x_189_1(const XArgs &a, cudaStream_t st) { if (x_iteration_op(a.op)) launch_x_iter_t<Rad<3, 7, 9>, 32, 4>(a, st); else launch_x_189_0(a, st); }
void launch_x_288_0(const XArgs &a, cudaStream_t st) { launch_x_t<Rad<4, 12, 6>, 64, 1>(a, st); }
void launch_x_288_1(const XArgs &a, cudaStream_t st) { if (x_iteration_op(a.op)) launch_x_iter_t<Rad<4, 8, 9>, 64, 1>(a, st); else launch_x_288_0(a, st); }
void launch_x_420_0(const XArgs &a, cudaStream_t st) { launch_x_t<Rad<4, 15, 7>, 64, 1>(a, st); }
void launch_x_420_1(const XArgs &a, cudaStream_t st) { if (x_iteration_op(a.op)) launch_x_iter_t<Rad<5, 12, 7>, 64, 1>(a, st); else launch_x_420_0(a, st); }
void launch_x_588_0(const XArgs &a, cudaStream_t st) { launch_x_t<Rad<6, 14, 7>, 96, 1>(a, st); }
void launch_x_588_1(const XArgs &a, cudaStream_t st) { if (x_iteration_op(a.op)) launch_x_iter_t<Rad<7, 12, 7>, 96, 1>(a, st); else launch_x_588_0(a, st); }
void launch_x_800_0(const XArgs &a, cudaStream_t st) { launch_x_t<Rad<8, 10, 10>, 96, 1>(a, st); }
void launch_x_800_1(const XArgs &a, cudaStream_t st) { if (x_iteration_op(a.op)) launch_x_iter_t<Rad<5, 16, 10>, 96, 1>(a, st); else launch_x_800_0(a, st); }
void launch_x_1120_0(const XArgs &a, cudaStream_t st) { launch_x_t<Rad<8, 14, 10>, 128, 1>(a, st); }
void launch_x_1120_1(const XArgs &a, cudaStream_t st) { if (x_iteration_op(a.op)) launch_x_iter_t<Rad<7, 16, 10>, 128, 1>(a, st); else launch_x_1120_0(a, st); }
void launch_x_1500_0(const XArgs &a, cudaStream_t st) { launch_x_t<Rad<10, 15, 10>, 160, 1>(a, st); }
void launch_x_1500_1(const XArgs &a, cudaStream_t st) { if (x_iteration_op(a.op)) launch_x_iter_t<Rad<10, 10, 15>, 160, 1>(a, st); else launch_x_1500_0(a, st); }
void launch_x_2025_0(const XArgs &a, cudaStream_t st) { launch_x_t<Rad<9, 15, 15>, 160, 1>(a, st); }
void launch_x_2025_1(const XArgs &a, cudaStream_t st) { if (x_iteration_op(a.op)) launch_x_iter_t<Rad<15, 15, 9>, 256, 1>(a, st); else launch_x_2025_0(a, st); }
}  // namespace dwcu

// generated by gen_plans.py -- do not edit
#include "launch_x.cuh"
namespace dwcu {
void launch_x_12_0(const XArgs &, cudaStream_t);
void launch_x_42_0(const XArgs &, cudaStream_t);
void launch_x_90_0(const XArgs &, cudaStream_t);
void launch_x_160_0(const XArgs &, cudaStream_t);
void launch_x_250_0(const XArgs &, cudaStream_t);
void launch_x_378_0(const XArgs &, cudaStream_t);
void launch_x_525_0(const XArgs &, cudaStream_t);
void launch_x_735_0(const XArgs &, cudaStream_t);
void launch_x_1000_0(const XArgs &, cudaStream_t);
void launch_x_1350_0(const XArgs &, cudaStream_t);
void launch_x_1800_0(const XArgs &, cudaStream_t);
void launch_x_12_0(const XArgs &a, cudaStream_t st) { launch_x_t<Rad<2, 2, 3>, 4, 32>(a, st); }
void launch_x_42_0(const XArgs &a, cudaStream_t st) { launch_x_t<Rad<3, 2, 7>, 8, 16>(a, st); }
void launch_x_90_0(const XArgs &a, cudaStream_t st) { launch_x_t<Rad<3, 5, 6>, 16, 8>(a, st); }
void launch_x_160_0(const XArgs &a, cudaStream_t st) { launch_x_t<Rad<4, 8, 5>, 32, 4>(a, st); }
void launch_x_160_1(const XArgs &a, cudaStream_t st) { if (x_iteration_op(a.op)) launch_x_iter_t<Rad<4, 5, 8>, 32, 4>(a, st); else launch_x_160_0(a, st); }
void launch_x_250_0(const XArgs &a, cudaStream_t st) { launch_x_t<Rad<5, 10, 5>, 64, 1>(a, st); }
void launch_x_250_1(const XArgs &a, cudaStream_t st) { if (x_iteration_op(a.op)) launch_x_iter_t<Rad<5, 5, 10>, 64, 1>(a, st); else launch_x_250_0(a, st); }
void launch_x_378_0(const XArgs &a, cudaStream_t st) { launch_x_t<Rad<6, 9, 7>, 64, 1>(a, st); }
void launch_x_378_1(const XArgs &a, cudaStream_t st) { if (x_iteration_op(a.op)) launch_x_iter_t<Rad<7, 9, 6>, 64, 1>(a, st); else launch_x_378_0(a, st); }
void launch_x_525_0(const XArgs &a, cudaStream_t st) { launch_x_t<Rad<5, 15, 7>, 96, 1>(a, st); }
void launch_x_525_1(const XArgs &a, cudaStream_t st) { if (x_iteration_op(a.op)) launch_x_iter_t<Rad<7, 15, 5>, 128, 1>(a, st); else launch_x_525_0(a, st); }
void launch_x_735_0(const XArgs &a, cudaStream_t st) { launch_x_t<Rad<7, 15, 7>, 128, 1>(a, st); }
void launch_x_735_1(const XArgs &a, cudaStream_t st) { if (x_iteration_op(a.op)) launch_x_iter_t<Rad<7, 7, 15>, 64, 1>(a, st); else launch_x_735_0(a, st); }
void launch_x_1000_0(const XArgs &a, cudaStream_t st) { launch_x_t<Rad<10, 10, 10>, 128, 1>(a, st); }
void launch_x_1350_0(const XArgs &a, cudaStream_t st) { launch_x_t<Rad<6, 15, 15>, 128, 1>(a, st); }
void launch_x_1350_1(const XArgs &a, cudaStream_t st) { if (x_iteration_op(a.op)) launch_x_iter_t<Rad<9, 15, 10>, 160, 1>(a, st); else launch_x_1350_0(a, st); }
void launch_x_1800_0(const XArgs &a, cudaStream_t st) { launch_x_t<Rad<8, 15, 15>, 160, 1>(a, st); }
void launch_x_1800_1(const XArgs &a, cudaStream_t st) { if (x_iteration_op(a.op)) launch_x_iter_t<Rad<10, 15, 12>, 160, 1>(a, st); else launch_x_1800_0(a, st); }
}  // namespace dwcu

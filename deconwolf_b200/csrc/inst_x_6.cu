// generated by gen_plans.py -- do not edit
#include "launch_x.cuh"
namespace dwcu {
void launch_x_8_0(const XArgs &, cudaStream_t);
void launch_x_35_0(const XArgs &, cudaStream_t);
void launch_x_80_0(const XArgs &, cudaStream_t);
void launch_x_144_0(const XArgs &, cudaStream_t);
void launch_x_240_0(const XArgs &, cudaStream_t);
void launch_x_350_0(const XArgs &, cudaStream_t);
void launch_x_500_0(const XArgs &, cudaStream_t);
void launch_x_700_0(const XArgs &, cudaStream_t);
void launch_x_960_0(const XArgs &, cudaStream_t);
void launch_x_1280_0(const XArgs &, cudaStream_t);
void launch_x_1728_0(const XArgs &, cudaStream_t);
void launch_x_8_0(const XArgs &a, cudaStream_t st) { launch_x_t<Rad<2, 2, 2>, 4, 32>(a, st); }
void launch_x_35_0(const XArgs &a, cudaStream_t st) { launch_x_t<Rad<5, 7, 1>, 8, 16>(a, st); }
void launch_x_80_0(const XArgs &a, cudaStream_t st) { launch_x_t<Rad<4, 4, 5>, 16, 8>(a, st); }
void launch_x_144_0(const XArgs &a, cudaStream_t st) { launch_x_t<Rad<4, 6, 6>, 32, 4>(a, st); }
void launch_x_144_1(const XArgs &a, cudaStream_t st) { if (x_iteration_op(a.op)) launch_x_iter_t<Rad<3, 8, 6>, 32, 4>(a, st); else launch_x_144_0(a, st); }
void launch_x_240_0(const XArgs &a, cudaStream_t st) { launch_x_t<Rad<3, 10, 8>, 32, 4>(a, st); }
void launch_x_240_1(const XArgs &a, cudaStream_t st) { if (x_iteration_op(a.op)) launch_x_iter_t<Rad<5, 6, 8>, 32, 4>(a, st); else launch_x_240_0(a, st); }
void launch_x_350_0(const XArgs &a, cudaStream_t st) { launch_x_t<Rad<5, 10, 7>, 64, 1>(a, st); }
void launch_x_350_1(const XArgs &a, cudaStream_t st) { if (x_iteration_op(a.op)) launch_x_iter_t<Rad<5, 14, 5>, 96, 1>(a, st); else launch_x_350_0(a, st); }
void launch_x_500_0(const XArgs &a, cudaStream_t st) { launch_x_t<Rad<5, 10, 10>, 64, 1>(a, st); }
void launch_x_500_1(const XArgs &a, cudaStream_t st) { if (x_iteration_op(a.op)) launch_x_iter_t<Rad<10, 5, 10>, 64, 1>(a, st); else launch_x_500_0(a, st); }
void launch_x_700_0(const XArgs &a, cudaStream_t st) { launch_x_t<Rad<5, 14, 10>, 96, 1>(a, st); }
void launch_x_700_1(const XArgs &a, cudaStream_t st) { if (x_iteration_op(a.op)) launch_x_iter_t<Rad<7, 10, 10>, 96, 1>(a, st); else launch_x_700_0(a, st); }
void launch_x_960_0(const XArgs &a, cudaStream_t st) { launch_x_t<Rad<8, 12, 10>, 96, 1>(a, st); }
void launch_x_960_1(const XArgs &a, cudaStream_t st) { if (x_iteration_op(a.op)) launch_x_iter_t<Rad<6, 16, 10>, 96, 1>(a, st); else launch_x_960_0(a, st); }
void launch_x_1280_0(const XArgs &a, cudaStream_t st) { launch_x_t<Rad<8, 16, 10>, 128, 1>(a, st); }
void launch_x_1280_1(const XArgs &a, cudaStream_t st) { if (x_iteration_op(a.op)) launch_x_iter_t<Rad<10, 16, 8>, 160, 1>(a, st); else launch_x_1280_0(a, st); }
void launch_x_1728_0(const XArgs &a, cudaStream_t st) { launch_x_t<Rad<9, 16, 12>, 160, 1>(a, st); }
void launch_x_1728_1(const XArgs &a, cudaStream_t st) { if (x_iteration_op(a.op)) launch_x_iter_t<Rad<9, 12, 16>, 160, 1>(a, st); else launch_x_1728_0(a, st); }
}  // namespace dwcu

// generated by gen_plans.py -- do not edit
#include "launch_x.cuh"
namespace dwcu {
void launch_x_6_0(const XArgs &, cudaStream_t);
void launch_x_30_0(const XArgs &, cudaStream_t);
void launch_x_72_0(const XArgs &, cudaStream_t);
void launch_x_135_0(const XArgs &, cudaStream_t);
void launch_x_224_0(const XArgs &, cudaStream_t);
void launch_x_336_0(const XArgs &, cudaStream_t);
void launch_x_486_0(const XArgs &, cudaStream_t);
void launch_x_675_0(const XArgs &, cudaStream_t);
void launch_x_900_0(const XArgs &, cudaStream_t);
void launch_x_1215_0(const XArgs &, cudaStream_t);
void launch_x_1620_0(const XArgs &, cudaStream_t);
void launch_x_6_0(const XArgs &a, cudaStream_t st) { launch_x_t<Rad<3, 2, 1>, 4, 32>(a, st); }
void launch_x_30_0(const XArgs &a, cudaStream_t st) { launch_x_t<Rad<3, 5, 2>, 8, 16>(a, st); }
void launch_x_72_0(const XArgs &a, cudaStream_t st) { launch_x_t<Rad<3, 4, 6>, 16, 8>(a, st); }
void launch_x_135_0(const XArgs &a, cudaStream_t st) { launch_x_t<Rad<5, 3, 9>, 16, 8>(a, st); }
void launch_x_135_1(const XArgs &a, cudaStream_t st) { if (x_iteration_op(a.op)) launch_x_iter_t<Rad<3, 5, 9>, 16, 8>(a, st); else launch_x_135_0(a, st); }
void launch_x_224_0(const XArgs &a, cudaStream_t st) { launch_x_t<Rad<4, 8, 7>, 32, 4>(a, st); }
void launch_x_224_1(const XArgs &a, cudaStream_t st) { if (x_iteration_op(a.op)) launch_x_iter_t<Rad<4, 7, 8>, 32, 4>(a, st); else launch_x_224_0(a, st); }
void launch_x_336_0(const XArgs &a, cudaStream_t st) { launch_x_t<Rad<4, 12, 7>, 64, 1>(a, st); }
void launch_x_336_1(const XArgs &a, cudaStream_t st) { if (x_iteration_op(a.op)) launch_x_iter_t<Rad<6, 8, 7>, 64, 1>(a, st); else launch_x_336_0(a, st); }
void launch_x_486_0(const XArgs &a, cudaStream_t st) { launch_x_t<Rad<6, 9, 9>, 64, 1>(a, st); }
void launch_x_486_1(const XArgs &a, cudaStream_t st) { if (x_iteration_op(a.op)) launch_x_iter_t<Rad<9, 9, 6>, 96, 1>(a, st); else launch_x_486_0(a, st); }
void launch_x_675_0(const XArgs &a, cudaStream_t st) { launch_x_t<Rad<5, 15, 9>, 96, 1>(a, st); }
void launch_x_675_1(const XArgs &a, cudaStream_t st) { if (x_iteration_op(a.op)) launch_x_iter_t<Rad<3, 15, 15>, 64, 1>(a, st); else launch_x_675_0(a, st); }
void launch_x_900_0(const XArgs &a, cudaStream_t st) { launch_x_t<Rad<6, 15, 10>, 96, 1>(a, st); }
void launch_x_900_1(const XArgs &a, cudaStream_t st) { if (x_iteration_op(a.op)) launch_x_iter_t<Rad<5, 15, 12>, 96, 1>(a, st); else launch_x_900_0(a, st); }
void launch_x_1215_0(const XArgs &a, cudaStream_t st) { launch_x_t<Rad<9, 15, 9>, 160, 1>(a, st); }
void launch_x_1215_1(const XArgs &a, cudaStream_t st) { if (x_iteration_op(a.op)) launch_x_iter_t<Rad<9, 9, 15>, 160, 1>(a, st); else launch_x_1215_0(a, st); }
void launch_x_1620_0(const XArgs &a, cudaStream_t st) { launch_x_t<Rad<9, 15, 12>, 160, 1>(a, st); }
void launch_x_1620_1(const XArgs &a, cudaStream_t st) { if (x_iteration_op(a.op)) launch_x_iter_t<Rad<9, 12, 15>, 160, 1>(a, st); else launch_x_1620_0(a, st); }
}  // namespace dwcu

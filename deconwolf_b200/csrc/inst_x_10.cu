// generated by gen_plans.py -- do not edit
#include "launch_x.cuh"
namespace dwcu {
void launch_x_14_0(const XArgs &, cudaStream_t);
void launch_x_45_0(const XArgs &, cudaStream_t);
void launch_x_96_0(const XArgs &, cudaStream_t);
void launch_x_162_0(const XArgs &, cudaStream_t);
void launch_x_252_0(const XArgs &, cudaStream_t);
void launch_x_384_0(const XArgs &, cudaStream_t);
void launch_x_540_0(const XArgs &, cudaStream_t);
void launch_x_750_0(const XArgs &, cudaStream_t);
void launch_x_1008_0(const XArgs &, cudaStream_t);
void launch_x_1372_0(const XArgs &, cudaStream_t);
void launch_x_1890_0(const XArgs &, cudaStream_t);
void launch_x_14_0(const XArgs &a, cudaStream_t st) { launch_x_t<Rad<2, 7, 1>, 4, 32>(a, st); }
void launch_x_45_0(const XArgs &a, cudaStream_t st) { launch_x_t<Rad<3, 5, 3>, 16, 8>(a, st); }
void launch_x_96_0(const XArgs &a, cudaStream_t st) { launch_x_t<Rad<4, 4, 6>, 16, 8>(a, st); }
void launch_x_96_1(const XArgs &a, cudaStream_t st) { if (x_iteration_op(a.op)) launch_x_iter_t<Rad<2, 8, 6>, 16, 8>(a, st); else launch_x_96_0(a, st); }
void launch_x_162_0(const XArgs &a, cudaStream_t st) { launch_x_t<Rad<3, 9, 6>, 32, 4>(a, st); }
void launch_x_162_1(const XArgs &a, cudaStream_t st) { if (x_iteration_op(a.op)) launch_x_iter_t<Rad<3, 6, 9>, 32, 4>(a, st); else launch_x_162_0(a, st); }
void launch_x_252_0(const XArgs &a, cudaStream_t st) { launch_x_t<Rad<7, 9, 4>, 32, 4>(a, st); }
void launch_x_252_1(const XArgs &a, cudaStream_t st) { if (x_iteration_op(a.op)) launch_x_iter_t<Rad<4, 7, 9>, 32, 4>(a, st); else launch_x_252_0(a, st); }
void launch_x_384_0(const XArgs &a, cudaStream_t st) { launch_x_t<Rad<4, 12, 8>, 64, 1>(a, st); }
void launch_x_384_1(const XArgs &a, cudaStream_t st) { if (x_iteration_op(a.op)) launch_x_iter_t<Rad<6, 8, 8>, 64, 1>(a, st); else launch_x_384_0(a, st); }
void launch_x_540_0(const XArgs &a, cudaStream_t st) { launch_x_t<Rad<5, 12, 9>, 64, 1>(a, st); }
void launch_x_540_1(const XArgs &a, cudaStream_t st) { if (x_iteration_op(a.op)) launch_x_iter_t<Rad<6, 10, 9>, 64, 1>(a, st); else launch_x_540_0(a, st); }
void launch_x_750_0(const XArgs &a, cudaStream_t st) { launch_x_t<Rad<5, 15, 10>, 96, 1>(a, st); }
void launch_x_750_1(const XArgs &a, cudaStream_t st) { if (x_iteration_op(a.op)) launch_x_iter_t<Rad<5, 10, 15>, 96, 1>(a, st); else launch_x_750_0(a, st); }
void launch_x_1008_0(const XArgs &a, cudaStream_t st) { launch_x_t<Rad<6, 14, 12>, 96, 1>(a, st); }
void launch_x_1008_1(const XArgs &a, cudaStream_t st) { if (x_iteration_op(a.op)) launch_x_iter_t<Rad<7, 12, 12>, 96, 1>(a, st); else launch_x_1008_0(a, st); }
void launch_x_1372_0(const XArgs &a, cudaStream_t st) { launch_x_t<Rad<7, 14, 14>, 128, 1>(a, st); }
void launch_x_1372_1(const XArgs &a, cudaStream_t st) { if (x_iteration_op(a.op)) launch_x_iter_t<Rad<14, 14, 7>, 256, 1>(a, st); else launch_x_1372_0(a, st); }
void launch_x_1890_0(const XArgs &a, cudaStream_t st) { launch_x_t<Rad<9, 14, 15>, 160, 1>(a, st); }
void launch_x_1890_1(const XArgs &a, cudaStream_t st) { if (x_iteration_op(a.op)) launch_x_iter_t<Rad<9, 15, 14>, 160, 1>(a, st); else launch_x_1890_0(a, st); }
}  // namespace dwcu

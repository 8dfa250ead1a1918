// generated by gen_plans.py -- do not edit
#include "launch_x.cuh"
namespace dwcu {
void launch_x_9_0(const XArgs &, cudaStream_t);
void launch_x_36_0(const XArgs &, cudaStream_t);
void launch_x_81_0(const XArgs &, cudaStream_t);
void launch_x_147_0(const XArgs &, cudaStream_t);
void launch_x_243_0(const XArgs &, cudaStream_t);
void launch_x_360_0(const XArgs &, cudaStream_t);
void launch_x_504_0(const XArgs &, cudaStream_t);
void launch_x_720_0(const XArgs &, cudaStream_t);
void launch_x_972_0(const XArgs &, cudaStream_t);
void launch_x_1296_0(const XArgs &, cudaStream_t);
void launch_x_1764_0(const XArgs &, cudaStream_t);
void launch_x_9_0(const XArgs &a, cudaStream_t st) { launch_x_t<Rad<3, 3, 1>, 4, 32>(a, st); }
void launch_x_36_0(const XArgs &a, cudaStream_t st) { launch_x_t<Rad<3, 2, 6>, 8, 16>(a, st); }
void launch_x_81_0(const XArgs &a, cudaStream_t st) { launch_x_t<Rad<3, 9, 3>, 16, 8>(a, st); }
void launch_x_147_0(const XArgs &a, cudaStream_t st) { launch_x_t<Rad<3, 7, 7>, 32, 4>(a, st); }
void launch_x_147_1(const XArgs &a, cudaStream_t st) { if (x_iteration_op(a.op)) launch_x_iter_t<Rad<7, 7, 3>, 32, 4>(a, st); else launch_x_147_0(a, st); }
void launch_x_243_0(const XArgs &a, cudaStream_t st) { launch_x_t<Rad<3, 9, 9>, 32, 4>(a, st); }
void launch_x_243_1(const XArgs &a, cudaStream_t st) { if (x_iteration_op(a.op)) launch_x_iter_t<Rad<9, 3, 9>, 32, 4>(a, st); else launch_x_243_0(a, st); }
void launch_x_360_0(const XArgs &a, cudaStream_t st) { launch_x_t<Rad<5, 12, 6>, 64, 1>(a, st); }
void launch_x_360_1(const XArgs &a, cudaStream_t st) { if (x_iteration_op(a.op)) launch_x_iter_t<Rad<6, 10, 6>, 64, 1>(a, st); else launch_x_360_0(a, st); }
void launch_x_504_0(const XArgs &a, cudaStream_t st) { launch_x_t<Rad<7, 9, 8>, 64, 1>(a, st); }
void launch_x_504_1(const XArgs &a, cudaStream_t st) { if (x_iteration_op(a.op)) launch_x_iter_t<Rad<4, 14, 9>, 64, 1>(a, st); else launch_x_504_0(a, st); }
void launch_x_720_0(const XArgs &a, cudaStream_t st) { launch_x_t<Rad<6, 12, 10>, 96, 1>(a, st); }
void launch_x_720_1(const XArgs &a, cudaStream_t st) { if (x_iteration_op(a.op)) launch_x_iter_t<Rad<6, 15, 8>, 96, 1>(a, st); else launch_x_720_0(a, st); }
void launch_x_972_0(const XArgs &a, cudaStream_t st) { launch_x_t<Rad<9, 12, 9>, 128, 1>(a, st); }
void launch_x_972_1(const XArgs &a, cudaStream_t st) { if (x_iteration_op(a.op)) launch_x_iter_t<Rad<9, 9, 12>, 128, 1>(a, st); else launch_x_972_0(a, st); }
void launch_x_1296_0(const XArgs &a, cudaStream_t st) { launch_x_t<Rad<9, 12, 12>, 128, 1>(a, st); }
void launch_x_1296_1(const XArgs &a, cudaStream_t st) { if (x_iteration_op(a.op)) launch_x_iter_t<Rad<9, 16, 9>, 160, 1>(a, st); else launch_x_1296_0(a, st); }
void launch_x_1764_0(const XArgs &a, cudaStream_t st) { launch_x_t<Rad<9, 14, 14>, 128, 1>(a, st); }
void launch_x_1764_1(const XArgs &a, cudaStream_t st) { if (x_iteration_op(a.op)) launch_x_iter_t<Rad<14, 9, 14>, 128, 1>(a, st); else launch_x_1764_0(a, st); }
}  // namespace dwcu

// generated by gen_plans.py -- do not edit
#include "launch_x.cuh"
namespace dwcu {
void launch_x_2_0(const XArgs &, cudaStream_t);
void launch_x_24_0(const XArgs &, cudaStream_t);
void launch_x_60_0(const XArgs &, cudaStream_t);
void launch_x_120_0(const XArgs &, cudaStream_t);
void launch_x_196_0(const XArgs &, cudaStream_t);
void launch_x_300_0(const XArgs &, cudaStream_t);
void launch_x_441_0(const XArgs &, cudaStream_t);
void launch_x_630_0(const XArgs &, cudaStream_t);
void launch_x_840_0(const XArgs &, cudaStream_t);
void launch_x_1134_0(const XArgs &, cudaStream_t);
void launch_x_1536_0(const XArgs &, cudaStream_t);
void launch_x_2_0(const XArgs &a, cudaStream_t st) { launch_x_t<Rad<2, 1, 1>, 4, 32>(a, st); }
void launch_x_24_0(const XArgs &a, cudaStream_t st) { launch_x_t<Rad<2, 4, 3>, 8, 16>(a, st); }
void launch_x_60_0(const XArgs &a, cudaStream_t st) { launch_x_t<Rad<3, 5, 4>, 16, 8>(a, st); }
void launch_x_120_0(const XArgs &a, cudaStream_t st) { launch_x_t<Rad<5, 3, 8>, 16, 8>(a, st); }
void launch_x_120_1(const XArgs &a, cudaStream_t st) { if (x_iteration_op(a.op)) launch_x_iter_t<Rad<3, 5, 8>, 16, 8>(a, st); else launch_x_120_0(a, st); }
void launch_x_196_0(const XArgs &a, cudaStream_t st) { launch_x_t<Rad<4, 7, 7>, 32, 4>(a, st); }
void launch_x_196_1(const XArgs &a, cudaStream_t st) { if (x_iteration_op(a.op)) launch_x_iter_t<Rad<2, 14, 7>, 32, 4>(a, st); else launch_x_196_0(a, st); }
void launch_x_300_0(const XArgs &a, cudaStream_t st) { launch_x_t<Rad<3, 10, 10>, 32, 4>(a, st); }
void launch_x_300_1(const XArgs &a, cudaStream_t st) { if (x_iteration_op(a.op)) launch_x_iter_t<Rad<5, 6, 10>, 32, 4>(a, st); else launch_x_300_0(a, st); }
void launch_x_441_0(const XArgs &a, cudaStream_t st) { launch_x_t<Rad<7, 9, 7>, 64, 1>(a, st); }
void launch_x_441_1(const XArgs &a, cudaStream_t st) { if (x_iteration_op(a.op)) launch_x_iter_t<Rad<7, 7, 9>, 64, 1>(a, st); else launch_x_441_0(a, st); }
void launch_x_630_0(const XArgs &a, cudaStream_t st) { launch_x_t<Rad<6, 15, 7>, 96, 1>(a, st); }
void launch_x_630_1(const XArgs &a, cudaStream_t st) { if (x_iteration_op(a.op)) launch_x_iter_t<Rad<7, 9, 10>, 96, 1>(a, st); else launch_x_630_0(a, st); }
void launch_x_840_0(const XArgs &a, cudaStream_t st) { launch_x_t<Rad<6, 14, 10>, 96, 1>(a, st); }
void launch_x_840_1(const XArgs &a, cudaStream_t st) { if (x_iteration_op(a.op)) launch_x_iter_t<Rad<7, 12, 10>, 96, 1>(a, st); else launch_x_840_0(a, st); }
void launch_x_1134_0(const XArgs &a, cudaStream_t st) { launch_x_t<Rad<9, 14, 9>, 128, 1>(a, st); }
void launch_x_1134_1(const XArgs &a, cudaStream_t st) { if (x_iteration_op(a.op)) launch_x_iter_t<Rad<9, 9, 14>, 128, 1>(a, st); else launch_x_1134_0(a, st); }
void launch_x_1536_0(const XArgs &a, cudaStream_t st) { launch_x_t<Rad<8, 16, 12>, 128, 1>(a, st); }
void launch_x_1536_1(const XArgs &a, cudaStream_t st) { if (x_iteration_op(a.op)) launch_x_iter_t<Rad<8, 12, 16>, 128, 1>(a, st); else launch_x_1536_0(a, st); }
}  // namespace dwcu

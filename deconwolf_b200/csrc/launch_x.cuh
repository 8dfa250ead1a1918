// launch_x.cuh -- launch wrappers for the templated x pass.
#pragma once
#include "launch.cuh"
#include "xpass.cuh"

namespace dwcu {

// a.ntiles counts the plan's tiles (R rows of one plane); this family's
// kernel takes RF rows per CTA
template <class RD, int TP, int R, int RF, int FAM>
void launch_x_fam(const XArgs &a, cudaStream_t st)
{
    static KernelOnce ko;
    using C = XCfg<RD, TP, RF, FAM>;
    const int planes = a.ntiles / ((a.Y + R - 1) / R);
    if (planes < 1) return;
    ensure_smem(ko, k_xpass<RD, TP, RF, FAM>, C::SMEM_BYTES);
    launch_dep(k_xpass<RD, TP, RF, FAM>, dim3((a.Y + RF - 1) / RF, planes), dim3(TP, RF), C::SMEM_BYTES, st, a);
}

// Rows that fill whole warps by themselves run one per CTA, except in the
// ratio family, whose error partials are counted per plan tile.
template <int TP, int R>
constexpr int x_rows() { return TP > 32 ? 1 : R; }

// the ops of one SHB / RL iteration (ratio + error, update); an alternate
// radix plan of the autotuner is compiled for these families only
inline bool x_iteration_op(int op)
{
    const int f = x_family(op);
    return f == XFAM_RATIO || f == XFAM_UPDATE;
}

template <class RD, int TP, int R>
void launch_x_iter_t(const XArgs &a, cudaStream_t st)
{
    if (x_family(a.op) == XFAM_RATIO)
        launch_x_fam<RD, TP, R, R, XFAM_RATIO>(a, st);
    else
        launch_x_fam<RD, TP, R, x_rows<TP, R>(), XFAM_UPDATE>(a, st);
}

template <class RD, int TP, int R>
void launch_x_t(const XArgs &a, cudaStream_t st)
{
    switch (x_family(a.op)) {
    case XFAM_FWD: launch_x_fam<RD, TP, R, x_rows<TP, R>(), XFAM_FWD>(a, st); break;
    case XFAM_STORE: launch_x_fam<RD, TP, R, x_rows<TP, R>(), XFAM_STORE>(a, st); break;
    default: launch_x_iter_t<RD, TP, R>(a, st); break;
    }
}

}  // namespace dwcu

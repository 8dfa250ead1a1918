// launch_x.cuh -- launch wrappers for the templated x pass.
#pragma once
#include "launch.cuh"
#include "xpass.cuh"

namespace dwcu {

// a.ntiles counts tiles of R rows of one plane
template <class RD, int TP, int R, int FAM>
void launch_x_fam(const XArgs &a, cudaStream_t st)
{
    static KernelOnce ko;
    using C = XCfg<RD, TP, R, FAM>;
    const int ytiles = (a.Y + R - 1) / R, planes = a.ntiles / ytiles;
    if (planes < 1) return;
    ensure_smem(ko, k_xpass<RD, TP, R, FAM>, C::SMEM_BYTES);
    launch_dep(k_xpass<RD, TP, R, FAM>, dim3(ytiles, planes), dim3(TP, R), C::SMEM_BYTES, st, a);
}

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
        launch_x_fam<RD, TP, R, XFAM_RATIO>(a, st);
    else
        launch_x_fam<RD, TP, R, XFAM_UPDATE>(a, st);
}

template <class RD, int TP, int R>
void launch_x_t(const XArgs &a, cudaStream_t st)
{
    switch (x_family(a.op)) {
    case XFAM_FWD: launch_x_fam<RD, TP, R, XFAM_FWD>(a, st); break;
    case XFAM_STORE: launch_x_fam<RD, TP, R, XFAM_STORE>(a, st); break;
    default: launch_x_iter_t<RD, TP, R>(a, st); break;
    }
}

}  // namespace dwcu

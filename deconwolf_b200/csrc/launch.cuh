// launch.cuh -- launch wrappers for the templated y and z passes (x: launch_x.cuh).
#pragma once
#include <cuda_runtime.h>
#include <atomic>
#include "passes.cuh"

namespace dwcu {

// Opt a kernel into more than 48 KB of dynamic shared memory, and size a
// persistent grid (resident CTAs per SM x SMs), once per device.
struct KernelOnce {
    std::atomic<unsigned long long> smem_done{0};
    std::atomic<int> grid[64];
    KernelOnce()
    {
        for (auto &g : grid) g.store(0);
    }
};

template <class K>
inline void ensure_smem(KernelOnce &ko, K kernel, size_t bytes)
{
    int dev = 0;
    cudaGetDevice(&dev);
    unsigned long long bit = 1ull << (dev & 63);
    if (bytes > 48 * 1024 && !(ko.smem_done.load() & bit)) {
        cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int) bytes);
        ko.smem_done.fetch_or(bit);
    }
}

template <class K>
inline int persistent_grid(KernelOnce &ko, K kernel, int threads, size_t smem, int ntiles)
{
    int dev = 0;
    cudaGetDevice(&dev);
    int g = ko.grid[dev & 63].load();
    if (g == 0) {
        int per_sm = 0, sms = 0;
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, threads, smem);
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
        g = (per_sm > 0 ? per_sm : 1) * (sms > 0 ? sms : 1);
        ko.grid[dev & 63].store(g);
    }
    return ntiles < g ? ntiles : g;
}

// A launch that may overlap the end of the kernel before it on the stream
// (the kernel calls dep_wait, tma.cuh).  It hides the launch latency between
// passes: 48 x 40 x 10, SHB 10 (102 launches) 408 -> 370 us, 317 x 241 x 33
// periodic 2372 -> 2309, 2048 x 2048 x 60 unchanged.
template <class A>
inline void launch_dep(void (*kernel)(A), dim3 grid, dim3 block, size_t smem, cudaStream_t st, const A &a)
{
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    cudaLaunchKernelEx(&cfg, kernel, a);
}

template <class RD, int T>
void launch_lines_t(const LinesArgs &a, int nblocks, cudaStream_t st)
{
    static KernelOnce ko, kp;
    using C = LinesCfg<RD, T>;
    constexpr int tpl = C::THREADS / T;
    size_t smem = a.mode >= LINES_CONV ? C::SMEM_BYTES : C::SMEM_FFT;
    if (a.es.part) {  // one block more, with room for its sums
        ++nblocks;
        if (smem < sizeof(double) * kErrLanes) smem = sizeof(double) * kErrLanes;
    }
    if (a.planes || a.packed) {
        ensure_smem(kp, k_lines<RD, T, true>, C::SMEM_BYTES);
        launch_dep(k_lines<RD, T, true>, dim3(nblocks), dim3(T, tpl), smem, st, a);
    } else {
        ensure_smem(ko, k_lines<RD, T>, C::SMEM_BYTES);
        launch_dep(k_lines<RD, T>, dim3(nblocks), dim3(T, tpl), smem, st, a);
    }
}

template <class RD, int DIR>
void launch_y_dir(const YArgs &a, cudaStream_t st)
{
    static KernelOnce ko;
    using C = YCfg<RD>;
    ensure_smem(ko, k_ypass<RD, DIR>, C::SMEM_BYTES);
    const int grid = persistent_grid(ko, k_ypass<RD, DIR>, C::THREADS, C::SMEM_BYTES, a.ntiles);
    launch_dep(k_ypass<RD, DIR>, dim3(grid), dim3(C::TX, RD::TPL), C::SMEM_BYTES, st, a);
}

template <class RD>
void launch_y_t(const YArgs &a, cudaStream_t st)
{
    if (a.dir < 0)
        launch_y_dir<RD, -1>(a, st);
    else
        launch_y_dir<RD, +1>(a, st);
}

template <class RD>
void launch_yconv_t(const YArgs &a, cudaStream_t st)
{
    static KernelOnce ko;
    using C = YConvCfg<RD>;
    ensure_smem(ko, k_yconv<RD>, C::SMEM_BYTES);
    const size_t room = a.es.part && C::SMEM_BYTES < sizeof(double) * kErrLanes ? sizeof(double) * kErrLanes : C::SMEM_BYTES;
    launch_dep(k_yconv<RD>, dim3(a.ntiles + (a.es.part ? 1 : 0)), dim3(KB, C::TPL), room, st, a);
}

}  // namespace dwcu

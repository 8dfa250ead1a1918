// passes.cuh -- the y and z FFT passes of one RL/SHB iteration (sm_100a).
//
// Data layout in HBM (per job):
//   real volumes  X x Y x Z floats, x fastest, row pitch X (X even)
//   spectrum      (X/2+1) x Y x Z complex, row pitch XC complex (XC even)
//   image g       M x N x P floats, row pitch GP (even)
//
// Line transforms are self-sorting (Stockham) mixed-radix FFTs of length
// N = RA*RB*RC (RC may be 1) with radices <= 16.  One line is handled by
// TPL = N / min(R) threads; in stage s each active thread runs one radix-R_s
// butterfly fully in registers (dft.cuh), and stages exchange through shared
// memory.  The last stage leaves thread t holding elements t + r*N/R_last,
// which is exactly what the first stage of a transform with the reversed
// radix list reads -- so a forward transform followed by an inverse one (the
// OTF multiply in between) or an inverse followed by a forward one (the
// pointwise op in between) hands over in registers, with no extra exchange.
//
// k_lines  : complex transforms along a strided axis (y or z), T adjacent
//            lines per CTA so every global access is T*8 contiguous bytes.
//            Modes: forward, inverse, and convolve = forward, multiply by the
//            OTF (or its conjugate), inverse: the spectrum is read and
//            written once.
// k_ypass  : the y axis, persistent, one contiguous tile of 4 lines at a time.
// (the x axis: xpass.cuh)
#pragma once
#include <cstdint>
#include "dft.cuh"
#include "tma.cuh"

namespace dwcu {

__host__ __device__ constexpr int cmax(int a, int b) { return a > b ? a : b; }
__host__ __device__ constexpr int cmin(int a, int b) { return a < b ? a : b; }

// Compile-time description of one line length.
template <int RA_, int RB_, int RC_>
struct Rad {
    static constexpr int RA = RA_, RB = RB_, RC = RC_;
    static constexpr int N = RA * RB * RC;
    static constexpr bool THREE = (RC > 1);
    static constexpr int RL = THREE ? RC : RB;  // last radix
    static constexpr int TPL = cmax(cmax(N / RA, N / RB), THREE ? N / RC : 0);
    // padded exchange index: for an even first radix, one spare slot per RA
    // block makes the first stage's stride-RA writes an odd number of
    // float2 apart, which keeps them free of bank conflicts; an odd RA
    // already is, and a spare slot would make the stride even (for RA = 15,
    // every thread of a warp on the same bank), so odd RA is not padded.
    // PADN (the tile size) is the padded bound either way.
    static constexpr int PK = (RA % 2 == 0) ? 1 : 0;
    static constexpr int PADN = N + N / RA + 1;
    static __device__ __forceinline__ int pad(int idx) { return idx + PK * (idx / RA); }
};

// Twiddles of one Stockham stage for butterfly index j: W^r with
// W = W_{NS*R}^{j mod NS}, r = 1 .. R-1.  One value comes from the length-N
// table; the other powers are products of it (squarings for even r), at most
// six products deep, so the twiddles cost one load per stage instead of R-1
// (with most of shared memory in use, the table does not stay in L1).
template <int N, int NS, int R>
__device__ __forceinline__ void stage_twiddles(float2 (&w)[R], int j, const float2 *__restrict__ tw)
{
    constexpr int step = N / (NS * R);
    const int u = (j % NS) * step;
    if constexpr (R > 1) w[1] = __ldg(&tw[u]);
#pragma unroll
    for (int r = 2; r < R; ++r) w[r] = (r % 2 == 0) ? cmul(w[r / 2], w[r / 2]) : cmul(w[r - 1], w[1]);
}
// the table value stage_twiddles loads (for callers that keep it in a register)
template <int N, int NS, int R>
__device__ __forceinline__ float2 stage_twiddle_base(int j, const float2 *__restrict__ tw)
{
    constexpr int step = N / (NS * R);
    return __ldg(&tw[(j % NS) * step]);
}
// stage_twiddles from that value
template <int R>
__device__ __forceinline__ void stage_twiddles_from(float2 (&w)[R], float2 b)
{
    if constexpr (R > 1) w[1] = b;
#pragma unroll
    for (int r = 2; r < R; ++r) w[r] = (r % 2 == 0) ? cmul(w[r / 2], w[r / 2]) : cmul(w[r - 1], w[1]);
}

// one Stockham butterfly on Q rows that share the butterfly index:
// v[q][r] = x_q[j + r*N/R] on entry, multiplied by the stage twiddles w[r]
// (unless NS == 1) and transformed; output r belongs at
// (j/NS)*NS*R + j%NS + r*NS.
template <int NS, int R, int DIR, int Q>
__device__ __forceinline__ void butterfly(float2 (&v)[Q][R], const float2 (&w)[R])
{
    if constexpr (NS > 1) {
#pragma unroll
        for (int r = 1; r < R; ++r)
#pragma unroll
            for (int q = 0; q < Q; ++q) v[q][r] = (DIR < 0) ? cmul(v[q][r], w[r]) : cmulc(v[q][r], w[r]);
    }
#pragma unroll
    for (int q = 0; q < Q; ++q) Dft<R, DIR>::run(v[q]);
}

// Full line transform of Q rows per thread.  On entry thread t (< N/RA)
// holds its first-stage inputs v[q][r] = x_q[t + r*N/RA].  On exit thread t
// (< N/RL) holds o[q][r] = X_q[t + r*N/RL].  smem(q, i) is row q's exchange
// slot for padded index i (RD::pad); every index a thread touches in a stage
// is its base plus a compile-time multiple, so addressing is one add per
// access.  Contains __syncthreads(): call uniformly from the whole block; the
// exchange tiles may be reused by the caller only after another barrier.
// PP (ping-pong): stage 2 writes a second exchange tile, smem2, so that no
// barrier is needed between its reads and its writes; stage 3 reads smem2.
// HOIST: the stage twiddles come from tb2 / tb3 (stage_twiddle_base of
// stages 2 and 3 for this thread, kept by the caller) instead of the table
template <class RD, int DIR, int Q, bool PP, class SM, class SM2, bool HOIST = false>
__device__ __forceinline__ void line_fft_impl(float2 (&v)[Q][RD::RA], float2 (&o)[Q][RD::RL], int t,
                                              const float2 *__restrict__ tw, SM smem, SM2 smem2,
                                              float2 tb2 = float2{}, float2 tb3 = float2{});

template <class RD, int DIR, int Q, class SM>
__device__ __forceinline__ void line_fft(float2 (&v)[Q][RD::RA], float2 (&o)[Q][RD::RL], int t,
                                         const float2 *__restrict__ tw, SM smem)
{
    line_fft_impl<RD, DIR, Q, false, SM, SM>(v, o, t, tw, smem, smem);
}

template <class RD, int DIR, int Q, bool PP, class SM, class SM2, bool HOIST>
__device__ __forceinline__ void line_fft_impl(float2 (&v)[Q][RD::RA], float2 (&o)[Q][RD::RL], int t,
                                              const float2 *__restrict__ tw, SM smem, SM2 smem2, float2 tb2,
                                              float2 tb3)
{
    constexpr int P2 = RD::PK;  // padding of the second exchange
    constexpr int N = RD::N, RA = RD::RA, RB = RD::RB, RC = RD::RC;
    constexpr int M2 = N / RB;  // stage-2 butterflies; read stride, a multiple of RA
    // stage 1 writes t*RA + r  ->  padded t*(RA+PK) + r
    if (t < N / RA) {
        float2 none[RA];
        butterfly<1, RA, DIR, Q>(v, none);
        const int b1 = t * (RA + RD::PK);
#pragma unroll
        for (int q = 0; q < Q; ++q)
#pragma unroll
            for (int r = 0; r < RA; ++r) *smem(q, b1 + r) = v[q][r];
    }
    float2 w2[RB];
    __syncthreads();
    if constexpr (RD::THREE) {
        constexpr int M3 = N / RC;
        float2 u[Q][RB];
        if (t < M2) {
            const int b2 = RD::pad(t);
#pragma unroll
            for (int q = 0; q < Q; ++q)
#pragma unroll
                for (int r = 0; r < RB; ++r) u[q][r] = *smem(q, b2 + r * (M2 + RD::PK * (M2 / RA)));
        }
        if constexpr (!PP) __syncthreads();
        if (t < M2) {
            if constexpr (HOIST) stage_twiddles_from<RB>(w2, tb2);
            else stage_twiddles<N, RA, RB>(w2, t, tw);
            butterfly<RA, RB, DIR, Q>(u, w2);
            const int base = (t / RA) * RA * RB + t % RA;  // writes base + r*RA
            const int b3 = base + P2 * (base / RA);
#pragma unroll
            for (int q = 0; q < Q; ++q)
#pragma unroll
                for (int r = 0; r < RB; ++r) *smem2(q, b3 + r * (RA + P2)) = u[q][r];
        }
        float2 w3[RC];
        __syncthreads();
        if (t < M3) {
            const int b4 = t + P2 * (t / RA);
#pragma unroll
            for (int q = 0; q < Q; ++q)
#pragma unroll
                for (int r = 0; r < RC; ++r) o[q][r] = *smem2(q, b4 + r * (M3 + P2 * (M3 / RA)));
            if constexpr (HOIST) stage_twiddles_from<RC>(w3, tb3);
            else stage_twiddles<N, RA * RB, RC>(w3, t, tw);
            butterfly<RA * RB, RC, DIR, Q>(o, w3);
        }
    } else {
        if (t < M2) {
            const int b2 = RD::pad(t);
#pragma unroll
            for (int q = 0; q < Q; ++q)
#pragma unroll
                for (int r = 0; r < RB; ++r) o[q][r] = *smem(q, b2 + r * (M2 + RD::PK * (M2 / RA)));
            if constexpr (HOIST) stage_twiddles_from<RB>(w2, tb2);
            else stage_twiddles<N, RA, RB>(w2, t, tw);
            butterfly<RA, RB, DIR, Q>(o, w2);
        }
    }
}

template <class RD>
using RevRad = Rad<(RD::THREE ? RD::RC : RD::RB), (RD::THREE ? RD::RB : RD::RA), (RD::THREE ? RD::RA : 1)>;

// ------------------------------------------------------------ spectrum layout
//
// The half-spectrum (kx < X/2+1) is stored blocked by KB = 4 along kx:
//   element (kx, y, z) at  ((z * nkb + kx / KB) * Y + y) * KB + kx % KB
// (nkb = ceil((X/2+1) / KB)).  A y line group (4 neighbouring kx) is then one
// contiguous Y*32-byte block, a z line is strided by the plane size, and the
// two rows y, y+1 of one kx block are 64 contiguous bytes for the x pass.
constexpr int KB = 4;

// ------------------------------------------------------------ error sums
//
// The iteration's error is the sum of the ratio pass's partials.  The
// back-projection's z pass (or single-plane convolution) that follows has one
// block more to form it, off the chain of passes, where nothing needs it
// before that: one launch less per iteration (48 x 40 x 10, SHB 10: 2 us of
// 22 per iteration).
constexpr int kErrLanes = 1024;

struct ErrSum {
    const double *part = nullptr;
    int nb = 0;
    double count = 1;
    float *out = nullptr;
};

// the sum of nb partials by one block of any size, in the fixed order of
// kErrLanes strided sums and a tree over them (valid on thread 0); s: kErrLanes doubles
__device__ __forceinline__ double err_block_sum(const double *part, int nb, double *s, int tid, int threads)
{
    // eight lanes of a thread at a time, so that their loads overlap
    constexpr int G = 8;
    for (int l0 = tid; l0 < kErrLanes; l0 += G * threads) {
        double v[G];
#pragma unroll
        for (int q = 0; q < G; ++q) v[q] = 0.0;
        for (int i0 = 0; i0 < nb; i0 += kErrLanes) {
#pragma unroll
            for (int q = 0; q < G; ++q) {
                const int l = l0 + q * threads;
                if (l < kErrLanes && i0 + l < nb) v[q] += part[i0 + l];
            }
        }
#pragma unroll
        for (int q = 0; q < G; ++q)
            if (l0 + q * threads < kErrLanes) s[l0 + q * threads] = v[q];
    }
    __syncthreads();
    for (int o = kErrLanes / 2; o > 0; o >>= 1) {
        for (int l = tid; l < o; l += threads) s[l] += s[l + o];
        __syncthreads();
    }
    return s[0];
}

__device__ __forceinline__ void err_store(const ErrSum &e, double *s, int tid, int threads)
{
    const double v = err_block_sum(e.part, e.nb, s, tid, threads);
    if (tid == 0) *e.out = (float) (v / e.count);
}

// ------------------------------------------------------------ k_lines

enum LinesMode { LINES_FWD = 0, LINES_INV = 1, LINES_CONV = 2, LINES_CONV_CONJ = 3 };

struct LinesArgs {
    float2 *data;            // spectrum
    const float2 *otf;       // OTF, same layout as data (convolve modes)
    const float2 *tw;        // tw[m] = exp(-2 pi i m / N), m < N
    long long line_stride;   // complex elements between neighbours on a line
    long long outer_stride;  // complex elements between outer blocks
    int ncols;               // adjacent lines (contiguous columns) per outer block
    int ntiles;              // ceil(ncols / T)
    int mode;
    int nin;                 // elements [0, nin) of a line are read; the rest are zero
    int nout;                // elements [0, nout) of a line are written
    // planes mode (a job split by z planes over GPUs): element n of column c
    // is planes[n][col0 + c], plane n on whichever GPU holds it (peer
    // loads and stores); `data` is unused and `line_stride` is the OTF's
    float2 *const *planes = nullptr;
    long long col0 = 0;
    // packed mode (the standalone transforms' last or first pass): a forward
    // pass writes, an inverse pass reads, element n of the column (kx, y) at
    // packed[n * packed_stride + y * packed_row + kx], kx < packed_row: the
    // caller's plain half-spectrum, with no pass of its own to reorder it
    float2 *packed = nullptr;
    long long packed_stride = 0;
    int packed_row = 0;
    int packed_y = 0;  // rows per plane
    ErrSum es;         // (part not null) formed by the first block
};

template <class RD, int T>
struct LinesCfg {
    static constexpr int THREADS = T * cmax(RD::TPL, RevRad<RD>::TPL);
    // exchange tile, then (convolve modes) the OTF tile, prefetched at entry
    static constexpr int XCH_F2 = cmax(RD::PADN, RevRad<RD>::PADN) * T;
    static constexpr size_t SMEM_FFT = sizeof(float2) * (size_t) XCH_F2;
    static constexpr size_t SMEM_BYTES = SMEM_FFT + sizeof(float2) * (size_t) RD::N * T;
    // as many resident CTAs (up to four) as leave at least 64 registers a thread
    static constexpr int MIN_BLOCKS =
        (THREADS * 4 <= 1024 && SMEM_BYTES * 4 <= 225 * 1024) ? 4
        : (THREADS * 3 <= 1024 && SMEM_BYTES * 3 <= 225 * 1024) ? 3
        : (THREADS * 2 <= 1024 && SMEM_BYTES * 2 <= 225 * 1024) ? 2 : 1;
};

// PL: planes or packed mode
template <class RD, int T, bool PL = false>
__global__ void __launch_bounds__(LinesCfg<RD, T>::THREADS, LinesCfg<RD, T>::MIN_BLOCKS)
k_lines(LinesArgs a)
{
    using RV = RevRad<RD>;
    constexpr int N = RD::N;
    extern __shared__ float2 sm[];
    const int line = threadIdx.x;
    const int t = threadIdx.y;
    // (the error's block comes first, so that it is not the launch's tail)
    const bool es = !PL && a.es.part;
    const unsigned bx = es ? blockIdx.x - 1 : blockIdx.x;
    const int tile = bx % a.ntiles;
    const long long outer = bx / a.ntiles;
    const int col = tile * T + line;
    const bool valid = col < a.ncols;
    const long long off = outer * a.outer_stride + col;
    float2 *base = a.data + off;
    const long long ls = a.line_stride;
    const int mode = a.mode;
    // the packed half-spectrum's element 0 of this line, and whether it has one
    float2 *pk = nullptr;
    bool pk_in = false, pk_out = false, valid_in = valid, valid_out = valid;
    if constexpr (PL) {
        if (a.packed) {
            const int q = col / KB, kb = q / a.packed_y, kx = kb * KB + col % KB;
            pk = a.packed + (long long) (q - kb * a.packed_y) * a.packed_row + kx;
            pk_in = mode == LINES_INV;
            pk_out = !pk_in;
            if (kx >= a.packed_row) (pk_in ? valid_in : valid_out) = false;
        }
    }
    // element n of this thread's line
    auto elem = [&](int n, bool packed) -> float2 * {
        if constexpr (PL) {
            if (a.planes) return a.planes[n] + (a.col0 + col);
            if (packed) return pk + (long long) n * a.packed_stride;
        }
        return base + (long long) n * ls;
    };
    auto smem = [&](int, int i) { return sm + (size_t) i * T + line; };
    using Cfg = LinesCfg<RD, T>;
    float2 *sotf = sm + Cfg::XCH_F2;  // OTF tile [n][col] (convolve modes)
    const int col0 = tile * T;
    dep_wait();  // (no dep_start_next: ahead of the stores it cost 3 % at z 120)
    if (es && blockIdx.x == 0) {
        err_store(a.es, reinterpret_cast<double *>(sm), t * T + line, LinesCfg<RD, T>::THREADS);
        return;
    }
    if (mode >= LINES_CONV && (T % 2) == 0) {
        // the tile's OTF columns arrive while the forward transform runs:
        // 16-byte pieces (two columns) of each of the N rows
        const int tid = t * T + line;
        const float2 *h0 = a.otf + outer * a.outer_stride + col0;
        constexpr int PPR = T / 2;  // pieces per row
        for (int e = tid; e < N * PPR; e += Cfg::THREADS) {
            const int n = e / PPR, p = e - n * PPR;
            if (col0 + 2 * p < a.ncols) cp_async16(sotf + n * T + 2 * p, h0 + (long long) n * ls + 2 * p);
        }
        cp_async_commit();
    }

    float2 v[1][RD::RA];
    if (t < N / RD::RA) {
#pragma unroll
        for (int r = 0; r < RD::RA; ++r) {
            const int n = t + r * (N / RD::RA);
            v[0][r] = (valid_in && n < a.nin) ? *elem(n, pk_in) : make_float2(0.f, 0.f);
        }
    }
    float2 o[1][RD::RL];
    if (mode == LINES_INV)
        line_fft<RD, +1, 1>(v, o, t, a.tw, smem);
    else
        line_fft<RD, -1, 1>(v, o, t, a.tw, smem);
    constexpr int SL = N / RD::RL;
    if (mode == LINES_FWD || mode == LINES_INV) {
        if (t < SL && valid_out) {
#pragma unroll
            for (int r = 0; r < RD::RL; ++r)
                if (t + r * SL < a.nout) *elem(t + r * SL, pk_out) = o[0][r];
        }
        return;
    }
    // multiply by the OTF (conjugated for the back-projection)
    if constexpr ((T % 2) == 0) {
        cp_async_wait_all();
        __syncthreads();  // every thread's pieces of the OTF tile have landed
        if (t < SL && valid) {
#pragma unroll
            for (int r = 0; r < RD::RL; ++r) {
                const float2 q = sotf[(t + r * SL) * T + line];
                o[0][r] = (mode == LINES_CONV) ? cmul(o[0][r], q) : cmulc(o[0][r], q);
            }
        }
    } else if (t < SL && valid) {
        const float2 *h = a.otf + off;
#pragma unroll
        for (int r = 0; r < RD::RL; ++r) {
            float2 q = __ldg(&h[(long long) (t + r * SL) * ls]);
            o[0][r] = (mode == LINES_CONV) ? cmul(o[0][r], q) : cmulc(o[0][r], q);
        }
    }
    __syncthreads();  // the exchange tile is free again
    float2 q[1][RV::RL];
    line_fft<RV, +1, 1>(o, q, t, a.tw, smem);
    constexpr int SQ = N / RV::RL;
    if (t < SQ && valid) {
#pragma unroll
        for (int r = 0; r < RV::RL; ++r)
            if (t + r * SQ < a.nout) *elem(t + r * SQ, false) = q[0][r];
    }
}

// ------------------------------------------------------------ k_ypass

struct YArgs {
    float2 *data;
    const float2 *tw;   // tw[m] = exp(-2 pi i m / Y)
    int *err;           // error flags (bounded waits)
    int ntiles;         // Z * nkb
    int dir;            // -1 forward, +1 inverse
    const float2 *otf = nullptr;  // convolution (k_yconv): the OTF, same layout as data
    int conj = 0;       // multiply by its conjugate
    ErrSum es;          // (k_yconv, part not null) formed by the first block
};

template <class RD>
struct YCfg {
    static constexpr int Q = 1;                  // lines per thread
    static constexpr int TX = KB / Q;            // threads across the 4 lines
    static constexpr int THREADS = TX * RD::TPL;
    static constexpr int BUF_F2 = RD::PADN * KB;
    // two tile buffers (the next tile's copy lands in one while the other is
    // transformed) and, where it fits, a third exchange tile so that the
    // transform's stages need fewer barriers (line_fft_impl, PP)
    static constexpr bool PP = 3 * sizeof(float2) * (size_t) BUF_F2 + 64 <= 227 * 1024;
    static constexpr size_t SMEM_BYTES = (PP ? 3 : 2) * sizeof(float2) * (size_t) BUF_F2 + 64;
    static constexpr uint32_t TILE_BYTES = (uint32_t) (RD::N * KB * sizeof(float2));
};

// Persistent y transform: one CTA loops over (z, kx-block) tiles; each tile
// (4 lines of length Y, contiguous) arrives by one bulk copy, the next
// tile's copy is in flight while this one is transformed.
template <class RD, int DIR>
__global__ void __launch_bounds__(YCfg<RD>::THREADS)
k_ypass(YArgs a)
{
    using C = YCfg<RD>;
    constexpr int N = RD::N;
    constexpr int Q = C::Q;
    extern __shared__ __align__(128) unsigned char ysm[];
    uint64_t *bars = reinterpret_cast<uint64_t *>(ysm);
    float2 *bufs = reinterpret_cast<float2 *>(ysm + 64);
    const int l0 = threadIdx.x * Q;  // this thread's first line in the tile
    const int t = threadIdx.y;
    const int tid = t * C::TX + threadIdx.x;
    if (tid == 0) {
        mbar_init(&bars[0], 1);
        mbar_init(&bars[1], 1);
        fence_mbar_init();
    }
    __syncthreads();
    // this thread's stage twiddle values are the same for every tile
    const float2 tb2 = stage_twiddle_base<N, RD::RA, RD::RB>(t < N / RD::RB ? t : 0, a.tw);
    const float2 tb3 = RD::THREE ? stage_twiddle_base<N, RD::RA * RD::RB, (RD::THREE ? RD::RC : 1)>(
                                       t < N / (RD::THREE ? RD::RC : 1) ? t : 0, a.tw)
                                 : make_float2(1.f, 0.f);
    int tile = blockIdx.x;
    dep_wait();
    if (tid == 0 && tile < a.ntiles) {
        mbar_arrive_expect_tx(&bars[0], C::TILE_BYTES);
        tma_load_1d(bufs, a.data + (size_t) tile * N * KB, C::TILE_BYTES, &bars[0]);
    }
    for (int it = 0; tile < a.ntiles; ++it, tile += gridDim.x) {
        const int b = it & 1;
        float2 *buf = bufs + (size_t) b * C::BUF_F2;
        fence_proxy_async();  // this thread's accesses to the other buffer precede the next bulk copy into it
        __syncthreads();      // the other buffer is no longer read
        const int next = tile + gridDim.x;
        if (next >= a.ntiles) dep_start_next();
        if (tid == 0 && next < a.ntiles) {
            fence_proxy_async();
            mbar_arrive_expect_tx(&bars[b ^ 1], C::TILE_BYTES);
            tma_load_1d(bufs + (size_t) (b ^ 1) * C::BUF_F2, a.data + (size_t) next * N * KB, C::TILE_BYTES,
                        &bars[b ^ 1]);
        }
        if (!wait_all(&bars[b], (it >> 1) & 1, a.err, 1 << 8)) {
            if (tid == 0 && next < a.ntiles) drain(&bars[b ^ 1], ((it + 1) >> 1) & 1);
            return;
        }
        float2 v[Q][RD::RA];
        if (t < N / RD::RA) {
#pragma unroll
            for (int r = 0; r < RD::RA; ++r)
#pragma unroll
                for (int q = 0; q < Q; ++q) v[q][r] = buf[(t + r * (N / RD::RA)) * KB + l0 + q];
        }
        auto smem = [&](int q, int i) { return buf + (size_t) i * KB + l0 + q; };
        float2 o[Q][RD::RL];
        if constexpr (C::PP) {
            // stage 1 writes the third tile (no barrier after the natural-order
            // reads), stage 2 writes the tile buffer back
            float2 *ex = bufs + (size_t) 2 * C::BUF_F2;
            auto smemx = [&](int q, int i) { return ex + (size_t) i * KB + l0 + q; };
            line_fft_impl<RD, DIR, Q, true, decltype(smemx), decltype(smem), true>(v, o, t, a.tw, smemx,
                                                                                          smem, tb2, tb3);
        } else {
            __syncthreads();  // natural-order reads done; the buffer becomes the exchange tile
            line_fft<RD, DIR, Q>(v, o, t, a.tw, smem);
        }
        constexpr int SL = N / RD::RL;
        if (t < SL) {
            float2 *dst = a.data + (size_t) tile * N * KB + l0;
#pragma unroll
            for (int r = 0; r < RD::RL; ++r)
#pragma unroll
                for (int q = 0; q < Q; ++q) dst[(size_t) (t + r * SL) * KB + q] = o[q][r];
        }
    }
}

// ------------------------------------------------------------ k_yconv
//
// The convolution of a job of one plane (Z = 1: no z transform): forward y
// transform, OTF multiply and inverse y transform of one tile in one kernel,
// instead of a y pass, a z pass that only multiplies, and a y pass.  One CTA
// per tile (a plane has at most a few hundred); the OTF's elements, which sit
// where the forward transform leaves its outputs, are loaded ahead of it.
// 972 x 768 plane: 35 -> 9 us per convolution.
template <class RD>
struct YConvCfg {
    using RV = RevRad<RD>;
    static constexpr int TPL = cmax(RD::TPL, RV::TPL);
    static constexpr int THREADS = KB * TPL;
    static constexpr int BUF_F2 = cmax(RD::PADN, RV::PADN) * KB;
    static constexpr size_t SMEM_BYTES = 2 * sizeof(float2) * (size_t) BUF_F2 + 64;
    static constexpr uint32_t TILE_BYTES = (uint32_t) (RD::N * KB * sizeof(float2));
};

template <class RD>
__global__ void __launch_bounds__(YConvCfg<RD>::THREADS)
k_yconv(YArgs a)
{
    using C = YConvCfg<RD>;
    using RV = RevRad<RD>;
    constexpr int N = RD::N, SL = N / RD::RL, SQ = N / RV::RL;
    extern __shared__ __align__(128) unsigned char ysm[];
    uint64_t *bar = reinterpret_cast<uint64_t *>(ysm);
    float2 *A = reinterpret_cast<float2 *>(ysm + 64), *B = A + C::BUF_F2;
    const int l = threadIdx.x, t = threadIdx.y;
    const unsigned bx = a.es.part ? blockIdx.x - 1 : blockIdx.x;  // the error's block comes first
    float2 *tile = a.data + (size_t) bx * N * KB;
    dep_wait();
    if (a.es.part && blockIdx.x == 0) {
        err_store(a.es, reinterpret_cast<double *>(ysm), t * KB + l, C::THREADS);
        return;
    }
    if (t == 0 && l == 0) {
        mbar_init(bar, 1);
        fence_mbar_init();
        mbar_arrive_expect_tx(bar, C::TILE_BYTES);
        tma_load_1d(A, tile, C::TILE_BYTES, bar);
    }
    float2 h[RD::RL];
    if (t < SL) {
        const float2 *src = a.otf + (size_t) bx * N * KB + l;
#pragma unroll
        for (int r = 0; r < RD::RL; ++r) h[r] = __ldg(&src[(size_t) (t + r * SL) * KB]);
    }
    __syncthreads();  // the barrier is initialised
    if (!wait_all(bar, 0, a.err, 1 << 8)) {
        if (t == 0 && l == 0) drain(bar, 0);
        return;
    }
    auto inA = [&](int, int i) { return A + (size_t) i * KB + l; };
    auto inB = [&](int, int i) { return B + (size_t) i * KB + l; };
    float2 v[1][RD::RA], o[1][RD::RL], q[1][RV::RL];
    if (t < N / RD::RA) {
#pragma unroll
        for (int r = 0; r < RD::RA; ++r) v[0][r] = A[(size_t) (t + r * (N / RD::RA)) * KB + l];
    }
    // three stages: B, then A; the inverse's first stage writes B again while
    // the forward's last may still read A.  Two stages: B, then A.
    line_fft_impl<RD, -1, 1, true, decltype(inB), decltype(inA)>(v, o, t, a.tw, inB, inA);
    if (t < SL) {
#pragma unroll
        for (int r = 0; r < RD::RL; ++r) o[0][r] = a.conj ? cmulc_paired(o[0][r], h[r]) : cmul_paired(o[0][r], h[r]);
    }
    if constexpr (RD::THREE)
        line_fft_impl<RV, +1, 1, true, decltype(inB), decltype(inA)>(o, q, t, a.tw, inB, inA);
    else
        line_fft_impl<RV, +1, 1, true, decltype(inA), decltype(inB)>(o, q, t, a.tw, inA, inB);
    if (t < SQ) {
#pragma unroll
        for (int r = 0; r < RV::RL; ++r) tile[(size_t) (t + r * SQ) * KB + l] = q[0][r];
    }
}

}  // namespace dwcu

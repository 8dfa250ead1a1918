// xpass.cuh -- the x axis of one RL/SHB iteration (sm_100a): R rows per CTA,
// optional C2R (Hermitian pre-processing + half-length complex inverse), one
// pointwise op on the real values (ratio + I-divergence, SHB/RL update,
// Bertero weights, ...), optional R2C (half-length forward + Hermitian
// post-processing), all in one kernel.  Layouts: passes.cuh.
#pragma once
#include "passes.cuh"

namespace dwcu {

enum XOp {
    XOP_FWD_COPY = 0,    // src real volume -> R2C
    XOP_FWD_ONES = 1,    // 1 on the image region, 0 elsewhere -> R2C
    XOP_FWD_SHBP = 2,    // p = max(x + a(x - xp), bg) -> R2C
    XOP_RATIO_SHB = 3,   // C2R -> error partial -> ratio (SHB guard) -> R2C
    XOP_RATIO_RL = 4,    // C2R -> error partial -> ratio (RL guard) -> R2C
    XOP_ERROR_ONLY = 5,  // C2R -> error partial
    XOP_UPDATE_SHB = 6,  // C2R -> x' = clamp(t * (p*W)), store -> [p' -> R2C]
    XOP_UPDATE_RL = 7,   // C2R -> x' = clamp(t * (x*W)), store -> [x' -> R2C]
    XOP_WEIGHTS = 8,     // C2R -> W = P1 > 0.01 ? 1/P1 : 0, store
    XOP_STORE = 9,       // C2R -> store real
    XOP_FWD_PSF = 10,    // the PSF, its peak moved to the origin, scaled -> R2C
};

struct JobScalars {
    float bg;        // background level (auto: max(min(g), 0.01))
    float x0;        // flat start value
    double sumg;     // sum of the image in double
    float gmin;
    float gmax;      // largest magnitude in the image
    double psfsum;   // sum of the PSF in double
    int flags;       // bit 0/1: non-finite image/PSF; bits 8+: bounded waits that gave up
};

struct PsfPeak;

struct XArgs {
    float2 *S;             // spectrum (blocked layout)
    const float2 *tw;      // tw[m] = exp(-2 pi i m / X), m < X (Hermitian pre/post)
    const float2 *twL;     // twL[m] = exp(-2 pi i m / L), m < L (stage twiddles)
    const float *g;        // image, row pitch GP
    const float *src;      // FWD_COPY source / x_k for SHB and RL
    const float *srcp;     // x_{k-1} for SHB
    const float *Wt;       // Bertero weights (may be null)
    float *dst;            // real output (UPDATE: x_{k+1}; WEIGHTS/STORE)
    double *partial;       // per-tile error partials (ops with an error)
    const JobScalars *sc;  // bg, ...
    long long X;           // real row pitch in floats (even)
    int bulk;              // real rows start at multiples of 16 bytes, X a multiple of 4
    long long GP;          // image row pitch, multiple of 4
    int Y, Z;              // padded dims
    int M, N, P;           // image dims
    int nkb;               // kx blocks
    int ntiles;            // Z * ceil(Y / R)
    int op;
    int r2c;               // run the forward transform after the op
    int metric;            // 1: I-divergence, 0: squared error
    int positivity;        // SHB: clamp x' at bg
    int rl_clamp;          // RL: clamp x' at bg when bg > 0
    double alpha;          // SHB extrapolation weight of the step being finished
    double alpha_next;     // SHB extrapolation weight of the next step
    // periodic x (wrapx): the row is wM-periodic; before the forward
    // transform, [wM, wM+hx) and [X-hx, X) take copies of [0, hx) and
    // [wM-hx, wM), the rest of [wM, X) is zero
    int wrapx, wM, hx;
    // XOP_FWD_PSF: src is the compact PSF, no larger than the volume
    int pM, pN, pP;
    const int *peak;       // its first maximum (x, y, z)
    float scale;
};

__device__ __forceinline__ float shb_p(float xv, float xpv, double alpha, float bg)
{
    // method_shb.c:337-338: p = x + alpha*(x - xp) in double, stored as float; p < bg -> bg
    float p = (float) ((double) xv + alpha * (double) (xv - xpv));
    return p < bg ? bg : p;
}

// ops are compiled in four families, one kernel each, so that every kernel's
// code stays small: forward-only, ratio/error, update, and C2R-store ops
enum XFam { XFAM_FWD = 0, XFAM_RATIO = 1, XFAM_UPDATE = 2, XFAM_STORE = 3 };
__host__ __device__ constexpr int x_family(int op)
{
    return op <= XOP_FWD_SHBP || op == XOP_FWD_PSF ? XFAM_FWD
         : op <= XOP_ERROR_ONLY ? XFAM_RATIO
         : op <= XOP_UPDATE_RL ? XFAM_UPDATE : XFAM_STORE;
}

// one voxel's error: squared, or g*logf(g/y) - (g - y) for y > 0 and g > 0
// (dw.c:1514-1517, which divides in double and rounds to float for logf; the
// float division gives the same float except in double-rounding ties), with
// the quotient q = g/y already computed (only read when y > 0 and g > 0)
__device__ __forceinline__ double err_term_q(float yv, float gv, float q, int metric)
{
    const double y = yv, g = gv;
    if (metric == 0) return (y - g) * (y - g);
    if (yv > 0.f && gv > 0.f) return g * (double) logf(q) - (g - y);
    return 0.0;
}
__device__ __forceinline__ bool op_reads_x(int op)
{
    return op == XOP_FWD_COPY || op == XOP_FWD_SHBP || op == XOP_UPDATE_SHB || op == XOP_UPDATE_RL;
}
__device__ __forceinline__ bool op_reads_xp(int op) { return op == XOP_FWD_SHBP || op == XOP_UPDATE_SHB; }

// Quotients g/d of two lanes: a reciprocal refined by one Newton step, the
// product, and one correction by its exact residual (Markstein, "Computation
// of elementary functions on the IBM RISC System/6000 processor", 1990),
// which rounds the quotient correctly while nothing leaves the normal range:
// |d| in [2^-60, 2^60], |g| <= 2^60 (a quotient below the normal range is
// within a unit in its last place).  In paired instructions and without a
// branch, where the division operator has one per quotient.
__device__ __forceinline__ float2 div_pair(float2 g, float2 d)
{
    float2 r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r.x) : "f"(d.x));
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r.y) : "f"(d.y));
    const float2 nd = make_float2(-d.x, -d.y);
    const float2 e = __ffma2_rn(nd, r, make_float2(1.f, 1.f));
    r = __ffma2_rn(r, e, r);
    const float2 q = __fmul2_rn(g, r);
    const float2 rem = __ffma2_rn(nd, q, g);
    return __ffma2_rn(rem, r, q);
}

// Natural logarithms of two lanes, normal and positive: q = 2^e m with m in
// [sqrt(1/2), sqrt(2)), log q = e ln 2 + f - f^2/2 + f^3 P(f) with f = m - 1
// and P of degree 8 fitted (weighted minimax) to that interval; ln 2 is split
// as by Cody and Waite (Software Manual for the Elementary Functions, 1980),
// 355/512 and the rest, so that e times its high part is exact.  Over all
// positive normal floats the largest error is 0.852 units in the last place,
// the mean 0.25 (that of correct rounding).
__device__ __forceinline__ float2 log_pair(float2 q)
{
    auto both = [](float c) { return make_float2(c, c); };
    // 2^23 e, as an integer: the distance from sqrt(1/2) without its low bits
    const int i0 = __float_as_int(q.x), i1 = __float_as_int(q.y);
    const int k0 = (i0 - 0x3f3504f3) & 0xff800000, k1 = (i1 - 0x3f3504f3) & 0xff800000;
    const float2 e = make_float2((float) k0, (float) k1);  // 2^23 e, exact
    const float2 m = make_float2(__int_as_float(i0 - k0), __int_as_float(i1 - k1));
    const float2 f = __fadd2_rn(m, both(-1.f));
    float2 p = both(0.06746644f);
    p = __ffma2_rn(p, f, both(-0.116756566f));
    p = __ffma2_rn(p, f, both(0.118881635f));
    p = __ffma2_rn(p, f, both(-0.124055885f));
    p = __ffma2_rn(p, f, both(0.14219552f));
    p = __ffma2_rn(p, f, both(-0.16667996f));
    p = __ffma2_rn(p, f, both(0.20002119f));
    p = __ffma2_rn(p, f, both(-0.2500001f));
    p = __ffma2_rn(p, f, both(0.33333313f));
    p = __ffma2_rn(p, f, both(-0.5f));
    const float2 t = __fmul2_rn(__fmul2_rn(f, f), p);
    constexpr float kScale = 1.f / 8388608.f;
    const float2 lo = __ffma2_rn(e, both(-2.1219444e-4f * kScale), t);
    return __ffma2_rn(e, both(0.693359375f * kScale), __fadd2_rn(f, lo));
}

constexpr float kRatioBig = 1152921504606846976.f;  // 2^60: the range div_pair is exact in

// the smaller of two values, NaN if either is
__device__ __forceinline__ float min_nan(float a, float b)
{
    float m;
    asm("min.NaN.f32 %0, %1, %2;" : "=f"(m) : "f"(a), "f"(b));
    return m;
}
constexpr int XCH = 4;  // elements whose real inputs an update loads together (2 and 8: 2-10 % slower)

// The pointwise op of one row: w[r] holds z[n] = (x[2n], x[2n+1]) for
// n = t + r*SL -- the C2R output for the C2R ops -- and is replaced by the
// values handed to the forward transform.  sx, sxp, sw: the row's real inputs
// in global memory (x or the image row, x_{k-1}, weights), brought into L2 by
// an earlier block's prefetch.
// The switch is outside the element loop so each op is one straight loop.
template <int FAM, int RL, int SL>
__device__ __forceinline__ void x_row_op(const XArgs &a, int op, int t, long long rbase, const float *sx,
                                         const float *sxp, const float *sw, bool in_img_row, float bg,
                                         float2 (&w)[RL], double &acc)
{
    const int M = a.M;
    // only this family's cases are compiled into the kernel
    if (x_family(op) != FAM) return;
    if constexpr (FAM == XFAM_RATIO) {
        // The usual case: every y of this thread is positive and above the
        // guard, and nothing is near the ends of the float range.  The three
        // ops then share the quotient and differ outside the image only, and
        // neither the quotient nor the logarithm needs a branch.  (Everything
        // else, NaN among it: below.)
        float lo = 1.f, hi = 1.f;
#pragma unroll
        for (int r = 0; r < RL; ++r) {
            const int c0 = 2 * (t + r * SL);
            if (!(in_img_row && c0 < M)) w[r].x = 1.f;
            if (!(in_img_row && c0 + 1 < M)) w[r].y = 1.f;
            lo = min_nan(lo, min_nan(w[r].x, w[r].y));
            hi = fmaxf(hi, fmaxf(w[r].x, w[r].y));
        }
        if (lo > 1e-6f && hi <= kRatioBig && a.sc->gmax <= kRatioBig) {
            const float outside = op == XOP_RATIO_RL ? 1e-6f : 0.f;
            // (one loop per metric: a branch inside it cost 8 % of the pass)
            auto each = [&](auto idiv) {
#pragma unroll
                for (int r = 0; r < RL; ++r) {
                    const int c0 = 2 * (t + r * SL);
                    const bool img0 = in_img_row && c0 < M, img1 = in_img_row && c0 + 1 < M;
                    float2 gv = img0 ? *reinterpret_cast<const float2 *>(sx + c0) : make_float2(0.f, 0.f);
                    if (!img1) gv.y = 0.f;
                    const float2 v = div_pair(gv, w[r]);
                    if constexpr (decltype(idiv)::value) {
                        // g logf(g/y) - (g - y) where g > 0 (dw.c:1514-1517)
                        const float2 lg = log_pair(v);
                        if (gv.x > 0.f) acc += (double) gv.x * (double) lg.x - ((double) gv.x - (double) w[r].x);
                        if (gv.y > 0.f) acc += (double) gv.y * (double) lg.y - ((double) gv.y - (double) w[r].y);
                    } else {
                        const double d0 = img0 ? (double) w[r].x - (double) gv.x : 0.0;
                        const double d1 = img1 ? (double) w[r].y - (double) gv.y : 0.0;
                        acc += d0 * d0;
                        acc += d1 * d1;
                    }
                    w[r] = make_float2(img0 ? v.x : outside, img1 ? v.y : outside);
                }
            };
            if (a.metric != 0) each(std::true_type{});
            else each(std::false_type{});
            return;
        }
    }
    switch (op) {
    case XOP_FWD_COPY:
        if constexpr (FAM == XFAM_FWD) {
#pragma unroll
            for (int r = 0; r < RL; ++r) w[r] = *reinterpret_cast<const float2 *>(sx + 2 * (t + r * SL));
        }
        break;
    case XOP_FWD_ONES:  // initial_guess, dw.c:2497-2520
        if constexpr (FAM == XFAM_FWD) {
#pragma unroll
            for (int r = 0; r < RL; ++r) {
                const int c0 = 2 * (t + r * SL);
                w[r] = make_float2(in_img_row && c0 < M ? 1.f : 0.f, in_img_row && c0 + 1 < M ? 1.f : 0.f);
            }
        }
        break;
    case XOP_FWD_SHBP:
        if constexpr (FAM == XFAM_FWD) {
#pragma unroll
            for (int r = 0; r < RL; ++r) {
                const int c0 = 2 * (t + r * SL);
                const float2 xv = *reinterpret_cast<const float2 *>(sx + c0);
                const float2 xq = *reinterpret_cast<const float2 *>(sxp + c0);
                w[r] = make_float2(shb_p(xv.x, xq.x, a.alpha, bg), shb_p(xv.y, xq.y, a.alpha, bg));
            }
        }
        break;
    case XOP_FWD_PSF:
        // sx: the PSF row that lands here (null: none); column c holds the
        // PSF's column (c + peak) mod X
        if constexpr (FAM == XFAM_FWD) {
            const int px = a.peak[0];
#pragma unroll
            for (int r = 0; r < RL; ++r) {
                const int c0 = 2 * (t + r * SL);
                int s0 = c0 + px, s1 = c0 + 1 + px;
                if (s0 >= 2 * RL * SL) s0 -= 2 * RL * SL;
                if (s1 >= 2 * RL * SL) s1 -= 2 * RL * SL;
                w[r] = make_float2(sx && s0 < a.pM ? sx[s0] * a.scale : 0.f, sx && s1 < a.pM ? sx[s1] * a.scale : 0.f);
            }
        }
        break;
    case XOP_RATIO_SHB:
        if constexpr (FAM != XFAM_RATIO) break;
#pragma unroll
        for (int r = 0; r < RL; ++r) {
            const int c0 = 2 * (t + r * SL);
            const bool img0 = in_img_row && c0 < M;
            const bool img1 = in_img_row && c0 + 1 < M;
            const float y0 = w[r].x, y1 = w[r].y;
            const float2 gv = img0 ? *reinterpret_cast<const float2 *>(sx + c0) : make_float2(0.f, 0.f);
            const float g0 = gv.x, g1 = img1 ? gv.y : 0.f;
            // method_shb.c:31-48: |y| < 1e-6 -> +-1e-6; r = g/y on the image, 0 elsewhere.
            // (double)|y| < 1e-6 holds exactly when |y| <= 1e-6f, the float just below 1e-6.
            const float d0 = fabsf(y0) <= 1e-6f ? copysignf(1e-6f, y0) : y0;
            const float d1 = fabsf(y1) <= 1e-6f ? copysignf(1e-6f, y1) : y1;
            const float v0 = img0 ? g0 / d0 : 0.f;
            const float v1 = img1 ? g1 / d1 : 0.f;
            // the error's g/y is the same quotient unless the guard changed y
            // (a branch, so that the second division runs only then)
            float q0 = v0, q1 = v1;
            if (d0 != y0) q0 = g0 / y0;
            if (d1 != y1) q1 = g1 / y1;
            if (img0) acc += err_term_q(y0, g0, q0, a.metric);
            if (img1) acc += err_term_q(y1, g1, q1, a.metric);
            w[r] = make_float2(v0, v1);
        }
        break;
    case XOP_RATIO_RL:
        if constexpr (FAM != XFAM_RATIO) break;
#pragma unroll
        for (int r = 0; r < RL; ++r) {
            const int c0 = 2 * (t + r * SL);
            const bool img0 = in_img_row && c0 < M;
            const bool img1 = in_img_row && c0 + 1 < M;
            const float y0 = w[r].x, y1 = w[r].y;
            const float2 gv = img0 ? *reinterpret_cast<const float2 *>(sx + c0) : make_float2(0.f, 0.f);
            const float g0 = gv.x, g1 = img1 ? gv.y : 0.f;
            // method_rl.c:46-67: r = g/y if y > 0 else bg on the image, 1e-6 elsewhere
            const float v0 = img0 ? (y0 > 0.f ? g0 / y0 : bg) : 1e-6f;
            const float v1 = img1 ? (y1 > 0.f ? g1 / y1 : bg) : 1e-6f;
            if (img0) acc += err_term_q(y0, g0, v0, a.metric);  // q used only when y > 0
            if (img1) acc += err_term_q(y1, g1, v1, a.metric);
            w[r] = make_float2(v0, v1);
        }
        break;
    case XOP_ERROR_ONLY:
        if constexpr (FAM != XFAM_RATIO) break;
#pragma unroll
        for (int r = 0; r < RL; ++r) {
            const int c0 = 2 * (t + r * SL);
            const bool img0 = in_img_row && c0 < M;
            const bool img1 = in_img_row && c0 + 1 < M;
            const float y0 = w[r].x, y1 = w[r].y;
            const float2 gv = img0 ? *reinterpret_cast<const float2 *>(sx + c0) : make_float2(0.f, 0.f);
            const float g0 = gv.x, g1 = img1 ? gv.y : 0.f;
            if (img0) acc += err_term_q(y0, g0, y0 > 0.f ? g0 / y0 : 0.f, a.metric);
            if (img1) acc += err_term_q(y1, g1, y1 > 0.f ? g1 / y1 : 0.f, a.metric);
        }
        break;
    case XOP_UPDATE_SHB:
        // method_shb.c:56-62 (x = Kt r * (p*W)), :366-376 (positivity), and the
        // next extrapolation :333-339; p_k is recomputed from x_k, x_{k-1}
        if constexpr (FAM != XFAM_UPDATE) break;
        // loads in groups ahead of the stores: the output may be x_{k-1}'s
        // own buffer, so the compiler moves no load across a store
#pragma unroll
        for (int r0 = 0; r0 < RL; r0 += XCH) {
            float2 xv[XCH], xq[XCH], ww[XCH];
#pragma unroll
            for (int i = 0; i < XCH; ++i) {
                if (r0 + i >= RL) break;
                const int c0 = 2 * (t + (r0 + i) * SL);
                xv[i] = *reinterpret_cast<const float2 *>(sx + c0);
                xq[i] = *reinterpret_cast<const float2 *>(sxp + c0);
                ww[i] = sw ? *reinterpret_cast<const float2 *>(sw + c0) : make_float2(1.f, 1.f);
            }
#pragma unroll
            for (int i = 0; i < XCH; ++i) {
                const int r = r0 + i;
                if (r >= RL) break;
                const int c0 = 2 * (t + r * SL);
                const float p0 = shb_p(xv[i].x, xq[i].x, a.alpha, bg);
                const float p1 = shb_p(xv[i].y, xq[i].y, a.alpha, bg);
                float n0 = w[r].x * (p0 * ww[i].x);
                float n1 = w[r].y * (p1 * ww[i].y);
                if (a.positivity) {
                    n0 = n0 < bg ? bg : n0;
                    n1 = n1 < bg ? bg : n1;
                }
                *reinterpret_cast<float2 *>(a.dst + rbase + c0) = make_float2(n0, n1);
                w[r] = make_float2(shb_p(n0, xv[i].x, a.alpha_next, bg), shb_p(n1, xv[i].y, a.alpha_next, bg));
            }
        }
        break;
    case XOP_UPDATE_RL:
        // method_rl.c:84-98 and :362-372
        if constexpr (FAM != XFAM_UPDATE) break;
#pragma unroll
        for (int r0 = 0; r0 < RL; r0 += XCH) {
            float2 xv[XCH], ww[XCH];
#pragma unroll
            for (int i = 0; i < XCH; ++i) {
                if (r0 + i >= RL) break;
                const int c0 = 2 * (t + (r0 + i) * SL);
                xv[i] = *reinterpret_cast<const float2 *>(sx + c0);
                ww[i] = sw ? *reinterpret_cast<const float2 *>(sw + c0) : make_float2(1.f, 1.f);
            }
#pragma unroll
            for (int i = 0; i < XCH; ++i) {
                const int r = r0 + i;
                if (r >= RL) break;
                const int c0 = 2 * (t + r * SL);
                float n0 = w[r].x * (xv[i].x * ww[i].x);
                float n1 = w[r].y * (xv[i].y * ww[i].y);
                if (a.rl_clamp && bg > 0.f) {
                    n0 = n0 < bg ? bg : n0;
                    n1 = n1 < bg ? bg : n1;
                }
                *reinterpret_cast<float2 *>(a.dst + rbase + c0) = make_float2(n0, n1);
                w[r] = make_float2(n0, n1);
            }
        }
        break;
    case XOP_WEIGHTS:
        // method_shb.c:224-234: W = 1/P1 where P1 > 0.01, else 0
        if constexpr (FAM != XFAM_STORE) break;
#pragma unroll
        for (int r = 0; r < RL; ++r) {
            const int c0 = 2 * (t + r * SL);
            const float q0 = w[r].x > 0.01f ? (float) (1.0 / (double) w[r].x) : 0.f;
            const float q1 = w[r].y > 0.01f ? (float) (1.0 / (double) w[r].y) : 0.f;
            *reinterpret_cast<float2 *>(a.dst + rbase + c0) = make_float2(q0, q1);
        }
        break;
    case XOP_STORE:
        if constexpr (FAM == XFAM_STORE) {
#pragma unroll
            for (int r = 0; r < RL; ++r) *reinterpret_cast<float2 *>(a.dst + rbase + 2 * (t + r * SL)) = w[r];
        }
        break;
    default:
        break;
    }
}

// The x transform of a real row of X = 2L samples is a complex transform of
// length L = RD::N, z[n] = x[2n] + i x[2n+1], and the row's half-spectrum is
// S[k] = E[k] + W_X^k O[k] with E and O made of Z[k] and Z[L-k].  The inverse
// runs the radices (RA, RB, RC), the forward the reversed list, so both meet
// the spectrum in a stage of radix RA, whose butterfly j holds the elements
// j + r*M, M = L/RA.  The mirror L-k of such an element is
// (M-j) + (RA-1-r)*M, an element of butterfly M-j: a thread that owns the
// butterflies j and M-j has both ends of every mirrored pair in registers.
// So the spectrum goes from global memory to registers and back once, and a
// pair's Hermitian arithmetic is done once for both of its elements; only the
// stages' own exchanges go through shared memory.  Butterfly 0 (and M/2, for
// even M) is its own mirror; the row's thread 0 owns both.
//
// A row is worked on by TP threads; in a stage of M butterflies thread t has
// the butterflies t, t + TP, ...  TP is a power of two up to 32 -- the row
// lies within a warp and needs no block barrier -- or a multiple of 32, where
// the row has a CTA to itself.
template <class RD, int TP>
struct XLine {
    static constexpr int L = RD::N;
    static constexpr int RA = RD::RA, RB = RD::RB, RL = RD::RL;
    static constexpr int M = L / RA;              // spectrum-side butterflies
    static constexpr int NP = (M + 1) / 2;        // mirrored pairs of them
    static constexpr int QP = (NP + TP - 1) / TP; // pairs per thread
    static constexpr int M2 = L / RB;             // middle stage (three stages)
    static constexpr int Q2 = (M2 + TP - 1) / TP;
    static constexpr int SL = L / RL;             // op-side butterflies
    static constexpr int QL = (SL + TP - 1) / TP;
    // complex values a thread holds at most
    static constexpr int HELD = cmax(2 * RA * QP, cmax(RD::THREE ? Q2 * RB : 0, QL * RL));
    // First exchange of a transform with first radix R: index i at i + i/R
    // for even R (its writes, R apart, then are an odd number of float2
    // apart).  Second exchange, after radices R and B: runs of R consecutive
    // butterflies write R consecutive elements, R*B apart; gap(R, B) elements
    // after each block of R*B (the fewest that do) keep the runs that a
    // half-warp writes at once on different banks.
    static constexpr bool apart(int r, int pitch)
    {
        unsigned seen = 0;
        for (int j = 0; j < 16; ++j) {
            const unsigned bit = 1u << ((j / r * pitch + j % r) % 16);
            if (seen & bit) return false;
            seen |= bit;
        }
        return true;
    }
    static constexpr int gap(int r, int b)
    {
        for (int g = 0; g < 16; ++g)
            if (apart(r, r * b + g)) return g;
        return 0;
    }
    static constexpr int room1(int r) { return L + (r % 2 == 0 ? L / r : 0); }
    static constexpr int room2(int r, int b) { return L + L / (r * b) * gap(r, b); }
    static constexpr int ROOM = cmax(cmax(room1(RA), room1(RL)),
                                     RD::THREE ? cmax(room2(RA, RB), room2(RL, RB)) : 0);
    // row pitch of an exchange tile (float2, even for 16-byte alignment);
    // where several rows share a half-warp's access, they start TP banks apart
    static constexpr int ROW_F2 = TP < 16 ? ROOM + ((TP - ROOM) % 16 + 16) % 16 : (ROOM + 1) / 2 * 2;
};

// real rows a family reads: forward: x, x_{k-1}; ratio: the image row;
// update: x, x_{k-1}, W; C2R-store: none
__host__ __device__ constexpr int x_real_rows(int fam)
{
    return fam == XFAM_FWD ? 2 : fam == XFAM_RATIO ? 1 : fam == XFAM_UPDATE ? 3 : 0;
}

template <class RD, int TP, int R, int FAM>
struct XCfg {
    using XL = XLine<RD, TP>;
    static constexpr int L = RD::N;
    static constexpr int X = 2 * L;
    static constexpr int NKB = (L + 1 + KB - 1) / KB;
    static constexpr int THREADS = R * TP;
    static constexpr size_t ROW_BYTES = sizeof(float2) * (size_t) XL::ROW_F2;
    // registers planned for a thread (two per value held, plus twiddles,
    // addresses and the op's operands), and the CTAs that leaves.  Most
    // kernels fit; a few spill 8 to 24 bytes, the ratio with a radix of 15 or
    // 16 on the op side 200 to 430.
    static constexpr int REGS = cmin(255, cmax(48, (2 * XL::HELD + 32 + 7) / 8 * 8));
    static constexpr int FIT_REGS = cmax(1, cmin(cmin(32, 2048 / THREADS), 65536 / (REGS * THREADS)));
    // two exchange tiles per row: consecutive exchanges alternate, so each
    // needs one barrier only
    static constexpr size_t RED_OFF = (size_t) R * ROW_BYTES * 2;
    static constexpr size_t SMEM_BYTES = RED_OFF + sizeof(double) * ((THREADS + 31) / 32);
    static constexpr int MIN_BLOCKS = cmax(1, cmin(FIT_REGS, (int) (227 * 1024 / (SMEM_BYTES + 1024))));
    static_assert(THREADS % 32 == 0, "the error reduction needs full warps");
    static_assert(TP % 32 == 0 || 32 % TP == 0, "a row lies within a warp or fills whole warps");
    static_assert(TP <= 32 || R == 1, "a row of several warps has the CTA to itself");
    static_assert(SMEM_BYTES <= 227 * 1024, "the exchange tiles fit shared memory");
};

// barrier of the threads of one row
template <int TP>
__device__ __forceinline__ void row_sync()
{
    if constexpr (TP <= 32)
        __syncwarp();
    else
        __syncthreads();
}

// stage twiddles applied, then the butterfly (CONJ: the conjugate twiddles)
template <int R, int DIR, bool CONJ = false>
__device__ __forceinline__ void x_butterfly(float2 *v, const float2 (&w)[R])
{
#pragma unroll
    for (int r = 1; r < R; ++r) v[r] = ((DIR < 0) != CONJ) ? cmul(v[r], w[r]) : cmulc(v[r], w[r]);
    Dft<R, DIR>::run(v);
}

// A stage's twiddles are the powers w^r, r < RS, of one root: every D-th is
// loaded from the table, the others are a loaded one times one of the first.
// Powers of a single value carry its rounding error r times, which is what
// bounds a transform's accuracy here (the wide radices are in stages that
// have twiddles): the table values halve or third the chain.  Short rows have
// few stages to average over and take more of them; their pass is latency
// bound, where the loads cost nothing.  C2R error in units of 2^-24, half
// lengths 375 / 420 / 1350: 3.9 / 4.4 / 5.5 with one value, 2.2 / 2.2 / 2.6
// with these (largest over the 176 lengths and both directions, relative to
// the square root of the transform's factors of two: 1.62 -> 0.86); x 2240
// update 2 to 4 % more (4.37 -> 4.45 ms, 4.20 -> 4.36 on another box), x 700
// 4 % (RL, 0.279 -> 0.290), whole deconvolutions 0 to 1 %.
template <int L, int RS>
struct XTw {
    static constexpr int D = L < 128 ? (RS <= 7 ? 2 : 4) : RS <= 4 ? RS : RS <= 10 ? (RS + 1) / 2 : (RS + 2) / 3;
    static constexpr int NB = 1 + (RS - 1) / D;  // table values: w, w^D, w^2D, ...
};

// The table values of a stage (radix RS after NS), for each of this thread's
// butterflies.  Loaded before the barrier in front of the stage: with most of
// shared memory in use the tables miss the L1 cache, and behind the barrier
// every warp of the row would wait for them.
template <int L, int NS, int RS, int TP, int Q>
__device__ __forceinline__ void x_bases(float2 (&b)[Q][XTw<L, RS>::NB], int t, const float2 *__restrict__ tw)
{
    constexpr int step = L / (NS * RS);
#pragma unroll
    for (int q = 0; q < Q; ++q) {
        const int j = t + q * TP;
        const int u = (j < L / RS ? j % NS : 0) * step;
        b[q][0] = __ldg(&tw[u]);
#pragma unroll
        for (int i = 1; i < XTw<L, RS>::NB; ++i) b[q][i] = __ldg(&tw[u * (i * XTw<L, RS>::D)]);
    }
}

// the twiddles from those values
template <int L, int RS>
__device__ __forceinline__ void x_twiddles(float2 (&w)[RS], const float2 (&b)[XTw<L, RS>::NB])
{
    constexpr int D = XTw<L, RS>::D;
    if constexpr (RS > 1) w[1] = b[0];
#pragma unroll
    for (int r = 2; r < RS; ++r)
        w[r] = r % D == 0 ? b[r / D]
             : r > D      ? cmul(w[r / D * D], w[r % D])
             : r % 2 == 0 ? cmul(w[r / 2], w[r / 2]) : cmul(w[r - 1], w[1]);
}

// middle stage (radix B after a first radix R1): first exchange in, second
// out; tb: x_bases of the stage
template <int L, int R1, int B, int DIR, int TP, int Q>
__device__ __forceinline__ void x_mid(const float2 *in, float2 *out, int t, const float2 (&tb)[Q][XTw<L, B>::NB], int gap)
{
    constexpr int M2 = L / B, PK = R1 % 2 == 0 ? 1 : 0;
#pragma unroll
    for (int q = 0; q < Q; ++q) {
        const int j = t + q * TP;
        if (j < M2) {
            float2 u[B], w[B];
            const int b = j + PK * (j / R1);
#pragma unroll
            for (int r = 0; r < B; ++r) u[r] = in[b + r * (M2 + PK * (M2 / R1))];
            x_twiddles<L, B>(w, tb[q]);
            x_butterfly<B, DIR>(u, w);
            float2 *o = out + (j / R1) * (R1 * B + gap) + j % R1;
#pragma unroll
            for (int r = 0; r < B; ++r) o[r * R1] = u[r];
        }
    }
}

template <class RD, int TP, int R, int FAM>
__global__ void __launch_bounds__(XCfg<RD, TP, R, FAM>::THREADS, XCfg<RD, TP, R, FAM>::MIN_BLOCKS)
k_xpass(XArgs a)
{
    using C = XCfg<RD, TP, R, FAM>;
    using XL = typename C::XL;
    constexpr int L = C::L, X = C::X;
    constexpr int RA = RD::RA, RB = RD::RB, RL = RD::RL, M = XL::M, SL = XL::SL, QL = XL::QL;
    constexpr bool EVEN = M % 2 == 0;  // butterfly M/2 exists
    constexpr bool c2r = FAM != XFAM_FWD;
    extern __shared__ __align__(128) unsigned char xsm[];
    const int t = threadIdx.x, row = threadIdx.y;
    const int op = a.op;
    const int z = blockIdx.y, y0 = blockIdx.x * R, yy = y0 + row;
    const bool row_ok = R == 1 || yy < a.Y;
    const long long plane = (long long) a.nkb * a.Y * KB;  // complex elements per z plane
    const int ks = a.Y * KB;                               // complex elements between kx blocks
    dep_wait();

    if constexpr (FAM == XFAM_RATIO) {
        // (with a periodic x, RL's constant row is not constant over the
        // transform length: such rows take the general path)
        if ((z >= a.P || y0 >= a.N) && !(a.wrapx && op == XOP_RATIO_RL)) {
            // No image row in this tile: the ratio is the same constant on
            // every row (0 for SHB, method_shb.c:44-46; 1e-6 for RL,
            // method_rl.c:62-64) and the rows add nothing to the error, so
            // neither transform is needed: the rows' spectra are c*X at kx = 0
            // and 0 elsewhere.
            const int tid = row * TP + t;
            if (tid == 0) a.partial[(long long) z * gridDim.x + blockIdx.x] = 0.0;
            if (a.r2c) {
                const float dc = (op == XOP_RATIO_RL) ? 1e-6f * (float) X : 0.f;
                float2 *Sz = a.S + (long long) z * plane + (long long) y0 * KB;
                for (int e = tid; e < C::NKB * R * KB; e += C::THREADS) {
                    const int ki = e % KB;
                    const int r2 = (e / KB) % R;
                    const int kb = e / (KB * R);
                    const int k = kb * KB + ki;
                    if (k > L || y0 + r2 >= a.Y) continue;
                    Sz[(long long) kb * ks + r2 * KB + ki] = make_float2(k == 0 ? dc : 0.f, 0.f);
                }
            }
            return;
        }
    }

    const float *psf_row = nullptr;
    if constexpr (FAM == XFAM_FWD) {
        if (op == XOP_FWD_PSF) {
            int sy = yy + a.peak[1], sz = z + a.peak[2];
            if (sy >= a.Y) sy -= a.Y;
            if (sz >= a.Z) sz -= a.Z;
            if (row_ok && sy < a.pN && sz < a.pP) psf_row = a.src + ((long long) sz * a.pN + sy) * a.pM;
            if (!__syncthreads_or(psf_row != nullptr)) {
                // no row of this tile holds any of the PSF
                if (row_ok) {
                    float2 *Sr = a.S + (long long) z * plane + (long long) yy * KB;
                    for (int k = t; k <= L; k += TP) Sr[(long long) (k >> 2) * ks + (k & 3)] = make_float2(0.f, 0.f);
                }
                return;
            }
        }
    }
    const bool rw = FAM == XFAM_UPDATE && a.Wt != nullptr;
    const bool in_img_row = yy < a.N && z < a.P;
    {
        // The rows a CTA starting a little later will read, into L2: without
        // it every row's first loads wait for HBM with little else resident
        // to run.  About 2 MB ahead (x 2240 update: 0.33 -> 0.29 ms per 32 Mi
        // spectrum elements; 10 MB ahead gains nothing, and beyond that it
        // evicts rows before they are used).
        constexpr int kRowBytes = 8 * L * ((c2r ? 1 : 0) + x_real_rows(FAM));
        const int lin = z * (int) gridDim.x + (int) blockIdx.x + cmax(1, (2 << 20) / (kRowBytes * R));
        const int z2 = lin / (int) gridDim.x, yy2 = (lin - z2 * (int) gridDim.x) * R + row;
        const bool img2 = z2 < a.P && yy2 < a.N;
        if (z2 < (int) gridDim.y && yy2 < a.Y && (FAM != XFAM_RATIO || img2)) {
            if constexpr (c2r) {
                const float2 *S2 = a.S + (long long) z2 * plane + (long long) yy2 * KB;
                for (int kb = t; kb < C::NKB; kb += TP) prefetch_l2(S2 + (long long) kb * ks);
            }
            if (t == 0) {
                const long long r2 = ((long long) z2 * a.Y + yy2) * a.X;
                const uint32_t rb = (uint32_t) (a.X * sizeof(float));
                if (op_reads_x(op) && a.bulk) prefetch_l2_bulk(a.src + r2, rb);
                if (op_reads_xp(op) && a.bulk) prefetch_l2_bulk(a.srcp + r2, rb);
                if (rw && a.bulk) prefetch_l2_bulk(a.Wt + r2, rb);
                if (FAM == XFAM_RATIO)
                    prefetch_l2_bulk(a.g + ((long long) z2 * a.N + yy2) * a.GP, (uint32_t) (a.GP * sizeof(float)));
            }
        }
    }
    // exchange tiles: the inverse's first is T0, and so on alternately
    float2 *T0 = reinterpret_cast<float2 *>(xsm) + (size_t) row * XL::ROW_F2;
    float2 *T1 = T0 + (size_t) R * XL::ROW_F2;
    float2 *Srow = a.S + (long long) z * plane + (long long) yy * KB;
    // offset of kx = k0 + r*M in the row's blocked spectrum, o0 that of k0
    auto koff = [&](int k) { return (k >> 2) * ks + (k & 3); };
    auto koff_r = [&](int k0, int o0, int r) { return M % 4 == 0 ? o0 + r * (M / 4) * ks : koff(k0 + r * M); };
    static_assert(KB == 4, "koff");
    double acc = 0.0;
    const float bg = a.sc->bg;

    float2 w[QL][RL];  // butterfly j = t + q*TP < SL: z[j + r*SL] = x[2n] + i x[2n+1]
#pragma unroll
    for (int q = 0; q < QL; ++q)
#pragma unroll
        for (int r = 0; r < RL; ++r) w[q][r] = make_float2(0.f, 0.f);

    if constexpr (c2r) {
        // Z[k] = s + i e with s = X[k] + X*[L-k], e = W_X^{-k} (X[k] - X*[L-k]);
        // the mirror's is Z[L-k] = conj(s - i e)
        auto herm = [](float2 xk, float2 xm, float2 tk, float2 &zk, float2 &zm) {
            xm.y = -xm.y;
            const float2 s = cadd(xk, xm), d = csub(xk, xm);
            const float2 e = cmulc(d, tk);
            zk = make_float2(s.x - e.y, s.y + e.x);
            zm = make_float2(s.x + e.y, e.x - s.y);
        };
        constexpr int PK = RA % 2 == 0 ? 1 : 0;
#pragma unroll
        for (int q = 0; q < XL::QP; ++q) {
            const int p = t + q * TP;
            if (p < XL::NP && row_ok) {
                const int j2 = p == 0 ? (EVEN ? M / 2 : 0) : M - p;
                const int o1 = koff(p), o2 = koff(j2);
                float2 v1[RA], v2[RA];
                const float2 tb = __ldg(&a.tw[p]);
#pragma unroll
                for (int r = 0; r < RA; ++r) {
                    v1[r] = Srow[koff_r(p, o1, r)];
                    v2[r] = Srow[koff_r(j2, o2, r)];
                }
                if (p != 0) {
                    // W_X^k for k = p + r*M: one table value, times
                    // compile-time factors W_X^{r*M}
                    static_for<RA>([&](auto rc) {
                        constexpr int r = decltype(rc)::value;
                        herm(v1[r], v2[RA - 1 - r], twiddle<2 * RA, r, -1>(tb), v1[r], v2[RA - 1 - r]);
                    });
                } else {
                    // Im X[0] and Im X[L] are ignored, as by any real inverse transform
                    const float x0 = v1[0].x, xl = Srow[koff(L)].x;
                    v1[0] = make_float2(x0 + xl, x0 - xl);
                    const float2 one = make_float2(1.f, 0.f);
                    float2 drop;
                    static_for<RA / 2>([&](auto rc) {
                        constexpr int r = decltype(rc)::value + 1;
                        if constexpr (2 * r == RA)
                            herm(v1[r], v1[r], twiddle<2 * RA, r, -1>(one), v1[r], drop);
                        else
                            herm(v1[r], v1[RA - r], twiddle<2 * RA, r, -1>(one), v1[r], v1[RA - r]);
                    });
                    if constexpr (EVEN)
                        static_for<(RA + 1) / 2>([&](auto rc) {
                            constexpr int r = decltype(rc)::value;
                            if constexpr (2 * r == RA - 1)
                                herm(v2[r], v2[r], twiddle<4 * RA, 2 * r + 1, -1>(one), v2[r], drop);
                            else
                                herm(v2[r], v2[RA - 1 - r], twiddle<4 * RA, 2 * r + 1, -1>(one), v2[r], v2[RA - 1 - r]);
                        });
                }
                Dft<RA, +1>::run(v1);
                Dft<RA, +1>::run(v2);
#pragma unroll
                for (int r = 0; r < RA; ++r) T0[p * (RA + PK) + r] = v1[r];
                if (EVEN || p != 0) {
#pragma unroll
                    for (int r = 0; r < RA; ++r) T0[j2 * (RA + PK) + r] = v2[r];
                }
            }
        }
        const float2 *in = T0;
        float2 tl[QL][XTw<L, RL>::NB];
        if constexpr (RD::THREE) {
            float2 tm[XL::Q2][XTw<L, RB>::NB];
            x_bases<L, RA, RB, TP>(tm, t, a.twL);
            row_sync<TP>();
            x_mid<L, RA, RB, +1, TP>(T0, T1, t, tm, XL::gap(RA, RB));
            in = T1;
        }
        x_bases<L, SL, RL, TP>(tl, t, a.twL);
        row_sync<TP>();
#pragma unroll
        for (int q = 0; q < QL; ++q) {
            const int j = t + q * TP;
            if (j < SL) {
                float2 tw[RL];
                x_twiddles<L, RL>(tw, tl[q]);
                if constexpr (RD::THREE) {
#pragma unroll
                    for (int r = 0; r < RL; ++r) w[q][r] = in[j + r * (SL + XL::gap(RA, RB))];
                } else {
                    const int b = j + PK * (j / RA);
#pragma unroll
                    for (int r = 0; r < RL; ++r) w[q][r] = in[b + r * (SL + PK * (SL / RA))];
                }
                x_butterfly<RL, +1>(w[q], tw);
            }
        }
    }

    // ---- pointwise op on x[2n], x[2n+1], n = j + r*SL
    if (row_ok) {
        const long long rbase = ((long long) z * a.Y + yy) * a.X;
#pragma unroll
        for (int q = 0; q < QL; ++q) {
            const int j = t + q * TP;
            if (j < SL)
                x_row_op<FAM, RL, SL>(a, op, j, rbase,
                                      FAM == XFAM_RATIO ? a.g + ((long long) z * a.N + yy) * a.GP
                                      : FAM == XFAM_FWD && op == XOP_FWD_PSF ? psf_row : a.src + rbase,
                                      a.srcp + rbase, rw ? a.Wt + rbase : nullptr, in_img_row, bg, w[q], acc);
        }
    }
    if constexpr (FAM == XFAM_STORE) return;

    double *red = reinterpret_cast<double *>(xsm + C::RED_OFF);
    if constexpr (FAM == XFAM_RATIO) {
        // deterministic reduction of the tile's error partial (fixed order):
        // lanes, then (at the end) warps
        for (int o = 16; o > 0; o >>= 1) acc += __shfl_down_sync(0xffffffffu, acc, o);
        const int tid = row * TP + t;
        if (tid % 32 == 0) red[tid / 32] = acc;
    }

    if (a.r2c) {
        // ---- forward with the reversed radix list; w is its first-stage input.
        // Its exchanges continue the alternation: two-stage transforms leave
        // T0 being read, three-stage ones T1.
        float2 *F0 = (!RD::THREE && c2r) ? T1 : T0;
        float2 *F1 = F0 == T0 ? T1 : T0;
        if (a.wrapx) {
            // periodic margins of the row (see XArgs), through shared memory
            row_sync<TP>();
            float *rowf = reinterpret_cast<float *>(T0);
#pragma unroll
            for (int q = 0; q < QL; ++q) {
                const int j = t + q * TP;
                if (j < SL) {
#pragma unroll
                    for (int r = 0; r < RL; ++r) reinterpret_cast<float2 *>(rowf)[j + r * SL] = w[q][r];
                }
            }
            row_sync<TP>();
#pragma unroll
            for (int q = 0; q < QL; ++q) {
                const int j = t + q * TP;
                if (j < SL) {
#pragma unroll
                    for (int r = 0; r < RL; ++r) {
                        float e[2];
#pragma unroll
                        for (int h = 0; h < 2; ++h) {
                            const int c = 2 * (j + r * SL) + h;
                            const int src = c < a.wM ? c
                                          : c < a.wM + a.hx ? c - a.wM
                                          : c >= X - a.hx ? c - X + a.wM : -1;
                            e[h] = src >= 0 ? rowf[src] : 0.f;
                        }
                        w[q][r] = make_float2(e[0], e[1]);
                    }
                }
            }
            row_sync<TP>();
        }
        constexpr int PK = RL % 2 == 0 ? 1 : 0;
#pragma unroll
        for (int q = 0; q < QL; ++q) {
            const int j = t + q * TP;
            if (j < SL) {
                Dft<RL, -1>::run(w[q]);
#pragma unroll
                for (int r = 0; r < RL; ++r) F0[j * (RL + PK) + r] = w[q][r];
            }
        }
        const float2 *in = F0;
        float2 tl[XL::QP][XTw<L, RA>::NB], tx[XL::QP];
        if constexpr (RD::THREE) {
            float2 tm[XL::Q2][XTw<L, RB>::NB];
            x_bases<L, RL, RB, TP>(tm, t, a.twL);
            row_sync<TP>();
            x_mid<L, RL, RB, -1, TP>(F0, F1, t, tm, XL::gap(RL, RB));
            in = F1;
        }
        x_bases<L, M, RA, TP>(tl, t, a.twL);
#pragma unroll
        for (int q = 0; q < XL::QP; ++q) tx[q] = __ldg(&a.tw[t + q * TP < XL::NP ? t + q * TP : 0]);
        row_sync<TP>();
        dep_start_next();
        // last stage: both butterflies of a mirrored pair.  Butterfly M-p's
        // twiddles are W_L^{r(M-p)} = conj(w_r) e^{-2 pi i r/RA} with w_r those
        // of butterfly p; the second factor shifts the outputs by one.
        auto at = [&](int j, int r) {
            if constexpr (RD::THREE) return j + r * (M + XL::gap(RL, RB));
            else return j + PK * (j / RL) + r * (M + PK * (M / RL));
        };
        // X[k] = s/2 + W_X^k o, X[L-k] = conj(s/2 - W_X^k o), with
        // s = Z[k] + Z*[L-k], o = -(i/2)(Z[k] - Z*[L-k]); hk = W_X^k / 2
        auto post = [](float2 zk, float2 zm, float2 hk, float2 &xk, float2 &xm) {
            zm.y = -zm.y;
            const float2 s = cadd(zk, zm), d = csub(zk, zm);
            const float2 o = cmul(make_float2(d.y, -d.x), hk);
            xk = make_float2(fmaf(0.5f, s.x, o.x), fmaf(0.5f, s.y, o.y));
            xm = make_float2(fmaf(0.5f, s.x, -o.x), -fmaf(0.5f, s.y, -o.y));
        };
#pragma unroll
        for (int q = 0; q < XL::QP; ++q) {
            const int p = t + q * TP;
            if (p < XL::NP && row_ok) {
                const int j2 = p == 0 ? (EVEN ? M / 2 : 0) : M - p;
                float2 v1[RA], v2[RA], tw[RA];
#pragma unroll
                for (int r = 0; r < RA; ++r) {
                    v1[r] = in[at(p, r)];
                    v2[r] = in[at(j2, r)];
                }
                x_twiddles<L, RA>(tw, tl[q]);
                x_butterfly<RA, -1>(v1, tw);
                if (p == 0) {
                    static_for<RA>([&](auto rc) {
                        constexpr int r = decltype(rc)::value;
                        tw[r] = twiddle<2 * RA, r, -1>(make_float2(1.f, 0.f));
                    });
                }
                x_butterfly<RA, -1, true>(v2, tw);  // Z[j2 + k*M] = v2[(k + 1) % RA]
                const int o1 = koff(p), o2 = koff(j2);
                if (p != 0) {
                    const float2 hb = make_float2(0.5f * tx[q].x, 0.5f * tx[q].y);
                    static_for<RA>([&](auto rc) {
                        constexpr int r = decltype(rc)::value;
                        float2 xk, xm;
                        post(v1[r], v2[(RA - r) % RA], twiddle<2 * RA, r, -1>(hb), xk, xm);
                        Srow[koff_r(p, o1, r)] = xk;
                        Srow[koff_r(j2, o2, RA - 1 - r)] = xm;
                    });
                } else {
                    const float2 half = make_float2(0.5f, 0.f);
                    static_for<RA / 2 + 1>([&](auto rc) {
                        constexpr int r = decltype(rc)::value;
                        float2 xk, xm;
                        post(v1[r], v1[(RA - r) % RA], twiddle<2 * RA, r, -1>(half), xk, xm);
                        Srow[koff(r * M)] = xk;
                        if constexpr (2 * r != RA) Srow[koff(L - r * M)] = xm;
                    });
                    if constexpr (EVEN)
                        static_for<(RA + 1) / 2>([&](auto rc) {
                            constexpr int r = decltype(rc)::value;
                            float2 xk, xm;
                            post(v2[(r + 1) % RA], v2[(RA - r) % RA], twiddle<4 * RA, 2 * r + 1, -1>(half), xk, xm);
                            Srow[koff(M / 2 + r * M)] = xk;
                            if constexpr (2 * r != RA - 1) Srow[koff(L - M / 2 - r * M)] = xm;
                        });
                }
            }
        }
    }
    if constexpr (FAM == XFAM_RATIO) {
        __syncthreads();
        if (t == 0 && row == 0) {
            double s2 = 0.0;
#pragma unroll 1
            for (int i = 0; i < C::THREADS / 32; ++i) s2 += red[i];
            a.partial[(long long) z * gridDim.x + blockIdx.x] = s2;
        }
    }
}

}  // namespace dwcu

// misc_kernels.cuh -- setup / bookkeeping kernels of a deconvolution job.
//
// All reductions run in a fixed order (fixed partition of the data over
// blocks, fixed order inside a block, one finishing block), so every result
// is bitwise reproducible from run to run and independent of scheduling.
#pragma once
#include <cuda_runtime.h>
#include <cstdint>
#include "xpass.cuh"

namespace dwcu {

constexpr int kRedThreads = 256;

struct StatsPartial {
    double sum;
    float mn;
    float mx;  // largest magnitude
    int nonfinite;
};

// Per-block min / double sum / non-finite count over the image rows
// [b*rpb, (b+1)*rpb) (fim_min fim.c:398-408, fim_sum fim.c:368-378).
__global__ void __launch_bounds__(kRedThreads)
k_stats_partial(const float *__restrict__ g, long long GP, int M, long long nrows, long long rpb,
                StatsPartial *__restrict__ part)
{
    __shared__ double ssum[kRedThreads];
    __shared__ float smin[kRedThreads], smax[kRedThreads];
    __shared__ int snf[kRedThreads];
    double s = 0.0;
    float mn = INFINITY, mx = 0.f;
    int nf = 0;
    const long long r0 = (long long) blockIdx.x * rpb;
    const long long r1 = min(nrows, r0 + rpb);
    for (long long r = r0; r < r1; ++r) {
        const float *row = g + r * GP;
        for (int c = threadIdx.x; c < M; c += kRedThreads) {
            float v = row[c];
            if (!isfinite(v)) nf++;
            s += (double) v;
            mn = fminf(mn, v);
            mx = fmaxf(mx, fabsf(v));
        }
    }
    ssum[threadIdx.x] = s;
    smin[threadIdx.x] = mn;
    smax[threadIdx.x] = mx;
    snf[threadIdx.x] = nf;
    __syncthreads();
    for (int o = kRedThreads / 2; o > 0; o >>= 1) {
        if (threadIdx.x < o) {
            ssum[threadIdx.x] += ssum[threadIdx.x + o];
            smin[threadIdx.x] = fminf(smin[threadIdx.x], smin[threadIdx.x + o]);
            smax[threadIdx.x] = fmaxf(smax[threadIdx.x], smax[threadIdx.x + o]);
            snf[threadIdx.x] += snf[threadIdx.x + o];
        }
        __syncthreads();
    }
    if (threadIdx.x == 0) part[blockIdx.x] = StatsPartial{ssum[0], smin[0], smax[0], snf[0]};
}

// Finish the statistics: bg (method_shb.c:108-117), start value
// sumg / wMNP (method_shb.c:255-268, with the job's logical voxel count).
__global__ void __launch_bounds__(kRedThreads)
k_stats_final(const StatsPartial *__restrict__ part, int nb, JobScalars *sc, int bg_auto, float bg_user,
              unsigned long long wmnp_logical)
{
    __shared__ double ssum[kRedThreads];
    __shared__ float smin[kRedThreads], smax[kRedThreads];
    __shared__ int snf[kRedThreads];
    double s = 0.0;
    float mn = INFINITY, mx = 0.f;
    int nf = 0;
    for (int i = threadIdx.x; i < nb; i += kRedThreads) {
        s += part[i].sum;
        mn = fminf(mn, part[i].mn);
        mx = fmaxf(mx, part[i].mx);
        nf += part[i].nonfinite;
    }
    ssum[threadIdx.x] = s;
    smin[threadIdx.x] = mn;
    smax[threadIdx.x] = mx;
    snf[threadIdx.x] = nf;
    __syncthreads();
    for (int o = kRedThreads / 2; o > 0; o >>= 1) {
        if (threadIdx.x < o) {
            ssum[threadIdx.x] += ssum[threadIdx.x + o];
            smin[threadIdx.x] = fminf(smin[threadIdx.x], smin[threadIdx.x + o]);
            smax[threadIdx.x] = fmaxf(smax[threadIdx.x], smax[threadIdx.x + o]);
            snf[threadIdx.x] += snf[threadIdx.x + o];
        }
        __syncthreads();
    }
    if (threadIdx.x == 0) {
        float gmin = smin[0];
        sc->gmin = gmin;
        sc->gmax = smax[0];
        sc->sumg = ssum[0];
        sc->bg = bg_auto ? (gmin < 1e-2f ? 1e-2f : gmin) : bg_user;
        const float sumg = (float) ssum[0];
        sc->x0 = sumg / (float) wmnp_logical;
        if (snf[0]) sc->flags |= 1;
    }
}

struct ArgmaxPartial {
    float v;
    long long i;
    double sum;
};
// where the PSF's first maximum lies: linear index, x, y, z
struct PsfPeak {
    long long i;
    int x, y, z;
};

// first maximum (lowest linear index), fim_argmax_max fim.c:269-332
__device__ __forceinline__ void amax_merge(float &v, long long &i, float v2, long long i2)
{
    if (v2 > v || (v2 == v && i2 < i)) {
        v = v2;
        i = i2;
    }
}

__global__ void __launch_bounds__(kRedThreads)
k_argmax_partial(const float *__restrict__ a, long long n, long long per_block, ArgmaxPartial *part, int *flags)
{
    __shared__ float sv[kRedThreads];
    __shared__ long long si[kRedThreads];
    __shared__ double ss[kRedThreads];
    float v = -INFINITY;
    long long idx = LLONG_MAX;
    double sum = 0.0;
    const long long b0 = (long long) blockIdx.x * per_block;
    const long long b1 = min(n, b0 + per_block);
    int nf = 0;
    for (long long k = b0 + threadIdx.x; k < b1; k += kRedThreads) {
        float x = a[k];
        if (!isfinite(x)) nf = 1;
        amax_merge(v, idx, x, k);
        sum += (double) x;
    }
    if (nf) atomicOr(flags, 2);
    sv[threadIdx.x] = v;
    si[threadIdx.x] = idx;
    ss[threadIdx.x] = sum;
    __syncthreads();
    for (int o = kRedThreads / 2; o > 0; o >>= 1) {
        if (threadIdx.x < o) {
            float v2 = sv[threadIdx.x + o];
            long long i2 = si[threadIdx.x + o];
            float v1 = sv[threadIdx.x];
            long long i1 = si[threadIdx.x];
            amax_merge(v1, i1, v2, i2);
            sv[threadIdx.x] = v1;
            si[threadIdx.x] = i1;
            ss[threadIdx.x] += ss[threadIdx.x + o];
        }
        __syncthreads();
    }
    if (threadIdx.x == 0) part[blockIdx.x] = ArgmaxPartial{sv[0], si[0], ss[0]};
}

// One block of kRedThreads: the peak and the PSF's sum (in double, fixed order).
__global__ void __launch_bounds__(kRedThreads)
k_argmax_final(const ArgmaxPartial *part, int nb, int pM, int pN, PsfPeak *out, JobScalars *sc)
{
    __shared__ float sv[kRedThreads];
    __shared__ long long si[kRedThreads];
    __shared__ double ss[kRedThreads];
    const int t = threadIdx.x;
    float v = -INFINITY;
    long long i = LLONG_MAX;
    double sum = 0.0;
    for (int b = t; b < nb; b += kRedThreads) {
        amax_merge(v, i, part[b].v, part[b].i);
        sum += part[b].sum;
    }
    sv[t] = v;
    si[t] = i;
    ss[t] = sum;
    __syncthreads();
    for (int o = kRedThreads / 2; o > 0; o >>= 1) {
        if (t < o) {
            float v1 = sv[t];
            long long i1 = si[t];
            amax_merge(v1, i1, sv[t + o], si[t + o]);
            sv[t] = v1;
            si[t] = i1;
            ss[t] += ss[t + o];
        }
        __syncthreads();
    }
    if (t == 0) {
        // (no maximum, every value NaN: any place inside the PSF will do, as
        // the x pass reads it from there before the set-up refuses it)
        const long long am = si[0] == LLONG_MAX ? 0 : si[0], r = am / pM;
        *out = PsfPeak{am, (int) (am % pM), (int) (r % pN), (int) (r / pN)};
        sc->psfsum = ss[0];
    }
}

// Place the PSF into a zeroed X x Y x Z volume so that its first maximum
// lands at the origin (fim_insert fim.c:585-623 followed by fim_circshift
// fim.c:982-1057 by minus the argmax), scaled by `scale` (the inverse
// transform normalisation 1/(X*Y*Z) is folded into the OTF here).  For PSFs
// larger than the job along an axis; others are read by the x pass as they
// lie (XOP_FWD_PSF).
__global__ void k_psf_embed(const float *__restrict__ psf, int pM, int pN, int pP, const PsfPeak *peak,
                            float *__restrict__ dst, int X, int Y, int Z, int XP, float scale)
{
    const long long n = (long long) pM * pN * pP;
    const int aa = peak->x, ab = peak->y, ac = peak->z;
    for (long long k = blockIdx.x * (long long) blockDim.x + threadIdx.x; k < n;
         k += (long long) gridDim.x * blockDim.x) {
        const int c = (int) (k / ((long long) pM * pN));
        const int b = (int) ((k - (long long) c * pM * pN) / pM);
        const int a = (int) (k - (long long) c * pM * pN - (long long) b * pM);
        int x = (a - aa) % X; if (x < 0) x += X;
        int y = (b - ab) % Y; if (y < 0) y += Y;
        int z = (c - ac) % Z; if (z < 0) z += Z;
        dst[((long long) z * Y + y) * XP + x] = psf[k] * scale;
    }
}

// the flat start: x_0, and x_{-1} = x_0 where there is one (n: a multiple of 4)
__global__ void k_fill_scalar(float *__restrict__ x, float *__restrict__ xp, long long n, const JobScalars *sc)
{
    const float v = sc->x0;
    const float4 v4 = make_float4(v, v, v, v);
    for (long long k = blockIdx.x * (long long) blockDim.x + threadIdx.x; k < n / 4;
         k += (long long) gridDim.x * blockDim.x) {
        reinterpret_cast<float4 *>(x)[k] = v4;
        if (xp) reinterpret_cast<float4 *>(xp)[k] = v4;
    }
}

// The first forward convolution of a flat start, as the inverse y pass would
// leave it on the image planes: K p of a constant p is the constant p times
// the PSF's sum (in double, rounded once), whose rows have a spectrum at
// kx = 0 only.  `clamp`: SHB's p_0 = max(x_0, bg).  Block z: plane blockIdx.z.
struct FlatArgs {
    float2 *S;
    const JobScalars *sc;
    int Y, nkb, clamp;
};
__global__ void k_flat_rows(FlatArgs a)
{
    dep_wait();
    const int h = blockIdx.x * blockDim.x + threadIdx.x;  // half of a row's kx block: 16 bytes
    if (h >= 2 * a.Y) return;
    float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
    if (blockIdx.y == 0 && h % 2 == 0) {
        const float x0 = a.sc->x0, bg = a.sc->bg;
        v.x = (float) ((double) (a.clamp && x0 < bg ? bg : x0) * a.sc->psfsum);
    }
    reinterpret_cast<float4 *>(a.S + ((long long) blockIdx.z * a.nkb + blockIdx.y) * a.Y * KB)[h] = v;
}

// image into the corner of a zeroed real volume (start_condition IDENTITY)
__global__ void k_embed_image(const float *__restrict__ g, long long GP, int M, int N, int P,
                              float *__restrict__ x, int X, int Y)
{
    const long long n = (long long) M * N * P;
    for (long long k = blockIdx.x * (long long) blockDim.x + threadIdx.x; k < n;
         k += (long long) gridDim.x * blockDim.x) {
        const int c = (int) (k / ((long long) M * N));
        const int b = (int) ((k - (long long) c * M * N) / M);
        const int a = (int) (k - (long long) c * M * N - (long long) b * M);
        x[((long long) c * Y + b) * X + a] = g[((long long) c * N + b) * GP + a];
    }
}

// One axis of fim_gsmooth (fim.c:2240-2278): each line convolved with the
// taps as fim_conv1_vector does it with normalized = 1 (fim.c:1944-2066):
// float products summed in double in tap order, the kernel renormalised by
// the sum of the taps that fall inside the line, one rounding to float.
// in and out are M x N x P, x fastest; axis 0, 1, 2 = x, y, z.
struct GaussTaps {
    float k[64];
    int n;
};
__global__ void k_gsmooth_axis(const float *__restrict__ in, float *__restrict__ out, int M, int N, int P, int axis,
                               GaussTaps K)
{
    const long long total = (long long) M * N * P;
    const int nV = axis == 0 ? M : axis == 1 ? N : P;
    const long long stride = axis == 0 ? 1 : axis == 1 ? (long long) M : (long long) M * N;
    const int nK = K.n, k2 = (nK - 1) / 2;
    for (long long e = blockIdx.x * (long long) blockDim.x + threadIdx.x; e < total;
         e += (long long) gridDim.x * blockDim.x) {
        const int a = (int) (e % M);
        const int b = (int) ((e / M) % N);
        const int c = (int) (e / ((long long) M * N));
        const int v = axis == 0 ? a : axis == 1 ? b : c;
        const float *line = in + (e - (long long) v * stride);  // element 0 of this line
        double acc = 0.0, kacc = 0.0;
        float r;
        if (nK > nV) {
            const int from = v > k2 ? v - k2 : 0;
            const int to = v + k2 + 1 > nV ? nV : v + k2 + 1;
            for (int l = from; l < to; ++l) {
                acc += (double) __fmul_rn(line[l * stride], K.k[l - v + k2]);
                kacc += (double) K.k[l - v + k2];
            }
            r = (float) (acc / kacc);
        } else if (v < k2) {
            for (int kk = k2 - v; kk < nK; ++kk) {
                acc += (double) __fmul_rn(K.k[kk], line[(v - k2 + kk) * stride]);
                kacc += (double) K.k[kk];
            }
            r = (float) (acc / kacc);
        } else if (v + k2 < nV) {
            for (int kk = 0; kk < nK; ++kk) acc += (double) __fmul_rn(K.k[kk], line[(v - k2 + kk) * stride]);
            r = (float) acc;
        } else {
            for (int kk = 0; kk < nV - v + k2; ++kk) {
                acc += (double) __fmul_rn(K.k[kk], line[(v - k2 + kk) * stride]);
                kacc += (double) K.k[kk];
            }
            r = (float) (acc / kacc);
        }
        out[e] = r;
    }
}

// Periodic y and/or z (bq 0/1 axes transformed at a larger length): after a
// forward x pass, every spectrum row (y, z) outside [0, wN) x [0, wP) takes
// a copy of the row it wraps to -- [w, w+h) from [0, h), [len-h, len) from
// [w-h, w) -- and the rows in between are cleared.  A launch covers the rows
// [y0, y0+ny) of the planes z0 + blockIdx.z, margins only; two threads per
// 4-wide kx block of a row.
struct WrapArgs {
    float2 *S;
    int Y, Z, nkb, wN, hy, wrapy, wP, hz, wrapz;
    int y0, ny, z0;
};
__global__ void k_wrap_rows(WrapArgs a)
{
    dep_wait();
    const int h = blockIdx.x * blockDim.x + threadIdx.x;  // half of a row's kx block: 16 bytes
    if (h >= 2 * a.ny) return;
    const int y = a.y0 + h / 2, kb = blockIdx.y, z = a.z0 + (int) blockIdx.z;
    auto src = [](int v, int w, int h, int len) { return v < w ? v : v < w + h ? v - w : v >= len - h ? v - len + w : -1; };
    const int ys = a.wrapy ? src(y, a.wN, a.hy, a.Y) : y;
    const int zs = a.wrapz ? src(z, a.wP, a.hz, a.Z) : z;
    auto at = [&](int zz, int yy) {
        return reinterpret_cast<float4 *>(a.S + (((long long) zz * a.nkb + kb) * a.Y + yy) * KB) + h % 2;
    };
    *at(z, y) = ys < 0 || zs < 0 ? make_float4(0.f, 0.f, 0.f, 0.f) : *at(zs, ys);
}

// fim_subregion (fim.c:695-718): the image-sized corner of a job volume
__global__ void k_crop(const float *__restrict__ x, int X, int Y, int M, int N, int P, float *__restrict__ out)
{
    const long long n = (long long) M * N * P;
    for (long long k = blockIdx.x * (long long) blockDim.x + threadIdx.x; k < n;
         k += (long long) gridDim.x * blockDim.x) {
        const int c = (int) (k / ((long long) M * N));
        const int b = (int) ((k - (long long) c * M * N) / M);
        const int a = (int) (k - (long long) c * M * N - (long long) b * M);
        out[k] = x[((long long) c * Y + b) * X + a];
    }
}

// finish one iteration's error: mean over the image of the x-pass partials
// (get_fIdiv dw.c:1492-1524 / get_fMSE dw.c:1461-1490)
__global__ void __launch_bounds__(kErrLanes) k_err_final(ErrSum e)
{
    __shared__ double s[kErrLanes];
    dep_wait();
    err_store(e, s, threadIdx.x, kErrLanes);
}

}  // namespace dwcu

// Projection preprocessing kernels: flat/dark averages and log-normalisation
// (tomography/fits_to_hpc.F90:183-244), the 0/180-degree pick
// (projections_to_sinogram_hpc.F90:141-224), rotation-axis registration
// (:231-364, plus a cross-correlation variant), the 27-point median (:426-452),
// the bilinear resample (:456-470) and the transpose to slice-major sinograms
// (:481-487).
//
// Arithmetic that decides an index or a comparison is written with explicit
// round-to-nearest operations so that it matches the single-precision
// reference operation for operation.
#include <algorithm>
#include <climits>
#include <cmath>

#include "../../include/acumen_gpu.h"
#include "common.cuh"
#include "prep.h"

namespace acu {

template <typename Tin>
__device__ __forceinline__ float to_f(Tin v) { return (float)v; }

// ---- frame averages (fits_to_hpc.F90:183-210): running sum in frame order ----
template <typename Tin>
__global__ void k_frame_average(int nframes, long npix, const Tin* __restrict__ frames, float* __restrict__ out)
{
    for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < npix; i += (long)gridDim.x * blockDim.x) {
        float s = 0.0f;
        for (int j = 0; j < nframes; ++j) s = __fadd_rn(s, to_f(frames[(size_t)j * npix + i]));
        out[i] = __fdiv_rn(s, (float)nframes);
    }
}

// ---- log-normalisation (fits_to_hpc.F90:243 mode 0, :244 mode 1) ------------
template <typename Tin>
__global__ void k_normalize(int mode, long npix, long total, const Tin* __restrict__ raw, const float* __restrict__ ob,
                            const float* __restrict__ df, float* __restrict__ out)
{
    for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < total; i += (long)gridDim.x * blockDim.x) {
        const long k = i % npix;
        const float I = to_f(raw[i]);
        float v;
        if (mode == 0) {
            v = -logf(__fdiv_rn(I, fmaxf(ob[k], 1.0f)));
        } else {
            const float d = df[k];
            v = -logf(__fdiv_rn(fmaxf(__fsub_rn(I, d), 1e-16f), fmaxf(__fsub_rn(ob[k], d), 1.0f)));
        }
        out[i] = v;
    }
}

// Vectorised form for frames of a multiple of 8 pixels with 16-byte aligned
// arrays: one thread normalises 8 consecutive pixels of one projection (a
// 16-byte load of uint16 counts or two of floats, two 16-byte loads of each
// flat/dark average, two 16-byte stores); grid.y walks the projections, so no
// 64-bit division is needed.  Same arithmetic per pixel as k_normalize.
__device__ __forceinline__ void load8(const uint16_t* p, float (&v)[8])
{
    const uint4 u = __ldg(reinterpret_cast<const uint4*>(p));
    const unsigned w[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        v[2 * i] = (float)(w[i] & 0xffffu);
        v[2 * i + 1] = (float)(w[i] >> 16);
    }
}
__device__ __forceinline__ void load8(const float* p, float (&v)[8])
{
    const float4 a = __ldg(reinterpret_cast<const float4*>(p)), b = __ldg(reinterpret_cast<const float4*>(p) + 1);
    v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w;
    v[4] = b.x; v[5] = b.y; v[6] = b.z; v[7] = b.w;
}

template <typename Tin>
__global__ void __launch_bounds__(256) k_normalize8(int mode, int nproj, long nvec, const Tin* __restrict__ raw,
                                                    const float* __restrict__ ob, const float* __restrict__ df,
                                                    float* __restrict__ out)
{
    for (int p = blockIdx.y; p < nproj; p += gridDim.y) {
        const Tin* rp = raw + (size_t)p * nvec * 8;
        float* op = out + (size_t)p * nvec * 8;
        for (long v = blockIdx.x * (long)blockDim.x + threadIdx.x; v < nvec; v += (long)gridDim.x * blockDim.x) {
            float I[8], o[8], d[8];
            load8(rp + v * 8, I);
            load8(ob + v * 8, o);
            if (mode == 0) {
#pragma unroll
                for (int i = 0; i < 8; ++i) I[i] = -logf(__fdiv_rn(I[i], fmaxf(o[i], 1.0f)));
            } else {
                load8(df + v * 8, d);
#pragma unroll
                for (int i = 0; i < 8; ++i)
                    I[i] = -logf(__fdiv_rn(fmaxf(__fsub_rn(I[i], d[i]), 1e-16f), fmaxf(__fsub_rn(o[i], d[i]), 1.0f)));
            }
            float4* q = reinterpret_cast<float4*>(op + v * 8);
            q[0] = make_float4(I[0], I[1], I[2], I[3]);
            q[1] = make_float4(I[4], I[5], I[6], I[7]);
        }
    }
}

// ---- lerp between two projections (projections_to_sinogram_hpc.F90:162) ------
__global__ void k_lerp(long n, const float* __restrict__ a, const float* __restrict__ b, float ta, float tb,
                       float target, float* __restrict__ out)
{
    for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < n; i += (long)gridDim.x * blockDim.x)
        out[i] = __fadd_rn(__fdiv_rn(__fmul_rn(__fsub_rn(target, ta), __fsub_rn(b[i], a[i])), __fsub_rn(tb, ta)),
                           a[i]);
}

// ---- bilinear resample with the reference's clamps (:456-470) ---------------
struct ResampleGeom {
    int ndet, nrows, add;
    float cth, sth, shift;
};

// The taps of one resampled pixel: where, and their weights.
struct Taps {
    size_t a, b, c, d;
    float wxl, wxh, wyl, wyh;
};

__device__ __forceinline__ Taps resample_taps(const ResampleGeom& g, int jx, int jy)
{
    const float mx = __fdiv_rn((float)(g.ndet + g.add - 1), 2.0f);
    const float my = __fdiv_rn((float)(g.nrows - 1), 2.0f);
    const float ss = (float)g.ndet;
    const float ax = __fsub_rn(__fsub_rn((float)jx, mx), __fmul_rn(ss, g.shift));
    const float ay = __fsub_rn((float)jy, my);
    float xr = __fadd_rn(__fsub_rn(__fmul_rn(g.cth, ax), __fmul_rn(g.sth, ay)), mx);
    float yr = __fadd_rn(__fadd_rn(__fmul_rn(g.sth, ax), __fmul_rn(g.cth, ay)), my);
    xr = fminf(fmaxf(xr, 1.0f), (float)g.ndet);
    yr = fminf(fmaxf(yr, 1.0f), (float)g.nrows);
    int y1 = min(max((int)floorf(yr), 1), g.nrows);
    int y2 = min(max(y1 + 1, 1), g.nrows);
    int x1 = min(max((int)floorf(xr), 1), g.ndet);
    int x2 = min(max(x1 + 1, 1), g.ndet);
    Taps t;
    t.wxl = __fsub_rn((float)x2, xr);
    t.wxh = __fsub_rn(xr, (float)x1);
    t.wyl = __fsub_rn((float)y2, yr);
    t.wyh = __fsub_rn(yr, (float)y1);
    const size_t r1 = (size_t)(y1 - 1) * g.ndet, r2 = (size_t)(y2 - 1) * g.ndet;
    t.a = r1 + x1 - 1;
    t.b = r1 + x2 - 1;
    t.c = r2 + x1 - 1;
    t.d = r2 + x2 - 1;
    return t;
}

__device__ __forceinline__ float resample_with(const Taps& t, const float* __restrict__ src)
{
    float acc = __fmul_rn(__fmul_rn(src[t.a], t.wxl), t.wyl);
    acc = __fadd_rn(acc, __fmul_rn(__fmul_rn(src[t.b], t.wxh), t.wyl));
    acc = __fadd_rn(acc, __fmul_rn(__fmul_rn(src[t.c], t.wxl), t.wyh));
    return __fadd_rn(acc, __fmul_rn(__fmul_rn(src[t.d], t.wxh), t.wyh));
}

__device__ __forceinline__ float resample_at(const ResampleGeom& g, const float* __restrict__ src, int jx, int jy)
{
    return resample_with(resample_taps(g, jx, jy), src);
}

__global__ void k_resample(ResampleGeom g, const float* __restrict__ src, float* __restrict__ out)
{
    const int nx = g.ndet + g.add;
    const long n = (long)nx * g.nrows;
    for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < n; i += (long)gridDim.x * blockDim.x) {
        const int jx = (int)(i % nx) + 1, jy = (int)(i / nx) + 1;
        out[i] = resample_at(g, src, jx, jy);
    }
}

// ---- registration objective (:279-284 / :308-313 / :346-351) ----------------
// sum |V0(jx,jy) - V180(nx-jx+1,jy)| over the padded grid for up to MIRROR_MAX
// candidates (grid.y): one FP64 partial per block, summed in block order
// (deterministic) by the candidate's last block, into host memory.  An evaluation is
// bound by its latency: one launch and a synchronisation per candidate sweep in place of two
// launches, a copy and a synchronisation per candidate, and no 64-bit division per
// pixel, take a search at 1025 x 64 from 27 to 5 us per candidate.
__global__ void __launch_bounds__(256) k_mirror_errors(int ndet, int nrows, MirrorCandidates cand,
                                                       const float* __restrict__ p0, const float* __restrict__ p180,
                                                       double* __restrict__ part, unsigned* __restrict__ done,
                                                       double* __restrict__ out)
{
    __shared__ double sh[32];
    __shared__ bool last;
    const int k = blockIdx.y, nblk = gridDim.x;
    const ResampleGeom g{ndet, nrows, ndet % 2 == 0 ? 1 : 0, cand.cth[k], cand.sth[k], cand.shift[k]};
    const int nx = g.ndet + g.add;
    const long n = (long)nx * g.nrows, first = blockIdx.x * 256l + threadIdx.x;
    const int stride = nblk * 256, dx = stride % nx, dy = stride / nx;
    int jx = (int)(first % nx) + 1, jy = (int)(first / nx) + 1;
    double acc = 0.0;
    for (long i = first; i < n; i += stride) {
        const float a = resample_at(g, p0, jx, jy);
        const float b = resample_at(g, p180, nx - jx + 1, jy);
        acc += (double)fabsf(__fsub_rn(a, b));
        jx += dx;
        jy += dy;
        if (jx > nx) {
            jx -= nx;
            ++jy;
        }
    }
    double r = block_sum(acc, sh);
    if (threadIdx.x == 0) {
        part[k * nblk + blockIdx.x] = r;
        __threadfence();
        last = atomicAdd(done + k, 1u) == nblk - 1;
    }
    __syncthreads();
    if (!last) return;
    __threadfence();
    acc = 0.0;
    for (int i = threadIdx.x; i < nblk; i += 256) acc += __ldcg(part + k * nblk + i);
    r = block_sum(acc, sh);
    if (threadIdx.x == 0) {
        done[k] = 0;
        out[k] = r;
    }
}

// centre-of-mass sums (:234-243): tm, cmx_0, cmx_180 as FP64 partials
__global__ void __launch_bounds__(256) k_com(int ndet, int nrows, int add, const float* __restrict__ p0,
                                             const float* __restrict__ p180, double* __restrict__ part)
{
    __shared__ double sh[32];
    double tm = 0.0, c0 = 0.0, c1 = 0.0;
    const long n = (long)ndet * nrows;
    const float nda = (float)(ndet + add);
    for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < n; i += (long)gridDim.x * blockDim.x) {
        const int jx = (int)(i % ndet) + 1;
        const float a = p0[i], b = p180[i];
        const float w = __fsub_rn(__fsub_rn(__fdiv_rn(__fmul_rn(__fmul_rn(2.0f, nda), (float)(jx - 1)),
                                                      (float)(ndet + add - 1)),
                                            (float)ndet),
                                  (float)add);
        tm += (double)a + (double)b;
        c0 += (double)__fmul_rn(a, w);
        c1 += (double)__fmul_rn(b, w);
    }
    double r = block_sum(tm, sh);
    if (threadIdx.x == 0) part[3 * blockIdx.x] = r;
    r = block_sum(c0, sh);
    if (threadIdx.x == 0) part[3 * blockIdx.x + 1] = r;
    r = block_sum(c1, sh);
    if (threadIdx.x == 0) part[3 * blockIdx.x + 2] = r;
}

// fixed-order sums of n interleaved partials, one per block, into out[block]
__global__ void k_sum_partials(const double* __restrict__ part, int n, double* __restrict__ out)
{
    __shared__ double sh[32];
    double v = 0.0;
    for (int i = threadIdx.x; i < n; i += blockDim.x) v += part[(size_t)i * gridDim.x + blockIdx.x];
    const double r = block_sum(v, sh);
    if (threadIdx.x == 0) out[blockIdx.x] = r;
}

// ---- cross-correlation registration (new) --------------------------------------
// C(k) = sum_{x,y} p0(x,y) * p180(ndet-1-x+k, y) with every product truncated
// to 2^-32 fixed point and summed exactly in 128-bit integers: integer sums do
// not depend on their order, so the argmax is bit-exact against the CPU oracle,
// and a 128-bit sum of n terms below 2^63 cannot wrap for n < 2^64.  A product
// that is not finite or not below 2^31 in magnitude (its fixed-point value would
// not fit 64 bits) sets the range flag and is left out; the host then rejects
// the input.  Every element of p0 and p180 meets a partner at k = 0, so every
// element is checked.
//
// Scratch layout (unsigned 64-bit words): lag i's sum at [2i] (low word) and
// [2i+1] (high word, two's complement), then one word holding the argmax
// index (low 32 bits) and the range flag (high 32 bits).
constexpr double kFixScale = 4294967296.0;     // 2^32
constexpr double kFixLimit = 2147483648.0;     // |product| < 2^31

// 128-bit atomic add from two 64-bit atomics: the low words add modulo 2^64
// and each addition that wraps carries one into the high word, so the pair
// holds the exact sum modulo 2^128 whatever the order of the additions.
__device__ __forceinline__ void atomic_add_i128(unsigned long long* w, __int128 v)
{
    const unsigned long long lo = (unsigned long long)v, hi = (unsigned long long)(v >> 64);
    const unsigned long long old = atomicAdd(w, lo);
    const unsigned long long carry = (old + lo < old) ? 1ull : 0ull;
    if (hi + carry) atomicAdd(w + 1, hi + carry);
}

__device__ __forceinline__ __int128 shfl_down_i128(__int128 v, int o)
{
    const unsigned long long lo = __shfl_down_sync(0xffffffffu, (unsigned long long)v, o);
    const long long hi = __shfl_down_sync(0xffffffffu, (long long)(v >> 64), o);
    return ((__int128)hi << 64) | (__int128)lo;
}

// A block takes XC_LAGS lags and, one by one, its share of the frame's items (a
// row's stretch of XC_X pixels).  In integers, a product is the 48-bit product of
// two mantissas shifted right by what both exponents say, which is its floor at
// 2^-32: six instructions.  (In FP64, of which an SM does two a clock, with the
// conversion to 64 bits, 2048 x 256 pixels and 1025 lags took 5.24 ms; so: 0.24 ms,
// with products of 2^14 and more 0.5 ms.)
// Both operands are staged as (mantissa * 2^7, 14 - exponent), a product of two
// is shifted right by the sum of the second parts; a thread takes 8 pixels x 8 lags from
// 8 + 15 of them, read at a pitch of 9 per 8, so that neither 8-element stride meets a
// bank twice.  An item's largest magnitudes say how: below 2^14 its floors add up in 64
// bits; below 2^31 the shift may go left by up to two, and high and low words add
// up apart; else, or with a value that is not finite, product by product in FP64.
constexpr int XC_X = 1024, XC_LAGS = 64, XC_ITEMS = 256;   // XC_ITEMS: items a block sums up in 64 bits at most
constexpr int XC_Q = XC_X + XC_LAGS;

__device__ __forceinline__ int xc_slot(int i) { return i + (i >> 3); }
__device__ __forceinline__ int2 xc_split(float v, unsigned& top)
{
    const unsigned b = __float_as_uint(v);
    const int e = (int)(b >> 23 & 255u);
    top = max(top, b & 0x7fffffffu);
    const int m = (int)((b & 0x7fffffu) << 7 | (e ? 0x40000000u : 0u));
    return make_int2((int)b < 0 ? -m : m, 14 + 127 - max(e, 1));
}
// v >> n, n = 0..; 63 and more leave the sign
__device__ __forceinline__ long long shr_floor(long long v, int n)
{
    long long r;
    asm("shr.s64 %0, %1, %2;" : "=l"(r) : "l"(v), "r"(n));
    return r;
}

// what(j, product of the mantissas, shift) for a thread's pixels and its lags lg * 8 + j (n: pixels in the stretch)
template <class F>
__device__ __forceinline__ void xc_products(const int2* s_a, const int2* s_q, int xg, int lg, int n, F&& what)
{
#pragma unroll 1
    for (int x8 = xg; x8 < XC_X / 8 && x8 * 8 < n; x8 += 32) {
        const int2* pa = s_a + x8 * 9;
        const int2* pq = s_q + (x8 - lg + XC_LAGS / 8) * 9;   // q of the first pixel at the first lag
        int2 b[15];
#pragma unroll
        for (int j = 0; j < 15; ++j) b[j] = pq[j < 7 ? j - 8 : j - 7];   // pixel - lag = j - 7
#pragma unroll
        for (int x = 0; x < 8; ++x) {
            const int2 v = pa[x];
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                const int2 u = b[x - j + 7];
                what(j, (long long)v.x * u.x, v.y + u.y);
            }
        }
    }
}

// adds the sums of the four lanes with the same lags to the warp's
__device__ __forceinline__ void xc_gather(__int128 v, __int128* sum, int lag)
{
    v += shfl_down_i128(v, 16);
    v += shfl_down_i128(v, 8);
    if ((threadIdx.x & 31) < 8) sum[lag] += v;
}

__global__ void __launch_bounds__(256, 2) k_xcorr(int ndet, int nrows, int kmax, const float* __restrict__ p0,
                                               const float* __restrict__ p180, unsigned long long* __restrict__ w)
{
    __shared__ int2 s_a[XC_X * 9 / 8], s_q[XC_Q * 9 / 8];
    __shared__ unsigned s_top[2][2];
    __shared__ __int128 s_sum[8][XC_LAGS];
    const int tid = threadIdx.x, lg = tid & 7, xg = tid >> 3;
    const int nk = 2 * kmax + 1, i0 = blockIdx.y * XC_LAGS;
    const int nxt = (ndet + XC_X - 1) / XC_X, items = nxt * nrows;
    long long acc[8];
    bool bad = false;
#pragma unroll
    for (int j = 0; j < 8; ++j) acc[j] = 0;
    if (tid < 4) s_top[tid >> 1][tid & 1] = 0u;
    for (int i = tid; i < 8 * XC_LAGS; i += 256) s_sum[i / XC_LAGS][i % XC_LAGS] = 0;
    __syncthreads();
    int buf = 0;
    for (int it = blockIdx.x; it < items; it += gridDim.x) {
        const int y = it / nxt, xt = it % nxt * XC_X;
        // C(k) = sum_x p0(x) q(x - k), q(z) = p180(ndet - 1 - z); place of q(z): z - z0
        const int z0 = xt - i0 - XC_LAGS + kmax;
        if (z0 >= ndet || z0 + XC_Q <= 0) continue;   // no partner for any of its pixels
        const float* a = p0 + (size_t)y * ndet;
        const float* q = p180 + (size_t)y * ndet;
        unsigned ta = 0u, tq = 0u;
        for (int i = tid; i < XC_X; i += 256)
            s_a[xc_slot(i)] = xc_split(xt + i < ndet ? __ldg(a + xt + i) : 0.f, ta);
        for (int i = tid; i < XC_Q; i += 256) {
            const int z = z0 + i;
            s_q[xc_slot(i)] = xc_split(z >= 0 && z < ndet ? __ldg(q + ndet - 1 - z) : 0.f, tq);
        }
        ta = __reduce_max_sync(0xffffffffu, ta);
        tq = __reduce_max_sync(0xffffffffu, tq);
        if ((tid & 31) == 0) {
            atomicMax(&s_top[buf][0], ta);
            atomicMax(&s_top[buf][1], tq);
        }
        __syncthreads();
        const double top = (double)__uint_as_float(s_top[buf][0]) * (double)__uint_as_float(s_top[buf][1]);
        const bool finite = max(s_top[buf][0], s_top[buf][1]) < 0x7f800000u;
        if (tid < 2) s_top[buf ^ 1][tid] = 0u;
        buf ^= 1;
        if (finite && top < 16384.) {
            xc_products(s_a, s_q, xg, lg, ndet - xt, [&](int j, long long m, int n) { acc[j] += shr_floor(m, n); });
        } else if (finite && top < kFixLimit) {
            long long hi[8];
            unsigned long long lo[8];
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                hi[j] = 0;
                lo[j] = 0;
            }
            xc_products(s_a, s_q, xg, lg, ndet - xt, [&](int j, long long m, int n) {
                const long long t = shr_floor(m, max(n, 0)) << max(-n, 0);
                hi[j] += t >> 32;
                lo[j] += (unsigned)t;
            });
#pragma unroll
            for (int j = 0; j < 8; ++j) xc_gather(((__int128)hi[j] << 32) + lo[j], s_sum[tid >> 5], lg * 8 + j);
        } else {
#pragma unroll 1
            for (int j = 0; j < 8; ++j) {
                const int i = i0 + lg * 8 + j;
                __int128 v = 0;
                if (i < nk)
#pragma unroll 1
                    for (int x = xt + xg; x < min(xt + XC_X, ndet); x += 32) {
                        const int z = x - (i - kmax);
                        if (z < 0 || z >= ndet) continue;
                        const double p = (double)a[x] * (double)q[ndet - 1 - z];   // exact
                        if (fabs(p) < kFixLimit) v += (__int128)__double2ll_rd(p * kFixScale);
                        else bad = true;                                            // also NaN
                    }
                __syncwarp();
                xc_gather(v, s_sum[tid >> 5], lg * 8 + j);
            }
        }
        __syncthreads();
    }
#pragma unroll
    for (int j = 0; j < 8; ++j) xc_gather(acc[j], s_sum[tid >> 5], lg * 8 + j);
    __syncthreads();
    if (tid < XC_LAGS && i0 + tid < nk) {
        __int128 v = 0;
#pragma unroll
        for (int k = 0; k < 8; ++k) v += s_sum[k][tid];
        if (v != 0) atomic_add_i128(&w[2 * (i0 + tid)], v);
    }
    if (__any_sync(0xffffffffu, bad) && (tid & 31) == 0) {
        unsigned int* flag = reinterpret_cast<unsigned int*>(w + 2 * nk) + 1;
        atomicOr(flag, 1u);
    }
}

__device__ __forceinline__ bool i128_better(long long ah, unsigned long long al, int ai, long long bh,
                                            unsigned long long bl, int bi)
{
    if (ah != bh) return ah > bh;
    if (al != bl) return al > bl;
    return ai < bi;
}

// Argmax over the nk 128-bit correlation values (ties: lowest index), one block of 256.
__global__ void k_argmax(int nk, unsigned long long* __restrict__ w)
{
    long long bh = LLONG_MIN;
    unsigned long long bl = 0;
    int bi = 0x7fffffff;
    for (int i = threadIdx.x; i < nk; i += 256) {
        const long long h = (long long)w[2 * i + 1];
        const unsigned long long l = w[2 * i];
        if (i128_better(h, l, i, bh, bl, bi)) { bh = h; bl = l; bi = i; }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const long long oh = __shfl_down_sync(0xffffffffu, bh, o);
        const unsigned long long ol = __shfl_down_sync(0xffffffffu, bl, o);
        const int oi = __shfl_down_sync(0xffffffffu, bi, o);
        if (i128_better(oh, ol, oi, bh, bl, bi)) { bh = oh; bl = ol; bi = oi; }
    }
    __shared__ long long s_h[8];
    __shared__ unsigned long long s_l[8];
    __shared__ int s_i[8];
    if ((threadIdx.x & 31) == 0) {
        s_h[threadIdx.x >> 5] = bh;
        s_l[threadIdx.x >> 5] = bl;
        s_i[threadIdx.x >> 5] = bi;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int k = 1; k < 8; ++k)
            if (i128_better(s_h[k], s_l[k], s_i[k], bh, bl, bi)) { bh = s_h[k]; bl = s_l[k]; bi = s_i[k]; }
        reinterpret_cast<int*>(w + 2 * nk)[0] = bi;
    }
}

// ---- 27-point median (:426-452): the reference's descending exchange sort,
// passes 1..14 (the later passes do not touch element 14), with the
// intended slots 1..27 ------------------------------------------------------------
// Without a NaN, and unless it is a zero (of either sign), any selection of the
// 14th largest returns the same bits: equal floats that are not zero, infinities too,
// are bitwise equal.  With a NaN (whose comparisons are false) among the 27, or a zero
// as the result, the exchange sort itself decides, bit for bit.
//
// The cheaper selection: a thread walks the projections at R pixels, one above
// the other.  Per projection it sorts the R + 2 rows of three values that
// their 3 x 3 neighbourhoods are made of (3 comparisons each), and from these each
// pixel's nine (16 more: the rest of Floyd's network of 25), which serve three
// projections.  Of three sorted lists of nine, the minima, medians and maxima of
// the values of equal rank are sorted too; at least 14 values lie on one side of the
// lowest five minima and two medians, and of the highest two medians and five maxima,
// so the result is the middle of the other 13 (4 + 5 + 4): some 100 minima and maxima a
// pixel, which bound it (half rate), where a selection from 27 values anew took 390
// (180 projections of 2048 x 256: 2.47 ms, so: 0.77 ms).
__device__ __noinline__ float median27_exchange(const float* __restrict__ dl, const float* __restrict__ dc,
                                                const float* __restrict__ dr, int ndet, int nrows, int jx, int jy)
{
    float r[27];
#pragma unroll
    for (int jxs = -1; jxs <= 1; ++jxs)
#pragma unroll
        for (int jys = -1; jys <= 1; ++jys) {
            const int cx = min(max(jx + jxs, 1), ndet), cy = min(max(jy + jys, 1), nrows);
            const size_t o = (size_t)(cy - 1) * ndet + (cx - 1);
            const int slot = 3 * (jxs + 1) + (jys + 1);
            r[slot] = __ldg(dl + o);
            r[slot + 9] = __ldg(dc + o);
            r[slot + 18] = __ldg(dr + o);
        }
#pragma unroll
    for (int a = 0; a < 14; ++a) {
        float ra = r[a];
#pragma unroll
        for (int b = a + 1; b < 27; ++b) {
            const float rb = r[b];
            const bool sw = rb > ra;
            r[b] = sw ? ra : rb;
            ra = sw ? rb : ra;
        }
        r[a] = ra;
    }
    return r[13];
}

__device__ __forceinline__ void cx_minmax(float& a, float& b)
{
    const float lo = fminf(a, b), hi = fmaxf(a, b);
    a = lo;
    b = hi;
}

struct Nine {
    float v[9];   // ascending
    float sum;    // NaN if a value is (or infinities cancel)
};

template <int M>
__device__ __forceinline__ Nine sort9(const float (&t)[M][3], const float (&sum)[M], int first)
{
    Nine n;
#pragma unroll
    for (int i = 0; i < 9; ++i) n.v[i] = t[first + i / 3][i % 3];
    constexpr int net[16][2] = {{2, 5}, {0, 3}, {1, 4}, {5, 8}, {3, 6}, {4, 7}, {2, 5}, {0, 3},
                                {1, 4}, {5, 7}, {2, 6}, {1, 3}, {4, 6}, {2, 4}, {5, 6}, {2, 3}};
#pragma unroll
    for (int k = 0; k < 16; ++k) cx_minmax(n.v[net[k][0]], n.v[net[k][1]]);
    n.sum = sum[first] + sum[first + 1] + sum[first + 2];
    return n;
}

__device__ __forceinline__ float median_of_nines(const Nine& a, const Nine& b, const Nine& c)
{
    float x[8], y[5];   // the minima of ranks 5..8 and the maxima of ranks 0..3; the medians of ranks 2..6
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        x[i] = fminf(fminf(a.v[5 + i], b.v[5 + i]), c.v[5 + i]);
        x[4 + i] = fmaxf(fmaxf(a.v[i], b.v[i]), c.v[i]);
    }
#pragma unroll
    for (int i = 0; i < 5; ++i) {
        const float lo = fminf(a.v[2 + i], b.v[2 + i]), hi = fmaxf(a.v[2 + i], b.v[2 + i]);
        y[i] = fmaxf(lo, fminf(hi, c.v[2 + i]));
    }
    constexpr int net[9][2] = {{0, 4}, {1, 5}, {2, 6}, {3, 7}, {2, 4}, {3, 5}, {1, 2}, {3, 4}, {5, 6}};
#pragma unroll
    for (int k = 0; k < 9; ++k) cx_minmax(x[net[k][0]], x[net[k][1]]);
    // the 7th of the merged 8 and the 5: the least of max(x_i, y_j) over i + j = 7
    float m = x[6];
#pragma unroll
    for (int j = 0; j < 5; ++j) m = fminf(m, fmaxf(x[5 - j], y[j]));
    return m;
}

// Threads 32 x 8, a block's tile 32 x 8 R pixels (grid.x: tiles), `len` projections (grid.y).
template <int R>
__global__ void __launch_bounds__(256, 2) k_median27(int ndet, int nrows, int nproj_chunk, int p_first, int nfiles,
                                                  int len, const float* __restrict__ proj, float* __restrict__ out)
{
    const size_t npix = (size_t)ndet * nrows;
    const int ntx = (ndet + 31) / 32, yb = blockIdx.x / ntx * (8 * R);
    const int x = blockIdx.x % ntx * 32 + threadIdx.x, y = yb + R * threadIdx.y;   // 0-based
    int off[R + 2][3];   // from the tile's first row
#pragma unroll
    for (int r = 0; r < R + 2; ++r)
#pragma unroll
        for (int k = 0; k < 3; ++k)
            off[r][k] = (min(max(y + r - 1, 0), nrows - 1) - yb) * ndet + min(max(x + k - 1, 0), ndet - 1);
    const float* tile = proj + (size_t)yb * ndet;
    auto load = [&](int p, Nine (&n)[R]) {
        const float* f = tile + p * npix;
        float t[R + 2][3], sum[R + 2];
#pragma unroll
        for (int r = 0; r < R + 2; ++r) {
#pragma unroll
            for (int k = 0; k < 3; ++k) t[r][k] = __ldg(f + off[r][k]);
            sum[r] = t[r][0] + t[r][1] + t[r][2];
            cx_minmax(t[r][0], t[r][1]);
            cx_minmax(t[r][1], t[r][2]);
            cx_minmax(t[r][0], t[r][1]);
        }
#pragma unroll
        for (int k = 0; k < R; ++k) n[k] = sort9(t, sum, k);
    };
    auto put = [&](int pc, int row, const Nine& l, const Nine& c, const Nine& r) {
        float m = median_of_nines(l, c, r);
        if (x >= ndet || row >= nrows) return;
        const float s = l.sum + c.sum + r.sum;
        if (m == 0.f || s != s) {
            const int p = p_first + pc;
            const float* dc = proj + p * npix;
            m = median27_exchange(p > 0 ? dc - npix : dc, dc, p < nfiles - 1 ? dc + npix : dc, ndet, nrows, x + 1,
                                  row + 1);
        }
        out[pc * npix + (size_t)row * ndet + x] = m;
    };
    const int pc0 = blockIdx.y * len, pc1 = min(pc0 + len, nproj_chunk);
    Nine l[R], c[R], r[R];
    load(p_first + pc0, c);
    if (p_first + pc0 > 0) {
        load(p_first + pc0 - 1, l);
    } else {
#pragma unroll
        for (int k = 0; k < R; ++k) l[k] = c[k];
    }
#pragma unroll 3
    for (int pc = pc0; pc < pc1; ++pc) {
        if (p_first + pc < nfiles - 1) {
            load(p_first + pc + 1, r);
        } else {
#pragma unroll
            for (int k = 0; k < R; ++k) r[k] = c[k];
        }
#pragma unroll
        for (int k = 0; k < R; ++k) {
            put(pc, y + k, l[k], c[k], r[k]);
            l[k] = c[k];
            c[k] = r[k];
        }
    }
}

// resample + transpose of a chunk of projections into the slice-major
// sinograms sino[row][projection][det] (:456-487).  The taps are the same for every
// projection: a thread forms them once and walks `len` projections (grid: 256
// pixels of a row, rows, walks).  Bound by the traffic (2.8 TB/s: two rows of the
// median are read per row); 180 projections of 2048 x 256: 487 us with the taps and three 64-bit
// divisions per value, so 273 us.
__global__ void __launch_bounds__(256) k_resample_to_sino(ResampleGeom g, int nproj_chunk, int p_first, int nfiles,
                                                          int len, const float* __restrict__ med,
                                                          float* __restrict__ sino)
{
    const int nx = g.ndet + g.add, jx = blockIdx.x * 256 + threadIdx.x + 1;
    if (jx > nx) return;
    const size_t npix = (size_t)g.ndet * g.nrows;
    const int pc0 = blockIdx.z * len, pc1 = min(pc0 + len, nproj_chunk);
    for (int jy = blockIdx.y + 1; jy <= g.nrows; jy += gridDim.y) {
        const Taps t = resample_taps(g, jx, jy);
        float* o = sino + ((size_t)(jy - 1) * nfiles + p_first) * nx + (jx - 1);
#pragma unroll 4
        for (int pc = pc0; pc < pc1; ++pc) o[(size_t)pc * nx] = resample_with(t, med + pc * npix);
    }
}

// ---- launchers -----------------------------------------------------------------
static inline unsigned nblocks(long n, int threads, unsigned cap = 8192)
{
    long b = (n + threads - 1) / threads;
    return (unsigned)(b < (long)cap ? (b < 1 ? 1 : b) : cap);
}

void launch_frame_average_u16(int nf, long npix, const uint16_t* f, float* out, cudaStream_t st)
{
    k_frame_average<uint16_t><<<nblocks(npix, 256), 256, 0, st>>>(nf, npix, f, out);
}
void launch_frame_average_f32(int nf, long npix, const float* f, float* out, cudaStream_t st)
{
    k_frame_average<float><<<nblocks(npix, 256), 256, 0, st>>>(nf, npix, f, out);
}
static bool aligned16(const void* p) { return ((uintptr_t)p & 15u) == 0; }

template <typename Tin>
static void launch_normalize(int mode, int nproj, long npix, const Tin* raw, const float* ob, const float* df,
                             float* out, cudaStream_t st)
{
    if (npix % 8 == 0 && aligned16(raw) && aligned16(ob) && aligned16(out) && (mode == 0 || aligned16(df))) {
        const long nvec = npix / 8;
        dim3 grd(nblocks(nvec, 256, 2048), (unsigned)std::min(nproj, 32768));
        k_normalize8<Tin><<<grd, 256, 0, st>>>(mode, nproj, nvec, raw, ob, df, out);
    } else {
        const long total = npix * nproj;
        k_normalize<Tin><<<nblocks(total, 256), 256, 0, st>>>(mode, npix, total, raw, ob, df, out);
    }
}
void launch_normalize_u16(int mode, int nproj, long npix, const uint16_t* raw, const float* ob, const float* df,
                          float* out, cudaStream_t st)
{
    launch_normalize<uint16_t>(mode, nproj, npix, raw, ob, df, out, st);
}
void launch_normalize_f32(int mode, int nproj, long npix, const float* raw, const float* ob, const float* df,
                          float* out, cudaStream_t st)
{
    launch_normalize<float>(mode, nproj, npix, raw, ob, df, out, st);
}
void launch_lerp(long n, const float* a, const float* b, float ta, float tb, float target, float* out,
                 cudaStream_t st)
{
    k_lerp<<<nblocks(n, 256), 256, 0, st>>>(n, a, b, ta, tb, target, out);
}
void launch_resample(int ndet, int nrows, const float* src, float cth, float sth, float shift, float* out,
                     cudaStream_t st)
{
    ResampleGeom g{ndet, nrows, ndet % 2 == 0 ? 1 : 0, cth, sth, shift};
    k_resample<<<nblocks((long)(ndet + g.add) * nrows, 256), 256, 0, st>>>(g, src, out);
}
int mirror_error_blocks(int ndet, int nrows)
{
    return (int)nblocks((long)(ndet + 1) * nrows, 256, 1024);
}
void launch_mirror_errors(int ndet, int nrows, const float* p0, const float* p180, const MirrorCandidates& cand, int n,
                          double* part, int nblk, unsigned* done, double* out, cudaStream_t st)
{
    k_mirror_errors<<<dim3(nblk, n), 256, 0, st>>>(ndet, nrows, cand, p0, p180, part, done, out);
}
void launch_com(int ndet, int nrows, const float* p0, const float* p180, double* part, int nblk, double* out3,
                cudaStream_t st)
{
    k_com<<<nblk, 256, 0, st>>>(ndet, nrows, ndet % 2 == 0 ? 1 : 0, p0, p180, part);
    k_sum_partials<<<3, 256, 0, st>>>(part, nblk, out3);
}
size_t xcorr_scratch_words(int kmax) { return 2 * (size_t)(2 * kmax + 1) + 1; }

namespace {
template <typename T>
struct same_t {
    using type = T;
};
// cudaLaunchKernel with typed arguments: returns this launch's own error and
// leaves earlier, unrelated errors of the caller pending.
template <typename... P>
cudaError_t launch_k(void (*k)(P...), dim3 grd, dim3 blk, cudaStream_t st, typename same_t<P>::type... args)
{
    void* a[] = {&args...};
    return cudaLaunchKernel(reinterpret_cast<const void*>(k), grd, blk, a, 0, st);
}
}  // namespace

cudaError_t launch_xcorr(int ndet, int nrows, int kmax, const float* p0, const float* p180,
                         unsigned long long* scratch, cudaStream_t st)
{
    const int nk = 2 * kmax + 1;
    cudaError_t e = cudaMemsetAsync(scratch, 0, sizeof(unsigned long long) * xcorr_scratch_words(kmax), st);
    if (e != cudaSuccess) return e;
    // a few blocks for every SM, each with a whole number of items, and no more items than its sums hold
    const int items = (ndet + XC_X - 1) / XC_X * nrows, tiles = (nk + XC_LAGS - 1) / XC_LAGS;
    const int want = std::max(1, std::min(items, 152 * 8 / tiles)), per = std::min((items + want - 1) / want, XC_ITEMS);
    dim3 grd((items + per - 1) / per, tiles);
    e = launch_k(k_xcorr, grd, dim3(256), st, ndet, nrows, kmax, p0, p180, scratch);
    if (e != cudaSuccess) return e;
    return launch_k(k_argmax, dim3(1), dim3(256), st, nk, scratch);
}

int xcorr_finish(int kmax, const unsigned long long* h, int64_t* corr_out, int* k_best, double* k_sub,
                 const char** why)
{
    const int nk = 2 * kmax + 1;
    const int bi = (int)(unsigned int)(h[2 * nk] & 0xffffffffu);
    const unsigned int flag = (unsigned int)(h[2 * nk] >> 32);
    if (flag) {
        *why = "a projection holds a value that is not finite, or a product p0*p180 of magnitude >= 2^31";
        return ACU_ERR_INVALID;
    }
    if (bi < 0 || bi >= nk) {
        *why = "the correlation argmax is out of range";
        return ACU_ERR_CUDA;
    }
    auto fits = [&](int i) {
        const long long hi = (long long)h[2 * i + 1];
        const long long lo = (long long)h[2 * i];
        return hi == (lo < 0 ? -1ll : 0ll);
    };
    auto to_double = [&](int i) {   // the sum as a double (exact conversion of an int64 when it fits)
        if (fits(i)) return (double)(long long)h[2 * i];
        return ldexp((double)(long long)h[2 * i + 1], 64) + (double)h[2 * i];
    };
    if (corr_out) {
        for (int i = 0; i < nk; ++i)
            if (!fits(i)) {
                *why = "a correlation sum exceeds the int64 range of corr_out (pass corr_out = NULL for the lag "
                       "alone)";
                return ACU_ERR_UNSUPPORTED;
            }
        for (int i = 0; i < nk; ++i) corr_out[i] = (int64_t)(long long)h[2 * i];
    }
    double frac = 0.0;
    if (bi > 0 && bi < nk - 1) {
        const double cm = to_double(bi - 1), c0 = to_double(bi), cp = to_double(bi + 1);
        const double den = cm - 2.0 * c0 + cp;
        if (den < 0.0) frac = 0.5 * (cm - cp) / den;
    }
    *k_best = bi - kmax;
    *k_sub = (double)(bi - kmax) + frac;
    return ACU_OK;
}
void launch_median27(int ndet, int nrows, int nchunk, int p_first, int nfiles, const float* proj, float* out,
                     cudaStream_t st)
{
    // projections per thread: a walk of 32 sorts a sixteenth more than it needs; shorter ones where blocks are too few, and with walks of one, one pixel per thread (two pixels or one in walks of 32, 180
    // projections of 2048 x 256, with the resampling: 1.27 and 1.55 ms; a single 1025 x 64 frame: 28 and 24 us)
    auto grid = [&](int rows, int len) {
        return dim3((ndet + 31) / 32 * ((nrows + rows - 1) / rows), (nchunk + len - 1) / len);
    };
    int len = 32;
    while (len > 1 && (size_t)grid(16, len).x * grid(16, len).y < 152 * 8) len /= 2;
    len = std::max(len, (nchunk + 65534) / 65535);
    if (len > 1)
        k_median27<2><<<grid(16, len), dim3(32, 8), 0, st>>>(ndet, nrows, nchunk, p_first, nfiles, len, proj, out);
    else
        k_median27<1><<<grid(8, len), dim3(32, 8), 0, st>>>(ndet, nrows, nchunk, p_first, nfiles, len, proj, out);
}
void launch_resample_to_sino(int ndet, int nrows, int nchunk, int p_first, int nfiles, const float* med,
                             float cth, float sth, float shift, float* sino, cudaStream_t st)
{
    ResampleGeom g{ndet, nrows, ndet % 2 == 0 ? 1 : 0, cth, sth, shift};
    const unsigned gx = (ndet + g.add + 255) / 256, gy = std::min(nrows, 65535);
    int len = 16;
    while (len > 1 && (size_t)gx * gy * ((nchunk + len - 1) / len) < 152 * 8) len /= 2;
    len = std::max(len, (nchunk + 65534) / 65535);
    k_resample_to_sino<<<dim3(gx, gy, (nchunk + len - 1) / len), 256, 0, st>>>(g, nchunk, p_first, nfiles, len, med, sino);
}

}  // namespace acu

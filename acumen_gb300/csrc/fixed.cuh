// Sample positions in fixed point for the kernels that carry one slice per
// thread, which are held by the instructions a position takes (exact positions,
// sides up to FX_MAX_SIDE).
//
// Along a ray both coordinates advance by a constant, so they are kept as
// 64-bit integers with 32 fraction bits: the cell is the high word, the fraction
// the low word's leading 23 bits, and a step is an addition.  A sine or cosine is
// rounded to 2^-33 and multiplied by at most FX_MAX_SIDE / 2 from the middle of
// the grid, so a coordinate is within 2.4e-7 of double precision at a side of
// 2049 (6e-8 rms) and exact at grid-aligned angles, as with split tables
// (common.cuh), at five instructions in place of thirteen.
#pragma once
#include <type_traits>

#include "common.cuh"
#include "kernels.h"

namespace acu {

__device__ __forceinline__ int fx_cell(long long v) { return (int)(v >> 32); }
__device__ __forceinline__ float fx_frac(long long v)
{
    return __uint_as_float(__funnelshift_r((unsigned)v, 0x3f800000u >> 23, 9)) - 1.f;   // 1.fraction, less 1
}
constexpr long long FX_HALF = 1ll << 8;   // half of the fraction's last kept bit: fractions are rounded, not cut

// One 32 x 32 tile (at x0, y0, 0-based) of an image as pairs (pixel, next pixel of
// the row) and of its transpose likewise, by a block of 256: a tap row of the
// projector is one load.
__device__ __forceinline__ void pair_tile(const float* __restrict__ img, float2* __restrict__ P, float2* __restrict__ PT,
                                          int N, int x0, int y0)
{
    __shared__ float tile[33][34];
    for (int i = threadIdx.x; i < 33 * 33; i += 256) {
        const int ty = i / 33, tx = i % 33;
        tile[ty][tx] = x0 + tx < N && y0 + ty < N ? img[(size_t)(y0 + ty) * N + x0 + tx] : 0.f;
    }
    __syncthreads();
    const int a = threadIdx.x & 31;
    for (int b = threadIdx.x >> 5; b < 32; b += 8) {
        if (x0 + a < N && y0 + b < N) P[(size_t)(y0 + b) * N + x0 + a] = make_float2(tile[b][a], tile[b][a + 1]);
        if (y0 + a < N && x0 + b < N) PT[(size_t)(x0 + b) * N + y0 + a] = make_float2(tile[a][b], tile[a + 1][b]);
    }
}

// One ray (bin jy) of the single-slice projector: the sum of its samples.  The
// rays of a warp are staggered so that the 32 samples of a step lie in one or two
// rows of the copy read.  TR: through the transpose (rows follow x), else the
// image (rows follow y).
template <bool TR>
__device__ __forceinline__ float fx_ray(const float2* __restrict__ base, int N, FxAngle a,
                                        const ProjRay<float, true>& ray, int jy, int lane)
{
    const int m = (N + 1) / 2;
    const float s = (float)a.s * 0x1p-32f, c = (float)a.c * 0x1p-32f;
    // |c| <= |s| without TR and the other way round with it
    const float ratio = TR ? -s / c : c / s;
    const int kb = __float2int_rn((float)lane * ratio);
    long long xm = ((long long)m << 32) - a.s * (jy - m) + FX_HALF, ym = ((long long)m << 32) + a.c * (jy - m) + FX_HALF;
    bool some = jy <= N;
    // The ray's steps whose cell is valid are an interval.  It is estimated with a margin and narrowed by the fixed-point
    // positions, then its ends are settled by the exact ones, which differ by less than 1e-6: at most one sample at
    // each end, unless the ray is nearly parallel to an axis and runs along the rim, where only those tell.
    int lo, hi;
    valid_steps(s, c, (float)(jy - m), (float)m, N, lo, hi);
    auto valid = [&](int jx) {
        int x, y;
        float w0, w1, w2, w3;
        ray.at((float)(jx - m), x, y, w0, w1, w2, w3);
        return min(x, y) > 1 && max(x, y) < N;
    };
    auto inside = [&](int jx) {
        const int x = fx_cell(xm + (jx - m) * a.c), y = fx_cell(ym + (jx - m) * a.s);
        return (unsigned)(x - 2) < (unsigned)(N - 2) && (unsigned)(y - 2) < (unsigned)(N - 2);
    };
    if (some) {
        if (fminf(fabsf(s), fabsf(c)) >= 1e-3f) {
            const int lo0 = lo, hi0 = hi;
            while (lo <= hi && !inside(lo)) ++lo;
            while (lo <= hi && !inside(hi)) --hi;
            if (lo > hi) {   // a corner: at most a sample or two, if any
                lo = lo0;
                hi = hi0;
            } else {
                lo = max(lo - 1, lo0);
                hi = min(hi + 1, hi0);
            }
        }
        while (lo <= hi && !valid(lo)) ++lo;
        while (lo <= hi && !valid(hi)) --hi;
        some = lo <= hi;
        // where that puts a fixed-point sample on the rim, the ray moves in by the difference: its cells are in 1..N-1
        const long long end = ((long long)N << 32) - 1;
        xm -= max(0ll, max(xm + (lo - m) * a.c, xm + (hi - m) * a.c) - end);
        ym -= max(0ll, max(ym + (lo - m) * a.s, ym + (hi - m) * a.s) - end);
    }
    if (!some) {
        lo = 0x3fffffff;
        hi = -0x3fffffff;
    } else {
        lo += kb;
        hi += kb;
    }
    // steps of the warp: where some ray has a sample, and where all have
    const int i0 = __reduce_min_sync(0xffffffffu, lo), i1 = __reduce_max_sync(0xffffffffu, hi);
    const int a0 = __reduce_max_sync(0xffffffffu, lo), a1 = __reduce_min_sync(0xffffffffu, hi);
    const long long dr = TR ? a.c : a.s, dc = TR ? a.s : a.c;
    const long long steps = (long long)i0 - kb - m;
    long long r = (TR ? xm : ym) + steps * dr, q = (TR ? ym : xm) + steps * dc;
    const float2* const base0 = base - (N + 1);   // of cell (0, 0)
    float sum = 0.f;
    // a step in which some rays have no sample reads a pixel of the image all the same and drops it: without a branch,
    // the loads of several steps are in flight together
    auto sample = [&](auto partial, int i) {
        int cr = fx_cell(r), cq = fx_cell(q);
        bool ok = true;
        if constexpr (decltype(partial)::value) {
            ok = i >= lo && i <= hi;
            cr = min(max(cr, 1), N - 1);
            cq = min(max(cq, 1), N - 1);
        }
        const float2* p = base0 + (unsigned)(cr * N + cq);
        const float fr = fx_frac(r), fc = fx_frac(q);
        const float2 v0 = __ldg(p), v1 = __ldg(p + N);
        const float gr = 1.f - fr, gc = 1.f - fc;
        const float t = fmaf(v0.y, fc, v0.x * gc), b = fmaf(v1.y, fc, v1.x * gc);
        const float next = fmaf(b, fr, fmaf(t, gr, sum));
        sum = ok ? next : sum;
        r += dr;
        q += dc;
    };
    using Some = std::true_type;
    using All = std::false_type;
    int i = i0;
    const int b0 = a0 <= a1 ? a0 : i1 + 1;   // steps before all rays have samples (all steps, if there are none)
#pragma unroll 4
    for (; i < b0; ++i) sample(Some{}, i);
#pragma unroll 2
    for (; i <= a1; ++i) sample(All{}, i);
#pragma unroll 4
    for (; i <= i1; ++i) sample(Some{}, i);
    return sum;
}

// Backprojection of one 32-pixel-wide tile by a block of 32 x BY threads, R rows
// a thread (column-wise neighbours), one slice.  q: [T][N] pairs (bins y and
// y + 1: one load per pixel), zeros in the first and the last, which are never
// tapped.  Per angle the position of the tile's middle pixel is formed once per
// block (split tables, common.cuh) and kept with 26 fraction bits; the pixels'
// positions follow by additions.  |position - middle| < 32 bins: the tile is at
// most 32 pixels high.  FH > 0: every FH rows have a middle of their own, so that the
// bits do not depend on the tile's height.
constexpr int FX_CHUNK = 256;   // angles whose entries are held in shared memory

template <int R, int FH = 0>
__device__ __forceinline__ void fx_backproject(const float2* __restrict__ q, const float4* __restrict__ xsc, int N,
                                               int T, float mid, int x0, int y0, int4* tab, float (&out)[R])
{
    const int tid = threadIdx.y * 32 + threadIdx.x, nthreads = 32 * blockDim.y, height = R * blockDim.y;
    const int fh = FH ? FH : height, frames = FH ? height / FH : 1, frame = FH ? (int)threadIdx.y * R / fh : 0;
    const int lx = (int)threadIdx.x - 16, ly = (int)threadIdx.y * R - frame * fh - fh / 2;
    const int4* const mine = tab + frame * FX_CHUNK;
#pragma unroll
    for (int r = 0; r < R; ++r) out[r] = 0.f;
    for (int t0 = 0; t0 < T; t0 += FX_CHUNK) {
        const int n = min(FX_CHUNK, T - t0);
        __syncthreads();
        for (int f = 0; f < frames; ++f)
        for (int a = tid; a < n; a += nthreads) {
            const float4 x = __ldg(xsc + t0 + a);
            float cell, frac;
            exact_coord(x.x, x.y, x.z, x.w, (float)(x0 + 16) - mid, (float)(y0 + f * fh + fh / 2) - mid, mid, cell, frac);
            constexpr float ONE = 67108864.f;   // 2^26
            // cell - 1: the pair's index; 4: half of the fraction's last kept bit
            tab[f * FX_CHUNK + a] = make_int4((int)(frac * ONE) + 4, (int)(x.x * ONE) + __float2int_rn(x.z * ONE),
                               (int)(x.y * ONE) + __float2int_rn(x.w * ONE), (int)cell - 1);
        }
        __syncthreads();
        const float2* row = q + (size_t)t0 * N;
        // a block's first touch of an angle's bins comes from L2: 32 loads in flight per thread
#pragma unroll (32 / R)
        for (int a = 0; a < n; ++a, row += N) {
            const int4 e = mine[a];
            int p = e.x + lx * e.y + ly * e.z;
#pragma unroll
            for (int r = 0; r < R; ++r) {
                const unsigned i = min((unsigned)((p >> 26) + e.w), (unsigned)(N - 1));
                const float w = __uint_as_float(((unsigned)(p << 6) >> 9) | 0x3f800000u);   // fraction + 1
                const float2 v = __ldg(row + i);
                out[r] = fmaf(v.y, w - 1.f, fmaf(v.x, 2.f - w, out[r]));
                p += e.z;
            }
        }
    }
}

}  // namespace acu

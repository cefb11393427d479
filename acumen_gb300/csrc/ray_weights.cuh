// The projector's weights seen from a pixel (exact positions): shared by the
// tensor-core projector, which gathers them into a matrix, and the transpose.
#pragma once
#include "common.cuh"
#include "fixed.cuh"
#include "kernels.h"

namespace acu {

// Whether step k of ray j lies in a valid cell, by the projector's arithmetic (ProjRay, common.cuh).
__device__ __forceinline__ bool sample_valid(float4 x, float k, int j, float off, float mid, int N)
{
    const float dy = (float)j - mid, dx = k - mid;
    float cx, cy, f;
    split_floor(__fmaf_rn(x.y, dx, __fmaf_rn(-x.x, dy, mid)),
                __fmaf_rn(x.w, dx, __fmaf_rn(-x.x, off, __fmaf_rn(-x.z, off, __fmul_rn(-x.z, dy)))), cx, f);
    split_floor(__fmaf_rn(x.x, dx, __fmaf_rn(x.y, dy, mid)),
                __fmaf_rn(x.z, dx, __fmaf_rn(x.y, off, __fmaf_rn(x.w, off, __fmul_rn(x.w, dy)))), cy, f);
    return fminf(cx, cy) > 1.f && fmaxf(cx, cy) < (float)N;
}

// A pixel's coordinates along (u) and across (w) the rays: cells and fractions.
struct RayPos {
    int cu, cw;
    float uf, wf;
};

// Exact positions (split tables); ex, ey: the pixel's place relative to the middle, off: the angle's detector offset.
__device__ __forceinline__ RayPos ray_pos(float4 x, float ex, float ey, float off, float mid)
{
    RayPos p;
    float cell;
    split_floor(__fmaf_rn(x.y, ex, __fmaf_rn(x.x, ey, mid)), __fmaf_rn(x.w, ex, __fmul_rn(x.z, ey)), cell, p.uf);
    p.cu = (int)cell;
    split_floor(__fmaf_rn(-x.x, ex, __fmaf_rn(x.y, ey, mid)), __fmaf_rn(-x.z, ex, __fmul_rn(x.w, ey)) - off, cell, p.wf);
    p.cw = fabsf(off) < 1e6f ? (int)cell : -(1 << 30);   // no number, or too far out: meets no ray
    return p;
}

// The pixels around one pixel: its exact coordinates, and the
// steps from one to the next, with 26 fraction bits.  Within 31 cells a fraction is off by
// 5e-7 at most (half a bit of either step per pixel); 6 instructions a
// coordinate in place of 14.  It pays where a frame serves many pixels (the transpose);
// in the tensor-core projector, where it serves two, it took 3 % longer.
struct RayFrame {
    int u, w, c, s, cu, cw;
    RayFrame() = default;
    __device__ __forceinline__ RayFrame(float4 x, float ex, float ey, float off, float mid)
    {
        constexpr float ONE = 67108864.f;   // 2^26
        const RayPos p = ray_pos(x, ex, ey, off, mid);
        cu = p.cu;
        cw = p.cw;
        u = (int)(p.uf * ONE) + 4;   // 4: half of the fraction's last kept bit
        w = (int)(p.wf * ONE) + 4;
        s = (int)(x.x * ONE) + __float2int_rn(x.z * ONE);
        c = (int)(x.y * ONE) + __float2int_rn(x.w * ONE);
    }
    __device__ __forceinline__ void move(int dx, int dy)
    {
        u += dx * c + dy * s;
        w += dy * c - dx * s;
    }
    __device__ __forceinline__ RayPos pos() const
    {
        return {cu + (u >> 26), cw + (w >> 26), fx_frac((long long)(unsigned)(u << 6)), fx_frac((long long)(unsigned)(w << 6))};
    }
};

// The weights of the three rays j, j+1, j+2 nearest to pixel (px, py) at p (off:
// the angle's detector offset).  Ray j's samples sit at the pixel's distance (dx, dy) = (c e - s d, s e + c d) with d = j - w,
// e = k - u, where (u, w) are the pixel's coordinates along and across the rays;
// the bilinear weight of a sample is (1 - |dx|)+ (1 - |dy|)+.  Of the integers
// e + u only the three nearest to the ray's closest approach reach the pixel.
// INNER: every sample that reaches the pixel exists and is valid; ENDS: some may
// lie beyond a ray's ends; RIM: some may lie in a cell outside 2..N-1 too.
enum { INNER, ENDS, RIM };

template <int WHERE>
__device__ __forceinline__ void ray_weights(const MmaAngle& a, RayPos at, float off, float mid, int px, int py, int N,
                                            int& j, float (&wv)[3])
{
    const float uf = at.uf;
    const bool up = at.wf > 0.5f;   // |d| < |c| + |s| <= 1.42 leaves three candidates
    j = at.cw - (up ? 0 : 1);
    const float d0 = (up ? 0.f : -1.f) - at.wf;
    const float2 along = make_float2(a.c, a.s), back = make_float2(-a.c, -a.s), across = make_float2(-a.s, a.c);
    const float2 one = make_float2(1.f, 1.f);
#pragma unroll
    for (int r = 0; r < 3; ++r) {
        const float d = d0 + (float)r;
        const float ctr = __fmaf_rn(a.t, d, uf);
        const float kf = __fsub_rn(__fadd_rn(ctr, 12582912.f), 12582912.f);   // nearest integer
        const float e = kf - uf;
        const float2 p0 = fma2(along, make_float2(e, e), mul2(across, make_float2(d, d)));
        float w = 0.f;
#pragma unroll
        for (int q = -1; q <= 1; ++q) {
            const float2 p = q < 0 ? fma2(back, one, p0) : q > 0 ? fma2(along, one, p0) : p0;
            const float hx = __saturatef(1.f - fabsf(p.x)), hy = __saturatef(1.f - fabsf(p.y));
            if constexpr (WHERE == INNER) {
                w = fmaf(hx, hy, w);
            } else {
                const float k = (float)at.cu + kf + (float)q;
                bool ok = k >= 1.f && k <= (float)N;
                if constexpr (WHERE == RIM) {
                    // within 1e-5 of a cell edge at the rim the projector's own position decides
                    const float xl = p.x - (float)(2 - px), xh = p.x - (float)(N - px);
                    const float yl = p.y - (float)(2 - py), yh = p.y - (float)(N - py);
                    if (fminf(fminf(fabsf(xl), fabsf(xh)), fminf(fabsf(yl), fabsf(yh))) < 1e-5f)
                        ok = ok && sample_valid(a.x, k, j + r, off, mid, N);
                    else
                        ok = ok && xl >= 0.f && xh < 0.f && yl >= 0.f && yh < 0.f;
                }
                w = ok ? fmaf(hx, hy, w) : w;
            }
        }
        wv[r] = w;
    }
}

// pixels whose taps can belong to samples outside the valid cells
__device__ __forceinline__ bool on_rim(int px, int py, int N) { return px < 3 || py < 3 || px >= N || py >= N; }

}  // namespace acu

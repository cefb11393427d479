// Kernels that carry one slice per thread at exact positions: projector
// (tomography/tv_hpc.F90:129-159) and filtered backprojection's second half
// (:107-123).
// Batches share a sample position among four slices or more; here the position
// is most of the work, so it is kept in fixed point (fixed.cuh).
#include <algorithm>
#include <cmath>

#include "common.cuh"
#include "fixed.cuh"
#include "kernels.h"

namespace acu {

namespace {

// grid (128 rays, angle in copy order, slice).  Held by the instructions of a
// sample (31 issue slots, 4 of them loads) and the latency of its four loads: 12 blocks an SM
// rather than 9 gain 6 %, deeper unrolling nothing.  Against positions from split
// tables (us, before / now): 363^2 x 360 159 / 99, 725^2 x 720 882 / 453,
// 1449^2 x 900 3896 / 1955, 2049^2 x 1200 9979 / 4969.
__global__ void __launch_bounds__(128, 12) k_ray_fx(const float* __restrict__ I, const float* __restrict__ IT,
                                                    const FxAngle* __restrict__ fx, const float4* __restrict__ xsc,
                                                    const int* __restrict__ order, float* __restrict__ sino, int N,
                                                    int T, float mid)
{
    const int lane = threadIdx.x, t = order[blockIdx.y];
    const int jy = blockIdx.x * 128 + threadIdx.y * 32 + lane + 1;
    const size_t g = blockIdx.z;
    const FxAngle a = fx[t];
    const ProjRay<float, true> ray(nullptr, xsc, t, jy, mid, nullptr);
    const float v = llabs(a.c) > llabs(a.s) ? fx_ray<true>(IT + g * N * N, N, a, ray, jy, lane)
                                            : fx_ray<false>(I + g * N * N, N, a, ray, jy, lane);
    if (jy <= N) sino[(g * T + t) * N + (jy - 1)] = v / (float)N;
}

// Held by issue slots: an update is one 64-bit load, an addition, a shift, a
// subtraction and two multiply-adds.  Against the gather with both bins loaded and
// positions from split tables (us, before / now): 725^2 x 720 328 / 195,
// 1449^2 x 900 1261 / 734, 2049^2 x 1200 3215 / 1712.
template <int R>
__global__ void __launch_bounds__(256) k_backproject_fx(const float2* __restrict__ q, const float* __restrict__ cmask,
                                                        const float4* __restrict__ xsc, float* __restrict__ img, int N,
                                                        int T, float mid)
{
    __shared__ int4 tab[FX_CHUNK];
    const int x0 = blockIdx.x * 32 + 1, y0 = blockIdx.y * (8 * R) + 1;
    const int x = x0 + threadIdx.x - 1, y = y0 + threadIdx.y * R - 1;   // 0-based
    float cm[R];
    bool any = false;
#pragma unroll
    for (int r = 0; r < R; ++r) {
        cm[r] = x < N && y + r < N ? cmask[(size_t)(y + r) * N + x] : 0.f;
        any |= cm[r] != 0.f;
    }
    float v[R];
#pragma unroll
    for (int r = 0; r < R; ++r) v[r] = 0.f;
    if (__syncthreads_or(any))
        fx_backproject<R>(q + (size_t)blockIdx.z * T * N, xsc, N, T, mid, x0, y0, tab, v);
    float* const o = img + (size_t)blockIdx.z * N * N;
#pragma unroll
    for (int r = 0; r < R; ++r)
        if (x < N && y + r < N) o[(size_t)(y + r) * N + x] = cm[r] != 0.f ? cm[r] * v[r] : 0.f;
}

// bins -> pairs (bin, next bin), zeros in the first and the last
__global__ void __launch_bounds__(256) k_pairs(const float* __restrict__ q, float2* __restrict__ out, int N, size_t n)
{
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
        const int k = (int)(i % N);
        float2 p = make_float2(0.f, 0.f);
        if (k > 0 && k < N - 1) {
            p.x = q[i];
            p.y = q[i + 1];
        }
        out[i] = p;
    }
}

}  // namespace

std::vector<FxAngle> fx_angles(const float* xsc, int T)
{
    std::vector<FxAngle> out((size_t)T);
    for (int t = 0; t < T; ++t) {
        out[t].s = (long long)std::llround(((double)xsc[4 * t] + (double)xsc[4 * t + 2]) * 0x1p32);
        out[t].c = (long long)std::llround(((double)xsc[4 * t + 1] + (double)xsc[4 * t + 3]) * 0x1p32);
    }
    return out;
}

void launch_radon_fx(const DevGeom<float>& g, int S, const float* img, float* IT, float* sino, cudaStream_t st)
{
    launch_transpose_v1(g.N, S, img, IT, st);
    k_ray_fx<<<dim3((g.N + 127) / 128, g.T, S), dim3(32, 4), 0, st>>>(img, IT, g.fx_fp, g.xsc_fp, g.fp_order, sino, g.N,
                                                                     g.T, g.mid);
}

void launch_backproject_fx(const DevGeom<float>& g, int S, const float2* q, float* img, cudaStream_t st)
{
    const dim3 blk(32, 8);
    auto grid = [&](int r) { return dim3((g.N + 31) / 32, (g.N + 8 * r - 1) / (8 * r), S); };
    // rows per thread: more share an angle's entry, fewer keep the chip busy.  Measured with 1 / 2 / 4 rows (us): 363^2 x
    // 360 55 / 90 / -, 725^2 x 720 200 / 196 / 242, 1449^2 x 900 795 / 768 / 735
    if (g.N < 500)
        k_backproject_fx<1><<<grid(1), blk, 0, st>>>(q, g.cmask, g.xsc_bp, img, g.N, g.T, g.mid);
    else if (g.N < 1000)
        k_backproject_fx<2><<<grid(2), blk, 0, st>>>(q, g.cmask, g.xsc_bp, img, g.N, g.T, g.mid);
    else
        k_backproject_fx<4><<<grid(4), blk, 0, st>>>(q, g.cmask, g.xsc_bp, img, g.N, g.T, g.mid);
}

void launch_pairs(const float* q, float2* out, int N, size_t n, cudaStream_t st)
{
    k_pairs<<<(unsigned)std::min<size_t>((n + 255) / 256, (size_t)152 * 32), 256, 0, st>>>(q, out, N, n);
}

}  // namespace acu

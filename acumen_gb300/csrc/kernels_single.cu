// Kernels that carry one slice per thread at exact positions: projector
// (tomography/tv_hpc.F90:129-159) with its offset derivative, filtered
// backprojection's second half (:107-123), and the projector's transpose.
// Batches share a sample position among four slices or more; here the position
// is most of the work, so it is kept in fixed point (fixed.cuh).
#include <algorithm>
#include <cmath>

#include "common.cuh"
#include "fixed.cuh"
#include "kernels.h"
#include "ray_weights.cuh"

namespace acu {

namespace {

__global__ void __launch_bounds__(256) k_pair_images(const float* __restrict__ img, float2* __restrict__ P,
                                                     float2* __restrict__ PT, int N)
{
    const size_t g = blockIdx.z, at = g * N * N;
    pair_tile(img + at, P + at, PT + at, N, blockIdx.x * 32, blockIdx.y * 32);
}

// grid (128 rays, angle in copy order, slice).  Held by the instructions of a
// sample and by its two loads (the taps of a row as pairs: four single loads took 4 to 15 %
// longer); deeper unrolling and more blocks an SM gain nothing.  Against positions
// from split tables (us, before / now): 363^2 x 360 159 / 84, 725^2 x 720 882 / 408,
// 1449^2 x 900 3896 / 1802, 2049^2 x 1200 9979 / 4761.
__global__ void __launch_bounds__(128, 8) k_ray_fx(const float2* __restrict__ I, const float2* __restrict__ IT,
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

// Projection with per-angle detector offsets and, GRAD, its derivative with
// respect to them, from one walk along staggered rays (as fx_ray) where the
// general kernels (k_radon, k_radon_doff) walk twice and read a column of the
// image per step.  Positions, taps and the order of the sums are theirs: the loss
// is a sum of squares of these values, and the derivative jumps where a sample
// changes its cell, so neither would stand another rounding.
// Held by the instructions of the positions.  Two slices, 1025^2 x 600: 3.31 ms the
// projection and 3.40 ms the derivative there, 2.4 ms both here.
template <bool TR, bool GRAD>
__device__ __forceinline__ void ray_off(const float2* __restrict__ base, int N, float s, float c,
                                        const ProjRay<float, true>& ray, float mid, int jy, float off, int lane,
                                        float& sum, float& der)
{
    const float ratio = TR ? -s / c : c / s;
    const int kb = __float2int_rn((float)lane * ratio);
    int lo, hi;
    valid_steps(s, c, (float)jy - mid + off, mid, N, lo, hi);
    if (jy > N || !(fabsf(off) < 4.f * N) || lo > hi) {   // no ray, no number, or too far out to meet a pixel
        lo = 0x3fffffff;
        hi = -0x3fffffff;
    }
    const int i0 = __reduce_min_sync(0xffffffffu, lo + kb), i1 = __reduce_max_sync(0xffffffffu, hi + kb);
#pragma unroll 4
    for (int i = i0; i <= i1; ++i) {
        const int jx = i - kb;
        int x1, y1;
        float wxl, wxh, wyl, wyh;
        ray.at((float)jx - mid, x1, y1, wxl, wxh, wyl, wyh);
        if (jx >= lo && jx <= hi && min(x1, y1) > 1 && max(x1, y1) < N) {
            const float2* p = base + (TR ? (unsigned)((x1 - 1) * N + y1 - 1) : (unsigned)((y1 - 1) * N + x1 - 1));
            const float2 v0 = __ldg(p), v1 = __ldg(p + N);
            const float a = v0.x, b = TR ? v1.x : v0.y, cc = TR ? v0.y : v1.x, d = v1.y;
            const float w11 = wxl * wyl, w21 = wxh * wyl, w12 = wxl * wyh, w22 = wxh * wyh;
            sum = fmaf(d, w22, fmaf(cc, w12, fmaf(b, w21, fmaf(a, w11, sum))));
            if constexpr (GRAD) {
                const float gx = (b - a) * wyl + (d - cc) * wyh;
                const float gy = (cc - a) * wxl + (d - b) * wxh;
                der += gy * c - gx * s;
            }
        }
    }
}

template <bool GRAD>
__global__ void __launch_bounds__(128) k_ray_off(const float2* __restrict__ I, const float2* __restrict__ IT,
                                                 const float* __restrict__ sc, const float4* __restrict__ xsc,
                                                 const int* __restrict__ order, const float* __restrict__ off,
                                                 float* __restrict__ sino, float* __restrict__ dsino, int N, int T,
                                                 float mid)
{
    const int nb = (N + 127) / 128, lane = threadIdx.x, t = order[blockIdx.x / nb];
    const int jy = blockIdx.x % nb * 128 + threadIdx.y * 32 + lane + 1;
    const size_t g = blockIdx.z;
    const float s = sc[2 * t], c = sc[2 * t + 1], o = off ? off[g * T + t] : 0.f;
    const ProjRay<float, true> ray(sc, xsc, t, jy, mid, off ? off + g * T + t : nullptr);
    float v = 0.f, d = 0.f;
    if (fabsf(c) > fabsf(s))
        ray_off<true, GRAD>(IT + g * N * N, N, s, c, ray, mid, jy, o, lane, v, d);
    else
        ray_off<false, GRAD>(I + g * N * N, N, s, c, ray, mid, jy, o, lane, v, d);
    if (jy > N) return;
    const size_t at = (g * T + t) * N + (jy - 1);
    sino[at] = v / (float)N;
    if constexpr (GRAD) dsino[at] = d / (float)N;
}

// Held by issue slots: an update is one 64-bit load, an addition, a shift, a
// subtraction and two multiply-adds.  Against the gather with both bins loaded and
// positions from split tables (us, before / now): 725^2 x 720 328 / 180,
// 1449^2 x 900 1261 / 713, 2049^2 x 1200 3215 / 1652.  Registers for the loads in flight
// count more than blocks: with five blocks an SM instead of four 725^2 took 50 % longer.
template <int R>
__global__ void __launch_bounds__(256, R == 1 ? 3 : 4) k_backproject_fx(const float2* __restrict__ q, const float* __restrict__ cmask,
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

template <int V>
__device__ __forceinline__ void add_rays(Lanes<float, V>& acc, const float* __restrict__ y, const float (&w)[3], int j,
                                         int N)
{
#pragma unroll
    for (int r = 0; r < 3; ++r)
        if ((unsigned)(j + r - 1) < (unsigned)N && w[r] != 0.f) {
            const Lanes<float, V> v = ld_lanes<float, V>(y + (size_t)(j + r - 1) * V);
#pragma unroll
            for (int k = 0; k < V; ++k) acc.v[k] = fmaf(w[r], v.v[k], acc.v[k]);
        }
}

template <int V>
__device__ __forceinline__ void put_image(float* __restrict__ img, Lanes<float, V> acc, size_t g, int px, int py, int N)
{
#pragma unroll
    for (int k = 0; k < V; ++k) acc.v[k] = acc.v[k] / (float)N;
    st_lanes<float, V>(img + (g * N * N + (size_t)(py - 1) * N + (px - 1)) * V, acc);
}

// Transpose of the projector (at positions 5e-7 px from its own, but on the
// rim), as a gather over the angles: the at most
// three rays whose samples read the pixel, each with the sum of its samples'
// weights there.  The general kernel (k_radon_adjoint) evaluates the projector at
// 16 candidate samples per pixel and angle; this one evaluates the nine bilinear
// weights that can differ from zero, from one position (ray_weights.cuh): held by
// those instructions; a block forms an angle's position once and its pixels step
// from there.  One slice (ms, before / now): 725^2 x 720 14.7 / 1.4,
// 1449^2 x 900 66.0 / 6.2, 2049^2 x 1200 170.9 / 15.5.  V slices per thread; off:
// per-slice angle offsets or null (V = 1).
template <int V, int R>   // R: pixel rows a thread
__global__ void __launch_bounds__(256, V == 1 ? 6 : 1) k_adjoint_fx(const float* __restrict__ sino, const MmaAngle* __restrict__ ang,
                                                    const float* __restrict__ off, float* __restrict__ img, int N,
                                                    int T, float mid)
{
    __shared__ RayFrame frames[FX_CHUNK];
    __shared__ float4 slopes[FX_CHUNK];
    const int tid = threadIdx.y * 32 + threadIdx.x, x0 = blockIdx.x * 32 + 1, y0 = blockIdx.y * (8 * R) + 1;
    const int px = x0 + threadIdx.x, py = y0 + threadIdx.y * R;
    const size_t g = blockIdx.z;
    bool inside[R], any = false;   // the rim: k_adjoint_rim
    Lanes<float, V> acc[R];
#pragma unroll
    for (int r = 0; r < R; ++r) {
        inside[r] = px <= N && py + r <= N && !on_rim(px, py + r, N);
        any |= inside[r];
        acc[r] = Lanes<float, V>{};
    }
    const float* y = sino + g * T * N * V;
    for (int t0 = 0; t0 < T; t0 += FX_CHUNK) {
        const int n = min(FX_CHUNK, T - t0);
        __syncthreads();
        if (tid < n) {
            const MmaAngle a = ang[t0 + tid];
            frames[tid] = RayFrame(a.x, (float)(x0 + 16) - mid, (float)(y0 + 4 * R) - mid, off ? off[g * T + t0 + tid] : 0.f, mid);
            slopes[tid] = make_float4(a.c, a.s, a.t, 0.f);
        }
        __syncthreads();
        if (!any) continue;
#pragma unroll (V == 1 ? 2 : 1)
        for (int i = 0; i < n; ++i, y += (size_t)N * V) {
            RayFrame f = frames[i];
            f.move((int)threadIdx.x - 16, (int)threadIdx.y * R - 4 * R);
            MmaAngle a;
            a.c = slopes[i].x;
            a.s = slopes[i].y;
            a.t = slopes[i].z;
#pragma unroll
            for (int r = 0; r < R; ++r) {
                const RayPos p = f.pos();
                int j;
                float w[3];
                if (p.cu < 4 || p.cu > N - 4)
                    ray_weights<ENDS>(a, p, 0.f, mid, px, py + r, N, j, w);
                else
                    ray_weights<INNER>(a, p, 0.f, mid, px, py + r, N, j, w);
                add_rays<V>(acc[r], y, w, j, N);
                f.move(0, 1);
            }
        }
    }
#pragma unroll
    for (int r = 0; r < R; ++r)
        if (inside[r]) put_image<V>(img, acc[r], g, px, py + r, N);
}

// The pixels on the rim, whose samples may lie outside and are looked at one by one: 40 times the work, so in a kernel
// of their own (in k_adjoint_fx their warps would be the last to end).  One pixel per warp, its lanes sharing out the angles (grid.x: 6 N pixels, grid.y: slices).
template <int V>
__global__ void __launch_bounds__(256) k_adjoint_rim(const float* __restrict__ sino, const MmaAngle* __restrict__ ang,
                                                     const float* __restrict__ off, float* __restrict__ img, int N,
                                                     int T, float mid)
{
    const int i = blockIdx.x * 8 + (threadIdx.x >> 5), lane = threadIdx.x & 31, side = i / N, at = i % N + 1;
    if (side > 5) return;
    // columns 1, 2, N and rows 1, 2, N (corners twice, with the same value)
    const int edge = side % 3 == 2 ? N : side % 3 + 1;
    const int px = side < 3 ? edge : at, py = side < 3 ? at : edge;
    const size_t g = blockIdx.y;
    Lanes<float, V> acc{};
    if (px >= 2 && py >= 2)   // a pixel of the first column or row is never a tap (taps span 2..N)
        for (int t = lane; t < T; t += 32) {
            int j;
            float w[3];
            const MmaAngle a = ang[t];
            const float o = off ? off[g * T + t] : 0.f;
            ray_weights<RIM>(a, ray_pos(a.x, (float)px - mid, (float)py - mid, o, mid), o, mid, px, py, N, j, w);
            add_rays<V>(acc, sino + (g * T + t) * N * V, w, j, N);
        }
#pragma unroll
    for (int k = 0; k < V; ++k)
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) acc.v[k] += __shfl_down_sync(0xffffffffu, acc.v[k], o);
    if (lane == 0) put_image<V>(img, acc, g, px, py, N);
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

// f(first slice, slices, pairs of their images, pairs of the transposes), the slices' pairs made before
template <class F>
static void for_pairs(int N, int S, const float* img, float* buf, cudaStream_t st, F&& f)
{
    const size_t NN = (size_t)N * N;
    const int at_once = pair_slices(16 * NN, S);
    float2 *const P = reinterpret_cast<float2*>(buf), *const PT = P + NN * at_once;
    for (int s0 = 0; s0 < S; s0 += at_once) {
        const int n = std::min(at_once, S - s0);
        k_pair_images<<<dim3((N + 31) / 32, (N + 31) / 32, n), 256, 0, st>>>(img + s0 * NN, P, PT, N);
        f(s0, n, P, PT);
    }
}

void launch_radon_fx(const DevGeom<float>& g, int S, const float* img, float* IT, float* sino, cudaStream_t st)
{
    for_pairs(g.N, S, img, IT, st, [&](int s0, int n, const float2* P, const float2* PT) {
        k_ray_fx<<<dim3((g.N + 127) / 128, g.T, n), dim3(32, 4), 0, st>>>(
            P, PT, g.fx_fp, g.xsc_fp, g.fp_order, sino + (size_t)s0 * g.T * g.N, g.N, g.T, g.mid);
    });
}

void launch_ray_off(const DevGeom<float>& g, int S, const float* img, float* IT, const float* off, float* sino,
                    float* dsino, cudaStream_t st)
{
    for_pairs(g.N, S, img, IT, st, [&](int s0, int n, const float2* P, const float2* PT) {
        const dim3 blk(32, 4), grd((g.N + 127) / 128 * g.T, 1, n);
        const size_t at = (size_t)s0 * g.T;
        (dsino ? k_ray_off<true> : k_ray_off<false>)<<<grd, blk, 0, st>>>(
            P, PT, g.sc_fp, g.xsc_fp, g.fp_order, off ? off + at : nullptr, sino + at * g.N,
            dsino ? dsino + at * g.N : nullptr, g.N, g.T, g.mid);
    });
}

void launch_backproject_fx(const DevGeom<float>& g, int S, const float2* q, float* img, cudaStream_t st)
{
    const dim3 blk(32, 8);
    auto grid = [&](int r) { return dim3((g.N + 31) / 32, (g.N + 8 * r - 1) / (8 * r), S); };
    // rows per thread: more share an angle's entry, fewer keep the chip busy.  Measured with 1 / 2 / 4 rows (us): 363^2 x
    // 360 50 / 54 / 94, 725^2 x 720 193 / 190 / 252, 1449^2 x 900 813 / 748 / 738
    if (g.N < 500)
        k_backproject_fx<1><<<grid(1), blk, 0, st>>>(q, g.cmask, g.xsc_bp, img, g.N, g.T, g.mid);
    else if (g.N < 1000)
        k_backproject_fx<2><<<grid(2), blk, 0, st>>>(q, g.cmask, g.xsc_bp, img, g.N, g.T, g.mid);
    else
        k_backproject_fx<4><<<grid(4), blk, 0, st>>>(q, g.cmask, g.xsc_bp, img, g.N, g.T, g.mid);
}

template <int V>
void launch_adjoint_fx(const DevGeom<float>& g, int G, const float* sino, const float* off, float* img, cudaStream_t st)
{
    // rows per thread: more share an angle's entry, fewer keep the chip busy.  Measured with 1 / 2 / 4 rows (ms): 725^2 x
    // 720 1.47 / 1.44 / 1.77, two of 1025^2 x 600 4.36 / 4.23 / 4.30, 1449^2 x 900 6.58 / 6.43 / 6.35
    auto run = [&](auto kernel, int rows) {
        kernel<<<dim3((g.N + 31) / 32, (g.N + 8 * rows - 1) / (8 * rows), G), dim3(32, 8), 0, st>>>(sino, g.angles, off, img,
                                                                                                 g.N, g.T, g.mid);
    };
    if (g.N < 500)
        run(k_adjoint_fx<V, 1>, 1);
    else if (g.N < 1400 || V > 1)
        run(k_adjoint_fx<V, 2>, 2);
    else
        run(k_adjoint_fx<V, 4>, 4);
    k_adjoint_rim<V><<<dim3((6 * g.N + 7) / 8, G), 256, 0, st>>>(sino, g.angles, off, img, g.N, g.T, g.mid);
}
template void launch_adjoint_fx<1>(const DevGeom<float>&, int, const float*, const float*, float*, cudaStream_t);
template void launch_adjoint_fx<4>(const DevGeom<float>&, int, const float*, const float*, float*, cudaStream_t);

void launch_pairs(const float* q, float2* out, int N, size_t n, cudaStream_t st)
{
    k_pairs<<<(unsigned)std::min<size_t>((n + 255) / 256, (size_t)152 * 32), 256, 0, st>>>(q, out, N, n);
}

}  // namespace acu

// FFT form of iradon's ramp filter (tomography/tv_hpc.F90:93-105).
//
// The reference convolves every sinogram column directly with the 2N+1 taps
// (O(N^2) per column).  Here each block packs two real columns into one
// complex signal z = a + i b, zero-pads it to L >= 2N-2 (a power of two),
// and computes y = IFFT(H . FFT(z)) with H the real spectrum of the wrapped,
// symmetric tap sequence (computed in double on the host, 1/L folded in).
// Because H is real, Re(y) and Im(y) are the two filtered columns.  In single
// precision at L = 512 to 4096 (grids 130 to 2049) the transforms are passes of
// radix 16, L / 256 and 16 held in registers (k_filter_fft_r16); otherwise radix-4
// Stockham stages (a radix-2 stage last when log2 L is odd) in shared memory.
// All twiddles come from double-precision-built tables.
#include "common.cuh"
#include "kernels.h"

namespace acu {

template <typename Real>
struct Cplx;
template <>
struct Cplx<float> {
    using T = float2;
};
template <>
struct Cplx<double> {
    using T = double2;
};

template <typename C>
__device__ __forceinline__ C cmul(C a, C b)
{
    C r;
    r.x = a.x * b.x - a.y * b.y;
    r.y = a.x * b.y + a.y * b.x;
    return r;
}
template <typename C>
__device__ __forceinline__ C cadd(C a, C b)
{
    C r;
    r.x = a.x + b.x;
    r.y = a.y + b.y;
    return r;
}
template <typename C>
__device__ __forceinline__ C csub(C a, C b)
{
    C r;
    r.x = a.x - b.x;
    r.y = a.y - b.y;
    return r;
}

// Forward DFT of length L (power of two >= 16) held in d0; returns the buffer
// holding the natural-order result (d0 or d1).
// Ns and L are powers of two: indices are formed with shifts and masks.
template <typename C>
__device__ C* fft_stockham(C* d0, C* d1, const C* __restrict__ tw, int L)
{
    const int lgL = 31 - __clz(L);
    for (int Ns = 1, lgNs = 0; Ns < L;) {
        const int R = ((lgL - lgNs) >= 2) ? 4 : 2;
        const int lgR = R == 4 ? 2 : 1;
        const int stride = L >> (lgNs + lgR);
        const int nb = L >> lgR;
        for (int j = threadIdx.x; j < nb; j += blockDim.x) {
            const int k = j & (Ns - 1);
            const int idxD = ((j >> lgNs) << (lgNs + lgR)) + k;
            if (R == 4) {
                C v0 = d0[j];
                C v1 = cmul(d0[j + nb], tw[k * stride]);
                C v2 = cmul(d0[j + 2 * nb], tw[2 * k * stride]);
                C v3 = cmul(d0[j + 3 * nb], tw[3 * k * stride]);
                C a = cadd(v0, v2), b = csub(v0, v2), c = cadd(v1, v3), e = csub(v1, v3);
                C d;               // e * (-i)
                d.x = e.y;
                d.y = -e.x;
                d1[idxD] = cadd(a, c);
                d1[idxD + Ns] = cadd(b, d);
                d1[idxD + 2 * Ns] = csub(a, c);
                d1[idxD + 3 * Ns] = csub(b, d);
            } else {
                C v0 = d0[j];
                C v1 = cmul(d0[j + nb], tw[k * stride]);
                d1[idxD] = cadd(v0, v1);
                d1[idxD + Ns] = csub(v0, v1);
            }
        }
        __syncthreads();
        C* t = d0;
        d0 = d1;
        d1 = t;
        Ns <<= lgR;
        lgNs += lgR;
    }
    return d0;
}

// One block filters two real columns: (a, b) with element n at a[n*stride],
// b[n*stride] (b may be null: treated as zero and not written).
template <typename Real>
__global__ void __launch_bounds__(512) k_filter_fft(const Real* __restrict__ sino, Real* __restrict__ out,
                                                    const Real* __restrict__ H,
                                                    const typename Cplx<Real>::T* __restrict__ tw, int N, int T,
                                                    int L, int V, bool pairs)
{
    using C = typename Cplx<Real>::T;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    C* d0 = reinterpret_cast<C*>(smem_raw);
    C* d1 = d0 + L;
    const int g = blockIdx.y;
    size_t offa, offb;
    int stride;
    bool has_b = true;
    if (V == 4) {
        const int t = blockIdx.x >> 1, h = blockIdx.x & 1;
        offa = (((size_t)g * T + t) * N) * 4 + 2 * h;
        offb = offa + 1;
        stride = 4;
    } else {
        const int t0 = 2 * blockIdx.x;
        offa = ((size_t)g * T + t0) * N;
        offb = offa + N;
        stride = 1;
        has_b = (t0 + 1) < T;
    }
    // 4-slice lanes: the two columns of a half-lane sit side by side (8 or 16
    // bytes, aligned), so they move as one vector
    for (int n = threadIdx.x; n < L; n += blockDim.x) {
        C z;
        if (V == 4) {
            z = n < N ? __ldg(reinterpret_cast<const C*>(sino + offa + (size_t)n * 4)) : C{Real(0), Real(0)};
        } else {
            z.x = n < N ? sino[offa + (size_t)n * stride] : Real(0);
            z.y = (n < N && has_b) ? sino[offb + (size_t)n * stride] : Real(0);
        }
        d0[n] = z;
    }
    __syncthreads();
    C* res = fft_stockham<C>(d0, d1, tw, L);
    C* other = (res == d0) ? d1 : d0;
    // W = H/L * conj(Z); y = conj(FFT(W))
    for (int m = threadIdx.x; m < L; m += blockDim.x) {
        C z = res[m];
        const Real h = H[m];
        C w;
        w.x = h * z.x;
        w.y = -h * z.y;
        res[m] = w;
    }
    __syncthreads();
    C* y = fft_stockham<C>(res, other, tw, L);
    for (int n = threadIdx.x; n < N; n += blockDim.x) {
        const C v = y[n];
        if (pairs) {   // (bin, next bin), zeros in the first and the last
            const bool in = n > 0 && n < N - 1;
            const C w = y[in ? n + 1 : n];
            reinterpret_cast<C*>(out + 2 * offa)[n] = in ? C{v.x, w.x} : C{Real(0), Real(0)};
            if (has_b) reinterpret_cast<C*>(out + 2 * offb)[n] = in ? C{-v.y, -w.y} : C{Real(0), Real(0)};
        } else if (V == 4) {
            *reinterpret_cast<C*>(out + offa + (size_t)n * 4) = C{v.x, -v.y};
        } else {
            out[offa + (size_t)n * stride] = v.x;
            if (has_b) out[offb + (size_t)n * stride] = -v.y;
        }
    }
}

// ---- L = 256 M, M = 2, 4, 8, 16, in single precision: passes of radix 16, M, 16 ------
// Each of 16 M threads holds 16 values of a pass: those j + 16 M m of the first
// and the last, read from the shared buffer, multiplied by the pass's twiddles,
// transformed (16 points as 4 x 4: 4-point DFTs, the internal twiddles w16^(m1 q2),
// 4-point DFTs) and written to their Stockham places.  The first pass reads the
// sinogram itself; the last pass's values are those that the inverse
// transform's first pass needs, so the spectrum never leaves the registers; the
// last pass writes the result.  That leaves four exchanges through shared memory
// per filtered pair, of eight with separate transforms (its data pipe was 93 % busy
// with radix-4 stages).  One buffer per transform, padded by one slot per 16 so that the
// strided writes of the first pass spread over the banks.
// Measured (us, before / now; before: radix-4 stages, three separate radix-16
// passes at L = 4096): 257 x 180 angles, 64 slices 63 / 15; 513 x 360, 64 slices 213 / 49;
// 725 x 720 22.5 / 8.4; 1025 x 600, 64 slices 788 / 183; 1449 x 900 18.0 / 13.0;
// 2049 x 300, 64 slices 294 / 186.  Fewer registers for more warps (128 now) gained nothing.
__device__ __forceinline__ int pad16(int i) { return i + (i >> 4); }

// (a0..a3) -> their 4-point DFT, e^(-2 pi i / 4) = -i
__device__ __forceinline__ void dft4(float2& a0, float2& a1, float2& a2, float2& a3)
{
    const float2 t0 = cadd(a0, a2), t1 = csub(a0, a2), t2 = cadd(a1, a3), e = csub(a1, a3);
    const float2 t3 = make_float2(e.y, -e.x);   // e * (-i)
    a0 = cadd(t0, t2);
    a1 = cadd(t1, t3);
    a2 = csub(t0, t2);
    a3 = csub(t1, t3);
}

// a times the constant (rh + rl) + i (ih + il): constants in two parts, as their
// rounding would otherwise be in every value (a filtered row's error 1.5e-7
// instead of 1.8e-7 at L = 4096, 1.7e-7 with radix-4 stages)
__device__ __forceinline__ float2 cmul_const(float2 a, float rh, float rl, float ih, float il)
{
    return make_float2(fmaf(a.x, rh, -fmaf(a.y, ih, fmaf(a.y, il, -(a.x * rl)))),
                       fmaf(a.x, ih, fmaf(a.y, rh, fmaf(a.y, rl, a.x * il))));
}

// cos(pi/8), sin(pi/8), sqrt(1/2)
constexpr double C8 = 0.92387953251128675613, S8 = 0.38268343236508977173, R2 = 0.70710678118654752440;

__device__ __forceinline__ float2 mul_w(float2 a, double re, double im)   // re, im: compile-time constants
{
    return cmul_const(a, (float)re, (float)(re - (double)(float)re), (float)im, (float)(im - (double)(float)im));
}

// x -> its 16-point DFT y, y[q2 + 4 q1] = sum_m x[m] w16^(m (q2 + 4 q1)),
// m = m1 + 4 m2; the result is returned in x in natural order
__device__ __forceinline__ void dft16(float2 (&x)[16])
{
#pragma unroll
    for (int m1 = 0; m1 < 4; ++m1) dft4(x[m1], x[m1 + 4], x[m1 + 8], x[m1 + 12]);   // over m2 -> q2 = 0..3
    // x[m1 + 4 q2] *= w16^(m1 q2)
    x[5] = mul_w(x[5], C8, -S8);     // 1
    x[9] = mul_w(x[9], R2, -R2);     // 2
    x[13] = mul_w(x[13], S8, -C8);   // 3
    x[6] = mul_w(x[6], R2, -R2);     // 2
    x[10] = make_float2(x[10].y, -x[10].x);   // 4: -i
    x[14] = mul_w(x[14], -R2, -R2);  // 6
    x[7] = mul_w(x[7], S8, -C8);     // 3
    x[11] = mul_w(x[11], -R2, -R2);  // 6
    x[15] = mul_w(x[15], -C8, S8);   // 9
#pragma unroll
    for (int q2 = 0; q2 < 4; ++q2) dft4(x[4 * q2], x[4 * q2 + 1], x[4 * q2 + 2], x[4 * q2 + 3]);   // over m1 -> q1
    // now x[4 q2 + q1] holds y[q2 + 4 q1]: transpose the 4 x 4 index
    float2 y[16];
#pragma unroll
    for (int q2 = 0; q2 < 4; ++q2)
#pragma unroll
        for (int q1 = 0; q1 < 4; ++q1) y[q2 + 4 * q1] = x[4 * q2 + q1];
#pragma unroll
    for (int r = 0; r < 16; ++r) x[r] = y[r];
}

// x[0..R-1] -> their R-point DFT in natural order
template <int R>
__device__ __forceinline__ void dft(float2* x)
{
    if constexpr (R == 2) {
        const float2 a = cadd(x[0], x[1]), b = csub(x[0], x[1]);
        x[0] = a;
        x[1] = b;
    } else if constexpr (R == 4) {
        dft4(x[0], x[1], x[2], x[3]);
    } else if constexpr (R == 8) {
        float2 e[4] = {x[0], x[2], x[4], x[6]}, o[4] = {x[1], x[3], x[5], x[7]};
        dft4(e[0], e[1], e[2], e[3]);
        dft4(o[0], o[1], o[2], o[3]);
        o[1] = mul_w(o[1], R2, -R2);
        o[2] = make_float2(o[2].y, -o[2].x);
        o[3] = mul_w(o[3], -R2, -R2);
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            x[q] = cadd(e[q], o[q]);
            x[q + 4] = csub(e[q], o[q]);
        }
    } else {
        dft16(*reinterpret_cast<float2(*)[16]>(x));
    }
}

// The passes after the first of a DFT of 256 M points: the first pass's outputs
// x (thread j: places 16 j + r) -> the thread's values j + 16 M r.
// tw1: [M - 1][16] = w^(m k 16), tw2: [15][16 M] = w^(m k), w = e^(-2 pi i / L)
template <int M>
__device__ __forceinline__ void fft_passes(float2 (&x)[16], float2* b, int j, const float2* __restrict__ tw1,
                                           const float2* __restrict__ tw2)
{
    constexpr int TH = 16 * M;
#pragma unroll
    for (int r = 0; r < 16; ++r) b[pad16(16 * j + r)] = x[r];
    __syncthreads();
#pragma unroll
    for (int q = 0; q < 16 / M; ++q)
#pragma unroll
        for (int m = 0; m < M; ++m) x[q * M + m] = b[pad16(j + q * TH + 256 * m)];
    __syncthreads();
#pragma unroll
    for (int q = 0; q < 16 / M; ++q) {
        const int jj = j + q * TH, k = jj & 15;
#pragma unroll
        for (int m = 1; m < M; ++m) x[q * M + m] = cmul(x[q * M + m], __ldg(tw1 + (m - 1) * 16 + k));
        dft<M>(x + q * M);
#pragma unroll
        for (int r = 0; r < M; ++r) b[pad16((jj >> 4) * TH + k + 16 * r)] = x[q * M + r];
    }
    __syncthreads();
#pragma unroll
    for (int m = 0; m < 16; ++m) x[m] = b[pad16(j + TH * m)];
    __syncthreads();
#pragma unroll
    for (int m = 1; m < 16; ++m) x[m] = cmul(x[m], __ldg(tw2 + (m - 1) * TH + j));
    dft16(x);
}

// k_filter_fft for these lengths: RB column pairs per block of 16 M RB threads.
template <int M, int RB>
__global__ void __launch_bounds__(16 * M * RB) k_filter_fft_r16(const float* __restrict__ sino, float* __restrict__ out,
                                                                const float* __restrict__ H,
                                                                const float2* __restrict__ tw16, int N, int T, int V,
                                                                bool pairs)
{
    constexpr int L = 256 * M, TH = 16 * M;
    __shared__ float2 s_b[RB][L + L / 16];
    const int j = threadIdx.x % TH, col = blockIdx.x * RB + threadIdx.x / TH, g = blockIdx.y;
    float2* const b = s_b[threadIdx.x / TH];
    const float2* const tw2 = tw16 + (M - 1) * 16;
    size_t offa, offb;
    bool live, has_b = true;
    if (V == 4) {
        offa = (((size_t)g * T + (col >> 1)) * N) * 4 + 2 * (col & 1);
        offb = offa + 1;
        live = col < 2 * T;
    } else {
        const int t0 = 2 * col;
        offa = ((size_t)g * T + t0) * N;
        offb = offa + N;
        live = t0 < T;
        has_b = t0 + 1 < T;
    }
    float2 x[16];
#pragma unroll
    for (int m = 0; m < 16; ++m) {
        const int n = j + TH * m;
        x[m] = make_float2(0.f, 0.f);
        if (live && n < N) {
            if (V == 4) {
                x[m] = __ldg(reinterpret_cast<const float2*>(sino + offa + (size_t)n * 4));
            } else {
                x[m].x = sino[offa + n];
                if (has_b) x[m].y = sino[offb + n];
            }
        }
    }
    dft16(x);
    fft_passes<M>(x, b, j, tw16, tw2);
    // W = H/L * conj(Z); y = conj(FFT(W))
#pragma unroll
    for (int r = 0; r < 16; ++r) {
        const float h = __ldg(H + j + TH * r);
        x[r] = make_float2(h * x[r].x, -h * x[r].y);
    }
    dft16(x);
    fft_passes<M>(x, b, j, tw16, tw2);
    if (pairs) {   // (bin, next bin), zeros in the first and the last
#pragma unroll
        for (int r = 0; r < 16; ++r) b[pad16(j + TH * r)] = x[r];
        __syncthreads();
    }
    if (!live) return;
#pragma unroll
    for (int r = 0; r < 16; ++r) {
        const int n = j + TH * r;
        if (n >= N) continue;
        const float2 v = x[r];
        if (pairs) {
            const bool in = n > 0 && n < N - 1;
            const float2 w = b[pad16(in ? n + 1 : n)];
            reinterpret_cast<float2*>(out + 2 * offa)[n] = in ? make_float2(v.x, w.x) : make_float2(0.f, 0.f);
            if (has_b)
                reinterpret_cast<float2*>(out + 2 * offb)[n] = in ? make_float2(-v.y, -w.y) : make_float2(0.f, 0.f);
        } else if (V == 4) {
            *reinterpret_cast<float2*>(out + offa + (size_t)n * 4) = make_float2(v.x, -v.y);
        } else {
            out[offa + n] = v.x;
            if (has_b) out[offb + n] = -v.y;
        }
    }
}

template <int M, int RB>
void filter_fft_r16(const DevGeom<float>& g, int G, int V, const float* sino, float* out, const float* H, bool pairs,
                    cudaStream_t st)
{
    const int cols = V == 4 ? 2 * g.T : (g.T + 1) / 2;
    k_filter_fft_r16<M, RB><<<dim3((cols + RB - 1) / RB, G), 16 * M * RB, 0, st>>>(sino, out, H, g.fft_tw16, g.N, g.T, V,
                                                                                   pairs);
}

template <typename Real, int V>
void launch_filter_fft(const DevGeom<Real>& g, int G, const Real* sino, Real* out, cudaStream_t st, bool pairs)
{
    using C = typename Cplx<Real>::T;
    const size_t sm = 2 * (size_t)g.fft_L * sizeof(C);
    max_dynamic_smem<k_filter_fft<Real>>();
    const C* tw = reinterpret_cast<const C*>(sizeof(Real) == 4 ? (const void*)g.fft_tw : (const void*)g.fft_tw64);
    dim3 grd(V == 4 ? 2 * g.T : (g.T + 1) / 2, G);
    // 512 threads: 8 % faster than 256 at L = 4096 (more warps between the
    // stages' barriers), 1024 slower; the results do not depend on it
    // exact positions filter with the spectrum of the FP64 taps
    const Real* H = (g.exact && g.fft_h_x) ? g.fft_h_x : g.fft_h;
    if constexpr (sizeof(Real) == 4) {
        // column pairs per block: the two of a 4-slice lane together, and 128 threads or more
        if (g.fft_tw16) {
            if (g.fft_L == 4096)
                return filter_fft_r16<16, 1>(g, G, V, sino, out, H, pairs, st);
            if (g.fft_L == 2048)
                return filter_fft_r16<8, 2>(g, G, V, sino, out, H, pairs, st);
            if (g.fft_L == 1024)
                return filter_fft_r16<4, 2>(g, G, V, sino, out, H, pairs, st);
            if (g.fft_L == 512)
                return filter_fft_r16<2, 4>(g, G, V, sino, out, H, pairs, st);
        }
    }
    k_filter_fft<Real><<<grd, 512, sm, st>>>(sino, out, H, tw, g.N, g.T, g.fft_L, V, pairs);
}

// Largest FFT length whose two shared-memory buffers fit in one block.
template <typename Real>
bool fft_fits(int L)
{
    return 2 * (size_t)L * 2 * sizeof(Real) <= 227 * 1024;
}

template void launch_filter_fft<float, 1>(const DevGeom<float>&, int, const float*, float*, cudaStream_t, bool);
template void launch_filter_fft<float, 4>(const DevGeom<float>&, int, const float*, float*, cudaStream_t, bool);
template void launch_filter_fft<double, 1>(const DevGeom<double>&, int, const double*, double*, cudaStream_t, bool);
template bool fft_fits<float>(int);
template bool fft_fits<double>(int);

}  // namespace acu

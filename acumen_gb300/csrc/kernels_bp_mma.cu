// Backprojection on the tensor cores for large batches (tomography/tv_hpc.F90:107-123,
// exact sample positions).
//
// For a tile of 16 x 16 pixels and one angle the update is a small matrix
// product: image [256 pixels x slices] += W [256 pixels x 24 bins] times the
// bins the tile meets [24 bins x slices]; W holds each pixel's two linear
// interpolation weights.  The gather kernel reads two bins per pixel, angle and
// slice through the L1 data path and forms the sample position once per four
// slices; here the position is formed once per 64 or 128 slices and the
// products run from shared memory.  Sums stay on the chip for all angles.
//
// Both operands are split in two halves, v = hi + lo with 11 bits each, after a
// power-of-two scale per slice for the sinogram; lo lo (2^-24 of a product) is
// left out.  The tensor core truncates when it adds, so a chain in tensor memory
// is two or four angles long; it is then added to FP32 sums in registers with
// rounding to nearest.
//
//   k_bp_max      largest magnitude of each slice's filtered sinogram
//   k_bp_bins     lane sinogram -> bins in operand layout [angle][8 slices, hi then lo][bin][8]
//   k_bp_mma      the products (tiles that meet the mask)
//   k_bp_zero     zeros in the other tiles
//   k_bp_flagged  plain gathers of slices with a value that is not finite or a few that dwarf the others, NaN if a wait gave up
#include <cuda.h>

#include <algorithm>
#include <cmath>
#include <vector>

#include "common.cuh"
#include "kernels.h"
#include "umma.cuh"

namespace acu {

namespace {

constexpr int TP = 16, PIX = TP * TP;
constexpr int NS = 64;                         // slices per block
constexpr int WIN = 24;                        // bins per angle: 15 (|s| + |c|) < 21.3 pixels and a tap each side
constexpr int PAIR = 2;                        // angles per stage: K = 48, three steps of 16
constexpr int KBLK = PAIR * WIN / 8;           // K blocks of 8
constexpr int W_PART = KBLK * 128 * 16;        // one half (hi or lo) of W for 128 pixels
constexpr int W_BYTES = 4 * W_PART;            // [hi, lo][pixels 0-127, 128-255]
constexpr uint32_t NONE = ~0u;                 // no place in shared memory
constexpr int W_STAGES = 2, Q_STAGES = 4;       // a tile's stages are padded to a multiple of W_STAGES

// 28 warps are launched with 72 registers a thread; the warps that add need more, the others less
constexpr int REG_ACC = 88, REG_REST = 48;

template <int BLK>
struct Bp {
    static constexpr int CHUNKS = 2 * BLK * NS / 8;            // of 8 slices: hi, then lo
    static constexpr int ANGLE_BYTES = CHUNKS * WIN * 16;
    static constexpr int Q_BYTES = PAIR * ANGLE_BYTES;
    static constexpr int CHAIN = BLK == 2 ? 1 : 2;             // stages added up in tensor memory
    static constexpr int PROD = 8, MMA = PROD, LOAD = PROD + 1, ACC = PROD + 4, WARPS = ACC + 8 * BLK;
    static constexpr int W = 0, Q = W_STAGES * W_BYTES, BARS = Q + Q_STAGES * Q_BYTES;
};

struct Shared {
    uint64_t w_full[W_STAGES], w_empty[W_STAGES], q_full[Q_STAGES], q_empty[Q_STAGES], d_full[2], d_empty[2], drained;
    uint32_t tmem;
};
static_assert(Bp<2>::BARS + sizeof(Shared) <= 227 * 1024, "smem");

// First bin of a tile's window at one angle (1-based).
__device__ __forceinline__ int window_bin(float4 x, float mid, int x0, int y0)
{
    const float s = x.x + x.z, c = x.y + x.w;
    const float dx = (float)(s >= 0.f ? x0 : x0 + TP - 1) - mid, dy = (float)(c >= 0.f ? y0 : y0 + TP - 1) - mid;
    return (int)floorf(__fsub_rn(__fmaf_rn(s, dx, __fmaf_rn(c, dy, mid)), 0.01f));
}

__device__ __forceinline__ uint32_t pack(float a, float b)
{
    const __half2 h = __floats2half2_rn(a, b);
    return *reinterpret_cast<const uint32_t*>(&h);
}

__device__ __forceinline__ uint64_t desc(uint32_t addr, uint32_t lbo, uint32_t sbo)
{
    return (uint64_t)((addr & 0x3ffffu) >> 4) | ((uint64_t)(lbo >> 4) << 16) | ((uint64_t)(sbo >> 4) << 32) |
           (1ull << 46);
}

// A block walks the tiles list[blockIdx.x], + gridDim.x, ...  Roles by warp:
//   0..7    form W, one pixel per lane: both angles of a stage
//   8       issues the products
//   9       loads the bins (one lane), one box per angle
//   12..    add the chains up in registers (64 slices of one pixel per lane) and write the tile
// Waits are bounded; one that gives up sets *err, and k_bp_flagged then writes
// NaN: the block leaves its other tiles as they were.
template <int BLK>
__global__ void __launch_bounds__(32 * Bp<BLK>::WARPS, 1) k_bp_mma(const __grid_constant__ CUtensorMap bins,
                                                                   const float4* __restrict__ xsc,
                                                                   const int* __restrict__ list, int ntiles,
                                                                   const float* __restrict__ cmask,
                                                                   const float* __restrict__ scale,
                                                                   float* __restrict__ img, int N, int T, int nt, int G,
                                                                   int g0, float mid, int* err)
{
    using B = Bp<BLK>;
    extern __shared__ __align__(128) unsigned char sm[];
    Shared& sh = *reinterpret_cast<Shared*>(sm + B::BARS);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int nst = (T + PAIR * W_STAGES - 1) / (PAIR * W_STAGES) * W_STAGES;   // stages per tile
    if (threadIdx.x == 0) {
        for (int i = 0; i < W_STAGES; ++i) {
            umma::bar_init(&sh.w_full[i], B::PROD);
            umma::bar_init(&sh.w_empty[i], 1);
        }
        for (int i = 0; i < Q_STAGES; ++i) {
            umma::bar_init(&sh.q_full[i], 1);
            umma::bar_init(&sh.q_empty[i], 1);
        }
        for (int i = 0; i < 2; ++i) {
            umma::bar_init(&sh.d_full[i], 1);
            umma::bar_init(&sh.d_empty[i], 8 * BLK);
        }
        umma::bar_init(&sh.drained, 1);
        umma::bar_init_fence();
    }
    if (warp == B::MMA) umma::tmem_alloc<512>(&sh.tmem);
    for (int i = threadIdx.x; i < W_STAGES * W_BYTES / 16; i += blockDim.x)
        reinterpret_cast<uint4*>(sm + B::W)[i] = make_uint4(0, 0, 0, 0);
    umma::fence_async_smem();
    umma::fence_before();
    __syncthreads();
    umma::fence_after();
    const uint32_t tmem = sh.tmem;
    bool ok = true;

    if (warp < B::PROD) {
        if constexpr (BLK == 2) umma::setmaxnreg_dec<REG_REST>();
        // pixel = row of W: half m of the tile, row p % 128
        const int p = threadIdx.x, m = p >> 7;
        const uint32_t row = B::W + m * W_PART + (p & 127) * 16;
        uint32_t last[W_STAGES][PAIR][2];   // words written last time
#pragma unroll
        for (int i = 0; i < W_STAGES; ++i)
#pragma unroll
            for (int a = 0; a < PAIR; ++a) last[i][a][0] = last[i][a][1] = NONE;
        auto put = [&](uint32_t at, uint32_t hi, uint32_t lo) {
            if (at != NONE) {
                *reinterpret_cast<uint32_t*>(sm + at) = hi;
                *reinterpret_cast<uint32_t*>(sm + at + 2 * W_PART) = lo;
            }
        };
        unsigned n = 0;   // rounds through the stages
        for (int it = blockIdx.x; it < ntiles && ok; it += gridDim.x) {
            const int tile = list[it];
            const int x0 = (tile % nt) * TP + 1, y0 = (tile / nt) * TP + 1;
            const float dx = (float)(x0 + (p & 15)) - mid, dy = (float)(y0 + (p >> 4)) - mid;
            for (int s0 = 0; s0 < nst && ok; s0 += W_STAGES, ++n) {
#pragma unroll
                for (int st = 0; st < W_STAGES; ++st) {
                    uint32_t at[PAIR][2], hi[PAIR][2], lo[PAIR][2];
#pragma unroll
                    for (int a = 0; a < PAIR; ++a) {
                        const int t = (s0 + st) * PAIR + a;
                        at[a][0] = at[a][1] = NONE;
                        if (t < T) {
                            const float4 x = __ldg(xsc + t);
                            float cell, wh;
                            exact_coord(x.x, x.y, x.z, x.w, dx, dy, mid, cell, wh);
                            const int y1 = (int)cell;
                            if (y1 > 1 && y1 < N) {
                                const int k = y1 - window_bin(x, mid, x0, y0);
                                const float wl = 1.f - wh;
                                // the leading 11 bits are exact in half precision, the rest is rounded
                                const float hl = __uint_as_float(__float_as_uint(wl) & 0xffffe000u);
                                const float hh = __uint_as_float(__float_as_uint(wh) & 0xffffe000u);
                                const int sft = (k & 1) << 4;   // bins k, k + 1 in words k / 2 and the next
                                const uint32_t ph = pack(hl, hh), pl = pack(wl - hl, wh - hh);
                                hi[a][0] = ph << sft;
                                hi[a][1] = __funnelshift_l(ph, 0, sft);
                                lo[a][0] = pl << sft;
                                lo[a][1] = __funnelshift_l(pl, 0, sft);
                                const int w = k >> 1;
                                if ((unsigned)k < (unsigned)(WIN - 1)) {   // always, by the window's choice
                                    const uint32_t b = row + st * W_BYTES + a * (WIN / 8) * 2048;
                                    at[a][0] = b + (w >> 2) * 2048 + (w & 3) * 4;
                                    at[a][1] = sft ? b + ((w + 1) >> 2) * 2048 + ((w + 1) & 3) * 4 : NONE;
                                }
                            }
                        }
                    }
                    ok = umma::bar_wait_warp(&sh.w_empty[st], (n & 1) ^ 1);
                    if (!ok) break;
#pragma unroll
                    for (int a = 0; a < PAIR; ++a) {
                        put(last[st][a][0], 0, 0);
                        put(last[st][a][1], 0, 0);
                    }
#pragma unroll
                    for (int a = 0; a < PAIR; ++a) {
                        put(at[a][0], hi[a][0], lo[a][0]);
                        put(at[a][1], hi[a][1], lo[a][1]);
                        last[st][a][0] = at[a][0];
                        last[st][a][1] = at[a][1];
                    }
                    umma::fence_async_smem();
                    __syncwarp();
                    if (lane == 0) umma::bar_arrive(&sh.w_full[st]);
                }
            }
        }
    } else if (warp < B::ACC) {
        if constexpr (BLK == 2) umma::setmaxnreg_dec<REG_REST>();
        if (warp == B::MMA) {
            constexpr uint32_t B_N_MAJOR = 1u << 16;
            constexpr uint32_t ID_128 = umma::instr_desc_f16(128, 128) | B_N_MAJOR,
                               ID_64 = umma::instr_desc_f16(128, 64) | B_N_MAJOR;
            constexpr uint32_t LO_OFF = BLK * (NS / 8) * WIN * 16 >> 4;   // lo bins, in descriptor units
            const uint32_t acc0 = __reduce_max_sync(0xffffffffu, tmem);   // the same in all lanes, and known to be
            const uint64_t w0 = umma::smem_desc(umma::smem_addr(sm + B::W), 2048);
            const uint32_t q0 = umma::smem_addr(sm + B::Q);
            // the three K steps of a stage: bins 0-15 of the first angle, 16-23 and 0-7 of the second, 8-23
            const uint64_t b0 = desc(q0, 128, WIN * 16), b1 = desc(q0 + 256, B::ANGLE_BYTES - 256, WIN * 16),
                           b2 = desc(q0 + B::ANGLE_BYTES + 128, 128, WIN * 16);
            unsigned n = 0;   // stages
            for (int it = blockIdx.x; it < ntiles && ok; it += gridDim.x) {
#pragma unroll 1
                for (int s = 0; s < nst; ++s, ++n) {
                    const unsigned m = n / B::CHAIN, ws = n % W_STAGES, qs = n % Q_STAGES;
                    const bool first = n % B::CHAIN == 0, last = n % B::CHAIN == B::CHAIN - 1;
                    if (first) ok = umma::bar_wait_warp(&sh.d_empty[m & 1], ((m >> 1) & 1) ^ 1);
                    ok = umma::bar_wait_warp(&sh.q_full[qs], (n / Q_STAGES) & 1) && ok;
                    ok = umma::bar_wait_warp(&sh.w_full[ws], (n / W_STAGES) & 1) && ok;
                    if (!ok) break;
                    umma::fence_after();
                    const uint64_t w = w0 + ws * (W_BYTES >> 4);
                    const uint32_t qo = qs * (B::Q_BYTES >> 4);
                    const uint64_t bq[3] = {b0 + qo, b1 + qo, b2 + qo};
#pragma unroll
                    for (int h = 0; h < 2; ++h) {   // pixels 0-127, 128-255
                        const uint32_t d = acc0 + (m & 1) * 256 + h * 128;
                        const uint64_t whi = w + (h * W_PART >> 4), wlo = whi + (2 * W_PART >> 4);
                        if constexpr (BLK == 1) {
                            // columns 0-63 hi hi, 64-127 the small products
#pragma unroll
                            for (int ks = 0; ks < 3; ++ks) {
                                umma::mma_f16(d, whi + (ks * 4096 >> 4), bq[ks], ID_128, !first || ks > 0);
                                umma::mma_f16(d + NS, wlo + (ks * 4096 >> 4), bq[ks], ID_64, true);
                            }
                        } else {
                            // the small products first, while the sums are small
#pragma unroll
                            for (int ks = 0; ks < 3; ++ks) {
                                umma::mma_f16(d, wlo + (ks * 4096 >> 4), bq[ks], ID_128, ks > 0);
                                umma::mma_f16(d, whi + (ks * 4096 >> 4), bq[ks] + LO_OFF, ID_128, true);
                            }
#pragma unroll
                            for (int ks = 0; ks < 3; ++ks) umma::mma_f16(d, whi + (ks * 4096 >> 4), bq[ks], ID_128, true);
                        }
                    }
                    umma::mma_commit(umma::smem_addr(&sh.w_empty[ws]));
                    umma::mma_commit(umma::smem_addr(&sh.q_empty[qs]));
                    if (last) umma::mma_commit(umma::smem_addr(&sh.d_full[m & 1]));
                }
            }
            // every MMA is done before the tensor memory is given back
            umma::mma_commit(umma::smem_addr(&sh.drained));
            ok = umma::bar_wait(&sh.drained, 0) && ok;
        } else if (warp == B::LOAD && lane == 0) {
            unsigned n = 0;
            for (int it = blockIdx.x; it < ntiles && ok; it += gridDim.x) {
                const int tile = list[it];
                const int x0 = (tile % nt) * TP + 1, y0 = (tile / nt) * TP + 1;
                for (int s = 0; s < nst; ++s, ++n) {
                    const unsigned qs = n % Q_STAGES;
                    int lo[PAIR];
#pragma unroll
                    for (int a = 0; a < PAIR; ++a) {
                        const int t = s * PAIR + a;
                        lo[a] = t < T ? window_bin(__ldg(xsc + t), mid, x0, y0) : 1;
                    }
                    ok = umma::bar_wait(&sh.q_empty[qs], ((n / Q_STAGES) & 1) ^ 1);
                    if (!ok) break;
                    umma::bar_expect(&sh.q_full[qs], B::Q_BYTES);
                    // whatever lies outside the sinogram (bins, angles) arrives as zeros
#pragma unroll
                    for (int a = 0; a < PAIR; ++a)
                        umma::tensor_load_3d(sm + B::Q + qs * B::Q_BYTES + a * B::ANGLE_BYTES, &bins, (lo[a] - 1) * 8, 0,
                                             s * PAIR + a, &sh.q_full[qs]);
                }
            }
            // loads in flight land before the block leaves
            for (unsigned i = n > Q_STAGES ? n - Q_STAGES : 0; i < n; ++i)
                umma::bar_wait(&sh.q_full[i % Q_STAGES], (i / Q_STAGES) & 1);
        }
        __syncwarp();
    } else {
        if constexpr (BLK == 2) umma::setmaxnreg_inc<REG_ACC>();
        const int aw = warp - B::ACC, h = (aw >> 2) & 1, k = aw >> 3;
        const int p = h * 128 + (warp & 3) * 32 + lane;
        unsigned m = 0;
        for (int it = blockIdx.x; it < ntiles && ok; it += gridDim.x) {
            const int tile = list[it];
            float2 sum[NS / 2];
#pragma unroll
            for (int i = 0; i < NS / 2; ++i) sum[i] = make_float2(0.f, 0.f);
#pragma unroll 1
            for (int s = 0; s < nst; s += B::CHAIN, ++m) {
                ok = umma::bar_wait_warp(&sh.d_full[m & 1], (m >> 1) & 1);
                if (!ok) break;
                umma::fence_after();
                const uint32_t d = tmem + ((uint32_t)((warp & 3) * 32) << 16) + (m & 1) * 256 + h * 128 + (BLK == 2 ? k * NS : 0);
#pragma unroll
                for (int c = 0; c < NS / 8; ++c) {
                    float2 v[4];
                    umma::tmem_ld8(d + 8 * c, v);
                    if constexpr (BLK == 1) {
                        float2 x[4];
                        umma::tmem_ld8(d + NS + 8 * c, x);
                        umma::tmem_ld_wait(v, x);
#pragma unroll
                        for (int i = 0; i < 4; ++i) sum[4 * c + i] = add2(sum[4 * c + i], add2(v[i], x[i]));
                    } else {
                        umma::tmem_ld_wait(v);
#pragma unroll
                        for (int i = 0; i < 4; ++i) sum[4 * c + i] = add2(sum[4 * c + i], v[i]);
                    }
                }
                umma::fence_before();
                __syncwarp();
                if (lane == 0) umma::bar_arrive(&sh.d_empty[m & 1]);
            }
            const int x = (tile % nt) * TP + (p & 15), y = (tile / nt) * TP + (p >> 4);
            if (x < N && y < N) {
                const size_t NN = (size_t)N * N, pix = (size_t)y * N + x;
                const float cm = cmask[pix];
#pragma unroll
                for (int i = 0; i < NS / 4; ++i) {
                    const int g = g0 + k * (NS / 4) + i;
                    if (g < G) {
                        const float4 f = __ldg(reinterpret_cast<const float4*>(scale) + g);
                        const float2 a = mul2(mul2(sum[2 * i], make_float2(f.x, f.y)), make_float2(cm, cm));
                        const float2 b = mul2(mul2(sum[2 * i + 1], make_float2(f.z, f.w)), make_float2(cm, cm));
                        reinterpret_cast<float4*>(img)[(size_t)g * NN + pix] = make_float4(a.x, a.y, b.x, b.y);
                    }
                }
            }
        }
    }
    if (!ok) atomicExch(err, 1);
    umma::fence_before();
    __syncthreads();
    if (warp == B::MMA) umma::tmem_free<512>(tmem);
}

// Largest magnitude (as bits) of every slice; a NaN or an infinity compares above all finite values.
__global__ void __launch_bounds__(256) k_bp_max(const float4* __restrict__ q, unsigned* __restrict__ top, size_t npos)
{
    __shared__ unsigned s_top[4];
    if (threadIdx.x < 4) s_top[threadIdx.x] = 0;
    __syncthreads();
    const float4* qg = q + (size_t)blockIdx.y * npos;
    unsigned m[4] = {0, 0, 0, 0};
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < npos; i += (size_t)gridDim.x * blockDim.x) {
        const float4 v = __ldg(qg + i);
        m[0] = max(m[0], __float_as_uint(v.x) & 0x7fffffffu);
        m[1] = max(m[1], __float_as_uint(v.y) & 0x7fffffffu);
        m[2] = max(m[2], __float_as_uint(v.z) & 0x7fffffffu);
        m[3] = max(m[3], __float_as_uint(v.w) & 0x7fffffffu);
    }
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        m[k] = __reduce_max_sync(0xffffffffu, m[k]);
        if ((threadIdx.x & 31) == 0) atomicMax(&s_top[k], m[k]);
    }
    __syncthreads();
    if (threadIdx.x < 4) atomicMax(top + blockIdx.y * 4 + threadIdx.x, s_top[threadIdx.x]);
}

// power of two that brings the largest magnitude into [2^14, 2^15), as its exponent
__device__ __forceinline__ int scale_exp(unsigned top)
{
    return top && top < 0x7f800000u ? max((int)(top >> 23) - 127, -98) : 0;
}

// One bin and angle per thread (grid.x: 128 bins of every angle, of which there may be more than a grid has
// rows): its 64 slices of block blockIdx.y as eight pieces of hi and eight of lo halves.  A half ends at 2^-24, so a value
// keeps 23 bits down to 2^-16 of its slice's largest and 19 down to 2^-20: brief counts the values below that.
__global__ void __launch_bounds__(128) k_bp_bins(const float4* __restrict__ q, const unsigned* __restrict__ top,
                                                 float* __restrict__ scale, unsigned* __restrict__ brief,
                                                 uint4* __restrict__ bins, int N, int T, int G, int g0)
{
    const int nb = (N + 127) / 128, t = blockIdx.x / nb, k = blockIdx.y;
    const int i = (blockIdx.x - t * nb) * 128 + threadIdx.x;
    uint4* const out = bins + (size_t)t * gridDim.y * (2 * NS / 8) * N + i;
    unsigned long long few = 0;   // slices whose value keeps fewer bits than others
#pragma unroll 2
    for (int c = 0; c < NS / 8; ++c) {
        __align__(16) __half hi[8], lo[8];
#pragma unroll
        for (int e = 0; e < 2; ++e) {
            const int g = g0 + k * (NS / 4) + 2 * c + e;
            float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
            uint4 m = make_uint4(0, 0, 0, 0);
            if (g < G && i < N) {
                v = __ldg(q + ((size_t)g * T + t) * N + i);
                m = __ldg(reinterpret_cast<const uint4*>(top) + g);
                if (i == 0 && t == 0) {
                    auto inv = [](unsigned b) { return __int_as_float((scale_exp(b) - 14 + 127) << 23); };
                    reinterpret_cast<float4*>(scale)[g] = make_float4(inv(m.x), inv(m.y), inv(m.z), inv(m.w));
                }
            }
            const float f[4] = {v.x, v.y, v.z, v.w};
            const unsigned b[4] = {m.x, m.y, m.z, m.w};
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const float s = f[j] * __int_as_float((14 - scale_exp(b[j]) + 127) << 23);
                if (s != 0.f && fabsf(s) < 0x1p-6f) few |= 1ull << (8 * c + 4 * e + j);
                hi[4 * e + j] = __float2half_rn(s);
                lo[4 * e + j] = __float2half_rn(s - __half2float(hi[4 * e + j]));
            }
        }
        if (i < N) {
            out[(size_t)(k * (NS / 8) + c) * N] = *reinterpret_cast<const uint4*>(hi);
            out[(size_t)((gridDim.y + k) * (NS / 8) + c) * N] = *reinterpret_cast<const uint4*>(lo);
        }
    }
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        const unsigned mine = (unsigned)(few >> 32 * h);
        for (unsigned any = __reduce_or_sync(0xffffffffu, mine); any; any &= any - 1) {
            const int b = __ffs(any) - 1;
            const unsigned n = __popc(__ballot_sync(0xffffffffu, mine >> b & 1));
            if ((threadIdx.x & 31) == 0) atomicAdd(brief + 4 * g0 + k * NS + 32 * h + b, n);
        }
    }
}

// Zeros in the tiles outside the mask.
__global__ void __launch_bounds__(PIX) k_bp_zero(const int* __restrict__ list, float4* __restrict__ img, int N, int nt,
                                                 int G)
{
    const int tile = list[blockIdx.x];
    const int x = (tile % nt) * TP + (threadIdx.x & 15), y = (tile / nt) * TP + (threadIdx.x >> 4);
    if (x >= N || y >= N) return;
    for (int g = 0; g < G; ++g) img[((size_t)g * N + y) * N + x] = make_float4(0.f, 0.f, 0.f, 0.f);
}

// The slices that held a value that is not finite by plain gathers (as k_backproject_exact): a slice is a column of the
// product, which spreads such a value over its tiles and no further; and, in bins that no filter of this library
// made, the slices of which more than half of the values are below 2^-20 of the largest.  (Where a filter did, the row of
// the largest value holds that value's rounding, some 2^-28 of it in every bin, which is more in every pixel than the
// 2^-40 lost here; and the filter's tails of a small object alone go below 2^-20.)  (One such slice of 256 at
// 2049^2 x 1200: 8 ms, after 81).  NaN in all of the image if a wait gave up.
__global__ void __launch_bounds__(256) k_bp_flagged(const float* __restrict__ q, const float* __restrict__ cmask,
                                                    const float4* __restrict__ xsc, float* __restrict__ img, int N,
                                                    int T, int G, float mid, const unsigned* __restrict__ top,
                                                    const unsigned* __restrict__ brief, bool filtered,
                                                    const int* __restrict__ err)
{
    const bool lost = *err != 0;
    const size_t half = (size_t)T * N / 2;
    auto wanted = [&](int s) { return lost || top[s] >= 0x7f800000u || (!filtered && brief[s] > half); };
    bool any = false;
    for (int i = threadIdx.x; i < 4 * G; i += 256) any |= wanted(i);
    if (!__syncthreads_or(any)) return;
    const size_t NN = (size_t)N * N;
    for (size_t g = 0; g < G; ++g) {
        bool marked[4];
#pragma unroll
        for (int v = 0; v < 4; ++v) marked[v] = wanted((int)g * 4 + v);
        if (!(marked[0] || marked[1] || marked[2] || marked[3])) continue;
        for (size_t pix = blockIdx.x * (size_t)blockDim.x + threadIdx.x; pix < NN; pix += (size_t)gridDim.x * blockDim.x) {
            const float dx = (float)(pix % N + 1) - mid, dy = (float)(pix / N + 1) - mid;
            const float cm = cmask[pix];
            Lanes<float, 4> acc{};
            if (cm != 0.f && !lost) {
                for (int t = 0; t < T; ++t) {
                    const float4 x = __ldg(xsc + t);
                    float cell, wh;
                    exact_coord(x.x, x.y, x.z, x.w, dx, dy, mid, cell, wh);
                    const int y1 = (int)cell;
                    if (y1 > 1 && y1 < N) {
                        const float* row = q + ((g * T + t) * N + (y1 - 1)) * 4;
                        const Lanes<float, 4> a = ld_lanes<float, 4>(row), b = ld_lanes<float, 4>(row + 4);
#pragma unroll
                        for (int v = 0; v < 4; ++v) acc.v[v] = fmaf(b.v[v], wh, fmaf(a.v[v], 1.f - wh, acc.v[v]));
                    }
                }
            }
#pragma unroll
            for (int v = 0; v < 4; ++v)
                if (marked[v]) img[(g * NN + pix) * 4 + v] = lost ? __int_as_float(0x7fc00000) : acc.v[v] * cm;
        }
    }
}

// Tensor map of one pass: [T][chunks][N] pieces of 8 half-precision values.
bool bins_map(CUtensorMap* map, void* bins, int N, int T, int chunks)
{
    using Encode = CUresult (*)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
    static const Encode encode = [] {
        void* p = nullptr;
        cudaDriverEntryPointQueryResult st;
        if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &p, 12000, cudaEnableDefault, &st) != cudaSuccess)
            p = nullptr;
        return reinterpret_cast<Encode>(p);
    }();
    if (!encode) return false;
    const cuuint64_t dims[3] = {(cuuint64_t)N * 8, (cuuint64_t)chunks, (cuuint64_t)T};
    const cuuint64_t strides[2] = {(cuuint64_t)N * 16, (cuuint64_t)N * 16 * chunks};
    const cuuint32_t box[3] = {WIN * 8, (cuuint32_t)chunks, 1}, one[3] = {1, 1, 1};
    return encode(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 3, bins, dims, strides, box, one, CU_TENSOR_MAP_INTERLEAVE_NONE,
                  CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                  CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

template <int BLK>
bool bp_pass(const DevGeom<float>& g, int G, int g0, const float* q, void* bins, unsigned* top, float* scale,
             unsigned* brief, float* img, int* err, int sms, cudaStream_t st)
{
    CUtensorMap map;
    if (!bins_map(&map, bins, g.N, g.T, Bp<BLK>::CHUNKS)) return false;
    const int nt = (g.N + TP - 1) / TP;
    k_bp_bins<<<dim3((g.N + 127) / 128 * g.T, BLK), 128, 0, st>>>(reinterpret_cast<const float4*>(q), top, scale, brief,
                                                                reinterpret_cast<uint4*>(bins), g.N, g.T, G, g0);
    max_dynamic_smem<k_bp_mma<BLK>>();
    k_bp_mma<BLK><<<std::min(sms, g.n_tiles_in), 32 * Bp<BLK>::WARPS, Bp<BLK>::BARS + sizeof(Shared), st>>>(
        map, g.xsc_bp, g.tiles_in, g.n_tiles_in, g.cmask, scale, img, g.N, g.T, nt, G, g0, g.mid, err);
    return true;
}

}  // namespace

// Tiles (16 x 16 pixels, row by row) that meet the mask first, then the others; returns how many meet it.
int bp_tiles(const float* cmask, int N, std::vector<int>& list)
{
    const int nt = (N + TP - 1) / TP;
    std::vector<int> out;
    list.clear();
    for (int tile = 0; tile < nt * nt; ++tile) {
        bool in = false;
        for (int y = tile / nt * TP; y < std::min(N, (tile / nt + 1) * TP) && !in; ++y)
            for (int x = tile % nt * TP; x < std::min(N, (tile % nt + 1) * TP); ++x) in |= cmask[(size_t)y * N + x] != 0.f;
        (in ? list : out).push_back(tile);
    }
    const int n = (int)list.size();
    list.insert(list.end(), out.begin(), out.end());
    return n;
}

size_t bp_mma_bins_bytes(int N, int T, int G)
{
    return (size_t)T * N * NS * 4 * (G > NS / 4 ? 2 : 1);
}
size_t bp_mma_scalars(int G) { return (size_t)8 * G + (G * 4 + NS - 1) / NS * NS + 1; }

bool launch_backproject_mma(const DevGeom<float>& g, int G, const float* q, bool filtered, void* bins, unsigned* scalars,
                            float* img, cudaStream_t st)
{
    const size_t npos = (size_t)g.T * g.N;
    int sms = 0, dev = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    unsigned* top = scalars;
    float* scale = reinterpret_cast<float*>(scalars + 4 * (size_t)G);
    unsigned* brief = scalars + 8 * (size_t)G;                     // of whole blocks of 64 slices
    int* err = reinterpret_cast<int*>(scalars + bp_mma_scalars(G) - 1);   // a wait gave up
    cudaMemsetAsync(scalars, 0, bp_mma_scalars(G) * sizeof(unsigned), st);
    k_bp_max<<<dim3((unsigned)std::min<size_t>((npos + 1023) / 1024, 512), G), 256, 0, st>>>(
        reinterpret_cast<const float4*>(q), top, npos);
    if (g.n_tiles_in > 0)
        for (int g0 = 0; g0 < G;) {
            const bool two = G - g0 > NS / 4;
            if (!(two ? bp_pass<2>(g, G, g0, q, bins, top, scale, brief, img, err, sms, st)
                      : bp_pass<1>(g, G, g0, q, bins, top, scale, brief, img, err, sms, st)))
                return false;
            g0 += (two ? 2 : 1) * (NS / 4);
        }
    const int nt = (g.N + TP - 1) / TP, rest = nt * nt - g.n_tiles_in;
    if (rest > 0)
        k_bp_zero<<<rest, PIX, 0, st>>>(g.tiles_in + g.n_tiles_in, reinterpret_cast<float4*>(img), g.N, nt, G);
    k_bp_flagged<<<sms * 8, 256, 0, st>>>(q, g.cmask, g.xsc_bp, img, g.N, g.T, G, g.mid, top, brief, filtered, err);
    return true;
}

}  // namespace acu

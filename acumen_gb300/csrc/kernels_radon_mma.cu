// Projector on the tensor cores for large batches (tomography/tv_hpc.F90:129-159,
// exact sample positions).
//
// For one tile of 16 x 16 pixels and one angle the projection is a small matrix
// product: partial ray sums [rays x slices] = W [rays x 256 pixels] times the
// tile [256 pixels x slices], W(ray, pixel) being the sum of the bilinear
// weights with which the ray's samples read the pixel.  At most 25 rays meet a
// tile, so five angles make one M = 128 operand (25 rows each); about one
// weight in six of a row is not zero.  The gather kernels are held by the
// L1 data path (a tap feeds one multiply-add per slice); here a weight is
// formed once per 64 slices and the multiply-adds cost no loads.
//
// Both operands are split in two halves, v = hi + lo with 11 bits each, after
// a power-of-two scale (per tile and slice for the image, fixed for W).
// hi hi + hi lo + lo hi is accumulated; the term left out is 2^-24 of a
// product.  The tensor core truncates when it adds, so a chain in tensor memory
// is short: hi hi and the small terms have their own columns, and each half
// tile its own accumulator (8 steps of K = 16); the rest of every sum is added
// in FP32 with rounding to nearest.
//
// Measured at 2049^2 x 1200 angles: 256 slices 213.9 ms against 737.5 ms with
// the pixel-line gathers (64 slices: 72 against 185), 37 slices of 1025^2 x 601
// 9.5 against 16.3 ms.  Of the 213.9 ms the products take ~138 (the tensor cores
// busy about two thirds of it; a product of N = 64 columns takes 48 clocks,
// of 128 columns 64), the reduction ~75 at 80 % of the HBM bandwidth: 1.76 KB of
// partial sums a tile, angle and 20 rays of 64 slices are written and read once.
//
//   k_mma_tiles     lane image -> tiles in operand layout, with scales
//   k_mma_project   tiles -> partial sums P[block][half][tile][row][32 slices]
//   k_mma_reduce    P -> sinogram: a ray's partial sums in tile order (fixed, so
//                   results do not depend on the schedule)
//   k_radon_flagged the sinogram by plain gathers if the image held a value
//                   that is not finite (a matrix product would spread it)
#include <algorithm>
#include <cmath>
#include <vector>

#include "common.cuh"
#include "kernels.h"
#include "ray_weights.cuh"
#include "umma.cuh"

namespace acu {

namespace {

constexpr int TP = 16;                  // tile side
constexpr int NS = 64;                  // slices per block
constexpr int SLOTS = 5;                // angles per M = 128 operand, 26 rows apart (the last has 24)
constexpr int PITCH = 26;
constexpr int WIN = 25;                 // most rows (rays) of an angle
constexpr int TILE_OP = TP * TP * NS * 4;        // operand bytes of one tile: hi and lo halves
constexpr int SCALE_BYTES = NS * 4;              // the slices' scales of a tile
constexpr int TILE_BYTES = TILE_OP + SCALE_BYTES;
constexpr int PARTS = 4, PART_ROWS = TP / PARTS;        // a tile is walked four pixel rows at a time
constexpr int PART_OP = TILE_OP / PARTS;                // their operand bytes
constexpr int STAGE_HALF = PART_ROWS * TP * 128 * 2;    // a stage of W: four pixel rows x 128 rays; hi then lo
constexpr int STAGE_BYTES = 2 * STAGE_HALF;
constexpr int STAGES = 2, CREW = 2 * SLOTS;             // a stage is filled by ten warps, one pixel-angle per lane
constexpr int HALF = NS / 2;                            // partial sums are stored 32 slices at a time
// Warps by role.  With two blocks per tile W is needed at half the rate and the
// accumulators hold twice as much: one crew forms W, two sets of warps store.
template <int BLK>
struct Roles {
    static constexpr int CREWS = BLK == 2 ? 1 : 2, OUTS = BLK;
    static constexpr int MMA = CREWS * CREW, LOAD = MMA + 1, OUT = MMA + 2 + (4 - (MMA + 2) % 4) % 4,
                         WARPS = OUT + 4 * OUTS;
};
template <int BLK>
struct Smem {   // BLK tiles (64-slice blocks), stages of W, staged output rows, scales, barriers
    static constexpr int IMG = 0, W = BLK * TILE_OP, OUT = W + STAGES * STAGE_BYTES, SCALE = OUT + 128 * NS * 4,
                         BARS = SCALE + 2 * BLK * SCALE_BYTES;
};

// Lowest ray coordinate a tile's pixels reach (pixels x0..x0+15, y0..y0+15,
// 1-based), less the reach of their taps: the first ray of the tile's window
// is its ceiling.  Evaluated by the same instructions wherever a window is used.
__device__ __forceinline__ float window_lo(const MmaAngle& a, float mid, int x0, int y0)
{
    const float ex = (float)(a.s >= 0.f ? x0 + TP - 1 : x0) - mid;
    const float ey = (float)(a.c >= 0.f ? y0 : y0 + TP - 1) - mid;
    return __fsub_rn(__fmaf_rn(-a.s, ex, __fmaf_rn(a.c, ey, mid)), a.reach);
}

__device__ __forceinline__ uint32_t pack(float a, float b)   // a in the low half
{
    const __half2 h = __floats2half2_rn(a, b);
    return *reinterpret_cast<const uint32_t*>(&h);
}

struct Shared {
    uint64_t w_full[STAGES], w_empty[STAGES], d_full[4], d_empty[4], img_full[PARTS], img_empty[PARTS], sc_full[2], sc_empty[2],
        drained;
    uint32_t tmem;
};
static_assert(Smem<1>::BARS + sizeof(Shared) <= 227 * 1024 && Smem<2>::BARS + sizeof(Shared) <= 227 * 1024, "smem");

// Persistent: a block walks tiles blockIdx.x, + gridDim.x, ...  Roles by warp:
//   the first 20 or 10  form W, one pixel-angle per lane: ten warps (five angles) for each of two parts of the tile
//   MMA                 issues the products
//   LOAD                loads the tiles (one lane): a part of the next tile as soon as the last group is done with it
//   the last 4 or 8     add up the accumulators and store the partial sums
// W's rows are contiguous (M-major), so that a pixel's three rays are two
// aligned 32-bit words; a lane clears the two words it wrote last, never the
// whole stage.  Waits are bounded; one that gives up sets *err, and
// k_mma_reduce then writes NaN.
template <int BLK>
__global__ void __launch_bounds__(32 * Roles<BLK>::WARPS, 1) k_mma_project(const unsigned char* __restrict__ tiles,
                                                               float* __restrict__ P,
                                                               const MmaAngle* __restrict__ ang,
                                                               const int* __restrict__ groups, int N, int nt, int items,
                                                               int ngroups, int row0, int rows, float mid, int* err)
{
    extern __shared__ __align__(128) unsigned char sm[];
    using L = Smem<BLK>;
    using R = Roles<BLK>;
    Shared& sh = *reinterpret_cast<Shared*>(sm + L::BARS);
    constexpr int ACC_COLS = 2 * NS * BLK, ACCS = 512 / ACC_COLS;   // a ring of accumulators
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (threadIdx.x == 0) {
        for (int i = 0; i < STAGES; ++i) {
            umma::bar_init(&sh.w_full[i], CREW);
            umma::bar_init(&sh.w_empty[i], 1);
        }
        for (int i = 0; i < PARTS; ++i) {
            umma::bar_init(&sh.img_full[i], 1);
            umma::bar_init(&sh.img_empty[i], 1);
        }
        for (int i = 0; i < 2; ++i) {
            umma::bar_init(&sh.sc_full[i], 1);
            umma::bar_init(&sh.sc_empty[i], 4 * R::OUTS);
        }
        for (int i = 0; i < ACCS; ++i) {
            umma::bar_init(&sh.d_full[i], 1);
            umma::bar_init(&sh.d_empty[i], 4 * R::OUTS);
        }
        umma::bar_init(&sh.drained, 1);
        umma::bar_init_fence();
    }
    if (warp == R::MMA) umma::tmem_alloc<512>(&sh.tmem);
    for (int i = threadIdx.x; i < STAGES * STAGE_BYTES / 16; i += blockDim.x)
        reinterpret_cast<uint4*>(sm + L::W)[i] = make_uint4(0, 0, 0, 0);
    umma::fence_async_smem();
    umma::fence_before();
    __syncthreads();
    umma::fence_after();
    const uint32_t tmem = sh.tmem;
    bool ok = true;

    if (warp < R::MMA) {
        const int crew = warp / CREW, slot = warp % CREW >> 1, half = warp & 1;
        const int trow = lane >> 3, tx = half * 8 + (lane & 7);
        const int words = slot == SLOTS - 1 ? (128 - (SLOTS - 1) * PITCH) / 2 : PITCH / 2;
        // this lane's K column of the stage: chunk 2 trow + half, element lane % 8; row pair i of the angle sits
        // at ((slot * 13 + i) / 4) * 128 + ((slot * 13 + i) % 4) * 4
        const uint32_t base = L::W + (2 * trow + half) * 2048 + (lane & 7) * 16;
        auto place = [&](int i, int st) -> uint32_t {   // 0: outside the window
            const int w = slot * (PITCH / 2) + i;
            return (unsigned)i < (unsigned)words ? base + st * STAGE_BYTES + w * 4 + (w >> 2) * 112 : 0u;
        };
        auto put = [&](uint32_t at, uint32_t hi, uint32_t lo) {
            if (at) {
                *reinterpret_cast<uint32_t*>(sm + at) = hi;
                *reinterpret_cast<uint32_t*>(sm + at + STAGE_HALF) = lo;
            }
        };
        uint32_t last0[STAGES] = {0, 0}, last1[STAGES] = {0, 0};   // the two words written last time, per stage
        unsigned n = 0;                                            // groups
        for (int it = blockIdx.x; it < items && ok; it += gridDim.x) {
            const int tile = it % (nt * nt);
            const int x0 = (tile % nt) * TP + 1, y0 = (tile / nt) * TP + 1;
            const int px = x0 + tx;
            const float ex = (float)px - mid;
            const bool rim = x0 < 3 || y0 < 3 || x0 + TP > N || y0 + TP > N;
            for (int g = 0; g < ngroups && ok; ++g, ++n) {
                const int t = groups[g] + slot;
                const bool live = t < groups[g + 1];
                MmaAngle a;
                int j0 = 0;
                bool ends = false;
                if (live) {
                    a = ang[t];
                    j0 = (int)ceilf(window_lo(a, mid, x0, y0));
                    const float uc = fmaf(a.c, (float)x0 + 7.5f - mid, fmaf(a.s, (float)y0 + 7.5f - mid, mid));
                    const float ur = 7.5f * a.reach + 4.f;
                    ends = uc - ur < 1.f || uc + ur > (float)N;   // some rays may end in the tile
                }
#pragma unroll 1
                for (int q0 = 0; q0 < PARTS && ok; q0 += STAGES)
#pragma unroll
                for (int own = 0; own < STAGES / R::CREWS; ++own) {
                    const int st = R::CREWS == 1 ? own : crew, q = q0 + st;
                    const unsigned fills = (n * PARTS + q) / STAGES;   // of this stage, before
                    const int py = y0 + PART_ROWS * q + trow;
                    uint32_t h0 = 0, h1 = 0, l0 = 0, l1 = 0;
                    int pair = -100;
                    if (live) {
                        const float ey = (float)py - mid;
                        float wv[3];
                        int j;
                        if (rim) {
                            ray_weights<RIM>(a, ex, ey, 0.f, mid, px, py, N, j, wv);
                        } else if (ends) {
                            ray_weights<ENDS>(a, ex, ey, 0.f, mid, px, py, N, j, wv);
                        } else {
                            ray_weights<INNER>(a, ex, ey, 0.f, mid, px, py, N, j, wv);
                        }
                        // the leading 11 bits are exact in half precision, the rest is rounded
                        float hi[3];
#pragma unroll
                        for (int r = 0; r < 3; ++r) hi[r] = __uint_as_float(__float_as_uint(wv[r]) & 0xffffe000u);
                        const int row = j - j0;
                        pair = row >> 1;
                        // three rows as two row pairs: moved up by one row if the first row is odd
                        const int sft = (row & 1) << 4;
                        const uint32_t ha = pack(hi[0], hi[1]), hb = pack(hi[2], 0.f);
                        const uint32_t la = pack(wv[0] - hi[0], wv[1] - hi[1]), lb = pack(wv[2] - hi[2], 0.f);
                        h0 = ha << sft;
                        h1 = __funnelshift_l(ha, hb, sft);
                        l0 = la << sft;
                        l1 = __funnelshift_l(la, lb, sft);
                    }
                    ok = umma::bar_wait_warp(&sh.w_empty[st], (fills & 1) ^ 1);
                    if (!ok) break;
                    put(last0[own], 0, 0);
                    put(last1[own], 0, 0);
                    last0[own] = place(pair, st);
                    last1[own] = place(pair + 1, st);
                    put(last0[own], h0, l0);
                    put(last1[own], h1, l1);
                    umma::fence_async_smem();
                    __syncwarp();
                    if (lane == 0) umma::bar_arrive(&sh.w_full[st]);
                }
            }
        }
    } else if (warp == R::MMA) {
        constexpr uint32_t A_M_MAJOR = 1u << 15;
        constexpr uint32_t ID_HI = umma::instr_desc_f16(128, 2 * NS) | A_M_MAJOR,
                           ID_LO = umma::instr_desc_f16(128, NS) | A_M_MAJOR;
        const uint32_t acc0 = __reduce_max_sync(0xffffffffu, tmem);   // the same in all lanes, and known to be
        const uint64_t w0 = umma::smem_desc(umma::smem_addr(sm + L::W), 2048),
                       img = umma::smem_desc(umma::smem_addr(sm + L::IMG), 2048);
        unsigned n = 0, m = 0, b = 0;   // parts, groups, tiles
        bool ready = false, room = false;   // seen before it was needed: the next stage is full, the accumulator free
        for (int it = blockIdx.x; it < items && ok; it += gridDim.x, ++b) {
            for (int g = 0; g < ngroups && ok; ++g, ++m) {
                if (!__all_sync(0xffffffffu, room)) ok = umma::bar_wait_warp(&sh.d_empty[m % ACCS], ((m / ACCS) & 1) ^ 1);
                if (!ok) break;
                const uint32_t d = acc0 + (m % ACCS) * ACC_COLS;
#pragma unroll 1
                for (int q = 0; q < PARTS; ++q, ++n) {
                    const int st = n % STAGES;
                    if (g == 0) ok = umma::bar_wait_warp(&sh.img_full[q], b & 1);
                    if (!__all_sync(0xffffffffu, ready)) ok = umma::bar_wait_warp(&sh.w_full[st], (n / STAGES) & 1) && ok;
                    if (!ok) break;
                    umma::fence_after();
                    ready = umma::bar_test(&sh.w_full[(n + 1) % STAGES], ((n + 1) / STAGES) & 1);
                    if (q == PARTS - 1) room = umma::bar_test(&sh.d_empty[(m + 1) % ACCS], (((m + 1) / ACCS) & 1) ^ 1);
                    const uint64_t w = w0 + (uint32_t)(st * (STAGE_BYTES >> 4));
                    const uint64_t bd = img + (uint32_t)(q * (PART_OP >> 4));
#pragma unroll
                    for (int ks = 0; ks < PART_ROWS; ++ks) {
#pragma unroll
                        for (int k = 0; k < BLK; ++k) {
                            // hi x [hi | lo], then lo x hi on top of hi x lo
                            umma::mma_f16(d + k * 2 * NS, w + (ks * 4096 >> 4), bd + ((k * TILE_OP + ks * 4096) >> 4),
                                          ID_HI, q > 0 || ks > 0);
                            umma::mma_f16(d + k * 2 * NS + NS, w + ((STAGE_HALF + ks * 4096) >> 4),
                                          bd + ((k * TILE_OP + ks * 4096) >> 4), ID_LO, true);
                        }
                    }
                    umma::mma_commit(umma::smem_addr(&sh.w_empty[st]));
                    if (g == ngroups - 1) umma::mma_commit(umma::smem_addr(&sh.img_empty[q]));
                }
                if (ok) umma::mma_commit(umma::smem_addr(&sh.d_full[m % ACCS]));
            }
        }
        // every MMA is done before the tensor memory is given back
        umma::mma_commit(umma::smem_addr(&sh.drained));
        ok = umma::bar_wait(&sh.drained, 0) && ok;
    } else if (warp == R::LOAD) {
        if (lane == 0) {
            unsigned b = 0, nsc = 0, parts = 0;   // tiles, scale loads, parts of the tile being loaded
            for (int it = blockIdx.x; it < items && ok; it += gridDim.x, ++b) {
                // the tiles of a block lie together
                const unsigned char* src =
                    tiles + ((size_t)(it / (nt * nt)) * BLK * (nt * nt) + it % (nt * nt)) * TILE_BYTES;
                const size_t next = (size_t)nt * nt * TILE_BYTES;   // the tile's next block
                ok = umma::bar_wait(&sh.sc_empty[b & 1], ((b >> 1) & 1) ^ 1);
                if (!ok) break;
                umma::bar_expect(&sh.sc_full[b & 1], BLK * SCALE_BYTES);
                for (int k = 0; k < BLK; ++k)
                    umma::bulk_load(sm + L::SCALE + ((b & 1) * BLK + k) * SCALE_BYTES, src + k * next + TILE_OP,
                                    SCALE_BYTES, &sh.sc_full[b & 1]);
                ++nsc;
                for (parts = 0; parts < PARTS; ++parts) {
                    const int q = parts;
                    ok = umma::bar_wait(&sh.img_empty[q], (b & 1) ^ 1);
                    if (!ok) break;
                    umma::bar_expect(&sh.img_full[q], BLK * PART_OP);
                    for (int k = 0; k < BLK; ++k)
                        umma::bulk_load(sm + L::IMG + k * TILE_OP + q * PART_OP, src + k * next + q * PART_OP, PART_OP,
                                        &sh.img_full[q]);
                }
                if (!ok) break;
                parts = 0;
            }
            // loads in flight land before the block leaves
            for (unsigned q = 0; q < PARTS; ++q)
                if (b + (q < parts) > 0) umma::bar_wait(&sh.img_full[q], (b + (q < parts) - 1) & 1);
            for (unsigned i = 0; i < 2; ++i)
                if (nsc > i) umma::bar_wait(&sh.sc_full[i], ((nsc - i + 1) / 2 - 1) & 1);
        }
        __syncwarp();
    } else if (warp >= R::OUT) {
        const int row = (warp & 3) * 32 + lane;   // a warp reads the 32 tensor-memory lanes of its number modulo 4
        const int slot = row / PITCH, r = row % PITCH;
        const int k = (warp - R::OUT) >> 2;       // block
        // 4 KB of staged rows at a time; with one set of warps there is room for two
        unsigned char* const stage0 = sm + L::OUT + (warp - R::OUT) * (128 * NS * 4 / (4 * R::OUTS));
        constexpr int STAGE_STEP = R::OUTS == 1 ? 32 * HALF * 4 : 0;
        const size_t plane = (size_t)nt * nt * rows * HALF;
        unsigned m = 0, b = 0;
        for (int it = blockIdx.x; it < items && ok; it += gridDim.x, ++b) {
            ok = umma::bar_wait_warp(&sh.sc_full[b & 1], (b >> 1) & 1);
            const float4* const scale = reinterpret_cast<const float4*>(sm + L::SCALE + ((b & 1) * BLK + k) * SCALE_BYTES);
            float* const out =
                P + ((size_t)(it / (nt * nt) * BLK + k) * 2 * nt * nt + it % (nt * nt)) * rows * HALF;
            for (int g = 0; g < ngroups; ++g, ++m) {
                const int tg = groups[g], te = groups[g + 1];
                int prow = -1;   // this row's place among all rows
                if (slot < te - tg && r < ang[tg + slot].nr) prow = ang[tg + slot].roff + r;
                // the warp's rows lie together
                const unsigned used = __ballot_sync(0xffffffffu, prow >= 0);
                const int n_rows = __popc(used), first = __shfl_sync(0xffffffffu, prow, used ? __ffs(used) - 1 : 0);
                ok = ok && umma::bar_wait_warp(&sh.d_full[m % ACCS], (m / ACCS) & 1);
                if (!ok) break;
                umma::fence_after();
                const uint32_t d = tmem + ((uint32_t)((warp & 3) * 32) << 16) + (m % ACCS) * ACC_COLS + k * 2 * NS;
                // eight columns at a time, the next ones on their way while these are added up
                float2 v[2][4], x[2][4];
                umma::tmem_ld8(d, v[0]);
                umma::tmem_ld8(d + NS, x[0]);
#pragma unroll
                for (int c = 0; c < NS / 8; ++c) {
                    const int h = c / (HALF / 8);   // 32-slice half
                    umma::tmem_ld_wait(v[c & 1], x[c & 1]);
                    if (c + 1 < NS / 8) {
                        umma::tmem_ld8(d + 8 * (c + 1), v[(c + 1) & 1]);
                        umma::tmem_ld8(d + NS + 8 * (c + 1), x[(c + 1) & 1]);
                    } else {
                        umma::fence_before();
                        __syncwarp();
                        if (lane == 0) umma::bar_arrive(&sh.d_empty[m % ACCS]);
                    }
                    if (c % (HALF / 8) == 0) {   // the staged rows of this half are on their way out no longer
                        if (lane == 0) umma::bulk_store_wait_read<R::OUTS == 1 ? 1 : 0>();
                        __syncwarp();
                    }
                    if (prow >= 0) {
                        // a row's 16-byte pieces are permuted by its number: no bank conflicts
                        unsigned char* const to = stage0 + h * STAGE_STEP + (prow - first) * (HALF * 4);
#pragma unroll
                        for (int i = 0; i < 2; ++i) {
                            const float4 s = scale[2 * c + i];
                            const float2 e = mul2(add2(v[c & 1][2 * i], x[c & 1][2 * i]), make_float2(s.x, s.y));
                            const float2 f = mul2(add2(v[c & 1][2 * i + 1], x[c & 1][2 * i + 1]), make_float2(s.z, s.w));
                            *reinterpret_cast<float4*>(to + (((2 * c % (HALF / 4) + i) ^ (prow & 7)) << 4)) =
                                make_float4(e.x, e.y, f.x, f.y);
                        }
                    }
                    if ((c + 1) % (HALF / 8) == 0) {
                        umma::fence_async_smem();
                        __syncwarp();
                        if (lane == 0) {
                            if (n_rows > 0)
                                umma::bulk_store(out + h * plane + (size_t)(first - row0) * HALF, stage0 + h * STAGE_STEP,
                                                 n_rows * HALF * 4);
                            else
                                umma::bulk_store_none();
                        }
                    }
                }
            }
            __syncwarp();
            if (ok && lane == 0) umma::bar_arrive(&sh.sc_empty[b & 1]);
        }
        if (lane == 0) umma::bulk_store_wait();
    }
    if (!ok) atomicExch(err, 1);
    umma::fence_before();
    __syncthreads();
    if (warp == R::MMA) umma::tmem_free<512>(tmem);
}

// One ray and 16 slices per thread (four pieces of 16 bytes): the partial sums
// of the tiles whose window holds the ray, along its major axis; along the
// other axis at most three tiles can hold it.  Four threads read the 128
// contiguous bytes of a row and 32 slices.
__global__ void __launch_bounds__(256) k_mma_reduce(const float* __restrict__ P, float* __restrict__ sino,
                                                    const MmaAngle* __restrict__ ang, int N, int T, int nt, int G,
                                                    int g0, int t0, int row0, int rows, float mid,
                                                    const int* __restrict__ err)
{
    const int c = threadIdx.x & 3, t = t0 + blockIdx.y;
    const int j = blockIdx.x * 64 + (threadIdx.x >> 2) + 1;
    if (j > N) return;
    const MmaAngle a = ang[t];
    const bool xm = fabsf(a.c) >= fabsf(a.s);
    const float step = TP * (xm ? a.c : -a.s), inv = 1.f / step;
    const size_t plane = (size_t)nt * nt * rows * (HALF / 4);   // 32 slices of every partial sum
    const float4* base = reinterpret_cast<const float4*>(P) + (size_t)blockIdx.z * 2 * plane;
    const int lrow = a.roff - row0;
    float4 acc[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) acc[k] = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 2
    for (int k = 0; k < nt; ++k) {
        const float v0 = xm ? window_lo(a, mid, k * TP + 1, 1) : window_lo(a, mid, 1, k * TP + 1);
        const float lim = step > 0.f ? (float)(j - a.nr) - v0 : (float)j - v0;
        const int b0 = (int)ceilf(fminf(fmaxf(__fmaf_rn(lim, inv, -1e-3f), -8.f), (float)nt + 8.f));
#pragma unroll
        for (int i = 0; i < 3; ++i) {
            const int b = b0 + i;
            const int bx = xm ? k : b, by = xm ? b : k;
            const int r = j - (int)ceilf(window_lo(a, mid, bx * TP + 1, by * TP + 1));
            if ((unsigned)b < (unsigned)nt && (unsigned)r < (unsigned)a.nr) {
                const float4* row = base + ((size_t)(by * nt + bx) * rows + lrow + r) * (HALF / 4);
                const int sw = (a.roff + r) & 7;
#pragma unroll
                for (int p = 0; p < 4; ++p) {
                    const float4 v = __ldcs(row + (p >> 1) * plane + ((4 * (p & 1) + c) ^ sw));
                    acc[p].x += v.x;
                    acc[p].y += v.y;
                    acc[p].z += v.z;
                    acc[p].w += v.w;
                }
            }
        }
    }
    const float fN = (float)N;
    const bool bad = *err != 0;
#pragma unroll
    for (int p = 0; p < 4; ++p) {
        const int g = g0 + blockIdx.z * 16 + 4 * p + c;
        if (g >= G) continue;
        float4 o = make_float4(acc[p].x / fN, acc[p].y / fN, acc[p].z / fN, acc[p].w / fN);
        if (bad) o.x = o.y = o.z = o.w = __int_as_float(0x7fc00000);
        reinterpret_cast<float4*>(sino)[((size_t)g * T + t) * N + (j - 1)] = o;
    }
}

// One block per tile and 64-slice block: the tile's values, scaled per slice so
// that the largest lies in [2^14, 2^15), as hi and lo halves in operand layout
// ([pixel / 8][hi: 64 slices, lo: 64 slices][pixel % 8]), then the factors that
// undo the scales of image and weights.
__global__ void __launch_bounds__(256) k_mma_tiles(const float4* __restrict__ img, unsigned char* __restrict__ tiles,
                                                   int N, int nt, int G, int g0, int* flag)
{
    extern __shared__ __align__(16) float s_v[];   // [64][260], then 64 scales
    constexpr int LD = TP * TP + 4;
    float* const s_scale = s_v + NS * LD;
    const int tile = blockIdx.x, tid = threadIdx.x;
    const int x = (tile % nt) * TP + (tid & 15), y = (tile / nt) * TP + (tid >> 4);
    const bool in = x < N && y < N;
    const size_t NN = (size_t)N * N;
#pragma unroll 4
    for (int k = 0; k < NS / 4; ++k) {
        const int g = g0 + blockIdx.y * 16 + k;
        const float4 v = in && g < G ? __ldg(img + (size_t)g * NN + (size_t)y * N + x) : make_float4(0.f, 0.f, 0.f, 0.f);
        s_v[(4 * k) * LD + tid] = v.x;
        s_v[(4 * k + 1) * LD + tid] = v.y;
        s_v[(4 * k + 2) * LD + tid] = v.z;
        s_v[(4 * k + 3) * LD + tid] = v.w;
    }
    __syncthreads();
    unsigned char* const out = tiles + ((size_t)blockIdx.y * gridDim.x + tile) * TILE_BYTES;
    const int warp = tid >> 5, lane = tid & 31;
    for (int n = warp; n < NS; n += 8) {
        unsigned m = 0;
#pragma unroll
        for (int k = 0; k < TP * TP; k += 32) m = max(m, __float_as_uint(s_v[n * LD + k + lane]) & 0x7fffffffu);
        m = __reduce_max_sync(0xffffffffu, m);
        if (lane == 0) {
            if (m >= 0x7f800000u) {
                atomicOr(flag, 1);
                m = 0;
            }
            const int e = m ? max((int)(m >> 23) - 127, -98) : 0;
            s_scale[n] = __int_as_float((14 - e + 127) << 23);
            reinterpret_cast<float*>(out + TILE_OP)[n] = __int_as_float((e - 14 + 127) << 23);
        }
    }
    __syncthreads();
    for (int u = tid; u < TILE_OP / 16; u += 256) {
        const int n = u & (NS - 1), lo = (u >> 6) & 1, kc = u >> 7;
        const float sc = s_scale[n];
        const float4 a = *reinterpret_cast<const float4*>(s_v + n * LD + kc * 8);
        const float4 b = *reinterpret_cast<const float4*>(s_v + n * LD + kc * 8 + 4);
        const float v[8] = {a.x * sc, a.y * sc, a.z * sc, a.w * sc, b.x * sc, b.y * sc, b.z * sc, b.w * sc};
        __align__(16) __half h[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            h[i] = __float2half_rn(v[i]);
            if (lo) h[i] = __float2half_rn(v[i] - __half2float(h[i]));
        }
        reinterpret_cast<uint4*>(out)[u] = *reinterpret_cast<const uint4*>(h);
    }
}

// The projection by plain gathers (as k_radon), done only if *flag is set.
__global__ void __launch_bounds__(128) k_radon_flagged(const float* __restrict__ img, const float* __restrict__ sc,
                                                       const float4* __restrict__ xsc, float* __restrict__ sino, int N,
                                                       int T, int G, float mid, const int* __restrict__ flag)
{
    if (*flag == 0) return;
    const int nb = (N + 127) / 128;
    const long long total = (long long)nb * T * G;
    for (long long it = blockIdx.x; it < total; it += gridDim.x) {
        const int jy = (int)(it % nb) * 128 + threadIdx.x + 1, t = (int)((it / nb) % T);
        const size_t g = (size_t)(it / nb / T);
        if (jy > N) continue;
        const ProjRay<float, true> ray(sc, xsc, t, jy, mid, nullptr);
        const float* u = img + g * N * N * 4;
        Lanes<float, 4> acc{};
        for (int jx = 1; jx <= N; ++jx) {
            int x1, y1;
            float wxl, wxh, wyl, wyh;
            ray.at((float)jx - mid, x1, y1, wxl, wxh, wyl, wyh);
            if (min(x1, y1) > 1 && max(x1, y1) < N) {
                const float w11 = wxl * wyl, w21 = wxh * wyl, w12 = wxl * wyh, w22 = wxh * wyh;
                const float* p = u + ((size_t)(y1 - 1) * N + (x1 - 1)) * 4;
                const Lanes<float, 4> a = ld_lanes<float, 4>(p), b = ld_lanes<float, 4>(p + 4);
                const Lanes<float, 4> cc = ld_lanes<float, 4>(p + (size_t)N * 4), d = ld_lanes<float, 4>(p + (size_t)N * 4 + 4);
#pragma unroll
                for (int v = 0; v < 4; ++v)
                    acc.v[v] = fmaf(d.v[v], w22, fmaf(cc.v[v], w12, fmaf(b.v[v], w21, fmaf(a.v[v], w11, acc.v[v]))));
            }
        }
#pragma unroll
        for (int v = 0; v < 4; ++v) acc.v[v] = acc.v[v] / (float)N;
        st_lanes<float, 4>(sino + ((g * T + t) * N + (jy - 1)) * 4, acc);
    }
}

}  // namespace

std::vector<MmaAngle> mma_angles(const float* xsc, int T)
{
    std::vector<MmaAngle> out((size_t)T);
    int roff = 0;
    for (int t = 0; t < T; ++t) {
        MmaAngle& a = out[t];
        a.x = make_float4(xsc[4 * t], xsc[4 * t + 1], xsc[4 * t + 2], xsc[4 * t + 3]);
        a.s = a.x.x + a.x.z;
        a.c = a.x.y + a.x.w;
        a.t = std::fabs(a.c) >= std::fabs(a.s) ? a.s / a.c : -a.c / a.s;
        const float sum = std::fabs(a.c) + std::fabs(a.s);
        a.reach = sum + 1e-3f;   // window_lo's own rounding is below 1e-3
        // integers an interval of 17 (|c| + |s|) + 0.002 (15 across the tile, one reach at each end) can hold
        a.nr = std::min(WIN, (int)std::floor((TP + 1) * sum + 0.002f) + 1);
        a.roff = roff;
        roff += a.nr;
    }
    return out;
}

// First angles of the groups that share an operand: five angles, or four when
// the fifth would need 25 rows.
std::vector<int> mma_groups(const std::vector<MmaAngle>& ang)
{
    std::vector<int> g;
    const int T = (int)ang.size();
    for (int t = 0; t < T;) {
        g.push_back(t);
        const int n = std::min(SLOTS, T - t);
        t += n == SLOTS && ang[t + SLOTS - 1].nr > 128 - (SLOTS - 1) * PITCH ? SLOTS - 1 : n;
    }
    g.push_back(T);
    return g;
}

static size_t part_rows(const DevGeom<float>& g, int ga, int gb)   // rows of the groups [ga, gb)
{
    const MmaAngle& last = g.h_mma[g.h_groups[gb] - 1];
    return last.roff + last.nr - g.h_mma[g.h_groups[ga]].roff;
}

// The cap on partial sums held at once sets the angles per chunk.  Larger
// chunks read the tiles less often (64 KB per tile and chunk against ~5.6 KB
// written per angle).
MmaPlan mma_plan(const DevGeom<float>& g, int G)
{
    MmaPlan p;
    p.nt = (g.N + TP - 1) / TP;
    p.nblk = (G * 4 + NS - 1) / NS;
    const size_t row = (size_t)p.nt * p.nt * NS * sizeof(float);
    const size_t all = row * part_rows(g, 0, g.n_groups);
    // blocks go in pairs, which share every W
    p.nb = std::min(p.nblk, 2);
    p.ng = g.n_groups;
    if (all * p.nb <= MMA_PART_CAP) {
        p.nb = (int)std::min<size_t>(p.nblk, MMA_PART_CAP / all);
        if (p.nb > 2) p.nb &= ~1;
    } else {
        p.ng = std::max(1, (int)(MMA_PART_CAP / (row * WIN * SLOTS * p.nb)));
    }
    size_t rows = 0;
    for (int a = 0; a < g.n_groups; a += p.ng) rows = std::max(rows, part_rows(g, a, std::min(a + p.ng, g.n_groups)));
    p.tile_bytes = (size_t)p.nt * p.nt * p.nb * TILE_BYTES;
    p.part_bytes = row * rows * p.nb;
    return p;
}

// Sides whose five-angle chunks of partial sums exceed the cap keep the gather kernels.
bool mma_fits(int N)
{
    const size_t nt = (size_t)(N + TP - 1) / TP;
    return nt * nt * NS * sizeof(float) * WIN * SLOTS <= MMA_PART_CAP;
}

void launch_radon_mma(const DevGeom<float>& g, int G, const float* img, unsigned char* tiles, float* P, int* flags,
                      const MmaPlan& p, float* sino, cudaStream_t st)
{
    const int N = g.N, T = g.T, nt2 = p.nt * p.nt;
    max_dynamic_smem<k_mma_tiles>();
    max_dynamic_smem<k_mma_project<1>>();
    max_dynamic_smem<k_mma_project<2>>();
    cudaMemsetAsync(flags, 0, 2 * sizeof(int), st);   // [0] not finite, [1] a wait gave up
    int sms = 0, dev = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    for (int b = 0; b < p.nblk; b += p.nb) {
        const int nb = std::min(p.nb, p.nblk - b);
        k_mma_tiles<<<dim3(nt2, nb), 256, NS * (TP * TP + 5) * sizeof(float), st>>>(
            reinterpret_cast<const float4*>(img), tiles, N, p.nt, G, b * (NS / 4), flags);
        for (int ga = 0; ga < g.n_groups; ga += p.ng) {
            const int gb = std::min(ga + p.ng, g.n_groups);
            const int t0 = g.h_groups[ga], t1 = g.h_groups[gb];
            const int row0 = g.h_mma[t0].roff, rows = (int)part_rows(g, ga, gb);
            const int blk = nb % 2 == 0 ? 2 : 1;   // 64-slice blocks per operand W
            const int items = nt2 * (nb / blk);
            (blk == 2 ? k_mma_project<2> : k_mma_project<1>)<<<std::min(sms, items),
                                                               32 * (blk == 2 ? Roles<2>::WARPS : Roles<1>::WARPS),
                                                               (blk == 2 ? Smem<2>::BARS : Smem<1>::BARS) + sizeof(Shared), st>>>(
                tiles, P, g.mma, g.groups + ga, N, p.nt, items, gb - ga, row0, rows, g.mid, flags + 1);
            k_mma_reduce<<<dim3((N + 63) / 64, t1 - t0, nb), 256, 0, st>>>(P, sino, g.mma, N, T, p.nt, G, b * (NS / 4),
                                                                          t0, row0, rows, g.mid, flags + 1);
        }
    }
    k_radon_flagged<<<sms * 8, 128, 0, st>>>(img, g.sc_fp, g.xsc_fp, sino, N, T, G, g.mid, flags);
}

}  // namespace acu

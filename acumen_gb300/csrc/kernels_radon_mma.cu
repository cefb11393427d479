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
// is short: one tile (16 steps of K = 16), hi hi and the small terms in columns of their
// own; the rest of every sum is added in FP32 with rounding to nearest.
//
// Blocks walk stretches of tiles along the rays.  A ray that leaves one tile
// enters the next, so the rows both tiles met are added to in the L2 cache, by bulk
// reductions in tile order; only the finished rows of a stretch, a third of
// what the tiles would write one by one, go to memory and are read back.
// The order is kept by the four warps that send a block's rows: a ray's place in the
// operand moves from tile to tile, so two tiles' rows of it may be in the hands of two warps, and
// a bulk operation is known to have arrived only to the thread that issued it.
// Once a tile every warp waits until all that it sent has arrived, and the four meet
// before the next tile's rows go out.
//
// Measured at 2049^2 x 1200 angles, 256 slices: 737 ms with the pixel-line
// gathers, 217 ms with every tile's rows written and read (75 of them the
// reduction at 80 % of the HBM bandwidth), now 168 ms, 20 of them the reduction (the
// meetings of the warps 1.5 ms, whether for all rows once a tile or at two groups for those two groups old).  1025^2 x
// 600, 128 slices 14.7 / 12.0 ms, 64 slices 9.8 / 9.6 ms (23.4 with gathers).
// What holds the products is shared memory: 14 KB of operands per K step of one
// block (20 KB of two, which share W) and the stores of W and of the staged rows
// come to its 128 bytes a clock.
//
//   k_mma_tiles     lane image -> tiles in operand layout, with scales
//   k_mma_project   tiles -> partial sums P[block][half][stretch][row][32 slices]
//   k_mma_reduce    P -> sinogram: a ray's partial sums in the order of the
//                   stretches (fixed, so results do not depend on the schedule)
//   k_radon_flagged by plain gathers the slices that held a value that is not
//                   finite, and those of subnormal magnitude
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
constexpr int ROW_W = TP * 128 * 2 + 64;                // W of a pixel row: 16 pixels x 128 rays, set off against bank conflicts
constexpr int STAGE_HALF = PART_ROWS * ROW_W;           // a stage of W: four pixel rows; hi then lo
constexpr int STAGE_BYTES = 2 * STAGE_HALF;
constexpr int STAGES = 2, CREW = 2 * SLOTS;             // a stage is filled by ten warps, one pixel-angle per lane
constexpr size_t MMA_L2_ROWS = (size_t)144 << 20;   // bytes of partial sums that the SMs add to at a time
constexpr int HALF = NS / 2;                            // partial sums are stored 32 slices at a time
// Warps by role.  Two crews take turns at the stages of W; four warps store a block.
template <int BLK>
struct Roles {
    static constexpr int OUTS = BLK;
    static constexpr int MMA = STAGES * CREW, LOAD = MMA + 1, OUT = MMA + 2, ROWS = OUT + 4 * OUTS, WARPS = ROWS + 1;
};
template <int BLK>
struct Smem {   // tiles of BLK blocks, stages of W, staged output rows, scales, barriers
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

__device__ __forceinline__ int first_ray(const MmaAngle& a, float mid, int bx, int by)
{
    return (int)ceilf(window_lo(a, mid, bx * TP + 1, by * TP + 1));
}

// The tiles of a grid as lines of them along the rays (rows of tiles for angles
// along x, else columns), every line cut into stretches.
struct Stretch {
    int block, line, k0, k1;   // unit of BLK blocks; tiles k0..k1-1 of the line
    __device__ __forceinline__ Stretch(int unit, int nt, int stretches)
    {
        block = unit / (nt * stretches);
        const int u = unit % (nt * stretches), q = u % stretches;
        line = u / stretches;
        k0 = q * nt / stretches;
        k1 = (q + 1) * nt / stretches;
    }
};

__device__ __forceinline__ uint32_t pack(float a, float b)   // a in the low half
{
    const __half2 h = __floats2half2_rn(a, b);
    return *reinterpret_cast<const uint32_t*>(&h);
}

// What becomes of an angle's rows in a tile: the first one's place among the
// stretch's partial sums, their number, and which of them (from, to) the tile
// before met too.
struct Rows {
    int place;
    unsigned char nr, from, to, pad;
};

struct Shared {
    uint64_t w_full[STAGES], w_empty[STAGES], d_full[4], d_empty[4], img_full[PARTS], img_empty[PARTS], sc_full[2], sc_empty[2],
        rows_full[4], sent[2], drained;
    Rows rows[4][SLOTS];   // per accumulator
    uint32_t tmem;
};
static_assert(Smem<1>::BARS + sizeof(Shared) <= 227 * 1024 && Smem<2>::BARS + sizeof(Shared) <= 227 * 1024, "smem");

// Persistent: a block walks the tiles of stretches blockIdx.x, + gridDim.x, ...  Roles by warp:
//   the first 20        form W, one pixel-angle per lane: ten warps (five angles) for each of two parts of the tile
//   MMA                 issues the products
//   LOAD                loads the tiles (one lane): a part of the next tile as soon as the last group is done with it
//   ROWS                finds where the rows of a tile go
//   the others          add up the accumulators and add them to the stretch's partial sums: rows that the
//                       tile before met too by a bulk reduction in L2, the others by a bulk store
// W's rows are contiguous (M-major), so that a pixel's three rays are two
// aligned 32-bit words; a lane clears the two words it wrote last, never the
// whole stage.  Waits are bounded; one that gives up sets *err, and
// k_mma_reduce then writes NaN.
template <int BLK>
__global__ void __launch_bounds__(32 * Roles<BLK>::WARPS, 1) k_mma_project(const unsigned char* __restrict__ tiles,
                                                               float* __restrict__ P,
                                                               const MmaAngle* __restrict__ ang,
                                                               const int* __restrict__ groups, int N, int nt, int stretches,
                                                               bool xm, int units, int ngroups, int row0, int rows,
                                                               float mid, int* err)
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
            umma::bar_init(&sh.rows_full[i], 1);
            umma::bar_init(&sh.d_empty[i], 4 * R::OUTS);
        }
        for (int i = 0; i < R::OUTS; ++i) umma::bar_init(&sh.sent[i], 4);
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
        // this lane's K column of the stage: row trow, chunk half, element lane % 8; row pair i of the angle sits
        // at ((slot * 13 + i) / 4) * 128 + ((slot * 13 + i) % 4) * 4.  The rows' offset spreads the four lanes of an
        // element over the banks: 2.2 wavefronts a store on average over all angles, 3.2 without
        const uint32_t base = L::W + trow * ROW_W + half * 2048 + (lane & 7) * 16;
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
        uint32_t last0 = 0, last1 = 0;   // the two words written last time
        unsigned n = 0;                  // groups
        for (int u = blockIdx.x; u < units && ok; u += gridDim.x)
        for (Stretch w(u, nt, stretches); w.k0 < w.k1 && ok; ++w.k0) {
            const int x0 = (xm ? w.k0 : w.line) * TP + 1, y0 = (xm ? w.line : w.k0) * TP + 1;
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
                for (int q = crew; q < PARTS && ok; q += STAGES) {
                    const int st = crew;   // a crew has a stage of its own
                    const unsigned fills = (n * PARTS + q) / STAGES;   // of this stage, before
                    const int py = y0 + PART_ROWS * q + trow;
                    uint32_t h0 = 0, h1 = 0, l0 = 0, l1 = 0;
                    int pair = -100;
                    if (live && __any_sync(0xffffffffu, px <= N && py <= N)) {
                        const RayPos at = ray_pos(a.x, ex, (float)py - mid, 0.f, mid);
                        float wv[3];
                        int j;
                        if (rim && __any_sync(0xffffffffu, on_rim(px, py, N))) {
                            ray_weights<RIM>(a, at, 0.f, mid, px, py, N, j, wv);
                        } else if (ends) {
                            ray_weights<ENDS>(a, at, 0.f, mid, px, py, N, j, wv);
                        } else {
                            ray_weights<INNER>(a, at, 0.f, mid, px, py, N, j, wv);
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
                    put(last0, 0, 0);
                    put(last1, 0, 0);
                    last0 = place(pair, st);
                    last1 = place(pair + 1, st);
                    put(last0, h0, l0);
                    put(last1, h1, l1);
                    umma::fence_async_smem();
                    __syncwarp();
                    if (lane == 0) umma::bar_arrive(&sh.w_full[st]);
                }
            }
        }
    } else if (warp == R::MMA) {
        constexpr uint32_t A_M_MAJOR = 1u << 15;
        constexpr uint32_t ID_HI = umma::instr_desc_f16(128, 2 * NS * BLK) | A_M_MAJOR,
                           ID_LO = umma::instr_desc_f16(128, NS * BLK) | A_M_MAJOR;
        const uint32_t acc0 = __reduce_max_sync(0xffffffffu, tmem);   // the same in all lanes, and known to be
        const uint64_t w0 = umma::smem_desc(umma::smem_addr(sm + L::W), 2048),
                       img = umma::smem_desc(umma::smem_addr(sm + L::IMG), 2048 * BLK);
        unsigned n = 0, m = 0, b = 0;   // parts, groups, tiles
        bool ready = false, room = false;   // seen before it was needed: the next stage is full, the accumulator free
        for (int u = blockIdx.x; u < units && ok; u += gridDim.x)
        for (Stretch s(u, nt, stretches); s.k0 < s.k1 && ok; ++s.k0, ++b) {
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
                    const uint64_t bd = img + (uint32_t)(q * (BLK * PART_OP >> 4));
#pragma unroll
                    for (int ks = 0; ks < PART_ROWS; ++ks) {
                        // hi x [hi | lo], then lo x hi on top of hi x lo: of all blocks at once, which reads W once
                        umma::mma_f16(d, w + (ks * ROW_W >> 4), bd + (ks * 4096 * BLK >> 4), ID_HI, q > 0 || ks > 0);
                        umma::mma_f16(d + NS * BLK, w + ((STAGE_HALF + ks * ROW_W) >> 4), bd + (ks * 4096 * BLK >> 4), ID_LO,
                                      true);
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
            for (int u = blockIdx.x; u < units && ok; u += gridDim.x)
            for (Stretch s(u, nt, stretches); s.k0 < s.k1 && ok; ++s.k0, ++b) {
                const int tile = xm ? s.line * nt + s.k0 : s.k0 * nt + s.line;
                const unsigned char* src = tiles + ((size_t)s.block * (nt * nt) + tile) * (BLK * TILE_BYTES);
                ok = umma::bar_wait(&sh.sc_empty[b & 1], ((b >> 1) & 1) ^ 1);
                if (!ok) break;
                umma::bar_expect(&sh.sc_full[b & 1], BLK * SCALE_BYTES);
                umma::bulk_load(sm + L::SCALE + (b & 1) * BLK * SCALE_BYTES, src + BLK * TILE_OP, BLK * SCALE_BYTES,
                                &sh.sc_full[b & 1]);
                ++nsc;
                for (parts = 0; parts < PARTS; ++parts) {
                    const int q = parts;
                    ok = umma::bar_wait(&sh.img_empty[q], (b & 1) ^ 1);
                    if (!ok) break;
                    umma::bar_expect(&sh.img_full[q], BLK * PART_OP);
                    umma::bulk_load(sm + L::IMG + q * BLK * PART_OP, src + q * BLK * PART_OP, BLK * PART_OP, &sh.img_full[q]);
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
    } else if (warp == R::ROWS) {
        // where the rows of every tile and group go: a lane per angle
        unsigned m = 0;
        for (int u = blockIdx.x; u < units && ok; u += gridDim.x) {
            const Stretch w(u, nt, stretches);
            for (int kt = w.k0; kt < w.k1 && ok; ++kt)
                for (int g = 0; g < ngroups && ok; ++g, ++m) {
                    Rows to{};
                    const int t = groups[g] + lane;
                    if (lane < SLOTS && t < groups[g + 1]) {
                        const MmaAngle a = ang[t];
                        auto ray = [&](int i) { return xm ? first_ray(a, mid, i, w.line) : first_ray(a, mid, w.line, i); };
                        const int j = ray(kt);
                        to.place = a.roff - row0 + j - min(ray(w.k0), ray(w.k1 - 1));
                        to.nr = (unsigned char)a.nr;
                        if (kt > w.k0) {
                            const int d = j - ray(kt - 1);   // rays the window moved by
                            to.from = (unsigned char)max(-d, 0);
                            to.to = (unsigned char)(a.nr - max(d, 0));
                        }
                    }
                    ok = umma::bar_wait_warp(&sh.d_empty[m % ACCS], ((m / ACCS) & 1) ^ 1);
                    if (!ok) break;
                    if (lane < SLOTS) sh.rows[m % ACCS][lane] = to;
                    __syncwarp();
                    if (lane == 0) umma::bar_arrive(&sh.rows_full[m % ACCS]);
                }
        }
    } else if (warp >= R::OUT) {
        const int row = (warp & 3) * 32 + lane;   // a warp reads the 32 tensor-memory lanes of its number modulo 4
        const int slot = row / PITCH, r = row % PITCH;
        const int k = (warp - R::OUT) >> 2;       // block
        // 32 staged rows; with one set of warps there is room for two times as many
        unsigned char* const stage0 = sm + L::OUT + (warp - R::OUT) * (128 * NS * 4 / (4 * R::OUTS));
        constexpr int STAGE_STEP = R::OUTS == 1 ? 32 * HALF * 4 : 0;
        const int lines = nt * stretches, slot0 = (warp & 3) * 32 / PITCH;   // a warp's rows belong to two angles
        const size_t plane = (size_t)lines * rows * HALF;
        constexpr int STEPS = NS / 16;   // 16 columns at a time
        unsigned m = 0, b = 0, met = 0;
        for (int u = blockIdx.x; u < units && ok; u += gridDim.x) {
        const Stretch w(u, nt, stretches);
        float* const out = P + ((size_t)(w.block * BLK + k) * 2 * lines + u % lines) * rows * HALF;
        for (int kt = w.k0; kt < w.k1 && ok; ++kt, ++b) {
            ok = umma::bar_wait_warp(&sh.sc_full[b & 1], (b >> 1) & 1);
            const float4* const scale = reinterpret_cast<const float4*>(sm + L::SCALE + ((b & 1) * BLK + k) * SCALE_BYTES);
            for (int g = 0; g < ngroups; ++g, ++m) {
                const bool meet = g == 0;   // all that the four warps sent of the tile before has arrived
                if (ok && meet) {
                    if (lane < 4) umma::bulk_store_wait();
                    __syncwarp();
                    if (lane == 0) umma::bar_arrive(&sh.sent[k]);
                }
                ok = ok && umma::bar_wait_warp(&sh.rows_full[m % ACCS], (m / ACCS) & 1);
                if (!ok) break;
                const Rows to = sh.rows[m % ACCS][slot];
                const int prow = to.place + r;
                const bool live = r < to.nr, old = r >= to.from && r < to.to;
                // lanes 0..3 send the rows: of either angle those to be added, and those to be stored
                const unsigned all = __ballot_sync(0xffffffffu, live), first = __ballot_sync(0xffffffffu, slot == slot0),
                               added = __ballot_sync(0xffffffffu, old);
                const unsigned mine = all & (lane & 2 ? ~first : first) & (lane & 1 ? ~added : added);
                const int from = mine ? __ffs(mine) - 1 : 0, n_rows = lane < 4 ? __popc(mine) : 0;
                const int to_row = __shfl_sync(0xffffffffu, prow, from);
                ok = umma::bar_wait_warp(&sh.d_full[m % ACCS], (m / ACCS) & 1);
                if (ok && meet) {
                    ok = umma::bar_wait_warp(&sh.sent[k], met++ & 1);
                    umma::fence_async_global();
                }
                if (!ok) break;
                umma::fence_after();
                const uint32_t d = tmem + ((uint32_t)((warp & 3) * 32) << 16) + (m % ACCS) * ACC_COLS + k * NS;
                // with the next columns on their way meanwhile, in more registers, it took 9 % longer
                float2 v[8], x[8];
                auto fetch = [&](int i) {
                    umma::tmem_ld16(d + 16 * i, v);
                    umma::tmem_ld16(d + NS * BLK + 16 * i, x);
                };
                fetch(0);
#pragma unroll
                for (int i = 0; i < STEPS; ++i) {
                    umma::tmem_ld_wait(v, x);
                    if (i + 1 == STEPS) {
                        umma::fence_before();
                        __syncwarp();
                        if (lane == 0) umma::bar_arrive(&sh.d_empty[m % ACCS]);
                    }
                    if (i % 2 == 0) {
                        // the staged rows are on their way out no longer
                        if (lane < 4) umma::bulk_store_wait_read<R::OUTS == 1 ? 1 : 0>();
                        __syncwarp();
                    }
                    if (live) {
                        // a row's 16-byte pieces are permuted by its number: no bank conflicts
                        unsigned char* const to = stage0 + i / 2 * STAGE_STEP + lane * (HALF * 4);
                        const float4* const sc = scale + 4 * i;
#pragma unroll
                        for (int c = 0; c < 4; ++c) {
                            const float4 f = sc[c];
                            const float2 e0 = mul2(add2(v[2 * c], x[2 * c]), make_float2(f.x, f.y));
                            const float2 e1 = mul2(add2(v[2 * c + 1], x[2 * c + 1]), make_float2(f.z, f.w));
                            *reinterpret_cast<float4*>(to + ((4 * (i % 2) + c) ^ (prow & 7)) * 16) =
                                make_float4(e0.x, e0.y, e1.x, e1.y);
                        }
                    }
                    if (i + 1 < STEPS) fetch(i + 1);
                    if (i % 2 == 1) {
                        umma::fence_async_smem();
                        __syncwarp();
                        if (lane < 4) {
                            float* const dst = out + i / 2 * plane + (size_t)to_row * HALF;
                            const unsigned char* const src = stage0 + i / 2 * STAGE_STEP + from * (HALF * 4);
                            if (n_rows == 0)
                                umma::bulk_store_none();
                            else if (lane & 1)
                                umma::bulk_store(dst, src, n_rows * HALF * 4);
                            else
                                umma::bulk_add(dst, src, n_rows * HALF * 4);
                        }
                    }
                }
            }
            __syncwarp();
            if (ok && lane == 0) umma::bar_arrive(&sh.sc_empty[b & 1]);
        }
        }
        if (lane < 4) umma::bulk_store_wait();
    }
    if (!ok) atomicExch(err, 1);
    umma::fence_before();
    __syncthreads();
    if (warp == R::MMA) umma::tmem_free<512>(tmem);
}

// One ray and 16 slices per thread (four pieces of 16 bytes): the partial sums
// of the stretches whose window holds the ray, stretch by stretch along the lines and in
// a stretch's column from line to line.  Four threads read the 128 contiguous bytes
// of a row and 32 slices.
__global__ void __launch_bounds__(256) k_mma_reduce(const float* __restrict__ P, float* __restrict__ sino,
                                                    const MmaAngle* __restrict__ ang, int N, int T, int nt,
                                                    int stretches, int G, int g0, int t0, int row0, int rows, float mid,
                                                    const int* __restrict__ err)
{
    const int c = threadIdx.x & 3;
    const int j = blockIdx.x * 64 + (threadIdx.x >> 2) + 1;
    if (j > N) return;
    const MmaAngle a = ang[t0 + blockIdx.y];
    const bool xm = fabsf(a.c) >= fabsf(a.s);
    const float inv = 1.f / (TP * (xm ? a.c : -a.s));   // lines per ray
    const size_t plane = (size_t)nt * stretches * rows * (HALF / 4);   // 32 slices of every partial sum
    const float4* base = reinterpret_cast<const float4*>(P) + (size_t)blockIdx.z * 2 * plane;
    const int lrow = a.roff - row0;
    float4 acc[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) acc[k] = make_float4(0.f, 0.f, 0.f, 0.f);
    for (int q = 0; q < stretches; ++q) {
        const int k0 = q * nt / stretches, k1 = (q + 1) * nt / stretches - 1;
        // the lines that can hold the ray, with a margin
        const float va = xm ? window_lo(a, mid, k0 * TP + 1, 1) : window_lo(a, mid, 1, k0 * TP + 1);
        const float vb = xm ? window_lo(a, mid, k1 * TP + 1, 1) : window_lo(a, mid, 1, k1 * TP + 1);
        const float e0 = ((float)j - fminf(va, vb)) * inv, e1 = ((float)(j - a.nr) - fmaxf(va, vb)) * inv;
        const int l0 = max((int)ceilf(fminf(e0, e1) - 0.01f), 0), l1 = min((int)floorf(fmaxf(e0, e1) + 0.01f), nt - 1);
        for (int l = l0; l <= l1; l += 4)
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const int b = l + i;
                const int ja = xm ? first_ray(a, mid, k0, b) : first_ray(a, mid, b, k0);
                const int jb = xm ? first_ray(a, mid, k1, b) : first_ray(a, mid, b, k1);
                const int r = j - min(ja, jb);
                if (b <= l1 && (unsigned)r < (unsigned)(abs(ja - jb) + a.nr)) {
                    const float4* row = base + ((size_t)(b * stretches + q) * rows + lrow + r) * (HALF / 4);
                    const int sw = (lrow + r) & 7;
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
        reinterpret_cast<float4*>(sino)[((size_t)g * T + a.at) * N + (j - 1)] = o;
    }
}

// One block per tile and 64-slice block: the tile's values, scaled per slice so
// that the largest lies in [2^14, 2^15), as hi and lo halves in operand layout
// ([pixel / 8][hi: 64 slices, lo: 64 slices][pixel % 8], of two blocks 128 slices
// each), then the factors that undo the scales of image and weights.
__global__ void __launch_bounds__(256) k_mma_tiles(const float4* __restrict__ img, unsigned char* __restrict__ tiles,
                                                   int N, int nt, int G, int g0, int blk, unsigned* top)
{
    top += g0 * 4 + blockIdx.y * NS;   // the slices' largest magnitudes
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
    unsigned char* const out = tiles + ((size_t)(blockIdx.y / blk) * gridDim.x + tile) * (blk * TILE_BYTES);
    const int kb = blockIdx.y % blk;
    const int warp = tid >> 5, lane = tid & 31;
    for (int n = warp; n < NS; n += 8) {
        unsigned m = 0;
#pragma unroll
        for (int k = 0; k < TP * TP; k += 32) m = max(m, __float_as_uint(s_v[n * LD + k + lane]) & 0x7fffffffu);
        m = __reduce_max_sync(0xffffffffu, m);
        if (lane == 0) {
            if (m > top[n]) atomicMax(top + n, m);
            if (m >= 0x7f800000u) m = 0;
            const int e = m ? max((int)(m >> 23) - 127, -98) : 0;
            s_scale[n] = __int_as_float((14 - e + 127) << 23);
            reinterpret_cast<float*>(out + blk * TILE_OP)[kb * NS + n] = __int_as_float((e - 14 + 127) << 23);
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
        reinterpret_cast<uint4*>(out)[(kc * 2 + lo) * blk * NS + kb * NS + n] = *reinterpret_cast<const uint4*>(h);
    }
}

// Slices by plain gathers (as k_radon): those that held a value that is not finite (a slice is a column of the product,
// which spreads such a value over its tiles and no further), and those whose values are all below 2^-80 (partial sums in
// subnormals would be lost).  Held by the L1 data path; one such slice of 256 at 2049^2 x 1200: 17 ms (168 / 185 ms the
// projection), 23 ms with eight steps of a ray side by side at all angles.
__global__ void __launch_bounds__(128) k_radon_flagged(const float* __restrict__ img, const float* __restrict__ sc,
                                                       const float4* __restrict__ xsc, float* __restrict__ sino, int N,
                                                       int T, int G, float mid, const unsigned* __restrict__ top)
{
    auto marked = [&](int s) { return top[s] >= 0x7f800000u || top[s] - 1u < 0x17800000u - 1u; };   // 2^-80
    bool any = false;
    for (int i = threadIdx.x; i < 4 * G; i += 128) any |= marked(i);
    if (!__syncthreads_or(any)) return;
    const int nb = (N + 127) / 128, lane = threadIdx.x & 31;
    for (size_t g = 0; g < G; ++g) {
    bool m[4];
#pragma unroll
    for (int v = 0; v < 4; ++v) m[v] = marked((int)g * 4 + v);
    if (!(m[0] || m[1] || m[2] || m[3])) continue;
    // eight neighbouring lanes read pixels of the same row or of few: they take eight steps of a ray, or with steeper rays
    // neighbouring ones, staggered so that a step of theirs stays in a row
    for (long long it = blockIdx.x; it < (long long)nb * T; it += gridDim.x) {
        const int t = (int)(it / nb);
        const float s = sc[2 * t], c = sc[2 * t + 1];
        const int ns = fabsf(s) < 0.3f ? 8 : 1, kb = ns == 1 ? __float2int_rn((float)lane * (c / s)) : 0;
        for (int i = 0; i < 32; i += 32 / ns) {
            const int jy = (int)(it % nb) * 128 + (threadIdx.x & ~31) + 1 + i + lane / ns;
            const ProjRay<float, true> ray(sc, xsc, t, jy, mid, nullptr);
            const float* u = img + g * N * N * 4;
            int lo, hi;
            valid_steps(s, c, (float)jy - mid, mid, N, lo, hi);
            if (jy > N || lo > hi) {
                lo = 0x3fffffff;
                hi = -0x3fffffff;
            }
            const int from = ns == 1 ? __reduce_min_sync(0xffffffffu, lo + kb) : lo + lane % ns;
            const int to = ns == 1 ? __reduce_max_sync(0xffffffffu, hi + kb) : hi;
            Lanes<float, 4> acc{};
#pragma unroll 2
            for (int k = from; k <= to; k += ns) {
                const int jx = k - kb;
                if (jx < lo || jx > hi) continue;
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
            for (int o = ns / 2; o > 0; o >>= 1)
#pragma unroll
                for (int v = 0; v < 4; ++v) acc.v[v] += __shfl_xor_sync(0xffffffffu, acc.v[v], o);
            if (lane % ns > 0 || jy > N) continue;
#pragma unroll
            for (int v = 0; v < 4; ++v)
                if (m[v]) sino[((g * T + t) * N + (jy - 1)) * 4 + v] = acc.v[v] / (float)N;
        }
    }
    }
}

}  // namespace

// Stretches per line of tiles: the longer, the fewer partial sums leave the
// L2 cache and are read back (22 rows for the first tile and 6 on average for
// every further one, against 22 for every tile), but the SMs have to share them evenly.
int mma_stretches(int N, int sms)
{
    const int nt = (N + TP - 1) / TP;
    int best = 1;
    double least = 0;
    for (int q = 1; q <= nt; ++q) {
        const int len = (nt + q - 1) / q;
        const double rows = (6. * (len - 1) + 22.) / len;
        const double cost = (double)((nt * q + sms - 1) / sms) * len * (1. + 0.5 * rows / 22.);
        if (q == 1 || cost < least) {
            least = cost;
            best = q;
        }
    }
    return best;
}

std::vector<MmaAngle> mma_angles(const float* xsc, int T, int N, int stretches)
{
    const int nt = (N + TP - 1) / TP, len = (nt + stretches - 1) / stretches;
    std::vector<MmaAngle> out;
    out.reserve(T);
    int roff = 0;
    for (int pass = 0; pass < 2; ++pass)
        for (int t = 0; t < T; ++t) {
            MmaAngle a;
            a.x = make_float4(xsc[4 * t], xsc[4 * t + 1], xsc[4 * t + 2], xsc[4 * t + 3]);
            a.s = a.x.x + a.x.z;
            a.c = a.x.y + a.x.w;
            const bool xm = std::fabs(a.c) >= std::fabs(a.s);
            if (xm == (pass == 1)) continue;
            a.t = xm ? a.s / a.c : -a.c / a.s;
            const float sum = std::fabs(a.c) + std::fabs(a.s);
            a.reach = sum + 1e-3f;   // window_lo's own rounding is below 1e-3
            // integers an interval of 17 (|c| + |s|) + 0.002 (15 across the tile, one reach at each end) can hold
            a.nr = std::min(WIN, (int)std::floor((TP + 1) * sum + 0.002f) + 1);
            a.span = (int)std::floor(TP * (len - 1) * std::fabs(xm ? a.s : a.c) + 0.01f) + 1 + a.nr;
            a.roff = roff;
            a.at = t;
            roff += a.span;
            out.push_back(a);
        }
    return out;
}

// First angles of the groups that share an operand: five angles along the same
// axis, or four when the fifth would need 25 rows.
std::vector<int> mma_groups(const std::vector<MmaAngle>& ang)
{
    std::vector<int> g;
    const int T = (int)ang.size();
    auto xm = [&](int t) { return std::fabs(ang[t].c) >= std::fabs(ang[t].s); };
    for (int t = 0; t < T;) {
        g.push_back(t);
        int n = 1;
        while (n < SLOTS && t + n < T && xm(t + n) == xm(t)) ++n;
        t += n == SLOTS && ang[t + SLOTS - 1].nr > 128 - (SLOTS - 1) * PITCH ? SLOTS - 1 : n;
    }
    g.push_back(T);
    return g;
}

static size_t part_rows(const DevGeom<float>& g, int ga, int gb)   // rows of the groups [ga, gb)
{
    const MmaAngle& last = g.h_mma[g.h_groups[gb] - 1];
    return last.roff + last.span - g.h_mma[g.h_groups[ga]].roff;
}

// Groups [first, last) cut into chunks of at most ng, even ones: the first group after ga's chunk.
static int chunk_end(int first, int last, int ng, int ga)
{
    const int n = last - first, chunks = (n + ng - 1) / ng, i = (int)(((long long)(ga - first) * chunks + chunks - 1) / n);
    return first + (int)((long long)(i + 1) * n / chunks);
}

// Groups of angles at once: as many as keep the rows that the SMs are adding to
// in the L2 cache (bulk reductions there ran at 6.3 TB/s, at 3.3 where the rows
// were 150 MB).  More would read the tiles less often (64 KB per tile and chunk).
MmaPlan mma_plan(const DevGeom<float>& g, int G, size_t cap)
{
    MmaPlan p;
    p.nt = (g.N + TP - 1) / TP;
    p.nblk = (G * 4 + NS - 1) / NS;
    const int units = p.nt * g.stretches;
    // blocks go in pairs, which share every W; more where a pair's units are few
    p.nb = std::min(p.nblk, 2);
    if (p.nb == 2 && units < 4 * g.sms) p.nb = std::min(p.nblk, 2 * ((4 * g.sms + units - 1) / units));
    if (p.nb > 2) p.nb &= ~1;
    const size_t row = (size_t)NS * sizeof(float), active = row * 22 * SLOTS * std::min(g.sms, units) * std::min(p.nb, 2);
    p.ng = (int)std::min<size_t>(g.n_groups, std::max<size_t>(1, MMA_L2_ROWS / active));
    size_t rows;
    for (;;) {
        rows = 0;
        for (int x = 0; x < 2; ++x) {
            const int first = x ? g.n_groups_x : 0, last = x ? g.n_groups : g.n_groups_x;
            for (int a = first, b; a < last; a = b) {
                b = chunk_end(first, last, p.ng, a);
                rows = std::max(rows, part_rows(g, a, b));
            }
        }
        if (row * rows * units * p.nb <= cap || (p.nb <= 2 && p.ng == 1)) break;
        if (p.nb > 2) p.nb -= 2;
        else --p.ng;
    }
    p.tile_bytes = (size_t)p.nt * p.nt * p.nb * TILE_BYTES;
    p.part_bytes = row * rows * units * p.nb;
    return p;
}

size_t mma_flag_words(int G) { return 1 + (size_t)(G * 4 + NS - 1) / NS * NS; }

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
    // [0] a wait gave up, then the slices' largest magnitudes
    unsigned* const top = reinterpret_cast<unsigned*>(flags) + 1;
    cudaMemsetAsync(flags, 0, sizeof(int) * mma_flag_words(G), st);
    for (int b = 0; b < p.nblk; b += p.nb) {
        const int nb = std::min(p.nb, p.nblk - b);
        k_mma_tiles<<<dim3(nt2, nb), 256, NS * (TP * TP + 5) * sizeof(float), st>>>(
            reinterpret_cast<const float4*>(img), tiles, N, p.nt, G, b * (NS / 4), nb % 2 == 0 ? 2 : 1, top);
        for (int x = 0; x < 2; ++x) {
            const int first = x ? g.n_groups_x : 0, last = x ? g.n_groups : g.n_groups_x;
            for (int ga = first, gb; ga < last; ga = gb) {
                gb = chunk_end(first, last, p.ng, ga);
                const int t0 = g.h_groups[ga], t1 = g.h_groups[gb];
                const int row0 = g.h_mma[t0].roff, rows = (int)part_rows(g, ga, gb);
                const int blk = nb % 2 == 0 ? 2 : 1;   // 64-slice blocks per operand W
                const int units = p.nt * g.stretches * (nb / blk);
                (blk == 2 ? k_mma_project<2> : k_mma_project<1>)<<<
                    std::min(g.sms, units), 32 * (blk == 2 ? Roles<2>::WARPS : Roles<1>::WARPS),
                    (blk == 2 ? Smem<2>::BARS : Smem<1>::BARS) + sizeof(Shared), st>>>(
                    tiles, P, g.mma, g.groups + ga, N, p.nt, g.stretches, x == 0, units, gb - ga, row0, rows, g.mid,
                    flags);
                k_mma_reduce<<<dim3((N + 63) / 64, t1 - t0, nb), 256, 0, st>>>(
                    P, sino, g.mma, N, T, p.nt, g.stretches, G, b * (NS / 4), t0, row0, rows, g.mid, flags);
            }
        }
    }
    k_radon_flagged<<<g.sms * 8, 128, 0, st>>>(img, g.sc_fp, g.xsc_fp, sino, N, T, G, g.mid, top);
}

}  // namespace acu

// Internal launcher declarations shared by the .cu translation units.
#pragma once
#include <algorithm>
#include <cuda_runtime.h>
#include <stddef.h>
#include <stdint.h>

#include <vector>

namespace acu {

// The exact backprojection's per-angle table as a kernel parameter (up to
// BP_TMAX angles; kernel parameters may take up to 32 KB).
constexpr int BP_TMAX = 1920;
struct BpTable {
    float4 v[BP_TMAX];
};

// Sine and cosine of an angle times 2^32 (fixed.cuh)
struct FxAngle {
    long long s, c;
};
constexpr int FX_MAX_SIDE = 4097;

// One angle of the tensor-core projector (kernels_radon_mma.cu), for which angles whose
// rays run along x (|c| >= |s|) come before the others, and of the transpose.
struct MmaAngle {
    float4 x;         // split sine and cosine, as xsc_fp
    float c, s, t;    // cosine, sine, slope of a ray's closest approach
    float reach;      // |c| + |s| and a margin: how far a pixel's taps reach across the rays
    int nr;           // rows (rays) of the angle's window in a tile
    int span, roff;   // rows of its window in a stretch of tiles, and those of the angles before it
    int at;           // the angle's number
};

// Geometry of one reconstruction grid on the device, for one precision.
// All tables are computed on the host (tables.cpp) with the reference's
// arithmetic and uploaded once.
template <typename Real>
struct DevGeom {
    int N = 0, T = 0;
    Real mid = 0;                 // (N+1)/2, integer division (tv_hpc.F90:15)
    const Real* sc_bp = nullptr;  // [T][2] sin, cos of pi*(90-theta)/180
    const Real* sc_fp = nullptr;  // [T][2] sin, cos of pi*(theta-90)/180
    const Real* filt = nullptr;   // [2N+1] filter taps (tv_hpc.F90:53-56)
    const Real* cmask = nullptr;  // [N][N] tapered mask times pi/T (tv_hpc.F90:58-74)
    const Real* fft_h = nullptr;  // [L] real spectrum of the wrapped filter
    const Real* fft_h_x = nullptr;  // [L] the same from FP64 taps, used with exact positions
    const float2* fft_tw16 = nullptr;  // L = 512 to 4096, single precision: twiddles per pass (tables.h)
    const float2* fft_tw = nullptr; // [L/2] twiddles exp(-2 pi i k / L) (float)
    const double2* fft_tw64 = nullptr;
    int fft_L = 0, fft_log2L = 0;
    const int* fp_order = nullptr;  // [T] projector angles, |sin| >= |cos| first
    const int* lines_order = nullptr;  // projector variant 6: lines_angle_order (chunks of angles, -1 padded)
    // exact positions (single precision only): split FP64 angle tables,
    // [T] x (s_a, c_a, s_r, c_r); exact != 0 selects them
    const float4* xsc_bp = nullptr;
    const float4* xsc_fp = nullptr;
    int exact = 0;
    const FxAngle* fx_fp = nullptr;     // projector's angles in fixed point (single precision)
    const MmaAngle* angles = nullptr;   // single precision: the angles in order
    const MmaAngle* mma = nullptr;      // those along x first, and their host copy
    const MmaAngle* h_mma = nullptr;
    const int* groups = nullptr;        // first angles of its groups, n_groups + 1 of them, and their host copy
    const int* h_groups = nullptr;
    int n_groups = 0, n_groups_x = 0;   // those along x come first
    int stretches = 1;                  // of tiles, per line of them
    int sms = 152;
    const int* tiles_in = nullptr;      // 16 x 16 pixel tiles that meet the mask (n_tiles_in), then the others
    int n_tiles_in = 0;
    const float4* h_xsc_bp = nullptr;   // host copy of xsc_bp (for the parameter table)
    const float4* h_sc_bp = nullptr;    // host copy of sc_bp as (sin, cos, 0, 0), single precision
    int bp_param = 1;                   // backprojection: angle table in the launch parameters when T <= BP_TMAX
    int bp_groups = 0;   // slice groups per backprojection thread: 0 auto (1 with the parameter table, else 2), 1, 2 or 4
    int bp_tma = 0;      // 1: exact backprojection from sinogram bins staged in shared memory by bulk copies
};

// ---- radon operators (kernels_radon.cu); arrays in lane layout ------------
template <typename Real, int V>
void launch_backproject(const DevGeom<Real>& g, int G, const Real* q, Real* img, cudaStream_t st);
template <typename Real, int V>
void launch_radon(const DevGeom<Real>& g, int G, const Real* img, Real* sino, cudaStream_t st);
// Projector through pair images (float, 4 slices per thread): P and PT are
// work buffers of 2 * N * N * 4 floats per slice group each.
void launch_radon_pairs(const DevGeom<float>& g, int G, const float* img, float* P, float* PT, float* sino,
                        cudaStream_t st);
// Same projector on the lane image and its transpose IT (N * N * 4 floats per
// slice group), four 128-bit loads per sample.
// par: the four taps loaded by row parity (odd row of the cell first);
// reuse: taps of the previous sample kept in registers; clip (with reuse):
// steps limited to those that can meet a valid cell.
void launch_radon_quads(const DevGeom<float>& g, int G, const float* img, float* IT, float* sino, cudaStream_t st,
                        bool par = false, bool reuse = false, bool clip = false, bool f2 = false);
// Projector variant 6 (kernels_lines.cu): the batch regrouped into 128-byte
// pixel lines of 32 slices, walked in bands of rows that stay in L2.  L and A
// are work buffers of lines_image_floats and lines_sums_floats floats.
void launch_radon_lines(const DevGeom<float>& g, int G, const float* img, float* L, float* A, float* sino,
                        cudaStream_t st);
size_t lines_image_floats(int N, int G);
size_t lines_sums_floats(int N, int T, int G);
int lines_band_rows(int N);
// The band launches' angle order for single-precision (sin, cos) pairs sc[2T].
std::vector<int> lines_angle_order(const float* sc, int T);
// Projector on the tensor cores (kernels_radon_mma.cu; exact positions):
// 64-slice blocks of 16 x 16 pixel tiles in operand layout, partial sums of a
// chunk of angles, a flag (a wait gave up) and the slices' largest magnitudes.
struct MmaPlan {
    int nt = 0;        // tiles per side
    int nblk = 0;      // 64-slice blocks of the batch
    int nb = 0;        // of them at once
    int ng = 0;        // groups of angles at once, at most
    size_t tile_bytes = 0, part_bytes = 0;
};
constexpr size_t MMA_PART_CAP = (size_t)4 << 30;   // bytes of partial sums at once
int mma_stretches(int N, int sms);
std::vector<MmaAngle> mma_angles(const float* xsc, int T, int N, int stretches);
bool mma_fits(int N);
std::vector<int> mma_groups(const std::vector<MmaAngle>& ang);
size_t mma_flag_words(int G);
MmaPlan mma_plan(const DevGeom<float>& g, int G, size_t cap);
void launch_radon_mma(const DevGeom<float>& g, int G, const float* img, unsigned char* tiles, float* P, int* flags,
                      const MmaPlan& p, float* sino, cudaStream_t st);
// Backprojection on the tensor cores (kernels_bp_mma.cu; exact positions): work
// buffers of bp_mma_bins_bytes bytes and bp_mma_scalars words.  filtered: q comes
// from this library's filter.  False if the
// driver has no tensor maps (nothing usable was written).
int bp_tiles(const float* cmask, int N, std::vector<int>& list);
size_t bp_mma_bins_bytes(int N, int T, int G);
size_t bp_mma_scalars(int G);
bool launch_backproject_mma(const DevGeom<float>& g, int G, const float* q, bool filtered, void* bins, unsigned* scalars,
                            float* img, cudaStream_t st);
// Single-slice kernels at exact positions (kernels_single.cu).  launch_radon_fx
// (sides up to FX_MAX_SIDE); launch_ray_off: with per-angle offsets or null, dsino
// the derivative with respect to them or null; launch_backproject_fx: q as pairs
// (bin, next bin), which the filter writes or launch_pairs makes from
// n = slices * T * N bins; launch_adjoint_fx: the projector's transpose.
// Their buffers of pairs hold 1 GB at most, as many slices as that takes: slices
// at once of so many bytes each, and the floats of a projector's buffer.
inline int pair_slices(size_t bytes, int S)
{
    return (int)std::max<size_t>(1, std::min<size_t>(S, ((size_t)1 << 30) / bytes));
}
inline size_t pair_image_floats(int N, int S) { return (size_t)4 * N * N * pair_slices((size_t)16 * N * N, S); }
std::vector<FxAngle> fx_angles(const float* xsc, int T);
void launch_radon_fx(const DevGeom<float>& g, int S, const float* img, float* IT, float* sino, cudaStream_t st);
void launch_ray_off(const DevGeom<float>& g, int S, const float* img, float* IT, const float* off, float* sino,
                    float* dsino, cudaStream_t st);
void launch_backproject_fx(const DevGeom<float>& g, int S, const float2* q, float* img, cudaStream_t st);
template <int V>
void launch_adjoint_fx(const DevGeom<float>& g, int G, const float* sino, const float* off, float* img, cudaStream_t st);
void launch_pairs(const float* q, float2* out, int N, size_t n, cudaStream_t st);
void launch_transpose_v1(int N, int S, const float* img, float* IT, cudaStream_t st);
// The single-slice projector: through pairs (IT of pair_image_floats floats), else along
// staggered rays through the image and its transpose (IT of N * N floats per slice).
inline bool radon_v1_pairs(const DevGeom<float>& g) { return g.exact && g.N <= FX_MAX_SIDE; }
void launch_radon_v1_fast(const DevGeom<float>& g, int S, const float* img, float* IT, float* sino, cudaStream_t st);
template <typename Real, int V>
void launch_radon_adjoint(const DevGeom<Real>& g, int G, const Real* sino, Real* img, cudaStream_t st);
template <typename Real, int V>
void launch_filter_direct(const DevGeom<Real>& g, int G, const Real* sino, Real* out, cudaStream_t st);
template <typename Real, int V>
void launch_filter_fft(const DevGeom<Real>& g, int G, const Real* sino, Real* out, cudaStream_t st,
                       bool pairs = false);   // pairs (V = 1): as launch_backproject_fx reads them
template <typename Real>
bool fft_fits(int L);

// ---- projector / adjoint with per-slice, per-angle detector offsets off[S][T]
// (plain layout, one slice per thread) and the offset derivative of the
// projector (kernels_radon.cu); the loss / gradient steps (kernels_grad.cu).
template <typename Real>
void launch_radon_off(const DevGeom<Real>& g, int S, const Real* img, const Real* off, Real* sino, cudaStream_t st);
template <typename Real>
void launch_radon_adjoint_off(const DevGeom<Real>& g, int S, const Real* sino, const Real* off, Real* img,
                              cudaStream_t st);
template <typename Real>
void launch_radon_doff(const DevGeom<Real>& g, int S, const Real* img, const Real* off, Real* dsino, cudaStream_t st);
template <typename Real>
struct GradEw {
    // r = A u - y in place (r holds A u), per-slice FP64 partials of 1/2 |r|^2
    static void residual(size_t n_per, int S, Real* r, const Real* y, double* part, int nblk, cudaStream_t st);
    // grad_u += lambda * dTV_eps/du; per-slice partials of lambda * TV_eps(u)
    static void tv_grad(int N, int S, Real lambda, Real eps, const Real* u, Real* grad, double* part, int nblk,
                        cudaStream_t st);
    // grad_off[s][t] = sum_jy r * D
    static void off_grad(int N, int T, int S, const Real* r, const Real* D, Real* grad_off, cudaStream_t st);
};
void launch_sum_rows(const double* part, int rows, int nblk, double* out, cudaStream_t st);

// ---- layout conversion (kernels_tv.cu) ------------------------------------
// plain [S][npos] <-> lanes [G][npos][V]; slices >= S of the last group are 0.
template <typename Real, int V>
void launch_to_lanes(const Real* plain, Real* lanes, int S, size_t npos, cudaStream_t st);
template <typename Real, int V>
void launch_from_lanes(const Real* lanes, Real* plain, int S, size_t npos, cudaStream_t st);
template <typename Real>
void launch_convert(const float* in, Real* out, size_t n, cudaStream_t st);

// ---- split-Bregman / CG elementwise steps (kernels_tv.cu) ----------------
// All images are [G][N][N][V]; per-slice scalars are double[G*V].
struct TvScalars {
    double* rsold;   // [S]
    double* alpha;   // [S]
    double* beta;    // [S]
    double* delta;   // [S] Err_diff
    double* part;    // [nblk_max * S] block partial sums
    int nblk;        // blocks of the elementwise grid
};

template <typename Real, int V>
struct TvEw {
    // ifkt2 (optional) is added to ifkt
    static void rhs(int N, int G, Real mu, Real lambda, const Real* ifkt, const Real* dx,
                    const Real* bx, const Real* dy, const Real* by, Real* rhs, cudaStream_t st,
                    const Real* ifkt2 = nullptr);
    static void resid(int N, int G, Real mu, Real lambda, const Real* rhs, const Real* iukt,
                      const Real* uk, Real* r, Real* p, const TvScalars& sc, cudaStream_t st);
    static void apply(int N, int G, Real mu, Real lambda, const Real* irpt, const Real* p,
                      Real* Ap, const TvScalars& sc, cudaStream_t st);
    // with irpt and bd: bd -= alpha irpt as well (the carried iradon(f - radon(uk)))
    static void update(int N, int G, const Real* p, const Real* Ap, Real* uk, Real* r,
                       const TvScalars& sc, cudaStream_t st, const Real* irpt = nullptr, Real* bd = nullptr);
    static void pupdate(int N, int G, const Real* r, Real* p, const TvScalars& sc, cudaStream_t st);
    static void shrink(int N, int G, Real lambda, const Real* uk, Real* dx, Real* bx, Real* dy,
                       Real* by, const Real* ukp, const TvScalars& sc, cudaStream_t st);
    static void fk_update(size_t n, Real* fk, const Real* f, const Real* ruk, cudaStream_t st);
    // y += alpha_slice * x over sinograms (radon(uk) carried through uk += alpha p)
    static void sino_axpy(int T, int N, int G, const Real* x, Real* y, const TvScalars& sc, cudaStream_t st);
    // out = a - b (the data residual fk - radon(uk) of the merged initial residual)
    static void diff(size_t n, const Real* a, const Real* b, Real* out, cudaStream_t st);
    // y += x
    static void add(size_t n, const Real* x, Real* y, cudaStream_t st);
};

// Finalisers of the FP64 CG scalars (one block per slice, fixed order).
// which: 0 -> rsold = sum;  1 -> alpha = rsold / sum;  2 -> beta = sum / rsold,
// rsold = sum;  3 -> delta = sum.
void launch_cg_finalize(int which, int S, const TvScalars& sc, cudaStream_t st);

}  // namespace acu

// Internal definitions shared by the host planner (plan.cpp, capi.cpp) and the
// CUDA kernels (radiality.cu, temporal.cu). Not part of the public C-ABI.
#pragma once
#include <vector_types.h>

#include <array>
#include <cstdint>
#include <cstddef>
#include <string>
#include <vector>

#include "../../include/rfba_srrf.h"

namespace rfba {

// Output tile of the radiality kernel: 16 x TY subvoxel columns (one per thread,
// TY = kTileRows unless tuned) and FZ = MZ * CZ subvoxels deep along its innermost axis, held in registers.
constexpr int kTileX = 16;
constexpr int kTileRows = 8;
constexpr int kMaxThreads = 256;  // 16 x 16, the taller tile of the schedule search
constexpr int kMaxMag = 8;
constexpr int kMaxGradRange = 3;
// Bound on the static shared memory of the radiality kernel and its adjoint; no configuration
// needs more dynamic shared memory than it leaves of a block's.
constexpr size_t kStaticShared = 1024;
// The forward kernel's register limit for MZ x CZ tiles: MZ CZ for the sums and
// 6 (CZ / 2 + 4) for the x-filtered columns are live through the point loop.
constexpr int fwd_regs(int mz, int cz) { return mz * cz + 6 * (cz / 2 + 4) <= 88 ? 128 : 168; }

// The adjoint's tile depth (it holds two sets of columns), its register limit (12
// (CZ / 2 + 4) for the columns and MZ CZ for dL/dS leave no instance below 128) and the
// width of an exchange row per x phase (the tile's coarse cells and four zeros).
constexpr int adj_cz(int mz) { return mz <= 4 ? 8 : 4; }  // half of it for launches of few items
constexpr int kAdjRegs = 168;
#ifdef __CUDACC__
__host__ __device__
#endif
constexpr int adj_cells(int mx) { return 15 / mx + 2 + 4; }

// One independent block of the input with the fine region it computes.
struct BlockDev {
    int origin[3];   // input voxel origin in the full volume
    int size[3];     // block dims (input voxels)
    int lo[3];       // fine region [lo, hi) in block-local magnified coords
    int hi[3];
    int rad_lo[3];   // fine indices whose ring samples all pass the window (inclusive)
    int rad_hi[3];
    int int_lo[3];   // fine indices whose centre passes the window (inclusive)
    int int_hi[3];
    int ntile[3];    // tiles along x, y, z
    int nreg[3];     // region extent hi - lo
    int cz;          // coarse cells per tile along its innermost axis
    long long vox;        // region voxels
    long long stack_off;  // element offset of this block's [t][v] stack slice
    long long out_offset;
    long long out_stride[3];
};

// Tile work unit: block index and tile coordinates along x, y, z.
struct TileDesc {
    int block, t[3];
};

// Deduplicated ring and its factorisation per axis. The n^2 ring samples of
// kernel.cu:23-33 collapse to distinct points (62 for n = 12) with integer
// multiplicities; distinct x / y / z coordinate values index the separable
// Catmull-Rom weight tables.
struct RingPlan {
    int n = 0;                     // samples per angle (2 * AxesinRing)
    std::vector<float> xv, yv, zv; // distinct coordinate values per axis
    // Point list grouped by x value, then y value: group g covers pairs
    // [grp[g], grp[g+1]); pair p covers points [pair_pt[p], pair_pt[p+1]).
    std::vector<int> grp_xval;     // per group: x value index
    std::vector<int> grp;          // ngroups + 1
    std::vector<int> pair_yval;    // per pair: y value index
    std::vector<int> pair_pt;      // npairs + 1
    std::vector<int> pt_zval;      // per point: z value index
    int zero_x = -1, zero_y = -1;  // value index of 0 on x and y
    int npoints_raw = 0;
    // Raw float ring (n*n points) exactly as the reference builds it.
    std::vector<float> rx, ry, rz;
};

// The adjoint's least c2 g2 under 1 / sqrt(c2 g2).
constexpr float kGuard = 1e-30f;

// Largest uniform table (float4s) that travels in the parameters of the radiality kernel
// or its adjoint: parameters hold 32764 bytes. Rings of 12 axes and most of 13 fit (the
// adjoint's table, which has the x weights too, up to 10 to 12). 20 volumes of 32^3 at 2 x 2
// x 2, ms with a limit of 768 (1024), whose rings of 9 axes and more read global memory, and
// now: 9 axes 1.34 and 1.02, 12 axes 2.20 and 1.76; with the adjoint 4.46 and 4.14, 8.79
// and 6.91.
constexpr int kUTabMax = 1984;
// Largest table in the smaller parameters: every launch copies all of them, and a call on a
// host buffer of 5 x 10x12x12 takes 102 us with 1984 records, 98 with 768.
constexpr int kUTabSmall = 768;
// Deepest innermost magnification with tiles of 8 cells: above it the sums would not fit
// the registers beside the columns.
constexpr int kDeepMag = 5;
// Innermost magnifications from this on have tiles of 2 cells too, for launches of few items.
constexpr int kFlatMag = 5;
// Quads of innermost cells that a tile of cz cells and its taps take.
#ifdef __CUDACC__
__host__ __device__
#endif
constexpr int tile_quads(int cz) { return (cz + 7) / 4; }

// The forward kernel's plan of a configuration. Its tiles run over (x, mid,
// innermost) = (x, y, z) or (x, z, y). The first pass filters along mid, once for
// each of its distinct ring values; the second along x, once for each (mid, x) pair
// and cell of the innermost axis, (CZ + 4) / (MZ CZ) per subvoxel, so less the larger
// the innermost magnification MZ; the third along the innermost axis for each point.
// The ring has fewer distinct z than y values (7 against 13 at 6 axes), so z is the
// mid axis unless its magnification is the larger one (arrange() in plan.cpp
// compares the two orders' costs).
//
// A ring point u = (x, m, n)/r belongs to the pair of its (m, x) values. The pair's
// columns are turned into a frame where u lies in the P-Z plane (P along (x, m), E
// across it) with every component scaled by 1 / cos of u's elevation, so that most
// products drop out: with kappa = tan of the elevation dot = P + kappa Z and cp = Z -
// kappa P are the same positive multiple of g.u/|u| and of the part of g across u
// in that plane, and E carries the scale itself. On the axis (x = m = 0) P is the
// innermost component, one pair per direction.
//
// utab, records of float4 (words as int bits where marked *):
//   groups [ngroups]     {mid value*, first pair*, end pair*, 0}
//   pairs  [npairs][4]   P = r0.x A + r0.z B: {r0.x, r0.x, r0.z, r0.z}, E likewise,
//                        {plane of A*, B*, Z*, x value*}, {first point*, end point*, offset mask of the x value*, kGuard x scale^4}
//   points [npoints][3]  {kappa, kappa, -kappa, -kappa}, {-sqrt(rho)|u| x 2, sqrt(rho) x 2},
//                        {first record of the n value's weights*, offset mask*, 0, 0}
//   wz     [nzv][mz][2]  {w0, w0, w1, w1}, {w2, w2, w3, w3}
//   wi     [mz]          the intensity's four weights
// Offset masks: bit ph says that phase ph's taps start one coarse cell later. rho is
// the point's multiplicity over the commonest one, whose weight is neg_weight. lane:
// per x and per mid value and phase the 4 tap weights and their offset, looked up by
// lane and row in shared memory.
struct FwdPlan {
    int mag[3] = {0, 0, 0};  // tile axis order
    int ax1 = 1, ax2 = 2;    // volume axes of the mid and innermost tile axis
    std::vector<float> utab, lane;
    // the adjoint's uniform table: utab with {-2 weight |u|^2 x 2, 2 weight |u| x 2} as the
    // points' second record, and wx [nxv][mx][2] {w0, w0, w1, w1}, {w2, w2, w3, w3} at u_wx
    std::vector<float> adj_utab;
    int u_wx = 0;
    // per point, for the adjoint's samples in a fixed order: {ca, sb, h, c} with u = |u| (h x' +
    // c z), x' = (ca, sb) along the volume's (x, y), and {2 weight |u|, |u|, scale, 0}, scale
    // that of the pair's frame
    std::vector<float> fix;
    int u_grp = 0, u_pair = 0, u_pt = 0, u_wz = 0, u_wi = 0;
    int l_wx = 0, l_offx = 0, l_wm = 0, l_offm = 0;
    int ngroups = 0, npairs = 0, npoints = 0, zero_x = 0, zero_xoff = 0, zero_m = 0;
    float neg_weight = 0.f;
};

// Everything the radiality kernel and its adjoint need; passed by value (the
// adjoint reads float input without TMA staging and writes no stacks).
struct FwdParams {
    const void* in;       // input volume [t][z][y][x]
    int W, H, D, T;       // full input dims
    int in_u16;
    int mag[3];           // tile axis order (x, mid, innermost), as gr
    int ax1, ax2;
    int gr[4];            // gradient ranges: main, x, mid, innermost (smooth=0 => 1,0,0,0)
    int grad_mode;        // 1: ranges (1,1,1,1), 2: (1,0,0,0), 0: generic loops
    int R;                // gradient halo
    int TY, cz;           // subvoxel rows (threads = 16 * TY) and innermost cells per tile
    int NU, NV;           // coarse G tile extents
    int NIX, NIY, NIZ;    // input tile extents (G tile + halo)
    int u_region;         // float4s of the U planes / input tile
    int renorm, poscon;
    int t_chunk, nchunks;
    int ntiles;
    long long nitems;
    const float* lane;    // lane tables
    int lane_words, l_wx, l_offx, l_wm, l_offm;
    const float4* utab;   // uniform tables in global memory (read when they do not fit the parameters)
    int u_count, u_grp, u_pair, u_pt, u_wz, u_wi, u_wx;
    int ngroups, zero_x, zero_xoff, zero_m;
    float neg_weight;     // minus the commonest point's weight
    const BlockDev* blocks;
    const TileDesc* tiles;
    float* rad_stack;     // [block slice][t][v]
    float* int_stack;
    unsigned int* work_counter;
    // TMA staging of the input tile: box width in elements (0 = no staging area)
    // and whether this launch uses it
    int tma_bx;
    int use_tma;
    unsigned long long* err;  // bounded-wait failures (may be null)
    // failure-detection test (RFBA_TEST_TMA_STALL): the first copy request of
    // every work item is left out, so the bounded staging wait gives up
    int test_skip_copy;
    // time window of this launch: volumes [t_lo, t_hi) (t_hi 0: up to T), and
    // the volume held by the first [t] row of the stacks (0 when they hold the
    // whole series, t_lo when they hold one batch)
    int t_lo, t_hi, stack_t0;
};

// Temporal reduction parameters.
struct TemporalParams {
    const BlockDev* blocks;
    const long long* vox_prefix;  // nblocks + 1 cumulative region voxels
    int nblocks;
    long long total_vox;
    int T;
    int method, itc, order, iw;
    float* rad_stack;             // ITC=1 bins the series in place
    const float* int_stack;
    float* out;
};

// Temporal reduction of one time batch into the carried state
// (temporal_stream.cu).
struct StreamParams {
    const BlockDev* blocks;
    const long long* vox_prefix;
    int nblocks;
    long long total_vox;
    int T;                 // the whole series
    int t_lo, t_hi;        // this batch; the stacks hold its [t_hi - t_lo][v]
    int method, order, iw;
    int last;              // write the map after this batch
    int keep;              // after the last batch, store the state as well (for a backward)
    float* state;          // [field][state_stride]
    long long state_stride;
    const float* rad_stack;
    const float* int_stack;
    float* out;
};

// Adjoint of the carried temporal reduction for one batch of one block
// (temporal_stream.cu): dL/dS and dL/dI of the volumes [t_lo, t_hi) from
// dL/dmap, the final carried state and the window stacks [w_lo, w_hi).
struct StreamAdjParams {
    const BlockDev* block;  // stack_off 0
    int T, t_lo, t_hi, w_lo, w_hi;
    int method, order, iw, renorm, poscon;
    const float* state;
    long long state_stride;
    const float* rad;    // [t - w_lo][v]
    const float* inten;
    const float* gmap;
    long long nmap;
    float* gS;           // [t - t_lo][v]
    float* gI;
    unsigned long long* err;
};

// Adjoint inputs and output of the radiality adjoint kernel.
struct AdjParams {
    const float* gS;  // dL/d(radiality before transforms) per subvoxel and time, [t][v]
    const float* gI;  // dL/d(interpolated intensity), [t][v]
    float* gin;       // dL/dI' accumulated, [t][z][y][x] of the full input
    const float4* fix;  // FwdPlan::fix
    long long n_in;   // elements of the input / gin
    long long n_stack;  // elements of gS / gI
    unsigned long long* err;  // first out-of-range global index (site << 56 | index), 0 if none
};

// Launchers (radiality.cu / temporal.cu / adjoint.cu). Return a cudaError_t as int.
int launch_radiality_adjoint(const FwdParams& p, const FwdPlan& plan, const AdjParams& a, int grid, size_t smem,
                             void* stream);
int radiality_adjoint_u_region(const FwdParams& p);
size_t radiality_adjoint_smem_bytes(const FwdParams& p);
int radiality_adjoint_max_ctas_per_sm(const FwdParams& p, int* out);
int launch_temporal_adjoint(const BlockDev* blocks, long long vox, const float* rad, const float* inten,
                            const float* gmap, int T, int method, int itc, int order, int iw, int renorm, int poscon,
                            float* gS, float* gI, long long nmap, unsigned long long* err, void* stream);
int launch_shift_adjoint(const float* src, float* dst, int W, int H, int D, int T, int axis, const float* shifts,
                         int sms, void* stream);
// Drift operator, all axes fused: mode 0 resamples src into dst; mode 1 adds
// sum_voxels g * dI'/dd_a into out[3 t + a] (FP64).
int launch_drift3d(const float* src, float* dst, const float* g, int W, int H, int D, int T, const float* shifts,
                   int mode, double* out, int sms, void* stream);
int launch_double_to_float(const double* src, float* dst, int n, void* stream);
int launch_radiality(const FwdParams& p, const FwdPlan& plan, int grid, size_t smem, void* stream);
// Box width (elements) of the TMA input staging for this tile, 0 when the input
// rows cannot be addressed by a tensor map (row pitch not a multiple of 16 B).
int radiality_tma_box_x(const FwdParams& p);
int radiality_u_region(const FwdParams& p);
size_t radiality_smem_bytes(const FwdParams& p);
int radiality_max_ctas_per_sm(const FwdParams& p, int* out);
int launch_temporal(const TemporalParams& p, void* stream);
int launch_temporal_stream(const StreamParams& p, void* stream);
int launch_temporal_stream_adjoint(const StreamAdjParams& p, long long vox, void* stream);
// state floats per subvoxel for a method (0 TRM, 1 TRA, 2 TRPPM, 3 TRAC ITC 0) and TRAC order
int temporal_stream_fields(int method, int order);
int launch_combine(const double* spots, long long n, int zoom, int Xp, int Yp, int Zp, int r, int rz, int thr,
                   const uint16_t* psf, int Kx, int Ky, int Kz, unsigned int* hist, unsigned char* L,
                   unsigned short* S, unsigned long long* idx, unsigned int* val, unsigned long long cap,
                   unsigned long long* counters, unsigned long long* out, uint16_t* out16, void* stream);
int launch_seed_spots(const float* map, const int map_dims[3], int mag, const int* vox, long long nvox, int nspots,
                      unsigned long long seed, float* xyz, double* w, double* sums, double* carry,
                      unsigned long long* err, void* stream);

// Host planning (plan.cpp).
bool build_ring_plan(const rfba_srrf_config& c, RingPlan* rp, std::string* err);
bool build_forward_plan(const rfba_srrf_config& c, FwdPlan* fp, std::string* err);
// Parameters of a forward launch that follow from the plan and configuration
// (not the block and tile lists, stacks and schedule). ty: tile rows, 0 = default.
FwdParams forward_params(const FwdPlan& fp, const rfba_srrf_config& c, const void* in, int in_u16, const int dims[4],
                         int ty, int cz);
// The same for the adjoint kernel.
FwdParams adjoint_params(const FwdPlan& fp, const rfba_srrf_config& c, const void* in, const int dims[4], int cz);
// Tiles of a block's region [lo, hi) in the plan's tile axes (b->cz set).
void forward_tiles(const FwdPlan& fp, int ty, BlockDev* b);
// Tile depth (innermost cells: 2, 4 or 8) for launches of these regions of T volumes on sms SMs,
// and that of the adjoint for one region.
struct FwdRegion {
    int lo[3], hi[3];
};
int forward_depth(const FwdPlan& fp, const std::vector<FwdRegion>& regions, int T, int sms);
int adjoint_depth(const FwdPlan& fp, const FwdRegion& region, int T, int sms);
bool window_range(float ring_radius_dummy, const std::vector<float>& rcoord, int mag, int dim, int* lo, int* hi);
int fine_window_int(int mag, int dim, int* lo, int* hi);

void set_error(const std::string& msg);

// FP32 FMA throughput probe (probe.cu): best of three timed launches, TFLOP/s.
int probe_fp32_fma(int device, double* tflops);

// 3B Gibbs sampling of the spot states (gibbs.cu): one chain per launch,
// frames dealt out to co-resident CTAs (cooperative launch).
struct GibbsParams {
    const double* pix;        // [F][P] data
    const double* si;         // [K][P] each spot's intensity at every pixel
    const int* moff;          // [K + 1] mask offsets
    const int* midx;          // mask pixel indices
    int K, F, P;
    double A[9], pi[3];
    double variance;          // noise variance (when var_draw is null)
    const double* var_draw;   // [n_draws] variance of each draw, or null
    int sweeps;               // sweeps over all spots per draw
    int n_draws;
    unsigned long long seed;
    unsigned long long draw_base;  // counter offset of the first draw
    unsigned char* state;     // [K][F] current states, in/out
    double* cur;              // [F][P] current sample intensities, in/out
    double* em;               // [2][F][4] scratch: emission mantissas / exponents (two buffers)
    unsigned int* bar;        // grid barrier: count, generation (zeroed)
    unsigned long long* err;  // barrier failures (site << 56 | spot)
    unsigned char* out_state;  // [n_draws][K][F] or null
    double* out_int;           // [n_draws][F][P] or null
    int exclude_spot;          // >= 0: out_int without that spot where it is on (all pixels)
    double* out_err;           // [n_draws][F] sums of squared residuals, or null
    double* rec_lp;            // [K][F][2] log p(on), log p(off) of the first sweep, or null
    double* rec_filt;          // [K][F][3] filtering distribution of the first sweep, or null
};
size_t gibbs_smem_bytes(int F);
int gibbs_max_blocks(int F, int* out);
// chains_dev: nchains parameter sets in device memory, all with the same F.
int launch_gibbs(const GibbsParams* chains_dev, int nchains, int grid_per_chain, int F, void* stream);
int launch_spot_intensity(const int* pixels, int P, const double* spots, int K, double zf, double* out, void* stream);

// 3B sampled-background spot Hessian (hessian.cu). Sizes: tab [P][21],
// part [nc][S * F][22], gg [15], frame [S][F][20], out [S][20].
struct HessParams {
    const double* bg;      // [S][F][P] background samples (the spot taken off)
    const double* pix;     // [F][P] data
    const int* pixels;     // [P][3]
    const double* phi;     // [5] spot, device
    double zf, variance;
    double A[9], pi[3];
    int S, F, P, nc, bs;
    unsigned long long seed;
    double *tab, *part, *gg, *frame, *out;
};
int hessian_chunks(long long S, long long F, int P, int sm_count);
size_t hessian_ffbs_smem(int F);
int launch_spot_hessian(const HessParams& h, void* stream);
// The table, the per-(frame, sample) parts and sum g g^T only (part, gg);
// samples_hold_spot: the draws include the spot (e = data - sample).
int launch_hessian_parts(const HessParams& h, bool samples_hold_spot, void* stream);

// 3B spot gradient (threeb.cu): spot voxel table, emission sums per (sample,
// frame), forward algorithm per sample; res[s] = (gradient[5], log probability).
struct ThreeBPar {
    double phi[5], A[9], pi[3];  // the spot, the transitions (row-major), the start
};
int launch_threeb(const double* bg, const double* pix, const int* pixels, int S, int F, int P, const ThreeBPar& par,
                  double zf, double variance, double c0, double* val, double* der, double* em, double* res,
                  const float2* dfd, float2* vdf, void* stream);
// The samples' residuals (data minus background) as double-floats [S][F][P],
// for the gradient-only evaluations of launch_threeb (dfd; vdf is [P][6]).
int launch_threeb_residual(const double* bg, const double* pix, int S, int F, int P, float2* dfd, void* stream);

}  // namespace rfba

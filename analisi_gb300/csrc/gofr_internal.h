// Internal declarations shared by the host side (gofr_capi.cu) and the
// kernels (gofr_kernels.cu).  Not part of the C ABI.
#pragma once
#include <cmath>
#include <cstddef>
#include <cstdint>
#include <cuda_runtime.h>

namespace gofr {

// Bits of the device error word.
enum : unsigned {
    ERRW_WAIT_TIMEOUT = 1u,   // a bounded mbarrier wait ran out
    ERRW_WRAP_LOOP = 2u,      // the FP64 iterative minimum image exceeded its iteration cap
    ERRW_QUEUE = 4u,          // a work queue overflowed its capacity
    ERRW_BOUNDS = 8u,         // a bounds check failed (GOFR_CHECK in GOFR_DEBUG_BOUNDS builds;
                              // the warp-streamed kernel's neighbourhood tables always)
    ERRW_HIST_OVERFLOW = 16u  // an item could have overflowed a u32 shared bin (run discarded)
};

// Debug builds (-DGOFR_DEBUG_BOUNDS): GOFR_CHECK(cond, err) records a failed
// index check in the error word (no trap) and is false, so the access it
// guards is skipped; in normal builds it is `true` and costs nothing.
#ifdef GOFR_DEBUG_BOUNDS
#define GOFR_CHECK(cond, err) ((cond) ? true : (atomicOr((err), (unsigned)ERRW_BOUNDS), false))
#else
#define GOFR_CHECK(cond, err) true
#endif

// Stats slots (unsigned long long) on the device.
// ST_QUEUE: the two words of the warp-streamed kernel's chunk queue.
// ST_ERR: the error word, cleared and read back with the counters.
enum : int {
    ST_CANDIDATES = 0,
    ST_RECHECKS = 1,
    ST_EVALUATED = 2,
    ST_QUEUE = 3,
    ST_ERR = 4,
    ST_COUNT = 5
};

// Per-frame FP32 box parameters for the FP32 kernels (12 floats, 48 B).
//   L[3]    full edges 2*lh rounded to float
//   invL[3] 1/(2*lh) rounded to float
//   tilt[3] {xy, xz, yz} rounded to float
struct Box32 {
    float L[3];
    float invL[3];
    float tilt[3];
    float pad[3];
};

// Bin map of the kernels that bin a pair where they find it (the comment at
// bin_pair2 in gofr_device.cuh): q' = sqrt(d2) inv_dr + q_off, n = rint(q'); the
// pair is in bin n for certain when |q' - n| <= lim (t_lo and t_hi: the n, plus
// 1.5 2^23, that a pair of the window can come out at).
//   mode 0: rmin = 0 (n is never negative); 1: rmin > 0; 2: rmin < 0 (only
//   pairs beyond -rmin count: n < t_ok - 1.5 2^23 is never certain)
struct RadialMap {
    float inv_dr, q_off;
    float q_end;      // nbin: the unread cell
    float t_hi, t_lo, t_ok;
    float lim;        // negative: no pair is certain
    float lim_self;   // the same for an unwrapped difference of the FP32 frames
    float self_max;   // |component| up to which that difference needs no image
    int mode;
};

// One launch of an all-pairs kernel over (lag, i-tile, origin) items.
struct PairLaunch {
    const float *pos32;       // [T][3][NP] SoA {x-cx | y-cy | z-cz}, padding NaN
    const unsigned char *types8; // [NP] dense type ids (padding 0)
    const double *pos64;      // [T][N][3] internal FP64 positions (reference values)
    const double *box64;      // [T][9] internal boxes (tilts zero when orthorhombic)
    const Box32 *box32;       // [T]
    const float2 *win;        // [nbin] certified FP32 window {lo, hi} of each bin
    unsigned long long *counts;  // [leff][nch][nbin]
    unsigned *err;
    unsigned long long *stats;
    int N, NP, nbin, nch, ntypes;
    int a0, a1;               // first-atom range [a0, a1) (one reference thread partition)
    // gofr_allpairs.cu: every window and partition in one launch
    int nwin;                 // calculate(primos[w]) windows (primos null: one, primo)
    const long long *primos;
    long long win_stride;     // counts of a window
    int nparts;               // first atom a belongs to partition min(a / (N / nparts), nparts - 1)
    long long part_stride;    // counts of a partition
    int gs, ng;               // first atoms per unit, groups of them per partition
    int jc, nj;               // chunks of second atoms per unit, parts of the frame they make
    long long most;           // units of a CTA's chunk at most
    float far2;               // FP32 d2 from which a pair is certainly beyond the bins (infinite:
                              // not looked for)
    unsigned *queue;          // {next chunk, CTAs done}, zero before and after a launch
    int n_lags, every;        // lags t = l*every, l < n_lags
    int n_orig, skip;         // origins primo + k*skip, k < n_orig
    long long primo;
    int n_itiles;             // tiles of the first-atom range
    long long n_items;        // n_lags * n_itiles * n_orig
    float hi_f, lo_f;         // certain reject above hi_f / below lo_f
    float rmin_f, inv_dr_f;   // bin guess
    float wlim;               // wrap check: |frac| > wlim flags a recheck (triclinic; the
                              // global-memory histogram form)
    float wtol;               // orthorhombic: |component| > L / 2 - wtol flags a recheck
    double rmin, rmax, dr, rmin2, rmax2;  // reference binning constants
    int self0;                   // the reference's bin of distance zero (-1: not counted)
    RadialMap rm;
    int tric;
    int wchk;                 // batched kernel: per-pair wrap-decision check on
    int ghist;                // histogram too large for shared memory: atomics go
                              // straight to the u64 counts in global memory
    int dbg_stall;            // GOFR_DEBUG_BOUNDS builds only: the first tile's
                              // barrier expects bytes that no copy brings, so the
                              // bounded wait runs out (test of that path)
};

// One work descriptor of the batched kernel: units [u0, u1) of one trajectory
// (units as the single launch's: lag, origin, group of first atoms, part of the
// second atoms).
struct WorkDesc {
    int traj, pad;
    long long u0, u1;
};

constexpr int ALLPAIRS_GROUP = 64;   // first atoms of a warp's unit at most (gofr_allpairs.cu)
constexpr int ALLPAIRS_CHUNK = 128;  // second atoms a warp holds at a time: 4 per lane

// One launch of the cell-list pair kernel (gofr_cells.cu): items are
// (lag, block of cells, origin), pair.n_items = n_lags * nblocks * n_orig.
struct CellLaunch {
    PairLaunch pair;
    const int *start;              // [T][ncell+1] sorted-atom offset of each cell
    const float *spos;             // [T][3][NP] FP32 frames sorted by cell
    const unsigned *sidt;          // [T][NP] type << 24 | original atom id of each sorted slot
    int nc[3];                     // cells per axis
    int b[3];                      // cells per block per axis
    int nb[3];                     // blocks per axis
    int reach;                     // neighbour cells per side (cell edge >= rmax / reach)
    int r;                         // first atoms per thread (2, 3 or 4)
};

// One launch of the warp-streamed cell-list kernel (gofr_cellw.cu): items
// are (lag, origin), pair.n_items = n_lags * n_orig, each of nw[0] nw[1] nw[2]
// warp blocks of w[0] x w[1] x w[2] cells; a warp takes one block at a time.
//
// Cells are an axis-aligned grid of the box [lo, lo + L) (triclinic: the
// upper-triangular cell's axis-aligned fundamental domain).  A warp block's
// neighbourhood is given relative to the block, per lattice image
// (sx, sy, sz) of the cells reached: layers uz in [cz0 + nz_lo, cz0 + cnz +
// nz_hi] (image sz = floor(uz / ncz)); in a layer of image sz, rows uy in
// [cy0 + ny_lo[sz+1], cy0 + cny + ny_hi[sz+1]] (image sy); in a row of images
// (sy, sz), cells ux in [cx0 + nx_lo[k], cx0 + cnx + nx_hi[k]], k = (sz + 1) 5 +
// sy + 2 (image sx).  Orthorhombic boxes have lo = -reach, hi = reach - 1
// everywhere; a triclinic layer or row is shifted by the tilts, so its range
// starts a fraction of a cell off and may take one cell more.  shift[]
// holds the FP32 lattice vector of each image, index (sx + 2) + 5 (sy + 2) +
// 25 (sz + 1).
constexpr int CELLW_MAX_ROWS = 64;  // neighbourhood rows of a warp block (all its layers)
constexpr int CELLW_NSHIFT = 75;    // images sx, sy in -2..2, sz in -1..1
constexpr int CELLW_SHIFT0 = 37;    // index of the image (0, 0, 0)
// A row of a neighbourhood holds the cells that come within the reach of the
// warp block at the row's distance in y and z, so that the rows' ends follow
// the sphere around the block; cells are finer in x (Plan::fx) for it.
//
// Gap along an axis between the cell [r + o, r + o + 1) and the block [0, c),
// in cells, less a thousandth of a cell for the FP32 rounding and the cells'.
__host__ __device__ inline float cellw_gap(int r, float o, int c)
{
    const float below = -(float)(r + 1) - o, above = (float)r + o - (float)c;
    return fmaxf(fmaxf(below, above) - 1e-3f, 0.0f);
}
// Trims the cells [lo, hi] (from the block's first and last cell) of row ry,
// layer lz (from the block's first; images oy, ox cells off; the block is
// cny, cnz cells) to those within the radius; false when the row has none.
__host__ __device__ inline bool cellw_row(float rm2, float hy, float hz, float inv_hx, int ry,
                                          float oy, int cny, int lz, int cnz, float ox, int &lo,
                                          int &hi)
{
    const float gy = hy * cellw_gap(ry, oy, cny), gz = hz * cellw_gap(lz, 0.0f, cnz);
    const float e2 = rm2 - gy * gy - gz * gz;
    if (!(e2 > 0.0f)) return false;
    const float rho = sqrtf(e2) * inv_hx * 1.00001f + 1e-3f;
    const int a = (int)floorf(-rho - ox), b = (int)floorf(rho - ox);
    if (a > lo) lo = a;
    if (b < hi) hi = b;
    return true;
}

struct CellwLaunch {
    PairLaunch pair;
    const int *start;              // [T][ncell+1] sorted-record offset of each cell
    const float4 *wpos;            // [T][NP] {x, y, z, type << 24 | atom id} sorted by cell
    int nc[3];                     // cells per axis (fx times the planner's in x)
    int w[3];                      // cells per warp block per axis (the same)
    int nw[3];                     // warp blocks per axis
    int reach;                     // neighbour cells per side
    int r;                         // records per lane (4; kept in plans and tuner keys)
    int pg, npg;                   // partitions per histogram, groups of them (pair.nparts)
    long long most;                // warp blocks of a CTA's chunk at most
    unsigned *queue;               // {next chunk, CTAs done}, zero before and after a launch
    int cta_warps;                 // warps per CTA: 8 or 16 (one CTA of 32 where 16 leave half an SM)
    int hcopy;                     // copies of the shared histogram (privatisation depth: 1, 2)
    int nz_lo, nz_hi;              // neighbourhood layers (see above)
    int ny_lo[3], ny_hi[3];        // rows, per layer image sz + 1
    int nx_lo[15], nx_hi[15];      // cells, per row images (sz + 1) 5 + sy + 2
    int ny_span;                   // max over sz of ny_hi - ny_lo + 1
    float oy[3], ox[15];           // image offsets in cells: rows of layer image sz + 1, cells
    float hy, hz, inv_hx, rm2;     // cell edges, 1 / edge, radius^2 (with room for rounding)
    float4 shift[CELLW_NSHIFT];    // FP32 lattice vector {x, y, z, 0} of each image
};
int cellw_smem_bytes(int nch, int nbin, int ntypes, int cta_warps = 8, int hcopy = 1);
int cellw_chunk_records();  // neighbour records per chunk (4 per lane)
int cellw_batch_atoms();    // first atoms per batch (each batch streams the neighbourhood)
// box_internal {xlo, ylo, zlo, lx/2, ly/2, lz/2, xy, xz, yz}; tric: the
// coordinates are reduced into the axis-aligned cell by the lattice (z, then
// y, then x), else per axis.
int launch_cell_scatter_w(const double *pos64, const unsigned char *types8, size_t T, size_t N,
                          const double *box_internal, const double *centre, const int *nc,
                          bool tric, const int *cell_of, const int *rank_of, const int *start,
                          float4 *wpos, cudaStream_t s);
int launch_cellw_pairs(const CellwLaunch &C, int num_sms, cudaStream_t s);

// FP64 normalisation of window counts on the device (gofr_norm.cu).
// s(k), the FP64 sum of k additions of incr from 0 (lib/src/gofrt.cpp:118), as
// the runs of equal steps it consists of: within one binade the rounded step
// is the same for every addition (but for the first, where the step is half
// an ulp off an odd sum), so s(k) = s0 + (k - k0) delta exactly from each run's
// first addition k0 on.  At most a tie, a run and a step over the end per
// binade, and the sum stands still 54 binades above incr.
constexpr int FOLD_RUNS = 176;
struct FoldTable {
    unsigned long long k0[FOLD_RUNS];
    double s0[FOLD_RUNS], delta[FOLD_RUNS];
    unsigned char first[64];  // the run that holds 2^b
    int n;
};
FoldTable fold_table(double incr);
__host__ __device__ inline double fold_sum(const FoldTable &t, unsigned long long k)
{
    if (k == 0) return 0.0;
#ifdef __CUDA_ARCH__
    int i = t.first[63 - __clzll((long long)k)];
#else
    int i = t.first[63 - __builtin_clzll(k)];
#endif
    while (i + 1 < t.n && t.k0[i + 1] <= k) ++i;
    const double j = (double)(k - t.k0[i]);
#ifdef __CUDA_ARCH__
    return __dadd_rn(t.s0[i], __dmul_rn(j, t.delta[i]));  // both exact
#else
    return t.s0[i] + j * t.delta[i];
#endif
}

struct NormLaunch {
    const unsigned long long *counts;  // [nwin][nparts][n] exact counts
    double *out;                       // [nwin][n]
    const double *chfac;               // [nch] pair-density factors (mode 2)
    size_t n;                          // leff * nch * nbin
    int nwin, nparts, nbin, nch;
    int mode;                          // 0 buffer, 1 / shell volume, 2 / shell volume / density
    double r0, dr;                     // bin b spans [b dr + r0, (b + 1) dr + r0)
    double c43pi;                      // fl(fl(4 pi) / 3)
    FoldTable fold;                    // of 1 / int(ntimesteps / skip)
};
int launch_counts_to_gofr(const NormLaunch &L, int num_sms, cudaStream_t s);

int cell_smem_bytes(int nch, int nbin, int ntypes);
int cell_block_atoms(int r);
int cell_max_ranges();
// Mean square displacement (gofr_msd.cu)
struct MsdLaunch {
    const double *pos64;    // [T][N][3]
    const double *cm;       // [T][ntypes][3] centres of mass (or null)
    const int *perm;        // [N] atom ids sorted by type (stable)
    const int *tbegin;      // [ntypes + 1] start of each type in perm
    double *partial;        // [leff][n_orig][f_cm * ntypes] sums over atoms
    int N, ntypes, leff, n_orig, skip;
    long long primo;
    int cm_msd, cm_self;
};
int launch_msd(const MsdLaunch &M, double *out_device, int num_sms, cudaStream_t s);
// The same in exact integer sums (k_msd_fixed).
struct MsdFixed {
    int atoms, origins, tiles;  // atoms and origins of a chunk, tiles of origins
    int frames;                 // frames of a chunk (its row length in shared memory)
    int lags, phases, passes;   // lags and origin phases of a CTA's threads, CTAs per chunk range
    int apart;                  // no frame is in the lags of two origins: phases of the atoms
    long long chunks, per;      // chunks, chunks per CTA
    int grid;
    const unsigned *ext;        // [256] largest extent per type, FP32 bits (launch_extent)
    const double *cm_ext;       // [ntypes] the same of the centres (cm_self)
    double pad;                 // what the FP32 frames' rounding can add to an extent
    long long *partial;         // [grid + ntypes][leff][6]
    long long *lost;            // [grid + ntypes] values that are not held exactly
    // results (lag ntypes + type) in which that could show, their number and terms
    int *entries;
    unsigned long long *n_entries, *n_terms;
};
// FP64 sums for n results (lag ntypes + type) alone; M.partial: [n][n_orig].
int launch_msd_entries(const MsdLaunch &M, const int *entries, int n, double *out_device,
                       int num_sms, cudaStream_t s);
// Largest extent per type over `len` frames from `first` on, or within each of
// `groups` runs of them; raises ext[256], FP32 bits.
int launch_extent(const float *pos32, const unsigned char *types8, size_t N, long long first,
                  int groups, int len, int stride, unsigned *ext, cudaStream_t s);
bool msd_fixed_plan(const MsdLaunch &M, const int *h_tbegin, int num_sms, MsdFixed &X);
size_t msd_fixed_partial(const MsdLaunch &M, const MsdFixed &X);  // 8-byte words of both
int launch_msd_fixed(const MsdLaunch &M, const MsdFixed &X, double *out_device, cudaStream_t s);

// Neighbour lists (gofr_neigh.cu)
constexpr int NEIGH_MAXT = 32;
struct NeighLaunch {
    const double *pos64;                  // [T][N][3]
    const double *box64;                  // [T][9] internal boxes
    const int *types;                     // [N] dense type ids
    const unsigned long long *nneigh;     // [ntypes] list capacities
    const unsigned long long *loff, *roff;  // [ntypes] offsets in list / rpos
    const double *cut2;                   // [ntypes] cutoffs^2
    unsigned long long *list;             // the reference's list array
    double *rpos;                         // the reference's rpos array
    int *full;                            // [N][ntypes] neighbour that filled a list (N: not full)
    unsigned *flags;                      // bit 0: some list is full; bit 1: a cell
                                          // neighbourhood held too many candidates
    unsigned long long *first_err;        // min i*N + j over overflowing pairs
    unsigned *err;                        // error word (minimum-image iteration cap)
    int N, ntypes;
    long long timestep;
    int tric;
    // FP32 prefilter (the all-pairs kernel's certified arithmetic): a pair
    // with d2_f32 > hi_f has reference d2 > the largest cutoff
    int prefilter;
    const float *pos32;                   // [T][3][NP]
    const Box32 *box32;                   // [T]
    long long NP;
    float hi_f;
    // cell-list form (orthorhombic boxes, prefilter on): the frame's cells of
    // edge >= the largest cutoff, at least 3 per axis
    int cells;
    int nc[3];
    const int *cstart;                    // [ncell + 1] first sorted slot of each cell
    const unsigned *csidt;                // [N] type << 24 | atom id in cell order
};
int launch_neigh_build(const NeighLaunch &L, int num_sms, cudaStream_t s);
int launch_neigh_check(const NeighLaunch &L, int num_sms, cudaStream_t s);
int launch_neigh_sort(const NeighLaunch &L, int num_sms, cudaStream_t s);

// Cell assignment and per-frame cell starts (and, with spos/sidt non-null,
// the block kernel's SoA sorted frames); cell_of and rank_of are left for
// launch_cell_scatter_w.  tric: cells of the coordinates reduced into the
// axis-aligned cell by the lattice (spos/sidt must then be null).
int launch_cell_build(const double *pos64, const unsigned char *types8, size_t T, size_t N,
                      const double *box_internal, const double *centre, const int *nc, bool tric,
                      int *cell_of, int *rank_of, int *count, int *start, float *spos,
                      unsigned *sidt, cudaStream_t s);
// One trajectory's cell-list items in one launch.
int launch_cell_pairs(const CellLaunch &C, int num_sms, cudaStream_t s);
// One launch over the items of nmem trajectories: Cs[m] (device) holds
// trajectory m's parameters, item_end[m] (device) the end of its items in the
// global item order; shared memory is sized for the largest histogram.
// prepare_* sets the kernel attributes and the grid (outside graph capture).
int prepare_cell_pairs_multi(int r, int max_nbin, int max_nch, int max_ntypes, int num_sms,
                             long long total, int *grid);
int launch_cell_pairs_multi(const CellLaunch *d_cells, const long long *d_end, int nmem,
                            int r, int max_nbin, int max_nch, int max_ntypes, int grid,
                            cudaStream_t s);

// Launch configuration helpers implemented in gofr_kernels.cu.
int launch_minmax(const double *pos64, size_t n3, double *d_out6, unsigned *d_nonfinite,
                  cudaStream_t s);
// Padded per-frame stride of the FP32 SoA frames.
inline size_t padded_natoms(size_t N) { return (N + 15) / 16 * 16; }
int launch_convert(const double *pos64, const int *types, size_t T, size_t N, double cx,
                   double cy, double cz, float *pos32, unsigned char *types8, cudaStream_t s);
// kind: 0 = FP32+recheck, 1 = FP64.  wrapcheck only for kind 0.
int launch_pairs(const PairLaunch &P, int kind, bool wrapcheck, int num_sms, cudaStream_t s,
                 size_t *smem_bytes_out);
int pairs_smem_bytes(int kind, int nch, int nbin, int ntypes, bool ghist = false);
int pairs_tile_atoms(int kind);
size_t allpairs_smem_bytes(int nch, int nbin, int ntypes);
int launch_allpairs(const PairLaunch &P, bool wrapcheck, int num_sms, cudaStream_t s);
// cells: nch (nbin + 1) + 1 of the member with the most; mode: 0 when every
// member's bin map is of mode 0, else 2.
int prepare_batch(int max_cells, int max_ntypes, bool tric, int mode, int num_sms, int n_work,
                  int *grid);
int launch_batch_grid(const PairLaunch *d_trajs, const WorkDesc *d_work, int n_work,
                      unsigned *d_head, int max_cells, int max_ntypes, bool tric, int mode,
                      unsigned *d_err, unsigned long long *d_stats, int grid, cudaStream_t s);
int launch_zero_u64(unsigned long long *p, size_t n, cudaStream_t s);

}  // namespace gofr

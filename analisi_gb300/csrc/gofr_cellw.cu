// Warp-streamed cell-list form of the FP32 + FP64-recheck pair kernel.
//
// The reference evaluates all N^2 ordered pairs of every (lag, origin)
// (lib/src/gofrt.cpp:101-102).  As in the block cell-list kernel
// (gofr_cells.cu), the atoms of every frame are binned into cells of edge
// >= rmax / reach and sorted by cell, so a pair the reference counts lies in
// cells at most `reach` apart on every axis; here the unit of neighbourhood
// is much smaller: each WARP owns a small block of cells and streams only
// that block's own neighbourhood, so the pairs evaluated per first atom
// shrink from the neighbourhood of a CTA-sized block to the neighbourhood of
// a warp-sized one.
//
// Lanes hold neighbours, not first atoms: the records of the neighbourhood,
// rows back to back, are taken 128 at a time, four per lane in registers, and
// the warp walks the block's first atoms one at a time, each broadcast from
// shared memory, so no lane idles for want of a first atom whatever the
// block's atom count (only the last chunk of a neighbourhood is partly empty).
//
// Layout per frame (built once per upload and grid): records
// {x, y, z, type << 24 | atom id} (float4, the coordinates wrapped into the
// box in FP64 and rounded to FP32 about the box centre, exactly as the block
// kernel's), sorted by cell, x fastest; cell start offsets.  A row of cells
// of a neighbourhood is one or two contiguous runs of 16-byte records; a warp
// lists the runs that hold records with their prefix sums, and a lane finds
// the run of its record by counting run starts among the 32 records of its
// group (one OR-reduction of start bits), then loads it from L2: coalesced
// 512-byte loads straight into registers.  (Staging through shared memory by
// bulk copies cost the copies' issue, an mbarrier wait and a pass over the
// records per chunk, and needed the buffers for a candidate queue that is
// gone.)  Cells reached across the box boundary are the periodic image of the
// cell: each record is moved to its run's image (x += fl32 of the lattice
// vector, one FP32 rounding per axis; orthorhombic: s fl32(L), the block
// kernel's arithmetic).
//
// Triclinic boxes (upper-triangular cell vectors a, b, c) use the same
// kernel.  The reference's minimum image (z, then y, then x) leaves every
// component within half the box edge, so its image of a pair is the one
// lattice translate inside the axis-aligned box [-L/2, L/2]^3, and a pair it
// counts (distance < rmax < L/2) has exactly one image within rmax.  Cells
// are therefore an axis-aligned grid of the cell's axis-aligned fundamental
// domain, atoms reduced into it by the lattice; a layer reached across a z
// face is the image +-c, shifted in y and x by the tilts, and a row reached
// across a y face the image +-b, shifted in x: each layer's rows and each
// row's cells start a fraction of a cell off, which host tables give (one
// more cell where the shift is not whole), together with the FP32 lattice
// vector of each image.
//
// A row keeps only the cells within reach of the block at the row's distance
// in y and z (cellw_row), and cells are up to eight to the reach in x, so the
// rows' ends follow the sphere around the block: at reach 2, 3.43 times the
// sphere's volume instead of 3.73 for whole cells (66.3 to 60.9 ms at 16k
// atoms, 20.3 to 17.8 at 32k triclinic, 8.4 to 7.8 at 131k).  Finer rows in y
// and z would leave 3.13 but are four times as many to list; leaving out
// (first atom, chunk) pairs by the chunk's bounding box would save another 4 %
// of the pairs, less than the boxes cost.
//
// Every evaluated pair goes straight into the CTA's shared histogram
// (bin_pair2, gofr_device.cuh), and the pairs near a bin edge (the radial
// margin of gofr_capi.cu; 0.13 % of them at 16k atoms) are noted in a bit per
// first atom and record, then taken out of their cell and recomputed in FP64,
// 32 at a time.
//
// Counts per reference thread partition of the first atoms take a histogram
// of as many partitions as fit shared memory, and the first atoms of a block
// in the order of (partition, type); the blocks are streamed once per such
// group of partitions.
//
// Work is a list of (lag, origin, warp block) units, dealt to the CTAs in
// chunks of decreasing size from one counter; the warps of a CTA take the
// chunk's units one by one and never wait for one another inside a chunk.
// The histogram is added to the counts when the lag changes, and before 2^32
// pairs were evaluated since (a u32 bin could overflow): a warp whose unit finds
// no room for its pairs keeps it for after the flush.  (Items of one
// (lag, origin) dealt round-robin, a barrier and a flush after each, left 10 % of
// the 16k-atom job idle in the last round and 18 % of the 131k-atom one.)
//
// Bound by instruction issue: 71 instructions per 128 pairs (46 of them the
// pairs' own), 77 % of the issue slots used, the shared-memory pipe 57 %
// busy, the FP32 pipe 59 %, no DRAM traffic to speak of.  16384 atoms, 25
// origins x 100 lags (16 % of N^2 evaluated, 28 % of those within rmax): 59.5
// ms, where the form that queued its candidates and binned the queue took
// 178.9; 131072 atoms, 5 x 10: 7.7 ms against 21.7; 32768 atoms, triclinic,
// 10 x 20: 17.5 ms against 59.8.  64 registers (spilling 290 to 298 bytes stored, 472
// to 508 loaded, outside the loop over first atoms), 32 warps per SM (two CTAs of
// 16, one of 32 for a large histogram): with 128 registers and 16 warps 74.9 ms.
#include <cstdint>
#include <cuda_runtime.h>

#include "gofr_device.cuh"
#include "gofr_internal.h"

namespace gofr {
namespace cellw {

constexpr int CH = 128;        // neighbour records per chunk: 4 per lane
constexpr int FA = 64;         // first atoms per batch
constexpr int MAXROWS = CELLW_MAX_ROWS;  // neighbourhood rows of a warp block
constexpr int MAXSEG = 2 * MAXROWS;      // sorted ranges of them (two when a row wraps the box)
constexpr int QW = 64;         // FP64 recheck queue of a warp
static_assert(CH == 4 * 32, "four records per lane");
static_assert(FA == 64, "two groups of first atoms");
static_assert(QW >= 64, "a round adds at most 32 entries to a queue drained at 32");

constexpr unsigned SLOT_MASK = 0x1ffffffu;  // a sorted slot below its image's index

// floor(a / n) for n > 0
__device__ __forceinline__ int floordiv(int a, int n) { return a >= 0 ? a / n : -((n - 1 - a) / n); }

// Shared memory of one warp.
struct WarpArea {
    ulonglong2 fa[FA][2];        // first atoms {x x | y y}, {z z | w, run end << 16 | class}:
                                 // coordinates duplicated for f32x2, w = type << 24 | id, the class
                                 // partition ntypes + type (the partition's place in the histogram)
                                 // and the end of the run of first atoms of the class
    uint2 near[QW];              // pairs near a bin edge: {first atom, image << 25 | sorted slot}
    uint2 q[QW];                 // FP64 recheck queue: w of both atoms
    int2 src[MAXSEG];            // {sorted slot of the segment's first record - its flat index, image}
    int pre[MAXSEG + 33];        // flat index of each segment's first record (INT_MAX past the last)
    int held;                    // unit left for after the next flush (-1: none)
};

// NWARP warps per CTA, HCOPY copies of the shared histogram (warp w adds to
// copy w HCOPY / NWARP: the privatisation depth, fewer warps contending for
// each bin), MODE the bin map's (RadialMap), PARTS: counts per partition (apart:
// the first atoms' partitions cost the form without them 2 % in registers).
template <int NWARP, int HCOPY, int MODE, bool PARTS>
__global__ void __launch_bounds__(NWARP * 32, 32 / NWARP) k_pairs_cellw(const CellwLaunch C)
{
    constexpr int NT = NWARP * 32;
    extern __shared__ __align__(128) unsigned char smem[];
    const PairLaunch &P = C.pair;
    const int nbin = P.nbin, nrow = nbin + 1;  // histogram row: nbin bins and an unread cell
    const int nch = PARTS ? P.nch * C.pg : P.nch;  // rows: C.pg partitions' channels
    const int hist_cap = nch * nrow + 1;        // the first row has its cell -1, too
    WarpArea *const areas = reinterpret_cast<WarpArea *>(smem);
    unsigned *const hist = reinterpret_cast<unsigned *>(areas + NWARP);
    unsigned short *const chtab = reinterpret_cast<unsigned short *>(hist + HCOPY * hist_cap);
    __shared__ int s_next, s_full;
    __shared__ long long s_u0, s_u1;
    __shared__ unsigned long long s_pairs;  // pairs evaluated since the last flush
    __shared__ float4 s_shift[CELLW_NSHIFT];
    __shared__ int2 s_ny[3], s_nx[15];
    __shared__ float s_oy[3], s_ox[15];

    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const unsigned lt = (1u << lane) - 1u;  // the lanes below this one
    WarpArea &A = areas[warp];
    const int per_part = PARTS ? P.N / P.nparts : 1;  // first atom a: partition min(a / per_part, nparts - 1)
    unsigned *const whist = hist + (warp * HCOPY / NWARP) * hist_cap + 1;  // this warp's row 0
    // row address of channel ch as bin_pair2 takes it: row0 + ch * rowb
    const unsigned row0 = smem_u32(whist) - 4u * RADIAL_MAGIC_BITS, rowb = 4u * (unsigned)nrow;
    const int half_ch = P.nch / 2;
    const int ncx = C.nc[0], ncy = C.nc[1], ncz = C.nc[2];
    const int ncell = ncx * ncy * ncz;
    const int nwx = C.nw[0], nwy = C.nw[1], nwz = C.nw[2];
    const int nwb = nwx * nwy * nwz;
    const long long NP = P.NP;
    const float qnan = __int_as_float(0x7fc00000);

    for (int i = tid; i < HCOPY * hist_cap; i += NT) hist[i] = 0u;
    for (int i = tid; i < P.ntypes * P.ntypes; i += NT) chtab[i] = type_channel(i, P.ntypes);
    for (int i = tid; i < CELLW_NSHIFT; i += NT) s_shift[i] = C.shift[i];
    if (tid < 3) {
        s_ny[tid] = make_int2(C.ny_lo[tid], C.ny_hi[tid]);
        s_oy[tid] = C.oy[tid];
    }
    if (tid < 15) {
        s_nx[tid] = make_int2(C.nx_lo[tid], C.nx_hi[tid]);
        s_ox[tid] = C.ox[tid];
    }
    if (tid == 0) s_pairs = 0ull;
    if (lane == 0) A.held = -1;

    int nn = 0, qn = 0;  // entries of the warp's two queues (the same in every lane)
    unsigned long long n_cand = 0, n_rech = 0, n_eval = 0;  // n_cand: counts flushed
    bool lost = false;                                      // a u32 bin could have overflowed

    // Adds the CTA's histogram copies to the counts of plane (partition group,
    // lag) and clears them (all threads; every warp is done with its pairs).  A
    // u32 bin holds its hits exactly only while fewer than 2^32 pairs were
    // evaluated: only a single unit can have more.
    auto flush = [&](int plane) {
        if (s_pairs > 0xffffffffull) lost = true;
        const int grp = PARTS ? plane / P.n_lags : 0, lag_idx = plane - grp * P.n_lags;
        unsigned long long *const out = P.counts + (PARTS ? grp * C.pg * P.part_stride : 0) +
                                        (long long)lag_idx * P.every * P.nch * nbin;
        for (int i = tid; i < nch * nbin; i += NT) {
            const int row = i / nbin, b = i - row * nbin, at = row * nrow + b + 1;
            unsigned v = 0;  // modulo 2^32: a copy may hold the self pairs another one counted
#pragma unroll
            for (int c = 0; c < HCOPY; ++c) v += hist[c * hist_cap + at];
#pragma unroll
            for (int c = 0; c < HCOPY; ++c) hist[c * hist_cap + at] = 0u;
            n_cand += v;
            if (v && !lost) {
                const int part = PARTS ? row / P.nch : 0;
                atomicAdd(out + part * P.part_stride + (row - part * P.nch) * nbin + b,
                          (unsigned long long)v);
            }
        }
        __syncthreads();
        if (tid == 0) s_pairs = 0ull;
        __syncthreads();
    };

    // units: (partition group, lag, origin, warp block), the warp block fastest
    const long long per_plane = (long long)P.n_orig * nwb, U = per_plane * P.n_lags * (PARTS ? C.npg : 1);
    int cur = -1;  // plane (partition group, lag) of the histogram
    while (!lost) {
        __syncthreads();  // every warp has read the last chunk's range
        if (tid == 0) {
            const long long c = (long long)atomicAdd(C.queue, 1u);
            long long u0 = 0, u1 = 0;
            chunk_range(c, gridDim.x, U, C.most, NWARP, u0, u1);
            s_u0 = u0;
            s_u1 = u1;
            s_next = 0;
            s_full = s_pairs > 0x7fffffffull;
        }
        __syncthreads();
        const long long c0 = s_u0, c1 = s_u1;
        if (c0 >= c1) break;
        bool again = false;  // a warp holds a unit of this segment back: a flush, then the rest
        for (long long g0 = c0; g0 < c1 && !lost;) {
        const int plane = (int)(g0 / per_plane);
        const int lag_idx = PARTS ? plane % P.n_lags : plane;
        const int part0 = PARTS ? plane / P.n_lags * C.pg : 0;
        const long long g1 = min(c1, (plane + 1) * per_plane);
        if (g0 != c0 && !again) {
            __syncthreads();  // the warps are done with the chunk's last plane
            if (tid == 0) {
                s_next = 0;
                s_full = s_pairs > 0x7fffffffull;
            }
            __syncthreads();
        }
        if (cur >= 0 && (plane != cur || s_full || again)) flush(cur);
        cur = plane;
        int k = -1;  // origin of the warp's queues
        long long fo = 0, fl = 0;
        const int *st_o = nullptr, *st_l = nullptr;
        const float4 *rec_o = nullptr, *rec_l = nullptr;
        const long long seg_orig = (g0 - plane * per_plane) / nwb;  // the segment's first origin
        const long long seg_off = (g0 - plane * per_plane) - seg_orig * nwb;

        // First row of the histogram of atom ia's partition (negative, or C.pg
        // partitions on: not one of the histogram's).
        auto part_row = [&](int ia) {
            return PARTS ? (min(ia / per_part, P.nparts - 1) - part0) * P.nch : 0;
        };
        // Recomputes queued pairs [0, n) in exact FP64 (reference arithmetic),
        // one per lane; into the channel of distinct atoms, like every pair.
        auto recheck = [&](int n) {
            __syncwarp();
            if (lane < n) {
                const uint2 e = A.q[lane];
                const double *xi = P.pos64 + (fo * P.N + (int)(e.x & 0xffffffu)) * 3;
                const double *xj = P.pos64 + (fl * P.N + (int)(e.y & 0xffffffu)) * 3;
                const double *box = P.box64 + fo * 9;
                const double d2 = P.tric ? ref_d2<true>(xi[0], xi[1], xi[2], xj[0], xj[1], xj[2],
                                                        box, P.err)
                                         : ref_d2<false>(xi[0], xi[1], xi[2], xj[0], xj[1], xj[2],
                                                         box, P.err);
                const int b = ref_bin(d2, P.rmin, P.dr, P.rmin2, P.rmax2, nbin);
                const int ch = part_row((int)(e.x & 0xffffffu)) +
                               chtab[(int)(e.x >> 24) * P.ntypes + (int)(e.y >> 24)];
                if (b >= 0 && GOFR_CHECK(ch >= 0 && ch < nch && b < nbin, P.err))
                    atomicAdd(whist + ch * nrow + b, 1u);
                ++n_rech;
            }
            __syncwarp();
        };
        // Takes entries [0, n) of `near`, one per lane: the pair's bin again with
        // the pair loop's operations (the same value), out of the cell it was
        // added to, and into the recheck queue where it can be within the
        // window.
        auto resolve = [&](int n) {
            __syncwarp();
            bool need = false;
            unsigned wi = 0u, wj = 0u;
            if (lane < n) {
                const uint2 e = A.near[lane];
                const ulonglong2 u0 = A.fa[e.x][0], u1 = A.fa[e.x][1];
                const float4 v = rec_l[e.y & SLOT_MASK];
                const float4 sh = s_shift[e.y >> 25];
                wi = (unsigned)u1.y;
                wj = __float_as_uint(v.w);
                const float dx = __fsub_rn(__uint_as_float((unsigned)u0.x), __fadd_rn(v.x, sh.x)),
                            dy = __fsub_rn(__uint_as_float((unsigned)u0.y), __fadd_rn(v.y, sh.y)),
                            dz = __fsub_rn(__uint_as_float((unsigned)u1.x), __fadd_rn(v.z, sh.z));
                const float q = radial_q(
                    __fmaf_rn(dz, dz, __fmaf_rn(dy, dy, __fmaf_rn(dx, dx, RADIAL_TINY))), P.rm);
                const float t = __fadd_rn(q, RADIAL_MAGIC);
                need = t <= P.rm.t_hi && t >= P.rm.t_lo;
                const int b = (int)(__float_as_uint(t) - RADIAL_MAGIC_BITS);
                if (b >= 0 && b < nbin)
                    atomicSub(whist + (part_row((int)(wi & 0xffffffu)) +
                                       chtab[(int)(wi >> 24) * P.ntypes + (int)(wj >> 24)]) * nrow + b,
                              1u);
            }
            const unsigned m = __ballot_sync(0xffffffffu, need);
            if (need) A.q[qn + __popc(m & lt)] = make_uint2(wi, wj);
            qn += __popc(m);
            if (qn >= 32) {
                recheck(32);
                qn -= 32;
                if (lane < qn) A.q[lane] = A.q[32 + lane];
                __syncwarp();
            }
        };

        for (;;) {
            int nx = 0;
            if (lane == 0) {
                nx = A.held;
                if (nx < 0) nx = atomicAdd(&s_next, 1);
                A.held = -1;
            }
            nx = __shfl_sync(0xffffffffu, nx, 0);
            if (g0 + nx >= g1) break;
            const long long uo = seg_off + nx;
            const int kk = (int)(seg_orig + uo / nwb), wb = (int)(uo % nwb);
            if (kk != k) {
                recheck(qn);  // the queue names the last origin's frames
                qn = 0;
                k = kk;
                fo = P.primo + (long long)k * P.skip;
                fl = fo + (long long)lag_idx * P.every;
                st_o = C.start + fo * (long long)(ncell + 1);
                st_l = C.start + fl * (long long)(ncell + 1);
                rec_o = C.wpos + fo * NP;
                rec_l = C.wpos + fl * NP;
            }
            const int wz = wb / (nwx * nwy), wy = (wb / nwx) % nwy, wx = wb % nwx;
            const int cx0 = wx * C.w[0], cy0 = wy * C.w[1], cz0 = wz * C.w[2];
            const int cnx = min(C.w[0], ncx - cx0), cny = min(C.w[1], ncy - cy0),
                      cnz = min(C.w[2], ncz - cz0);
            // rows of the warp block (w_y w_z <= 16 of them): lane r holds row
            // r's range and the inclusive prefix of the row lengths
            const int nir = cny * cnz;
            int ib = 0, ilen = 0;
            if (lane < nir) {
                const int ry = lane % cny, rz = lane / cny;
                const int base = ((cz0 + rz) * ncy + (cy0 + ry)) * ncx + cx0;
                ib = st_o[base];
                ilen = st_o[base + cnx] - ib;
            }
            int ipre = ilen;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int v = __shfl_up_sync(0xffffffffu, ipre, o);
                if (lane >= o) ipre += v;
            }
            const int n_i = __shfl_sync(0xffffffffu, ipre, 31);
            if (n_i == 0) continue;
            // the neighbourhood: layers uz (image sz), in each the rows uy
            // (image sy), each row the cells ux in one or two sorted ranges
            // (two when the row wraps the box: images sx and sx + 1); the
            // ranges that hold records, back to back, are the flat list the
            // chunks take their records from
            const int jny = cny + C.ny_span;
            const int nrows = (cnz + C.nz_hi - C.nz_lo + 1) * jny;
            int nseg = 0, n_j = 0;
            for (int r0 = 0; r0 < nrows; r0 += 32) {
                const int rr = r0 + lane;
                const int lz = rr / jny, ky = rr - lz * jny;
                const int uz = cz0 + C.nz_lo + lz;
                const int sz = floordiv(uz, ncz), cz = uz - sz * ncz;
                int beg0 = 0, len0 = 0, beg1 = 0, len1 = 0, code = 0;
                if (rr < nrows) {
                    // the host keeps every image reached inside the tables and every
                    // row within one wrap of the box; a row outside them is reported
                    // and left empty (no access outside the tables or the frame)
                    bool ok = sz >= -1 && sz <= 1;
                    const int2 yr = ok ? s_ny[sz + 1] : make_int2(0, -1 - cny);
                    if (ky <= cny + yr.y - yr.x) {
                        const int uy = cy0 + yr.x + ky;
                        const int sy = floordiv(uy, ncy), cy = uy - sy * ncy;
                        ok = sy >= -2 && sy <= 2;
                        int2 xr = make_int2(0, -1 - cnx);
                        if (ok) {
                            const int im = (sz + 1) * 5 + sy + 2;
                            xr = s_nx[im];
                            if (!cellw_row(C.rm2, C.hy, C.hz, C.inv_hx, yr.x + ky, s_oy[sz + 1],
                                           cny, C.nz_lo + lz, cnz, s_ox[im], xr.x, xr.y) ||
                                cnx + xr.y < xr.x)
                                xr.y = xr.x - 1 - cnx;  // no cell
                        }
                        const int ux = cx0 + xr.x, len = cnx + xr.y - xr.x + 1;
                        const int sx = floordiv(ux, ncx), a = ux - sx * ncx, b = a + len;
                        ok = ok && sx >= -2 && len >= 0 && len <= ncx &&
                             (b <= ncx ? sx <= 2 : sx <= 1);
                        if (ok) {
                            const int base = (cz * ncy + cy) * ncx;
                            code = (sx + 2) + 5 * (sy + 2) + 25 * (sz + 1);
                            beg0 = st_l[base + a];
                            len0 = st_l[base + min(b, ncx)] - beg0;
                            if (b > ncx) {
                                beg1 = st_l[base];
                                len1 = st_l[base + b - ncx] - beg1;
                            }
                        }
                    }
                    if (!ok) atomicOr(P.err, ERRW_BOUNDS);
                }
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const int beg = h ? beg1 : beg0, len = h ? len1 : len0;
                    const unsigned m = __ballot_sync(0xffffffffu, len > 0);
                    if (!m) continue;
                    int incl = len;
#pragma unroll
                    for (int o = 1; o < 32; o <<= 1) {
                        const int v = __shfl_up_sync(0xffffffffu, incl, o);
                        if (lane >= o) incl += v;
                    }
                    const int at = nseg + __popc(m & lt), f = n_j + incl - len;
                    if (len > 0 && GOFR_CHECK(at < MAXSEG, P.err)) {
                        A.pre[at] = f;
                        A.src[at] = make_int2(beg - f, code + h);
                    }
                    nseg += __popc(m);
                    n_j += __shfl_sync(0xffffffffu, incl, 31);
                }
            }
            A.pre[nseg + lane] = 0x7fffffff;
            // room for the unit's pairs in the u32 bins: a unit that finds none waits for
            // the next flush (the first unit after one always has it)
            bool room = true;
            if (lane == 0) {
                A.pre[nseg + 32] = 0x7fffffff;
                const unsigned long long pe = (unsigned long long)n_i * (unsigned long long)n_j,
                                         was = atomicAdd(&s_pairs, pe);
                room = was == 0ull || was + pe <= 0xffffffffull;
                if (!room) {
                    atomicAdd(&s_pairs, 0ull - pe);
                    A.held = nx;
                }
            }
            if (!__shfl_sync(0xffffffffu, (int)room, 0)) break;

            for (int ibase = 0; ibase < n_i; ibase += FA) {
                // first atoms ibase .. ibase + n - 1 of the block, those of the
                // histogram's partitions, each group of 32 in the order of their
                // classes (the row addresses of a lane's records change only with
                // the first atom's class)
                const int n = min(FA, n_i - ibase);
                int nag[FA / 32];  // first atoms of each group (slots 32 g ...)
                int na = 0;
#pragma unroll
                for (int g = 0; g < FA / 32; ++g) {
                    const int q0 = 32 * g, q = q0 + lane;
                    nag[g] = 0;
                    if (q0 >= n) continue;
                    // row of atom ibase + q (every lane takes part in the shuffles)
                    const int qq = min(ibase + q, n_i - 1);
                    int row = 0;
                    for (int rr = 0; rr < nir; ++rr)
                        row += (qq >= __shfl_sync(0xffffffffu, ipre, rr)) ? 1 : 0;
                    const int rb = __shfl_sync(0xffffffffu, ib, row);
                    const int rp = __shfl_sync(0xffffffffu, ipre - ilen, row);
                    float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
                    if (q < n) v = rec_o[rb + (qq - rp)];
                    const unsigned w = __float_as_uint(v.w);
                    const int ia = (int)(w & 0xffffffu), prow = part_row(ia);
                    const bool have = q < n && (!PARTS || (prow >= 0 && prow < nch));
                    const int ti = (int)(w >> 24),
                              cls = PARTS ? prow / P.nch * P.ntypes + ti : ti;
                    unsigned left = __ballot_sync(0xffffffffu, have);
                    nag[g] = __popc(left);
                    na += nag[g];
                    int at = q0, end = q0;  // its place, the end of its class's run
                    for (int base = q0; left;) {
                        const int c = __shfl_sync(0xffffffffu, cls, __ffs(left) - 1);
                        const unsigned m = __ballot_sync(0xffffffffu, have && cls == c);
                        if (have && cls == c) {
                            at = base + __popc(m & lt);
                            end = base + __popc(m);
                        }
                        base += __popc(m);
                        left &= ~m;
                    }
                    if (have) {
                        const f2 z = f2pk(v.z, v.z);
                        A.fa[at][0] = make_ulonglong2(f2pk(v.x, v.x), f2pk(v.y, v.y));
                        A.fa[at][1] = make_ulonglong2(
                            z, (unsigned long long)((unsigned)end << 16 | (unsigned)cls) << 32 | w);
                        // the atom's pair with itself: from the channel of distinct
                        // atoms, where the loop below counts it, to its own
                        const int b = P.tric ? self_bin<true>(P, fo, fl, ia)
                                             : self_bin<false>(P, fo, fl, ia);
                        if (b >= 0) {
                            const int ch = prow + chtab[ti * P.ntypes + ti];
                            atomicSub(whist + ch * nrow + b, 1u);
                            atomicAdd(whist + (ch + half_ch) * nrow + b, 1u);
                        }
                    }
                }
                if (na == 0) continue;
                if (lane == 0) n_eval += (unsigned long long)na * (unsigned long long)n_j;
                __syncwarp();
                const f2 inv = f2pk(P.rm.inv_dr, P.rm.inv_dr), off = f2pk(P.rm.q_off, P.rm.q_off),
                         tiny = f2pk(RADIAL_TINY, RADIAL_TINY);
                int seg = 0;  // the segment that holds flat record f0 (or the one before it)
                for (int f0 = 0; f0 < n_j; f0 += CH) {
                    // this lane's records f0 + lane + 32 t: the starts of the
                    // segments after `seg` that fall into a group of 32, as bits,
                    // give each lane its segment by a count of the bits up to it
                    float x[4], y[4], z[4];
                    unsigned tj[4], sj[4];  // type; image << 25 | sorted slot
#pragma unroll
                    for (int t = 0; t < 4; ++t) {
                        const int fb = f0 + 32 * t;
                        const unsigned rel = (unsigned)(A.pre[seg + 1 + lane] - fb);
                        const unsigned m =
                            __reduce_or_sync(0xffffffffu, rel < 32u ? 1u << rel : 0u);
                        const int mine = seg + __popc(m & (lt | 1u << lane));
                        seg += __popc(m);
                        x[t] = y[t] = z[t] = qnan;  // no record: never within rmax
                        tj[t] = sj[t] = 0u;
                        if (fb + lane < n_j) {
                            const int2 sc = A.src[mine];
                            const float4 v = rec_l[sc.x + fb + lane];
                            sj[t] = (unsigned)(sc.x + fb + lane) | (unsigned)sc.y << 25;
                            // moved to its image ((0, 0, 0) adds zeros: x + 0 = x)
                            const float4 sh = s_shift[sc.y];
                            x[t] = __fadd_rn(v.x, sh.x);
                            y[t] = __fadd_rn(v.y, sh.y);
                            z[t] = __fadd_rn(v.z, sh.z);
                            tj[t] = __float_as_uint(v.w) >> 24;
                        }
                    }
                    const f2 xa = f2pk(x[0], x[1]), xb = f2pk(x[2], x[3]);
                    const f2 ya = f2pk(y[0], y[1]), yb = f2pk(y[2], y[3]);
                    const f2 za = f2pk(z[0], z[1]), zb = f2pk(z[2], z[3]);
                    for (int g = 0; g < FA / 32; ++g) {
                        const int q0 = 32 * g, q1 = q0 + (g ? nag[1] : nag[0]);
                        unsigned mk[4] = {0u, 0u, 0u, 0u}, bit = 1u;
                        // one first atom (broadcast) against the lane's four records
                        auto four = [&](f2 fx, f2 fy, f2 fz, const unsigned *row) {
                            // one difference per axis, three FMAs
                            const f2 dxa = f2sub(fx, xa), dya = f2sub(fy, ya), dza = f2sub(fz, za);
                            const f2 dxb = f2sub(fx, xb), dyb = f2sub(fy, yb), dzb = f2sub(fz, zb);
                            const f2 da = f2fma(dza, dza, f2fma(dya, dya, f2fma(dxa, dxa, tiny)));
                            const f2 db = f2fma(dzb, dzb, f2fma(dyb, dyb, f2fma(dxb, dxb, tiny)));
                            bin_pair2<MODE>(da, inv, off, P.rm, row[0], row[1], bit, mk[0], mk[1]);
                            bin_pair2<MODE>(db, inv, off, P.rm, row[2], row[3], bit, mk[2], mk[3]);
                        };
                        // first atoms of one class at a time; one a turn: the loop is
                        // small (unrolled by two it measured 3 % slower, by four
                        // 50 %: instruction fetches)
                        for (int i = q0; i < q1;) {
                            const unsigned hi = (unsigned)(A.fa[i][1].y >> 32);
                            const int e = (int)(hi >> 16), cls = (int)(hi & 0xffffu);
                            const int part = PARTS ? cls / P.ntypes : 0;
                            const unsigned short *ct = chtab + (cls - part * P.ntypes) * P.ntypes;
                            const unsigned rowp = row0 + rowb * (unsigned)(part * P.nch);
                            unsigned row[4];
#pragma unroll
                            for (int t = 0; t < 4; ++t) row[t] = rowp + rowb * ct[tj[t]];
                            for (; i < e; ++i) {
                                const ulonglong2 u0 = A.fa[i][0];
                                four(u0.x, u0.y, A.fa[i][1].x, row);
                                bit <<= 1;
                            }
                        }
                        if (P.rm.lim < 0.0f) {  // every pair is noted: not those without a record
#pragma unroll
                            for (int t = 0; t < 4; ++t)
                                if (f0 + 32 * t + lane >= n_j) mk[t] = 0u;
                        }
                        // pairs within the margin of a bin edge, one per lane and
                        // round, into their queue; it is taken 32 at a time
                        while (__any_sync(0xffffffffu, (mk[0] | mk[1] | mk[2] | mk[3]) != 0u)) {
                            unsigned bits = 0u, sl = 0u;
#pragma unroll
                            for (int t = 3; t >= 0; --t)
                                if (mk[t]) { bits = mk[t]; sl = sj[t]; }
                            const bool have = bits != 0u;
                            bool first = have;
#pragma unroll
                            for (int t = 0; t < 4; ++t)
                                if (first && mk[t]) { mk[t] &= mk[t] - 1u; first = false; }
                            const unsigned m = __ballot_sync(0xffffffffu, have);
                            if (have)
                                A.near[nn + __popc(m & lt)] =
                                    make_uint2((unsigned)(q0 + __ffs(bits) - 1), sl);
                            nn += __popc(m);
                            if (nn >= 32) {
                                resolve(32);
                                nn -= 32;
                                if (lane < nn) A.near[lane] = A.near[32 + lane];
                                __syncwarp();
                            }
                        }
                    }
                }
                resolve(nn);  // the entries name first atoms of this batch
                nn = 0;
                __syncwarp();  // every lane done with the first atoms and segments
            }
        }
        recheck(qn);
        qn = 0;
        again = __syncthreads_or(lane == 0 && A.held >= 0) != 0;
        if (!again) g0 = g1;
        }
    }
    __syncthreads();
    if (cur >= 0 && !lost) flush(cur);
    if (tid == 0) {
        if (lost) atomicOr(P.err, ERRW_HIST_OVERFLOW);
        // the last CTA leaves the queue as the next launch on the stream takes it
        __threadfence();
        if (atomicAdd(C.queue + 1, 1u) == gridDim.x - 1) {
            C.queue[0] = 0u;
            C.queue[1] = 0u;
        }
    }
    for (int o = 16; o > 0; o >>= 1) {
        n_cand += __shfl_xor_sync(0xffffffffu, n_cand, o);
        n_rech += __shfl_xor_sync(0xffffffffu, n_rech, o);
        n_eval += __shfl_xor_sync(0xffffffffu, n_eval, o);
    }
    if (lane == 0) {
        if (n_cand) atomicAdd(P.stats + ST_CANDIDATES, n_cand);
        if (n_rech) atomicAdd(P.stats + ST_RECHECKS, n_rech);
        if (n_eval) atomicAdd(P.stats + ST_EVALUATED, n_eval);
    }
}

}  // namespace cellw

int cellw_smem_bytes(int nch, int nbin, int ntypes, int cta_warps, int hcopy)
{
    using namespace cellw;
    const size_t hist_cap = (size_t)nch * (nbin + 1) + 1;
    size_t b = sizeof(WarpArea) * cta_warps + (size_t)hcopy * hist_cap * 4 +
               (size_t)ntypes * ntypes * 2;
    return (int)((b + 127) / 128 * 128);
}

int cellw_chunk_records() { return cellw::CH; }
int cellw_batch_atoms() { return cellw::FA; }

// Sorted AoS copy of every frame: {x, y, z, type << 24 | id} with the block
// kernel's coordinates (w = x - n L, n = floor((x - xlo) / L), one FMA in
// FP64, then fl32(fl64(w - c)), c the box centre); triclinic: w the lattice
// reduction of wrap_tric64, the same FP32 rounding about the centre.
__global__ void k_cell_scatter_w(const double *__restrict__ pos64,
                                 const unsigned char *__restrict__ types8, size_t T, size_t N,
                                 size_t NP, int ncell, double xlo, double ylo, double zlo,
                                 double Lx, double Ly, double Lz, double xy, double xz, double yz,
                                 int tric, double cx, double cy, double cz,
                                 const int *__restrict__ cell_of, const int *__restrict__ rank_of,
                                 const int *__restrict__ start, float4 *__restrict__ wpos)
{
    const double lo[3] = {xlo, ylo, zlo}, L[3] = {Lx, Ly, Lz}, c[3] = {cx, cy, cz};
    const double tilt[3] = {xy, xz, yz};
    for (size_t g = blockIdx.x * (size_t)blockDim.x + threadIdx.x; g < T * N;
         g += (size_t)gridDim.x * blockDim.x) {
        const size_t f = g / N, a = g - f * N;
        const size_t d = (size_t)start[f * (size_t)(ncell + 1) + cell_of[g]] + rank_of[g];
        const double *p = pos64 + g * 3;
        float v[3];
        if (tric) {
            double w[3];
            wrap_tric64(p, lo, L, tilt, w);
#pragma unroll
            for (int k = 0; k < 3; ++k) v[k] = __double2float_rn(__dsub_rn(w[k], c[k]));
        } else {
#pragma unroll
            for (int k = 0; k < 3; ++k) {
                const double n = floor(__ddiv_rn(__dsub_rn(p[k], lo[k]), L[k]));
                const double w = __fma_rn(-n, L[k], p[k]);
                v[k] = __double2float_rn(__dsub_rn(w, c[k]));
            }
        }
        wpos[f * NP + d] =
            make_float4(v[0], v[1], v[2], __uint_as_float(((unsigned)types8[a] << 24) | (unsigned)a));
    }
}

int launch_cell_scatter_w(const double *pos64, const unsigned char *types8, size_t T, size_t N,
                          const double *box_internal, const double *centre, const int *nc,
                          bool tric, const int *cell_of, const int *rank_of, const int *start,
                          float4 *wpos, cudaStream_t s)
{
    const int ncell = nc[0] * nc[1] * nc[2];
    const size_t NP = padded_natoms(N);
    // padding records: NaN coordinates (never read as atoms)
    if (cudaMemsetAsync(wpos, 0xff, T * NP * sizeof(float4), s) != cudaSuccess) return -1;
    const size_t total = T * N;
    int blocks = (int)((total + 255) / 256);
    if (blocks > 152 * 16) blocks = 152 * 16;
    const double Lx = 2.0 * box_internal[3], Ly = 2.0 * box_internal[4], Lz = 2.0 * box_internal[5];
    k_cell_scatter_w<<<blocks, 256, 0, s>>>(pos64, types8, T, N, NP, ncell, box_internal[0],
                                            box_internal[1], box_internal[2], Lx, Ly, Lz,
                                            box_internal[6], box_internal[7], box_internal[8],
                                            tric ? 1 : 0, centre[0], centre[1], centre[2],
                                            cell_of, rank_of, start, wpos);
    return cudaGetLastError() == cudaSuccess ? 0 : -1;
}

template <int NWARP, int HCOPY, int MODE, bool PARTS>
static int launch_cellw_shape(const CellwLaunch &C, int num_sms, cudaStream_t s)
{
    using namespace cellw;
    constexpr int NT = NWARP * 32;
    auto kern = k_pairs_cellw<NWARP, HCOPY, MODE, PARTS>;
    const int smem = cellw_smem_bytes(C.pair.nch * C.pg, C.pair.nbin, C.pair.ntypes, NWARP, HCOPY);
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem) !=
        cudaSuccess)
        return -1;
    int per_sm = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, NT, smem) != cudaSuccess)
        return -1;
    if (per_sm < 1) return -2;
    // at least a warp block a warp
    const long long units = C.pair.n_items * C.npg * C.nw[0] * C.nw[1] * C.nw[2];
    long long grid = (long long)num_sms * per_sm;
    if (grid > (units + NWARP - 1) / NWARP) grid = (units + NWARP - 1) / NWARP;
    kern<<<(unsigned)grid, NT, smem, s>>>(C);
    return cudaGetLastError() == cudaSuccess ? 0 : -1;
}

// Whether one CTA of 32 warps takes the place of the CTAs of 16: where the
// histogram lets only one of those on an SM, and 32 warps' areas fit beside it
// (half the warps left the SM waiting on latencies: 5488 atoms, 4 partitions
// of 14 KB, 5.55 to 4.67 ms; 16384 atoms, 4 types, 800 bins, 3.71 to 3.06).
static bool cellw_wide(const CellwLaunch &C)
{
    if (C.cta_warps != 16 || C.hcopy != 1 || C.most < 32) return false;
    int dev = 0, sm = 0, cta = 0;
    if (cudaGetDevice(&dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&sm, cudaDevAttrMaxSharedMemoryPerMultiprocessor, dev) !=
            cudaSuccess ||
        cudaDeviceGetAttribute(&cta, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev) != cudaSuccess)
        return false;
    auto bytes = [&C](int warps) {  // with the static shared memory
        return cellw_smem_bytes(C.pair.nch * C.pg, C.pair.nbin, C.pair.ntypes, warps, 1) + 2048;
    };
    const int reserved = sm - cta;  // per CTA
    return 2 * (bytes(16) + reserved) > sm && bytes(32) <= cta;
}

template <int MODE>
static int launch_cellw_mode(const CellwLaunch &C, int num_sms, cudaStream_t s)
{
    if (cellw_wide(C))
        return C.pair.nparts > 1 ? launch_cellw_shape<32, 1, MODE, true>(C, num_sms, s)
                                 : launch_cellw_shape<32, 1, MODE, false>(C, num_sms, s);
    if (C.pair.nparts > 1) {
        return C.cta_warps == 16 ? launch_cellw_shape<16, 1, MODE, true>(C, num_sms, s)
                                 : launch_cellw_shape<8, 1, MODE, true>(C, num_sms, s);
    }
    if (C.cta_warps == 16) {
        return C.hcopy == 2 ? launch_cellw_shape<16, 2, MODE, false>(C, num_sms, s)
                            : launch_cellw_shape<16, 1, MODE, false>(C, num_sms, s);
    }
    return C.hcopy == 2 ? launch_cellw_shape<8, 2, MODE, false>(C, num_sms, s)
                        : launch_cellw_shape<8, 1, MODE, false>(C, num_sms, s);
}

int launch_cellw_pairs(const CellwLaunch &C, int num_sms, cudaStream_t s)
{
    if (C.pair.n_items <= 0) return 0;
    switch (C.pair.rm.mode) {
    case 0: return launch_cellw_mode<0>(C, num_sms, s);
    case 1: return launch_cellw_mode<1>(C, num_sms, s);
    default: return launch_cellw_mode<2>(C, num_sms, s);
    }
}

}  // namespace gofr

// All-pairs FP32 kernel with FP64 recheck: every ordered pair of every (lag,
// origin) of a Gofrt::calculate (lib/src/gofrt.cpp:96-122, minimum image
// lib/include/basetrajectory.h:181-268), for boxes and histograms that the
// cell-list kernels do not take or do not gain on: boxes of a few rmax, boxes
// that change from frame to frame, counts per reference thread partition, and
// (k_allpairs_batch) many trajectories or windows in one launch.
//
// A warp takes a group of up to 64 first atoms (frame `origin`, duplicated
// into f32x2 operands in its own shared memory, in the order of their types)
// and walks the frame `origin + lag` 128 second atoms at a time, four
// consecutive ones per lane in registers (three 16-byte loads and the types);
// each first atom is broadcast against them.  Both atoms' coordinates are moved
// into the box as they are loaded, so a pair's d2 takes three differences, per
// axis |d| or L - |d| (nearest; triclinic: an FMA with a 1.5*2^23 offset and a
// subtraction that round d/L to the nearest integer k and an FMA d - k*L), and
// three FMAs, two pairs per packed instruction; it is binned where it is found
// (bin_pair2, gofr_device.cuh), the pairs near a bin edge (WCHK: or near a wrap
// decision) in FP64.  The bound behind the margins is derived on the host
// (gofr_capi.cu, error_bound_boxed, error_bound, radial_margin).
//
// Warps share nothing but the CTA's histogram, so neither a remainder of
// first atoms nor one of a barrier's worth of second atoms idles a CTA: the
// only waste is the last, partly empty chunk of 128.
//
// Bound by instruction issue (77 % of the slots used, the FMA pipe 56 %, the
// ALU 50 %, the shared-memory pipe 46 %): 80 instructions for a first atom
// against a chunk, 94 with the loads and the pairs near an edge (fewer where FAR
// leaves most pairs out).  2187 atoms to
// 13.5 A in a box of 28 A (47 % of the pairs counted), 40 origins x 50 lags: 7.6
// ms = 1260 Gpairs/s, where the form with tiles of 1024 atoms staged by bulk
// copies and per-thread candidate slots binned by the warp took 26.1; with the
// rounded quotient of the triclinic form 8.2.  5488 atoms to 9 A in four
// partitions, 20 x 40: 18.3 ms against 32.7; 1000 atoms to 3.5 A (1.7 %
// counted), 18 x 20: 0.32 against 0.44; 300 atoms, 6 x 6: 23 us against 78.  64
// registers, spilling outside the loops (bytes stored / loaded: 90 / 104, triclinic
// 130 / 140, FAR 102 / 116 and 158 / 176, batch 220 / 424 and 276 / 640): with 80 and
// three CTAs per SM within 2 %.
#include <cstdint>
#include <cuda_runtime.h>

#include "gofr_device.cuh"
#include "gofr_internal.h"

namespace gofr {
namespace allpairs {

constexpr int NWARP = 8;
constexpr int NT = NWARP * 32;
constexpr int CH = ALLPAIRS_CHUNK;
constexpr int FA = ALLPAIRS_GROUP;
constexpr int QW = 64;   // entries of a warp's queues (a round adds at most 32, taken at 32)

// Shared memory of one warp.
struct WarpArea {
    ulonglong2 fa[FA][2];  // first atoms {x x | y y}, {z z | id, run end << 8 | type}: coordinates
                           // duplicated for f32x2, and the end of the run of the same type
    uint2 near[QW];        // pairs near a bin edge: {first atom, second atom's id}
    uint2 q[QW];           // FP64 recheck queue: ids of both atoms
};

// Box constants of one origin frame (f2: duplicated into both lanes).
struct BoxReg {
    f2 invL[3], negL[3];
    f2 negT[3];       // -{xy, xz, yz}
    float L[3];
    float wmax[3];    // orthorhombic: |component| from which the image is not certain
};

// Triclinic, k = d / L rounded to the nearest integer; WCHK: w0, w1 the largest
// distance of a quotient from its integer so far, per lane.
template <bool WCHK>
__device__ __forceinline__ f2 wraps(f2 d, f2 invL, float &w0, float &w1)
{
    const f2 MAG = f2pk(RADIAL_MAGIC, RADIAL_MAGIC);
    if (!WCHK) return f2sub(f2fma(d, invL, MAG), MAG);
    const f2 q = f2mul(d, invL);
    const f2 k = f2sub(f2add(q, MAG), MAG);
    float a, b;
    f2up(f2sub(q, k), a, b);
    w0 = fmaxf(w0, fabsf(a));
    w1 = fmaxf(w1, fabsf(b));
    return k;
}

// Coordinates moved into [-L/2, L/2] (orthorhombic: both atoms of a pair are,
// so that an FP32 difference needs one subtraction for its image; triclinic: as
// they are).
template <bool TRI>
__device__ __forceinline__ f2 into_box(f2 x, const BoxReg &b, int k)
{
    if (TRI) return x;
    float u0, u1;
    return f2fma(wraps<false>(x, b.invL[k], u0, u1), b.negL[k], x);
}

// |minimum image| of two differences of coordinates within the box: |d| or L -
// |d|, the smaller (one FP32 addition and one minimum, which runs beside the
// FMA pipe, for the FMA, subtraction and FMA of a rounded quotient: the pipe
// those share with everything else of a pair is what bounds the kernel).
template <bool WCHK>
__device__ __forceinline__ f2 nearest(f2 d, float L, float wmax, bool &w0, bool &w1)
{
    float a, b;
    f2up(d, a, b);
    a = fminf(fabsf(a), __fsub_rn(L, fabsf(a)));
    b = fminf(fabsf(b), __fsub_rn(L, fabsf(b)));
    if (WCHK) {
        w0 = w0 || a > wmax;
        w1 = w1 || b > wmax;
    }
    return f2pk(a, b);
}

// Minimum-image d2 of two pairs (triclinic: z, then y, then x); WCHK: w0, w1
// set when the image is not certain.
template <bool TRI, bool WCHK>
__device__ __forceinline__ f2 image_d2(f2 dx, f2 dy, f2 dz, const BoxReg &b, float wlim, bool &w0,
                                       bool &w1)
{
    w0 = w1 = false;
    if (TRI) {
        float u0 = 0.0f, u1 = 0.0f;
        const f2 kz = wraps<WCHK>(dz, b.invL[2], u0, u1);
        dz = f2fma(kz, b.negL[2], dz);
        dy = f2fma(kz, b.negT[2], dy);
        dx = f2fma(kz, b.negT[1], dx);
        const f2 ky = wraps<WCHK>(dy, b.invL[1], u0, u1);
        dy = f2fma(ky, b.negL[1], dy);
        dx = f2fma(ky, b.negT[0], dx);
        const f2 kx = wraps<WCHK>(dx, b.invL[0], u0, u1);
        dx = f2fma(kx, b.negL[0], dx);
        if (WCHK) {
            w0 = u0 > wlim;
            w1 = u1 > wlim;
        }
    } else {
        dx = nearest<WCHK>(dx, b.L[0], b.wmax[0], w0, w1);
        dy = nearest<WCHK>(dy, b.L[1], b.wmax[1], w0, w1);
        dz = nearest<WCHK>(dz, b.L[2], b.wmax[2], w0, w1);
    }
    const f2 tiny = f2pk(RADIAL_TINY, RADIAL_TINY);
    return f2fma(dz, dz, f2fma(dy, dy, f2fma(dx, dx, tiny)));
}

// What a warp carries from unit to unit.
struct WarpState {
    unsigned long long n_rech = 0;
};

// One unit: first atoms [i0, i1) (at most FA) of frame fo against part jp of
// the atoms of frame fl (jc chunks), into the histogram at whist (rows of
// nbin + 1 cells).  All lanes of the warp call it.  FAR: 64 pairs of a first
// atom that all lie beyond P.far2 are not binned (they end in the unread cell), for
// jobs in which few pairs are within rmax (gofr_capi.cu, far_limit).
template <bool TRI, bool WCHK, int MODE, bool FAR = false>
__device__ __forceinline__ void unit(const PairLaunch &P, WarpArea &A, unsigned *whist,
                                     const unsigned short *chtab, long long fo, long long fl,
                                     int i0, int i1, int jp, WarpState &ws)
{
    const int lane = threadIdx.x & 31;
    const unsigned lt = (1u << lane) - 1u;
    const int nbin = P.nbin, nrow = nbin + 1, half_ch = P.nch / 2;
    const unsigned row0 = smem_u32(whist) - 4u * RADIAL_MAGIC_BITS, rowb = 4u * (unsigned)nrow;
    const long long NP = P.NP;
    const float qnan = __int_as_float(0x7fc00000);
    const float *const fi = P.pos32 + fo * 3 * NP;
    const float *const fj = P.pos32 + fl * 3 * NP;
    BoxReg bx;
    {
        const Box32 b = P.box32[fo];
#pragma unroll
        for (int a = 0; a < 3; ++a) {
            bx.L[a] = b.L[a];
            bx.wmax[a] = 0.5f * b.L[a] - P.wtol;
            bx.invL[a] = f2pk(b.invL[a], b.invL[a]);
            bx.negL[a] = f2pk(-b.L[a], -b.L[a]);
            bx.negT[a] = f2pk(-b.tilt[a], -b.tilt[a]);
        }
    }
    const int na = i1 - i0;
    for (int q0 = 0; q0 < na; q0 += 32) {
        // each group of 32 in the order of types: the row addresses of a lane's
        // second atoms change only with the first atom's type
        const bool have = q0 + lane < na;
        const int ia = i0 + q0 + lane;
        const unsigned ti = have ? P.types8[ia] : 0u;
        unsigned left = __ballot_sync(0xffffffffu, have);
        int at = q0, end = q0;
        for (int base = q0; left;) {
            const unsigned t = __shfl_sync(0xffffffffu, ti, __ffs(left) - 1);
            const unsigned m = __ballot_sync(0xffffffffu, have && ti == t);
            if (have && ti == t) {
                at = base + __popc(m & lt);
                end = base + __popc(m);
            }
            base += __popc(m);
            left &= ~m;
        }
        if (have) {
            const float x = fi[ia], y = fi[NP + ia], z = fi[2 * NP + ia];
            A.fa[at][0] = make_ulonglong2(into_box<TRI>(f2pk(x, x), bx, 0),
                                          into_box<TRI>(f2pk(y, y), bx, 1));
            A.fa[at][1] = make_ulonglong2(
                into_box<TRI>(f2pk(z, z), bx, 2),
                (unsigned long long)((unsigned)end << 8 | ti) << 32 | (unsigned)ia);
            // the atom's pair with itself: from the channel of distinct atoms,
            // where the loop below counts it, to its own (in the unit that counts
            // it: a cell is never below zero when it is flushed)
            // At lag 0 the distance is exactly zero, which lies on a bin edge when
            // rmin is 0: given here, and in `resolve`, since every atom took the
            // FP64 arithmetic twice otherwise (68 us a call of 300 atoms against 63;
            // the cell-list kernel loses 1 % to the test and has less of lag 0)
            const int s0 = jp * P.jc * CH;
            const int b = ia < s0 || ia >= s0 + P.jc * CH ? -1
                          : fo == fl                      ? P.self0
                                                          : self_bin<TRI>(P, fo, fl, ia);
            if (b >= 0) {
                const int ch = chtab[(int)ti * P.ntypes + (int)ti];
                atomicSub(whist + ch * nrow + b, 1u);
                atomicAdd(whist + (ch + half_ch) * nrow + b, 1u);
            }
        }
    }
    __syncwarp();

    int nn = 0, qn = 0;  // entries of the two queues (the same in every lane)
    // Recomputes queued pairs [0, n) in exact FP64 (reference arithmetic), one
    // per lane; into the channel of distinct atoms, like every pair.
    auto recheck = [&](int n) {
        __syncwarp();
        if (lane < n) {
            const uint2 e = A.q[lane];
            const double *xi = P.pos64 + (fo * P.N + (int)e.x) * 3;
            const double *xj = P.pos64 + (fl * P.N + (int)e.y) * 3;
            const double d2 =
                ref_d2<TRI>(xi[0], xi[1], xi[2], xj[0], xj[1], xj[2], P.box64 + fo * 9, P.err);
            const int b = ref_bin(d2, P.rmin, P.dr, P.rmin2, P.rmax2, nbin);
            const int ch = chtab[(int)P.types8[e.x] * P.ntypes + (int)P.types8[e.y]];
            if (b >= 0 && GOFR_CHECK(ch < P.nch && b < nbin, P.err))
                atomicAdd(whist + ch * nrow + b, 1u);
            ++ws.n_rech;
        }
        __syncwarp();
    };
    // Takes entries [0, n) of `near`, one per lane: the pair's bin again with
    // the pair loop's operations (the same value), out of the cell it was
    // added to, and into the recheck queue where it can be within the window.
    auto resolve = [&](int n) {
        __syncwarp();
        bool need = false;
        uint2 e = make_uint2(0u, 0u);
        unsigned ia = 0u;
        if (lane < n) {
            e = A.near[lane];
            const ulonglong2 u0 = A.fa[e.x][0], u1 = A.fa[e.x][1];
            ia = (unsigned)u1.y;
            const float xj = fj[e.y], yj = fj[NP + e.y], zj = fj[2 * NP + e.y];
            float d2, unused;
            bool w0, w1;
            f2up(image_d2<TRI, WCHK>(f2sub(u0.x, into_box<TRI>(f2pk(xj, xj), bx, 0)),
                                     f2sub(u0.y, into_box<TRI>(f2pk(yj, yj), bx, 1)),
                                     f2sub(u1.x, into_box<TRI>(f2pk(zj, zj), bx, 2)), bx, P.wlim,
                                     w0, w1),
                 d2, unused);
            const float t = __fadd_rn(radial_q(d2, P.rm), RADIAL_MAGIC);
            const int b = (int)(__float_as_uint(t) - RADIAL_MAGIC_BITS);
            need = (t <= P.rm.t_hi && t >= P.rm.t_lo) || (WCHK && w0);
            unsigned *const row =
                whist + chtab[(int)(u1.y >> 32 & 0xffu) * P.ntypes + (int)P.types8[e.y]] * nrow;
            if (b >= 0 && b < nbin) atomicSub(row + b, 1u);
            if (fo == fl && ia == e.y) {
                need = false;
                if (P.self0 >= 0) atomicAdd(row + P.self0, 1u);
            }
        }
        const unsigned m = __ballot_sync(0xffffffffu, need);
        if (need) A.q[qn + __popc(m & lt)] = make_uint2(ia, e.y);
        qn += __popc(m);
        if (qn >= 32) {
            recheck(32);
            qn -= 32;
            if (lane < qn) A.q[lane] = A.q[32 + lane];
            __syncwarp();
        }
    };

    const f2 inv = f2pk(P.rm.inv_dr, P.rm.inv_dr), off = f2pk(P.rm.q_off, P.rm.q_off);
    const int jend = min(P.N, (jp + 1) * P.jc * CH);
    for (int f0 = jp * P.jc * CH; f0 < jend; f0 += CH) {
        const int j0 = f0 + 4 * lane;  // the frame is padded with NaN to a multiple of 16
        float4 X = make_float4(qnan, qnan, qnan, qnan), Y = X, Z = X;
        unsigned tj = 0u;
        if (j0 < NP) {
            X = *reinterpret_cast<const float4 *>(fj + j0);
            Y = *reinterpret_cast<const float4 *>(fj + NP + j0);
            Z = *reinterpret_cast<const float4 *>(fj + 2 * NP + j0);
            tj = *reinterpret_cast<const unsigned *>(P.types8 + j0);
        }
        const f2 xa = into_box<TRI>(f2pk(X.x, X.y), bx, 0), xb = into_box<TRI>(f2pk(X.z, X.w), bx, 0);
        const f2 ya = into_box<TRI>(f2pk(Y.x, Y.y), bx, 1), yb = into_box<TRI>(f2pk(Y.z, Y.w), bx, 1);
        const f2 za = into_box<TRI>(f2pk(Z.x, Z.y), bx, 2), zb = into_box<TRI>(f2pk(Z.z, Z.w), bx, 2);
        for (int q0 = 0; q0 < na; q0 += 32) {
            const int q1 = min(na, q0 + 32);
            unsigned mk[4] = {0u, 0u, 0u, 0u}, bit = 1u;
            for (int i = q0; i < q1;) {
                const unsigned hi = (unsigned)(A.fa[i][1].y >> 32);
                const int e = (int)(hi >> 8);
                const unsigned short *ct = chtab + (int)(hi & 0xffu) * P.ntypes;
                unsigned row[4];
#pragma unroll
                for (int t = 0; t < 4; ++t) row[t] = row0 + rowb * ct[tj >> (8 * t) & 0xffu];
                for (; i < e; ++i) {
                    const ulonglong2 u0 = A.fa[i][0];
                    const f2 uz = A.fa[i][1].x;
                    bool wa0, wa1, wb0, wb1;
                    const f2 da = image_d2<TRI, WCHK>(f2sub(u0.x, xa), f2sub(u0.y, ya),
                                                      f2sub(uz, za), bx, P.wlim, wa0, wa1);
                    const f2 db = image_d2<TRI, WCHK>(f2sub(u0.x, xb), f2sub(u0.y, yb),
                                                      f2sub(uz, zb), bx, P.wlim, wb0, wb1);
                    if (FAR) {
                        float d0, d1, d2, d3;
                        f2up(da, d0, d1);
                        f2up(db, d2, d3);
                        if (__any_sync(0xffffffffu, fminf(d0, d1) <= P.far2))
                            bin_pair2<MODE>(da, inv, off, P.rm, row[0], row[1], bit, mk[0], mk[1]);
                        if (__any_sync(0xffffffffu, fminf(d2, d3) <= P.far2))
                            bin_pair2<MODE>(db, inv, off, P.rm, row[2], row[3], bit, mk[2], mk[3]);
                        bit <<= 1;
                        continue;
                    }
                    bin_pair2<MODE>(da, inv, off, P.rm, row[0], row[1], bit, mk[0], mk[1]);
                    bin_pair2<MODE>(db, inv, off, P.rm, row[2], row[3], bit, mk[2], mk[3]);
                    if (WCHK) {
                        mk[0] |= wa0 ? bit : 0u;
                        mk[1] |= wa1 ? bit : 0u;
                        mk[2] |= wb0 ? bit : 0u;
                        mk[3] |= wb1 ? bit : 0u;
                    }
                    bit <<= 1;
                }
            }
            if (P.rm.lim < 0.0f) {  // every pair is noted: not those without an atom
#pragma unroll
                for (int t = 0; t < 4; ++t)
                    if (j0 + t >= P.N) mk[t] = 0u;
            }
            while (__any_sync(0xffffffffu, (mk[0] | mk[1] | mk[2] | mk[3]) != 0u)) {
                unsigned bits = 0u, j = 0u;
#pragma unroll
                for (int t = 3; t >= 0; --t)
                    if (mk[t]) { bits = mk[t]; j = (unsigned)(j0 + t); }
                const bool have = bits != 0u;
                bool first = have;
#pragma unroll
                for (int t = 0; t < 4; ++t)
                    if (first && mk[t]) { mk[t] &= mk[t] - 1u; first = false; }
                const unsigned m = __ballot_sync(0xffffffffu, have);
                if (have)
                    A.near[nn + __popc(m & lt)] = make_uint2((unsigned)(q0 + __ffs(bits) - 1), j);
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
    resolve(nn);
    recheck(qn);
}

// Adds the CTA's histogram to counts (rows of nbin) and clears it, the unread
// cells too; the pairs counted (all threads; every warp is done with its units).
__device__ __forceinline__ unsigned long long flush(unsigned *hist, int nch, int nbin,
                                                    unsigned long long *counts, bool add)
{
    unsigned long long n = 0;
    const int nrow = nbin + 1;
    for (int i = threadIdx.x; i <= nch * nrow; i += NT) {
        const unsigned v = hist[i];
        if (!v) continue;
        hist[i] = 0u;
        const int ch = (i - 1) / nrow, b = i - 1 - ch * nrow;  // the cell before the first row: 0
        if (i == 0 || b == nbin) continue;
        n += v;
        if (add) atomicAdd(counts + ch * nbin + b, (unsigned long long)v);
    }
    __syncthreads();
    return n;
}

__device__ __forceinline__ void add_stats(unsigned long long *stats, unsigned long long cand,
                                          unsigned long long rech)
{
    for (int o = 16; o > 0; o >>= 1) {
        cand += __shfl_xor_sync(0xffffffffu, cand, o);
        rech += __shfl_xor_sync(0xffffffffu, rech, o);
    }
    if ((threadIdx.x & 31) == 0) {
        if (cand) atomicAdd(stats + ST_CANDIDATES, cand);
        if (rech) atomicAdd(stats + ST_RECHECKS, rech);
    }
}

// One trajectory: units are (window, partition, lag, origin, group of first
// atoms, part of the second atoms), the part fastest, dealt in chunks of
// decreasing size (chunk_range); the histogram is flushed when the window,
// partition or lag changes.
template <bool TRI, bool WCHK, int MODE, bool FAR>
__global__ void __launch_bounds__(NT, 4) k_allpairs(const PairLaunch P)
{
    extern __shared__ __align__(128) unsigned char smem[];
    WarpArea *const areas = reinterpret_cast<WarpArea *>(smem);
    unsigned *const hist = reinterpret_cast<unsigned *>(areas + NWARP);
    const int hcells = P.nch * (P.nbin + 1) + 1;
    unsigned short *const chtab = reinterpret_cast<unsigned short *>(hist + hcells);
    __shared__ int s_next, s_full;
    __shared__ long long s_u0, s_u1;
    __shared__ unsigned long long s_pairs;  // pairs evaluated since the last flush
    const int tid = threadIdx.x, lane = tid & 31;
    WarpArea &A = areas[tid >> 5];
    for (int i = tid; i < hcells; i += NT) hist[i] = 0u;
    for (int i = tid; i < P.ntypes * P.ntypes; i += NT) chtab[i] = type_channel(i, P.ntypes);
    if (tid == 0) s_pairs = 0ull;

    const int per = P.N / P.nparts;
    const int ngj = P.ng * P.nj;  // units of a (lag, origin)
    const long long per_plane = (long long)P.n_orig * ngj;
    const long long U = per_plane * P.n_lags * P.nparts * P.nwin;
    unsigned long long n_cand = 0;
    bool lost = false;  // a u32 bin could have overflowed
    int cur = -1;       // plane (window, partition, lag) of the histogram
    auto flush_plane = [&]() {
        if (s_pairs > 0xffffffffull) lost = true;
        const int lag = cur % P.n_lags, part = cur / P.n_lags % P.nparts,
                  win = cur / P.n_lags / P.nparts;
        n_cand += flush(hist, P.nch, P.nbin,
                        P.counts + win * P.win_stride + part * P.part_stride +
                            (long long)lag * P.every * P.nch * P.nbin,
                        !lost);
        if (tid == 0) s_pairs = 0ull;
        __syncthreads();
    };
    WarpState ws;
    while (!lost) {
        __syncthreads();  // every warp has read the last chunk's range
        if (tid == 0) {
            long long u0 = 0, u1 = 0;
            chunk_range((long long)atomicAdd(P.queue, 1u), gridDim.x, U, P.most, NWARP, u0, u1);
            s_u0 = u0;
            s_u1 = u1;
            s_next = 0;
            s_full = s_pairs > 0x7fffffffull;
        }
        __syncthreads();
        const long long c0 = s_u0, c1 = s_u1;
        if (c0 >= c1) break;
        for (long long g0 = c0; g0 < c1 && !lost;) {
            const int plane = (int)(g0 / per_plane);
            const long long g1 = min(c1, (plane + 1) * per_plane);
            if (g0 != c0) {
                __syncthreads();  // the warps are done with the chunk's last plane
                if (tid == 0) {
                    s_next = 0;
                    s_full = s_pairs > 0x7fffffffull;
                }
                __syncthreads();
            }
            if (cur >= 0 && (plane != cur || s_full)) flush_plane();
            cur = plane;
            const int lag_idx = plane % P.n_lags, part = plane / P.n_lags % P.nparts;
            const long long first =
                P.primos ? P.primos[plane / P.n_lags / P.nparts] : P.primo;
            const int a0 = part * per, a1 = part == P.nparts - 1 ? P.N : a0 + per;
            for (;;) {
                int nx = 0;
                if (lane == 0) nx = atomicAdd(&s_next, 1);
                nx = __shfl_sync(0xffffffffu, nx, 0);
                if (g0 + nx >= g1) break;
                const long long u = g0 + nx - plane * per_plane;
                const int k = (int)(u / ngj), gj = (int)(u - (long long)k * ngj);
                const int grp = gj / P.nj, jp = gj - grp * P.nj;
                const int i0 = a0 + grp * P.gs, i1 = min(a1, i0 + P.gs);
                if (i0 >= i1) continue;
                if (lane == 0)
                    atomicAdd(&s_pairs, (unsigned long long)(i1 - i0) *
                                            (unsigned long long)min(P.N, P.jc * CH));
                const long long fo = first + (long long)k * P.skip;
                unit<TRI, WCHK, MODE, FAR>(P, A, hist + 1, chtab, fo,
                                           fo + (long long)lag_idx * P.every, i0, i1, jp, ws);
                __syncwarp();  // every lane done with the first atoms
            }
            g0 = g1;
        }
    }
    __syncthreads();
    if (cur >= 0 && !lost) flush_plane();
    if (tid == 0) {
        if (lost) atomicOr(P.err, ERRW_HIST_OVERFLOW);
        // the last CTA leaves the queue as the next launch on the stream takes it
        __threadfence();
        if (atomicAdd(P.queue + 1, 1u) == gridDim.x - 1) {
            P.queue[0] = 0u;
            P.queue[1] = 0u;
        }
    }
    add_stats(P.stats, n_cand, ws.n_rech);
}

// Many trajectories in one persistent launch.  Each CTA pulls work
// descriptors (trajectory, range of its units) from a device queue (one atomic
// counter; descriptors sorted by decreasing cost on the host), switches the
// shared tables when the trajectory changes, and flushes its histogram into
// that trajectory's counts at every new lag and at the end of a descriptor.
template <bool TRI, int MODE>
__global__ void __launch_bounds__(NT, 4) k_allpairs_batch(const PairLaunch *__restrict__ trajs,
                                                          const WorkDesc *__restrict__ work,
                                                          int n_work, unsigned *head, int max_cells,
                                                          unsigned *err, unsigned long long *stats)
{
    extern __shared__ __align__(128) unsigned char smem[];
    WarpArea *const areas = reinterpret_cast<WarpArea *>(smem);
    unsigned *const hist = reinterpret_cast<unsigned *>(areas + NWARP);
    unsigned short *const chtab = reinterpret_cast<unsigned short *>(hist + max_cells);
    __shared__ int s_idx, s_next;
    // the current trajectory's parameters live in shared memory: a register
    // copy of the whole struct would crowd out the hot loop
    __shared__ __align__(16) PairLaunch sP;
    const PairLaunch &P = sP;
    const int tid = threadIdx.x, lane = tid & 31;
    WarpArea &A = areas[tid >> 5];
    for (int i = tid; i < max_cells; i += NT) hist[i] = 0u;
    int cur = -1;
    unsigned long long n_cand = 0;
    WarpState ws;
    for (;;) {
        __syncthreads();
        if (tid == 0) {
            s_idx = (int)atomicAdd(head, 1u);
            s_next = 0;
        }
        __syncthreads();
        const int idx = s_idx;
        if (idx >= n_work) break;
        const WorkDesc w = work[idx];
        if (w.traj != cur) {
            constexpr int words = (int)(sizeof(PairLaunch) / 4);
            const unsigned *src = reinterpret_cast<const unsigned *>(trajs + w.traj);
            for (int i = tid; i < words; i += NT) reinterpret_cast<unsigned *>(&sP)[i] = src[i];
            __syncthreads();
            for (int i = tid; i < P.ntypes * P.ntypes; i += NT) chtab[i] = type_channel(i, P.ntypes);
            cur = w.traj;
            __syncthreads();
        }
        const bool wchk = P.wchk != 0;
        const int ngj = P.ng * P.nj;
        const long long per_lag = (long long)P.n_orig * ngj;
        for (long long g0 = w.u0; g0 < w.u1;) {
            const int lag_idx = (int)(g0 / per_lag);
            const long long g1 = min(w.u1, (lag_idx + 1) * per_lag);
            for (;;) {
                int nx = 0;
                if (lane == 0) nx = atomicAdd(&s_next, 1);
                nx = __shfl_sync(0xffffffffu, nx, 0);
                if (g0 + nx >= g1) break;
                const long long u = g0 + nx - lag_idx * per_lag;
                const int k = (int)(u / ngj), gj = (int)(u - (long long)k * ngj);
                const int grp = gj / P.nj, jp = gj - grp * P.nj;
                const int i0 = grp * P.gs, i1 = min(P.N, i0 + P.gs);
                const long long fo = P.primo + (long long)k * P.skip;
                const long long fl = fo + (long long)lag_idx * P.every;
                if (wchk) unit<TRI, true, MODE>(P, A, hist + 1, chtab, fo, fl, i0, i1, jp, ws);
                else unit<TRI, false, MODE>(P, A, hist + 1, chtab, fo, fl, i0, i1, jp, ws);
                __syncwarp();
            }
            __syncthreads();
            if (tid == 0) s_next = 0;
            n_cand += flush(hist, P.nch, P.nbin,
                            P.counts + (long long)lag_idx * P.every * P.nch * P.nbin, true);
            g0 = g1;
        }
    }
    add_stats(stats, n_cand, ws.n_rech);
}

size_t smem_bytes(int cells, int ntypes)
{
    const size_t b = sizeof(WarpArea) * NWARP + (size_t)cells * 4 + (size_t)ntypes * ntypes * 2;
    return (b + 127) / 128 * 128;
}

template <typename K>
int grid_of(K kernel, size_t smem, int num_sms, long long blocks, int *grid)
{
    if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) !=
        cudaSuccess)
        return -1;
    int per_sm = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, NT, smem) != cudaSuccess)
        return -1;
    if (per_sm < 1) return -2;
    long long g = (long long)num_sms * per_sm;
    if (g > blocks) g = blocks;
    *grid = (int)(g < 1 ? 1 : g);
    return 0;
}

template <bool TRI, bool WCHK, int MODE, bool FAR>
int launch(const PairLaunch &P, int num_sms, cudaStream_t s)
{
    const size_t smem = smem_bytes(P.nch * (P.nbin + 1) + 1, P.ntypes);
    const long long units = (long long)P.nwin * P.nparts * P.n_lags * P.n_orig * P.ng * P.nj;
    int grid = 0;
    const int rc = grid_of(k_allpairs<TRI, WCHK, MODE, FAR>, smem, num_sms,
                           (units + NWARP - 1) / NWARP, &grid);
    if (rc) return rc;
    k_allpairs<TRI, WCHK, MODE, FAR><<<(unsigned)grid, NT, smem, s>>>(P);
    return cudaGetLastError() == cudaSuccess ? 0 : -1;
}

template <bool TRI, bool WCHK, bool FAR>
int launch_mode(const PairLaunch &P, int num_sms, cudaStream_t s)
{
    switch (P.rm.mode) {
    case 0: return launch<TRI, WCHK, 0, FAR>(P, num_sms, s);
    case 1: return launch<TRI, WCHK, 1, FAR>(P, num_sms, s);
    default: return launch<TRI, WCHK, 2, FAR>(P, num_sms, s);
    }
}

}  // namespace allpairs

size_t allpairs_smem_bytes(int nch, int nbin, int ntypes)
{
    return allpairs::smem_bytes(nch * (nbin + 1) + 1, ntypes);
}

int launch_allpairs(const PairLaunch &P, bool wrapcheck, int num_sms, cudaStream_t s)
{
    using namespace allpairs;
    if (P.n_lags <= 0 || P.n_orig <= 0 || P.ng <= 0) return 0;
    if (wrapcheck)
        return P.tric ? launch_mode<true, true, false>(P, num_sms, s)
                      : launch_mode<false, true, false>(P, num_sms, s);
    if (P.far2 < INFINITY)
        return P.tric ? launch_mode<true, false, true>(P, num_sms, s)
                      : launch_mode<false, false, true>(P, num_sms, s);
    return P.tric ? launch_mode<true, false, false>(P, num_sms, s)
                  : launch_mode<false, false, false>(P, num_sms, s);
}

// The batch's bin map is mode 0's when every member's is, else the general one.
int prepare_batch(int max_cells, int max_ntypes, bool tric, int mode, int num_sms, int n_work,
                  int *grid)
{
    using namespace allpairs;
    const size_t smem = smem_bytes(max_cells, max_ntypes);
    if (tric)
        return mode == 0 ? grid_of(k_allpairs_batch<true, 0>, smem, num_sms, n_work, grid)
                         : grid_of(k_allpairs_batch<true, 2>, smem, num_sms, n_work, grid);
    return mode == 0 ? grid_of(k_allpairs_batch<false, 0>, smem, num_sms, n_work, grid)
                     : grid_of(k_allpairs_batch<false, 2>, smem, num_sms, n_work, grid);
}

int launch_batch_grid(const PairLaunch *d_trajs, const WorkDesc *d_work, int n_work,
                      unsigned *d_head, int max_cells, int max_ntypes, bool tric, int mode,
                      unsigned *d_err, unsigned long long *d_stats, int grid, cudaStream_t s)
{
    using namespace allpairs;
    if (n_work <= 0) return 0;
    const size_t smem = smem_bytes(max_cells, max_ntypes);
    auto kernel = tric ? (mode == 0 ? k_allpairs_batch<true, 0> : k_allpairs_batch<true, 2>)
                       : (mode == 0 ? k_allpairs_batch<false, 0> : k_allpairs_batch<false, 2>);
    kernel<<<(unsigned)grid, NT, smem, s>>>(d_trajs, d_work, n_work, d_head, max_cells, d_err,
                                            d_stats);
    return cudaGetLastError() == cudaSuccess ? 0 : -1;
}

}  // namespace gofr

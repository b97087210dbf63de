// Mean square displacement on the resident FP64 frames (the reference's
// MSD<T>::calc_single_th, lib/src/msd.cpp:70-118).
//
// The reference loops lag -> origin -> atom and keeps, per (lag, type), a
// running mean of |x_i(o) - x_i(o+t)|^2 (optionally minus the type's
// centre-of-mass displacement), and of the centres' own squared displacement.
//
// k_msd_fixed: FP64 instructions issue at 1/64 of the FP32 rate here, so the
// sums are taken in integers, exactly.  A coordinate (minus its type's centre
// where asked for) is rint(x 2^s) modulo 2^64, s so that the displacements of
// its type are below 2^57 (k_extent: the frames' extents, from their FP32
// copies).  Coordinates of a 32nd of the largest displacement and more are held
// exactly; those nearer to zero lose what lies below 2^-57 of that displacement,
// a sixteenth of what FP64 resolves it to.  A displacement is one 64-bit subtraction, its
// square three 29-bit products (64-bit multiply-adds), whose sums are combined
// in 128 bits and rounded once per (lag, type): no term is rounded at all,
// where the FP64 sums rounded every one.  Where coordinates lost bits and the
// displacements of a (lag, type) are so small that the bound on the result's
// error (lost_shows) exceeds the FP64 sums' own, the caller has the FP64 sums
// taken for that (lag, type) alone (k_msd_entries).
// (With the unit taken from the largest coordinate instead, a tracer near the
// origin of a box of 130 had an error of 5.5e-14 against the FP64 sums' 5.5e-16.)
// A CTA holds the frames of a few atoms of one type in shared memory, so each
// coordinate is read from HBM once and every (origin, lag) pair comes from
// shared memory: thread = (lag, phase of the origins), consecutive lags reading
// consecutive frames.
//   Bound by the 32-bit integer multiplier.  16384 atoms in
// three types, 100 origins x 100 lags: 0.45 ms against 2.79 for the FP64 form;
// 5003 atoms with both centre-of-mass options, 60 x 80: 0.12 against 0.48.
//
// k_msd_partial: the FP64 form, for windows of lags whose frames of one atom
// do not fit shared memory (more than about 4000 lags) and for origins too far
// apart to share frames (msd_fixed_plan).  Every (origin, lag)
// item is one CTA: it forms each atom's displacement with the reference's FP64
// operations, adds its squared components into the type's sum with FMAs
// (atoms visited in type-sorted order, one block reduction per type) and
// writes one partial sum per (lag, origin, type).  A second kernel adds the
// origins of each (lag, type) in a fixed order and divides by the count.
// Items are ordered origin-major so that consecutive CTAs share the origin
// frame and slide the lagged frame, which keeps the frames they read in L2.
#include <algorithm>
#include <cstdint>
#include <cuda_runtime.h>

#include "gofr_internal.h"

namespace gofr {
namespace msd {

constexpr int NT = 256;

__device__ __forceinline__ double sq3(double dx, double dy, double dz)
{
    // pow(dx,2) + pow(dy,2) + pow(dz,2), left to right (lib/src/msd.cpp:98-100)
    return __dadd_rn(__dadd_rn(__dmul_rn(dx, dx), __dmul_rn(dy, dy)), __dmul_rn(dz, dz));
}

__device__ double block_sum(double v, double *red)
{
    for (int o = 16; o > 0; o >>= 1) v = __dadd_rn(v, __shfl_down_sync(0xffffffffu, v, o));
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (lane == 0) red[w] = v;
    __syncthreads();
    double s = 0.0;
    if (threadIdx.x == 0)
        for (int k = 0; k < NT / 32; ++k) s = __dadd_rn(s, red[k]);
    __syncthreads();
    return s;  // valid in thread 0
}

// Sum over the atoms of type k of their squared displacements between frames fo
// and fl; valid in thread 0 (all threads of the CTA).
__device__ __forceinline__ double type_sum(const MsdLaunch &M, long long fo, long long fl, int k,
                                           double *red)
{
    const double *po = M.pos64 + (size_t)fo * M.N * 3;
    const double *pl = M.pos64 + (size_t)fl * M.N * 3;
    double cx = 0.0, cy = 0.0, cz = 0.0;
    if (M.cm_self) {
        const double *co = M.cm + ((size_t)fo * M.ntypes + k) * 3;
        const double *cl = M.cm + ((size_t)fl * M.ntypes + k) * 3;
        cx = __dsub_rn(co[0], cl[0]);
        cy = __dsub_rn(co[1], cl[1]);
        cz = __dsub_rn(co[2], cl[2]);
    }
    double acc = 0.0;
    for (int q = M.tbegin[k] + threadIdx.x; q < M.tbegin[k + 1]; q += NT) {
        const size_t a = (size_t)M.perm[q] * 3;
        double dx = __dsub_rn(po[a], pl[a]);
        double dy = __dsub_rn(po[a + 1], pl[a + 1]);
        double dz = __dsub_rn(po[a + 2], pl[a + 2]);
        if (M.cm_self) {
            dx = __dsub_rn(dx, cx);
            dy = __dsub_rn(dy, cy);
            dz = __dsub_rn(dz, cz);
        }
        // the squares go straight into the sum (three FMAs instead of
        // three products, two additions and one accumulation: the
        // kernel is bound by the FP64 pipe)
        acc = __fma_rn(dz, dz, __fma_rn(dy, dy, __fma_rn(dx, dx, acc)));
    }
    return block_sum(acc, red);
}

__global__ void __launch_bounds__(NT) k_msd_partial(const MsdLaunch M)
{
    __shared__ double red[NT / 32];
    const int fk = M.cm_msd ? 2 * M.ntypes : M.ntypes;
    const long long n_items = (long long)M.n_orig * M.leff;
    for (long long item = blockIdx.x; item < n_items; item += gridDim.x) {
        const int o = (int)(item / M.leff);
        const int lag = (int)(item - (long long)o * M.leff);
        const long long fo = (long long)M.primo + (long long)o * M.skip;
        const long long fl = fo + lag;
        double *out = M.partial + ((size_t)lag * M.n_orig + o) * fk;
        for (int k = 0; k < M.ntypes; ++k) {
            const double s = type_sum(M, fo, fl, k, red);
            if (threadIdx.x == 0) out[k] = s;
        }
        if (M.cm_msd && threadIdx.x < M.ntypes) {
            const int k = threadIdx.x;
            const double *co = M.cm + ((size_t)fo * M.ntypes + k) * 3;
            const double *cl = M.cm + ((size_t)fl * M.ntypes + k) * 3;
            out[M.ntypes + k] =
                sq3(__dsub_rn(co[0], cl[0]), __dsub_rn(co[1], cl[1]), __dsub_rn(co[2], cl[2]));
        }
    }
}

// The same for the n results (lag ntypes + type) of `entries` alone: partial sums
// [n][n_orig], then the results in their places.
__global__ void __launch_bounds__(NT) k_msd_entries(const MsdLaunch M, const int *entries, int n)
{
    __shared__ double red[NT / 32];
    const long long n_items = (long long)n * M.n_orig;
    for (long long item = blockIdx.x; item < n_items; item += gridDim.x) {
        const int at = entries[item / M.n_orig], o = (int)(item % M.n_orig);
        const long long fo = (long long)M.primo + (long long)o * M.skip;
        const double s = type_sum(M, fo, fo + at / M.ntypes, at % M.ntypes, red);
        if (threadIdx.x == 0) M.partial[item] = s;
    }
}

__global__ void k_msd_entries_final(const MsdLaunch M, const int *entries, int n, double *out)
{
    const int fk = M.cm_msd ? 2 * M.ntypes : M.ntypes;
    const int g = blockIdx.x * blockDim.x + threadIdx.x;
    if (g >= n) return;
    const int k = entries[g] % M.ntypes;
    double s = 0.0;
    for (int o = 0; o < M.n_orig; ++o) s = __dadd_rn(s, M.partial[(size_t)g * M.n_orig + o]);
    out[(size_t)(entries[g] / M.ntypes) * fk + k] =
        __ddiv_rn(s, (double)M.n_orig * (double)(M.tbegin[k + 1] - M.tbegin[k]));
}

// out[lag][c][k] = sum over origins (in order) / count
__global__ void k_msd_final(const MsdLaunch M, double *out)
{
    const int fk = M.cm_msd ? 2 * M.ntypes : M.ntypes;
    const long long n = (long long)M.leff * fk;
    for (long long g = blockIdx.x * (long long)blockDim.x + threadIdx.x; g < n;
         g += (long long)gridDim.x * blockDim.x) {
        const int lag = (int)(g / fk), c = (int)(g - (long long)lag * fk);
        const double *p = M.partial + (size_t)lag * M.n_orig * fk + c;
        double s = 0.0;
        for (int o = 0; o < M.n_orig; ++o) s = __dadd_rn(s, p[(size_t)o * fk]);
        const double count = c < M.ntypes
                                 ? (double)M.n_orig * (double)(M.tbegin[c + 1] - M.tbegin[c])
                                 : (double)M.n_orig;
        out[g] = __ddiv_rn(s, count);
    }
}

// ---------------------------------------------------------------------------
// exact integer sums
// ---------------------------------------------------------------------------
constexpr int FT = 512;    // threads per CTA
constexpr int NACC = 6;    // sums h h, h l, l l: low 32 bits and the rest of each
constexpr int TERMS = 8;   // squared displacements (three axes each) between two carries
constexpr int PLANE = 105 * 1024 / 24;  // (atom, frame) entries of an axis in shared memory: a
                                        // constant, so the axes are offsets of one address
constexpr int BITS = 57;   // displacements are below 2^BITS: the products of add_square

// Sums of the products of d = h 2^29 + l (|d| < 2^57, h signed, l in [0,
// 2^29)): hh < 2^56, |hl| < 2^57 and ll < 2^58 in 64 bits, carried into the
// sums of the high words every TERMS displacements (24 products of 2^58 and a
// low word stay below 2^63).
struct Acc {
    long long p[3], hi[3];
};

// rint(x 2^shift) modulo 2^64, halves away from zero: integer
// instructions alone (a product and a conversion of the FP64 pipe took a
// fifth of the kernel's time).  lost counts the values that were rounded.
__device__ __forceinline__ unsigned long long to_fixed(double x, int shift, unsigned &lost)
{
    const long long u = __double_as_longlong(x);
    const int e = (int)(u >> 52 & 0x7ff);
    const unsigned long long m = (u & 0xfffffffffffffull) | 0x10000000000000ull;
    const int r = 1075 - shift - e;  // bits below the point
    if (r > 53 || e == 0) {          // less than half a unit (and below 2^-1022)
        if (x != 0.0) ++lost;
        return 0;
    }
    if (r > 0 && (m & ((1ull << r) - 1)) != 0) ++lost;
    const unsigned long long v =
        r > 0 ? (m + (1ull << (r - 1))) >> r : (r > -64 ? m << -r : 0ull);
    return u < 0 ? 0ull - v : v;
}

// s of type k: the bound on its displacements, taken from the FP32 frames with
// their rounding (pad), and of the centres', is below 2^(BITS - s).
__device__ __forceinline__ int unit_shift(const MsdLaunch &M, const MsdFixed &X, int k)
{
    double d = __dadd_ru((double)__uint_as_float(X.ext[k]), X.pad);
    if (M.cm_self) d = __dadd_ru(d, X.cm_ext[k]);
    return BITS - ((int)(__double_as_longlong(d) >> 52) - 1022);
}

// Whether the bits lost can show in the sum S of a result (units squared; count
// terms, na atoms).  A value is off by half a unit at most, a displacement by the
// errors of its two ends (and of their centres), and an end takes part in two
// terms of a lag, so the squares of the displacements' errors sum up to 2 lost at most
// and S is off by 2 sqrt(S 2 lost) and less than a millionth of that.  The FP64
// sums' own bound is more than c 2^-53 of S: a rounded displacement squared (2), the
// block's sum (8 and more), three FMAs per 256 atoms, an addition per origin.  S is
// kept where the former is no larger than c 2^-53, c at most 32 (3.6e-15).
__device__ __forceinline__ bool lost_shows(double S, double lost, int na, int n_orig)
{
    const double c = fmin(32.0, 10.0 + n_orig + 3.0 * ((na + NT - 1) / NT));
    return lost > 0.0 && S * (c * c) < lost * 649037107316853453566312041152512.0;  // 2^109
}

__device__ __forceinline__ void mad_wide(long long &a, int x, int y)
{
    asm("mad.wide.s32 %0, %1, %2, %0;" : "+l"(a) : "r"(x), "r"(y));
}

__device__ __forceinline__ void add_square(Acc &a, long long d)
{
    const int h = (int)(d >> 29), l = (int)d & 0x1fffffff;
    mad_wide(a.p[0], h, h);
    mad_wide(a.p[1], h, l);
    mad_wide(a.p[2], l, l);
}

// The displacement of two values held modulo 2^64.
__device__ __forceinline__ long long minus(long long a, long long b)
{
    return (long long)((unsigned long long)a - (unsigned long long)b);
}

// p keeps its low 32 bits; the rest goes to hi.
__device__ __forceinline__ void carry(Acc &a)
{
#pragma unroll
    for (int i = 0; i < 3; ++i) {
        a.hi[i] += a.p[i] >> 32;
        a.p[i] &= 0xffffffffll;
    }
}

// Chunks of type k: tiles of origins of groups of `atoms` atoms.
__device__ __forceinline__ long long chunks_of(const MsdLaunch &M, const MsdFixed &X, int k)
{
    return (long long)((M.tbegin[k + 1] - M.tbegin[k] + X.atoms - 1) / X.atoms) * X.tiles;
}

// CTA b takes chunks [b per, (b + 1) per) of the types' chunks back to back.  The sums of the CTA's
// chunks of type k go to partial[b + k] (CTAs and types both ascend, so the
// entry is one (CTA, type)'s own).
// APART: no frame is in the lags of two origins.  A tile is then one origin, its
// threads (lag, lane of the atoms), and a chunk takes as many atoms as fit, so that it
// reads long pieces of each frame.  A call for 3000 atoms, 40 origins x 10 lags
// every 500 frames: 79 us; 535 with the origins' phases on the threads and the
// frames between the origins staged; 97 for the FP64 form.
template <bool APART>
__global__ void __launch_bounds__(FT, 2) k_msd_fixed(const MsdLaunch M, const MsdFixed X)
{
    extern __shared__ __align__(16) long long smem[];
    const int tid = threadIdx.x, F = X.frames;
    const int l0 = blockIdx.y * X.lags, nl = min(X.lags, M.leff - l0);
    const int lag = l0 + tid % X.lags, part = tid / X.lags;
    const int phase = APART ? 0 : part, lane = APART ? part : 0;
    const bool busy = part < X.phases && lag < l0 + nl;
    const long long c0 = (long long)blockIdx.x * X.per, c1 = min(c0 + X.per, X.chunks);
    Acc acc{};
    unsigned lost = 0;  // values of the type that are not held exactly
    __shared__ unsigned long long s_lost;
    if (tid == 0) s_lost = 0ull;  // (every flush starts with a barrier)
    const int step = X.phases * M.skip;
    // loading: thread = (frame phase lf, atom la, axis lx)
    const int per_frame = 3 * X.atoms, lstep = FT / per_frame, lf = tid / per_frame,
              la = (tid - lf * per_frame) / 3, lx = tid - lf * per_frame - 3 * la;
    int k = 0;
    long long kb = 0, ke = chunks_of(M, X, 0);  // chunks of type k
    auto to_type_of = [&](long long c) {
        while (c >= ke) {
            kb = ke;
            ke += chunks_of(M, X, ++k);
        }
    };
    to_type_of(c0);
    int shift = unit_shift(M, X, k);
    // the sums of the CTA's chunks of type k, every phase's, to their entry
    auto flush = [&]() {
        long long *out = X.partial + ((long long)(blockIdx.x + k) * M.leff + l0) * NACC;
        carry(acc);
#pragma unroll
        for (int i = 0; i < NACC; ++i) {
            __syncthreads();  // the tile, or the last sum, is no longer read
            smem[tid] = busy ? (i < 3 ? acc.p[i] : acc.hi[i - 3]) : 0;
            __syncthreads();
            if (tid < nl) {
                long long v = 0;
                for (int ph = 0; ph < X.phases; ++ph) v += smem[ph * X.lags + tid];
                out[tid * NACC + i] = v;
            }
        }
        acc = Acc{};
        if (lost) atomicAdd(&s_lost, (unsigned long long)lost);
        lost = 0;
        __syncthreads();
        if (tid == 0) {
            X.lost[blockIdx.x + k] = (long long)s_lost;
            s_lost = 0ull;
        }
    };
    for (long long c = c0; c < c1; ++c) {
        if (c >= ke) {
            flush();
            to_type_of(c);
            shift = unit_shift(M, X, k);
        }
        const int group = (int)((c - kb) / X.tiles),
                  tile = (int)((c - kb) - (long long)group * X.tiles);
        const int a0 = M.tbegin[k] + group * X.atoms, na = min(X.atoms, M.tbegin[k + 1] - a0);
        const int o0 = tile * X.origins, no = min(X.origins, M.n_orig - o0);
        const long long f0 = M.primo + (long long)o0 * M.skip;
        const int nf = (no - 1) * M.skip + M.leff;
        __syncthreads();  // the last tile is no longer read
        if (la < na && lf < lstep) {
            const double *x = M.pos64 + ((f0 + lf) * M.N + M.perm[a0 + la]) * 3 + lx;
            const double *cm = M.cm_self ? M.cm + ((f0 + lf) * M.ntypes + k) * 3 + lx : nullptr;
            long long *out = smem + lx * PLANE + la * F;
#pragma unroll 4
            for (int f = lf; f < nf; f += lstep) {
                unsigned long long v = to_fixed(*x, shift, lost);
                x += (long long)lstep * M.N * 3;
                if (cm) {
                    v -= to_fixed(*cm, shift, lost);
                    cm += (long long)lstep * M.ntypes * 3;
                }
                out[f] = (long long)v;
            }
        }
        __syncthreads();
        if (busy) {
            for (int a = lane; a < na; a += APART ? X.phases : 1) {
                int i = a * F + phase * M.skip;
                for (int o = phase; o < no;) {
                    // TERMS origins between two carries
                    const int oe = min(no, o + TERMS * X.phases);
#pragma unroll 2
                    for (; o < oe; o += X.phases, i += step) {
                        const int j = i + lag;
                        add_square(acc, minus(smem[j], smem[i]));
                        add_square(acc, minus(smem[j + PLANE], smem[i + PLANE]));
                        add_square(acc, minus(smem[j + 2 * PLANE], smem[i + 2 * PLANE]));
                    }
                    carry(acc);
                }
            }
        }
    }
    flush();
}

__device__ __forceinline__ double to_double(__int128 v)  // v >= 0, one rounding of each half
{
    return __dadd_rn(__dmul_rn((double)(long long)(v >> 64), 18446744073709551616.0),
                     __ull2double_rn((unsigned long long)v));
}

// One warp per result: the sums of a (lag, type) over its entries, exactly, or
// the centres' squared displacement over the origins.
__global__ void k_msd_fixed_final(const MsdLaunch M, const MsdFixed X, double *out)
{
    const int lane = threadIdx.x & 31;
    const int fk = M.cm_msd ? 2 * M.ntypes : M.ntypes;
    const int g = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    if (g >= M.leff * fk) return;
    const int lag = g / fk, c = g - lag * fk;
    if (c >= M.ntypes) {
        const int k = c - M.ntypes;
        double s = 0.0;
        for (int o = lane; o < M.n_orig; o += 32) {
            const long long fo = M.primo + (long long)o * M.skip;
            const double *co = M.cm + (fo * M.ntypes + k) * 3;
            const double *cl = M.cm + ((fo + lag) * M.ntypes + k) * 3;
            s = __dadd_rn(s, sq3(__dsub_rn(co[0], cl[0]), __dsub_rn(co[1], cl[1]),
                                 __dsub_rn(co[2], cl[2])));
        }
        for (int o = 16; o > 0; o >>= 1) s = __dadd_rn(s, __shfl_xor_sync(0xffffffffu, s, o));
        if (lane == 0) out[g] = __ddiv_rn(s, (double)M.n_orig);
        return;
    }
    __int128 hi = 0, lo = 0;  // the sum is hi 2^64 + lo
    double lost = 0.0;
    long long kb = 0;
    for (int k = 0; k < c; ++k) kb += chunks_of(M, X, k);
    const long long ke = kb + chunks_of(M, X, c);
    if (ke > kb) {
        const long long b0 = kb / X.per, b1 = (ke - 1) / X.per;
        for (long long b = b0 + lane; b <= b1; b += 32) {
            const long long *v = X.partial + ((b + c) * M.leff + lag) * NACC;
            lost += (double)X.lost[b + c];
            // h h 2^58 + 2 h l 2^29 + l l, each sum high 2^32 + low
            hi += ((__int128)v[3] << 26) + (v[4] >> 2);
            lo += ((__int128)v[0] << 58) + ((__int128)v[1] << 30) + v[2] +
                  ((__int128)(v[4] & 3) << 62) + ((__int128)v[5] << 32);
        }
    }
    for (int o = 16; o > 0; o >>= 1) {
        const unsigned long long h0 = __shfl_xor_sync(0xffffffffu, (unsigned long long)hi, o),
                                 l0 = __shfl_xor_sync(0xffffffffu, (unsigned long long)lo, o);
        const long long h1 = __shfl_xor_sync(0xffffffffu, (long long)(hi >> 64), o),
                        l1 = __shfl_xor_sync(0xffffffffu, (long long)(lo >> 64), o);
        hi += ((__int128)h1 << 64) + h0;
        lo += ((__int128)l1 << 64) + l0;
        lost += __shfl_xor_sync(0xffffffffu, lost, o);
    }
    if (lane) return;
    hi += lo >> 64;
    const double sum = __dadd_rn(__dmul_rn(to_double(hi), 18446744073709551616.0),
                                 __ull2double_rn((unsigned long long)lo));
    const int na = M.tbegin[c + 1] - M.tbegin[c];
    const double mean = __ddiv_rn(sum, (double)M.n_orig * (double)na);
    out[g] = scalbn(mean, -2 * unit_shift(M, X, c));
    if (lag > 0 && lost_shows(sum, lost, na, M.n_orig)) {
        X.entries[atomicAdd(X.n_entries, 1ull)] = lag * M.ntypes + c;
        atomicAdd(X.n_terms, (unsigned long long)M.n_orig * na);
    }
}

// The largest extent of a component over the frames, per type of atom, from the
// FP32 frames: of all `len` frames from `first` on, or (groups > 1) within each of
// `groups` runs of `len` frames, `stride` apart.  ext: FP32 bits, rounded up; zero
// before the first launch.  Thread = (four components, phase of the frames or
// runs); a block to a run (gridDim.y of them, groups = 1) where these are few or
// long.  Bound by the read: 16384 atoms, 398 frames 78 MB.
__global__ void __launch_bounds__(1024) k_extent(const float *__restrict__ pos32,
                                                 const unsigned char *__restrict__ types8, int N,
                                                 int NP, long long first, int groups, int len,
                                                 int stride, unsigned *ext)
{
    __shared__ float4 s_mx[32][33], s_mn[32][33];
    __shared__ unsigned s_ext[256];
    const int lane = threadIdx.x & 31, phase = threadIdx.x >> 5;
    if (threadIdx.x < 256) s_ext[threadIdx.x] = 0u;
    first += (long long)blockIdx.y * stride;
    const unsigned row = 3u * NP / 4u, c4 = blockIdx.x * 32 + lane;  // NP: a multiple of 16
    const float4 *const src = reinterpret_cast<const float4 *>(pos32);
    float4 mx = make_float4(-INFINITY, -INFINITY, -INFINITY, -INFINITY),
           mn = make_float4(INFINITY, INFINITY, INFINITY, INFINITY);
    auto take = [&](long long f) {
        const float4 v = src[f * row + c4];
        mx = make_float4(fmaxf(mx.x, v.x), fmaxf(mx.y, v.y), fmaxf(mx.z, v.z), fmaxf(mx.w, v.w));
        mn = make_float4(fminf(mn.x, v.x), fminf(mn.y, v.y), fminf(mn.z, v.z), fminf(mn.w, v.w));
    };
    if (c4 < row && groups == 1) {
#pragma unroll 4
        for (int j = phase; j < len; j += 32) take(first + j);
    } else if (c4 < row) {
        float4 e = make_float4(-INFINITY, -INFINITY, -INFINITY, -INFINITY);
        for (int g = phase; g < groups; g += 32) {
            mx = make_float4(-INFINITY, -INFINITY, -INFINITY, -INFINITY);
            mn = make_float4(INFINITY, INFINITY, INFINITY, INFINITY);
#pragma unroll 4
            for (int j = 0; j < len; ++j) take(first + (long long)g * stride + j);
            e = make_float4(fmaxf(e.x, __fsub_ru(mx.x, mn.x)), fmaxf(e.y, __fsub_ru(mx.y, mn.y)),
                            fmaxf(e.z, __fsub_ru(mx.z, mn.z)), fmaxf(e.w, __fsub_ru(mx.w, mn.w)));
        }
        mx = e;
        mn = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    }
    s_mx[phase][lane] = mx;
    s_mn[phase][lane] = mn;
    __syncthreads();
    if (threadIdx.x < 128) {
        const unsigned l = threadIdx.x >> 2, k = threadIdx.x & 3, at = blockIdx.x * 32 + l,
                       atom = (4u * at + k) % (unsigned)NP;
        float a = -INFINITY, b = INFINITY;
        for (int p = 0; p < 32; ++p) {
            a = fmaxf(a, reinterpret_cast<const float *>(&s_mx[p][l])[k]);
            b = fminf(b, reinterpret_cast<const float *>(&s_mn[p][l])[k]);
        }
        const float v = __fsub_ru(a, b);
        if (at < row && atom < (unsigned)N && v > 0.0f)
            atomicMax(s_ext + types8[atom], __float_as_uint(v));
    }
    __syncthreads();
    if (threadIdx.x < 256 && s_ext[threadIdx.x] > ext[threadIdx.x])
        atomicMax(ext + threadIdx.x, s_ext[threadIdx.x]);
}

}  // namespace msd

int launch_msd(const MsdLaunch &M, double *out_device, int num_sms, cudaStream_t s)
{
    using namespace msd;
    const long long n_items = (long long)M.n_orig * M.leff;
    if (n_items <= 0) return 0;
    long long grid = n_items;
    if (grid > (long long)num_sms * 64) grid = (long long)num_sms * 64;
    k_msd_partial<<<(unsigned)grid, NT, 0, s>>>(M);
    const long long nout = (long long)M.leff * (M.cm_msd ? 2 : 1) * M.ntypes;
    long long g2 = (nout + NT - 1) / NT;
    if (g2 > (long long)num_sms * 8) g2 = (long long)num_sms * 8;
    k_msd_final<<<(unsigned)g2, NT, 0, s>>>(M, out_device);
    return cudaGetLastError() == cudaSuccess ? 0 : -1;
}

int launch_msd_entries(const MsdLaunch &M, const int *entries, int n, double *out_device,
                       int num_sms, cudaStream_t s)
{
    using namespace msd;
    const long long items = (long long)n * M.n_orig;
    const long long grid = items < num_sms * 16LL ? items : num_sms * 16LL;
    k_msd_entries<<<(unsigned)grid, NT, 0, s>>>(M, entries, n);
    k_msd_entries_final<<<(n + 127) / 128, 128, 0, s>>>(M, entries, n, out_device);
    return cudaGetLastError() == cudaSuccess ? 0 : -1;
}

int launch_extent(const float *pos32, const unsigned char *types8, size_t N, long long first,
                  int groups, int len, int stride, unsigned *ext, cudaStream_t s)
{
    const size_t NP = padded_natoms(N);
    const unsigned blocks = (unsigned)((3 * NP / 4 + 31) / 32);
    const unsigned runs = (groups < 32 || len >= 256) && groups < 65536 ? groups : 1;
    msd::k_extent<<<dim3(blocks, runs), 1024, 0, s>>>(pos32, types8, (int)N, (int)NP, first,
                                                      runs > 1 ? 1 : groups, len, stride, ext);
    return cudaGetLastError() == cudaSuccess ? 0 : -1;
}

size_t msd_fixed_partial(const MsdLaunch &M, const MsdFixed &X)
{
    return (size_t)(X.grid + M.ntypes) * ((size_t)M.leff * msd::NACC + 1);
}

// Atoms, origins and threads of a CTA of k_msd_fixed, for the type counts in
// h_tbegin; false when the frames of one atom's lags do not fit shared memory
// (two CTAs of 512 threads per SM).
bool msd_fixed_plan(const MsdLaunch &M, const int *h_tbegin, int num_sms, MsdFixed &X)
{
    using namespace msd;
    const long long budget = PLANE;
    const long long all = (long long)(M.n_orig - 1) * M.skip + M.leff;
    X.lags = M.leff < FT ? M.leff : FT;
    X.passes = (M.leff + X.lags - 1) / X.lags;
    X.apart = M.skip >= M.leff || M.n_orig == 1;
    // Where a frame is in the lags of fewer than 1.6 origins, converting and staging it
    // costs what the FP64 arithmetic of its one or two displacements does, and a CTA of
    // long lags waits for its loads: FP64 sums, where their (origin, lag) items fill
    // the GPU.  us a call, FP64 / integers: 3000 atoms, 200 x 50 every 50 frames 651 /
    // 976, every 40 649 / 653, every 30 650 / 544; 16384 atoms, 6 x 200 every 300 416 /
    // 482; 90 x 20 every 20 585 / 544; minus centres, 3000 atoms, 120 x 10 every 100
    // 156 / 172.
    if (8ll * M.skip > 5ll * M.leff && (M.leff >= 32 || M.cm_self) &&
        (long long)M.n_orig * M.leff >= 4ll * num_sms)
        return false;
    auto count = [&](int atoms, int tiles) {
        long long c = 0;
        for (int k = 0; k < M.ntypes; ++k)
            c += (long long)((h_tbegin[k + 1] - h_tbegin[k] + atoms - 1) / atoms) * tiles;
        return c;
    };
    X.atoms = 0;
    if (X.apart) {
        // a thread per component when loading; two chunks per CTA or more
        if (M.leff > budget) return false;
        X.atoms = (int)std::min<long long>(FT / 3, budget / M.leff);
        while (X.atoms > 8 && count(X.atoms, M.n_orig) < 4LL * num_sms) X.atoms /= 2;
        X.origins = 1;
        X.phases = std::min(FT / X.lags, X.atoms);
    } else {
        X.origins = M.n_orig;
        for (int a = 16; a >= 1 && !X.atoms; a /= 2)  // every origin in one tile
            if (all * a <= budget && (a <= 2 || count(a, 1) >= 16LL * num_sms)) X.atoms = a;
        for (int a = 8; a >= 1 && !X.atoms; a /= 2) {
            // tiles of origins: each reads its lags' frames again, so three times
            // as many frames as lags where more than one atom fits
            const long long f = budget / a;
            if (f < (a > 1 ? 3LL * M.leff : (long long)M.leff + M.skip)) continue;
            X.atoms = a;
            X.origins = (int)((f - M.leff) / M.skip + 1);
        }
        if (!X.atoms) return false;
        X.origins = X.origins < M.n_orig ? X.origins : M.n_orig;
        X.phases = std::min(FT / X.lags, X.origins);
    }
    X.tiles = (M.n_orig + X.origins - 1) / X.origins;
    X.frames = (X.origins - 1) * M.skip + M.leff;
    X.chunks = count(X.atoms, X.tiles);
    // contiguous chunks per CTA, two CTAs per SM; no 64-bit sum of 2^17 squares
    // of three axes overflows
    long long per = (X.chunks + 2LL * num_sms - 1) / (2LL * num_sms);
    const long long most = (1LL << 17) / ((long long)X.atoms * X.origins);
    if (most < 1) return false;
    X.per = per < most ? (per > 0 ? per : 1) : most;
    const long long grid = (X.chunks + X.per - 1) / X.per;
    if (grid > (1LL << 30) || X.chunks == 0) return false;
    X.grid = (int)grid;
    return true;
}

int launch_msd_fixed(const MsdLaunch &M, const MsdFixed &X, double *out_device, cudaStream_t s)
{
    using namespace msd;
    const size_t smem = (size_t)3 * PLANE * 8;
    auto kernel = X.apart ? k_msd_fixed<true> : k_msd_fixed<false>;
    if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) !=
        cudaSuccess)
        return -1;
    kernel<<<dim3((unsigned)X.grid, (unsigned)X.passes), FT, smem, s>>>(M, X);
    const long long warps = (long long)M.leff * (M.cm_msd ? 2 : 1) * M.ntypes;
    k_msd_fixed_final<<<(unsigned)((warps + 7) / 8), 256, 0, s>>>(M, X, out_device);
    return cudaGetLastError() == cudaSuccess ? 0 : -1;
}

}  // namespace gofr

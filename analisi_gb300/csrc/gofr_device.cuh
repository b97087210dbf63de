// Device helpers for the Gofrt kernels: inline-PTX TMA bulk copies and
// mbarriers (sm_90+ forms, compiled for sm_103a), bounded waits, and the FP64
// restatement of the reference's pair arithmetic used by the plain FP64 kernel
// and by the edge recheck of the FP32 kernel.
#pragma once
#include <cstdint>
#include <cuda_runtime.h>
#include "gofr_internal.h"

namespace gofr {

// Channel of distinct atoms of the type pair k = a ntypes + c
// (lib/include/gofrt.h:86-104): filled into shared memory by each CTA, which
// takes less than a table's copy to the device before the launch did (8 us).
__device__ __forceinline__ unsigned short type_channel(int k, int ntypes)
{
    const int a = k / ntypes, c = k - a * ntypes, t1 = min(a, c), t2 = max(a, c);
    return (unsigned short)(ntypes * (ntypes + 1) / 2 - (t2 + 1) * (t2 + 2) / 2 + t1);
}

// ---------------------------------------------------------------------------
// mbarrier + cp.async.bulk (1-D TMA) wrappers
// ---------------------------------------------------------------------------
__device__ __forceinline__ unsigned smem_u32(const void *p)
{
    return static_cast<unsigned>(__cvta_generic_to_shared(p));
}

__device__ __forceinline__ void mbar_init(uint64_t *bar, unsigned count)
{
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count)
                 : "memory");
}

// Makes barrier initialisation visible to the async (TMA) proxy.
__device__ __forceinline__ void fence_mbar_init()
{
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}

__device__ __forceinline__ void mbar_arrive_expect_tx(uint64_t *bar, unsigned bytes)
{
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)),
                 "r"(bytes)
                 : "memory");
}

// Global -> shared bulk copy; dst, src 16-byte aligned, bytes a multiple of 16.
__device__ __forceinline__ void bulk_g2s(void *dst, const void *src, unsigned bytes, uint64_t *bar)
{
    asm volatile(
        "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::
            "r"(smem_u32(dst)),
        "l"(src), "r"(bytes), "r"(smem_u32(bar))
        : "memory");
}

__device__ __forceinline__ bool mbar_try_wait(uint64_t *bar, unsigned parity)
{
    unsigned ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}\n"
        : "=r"(ok)
        : "r"(smem_u32(bar)), "r"(parity)
        : "memory");
    return ok != 0;
}

// Iteration cap of every spin wait: each try_wait suspends for a bounded,
// hardware-defined time, so the whole wait is bounded (well under a minute).
constexpr unsigned WAIT_CAP = 1u << 20;
// Cap of the waits of the debug builds' bounded-wait test (a barrier that no
// copy completes): the wait and the abort that follows end within microseconds.
constexpr unsigned DBG_WAIT_CAP = 256u;

__device__ __forceinline__ bool mbar_wait_bounded(uint64_t *bar, unsigned parity,
                                                  unsigned cap = WAIT_CAP)
{
    for (unsigned it = 0; it < cap; ++it)
        if (mbar_try_wait(bar, parity)) return true;
    return false;
}

// Square root for the bin guess of a candidate only.  The certified window
// test that follows decides whether the pair is counted in the guessed bin,
// so the hardware approximation (a few ulp) is enough: a guess that is wrong
// near a bin edge fails the window test and the pair goes to the FP64
// recheck, exactly as a pair inside a window margin does.
__device__ __forceinline__ float sqrt_guess(float x)
{
    float r;
    asm("sqrt.approx.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}

// Adds 1 to the shared-memory word at addr when p holds, as one predicated
// reduction: the histogram updates of a warp flush issue without a branch
// (and its convergence bookkeeping) around each of them.
__device__ __forceinline__ void red_shared_add1_if(unsigned addr, bool p)
{
    asm volatile("{\n\t.reg .pred q;\n\tsetp.ne.u32 q, %1, 0;\n\t@q red.shared.add.u32 [%0], 1;\n\t}"
                 ::"r"(addr), "r"((unsigned)p)
                 : "memory");
}

// ---------------------------------------------------------------------------
// packed f32x2 arithmetic (PTX ISA add/sub/mul/fma .f32x2, sm_100+)
// ---------------------------------------------------------------------------
typedef unsigned long long f2;

__device__ __forceinline__ f2 f2pk(float a, float b)
{
    f2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ void f2up(f2 v, float &a, float &b)
{
    asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v));
}
__device__ __forceinline__ f2 f2add(f2 a, f2 b)
{
    f2 r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ f2 f2sub(f2 a, f2 b)
{
    f2 r;
    asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ f2 f2mul(f2 a, f2 b)
{
    f2 r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ f2 f2fma(f2 a, f2 b, f2 c)
{
    f2 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}


// ---------------------------------------------------------------------------
// Binning a pair where it is found
// ---------------------------------------------------------------------------
//
// Every pair whose d2 is formed is added to a histogram cell at once: two
// pairs of a lane (FP32 d2 in one f32x2) take rs = rsqrt(d2) (hardware
// approximation, relative error <= 2^-22.9), q' = (d2 inv_dr) rs + q_off =
// r / dr - rmin / dr - 1/2, t = q' + 1.5 2^23, whose low mantissa bits are
// n = rint(q'), and fr = q' - n.  The cell is n, with q' clamped to the
// histogram row's ends: a row has nbin cells and an unread one, and a pair beyond
// rmax ends in the unread cell, one below rmin in that of the row before (the
// lanes of a warp that add to one cell are merged: an unread cell for every lane
// took a quarter more shared-memory wavefronts), half a bin from the edge and
// with fr = 0: q', not t, is clamped, so that only the pairs of the window are
// ever noted below (16384 atoms, 72 % of the pairs evaluated beyond rmax: 61.1 to
// 60.1 ms).
// A pair with |fr| > lim may belong to
// the next bin (lim leaves out what r, d2 and the reference's own rounding can
// move a pair by; host: radial_map): `bit` is set in the lane's mask, and the
// caller takes the pair out of its cell again and recomputes it in FP64.
//
// Eleven and a half issue slots per 32 pairs with d2's own (packed: 5 1/2;
// rsqrt, clamp, address, reduction, compare, mask), whatever share of the
// pairs is within rmax.  Queueing the candidates and binning the queue 32 at a
// time cost ~45 (a queue entry ~80 lane instructions).  The reduction is not
// predicated: a predicated red.shared is compiled into a branch around it
// (three more slots and a divergence each), which measured 5 % slower than
// letting every lane add somewhere.
constexpr float RADIAL_MAGIC = 12582912.0f;       // 1.5 * 2^23
constexpr unsigned RADIAL_MAGIC_BITS = 0x4b400000u;
// start of the sum d2: d2 = 0 would make rsqrt infinite and q' NaN (adds 1e-15 to r at most)
constexpr float RADIAL_TINY = 1e-30f;

__device__ __forceinline__ float rsqrt_bin(float x)
{
    float r;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}

// q' of one pair's d2, with bin_pair2's operations.
__device__ __forceinline__ float radial_q(float d2, const RadialMap &m)
{
    return __fmaf_rn(__fmul_rn(d2, m.inv_dr), rsqrt_bin(d2), m.q_off);
}

// row: shared-memory address of the pair's histogram row minus 4 times the
// bits of 1.5 2^23, so cell n is t's bits shifted by two plus it.
template <int MODE>
__device__ __forceinline__ void bin_one(float t, float fr, const RadialMap &m, unsigned row,
                                        unsigned bit, unsigned &mask)
{
    asm volatile("red.shared.add.u32 [%0], 1;" ::"r"((__float_as_uint(t) << 2) + row) : "memory");
    if (MODE == 2) {
        asm("{\n\t.reg .pred p;\n\t.reg .f32 a;\n\tabs.f32 a, %1;\n\t"
            "setp.lt.f32 p, %4, %5;\n\tsetp.gt.or.f32 p, a, %2, p;\n\t@p or.b32 %0, %0, %3;\n\t}"
            : "+r"(mask)
            : "f"(fr), "f"(m.lim), "r"(bit), "f"(t), "f"(m.t_ok));
    } else {
        asm("{\n\t.reg .pred p;\n\t.reg .f32 a;\n\tabs.f32 a, %1;\n\t"
            "setp.gt.f32 p, a, %2;\n\t@p or.b32 %0, %0, %3;\n\t}"
            : "+r"(mask)
            : "f"(fr), "f"(m.lim), "r"(bit));
    }
}

// d2 of two pairs into their histogram rows; inv, off: inv_dr and q_off in both lanes.
template <int MODE>
__device__ __forceinline__ void bin_pair2(f2 d2, f2 inv, f2 off, const RadialMap &m, unsigned row0,
                                          unsigned row1, unsigned bit, unsigned &mask0,
                                          unsigned &mask1)
{
    const f2 MAG = f2pk(RADIAL_MAGIC, RADIAL_MAGIC);
    float a, b;
    f2up(d2, a, b);
    float q0, q1;
    f2up(f2fma(f2mul(d2, inv), f2pk(rsqrt_bin(a), rsqrt_bin(b)), off), q0, q1);
    q0 = fminf(q0, m.q_end);  // no record (NaN): the unread cell
    q1 = fminf(q1, m.q_end);
    if (MODE != 0) {
        q0 = fmaxf(q0, -1.0f);
        q1 = fmaxf(q1, -1.0f);
    }
    const f2 q = f2pk(q0, q1);
    const f2 t = f2add(q, MAG);
    const f2 fr = f2sub(q, f2sub(t, MAG));
    float t0, t1, f0, f1;
    f2up(t, t0, t1);
    f2up(fr, f0, f1);
    bin_one<MODE>(t0, f0, m, row0, bit, mask0);
    bin_one<MODE>(t1, f1, m, row1, bit, mask1);
}

// Units [u0, u1) of chunk c of a launch of G CTAs over U units: every round of G
// chunks takes half of what is left (a CTA meets few chunk ends, and the last
// chunks are small enough for the CTAs to finish together), no chunk more
// than `most` units or fewer than `warps`, and every chunk a multiple of
// `warps`, so that equal units leave no warp of a CTA idle at its end (chunks
// of 9 units for 8 warps kept 44 % of them waiting).
__device__ __forceinline__ void chunk_range(long long c, long long G, long long U, long long most,
                                            long long warps, long long &u0, long long &u1)
{
    most = most < warps ? warps : most / warps * warps;
    long long r = c / G;
    // rounds of full chunks, while half of the rest is more than G of them
    const long long capped = U > 2 * G * most ? (U - 2 * G * most + G * most - 1) / (G * most) : 0;
    const long long full = r < capped ? r : capped;
    long long s = full * G * most, len = most;
    r -= full;
    if (full == capped) {
        for (;; --r) {
            len = (U - s + 2 * G * warps - 1) / (2 * G * warps) * warps;
            if (len < warps) len = warps;
            if (len > most) len = most;
            if (len == warps) s += r * G * len;  // from here on every round is the same
            if (len == warps || r == 0) break;
            s += G * len;
        }
    }
    u0 = s + (c % G) * len;
    u1 = u0 + len < U ? u0 + len : U;
}

// ---------------------------------------------------------------------------
// FP64 restatement of the reference pair arithmetic.
// Every operation is an explicitly rounded IEEE intrinsic, so nvcc cannot
// contract a multiply and an add into an FMA: the result is bit-identical to
// the reference compiled without FMA contraction.
// ---------------------------------------------------------------------------

// Cap on the iterations of one axis of the iterative minimum image.  The
// reference loops until |d| <= l/2 (lib/include/basetrajectory.h:236-267);
// finite coordinates need at most |d|/l+1 iterations, and non-finite ones are
// rejected when frames are uploaded, so the cap only guards the GPU.
constexpr int WRAP_CAP = 1 << 20;

// Iterative minimum image, z then y then x, strict '>' (basetrajectory.h:224-268).
template <bool TRI>
__device__ __forceinline__ void ref_min_image(double &d0, double &d1, double &d2, const double *box,
                                              unsigned *err)
{
    const double lh0 = box[3], lh1 = box[4], lh2 = box[5];
    const double L0 = __dmul_rn(lh0, 2.0), L1 = __dmul_rn(lh1, 2.0), L2 = __dmul_rn(lh2, 2.0);
    double xy = 0.0, xz = 0.0, yz = 0.0;
    if (TRI) { xy = box[6]; xz = box[7]; yz = box[8]; }
    int g = 0;
    while (fabs(d2) > lh2) {
        if (d2 < 0.0) {
            d2 = __dadd_rn(d2, L2);
            if (TRI) { d1 = __dadd_rn(d1, yz); d0 = __dadd_rn(d0, xz); }
        } else {
            d2 = __dsub_rn(d2, L2);
            if (TRI) { d1 = __dsub_rn(d1, yz); d0 = __dsub_rn(d0, xz); }
        }
        if (++g > WRAP_CAP) { atomicOr(err, ERRW_WRAP_LOOP); break; }
    }
    g = 0;
    while (fabs(d1) > lh1) {
        if (d1 < 0.0) {
            d1 = __dadd_rn(d1, L1);
            if (TRI) d0 = __dadd_rn(d0, xy);
        } else {
            d1 = __dsub_rn(d1, L1);
            if (TRI) d0 = __dsub_rn(d0, xy);
        }
        if (++g > WRAP_CAP) { atomicOr(err, ERRW_WRAP_LOOP); break; }
    }
    g = 0;
    while (fabs(d0) > lh0) {
        if (d0 < 0.0) d0 = __dadd_rn(d0, L0);
        else d0 = __dsub_rn(d0, L0);
        if (++g > WRAP_CAP) { atomicOr(err, ERRW_WRAP_LOOP); break; }
    }
}

// d2 of the reference (basetrajectory.h:200-219): ((0 + x*x) + y*y) + z*z.
template <bool TRI>
__device__ __forceinline__ double ref_d2(double xi0, double xi1, double xi2, double xj0, double xj1,
                                         double xj2, const double *box, unsigned *err)
{
    double d0 = __dsub_rn(xi0, xj0), d1 = __dsub_rn(xi1, xj1), d2 = __dsub_rn(xi2, xj2);
    ref_min_image<TRI>(d0, d1, d2, box, err);
    double s = __dmul_rn(d0, d0);
    s = __dadd_rn(s, __dmul_rn(d1, d1));
    s = __dadd_rn(s, __dmul_rn(d2, d2));
    return s;
}

// Bin of the reference (lib/src/gofrt.cpp:104,114-118): filter on d2, then
// (int)floorf((float)((sqrt(d2)-rmin)/dr)), kept when 0 <= idx < nbin.
// A NaN quotient is dropped, as an x86-64 build of the reference does
// (cvttss2si yields INT_MIN); CUDA's float->int of NaN would give 0.
__device__ __forceinline__ int ref_bin(double d2, double rmin, double dr, double rmin2,
                                       double rmax2, int nbin)
{
    if (d2 > rmax2 || d2 < rmin2) return -1;
    double d = __dsqrt_rn(d2);
    double q = __ddiv_rn(__dsub_rn(d, rmin), dr);
    float qf = __double2float_rn(q);
    float fl = floorf(qf);
    if (!(fl >= 0.0f) || fl >= 2147483648.0f) return -1;  // negative, NaN, or beyond int
    int idx = (int)fl;
    return ((unsigned)idx < (unsigned)nbin) ? idx : -1;
}

// Lattice translate of p into the axis-aligned cell [lo, lo + L) of an
// upper-triangular box (cell vectors a = (Lx, 0, 0), b = (xy, Ly, 0),
// c = (xz, yz, Lz); tilt = {xy, xz, yz}), in FP64: the z count from one
// quotient and floor, the z, y and x components moved by FMAs, then y, then
// x.  Each FMA rounds once, so w differs from p - (nz c + ny b + nx a) by at
// most 2^-53 (|y1| + |w_y|) in y and 2^-53 (|x1| + |x2| + |w_x|) in x.  A
// quotient that rounds across an integer leaves w just outside the cell.
__device__ __forceinline__ void wrap_tric64(const double p[3], const double lo[3],
                                            const double L[3], const double tilt[3], double w[3])
{
    const double nz = floor(__ddiv_rn(__dsub_rn(p[2], lo[2]), L[2]));
    w[2] = __fma_rn(-nz, L[2], p[2]);
    const double y1 = __fma_rn(-nz, tilt[2], p[1]);
    const double x1 = __fma_rn(-nz, tilt[1], p[0]);
    const double ny = floor(__ddiv_rn(__dsub_rn(y1, lo[1]), L[1]));
    w[1] = __fma_rn(-ny, L[1], y1);
    const double x2 = __fma_rn(-ny, tilt[0], x1);
    const double nx = floor(__ddiv_rn(__dsub_rn(x2, lo[0]), L[0]));
    w[0] = __fma_rn(-nx, L[0], x2);
}

// The reference's bin of atom ia with itself, frame fo against frame fl (-1:
// not counted).  The pair kernels bin an atom's pair with itself like any
// other, into the channel of distinct atoms (an index compare per pair would
// cost a tenth of their inner loop); this bin is where that count went, to be
// moved to the channel of the same atom.  FP32 on the frames' own coordinates
// where the difference needs no minimum image and lies off every bin edge by
// the all-pairs kernel's bound, else the reference's FP64.
template <bool TRI>
__device__ __forceinline__ int self_bin(const PairLaunch &P, long long fo, long long fl, int ia)
{
    const float *a = P.pos32 + fo * 3 * (long long)P.NP + ia;
    const float *b = P.pos32 + fl * 3 * (long long)P.NP + ia;
    const float dx = __fsub_rn(a[0], b[0]), dy = __fsub_rn(a[P.NP], b[P.NP]),
                dz = __fsub_rn(a[2 * (long long)P.NP], b[2 * (long long)P.NP]);
    if (fmaxf(fabsf(dx), fmaxf(fabsf(dy), fabsf(dz))) <= P.rm.self_max) {
        const float q = radial_q(
            __fmaf_rn(dz, dz, __fmaf_rn(dy, dy, __fmaf_rn(dx, dx, RADIAL_TINY))), P.rm);
        const float t = __fadd_rn(q, RADIAL_MAGIC);
        if (fabsf(__fsub_rn(q, __fsub_rn(t, RADIAL_MAGIC))) <= P.rm.lim_self &&
            (P.rm.mode != 2 || t >= P.rm.t_ok || t < P.rm.t_lo)) {
            const int n = (int)(__float_as_uint(t) - RADIAL_MAGIC_BITS);
            return t <= P.rm.t_hi && t >= P.rm.t_lo && n >= 0 && n < P.nbin ? n : -1;
        }
    }
    const double *xi = P.pos64 + (fo * P.N + ia) * 3, *xj = P.pos64 + (fl * P.N + ia) * 3;
    const double d2 = ref_d2<TRI>(xi[0], xi[1], xi[2], xj[0], xj[1], xj[2], P.box64 + fo * 9, P.err);
    return ref_bin(d2, P.rmin, P.dr, P.rmin2, P.rmax2, P.nbin);
}

}  // namespace gofr

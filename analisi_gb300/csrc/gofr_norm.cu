// FP64 normalisation of g(r,t) counts on the device.
//
// From the exact counts of one or several calculate(primo) windows (per
// reference thread partition) to the reference's double result, on the GPU:
//   mode 0  the Gofrt buffer (lib/src/gofrt.cpp:118,127-132): each
//           partition's bin is incr added count times in sequence, the
//           partitions folded in order -- bit for bit the reference's doubles;
//   mode 1  that buffer divided by the shell volume 4 pi / 3 (r+^3 - r-^3),
//           r- = b dr + r0, r+ = (b + 1) dr + r0 (pyanalisi/analysis.py:101-105,
//           hist2gofr);
//   mode 2  mode 1 further divided by the channel's pair density: distinct
//           pairs of types a != b: 2 N_a N_b / V, of one type: N_a (N_a - 1) / V;
//           the self channel of type a: N_a (the self part of the van Hove
//           function as a probability density).
// Every operation is an explicitly rounded FP64 intrinsic (no contraction).
// The cubes are computed in double-double arithmetic and rounded once, so
// each is the correctly rounded cube; numpy's `r ** 3` is within one unit in
// the last place of it, which bounds the difference of modes 1 and 2 from a
// host evaluation (the host states that bound with each result).
#include <algorithm>
#include <cmath>
#include <cuda_runtime.h>

#include "gofr_internal.h"

namespace gofr {

// The runs of s(k) (gofr_internal.h), each step the host's FP64 addition.
FoldTable fold_table(double incr)
{
    FoldTable t{};
    auto put = [&t](unsigned long long k, double s, double d) {
        t.k0[t.n] = k;
        t.s0[t.n] = s;
        t.delta[t.n++] = d;
    };
    const double a = std::fabs(incr);
    put(0, 0.0, a);
    unsigned long long k = 1;
    double s = a;
    // two more entries fit at the top of each pass
    while (t.n + 2 <= FOLD_RUNS) {
        const double n1 = s + a;
        if (n1 == s) {  // the sum no longer moves
            put(k, s, 0.0);
            break;
        }
        const int e = std::ilogb(s);
        const double u = std::ldexp(1.0, e - 52), top = std::ldexp(1.0, e + 1);
        const double r = a / u;  // exact (power-of-two scaling)
        const long long M = (long long)(s / u);
        const bool tie = r - std::floor(r) == 0.5;
        // additions that start where s + a stays within the binade
        const long long room = (1LL << 53) - M - (long long)std::ceil(r);
        if (room < 0 || (tie && (M & 1))) {
            put(k, s, n1 - s);  // exact: s <= n1 <= 2 s
            s = n1;
            ++k;
            continue;
        }
        const double delta = n1 - s;
        const long long j = room / (long long)(delta / u) + 1;
        put(k, s, delta);
        s = std::min(s + (double)j * delta, top);
        k += (unsigned long long)j;
    }
    for (int b = 0, i = 0; b < 64; ++b) {
        while (i + 1 < t.n && t.k0[i + 1] <= (1ull << b)) ++i;
        t.first[b] = (unsigned char)i;
    }
    if (incr < 0.0)
        for (int i = 0; i < t.n; ++i) {
            t.s0[i] = -t.s0[i];
            t.delta[i] = -t.delta[i];
        }
    return t;
}
namespace norm {

// Correctly rounded x^3: x^2 = h + l exactly (FMA), x^3 = h x + l x with the
// product h x split exactly again; one final rounding of the sum.
__device__ __forceinline__ double cube_rn(double x)
{
    const double h = __dmul_rn(x, x);
    const double l = __fma_rn(x, x, -h);
    const double p = __dmul_rn(h, x);
    const double e = __fma_rn(h, x, -p);
    return __dadd_rn(p, __dadd_rn(e, __dmul_rn(l, x)));
}

// Bound by the counts' read: every sum is a look-up of the run that holds its
// count (two or three compares from the power of two below it) and two FP64
// operations.  144,000 bins of 4 partitions: 2.23 ms when each thread stepped
// through the binades of its own count (an FP64 division and a dozen of
// operations each, on a chip with two FP64 lanes per SM), 0.012 ms from the
// table.
__global__ void __launch_bounds__(256) k_counts_to_gofr(const __grid_constant__ NormLaunch L)
{
    __shared__ FoldTable T;
    for (int i = threadIdx.x; i < (int)(sizeof(FoldTable) / 4); i += 256)
        reinterpret_cast<unsigned *>(&T)[i] = reinterpret_cast<const unsigned *>(&L.fold)[i];
    __syncthreads();
    const size_t total = (size_t)L.nwin * L.n;
    for (size_t g = blockIdx.x * (size_t)blockDim.x + threadIdx.x; g < total;
         g += (size_t)gridDim.x * blockDim.x) {
        const size_t w = g / L.n, i = g - w * L.n;
        const unsigned long long *c = L.counts + w * L.n * L.nparts + i;
        double acc = fold_sum(T, c[0]);
#pragma unroll 4
        for (int q = 1; q < L.nparts; ++q)
            acc = __dadd_rn(acc, fold_sum(T, c[(size_t)q * L.n]));
        if (L.mode >= 1) {
            const int b = (int)(i % L.nbin);
            const int ch = (int)((i / L.nbin) % L.nch);
            const double rm = __dadd_rn(__dmul_rn((double)b, L.dr), L.r0);
            const double rp = __dadd_rn(__dmul_rn((double)(b + 1), L.dr), L.r0);
            const double vol = __dmul_rn(L.c43pi, __dsub_rn(cube_rn(rp), cube_rn(rm)));
            acc = __ddiv_rn(acc, vol);
            if (L.mode == 2) acc = __ddiv_rn(acc, L.chfac[ch]);
        }
        L.out[g] = acc;
    }
}

}  // namespace norm

int launch_counts_to_gofr(const NormLaunch &L, int num_sms, cudaStream_t s)
{
    const size_t total = (size_t)L.nwin * L.n;
    if (total == 0) return 0;
    size_t blocks = (total + 255) / 256;
    if (blocks > (size_t)num_sms * 8) blocks = (size_t)num_sms * 8;
    norm::k_counts_to_gofr<<<(unsigned)blocks, 256, 0, s>>>(L);
    return cudaGetLastError() == cudaSuccess ? 0 : -1;
}

}  // namespace gofr

// Sums of many terms in a fixed order, several sums per CTA: the MI and TE
// reductions, whose terms have to be added in frame order to equal the
// reference's value.
#pragma once

#include "gc_common.cuh"

namespace gc {

constexpr int kSumThreads = 256;
constexpr int kSumTerms   = 1024; // terms of a chunk over all sums of the CTA
constexpr int kSumMost    = 32;   // most sums per CTA
static_assert(kSumTerms / kSumMost >= 32, "a warp evaluates 32 consecutive terms of a sum");

// Sums per CTA (a power of two): enough CTAs for every SM before the sums of
// a CTA grow to 32, the width of the adding warp.
inline int sums_per_cta(long sums, int sms)
{
    int p = 1;
    while (p < kSumMost && (sums + p - 1) / p > 2L * sms)
        p <<= 1;
    return p;
}

// The CTA's sums p = 0 .. P - 1 (P a power of two) over T terms each,
// term(p, f): seven warps evaluate a chunk of terms, 32 consecutive f at a
// time (so the counts behind them are read coalesced), into shared memory
// while the lanes of warp 0 add the previous chunk, each its own sum in order
// of f.  Lane p of warp 0 returns sum p.
//
// Bound by the chain of dependent FP64 additions (T of them), so a second wave
// of CTAs doubles it: chunks of 1024 terms (17 KB) let eight CTAs share an SM,
// 2048 six.  All of a KSG run but its neighbour kernels (normalisation, FP32
// copy and this), a thread per sum that fetches its own terms / chunks of 2048 /
// of 1024: 30,381 sums of 2000 terms 361 / 471 / 295 us, 11,325 of 4999 799 /
// 663 / 712, 2016 of 500 77 / 38 / 39, one of 2000 134 / 69 / 67, 124,750 of 300
// 138 / 170 / 151.
template <class Term>
__device__ __forceinline__ double ordered_sums(int P, int live, int T, Term&& term)
{
    __shared__ double buf[2][kSumTerms + kSumMost];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int logF = __ffs(kSumTerms / P) - 1, F = 1 << logF;
    const int chunks = (T + F - 1) >> logF;
    double    s      = 0.0;
    for (int c = 0; c <= chunks; ++c)
    {
        if (warp > 0 && c < chunks)
        {
            double*   b  = buf[c & 1];
            const int f0 = c << logF, n = min(F, T - f0);
#pragma unroll 5
            for (int tile = warp - 1; tile < kSumTerms / 32; tile += kSumThreads / 32 - 1)
            {
                const int p = tile >> (logF - 5), f = ((tile << 5) & (F - 1)) + lane;
                if (p < live && f < n)
                    b[p * (F + 1) + f] = term(p, f0 + f);
            }
        }
        if (warp == 0 && c > 0 && lane < live)
        {
            const double* b = buf[(c - 1) & 1] + lane * (F + 1);
            const int     n = min(F, T - (c - 1) * F);
            int           f = 0;
            for (; f + 8 <= n; f += 8)
            {
                double t[8];
#pragma unroll
                for (int u = 0; u < 8; ++u)
                    t[u] = b[f + u];
#pragma unroll
                for (int u = 0; u < 8; ++u)
                    s = __dadd_rn(s, t[u]);
            }
            for (; f < n; ++f)
                s = __dadd_rn(s, b[f]);
        }
        __syncthreads();
    }
    return s;
}

} // namespace gc

// Sorted distance rows on B200: the row sort shared by the KSG and the
// transfer-entropy fast paths (ksg_fast.cu, te_walk.cu).
#pragma once

#include <type_traits>

#include "gc_common.cuh"
#include "ksg_fast.h"

namespace gc {

// One CTA per row: a query frame's distances to every other frame, sorted
// with their frames by a counting sort over fine buckets of 2^kRowFine float
// ulps (an eighth of the walks' narrowest buckets).  kRowBins buckets end at the
// largest possible distance (8 octaves); entries below them are put in full
// order, or, if they are many, sorted again in the same way by the buckets that
// end at the largest of them.  That happens where an atom's largest distance is
// over 256 times a usual one: a broken frame, a stretch of frames in another
// periodic image.  FP32 coordinates leave no room for a fourth level but
// distances of zero.  One frame 200 nm off, by a bitonic network over the whole
// row and by levels: 80 x 4999, k = 100: 236 -> 59.6 ms for the matrix, TE
// 30 x 5000 167 -> 35.6 ms, 64 x 900 4.37 -> 2.40 ms.
// R > 0: each thread keeps its R distances (entries tid + r * threads) in
// registers; R = 0: they are recomputed (from L1-resident coordinate rows)
// for the second pass.
//
// Entries are in bucket order, those of one fine bucket (a few) in any order.
// That is all the walks need (their own buckets are whole fine ones); the
// finish and count kernels look at a value's whole fine bucket.
//
// Bound by shared memory (L1 97% busy at 247 x 2000, issue slots 68%): the
// atomics and the scatter.  The full sort it replaces (range, coarse
// distribution, histogram, scan, scatter and one thread's insertion sort per
// bucket, over eight barriers) took 10.7 ms for the rows of 247 atoms x 2000
// frames, 51.8 ms for 151 x 4999 and 289 us for 64 x 500; this one 6.55 ms, 28.2
// ms and 134 us written in single groups, 3.93, 16.3 and .099 in the runs that
// row_run gives.  Fine buckets of 2^15 ulps make it 2% faster and the finish 3%
// slower, 2^13 the rows 8% slower; putting the entries of each bucket in order as
// well costs as much as the full sort (all these in single groups).

constexpr int kRowBins  = 4096;
constexpr int kRowFine  = 14; // log2 of a fine bucket's width in float ulps
constexpr int kRowLow   = 32; // entries below the buckets that one thread sorts

// CTAs an SM should hold (the register limit of the row kernels).
constexpr int row_ctas(int threads, int regs)
{
    return threads == 1024 ? 1 : (regs == 8 || threads == 512 ? 1536 : 1280) / threads;
}

// Two 16-bit counters per word (a row has at most 16,384 entries).  Place of
// counter word w: the 16-byte vectors are permuted so that eight threads
// scanning neighbouring slices of up to 32 words by vectors hit eight
// different bank groups.
__device__ __forceinline__ int rows_word(int w) { return w ^ ((w >> 3) & 0x1C); }

// Static shared memory of sort_row: the caller's kernel declares one (so a
// kernel that sorts rows of several kinds holds it once).
template <int THREADS>
struct RowSortShared
{
    unsigned wsum[THREADS / 32];
    unsigned low;                // entries below the buckets
    unsigned wmax[THREADS / 32]; // largest of them by warp
};

// Bucket of a distance, where cb is the code of bucket 0.
__device__ __forceinline__ int rows_bin(float d, int cb)
{
    return min(max((int)(__float_as_uint(d) >> kRowFine) - cb, 0), kRowBins - 1);
}

// Counter b of the cursors: adds 1 and returns its value before.
__device__ __forceinline__ unsigned rows_bump(unsigned* cursor, int b)
{
    const int sh = (b & 1) * 16;
    return (atomicAdd(&cursor[rows_word(b >> 1)], 1u << sh) >> sh) & 0xFFFFu;
}

template <int THREADS>
__device__ __forceinline__ void rows_clear(unsigned* cursor, int tid)
{
    for (int b = tid * 4; b < kRowBins / 2; b += THREADS * 4)
        *reinterpret_cast<uint4*>(cursor + b) = make_uint4(0u, 0u, 0u, 0u);
}

// Exclusive scan of the counters in place (each thread a contiguous slice),
// with a barrier before and after.  Returns the first counter.
template <int THREADS>
__device__ __forceinline__ unsigned rows_scan(RowSortShared<THREADS>& sh, unsigned* cursor, int tid)
{
    const int     lane = tid & 31, warp = tid >> 5;
    constexpr int kSlice = kRowBins / 2 / THREADS; // words
    constexpr int kVec   = kSlice < 4 ? kSlice : 4;
    using Vec            = typename std::conditional<kVec == 4, uint4, uint2>::type;
    static_assert(kVec >= 2 && kSlice % kVec == 0, "slices by vectors");
    union Words
    {
        Vec      v;
        unsigned w[kVec];
    };
    auto slice = [cursor, tid](int v) { return reinterpret_cast<Vec*>(cursor + rows_word(tid * kSlice + v)); };
    __syncthreads();
    unsigned loc = 0;
#pragma unroll
    for (int v = 0; v < kSlice; v += kVec)
    {
        Words c;
        c.v = *slice(v);
        if (v == 0 && tid == 0)
            sh.low = c.w[0] & 0xFFFFu;
#pragma unroll
        for (int e = 0; e < kVec; ++e)
        {
            loc += (c.w[e] & 0xFFFFu) + (c.w[e] >> 16);
        }
    }
    unsigned incl = loc;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1)
    {
        const unsigned y = __shfl_up_sync(kFull, incl, o);
        if (lane >= o)
            incl += y;
    }
    if (lane == 31)
        sh.wsum[warp] = incl;
    __syncthreads();
    const unsigned low = sh.low;
    unsigned       run = incl - loc;
    for (int w = 0; w < warp; ++w)
        run += sh.wsum[w];
#pragma unroll
    for (int v = 0; v < kSlice; v += kVec)
    {
        Words c;
        c.v = *slice(v);
#pragma unroll
        for (int e = 0; e < kVec; ++e)
        {
            const unsigned n = c.w[e], mid = run + (n & 0xFFFFu);
            c.w[e]           = run | (mid << 16);
            run              = mid + (n >> 16);
        }
        *slice(v) = c.v;
    }
    __syncthreads();
    return low;
}

// blockIdx.x as a value of its own: what is computed from it is not what was
// computed before, kept in registers.
__device__ __forceinline__ long long rows_block()
{
    long long r = blockIdx.x;
    asm volatile("" : "+l"(r));
    return r;
}

// Sorts the row of query frame i over frames 0 .. N (i excluded, N entries
// in all): dist(j) gives the FP32 distance from the query to frame j, at most
// top.  The distances and frames go to S / P at base + row_entry(m, gstride,
// run_log) for entry m (the transposed layout of the walk), the last 4-entry
// group padded with NaN and frame 0.  Every thread of the CTA calls it; it
// uses the dynamic shared memory of row_sort_smem.  again() gives dist anew,
// for the further levels, so that the usual rows' registers do not carry it.
// U_row (optional) receives the unsorted distances at U_row[j].
template <int THREADS, int R, class DistFn, class AgainFn>
__device__ __forceinline__ void sort_row(RowSortShared<THREADS>& sh, int N, int i, float top, DistFn&& dist,
                                         AgainFn&& again, float* __restrict__ S, uint16_t* __restrict__ P, size_t base,
                                         size_t gstride, int run_log,
                                         float* __restrict__ U_row = nullptr)
{
    extern __shared__ __align__(16) unsigned char rows_smem[];
    const int tid = threadIdx.x;
    const int Np     = (N + 3) & ~3;                               // whole 4-entry groups
    unsigned* cursor = reinterpret_cast<unsigned*>(rows_smem);     // [kRowBins / 2]
    unsigned* vals   = cursor + kRowBins / 2;                        // [Np] distance bits in bucket order
    uint16_t* frm    = reinterpret_cast<uint16_t*>(vals + Np);     // [Np] their frames
    auto      frame_of = [i](int m) { return m < i ? m : m + 1; };
    const int cb       = (int)(__float_as_uint(top) >> kRowFine) - (kRowBins - 1); // code of bucket 0
    auto      start_of = [cursor](int b) -> unsigned { return (cursor[rows_word(b >> 1)] >> ((b & 1) * 16)) & 0xFFFFu; };
    rows_clear<THREADS>(cursor, tid);
    // the row's distances, and later each key's arrival in its bucket
    float    dreg[R > 0 ? R : 1];
    unsigned areg[R > 0 ? (R + 1) / 2 : 1] = {}; // two 16-bit numbers each
    if constexpr (R > 0)
    {
#pragma unroll
        for (int k = 0; k < R; ++k)
        {
            const int m = tid + k * THREADS;
            dreg[k]     = m < N ? dist(frame_of(m)) : 0.0f;
        }
    }
    auto each = [&](auto&& fn) {
        if constexpr (R > 0)
        {
#pragma unroll
            for (int k = 0; k < R; ++k)
            {
                const int m = tid + k * THREADS;
                if (m < N)
                    fn(k, m, dreg[k]);
            }
        }
        else
        {
            for (int m = tid; m < N; m += THREADS)
                fn(0, m, dist(frame_of(m)));
        }
    };
    // optional unsorted copy of the row, indexed by frame (the query's own
    // frame is left unwritten: no walk reads it)
    if (U_row)
        each([&](int, int m, float d) { U_row[frame_of(m)] = d; });
    __syncthreads();
    each([&](int k, int, float d) {
        const unsigned o = rows_bump(cursor, rows_bin(d, cb));
        if constexpr (R > 0)
        {
            if (k & 1)
                areg[k >> 1] |= o << 16;
            else
                areg[k >> 1] = o;
        }
    });
    unsigned low = rows_scan<THREADS>(sh, cursor, tid);
    each([&](int k, int m, float d) {
        unsigned at;
        if constexpr (R > 0)
            at = start_of(rows_bin(d, cb)) + ((areg[k >> 1] >> ((k & 1) * 16)) & 0xFFFFu);
        else
            at = rows_bump(cursor, rows_bin(d, cb));
        vals[at] = __float_as_uint(d);
        frm[at]  = (uint16_t)frame_of(m);
    });
    if (tid < Np - N)
    {
        vals[N + tid] = 0x7fc00000u;
        frm[N + tid]  = 0;
    }
    __syncthreads();
    // Further levels: the entries in bucket 0 or below it, which lie in the
    // row's first places, go there again by the buckets that end at the largest
    // of them (their distances recomputed: the first level's registers are free).
#pragma unroll 1
    while (low > (unsigned)kRowLow)
    {
        int t = tid;
        asm volatile("" : "+r"(t)); // its addresses are not the first level's, kept in registers
        unsigned most = 0;
#pragma unroll 1
        for (unsigned e = t; e < low; e += THREADS)
            most = max(most, vals[e]);
        most = __reduce_max_sync(kFull, most);
        if ((t & 31) == 0)
            sh.wmax[t >> 5] = most;
        rows_clear<THREADS>(cursor, t);
        __syncthreads();
#pragma unroll 1
        for (int w = 0; w < THREADS / 32; ++w)
            most = max(most, sh.wmax[w]);
        const int  at0  = (int)(most >> kRowFine) - (kRowBins - 1);
        const auto same = again();
        auto       here = [&](auto&& fn) {
#pragma unroll 1
            for (int m = t; m < N; m += THREADS)
            {
                const int   j = frame_of(m);
                const float d = same(j);
                if (__float_as_uint(d) <= most)
                    fn(j, d);
            }
        };
        here([&](int, float d) { rows_bump(cursor, rows_bin(d, at0)); });
        low = rows_scan<THREADS>(sh, cursor, t);
        here([&](int j, float d) {
            const unsigned at = rows_bump(cursor, rows_bin(d, at0));
            vals[at]          = __float_as_uint(d);
            frm[at]           = (uint16_t)j;
        });
        __syncthreads();
    }
    if (tid == 0) // the entries below the buckets, by insertion
        for (unsigned x = 1; x < low; ++x)
        {
            const unsigned v = vals[x];
            const uint16_t f = frm[x];
            unsigned       y = x;
            for (; y > 0 && vals[y - 1] > v; --y)
            {
                vals[y] = vals[y - 1];
                frm[y]  = frm[y - 1];
            }
            vals[y] = v;
            frm[y]  = f;
        }
    __syncthreads();
    // transposed layout: one thread per group of 4 consecutive entries, the
    // queries of a block side by side (see WalkParams).  The last group runs
    // out in NaN (never <= any stop value) with frame 0, so the walk reads
    // whole groups without a bounds test.
    for (int g = tid; g * 4 < N; g += THREADS)
    {
        const size_t at                  = base + row_entry(g * 4, gstride, run_log);
        *reinterpret_cast<uint4*>(S + at) = *reinterpret_cast<const uint4*>(vals + g * 4);
        *reinterpret_cast<uint2*>(P + at) = *reinterpret_cast<const uint2*>(frm + g * 4);
    }
}

// The first value of a's fine bucket, and of the next one (a >= 0).
__device__ __forceinline__ float fine_start(float a) { return __uint_as_float(__float_as_uint(a) >> kRowFine << kRowFine); }
__device__ __forceinline__ float fine_after(float a)
{
    return __uint_as_float(((__float_as_uint(a) >> kRowFine) + 1u) << kRowFine);
}

// Upper bound of an atom's distances from its FP32 error bound: 2 R, eps >= R 2^-21.
__device__ __forceinline__ float row_top(float eps_atom) { return eps_atom * 4194304.0f * 1.0001f; }

// Shared memory of one row of N entries; *threads and *regs pick the sort_row
// instantiation (threads per row, distances per thread kept in registers).
// The passes are short, so what counts is how little a barrier holds up:
// few threads a row, many rows an SM.  In single groups, 64 x 500: 209 us by 256 threads, 169
// by 256 with 4 distances, 142 by 128, 134 by 64; 247 x 2000: 6.78 ms by 256,
// 6.55 by 128; 150 x 3000: 11.2 ms by 512, 9.7 by 256; 151 x 4999: 29.8 ms by
// 512 (two rows an SM), 28.2 (three), 30.3 by 256 with 32 distances.
inline size_t row_sort_smem(int N, int* threads, int* regs)
{
    *threads = N <= 8 * 64 ? 64 : (N <= 16 * 128 ? 128 : (N <= 16 * 256 ? 256 : (N <= 16 * 512 ? 512 : 1024)));
    *regs    = N <= 8 * 128 ? 8 : (N <= 16 * 512 ? 16 : 0);
    return (size_t)kRowBins * 2 + (((size_t)N + 3) & ~(size_t)3) * 6;
}

} // namespace gc

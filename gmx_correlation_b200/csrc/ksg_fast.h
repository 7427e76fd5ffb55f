// Parameters of the KSG fast-path kernels (host and device).
#pragma once

#include <cstdint>
#include <cuda_runtime.h>

namespace gc {

constexpr int kWalkWarps   = 32;       // most warps per walk CTA
#ifndef GC_FINISH_WARPS
#define GC_FINISH_WARPS 25 // a build-time setting for timing other finish CTA shapes
#endif
// Warps per finish CTA.  The finish gathers coordinates through L1, which has
// what the band entries leave of an SM's 256 KB.  20 warps with 14-byte
// entries leave about 60 KB: 30.6 ms at 247 x 2000 k=100 and 44.1 at 151 x
// 4999 (24 such warps leave 28 KB: 43.8 and 68.7 ms); with 10-byte entries 20
// warps take 29.4 and 41.2 ms, 24 28.1 and 39.4, 25 (72 registers, 136 bytes
// spilled) 27.4 and 38.7; with the rows in runs (row_run) 27.0 and 36.5.
constexpr int kFinishWarps = GC_FINISH_WARPS;
constexpr int kWalkBuckets = 128;      // per-lane histogram buckets
#ifndef GC_BAND_CAP
#define GC_BAND_CAP 20 // a build-time setting for timing other capacities
#endif
constexpr int kRwChunk     = 128;       // row walk: row entries staged at a time
constexpr int kRwHistBytes  = kWalkBuckets * 32; // row walk: a warp's histogram
constexpr int kRwStageBytes = kRwChunk * 5;      // row walk: a warp's staged entries
constexpr int kRwMaxOffset  = 128; // row walk: largest window offset the 256 codes of a tile cover
constexpr int kRwMaxAtoms   = 4096; // row walk: atoms the per-query ordering takes
// Row walk: bytes of the code tile of T frames.
__host__ __device__ inline size_t rw_tile_bytes(int T) { return ((size_t)T * 32 + 127) & ~(size_t)127; }
constexpr int kBandCap     = GC_BAND_CAP; // band entries kept per lane
constexpr int kBandSlotBytes = 10;     // joint and smaller marginal value (f32), row position in its range (u16)
constexpr uint32_t kHandOver = 0xFFFFFFFFu; // cnt value of a query handed to the exact kernel

// Rows are stored in runs of 2^run 4-entry groups, the runs of a block's queries
// side by side.  Place of entry m / of group g in a row; stride: elements /
// groups from one of its runs to the next.
__host__ __device__ inline size_t row_entry(int m, size_t stride, int run)
{
    return (size_t)(m >> (2 + run)) * stride + (m & ((4 << run) - 1));
}
__host__ __device__ inline size_t row_group(int g, size_t stride, int run)
{
    return (size_t)(g >> run) * stride + (g & ((1 << run) - 1));
}
// The run of a launch's rows.  A walk with one query per lane reads the same
// group of 32 queries at once: single groups.  The row sort writes a row and the
// row walk reads it from one CTA or warp, where single groups are a cache line
// each: 247 x 2000: 55.2 ms with single groups, 51.7 / 50.3 / 49.9 with runs of
// 2 / 4 / 8; 151 x 4999: 111.7, 101.1 / 96.8 / 95.2; TE 247 x 2000: 150.4, 144.3
// / 140.6 / 140.2.  Short rows end in the finish, whose lanes read neighbouring
// queries: 64 x 500: 700 us, 664 / 651 / 661; TE 40 x 700: finish 316, 340 / 343 /
// 363 us.  A pair list at 247 x 2000: lane walk 2.3 ms, 2.6 / 3.2 / 4.1.
// With up to 24 pairs an atom (pair lists, few atoms) the rows outweigh the lane
// walk: runs of 2.  16 atoms x 2000: 1.14 -> 1.03 ms, 8 x 5000: 2.38 -> 1.94, 23 x
// 500 218 -> 204 us, TE 22 x 2000 4.35 -> 4.06 ms; 1,519 pairs of 247 x 2000 save
// 1.7 ms of rows and finish for .3 ms of walk, so about 40 pairs an atom break even.
inline int row_run(bool row_walk, int maxLen, long long pairs, int natoms)
{
    if (!row_walk)
        return pairs <= 24LL * natoms ? 1 : 0;
    return maxLen > 1024 ? 3 : 2;
}

// Sorted marginal rows of one query block, transposed so that the 32
// queries of a warp read neighbouring addresses: entry m of the row of
// (atom a, query i0 + iq) is element (a * Lq * Qp + (iq << run)) * 4 +
// row_entry(m, (Qp * 4) << run, run) of S (distances) and of P (frames),
// Lq = Lpad / 4 (a multiple of 8).
struct WalkParams
{
    const float4*   X32;      // [natoms][T] centred FP32 coordinates
    const double*   X64;      // [3*natoms][T] normalised rows (reference arithmetic)
    const float*    eps_atom; // [natoms] |d32 - d64| bound
    float*          S;
    uint16_t*       P;
    int             natoms, Lpad, Qp, i0, Q, T, K, box, rank_shift;
    int             run; // row_run of the launch
    long            pair_begin, pair_count;
    const int2*     pair_ab;    // optional [pair_count] (a1, a2) of an explicit pair list
    const int*      pair_order; // optional task order: task k computes local pair pair_order[k]
    int             shift;      // histogram bucket = 2^shift float ulps above the lower bound
    uint32_t*       cnt;        // [pair_count][T] n_x | n_y << 16, or kHandOver
    unsigned long long* wres;   // [pair_count][Q] walk results of the block (a warp's 32 queries side by side)
    unsigned long long* hq;     // hand-over queue: cnt indices pl * T + i
    unsigned*           hq_len;
    unsigned            hq_cap;
    int*                status;
    unsigned long long* walk_elems; // optional: total walked row entries
    unsigned*           reasons;    // optional [8]: hand-overs by cause
    // optional unsorted distance rows of the block: the distance from query
    // i0 + iq of atom a to frame j at U[((size_t)a * Qp + iq) * Tpad + j]
    // (GC_VARIANT_HBM_GATHER: the walk reads the other marginal here)
    float* U;
    int    Tpad;
    // full pair matrices walked row by row (row_walk.cuh): the block's atoms
    // by ascending k-th distance, [Q][natoms] (atom, code of that distance);
    // null where the walk with one query per lane runs
    uint2* order;
};

// One launch over the query blocks of several trajectories (or of one): the
// launch's tasks are numbered across the descriptors, descriptor d owning
// tasks [prefix[d], prefix[d + 1]).  Every array lives in device memory.
struct WalkBatch
{
    const WalkParams*   d;       // [n]
    const long long*    rprefix; // [n + 1] row-sort tasks: natoms * Q per descriptor
    const long long*    wprefix; // [n + 1] walk tasks: ceil(groups / chunk) * pairs
    const long long*    fprefix; // [n + 1] finish tasks: query groups * pairs
    const long long*    qprefix; // [n + 1] queries (row walk only)
    const long long*    uprefix; // [n + 1] row-walk tasks: Q * ceil(natoms / 32)
    int                 n;
    int                 maxT;    // largest frame count (shared-memory layout)
    int                 maxK;    // largest k
    int                 chunk;   // query groups per walk task (shared by the CTA's warps)
    unsigned long long* counter; // [2] walk and finish task counters, zero at launch
};

// Bucket width of the walk histogram for k: about 0.33/k of the value (two or
// three entries per bucket near the k-th value), between 2^17 ulps, so that
// the 128 buckets span two octaves above the lower bound, and 2^21.  Four
// times wider buckets, eight entries each, make the finish kernels enumerate
// that many more: 64 x 500, k = 10: finish 552 -> 405 us, hand-overs 163 ->
// 0; 150 x 4000, k = 10: 54.7 -> 33.1 ms; TE 40 x 700, k = 10: 705 -> 348 us.
// Half the width again (2^17 ulps already at k = 10) gains 5-10% of the
// finish and loses it in the walk; 2^16 ulps span one octave: 4% of the
// queries at 100 x 4999, k = 100 lie beyond and the matrix takes 311 ms for 82.
inline int walk_histogram_shift(int K)
{
    const double target = 22.0 + __builtin_log2(0.67 / (double)K);
    int          s      = (int)(target + 0.5);
    return s < 17 ? 17 : (s > 21 ? 21 : s);
}

// Walk launch shape for trajectories of up to maxT frames: warps per CTA and
// whether the pair's coordinate rows are staged in shared memory.
void walk_shape(int maxT, int* warps, bool* staged);
// Largest walk warps per CTA that the staged layout allows (0: not staged).
int walk_max_staged_warps(int maxT);

// Each launcher returns the launch status (cudaGetLastError right after it).
cudaError_t launch_ksg_x32(const double* X64, int natoms, int T, float4* X32, float* eps_atom, cudaStream_t s);
cudaError_t launch_ksg_rows(const WalkBatch& b, long long rows, cudaStream_t s);
// gather_u: the other marginal's distances come from the descriptors' U rows;
// double_buffer: the double-buffered walk (two staged tasks per CTA).
cudaError_t launch_ksg_walk(const WalkBatch& b, int warps, bool staged, int sms, cudaStream_t s,
                            bool gather_u = false, bool double_buffer = false);
// Warps per CTA the double-buffered walk leaves room for (0: its rows do not fit).
int walk_max_db_warps(int maxT);
// The row walk (row_walk.cuh) of descriptors with an order array; queries:
// qprefix[n], maxn: the most atoms of a descriptor.
cudaError_t launch_ksg_row_walk(const WalkBatch& b, long long queries, int maxn, int sms, cudaStream_t s);
// Warps per CTA of the row walk (0: the tile of maxT frames does not fit) and CTAs per SM.
int row_walk_warps(int maxT, int* ctas);
cudaError_t launch_ksg_finish(const WalkBatch& b, int sms, cudaStream_t s);
// Exact FP64 statistics for every queued hand-over of the batch's
// descriptors, then for any hand-over mark a queue could not hold (a scan of
// cnt).  One descriptor per trajectory.
cudaError_t launch_ksg_fixup(const WalkBatch& b, int sms, cudaStream_t s);

} // namespace gc

// KSG walk with one sorted row for 32 pairs (see row_walk.cuh): the walk of
// full pair matrices whose code tile fits in shared memory.
//
//   ksg_order_kernel     per query: the atoms in ascending order of their
//                        k-th marginal distance.
//   ksg_row_walk_kernel  one CTA task per (query, block of 32 atoms in that
//                        order): the block's bucket codes of every frame in
//                        a shared-memory tile, then one warp per atom a above
//                        the block walks a's row for the pairs with the
//                        block's atoms below a.  Every pair is walked on the
//                        row of its atom with the larger k-th distance, an
//                        exact lower bound of the joint k-th distance.
//
// Replaces, for these shapes, the walk with one query per lane (ksg_fast.cu),
// which stays for pair lists and shards, few atoms, k >= 256 and rows whose
// tile does not fit.

#include "gc_common.cuh"
#include "gc_internal.h"
#include "ksg_fast.h"
#include "ksg_device.cuh"
#include "row_walk.cuh"

namespace gc {

constexpr int kOrderThreads = 256;
constexpr int kRwAhead      = 8; // frames of a tile column a lane loads together

// One CTA per (descriptor, query of its block): rank of every atom by its
// k-th marginal distance (ties by atom), and the code of that distance.
__global__ void __launch_bounds__(kOrderThreads) ksg_order_kernel(WalkBatch B)
{
    extern __shared__ unsigned kth[]; // [natoms] distance bits
    const long long   r  = blockIdx.x;
    const int         d  = batch_desc(B.qprefix, B.n, r);
    const WalkParams& p  = B.d[d];
    const int         iq = (int)(r - B.qprefix[d]), n = p.natoms;
    for (int a = threadIdx.x; a < n; a += kOrderThreads)
        kth[a] = __float_as_uint(lane_row(p, a, iq).s(p.K - 1));
    __syncthreads();
    uint2* ord = p.order + (size_t)iq * n;
    for (int a = threadIdx.x; a < n; a += kOrderThreads)
    {
        const unsigned v  = kth[a];
        int            rk = 0;
        for (int b = 0; b < n; ++b)
        {
            const unsigned u = kth[b];
            rk += u < v || (u == v && b < a);
        }
        ord[rk] = make_uint2((unsigned)a, v >> p.shift);
    }
}

__global__ void __launch_bounds__(1024, 1) ksg_row_walk_kernel(WalkBatch B)
{
    extern __shared__ __align__(128) unsigned char smem_raw[];
    __shared__ long long s_task;
    __shared__ int       s_next;
    const int      warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nwarps = blockDim.x >> 5;
    unsigned char* tile  = smem_raw;
    unsigned char* hist  = smem_raw + rw_tile_bytes(B.maxT) + (size_t)warp * (kRwHistBytes + kRwStageBytes);
    unsigned char* stage = hist + kRwHistBytes;
    const long long total = B.uprefix[B.n];
    for (;;)
    {
        __syncthreads(); // the previous task's tile and counters are done with
        if (threadIdx.x == 0)
            s_task = (long long)atomicAdd(B.counter, 1ull);
        __syncthreads();
        const long long t = s_task;
        if (t >= total)
            break;
        const int         dsc = batch_desc(B.uprefix, B.n, t);
        const WalkParams& p   = B.d[dsc];
        const int         n = p.natoms, T = p.T, shift = p.shift, nblk = (n + 31) >> 5;
        const long long   lt = t - B.uprefix[dsc];
        const int         iq = (int)(lt / nblk), b0 = (int)(lt - (long long)iq * nblk) * 32;
        const int         i   = p.i0 + iq;
        const uint2*      ord = p.order + (size_t)iq * n;
        const int         pb  = b0 + lane;
        const int         b   = pb < n ? (int)ord[pb].x : 0;
        // rows of the atoms above the block's first, in phases whose windows
        // all fit the tile's 256 codes
        for (int pa0 = b0 + 1; pa0 < n;)
        {
            const int base = (int)ord[pa0].y - 1;
            int       pa1  = pa0; // first atom above whose window no longer fits
            {
                int lo = pa0, hi = n;
                while (lo < hi)
                {
                    const int mid = (lo + hi) >> 1;
                    if ((int)ord[mid].y - 1 - base <= kRwMaxOffset)
                        lo = mid + 1;
                    else
                        hi = mid;
                }
                pa1 = lo;
            }
            if (threadIdx.x == 0)
                s_next = pa0;
            rw_fill(min(32, n - b0), T, kRwAhead, warp, nwarps, [&](int c, int j0) {
                const float4* xr = p.X32 + (size_t)ord[b0 + c].x * T;
                const float4  q  = xr[i];
                float4        v[kRwAhead];
#pragma unroll
                for (int e = 0; e < kRwAhead; ++e)
                    v[e] = xr[min(j0 + e * 32 + lane, T - 1)];
#pragma unroll
                for (int e = 0; e < kRwAhead; ++e)
                {
                    const int j = j0 + e * 32 + lane;
                    if (j < T)
                        tile[rw_row((unsigned)j) ^ (unsigned)c] = rw_code(dist3f(q, v[e]), shift, base);
                }
            });
            __syncthreads();
            for (;;)
            {
                int pa = 0;
                if (lane == 0)
                    pa = atomicAdd(&s_next, 1);
                pa = __shfl_sync(kFull, pa, 0);
                if (pa >= pa1)
                    break;
                const int       a    = (int)ord[pa].x, w0 = (int)ord[pa].y;
                const bool      live = pb < pa;
                const LaneRow   row  = lane_row(p, a, iq);
                const RwBracket r    = rw_walk(tile, reinterpret_cast<const float4*>(row.S),
                                               reinterpret_cast<const uint2*>(row.P), row.gstride >> 2, row.run, T - 1, p.K, shift, w0,
                                               w0 - 1 - base, live, hist, stage, lane);
                if (live)
                {
                    const int  a1 = max(a, b), a2 = min(a, b);
                    const long pl = (long)a1 * (a1 - 1) / 2 + a2;
                    // index 0 holds fewer than k entries, so the k-th value lies
                    // above it unless the input is not finite
                    const int reason = (r.wrapped || r.lev == 0) ? kReasonBand
                                       : (r.lev >= kWalkBuckets - 1 ? kReasonRange : 0);
                    p.wres[(size_t)pl * p.Q + iq] = pack_walk(r.lev - 1, r.below, r.walked, reason);
                }
                if (p.walk_elems)
                {
                    const unsigned we = __reduce_add_sync(kFull, live ? (unsigned)r.walked : 0u);
                    if (lane == 0)
                        atomicAdd(p.walk_elems, (unsigned long long)we);
                }
                __syncwarp(); // the histogram and the stage are free for the next row
            }
            __syncthreads(); // the tile may be rebuilt
            pa0 = pa1;
        }
    }
}

int row_walk_warps(int maxT, int* ctas)
{
    const size_t tile = rw_tile_bytes(maxT), warp = kRwHistBytes + kRwStageBytes, all = kMaxDynamicSmem;
    *ctas             = 1;
    if (tile + 8 * warp > all)
        return 0;
    // two CTAs an SM (one builds its tile while the other walks) where each
    // gets 16 warps, else one of up to 32: at 2000 frames one CTA of 32 warps
    // takes 20.4 ms for 247 atoms, two of 10 warps 22.1 ms
    const size_t half = all / 2 - 1024;
    if (tile + 16 * warp <= half)
    {
        *ctas = 2;
        return 16;
    }
    const size_t w = (all - tile) / warp;
    return (int)(w > 32 ? 32 : w);
}

cudaError_t launch_ksg_row_walk(const WalkBatch& b, long long queries, int maxn, int sms, cudaStream_t s)
{
    if (queries <= 0)
        return cudaSuccess;
    ksg_order_kernel<<<(unsigned)queries, kOrderThreads, sizeof(unsigned) * (size_t)maxn, s>>>(b);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess)
        return e;
    int          ctas  = 1;
    const int    warps = row_walk_warps(b.maxT, &ctas);
    const size_t smem  = rw_tile_bytes(b.maxT) + (size_t)warps * (kRwHistBytes + kRwStageBytes);
    e = allow_dynamic_smem(ksg_row_walk_kernel);
    if (e != cudaSuccess)
        return e;
    ksg_row_walk_kernel<<<sms * ctas, warps * 32, smem, s>>>(b);
    return cudaGetLastError();
}

} // namespace gc

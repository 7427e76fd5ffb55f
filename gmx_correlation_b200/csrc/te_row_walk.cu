// Transfer-entropy walk and count with one sorted row for 32 pairs (see
// row_walk.cuh): for full ordered-pair matrices whose code tile fits in
// shared memory.
//
//   te_order_kernel     per query: the atoms in ascending order of the k-th
//                       value of their G row, and of their M row.
//   te_row_walk_kernel  the joint values max(G, Y) of an ordered pair (target
//                       a1, source a2) are walked on the row with the larger
//                       k-th value: G rows for 32 sources at a time (the tile
//                       holds their 3-D distance codes), M rows for 32
//                       targets (their 6-D codes).
//   te_row_count_kernel n_ypxp = #{j : max(D1, D2) < eps}.  Both marginals are
//                       3-D, so one walk of an atom's M row counts for both
//                       ordered pairs of 32 atom pairs: a frame whose code (16
//                       bits here, so that few frames share eps's bucket) is
//                       below eps's is counted, one in eps's own bucket is
//                       listed and settled from its FP32 distance, or in FP64
//                       within the error bound.
//
// Replaces, for these shapes, the walk and the count with one query per lane
// (te_walk.cu), which gather 12 to 32 bytes of coordinates from a different
// frame in every lane for each row entry.

#include "gc_common.cuh"
#include "gc_internal.h"
#include "ksg_fast.h"
#include "row_sort.cuh"
#include "row_walk.cuh"
#include "te_device.cuh"
#include "te_walk.h"

namespace gc {

constexpr int kTeOrderThreads = 256;

// One CTA per (descriptor, query of its block).
__global__ void __launch_bounds__(kTeOrderThreads) te_order_kernel(TeBatch B)
{
    extern __shared__ unsigned kth[]; // [natoms] value bits
    const long long r  = blockIdx.x;
    const int       d  = te_desc_of(B.qprefix, B.n, r);
    const TeParams& p  = B.d[d];
    const int       iq = (int)(r - B.qprefix[d]), n = p.natoms;
    for (int side = 0; side < 2; ++side)
    {
        __syncthreads(); // the first side's values are consumed
        for (int a = threadIdx.x; a < n; a += kTeOrderThreads)
            kth[a] = __float_as_uint(side == 0 ? te_row(p.SG, p.PG, p, a, iq).s(p.K - 1)
                                               : te_row(p.SM, p.PM, p, a, iq).s(p.K - 1));
        __syncthreads();
        uint2* ord = (side == 0 ? p.orderG : p.orderM) + (size_t)iq * n;
        for (int a = threadIdx.x; a < n; a += kTeOrderThreads)
        {
            const unsigned v  = kth[a];
            int            rk = 0;
            for (int b = 0; b < n; ++b)
            {
                const unsigned u = kth[b];
                rk += u < v || (u == v && b < a);
            }
            ord[rk] = make_uint2((unsigned)a, v);
        }
    }
}

namespace {

// First position of an order with a k-th value of at least v (above v: strict).
__device__ __forceinline__ int te_first(const uint2* ord, int lo, int n, unsigned v, bool strict)
{
    int hi = n;
    while (lo < hi)
    {
        const int mid = (lo + hi) >> 1;
        if (strict ? ord[mid].y <= v : ord[mid].y < v)
            lo = mid + 1;
        else
            hi = mid;
    }
    return lo;
}

__device__ __forceinline__ long te_pair_index(int a1, int a2, int n)
{
    return (long)a1 * (n - 1) + (a2 < a1 ? a2 : a2 - 1);
}

// Fills the tile's columns c0 .. c0 + 31 of an order with bucket codes
// relative to base: G distances (6-D) or M distances (3-D) of query qi.
__device__ __forceinline__ void te_tile(const TeParams& p, const uint2* ord, int c0, int qi, bool g, int base,
                                        unsigned char* tile, int warp, int nwarps, int lane)
{
    const int lag = p.lag, Nv = p.Nv, shift = p.shift;
    for (int c = warp; c < 32 && c0 + c < p.natoms; c += nwarps)
    {
        const float4* x = p.X32 + (size_t)ord[c0 + c].x * p.T;
        const float4  q = x[qi], f = x[qi + lag];
        for (int j = lane; j < Nv; j += 32)
        {
            float d = te3(q, x[j]);
            if (g)
                d = fmaxf(te3(f, x[j + lag]), d);
            tile[rw_row((unsigned)j) ^ (unsigned)c] = rw_code(d, shift, base);
        }
    }
}

// The count's 16-bit codes: 2^13 float ulps wide (a tenth of a percent: one
// or two frames of a pair share eps's bucket), relative to the base.
constexpr int kTeCountShift = 13;
constexpr int kTeAhead      = 8; // frames of a tile column a lane loads together
__device__ __forceinline__ int te_code16(float d, int base)
{
    return min(max((int)(__float_as_uint(d) >> kTeCountShift) - base, 0), 65535);
}

// Byte offset of frame j's row of the count's tile (64 bytes); lane l's code
// at (offset ^ 2 l), permuted as rw_row so that a warp filling a column for 32
// consecutive frames hits 32 different banks.
__device__ __forceinline__ unsigned te_row16(unsigned j) { return (j << 6) | ((j & 0x1Eu) << 1); }

} // namespace

__global__ void __launch_bounds__(1024, 1) te_row_walk_kernel(TeBatch B)
{
    extern __shared__ __align__(128) unsigned char smem_raw[];
    __shared__ long long s_task;
    __shared__ int       s_next;
    const int      warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nwarps = blockDim.x >> 5;
    unsigned char* tile  = smem_raw;
    unsigned char* hist  = smem_raw + rw_tile_bytes(B.maxNv) + (size_t)warp * (kRwHistBytes + kRwStageBytes);
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
        const int       dsc = te_desc_of(B.uprefix, B.n, t);
        const TeParams& p   = B.d[dsc];
        const int       n = p.natoms, nblk = (n + 31) >> 5, shift = p.shift;
        const long long lt = t - B.uprefix[dsc];
        const int       iq = (int)(lt / (2 * nblk)), sub = (int)(lt - (long long)iq * 2 * nblk);
        // G rows for blocks of sources, then M rows for blocks of targets
        const bool   wg   = sub < nblk;
        const int    c0   = (wg ? sub : sub - nblk) * 32;
        const uint2* rows = (wg ? p.orderG : p.orderM) + (size_t)iq * n;
        const uint2* cols = (wg ? p.orderM : p.orderG) + (size_t)iq * n;
        const bool   col  = c0 + lane < n;
        const uint2  oc   = col ? cols[c0 + lane] : make_uint2(0u, 0u);
        // a pair walks the G row when its k-th value is at least the M row's
        for (int pa0 = te_first(rows, 0, n, cols[c0].y, !wg); pa0 < n;)
        {
            const int base = (int)(rows[pa0].y >> shift) - 1;
            // first row above whose window no longer fits the tile's 256 codes
            const int pa1 = te_first(rows, pa0, n, (unsigned)(base + 2 + kRwMaxOffset) << shift, false);
            if (threadIdx.x == 0)
                s_next = pa0;
            te_tile(p, cols, c0, p.i0 + iq, !wg, base, tile, warp, nwarps, lane);
            __syncthreads();
            for (;;)
            {
                int pa = 0;
                if (lane == 0)
                    pa = atomicAdd(&s_next, 1);
                pa = __shfl_sync(kFull, pa, 0);
                if (pa >= pa1)
                    break;
                const uint2 oa = rows[pa];
                const int   w0 = (int)(oa.y >> shift);
                const bool  live = col && oc.x != oa.x && (wg ? oc.y <= oa.y : oc.y < oa.y);
                if (!__any_sync(kFull, live))
                    continue;
                const TeRow row = wg ? te_row(p.SG, p.PG, p, (int)oa.x, iq) : te_row(p.SM, p.PM, p, (int)oa.x, iq);
                const RwBracket r = rw_walk(tile, reinterpret_cast<const float4*>(row.S),
                                            reinterpret_cast<const uint2*>(row.P), row.gstride >> 2, row.run, p.Nv - 1, p.K, shift,
                                            w0, w0 - 1 - base, live, hist, stage, lane);
                if (live)
                {
                    const long q = wg ? te_pair_index((int)oa.x, (int)oc.x, n) : te_pair_index((int)oc.x, (int)oa.x, n);
                    // window index 0 holds fewer than k entries, so the k-th value
                    // lies above it unless the input is not finite
                    const int reason = (r.wrapped || r.lev == 0) ? kTeReasonBand
                                       : (r.lev >= kWalkBuckets - 1 ? kTeReasonRange : 0);
                    p.wres[(size_t)q * p.Q + iq] = te_pack_walk(r.lev - 1, r.below, p.Nv - 1, reason);
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

namespace {

constexpr int kTeListCap = 16; // listed frames per lane
constexpr int kTeCountStage = kRwChunk * 6; // row offsets and codes of the staged entries
constexpr int kTeCountWarpBytes = kTeCountStage + kTeListCap * 64;

// One ordered pair of a lane in the count: eps, its bounds and codes.
struct TeCut
{
    bool   on;
    double eps;
    float  tlo, thi; // FP32 values below tlo are below eps, those above thi are not
    int    lo, hi;   // codes relative to the tile's base: below lo counted, lo .. hi listed
};

__device__ __forceinline__ TeCut te_cut(const TeParams& p, long q, int iq, bool live, float e, int base)
{
    TeCut c{};
    c.lo = 0;
    c.hi = -1;
    if (!live || p.cnt[(size_t)q * p.Nv + p.i0 + iq].x == kTeHandOver)
        return c;
    c.on  = true;
    c.eps = __longlong_as_double((long long)p.wres[(size_t)q * p.Q + iq]);
    c.tlo = __double2float_rd(__dsub_rd(c.eps, (double)e));
    c.thi = __double2float_ru(__dadd_ru(c.eps, (double)e));
    c.lo  = (int)(__float_as_uint(fmaxf(c.tlo, 0.0f)) >> kTeCountShift) - base;
    c.hi  = (int)(__float_as_uint(c.thi) >> kTeCountShift) - base;
    return c;
}

} // namespace

__global__ void __launch_bounds__(1024, 1) te_row_count_kernel(TeBatch B)
{
    extern __shared__ __align__(128) unsigned char smem_raw[];
    __shared__ long long s_task;
    __shared__ int       s_next;
    const int      warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nwarps = blockDim.x >> 5;
    unsigned char* tile  = smem_raw;
    unsigned char* stage = smem_raw + 2 * rw_tile_bytes(B.maxNv) + (size_t)warp * kTeCountWarpBytes;
    uint4*         so    = reinterpret_cast<uint4*>(stage);                // [32] row offsets of 4 entries
    uint2*         sc    = reinterpret_cast<uint2*>(stage + kRwChunk * 4); // [32] codes of 4 entries
    uint16_t*      list  = reinterpret_cast<uint16_t*>(stage + kTeCountStage) + lane; // [kTeListCap] of this lane
    const long long total = B.vprefix[B.n];
    const float     nan   = __int_as_float(0x7fc00000);
    for (;;)
    {
        __syncthreads(); // the previous task's tile and counters are done with
        if (threadIdx.x == 0)
            s_task = (long long)atomicAdd(B.counter, 1ull);
        __syncthreads();
        const long long t = s_task;
        if (t >= total)
            break;
        const int       dsc = te_desc_of(B.vprefix, B.n, t);
        const TeParams& p   = B.d[dsc];
        const int       n = p.natoms, nblk = (n + 31) >> 5, Nv = p.Nv, Llen = Nv - 1, T = p.T;
        const long long lt = t - B.vprefix[dsc];
        const int       iq = (int)(lt / nblk), c0 = (int)(lt - (long long)iq * nblk) * 32, qi = p.i0 + iq;
        const uint2*    ord = p.orderM + (size_t)iq * n;
        const int       b   = c0 + lane < n ? (int)ord[c0 + lane].x : 0;
        const float4*   xb  = p.X32 + (size_t)b * T;
        const float     eb  = p.eps_atom[b];
        if (c0 + 1 >= n) // the last block's only atom: no pair
            continue;
        // every pair on the row of its atom later in the order; codes from the
        // block's smallest k-th distance on (eps is at least that)
        // (rows are in fine-bucket order, so from that distance's fine bucket on)
        const int base = (int)(ord[c0].y >> kRowFine << (kRowFine - kTeCountShift)) - 1;
        if (threadIdx.x == 0)
            s_next = c0 + 1;
        rw_fill(min(32, n - c0), Nv, kTeAhead, warp, nwarps, [&](int c, int j0) {
            const float4* x = p.X32 + (size_t)ord[c0 + c].x * T;
            const float4  q = x[qi];
            float         d[kTeAhead];
#pragma unroll
            for (int e = 0; e < kTeAhead; ++e)
                d[e] = te3(q, x[min(j0 + e * 32 + lane, Nv - 1)]);
#pragma unroll
            for (int e = 0; e < kTeAhead; ++e)
            {
                const int j = j0 + e * 32 + lane;
                if (j < Nv)
                    *reinterpret_cast<uint16_t*>(tile + (te_row16((unsigned)j) ^ (unsigned)(2 * c))) =
                        (uint16_t)te_code16(d[e], base);
            }
        });
        __syncthreads();
        const unsigned lane2 = (unsigned)lane * 2u;
        for (;;)
        {
            int pa = 0;
            if (lane == 0)
                pa = atomicAdd(&s_next, 1);
            pa = __shfl_sync(kFull, pa, 0);
            if (pa >= n)
                break;
            const int   a    = (int)ord[pa].x;
            const bool  live = c0 + lane < pa; // pa < n
            const float e    = fmaxf(p.eps_atom[a], eb);
            const long  q1 = live ? te_pair_index(a, b, n) : 0, q2 = live ? te_pair_index(b, a, n) : 0;
            const TeCut k1 = te_cut(p, q1, iq, live, e, base), k2 = te_cut(p, q2, iq, live, e, base);
            if (!__any_sync(kFull, k1.on || k2.on))
                continue;
            const TeRow   row = te_row(p.SM, p.PM, p, a, iq);
            const float4* Sg  = reinterpret_cast<const float4*>(row.S);
            const uint2*  Pg  = reinterpret_cast<const uint2*>(row.P);
            const size_t  gs  = row.gstride >> 2;
            // the row is done when its codes pass the fine bucket of every
            // lane's last one
            const int top  = (int)__reduce_max_sync(kFull, (unsigned)max(max(k1.hi, k2.hi), 0));
            const int last = ((top + base) | ((1 << (kRowFine - kTeCountShift)) - 1)) - base;
            const int ngr  = (Llen + 3) >> 2;
            int       n1 = 0, n2 = 0, nl = 0;
            float4    s4 = make_float4(nan, nan, nan, nan);
            uint2     j4 = make_uint2(0u, 0u);
            if (lane < ngr)
            {
                s4 = Sg[row_group(lane, gs, row.run)];
                j4 = Pg[row_group(lane, gs, row.run)];
            }
            bool more = true; // warp-uniform
            for (int m0 = 0; more && m0 < Llen; m0 += kRwChunk)
            {
                so[lane] = make_uint4(te_row16(j4.x & 0xFFFFu), te_row16(j4.x >> 16), te_row16(j4.y & 0xFFFFu),
                                      te_row16(j4.y >> 16));
                sc[lane] = make_uint2((unsigned)te_code16(s4.x, base) | ((unsigned)te_code16(s4.y, base) << 16),
                                      (unsigned)te_code16(s4.z, base) | ((unsigned)te_code16(s4.w, base) << 16));
                __syncwarp();
                const int g = (m0 + kRwChunk) / 4 + lane;
                s4          = make_float4(nan, nan, nan, nan);
                if (g < ngr)
                {
                    s4 = Sg[row_group(g, gs, row.run)];
                    j4 = Pg[row_group(g, gs, row.run)];
                }
                const int nsub = min(kRwChunk / 8, (Llen - m0 + 7) >> 3);
                for (int sub = 0; more && sub < nsub; ++sub)
                {
                    const uint4    cv = *reinterpret_cast<const uint4*>(sc + sub * 2);
                    const uint4    o0 = so[sub * 2], o1 = so[sub * 2 + 1];
                    const unsigned of[8] = {o0.x, o0.y, o0.z, o0.w, o1.x, o1.y, o1.z, o1.w};
                    const unsigned cw[4] = {cv.x, cv.y, cv.z, cv.w};
                    int            v[8];
#pragma unroll
                    for (int u = 0; u < 8; ++u)
                        v[u] = max((int)*reinterpret_cast<const uint16_t*>(tile + (of[u] ^ lane2)),
                                   (int)(u & 1 ? cw[u >> 1] >> 16 : cw[u >> 1] & 0xFFFFu));
#pragma unroll
                    for (int u = 0; u < 8; ++u)
                    {
                        const bool b1 = v[u] < k1.lo, b2 = v[u] < k2.lo;
                        n1 += b1;
                        n2 += b2;
                        if ((!b1 && v[u] <= k1.hi) || (!b2 && v[u] <= k2.hi))
                        {
                            if (nl < kTeListCap)
                                list[nl * 32] = (uint16_t)(of[u] >> 6);
                            ++nl;
                        }
                    }
                    more = (int)(cv.w >> 16) <= last;
                }
                __syncwarp(); // the stage is consumed
            }
            // the listed frames: in eps's bucket by code
            if (live)
            {
                const float4* xa = p.X32 + (size_t)a * T;
                // codes beyond the tile's, or too many frames: the count with one query per lane
                if (nl <= kTeListCap && max(k1.hi, k2.hi) < 65535)
                {
                    const float4  qa = xa[qi], qb = xb[qi];
                    const double *ra = p.XT + (size_t)a * 3 * T, *rb = p.XT + (size_t)b * 3 * T;
                    for (int i = 0; i < nl; ++i)
                    {
                        const int   j  = (int)list[i * 32];
                        const float f  = fmaxf(te3(qa, xa[j]), te3(qb, xb[j]));
                        const int   fc = te_code16(f, base);
                        const bool  m1 = fc >= k1.lo && fc <= k1.hi, m2 = fc >= k2.lo && fc <= k2.hi;
                        bool        in1 = m1 && f < k1.tlo, in2 = m2 && f < k2.tlo;
                        if ((m1 && !in1 && f <= k1.thi) || (m2 && !in2 && f <= k2.thi))
                        {
                            double d = 0.0; // rare: FP64 on the raw coordinates
#pragma unroll 1
                            for (int c3 = 0; c3 < 3; ++c3)
                                d = fmax(d, fmax(fabs(ra[c3 * T + qi] - ra[c3 * T + j]),
                                                 fabs(rb[c3 * T + qi] - rb[c3 * T + j])));
                            in1 = in1 || (m1 && f <= k1.thi && d < k1.eps);
                            in2 = in2 || (m2 && f <= k2.thi && d < k2.eps);
                        }
                        n1 += in1;
                        n2 += in2;
                    }
                    if (k1.on)
                        p.cnt[(size_t)q1 * Nv + qi].y = (unsigned)n1;
                    if (k2.on)
                        p.cnt[(size_t)q2 * Nv + qi].y = (unsigned)n2;
                }
                else
#pragma unroll 1
                    for (int s = 0; s < 2; ++s)
                    {
                        const TeTask tk{0, s == 0 ? q1 : q2, s == 0 ? a : b, s == 0 ? b : a};
                        te_count_query(p, tk, iq, s == 0 ? xa : xb, s == 0 ? xb : xa, p.eps_atom[tk.a1],
                                       p.eps_atom[tk.a2]);
                    }
            }
            __syncwarp(); // the list is free for the next row
        }
    }
}

namespace {

// Warps per CTA and CTAs per SM beside a tile (0: it does not leave room for `least`).
int te_row_warps(size_t tile, size_t warp_bytes, int least, int* ctas)
{
    const size_t all = kMaxDynamicSmem, half = all / 2 - 1024;
    *ctas            = 1;
    if (tile + least * warp_bytes > all)
        return 0;
    if (tile + 16 * warp_bytes <= half)
    {
        *ctas = 2;
        return 16;
    }
    const size_t w = (all - tile) / warp_bytes;
    return (int)(w > 32 ? 32 : w);
}

} // namespace

bool te_row_walk_fits(int natoms, int Nv, int k)
{
    int ctas = 0;
    return natoms >= 24 && natoms <= kRwMaxAtoms && k < 256 &&
           te_row_warps(rw_tile_bytes(Nv), kRwHistBytes + kRwStageBytes, 8, &ctas) > 0;
}

bool te_row_count_fits(int Nv)
{
    int ctas = 0;
    return te_row_warps(2 * rw_tile_bytes(Nv), kTeCountWarpBytes, 16, &ctas) > 0;
}

cudaError_t launch_te_row_walk(const TeBatch& b, long long queries, int maxn, int sms, cudaStream_t s)
{
    if (queries <= 0)
        return cudaSuccess;
    te_order_kernel<<<(unsigned)queries, kTeOrderThreads, sizeof(unsigned) * (size_t)maxn, s>>>(b);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess)
        return e;
    int          ctas  = 1;
    const size_t tile  = rw_tile_bytes(b.maxNv);
    const int    warps = te_row_warps(tile, kRwHistBytes + kRwStageBytes, 8, &ctas);
    const size_t smem  = tile + (size_t)warps * (kRwHistBytes + kRwStageBytes);
    e = allow_dynamic_smem(te_row_walk_kernel);
    if (e != cudaSuccess)
        return e;
    te_row_walk_kernel<<<sms * ctas, warps * 32, smem, s>>>(b);
    return cudaGetLastError();
}

cudaError_t launch_te_row_count(const TeBatch& b, long long queries, int sms, cudaStream_t s)
{
    if (queries <= 0)
        return cudaSuccess;
    int          ctas  = 1;
    const size_t tile  = 2 * rw_tile_bytes(b.maxNv);
    const int    warps = te_row_warps(tile, kTeCountWarpBytes, 16, &ctas);
    const size_t smem  = tile + (size_t)warps * kTeCountWarpBytes;
    cudaError_t  e = allow_dynamic_smem(te_row_count_kernel);
    if (e != cudaSuccess)
        return e;
    te_row_count_kernel<<<sms * ctas, warps * 32, smem, s>>>(b);
    return cudaGetLastError();
}

} // namespace gc

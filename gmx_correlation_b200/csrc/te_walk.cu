// Transfer entropy on B200: sorted-row walk with exact FP64 repair.
//
// Reference: te_matrix, lib/transfer_entropy.cpp:63-221 (the FP64 brute
// force te_exact_kernel restates it query by query).  Restructured around
// the split of te_walk.h: the 9-D distance of an ordered pair is
// max(G, Y), G the target's 6-D (future, past) embedding distance and Y the
// source's 3-D distance, and both are rows of one atom shared by every pair
// it takes part in.
//
//   te_rows_kernel    per (atom, query): the G row and the M row (3-D
//                     distances over frames j < N_valid), in the order of
//                     narrow buckets, with frames (row_sort.cuh).
//   te_walk_kernel    one ordered pair per CTA task, one query per lane: walk
//                     the row (target G or source M) whose k-th value is
//                     larger, gathering the other distance from the pair's
//                     coordinates staged in shared memory, and histogram the
//                     joint values from the lower bound until the k-th is
//                     provably passed (the KSG walk's scheme, ksg_fast.cu).
//   te_finish_kernel  band around the k-th bucket from two row ranges, the
//                     FP32 k-th value, the FP64 eps from the few values
//                     within the error bound of it; then n_xfxp and n_xp from
//                     eps's place in the target's G and M rows and n_ypxp
//                     by enumerating the shorter of the target's and the
//                     source's M-row prefixes, every decision within the
//                     error bound of eps re-evaluated in FP64.
//   te_fixup_*        queries handed over (too many values near a bound, a
//                     histogram overflow) get the exact FP64 query.
//   te_reduce_kernel  the reference's te_sum in query order.
//
// Error bound: x32 = fl32(x64 - c) (te_x32_kernel) gives |d32 - d64| <=
// eps_a for every 3-D distance of atom a, so a G value is within eps_a1, a
// Y value within eps_a2 and a 9-D value within e = max of the two.  Only the
// value of eps enters the counts (strict <), so there is no tie rule.

#include "gc_common.cuh"
#include "gc_internal.h"
#include "ksg_fast.h"
#include "ordered_sum.cuh"
#include "row_sort.cuh"
#include "te_device.cuh"
#include "te_exact_query.cuh"
#include "te_walk.h"

namespace gc {

namespace {

// Ordered pair of walk / finish task k of descriptor p.
__device__ __forceinline__ void te_pair(const TeParams& p, long k, long& q, int& a1, int& a2)
{
    q            = p.pair_order ? (long)p.pair_order[k] : k;
    a1           = (int)(q / (p.natoms - 1));
    const int rr = (int)(q - (long)a1 * (p.natoms - 1));
    a2           = rr < a1 ? rr : rr + 1;
}

// Independent binary searches advanced together: lo[q] becomes the first
// position in [lo[q], hi[q]] of row r[q] whose value is not < t[q].  Rows are
// in fine-bucket order, so every t[q] is the first value of a fine bucket.
template <int NS>
__device__ __forceinline__ void te_bounds(const TeRow (&r)[NS], int (&lo)[NS], int (&hi)[NS], const float (&t)[NS])
{
    for (;;)
    {
        int   mid[NS];
        float v[NS];
        bool  any = false;
#pragma unroll
        for (int q = 0; q < NS; ++q)
        {
            mid[q] = (lo[q] + hi[q]) >> 1;
            v[q]   = lo[q] < hi[q] ? r[q].s(mid[q]) : 0.0f;
        }
#pragma unroll
        for (int q = 0; q < NS; ++q)
            if (lo[q] < hi[q])
            {
                if (v[q] < t[q])
                    lo[q] = mid[q] + 1;
                else
                    hi[q] = mid[q];
                any |= lo[q] < hi[q];
            }
        if (!any)
            break;
    }
}

constexpr int kTeAmbCap = 8;

} // namespace

// ---------------------------------------------------------------------------
// Sorted rows: blocks [0, natoms * Q) of a descriptor are G rows, the next
// natoms * Q the M rows, each over the frames j < N_valid, j != qi.
// ---------------------------------------------------------------------------
namespace {

// Row r of a launch's row sort.
struct TeRowOf
{
    const TeParams* p;
    int             a, iq;
    bool            g;
};

__device__ __forceinline__ TeRowOf te_row_of(const TeBatch& B, long long r)
{
    const int       dsc = te_desc_of(B.rprefix, B.n, r);
    const TeParams* p   = B.d + dsc;
    const int       row = (int)(r - B.rprefix[dsc]), per = p->natoms * p->Q;
    const bool      g   = row < per;
    const int       rem = g ? row : row - per, a = rem / p->Q;
    return TeRowOf{p, a, rem - a * p->Q, g};
}

// Distances of the row's query over its atom's frames: future and past (G), or
// the past alone.
template <bool G>
struct TeRowDist
{
    const float4*                    x;
    float4                           qp, qf;
    int                              lag;
    __device__ __forceinline__ explicit TeRowDist(const TeRowOf& o)
        : x(o.p->X32 + (size_t)o.a * o.p->T), qp(x[o.p->i0 + o.iq]), qf(qp), lag(o.p->lag)
    {
        if (G)
            qf = x[o.p->i0 + o.iq + lag];
    }
    __device__ __forceinline__ float operator()(int j) const
    {
        return G ? fmaxf(te3(qf, x[j + lag]), te3(qp, x[j])) : te3(qp, x[j]);
    }
};

} // namespace

template <int THREADS, int R>
__global__ void __launch_bounds__(THREADS, row_ctas(THREADS, R)) te_rows_kernel(TeBatch B)
{
    const TeRowOf   o   = te_row_of(B, blockIdx.x);
    const TeParams& p   = *o.p;
    const size_t    base = ((size_t)o.a * (p.Lpad >> 2) * p.Qp + ((size_t)o.iq << p.run)) * 4;
    const size_t    gs   = ((size_t)p.Qp * 4) << p.run;
    const float     top  = row_top(p.eps_atom[o.a]);
    __shared__ RowSortShared<THREADS> sh;
    if (o.g)
        sort_row<THREADS, R>(
            sh, p.Nv - 1, p.i0 + o.iq, top, TeRowDist<true>(o),
            [&B]() { return TeRowDist<true>(te_row_of(B, rows_block())); }, p.SG, p.PG, base, gs, p.run);
    else
        sort_row<THREADS, R>(
            sh, p.Nv - 1, p.i0 + o.iq, top, TeRowDist<false>(o),
            [&B]() { return TeRowDist<false>(te_row_of(B, rows_block())); }, p.SM, p.PM, base, gs, p.run);
}

// ---------------------------------------------------------------------------
// Walk
// ---------------------------------------------------------------------------
namespace {

__device__ __forceinline__ bool te_next_task(const TeBatch& B, long long total, long long* s_task, int* s_desc,
                                             int* s_next, TeTask& tk, int& d)
{
    if (threadIdx.x == 0)
    {
        const long long t = (long long)atomicAdd(B.counter, 1ull);
        *s_task           = t;
        *s_next           = 0;
        if (t < total)
            *s_desc = te_desc_of(B.wprefix, B.n, t);
    }
    __syncthreads();
    const long long t = *s_task;
    if (t >= total)
        return false;
    d                 = *s_desc;
    const TeParams& p = B.d[d];
    const long long lt = t - B.wprefix[d];
    tk.c               = (int)(lt / p.pair_count);
    te_pair(p, (long)(lt - (long long)tk.c * p.pair_count), tk.pl, tk.a1, tk.a2);
    return true;
}

} // namespace

// Pass 1 (see ksg_walk_kernel for the histogram scheme): per lane, walk the
// row whose k-th value L is larger (the target's G row, gathering the
// source's Y, or the source's M row, gathering the target's G from two
// staged frames) and histogram the joint value max(s, other).  STAGED: the
// pair's two coordinate rows in shared memory.  LO (every k < 256): values
// below L counted in histogram index 0.
// An atom's FP32 coordinate row as float4 (global or shared memory) ...
struct TeRows4
{
    const float4* x;
    __device__ __forceinline__ float4 at(int j) const { return x[j]; }
    __device__ __forceinline__ float  d3(const float4& q, int j) const { return te3(q, x[j]); }
};

// ... or as x,y float2 and z float in shared memory (12 bytes a frame).
struct TeRows12
{
    const float2* xy;
    const float*  z;
    __device__ __forceinline__ float4 at(int j) const
    {
        const float2 v = xy[j];
        return make_float4(v.x, v.y, z[j], 0.0f);
    }
    __device__ __forceinline__ float d3(const float4& q, int j) const
    {
        const float2 v = xy[j];
        return fmaxf(fmaxf(fabsf(q.x - v.x), fabsf(q.y - v.y)), fabsf(q.z - z[j]));
    }
};

// Walk of query group g of a staged pair task (x1, x2: the pair's FP32
// rows; base: this warp's histogram): the body of both walk kernels.
template <bool LO, class V>
__device__ __forceinline__ void te_walk_group(const TeParams& p, const TeTask& tk, int g, const V& x1, const V& x2,
                                              unsigned char* base, int lane)
{
    uint8_t*           hist = base + lane * 4;
    auto               H    = [hist](unsigned b) -> uint8_t& { return hist[(b >> 2) * 128 + (b & 3)]; };
    constexpr unsigned kTop = kWalkBuckets - 1;
    const float        inf  = __int_as_float(0x7f800000);
    const int          K = p.K, lag = p.lag, Llen = p.Nv - 1, shift = p.shift;
    const float        ebig = fmaxf(p.eps_atom[tk.a1], p.eps_atom[tk.a2]);
    const float        e2   = __fmul_ru(2.0f, ebig);
    const int   iq   = g * 32 + lane;
    const bool  live = iq < p.Q;
    const int   iql  = live ? iq : 0;
    const int   qi   = p.i0 + iql;
    const TeRow G1   = te_row(p.SG, p.PG, p, tk.a1, iql);
    const TeRow M2   = te_row(p.SM, p.PM, p, tk.a2, iql);
    const float gk = G1.s(K - 1), yk = M2.s(K - 1);
    const bool  wg = gk >= yk; // walk the target's G row (gather the source's Y)
    const TeRow rw = wg ? G1 : M2;
    // bucket edges are multiples of 2^shift float ulps, the same for every
    // pair: the lower bound is rounded down to one
    const unsigned Lb = __float_as_uint(wg ? gk : yk) >> shift << shift;
    const float    L  = __uint_as_float(Lb);
    // other distance of frame j: Y = |y(qi) - y(j)| or G = max over the
    // target's past (qi, j) and future (qi + lag, j + lag)
    const V&      oa = wg ? x2 : x1;
    const float4  oq = oa.at(qi);
    const float4  fq = x1.at(qi + lag);
    {
        uint4* h4 = reinterpret_cast<uint4*>(base);
        for (int e = lane; e < kWalkBuckets * 32 / 16; e += 32)
            h4[e] = make_uint4(0u, 0u, 0u, 0u);
    }
    __syncwarp();
    const unsigned Lh   = LO ? Lb - (1u << shift) : Lb;
    auto           hidx = [Lh, shift](float v) -> unsigned {
        if (LO)
            return (unsigned)min(max((int)(__float_as_uint(v) - Lh) >> shift, 0), (int)kTop);
        return min((__float_as_uint(v) - Lh) >> shift, kTop);
    };
    const float4* Sg = reinterpret_cast<const float4*>(rw.S);
    const uint2*  Pg = reinterpret_cast<const uint2*>(rw.P);
    const size_t  gs = (size_t)p.Qp << p.run;
    int           m_end = 0, cnt_lo = 0, Rs = 0, thr = 0, grp = 0;
    unsigned      wrap = 0u;
    float         stop = inf;
    bool          walking = live;
    float4        s4      = make_float4(inf, inf, inf, inf);
    uint2         j4      = make_uint2(0u, 0u);
    if (live)
    {
        s4 = Sg[0];
        j4 = Pg[0];
    }
    const int last = (Llen - 1) >> 2;
    while (walking)
    {
        if (grp > last)
        {
            m_end = Llen;
            break;
        }
        const int      nxt   = grp < last ? grp + 1 : grp;
        const float4   ns4   = Sg[row_group(nxt, gs, p.run)];
        const uint2    nj4   = Pg[row_group(nxt, gs, p.run)];
        const float    sv[4] = {s4.x, s4.y, s4.z, s4.w};
        const unsigned jv[4] = {j4.x & 0xFFFFu, j4.x >> 16, j4.y & 0xFFFFu, j4.y >> 16};
        bool           tkn[4];
#pragma unroll
        for (int q = 0; q < 4; ++q)
        {
            tkn[q] = sv[q] <= stop;
            float o = oa.d3(oq, (int)jv[q]);
            if (!wg)
                o = fmaxf(o, x1.d3(fq, (int)jv[q] + lag));
            const float v   = fmaxf(sv[q], o);
            bool        inc = tkn[q];
            if (!LO)
            {
                const bool below = v < L;
                cnt_lo += inc && below;
                inc = inc && !below;
            }
            uint8_t&       c  = H(hidx(v));
            const unsigned h1 = (unsigned)c + (inc ? 1u : 0u);
            c                 = (uint8_t)h1;
            wrap |= h1;
        }
        ++grp;
        if (!tkn[3])
        {
            walking = false;
            m_end   = (grp - 1) * 4 + (int)tkn[0] + (int)tkn[1] + (int)tkn[2];
        }
        else if ((grp & 3) == 0)
        {
            H(kTop) = 0;
            if (stop == inf)
            {
                const float sl = sv[3];
                const int   bn = (LO || sl >= L) ? (int)hidx(sl) : 0;
                for (int b = thr; b < bn; ++b)
                    Rs += H(b);
                thr = max(thr, bn);
                if (cnt_lo + Rs >= K)
                    stop = __fadd_ru(__uint_as_float(Lh + ((unsigned)bn << shift)), e2);
            }
        }
        s4 = ns4;
        j4 = nj4;
    }
    if (live)
    {
        int bstar, prefix;
        if (stop != inf)
        {
            int cum = cnt_lo + Rs, b = thr - 1;
            while (b > 0 && cum - (int)H(b) >= K)
            {
                cum -= H(b);
                --b;
            }
            bstar  = b;
            prefix = cum - H(b);
        }
        else
        {
            int cum = cnt_lo, b = 0;
            while (b < (int)kTop && cum + (int)H(b) < K)
            {
                cum += H(b);
                ++b;
            }
            bstar  = b;
            prefix = cum;
        }
        const int reason = (wrap > 255u || (LO && bstar == 0)) ? kTeReasonBand
                           : (bstar >= (int)kTop ? kTeReasonRange : 0);
        p.wres[(size_t)tk.pl * p.Q + iq] = te_pack_walk(LO ? bstar - 1 : bstar, prefix, m_end, reason);
    }
    if (p.walk_elems)
    {
        const unsigned we = __reduce_add_sync(kFull, live ? (unsigned)m_end : 0u);
        if (lane == 0 && we)
            atomicAdd(p.walk_elems, (unsigned long long)we);
    }
    __syncwarp();
}

template <bool STAGED, bool LO>
__global__ void __launch_bounds__(1024, 1) te_walk_kernel(TeBatch B)
{
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ long long s_task;
    __shared__ int       s_desc, s_next;
    const int            warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    float4*              sx   = reinterpret_cast<float4*>(smem_raw);
    unsigned char*       base = smem_raw + (STAGED ? (size_t)2 * B.maxT * 16 : 0) + (size_t)warp * kWalkBuckets * 32;

    const long long total = B.wprefix[B.n];
    TeTask          tk;
    int             dsc;
    while (te_next_task(B, total, &s_task, &s_desc, &s_next, tk, dsc))
    {
        const TeParams& p       = B.d[dsc];
        const int       T       = p.T;
        const int       ngroups = (p.Q + 31) >> 5;
        const float4*   x1      = p.X32 + (size_t)tk.a1 * T;
        const float4*   x2      = p.X32 + (size_t)tk.a2 * T;
        if (STAGED)
        {
            for (int e = threadIdx.x; e < T; e += blockDim.x)
            {
                sx[e]     = x1[e];
                sx[T + e] = x2[e];
            }
            __syncthreads();
            x1 = sx;
            x2 = sx + T;
        }
        for (;;)
        {
            int gi = 0;
            if (lane == 0)
                gi = atomicAdd(&s_next, 1);
            gi          = __shfl_sync(kFull, gi, 0);
            const int g = tk.c * B.chunk + gi;
            if (gi >= B.chunk || g >= ngroups)
                break;
            te_walk_group<LO>(p, tk, g, TeRows4{x1}, TeRows4{x2}, base, lane);
        }
        __syncthreads();
    }
}

// ---------------------------------------------------------------------------
// Finish
// ---------------------------------------------------------------------------
namespace {

// FP64 distances of one query on the raw coordinates (the reference's
// arithmetic: |q - x| per component, max over components).
struct TeQuery64
{
    const double* a; // target rows [3][T]
    const double* b; // source rows [3][T]
    int           T, lag, qi;
    double        f0, f1, f2, p0, p1, p2, y0, y1, y2;

    __device__ __forceinline__ TeQuery64(const double* XT, int T_, int lag_, int a1, int a2, int qi_)
        : a(XT + (size_t)a1 * 3 * T_), b(XT + (size_t)a2 * 3 * T_), T(T_), lag(lag_), qi(qi_)
    {
        f0 = a[qi + lag];
        f1 = a[T + qi + lag];
        f2 = a[2 * T + qi + lag];
        p0 = a[qi];
        p1 = a[T + qi];
        p2 = a[2 * T + qi];
        y0 = b[qi];
        y1 = b[T + qi];
        y2 = b[2 * T + qi];
    }
    __device__ __forceinline__ double past(int j) const
    {
        return fmax(fmax(fabs(p0 - a[j]), fabs(p1 - a[T + j])), fabs(p2 - a[2 * T + j]));
    }
    __device__ __forceinline__ double fut(int j) const
    {
        const int jj = j + lag;
        return fmax(fmax(fabs(f0 - a[jj]), fabs(f1 - a[T + jj])), fabs(f2 - a[2 * T + jj]));
    }
    __device__ __forceinline__ double src(int j) const
    {
        return fmax(fmax(fabs(y0 - b[j]), fabs(y1 - b[T + j])), fabs(y2 - b[2 * T + j]));
    }
};

} // namespace

__global__ void __launch_bounds__(kTeFinishWarps * 32, 1) te_finish_kernel(TeBatch B)
{
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int      warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    unsigned char* base = smem_raw + (size_t)warp * 6 * kTeBandCap * 32;
    // per-lane columns: band entry e of lane l at [e * 32 + l]: joint FP32
    // value and frame
    float*    bv = reinterpret_cast<float*>(base) + lane;
    uint16_t* bj = reinterpret_cast<uint16_t*>(base + 4 * kTeBandCap * 32) + lane;

    const long long total = B.fprefix[B.n];
    for (;;)
    {
        long long t   = 0;
        int       dsc = 0;
        if (lane == 0)
        {
            t = (long long)atomicAdd(B.counter + 1, 1ull);
            if (t < total)
                dsc = te_desc_of(B.fprefix, B.n, t);
        }
        t   = __shfl_sync(kFull, t, 0);
        dsc = __shfl_sync(kFull, dsc, 0);
        if (t >= total)
            break;
        const TeParams& p  = B.d[dsc];
        const int       T = p.T, K = p.K, lag = p.lag, Nv = p.Nv, Llen = Nv - 1, shift = p.shift;
        const long long lt = t - B.fprefix[dsc];
        const int       g  = (int)(lt / p.pair_count);
        long            pl;
        int             a1, a2;
        te_pair(p, (long)(lt - (long long)g * p.pair_count), pl, a1, a2);
        const int  iq   = g * 32 + lane;
        const bool live = iq < p.Q;
        if (live)
        {
            const int                qi = p.i0 + iq;
            const unsigned long long wr = p.wres[(size_t)pl * p.Q + iq];
            const int                bstar = (int)(wr & 0xFF), prefix = (int)((wr >> 8) & 0xFFFF);
            const int                m_end = (int)((wr >> 24) & 0xFFFF);
            int                      reason = (int)((wr >> 40) & 0xFF);
            if (m_end > Llen) // not a walk result: never read past the row
                reason = kTeReasonBand;
            uint2                    out    = make_uint2(kTeHandOver, kTeHandOver);
            const TeRow   G1 = te_row(p.SG, p.PG, p, a1, iq);
            const TeRow   M1 = te_row(p.SM, p.PM, p, a1, iq);
            const TeRow   M2 = te_row(p.SM, p.PM, p, a2, iq);
            const float   gk = G1.s(K - 1), yk = M2.s(K - 1);
            const bool    wg = gk >= yk;
            const unsigned Lb = __float_as_uint(wg ? gk : yk) >> shift << shift;
            const float4* x1 = p.X32 + (size_t)a1 * T;
            const float4* x2 = p.X32 + (size_t)a2 * T;
            const float4  qp = x1[qi], qf = x1[qi + lag], qy = x2[qi];
            auto gval = [&](int j) { return fmaxf(te3(qf, x1[j + lag]), te3(qp, x1[j])); };
            auto yval = [&](int j) { return te3(qy, x2[j]); };
            const float e1 = p.eps_atom[a1], e2a = p.eps_atom[a2];
            const float e2 = __fmul_ru(2.0f, fmaxf(e1, e2a));
            if (reason == 0)
            {
                // ---- band: every joint value in [inlo, bandhi], from two row ranges
                const float elo    = __uint_as_float(Lb + ((unsigned)bstar << shift));
                const float ehi    = __uint_as_float(Lb + ((unsigned)(bstar + 1) << shift));
                const float inlo   = __fsub_rd(elo, e2);
                const float bandhi = __fadd_ru(ehi, e2);
                // the rows are in the order of their fine buckets: from the one of
                // inlo to the one of bandhi
                const TeRow rr[2] = {G1, M2};
                int         lo[2] = {0, 0}, hi[2] = {Llen, Llen};
                const float from = fine_start(fmaxf(inlo, 0.0f)), tt[2] = {from, from};
                te_bounds<2>(rr, lo, hi, tt);
                const int g0 = lo[0], y0 = lo[1];
                int       nband = 0, nlo = 0;
                auto add = [&](float v, int j) {
                    if (nband < kTeBandCap)
                    {
                        bv[nband * 32] = v;
                        bj[nband * 32] = (uint16_t)j;
                    }
                    ++nband;
                    nlo += v < elo;
                };
                // The walked row's values in the band with the other value up to
                // bandhi, and the other row's with the walked value below inlo.  Row
                // by row and not walked row first, so that all lanes gather alike.
                int g1 = min(g0, Llen - 1) >> 2;
                for (bool more = true; more;)
                {
                    const float4 s4 = G1.s4(g1);
                    const uint2  j4 = G1.j4(g1);
#pragma unroll
                    for (int q = 0; q < 4; ++q)
                    {
                        const float gv = f4at(s4, q); // NaN behind the row: not in the band
                        if (gv >= inlo && gv <= bandhi)
                        {
                            const int   j  = (int)u2at16(j4, q);
                            const float yv = yval(j);
                            if (wg ? yv <= bandhi : yv < inlo)
                                add(fmaxf(gv, yv), j);
                        }
                    }
                    ++g1;
                    more = g1 * 4 < Llen && fine_start(s4.w) <= bandhi;
                }
                int y1 = min(y0, Llen - 1) >> 2;
                for (bool more = true; more;)
                {
                    const float4 s4 = M2.s4(y1);
                    const uint2  j4 = M2.j4(y1);
#pragma unroll
                    for (int q = 0; q < 4; ++q)
                    {
                        const float yv = f4at(s4, q);
                        if (yv >= inlo && yv <= bandhi)
                        {
                            const int   j  = (int)u2at16(j4, q);
                            const float gv = gval(j);
                            if (wg ? gv < inlo : gv <= bandhi)
                                add(fmaxf(gv, yv), j);
                        }
                    }
                    ++y1;
                    more = y1 * 4 < Llen && fine_start(s4.w) <= bandhi;
                }
                g1 = min(g1 * 4, Llen);
                y1 = min(y1 * 4, Llen);
                int       n_in = prefix - nlo; // #{v < inlo}
                const int r    = K - n_in;     // rank of the k-th value in the band
                if (!reason && (nband > kTeBandCap || r < 1 || r > nband))
                    reason = kTeReasonBand;

                // ---- the FP32 k-th value, then eps in FP64 from the values near it
                double eps = 0.0;
                const TeQuery64 q64(p.XT, T, lag, a1, a2, qi);
                if (!reason)
                {
                    float d32 = 0.0f;
                    for (int e = 0; e < nband; ++e)
                    {
                        const float v  = bv[e * 32];
                        int         rk = 0;
                        for (int f = 0; f < nband; ++f)
                        {
                            const float u = bv[f * 32];
                            rk += u < v || (u == v && f < e);
                        }
                        if (rk == r - 1)
                        {
                            d32 = v;
                            break;
                        }
                    }
                    const float lower = __fsub_rd(d32, e2), upper = __fadd_ru(d32, e2);
                    unsigned    amb   = 0u;
                    for (int e = 0; e < nband; ++e)
                    {
                        const float v = bv[e * 32];
                        if (v < lower)
                            ++n_in;
                        else if (v <= upper)
                            amb |= 1u << e;
                    }
                    const int need = K - n_in, n_amb = __popc(amb);
                    if (need < 1 || need > n_amb || n_amb > kTeAmbCap)
                        reason = kTeReasonAmbig;
                    else
                    {
                        double val[kTeAmbCap];
                        int    c = 0;
                        for (unsigned am = amb; am; am &= am - 1, ++c)
                        {
                            const int j = bj[(__ffs(am) - 1) * 32];
                            val[c]      = fmax(fmax(q64.fut(j), q64.past(j)), q64.src(j));
                        }
                        for (int x = 0; x < n_amb; ++x)
                        {
                            int rk = 0;
                            for (int y = 0; y < n_amb; ++y)
                                rk += val[y] < val[x] || (val[y] == val[x] && y < x);
                            if (rk == need - 1)
                                eps = val[x];
                        }
                    }
                }

                // ---- counts, strict < eps ------------------------------------------
                if (!reason)
                {
                    const float tlo1 = __double2float_rd(__dsub_rd(eps, (double)e1));
                    const float thi1 = __double2float_ru(__dadd_ru(eps, (double)e1));
                    const float thi2 = __double2float_ru(__dadd_ru(eps, (double)e2a));
                    const TeRow cr[3] = {G1, M1, M2};
                    // eps's fine buckets in G1 and M2 lie in the band's entries
                    int clo[3] = {g0, 0, y0}, chi[3] = {g1, Llen, y1};
                    const float ct[3] = {fine_start(fmaxf(tlo1, 0.0f)), fine_start(fmaxf(tlo1, 0.0f)), fine_after(thi2)};
                    te_bounds<3>(cr, clo, chi, ct);
                    // Entries of G1 (n_xfxp) and M1 (n_xp) below eps: those before
                    // the fine bucket of tlo1, and of the groups up to the fine
                    // bucket of thi1 the ones below tlo1 and, in FP64, those up to
                    // thi1.  Both rows' groups are loaded together; the FP64
                    // looks come after them, so the lanes take theirs at once.
                    int  gg = min(clo[0], Llen - 1) >> 2, gm = min(clo[1], Llen - 1) >> 2;
                    int  n_xfxp = gg * 4, n_xp = gm * 4;
                    bool on_g = true, on_m = true;
                    auto look = [&](const TeRow& row, int& g, bool& on, int& n, unsigned& amb, int at) {
                        const float4 s4 = row.s4(g);
#pragma unroll
                        for (int q = 0; q < 4; ++q)
                        {
                            const float s = f4at(s4, q); // NaN behind the row: neither
                            n += s < tlo1;
                            amb |= (unsigned)(s >= tlo1 && s <= thi1) << (at + q);
                        }
                        ++g;
                        on = g * 4 < Llen && fine_start(s4.w) <= thi1;
                    };
                    do
                    {
                        const int gb = gg * 4, mb = gm * 4;
                        unsigned  ag = 0u, am = 0u;
                        for (int at = 0; at < 32 && (on_g || on_m); at += 4)
                        {
                            if (on_g)
                                look(G1, gg, on_g, n_xfxp, ag, at);
                            if (on_m)
                                look(M1, gm, on_m, n_xp, am, at);
                        }
                        for (; ag; ag &= ag - 1)
                        {
                            const int j = G1.j(gb + __ffs(ag) - 1);
                            n_xfxp += fmax(q64.fut(j), q64.past(j)) < eps;
                        }
                        for (; am; am &= am - 1)
                            n_xp += q64.past(M1.j(mb + __ffs(am) - 1)) < eps;
                    } while (on_g || on_m);
                    const int end1 = min(gm * 4, Llen); // M1's entries up to thi1 lie before
                    // n_ypxp is counted by te_count_kernel over the shorter of
                    // the two M-row prefixes that can hold a value below eps:
                    // it gets eps (in wres) and the prefix (in cnt.y).
                    const int  end2 = clo[2];
                    const bool on1  = end1 <= end2;
                    const int  ne   = on1 ? end1 : end2;
                    p.wres[(size_t)pl * p.Q + iq] = (unsigned long long)__double_as_longlong(eps);
                    out = make_uint2((unsigned)n_xp | ((unsigned)n_xfxp << 16),
                                     (unsigned)ne | (on1 ? kTeCountOn1 : 0u));
                }
            }
            if (reason)
            {
                out = make_uint2(kTeHandOver, kTeHandOver);
                atomicOr(p.status, kStatFallback);
                if (p.reasons)
                    atomicAdd(p.reasons + reason, 1u);
                if (p.hq)
                {
                    const unsigned hqi = atomicAdd(p.hq_len, 1u);
                    if (hqi < p.hq_cap)
                        p.hq[hqi] = (unsigned long long)pl * Nv + qi;
                }
            }
            p.cnt[(size_t)pl * Nv + qi] = out;
        }
        __syncwarp();
    }
}

// ---------------------------------------------------------------------------
// n_ypxp = #{j : max(D1(qi, j), Y(qi, j)) < eps}: one ordered pair per CTA
// task with its two coordinate rows staged in shared memory (the walk's
// task scheme), one query per lane.  Each lane enumerates the prefix the
// finish kernel chose (the target's or the source's M row, every entry whose
// FP32 value may lie below eps), gathers the other marginal from shared
// memory, and re-evaluates in FP64 every entry within the error bound of
// eps.
// ---------------------------------------------------------------------------
template <bool STAGED>
__global__ void __launch_bounds__(1024, 1) te_count_kernel(TeBatch B)
{
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ long long s_task;
    __shared__ int       s_desc, s_next;
    const int            lane = threadIdx.x & 31;
    float4*              sx   = reinterpret_cast<float4*>(smem_raw);
    const long long      total = B.wprefix[B.n];
    TeTask               tk;
    int                  dsc;
    while (te_next_task(B, total, &s_task, &s_desc, &s_next, tk, dsc))
    {
        const TeParams& p       = B.d[dsc];
        const int       T = p.T, Nv = p.Nv;
        const int       ngroups = (p.Q + 31) >> 5;
        const float4*   x1      = p.X32 + (size_t)tk.a1 * T;
        const float4*   x2      = p.X32 + (size_t)tk.a2 * T;
        if (STAGED)
        {
            for (int e = threadIdx.x; e < T; e += blockDim.x)
            {
                sx[e]     = x1[e];
                sx[T + e] = x2[e];
            }
            __syncthreads();
            x1 = sx;
            x2 = sx + T;
        }
        const float e1 = p.eps_atom[tk.a1], e2a = p.eps_atom[tk.a2];
        for (;;)
        {
            int gi = 0;
            if (lane == 0)
                gi = atomicAdd(&s_next, 1);
            gi          = __shfl_sync(kFull, gi, 0);
            const int g = tk.c * B.chunk + gi;
            if (gi >= B.chunk || g >= ngroups)
                break;
            const int iq = g * 32 + lane;
            if (iq < p.Q)
                te_count_query(p, tk, iq, x1, x2, e1, e2a);
        }
        __syncthreads(); // every warp is done with the staged rows
    }
}

// A staged pair task of the double-buffered count kernel.
struct TeSlot
{
    long long    t;    // global task, or -1: no more tasks
    int          desc; // descriptor of the task
    int          next; // query groups handed out
    int          left; // warps done with the task
    volatile int gen;  // CTA-local index of the task this slot holds
    TeTask       tk;
};

// Fills slot S with the next global task as CTA-local task `gen`: one warp
// (lane 0 takes the task, all lanes copy the pair's two FP32 rows through
// put(T, frame e, a1's value, a2's value)).
template <class Put>
__device__ __forceinline__ void te_slot_fill_with(const TeBatch& B, long long total, TeSlot& S, int gen, int lane,
                                                  Put put)
{
    long long t = 0;
    int       d = 0;
    if (lane == 0)
    {
        t = (long long)atomicAdd(B.counter, 1ull);
        if (t < total)
            d = te_desc_of(B.wprefix, B.n, t);
        else
            t = -1;
    }
    t = __shfl_sync(kFull, t, 0);
    d = __shfl_sync(kFull, d, 0);
    TeTask tk{};
    if (t >= 0)
    {
        const TeParams& p  = B.d[d];
        const long long lt = t - B.wprefix[d];
        tk.c               = (int)(lt / p.pair_count);
        te_pair(p, (long)(lt - (long long)tk.c * p.pair_count), tk.pl, tk.a1, tk.a2);
        const int     T  = p.T;
        const float4* x1 = p.X32 + (size_t)tk.a1 * T;
        const float4* x2 = p.X32 + (size_t)tk.a2 * T;
        for (int e = lane; e < T; e += 32)
            put(T, e, x1[e], x2[e]);
    }
    __syncwarp();
    if (lane == 0)
    {
        S.t    = t;
        S.desc = d;
        S.tk   = tk;
        S.next = 0;
        S.left = 0;
        __threadfence_block(); // the rows and fields before the generation
        S.gen = gen;
    }
    __syncwarp();
}

__device__ __forceinline__ void te_slot_fill(const TeBatch& B, long long total, TeSlot& S, float4* rows, int gen,
                                             int lane)
{
    te_slot_fill_with(B, total, S, gen, lane, [rows](int T, int e, const float4& a, const float4& b) {
        rows[e]     = a;
        rows[T + e] = b;
    });
}

__device__ __forceinline__ void te_slot_fill12(const TeBatch& B, long long total, TeSlot& S, float2* xy, float* z,
                                               int gen, int lane)
{
    te_slot_fill_with(B, total, S, gen, lane, [xy, z](int T, int e, const float4& a, const float4& b) {
        xy[e]     = make_float2(a.x, a.y);
        z[e]      = a.z;
        xy[T + e] = make_float2(b.x, b.y);
        z[T + e]  = b.z;
    });
}

// The count kernel with two staged pair tasks per CTA (2 x 2 x maxT float4):
// a warp done with its query groups of task i moves on to task i + 1 without
// waiting for the CTA; the last warp to leave task i refills its buffer with
// task i + 2.  Tasks reach a CTA in its local index order (one warp fills
// both buffers first), so a warp stops at the first slot without a task.
__global__ void __launch_bounds__(1024, 1) te_count_db_kernel(TeBatch B)
{
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ TeSlot slot[2];
    const int         warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nwarps = blockDim.x >> 5;
    const long long   total = B.wprefix[B.n];
    auto              rows  = [&](int b) { return reinterpret_cast<float4*>(smem_raw) + (size_t)b * 2 * B.maxT; };
    if (warp == 0)
    {
        te_slot_fill(B, total, slot[0], rows(0), 0, lane);
        te_slot_fill(B, total, slot[1], rows(1), 1, lane);
    }
    __syncthreads();
    for (int i = 0;; ++i)
    {
        const int b = i & 1;
        TeSlot&   S = slot[b];
        // bounded wait for the refilling warp (resident, never waiting itself)
        int spins = 0;
        while (S.gen != i)
        {
            if (++spins > (1 << 24))
            {
                if (lane == 0)
                    atomicOr(B.d[0].status, kStatTimeout);
                return;
            }
            __nanosleep(64);
        }
        __threadfence_block();
        if (S.t < 0)
            break;
        const TeParams& p       = B.d[S.desc];
        const TeTask    tk      = S.tk;
        const int       ngroups = (p.Q + 31) >> 5;
        const float4*   x1      = rows(b);
        const float4*   x2      = x1 + p.T;
        const float     e1 = p.eps_atom[tk.a1], e2a = p.eps_atom[tk.a2];
        for (;;)
        {
            int gi = 0;
            if (lane == 0)
                gi = atomicAdd(&S.next, 1);
            gi          = __shfl_sync(kFull, gi, 0);
            const int g = tk.c * B.chunk + gi;
            if (gi >= B.chunk || g >= ngroups)
                break;
            const int iq = g * 32 + lane;
            if (iq < p.Q)
                te_count_query(p, tk, iq, x1, x2, e1, e2a);
        }
        int last = 0;
        if (lane == 0)
            last = atomicAdd(&S.left, 1) == nwarps - 1;
        last = __shfl_sync(kFull, last, 0);
        if (last) // every warp has left task i: its buffer takes task i + 2
            te_slot_fill(B, total, S, rows(b), i + 2, lane);
    }
}

// The walk with two staged pair tasks per CTA (the count kernel's scheme):
// per buffer the pair's rows as x,y float2 [2 maxT] and z float [2 maxT]
// (24 maxT bytes), then each warp's histogram.
template <bool LO>
__global__ void __launch_bounds__(1024, 1) te_walk_db_kernel(TeBatch B)
{
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ TeSlot slot[2];
    const int         warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nwarps = blockDim.x >> 5;
    const long long   total = B.wprefix[B.n];
    const int         maxT  = B.maxT;
    auto              xyb   = [&](int b) { return reinterpret_cast<float2*>(smem_raw + (size_t)b * 24 * maxT); };
    auto zb = [&](int b) { return reinterpret_cast<float*>(smem_raw + (size_t)b * 24 * maxT + (size_t)16 * maxT); };
    unsigned char* base = smem_raw + (size_t)48 * maxT + (size_t)warp * kWalkBuckets * 32;
    if (warp == 0)
    {
        te_slot_fill12(B, total, slot[0], xyb(0), zb(0), 0, lane);
        te_slot_fill12(B, total, slot[1], xyb(1), zb(1), 1, lane);
    }
    __syncthreads();
    for (int i = 0;; ++i)
    {
        const int b = i & 1;
        TeSlot&   S = slot[b];
        int       spins = 0;
        while (S.gen != i)
        {
            if (++spins > (1 << 24))
            {
                if (lane == 0)
                    atomicOr(B.d[0].status, kStatTimeout);
                return;
            }
            __nanosleep(64);
        }
        __threadfence_block();
        if (S.t < 0)
            break;
        const TeParams& p       = B.d[S.desc];
        const TeTask    tk      = S.tk;
        const int       ngroups = (p.Q + 31) >> 5;
        const TeRows12  r1{xyb(b), zb(b)}, r2{xyb(b) + p.T, zb(b) + p.T};
        for (;;)
        {
            int gi = 0;
            if (lane == 0)
                gi = atomicAdd(&S.next, 1);
            gi          = __shfl_sync(kFull, gi, 0);
            const int g = tk.c * B.chunk + gi;
            if (gi >= B.chunk || g >= ngroups)
                break;
            te_walk_group<LO>(p, tk, g, r1, r2, base, lane);
        }
        int last = 0;
        if (lane == 0)
            last = atomicAdd(&S.left, 1) == nwarps - 1;
        last = __shfl_sync(kFull, last, 0);
        if (last)
            te_slot_fill12(B, total, S, xyb(b), zb(b), i + 2, lane);
    }
}

// ---------------------------------------------------------------------------
// Hand-overs, reduction
// ---------------------------------------------------------------------------
__device__ __forceinline__ void te_fixup_one(const TeParams& p, long long idx, unsigned* hist, int lane)
{
    const long pl = (long)(idx / p.Nv);
    const int  qi = (int)(idx - (long long)pl * p.Nv);
    const int  a1 = (int)(pl / (p.natoms - 1));
    const int  rr = (int)(pl - (long)a1 * (p.natoms - 1));
    const int  a2 = rr < a1 ? rr : rr + 1;
    const uint2 c = te_exact_query(p.XT, p.T, p.K, p.lag, a1, a2, qi, hist, lane);
    if (lane == 0)
        p.cnt[idx] = c;
    __syncwarp();
}

__global__ void __launch_bounds__(256) te_fixup_queue_kernel(TeBatch B)
{
    __shared__ unsigned hist[8][256];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    for (int d = 0; d < B.n; ++d)
    {
        const TeParams& p = B.d[d];
        if (!p.hq)
            continue;
        const unsigned n = min(*p.hq_len, p.hq_cap);
        for (unsigned e = blockIdx.x * 8 + warp; e < n; e += gridDim.x * 8)
            te_fixup_one(p, (long long)p.hq[e], hist[warp], lane);
    }
}

__global__ void __launch_bounds__(256) te_fixup_scan_kernel(TeBatch B)
{
    __shared__ unsigned hist[8][256];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    for (int d = 0; d < B.n; ++d)
    {
        const TeParams& p = B.d[d];
        if (p.hq && *p.hq_len <= p.hq_cap)
            continue;
        const long long n = (long long)p.Nv * p.pair_count;
        for (long long c0 = ((long long)blockIdx.x * 8 + warp) * 32; c0 < n; c0 += (long long)gridDim.x * 8 * 32)
        {
            const long long e  = c0 + lane;
            unsigned        hm = __ballot_sync(kFull, e < n && p.cnt[e].x == kTeHandOver);
            while (hm)
            {
                const int src = __ffs(hm) - 1;
                hm &= hm - 1;
                te_fixup_one(p, c0 + src, hist[warp], lane);
            }
        }
    }
}

// te_sum += psi_k + psi[n_xp + 1] - psi[n_xfxp + 1] - psi[n_ypxp + 1] with
// the counts clamped to N_valid, in query order; te_sum / N_valid
// (lib/transfer_entropy.cpp:188-204).  cnt is pair-major [q][Nv].
__global__ void __launch_bounds__(kSumThreads)
    te_reduce_kernel(const uint2* __restrict__ cnt, int natoms, int Nv, int K, int P, const double* __restrict__ psi,
                     double* __restrict__ te_mat)
{
    const long   npairs = (long)natoms * (natoms - 1);
    const long   q0     = (long)blockIdx.x * P;
    const int    live   = (int)min((long)P, npairs - q0);
    const uint2* c      = cnt + (size_t)q0 * Nv;
    const double pk     = psi[K];
    const double sum    = ordered_sums(P, live, Nv, [&](int p, int f) {
        const uint2 v  = c[(size_t)p * Nv + f];
        const int   xp = min((int)(v.x & 0xFFFFu), Nv);
        const int   xf = min((int)(v.x >> 16), Nv);
        const int   yp = min((int)v.y, Nv);
        return __dsub_rn(__dsub_rn(__dadd_rn(pk, psi[xp + 1]), psi[xf + 1]), psi[yp + 1]);
    });
    if ((int)threadIdx.x < live)
    {
        const long q  = q0 + threadIdx.x;
        const int  a1 = (int)(q / (natoms - 1));
        const int  rr = (int)(q - (long)a1 * (natoms - 1));
        const int  a2 = rr < a1 ? rr : rr + 1;
        te_mat[(size_t)a1 * natoms + a2] = __ddiv_rn(sum, (double)Nv);
    }
}

// ---------------------------------------------------------------------------
// Launchers
// ---------------------------------------------------------------------------
cudaError_t launch_te_rows(const TeBatch& b, long long rows, cudaStream_t s)
{
    if (rows <= 0)
        return cudaSuccess;
    int          threads = 256, regs = 0;
    const size_t smem    = row_sort_smem(b.maxNv - 1, &threads, &regs);
    void (*kernel)(TeBatch) = te_rows_kernel<1024, 0>;
    if (threads == 64)
        kernel = te_rows_kernel<64, 8>;
    else if (threads == 128)
        kernel = regs == 8 ? te_rows_kernel<128, 8> : te_rows_kernel<128, 16>;
    else if (threads == 256)
        kernel = te_rows_kernel<256, 16>;
    else if (threads == 512)
        kernel = te_rows_kernel<512, 16>;
    cudaError_t e = allow_dynamic_smem(kernel);
    if (e != cudaSuccess)
        return e;
    kernel<<<(unsigned)rows, threads, smem, s>>>(b);
    return cudaGetLastError();
}

cudaError_t launch_te_walk(const TeBatch& b, int warps, bool staged, int sms, cudaStream_t s)
{
    const bool lo = b.maxK < 256;
    // two staged pair tasks per CTA (12-byte rows) where they fit beside the
    // warps' histograms, else one (16-byte rows)
    const size_t hist = (size_t)warps * kWalkBuckets * 32;
    const bool   dbuf = staged && (size_t)48 * b.maxT + hist <= kMaxDynamicSmem;
    void (*kernel)(TeBatch) = dbuf     ? (lo ? te_walk_db_kernel<true> : te_walk_db_kernel<false>)
                              : staged ? (lo ? te_walk_kernel<true, true> : te_walk_kernel<true, false>)
                                       : (lo ? te_walk_kernel<false, true> : te_walk_kernel<false, false>);
    const size_t smem = (dbuf ? (size_t)48 * b.maxT : (staged ? (size_t)2 * b.maxT * 16 : 0)) + hist;
    cudaError_t  e    = allow_dynamic_smem(kernel);
    if (e != cudaSuccess)
        return e;
    int per_sm = 0;
    e          = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, warps * 32, smem);
    if (e != cudaSuccess)
        return e;
    per_sm = per_sm < 1 ? 1 : per_sm;
    kernel<<<sms * per_sm, warps * 32, smem, s>>>(b);
    return cudaGetLastError();
}

cudaError_t launch_te_finish(const TeBatch& b, int sms, cudaStream_t s)
{
    const size_t smem = (size_t)kTeFinishWarps * 6 * kTeBandCap * 32;
    cudaError_t  e    = allow_dynamic_smem(te_finish_kernel);
    if (e != cudaSuccess)
        return e;
    int per_sm = 0;
    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, te_finish_kernel, kTeFinishWarps * 32, smem);
    if (e != cudaSuccess)
        return e;
    per_sm = per_sm < 1 ? 1 : per_sm;
    te_finish_kernel<<<sms * per_sm, kTeFinishWarps * 32, smem, s>>>(b);
    return cudaGetLastError();
}

cudaError_t launch_te_count(const TeBatch& b, int warps, bool staged, int sms, cudaStream_t s)
{
    // two staged pair tasks per CTA where they fit (rows of up to 3584
    // frames), else one
    const size_t db      = (size_t)4 * b.maxT * 16;
    const bool   dbuf    = staged && db <= (size_t)224 * 1024;
    void (*kernel)(TeBatch) = dbuf ? te_count_db_kernel : (staged ? te_count_kernel<true> : te_count_kernel<false>);
    const size_t smem = dbuf ? db : (staged ? (size_t)2 * b.maxT * 16 : 0);
    cudaError_t  e    = allow_dynamic_smem(kernel);
    if (e != cudaSuccess)
        return e;
    int per_sm = 0;
    e          = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, warps * 32, smem);
    if (e != cudaSuccess)
        return e;
    per_sm = per_sm < 1 ? 1 : per_sm;
    kernel<<<sms * per_sm, warps * 32, smem, s>>>(b);
    return cudaGetLastError();
}

cudaError_t launch_te_fixup(const TeBatch& b, int sms, cudaStream_t s)
{
    te_fixup_queue_kernel<<<sms * 4, 256, 0, s>>>(b);
    const cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess)
        return e;
    te_fixup_scan_kernel<<<sms * 4, 256, 0, s>>>(b);
    return cudaGetLastError();
}

cudaError_t launch_te_reduce(const uint2* cnt, int natoms, int Nv, int K, const double* psi, double* te_mat, int sms,
                             cudaStream_t s)
{
    const long npairs = (long)natoms * (natoms - 1);
    const int  P      = sums_per_cta(npairs, sms);
    te_reduce_kernel<<<(unsigned)((npairs + P - 1) / P), kSumThreads, 0, s>>>(cnt, natoms, Nv, K, P, psi, te_mat);
    return cudaGetLastError();
}

} // namespace gc

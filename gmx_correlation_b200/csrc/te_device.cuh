// Device helpers shared by the transfer-entropy fast-path kernels (te_walk.cu, te_row_walk.cu).
#pragma once

#include "gc_common.cuh"
#include "ksg_fast.h"
#include "te_walk.h"

namespace gc {

__device__ __forceinline__ float te3(const float4 a, const float4 b)
{
    return fmaxf(fmaxf(fabsf(a.x - b.x), fabsf(a.y - b.y)), fabsf(a.z - b.z));
}

// The descriptor owning task t: the largest d with prefix[d] <= t.
__device__ __forceinline__ int te_desc_of(const long long* __restrict__ prefix, int n, long long t)
{
    int lo = 0, hi = n - 1;
    while (lo < hi)
    {
        const int mid = (lo + hi + 1) >> 1;
        if (prefix[mid] <= t)
            lo = mid;
        else
            hi = mid - 1;
    }
    return lo;
}

// One lane's view of a transposed sorted row.
struct TeRow
{
    const float*    S;
    const uint16_t* P;
    size_t          gstride; // elements from a run to the next
    int             run;     // log2 of a run's 4-entry groups

    __device__ __forceinline__ float s(int m) const { return S[row_entry(m, gstride, run)]; }
    __device__ __forceinline__ int   j(int m) const { return P[row_entry(m, gstride, run)]; }
    __device__ __forceinline__ float4 s4(int g) const
    {
        return *reinterpret_cast<const float4*>(S + row_entry(g * 4, gstride, run));
    }
    __device__ __forceinline__ uint2 j4(int g) const { return *reinterpret_cast<const uint2*>(P + row_entry(g * 4, gstride, run)); }
};

__device__ __forceinline__ TeRow te_row(const float* S, const uint16_t* P, const TeParams& p, int atom, int iq)
{
    const size_t base = ((size_t)atom * (p.Lpad >> 2) * p.Qp + ((size_t)iq << p.run)) * 4;
    return TeRow{S + base, P + base, ((size_t)p.Qp * 4) << p.run, p.run};
}

__device__ __forceinline__ float f4at(const float4& v, int q)
{
    return q == 0 ? v.x : (q == 1 ? v.y : (q == 2 ? v.z : v.w));
}

__device__ __forceinline__ unsigned u2at16(const uint2& v, int q)
{
    return q < 2 ? ((v.x >> (16 * q)) & 0xFFFFu) : ((v.y >> (16 * (q - 2))) & 0xFFFFu);
}

// Hand-over causes (TeParams::reasons index).
enum
{
    kTeReasonRange  = 2, // k-th value beyond the histogram's range
    kTeReasonBand   = 3, // band larger than kTeBandCap or inconsistent with the histogram
    kTeReasonAmbig  = 4  // more than kTeAmbCap values within the error bound of the k-th
};
__device__ __forceinline__ unsigned long long te_pack_walk(int bstar, int prefix, int m_end, int reason)
{
    return (unsigned long long)(bstar & 0xFF) | ((unsigned long long)(prefix & 0xFFFF) << 8) |
           ((unsigned long long)(m_end & 0xFFFF) << 24) | ((unsigned long long)(reason & 0xFF) << 40);
}

struct TeTask
{
    int  c;  // chunk of query groups
    long pl; // ordered pair (local index)
    int  a1, a2;
};

// n_ypxp of query iq of a staged pair task (x1, x2: the pair's FP32 rows,
// in shared or global memory): the body of both count kernels.
__device__ __forceinline__ void te_count_query(const TeParams& p, const TeTask& tk, int iq, const float4* x1,
                                               const float4* x2, float e1, float e2a)
{
    const int T = p.T, Nv = p.Nv;
    const int    qi = p.i0 + iq;
    uint2* const cp = p.cnt + (size_t)tk.pl * Nv + qi;
    const uint2  c  = *cp;
    if (c.x != kTeHandOver)
    {
        const double eps = __longlong_as_double((long long)p.wres[(size_t)tk.pl * p.Q + iq]);
        const int    ne  = (int)(c.y & 0xFFFFu);
        const bool   on1 = (c.y & kTeCountOn1) != 0u;
        const double es = on1 ? (double)e1 : (double)e2a, eo = on1 ? (double)e2a : (double)e1;
        const float  tlo_s = __double2float_rd(__dsub_rd(eps, es));
        const float  tlo_o = __double2float_rd(__dsub_rd(eps, eo));
        const float  thi_o = __double2float_ru(__dadd_ru(eps, eo));
        const float  thi_s = __double2float_ru(__dadd_ru(eps, es));
        const TeRow  er = te_row(p.SM, p.PM, p, on1 ? tk.a1 : tk.a2, iq);
        const float4* ox = on1 ? x2 : x1;
        const float4  oq = ox[qi];
        const float4* Sg = reinterpret_cast<const float4*>(er.S);
        const uint2*  Pg = reinterpret_cast<const uint2*>(er.P);
        const size_t  gs = (size_t)p.Qp << p.run;
        const int     ng = (ne + 3) >> 2;
        int           n  = 0;
        float4        s4 = make_float4(0.f, 0.f, 0.f, 0.f);
        uint2         j4 = make_uint2(0u, 0u);
        if (ng > 0)
        {
            s4 = Sg[0];
            j4 = Pg[0];
        }
        for (int g0 = 0; g0 < ng; ++g0)
        {
            // the next group is loaded while this one is counted
            const int    nx  = g0 + 1 < ng ? g0 + 1 : g0;
            const float4 ns4 = Sg[row_group(nx, gs, p.run)];
            const uint2  nj4 = Pg[row_group(nx, gs, p.run)];
            const float  sv[4] = {s4.x, s4.y, s4.z, s4.w};
            const unsigned jv[4] = {j4.x & 0xFFFFu, j4.x >> 16, j4.y & 0xFFFFu, j4.y >> 16};
            unsigned     amb = 0u;
#pragma unroll
            for (int q = 0; q < 4; ++q)
            {
                const bool  in = g0 * 4 + q < ne;
                const float ov = te3(oq, ox[jv[q]]);
                if (in && sv[q] < tlo_s && ov < tlo_o)
                    ++n;
                else if (in && sv[q] <= thi_s && ov <= thi_o)
                    amb |= 1u << q;
            }
            for (; amb; amb &= amb - 1) // rare: FP64 on the raw coordinates
            {
                const int     j  = (int)u2at16(j4, __ffs(amb) - 1);
                const double* ra = p.XT + (size_t)tk.a1 * 3 * T;
                const double* rb = p.XT + (size_t)tk.a2 * 3 * T;
                double        d  = 0.0;
#pragma unroll 1
                for (int c3 = 0; c3 < 3; ++c3)
                    d = fmax(d, fmax(fabs(ra[c3 * T + qi] - ra[c3 * T + j]),
                                     fabs(rb[c3 * T + qi] - rb[c3 * T + j])));
                n += d < eps;
            }
            s4 = ns4;
            j4 = nj4;
        }
        cp->y = (unsigned)n;
    }
}

} // namespace gc

// Device helpers shared by the KSG fast-path kernels (ksg_fast.cu, ksg_row_walk.cu).
#pragma once

#include "gc_common.cuh"
#include "ksg_fast.h"

namespace gc {

__device__ __forceinline__ float dist3f(const float4 a, const float4 b)
{
    return fmaxf(fmaxf(fabsf(a.x - b.x), fabsf(a.y - b.y)), fabsf(a.z - b.z));
}

// The descriptor owning task t: the largest d with prefix[d] <= t.
__device__ __forceinline__ int batch_desc(const long long* __restrict__ prefix, int n, long long t)
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

// One lane's view of a transposed sorted row (see WalkParams).
struct LaneRow
{
    const float*    S;
    const uint16_t* P;
    size_t          gstride; // elements from a run to the next
    int             run;     // log2 of a run's 4-entry groups

    __device__ __forceinline__ float  s(int m) const { return S[row_entry(m, gstride, run)]; }
    __device__ __forceinline__ int    j(int m) const { return P[row_entry(m, gstride, run)]; }
    __device__ __forceinline__ float4 s4(int g) const
    {
        return *reinterpret_cast<const float4*>(S + row_entry(g * 4, gstride, run));
    }
    __device__ __forceinline__ uint2 j4(int g) const { return *reinterpret_cast<const uint2*>(P + row_entry(g * 4, gstride, run)); }
};

__device__ __forceinline__ LaneRow lane_row(const WalkParams& p, int atom, int iq)
{
    const size_t base = ((size_t)atom * (p.Lpad >> 2) * p.Qp + ((size_t)iq << p.run)) * 4;
    return LaneRow{p.S + base, p.P + base, ((size_t)p.Qp * 4) << p.run, p.run};
}

__device__ __forceinline__ double dist3r(const double* __restrict__ r, int T, double q0, double q1, double q2, int j)
{
    return fmax(fmax(fabs(q0 - r[j]), fabs(q1 - r[T + j])), fabs(q2 - r[2 * T + j]));
}

// Hand-over causes (WalkParams::reasons index).
enum
{
    kReasonRange    = 2, // k-th value beyond the histogram's two octaves
    kReasonBand     = 3, // band larger than kBandCap or inconsistent with the histogram
    kReasonAmbig    = 4, // ambiguous set inconsistent or larger than kAmbCap
    kReasonScan     = 5  // scan for the maxima or their counts exceeded kScanCap
};

// Walk result of one (pair, query): bucket of the k-th value, the number of
// entries below that bucket, the walked length, and a hand-over cause.
__device__ __forceinline__ unsigned long long pack_walk(int bstar, int prefix, int m_end, int reason)
{
    return (unsigned long long)(bstar & 0xFF) | ((unsigned long long)(prefix & 0xFFFF) << 8) |
           ((unsigned long long)(m_end & 0xFFFF) << 24) | ((unsigned long long)(reason & 0xFF) << 40);
}

} // namespace gc

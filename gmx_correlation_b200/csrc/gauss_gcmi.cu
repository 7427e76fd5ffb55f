// Gaussian (-linear) and Gaussian-copula (GCMI) mutual information on B200.
//
// Reference:
//   gauss_corrmatrix / covarianceMatrix / matrixDet / entropy
//       lib/correlation_core.cpp:280-311, :140-166, :49-98, :100-111
//   gcmi_corrmatrix / copula_transform / gcmi_erfinv / lu_det / gcmi_pair
//       lib/gcmi.cpp:246-317, :95-146, :26-79, :152-184, :190-231
//
// Both estimators need, per atom pair, the 6x6 co-moment matrix of the two
// atoms' 3-D series.  Its 3x3 blocks depend only on the two atoms, so one
// kernel sums every block (lo <= hi) once, sequentially over frames with
// round-to-nearest intrinsics (the reference's plain double loop, so the
// sums are bit-identical), and a second kernel assembles each pair's
// matrices and log-determinants.

#include "gc_common.cuh"
#include "gc_internal.h"

namespace gc {

// gcmi_erfinv (lib/gcmi.cpp:26-79): Acklam's rational approximation of the
// inverse normal CDF (published coefficients), mapped to erfinv, then one
// Newton step with erf/exp.
__device__ double acklam_erfinv(double x)
{
    const double a0 = -3.969683028665376e+01, a1 = 2.209460984245205e+02, a2 = -2.759285104469687e+02,
                 a3 = 1.383577518672690e+02, a4 = -3.066479806614716e+01, a5 = 2.506628277459239e+00;
    const double b0 = -5.447609879822406e+01, b1 = 1.615858368580409e+02, b2 = -1.556989798598866e+02,
                 b3 = 6.680131188771972e+01, b4 = -1.328068155288572e+01;
    const double c0 = -7.784894002430293e-03, c1 = -3.223964580411365e-01, c2 = -2.400758277161838e+00,
                 c3 = -2.549732539343734e+00, c4 = 4.374664141464968e+00, c5 = 2.938163982698783e+00;
    const double d0 = 7.784695709041462e-03, d1 = 3.224671290700398e-01, d2 = 2.445134137142996e+00,
                 d3 = 3.754408661907416e+00;
    if (x >= 1.0)
        return 1e30;
    if (x <= -1.0)
        return -1e30;
    if (x == 0.0)
        return 0.0;
    const double p = __dmul_rn(__dadd_rn(x, 1.0), 0.5);
    double       r, q;
#define M_(u, v) __dmul_rn(u, v)
#define A_(u, v) __dadd_rn(u, v)
    if (p < 0.02425)
    {
        q = sqrt(M_(-2.0, log(p)));
        r = __ddiv_rn(A_(M_(A_(M_(A_(M_(A_(M_(A_(M_(c0, q), c1), q), c2), q), c3), q), c4), q), c5),
                      A_(M_(A_(M_(A_(M_(A_(M_(d0, q), d1), q), d2), q), d3), q), 1.0));
    }
    else if (p <= 0.97575)
    {
        q              = __dsub_rn(p, 0.5);
        const double s = M_(q, q);
        r = __ddiv_rn(M_(A_(M_(A_(M_(A_(M_(A_(M_(A_(M_(a0, s), a1), s), a2), s), a3), s), a4), s), a5), q),
                      A_(M_(A_(M_(A_(M_(A_(M_(A_(M_(b0, s), b1), s), b2), s), b3), s), b4), s), 1.0));
    }
    else
    {
        q = sqrt(M_(-2.0, log(__dsub_rn(1.0, p))));
        r = -__ddiv_rn(A_(M_(A_(M_(A_(M_(A_(M_(A_(M_(c0, q), c1), q), c2), q), c3), q), c4), q), c5),
                       A_(M_(A_(M_(A_(M_(A_(M_(d0, q), d1), q), d2), q), d3), q), 1.0));
    }
    r = __ddiv_rn(r, sqrt(2.0));
    r = __dsub_rn(r, M_(M_(M_(__dsub_rn(erf(r), x), sqrt(3.14159265358979323846)), 0.5), exp(M_(r, r))));
#undef M_
#undef A_
    return r;
}

// zt[t] = sqrt(2) * erfinv(2 p - 1), p = (t + 0.5) / T (lib/gcmi.cpp:133-136).
__global__ void probit_table_kernel(int T, double* __restrict__ zt)
{
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= T)
        return;
    const double p = __ddiv_rn(__dadd_rn((double)t, 0.5), (double)T);
    zt[t]          = __dmul_rn(sqrt(2.0), acklam_erfinv(__dsub_rn(__dmul_rn(2.0, p), 1.0)));
}

// Longest series the shared-memory sort below takes (next_pow2(T) * 12 bytes).
constexpr int kCopulaSortMax = 16384;

// One CTA per component: bitonic sort of (value, frame) in shared memory,
// then midrank averaging of the probit scores over runs of equal values
// (lib/gcmi.cpp:113-143).  Requires next_pow2(T) * 12 bytes of shared memory
// (P >= 64).  A warp's threads take 32 neighbouring pairs, so the steps of
// stride 32 and below stay inside its 64 entries and need no CTA barrier (51
// of the 66 steps at 2048 entries): 247 x 2000 copulas 150 -> 131 us.
__global__ void __launch_bounds__(512) copula_kernel(const double* __restrict__ xyz, int T, int P,
                                                     const double* __restrict__ zt, double* __restrict__ Z,
                                                     int* __restrict__ status)
{
    extern __shared__ unsigned char smem_raw[];
    double*       val  = reinterpret_cast<double*>(smem_raw);
    int*          idx  = reinterpret_cast<int*>(val + P);
    const int     comp = blockIdx.x;
    const double* src  = xyz + (size_t)(comp / 3) * T * 3 + comp % 3;
    bool          bad  = false;
    for (int t = threadIdx.x; t < P; t += blockDim.x)
    {
        const double v = t < T ? src[(size_t)t * 3] : __longlong_as_double(0x7ff0000000000000LL);
        bad |= t < T && !isfinite(v);
        val[t] = v;
        idx[t] = t < T ? t : -1;
    }
    // a value that is not finite is not ranked: the padding (frame -1) would come
    // before it in the order, and its score has no place
    if (__syncthreads_or(bad))
    {
        if (threadIdx.x == 0)
            atomicOr(status, kStatNonFinite);
        return;
    }
    for (int k = 2; k <= P; k <<= 1)
        for (int j = k >> 1; j > 0; j >>= 1)
        {
            for (int p = threadIdx.x; p < P / 2; p += blockDim.x)
            {
                const int    t = 2 * p - (p & (j - 1)), u = t + j; // pair p of the step
                const bool   up = (t & k) == 0;
                const double vt = val[t], vu = val[u];
                if ((vt > vu) == up)
                {
                    val[t] = vu;
                    val[u] = vt;
                    const int it = idx[t];
                    idx[t]       = idx[u];
                    idx[u]       = it;
                }
            }
            // the next step's entries: the warp's own while its stride (j / 2, or
            // k for the next merge's first) is at most 32
            if (j > 32 || (j == 1 && k > 32))
                __syncthreads();
            else
                __syncwarp();
        }
    __syncthreads();
    double* z = Z + (size_t)comp * T;
    for (int r = threadIdx.x; r < T; r += blockDim.x)
    {
        if (r > 0 && val[r] == val[r - 1])
            continue; // not the start of a run
        int s = r + 1;
        while (s < T && val[s] == val[r])
            ++s;
        double avg = 0.0;
        for (int t = r; t < s; ++t)
            avg = __dadd_rn(avg, zt[t]);
        avg = __ddiv_rn(avg, (double)(s - r));
        for (int t = r; t < s; ++t)
            z[idx[t]] = avg;
    }
}

// The same copula scores for series too long to sort in shared memory: a
// frame's run of equal values starts at rank r = #{g : x_g < x_f} and holds
// m = #{g : x_g == x_f} frames, so its score is the average of zt[r .. r+m)
// summed in rank order, as in the sorted form.  Grid (frame blocks,
// components); the component's values pass through shared memory in tiles.
constexpr int kCopulaTile = 4096;

__global__ void __launch_bounds__(256) copula_count_kernel(const double* __restrict__ xyz, int T,
                                                           const double* __restrict__ zt, double* __restrict__ Z,
                                                           int* __restrict__ status)
{
    __shared__ double tile[kCopulaTile];
    const int     comp = blockIdx.y;
    const double* src  = xyz + (size_t)(comp / 3) * T * 3 + comp % 3;
    const int     f    = blockIdx.x * blockDim.x + threadIdx.x;
    const double  v    = f < T ? src[(size_t)f * 3] : 0.0;
    if (!isfinite(v))
        atomicOr(status, kStatNonFinite);
    int lt = 0, eq = 0;
    for (int t0 = 0; t0 < T; t0 += kCopulaTile)
    {
        const int n = min(kCopulaTile, T - t0);
        __syncthreads(); // the previous tile is consumed
        for (int e = threadIdx.x; e < n; e += blockDim.x)
            tile[e] = src[(size_t)(t0 + e) * 3];
        __syncthreads();
        for (int e = 0; e < n; ++e)
        {
            const double u = tile[e];
            lt += u < v;
            eq += u == v;
        }
    }
    if (f >= T)
        return;
    double avg = 0.0;
    for (int t = lt; t < lt + eq; ++t)
        avg = __dadd_rn(avg, zt[t]);
    Z[(size_t)comp * T + f] = __ddiv_rn(avg, (double)eq);
}

// Co-moment blocks b = hi (hi + 1) / 2 + lo (lo <= hi): 9 sums over frames in
// order.  A CTA takes TILE x TILE atom pairs, ROWS hi atoms per thread (two
// halve the shared-memory reads, which else take as long as the arithmetic);
// the tile's 2 TILE atoms pass through shared memory 8 frames at a time, atoms side by side (the
// lanes of a warp read neighbouring lo atoms and two hi atoms), copied
// asynchronously three stages ahead.  SERIES: V holds each
// component's series [3 natoms][T]; otherwise frames of xyz [natoms][T][3].
//
// Bound by the FP64 pipe (9 multiplications and 9 additions per pair and
// frame, which the reference's rounding forbids to fuse) and, with few
// tiles, by one SM's share of it: T * 72 cycles for a 16 x 16 tile.  One
// thread per block reading frame-major rows from L2 took 570 us at 247 x 2000
// and 1660 us at 600 x 4000, after a 54 us transposition; now
// 190 and 1300 us (10 T FP64 operations/s).
constexpr int kMomentFrames = 8; // frames per stage
constexpr int kMomentStages = 4;

template <int TILE, int ROWS, bool SERIES>
__global__ void __launch_bounds__(TILE * TILE / ROWS) comoment_kernel(const double* __restrict__ V, int natoms, int T,
                                                                      double* __restrict__ blk, int* __restrict__ status)
{
    constexpr int F = kMomentFrames, kThreads = TILE * TILE / ROWS, kElems = 2 * TILE * 3 * F, kRow = 2 * TILE + 1;
    constexpr int kPer = kElems / kThreads;
    static_assert(kElems % kThreads == 0, "whole elements per thread");
    __shared__ double buf[kMomentStages][F * 3][kRow]; // [frame * 3 + component][lo atoms, hi atoms]
    const int tid = threadIdx.x, tx = tid % TILE, ty = tid / TILE;
    // tile pair index -> (th, tl), tl <= th
    int th = (int)((sqrtf(8.0f * (float)blockIdx.x + 1.0f) - 1.0f) * 0.5f);
    while (th * (th + 1) / 2 > (int)blockIdx.x)
        --th;
    while ((th + 1) * (th + 2) / 2 <= (int)blockIdx.x)
        ++th;
    const int tl = (int)blockIdx.x - th * (th + 1) / 2;
    // this thread's elements of a stage: consecutive threads take consecutive
    // addresses of one atom's frames
    const double* src[kPer];
    unsigned      dst[kPer];
    int           fr[kPer];
#pragma unroll
    for (int k = 0; k < kPer; ++k)
    {
        const int e = tid + k * kThreads, at = e / (3 * F), r = e - at * 3 * F;
        const int f = SERIES ? r % F : r / 3, d = SERIES ? r / F : r - r / 3 * 3;
        const int a = min(at < TILE ? tl * TILE + at : th * TILE + at - TILE, natoms - 1);
        src[k]      = SERIES ? V + ((size_t)a * 3 + d) * T + f : V + ((size_t)a * T + f) * 3 + d;
        dst[k]      = (unsigned)__cvta_generic_to_shared(&buf[0][f * 3 + d][at]);
        fr[k]       = f;
    }
    const int chunks = (T + F - 1) / F;
    auto      fetch  = [&](int c) {
        if (c < chunks)
        {
            const unsigned stage = (unsigned)(c % kMomentStages) * (unsigned)sizeof(buf[0]);
#pragma unroll
            for (int k = 0; k < kPer; ++k)
                if (c * F + fr[k] < T)
                    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(dst[k] + stage),
                                 "l"(src[k] + (size_t)c * F * (SERIES ? 1 : 3))
                                 : "memory");
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    constexpr int kStep = TILE / ROWS; // a thread's hi atoms: ty, ty + kStep, ...
    double        acc[ROWS][9];
#pragma unroll
    for (int h = 0; h < ROWS; ++h)
#pragma unroll
        for (int e = 0; e < 9; ++e)
            acc[h][e] = 0.0;
    bool bad = false;
#pragma unroll
    for (int c = 0; c < kMomentStages - 1; ++c)
        fetch(c);
    for (int c = 0; c < chunks; ++c)
    {
        // this thread's part of stage c has arrived, then everyone's; the stage
        // fetched next was read in the round before the barrier
        asm volatile("cp.async.wait_group %0;" ::"n"(kMomentStages - 2) : "memory");
        __syncthreads();
        fetch(c + kMomentStages - 1);
        const double(*b)[kRow] = buf[c % kMomentStages];
        const int n            = min(F, T - c * F);
        // a frame's values are read while the frame before it is summed
        double l[2][3], v[2][ROWS][3];
        auto   read = [&](int f, int w) {
#pragma unroll
            for (int d = 0; d < 3; ++d)
            {
                l[w][d] = b[f * 3 + d][tx];
#pragma unroll
                for (int h = 0; h < ROWS; ++h)
                    v[w][h][d] = b[f * 3 + d][TILE + ty + h * kStep];
            }
        };
        read(0, 0);
#pragma unroll
        for (int f = 0; f < F; ++f)
        {
            if (f + 1 < F)
                read(f + 1, (f + 1) & 1); // behind the last frame: stale values, not used
            if (f < n)
#pragma unroll
                for (int h = 0; h < ROWS; ++h)
#pragma unroll
                    for (int r = 0; r < 3; ++r)
#pragma unroll
                        for (int d = 0; d < 3; ++d)
                            acc[h][r * 3 + d] =
                                __dadd_rn(acc[h][r * 3 + d], __dmul_rn(l[f & 1][r], v[f & 1][h][d]));
        }
        if (status && tl == th) // every atom is in one tile of the diagonal
            for (int f = 0; f < n; ++f)
#pragma unroll
                for (int d = 0; d < 3; ++d)
                    bad |= !isfinite(b[f * 3 + d][tx]);
    }
    if (status && bad)
        atomicOr(status, kStatNonFinite);
#pragma unroll
    for (int h = 0; h < ROWS; ++h)
    {
        const int lo = tl * TILE + tx, hi = th * TILE + ty + h * kStep;
        if (lo <= hi && hi < natoms)
        {
            double* o = blk + ((size_t)hi * (hi + 1) / 2 + lo) * 9;
#pragma unroll
            for (int e = 0; e < 9; ++e)
                o[e] = acc[h][e];
        }
    }
}

// Determinant by LU with partial pivoting (lib/correlation_core.cpp:49-98,
// lib/gcmi.cpp:152-184; the two differ only in a store that never feeds
// the determinant).
__device__ double lu_det(double* m, int n)
{
    double sign = 1.0;
    for (int col = 0; col < n; ++col)
    {
        int    pivot = col;
        double best  = fabs(m[col * n + col]);
        for (int row = col + 1; row < n; ++row)
        {
            const double v = fabs(m[row * n + col]);
            if (v > best)
            {
                best  = v;
                pivot = row;
            }
        }
        if (best == 0.0)
            return 0.0;
        if (pivot != col)
        {
            for (int j = 0; j < n; ++j)
            {
                const double t   = m[col * n + j];
                m[col * n + j]   = m[pivot * n + j];
                m[pivot * n + j] = t;
            }
            sign = -sign;
        }
        const double diag = m[col * n + col];
        for (int row = col + 1; row < n; ++row)
        {
            const double factor = __ddiv_rn(m[row * n + col], diag);
            for (int j = col + 1; j < n; ++j)
                m[row * n + j] = __dsub_rn(m[row * n + j], __dmul_rn(factor, m[col * n + j]));
        }
    }
    double det = sign;
    for (int i = 0; i < n; ++i)
        det = __dmul_rn(det, m[i * n + i]);
    return det;
}

__device__ __forceinline__ long block_index(long lo, long hi) { return hi * (hi + 1) / 2 + lo; }

// entropy (lib/correlation_core.cpp:100-111).
__device__ double gauss_entropy(double* m, int n, double log2pi)
{
    const double det = lu_det(m, n);
    if (det <= 0.0)
        return 0.0;
    return __dmul_rn(0.5, __dadd_rn(__dmul_rn((double)n, __dadd_rn(1.0, log2pi)), log(det)));
}

__global__ void pair_logdet_kernel(const double* __restrict__ blk, int natoms, int T, int mode, double log2pi,
                                   double* __restrict__ mat)
{
    const long np = (long)natoms * (natoms - 1) / 2;
    const long p  = blockIdx.x * (long)blockDim.x + threadIdx.x;
    if (p < natoms)
        mat[(size_t)p * natoms + p] = 2000.0;
    if (p >= np)
        return;
    int hi, lo;
    pair_from_index(p, &hi, &lo); // hi > lo
    const double* bll = blk + block_index(lo, lo) * 9;
    const double* bhh = blk + block_index(hi, hi) * 9;
    const double* blh = blk + block_index(lo, hi) * 9; // sum V_lo,r * V_hi,c
    double        mi;
    if (mode == 0)
    {
        // gauss_corrmatrix iterates a1 < a2: first = a1 = lo, second = hi.
        double first[9], second[9], comb[36];
        for (int r = 0; r < 3; ++r)
            for (int c = 0; c < 3; ++c)
            {
                first[r * 3 + c]          = __ddiv_rn(bll[r * 3 + c], (double)T);
                second[r * 3 + c]         = __ddiv_rn(bhh[r * 3 + c], (double)T);
                const double cr           = __ddiv_rn(blh[r * 3 + c], (double)T);
                comb[r * 6 + c]           = first[r * 3 + c];
                comb[(r + 3) * 6 + c + 3] = second[r * 3 + c];
                comb[r * 6 + c + 3]       = cr;
                comb[(c + 3) * 6 + r]     = cr;
            }
        const double e1 = gauss_entropy(first, 3, log2pi);
        const double e2 = gauss_entropy(second, 3, log2pi);
        mi              = __dsub_rn(__dadd_rn(e1, e2), gauss_entropy(comb, 6, log2pi));
    }
    else
    {
        // gcmi_pair(z, N, a1, a2) with a1 = hi > a2 = lo: v = [hi, lo].
        const double invN = __ddiv_rn(1.0, (double)T);
        double       c6[36], c1[9], c2[9];
        for (int r = 0; r < 3; ++r)
            for (int c = 0; c < 3; ++c)
            {
                c6[r * 6 + c]           = __dmul_rn(bhh[r * 3 + c], invN);
                c6[(r + 3) * 6 + c + 3] = __dmul_rn(bll[r * 3 + c], invN);
                c6[r * 6 + c + 3]       = __dmul_rn(blh[c * 3 + r], invN); // sum z_hi,r z_lo,c
                c6[(r + 3) * 6 + c]     = __dmul_rn(blh[r * 3 + c], invN); // sum z_lo,r z_hi,c
            }
        for (int r = 0; r < 3; ++r)
            for (int c = 0; c < 3; ++c)
            {
                c1[r * 3 + c] = c6[r * 6 + c];
                c2[r * 3 + c] = c6[(r + 3) * 6 + c + 3];
            }
        const double d1 = lu_det(c1, 3), d2 = lu_det(c2, 3), dJ = lu_det(c6, 6);
        if (d1 <= 0.0 || d2 <= 0.0 || dJ <= 0.0)
            mi = 0.0;
        else
            mi = __dmul_rn(0.5, __dsub_rn(__dadd_rn(log(d1), log(d2)), log(dJ)));
    }
    mat[(size_t)hi * natoms + lo] = mi;
    mat[(size_t)lo * natoms + hi] = mi;
}

void launch_copula(const double* xyz, int natoms, int T, double* zt, double* Z, int* status, cudaStream_t s)
{
    probit_table_kernel<<<(T + 127) / 128, 128, 0, s>>>(T, zt);
    if (T > kCopulaSortMax)
    {
        copula_count_kernel<<<dim3((unsigned)((T + 255) / 256), (unsigned)(natoms * 3)), 256, 0, s>>>(xyz, T, zt, Z,
                                                                                                     status);
        return;
    }
    int P = 64;
    while (P < T)
        P <<= 1;
    const size_t smem = (size_t)P * (sizeof(double) + sizeof(int));
    if (smem > 48 * 1024 && allow_dynamic_smem(copula_kernel) != cudaSuccess)
        return; // the caller finds the error
    const int threads = P / 2 < 512 ? P / 2 : 512;
    copula_kernel<<<natoms * 3, threads, smem, s>>>(xyz, T, P, zt, Z, status);
}

void launch_blocks(const double* V, bool series, int natoms, int T, double* blk, int* status, cudaStream_t s)
{
    // 16 x 16 tiles, or 8 x 8 where those would leave most SMs idle (fewer
    // than 74 tiles, up to 180 atoms)
    const long t16 = (natoms + 15) / 16, t8 = (natoms + 7) / 8;
    if (t16 * (t16 + 1) / 2 >= 74)
    {
        const unsigned g = (unsigned)(t16 * (t16 + 1) / 2);
        if (series)
            comoment_kernel<16, 2, true><<<g, 128, 0, s>>>(V, natoms, T, blk, status);
        else
            comoment_kernel<16, 2, false><<<g, 128, 0, s>>>(V, natoms, T, blk, status);
    }
    else
    {
        const unsigned g = (unsigned)(t8 * (t8 + 1) / 2);
        if (series)
            comoment_kernel<8, 1, true><<<g, 64, 0, s>>>(V, natoms, T, blk, status);
        else
            comoment_kernel<8, 1, false><<<g, 64, 0, s>>>(V, natoms, T, blk, status);
    }
}

void launch_pair_logdet(const double* blk, int natoms, int T, int mode, double log2pi, double* mat,
                        cudaStream_t s)
{
    long np = (long)natoms * (natoms - 1) / 2;
    if (np < natoms)
        np = natoms;
    pair_logdet_kernel<<<(unsigned)((np + 127) / 128), 128, 0, s>>>(blk, natoms, T, mode, log2pi, mat);
}

} // namespace gc

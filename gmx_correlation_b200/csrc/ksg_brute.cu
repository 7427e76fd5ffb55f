// KSG neighbour statistics by FP32 brute force with exact FP64 repair: for
// trajectories whose rows are too long to sort in shared memory, for single
// pairs, and for callers without room for sorted rows.
//
// Same counts as ksg_exact.cu (mir_xnyn, lib/kraskov.cpp:1228-1331).  A warp
// handles Q queries of one pair at a time; the pair's frames pass through
// shared memory as centred FP32 coordinates (x32 = fl32(x64 - c), c the
// component midrange, so |d32 - d64| <= eps_a for the marginal distances of
// atom a, see ksg_fast.cu), each staged frame serving all of the CTA's
// queries.  Three passes over the frames:
//
//   1. histogram of the joint distances (256 buckets of 2^18 float ulps, the
//      top one holding the largest possible distance): the bucket of the k-th
//      value.  Where that lies 8 octaves and more below the top (an atom with a
//      frame or a stretch of frames far off), the buckets move down and the
//      frames are counted again.  A bucket with more than kBfRefine values is
//      split by a further histogram.
//   2. the values below the bucket are counted and their marginal maxima
//      taken; the bucket's values, and 2 eps around it, are listed.  The
//      k-th value by rank, the values within 2 eps of it ordered in FP64 with
//      the grid-scan tie order, the maxima over all members.
//   3. marginal distances below each maximum are counted, those within 2 eps
//      listed and settled in FP64.
//
// Where more marginal distances lie within 2 eps than are listed (coordinates
// stored with few digits: many equal distances), the frames are looked at twice
// more for them.  With k frames at distance zero (repeated frames) the counts are
// those of the marginal distances of zero.  A query the scheme cannot settle (too
// many joint values near a bound, a k-th distance near zero, coordinates FP32 does
// not hold) takes the exact FP64 routine.
//
// The exact FP64 kernel evaluates every distance in about seven FP64 passes
// (radix selection); measured against it on one B200: 28 pairs of 20,001
// frames, k = 50: 282 -> 27.7 ms; 1128 pairs of 901 frames, k = 20: 20.0 ->
// 4.0 ms; one pair of 2000 frames, k = 100: 764 -> 42 us.

#include "gc_common.cuh"
#include "gc_internal.h"
#include "ksg_device.cuh"
#include "ksg_exact_query.cuh"

namespace gc {

namespace {

constexpr int kBfBins   = 256;
constexpr int kBfShift  = 18;  // bucket width in float ulps, log2
constexpr int kBfSplit  = 8;   // a split bucket: 2^8 parts
constexpr int kBfRefine = 40;  // values in a bucket beyond which it is split
constexpr int kBfList   = 64;  // listed values per query
constexpr int kBfNear   = 16;  // listed marginal distances per query and side

// What a warp keeps per query between the passes.
struct BfQuery
{
    unsigned lo, hi;         // bits of the bucket's edges [lo, hi)
    float    inlo, bandhi;   // the band: the bucket and 2 eps around it
    float    lower, upper;   // k-th value -+ 2 eps
    float    top[2];         // marginal maxima over the members
    int      code;           // float code of the lowest bucket
    int      open;           // the k-th value lies below it: counted again
    int      below;          // frames below the bucket, the query's own included
    int      nlist, nnear[2];
    int      n[2];           // marginal distances below 2 eps of the maxima, the query's own included
    int      state;          // 0: running, 1: left to the FP64 routine, 2: no query, 3: k-th distance near zero
};

// Both sums of two packed FP32 additions (round to nearest, as the single ones).
__device__ __forceinline__ float2 add2(const float2 a, const float2 b)
{
    float2 r;
    asm("{\n\t.reg .b64 x, y, z;\n\tmov.b64 x, {%2, %3};\n\tmov.b64 y, {%4, %5};\n\tadd.rn.f32x2 z, x, y;\n\t"
        "mov.b64 {%0, %1}, z;\n\t}"
        : "=f"(r.x), "=f"(r.y)
        : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
    return r;
}

__host__ __device__ constexpr size_t bf_warp_bytes(int q)
{
    // histogram, later the list (value, frame); near frames; query states
    return (size_t)q * (kBfBins * 4 + 2 * kBfNear * 4 + sizeof(BfQuery));
}

} // namespace

// Midrange of every component and the atom's FP32 error bound (as ksg_x32_kernel;
// infinite where FP32 does not hold the centred coordinates).
__global__ void __launch_bounds__(256) ksg_range_kernel(const double* __restrict__ X, int T, double* __restrict__ mid,
                                                        float* __restrict__ eps_atom)
{
    __shared__ double s_lo[8], s_hi[8];
    __shared__ double s_R;
    const int a = blockIdx.x, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (threadIdx.x == 0)
        s_R = 0.0;
    for (int d = 0; d < 3; ++d)
    {
        const double* r  = X + (size_t)(a * 3 + d) * T;
        double        lo = r[0], hi = lo;
        for (int f = threadIdx.x; f < T; f += 256)
        {
            const double v = r[f];
            lo             = fmin(lo, v);
            hi             = fmax(hi, v);
        }
        lo = -warp_max(-lo);
        hi = warp_max(hi);
        __syncthreads(); // the previous component is consumed
        if (lane == 0)
        {
            s_lo[warp] = lo;
            s_hi[warp] = hi;
        }
        __syncthreads();
        if (threadIdx.x == 0)
        {
            for (int w = 1; w < 8; ++w)
            {
                lo = fmin(lo, s_lo[w]);
                hi = fmax(hi, s_hi[w]);
            }
            const double c = 0.5 * (lo + hi), R = fmax(hi - c, c - lo);
            mid[a * 3 + d] = c;
            // rows may hold anything (gc_ksg_pair): beyond FP32, or with no
            // midrange, no bound holds, and with an infinite one every query of
            // the atom's pairs is left to the FP64 routine
            s_R = R < 1e38 ? fmax(s_R, R) : __longlong_as_double(0x7ff0000000000000LL);
        }
    }
    if (threadIdx.x == 0)
        eps_atom[a] = __double2float_ru(s_R * (1.0 + 0x1p-40) * 0x1p-21) + 1e-30f;
}

// Bound by issue slots: 20-23 instructions per distance and pass, 2 of 3
// issue slots used.  Q:
// queries per warp; chunk: frames staged at a time (all of them when they
// fit, then they are staged once).
template <int Q>
__global__ void __launch_bounds__(512) ksg_brute_kernel(const double* __restrict__ X, const double* __restrict__ mid,
                                                        const float* __restrict__ eps_atom, int T, int K,
                                                        long pair_begin, long pair_count,
                                                        const int2* __restrict__ pair_ab, int nqb, int chunk, int box,
                                                        int rank_shift, uint32_t* __restrict__ cnt,
                                                        uint32_t* __restrict__ cnt_y)
{
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int  warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nwarps = blockDim.x >> 5;
    const long pl = (long)blockIdx.x / nqb;
    const int  qb = (int)((long)blockIdx.x - pl * nqb);
    if (pl >= pair_count)
        return;
    int a1, a2;
    if (pair_ab)
    {
        a1 = pair_ab[pl].x;
        a2 = pair_ab[pl].y;
    }
    else
        pair_from_index(pair_begin + pl, &a1, &a2);
    // staged component d of frame j: (a1's, a2's) at st[d * chunk + j]
    float2*        st   = reinterpret_cast<float2*>(smem_raw);
    unsigned char* wmem = smem_raw + (size_t)3 * chunk * sizeof(float2) + (size_t)warp * bf_warp_bytes(Q);
    unsigned*      hist = reinterpret_cast<unsigned*>(wmem);              // [Q][kBfBins]
    unsigned*      near = hist + Q * kBfBins;                             // [Q][2][kBfNear] frames
    BfQuery*       qs   = reinterpret_cast<BfQuery*>(near + Q * 2 * kBfNear); // [Q]
    auto list_v = [&](int q, int e) -> float& { return reinterpret_cast<float*>(hist)[q * kBfBins + e]; };
    auto list_j = [&](int q, int e) -> unsigned& { return hist[q * kBfBins + kBfList + e]; };
    constexpr unsigned kMember = 1u << 31; // flag of a listed frame that is one of the k nearest

    const double* xa = X + (size_t)a1 * 3 * T;
    const double* xb = X + (size_t)a2 * 3 * T;
    double        c[6];
#pragma unroll
    for (int d = 0; d < 3; ++d)
    {
        c[d]     = mid[a1 * 3 + d];
        c[3 + d] = mid[a2 * 3 + d];
    }
    const float ea = eps_atom[a1], eb = eps_atom[a2], e2 = __fmul_ru(2.0f, fmaxf(ea, eb));
    // code of the largest possible distance 2 R: R <= eps 2^21
    const int ctop = (int)(__float_as_uint(fmaxf(ea, eb) * 4194304.0f * 1.0001f) >> kBfShift), cbase = ctop - (kBfBins - 1);
    auto x32 = [&](int d, int j) -> float2 {
        return make_float2((float)(xa[(size_t)d * T + j] - c[d]), (float)(xb[(size_t)d * T + j] - c[3 + d]));
    };
    // FP32 marginal distances of query i to frame j, from the rows
    auto dist32 = [&](int i, int j, float& dx, float& dy) {
        dx = dy = 0.0f;
#pragma unroll
        for (int d = 0; d < 3; ++d)
        {
            const float2 u = x32(d, i), w = x32(d, j);
            dx             = fmaxf(dx, fabsf(u.x - w.x));
            dy             = fmaxf(dy, fabsf(u.y - w.y));
        }
    };
    const int i0 = (qb * nwarps + warp) * Q;
    // the queries' coordinates, negated: x - q is the packed sum x + (-q)
    float2    q3[Q][3];
#pragma unroll
    for (int q = 0; q < Q; ++q)
    {
        const int i = min(i0 + q, T - 1);
#pragma unroll
        for (int d = 0; d < 3; ++d)
        {
            const float2 u = x32(d, i);
            q3[q][d]       = make_float2(-u.x, -u.y);
        }
        if (lane == 0)
        {
            qs[q].state = i0 + q < T ? 0 : 2;
            qs[q].code  = cbase;
        }
    }
    const bool whole = chunk >= T;
    // fn(j, q, dx, dy) for every frame and query; every thread of the CTA calls it
    bool staged  = false;
    auto frames = [&](auto&& fn) {
        for (int f0 = 0; f0 < T; f0 += chunk)
        {
            const int n = min(chunk, T - f0);
            if (!(whole && staged))
            {
                __syncthreads(); // the previous frames are consumed
                for (int e = threadIdx.x; e < n; e += blockDim.x)
#pragma unroll
                    for (int d = 0; d < 3; ++d)
                        st[d * chunk + e] = x32(d, f0 + e);
                __syncthreads();
                staged = true;
            }
            for (int e = lane; e < n; e += 32)
            {
                const float2 x0 = st[e], x1 = st[chunk + e], x2 = st[2 * chunk + e];
#pragma unroll
                for (int q = 0; q < Q; ++q)
                {
                    const float2 d0 = add2(x0, q3[q][0]), d1 = add2(x1, q3[q][1]), d2 = add2(x2, q3[q][2]);
                    fn(f0 + e, q, fmaxf(fmaxf(fabsf(d0.x), fabsf(d1.x)), fabsf(d2.x)),
                       fmaxf(fmaxf(fabsf(d0.y), fabsf(d1.y)), fabsf(d2.y)));
                }
            }
        }
    };
    auto clear = [&]() {
        for (int e = lane; e < Q * kBfBins; e += 32)
            hist[e] = 0u;
        __syncwarp();
    };
    // the bucket of rank k (of the frames counted so far and the query's own): its
    // index, the number below it and in it
    auto find = [&](const unsigned* h, int rank, int& bin, int& below, int& in) {
        unsigned v[kBfBins / 32], s = 0;
#pragma unroll
        for (int b = 0; b < kBfBins / 32; ++b)
        {
            v[b] = h[lane * (kBfBins / 32) + b];
            s += v[b];
        }
        unsigned incl = s;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1)
        {
            const unsigned y = __shfl_up_sync(kFull, incl, o);
            if (lane >= o)
                incl += y;
        }
        unsigned       acc   = incl - s;
        const bool     here  = acc < (unsigned)rank && (unsigned)rank <= incl;
        const unsigned owner = __ballot_sync(kFull, here);
        int            mb = -1, ml = 0, mi = 0;
        if (here)
        {
#pragma unroll
            for (int b = 0; b < kBfBins / 32; ++b)
            {
                if (mb < 0 && acc + v[b] >= (unsigned)rank)
                {
                    mb = lane * (kBfBins / 32) + b;
                    ml = (int)acc;
                    mi = (int)v[b];
                }
                acc += v[b];
            }
        }
        const int src = owner ? __ffs(owner) - 1 : 0;
        bin           = __shfl_sync(kFull, mb, src);
        below         = __shfl_sync(kFull, ml, src);
        in            = __shfl_sync(kFull, mi, src);
    };

    // ---- pass 1: the bucket of the k-th value --------------------------------
    clear();
    frames([&](int, int q, float dx, float dy) {
        const int b = (int)(__float_as_uint(fmaxf(dx, dy)) >> kBfShift) - cbase;
        atomicAdd(&hist[q * kBfBins + min(max(b, 0), kBfBins - 1)], 1u);
    });
    __syncwarp();
    bool split = false, lower = false; // a bucket of this warp has to be split, a query counted again below
    auto bucket = [&](int q) {
        int bin, below, in;
        find(hist + q * kBfBins, K + 1, bin, below, in); // the query itself is the first, in bucket 0
        const int  code = qs[q].code;
        const bool down = qs[q].state == 0 && bin == 0 && code > kBfBins &&
                          __uint_as_float((unsigned)code << kBfShift) > 32.0f * e2; // buckets wider than 2 eps
        __syncwarp();
        if (lane == 0)
        {
            BfQuery& u = qs[q];
            u.below    = below;
            u.lo       = (unsigned)(max(bin, 0) + code) << kBfShift;
            u.hi       = u.lo + (1u << kBfShift);
            u.nlist    = in;
            u.open     = down;
            if (down)
                u.code = code - (kBfBins - 1); // the lowest bucket becomes the top one
            else if (u.state == 0 && (bin < 1 || code < 1))
                u.state = bin == 0 ? 3 : 1;
        }
        lower |= down;
        split |= !down && in > kBfRefine;
    };
#pragma unroll 1
    for (int q = 0; q < Q; ++q)
        bucket(q);
    __syncwarp();
    const bool more = __syncthreads_or(split || lower);
    while (more && __syncthreads_or(lower))
    {
        clear();
        int base[Q];
#pragma unroll
        for (int q = 0; q < Q; ++q)
            base[q] = qs[q].code;
        frames([&](int, int q, float dx, float dy) {
            const int b = (int)(__float_as_uint(fmaxf(dx, dy)) >> kBfShift) - base[q];
            if (b < kBfBins)
                atomicAdd(&hist[q * kBfBins + max(b, 0)], 1u);
        });
        __syncwarp();
        lower = false;
#pragma unroll 1
        for (int q = 0; q < Q; ++q)
            if (qs[q].open)
                bucket(q);
        __syncwarp();
    }
    if (more && __syncthreads_or(split))
    {
        clear();
        unsigned lo[Q], hi[Q];
#pragma unroll
        for (int q = 0; q < Q; ++q)
        {
            lo[q] = qs[q].lo;
            hi[q] = qs[q].hi;
        }
        frames([&](int, int q, float dx, float dy) {
            const unsigned v = __float_as_uint(fmaxf(dx, dy));
            if (v >= lo[q] && v < hi[q])
                atomicAdd(&hist[q * kBfBins + ((v - lo[q]) >> (kBfShift - kBfSplit))], 1u);
        });
        __syncwarp();
#pragma unroll 1
        for (int q = 0; q < Q; ++q)
        {
            const int was = qs[q].nlist, before = qs[q].below;
            int       bin, below, in;
            find(hist + q * kBfBins, K + 1 - before, bin, below, in);
            __syncwarp();
            if (lane == 0 && qs[q].state == 0 && was > kBfRefine)
            {
                BfQuery& u = qs[q];
                u.lo += (unsigned)max(bin, 0) << (kBfShift - kBfSplit);
                u.hi = u.lo + (1u << (kBfShift - kBfSplit));
                u.below += below;
                if (bin < 0)
                    u.state = 1;
            }
        }
    }
    __syncwarp();

    // ---- pass 2: counts and maxima below the band, the band's values ---------
    float inlo[Q], bandhi[Q], mx[Q], my[Q];
    int   nb[Q];
#pragma unroll
    for (int q = 0; q < Q; ++q)
    {
        const float lo = __uint_as_float(qs[q].lo), hi = __uint_as_float(qs[q].hi);
        inlo[q]   = __fsub_rd(lo, e2);
        bandhi[q] = __fadd_ru(hi, e2);
        mx[q] = my[q] = 0.0f;
        nb[q]         = 0;
        __syncwarp();
        if (lane == 0)
        {
            qs[q].inlo   = inlo[q];
            qs[q].bandhi = bandhi[q];
            qs[q].nlist  = 0;
            // the error bound has to stay inside the bucket, the query's own frame below the band
            if (qs[q].state == 0 && !(e2 < hi - lo && inlo[q] > 0.0f))
                qs[q].state = 1;
        }
    }
    __syncwarp();
    frames([&](int j, int q, float dx, float dy) {
        const float v = fmaxf(dx, dy);
        if (v <= bandhi[q]) // few frames
        {
            if (v < inlo[q])
            {
                ++nb[q];
                mx[q] = fmaxf(mx[q], dx);
                my[q] = fmaxf(my[q], dy);
            }
            else
            {
                const int e = atomicAdd(&qs[q].nlist, 1);
                if (e < kBfList)
                {
                    list_v(q, e) = v;
                    list_j(q, e) = (unsigned)j;
                }
            }
        }
    });
    __syncwarp();
#pragma unroll
    for (int q = 0; q < Q; ++q)
    {
        const int   i = min(i0 + q, T - 1);
        const int   below = (int)__reduce_add_sync(kFull, (unsigned)nb[q]) - 1; // without the query itself
        const int   m = qs[q].nlist, r = K - below;
        const bool  run = qs[q].state == 0 && m <= kBfList && r >= 1 && r <= m;
        float       tx = mx[q], ty = my[q];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1)
        {
            tx = fmaxf(tx, __shfl_xor_sync(kFull, tx, o));
            ty = fmaxf(ty, __shfl_xor_sync(kFull, ty, o));
        }
        bool ok = run;
        if (run)
        {
            // two listed values a lane: their ranks (ties by index), the k-th value
            float v[2];
            int   rk[2] = {0, 0};
#pragma unroll
            for (int s = 0; s < 2; ++s)
                v[s] = s * 32 + lane < m ? list_v(q, s * 32 + lane) : __int_as_float(0x7f800000);
            for (int f = 0; f < m; ++f)
            {
                const float u = list_v(q, f);
#pragma unroll
                for (int s = 0; s < 2; ++s)
                    rk[s] += u < v[s] || (u == v[s] && f < s * 32 + lane);
            }
            float d32 = -1.0f;
#pragma unroll
            for (int s = 0; s < 2; ++s)
                if (s * 32 + lane < m && rk[s] == r - 1)
                    d32 = v[s];
#pragma unroll
            for (int o = 16; o > 0; o >>= 1)
                d32 = fmaxf(d32, __shfl_xor_sync(kFull, d32, o));
            const float lower = __fsub_rd(d32, e2), upper = __fadd_ru(d32, e2);
            bool        mem[2], amb[2];
            int         n_mem = 0, n_amb = 0;
#pragma unroll
            for (int s = 0; s < 2; ++s)
            {
                const bool in = s * 32 + lane < m;
                mem[s]        = in && v[s] < lower;
                amb[s]        = in && !mem[s] && v[s] <= upper;
                n_mem += __popc(__ballot_sync(kFull, mem[s]));
                n_amb += __popc(__ballot_sync(kFull, amb[s]));
            }
            const int need = r - n_mem;
            ok             = need >= 1 && need <= n_amb;
            if (ok && need < n_amb)
            {
                // order the values within 2 eps by (FP64 joint distance, scan rank)
                const ScanGrid     grid(box);
                unsigned long long kh[2], kl[2];
                int                ar[2] = {0, 0};
#pragma unroll
                for (int s = 0; s < 2; ++s)
                {
                    kh[s] = kl[s] = ~0ull;
                    if (amb[s])
                    {
                        const int j = (int)list_j(q, s * 32 + lane);
                        kh[s] = dbits(fmax(dist3r(xa, T, xa[i], xa[T + i], xa[2 * T + i], j),
                                           dist3r(xb, T, xb[i], xb[T + i], xb[2 * T + i], j)));
                        kl[s] = grid.rank(grid.qcell(xa[i]), grid.qcell(xb[i]), xa[j], xb[j], j, T);
                    }
                }
#pragma unroll
                for (int f = 0; f < 2; ++f)
                    for (int l = 0; l < 32; ++l)
                    {
                        const unsigned long long fh = __shfl_sync(kFull, kh[f], l), fl = __shfl_sync(kFull, kl[f], l);
#pragma unroll
                        for (int s = 0; s < 2; ++s)
                            ar[s] += fh < kh[s] || (fh == kh[s] && fl < kl[s]);
                    }
#pragma unroll
                for (int s = 0; s < 2; ++s)
                    amb[s] = amb[s] && ar[s] < need;
            }
            // the listed members' marginal distances
#pragma unroll
            for (int s = 0; s < 2; ++s)
                if (mem[s] || amb[s])
                {
                    const int j = (int)list_j(q, s * 32 + lane);
                    float     dx, dy;
                    dist32(i, j, dx, dy);
                    tx = fmaxf(tx, dx);
                    ty = fmaxf(ty, dy);
                    list_j(q, s * 32 + lane) |= kMember;
                }
#pragma unroll
            for (int o = 16; o > 0; o >>= 1)
            {
                tx = fmaxf(tx, __shfl_xor_sync(kFull, tx, o));
                ty = fmaxf(ty, __shfl_xor_sync(kFull, ty, o));
            }
            if (lane == 0)
            {
                qs[q].lower  = lower;
                qs[q].upper  = upper;
                qs[q].top[0] = tx;
                qs[q].top[1] = ty;
            }
        }
        if (lane == 0)
        {
            qs[q].nnear[0] = qs[q].nnear[1] = 0;
            if (qs[q].state == 0 && !ok)
                qs[q].state = 1;
        }
        __syncwarp();
    }

    // ---- pass 3: marginal distances below each maximum, those within 2 eps ---
    float lo_x[Q], hi_x[Q], lo_y[Q], hi_y[Q];
    int   nx[Q], ny[Q];
    const float e2a = __fmul_ru(2.0f, ea), e2b = __fmul_ru(2.0f, eb);
#pragma unroll
    for (int q = 0; q < Q; ++q)
    {
        const bool on = qs[q].state == 0;
        lo_x[q]       = on ? __fsub_rd(qs[q].top[0], e2a) : 0.0f;
        hi_x[q]       = on ? __fadd_ru(qs[q].top[0], e2a) : -1.0f;
        lo_y[q]       = on ? __fsub_rd(qs[q].top[1], e2b) : 0.0f;
        hi_y[q]       = on ? __fadd_ru(qs[q].top[1], e2b) : -1.0f;
        nx[q] = ny[q] = 0;
    }
    frames([&](int j, int q, float dx, float dy) {
        const bool bx = dx < lo_x[q], by = dy < lo_y[q], cx = !bx && dx <= hi_x[q], cy = !by && dy <= hi_y[q];
        nx[q] += bx;
        ny[q] += by;
        if (cx || cy)
        {
            if (cx)
            {
                const int e = atomicAdd(&qs[q].nnear[0], 1);
                if (e < kBfNear)
                    near[(q * 2 + 0) * kBfNear + e] = (unsigned)j;
            }
            if (cy)
            {
                const int e = atomicAdd(&qs[q].nnear[1], 1);
                if (e < kBfNear)
                    near[(q * 2 + 1) * kBfNear + e] = (unsigned)j;
            }
        }
    });
    __syncwarp();
    auto store = [&](int i, int n0, int n1) {
        const size_t at = (size_t)pl * T + i;
        if (cnt_y) // wide counts: n_x and n_y in separate planes
        {
            cnt[at]   = (uint32_t)n0;
            cnt_y[at] = (uint32_t)n1;
        }
        else
            cnt[at] = (uint32_t)n0 | ((uint32_t)n1 << 16);
    };
    // whether frame j is one of the k nearest of query q, from its joint distance
    auto member = [&](int q, int j, float v) -> bool {
        bool is = v < qs[q].lower;
        if (!is && v <= qs[q].upper) // one of the ordered values: listed as a member
            for (int e = 0; e < qs[q].nlist && !is; ++e)
                is = list_j(q, e) == ((unsigned)j | kMember);
        return is;
    };
    unsigned late = 0u; // queries the lists do not settle
#pragma unroll
    for (int q = 0; q < Q; ++q)
    {
        const int i = min(i0 + q, T - 1);
        int       n[2];
        n[0]    = (int)__reduce_add_sync(kFull, (unsigned)nx[q]);
        n[1]    = (int)__reduce_add_sync(kFull, (unsigned)ny[q]);
        bool ok = qs[q].state == 0 && qs[q].nnear[0] <= kBfNear && qs[q].nnear[1] <= kBfNear;
        if (lane == 0)
        {
            qs[q].n[0] = n[0];
            qs[q].n[1] = n[1];
        }
#pragma unroll
        for (int side = 0; side < 2; ++side)
        {
            const double* x  = side == 0 ? xa : xb;
            double        d  = -1.0;
            bool          is = false;
            if (ok && lane < qs[q].nnear[side])
            {
                const int j = (int)near[(q * 2 + side) * kBfNear + lane];
                if (j != i)
                {
                    d = dist3r(x, T, x[i], x[T + i], x[2 * T + i], j);
                    float dx, dy;
                    dist32(i, j, dx, dy);
                    is = member(q, j, fmaxf(dx, dy));
                }
            }
            const double best = warp_max(is ? d : -1.0);
            const int    add  = __popc(__ballot_sync(kFull, d >= 0.0 && d <= best));
            ok                = ok && best >= 0.0;
            // the query's own frame was counted when it lies below the bound
            n[side] += add - ((side == 0 ? lo_x[q] : lo_y[q]) > 0.0f ? 1 : 0);
        }
        if (ok && lane == 0)
            store(i, n[0], n[1]);
        late |= (unsigned)(!ok && qs[q].state != 2) << q;
        __syncwarp();
    }
#pragma unroll 1
    for (; late; late &= late - 1)
    {
        const int q = __ffs(late) - 1, i = min(i0 + q, T - 1);
        int       n[2] = {qs[q].n[0], qs[q].n[1]};
        bool      ok   = false;
        if (qs[q].state == 0)
        {
            // more marginal distances near a maximum than are listed, or no
            // member among them: the maximum, then the count
            ok = true;
#pragma unroll 1
            for (int side = 0; side < 2; ++side)
            {
                const double* x   = side == 0 ? xa : xb;
                const float   top = qs[q].top[side], e = side == 0 ? e2a : e2b;
                const float   lo = __fsub_rd(top, e), hi = __fadd_ru(top, e);
                // the frames to look at: those listed, or all
                const int     nl = qs[q].nnear[side], frames_end = nl <= kBfNear ? nl : T;
                double        best = -1.0;
                int           add  = 0;
#pragma unroll 1
                for (int pass = 0; pass < 2; ++pass)
                {
                    double m = -1.0;
                    for (int f = lane; f < frames_end; f += 32)
                    {
                        const int j = nl <= kBfNear ? (int)near[(q * 2 + side) * kBfNear + f] : f;
                        float     dx, dy;
                        dist32(i, j, dx, dy);
                        const float v = side == 0 ? dx : dy;
                        if (j == i || !(v >= lo && v <= hi) || (pass == 0 && !member(q, j, fmaxf(dx, dy))))
                            continue;
                        const double d = dist3r(x, T, x[i], x[T + i], x[2 * T + i], j);
                        m              = fmax(m, d);
                        add += pass != 0 && d <= best;
                    }
                    if (pass == 0)
                        best = warp_max(m);
                }
                ok      = ok && best >= 0.0;
                n[side] += (int)__reduce_add_sync(kFull, (unsigned)add) - (lo > 0.0f ? 1 : 0);
            }
        }
        else if (qs[q].state == 3)
        {
            // distances of zero: with k of the joint ones both maxima are zero
            int z = 0, zx = 0, zy = 0;
            for (int j = lane; j < T; j += 32)
                if (j != i)
                {
                    const bool x0 = dist3r(xa, T, xa[i], xa[T + i], xa[2 * T + i], j) == 0.0;
                    const bool y0 = dist3r(xb, T, xb[i], xb[T + i], xb[2 * T + i], j) == 0.0;
                    zx += x0;
                    zy += y0;
                    z += x0 && y0;
                }
            n[0] = (int)__reduce_add_sync(kFull, (unsigned)zx);
            n[1] = (int)__reduce_add_sync(kFull, (unsigned)zy);
            ok   = (int)__reduce_add_sync(kFull, (unsigned)z) >= K;
        }
        if (!ok)
            exact_query_nxy(X, T, K, a1, a2, i, box, rank_shift, hist, lane, n[0], n[1]);
        if (lane == 0)
            store(i, n[0], n[1]);
        __syncwarp();
    }
}

size_t ksg_brute_scratch(int natoms) { return (size_t)natoms * (3 * sizeof(double) + sizeof(float)); }

void launch_ksg_brute(const double* X, int natoms, int T, int K, long pair_begin, long pair_count, uint32_t* cnt,
                      void* scratch, int sms, cudaStream_t s, const int2* pair_ab, uint32_t* cnt_y)
{
    double* mid = static_cast<double*>(scratch);
    float*  eps = reinterpret_cast<float*>(mid + (size_t)3 * natoms);
    ksg_range_kernel<<<natoms, 256, 0, s>>>(X, T, mid, eps);
    // Up to 2048 frames are staged once (48 KB, two CTAs of 8 warps an SM);
    // longer trajectories pass in chunks of 2048, for 16 warps at a time.  Few
    // queries: two per warp and four warps a CTA, so that every SM has work.
    constexpr int kChunk = 2048;
    const bool    small  = pair_count * T <= (long)sms * 64;
    const int     Q = small ? 2 : 4, warps = small ? 4 : (T <= kChunk ? 8 : 16), chunk = T < kChunk ? T : kChunk;
    const int  nqb   = (T + Q * warps - 1) / (Q * warps);
    const int  box   = ksg_box_count(T, K), shift = rank_top_shift(box, T);
    const size_t smem = (size_t)3 * chunk * sizeof(float2) + (size_t)warps * bf_warp_bytes(Q);
    auto         go   = [&](auto kernel) {
        if (allow_dynamic_smem(kernel) != cudaSuccess)
            return; // the caller finds the error
        kernel<<<(unsigned)(pair_count * nqb), warps * 32, smem, s>>>(X, mid, eps, T, K, pair_begin, pair_count, pair_ab,
                                                                     nqb, chunk, box, shift, cnt, cnt_y);
    };
    if (small)
        go(ksg_brute_kernel<2>);
    else
        go(ksg_brute_kernel<4>);
}

} // namespace gc

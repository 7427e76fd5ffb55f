// Walking one sorted distance row for 32 pairs at once (ksg_row_walk.cu,
// te_row_walk.cu).
//
// For one query frame, the joint value of the pair (a, b) at frame j is
// max(d_a(j), d_b(j)).  A warp walks the sorted row of atom a; its 32 lanes
// hold 32 different atoms b.  Every lane is at the same frame j at the same
// time, so d_b(j) comes from a tile in shared memory with a frame's 32
// values side by side: one wavefront for the 32 pairs, where a lane per
// query has to gather 12-byte coordinates from 32 different frames (about
// 9.5 wavefronts).  The k-th value is only bracketed here, so the tile holds
// one-byte bucket codes: bits(d) >> shift, relative to the tile's base code,
// clamped to 0 .. 255.
//
// The tile's row of frame j is permuted by XOR with a function of j: reads
// (32 lanes, one frame) take the same 32 bytes in any order, and a warp that
// fills one atom's column for 32 consecutive frames hits 32 different banks.
#pragma once

#include "gc_common.cuh"
#include "ksg_fast.h"

namespace gc {

// Byte offset of frame j's row; the value of lane l is at (offset ^ l).
__device__ __forceinline__ unsigned rw_row(unsigned j) { return (j << 5) | (j & 0x1Cu); }

__device__ __forceinline__ unsigned char rw_code(float d, int shift, int base)
{
    const int c = (int)(__float_as_uint(d) >> shift) - base;
    return (unsigned char)min(max(c, 0), 255);
}

// Work split of a CTA that fills a tile of ncol columns and nfr frames: units of
// one column and 32 * ahead frames, a lane's `ahead` loads in flight together.
// unit(c, j0) handles frames j0 + 32 e + lane of column c.  A column per warp
// with the loads as they come keeps 14 warps (a tile of 4999 frames) waiting
// for memory: the walk of 151 x 4999 takes 50.1 ms so, 43.3 in units with 4
// loads ahead, 42.2 with 8; the count of TE at 2000 frames 36.3, 35.7 and
// 35.0 ms.  The TE walk's two-row columns leave no registers for it (39.5 ms
// by column, 40.0 with 8).
template <class Unit>
__device__ __forceinline__ void rw_fill(int ncol, int nfr, int ahead, int warp, int nwarps, Unit&& unit)
{
    const int per = (nfr + 32 * ahead - 1) / (32 * ahead);
    int       c = warp / per, ch = warp - c * per;
    const int dc = nwarps / per, dch = nwarps - dc * per;
    while (c < ncol)
    {
        unit(c, ch * 32 * ahead);
        c += dc;
        ch += dch;
        if (ch >= per)
        {
            ch -= per;
            ++c;
        }
    }
}

// Bracket of the k-th joint value of one lane's pair.
struct RwBracket
{
    int  lev;    // window index of its bucket: codes w0 - 1 + lev; kWalkBuckets - 1 when beyond the window
    int  below;  // joint values in the buckets below
    int  walked; // row entries walked until the bucket was known
    bool wrapped; // a counter overflowed before: the bracket is not usable
};

// The warp walks the sorted row (4-entry groups Sg / Pg in runs, see row_group, Llen
// entries, NaN behind the last) until every live lane's k-th joint value is
// bracketed.  w0: the code of the row's own k-th value, a lower bound of
// every lane's k-th joint value; woff = w0 - 1 - base of the tile (0 .. 128,
// so the clamped code 255 lands on the top index).  Window index 0 holds the
// codes below w0 (fewer than K <= 255 entries, since they are also row
// entries below the k-th), index kWalkBuckets - 1 everything above the
// window; it is never read and cleared every 16 entries.  hist and stage are
// this warp's kRwHistBytes and kRwStageBytes of shared memory, 16-byte
// aligned.
//
// Bound by issue slots and the histogram's read-modify-write (two
// conflict-free wavefronts): about 13 instructions per entry and lane.  A lane
// whose bracket is known counts no further, or the entries that follow for the
// other lanes could overflow its counters: with stretches of frames 50 nm off,
// 100 atoms x 2000, k = 100, 1,017,000 queries went to the exact kernel for
// 485,000 and the matrix took 111 ms for 68.
__device__ __forceinline__ RwBracket rw_walk(const unsigned char* tile, const float4* __restrict__ Sg,
                                             const uint2* __restrict__ Pg, size_t gs, int rrun, int Llen, int K, int shift,
                                             int w0, int woff, bool live, unsigned char* hist, unsigned char* stage,
                                             int lane)
{
    constexpr int kTop = kWalkBuckets - 1;
    {
        uint4* h4 = reinterpret_cast<uint4*>(hist);
#pragma unroll
        for (int e = 0; e < kRwHistBytes / 512; ++e)
            h4[e * 32 + lane] = make_uint4(0u, 0u, 0u, 0u);
    }
    const unsigned lane4 = (unsigned)lane * 4u;
    // index b of this lane: byte b % 4 of word (b / 4) * 32 + lane, so the 32
    // lanes always hit 32 different banks
    auto at = [lane4](unsigned b) -> unsigned { return ((b << 5) & 0xF80u) | ((b & 3u) | lane4); };
    uint4*         so  = reinterpret_cast<uint4*>(stage);                 // [32] row offsets of 4 entries
    unsigned*      sc  = reinterpret_cast<unsigned*>(stage + kRwChunk * 4); // [32] window indices of 4 entries
    const int      ngr = (Llen + 3) >> 2;
    const float    nan = __int_as_float(0x7fc00000);
    float4         s4  = make_float4(nan, nan, nan, nan);
    uint2          j4  = make_uint2(0u, 0u);
    if (lane < ngr)
    {
        s4 = Sg[row_group(lane, gs, rrun)];
        j4 = Pg[row_group(lane, gs, rrun)];
    }
    RwBracket r{kTop, 0, Llen, false};
    bool      done = !live;
    int       run = 0, thr = 0;
    unsigned  wrap = 0u;
    auto      levels = [&](int upto, int walked) {
        for (; thr < upto; ++thr)
        {
            const int c = hist[at((unsigned)thr)];
            if (!done && run + c >= K)
            {
                done     = true;
                r.lev    = thr;
                r.below  = run;
                r.walked = walked;
            }
            run += c;
        }
    };
    for (int m0 = 0; m0 < Llen; m0 += kRwChunk)
    {
        auto idx = [&](float s) -> unsigned {
            return (unsigned)min(max((int)(__float_as_uint(s) >> shift) - w0 + 1, 0), kTop);
        };
        so[lane] = make_uint4(rw_row(j4.x & 0xFFFFu), rw_row(j4.x >> 16), rw_row(j4.y & 0xFFFFu), rw_row(j4.y >> 16));
        sc[lane] = idx(s4.x) | (idx(s4.y) << 8) | (idx(s4.z) << 16) | (idx(s4.w) << 24);
        __syncwarp();
        // the next chunk's groups are in flight while this one is counted
        const int g = (m0 + kRwChunk) / 4 + lane;
        s4          = make_float4(nan, nan, nan, nan);
        if (g < ngr)
        {
            s4 = Sg[row_group(g, gs, rrun)];
            j4 = Pg[row_group(g, gs, rrun)];
        }
        const int nsub = min(kRwChunk / 16, (Llen - m0 + 15) >> 4);
        for (int sub = 0; sub < nsub; ++sub)
        {
            const uint4 cv = *reinterpret_cast<const uint4*>(sc + sub * 4);
            int         d[16];
#pragma unroll
            for (int q = 0; q < 4; ++q)
            {
                const uint4 o = so[sub * 4 + q];
                d[q * 4 + 0]  = tile[o.x ^ (unsigned)lane];
                d[q * 4 + 1]  = tile[o.y ^ (unsigned)lane];
                d[q * 4 + 2]  = tile[o.z ^ (unsigned)lane];
                d[q * 4 + 3]  = tile[o.w ^ (unsigned)lane];
            }
#pragma unroll
            for (int q = 0; q < 16; ++q)
            {
                const unsigned w  = q < 4 ? cv.x : (q < 8 ? cv.y : (q < 12 ? cv.z : cv.w));
                const int      sx = (int)((w >> (8 * (q & 3))) & 0xFFu);
                const unsigned o  = at((unsigned)min(max(d[q] - woff, sx), kTop));
                const unsigned h  = (unsigned)hist[o] + 1u;
                hist[o]           = (unsigned char)h;
                wrap |= h;
            }
            hist[at(kTop)] = 0;
            levels((int)(cv.w >> 24), min(Llen, m0 + sub * 16 + 16));
            if (done) // the row goes on for the other lanes: this one counts above the window
                woff = -4 * kWalkBuckets;
            if (__all_sync(kFull, done))
            {
                r.wrapped = wrap > 255u;
                return r;
            }
        }
        __syncwarp(); // the stage is consumed
    }
    levels(kTop, Llen);
    r.wrapped = wrap > 255u;
    return r;
}

} // namespace gc

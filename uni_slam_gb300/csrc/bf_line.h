// bf_line.h — how the two brute-force matchers share their work out.
//
// A pair is its query blocks times the train set's tiles.  All blocks of all
// pairs, each with its tiles in order, form one line of tiles, and a CTA takes
// an equal contiguous share of it: whole blocks, and parts of the blocks that
// its ends cut.  The kept counts are known on the device alone, and whole
// blocks (or blocks cut into a fixed number of parts) come out uneven over
// the SMs: 4 pairs of 20000 features are 316 blocks for the 152 CTAs of k_bf_mma,
// 2.08 each, so a third of its launch waited for the last ones (637 us for it,
// 469 in equal shares).
//
// A cut block's parts leave one record (best, second, id, number of parts)
// per query each, which the emit merges.  A share is at least so long that no
// block has more than bf_splits parts, for which the batch has records;
// without records (bf_splits 1) a block goes as a whole to the CTA in whose
// share it starts.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include "uslam_internal.h"

namespace uslam {

__device__ __forceinline__ uint32_t bf_total_kept(const FrameDev& F) {
    uint32_t n = 0;
    for (int l = 0; l < F.levels; ++l) n += F.kept[l];
    return n;
}

struct BfLine {
    unsigned long long pos, end;  // this CTA's share
    unsigned long long share;
};

struct BfUnit {
    const PairDev* P;
    uint32_t blk;           // query block of the pair
    uint32_t tile, ntiles;  // train tiles [tile, tile + ntiles)
    uint32_t nq, nt;        // features of the pair's frames
    uint32_t part, parts;   // this part of the block's tiles, and their number
};

// s_pref[p] = tiles of the line before pair p (npairs + 1 entries), and the
// calling CTA's share.  For all threads of the CTA, which are whole warps;
// s_warp: 33 words.
template <int QUERIES, int TILE>
__device__ BfLine bf_line(const FrameDev* frames, const PairDev* pairs, const SegDev* psegs, int npairs,
                          unsigned long long* s_pref, unsigned long long* s_warp) {
    __shared__ uint32_t s_longest;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, warps = blockDim.x >> 5;
    const int per = (npairs + (int)blockDim.x - 1) / (int)blockDim.x, first = (int)threadIdx.x * per;
    auto tiles = [&](int p, uint32_t* longest) {
        const PairDev& P = pairs[psegs[p].frame];
        const uint32_t nt = (bf_total_kept(frames[P.curr]) + TILE - 1) / TILE;
        *longest = max(*longest, nt);
        return (unsigned long long)((bf_total_kept(frames[P.prev]) + QUERIES - 1) / QUERIES) * nt;
    };
    if (threadIdx.x == 0) s_longest = 0u;
    unsigned long long sum = 0, incl;
    uint32_t longest = 0;
    for (int k = 0; k < per; ++k)
        if (first + k < npairs) sum += tiles(first + k, &longest);
    incl = sum;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const unsigned long long v = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += v;
    }
    if (lane == 31) s_warp[warp] = incl;
    __syncthreads();
    if (longest) atomicMax(&s_longest, longest);
    unsigned long long run = incl - sum;
    for (int w = 0; w < warp; ++w) run += s_warp[w];
    for (int k = 0; k < per; ++k)
        if (first + k < npairs) {
            s_pref[first + k] = run;
            run += tiles(first + k, &longest);
        }
    if (threadIdx.x == 0) {
        unsigned long long total = 0;
        for (int w = 0; w < warps; ++w) total += s_warp[w];
        s_pref[npairs] = total;
    }
    __syncthreads();
    BfLine L;
    const unsigned long long total = s_pref[npairs];
    const int splits = npairs > 0 ? pairs[psegs[0].frame].bf_splits : 1;  // one number for all pairs
    L.share = (total + gridDim.x - 1) / gridDim.x;
    if (splits > 1) {
        const unsigned long long least = (s_longest + (uint32_t)splits - 2u) / ((uint32_t)splits - 1u);
        if (L.share < least) L.share = least;
    }
    if (L.share == 0) L.share = 1;
    L.pos = min(L.share * blockIdx.x, total);
    L.end = min(L.pos + L.share, total);
    if (splits <= 1) {
        // to the starts of blocks
        auto snap = [&](unsigned long long at) {
            if (at >= total) return total;
            int lo = 0, hi = npairs - 1;  // the largest p with s_pref[p] <= at: its line is not empty
            while (lo < hi) {
                const int mid = (lo + hi + 1) >> 1;
                if (s_pref[mid] <= at) lo = mid;
                else hi = mid - 1;
            }
            const uint32_t nt = (bf_total_kept(frames[pairs[psegs[lo].frame].curr]) + TILE - 1) / TILE;
            const uint32_t r = (uint32_t)((at - s_pref[lo]) % nt);
            return r ? at + (nt - r) : at;
        };
        L.pos = snap(L.pos);
        L.end = snap(L.end);
    }
    return L;
}

// The next unit of the share, if there is one.
template <int QUERIES, int TILE>
__device__ __forceinline__ bool bf_next(const FrameDev* frames, const PairDev* pairs, const SegDev* psegs, int npairs,
                                        const unsigned long long* s_pref, BfLine& L, BfUnit& u) {
    if (L.pos >= L.end) return false;
    int lo = 0, hi = npairs - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (s_pref[mid] <= L.pos) lo = mid;
        else hi = mid - 1;
    }
    u.P = &pairs[psegs[lo].frame];
    u.nq = bf_total_kept(frames[u.P->prev]);
    u.nt = bf_total_kept(frames[u.P->curr]);
    const uint32_t nt = (u.nt + TILE - 1) / TILE;
    const unsigned long long at = L.pos - s_pref[lo];
    u.blk = (uint32_t)(at / nt);
    const unsigned long long b0 = s_pref[lo] + (unsigned long long)u.blk * nt, b1 = b0 + nt;
    const unsigned long long stop = min(L.end, b1);
    u.tile = (uint32_t)(L.pos - b0);
    u.ntiles = (uint32_t)(stop - L.pos);
    u.part = 0u;
    u.parts = 1u;
    if (u.ntiles < nt) {
        const unsigned long long p0 = b0 / L.share;
        u.part = (uint32_t)(L.pos / L.share - p0);
        u.parts = (uint32_t)((b1 - 1) / L.share - p0) + 1u;
    }
    L.pos = stop;
    return true;
}

// Record of one query of a unit: distances (all ones: none) in the upper 24 bits.
__device__ __forceinline__ void bf_record(const BfUnit& u, size_t stride, size_t q, uint32_t bd, uint32_t sd, int32_t id) {
    *reinterpret_cast<uint4*>(u.P->bf_part + (u.part * stride + q) * 4u) = make_uint4(bd << 8, sd << 8, (uint32_t)id, u.parts);
}

}  // namespace uslam

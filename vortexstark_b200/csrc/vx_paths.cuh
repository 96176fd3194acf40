// Authentication paths rebuilt from a tree's stored levels.
//
// One (query, stored-level group) pair is the block of 2^k <= 16 nodes of one
// stored level (or leaves) around the query's node: re-hashing it gives the
// siblings at k consecutive heights.  Eight lanes share a pair, with the
// block's nodes in shared memory: at most two leaves per lane, then one
// compression per lane and level, and the block's root, which no path
// contains, is left out.  A thread per pair spends up to 31 dependent
// compressions and keeps its nodes in local memory; eight lanes spend 5.
#pragma once
#include <cstdint>

#include "vx_merkle.cuh"

namespace vx {

constexpr uint32_t kPathLanes = 8, kPathThreads = 128, kPathItems = kPathThreads / kPathLanes;
constexpr uint32_t kPathWords = 8 * 30 + 4;  // 16 + 8 + 4 + 2 nodes; items start 4 banks apart modulo 8

// The group g of the tree `lv` around leaf `idx`; leaf(i, h) hashes leaf i.
// p, sp: the paths of the leaf and of its sibling (p[1 + 8 height] ..).
// Every lane of the warp calls it; `act` is false for lanes without a pair.
template <class Leaf>
__device__ __forceinline__ void path_group(const Leaf &leaf, const TreeLevels &lv, uint32_t g, uint64_t idx, bool act,
                                           uint32_t *nh, uint32_t *p, uint32_t *sp) {
    const uint32_t lane = threadIdx.x & (kPathLanes - 1u);
    const uint32_t lo = lv.height[g], k = act ? lv.height[g + 1] - lo : 0u;
    const uint64_t node = idx >> lo, first = (node >> k) << k;
    const uint32_t K = act ? 1u << k : 0u;
    if (g == 0) {
        for (uint32_t j = lane; j < K; j += kPathLanes) {
            uint32_t h[8];
            leaf(first + j, h);
            store_hash(nh + 8 * j, h);
        }
    } else {
        const uint4 *s = (const uint4 *)(lv.hashes[g] + 8ull * first);
        for (uint32_t j = lane; j < 2 * K; j += kPathLanes) ((uint4 *)nh)[j] = s[j];
    }
    __syncwarp();
    uint32_t off = 0, cnt = K;
#pragma unroll 1
    for (uint32_t d = 1; d < 4; d++) {  // at most 4 heights per group; the block's root is not needed
        if (d < k && lane < cnt / 2) {
            uint32_t h[8];
            blake2s_node(h, nh + 8 * (off + 2 * lane), nh + 8 * (off + 2 * lane) + 8);
            store_hash(nh + 8 * (off + cnt + lane), h);
        }
        off += cnt;
        cnt /= 2;
        __syncwarp();
    }
    off = 0; cnt = K;
    uint32_t local = (uint32_t)node & (K - 1u);
    for (uint32_t d = 0; d < k; d++) {
        const uint32_t hgt = lo + d;
        const uint32_t sib = nh[8 * (off + (local ^ 1u)) + lane];
        p[1 + 8 * hgt + lane] = sib;
        sp[1 + 8 * hgt + lane] = hgt == 0 ? nh[8 * (off + local) + lane] : sib;
        off += cnt; cnt /= 2; local >>= 1;
    }
}

}  // namespace vx

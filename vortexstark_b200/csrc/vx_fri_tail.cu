// The FRI layers of at most 2048 values in one launch.
//
// Each layer waits for the challenge drawn from the layer before it, so the
// time is a chain of dependent compressions (leaf, one per level, mix,
// squeeze) whatever the number of blocks; a launch per layer adds its drain,
// start and reload of values, twiddles and state to every link, and a tree of
// several blocks a hand-over through global memory.  One block of 256 threads
// keeps the chain of a layer of at most 256 values: 256 leaves are one per
// thread, and from 64 hashes down a quad of lanes takes each (vx_quad.cuh).
// Layers of 512 to 2048 values are split over a cluster of eight blocks: an
// eighth of a layer folds from the same eighth of the one before, so values
// stay in their block; the eight subtree roots go to block 0's shared memory,
// which finishes the tree and the transcript step and sends the challenge to
// every block.  Shared memory of another block may be written only once that
// block runs: every block arrives at the cluster barrier first of all and
// waits for the others right before its first remote store, so the wait is
// over by then and costs nothing on the chain.
//
// Line folds of a log_n 10 proof: 88 us with a launch per layer, 82 with the
// layers of at most 256 values in one block, 79-80 with the cluster above.
#include <cooperative_groups.h>

#include "vx_common.cuh"
#include "vx_fri.cuh"
#include "vx_merkle.cuh"

namespace vx {
namespace {

namespace cg = cooperative_groups;
static_assert(kTailCluster == 8 && (1u << kTailLog) / kTailCluster <= kReduceThreads, "one leaf per thread");

__global__ void __launch_bounds__(kReduceThreads) fri_tail_kernel(const __grid_constant__ FriTailArgs a, uint32_t one) {
    __shared__ __align__(16) uint32_t buf[2][128 * kMsgWords];
    // the cluster's subtree roots, as 4 messages; a warp of quads reads 8
    __shared__ __align__(16) uint32_t roots[2][8 * kMsgWords];
    __shared__ uint4 vals[2][1 << kTailBlockLog];
    __shared__ uint32_t al[4];
    cg::cluster_group cl = cg::this_cluster();
    bool split = a.d0 > kTailBlockLog;
    if (split) cl.barrier_arrive();  // this block has started; the wait is before the first remote store
    Quad q;
    q.init();
    pdl_wait();
    const uint32_t rank = blockIdx.x;  // one cluster per launch
    const uint32_t tid = threadIdx.x, warp = tid >> 5;
    uint32_t s0 = 0, s1 = 0;
    if (tid < 4) {
        s0 = a.ch->state[tid]; s1 = a.ch->state[4 + tid];
        al[tid] = a.alpha_in[tid];
    }
    qm31 f0{}, f1{};
    uint32_t tw = 0;
    // values 2j, 2j + 1 of a layer in global memory
    auto load_pair = [&](const uint32_t *const *in, uint32_t j) {
#pragma unroll
        for (int c = 0; c < 4; c++) {
            const uint2 x = __ldcg((const uint2 *)in[c] + j);
            f0.v[c] = x.x; f1.v[c] = x.y;
        }
    };
    uint32_t m = 1u << a.d0;                                  // values of the layer
    uint32_t n = split ? m / kTailCluster : m;                // of which this block's
    uint32_t first = split ? rank * n : 0u;
    if (tid < n) {
        load_pair(a.in, first + tid);
        tw = a.l[0].tw[first + tid];
    }
    __syncthreads();
#pragma unroll 1
    for (uint32_t k = 0; k < a.n; k++) {
        const FriTailLayer &L = a.l[k];
        uint32_t *cur = buf[0], *nxt = buf[1];
        if (tid < n) {
            const qmat am = qmat_of(qm31{{al[0], al[1], al[2], al[3]}});
            const qm31 r = qadd2_mul_mat(f0, f1, am, qmulm(qsub(f0, f1), tw));
#pragma unroll
            for (int c = 0; c < 4; c++) L.out[c][first + tid] = r.v[c];
            vals[k & 1][tid] = make_uint4(r.v[0], r.v[1], r.v[2], r.v[3]);
            if (n > 64u) {
                uint32_t mm[16], hv[8];
#pragma unroll
                for (int w = 0; w < 16; w++) mm[w] = w < 4 ? r.v[w] : 0u;
                blake2s_block(hv, mm, 16u, one);
                store_hash(cur + kMsgWords * (tid >> 1) + 8u * (tid & 1u), hv);
            } else {
                uint4 *d = (uint4 *)(cur + kMsgWords * tid);
                d[0] = make_uint4(r.v[0], r.v[1], r.v[2], r.v[3]);
                d[1] = d[2] = d[3] = make_uint4(0u, 0u, 0u, 0u);
            }
        }
        __syncthreads();
        // half: nodes of the first level that quads hash, at height lev
        uint32_t half = n > 64u ? n >> 1 : n, lev = n > 64u ? 1u : 0u;
        if (half == 128u) {
            if (tid < 128u) {
                uint32_t hv[8];
                blake2s_node(hv, cur + kMsgWords * tid, cur + kMsgWords * tid + 8, one);
                store_hash(nxt + kMsgWords * (tid >> 1) + 8u * (tid & 1u), hv);
                uint32_t *g = stored_node(L.lv, lev, (split ? rank * 128u : 0u) + tid);
                if (g) store_hash(g, hv);
            }
            __syncthreads();
            uint32_t *t = cur; cur = nxt; nxt = t;
            half = 64u; lev++;
        }
        uint32_t o0, o1;
        nxt = quad_levels(q, L.lv, cur, nxt, half, lev, split ? rank : 0u, lev ? 64u : 16u, o0, o1);
        if (split) {
            // subtree roots at height d - 3 -> block 0
            uint32_t h = 0;
            while ((n >> h) > 1u) h++;
            if (k == 0) cl.barrier_wait();
            if (tid < 4) {
                uint32_t *d = cl.map_shared_rank(&roots[0][0], 0) + kMsgWords * (rank >> 1) + 8u * (rank & 1u) + tid;
                d[0] = o0; d[4] = o1;
            }
            cl.sync();
            if (rank == 0) nxt = quad_levels(q, L.lv, roots[0], roots[1], kTailCluster / 2, h + 1, 0, 64u, o0, o1);
        }
        uint32_t w = 0;
        if (warp == 0 && rank == 0)
            w = chan_commit_quad(q, ChanStep{a.ch, L.root, L.alpha_out}, nxt, s0, s1, o0, o1);
        if (split) {
            if (warp == 0 && rank == 0) {  // lane 4 b + i: word i of the challenge to block b
                w = __shfl_sync(0xFFFFFFFFu, w, tid & 3u);
                cl.map_shared_rank(al, tid >> 2)[tid & 3u] = w;
            }
            cl.sync();
        } else {
            if (tid < 4) al[tid] = w;
            __syncthreads();
        }
        // the next layer
        if (k + 1 == a.n) break;
        m >>= 1;
        const bool was_split = split;
        split = m > (1u << kTailBlockLog);
        if (was_split && !split && rank != 0) break;  // block 0 goes on alone
        n = split ? m / kTailCluster : m;
        first = split ? rank * n : 0u;
        if (tid < n) {
            if (was_split && !split) {
                load_pair(L.out, tid);
            } else {
                const uint4 x = vals[k & 1][2 * tid], y = vals[k & 1][2 * tid + 1];
                f0 = qm31{{x.x, x.y, x.z, x.w}};
                f1 = qm31{{y.x, y.y, y.z, y.w}};
            }
            tw = a.l[k + 1].tw[first + tid];
        }
    }
}

}  // namespace

cudaError_t fri_tail(const FriTailArgs &a, cudaStream_t stream) {
    if (a.n == 0) return cudaSuccess;
    if (a.d0 <= kTailBlockLog) return launch_pdl(fri_tail_kernel, dim3(1), dim3(kReduceThreads), 0, stream, a, 1u);
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(kTailCluster);
    cfg.blockDim = dim3(kReduceThreads);
    cfg.stream = stream;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    attr[1].id = cudaLaunchAttributeClusterDimension;
    attr[1].val.clusterDim.x = kTailCluster;
    attr[1].val.clusterDim.y = 1;
    attr[1].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 2;
    return cudaLaunchKernelEx(&cfg, fri_tail_kernel, a, 1u);
}

}  // namespace vx

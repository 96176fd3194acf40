// The FRI layers of at most 256 values in one launch.
//
// Each layer waits for the challenge drawn from the layer before it, so the
// time is a chain of dependent compressions (leaf, one per level, mix,
// squeeze) whatever the number of blocks; a launch per layer adds its drain,
// start and reload of values, twiddles and state to every link.  One block of
// 256 threads keeps the chain: 256 leaves are one per thread, and from 64
// hashes down a quad of lanes takes each (vx_quad.cuh).
#include "vx_common.cuh"
#include "vx_fri.cuh"
#include "vx_merkle.cuh"

namespace vx {
namespace {

__global__ void __launch_bounds__(kReduceThreads) fri_tail_kernel(const __grid_constant__ FriTailArgs a, uint32_t one) {
    __shared__ __align__(16) uint32_t buf[2][128 * kMsgWords];
    __shared__ uint4 vals[2][1 << kTailLog];
    __shared__ uint32_t al[4];
    Quad q;
    q.init();
    pdl_wait();
    const uint32_t tid = threadIdx.x, warp = tid >> 5;
    uint32_t m = 1u << a.d0;
    uint32_t s0 = 0, s1 = 0;
    if (tid < 4) {
        s0 = a.ch->state[tid]; s1 = a.ch->state[4 + tid];
        al[tid] = a.alpha_in[tid];
    }
    qm31 f0{}, f1{};
    uint32_t tw = 0;
    if (tid < m) {
#pragma unroll
        for (int c = 0; c < 4; c++) {
            const uint2 x = *((const uint2 *)a.in[c] + tid);
            f0.v[c] = x.x; f1.v[c] = x.y;
        }
        tw = a.l[0].tw[tid];
    }
    __syncthreads();
#pragma unroll 1
    for (uint32_t k = 0; k < a.n; k++, m >>= 1) {
        const FriTailLayer &L = a.l[k];
        uint32_t *cur = buf[0], *nxt = buf[1];
        if (tid < m) {
            if (k) {
                const uint4 x = vals[(k - 1) & 1][2 * tid], y = vals[(k - 1) & 1][2 * tid + 1];
                f0 = qm31{{x.x, x.y, x.z, x.w}};
                f1 = qm31{{y.x, y.y, y.z, y.w}};
            }
            const qmat am = qmat_of(qm31{{al[0], al[1], al[2], al[3]}});
            const qm31 r = qadd(qadd(f0, f1), qmul_mat(am, qmulm(qsub(f0, f1), tw)));
#pragma unroll
            for (int c = 0; c < 4; c++) L.out[c][tid] = r.v[c];
            vals[k & 1][tid] = make_uint4(r.v[0], r.v[1], r.v[2], r.v[3]);
            if (m > 64u) {
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
            if (k + 1 < a.n && tid < m / 2) tw = a.l[k + 1].tw[tid];
        }
        __syncthreads();
        // half: nodes of the first level that quads hash, at height lev
        uint32_t half = m > 64u ? m >> 1 : m, lev = m > 64u ? 1u : 0u;
        if (half == 128u) {
            if (tid < 128u) {
                uint32_t hv[8];
                blake2s_node(hv, cur + kMsgWords * tid, cur + kMsgWords * tid + 8, one);
                store_hash(nxt + kMsgWords * (tid >> 1) + 8u * (tid & 1u), hv);
                uint32_t *g = stored_node(L.lv, lev, tid);
                if (g) store_hash(g, hv);
            }
            __syncthreads();
            uint32_t *t = cur; cur = nxt; nxt = t;
            half = 64u; lev++;
        }
        uint32_t o0, o1;
        nxt = quad_levels(q, L.lv, cur, nxt, half, lev, 0, lev ? 64u : 16u, o0, o1);
        if (warp == 0) {
            const uint32_t w = chan_commit_quad(q, ChanStep{a.ch, L.root, L.alpha_out}, nxt, s0, s1, o0, o1);
            if (tid < 4) al[tid] = w;
        }
        __syncthreads();
    }
}

}  // namespace

cudaError_t fri_tail(const FriTailArgs &a, cudaStream_t stream) {
    if (a.n == 0) return cudaSuccess;
    return launch_pdl(fri_tail_kernel, dim3(1), dim3(kReduceThreads), 0, stream, a, 1u);
}

}  // namespace vx

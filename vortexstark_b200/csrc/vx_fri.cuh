// FRI fold fused with the commitment of the folded layer.
#pragma once
#include <cstdint>

#include "vx_field.cuh"
#include "vx_merkle.cuh"

namespace vx {

// Leaf source for a tree over a folded SoA4 QM31 layer: output j pairs
// f0 = in[2j] and f1 = in[2j + 1] (fri.cu:58-126),
//   out[j] = (f0 + f1) + alpha * ((f0 - f1) * tw[j]),
// stored to the output layer and hashed as its 4-word leaf.  The circle fold
// into a pre-zeroed line (fri.cu:92-126) is the same formula; line and
// circle folds differ only in their twiddles.
struct LeafFold {
    const uint32_t *i0, *i1, *i2, *i3;
    const uint32_t *tw;
    const uint32_t *alpha_ptr;
    uint32_t *o0, *o1, *o2, *o3;
    qmat am;  // multiplication by the fold challenge
    __device__ __forceinline__ void init() { am = qmat_of(qm31{{alpha_ptr[0], alpha_ptr[1], alpha_ptr[2], alpha_ptr[3]}}); }
    __device__ __forceinline__ uint32_t load(uint64_t j, uint32_t m[16]) const {
        uint2 a0 = __ldg((const uint2 *)i0 + j), a1 = __ldg((const uint2 *)i1 + j);
        uint2 a2 = __ldg((const uint2 *)i2 + j), a3 = __ldg((const uint2 *)i3 + j);
        qm31 f0{{a0.x, a1.x, a2.x, a3.x}}, f1{{a0.y, a1.y, a2.y, a3.y}};
        qm31 r = qadd2_mul_mat(f0, f1, am, qmulm(qsub(f0, f1), __ldg(tw + j)));
        o0[j] = r.v[0]; o1[j] = r.v[1]; o2[j] = r.v[2]; o3[j] = r.v[3];
        m[0] = r.v[0]; m[1] = r.v[1]; m[2] = r.v[2]; m[3] = r.v[3];
        return 16u;
    }
};

// The last FRI layers, of at most 2^kTailLog values each, in one launch: fold,
// tree and transcript step of every layer, with the folded values, messages
// and transcript state in shared memory.  Layers of up to 2^kTailBlockLog
// values run in one block, larger ones in a cluster of kTailCluster.
constexpr uint32_t kTailLog = 11, kTailBlockLog = 8, kTailCluster = 8;
struct FriTailLayer {
    const uint32_t *tw;
    uint32_t *out[4];
    uint32_t *root;       // 8 words in the proof
    uint32_t *alpha_out;  // challenge drawn after this layer; null: none
    TreeLevels lv;
};
struct FriTailArgs {
    const uint32_t *in[4];     // the layer before, 2^(d0 + 1) values
    const uint32_t *alpha_in;  // challenge of the first fold
    DevChannel *ch;
    uint32_t n, d0;            // layers; log size of the first
    FriTailLayer l[kTailLog];
};
cudaError_t fri_tail(const FriTailArgs &a, cudaStream_t stream);

// Line folds of layers k0 .. k1 - 1: layer k (log size log0 - k, columns
// F[k][0..3]) folds layer k - 1 with twiddles tw(k) and challenge
// alpha + 4 k, is committed as tree lv[k], its root goes to root(k), and
// challenge alpha + 4 (k + 1) is drawn unless k + 1 == n.  Layers of at most
// 2^kTailLog values share one launch.
template <class Tw, class Cols, class Root>
cudaError_t fri_line_layers(uint32_t k0, uint32_t k1, uint32_t n, uint32_t log0, const Cols &F, const TreeLevels *lv,
                            const Tw &tw, uint32_t *alpha, DevChannel *ch, const Root &root, cudaStream_t st,
                            uint32_t *launches) {
    for (uint32_t k = k0; k < k1; k++) {
        auto next_alpha = [&](uint32_t j) { return j + 1 < n ? alpha + 4 * (j + 1) : nullptr; };
        if (log0 - k <= kTailLog && k1 - k <= kTailLog) {
            FriTailArgs a{};
            for (int c = 0; c < 4; c++) a.in[c] = F(k - 1)[c];
            a.alpha_in = alpha + 4 * k;
            a.ch = ch;
            a.n = k1 - k;
            a.d0 = log0 - k;
            for (uint32_t j = k; j < k1; j++) {
                FriTailLayer &t = a.l[j - k];
                t.tw = tw(j);
                for (int c = 0; c < 4; c++) t.out[c] = F(j)[c];
                t.root = root(j);
                t.alpha_out = next_alpha(j);
                t.lv = lv[j];
            }
            *launches += 1;
            return fri_tail(a, st);
        }
        uint32_t *const *in = F(k - 1), *const *out = F(k);
        LeafFold lf{in[0], in[1], in[2], in[3], tw(k), alpha + 4 * k, out[0], out[1], out[2], out[3], {}};
        cudaError_t e = tree_build(lf, lv[k], ChanStep{ch, root(k), next_alpha(k)}, st);
        if (e != cudaSuccess) return e;
        *launches += tree_launches(lv[k]);
    }
    return cudaSuccess;
}

}  // namespace vx

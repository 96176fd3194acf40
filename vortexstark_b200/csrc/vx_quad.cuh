// Blake2s-256 compression spread over four lanes, for the serial parts of a
// commitment: the upper levels of a tree and the transcript, where few hashes
// are in flight and the time is the length of the dependent chain.
//
// Lane l of a quad holds column l of the 4 x 4 working state (v[l], v[4+l],
// v[8+l], v[12+l]), so each half round is one G per lane.  Between half
// rounds three of the four rows rotate by shuffles.  The row that stays is
// b, the last one a G finishes: a, d and c are final 5, 4 and 2 operations
// before b, which hides most of their shuffles' latency.  d is shuffled
// before its last rotation (e = d ^ a, d = ror8(e)); the receiver folds that
// rotation into the next one: ror16(d ^ a') = ror24(e) ^ ror16(a').
//
// The 16 message words lie in shared memory; a lane reads the four words of
// its two G's of a round at byte offsets packed in one register per round.
#pragma once
#include <cstdint>

#include "vx_blake2s.cuh"

namespace vx {

constexpr uint8_t kSigma[10][16] = {
    {0, 1, 2, 3, 4, 5, 6, 7, 8, 9, 10, 11, 12, 13, 14, 15}, {14, 10, 4, 8, 9, 15, 13, 6, 1, 12, 0, 2, 11, 7, 5, 3},
    {11, 8, 12, 0, 5, 2, 15, 13, 10, 14, 3, 6, 7, 1, 9, 4}, {7, 9, 3, 1, 13, 12, 11, 14, 2, 6, 5, 10, 4, 0, 15, 8},
    {9, 0, 5, 7, 2, 4, 10, 15, 14, 1, 11, 12, 6, 8, 3, 13}, {2, 12, 6, 10, 0, 11, 8, 3, 4, 13, 7, 5, 15, 14, 1, 9},
    {12, 5, 1, 15, 14, 13, 4, 10, 0, 7, 6, 3, 9, 2, 8, 11}, {13, 11, 7, 14, 12, 1, 3, 9, 5, 0, 15, 4, 8, 6, 2, 10},
    {6, 15, 14, 9, 11, 3, 0, 8, 12, 2, 13, 7, 1, 4, 10, 5}, {10, 2, 8, 4, 7, 6, 1, 5, 15, 11, 9, 14, 3, 12, 13, 0}};

// Byte offsets of the message words of lane l's G's in round r: byte 0 and 1
// the column step's x and y, 2 and 3 the diagonal step's.  With b fixed, lane
// l runs diagonal l - 1 (the one that uses v[4 + l]).
constexpr uint32_t quad_words(int r, int l) {
    const int j = (l + 3) & 3;
    return 4u * kSigma[r][2 * l] | 4u * kSigma[r][2 * l + 1] << 8 | 4u * kSigma[r][8 + 2 * j] << 16 |
           4u * kSigma[r][9 + 2 * j] << 24;
}
struct QuadTab { uint32_t v[10][4]; };
constexpr QuadTab quad_tab() {
    QuadTab t{};
    for (int r = 0; r < 10; r++)
        for (int l = 0; l < 4; l++) t.v[r][l] = quad_words(r, l);
    return t;
}

// Per-lane constants, formed once per kernel.
struct Quad {
    uint32_t w[10];         // message word offsets
    uint32_t iv0, iv1;      // IV[l], IV[4 + l]
    uint32_t l;             // lane within the quad
    uint32_t prev, next, opp;  // source lanes l - 1, l + 1, l + 2 of this quad
    __device__ __forceinline__ uint32_t pick(uint32_t a, uint32_t b, uint32_t c, uint32_t d) const {
        return l == 0 ? a : l == 1 ? b : l == 2 ? c : d;
    }
    __device__ __forceinline__ void init() {
        constexpr QuadTab T = quad_tab();
        const uint32_t lane = threadIdx.x & 31u, q = lane & ~3u;
        l = lane & 3u;
#pragma unroll
        for (int r = 0; r < 10; r++) w[r] = pick(T.v[r][0], T.v[r][1], T.v[r][2], T.v[r][3]);
        iv0 = pick(VX_IV0, VX_IV1, VX_IV2, VX_IV3);
        iv1 = pick(VX_IV4, VX_IV5, VX_IV6, VX_IV7);
        prev = q | ((l + 3u) & 3u);
        next = q | ((l + 1u) & 3u);
        opp = q | ((l + 2u) & 3u);
    }
};

__device__ __forceinline__ uint32_t ror24(uint32_t x) { return __byte_perm(x, 0, 0x2103); }

// Final-block hash of the 16 words at m (shared memory): out0 = h[l],
// out1 = h[4 + l].  All 32 lanes of the warp take part.
__device__ __forceinline__ void quad_hash(const Quad &q, const uint32_t *m, uint32_t nbytes, uint32_t &out0,
                                          uint32_t &out1) {
    auto word = [&](uint32_t w, int k) {
        return *(const uint32_t *)((const char *)m + __byte_perm(w, 0, 0x4440 + k));
    };
    const uint32_t h0 = q.iv0 ^ (q.l == 0 ? 0x01010020u : 0u), h1 = q.iv1;
    const uint32_t d0 = q.iv1 ^ (q.l == 0 ? nbytes : q.l == 2 ? ~0u : 0u);
    uint32_t a = h0, b = h1, c = q.iv0, d, e = __byte_perm(d0, 0, 0x2103);  // e = rol8(d0): d0 = ror8(e)
#pragma unroll
    for (int r = 0; r < 10; r++) {
        const uint32_t x0 = word(q.w[r], 0), y0 = word(q.w[r], 1), x1 = word(q.w[r], 2), y1 = word(q.w[r], 3);
#pragma unroll
        for (int half = 0; half < 2; half++) {
            a = a + b + (half ? x1 : x0);
            d = ror24(e) ^ ror16(a);
            c = c + d;
            b = ror12(b ^ c);
            a = a + b + (half ? y1 : y0);
            e = d ^ a;
            a = __shfl_sync(0xFFFFFFFFu, a, half ? q.next : q.prev);
            d = ror8(e);
            e = __shfl_sync(0xFFFFFFFFu, e, q.opp);
            c = c + d;
            b = ror7(b ^ c);
            c = __shfl_sync(0xFFFFFFFFu, c, half ? q.prev : q.next);
        }
    }
    out0 = h0 ^ a ^ c;
    out1 = h1 ^ b ^ ror8(e);
}

}  // namespace vx

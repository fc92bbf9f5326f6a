// Softmax, top-k and renormalisation of one token's logits, for the routing kernels and for the
// kernel that routes a few tokens by itself.  Reference: engine/src/model.rs:259-268 (route),
// engine/src/ops.rs:192-201 (softmax).
#pragma once
#include <stdint.h>

namespace bivmoe {

// One warp per token: softmax in the reference's order (max, exp, sequential
// sum, multiply by 1/sum), the k best by (probability descending, expert id
// ascending), weights p / max(sum of the k in rank order, 2^-14).
// The order of the probabilities is f32::total_cmp's, as in the reference's sort
// (model.rs:263): a total order, so a row with NaN or Inf activations - whose
// probabilities are all NaN - still selects k distinct, valid experts (the first k,
// all keys being equal) and only that token's weights and output are NaN.
// total_cmp's key: the bits with the magnitude inverted for negative values, compared
// as signed integers; the mapping is its own inverse
__device__ __forceinline__ int tk_total_key(int bits) { return bits ^ (int)(((uint32_t)(bits >> 31)) >> 1); }

// One warp, one token.  The M * 32 >= n_expert probabilities live in registers (lane + 32 m);
// `p` (shared memory, 16-byte aligned, n_expert floats) holds them once for the sum in the
// reference's order.  Every selection is two warp reductions (redux): the largest key, then
// the lowest id that has it.  A chain of a few thousand clocks is what bounds it at any small
// number of tokens: 6.5 us with the keys in shared memory and five shuffle steps per
// reduction, 4 so.
template <int M>
__device__ __forceinline__ void topk_token(const float* __restrict__ l, float* p, int n_expert, int k, int lane,
                                           int& sel_id, float& weight) {
    float v[M];
    float mx = -INFINITY;
#pragma unroll
    for (int m = 0; m < M; m++) v[m] = lane + 32 * m < n_expert ? l[lane + 32 * m] : -INFINITY;
#pragma unroll
    for (int m = 0; m < M; m++) mx = fmaxf(mx, v[m]);   // f32::max: a NaN is passed over
#pragma unroll
    for (int o = 16; o; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
#pragma unroll
    for (int m = 0; m < M; m++) {
        v[m] = expf(__fsub_rn(v[m], mx));
        if (lane + 32 * m < n_expert) p[lane + 32 * m] = v[m];
    }
    __syncwarp();
    float sum = 0.0f;   // the order of the adds is the reference's; every lane adds the same numbers
    int i = 0;
#pragma unroll 4
    for (; i + 4 <= n_expert; i += 4) {
        const float4 q = *(const float4*)(p + i);
        sum = __fadd_rn(__fadd_rn(__fadd_rn(__fadd_rn(sum, q.x), q.y), q.z), q.w);
    }
    for (; i < n_expert; i++) sum = __fadd_rn(sum, p[i]);
    const float inv = __fdiv_rn(1.0f, sum);
    // keys as unsigned numbers from 1 on (the two lowest are NaNs both); 0 marks a taken or
    // absent entry
    uint32_t key[M];
#pragma unroll
    for (int m = 0; m < M; m++) {
        int bits = __float_as_int(__fmul_rn(v[m], inv));
        asm("" : "+r"(bits));   // or the flipped sign bit is folded into the product, which a NaN does not show
        key[m] = lane + 32 * m < n_expert ? max((uint32_t)tk_total_key(bits) ^ 0x80000000u, 1u) : 0u;
    }
    float sel_p = 0.0f, tot = 0.0f;   // lane j keeps the j-th selection
    sel_id = 0;
    for (int j = 0; j < k; j++) {
        uint32_t best = key[0];
#pragma unroll
        for (int m = 1; m < M; m++) best = max(best, key[m]);
        best = __reduce_max_sync(0xffffffffu, best);
        uint32_t id = 0xffffffffu;
#pragma unroll
        for (int m = M - 1; m >= 0; m--)
            if (key[m] == best) id = (uint32_t)(lane + 32 * m);
        id = __reduce_min_sync(0xffffffffu, id);   // ties go to the lower id
#pragma unroll
        for (int m = 0; m < M; m++)
            if (id == (uint32_t)(lane + 32 * m)) key[m] = 0u;
        const float pj = __int_as_float(tk_total_key((int)(best ^ 0x80000000u)));
        tot = __fadd_rn(tot, pj);
        if (lane == j) { sel_p = pj; sel_id = (int)min(id, (uint32_t)(n_expert - 1)); }
    }
    tot = fmaxf(tot, 1.0f / 16384.0f);   // f32::max: a NaN sum gives the floor
    weight = __fdiv_rn(sel_p, tot);
}

}  // namespace bivmoe

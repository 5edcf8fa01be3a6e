// What the tensor-core kernels of the latent attention share (latent_mma.cu, latent_tc.cu).
#pragma once
#include "common.cuh"

struct LatentMmaArgs {
    const __nv_bfloat16* qa;     // [nt, H, rank]
    const __nv_bfloat16* q;      // [nt, ldq]; head h's rotated part at h * q_head + q_plain
    __nv_bfloat16* out;          // [nt, H, rank]
    float* partial;              // [nt, H, splits, rank + 2] when splits > 1
    const __nv_bfloat16* cache;  // [pages, TB_PAGE, rank + rot]
    const int* tile_seq;
    const int* tile_t0;
    const int* tile_nq;
    const int* tok_pos;
    const int* page_table;
    const float* cosT;
    const float* sinT;
    int max_pages, ldq, q_head, q_plain, H, rank, rot, rdims, window, heads_per_block, tokens_per_block, splits;
    float scale;
    const float* sinks;          // [H] or null: a number per head that joins the softmax's denominator once
    const __nv_bfloat16* gate;   // [nt, ldg] or null: head h's output is multiplied by sigmoid(gate[t, h])
    int ldg;
};

// What a sink and a gate make of a row's (maximum, sum): the factor for its unnormalized output.
__device__ __forceinline__ float lm_finish(float m, float l, const float* sinks, const __nv_bfloat16* gate, int ldg,
                                           int t, int h) {
    float f = 1.f;
    if (sinks) {
        const float sk = sinks[h], m2 = fmaxf(m, sk);
        f = m > -INFINITY ? __expf(m - m2) : 0.f;
        l = l * f + __expf(sk - m2);
    }
    f = l > 0.f ? f / l : 0.f;
    if (gate) f *= 1.0f / (1.0f + __expf(-__bfloat162float(gate[(size_t)t * ldg + h])));
    return f;
}

// The pair (x0, x1) turned by the angle of cosine co and sine si; which product is rounded by itself is said, so that all
// kernels have the same bits.
__device__ __forceinline__ float lm_turn_low(float x0, float x1, float co, float si) { return __fmaf_rn(x0, co, -__fmul_rn(x1, si)); }
__device__ __forceinline__ float lm_turn_high(float x0, float x1, float co, float si) { return __fmaf_rn(x1, co, __fmul_rn(x0, si)); }

// Entry r of a head's rotated part (its queries as the product left them: qr), turned for its position.
__device__ __forceinline__ float lm_turned(const LatentMmaArgs& a, const __nv_bfloat16* qr, int r, int pos) {
    const int half = a.rdims / 2;
    const float v = __bfloat162float(qr[r]);
    if (r >= a.rdims) return v;
    const size_t at = (size_t)pos * half + (r < half ? r : r - half);
    return r < half ? lm_turn_low(v, __bfloat162float(qr[r + half]), a.cosT[at], a.sinT[at])
                    : lm_turn_high(__bfloat162float(qr[r - half]), v, a.cosT[at], a.sinT[at]);
}

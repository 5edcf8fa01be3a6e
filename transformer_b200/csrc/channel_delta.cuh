// What the kernels of the gated delta rule with a decay per key channel (channel_delta.cu, channel_delta_chunk.cu) share.
#pragma once
#include "common.cuh"

#define CD_UNIT_EPS 1e-6f
#define CD_MAX_TAPS 16

struct DeltaPrepArgs {
    const void* z;          // [nt, ldz]: q (G dim) | k (G dim) | v (H vdim) | whatever else the product made
    const float* wconv;     // [C, taps], the last column is the current token's
    float* state;           // [slots, state_stride]
    const float* a;         // [nt, H dim]  pre-activation of the decay
    const float* dt_bias;   // [H dim]
    const float* A_log;     // [H]
    const float* bz;        // [nt, H]      pre-activation of beta
    float* rec;             // out [nt, H, cd_record(dim)]
    float* vbuf;            // out [nt, H, cd_vpitch(vdim)]
    const int* tok_seq;
    const int* seq_start;
    const int* slots;
    long long state_stride, conv_offset;
    int ldz, G, H, dim, vdim, taps, update_state;
    int lda, ldb;           // row pitches of a and bz (floats)
    int head_decay;         // 1: one decay per head: a [nt, H], dt_bias [H], the same g for every key channel
};

__device__ __forceinline__ float cd_softplus(float x) { return fmaxf(x, 0.f) + log1pf(expf(-fabsf(x))); }

// After a step that brought a sequence more than one token: the last taps - 1 inputs of every channel, from the
// step's rows and, where the step was shorter than that, from what the state held.
template <typename T>
__global__ void __launch_bounds__(256) delta_conv_state_kernel(const DeltaPrepArgs p) {
    pdl_sync();
    const int b = blockIdx.x, c = blockIdx.y * blockDim.x + threadIdx.x;
    const int C = 2 * p.G * p.dim + p.H * p.vdim, keep = p.taps - 1;
    if (c >= C) return;
    const int t0 = p.seq_start[b], n = p.seq_start[b + 1] - t0;
    if (n <= 0) return;
    const T* z = static_cast<const T*>(p.z);
    float* cs = p.state + (size_t)p.slots[b] * p.state_stride + p.conv_offset;
    float fresh[CD_MAX_TAPS];
    for (int r = 0; r < keep; ++r) {
        const int li = n - keep + r;
        fresh[r] = li >= 0 ? ldf(z + (size_t)(t0 + li) * p.ldz + c) : cs[(size_t)(keep + li) * C + c];
    }
    for (int r = 0; r < keep; ++r) cs[(size_t)r * C + c] = fresh[r];
}

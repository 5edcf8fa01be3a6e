// What the kernels of the matrix memory with exponential gates (mlstm.cu, mlstm_parallel.cu) share.
#pragma once
#include "common.cuh"

#define ML_COLS 32              // columns of v per copy of n and m in the state
#define ML_DENOM_FLOOR 1e-6f
#define MC_L 64                 // tokens of a chunk

struct MlstmArgs {
    const void* qkv;        // [nt, ld]: q heads | k heads | v heads (| anything else)
    const float* gates;     // [nt, 2 H]: zi of every head, then zf
    const float* bias;      // [2 H]
    float* state;           // [slots, H, state_size]
    float* out;             // [nt, H * vdim] unnormalized o
    const int* seq_start;   // [B + 1]
    const int* slots;       // [B]
    int ld, H, dim, vdim;
    float cap, qscale;
};

__device__ __forceinline__ float log_sigmoid(float z) { return fminf(z, 0.f) - log1pf(expf(-fabsf(z))); }

__device__ __forceinline__ float warp_scan_add(float v, int lane) {
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const float u = __shfl_up_sync(0xffffffffu, v, o);
        if (lane >= o) v += u;
    }
    return v;
}
__device__ __forceinline__ float warp_scan_max(float v, int lane) {
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const float u = __shfl_up_sync(0xffffffffu, v, o);
        if (lane >= o) v = fmaxf(v, u);
    }
    return v;
}

// Embedding gather and the fused residual-add + RMSNorm.
//
// The residual stream is float on both paths, so the residual sum is a 32-bit sum.
#include "common.cuh"
#include "attention_prefill.cuh"        // cp_async16, cp_async_commit, cp_async_wait
#include "router_pick.cuh"

#include <type_traits>

// x[i, :] = table[tokens[i], :]   (models/llama/cuda/src/infer.rs:98-104 copies row by row)
template <typename T>
__global__ void embed_kernel(const int* __restrict__ tokens, const T* __restrict__ table,
                             float* __restrict__ x, int d, float scale) {
    pdl_sync();
    const int i = blockIdx.x;
    const T* src = table + (size_t)tokens[i] * d;
    float* dst = x + (size_t)i * d;
    for (int c = threadIdx.x; c < d; c += blockDim.x) dst[c] = ldf(src + c) * scale;
}

// Row r = rows ? rows[i] : i.
//   v = x[r] + delta(r)                                    float sum
//   if (!rows && there is a delta) x[r] = v                the stream is updated in place
//   y[i] = v / sqrt(mean(v^2) + eps) * w                   statistics in float, one rounding to T
// delta(r) is delta[r] (a part's output), or, when wy is given, the weighted sum of rows of wy:
//   sum_j topk_w[r, j] * wy[pair_row[r * k + j]]           j ascending, in float
// which is the combine of the experts' outputs (compute.rs:329-330) fused into the norm that follows.
// (call sites of rms_norm: models/llama/common/src/compute.rs:207,275,362; the residual sum is the
//  beta = 1 of the output products, :270,:330.)
// Bytes that the kernel AFTER this one reads first and that are weights (a router's matrix: 128 KB that one block
// per token would otherwise wait for from HBM): the last block asks for them to be brought into L2, before it
// waits for the kernel before it.  Weights do not change, so asking early is always safe.
__device__ __forceinline__ void warm_l2(const void* warm, int warm_bytes) {
    if (warm && blockIdx.x == gridDim.x - 1)
        for (int off = threadIdx.x * 128; off < warm_bytes; off += blockDim.x * 128)
            asm volatile("prefetch.global.L2 [%0];" ::"l"(static_cast<const char*>(warm) + off));
}

template <typename T>
__global__ void add_rmsnorm_kernel(float* __restrict__ x, const T* __restrict__ delta,
                                   const T* __restrict__ wy, const int* __restrict__ pair_row,
                                   const float* __restrict__ topk_w, int k,
                                   const int* __restrict__ rows, const float* __restrict__ w,
                                   float eps, T* __restrict__ y, int d, const void* warm, int warm_bytes) {
    warm_l2(warm, warm_bytes);
    pdl_sync();
    __shared__ float red[33];
    const int i = blockIdx.x;
    const int r = rows ? rows[i] : i;
    float* xr = x + (size_t)r * d;
    const T* dr = delta ? delta + (size_t)r * d : nullptr;
    const bool has_delta = dr != nullptr || wy != nullptr;
    const bool write_back = (rows == nullptr) && has_delta;
    auto delta_at = [&](int c) -> float {
        if (dr) return ldf(dr + c);
        float acc = 0.f;
        for (int j = 0; j < k; ++j)
            acc += topk_w[(size_t)r * k + j] * ldf(wy + (size_t)pair_row[(size_t)r * k + j] * d + c);
        return acc;
    };
    float ss = 0.f;
    for (int c = threadIdx.x; c < d; c += blockDim.x) {
        float v = xr[c];
        if (has_delta) v += delta_at(c);
        if (write_back) xr[c] = v;
        ss += v * v;
    }
    ss = block_sum(ss, red);
    const float rs = w ? 1.0f / sqrtf(ss / (float)d + eps) : 1.f;      // no weights: the sum itself, rounded to T
    T* yr = y + (size_t)i * d;
    for (int c = threadIdx.x; c < d; c += blockDim.x) {
        float v = xr[c];
        if (has_delta && !write_back) v += delta_at(c);
        stf(yr + c, w ? v * rs * w[c] : v);
    }
}

// The same, eight values at a time with 16-byte accesses, the row kept in registers between the two
// passes.  For widths that are a multiple of 8 and at most threads * 8 * NORM_CHUNKS.
#define NORM_CHUNKS 4
// Two forms: for a few rows (decoding) 512 threads per row and the weights read before the dependency wait; for
// many rows (prompts) 256 lean threads, four blocks to an SM, since there the kernel is bound by memory traffic
// and the registers of the early read would halve what is resident.
// What a feed-forward may ask the norm before it to do in the same kernel (TAIL): the router of the row it has
// just normalized, i.e. the row's k experts and their weights, by the rules of router_kernel.  The row goes to
// shared memory as it goes to y (rounded to T), one warp per expert takes its dot product with the router's
// matrix (which it has asked for before the dependency wait), one warp picks.  A router kernel of its
// own would first wait for this kernel to end and then read the row back.
template <typename T> struct RouterTail {
    const T* w;        // [E, d], or null: none
    int E, k;
    int* idx;          // [rows, k]
    float* wts;        // [rows, k]
    RouterRule rule;   // how the logits become a choice
    int staged_at = 0; // where in shared memory the first row of the matrix of every warp goes (0: not staged)
};

// acc[0..8) += the weighted sum of row r's k rows of wy at column c: four rows' loads in flight, added in their order.
template <typename T> struct Raw8;
template <> struct Raw8<__nv_bfloat16> {
    uint4 a;
    __device__ __forceinline__ void load(const __nv_bfloat16* p) { a = *reinterpret_cast<const uint4*>(p); }
    __device__ __forceinline__ void get(float (&f)[8]) const { Vec16<__nv_bfloat16>::unpack(a, f); }
};
template <> struct Raw8<float> {
    float4 a, b;
    __device__ __forceinline__ void load(const float* p) {
        a = *reinterpret_cast<const float4*>(p);
        b = *reinterpret_cast<const float4*>(p + 4);
    }
    __device__ __forceinline__ void get(float (&f)[8]) const {
        f[0] = a.x; f[1] = a.y; f[2] = a.z; f[3] = a.w; f[4] = b.x; f[5] = b.y; f[6] = b.z; f[7] = b.w;
    }
};
template <typename T>
__device__ __forceinline__ void experts_sum(const T* __restrict__ wy, const int* __restrict__ pair_row,
                                            const float* __restrict__ topk_w, int k, int r, int d, int c, float (&acc)[8]) {
    for (int q0 = 0; q0 < k; q0 += 4) {
        Raw8<T> raw[4];
        float wq[4];
#pragma unroll
        for (int u = 0; u < 4; ++u)
            if (q0 + u < k) {
                raw[u].load(wy + (size_t)pair_row[(size_t)r * k + q0 + u] * d + c);
                wq[u] = topk_w[(size_t)r * k + q0 + u];
            }
#pragma unroll
        for (int u = 0; u < 4; ++u)
            if (q0 + u < k) {
                float t[8];
                raw[u].get(t);
#pragma unroll
                for (int e = 0; e < 8; ++e) acc[e] += wq[u] * t[e];
            }
    }
}

// CH: pieces of 8 values a thread keeps (NORM_THREADS * 8 * CH >= d), POST: whether post_w is given.  What a width or a form does
// not need costs registers, hence blocks on an SM, and code: 2,048 rows of 4,096 took 31 us (sums and experts' sums, mean)
// with room for 8,192 values and the experts' rows loaded one after the other, and take 24.
// TAIL: 0 no router behind the norm; otherwise where its matrix comes from: TAIL_EARLY a warp's first 8 KB in registers before the
// wait and the rest eight loads at a time, TAIL_SHORT from shared memory (`staged_at`) or four loads at a time.
#define TAIL_EARLY 1
#define TAIL_SHORT 2
template <typename T, int NORM_THREADS, bool EARLY, int TAIL, int CH, bool POST>
__global__ void __launch_bounds__(NORM_THREADS)
add_rmsnorm_vec_kernel(float* __restrict__ x, const T* __restrict__ delta, const T* __restrict__ wy,
                       const int* __restrict__ pair_row, const float* __restrict__ topk_w, int k,
                       const int* __restrict__ rows, const float* __restrict__ w, float eps, T* __restrict__ y,
                       int d, const void* warm, int warm_bytes, const RouterTail<T> tail,
                       const float* __restrict__ post_w, float post_eps) {
    // post_w: the delta is normed by itself first (delta / rms(delta) * post_w, with post_eps) and then added
    constexpr int EPL = Vec16<T>::N, UN = 8;
    // TAIL: the row as T [d], the logits [E] (and scores), and, if `staged`, a row of the router's matrix per warp [warps][d]
    extern __shared__ __align__(16) unsigned char tail_smem[];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    T* const ys = reinterpret_cast<T*>(tail_smem);
    T* const my_w = TAIL ? reinterpret_cast<T*>(tail_smem + tail.staged_at) + (size_t)warp * d : nullptr;
    uint4 first[TAIL == TAIL_EARLY ? UN : 1];
    if (TAIL == TAIL_EARLY) {
        if (warp < tail.E) {
#pragma unroll
            for (int u = 0; u < UN; ++u) {
                const int c = (lane + u * 32) * EPL;
                first[u] = make_uint4(0u, 0u, 0u, 0u);
                if (c < d) first[u] = *reinterpret_cast<const uint4*>(tail.w + (size_t)warp * d + c);
            }
        }
    } else if (TAIL == TAIL_SHORT) {
        if (tail.staged_at && warp < tail.E) {
#pragma unroll 1
            for (int c = lane * EPL; c < d; c += 32 * EPL)
                cp_async16((uint32_t)__cvta_generic_to_shared(my_w + c), tail.w + (size_t)warp * d + c);
            cp_async_commit();
        }
    }
    warm_l2(warm, warm_bytes);
    // this kernel's own weights do not depend on the kernel before it either: they are in registers by the time
    // the wait is over (they are read once per layer and have left L2 since the last step)
    float ww[EARLY ? CH : 1][8];
    if (EARLY && w) {
#pragma unroll
        for (int j = 0; j < CH; ++j) {
            const int c = (threadIdx.x + j * NORM_THREADS) * 8;
            if (c < d) load8(w + c, ww[j]);
        }
    }
    pdl_sync();
    __shared__ float red[33];
    const int i = blockIdx.x;
    const int r = rows ? rows[i] : i;
    float* xr = x + (size_t)r * d;
    const T* dr = delta ? delta + (size_t)r * d : nullptr;
    const bool has_delta = dr != nullptr || wy != nullptr;
    const bool write_back = (rows == nullptr) && has_delta;
    float v[CH][8];
    float ss = 0.f;
    if constexpr (POST) {
        float ss1 = 0.f;
#pragma unroll
        for (int j = 0; j < CH; ++j) {
            const int c = (threadIdx.x + j * NORM_THREADS) * 8;
            if (c < d) {
                if (dr) {
                    load8(dr + c, v[j]);
                } else {
#pragma unroll
                    for (int e = 0; e < 8; ++e) v[j][e] = 0.f;
                    experts_sum(wy, pair_row, topk_w, k, r, d, c, v[j]);
                }
#pragma unroll
                for (int e = 0; e < 8; ++e) ss1 += v[j][e] * v[j][e];
            }
        }
        ss1 = block_sum(ss1, red);
        const float rs1 = 1.0f / sqrtf(ss1 / (float)d + post_eps);
#pragma unroll
        for (int j = 0; j < CH; ++j) {
            const int c = (threadIdx.x + j * NORM_THREADS) * 8;
            if (c < d) {
                float xv[8], pw[8];
                load8(xr + c, xv);
                load8(post_w + c, pw);
#pragma unroll
                for (int e = 0; e < 8; ++e) {
                    v[j][e] = xv[e] + v[j][e] * rs1 * pw[e];
                    ss += v[j][e] * v[j][e];
                }
                if (write_back) store8(xr + c, v[j]);
            }
        }
    }
#pragma unroll
    for (int j = 0; j < CH; ++j) {
        const int c = (threadIdx.x + j * NORM_THREADS) * 8;
        if (c < d && !POST) {
            load8(xr + c, v[j]);
            if (dr) {
                float t[8];
                load8(dr + c, t);
#pragma unroll
                for (int e = 0; e < 8; ++e) v[j][e] += t[e];
            } else if (wy) {
                float acc[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
                experts_sum(wy, pair_row, topk_w, k, r, d, c, acc);
#pragma unroll
                for (int e = 0; e < 8; ++e) v[j][e] += acc[e];
            }
            if (write_back) store8(xr + c, v[j]);
#pragma unroll
            for (int e = 0; e < 8; ++e) ss += v[j][e] * v[j][e];
        }
    }
    if (!y) return;                 // the sum alone
    T* yr = y + (size_t)i * d;
    if (!w) {                       // no weights: y is the sum itself, rounded to T (a part that reads the stream as it is)
#pragma unroll
        for (int j = 0; j < CH; ++j) {
            const int c = (threadIdx.x + j * NORM_THREADS) * 8;
            if (c < d) store8(yr + c, v[j]);
        }
        return;
    }
    ss = block_sum(ss, red);
    const float rs = 1.0f / sqrtf(ss / (float)d + eps);
#pragma unroll
    for (int j = 0; j < CH; ++j) {
        const int c = (threadIdx.x + j * NORM_THREADS) * 8;
        if (c < d) {
            float o[8];
            if (!EARLY) load8(w + c, ww[0]);
#pragma unroll
            for (int e = 0; e < 8; ++e) o[e] = v[j][e] * rs * ww[EARLY ? j : 0][e];
            store8(yr + c, o);
            if (TAIL) store8(ys + c, o);
        }
    }
    if (!TAIL) return;
    __syncthreads();
    float* lg = reinterpret_cast<float*>(tail_smem + (size_t)d * sizeof(T));
    if (TAIL == TAIL_SHORT && tail.staged_at) cp_async_wait<0>();         // a lane reads what it copied itself
    for (int e = warp; e < tail.E; e += NORM_THREADS / 32) {
        const T* we = TAIL == TAIL_SHORT && tail.staged_at && e == warp ? my_w : tail.w + (size_t)e * d;
        float acc = 0.f;
        if (TAIL == TAIL_EARLY) {
            for (int c0 = lane * EPL; c0 < d; c0 += 32 * EPL * UN) {
                uint4 xv[UN], wv[UN];
                const bool have = e == warp && c0 == lane * EPL;     // the batch read before the wait
#pragma unroll
                for (int u = 0; u < UN; ++u) {
                    const int c = c0 + u * 32 * EPL;
                    xv[u] = wv[u] = make_uint4(0u, 0u, 0u, 0u);
                    if (c < d) {
                        xv[u] = *reinterpret_cast<const uint4*>(ys + c);
                        wv[u] = have ? first[TAIL == TAIL_EARLY ? u : 0] : *reinterpret_cast<const uint4*>(we + c);
                    }
                }
#pragma unroll
                for (int u = 0; u < UN; ++u) {
                    float xf[EPL], wf[EPL];
                    Vec16<T>::unpack(xv[u], xf);
                    Vec16<T>::unpack(wv[u], wf);
#pragma unroll
                    for (int q = 0; q < EPL; ++q) acc += xf[q] * wf[q];
                }
            }
        } else {
            // A loop of a few instructions: the block runs once, and code that has to be fetched for it costs more than it
            // saves (a step of one sequence, width 4,096, 16 experts: 9.0 us behind the kernel before with the row unrolled
            // in registers, 7.7 so)
#pragma unroll 4
            for (int c = lane * EPL; c < d; c += 32 * EPL) {
                float xf[EPL], wf[EPL];
                Vec16<T>::unpack(*reinterpret_cast<const uint4*>(ys + c), xf);
                Vec16<T>::unpack(*reinterpret_cast<const uint4*>(we + c), wf);
#pragma unroll
                for (int q = 0; q < EPL; ++q) acc += xf[q] * wf[q];
            }
        }
        acc = warp_sum(acc);
        if (lane == 0) lg[e] = acc;
    }
    __syncthreads();
    if (warp == 0) {
        if (tail.rule.scored == 1)
            router_pick_scored(lg, lg + tail.E, tail.rule.bias, tail.idx + (size_t)i * tail.k,
                               tail.wts + (size_t)i * tail.k, tail.E, tail.k, lane);
        else
            router_pick(lg, tail.idx + (size_t)i * tail.k, tail.wts + (size_t)i * tail.k, tail.E, tail.k, lane,
                        tail.rule.scored == 2);
    }
}

template <typename T>
__global__ void embed_vec_kernel(const int* __restrict__ tokens, const T* __restrict__ table, float* __restrict__ x,
                                 int d, float scale) {
    pdl_sync();
    const int i = blockIdx.x;
    const T* src = table + (size_t)tokens[i] * d;
    float* dst = x + (size_t)i * d;
    for (int c = threadIdx.x * 8; c < d; c += blockDim.x * 8) {
        float f[8];
        load8(src + c, f);
#pragma unroll
        for (int e = 0; e < 8; ++e) f[e] *= scale;      // a multiplication by one changes nothing
        store8(dst + c, f);
    }
}


// A block whose parts are normed AFTER they ran as well (x <- x + N_b(part(N_a(x)))) leaves this to the norm that
// follows it.  Row r = rows ? rows[i] : i:
//   u    = delta(r)                                         a part's output (or the experts' weighted sum, as above)
//   v    = x[r] + u / sqrt(mean(u^2) + post_eps) * post_w   both statistics and the sum in float
//   if (!rows) x[r] = v
//   if (y) y[i] = v / sqrt(mean(v^2) + eps) * w             one rounding to T
// The row lives in shared memory (d floats) between the passes.
template <typename T>
__global__ void __launch_bounds__(256)
post_add_rmsnorm_kernel(float* __restrict__ x, const T* __restrict__ delta, const T* __restrict__ wy,
                        const int* __restrict__ pair_row, const float* __restrict__ topk_w, int k,
                        const float* __restrict__ post_w, float post_eps, const int* __restrict__ rows,
                        const float* __restrict__ w, float eps, T* __restrict__ y, int d, const RouterTail<T> tail) {
    pdl_sync();
    extern __shared__ float row[];      // [d], and with a router tail its logits (and scores) behind
    __shared__ float red[33];
    const int i = blockIdx.x;
    const int r = rows ? rows[i] : i;
    float* xr = x + (size_t)r * d;
    const T* dr = delta ? delta + (size_t)r * d : nullptr;
    float ss = 0.f;
    for (int c = threadIdx.x; c < d; c += blockDim.x) {
        float u;
        if (dr) {
            u = ldf(dr + c);
        } else {
            u = 0.f;
            for (int j = 0; j < k; ++j)
                u += topk_w[(size_t)r * k + j] * ldf(wy + (size_t)pair_row[(size_t)r * k + j] * d + c);
        }
        row[c] = u;
        ss += u * u;
    }
    ss = block_sum(ss, red);
    const float rs1 = 1.0f / sqrtf(ss / (float)d + post_eps);
    float ss2 = 0.f;
    for (int c = threadIdx.x; c < d; c += blockDim.x) {
        const float v = xr[c] + row[c] * rs1 * post_w[c];
        if (!rows) xr[c] = v;
        row[c] = v;
        ss2 += v * v;
    }
    if (!y) return;
    T* yr = y + (size_t)i * d;
    if (!w) {                       // no weights: the sum itself, rounded to T (each thread wrote these entries itself)
        for (int c = threadIdx.x; c < d; c += blockDim.x) stf(yr + c, row[c]);
        return;
    }
    ss2 = block_sum(ss2, red);
    const float rs2 = 1.0f / sqrtf(ss2 / (float)d + eps);
    for (int c = threadIdx.x; c < d; c += blockDim.x) {
        stf(yr + c, row[c] * rs2 * w[c]);
        if (tail.w) row[c] = ldf(yr + c);       // what the router reads: the row as stored
    }
    if (!tail.w) return;
    // the router of the row just normed, by the rules of router_kernel: a warp per output, one warp picks
    __syncthreads();
    float* lg = row + d;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    for (int e = warp; e < tail.E; e += nw) {
        const T* we = tail.w + (size_t)e * d;
        float acc = 0.f;
        for (int c = lane; c < d; c += 32) acc += row[c] * ldf(we + c);
        acc = warp_sum(acc);
        if (lane == 0) lg[e] = acc;
    }
    __syncthreads();
    if (warp == 0) {
        if (tail.rule.scored == 1)
            router_pick_scored(lg, lg + tail.E, tail.rule.bias, tail.idx + (size_t)i * tail.k,
                               tail.wts + (size_t)i * tail.k, tail.E, tail.k, lane);
        else
            router_pick(lg, tail.idx + (size_t)i * tail.k, tail.wts + (size_t)i * tail.k, tail.E, tail.k, lane,
                        tail.rule.scored == 2);
    }
}

// x[i, :] = table[tok_i, :] * scale + pairs[row_i, :], where row_i is a hash of the token and the one before it in
// its sequence:  (prev * mul_prev + tok * mul_cur) mod buckets;  a sequence's first token takes row `buckets` (the
// table's last).  The token before a step's first one is per-sequence state (last_token [slots]); the thread
// block of a sequence's first token of the step reads it and then leaves the sequence's last token of the step there.
template <typename T>
__global__ void embed_bigram_kernel(const int* __restrict__ tokens, const int* __restrict__ tok_seq,
                                    const int* __restrict__ tok_pos, const int* __restrict__ seq_start,
                                    const int* __restrict__ slots, int* __restrict__ last_token,
                                    const T* __restrict__ table, const T* __restrict__ pairs, float* __restrict__ x,
                                    int d, float scale, int buckets, int mul_prev, int mul_cur) {
    pdl_sync();
    __shared__ int prev_s;
    const int i = blockIdx.x;
    const int tok = tokens[i];
    if (threadIdx.x == 0) {
        const int b = tok_seq[i];
        int prev;
        if (i == seq_start[b]) {
            int* keep = last_token + slots[b];
            prev = *keep;
            *keep = tokens[seq_start[b + 1] - 1];
        } else {
            prev = tokens[i - 1];
        }
        prev_s = prev;
    }
    __syncthreads();
    const int r = tok_pos[i] == 0 ? buckets
                                  : (int)(((long long)prev_s * mul_prev + (long long)tok * mul_cur) % (long long)buckets);
    const T* src = table + (size_t)tok * d;
    const T* add = pairs + (size_t)r * d;
    float* dst = x + (size_t)i * d;
    for (int c = threadIdx.x; c < d; c += blockDim.x) dst[c] = ldf(src + c) * scale + ldf(add + c);
}

template <typename T>
static int embed_bigram_launch(const int* tokens, const int* tok_seq, const int* tok_pos, const int* seq_start,
                               const int* slots, int* last_token, const void* table, const void* pairs, float* x,
                               int nt, int d, float scale, int buckets, int mul_prev, int mul_cur, cudaStream_t s) {
    if (nt < 0 || d <= 0 || buckets <= 0 || mul_prev < 0 || mul_cur < 0 || !last_token) return TB_ERR_ARG;
    if (nt == 0) return 0;
    TB_LAUNCH((embed_bigram_kernel<T>), nt, d >= 1024 ? 256 : 128, 0, s, tokens, tok_seq, tok_pos, seq_start, slots,
              last_token, (const T*)table, (const T*)pairs, x, d, scale, buckets, mul_prev, mul_cur);
    return tb_last_error();
}

// v[i] *= scale over n floats (logits with a fixed multiplier)
__global__ void scale_f32_kernel(float* __restrict__ v, long long n, float scale) {
    pdl_sync();
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
        v[i] *= scale;
}

template <typename T>
static int embed_launch(const int* tokens, const void* table, float* x, int nt, int d, float scale, cudaStream_t s) {
    if (nt < 0 || d <= 0) return TB_ERR_ARG;
    if (nt == 0) return 0;
    if (d % 8 == 0)
        TB_LAUNCH((embed_vec_kernel<T>), nt, 128, 0, s, tokens, (const T*)table, x, d, scale);
    else
        TB_LAUNCH((embed_kernel<T>), nt, 256, 0, s, tokens, (const T*)table, x, d, scale);
    return tb_last_error();
}
#define TAIL_SMEM (200 * 1024)
#define TAIL_STAGED_ROWS 16     // more rows: the blocks find the router's matrix in L2
#define TAIL_EARLY_ROWS 148     // more rows: the SMs take a second block, which the registers of the early read would not leave room for
// The kernel, allowed that much shared memory.
template <auto Kernel> static auto tail_kernel() {
    static PerDevice raised;
    tb_allow_smem(raised, (const void*)Kernel, TAIL_SMEM);
    return Kernel;
}

template <typename T>
static int add_rmsnorm_launch(float* x, const void* delta, const void* wy, const int* pair_row,
                              const float* topk_w, int k, const int* rows, const float* w, float eps,
                              void* y, int n_out, int d, const void* warm, int warm_bytes, cudaStream_t s,
                              RouterTail<T> tail = RouterTail<T>{nullptr, 0, 0, nullptr, nullptr, RouterRule{0, nullptr}},
                              const float* post_w = nullptr, float post_eps = 0.f) {
    if (n_out < 0 || d <= 0) return TB_ERR_ARG;
    if (post_w && !delta && !wy) return TB_ERR_ARG;
    if (!y && (!post_w || tail.w)) return TB_ERR_ARG;
    if (wy && (delta || !pair_row || !topk_w || k <= 0)) return TB_ERR_ARG;
    if (tail.w && (tail.E <= 0 || tail.k <= 0 || tail.k > tail.E || !tail.idx || !tail.wts)) return TB_ERR_ARG;
    if (n_out == 0) return 0;
    if (tail.w) {
        // the form that also routes: a few rows, a width of 16-byte pieces, the row and the logits in 40 KB
        const size_t smem = (size_t)d * sizeof(T) + (size_t)tail.E * sizeof(float) * (tail.rule.scored == 1 ? 2 : 1);
        if (d % 8 || d > 512 * 8 * NORM_CHUNKS || n_out > 256 || smem > 40 * 1024 ||
            (reinterpret_cast<uintptr_t>(tail.w) & 15))
            return TB_ERR_UNSUPPORTED;           // the caller runs the router by itself
        // a row of the router's matrix per warp joins them where it fits (128 KB for bfloat16 and a width of 4,096)
        const size_t at = (smem + 15) / 16 * 16, staged = (size_t)(tail.E < 16 ? tail.E : 16) * d * sizeof(T);
        if (at + staged <= TAIL_SMEM && n_out <= TAIL_STAGED_ROWS) tail.staged_at = (int)at;
        auto go = [&](auto kernel) {
            TB_LAUNCH(kernel, n_out, 512, tail.staged_at ? at + staged : smem, s, x, (const T*)delta, (const T*)wy, pair_row, topk_w, k,
                      rows, w, eps, (T*)y, d, nullptr, 0, tail, post_w, post_eps);
        };
        auto pick = [&](auto form) {
            constexpr int F = decltype(form)::value;
            if (post_w && d <= 512 * 8) go(tail_kernel<add_rmsnorm_vec_kernel<T, 512, true, F, 1, true>>());
            else if (post_w) go(tail_kernel<add_rmsnorm_vec_kernel<T, 512, true, F, NORM_CHUNKS, true>>());
            else if (d <= 512 * 8) go(tail_kernel<add_rmsnorm_vec_kernel<T, 512, true, F, 1, false>>());
            else go(tail_kernel<add_rmsnorm_vec_kernel<T, 512, true, F, NORM_CHUNKS, false>>());
        };
        if (!tail.staged_at && n_out <= TAIL_EARLY_ROWS) pick(std::integral_constant<int, TAIL_EARLY>());
        else pick(std::integral_constant<int, TAIL_SHORT>());
        return tb_last_error();
    }
    auto go = [&](auto kernel, int threads) {
        TB_LAUNCH(kernel, n_out, threads, 0, s, x, (const T*)delta, (const T*)wy, pair_row, topk_w, k, rows, w, eps, (T*)y, d, warm,
                  warm_bytes, tail, post_w, post_eps);
    };
    if (d % 8 == 0 && n_out <= 256 && d <= 512 * 8 * NORM_CHUNKS && y) {
        if (post_w && d <= 512 * 8) go(add_rmsnorm_vec_kernel<T, 512, true, 0, 1, true>, 512);
        else if (post_w) go(add_rmsnorm_vec_kernel<T, 512, true, 0, NORM_CHUNKS, true>, 512);
        else if (d <= 512 * 8) go(add_rmsnorm_vec_kernel<T, 512, true, 0, 1, false>, 512);
        else go(add_rmsnorm_vec_kernel<T, 512, true, 0, NORM_CHUNKS, false>, 512);
        return tb_last_error();
    }
    if (d % 8 == 0 && d <= 256 * 8 * NORM_CHUNKS) {
        if (post_w && d <= 256 * 8) go(add_rmsnorm_vec_kernel<T, 256, false, 0, 1, true>, 256);
        else if (post_w) go(add_rmsnorm_vec_kernel<T, 256, false, 0, NORM_CHUNKS, true>, 256);
        else if (d <= 256 * 8) go(add_rmsnorm_vec_kernel<T, 256, false, 0, 1, false>, 256);
        else if (d <= 256 * 8 * 2) go(add_rmsnorm_vec_kernel<T, 256, false, 0, 2, false>, 256);
        else go(add_rmsnorm_vec_kernel<T, 256, false, 0, NORM_CHUNKS, false>, 256);
        return tb_last_error();
    }
    if (post_w) return TB_ERR_UNSUPPORTED;      // the caller takes the kernel that keeps the row in shared memory
    int threads = d >= 2048 ? 512 : 256;
    TB_LAUNCH((add_rmsnorm_kernel<T>), n_out, threads, 0, s, x, (const T*)delta, (const T*)wy, pair_row, topk_w, k, rows, w, eps,
                                                   (T*)y, d, warm, warm_bytes);
    return tb_last_error();
}

template <typename T>
static int post_add_rmsnorm_launch(float* x, const void* delta, const void* wy, const int* pair_row,
                                   const float* topk_w, int k, const float* post_w, float post_eps, const int* rows,
                                   const float* w, float eps, void* y, int n_out, int d, cudaStream_t s,
                                   RouterTail<T> tail = RouterTail<T>{nullptr, 0, 0, nullptr, nullptr,
                                                                      RouterRule{0, nullptr}}) {
    if (n_out < 0 || d <= 0 || !post_w || (tail.w && !w)) return TB_ERR_ARG;
    if ((delta == nullptr) == (wy == nullptr)) return TB_ERR_ARG;
    if (wy && (!pair_row || !topk_w || k <= 0)) return TB_ERR_ARG;
    if (tail.w && (!y || tail.E <= 0 || tail.k <= 0 || tail.k > tail.E || !tail.idx || !tail.wts)) return TB_ERR_ARG;
    const size_t smem = ((size_t)d + (tail.w ? 2 * (size_t)tail.E : 0)) * sizeof(float);
    if (smem > 48 * 1024) return TB_ERR_UNSUPPORTED;
    if (n_out == 0) return 0;
    {
        // the forms that keep the row in registers and move 16 bytes at a time, for the widths they take
        const int rc = add_rmsnorm_launch<T>(x, delta, wy, pair_row, topk_w, k, rows, w, eps, y, n_out, d, nullptr, 0, s,
                                             tail, post_w, post_eps);
        if (rc != TB_ERR_UNSUPPORTED) return rc;
    }
    TB_LAUNCH((post_add_rmsnorm_kernel<T>), n_out, 256, smem, s, x, (const T*)delta, (const T*)wy,
              pair_row, topk_w, k, post_w, post_eps, rows, w, eps, (T*)y, d, tail);
    return tb_last_error();
}

extern "C" {
#define TB_EMBED_BIGRAM(NAME, T)                                                                                      \
    int NAME(const int* tokens, const int* tok_seq, const int* tok_pos, const int* seq_start, const int* slots,       \
             int* last_token, const void* table, const void* pairs, float* x, int nt, int d, float scale,             \
             int buckets, int mul_prev, int mul_cur, cudaStream_t s) {                                                \
        return embed_bigram_launch<T>(tokens, tok_seq, tok_pos, seq_start, slots, last_token, table, pairs, x, nt, d, \
                                      scale, buckets, mul_prev, mul_cur, s);                                          \
    }
TB_EMBED_BIGRAM(tb_embed_bigram_f32, float)
TB_EMBED_BIGRAM(tb_embed_bigram_bf16, __nv_bfloat16)
int tb_scale_f32(float* v, long long n, float scale, cudaStream_t s) {
    if (n < 0) return TB_ERR_ARG;
    if (n == 0) return 0;
    const long long blocks = (n + 255) / 256;
    TB_LAUNCH(scale_f32_kernel, (int)(blocks > 4096 ? 4096 : blocks), 256, 0, s, v, n, scale);
    return tb_last_error();
}
int tb_embed_f32(const int* tokens, const void* table, float* x, int nt, int d, cudaStream_t s) {
    return embed_launch<float>(tokens, table, x, nt, d, 1.0f, s);
}
// x[i] = table[tokens[i]] * scale, the product in float
int tb_embed_scaled_f32(const int* tokens, const void* table, float* x, int nt, int d, float scale, cudaStream_t s) {
    return embed_launch<float>(tokens, table, x, nt, d, scale, s);
}
int tb_embed_scaled_bf16(const int* tokens, const void* table, float* x, int nt, int d, float scale, cudaStream_t s) {
    return embed_launch<__nv_bfloat16>(tokens, table, x, nt, d, scale, s);
}
int tb_embed_bf16(const int* tokens, const void* table, float* x, int nt, int d, cudaStream_t s) {
    return embed_launch<__nv_bfloat16>(tokens, table, x, nt, d, 1.0f, s);
}
// x += norm(delta; post_w, post_eps), then y = norm(x; w, eps) (y may be null: the sum alone)
int tb_post_add_rmsnorm_f32(float* x, const void* delta, const void* wy, const int* pair_row, const float* topk_w,
                            int k, const float* post_w, float post_eps, const int* rows, const float* w, float eps,
                            void* y, int n_out, int d, cudaStream_t s) {
    return post_add_rmsnorm_launch<float>(x, delta, wy, pair_row, topk_w, k, post_w, post_eps, rows, w, eps, y, n_out,
                                          d, s);
}
int tb_post_add_rmsnorm_bf16(float* x, const void* delta, const void* wy, const int* pair_row, const float* topk_w,
                             int k, const float* post_w, float post_eps, const int* rows, const float* w, float eps,
                             void* y, int n_out, int d, cudaStream_t s) {
    return post_add_rmsnorm_launch<__nv_bfloat16>(x, delta, wy, pair_row, topk_w, k, post_w, post_eps, rows, w, eps,
                                                  y, n_out, d, s);
}
// The same, and the router of the rows just normed in the same kernel (router_w [E, d]; scored: the rule of
// tb_router_scored_*, with bias [E] or null; else the rule of tb_router_*).
#define TB_POST_ROUTER(NAME, T)                                                                                      \
    int NAME(float* x, const void* delta, const void* wy, const int* pair_row, const float* topk_w, int k,           \
             const float* post_w, float post_eps, const float* w, float eps, void* y, const void* router_w,          \
             const float* bias, int* route_idx, float* route_w, int n_out, int d, int E, int route_k, int scored,    \
             cudaStream_t s) {                                                                                       \
        if (!router_w) return TB_ERR_ARG;                                                                            \
        return post_add_rmsnorm_launch<T>(x, delta, wy, pair_row, topk_w, k, post_w, post_eps, nullptr, w, eps, y,   \
                                          n_out, d, s,                                                               \
                                          RouterTail<T>{(const T*)router_w, E, route_k, route_idx, route_w,          \
                                                        RouterRule{scored, bias}});                                  \
    }
TB_POST_ROUTER(tb_post_add_rmsnorm_router_f32, float)
TB_POST_ROUTER(tb_post_add_rmsnorm_router_bf16, __nv_bfloat16)
// warm / warm_bytes: weights that the next kernel reads first, to be asked into L2 meanwhile (or null / 0).
int tb_add_rmsnorm_f32(float* x, const void* delta, const void* wy, const int* pair_row, const float* topk_w, int k,
                       const int* rows, const float* w, float eps, void* y, int n_out, int d, const void* warm,
                       int warm_bytes, cudaStream_t s) {
    return add_rmsnorm_launch<float>(x, delta, wy, pair_row, topk_w, k, rows, w, eps, y, n_out, d, warm, warm_bytes, s);
}
int tb_add_rmsnorm_bf16(float* x, const void* delta, const void* wy, const int* pair_row, const float* topk_w, int k,
                        const int* rows, const float* w, float eps, void* y, int n_out, int d, const void* warm,
                        int warm_bytes, cudaStream_t s) {
    return add_rmsnorm_launch<__nv_bfloat16>(x, delta, wy, pair_row, topk_w, k, rows, w, eps, y, n_out, d, warm,
                                             warm_bytes, s);
}
// The same, and the router of the rows just normalized in the same kernel (router_w [E, d]; each row's route_k
// experts and weights into route_idx / route_w [n_out, route_k]).  TB_ERR_UNSUPPORTED for what it does not take
// (many rows, widths that are no multiple of 8 or do not fit shared memory): nothing has been done then.
int tb_add_rmsnorm_router_f32(float* x, const void* delta, const void* wy, const int* pair_row, const float* topk_w,
                              int k, const int* rows, const float* w, float eps, void* y, const void* router_w,
                              int* route_idx, float* route_w, int n_out, int d, int E, int route_k, cudaStream_t s) {
    if (!router_w) return TB_ERR_ARG;
    return add_rmsnorm_launch<float>(x, delta, wy, pair_row, topk_w, k, rows, w, eps, y, n_out, d, nullptr, 0, s,
                                     RouterTail<float>{(const float*)router_w, E, route_k, route_idx, route_w,
                                                       RouterRule{0, nullptr}});
}
int tb_add_rmsnorm_router_bf16(float* x, const void* delta, const void* wy, const int* pair_row, const float* topk_w,
                               int k, const int* rows, const float* w, float eps, void* y, const void* router_w,
                               int* route_idx, float* route_w, int n_out, int d, int E, int route_k, cudaStream_t s) {
    if (!router_w) return TB_ERR_ARG;
    return add_rmsnorm_launch<__nv_bfloat16>(
        x, delta, wy, pair_row, topk_w, k, rows, w, eps, y, n_out, d, nullptr, 0, s,
        RouterTail<__nv_bfloat16>{(const __nv_bfloat16*)router_w, E, route_k, route_idx, route_w,
                                  RouterRule{0, nullptr}});
}
// The same with the scored rule of choice (softmax over all outputs, the largest of score + bias, weights = scores).
int tb_add_rmsnorm_router_scored_f32(float* x, const void* delta, const void* wy, const int* pair_row,
                                     const float* topk_w, int k, const int* rows, const float* w, float eps, void* y,
                                     const void* router_w, const float* bias, int* route_idx, float* route_w, int n_out,
                                     int d, int E, int route_k, cudaStream_t s) {
    if (!router_w) return TB_ERR_ARG;
    return add_rmsnorm_launch<float>(x, delta, wy, pair_row, topk_w, k, rows, w, eps, y, n_out, d, nullptr, 0, s,
                                     RouterTail<float>{(const float*)router_w, E, route_k, route_idx, route_w,
                                                       RouterRule{1, bias}});
}
int tb_add_rmsnorm_router_scored_bf16(float* x, const void* delta, const void* wy, const int* pair_row,
                                      const float* topk_w, int k, const int* rows, const float* w, float eps, void* y,
                                      const void* router_w, const float* bias, int* route_idx, float* route_w,
                                      int n_out, int d, int E, int route_k, cudaStream_t s) {
    if (!router_w) return TB_ERR_ARG;
    return add_rmsnorm_launch<__nv_bfloat16>(
        x, delta, wy, pair_row, topk_w, k, rows, w, eps, y, n_out, d, nullptr, 0, s,
        RouterTail<__nv_bfloat16>{(const __nv_bfloat16*)router_w, E, route_k, route_idx, route_w, RouterRule{1, bias}});
}
}

// replayable from C++ (tape.h)
#include "tape.h"
TB_TAPE_REGISTER(tb_embed_f32)
TB_TAPE_REGISTER(tb_embed_bf16)
TB_TAPE_REGISTER(tb_embed_scaled_f32)
TB_TAPE_REGISTER(tb_embed_scaled_bf16)
TB_TAPE_REGISTER(tb_post_add_rmsnorm_f32)
TB_TAPE_REGISTER(tb_post_add_rmsnorm_bf16)
TB_TAPE_REGISTER(tb_post_add_rmsnorm_router_f32)
TB_TAPE_REGISTER(tb_post_add_rmsnorm_router_bf16)
TB_TAPE_REGISTER(tb_add_rmsnorm_f32)
TB_TAPE_REGISTER(tb_add_rmsnorm_bf16)
TB_TAPE_REGISTER(tb_add_rmsnorm_router_f32)
TB_TAPE_REGISTER(tb_add_rmsnorm_router_bf16)
TB_TAPE_REGISTER(tb_add_rmsnorm_router_scored_f32)
TB_TAPE_REGISTER(tb_add_rmsnorm_router_scored_bf16)
TB_TAPE_REGISTER(tb_embed_bigram_f32)
TB_TAPE_REGISTER(tb_embed_bigram_bf16)
TB_TAPE_REGISTER(tb_scale_f32)

// The matrix memory of mlstm.cu for long prompts: the chunks of a sequence side by side.
//
// mlstm_chunk_kernel walks a sequence chunk by chunk, and everything of a chunk of 64 tokens lies on that chain: 22 us a
// chunk, 700 us for 2,039 tokens of 8 heads (128 x 256), on 64 SMs.  But only two things have to follow one another: the
// running maximum m (a number per chunk) and S <- G S + U.  So:
//   mlstm_gates_kernel     a block = a sequence x a head: decays, weights and maxima of all its chunks
//   mlstm_update_kernel    a block = a chunk x a head x 128 rows x 128 columns: U = sum_j w_j k_j v_j^T (and n's alike)
//   mlstm_state_kernel     a thread = four entries of S: walks the chunks, leaves the state before each where U was
//   mlstm_rows_kernel      a block = a chunk x a head x 128 columns: scores, denominators, outputs
// A state per chunk is a lot of memory (8 heads of 128 x 256: 1 MB), so the last three take a portion of the chunks at a time, as
// many as the caller's scratch holds.
// 154 us for the 2,039 tokens (walked and side by side, us: two sequences of 4,000 1,385 and 621, 16 of 200 621 and 302; of 72 forms
// measured one lost: one head of 64 x 32 in 80 sequences of 200, 71 and 88).  Every sum is taken in the order of mlstm_chunk_kernel: the results are the same bit for bit.  Float throughout; the
// products are bound by multiply-adds on the CUDA cores with their operands in shared memory, 16 x 4 and 8 x 4 results a
// thread so that a 16-byte read feeds 13 and 11 of them.
#include "mlstm.cuh"

#define MP_THREADS 256
#define MP_COLS 128
#define MP_ROWS 128
#define MP_GATES 324            // floats of a chunk's gates: b, i, m, g, w [64] each, G, three of padding
#define MP_C (MC_L + 4)         // pitch of the scores

struct MlstmParallelArgs {
    MlstmArgs a;
    float* gates;               // [H][max_chunks][MP_GATES]
    float* work;                // [H][portion][mp_record]: n's sum [dim] | U, then the state before [dim][vdim]
    int max_chunks, portion;
    int base;                   // the portion's first chunk
};

__host__ __device__ inline size_t mp_record(int dim, int vdim) { return dim + (size_t)dim * vdim; }

// The sequence of chunk `chunk` of the step (counted over its sequences), or -1; `chunk` becomes its own number there.
__device__ __forceinline__ int mp_find(const int* seq_start, int B, int& chunk, int& t0, int& n) {
    for (int b = 0; b < B; ++b) {
        const int s = seq_start[b], len = seq_start[b + 1] - s, chunks = (len + MC_L - 1) / MC_L;
        if (chunk < chunks) {
            t0 = s + chunk * MC_L;
            n = min(MC_L, len - chunk * MC_L);
            return b;
        }
        chunk -= chunks;
    }
    return -1;
}

__device__ __forceinline__ size_t mp_state_size(int dim, int vdim) {
    return (size_t)dim * vdim + (size_t)((vdim + ML_COLS - 1) / ML_COLS) * (dim + 1);
}

__global__ void __launch_bounds__(MP_THREADS) mlstm_gates_kernel(const MlstmParallelArgs p) {
    pdl_sync();
    __shared__ float bL_s[MP_THREADS], xL_s[MP_THREADS], mp_s[MP_THREADS + 1];
    const MlstmArgs& a = p.a;
    const int b = blockIdx.x, h = blockIdx.y, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int t0 = a.seq_start[b], len = a.seq_start[b + 1] - t0;
    if (len <= 0) return;
    int first = 0;
    for (int i = 0; i < b; ++i) first += (a.seq_start[i + 1] - a.seq_start[i] + MC_L - 1) / MC_L;
    const int chunks = (len + MC_L - 1) / MC_L;
    float* n0 = a.state + ((size_t)a.slots[b] * a.H + h) * mp_state_size(a.dim, a.vdim) + (size_t)a.dim * a.vdim;
    const float bi = a.bias[h], bf = a.bias[a.H + h], cap = a.cap, inv_cap = 1.0f / a.cap;
    float m_prev = n0[a.dim];
    for (int base = 0; base < chunks; base += MP_THREADS) {
        const int here = min(MP_THREADS, chunks - base);
        for (int c = warp; c < here; c += MP_THREADS / 32) {
            float* w = p.gates + ((size_t)h * p.max_chunks + first + base + c) * MP_GATES;
            const int c0 = t0 + (base + c) * MC_L, nc = min(MC_L, len - (base + c) * MC_L);
            float fg[2], ig[2];
#pragma unroll
            for (int u = 0; u < 2; ++u) {
                const int t = lane + 32 * u;
                fg[u] = 0.f;
                ig[u] = -1e30f;            // a token that is not there: forgets nothing, writes nothing
                if (t < nc) {
                    const float zi = a.gates[(size_t)(c0 + t) * 2 * a.H + h], zf = a.gates[(size_t)(c0 + t) * 2 * a.H + a.H + h];
                    ig[u] = cap * tanhf((zi + bi) * inv_cap);
                    fg[u] = log_sigmoid(cap * tanhf((zf + bf) * inv_cap));
                }
            }
            const float b0 = warp_scan_add(fg[0], lane);
            const float b1 = warp_scan_add(fg[1], lane) + __shfl_sync(0xffffffffu, b0, 31);
            const float x0 = warp_scan_max(ig[0] - b0, lane);
            const float x1 = fmaxf(warp_scan_max(ig[1] - b1, lane), __shfl_sync(0xffffffffu, x0, 31));
            w[lane] = b0;                   w[lane + 32] = b1;
            w[MC_L + lane] = ig[0];         w[MC_L + lane + 32] = ig[1];
            w[2 * MC_L + lane] = x0;        w[2 * MC_L + lane + 32] = x1;      // becomes m below
            if (lane == 31) {
                bL_s[c] = b1;
                xL_s[c] = x1;
            }
        }
        __syncthreads();
        if (threadIdx.x == 0) {
            for (int c = 0; c < here; ++c) {
                mp_s[c] = m_prev;
                m_prev = bL_s[c] + fmaxf(m_prev, xL_s[c]);
            }
            mp_s[here] = m_prev;
        }
        __syncthreads();
        m_prev = mp_s[here];
        for (int c = warp; c < here; c += MP_THREADS / 32) {
            float* w = p.gates + ((size_t)h * p.max_chunks + first + base + c) * MP_GATES;
            const float mp = mp_s[c], bL = bL_s[c], mL = mp_s[c + 1];
#pragma unroll
            for (int u = 0; u < 2; ++u) {       // what this lane wrote above
                const int t = lane + 32 * u;
                const float bt = w[t], ig = w[MC_L + t], m = bt + fmaxf(mp, w[2 * MC_L + t]);
                w[2 * MC_L + t] = m;
                w[3 * MC_L + t] = expf(bt + mp - m);
                w[4 * MC_L + t] = expf(bL - bt + ig - mL);
            }
            if (lane == 0) w[5 * MC_L] = expf(bL + mp - mL);
        }
        __syncthreads();
    }
    for (int cb = threadIdx.x; cb < (a.vdim + ML_COLS - 1) / ML_COLS; cb += MP_THREADS) n0[(size_t)cb * (a.dim + 1) + a.dim] = m_prev;
}

// rows [64][cols] of a piece of the projections, as floats, zeros for tokens that are not there
__device__ __forceinline__ void mp_load(const MlstmArgs& a, int t0, int n, size_t at, int cols, int pitch, float scale, bool scaled,
                                        float* dst) {
    const __nv_bfloat16* X = static_cast<const __nv_bfloat16*>(a.qkv);
    const int per = cols / 8;
    for (int idx = threadIdx.x; idx < MC_L * per; idx += MP_THREADS) {
        const int t = idx / per, c = (idx - t * per) * 8;
        float f[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
        if (t < n) load8(X + (size_t)(t0 + t) * a.ld + at + c, f);
        if (scaled) {
#pragma unroll
            for (int e = 0; e < 8; ++e) f[e] *= scale;
        }
        store8(dst + t * pitch + c, f);
    }
}

__global__ void __launch_bounds__(MP_THREADS) mlstm_update_kernel(const MlstmParallelArgs p, int B) {
    pdl_sync();
    extern __shared__ __align__(16) float mp_sm[];
    const MlstmArgs& a = p.a;
    float* k_s = mp_sm;                         // [64][128]
    float* v_s = k_s + MC_L * MP_ROWS;          // [64][128], times w
    __shared__ float w_s[MC_L];
    const int row_blocks = (a.dim + MP_ROWS - 1) / MP_ROWS;
    const int h = blockIdx.y / row_blocks, r0 = blockIdx.y % row_blocks * MP_ROWS, col0 = blockIdx.z * MP_COLS;
    int chunk = p.base + blockIdx.x, t0, n;
    if (mp_find(a.seq_start, B, chunk, t0, n) < 0) return;
    const float* gates = p.gates + ((size_t)h * p.max_chunks + p.base + blockIdx.x) * MP_GATES;
    float* w = p.work + ((size_t)h * p.portion + blockIdx.x) * mp_record(a.dim, a.vdim);
    if (threadIdx.x < MC_L) w_s[threadIdx.x] = gates[4 * MC_L + threadIdx.x];
    const int rows = min(MP_ROWS, a.dim - r0), cols = min(MP_COLS, a.vdim - col0);
    mp_load(a, t0, n, (size_t)(a.H + h) * a.dim + r0, rows, MP_ROWS, 1.f, false, k_s);
    mp_load(a, t0, n, (size_t)2 * a.H * a.dim + (size_t)h * a.vdim + col0, cols, MP_COLS, 1.f, false, v_s);
    __syncthreads();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (lane * 4 < cols && warp * 16 < rows) {
        float upd[16][4];
#pragma unroll
        for (int i = 0; i < 16; ++i) upd[i][0] = upd[i][1] = upd[i][2] = upd[i][3] = 0.f;
#pragma unroll 2
        for (int j = 0; j < MC_L; ++j) {
            float4 v4 = *reinterpret_cast<const float4*>(v_s + j * MP_COLS + lane * 4);
            const float wj = w_s[j];
            v4.x *= wj; v4.y *= wj; v4.z *= wj; v4.w *= wj;
#pragma unroll
            for (int i4 = 0; i4 < 4; ++i4) {
                const float4 k4 = *reinterpret_cast<const float4*>(k_s + j * MP_ROWS + warp * 16 + i4 * 4);
                const float kv[4] = {k4.x, k4.y, k4.z, k4.w};
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    float* u = upd[i4 * 4 + e];
                    u[0] += kv[e] * v4.x; u[1] += kv[e] * v4.y; u[2] += kv[e] * v4.z; u[3] += kv[e] * v4.w;
                }
            }
        }
        float* U = w + a.dim;
#pragma unroll
        for (int i = 0; i < 16; ++i)
            if (warp * 16 + i < rows)
                *reinterpret_cast<float4*>(U + (size_t)(r0 + warp * 16 + i) * a.vdim + col0 + lane * 4) =
                    make_float4(upd[i][0], upd[i][1], upd[i][2], upd[i][3]);
    }
    if (blockIdx.z == 0 && threadIdx.x < rows) {
        float acc = 0.f;
        for (int j = 0; j < MC_L; ++j) acc += w_s[j] * k_s[j * MP_ROWS + threadIdx.x];
        w[r0 + threadIdx.x] = acc;
    }
}

// Entries of (n, S) four at a time: n's sums lie right before U in a chunk's record.  Loads run four chunks ahead.  A sequence that
// goes on in the next portion leaves its state where that portion finds it: in the cache.
__global__ void __launch_bounds__(MP_THREADS) mlstm_state_kernel(const MlstmParallelArgs p) {
    pdl_sync();
    const MlstmArgs& a = p.a;
    const int b = blockIdx.x, h = blockIdx.y, dim = a.dim, vdim = a.vdim;
    const int t0 = a.seq_start[b], len = a.seq_start[b + 1] - t0;
    const int at = (blockIdx.z * MP_THREADS + threadIdx.x) * 4;
    if (len <= 0 || at >= dim + dim * vdim) return;
    int first = 0;
    for (int i = 0; i < b; ++i) first += (a.seq_start[i + 1] - a.seq_start[i] + MC_L - 1) / MC_L;
    // its chunks in this portion, counted from the portion's first
    const int lo = max(first, p.base) - p.base, chunks = min(first + (len + MC_L - 1) / MC_L, p.base + p.portion) - p.base - lo;
    if (chunks <= 0) return;
    const size_t rec = mp_record(dim, vdim);
    float* S = a.state + ((size_t)a.slots[b] * a.H + h) * mp_state_size(dim, vdim);
    float* w = p.work + ((size_t)h * p.portion + lo) * rec;
    const float* gates = p.gates + ((size_t)h * p.max_chunks + p.base + lo) * MP_GATES;
    const bool is_n = at < dim;                 // dim is a multiple of four
    float s[4];
#pragma unroll
    for (int e = 0; e < 4; ++e) s[e] = is_n ? S[(size_t)dim * vdim + at + e] : S[at - dim + e];
    for (int c0 = 0; c0 < chunks; c0 += 4) {
        float4 u[4];
        float G[4];
#pragma unroll
        for (int i = 0; i < 4; ++i)
            if (c0 + i < chunks) {
                u[i] = *reinterpret_cast<const float4*>(w + (c0 + i) * rec + at);
                G[i] = gates[(c0 + i) * MP_GATES + 5 * MC_L];
            }
#pragma unroll
        for (int i = 0; i < 4; ++i)
            if (c0 + i < chunks) {
                *reinterpret_cast<float4*>(w + (c0 + i) * rec + at) = make_float4(s[0], s[1], s[2], s[3]);
                s[0] = G[i] * s[0] + u[i].x;
                s[1] = G[i] * s[1] + u[i].y;
                s[2] = G[i] * s[2] + u[i].z;
                s[3] = G[i] * s[3] + u[i].w;
            }
    }
    if (is_n) {
        for (int cb = 0; cb < (vdim + ML_COLS - 1) / ML_COLS; ++cb)
#pragma unroll
            for (int e = 0; e < 4; ++e) S[(size_t)dim * vdim + (size_t)cb * (dim + 1) + at + e] = s[e];
    } else {
#pragma unroll
        for (int e = 0; e < 4; ++e) S[at - dim + e] = s[e];
    }
}

__global__ void __launch_bounds__(MP_THREADS, 2) mlstm_rows_kernel(const MlstmParallelArgs p, int B) {
    pdl_sync();
    extern __shared__ __align__(16) float mp_sm[];
    const MlstmArgs& a = p.a;
    const int dim = a.dim, vdim = a.vdim, H = a.H, kp = dim + 4;
    float* q_s = mp_sm;                                             // [64][dim], later v [64][128]
    float* k_s = q_s + MC_L * (dim > MP_COLS ? dim : MP_COLS);      // [64][dim + 4], later rows of S
    float* C_s = k_s + MC_L * kp;                                   // [64][MP_C]
    __shared__ float gate[5 * MC_L], den_s[MC_L];
    __shared__ float n_s[256];
    const int h = blockIdx.y, col0 = blockIdx.z * MP_COLS, tid = threadIdx.x;
    int chunk = p.base + blockIdx.x, t0, n;
    if (mp_find(a.seq_start, B, chunk, t0, n) < 0) return;
    const float* gates = p.gates + ((size_t)h * p.max_chunks + p.base + blockIdx.x) * MP_GATES;
    const float* w = p.work + ((size_t)h * p.portion + blockIdx.x) * mp_record(dim, vdim);
    for (int i = tid; i < 5 * MC_L; i += MP_THREADS) gate[i] = gates[i];
    if (tid < dim) n_s[tid] = w[tid];
    const float *b_s = gate, *ig_s = gate + MC_L, *m_s = gate + 2 * MC_L, *g_s = gate + 3 * MC_L;
    mp_load(a, t0, n, (size_t)h * dim, dim, dim, a.qscale, true, q_s);
    mp_load(a, t0, n, (size_t)(H + h) * dim, dim, kp, 1.f, false, k_s);
    __syncthreads();
    {   // C_tj = D_tj (q_t . k_j): a thread takes tokens ti + 16 u and keys ji + 16 u'
        const int ti = tid >> 4, ji = tid & 15;
        float acc[4][4];
#pragma unroll
        for (int u = 0; u < 4; ++u)
#pragma unroll
            for (int x = 0; x < 4; ++x) acc[u][x] = 0.f;
        for (int c = 0; c < dim; c += 4) {
            float4 q4[4], k4[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                q4[u] = *reinterpret_cast<const float4*>(q_s + (ti + 16 * u) * dim + c);
                k4[u] = *reinterpret_cast<const float4*>(k_s + (ji + 16 * u) * kp + c);
            }
#pragma unroll
            for (int u = 0; u < 4; ++u)
#pragma unroll
                for (int x = 0; x < 4; ++x) {
                    acc[u][x] += q4[u].x * k4[x].x;
                    acc[u][x] += q4[u].y * k4[x].y;
                    acc[u][x] += q4[u].z * k4[x].z;
                    acc[u][x] += q4[u].w * k4[x].w;
                }
        }
#pragma unroll
        for (int u = 0; u < 4; ++u)
#pragma unroll
            for (int x = 0; x < 4; ++x) {
                const int t = ti + 16 * u, j = ji + 16 * x;
                C_s[t * MP_C + j] = j <= t ? acc[u][x] * expf(b_s[t] - b_s[j] + ig_s[j] - m_s[t]) : 0.f;
            }
    }
    __syncthreads();
    const int cols = min(MP_COLS, vdim - col0), lane = tid & 31, warp = tid >> 5, half = dim / 2;
    float* S_s = k_s;                   // [dim / 2][128]: fits 64 x (dim + 4)
    auto load_state = [&](int r0) {
        const float* S = w + dim + (size_t)r0 * vdim + col0;
        for (int idx = tid; idx < half * (MP_COLS / 4); idx += MP_THREADS) {
            const int r = idx / (MP_COLS / 4), c = idx % (MP_COLS / 4) * 4;
            if (c < cols) *reinterpret_cast<float4*>(S_s + r * MP_COLS + c) = *reinterpret_cast<const float4*>(S + (size_t)r * vdim + c);
        }
    };
    load_state(0);
    {   // denominators: four neighbouring lanes share a token's dot products (q_t . n' and the row sum of C)
        const int t = tid >> 2, part = tid & 3;
        float dot = 0.f;
        for (int r = part; r < dim; r += 4) dot += q_s[t * dim + r] * n_s[r];
        dot *= g_s[t];
        for (int j = part; j <= t; j += 4) dot += C_s[t * MP_C + j];
        dot += __shfl_xor_sync(0xffffffffu, dot, 1);
        dot += __shfl_xor_sync(0xffffffffu, dot, 2);
        if (part == 0) den_s[t] = fmaxf(fabsf(dot), expf(-m_s[t])) + ML_DENOM_FLOOR;
    }
    // numerators: a warp takes 8 tokens, a lane 4 columns
    float num[8][4];
#pragma unroll
    for (int i = 0; i < 8; ++i) num[i][0] = num[i][1] = num[i][2] = num[i][3] = 0.f;
    auto add = [&](const float* left, int pitch, const float* right, int count) {
#pragma unroll 1
        for (int r = 0; r < count; r += 4) {
            float4 s4[4];
#pragma unroll
            for (int e = 0; e < 4; ++e) s4[e] = *reinterpret_cast<const float4*>(right + (r + e) * MP_COLS + lane * 4);
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                const float4 x4 = *reinterpret_cast<const float4*>(left + (warp * 8 + i) * pitch + r);
                const float x[4] = {x4.x, x4.y, x4.z, x4.w};
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    num[i][0] += x[e] * s4[e].x; num[i][1] += x[e] * s4[e].y;
                    num[i][2] += x[e] * s4[e].z; num[i][3] += x[e] * s4[e].w;
                }
            }
        }
    };
    __syncthreads();
    add(q_s, dim, S_s, half);
    __syncthreads();
    load_state(half);
    __syncthreads();
    add(q_s + half, dim, S_s, half);
    __syncthreads();
    mp_load(a, t0, n, (size_t)2 * H * dim + (size_t)h * vdim + col0, cols, MP_COLS, 1.f, false, q_s);
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const float g = g_s[warp * 8 + i];
#pragma unroll
        for (int e = 0; e < 4; ++e) num[i][e] *= g;
    }
    __syncthreads();
    add(C_s, MP_C, q_s, MC_L);
    if (lane * 4 >= cols) return;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const int t = warp * 8 + i;
        if (t < n) {
            const float den = den_s[t];
            *reinterpret_cast<float4*>(a.out + (size_t)(t0 + t) * H * vdim + (size_t)h * vdim + col0 + lane * 4) =
                make_float4(num[i][0] / den, num[i][1] / den, num[i][2] / den, num[i][3] / den);
        }
    }
}

static bool mlstm_parallel_takes(int H, int dim, int vdim, int ld) {
    return dim > 0 && dim <= 256 && dim % 8 == 0 && vdim > 0 && vdim % ML_COLS == 0 && ld % 8 == 0 && H > 0;
}

extern "C" {
// Floats of scratch per (head, chunk of 64 tokens of a portion), or 0 where these kernels do not take such heads and rows, and
// per (head, chunk of the step).
int tb_mlstm_parallel_size(int H, int dim, int vdim, int ld) {
    return mlstm_parallel_takes(H, dim, vdim, ld) ? (int)mp_record(dim, vdim) : 0;
}
int tb_mlstm_parallel_gates() { return MP_GATES; }
int tb_mlstm_parallel_tokens() { return MC_L; }

// As tb_mlstm_chunk_bf16; gate_work [H][max_chunks][tb_mlstm_parallel_gates], max_chunks >= nt / 64 + B; work
// [H][portion][tb_mlstm_parallel_size].
int tb_mlstm_parallel_bf16(const void* qkv, const float* gates, const float* bias, float* state, float* out, float* work,
                           float* gate_work, const int* seq_start, const int* slots, int nt, int B, int ld, int H, int dim,
                           int vdim, int max_chunks, int portion, float cap, float qscale, cudaStream_t s) {
    if (nt < 0 || B < 0 || H <= 0 || dim <= 0 || vdim <= 0 || max_chunks < 0 || portion < 1 || !(cap > 0.f)) return TB_ERR_ARG;
    if (!mlstm_parallel_takes(H, dim, vdim, ld) || (((uintptr_t)qkv | (uintptr_t)work | (uintptr_t)out) & 15)) return TB_ERR_UNSUPPORTED;
    if (nt == 0 || B == 0) return 0;
    if (max_chunks < nt / MC_L + (B < nt ? B : nt)) return TB_ERR_ARG;
    MlstmParallelArgs p{MlstmArgs{qkv, gates, bias, state, out, seq_start, slots, ld, H, dim, vdim, cap, qscale}, gate_work, work,
                        max_chunks, portion, 0};
    const size_t smem_u = (size_t)2 * MC_L * 128 * sizeof(float);
    const size_t smem_r = (size_t)MC_L * ((dim > MP_COLS ? dim : MP_COLS) + dim + 4 + MP_C) * sizeof(float);      // 147 KB for dim 256
    static PerDevice raised[2];
    tb_allow_smem(raised[0], (const void*)mlstm_update_kernel, 80 * 1024);
    tb_allow_smem(raised[1], (const void*)mlstm_rows_kernel, 160 * 1024);
    const int col_blocks = (vdim + MP_COLS - 1) / MP_COLS, row_blocks = (dim + MP_ROWS - 1) / MP_ROWS;
    TB_LAUNCH(mlstm_gates_kernel, dim3(B, H), MP_THREADS, 0, s, p);
    for (; p.base < max_chunks; p.base += portion) {
        const int count = max_chunks - p.base < portion ? max_chunks - p.base : portion;
        TB_LAUNCH(mlstm_update_kernel, dim3(count, H * row_blocks, col_blocks), MP_THREADS, smem_u, s, p, B);
        TB_LAUNCH(mlstm_state_kernel, dim3(B, H, (dim + dim * vdim + 4 * MP_THREADS - 1) / (4 * MP_THREADS)), MP_THREADS, 0, s, p);
        TB_LAUNCH(mlstm_rows_kernel, dim3(count, H, col_blocks), MP_THREADS, smem_r, s, p, B);
    }
    return tb_last_error();
}
}

#include "tape.h"
TB_TAPE_REGISTER(tb_mlstm_parallel_bf16)

// Grouped matrix product on the CUDA cores, float accumulation:  C[m, :] = A[row(m), :] . B[g(m)]^T
//
// This is the matrix product of the true 32-bit path (plain FFMA, no reduced-precision matrix
// mode) and the fallback of the bfloat16 path for shapes the tensor-core kernels refuse.
//
//  * B holds G matrices [N, K] row-major (weights as stored: y = x W^T,
//    models/llama/common/src/lib.rs:168-180); rows of the problem are sorted by group and
//    group_offsets[g] .. group_offsets[g+1] are the rows of group g (the experts of
//    models/llama/common/src/compute.rs:319-330, all tokens of one expert in one product instead of
//    a product per token).  G = 1 with no offsets is the plain product.
//  * a_rows, when given, gathers: row m reads A[a_rows[m]].
//  * DUAL: B[g] is [2N, K]; the block computes gate = A.B[g][n] and up = A.B[g][N + n] together and
//    stores silu(gate) * up  (swiglu, compute.rs:324-326), in float, rounded once.
//  Any M, N, K >= 1; edges are predicated.
//
// Three kernels: gemm_simt_kernel takes anything; for float with 16-byte rows of GF_K entries or more, gemm_rows_f32_kernel
// streams the weights past a few rows (decoding), and gemm_tile_f32_kernel multiplies tiles fed by cp.async (prompts).  The three
// take a sum in different orders, so the last bits of a row depend on how many rows (of its group, on average) the call has.
#include "attention_prefill.cuh"        // cp_async16, cp_async_commit, cp_async_wait
#include "memory_common.cuh"            // fma2

#include <type_traits>

struct GemmArgs {
    const void* A;
    const int* a_rows;
    const void* B;
    void* C;
    const int* group_offsets;
    long long b_group_stride;   // elements between B[g] and B[g+1]
    int lda, ldb, ldc;
    int M, N, K, G;
    GluRule glu;                // DUAL: how the (gate, up) pair becomes one value
    long long a_batch_stride;   // blockIdx.z = batch: elements between the batches' A, B (b_group_stride) and C;
    long long c_batch_stride;   // zero without batches
};

// Which rows does tile `tile` of BM rows hold?  False: none.
template <int BM>
__device__ __forceinline__ bool gemm_tile_rows(const GemmArgs& a, int tile, int& g, int& row0, int& row_end) {
    g = 0;
    row0 = tile * BM;
    row_end = a.M;
    if (!a.group_offsets) return row0 < a.M;
    int cum = 0;
    for (g = 0; g < a.G; ++g) {
        const int lo = a.group_offsets[g], hi = a.group_offsets[g + 1];
        const int tiles = (hi - lo + BM - 1) / BM;
        if (tile < cum + tiles) {
            row0 = lo + (tile - cum) * BM;
            row_end = hi;
            return true;
        }
        cum += tiles;
    }
    return false;
}

__device__ __forceinline__ float gemm_act(float v, float v2, bool dual, const GluRule r) {
    if (dual) return glu_apply(v, v2, r);
    if (r.kind == TB_ACT_RELU2) {
        v = fmaxf(v, 0.f);
        v *= v;
    }
    return v;
}

#define GB_N 64
#define GB_K 16

template <typename T, typename TC, int BM, bool DUAL>
__global__ void __launch_bounds__(256) gemm_simt_kernel(const GemmArgs a) {
    pdl_sync();
    constexpr int TM = BM / 16;
    __shared__ float As[GB_K][BM + 1];
    __shared__ float Bs[GB_K][GB_N + 1];
    __shared__ float B2s[DUAL ? GB_K : 1][GB_N + 1];

    int g, row0, row_end;
    if (!gemm_tile_rows<BM>(a, blockIdx.x, g, row0, row_end)) return;
    const int n0 = blockIdx.y * GB_N;
    if (gridDim.z > 1) g = blockIdx.z;      // batches: every batch has a matrix of its own and all the rows
    const T* A = static_cast<const T*>(a.A) + (size_t)blockIdx.z * a.a_batch_stride;
    const T* B = static_cast<const T*>(a.B) + (size_t)g * a.b_group_stride;

    const int tid = threadIdx.x;
    const int tx = tid & 15, ty = tid >> 4;   // tx: columns (4 each), ty: rows (TM each)
    float acc[TM][4], acc2[DUAL ? TM : 1][4];
#pragma unroll
    for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = 0.f;
#pragma unroll
    for (int i = 0; i < (DUAL ? TM : 1); ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc2[i][j] = 0.f;

    // loader roles: B tile 64 x 16 -> 4 elements a thread; A tile BM x 16 -> BM*16/256 a thread
    const int lb_r = tid >> 2, lb_k = (tid & 3) * 4;
    constexpr int A_PER = BM * GB_K / 256;   // 4 (BM 64) or 1 (BM 16)
    const int la_r = (tid * A_PER) / GB_K, la_k = (tid * A_PER) % GB_K;
    const int a_row = row0 + la_r;
    const T* a_ptr = nullptr;
    if (a_row < row_end) a_ptr = A + (size_t)(a.a_rows ? a.a_rows[a_row] : a_row) * a.lda;
    const int b_row = n0 + lb_r;
    const T* b_ptr = b_row < a.N ? B + (size_t)b_row * a.ldb : nullptr;
    const T* b2_ptr = (DUAL && b_row < a.N) ? B + (size_t)(a.N + b_row) * a.ldb : nullptr;

    for (int k0 = 0; k0 < a.K; k0 += GB_K) {
#pragma unroll
        for (int i = 0; i < A_PER; ++i) {
            const int k = k0 + la_k + i;
            As[la_k + i][la_r] = (a_ptr && k < a.K) ? ldf(a_ptr + k) : 0.f;
        }
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int k = k0 + lb_k + i;
            Bs[lb_k + i][lb_r] = (b_ptr && k < a.K) ? ldf(b_ptr + k) : 0.f;
            if (DUAL) B2s[lb_k + i][lb_r] = (b2_ptr && k < a.K) ? ldf(b2_ptr + k) : 0.f;
        }
        __syncthreads();
#pragma unroll
        for (int k = 0; k < GB_K; ++k) {
            float av[TM], bv[4], b2v[4];
#pragma unroll
            for (int i = 0; i < TM; ++i) av[i] = As[k][ty * TM + i];
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                bv[j] = Bs[k][tx * 4 + j];
                if (DUAL) b2v[j] = B2s[k][tx * 4 + j];
            }
#pragma unroll
            for (int i = 0; i < TM; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    acc[i][j] += av[i] * bv[j];
                    if (DUAL) acc2[i][j] += av[i] * b2v[j];
                }
        }
        __syncthreads();
    }

    TC* C = static_cast<TC*>(a.C) + (size_t)blockIdx.z * a.c_batch_stride;
#pragma unroll
    for (int i = 0; i < TM; ++i) {
        const int m = row0 + ty * TM + i;
        if (m >= row_end) continue;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int n = n0 + tx * 4 + j;
            if (n >= a.N) continue;
            stf(C + (size_t)m * a.ldc + n, gemm_act(acc[i][j], acc2[DUAL ? i : 0][j], DUAL, a.glu));
        }
    }
}

// ---- a few rows (decoding) -----------------------------------------------------------------------------------------
// Bound by reading the weights once.  A warp owns CT rows of W (DUAL: CT / 2 gate rows and their up rows) and every
// WK-th piece of 128 entries of K: a lane holds 16 bytes of each row, so a warp has CT x 512 bytes in flight, and the
// rows of A (up to MT at a time, from L1) meet them in registers.  WK warps of a block share its columns; a warp's
// MT x CT sums are joined by a reduce-scatter (31 shuffles for 32 sums), the warps' through shared memory.  The general
// kernel walks K in steps of 16 with two barriers each and was bound by that chain: 3 rows x 1,536
// x 1,024 took 55.7 us and take 3.0 (2.1 TB/s), x 32,000 x 1,024 275 and 34 us (3.9 TB/s), 16 rows x 1,536 x 1,024 56.4
// and 7.1 us; a decode step of three sequences (width 1,024, 8 layers, 8 experts of 512) 4.6 and 0.58 ms.
// SLICED (many rows, no pair): the rows of a crowded group are dealt to several blocks, 16 passes each.  2,048 rows for 128 experts
// (512 -> 1,024) that all went to one: 442 us by the blocks of that expert alone (the general kernel: 390), 217 so; evenly
// spread 223 and 212.  A pair has twice the work a row and stays ahead of the general kernel without (424 and 714 us; dealt out, its
// registers run out and an even spread costs 7 % more).
#define GR_PASSES 16
template <int MT, int CT, bool DUAL, bool SLICED>
__global__ void __launch_bounds__(256) gemm_rows_f32_kernel(const GemmArgs a, int wk_count) {
    constexpr int COLS = DUAL ? CT / 2 : CT;
    constexpr int SETS = MT * CT / 32;
    static_assert(MT * CT % 32 == 0, "the reduce-scatter takes 32 sums at a time");
    __shared__ float red[8][MT * CT];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int wk = warp % wk_count, wn = warp / wk_count, wn_count = (blockDim.x >> 5) / wk_count;
    int g = blockIdx.y;
    const int n0 = (blockIdx.x * wn_count + wn) * COLS;
    if (!a.group_offsets && lane % 8 == 0) {
        // Which rows of W a block reads does not depend on the kernel before it: their first pieces are asked into L2 while
        // that one still runs (into L2 only, where a W that it is writing stays what it is): a request of 3 sequences and 12
        // sampled tokens, 8 layers of width 1,024, 6.54 to 6.39 ms.
        const int k = wk * 128 + lane * 4;
        if (k < a.K)
#pragma unroll
            for (int c = 0; c < CT; ++c)
                asm volatile("prefetch.global.L2 [%0];" ::"l"(static_cast<const float*>(a.B) + (size_t)g * a.b_group_stride +
                             (size_t)(min(n0 + c % COLS, a.N - 1) + (DUAL && c >= COLS ? a.N : 0)) * a.ldb + k));
    }
    pdl_sync();
    int row_lo = 0, row_hi = a.M;
    if (!SLICED && a.group_offsets) {
        row_lo = a.group_offsets[g];
        row_hi = a.group_offsets[g + 1];
    }
    if (SLICED) {
        constexpr int SLICE = GR_PASSES * MT;
        int slice = 0;
        if (g >= a.G) {         // a slice behind some group's first: which?  (32 groups at a time, every warp by itself)
            int want = g - a.G;
            g = -1;
            for (int g0 = 0; g0 < a.G && g < 0; g0 += 32) {
                int more = 0;
                if (g0 + lane < a.G) more = (a.group_offsets[g0 + lane + 1] - a.group_offsets[g0 + lane] - 1) / SLICE;
                int upto = more;
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) {
                    const int u = __shfl_up_sync(0xffffffffu, upto, o);
                    if (lane >= o) upto += u;
                }
                const unsigned past = __ballot_sync(0xffffffffu, want < upto);
                if (past) {
                    const int src = __ffs(past) - 1;
                    g = g0 + src;
                    slice = want - __shfl_sync(0xffffffffu, upto - more, src) + 1;
                }
                want -= __shfl_sync(0xffffffffu, upto, 31);
            }
            if (g < 0) return;
        }
        row_lo = a.group_offsets[g] + slice * SLICE;
        row_hi = min(a.group_offsets[g + 1], row_lo + SLICE);
    }
    if (row_lo >= row_hi) return;
    const float* B = static_cast<const float*>(a.B) + (size_t)g * a.b_group_stride;
    const float* A = static_cast<const float*>(a.A);
    const float* wp[CT];
#pragma unroll
    for (int c = 0; c < CT; ++c) {      // columns past the end repeat the last one and are not stored
        const int n = min(n0 + c % COLS, a.N - 1) + (DUAL && c >= COLS ? a.N : 0);
        wp[c] = B + (size_t)n * a.ldb;
    }
    for (int chunk = row_lo; chunk < row_hi; chunk += MT) {
        const int rows = min(MT, row_hi - chunk);
        float acc[MT * CT];
        const float* xp[MT];            // rows past the end repeat the last one and are not stored
#pragma unroll
        for (int i = 0; i < MT * CT; ++i) acc[i] = 0.f;
#pragma unroll
        for (int m = 0; m < MT; ++m) {
            const int r = chunk + min(m, rows - 1);
            xp[m] = A + (size_t)(a.a_rows ? a.a_rows[r] : r) * a.lda;
        }
        for (int k = wk * 128 + lane * 4; k < a.K; k += wk_count * 128) {
            float4 w[CT];
#pragma unroll
            for (int c = 0; c < CT; ++c) w[c] = __ldcs(reinterpret_cast<const float4*>(wp[c] + k));
#pragma unroll
            for (int m0 = 0; m0 < MT; m0 += 4) {
                if (m0 < rows) {
                    float4 x[4];
#pragma unroll
                    for (int m = 0; m < 4; ++m) x[m] = *reinterpret_cast<const float4*>(xp[m0 + m] + k);
#pragma unroll
                    for (int m = 0; m < 4; ++m)
#pragma unroll
                        for (int c = 0; c < CT; ++c) {
                            float& v = acc[(m0 + m) * CT + c];
                            v = fmaf(x[m].x, w[c].x, v);
                            v = fmaf(x[m].y, w[c].y, v);
                            v = fmaf(x[m].z, w[c].z, v);
                            v = fmaf(x[m].w, w[c].w, v);
                        }
                }
            }
        }
        if (chunk != row_lo) __syncthreads();       // the sums of the rows before have been read
#pragma unroll
        for (int set = 0; set < SETS; ++set) {
            float* v = acc + set * 32;
#pragma unroll
            for (int half = 16; half > 0; half >>= 1) {      // a lane keeps the half of the sums that its bit names
                const bool up = lane & half;
#pragma unroll
                for (int i = 0; i < half; ++i) {
                    const float keep = up ? v[i + half] : v[i], give = up ? v[i] : v[i + half];
                    v[i] = keep + __shfl_xor_sync(0xffffffffu, give, half);
                }
            }
            red[warp][set * 32 + lane] = v[0];
        }
        __syncthreads();
        for (int idx = threadIdx.x; idx < wn_count * rows * COLS; idx += blockDim.x) {
            const int c = idx % COLS, m = idx / COLS % rows, w_n = idx / (COLS * rows);
            const int n = (blockIdx.x * wn_count + w_n) * COLS + c;
            if (n >= a.N) continue;
            float v = 0.f, v2 = 0.f;
            for (int w = 0; w < wk_count; ++w) {
                v += red[w_n * wk_count + w][m * CT + c];
                if (DUAL) v2 += red[w_n * wk_count + w][m * CT + COLS + c];
            }
            static_cast<float*>(a.C)[(size_t)(chunk + m) * a.ldc + n] = gemm_act(v, v2, DUAL, a.glu);
        }
    }
}

template <int MT, int CT, bool DUAL>
static void gemm_rows_f32_go(const GemmArgs& a, cudaStream_t s) {
    // as many warps on K as it has pieces of 128 entries, up to eight; with fewer than four (K below GF_K, which the launcher keeps
    // away), more columns a block
    const int wk = a.K >= 1024 ? 8 : a.K >= 512 ? 4 : a.K >= 256 ? 2 : 1;
    const int warps = wk == 8 ? 8 : 4, cols = (DUAL ? CT / 2 : CT) * (warps / wk);
    // Without offsets all rows belong to matrix 0, whatever G is: a block for every g would write the same places.
    const int groups = a.group_offsets ? a.G : 1, blocks = (a.N + cols - 1) / cols;
    const int more = a.group_offsets ? (a.M - 1) / (GR_PASSES * MT) : 0;        // slices behind the groups' first: at most so many
    if (!DUAL && more > 0) TB_LAUNCH((gemm_rows_f32_kernel<MT, CT, DUAL, !DUAL>), dim3(blocks, groups + more), warps * 32, 0, s, a, wk);
    else TB_LAUNCH((gemm_rows_f32_kernel<MT, CT, DUAL, false>), dim3(blocks, groups), warps * 32, 0, s, a, wk);
}

// ---- many rows (prompts) -------------------------------------------------------------------------------------------
// 64 x 64 outputs a block, 32 x 32 a warp, 8 x 4 a thread; K in steps of 32 through a ring of three stages filled by
// cp.async.  Four warps take the first 16 entries of a step and four the others, and their sums are joined at the end:
// a prompt of a few hundred tokens has fewer tiles than the GPU has SMs, and one warp a scheduler does not hide the
// latencies of its own loads.  Tiles lie in shared memory as in memory (K innermost, rows 36 floats apart: the eight
// rows that a quarter of a warp reads start in different banks), so a thread's operands are 16-byte loads of four
// entries of K: 12 of them feed 128 multiply-adds, two an instruction.  Bound by multiply-add issue.  The general kernel reads one float
// at a time (8 loads for 16 multiply-adds) and waits for global memory in every step.  us, here and there:
// 254 rows x 1,536 x 1,024 38 and 84, a pair of 2,816 125 and 258, pairs of 8 experts (1,024 -> 512, 508 rows) 64 and 182, 2,048 x 4,096 x
// 4,096 1,956 and 3,240.
#define GT_BK 32
#define GT_PITCH (GT_BK + 4)
#define GT_STAGES 3
template <bool DUAL>
__global__ void __launch_bounds__(256) gemm_tile_f32_kernel(const GemmArgs a) {
    constexpr int NB = DUAL ? 2 : 1;
    extern __shared__ __align__(16) float gt[];
    constexpr int STAGE = (1 + NB) * 64 * GT_PITCH;        // A, then the one or two tiles of B
    pdl_sync();
    int g, row0, row_end;
    if (!gemm_tile_rows<64>(a, blockIdx.x, g, row0, row_end)) return;
    const int n0 = blockIdx.y * 64, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const float* A = static_cast<const float*>(a.A);
    const float* B = static_cast<const float*>(a.B) + (size_t)g * a.b_group_stride;
    // a thread copies 16 bytes of rows r0 and r0 + 32 of each tile; rows and columns past the end repeat the last one
    const int r0 = tid >> 3, kq = (tid & 7) * 4;
    const float* src[(1 + NB) * 2];
#pragma unroll
    for (int i = 0; i < 2; ++i) {
        const int m = min(row0 + r0 + 32 * i, row_end - 1), n = min(n0 + r0 + 32 * i, a.N - 1);
        src[i] = A + (size_t)(a.a_rows ? a.a_rows[m] : m) * a.lda + kq;
        src[2 + i] = B + (size_t)n * a.ldb + kq;
        if (DUAL) src[2 * NB + i] = B + (size_t)(a.N + n) * a.ldb + kq;
    }
    const int steps = (a.K + GT_BK - 1) / GT_BK;
    auto issue = [&](int step) {
        float* st = gt + (step % GT_STAGES) * STAGE;
        const int k = step * GT_BK;
#pragma unroll
        for (int i = 0; i < (1 + NB) * 2; ++i) {
            float* dst = st + ((i >> 1) * 64 + r0 + 32 * (i & 1)) * GT_PITCH + kq;
            if (k + kq < a.K) cp_async16((uint32_t)__cvta_generic_to_shared(dst), src[i] + k);
            else *reinterpret_cast<float4*>(dst) = make_float4(0.f, 0.f, 0.f, 0.f);
        }
    };
    F2 acc2[NB][8][4];              // sums over the even and the odd entries of K
#pragma unroll
    for (int b = 0; b < NB; ++b)
#pragma unroll
        for (int i = 0; i < 8; ++i)
#pragma unroll
            for (int j = 0; j < 4; ++j) acc2[b][i][j].f = make_float2(0.f, 0.f);
#pragma unroll
    for (int st = 0; st < GT_STAGES - 1; ++st) {
        if (st < steps) issue(st);
        cp_async_commit();
    }
    const int ty = lane >> 3, tx = lane & 7, wm = (warp >> 1 & 1) * 32, wn = (warp & 1) * 32;
    const int k_half = warp >> 2;
    union Four { float4 f; F2 p[2]; };
    for (int st = 0; st < steps; ++st) {
        cp_async_wait<GT_STAGES - 2>();
        __syncthreads();            // this stage is there for everyone, and everyone is done with the one before
        if (st + GT_STAGES - 1 < steps) issue(st + GT_STAGES - 1);
        cp_async_commit();
        const float* As = gt + (st % GT_STAGES) * STAGE + (wm + ty) * GT_PITCH + k_half * (GT_BK / 2);
        const float* Bs = gt + (st % GT_STAGES) * STAGE + (64 + wn + tx) * GT_PITCH + k_half * (GT_BK / 2);
#pragma unroll 2
        for (int k = 0; k < GT_BK / 2; k += 4) {
            Four av[8];
#pragma unroll
            for (int i = 0; i < 8; ++i) av[i].f = *reinterpret_cast<const float4*>(As + 4 * i * GT_PITCH + k);
#pragma unroll
            for (int b = 0; b < NB; ++b)
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    Four bv;
                    bv.f = *reinterpret_cast<const float4*>(Bs + (b * 64 + 8 * j) * GT_PITCH + k);
#pragma unroll
                    for (int i = 0; i < 8; ++i) {
                        F2& v = acc2[b][i][j];
                        v = fma2(av[i].p[0], bv.p[0], v);
                        v = fma2(av[i].p[1], bv.p[1], v);
                    }
                }
        }
    }
    float acc[NB][8][4];
#pragma unroll
    for (int b = 0; b < NB; ++b)
#pragma unroll
        for (int i = 0; i < 8; ++i)
#pragma unroll
            for (int j = 0; j < 4; ++j) acc[b][i][j] = acc2[b][i][j].f.x + acc2[b][i][j].f.y;
    // the second half's sums to shared memory (a warp's 32 x NB values a lane, lane innermost), the first half adds them
    __syncthreads();
    float* part = gt + (warp & 3) * (NB * 1024) + lane;
    if (k_half) {
#pragma unroll
        for (int b = 0; b < NB; ++b)
#pragma unroll
            for (int i = 0; i < 32; ++i) part[(b * 32 + i) * 32] = acc[b][i >> 2][i & 3];
    }
    __syncthreads();
    if (k_half) return;
#pragma unroll
    for (int b = 0; b < NB; ++b)
#pragma unroll
        for (int i = 0; i < 32; ++i) acc[b][i >> 2][i & 3] += part[(b * 32 + i) * 32];
    float* C = static_cast<float*>(a.C);
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const int m = row0 + wm + ty + 4 * i;
        if (m >= row_end) continue;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int n = n0 + wn + tx + 8 * j;
            if (n < a.N) C[(size_t)m * a.ldc + n] = gemm_act(acc[0][i][j], acc[NB - 1][i][j], DUAL, a.glu);
        }
    }
}

// The float kernels with 16-byte loads, for rows that start on such a boundary and K in multiples of four; false: the
// caller takes the general kernel.  Up to 16 rows (a group, on average) the weights are what is read, and the rows are
// taken 4, 8 or 16 at a time by what most groups hold, as gemm_skinny does; above, tiles.  Measured at the border: 16
// rows x 1,536 x 1,024 7.1 us here, 17 rows 39 us in tiles; a pair of 8 experts (1,024 -> 512) 25 us for groups of 15 rows
// here, 73 for groups of 25 in tiles (one tile a group, mostly empty, and the general kernel's 200 and 219).
// Rows shorter than GF_K stay with the general kernel, not because it is faster (calls from Python one after the other: 254 rows x
// 1,024 x 252 22.6 us, x 256 in tiles 12.8; 3 rows x 512 x 128 13 us with either) but because its walk over K is short there and models
// that small keep the results they had: a tiny model of the tests has a token whose logits another order of the sums moves by 1.1e-4
// where the mean error is 6e-6 in either order.
#define GF_K 512
static bool gemm_f32_launch(const GemmArgs& a, bool dual, cudaStream_t s) {
    if (a.K < GF_K || a.K % 4 || a.lda % 4 || a.ldb % 4 || a.b_group_stride % 4 || (((uintptr_t)a.A | (uintptr_t)a.B) & 15)) return false;
    const int G = a.group_offsets ? a.G : 1;
    if (a.M <= 16 * G && G + a.M / (GR_PASSES * 4) <= 65535) {       // blocks in y, with passes of four rows
        const int usual = G > 1 ? (3 * a.M / G + 1) / 2 : a.M;
        if (usual <= 4) dual ? gemm_rows_f32_go<4, 8, true>(a, s) : gemm_rows_f32_go<4, 8, false>(a, s);
        else if (usual <= 8) dual ? gemm_rows_f32_go<8, 8, true>(a, s) : gemm_rows_f32_go<8, 8, false>(a, s);
        else dual ? gemm_rows_f32_go<16, 4, true>(a, s) : gemm_rows_f32_go<16, 4, false>(a, s);
        return true;
    }
    const int tiles = (a.M + 63) / 64 + (a.group_offsets ? a.G : 0), cols = (a.N + 63) / 64;
    if (cols > 65535) return false;
    const size_t smem = (size_t)GT_STAGES * (dual ? 3 : 2) * 64 * GT_PITCH * sizeof(float);
    static PerDevice raised[2];
    tb_allow_smem(raised[dual], dual ? (const void*)gemm_tile_f32_kernel<true> : (const void*)gemm_tile_f32_kernel<false>, smem);
    if (dual) TB_LAUNCH((gemm_tile_f32_kernel<true>), dim3(tiles, cols), 256, smem, s, a);
    else TB_LAUNCH((gemm_tile_f32_kernel<false>), dim3(tiles, cols), 256, smem, s, a);
    return true;
}

template <typename T, typename TC, bool DUAL>
static int gemm_simt_launch(const GemmArgs& a, cudaStream_t s, int batches = 1) {
    if (a.M < 0 || a.N <= 0 || a.K <= 0 || a.G <= 0 || batches <= 0 || batches > 65535) return TB_ERR_ARG;
    if (a.M == 0) return 0;
    if constexpr (std::is_same<T, float>::value) {
        if (batches == 1 && gemm_f32_launch(a, DUAL, s)) return tb_last_error();
    }
    const bool small = a.M <= 16 * a.G;
    const int bm = small ? 16 : 64;
    // every group may end in a partly filled tile
    const int tiles = a.group_offsets ? (a.M + bm - 1) / bm + a.G : (a.M + bm - 1) / bm;
    dim3 grid(tiles, (a.N + GB_N - 1) / GB_N, batches);
    if (small)
        TB_LAUNCH((gemm_simt_kernel<T, TC, 16, DUAL>), grid, 256, 0, s, a);
    else
        TB_LAUNCH((gemm_simt_kernel<T, TC, 64, DUAL>), grid, 256, 0, s, a);
    return tb_last_error();
}

// A few rows against one matrix per batch (decoding: the heads of a mixer whose heads have matrices of their own):
// C[m, b, n] = sum_k A[m, b, k] B[b, n, k].  One warp per output column streams that column's row of B once (its
// lanes stride over k) and keeps one sum per row of A; A is small and comes from cache.  Up to BR_ROWS rows.
// (Measured and dropped: a column per lane with 16-byte loads of its row, A in shared memory, the warps splitting K:
// the same time alone, and 5 % slower in the replayed decode step, where these many small blocks overlap better with
// their neighbours in the stream.)
#define BR_ROWS 16
template <typename T>
__global__ void __launch_bounds__(256)
batched_rows_kernel(const T* __restrict__ A, const T* __restrict__ B, T* __restrict__ C, long long a_stride,
                    long long b_stride, long long c_stride, int lda, int ldb, int ldc, int M, int N, int K) {
    pdl_sync();
    const int lane = threadIdx.x & 31, n = blockIdx.x * 8 + (threadIdx.x >> 5), b = blockIdx.y;
    if (n >= N) return;
    const T* Bn = B + (size_t)b * b_stride + (size_t)n * ldb;
    const T* Ab = A + (size_t)b * a_stride;
    float acc[BR_ROWS];
#pragma unroll
    for (int m = 0; m < BR_ROWS; ++m) acc[m] = 0.f;
    for (int k = lane; k < K; k += 32) {
        const float w = ldf(Bn + k);
#pragma unroll
        for (int m = 0; m < BR_ROWS; ++m)
            if (m < M) acc[m] += w * ldf(Ab + (size_t)m * lda + k);
    }
#pragma unroll
    for (int m = 0; m < BR_ROWS; ++m) {
        if (m < M) {
            const float v = warp_sum(acc[m]);
            if (lane == 0) stf(C + (size_t)b * c_stride + (size_t)m * ldc + n, v);
        }
    }
}



extern "C" {
// out_kind: 0 = C has the type of A and B, 1 = C is float, 2 = swiglu pair (C has the type of A),
// 3 = max(., 0)^2 of the product (C has the type of A)
#define TB_GEMM(NAME, T)                                                                                        \
    int NAME(const void* A, const int* a_rows, const void* B, void* C, const int* group_offsets,               \
             long long b_group_stride, int lda, int ldb, int ldc, int M, int N, int K, int G, int out_kind,    \
             cudaStream_t s) {                                                                                  \
        GemmArgs a{A, a_rows, B, C, group_offsets, b_group_stride, lda, ldb, ldc, M, N, K, G, GluRule{0, 0.f, 0.f}, \
                   0, 0};                                                                                       \
        if (out_kind == 0) return gemm_simt_launch<T, T, false>(a, s);                                          \
        if (out_kind == 1) return gemm_simt_launch<T, float, false>(a, s);                                      \
        if (out_kind == 2) return gemm_simt_launch<T, T, true>(a, s);                                           \
        if (out_kind == 3) {                                                                                    \
            a.glu.kind = TB_ACT_RELU2;                                                                          \
            return gemm_simt_launch<T, T, false>(a, s);                                                         \
        }                                                                                                       \
        return TB_ERR_ARG;                                                                                      \
    }
TB_GEMM(tb_gemm_simt_f32, float)
TB_GEMM(tb_gemm_simt_bf16, __nv_bfloat16)

// The (gate, up) pair product with another form of the pair than silu(g) u (see GluRule): kind 1 the clamped form with
// alpha and limit, kind 3 the tanh form of gelu on the gate.
#define TB_GEMM_GLU(NAME, T)                                                                                    \
    int NAME(const void* A, const int* a_rows, const void* B, void* C, const int* group_offsets,               \
             long long b_group_stride, int lda, int ldb, int ldc, int M, int N, int K, int G, float alpha,     \
             float limit, int kind, cudaStream_t s) {                                                           \
        if (kind != 1 && kind != TB_GLU_GELU_TANH) return TB_ERR_ARG;                                           \
        GemmArgs a{A, a_rows, B, C, group_offsets, b_group_stride, lda, ldb, ldc, M, N, K, G,                   \
                   GluRule{kind, alpha, limit}, 0, 0};                                                             \
        return gemm_simt_launch<T, T, true>(a, s);                                                              \
    }
TB_GEMM_GLU(tb_gemm_simt_glu_f32, float)
TB_GEMM_GLU(tb_gemm_simt_glu_bf16, __nv_bfloat16)

// `batches` independent products of the same shape: batch b reads A + b * a_stride (rows M, pitch lda), the matrix
// B + b * b_stride [N, K] and writes C + b * c_stride (the heads of a mixer whose heads have matrices of their own).
#define TB_GEMM_BATCHED(NAME, T)                                                                                \
    int NAME(const void* A, const void* B, void* C, long long a_stride, long long b_stride, long long c_stride, \
             int lda, int ldb, int ldc, int M, int N, int K, int batches, cudaStream_t s) {                     \
        if (M > 0 && M <= BR_ROWS && N > 0 && K > 0 && batches > 0 && batches <= 65535) {                       \
            TB_LAUNCH((batched_rows_kernel<T>), dim3((N + 7) / 8, batches), 256, 0, s, (const T*)A, (const T*)B, (T*)C, \
                      a_stride, b_stride, c_stride, lda, ldb, ldc, M, N, K);                                    \
            return tb_last_error();                                                                             \
        }                                                                                                       \
        GemmArgs a{A, nullptr, B, C, nullptr, b_stride, lda, ldb, ldc, M, N, K, 1, GluRule{0, 0.f, 0.f},        \
                   a_stride, c_stride};                                                                         \
        return gemm_simt_launch<T, T, false>(a, s, batches);                                                    \
    }
TB_GEMM_BATCHED(tb_gemm_simt_batched_f32, float)
TB_GEMM_BATCHED(tb_gemm_simt_batched_bf16, __nv_bfloat16)
}

// replayable from C++ (tape.h)
#include "tape.h"
TB_TAPE_REGISTER(tb_gemm_simt_f32)
TB_TAPE_REGISTER(tb_gemm_simt_bf16)
TB_TAPE_REGISTER(tb_gemm_simt_glu_f32)
TB_TAPE_REGISTER(tb_gemm_simt_glu_bf16)
TB_TAPE_REGISTER(tb_gemm_simt_batched_f32)
TB_TAPE_REGISTER(tb_gemm_simt_batched_bf16)

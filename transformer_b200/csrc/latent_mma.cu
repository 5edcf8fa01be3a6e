// Attention over the cached latents on the tensor cores (bfloat16, mma.sync.m16n8k16), for prompts and decoding.
//
// The math is that of latent.cu: rows (token, head) of one sequence, all reading the same cached rows [c | kr]
// as keys and their first `rank` entries as values; a query at position p sees 0 <= p - j < window.
//
// One block = 16 rows (the M of one mma tile: up to 16 heads of a token, or several tokens of a few heads) x one
// slice of the key range.  Keys come a page (64 keys) at a time into shared memory with cp.async.  Per page:
//   1. scores: warp w takes keys 16 w .. 16 w + 15:  S_w = Q K_w^T over all rank + rot entries (A: the queries from
//      shared memory, B: the page's rows as they lie, both by ldmatrix), scaled, to shared memory as floats;
//   2. softmax: warp w takes rows 4 w .. 4 w + 3: mask by position and window, running maximum and sum (float, in
//      registers), the weights as bfloat16 and the rows' rescaling factors to shared memory;
//   3. values: warp w owns rank / 4 of the output's columns: O_w = O_w * factor + P V_w (B: the page's rows by
//      ldmatrix.trans), float accumulators in registers for the whole key range.
// With more than one slice a block leaves (maximum, sum, unnormalized output) and latent_merge_kernel joins them.
//
// Sizes: rank a multiple of 32 up to 512, rank + rot a multiple of 16; anything else goes to the general kernel.
#include "latent_common.cuh"

// warps per block: 4 (any rank that is a multiple of 32), or 8 when the rank is a multiple of 64: twice the warps
// on an SM to hide the latencies of a k-step's chain of ldmatrix and mma (with four, no unit was busy for more than
// a third of the time and an SM held eight warps)
#define LM_ROWS 16
#define LM_KEYS TB_PAGE     // keys per tile = one page

__device__ __forceinline__ void lm_ldmatrix_x4(unsigned (&r)[4], const void* p) {
    const unsigned addr = (unsigned)__cvta_generic_to_shared(p);
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr));
}
__device__ __forceinline__ void lm_ldmatrix_x4_trans(unsigned (&r)[4], const void* p) {
    const unsigned addr = (unsigned)__cvta_generic_to_shared(p);
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr));
}
__device__ __forceinline__ void lm_mma(float (&d)[4], const unsigned (&a)[4], unsigned b0, unsigned b1) {
    asm volatile(
        "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ void lm_cp16(void* dst, const void* src) {
    const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(d), "l"(src));
}

// The 16 rows' queries to shared memory: the latent's side as it is (16 bytes at a time), the rotated part rotated here,
// both unscaled.
__device__ __forceinline__ void lm_load_queries(const LatentMmaArgs& a, __nv_bfloat16* q_s, int pitch, int t0, int n_tok, int h0) {
    const int hc = a.heads_per_block;
    const int chunks_q = a.rank / 8;
    for (int idx = threadIdx.x; idx < LM_ROWS * chunks_q; idx += blockDim.x) {
        const int row = idx / chunks_q, c = (idx - row * chunks_q) * 8;
        const int ti = row / hc, h = h0 + row % hc;
        uint4 v = make_uint4(0u, 0u, 0u, 0u);
        if (ti < n_tok && h < a.H)
            v = *reinterpret_cast<const uint4*>(a.qa + ((size_t)(t0 + ti) * a.H + h) * a.rank + c);
        *reinterpret_cast<uint4*>(q_s + row * pitch + c) = v;
    }
    for (int idx = threadIdx.x; idx < LM_ROWS * a.rot; idx += blockDim.x) {
        const int row = idx / a.rot, r = idx - row * a.rot;
        const int ti = row / hc, h = h0 + row % hc;
        float v = 0.f;
        if (ti < n_tok && h < a.H) {
            const int t = t0 + ti;
            v = lm_turned(a, a.q + (size_t)t * a.ldq + (size_t)h * a.q_head + a.q_plain, r, a.tok_pos[t]);
        }
        q_s[row * pitch + a.rank + r] = __float2bfloat16_rn(v);
    }
}

// NT = n8 tiles of the output per warp (rank / 4 / 8, rounded up to the instantiated sizes)
template <int NT, int LM_WARPS>
__global__ void __launch_bounds__(LM_WARPS * 32) latent_mma_kernel(const LatentMmaArgs a) {
    constexpr int KPW = LM_KEYS / LM_WARPS;      // keys of a page per warp in the scores' phase: 16 or 8
    constexpr int RPW = LM_ROWS / LM_WARPS;      // rows per warp in the softmax phase: 4 or 2
    pdl_sync();
    extern __shared__ __align__(16) unsigned char lm_smem[];
    const int DK = a.rank + a.rot;
    const int pitch = DK + 8;                                   // in elements: rows 16 bytes apart modulo 128
    __nv_bfloat16* q_s = reinterpret_cast<__nv_bfloat16*>(lm_smem);                    // [16][pitch]
    __nv_bfloat16* k_s = q_s + LM_ROWS * pitch;                                         // [64][pitch]
    float* s_s = reinterpret_cast<float*>(k_s + LM_KEYS * pitch);                       // [16][64 + 1]
    __nv_bfloat16* p_s = reinterpret_cast<__nv_bfloat16*>(s_s + LM_ROWS * (LM_KEYS + 1));   // [16][64 + 8]
    float* corr_s = reinterpret_cast<float*>(p_s + LM_ROWS * (LM_KEYS + 8));            // [16] factors, then [16] sums
    int* pos_s = reinterpret_cast<int*>(corr_s + 2 * LM_ROWS);                          // [16] positions, -1: no row
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int g = lane >> 2, t4 = lane & 3;
    const int tile = blockIdx.x, h0 = blockIdx.y * a.heads_per_block, slice = blockIdx.z;
    const int seq = a.tile_seq[tile], t0 = a.tile_t0[tile];
    const int hc = a.heads_per_block;
    const int n_tok = min(a.tile_nq[tile], a.tokens_per_block);
    lm_load_queries(a, q_s, pitch, t0, n_tok, h0);
    if (threadIdx.x < LM_ROWS) {
        const int ti = threadIdx.x / hc, h = h0 + threadIdx.x % hc;
        pos_s[threadIdx.x] = (ti < n_tok && h < a.H) ? a.tok_pos[t0 + ti] : -1;
    }
    const int p_first = a.tok_pos[t0], p_last = a.tok_pos[t0 + n_tok - 1];
    const int lo = max(p_first - a.window + 1, 0);
    // pages of this slice
    const int pg_lo = lo / LM_KEYS, pg_hi = p_last / LM_KEYS;          // inclusive
    const int per = (pg_hi - pg_lo + 1 + a.splits - 1) / a.splits;
    const int pg0 = pg_lo + slice * per, pg1 = min(pg_hi, pg0 + per - 1);
    const int* table = a.page_table + (size_t)seq * a.max_pages;
    float acc[NT][4];
#pragma unroll
    for (int i = 0; i < NT; ++i) acc[i][0] = acc[i][1] = acc[i][2] = acc[i][3] = 0.f;
    float mx[RPW], sum[RPW];           // of rows RPW warp .. (the same in every lane)
#pragma unroll
    for (int r = 0; r < RPW; ++r) {
        mx[r] = -INFINITY;
        sum[r] = 0.f;
    }
    const int cols_w = a.rank / LM_WARPS;                                // output columns of this warp
    const int chunks = DK / 8;                                           // 16-byte pieces of a cached row
    __syncthreads();
    for (int pg = pg0; pg <= pg1; ++pg) {
        const __nv_bfloat16* src = a.cache + (size_t)table[pg] * TB_PAGE * DK;
        for (int idx = threadIdx.x; idx < LM_KEYS * chunks; idx += blockDim.x) {
            const int kk = idx / chunks, c8 = idx - kk * chunks;
            lm_cp16(k_s + kk * pitch + c8 * 8, src + (size_t)kk * DK + c8 * 8);
        }
        asm volatile("cp.async.commit_group;\ncp.async.wait_group 0;" ::: "memory");
        __syncthreads();
        // ---- 1. scores of this warp's keys ----------------------------------------------------------------------
        if constexpr (LM_WARPS == 8) {
            // 8 keys = one tile of 8 columns; one ldmatrix.x4 of the keys serves two k-steps
            float sc[4] = {0.f, 0.f, 0.f, 0.f}, sd[4] = {0.f, 0.f, 0.f, 0.f};
            const __nv_bfloat16* qa_p = q_s + (lane & 15) * pitch + (lane >> 4) * 8;
            const __nv_bfloat16* kb_p = k_s + (warp * 8 + (lane & 7)) * pitch + (lane >> 3) * 8;
            int k0 = 0;
#pragma unroll 2
            for (; k0 + 32 <= DK; k0 += 32) {
                unsigned af[4], ag[4], bf[4];
                lm_ldmatrix_x4(bf, kb_p + k0);
                lm_ldmatrix_x4(af, qa_p + k0);
                lm_ldmatrix_x4(ag, qa_p + k0 + 16);
                lm_mma(sc, af, bf[0], bf[1]);
                lm_mma(sd, ag, bf[2], bf[3]);
            }
            if (k0 < DK) {        // 16 entries left: the second half of the keys' fragment lies past them and is not used
                unsigned af[4], bf[4];
                lm_ldmatrix_x4(bf, kb_p + k0);
                lm_ldmatrix_x4(af, qa_p + k0);
                lm_mma(sc, af, bf[0], bf[1]);
            }
            const int c = warp * 8 + 2 * t4;
            s_s[g * (LM_KEYS + 1) + c] = (sc[0] + sd[0]) * a.scale;
            s_s[g * (LM_KEYS + 1) + c + 1] = (sc[1] + sd[1]) * a.scale;
            s_s[(g + 8) * (LM_KEYS + 1) + c] = (sc[2] + sd[2]) * a.scale;
            s_s[(g + 8) * (LM_KEYS + 1) + c + 1] = (sc[3] + sd[3]) * a.scale;
        } else
        {
            // two chains of sums (even and odd k-steps), so that a product does not wait for the one before it, and
            // the fragments of several k-steps in flight
            float sc[2][4] = {{0.f, 0.f, 0.f, 0.f}, {0.f, 0.f, 0.f, 0.f}};
            float sd[2][4] = {{0.f, 0.f, 0.f, 0.f}, {0.f, 0.f, 0.f, 0.f}};
            const __nv_bfloat16* qa_p = q_s + (lane & 15) * pitch + (lane >> 4) * 8;
            const __nv_bfloat16* kb_p = k_s + (warp * 16 + (lane & 7) + ((lane >> 4) << 3)) * pitch + ((lane >> 3) & 1) * 8;
            int k0 = 0;
#pragma unroll 2
            for (; k0 + 32 <= DK; k0 += 32) {
                unsigned af[4], bf[4], ag[4], bg[4];
                lm_ldmatrix_x4(af, qa_p + k0);
                lm_ldmatrix_x4(bf, kb_p + k0);
                lm_ldmatrix_x4(ag, qa_p + k0 + 16);
                lm_ldmatrix_x4(bg, kb_p + k0 + 16);
                lm_mma(sc[0], af, bf[0], bf[1]);
                lm_mma(sc[1], af, bf[2], bf[3]);
                lm_mma(sd[0], ag, bg[0], bg[1]);
                lm_mma(sd[1], ag, bg[2], bg[3]);
            }
            if (k0 < DK) {
                unsigned af[4], bf[4];
                lm_ldmatrix_x4(af, qa_p + k0);
                lm_ldmatrix_x4(bf, kb_p + k0);
                lm_mma(sc[0], af, bf[0], bf[1]);
                lm_mma(sc[1], af, bf[2], bf[3]);
            }
#pragma unroll
            for (int nt = 0; nt < 2; ++nt)
#pragma unroll
                for (int e = 0; e < 4; ++e) sc[nt][e] += sd[nt][e];
#pragma unroll
            for (int nt = 0; nt < 2; ++nt) {
                const int c = warp * 16 + nt * 8 + 2 * t4;
                s_s[g * (LM_KEYS + 1) + c] = sc[nt][0] * a.scale;
                s_s[g * (LM_KEYS + 1) + c + 1] = sc[nt][1] * a.scale;
                s_s[(g + 8) * (LM_KEYS + 1) + c] = sc[nt][2] * a.scale;
                s_s[(g + 8) * (LM_KEYS + 1) + c + 1] = sc[nt][3] * a.scale;
            }
        }
        __syncthreads();
        // ---- 2. softmax of this warp's rows --------------------------------------------------------------------
#pragma unroll
        for (int r = 0; r < RPW; ++r) {
            const int row = warp * RPW + r, pos = pos_s[row];
            const int j0 = pg * LM_KEYS + lane, j1 = j0 + 32;
            const bool see0 = pos >= 0 && j0 <= pos && pos - j0 < a.window;
            const bool see1 = pos >= 0 && j1 <= pos && pos - j1 < a.window;
            const float v0 = see0 ? s_s[row * (LM_KEYS + 1) + lane] : -INFINITY;
            const float v1 = see1 ? s_s[row * (LM_KEYS + 1) + lane + 32] : -INFINITY;
            const float m_new = fmaxf(mx[r], warp_max(fmaxf(v0, v1)));
            float p0 = 0.f, p1 = 0.f, corr = 1.f;
            if (m_new > -INFINITY) {
                p0 = see0 ? __expf(v0 - m_new) : 0.f;
                p1 = see1 ? __expf(v1 - m_new) : 0.f;
                corr = __expf(mx[r] - m_new);
            }
            mx[r] = m_new;
            sum[r] = sum[r] * corr + warp_sum(p0 + p1);
            p_s[row * (LM_KEYS + 8) + lane] = __float2bfloat16_rn(p0);
            p_s[row * (LM_KEYS + 8) + lane + 32] = __float2bfloat16_rn(p1);
            if (lane == 0) corr_s[row] = corr;
        }
        __syncthreads();
        // ---- 3. this warp's columns of the output ----------------------------------------------------------------
        {
            const float c_lo = corr_s[g], c_hi = corr_s[g + 8];
#pragma unroll
            for (int i = 0; i < NT; ++i) {
                acc[i][0] *= c_lo;
                acc[i][1] *= c_lo;
                acc[i][2] *= c_hi;
                acc[i][3] *= c_hi;
            }
            const __nv_bfloat16* pa_p = p_s + (lane & 15) * (LM_KEYS + 8) + (lane >> 4) * 8;
            // .trans: lanes 0-7 keys k0..k0+7 of columns n0.., 8-15 keys k0+8.., 16-23 and 24-31 the same of n0+8..
            const __nv_bfloat16* vb_p = k_s + ((lane & 7) + ((lane >> 3) & 1) * 8) * pitch + warp * cols_w + (lane >> 4) * 8;
#pragma unroll
            for (int k0 = 0; k0 < LM_KEYS; k0 += 16) {
                unsigned af[4];
                lm_ldmatrix_x4(af, pa_p + k0);
#pragma unroll
                for (int i = 0; i < NT; i += 2) {
                    if (i * 8 < cols_w) {
                        unsigned bf[4];
                        lm_ldmatrix_x4_trans(bf, vb_p + (size_t)k0 * pitch + i * 8);
                        lm_mma(acc[i], af, bf[0], bf[1]);
                        if (i + 1 < NT && (i + 1) * 8 < cols_w) lm_mma(acc[i + 1], af, bf[2], bf[3]);
                    }
                }
            }
        }
        __syncthreads();        // the page's rows and the weights are free again
    }
    // ---- the end: sums to shared memory, then every warp stores its columns ------------------------------------
    float* sum_s = corr_s + LM_ROWS;
    float* max_s = s_s;             // free by now
    if (lane == 0) {
#pragma unroll
        for (int r = 0; r < RPW; ++r) {
            sum_s[warp * RPW + r] = sum[r];
            max_s[warp * RPW + r] = mx[r];
        }
    }
    __syncthreads();
#pragma unroll
    for (int hh = 0; hh < 2; ++hh) {
        const int row = g + 8 * hh;
        if (pos_s[row] < 0) continue;
        const int t = t0 + row / hc, h = h0 + row % hc;
        const float l = sum_s[row];
        if (a.splits == 1) {
            const float inv = lm_finish(max_s[row], l, a.sinks, a.gate, a.ldg, t, h);
            __nv_bfloat16* o = a.out + ((size_t)t * a.H + h) * a.rank + warp * cols_w;
#pragma unroll
            for (int i = 0; i < NT; ++i) {
                const int c = i * 8 + 2 * t4;
                if (c < cols_w)
                    *reinterpret_cast<__nv_bfloat162*>(o + c) =
                        __floats2bfloat162_rn(acc[i][2 * hh] * inv, acc[i][2 * hh + 1] * inv);
            }
        } else {
            float* o = a.partial + (((size_t)t * a.H + h) * a.splits + slice) * (a.rank + 2);
            if (warp == 0 && t4 == 0) {
                o[0] = max_s[row];
                o[1] = l;
            }
#pragma unroll
            for (int i = 0; i < NT; ++i) {
                const int c = i * 8 + 2 * t4;
                if (c < cols_w) {
                    o[2 + warp * cols_w + c] = acc[i][2 * hh];
                    o[2 + warp * cols_w + c + 1] = acc[i][2 * hh + 1];
                }
            }
        }
    }
}

// ---- many tokens (prompts): 64 rows a block ------------------------------------------------------------------------
// The kernel above reads a page (74 KB for a rank of 512 and 64 rotated entries) for 16 rows, waits for it, and feeds every
// mma from two ldmatrix: 2,039 tokens of 16 heads took 720 us.  Here (439 us; the tensor pipe a quarter busy, bound by latencies with
// eight warps an SM) four
// neighbouring tiles share a page and the fragments: a warp's tile of the scores is 32 rows x 32 keys of the even or of
// the odd k-steps (the two chains of sums of the kernel above, so every bit of the result is the same), 8 mma for 4
// ldmatrix, and its tile of the values 64 rows x rank / 8 columns, 32 mma for 8.  Pages come as halves of 32 keys through
// a ring of three: the first half of the next page while this one is multiplied, its second half as soon as this
// page's first has been used.  One block an SM (230 KB), the latest tiles (the most keys) first.
// Tiles of several sequences in one block are done one sequence after the other.
#define LR_TILES 4
#define LR_ROWS (LR_TILES * LM_ROWS)
#define LR_HALF (LM_KEYS / 2)
template <int NT>       // rank = 64 NT
__global__ void __launch_bounds__(256, 1) latent_rows_kernel(const LatentMmaArgs a, int tiles) {
    pdl_sync();
    extern __shared__ __align__(16) unsigned char lm_smem[];
    const int DK = a.rank + a.rot, pitch = DK + 8;
    __nv_bfloat16* q_s = reinterpret_cast<__nv_bfloat16*>(lm_smem);                     // [64][pitch]
    __nv_bfloat16* k_s = q_s + LR_ROWS * pitch;                                          // [3][32][pitch]
    float* s_s = reinterpret_cast<float*>(k_s + 3 * LR_HALF * pitch);                    // [2][64][64 + 1]: even, odd k-steps
    __nv_bfloat16* p_s = reinterpret_cast<__nv_bfloat16*>(s_s + 2 * LR_ROWS * (LM_KEYS + 1));   // [64][64 + 8]
    float* corr_s = reinterpret_cast<float*>(p_s + LR_ROWS * (LM_KEYS + 8));             // [64]
    int* pos_s = reinterpret_cast<int*>(corr_s + LR_ROWS);                               // [64] positions, -1: no row
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, t4 = lane & 3;
    const int first = ((int)gridDim.x - 1 - (int)blockIdx.x) * LR_TILES, count = min(LR_TILES, tiles - first);
    const int hc = a.heads_per_block, h0 = blockIdx.y * hc;
    for (int i = 0; i < LR_TILES; ++i) {
        const bool there = i < count;       // rows of tiles that are not there: zeros
        const int t0 = there ? a.tile_t0[first + i] : 0, n = there ? min(a.tile_nq[first + i], a.tokens_per_block) : 0;
        lm_load_queries(a, q_s + i * LM_ROWS * pitch, pitch, t0, n, h0);
        if (threadIdx.x < LM_ROWS) {
            const int ti = threadIdx.x / hc, h = h0 + threadIdx.x % hc;
            pos_s[i * LM_ROWS + threadIdx.x] = (ti < n && h < a.H) ? a.tok_pos[t0 + ti] : -1;
        }
    }
    float acc[LR_TILES][NT][4];
#pragma unroll
    for (int m = 0; m < LR_TILES; ++m)
#pragma unroll
        for (int i = 0; i < NT; ++i) acc[m][i][0] = acc[m][i][1] = acc[m][i][2] = acc[m][i][3] = 0.f;
    float mx[8], sum[8];            // of rows 8 warp .. (the same in every lane)
#pragma unroll
    for (int r = 0; r < 8; ++r) {
        mx[r] = -INFINITY;
        sum[r] = 0.f;
    }
    const int chunks = DK / 8;
    const int wr = warp & 1, wk = (warp >> 1) & 1, odd = warp >> 2;     // rows, keys (a half) and k-steps of the scores
    __syncthreads();
    for (int s0 = 0; s0 < count;) {
        const int seq = a.tile_seq[first + s0];
        int s1 = s0 + 1;
        while (s1 < count && a.tile_seq[first + s1] == seq) ++s1;
        // pages of each tile (the others' are none), and of the tiles together
        int pg_lo[LR_TILES], pg_hi[LR_TILES], pg0 = 0, pg1 = -1;
#pragma unroll
        for (int i = 0; i < LR_TILES; ++i) {
            pg_lo[i] = 0;
            pg_hi[i] = -1;
            if (i >= s0 && i < s1) {
                const int t0 = a.tile_t0[first + i], n = min(a.tile_nq[first + i], a.tokens_per_block);
                pg_lo[i] = max(a.tok_pos[t0] - a.window + 1, 0) / LM_KEYS;
                pg_hi[i] = a.tok_pos[t0 + n - 1] / LM_KEYS;
                if (i == s0) pg0 = pg_lo[i];
                pg1 = pg_hi[i];
            }
        }
        const int* table = a.page_table + (size_t)seq * a.max_pages;
        const int halves = 2 * (pg1 - pg0 + 1);
        auto issue = [&](int half) {
            if (half < halves) {
                const __nv_bfloat16* src = a.cache + ((size_t)table[pg0 + (half >> 1)] * TB_PAGE + (half & 1) * LR_HALF) * DK;
                __nv_bfloat16* dst = k_s + (half % 3) * LR_HALF * pitch;
                const int kk = threadIdx.x >> 3;                // eight neighbouring threads a row
                for (int c8 = threadIdx.x & 7; c8 < chunks; c8 += 8)
                    lm_cp16(dst + kk * pitch + c8 * 8, src + (size_t)kk * DK + c8 * 8);
            }
            asm volatile("cp.async.commit_group;" ::: "memory");
        };
        issue(0);
        issue(1);
        for (int pg = pg0; pg <= pg1; ++pg) {
            const int half = 2 * (pg - pg0);
            issue(half + 2);
            asm volatile("cp.async.wait_group 1;" ::: "memory");
            __syncthreads();
            // ---- 1. scores
            {
                float sc[2][4][4];
#pragma unroll
                for (int m = 0; m < 2; ++m)
#pragma unroll
                    for (int n = 0; n < 4; ++n) sc[m][n][0] = sc[m][n][1] = sc[m][n][2] = sc[m][n][3] = 0.f;
                const __nv_bfloat16* qa_p = q_s + (wr * 32 + (lane & 15)) * pitch + (lane >> 4) * 8;
                const __nv_bfloat16* kb_p = k_s + ((half + wk) % 3 * LR_HALF + (lane & 7) + ((lane >> 4) << 3)) * pitch +
                                            ((lane >> 3) & 1) * 8;
#pragma unroll 2
                for (int k0 = odd * 16; k0 < DK; k0 += 32) {
                    unsigned af[2][4], bf[2][4];
                    lm_ldmatrix_x4(af[0], qa_p + k0);
                    lm_ldmatrix_x4(af[1], qa_p + 16 * pitch + k0);
                    lm_ldmatrix_x4(bf[0], kb_p + k0);
                    lm_ldmatrix_x4(bf[1], kb_p + 16 * pitch + k0);
#pragma unroll
                    for (int m = 0; m < 2; ++m)
#pragma unroll
                        for (int n = 0; n < 4; ++n) lm_mma(sc[m][n], af[m], bf[n >> 1][(n & 1) * 2], bf[n >> 1][(n & 1) * 2 + 1]);
                }
                float* to = s_s + odd * LR_ROWS * (LM_KEYS + 1) + (wr * 32 + g) * (LM_KEYS + 1) + wk * 32 + 2 * t4;
#pragma unroll
                for (int m = 0; m < 2; ++m)
#pragma unroll
                    for (int n = 0; n < 4; ++n)
#pragma unroll
                        for (int e = 0; e < 4; ++e)
                            to[(m * 16 + (e >> 1) * 8) * (LM_KEYS + 1) + n * 8 + (e & 1)] = sc[m][n][e];
            }
            __syncthreads();
            // ---- 2. softmax of this warp's rows, if their tile sees the page
            int lo = pg_lo[0], hi = pg_hi[0];
#pragma unroll
            for (int i = 1; i < LR_TILES; ++i)
                if (warp / 2 == i) {
                    lo = pg_lo[i];
                    hi = pg_hi[i];
                }
            if (pg >= lo && pg <= hi) {
                // the eight rows step by step side by side: their shuffles' latencies overlap
                float v0[8], v1[8], red[8];
                unsigned see0 = 0, see1 = 0;
                const int j0 = pg * LM_KEYS + lane, j1 = j0 + 32;
#pragma unroll
                for (int r = 0; r < 8; ++r) {
                    const int row = warp * 8 + r, pos = pos_s[row];
                    const bool s0r = pos >= 0 && j0 <= pos && pos - j0 < a.window;
                    const bool s1r = pos >= 0 && j1 <= pos && pos - j1 < a.window;
                    see0 |= s0r ? 1u << r : 0u;
                    see1 |= s1r ? 1u << r : 0u;
                    const float* sr = s_s + row * (LM_KEYS + 1) + lane;
                    const float* so = sr + LR_ROWS * (LM_KEYS + 1);
                    v0[r] = s0r ? __fmul_rn(sr[0] + so[0], a.scale) : -INFINITY;
                    v1[r] = s1r ? __fmul_rn(sr[32] + so[32], a.scale) : -INFINITY;
                    red[r] = fmaxf(v0[r], v1[r]);
                }
#pragma unroll
                for (int o = 16; o > 0; o >>= 1)
#pragma unroll
                    for (int r = 0; r < 8; ++r) red[r] = fmaxf(red[r], __shfl_xor_sync(0xffffffffu, red[r], o));
                float corr[8];
#pragma unroll
                for (int r = 0; r < 8; ++r) {
                    const float m_new = fmaxf(mx[r], red[r]);
                    float p0 = 0.f, p1 = 0.f;
                    corr[r] = 1.f;
                    if (m_new > -INFINITY) {
                        p0 = see0 >> r & 1 ? __expf(v0[r] - m_new) : 0.f;
                        p1 = see1 >> r & 1 ? __expf(v1[r] - m_new) : 0.f;
                        corr[r] = __expf(mx[r] - m_new);
                    }
                    mx[r] = m_new;
                    const int row = warp * 8 + r;
                    p_s[row * (LM_KEYS + 8) + lane] = __float2bfloat16_rn(p0);
                    p_s[row * (LM_KEYS + 8) + lane + 32] = __float2bfloat16_rn(p1);
                    if (lane == 0) corr_s[row] = corr[r];
                    red[r] = p0 + p1;
                }
#pragma unroll
                for (int o = 16; o > 0; o >>= 1)
#pragma unroll
                    for (int r = 0; r < 8; ++r) red[r] += __shfl_xor_sync(0xffffffffu, red[r], o);
#pragma unroll
                for (int r = 0; r < 8; ++r) sum[r] = sum[r] * corr[r] + red[r];
            }
            __syncthreads();
            // ---- 3. this warp's columns of the output; tiles that do not see the page are left alone
            const __nv_bfloat16* pa_p = p_s + (lane & 15) * (LM_KEYS + 8) + (lane >> 4) * 8;
            const int vb = ((lane & 7) + ((lane >> 3) & 1) * 8) * pitch + warp * (NT * 8) + (lane >> 4) * 8;
#pragma unroll
            for (int m = 0; m < LR_TILES; ++m) {
                if (pg < pg_lo[m] || pg > pg_hi[m]) continue;
                const float c_lo = corr_s[m * LM_ROWS + g], c_hi = corr_s[m * LM_ROWS + g + 8];
#pragma unroll
                for (int i = 0; i < NT; ++i) {
                    acc[m][i][0] *= c_lo;
                    acc[m][i][1] *= c_lo;
                    acc[m][i][2] *= c_hi;
                    acc[m][i][3] *= c_hi;
                }
            }
#pragma unroll
            for (int hf = 0; hf < 2; ++hf) {
                const __nv_bfloat16* v_p = k_s + (half + hf) % 3 * LR_HALF * pitch + vb;
#pragma unroll
                for (int k0 = 0; k0 < LR_HALF; k0 += 16) {
                    unsigned af[LR_TILES][4];
#pragma unroll
                    for (int m = 0; m < LR_TILES; ++m) lm_ldmatrix_x4(af[m], pa_p + m * LM_ROWS * (LM_KEYS + 8) + hf * LR_HALF + k0);
#pragma unroll
                    for (int i = 0; i < NT; i += 2) {
                        unsigned bf[4];
                        lm_ldmatrix_x4_trans(bf, v_p + k0 * pitch + i * 8);
#pragma unroll
                        for (int m = 0; m < LR_TILES; ++m) {
                            if (pg < pg_lo[m] || pg > pg_hi[m]) continue;
                            lm_mma(acc[m][i], af[m], bf[0], bf[1]);
                            lm_mma(acc[m][i + 1], af[m], bf[2], bf[3]);
                        }
                    }
                }
                __syncthreads();            // this half's rows (and behind the second, the weights) are free again
                if (hf == 0) issue(half + 3);
            }
        }
        asm volatile("cp.async.wait_group 0;" ::: "memory");
        s0 = s1;
    }
    // ---- the end: sums to shared memory, then every warp stores its columns
    float* max_s = s_s;
    float* sum_s = s_s + LR_ROWS;
    if (lane == 0) {
#pragma unroll
        for (int r = 0; r < 8; ++r) {
            max_s[warp * 8 + r] = mx[r];
            sum_s[warp * 8 + r] = sum[r];
        }
    }
    __syncthreads();
#pragma unroll
    for (int m = 0; m < LR_TILES; ++m)
#pragma unroll
        for (int hh = 0; hh < 2; ++hh) {
            const int in_tile = g + 8 * hh, row = m * LM_ROWS + in_tile;
            if (pos_s[row] < 0) continue;
            const int t = a.tile_t0[first + m] + in_tile / hc, h = h0 + in_tile % hc;
            const float inv = lm_finish(max_s[row], sum_s[row], a.sinks, a.gate, a.ldg, t, h);
            __nv_bfloat16* o = a.out + ((size_t)t * a.H + h) * a.rank + warp * (NT * 8);
#pragma unroll
            for (int i = 0; i < NT; ++i)
                *reinterpret_cast<__nv_bfloat162*>(o + i * 8 + 2 * t4) =
                    __floats2bfloat162_rn(acc[m][i][2 * hh] * inv, acc[m][i][2 * hh + 1] * inv);
        }
}

static size_t latent_rows_smem(int DK) {
    return (size_t)(LR_ROWS + 3 * LR_HALF) * (DK + 8) * 2 + 2 * LR_ROWS * (LM_KEYS + 1) * 4 + LR_ROWS * (LM_KEYS + 8) * 2 + LR_ROWS * 8;
}

template <int NT>
static int latent_rows_go(const LatentMmaArgs& a, int tiles, cudaStream_t s) {
    static PerDevice raised;
    tb_allow_smem(raised, (const void*)latent_rows_kernel<NT>, 227 * 1024);
    dim3 grid((tiles + LR_TILES - 1) / LR_TILES, (a.H + a.heads_per_block - 1) / a.heads_per_block);
    TB_LAUNCH((latent_rows_kernel<NT>), grid, 256, latent_rows_smem(a.rank + a.rot), s, a, tiles);
    return tb_last_error();
}

// out[t, h] = sum_s e^{m_s - m} O_s / sum_s e^{m_s - m} l_s        one block per (token, head): the slices' factors
// once, then every thread its columns with the loads of all slices in flight together
#define LM_MAX_SPLITS 16
__global__ void __launch_bounds__(128)
latent_merge_kernel(const float* __restrict__ partial, __nv_bfloat16* __restrict__ out, int splits, int rank,
                    const float* __restrict__ sinks, const __nv_bfloat16* __restrict__ gate, int ldg, int H) {
    pdl_sync();
    __shared__ float f_s[LM_MAX_SPLITS];
    const float* p = partial + (size_t)blockIdx.x * splits * (rank + 2);
    if (threadIdx.x < 32) {
        const int lane = threadIdx.x;
        const float ms = lane < splits ? p[(size_t)lane * (rank + 2)] : -INFINITY;
        const float ls = lane < splits ? p[(size_t)lane * (rank + 2) + 1] : 0.f;
        const float m = warp_max(ms);
        const float f = ms > -INFINITY ? __expf(ms - m) : 0.f;
        const float l = warp_sum(f * ls);
        const float fin = lm_finish(m, l, sinks, gate, ldg, blockIdx.x / H, blockIdx.x % H);
        if (lane < splits) f_s[lane] = f * fin;
    }
    __syncthreads();
    for (int c = threadIdx.x; c < rank; c += blockDim.x) {
        float v[LM_MAX_SPLITS];
#pragma unroll
        for (int s = 0; s < LM_MAX_SPLITS; ++s) v[s] = s < splits ? p[(size_t)s * (rank + 2) + 2 + c] : 0.f;
        float acc = 0.f;
#pragma unroll
        for (int s = 0; s < LM_MAX_SPLITS; ++s)
            if (s < splits) acc += f_s[s] * v[s];
        out[(size_t)blockIdx.x * rank + c] = __float2bfloat16_rn(acc);
    }
}

template <int NT, int W>
static int latent_mma_go(const LatentMmaArgs& a, int tiles, size_t smem, cudaStream_t s) {
    static bool raised = false;
    if (smem > 48 * 1024 && !raised) {
        tb_note_error(cudaFuncSetAttribute(latent_mma_kernel<NT, W>, cudaFuncAttributeMaxDynamicSharedMemorySize, 120 * 1024));
        raised = true;
    }
    dim3 grid(tiles, (a.H + a.heads_per_block - 1) / a.heads_per_block, a.splits);
    TB_LAUNCH((latent_mma_kernel<NT, W>), grid, W * 32, smem, s, a);
    return tb_last_error();
}

extern "C" {
// As tb_latent_attention_bf16, on the tensor cores.  splits > 1: the key range of every block is cut into that many
// slices, `partial` [nt, H, splits, rank + 2] floats receives them and a second kernel joins them.
// TB_ERR_UNSUPPORTED for sizes it does not take (nothing has been done then).
int tb_latent_attention_mma_bf16(const void* qa, const void* q, void* out, float* partial, const void* cache,
                                 const int* tile_seq, const int* tile_t0, const int* tile_nq, const int* tok_pos,
                                 const int* page_table, const float* cosT, const float* sinT, int tiles, int nt,
                                 int max_pages, int ldq, int q_head, int H, int rank, int rot, int rdims, int window,
                                 int splits, float scale, const float* sinks, const void* gate, int ldg,
                                 cudaStream_t s) {
    const int q_plain = q_head - rot;      // a head's queries: the plain entries, then the rotated ones
    if (tiles < 0 || nt < 0 || H <= 0 || rank <= 0 || rot < 0 || window <= 0 || rdims < 0 || rdims > rot || rdims % 2 ||
        splits < 1 || splits > LM_MAX_SPLITS || (splits > 1 && !partial))
        return TB_ERR_ARG;
    if (rank % 32 || rank > 512 || (rank + rot) % 16 || ((((uintptr_t)cache) | ((uintptr_t)qa)) & 15))
        return TB_ERR_UNSUPPORTED;
    if (tiles == 0) return 0;
    const int hc = H < LM_ROWS ? H : LM_ROWS;
    LatentMmaArgs a{(const __nv_bfloat16*)qa, (const __nv_bfloat16*)q, (__nv_bfloat16*)out, partial,
                    (const __nv_bfloat16*)cache, tile_seq, tile_t0, tile_nq, tok_pos, page_table, cosT, sinT, max_pages,
                    ldq, q_head, q_plain, H, rank, rot, rdims, window, hc, LM_ROWS / hc, splits, scale, sinks,
                    (const __nv_bfloat16*)gate, ldg};
    const int DK = rank + rot, pitch = DK + 8;
    const size_t smem = (size_t)(LM_ROWS + LM_KEYS) * pitch * 2 + LM_ROWS * (LM_KEYS + 1) * 4 + LM_ROWS * (LM_KEYS + 8) * 2 +
                        2 * LM_ROWS * 4 + LM_ROWS * 4;
    if (smem > 120 * 1024) return TB_ERR_UNSUPPORTED;
    int rc;
    if (rank % 64 == 0) {               // eight warps: rank / 8 columns of the output each
        const int nt8 = rank / 8 / 8;
        if (nt8 <= 2) rc = latent_mma_go<2, 8>(a, tiles, smem, s);
        else if (nt8 <= 4) rc = latent_mma_go<4, 8>(a, tiles, smem, s);
        else rc = latent_mma_go<8, 8>(a, tiles, smem, s);
    } else {
        const int nt8 = rank / 4 / 8;
        if (nt8 <= 2) rc = latent_mma_go<2, 4>(a, tiles, smem, s);
        else if (nt8 <= 4) rc = latent_mma_go<4, 4>(a, tiles, smem, s);
        else if (nt8 <= 8) rc = latent_mma_go<8, 4>(a, tiles, smem, s);
        else rc = latent_mma_go<16, 4>(a, tiles, smem, s);
    }
    if (rc || splits == 1) return rc;
    TB_LAUNCH((latent_merge_kernel), nt * H, 128, 0, s, (const float*)partial, (__nv_bfloat16*)out, splits, rank, sinks,
              (const __nv_bfloat16*)gate, ldg, H);
    return tb_last_error();
}
// The same without slices, 64 rows a block (latent_rows_kernel): the same bits, faster or slower by what the step brings (see
// parts/latent_attention.py).  TB_ERR_UNSUPPORTED for sizes it does not take.
int tb_latent_attention_rows_bf16(const void* qa, const void* q, void* out, const void* cache, const int* tile_seq,
                                  const int* tile_t0, const int* tile_nq, const int* tok_pos, const int* page_table,
                                  const float* cosT, const float* sinT, int tiles, int nt, int max_pages, int ldq, int q_head,
                                  int H, int rank, int rot, int rdims, int window, float scale, const float* sinks,
                                  const void* gate, int ldg, cudaStream_t s) {
    if (tiles < 0 || nt < 0 || H <= 0 || rank <= 0 || rot < 0 || window <= 0 || rdims < 0 || rdims > rot || rdims % 2)
        return TB_ERR_ARG;
    if ((rank != 256 && rank != 512) || (rank + rot) % 16 || latent_rows_smem(rank + rot) > 227 * 1024 ||
        ((((uintptr_t)cache) | ((uintptr_t)qa)) & 15))
        return TB_ERR_UNSUPPORTED;
    if (tiles == 0) return 0;
    const int hc = H < LM_ROWS ? H : LM_ROWS;
    const LatentMmaArgs a{(const __nv_bfloat16*)qa, (const __nv_bfloat16*)q, (__nv_bfloat16*)out, nullptr,
                          (const __nv_bfloat16*)cache, tile_seq, tile_t0, tile_nq, tok_pos, page_table, cosT, sinT, max_pages,
                          ldq, q_head, q_head - rot, H, rank, rot, rdims, window, hc, LM_ROWS / hc, 1, scale, sinks,
                          (const __nv_bfloat16*)gate, ldg};
    return rank == 512 ? latent_rows_go<8>(a, tiles, s) : latent_rows_go<4>(a, tiles, s);
}
}

#include "tape.h"
TB_TAPE_REGISTER(tb_latent_attention_mma_bf16)
TB_TAPE_REGISTER(tb_latent_attention_rows_bf16)

// Attention over the cached latents for prompts on the 5th-generation tensor cores (tcgen05), bfloat16 in, float accumulation in
// tensor memory.  The math and every rounding are those of latent_mma.cu, whose results it gives to the bit: scores in
// two chains of sums (even and odd k-steps of 16 entries), a running maximum that moves page by page, weights rounded to
// bfloat16 against it, the sum of a page's weights in the order of a warp's reduction.
//
// A block = 128 rows (token, head), neighbours in memory: 128 / H tokens of one sequence, with all their heads, x 256 columns
// of the output (a rank of 512 takes two blocks a tile, which both form the scores: tensor memory holds 128 x 256 sums and
// two pages' scores, no more).  Shared memory: the rows' queries (144 KB for 576 entries) and a ring of ten boxes of 64
// entries x 64 keys, 8 KB each, through which a page passes twice, as keys and as values.
//
//   warp 0    TMA: the queries' latent side, then the boxes in the order of their use: keys of page 0, keys of page 1,
//             values of page 0, keys of page 2, ...
//   warp 1    the scores of page j + 1 and then O += P V of page j; a box is free when its products have read it
//   warps 2-5 a thread a row: rotates its query's last entries into shared memory once; then, page by page, scores
//             from tensor memory, mask, maximum, weights (back into tensor memory, over the scores they came from), the sum, and
//             O times the factor by which the maximum moved, where it moved for any row of the warp
//
// One prompt of 2,039 tokens, 16 heads, rank 512 + 64: 212 us, 440 with 64 rows a block and mma.sync.  A page takes a block some 7,000
// clocks; the products' share is 2,300 (a k-step of the scores reads 6 KB of shared memory for 128 x 64 x 16, 48 clocks), the
// rest is the chain of the row's thread: scores out of tensor memory, 64 exponentials, 256 sums rescaled while the maximum still moves.
#include "latent_common.cuh"
#include "tc_common.cuh"

#define LT_ROWS 128
#define LT_KEYS TB_PAGE
#define LT_THREADS 192
#define LT_RING 10
#define LT_COLS 256                                  // output columns of a block
#define LT_BOX_BYTES (LT_KEYS * 128)
#define LT_QBOX_BYTES (LT_ROWS * 128)
#define LT_BARS (2 * LT_RING + 8)

struct LatentTcArgs {
    LatentMmaArgs l;          // tiles of tokens_per_block tokens; heads_per_block = H
    int* error;
    int tiles, cols;          // cols: blocks a tile (rank / LT_COLS)
    int wide;                 // the queries' rotated entries and the angles can be read 16 bytes at a time
};

__device__ __forceinline__ uint64_t lt_desc_v(uint32_t addr) {       // MN-major: rows of 64 entries (128 bytes, swizzled), 8 keys 1024 bytes apart
    uint64_t d = 0;
    d |= (uint64_t)((addr & 0x3FFFFu) >> 4);
    d |= (uint64_t)(LT_BOX_BYTES >> 4) << 16;
    d |= (uint64_t)(1024 >> 4) << 32;
    d |= (uint64_t)1 << 46;
    d |= (uint64_t)2 << 61;
    return d;
}
__device__ __forceinline__ void lt_ld32(uint32_t taddr, uint32_t (&r)[32]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
        "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
        "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
          "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]),
          "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]),
          "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
        : "r"(taddr)
        : "memory");
}
__device__ __forceinline__ void lt_st32(uint32_t taddr, const uint32_t (&v)[32]) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], "
        "{%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16, "
        "%17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31, %32};"
        ::"r"(taddr), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]), "r"(v[8]),
        "r"(v[9]), "r"(v[10]), "r"(v[11]), "r"(v[12]), "r"(v[13]), "r"(v[14]), "r"(v[15]), "r"(v[16]), "r"(v[17]),
        "r"(v[18]), "r"(v[19]), "r"(v[20]), "r"(v[21]), "r"(v[22]), "r"(v[23]), "r"(v[24]), "r"(v[25]), "r"(v[26]),
        "r"(v[27]), "r"(v[28]), "r"(v[29]), "r"(v[30]), "r"(v[31])
        : "memory");
}
__device__ __forceinline__ void lt_wait_ld() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void lt_wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }

__global__ void __launch_bounds__(LT_THREADS, 1) latent_tc_kernel(const __grid_constant__ CUtensorMap map_q,
                                                                 const __grid_constant__ CUtensorMap map_c,
                                                                 const LatentTcArgs g) {
    pdl_sync();
    const LatentMmaArgs& a = g.l;
    extern __shared__ __align__(1024) uint8_t smem_lt[];
    const uint32_t smem_base = smem_u32(smem_lt);
    const int DK = a.rank + a.rot, boxes = (DK + 63) / 64, steps = DK / 16;
    const uint32_t sq = smem_base, ring = sq + boxes * LT_QBOX_BYTES;
    uint64_t* bars = reinterpret_cast<uint64_t*>(smem_lt + boxes * LT_QBOX_BYTES + LT_RING * LT_BOX_BYTES);
    uint32_t& tmem_slot = *reinterpret_cast<uint32_t*>(bars + LT_BARS);
    // What is no number stays with the rows that see it: a key that a row does not see has the weight 0, and 0 times an infinite or NaN
    // value is NaN.  A key with such an entry has no finite score for any row, so a row that meets one at a masked place says so
    // (suspect, by the page's parity, = the page's number + 1; suspect[2]: any page), the products' warp makes those entries of the
    // page's values 0 before it multiplies them, and the epilogue adds them to the rows that do see them.
    volatile uint32_t* suspect = &tmem_slot + 1;
    const int warp = warp_number(), lane = threadIdx.x & 31;
    if (smem_base & 1023u) {                              // never expected; refuse rather than compute garbage
        if (threadIdx.x == 0) atomicCAS(g.error, 0, 41);
        return;
    }
    // the latest tiles, which see the most keys, first; a tile's blocks side by side
    const int tile = g.tiles - 1 - (int)blockIdx.x / g.cols, part = (int)blockIdx.x % g.cols;
    const int seq = a.tile_seq[tile], t0 = a.tile_t0[tile], n_tok = min(a.tile_nq[tile], a.tokens_per_block);
    const int p_first = a.tok_pos[t0], p_last = p_first + n_tok - 1;
    const int pg0 = max(p_first - a.window + 1, 0) / LT_KEYS, pages = p_last / LT_KEYS + 1 - pg0;
    const int* table = a.page_table + (size_t)seq * a.max_pages;

    const uint32_t bar0 = smem_u32(bars);
    auto full = [&](int s) { return bar0 + 8u * s; };
    auto empty = [&](int s) { return bar0 + 8u * (LT_RING + s); };
    const uint32_t q_full = bar0 + 8u * (2 * LT_RING), q_turned = q_full + 8;
    // two of each, by the page's parity (see attention_tc.cu)
    auto s_full = [&](int i) { return q_full + 16 + 8u * i; };
    auto p_ready = [&](int i) { return q_full + 32 + 8u * i; };
    auto o_done = [&](int i) { return q_full + 48 + 8u * i; };
    if (threadIdx.x == 0) {
        suspect[0] = suspect[1] = suspect[2] = 0;
        for (int s = 0; s < LT_RING; ++s) {
            mbar_init(full(s), 1);
            mbar_init(empty(s), 1);
        }
        mbar_init(q_full, 1);
        mbar_init(q_turned, 4);
        for (int i = 0; i < 2; ++i) {
            mbar_init(s_full(i), 1);
            mbar_init(p_ready(i), 4);
            mbar_init(o_done(i), 1);
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) tmem_alloc(smem_u32(&tmem_slot), 512);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    // a page that not every row of the block sees whole
    auto masked_page = [&](int key0) { return key0 + LT_KEYS - 1 > p_first || p_last - key0 >= a.window; };
    const uint32_t tmem_o = tmem_slot, tmem_s = tmem_slot + LT_COLS;      // page j: even sums at tmem_s + (j & 1) * 128, odd ones 64 further

    if (warp == 0) {
        // ---------------- TMA producer ----------------
        if (elect_one()) {
            const int q_boxes = a.rank / 64;
            mbar_expect_tx(q_full, q_boxes * LT_QBOX_BYTES);
            for (int b = 0; b < q_boxes; ++b) tma_load_2d(sq + b * LT_QBOX_BYTES, &map_q, q_full, b * 64, t0 * a.H);
        }
        __syncwarp();
        bool ok = true;
        int it = 0, slot = 0;
        uint32_t used = 1;                                // parity of the slot's last use
        auto box = [&](int x, int row) {
            if (it >= LT_RING) ok = mbar_wait_warp(empty(slot), used, g.error, 42);
            if (!ok) return;
            if (elect_one()) {
                mbar_expect_tx(full(slot), LT_BOX_BYTES);
                tma_load_2d(ring + slot * LT_BOX_BYTES, &map_c, full(slot), x, row);
            }
            __syncwarp();
            ++it;
            if (++slot == LT_RING) {
                slot = 0;
                used ^= 1;
            }
        };
        int row = 0, next_row = table[pg0] * LT_KEYS;
        for (int j = 0; j <= pages && ok; ++j) {          // keys of page j, then values of page j - 1
            const int before = row;
            row = next_row;
            if (j + 1 < pages) next_row = table[pg0 + j + 1] * LT_KEYS;
            if (j < pages)
                for (int b = 0; b < boxes && ok; ++b) box(b * 64, row);
            if (j > 0)
                for (int b = 0; b < LT_COLS / 64 && ok; ++b) box(part * LT_COLS + b * 64, before);
        }
        if (*(volatile int*)g.error != 0) {
            mbar_wait(q_full, 0, g.error, 43);
            for (int i = max(0, it - LT_RING); i < it; ++i) mbar_wait(full(i % LT_RING), (i / LT_RING) & 1, g.error, 43);
        }
    } else if (warp == 1) {
        // ---------------- MMA issuer ----------------
        const uint32_t idesc_s = umma_idesc(LT_ROWS, LT_KEYS), idesc_o = umma_idesc(LT_ROWS, 64) | (1u << 16);
        int slot = 0;
        uint32_t use = 0;
        bool ok = mbar_wait_warp(q_full, 0, g.error, 44) && mbar_wait_warp(q_turned, 0, g.error, 44);
        auto arrived = [&]() {
            ok = mbar_wait_warp(full(slot), use, g.error, 44);
            tc_fence_after();
            return ok;
        };
        auto next = [&]() {
            __syncwarp();
            if (++slot == LT_RING) {
                slot = 0;
                use ^= 1;
            }
        };
        auto scores = [&](int j) {
            for (int b = 0; b < boxes; ++b) {
                if (!arrived()) return;
                if (elect_one()) {
                    const uint64_t dq = umma_desc(sq + b * LT_QBOX_BYTES), dk = umma_desc(ring + slot * LT_BOX_BYTES);
                    const int n = min(4, steps - 4 * b);
#pragma unroll
                    for (int k = 0; k < 4; ++k)           // an even number of steps a box: k says which chain
                        if (k < n) umma_bf16(tmem_s + (j & 1) * 128 + (k & 1) * 64, dq + 2 * k, dk + 2 * k, idesc_s, (b | (k >> 1)) != 0);
                    umma_commit(empty(slot));
                    if (b == boxes - 1) umma_commit(s_full(j & 1));
                }
                next();
            }
        };
        if (ok) scores(0);
        for (int j = 0; j < pages && ok; ++j) {
            if (j + 1 < pages) scores(j + 1);             // while the softmax warps work on page j
            if (!ok) break;
            ok = mbar_wait_warp(p_ready(j & 1), (j >> 1) & 1, g.error, 45);
            if (!ok) break;
            tc_fence_after();
            const bool look = suspect[j & 1] == (uint32_t)j + 1;
            for (int b = 0; b < LT_COLS / 64; ++b) {
                if (!arrived()) break;
                if (look) {
                    uint32_t* box = reinterpret_cast<uint32_t*>(smem_lt + (ring - smem_base) + slot * LT_BOX_BYTES);
                    for (int i = lane; i < LT_BOX_BYTES / 4; i += 32)
                        if (not_finite_pair(box[i]) & 0x80008000u) box[i] = finite_pair(box[i]);
                    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");     // the product reads these writes
                    __syncwarp();
                }
                if (elect_one()) {
#pragma unroll
                    for (int k = 0; k < LT_KEYS / 16; ++k)
                        umma_bf16_ts(tmem_o + b * 64, tmem_s + (j & 1) * 128 + 8 * k, lt_desc_v(ring + slot * LT_BOX_BYTES + k * 2048),
                                     idesc_o, (j | k) != 0);
                    umma_commit(empty(slot));
                    if (b == LT_COLS / 64 - 1) umma_commit(o_done(j & 1));
                }
                next();
            }
        }
    } else {
        // ---------------- softmax / correction / epilogue: thread = row ----------------
        const int quad = warp & 3, row = quad * 32 + lane;
        const uint32_t lane_sel = (uint32_t)(quad * 32) << 16;
        const int ti = row / a.H, h = row - ti * a.H;
        const bool live = ti < n_tok;
        const int t = t0 + ti, pos = live ? p_first + ti : -1;
        // the rotated entries behind the latent's: 16-byte pieces of the last box's rows, swizzled by the row
        {
            uint8_t* qr = smem_lt + (boxes - 1) * LT_QBOX_BYTES + row * 128;
            const __nv_bfloat16* src = a.q + (size_t)t * a.ldq + (size_t)h * a.q_head + a.q_plain;
            auto piece = [&](int c) { return reinterpret_cast<__nv_bfloat16*>(qr + (((c >> 3) ^ (row & 7)) << 4)); };
            const int half = a.rdims / 2;
            if (g.wide) {       // eight pairs (c, c + half) at a time
                const float *co = a.cosT + (size_t)max(pos, 0) * half, *si = a.sinT + (size_t)max(pos, 0) * half;
                for (int c = 0; c < half; c += 8) {
                    float x0[8] = {}, x1[8] = {}, y0[8], y1[8], cs[8], sn[8];
                    if (live) {
                        load8(src + c, x0);
                        load8(src + c + half, x1);
                    }
                    load8(co + c, cs);
                    load8(si + c, sn);
#pragma unroll
                    for (int e = 0; e < 8; ++e) {
                        y0[e] = lm_turn_low(x0[e], x1[e], cs[e], sn[e]);
                        y1[e] = lm_turn_high(x0[e], x1[e], cs[e], sn[e]);
                    }
                    store8(piece(c), y0);
                    store8(piece(c + half), y1);
                }
            }
            for (int c = g.wide ? a.rdims : 0; c < a.rot; c += 8) {
                float f[8];
#pragma unroll
                for (int e = 0; e < 8; ++e) f[e] = live ? lm_turned(a, src, c + e, pos) : 0.f;
                store8(piece(c), f);
            }
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");     // the products read these writes
            __syncwarp();
            if (lane == 0) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(q_turned) : "memory");
        }
        float mx = -INFINITY, sum = 0.f;
        bool ok = true;
        for (int j = 0; j < pages && ok; ++j) {
            ok = mbar_wait_warp(s_full(j & 1), (j >> 1) & 1, g.error, 46);
            tc_fence_after();
            if (!ok) break;
            const uint32_t ts = tmem_s + (j & 1) * 128 + lane_sel;
            float v[LT_KEYS];
#pragma unroll
            for (int half = 0; half < 2; ++half) {
                uint32_t e[32], o[32];
                lt_ld32(ts + half * 32, e);
                lt_ld32(ts + 64 + half * 32, o);
                lt_wait_ld();
#pragma unroll
                for (int i = 0; i < 32; ++i) v[half * 32 + i] = __fmul_rn(__uint_as_float(e[i]) + __uint_as_float(o[i]), a.scale);
            }
            const int key0 = (pg0 + j) * LT_KEYS;
            const bool masked = masked_page(key0);
            if (masked || !live) {
                bool odd = false;
#pragma unroll
                for (int i = 0; i < LT_KEYS; ++i)
                    if (key0 + i > pos || pos - (key0 + i) >= a.window) {
                        odd |= !(fabsf(v[i]) < INFINITY);
                        v[i] = -INFINITY;
                    }
                if (masked && odd) suspect[j & 1] = suspect[2] = j + 1;
            }
            float top = -INFINITY;
#pragma unroll
            for (int i = 0; i < LT_KEYS; i += 2) asm("max.f32 %0, %0, %1, %2;" : "+f"(top) : "f"(v[i]), "f"(v[i + 1]));
            const float m_new = fmaxf(mx, top);
            const float ref = m_new > -INFINITY ? m_new : 0.f;
            const float corr = m_new > -INFINITY ? __expf(mx - m_new) : 1.f;
            mx = m_new;
            uint32_t pk[32];
#pragma unroll
            for (int i = 0; i < LT_KEYS; ++i) v[i] = __expf(v[i] - ref);
#pragma unroll
            for (int i = 0; i < LT_KEYS; i += 2) {
                const __nv_bfloat162 p2 = __floats2bfloat162_rn(v[i], v[i + 1]);
                pk[i / 2] = *reinterpret_cast<const uint32_t*>(&p2);
            }
            // the sum in the order of a warp that holds keys i and i + 32 in lane i
#pragma unroll
            for (int o = 32; o > 0; o >>= 1)
#pragma unroll
                for (int i = 0; i < o; ++i) v[i] += v[i + o];
            sum = sum * corr + v[0];
            const bool move = j > 0 && __any_sync(0xffffffffu, corr != 1.f);
            if (move) {         // O is touched once the previous page's product is done
                ok = mbar_wait_warp(o_done((j - 1) & 1), ((j - 1) >> 1) & 1, g.error, 47);
                tc_fence_after();
                if (!ok) break;
#pragma unroll
                for (int c = 0; c < LT_COLS; c += 64) {
                    uint32_t x[32], y[32];
                    lt_ld32(tmem_o + lane_sel + c, x);
                    lt_ld32(tmem_o + lane_sel + c + 32, y);
                    lt_wait_ld();
#pragma unroll
                    for (int i = 0; i < 32; ++i) {
                        x[i] = __float_as_uint(__uint_as_float(x[i]) * corr);
                        y[i] = __float_as_uint(__uint_as_float(y[i]) * corr);
                    }
                    lt_st32(tmem_o + lane_sel + c, x);
                    lt_st32(tmem_o + lane_sel + c + 32, y);
                }
            }
            lt_st32(ts, pk);
            lt_wait_st();
            tc_fence_before();
            __syncwarp();
            if (lane == 0) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(p_ready(j & 1)) : "memory");
            // keep in step with the products, phase by phase
            if (j > 0 && !move) {
                ok = mbar_wait_warp(o_done((j - 1) & 1), ((j - 1) >> 1) & 1, g.error, 47);
                tc_fence_after();
            }
        }
        if (ok) {
            ok = mbar_wait_warp(o_done((pages - 1) & 1), ((pages - 1) >> 1) & 1, g.error, 48);
            tc_fence_after();
        }
        asm volatile("bar.sync 1, 128;" ::: "memory");      // suspect[2], as any of the four warps left it
        if (ok) {
            const float inv = live ? lm_finish(mx, sum, a.sinks, a.gate, a.ldg, t, h) : 0.f;
            __nv_bfloat16* out = a.out + ((size_t)t * a.H + h) * a.rank + part * LT_COLS;
#pragma unroll
            for (int c = 0; c < LT_COLS; c += 32) {
                uint32_t x[32];
                lt_ld32(tmem_o + lane_sel + c, x);        // warp-collective: rows without a query store nothing
                lt_wait_ld();
                if (live && suspect[2]) {
                    for (int j = 0; j < pages; ++j) {
                        const int key0 = (pg0 + j) * LT_KEYS;
                        if (!masked_page(key0)) continue;
                        const __nv_bfloat16* page = a.cache + (size_t)table[pg0 + j] * LT_KEYS * DK + part * LT_COLS + c;
                        for (int k = max(0, pos - a.window + 1 - key0); k < LT_KEYS && key0 + k <= pos; ++k)
#pragma unroll
                            for (int i = 0; i < 32; ++i) {
                                const float y = __bfloat162float(page[(size_t)k * DK + i]);
                                if (!(fabsf(y) < INFINITY)) x[i] = __float_as_uint(__uint_as_float(x[i]) + y);
                            }
                    }
                }
                if (live) {
#pragma unroll
                    for (int i = 0; i < 32; i += 8) {
                        float f[8];
#pragma unroll
                        for (int e = 0; e < 8; ++e) f[e] = __uint_as_float(x[i + e]) * inv;
                        store8(out + c + i, f);
                    }
                }
            }
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 1) tmem_dealloc(tmem_slot, 512);
}

extern "C" {
// Query tokens a tile of this kernel takes, for a mixer of H heads with such a cache; 0 where it takes none.
int tb_latent_tc_tile_tokens(int H, int rank, int rot) {
    return H >= 1 && H <= LT_ROWS && (rank == 256 || rank == 512) && rot >= 0 && rot <= 64 && rot % 32 == 0 ? LT_ROWS / H : 0;
}
// As tb_latent_attention_rows_bf16 (the same bits), tiles of tb_latent_tc_tile_tokens tokens.  TB_ERR_UNSUPPORTED for sizes it does
// not take.
int tb_latent_attention_tc_bf16(const void* qa, const void* q, void* out, const void* cache, const int* tile_seq,
                                const int* tile_t0, const int* tile_nq, const int* tok_pos, const int* page_table,
                                const float* cosT, const float* sinT, int tiles, int nt, int max_pages, int ldq, int q_head,
                                int H, int rank, int rot, int rdims, int cache_pages, int window, float scale, const float* sinks,
                                const void* gate, int ldg, cudaStream_t s) {
    if (tiles < 0 || nt < 0 || H <= 0 || rank <= 0 || rot < 0 || window <= 0 || rdims < 0 || rdims > rot || rdims % 2 || cache_pages <= 0)
        return TB_ERR_ARG;
    const int tokens = tb_latent_tc_tile_tokens(H, rank, rot);
    const long long rows = (long long)cache_pages * TB_PAGE;
    if (!tokens || rows > 0x7fffffffLL || (long long)nt * H > 0x7fffffffLL || ((((uintptr_t)cache) | ((uintptr_t)qa) | ((uintptr_t)out)) & 15))
        return TB_ERR_UNSUPPORTED;
    if (tiles == 0) return 0;
    const int DK = rank + rot;
    CUtensorMap mq, mc;
    int rc = make_map(&mq, qa, (long long)nt * H, rank, rank, LT_ROWS);
    if (!rc) rc = make_map(&mc, cache, rows, DK, DK, LT_KEYS);
    if (rc) return rc;
    int* err = tc_error_ptr();
    if (!err) return tb_last_error();
    LatentTcArgs g{{(const __nv_bfloat16*)qa, (const __nv_bfloat16*)q, (__nv_bfloat16*)out, nullptr, (const __nv_bfloat16*)cache,
                    tile_seq, tile_t0, tile_nq, tok_pos, page_table, cosT, sinT, max_pages, ldq, q_head, q_head - rot, H, rank, rot,
                    rdims, window, H, tokens, 1, scale, sinks, (const __nv_bfloat16*)gate, ldg},
                   err, tiles, rank / LT_COLS,
                   rdims % 16 == 0 && ldq % 8 == 0 && q_head % 8 == 0 && (q_head - rot) % 8 == 0 &&
                       !(((uintptr_t)q | (uintptr_t)cosT | (uintptr_t)sinT) & 15)};
    const size_t smem = (size_t)((DK + 63) / 64) * LT_QBOX_BYTES + LT_RING * LT_BOX_BYTES + (LT_BARS + 2) * 8;
    static PerDevice raised;
    tb_allow_smem(raised, (const void*)latent_tc_kernel, 227 * 1024);
    TB_LAUNCH((latent_tc_kernel), tiles * g.cols, LT_THREADS, smem, s, mq, mc, g);
    return tb_last_error();
}
}

#include "tape.h"
TB_TAPE_REGISTER(tb_latent_attention_tc_bf16)

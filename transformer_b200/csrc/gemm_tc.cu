// Matrix products for prompts on the 5th-generation tensor cores (tcgen05), bfloat16 in, float
// accumulation in tensor memory:   C[m, :] = A[m, :] . B[g(m)]^T
//
//   Two forms of one kernel (template parameter CTAS):
//   * CTAS = 1: a block works on a tile of 128 rows x 256 columns (tcgen05.mma.cta_group::1, M = 128, N = 256);
//   * CTAS = 2: two blocks (a cluster of two CTAs, cta_group::2) work on one tile of 256 rows x 256 columns:
//     each holds its own 128 rows of A and HALF of the B tile (128 of the 256 rows of B) in shared memory, and
//     one tcgen05.mma issued by the leader reads both blocks' operands and writes rows 0..127 of the product
//     into the leader's tensor memory and rows 128..255 into the other's.  Per block and k-block that is 32 KB
//     from L2 for 128 x 256 x 64 of product instead of 48 KB, and six ring stages fit instead of four.
//     With few rows per group the 256-row tiles are mostly padding and there are half as many work items (decoding at
//     batch 64: -7 %); the launcher goes by the rounds either form takes (see gemm_tc_entry, with the measurements);
//   * operands are staged by TMA (cp.async.bulk.tensor, 128-byte swizzle) into a ring of TC_STAGES stages;
//     with pairs, both blocks' copies are counted on the LEADER's barrier of the stage;
//   * tcgen05.commit (with pairs: multicast to both blocks) hands a finished stage back to the TMA warps and, after
//     the last k-block, the accumulator [128 x 256] float (256 TMEM columns, two of them: the next tile's
//     products overlap this tile's epilogue) to both blocks' four epilogue warps, which read it with
//     tcgen05.ld, apply the epilogue in float and store; they hand it back by an arrival on the leader's
//     barrier.  A lane reads one ROW of the accumulator; bfloat16 results therefore pass through a strip of
//     shared memory per warp and leave as whole 128-byte lines (the product with the short K, the experts'
//     down projection, was bound by its row-by-row stores: 68.6 -> 60.4 us at 16 x 512 rows, 0.88 -> 1.15
//     PFLOP/s at 16 x 2,048);
//   Warp roles: 0 = TMA producer, 1 = TMEM allocation (+ MMA issue in the leader), 2..9 = epilogue: a warp reads the
//   32 lanes of tensor memory its number allows (warp % 4), so two warps share each quarter of the rows and take
//   alternate 64-column pieces.  (With four epilogue warps the product with the short K, 11 k-blocks a tile, was bound
//   by its epilogue: the accumulator of a tile took as long to store as the next tile's products to compute.)
//
//   * grouped (the experts, models/llama/common/src/compute.rs:319-330 done as one product per
//     expert over all of its tokens): rows of A are sorted by group; B is the stack of the groups'
//     matrices viewed as one [G * rows, K] tensor; a pair finds its (group, first row) from
//     group_offsets.  Rows of the tile that belong to the next group are computed and not stored.
//   * DUAL (swiglu, compute.rs:324-326): the B tile is 128 gate rows (the leader's half) followed by the
//     128 matching up rows (the other block's), so one N = 256 instruction yields both; the epilogue stores
//     silu(gate) * up.
//   * edges: TMA fills out-of-range rows and the K tail with zeros; stores are predicated.
//
// Every wait on an mbarrier is bounded; a wait that runs out sets *error (nonzero), the block
// stops issuing work, the leader waits (bounded) for the pair's copies in flight, both blocks meet at the
// cluster barrier, free their TMEM and return.
#include <map>
#include <mutex>
#include <tuple>

#include "tc_common.cuh"

#define TC_BM 128                                  // rows of a tile per block; a pair covers 2 * TC_BM
#define TC_BN 256
#define TC_BK 64
#define TC_THREADS 320
#define TC_EPI_WARPS 8                             // two per quarter of the tensor memory's lanes
#define TC_SHARED_GROUPS 256                       // up to this many groups their offsets are kept in shared memory
#define TC_MAX_STAGES 6
#define TC_A_BYTES (TC_BM * TC_BK * 2)
#define TC_BHALF_BYTES (TC_BN / 2 * TC_BK * 2)     // half of the B tile: all that a block of a pair stages
#define TC_EPI_BF16 0                              // bfloat16, the (gate, up) pair among it
#define TC_EPI_BIASED 1                            // the pair with biases
#define TC_EPI_FLOAT 2
#define TC_STRIP_BYTES (32 * 128)                  // an epilogue warp's strip: 32 rows x 64 bfloat16, on their way out

template <int CTAS> struct TcShape {
    static constexpr int STAGES = CTAS == 2 ? 6 : 4;
    static constexpr int STAGE_BYTES = TC_A_BYTES + (CTAS == 2 ? 1 : 2) * TC_BHALF_BYTES;
    static constexpr int ROWS = CTAS * TC_BM;      // rows of a tile
};

struct TcArgs {
    void* C;
    const int* group_offsets;
    int* error;
    int ldc, M, N, K, G;
    int b_group_rows;   // rows of B per group in the stacked view (N, or 2N when dual)
    int dual;
    int tiles_m;        // row tiles (with groups: an upper bound; tiles past the last group are skipped)
    int n_tile;         // rows of B in a tile: a multiple of 16 up to TC_BN (fewer when that fills the SMs better)
    GluRule glu;        // dual: how the (gate, up) pair becomes one value
};

// ---- the kernel ----------------------------------------------------------------------------
// Persistent: a block (or pair) walks the tiles  unit, unit + units, ...  in the order tc_tile gives them (one
// matrix: column tiles of one row tile are neighbours, so concurrent units share its A tile in L2; groups: see
// there).  The TMA ring runs on across tile boundaries.
struct TcTile {
    int g, row0, row_end, n0;
    bool valid;
};

// `offsets`: the groups' row offsets, in shared memory when there are few enough groups (every role of the block
// walks them for every tile: from global memory that is a chain of dependent loads, some 10 us for the last of 16
// groups, on the way to the block's first copy).
__device__ __forceinline__ TcTile tc_tile(const TcArgs& a, const int* offsets, int t, int tiles_n, int n_out, int rows) {
    TcTile r;
    if (!offsets) {
        const int tm = t / tiles_n;
        r.n0 = (t - tm * tiles_n) * n_out;
        r.g = 0;
        r.row0 = tm * rows;
        r.row_end = a.M;
        r.valid = r.row0 < a.M;
        return r;
    }
    // Groups: the tiles of a group are numbered column tile by column tile, the group's row tiles innermost.  Blocks
    // that run at the same time take consecutive numbers, so the few row tiles of a group that need the SAME tile
    // of its weights fetch it together (once from memory, the others from L2), and what they do not share, the
    // group's rows of A, is a few megabytes that stay in L2.  With the row tiles outermost every weight came from
    // memory once per row tile whenever a group's weights exceed L2 (experts 14,336 wide: 235 MB per group,
    // four row tiles: four times the traffic, and the product was bound by it).
    r.valid = false;
    r.g = 0;
    r.row0 = r.row_end = r.n0 = 0;
    int cum = 0;
    for (int g = 0; g < a.G; ++g) {
        const int lo = offsets[g], hi = offsets[g + 1];
        const int tiles_r = (hi - lo + rows - 1) / rows;
        const int n = tiles_r * tiles_n;
        if (t < cum + n) {
            const int local = t - cum;
            const int tn = local / tiles_r, tr = local - tn * tiles_r;
            r.g = g;
            r.row0 = lo + tr * rows;
            r.row_end = hi;
            r.n0 = tn * n_out;
            r.valid = true;
            break;
        }
        cum += n;
    }
    return r;
}

// EPI: what the epilogue makes of the accumulator (TC_EPI_*).  Kernels of their own: with all of it in one the products that stream
// weights for a few rows took 2 to 6 % longer (256 rows of 16 experts, (gate, up) of 688 x 4,096: 51.2 and 54.3 us).
template <int CTAS, int EPI>
__global__ void __launch_bounds__(TC_THREADS) gemm_tc_kernel(const __grid_constant__ CUtensorMap map_a,
                                                            const __grid_constant__ CUtensorMap map_b,
                                                            const TcArgs a) {
    pdl_sync();
    extern __shared__ uint8_t smem_raw[];
    constexpr int TC_STAGES = TcShape<CTAS>::STAGES, TC_STAGE_BYTES = TcShape<CTAS>::STAGE_BYTES;
    constexpr bool PAIR = CTAS == 2, BIASED = EPI == TC_EPI_BIASED, FLOAT = EPI == TC_EPI_FLOAT;
    __shared__ __align__(8) uint64_t bars[2 * TC_MAX_STAGES + 4];
    __shared__ uint32_t tmem_slot;
    __shared__ int group_rows[TC_SHARED_GROUPS + 1];
    const int* offsets = a.group_offsets;
    if (a.group_offsets && a.G <= TC_SHARED_GROUPS) {
        for (int i = threadIdx.x; i <= a.G; i += TC_THREADS) group_rows[i] = a.group_offsets[i];
        offsets = group_rows;        // visible to all after the block-wide barrier below
    }
    const uint32_t smem_base = (smem_u32(smem_raw) + 1023u) & ~1023u;
    const int warp = PAIR ? warp_number() : (int)(threadIdx.x >> 5), lane = threadIdx.x & 31;
    const uint32_t rank = PAIR ? cluster_ctarank() : 0;  // 0 leads the pair
    const int pair = blockIdx.x / CTAS, pairs = gridDim.x / CTAS;     // this unit of work and how many there are
    const int n_out = a.dual ? a.n_tile / 2 : a.n_tile; // output columns of a tile
    const int tiles_n = (a.N + n_out - 1) / n_out;
    const uint32_t half_bytes = (uint32_t)(a.n_tile / 2) * TC_BK * 2;      // half of the B tile in shared memory
    const uint32_t stage_tx = TC_A_BYTES + (PAIR ? 1 : 2) * half_bytes;    // bytes one block copies per stage
    const int total = a.tiles_m * tiles_n;
    const int nkb = (a.K + TC_BK - 1) / TC_BK;

    const uint32_t bar0 = smem_u32(bars);
    auto full_bar = [&](int s) { return bar0 + 8u * s; };
    auto empty_bar = [&](int s) { return bar0 + 8u * (TC_MAX_STAGES + s); };
    auto acc_full = [&](int i) { return bar0 + 8u * (2 * TC_MAX_STAGES + i); };
    auto acc_empty = [&](int i) { return bar0 + 8u * (2 * TC_MAX_STAGES + 2 + i); };

    if (threadIdx.x == 0) {
        for (int s = 0; s < TC_STAGES; ++s) {
            mbar_init(full_bar(s), 1);        // the leader's: its producer arms it with both blocks' bytes
            mbar_init(empty_bar(s), 1);       // one multicast commit per use
        }
        for (int i = 0; i < 2; ++i) {
            mbar_init(acc_full(i), 1);
            mbar_init(acc_empty(i), TC_EPI_WARPS * CTAS);    // the leader's: one arrival per epilogue warp of every block
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) {
        if (PAIR) tmem_alloc_pair(smem_u32(&tmem_slot), 2 * TC_BN);
        else tmem_alloc(smem_u32(&tmem_slot), 2 * TC_BN);
    }
    tc_fence_before();
    if (PAIR) cluster_sync_all();             // both blocks' barriers exist before either signals the other's
    else __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = tmem_slot;

    // Pairs: these two loops are the whole warp's, and one elected lane issues (see elect_one).  As one thread's loops they cost the down
    // product of 16 experts at 2,048 rows each 163 us for 156; single blocks are 1 to 2 % faster with a thread's loops.
    auto agreed = [&](bool ok) { return PAIR ? (bool)__all_sync(0xffffffffu, ok) : ok; };
    if (warp == 0) {
        // ---------------- TMA producer (both blocks; bytes are counted on the leader's barrier) ----------------
        if (PAIR || lane == 0) {
            bool ok = true;
            int it = 0;                       // k-blocks handed to the ring so far, over all tiles
            int s = 0;                        // its stage, and the parity of the stage's last use:
            uint32_t used = 1;                // kept as counters, since this one thread paces the whole block
            for (int t = pair; t < total && ok; t += pairs) {
                const TcTile tl = tc_tile(a, offsets, t, tiles_n, n_out, TcShape<CTAS>::ROWS);
                if (!tl.valid) continue;
                const int a_row = tl.row0 + (int)rank * TC_BM;
                const int b_row = tl.g * a.b_group_rows + tl.n0 + (int)rank * (a.dual ? a.N : a.n_tile / 2);
                for (int kb = 0; kb < nkb && ok; ++kb, ++it) {
                    if (it >= TC_STAGES) ok = agreed(mbar_wait(empty_bar(s), used, a.error, 1));
                    if (!ok) break;
                    const uint32_t sa = smem_base + s * TC_STAGE_BYTES, sb = sa + TC_A_BYTES;
                    if (PAIR) {
                        const uint32_t counted = mapa_shared(full_bar(s), 0);
                        if (elect_one()) {
                            if (rank == 0) mbar_expect_tx(full_bar(s), CTAS * stage_tx);
                            tma_load_2d_pair(sa, &map_a, counted, kb * TC_BK, a_row);
                            tma_load_2d_pair(sb, &map_b, counted, kb * TC_BK, b_row);
                        }
                    } else {
                        mbar_expect_tx(full_bar(s), CTAS * stage_tx);
                        tma_load_2d(sa, &map_a, full_bar(s), kb * TC_BK, a_row);
                        tma_load_2d(sb, &map_b, full_bar(s), kb * TC_BK, b_row);
                        tma_load_2d(sb + half_bytes, &map_b, full_bar(s), kb * TC_BK,
                                    b_row + (a.dual ? a.N : a.n_tile / 2));
                    }
                    if (++s == TC_STAGES) {
                        s = 0;
                        used ^= 1;
                    }
                }
            }
            if (rank == 0 && *(volatile int*)a.error != 0) {
                // something gave up: let the pair's copies land before the blocks go away
                for (int i = max(0, it - TC_STAGES); i < it; ++i)
                    mbar_wait(full_bar(i % TC_STAGES), (i / TC_STAGES) & 1, a.error, 4);
            }
        }
    } else if (warp == 1) {
        // ---------------- MMA issuer: one thread, or of a pair the leader's warp for both blocks ----------------
        if ((PAIR || lane == 0) && rank == 0) {
            const uint32_t idesc = umma_idesc(TcShape<CTAS>::ROWS, a.n_tile);
            bool ok = true;
            int lt = 0;                       // tiles done by this unit
            int s = 0;                        // the stage of the next k-block and the parity of its use
            uint32_t use = 0;
            for (int t = pair; t < total && ok; t += pairs) {
                const TcTile tl = tc_tile(a, offsets, t, tiles_n, n_out, TcShape<CTAS>::ROWS);
                if (!tl.valid) continue;
                const int buf = lt & 1;
                if (lt >= 2) ok = agreed(mbar_wait(acc_empty(buf), ((lt >> 1) - 1) & 1, a.error, 5));   // drained two tiles ago
                if (!ok) break;
                tc_fence_after();
                const uint32_t acc = tmem_base + buf * TC_BN;
                for (int kb = 0; kb < nkb && ok; ++kb) {
                    ok = agreed(mbar_wait(full_bar(s), use, a.error, 2));
                    if (!ok) break;
                    tc_fence_after();
                    const uint32_t sa = smem_base + s * TC_STAGE_BYTES, sb = sa + TC_A_BYTES;
                    const uint64_t da = umma_desc(sa), db = umma_desc(sb);
                    if (!PAIR || elect_one()) {
#pragma unroll
                        for (int k = 0; k < TC_BK / 16; ++k)   // 16 bfloat16 = 32 bytes further along K: +2 in units of 16 bytes
                            if (PAIR) umma_bf16_pair(acc, da + 2 * k, db + 2 * k, idesc, (kb | k) != 0);
                            else umma_bf16(acc, da + 2 * k, db + 2 * k, idesc, (kb | k) != 0);
                        // the stage is free (in both blocks) once these MMAs have read it
                        if (PAIR) umma_commit_pair(empty_bar(s), 3);
                        else umma_commit(empty_bar(s));
                    }
                    if (++s == TC_STAGES) {
                        s = 0;
                        use ^= 1;
                    }
                }
                // the accumulator is complete (or abandoned), in both blocks
                if (!PAIR) umma_commit(acc_full(buf));
                else if (elect_one()) umma_commit_pair(acc_full(buf), 3);
                ++lt;
            }
        }
    } else {
        // ---------------- epilogue: warps 2..9 of both blocks, TMEM lanes 32 * (warp % 4) ----------------
        const int quad = warp & 3;
        const int piece = (warp - 2) >> 2;      // which of the alternate 64-column pieces this warp takes
        const int row = quad * 32 + lane;
        // results whose rows start on 16-byte boundaries leave through this warp's strip of shared memory
        uint8_t* strip = smem_raw + (smem_base - smem_u32(smem_raw)) + TC_STAGES * TC_STAGE_BYTES + (warp - 2) * TC_STRIP_BYTES;
        const bool wide = !FLOAT && a.N % 8 == 0 && a.ldc % 8 == 0 && (reinterpret_cast<uintptr_t>(a.C) & 15) == 0;
        const bool wide_float = FLOAT && a.N % 4 == 0 && a.ldc % 4 == 0 && (reinterpret_cast<uintptr_t>(a.C) & 15) == 0;
        bool ok = true;
        int lt = 0;
        for (int t = pair; t < total && ok; t += pairs) {
            const TcTile tl = tc_tile(a, offsets, t, tiles_n, n_out, TcShape<CTAS>::ROWS);
            if (!tl.valid) continue;
            const int buf = lt & 1;
            const int m = tl.row0 + (int)rank * TC_BM + row, n0 = tl.n0;
            ok = mbar_wait_warp(acc_full(buf), (lt >> 1) & 1, a.error, 3);
            tc_fence_after();
            if (!ok) break;
            const uint32_t trow = tmem_base + buf * TC_BN + ((uint32_t)(quad * 32) << 16);
            // A warp whose 32 rows all lie beyond the group's rows has nothing to store (with a few rows per group
            // that is most warps of most tiles): it skips the work and only hands the accumulator back.
            const bool any_row = m - lane < tl.row_end;
            for (int c0 = 0; any_row && c0 < n_out; c0 += 32) {
                if (((c0 >> 6) & 1) != piece) continue;
                float v[32];
                tmem_ld32(trow + c0, v);               // warp-collective: every lane takes part
                if (!FLOAT && a.dual) {
                    float u[32];
                    tmem_ld32(trow + a.n_tile / 2 + c0, u);
                    // silu(g) * u = g * u / (1 + e^-g) in float, with the hardware's exponential and division
                    // (2 ulp; the result is rounded to bfloat16 next).  The exact forms cost some hundred clocks
                    // per value with only these four warps on the SM to hide them: measured, the epilogue of a tile
                    // took 7 to 18 us, as long as streaming half of the tile's weights.
                    if constexpr (BIASED) {
                        const float* bg = a.glu.bias + n0 + c0;
                        const int last = a.N - 1 - n0 - c0;           // columns past the last are computed and not stored
#pragma unroll
                        for (int i = 0; i < 32; ++i) {
                            const float* b = bg + min(i, last);
                            v[i] = glu_apply_biased(v[i], u[i], __ldg(b), __ldg(b + a.N));
                        }
                    } else {
#pragma unroll
                        for (int i = 0; i < 32; ++i) v[i] = glu_apply_fast(v[i], u[i], a.glu);
                    }
                }
                if (!FLOAT && wide) {
                    // A lane holds 32 columns of ONE row: stored from here, every instruction of the warp would touch
                    // 32 lines of memory.  So the warp passes two such chunks through its strip of shared memory
                    // (32 rows x 128 bytes; the 16-byte pieces of a row are XOR-swizzled by the row, so that neither
                    // side meets a bank twice) and stores whole 128-byte lines, four rows an instruction.
                    const int half = (c0 >> 5) & 1;
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        __nv_bfloat162 p0 = __floats2bfloat162_rn(v[8 * j], v[8 * j + 1]);
                        __nv_bfloat162 p1 = __floats2bfloat162_rn(v[8 * j + 2], v[8 * j + 3]);
                        __nv_bfloat162 p2 = __floats2bfloat162_rn(v[8 * j + 4], v[8 * j + 5]);
                        __nv_bfloat162 p3 = __floats2bfloat162_rn(v[8 * j + 6], v[8 * j + 7]);
                        uint4 pk;
                        pk.x = *reinterpret_cast<uint32_t*>(&p0);
                        pk.y = *reinterpret_cast<uint32_t*>(&p1);
                        pk.z = *reinterpret_cast<uint32_t*>(&p2);
                        pk.w = *reinterpret_cast<uint32_t*>(&p3);
                        *reinterpret_cast<uint4*>(strip + lane * 128 + (((half * 4 + j) ^ (lane & 7)) << 4)) = pk;
                    }
                    if (half == 1 || c0 + 32 >= n_out) {
                        __syncwarp();
                        const int cb = c0 - half * 32;                       // the strip's first column in the tile
                        const int cols = min(n_out - cb, a.N - n0 - cb);     // its columns that exist (may be <= 0)
                        const int p = lane & 7;
#pragma unroll
                        for (int i = 0; i < 8; ++i) {
                            const int r = (lane >> 3) + 4 * i;
                            const int mr = m - lane + r;
                            if (mr < tl.row_end && 8 * p + 8 <= cols) {       // N is a multiple of 8 here: no torn piece
                                const uint4 pk = *reinterpret_cast<const uint4*>(strip + r * 128 + ((p ^ (r & 7)) << 4));
                                *reinterpret_cast<uint4*>(static_cast<__nv_bfloat16*>(a.C) + (size_t)mr * a.ldc + n0 + cb +
                                                          8 * p) = pk;
                            }
                        }
                        __syncwarp();
                    }
                    continue;
                }
                if (FLOAT && wide_float) {
                    // the same for floats: a chunk's 32 columns are a whole line.  (Logits of 1,000 rows, K 2,048, N 32,000, single blocks: 290 us
                    // row by row, 172 so.)
#pragma unroll
                    for (int j = 0; j < 8; ++j)
                        *reinterpret_cast<float4*>(strip + lane * 128 + ((j ^ (lane & 7)) << 4)) =
                            make_float4(v[4 * j], v[4 * j + 1], v[4 * j + 2], v[4 * j + 3]);
                    __syncwarp();
                    const int cols = min(n_out - c0, a.N - n0 - c0), p = lane & 7;
#pragma unroll
                    for (int i = 0; i < 8; ++i) {
                        const int r = (lane >> 3) + 4 * i, mr = m - lane + r;
                        if (mr < tl.row_end && 4 * p + 4 <= cols)
                            *reinterpret_cast<float4*>(static_cast<float*>(a.C) + (size_t)mr * a.ldc + n0 + c0 + 4 * p) =
                                *reinterpret_cast<const float4*>(strip + r * 128 + ((p ^ (r & 7)) << 4));
                    }
                    __syncwarp();
                    continue;
                }
                const int c_end = min(n_out - c0, a.N - n0 - c0);   // columns of this chunk that exist (may be <= 0)
                if (m < tl.row_end && c_end > 0) {
                    if constexpr (FLOAT) {
                        float* dst = static_cast<float*>(a.C) + (size_t)m * a.ldc + n0 + c0;
#pragma unroll
                        for (int i = 0; i < 32; ++i)
                            if (i < c_end) dst[i] = v[i];
                    } else {
                        __nv_bfloat16* dst = static_cast<__nv_bfloat16*>(a.C) + (size_t)m * a.ldc + n0 + c0;
#pragma unroll
                        for (int i = 0; i < 32; ++i)
                            if (i < c_end) dst[i] = __float2bfloat16_rn(v[i]);
                    }
                }
            }
            if (BIASED && a.glu.fill && piece == 0 && n0 + n_out >= a.N && m < tl.row_end) {
                __nv_bfloat16* pad = static_cast<__nv_bfloat16*>(a.C) + (size_t)m * a.ldc + a.N;
                for (int e = 0; e < a.glu.fill; ++e) pad[e] = __float2bfloat16_rn(e == 0 ? 1.f : 0.f);
            }
            // this warp has read its lanes of the accumulator: tell the leader's MMA thread
            tc_fence_before();
            __syncwarp();
            if (lane == 0) {
                if (PAIR) mbar_arrive_cluster(mapa_shared(acc_empty(buf), 0));
                else asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(acc_empty(buf)) : "memory");
            }
            ++lt;
        }
    }
    __syncwarp();
    tc_fence_before();
    if (PAIR) cluster_sync_all();             // neither block leaves while the other may still signal it
    else __syncthreads();
    if (warp == 1) {
        if (PAIR) tmem_dealloc_pair(tmem_base, 2 * TC_BN);
        else tmem_dealloc(tmem_base, 2 * TC_BN);
    }
}

// Gather rows: out[m, :] = x[rows[m], :]  (activations sorted by expert, so that TMA can fetch tiles)
__global__ void gather_rows_kernel(const __nv_bfloat16* __restrict__ x, const int* __restrict__ rows,
                                   __nv_bfloat16* __restrict__ out, int d) {
    pdl_sync();
    const int m = blockIdx.x;
    const uint4* src = reinterpret_cast<const uint4*>(x + (size_t)rows[m] * d);
    uint4* dst = reinterpret_cast<uint4*>(out + (size_t)m * d);
    for (int c = threadIdx.x; c < d / 8; c += blockDim.x) dst[c] = src[c];
}

// ---- host side -----------------------------------------------------------------------------
typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

static EncodeTiledFn encode_fn() {
    static EncodeTiledFn fn = nullptr;
    static std::once_flag once;
    std::call_once(once, [] {
        void* p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            fn = reinterpret_cast<EncodeTiledFn>(p);
    });
    return fn;
}

// [rows, K] bfloat16, row pitch ld elements; box = 64 columns x box_rows rows, 128-byte swizzle.
int make_map(CUtensorMap* out, const void* base, long long rows, int K, long long ld, int box_rows) {
    static std::map<std::tuple<const void*, long long, int, long long, int>, CUtensorMap> cache;
    static std::mutex lock;
    std::lock_guard<std::mutex> hold(lock);
    auto key = std::make_tuple(base, rows, K, ld, box_rows);
    auto it = cache.find(key);
    if (it != cache.end()) {
        *out = it->second;
        return 0;
    }
    EncodeTiledFn fn = encode_fn();
    if (!fn) return TB_ERR_UNSUPPORTED;
    cuuint64_t dims[2] = {(cuuint64_t)K, (cuuint64_t)rows};
    cuuint64_t strides[1] = {(cuuint64_t)ld * 2};
    cuuint32_t box[2] = {TC_BK, (cuuint32_t)box_rows};
    cuuint32_t estr[2] = {1, 1};
    CUresult r = fn(out, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(base), dims, strides, box, estr,
                    CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                    CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) return TB_ERR_ARG;
    if (cache.size() > 4096) cache.clear();
    cache[key] = *out;
    return 0;
}

static __device__ int tc_error_word;

int* tc_error_ptr() {
    static int* p = nullptr;
    if (!p) {
        const cudaError_t e = cudaGetSymbolAddress((void**)&p, tc_error_word);
        if (e != cudaSuccess) {
            p = nullptr;
            tb_note_error(e);     // the launcher that asked returns this code
        }
    }
    return p;
}

template <int CTAS, int EPI>
static int tc_launch(const CUtensorMap& ma, const CUtensorMap& mb, TcArgs a, cudaStream_t s) {
    const size_t smem = (size_t)TcShape<CTAS>::STAGES * TcShape<CTAS>::STAGE_BYTES + TC_EPI_WARPS * TC_STRIP_BYTES + 1024;
    static bool configured = false;
    if (!configured) {
        cudaError_t e = cudaFuncSetAttribute(gemm_tc_kernel<CTAS, EPI>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (e != cudaSuccess) return (int)e;
        configured = true;
    }
    const int n_out = a.dual ? a.n_tile / 2 : a.n_tile, rows = TcShape<CTAS>::ROWS;
    a.tiles_m = a.group_offsets ? (a.M + rows - 1) / rows + a.G : (a.M + rows - 1) / rows;
    cudaLaunchConfig_t cfg = {};
    cfg.blockDim = dim3(TC_THREADS);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    attr[1].id = cudaLaunchAttributeClusterDimension;
    attr[1].val.clusterDim.x = CTAS;
    attr[1].val.clusterDim.y = 1;
    attr[1].val.clusterDim.z = 1;
    cfg.attrs = attr;
    static int max_units = 0;                  // blocks (or pairs of blocks) that can be resident at once
    if (!max_units) {
        int sms = 0, dev = 0;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
        max_units = sms > 0 ? sms : 1;         // one persistent block per SM
        if (CTAS == 2) {
            int n = 0;
            cfg.gridDim = dim3(sms > 1 ? sms / 2 * 2 : 2);
            cfg.numAttrs = 2;
            const cudaError_t e = cudaOccupancyMaxActiveClusters(&n, gemm_tc_kernel<CTAS, EPI>, &cfg);
            if (e != cudaSuccess) {
                cudaGetLastError();
                max_units = 0;                 // asked again at the next launch
                return (int)e;                 // a failed query is an error, not "no room"
            }
            if (n <= 0) {
                max_units = 0;
                return TB_ERR_UNSUPPORTED;     // no room for a pair of these blocks on this device
            }
            max_units = n;
        }
    }
    const int total = a.tiles_m * ((a.N + n_out - 1) / n_out);
    const int units = total < max_units ? total : max_units;
    cfg.gridDim = dim3(CTAS * units);
    cfg.numAttrs = CTAS == 2 ? 2 : 1;
    tb_state_carveout((const void*)gemm_tc_kernel<CTAS, EPI>, TC_THREADS, smem);
    cudaLaunchKernelEx(&cfg, gemm_tc_kernel<CTAS, EPI>, ma, mb, a);
    return tb_last_error();
}

static int tc_sms() {
    static int sms = 0;
    if (!sms) {
        int dev = 0;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
        if (sms < 2) sms = 2;
    }
    return sms;
}

static int tc_tiles_n(int N, bool dual) { return (N + (dual ? TC_BN / 2 : TC_BN) - 1) / (dual ? TC_BN / 2 : TC_BN); }

// Pairs of blocks, where they take at most a seventh more rounds over the SMs than single blocks would (a round of theirs takes about 7/8 of the
// time: B is staged once for 256 rows), counting half a tile of padding a group.  What fits one round stays with single blocks, and so does
// a short K (below 512, or 1,024 with fewer than 512 rows a group), whose start counts.  Single blocks / pairs, us (many launches between two
// events, weights from memory; profiles/gemm_tc_pairs.md has more):
//   (gate, up) 5,632 wide, K 2,048: 520 rows 29.3 / 26.8, 1,000 42 / 38, 2,048 73 / 64, 4,096 162 / 137; 300 rows 17.9 / 25.4 (1 round, 2)
//   logits of 32,000 tokens, K 2,048: 200 rows 49 / 36, 500 93 / 66, 1,000 172 / 128; 64 rows 33 / 41
//   16 experts, (gate, up) 688 wide, K 4,096: 200 rows each 59 / 55, 384 84 / 80, 640 130 / 114, 1,024 169 / 165; 512 93 / 103 (3 rounds, 4)
//   their down product (4,096 wide, K 688): 512 rows each 59 / 55, 1,024 113 / 95, 2,048 216 / 181; 128 31 / 33
//   8 experts 14,336 wide, K 4,096, by themselves at the power limit, where two runs differ by a tenth: 512 rows each 828 / 829 and 777 / 803,
//   768 1,240 / 1,169, 1,024 1,544 / 1,338, 2,048 2,904 / 2,538; in a model of 32 such layers 2,048 tokens take 56.0 ms / 54.1
//   2,048 wide, K 128: 3,000 rows 6.8 / 7.5
static bool tc_takes_pairs(int M, int N, int K, int G, bool grouped, bool dual, int sms) {
    if (M <= TC_BM * (long long)G || K < (M >= 512ll * G ? 512 : 1024)) return false;
    const long long pad = grouped ? G : 0, tiles_n = tc_tiles_n(N, dual);
    const long long single = (((long long)M + TC_BM - 1) / TC_BM + pad / 2) * tiles_n, twos = (((long long)M + 2 * TC_BM - 1) / (2 * TC_BM) + pad / 2) * tiles_n;
    const long long rounds = (single + sms - 1) / sms, pair_rounds = (twos + sms / 2 - 1) / (sms / 2);
    return rounds >= 2 && 7 * pair_rounds <= 8 * rounds;
}

// C[m] = A[m] . B[g(m)]^T.  A [M, K] (rows sorted by group), B [G, rows_b, K] with rows_b = N (or 2N when
// out_kind == 2: gate rows then up rows).  out_kind: 0 bfloat16, 1 float, 2 swiglu (bfloat16).
// Refuses (TB_ERR_UNSUPPORTED) what TMA cannot address: K or a pitch that is no multiple of 8,
// a base that is not 16-byte aligned.
static int gemm_tc_entry(const void* A, const void* B, void* C, const int* group_offsets, int lda, int ldb, int ldc,
                         int M, int N, int K, int G, int out_kind, GluRule glu, cudaStream_t s) {
    if (M < 0 || N <= 0 || K <= 0 || G <= 0 || out_kind < 0 || out_kind > 2) return TB_ERR_ARG;
    if (K % 8 || lda % 8 || ldb % 8) return TB_ERR_UNSUPPORTED;
    if (((uintptr_t)A | (uintptr_t)B) & 15) return TB_ERR_UNSUPPORTED;
    if (M == 0) return 0;
    const int dual = out_kind == 2;
    const int rows_b = dual ? 2 * N : N;
    // Rows of B per tile: as many column tiles as the full width would need, but of equal widths (N = 688 with
    // swiglu: six tiles of 120 gate and 120 up rows instead of five of 128 and one of 48 padded to 128).
    const int sms = tc_sms(), tiles_n = tc_tiles_n(N, dual);
    const bool pair = tc_takes_pairs(M, N, K, G, group_offsets != nullptr, dual, sms);
    int n_tile;
    {
        const int unit = (pair ? 32 : 16) >> dual;      // a pair's B tile is a multiple of 32 rows
        const int out = ((N + tiles_n - 1) / tiles_n + unit - 1) / unit * unit;
        n_tile = dual ? 2 * out : out;
    }
    // With about one row tile per group (decoding with many sequences: the product streams
    // the experts' weights once and has G x column tiles to spread over the SMs) narrower tiles can fill a round
    // of SMs where the full width leaves a third of them idle; costs in rows loaded per k-block and round.
    if (group_offsets && (long long)M <= (long long)TC_BM * G) {
        long long best = -1;
        for (int nt = TC_BN; nt >= 64; nt -= 16) {
            const int out = dual ? nt / 2 : nt;
            const long long tiles = (long long)G * ((N + out - 1) / out);
            const long long cost = (tiles + sms - 1) / sms * (64 + nt);
            if (best < 0 || cost < best) {
                best = cost;
                n_tile = nt;
            }
        }
    }
    CUtensorMap ma, mb;
    int rc = make_map(&ma, A, M, K, lda, TC_BM);
    if (rc) return rc;
    rc = make_map(&mb, B, (long long)G * rows_b, K, ldb, n_tile / 2);     // a box is half of the B tile
    if (rc) return rc;
    int* err_ptr = tc_error_ptr();
    if (!err_ptr) return tb_last_error();
    TcArgs a{C, group_offsets, err_ptr, ldc, M, N, K, G, rows_b, dual, 0, n_tile, glu};
    if (glu.bias) {
        rc = pair ? tc_launch<2, TC_EPI_BIASED>(ma, mb, a, s) : TB_ERR_UNSUPPORTED;
        if (rc == TB_ERR_UNSUPPORTED) rc = tc_launch<1, TC_EPI_BIASED>(ma, mb, a, s);
        return rc;
    }
    if (out_kind == 1) {
        rc = pair ? tc_launch<2, TC_EPI_FLOAT>(ma, mb, a, s) : TB_ERR_UNSUPPORTED;
        return rc == TB_ERR_UNSUPPORTED ? tc_launch<1, TC_EPI_FLOAT>(ma, mb, a, s) : rc;
    }
    rc = pair ? tc_launch<2, TC_EPI_BF16>(ma, mb, a, s) : TB_ERR_UNSUPPORTED;
    if (rc == TB_ERR_UNSUPPORTED) rc = tc_launch<1, TC_EPI_BF16>(ma, mb, a, s);
    return rc;
}

extern "C" {
int tb_gemm_tc_bf16(const void* A, const void* B, void* C, const int* group_offsets, int lda, int ldb, int ldc, int M,
                    int N, int K, int G, int out_kind, cudaStream_t s) {
    return gemm_tc_entry(A, B, C, group_offsets, lda, ldb, ldc, M, N, K, G, out_kind, GluRule{0, 0.f, 0.f}, s);
}
// The (gate, up) pair product with another form of the pair (see GluRule, kinds 1 and 3).
int tb_gemm_tc_glu_bf16(const void* A, const void* B, void* C, const int* group_offsets, int lda, int ldb, int ldc,
                        int M, int N, int K, int G, float alpha, float limit, int kind, cudaStream_t s) {
    if (kind != 1 && kind != TB_GLU_GELU_TANH) return TB_ERR_ARG;
    return gemm_tc_entry(A, B, C, group_offsets, lda, ldb, ldc, M, N, K, G, 2, GluRule{kind, alpha, limit}, s);
}

// The (gate, up) pair with biases: C[m, n] = silu(g + bias[n]) (u + bias[N + n]), then `fill` columns of a one and zeros.
int tb_gemm_tc_bias_glu_bf16(const void* A, const void* B, const float* bias, void* C, int lda, int ldb, int ldc, int M, int N, int K,
                             int fill, cudaStream_t s) {
    if (!bias || fill < 0 || ldc < N + fill) return TB_ERR_ARG;
    return gemm_tc_entry(A, B, C, nullptr, lda, ldb, ldc, M, N, K, 1, 2, GluRule{0, 0.f, 0.f, bias, fill}, s);
}

// Whether tb_gemm_tc_bf16 takes pairs of blocks on a GPU of so many SMs (0: on this one).
int tb_gemm_tc_takes_pairs(int M, int N, int K, int G, int grouped, int out_kind, int sms) {
    return tc_takes_pairs(M, N, K, G, grouped != 0, out_kind == 2, sms > 0 ? sms : tc_sms());
}

// Nonzero if any tensor-core product gave up on a wait since the last call (1 producer, 2 MMA,
// 3 epilogue, 4 drain, 5 accumulator hand-back); reading it synchronises the device and clears it.
int tb_gemm_tc_status() {
    int v = 0, zero = 0;
    if (cudaMemcpyFromSymbol(&v, tc_error_word, sizeof(int)) != cudaSuccess) return -1;
    if (v) cudaMemcpyToSymbol(tc_error_word, &zero, sizeof(int));
    return v;
}

// The same word copied to `host_dst` (pinned host memory) in stream order, without waiting: it arrives with
// whatever else the caller reads back from that stream, and is not cleared.
int tb_kernel_status_async(int* host_dst, cudaStream_t s) {
    int* p = tc_error_ptr();
    if (!p) return tb_last_error();
    return (int)cudaMemcpyAsync(host_dst, p, sizeof(int), cudaMemcpyDeviceToHost, s);
}

int tb_gather_rows_bf16(const void* x, const int* rows, void* out, int M, int d, cudaStream_t s) {
    if (M < 0 || d <= 0) return TB_ERR_ARG;
    if (d % 8 || (((uintptr_t)x | (uintptr_t)out) & 15)) return TB_ERR_UNSUPPORTED;
    if (M == 0) return 0;
    TB_LAUNCH((gather_rows_kernel), M, 128, 0, s, (const __nv_bfloat16*)x, rows, (__nv_bfloat16*)out, d);
    return tb_last_error();
}
}

// replayable from C++ (tape.h)
#include "tape.h"
TB_TAPE_REGISTER(tb_gemm_tc_bf16)
TB_TAPE_REGISTER(tb_gemm_tc_glu_bf16)
TB_TAPE_REGISTER(tb_gemm_tc_bias_glu_bf16)
TB_TAPE_REGISTER(tb_gather_rows_bf16)

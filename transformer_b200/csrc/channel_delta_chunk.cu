// The gated delta rule of channel_delta.cu for prompts: 16 tokens at a time through the closed form of a chunk.
//
// With G_t the product of the chunk's decays up to token t (per key channel) and S the state before the chunk:
//   A_tj = sum_c k_tc (G_t / G_j)_c k_jc  (j < t),   B_tj = sum_c q_tc (G_t / G_j)_c k_jc  (j <= t)
//   u_t = beta_t (v_t - S^T (G_t k_t) - sum_{j<t} A_tj u_j)     o_t = S^T (G_t q_t) + sum_{j<=t} B_tj u_j
//   S <- diag(G_last) S + sum_j (G_last / G_j k_j) u_j^T
// The u are linear in S: u = U0 - W S, where U0 and W solve the same unit triangular system with beta v and beta G k on
// the right.  So everything but three products with S is made for all chunks at once, and only the products walk the
// sequence.  The ratios G_t / G_j are products of the decays between the two tokens, never quotients: a decay may be
// as small as float allows.  All of it in float, as token by token.
//
//   delta_chunk_kernel        a block = a chunk x a head: convolution, silu, unit norms, decays, A and B, the two
//                             solutions, one record for the scan
//   delta_chunk_scan_kernel   a block = a sequence x a head x 16 or 32 columns of S
// Measured with 16 heads of 128 x 128 (both kernels; before: records and scan token by token): one prompt of 2,048 tokens
// 310 us (812), two of 1,500 351 (837), eight of 1,024 784 (1,770).  The first kernel is bound by instruction issue
// and shared-memory reads in equal parts (34 KB and 64 registers a thread leave four blocks an SM); a warp leaves out the
// tokens before its first key (135 to 126 us for two prompts of 1,500 tokens).  The scan of few sequences is bound by the
// chain of a chunk (1.7 us; one block an SM), that of many by what goes through shared memory: a piece of a record that a
// lane loads serves its four columns, and 16 lanes to a column instead of 32 halve the exchange of the sums: eight
// prompts 465 us (563 with 32 lanes), four of 600 143 (188).  Eight lanes to a column: 481 and 163.  All forms add in one order and
// have the same bits.
#include "channel_delta.cuh"
#include "memory_common.cuh"            // fma2, mul2
#include "tc_common.cuh"                // bulk copies, barriers with bounded waits

#define DC_TOK 16           // tokens of a chunk
#define DC_TAPS 4           // the convolution's width that these kernels take
#define DC_BP 20            // pitch of B's rows: the 16 lanes that read a row each start in different banks
#define DC_COLS 16          // columns of the state per scan block
#define DC_STAGES 3

// A record of one (head, chunk):  W | G q | G_last / G_j k, [16][dim] each | G_last [dim] | B [16][DC_BP], then
// U0 as [vdim / 16][16 tokens][16 columns], so that a scan block's share is one piece.
__host__ __device__ inline int dc_main(int dim) { return (3 * DC_TOK + 1) * dim + DC_TOK * DC_BP; }
__host__ __device__ inline int dc_record(int dim, int vdim) { return dc_main(dim) + DC_TOK * vdim; }

// Two neighbouring channels.
__device__ __forceinline__ float2 dc_load2(const float* p) { return *reinterpret_cast<const float2*>(p); }
__device__ __forceinline__ float2 dc_load2(const __nv_bfloat16* p) {
    return __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(p));
}

// Chunks are counted over the step's sequences; the grid covers the most there can be (max_chunks).
template <typename T, int DIM>
__global__ void __launch_bounds__(256, 4) delta_chunk_kernel(const DeltaPrepArgs p, int B, int max_chunks) {
    pdl_sync();
    extern __shared__ __align__(16) float dc_sm[];
    const int vdim = p.vdim, gd = p.G * DIM, taps = DC_TAPS;
    float* q = dc_sm;                       // [16][DIM]
    float* k = q + DC_TOK * DIM;            // [16][DIM]
    float* g = k + DC_TOK * DIM;            // [16][DIM]
    float* v = g + DC_TOK * DIM;            // [16][vdim]
    float* A = v + DC_TOK * vdim;           // [16][16]
    __shared__ float beta[DC_TOK];
    const int hh = blockIdx.y, kv = hh / (p.H / p.G), tid = threadIdx.x;
    int chunk = blockIdx.x, b = 0, t0 = 0, n = 0;
    for (; b < B; ++b) {
        t0 = p.seq_start[b];
        n = p.seq_start[b + 1] - t0;
        const int chunks = (n + DC_TOK - 1) / DC_TOK;
        if (chunk < chunks) break;
        chunk -= chunks;
    }
    if (b == B) return;
    const int li0 = chunk * DC_TOK, tb = t0 + li0;          // the chunk's first token: in its sequence, in the step
    n = min(DC_TOK, n - li0);
    float* rec = p.rec + ((size_t)hh * max_chunks + blockIdx.x) * dc_record(DIM, vdim);
    const T* z = static_cast<const T*>(p.z);
    const int C = 2 * gd + p.H * vdim;
    const float* cs = p.state + (size_t)p.slots[b] * p.state_stride + p.conv_offset;
    // convolution and silu: a thread has two neighbouring channels, its 16 tokens and the 3 before them in registers
    for (int i = tid * 2; i < 2 * DIM + vdim; i += 512) {
        const int c = i < DIM ? kv * DIM + i : i < 2 * DIM ? gd + kv * DIM + (i - DIM) : 2 * gd + hh * vdim + (i - 2 * DIM);
        float2 x[DC_TOK + DC_TAPS - 1];
#pragma unroll
        for (int j = 0; j < DC_TOK + DC_TAPS - 1; ++j) {
            const int back = taps - 1 - j;              // x[j] is the input of the chunk's token -back
            if (j >= taps - 1 + n) x[j] = make_float2(0.f, 0.f);
            else if (li0 >= back) x[j] = dc_load2(z + (size_t)(tb - back) * p.ldz + c);
            else x[j] = make_float2(cs[(size_t)(taps - 1 + li0 - back) * C + c], cs[(size_t)(taps - 1 + li0 - back) * C + c + 1]);
        }
        const float4 w0 = *reinterpret_cast<const float4*>(p.wconv + (size_t)c * taps);
        const float4 w1 = *reinterpret_cast<const float4*>(p.wconv + (size_t)(c + 1) * taps);
        float* to = i < DIM ? q + i : i < 2 * DIM ? k + (i - DIM) : v + (i - 2 * DIM);
        const int pitch = i < 2 * DIM ? DIM : vdim;
#pragma unroll
        for (int t = 0; t < DC_TOK; ++t) {
            const float a0 = w0.x * x[t].x + w0.y * x[t + 1].x + w0.z * x[t + 2].x + w0.w * x[t + 3].x;
            const float a1 = w1.x * x[t].y + w1.y * x[t + 1].y + w1.z * x[t + 2].y + w1.w * x[t + 3].y;
            const bool there = t < n;
            *reinterpret_cast<float2*>(to + t * pitch) =
                make_float2(there ? a0 / (1.0f + expf(-a0)) : 0.f, there ? a1 / (1.0f + expf(-a1)) : 0.f);
        }
    }
    // decays (1 for tokens that are not there) and betas (0)
    const float rate = expf(p.A_log[hh]);
    for (int i = tid; i < DC_TOK * DIM; i += 256) {
        const int t = i / DIM, c = i % DIM;
        float gg = 1.f;
        if (t < n) {
            const int e = p.head_decay ? hh : hh * DIM + c;
            gg = expf(-rate * cd_softplus(p.a[(size_t)(tb + t) * p.lda + e] + p.dt_bias[e]));
        }
        g[i] = gg;
    }
    if (tid < DC_TOK) beta[tid] = tid < n ? 1.0f / (1.0f + expf(-p.bz[(size_t)(tb + tid) * p.ldb + hh])) : 0.f;
    __syncthreads();
    // unit norms: a warp per token
    const int lane = tid & 31, warp = tid >> 5;
#pragma unroll
    for (int t = warp; t < DC_TOK; t += 8) {
        float qv[DIM / 32], kvv[DIM / 32], sq = 0.f, sk = 0.f;
#pragma unroll
        for (int e = 0; e < DIM / 32; ++e) {
            qv[e] = q[t * DIM + lane + 32 * e];
            kvv[e] = k[t * DIM + lane + 32 * e];
            sq += qv[e] * qv[e];
            sk += kvv[e] * kvv[e];
        }
        sq = warp_sum(sq);
        sk = warp_sum(sk);
        const float iq = rsqrtf((float)DIM) / sqrtf(sq + CD_UNIT_EPS), ik = 1.0f / sqrtf(sk + CD_UNIT_EPS);
#pragma unroll
        for (int e = 0; e < DIM / 32; ++e) {
            q[t * DIM + lane + 32 * e] = qv[e] * iq;
            k[t * DIM + lane + 32 * e] = kvv[e] * ik;
        }
    }
    __syncthreads();
    // A and B: 16 lanes hold key j, which fades from token to token; the lanes' sums are scattered so that lane i of
    // the 16 ends with row i
    {
        constexpr int R4 = DIM / 64;
        const int j = tid >> 4, part = tid & 15, first = __shfl_sync(0xffffffffu, j, 0);     // no key of the warp is there earlier
        float kt[R4 * 4], s[2 * DC_TOK];
#pragma unroll
        for (int e = 0; e < R4 * 4; ++e) kt[e] = 0.f;
#pragma unroll
        for (int i = 0; i < DC_TOK; ++i) {
            float sa = 0.f, sb = 0.f;
            if (i >= first)
#pragma unroll
            for (int r = 0; r < R4; ++r) {
                const int c = i * DIM + r * 64 + part * 4;
                const float4 ki = *reinterpret_cast<const float4*>(k + c), qi = *reinterpret_cast<const float4*>(q + c);
                const float4 gi = *reinterpret_cast<const float4*>(g + c);
                float* kr = kt + r * 4;
                kr[0] = i == j ? ki.x : kr[0] * gi.x;
                kr[1] = i == j ? ki.y : kr[1] * gi.y;
                kr[2] = i == j ? ki.z : kr[2] * gi.z;
                kr[3] = i == j ? ki.w : kr[3] * gi.w;
                sa += kr[0] * ki.x + kr[1] * ki.y + kr[2] * ki.z + kr[3] * ki.w;
                sb += kr[0] * qi.x + kr[1] * qi.y + kr[2] * qi.z + kr[3] * qi.w;
            }
            s[2 * i] = sa;
            s[2 * i + 1] = sb;
        }
#pragma unroll
        for (int half = 8; half > 0; half >>= 1) {
            const bool up = part & half;
#pragma unroll
            for (int i = 0; i < 2 * half; ++i) {
                const float keep = up ? s[i + 2 * half] : s[i], give = up ? s[i] : s[i + 2 * half];
                s[i] = keep + __shfl_xor_sync(0xffffffffu, give, half);
            }
        }
        A[part * DC_TOK + j] = s[0];
        rec[(3 * DC_TOK + 1) * DIM + part * DC_BP + j] = s[1];      // 0 for j > i
    }
    __syncthreads();
    // a thread solves for a column of W or of U0, and carries the decays along
    for (int col = tid; col < DIM + vdim; col += 256) {
        float x[DC_TOK];
        const bool key = col < DIM;
        const int vc = col - DIM;
        float G = 1.f;
        float* out = key ? rec + col : rec + dc_main(DIM) + (vc >> 4) * (DC_TOK * DC_COLS) + (vc & 15);
        const int pitch = key ? DIM : DC_COLS;
#pragma unroll
        for (int i = 0; i < DC_TOK; ++i) {
            float r;
            if (key) {
                G *= g[i * DIM + col];
                r = G * k[i * DIM + col];
                rec[(DC_TOK + i) * DIM + col] = G * q[i * DIM + col];
            } else {
                r = v[i * vdim + vc];
            }
#pragma unroll
            for (int l = 0; l < i; ++l) r -= A[i * DC_TOK + l] * x[l];
            x[i] = beta[i] * r;
            out[i * pitch] = x[i];
        }
        if (key) {
            rec[3 * DC_TOK * DIM + col] = G;
            float f = 1.f;
#pragma unroll
            for (int i = DC_TOK - 1; i >= 0; --i) {
                rec[(2 * DC_TOK + i) * DIM + col] = f * k[i * DIM + col];
                f *= g[i * DIM + col];
            }
        }
    }
}

struct DeltaChunkScanArgs {
    const float* rec;       // [H][max_chunks][dc_record]
    float* state;           // [slots, state_stride], S first
    int* error;             // set by a wait that runs out
    float* out;             // [nt, H vdim]
    const int* seq_start;
    const int* slots;
    long long state_stride;
    int max_chunks, H, vdim;
};

// 128 threads: LANES lanes share C columns and split the rows (DIM / LANES each, in registers, pieces of four
// interleaved).  Per chunk: the sums over S for W and G q (16 tokens x C columns each), scattered so that every lane ends
// with one token's sums for C or, of 32 lanes, C / 2 columns; u through shared memory to all lanes of the columns; the
// update.  OWN: a lane takes the tokens in an order of its own (place t holds token t ^ its number), so the half that it gives
// away is at the same places in every lane and nothing is selected.  With two rows' pieces a lane that is the faster way;
// with one, where the chain of a chunk counts, the addresses that the lane's number enters cost more than the selects (one prompt of 2,048
// tokens 235 us and 221; heads of 64: 179 and 157).  A lane's two pieces are summed apart and then together, as the
// first exchange of 32 lanes has them.  The records come by bulk copy, two chunks ahead, with bounded waits.
template <int DIM, int LANES, int C, bool OWN>
__global__ void __launch_bounds__(128) delta_chunk_scan_kernel(const DeltaChunkScanArgs a) {
    pdl_sync();
    constexpr int R4 = DIM / (4 * LANES), CB = LANES / DC_TOK, OUT = C / CB, COLS = 128 / LANES * C;
    static_assert((CB == 1 || CB == 2) && OUT % 2 == 0 && COLS % DC_COLS == 0 && R4 * 4 * LANES == DIM, "a lane ends with a token's sums");
    constexpr int MAIN = (3 * DC_TOK + 1) * DIM + DC_TOK * DC_BP, STAGE = MAIN + DC_TOK * COLS;
    extern __shared__ __align__(16) float dc_sm[];          // [DC_STAGES][STAGE]
    __shared__ __align__(16) float us[COLS / C][DC_TOK][C];
    __shared__ __align__(8) unsigned long long bars[DC_STAGES];
    const int b = blockIdx.x, h = blockIdx.y, tid = threadIdx.x;
    const int part = tid & (LANES - 1), group = tid / LANES, col = blockIdx.z * COLS + group * C;
    const int my_tok = part / CB, my_col = part % CB * OUT;     // whose sums this lane ends with
    const int H = a.H, vdim = a.vdim;
    const int t0 = a.seq_start[b], n_tok = a.seq_start[b + 1] - t0;
    if (n_tok <= 0) return;
    int first = 0;                                          // chunks of the sequences before this one
    for (int i = 0; i < b; ++i) first += (a.seq_start[i + 1] - a.seq_start[i] + DC_TOK - 1) / DC_TOK;
    const int chunks = (n_tok + DC_TOK - 1) / DC_TOK;
    float* S = a.state + (size_t)a.slots[b] * a.state_stride + (size_t)h * DIM * vdim;
    F2 s[C][R4 * 2];                                        // [column][pairs of rows]
#pragma unroll
    for (int i = 0; i < R4 * 2; ++i) {
        const int r = (i >> 1) * (4 * LANES) + part * 4 + (i & 1) * 2;
#pragma unroll
        for (int c = 0; c < C; c += 2) {
            const float2 x = *reinterpret_cast<const float2*>(S + (size_t)r * vdim + col + c);
            const float2 y = *reinterpret_cast<const float2*>(S + (size_t)(r + 1) * vdim + col + c);
            s[c][i].f = make_float2(x.x, y.x);
            s[c + 1][i].f = make_float2(x.y, y.y);
        }
    }
    const size_t rec_floats = dc_record(DIM, vdim);
    const float* rec = a.rec + ((size_t)h * a.max_chunks + first) * rec_floats;
    const uint32_t bar0 = smem_u32(bars);
    if (tid == 0) {
        for (int i = 0; i < DC_STAGES; ++i) mbar_init(bar0 + 8u * i, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();
    auto issue = [&](int ch) {
        if (tid != 0) return;
        const uint32_t to = smem_u32(dc_sm + (size_t)(ch % DC_STAGES) * STAGE), bar = bar0 + 8u * (ch % DC_STAGES);
        const float* from = rec + (size_t)ch * rec_floats;
        mbar_expect_tx(bar, STAGE * sizeof(float));
        bulk_load(to, from, MAIN * sizeof(float), bar);
        bulk_load(to + MAIN * sizeof(float), from + MAIN + (size_t)blockIdx.z * (DC_TOK * COLS), DC_TOK * COLS * sizeof(float), bar);
    };
    union Four { float4 f; F2 p[2]; };
    // this lane's part of the sums over S for 16 rows of a record, [token][pair of columns]
    auto sums = [&](const float* rows, F2 (&sum)[DC_TOK][C / 2]) {
#pragma unroll
        for (int t = 0; t < DC_TOK; ++t) {
            const float* row = rows + (OWN ? t ^ my_tok : t) * DIM + part * 4;
#pragma unroll
            for (int r = 0; r < R4; ++r) {
                Four w;
                F2 acc[C];
                w.f = *reinterpret_cast<const float4*>(row + r * (4 * LANES));
#pragma unroll
                for (int c = 0; c < C; ++c) acc[c] = fma2(w.p[1], s[c][r * 2 + 1], mul2(w.p[0], s[c][r * 2]));
#pragma unroll
                for (int c = 0; c < C; c += 2) {
                    F2 two;
                    two.f = make_float2(acc[c].f.x + acc[c].f.y, acc[c + 1].f.x + acc[c + 1].f.y);
                    sum[t][c / 2] = r == 0 ? two : add2(sum[t][c / 2], two);
                }
            }
        }
    };
    // the lanes' parts together: every lane ends with its own token's columns (the same pairs of lanes are added in both forms)
    auto meet = [&](F2 (&sum)[DC_TOK][C / 2], float (&mine)[OUT]) {
#pragma unroll
        for (int half = DC_TOK / 2; half > 0; half >>= 1) {
            const bool up = my_tok & half;
#pragma unroll
            for (int t = 0; t < half; ++t)
#pragma unroll
                for (int c = 0; c < C / 2; ++c) {
                    const F2 keep = !OWN && up ? sum[t + half][c] : sum[t][c], give = !OWN && up ? sum[t][c] : sum[t + half][c];
                    F2 in;
                    in.f.x = __shfl_xor_sync(0xffffffffu, give.f.x, half * CB);
                    in.f.y = __shfl_xor_sync(0xffffffffu, give.f.y, half * CB);
                    sum[t][c] = add2(keep, in);
                }
        }
#pragma unroll
        for (int c = 0; c < OUT / 2; ++c) {
            F2 keep = sum[0][c];
            if (CB == 2) {
                const F2 give = my_col ? keep : sum[0][c + OUT / 2];
                F2 in;
                in.f.x = __shfl_xor_sync(0xffffffffu, give.f.x, 1);
                in.f.y = __shfl_xor_sync(0xffffffffu, give.f.y, 1);
                keep = add2(my_col ? sum[0][c + OUT / 2] : keep, in);
            }
            mine[2 * c] = keep.f.x;
            mine[2 * c + 1] = keep.f.y;
        }
    };
    int issued = 0;
    for (; issued < DC_STAGES - 1 && issued < chunks; ++issued) issue(issued);
    for (int ch = 0; ch < chunks; ++ch) {
        const bool ok = mbar_wait(bar0 + 8u * (ch % DC_STAGES), (ch / DC_STAGES) & 1, a.error, 35);
        // the record has landed for everyone, and everyone is done with the one before
        if (!__syncthreads_and(ok)) {
            if (tid == 0)
                for (int i = ch; i < issued; ++i) mbar_wait(bar0 + 8u * (i % DC_STAGES), (i / DC_STAGES) & 1, a.error, 36);
            return;
        }
        if (issued < chunks) issue(issued++);
        const float* W = dc_sm + (size_t)(ch % DC_STAGES) * STAGE;
        const float* G = W + 3 * DC_TOK * DIM;
        float su[OUT], o[OUT];
        F2 sw[DC_TOK][C / 2], sg[DC_TOK][C / 2];
        sums(W, sw);
        meet(sw, su);
        const int lc = group * C + my_col;
        const float* u0 = W + MAIN + lc / DC_COLS * (DC_TOK * DC_COLS) + my_tok * DC_COLS + lc % DC_COLS;
#pragma unroll
        for (int c = 0; c < OUT; c += 2) {
            const float2 x = *reinterpret_cast<const float2*>(u0 + c);
            *reinterpret_cast<float2*>(&us[group][my_tok][my_col + c]) = make_float2(x.x - su[c], x.y - su[c + 1]);
        }
        sums(W + DC_TOK * DIM, sg);
        __syncwarp();           // the lanes of a group of columns are lanes of one warp
        meet(sg, o);            // behind the hand-over of u: nothing in the update waits for it
#pragma unroll
        for (int r = 0; r < R4; ++r) {
            Four gl;
            gl.f = *reinterpret_cast<const float4*>(G + r * (4 * LANES) + part * 4);
#pragma unroll
            for (int c = 0; c < C; ++c)
#pragma unroll
                for (int e = 0; e < 2; ++e) s[c][r * 2 + e] = mul2(gl.p[e], s[c][r * 2 + e]);
        }
#pragma unroll
        for (int j4 = 0; j4 < DC_TOK / 4; ++j4) {
            const float4 bb = *reinterpret_cast<const float4*>(G + DIM + my_tok * DC_BP + j4 * 4);
            const float bj[4] = {bb.x, bb.y, bb.z, bb.w};
#pragma unroll
            for (int e4 = 0; e4 < 4; ++e4) {
                const int j = j4 * 4 + e4;
                float u[C];
                if constexpr (C == 4) {
                    *reinterpret_cast<float4*>(u) = *reinterpret_cast<const float4*>(us[group][j]);
                } else {
                    *reinterpret_cast<float2*>(u) = *reinterpret_cast<const float2*>(us[group][j]);
                }
                // B is zero for later tokens, but a later token's u may be no number, and that is not this one's affair
                if (j <= my_tok)
#pragma unroll
                    for (int c = 0; c < OUT; ++c) o[c] = __fmaf_rn(bj[e4], CB == 2 && my_col ? u[C - OUT + c] : u[c], o[c]);
#pragma unroll
                for (int r = 0; r < R4; ++r) {
                    Four kd;
                    kd.f = *reinterpret_cast<const float4*>(W + (2 * DC_TOK + j) * DIM + r * (4 * LANES) + part * 4);
#pragma unroll
                    for (int c = 0; c < C; ++c)
#pragma unroll
                        for (int e = 0; e < 2; ++e) {
                            F2 ub;
                            ub.f = make_float2(u[c], u[c]);
                            s[c][r * 2 + e] = fma2(kd.p[e], ub, s[c][r * 2 + e]);
                        }
                }
            }
        }
        const int t = ch * DC_TOK + my_tok;
        if (t < n_tok)
#pragma unroll
            for (int c = 0; c < OUT; c += 2)
                *reinterpret_cast<float2*>(a.out + ((size_t)(t0 + t) * H + h) * vdim + col + my_col + c) = make_float2(o[c], o[c + 1]);
    }
#pragma unroll
    for (int i = 0; i < R4 * 2; ++i) {
        const int r = (i >> 1) * (4 * LANES) + part * 4 + (i & 1) * 2;
#pragma unroll
        for (int c = 0; c < C; c += 2) {
            *reinterpret_cast<float2*>(S + (size_t)r * vdim + col + c) = make_float2(s[c][i].f.x, s[c + 1][i].f.x);
            *reinterpret_cast<float2*>(S + (size_t)(r + 1) * vdim + col + c) = make_float2(s[c][i].f.y, s[c + 1][i].f.y);
        }
    }
}

static bool delta_chunk_takes(int dim, int vdim, int taps) {
    return (dim == 64 || dim == 128) && vdim > 0 && vdim <= 256 && vdim % DC_COLS == 0 && taps == DC_TAPS;
}

template <typename T, int DIM>
static int delta_chunk_go(const DeltaPrepArgs& p, int nt, int B, int max_chunks, cudaStream_t s) {
    const size_t smem = (size_t)(DC_TOK * (3 * DIM + p.vdim) + DC_TOK * DC_TOK) * sizeof(float);     // at most 41 KB
    TB_LAUNCH((delta_chunk_kernel<T, DIM>), dim3(max_chunks, p.H), 256, smem, s, p, B, max_chunks);
    const int rc = tb_last_error();
    if (rc) return rc;
    const int C = 2 * p.G * p.dim + p.H * p.vdim;
    TB_LAUNCH((delta_conv_state_kernel<T>), dim3(B, (C + 255) / 256), 256, 0, s, p);
    return tb_last_error();
}

template <int DIM, int LANES, int C, bool OWN>
static int delta_chunk_scan_go(const DeltaChunkScanArgs& a, int B, cudaStream_t s) {
    constexpr int COLS = 128 / LANES * C;
    constexpr size_t smem = (size_t)DC_STAGES * ((3 * DC_TOK + 1) * DIM + DC_TOK * DC_BP + DC_TOK * COLS) * sizeof(float);
    static PerDevice raised;
    tb_allow_smem(raised, (const void*)delta_chunk_scan_kernel<DIM, LANES, C, OWN>, smem);
    // the blocks run for the whole sequence and want an SM each (see tb_launch_plain)
    tb_launch_plain(delta_chunk_scan_kernel<DIM, LANES, C, OWN>, dim3(B, a.H, a.vdim / COLS), dim3(128), smem, s, a);
    return tb_last_error();
}

static int delta_chunk_scan_entry(const float* rec, float* state, float* out, const int* seq_start, const int* slots, int nt, int B,
                                  int G, int H, int dim, int vdim, int taps, int max_chunks, bool wide, cudaStream_t s) {
    if (nt < 0 || B < 0 || G <= 0 || H <= 0 || max_chunks < 0) return TB_ERR_ARG;
    if (!delta_chunk_takes(dim, vdim, taps) || (wide && (dim != 128 || vdim % 32))) return TB_ERR_UNSUPPORTED;
    if (((uintptr_t)rec & 15) || (((uintptr_t)state | (uintptr_t)out) & 7)) return TB_ERR_ARG;
    if (nt == 0 || B == 0) return 0;
    if (max_chunks < nt / DC_TOK + (B < nt ? B : nt)) return TB_ERR_ARG;
    const long long per = (long long)H * dim * vdim + (taps - 1) * (2LL * G * dim + H * vdim);
    if (per % 2) return TB_ERR_ARG;
    DeltaChunkScanArgs a{rec, state, tc_error_ptr(), out, seq_start, slots, per, max_chunks, H, vdim};
    if (!a.error) return tb_last_error();
    if (wide) return delta_chunk_scan_go<128, 16, 4, true>(a, B, s);
    return dim == 64 ? delta_chunk_scan_go<64, 16, 2, false>(a, B, s) : delta_chunk_scan_go<128, 32, 4, false>(a, B, s);
}

extern "C" {
// Floats of one (head, chunk) record, or 0 where these kernels do not take such heads.
int tb_delta_chunk_record_size(int dim, int vdim, int taps) {
    return delta_chunk_takes(dim, vdim, taps) ? dc_record(dim, vdim) : 0;
}
int tb_delta_chunk_tokens() { return DC_TOK; }

// z's rows, the convolution's weights and the state's start on the boundaries of the loads above, or TB_ERR_ARG.
#define TB_DELTA_CHUNK(SFX, T)                                                                                        \
    int tb_delta_chunk_##SFX(const void* z, int ldz, const float* wconv, float* state, const float* a,                \
                             const float* dt_bias, const float* A_log, const float* bz, float* rec,                   \
                             const int* seq_start, const int* slots, int nt, int B, int G, int H, int dim, int vdim,  \
                             int taps, int max_chunks, int lda, int ldb, int head_decay, cudaStream_t s) {            \
        if (nt < 0 || B < 0 || G <= 0 || H <= 0 || H % G || max_chunks < 0) return TB_ERR_ARG;                        \
        if (!delta_chunk_takes(dim, vdim, taps)) return TB_ERR_UNSUPPORTED;                                           \
        if (lda < (head_decay ? H : H * dim) || ldb < H || ldz % 2 || ((uintptr_t)z % (2 * sizeof(T))) ||             \
            (((uintptr_t)wconv | (uintptr_t)rec) & 15))                                                               \
            return TB_ERR_ARG;                                                                                        \
        if (nt == 0 || B == 0) return 0;                                                                              \
        if (max_chunks < nt / DC_TOK + (B < nt ? B : nt)) return TB_ERR_ARG;                                          \
        const long long conv = (long long)H * dim * vdim, per = conv + (taps - 1) * (2LL * G * dim + H * vdim);       \
        DeltaPrepArgs p{z, wconv, state, a, dt_bias, A_log, bz, rec, nullptr, nullptr, seq_start, slots, per, conv,   \
                        ldz, G, H, dim, vdim, taps, 0, lda, ldb, head_decay ? 1 : 0};                                 \
        return dim == 64 ? delta_chunk_go<T, 64>(p, nt, B, max_chunks, s)                                             \
                         : delta_chunk_go<T, 128>(p, nt, B, max_chunks, s);                                           \
    }
TB_DELTA_CHUNK(f32, float)
TB_DELTA_CHUNK(bf16, __nv_bfloat16)

int tb_delta_chunk_scan(const float* rec, float* state, float* out, const int* seq_start, const int* slots, int nt, int B,
                        int G, int H, int dim, int vdim, int taps, int max_chunks, cudaStream_t s) {
    return delta_chunk_scan_entry(rec, state, out, seq_start, slots, nt, B, G, H, dim, vdim, taps, max_chunks, false, s);
}
// The same, to the bit, with 32 columns a block (see wide_scan_pays in parts/channel_delta.py); heads of 128, vdim a multiple of 32.
int tb_delta_chunk_scan_wide(const float* rec, float* state, float* out, const int* seq_start, const int* slots, int nt, int B,
                             int G, int H, int dim, int vdim, int taps, int max_chunks, cudaStream_t s) {
    return delta_chunk_scan_entry(rec, state, out, seq_start, slots, nt, B, G, H, dim, vdim, taps, max_chunks, true, s);
}
}

#include "tape.h"
TB_TAPE_REGISTER(tb_delta_chunk_f32)
TB_TAPE_REGISTER(tb_delta_chunk_bf16)
TB_TAPE_REGISTER(tb_delta_chunk_scan)
TB_TAPE_REGISTER(tb_delta_chunk_scan_wide)

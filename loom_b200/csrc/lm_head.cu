// lm_head.cu -- the fp32 tied LM head as a streaming kernel: logits[v] = float(sum_d float64(h_d) * float64(W_vd)) over the
// final-normalised hidden row (applyFP32LMHeadRows, poly/transformer.go:659-719; final RMSNorm poly/norm.go:102-138),
// with the greedy step folded into its tail (poly/sampling.go:45-55, poly/transformer.go:434-485).
//
// The head is 63 % of the bytes of a BitNet-2B decode step (1.31 GB), so this kernel is a pure HBM stream: one CTA per
// SM, every warp owns a contiguous range of vocabulary rows and pulls them through a private two-stage shared-memory
// ring with one bulk async copy (TMA engine) per row, first two rows requested before the dependency wait.  The
// normalised hidden row sits in shared memory as float64 in the order the lanes read it (conflict-free 16-byte loads).
// The CTA that finishes last reduces the per-CTA maxima to the next token, appends it to the output ring, advances the
// position and gathers the token's embedding row for the next step: no argmax, position or embedding launch.
#include "glue.cuh"
#include "tp_xchg.cuh"

namespace {

// floats from one hidden row to the next in shared memory: 64 bytes off a multiple of 128, so that the eight lanes of a phase (two rows
// x four chunks) meet no bank twice
__host__ __device__ constexpr int head_row_stride(int H) { return ((H + 31) & ~31) + 16; }
constexpr int kHeadMaxRows = 8;  // hidden rows (independent sequences) one pass of the table serves at most

__device__ __forceinline__ void argmax_merge(float& best, int& idx, float ov, int oi) {
    if (ov > best || (ov == best && oi < idx)) {
        best = ov;
        idx = oi;
    }
}

// The greedy step, once per hidden row: sv / si hold `ways` partial (maximum, index) pairs of this CTA per row.  The CTA that
// arrives last reduces every CTA's pair, publishes the tokens and advances the sequences.  All threads call it.
__device__ __forceinline__ void greedy_tail(const LbLmHeadParams& p, int nb, const float* sv, const int* si, int ways) {
    __shared__ int s_last, s_tok;
    const int H = p.hidden, tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, T = blockDim.x;
    __syncthreads();
    if (tid < nb) {
        float bv = sv[tid * ways];
        int bi = si[tid * ways];
        for (int w = 1; w < ways; ++w) argmax_merge(bv, bi, sv[tid * ways + w], si[tid * ways + w]);
        p.part_val[(size_t)tid * gridDim.x + blockIdx.x] = bv;
        p.part_idx[(size_t)tid * gridDim.x + blockIdx.x] = bi;
    }
    __syncthreads();
    if (tid == 0) {
        __threadfence();
        const unsigned old = atomicAdd(p.cnt, 1u);
        s_last = old + 1 == gridDim.x;
    }
    __syncthreads();
    if (!s_last) return;
    __threadfence();
    if (warp < nb) {  // warp b reduces row b
        const int b = warp;
        float bv = -INFINITY;
        int bi = 0x7fffffff;
        for (int i = lane; i < (int)gridDim.x; i += 32) argmax_merge(bv, bi, __ldcg(p.part_val + (size_t)b * gridDim.x + i), __ldcg(p.part_idx + (size_t)b * gridDim.x + i));
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            const float ov = __shfl_xor_sync(0xffffffffu, bv, o);
            const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
            argmax_merge(bv, bi, ov, oi);
        }
        if (lane == 0 && p.xchg_peers) {
            // every rank's (maximum, index) of row b to every other rank, then the merge in rank order
            const uint32_t seq = p.xchg_ctr[5];
            const size_t half = (size_t)(seq & 1);
            const int W = p.xchg_world, me = p.xchg_rank;
            const float mv = bv;
            const int mi = bi == 0x7fffffff ? bi : bi + p.vocab_offset;
            for (int q = 0; q < W; ++q) {
                if (q == me) continue;
                char* dst = (char*)p.xchg_peers[q] + kXRegionD + (((half * kXMaxRanks + me) * 8 + b) * 2) * 8;
                ll_store(dst, __float_as_uint(mv), seq);
                ll_store(dst + 8, (uint32_t)mi, seq);
            }
            bv = -INFINITY;
            bi = 0x7fffffff;
            bool ok = true;
            for (int q = 0; q < W; ++q) {
                uint32_t dv = __float_as_uint(mv), di = (uint32_t)mi;
                if (q != me) {
                    const char* src = (const char*)p.xchg_peers[me] + kXRegionD + (((half * kXMaxRanks + q) * 8 + b) * 2) * 8;
                    ok = ll_wait(src, seq, &dv) && ok;
                    ok = ll_wait(src + 8, seq, &di) && ok;
                }
                argmax_merge(bv, bi, __uint_as_float(dv), (int)di);
            }
            if (!ok) atomicExch(p.status, 5);
        }
        if (lane == 0) {
            if (bi == 0x7fffffff) bi = 0;  // only NaNs: the reference keeps index 0
            if (b == 0) s_tok = bi;
            p.tok_out[b] = bi;
            if (p.out_tokens && p.step) {
                const int s = p.step[b];
                if (s < p.out_cap) p.out_tokens[(size_t)b * p.out_tokens_stride + s] = bi;
                p.step[b] = s + 1;
            }
            if (p.pos) p.pos[b] += p.pos_delta;
        }
    }
    __syncthreads();
    if (tid == 0) {
        *p.cnt = 0;
        if (p.xchg_peers) p.xchg_ctr[5] += 1;  // every warp of this CTA has read the old value (barrier above)
    }
    if (p.x_next && p.emb) {  // the embedding row of the new token, for the step that follows (poly/transformer.go:551-577)
        const int t = s_tok;
        const bool ok = t >= 0 && t < p.emb_vocab;
        const float* src = p.emb + (size_t)(ok ? t : 0) * H;
        for (int i = tid; i < H; i += T) p.x_next[i] = ok ? src[i] : 0.0f;
    }
}

template <int NW>
__global__ void __launch_bounds__(NW * 32, 1) lb_lm_head_stream_kernel(const LbLmHeadParams p) {
    extern __shared__ __align__(128) uint8_t smem_raw[];
    __shared__ double red[32];
    __shared__ float sv[NW];
    __shared__ int si[NW];
    constexpr int T = NW * 32;
    const int H = p.hidden, H4 = H >> 2, tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int kiter = (H4 + 31) >> 5;                       // float4 columns per lane
    double* sh = reinterpret_cast<double*>(smem_raw);      // [kiter][2][32][2] doubles: the row in lane order, zero padded
    const size_t sh_bytes = (size_t)kiter * 128 * sizeof(double);
    float* ring = reinterpret_cast<float*>(smem_raw + sh_bytes) + (size_t)warp * 2 * H;  // this warp's two stages of one row
    uint64_t* bars = reinterpret_cast<uint64_t*>(smem_raw + sh_bytes + (size_t)NW * 2 * H * sizeof(float)) + warp * 2;
    // rows of this CTA and of this warp: contiguous slices
    const int r0 = (int)((long long)p.vocab * blockIdx.x / gridDim.x), r1 = (int)((long long)p.vocab * (blockIdx.x + 1) / gridDim.x);
    const int w0 = r0 + (r1 - r0) * warp / NW, w1 = r0 + (r1 - r0) * (warp + 1) / NW;
    const uint32_t row_bytes = (uint32_t)H * 4;
    const uint64_t stream_policy = lb_policy_evict_first();  // 1.3 GB read once per token: do not let it own the L2
    if (lane == 0) {
        lb_mbar_init(&bars[0], 1);
        lb_mbar_init(&bars[1], 1);
        lb_fence_mbar_init();
    }
    __syncwarp();
    lb_pdl_launch_dependents();
    // the head is a weight: its first rows are requested while the last block is still running
    if (lane == 0) {
        for (int s = 0; s < 2 && w0 + s < w1; ++s) {
            lb_mbar_expect_tx(&bars[s], row_bytes);
            lb_bulk_g2s_stream(ring + (size_t)s * H, p.head + (size_t)(w0 + s) * H, row_bytes, &bars[s], stream_policy);
        }
    }
    lb_pdl_wait();
    lb_trace(p.trace, 2);
    // final RMSNorm of the hidden row (float64 like the reference), rounded to float32 and kept as float64
    double ss = 0.0;
    for (int i = tid; i < H; i += T) {
        const double v = (double)p.x[i];
        ss = __dadd_rn(ss, __dmul_rn(v, v));
    }
    ss = lb_warp_sum(ss);
    if (lane == 0) red[warp] = ss;
    __syncthreads();
    ss = 0.0;
    for (int i = 0; i < NW; ++i) ss += red[i];
    const double rms = sqrt(__dadd_rn(__ddiv_rn(ss, (double)H), p.eps));
    const double rrms = __ddiv_rn(1.0, rms);
    for (int i = tid; i < kiter * 128; i += T) {
        // slot i holds column 4 * (k * 32 + l) + 2 * half + j
        const int j = i & 1, l = (i >> 1) & 31, half = (i >> 6) & 1, k = i >> 7;
        const int col = 4 * (k * 32 + l) + 2 * half + j;
        double y = 0.0;
        if (col < H) {
            const double g = p.gain ? (double)p.gain[col] : 1.0;
            const float yf = (float)__dmul_rn(lb_div_by((double)p.x[col], rms, rrms), g);
            y = (double)yf;
            if (blockIdx.x == 0 && p.hidden_out) p.hidden_out[col] = yf;
        }
        sh[i] = y;
    }
    __syncthreads();
    lb_trace(p.trace, 3);

    float best = -INFINITY;
    int bidx = 0x7fffffff;
    bool failed = false;
    for (int r = w0; r < w1; ++r) {
        const int st = (r - w0) & 1;
        const uint32_t parity = (uint32_t)(((r - w0) >> 1) & 1);
        if (!failed && !lb_mbar_wait_bounded(&bars[st], parity)) {
            failed = true;
            if (lane == 0) atomicExch(p.status, 1);
        }
        const float4* row = reinterpret_cast<const float4*>(ring + (size_t)st * H);
        double a[4] = {0.0, 0.0, 0.0, 0.0};
        if (!failed) {
#pragma unroll 2
            for (int k = 0; k < kiter; ++k) {
                const int c4 = k * 32 + lane;
                float4 w = make_float4(0.f, 0.f, 0.f, 0.f);
                if (c4 < H4) w = row[c4];
                const double2 s01 = *reinterpret_cast<const double2*>(sh + ((size_t)(k * 2 + 0) * 32 + lane) * 2);
                const double2 s23 = *reinterpret_cast<const double2*>(sh + ((size_t)(k * 2 + 1) * 32 + lane) * 2);
                a[0] = fma((double)w.x, s01.x, a[0]);
                a[1] = fma((double)w.y, s01.y, a[1]);
                a[2] = fma((double)w.z, s23.x, a[2]);
                a[3] = fma((double)w.w, s23.y, a[3]);
            }
        }
        __syncwarp();
        if (lane == 0 && r + 2 < w1) {  // the stage is free again: request the row after next
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            lb_mbar_expect_tx(&bars[st], row_bytes);
            lb_bulk_g2s_stream(ring + (size_t)st * H, p.head + (size_t)(r + 2) * H, row_bytes, &bars[st], stream_policy);
        }
        const float lg = (float)lb_warp_sum((a[0] + a[1]) + (a[2] + a[3]));
        if (lane == 0) p.logits[r] = lg;
        argmax_merge(best, bidx, lg, r);  // rows ascend: a later equal value never replaces an earlier one
    }
    lb_trace(p.trace, 4);
    if (!p.tok_out) return;

    if (lane == 0) {
        sv[warp] = best;
        si[warp] = bidx;
    }
    greedy_tail(p, 1, sv, si, NW);
    lb_trace(p.trace, 5);
}

// ---- several hidden rows (independent sequences) per pass over the table ----
//
// A pass of up to eight rows is a product of the table with an [H, 8] matrix in float64: eight table rows x four columns against
// four columns x eight hidden rows is one m8n8k4 MMA.  A warp holds 32 table rows (four MMA tiles) so that a hidden value is
// converted to float64 once per 32 rows; lane (g, t) takes 16 bytes of row g, columns 4t.. of a 16-column step, for the table
// (global memory, straight into registers, three steps ahead) and for the hidden rows (shared memory, float32: they are float32
// values by definition) alike, so which column an MMA calls its k-th is the same for both and needs no shuffle.  Four warps share
// a strip of 32 rows by columns and add up in shared memory: 867 rows of a CTA's share are 28 strips for four groups.
// Bound: the table's way from HBM.  A load takes 64 bytes each of eight rows 16 KB apart, and DRAM pays for every page it opens for so
// little; so a load asks L2 for the 256 bytes around it.  128256 rows x 4096 columns, eight hidden rows, us: without that 500 (606 with
// the MMAs left out, 274 with the loads left out: the MMAs are 240), with it 446, three steps ahead instead of two 432; fewer rows and more
// columns of each a step 570 to 670, explicit prefetches of 256 to 1024 bytes a row 505 to 657, CTAs that start at different columns 530.
// HBM alone would be 300.  (Conversions to float64 run beside the MMAs.)
constexpr int kHmWarps = 16, kHmSplit = 4, kHmGroups = kHmWarps / kHmSplit, kHmTiles = 4, kHmRows = 8 * kHmTiles;

__device__ __forceinline__ float4 ldg_table(const float* p, uint64_t policy) {
    float4 v;
    asm volatile("ld.global.nc.L1::no_allocate.L2::cache_hint.L2::256B.v4.f32 {%0,%1,%2,%3}, [%4], %5;" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "l"(p), "l"(policy));
    return v;
}

__global__ void __launch_bounds__(kHmWarps * 32, 1) lb_lm_head_rows_kernel(const LbLmHeadParams p) {
    extern __shared__ __align__(128) uint8_t smem_raw[];
    __shared__ double s_ss[kHmWarps];
    __shared__ float sv[kHeadMaxRows * kHmGroups];
    __shared__ int si[kHeadMaxRows * kHmGroups];
    const int H = p.hidden, nb = p.nb, tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3;
    const int group = warp / kHmSplit, part = warp % kHmSplit;
    const int ld = head_row_stride(H);
    float* sh = reinterpret_cast<float*>(smem_raw);                                                   // [nb][ld] normalised rows
    double* sums = reinterpret_cast<double*>(smem_raw + (size_t)nb * ld * sizeof(float)) + (size_t)group * kHmSplit * kHmRows * 8;  // [part][token][row]
    const int r0 = (int)((long long)p.vocab * blockIdx.x / gridDim.x), r1 = (int)((long long)p.vocab * (blockIdx.x + 1) / gridDim.x);
    const int steps = (H + 15) >> 4, k0 = steps * part / kHmSplit, k1 = steps * (part + 1) / kHmSplit;
    const uint64_t policy = lb_policy_evict_first();
    // rows beyond the share are read as its last row, columns beyond H as zeros
    auto fetch = [&](float4 (&w)[kHmTiles], int row, int k) {
        const int col = 16 * k + 4 * t;
#pragma unroll
        for (int i = 0; i < kHmTiles; ++i) {
            const int r = row + 8 * i + g;
            w[i] = col < H ? ldg_table(p.head + (size_t)(r < r1 ? r : r1 - 1) * H + col, policy) : make_float4(0.f, 0.f, 0.f, 0.f);
        }
    };
    constexpr int kAhead = 3;
    float4 ring[kAhead][kHmTiles];
    lb_pdl_launch_dependents();
    int row = r0 + group * kHmRows;
    if (row < r1)
#pragma unroll
        for (int a = 0; a < kAhead; ++a)
            if (k0 + a < k1) fetch(ring[a], row, k0 + a);
    lb_pdl_wait();
    lb_trace(p.trace, 2);
    // final RMSNorm (float64 like the reference, rounded to float32): two warps per row
    {
        const int b = warp >> 1, lt = (warp & 1) * 32 + lane;
        const float* xb = p.x + (size_t)(b < nb ? b : 0) * p.x_stride;
        double ss = 0.0;
        if (b < nb)
            for (int i = lt; i < H; i += 64) {
                const double v = (double)xb[i];
                ss = __dadd_rn(ss, __dmul_rn(v, v));
            }
        ss = lb_warp_sum(ss);
        if (lane == 0) s_ss[warp] = ss;
        __syncthreads();
        if (b < nb) {
            const double rms = sqrt(__dadd_rn(__ddiv_rn(s_ss[warp & ~1] + s_ss[warp | 1], (double)H), p.eps));
            const double rrms = __ddiv_rn(1.0, rms);
            for (int i = lt; i < H; i += 64) {
                const double gn = p.gain ? (double)p.gain[i] : 1.0;
                const float yf = (float)__dmul_rn(lb_div_by((double)xb[i], rms, rrms), gn);
                sh[(size_t)b * ld + i] = yf;
                if (b == 0 && blockIdx.x == 0 && p.hidden_out) p.hidden_out[i] = yf;
            }
        }
        __syncthreads();
    }
    lb_trace(p.trace, 3);
    float best[2] = {-INFINITY, -INFINITY};  // rows of tokens part and part + 4, over the rows this lane finishes
    int bidx[2] = {0x7fffffff, 0x7fffffff};
    for (; row < r1; row += kHmGroups * kHmRows) {
        double c[kHmTiles][2];
#pragma unroll
        for (int i = 0; i < kHmTiles; ++i) c[i][0] = c[i][1] = 0.0;
        const int next = row + kHmGroups * kHmRows;
        for (int k = k0; k < k1; k += kAhead) {
#pragma unroll
            for (int a = 0; a < kAhead; ++a) {
                if (k + a >= k1) break;
                float4 w[kHmTiles];
#pragma unroll
                for (int i = 0; i < kHmTiles; ++i) w[i] = ring[a][i];
                if (k + a + kAhead < k1) fetch(ring[a], row, k + a + kAhead);
                const int col = 16 * (k + a) + 4 * t;
                float4 h = make_float4(0.f, 0.f, 0.f, 0.f);
                if (g < nb && col < H) h = *reinterpret_cast<const float4*>(sh + (size_t)g * ld + col);
                const double h0 = (double)h.x, h1 = (double)h.y, h2 = (double)h.z, h3 = (double)h.w;
#pragma unroll
                for (int i = 0; i < kHmTiles; ++i) lb_dmma_884(c[i], (double)w[i].x, h0);
#pragma unroll
                for (int i = 0; i < kHmTiles; ++i) lb_dmma_884(c[i], (double)w[i].y, h1);
#pragma unroll
                for (int i = 0; i < kHmTiles; ++i) lb_dmma_884(c[i], (double)w[i].z, h2);
#pragma unroll
                for (int i = 0; i < kHmTiles; ++i) lb_dmma_884(c[i], (double)w[i].w, h3);
            }
        }
        if (next < r1)  // the next strip's first steps travel while the sums meet
#pragma unroll
            for (int a = 0; a < kAhead; ++a)
                if (k0 + a < k1) fetch(ring[a], next, k0 + a);
#pragma unroll
        for (int i = 0; i < kHmTiles; ++i) {
            sums[(part * 8 + 2 * t) * kHmRows + 8 * i + g] = c[i][0];
            sums[(part * 8 + 2 * t + 1) * kHmRows + 8 * i + g] = c[i][1];
        }
        asm volatile("bar.sync %0, %1;" ::"r"(1 + group), "r"(kHmSplit * 32) : "memory");
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int b = part + 4 * h, r = row + lane;
            double v = 0.0;
#pragma unroll
            for (int q = 0; q < kHmSplit; ++q) v += sums[(q * 8 + b) * kHmRows + lane];
            if (b < nb && r < r1) {
                const float lg = (float)v;
                p.logits[(size_t)b * p.logits_stride + r] = lg;
                argmax_merge(best[h], bidx[h], lg, r);  // rows ascend
            }
        }
        asm volatile("bar.sync %0, %1;" ::"r"(1 + group), "r"(kHmSplit * 32) : "memory");  // the sums are read
    }
    lb_trace(p.trace, 4);
    if (!p.tok_out) return;
#pragma unroll
    for (int h = 0; h < 2; ++h) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            const float ov = __shfl_xor_sync(0xffffffffu, best[h], o);
            const int oi = __shfl_xor_sync(0xffffffffu, bidx[h], o);
            argmax_merge(best[h], bidx[h], ov, oi);
        }
        if (lane == 0) {
            sv[(part + 4 * h) * kHmGroups + group] = best[h];
            si[(part + 4 * h) * kHmGroups + group] = bidx[h];
        }
    }
    greedy_tail(p, nb, sv, si, kHmGroups);
    lb_trace(p.trace, 5);
}

constexpr size_t kHeadSmem = 220 * 1024;

template <int NW>
size_t head_smem(int H) {
    const int kiter = ((H >> 2) + 31) >> 5;
    return (size_t)kiter * 128 * sizeof(double) + (size_t)NW * 2 * H * sizeof(float) + (size_t)NW * 2 * sizeof(uint64_t);
}
size_t head_rows_smem(int H, int nb) { return (size_t)nb * head_row_stride(H) * sizeof(float) + (size_t)kHmWarps * kHmRows * 8 * sizeof(double); }

int launch_head(loom_b200_ctx* ctx, void (*kern)(LbLmHeadParams), int threads, size_t smem, int grid, const LbLmHeadParams& p, unsigned attr_bit) {
    if (!(ctx->func_attr_mask2 & attr_bit)) {
        LB_CUDA(ctx, cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kHeadSmem));
        ctx->func_attr_mask2 |= attr_bit;
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(grid < 1 ? 1 : grid > ctx->sm_count ? ctx->sm_count : grid);
    cfg.blockDim = dim3(threads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = ctx->stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = ctx->opt_pdl ? 1 : 0;
    LB_CUDA(ctx, cudaLaunchKernelEx(&cfg, kern, p));
    ctx->launches++;
    return 0;
}

}  // namespace

int lb_launch_lm_head_legacy(loom_b200_ctx* ctx, const LbLmHeadParams& p);

bool lb_lm_head_streams(const loom_b200_ctx* ctx, const float* head, int hidden) {
    return ctx->opt_head_stream && (hidden & 3) == 0 && (((uintptr_t)head) & 15) == 0 && head_smem<4>(hidden) <= kHeadSmem;
}

int lb_launch_lm_head(loom_b200_ctx* ctx, const LbLmHeadParams& pin) {
    LbLmHeadParams p = pin;
    p.status = ctx->status_dev;
    if (!lb_lm_head_streams(ctx, p.head, p.hidden)) {
        if (p.tok_out) return lb_fail(ctx, LOOM_B200_ERR_UNSUPPORTED, "lm_head: the greedy tail needs the streaming kernel (hidden %d)", p.hidden);
        return lb_launch_lm_head_legacy(ctx, p);
    }
    if (p.nb < 1) p.nb = 1;
    if (p.nb > kHeadMaxRows) return lb_fail(ctx, LOOM_B200_ERR_INVALID, "lm_head: %d hidden rows in one pass (at most %d)", p.nb, kHeadMaxRows);
    if (p.tok_out) {
        if (!ctx->head_scratch) {
            if (ctx->capturing) return lb_fail(ctx, LOOM_B200_ERR_INVALID, "lm_head scratch would be allocated while recording a graph");
            const size_t bytes = (size_t)kHeadMaxRows * ctx->sm_count * 8 + 64;
            LB_CUDA(ctx, cudaMalloc(&ctx->head_scratch, bytes));
            LB_CUDA(ctx, cudaMemsetAsync(ctx->head_scratch, 0, bytes, ctx->stream));
        }
        p.part_val = reinterpret_cast<float*>(ctx->head_scratch);
        p.part_idx = reinterpret_cast<int*>(p.part_val + (size_t)kHeadMaxRows * ctx->sm_count);
        p.cnt = reinterpret_cast<unsigned int*>(p.part_idx + (size_t)kHeadMaxRows * ctx->sm_count);
    }
    p.trace = lb_trace_row(ctx, "lm_head");
    if (p.nb > 1) return launch_head(ctx, lb_lm_head_rows_kernel, kHmWarps * 32, head_rows_smem(p.hidden, p.nb), p.vocab / kHmRows, p, 1u << 10);
    if (head_smem<8>(p.hidden) <= kHeadSmem) return launch_head(ctx, lb_lm_head_stream_kernel<8>, 256, head_smem<8>(p.hidden), p.vocab / 8, p, 1u << 8);
    return launch_head(ctx, lb_lm_head_stream_kernel<4>, 128, head_smem<4>(p.hidden), p.vocab / 4, p, 1u << 9);
}

int lb_lm_head_rows_per_pass(const loom_b200_ctx* ctx, const float* head, int hidden) {
    return lb_lm_head_streams(ctx, head, hidden) ? kHeadMaxRows : 0;  // (the rings of one row end below 5632 columns; eight rows fit there)
}

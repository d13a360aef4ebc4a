// gemm_bf16.cu -- token-block GEMM of bf16 matrices on the 5th-generation tensor cores (tcgen05, kind::f16).
//
//   D[128 tokens, N rows] (float, TMEM) += X[128 tokens, 64] (bf16, shared) * W[N rows, 64]^T (bf16, shared)
//
// The same machine as the persistent int8 GEMM (gemm_ternary_i8.cu): both operands are stored in HBM as the shared-memory
// image the tensor core reads (dense.cuh), two threads bring one K slice of 64 columns per pipeline stage with bulk
// copies, one issues four K = 16 MMAs per slice, tensor memory holds two accumulator buffers and eight
// epilogue warps drain tile i while tile i + 1 accumulates.  Tokens are the M side, so a thread of the epilogue owns a
// token and eight consecutive output columns of it are one 16-byte chunk of the next product's input image.
// N, a tile's columns, is any multiple of 16 up to 256 (gate and up side by side: up to 128 of each): plan() takes what makes the
// busiest CTA finish first.  One accumulator takes all of K, so that an output's bits depend on its row of X and its row of W alone.
// Routed experts: the token blocks of the image
// are grouped by expert and a table names each block's expert; the number of blocks in use is read on the device.
// Every mbarrier wait is bounded; on expiry the kernel raises the context's status word, frees its tensor memory and returns.
#include "dense.cuh"
#include "umma.cuh"

namespace {

constexpr int kEpiThreads = 256;
constexpr int kMmaWarp = kEpiThreads / 32, kRowsWarp = kMmaWarp + 1, kWeightsWarp = kMmaWarp + 2;
constexpr int kThreads = kEpiThreads + 96;
constexpr int kRing = 200 * 1024, kMaxStages = 8;
constexpr size_t kSmem = kRing + 1024;

struct Plan {
    int n, row_tiles;  // columns of a tile (of each matrix), tiles over the rows of W
};
__host__ __device__ __forceinline__ int stage_bytes(int cols) { return kImgBlock + cols * 128; }  // cols: of both matrices

// RESID: sixteen columns of a token's residual row from column r on
__device__ __forceinline__ void load_residual(const LbDenseGemm& p, int tok, int r, float4 (&x)[4]) {
    const float4* o = reinterpret_cast<const float4*>(p.out + (size_t)tok * p.ldo + r);
    if (r < p.ldo) {
        x[0] = o[0];
        x[1] = o[1];
    }
    if (r + 8 < p.ldo) {
        x[2] = o[2];
        x[3] = o[3];
    }
}

// eight consecutive columns of a token from column r on: v8 of the first matrix, u8 of the second; RESID: res, the residual's
template <int EPI>
__device__ __forceinline__ void emit8(const LbDenseGemm& p, int tok, int r, const float* v8, const float* u8, const float4* res) {
    if (EPI == LB_DEPI_F32 || EPI == LB_DEPI_RESID) {
        if (r >= p.ldo) return;
        float4* o = reinterpret_cast<float4*>(p.out + (size_t)tok * p.ldo + r);
        if (EPI == LB_DEPI_F32) {
            o[0] = make_float4(v8[0], v8[1], v8[2], v8[3]);
            o[1] = make_float4(v8[4], v8[5], v8[6], v8[7]);
        } else {
            float4 x = res[0], y = res[1];
            x.x = fmaf(p.mult, v8[0], p.res_mult * x.x);
            x.y = fmaf(p.mult, v8[1], p.res_mult * x.y);
            x.z = fmaf(p.mult, v8[2], p.res_mult * x.z);
            x.w = fmaf(p.mult, v8[3], p.res_mult * x.w);
            y.x = fmaf(p.mult, v8[4], p.res_mult * y.x);
            y.y = fmaf(p.mult, v8[5], p.res_mult * y.y);
            y.z = fmaf(p.mult, v8[6], p.res_mult * y.z);
            y.w = fmaf(p.mult, v8[7], p.res_mult * y.w);
            o[0] = x;
            o[1] = y;
        }
        return;
    }
    if (EPI == LB_DEPI_HEADS ? r >= p.rows : r / 64 >= p.img_slices) return;
    float f[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) {
        f[j] = v8[j];
        if (EPI == LB_DEPI_GELU) f[j] = lb_gelu_erff(v8[j]);
        if (EPI == LB_DEPI_GLU) f[j] = lb_clamped_glu(v8[j], u8[j], p.limit);
        if (EPI == LB_DEPI_SILU) f[j] = lb_siluf(v8[j]) * u8[j];
    }
    if (EPI == LB_DEPI_HEADS)
        *reinterpret_cast<uint4*>(p.img + lb_heads_chunk(tok, r, p.heads, p.head_dim, p.head_chunks)) = lb_pack_chunk<__nv_bfloat16>(f);
    else
        lb_img_store8<__nv_bfloat16>(p.img, tok, r, p.img_slices, f);
}

template <int EPI>
__global__ void __launch_bounds__(kThreads, 1) lb_gemm_bf16_kernel(const LbDenseGemm p, const Plan plan) {
    constexpr bool kDual = EPI == LB_DEPI_GLU || EPI == LB_DEPI_SILU;
    extern __shared__ __align__(1024) uint8_t smem[];
    __shared__ __align__(8) uint64_t load_bar[kMaxStages], empty_bar[kMaxStages], acc_full[2], acc_empty[2];
    __shared__ uint32_t tmem_base_s;
    __shared__ int s_failed;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int n = plan.n, cols = kDual ? 2 * n : n, row_tiles = plan.row_tiles;
    const int stage = stage_bytes(cols), stages = kRing / stage < kMaxStages ? kRing / stage : kMaxStages;
    const int padded_rows = lb_round_up(p.rows, kImgRows);

    if (tid == 0) {
        for (int s = 0; s < stages; ++s) {
            lb_mbar_init(&load_bar[s], 2);
            lb_mbar_init(&empty_bar[s], 1);
        }
        for (int b = 0; b < 2; ++b) {
            lb_mbar_init(&acc_full[b], 1);
            lb_mbar_init(&acc_empty[b], kEpiThreads / 32);
        }
        lb_fence_mbar_init();
        s_failed = 0;
    }
    if (warp == kMmaWarp) lb_tmem_alloc(&tmem_base_s, 512);
    lb_tc_fence_before();
    __syncthreads();
    lb_tc_fence_after();
    const uint32_t tmem_base = tmem_base_s;
    lb_pdl_launch_dependents();
    lb_pdl_wait();
    const int nblocks = p.nblocks ? *p.nblocks : lb_ceil_div(p.tokens, kImgRows);
    const int ntiles = nblocks * row_tiles;
    const int first_tile = (int)blockIdx.x, tile_step = (int)gridDim.x;
    const int my_tiles = first_tile < ntiles ? (ntiles - first_tile + tile_step - 1) / tile_step : 0;

    if (warp == kRowsWarp || warp == kWeightsWarp) {
        if (lb_elect()) {
            bool failed = false;
            int s = 0;
            uint32_t parity = 1;  // (the first round's waits are over at once)
            for (int i = 0; i < my_tiles && !failed; ++i) {
                const int t = first_tile + i * tile_step, rt = t % row_tiles, tb = t / row_tiles;
                const uint8_t* xb = p.x + (size_t)tb * p.slices * kImgBlock;
                // the tile's rows of W: pieces of up to three blocks of 128
                const size_t goff = p.block_group ? (size_t)p.block_group[tb] * p.group_bytes : 0;
                const int r0 = rt * n, rows = padded_rows - r0 < n ? padded_rows - r0 : n;
                for (int ks = 0; ks < p.slices; ++ks) {
                    if (!lb_mbar_wait_bounded(&empty_bar[s], parity, kTcWaitLimit)) {
                        failed = true;
                        break;
                    }
                    uint8_t* st = smem + (size_t)s * stage;
                    if (warp == kRowsWarp) {
                        lb_mbar_expect_tx(&load_bar[s], kImgBlock);
                        lb_bulk_g2s(st, xb, kImgBlock, &load_bar[s]);
                        xb += kImgBlock;
                    } else {
                        lb_mbar_expect_tx(&load_bar[s], (uint32_t)rows * 128 * (kDual ? 2 : 1));
                        for (int r = r0; r < r0 + rows;) {
                            const int m = (r & ~127) + 128 - r < r0 + rows - r ? (r & ~127) + 128 - r : r0 + rows - r;
                            const size_t at = goff + ((size_t)(r >> 7) * p.slices + ks) * kImgBlock + (size_t)(r & 127) * 128;
                            lb_bulk_g2s(st + kImgBlock + (r - r0) * 128, p.w + at, (uint32_t)m * 128, &load_bar[s]);
                            if (kDual) lb_bulk_g2s(st + kImgBlock + (n + r - r0) * 128, p.w2 + at, (uint32_t)m * 128, &load_bar[s]);
                            r += m;
                        }
                    }
                    if (++s == stages) {
                        s = 0;
                        parity ^= 1;
                    }
                }
            }
            if (failed) atomicExch(&s_failed, 1);
        }
        __syncwarp();
    } else if (warp == kMmaWarp) {
        if (lb_elect()) {
            const uint32_t idesc = lb_idesc_bf16(128, cols, false);
            bool failed = false;
            int s = 0;
            uint32_t parity = 0;
            for (int i = 0; i < my_tiles && !failed; ++i) {
                const int buf = i & 1;
                if (i >= 2 && !lb_mbar_wait_bounded(&acc_empty[buf], (uint32_t)(((i >> 1) - 1) & 1), kTcWaitLimit)) {
                    failed = true;
                    break;
                }
                lb_tc_fence_after();
                const uint32_t d = tmem_base + (uint32_t)(buf * 256);
                for (int ks = 0; ks < p.slices; ++ks) {
                    if (!lb_mbar_wait_bounded(&load_bar[s], parity, kTcWaitLimit)) {
                        failed = true;
                        break;
                    }
                    lb_tc_fence_after();
                    const uint64_t a = lb_smem_desc(lb_smem_u32(smem + (size_t)s * stage), 128, 1024), b = a + (kImgBlock >> 4);
#pragma unroll
                    for (int k = 0; k < 4; ++k) lb_mma_f16(d, a + k * 16, b + k * 16, idesc, (ks > 0 || k > 0) ? 1u : 0u);
                    lb_mma_commit(&empty_bar[s]);
                    if (++s == stages) {
                        s = 0;
                        parity ^= 1;
                    }
                }
                if (!failed) lb_mma_commit(&acc_full[buf]);
            }
            if (failed) atomicExch(&s_failed, 1);
        }
        __syncwarp();
        lb_tc_fence_before();
    }
    // a warp reads the 32 TMEM lanes (= tokens) of its quarter; the two warps of a quarter take turns at sixteen columns
    const int quarter = warp & 3, half = warp >> 2;
    bool failed = false;
    if (warp < kMmaWarp) {
        for (int i = 0; i < my_tiles && !failed; ++i) {
            const int t = first_tile + i * tile_step, rt = t % row_tiles, tb = t / row_tiles, buf = i & 1;
            const int tok = tb * kImgRows + quarter * 32 + lane;
            const bool tok_ok = p.nblocks || tok < p.tokens;
            // RESID: the residual's columns are asked for sixteen ahead, the first ones and the rest's way into L2 while the sums are made (a
            // read behind every accumulator: 2048 x 2560 x 6912 in tiles of 144 took 97 us, 78 so)
            float4 next[4] = {};
            if (EPI == LB_DEPI_RESID && tok_ok) {
                load_residual(p, tok, rt * n + half * 16, next);
                for (int c = half * 32; c < n; c += 64)
                    if (rt * n + c < p.ldo) asm volatile("prefetch.global.L2 [%0];" ::"l"(p.out + (size_t)tok * p.ldo + rt * n + c));
            }
            failed = __any_sync(0xffffffffu, !lb_mbar_wait_bounded(&acc_full[buf], (uint32_t)((i >> 1) & 1), kTcWaitLimit));
            if (failed) {
                if (lane == 0) atomicExch(&s_failed, 1);
                break;
            }
            lb_tc_fence_after();
            const uint32_t tacc = tmem_base + (uint32_t)(buf * 256) + ((uint32_t)(quarter * 32) << 16);
#pragma unroll 1
            for (int c0 = half * 16; c0 < n; c0 += 32) {
                float v[16], u[16];
                float4 res[4];
                if (EPI == LB_DEPI_RESID) {
#pragma unroll
                    for (int e = 0; e < 4; ++e) res[e] = next[e];
                    if (tok_ok && c0 + 32 < n) load_residual(p, tok, rt * n + c0 + 32, next);
                }
                lb_tmem_ld16(tacc + (uint32_t)c0, v);
                if (kDual) lb_tmem_ld16(tacc + (uint32_t)(n + c0), u);
                lb_tmem_wait_ld();
                if (tok_ok)
#pragma unroll
                    for (int h = 0; h < 16; h += 8) emit8<EPI>(p, tok, rt * n + c0 + h, v + h, u + h, res + h / 4);
            }
            lb_tc_fence_before();
            __syncwarp();
            if (lane == 0) lb_mbar_arrive(&acc_empty[buf]);
        }
    }
    __syncthreads();
    if (warp == kMmaWarp) {
        lb_tc_fence_after();
        lb_tmem_dealloc(tmem_base, 512);
    }
    if (tid == 0 && s_failed) atomicExch(p.status, 3);
}

// Columns of a tile.  Measured: a slice takes 0.28 us with 32 columns (both matrices together), 0.29 with 64 and 0.31 with 128; 0.05 us more
// where tiles cross blocks of 128 rows of W and need two copies of it; with every SM at work 0.355 with 144, 0.40 with 192 and 0.46 with
// 256; an epilogue behind the last MMA 0.015 us a column.  Wide tiles leave a last wave of few of them: 2048 x 2560 x 6912 takes 96 us as
// 160 tiles of 256, 83 as 224 of 192 and 78 as 288 of 144 (100 before residual rows were asked for ahead); 2048 x 7696 x 2560 78 us with
// 256, 75 with 224, 84 with 144.  100 tokens x 2560 x 6912: 30 us with 32 columns, 31 with 64, 34 with 128, 38 with 96, 55 (two waves) with 16.
// (Few tiles split over K by the CTAs of a cluster took 25 us there, but sums of parts are other bits than one accumulator's, and a
// token's result then depends on how many others are in its block.)
Plan plan(const loom_b200_ctx* ctx, const LbDenseGemm& p, bool dual) {
    const int blocks = p.nblocks ? p.max_blocks : lb_ceil_div(p.tokens, kImgRows), most = dual ? 128 : 256, rows = lb_round_up(p.rows, kImgRows);  // (the padding's zeros too)
    Plan best = {};
    double best_us = 1e30;
    for (int n = most < rows ? most : rows; n >= 32; n -= 16) {
        const int tiles = lb_ceil_div(rows, n) * blocks, cols = dual ? 2 * n : n;
        const double slice = cols > 128 ? 0.22 + cols * 0.00094 : 0.27 + cols * 0.00035 + (kImgRows % n ? 0.05 : 0.0);
        const double us = lb_ceil_div(tiles, ctx->sm_count) * p.slices * slice + cols * 0.015;
        if (us < 0.98 * best_us) {
            best_us = us;
            best = {n, lb_ceil_div(rows, n)};
        }
    }
    return best;
}

template <int EPI>
int launch(loom_b200_ctx* ctx, const LbDenseGemm& p) {
    constexpr bool kDual = EPI == LB_DEPI_GLU || EPI == LB_DEPI_SILU;
    const Plan pl = plan(ctx, p, kDual);
    const int blocks = p.nblocks ? p.max_blocks : lb_ceil_div(p.tokens, kImgRows), tiles = pl.row_tiles * blocks;
    LB_BIG_SMEM(ctx, lb_gemm_bf16_kernel<EPI>, kSmem);
    LB_LAUNCH(ctx, lb_gemm_bf16_kernel<EPI>, dim3(tiles < ctx->sm_count ? tiles : ctx->sm_count), dim3(kThreads), kSmem, p, pl);
    return 0;
}

}  // namespace

int lb_gemm_bf16_run(loom_b200_ctx* ctx, int epi, const LbDenseGemm& p) {
    switch (epi) {
        case LB_DEPI_F32: return launch<LB_DEPI_F32>(ctx, p);
        case LB_DEPI_RESID: return launch<LB_DEPI_RESID>(ctx, p);
        case LB_DEPI_GELU: return launch<LB_DEPI_GELU>(ctx, p);
        case LB_DEPI_IMG: return launch<LB_DEPI_IMG>(ctx, p);
        case LB_DEPI_HEADS: return launch<LB_DEPI_HEADS>(ctx, p);
        case LB_DEPI_GLU: return launch<LB_DEPI_GLU>(ctx, p);
        case LB_DEPI_SILU: return launch<LB_DEPI_SILU>(ctx, p);
    }
    return lb_fail(ctx, LOOM_B200_ERR_UNSUPPORTED, "gemm_bf16: epilogue %d is not built", epi);
}

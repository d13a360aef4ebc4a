// gemv_tokens.cu -- packed ternary x int8 products of three to 24 tokens (a pass of several sequences, a short prompt, a layer call).
//
// The weights are the traffic of one token, so what counts is everything else a launch does.  The one-token kernel (gemv_ternary.cu) has
// every CTA bring all columns of its tokens into shared memory and turn their bytes: for eight rows of 14336 columns that is 115 KB a
// CTA and most of its 25 us.  Here
//   * a launch in front quantizes the rows once and stores them as the MMA's B fragments, [128 columns][half][token][16 bytes x 4], with
//     their sums: a CTA's share of columns is one bulk copy, and a lane's fragments are conflict-free 16-byte reads;
//   * the CTAs of a cluster share strips of rows by columns, so a CTA holds an eighth to all of the columns; their int32 sums meet in
//     distributed shared memory (exact in any order) and every CTA finishes a share of the outputs;
//   * up to 24 tokens go through one pass over the weights, eight per MMA.
// Bound: latencies (launch, rows, cluster) of about 5 us, then the integer MMAs.  Measured in a step of 16 sequences, 8B shape: the four
// products of a block with their quantizers 60 us, 154 in two passes of eight through the one-token kernel; 23 tokens through the layers of
// the 2B shape 76 us of kernels where three passes took 195.
#include "dense.cuh"
#include "gemv_device.cuh"
#include "layers.cuh"

namespace {

constexpr int kGtMaxTokens = kPassTokens;
constexpr int kGtRowsBytes = 32 * 1024;  // share of the rows a CTA should not exceed
constexpr int kGtSmemHalf = 112 * 1024;
size_t gt_scratch(int kblocks) { return (size_t)kblocks * kGtMaxTokens * 128 + 2 * kGtMaxTokens * 4; }  // fragments, largest values, sums

// ---- rows -> fragments --------------------------------------------------------------------------------------------------------
//
// A CTA per token.  The row stays in registers between its sum of squares, its largest value and its codes (same arithmetic per element as
// stage_row_fast); 4 neighbouring lanes hold the 16 columns of a chunk and exchange bytes.
__device__ __forceinline__ size_t gt_fragment(int kb, int half, int Mp, int token, int t) { return ((size_t)(kb * 2 + half) * Mp + token) * 64 + t * 16; }

template <int PRO, int UPT>
__global__ void __launch_bounds__(1024) lb_tokens_prepare_kernel(const LbGemvParams p, int Mp, uint8_t* __restrict__ img, float* __restrict__ amax_out, int* __restrict__ xsum_out) {
    constexpr bool f64 = PRO == LB_PRO_INNERNORM64, q8 = PRO == LB_PRO_Q8, kNorm = PRO >= LB_PRO_BLOCKNORM;
    using VT = typename std::conditional<f64, double, typename std::conditional<q8, int8_t, float>::type>::type;
    __shared__ double s_ss[32];
    __shared__ unsigned s_m;
    __shared__ int s_sum;
    const int n = blockIdx.x, tid = threadIdx.x, T = blockDim.x, lane = tid & 31, warp = tid >> 5, K = p.K, units = p.kblocks * 32;
    if (tid == 0) {
        s_m = 0u;
        s_sum = 0;
    }
    __syncthreads();
    lb_pdl_launch_dependents();
    lb_pdl_wait();
    if (n >= p.M) {  // padding token
        for (int i = tid; i < p.kblocks * 8; i += T) *reinterpret_cast<uint4*>(img + gt_fragment(i >> 3, (i >> 2) & 1, Mp, n, i & 3)) = make_uint4(0u, 0u, 0u, 0u);
        return;
    }
    const VT* row = static_cast<const VT*>(p.x) + (size_t)n * K;
    const bool vec = (((uintptr_t)row) & (q8 ? 3 : 15)) == 0, vec_w = kNorm && (((uintptr_t)p.norm_w) & 15) == 0;
    VT v[UPT][4];
    float w[kNorm ? UPT : 1][4];
#pragma unroll
    for (int u = 0; u < UPT; ++u) {
        const int c = 4 * (tid + u * T);
        if (vec && c + 4 <= K) {
            if (q8) {
                const char4 d = *reinterpret_cast<const char4*>(row + c);
                v[u][0] = (VT)d.x; v[u][1] = (VT)d.y; v[u][2] = (VT)d.z; v[u][3] = (VT)d.w;
            } else if (f64) {
                const double2 a = *reinterpret_cast<const double2*>(row + c), b = *reinterpret_cast<const double2*>(row + c + 2);
                v[u][0] = (VT)a.x; v[u][1] = (VT)a.y; v[u][2] = (VT)b.x; v[u][3] = (VT)b.y;
            } else {
                const float4 d = *reinterpret_cast<const float4*>(row + c);
                v[u][0] = (VT)d.x; v[u][1] = (VT)d.y; v[u][2] = (VT)d.z; v[u][3] = (VT)d.w;
            }
        } else {
#pragma unroll
            for (int k = 0; k < 4; ++k) v[u][k] = c + k < K ? row[c + k] : (VT)0;
        }
        if (kNorm) {
            if (p.norm_w && vec_w && c + 4 <= p.norm_w_len) {
                const float4 d = __ldg(reinterpret_cast<const float4*>(p.norm_w + c));
                w[u][0] = d.x; w[u][1] = d.y; w[u][2] = d.z; w[u][3] = d.w;
            } else {
#pragma unroll
                for (int k = 0; k < 4; ++k) w[u][k] = p.norm_w && c + k < p.norm_w_len ? __ldg(p.norm_w + c + k) : 1.f;
            }
        }
    }
    float amax = 0.f;
    if (q8) {
        amax = p.amax_in[n];
    } else {
        float m = 0.f;
        if (kNorm) {
            double ss = 0.0;
#pragma unroll
            for (int u = 0; u < UPT; ++u)
#pragma unroll
                for (int k = 0; k < 4; ++k) ss = __dadd_rn(ss, __dmul_rn((double)v[u][k], (double)v[u][k]));
            ss = lb_warp_sum(ss);
            if (lane == 0) s_ss[warp] = ss;
            __syncthreads();
            ss = lb_warp_sum(lane < (T >> 5) ? s_ss[lane] : 0.0);
            const double root = sqrt(__dadd_rn(__ddiv_rn(ss, (double)K), p.eps)), rr = __ddiv_rn(1.0, root);
#pragma unroll
            for (int u = 0; u < UPT; ++u)
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    const int c = 4 * (tid + u * T) + k;
                    if (c < K) {
                        if (f64) v[u][k] = (VT)lb_pro_value<PRO>((double)v[u][k], root, rr, (double)w[kNorm ? u : 0][k]);
                        else v[u][k] = (VT)(float)__dmul_rn(PRO == LB_PRO_BLOCKNORM ? lb_div_by((double)v[u][k], root, rr) : __dmul_rn((double)v[u][k], rr), (double)w[kNorm ? u : 0][k]);
                        if (p.norm_out) p.norm_out[(size_t)n * K + c] = (float)v[u][k];
                    }
                }
        }
#pragma unroll
        for (int u = 0; u < UPT; ++u)
#pragma unroll
            for (int k = 0; k < 4; ++k) m = fmaxf(m, (float)fabs((double)v[u][k]));
        const unsigned wm = __reduce_max_sync(0xffffffffu, __float_as_uint(m));  // (not negative: the order of the bits)
        if (lane == 0) atomicMax(&s_m, wm);
        __syncthreads();
        amax = __uint_as_float(s_m);
        if (amax < 1e-5f) amax = 1e-5f;
    }
    const double s = q8 ? 0.0 : __ddiv_rn(127.0, (double)amax);
    int sum = 0;
#pragma unroll
    for (int u = 0; u < UPT; ++u) {
        const int idx = tid + u * T;
        if (idx >= units) break;  // (whole warps)
        uint32_t packed = 0;
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            int qv = 0;
            if (q8) qv = (int)v[u][k];
            else if (4 * idx + k < K) qv = lb_quant_i8((double)v[u][k], s);
            packed |= (uint32_t)(qv & 0xff) << (8 * k);
            if (!q8 && p.q_out && 4 * idx + k < K) p.q_out[(size_t)n * K + 4 * idx + k] = (int8_t)qv;
        }
        sum = __dp4a((int)packed, 0x01010101, sum);
        // the four words of a chunk are with four neighbours: lane j of them takes byte j of each
        const int q4 = lane & ~3, j = lane & 3;
        const uint32_t sel = 0x40 | j | ((uint32_t)j << 4);
        const uint32_t r0 = __shfl_sync(0xffffffffu, packed, q4), r1 = __shfl_sync(0xffffffffu, packed, q4 + 1), r2 = __shfl_sync(0xffffffffu, packed, q4 + 2),
                       r3 = __shfl_sync(0xffffffffu, packed, q4 + 3);
        const uint32_t word = __byte_perm(__byte_perm(r0, r1, sel), __byte_perm(r2, r3, sel), 0x5410);
        const int chunk = idx >> 2, w8 = chunk & 7;
        *reinterpret_cast<uint32_t*>(img + gt_fragment(chunk >> 3, j >> 1, Mp, n, w8 & 3) + ((j & 1) * 2 + (w8 >> 2)) * 4) = word;
    }
    sum = __reduce_add_sync(0xffffffffu, sum);
    if (lane == 0) atomicAdd(&s_sum, sum);
    __syncthreads();
    if (tid == 0) {
        xsum_out[n] = s_sum;
        amax_out[n] = amax;
        if (!q8 && p.amax_out) p.amax_out[n] = amax;
    }
}

// ---- the product --------------------------------------------------------------------------------------------------------------

template <int EPI, int NT>
__global__ void __launch_bounds__(kThreads, 2) lb_gemv_tokens_kernel(const __grid_constant__ LbGemvParams p, const uint8_t* __restrict__ img, const int* __restrict__ xsum, int rows_bytes) {
    extern __shared__ __align__(128) uint8_t smem[];
    __shared__ __align__(8) uint64_t bars[kWarps * kStages], bar_rows;
    __shared__ double s_os[3][8 * NT];
    __shared__ int s_xsum[8 * NT];
    constexpr int Mp = 8 * NT;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3, M = p.M;
    uint32_t C;
    asm volatile("mov.u32 %0, %%cluster_nctarank;" : "=r"(C));
    const uint32_t rank = lb_cluster_rank();
    const int cid = (int)(blockIdx.x / C);
    const int kb0 = p.kblocks * (int)rank / (int)C, nkb = p.kblocks * ((int)rank + 1) / (int)C - kb0;
    uint8_t* ring = smem + (size_t)warp * p.stages * kStageBytes;
    const uint4* rows = reinterpret_cast<const uint4*>(smem + (size_t)kWarps * p.stages * kStageBytes);
    int* sacc = reinterpret_cast<int*>(smem + (size_t)kWarps * p.stages * kStageBytes + rows_bytes);  // [strip][token][16]
    // whole strip groups per cluster, this CTA's columns of them; a warp takes a run of (strip, k-block) tiles
    const int g0 = cid * p.part_q + (cid < p.part_r ? cid : p.part_r), ng = p.part_q + (cid < p.part_r ? 1 : 0);
    const int strips = ng * p.group, v0 = g0 * p.group, tiles = strips * nkb;
    const int w0 = tiles * warp / kWarps, w1 = tiles * (warp + 1) / kWarps;
    uint64_t* my_bars = bars + warp * kStages;
    if (tid < kWarps * kStages) lb_mbar_init(&bars[tid], 1);
    if (tid == 0) {
        lb_mbar_init(&bar_rows, 1);
        lb_fence_mbar_init();
    }
    for (int i = tid; i < strips * M * 16; i += kThreads) sacc[i] = 0;
    __syncthreads();
    struct Cursor {
        int pos, v, kb;  // tile of the run, strip (local), k-block (local)
    };
    auto chunk_len = [&](const Cursor& c) {
        int len = nkb - c.kb;
        if (len > kStageTiles) len = kStageTiles;
        if (len > w1 - c.pos) len = w1 - c.pos;
        return len;
    };
    auto advance = [&](Cursor& c, int len) {
        c.pos += len;
        c.kb += len;
        if (c.kb >= nkb) {
            c.kb = 0;
            c.v++;
        }
    };
    const uint64_t policy = lb_policy_evict_first();
    auto issue = [&](int stage, const Cursor& c, int len) {  // lane 0 only
        lb_mbar_expect_tx(&my_bars[stage], (uint32_t)len * kTileBytes);
        lb_bulk_g2s_stream(ring + (size_t)stage * kStageBytes, tile_ptr<EPI, false>(p, v0 + c.v, kb0 + c.kb), (uint32_t)len * kTileBytes, &my_bars[stage], policy);
    };
    Cursor ic;
    ic.pos = w0;
    ic.v = w0 / nkb;
    ic.kb = w0 - ic.v * nkb;
    Cursor cc = ic;
    for (int s = 0; s < p.stages && ic.pos < w1; ++s) {  // the weights do not depend on the rows
        const int len = chunk_len(ic);
        if (lane == 0) issue(s, ic, len);
        advance(ic, len);
    }
    lb_pdl_launch_dependents();
    lb_pdl_wait();
    if (tid == 0) {
        const uint32_t bytes = (uint32_t)nkb * Mp * 128;
        lb_mbar_expect_tx(&bar_rows, bytes);
        lb_bulk_g2s(smem + (size_t)kWarps * p.stages * kStageBytes, img + (size_t)kb0 * Mp * 128, bytes, &bar_rows);
    }
    const int pos0 = p.pos_ptr ? *p.pos_ptr : 0;
    if (tid < 3 * Mp) {
        const int sg = tid / Mp, n = tid - sg * Mp;
        if (sg == 0) s_xsum[n] = n < M ? xsum[n] : 0;
        s_os[sg][n] = sg < p.nseg && n < M ? lb_output_scale(p.seg[sg].scale, p.amax_in[n]) : 1.0;
    }
    bool failed = false;
    if (!lb_mbar_wait_bounded(&bar_rows, 0)) failed = true;

    int acc[NT][4][4];
    auto clear = [&]() {
#pragma unroll
        for (int q = 0; q < NT; ++q)
#pragma unroll
            for (int j = 0; j < 4; ++j)
#pragma unroll
                for (int k = 0; k < 4; ++k) acc[q][j][k] = 0;
    };
    clear();
    int cur_v = -1, cstage = 0;
    uint32_t cphase = 0;
    for (;;) {
        const bool done = cc.pos >= w1;
        if (done || cc.v != cur_v) {  // the strip's sums are handed over when the next one, or the end, comes up
            if (cur_v >= 0) {
                int* dst = sacc + (size_t)cur_v * M * 16;
#pragma unroll
                for (int q = 0; q < NT; ++q)
#pragma unroll
                    for (int k = 0; k < 4; ++k) {  // rows g and g + 8, tokens 2t and 2t + 1
                        const int n = q * 8 + 2 * t + (k & 1);
                        if (n < M) atomicAdd(&dst[n * 16 + g + 8 * (k >> 1)], acc[q][0][k] + (acc[q][1][k] >> 2) + (acc[q][2][k] >> 4) + (acc[q][3][k] >> 6));
                    }
                clear();
            }
            cur_v = cc.v;
        }
        if (done) break;
        const int len = chunk_len(cc);
        if (!failed && !lb_mbar_wait_bounded(&my_bars[cstage], cphase)) failed = true;
        const uint4* tile = reinterpret_cast<const uint4*>(ring + (size_t)cstage * kStageBytes) + lane;
        const uint4* x = rows + (size_t)cc.kb * Mp * 8 + g * 4 + t;
#pragma unroll 2
        for (int i = 0; i < len; ++i) {
            const uint4 w = tile[i * 32];
#pragma unroll
            for (int q = 0; q < NT; ++q) {
                const uint4 b01 = x[(i * 2 * Mp + q * 8) * 4], b23 = x[((i * 2 + 1) * Mp + q * 8) * 4];
                mma_u8s8(acc[q][0], w.x & 0x03030303u, w.y & 0x03030303u, w.z & 0x03030303u, w.w & 0x03030303u, b01.x, b01.y);
                mma_u8s8(acc[q][1], w.x & 0x0c0c0c0cu, w.y & 0x0c0c0c0cu, w.z & 0x0c0c0c0cu, w.w & 0x0c0c0c0cu, b01.z, b01.w);
                mma_u8s8(acc[q][2], w.x & 0x30303030u, w.y & 0x30303030u, w.z & 0x30303030u, w.w & 0x30303030u, b23.x, b23.y);
                mma_u8s8(acc[q][3], w.x & 0xc0c0c0c0u, w.y & 0xc0c0c0c0u, w.z & 0xc0c0c0c0u, w.w & 0xc0c0c0c0u, b23.z, b23.w);
            }
        }
        advance(cc, len);
        __syncwarp();
        if (ic.pos < w1) {
            const int len2 = chunk_len(ic);
            if (lane == 0) {
                fence_proxy_async();
                issue(cstage, ic, len2);
            }
            advance(ic, len2);
        }
        if (++cstage == p.stages) {
            cstage = 0;
            cphase ^= 1u;
        }
    }
    if (failed && lane == 0) atomicExch(p.status, 1);
    __syncthreads();
    if (C > 1) lb_cluster_sync();  // every CTA's sums are in its shared memory
    const int all = ng * M * 16;
    const uint32_t base = lb_smem_u32(sacc);
    for (int u = all * (int)rank / (int)C + tid; u < all * ((int)rank + 1) / (int)C; u += kThreads) {
        const int gl = u / (M * 16), i = u & 15, n = (u >> 4) - gl * M;
        int a[2] = {0, 0};
#pragma unroll
        for (int e = 0; e < (EPI == LB_EPI_SWIGLU ? 2 : 1); ++e) {
            const int at = ((gl * p.group + e) * M + n) * 16 + i;
            if (C == 1) {
                a[e] = sacc[at];
            } else {
                for (uint32_t q = 0; q < C; ++q) {
                    int v;
                    asm volatile("ld.shared::cluster.s32 %0, [%1];" : "=r"(v) : "r"(lb_cluster_addr(base + (uint32_t)at * 4, q)) : "memory");
                    a[e] += v;
                }
            }
        }
        finish_value<EPI>(p, &s_os[0][0], Mp, s_xsum[n], pos0, (g0 + gl) * p.group, 0, n, i, a[0], a[1]);
    }
    if (C > 1) lb_cluster_sync();  // nobody leaves while its sums are read
}

// Clusters of C CTAs to launch at most, two CTAs to an SM (or one): what the SMs' groups hold of whole clusters, and a few SMs
// fewer for clusters of several, since one that finds no place at once is a second wave: 16384 x 14336, three tokens, 64 clusters of four
// 18.8 us, the 71 that the occupancy query reports 25.4.
int most_clusters(const loom_b200_ctx* ctx, int C, int per_sm) {
    const int left[2][4] = {{0, 4, 16, 28}, {0, 4, 20, 20}};
    return per_sm * (ctx->sm_count - left[per_sm - 1][C == 1 ? 0 : C == 2 ? 1 : C == 4 ? 2 : 3]) / C;
}

template <int EPI>
int launch(loom_b200_ctx* ctx, LbGemvParams& p, const uint8_t* img, const int* xsum) {
    const int NT = (p.M + 7) / 8, Mp = 8 * NT, groups = p.total_tiles / p.kblocks / p.group;
    // as many CTAs to a cluster as keep the rows' share small and the device busy
    int C = 1;
    while (C < 8 && p.kblocks >= 4 * C && (((p.kblocks + C - 1) / C) * Mp * 128 > kGtRowsBytes || groups * C < ctx->sm_count)) C *= 2;
    const int rows_bytes = ((p.kblocks + C - 1) / C) * Mp * 128;
    auto smem_of = [&](int clusters, int stages) {
        return (size_t)kWarps * stages * kStageBytes + rows_bytes + (size_t)((groups + clusters - 1) / clusters) * p.group * p.M * 64;
    };
    // two CTAs to an SM, or one with the whole of its shared memory: where no SM gets a second one, or two do not fit
    const int one = most_clusters(ctx, C, 1), two = most_clusters(ctx, C, 2);
    int clusters = groups < two ? groups : two;
    const bool alone = groups <= one || smem_of(clusters, 1) > kGtSmemHalf;
    if (alone) clusters = groups < one ? groups : one;
    const size_t most = alone ? 2 * kGtSmemHalf : kGtSmemHalf;
    p.stages = kStages;
    while (p.stages > 1 && smem_of(clusters, p.stages) > most) --p.stages;
    while (smem_of(clusters, p.stages) > 2 * kGtSmemHalf && clusters < groups) clusters = clusters * 2 < groups ? clusters * 2 : groups;  // (many rows: several waves)
    const size_t smem = smem_of(clusters, p.stages);
    if (smem > 2 * kGtSmemHalf) return lb_fail(ctx, LOOM_B200_ERR_UNSUPPORTED, "gemv: %d tokens of %d columns need %zu B of shared memory", p.M, p.K, smem);
    p.part_q = groups / clusters;
    p.part_r = groups % clusters;
    p.status = ctx->status_dev;
    using Kern = void (*)(const LbGemvParams, const uint8_t*, const int*, int);
    const Kern kern = NT == 1 ? (Kern)lb_gemv_tokens_kernel<EPI, 1> : NT == 2 ? (Kern)lb_gemv_tokens_kernel<EPI, 2> : (Kern)lb_gemv_tokens_kernel<EPI, 3>;
    if (NT == 1) LB_BIG_SMEM(ctx, (lb_gemv_tokens_kernel<EPI, 1>), 2 * kGtSmemHalf);
    if (NT == 2) LB_BIG_SMEM(ctx, (lb_gemv_tokens_kernel<EPI, 2>), 2 * kGtSmemHalf);
    if (NT == 3) LB_BIG_SMEM(ctx, (lb_gemv_tokens_kernel<EPI, 3>), 2 * kGtSmemHalf);
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(clusters * C);
    cfg.blockDim = dim3(kThreads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = ctx->stream;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = C;
    attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = ctx->opt_pdl ? 2 : 1;
    LB_CUDA(ctx, cudaLaunchKernelEx(&cfg, kern, p, img, xsum, rows_bytes));
    ctx->launches++;
    return 0;
}

template <int PRO>
int prepare(loom_b200_ctx* ctx, const LbGemvParams& p, int Mp, uint8_t* img, float* amax, int* xsum) {
    const int units = p.kblocks * 32, T = units < 1024 ? units : 1024, upt = (units + T - 1) / T;
    if (upt <= 1) LB_LAUNCH(ctx, (lb_tokens_prepare_kernel<PRO, 1>), dim3(Mp), dim3(T), 0, p, Mp, img, amax, xsum);
    else if (upt <= 2) LB_LAUNCH(ctx, (lb_tokens_prepare_kernel<PRO, 2>), dim3(Mp), dim3(T), 0, p, Mp, img, amax, xsum);
    else if (upt <= 4) LB_LAUNCH(ctx, (lb_tokens_prepare_kernel<PRO, 4>), dim3(Mp), dim3(T), 0, p, Mp, img, amax, xsum);
    else LB_LAUNCH(ctx, (lb_tokens_prepare_kernel<PRO, 8>), dim3(Mp), dim3(T), 0, p, Mp, img, amax, xsum);
    return 0;
}

}  // namespace

// whether this launch is one of these: at least three tokens (one or two are quicker with the rows made inside every CTA), no agreed
// statistics and no exchange (tensor-parallel shards)
bool lb_gemv_tokens_takes(const loom_b200_ctx* ctx, const LbGemvParams& p) {
    if (p.M < kSplitQuantTokens || p.M > kGtMaxTokens || p.K > kGtMaxColumns || p.given_ss || p.given_amax || p.norm_count > 0 || p.epi == LB_EPI_TPSUM) return false;
    // int8 rows of one block of columns and few rows: the launch in front costs more than every CTA's own fragments (3 x 256 x 128 4.4 us in
    // one launch, 6.8 in two; 5 x 1024 x 128 5.9 and 6.8, 6 x 16 x 128 6.4 and 6.6; 5 x 256 x 64, read byte by byte, 7.7 and 6.6; 3 x 4096 x 128
    // 7.4 and 6.8, 3 x 256 x 256 7.1 and 6.7)
    if (p.pro == LB_PRO_Q8 && p.kblocks == 1 && p.M <= (p.K == kTileCols ? 5 : 4) && p.total_tiles <= 64) return false;
    // the options that ask for something of the one-token kernel, and a recording that the scratch would have to grow for
    return p.M > kMaxM || (!ctx->opt_gemv_partition && !ctx->trace_dev && !(ctx->capturing && gt_scratch(p.kblocks) > ctx->quant_scratch_bytes));
}

int lb_pass_tokens(const loom_b200_ctx* ctx, int K) {
    const bool fits = !ctx->capturing || gt_scratch((K + kTileCols - 1) / kTileCols) <= ctx->quant_scratch_bytes;
    if (ctx->tp_world == 1 && K <= kGtMaxColumns && fits) return kPassTokens;
    const int n = lb_gemv_max_tokens(K);
    return n < kMaxM ? n : kMaxM;
}

int lb_launch_gemv_tokens(loom_b200_ctx* ctx, const LbGemvParams& pin) {
    LbGemvParams p = pin;
    const int Mp = (p.M + 7) / 8 * 8;
    const size_t img_bytes = (size_t)p.kblocks * Mp * 128;
    if (int rc = lb_ensure_quant_scratch(ctx, gt_scratch(p.kblocks))) return rc;
    uint8_t* img = static_cast<uint8_t*>(ctx->quant_scratch);
    float* amax = reinterpret_cast<float*>(img + img_bytes);
    int* xsum = reinterpret_cast<int*>(amax + Mp);
    int rc;
    switch (p.pro) {
        case LB_PRO_Q8: rc = prepare<LB_PRO_Q8>(ctx, p, Mp, img, amax, xsum); break;
        case LB_PRO_F32: rc = prepare<LB_PRO_F32>(ctx, p, Mp, img, amax, xsum); break;
        case LB_PRO_BLOCKNORM: rc = prepare<LB_PRO_BLOCKNORM>(ctx, p, Mp, img, amax, xsum); break;
        case LB_PRO_INNERNORM: rc = prepare<LB_PRO_INNERNORM>(ctx, p, Mp, img, amax, xsum); break;
        case LB_PRO_INNERNORM64: rc = prepare<LB_PRO_INNERNORM64>(ctx, p, Mp, img, amax, xsum); break;
        default: return lb_fail(ctx, LOOM_B200_ERR_INVALID, "gemv: prologue %d", p.pro);
    }
    if (rc) return rc;
    p.amax_in = amax;
    switch (p.epi) {
        case LB_EPI_GENERIC: return launch<LB_EPI_GENERIC>(ctx, p, img, xsum);
        case LB_EPI_QKV: return launch<LB_EPI_QKV>(ctx, p, img, xsum);
        case LB_EPI_RESID: return launch<LB_EPI_RESID>(ctx, p, img, xsum);
        case LB_EPI_SWIGLU: return launch<LB_EPI_SWIGLU>(ctx, p, img, xsum);
    }
    return lb_fail(ctx, LOOM_B200_ERR_UNSUPPORTED, "gemv: no kernel for epilogue %d of several tokens", p.epi);
}

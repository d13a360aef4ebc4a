// attention_prompt.cu -- causal GQA attention of a block of prompt tokens in float64 (poly/mha.go:296-356), head dimensions 64 and 128.
//
// A CTA takes 64 query rows of a KV head: the heads of its group times 64 / group consecutive tokens.  Eight warps keep eight rows
// each to themselves from the scores to the output -- scores, running maximum and sum, weights and the output row never leave their
// registers -- so that nothing but the arrival of keys and values is waited for, and the exponentials of one warp run beside the
// matrix instructions of the others.  Two such groups of eight share the CTA: one takes the even tiles of positions, the other the odd ones,
// and they merge at the end, half of the dimensions each.  (Two CTAs of one group on an SM took 337 us: jobs are as long as their tokens
// are far into the sequence, and two long ones that share an SM end when everything else is done.)
//   * Products on m8n8k4 float64 MMAs.  Which column an MMA calls its k-th is free as long as both operands agree: a lane reads 16
//     bytes (four dimensions) of its key row and the same four of its query row, and takes two neighbouring score columns as the
//     k-th columns of two MMAs of the second product, which is how the first one's accumulators lie.  Four accumulators side by side:
//     one MMA keeps the pipe for 16 clocks, the next on the same accumulator waits for 27.
//   * Keys and values stay float32 in shared memory, in tiles of 32 positions, row strides chosen so that 16-byte loads touch every
//     bank once, and are widened where they are used.
//   * Two buffers: the last warp done with the keys of a tile asks for those two tiles on, for the values likewise; 16-byte copies of a
//     warp (bulk copies of a row each, which the strides would need, take the copy engine 30 ns apiece).
//   * Jobs in descending order of their length.
// Bound: the float64 pipe (64 multiply-adds a clock): 1024 tokens of 20 heads x 128 are 2.8e9 of them, 152 us, and the
// exponentials 12 us more.  Measured 232 us (16 rows a warp and half the warps 255; one buffer 244; bulk copies 264); 299 with the
// kernel in glue.cu, whose eight warps meet six times a tile and which stays for other head dimensions.  What is left: the pipe idles a quarter
// of the loop and at both ends of a job; widening by integer instructions instead changed nothing.
#include "dense.cuh"
#include "glue.cuh"

namespace {

constexpr int kPqRows = 64, kPqKeys = 32, kPqWarps = kPqRows / 8, kPqGroups = 2, kPqThreads = kPqGroups * kPqWarps * 32, kPqStages = 2;

template <int HD>
struct PqCfg {
    static constexpr int kQ = HD + 2;    // row strides: doubles of a query row,
    static constexpr int kK = HD + 16;   // floats of a key row,
    static constexpr int kV = HD + 4;    // floats of a value row
    static constexpr size_t kTile = (size_t)kPqKeys * (kK + kV) * 4;
    static constexpr size_t kSmem = (size_t)kPqRows * kQ * 8 + kPqGroups * kPqStages * kTile;
};

template <int HD>
__global__ void __launch_bounds__(kPqThreads, 1) lb_attention_prompt_kernel(const LbAttnParams p) {
    using C = PqCfg<HD>;
    extern __shared__ __align__(128) uint8_t smem_raw[];
    __shared__ __align__(8) uint64_t bars[kPqGroups][kPqStages][2];
    __shared__ unsigned s_done[kPqGroups][kPqStages][2];  // warps done with keys / values, over all tiles
    __shared__ double s_mx[kPqGroups][kPqRows], s_sum[kPqGroups][kPqRows];
    const int tid = threadIdx.x, grp = tid / (kPqWarps * 32), warp = (tid >> 5) % kPqWarps, lane = tid & 31, g = lane >> 2, t4 = lane & 3;
    double* sq = reinterpret_cast<double*>(smem_raw);
    float* sk = reinterpret_cast<float*>(smem_raw + (size_t)kPqRows * C::kQ * 8 + grp * kPqStages * C::kTile);
    // stage s: keys at sk + s * kStage, values kPqKeys * kK behind them
    constexpr int kStage = (int)(C::kTile / 4), kVals = kPqKeys * C::kK;
    const int group = p.heads / p.kv_heads, TQ = kPqRows / group, qd = p.heads * HD;
    const int kvh = (int)blockIdx.x % p.kv_heads, tok0 = ((int)gridDim.x / p.kv_heads - 1 - (int)blockIdx.x / p.kv_heads) * TQ;
    if (tid < kPqGroups * kPqStages * 2) {
        lb_mbar_init(&bars[0][0][0] + tid, 32);
        lb_fence_mbar_init();
        (&s_done[0][0][0])[tid] = 0;
    }
    __syncthreads();
    lb_pdl_launch_dependents();
    lb_pdl_wait();
    const int pos0 = *p.pos_ptr;
    const int ntok = p.M - tok0 < TQ ? p.M - tok0 : TQ, max_pos = pos0 + tok0 + ntok - 1, ntiles = max_pos / kPqKeys + 1;
    const float* kbase = p.cache_k + (size_t)kvh * p.msl * HD;
    const float* vbase = p.cache_v + (size_t)kvh * p.msl * HD;
    // the rows of tile t, 16 bytes a lane and copy; a whole warp.  (Bulk copies of a row each, which the strides would need, take the copy
    // engine 30 ns apiece: four tiles of 32 in 8 us.)
    auto fetch = [&](bool keys, int t) {
        constexpr int kLanes = HD / 4, kStep = 32 / kLanes;  // lanes of a row, rows of a copy
        const int rows = max_pos + 1 - t * kPqKeys < kPqKeys ? max_pos + 1 - t * kPqKeys : kPqKeys;
        const int ld = keys ? C::kK : C::kV, r0 = lane / kLanes, c = lane % kLanes * 4;
        const float *src0 = keys ? kbase : vbase, *src = src0 + (size_t)(t * kPqKeys + r0) * HD + c;  // (rows beyond the last position: zeros)
        const int stage = t / kPqGroups % kPqStages;
        const uint32_t dst = lb_smem_u32(sk + stage * kStage + (keys ? 0 : kVals) + r0 * ld + c);
#pragma unroll 8
        for (int r = 0; r < kPqKeys; r += kStep)
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst + (uint32_t)(r * ld) * 4), "l"(r + r0 < rows ? src + (size_t)r * HD : src0), "r"(r + r0 < rows ? 16 : 0) : "memory");
        asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(lb_smem_u32(&bars[grp][stage][keys ? 0 : 1])) : "memory");
    };
    // this warp no longer reads the keys (values) of tile t: the last one asks for the next tile's
    auto release = [&](bool keys, int t) {
        unsigned n = 0;
        __syncwarp();
        if (lane == 0) {
            __threadfence_block();
            n = atomicAdd(&s_done[grp][t / kPqGroups % kPqStages][keys ? 0 : 1], 1u) + 1;
        }
        n = __shfl_sync(0xffffffffu, n, 0);
        if (n == (unsigned)(t / kPqGroups / kPqStages + 1) * kPqWarps && t + kPqGroups * kPqStages < ntiles) {
            __threadfence_block();
            fetch(keys, t + kPqGroups * kPqStages);
        }
    };
    if (warp < kPqStages && grp + warp * kPqGroups < ntiles) {
        fetch(true, grp + warp * kPqGroups);
        fetch(false, grp + warp * kPqGroups);
    }
    // query row r = (head r / TQ of the group, token r % TQ); rows of absent tokens are zero and never written back
    for (int idx = tid; idx < kPqRows * (HD / 2); idx += kPqThreads) {
        const int r = idx / (HD / 2), d = (idx - r * (HD / 2)) * 2, hi = r / TQ, ti = r - hi * TQ;
        const double* src = ti < ntok ? p.q + (size_t)(tok0 + ti) * qd + (size_t)(kvh * group + hi) * HD + d : p.q;
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(lb_smem_u32(sq + (size_t)r * C::kQ + d)), "l"(src), "r"(ti < ntok ? 16 : 0) : "memory");
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
    __syncthreads();
    const double scale = __ddiv_rn(1.0, sqrt((double)HD));
    const int row = warp * 8 + g, qpos = row % TQ < ntok ? pos0 + tok0 + row % TQ : -1;  // this lane's row and its position (-1: absent)
    const int wmax = __reduce_max_sync(0xffffffffu, qpos), wmin = __reduce_min_sync(0xffffffffu, qpos);
    double o[HD / 8][2], mx = -1e300, sum = 0.0;
#pragma unroll
    for (int j = 0; j < HD / 8; ++j) o[j][0] = o[j][1] = 0.0;
    const double* qa = sq + (size_t)row * C::kQ + 4 * t4;
    const float* kb = sk + g * C::kK + 4 * t4;
    const float* vb = sk + kVals + 2 * t4 * C::kV + 4 * g;
    bool failed = false;
    for (int t = grp; t < ntiles; t += kPqGroups) {
        const int stage = t / kPqGroups % kPqStages, off = stage * kStage;
        const uint32_t parity = (uint32_t)(t / kPqGroups / kPqStages & 1);
        const int kpos0 = t * kPqKeys;
        const bool seen = kpos0 <= wmax;  // some row of this warp sees the tile
        if (!failed && !lb_mbar_wait_bounded(&bars[grp][stage][0], parity)) failed = true;
        double c[4][2];
        if (seen) {
#pragma unroll
            for (int n = 0; n < 4; ++n) c[n][0] = c[n][1] = 0.0;
#pragma unroll 1
            for (int s = 0; s < HD / 16; ++s) {
                const double2 lo = *reinterpret_cast<const double2*>(qa + 16 * s), hi = *reinterpret_cast<const double2*>(qa + 16 * s + 2);
                const double a[4] = {lo.x, lo.y, hi.x, hi.y};
                double kd[4][4];
#pragma unroll
                for (int n = 0; n < 4; ++n) {
                    const float4 k4 = *reinterpret_cast<const float4*>(kb + off + 8 * n * C::kK + 16 * s);
                    kd[n][0] = (double)k4.x;
                    kd[n][1] = (double)k4.y;
                    kd[n][2] = (double)k4.z;
                    kd[n][3] = (double)k4.w;
                }
#pragma unroll
                for (int e = 0; e < 4; ++e)
#pragma unroll
                    for (int n = 0; n < 4; ++n) lb_dmma_884(c[n], a[e], kd[n][e]);
            }
        }
        release(true, t);
        if (seen) {
            double m = -1e300;
#pragma unroll
            for (int n = 0; n < 4; ++n)
#pragma unroll
                for (int e = 0; e < 2; ++e) {
                    double v = __dmul_rn(c[n][e], scale);
                    if (kpos0 + kPqKeys - 1 > wmin && kpos0 + 8 * n + 2 * t4 + e > qpos) v = -INFINITY;  // not visible
                    c[n][e] = v;
                    m = fmax(m, v);
                }
            m = fmax(m, __shfl_xor_sync(0xffffffffu, m, 1));
            m = fmax(m, __shfl_xor_sync(0xffffffffu, m, 2));
            m = fmax(m, mx);
            if (__any_sync(0xffffffffu, m != mx)) {  // (a factor of one changes nothing)
                const double f = m != mx ? exp(__dsub_rn(mx, m)) : 1.0;
                sum = __dmul_rn(sum, f);
#pragma unroll
                for (int j = 0; j < HD / 8; ++j) {
                    o[j][0] = __dmul_rn(o[j][0], f);
                    o[j][1] = __dmul_rn(o[j][1], f);
                }
                mx = m;
            }
#pragma unroll
            for (int n = 0; n < 4; ++n)
#pragma unroll
                for (int e = 0; e < 2; ++e) {
                    c[n][e] = exp(__dsub_rn(c[n][e], m));
                    sum = __dadd_rn(sum, c[n][e]);
                }
        }
        if (!failed && !lb_mbar_wait_bounded(&bars[grp][stage][1], parity)) failed = true;
        if (seen) {
#pragma unroll
            for (int n = 0; n < 4; ++n)
#pragma unroll
                for (int e = 0; e < 2; ++e)
#pragma unroll
                    for (int q = 0; q < HD / 32; ++q) {
                        const float4 v4 = *reinterpret_cast<const float4*>(vb + off + (8 * n + e) * C::kV + 32 * q);
                        lb_dmma_884(o[4 * q], c[n][e], (double)v4.x);
                        lb_dmma_884(o[4 * q + 1], c[n][e], (double)v4.y);
                        lb_dmma_884(o[4 * q + 2], c[n][e], (double)v4.z);
                        lb_dmma_884(o[4 * q + 3], c[n][e], (double)v4.w);
                    }
        }
        release(false, t);
    }
    if (__any_sync(0xffffffffu, failed) && lane == 0) atomicExch(p.status, 1);
    sum += __shfl_xor_sync(0xffffffffu, sum, 1);
    sum += __shfl_xor_sync(0xffffffffu, sum, 2);
    // The groups merge through the shared memory of the queries, lane by lane: each finishes one half of the dimensions and hands over
    // the other.
    __syncthreads();
    double2* meet = reinterpret_cast<double2*>(smem_raw);  // [group][output][thread of a group]
    constexpr int kHalf = HD / 16;
    const int at = warp * 32 + lane;
#pragma unroll
    for (int j = 0; j < kHalf; ++j) meet[(grp * kHalf + j) * kPqWarps * 32 + at] = grp ? make_double2(o[j][0], o[j][1]) : make_double2(o[kHalf + j][0], o[kHalf + j][1]);
    if (t4 == 0) {
        s_mx[grp][row] = mx;
        s_sum[grp][row] = sum;
    }
    __syncthreads();
    const int hi = row / TQ, ti = row - hi * TQ;
    if (ti >= ntok) return;
    const double mo = s_mx[grp ^ 1][row], m = fmax(mx, mo), f0 = exp(__dsub_rn(mx, m)), f1 = exp(__dsub_rn(mo, m));
    const double den = __dadd_rn(__dmul_rn(sum, f0), __dmul_rn(s_sum[grp ^ 1][row], f1));
#pragma unroll
    for (int j = 0; j < kHalf; ++j) {
        const double2 v = meet[((grp ^ 1) * kHalf + j) * kPqWarps * 32 + at];
        const double x = grp ? o[kHalf + j][0] : o[j][0], y = grp ? o[kHalf + j][1] : o[j][1];
        o[j][0] = __ddiv_rn(__dadd_rn(__dmul_rn(x, f0), __dmul_rn(v.x, f1)), den);
        o[j][1] = __ddiv_rn(__dadd_rn(__dmul_rn(y, f0), __dmul_rn(v.y, f1)), den);
    }
    // lane (g, t4) holds dimensions 32 q + 8 t4 .. + 7 of row g
    double* out = p.out + (size_t)(tok0 + ti) * qd + (size_t)(kvh * group + hi) * HD + grp * (HD / 2) + 8 * t4;
#pragma unroll
    for (int q = 0; q < HD / 64; ++q)
#pragma unroll
        for (int e = 0; e < 2; ++e)
#pragma unroll
            for (int d = 0; d < 4; d += 2) *reinterpret_cast<double2*>(out + 32 * q + 4 * e + d) = make_double2(o[4 * q + d][e], o[4 * q + d + 1][e]);
}

template <int HD>
int launch(loom_b200_ctx* ctx, const LbAttnParams& p) {
    using C = PqCfg<HD>;
    LB_BIG_SMEM(ctx, lb_attention_prompt_kernel<HD>, C::kSmem);
    const int TQ = kPqRows / (p.heads / p.kv_heads);
    LB_LAUNCH(ctx, lb_attention_prompt_kernel<HD>, dim3(p.kv_heads * ((p.M + TQ - 1) / TQ)), dim3(kPqThreads), C::kSmem, p);
    return 0;
}

}  // namespace

// the caller has checked lb_attention_prefill_supported; false: not a head dimension of this kernel
bool lb_attention_prompt_takes(const LbAttnParams& p) { return p.hd == 64 || p.hd == 128; }
int lb_launch_attention_prompt(loom_b200_ctx* ctx, const LbAttnParams& p) { return p.hd == 128 ? launch<128>(ctx, p) : launch<64>(ctx, p); }

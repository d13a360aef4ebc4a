// dense.cu -- 16-bit / 32-bit float matrices: storage (loom_b200_matrix_*), the small-batch GEMV and the plain token-block
// GEMM for 32-bit floats.  The bf16 token-block GEMM on the tensor cores is in gemm_bf16.cu.
#include "dense.cuh"

#include <vector>

namespace {

constexpr int kGemvThreads = 256;
constexpr int kGemvWarps = kGemvThreads / 32;
constexpr size_t kGemvSmemX = 200 * 1024;
constexpr int kGemvSmemHalf = 103 * 1024;  // dynamic part of a CTA when two share an SM (228 KB, 1 KB reserved and up to 9.3 KB static each)

// one thread per 16-byte chunk of the source rows
template <typename WT>
__global__ void lb_image_put_kernel(const void* __restrict__ src, int src_dtype, int rows, int cols, int row0, int slices, uint8_t* __restrict__ img) {
    constexpr int C = LbElem<WT>::kChunk;
    const int chunks = slices * 8;
    const size_t idx = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (idx >= (size_t)rows * chunks) return;
    const int r = (int)(idx / chunks), c = (int)(idx % chunks);
    float f[C];
#pragma unroll
    for (int i = 0; i < C; ++i) {
        const int col = c * C + i;
        float v = 0.f;
        if (col < cols)
            v = src_dtype == LOOM_B200_DTYPE_BF16 ? __bfloat162float(static_cast<const __nv_bfloat16*>(src)[(size_t)r * cols + col])
                                                  : static_cast<const float*>(src)[(size_t)r * cols + col];
        f[i] = v;
    }
    *reinterpret_cast<uint4*>(img + lb_img_chunk(row0 + r, c, slices)) = lb_pack_chunk<WT>(f);
}

// ---- GEMV -------------------------------------------------------------------------------------------------

__device__ __forceinline__ uint4 ldg_stream(const uint8_t* p) {
    uint4 v;
    asm volatile("ld.global.nc.L1::no_allocate.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p));
    return v;
}
__device__ __forceinline__ void mma_bf16(float* d, uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
                 : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

// Accumulator of a warp's 16 rows.  bf16: the m16n8 fragment of lane (g, t) = rows g, g+8 x tokens 2t, 2t+1.  float: rows
// g, g+8 x all eight tokens, over the K chunks of lane column t (summed over t at the end).
template <typename WT>
struct GemvAcc;
template <>
struct GemvAcc<__nv_bfloat16> {
    float d[4];
    __device__ __forceinline__ void zero() { d[0] = d[1] = d[2] = d[3] = 0.f; }
    // one 16-byte chunk of rows g and g+8 against the same chunk of token g: which two k of a chunk an MMA takes as its
    // "low" and "high" pair is the same for both operands, so the order inside the chunk cancels
    __device__ __forceinline__ void step(const uint4& w0, const uint4& w1, const uint4* xs, int Mp, int M, int g) {
        const uint4 x = g < Mp ? xs[g] : make_uint4(0, 0, 0, 0);
        mma_bf16(d, w0.x, w1.x, w0.y, w1.y, x.x, x.y);
        mma_bf16(d, w0.z, w1.z, w0.w, w1.w, x.z, x.w);
    }
    __device__ __forceinline__ void store(float* red, int g, int t) {
        red[g * 8 + 2 * t] = d[0];
        red[g * 8 + 2 * t + 1] = d[1];
        red[(g + 8) * 8 + 2 * t] = d[2];
        red[(g + 8) * 8 + 2 * t + 1] = d[3];
    }
};
template <>
struct GemvAcc<float> {
    float a[2][8];
    __device__ __forceinline__ void zero() {
#pragma unroll
        for (int m = 0; m < 8; ++m) a[0][m] = a[1][m] = 0.f;
    }
    __device__ __forceinline__ void step(const uint4& w0, const uint4& w1, const uint4* xs, int Mp, int M, int g) {
        float p[4], q[4], x[4];
        lb_unpack_chunk<float>(w0, p);
        lb_unpack_chunk<float>(w1, q);
#pragma unroll
        for (int m = 0; m < 8; ++m) {
            if (m >= M) break;
            lb_unpack_chunk<float>(xs[m], x);
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                a[0][m] = fmaf(p[i], x[i], a[0][m]);
                a[1][m] = fmaf(q[i], x[i], a[1][m]);
            }
        }
    }
    __device__ __forceinline__ void store(float* red, int g, int t) {
#pragma unroll
        for (int m = 0; m < 8; ++m)
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                float v = a[h][m];
                v += __shfl_xor_sync(0xffffffffu, v, 1);
                v += __shfl_xor_sync(0xffffffffu, v, 2);
                if (t == 0) red[(g + 8 * h) * 8 + m] = v;
            }
    }
};

// the same for rows of (token, choice) pairs (routed experts, second product): xw points at the chunks that the lanes of this
// warp fetched, lane (g, t) the one of token g, zeros where the token did not choose the expert (bit m of `chose` is not set).
// Multiply-adds leave those tokens out: an infinite weight times such a zero would reach a token that has nothing to do with it.
template <typename WT>
__device__ __forceinline__ void step_pairs(GemvAcc<WT>& acc, const uint4& w0, const uint4& w1, const uint4* xw, unsigned chose, int lane);
template <>
__device__ __forceinline__ void step_pairs<__nv_bfloat16>(GemvAcc<__nv_bfloat16>& acc, const uint4& w0, const uint4& w1, const uint4* xw, unsigned chose, int lane) {
    const uint4 x = xw[lane];
    mma_bf16(acc.d, w0.x, w1.x, w0.y, w1.y, x.x, x.y);
    mma_bf16(acc.d, w0.z, w1.z, w0.w, w1.w, x.z, x.w);
}
template <>
__device__ __forceinline__ void step_pairs<float>(GemvAcc<float>& acc, const uint4& w0, const uint4& w1, const uint4* xw, unsigned chose, int lane) {
    float p[4], q[4], x[4];
    lb_unpack_chunk<float>(w0, p);
    lb_unpack_chunk<float>(w1, q);
#pragma unroll
    for (int m = 0; m < 8; ++m) {
        if (!(chose >> m & 1)) continue;
        lb_unpack_chunk<float>(xw[m * 4 + (lane & 3)], x);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            acc.a[0][m] = fmaf(p[i], x[i], acc.a[0][m]);
            acc.a[1][m] = fmaf(q[i], x[i], acc.a[1][m]);
        }
    }
}

// ---- the weight ring: every warp copies the chunks it will multiply itself (16 bytes a lane and copy, so no barrier of the
// block is needed between the copies and their use), `depth` K slices ahead.  One batch in registers and one in flight (32 KB an
// SM) left the routed products at half of HBM's rate: a step of eight sequences over 32 experts of 4096 x 1792 (four layers) took
// 1.53 ms, 1.27 ms with the ring (96 KB a CTA, two CTAs an SM); a one-sequence step with gated feed-forwards of 6912 572 and 533 us.  Products
// whose 16-row strips are fewer than the CTAs that fit are bound by the chain of their input rows, not by this. ----
constexpr int kRingUnit = kGemvThreads * 16;  // bytes of one 16-byte chunk per thread
constexpr int kRingMax = 8;
__device__ __forceinline__ void ring_copy(uint32_t dst, const uint8_t* src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void ring_copy_or_zero(uint32_t dst, const uint8_t* src, bool ok) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(ok ? 16 : 0) : "memory");
}
__device__ __forceinline__ void ring_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
// the oldest of `depth` groups has arrived
__device__ __forceinline__ void ring_wait(int depth) {
    switch (depth) {
        case 8: asm volatile("cp.async.wait_group 7;" ::: "memory"); break;
        case 7: asm volatile("cp.async.wait_group 6;" ::: "memory"); break;
        case 6: asm volatile("cp.async.wait_group 5;" ::: "memory"); break;
        case 5: asm volatile("cp.async.wait_group 4;" ::: "memory"); break;
        case 4: asm volatile("cp.async.wait_group 3;" ::: "memory"); break;
        case 3: asm volatile("cp.async.wait_group 2;" ::: "memory"); break;
        case 2: asm volatile("cp.async.wait_group 1;" ::: "memory"); break;
        default: asm volatile("cp.async.wait_group 0;" ::: "memory"); break;
    }
}

// KW warps share a strip of 16 rows by K slices, 8/KW strips run side by side in a CTA.
// RING: weights through the ring; else (the input rows leave room for less than two slots) straight into registers, as far ahead as
// those allow.  Requests on four layers with second products of 24576 columns, short prompts and 24 steps: four bf16 sequences 11.9 ms
// (12.3 before there was a ring, 12.5 with a ring of one slot), two float32 ones 15.7 ms (17.0 with one slot).  A kernel of its own:
// as a branch it cost the ring's registers, 31.7 -> 30.4 ms for 48 steps of the 2560-wide Zitupel behind 100 tokens without it.
template <typename WT, int PRO, int EPI, bool RING>
__global__ void __launch_bounds__(kGemvThreads, 2) lb_dense_gemv_kernel(const LbDenseGemv p, int Mp_launch, int KW, bool vec, int ring_off, int depth) {
    extern __shared__ __align__(16) uint8_t smem[];
    constexpr int C = LbElem<WT>::kChunk;
    constexpr bool kDual = EPI == LB_DEPI_GLU || EPI == LB_DEPI_SILU;
    constexpr int kUnits = kDual ? 8 : PRO == LB_DPRO_PAIRS ? 6 : 4;  // 16-byte chunks of a thread per K slice
    __shared__ float red[kGemvWarps][128];
    __shared__ float red2[kDual ? kGemvWarps : 1][128];
    __shared__ float s_stat[kGemvWarps];
    __shared__ int s_pair[kMaxLanesPerPass], s_tok[kMaxLanesPerPass], s_n;
    __shared__ float s_w[kMaxLanesPerPass];
    constexpr bool kStage = EPI == LB_DEPI_STAGE;
    // columns of this CTA: every token; the token of a staging CTA; the tokens that chose this CTA's expert
    int M = kStage ? 1 : p.M, Mp = kStage ? 1 : Mp_launch;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3;
    const int SP = kGemvWarps / KW, kw = warp % KW, sp = warp / KW;
    const int strips = lb_ceil_div(p.rows, 16), chunks = p.slices * 8;
    uint4* xs = reinterpret_cast<uint4*>(smem);  // [chunk][Mp]
    const uint8_t *w1 = p.w, *w2 = p.w2;

    int strip = (int)blockIdx.x * SP + sp;
    const int step = (int)gridDim.x * SP;
    auto strip_ptr = [&](const uint8_t* base, int st) { return base + (size_t)(st >> 3) * p.slices * kImgBlock + (size_t)(st & 7) * 2048; };
    const size_t lane_off = (size_t)t * 128 + (size_t)g * 16;  // lane (g, t) takes chunks t, t+4 of rows g, g+8

    // The lanes of a warp copy 512 consecutive bytes in order (a line whose bytes land in four places costs four writes: the
    // 656 MB head took 172 us that way) and read them across: the chunk of lane (g, t) lies at t * 8 + (g ^ 2t), which is free
    // of bank conflicts both ways.
    const uint8_t* ring = smem + ring_off + (size_t)warp * 512;
    const int at_read = t * 8 + (g ^ (2 * t));
    const uint32_t ring_x = lb_smem_u32(ring) + (uint32_t)lane * 16;
    const uint32_t ring_s = lb_smem_u32(ring) + (uint32_t)((lane & 24) + ((lane & 7) ^ (2 * (lane >> 3)))) * 16;
    // the ring's head: the strip and slice the next copy takes, over all strips of this warp (routed second product: K runs over
    // the experts of the list one after the other)
    int* s_route = reinterpret_cast<int*>(smem);  // PAIRS: experts of the list, then their pairs
    int nact = 1, head_strip = strip, head_sl = kw, head_at = 0, head_slot = 0;
    auto fetch = [&]() {
        if (head_strip < strips) {
            const uint32_t dst = ring_s + (uint32_t)(head_slot * kUnits * kRingUnit);
            const size_t group = PRO == LB_DPRO_PAIRS ? (size_t)s_route[head_at] * p.group_bytes : 0;
            const size_t off = (size_t)head_sl * kImgBlock + (size_t)lane * 16;
            const uint8_t* q = strip_ptr(w1 + group, head_strip) + off;
            ring_copy(dst, q);
            ring_copy(dst + kRingUnit, q + 512);
            ring_copy(dst + 2 * kRingUnit, q + 1024);
            ring_copy(dst + 3 * kRingUnit, q + 1536);
            if (kDual) {
                const uint8_t* q2 = strip_ptr(w2, head_strip) + off;
                ring_copy(dst + 4 * kRingUnit, q2);
                ring_copy(dst + 5 * kRingUnit, q2 + 512);
                ring_copy(dst + 6 * kRingUnit, q2 + 1024);
                ring_copy(dst + 7 * kRingUnit, q2 + 1536);
            }
            if (PRO == LB_DPRO_PAIRS) {
                const int pr = s_route[kMaxLanesPerPass * kMaxTop + head_at * kMaxLanesPerPass + g];
                const uint8_t* x = p.pairs + (size_t)(pr < 0 ? 0 : pr) * p.ldp * sizeof(WT) + (size_t)(head_sl * 8 + t) * 16;
                const uint32_t dx = ring_x + (uint32_t)(head_slot * kUnits * kRingUnit);
                ring_copy_or_zero(dx + 4 * kRingUnit, x, pr >= 0);
                ring_copy_or_zero(dx + 5 * kRingUnit, x + 64, pr >= 0);
            }
            head_sl += KW;
            if (head_sl >= p.slices) {
                head_sl -= p.slices;
                if (++head_at == nact) {
                    head_at = 0;
                    head_sl = kw;
                    head_strip += step;
                }
            }
        }
        ring_commit();
        head_slot = head_slot + 1 == depth ? 0 : head_slot + 1;
    };
    // the weights do not depend on earlier launches: the ring is filled before the dependency wait
    constexpr bool kEarly = PRO != LB_DPRO_MOE && PRO != LB_DPRO_PAIRS && !kStage;
    if (kEarly && RING)
        for (int i = 0; i < depth; ++i) fetch();
    // nor do the vectors of the prologue, which a layer's weights have pushed out of the L2 cache since the last token
    if (kEarly || kStage) {
        auto prefetch = [&](const float* v, int n) {
            if (v)
                for (int i = tid * 32; i < n; i += kGemvThreads * 32) asm volatile("prefetch.global.L2 [%0];" ::"l"(v + i));
        };
        if (PRO == LB_DPRO_NORM || PRO == LB_DPRO_MOE) prefetch(p.gain_w, p.K);
        if (PRO == LB_DPRO_GATED) prefetch(p.head_w, p.K);
        if (PRO == LB_DPRO_CONV) prefetch(p.conv_w, p.taps * p.ring_ld);
    }
    if (kStage) lb_pdl_launch_dependents();
    lb_pdl_wait();

    if (PRO == LB_DPRO_MOE) {
        // every CTA repeats the choice of experts: a warp per token, `top` rounds of a warp-wide first maximum
        float* sl = reinterpret_cast<float*>(smem + (size_t)chunks * Mp * 16);  // [M][experts]
        int* s_idx = reinterpret_cast<int*>(sl + (size_t)p.M * p.experts);     // [M][top]
        if (warp < p.M) {
            float* row = sl + (size_t)warp * p.experts;
            for (int e = lane; e < p.experts; e += 32) row[e] = p.logits[(size_t)warp * p.ldl + e];
            __syncwarp();
            for (int j = 0; j < p.top; ++j) {
                float best = -INFINITY;
                int bi = 0x7fffffff;
                for (int e = lane; e < p.experts; e += 32)
                    if (row[e] > best) {
                        best = row[e];
                        bi = e;
                    }
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) {
                    const float ov = __shfl_xor_sync(0xffffffffu, best, o);
                    const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
                    if (ov > best || (ov == best && oi < bi)) {
                        best = ov;
                        bi = oi;
                    }
                }
                if (bi >= p.experts) bi = 0;  // only NaNs left
                if (lane == 0) {
                    s_idx[warp * p.top + j] = bi;
                    row[bi] = -INFINITY;
                }
                __syncwarp();
            }
        }
        __syncthreads();
        const int pairs = p.M * p.top;
        auto first_of = [&](int pr) {  // whether this (token, choice) is the first that names its expert
            for (int q = 0; q < pr; ++q)
                if (s_idx[q] == s_idx[pr]) return false;
            return true;
        };
        if (blockIdx.x == 0 && blockIdx.y == 0 && tid < pairs && first_of(tid)) {
            int at = 0;
            for (int q = 0; q < tid; ++q) at += first_of(q) ? 1 : 0;
            p.list->expert[at] = s_idx[tid];
            for (int m = 0; m < p.M; ++m) {
                int found = -1;
                for (int j = 0; j < p.top; ++j)
                    if (s_idx[m * p.top + j] == s_idx[tid]) found = m * p.top + j;
                p.list->pair[at][m] = found;
            }
        }
        if (blockIdx.x == 0 && blockIdx.y == 0 && tid == 0) {
            int n = 0;
            for (int q = 0; q < pairs; ++q) n += first_of(q) ? 1 : 0;
            p.list->n = n;
        }
        const int mine = blockIdx.y;
        if (!first_of(mine)) return;  // uniform over the CTA
        const int e = s_idx[mine];
        w1 += (size_t)e * p.group_bytes;
        w2 += (size_t)e * p.group_bytes;
        if (tid == 0) {
            int n = 0;
            for (int q = 0; q < pairs; ++q)
                if (s_idx[q] == e) {
                    s_pair[n] = q;
                    s_tok[n] = q / p.top;
                    s_w[n] = lb_sigmoidf(p.logits[(size_t)(q / p.top) * p.ldl + e]);
                    ++n;
                }
            s_n = n;
        }
        if (RING)
            for (int i = 0; i < depth; ++i) fetch();
        __syncthreads();
        M = s_n;
        Mp = 1;
        while (Mp < M) Mp *= 2;
    }

    if (PRO == LB_DPRO_STAGED) {
        const int n = chunks * Mp;
        for (int i0 = tid; i0 < n; i0 += 8 * kGemvThreads) {
            uint4 v[8];
#pragma unroll
            for (int i = 0; i < 8; ++i)
                if (i0 + i * kGemvThreads < n) v[i] = p.staged[i0 + i * kGemvThreads];
#pragma unroll
            for (int i = 0; i < 8; ++i)
                if (i0 + i * kGemvThreads < n) xs[i0 + i * kGemvThreads] = v[i];
        }
        __syncthreads();
    } else if (PRO != LB_DPRO_PAIRS) {
        // ---- input rows: 8/Mp warps per token.  This is on the critical path of every step (the weights are on their way), so a
        // thread asks for all it needs of R chunks at once -- the row, the gate, the convolution's history -- and keeps the row in
        // registers over the meeting of the sums; only columns beyond those are read again. ----
        const int WPT = kGemvWarps / Mp, m = warp / WPT, wt = warp % WPT, lt = wt * 32 + lane, nt = WPT * 32;
        const bool live = m < M;
        const int tok = !live ? 0 : kStage ? (int)blockIdx.x : PRO == LB_DPRO_MOE ? s_tok[m] : m;
        int pos = 0;
        if (PRO == LB_DPRO_CONV && live) pos = p.pos[tok];
        const int src = p.row_idx ? p.row_idx[tok] : tok;
        const float* xr = p.x + (size_t)src * p.ldx;
        const float* gate_row = PRO == LB_DPRO_GATED ? p.gate + (size_t)tok * p.gate_ld : nullptr;
        float* conv_ring = PRO == LB_DPRO_CONV ? p.conv_ring + (size_t)(p.lane0 + tok) * p.taps * p.ring_ld : nullptr;
        constexpr bool kNormed = PRO == LB_DPRO_NORM || PRO == LB_DPRO_CONV || PRO == LB_DPRO_MOE;
        constexpr int R = PRO == LB_DPRO_CONV || PRO == LB_DPRO_GATED ? 2 : 4;
        constexpr bool kSide = PRO == LB_DPRO_CONV || PRO == LB_DPRO_GATED;
        float xc[R][C], side[kSide ? R : 1][C];
        auto load = [&](int base) {
#pragma unroll
            for (int i = 0; i < R; ++i) {
                const int c = base + i * nt, k0 = c * C;
#pragma unroll
                for (int j = 0; j < C; ++j) xc[i][j] = 0.f;
                if (live && c < chunks && k0 < p.K) lb_load_cols<C>(xr, k0, p.K, vec, xc[i]);
            }
            if (PRO == LB_DPRO_GATED) {
#pragma unroll
                for (int i = 0; i < R; ++i) {
                    const int c = base + i * nt, k0 = c * C;
                    if (live && c < chunks && k0 < p.K) lb_load_cols<C>(gate_row, k0, p.K, vec, side[i]);
                }
            }
            if (PRO == LB_DPRO_CONV) {  // what the earlier positions add
#pragma unroll
                for (int i = 0; i < R; ++i) {
                    const int c = base + i * nt, k0 = c * C;
#pragma unroll
                    for (int j = 0; j < C; ++j) side[i][j] = 0.f;
                    if (!live || c >= chunks || k0 >= p.K) continue;
                    for (int j0 = 0; j0 + 1 < p.taps; j0 += 3) {  // tap j looks back taps - 1 - j positions
                        float w[3][C], y[3][C];
#pragma unroll
                        for (int j = 0; j < 3; ++j) {
                            const int ps = pos - (p.taps - 1) + j0 + j;
                            if (j0 + j + 1 < p.taps && ps >= 0) {
                                lb_load_cols<C>(p.conv_w + (size_t)(j0 + j) * p.ring_ld, k0, p.K, vec, w[j]);
                                lb_load_cols<C>(conv_ring + (size_t)(ps % p.taps) * p.ring_ld, k0, p.K, vec, y[j]);
                            }
                        }
#pragma unroll
                        for (int j = 0; j < 3; ++j)
                            if (j0 + j + 1 < p.taps && pos - (p.taps - 1) + j0 + j >= 0)
#pragma unroll
                                for (int e = 0; e < C; ++e) side[i][e] = fmaf(w[j][e], y[j][e], side[i][e]);
                    }
                }
            }
        };
        // Sums take the columns one by one across the lanes, whatever chunks the registers hold: a row's last bits, and what bf16 makes
        // of them layer by layer, do not depend on how the row is read.  The columns come with the same lines as the chunks: 48 steps of
        // the 2560-wide Zitupel behind 100 tokens take 32.1 ms, 32.0 with sums over a thread's own chunks, whose order also left twice
        // the error against 64 bits in a float32 stack (1.9e-6; 0.6e-6 so).
        float rstd = 0.f, gain = 1.f;
        float* s_head = nullptr;
        if (kNormed) {
            if (p.gain) gain = *p.gain;
            constexpr int U = 12;
            float v[U];
            auto columns = [&](int k0) {
#pragma unroll
                for (int i = 0; i < U; ++i) {
                    const int k = k0 + i * nt;
                    v[i] = live && k < p.K ? xr[k] : 0.f;
                }
            };
            columns(lt);
            load(lt);
            float ss = 0.f;
            for (int k0 = lt;;) {
#pragma unroll
                for (int i = 0; i < U; ++i) ss = fmaf(v[i], v[i], ss);
                k0 += U * nt;
                if (k0 >= p.K) break;
                columns(k0);
            }
            ss = lb_warp_sumf(ss);
            if (lane == 0) s_stat[warp] = ss;
            __syncthreads();
            float tot = 0.f;
            for (int i = 0; i < WPT; ++i) tot += s_stat[m * WPT + i];
            rstd = __fdiv_rn(1.f, sqrtf(__fadd_rn(__fdiv_rn(tot, (float)p.K), p.eps)));
        } else if (PRO == LB_DPRO_GATED) {
            // a warp per head, two heads' columns asked for at once
            constexpr int U = 8;
            const int heads = p.K / p.head_dim;
            s_head = reinterpret_cast<float*>(smem + (size_t)chunks * Mp * 16) + (size_t)m * heads;
            float v[2][U];
            auto columns = [&](int h0, int d0) {
#pragma unroll
                for (int q = 0; q < 2; ++q)
#pragma unroll
                    for (int i = 0; i < U; ++i) {
                        const int h = h0 + q * WPT, d = d0 + 32 * i;
                        v[q][i] = live && h < heads && d < p.head_dim ? xr[h * p.head_dim + d] : 0.f;
                    }
            };
            columns(wt, lane);
            load(lt);
            for (int h0 = wt; h0 < heads; h0 += 2 * WPT) {
                float ss[2] = {0.f, 0.f};
                if (h0 != wt) columns(h0, lane);
                for (int d0 = lane;;) {
#pragma unroll
                    for (int q = 0; q < 2; ++q)
#pragma unroll
                        for (int i = 0; i < U; ++i) ss[q] = fmaf(v[q][i], v[q][i], ss[q]);
                    d0 += 32 * U;
                    if (d0 - lane >= p.head_dim) break;
                    columns(h0, d0);
                }
#pragma unroll
                for (int q = 0; q < 2; ++q) {
                    const float s = lb_warp_sumf(ss[q]);
                    const int h = h0 + q * WPT;
                    if (live && lane == 0 && h < heads) s_head[h] = __fdiv_rn(1.f, sqrtf(__fadd_rn(__fdiv_rn(s, (float)p.head_dim), p.eps)));
                }
            }
            __syncthreads();
        } else {
            load(lt);
        }
        for (int base = lt; base < chunks; base += R * nt) {
            if (base != lt) load(base);
#pragma unroll
            for (int i = 0; i < R; ++i) {
                const int c = base + i * nt, k0 = c * C;
                float (&f)[C] = xc[i];
                if (c >= chunks) continue;
                if (live && k0 < p.K) {
                    if (kNormed) {
#pragma unroll
                        for (int j = 0; j < C; ++j) f[j] = f[j] * rstd * gain;
                        if (p.gain_w) {
                            float w[C];
                            lb_load_cols<C>(p.gain_w, k0, p.K, vec, w);
#pragma unroll
                            for (int j = 0; j < C; ++j) f[j] *= w[j];
                        }
                        if (PRO == LB_DPRO_NORM && p.x_out && (kStage || blockIdx.x == 0)) {
#pragma unroll
                            for (int j = 0; j < C; ++j)
                                if (k0 + j < p.K) p.x_out[(size_t)tok * p.ldx + k0 + j] = f[j];
                        }
                    }
                    if (PRO == LB_DPRO_MOE) {
#pragma unroll
                        for (int j = 0; j < C; ++j) f[j] *= s_w[m];
                    }
                    if (PRO == LB_DPRO_GATED) {
                        float hw[C];
                        lb_load_cols<C>(p.head_w, k0, p.K, vec, hw);
                        const bool whole = p.head_dim % C == 0;
#pragma unroll
                        for (int j = 0; j < C; ++j) {
                            if (k0 + j < p.K) f[j] = f[j] * s_head[whole ? k0 / p.head_dim : (k0 + j) / p.head_dim] * hw[j] * (p.gate_sigmoid ? lb_sigmoidf(side[i][j]) : lb_siluf(side[i][j]));
                        }
                    }
                    if (PRO == LB_DPRO_CONV) {
                        float w[C];
                        lb_load_cols<C>(p.conv_w + (size_t)(p.taps - 1) * p.ring_ld, k0, p.K, vec, w);
                        float* slot = conv_ring + (size_t)(pos % p.taps) * p.ring_ld + k0;  // no CTA of this launch reads this slot
#pragma unroll
                        for (int j = 0; j < C; ++j) {
                            if ((kStage || blockIdx.x == 0) && k0 + j < p.K) slot[j] = f[j];
                            f[j] += fmaf(w[j], f[j], side[i][j]);
                        }
                    }
                } else {
#pragma unroll
                    for (int j = 0; j < C; ++j) f[j] = 0.f;
                }
                if (kStage)
                    p.staged[(size_t)c * Mp_launch + tok] = lb_pack_chunk<WT>(f);
                else
                    xs[(size_t)c * Mp + m] = lb_pack_chunk<WT>(f);
            }
        }
        __syncthreads();
    }

    if (kStage) return;

    if (PRO == LB_DPRO_PAIRS) {
        nact = p.list->n;
        for (int i = tid; i < nact; i += kGemvThreads) s_route[i] = p.list->expert[i];
        for (int i = tid; i < nact * kMaxLanesPerPass; i += kGemvThreads) {
            const int m = i % kMaxLanesPerPass;
            s_route[kMaxLanesPerPass * kMaxTop + i] = m < p.M ? p.list->pair[i / kMaxLanesPerPass][m] : -1;
        }
        __syncthreads();
        for (int i = 0; i < depth; ++i) fetch();
    }

    // The next launch may start once this one's input rows are made, not before: its CTAs fetch weights as soon as they sit on an SM,
    // in front of this launch's own.  One sequence, Zitupel of 2560: 538 us a step so, 561 when told at the start, 564 after the
    // products, 580 at the end; two float32 sequences 219, 232, 222, 218.
    lb_pdl_launch_dependents();
    int slot = 0;
    for (; strip - sp < strips; strip += step) {
        // the residual rows are asked for before the products (two strips at most a CTA: one element a thread)
        float before = 0.f;
        const int brow = (strip - sp + (tid >> 7)) * 16 + ((tid & 127) >> 3);
        const bool early_res = EPI == LB_DEPI_RESID && SP <= 2;
        if (early_res && tid < SP * 128 && (tid & 7) < M && brow < p.rows) before = (p.res ? p.res : p.out)[(size_t)(tid & 7) * p.ldo + brow];
        GemvAcc<WT> acc, acc2;
        acc.zero();
        if (kDual) acc2.zero();
        if (strip < strips) {
            const int total = nact * p.slices;
            int at_end = 0, at = -1;  // PAIRS: end of the present expert's slices, its place in the list
            unsigned chose = 0;
            const uint8_t *d1 = strip_ptr(w1, strip) + lane_off, *d2 = kDual ? strip_ptr(w2, strip) + lane_off : nullptr;
            constexpr int kParts = kDual ? 8 : 4, kDirect = kDual ? 1 : 2;
            uint4 ahead[kDirect][kParts];
            auto direct = [&](uint4 (&d)[kParts], int s) {
                if (s >= total) return;
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                    d[u] = ldg_stream(d1 + (size_t)s * kImgBlock + u * 512);
                    if (kDual) d[4 + u] = ldg_stream(d2 + (size_t)s * kImgBlock + u * 512);
                }
            };
            if (!RING)
#pragma unroll
                for (int i = 0; i < kDirect; ++i) direct(ahead[i], kw + i * KW);
            for (int s = kw; s < total; s += KW) {
                uint4 w[8];
                const uint4* rs = reinterpret_cast<const uint4*>(ring + (size_t)slot * kUnits * kRingUnit);
                if (RING) {
                    ring_wait(depth);
                    __syncwarp();  // a lane reads what other lanes fetched
#pragma unroll
                    for (int u = 0; u < (kDual ? 8 : 4); ++u) w[u] = rs[u * kGemvThreads + at_read];
                } else {
#pragma unroll
                    for (int u = 0; u < kParts; ++u) w[u] = ahead[0][u];
#pragma unroll
                    for (int i = 0; i + 1 < kDirect; ++i)
#pragma unroll
                        for (int u = 0; u < kParts; ++u) ahead[i][u] = ahead[i + 1][u];
                    direct(ahead[kDirect - 1], s + kDirect * KW);
                }
                if (PRO == LB_DPRO_PAIRS) {
                    if (s >= at_end) {  // (KW <= slices: the next expert, never one further)
                        at_end += p.slices;
                        ++at;
                        chose = __ballot_sync(0xffffffffu, lane < kMaxLanesPerPass && s_route[kMaxLanesPerPass * kMaxTop + at * kMaxLanesPerPass + (lane & 7)] >= 0);
                    }
                    step_pairs<WT>(acc, w[0], w[2], rs + 4 * kGemvThreads, chose, lane);
                    step_pairs<WT>(acc, w[1], w[3], rs + 5 * kGemvThreads, chose, lane);
                } else {
                    const uint4* x0 = xs + (size_t)(s * 8 + t) * Mp;
                    acc.step(w[0], w[2], x0, Mp, M, g);
                    acc.step(w[1], w[3], x0 + 4 * Mp, Mp, M, g);
                    if (kDual) {
                        acc2.step(w[4], w[6], x0, Mp, M, g);
                        acc2.step(w[5], w[7], x0 + 4 * Mp, Mp, M, g);
                    }
                }
                if (RING) {
                    slot = slot + 1 == depth ? 0 : slot + 1;
                    __syncwarp();  // every lane has read the slot that is filled again
                    fetch();
                }
            }
        }
        __syncthreads();  // the previous strip's sums are no longer read
        acc.store(red[warp], g, t);
        if (kDual) acc2.store(red2[warp], g, t);
        __syncthreads();
        for (int o = tid; o < SP * 128; o += kGemvThreads) {
            const int s = o >> 7, e = o & 127, r = e >> 3, m = e & 7;
            const int row = (strip - sp + s) * 16 + r;
            if (m >= M || row >= p.rows) continue;
            float v = 0.f, u = 0.f;
            for (int k = 0; k < KW; ++k) {
                v += red[s * KW + k][e];
                if (kDual) u += red2[s * KW + k][e];
            }
            if (EPI == LB_DEPI_F32) p.out[(size_t)m * p.ldo + row] = v;
            if (EPI == LB_DEPI_RESID) {
                const size_t at = (size_t)m * p.ldo + row;
                p.out[at] = fmaf(p.mult, v, p.res_mult * (early_res ? before : (p.res ? p.res : p.out)[at]));
            }
            if (EPI == LB_DEPI_GELU) p.out[(size_t)m * p.ldo + row] = lb_gelu_erff(v);
            if (EPI == LB_DEPI_SILU) p.out[(size_t)m * p.ldo + row] = lb_siluf(v) * u;
            if (EPI == LB_DEPI_GLU) {
                reinterpret_cast<WT*>(p.out_pairs)[(size_t)s_pair[m] * p.ldo + row] = (WT)lb_clamped_glu(v, u, p.limit);
            }
        }
    }
}

constexpr int kStageTokens = 3;  // from this many tokens on the input rows are made once, by a launch of their own

template <typename WT, int PRO, int EPI>
int gemv_launch(loom_b200_ctx* ctx, const LbDenseGemv& pin) {
    LbDenseGemv p = pin;
    LB_REQUIRE(ctx, p.M >= 1 && p.M <= kMaxLanesPerPass, "dense_gemv: %d tokens", p.M);
    int Mp = 1;
    while (Mp < p.M) Mp *= 2;
    const int strips = lb_ceil_div(p.rows, 16), cap = ctx->sm_count * 2;
    int KW = 1;
    while (KW < kGemvWarps && KW * 2 <= p.slices) KW *= 2;
    // many strips per CTA: fewer warps per strip, so that a warp streams longer runs between two meetings of the sums
    while (KW > 1 && (long long)strips >= 6ll * (2 * kGemvWarps / KW) * cap) KW /= 2;
    const int SP = kGemvWarps / KW;
    bool vec = PRO == LB_DPRO_STAGED || PRO == LB_DPRO_PAIRS || lb_vec_rows(p.x, p.ldx);
    if (PRO == LB_DPRO_GATED) vec = vec && lb_vec_rows(p.gate, p.gate_ld) && lb_vec_rows(p.head_w, 4);
    if (p.gain_w) vec = vec && lb_vec_rows(p.gain_w, 4);
    if (PRO == LB_DPRO_CONV) vec = vec && lb_vec_rows(p.conv_w, p.ring_ld) && lb_vec_rows(p.conv_ring, p.ring_ld);
    const size_t rows_smem = (size_t)p.slices * 8 * (EPI == LB_DEPI_STAGE ? 1 : Mp) * 16;
    size_t smem = PRO == LB_DPRO_PAIRS || EPI == LB_DEPI_STAGE ? 0 : rows_smem;
    if (PRO == LB_DPRO_MOE) smem += (size_t)p.M * p.experts * 4 + (size_t)p.M * p.top * 4;
    if (PRO == LB_DPRO_GATED) smem = rows_smem + (size_t)Mp * (p.K / p.head_dim) * 4;
    if (smem > kGemvSmemX + 16 * 1024) return lb_fail(ctx, LOOM_B200_ERR_UNSUPPORTED, "dense_gemv: %d tokens of %d columns need %zu B of shared memory", p.M, p.K, smem);
    // the weight ring takes what the input rows leave: of half an SM's shared memory if that is room for two slices, else of all
    constexpr bool kPairs = PRO == LB_DPRO_PAIRS;
    constexpr int kSlot = (EPI == LB_DEPI_GLU || EPI == LB_DEPI_SILU ? 8 : kPairs ? 6 : 4) * kRingUnit;
    int depth = 0;
    const int ring_off = kPairs ? kMaxLanesPerPass * kMaxTop * (1 + kMaxLanesPerPass) * 4 : lb_round_up((int)smem, 16);
    if (EPI != LB_DEPI_STAGE) {
        const int room = ring_off + 2 * kSlot <= kGemvSmemHalf ? kGemvSmemHalf : (int)kGemvSmemX + 16 * 1024;
        depth = room > ring_off ? (room - ring_off) / kSlot : 0;
        if (depth > kRingMax) depth = kRingMax;
        if (depth < 2) depth = 0;
        smem = (size_t)ring_off + (size_t)depth * kSlot;
    }
    constexpr bool kStage = EPI == LB_DEPI_STAGE, kNoRing = !kPairs && !kStage;  // (routed pairs always have their slots, staging multiplies nothing)
    const bool direct = kNoRing && depth == 0;
    if (direct) {
        LB_BIG_SMEM(ctx, (lb_dense_gemv_kernel<WT, PRO, EPI, !kNoRing>), kGemvSmemX + 16 * 1024);
    } else if (smem > 36 * 1024) {
        LB_BIG_SMEM(ctx, (lb_dense_gemv_kernel<WT, PRO, EPI, true>), kGemvSmemX + 16 * 1024);
    }
    int gx = lb_ceil_div(strips, SP), gy = 1, share = cap;
    if (EPI == LB_DEPI_STAGE) {
        gx = share = p.M;
    } else if (PRO == LB_DPRO_MOE) {
        gy = p.M * p.top;
        share = cap / (gy < p.experts ? gy : p.experts);
        if (share < 1) share = 1;
    }
    if (gx > share) gx = lb_ceil_div(gx, lb_ceil_div(gx, share));  // equal numbers of strips per CTA
    if (direct) {
        LB_LAUNCH(ctx, (lb_dense_gemv_kernel<WT, PRO, EPI, !kNoRing>), dim3(gx, gy), dim3(kGemvThreads), smem, p, Mp, KW, vec, ring_off, depth);
        return 0;
    }
    LB_LAUNCH(ctx, (lb_dense_gemv_kernel<WT, PRO, EPI, true>), dim3(gx, gy), dim3(kGemvThreads), smem, p, Mp, KW, vec, ring_off, depth);
    return 0;
}

// a product whose input rows take some work: inside every CTA for one or two tokens, as a launch of their own for more
template <typename WT, int PRO, int EPI>
int gemv_rows(loom_b200_ctx* ctx, const LbDenseGemv& pin) {
    if (pin.M < kStageTokens) return gemv_launch<WT, PRO, EPI>(ctx, pin);
    LbDenseGemv p = pin;
    const size_t bytes = (size_t)p.slices * 8 * kMaxLanesPerPass * 16;
    if (int rc = lb_grow(ctx, &ctx->stage_scratch, &ctx->stage_scratch_bytes, bytes, bytes, "the staging buffer of the GEMV")) return rc;
    p.staged = static_cast<uint4*>(ctx->stage_scratch);
    if (int rc = gemv_launch<WT, PRO, LB_DEPI_STAGE>(ctx, p)) return rc;
    return gemv_launch<WT, LB_DPRO_STAGED, EPI>(ctx, p);
}

template <typename WT>
int gemv_dispatch(loom_b200_ctx* ctx, int pro, int epi, const LbDenseGemv& p) {
#define LB_CASE(P, E, RUN) \
    if (pro == P && epi == E) return RUN<WT, P, E>(ctx, p)
    LB_CASE(LB_DPRO_CONV, LB_DEPI_F32, gemv_rows);
    LB_CASE(LB_DPRO_NORM, LB_DEPI_F32, gemv_rows);
    LB_CASE(LB_DPRO_NORM, LB_DEPI_GELU, gemv_rows);
    LB_CASE(LB_DPRO_NORM, LB_DEPI_SILU, gemv_rows);
    LB_CASE(LB_DPRO_PLAIN, LB_DEPI_F32, gemv_launch);
    LB_CASE(LB_DPRO_PLAIN, LB_DEPI_RESID, gemv_launch);
    LB_CASE(LB_DPRO_GATED, LB_DEPI_RESID, gemv_rows);
    LB_CASE(LB_DPRO_MOE, LB_DEPI_GLU, gemv_launch);
    LB_CASE(LB_DPRO_PAIRS, LB_DEPI_RESID, gemv_launch);
#undef LB_CASE
    return lb_fail(ctx, LOOM_B200_ERR_UNSUPPORTED, "dense_gemv: prologue %d with epilogue %d is not built", pro, epi);
}

// ---- token-block GEMM with plain fused multiply-adds (32-bit floats) -------------------------------------------
//
// Bound by the multiply-adds (74 TFLOP/s) once the loads are hidden: K slices arrive by asynchronous copies, two ahead, in the
// image's own order; a thread owns 8 tokens x 4 rows and multiplies two columns at a time (packed multiply-adds on register pairs
// as they were loaded), 12 shared-memory reads of one wavefront each for 64 of them.  Few tiles are split over K by the CTAs of a
// cluster, which meet in shared memory in the order of K.  The former kernel (2 x 8 per thread, one slice at a time between two
// barriers) took 159 us for 333 tokens x 1024 rows x 2816 columns, this one 69 us (gate and up of 2816 together 145 and 127 us).

constexpr int kSimtTile = 64, kSimtThreads = 128, kSimtStages = 3, kSimtHalf = kSimtTile * 128, kSimtLd = kSimtTile + 4;

__device__ __forceinline__ float4 simt_peer(uint32_t addr, uint32_t rank) {
    const uint32_t a = lb_cluster_addr(addr, rank);
    float4 v;
    asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(a) : "memory");
    return v;
}
// a 16-byte chunk as pairs of floats
template <typename WT>
__device__ __forceinline__ void simt_pairs(const uint8_t* p, uint64_t* f);
template <>
__device__ __forceinline__ void simt_pairs<float>(const uint8_t* p, uint64_t* f) {
    const ulonglong2 v = *reinterpret_cast<const ulonglong2*>(p);
    f[0] = v.x;
    f[1] = v.y;
}
template <>
__device__ __forceinline__ void simt_pairs<__nv_bfloat16>(const uint8_t* p, uint64_t* f) {
    float v[8];
    lb_unpack_chunk<__nv_bfloat16>(*reinterpret_cast<const uint4*>(p), v);
#pragma unroll
    for (int i = 0; i < 4; ++i) f[i] = lb_pack2(v[2 * i], v[2 * i + 1]);
}

// grid: (row tiles x S, token tiles), clusters of S CTAs along x
template <typename WT, int EPI>
__global__ void __launch_bounds__(kSimtThreads, EPI == LB_DEPI_GLU || EPI == LB_DEPI_SILU ? 2 : 3) lb_dense_gemm_simt_kernel(const LbDenseGemm p, int S) {
    constexpr int P = LbElem<WT>::kChunk / 2;
    constexpr bool kDual = EPI == LB_DEPI_GLU || EPI == LB_DEPI_SILU;
    constexpr int kParts = kDual ? 3 : 2;
    extern __shared__ __align__(16) uint8_t smem[];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const uint32_t rank = S > 1 ? lb_cluster_rank() : 0;
    const int row0 = (int)(blockIdx.x / S) * kSimtTile, tok0 = blockIdx.y * kSimtTile;
    lb_pdl_launch_dependents();
    lb_pdl_wait();
    const uint8_t *w = p.w, *w2 = p.w2;
    if (p.nblocks) {
        if (tok0 / kImgRows >= *p.nblocks) return;  // (the whole cluster)
        const size_t off = (size_t)p.block_group[tok0 / kImgRows] * p.group_bytes;
        w += off;
        w2 += kDual ? off : 0;
    }
    const size_t abase = (size_t)(tok0 >> 7) * p.slices * kImgBlock + (size_t)((tok0 & 127) >> 3) * 1024;
    const size_t bbase = (size_t)(row0 >> 7) * p.slices * kImgBlock + (size_t)((row0 & 127) >> 3) * 1024;
    const int first = p.slices * (int)rank / S, last = p.slices * ((int)rank + 1) / S;
    const uint32_t base = lb_smem_u32(smem);
    auto fetch = [&](int s) {
        if (s < last) {
            const uint32_t dst = base + (uint32_t)((s - first) % kSimtStages * kParts * kSimtHalf);
            const size_t off = (size_t)s * kImgBlock;
#pragma unroll
            for (int i = 0; i < kSimtHalf / 16 / kSimtThreads; ++i) {
                const int at = (tid + i * kSimtThreads) * 16;
                ring_copy(dst + at, p.x + abase + off + at);
                ring_copy(dst + kSimtHalf + at, w + bbase + off + at);
                if (kDual) ring_copy(dst + 2 * kSimtHalf + at, w2 + bbase + off + at);
            }
        }
        ring_commit();
    };
    // tokens tq + 8 i, rows rq + 8 j + 32 (warp / 2)
    const int tq = (lane >> 3) + 4 * (warp & 1), rq = lane & 7, rh = warp >> 1;
    uint64_t acc[8][4], acc2[kDual ? 8 : 1][4];
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            acc[i][j] = 0;
            if (kDual) acc2[i][j] = 0;
        }
    for (int i = 0; i < kSimtStages - 1; ++i) fetch(first + i);
    for (int s = first; s < last; ++s) {
        asm volatile("cp.async.wait_group %0;" ::"n"(kSimtStages - 2) : "memory");
        __syncthreads();  // slice s is there for everyone, and everyone is done with the slot that is filled next
        fetch(s + kSimtStages - 1);
        const uint8_t* sa = smem + (s - first) % kSimtStages * kParts * kSimtHalf;
        const uint8_t* xa = sa + tq * 16;
        const uint8_t* wa = sa + kSimtHalf + rh * 4096 + rq * 16;
#pragma unroll 2
        for (int c = 0; c < 8; ++c) {
            uint64_t a[8][P], b[4][P];
#pragma unroll
            for (int i = 0; i < 8; ++i) simt_pairs<WT>(xa + i * 1024 + c * 128, a[i]);
#pragma unroll
            for (int j = 0; j < 4; ++j) simt_pairs<WT>(wa + j * 1024 + c * 128, b[j]);
#pragma unroll
            for (int h = 0; h < P; ++h)
#pragma unroll
                for (int i = 0; i < 8; ++i)
#pragma unroll
                    for (int j = 0; j < 4; ++j) acc[i][j] = lb_fma2(a[i][h], b[j][h], acc[i][j]);
            if (kDual) {
#pragma unroll
                for (int j = 0; j < 4; ++j) simt_pairs<WT>(wa + kSimtHalf + j * 1024 + c * 128, b[j]);
#pragma unroll
                for (int h = 0; h < P; ++h)
#pragma unroll
                    for (int i = 0; i < 8; ++i)
#pragma unroll
                        for (int j = 0; j < 4; ++j) acc2[i][j] = lb_fma2(a[i][h], b[j][h], acc2[i][j]);
            }
        }
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();
    // the sums go through shared memory: eight consecutive rows of a token are one thread's to write
    float* tile = reinterpret_cast<float*>(smem);  // [64 tokens][64 rows], a second one for the second product
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int at = (tq + 8 * i) * kSimtLd + rq + 8 * j + 32 * rh;
            float lo, hi;
            lb_unpack2(acc[i][j], lo, hi);
            tile[at] = lo + hi;
            if (kDual) {
                lb_unpack2(acc2[i][j], lo, hi);
                tile[kSimtTile * kSimtLd + at] = lo + hi;
            }
        }
    if (S > 1)
        lb_cluster_sync();
    else
        __syncthreads();
    const int per = 512 / S;  // (token, eight rows) pairs of a CTA
    for (int idx = (int)rank * per + tid; idx < ((int)rank + 1) * per; idx += kSimtThreads) {
        const int tk = idx >> 3, r8 = (idx & 7) * 8;
        float v[8], u[8];
#pragma unroll
        for (int d = 0; d < (kDual ? 2 : 1); ++d) {
            float* f = d ? u : v;
            const uint32_t at = base + (uint32_t)(d * kSimtTile * kSimtLd + tk * kSimtLd + r8) * 4;
#pragma unroll
            for (int j = 0; j < 8; ++j) f[j] = 0.f;
            for (int q = 0; q < S; ++q) {
                float4 lo, hi;
                if (S > 1) {
                    lo = simt_peer(at, (uint32_t)q);
                    hi = simt_peer(at + 16, (uint32_t)q);
                } else {
                    const float4* o = reinterpret_cast<const float4*>(tile + d * kSimtTile * kSimtLd + tk * kSimtLd + r8);
                    lo = o[0];
                    hi = o[1];
                }
                f[0] += lo.x;
                f[1] += lo.y;
                f[2] += lo.z;
                f[3] += lo.w;
                f[4] += hi.x;
                f[5] += hi.y;
                f[6] += hi.z;
                f[7] += hi.w;
            }
        }
        const int tok = tok0 + tk, r = row0 + r8;
        if (!p.nblocks && tok >= p.tokens) continue;
        if (EPI == LB_DEPI_F32 || EPI == LB_DEPI_RESID) {
            if (r >= p.ldo) continue;
            float* o = p.out + (size_t)tok * p.ldo + r;
#pragma unroll
            for (int j = 0; j < 8; ++j) o[j] = EPI == LB_DEPI_F32 ? v[j] : fmaf(p.mult, v[j], p.res_mult * o[j]);
        } else {
            float f[8];
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                f[j] = v[j];
                if (EPI == LB_DEPI_GELU) f[j] = lb_gelu_erff(v[j]);
                if (EPI == LB_DEPI_GLU) f[j] = lb_clamped_glu(v[j], u[j], p.limit);
                if (EPI == LB_DEPI_SILU) f[j] = lb_siluf(v[j]) * u[j];
            }
            if (EPI == LB_DEPI_HEADS) {
                if (r < p.rows) *reinterpret_cast<uint4*>(p.img + lb_heads_chunk(tok, r, p.heads, p.head_dim, p.head_chunks)) = lb_pack_chunk<__nv_bfloat16>(f);
            } else if (r / LbElem<WT>::kSlice < p.img_slices) {
                lb_img_store8<WT>(p.img, tok, r, p.img_slices, f);
            }
        }
    }
    if (S > 1)  // a neighbour may still read this CTA's sums
        lb_cluster_sync();
}

template <typename WT, int EPI>
int gemm_simt_launch(loom_b200_ctx* ctx, const LbDenseGemm& p) {
    constexpr bool kDual = EPI == LB_DEPI_GLU || EPI == LB_DEPI_SILU;
    constexpr size_t kSmem = (size_t)kSimtStages * (kDual ? 3 : 2) * kSimtHalf;
    static_assert(kSmem >= (kDual ? 2 : 1) * kSimtTile * kSimtLd * sizeof(float), "the sums fit the stages");
    // rows: every 64-row tile that holds a row or a column of the output image's padding
    const int tiles = lb_ceil_div(p.rows, kSimtTile), blocks = p.nblocks ? p.max_blocks * 2 : lb_ceil_div(p.tokens, kSimtTile);
    // CTAs that share a tile: as many as the SMs hold at once (two or three CTAs each), four slices each at least
    int S = 1;
    while (S < 8 && (long long)tiles * blocks * S * 2 <= (kDual ? 2ll : 3ll) * ctx->sm_count && p.slices / (S * 2) >= 4) S *= 2;
    LB_BIG_SMEM(ctx, (lb_dense_gemm_simt_kernel<WT, EPI>), kSmem);
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(tiles * S, blocks);
    cfg.blockDim = dim3(kSimtThreads);
    cfg.dynamicSmemBytes = kSmem;
    cfg.stream = ctx->stream;
    cudaLaunchAttribute attr[2];
    int n = 0;
    if (S > 1) {
        attr[n].id = cudaLaunchAttributeClusterDimension;
        attr[n].val.clusterDim.x = S;
        attr[n].val.clusterDim.y = attr[n].val.clusterDim.z = 1;
        ++n;
    }
    if (ctx->opt_pdl) {
        attr[n].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[n].val.programmaticStreamSerializationAllowed = 1;
        ++n;
    }
    cfg.attrs = attr;
    cfg.numAttrs = n;
    LB_CUDA(ctx, cudaLaunchKernelEx(&cfg, lb_dense_gemm_simt_kernel<WT, EPI>, p, S));
    ctx->launches++;
    return 0;
}

template <typename WT>
int gemm_simt(loom_b200_ctx* ctx, int epi, const LbDenseGemm& p) {
    switch (epi) {
        case LB_DEPI_F32: return gemm_simt_launch<WT, LB_DEPI_F32>(ctx, p);
        case LB_DEPI_RESID: return gemm_simt_launch<WT, LB_DEPI_RESID>(ctx, p);
        case LB_DEPI_GELU: return gemm_simt_launch<WT, LB_DEPI_GELU>(ctx, p);
        case LB_DEPI_GLU: return gemm_simt_launch<WT, LB_DEPI_GLU>(ctx, p);
        case LB_DEPI_SILU: return gemm_simt_launch<WT, LB_DEPI_SILU>(ctx, p);
        case LB_DEPI_IMG: return gemm_simt_launch<WT, LB_DEPI_IMG>(ctx, p);
        case LB_DEPI_HEADS: return gemm_simt_launch<WT, LB_DEPI_HEADS>(ctx, p);
    }
    return lb_fail(ctx, LOOM_B200_ERR_UNSUPPORTED, "dense_gemm: epilogue %d is not built", epi);
}

}  // namespace

int lb_gemm_bf16_run(loom_b200_ctx* ctx, int epi, const LbDenseGemm& p);  // gemm_bf16.cu

int lb_dense_gemv_max_tokens(int K, int dtype) {
    const size_t row = (size_t)lb_slices_of(K, dtype) * 128;
    int m = kMaxLanesPerPass;
    while (m > 1 && (size_t)m * row > kGemvSmemX) m /= 2;
    return m;
}

int lb_dense_gemv(loom_b200_ctx* ctx, int dtype, int pro, int epi, const LbDenseGemv& p) {
    return dtype == LOOM_B200_DTYPE_BF16 ? gemv_dispatch<__nv_bfloat16>(ctx, pro, epi, p) : gemv_dispatch<float>(ctx, pro, epi, p);
}

int lb_dense_gemm(loom_b200_ctx* ctx, int dtype, int epi, const LbDenseGemm& pin) {
    LbDenseGemm p = pin;
    p.status = ctx->status_dev;
    LB_REQUIRE(ctx, p.x && p.w && p.rows > 0 && p.slices > 0 && (p.tokens > 0 || p.nblocks), "dense_gemm: bad arguments");
    LB_REQUIRE(ctx, (epi != LB_DEPI_F32 && epi != LB_DEPI_RESID) || p.ldo % 8 == 0, "dense_gemm: output rows of %d floats", p.ldo);
    if (dtype == LOOM_B200_DTYPE_F32) return gemm_simt<float>(ctx, epi, p);
    if (!ctx->opt_dense_tc) return gemm_simt<__nv_bfloat16>(ctx, epi, p);
    return lb_gemm_bf16_run(ctx, epi, p);
}

extern "C" {

int loom_b200_matrix_create(loom_b200_ctx* ctx, int rows, int cols, int groups, int dtype, loom_b200_matrix** out) {
    if (!ctx) return lb_fail(nullptr, LOOM_B200_ERR_INVALID, "matrix_create: ctx is NULL");
    LB_REQUIRE(ctx, out != nullptr, "matrix_create: out is NULL");
    *out = nullptr;
    LB_REQUIRE(ctx, rows > 0 && cols > 0 && groups > 0, "matrix_create: bad shape %dx%d (%d groups)", rows, cols, groups);
    LB_REQUIRE(ctx, dtype == LOOM_B200_DTYPE_F32 || dtype == LOOM_B200_DTYPE_BF16, "matrix_create: dtype %d", dtype);
    if (ctx->capturing) return lb_fail(ctx, LOOM_B200_ERR_INVALID, "matrix_create cannot be recorded");
    if (int rc = lb_set_device(ctx)) return rc;
    auto* m = new loom_b200_matrix();
    m->rows = rows;
    m->cols = cols;
    m->groups = groups;
    m->dtype = dtype;
    m->slices = lb_slices_of(cols, dtype);
    m->group_bytes = lb_img_bytes(rows, cols, dtype);
    m->device = ctx->device;
    const size_t bytes = m->group_bytes * groups;
    cudaError_t e = cudaMalloc(&m->data, bytes);
    if (e == cudaSuccess) e = cudaMemsetAsync(m->data, 0, bytes, ctx->stream);
    if (e != cudaSuccess) {
        if (m->data) cudaFree(m->data);
        delete m;
        return lb_fail(ctx, LOOM_B200_ERR_CUDA, "matrix_create: %zu bytes: %s", bytes, cudaGetErrorString(e));
    }
    *out = m;
    return 0;
}

int loom_b200_matrix_put(loom_b200_ctx* ctx, loom_b200_matrix* m, int group, int row0, int rows, const void* src, int src_dtype, int src_on_device) {
    if (!ctx) return lb_fail(nullptr, LOOM_B200_ERR_INVALID, "matrix_put: ctx is NULL");
    LB_REQUIRE(ctx, m && src, "matrix_put: NULL argument");
    LB_REQUIRE(ctx, group >= 0 && group < m->groups && row0 >= 0 && rows > 0 && row0 + rows <= m->rows, "matrix_put: rows %d..%d of group %d in %dx%d (%d groups)",
               row0, row0 + rows, group, m->rows, m->cols, m->groups);
    LB_REQUIRE(ctx, src_dtype == LOOM_B200_DTYPE_F32 || src_dtype == LOOM_B200_DTYPE_BF16, "matrix_put: dtype %d", src_dtype);
    LB_REQUIRE(ctx, m->device == ctx->device, "matrix_put: matrix lives on device %d", m->device);
    if (ctx->capturing) return lb_fail(ctx, LOOM_B200_ERR_INVALID, "matrix_put cannot be recorded");
    if (int rc = lb_set_device(ctx)) return rc;
    const size_t bytes = (size_t)rows * m->cols * (src_dtype == LOOM_B200_DTYPE_BF16 ? 2 : 4);
    const void* dev = src;
    if (!src_on_device) {
        if (int rc = lb_ensure_scratch(ctx, bytes)) return rc;
        LB_CUDA(ctx, cudaMemcpyAsync(ctx->scratch, src, bytes, cudaMemcpyHostToDevice, ctx->stream));
        dev = ctx->scratch;
    }
    const size_t threads = (size_t)rows * m->slices * 8;
    const unsigned grid = (unsigned)((threads + 255) / 256);
    uint8_t* img = m->data + (size_t)group * m->group_bytes;
    if (m->dtype == LOOM_B200_DTYPE_BF16)
        lb_image_put_kernel<__nv_bfloat16><<<grid, 256, 0, ctx->stream>>>(dev, src_dtype, rows, m->cols, row0, m->slices, img);
    else
        lb_image_put_kernel<float><<<grid, 256, 0, ctx->stream>>>(dev, src_dtype, rows, m->cols, row0, m->slices, img);
    LB_CHECK_LAUNCH(ctx, "lb_image_put_kernel");
    LB_CUDA(ctx, cudaStreamSynchronize(ctx->stream));
    return 0;
}

int loom_b200_matrix_info(const loom_b200_matrix* m, int* rows, int* cols, int* groups, int* dtype) {
    if (!m) return lb_fail(nullptr, LOOM_B200_ERR_INVALID, "matrix_info: matrix is NULL");
    if (rows) *rows = m->rows;
    if (cols) *cols = m->cols;
    if (groups) *groups = m->groups;
    if (dtype) *dtype = m->dtype;
    return 0;
}

void loom_b200_matrix_free(loom_b200_ctx* ctx, loom_b200_matrix* m) {
    if (!m) return;
    if (ctx) {
        cudaSetDevice(ctx->device);
        cudaStreamSynchronize(ctx->stream);
    }
    if (m->data) cudaFree(m->data);
    delete m;
}

}  // extern "C"

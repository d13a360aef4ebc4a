// attention_decode.cu -- causal GQA attention of ONE new token over the fp32 KV ring, as a thread-block cluster.
//
// Arithmetic: poly/mha.go:292-354 (RoPE of the query and of the newest K row in float64, scores dot(Q, K_f32) / sqrt(hd),
// max-subtracted exp, sum(p*V) / sum(p), all float64 over float32 K/V rows).  Replaces the decode use of the WGSL
// tiled attention (ShaderTiledMHAN, poly/wgpu_shaders.go:1112-1388).
//
// Shape of the kernel
//   * One cluster per KV head and sequence; the S CTAs of a cluster split the positions 0..pos into S contiguous slices.
//     A CTA brings its K and V rows into shared memory with ONE bulk async copy each (the ring is head-major, so a slice is
//     one contiguous block) and serves all query heads of the GQA group from them: every K/V element is converted
//     to float64 once and used by every head of the group.  A slice that does not fit goes through in chunks with a running
//     softmax: the next K rows travel behind softmax and weighted V, the next V rows behind the next scores.
//     (Eight query heads per KV head over several chunks: two clusters of four heads each.)
//   * S: one sequence takes the largest cluster of which the device holds one per KV head; a pass of several takes the
//     largest of which it holds one per (sequence, KV head), down to single CTAs (eight sequences x eight KV heads: pairs).
//   * Bound: float64 issue and the float32 -> float64 conversions (16 lanes a clock) behind one another's latencies.  Measured:
//     five KV heads, context 1040, MaxSeqLen 4096: 10.9 us where the split kernel took 14.1 (no cluster held such a ring before);
//     eight sequences x eight KV heads at context 2048, pairs of CTAs: 58 us (2.3 TB/s) where one streaming CTA each took 101
//     (41 with lb_attention_stream_kernel, which takes passes of several sequences where a slice's scores fit in shared memory).
//   * Scores: a warp owns a position at a time, a lane four dimensions of it (the query slices live in registers);
//     sixteen (position, head) sums are reduced across the warp together so that the shuffle count per position stays small.
//   * The S partial results (max, sum, weighted V) never touch global memory: every CTA stores its partials straight
//     into the shared memory of the CTA that owns the output dimensions (distributed shared memory), one cluster
//     barrier orders the stores, and every CTA combines and writes hd/S dimensions of every head.  No atomics, no
//     last-arriver re-read, no global scratch.
//   * The K/V rows of the NEXT decoder block are prefetched into L2 while this block computes.
// The per-(head, split) kernel in glue.cu stays for chunks of several tokens, q/k norms and shapes this one refuses.
#include "glue.cuh"

namespace {

constexpr int kAcThreads = 512;
constexpr int kAcWarps = kAcThreads / 32;
constexpr int kAcMaxG = 8;   // query heads per KV head
constexpr int kAcMaxS = 16;  // CTAs per cluster

__device__ __forceinline__ uint32_t cluster_nctarank() {
    uint32_t r;
    asm volatile("mov.u32 %0, %%cluster_nctarank;" : "=r"(r));
    return r;
}
// address of the same shared-memory location in CTA `rank` of this cluster
__device__ __forceinline__ uint32_t map_to_rank(const void* smem_ptr, uint32_t rank) {
    return lb_cluster_addr(lb_smem_u32(smem_ptr), rank);
}
__device__ __forceinline__ void st_cluster_f64(uint32_t addr, double v) {
    asm volatile("st.shared::cluster.f64 [%0], %1;" ::"r"(addr), "d"(v) : "memory");
}
__device__ __forceinline__ void l2_prefetch(const void* gptr, uint32_t bytes) {
    asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(gptr), "r"(bytes) : "memory");
}

// Sums NV = 4*G values per lane across the 32 lanes of a warp.  Each step halves the values a lane carries (it keeps
// one half and sends the other to its partner), so NV values cost about NV double shuffles instead of 5*NV.  Afterwards
// lane L holds, in v[0], the complete sum of value index(L); lanes that differ only in the low (5 - log2 NV) bits hold the same.
template <int NV>
__device__ __forceinline__ void warp_reduce_halving(double (&v)[NV], int lane) {
    int off = 16;
#pragma unroll
    for (int n = NV; n > 1; n >>= 1) {
        const int half = n >> 1;
        const bool upper = (lane & off) != 0;
#pragma unroll
        for (int i = 0; i < half; ++i) {
            const double send = upper ? v[i] : v[i + half];
            const double keep = upper ? v[i + half] : v[i];
            v[i] = keep + __shfl_xor_sync(0xffffffffu, send, off);
        }
        off >>= 1;
    }
    for (; off > 0; off >>= 1) v[0] += __shfl_xor_sync(0xffffffffu, v[0], off);
}
// the value index lane L ends up with: one index bit per halving step, taken from the lane bits 16, 8, 4, ...
template <int NV>
__device__ __forceinline__ int halving_index(int lane) {
    int idx = 0, off = 16;
#pragma unroll
    for (int n = NV; n > 1; n >>= 1) {
        idx += (lane & off) ? (n >> 1) : 0;
        off >>= 1;
    }
    return idx;
}

// A CTA's maxima, sums and weighted sums over its slice meet those of the other CTAs of the cluster: every CTA writes hd / S dimensions.
template <int G, bool LEAN>
__device__ __forceinline__ void finish_cluster(const LbAttnParams& p, const double (&acc)[G][4], double* red, double* part, const double* s_m, const double* s_l, double* s_gw, int cnt, int n) {
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, hd = p.hd, kvh = blockIdx.y;
    const uint32_t rank = lb_cluster_rank(), S = cluster_nctarank();
    const int dps = hd / (int)S;
    const bool lane_on = 4 * lane < hd;
    __syncthreads();  // every warp is done with the K and V tiles: the reduction buffer takes their place
    if (lane_on) {
#pragma unroll
        for (int g = 0; g < G; ++g)
            *reinterpret_cast<double4*>(red + ((size_t)warp * G + g) * hd + 4 * lane) = make_double4(acc[g][0], acc[g][1], acc[g][2], acc[g][3]);
    }
    __syncthreads();
    if (!LEAN) lb_trace(p.trace, 4);

    // ---- hand this slice's partials to the CTAs that own the output dimensions ----
    asm volatile("barrier.cluster.wait.aligned;" ::: "memory");  // completes the arrive at the top: every CTA has started
    // part[(slice * G + g) * (dps + 2)] = { max, sum, dps weighted-V values } in the receiving CTA's shared memory
    for (int idx = tid; idx < G * hd; idx += kAcThreads) {
        const int g = idx / hd, d = idx - g * hd;
        double v = 0.0;
#pragma unroll 4
        for (int w = 0; w < kAcWarps; ++w) v += red[((size_t)w * G + g) * hd + d];  // fixed order: the same bits on every replay
        const uint32_t owner = (uint32_t)(d / dps);
        st_cluster_f64(map_to_rank(part + ((size_t)rank * G + g) * (dps + 2) + 2 + (d - (int)owner * dps), owner), v);
    }
    for (int idx = tid; idx < (int)S * G; idx += kAcThreads) {
        const uint32_t owner = (uint32_t)(idx / G);
        const int g = idx - (int)owner * G;
        double* slot = part + ((size_t)rank * G + g) * (dps + 2);
        st_cluster_f64(map_to_rank(slot, owner), cnt > 0 ? s_m[g] : -1e300);
        st_cluster_f64(map_to_rank(slot + 1, owner), cnt > 0 ? s_l[g] : 0.0);
    }
    lb_cluster_sync();

    // ---- combine the S slices for this CTA's dps dimensions of every head ----
    for (int idx = tid; idx < (int)S * G; idx += kAcThreads) {
        const int g = idx % G;
        double gm = -1e300;
        for (int r = 0; r < (int)S; ++r) gm = fmax(gm, part[((size_t)r * G + g) * (dps + 2)]);
        const int r = idx / G;
        const double ms = part[((size_t)r * G + g) * (dps + 2)], ls = part[((size_t)r * G + g) * (dps + 2) + 1];
        s_gw[r * G + g] = ls == 0.0 ? 0.0 : exp(__dsub_rn(ms, gm));
    }
    __syncthreads();
    for (int idx = tid; idx < G * dps; idx += kAcThreads) {
        const int g = idx / dps, dd = idx - g * dps;
        double num = 0.0, dn = 0.0;
        for (int r = 0; r < (int)S; ++r) {
            const double w = s_gw[r * G + g];
            if (w != 0.0) {  // not an empty slice
                const double* slot = part + ((size_t)r * G + g) * (dps + 2);
                num = fma(slot[2 + dd], w, num);
                dn = fma(slot[1], w, dn);
            }
        }
        p.out[(size_t)n * p.heads * hd + (size_t)(kvh * G + g) * hd + (int)rank * dps + dd] = __ddiv_rn(num, dn);
    }
    if (!LEAN) lb_trace(p.trace, 5);
}

// LEAN: one token of one sequence, no phase trace (what a decode step launches); the code of the other forms is left out.
// (Fixing the head dimension at compile time as well measured no better.)  ONE: a slice always fits in one chunk.
template <int G, bool LEAN, bool ONE>
__global__ void __launch_bounds__(kAcThreads, 1) lb_attention_cluster_kernel(const LbAttnParams p) {
    extern __shared__ __align__(128) uint8_t smem_raw[];
    __shared__ __align__(8) uint64_t bars[2];
    __shared__ double s_red[kAcWarps], s_red2[kAcWarps];  // per-warp maxima, per-warp sums (separate: no barrier between the two reductions)
    __shared__ double s_m[G], s_l[G], s_alpha[G];  // this CTA's running maximum and sum per head, factor of what came before the chunk
    __shared__ double s_gw[kAcMaxS * G];     // combine: weight of every (slice, head)
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int hd = p.hd, half = hd >> 1, kvh = blockIdx.y;  // (group of G query heads)
    const int ring = kvh >> p.kv_shift;                     // its KV head
    const int n = LEAN ? 0 : blockIdx.z;  // token of the pass; with seq_stride > 0 every token is a sequence of its own
    const size_t seq_off = LEAN ? 0 : (size_t)n * (size_t)p.seq_stride;
    const uint32_t rank = lb_cluster_rank(), S = cluster_nctarank();
    const int cmax = p.max_chunk;  // positions one CTA holds at a time
    float* kt = reinterpret_cast<float*>(smem_raw);            // [cmax, hd]
    float* vt = kt + (size_t)cmax * hd;                        // [cmax, hd]
    double* red = reinterpret_cast<double*>(smem_raw);         // after the weighted sums: [warps, G, hd] over the tiles
    double* sq = reinterpret_cast<double*>(smem_raw + p.tile); // p.tile = bytes of the tile / reduction region
    double* sc = sq + G * hd;                                  // [G, cmax] scores, then softmax weights
    double* part = sc + (size_t)G * cmax;                      // [S, G, hd / S + 2] partials received from every slice
    if (tid == 0) {
        lb_mbar_init(&bars[0], 1);
        lb_mbar_init(&bars[1], 1);
        lb_fence_mbar_init();
    }
    __syncthreads();
    // every CTA of the cluster is running before anyone stores into a neighbour's shared memory (waited for below)
    asm volatile("barrier.cluster.arrive.relaxed.aligned;" ::: "memory");
    lb_pdl_launch_dependents();
    lb_pdl_wait();
    if (!LEAN) lb_trace(p.trace, 2);
    const int last = (!LEAN && p.seq_stride > 0) ? p.pos_ptr[n] : *p.pos_ptr;  // the new token's position; it attends to 0..last
    const int total = last + 1;
    const int per = (total + (int)S - 1) / (int)S;
    const int k0 = (int)rank * per;
    int k1 = k0 + per;
    if (k1 > total) k1 = total;
    const int cnt = k1 > k0 ? k1 - k0 : 0;
    const float* kbase = p.cache_k + seq_off + (size_t)ring * p.msl * hd;
    const float* vbase = p.cache_v + seq_off + (size_t)ring * p.msl * hd;
    auto fetch = [&](int which, int c0) {  // the K (0) or V (1) rows of the chunk that starts at c0; one thread
        const uint32_t bytes = (uint32_t)(cnt - c0 < cmax ? cnt - c0 : cmax) * hd * 4;
        lb_mbar_expect_tx(&bars[which], bytes);
        lb_bulk_g2s_stream(which ? vt : kt, (which ? vbase : kbase) + (size_t)(k0 + c0) * hd, bytes, &bars[which], lb_policy_evict_first());
    };
    if (cnt > 0 && lane == 0) {
        if (warp == 0) {
            fetch(0, 0);
        } else if (warp == 1) {
            fetch(1, 0);
        } else if (warp == 2 && p.next_k && ring << p.kv_shift == kvh) {  // the next block's rows of the same positions, into L2
            const uint32_t bytes = (uint32_t)(cnt < p.next_rows ? cnt : p.next_rows) * hd * 4;
            l2_prefetch(p.next_k + ((size_t)ring * p.msl + k0) * hd, bytes);
            l2_prefetch(p.next_v + ((size_t)ring * p.msl + k0) * hd, bytes);
        }
    }
    // queries of the group, rotated (RoPE): thread idx owns the pair (d, d + hd/2) of head g
    double rsn = 0.0, rc = 1.0;
    for (int idx = tid; idx < G * half; idx += kAcThreads) {
        const int g = idx / half, d = idx - g * half;
        double sn, c;
        sincos(__ddiv_rn((double)last, p.rope_div[d]), &sn, &c);
        if (idx < half) {
            rsn = sn;
            rc = c;
        }
        const double* qrow = p.q + (size_t)n * p.heads * hd + (size_t)(kvh * G + g) * hd;
        const double v0 = qrow[d], v1 = qrow[d + half];
        sq[g * hd + d] = __dsub_rn(__dmul_rn(v0, c), __dmul_rn(v1, sn));
        sq[g * hd + d + half] = __dadd_rn(__dmul_rn(v0, sn), __dmul_rn(v1, c));
    }
    if (tid < G) {
        s_m[tid] = -1e300;
        s_l[tid] = 0.0;
    }
    bool failed = false;
    const double scale = __ddiv_rn(1.0, sqrt((double)hd));
    const bool lane_on = 4 * lane < hd;
    double acc[G][4];
#pragma unroll
    for (int g = 0; g < G; ++g)
#pragma unroll
        for (int c = 0; c < 4; ++c) acc[g][c] = 0.0;
    const int vi = halving_index<16>(lane);  // scores: this lane finishes value vi = pp * G + g
    // (ONE: the body runs once even for an empty slice, with no rows)
    for (int c0 = 0, chunk = 0; ONE ? chunk == 0 : c0 < cnt; c0 += cmax, ++chunk) {
        const int rows = ONE ? cnt : cnt - c0 < cmax ? cnt - c0 : cmax;
        const bool more = !ONE && c0 + cmax < cnt;
        if (rows > 0 && !failed && !lb_mbar_wait_bounded(&bars[0], (uint32_t)(chunk & 1))) failed = true;
        if (last >= k0 + c0 && last < k0 + c0 + rows && tid < half) {
            // the newest position belongs to this chunk: its ring row is not written yet; rotate the row the QKV projection
            // left in k_new into the tile and into the ring (threads 0..hd/2-1 hold the sine and cosine of their pair)
            const float* knew = p.k_new + (size_t)n * p.kv_heads * hd + (size_t)ring * hd;
            const double v0 = (double)knew[tid], v1 = (double)knew[tid + half];
            const float r0 = (float)__dsub_rn(__dmul_rn(v0, rc), __dmul_rn(v1, rsn));
            const float r1 = (float)__dadd_rn(__dmul_rn(v0, rsn), __dmul_rn(v1, rc));
            float* trow = kt + (size_t)(last - k0 - c0) * hd;
            trow[tid] = r0;
            trow[tid + half] = r1;
            float* grow = p.cache_k_w + seq_off + ((size_t)ring * p.msl + (size_t)(last % p.msl)) * hd;
            grow[tid] = r0;
            grow[tid + half] = r1;
        }
        __syncthreads();  // the newest row is in the tile; every warp is done with the weights and V rows of the chunk before
        if (!ONE && chunk > 0 && tid == 0 && !failed) {
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            fetch(1, c0);
        }

        // ---- scores: warp = position, lane = four dimensions; PP positions x G heads = 16 sums are reduced together ----
        {
            constexpr int PP = 16 / G;
            double qv[G][4];
#pragma unroll
            for (int g = 0; g < G; ++g)
#pragma unroll
                for (int c = 0; c < 4; ++c) qv[g][c] = lane_on ? sq[g * hd + 4 * lane + c] : 0.0;
            for (int j0 = warp * PP; j0 < rows; j0 += kAcWarps * PP) {
                double sums[16];
#pragma unroll
                for (int pp = 0; pp < PP; ++pp) {
                    float4 kv = make_float4(0.f, 0.f, 0.f, 0.f);
                    if (lane_on && j0 + pp < rows) kv = *reinterpret_cast<const float4*>(kt + (size_t)(j0 + pp) * hd + 4 * lane);
                    const double k0d = (double)kv.x, k1d = (double)kv.y, k2d = (double)kv.z, k3d = (double)kv.w;
#pragma unroll
                    for (int g = 0; g < G; ++g) {
                        double a = __dmul_rn(qv[g][0], k0d);
                        a = fma(qv[g][1], k1d, a);
                        a = fma(qv[g][2], k2d, a);
                        a = fma(qv[g][3], k3d, a);
                        sums[pp * G + g] = a;
                    }
                }
                warp_reduce_halving<16>(sums, lane);
                const int pp = vi / G, g = vi - pp * G;
                if ((lane & 1) == 0 && j0 + pp < rows) sc[g * cmax + j0 + pp] = __dmul_rn(sums[0], scale);
            }
        }
        __syncthreads();  // scores complete, the K rows are free
        if (more && tid == 0 && !failed) {
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            fetch(0, c0 + cmax);
        }
        if (!LEAN) lb_trace(p.trace, 3);

        // ---- running softmax, per head: the warps w with w % G == g share head g ----
        {
            constexpr int WPG = kAcWarps / G;  // warps per head
            const int g = warp % G, wq = warp / G;
            double mx = -1e300;
            for (int j = wq * 32 + lane; j < rows; j += WPG * 32) mx = fmax(mx, sc[g * cmax + j]);
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) mx = fmax(mx, __shfl_xor_sync(0xffffffffu, mx, o));
            if (lane == 0) s_red[warp] = mx;
            __syncthreads();
            mx = s_red[g];
#pragma unroll
            for (int w = 1; w < WPG; ++w) mx = fmax(mx, s_red[g + w * G]);
            const double m_old = s_m[g];
            mx = fmax(mx, m_old);
            double sum = 0.0;
            for (int j = wq * 32 + lane; j < rows; j += WPG * 32) {
                const double e = exp(__dsub_rn(sc[g * cmax + j], mx));
                sc[g * cmax + j] = e;
                sum = __dadd_rn(sum, e);
            }
            sum = lb_warp_sum(sum);
            if (lane == 0) s_red2[warp] = sum;
            __syncthreads();  // (everyone has read the old maximum)
            if (wq == 0 && lane == 0) {  // every warp of head g holds the same maximum
                double l = 0.0;
                for (int w = 0; w < WPG; ++w) l += s_red2[g + w * G];
                if (!ONE && chunk > 0) {
                    const double alpha = exp(__dsub_rn(m_old, mx));
                    s_alpha[g] = alpha;
                    l = __dadd_rn(__dmul_rn(s_l[g], alpha), l);
                }
                s_l[g] = l;
                s_m[g] = mx;
            }
        }
        if (rows > 0 && !failed && !lb_mbar_wait_bounded(&bars[1], (uint32_t)(chunk & 1))) failed = true;
        __syncthreads();

        // ---- weighted V: warp = position, lane = four dimensions, all heads of the group from one converted row ----
        if (!ONE && chunk > 0) {
#pragma unroll
            for (int g = 0; g < G; ++g)
#pragma unroll
                for (int c = 0; c < 4; ++c) acc[g][c] = __dmul_rn(acc[g][c], s_alpha[g]);
        }
        if (lane_on) {
            for (int j = warp; j < rows; j += kAcWarps) {
                const float4 vv = *reinterpret_cast<const float4*>(vt + (size_t)j * hd + 4 * lane);
                const double v0 = (double)vv.x, v1 = (double)vv.y, v2 = (double)vv.z, v3 = (double)vv.w;
#pragma unroll
                for (int g = 0; g < G; ++g) {
                    const double w = sc[g * cmax + j];
                    acc[g][0] = fma(w, v0, acc[g][0]);
                    acc[g][1] = fma(w, v1, acc[g][1]);
                    acc[g][2] = fma(w, v2, acc[g][2]);
                    acc[g][3] = fma(w, v3, acc[g][3]);
                }
            }
        }
    }
    if (failed && tid == 0) atomicExch(p.status, 1);
    finish_cluster<G, LEAN>(p, acc, red, part, s_m, s_l, s_gw, cnt, n);
}

// Several sequences with rings too long for a slice at once, four query heads per group: first all scores of the slice, then one softmax,
// then the values.  Keys and values go through one ring of four tiles of 64 positions, the first values while the last keys are worked
// on; the warp that is last to be done with a tile asks for the one four on.  No warp waits for another but around the softmax.
// Bound: HBM (20.5 us) and, a warp at a time, the chains of scores and weighted sums.  Eight sequences x eight KV heads in pairs of CTAs at
// context 2048: 41 us (3.3 TB/s); 58 with the chunks above, whose softmax and five barriers a chunk stand between the loads.  (Chunks of
// 160 positions 55, two CTAs an SM with chunks of 64 and 80 56 and 53.)  Where a slice's scores do not fit beside the tiles the chunks stay.
constexpr int kAsRows = 64, kAsTiles = 4;

template <int G>
__global__ void __launch_bounds__(kAcThreads, 1) lb_attention_stream_kernel(const LbAttnParams p) {
    extern __shared__ __align__(128) uint8_t smem_raw[];
    __shared__ __align__(8) uint64_t bars[kAsTiles];
    __shared__ unsigned s_done[kAsTiles];
    __shared__ double s_red[kAcWarps], s_red2[kAcWarps];
    __shared__ double s_m[G], s_l[G];
    __shared__ double s_gw[kAcMaxS * G];
    constexpr int PP = 16 / G;  // positions whose sums a warp reduces together: a tile is one such share per warp
    static_assert(PP * kAcWarps == kAsRows, "a tile of positions");
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int hd = p.hd, half = hd >> 1, kvh = blockIdx.y, ring = kvh >> p.kv_shift, n = blockIdx.z;
    const size_t seq_off = (size_t)n * (size_t)p.seq_stride;
    const uint32_t rank = lb_cluster_rank(), S = cluster_nctarank();
    const int cmax = p.max_chunk;  // positions a slice can have
    float* tiles = reinterpret_cast<float*>(smem_raw);         // [tiles][kAsRows, hd]
    double* red = reinterpret_cast<double*>(smem_raw);         // after the weighted sums: [warps, G, hd] over the tiles
    double* sq = reinterpret_cast<double*>(smem_raw + p.tile); // p.tile = bytes of the tiles / reduction region
    double* sc = sq + G * hd;                                  // [G, cmax] scores, then softmax weights
    double* part = sc + (size_t)G * cmax;                      // [S, G, hd / S + 2] partials received from every slice
    float* newest = reinterpret_cast<float*>(part + (size_t)S * G * (hd / (int)S + 2));  // [hd] the newest key, rotated
    if (tid == 0) {
        for (int i = 0; i < kAsTiles; ++i) {
            lb_mbar_init(&bars[i], 1);
            s_done[i] = 0;
        }
        lb_fence_mbar_init();
    }
    __syncthreads();
    asm volatile("barrier.cluster.arrive.relaxed.aligned;" ::: "memory");  // (waited for before a neighbour's memory is written)
    lb_pdl_launch_dependents();
    lb_pdl_wait();
    lb_trace(p.trace, 2);
    const int last = p.pos_ptr[n], total = last + 1;  // the new token's position; it attends to 0..last
    const int per = (total + (int)S - 1) / (int)S, k0 = (int)rank * per;
    const int cnt = min(per, max(total - k0, 0)), share = (cnt + kAsRows - 1) / kAsRows;  // tiles of keys; as many of values follow
    const float* kbase = p.cache_k + seq_off + ((size_t)ring * p.msl + k0) * hd;
    const float* vbase = p.cache_v + seq_off + ((size_t)ring * p.msl + k0) * hd;
    auto fetch = [&](int item) {  // one thread
        const int c0 = (item < share ? item : item - share) * kAsRows, slot = item % kAsTiles;
        const uint32_t bytes = (uint32_t)min(cnt - c0, kAsRows) * hd * 4;
        lb_mbar_expect_tx(&bars[slot], bytes);
        lb_bulk_g2s_stream(tiles + (size_t)slot * kAsRows * hd, (item < share ? kbase : vbase) + (size_t)c0 * hd, bytes, &bars[slot], lb_policy_evict_first());
    };
    if (tid == 0)
        for (int i = 0; i < kAsTiles && i < 2 * share; ++i) fetch(i);
    // queries of the group and the newest key, rotated: thread idx owns the pair (d, d + hd/2) of head g
    for (int idx = tid; idx < G * half; idx += kAcThreads) {
        const int g = idx / half, d = idx - g * half;
        double sn, c;
        sincos(__ddiv_rn((double)last, p.rope_div[d]), &sn, &c);
        const double* qrow = p.q + (size_t)n * p.heads * hd + (size_t)(kvh * G + g) * hd;
        const double v0 = qrow[d], v1 = qrow[d + half];
        sq[g * hd + d] = __dsub_rn(__dmul_rn(v0, c), __dmul_rn(v1, sn));
        sq[g * hd + d + half] = __dadd_rn(__dmul_rn(v0, sn), __dmul_rn(v1, c));
        if (g == 0 && last >= k0 && last < k0 + cnt) {  // its row of the ring is not written yet
            const float* knew = p.k_new + (size_t)n * p.kv_heads * hd + (size_t)ring * hd;
            const double w0 = (double)knew[d], w1 = (double)knew[d + half];
            const float r0 = (float)__dsub_rn(__dmul_rn(w0, c), __dmul_rn(w1, sn));
            const float r1 = (float)__dadd_rn(__dmul_rn(w0, sn), __dmul_rn(w1, c));
            newest[d] = r0;
            newest[d + half] = r1;
            float* grow = p.cache_k_w + seq_off + ((size_t)ring * p.msl + (size_t)(last % p.msl)) * hd;
            grow[d] = r0;
            grow[d + half] = r1;
        }
    }
    __syncthreads();
    bool failed = false;
    auto wait = [&](int item) {
        if (!failed && !lb_mbar_wait_bounded(&bars[item % kAsTiles], (uint32_t)(item / kAsTiles & 1))) failed = true;
    };
    auto done = [&](int item) {  // this warp has read its share of the tile
        __syncwarp();
        if (lane == 0) {
            __threadfence_block();
            if (atomicAdd(&s_done[item % kAsTiles], 1u) == kAcWarps - 1) {
                s_done[item % kAsTiles] = 0;
                __threadfence_block();
                if (item + kAsTiles < 2 * share && !failed) {
                    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                    fetch(item + kAsTiles);
                }
            }
        }
    };
    const double scale = __ddiv_rn(1.0, sqrt((double)hd));
    const bool lane_on = 4 * lane < hd;
    const int vi = halving_index<16>(lane), vp = vi / G, vg = vi - vp * G;  // this lane finishes the sum of position vp, head vg
    {
        double qv[G][4];
#pragma unroll
        for (int g = 0; g < G; ++g)
#pragma unroll
            for (int c = 0; c < 4; ++c) qv[g][c] = lane_on ? sq[g * hd + 4 * lane + c] : 0.0;
        for (int item = 0; item < share; ++item) {
            wait(item);
            const float* kt = tiles + (size_t)(item % kAsTiles) * kAsRows * hd;
            const int j0 = item * kAsRows + warp * PP;
            if (j0 < cnt) {
                double sums[16];
#pragma unroll
                for (int pp = 0; pp < PP; ++pp) {
                    float4 kv = make_float4(0.f, 0.f, 0.f, 0.f);
                    if (lane_on && j0 + pp < cnt) kv = *reinterpret_cast<const float4*>(k0 + j0 + pp == last ? newest + 4 * lane : kt + (size_t)(warp * PP + pp) * hd + 4 * lane);
                    const double k0d = (double)kv.x, k1d = (double)kv.y, k2d = (double)kv.z, k3d = (double)kv.w;
#pragma unroll
                    for (int g = 0; g < G; ++g) {
                        double a = __dmul_rn(qv[g][0], k0d);
                        a = fma(qv[g][1], k1d, a);
                        a = fma(qv[g][2], k2d, a);
                        a = fma(qv[g][3], k3d, a);
                        sums[pp * G + g] = a;
                    }
                }
                warp_reduce_halving<16>(sums, lane);
                if ((lane & 1) == 0 && j0 + vp < cnt) sc[vg * cmax + j0 + vp] = __dmul_rn(sums[0], scale);
            }
            done(item);
        }
    }
    __syncthreads();
    lb_trace(p.trace, 3);
    {  // softmax of the slice: the warps w with w % G == g share head g
        constexpr int WPG = kAcWarps / G;
        const int g = warp % G, wq = warp / G;
        double mx = -1e300;
        for (int j = wq * 32 + lane; j < cnt; j += WPG * 32) mx = fmax(mx, sc[g * cmax + j]);
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) mx = fmax(mx, __shfl_xor_sync(0xffffffffu, mx, o));
        if (lane == 0) s_red[warp] = mx;
        __syncthreads();
        mx = s_red[g];
#pragma unroll
        for (int w = 1; w < WPG; ++w) mx = fmax(mx, s_red[g + w * G]);
        double sum = 0.0;
#pragma unroll 2
        for (int j = wq * 32 + lane; j < cnt; j += WPG * 32) {
            const double e = exp(__dsub_rn(sc[g * cmax + j], mx));
            sc[g * cmax + j] = e;
            sum = __dadd_rn(sum, e);
        }
        sum = lb_warp_sum(sum);
        if (lane == 0) s_red2[warp] = sum;
        __syncthreads();
        if (wq == 0 && lane == 0) {
            double l = 0.0;
            for (int w = 0; w < WPG; ++w) l += s_red2[g + w * G];
            s_l[g] = l;
            s_m[g] = mx;
        }
    }
    double acc[G][4];
#pragma unroll
    for (int g = 0; g < G; ++g)
#pragma unroll
        for (int c = 0; c < 4; ++c) acc[g][c] = 0.0;
    for (int item = share; item < 2 * share; ++item) {
        wait(item);
        const float* vt = tiles + (size_t)(item % kAsTiles) * kAsRows * hd;
        const int c0 = (item - share) * kAsRows;
        if (lane_on) {
#pragma unroll
            for (int r = 0; r < kAsRows / kAcWarps; ++r) {
                const int j = warp + kAcWarps * r;
                if (c0 + j >= cnt) break;
                const float4 vv = *reinterpret_cast<const float4*>(vt + (size_t)j * hd + 4 * lane);
                const double v0 = (double)vv.x, v1 = (double)vv.y, v2 = (double)vv.z, v3 = (double)vv.w;
#pragma unroll
                for (int g = 0; g < G; ++g) {
                    const double w = sc[g * cmax + c0 + j];
                    acc[g][0] = fma(w, v0, acc[g][0]);
                    acc[g][1] = fma(w, v1, acc[g][1]);
                    acc[g][2] = fma(w, v2, acc[g][2]);
                    acc[g][3] = fma(w, v3, acc[g][3]);
                }
            }
        }
        done(item);
    }
    if (failed && lane == 0) atomicExch(p.status, 1);
    finish_cluster<G, false>(p, acc, red, part, s_m, s_l, s_gw, cnt, n);
}

constexpr size_t kAcSmem = 200 * 1024, kAsSmem = 220 * 1024;
// Bytes of the next block's rings that are asked into L2, over all clusters: what arrives before that block's projections do.  Asking
// for whole rings costs more the longer they are (us a block, 8 KV heads, none / 4 MB / 32 MB / all: context 4000 73.2, 72.9, 74.6, 74.7;
// 8000 95.9, 95.8, 97.5, 97.3; 32000 232.5, 232.7, 233.6, 233.4; five KV heads, context 8000: 59.6, 59.3, 60.5, 60.7).
constexpr size_t kAcAhead = 4 << 20;
constexpr int kAcChunk = 128;  // positions of a chunk when a slice does not fit at once

template <int G>
size_t cluster_smem(const LbAttnParams& p, int S, int rows, int* tile_bytes) {
    size_t tiles = (size_t)2 * rows * p.hd * sizeof(float);
    const size_t red = (size_t)kAcWarps * G * p.hd * sizeof(double);
    if (red > tiles) tiles = red;
    tiles = (tiles + 127) & ~(size_t)127;
    *tile_bytes = (int)tiles;
    const int dps = p.hd / S;
    return tiles + (size_t)G * p.hd * 8 + (size_t)G * rows * 8 + (size_t)S * G * (dps + 2) * 8;
}

template <int G>
int launch_cluster(loom_b200_ctx* ctx, LbAttnParams p, int S, bool probe_only, int* active_clusters) {
    int tile_bytes = 0;
    p.max_chunk = (p.msl + S - 1) / S;
    size_t smem = cluster_smem<G>(p, S, p.max_chunk, &tile_bytes);
    const bool one = smem <= kAcSmem;
    if (!one) {
        p.max_chunk = kAcChunk;
        smem = cluster_smem<G>(p, S, kAcChunk, &tile_bytes);
    }
    bool streams = false;
    if constexpr (G == 4)
        if (!one && p.seq_stride > 0 && (size_t)S * p.msl > 0) {
            // (in front of a slice's scores, which lie in shared memory whole)
            const int rows = (p.msl + S - 1) / S;
            int t = 0;
            const size_t need = cluster_smem<G>(p, S, kAsRows * kAsTiles / 2, &t) + (size_t)G * (rows - kAsRows * kAsTiles / 2) * 8 + (size_t)p.hd * 4;
            if (need <= kAsSmem) {
                streams = true;
                p.max_chunk = rows;
                tile_bytes = t;
                smem = need;
            }
        }
    p.tile = tile_bytes;
    p.next_rows = (int)(kAcAhead / ((size_t)p.kv_heads * S * p.hd * 2 * sizeof(float)));
    if (p.next_rows == 0) p.next_k = nullptr;
    const bool lean = !probe_only && !p.trace && p.M == 1 && p.seq_stride <= 0;
    void (*kern)(LbAttnParams) = lean ? lb_attention_cluster_kernel<G, true, true> : lb_attention_cluster_kernel<G, false, true>;
    if constexpr (G < 8)
        if (!one && !streams) kern = lean ? lb_attention_cluster_kernel<G, true, false> : lb_attention_cluster_kernel<G, false, false>;
    if constexpr (G == 4)
        if (streams) kern = lb_attention_stream_kernel<G>;
    // one bit per instantiation, per context (= per device)
    const unsigned bit = 1u << ((G == 1 ? 0 : G == 2 ? 1 : G == 4 ? 2 : 3) + (streams ? 24 : (lean ? 4 : 0) + (one ? 0 : 16)));
    if (!(ctx->func_attr_mask3 & bit)) {
        LB_CUDA(ctx, cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)(streams ? kAsSmem : kAcSmem)));
        LB_CUDA(ctx, cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
        ctx->func_attr_mask3 |= bit;
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(S, p.kv_heads << p.kv_shift, p.M);
    cfg.blockDim = dim3(kAcThreads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = ctx->stream;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = S;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = ctx->opt_pdl ? 2 : 1;
    if (probe_only) {
        cfg.numAttrs = 1;
        int n = 0;
        cudaError_t e = cudaOccupancyMaxActiveClusters(&n, kern, &cfg);
        if (e != cudaSuccess) {
            cudaGetLastError();
            n = 0;
        }
        *active_clusters = n;
        return 0;
    }
    LB_CUDA(ctx, cudaLaunchKernelEx(&cfg, kern, p));
    ctx->launches++;
    return 0;
}

// `active`: how many KV heads' clusters the device holds at once
int dispatch_cluster(loom_b200_ctx* ctx, LbAttnParams p, int S, bool probe_only, int* active) {
    switch (p.heads / p.kv_heads) {
        case 1: return launch_cluster<1>(ctx, p, S, probe_only, active);
        case 2: return launch_cluster<2>(ctx, p, S, probe_only, active);
        case 4: return launch_cluster<4>(ctx, p, S, probe_only, active);
        case 8: {
            int tile_bytes = 0;
            if (cluster_smem<8>(p, S, (p.msl + S - 1) / S, &tile_bytes) <= kAcSmem) return launch_cluster<8>(ctx, p, S, probe_only, active);
            // Eight heads' sums over several chunks do not fit the registers (404 bytes of spills): two clusters of four heads each
            // over the same KV head instead, which also fill more SMs.  Steps of one sequence, us a block with a ring of 4096, split
            // kernel / eight heads with spills / two times four: two KV heads 36.5, 41.0, 36.4 at context 300, 50.5, 64.2, 44.1 at 3500;
            // eight KV heads 61.7, 62.1, 57.0 and 125.7, 118.0, 92.4.
            p.kv_shift = 1;
            const int rc = launch_cluster<4>(ctx, p, S, probe_only, active);
            if (probe_only) *active /= 2;
            return rc;
        }
        default: return LOOM_B200_ERR_UNSUPPORTED;
    }
}

}  // namespace

int lb_attention_cluster_size(loom_b200_ctx* ctx, const LbAttnParams& p, int sequences) {
    if ((p.M != 1 && p.seq_stride <= 0) || !p.rope_div || !p.k_new || !p.cache_k_w) return 0;
    if (p.kv_heads <= 0 || p.heads % p.kv_heads != 0) return 0;
    const int G = p.heads / p.kv_heads;
    if (G != 1 && G != 2 && G != 4 && G != 8) return 0;
    if (p.hd % 16 != 0 || p.hd > 128 || p.hd < 16) return 0;
    // the largest cluster size of which the device holds one per KV head and sequence at once
    const int smax = ctx->opt_attn_cluster >= 2 && ctx->opt_attn_cluster < kAcMaxS ? ctx->opt_attn_cluster : kAcMaxS;  // option: 1 = the largest that fits, 2..16 = at most that
    const int clusters = p.kv_heads * (sequences > 0 ? sequences : 1);
    for (int S = kAcMaxS; S >= 2; S >>= 1) {
        if (S > smax) continue;
        if (p.hd % S != 0) continue;
        int active = 0;
        if (dispatch_cluster(ctx, p, S, true, &active) != 0) continue;
        if (active >= clusters || (sequences == 0 && S == 2 && active >= 1)) return S;
    }
    return sequences > 0 ? 1 : 0;  // more (sequence, KV head) pairs than pairs of SMs: single CTAs, in waves
}

int lb_launch_attention_cluster(loom_b200_ctx* ctx, const LbAttnParams& pin, int S) {
    LbAttnParams p = pin;
    p.trace = lb_trace_row(ctx, "attention");
    p.status = ctx->status_dev;
    int rc = dispatch_cluster(ctx, p, S, false, nullptr);
    if (rc == LOOM_B200_ERR_UNSUPPORTED) return lb_fail(ctx, rc, "attention (cluster): shape not supported");
    return rc;
}

// kernel_harness.cu -- C entries for tests of parts that no public call reaches one by one: the bf16 token-block product alone, the float64
// attention of a prompt block alone, and the second rank of a tensor-parallel pair whose messages lie in the mailbox before the first rank asks for them (so nothing waits).
//
//   nvcc -gencode arch=compute_100a,code=sm_100a -std=c++17 -shared -Xcompiler -fPIC -Iinclude -Iloom_b200/csrc tests/kernel_harness.cu
//        loom_b200/lib/libloom_b200.so -o kernel_harness.so
#include "dense.cuh"
#include "glue.cuh"
#include "tp_xchg.cuh"

#include <cstring>
#include <vector>

extern "C" {

int t_gemm_bf16(loom_b200_ctx* ctx, int epi, const loom_b200_matrix* x, const loom_b200_matrix* w, const loom_b200_matrix* w2, int tokens, float* out, int ldo,
                void* img, int img_slices, int heads, int head_dim, float mult, float res_mult, float limit) {
    LbDenseGemm p;
    p.x = x->data;
    p.w = w->data;
    p.w2 = w2 ? w2->data : nullptr;
    p.tokens = tokens;
    p.rows = w->rows;
    p.slices = w->slices;
    p.out = out;
    p.ldo = ldo;
    p.img = static_cast<uint8_t*>(img);
    p.img_slices = img_slices;
    p.heads = heads;
    p.head_dim = head_dim;
    p.head_chunks = heads ? lb_ceil_div(head_dim, 8) : 0;
    p.mult = mult;
    p.res_mult = res_mult;
    p.limit = limit;
    if (int rc = lb_dense_gemm(ctx, LOOM_B200_DTYPE_BF16, epi, p)) return rc;
    return lb_sync_checked(ctx);
}

// everything on the device; keys and values [kv_heads, msl, hd], pos: the first token's position
int t_attention_prompt(loom_b200_ctx* ctx, const double* q, const float* k, const float* v, const int* pos, double* out, int tokens, int heads, int kv_heads, int hd, int msl) {
    LbAttnParams p = {};
    p.q = q;
    p.cache_k = k;
    p.cache_v = v;
    p.pos_ptr = pos;
    p.out = out;
    p.M = tokens;
    p.heads = heads;
    p.kv_heads = kv_heads;
    p.hd = hd;
    p.msl = msl;
    p.splits = 1;
    p.max_chunk = msl;
    if (int rc = lb_launch_attention_prefill(ctx, p)) return rc;
    return lb_sync_checked(ctx);
}

// rank 0 of two: a mailbox of its own and, for what it sends, another one on the same device
int t_pair_begin(loom_b200_ctx* ctx, void** other) {
    LB_CUDA(ctx, cudaMalloc(&ctx->xbuf, kXBytes));
    LB_CUDA(ctx, cudaMalloc(other, kXBytes));
    LB_CUDA(ctx, cudaMemset(ctx->xbuf, 0, kXBytes));
    LB_CUDA(ctx, cudaMemset(*other, 0, kXBytes));
    const unsigned int init[8] = {1u, 0u, 1u, 0u, 0u, 1u, 0u, 0u};
    LB_CUDA(ctx, cudaMalloc(&ctx->x_ctr, sizeof(init)));
    LB_CUDA(ctx, cudaMemcpy(ctx->x_ctr, init, sizeof(init), cudaMemcpyHostToDevice));
    void* both[kXMaxRanks] = {ctx->xbuf, *other};
    LB_CUDA(ctx, cudaMalloc(&ctx->peer_xbuf_dev, sizeof(both)));
    LB_CUDA(ctx, cudaMemcpy(ctx->peer_xbuf_dev, both, sizeof(both), cudaMemcpyHostToDevice));
    ctx->tp_rank = 0;
    ctx->tp_world = 2;
    ctx->tp_peer = true;
    return 0;
}
// rank 1's part of exchange number seq: sums of squares and largest values of the tokens, and the partial sums [n]
int t_pair_message(loom_b200_ctx* ctx, unsigned int seq, int tokens, const double* ss, const float* amax, const int32_t* acc, int n) {
    struct Word {
        uint32_t data, seq;
    };
    const size_t half = seq & 1, from = half * kXMaxRanks + 1;
    char* box = static_cast<char*>(ctx->xbuf);
    for (int t = 0; t < tokens; ++t) {
        unsigned long long bits;
        memcpy(&bits, ss + t, 8);
        const Word s[2] = {{(uint32_t)bits, seq}, {(uint32_t)(bits >> 32), seq}};
        Word m = {0, seq};
        memcpy(&m.data, amax + t, 4);
        LB_CUDA(ctx, cudaMemcpy(box + kXRegionA + (from * 8 + t) * 2 * 8, s, sizeof(s), cudaMemcpyHostToDevice));
        LB_CUDA(ctx, cudaMemcpy(box + kXRegionB + (from * 8 + t) * 8, &m, sizeof(m), cudaMemcpyHostToDevice));
    }
    std::vector<Word> a(n);
    for (int i = 0; i < n; ++i) a[i] = {(uint32_t)acc[i], seq};
    LB_CUDA(ctx, cudaMemcpy(box + kXRegionC + from * kXMaxAcc * 8, a.data(), n * sizeof(Word), cudaMemcpyHostToDevice));
    return 0;
}
void t_pair_end(loom_b200_ctx* ctx, void* other) {
    cudaStreamSynchronize(ctx->stream);
    ctx->tp_peer = false;  // (the other mailbox is no mapped one)
    loom_b200_tp_finalize(ctx);
    cudaFree(other);
}

}  // extern "C"

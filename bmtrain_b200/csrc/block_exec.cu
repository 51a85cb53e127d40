// Native executors for whole transformer blocks: pre-LN GPT and, below, the Llama-shaped one.  GPT: the whole forward or backward of a
// transformer layer is issued from C++ by a single call, so the host cost per layer is a few microseconds instead
// of one Python/autograd round trip per operator.  Launches with the fused attention: 7 forward, one more with a mask and one more with GELU; 14
// backward, 18 for more than 2048 tokens, whose bias gradients take a kernel each.  Two more either way with
// scores in memory.  Every contraction goes to the tcgen05 GEMM (gemm_sm100.cu) with
// fused epilogues: bias, ReLU, residual add, ReLU-mask / GELU-derivative on the dgrad path.
// (The reference runs a block as ~40 separate PyTorch ops: example/layers/transformer.py:19-33.)
#include <math.h>
#include <string.h>

#include "api.h"
#include "common.cuh"

namespace {

#define RUN(expr)                 \
    do {                          \
        int _rc = (expr);         \
        if (_rc != 0) return _rc; \
    } while (0)

BmtGemmDesc plain(int64_t m, int64_t n, int64_t k, const void* a, int64_t lda, int a_major, const void* b, int64_t ldb, int b_major,
                  void* c, int64_t ldc, int dtype) {
    BmtGemmDesc g;
    memset(&g, 0, sizeof(g));
    g.m = m; g.n = n; g.k = k; g.a = a; g.lda = lda; g.a_major = a_major; g.b = b; g.ldb = ldb; g.b_major = b_major;
    g.c = c; g.ldc = ldc; g.c_dtype = dtype; g.ab_dtype = dtype; g.alpha = 1.f;
    g.batch_inner = g.batch_outer = g.b_inner_div = 1;
    return g;
}

int gemm(const BmtGptBlock& k, BmtGemmDesc& g, void* stream) {
    g.scratch = k.gemm_scratch; g.scratch_bytes = k.gemm_scratch_bytes;
    return bmt_gemm_ex(&g, stream);
}

struct Dims {
    int64_t T, d, h, dh, hd, dff, s, b, es;  // es = element size
};

Dims dims_of(const BmtGptBlock& k) {
    Dims q;
    q.b = k.batch; q.s = k.seq; q.T = k.batch * k.seq; q.d = k.d_model; q.h = k.n_heads; q.dh = k.d_head; q.hd = q.h * q.dh;
    q.dff = k.d_ff; q.es = 2;
    return q;
}

const char* off(const void* p, int64_t elems) { return (const char*)p + elems * 2; }
char* off(void* p, int64_t elems) { return (char*)p + elems * 2; }

// The fused attention takes a dense mask in its packed form: one without room for the other would attend everywhere.
bool mask_complete(const BmtGptBlock& k) { return !k.lse || (k.mask != nullptr) == (k.mask_packed != nullptr); }

// Part 0 (by query), 1 (by key) or 2 (tile classes) of the packed mask of the fused attention, or null.
const void* mask_part(const BmtGptBlock& k, const Dims& q, int part) {
    if (!k.mask_packed) return nullptr;
    int64_t at[3] = {0, 0, 0};
    bmt_attn_mask_layout(q.b, q.s, q.s, &at[1], &at[2]);
    return (const char*)k.mask_packed + at[part];
}

}  // namespace

// Steps [first_step, last_step] of the forward (1 = LN1, 2 = QKV projection, 3..5 attention core, 6 = output
// projection + residual, 7 = LN2, 8 = first FFN GEMM, 9 = second FFN GEMM + residual).  Running a sub-range lets the
// caller put its own QKV GEMM (fused with the parameter gather) or a stream wait between the steps.
extern "C" int bmt_gpt_block_forward_steps(const BmtGptBlock* blk, int first_step, int last_step, void* stream) {
    const BmtGptBlock& k = *blk;
    if (!mask_complete(k)) return -40;
    const Dims q = dims_of(k);
    const int dt = k.dtype;
    // Below a ReLU no product is divided along its reduction: the sum's last bit moves roundings of the 16-bit results, ReLU inputs near zero
    // change sides, and gradients of a bf16 model of three blocks move by 5 % (they are 6 % from the exact ones either way).  That keeps the bits
    // that this executor gave before tiles were divided; a block that runs operator by operator (no biases, tensor parallelism, fused blocks
    // switched off) has its products divided like any others, so it is as far from the exact result but not equal to the last bit.
    const auto product = [&](BmtGemmDesc& g) { return k.act == 1 ? bmt_gemm_ex(&g, stream) : gemm(k, g, stream); };
#define STEP(n) if (first_step <= (n) && (n) <= last_step)
    // 1. LN1
    STEP(1) RUN(bmt_norm_fwd(q.T, q.d, k.x, k.ln1_w, k.ln1_b, k.eps, 0, dt, k.ln1, k.stats1, stream));
    // 2. fused QKV projection (+ bias): qkv laid out (token, head, {q,k,v}, d_head)
    STEP(2) {
        BmtGemmDesc g = plain(q.T, 3 * q.hd, q.d, k.ln1, q.d, 0, k.qkv_w, q.d, 0, k.qkv, 3 * q.hd, dt);
        g.bias = k.qkv_b;
        RUN(product(g));
    }
    const int64_t tok = 3 * q.hd, head = 3 * q.dh;
    // 3-5 as one fused attention kernel: q, k, v are strided views of the packed projection, nothing of size s x s is stored
    if (k.lse) {
        STEP(3) {
            if (k.mask_packed) RUN(bmt_attn_mask_pack(q.b, q.s, q.s, k.mask, k.mask_packed, stream));
            const int64_t in_str[3] = {tok, head, q.s * tok}, out_str[3] = {q.hd, q.dh, q.s * q.hd};
            RUN(bmt_flash_attn_fwd(q.b, q.s, q.s, (int)q.h, (int)q.h, (int)q.dh, k.qkv, in_str, off(k.qkv, q.dh), in_str,
                                   off(k.qkv, 2 * q.dh), in_str, k.ctx, out_str, k.lse, 1.f / sqrtf((float)q.dh), k.causal,
                                   mask_part(k, q, 0), mask_part(k, q, 2), nullptr, dt, stream));
        }
    } else {
    // 3. scores = q k^T / sqrt(d_head)   -> probs (b, h, s, ld)
    STEP(3) {
        BmtGemmDesc g = plain(q.s, q.s, q.dh, k.qkv, tok, 0, off(k.qkv, q.dh), tok, 0, k.probs, k.probs_ld, dt);
        g.a_bs0 = head; g.a_bs1 = q.s * tok; g.b_bs0 = head; g.b_bs1 = q.s * tok;
        g.c_bs0 = q.s * k.probs_ld; g.c_bs1 = q.h * q.s * k.probs_ld;
        g.batch_inner = q.h; g.batch_outer = q.b; g.alpha = 1.f / sqrtf((float)q.dh);
        RUN(product(g));
    }
    // 4. masked softmax in place
    STEP(4) RUN(bmt_masked_softmax(q.b, q.h, q.s, q.s, k.probs_ld, k.probs, dt, k.causal, k.mask, nullptr, stream));
    // 5. ctx = probs v  -> (token, head, d_head)
    STEP(5) {
        BmtGemmDesc g = plain(q.s, q.dh, q.s, k.probs, k.probs_ld, 0, off(k.qkv, 2 * q.dh), tok, 1, k.ctx, q.hd, dt);
        g.a_bs0 = q.s * k.probs_ld; g.a_bs1 = q.h * q.s * k.probs_ld; g.b_bs0 = head; g.b_bs1 = q.s * tok;
        g.c_bs0 = q.dh; g.c_bs1 = q.s * q.hd;
        g.batch_inner = q.h; g.batch_outer = q.b;
        RUN(product(g));
    }
    }
    // 6. h1 = ctx W_o^T + b_o + x
    STEP(6) {
        BmtGemmDesc g = plain(q.T, q.d, q.hd, k.ctx, q.hd, 0, k.out_w, q.hd, 0, k.h1, q.d, dt);
        g.bias = k.out_b; g.residual = k.x; g.ldr = q.d;
        RUN(product(g));
    }
    // 7. LN2
    STEP(7) RUN(bmt_norm_fwd(q.T, q.d, k.h1, k.ln2_w, k.ln2_b, k.eps, 0, dt, k.ln2, k.stats2, stream));
    // 8. ff = act(ln2 W_1^T + b_1)
    STEP(8) {
        BmtGemmDesc g = plain(q.T, q.dff, q.d, k.ln2, q.d, 0, k.fc1_w, q.d, 0, k.act == 2 ? k.pre : k.ff, q.dff, dt);
        g.bias = k.fc1_b; g.act = k.act == 1 ? 1 : 0;
        RUN(product(g));
        if (k.act == 2) RUN(bmt_gelu_fwd(q.T * q.dff, k.pre, dt, k.ff, stream));
    }
    // 9. y = ff W_2^T + b_2 + h1
    STEP(9) {
        BmtGemmDesc g = plain(q.T, q.d, q.dff, k.ff, q.dff, 0, k.fc2_w, q.dff, 0, k.y, q.d, dt);
        g.bias = k.fc2_b; g.residual = k.h1; g.ldr = q.d;
        RUN(product(g));
    }
#undef STEP
    return 0;
}

extern "C" int bmt_gpt_block_backward(const BmtGptBlock* blk, const BmtGptBlockGrad* grad, void* stream) {
    const BmtGptBlock& k = *blk;
    const BmtGptBlockGrad& w = *grad;
    if (!mask_complete(k)) return -40;
    const Dims q = dims_of(k);
    const int dt = k.dtype;
    const int64_t tok = 3 * q.hd, head = 3 * q.dh;
    // ---- FFN
    {   // d_ff = (dy W_2) * act'(.)
        BmtGemmDesc g = plain(q.T, q.dff, q.d, w.dy, q.d, 0, k.fc2_w, q.dff, 1, w.d_ff, q.dff, dt);
        g.aux = k.act == 2 ? k.pre : k.ff; g.ld_aux = q.dff; g.aux_mode = k.act == 2 ? 2 : 1;
        RUN(gemm(k, g, stream));
    }
    {   // dW_2 = dy^T ff
        BmtGemmDesc g = plain(q.d, q.dff, q.T, w.dy, q.d, 1, k.ff, q.dff, 1, w.d_fc2_w, q.dff, dt);
        g.accumulate = w.acc_w;
        RUN(gemm(k, g, stream));
    }
    {   // d_ln2 = d_ff W_1
        BmtGemmDesc g = plain(q.T, q.d, q.dff, w.d_ff, q.dff, 0, k.fc1_w, q.d, 1, w.d_ln2, q.d, dt);
        RUN(gemm(k, g, stream));
    }
    {   // dW_1 = d_ff^T ln2
        BmtGemmDesc g = plain(q.dff, q.d, q.T, w.d_ff, q.dff, 1, k.ln2, q.d, 1, w.d_fc1_w, q.d, dt);
        g.accumulate = w.acc_w;
        RUN(gemm(k, g, stream));
    }
    // d_h1 = dy + LN2'(d_ln2)
    int rows2 = 0, rows1 = 0;
    RUN(bmt_norm_bwd_partial(q.T, q.d, k.h1, w.d_ln2, k.ln2_w, k.stats2, 0, dt, w.nblk, w.d_h1, w.norm_partial, w.dy, &rows2, stream));
    // ---- attention output projection
    {   // d_ctx = d_h1 W_o
        BmtGemmDesc g = plain(q.T, q.hd, q.d, w.d_h1, q.d, 0, k.out_w, q.hd, 1, w.d_ctx, q.hd, dt);
        RUN(gemm(k, g, stream));
    }
    {   // dW_o = d_h1^T ctx
        BmtGemmDesc g = plain(q.d, q.hd, q.T, w.d_h1, q.d, 1, k.ctx, q.hd, 1, w.d_out_w, q.hd, dt);
        g.accumulate = w.acc_w;
        RUN(gemm(k, g, stream));
    }
    // ---- attention core
    const int64_t pl = k.probs_ld;
    if (k.lse) {
        // fused backward: dq, dk, dv go straight into the packed d_qkv buffer
        const int64_t in_str[3] = {tok, head, q.s * tok}, out_str[3] = {q.hd, q.dh, q.s * q.hd};
        RUN(bmt_flash_attn_bwd(q.b, q.s, q.s, (int)q.h, (int)q.h, (int)q.dh, k.qkv, in_str, off(k.qkv, q.dh), in_str,
                               off(k.qkv, 2 * q.dh), in_str, k.ctx, out_str, w.d_ctx, out_str, k.lse, w.d_qkv, in_str,
                               off(w.d_qkv, q.dh), in_str, off(w.d_qkv, 2 * q.dh), in_str, w.dq_acc, w.delta,
                               1.f / sqrtf((float)q.dh), k.causal, mask_part(k, q, 1), mask_part(k, q, 2), nullptr, nullptr, dt, stream));
    } else {
    {   // dP = d_ctx v^T
        BmtGemmDesc g = plain(q.s, q.s, q.dh, w.d_ctx, q.hd, 0, off(k.qkv, 2 * q.dh), tok, 0, w.d_probs, pl, dt);
        g.a_bs0 = q.dh; g.a_bs1 = q.s * q.hd; g.b_bs0 = head; g.b_bs1 = q.s * tok;
        g.c_bs0 = q.s * pl; g.c_bs1 = q.h * q.s * pl; g.batch_inner = q.h; g.batch_outer = q.b;
        RUN(gemm(k, g, stream));
    }
    RUN(bmt_softmax_bwd(q.b * q.h * q.s, q.s, pl, k.probs, w.d_probs, 1.f / sqrtf((float)q.dh), dt, stream));
    {   // dq = dS k
        BmtGemmDesc g = plain(q.s, q.dh, q.s, w.d_probs, pl, 0, off(k.qkv, q.dh), tok, 1, w.d_qkv, tok, dt);
        g.a_bs0 = q.s * pl; g.a_bs1 = q.h * q.s * pl; g.b_bs0 = head; g.b_bs1 = q.s * tok;
        g.c_bs0 = head; g.c_bs1 = q.s * tok; g.batch_inner = q.h; g.batch_outer = q.b;
        RUN(gemm(k, g, stream));
    }
    {   // dk = dS^T q
        BmtGemmDesc g = plain(q.s, q.dh, q.s, w.d_probs, pl, 1, k.qkv, tok, 1, off(w.d_qkv, q.dh), tok, dt);
        g.a_bs0 = q.s * pl; g.a_bs1 = q.h * q.s * pl; g.b_bs0 = head; g.b_bs1 = q.s * tok;
        g.c_bs0 = head; g.c_bs1 = q.s * tok; g.batch_inner = q.h; g.batch_outer = q.b;
        RUN(gemm(k, g, stream));
    }
    {   // dv = P^T d_ctx
        BmtGemmDesc g = plain(q.s, q.dh, q.s, k.probs, pl, 1, w.d_ctx, q.hd, 1, off(w.d_qkv, 2 * q.dh), tok, dt);
        g.a_bs0 = q.s * pl; g.a_bs1 = q.h * q.s * pl; g.b_bs0 = q.dh; g.b_bs1 = q.s * q.hd;
        g.c_bs0 = head; g.c_bs1 = q.s * tok; g.batch_inner = q.h; g.batch_outer = q.b;
        RUN(gemm(k, g, stream));
    }
    }
    // ---- QKV projection
    {   // d_ln1 = d_qkv W_qkv   (reuses the d_ln2 buffer)
        BmtGemmDesc g = plain(q.T, q.d, 3 * q.hd, w.d_qkv, tok, 0, k.qkv_w, q.d, 1, w.d_ln2, q.d, dt);
        RUN(gemm(k, g, stream));
    }
    {   // dW_qkv = d_qkv^T ln1
        BmtGemmDesc g = plain(3 * q.hd, q.d, q.T, w.d_qkv, tok, 1, k.ln1, q.d, 1, w.d_qkv_w, q.d, dt);
        g.accumulate = w.acc_w;
        RUN(gemm(k, g, stream));
    }
    // dx = d_h1 + LN1'(d_ln1)
    RUN(bmt_norm_bwd_partial(q.T, q.d, k.x, w.d_ln2, k.ln1_w, k.stats1, 0, dt, w.nblk, w.dx, w.norm_partial2, w.d_h1, &rows1, stream));
    // everything that is a column sum, in one launch
    const float *p2 = (const float*)w.norm_partial, *p1 = (const float*)w.norm_partial2;
    const BmtColsum sums[8] = {{w.dy, q.T, q.d, w.d_fc2_b, 0, 0}, {w.d_ff, q.T, q.dff, w.d_fc1_b, 0, 0},
                               {w.d_h1, q.T, q.d, w.d_out_b, 0, 0}, {w.d_qkv, q.T, 3 * q.hd, w.d_qkv_b, 0, 0},
                               {p2, rows2, q.d, w.d_ln2_w, 1, 0}, {p2 + rows2 * q.d, rows2, q.d, w.d_ln2_b, 1, 0},
                               {p1, rows1, q.d, w.d_ln1_w, 1, 0}, {p1 + rows1 * q.d, rows1, q.d, w.d_ln1_b, 1, 0}};
    RUN(bmt_colsum_multi(sums, 8, dt, w.acc_small, k.colsum_scratch, k.colsum_scratch_bytes, stream));
    return 0;
}

// ------------------------------------------------------------------------------------------------- Llama-shaped block
// 9 launches forward, 16 backward, one more where query heads share a key head and the kernel divides them.  The residual additions happen in the epilogues of the projections and in the norms'
// backward (as operators of their own: six passes over (T, d) per block and step, 4 % of a block at 2048 x 8192).
namespace {

struct LlamaDims { int64_t T, d, h, hk, dh, hd, kd, qkv, dff; };
LlamaDims dims_of(const BmtLlamaBlock& k) {
    LlamaDims q;
    q.T = k.batch * k.seq; q.d = k.d_model; q.h = k.n_heads; q.hk = k.n_kv; q.dh = k.d_head; q.hd = q.h * q.dh; q.kd = q.hk * q.dh;
    q.qkv = q.hd + 2 * q.kd; q.dff = k.d_ff;
    return q;
}

}  // namespace

extern "C" int bmt_llama_block_forward(const BmtLlamaBlock* blk, int last_step, void* stream) {
    const BmtLlamaBlock& k = *blk;
    const LlamaDims q = dims_of(k);
    const int dt = k.dtype;
    auto gemm = [&](BmtGemmDesc g) {
        g.scratch = k.gemm_scratch; g.scratch_bytes = k.gemm_scratch_bytes;
        return bmt_gemm_ex(&g, stream);
    };
    RUN(bmt_norm_fwd(q.T, q.d, k.x, k.ln1_w, nullptr, k.eps1, 1, dt, k.ln1, k.stats1, stream));
    RUN(gemm(plain(q.T, q.qkv, q.d, k.ln1, q.d, 0, k.qkv_w, q.d, 0, k.packed, q.qkv, dt)));
    RUN(bmt_rope_qkv(k.batch, k.seq, (int)q.hk, (int)(q.h / q.hk), (int)q.dh, k.packed, q.qkv, k.seq * q.qkv, k.q, k.k, k.v, k.rope, 0, 1, dt,
                     stream));
    const int64_t qs[3] = {q.hd, q.dh, k.seq * q.hd}, ks[3] = {q.kd, q.dh, k.seq * q.kd};
    RUN(bmt_flash_attn_fwd(k.batch, k.seq, k.seq, (int)q.h, (int)q.hk, (int)q.dh, k.q, qs, k.k, ks, k.v, ks, k.ctx, qs, k.lse,
                           1.f / sqrtf((float)q.dh), 1, nullptr, nullptr, nullptr, dt, stream));
    {
        BmtGemmDesc g = plain(q.T, q.d, q.hd, k.ctx, q.hd, 0, k.out_w, q.hd, 0, k.h1, q.d, dt);
        g.residual = k.x; g.ldr = q.d; g.round_first = 1;      // the modules round the projection, and so does this
        RUN(gemm(g));
    }
    RUN(bmt_norm_fwd(q.T, q.d, k.h1, k.ln2_w, nullptr, k.eps2, 1, dt, k.ln2, k.stats2, stream));
    RUN(gemm(plain(q.T, 2 * q.dff, q.d, k.ln2, q.d, 0, k.gate_up_w, q.d, 0, k.gate_up, 2 * q.dff, dt)));
    RUN(bmt_swiglu_fwd(q.T, q.dff, k.gate_up, dt, k.ff, stream));
    if (last_step >= 9) {
        BmtGemmDesc g = plain(q.T, q.d, q.dff, k.ff, q.dff, 0, k.w_out, q.dff, 0, k.y, q.d, dt);
        g.residual = k.h1; g.ldr = q.d; g.round_first = 1;
        RUN(gemm(g));
    }
    return 0;
}

extern "C" int bmt_llama_block_backward(const BmtLlamaBlock* blk, const BmtLlamaBlockGrad* grad, void* stream) {
    const BmtLlamaBlock& k = *blk;
    const BmtLlamaBlockGrad& w = *grad;
    const LlamaDims q = dims_of(k);
    const int dt = k.dtype;
    auto gemm = [&](BmtGemmDesc g) {
        g.scratch = k.gemm_scratch; g.scratch_bytes = k.gemm_scratch_bytes;
        return bmt_gemm_ex(&g, stream);
    };
    // (T, n) gradient times an (n, m) weight; transposed (T, n) gradient times the (T, m) input of the layer
    auto dgrad = [&](const void* dy, int64_t n, const void* weight, int64_t m, void* dx) {
        return gemm(plain(q.T, m, n, dy, n, 0, weight, m, 1, dx, m, dt));
    };
    auto wgrad = [&](const void* dy, int64_t n, const void* x, int64_t m, void* dw) {
        return gemm(plain(n, m, q.T, dy, n, 1, x, m, 1, dw, m, dt));
    };
    RUN(dgrad(w.dy, q.d, k.w_out, q.dff, w.d_ff));
    RUN(wgrad(w.dy, q.d, k.ff, q.dff, w.d_w_out));
    RUN(bmt_swiglu_bwd(q.T, q.dff, k.gate_up, w.d_ff, dt, w.d_gate_up, stream));
    RUN(dgrad(w.d_gate_up, 2 * q.dff, k.gate_up_w, q.d, w.d_ln));
    RUN(wgrad(w.d_gate_up, 2 * q.dff, k.ln2, q.d, w.d_gate_up_w));
    int rows2 = 0, rows1 = 0;
    float *p2 = (float*)w.norm_partial, *p1 = p2 + 2 * w.nblk * q.d;
    RUN(bmt_norm_bwd_partial(q.T, q.d, k.h1, w.d_ln, k.ln2_w, k.stats2, 1, dt, (int)w.nblk, w.d_h1, p2, w.dy, &rows2, stream));
    RUN(dgrad(w.d_h1, q.d, k.out_w, q.hd, w.d_ctx));
    RUN(wgrad(w.d_h1, q.d, k.ctx, q.hd, w.d_out_w));
    const int64_t qs[3] = {q.hd, q.dh, k.seq * q.hd}, ks[3] = {q.kd, q.dh, k.seq * q.kd};
    RUN(bmt_flash_attn_bwd(k.batch, k.seq, k.seq, (int)q.h, (int)q.hk, (int)q.dh, k.q, qs, k.k, ks, k.v, ks, k.ctx, qs, w.d_ctx, qs, k.lse, w.dq,
                           qs, w.dk, ks, w.dv, ks, w.dq_acc, w.delta, 1.f / sqrtf((float)q.dh), 1, nullptr, nullptr, nullptr, w.dkv_part, dt,
                           stream));
    RUN(bmt_rope_qkv(k.batch, k.seq, (int)q.hk, (int)(q.h / q.hk), (int)q.dh, w.d_packed, q.qkv, k.seq * q.qkv, w.dq, w.dk, w.dv, k.rope, 0, 0, dt,
                     stream));
    RUN(dgrad(w.d_packed, q.qkv, k.qkv_w, q.d, w.d_ln));
    RUN(wgrad(w.d_packed, q.qkv, k.ln1, q.d, w.d_qkv_w));
    RUN(bmt_norm_bwd_partial(q.T, q.d, k.x, w.d_ln, k.ln1_w, k.stats1, 1, dt, (int)w.nblk, w.dx, p1, w.d_h1, &rows1, stream));
    const BmtColsum sums[2] = {{p2, rows2, q.d, w.d_ln2_w, 1, 0}, {p1, rows1, q.d, w.d_ln1_w, 1, 0}};
    RUN(bmt_colsum_multi(sums, 2, dt, 0, nullptr, 0, stream));
    return 0;
}

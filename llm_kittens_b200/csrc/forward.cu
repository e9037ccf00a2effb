// The forward pass of a model's transformer blocks in one library call: the same launches in the same order as the entry
// points called one by one from Python (models/transformer.py, _block_forward), on tensors that are stacked over the layers.
//
// Why: a launch costs 2 to 3 us here and 8 us through Python, where every call checks, converts and passes a dozen to
// sixteen arguments, and the forward of a sampler's window was bound by that: GPT-2 124M, 64 tokens, 88 launches of 3 to 6 us:
// 0.71 ms one by one, 0.56 from one call (0.30 of host time).
#include "block_ops.cuh"

using namespace llmk;

namespace {

// One tensor of a block, stacked over the layers `stride` bytes apart (0: one slot that every layer uses).
struct Stacked {
    char* base;
    long long stride;
    void* operator[](int l) const { return base == nullptr ? nullptr : base + (long long)l * stride; }
};
static_assert(sizeof(Stacked) == 16, "two 64-bit words");

// The 64-bit words of the argument block, in the order in which the Python side writes them.
struct Args {
    long long layers, B, T, C, NH, NKVH, HS, H, llama;
    long long rope_mode;                 // Llama: 1 = in the QKV projection's epilogue, 2 = a kernel of its own
    long long rope_interleaved, attention_tc, max_ctas;
    int* status;
    const void* rope;
    const void* x;                       // input of the first block
    Stacked ln1, ln1_mean, ln1_rstd, qkv, atty, lse, res2, ln2, ln2_mean, ln2_rstd, fch, up, gate, act, res3;
    Stacked ln1w, ln1b, qkvw, qkvb, attprojw, attprojb, ln2w, ln2b, fcw, fcb, fcw_up, fcw_gate, fcprojw, fcprojb;
};

enum { NT = 0, BIAS = 1, GELU = 2, ADD = 8 };

thread_local const char* g_refused = "";   // the entry point that this thread's last call ended in

}  // namespace

// The entry point whose refusal or failure the last call of this thread returned.
LLMK_API const char* llmk_forward_layers_refused() { return g_refused; }

// `args`: `words` 64-bit words, laid out as Args.
LLMK_API int llmk_forward_layers(const void* args, long words, float eps, void* stream) {
    g_refused = "llmk_forward_layers";
    if (words * (long)sizeof(long long) != (long)sizeof(Args)) return LLMK_ERR_SHAPE;
    const Args& a = *static_cast<const Args*>(args);
    const int B = (int)a.B, T = (int)a.T, C = (int)a.C, NH = (int)a.NH, KV = (int)a.NKVH, HS = (int)a.HS, H = (int)a.H, mc = (int)a.max_ctas;
    const int M = B * T, W = (NH + 2 * KV) * HS;
    const void* x = a.x;
#define LLMK_TRY(entry, ...)                     \
    do {                                         \
        const int rc_ = entry(__VA_ARGS__);      \
        if (rc_ != LLMK_OK) {                    \
            g_refused = #entry;                  \
            return rc_;                          \
        }                                        \
    } while (0)
    for (int l = 0; l < (int)a.layers; l++) {
        if (a.llama) LLMK_TRY(llmk_rmsnorm_fwd, a.ln1[l], a.ln1_rstd[l], x, a.ln1w[l], M, C, eps, stream);
        else LLMK_TRY(llmk_layernorm_fwd, a.ln1[l], a.ln1_mean[l], a.ln1_rstd[l], x, a.ln1w[l], a.ln1b[l], M, C, stream);
        if (a.llama && a.rope_mode == 1)
            LLMK_TRY(llmk_gemm_qkv_rope, a.ln1[l], a.qkvw[l], a.qkv[l], M, W, C, a.rope, T, (NH + KV) * HS, HS, a.status, mc, nullptr, 1, 0, 0, stream);
        else
            LLMK_TRY(llmk_gemm, NT, a.llama ? 0 : BIAS, a.ln1[l], a.qkvw[l], a.qkv[l], nullptr, a.qkvb[l], nullptr, M, W, C, nullptr, 0, a.status, mc, stream);
        if (a.llama && a.rope_mode == 2)
            LLMK_TRY(llmk_rope_qk, a.qkv[l], a.rope, B, T, NH, KV, HS, (int)a.rope_interleaved, 0, stream);
        if (a.attention_tc) LLMK_TRY(llmk_attention_fwd_tc, a.atty[l], a.lse[l], a.qkv[l], B, T, NH, KV, HS, a.status, stream);
        else LLMK_TRY(llmk_attention_fwd, a.atty[l], a.lse[l], a.qkv[l], B, T, NH, KV, HS, stream);
        LLMK_TRY(llmk_gemm, NT, ADD | (a.llama ? 0 : BIAS), a.atty[l], a.attprojw[l], a.res2[l], nullptr, a.attprojb[l], x, M, C, C, nullptr, 0, a.status,
                 mc, stream);
        if (a.llama) {
            LLMK_TRY(llmk_rmsnorm_fwd, a.ln2[l], a.ln2_rstd[l], a.res2[l], a.ln2w[l], M, C, eps, stream);
            LLMK_TRY(llmk_gemm_swiglu, a.ln2[l], a.fcw_up[l], a.fcw_gate[l], a.act[l], a.up[l], a.gate[l], M, H, C, a.status, mc, nullptr, nullptr, 1, 0,
                     0, stream);
        } else {
            LLMK_TRY(llmk_layernorm_fwd, a.ln2[l], a.ln2_mean[l], a.ln2_rstd[l], a.res2[l], a.ln2w[l], a.ln2b[l], M, C, stream);
            LLMK_TRY(llmk_gemm, NT, BIAS | GELU, a.ln2[l], a.fcw[l], a.act[l], a.fch[l], a.fcb[l], nullptr, M, H, C, nullptr, 0, a.status, mc, stream);
        }
        LLMK_TRY(llmk_gemm, NT, ADD | (a.llama ? 0 : BIAS), a.act[l], a.fcprojw[l], a.res3[l], nullptr, a.fcprojb[l], a.res2[l], M, C, H, nullptr, 0,
                 a.status, mc, stream);
        x = a.res3[l];
    }
#undef LLMK_TRY
    return LLMK_OK;
}

// One prompt portion through all layers of a transformer from one call: the launches of models/prefill.py in the same order, with the
// kernels that it chose, without the interpreter between them (some 12 us a launch there, 3 here; a verification step of five tokens is 36
// launches of 5 to 20 us). What is chosen, allocated and checked stays in Python: this file takes pointers, sizes and one route per
// projection, and keeps nothing. Reference counterpart: the shared command buffers of TransformerModel::forward_prefill_graph
// (crates/rmlx-nn/src/transformer.rs:4416-4620).
#include <cuda_runtime.h>
#include <stdint.h>

extern "C" {
int rmlx_rms_norm(const void* x, const void* residual, const void* w, void* out, void* sum_out, int T, int D, float eps, int pdl, cudaStream_t st);
int rmlx_embedding(const void* table, const int* ids, void* out, int T, int D, int vocab, int pdl, cudaStream_t st);
int rmlx_rope_kv_write(const void* qkv, int qkv_f32, void* q_out, void* k_cache, void* v_cache, const int* block_table, const int* positions,
                       const int* token_seq, const float* cos_t, const float* sin_t, int T, int Hq, int Hkv, int HD, int max_blocks, int page,
                       int traditional, int pdl, cudaStream_t st);
int rmlx_rope_kv_write_q8(const void* qkv, void* q_out, void* k_q, void* k_sb, void* v_q, void* v_sb, const int* block_table,
                          const int* positions, const int* token_seq, const float* cos_t, const float* sin_t, int T, int Hq, int Hkv, int HD,
                          int max_blocks, int page, int traditional, int pdl, cudaStream_t st);
int rmlx_kv_dequant_pages(const void* q, const void* sb, const int* table, void* out, int n_pages, int Hkv, int page, int HD, int pdl,
                          cudaStream_t st);
int rmlx_flash_prefill_paged(const void* q, const void* k_cache, const void* v_cache, const int* block_table, void* out, int T, int Hq, int Hkv,
                             int HD, int pos0, int window, float scale, int pdl, cudaStream_t st);
int rmlx_flash_decode_cluster(const void* q, const void* k_cache, const void* k_sb, const void* v_cache, const void* v_sb, const int* block_table,
                              const int* seq_lens, void* out, int B, int Hq, int Hkv, int HD, int max_blocks, int table_stride, int plan, int window,
                              float scale, int early, int pdl, cudaStream_t st);
int rmlx_flash_prefill_tc(const void* q, const void* k_cache, const void* v_cache, const int* block_table, void* out, int T, int Hq, int Hkv,
                          int HD, int num_blocks, int pos0, int window, float scale, int lanes, int* status, int pdl, cudaStream_t st);
int rmlx_moe_router(const void* gate_w, const void* x, int x_stride, const void* norm_w, float eps, const float* expert_bias, float* logits,
                    int* topk_idx, float* topk_w, int* counts, unsigned int* ticket, int B, int E, int K, int k, int pdl, cudaStream_t st);
int rmlx_topk_route(const float* logits, const float* expert_bias, int* topk_idx, float* topk_w, int* counts, int* offsets, int T, int E, int k,
                    cudaStream_t st);
int rmlx_moe_scatter_rows(const void* x, int x_stride, const int* topk_idx, const int* offsets, int* cursors, void* xs, int* row_of_pair, int T,
                          int top_k, int D, int E, cudaStream_t st);
int rmlx_moe_combine(const void* y, const int* row_of_pair, const float* topk_w, const void* residual, int res_stride, void* out,
                     int out_stride, int T, int top_k, int D, cudaStream_t st);
int rmlx_gemm_bf16(const void* A, const void* W, void* C, const void* residual, int M, int N, int K, int lda, int ldw, int ldc, int bn,
                   int* status, int pdl, cudaStream_t st);
int rmlx_gemm_bf16_f32(const void* A, const void* W, void* C, int M, int N, int K, int lda, int ldw, int ldc, int* status, int pdl,
                       cudaStream_t st);
int rmlx_silu_mul(const void* gate_up, void* act, long long T, int I, cudaStream_t st);
int rmlx_dequant_affine(const void* w, const void* scales, const void* biases, void* out, long long rows, int K, int bits, int scale_f16,
                        cudaStream_t st);
int rmlx_xgemm(int w_kind, const void* A, const void* W, const void* scales, const void* biases, void* C, const void* residual,
               const int* offsets, int E, int M, int N, int K, int lda, int ldc, int bn, int swiglu, float gate_limit, int* status, int pdl,
               cudaStream_t st);
int rmlx_pair_gemm(int w_kind, const void* A, const void* W, const void* scales, const void* biases, void* C, const void* residual,
                   const int* offsets, int E, int M, int N, int K, int lda, int ldc, int swiglu, float gate_limit, int* status, int pdl,
                   cudaStream_t st);
int rmlx_narrow_gemm(int w_kind, const void* w, const void* scales, const void* biases, const void* x, int x_stride, int x_div, const int* order,
                     const int* offsets, int E, const void* norm, float eps, const void* residual, int res_stride, void* out, int out_stride,
                     int out_f32, int M, int N, int K, int swiglu, int tiles, int ks, int pdl, cudaStream_t st);
int rmlx_narrow_group(const int* idx, int pairs, int E, int* offsets, int* order, int pdl, cudaStream_t st);
int rmlx_narrow_combine(const float* y, const int* idx, int E, const float* wts, const void* residual, int res_stride, void* out,
                        int out_stride, int rows, int top_k, int D, int pdl, cudaStream_t st);
int rmlx_row_gemm(const void* A, const void* W, const void* scales, const void* biases, void* C, int out_f32, const void* residual,
                  const int* offsets, int E, int M, int N, int K, int lda, int ldc, int swiglu, float gate_limit, int split, int* status,
                  int pdl, cudaStream_t st);
}

namespace {

// The routes of models/prefill.py (class PromptRun), in its order.
enum Route { kNone = 0, kNarrow = 1, kRow = 2, kPair = 3, kTiles = 4, kBf16 = 5, kExpand = 6 };
// Every launcher here that takes the attribute has kernels that wait for their predecessor before they touch what it writes.
constexpr int kPdl = 1;
constexpr int kWithNorm = 16, kSwiglu = 32;              // narrow: the norm is taken along; SwiGLU in the product's epilogue

struct Linear {
  int64_t w, scales, biases, n, k, experts, kind, scales_f16, route;
};
struct Layer {
  int64_t norm1, norm2, k, v, k_sb, v_sb, router, router_bias, experts, top_k;
  Linear qkv, out, up, down;
};
struct Prompt {
  int64_t layers, t, d, hq, hkv, hd, pos0, window, row_blocks, page, num_blocks, traditional, tensor_cores, lanes, pages, few, vocab;
  int64_t embed, ids, row, pos, zeros, iota, cos, sin, status;
  int64_t h0, h1, xn, qkv, q, attn, act, mid, dense, kk, vv;             // work space
  int64_t logits, idx, wts, counts, offsets, order, cursors, row_of, xs, y;
};

template <class T = void>
T* at(int64_t a) { return reinterpret_cast<T*>(static_cast<uintptr_t>(a)); }

struct Run {
  const Prompt& p;
  float eps;
  cudaStream_t st;
  int rc = 0, launches = 0;
  const char* what = "";

  bool done(int r, const char* name) {
    ++launches;
    if (r != 0 && rc == 0) { rc = r; what = name; }
    return rc == 0;
  }
  // c = x W^T (+ residual), or the gated halves of it
  bool linear(const Linear& w, const void* x, const void* norm, const void* residual, void* c, bool swiglu, const int* offsets = nullptr,
              int rows = 0) {
    const int m = rows ? rows : int(p.t), n = int(w.n), k = int(w.k), ldc = swiglu ? n / 2 : n, e = offsets ? int(w.experts) : 0;
    int* const status = at<int>(p.status);
    switch (w.route & 15) {
      case kNarrow:
        return done(rmlx_narrow_gemm(int(w.kind), at(w.w), at(w.scales), at(w.biases), x, k, 1, nullptr, nullptr, 1, norm, eps, residual, ldc, c,
                                     ldc, 0, m, n, k, swiglu, 0, 0, kPdl, st), "narrow_gemm");
      case kRow:
        return done(rmlx_row_gemm(x, at(w.w), at(w.scales), at(w.biases), c, 0, residual, offsets, e, m, n, k, k, ldc, swiglu, 0.f, 0, status, kPdl,
                                  st), "row_gemm");
      case kPair:
        return done(rmlx_pair_gemm(int(w.kind), x, at(w.w), at(w.scales), at(w.biases), c, residual, offsets, e, m, n, k, k, ldc, swiglu, 0.f,
                                   status, kPdl, st), "pair_gemm");
      case kTiles:
        return done(rmlx_xgemm(int(w.kind), x, at(w.w), at(w.scales), at(w.biases), c, residual, offsets, e, m, n, k, k, ldc, 0, swiglu, 0.f,
                               status, kPdl, st), "xgemm");
      case kExpand:
        if (!done(rmlx_dequant_affine(at(w.w), at(w.scales), at(w.biases), at(p.dense), w.n, k, w.kind == 1 ? 4 : 8, int(w.scales_f16), st),
                  "dequant_affine"))
          return false;
        return done(rmlx_gemm_bf16(x, at(p.dense), c, residual, m, n, k, k, k, ldc, 0, status, kPdl, st), "gemm_bf16");
      case kBf16:
        return done(rmlx_gemm_bf16(x, at(w.w), c, residual, m, n, k, k, k, ldc, 0, status, kPdl, st), "gemm_bf16");
    }
    return done(-2, "prompt_run");
  }
  // rmsnorm(h) W^T, the norm inside where the route says so
  bool norm_linear(const Linear& w, const void* h, const void* norm, void* c, bool swiglu) {
    if (w.route & kWithNorm) return linear(w, h, norm, nullptr, c, swiglu);
    return done(rmlx_rms_norm(h, nullptr, norm, at(p.xn), nullptr, int(p.t), int(p.d), eps, kPdl, st), "rms_norm") &&
           linear(w, at(p.xn), nullptr, nullptr, c, swiglu);
  }
  bool experts(const Layer& l, const void* h, void* out) {
    const int t = int(p.t), d = int(p.d), e = int(l.experts), k = int(l.top_k), pairs = t * k, inner = int(l.up.n / 2);
    int *const idx = at<int>(p.idx), *const offsets = at<int>(p.offsets), *const order = at<int>(p.order), *const row_of = at<int>(p.row_of);
    float* const wts = at<float>(p.wts);
    const bool inside = l.up.route & kWithNorm;          // few rows: their norm is taken along by the router and the experts
    const void* const xn = inside ? h : at(p.xn);
    const void* const norm = inside ? at(l.norm2) : nullptr;
    if (inside) {
      if (!done(rmlx_moe_router(at(l.router), h, d, norm, eps, at<float>(l.router_bias), at<float>(p.logits), idx, wts, nullptr,
                                nullptr, t, e, d, k, kPdl, st), "moe_router"))
        return false;
    } else if (!done(rmlx_rms_norm(h, nullptr, at(l.norm2), at(p.xn), nullptr, t, d, eps, kPdl, st), "rms_norm") ||
               !done(rmlx_gemm_bf16_f32(at(p.xn), at(l.router), at(p.logits), t, e, d, d, d, e, at<int>(p.status), kPdl, st),
                     "gemm_bf16_f32") ||
               !done(rmlx_topk_route(at<float>(p.logits), at<float>(l.router_bias), idx, wts, at<int>(p.counts), offsets, t, e, k, st),
                     "topk_route")) {
      return false;
    }
    if ((l.up.route & 15) == kNarrow) {                  // every chosen expert's weights once for all rows that chose it
      return done(rmlx_narrow_group(idx, pairs, e, offsets, order, kPdl, st), "narrow_group") &&
             done(rmlx_narrow_gemm(int(l.up.kind), at(l.up.w), at(l.up.scales), at(l.up.biases), xn, d, k, order, offsets, e, norm, eps,
                                   nullptr, 0, at(p.act), inner, 0, pairs, int(l.up.n), d, 1, 0, 0, kPdl, st), "narrow_gemm") &&
             done(rmlx_narrow_gemm(int(l.down.kind), at(l.down.w), at(l.down.scales), at(l.down.biases), at(p.act), inner, 1, order, offsets, e,
                                   nullptr, eps, nullptr, 0, at(p.y), d, 1, pairs, d, inner, 0, 0, 0, kPdl, st), "narrow_gemm") &&
             done(rmlx_narrow_combine(at<float>(p.y), idx, e, wts, h, d, out, d, t, k, d, kPdl, st), "narrow_combine");
    }
    return done(rmlx_moe_scatter_rows(at(p.xn), d, idx, offsets, at<int>(p.cursors), at(p.xs), row_of, t, k, d, e, st), "moe_scatter_rows") &&
           linear(l.up, at(p.xs), nullptr, nullptr, at(p.act), true, offsets, pairs) &&
           linear(l.down, at(p.act), nullptr, nullptr, at(p.y), false, offsets, pairs) &&
           done(rmlx_moe_combine(at(p.y), row_of, wts, h, d, out, d, t, k, d, st), "moe_combine");
  }
  bool attention(const Layer& l, float scale) {
    const int t = int(p.t), hq = int(p.hq), hkv = int(p.hkv), hd = int(p.hd), page = int(p.page);
    const int *const row = at<int>(p.row), *const pos = at<int>(p.pos), *const zeros = at<int>(p.zeros);
    const void *k = at(l.k), *v = at(l.v);
    const int* table = row;
    int blocks = int(p.num_blocks);
    if (l.k_sb ? !done(rmlx_rope_kv_write_q8(at(p.qkv), at(p.q), at(l.k), at(l.k_sb), at(l.v), at(l.v_sb), row, pos, zeros, at<float>(p.cos),
                                             at<float>(p.sin), t, hq, hkv, hd, int(p.row_blocks), page, int(p.traditional), kPdl, st),
                       "rope_kv_write_q8")
               : !done(rmlx_rope_kv_write(at(p.qkv), 0, at(p.q), at(l.k), at(l.v), row, pos, zeros, at<float>(p.cos), at<float>(p.sin), t, hq, hkv,
                                          hd, int(p.row_blocks), page, int(p.traditional), kPdl, st), "rope_kv_write"))
      return false;
    if (p.few)                                           // a few rows: the decode kernel, each row a sequence over the same pages
      return done(rmlx_flash_decode_cluster(at(p.q), k, at(l.k_sb), v, at(l.v_sb), row, at<int>(p.iota) + p.pos0 + 1, at(p.attn), t, hq, hkv, hd,
                                            int(p.row_blocks), 0, int(p.few), int(p.window), scale, 0, kPdl, st), "flash_decode_cluster");
    if (l.k_sb) {
      // the 8-bit cache's pages are expanded once per layer into contiguous bf16 pages
      if (!done(rmlx_kv_dequant_pages(at(l.k), at(l.k_sb), row, at(p.kk), int(p.pages), hkv, page, hd, kPdl, st), "kv_dequant_pages") ||
          !done(rmlx_kv_dequant_pages(at(l.v), at(l.v_sb), row, at(p.vv), int(p.pages), hkv, page, hd, kPdl, st), "kv_dequant_pages"))
        return false;
      k = at(p.kk); v = at(p.vv); table = at<int>(p.iota); blocks = int(p.pages);
    }
    if (p.tensor_cores)
      return done(rmlx_flash_prefill_tc(at(p.q), k, v, table, at(p.attn), t, hq, hkv, hd, blocks, int(p.pos0), int(p.window), scale, int(p.lanes),
                                        at<int>(p.status), kPdl, st), "flash_prefill_paged");
    return done(rmlx_flash_prefill_paged(at(p.q), k, v, table, at(p.attn), t, hq, hkv, hd, int(p.pos0), int(p.window), scale, kPdl, st),
                "flash_prefill_paged");
  }
  bool layer(const Layer& l, float scale) {              // h0 -> h0, through h1
    if (!norm_linear(l.qkv, at(p.h0), at(l.norm1), at(p.qkv), false) || !attention(l, scale) ||
        !linear(l.out, at(p.attn), nullptr, at(p.h0), at(p.h1), false))
      return false;
    if (l.router) return experts(l, at(p.h1), at(p.h0));
    const bool inside = l.up.route & kSwiglu;
    return norm_linear(l.up, at(p.h1), at(l.norm2), inside ? at(p.act) : at(p.mid), inside) &&
           (inside || done(rmlx_silu_mul(at(p.mid), at(p.act), p.t, int(l.up.n / 2), st), "silu_mul")) &&
           linear(l.down, at(p.act), nullptr, at(p.h1), at(p.h0), false);
  }
};

}  // namespace

extern "C" int rmlx_prompt_sizes(int* words) {           // of the two records, in 64-bit words: a reader's guard
  words[0] = int(sizeof(Prompt) / 8); words[1] = int(sizeof(Layer) / 8);
  return 0;
}

// Embedding and all layers of one portion: the residual stream ends in h0. Returns the first launch's error (its name in *what).
extern "C" int rmlx_prompt_run(const int64_t* prompt, const int64_t* layers, float eps, float scale, int* launches, const char** what,
                               cudaStream_t st) {
  if (!prompt || !layers || !launches || !what) return -2;
  const Prompt& p = *reinterpret_cast<const Prompt*>(prompt);
  const Layer* const l = reinterpret_cast<const Layer*>(layers);
  Run run{p, eps, st};
  if (run.done(rmlx_embedding(at(p.embed), at<int>(p.ids), at(p.h0), int(p.t), int(p.d), int(p.vocab), 0, st), "embedding"))
    for (int64_t i = 0; i < p.layers && run.layer(l[i], scale); ++i) {}
  *launches = run.launches;
  *what = run.what;
  return run.rc;
}

// Native executor of the packed FastConformer / Nemotron layer stack: one host call enqueues the whole fixed
// kernel sequence of NemotronEncoder.forward's layer loop (oasr/models/nemotron/encoder.py:217-267, 542-583) on the
// caller's stream -- per layer 14 launches, 17 where segments of up to 128 frames keep the
// general attention (4 more with an 8-bit kind: the add + norm kernels also write the quantised
// row for the Linear behind them) of this library's own C-ABI kernels: macaron FFN, Transformer-XL
// relative-position attention (q projected once per global bias, position scores as one batched GEMM over heads,
// one kernel for the relative shift + scale + chunked-limited window, head_dim 128 attention with that bias),
// conv module (GLU GEMM, causal depthwise conv per segment, LayerNorm + SiLU, pointwise GEMM), second FFN, with the
// fp32 residual stream and the fused add + LayerNorm between the sub-layers; with an 8-bit kind every Linear is a
// per-token quantisation of its input followed by the fp8 / int8 GEMM on the pre-quantised weight.  Host code only: no allocation, no host
// synchronisation; launch order and kernel choice are pure functions of the shapes.  The rows are the valid frames of
// all utterances back to back (no padding frame is ever computed).
#include <cmath>

#include "common.cuh"
#include "gemm_small.cuh"

namespace ob {
namespace {

struct FcWorkspace {
  float* res;      // (M, C)   fp32 residual stream
  uint8_t* h;      // (M, C)   16-bit normalised activation
  uint8_t* y;      // (M, C)   16-bit sub-layer output
  uint8_t* a_ffn;  // (M, F)
  uint8_t* qkv4;   // (M, 4C)
  uint8_t* att;    // (M, C)
  uint8_t* g;      // (M, C)
  uint8_t* cv;     // (M, C)
  uint8_t* rel_k;  // (Pp, C)  projected relative-position table of the current layer
  uint8_t* bd;     // (H, M, Pp) position scores
  uint8_t* bias;   // bias_numel elements: block-diagonal attention bias
  uint8_t* q8;     // (M, max(C, F)) 8-bit kinds: the per-token quantised input of the current Linear
  float* qs;       // (M) its row scales
  int64_t bytes;
};

int64_t fc_align(int64_t x) { return (x + 255) / 256 * 256; }

constexpr int64_t kWindowFrames = 128;

int64_t fc_left_chunks(const oasr_b200_fastconformer_model& m, int64_t max_seg) {
  return m.left_context >= 0 ? m.left_context / (m.right_context + 1) : max_seg;
}
// Windowed attention: chosen by the position table's size (2 * longest segment - 1 rows, rounded up to 8), so that scratch
// sizing and execution agree.
bool fc_windowed(const oasr_b200_fastconformer_model& m, int64_t table_rows) {
  return m.rel_window != nullptr && m.left_context >= 0 && table_rows > 2 * kWindowFrames &&
         oasr_b200_fmha_window_supported(m.hidden / m.heads, m.right_context + 1, fc_left_chunks(m, 0)) != 0;
}

FcWorkspace fc_carve(const oasr_b200_fastconformer_model& m, int64_t M, int64_t table_rows, int64_t bias_numel, uint8_t* base) {
  FcWorkspace w{};
  const int64_t C = m.hidden;
  int64_t off = 0;
  auto take = [&](int64_t bytes) {
    uint8_t* p = base ? base + off : nullptr;
    off += fc_align(bytes);
    return p;
  };
  w.res = reinterpret_cast<float*>(take(M * C * 4));
  w.h = take(M * C * 2);
  w.y = take(M * C * 2);
  w.a_ffn = take(M * m.ffn * 2);
  w.qkv4 = take(M * 4 * C * 2);
  w.att = take(M * C * 2);
  w.g = take(M * C * 2);
  w.cv = take(M * C * 2);
  if (!fc_windowed(m, table_rows)) {
    w.rel_k = take(table_rows * C * 2);
    w.bd = take(static_cast<int64_t>(m.heads) * M * table_rows * 2);
    w.bias = take(bias_numel * 2);
  }
  if (m.quant_kind != 0) {
    w.q8 = take(M * (m.ffn > C ? m.ffn : C));
    w.qs = reinterpret_cast<float*>(take(M * 4));
  }
  w.bytes = off;
  return w;
}

struct FcChunkWorkspace {
  float* res;
  uint8_t *h, *y, *a_ffn, *qkv4, *att, *g, *xcat, *cv;
  int64_t bytes;
};

FcChunkWorkspace fc_carve_chunk(const oasr_b200_fastconformer_model& m, int64_t B, int64_t Tq, uint8_t* base) {
  FcChunkWorkspace w{};
  const int64_t C = m.hidden, M = B * Tq;
  int64_t off = 0;
  auto take = [&](int64_t bytes) {
    uint8_t* p = base ? base + off : nullptr;
    off += fc_align(bytes);
    return p;
  };
  w.res = reinterpret_cast<float*>(take(M * C * 4));
  w.h = take(M * C * 2);
  w.y = take(M * C * 2);
  w.a_ffn = take(M * m.ffn * 2);
  w.qkv4 = take(M * 4 * C * 2);
  w.att = take(M * C * 2);
  w.g = take(M * C * 2);
  w.xcat = take(B * (Tq + m.kernel - 1) * C * 2);
  w.cv = take(M * C * 2);
  w.bytes = off;
  return w;
}

}  // namespace
}  // namespace ob

extern "C" {

int64_t oasr_b200_fastconformer_workspace_bytes(const oasr_b200_fastconformer_model* model, int64_t total,
                                                int64_t table_rows, int64_t bias_numel) {
  if (!model || total < 0 || table_rows < 0 || bias_numel < 0) return -1;
  return ob::fc_carve(*model, total, table_rows, bias_numel, nullptr).bytes;
}

#define FC_STEP(call)                  \
  do {                                 \
    int rc_ = (call);                  \
    if (rc_ != OASR_OK) return rc_;    \
  } while (0)

int oasr_b200_fastconformer_layers_packed(const oasr_b200_fastconformer_model* model, const void* rows, int rows_f32, float* out,
                                          const void* rel_table, int64_t table_rows, const int32_t* cu_seqlens,
                                          const int64_t* bias_offsets, int64_t bias_numel, int64_t num_segs,
                                          int64_t total, int64_t max_seg, void* workspace, int64_t workspace_bytes,
                                          void* stream) {
  using namespace ob;
  OB_REQUIRE(model && model->layers, OASR_ERR_INVALID, "fastconformer_layers_packed: null model");
  const oasr_b200_fastconformer_model& m = *model;
  OB_REQUIRE(m.num_layers > 0 && m.hidden > 0 && m.heads > 0 && m.hidden % m.heads == 0 &&
                 (m.hidden / m.heads == 64 || m.hidden / m.heads == 128),
             OASR_ERR_UNSUPPORTED, "fastconformer_layers_packed: head_dim must be 64 or 128 (hidden %d, heads %d)", m.hidden,
             m.heads);
  OB_REQUIRE(m.kernel > 0 && m.ffn > 0 && m.right_context >= 0, OASR_ERR_INVALID, "fastconformer_layers_packed: bad model geometry");
  OB_REQUIRE(num_segs >= 0 && total >= 0 && max_seg >= 0 && bias_numel >= 0, OASR_ERR_INVALID, "fastconformer_layers_packed: bad shape");
  if (total == 0 || num_segs == 0) return OASR_OK;
  const bool windowed = fc_windowed(m, table_rows);
  OB_REQUIRE(rows && out && cu_seqlens && workspace && (windowed || (rel_table && bias_offsets)), OASR_ERR_INVALID,
             "fastconformer_layers_packed: null pointer argument");
  OB_REQUIRE(table_rows >= 2 * max_seg - 1 && table_rows % 8 == 0, OASR_ERR_INVALID,
             "fastconformer_layers_packed: the position table needs >= 2*max_seg-1 rows, a multiple of 8 (got %lld for %lld frames)",
             (long long)table_rows, (long long)max_seg);
  OB_REQUIRE(is_aligned(workspace, 256), OASR_ERR_ALIGN, "fastconformer_layers_packed: workspace must be 256-byte aligned");
  FcWorkspace w = fc_carve(m, total, table_rows, bias_numel, static_cast<uint8_t*>(workspace));
  OB_REQUIRE(workspace_bytes >= w.bytes, OASR_ERR_INVALID, "fastconformer_layers_packed: workspace of %lld bytes, %lld needed",
             (long long)workspace_bytes, (long long)w.bytes);
  const int64_t M = total, C = m.hidden, F = m.ffn, H = m.heads, D = C / H, L = m.num_layers, Pp = table_rows;
  const int dt = m.dtype;
  const size_t es = 2;
  const double scale = 1.0 / std::sqrt(static_cast<double>(D));
  const int64_t chunk = m.right_context + 1;
  const int64_t left_chunks = fc_left_chunks(m, max_seg);
  const bool conv_norm = oasr_b200_dwconv_norm_swish_supported(C, m.kernel) != 0 && num_segs < 65536;
  const oasr_b200_fastconformer_layer* ly = m.layers;
  const double eps = m.eps;

  // One Linear: 16-bit GEMM, or per-token quantisation of the input followed by the 8-bit GEMM on the layer's
  // pre-quantised weight `qi` (order of oasr_b200_fastconformer_layer::q_w).
  const int qk = m.quant_kind;
  OB_REQUIRE(qk == 0 || qk == OASR_Q8_FP8_E4M3 || qk == OASR_Q8_INT8, OASR_ERR_INVALID, "fastconformer_layers_packed: bad quant_kind %d", qk);
#define FC_LINEAR(out, in, wt, bs, lay, qi, N, K, act, glu)                                                           \
  do {                                                                                                                \
    if (qk == 0) {                                                                                                    \
      if (glu) FC_STEP(oasr_b200_gemm_glu(out, in, wt, bs, M, N, K, dt, stream));                                       \
      else FC_STEP(oasr_b200_gemm(out, in, wt, bs, M, N, K, act, dt, stream));                                          \
    } else {                                                                                                          \
      OB_REQUIRE((lay).q_w[qi] && (lay).q_s[qi], OASR_ERR_INVALID, "fastconformer_layers_packed: layer without 8-bit weight %d", qi); \
      FC_STEP(oasr_b200_quantize_rows(w.q8, w.qs, in, M, K, qk, dt, stream));                                          \
      FC_STEP(oasr_b200_gemm_q8(out, w.q8, w.qs, (lay).q_w[qi], (lay).q_s[qi], bs, M, N, K, act, glu, qk, dt, stream)); \
    }                                                                                                                 \
  } while (0)

  // A Linear whose input h was produced (and, with an 8-bit kind, already quantised into w.q8 / w.qs) by the add + norm
  // directly before it.
#define FC_LINEAR_H(out, wt, bs, lay, qi, N, K, act, glu)                                                            \
  do {                                                                                                                \
    if (qk == 0) {                                                                                                    \
      FC_LINEAR(out, w.h, wt, bs, lay, qi, N, K, act, glu);                                                           \
    } else {                                                                                                          \
      OB_REQUIRE((lay).q_w[qi] && (lay).q_s[qi], OASR_ERR_INVALID, "fastconformer_layers_packed: layer without 8-bit weight %d", qi); \
      FC_STEP(oasr_b200_gemm_q8(out, w.q8, w.qs, (lay).q_w[qi], (lay).q_s[qi], bs, M, N, K, act, glu, qk, dt, stream)); \
    }                                                                                                                 \
  } while (0)
  // add + norm into w.h, and with an 8-bit kind the quantised row for the Linear that follows
#define FC_ADD_NORM(res_in_, y_, alpha_, mode_, wa, ba, wb, bb)                                                       \
  FC_STEP(oasr_b200_add_norm_f32_q8(w.h, res, res_in_, y_, alpha_, mode_, wa, ba, wb, bb, M, C, eps, 0,                \
                                    qk ? w.q8 : nullptr, qk ? w.qs : nullptr, qk, dt, stream))

  // the input rows (16-bit, or fp32 when rows_f32) start the fp32 residual stream; h = LN_ff1(x) of the first layer in
  // the same kernel
  float* res = w.res;
  if (rows_f32) {
    FC_ADD_NORM(static_cast<const float*>(rows), nullptr, 0.0, 0, ly[0].norm_ff1_w, ly[0].norm_ff1_b, nullptr, nullptr);
  } else {
    FC_ADD_NORM(nullptr, rows, 1.0, 0, ly[0].norm_ff1_w, ly[0].norm_ff1_b, nullptr, nullptr);
  }
  for (int64_t i = 0; i < L; ++i) {
    const oasr_b200_fastconformer_layer& l = ly[i];
    // macaron feed-forward: x += 0.5 * W2 silu(W1 h)
    FC_LINEAR_H(w.a_ffn, l.ff1_w1, l.ff1_b1, l, 0, F, C, OASR_ACT_SWISH, 0);
    FC_LINEAR(w.y, w.a_ffn, l.ff1_w2, l.ff1_b2, l, 1, C, F, OASR_ACT_NONE, 0);
    FC_ADD_NORM(res, w.y, 0.5, 0, l.norm_att_w, l.norm_att_b, nullptr, nullptr);
    // attention: [q+u | q+v | k | v] of every row, position scores (q+v) . rel_k^T per head, shifted bias, attention
    FC_LINEAR_H(w.qkv4, l.qkv4_w, l.qkv4_b, l, 2, 4 * C, C, OASR_ACT_NONE, 0);
    if (windowed) {
      FC_STEP(oasr_b200_fmha_window_packed(w.att, w.qkv4, static_cast<const uint8_t*>(m.rel_window) + i * 64 * C * es, 64,
                                           left_chunks * chunk + chunk - 1, cu_seqlens, num_segs, max_seg, M, H, D, chunk, left_chunks,
                                           scale, dt, stream));
    } else {
      FC_STEP(oasr_b200_gemm(w.rel_k, rel_table, l.rel_w, nullptr, Pp, C, C, OASR_ACT_NONE, dt, stream));
      FC_STEP(oasr_b200_bmm_strided(w.bd, w.qkv4 + C * es, w.rel_k, H, M, Pp, D, 4 * C, D, C, D, dt, stream));
      FC_STEP(oasr_b200_relshift_bias_packed(w.bias, w.bd, cu_seqlens, bias_offsets, num_segs, H, M, max_seg, Pp, scale, chunk,
                                             left_chunks, m.mask_floor, dt, stream));
      FC_STEP(oasr_b200_fmha_varlen_strided(w.att, w.qkv4, w.qkv4 + 2 * C * es, w.qkv4 + 3 * C * es, 4 * C, 4 * C, 4 * C, w.bias,
                                            bias_offsets, 1, 1, cu_seqlens, cu_seqlens, num_segs, M, M, max_seg, H, H, D, scale, dt,
                                            stream));
    }
    FC_LINEAR(w.y, w.att, l.o_w, l.o_b, l, 3, C, C, OASR_ACT_NONE, 0);
    FC_ADD_NORM(res, w.y, 1.0, 0, l.norm_conv_w, l.norm_conv_b, nullptr, nullptr);
    // conv module: pointwise + GLU, causal depthwise conv per segment, LayerNorm + SiLU, pointwise
    FC_LINEAR_H(w.g, l.pw1_w, l.pw1_b, l, 4, C, C, OASR_ACT_NONE, 1);
    if (conv_norm) {
      FC_STEP(oasr_b200_dwconv_norm_swish_packed(w.cv, w.g, l.dw_w, l.dw_b, l.conv_norm_w, l.conv_norm_b, cu_seqlens, num_segs, max_seg, M, C,
                                                 m.kernel, 1e-5, dt, stream));
    } else {
      FC_STEP(oasr_b200_depthwise_conv1d_packed_causal(w.att, w.g, l.dw_w, l.dw_b, cu_seqlens, num_segs, max_seg, C, m.kernel, -1, dt,
                                                       stream));
      FC_STEP(oasr_b200_layer_norm_activation(w.cv, w.att, l.conv_norm_w, l.conv_norm_b, M, C, 1e-5, OASR_ACT_SWISH, dt, stream));
    }
    FC_LINEAR(w.y, w.cv, l.pw2_w, l.pw2_b, l, 5, C, C, OASR_ACT_NONE, 0);
    FC_ADD_NORM(res, w.y, 1.0, 0, l.norm_ff2_w, l.norm_ff2_b, nullptr, nullptr);
    // second feed-forward, norm_out, then the next layer's first pre-norm in the same kernel
    FC_LINEAR_H(w.a_ffn, l.ff2_w1, l.ff2_b1, l, 6, F, C, OASR_ACT_SWISH, 0);
    FC_LINEAR(w.y, w.a_ffn, l.ff2_w2, l.ff2_b2, l, 7, C, F, OASR_ACT_NONE, 0);
    if (i + 1 < L) {
      FC_ADD_NORM(res, w.y, 0.5, 2, l.norm_out_w, l.norm_out_b, ly[i + 1].norm_ff1_w, ly[i + 1].norm_ff1_b);
    } else {
      FC_STEP(oasr_b200_add_norm_f32(w.h, out, res, w.y, 0.5, 2, l.norm_out_w, l.norm_out_b, l.norm_out_w, l.norm_out_b, M, C, eps, 0,
                                     dt, stream));
    }
  }
  return OASR_OK;
}

int64_t oasr_b200_fastconformer_chunk_workspace_bytes(const oasr_b200_fastconformer_model* model, int64_t B, int64_t Tq) {
  if (!model || B < 0 || Tq < 0) return -1;
  return ob::fc_carve_chunk(*model, B, Tq, nullptr).bytes;
}

int oasr_b200_fastconformer_chunk_paged(const oasr_b200_fastconformer_model* model, const void* rows, int rows_f32, float* out,
                                        int64_t B, int64_t Tq, void* const* k_pools, void* const* v_pools,
                                        const int32_t* block_table, const int32_t* cached, const int32_t* pos_start,
                                        int64_t blocks_per_seq, int64_t block_size, int64_t num_blocks, void* cnn_state,
                                        int64_t num_slots, const int64_t* slot_ids, void* workspace, int64_t workspace_bytes,
                                        void* stream) {
  using namespace ob;
  OB_REQUIRE(model && model->layers, OASR_ERR_INVALID, "fastconformer_chunk_paged: null model");
  const oasr_b200_fastconformer_model& m = *model;
  OB_REQUIRE(m.num_layers > 0 && m.hidden > 0 && m.heads > 0 && m.hidden % m.heads == 0 && m.kernel > 0 && m.ffn > 0 &&
                 m.right_context >= 0 && m.left_context >= 0,
             OASR_ERR_INVALID, "fastconformer_chunk_paged: bad model geometry");
  const int64_t C = m.hidden, F = m.ffn, H = m.heads, D = C / H, L = m.num_layers, M = B * Tq, SL = m.kernel - 1;
  const int64_t chunk = m.right_context + 1, left_chunks = fc_left_chunks(m, 0);
  OB_REQUIRE(m.rel_window && m.quant_kind == 0 && oasr_b200_fmha_window_supported(D, chunk, left_chunks) != 0, OASR_ERR_UNSUPPORTED,
             "fastconformer_chunk_paged: needs 16-bit Linears, the windowed position table and a window that fits it");
  OB_REQUIRE(B >= 0 && Tq > 0, OASR_ERR_INVALID, "fastconformer_chunk_paged: bad shape");
  if (B == 0) return OASR_OK;
  OB_REQUIRE(rows && out && k_pools && v_pools && block_table && cached && pos_start && cnn_state && slot_ids && workspace,
             OASR_ERR_INVALID, "fastconformer_chunk_paged: null pointer argument");
  OB_REQUIRE(is_aligned(workspace, 256), OASR_ERR_ALIGN, "fastconformer_chunk_paged: workspace must be 256-byte aligned");
  FcChunkWorkspace w = fc_carve_chunk(m, B, Tq, static_cast<uint8_t*>(workspace));
  OB_REQUIRE(workspace_bytes >= w.bytes, OASR_ERR_INVALID, "fastconformer_chunk_paged: workspace of %lld bytes, %lld needed",
             (long long)workspace_bytes, (long long)w.bytes);
  const int dt = m.dtype;
  const double scale = 1.0 / std::sqrt(static_cast<double>(D)), eps = m.eps;
  const oasr_b200_fastconformer_layer* ly = m.layers;
  const bool conv_norm = oasr_b200_dwconv_norm_swish_supported(C, m.kernel) != 0 && B < 65536;
  const Chain inner = inner_chain(starts_late(gsm::kStore, M, F, C));   // see gemm_small.cuh
  // last Linear of a sub-layer + residual + norm (mode 2: norm_out and the next pre-norm); few rows: the Linear adds into
  // the fp32 stream itself
#define FC_CHUNK_LINEAR_ADDNORM(in, wt, bs, K, alpha, mode, res_to, wa, ba, wb, bb)                                     \
  do {                                                                                                                \
    if (gsm::takes(gsm::kResid, M, C, K)) {                                                                           \
      FC_STEP(gemm_residual_f32_op(w.res, w.res, in, wt, bs, M, C, K, alpha, dt, stream, inner));                     \
      FC_STEP(oasr_b200_add_norm_f32(w.h, (mode) == 2 ? res_to : nullptr, w.res, nullptr, 0.0, mode, wa, ba, wb, bb, M, C, eps, 0, dt, stream)); \
    } else {                                                                                                          \
      FC_STEP(gemm_op(w.y, in, wt, bs, M, C, K, OASR_ACT_NONE, dt, stream, inner));                                   \
      FC_STEP(oasr_b200_add_norm_f32(w.h, res_to, w.res, w.y, alpha, mode, wa, ba, wb, bb, M, C, eps, 0, dt, stream)); \
    }                                                                                                                 \
  } while (0)
  if (rows_f32) {
    FC_STEP(oasr_b200_add_norm_f32(w.h, w.res, static_cast<const float*>(rows), nullptr, 0.0, 0, ly[0].norm_ff1_w, ly[0].norm_ff1_b,
                                   nullptr, nullptr, M, C, eps, 0, dt, stream));
  } else {
    FC_STEP(oasr_b200_add_norm_f32(w.h, w.res, nullptr, rows, 1.0, 0, ly[0].norm_ff1_w, ly[0].norm_ff1_b, nullptr, nullptr, M, C, eps, 0,
                                   dt, stream));
  }
  for (int64_t i = 0; i < L; ++i) {
    const oasr_b200_fastconformer_layer& l = ly[i];
    FC_STEP(gemm_op(w.a_ffn, w.h, l.ff1_w1, l.ff1_b1, M, F, C, OASR_ACT_SWISH, dt, stream, i == 0 ? Chain{0, 1} : inner));
    FC_CHUNK_LINEAR_ADDNORM(w.a_ffn, l.ff1_w2, l.ff1_b2, F, 0.5, 0, w.res, l.norm_att_w, l.norm_att_b, nullptr, nullptr);
    // attention over the cached pages and the chunk, which the kernel also appends to the pages
    FC_STEP(gemm_op(w.qkv4, w.h, l.qkv4_w, l.qkv4_b, M, 4 * C, C, OASR_ACT_NONE, dt, stream, inner));
    FC_STEP(oasr_b200_fmha_window_paged(w.att, w.qkv4, k_pools[i], v_pools[i], static_cast<const uint8_t*>(m.rel_window) + i * 64 * C * 2, 64,
                                        left_chunks * chunk + chunk - 1, block_table, cached, pos_start, B, Tq, H, D, blocks_per_seq,
                                        block_size, num_blocks, chunk, left_chunks, scale, dt, stream));
    FC_CHUNK_LINEAR_ADDNORM(w.att, l.o_w, l.o_b, C, 1.0, 0, w.res, l.norm_conv_w, l.norm_conv_b, nullptr, nullptr);
    // conv module continuing from the stream's post-GLU tail
    FC_STEP(gemm_glu_op(w.g, w.h, l.pw1_w, l.pw1_b, M, C, C, dt, stream, inner));
    uint8_t* state = static_cast<uint8_t*>(cnn_state) + i * num_slots * SL * C * 2;
    if (conv_norm) {
      FC_STEP(oasr_b200_dwconv_norm_swish_stream(w.cv, w.g, l.dw_w, l.dw_b, l.conv_norm_w, l.conv_norm_b, state, num_slots, slot_ids, B, Tq, C,
                                                 m.kernel, 1e-5, dt, stream));
    } else {
      FC_STEP(oasr_b200_conv_state_concat(w.xcat, state, num_slots, slot_ids, w.g, B, SL, Tq, C, dt, stream));
      FC_STEP(oasr_b200_depthwise_conv1d(w.att, w.xcat, l.dw_w, l.dw_b, B, SL + Tq, C, m.kernel, 0, 0, nullptr, 0, 0, OASR_ACT_NONE, dt, stream));
      FC_STEP(oasr_b200_layer_norm_activation(w.cv, w.att, l.conv_norm_w, l.conv_norm_b, M, C, 1e-5, OASR_ACT_SWISH, dt, stream));
    }
    FC_CHUNK_LINEAR_ADDNORM(w.cv, l.pw2_w, l.pw2_b, C, 1.0, 0, w.res, l.norm_ff2_w, l.norm_ff2_b, nullptr, nullptr);
    FC_STEP(gemm_op(w.a_ffn, w.h, l.ff2_w1, l.ff2_b1, M, F, C, OASR_ACT_SWISH, dt, stream, inner));
    if (i + 1 < L) {
      FC_CHUNK_LINEAR_ADDNORM(w.a_ffn, l.ff2_w2, l.ff2_b2, F, 0.5, 2, w.res, l.norm_out_w, l.norm_out_b, ly[i + 1].norm_ff1_w, ly[i + 1].norm_ff1_b);
    } else {
      FC_CHUNK_LINEAR_ADDNORM(w.a_ffn, l.ff2_w2, l.ff2_b2, F, 0.5, 2, out, l.norm_out_w, l.norm_out_b, l.norm_out_w, l.norm_out_b);
    }
  }
  return OASR_OK;
}

}  // extern "C"

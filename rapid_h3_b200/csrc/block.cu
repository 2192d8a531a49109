// One fused DiT block as a list of launches: the host side of the block in native code. Bound by the launches themselves:
// driven from Python, the 16 calls of a block cost 440 us of interpreter, argument conversion and buffer allocation, which
// is all of the time of a small step and most of that of one picture: two blocks on 115 tokens 1.26 -> 0.57 ms, two blocks
// on two samples of 1,008 tokens (width 4,096) 2.23 -> 2.01 ms.
// The buffers of a block overlap where their lifetimes do not: codes | bf16 rows (q|k|v, then the attention output, then the
// MLP's hidden rows) | attention operands, then the hidden rows' codes.
#include <math.h>

#include "common.cuh"
#include "rapidh3_b200.h"

namespace {

struct Workspace {
  int64_t bytes = 0;
  int64_t take(int64_t n) {
    const int64_t at = bytes;
    bytes += (n + 255) / 256 * 256;
    return at;
  }
};

int64_t pad(int64_t n, int64_t to) { return (n + to - 1) / to * to; }

// offsets of one block's buffers
struct Layout {
  int64_t codes, scales, rows, q8, k8, vt, hidden_codes, qs, ks, stats, scratch, scratch_bytes, text_codes, text_scales, text_kv;
  int64_t bytes;
  explicit Layout(const rh3_block_args& b) {
    const int64_t S = b.S, hd = b.heads * 128, T = b.cross ? b.text : 0, lk = S > T ? S : T;
    const int64_t qp = pad(S, 256), kp = pad(lk, 128);
    Workspace w;
    codes = w.take(S * (b.d > hd ? b.d : hd));
    scales = w.take(4 * S);
    rows = w.take(2 * S * (3 * hd > b.mlp ? 3 * hd : b.mlp));
    const int64_t operands = w.bytes;
    q8 = w.take(hd * qp);
    k8 = w.take(hd * kp);
    vt = w.take(hd * kp);
    hidden_codes = operands;
    if (w.bytes < operands + S * b.mlp) w.bytes = operands + pad(S * b.mlp, 256);
    qs = w.take(4 * b.heads * (b.token_attn ? qp : qp / 64));
    ks = w.take(4 * b.heads * (b.token_attn ? 2 * kp : kp / 64));
    stats = w.take(3 * 4 * hd);
    scratch_bytes = rh3_attn_kv_stats_scratch_bytes(lk, b.heads);
    scratch = w.take(scratch_bytes);
    text_codes = w.take(T * b.text_dim);
    text_scales = w.take(4 * T);
    text_kv = w.take(2 * T * 2 * hd);
    bytes = w.bytes;
  }
};

}  // namespace

extern "C" int64_t rh3_block_workspace_bytes(const rh3_block_args* b) {
  if (!b || b->S <= 0 || b->d <= 0 || b->heads <= 0 || b->mlp <= 0 || b->text < 0 || b->text_dim < 0) return 0;
  return Layout(*b).bytes;
}

extern "C" int rh3_block_forward(const rh3_block_args* args, void* workspace, int64_t workspace_bytes, cudaStream_t stream) {
  RH3_CHECK_ARG(args && workspace, "block_forward: null pointer");
  const rh3_block_args& b = *args;
  RH3_CHECK_ARG(b.S > 0 && b.d > 0 && b.heads > 0 && b.mlp > 0 && (!b.cross || (b.text > 0 && b.text_dim > 0)),
                "block_forward: bad shape S=%lld d=%lld heads=%lld mlp=%lld text=%lld", (long long)b.S, (long long)b.d,
                (long long)b.heads, (long long)b.mlp, (long long)b.text);
  RH3_CHECK_ARG((reinterpret_cast<uintptr_t>(workspace) & 255) == 0, "block_forward: the workspace must be 256-byte aligned");
  const Layout at(b);
  RH3_CHECK_ARG(workspace_bytes >= at.bytes, "block_forward: workspace of %lld bytes, %lld needed", (long long)workspace_bytes,
                (long long)at.bytes);
  const int64_t S = b.S, d = b.d, H = b.heads, hd = H * 128, f = b.mlp;
  uint8_t* const ws = static_cast<uint8_t*>(workspace);
  void* const codes = ws + at.codes;
  float* const scales = reinterpret_cast<float*>(ws + at.scales);
  __nv_bfloat16* const rows = reinterpret_cast<__nv_bfloat16*>(ws + at.rows);

  auto norm_quant = [&](const void* weight, double eps, const int32_t* idx, const float* shift, const float* scale, int64_t ld) {
    return (b.rotate ? rh3_norm_mod_rot_quant_rows_i8 : rh3_norm_mod_quant_rows_i8)(
        b.x, b.ldx, weight, static_cast<float>(eps), idx, shift, scale, ld, S, d, codes, d, scales, stream);
  };
  auto row_quant = [&](const void* x, int64_t M, int64_t K, void* q, float* s) {
    return (b.rotate ? rh3_rot_quant_rows_i8 : rh3_quant_rows_i8)(x, K, M, K, q, K, s, stream);
  };
  // q [S, H, 128] at row stride q_ss, k and v [L, H, 128] at row stride k_ss -> attention output in `rows` [S, H * 128].
  // The output may lie over q, k and v: the pre-pass has turned them into the operands by then.
  auto attention = [&](const __nv_bfloat16* q, int64_t q_ss, __nv_bfloat16* k, const __nv_bfloat16* v, int64_t k_ss, int64_t L,
                       const void* qw, const void* kw, double eps, const void* rope) -> int {
    const int64_t qp = pad(S, 256), kp = pad(L, 128);
    void *q8 = ws + at.q8, *k8 = ws + at.k8, *vt = ws + at.vt;
    float *qs = reinterpret_cast<float*>(ws + at.qs), *ks = reinterpret_cast<float*>(ws + at.ks);
    float *kmean = reinterpret_cast<float*>(ws + at.stats), *vmean = kmean + hd, *vscale = vmean + hd;
    const float softmax_scale = static_cast<float>(1.0 / sqrt(128.0));
    if (int e = (b.token_attn ? rh3_attn_tok_prepass : rh3_attn_prepass)(
            q, q_ss, 128, S, qp, k, k_ss, 128, v, k_ss, 128, L, kp, H, qw, kw, static_cast<float>(eps), rope, nullptr, 0, 0, k, k_ss,
            128, ws + at.scratch, at.scratch_bytes, q8, qs, k8, ks, vt, vscale, vmean, kmean, stream))
      return e;
    return (b.token_attn ? rh3_attn_int8_tok : rh3_attn_int8)(q8, qs, k8, ks, vt, vscale, vmean, S, qp, L, kp, H, softmax_scale, rows,
                                                              hd, 128, stream);
  };
#define RH3_STEP(call) \
  if (int e = (call)) return e

  // ---- self-attention ----
  RH3_STEP(norm_quant(b.norm1, b.eps1, b.idx, b.shift_msa, b.scale_msa, b.table_stride));
  RH3_STEP(rh3_gemm_w8a8(codes, d, b.qkv, scales, b.qkv_s, nullptr, S, 3 * hd, d, RH3_KIND_I8, rows, 3 * hd, nullptr, stream));
  RH3_STEP(attention(rows, 3 * hd, rows + hd, rows + 2 * hd, 3 * hd, S, b.q_norm, b.k_norm, b.eps_qk, b.rope));
  RH3_STEP(row_quant(rows, S, hd, codes, scales));
  RH3_STEP(rh3_gemm_w8a8_gated_residual2(codes, hd, b.out, scales, b.out_s, b.gate_msa + b.row0 * b.table_stride,
                                         b.gate_msa + b.row1 * b.table_stride, b.split, b.x, b.ldx, S, d, hd, RH3_KIND_I8, stream));
  // ---- cross-attention to text ----
  if (b.cross) {
    __nv_bfloat16* const kv = reinterpret_cast<__nv_bfloat16*>(ws + at.text_kv);
    void* const text_codes = ws + at.text_codes;
    float* const text_scales = reinterpret_cast<float*>(ws + at.text_scales);
    RH3_STEP(norm_quant(b.norm_c, b.eps_c, b.idx0, b.zeros, b.zeros, d));
    RH3_STEP(rh3_gemm_w8a8(codes, d, b.cq, scales, b.cq_s, nullptr, S, hd, d, RH3_KIND_I8, rows, hd, nullptr, stream));
    RH3_STEP((b.rotate ? rh3_rot_quant_rows_i8 : rh3_quant_rows_i8)(b.ctx, b.ld_ctx, b.text, b.text_dim, text_codes, b.text_dim,
                                                                    text_scales, stream));
    RH3_STEP(rh3_gemm_w8a8(text_codes, b.text_dim, b.ckv, text_scales, b.ckv_s, nullptr, b.text, 2 * hd, b.text_dim, RH3_KIND_I8, kv,
                           2 * hd, nullptr, stream));
    RH3_STEP(attention(rows, hd, kv, kv + hd, 2 * hd, b.text, b.cq_norm, b.ck_norm, b.eps_cqk, nullptr));
    RH3_STEP(row_quant(rows, S, hd, codes, scales));
    RH3_STEP(rh3_gemm_w8a8_gated_residual(codes, hd, b.co, scales, b.co_s, b.ones, b.x, b.ldx, S, d, hd, RH3_KIND_I8, stream));
  }
  // ---- MLP ----
  RH3_STEP(norm_quant(b.norm2, b.eps2, b.idx, b.shift_mlp, b.scale_mlp, b.table_stride));
  RH3_STEP(rh3_gemm_w8a8_swiglu(codes, d, b.fc1, scales, b.fc1_s, S, 2 * f, d, RH3_KIND_I8, rows, f, stream));
  RH3_STEP(row_quant(rows, S, f, ws + at.hidden_codes, scales));
  RH3_STEP(rh3_gemm_w8a8_gated_residual2(ws + at.hidden_codes, f, b.fc2, scales, b.fc2_s, b.gate_mlp + b.row0 * b.table_stride,
                                         b.gate_mlp + b.row1 * b.table_stride, b.split, b.x, b.ldx, S, d, f, RH3_KIND_I8, stream));
#undef RH3_STEP
  return 0;
}

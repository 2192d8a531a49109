// Per-token (row) activation quantizers: abs-max symmetric int8 / fp8-e4m3 with optional fused
// prologues. One CTA owns one row; the row is read ONCE from HBM with 128-bit loads, held in
// registers through the prologue, the abs-max reduction and the quantization, and the codes are
// written once. HBM-bound: algorithmic traffic is 2 bytes in + 1 byte out per element.
//
// Semantics follow the reference's PyTorch emulation exactly (bit-exact codes and scales):
//   int8: s = max(amax/127, 1e-12), q = clamp(round_half_even(x / s), -127, 127)
//   fp8 : s = max(amax/448, 1e-12), q = e4m3_rn(clamp(x / s, -448, 448))
// (reference: custom_nodes/rapid_h3/kernels.py:75-82; fast kernels triton_fp8.py:17-64).
// Prologues (reference: triton_fp8.py:128-148 `_load_act`):
//   KIND_PLAIN   x
//   KIND_SWIGLU  silu(x[:, k]) * x[:, F + k]
//   KIND_NORMMOD rms_norm(x) * w * (1 + scale[idx[row]]) + shift[idx[row]]
//   KIND_HEADS   x given group-major [G, M, gw] (gw = 128: head-major attention output);
//                output column k = group k/gw, channel k%gw
// The division x / s is done as fma(x, 1/s, 1.5 * 2^23) with an exact IEEE re-division only for the rare values
// whose product lands within 2^-14 of a rounding tie (product and rounded quotient are each at most 7.6e-6 away
// from the true quotient), which keeps the codes identical to a true division.
#include "common.cuh"
#include "rapidh3_b200.h"

namespace rh3 {
namespace {

enum { KIND_PLAIN = 0, KIND_SWIGLU = 1, KIND_NORMMOD = 2, KIND_HEADS = 3 };

struct QuantParams {
  const __nv_bfloat16* x;
  int64_t ldx;        // row stride of x in elements (KIND_HEADS: stride between heads)
  int64_t M, K;       // rows, quantized width
  void* q;
  int64_t ldq;
  float* s;
  // KIND_NORMMOD
  const __nv_bfloat16* w;  // may be null
  float eps;
  const int32_t* idx;
  const float* shift;
  const float* scale;
  int64_t ld_tab;
  // KIND_SWIGLU: F == K, the up half starts at column K
  int gw;  // KIND_HEADS: columns per group (128 for one head); x is [K/gw, M, gw] with group stride ldx
  const float* tensor_amax;  // when set: one abs-max for the whole tensor replaces every row's own (per-tensor scale)
};

__device__ __forceinline__ void unpack8(const uint4& u, float* v) {
  v[0] = bf16_lo(u.x); v[1] = bf16_hi(u.x); v[2] = bf16_lo(u.y); v[3] = bf16_hi(u.y);
  v[4] = bf16_lo(u.z); v[5] = bf16_hi(u.z); v[6] = bf16_lo(u.w); v[7] = bf16_hi(u.w);
}

// block-wide max over T threads; result returned to all threads
template <int T>
__device__ __forceinline__ float block_max(float v, float* red) {
  v = warp_max(v);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (lane == 0) red[warp] = v;
  __syncthreads();
  float r = red[0];
#pragma unroll
  for (int w = 1; w < T / 32; ++w) r = fmaxf(r, red[w]);
  __syncthreads();
  return r;
}
// block-wide sum in a fixed order: xor-butterfly inside each warp, then warps in index order
template <int T>
__device__ __forceinline__ float block_sum_fixed(float v, float* red) {
  v = warp_sum_xor(v);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (lane == 0) red[warp] = v;
  __syncthreads();
  float r = red[0];
#pragma unroll
  for (int w = 1; w < T / 32; ++w) r = __fadd_rn(r, red[w]);
  __syncthreads();
  return r;
}

// H256 ConvRot rotation of one 256-channel group held by a warp (lane l owns channels 8l..8l+7):
// y = H256 x with H256 = (H4 (x) H4 (x) H4 (x) H4) / 16 and H4 the regular 4x4 Hadamard matrix (all ones except
// a -1 on the anti-diagonal). One radix-4 stage over the four values e0..e3 that differ in one base-4 digit of
// the channel index is, unscaled,
//     y_k = (e_k + e_(k^1)) + (e_(k^2) - e_(k^3))
// i.e. with a = e0+e1, b = e2+e3, c = e0-e1, d = e2-e3:  y0 = a+d, y1 = a-d, y2 = b+c, y3 = b-c.
// Four stages (digit 0 = fastest first), then one multiplication by 1/16. Digit 0 and the low bit of digit 1
// live in the thread, the rest in the lane number; written this way a cross-lane stage costs two shuffles per
// value (the partner of the pair, then the other pair's difference) and the half-in-thread stage one shuffle per
// pair. Every operation is a single rounded fp32 add, so the CPU oracle repeats it bit for bit.
// (reference: triton_fp8.py:70-112 regular_hadamard / _rot256)
__device__ __forceinline__ void rotate256(float* x, int lane) {
  // digit 0: channels j & 3 inside the thread
#pragma unroll
  for (int b = 0; b < 8; b += 4) {
    const float sa = __fadd_rn(x[b], x[b + 1]), sb = __fadd_rn(x[b + 2], x[b + 3]);
    const float dc = __fsub_rn(x[b], x[b + 1]), dd = __fsub_rn(x[b + 2], x[b + 3]);
    x[b] = __fadd_rn(sa, dd), x[b + 1] = __fsub_rn(sa, dd), x[b + 2] = __fadd_rn(sb, dc), x[b + 3] = __fsub_rn(sb, dc);
  }
  // digit 1 = (j >> 2) + 2 * (lane & 1): the pair (e_k, e_(k^1)) is (x[j], x[j+4]); the other pair sits in lane ^ 1
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const float t = __fadd_rn(x[j], x[j + 4]);
    const float v = __shfl_xor_sync(0xffffffffu, __fsub_rn(x[j], x[j + 4]), 1);
    x[j] = __fadd_rn(t, v);
    x[j + 4] = __fsub_rn(t, v);
  }
  // digit 2 = (lane >> 1) & 3, digit 3 = lane >> 3: one value per lane
#pragma unroll
  for (int stage = 0; stage < 2; ++stage) {
    const int shift = stage == 0 ? 1 : 3;
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const float own = x[j];
      const float p1 = __shfl_xor_sync(0xffffffffu, own, 1 << shift);                      // e_(k^1)
      const float v = __shfl_xor_sync(0xffffffffu, __fsub_rn(own, p1), 2 << shift);        // e_(k^2) - e_(k^3)
      x[j] = __fadd_rn(__fadd_rn(own, p1), v);
    }
  }
#pragma unroll
  for (int j = 0; j < 8; ++j) x[j] = __fmul_rn(x[j], 0.0625f);
}

// Issue the 128-bit loads of one row (CPT chunks per thread); nothing waits on them here.
template <int KIND, int T, int CPT>
__device__ __forceinline__ void load_row(const QuantParams& p, int64_t row, int tid, int nchunk, uint4* raw,
                                         uint4* raw2) {
#pragma unroll
  for (int i = 0; i < CPT; ++i) {
    const int c = tid + i * T;
    raw[i] = make_uint4(0, 0, 0, 0);
    if (KIND == KIND_SWIGLU) raw2[i] = make_uint4(0, 0, 0, 0);
    if (c < nchunk) {
      const __nv_bfloat16* src;
      if (KIND == KIND_HEADS) {
        const int col = c << 3;
        const int grp = col / p.gw;
        src = p.x + static_cast<int64_t>(grp) * p.ldx + row * p.gw + (col - grp * p.gw);
      } else {
        src = p.x + row * p.ldx + (static_cast<int64_t>(c) << 3);
      }
      raw[i] = ld_global_16(src);
      if (KIND == KIND_SWIGLU) raw2[i] = ld_global_16(src + p.K);
    }
  }
}

// One CTA of T threads works on rows blockIdx.x, blockIdx.x + gridDim.x, ...; the loads of the next row
// are issued before the current row is reduced and stored, so every CTA always has a row in flight.
// CTAs that an SM has to hold, where the compiler by itself takes a few registers more than that leaves (0: its own choice).
// Plain rows of 4,096 with seven (72 registers) or six (75): 36,436 rows 88.1 / 91.6 us, e4m3 97.1 / 100.6.
__host__ __device__ constexpr int quant_min_ctas(int kind, int threads, int cpt, int rot) {
  return kind == KIND_PLAIN && threads == 128 && cpt == 4 && !rot ? 7 : kind == KIND_SWIGLU && threads == 128 && cpt == 2 && rot ? 8 : 0;
}
template <int KIND, int OUT_FP8, int T, int CPT, int ROT>
__global__ void __launch_bounds__(T, quant_min_ctas(KIND, T, CPT, ROT)) quant_rows_kernel(const QuantParams p) {
  grid_dependency_begin();
  __shared__ float red[T / 32];
  const int tid = threadIdx.x;
  const int nchunk = static_cast<int>(p.K >> 3);
  uint4 raw[CPT];
  uint4 raw2[KIND == KIND_SWIGLU ? CPT : 1];
  int64_t row = blockIdx.x;
  if (row < p.M) load_row<KIND, T, CPT>(p, row, tid, nchunk, raw, raw2);
  for (; row < p.M; row += gridDim.x) {
  float v[CPT][8];
#pragma unroll
  for (int i = 0; i < CPT; ++i) unpack8(raw[i], v[i]);

  if (KIND == KIND_SWIGLU) {
#pragma unroll
    for (int i = 0; i < CPT; ++i) {
      float u[8];
      unpack8(raw2[i], u);
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const float g = v[i][j];
        const float sg = __fdiv_rn(1.f, __fadd_rn(1.f, expf(-g)));
        v[i][j] = __fmul_rn(__fmul_rn(g, sg), u[j]);
      }
    }
  }
  // the registers of `raw` are free again: start fetching the next row of this CTA
  if (row + gridDim.x < p.M) load_row<KIND, T, CPT>(p, row + gridDim.x, tid, nchunk, raw, raw2);

  if (KIND == KIND_NORMMOD) {
    // sum of squares in a fixed order (thread-sequential over its chunks, then the block tree)
    float ss = 0.f;
#pragma unroll
    for (int i = 0; i < CPT; ++i) {
#pragma unroll
      for (int j = 0; j < 8; ++j) ss = __fadd_rn(ss, __fmul_rn(v[i][j], v[i][j]));
    }
    ss = block_sum_fixed<T>(ss, red);
    const float rstd = __fdiv_rn(1.f, __fsqrt_rn(__fadd_rn(__fdiv_rn(ss, static_cast<float>(p.K)), p.eps)));
    const int64_t trow = static_cast<int64_t>(p.idx[row]) * p.ld_tab;
#pragma unroll
    for (int i = 0; i < CPT; ++i) {
      const int c = tid + i * T;
      if (c < nchunk) {
        const int col = c << 3;
        float wv[8];
        if (p.w) {
          unpack8(__ldg(reinterpret_cast<const uint4*>(p.w + col)), wv);
        }
        const float4 sc0 = *reinterpret_cast<const float4*>(p.scale + trow + col);
        const float4 sc1 = *reinterpret_cast<const float4*>(p.scale + trow + col + 4);
        const float4 sh0 = *reinterpret_cast<const float4*>(p.shift + trow + col);
        const float4 sh1 = *reinterpret_cast<const float4*>(p.shift + trow + col + 4);
        const float sc[8] = {sc0.x, sc0.y, sc0.z, sc0.w, sc1.x, sc1.y, sc1.z, sc1.w};
        const float sh[8] = {sh0.x, sh0.y, sh0.z, sh0.w, sh1.x, sh1.y, sh1.z, sh1.w};
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          float y = __fmul_rn(v[i][j], rstd);
          if (p.w) y = __fmul_rn(y, wv[j]);
          y = __fadd_rn(__fmul_rn(y, __fadd_rn(1.f, sc[j])), sh[j]);
          v[i][j] = y;
        }
      }
    }
  }

  if (ROT) {
    // chunk c = tid + i * T: the 32 lanes of a warp hold one whole 256-channel group per i
#pragma unroll
    for (int i = 0; i < CPT; ++i)
      if (tid - (tid & 31) + i * T < nchunk) rotate256(v[i], tid & 31);
  }

  // ---- abs-max and scale ----
  float am = 0.f;
#pragma unroll
  for (int i = 0; i < CPT; ++i) {
#pragma unroll
    for (int j = 0; j < 8; ++j) am = fmaxf(am, fabsf(v[i][j]));
  }
  am = p.tensor_amax ? *p.tensor_amax : block_max<T>(am, red);
  const float qmax = OUT_FP8 ? 448.f : 127.f;
  const float s = fmaxf(__fdiv_rn(am, qmax), 1e-12f);
  const float inv = __fdiv_rn(1.f, s);
  if (tid == 0) p.s[row] = s;

  // ---- quantize + store ----
  uint8_t* qrow = reinterpret_cast<uint8_t*>(p.q) + row * p.ldq;
#pragma unroll
  for (int i = 0; i < CPT; ++i) {
    const int c = tid + i * T;
    if (c < nchunk) {
      const uint2 o = OUT_FP8 ? quant8_e4m3(v[i], s, inv) : quant8_i8(v[i], s, inv);
      *reinterpret_cast<uint2*>(qrow + (static_cast<int64_t>(c) << 3)) = o;
    }
  }
  }  // rows of this CTA
}

// RMSNorm of bf16 rows to bf16, out = bf16((x * r) * w) with r = rsqrt(mean(x^2) + eps): one read, one write. The loop of
// quant_rows_kernel: a row in registers, the next row's loads in flight. HBM-bound, 4 bytes per element; as a chain of
// elementwise kernels (fp32 copy, square, mean, rsqrt, two products, copy back) the same rows cost about 40 bytes per
// element (2 + 4, 4 + 4, 4, 4 + 4, 4 + 4, 4 + 2), in part out of L2: 80 us for 1,008 x 4,096, 5.9 us here; 6,196 x 4,096 take 16 us (6.3 TB/s).
template <int T, int CPT>
__global__ void __launch_bounds__(T, T == 128 ? 0 : 1024 / T) rms_norm_rows_kernel(const __nv_bfloat16* x, int64_t ldx,
                                                          const __nv_bfloat16* __restrict__ w, float eps, int64_t M, int K,
                                                          __nv_bfloat16* out, int64_t ldo) {
  grid_dependency_begin();
  __shared__ float red[T / 32];
  const int tid = threadIdx.x, nchunk = K >> 3;
  QuantParams p{};
  p.x = x; p.ldx = ldx; p.M = M; p.K = K;
  uint4 raw[CPT];
  int64_t row = blockIdx.x;
  if (row < M) load_row<KIND_PLAIN, T, CPT>(p, row, tid, nchunk, raw, nullptr);
  for (; row < M; row += gridDim.x) {
    float v[CPT][8];
    float ss = 0.f;
#pragma unroll
    for (int i = 0; i < CPT; ++i) {
      unpack8(raw[i], v[i]);
#pragma unroll
      for (int j = 0; j < 8; ++j) ss = fmaf(v[i][j], v[i][j], ss);
    }
    if (row + gridDim.x < M) load_row<KIND_PLAIN, T, CPT>(p, row + gridDim.x, tid, nchunk, raw, nullptr);
    ss = block_sum_fixed<T>(ss, red);
    const float r = rsqrtf(__fadd_rn(__fdiv_rn(ss, static_cast<float>(K)), eps));
#pragma unroll
    for (int i = 0; i < CPT; ++i) {
      const int c = tid + i * T;
      if (c < nchunk) {
        float wv[8];
        unpack8(__ldg(reinterpret_cast<const uint4*>(w + (c << 3))), wv);
        uint32_t o[4];
#pragma unroll
        for (int j = 0; j < 4; ++j)
          o[j] = pack_bf16x2(__fmul_rn(__fmul_rn(v[i][2 * j], r), wv[2 * j]), __fmul_rn(__fmul_rn(v[i][2 * j + 1], r), wv[2 * j + 1]));
        *reinterpret_cast<uint4*>(out + row * ldo + (static_cast<int64_t>(c) << 3)) = make_uint4(o[0], o[1], o[2], o[3]);
      }
    }
  }
}

// Second int8 pass on the quantization residual of selected rows (the text encoder's outlier rows):
//   r = rotate(x[rows[i]]) - q1[rows[i]] * s1[rows[i]]   (x fp32, so the residual also carries the bf16 rounding
//   of the first pass's input), then the plain int8 row quantizer on r. One CTA of K/8 threads per selected row.
// (reference: custom_nodes/rapid_h3/te_quant.py:96-105)
template <int T>
__global__ void __launch_bounds__(T) rot_residual_quant_kernel(const float* __restrict__ x, int64_t ldx,
                                                               const int8_t* __restrict__ q1, int64_t ldq1,
                                                               const float* __restrict__ s1,
                                                               const int32_t* __restrict__ rows, int64_t n, int K,
                                                               int8_t* __restrict__ q2, float* __restrict__ s2) {
  __shared__ float red[T / 32];
  const int tid = threadIdx.x;
  const int col = tid << 3;
  const bool active = col < K;
  for (int64_t i = blockIdx.x; i < n; i += gridDim.x) {
    const int64_t r = rows[i];
    float v[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) v[j] = 0.f;
    if (active) {
      const float4 a = __ldg(reinterpret_cast<const float4*>(x + r * ldx + col));
      const float4 b = __ldg(reinterpret_cast<const float4*>(x + r * ldx + col + 4));
      v[0] = a.x, v[1] = a.y, v[2] = a.z, v[3] = a.w, v[4] = b.x, v[5] = b.y, v[6] = b.z, v[7] = b.w;
    }
    if (tid - (tid & 31) < (K >> 3)) rotate256(v, tid & 31);
    if (active) {
      const uint2 c = __ldg(reinterpret_cast<const uint2*>(q1 + r * ldq1 + col));
      const float sc = s1[r];
      const int8_t* cb = reinterpret_cast<const int8_t*>(&c);
#pragma unroll
      for (int j = 0; j < 8; ++j) v[j] = __fsub_rn(v[j], __fmul_rn(static_cast<float>(cb[j]), sc));
    }
    float am = 0.f;
#pragma unroll
    for (int j = 0; j < 8; ++j) am = fmaxf(am, fabsf(v[j]));
    am = block_max<T>(am, red);
    const float s = fmaxf(__fdiv_rn(am, 127.f), 1e-12f);
    const float inv = __fdiv_rn(1.f, s);
    if (tid == 0) s2[i] = s;
    if (active) *reinterpret_cast<uint2*>(q2 + i * K + col) = quant8_i8(v, s, inv);
  }
}

// Everything the text encoder's linear does to its input before the first product, one CTA of K/8 threads per row, the row
// read once and held in registers:
//   q1, s1   the int8 row quantizer on rotate(bf16(x)) (the codes of rot_quant_rows on the bf16 copy of x)
//   outlier  127 s1 / max(rms(x), 1e-12) > ratio: H256 is orthonormal, so the rotated row has x's rms, and its abs-max is
//            127 s1 by construction of the scale. The squares are summed by fused multiply-adds in a fixed order; a sum in
//            another order (torch's mean, in the separate steps) can differ in its last places, so a row whose quotient is
//            within about 1e-6 of the ratio can fall on the other side there
//   an outlier row takes the next free slot i of the second pass: rows[i] = row, and q2[i], s2[i] are the int8 codes of
//   rotate(x) - q1 s1 (the arithmetic of rot_residual_quant_kernel). Slots are handed out by one atomic per outlier row, in
//   any order: a slot's content does not depend on its number. `count` is what the second product reads its row number
//   from, so the host never waits for it.
// Bound by HBM in principle (4 bytes in, 1 out per value), by launches in practice: as separate steps (bf16 copy,
// quantizer, square, mean, sqrt, clamp, compare, three kernels and a host round trip of the index list, residual
// quantizer) this took 14 launches and 55 us of device time for 512 x 4,096.
template <int T>
__global__ void __launch_bounds__(T) te_quant_kernel(const float* __restrict__ x, int64_t ldx, int64_t M, int K, float ratio,
                                                     int8_t* __restrict__ q1, float* __restrict__ s1,
                                                     uint8_t* __restrict__ flags, int* __restrict__ count,
                                                     int32_t* __restrict__ rows, int8_t* __restrict__ q2,
                                                     float* __restrict__ s2, unsigned long long* __restrict__ total,
                                                     unsigned long long* __restrict__ seen) {
  __shared__ float red[T / 32];
  __shared__ int slot_s;
  const int tid = threadIdx.x;
  if (seen && blockIdx.x == 0 && tid == 0) atomicAdd(seen, static_cast<unsigned long long>(M));
  const int col = tid << 3;
  const bool active = col < K;
  const bool whole = tid - (tid & 31) < (K >> 3);  // K is a multiple of 256: uniform over a warp
  for (int64_t row = blockIdx.x; row < M; row += gridDim.x) {
    float v[8], y[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) v[j] = 0.f;
    if (active) {
      const float4 a = __ldg(reinterpret_cast<const float4*>(x + row * ldx + col));
      const float4 b = __ldg(reinterpret_cast<const float4*>(x + row * ldx + col + 4));
      v[0] = a.x, v[1] = a.y, v[2] = a.z, v[3] = a.w, v[4] = b.x, v[5] = b.y, v[6] = b.z, v[7] = b.w;
    }
    float ss = 0.f;
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      ss = fmaf(v[j], v[j], ss);
      y[j] = bf16_round(v[j]);
    }
    if (whole) rotate256(y, tid & 31);
    float am = 0.f;
#pragma unroll
    for (int j = 0; j < 8; ++j) am = fmaxf(am, fabsf(y[j]));
    am = block_max<T>(am, red);
    const float s = fmaxf(__fdiv_rn(am, 127.f), 1e-12f);
    const uint2 code = quant8_i8(y, s, __fdiv_rn(1.f, s));
    if (active) *reinterpret_cast<uint2*>(q1 + row * K + col) = code;
    ss = block_sum_fixed<T>(ss, red);
    float rms = __fsqrt_rn(__fdiv_rn(ss, static_cast<float>(K)));
    if (rms < 1e-12f) rms = 1e-12f;                                   // a NaN stays: no comparison with it is true
    const bool outlier = __fdiv_rn(__fmul_rn(127.f, s), rms) > ratio;  // the same value in every thread
    if (tid == 0) {
      s1[row] = s;
      flags[row] = outlier;
    }
    if (!outlier) continue;
    if (tid == 0) {
      slot_s = atomicAdd(count, 1);
      rows[slot_s] = static_cast<int32_t>(row);
      if (total) atomicAdd(total, 1ull);
    }
    if (whole) rotate256(v, tid & 31);
    am = 0.f;
    if (active) {
      const int8_t* cb = reinterpret_cast<const int8_t*>(&code);
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        v[j] = __fsub_rn(v[j], __fmul_rn(static_cast<float>(cb[j]), s));
        am = fmaxf(am, fabsf(v[j]));
      }
    }
    am = block_max<T>(am, red);  // its barriers also publish the slot
    const int64_t slot = slot_s;
    const float sr = fmaxf(__fdiv_rn(am, 127.f), 1e-12f);
    if (tid == 0) s2[slot] = sr;
    if (active) *reinterpret_cast<uint2*>(q2 + slot * K + col) = quant8_i8(v, sr, __fdiv_rn(1.f, sr));
    __syncthreads();  // the slot has been read by all before the next outlier row of this CTA replaces it
  }
}

// max |x| over a whole [M, K] bf16 tensor into *out (which the caller zeroed): |x| >= 0, so the float order is the
// order of the bit patterns and one atomicMax on the bits per CTA finishes the reduction, in any order.
__global__ void __launch_bounds__(256) tensor_absmax_kernel(const __nv_bfloat16* __restrict__ x, int64_t ldx, int64_t M,
                                                            int64_t K, float* __restrict__ out) {
  __shared__ float red[8];
  const int64_t nchunk = K >> 3, total = M * nchunk;
  float am = 0.f;
  for (int64_t i = static_cast<int64_t>(blockIdx.x) * 256 + threadIdx.x; i < total; i += static_cast<int64_t>(gridDim.x) * 256) {
    const int64_t row = i / nchunk, c = i - row * nchunk;
    float v[8];
    unpack8(__ldg(reinterpret_cast<const uint4*>(x + row * ldx + (c << 3))), v);
#pragma unroll
    for (int j = 0; j < 8; ++j) am = fmaxf(am, fabsf(v[j]));
  }
  am = block_max<256>(am, red);
  if (threadIdx.x == 0) atomicMax(reinterpret_cast<unsigned int*>(out), __float_as_uint(am));
}

// Row kernels start under the kernel before them (launch_kernel) while they are small. us chained / not on a stream, a linear with
// its quantizer: 37 x 4,096 rows 11.1 / 12.4, 512 15.5 / 16.5, 2,016 34.4 / 35.2, 5,003 80.4 / 79.4; 512 x 16,384 42.2 / 42.8, 3,024 172 / 170; one
// block of 2,024 tokens 746 / 753. From graphs: 128 x 4,096 11.2 / 11.5, 148 11.3 / 10.8, 400 13.5 / 12.8, 400 x 1,024 6.5 / 7.0.
bool chain_rows(int64_t M, int64_t K, cudaStream_t stream) { return M * K <= (in_capture(stream) ? 1ll << 19 : 1ll << 23); }

template <int KIND, int OUT_FP8, int ROT = 0>
int launch_quant(const QuantParams& p, cudaStream_t stream) {
  const int64_t nchunk = p.K >> 3;
  if (p.M == 0) return 0;
  cudaError_t launched = cudaSuccess;
  // as many CTAs as are resident at once (a multiple of the SM count), each looping over its rows
#define RH3_Q(T_, CPT_)                                                                                \
  do {                                                                                                 \
    auto kern = quant_rows_kernel<KIND, OUT_FP8, T_, CPT_, ROT>;                                       \
    int occ = 1;                                                                                       \
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, kern, T_, 0) != cudaSuccess || occ < 1) occ = 1; \
    const int64_t resident = static_cast<int64_t>(device_sm_count()) * occ;                           \
    launched = launch_kernel(chain_rows(p.M, p.K, stream), kern, dim3(static_cast<unsigned>(p.M < resident ? p.M : resident)), T_, 0, stream, 1, p); \
  } while (0)
  if (nchunk <= 128) RH3_Q(128, 1);
  else if (nchunk <= 256) RH3_Q(128, 2);
  else if (nchunk <= 512) RH3_Q(128, 4);
  else if (nchunk <= 1024) RH3_Q(128, 8);
  else if (nchunk <= 2048) RH3_Q(256, 8);
  else if (nchunk <= 4096) RH3_Q(512, 8);
  else if (nchunk <= 8192) RH3_Q(1024, 8);
  else return set_error(RH3_ARG_ERROR, "quant_rows: K=%lld is larger than 65536", (long long)p.K);
#undef RH3_Q
  return check_cuda(launched, "quant_rows launch");
}

int check_common(const void* x, int64_t ldx, int64_t M, int64_t K, const void* q, int64_t ldq, const float* s) {
  RH3_CHECK_ARG(M >= 0 && K > 0, "quant_rows: bad shape M=%lld K=%lld", (long long)M, (long long)K);
  RH3_CHECK_ARG(M < (1ll << 31), "quant_rows: M too large");
  RH3_CHECK_ARG(K % 8 == 0, "quant_rows: K=%lld must be a multiple of 8", (long long)K);
  RH3_CHECK_ARG(M == 0 || (x && q && s), "quant_rows: null pointer");
  RH3_CHECK_ARG(ldx % 8 == 0 && (reinterpret_cast<uintptr_t>(x) & 15) == 0,
                "quant_rows: x must be 16-byte aligned with a row stride that is a multiple of 8 elements");
  RH3_CHECK_ARG(ldq % 8 == 0 && (reinterpret_cast<uintptr_t>(q) & 7) == 0,
                "quant_rows: q must be 8-byte aligned with a row stride that is a multiple of 8");
  return 0;
}

}  // namespace
}  // namespace rh3

using namespace rh3;

extern "C" int rh3_quant_rows_i8(const void* x, int64_t ldx, int64_t M, int64_t K, void* q, int64_t ldq, float* s,
                                 cudaStream_t stream) {
  if (int e = check_common(x, ldx, M, K, q, ldq, s)) return e;
  RH3_CHECK_ARG(ldx >= K && ldq >= K, "quant_rows_i8: row strides smaller than K");
  QuantParams p{};
  p.x = static_cast<const __nv_bfloat16*>(x); p.ldx = ldx; p.M = M; p.K = K; p.q = q; p.ldq = ldq; p.s = s;
  return launch_quant<KIND_PLAIN, 0>(p, stream);
}

extern "C" int rh3_quant_rows_fp8(const void* x, int64_t ldx, int64_t M, int64_t K, void* q, int64_t ldq, float* s,
                                  cudaStream_t stream) {
  if (int e = check_common(x, ldx, M, K, q, ldq, s)) return e;
  RH3_CHECK_ARG(ldx >= K && ldq >= K, "quant_rows_fp8: row strides smaller than K");
  QuantParams p{};
  p.x = static_cast<const __nv_bfloat16*>(x); p.ldx = ldx; p.M = M; p.K = K; p.q = q; p.ldq = ldq; p.s = s;
  return launch_quant<KIND_PLAIN, 1>(p, stream);
}

extern "C" int rh3_quant_tensor_fp8(const void* x, int64_t ldx, int64_t M, int64_t K, void* q, int64_t ldq, float* s,
                                    float* amax, cudaStream_t stream) {
  if (int e = check_common(x, ldx, M, K, q, ldq, s)) return e;
  RH3_CHECK_ARG(ldx >= K && ldq >= K, "quant_tensor_fp8: row strides smaller than K");
  RH3_CHECK_ARG(amax != nullptr, "quant_tensor_fp8: null abs-max word");
  if (int e = check_cuda(cudaMemsetAsync(amax, 0, sizeof(float), stream), "quant_tensor_fp8 memset")) return e;
  if (M == 0) return 0;
  const int64_t chunks = M * (K >> 3);
  const int64_t want = (chunks + 255) / 256, cap = static_cast<int64_t>(device_sm_count()) * 8;
  tensor_absmax_kernel<<<static_cast<unsigned>(want < cap ? want : cap), 256, 0, stream>>>(
      static_cast<const __nv_bfloat16*>(x), ldx, M, K, amax);
  if (int e = check_cuda(cudaGetLastError(), "tensor_absmax launch")) return e;
  QuantParams p{};
  p.x = static_cast<const __nv_bfloat16*>(x); p.ldx = ldx; p.M = M; p.K = K; p.q = q; p.ldq = ldq; p.s = s;
  p.tensor_amax = amax;
  return launch_quant<KIND_PLAIN, 1>(p, stream);
}

extern "C" int rh3_swiglu_quant_rows_i8(const void* x, int64_t ldx, int64_t M, int64_t F, void* q, int64_t ldq,
                                        float* s, cudaStream_t stream) {
  if (int e = check_common(x, ldx, M, F, q, ldq, s)) return e;
  RH3_CHECK_ARG(ldx >= 2 * F && ldq >= F, "swiglu_quant_rows_i8: row strides too small");
  QuantParams p{};
  p.x = static_cast<const __nv_bfloat16*>(x); p.ldx = ldx; p.M = M; p.K = F; p.q = q; p.ldq = ldq; p.s = s;
  return launch_quant<KIND_SWIGLU, 0>(p, stream);
}

extern "C" int rh3_quant_groups_i8(const void* o, int64_t stride_g, int64_t G, int64_t gw, int64_t M, void* q,
                                   int64_t ldq, float* s, cudaStream_t stream) {
  RH3_CHECK_ARG(G > 0 && gw > 0 && gw % 8 == 0 && gw < (1ll << 30), "quant_groups_i8: G must be positive, gw a multiple of 8");
  if (int e = check_common(o, stride_g, M, G * gw, q, ldq, s)) return e;
  RH3_CHECK_ARG(stride_g >= M * gw && ldq >= G * gw, "quant_groups_i8: strides too small");
  QuantParams p{};
  p.x = static_cast<const __nv_bfloat16*>(o); p.ldx = stride_g; p.M = M; p.K = G * gw; p.q = q; p.ldq = ldq; p.s = s;
  p.gw = static_cast<int>(gw);
  return launch_quant<KIND_HEADS, 0>(p, stream);
}

extern "C" int rh3_quant_heads_i8(const void* o, int64_t stride_h, int64_t H, int64_t M, void* q, int64_t ldq,
                                  float* s, cudaStream_t stream) {
  return rh3_quant_groups_i8(o, stride_h, H, 128, M, q, ldq, s, stream);
}

extern "C" int rh3_norm_mod_quant_rows_i8(const void* x, int64_t ldx, const void* w, float eps, const int32_t* idx,
                                          const float* shift, const float* scale, int64_t ld_tab, int64_t M,
                                          int64_t K, void* q, int64_t ldq, float* s, cudaStream_t stream) {
  if (int e = check_common(x, ldx, M, K, q, ldq, s)) return e;
  RH3_CHECK_ARG(ldx >= K && ldq >= K, "norm_mod_quant_rows_i8: row strides smaller than K");
  RH3_CHECK_ARG(M == 0 || (idx && shift && scale), "norm_mod_quant_rows_i8: null modulation pointer");
  RH3_CHECK_ARG(ld_tab % 4 == 0 && (reinterpret_cast<uintptr_t>(shift) & 15) == 0 &&
                    (reinterpret_cast<uintptr_t>(scale) & 15) == 0,
                "norm_mod_quant_rows_i8: shift/scale must be 16-byte aligned, row stride a multiple of 4");
  RH3_CHECK_ARG(!w || (reinterpret_cast<uintptr_t>(w) & 15) == 0, "norm_mod_quant_rows_i8: w must be 16-byte aligned");
  QuantParams p{};
  p.x = static_cast<const __nv_bfloat16*>(x); p.ldx = ldx; p.M = M; p.K = K; p.q = q; p.ldq = ldq; p.s = s;
  p.w = static_cast<const __nv_bfloat16*>(w); p.eps = eps; p.idx = idx; p.shift = shift; p.scale = scale;
  p.ld_tab = ld_tab;
  return launch_quant<KIND_NORMMOD, 0>(p, stream);
}

// ---- the same quantizers with the H256 ConvRot rotation applied before the abs-max (K % 256 == 0) ----
#define RH3_ROT_CHECK(K, name) RH3_CHECK_ARG((K) % 256 == 0, name ": the rotated width must be a multiple of 256")

extern "C" int rh3_rot_quant_rows_i8(const void* x, int64_t ldx, int64_t M, int64_t K, void* q, int64_t ldq, float* s,
                                     cudaStream_t stream) {
  if (int e = check_common(x, ldx, M, K, q, ldq, s)) return e;
  RH3_ROT_CHECK(K, "rot_quant_rows_i8");
  RH3_CHECK_ARG(ldx >= K && ldq >= K, "rot_quant_rows_i8: row strides smaller than K");
  QuantParams p{};
  p.x = static_cast<const __nv_bfloat16*>(x); p.ldx = ldx; p.M = M; p.K = K; p.q = q; p.ldq = ldq; p.s = s;
  return launch_quant<KIND_PLAIN, 0, 1>(p, stream);
}

extern "C" int rh3_swiglu_rot_quant_rows_i8(const void* x, int64_t ldx, int64_t M, int64_t F, void* q, int64_t ldq,
                                            float* s, cudaStream_t stream) {
  if (int e = check_common(x, ldx, M, F, q, ldq, s)) return e;
  RH3_ROT_CHECK(F, "swiglu_rot_quant_rows_i8");
  RH3_CHECK_ARG(ldx >= 2 * F && ldq >= F, "swiglu_rot_quant_rows_i8: row strides too small");
  QuantParams p{};
  p.x = static_cast<const __nv_bfloat16*>(x); p.ldx = ldx; p.M = M; p.K = F; p.q = q; p.ldq = ldq; p.s = s;
  return launch_quant<KIND_SWIGLU, 0, 1>(p, stream);
}

extern "C" int rh3_rot_quant_groups_i8(const void* o, int64_t stride_g, int64_t G, int64_t gw, int64_t M, void* q,
                                       int64_t ldq, float* s, cudaStream_t stream) {
  RH3_CHECK_ARG(G > 0 && gw > 0 && gw % 8 == 0 && gw < (1ll << 30), "rot_quant_groups_i8: bad group shape");
  if (int e = check_common(o, stride_g, M, G * gw, q, ldq, s)) return e;
  RH3_ROT_CHECK(G * gw, "rot_quant_groups_i8");
  RH3_CHECK_ARG(stride_g >= M * gw && ldq >= G * gw, "rot_quant_groups_i8: strides too small");
  QuantParams p{};
  p.x = static_cast<const __nv_bfloat16*>(o); p.ldx = stride_g; p.M = M; p.K = G * gw; p.q = q; p.ldq = ldq; p.s = s;
  p.gw = static_cast<int>(gw);
  return launch_quant<KIND_HEADS, 0, 1>(p, stream);
}

extern "C" int rh3_norm_mod_rot_quant_rows_i8(const void* x, int64_t ldx, const void* w, float eps, const int32_t* idx,
                                              const float* shift, const float* scale, int64_t ld_tab, int64_t M,
                                              int64_t K, void* q, int64_t ldq, float* s, cudaStream_t stream) {
  if (int e = check_common(x, ldx, M, K, q, ldq, s)) return e;
  RH3_ROT_CHECK(K, "norm_mod_rot_quant_rows_i8");
  RH3_CHECK_ARG(ldx >= K && ldq >= K, "norm_mod_rot_quant_rows_i8: row strides smaller than K");
  RH3_CHECK_ARG(M == 0 || (idx && shift && scale), "norm_mod_rot_quant_rows_i8: null modulation pointer");
  RH3_CHECK_ARG(ld_tab % 4 == 0 && (reinterpret_cast<uintptr_t>(shift) & 15) == 0 &&
                    (reinterpret_cast<uintptr_t>(scale) & 15) == 0,
                "norm_mod_rot_quant_rows_i8: shift/scale must be 16-byte aligned, row stride a multiple of 4");
  RH3_CHECK_ARG(!w || (reinterpret_cast<uintptr_t>(w) & 15) == 0, "norm_mod_rot_quant_rows_i8: w must be 16-byte aligned");
  QuantParams p{};
  p.x = static_cast<const __nv_bfloat16*>(x); p.ldx = ldx; p.M = M; p.K = K; p.q = q; p.ldq = ldq; p.s = s;
  p.w = static_cast<const __nv_bfloat16*>(w); p.eps = eps; p.idx = idx; p.shift = shift; p.scale = scale;
  p.ld_tab = ld_tab;
  return launch_quant<KIND_NORMMOD, 0, 1>(p, stream);
}

// ---- residual pass of the text encoder's int8_rot linears (no rotation-free form exists) ----
extern "C" int rh3_rot_residual_quant_rows_i8(const float* x, int64_t ldx, const void* q1, int64_t ldq1, const float* s1,
                                              const int32_t* rows, int64_t n, int64_t K, void* q2, float* s2,
                                              cudaStream_t stream) {
  RH3_CHECK_ARG(n >= 0 && K > 0 && K % 256 == 0 && K <= 8192, "rot_residual_quant: K=%lld must be a multiple of 256, <= 8192",
                (long long)K);
  RH3_CHECK_ARG(ldx >= K && ldx % 4 == 0 && ldq1 >= K && ldq1 % 8 == 0, "rot_residual_quant: bad row strides");
  if (n == 0) return 0;
  RH3_CHECK_ARG(x && q1 && s1 && rows && q2 && s2, "rot_residual_quant: null pointer");
  RH3_CHECK_ARG((reinterpret_cast<uintptr_t>(x) & 15) == 0 && (reinterpret_cast<uintptr_t>(q1) & 7) == 0 &&
                    (reinterpret_cast<uintptr_t>(q2) & 7) == 0,
                "rot_residual_quant: x must be 16-byte aligned, q1 and q2 8-byte aligned");
  const int64_t threads = K / 8;
  const unsigned grid = static_cast<unsigned>(n < 4 * device_sm_count() ? n : 4 * device_sm_count());
#define RH3_RR(T_)                                                                                       \
  rot_residual_quant_kernel<T_><<<grid, T_, 0, stream>>>(x, ldx, static_cast<const int8_t*>(q1), ldq1, s1, rows, n, \
                                                         (int)K, static_cast<int8_t*>(q2), s2)
  if (threads <= 128) RH3_RR(128);
  else if (threads <= 256) RH3_RR(256);
  else if (threads <= 512) RH3_RR(512);
  else RH3_RR(1024);
#undef RH3_RR
  return check_cuda(cudaGetLastError(), "rot_residual_quant launch");
}

extern "C" int rh3_rms_norm_rows(const void* x, int64_t ldx, const void* w, float eps, int64_t M, int64_t K, void* out,
                                 int64_t ldo, cudaStream_t stream) {
  if (int e = check_common(x, ldx, M, K, out, ldo, &eps)) return e;
  RH3_CHECK_ARG(ldx >= K && ldo >= K && (reinterpret_cast<uintptr_t>(out) & 15) == 0 && (reinterpret_cast<uintptr_t>(w) & 15) == 0,
                "rms_norm_rows: row strides smaller than K, or out / w not 16-byte aligned");
  RH3_CHECK_ARG(M == 0 || w, "rms_norm_rows: null weight");
  RH3_CHECK_ARG(K <= 16384, "rms_norm_rows: K=%lld is larger than 16384", (long long)K);
  if (M == 0) return 0;
  const int64_t nchunk = K >> 3;
  cudaError_t launched = cudaSuccess;
#define RH3_RN(T_, CPT_)                                                                                          \
  do {                                                                                                            \
    auto kern = rms_norm_rows_kernel<T_, CPT_>;                                                                   \
    const int64_t resident = static_cast<int64_t>(device_sm_count()) * (2048 / T_ < 8 ? 2048 / T_ : 8);           \
    launched = launch_kernel(chain_rows(M, K, stream), kern, dim3(static_cast<unsigned>(M < resident ? M : resident)), T_, 0, stream, 1, \
                             static_cast<const __nv_bfloat16*>(x), ldx, static_cast<const __nv_bfloat16*>(w),     \
                             eps, M, (int)K, static_cast<__nv_bfloat16*>(out), ldo);                              \
  } while (0)
  if (nchunk <= 128) RH3_RN(128, 1);
  else if (nchunk <= 256) RH3_RN(128, 2);
  else if (nchunk <= 512) RH3_RN(128, 4);
  else if (nchunk <= 1024) RH3_RN(256, 4);
  else RH3_RN(512, 4);
#undef RH3_RN
  return check_cuda(launched, "rms_norm_rows launch");
}

extern "C" int rh3_te_quant_counted(const float* x, int64_t ldx, int64_t M, int64_t K, float ratio, void* q1, float* s1,
                                    void* flags, int32_t* count, int32_t* rows, void* q2, float* s2, void* total,
                                    void* seen, cudaStream_t stream) {
  RH3_CHECK_ARG(M >= 0 && M < (1ll << 31) && K > 0 && K % 256 == 0 && K <= 8192,
                "te_quant: K=%lld must be a multiple of 256, <= 8192", (long long)K);
  RH3_CHECK_ARG(ldx >= K && ldx % 4 == 0, "te_quant: bad row stride");
  if (M == 0) return count ? check_cuda(cudaMemsetAsync(count, 0, sizeof(int32_t), stream), "te_quant count") : 0;
  RH3_CHECK_ARG(x && q1 && s1 && flags && count && rows && q2 && s2, "te_quant: null pointer");
  RH3_CHECK_ARG((reinterpret_cast<uintptr_t>(x) & 15) == 0 && (reinterpret_cast<uintptr_t>(q1) & 7) == 0 &&
                    (reinterpret_cast<uintptr_t>(q2) & 7) == 0 && (reinterpret_cast<uintptr_t>(total) & 7) == 0 &&
                    (reinterpret_cast<uintptr_t>(seen) & 7) == 0,
                "te_quant: x must be 16-byte aligned, q1, q2, total and seen 8-byte aligned");
  if (int e = check_cuda(cudaMemsetAsync(count, 0, sizeof(int32_t), stream), "te_quant count")) return e;
  const int64_t threads = K / 8;
  const unsigned grid = static_cast<unsigned>(M < 8 * device_sm_count() ? M : 8 * device_sm_count());
#define RH3_TE(T_)                                                                                                       \
  te_quant_kernel<T_><<<grid, T_, 0, stream>>>(x, ldx, M, (int)K, ratio, static_cast<int8_t*>(q1), s1,                   \
                                               static_cast<uint8_t*>(flags), count, rows, static_cast<int8_t*>(q2), s2, \
                                               static_cast<unsigned long long*>(total),                                 \
                                               static_cast<unsigned long long*>(seen))
  if (threads <= 128) RH3_TE(128);
  else if (threads <= 256) RH3_TE(256);
  else if (threads <= 512) RH3_TE(512);
  else RH3_TE(1024);
#undef RH3_TE
  return check_cuda(cudaGetLastError(), "te_quant launch");
}

extern "C" int rh3_te_quant(const float* x, int64_t ldx, int64_t M, int64_t K, float ratio, void* q1, float* s1, void* flags,
                            int32_t* count, int32_t* rows, void* q2, float* s2, void* total, cudaStream_t stream) {
  return rh3_te_quant_counted(x, ldx, M, K, ratio, q1, s1, flags, count, rows, q2, s2, total, nullptr, stream);
}

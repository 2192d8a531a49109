// Quantizer of the VAE transformer decoder's attention output (fp16 activations).
//
//   o [B, H, S, D] fp16 head-major (D = 64)  ->  q int8 [B*S, H*D], scale fp32 [B*S]
//
// Row (b, s) of the output gathers column c = head * D + d from o[b, head, s, d] (no transposed copy),
// replaces NaN by 0 and +-inf by +-65504 (torch.nan_to_num for fp16), rotates every group of 256 columns
// by the regular-Hadamard matrix H256 and quantizes the row to int8 with one scale:
//   scale = max(min(amax, 65504) * (1/127), 1e-30)
//   q     = clamp(rint(fp16(fp16(y) / fp16(scale))), -128, 127)     (value, scale and quotient pass through fp16)
// The rotation is written as four radix-4 stages with strides 1, 4, 16, 64 and, per stage,
//   y0 = 0.5 * (((x0 + x1) + x2) - x3)      y1 = 0.5 * (((x0 + x1) - x2) + x3)
//   y2 = 0.5 * (((x0 - x1) + x2) + x3)      y3 = 0.5 * (((-x0 + x1) + x2) + x3)
// evaluated left to right in fp32: the order of the reference's vae_out_quant
// (custom_nodes/rapid_h3/csrc/vae_ops.cu:63-142, which restates comfy-kitchen's ConvRot quantizer; the
// reference builds with approximate division, this kernel divides exactly, so the last code bit can differ
// from that binary: parity is defined by the CPU oracle, oracle/vae_ops.py).
//
// One CTA per row at a time (persistent), K / 16 threads, the next row's loads in flight while a row is worked on. A
// half-warp owns one 256-column group: thread t of it holds columns 16t .. 16t+15, i.e. the two low base-4 digits, so
// stages 1 and 4 run inside the thread; one 16 x 16 exchange through shared memory (4-float rows padded to 20: no bank
// conflicts, only the half-warp's own patch, so __syncwarp orders it) gives the thread columns t, t + 16, ... for
// stages 16 and 64, and the codes go back through the same patch as bytes for 16-byte stores. No value crosses lanes by
// shuffle: the form with eight columns per thread and shuffles for three of the four stages (9 shuffles per value, and
// 1,024 threads per 8,192-wide row, one CTA per SM) took 131 us for 3,594 x 8,192 and 35 us for 3,594 x 2,048 with the
// RMSNorm prologue, this one 40 and 16.
// Algorithmic traffic: 3 bytes per element (2 in, 1 out), 13.5 and 3.4 us at those sizes and the measured copy rate; what
// is left above it is instruction issue (about 25 per value).
#include "common.cuh"
#include "rapidh3_b200.h"

namespace rh3 {
namespace {

__device__ __forceinline__ float nan_to_num_h(__half h) {
  if (__hisnan(h)) return 0.f;
  if (__hisinf(h)) return __hgt(h, __float2half(0.f)) ? 65504.f : -65504.f;
  return __half2float(h);
}

// One radix-4 stage without its factor 1/2 (an exact scaling, applied once as 1/16 after the four stages):
// e0' = ((e0 + e1) + e2) - e3, e1' = ((e0 + e1) - e2) + e3, e2' = ((e0 - e1) + e2) + e3, e3' = ((e1 - e0) + e2) + e3
__device__ __forceinline__ void fht_quad(float& e0, float& e1, float& e2, float& e3) {
  const float s = __fadd_rn(e0, e1), d = __fsub_rn(e0, e1);  // e1 - e0 == -d exactly
  e0 = __fsub_rn(__fadd_rn(s, e2), e3);
  e1 = __fadd_rn(__fsub_rn(s, e2), e3);
  const float t2 = __fadd_rn(__fadd_rn(d, e2), e3), t3 = __fadd_rn(__fsub_rn(e2, d), e3);
  e2 = t2;
  e3 = t3;
}
// the two stages whose digits the thread's 16 values span
__device__ __forceinline__ void fht16(float* x) {
#pragma unroll
  for (int b = 0; b < 16; b += 4) fht_quad(x[b], x[b + 1], x[b + 2], x[b + 3]);
#pragma unroll
  for (int j = 0; j < 4; ++j) fht_quad(x[j], x[j + 4], x[j + 8], x[j + 12]);
}

enum { ACT_NONE = 0, ACT_RMS_NORM = 1, ACT_SWIGLU = 2 };

struct OutQuantParams {
  int act;                // prologue applied to the loaded row before the rotation
  const __half* act_w;    // ACT_RMS_NORM: norm weight [K] or null
  float eps;              // ACT_RMS_NORM
  int64_t up_offset;      // ACT_SWIGLU: the "up" half of a row starts this many elements after the gate half
  const __half* o;
  int8_t* q;
  float* scales;
  int K, D;               // row width and width of one contiguous piece (head)
  int64_t head_stride;    // elements between consecutive D-wide pieces of a row
  int64_t row_stride;     // elements between rows
  int64_t rows;
  int wide;               // q is 16-byte aligned: 16-byte stores (8-byte ones otherwise)
};

constexpr int ROW_F = 20;               // floats per 16-value row of a half-warp's exchange patch (16 + 4 padding)
constexpr int PATCH_F = 16 * ROW_F + 16;  // the two half-warps of a warp land on different banks

__device__ __forceinline__ void unpack16h(const uint4* raw, float* v) {
  const uint32_t w[8] = {raw[0].x, raw[0].y, raw[0].z, raw[0].w, raw[1].x, raw[1].y, raw[1].z, raw[1].w};
  uint32_t special = 0;  // a half with all exponent bits set (NaN or infinity) carries into its sign bit
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&w[j]));
    v[2 * j] = f.x;
    v[2 * j + 1] = f.y;
    special |= (w[j] & 0x7FFF7FFFu) + 0x04000400u;
  }
  if (special & 0x80008000u) {
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const __half2 h = *reinterpret_cast<const __half2*>(&w[j]);
      v[2 * j] = nan_to_num_h(__low2half(h));
      v[2 * j + 1] = nan_to_num_h(__high2half(h));
    }
  }
}

// With the RMS norm, rows of 4,097 to 8,192 columns keep two CTAs per SM and rows of up to 1,024 sixteen, which the compiler's own 74 and
// 69 registers do not leave (3,594 x 8,192: 66.3 us with one, 57.7 with two).
template <int T, int ACT>
__global__ void __launch_bounds__(T, ACT == ACT_RMS_NORM && (T == 64 || T == 512) ? 1024 / T : 0) vae_out_quant_kernel(const OutQuantParams p) {
  grid_dependency_begin();
  __shared__ __align__(16) float patch[T / 16][PATCH_F];
  __shared__ float red[2][T / 16], red_ss[2][T / 16];  // two sets: one barrier per reduction and row is enough
  const int tid = threadIdx.x, grp = tid >> 4, t = tid & 15;
  const int K = p.K;
  const int col = tid << 4;
  const bool active = col < K;  // K is a multiple of 256: uniform over a half-warp
  const int ngrp = K >> 8;
  int64_t off[2] = {0, 0};      // the row's two 8-wide pieces may belong to different heads
  if (active) {
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const int c = col + 8 * i, head = c / p.D;
      off[i] = head * p.head_stride + (c - head * p.D);
    }
  }
  uint4 raw[2], up[2];
  auto load = [&](int64_t row) {
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      raw[i] = make_uint4(0, 0, 0, 0);
      if (ACT == ACT_SWIGLU) up[i] = make_uint4(0, 0, 0, 0);
      if (active) {
        const __half* src = p.o + off[i] + row * p.row_stride;
        raw[i] = ld_global_16(src);
        if (ACT == ACT_SWIGLU) up[i] = ld_global_16(src + p.up_offset);
      }
    }
  };
  int64_t row = blockIdx.x;
  if (row < p.rows) load(row);
  for (int par = 0; row < p.rows; row += gridDim.x, par ^= 1) {
    float v[16];
    unpack16h(raw, v);
    if (ACT == ACT_SWIGLU) {
      // y = silu(gate) * up with gate = this row's first K values, up = the K values up_offset further on
      float u[16];
      unpack16h(up, u);
#pragma unroll
      for (int j = 0; j < 16; ++j)
        v[j] = __fmul_rn(__fmul_rn(v[j], __fdiv_rn(1.f, __fadd_rn(1.f, expf(-v[j])))), u[j]);
    }
    if (row + gridDim.x < p.rows) load(row + gridDim.x);  // in flight under the rest of this row
    if (ACT == ACT_RMS_NORM) {
      // y = (x * r) * w, r = 1 / sqrt(mean(x^2) + eps); the sum of squares in a fixed order: runs of 8 columns in order,
      // an xor butterfly (16, 8, 4, 2, 1) over the 32 runs of a group, then the groups in order. A thread holds the runs
      // 2t and 2t + 1: run distance 16, 8, 4, 2 is lane distance 8, 4, 2, 1, the last step is inside the thread.
      float sa = 0.f, sb = 0.f;
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        sa = __fadd_rn(sa, __fmul_rn(v[j], v[j]));
        sb = __fadd_rn(sb, __fmul_rn(v[8 + j], v[8 + j]));
      }
#pragma unroll
      for (int o = 8; o; o >>= 1) {
        sa = __fadd_rn(sa, __shfl_xor_sync(0xffffffffu, sa, o));
        sb = __fadd_rn(sb, __shfl_xor_sync(0xffffffffu, sb, o));
      }
      if (t == 0) red_ss[par][grp] = __fadd_rn(sa, sb);
      __syncthreads();
      float ss = red_ss[par][0];
      for (int w = 1; w < ngrp; ++w) ss = __fadd_rn(ss, red_ss[par][w]);
      const float r = __fdiv_rn(1.f, __fsqrt_rn(__fadd_rn(__fdiv_rn(ss, static_cast<float>(K)), p.eps)));
      if (active) {
        float wv[16];
#pragma unroll
        for (int j = 0; j < 16; ++j) wv[j] = 1.f;
        if (p.act_w) {
#pragma unroll
          for (int i = 0; i < 2; ++i) {
            const uint4 wr = __ldg(reinterpret_cast<const uint4*>(p.act_w + col + 8 * i));
            const __half* h = reinterpret_cast<const __half*>(&wr);
#pragma unroll
            for (int j = 0; j < 8; ++j) wv[8 * i + j] = __half2float(h[j]);
          }
        }
#pragma unroll
        for (int j = 0; j < 16; ++j) v[j] = __fmul_rn(__fmul_rn(v[j], r), wv[j]);
      }
    }
    // stages 1 and 4, exchange, stages 16 and 64: v[i] becomes column t + 16 i of the group
    float* mine = patch[grp];
    fht16(v);
#pragma unroll
    for (int j = 0; j < 16; j += 4)
      *reinterpret_cast<float4*>(mine + t * ROW_F + j) = make_float4(v[j], v[j + 1], v[j + 2], v[j + 3]);
    __syncwarp();
#pragma unroll
    for (int i = 0; i < 16; ++i) v[i] = mine[i * ROW_F + t];
    fht16(v);
    float am = 0.f;
#pragma unroll
    for (int j = 0; j < 16; ++j) {
      v[j] = __fmul_rn(v[j], 0.0625f);
      am = fmaxf(am, fabsf(v[j]));
    }
#pragma unroll
    for (int o = 8; o; o >>= 1) am = fmaxf(am, __shfl_xor_sync(0xffffffffu, am, o));
    if (t == 0) red[par][grp] = am;
    __syncthreads();
    am = red[par][0];
    for (int w = 1; w < ngrp; ++w) am = fmaxf(am, red[par][w]);
    const float scale = fmaxf(__fmul_rn(fminf(am, 65504.f), 1.0f / 127.0f), 1.0e-30f);
    const float scale_h = __half2float(__float2half_rn(scale));
    if (tid == 0) p.scales[row] = scale;
    // The quotient vh / scale_h is the correctly rounded one: with inv the rounded reciprocal, q0 = vh * inv and the exact
    // remainder fma(-q0, scale_h, vh), q = fma(remainder, inv, q0) equals the IEEE quotient (Markstein) as long as nothing
    // under- or overflows. vh and scale_h are fp16 values, so that holds whenever vh is finite and scale_h is not 0; a
    // row with a value beyond fp16's range, or so small that its scale rounds to 0, divides (uniform over the row).
    const bool exact_div = !(am <= 65504.f) || scale_h == 0.f;
    const float inv = __fdiv_rn(1.f, scale_h);
    uint8_t* bytes = reinterpret_cast<uint8_t*>(mine);
    __syncwarp();  // the group's values have been read
    const __half2 lo2 = __float2half2_rn(-128.f), hi2 = __float2half2_rn(127.f), magic2 = __float2half2_rn(1536.f);
#pragma unroll
    for (int i = 0; i < 16; i += 2) {
      const float2 vh = __half22float2(__floats2half2_rn(v[i], v[i + 1]));
      float q0, q1;
      if (exact_div) {
        q0 = __fdiv_rn(vh.x, scale_h);
        q1 = __fdiv_rn(vh.y, scale_h);
      } else {
        q0 = __fmul_rn(vh.x, inv);
        q1 = __fmul_rn(vh.y, inv);
        q0 = fmaf(fmaf(-q0, scale_h, vh.x), inv, q0);
        q1 = fmaf(fmaf(-q1, scale_h, vh.y), inv, q1);
      }
      // the quotient through fp16, clamped (a NaN quotient, 0 / 0, becomes -128), then rounded half to even by adding
      // 1.5 * 2^10, whose last place is 1: the code is the low byte of the sum's bits
      const __half2 c = __hadd2(__hmin2(__hmax2(__floats2half2_rn(q0, q1), lo2), hi2), magic2);
      const uint32_t bits = *reinterpret_cast<const uint32_t*>(&c);
      bytes[t + 16 * i] = static_cast<uint8_t>(bits);
      bytes[t + 16 * i + 16] = static_cast<uint8_t>(bits >> 16);
    }
    __syncwarp();
    if (active) {
      const uint4 o = *reinterpret_cast<const uint4*>(bytes + 16 * t);
      int8_t* dst = p.q + row * K + col;
      if (p.wide) {
        *reinterpret_cast<uint4*>(dst) = o;
      } else {
        *reinterpret_cast<uint2*>(dst) = make_uint2(o.x, o.y);
        *reinterpret_cast<uint2*>(dst + 8) = make_uint2(o.z, o.w);
      }
    }
    __syncwarp();  // before the next row's values overwrite the patch
  }
}

template <int T, int ACT>
int launch_out_quant(const OutQuantParams& p, cudaStream_t stream) {
  auto kern = vae_out_quant_kernel<T, ACT>;
  int occ = 1;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, kern, T, 0) != cudaSuccess || occ < 1) occ = 1;
  const int64_t resident = static_cast<int64_t>(device_sm_count()) * occ;
  // chained (launch_kernel) while small, and not in a graph. Feed-forward, us with both quantizers chained / not, on a stream: 64 rows
  // 30.7 / 32.5, 1,000 75.2 / 78.9, 3,594 208.0 / 206.7; from graphs 28.8 / 28.2, 70.8 / 71.5, 224 / 218
  return check_cuda(launch_kernel(!in_capture(stream) && p.rows * p.K <= (1ll << 23), kern, dim3(static_cast<unsigned>(p.rows < resident ? p.rows : resident)), T, 0, stream, 1, p),
                    "vae_out_quant launch");
}
template <int ACT>
int launch_out_quant_act(const OutQuantParams& p, cudaStream_t stream) {
  const int threads = p.K / 16;
  if (threads <= 64) return launch_out_quant<64, ACT>(p, stream);
  if (threads <= 128) return launch_out_quant<128, ACT>(p, stream);
  if (threads <= 256) return launch_out_quant<256, ACT>(p, stream);
  return launch_out_quant<512, ACT>(p, stream);
}

}  // namespace
}  // namespace rh3

using namespace rh3;

namespace {
int out_quant_launch(OutQuantParams p, cudaStream_t stream) {
  p.wide = (reinterpret_cast<uintptr_t>(p.q) & 15) == 0;
  if (p.act == ACT_RMS_NORM) return launch_out_quant_act<ACT_RMS_NORM>(p, stream);
  if (p.act == ACT_SWIGLU) return launch_out_quant_act<ACT_SWIGLU>(p, stream);
  return launch_out_quant_act<ACT_NONE>(p, stream);
}
}  // namespace

extern "C" int rh3_vae_out_quant(const void* o_f16, int64_t B, int64_t H, int64_t S, int64_t D, void* q, float* scales,
                                 cudaStream_t stream) {
  RH3_CHECK_ARG(B >= 0 && H > 0 && S >= 0 && D > 0 && D % 8 == 0, "vae_out_quant: bad shape B=%lld H=%lld S=%lld D=%lld",
                (long long)B, (long long)H, (long long)S, (long long)D);
  const int64_t K = H * D;
  RH3_CHECK_ARG(K % 256 == 0 && 256 % D == 0, "vae_out_quant: H*D must be a multiple of 256 and D must divide 256");
  RH3_CHECK_ARG(K <= 8192, "vae_out_quant: row width %lld is larger than 8192", (long long)K);
  RH3_CHECK_ARG(B * S < (1ll << 31), "vae_out_quant: too many rows");
  if (B == 0 || S == 0) return 0;
  RH3_CHECK_ARG(o_f16 && q && scales, "vae_out_quant: null pointer");
  RH3_CHECK_ARG((reinterpret_cast<uintptr_t>(o_f16) & 15) == 0 && (reinterpret_cast<uintptr_t>(q) & 7) == 0,
                "vae_out_quant: o must be 16-byte aligned and q 8-byte aligned");
  for (int64_t b = 0; b < B; ++b) {
    OutQuantParams p{};
    p.o = static_cast<const __half*>(o_f16) + b * H * S * D;
    p.q = static_cast<int8_t*>(q) + b * S * K;
    p.scales = scales + b * S;
    p.K = (int)K; p.D = (int)D; p.head_stride = S * D; p.row_stride = D; p.rows = S;
    if (int e = out_quant_launch(p, stream)) return e;
  }
  return 0;
}

// The same row arithmetic on a row-major fp16 matrix x [M, K] (row stride ldx): the quantizer the decoder's linears
// call on their inputs (vae_fast._quantize, custom_nodes/rapid_h3/vae_fast.py:71-85).
extern "C" int rh3_vae_quant_rows(const void* x_f16, int64_t ldx, int64_t M, int64_t K, void* q, float* scales,
                                  cudaStream_t stream) {
  RH3_CHECK_ARG(M >= 0 && K > 0 && K % 256 == 0 && K <= 8192, "vae_quant_rows: K=%lld must be a multiple of 256, <= 8192",
                (long long)K);
  RH3_CHECK_ARG(M < (1ll << 31) && ldx >= K && ldx % 8 == 0, "vae_quant_rows: bad M or row stride");
  if (M == 0) return 0;
  RH3_CHECK_ARG(x_f16 && q && scales, "vae_quant_rows: null pointer");
  RH3_CHECK_ARG((reinterpret_cast<uintptr_t>(x_f16) & 15) == 0 && (reinterpret_cast<uintptr_t>(q) & 7) == 0,
                "vae_quant_rows: x must be 16-byte aligned and q 8-byte aligned");
  OutQuantParams p{};
  p.o = static_cast<const __half*>(x_f16);
  p.q = static_cast<int8_t*>(q);
  p.scales = scales;
  p.K = (int)K; p.D = 256; p.head_stride = 256; p.row_stride = ldx; p.rows = M;
  return out_quant_launch(p, stream);
}

// The quantizer with a fused activation prologue (the `act` argument of the quantizer the reference calls in
// vae_fast._quantize, vae_fast.py:71-85: "rms_norm" for the inputs of to_qkv and w1, "swiglu" for the input of w2
// when the SwiGLU is not in w1's epilogue). act 1: x [M, K], y = (x * r) * weight (fp16 [K] or NULL),
// r = 1 / sqrt(mean(x^2) + eps); act 2: x [M, 2K] = [gate | up], y = gate / (1 + e^-gate) * up. y stays fp32 into
// the rotation. The per-row arithmetic of that fused form lives in a third-party binary (comfy-kitchen) whose source
// is not part of the reference repository; this entry defines it with IEEE operations (CPU oracle: oracle/vae_ops.py).
extern "C" int rh3_vae_quant_rows_act(const void* x_f16, int64_t ldx, int64_t M, int64_t K, int act,
                                      const void* act_weight_f16, float eps, void* q, float* scales,
                                      cudaStream_t stream) {
  RH3_CHECK_ARG(act == ACT_RMS_NORM || act == ACT_SWIGLU, "vae_quant_rows_act: act must be 1 (rms_norm) or 2 (swiglu)");
  RH3_CHECK_ARG(M >= 0 && K > 0 && K % 256 == 0 && K <= 8192, "vae_quant_rows_act: K=%lld must be a multiple of 256, <= 8192",
                (long long)K);
  RH3_CHECK_ARG(M < (1ll << 31) && ldx >= (act == ACT_SWIGLU ? 2 * K : K) && ldx % 8 == 0,
                "vae_quant_rows_act: bad M or row stride");
  if (M == 0) return 0;
  RH3_CHECK_ARG(x_f16 && q && scales, "vae_quant_rows_act: null pointer");
  RH3_CHECK_ARG((reinterpret_cast<uintptr_t>(x_f16) & 15) == 0 && (reinterpret_cast<uintptr_t>(q) & 7) == 0 &&
                    (reinterpret_cast<uintptr_t>(act_weight_f16) & 15) == 0,
                "vae_quant_rows_act: x and the norm weight must be 16-byte aligned and q 8-byte aligned");
  OutQuantParams p{};
  p.act = act;
  p.act_w = act == ACT_RMS_NORM ? static_cast<const __half*>(act_weight_f16) : nullptr;
  p.eps = eps;
  p.up_offset = K;
  p.o = static_cast<const __half*>(x_f16);
  p.q = static_cast<int8_t*>(q);
  p.scales = scales;
  p.K = (int)K; p.D = 256; p.head_stride = 256; p.row_stride = ldx; p.rows = M;
  return out_quant_launch(p, stream);
}

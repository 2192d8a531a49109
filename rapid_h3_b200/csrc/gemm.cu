// Row-wise-scaled W8A8 GEMM on the Blackwell tensor cores.
//
//   acc[m, n] = sum_k xq[m, k] * wq[n, k]          int8 x int8 -> int32 (tcgen05 kind::i8), or
//                                                   e4m3 x e4m3 -> fp32 (tcgen05 kind::f8f6f4)
//   EPI_PLAIN : out[m, n]   = bf16(((float(acc) * xs[m]) * ws[n]) + bias[n])
//   EPI_BIAS2 : out[m, n]   = bf16(bf16((float(acc) * xs[m]) * ws[n]) + bias[n]): a product that is rounded first and
//               gets its bias in bf16, as a separate addition would give it
//   EPI_F32   : out[m, n]   = float(bf16(...)) + bias[n] in fp32; rows flagged for a second pass leave the bias to it
//   EPI_F32_ADD: out[rows[m], n] = (out[rows[m], n] + float(bf16(...))) + bias[n]; the number of rows is read on the device
//   EPI_GATED : resid[m, n] = bf16(fma(bf16((float(acc) * xs[m]) * ws[n]), gate[n], resid[m, n]))   (in place)
//   EPI_GATED2: the same with two fp32 gate rows, rounded to bf16 here: rows below gate_split take the first, the rest the second
//   EPI_SWIGLU: columns come in groups of 8 = [g 4j..4j+3 | u 4j..4j+3];
//               out[m, n/2] = bf16(silu(bf16(g)) * bf16(u)), half-width store
// (reference: custom_nodes/rapid_h3/csrc/fp8_rowwise.cu:294-304 plain epilogue, :333-336 gated
//  residual, :74-93 SwiGLU store; PyTorch emulation custom_nodes/rapid_h3/kernels.py:129-137).
//
// Structure (one persistent CTA per SM, 320 threads), tiles of 128 rows (256 on CTA pairs) x 256, 128 or 64 columns:
//   warp 0      TMA producer: A rows and B rows of one to four 128-byte K slabs per stage, a 192 KB ring
//   warp 1      MMA issuer: 4 x tcgen05.mma (K32) per slab into a TMEM accumulator;
//               two accumulators so the epilogue of tile i overlaps the main loop of i+1
//   warps 2..9  epilogue: tcgen05.ld 32 columns at a time, dequantize, fused epilogue, 64-byte
//               contiguous bf16 stores per thread-row
// Tensor-core bound: 2*M*N*K operations per call.

#include <atomic>

#include "common.cuh"
#include "rapidh3_b200.h"

namespace rh3 {
namespace {

constexpr int BM = 128;
constexpr int BN = 256;
constexpr int BK = 128;  // bytes (= elements for 8-bit operands) along K per stage
constexpr int A_BYTES = BM * BK;
constexpr int RING_BYTES = 4 * (A_BYTES + BN * BK);   // what a ring may take: 192 KB
constexpr int MAX_STAGES = 10;
// Ring of a kernel whose CTAs load `brows` rows of B per stage: as many stages as fit, so that narrow tiles, whose stages
// hold less, still have enough bytes in flight to cover the latency of L2.
__host__ __device__ constexpr int slab_bytes(int brows) { return A_BYTES + brows * BK; }
// K slabs behind one barrier: the round trip of a stage (wait, four MMAs, commit) is a few hundred cycles in the issuing warp,
// which the 128 or 256 tensor cycles of a narrow slab do not cover. us at N = K = 4,096 with one, two and four slabs: 37 rows,
// 64-column tiles 10.8 / 8.7 / 7.5, 200 rows, 64-column pair tiles 11.3 / 8.4 / 8.9, 512 rows, 128-column pair tiles
// 12.7 / 10.3; two of 256 columns measure the same as one or worse (12.5 / 14.1 at 37 rows).
__host__ __device__ constexpr int slabs_per_stage(int tn, bool pair) { return tn == 64 && !pair ? 4 : tn < BN ? 2 : 1; }
__host__ __device__ constexpr int ring_stages(int brows, int slabs) {
  return RING_BYTES / (slabs * slab_bytes(brows)) < MAX_STAGES ? RING_BYTES / (slabs * slab_bytes(brows)) : MAX_STAGES;
}
// Two warps per TMEM lane quadrant, each draining half of the accumulator's columns: with one, the epilogue of a short K
// outlasts the main loop of the next tile (w1 + SwiGLU in fp16, 3,594 x 16,384 x 2,048: 187 us with four warps and the
// division routine, 85 with eight and silu_div; fp16 with residual, N = 2,048, K = 8,192: 61 -> 56; long-K bf16 shapes
// measure the same). The price is registers: 168 a thread at 320 threads, which every epilogue has to fit.
constexpr int EPI_WARPS = 8;
constexpr int EPI_THREADS = 32 * EPI_WARPS;
constexpr int GEMM_THREADS = 64 + EPI_THREADS;
#ifndef RH3_GEMM_GROUP_M
#define RH3_GEMM_GROUP_M 16
#endif
constexpr int GROUP_M = RH3_GEMM_GROUP_M;  // tile rasterisation: GROUP_M row-tiles share each column-tile in L2

enum { EPI_PLAIN = 0, EPI_GATED = 1, EPI_SWIGLU = 2, EPI_F16 = 3, EPI_SWIGLU_F16 = 4, EPI_BIAS2 = 5, EPI_F32 = 6, EPI_F32_ADD = 7, EPI_GATED2 = 8 };
__host__ __device__ constexpr bool is_gated(int epi) { return epi == EPI_GATED || epi == EPI_GATED2; }

struct GemmParams {
  int M, N, K;
  int a_rows;                 // rows of A that a load brings in: 128, or fewer where the call has fewer (the rest of the tile is not read out)
  const float* xs;
  const float* ws;
  const __nv_bfloat16* bias;  // EPI_PLAIN (optional), EPI_BIAS2
  __nv_bfloat16* out;         // EPI_PLAIN / EPI_SWIGLU
  int64_t ldo;
  int32_t* acc_dump;          // optional raw accumulator dump [M, N] (int32, or fp32 bits for fp8)
  const __nv_bfloat16* gate;  // EPI_GATED
  const float* gate_f[2];     // EPI_GATED2
  int gate_split;
  __nv_bfloat16* resid;       // EPI_GATED
  int64_t ldr;
  // fp16 epilogues of the VAE transformer decoder (EPI_F16 / EPI_SWIGLU_F16)
  const __half* bias_h;    // [N]
  const __half* rscale_h;  // [N] or null (EPI_F16 with residual)
  const __half* resid_h;   // [M, N] row stride ldr, or null
  __half* out_h;           // row stride ldo
  // fp32 epilogues of the text encoder's linears (EPI_F32 / EPI_F32_ADD)
  float* out_f;            // row stride ldo
  const float* bias_f;     // [N] or null
  const uint8_t* flags;    // EPI_F32: rows whose bias the second pass adds, or null
  const int32_t* rows;     // EPI_F32_ADD: output row of every row of xq
  const int32_t* m_dev;    // EPI_F32_ADD: number of rows, at most M
  int wide;                // bf16 output (and gated residual) rows are 32-byte aligned: 32-byte accesses in the epilogue
  int* status;
};

struct __align__(8) GemmSmemTail {
  uint64_t full[MAX_STAGES];
  uint64_t empty[MAX_STAGES];
  uint64_t acc_full[2];
  uint64_t acc_empty[2];
  uint32_t tmem_base;
  int abort_flag;
  float ws[BN];
  float aux[BN];   // bias or gate as fp32
  float aux2[BN];  // residual scale (EPI_F16) or second gate (EPI_GATED2) as fp32
};

constexpr int GEMM_SMEM_BYTES = RING_BYTES + sizeof(GemmSmemTail) + 1024;  // +1024 alignment slack

__device__ __forceinline__ void tile_coords(int tile, int num_m, int num_n, int& m_blk, int& n_blk) {
  const int per_group = GROUP_M * num_n;
  const int g = tile / per_group;
  const int first_m = g * GROUP_M;
  const int gsize = min(GROUP_M, num_m - first_m);
  const int t = tile - g * per_group;
  m_blk = first_m + t % gsize;
  n_blk = t / gsize;
}

// The epilogue of one accumulator row (epilogue_row below): EPI_COLS columns, 32 at a time from TMEM, dequantized and
// stored through the fused epilogue EPI. `t_row` = TMEM address of this thread's row (lane) at the accumulator's first
// column.
// The residual row of an epilogue that adds one (gated residual, fp16 residual): its EPI_COLS columns are asked into L2
// while the tile's MMAs still run, so the epilogue's loads do not wait on HBM (the residual of a step is far
// larger than L2 and cold by the time its tile comes up).
template <int EPI, int EPI_COLS>
__device__ __forceinline__ void prefetch_residual(const GemmParams& p, int row, bool row_ok, int n0) {  // n0: first of EPI_COLS columns
  if (!row_ok) return;
  if (is_gated(EPI)) {
    const __nv_bfloat16* r = p.resid + static_cast<int64_t>(row) * p.ldr + n0;
#pragma unroll
    for (int c = 0; c < EPI_COLS; c += 64)
      if (n0 + c < p.N) prefetch_l2(r + c);
  } else if (EPI == EPI_F16) {
    if (p.resid_h) {
      const __half* r = p.resid_h + static_cast<int64_t>(row) * p.ldr + n0;
#pragma unroll
      for (int c = 0; c < EPI_COLS; c += 64)
        if (n0 + c < p.N) prefetch_l2(r + c);
    }
  }
}

// 32 bf16 outputs of one row (four 16-byte groups) to o: 32-byte stores where the row allows it, 16-byte stores for
// what remains in range otherwise.
__device__ __forceinline__ void store_chunk_bf16(__nv_bfloat16* o, const uint4* w4, int col0, int N, int wide) {
#pragma unroll
  for (int g = 0; g < 4; g += 2) {
    if (wide && col0 + g * 8 + 16 <= N) {
      st_global_32(o + g * 8, w4[g], w4[g + 1]);
    } else {
      if (col0 + g * 8 + 8 <= N) *reinterpret_cast<uint4*>(o + g * 8) = w4[g];
      if (col0 + g * 8 + 16 <= N) *reinterpret_cast<uint4*>(o + g * 8 + 8) = w4[g + 1];
    }
  }
}

// The gated residual's values of chunk c of a row (four 16-byte pieces; zeros off the edge).
__device__ __forceinline__ void load_gated_residual(const GemmParams& p, int row, bool row_ok, int n0, int c, uint4* dst) {
  const int col0 = n0 + c * 32;
  const __nv_bfloat16* o = p.resid + static_cast<int64_t>(row) * p.ldr + col0;
#pragma unroll
  for (int g = 0; g < 4; g += 2) {
    if (p.wide && row_ok && col0 + g * 8 + 16 <= p.N) {
      ld_global_32(o + g * 8, dst[g], dst[g + 1]);
    } else {
      dst[g] = (row_ok && col0 + g * 8 + 8 <= p.N) ? *reinterpret_cast<const uint4*>(o + g * 8) : make_uint4(0, 0, 0, 0);
      dst[g + 1] = (row_ok && col0 + g * 8 + 16 <= p.N) ? *reinterpret_cast<const uint4*>(o + g * 8 + 8) : make_uint4(0, 0, 0, 0);
    }
  }
}

// g / (1 + e^-g) without the division routine: 1/d from the approximate reciprocal and one Newton step (to the last
// bit or its neighbour), times g, one correction by the exact remainder g - q d (Markstein's division: the remainder is
// exact in one fused multiply-add, and adding it times the reciprocal rounds the quotient once). The exponent is held at 80: beyond it
// d would leave the range the reciprocal works in, and g / e^80 is already far below fp16's smallest value (a NaN g
// still gives NaN; an infinite one gives what the division would: g itself, or NaN for -inf / inf).
__device__ __forceinline__ float silu_div(float g) {
  const float d = 1.f + __expf(fminf(-g, 80.f));
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(d));
  r = fmaf(fmaf(-d, r, 1.f), r, r);
  const float q = g * r;
  const float rem = fmaf(-q, d, g);
  return fabsf(g) <= 65504.f ? fmaf(rem, r, q) : (g > 0.f ? q : __int_as_float(0x7fffffff));
}

// rows of this call: the second pass reads its number from the device (the host never sees it)
template <int EPI>
__device__ __forceinline__ int gemm_rows(const GemmParams& p) {
  return EPI == EPI_F32_ADD ? min(p.M, *p.m_dev) : p.M;
}

template <int KIND_F8, int EPI, int EPI_COLS>
__device__ __forceinline__ void epilogue_row(const GemmParams& p, const GemmSmemTail* tail, uint32_t t_row, int row,
                                             bool row_ok, float xs, int n0, int c_first, const uint4* res0) {
  // `c_first`: first 32-column chunk of this warp's EPI_COLS columns
  // Two 32-column chunks are loaded per wait where no residual has to be held beside them, so a warp's half of a tile costs
  // two TMEM round trips instead of four; `old4` = the chunk's residual values (gated residual only), loaded one chunk ahead
  auto chunk = [&](const uint32_t* r, int c, const uint4* old4) {
    const int col0 = n0 + c * 32;
    if (row_ok && col0 < p.N) {
      if (p.acc_dump) {
        int32_t* d = p.acc_dump + static_cast<int64_t>(row) * p.N + col0;
#pragma unroll
        for (int j = 0; j < 32; j += 4)
          if (col0 + j + 4 <= p.N) *reinterpret_cast<uint4*>(d + j) = make_uint4(r[j], r[j + 1], r[j + 2], r[j + 3]);
      }
      float y[32];
#pragma unroll
      for (int j = 0; j < 32; ++j) {
        const float a = KIND_F8 ? __uint_as_float(r[j]) : __int2float_rn(static_cast<int>(r[j]));
        y[j] = __fmul_rn(__fmul_rn(a, xs), tail->ws[c * 32 + j]);
      }
      if (EPI == EPI_PLAIN || EPI == EPI_BIAS2) {
        __nv_bfloat16* o = p.out + static_cast<int64_t>(row) * p.ldo + col0;
        uint4 w4[4];
#pragma unroll
        for (int g = 0; g < 4; ++g) {
          uint32_t w[4];
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            const int e = g * 8 + 2 * j;
            const float y0 = EPI == EPI_BIAS2 ? bf16_round(y[e]) : y[e], y1 = EPI == EPI_BIAS2 ? bf16_round(y[e + 1]) : y[e + 1];
            w[j] = pack_bf16x2(__fadd_rn(y0, tail->aux[c * 32 + e]), __fadd_rn(y1, tail->aux[c * 32 + e + 1]));
          }
          w4[g] = make_uint4(w[0], w[1], w[2], w[3]);
        }
        store_chunk_bf16(o, w4, col0, p.N, p.wide);
      } else if (is_gated(EPI)) {
        const float* gate = EPI == EPI_GATED2 && row >= p.gate_split ? tail->aux2 : tail->aux;
        __nv_bfloat16* o = p.resid + static_cast<int64_t>(row) * p.ldr + col0;
        uint4 w4[4];
#pragma unroll
        for (int g = 0; g < 4; ++g) {
          const uint4 old = old4[g];
          const uint32_t ow[4] = {old.x, old.y, old.z, old.w};
          uint32_t w[4];
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            const int e = g * 8 + 2 * j;
            const float v0 = fmaf(bf16_round(y[e]), gate[c * 32 + e], bf16_lo(ow[j]));
            const float v1 = fmaf(bf16_round(y[e + 1]), gate[c * 32 + e + 1], bf16_hi(ow[j]));
            w[j] = pack_bf16x2(v0, v1);
          }
          w4[g] = make_uint4(w[0], w[1], w[2], w[3]);
        }
        store_chunk_bf16(o, w4, col0, p.N, p.wide);
      } else if (EPI == EPI_F32 || EPI == EPI_F32_ADD) {
        // aux holds the bias (-0 without one: adding it changes nothing)
        float* o = p.out_f + static_cast<int64_t>(EPI == EPI_F32_ADD ? p.rows[row] : row) * p.ldo + col0;
        const bool with_bias = EPI == EPI_F32_ADD || !(p.flags && p.flags[row]);
#pragma unroll
        for (int g = 0; g < 4; ++g) {
          if (col0 + g * 8 + 8 <= p.N) {
            uint4 old[2] = {};
            if (EPI == EPI_F32_ADD) ld_global_32(o + g * 8, old[0], old[1]);
            const uint32_t ow[8] = {old[0].x, old[0].y, old[0].z, old[0].w, old[1].x, old[1].y, old[1].z, old[1].w};
            uint32_t w[8];
#pragma unroll
            for (int j = 0; j < 8; ++j) {
              float v = bf16_round(y[g * 8 + j]);
              if (EPI == EPI_F32_ADD) v = __fadd_rn(__uint_as_float(ow[j]), v);
              if (with_bias) v = __fadd_rn(v, tail->aux[c * 32 + g * 8 + j]);
              w[j] = __float_as_uint(v);
            }
            st_global_32(o + g * 8, make_uint4(w[0], w[1], w[2], w[3]), make_uint4(w[4], w[5], w[6], w[7]));
          }
        }
      } else if (EPI == EPI_F16) {
        // y1 = fp16(y + bias); with a residual: out = fp16(float(y1) * rscale + resid), two separate roundings
        __half* o = p.out_h + static_cast<int64_t>(row) * p.ldo + col0;
        const __half* rs = p.resid_h ? p.resid_h + static_cast<int64_t>(row) * p.ldr + col0 : nullptr;
#pragma unroll
        for (int g = 0; g < 4; ++g) {
          if (col0 + g * 8 + 8 <= p.N) {
            uint4 old = make_uint4(0, 0, 0, 0);
            if (rs) old = *reinterpret_cast<const uint4*>(rs + g * 8);
            const __half2* oh = reinterpret_cast<const __half2*>(&old);
            uint32_t w[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) {
              const int e = g * 8 + 2 * j;
              float v0 = __half2float(__float2half_rn(__fadd_rn(y[e], tail->aux[c * 32 + e])));
              float v1 = __half2float(__float2half_rn(__fadd_rn(y[e + 1], tail->aux[c * 32 + e + 1])));
              if (rs) {
                const float2 r2 = __half22float2(oh[j]);
                v0 = __fadd_rn(__fmul_rn(v0, tail->aux2[c * 32 + e]), r2.x);
                v1 = __fadd_rn(__fmul_rn(v1, tail->aux2[c * 32 + e + 1]), r2.y);
              }
              const __half2 h2 = __floats2half2_rn(v0, v1);
              w[j] = *reinterpret_cast<const uint32_t*>(&h2);
            }
            *reinterpret_cast<uint4*>(o + g * 8) = make_uint4(w[0], w[1], w[2], w[3]);
          }
        }
      } else if (EPI == EPI_SWIGLU_F16) {
        // columns in groups of 8 = [g0..g3 | u0..u3]; g, u = fp16(y + bias); out = fp16(g / (1 + e^-g) * u)
        __half* o = p.out_h + static_cast<int64_t>(row) * p.ldo + (col0 >> 1);
#pragma unroll
        for (int hgrp = 0; hgrp < 2; ++hgrp) {
          if (col0 + hgrp * 16 + 16 <= p.N) {
            uint32_t w[4];
#pragma unroll
            for (int q = 0; q < 2; ++q) {
              const int b = hgrp * 16 + q * 8;
              float h[4];
#pragma unroll
              for (int j = 0; j < 4; ++j) {
                const float gv = __half2float(__float2half_rn(__fadd_rn(y[b + j], tail->aux[c * 32 + b + j])));
                const float uv = __half2float(__float2half_rn(__fadd_rn(y[b + 4 + j], tail->aux[c * 32 + b + 4 + j])));
                h[j] = silu_div(gv) * uv;
              }
              const __half2 h01 = __floats2half2_rn(h[0], h[1]), h23 = __floats2half2_rn(h[2], h[3]);
              w[q * 2] = *reinterpret_cast<const uint32_t*>(&h01);
              w[q * 2 + 1] = *reinterpret_cast<const uint32_t*>(&h23);
            }
            *reinterpret_cast<uint4*>(o + hgrp * 8) = make_uint4(w[0], w[1], w[2], w[3]);
          }
        }
      } else {  // EPI_SWIGLU: 32 columns = 4 groups of [g0..g3 | u0..u3] -> 16 outputs
        __nv_bfloat16* o = p.out + static_cast<int64_t>(row) * p.ldo + (col0 >> 1);
        uint4 w4[2];
#pragma unroll
        for (int hgrp = 0; hgrp < 2; ++hgrp) {  // 16 columns -> 8 outputs -> 16 bytes
          {
            uint32_t w[4];
#pragma unroll
            for (int q = 0; q < 2; ++q) {  // one group of 8 columns -> 4 outputs
              const int b = hgrp * 16 + q * 8;
              float h[4];
#pragma unroll
              for (int j = 0; j < 4; ++j) {
                const float gv = bf16_round(y[b + j]);
                const float uv = bf16_round(y[b + 4 + j]);
                h[j] = __fdividef(gv, 1.f + __expf(-gv)) * uv;
              }
              w[q * 2] = pack_bf16x2(h[0], h[1]);
              w[q * 2 + 1] = pack_bf16x2(h[2], h[3]);
            }
            w4[hgrp] = make_uint4(w[0], w[1], w[2], w[3]);
          }
        }
        if (p.wide && col0 + 32 <= p.N) {
          st_global_32(o, w4[0], w4[1]);
        } else {
          if (col0 + 16 <= p.N) *reinterpret_cast<uint4*>(o) = w4[0];
          if (col0 + 32 <= p.N) *reinterpret_cast<uint4*>(o + 8) = w4[1];
        }
      }
    }
  };
  if (is_gated(EPI)) {
    // The residual of the next chunk is fetched while the current one is computed (the loads of a row come from a cold
    // 8 KB-strided row: waiting for them chunk by chunk was most of this epilogue's time); the first chunk's, `res0`, was
    // fetched by the caller before it waited for the accumulator. One chunk per TMEM wait and one ahead is what 168
    // registers hold: two and two spilled 40-72 bytes a thread. With two gates, N = K = 4,096: 36,436 rows 549 -> 481 us,
    // 17,896 rows 278 -> 245, 6,196 rows 101 -> 88, 1,008 rows 23.1 -> 21.0 (four epilogue warps with two and two, which
    // do not spill either: no better than the spilling form at the first two sizes); K = 16,384 hides the epilogue and
    // measures the same within 2 %.
    uint4 res[2][4];
#pragma unroll
    for (int i = 0; i < 4; ++i) res[0][i] = res0[i];
#pragma unroll
    for (int it = 0; it < EPI_COLS / 32; ++it) {
      const int c = c_first + it;
      uint32_t r[32];
      tmem_ld32(t_row + c * 32, r);
      if (it + 1 < EPI_COLS / 32) load_gated_residual(p, row, row_ok, n0, c + 1, res[(it + 1) & 1]);
      tmem_ld_wait_regs(r);
      chunk(r, c, res[it & 1]);
    }
    return;
  }
  if (EPI_COLS == 32) {
    uint32_t r[32];
    tmem_ld32(t_row + c_first * 32, r);
    tmem_ld_wait_regs(r);
    chunk(r, c_first, nullptr);
    return;
  }
#pragma unroll 1
  for (int c = c_first; c < c_first + EPI_COLS / 32; c += 2) {
    uint32_t ra[32], rb[32];
    tmem_ld32(t_row + c * 32, ra);
    tmem_ld32(t_row + c * 32 + 32, rb);
    tmem_ld_wait_regs(ra);
    tmem_ld_wait_regs(rb);
    chunk(ra, c, nullptr);
    chunk(rb, c + 1, nullptr);
  }
}

template <int KIND_F8, int EPI, int TN>   // TN: columns of a tile
__global__ void __launch_bounds__(GEMM_THREADS, 1)
gemm_w8a8_kernel(const __grid_constant__ CUtensorMap tma_a, const __grid_constant__ CUtensorMap tma_b,
                 const GemmParams p) {
  constexpr int KS = slabs_per_stage(TN, false), STAGES = ring_stages(TN, KS), STAGE_BYTES = KS * slab_bytes(TN), EPI_COLS = TN / (EPI_WARPS / 4);
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  GemmSmemTail* tail = reinterpret_cast<GemmSmemTail*>(smem + RING_BYTES);
  volatile int* abort_flag = &tail->abort_flag;

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (EPI == EPI_F32_ADD) grid_dependency_wait();   // its row count is read on the device
  const int M = gemm_rows<EPI>(p);
  const int num_m = (M + BM - 1) / BM, num_n = (p.N + TN - 1) / TN;
  const int num_tiles = num_m * num_n;
  const int num_kb = (p.K + BK - 1) / BK;

  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(&tail->full[s], 1);
      mbar_init(&tail->empty[s], 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(&tail->acc_full[b], 1);
      mbar_init(&tail->acc_empty[b], EPI_WARPS);  // one arrival per epilogue warp
    }
    tail->abort_flag = 0;
    fence_barrier_init();
  }
  if (warp == 1) {
    tmem_alloc(&tail->tmem_base, 512);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  grid_dependency_trigger();
  if (EPI != EPI_F32_ADD) grid_dependency_wait();
  const uint32_t tmem_base = tail->tmem_base;

  if (warp == 0) {
    // ------------------------------ TMA producer ------------------------------
    if (lane == 0) {
      tma_prefetch_desc(&tma_a);
      tma_prefetch_desc(&tma_b);
      int stage = 0;
      uint32_t phase = 0;
      bool ok = true;
      for (int tile = blockIdx.x; tile < num_tiles && ok; tile += gridDim.x) {
        int m_blk, n_blk;
        tile_coords(tile, num_m, num_n, m_blk, n_blk);
        for (int kb = 0; kb < num_kb; kb += KS) {   // a slab past K reads zeros
          if (!mbar_wait(&tail->empty[stage], phase ^ 1, abort_flag, p.status, ST_TIMEOUT_STAGE_EMPTY)) {
            ok = false;
            break;
          }
          uint8_t* sa = smem + stage * STAGE_BYTES;
          mbar_arrive_expect_tx(&tail->full[stage], KS * (p.a_rows + TN) * BK);
#pragma unroll
          for (int q = 0; q < KS; ++q, sa += slab_bytes(TN)) {
            tma_load_2d(sa, &tma_a, (kb + q) * BK, m_blk * BM, &tail->full[stage]);
            tma_load_2d(sa + A_BYTES, &tma_b, (kb + q) * BK, n_blk * TN, &tail->full[stage]);
          }
          if (++stage == STAGES) { stage = 0; phase ^= 1; }
        }
      }
    }
  } else if (warp == 1) {
    // ------------------------------ MMA issuer ------------------------------
    // The whole warp runs the loop, converged: waits, counters, addresses and descriptors are then warp-uniform
    // values the compiler can keep in the uniform datapath, where the MMA instruction takes its operands from; one
    // elected lane (the same every time) issues the MMAs and the commits. On the bare issue pattern of this loop
    // (rh3_selftest_mma_rate, patterns 1 and 3) a single lane in the loop reaches 3.2 POP/s and the converged warp
    // 4.5; in this kernel the two forms measure the same (2.7 POP/s at K = 4096), so the issuing thread is not what
    // holds the tensor pipe at 70 % here.
    constexpr uint32_t idesc = KIND_F8 ? make_idesc(1, 0, 0, BM, TN) : make_idesc(2, 1, 1, BM, TN);
    int stage = 0;
    uint32_t phase = 0;
    int acc = 0;
    uint32_t acc_phase = 0;
    bool ok = true;
    for (int tile = blockIdx.x; tile < num_tiles && ok; tile += gridDim.x) {
      ok = __all_sync(0xffffffffu, mbar_wait(&tail->acc_empty[acc], acc_phase ^ 1, abort_flag, p.status, ST_TIMEOUT_ACC_EMPTY));
      if (!ok) break;
      tc_fence_after();
      const uint32_t d_tmem = tmem_base + acc * BN;
      for (int kb = 0; kb < num_kb; kb += KS) {   // a slab past K reads zeros
        ok = __all_sync(0xffffffffu, mbar_wait(&tail->full[stage], phase, abort_flag, p.status, ST_TIMEOUT_TMA_FULL));
        if (!ok) break;
        tc_fence_after();
        const uint32_t a_addr = smem_u32(smem + stage * STAGE_BYTES);
        if (elect_one()) {
#pragma unroll
          for (int q = 0; q < KS; ++q) {
            const uint32_t aq = a_addr + q * slab_bytes(TN);
            if (KIND_F8) mma4_f8_ss(d_tmem, make_desc_k128(aq), make_desc_k128(aq + A_BYTES), idesc, (kb + q) != 0);
            else mma4_i8_ss(d_tmem, make_desc_k128(aq), make_desc_k128(aq + A_BYTES), idesc, (kb + q) != 0);
          }
          mma_commit(&tail->empty[stage]);  // the stage is free once these MMAs have read it
        }
        __syncwarp();
        if (++stage == STAGES) { stage = 0; phase ^= 1; }
      }
      if (!ok) break;
      if (elect_one()) mma_commit(&tail->acc_full[acc]);
      __syncwarp();
      if (++acc == 2) { acc = 0; acc_phase ^= 1; }
    }
  } else {
    // ------------------------------ epilogue (warps 2..9) ------------------------------
    const int quad = warp & 3;           // TMEM lane quadrant this warp may read
    const int et = threadIdx.x - 64;     // 0 .. EPI_THREADS - 1
    const int c_first = ((warp - 2) >> 2) * (EPI_COLS / 32);
    int acc = 0;
    uint32_t acc_phase = 0;
    for (int tile = blockIdx.x; tile < num_tiles; tile += gridDim.x) {
      int m_blk, n_blk;
      tile_coords(tile, num_m, num_n, m_blk, n_blk);
      const int n0 = n_blk * TN;
      // stage the per-column scale (and bias / gate) of this tile in shared memory
      asm volatile("bar.sync 1, %0;" ::"n"(EPI_THREADS) : "memory");  // previous tile's readers are done
      for (int c = et; c < TN; c += EPI_THREADS) {
        const int n = n0 + c;
        tail->ws[c] = n < p.N ? p.ws[n] : 0.f;
        if (EPI == EPI_PLAIN || EPI == EPI_BIAS2) tail->aux[c] = (p.bias && n < p.N) ? __bfloat162float(p.bias[n]) : 0.f;
        if (EPI == EPI_F32 || EPI == EPI_F32_ADD) tail->aux[c] = (p.bias_f && n < p.N) ? p.bias_f[n] : -0.f;
        if (EPI == EPI_GATED2) {
          tail->aux[c] = n < p.N ? bf16_round(p.gate_f[0][n]) : 0.f;
          tail->aux2[c] = n < p.N ? bf16_round(p.gate_f[1][n]) : 0.f;
        }
        if (EPI == EPI_GATED) tail->aux[c] = n < p.N ? __bfloat162float(p.gate[n]) : 0.f;
        if (EPI == EPI_F16 || EPI == EPI_SWIGLU_F16) tail->aux[c] = n < p.N ? __half2float(p.bias_h[n]) : 0.f;
        if (EPI == EPI_F16) tail->aux2[c] = (p.rscale_h && n < p.N) ? __half2float(p.rscale_h[n]) : 0.f;
      }
      const int row = m_blk * BM + quad * 32 + lane;
      const bool row_ok = row < M;
      if (tile == static_cast<int>(blockIdx.x)) prefetch_residual<EPI, EPI_COLS>(p, row, row_ok, n0 + c_first * 32);
      if (tile + static_cast<int>(gridDim.x) < num_tiles) {   // the next tile's residual, a whole epilogue ahead
        int m2, n2;
        tile_coords(tile + gridDim.x, num_m, num_n, m2, n2);
        const int row2 = m2 * BM + quad * 32 + lane;
        prefetch_residual<EPI, EPI_COLS>(p, row2, row2 < M, n2 * TN + c_first * 32);
      }
      uint4 res0[4];
      if (is_gated(EPI)) load_gated_residual(p, row, row_ok, n0, c_first, res0);
      // the epilogue warps leave together: a warp that gave up its wait takes the others with it at this barrier
      // (which also publishes the staged columns), so none of them waits at the next tile's barrier alone
      const bool got = mbar_wait(&tail->acc_full[acc], acc_phase, abort_flag, p.status, ST_TIMEOUT_ACC_FULL);
      if (bar_sync_or(1, EPI_THREADS, !got)) break;
      tc_fence_after();
      const float xs = row_ok ? p.xs[row] : 0.f;
      const uint32_t t_row = tmem_base + acc * BN + (static_cast<uint32_t>(quad * 32) << 16);
      epilogue_row<KIND_F8, EPI, EPI_COLS>(p, tail, t_row, row, row_ok, xs, n0, c_first, res0);
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&tail->acc_empty[acc]);
      if (++acc == 2) { acc = 0; acc_phase ^= 1; }
    }
  }

  // ------------------------------ teardown ------------------------------
  __syncwarp();
  if (*abort_flag && threadIdx.x == 0) {
    // give copies that may still be in flight time to land before shared memory is released
    for (int i = 0; i < 64; ++i) __nanosleep(1000);
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base, 512);
  }
}

// ---------------------------------------------------------------------------------------------
// The same GEMM on CTA pairs (thread-block clusters of two, tcgen05 cta_group::2): a pair computes a tile of 256 rows x TN
// columns. CTA r of the pair loads A rows [128 r, 128 r + 128) and B rows (output columns) [TN/2 r, TN/2 r + TN/2) of the tile
// into its own shared memory (at TN = 256 32 KB per K slab instead of 48: what an SM has to take in per 512 tensor cycles is
// what bounds the single-CTA kernel), one thread of the even CTA issues MMAs of 256 x TN x 32 that read both CTAs'
// tiles, and each CTA's TMEM receives its 128 rows x TN columns, which its own epilogue warps drain as before.
// Barriers: the TMA loads of both CTAs count their bytes on the even CTA's `full`; stage release and accumulator
// hand-over are commits to the barrier of each CTA in turn (no multicast form anywhere); the epilogue warps of both
// CTAs arrive on the even CTA's `acc_empty`. Every wait is bounded as in the single-CTA kernel; the two cluster-wide
// barriers (after set-up, before tear-down) are reached by every thread on every path.
// ---------------------------------------------------------------------------------------------

struct __align__(8) PairSmemTail {
  uint64_t full[MAX_STAGES];
  uint64_t empty[MAX_STAGES];
  uint64_t acc_full[2];
  uint64_t acc_empty[2];
  uint32_t tmem_base;
  int abort_flag;
  GemmSmemTail cols;   // ws / aux / aux2 staging of the epilogue (its barrier fields are unused here)
};
constexpr int PAIR_SMEM_BYTES = RING_BYTES + sizeof(PairSmemTail) + 1024;

template <int KIND_F8, int EPI, int TN>   // TN: columns of a tile, half of whose B rows each CTA loads
__global__ void __launch_bounds__(GEMM_THREADS, 1)
gemm_pair_kernel(const __grid_constant__ CUtensorMap tma_a, const __grid_constant__ CUtensorMap tma_b,
                 const GemmParams p) {
  constexpr int KS = slabs_per_stage(TN, true), P_STAGES = ring_stages(TN / 2, KS), P_STAGE_BYTES = KS * slab_bytes(TN / 2), EPI_COLS = TN / (EPI_WARPS / 4);
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  PairSmemTail* tail = reinterpret_cast<PairSmemTail*>(smem + RING_BYTES);
  volatile int* abort_flag = &tail->abort_flag;

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t rank = cluster_cta_rank();          // 0 = the even CTA of the pair: it issues the MMAs
  const int pair = blockIdx.x >> 1, num_pairs = gridDim.x >> 1;
  if (EPI == EPI_F32_ADD) grid_dependency_wait();   // its row count is read on the device
  const int M = gemm_rows<EPI>(p);
  const int num_m = (M + 2 * BM - 1) / (2 * BM), num_n = (p.N + TN - 1) / TN;
  const int num_tiles = num_m * num_n;
  const int num_kb = (p.K + BK - 1) / BK;

  if (threadIdx.x == 0) {
    for (int s = 0; s < P_STAGES; ++s) {
      mbar_init(&tail->full[s], 1);     // the even CTA's: one arrive.expect_tx for the bytes of both CTAs
      mbar_init(&tail->empty[s], 1);    // one commit per CTA
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(&tail->acc_full[b], 1);
      mbar_init(&tail->acc_empty[b], 2 * EPI_WARPS);  // the even CTA's: one arrival per epilogue warp of both CTAs
    }
    tail->abort_flag = 0;
    fence_barrier_init();
  }
  if (warp == 1) {
    tmem_alloc_pair(&tail->tmem_base, 512);
    tmem_relinquish_pair();
  }
  tc_fence_before();
  __syncthreads();
  cluster_sync_all();   // both CTAs' barriers exist before anything arrives on them from the other side
  tc_fence_after();
  grid_dependency_trigger();
  if (EPI != EPI_F32_ADD) grid_dependency_wait();
  const uint32_t tmem_base = tail->tmem_base;

  if (warp == 0) {
    // ------------------------------ TMA producer (both CTAs) ------------------------------
    if (elect_one()) {
      tma_prefetch_desc(&tma_a);
      tma_prefetch_desc(&tma_b);
    }
    __syncwarp();
    int stage = 0;
    uint32_t phase = 0;
    bool ok = true;
    for (int tile = pair; tile < num_tiles && ok; tile += num_pairs) {
      int m_blk, n_blk;
      tile_coords(tile, num_m, num_n, m_blk, n_blk);
      const int row0 = m_blk * 2 * BM + static_cast<int>(rank) * BM, col0 = n_blk * TN + static_cast<int>(rank) * (TN / 2);
      for (int kb = 0; kb < num_kb; kb += KS) {
        ok = __all_sync(0xffffffffu, mbar_wait(&tail->empty[stage], phase ^ 1, abort_flag, p.status, ST_TIMEOUT_STAGE_EMPTY));
        if (!ok) break;
        uint8_t* sa = smem + stage * P_STAGE_BYTES;
        const uint32_t leader_full = cluster_addr(&tail->full[stage], 0);
        if (elect_one()) {
          if (rank == 0) mbar_arrive_expect_tx(&tail->full[stage], 2 * P_STAGE_BYTES);
#pragma unroll
          for (int q = 0; q < KS; ++q, sa += slab_bytes(TN / 2)) {
            tma_load_2d_pair(sa, &tma_a, (kb + q) * BK, row0, leader_full);
            tma_load_2d_pair(sa + A_BYTES, &tma_b, (kb + q) * BK, col0, leader_full);
          }
        }
        __syncwarp();
        if (++stage == P_STAGES) { stage = 0; phase ^= 1; }
      }
    }
  } else if (warp == 1) {
    // ------------------------------ MMA issuer (even CTA only; converged warp, one elected lane) ------------------------------
    if (rank == 0) {
      constexpr uint32_t idesc = KIND_F8 ? make_idesc(1, 0, 0, 2 * BM, TN) : make_idesc(2, 1, 1, 2 * BM, TN);
      int stage = 0;
      uint32_t phase = 0;
      int acc = 0;
      uint32_t acc_phase = 0;
      bool ok = true;
      for (int tile = pair; tile < num_tiles && ok; tile += num_pairs) {
        ok = __all_sync(0xffffffffu, mbar_wait(&tail->acc_empty[acc], acc_phase ^ 1, abort_flag, p.status, ST_TIMEOUT_ACC_EMPTY));
        if (!ok) break;
        tc_fence_after();
        const uint32_t d_tmem = tmem_base + acc * BN;
        for (int kb = 0; kb < num_kb; kb += KS) {
          ok = __all_sync(0xffffffffu, mbar_wait(&tail->full[stage], phase, abort_flag, p.status, ST_TIMEOUT_TMA_FULL));
          if (!ok) break;
          tc_fence_after();
          const uint32_t a_addr = smem_u32(smem + stage * P_STAGE_BYTES);
          const uint32_t empty0 = cluster_addr(&tail->empty[stage], 0), empty1 = cluster_addr(&tail->empty[stage], 1);
          if (elect_one()) {
#pragma unroll
            for (int q = 0; q < KS; ++q) {
              const uint32_t aq = a_addr + q * slab_bytes(TN / 2);
              if (KIND_F8) mma4_f8_pair(d_tmem, make_desc_k128(aq), make_desc_k128(aq + A_BYTES), idesc, (kb + q) != 0);
              else mma4_i8_pair(d_tmem, make_desc_k128(aq), make_desc_k128(aq + A_BYTES), idesc, (kb + q) != 0);
            }
            mma_commit_pair(empty0);   // the stage is free in both CTAs once these MMAs have read it
            mma_commit_pair(empty1);
          }
          __syncwarp();
          if (++stage == P_STAGES) { stage = 0; phase ^= 1; }
        }
        if (!ok) break;
        const uint32_t full0 = cluster_addr(&tail->acc_full[acc], 0), full1 = cluster_addr(&tail->acc_full[acc], 1);
        if (elect_one()) {
          mma_commit_pair(full0);
          mma_commit_pair(full1);
        }
        __syncwarp();
        if (++acc == 2) { acc = 0; acc_phase ^= 1; }
      }
    }
  } else {
    // ------------------------------ epilogue (warps 2..9 of both CTAs) ------------------------------
    const int quad = warp & 3;
    const int et = threadIdx.x - 64;
    const int c_first = ((warp - 2) >> 2) * (EPI_COLS / 32);
    GemmSmemTail* cols = &tail->cols;
    int acc = 0;
    uint32_t acc_phase = 0;
    for (int tile = pair; tile < num_tiles; tile += num_pairs) {
      int m_blk, n_blk;
      tile_coords(tile, num_m, num_n, m_blk, n_blk);
      const int n0 = n_blk * TN;
      asm volatile("bar.sync 1, %0;" ::"n"(EPI_THREADS) : "memory");  // previous tile's readers are done
      for (int c = et; c < TN; c += EPI_THREADS) {
        const int n = n0 + c;
        cols->ws[c] = n < p.N ? p.ws[n] : 0.f;
        if (EPI == EPI_PLAIN || EPI == EPI_BIAS2) cols->aux[c] = (p.bias && n < p.N) ? __bfloat162float(p.bias[n]) : 0.f;
        if (EPI == EPI_F32 || EPI == EPI_F32_ADD) cols->aux[c] = (p.bias_f && n < p.N) ? p.bias_f[n] : -0.f;
        if (EPI == EPI_GATED2) {
          cols->aux[c] = n < p.N ? bf16_round(p.gate_f[0][n]) : 0.f;
          cols->aux2[c] = n < p.N ? bf16_round(p.gate_f[1][n]) : 0.f;
        }
        if (EPI == EPI_GATED) cols->aux[c] = n < p.N ? __bfloat162float(p.gate[n]) : 0.f;
        if (EPI == EPI_F16 || EPI == EPI_SWIGLU_F16) cols->aux[c] = n < p.N ? __half2float(p.bias_h[n]) : 0.f;
        if (EPI == EPI_F16) cols->aux2[c] = (p.rscale_h && n < p.N) ? __half2float(p.rscale_h[n]) : 0.f;
      }
      const int row = m_blk * 2 * BM + static_cast<int>(rank) * BM + quad * 32 + lane;
      const bool row_ok = row < M;
      if (tile == pair) prefetch_residual<EPI, EPI_COLS>(p, row, row_ok, n0 + c_first * 32);
      if (tile + num_pairs < num_tiles) {   // the next tile's residual, a whole epilogue ahead
        int m2, n2;
        tile_coords(tile + num_pairs, num_m, num_n, m2, n2);
        const int row2 = m2 * 2 * BM + static_cast<int>(rank) * BM + quad * 32 + lane;
        prefetch_residual<EPI, EPI_COLS>(p, row2, row2 < M, n2 * TN + c_first * 32);
      }
      uint4 res0[4];
      if (is_gated(EPI)) load_gated_residual(p, row, row_ok, n0, c_first, res0);
      const bool got = mbar_wait(&tail->acc_full[acc], acc_phase, abort_flag, p.status, ST_TIMEOUT_ACC_FULL);
      if (bar_sync_or(1, EPI_THREADS, !got)) break;
      tc_fence_after();
      const float xs = row_ok ? p.xs[row] : 0.f;
      const uint32_t t_row = tmem_base + acc * BN + (static_cast<uint32_t>(quad * 32) << 16);
      epilogue_row<KIND_F8, EPI, EPI_COLS>(p, cols, t_row, row, row_ok, xs, n0, c_first, res0);
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive_remote(&tail->acc_empty[acc], 0);
      if (++acc == 2) { acc = 0; acc_phase ^= 1; }
    }
  }

  // ------------------------------ teardown ------------------------------
  __syncwarp();
  if (*abort_flag && threadIdx.x == 0) {
    for (int i = 0; i < 64; ++i) __nanosleep(1000);
  }
  tc_fence_before();
  __syncthreads();
  cluster_sync_all();   // nothing of the other CTA is in flight towards this CTA's shared memory or barriers any more
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc_pair(tmem_base, 512);
  }
}

std::atomic<int> g_use_pairs{1};

// Rows of A per load: a multiple of the swizzle's eight. Rows past the end of A are not free: a box that asks for 128 rows of a
// 16 x 4,096 operand took 15 us on 64 CTAs where one of 16 rows takes 10.9.
int box_rows(int64_t M) { return M < BM ? static_cast<int>((M + 7) / 8 * 8) : BM; }

// the tensor map of a call's activations, and what the one of its weights is made from once the tile is chosen
struct GemmMaps {
  CUtensorMap a;
  const void* wq;
  int64_t N, K;
  int weights(CUtensorMap* b, int rows) const {
    return make_tmap_2d(b, CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, wq, K, N, K, BK, rows, CU_TENSOR_MAP_SWIZZLE_128B);
  }
};

template <int KIND_F8, int EPI, int TN>
int launch_gemm_pair(const CUtensorMap& ta, const CUtensorMap& tb, const GemmParams& p, cudaStream_t stream) {
  auto kern = gemm_pair_kernel<KIND_F8, EPI, TN>;
  if (int e = check_cuda(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, PAIR_SMEM_BYTES),
                         "gemm pair smem attribute"))
    return e;
  const int num_tiles = ((p.M + 2 * BM - 1) / (2 * BM)) * ((p.N + TN - 1) / TN);
  // as many pairs as can be resident at once (one CTA per SM), never more than there are tiles
  cudaLaunchConfig_t cfg{};
  cudaLaunchAttribute attr{};
  attr.id = cudaLaunchAttributeClusterDimension;
  attr.val.clusterDim.x = 2;
  attr.val.clusterDim.y = 1;
  attr.val.clusterDim.z = 1;
  cfg.gridDim = dim3(2 * (device_sm_count() / 2));
  cfg.blockDim = dim3(GEMM_THREADS);
  cfg.dynamicSmemBytes = PAIR_SMEM_BYTES;
  cfg.stream = stream;
  cfg.attrs = &attr;
  cfg.numAttrs = 1;
  int max_clusters = 0;
  if (cudaOccupancyMaxActiveClusters(&max_clusters, kern, &cfg) != cudaSuccess || max_clusters < 1)
    return set_error(RH3_ARG_ERROR, "gemm pair: no cluster of two CTAs can be resident");
  const int pairs = num_tiles < max_clusters ? num_tiles : max_clusters;
  return check_cuda(launch_chained(kern, dim3(2 * pairs), GEMM_THREADS, PAIR_SMEM_BYTES, stream, 2, ta, tb, p), "gemm pair launch");
}

template <int KIND_F8, int EPI, int TN>
int launch_gemm_single(const CUtensorMap& ta, const CUtensorMap& tb, const GemmParams& p, cudaStream_t stream) {
  auto kern = gemm_w8a8_kernel<KIND_F8, EPI, TN>;
  if (int e = check_cuda(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, GEMM_SMEM_BYTES),
                         "gemm smem attribute"))
    return e;
  const int num_tiles = ((p.M + BM - 1) / BM) * ((p.N + TN - 1) / TN);
  const int grid = num_tiles < device_sm_count() ? num_tiles : device_sm_count();
  return check_cuda(launch_chained(kern, dim3(grid), GEMM_THREADS, GEMM_SMEM_BYTES, stream, 1, ta, tb, p), "gemm launch");
}

// Columns of a tile. A K slab of a tile takes as long as the SM needs to take its operands in or the tensor pipe to multiply them; a
// narrower tile loads the same A rows for fewer columns, so it pays where the full width leaves SMs idle in its only or its last
// wave: the width with the smallest waves x time of a slab. `tile_rows` by `ctas` CTAs that share a tile (each loads its rows of A and
// its part of B). The 72 bytes per clock are the model's, no measured rate (a ring filled by bulk copies alone, with all SMs at it,
// reaches 61): what they are held against is every fixed width at six N x K and fifteen M from 1 to 17,896, where the rule is
// within 8 % of the best one. Time at 256 columns for everything / now, us: N = K = 4,096: 37 rows 13.2 / 7.5,
// 200 rows 15.6 / 8.4, 512 rows 15.9 / 10.3, 1,500 rows 25.3 / 20.9; N = 4,096, K = 16,384: 37 rows 43 / 25, 512 rows 42 / 29;
// N = 12,288, K = 4,096: 37 rows 13.4 / 10.0, 512 rows 25.4 / 21.2.
int tile_columns(long long M, long long N, long long K, int tile_rows, int ctas) {
  const long long resident = device_sm_count() / ctas, m_tiles = (M + tile_rows - 1) / tile_rows;
  const long long kb = (K + BK - 1) / BK;
  long long best = 0;
  int width = 0;
  for (int tn = BN; tn >= 64; tn >>= 1) {
    const long long waves = (m_tiles * ((N + tn - 1) / tn) + resident - 1) / resident;
    const long long feed = BK * (box_rows(M) + tn / ctas) / 72, mma = 2 * tn + 50;
    const long long cost = waves * kb * (feed > mma ? feed : mma) + 8 * tn;   // + draining the last accumulator
    if (!width || cost < best) {
      best = cost;
      width = tn;
    }
  }
  return width;
}

// pairs need more than one 128-row tile to be worth their 256-row tiles
bool on_pairs(int64_t M, int64_t N) { return g_use_pairs.load(std::memory_order_relaxed) && M > BM && N > 128; }

template <int KIND_F8, int EPI>
int launch_gemm(const GemmMaps& maps, GemmParams p, cudaStream_t stream) {
  CUtensorMap tb;
  p.a_rows = box_rows(p.M);
  if (on_pairs(p.M, p.N)) {
    const int tn = tile_columns(p.M, p.N, p.K, 2 * BM, 2);
    if (int e = maps.weights(&tb, tn / 2)) return e;   // a CTA loads half of a tile's B rows
    return tn == 256   ? launch_gemm_pair<KIND_F8, EPI, 256>(maps.a, tb, p, stream)
           : tn == 128 ? launch_gemm_pair<KIND_F8, EPI, 128>(maps.a, tb, p, stream)
                       : launch_gemm_pair<KIND_F8, EPI, 64>(maps.a, tb, p, stream);
  }
  const int tn = tile_columns(p.M, p.N, p.K, BM, 1);
  if (int e = maps.weights(&tb, tn)) return e;
  return tn == 256   ? launch_gemm_single<KIND_F8, EPI, 256>(maps.a, tb, p, stream)
         : tn == 128 ? launch_gemm_single<KIND_F8, EPI, 128>(maps.a, tb, p, stream)
                     : launch_gemm_single<KIND_F8, EPI, 64>(maps.a, tb, p, stream);
}

int gemm_common(const void* xq, int64_t lda, const void* wq, const float* xs, const float* ws, int64_t M, int64_t N,
                int64_t K, int kind, GemmMaps* maps) {
  RH3_CHECK_ARG(kind == RH3_KIND_I8 || kind == RH3_KIND_F8, "gemm_w8a8: kind must be RH3_KIND_I8 or RH3_KIND_F8");
  RH3_CHECK_ARG(M >= 0 && N > 0 && K > 0 && M < (1ll << 31) && N < (1ll << 31) && K < (1ll << 31),
                "gemm_w8a8: bad shape M=%lld N=%lld K=%lld", (long long)M, (long long)N, (long long)K);
  RH3_CHECK_ARG(K % 16 == 0, "gemm_w8a8: K=%lld must be a multiple of 16", (long long)K);
  RH3_CHECK_ARG(N % 8 == 0, "gemm_w8a8: N=%lld must be a multiple of 8", (long long)N);
  RH3_CHECK_ARG(lda >= K && lda % 16 == 0, "gemm_w8a8: xq row stride must be >= K and a multiple of 16");
  if (M == 0) return 0;
  RH3_CHECK_ARG(xq && wq && xs && ws, "gemm_w8a8: null pointer");
  RH3_CHECK_ARG((reinterpret_cast<uintptr_t>(xq) & 15) == 0 && (reinterpret_cast<uintptr_t>(wq) & 15) == 0,
                "gemm_w8a8: xq and wq must be 16-byte aligned");
  maps->wq = wq, maps->N = N, maps->K = K;
  return make_tmap_2d(&maps->a, CU_TENSOR_MAP_DATA_TYPE_UINT8, 1, xq, K, M, lda, BK, box_rows(M), CU_TENSOR_MAP_SWIZZLE_128B);
}

}  // namespace
int pairs_enabled() { return g_use_pairs.load(std::memory_order_relaxed); }
}  // namespace rh3

using namespace rh3;

// Selects the kernel the GEMM entries launch: 0 = one CTA per tile of 128 rows, 1 (default) = CTA pairs on tiles of 256
// rows (gemm_pair_kernel) for every call with more than 128 rows and more than 128 columns. Returns the previous
// setting. Results are identical (int32 accumulators, same epilogue). The convolution follows the same switch
// (conv3d_pair_kernel: fp32 accumulation in the same order, identical results).
extern "C" int rh3_gemm_use_pairs(int on) { return g_use_pairs.exchange(on ? 1 : 0); }

extern "C" int rh3_gemm_tile(int64_t M, int64_t N, int64_t K, int64_t* rows, int64_t* columns) {
  RH3_CHECK_ARG(rows && columns && M > 0 && N > 0 && K > 0 && M < (1ll << 31) && N < (1ll << 31) && K < (1ll << 31),
                "gemm_tile: bad shape or null pointer");
  const bool pair = on_pairs(M, N);
  *rows = pair ? 2 * BM : BM;
  *columns = tile_columns(M, N, K, pair ? 2 * BM : BM, pair ? 2 : 1);
  return 0;
}

extern "C" int rh3_gemm_w8a8(const void* xq, int64_t lda, const void* wq, const float* xs, const float* ws,
                             const void* bias, int64_t M, int64_t N, int64_t K, int kind, void* out, int64_t ldo,
                             int32_t* acc_dump, cudaStream_t stream) {
  GemmMaps maps;
  if (int e = gemm_common(xq, lda, wq, xs, ws, M, N, K, kind, &maps)) return e;
  if (M == 0) return 0;
  RH3_CHECK_ARG(out && ldo >= N && ldo % 8 == 0 && (reinterpret_cast<uintptr_t>(out) & 15) == 0,
                "gemm_w8a8: out must be 16-byte aligned with a row stride >= N that is a multiple of 8");
  RH3_CHECK_ARG(!acc_dump || (reinterpret_cast<uintptr_t>(acc_dump) & 15) == 0, "gemm_w8a8: acc_dump misaligned");
  GemmParams p{};
  p.M = (int)M; p.N = (int)N; p.K = (int)K; p.xs = xs; p.ws = ws;
  p.bias = static_cast<const __nv_bfloat16*>(bias);
  p.out = static_cast<__nv_bfloat16*>(out); p.ldo = ldo; p.acc_dump = acc_dump; p.status = device_status_word();
  p.wide = (reinterpret_cast<uintptr_t>(out) & 31) == 0 && ldo % 16 == 0;
  return kind == RH3_KIND_F8 ? launch_gemm<1, EPI_PLAIN>(maps, p, stream) : launch_gemm<0, EPI_PLAIN>(maps, p, stream);
}

// The bias lands on the rounded product (two roundings), so the result is bit for bit that of rh3_gemm_w8a8 without a
// bias followed by a bf16 addition; what it saves is that addition's pass over the output (read and written once more;
// the host framework's broadcast kernel took 138 us for 5,003 x 12,288 beside 164 us for the GEMM itself).
extern "C" int rh3_gemm_w8a8_bias_after(const void* xq, int64_t lda, const void* wq, const float* xs, const float* ws,
                                        const void* bias, int64_t M, int64_t N, int64_t K, int kind, void* out,
                                        int64_t ldo, cudaStream_t stream) {
  GemmMaps maps;
  if (int e = gemm_common(xq, lda, wq, xs, ws, M, N, K, kind, &maps)) return e;
  if (M == 0) return 0;
  RH3_CHECK_ARG(bias, "gemm_w8a8_bias_after: bias is required");
  RH3_CHECK_ARG(out && ldo >= N && ldo % 8 == 0 && (reinterpret_cast<uintptr_t>(out) & 15) == 0,
                "gemm_w8a8_bias_after: out must be 16-byte aligned with a row stride >= N that is a multiple of 8");
  GemmParams p{};
  p.M = (int)M; p.N = (int)N; p.K = (int)K; p.xs = xs; p.ws = ws;
  p.bias = static_cast<const __nv_bfloat16*>(bias);
  p.out = static_cast<__nv_bfloat16*>(out); p.ldo = ldo; p.status = device_status_word();
  p.wide = (reinterpret_cast<uintptr_t>(out) & 31) == 0 && ldo % 16 == 0;
  return kind == RH3_KIND_F8 ? launch_gemm<1, EPI_BIAS2>(maps, p, stream) : launch_gemm<0, EPI_BIAS2>(maps, p, stream);
}

extern "C" int rh3_gemm_w8a8_gated_residual(const void* xq, int64_t lda, const void* wq, const float* xs,
                                            const float* ws, const void* gate, void* resid, int64_t ldr, int64_t M,
                                            int64_t N, int64_t K, int kind, cudaStream_t stream) {
  GemmMaps maps;
  if (int e = gemm_common(xq, lda, wq, xs, ws, M, N, K, kind, &maps)) return e;
  if (M == 0) return 0;
  RH3_CHECK_ARG(gate && resid && ldr >= N && ldr % 8 == 0 && (reinterpret_cast<uintptr_t>(resid) & 15) == 0,
                "gemm_w8a8_gated_residual: resid must be 16-byte aligned with a row stride >= N, multiple of 8");
  GemmParams p{};
  p.M = (int)M; p.N = (int)N; p.K = (int)K; p.xs = xs; p.ws = ws;
  p.gate = static_cast<const __nv_bfloat16*>(gate);
  p.resid = static_cast<__nv_bfloat16*>(resid); p.ldr = ldr; p.status = device_status_word();
  p.wide = (reinterpret_cast<uintptr_t>(resid) & 31) == 0 && ldr % 16 == 0;
  return kind == RH3_KIND_F8 ? launch_gemm<1, EPI_GATED>(maps, p, stream) : launch_gemm<0, EPI_GATED>(maps, p, stream);
}

// The gated residual over a packed sequence of two modalities in one launch: a launch per modality ran the 148 audio rows
// through the whole K loop on 32 SMs (20 us at K = 4,096, 54 us at K = 16,384) and needed the gate table converted first.
extern "C" int rh3_gemm_w8a8_gated_residual2(const void* xq, int64_t lda, const void* wq, const float* xs, const float* ws,
                                             const float* gate0, const float* gate1, int64_t split, void* resid,
                                             int64_t ldr, int64_t M, int64_t N, int64_t K, int kind, cudaStream_t stream) {
  GemmMaps maps;
  if (int e = gemm_common(xq, lda, wq, xs, ws, M, N, K, kind, &maps)) return e;
  if (M == 0) return 0;
  RH3_CHECK_ARG(gate0 && gate1 && split >= 0, "gemm_w8a8_gated_residual2: two gate rows and a split >= 0 are required");
  RH3_CHECK_ARG(resid && ldr >= N && ldr % 8 == 0 && (reinterpret_cast<uintptr_t>(resid) & 15) == 0,
                "gemm_w8a8_gated_residual2: resid must be 16-byte aligned with a row stride >= N, multiple of 8");
  GemmParams p{};
  p.M = (int)M; p.N = (int)N; p.K = (int)K; p.xs = xs; p.ws = ws;
  p.gate_f[0] = gate0; p.gate_f[1] = gate1; p.gate_split = (int)(split < M ? split : M);
  p.resid = static_cast<__nv_bfloat16*>(resid); p.ldr = ldr; p.status = device_status_word();
  p.wide = (reinterpret_cast<uintptr_t>(resid) & 31) == 0 && ldr % 16 == 0;
  return kind == RH3_KIND_F8 ? launch_gemm<1, EPI_GATED2>(maps, p, stream) : launch_gemm<0, EPI_GATED2>(maps, p, stream);
}

extern "C" int rh3_gemm_w8a8_swiglu(const void* xq, int64_t lda, const void* wq, const float* xs, const float* ws,
                                    int64_t M, int64_t N, int64_t K, int kind, void* out, int64_t ldo,
                                    cudaStream_t stream) {
  GemmMaps maps;
  if (int e = gemm_common(xq, lda, wq, xs, ws, M, N, K, kind, &maps)) return e;
  RH3_CHECK_ARG(N % 16 == 0, "gemm_w8a8_swiglu: N=%lld must be a multiple of 16", (long long)N);
  if (M == 0) return 0;
  RH3_CHECK_ARG(out && ldo >= N / 2 && ldo % 8 == 0 && (reinterpret_cast<uintptr_t>(out) & 15) == 0,
                "gemm_w8a8_swiglu: out must be 16-byte aligned with a row stride >= N/2 that is a multiple of 8");
  GemmParams p{};
  p.M = (int)M; p.N = (int)N; p.K = (int)K; p.xs = xs; p.ws = ws;
  p.out = static_cast<__nv_bfloat16*>(out); p.ldo = ldo; p.status = device_status_word();
  p.wide = (reinterpret_cast<uintptr_t>(out) & 31) == 0 && ldo % 16 == 0;
  return kind == RH3_KIND_F8 ? launch_gemm<1, EPI_SWIGLU>(maps, p, stream) : launch_gemm<0, EPI_SWIGLU>(maps, p, stream);
}

// ---- fp32 epilogues: the text encoder's linears (fp32 in and out, custom_nodes/rapid_h3/te_quant.py:90-115) ----
// First product: out = float(bf16(y)) + bias, the bias left out of the rows that `flags` marks. Second product over the
// rows in `rows` (their number is *count, at most M): out[rows[m]] = (out[rows[m]] + float(bf16(y2))) + bias. One call
// launches both; without `rows` only the first.
extern "C" int rh3_te_gemm(const void* q1, const float* s1, const void* wq, const float* ws, const float* bias, int64_t M,
                           int64_t N, int64_t K, const void* flags, const int32_t* count, const int32_t* rows,
                           const void* q2, const float* s2, float* out, int64_t ldo, cudaStream_t stream) {
  GemmMaps maps;
  if (int e = gemm_common(q1, K, wq, s1, ws, M, N, K, RH3_KIND_I8, &maps)) return e;
  if (M == 0) return 0;
  RH3_CHECK_ARG(out && ldo >= N && ldo % 8 == 0 && (reinterpret_cast<uintptr_t>(out) & 31) == 0,
                "te_gemm: out must be 32-byte aligned with a row stride >= N that is a multiple of 8");
  RH3_CHECK_ARG(!rows || (count && q2 && s2 && flags), "te_gemm: the second product needs its count, codes, scales and flags");
  GemmParams p{};
  p.M = (int)M; p.N = (int)N; p.K = (int)K; p.xs = s1; p.ws = ws; p.bias_f = bias;
  p.out_f = out; p.ldo = ldo; p.status = device_status_word();
  p.flags = rows ? static_cast<const uint8_t*>(flags) : nullptr;
  if (int e = launch_gemm<0, EPI_F32>(maps, p, stream)) return e;
  if (!rows) return 0;
  if (int e = gemm_common(q2, K, wq, s2, ws, M, N, K, RH3_KIND_I8, &maps)) return e;
  p.xs = s2; p.flags = nullptr; p.rows = rows; p.m_dev = count;
  return launch_gemm<0, EPI_F32_ADD>(maps, p, stream);
}

// ---- fp16 epilogues: the reference's VAE transformer-decoder GEMMs (custom_nodes/rapid_h3/csrc/vae_ops.cu:150-227
// plain + bias and residual addcmul, :228-345 w1 + SwiGLU) ----
extern "C" int rh3_vae_gemm(const void* xq, int64_t lda, const void* wq, const float* xs, const float* ws,
                            const void* bias_f16, const void* rscale_f16, const void* resid_f16, int64_t ldr,
                            int64_t M, int64_t N, int64_t K, void* out_f16, int64_t ldo, cudaStream_t stream) {
  GemmMaps maps;
  if (int e = gemm_common(xq, lda, wq, xs, ws, M, N, K, RH3_KIND_I8, &maps)) return e;
  if (M == 0) return 0;
  RH3_CHECK_ARG(bias_f16, "vae_gemm: bias is required (pass zeros for none)");
  RH3_CHECK_ARG(out_f16 && ldo >= N && ldo % 8 == 0 && (reinterpret_cast<uintptr_t>(out_f16) & 15) == 0,
                "vae_gemm: out must be 16-byte aligned with a row stride >= N that is a multiple of 8");
  RH3_CHECK_ARG((rscale_f16 == nullptr) == (resid_f16 == nullptr), "vae_gemm: rscale and resid come together");
  RH3_CHECK_ARG(!resid_f16 || (ldr >= N && ldr % 8 == 0 && (reinterpret_cast<uintptr_t>(resid_f16) & 15) == 0),
                "vae_gemm: resid must be 16-byte aligned with a row stride >= N that is a multiple of 8");
  GemmParams p{};
  p.M = (int)M; p.N = (int)N; p.K = (int)K; p.xs = xs; p.ws = ws;
  p.bias_h = static_cast<const __half*>(bias_f16); p.rscale_h = static_cast<const __half*>(rscale_f16);
  p.resid_h = static_cast<const __half*>(resid_f16); p.ldr = ldr;
  p.out_h = static_cast<__half*>(out_f16); p.ldo = ldo; p.status = device_status_word();
  return launch_gemm<0, EPI_F16>(maps, p, stream);
}

extern "C" int rh3_vae_gemm_swiglu(const void* xq, int64_t lda, const void* wq, const float* xs, const float* ws,
                                   const void* bias_f16, int64_t M, int64_t N, int64_t K, void* out_f16, int64_t ldo,
                                   cudaStream_t stream) {
  GemmMaps maps;
  if (int e = gemm_common(xq, lda, wq, xs, ws, M, N, K, RH3_KIND_I8, &maps)) return e;
  RH3_CHECK_ARG(N % 16 == 0, "vae_gemm_swiglu: N=%lld must be a multiple of 16", (long long)N);
  if (M == 0) return 0;
  RH3_CHECK_ARG(bias_f16, "vae_gemm_swiglu: bias is required (pass zeros for none)");
  RH3_CHECK_ARG(out_f16 && ldo >= N / 2 && ldo % 8 == 0 && (reinterpret_cast<uintptr_t>(out_f16) & 15) == 0,
                "vae_gemm_swiglu: out must be 16-byte aligned with a row stride >= N/2 that is a multiple of 8");
  GemmParams p{};
  p.M = (int)M; p.N = (int)N; p.K = (int)K; p.xs = xs; p.ws = ws;
  p.bias_h = static_cast<const __half*>(bias_f16);
  p.out_h = static_cast<__half*>(out_f16); p.ldo = ldo; p.status = device_status_word();
  return launch_gemm<0, EPI_SWIGLU_F16>(maps, p, stream);
}

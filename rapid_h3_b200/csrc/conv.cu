// Causal 3x3x3 convolution of the VAE decoder as an implicit GEMM on the Blackwell tensor cores, plus
// the GroupNorm + SiLU kernels that sit between convolutions.
//
//   x   [N, T, H, W, Cin]  bf16 channels-last          w [Cout, 27, Cin] bf16 (tap = (dt*3 + dh)*3 + dw)
//   out [N, T, H, W, Cout] bf16 = bf16( sum_{tap, ci} x[n, t+dt-2, h+dh-1, w+dw-1, ci] * w[co, tap, ci]
//                                      + bias[co] (+ residual[n, t, h, w, co]) )
//   zero padding: one pixel around H and W, two frames BEFORE t = 0 (causal: no frame after t is read).
//
// There is no im2col buffer: the A operand of the GEMM is a shifted box of the input, fetched by a 5-D TMA tensor copy
// whose out-of-range coordinates are filled with zeros (that is the padding): a box per tap in the single-CTA kernel, one
// box for the three dh of a (dt, dw) in the pair kernel. The K loop runs over (dt, dw, 64 channels, dh) in both, so their
// results agree bit for bit; with the order (dt, dh, dw, channels) of a plain tap loop the same fp32 sums round differently
// (whole decodes differ by 6.4e-3 to 7.8e-3 relative), equally far from the exact ones: over 93 M outputs of 13 layer shapes
// 0.2636 % against 0.2632 % are not the rounded 64-bit value, and decodes lie 7.524e-3 and 7.527e-3 from one in 64 bits.
// One output tile = bh x bw sites of one frame (bh * bw <= 128 rows of the MMA) x BN output
// channels; a K chunk is 64 channels of a tap (64 bf16 = one 128-byte swizzled row).
// Same warp roles and double-buffered TMEM accumulators as the W8A8 GEMM; the ring has as many stages as fit in
// shared memory (4 of 48 KB at 256 output channels per tile, up to 12 for narrow tiles): a stage of a narrow tile
// holds few tensor cycles of work, and the ring has to cover the L2 latency with them.
// The epilogue also emits per-tile partial sums (sum, sum of squares of the rounded outputs) per
// GroupNorm group, so the statistics of the next GroupNorm cost no extra pass over the activations.
//
// No counterpart exists in the reference repository (its VAE fast path is a transformer decoder,
// custom_nodes/rapid_h3/vae_fast.py:430-437); the CPU oracle (oracle/vae.py) defines the arithmetic.
// Tensor-core bound: 2 * sites * Cout * Cin * 27 operations per call.
#include "common.cuh"
#include "rapidh3_b200.h"

namespace rh3 {
namespace {

constexpr int CBM = 128;        // MMA rows (output sites per tile, bh * bw of them used)
constexpr int CBK = 64;         // channels per K chunk (128 bytes of bf16)
constexpr int CA_BYTES = CBM * 128;
constexpr int CMAX_STAGES = 12;       // ring depth: as many stages of CA_BYTES + (weight rows) * 128 bytes as fit
constexpr int CTAIL_BYTES = 2048;     // barriers and the staged bias, in front of the ring
constexpr int CRING_MAX_BYTES = 227 * 1024 - 1024 - CTAIL_BYTES;   // what the ring may take (1 KB of alignment slack)
constexpr int CONV_THREADS = 192;
constexpr int GN_GROUPS = 32;

struct ConvParams {
  int N, T, H, W, Cin, Cout;
  int halo;            // frames that precede output frame 0 inside x (0: causal zero padding, 2: a time shard's halo)
  int bh, bw;          // tile of output sites inside a frame
  int tiles_h, tiles_w;
  int BN;              // output channels per tile (multiple of 16, <= 256)
  const __nv_bfloat16* bias;      // [Cout] or null
  const __nv_bfloat16* residual;  // [N,T,H,W,Cout] or null
  __nv_bfloat16* out;
  float* gn_part;      // [num_m_tiles * 4][32][2] partial (sum, sumsq) per GroupNorm group, or null
  int stages, stage_bytes;   // ring
  int wide;                  // out (and residual) rows are 32-byte aligned: 32-byte accesses in the epilogue
  // single CTA: K chunks per stage (one barrier round trip each) of CA_BYTES + BN * 128 bytes. Pair: a stage is the box, of
  // chunk_bytes, and the weight rows of its three taps
  int kch, chunk_bytes;
  int* status;
};

struct __align__(8) ConvSmemTail {
  uint64_t full[CMAX_STAGES];
  uint64_t empty[CMAX_STAGES];
  uint64_t acc_full[2];
  uint64_t acc_empty[2];
  uint32_t tmem_base;
  int abort_flag;
  float bias[256];
};

static_assert(sizeof(ConvSmemTail) <= CTAIL_BYTES, "tail does not fit");

struct TileCoord {
  int n, t, h0, w0, n_blk;
};

__device__ __forceinline__ TileCoord conv_tile(int tile, const ConvParams& p, int num_n) {
  // column tiles fastest: the CTAs running together share the same input boxes through L2
  TileCoord c;
  c.n_blk = tile % num_n;
  int m = tile / num_n;
  c.w0 = (m % p.tiles_w) * p.bw;
  m /= p.tiles_w;
  c.h0 = (m % p.tiles_h) * p.bh;
  m /= p.tiles_h;
  c.t = m % p.T;
  c.n = m / p.T;
  return c;
}

// Sums over the 32 lanes of the REST values v[0..REST) each of them holds, by exchanges with the lanes O, O / 2, ... 1 away. As
// long as a lane holds more than one value it hands half of them over and keeps the other half (`at`: index of v[0] among all
// values); from then on both lanes of an exchange hold the same single value. REST and O are template parameters so that every
// index into v[] is static: with a run-time count in one unrolled loop the array went to local memory (256 bytes of stack in all
// four convolution kernels).
template <int REST, int O, int NV>
__device__ __forceinline__ void gn_exchange(float (&v)[NV], int lane, int& at) {
  if constexpr (O > 0) {
    const bool upper = lane & O;
    if constexpr (REST > 1) {
#pragma unroll
      for (int i = 0; i < REST / 2; ++i) {
        const float send = upper ? v[i] : v[i + REST / 2], keep = upper ? v[i + REST / 2] : v[i];
        v[i] = keep + __shfl_xor_sync(0xffffffffu, send, O);
      }
      if (upper) at += REST / 2;
      gn_exchange<REST / 2, O / 2>(v, lane, at);
    } else {
      v[0] += __shfl_xor_sync(0xffffffffu, v[0], O);
      gn_exchange<1, O / 2>(v, lane, at);
    }
  }
}

// GroupNorm partials of a warp's 32 rows over one 32-column chunk: the GS channels of a group are summed per row
// (in channel order), the 32 rows by gn_exchange; (sum, sum of squares) of every group the chunk holds are written. The
// exchanges take 16 shuffles for the 16 values of 4-channel groups where a butterfly of 5 for each takes 80, which made
// this epilogue longer than the 54 K chunks of a 128-channel tile: 9 x 48 x 84 sites 32.6 us a layer, 28.8
// with the exchanges, 27.5 with their values in registers. Every sum has the same operands in the same order either way.
template <int GS>
__device__ __forceinline__ void gn_partials_chunk(const float* y, float* part, int col0, int Cout, int lane) {
  constexpr int NV = 2 * (32 / GS);   // values: (sum, sum of squares) of each group
  float v[NV];
#pragma unroll
  for (int q = 0; q < 32 / GS; ++q) {
    float s1 = 0.f, s2 = 0.f;
#pragma unroll
    for (int j = q * GS; j < (q + 1) * GS; ++j) {
      s1 += y[j];
      s2 += y[j] * y[j];
    }
    v[2 * q] = s1;
    v[2 * q + 1] = s2;
  }
  int at = 0;
  gn_exchange<NV, 16>(v, lane, at);
  constexpr int HELD = NV > 32 ? NV / 32 : 1, COPIES = NV > 32 ? 1 : 32 / NV;   // values a lane ends with, lanes that end with the same one
  if ((lane & (COPIES - 1)) == 0) {
#pragma unroll
    for (int i = 0; i < HELD; ++i)
      if (col0 + (at + i) / 2 * GS < Cout) part[col0 / GS * 2 + at + i] = v[i];
  }
}

// The residual values of a thread's output site are asked into L2 while the tile's MMAs still run.
__device__ __forceinline__ void conv_prefetch_residual(const ConvParams& p, const TileCoord& c, int n0, bool tile_ok,
                                                       int quad, int lane) {
  if (!p.residual || !tile_ok) return;
  const int m = quad * 32 + lane;
  const int hh = m / p.bw, ww = m - hh * p.bw;
  const int h = c.h0 + hh, w = c.w0 + ww;
  if (m >= p.bh * p.bw || h >= p.H || w >= p.W) return;
  const int64_t site = ((static_cast<int64_t>(c.n) * p.T + c.t) * p.H + h) * p.W + w;
  const __nv_bfloat16* r = p.residual + site * p.Cout + n0;
  for (int cb = 0; cb < p.BN && n0 + cb < p.Cout; cb += 64) prefetch_l2(r + cb);
}

// The epilogue of one output tile for one thread (= one output site): BN columns, 32 at a time from TMEM, bias and
// residual added, bf16 stored, GroupNorm partials of the warp's 32 rows. `acc_tmem` = TMEM address of the
// accumulator's first column; `tile_ok` false = this CTA has no tile here (the odd tile of a pair): nothing is stored.
__device__ __forceinline__ void conv_epilogue_tile(const ConvParams& p, const float* bias_s, uint32_t acc_tmem,
                                                   const TileCoord& c, int n0, int m_tile, bool tile_ok, int quad, int lane) {
  const int gs = p.Cout / GN_GROUPS;  // channels per GroupNorm group (used only when gn_part != null)
  const int m = quad * 32 + lane;
  const int hh = m / p.bw, ww = m - hh * p.bw;
  const int h = c.h0 + hh, w = c.w0 + ww;
  const bool row_ok = tile_ok && m < p.bh * p.bw && h < p.H && w < p.W;
  const int64_t site = ((static_cast<int64_t>(c.n) * p.T + c.t) * p.H + h) * p.W + w;
  const uint32_t t_row = acc_tmem + (static_cast<uint32_t>(quad * 32) << 16);
  float* part = (p.gn_part && tile_ok) ? p.gn_part + (static_cast<int64_t>(m_tile) * 4 + quad) * GN_GROUPS * 2 : nullptr;
  // the residual of a chunk is loaded one chunk ahead (zeros where there is none), so its latency is spent under the
  // previous chunk's arithmetic and the TMEM round trip instead of in front of the additions
  const bool has_res = p.residual && row_ok;
  uint4 res_next[4];
  auto load_res = [&](int cb, uint4* dst) {
    const int col0 = n0 + cb;
    const __nv_bfloat16* rs = p.residual + site * p.Cout + col0;
#pragma unroll
    for (int g = 0; g < 4; g += 2) {
      if (p.wide && has_res && cb < p.BN && col0 + g * 8 + 16 <= p.Cout) {
        ld_global_32(rs + g * 8, dst[g], dst[g + 1]);
      } else {
        dst[g] = (has_res && cb < p.BN && col0 + g * 8 + 8 <= p.Cout) ? *reinterpret_cast<const uint4*>(rs + g * 8)
                                                                       : make_uint4(0, 0, 0, 0);
        dst[g + 1] = (has_res && cb < p.BN && col0 + g * 8 + 16 <= p.Cout) ? *reinterpret_cast<const uint4*>(rs + g * 8 + 8)
                                                                            : make_uint4(0, 0, 0, 0);
      }
    }
  };
  load_res(0, res_next);
#pragma unroll 1
  for (int cb = 0; cb < p.BN; cb += 32) {
    uint32_t r[32];
    tmem_ld32(t_row + cb, r);
    uint4 res[4];
#pragma unroll
    for (int g = 0; g < 4; ++g) res[g] = res_next[g];
    load_res(cb + 32, res_next);
    tmem_ld_wait_regs(r);
    const int col0 = n0 + cb;
    float y[32];
#pragma unroll
    for (int j = 0; j < 32; ++j) y[j] = __uint_as_float(r[j]) + bias_s[cb + j];
    if (has_res) {
#pragma unroll
      for (int g = 0; g < 4; ++g) {
        if (col0 + g * 8 + 8 <= p.Cout) {
          const uint4 v = res[g];
          const uint32_t vw[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            y[g * 8 + 2 * j] += bf16_lo(vw[j]);
            y[g * 8 + 2 * j + 1] += bf16_hi(vw[j]);
          }
        }
      }
    }
#pragma unroll
    for (int j = 0; j < 32; ++j) y[j] = row_ok ? bf16_round(y[j]) : 0.f;  // what is stored; rows off the edge add 0
    if (row_ok) {
      __nv_bfloat16* o = p.out + site * p.Cout + col0;
      uint4 w4[4];
#pragma unroll
      for (int g = 0; g < 4; ++g)
        w4[g] = make_uint4(pack_bf16x2(y[g * 8], y[g * 8 + 1]), pack_bf16x2(y[g * 8 + 2], y[g * 8 + 3]),
                           pack_bf16x2(y[g * 8 + 4], y[g * 8 + 5]), pack_bf16x2(y[g * 8 + 6], y[g * 8 + 7]));
#pragma unroll
      for (int g = 0; g < 4; g += 2) {
        if (p.wide && col0 + g * 8 + 16 <= p.Cout) {
          st_global_32(o + g * 8, w4[g], w4[g + 1]);
        } else {
          if (col0 + g * 8 + 8 <= p.Cout) *reinterpret_cast<uint4*>(o + g * 8) = w4[g];
          if (col0 + g * 8 + 16 <= p.Cout) *reinterpret_cast<uint4*>(o + g * 8 + 8) = w4[g + 1];
        }
      }
    }
    if (part) {
      // the group width is uniform over the launch; one instantiation per width keeps y[] in registers
      switch (gs) {
        case 1: gn_partials_chunk<1>(y, part, col0, p.Cout, lane); break;
        case 2: gn_partials_chunk<2>(y, part, col0, p.Cout, lane); break;
        case 4: gn_partials_chunk<4>(y, part, col0, p.Cout, lane); break;
        case 8: gn_partials_chunk<8>(y, part, col0, p.Cout, lane); break;
        case 16: gn_partials_chunk<16>(y, part, col0, p.Cout, lane); break;
        default: gn_partials_chunk<32>(y, part, col0, p.Cout, lane); break;
      }
    }
  }
}

template <int KCH>   // K chunks per ring stage
__global__ void __launch_bounds__(CONV_THREADS, 1)
conv3d_kernel(const __grid_constant__ CUtensorMap tma_x, const __grid_constant__ CUtensorMap tma_w,
              const ConvParams p) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  ConvSmemTail* tail = reinterpret_cast<ConvSmemTail*>(smem);
  smem += CTAIL_BYTES;
  const int CSTAGES = p.stages, CSTAGE_BYTES = p.stage_bytes;
  volatile int* abort_flag = &tail->abort_flag;

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int num_n = (p.Cout + p.BN - 1) / p.BN;
  const int num_m = p.N * p.T * p.tiles_h * p.tiles_w;
  const int num_tiles = num_m * num_n;
  const int chunks = p.Cin / CBK;
  const int num_kb = 27 * chunks;
  const uint32_t a_bytes = static_cast<uint32_t>(p.bh * p.bw) * 128u;
  const uint32_t b_bytes = static_cast<uint32_t>(p.BN) * 128u;

  if (threadIdx.x == 0) {
    for (int s = 0; s < CSTAGES; ++s) {
      mbar_init(&tail->full[s], 1);
      mbar_init(&tail->empty[s], 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(&tail->acc_full[b], 1);
      mbar_init(&tail->acc_empty[b], 4);  // one arrival per epilogue warp
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
  grid_dependency_begin();
  const uint32_t tmem_base = tail->tmem_base;

  if (warp == 0) {
    // ------------------------------ TMA producer ------------------------------
    if (lane == 0) {
      tma_prefetch_desc(&tma_x);
      tma_prefetch_desc(&tma_w);
      int stage = 0;
      uint32_t phase = 0;
      bool ok = true;
      for (int tile = blockIdx.x; tile < num_tiles && ok; tile += gridDim.x) {
        const TileCoord c = conv_tile(tile, p, num_n);
        int dh = 0, cc = 0, dw = 0, dt = 0;   // the three dh of a (dt, dw, 64 channels) follow each other, as in the pair kernel
        for (int kb = 0; kb < num_kb; kb += KCH) {
          if (!mbar_wait(&tail->empty[stage], phase ^ 1, abort_flag, p.status, ST_TIMEOUT_STAGE_EMPTY)) {
            ok = false;
            break;
          }
          mbar_arrive_expect_tx(&tail->full[stage], (a_bytes + b_bytes) * KCH);
#pragma unroll
          for (int q = 0; q < KCH; ++q) {
            const int tap = (dt * 3 + dh) * 3 + dw;
            uint8_t* sa = smem + stage * CSTAGE_BYTES + q * p.chunk_bytes;
            // out-of-range coordinates (negative or past the edge) read zeros: spatial and causal padding
            tma_load_5d(sa, &tma_x, cc * CBK, c.w0 + dw - 1, c.h0 + dh - 1, c.t + dt - 2 + p.halo, c.n, &tail->full[stage]);
            tma_load_2d(sa + CA_BYTES, &tma_w, tap * p.Cin + cc * CBK, c.n_blk * p.BN, &tail->full[stage]);
            if (++dh == 3) {
              dh = 0;
              if (++cc == chunks) {
                cc = 0;
                if (++dw == 3) {
                  dw = 0;
                  ++dt;
                }
              }
            }
          }
          if (++stage == CSTAGES) { stage = 0; phase ^= 1; }
        }
      }
    }
  } else if (warp == 1) {
    // ------------------------------ MMA issuer ------------------------------
    // the whole warp runs the loop converged (waits, counters and addresses are warp-uniform); one elected lane, the
    // same every time, issues the MMAs and the commits
    const uint32_t idesc = make_idesc(1, 1, 1, CBM, p.BN);  // f32 += bf16 * bf16
    int stage = 0;
    uint32_t phase = 0;
    int acc = 0;
    uint32_t acc_phase = 0;
    bool ok = true;
    for (int tile = blockIdx.x; tile < num_tiles && ok; tile += gridDim.x) {
      ok = __all_sync(0xffffffffu, mbar_wait(&tail->acc_empty[acc], acc_phase ^ 1, abort_flag, p.status, ST_TIMEOUT_ACC_EMPTY));
      if (!ok) break;
      tc_fence_after();
      const uint32_t d_tmem = tmem_base + acc * 256;
      for (int kb = 0; kb < num_kb; kb += KCH) {
        ok = __all_sync(0xffffffffu, mbar_wait(&tail->full[stage], phase, abort_flag, p.status, ST_TIMEOUT_TMA_FULL));
        if (!ok) break;
        tc_fence_after();
        const uint32_t a_addr = smem_u32(smem + stage * CSTAGE_BYTES);
        if (elect_one()) {
          // per K chunk four MMAs of 16 bf16 (32 bytes) each along K; one commit for the whole stage
#pragma unroll
          for (int q = 0; q < KCH; ++q) {
            const uint32_t aq = a_addr + q * p.chunk_bytes;
            mma4_f16_ss(d_tmem, make_desc_k128(aq), make_desc_k128(aq + CA_BYTES), idesc, (kb + q) != 0);
          }
          mma_commit(&tail->empty[stage]);
        }
        __syncwarp();
        if (++stage == CSTAGES) { stage = 0; phase ^= 1; }
      }
      if (!ok) break;
      if (elect_one()) mma_commit(&tail->acc_full[acc]);
      __syncwarp();
      if (++acc == 2) { acc = 0; acc_phase ^= 1; }
    }
  } else {
    // ------------------------------ epilogue (warps 2..5) ------------------------------
    const int quad = warp & 3;
    const int et = threadIdx.x - 64;
    int acc = 0;
    uint32_t acc_phase = 0;
    for (int tile = blockIdx.x; tile < num_tiles; tile += gridDim.x) {
      const TileCoord c = conv_tile(tile, p, num_n);
      const int n0 = c.n_blk * p.BN;
      asm volatile("bar.sync 1, 128;" ::: "memory");
      for (int i = et; i < p.BN; i += 128)
        tail->bias[i] = (p.bias && n0 + i < p.Cout) ? __bfloat162float(p.bias[n0 + i]) : 0.f;
      // the four warps leave together: a warp that gave up its wait takes the others with it at this barrier
      // (which also publishes the staged bias), so none of them waits at the next tile's barrier alone
      if (tile == static_cast<int>(blockIdx.x)) conv_prefetch_residual(p, c, n0, true, quad, lane);
      if (tile + static_cast<int>(gridDim.x) < num_tiles) {   // the next tile's residual, a whole epilogue ahead
        const TileCoord c2 = conv_tile(tile + gridDim.x, p, num_n);
        conv_prefetch_residual(p, c2, c2.n_blk * p.BN, true, quad, lane);
      }
      const bool got = mbar_wait(&tail->acc_full[acc], acc_phase, abort_flag, p.status, ST_TIMEOUT_ACC_FULL);
      if (bar_sync_or(1, 128, !got)) break;
      tc_fence_after();
      conv_epilogue_tile(p, tail->bias, tmem_base + acc * 256, c, n0, tile / num_n, true, quad, lane);
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&tail->acc_empty[acc]);
      if (++acc == 2) { acc = 0; acc_phase ^= 1; }
    }
  }

  __syncwarp();
  if (*abort_flag && threadIdx.x == 0) {
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
// The same convolution on CTA pairs (clusters of two, tcgen05 cta_group::2). A pair computes two neighbouring site
// tiles (m = 2 * pair_m + rank) x BN output channels with MMAs of 256 rows: every CTA fetches the input box of its own site
// tile and HALF of the BN weight rows (rank r: rows [r * BN/2, (r+1) * BN/2) of the column tile). Each CTA's TMEM receives its
// own 128 sites x BN channels and its own epilogue warps drain them exactly as in the single-CTA kernel (same fp32
// accumulation order: results are identical).
// A ring stage is 64 channels of one (dt, dw): the tile's box with one more row of sites above and below it, which serves
// all three dh, and the three taps' weight rows. What an SM has to take in and to write to its shared memory bounds tiles of
// few output channels (the operand reads of the MMAs want the same bandwidth); a box per tap was 16 KB of it, a third of a
// taller box is 6-9 KB. Before / after, us: 3 x 12 x 21 sites, 512 -> 512 channels 43.2 / 30.9, 5 x 24 x 42, 256 -> 256
// 27.2 / 24.9, 141 x 96 x 168, 128 -> 128 1,792 / 1,748; full-width tiles are bound by the tensor pipe and measure the same.
// Where a tile is one or two rows high (frames 56 to 64 or more than 112 sites wide) the box saves little and a stage of 256
// channels leaves room for two only: 7 x 26 x 62 of 256 channels 59.1 / 61.6, 8 x 23 x 128 76.0 / 79.0, but 4 x 9 x 125 28.1 / 18.5.
// When the number of site tiles is odd, the odd CTA of the last pair loads the last valid tile again and stores nothing.
// Barriers as in the GEMM's pair kernel: both CTAs' loads count on the even CTA's `full`; stage release and
// accumulator hand-over are one commit per CTA; every wait is bounded; the two cluster barriers are reached by all.
// ---------------------------------------------------------------------------------------------

struct __align__(8) ConvPairSmemTail {
  uint64_t full[CMAX_STAGES];
  uint64_t empty[CMAX_STAGES];
  uint64_t acc_full[2];
  uint64_t acc_empty[2];
  uint32_t tmem_base;
  int abort_flag;
  float bias[256];
};
static_assert(sizeof(ConvPairSmemTail) <= CTAIL_BYTES, "tail does not fit");

// site tile m and column tile of pair-tile index `tile` for CTA `rank`: column tiles fastest, then pairs of site tiles
__device__ __forceinline__ void conv_pair_tile(int tile, int rank, int num_m, int num_n, int& m, int& n_blk, bool& ok) {
  n_blk = tile % num_n;
  m = (tile / num_n) * 2 + rank;
  ok = m < num_m;
  if (!ok) m = num_m - 1;
}

__global__ void __launch_bounds__(CONV_THREADS, 1)
conv3d_pair_kernel(const __grid_constant__ CUtensorMap tma_x, const __grid_constant__ CUtensorMap tma_w,
                   const ConvParams p) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  ConvPairSmemTail* tail = reinterpret_cast<ConvPairSmemTail*>(smem);
  smem += CTAIL_BYTES;
  const int CP_STAGES = p.stages, CP_STAGE_BYTES = p.stage_bytes;
  volatile int* abort_flag = &tail->abort_flag;

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int rank = static_cast<int>(cluster_cta_rank());   // 0 = the even CTA: it issues the MMAs
  const int pair = blockIdx.x >> 1, num_pairs = gridDim.x >> 1;
  const int num_n = (p.Cout + p.BN - 1) / p.BN;
  const int num_m = p.N * p.T * p.tiles_h * p.tiles_w;
  const int num_tiles = ((num_m + 1) >> 1) * num_n;
  const int chunks = p.Cin / CBK;
  const int half_n = p.BN >> 1;
  const uint32_t stage_tx = 2u * 128u * static_cast<uint32_t>((p.bh + 2) * p.bw + 3 * half_n);

  if (threadIdx.x == 0) {
    for (int s = 0; s < CP_STAGES; ++s) {
      mbar_init(&tail->full[s], 1);     // the even CTA's: one arrive.expect_tx for the bytes of both CTAs
      mbar_init(&tail->empty[s], 1);    // one commit per CTA
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(&tail->acc_full[b], 1);
      mbar_init(&tail->acc_empty[b], 8);  // the even CTA's: one arrival per epilogue warp of both CTAs
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
  grid_dependency_begin();
  const uint32_t tmem_base = tail->tmem_base;

  if (warp == 0) {
    // ------------------------------ TMA producer (both CTAs) ------------------------------
    if (elect_one()) {
      tma_prefetch_desc(&tma_x);
      tma_prefetch_desc(&tma_w);
    }
    __syncwarp();
    int stage = 0;
    uint32_t phase = 0;
    bool ok = true;
    for (int tile = pair; tile < num_tiles && ok; tile += num_pairs) {
      int m, n_blk;
      bool tile_ok;
      conv_pair_tile(tile, rank, num_m, num_n, m, n_blk, tile_ok);
      const TileCoord c = conv_tile(m * num_n + n_blk, p, num_n);
      const int wrow0 = n_blk * p.BN + rank * half_n;
      for (int kb = 0; kb < 9 * chunks; ++kb) {
        ok = __all_sync(0xffffffffu, mbar_wait(&tail->empty[stage], phase ^ 1, abort_flag, p.status, ST_TIMEOUT_STAGE_EMPTY));
        if (!ok) break;
        const uint32_t leader_full = cluster_addr(&tail->full[stage], 0);
        const int dtw = kb / chunks, cc = kb - dtw * chunks, dt = dtw / 3, dw = dtw - 3 * dt;
        if (elect_one()) {
          if (rank == 0) mbar_arrive_expect_tx(&tail->full[stage], stage_tx);
          uint8_t* sa = smem + stage * CP_STAGE_BYTES;
          // the tile's rows and the one above and below them; out-of-range coordinates read zeros
          tma_load_5d_pair(sa, &tma_x, cc * CBK, c.w0 + dw - 1, c.h0 - 1, c.t + dt - 2 + p.halo, c.n, leader_full);
#pragma unroll
          for (int dh = 0; dh < 3; ++dh)
            tma_load_2d_pair(sa + p.chunk_bytes + dh * half_n * 128, &tma_w, ((dt * 3 + dh) * 3 + dw) * p.Cin + cc * CBK, wrow0,
                             leader_full);
        }
        __syncwarp();
        if (++stage == CP_STAGES) { stage = 0; phase ^= 1; }
      }
    }
  } else if (warp == 1) {
    // ------------------------------ MMA issuer (even CTA only; converged warp, one elected lane) ------------------------------
    if (rank == 0) {
      const uint32_t idesc = make_idesc(1, 1, 1, 2 * CBM, p.BN);  // f32 += bf16 * bf16, 256 rows over the pair
      int stage = 0;
      uint32_t phase = 0;
      int acc = 0;
      uint32_t acc_phase = 0;
      bool ok = true;
      for (int tile = pair; tile < num_tiles && ok; tile += num_pairs) {
        ok = __all_sync(0xffffffffu, mbar_wait(&tail->acc_empty[acc], acc_phase ^ 1, abort_flag, p.status, ST_TIMEOUT_ACC_EMPTY));
        if (!ok) break;
        tc_fence_after();
        const uint32_t d_tmem = tmem_base + acc * 256;
        for (int kb = 0; kb < 9 * chunks; ++kb) {
          ok = __all_sync(0xffffffffu, mbar_wait(&tail->full[stage], phase, abort_flag, p.status, ST_TIMEOUT_TMA_FULL));
          if (!ok) break;
          tc_fence_after();
          const uint32_t a_addr = smem_u32(smem + stage * CP_STAGE_BYTES), b_addr = a_addr + p.chunk_bytes;
          const uint32_t empty0 = cluster_addr(&tail->empty[stage], 0), empty1 = cluster_addr(&tail->empty[stage], 1);
          if (elect_one()) {
            // Tap row dh of a tile is the same box bw rows of shared memory further on. The swizzle goes by the address, and
            // the box starts on a 1,024-byte boundary, so an operand may start at any of its 128-byte rows.
#pragma unroll
            for (int dh = 0; dh < 3; ++dh)
              mma4_f16_pair(d_tmem, make_desc_k128(a_addr + dh * p.bw * 128), make_desc_k128(b_addr + dh * half_n * 128), idesc,
                            (kb + dh) != 0);
            mma_commit_pair(empty0);   // the stage is free in both CTAs once these MMAs have read it
            mma_commit_pair(empty1);
          }
          __syncwarp();
          if (++stage == CP_STAGES) { stage = 0; phase ^= 1; }
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
    // ------------------------------ epilogue (warps 2..5 of both CTAs) ------------------------------
    const int quad = warp & 3;
    const int et = threadIdx.x - 64;
    int acc = 0;
    uint32_t acc_phase = 0;
    for (int tile = pair; tile < num_tiles; tile += num_pairs) {
      int m, n_blk;
      bool tile_ok;
      conv_pair_tile(tile, rank, num_m, num_n, m, n_blk, tile_ok);
      const TileCoord c = conv_tile(m * num_n + n_blk, p, num_n);
      const int n0 = n_blk * p.BN;
      asm volatile("bar.sync 1, 128;" ::: "memory");
      for (int i = et; i < p.BN; i += 128)
        tail->bias[i] = (p.bias && n0 + i < p.Cout) ? __bfloat162float(p.bias[n0 + i]) : 0.f;
      if (tile == pair) conv_prefetch_residual(p, c, n0, tile_ok, quad, lane);
      if (tile + num_pairs < num_tiles) {   // the next tile's residual, a whole epilogue ahead
        int m2, nb2;
        bool ok2;
        conv_pair_tile(tile + num_pairs, rank, num_m, num_n, m2, nb2, ok2);
        conv_prefetch_residual(p, conv_tile(m2 * num_n + nb2, p, num_n), nb2 * p.BN, ok2, quad, lane);
      }
      const bool got = mbar_wait(&tail->acc_full[acc], acc_phase, abort_flag, p.status, ST_TIMEOUT_ACC_FULL);
      if (bar_sync_or(1, 128, !got)) break;
      tc_fence_after();
      conv_epilogue_tile(p, tail->bias, tmem_base + acc * 256, c, n0, m, tile_ok, quad, lane);
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive_remote(&tail->acc_empty[acc], 0);
      if (++acc == 2) { acc = 0; acc_phase ^= 1; }
    }
  }

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

// ---------------------------------------------------------------------------------------------
// GroupNorm statistics from the convolution's partials, GroupNorm + SiLU, causal 2x upsampling
// ---------------------------------------------------------------------------------------------
// sums[n][g] = (sum, sum of squares) over all row blocks of sample n, added in a fixed order in fp64. A cluster of eight CTAs
// per sample: a row of partials is 64 consecutive floats, so 16 threads read one coalesced and a CTA 32 at a time, four such
// in flight; the CTAs' sums meet in the first one's through distributed shared memory. With a CTA per group, each reading 8
// of a row's 256 bytes, the 71,064 rows of 141 x 96 x 168 sites took 76 us (of 1.3 ms for the convolution they come from);
// 28 now, 8,946 rows 5.5, 1,134 rows 2.5 in a chain.
constexpr int GNR_CTAS = 8, GNR_THREADS = 512, GNR_VEC = 2 * GN_GROUPS / 4, GNR_LANES = GNR_THREADS / GNR_VEC;
template <bool ALIGNED>   // the partials start on a 16-byte boundary
__global__ void __launch_bounds__(GNR_THREADS) gn_reduce_kernel(const float* part, int64_t rows_per_sample,
                                                                double* __restrict__ sums) {
  grid_dependency_begin();
  __shared__ double red[GNR_LANES][2 * GN_GROUPS];
  const int rank = static_cast<int>(cluster_cta_rank()), col = (threadIdx.x % GNR_VEC) * 4, lane = threadIdx.x / GNR_VEC;
  const int64_t n = blockIdx.x / GNR_CTAS;
  const float* p = part + n * rows_per_sample * (2 * GN_GROUPS) + col;
  auto load = [&](int64_t r) {
    const float* q = p + r * (2 * GN_GROUPS);
    return ALIGNED ? *reinterpret_cast<const float4*>(q) : make_float4(q[0], q[1], q[2], q[3]);
  };
  constexpr int64_t STEP = GNR_CTAS * GNR_LANES;
  double s0 = 0.0, s1 = 0.0, s2 = 0.0, s3 = 0.0;
  auto add = [&](const float4& v) {
    s0 += v.x;
    s1 += v.y;
    s2 += v.z;
    s3 += v.w;
  };
  int64_t r = rank * GNR_LANES + lane;
  for (; r + 3 * STEP < rows_per_sample; r += 4 * STEP) {
    float4 v[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) v[i] = load(r + i * STEP);
#pragma unroll
    for (int i = 0; i < 4; ++i) add(v[i]);
  }
  for (; r < rows_per_sample; r += STEP) add(load(r));
  red[lane][col] = s0;
  red[lane][col + 1] = s1;
  red[lane][col + 2] = s2;
  red[lane][col + 3] = s3;
  __syncthreads();
  const int c = threadIdx.x;
  double s = 0.0;
  if (c < 2 * GN_GROUPS) {
#pragma unroll 8
    for (int i = 0; i < GNR_LANES; ++i) s += red[i][c];
    red[0][c] = s;
  }
  cluster_sync_all();
  if (rank == 0 && c < 2 * GN_GROUPS) {
#pragma unroll
    for (uint32_t k = 1; k < GNR_CTAS; ++k) {
      double other;
      asm volatile("ld.shared::cluster.f64 %0, [%1];" : "=d"(other) : "r"(cluster_addr(&red[0][c], k)) : "memory");
      s += other;
    }
    sums[n * (2 * GN_GROUPS) + c] = s;
  }
  cluster_sync_all();   // the other CTAs' shared memory stays until it has been read
}

// y = silu((x - mean[g]) * rstd[g] * gamma[c] + beta[c]). A thread keeps one group of 8 channels for the whole
// launch (the block's 256 threads cover 256 / (C/8) sites per iteration), so the per-channel scale
// a = rstd * gamma and offset b = beta - mean * a are computed once and the loop body is one FMA and the SiLU
// per value: silu(t) = t / (1 + 2^(-t * log2 e)) with the hardware exponential and reciprocal (both good to
// about 1e-7 relative, far inside the bf16 rounding of the result; the hyperbolic-tangent form with its 2^-11
// error flipped too many of those roundings). Launched as (blocks, N); C/8 <= 256 (threads beyond the last
// whole site of the block idle).
__device__ __forceinline__ float silu_fast(float t) {
  float e, r;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(e) : "f"(t * -1.4426950408889634f));
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(1.f + e));
  return t * r;
}
// FROM_SUMS: mean and rstd are taken from the fp64 sums by the first warp of the block (a group per lane), in the order
// a chain of elementwise kernels would compute them (s * (1/count), E[x^2] - mean^2, clamped, + eps, rsqrt, all rounded
// one by one in fp64), so the bits are the same and the chain's eight launches of one tiny block each are gone: a decode
// runs 13 of these norms, 104 launches of about 3 us, which bounded small decodes on the host side.
// Six CTAs per SM: the compiler's own 50 registers leave five (141 x 96 x 168 sites of 128 channels 213 us, 237 with five; 9 x 48 x 84
// 8.6 and 9.0), and the first site is asked for ahead of the factors, whose barrier an ordinary load does not pass (8.6 for 9.6).
template <bool FROM_SUMS>
__global__ void __launch_bounds__(256, 6) gn_silu_kernel(const __nv_bfloat16* x,
                                                         const float* mean_rstd,  // [N][32][2]
                                                         const double* sums,      // [N][32][2]
                                                         double inv_count, double eps,
                                                         const __nv_bfloat16* __restrict__ gamma,
                                                         const __nv_bfloat16* __restrict__ beta, int64_t sites_per_sample,
                                                         int C, __nv_bfloat16* __restrict__ y) {
  grid_dependency_begin();
  __shared__ float2 mr_s[GN_GROUPS];
  const int vps = C >> 3;                       // 16-byte vectors per site
  const int lane_vec = threadIdx.x % vps;       // this thread's vector inside a site
  const int site_in_block = threadIdx.x / vps;
  const int sites_per_iter = 256 / vps;
  const int n = blockIdx.y;
  const int c0 = lane_vec << 3;
  const __nv_bfloat16* xs = x + static_cast<int64_t>(n) * sites_per_sample * C;
  const int64_t step = static_cast<int64_t>(gridDim.x) * sites_per_iter;
  int64_t site = site_in_block < sites_per_iter ? static_cast<int64_t>(blockIdx.x) * sites_per_iter + site_in_block : sites_per_sample;
  uint4 first;   // on its way while the factors are made
  if (site < sites_per_sample) first = ld_global_16(xs + site * C + c0);
  if (FROM_SUMS) {
    if (threadIdx.x < GN_GROUPS) {
      const double* sg = sums + (static_cast<int64_t>(blockIdx.y) * GN_GROUPS + threadIdx.x) * 2;
      const double mean = __dmul_rn(sg[0], inv_count);
      double var = __dsub_rn(__dmul_rn(sg[1], inv_count), __dmul_rn(mean, mean));
      if (var < 0.0) var = 0.0;  // a NaN stays
      mr_s[threadIdx.x] = make_float2(static_cast<float>(mean), static_cast<float>(rsqrt(__dadd_rn(var, eps))));
    }
    __syncthreads();
  }
  if (site >= sites_per_sample) return;
  const int gs = C / GN_GROUPS;
  float a[8], b[8];
  {
    const uint4 gr = __ldg(reinterpret_cast<const uint4*>(gamma + c0));
    const uint4 br = __ldg(reinterpret_cast<const uint4*>(beta + c0));
    const uint32_t gw[4] = {gr.x, gr.y, gr.z, gr.w}, bw[4] = {br.x, br.y, br.z, br.w};
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const float2 mr = FROM_SUMS ? mr_s[(c0 + j) / gs]
                                  : *reinterpret_cast<const float2*>(mean_rstd + (static_cast<int64_t>(n) * GN_GROUPS + (c0 + j) / gs) * 2);
      const float gv = (j & 1) ? bf16_hi(gw[j >> 1]) : bf16_lo(gw[j >> 1]);
      const float bv = (j & 1) ? bf16_hi(bw[j >> 1]) : bf16_lo(bw[j >> 1]);
      a[j] = mr.y * gv;
      b[j] = fmaf(-mr.x, a[j], bv);
    }
  }
  __nv_bfloat16* ys = y + static_cast<int64_t>(n) * sites_per_sample * C;
  auto apply = [&](const uint4& raw) {
    const uint32_t xw[4] = {raw.x, raw.y, raw.z, raw.w};
    uint32_t o[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const float t0 = fmaf(bf16_lo(xw[j]), a[2 * j], b[2 * j]);
      const float t1 = fmaf(bf16_hi(xw[j]), a[2 * j + 1], b[2 * j + 1]);
      o[j] = pack_bf16x2(silu_fast(t0), silu_fast(t1));
    }
    *reinterpret_cast<uint4*>(ys + site * C + c0) = make_uint4(o[0], o[1], o[2], o[3]);
  };
  apply(first);
  for (site += step; site < sites_per_sample; site += step) apply(ld_global_16(xs + site * C + c0));
}

// out[n, u, yy, xx, :] = in[n, (u + 1) / 2, yy / 2, xx / 2, :]: nearest 2x in space, causal 2x in time
// (the first frame is not repeated: T frames become 2T - 1). A thread per 16 bytes of the input, read once and stored to their
// four places in one or two frames. Bound by the stores. us with a thread per output vector (five 64-bit divisions each) / a CTA
// per input row / now: 71 x 48 x 84 sites of 256 channels (1.31 GB) 427 / 218 / 201 (of the measured copy rate 1.0), 36 x 24 x 42 of
// 512 109 / 69.5 / 53, and where rows are few, 3 x 12 x 21 of 512 3.5 / 4.3 / 2.3, 1 x 24 x 42 of 512 3.0 / 4.2 / 2.2.
__global__ void __launch_bounds__(256) upsample_kernel(const __nv_bfloat16* x, uint32_t total, uint32_t T, uint32_t H, uint32_t W,
                                                       uint32_t vec, __nv_bfloat16* __restrict__ y) {   // vec: 16-byte vectors per site
  grid_dependency_begin();
  const uint32_t v = blockIdx.x * 256 + threadIdx.x;
  if (v >= total) return;
  const uint4 q = ld_global_16(reinterpret_cast<const uint4*>(x) + v);
  const uint32_t site = v / vec, r = site / W, nt = r / H, n = nt / T;   // r: row of sites
  const uint32_t w = site - r * W, h = r - nt * H, t = nt - n * T;
  const int64_t row = 2ll * W * vec, frame = 2ll * H * row;
  uint4* d = reinterpret_cast<uint4*>(y) + (static_cast<int64_t>(n) * (2 * T - 1) + (t == 0 ? 0 : 2 * t - 1)) * frame +
             2ll * h * row + 2ll * w * vec + (v - site * vec);
  d[0] = q;
  d[vec] = q;
  d[row] = q;
  d[row + vec] = q;
  if (t) {
    d[frame] = q;
    d[frame + vec] = q;
    d[frame + row] = q;
    d[frame + row + vec] = q;
  }
}

// tile of output sites inside a frame: bh * bw <= 128, chosen to waste as few MMA rows as possible
void choose_tile(int H, int W, int* bh, int* bw) {
  double best = -1.0;
  for (int w = 1; w <= 128 && w <= 256; ++w) {
    const int h = 128 / w;
    if (h < 1) break;
    const int hh = h < H ? h : H, ww = w < W ? w : W;
    const double eff = static_cast<double>(H) * W / (static_cast<double>((H + hh - 1) / hh) * ((W + ww - 1) / ww) * 128.0);
    if (eff > best + 1e-9) {
      best = eff;
      *bh = hh;
      *bw = ww;
    }
  }
}

// K chunks per ring stage of the single-CTA kernel. A stage costs one barrier round trip in the producer and in the MMA
// issuer, a few hundred cycles that a narrow tile's four MMAs per chunk (2 * BN tensor cycles) do not cover: narrow tiles put two
// or four chunks behind one barrier. The count divides the 27 * chunks_per_tap chunks of a tile.
int choose_kch(int bn, int chunks_per_tap) {
  int want = bn > 128 ? 1 : (bn > 64 ? 2 : 4);
  while (want > 1 && chunks_per_tap % want != 0) want >>= 1;
  return want;
}

bool a16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; }

}  // namespace
}  // namespace rh3

using namespace rh3;

extern "C" int64_t rh3_conv3d_gn_part_rows(int64_t N, int64_t T, int64_t H, int64_t W) {
  int bh = 1, bw = 1;
  choose_tile((int)H, (int)W, &bh, &bw);
  return N * T * ((H + bh - 1) / bh) * ((W + bw - 1) / bw) * 4;
}

extern "C" int rh3_conv3d_causal(const void* x, const void* w, const void* bias, const void* residual, void* out,
                                 float* gn_part, int64_t N, int64_t T, int64_t H, int64_t W, int64_t Cin,
                                 int64_t Cout, int64_t halo_frames, cudaStream_t stream) {
  RH3_CHECK_ARG(N > 0 && T > 0 && H > 0 && W > 0 && N * T * H * W < (1ll << 31), "conv3d_causal: bad shape");
  RH3_CHECK_ARG(halo_frames == 0 || halo_frames == 2, "conv3d_causal: halo_frames must be 0 or 2");
  RH3_CHECK_ARG(Cin > 0 && Cin % 64 == 0, "conv3d_causal: Cin=%lld must be a multiple of 64", (long long)Cin);
  RH3_CHECK_ARG(Cout > 0 && Cout % 16 == 0, "conv3d_causal: Cout=%lld must be a multiple of 16", (long long)Cout);
  RH3_CHECK_ARG(!gn_part || (Cout % GN_GROUPS == 0 && 32 % (Cout / GN_GROUPS) == 0),
                "conv3d_causal: GroupNorm partials need Cout/32 in {1,2,4,8,16,32}");
  RH3_CHECK_ARG(x && w && out && a16(x) && a16(w) && a16(out) && (!residual || a16(residual)),
                "conv3d_causal: null or misaligned pointer");
  ConvParams p{};
  p.N = (int)N; p.T = (int)T; p.H = (int)H; p.W = (int)W; p.Cin = (int)Cin; p.Cout = (int)Cout;
  p.halo = (int)halo_frames;
  choose_tile(p.H, p.W, &p.bh, &p.bw);
  p.tiles_h = (p.H + p.bh - 1) / p.bh;
  p.tiles_w = (p.W + p.bw - 1) / p.bw;
  // output channels per tile: the whole width when it fits one accumulator, else an even split. The epilogue walks
  // a tile in 32-column chunks, so a split tile is a multiple of 32 wide: a chunk must never reach into the columns
  // of the next tile (weight rows past Cout are zero-filled by TMA and their stores are skipped).
  int splits = (p.Cout + 255) / 256;
  auto tile_width = [&](int n) {
    const int bn = ((p.Cout + n - 1) / n + 15) / 16 * 16;
    return n > 1 ? (bn + 31) / 32 * 32 : bn;
  };
  // Few sites leave most of the chip idle at full width (a 3 x 12 x 21 latent has 6 site tiles: 12 CTAs at 512 channels,
  // 79 us a layer), so the channels are split further while that lowers waves x time of a tile. A pair's tile takes as
  // long as an SM needs to take in its K chunks: a third of the box of bh + 2 rows, which serves three taps, and 64 B per channel
  // each, so a split is not free. us a layer with the 16 KB of a box per tap in that place / with the box's third: 13 x 22 x 82
  // sites of 256 channels 74.6 / 58.7, 36 x 24 x 11 of 512 137 / 113, 25 x 7 x 42 of 512 137 / 103 (full width in 1.03 to 1.5
  // waves, half the width in 2.05 to 3).
  {
    const int64_t pairs = (N * T * p.tiles_h * p.tiles_w + 1) / 2, resident = device_sm_count() / 2;
    auto cost = [&](int n) {
      const int bn = tile_width(n);
      return ((pairs * ((p.Cout + bn - 1) / bn) + resident - 1) / resident) * ((p.bh + 2) * p.bw * 128ll / 3 + 64ll * bn);
    };
    for (int n = splits * 2; tile_width(n) >= 64 && cost(n) < cost(splits); n *= 2) splits = n;
  }
  p.BN = tile_width(splits);
  p.bias = static_cast<const __nv_bfloat16*>(bias);
  p.residual = static_cast<const __nv_bfloat16*>(residual);
  p.out = static_cast<__nv_bfloat16*>(out);
  p.gn_part = gn_part;
  p.status = device_status_word();
  p.wide = (reinterpret_cast<uintptr_t>(out) & 31) == 0 && (!residual || (reinterpret_cast<uintptr_t>(residual) & 31) == 0);
  CUtensorMap tx, tw;
  const uint64_t Tin = (uint64_t)(T + halo_frames);  // frames held by x
  const uint64_t dims[5] = {(uint64_t)Cin, (uint64_t)W, (uint64_t)H, Tin, (uint64_t)N};
  const uint64_t strides[4] = {(uint64_t)Cin * 2, (uint64_t)W * Cin * 2, (uint64_t)H * W * Cin * 2,
                               Tin * H * W * Cin * 2};
  const int64_t num_m = N * T * p.tiles_h * p.tiles_w, num_n = (Cout + p.BN - 1) / p.BN;
  // CTA pairs: two site tiles per pair and BN/2 weight rows per CTA (a multiple of 16, so every MMA shape is legal)
  const bool pair = pairs_enabled() && num_m >= 2 && p.BN % 32 == 0;
  const uint32_t box[5] = {CBK, (uint32_t)p.bw, (uint32_t)(pair ? p.bh + 2 : p.bh), 1, 1};
  if (int e = make_tmap_nd(&tx, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, x, 5, dims, strides, box, CU_TENSOR_MAP_SWIZZLE_128B))
    return e;
  if (int e = make_tmap_2d(&tw, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, w, 27 * Cin, Cout, 27 * Cin * 2, CBK, pair ? p.BN / 2 : p.BN,
                           CU_TENSOR_MAP_SWIZZLE_128B))
    return e;
  if (pair) {
    // a stage: the box (128 rows can be read from row 2 * bw on), then three taps' weight rows
    p.chunk_bytes = (CBM + 2 * p.bw + 7) / 8 * 1024;
    p.stage_bytes = p.chunk_bytes + 3 * (p.BN / 2) * 128;
    p.stages = CRING_MAX_BYTES / p.stage_bytes < CMAX_STAGES ? CRING_MAX_BYTES / p.stage_bytes : CMAX_STAGES;
    const int CONV_PAIR_SMEM_BYTES = 1024 + CTAIL_BYTES + p.stages * p.stage_bytes;
    auto kern = conv3d_pair_kernel;
    if (int e = check_cuda(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, CONV_PAIR_SMEM_BYTES),
                           "conv3d pair smem attribute"))
      return e;
    cudaLaunchConfig_t cfg{};
    cudaLaunchAttribute attr{};
    attr.id = cudaLaunchAttributeClusterDimension;
    attr.val.clusterDim.x = 2;
    attr.val.clusterDim.y = 1;
    attr.val.clusterDim.z = 1;
    cfg.blockDim = dim3(CONV_THREADS);
    cfg.dynamicSmemBytes = CONV_PAIR_SMEM_BYTES;
    cfg.stream = stream;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    cfg.gridDim = dim3(2 * (device_sm_count() / 2));
    int max_clusters = 0;
    if (cudaOccupancyMaxActiveClusters(&max_clusters, kern, &cfg) != cudaSuccess || max_clusters < 1)
      return set_error(RH3_ARG_ERROR, "conv3d pair: no cluster of two CTAs can be resident");
    const int64_t pair_tiles = (num_m + 1) / 2 * num_n;
    const unsigned ctas = 2 * static_cast<unsigned>(pair_tiles < max_clusters ? pair_tiles : max_clusters);
    return check_cuda(launch_chained(kern, dim3(ctas), CONV_THREADS, CONV_PAIR_SMEM_BYTES, stream, 2, tx, tw, p), "conv3d pair launch");
  }
  p.chunk_bytes = CA_BYTES + p.BN * 128;
  p.kch = choose_kch(p.BN, (int)(Cin / CBK));
  p.stage_bytes = p.kch * p.chunk_bytes;
  p.stages = CRING_MAX_BYTES / p.stage_bytes < CMAX_STAGES ? CRING_MAX_BYTES / p.stage_bytes : CMAX_STAGES;
  const int CONV_SMEM_BYTES = 1024 + CTAIL_BYTES + p.stages * p.stage_bytes;
  const int64_t tiles = num_m * num_n;
  const int grid = tiles < device_sm_count() ? (int)tiles : device_sm_count();
  auto launch_single = [&](auto kern) -> int {
    if (int e = check_cuda(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, CONV_SMEM_BYTES),
                           "conv3d smem attribute"))
      return e;
    return check_cuda(launch_chained(kern, dim3(grid), CONV_THREADS, CONV_SMEM_BYTES, stream, 1, tx, tw, p), "conv3d launch");
  };
  if (int e = p.kch == 4 ? launch_single(conv3d_kernel<4>) : p.kch == 2 ? launch_single(conv3d_kernel<2>)
                                                                        : launch_single(conv3d_kernel<1>))
    return e;
  return check_cuda(cudaGetLastError(), "conv3d_causal launch");
}

extern "C" int rh3_gn_reduce(const float* gn_part, int64_t rows_per_sample, int64_t N, double* sums,
                             cudaStream_t stream) {
  RH3_CHECK_ARG(gn_part && sums && rows_per_sample > 0 && N > 0 && N * GN_GROUPS < (1ll << 31), "gn_reduce: bad argument");
  return check_cuda(launch_chained(a16(gn_part) ? gn_reduce_kernel<true> : gn_reduce_kernel<false>, dim3(static_cast<unsigned>(N * GNR_CTAS)), GNR_THREADS, 0, stream, GNR_CTAS, gn_part,
                                   rows_per_sample, sums),
                    "gn_reduce launch");
}

namespace {
int gn_silu_launch(const void* x, const float* mean_rstd, const double* sums, double count, double eps, const void* gamma,
                   const void* beta, int64_t N, int64_t sites_per_sample, int64_t C, void* y, cudaStream_t stream) {
  RH3_CHECK_ARG(x && (mean_rstd || sums) && gamma && beta && y && a16(x) && a16(y) && a16(gamma) && a16(beta),
                "gn_silu_apply: null or misaligned pointer");
  RH3_CHECK_ARG(N > 0 && sites_per_sample > 0 && C > 0 && C % 8 == 0 && C % GN_GROUPS == 0, "gn_silu_apply: bad shape");
  RH3_CHECK_ARG(C / 8 <= 256, "gn_silu_apply: C=%lld is larger than 2048", (long long)C);
  RH3_CHECK_ARG(N < 65536, "gn_silu_apply: too many samples");
  const int64_t sites_per_iter = 256 / (C / 8);
  const int64_t want = (sites_per_sample + sites_per_iter - 1) / sites_per_iter;
  const int64_t cap = static_cast<int64_t>(device_sm_count()) * 16;  // a few waves of resident blocks, grid-stride beyond
  const dim3 grid(static_cast<unsigned>(want < cap ? want : cap), static_cast<unsigned>(N));
  auto kern = sums ? gn_silu_kernel<true> : gn_silu_kernel<false>;
  return check_cuda(launch_chained(kern, grid, 256, 0, stream, 1, static_cast<const __nv_bfloat16*>(x), mean_rstd, sums, 1.0 / count, eps,
                                   static_cast<const __nv_bfloat16*>(gamma), static_cast<const __nv_bfloat16*>(beta),
                                   sites_per_sample, (int)C, static_cast<__nv_bfloat16*>(y)),
                    "gn_silu_apply launch");
}
}  // namespace

extern "C" int rh3_gn_silu_apply(const void* x, const float* mean_rstd, const void* gamma, const void* beta, int64_t N,
                                 int64_t sites_per_sample, int64_t C, void* y, cudaStream_t stream) {
  RH3_CHECK_ARG(mean_rstd, "gn_silu_apply: null or misaligned pointer");
  return gn_silu_launch(x, mean_rstd, nullptr, 1.0, 0.0, gamma, beta, N, sites_per_sample, C, y, stream);
}

extern "C" int rh3_gn_silu_from_sums(const void* x, const double* sums, double count, double eps, const void* gamma,
                                     const void* beta, int64_t N, int64_t sites_per_sample, int64_t C, void* y,
                                     cudaStream_t stream) {
  RH3_CHECK_ARG(sums, "gn_silu_from_sums: null sums");
  RH3_CHECK_ARG(count > 0.0, "gn_silu_from_sums: count must be greater than 0");
  return gn_silu_launch(x, nullptr, sums, count, eps, gamma, beta, N, sites_per_sample, C, y, stream);
}

// Depth-to-space by 8 of the decoder head: y [N, T, H, W, 3*8*8] (channel = (ch*8 + dy)*8 + dx) ->
// rgb [N, 3, T, 8H, 8W]. A CTA moves 32 sites of a row through shared memory: 24 vectors of 16 bytes per site come in as they
// lie, and each of the 24 output rows gets its 32 vectors as one contiguous run. With a thread per output vector, whose loads
// were 384 bytes apart, 141 x 96 x 168 sites (1.75 GB) took 359 us, 254 now.
constexpr int D2S_SITES = 32;
__global__ void __launch_bounds__(256) depth_to_space8_kernel(const __nv_bfloat16* y, int T, int H, int W, int w_blocks,
                                                              __nv_bfloat16* __restrict__ rgb) {
  grid_dependency_begin();
  __shared__ uint4 tile[D2S_SITES][25];   // one vector of padding: the column reads below meet no bank twice
  const int w0 = static_cast<int>(blockIdx.x % w_blocks) * D2S_SITES;
  const int64_t site_row = blockIdx.x / w_blocks;   // (n * T + t) * H + h
  const int h = static_cast<int>(site_row % H);
  const int64_t nt = site_row / H, n = nt / T, t = nt - n * T;
  const int sites = min(D2S_SITES, W - w0);
  const uint4* src = reinterpret_cast<const uint4*>(y) + (site_row * W + w0) * 24;
  for (int i = threadIdx.x; i < sites * 24; i += 256) tile[i / 24][i % 24] = ld_global_16(src + i);
  __syncthreads();
  const int lane = threadIdx.x & 31;
  for (int k = threadIdx.x >> 5; k < 24; k += 8) {
    const int ch = k >> 3, dy = k & 7;
    if (lane < sites)
      reinterpret_cast<uint4*>(rgb)[(((n * 3 + ch) * T + t) * 8 * H + 8 * h + dy) * W + w0 + lane] = tile[lane][k];
  }
}

extern "C" int rh3_upsample_causal2x(const void* x, void* y, int64_t N, int64_t T, int64_t H, int64_t W, int64_t C,
                                     cudaStream_t stream) {
  RH3_CHECK_ARG(x && y && a16(x) && a16(y) && N > 0 && T > 0 && H > 0 && W > 0 && C > 0 && C % 8 == 0,
                "upsample_causal2x: bad argument");
  // input vectors; one past 32 bits would need 64 GB of input and four to eight times that of output
  const int64_t total = N * T * H * W * (C / 8);
  RH3_CHECK_ARG(total <= 0xffffff00ll, "upsample_causal2x: tensor too large");
  return check_cuda(launch_chained(upsample_kernel, dim3(static_cast<unsigned>((total + 255) / 256)), 256, 0, stream, 1,
                                   static_cast<const __nv_bfloat16*>(x), static_cast<uint32_t>(total), static_cast<uint32_t>(T),
                                   static_cast<uint32_t>(H), static_cast<uint32_t>(W), static_cast<uint32_t>(C / 8),
                                   static_cast<__nv_bfloat16*>(y)),
                    "upsample_causal2x launch");
}

extern "C" int rh3_depth_to_space8(const void* y, void* rgb, int64_t N, int64_t T, int64_t H, int64_t W,
                                   cudaStream_t stream) {
  RH3_CHECK_ARG(y && rgb && a16(y) && a16(rgb) && N > 0 && T > 0 && H > 0 && W > 0, "depth_to_space8: bad argument");
  const int64_t total = N * 3 * T * 8 * H * W;
  RH3_CHECK_ARG((total + 255) / 256 < (1ll << 31), "depth_to_space8: tensor too large");
  const int64_t w_blocks = (W + D2S_SITES - 1) / D2S_SITES;
  return check_cuda(launch_chained(depth_to_space8_kernel, dim3(static_cast<unsigned>(N * T * H * w_blocks)), 256, 0, stream, 1,
                                   static_cast<const __nv_bfloat16*>(y), (int)T, (int)H, (int)W, (int)w_blocks,
                                   static_cast<__nv_bfloat16*>(rgb)),
                    "depth_to_space8 launch");
}

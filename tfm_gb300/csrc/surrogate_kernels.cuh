// Kernels of the contact-map surrogate network.
//
// Tensor-core kernels (tcgen05, TMA, TMEM):
//  * k_conv_tc: implicit-GEMM convolution over channels-last BF16 images
//    [B][H][W][C]. One CTA tile is 128 consecutive output pixels of one image
//    row (M = 128) times all output channels (N = 64 or 128); K runs over
//    taps x 64-channel input blocks. For each tap row one TMA load brings the
//    input window of the tile's pixels plus a margin on both sides
//    (out-of-image pixels arrive as zeros, which is the convolution's zero
//    padding); each tap of the row reads it at its own row offset. The
//    weights of all taps stay resident in shared memory. Accumulators live in
//    TMEM, 256 / N of them, so the epilogue of one tile overlaps the MMAs of
//    the next ones; the epilogue loads its global inputs before it waits.
//    The epilogue fuses bias, ReLU, the residual add, the ReLU mask bits and
//    the gradient masking of the backward pass. The same kernel computes the
//    input gradient of a convolution with negated tap offsets and transposed
//    weights.
//  * k_wgrad_tc: weight (and bias) gradients. D[(tap, ci)][co] = sum over
//    pixels p of X[p + tap offset][ci] dY[p][co] is a GEMM whose K dimension
//    is the pixel; both operands come from channels-last tiles, so they are
//    MN-major. Two (tap, channel block) "atoms" of 64 rows stack into M = 128;
//    an all-ones atom gives the bias gradient. Each CTA reduces a range of
//    pixels into FP32 partial sums that k_wgrad_reduce adds up in a fixed
//    order.
// CUDA-core kernels: sequence embedding, pooling, the outer-product pair
// features and their gradient, the loss and its gradient, AdamW. The output
// layer (64 -> 1) runs in the last head convolution's epilogue.
#pragma once

#include <cuda_bf16.h>
#include <cstdint>

#include "tc.cuh"

namespace sur {

using bf16 = __nv_bfloat16;

constexpr int MAX_TAPS = 9;
// warp 0: TMA; warps 1-2: MMA issue, alternate tiles, each from its own ring
// of input windows (warp 1 also owns TMEM); warps 3-10: epilogue (two warps per TMEM lane quarter, each taking
// half of the output channels). Two issuing warps keep the tensor core fed:
// one thread issues a 128 x N x 16 MMA every ~90 cycles, the tensor core
// runs a 128 x 64 x 16 MMA every 48.
constexpr int MMA_WARPS = 2;
constexpr int CONV_THREADS = 32 * (1 + MMA_WARPS + 8);
constexpr int EPI_WARPS = 8;
constexpr int MAX_STAGES = 8;
static_assert(MAX_STAGES % MMA_WARPS == 0, "window rings of equal size");
constexpr uint32_t TMEM_COLS_CONV = 256;  // 256 / N accumulators of N columns

// A-operand windows: the input pixels [w0 - WIN_RADIUS, w0 + 128 + WIN_RADIUS)
// of one image row, so that every tap of that row (column offset |dw| <=
// WIN_RADIUS) is a row-shifted view of the same shared-memory tile. A K-major
// 128-byte-swizzled operand may start at any row of such a tile: the swizzle
// is a function of the absolute shared-memory address.
constexpr int WIN_RADIUS = 8;
constexpr int WIN_ROWS = 128 + 2 * WIN_RADIUS;
constexpr uint32_t WIN_BYTES = (uint32_t)WIN_ROWS * 128u;  // a multiple of 1024

// Taps form an R x C grid (R in {1, 3}, C in {1, 5, ...}, both odd): tap
// t = r C + c reads the input at (dh, dw) = ((r - R/2) step_h, (c - C/2)
// step_w). The steps carry the dilation and its sign (negative for the
// input-gradient convolution); |dw| <= WIN_RADIUS.
struct ConvShape {
  int B, H, W;     // image (input = output size); W is a multiple of 128
  int stages;      // A-window slots (a multiple of MMA_WARPS, up to MAX_STAGES)
  int n_tiles;     // B * H * W / 128
  int step_h, step_w;
};

// Fused epilogue of k_conv_tc; every pointer is optional. Per output value:
// v = acc + bias; mask bit = v > 0; v = relu(v); v += resid (BF16 or FP32);
// v += resid_dy[p] wo[c]; out_f32 = v; out = v, zeroed where the bit of
// mask_in is clear;
// y[p] += wo . bf16(v[p]) + bo[0] (the network's output layer, N = 64 only;
// y must be zeroed before the launch).
struct ConvEpi {
  const float *bias;        // [N]
  int relu;
  const bf16 *resid;        // [P][N]
  const float *resid_f32;   // [P][N]
  float *out_f32;           // [P][N]
  const uint32_t *mask_in;  // [P][N / 32]
  bf16 *out;                // [P][N]
  uint32_t *mask_out;       // [P][N / 32]
  const float *wo, *bo;     // [64], [1]
  float *y;                 // [P]
  const float *resid_dy;    // [P]: adds resid_dy[p] * wo[c] (the output layer's gradient)
  int resid_is_input;       // resid is the convolution's input image (k_conv_rows)
};

// shared memory after the operand tiles: barriers (256 B), TMEM slot and
// abort flag (256 B), bias [128], output weights [64]
constexpr uint32_t CONV_SMEM_TAIL = 256u + 256u + 512u + 256u;
// then one 2 KB staging tile per epilogue warp (32 pixels x 32 BF16 channels)
constexpr uint32_t EPI_STAGE_BYTES = 32u * 32u * 2u;

__host__ __device__ constexpr uint32_t conv_smem_bytes(int ntaps, int cin_blocks, int N, int stages) {
  return 1024u + (uint32_t)(ntaps * cin_blocks) * (uint32_t)N * 128u + (uint32_t)stages * WIN_BYTES +
         CONV_SMEM_TAIL + (uint32_t)EPI_WARPS * EPI_STAGE_BYTES;
}

__device__ __forceinline__ uint32_t pack_bf16(float a, float b) {
  __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
  return *reinterpret_cast<uint32_t *>(&h);
}

__device__ __forceinline__ float bf_lo(uint32_t w) { return __uint_as_float(w << 16); }
__device__ __forceinline__ float bf_hi(uint32_t w) { return __uint_as_float(w & 0xFFFF0000u); }

__device__ __forceinline__ void load_bf16x16(const bf16 *src, float *v) {
  const uint4 *s = reinterpret_cast<const uint4 *>(src);
  uint4 a = s[0], b = s[1];
  uint32_t w[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    v[2 * i] = bf_lo(w[i]);
    v[2 * i + 1] = bf_hi(w[i]);
  }
}

__device__ __forceinline__ void store_bf16x16(bf16 *dst, const float *v) {
  uint4 a, b;
  a.x = pack_bf16(v[0], v[1]);
  a.y = pack_bf16(v[2], v[3]);
  a.z = pack_bf16(v[4], v[5]);
  a.w = pack_bf16(v[6], v[7]);
  b.x = pack_bf16(v[8], v[9]);
  b.y = pack_bf16(v[10], v[11]);
  b.z = pack_bf16(v[12], v[13]);
  b.w = pack_bf16(v[14], v[15]);
  uint4 *d = reinterpret_cast<uint4 *>(dst);
  d[0] = a;
  d[1] = b;
}

// Global inputs of one output pixel's epilogue, loaded before the
// accumulator is ready so their latency overlaps the tile's MMAs.
template <int N>
struct EpiLoads {
  uint4 rb[N / 64][4];
  float4 rf[N / 64][8];
  uint32_t mi[N / 64];
  float rdy;
};

// The 32 BF16 channels (c0 ..) of this lane's pixel pbase + lane, loaded for
// the whole warp: each load instruction reads 8 pixels' 64 contiguous bytes
// into the warp's staging tile (the swizzle of store_row_bf16x32), from
// which every lane takes its own pixel's 64 bytes.
template <int N>
__device__ __forceinline__ void load_row_bf16x32(const bf16 *src, size_t pbase, int c0, uint4 *dst,
                                                 uint4 *stage) {
  const int lane = threadIdx.x & 31;
  const int c = lane & 3;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int pr = (lane >> 2) + 8 * i;
    stage[pr * 4 + (c ^ ((pr >> 1) & 3))] =
        reinterpret_cast<const uint4 *>(src + (pbase + (size_t)pr) * N + c0)[c];
  }
  __syncwarp();
#pragma unroll
  for (int k = 0; k < 4; ++k) dst[k] = stage[lane * 4 + (k ^ ((lane >> 1) & 3))];
  __syncwarp();
}

// N: the CTA's channels, from c_base on, of the LD of a pixel.
template <int N, int LD>
__device__ __forceinline__ void conv_epilogue_load(const ConvEpi &e, size_t p, int c_base, int half,
                                                   EpiLoads<N> &ld, uint4 *stage) {
  constexpr int G = N / 64;  // 32-column groups per thread
  const int c_begin = c_base + half * (N / 2);
#pragma unroll
  for (int g = 0; g < G; ++g) {
    const size_t o = p * (size_t)LD + c_begin + 32 * g;
    if (e.resid)
      load_row_bf16x32<LD>(e.resid, p - (size_t)(threadIdx.x & 31), c_begin + 32 * g, ld.rb[g], stage);
    if (e.resid_f32) {
      const float4 *s = reinterpret_cast<const float4 *>(e.resid_f32 + o);
#pragma unroll
      for (int i = 0; i < 8; ++i) ld.rf[g][i] = s[i];
    }
    if (e.mask_in) ld.mi[g] = e.mask_in[p * (LD / 32) + (c_begin >> 5) + g];
  }
  ld.rdy = e.resid_dy ? e.resid_dy[p] : 0.0f;
}

// Stores the 32 BF16 channels v of this lane's pixel (pixel pbase + lane,
// channels c0 ..) for the whole warp: the 32 x 64 B are staged in the warp's
// shared-memory tile (16-byte chunks XOR-swizzled by pixel, so neither the
// lane-per-pixel writes nor the pixel-pair reads conflict on banks), then
// each store instruction writes 8 pixels' 64 contiguous bytes. Written
// directly, every 16-byte store would touch 32 different lines.
template <int N>
__device__ __forceinline__ void store_row_bf16x32(bf16 *out, size_t pbase, int c0, const float *v,
                                                  uint4 *stage) {
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int k = 0; k < 4; ++k)
    stage[lane * 4 + (k ^ ((lane >> 1) & 3))] =
        make_uint4(pack_bf16(v[8 * k], v[8 * k + 1]), pack_bf16(v[8 * k + 2], v[8 * k + 3]),
                   pack_bf16(v[8 * k + 4], v[8 * k + 5]), pack_bf16(v[8 * k + 6], v[8 * k + 7]));
  __syncwarp();
  const int c = lane & 3;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int pr = (lane >> 2) + 8 * i;
    reinterpret_cast<uint4 *>(out + (pbase + (size_t)pr) * N + c0)[c] =
        stage[pr * 4 + (c ^ ((pr >> 1) & 3))];
  }
  __syncwarp();
}

// Epilogue of one output pixel p for the thread's half of the N channels
// (32 N / 64 columns from TMEM address taddr), with its global inputs in ld;
// stage: the warp's 2 KB staging tile for the BF16 output.
// Returns this thread's partial output-layer dot (0 without wo).
template <int N, int LD>
__device__ __forceinline__ float conv_epilogue_row(const ConvEpi &e, const float *sbias, const float *swo,
                                                   size_t p, int c_base, int half, uint32_t taddr,
                                                   const EpiLoads<N> &ld, uint4 *stage) {
  constexpr int G = N / 64;
  const int c_begin = half * (N / 2);
  const float rdy = ld.rdy;
  float dot = 0.0f;
#pragma unroll
  for (int g = 0; g < G; ++g) {
    const int c0 = c_begin + 32 * g;
    float v[32];
    tc::tmem_ld32(taddr + (uint32_t)c0, v);
    if (e.bias) {
#pragma unroll
      for (int i = 0; i < 32; ++i) v[i] += sbias[c0 + i];
    }
    if (e.mask_out) {
      uint32_t bits = 0;
#pragma unroll
      for (int i = 0; i < 32; ++i) bits |= (v[i] > 0.0f ? 1u : 0u) << i;
      e.mask_out[p * (LD / 32) + ((c_base + c0) >> 5)] = bits;
    }
    if (e.relu) {
#pragma unroll
      for (int i = 0; i < 32; ++i) v[i] = fmaxf(v[i], 0.0f);
    }
    if (e.resid) {
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const uint32_t w[4] = {ld.rb[g][i].x, ld.rb[g][i].y, ld.rb[g][i].z, ld.rb[g][i].w};
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          v[8 * i + 2 * k] += bf_lo(w[k]);
          v[8 * i + 2 * k + 1] += bf_hi(w[k]);
        }
      }
    }
    if (e.resid_f32) {
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        v[4 * i] += ld.rf[g][i].x;
        v[4 * i + 1] += ld.rf[g][i].y;
        v[4 * i + 2] += ld.rf[g][i].z;
        v[4 * i + 3] += ld.rf[g][i].w;
      }
    }
    if (e.resid_dy) {
#pragma unroll
      for (int i = 0; i < 32; ++i) v[i] = fmaf(rdy, swo[c0 + i], v[i]);
    }
    const size_t o = p * (size_t)LD + c_base + c0;
    if (e.out_f32) {
      float4 *d = reinterpret_cast<float4 *>(e.out_f32 + o);
#pragma unroll
      for (int i = 0; i < 8; ++i) d[i] = make_float4(v[4 * i], v[4 * i + 1], v[4 * i + 2], v[4 * i + 3]);
    }
    if (e.y) {
#pragma unroll
      for (int i = 0; i < 32; ++i) dot = fmaf(swo[c0 + i], __bfloat162float(__float2bfloat16_rn(v[i])), dot);
    }
    if (e.mask_in) {
#pragma unroll
      for (int i = 0; i < 32; ++i) v[i] = ((ld.mi[g] >> i) & 1u) ? v[i] : 0.0f;
    }
    if (e.out) store_row_bf16x32<LD>(e.out, p - (size_t)(threadIdx.x & 31), c_base + c0, v, stage);
  }
  return dot;
}

// Implicit-GEMM convolution (see the file comment). tmx: 4-D map over the
// input image {C, W, H, B} with box {64, 128, 1, 1}; tmw: 2-D map over the
// weights {C_in, taps x LD} with box {64, N}, both with 128-byte swizzle.
// Grid: persistent, at most one CTA per SM; tiles strided by gridDim.x. A CTA
// computes N of the LD output channels, those of blockIdx.y: with too few tiles
// for the SMs two CTAs share a tile, which halves its weights, MMAs and
// epilogue. A value's sum is the same either way.
template <int N, int R, int C, int CB, int LD = N>
__global__ void __launch_bounds__(CONV_THREADS, 1)
    k_conv_tc(const __grid_constant__ CUtensorMap tmx, const __grid_constant__ CUtensorMap tmw,
              const ConvShape sh, const ConvEpi epi, int *err) {
  extern __shared__ uint8_t smem_raw[];
  const uint32_t raw = tc::smem_u32(smem_raw);
  const uint32_t base = (raw + 1023u) & ~1023u;
  constexpr int nwt = R * C * CB;  // resident weight tiles
  // A windows: S slots, S / MMA_WARPS in each MMA warp's own ring. The warps
  // take alternate tiles; with one shared ring a warp would skip the other's
  // windows and could wait on a slot's barrier a whole phase ahead of the
  // last one it saw, where a parity wait passes on the stale phase.
  const int S = sh.stages;
  const int Sm = S / MMA_WARPS;
  const uint32_t w_tile = (uint32_t)N * 128u;
  const uint32_t w_base = base;
  const uint32_t a_base = w_base + (uint32_t)nwt * w_tile;
  const uint32_t bar0 = a_base + (uint32_t)S * WIN_BYTES;
  // TMEM accumulators: ACC buffers of N columns within TMEM_COLS_CONV
  constexpr int ACC = (int)TMEM_COLS_CONV / N;
  // barriers: full[S], empty[S], tfull[ACC], tempty[ACC], weights, fin
  const uint32_t full0 = bar0, empty0 = bar0 + 8u * S, tfull0 = bar0 + 16u * S,
                 tempty0 = tfull0 + 8u * ACC, wbar = tempty0 + 8u * ACC, fin = wbar + 8u;
  uint8_t *tail = smem_raw + (bar0 + 256u - raw);
  uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(tail);
  volatile int *abort = reinterpret_cast<volatile int *>(tmem_slot + 1);
  float *sbias = reinterpret_cast<float *>(tail + 256);
  float *swo = sbias + 128;  // [64]
  uint4 *epi_stage = reinterpret_cast<uint4 *>(smem_raw + (bar0 + CONV_SMEM_TAIL - raw));

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    for (int s = 0; s < S; ++s) {
      tc::mbar_init(full0 + 8u * s, 1);
      tc::mbar_init(empty0 + 8u * s, 1);
    }
    for (int b = 0; b < ACC; ++b) {
      tc::mbar_init(tfull0 + 8u * b, 1);
      tc::mbar_init(tempty0 + 8u * b, EPI_WARPS);
    }
    tc::mbar_init(wbar, 1);
    tc::mbar_init(fin, MMA_WARPS);
    *abort = 0;
    tc::fence_barrier_init();
  }
  const int c_base = N == LD ? 0 : (int)blockIdx.y * N;
  for (int k = threadIdx.x; k < N; k += blockDim.x) sbias[k] = epi.bias ? epi.bias[c_base + k] : 0.0f;
  for (int k = threadIdx.x; k < 64; k += blockDim.x) swo[k] = epi.wo ? epi.wo[k] : 0.0f;
  if (warp == 1) tc::tmem_alloc(tc::smem_u32(tmem_slot), TMEM_COLS_CONV);
  tc::fence_before_sync();
  __syncthreads();
  tc::fence_after_sync();
  const uint32_t tmem = *tmem_slot;
  const int wtiles = sh.W >> 7;
  tc::pdl_trigger();

  if (warp == 0) {
    if (lane == 0) {
      // ---- TMA producer: resident weights once, then one A tile per K block
      tc::prefetch_map(&tmx);
      tc::prefetch_map(&tmw);
      tc::mbar_arrive_expect_tx(wbar, (uint32_t)nwt * w_tile);
      for (int t = 0; t < R * C; ++t)
        for (int cb = 0; cb < CB; ++cb)
          tc::tma_load_2d(w_base + (uint32_t)(t * CB + cb) * w_tile, &tmw, wbar, cb * 64, t * LD + c_base);
      tc::pdl_wait();  // the weights are older than the kernel before
      // windows issued so far to each MMA warp's ring
      uint32_t issued[MMA_WARPS] = {};
      int local = 0;
      for (int tile = blockIdx.x; tile < sh.n_tiles; tile += gridDim.x, ++local) {
        const int m = local % MMA_WARPS;
        const int wb = tile % wtiles, bh = tile / wtiles;
        const int h = bh % sh.H, b = bh / sh.H;
        for (int r = 0; r < R; ++r)
          for (int cb = 0; cb < CB; ++cb) {
            const uint32_t n = issued[m];
            const uint32_t slot = (uint32_t)(m * Sm) + n % (uint32_t)Sm;
            const uint32_t ph = (n / (uint32_t)Sm) & 1u;
            if (!tc::mbar_wait(empty0 + 8u * slot, ph ^ 1u, abort)) goto produced;
            tc::mbar_arrive_expect_tx(full0 + 8u * slot, WIN_BYTES);
            tc::tma_load_4d(a_base + slot * WIN_BYTES, &tmx, full0 + 8u * slot, cb * 64,
                            wb * 128 - WIN_RADIUS, h + (r - R / 2) * sh.step_h, b);
            issued[m] = n + 1u;
          }
      }
    produced:
      // nothing may still be landing in shared memory when the CTA exits:
      // wait for the last (up to Sm) windows issued to each ring
      tc::mbar_drain(wbar, 0);
      for (int m = 0; m < MMA_WARPS; ++m)
        for (uint32_t n = issued[m] - min(issued[m], (uint32_t)Sm); n < issued[m]; ++n)
          tc::mbar_drain(full0 + 8u * ((uint32_t)(m * Sm) + n % (uint32_t)Sm),
                         (n / (uint32_t)Sm) & 1u);
    }
  } else if (warp <= MMA_WARPS) {
    if (lane == 0) {
      // ---- MMA issuer m takes the CTA's tiles local = m, m + MMA_WARPS, ...
      const int m = warp - 1;
      constexpr uint32_t idesc = tc::idesc_bf16(128, N, false, false);
      // descriptor bits other than the start address (bits 0-13; shared
      // memory addresses are below 2^18)
      const uint64_t desc_hi = tc::sdesc(0u, 16u, 1024u);
      constexpr uint32_t KB = (uint32_t)(R * CB);  // windows per tile
      int local = m;
      if (tc::mbar_wait(wbar, 0, abort)) {
        for (int tile = blockIdx.x + m * gridDim.x; tile < sh.n_tiles;
             tile += MMA_WARPS * gridDim.x, local += MMA_WARPS) {
          const int buf = local % ACC;
          if (!tc::mbar_wait(tempty0 + 8u * buf, (((uint32_t)(local / ACC)) & 1u) ^ 1u, abort)) break;
          tc::fence_after_sync();
          // this tile's windows: indices (local / MMA_WARPS) * KB ... of this
          // warp's own ring
          const uint32_t n0 = (uint32_t)(local / MMA_WARPS) * KB;
          int s = (int)(n0 % (uint32_t)Sm);
          uint32_t ph = (n0 / (uint32_t)Sm) & 1u;
          const uint32_t d = tmem + (uint32_t)(buf * N);
          uint32_t acc = 0;
          bool ok = true;
#pragma unroll 1
          for (int r = 0; r < R && ok; ++r)
#pragma unroll
            for (int cb = 0; cb < CB; ++cb) {
              const uint32_t slot = (uint32_t)(m * Sm + s);
              if (!tc::mbar_wait(full0 + 8u * slot, ph, abort)) {
                ok = false;
                break;
              }
              tc::fence_after_sync();
              const uint32_t win = a_base + slot * WIN_BYTES;
#pragma unroll
              for (int c = 0; c < C; ++c) {
                const uint32_t a0 = win + (uint32_t)(WIN_RADIUS + (c - C / 2) * sh.step_w) * 128u;
                const uint32_t b0 = w_base + (uint32_t)(((r * C + c) * CB + cb)) * w_tile;
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                  tc::mma_bf16(d, desc_hi | ((a0 + 32u * k) >> 4), desc_hi | ((b0 + 32u * k) >> 4), idesc, acc);
                  acc = 1;
                }
              }
              tc::mma_commit(empty0 + 8u * slot);
              if (++s == Sm) {
                s = 0;
                ph ^= 1u;
              }
            }
          if (!ok) break;
          tc::mma_commit(tfull0 + 8u * buf);
        }
      }
      tc::mma_commit(fin);
      tc::mbar_drain(fin, 0);
    }
  } else {
    // ---- epilogue: warp w reads TMEM lanes 32 (w mod 4) .. +31, half of the columns
    const int q = warp & 3;
    const int half = (warp - 1 - MMA_WARPS) >> 2;
    const int row = q * 32 + lane;
    int local = 0;
    tc::pdl_wait();
    for (int tile = blockIdx.x; tile < sh.n_tiles; tile += gridDim.x, ++local) {
      const int buf = local % ACC;
      const uint32_t use = (uint32_t)(local / ACC);
      const int wb = tile % wtiles, bh = tile / wtiles;
      const size_t p = (size_t)bh * sh.W + (size_t)wb * 128 + row;
      EpiLoads<N> ld;
      uint4 *stage = epi_stage + (warp - 1 - MMA_WARPS) * (EPI_STAGE_BYTES / 16);
      conv_epilogue_load<N, LD>(epi, p, c_base, half, ld, stage);  // before the accumulator is ready
      if (!tc::mbar_wait(tfull0 + 8u * buf, use & 1u, abort)) break;
      tc::fence_after_sync();
      const uint32_t taddr = tmem + ((uint32_t)(q * 32) << 16) + (uint32_t)(buf * N);
      const float dot = conv_epilogue_row<N, LD>(epi, sbias, swo, p, c_base, half, taddr, ld, stage);
      tc::fence_before_sync();
      __syncwarp();
      if (lane == 0) tc::mbar_arrive(tempty0 + 8u * buf);
      // the two halves of a row add their partial dots to the zeroed y: a sum
      // of two terms onto zero does not depend on their order
      if (epi.y) atomicAdd(epi.y + p, half == 0 ? dot + epi.bo[0] : dot);
    }
  }
  tc::fence_before_sync();
  __syncthreads();
  if (warp == 1) {
    tc::fence_after_sync();
    tc::tmem_dealloc(tmem, TMEM_COLS_CONV);
  }
  if (threadIdx.x == 0 && *abort) atomicOr(err, 1);
}

// ------------------------------------------------------------------ 3x3 convolution, 64 channels

// The head's 3x3 convolution (64 -> 64 channels) with every input row read
// once. A CTA walks down runs of output rows that are step_h apart; the window
// of one input row is multiplied by the three taps of a column at once
// (N = 192: the weights of tap rows 2, 1, 0 one after the other) into the
// accumulators of the three output rows it belongs to, which lie side by side
// in TMEM. Against one output row at a time (k_conv_tc, N = 64) the tensor
// core reads 4 KB of pixels and 6 KB of weights for three taps instead of
// 3 x (4 + 2) KB: a 128 x 64 x 16 MMA is bound by these reads (48 cycles), a
// 128 x 192 x 16 one by the multipliers (96); and a window is copied from L2
// once instead of three times.
//
// An output row receives its tap rows in the order 0, 1, 2, each column by
// column, as in k_conv_tc, so the FP32 sums have the same bits.
//
// Measured on a GB300, 128 maps of 256^2, a forward layer, us: k_conv_tc 640;
// this kernel with one issuing lane inside a divergent branch 485, with the
// issue loop run by the converged warp 400. What bounds it now: HBM (2.2 GB read
// and written: 330 us at the measured copy rate) with the MMAs (250 us) close
// behind. Running six layers over groups of images small enough for L2 was
// slower (8.7 instead of 7.7 ms for 300 maps at 8 images a group): a launch
// costs 5 us to fill and drain the pipeline.
constexpr int ROWS_SLOTS = 8;       // accumulators of 64 TMEM columns
constexpr int ROWS_GROUPS = 2;      // groups of EPI_WARPS, taking alternate output rows
constexpr int ROWS_THREADS = 32 * (2 + ROWS_GROUPS * EPI_WARPS);
constexpr uint32_t ROWS_W_BYTES = 9u * 64u * 128u;

// Which fields of the epilogue apply. ROWS_FORWARD: bias, relu, mask_out,
// resid, out and the output layer; ROWS_GRADIENT: resid_f32, resid_dy, out_f32,
// mask_in, out.
enum : int { ROWS_FORWARD = 0, ROWS_GRADIENT = 1 };

// input windows in shared memory, and the staging tile of an epilogue warp's
// 32 pixels x 32 channels (BF16 or FP32)
__host__ __device__ constexpr int rows_stages(int kind) { return kind == ROWS_FORWARD ? 6 : 4; }
__host__ __device__ constexpr uint32_t rows_stage_bytes(int kind) {
  return kind == ROWS_FORWARD ? 2048u : 4096u;
}
__host__ __device__ constexpr uint32_t rows_smem_bytes(int kind) {
  return 1024u + ROWS_W_BYTES + (uint32_t)rows_stages(kind) * WIN_BYTES + CONV_SMEM_TAIL +
         (uint32_t)(ROWS_GROUPS * EPI_WARPS) * rows_stage_bytes(kind);
}

struct RowsShape {
  int H, W;    // W: a multiple of 128
  int d, sgn;  // tap rows read input row h + (r - 1) sgn d
  int step_w;
  int total;  // rows shared out: of 128 pixels (k_conv_rows: images * (W / 128) * H)
              // or whole (k_wgrad_rows: images * H)
};

// A run of output rows: row q (0 .. n - 1) is image row h0 + sgn d q of the
// 128-pixel column block wb of image b.
struct RowRun {
  int b, wb, h0, n;
};

// Rows h = c, c + d, ... of one image or column block are its class c; position
// g counts the rows class by class. The class of position g (made the position
// within the class), and the class's number of rows.
__device__ __forceinline__ int rows_class(const RowsShape &sh, int &g, int &nc) {
  int c = 0;
  for (;; ++c) {
    nc = (sh.H - c + sh.d - 1) / sh.d;
    if (g < nc) return c;
    g -= nc;
  }
}

__device__ __forceinline__ int rows_begin(const RowsShape &sh, int c, int g, int nc) {
  return sh.sgn > 0 ? c + g * sh.d : c + (nc - 1 - g) * sh.d;
}

// The run at flat row f (column block by column block), at most to f1; f moves
// behind it.
__device__ __forceinline__ bool rows_next(const RowsShape &sh, int &f, int f1, RowRun &r) {
  if (f >= f1) return false;
  const int col = f / sh.H, wt = sh.W >> 7;
  int g = f - col * sh.H, nc;
  const int c = rows_class(sh, g, nc);
  r.b = col / wt;
  r.wb = col - r.b * wt;
  r.n = min(nc - g, f1 - f);
  r.h0 = rows_begin(sh, c, g, nc);
  f += r.n;
  return true;
}

// The same for whole image rows f .. f1 (image by image): the run of the next
// column block wb, f moving on after the last one.
__device__ __forceinline__ bool bands_next(const RowsShape &sh, int &f, int &wb, int f1, RowRun &r) {
  if (f >= f1) return false;
  r.b = f / sh.H;
  int g = f - r.b * sh.H, nc;
  const int c = rows_class(sh, g, nc);
  r.wb = wb;
  r.n = min(nc - g, f1 - f);
  r.h0 = rows_begin(sh, c, g, nc);
  if (++wb == (sh.W >> 7)) {
    wb = 0;
    f += r.n;
  }
  return true;
}

// 32 FP32 channels of 32 pixels, one pixel a lane, to or from global memory
// through the warp's staging tile: an instruction moves 4 pixels' contiguous
// 128 bytes (16-byte chunks XOR-swizzled by pixel against bank conflicts).
__device__ __forceinline__ void rows_load_f32(const float *src, size_t pbase, int c0, float4 *r) {
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int i = 0; i < 8; ++i)
    r[i] = reinterpret_cast<const float4 *>(src + (pbase + (size_t)(4 * i + (lane >> 3))) * 64 +
                                            c0)[lane & 7];
}

__device__ __forceinline__ void rows_add_f32(const float4 *r, float *v, float4 *stage) {
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const int pr = 4 * i + (lane >> 3);
    stage[pr * 8 + ((lane & 7) ^ (pr & 7))] = r[i];
  }
  __syncwarp();
#pragma unroll
  for (int k = 0; k < 8; ++k) {
    const float4 q = stage[lane * 8 + (k ^ (lane & 7))];
    v[4 * k] += q.x;
    v[4 * k + 1] += q.y;
    v[4 * k + 2] += q.z;
    v[4 * k + 3] += q.w;
  }
  __syncwarp();
}

__device__ __forceinline__ void rows_store_f32(float *dst, size_t pbase, int c0, const float *v,
                                               float4 *stage) {
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int k = 0; k < 8; ++k)
    stage[lane * 8 + (k ^ (lane & 7))] =
        make_float4(v[4 * k], v[4 * k + 1], v[4 * k + 2], v[4 * k + 3]);
  __syncwarp();
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const int pr = 4 * i + (lane >> 3);
    reinterpret_cast<float4 *>(dst + (pbase + (size_t)pr) * 64 + c0)[lane & 7] =
        stage[pr * 8 + ((lane & 7) ^ (pr & 7))];
  }
  __syncwarp();
}

// tmx: 4-D map over the input {64, W, H, B} with box {64, WIN_ROWS, 1, 1};
// tmw: 2-D map over the weights {64, 9 x 64} with box {64, 64}; 128-byte
// swizzle. Grid: at most one CTA per SM; each takes an equal share of the rows.
// Warp 0: TMA, warp 1: MMA issue, warps 2-17: epilogue, two groups of eight that
// take alternate rows (one group's serial chain of an accumulator load, the
// arithmetic and the stores took 2600 cycles a row, the MMAs 1200). In
// ROWS_FORWARD they also hold on to the windows: a residual that is the
// convolution's own input is read there.
template <int KIND>
__global__ void __launch_bounds__(ROWS_THREADS, 1)
    k_conv_rows(const __grid_constant__ CUtensorMap tmx, const __grid_constant__ CUtensorMap tmw,
                const RowsShape sh, const ConvEpi e, int *err) {
  extern __shared__ uint8_t smem_raw[];
  const uint32_t raw = tc::smem_u32(smem_raw);
  const uint32_t base = (raw + 1023u) & ~1023u;
  constexpr int S = rows_stages(KIND);
  const uint32_t w_base = base;
  const uint32_t a_base = w_base + ROWS_W_BYTES;
  const uint32_t bar0 = a_base + (uint32_t)S * WIN_BYTES;
  // barriers: full[S], empty[S], tfull[8], tempty[8], weights, fin
  const uint32_t full0 = bar0, empty0 = bar0 + 8u * S, tfull0 = bar0 + 16u * S,
                 tempty0 = tfull0 + 8u * ROWS_SLOTS, wbar = tempty0 + 8u * ROWS_SLOTS, fin = wbar + 8u;
  uint8_t *tail = smem_raw + (bar0 + 256u - raw);
  uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(tail);
  volatile int *abort = reinterpret_cast<volatile int *>(tmem_slot + 1);
  float *sbias = reinterpret_cast<float *>(tail + 256);
  float *swo = sbias + 128;
  uint4 *epi_stage = reinterpret_cast<uint4 *>(smem_raw + (bar0 + CONV_SMEM_TAIL - raw));

  const int warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    for (int s = 0; s < S; ++s) {
      tc::mbar_init(full0 + 8u * s, 1);
      tc::mbar_init(empty0 + 8u * s, KIND == ROWS_FORWARD ? 1 + EPI_WARPS : 1);
    }
    for (int b = 0; b < ROWS_SLOTS; ++b) {
      tc::mbar_init(tfull0 + 8u * b, 1);
      tc::mbar_init(tempty0 + 8u * b, EPI_WARPS);
    }
    tc::mbar_init(wbar, 1);
    tc::mbar_init(fin, 1);
    *abort = 0;
    tc::fence_barrier_init();
  }
  if (threadIdx.x < 64) {
    sbias[threadIdx.x] = e.bias ? e.bias[threadIdx.x] : 0.0f;
    swo[threadIdx.x] = e.wo ? e.wo[threadIdx.x] : 0.0f;
  }
  if (warp == 1) tc::tmem_alloc(tc::smem_u32(tmem_slot), 64u * ROWS_SLOTS);
  tc::fence_before_sync();
  __syncthreads();
  tc::fence_after_sync();
  const uint32_t tmem = *tmem_slot;
  int f = (int)((long long)sh.total * blockIdx.x / gridDim.x);
  const int f1 = (int)((long long)sh.total * (blockIdx.x + 1) / gridDim.x);
  RowRun run;
  tc::pdl_trigger();

  if (warp == 0) {
    if (lane == 0) {
      tc::prefetch_map(&tmx);
      tc::prefetch_map(&tmw);
      // tap (r, c) goes to tile 3 c + 2 - r: the taps of a column side by side
      tc::mbar_arrive_expect_tx(wbar, ROWS_W_BYTES);
      for (int r = 0; r < 3; ++r)
        for (int c = 0; c < 3; ++c)
          tc::tma_load_2d(w_base + (uint32_t)(3 * c + 2 - r) * 8192u, &tmw, wbar, 0, (3 * r + c) * 64);
      tc::pdl_wait();  // the weights are older than the kernel before
      uint32_t n = 0;  // windows issued
      bool ok = true;
      while (ok && rows_next(sh, f, f1, run)) {
        for (int j = 0; j < run.n + 2; ++j, ++n) {
          const uint32_t slot = n % (uint32_t)S;
          if (!tc::mbar_wait(empty0 + 8u * slot, ((n / (uint32_t)S) & 1u) ^ 1u, abort)) {
            ok = false;
            break;
          }
          tc::mbar_arrive_expect_tx(full0 + 8u * slot, WIN_BYTES);
          tc::tma_load_4d(a_base + slot * WIN_BYTES, &tmx, full0 + 8u * slot, 0,
                          run.wb * 128 - WIN_RADIUS, run.h0 + (j - 1) * sh.sgn * sh.d, run.b);
        }
      }
      // nothing may still be landing in shared memory when the CTA exits
      tc::mbar_drain(wbar, 0);
      for (uint32_t k = n - min(n, (uint32_t)S); k < n; ++k)
        tc::mbar_drain(full0 + 8u * (k % (uint32_t)S), (k / (uint32_t)S) & 1u);
    }
  } else if (warp == 1) {
    // the whole warp runs the loop, so that the descriptors stay in uniform
    // registers; lane 0 issues
    const uint32_t mine = lane == 0 ? 1u : 0u;
    {
      constexpr uint32_t id64 = tc::idesc_bf16(128, 64, false, false);
      const uint64_t desc_hi = tc::sdesc(0u, 16u, 1024u);
      const uint32_t col_step = (uint32_t)(sh.step_w * 128);
      uint32_t s = 0, ph = 0;  // window slot and phase
      uint32_t q0 = 0;         // output rows of the runs before
      bool ok = tc::mbar_wait(wbar, 0, abort);
      while (ok && rows_next(sh, f, f1, run)) {
        const int n = run.n;
        for (int j = 0; j < n + 2; ++j) {
          // input row j belongs to output rows j - 2 .. j
          const int lo = max(0, j - 2), n_old = min(n - 1, j - 1) - lo + 1;
          const bool fresh = j < n;
          const uint32_t qn = q0 + (uint32_t)j;
          if (fresh &&
              !tc::mbar_wait(tempty0 + 8u * (qn % ROWS_SLOTS), ((qn / ROWS_SLOTS) & 1u) ^ 1u, abort)) {
            ok = false;
            break;
          }
          if (!tc::mbar_wait(full0 + 8u * s, ph, abort)) {
            ok = false;
            break;
          }
          tc::fence_after_sync();
          const uint32_t a0 = a_base + s * WIN_BYTES + WIN_RADIUS * 128u - col_step;
          // accumulators [lo .. j] in TMEM; those that wrap around its end
          // take a second instruction
          const uint32_t slot = (q0 + (uint32_t)lo) % ROWS_SLOTS;
          const uint32_t cnt = (uint32_t)n_old + (fresh ? 1u : 0u);
          const uint32_t n1 = min(cnt, (uint32_t)ROWS_SLOTS - slot), n2 = cnt - n1;
          const uint32_t b0 = w_base + (uint32_t)(lo - (j - 2)) * 8192u;
          const uint32_t d1 = tmem + slot * 64u;
          // N = 64 x accumulators: the descriptor's N field counts units of 8
          const uint32_t id1 = id64 + ((n1 - 1u) << 20), id2 = id64 + ((n2 - 1u) << 20);
          // the first instruction of the new row starts its accumulator
          const uint32_t o1 = min((uint32_t)n_old, (uint32_t)ROWS_SLOTS - slot), o2 = (uint32_t)n_old - o1;
          const uint64_t ad = desc_hi | (a0 >> 4), bd = desc_hi | (b0 >> 4);
          if (o1) tc::mma_bf16_warp(mine, d1, ad, bd, id64 + ((o1 - 1u) << 20), 1u);
          if (o2) tc::mma_bf16_warp(mine, tmem, ad, bd + o1 * 512u, id64 + ((o2 - 1u) << 20), 1u);
          if (fresh)
            tc::mma_bf16_warp(mine, tmem + (qn % ROWS_SLOTS) * 64u, ad, bd + (uint32_t)n_old * 512u, id64, 0u);
          if (n2 == 0u) {
#pragma unroll
            for (int t = 1; t < 12; ++t) {
              const int c = t >> 2, k = t & 3;
              tc::mma_bf16_warp(mine, d1, desc_hi | ((a0 + (uint32_t)c * col_step + 32u * k) >> 4),
                           bd + (uint32_t)(c * 1536 + 2 * k), id1, 1u);
            }
          } else {
#pragma unroll
            for (int t = 1; t < 12; ++t) {
              const int c = t >> 2, k = t & 3;
              const uint64_t a = desc_hi | ((a0 + (uint32_t)c * col_step + 32u * k) >> 4);
              const uint64_t b = bd + (uint32_t)(c * 1536 + 2 * k);
              tc::mma_bf16_warp(mine, d1, a, b, id1, 1u);
              tc::mma_bf16_warp(mine, tmem, a, b + n1 * 512u, id2, 1u);
            }
          }
          tc::mma_commit_warp(mine, empty0 + 8u * s);
          if (j >= 2) tc::mma_commit_warp(mine, tfull0 + 8u * ((qn - 2u) % ROWS_SLOTS));
          if (++s == (uint32_t)S) {
            s = 0;
            ph ^= 1u;
          }
        }
        q0 += (uint32_t)n;
      }
      tc::mma_commit_warp(mine, fin);
      tc::mbar_drain(fin, 0);
    }
  } else {
    // ---- epilogue: warp w reads TMEM lanes 32 (w mod 4) .. +31, half of the columns
    const int qd = warp & 3, half = ((warp - 2) >> 2) & 1, group = (warp - 2) >> 3;
    const int c0 = 32 * half, row = qd * 32 + lane;
    uint4 *stage = epi_stage + (warp - 2) * (rows_stage_bytes(KIND) / 16);
    uint32_t q = 0;  // output rows
    uint32_t w = 0;  // windows
    // Every window is released by one group (and by the MMAs that read it),
    // after it has been filled: an arrival before that would count for the
    // slot's previous window. A group waits for windows at most six apart
    // (the MMAs of its row before have read all up to five behind), so the
    // parity names the right phase.
    auto window_wait = [&](uint32_t n) {
      return tc::mbar_wait(full0 + 8u * (n % (uint32_t)S), (n / (uint32_t)S) & 1u, abort);
    };
    // The fence orders a lane's reads before the copy that the arrival allows:
    // without it (and with the loads' values not yet used) the arrival overtook
    // them, and one pass in fifteen returned wrong pixels.
    auto window_done = [&](uint32_t n) {
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      __syncwarp();
      if (lane == 0) tc::mbar_arrive(empty0 + 8u * (n % (uint32_t)S));
    };
    bool ok = true;
    tc::pdl_wait();
    while (ok && rows_next(sh, f, f1, run)) {
      for (int k = 0; k < run.n; ++k, ++q) {
        if ((int)(q % ROWS_GROUPS) != group) continue;
        const size_t pb = ((size_t)run.b * sh.H + (run.h0 + k * sh.sgn * sh.d)) * sh.W +
                          (size_t)run.wb * 128 + qd * 32;
        const size_t p = pb + lane;
        const uint32_t slot = q % ROWS_SLOTS, own = w + (uint32_t)k + 1u;  // own row's window
        if (KIND == ROWS_FORWARD && k == 0) {  // the halo row above the run
          if (!window_wait(w)) {
            ok = false;
            break;
          }
          window_done(w);
        }
        // global inputs, before the accumulator is ready
        uint4 rb[4];
        float4 rf[8];
        uint32_t mi = 0;
        float rdy = 0.0f;
        if (KIND == ROWS_FORWARD) {
          if (e.resid && !e.resid_is_input) load_row_bf16x32<64>(e.resid, pb, c0, rb, stage);
        } else {
          if (e.resid_f32) rows_load_f32(e.resid_f32, pb, c0, rf);
          if (e.mask_in) mi = e.mask_in[p * 2 + half];
          if (e.resid_dy) rdy = e.resid_dy[p];
        }
        if ((KIND == ROWS_FORWARD && !window_wait(own)) ||
            !tc::mbar_wait(tfull0 + 8u * slot, (q / ROWS_SLOTS) & 1u, abort)) {
          ok = false;
          break;
        }
        if (KIND == ROWS_FORWARD) {
          if (e.resid_is_input) {
            // this row's own pixels lie in the window it was computed from
            const uint4 *win =
                reinterpret_cast<const uint4 *>(smem_raw + (a_base + (own % (uint32_t)S) * WIN_BYTES - raw)) +
                (WIN_RADIUS + row) * 8;
#pragma unroll
            for (int t = 0; t < 4; ++t) rb[t] = win[(4 * half + t) ^ ((WIN_RADIUS + row) & 7)];
          }
        }
        tc::fence_after_sync();
        float v[32];
        tc::tmem_ld32(tmem + ((uint32_t)(qd * 32) << 16) + slot * 64u + (uint32_t)c0, v);
        tc::fence_before_sync();
        __syncwarp();
        if (lane == 0) tc::mbar_arrive(tempty0 + 8u * slot);
        const float4 *w4 = reinterpret_cast<const float4 *>(swo + c0);
        if (KIND == ROWS_FORWARD) {
          const float4 *b4 = reinterpret_cast<const float4 *>(sbias + c0);
#pragma unroll
          for (int i = 0; i < 8; ++i) {
            const float4 b = b4[i];
            v[4 * i] += b.x;
            v[4 * i + 1] += b.y;
            v[4 * i + 2] += b.z;
            v[4 * i + 3] += b.w;
          }
          if (e.mask_out) {
            uint32_t bits = 0;
#pragma unroll
            for (int i = 0; i < 32; ++i) bits |= (v[i] > 0.0f ? 1u : 0u) << i;
            e.mask_out[p * 2 + half] = bits;
          }
          if (e.relu) {
#pragma unroll
            for (int i = 0; i < 32; ++i) v[i] = fmaxf(v[i], 0.0f);
          }
          if (e.resid) {
#pragma unroll
            for (int i = 0; i < 4; ++i) {
              const uint32_t r[4] = {rb[i].x, rb[i].y, rb[i].z, rb[i].w};
#pragma unroll
              for (int t = 0; t < 4; ++t) {
                v[8 * i + 2 * t] += bf_lo(r[t]);
                v[8 * i + 2 * t + 1] += bf_hi(r[t]);
              }
            }
          }
          window_done(own);
          if (e.y) {
            float dot = 0.0f;
#pragma unroll
            for (int i = 0; i < 8; ++i) {
              const float4 o = w4[i];
              dot = fmaf(o.x, __bfloat162float(__float2bfloat16_rn(v[4 * i])), dot);
              dot = fmaf(o.y, __bfloat162float(__float2bfloat16_rn(v[4 * i + 1])), dot);
              dot = fmaf(o.z, __bfloat162float(__float2bfloat16_rn(v[4 * i + 2])), dot);
              dot = fmaf(o.w, __bfloat162float(__float2bfloat16_rn(v[4 * i + 3])), dot);
            }
            // two terms onto the zeroed y: their order does not matter
            atomicAdd(e.y + p, half == 0 ? dot + e.bo[0] : dot);
          }
        } else {
          if (e.resid_f32) rows_add_f32(rf, v, reinterpret_cast<float4 *>(stage));
          if (e.resid_dy) {
#pragma unroll
            for (int i = 0; i < 8; ++i) {
              const float4 o = w4[i];
              v[4 * i] = fmaf(rdy, o.x, v[4 * i]);
              v[4 * i + 1] = fmaf(rdy, o.y, v[4 * i + 1]);
              v[4 * i + 2] = fmaf(rdy, o.z, v[4 * i + 2]);
              v[4 * i + 3] = fmaf(rdy, o.w, v[4 * i + 3]);
            }
          }
          if (e.out_f32) rows_store_f32(e.out_f32, pb, c0, v, reinterpret_cast<float4 *>(stage));
          if (e.mask_in) {
#pragma unroll
            for (int i = 0; i < 32; ++i) v[i] = ((mi >> i) & 1u) ? v[i] : 0.0f;
          }
        }
        if (e.out) store_row_bf16x32<64>(e.out, pb, c0, v, stage);
        if (KIND == ROWS_FORWARD && k == run.n - 1) {  // the halo row below it
          if (!window_wait(own + 1u)) {
            ok = false;
            break;
          }
          window_done(own + 1u);
        }
      }
      w += (uint32_t)run.n + 2u;
    }
  }
  tc::fence_before_sync();
  __syncthreads();
  if (warp == 1) {
    tc::fence_after_sync();
    tc::tmem_dealloc(tmem, 64u * ROWS_SLOTS);
  }
  if (threadIdx.x == 0 && *abort) atomicOr(err, 1);
}

// ------------------------------------------------------------------ weight gradients

constexpr int MAX_ATOMS = 20;
constexpr int WG_THREADS = 192;
constexpr int WG_STAGES = 2;
constexpr uint32_t WG_TILE = 64u * 128u;  // 64 pixels x 64 BF16 channels

struct WgradShape {
  int B, H, W;          // image; W is a multiple of 64
  int N;                // dY channels (output channels of the layer): 64 or 128
  int n_atoms;          // even; X atoms first, then all-ones atoms
  int n_x;              // X atoms: (tap, input channel block), tap-major
  int jobs_per_group;   // atom pairs per CTA (grid.y = groups)
  int tmem_cols;        // power of two >= jobs_per_group * N
  int kb_total;         // B * H * W / 64
  int kb_per_cta;
  int dh[MAX_ATOMS], dw[MAX_ATOMS], cb[MAX_ATOMS];
};

__host__ __device__ constexpr uint32_t wgrad_smem_bytes(int N, int jobs_per_group) {
  return 1024u + (uint32_t)WG_STAGES * (uint32_t)(N / 64 + 2 * jobs_per_group) * WG_TILE + 2u * WG_TILE +
         256u;
}

// Partial sums: partial[blockIdx.x][atom][co][row of the atom (input channel)].
// tmx: map over X {C_in, W, H, B}, tmy: map over dY {N, W, H, B}, both with
// box {64, 64, 1, 1} and 128-byte swizzle.
__global__ void __launch_bounds__(WG_THREADS, 1)
    k_wgrad_tc(const __grid_constant__ CUtensorMap tmx, const __grid_constant__ CUtensorMap tmy,
               const WgradShape sh, float *__restrict__ partial, int *err) {
  extern __shared__ uint8_t smem_raw[];
  const uint32_t raw = tc::smem_u32(smem_raw);
  const uint32_t base = (raw + 1023u) & ~1023u;
  const int N = sh.N, ny = N / 64;
  const int n_jobs = sh.n_atoms / 2;
  const int j0 = blockIdx.y * sh.jobs_per_group;
  const int j1 = min(j0 + sh.jobs_per_group, n_jobs);
  const int a0 = 2 * j0, a1 = 2 * j1;
  const int nxg = max(0, min(a1, sh.n_x) - a0);  // X atoms loaded by this CTA
  const uint32_t stage_bytes = (uint32_t)(ny + 2 * sh.jobs_per_group) * WG_TILE;
  const uint32_t ones_base = base + WG_STAGES * stage_bytes;
  const uint32_t bar0 = ones_base + 2u * WG_TILE;
  const uint32_t full0 = bar0, empty0 = bar0 + 8u * WG_STAGES, done = bar0 + 16u * WG_STAGES,
                 fin = done + 8u;
  uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(smem_raw + (fin + 8u - raw));
  volatile int *abort = reinterpret_cast<volatile int *>(tmem_slot + 1);
  auto atom_addr = [&](int a, int s) -> uint32_t {
    return a < sh.n_x ? base + (uint32_t)s * stage_bytes + (uint32_t)(ny + a - a0) * WG_TILE
                      : ones_base + (uint32_t)(a - sh.n_x) * WG_TILE;
  };

  const int kb_begin = blockIdx.x * sh.kb_per_cta;
  const int kb_end = min(kb_begin + sh.kb_per_cta, sh.kb_total);
  const int nkb = kb_end - kb_begin;

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  // all-ones tiles (BF16 1.0), written through the generic proxy
  {
    uint32_t *ones = reinterpret_cast<uint32_t *>(smem_raw + (ones_base - raw));
    for (uint32_t k = threadIdx.x; k < 2u * WG_TILE / 4u; k += blockDim.x) ones[k] = 0x3F803F80u;
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  if (threadIdx.x == 0) {
    for (int s = 0; s < WG_STAGES; ++s) {
      tc::mbar_init(full0 + 8u * s, 1);
      tc::mbar_init(empty0 + 8u * s, 1);
    }
    tc::mbar_init(done, 1);
    tc::mbar_init(fin, 1);
    *abort = 0;
    tc::fence_barrier_init();
  }
  if (warp == 1) tc::tmem_alloc(tc::smem_u32(tmem_slot), (uint32_t)sh.tmem_cols);
  tc::fence_before_sync();
  __syncthreads();
  tc::fence_after_sync();
  const uint32_t tmem = *tmem_slot;
  const int HW = sh.H * sh.W;
  tc::pdl_trigger();

  if (warp == 0) {
    if (lane == 0) {
      tc::prefetch_map(&tmx);
      tc::prefetch_map(&tmy);
      tc::pdl_wait();
      const uint32_t bytes = (uint32_t)(ny + nxg) * WG_TILE;
      int i = 0;
      for (; i < nkb; ++i) {
        const int s = i % WG_STAGES;
        const uint32_t r = (uint32_t)(i / WG_STAGES);
        if (!tc::mbar_wait(empty0 + 8u * s, (r & 1u) ^ 1u, abort)) break;
        const int px0 = (kb_begin + i) * 64;
        const int b = px0 / HW, rem = px0 - b * HW;
        const int h = rem / sh.W, w0 = rem - h * sh.W;
        const uint32_t fb = full0 + 8u * s;
        tc::mbar_arrive_expect_tx(fb, bytes);
        const uint32_t sb = base + (uint32_t)s * stage_bytes;
        for (int c = 0; c < ny; ++c) tc::tma_load_4d(sb + (uint32_t)c * WG_TILE, &tmy, fb, c * 64, w0, h, b);
        for (int a = a0; a < a0 + nxg; ++a)
          tc::tma_load_4d(sb + (uint32_t)(ny + a - a0) * WG_TILE, &tmx, fb, sh.cb[a] * 64, w0 + sh.dw[a],
                          h + sh.dh[a], b);
      }
      for (int k = max(0, i - WG_STAGES); k < i; ++k)
        tc::mbar_drain(full0 + 8u * (k % WG_STAGES), (uint32_t)(k / WG_STAGES) & 1u);
    }
  } else if (warp == 1) {
    if (lane == 0) {
      const uint32_t idesc = tc::idesc_bf16(128, N, true, true);
      bool ok = true;
      for (int i = 0; i < nkb; ++i) {
        const int s = i % WG_STAGES;
        const uint32_t r = (uint32_t)(i / WG_STAGES);
        if (!tc::mbar_wait(full0 + 8u * s, r & 1u, abort)) {
          ok = false;
          break;
        }
        tc::fence_after_sync();
        const uint32_t yb = base + (uint32_t)s * stage_bytes;
        for (int j = j0; j < j1; ++j) {
          const uint32_t xa = atom_addr(2 * j, s), xb = atom_addr(2 * j + 1, s);
          const uint32_t d = tmem + (uint32_t)((j - j0) * N);
#pragma unroll
          for (int k = 0; k < 4; ++k)
            tc::mma_bf16(d, tc::sdesc(xa + 2048u * k, xb - xa, 1024u), tc::sdesc(yb + 2048u * k, WG_TILE, 1024u),
                         idesc, (i | k) != 0 ? 1u : 0u);
        }
        tc::mma_commit(empty0 + 8u * s);
      }
      if (ok) tc::mma_commit(done);
      tc::mma_commit(fin);
      tc::mbar_drain(fin, 0);
    }
  } else {
    const int q = warp & 3;
    const int row = q * 32 + lane;
    tc::pdl_wait();
    if (nkb > 0 && tc::mbar_wait(done, 0, abort)) {
      tc::fence_after_sync();
      for (int j = j0; j < j1; ++j) {
        const int atom = 2 * j + (row >> 6);
        float *dst = partial + ((size_t)blockIdx.x * sh.n_atoms + atom) * (size_t)N * 64 + (row & 63);
        const uint32_t taddr = tmem + ((uint32_t)(q * 32) << 16) + (uint32_t)((j - j0) * N);
        for (int c0 = 0; c0 < N; c0 += 16) {
          float v[16];
          tc::tmem_ld16(taddr + (uint32_t)c0, v);
#pragma unroll
          for (int i = 0; i < 16; ++i) dst[(size_t)(c0 + i) * 64] = v[i];
        }
      }
    }
  }
  tc::fence_before_sync();
  __syncthreads();
  if (warp == 1) {
    tc::fence_after_sync();
    tc::tmem_dealloc(tmem, (uint32_t)sh.tmem_cols);
  }
  if (threadIdx.x == 0 && *abort) atomicOr(err, 2);
}

// Weight and bias gradients of the 3x3, 64 -> 64 channel convolution with every
// input row and every gradient row read once (k_wgrad_tc copies the input once a
// tap: 80 KB from L2 for 64 pixels, which bounds it). A CTA walks down the runs
// of a band of whole image rows, as many pixels as k_wgrad_tc gives a CTA: the
// tensor core's FP32 sums round towards zero, so their error grows with their
// length, and it stays what it was. One input row's window meets the gradient
// rows q = j - 2, j - 1, j it belongs to (tap rows 2, 1, 0) as one N = 192
// operand, 128 pixels deep; two column shifts of the window stack into M = 128,
// the third column and an all-ones block (the bias) into a second. Accumulators:
// 2 x 192 TMEM columns, tap row r in columns 64 (2 - r) of each.
//
// Measured on a GB300, 32 maps of 256^2, us a layer: k_wgrad_tc 237, this
// kernel 130; HBM floor 80 (537 MB), MMAs 83 (16 of 96 cycles a row of 128 pixels).
constexpr int WR_X = 4, WR_Y = 6;           // windows and gradient rows in shared memory
constexpr uint32_t WR_Y_BYTES = 128u * 128u;
constexpr int WR_ATOMS = 10;                // nine taps, all-ones

__host__ __device__ constexpr uint32_t wgrad_rows_smem_bytes() {
  return 1024u + WR_X * WIN_BYTES + (WR_Y + 1) * WR_Y_BYTES + 256u;
}

// partial[blockIdx.x][tap or ones][co][ci]. tmx: map over X {64, W, H, B} with
// box {64, WIN_ROWS, 1, 1}, tmy: map over dY with box {64, 64, 1, 1}; sh.step_w > 0.
__global__ void __launch_bounds__(WG_THREADS, 1)
    k_wgrad_rows(const __grid_constant__ CUtensorMap tmx, const __grid_constant__ CUtensorMap tmy,
                 const RowsShape sh, float *__restrict__ partial, int *err) {
  extern __shared__ uint8_t smem_raw[];
  const uint32_t raw = tc::smem_u32(smem_raw);
  const uint32_t x_base = (raw + 1023u) & ~1023u;
  const uint32_t y_base = x_base + WR_X * WIN_BYTES;
  const uint32_t ones_base = y_base + WR_Y * WR_Y_BYTES;
  const uint32_t bar0 = ones_base + WR_Y_BYTES;
  const uint32_t xfull = bar0, xempty = xfull + 8u * WR_X, yfull = xempty + 8u * WR_X,
                 yempty = yfull + 8u * WR_Y, done = yempty + 8u * WR_Y, fin = done + 8u;
  uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(smem_raw + (fin + 8u - raw));
  volatile int *abort = reinterpret_cast<volatile int *>(tmem_slot + 1);

  const int warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;
  {
    uint32_t *ones = reinterpret_cast<uint32_t *>(smem_raw + (ones_base - raw));
    for (uint32_t k = threadIdx.x; k < WR_Y_BYTES / 4u; k += blockDim.x) ones[k] = 0x3F803F80u;
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  if (threadIdx.x == 0) {
    for (int s = 0; s < WR_X; ++s) {
      tc::mbar_init(xfull + 8u * s, 1);
      tc::mbar_init(xempty + 8u * s, 1);
    }
    for (int s = 0; s < WR_Y; ++s) {
      tc::mbar_init(yfull + 8u * s, 1);
      tc::mbar_init(yempty + 8u * s, 1);
    }
    tc::mbar_init(done, 1);
    tc::mbar_init(fin, 1);
    *abort = 0;
    tc::fence_barrier_init();
  }
  if (warp == 1) tc::tmem_alloc(tc::smem_u32(tmem_slot), 512u);
  tc::fence_before_sync();
  __syncthreads();
  tc::fence_after_sync();
  const uint32_t tmem = *tmem_slot;
  int f = (int)((long long)sh.total * blockIdx.x / gridDim.x);
  const int f1 = (int)((long long)sh.total * (blockIdx.x + 1) / gridDim.x);
  RowRun run;
  int wb = 0;
  tc::pdl_trigger();

  if (warp == 0) {
    if (lane == 0) {
      tc::prefetch_map(&tmx);
      tc::prefetch_map(&tmy);
      tc::pdl_wait();
      uint32_t nx = 0, ny = 0;  // windows and gradient rows issued
      bool ok = true;
      while (ok && bands_next(sh, f, wb, f1, run)) {
        for (int j = 0; j < run.n + 2; ++j) {
          const int h = run.h0 + j * sh.sgn * sh.d;
          const uint32_t xs = nx % WR_X;
          if (!tc::mbar_wait(xempty + 8u * xs, ((nx / WR_X) & 1u) ^ 1u, abort)) {
            ok = false;
            break;
          }
          tc::mbar_arrive_expect_tx(xfull + 8u * xs, WIN_BYTES);
          tc::tma_load_4d(x_base + xs * WIN_BYTES, &tmx, xfull + 8u * xs, 0, run.wb * 128 - WIN_RADIUS,
                          h - sh.sgn * sh.d, run.b);
          ++nx;
          if (j >= run.n) continue;
          const uint32_t ys = ny % WR_Y;
          if (!tc::mbar_wait(yempty + 8u * ys, ((ny / WR_Y) & 1u) ^ 1u, abort)) {
            ok = false;
            break;
          }
          tc::mbar_arrive_expect_tx(yfull + 8u * ys, WR_Y_BYTES);
          for (int k = 0; k < 2; ++k)
            tc::tma_load_4d(y_base + ys * WR_Y_BYTES + (uint32_t)k * (WR_Y_BYTES / 2), &tmy, yfull + 8u * ys, 0,
                            run.wb * 128 + 64 * k, h, run.b);
          ++ny;
        }
      }
      for (uint32_t k = nx - min(nx, (uint32_t)WR_X); k < nx; ++k)
        tc::mbar_drain(xfull + 8u * (k % WR_X), (k / WR_X) & 1u);
      for (uint32_t k = ny - min(ny, (uint32_t)WR_Y); k < ny; ++k)
        tc::mbar_drain(yfull + 8u * (k % WR_Y), (k / WR_Y) & 1u);
    }
  } else if (warp == 1) {
    // the converged warp runs the loop (descriptors in uniform registers),
    // lane 0 issues
    const uint32_t mine = lane == 0 ? 1u : 0u;
    constexpr uint32_t id64 = tc::idesc_bf16(128, 64, true, true);
    const uint32_t col = (uint32_t)sh.step_w * 128u;
    uint32_t nx = 0, q0 = 0;
    bool ok = true, first = true;
    while (ok && bands_next(sh, f, wb, f1, run)) {
      const int n = run.n;
      for (int j = 0; j < n + 2; ++j, ++nx) {
        const uint32_t xs = nx % WR_X, qj = q0 + (uint32_t)j;
        if (!tc::mbar_wait(xfull + 8u * xs, (nx / WR_X) & 1u, abort) ||
            (j < n && !tc::mbar_wait(yfull + 8u * (qj % WR_Y), (qj / WR_Y) & 1u, abort))) {
          ok = false;
          break;
        }
        tc::fence_after_sync();
        const int lo = max(0, j - 2);
        const uint32_t cnt = (uint32_t)(min(n - 1, j) - lo + 1);
        const uint32_t ys = (q0 + (uint32_t)lo) % WR_Y;
        // gradient rows lo .. lo + cnt - 1 = tap rows j - lo, ...; those
        // beyond the ring's end take a second instruction
        const uint32_t n1 = min(cnt, (uint32_t)WR_Y - ys), n2 = cnt - n1;
        const uint32_t d0 = tmem + 64u * (uint32_t)(2 - (j - lo));
        const uint32_t a0 = x_base + xs * WIN_BYTES + WIN_RADIUS * 128u - col;
        const uint64_t ad0 = tc::sdesc(a0, col, 1024u);
        const uint64_t ad1 = tc::sdesc(a0 + 2u * col, ones_base - (a0 + 2u * col), 1024u);
        const uint64_t bd1 = tc::sdesc(y_base + ys * WR_Y_BYTES, WR_Y_BYTES, 1024u);
        const uint64_t bd2 = tc::sdesc(y_base, WR_Y_BYTES, 1024u);
        const uint32_t id1 = id64 + ((n1 - 1u) << 20), id2 = id64 + ((n2 - 1u) << 20);
        if (first && j <= 2) {
          // row lo = 0 meets tap row j for the first time: its first
          // instruction starts the accumulator
          for (uint32_t p = 0; p < 2; ++p) {
            const uint64_t ad = p ? ad1 : ad0;
            const uint32_t d = d0 + 192u * p;
            for (uint32_t k = 0; k < 8; ++k)
              for (uint32_t g = 0; g < cnt; ++g) {
                const uint64_t bd = g < n1 ? bd1 + g * (WR_Y_BYTES / 16u) : bd2 + (g - n1) * (WR_Y_BYTES / 16u);
                tc::mma_bf16_warp(mine, d + 64u * g, ad + 128u * k, bd + 128u * k, id64,
                                  (g == 0 && k == 0) ? 0u : 1u);
              }
          }
        } else if (n2 == 0u) {
#pragma unroll
          for (uint32_t k = 0; k < 8; ++k) {
            tc::mma_bf16_warp(mine, d0, ad0 + 128u * k, bd1 + 128u * k, id1, 1u);
            tc::mma_bf16_warp(mine, d0 + 192u, ad1 + 128u * k, bd1 + 128u * k, id1, 1u);
          }
        } else {
#pragma unroll
          for (uint32_t k = 0; k < 8; ++k) {
            tc::mma_bf16_warp(mine, d0, ad0 + 128u * k, bd1 + 128u * k, id1, 1u);
            tc::mma_bf16_warp(mine, d0 + 64u * n1, ad0 + 128u * k, bd2 + 128u * k, id2, 1u);
            tc::mma_bf16_warp(mine, d0 + 192u, ad1 + 128u * k, bd1 + 128u * k, id1, 1u);
            tc::mma_bf16_warp(mine, d0 + 192u + 64u * n1, ad1 + 128u * k, bd2 + 128u * k, id2, 1u);
          }
        }
        tc::mma_commit_warp(mine, xempty + 8u * xs);
        if (j >= 2) tc::mma_commit_warp(mine, yempty + 8u * ((qj - 2u) % WR_Y));
      }
      q0 += (uint32_t)n;
      first = false;
    }
    if (ok) tc::mma_commit_warp(mine, done);
    tc::mma_commit_warp(mine, fin);
    tc::mbar_drain(fin, 0);
  } else {
    const int row = (warp & 3) * 32 + lane;
    tc::pdl_wait();
    if (tc::mbar_wait(done, 0, abort)) {
      tc::fence_after_sync();
      for (int p = 0; p < 2; ++p) {
        const int c = 2 * p + (row >> 6);  // tap column; 3: the all-ones block
        for (int r = 0; r < 3; ++r) {
          const int atom = c < 3 ? 3 * r + c : 9;
          float *dst = partial + ((size_t)blockIdx.x * WR_ATOMS + atom) * 4096u + (row & 63);
          const uint32_t taddr = tmem + ((uint32_t)((warp & 3) * 32) << 16) + 192u * (uint32_t)p + 64u * (uint32_t)(2 - r);
          for (int c0 = 0; c0 < 64; c0 += 16) {
            float v[16];
            tc::tmem_ld16(taddr + (uint32_t)c0, v);
            if (c < 3 || r == 1) {
#pragma unroll
              for (int i = 0; i < 16; ++i) dst[(size_t)(c0 + i) * 64] = v[i];
            }
          }
        }
      }
    }
  }
  tc::fence_before_sync();
  __syncthreads();
  if (warp == 1) {
    tc::fence_after_sync();
    tc::tmem_dealloc(tmem, 512u);
  }
  if (threadIdx.x == 0 && *abort) atomicOr(err, 2);
}

// dW[tap][co][ci] = sum over chunks of the X atoms' partials, in chunk order
// per thread group and then over the 4 groups; db[co] from the first all-ones
// atom. cin_blocks: input channel blocks (X atom a = tap * cin_blocks +
// block). Block (64 x 4 threads): one (atom, co) row of 64 entries;
// blockIdx.x = atom * N + co, and n_x * N + co for the bias.
__global__ void __launch_bounds__(256)
    k_wgrad_reduce(const float *__restrict__ partial, int chunks, int n_atoms, int n_x, int N, int cin_blocks,
                   float *__restrict__ dw, float *__restrict__ db) {
  tc::pdl_wait();
  tc::pdl_trigger();
  const int ci = threadIdx.x & 63, g = threadIdx.x >> 6;
  const int a = blockIdx.x / N, co = blockIdx.x - a * N;  // a == n_x: the bias row
  float s = 0.0f;
  for (int c = g; c < chunks; c += 4) s += partial[((size_t)c * n_atoms + a) * (size_t)N * 64 + (size_t)co * 64 + ci];
  __shared__ float r[4][64];
  r[g][ci] = s;
  __syncthreads();
  if (g) return;
  const float v = (r[0][ci] + r[1][ci]) + (r[2][ci] + r[3][ci]);
  if (a < n_x) {
    const int cin = cin_blocks * 64;
    const int tap = a / cin_blocks, blk = a - tap * cin_blocks;
    dw[((size_t)tap * N + co) * cin + blk * 64 + ci] = v;
  } else if (ci == 0) {
    db[co] = v;
  }
}

// ------------------------------------------------------------------ CUDA-core kernels

// Sequence -> channels-last input [n][L][64]: channel 0 = A bead, 1 = B bead,
// 2 = LAD bead, the rest zero. idx (optional) selects dataset rows.
__global__ void k_embed(const uint8_t *__restrict__ types, const uint8_t *__restrict__ lad,
                        const int32_t *__restrict__ idx, int L, int n, bf16 *__restrict__ x0) {
  tc::pdl_wait();
  tc::pdl_trigger();
  const long long k = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= (long long)n * L) return;
  const int b = (int)(k / L), l = (int)(k - (long long)b * L);
  const long long row = idx ? idx[b] : b;
  const uint8_t t = types[row * L + l];
  const uint8_t f = lad ? lad[row * L + l] : 0;
  uint4 *d = reinterpret_cast<uint4 *>(x0 + k * 64);
  uint4 z = make_uint4(0, 0, 0, 0);
  uint4 first = z;
  first.x = pack_bf16(t == 0 ? 1.0f : 0.0f, t == 1 ? 1.0f : 0.0f);
  first.y = pack_bf16(f ? 1.0f : 0.0f, 0.0f);
  d[0] = first;
#pragma unroll
  for (int i = 1; i < 8; ++i) d[i] = z;
}

// Mean over `f` consecutive positions: h [n][L][C] -> hp [n][L / f][C].
__global__ void k_pool(const bf16 *__restrict__ h, int L, int C, int f, int n, bf16 *__restrict__ hp) {
  tc::pdl_wait();
  tc::pdl_trigger();
  const long long k = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const int M = L / f;
  if (k >= (long long)n * M * C) return;
  const int c = (int)(k % C);
  const long long bm = k / C;
  const long long src = bm * f * C + c;
  float s = 0.0f;
  for (int i = 0; i < f; ++i) s += __bfloat162float(h[src + (long long)i * C]);
  hp[k] = __float2bfloat16_rn(s / (float)f);
}

// Pair features of the head input: z0[b][i][j][c] = u_i[c] v_j[c] + u_j[c] v_i[c]
// + E[|i - j|][c], u = uv[..][0, 64), v = uv[..][64, 128). Block: PAIR_ROWS
// consecutive rows i0.. of sample b; each warp walks runs of `cols` consecutive
// columns j, lane l holding channels 2l, 2l + 1 (one warp store covers a
// pixel's 64 channels). A lane keeps u_i, v_i of the block's rows and the
// distance embedding of every row in registers: the value row r needs at
// column j + 1, E[|i0 + r - j - 1|], is the one row r - 1 used at column j,
// so the window shifts by one row per column and only E[|i0 - j - 1|] is
// loaded. Per pixel and row: u_j, v_j and one E value per PAIR_ROWS outputs.
// A batch too small to fill the GPU takes shorter runs over more blocks
// (gridDim.z): one map of 256^2 took 15 us as 32 blocks with runs of 32 columns,
// 5.7 with 8.
constexpr int PAIR_ROWS = 8;

__device__ __forceinline__ float2 ld_bf16x2(const bf16 *p) {
  return __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162 *>(p));
}

__global__ void __launch_bounds__(256)
    k_pair_fwd(const bf16 *__restrict__ uv, const float *__restrict__ E, int M, int cols,
               bf16 *__restrict__ z0) {
  tc::pdl_wait();
  tc::pdl_trigger();
  const int i0 = blockIdx.x * PAIR_ROWS, b = blockIdx.y;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  const int c = 2 * lane;
  const bf16 *uvb = uv + (size_t)b * M * 128;
  const float2 *E2 = reinterpret_cast<const float2 *>(E) + lane;  // E2[d * 32] = E[d][c, c + 1]
  float2 ui[PAIR_ROWS], vi[PAIR_ROWS];
#pragma unroll
  for (int r = 0; r < PAIR_ROWS; ++r) {
    ui[r] = ld_bf16x2(uvb + (size_t)(i0 + r) * 128 + c);
    vi[r] = ld_bf16x2(uvb + (size_t)(i0 + r) * 128 + 64 + c);
  }
  __nv_bfloat162 *zb = reinterpret_cast<__nv_bfloat162 *>(z0 + (size_t)b * M * M * 64) + lane;
  for (int j0 = (blockIdx.z * nw + warp) * cols; j0 < M; j0 += gridDim.z * nw * cols) {
    float2 e[PAIR_ROWS];
#pragma unroll
    for (int r = 0; r < PAIR_ROWS; ++r) e[r] = __ldg(E2 + (size_t)abs(i0 + r - j0) * 32);
    const int j1 = min(j0 + cols, M);
    for (int j = j0; j < j1; ++j) {
      const float2 uj = ld_bf16x2(uvb + (size_t)j * 128 + c);
      const float2 vj = ld_bf16x2(uvb + (size_t)j * 128 + 64 + c);
#pragma unroll
      for (int r = 0; r < PAIR_ROWS; ++r) {
        const float zx = fmaf(ui[r].x, vj.x, fmaf(uj.x, vi[r].x, e[r].x));
        const float zy = fmaf(ui[r].y, vj.y, fmaf(uj.y, vi[r].y, e[r].y));
        zb[((size_t)(i0 + r) * M + j) * 32] = __floats2bfloat162_rn(zx, zy);
      }
#pragma unroll
      for (int r = PAIR_ROWS - 1; r > 0; --r) e[r] = e[r - 1];
      if (j + 1 < j1) e[0] = __ldg(E2 + (size_t)abs(i0 - j - 1) * 32);  // |.| < M
    }
  }
}

// The network predicts log contact probabilities; yhat = (y + y^T) / 2 is
// clamped to YHAT_MAX = 0 (probability 1) before exponentiation. The loss
// gradient is taken at the clamped value and passed through unchanged
// (straight-through), so a prediction above 1 is pulled back down.
constexpr float YHAT_MAX = 0.0f;

// Prediction: contact probability exp(yhat).
__global__ void k_predict_maps(const float *__restrict__ y, int M, int n, float *__restrict__ out) {
  tc::pdl_wait();
  tc::pdl_trigger();
  const long long k = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= (long long)n * M * M) return;
  const long long b = k / ((long long)M * M);
  const int r = (int)(k - b * M * M), i = r / M, j = r - i * M;
  const float yh = 0.5f * (y[k] + y[b * M * M + (long long)j * M + i]);
  out[k] = expf(fminf(yh, YHAT_MAX));
}

// P(s) of predicted maps: block b reduces map b, thread s (strided) the mean
// of its diagonal s, pred[b][i][i + s] for i < M - s, summed in FP64.
__global__ void __launch_bounds__(256)
    k_ps_curve(const float *__restrict__ pred, int M, float *__restrict__ ps) {
  tc::pdl_wait();
  tc::pdl_trigger();
  const float *m = pred + (size_t)blockIdx.x * M * M;
  for (int s = threadIdx.x; s < M; s += blockDim.x) {
    double acc = 0.0;
    for (int i = 0; i + s < M; ++i) acc += (double)m[(size_t)i * M + i + s];
    ps[(size_t)blockIdx.x * M + s] = (float)(acc / (double)(M - s));
  }
}

// Loss and the gradient entering the head. yhat = (y + y^T) / 2 and the
// Poisson deviance of the observed contact probability p against exp(yhat),
// weighted per separation s = |i - j| by w[s] (the inverse of the dataset's
// mean P(s)), averaged over n M^2 values:
//   loss = mean w[s] (exp(yhat) - p - p (yhat - log p)),
//   dL/dyhat = w[s] (exp(yhat) - p) / (n M^2).
// Targets are symmetric, so dL/dy = dL/dyhat.
// The gradient of the last head output is the rank-1 dz[p][c] = dy[p] wo[c]:
// only dy is stored (the next convolution's epilogue expands it); dc[p][c] =
// dz masked by the last head layer's ReLU bits (BF16). Accumulates d wo,
// d bo and the loss.
//
// A warp takes 32 pixels at a time: lane l computes pixel l's dy, then eight
// lanes a pixel (eight channels each) read z and write dc, 4 pixels' contiguous
// 128 bytes an instruction, and d wo gathers in registers over all of the
// warp's pixels. With a thread a pixel every pixel's 64 products went through a
// warp reduction of their own (320 shuffles): 232 us for 32 maps of 256^2, now
// 101; HBM floor 87 (580 MB).
__global__ void __launch_bounds__(256)
    k_loss_out_bwd(const float *__restrict__ y, const float *__restrict__ target, const float *__restrict__ sw,
                   const int32_t *__restrict__ idx, const bf16 *__restrict__ z, const uint32_t *__restrict__ mask,
                   const float *__restrict__ wo, int M, int n, float *__restrict__ dy, bf16 *__restrict__ dc,
                   float *__restrict__ gwo, float *__restrict__ gbo, double *__restrict__ loss) {
  tc::pdl_wait();
  tc::pdl_trigger();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int c0 = (lane & 7) * 8;
  const long long MM = (long long)M * M, P = (long long)n * MM;
  float w8[8], gw[8];
#pragma unroll
  for (int t = 0; t < 8; ++t) {
    w8[t] = wo[c0 + t];
    gw[t] = 0.0f;
  }
  float sum_dy = 0.0f, sum_l = 0.0f;
  for (long long g = (long long)blockIdx.x * 8 + warp; g * 32 < P; g += (long long)gridDim.x * 8) {
    const long long p0 = g * 32, p = p0 + lane;  // P is a multiple of 32
    uint4 zq[8];
#pragma unroll
    for (int s = 0; s < 8; ++s)
      zq[s] = *reinterpret_cast<const uint4 *>(z + (p0 + 4 * s + (lane >> 3)) * 64 + c0);
    const long long b = p / MM;
    const int r = (int)(p - b * MM), i = r / M, j = r - i * M;
    const float yh = fminf(0.5f * (y[p] + y[b * MM + (long long)j * M + i]), YHAT_MAX);
    const long long row = idx ? idx[b] : b;
    const float t = target[row * MM + r];
    const float w = sw[abs(i - j)];
    const float e = expf(yh);
    sum_l += w * (e - t - (t > 0.0f ? t * (yh - logf(t)) : 0.0f));
    const float dyv = w * (e - t) / (float)P;
    sum_dy += dyv;
    dy[p] = dyv;
    const uint2 m = *reinterpret_cast<const uint2 *>(mask + p * 2);
#pragma unroll
    for (int s = 0; s < 8; ++s) {
      const int src = 4 * s + (lane >> 3);
      const float d = __shfl_sync(0xffffffffu, dyv, src);
      const uint32_t m0 = __shfl_sync(0xffffffffu, m.x, src), m1 = __shfl_sync(0xffffffffu, m.y, src);
      const uint32_t bits = ((lane & 4) ? m1 : m0) >> (c0 & 31);
      const uint32_t q[4] = {zq[s].x, zq[s].y, zq[s].z, zq[s].w};
      float o[8];
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        gw[2 * k] = fmaf(d, bf_lo(q[k]), gw[2 * k]);
        gw[2 * k + 1] = fmaf(d, bf_hi(q[k]), gw[2 * k + 1]);
        o[2 * k] = ((bits >> (2 * k)) & 1u) ? d * w8[2 * k] : 0.0f;
        o[2 * k + 1] = ((bits >> (2 * k + 1)) & 1u) ? d * w8[2 * k + 1] : 0.0f;
      }
      *reinterpret_cast<uint4 *>(dc + (p0 + src) * 64 + c0) =
          make_uint4(pack_bf16(o[0], o[1]), pack_bf16(o[2], o[3]), pack_bf16(o[4], o[5]), pack_bf16(o[6], o[7]));
    }
  }
  // sums over the block: channels over the four lanes that share them, then all
  // warps in order
  __shared__ float red[8][64];
  __shared__ float rdy[8];
  __shared__ double rl[8];
#pragma unroll
  for (int t = 0; t < 8; ++t) {
    gw[t] += __shfl_xor_sync(0xffffffffu, gw[t], 8);
    gw[t] += __shfl_xor_sync(0xffffffffu, gw[t], 16);
    if (lane < 8) red[warp][c0 + t] = gw[t];
  }
  double vl = sum_l;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    sum_dy += __shfl_xor_sync(0xffffffffu, sum_dy, o);
    vl += __shfl_xor_sync(0xffffffffu, vl, o);
  }
  if (lane == 0) {
    rdy[warp] = sum_dy;
    rl[warp] = vl;
  }
  __syncthreads();
  if (threadIdx.x < 64) {
    float s = 0.0f;
    for (int w = 0; w < 8; ++w) s += red[w][threadIdx.x];
    atomicAdd(gwo + threadIdx.x, s);
  } else if (threadIdx.x == 64) {
    float s = 0.0f;
    double t = 0.0;
    for (int w = 0; w < 8; ++w) {
      s += rdy[w];
      t += rl[w];
    }
    atomicAdd(gbo, s);
    atomicAdd(loss, t / (double)P);
  }
}

// Gradients of the pair features from dz, the gradient of the head's input.
// Blocks below M / 4 of sample b: four rows i of u and v. With S_ij = dz_ij +
// dz_ji, du_i = sum_j S_ij v_j and dv_i = sum_j S_ij u_j per channel, output
// BF16. The other blocks: four separations s of the distance embedding,
// part[b][s][c] = sum over pairs with |i - j| = s of dz_ij[c] (both
// triangles); k_dist_reduce adds the samples in order. A row or separation has
// 64 threads: four channels each, four classes over j (over i), added in
// order.
//
// dz is read three times: as dz_ij, as dz_ji and by diagonals. Blocks of both
// kinds run side by side, sample by sample, so L2 serves two of the three, and
// a thread reads 16 bytes at a time. Measured at 32 maps of 256^2: a kernel per
// gradient with 4-byte loads 148 + 101 us, this one 147; HBM floor 80. L2
// bounds it: other unrolls (2, 8, 16), fewer or more resident blocks and another order of
// the blocks made no difference or were slower. The order of each sum (four
// classes of j) is kept on purpose: du and dv are rounded to BF16 next, and
// another order flips roundings (gradients of small batches then move by 8e-5).
constexpr int PAIR_BWD_ROWS = 4;
__device__ __forceinline__ float4 f4_add(float4 a, float4 b) {
  return make_float4(a.x + b.x, a.y + b.y, a.z + b.z, a.w + b.w);
}
__device__ __forceinline__ void f4_fma(float4 a, uint2 w, float4 &d) {
  d.x = fmaf(a.x, bf_lo(w.x), d.x);
  d.y = fmaf(a.y, bf_hi(w.x), d.y);
  d.z = fmaf(a.z, bf_lo(w.y), d.z);
  d.w = fmaf(a.w, bf_hi(w.y), d.w);
}
__global__ void __launch_bounds__(256)
    k_pair_bwd(const float *__restrict__ dz, const bf16 *__restrict__ uv, int M, bf16 *__restrict__ duv,
               float *__restrict__ part) {
  tc::pdl_wait();
  tc::pdl_trigger();
  const int b = blockIdx.y, row = threadIdx.x >> 6, g = (threadIdx.x >> 4) & 3, c = 4 * (threadIdx.x & 15);
  const size_t MM = (size_t)M * M;
  const float *dzb = dz + (size_t)b * MM * 64 + c;
  const bool dist = (int)blockIdx.x >= M / PAIR_BWD_ROWS;
  const int i = ((int)blockIdx.x - (dist ? M / PAIR_BWD_ROWS : 0)) * PAIR_BWD_ROWS + row;
  auto at = [&](int r, int k) { return *reinterpret_cast<const float4 *>(dzb + ((size_t)r * M + k) * 64); };
  __shared__ float4 su[4][4][16], sv[4][4][16];  // class, row, channels
  float4 du = make_float4(0.0f, 0.0f, 0.0f, 0.0f), dv = du;
  if (!dist) {
    const bf16 *uvb = uv + (size_t)b * M * 128 + c;
#pragma unroll 4
    for (int j = g; j < M; j += 4) {
      const float4 s = f4_add(at(i, j), at(j, i));
      f4_fma(s, *reinterpret_cast<const uint2 *>(uvb + (size_t)j * 128 + 64), du);
      f4_fma(s, *reinterpret_cast<const uint2 *>(uvb + (size_t)j * 128), dv);
    }
    sv[g][row][c / 4] = dv;
  } else if (i) {
#pragma unroll 4
    for (int k = g; k < M - i; k += 4) {
      du = f4_add(du, at(k, k + i));
      du = f4_add(du, at(k + i, k));
    }
  } else {
#pragma unroll 4
    for (int k = g; k < M; k += 4) du = f4_add(du, at(k, k));
  }
  su[g][row][c / 4] = du;
  __syncthreads();
  if (g) return;
  const int q = c / 4;
  const float4 a = f4_add(f4_add(f4_add(su[0][row][q], su[1][row][q]), su[2][row][q]), su[3][row][q]);
  if (dist) {
    *reinterpret_cast<float4 *>(part + ((size_t)b * M + i) * 64 + c) = a;
    return;
  }
  const float4 d = f4_add(f4_add(f4_add(sv[0][row][q], sv[1][row][q]), sv[2][row][q]), sv[3][row][q]);
  bf16 *o = duv + ((size_t)b * M + i) * 128 + c;
  *reinterpret_cast<uint2 *>(o) = make_uint2(pack_bf16(a.x, a.y), pack_bf16(a.z, a.w));
  *reinterpret_cast<uint2 *>(o + 64) = make_uint2(pack_bf16(d.x, d.y), pack_bf16(d.z, d.w));
}

__global__ void k_dist_reduce(const float *__restrict__ part, int M, int n, float *__restrict__ dE) {
  tc::pdl_wait();
  tc::pdl_trigger();
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= M * 64) return;
  float s = 0.0f;
  for (int b = 0; b < n; ++b) s += part[(size_t)b * M * 64 + k];
  dE[k] = s;
}

// Unpooling of the projection-input gradient: dz[b][l][c] = dhp[b][l / f][c] / f
// (FP32, the encoder's residual gradient) and dc = dz masked by the last
// encoder layer's ReLU bits (BF16). C = 128.
__global__ void k_unpool(const float *__restrict__ dhp, const uint32_t *__restrict__ mask, int L, int f,
                         int n, float *__restrict__ dz, bf16 *__restrict__ dc) {
  tc::pdl_wait();
  tc::pdl_trigger();
  const long long k = (long long)blockIdx.x * blockDim.x + threadIdx.x;  // (b, l, 16-channel chunk)
  if (k >= (long long)n * L * 8) return;
  const int c0 = (int)(k & 7) * 16;
  const long long bl = k >> 3;
  const long long b = bl / L;
  const int l = (int)(bl - b * L);
  const float *src = dhp + ((b * (L / f)) + l / f) * 128 + c0;
  const float inv = 1.0f / (float)f;
  float v[16];
#pragma unroll
  for (int t = 0; t < 16; ++t) v[t] = src[t] * inv;
  float4 *o = reinterpret_cast<float4 *>(dz + bl * 128 + c0);
#pragma unroll
  for (int t = 0; t < 4; ++t) o[t] = make_float4(v[4 * t], v[4 * t + 1], v[4 * t + 2], v[4 * t + 3]);
  const uint32_t w = mask[bl * 4 + (c0 >> 5)] >> (c0 & 16);
#pragma unroll
  for (int t = 0; t < 16; ++t) v[t] = ((w >> t) & 1u) ? v[t] : 0.0f;
  store_bf16x16(dc + bl * 128 + c0, v);
}

// Sum of squared gradients (FP64) for the global-norm clip.
__global__ void __launch_bounds__(256) k_grad_sq(const float *__restrict__ g, long long n, double *__restrict__ out) {
  double s = 0.0;
  for (long long k = (long long)blockIdx.x * blockDim.x + threadIdx.x; k < n; k += (long long)gridDim.x * blockDim.x)
    s += (double)g[k] * g[k];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  __shared__ double r[8];
  if ((threadIdx.x & 31) == 0) r[threadIdx.x >> 5] = s;
  __syncthreads();
  if (threadIdx.x == 0) {
    double t = 0.0;
    for (int w = 0; w < (int)(blockDim.x >> 5); ++w) t += r[w];
    atomicAdd(out, t);
  }
}

// AdamW over the whole FP32 parameter vector; decay[k] selects weight decay.
// The gradient is scaled by min(1, clip / ||g||) when clip > 0 (gsq: the
// squared norm from k_grad_sq).
__global__ void k_adamw(float *__restrict__ p, const float *__restrict__ g, float *__restrict__ m,
                        float *__restrict__ v, const uint8_t *__restrict__ decay, long long n, float lr, float b1,
                        float b2, float eps, float wd, float bc1, float bc2, float clip,
                        const double *__restrict__ gsq) {
  const long long k = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= n) return;
  float scale = 1.0f;
  if (clip > 0.0f) {
    const double norm = sqrt(*gsq);
    if (norm > clip) scale = (float)(clip / norm);
  }
  const float gk = g[k] * scale;
  const float mk = b1 * m[k] + (1.0f - b1) * gk;
  const float vk = b2 * v[k] + (1.0f - b2) * gk * gk;
  m[k] = mk;
  v[k] = vk;
  const float upd = (mk / bc1) / (sqrtf(vk / bc2) + eps);
  p[k] = p[k] * (1.0f - lr * (decay[k] ? wd : 0.0f)) - lr * upd;
}

// BF16 copies of every convolution's weights: W [taps][co][ci] and the
// transposed WT [taps][ci][co] used by the input-gradient convolution.
// blockIdx.y selects the layer.
constexpr int MAX_LAYERS = 80;
struct WeightTable {
  int n;
  int taps[MAX_LAYERS], co[MAX_LAYERS], ci[MAX_LAYERS];
  long long off[MAX_LAYERS];
  bf16 *wb[MAX_LAYERS], *wt[MAX_LAYERS];
};

__global__ void k_weights_bf16(const float *__restrict__ params, const __grid_constant__ WeightTable t) {
  const int l = blockIdx.y;
  const long long k = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const int taps = t.taps[l], co = t.co[l], ci = t.ci[l];
  if (k >= (long long)taps * co * ci) return;
  const int i = (int)(k % ci), o = (int)((k / ci) % co), tp = (int)(k / ((long long)ci * co));
  const bf16 x = __float2bfloat16_rn(params[t.off[l] + k]);
  t.wb[l][k] = x;
  t.wt[l][((long long)tp * ci + i) * co + o] = x;
}

}  // namespace sur

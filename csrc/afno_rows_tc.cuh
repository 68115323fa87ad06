// Row transforms of the AFNO filter on the tensor cores, for tokens of one owner.
//
//   Y[row, kx, c] = kweight(kx) / sqrt(W) sum_w x[row, w, c] e^{-2 pi i kx w / W},  kx < KX
//
// is, per row, a product of the transposed tokens [c, w] with a matrix of twiddles [w, 2 kx + {re, im}].  Tokens are bf16 as they are; a
// twiddle is the sum of three bf16 values (24 bits), so three products with exact terms add up to what the sum in fp32 gives: error
// against 64 bits, W = 60 / 90 / 120 / 180, 0.70 / 0.71 / 1.00 / 1.08e-7 (the sum in fp32: 1.13 / 1.39 / 1.48 / 1.94e-7).  That sum on the fp32
// units (afno_spectral.cu) reads 2 + 3 vectors of shared memory for 24 multiply-adds, and is bound by that: 2 x 90 x 180 tokens of 768
// channels 123 us, here 35 us; 45 x 90 tokens 20.5 and 14.3 us.  (The token rows and the spectrum are 101 MB, 16 us.)  The twiddles stay in shared memory for the life of a persistent CTA; a tile is one row of tokens x 128 channels, brought by TMA
// as an MN-major operand (w along K, zeros past W), its spectrum leaves from tensor memory, a channel per lane, as whole lines.
#pragma once
#include "common.cuh"
#include "tmap.cuh"
#include "pnm_internal.h"

namespace pnm {

constexpr int kRowTcThreads = 320;               // warp 0 producer, warp 1 products, warps 2 .. 9 epilogue

struct RowTcArgs {
  float2* Y;
  int rows, W, C, KX, kweight;
  int k16, n16;                                  // W and 2 KX, rounded up to multiples of 16
  int chunks;                                    // of 64 positions
  int stages, tiles_c;
  float scale;
  int* err;
};

__host__ __device__ inline int row_tc_stage_bytes(int k16) { return 2 * k16 * 128; }
__host__ __device__ inline int row_tc_table_bytes(int n16, int chunks) { return n16 * chunks * 128; }

__global__ void __launch_bounds__(kRowTcThreads, 1)
afno_rows_r2c_tc_kernel(const __grid_constant__ CUtensorMap tmX, const RowTcArgs g) {
  extern __shared__ uint8_t smem_raw[];
  __shared__ uint64_t full[4], empty[4], tfull[2], tempty[2];
  __shared__ uint32_t tmem_slot;
  __shared__ int abort_word;
  volatile int* abort_flag = &abort_word;
  uint8_t* base = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  const int stage_bytes = row_tc_stage_bytes(g.k16), table = row_tc_table_bytes(g.n16, g.chunks);
  uint8_t* tw = base + g.stages * stage_bytes;   // three tables, K-major
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int tiles = g.rows * g.tiles_c;

  if (threadIdx.x == 0) {
    for (int s = 0; s < g.stages; ++s) { mbar_init(&full[s], 1); mbar_init(&empty[s], 1); }
    for (int a = 0; a < 2; ++a) { mbar_init(&tfull[a], 1); mbar_init(&tempty[a], 8); }
    abort_word = 0;
    mbar_fence_init();
    tma_prefetch_desc(&tmX);
  }
  if (warp == 1) { tmem_alloc(&tmem_slot, 512); tmem_relinquish(); }
  // ---- twiddles: only W values occur; they are computed once, in the memory of the first stage
  float2* values = reinterpret_cast<float2*>(base);
  for (int m = threadIdx.x; m < g.W; m += kRowTcThreads) {
    double s, c;
    sincospi(2.0 * m / g.W, &s, &c);
    values[m] = make_float2(float(c), float(-s));
  }
  for (int i = threadIdx.x; i < 3 * table / 16; i += kRowTcThreads) reinterpret_cast<uint4*>(tw)[i] = make_uint4(0, 0, 0, 0);
  __syncthreads();
  for (int kx = warp; kx < g.KX; kx += kRowTcThreads / 32)
    for (int w = lane; w < g.W; w += 32) {
      const float2 v = values[(kx * w) % g.W];
      const int n = 2 * kx, chunk = w >> 6, k = w & 63;
      float part[2] = {v.x, v.y};
#pragma unroll
      for (int term = 0; term < 3; ++term)
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          const __nv_bfloat16 b = __float2bfloat16(part[e]);
          part[e] -= __bfloat162float(b);
          *reinterpret_cast<__nv_bfloat16*>(tw + term * table + (chunk * g.n16 + n + e) * 128 + (((k >> 3) ^ ((n + e) & 7)) << 4) + (k & 7) * 2) = b;
        }
    }
  fence_async_smem();
  tc_fence_before();
  __syncthreads();                               // also: the values' memory belongs to the copies from here on
  tc_fence_after();
  const uint32_t tmem = tmem_slot;               // accumulators at 0 and 256

  if (warp == 0) {
    if (elect_one()) {
      uint32_t it = 0;
      for (int t = blockIdx.x; t < tiles; t += gridDim.x, ++it) {
        const int s = it % g.stages, row = t / g.tiles_c, c0 = (t - row * g.tiles_c) * 128;
        if (!mbar_wait(&empty[s], ((it / g.stages) & 1) ^ 1, abort_flag, g.err, ERR_WAIT_EMPTY)) break;
        uint8_t* dst = base + s * stage_bytes;
        mbar_expect_tx(&full[s], stage_bytes);
        for (int i = 0; i < 2; ++i) tma_load_3d(dst + i * g.k16 * 128, &tmX, &full[s], c0 + i * 64, 0, row);
      }
      ring_drain(full, g.stages, it);
    }
  } else if (warp == 1) {
    if (elect_one()) {
      const uint32_t idesc = make_idesc_bf16(128, g.n16, true, false);
      uint32_t it = 0;
      for (int t = blockIdx.x; t < tiles; t += gridDim.x, ++it) {
        const int s = it % g.stages, a = it & 1;
        if (!mbar_wait(&tempty[a], ((it >> 1) & 1) ^ 1, abort_flag, g.err, ERR_WAIT_TMEM_EMPTY)) break;
        if (!mbar_wait(&full[s], (it / g.stages) & 1, abort_flag, g.err, ERR_WAIT_FULL)) break;
        tc_fence_after();
        const uint64_t xd = make_smem_desc(smem_u32(base + s * stage_bytes), g.k16 * 128, 1024, 2);
        const uint32_t table0 = smem_u32(tw);
        uint32_t more = 0;
        for (int term = 2; term >= 0; --term)    // small terms first
          for (int k = 0; k < g.k16; k += 16) {
            const uint64_t td = make_smem_desc(table0 + term * table + (k >> 6) * g.n16 * 128, 16, 1024, 2) + 2 * ((k >> 4) & 3);
            umma_f16(tmem + a * 256, xd + 8 * k, td, idesc, more);         // 16 positions = 2048 bytes = 128 units
            more = 1;
          }
        umma_commit(&empty[s]);
        umma_commit(&tfull[a]);
      }
    }
  } else {
    const int q = warp & 3, half = (warp - 2) >> 2;
    uint32_t it = 0;
    for (int t = blockIdx.x; t < tiles; t += gridDim.x, ++it) {
      const int a = it & 1, row = t / g.tiles_c, c = (t - row * g.tiles_c) * 128 + q * 32 + lane;
      const bool ok = mbar_wait(&tfull[a], (it >> 1) & 1, abort_flag, g.err, ERR_WAIT_TMEM_FULL);
      if (!__all_sync(0xffffffffu, ok)) break;
      tc_fence_after();
      float2* dst = g.Y + (long long)row * g.KX * g.C + c;
      for (int j = half; j < g.n16 / 16; j += 2) {           // eight modes
        float v[16];
        tmem_ld16(tmem + a * 256 + (uint32_t(q * 32) << 16) + 16 * j, v);
        tmem_ld_wait();
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          const int kx = 8 * j + i;
          const float s = g.kweight && kx > 0 ? 2.f * g.scale : g.scale;
          if (kx < g.KX && c < g.C) dst[(long long)kx * g.C] = make_float2(v[2 * i] * s, v[2 * i + 1] * s);
        }
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&tempty[a]);
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    if (abort_word) abort_settle();
    tc_fence_after();
    tmem_dealloc(tmem, 512);
  }
}

// Whether the transform of these tokens fits (a box of the whole row, one accumulator of 2 KX columns, three tables beside two stages),
// and its launch: 0, or an error; 1 where it does not apply.
inline int launch_rows_r2c_tc(const void* tokens, float2* Y, int rows, int W, int C, int KX, int kweight, int num_sms, int* err, cudaStream_t stream) {
  RowTcArgs g;
  g.Y = Y; g.rows = rows; g.W = W; g.C = C; g.KX = KX; g.kweight = kweight; g.err = err;
  g.k16 = (W + 15) / 16 * 16; g.n16 = (2 * KX + 15) / 16 * 16; g.chunks = (g.k16 + 63) / 64;
  g.scale = 1.f / sqrtf(float(W));
  if (g.k16 > 256 || g.n16 > 256 || (reinterpret_cast<uintptr_t>(tokens) & 15) || C % 8) return 1;
  const int fixed = 1024 + 3 * row_tc_table_bytes(g.n16, g.chunks), stage = row_tc_stage_bytes(g.k16);
  g.stages = (225 * 1024 - fixed) / stage;
  if (g.stages < 2) return 1;
  if (g.stages > 4) g.stages = 4;
  if (g.stages * stage < W * 8) return 1;        // the table's values are made there
  g.tiles_c = (C + 127) / 128;
  CUtensorMap tm;
  if (make_tmap_3d_b16(&tm, tokens, rows, W, C, C, (uint64_t)W * C, g.k16)) return 1;
  static DeviceMask smem_set{0};
  if (!allow_smem(afno_rows_r2c_tc_kernel, 225 * 1024, smem_set)) return -4;
  const int tiles = rows * g.tiles_c;
  afno_rows_r2c_tc_kernel<<<tiles < num_sms ? tiles : num_sms, kRowTcThreads, fixed + g.stages * stage, stream>>>(tm, g);
  return cudaGetLastError() == cudaSuccess ? 0 : -3;
}

}  // namespace pnm

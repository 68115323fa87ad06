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

// D (+)= the K-slices of one term: 16 values of K are 2048 bytes of the MN-major operand and 32 of the table, whose chunks of 64 lie
// `chunk` units of 16 bytes apart.  The thread that issues has 48 cycles for a product of 96 columns: additions only.
__device__ __forceinline__ void row_tc_products(uint32_t d, uint64_t xd, uint64_t td, int slices, int chunk, uint32_t idesc, uint32_t more) {
  umma_f16(d, xd, td, idesc, more);
#pragma unroll 4
  for (int k = 1; k < slices; ++k) {
    xd += 128;
    td += (k & 3) ? 2 : chunk - 6;
    umma_f16(d, xd, td, idesc, 1u);
  }
}

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
      const uint64_t td0 = make_smem_desc(smem_u32(tw), 16, 1024, 2);
      uint32_t it = 0;
      for (int t = blockIdx.x; t < tiles; t += gridDim.x, ++it) {
        const int s = it % g.stages, a = it & 1;
        if (!mbar_wait(&tempty[a], ((it >> 1) & 1) ^ 1, abort_flag, g.err, ERR_WAIT_TMEM_EMPTY)) break;
        if (!mbar_wait(&full[s], (it / g.stages) & 1, abort_flag, g.err, ERR_WAIT_FULL)) break;
        tc_fence_after();
        const uint64_t xd = make_smem_desc(smem_u32(base + s * stage_bytes), g.k16 * 128, 1024, 2);
        uint64_t td = td0 + 2 * (table >> 4);    // small terms first
#pragma unroll 1
        for (int term = 2; term >= 0; --term, td -= table >> 4)
          row_tc_products(tmem + a * 256, xd, td, g.k16 >> 4, g.n16 * 8, idesc, term == 2 ? 0u : 1u);
        umma_commit(&empty[s]);
        umma_commit(&tfull[a]);
      }
    }
  } else {
    const int q = warp & 3, half = (warp - 2) >> 2;
    uint32_t it = 0;
    for (int t = blockIdx.x; t < tiles; t += gridDim.x, ++it) {
      const int a = it & 1, row = t / g.tiles_c, c = (t - row * g.tiles_c) * 128 + q * 32 + lane;
      if (!mbar_wait_warp(&tfull[a], (it >> 1) & 1, abort_flag, g.err, ERR_WAIT_TMEM_FULL)) break;
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

// ------------------------------------------------------------------------------------------------ back to the tokens
//   y[row, w, c] = 1 / sqrt(W) sum_kx kweight(kx) Re( X[row, kx, c] e^{2 pi i kx w / W} ) (+ addends)
// With A[w] = sum Re X cos, B[w] = sum Im X sin for w <= W / 2, y[w] = A - B and y[W - w] = A + B: two products of [channels, modes] with
// [modes, positions].  Here both operands are fp32, each the sum of three bf16 values, of whose nine products the six that matter are
// formed (the rest is below 2^-24 of a term); the results are rounded to bf16 as before.  Twelve warps read a tile of the spectrum (one row, 128
// channels) and split it into MN-major operands while the tile before it is multiplied, eight bring results from
// tensor memory through shared memory to whole lines.  2 x 90 x 180 tokens of 768 channels 106 -> 57 us, with two
// addends 127 -> 86 (200 MB, 31 us at the copy rate; what is left is the way of the results from tensor memory, about 5 000 cycles a tile).
constexpr int kRowInvLoaders = 12, kRowInvEpilogue = 8;
constexpr int kRowInvThreads = 32 * (kRowInvLoaders + 1 + kRowInvEpilogue);
constexpr int kRowInvLd = 160;                   // channels of a row of results in shared memory: the next row starts 16 banks on
constexpr int kRowInvLoads = 8;                  // vectors that a loading thread holds: the modes of two boxes over twelve warps, 48 at a time

struct RowInvArgs {
  const float2* X;
  __nv_bfloat16* y;
  const __nv_bfloat16 *add0, *add1;              // [rows W, C] or null
  int rows, W, C, KX, kweight;
  int k16, n16;                                  // KX and W / 2 + 1, rounded up to multiples of 16
  int chunks;                                    // of 64 modes
  int tiles_c;
  float scale;
  int* err;
};

// 16-byte aligned, a multiple of 16 bytes
__device__ __forceinline__ void l2_prefetch(const void* p, uint32_t bytes) {
  asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(p), "r"(bytes) : "memory");
}

__global__ void __launch_bounds__(kRowInvThreads, 1) afno_rows_c2r_tc_kernel(const RowInvArgs g) {
  extern __shared__ uint8_t smem_raw[];
  __shared__ uint64_t afull, aempty, tfull[2], tempty[2];
  __shared__ uint32_t tmem_slot;
  __shared__ int abort_word;
  volatile int* abort_flag = &abort_word;
  uint8_t* base = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  const int table = row_tc_table_bytes(g.n16, g.chunks), part = 2 * g.k16 * 128;
  uint8_t* tw = base;                            // cos, sin: three terms each, K-major
  uint8_t* xs = tw + 6 * table;                  // Re, Im: three terms each, MN-major boxes of 64 channels
  __nv_bfloat16* ys = reinterpret_cast<__nv_bfloat16*>(xs + 6 * part);     // [W][kRowInvLd]
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int tiles = g.rows * g.tiles_c;

  if (threadIdx.x == 0) {
    mbar_init(&afull, kRowInvLoaders); mbar_init(&aempty, 1);
    for (int a = 0; a < 2; ++a) { mbar_init(&tfull[a], 1); mbar_init(&tempty[a], kRowInvEpilogue); }
    abort_word = 0;
    mbar_fence_init();
  }
  if (warp == kRowInvLoaders) { tmem_alloc(&tmem_slot, 512); tmem_relinquish(); }
  float2* values = reinterpret_cast<float2*>(ys);            // (cos, sin)(2 pi m / W): W 8 bytes, the tile of results has W 320
  for (int m = threadIdx.x; m < g.W; m += kRowInvThreads) {
    double s, c;
    sincospi(2.0 * m / g.W, &s, &c);
    values[m] = make_float2(float(c), float(s));
  }
  for (int i = threadIdx.x; i < (6 * table + 6 * part) / 16; i += kRowInvThreads) reinterpret_cast<uint4*>(base)[i] = make_uint4(0, 0, 0, 0);
  __syncthreads();
  for (int w = warp; w <= g.W / 2; w += kRowInvThreads / 32)
    for (int kx = lane; kx < g.KX; kx += 32) {
      const float2 v = values[(kx * w) % g.W];
      float rest[2] = {v.x, v.y};
      const int at = ((kx >> 6) * g.n16 + w) * 128 + ((((kx & 63) >> 3) ^ (w & 7)) << 4) + (kx & 7) * 2;
#pragma unroll
      for (int term = 0; term < 3; ++term)
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          const __nv_bfloat16 b = __float2bfloat16(rest[e]);
          rest[e] -= __bfloat162float(b);
          *reinterpret_cast<__nv_bfloat16*>(tw + (3 * e + term) * table + at) = b;
        }
    }
  fence_async_smem();
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = tmem_slot;               // A at 0 and 256, B 128 columns on

  if (warp < kRowInvLoaders) {
    // ---- one mode of one box of 64 channels at a time, two channels per lane
    uint32_t it = 0;
    for (int t = blockIdx.x; t < tiles; t += gridDim.x, ++it) {
      const int row = t / g.tiles_c, c0 = (t - row * g.tiles_c) * 128;
      bool ok = true;
      if (g.add0) {                              // the addends of this tile, 256 bytes per position, to L2 a tile ahead of their use
        const uint32_t bytes = 2 * min(128, g.C - c0);
        for (int w = threadIdx.x; w < g.W; w += 32 * kRowInvLoaders) {
          const long long at = ((long long)row * g.W + w) * g.C + c0;
          l2_prefetch(g.add0 + at, bytes);
          if (g.add1) l2_prefetch(g.add1 + at, bytes);
        }
      }
#pragma unroll 1
      for (int first = 0; first < 2 * g.KX; first += kRowInvLoads * kRowInvLoaders) {
        float4 v[kRowInvLoads];
#pragma unroll
        for (int n = 0; n < kRowInvLoads; ++n) {
          const int i = first + warp + n * kRowInvLoaders, kx = i >> 1, c = c0 + (i & 1) * 64 + 2 * lane;
          v[n] = make_float4(0.f, 0.f, 0.f, 0.f);
          if (kx < g.KX && c < g.C) v[n] = __ldcs(reinterpret_cast<const float4*>(g.X + ((long long)row * g.KX + kx) * g.C + c));
        }
        if (first == 0) {                        // the first loads are on their way meanwhile
          ok = mbar_wait_warp(&aempty, (it & 1) ^ 1, abort_flag, g.err, ERR_WAIT_EMPTY);
          if (!ok) break;
        }
#pragma unroll
        for (int n = 0; n < kRowInvLoads; ++n) {
          const int i = first + warp + n * kRowInvLoaders, kx = i >> 1;
          if (kx < g.KX) {
            const float s = g.kweight && kx > 0 ? 2.f : 1.f;
            float re[2] = {v[n].x * s, v[n].z * s}, im[2] = {v[n].y * s, v[n].w * s};
            uint8_t* dst = xs + (i & 1) * g.k16 * 128 + kx * 128 + (((lane >> 2) ^ (kx & 7)) << 4) + (lane & 3) * 4;
#pragma unroll
            for (int term = 0; term < 3; ++term) {
              const uint32_t a = pack_bf16x2(re[0], re[1]), b = pack_bf16x2(im[0], im[1]);
              *reinterpret_cast<uint32_t*>(dst + term * part) = a;
              *reinterpret_cast<uint32_t*>(dst + (3 + term) * part) = b;
              const float2 fa = unpack_bf16x2(a), fb = unpack_bf16x2(b);
              re[0] -= fa.x; re[1] -= fa.y; im[0] -= fb.x; im[1] -= fb.y;
            }
          }
        }
      }
      if (!ok) break;
      fence_async_smem();
      __syncwarp();
      if (lane == 0) mbar_arrive(&afull);
    }
  } else if (warp == kRowInvLoaders) {
    if (elect_one()) {
      const uint32_t idesc = make_idesc_bf16(128, g.n16, true, false);
      const uint64_t xd0 = make_smem_desc(smem_u32(xs), g.k16 * 128, 1024, 2), td0 = make_smem_desc(smem_u32(tw), 16, 1024, 2);
      const uint64_t part16 = part >> 4, table16 = table >> 4;
      uint32_t it = 0;
      for (int t = blockIdx.x; t < tiles; t += gridDim.x, ++it) {
        const int a = it & 1;
        if (!mbar_wait(&tempty[a], ((it >> 1) & 1) ^ 1, abort_flag, g.err, ERR_WAIT_TMEM_EMPTY)) break;
        if (!mbar_wait(&afull, it & 1, abort_flag, g.err, ERR_WAIT_FULL)) break;
        tc_fence_after();
#pragma unroll 1
        for (int e = 0; e < 2; ++e)              // Re cos, Im sin
#pragma unroll
          for (int order = 2; order >= 0; --order)           // small terms first
#pragma unroll
            for (int i = order; i >= 0; --i)
              row_tc_products(tmem + a * 256 + e * 128, xd0 + (3 * e + i) * part16, td0 + (3 * e + order - i) * table16, g.k16 >> 4, g.n16 * 8, idesc,
                              order == 2 && i == 2 ? 0u : 1u);
        umma_commit(&aempty);
        umma_commit(&tfull[a]);
      }
    }
  } else {
    const int e = warp - kRowInvLoaders - 1, q = warp & 3, half = e >> 2, tid = e * 32 + lane;
    uint32_t it = 0;
    for (int t = blockIdx.x; t < tiles; t += gridDim.x, ++it) {
      const int a = it & 1, row = t / g.tiles_c, c0 = (t - row * g.tiles_c) * 128;
      // results leave in sets of kSet vectors a thread, whose addends the loading warps have brought to L2
      constexpr int kSet = 4, kStride = 32 * kRowInvEpilogue;
      uint4 b0[kSet], b1[kSet];
      auto inside = [&](int i) { return i < g.W * 16 && c0 + 8 * (i & 15) < g.C; };
      auto address = [&](int i) { return ((long long)row * g.W + (i >> 4)) * g.C + c0 + 8 * (i & 15); };
      auto load = [&](int i0) {
#pragma unroll
        for (int n = 0; n < kSet; ++n) {
          const int i = i0 + n * kStride;
          if (g.add0 && inside(i)) b0[n] = __ldg(reinterpret_cast<const uint4*>(g.add0 + address(i)));
          if (g.add1 && inside(i)) b1[n] = __ldg(reinterpret_cast<const uint4*>(g.add1 + address(i)));
        }
      };
      const bool ok = mbar_wait_warp(&tfull[a], (it >> 1) & 1, abort_flag, g.err, ERR_WAIT_TMEM_FULL);
      tc_fence_after();
      const uint32_t acc = tmem + a * 256 + (uint32_t(q * 32) << 16);
      // A thread has one channel; with its neighbour's values of the same two positions it stores two channels of one of them.
      const int odd = lane & 1;
      uint32_t* col = reinterpret_cast<uint32_t*>(ys) + (q * 32 + lane) / 2;
      auto put = [&](int w, uint64_t v) {        // v: positions of even and of odd lanes; w: this lane's
        const uint32_t own = f2_to_bf16x2(v), other = __shfl_xor_sync(0xffffffffu, own, 1);
        if (w >= 0) col[w * (kRowInvLd / 2)] = odd ? __byte_perm(other, own, 0x7632) : __byte_perm(own, other, 0x5410);
      };
      if (ok)
        for (int j = half; j < g.n16 / 16; j += 2) {
          float A[16], B[16];
          tmem_ld16(acc + 16 * j, A);
          tmem_ld16(acc + 128 + 16 * j, B);
          tmem_ld_wait();
          const uint64_t scale = f2_all(g.scale);
#pragma unroll
          for (int i = 0; i < 16; i += 2) {
            const uint64_t x = f2_make(A[i], A[i + 1]), z = f2_make(B[i], B[i + 1]);
            const int w = 16 * j + i + odd;
            put(2 * w <= g.W ? w : -1, f2_mul(f2_fma(z, f2_all(-1.f), x), scale));
            put(w > 0 && 2 * w < g.W ? g.W - w : -1, f2_mul(f2_add(x, z), scale));
          }
        }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&tempty[a]);
      asm volatile("bar.sync 1, 256;" ::: "memory");         // all eight warps come here for every tile, also after a wait that ran out
      for (int i0 = tid; i0 < g.W * 16; i0 += kSet * kStride) {
        if (g.add0) load(i0);
#pragma unroll
        for (int n = 0; n < kSet; ++n) {
          const int i = i0 + n * kStride;
          if (!inside(i) || !ok) continue;
          uint4 u = *reinterpret_cast<const uint4*>(ys + (i >> 4) * kRowInvLd + 8 * (i & 15));
          if (g.add0) {                          // residual terms of the surrounding block: added in fp32 to the rounded transform, rounded again
            uint64_t f[4] = {f2_from_bf16x2(u.x), f2_from_bf16x2(u.y), f2_from_bf16x2(u.z), f2_from_bf16x2(u.w)};
            auto add = [&](const uint4& b) {
              f[0] = f2_add(f[0], f2_from_bf16x2(b.x)); f[1] = f2_add(f[1], f2_from_bf16x2(b.y));
              f[2] = f2_add(f[2], f2_from_bf16x2(b.z)); f[3] = f2_add(f[3], f2_from_bf16x2(b.w));
            };
            add(b0[n]);
            if (g.add1) add(b1[n]);
            u = make_uint4(f2_to_bf16x2(f[0]), f2_to_bf16x2(f[1]), f2_to_bf16x2(f[2]), f2_to_bf16x2(f[3]));
          }
          *reinterpret_cast<uint4*>(g.y + address(i)) = u;
        }
      }
      asm volatile("bar.sync 1, 256;" ::: "memory");
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == kRowInvLoaders) {
    if (abort_word) abort_settle();
    tc_fence_after();
    tmem_dealloc(tmem, 512);
  }
}

// 0, an error, or 1 where it does not apply: two accumulators of W / 2 + 1 columns, shared memory, alignment.
inline int launch_rows_c2r_tc(const float2* X, void* y, const void* add0, const void* add1, int rows, int W, int C, int KX, int kweight, int num_sms,
                              int* err, cudaStream_t stream) {
  RowInvArgs g;
  g.X = X; g.y = reinterpret_cast<__nv_bfloat16*>(y);
  g.add0 = reinterpret_cast<const __nv_bfloat16*>(add0); g.add1 = reinterpret_cast<const __nv_bfloat16*>(add1);
  g.rows = rows; g.W = W; g.C = C; g.KX = KX; g.kweight = kweight; g.err = err;
  g.k16 = (KX + 15) / 16 * 16; g.n16 = (W / 2 + 1 + 15) / 16 * 16; g.chunks = (g.k16 + 63) / 64;
  g.scale = 1.f / sqrtf(float(W));
  g.tiles_c = (C + 127) / 128;
  const uintptr_t all = reinterpret_cast<uintptr_t>(X) | reinterpret_cast<uintptr_t>(y) | reinterpret_cast<uintptr_t>(add0) | reinterpret_cast<uintptr_t>(add1);
  if (g.n16 > 128 || (all & 15) || C % 8) return 1;
  // The tables cost a CTA 6 us: rows of an even length, which have a fast direct sum, want tiles to share them (45 x 90 tokens of 768, 270
  // tiles: 20.5 -> 16.4 us; 30 x 60, 180 tiles: 12.3 -> 14.3).  Odd rows always gain (12 x 255 tokens of 64 61 -> 18 us).
  if (W % 2 == 0 && 2LL * rows * g.tiles_c < 3LL * num_sms) return 1;
  const int smem = 1024 + 6 * row_tc_table_bytes(g.n16, g.chunks) + 6 * 2 * g.k16 * 128 + W * kRowInvLd * 2;
  if (smem > 225 * 1024) return 1;
  static DeviceMask smem_set{0};
  if (!allow_smem(afno_rows_c2r_tc_kernel, 225 * 1024, smem_set)) return -4;
  const int tiles = rows * g.tiles_c;
  afno_rows_c2r_tc_kernel<<<tiles < num_sms ? tiles : num_sms, kRowInvThreads, smem, stream>>>(g);
  return cudaGetLastError() == cudaSuccess ? 0 : -3;
}

}  // namespace pnm

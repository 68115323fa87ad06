// C[M,N] = epilogue( A[M,K] * B[N,K]^T ), bf16 operands, fp32 accumulation in TMEM.
//
// One persistent CTA per SM, warp-specialised:
//   warp 0      TMA producer (A and B k-blocks of 64 -> 128-byte-swizzled shared tiles)
//   warp 1      tcgen05.mma issuer (one lane), owns the TMEM allocation
//   warps 2..   epilogue: TMEM -> registers -> fused math -> swizzled staging -> TMA store; one warp per 32 x 64 block of the
//               tile, i.e. 8 warps for 128 columns and 16 for 256.  With 8 warps on 256 columns (two blocks each) the products
//               with a heavy epilogue were bound by the latency of its instructions, not by memory or the tensor cores:
//               1 M rows, softmax 256 -> 512 0.85 -> 0.53 ms.  With an auxiliary operand the tiles were 128 columns wide and
//               read A twice as often: GELU' 256 -> 1024 1.40 -> 0.99 ms, softmax backward 512 -> 512 1.28 -> 0.83 ms.
// Two TMEM accumulators let the epilogue of tile i overlap the main loop of tile i+1.
// The arithmetic of an epilogue works on two columns per instruction (f2_*): one by one, a softmax took 20 instructions a value, its
// backward 35, GELU' 20.  1 M rows, softmax 256 -> 512 532 -> 352 us (its writes alone are worth 262: a stream of writes runs at 3.9 TB/s
// here), softmax backward 512 -> 512 986 -> 850 us (bound by the operands' way from L2, 448 KB a tile), GELU' 256 -> 1024 990 -> 950 us.
//
// Fused epilogues (all optional, all applied on fp32 values):
//   x = (acc + bias[col]) * scale[col]            (scale before the activation unless scale_post)
//   Z = x                                         (second output: the pre-activation, MODE_Z)
//   y = act(x)   act in {none, GELU, SiLU, ReLU, softmax over aligned groups of 64 columns}
//   y = y + aux | y * GELU'(aux) | y * SiLU'(aux) | y * ReLU'(aux) | softmax-backward(y; aux = p)
// The auxiliary tile is prefetched by TMA into the same staging buffer the result leaves from.
// A may be split along K into up to three tensors (A | A2 | A3), which gives K-concatenated GEMMs
// without materialising the concatenation.
#pragma once
#include "common.cuh"
#include "tmap.cuh"
#include "pnm_internal.h"

namespace pnm {

enum { ACT_NONE = 0, ACT_GELU = 1, ACT_SILU = 2, ACT_RELU = 3, ACT_SOFTMAX64 = 4 };
enum { AUX_NONE = 0, AUX_ADD = 1, AUX_DGELU = 2, AUX_DSOFTMAX = 3, AUX_DSILU = 4, AUX_DRELU = 5 };
enum { MODE_PLAIN = 0, MODE_Z = 1, MODE_AUX = 2 };

struct GemmArgs {
  int M, N, K, K1, K2;
  const float* bias;
  const float* scale;
  float* group_out;
  int act;
  int aux_mode;
  int scale_post;
  int num_m_tiles, num_n_tiles;
  int* err;
  // stacked batch (batch_m_tiles != 0): A / C hold `batch` problems of batch_m_tiles * 128 rows one after the other, B holds
  // their [N, K] matrices one after the other, bias / scale their [N] vectors: M tile mt belongs to problem mt / batch_m_tiles
  int batch_m_tiles;
  // split_m (BN = 256 instantiation only): a tile is TWO 128-row sub-tiles that share one 128-column B tile, i.e. 256 x 128
  // outputs.  For N <= 128 this reads B once per 256 rows instead of once per 128 (the 128 x 128 tile is bound by the
  // L2 -> shared-memory traffic of its operands); stage size, TMEM layout and the epilogue's warp mapping are those of
  // the 128 x 256 tile with "column half" replaced by "row half".  num_m_tiles counts 256-row tiles.
  int split_m;
  // implicit-GEMM convolution (conv != 0): rows of A are output pixels of an NHWC image, tiled 8 x 16 per M tile;
  // K runs over (tap, input channel); the A tile of k-block (tap, c0) is the input window shifted by the tap
  int conv, tiles_x, tiles_y, cin, ksize, pad, img_h;
  // halo != 0 (3 x 3, img_h % 8 == 0): the image is one horizontal slab of a taller image split over ranks.  The row
  // above / below the slab comes from the neighbour's published boundary row (a peer-mapped buffer read by plain,
  // non-multicast TMA loads) once its flag carries halo_epoch; tiles that need it are scheduled last.
  int halo, has_up, has_down, img_n;
  const uint32_t* flag_up;
  const uint32_t* flag_down;
  uint32_t halo_epoch;
  unsigned long long halo_budget_ns;  // budget of the waits on the neighbours' flags
};

constexpr int kConvTileH = 8;
constexpr int kConvTileW = 16;

__device__ __forceinline__ void conv_tile_origin(const GemmArgs& g, int mt, int& n, int& y0, int& x0) {
  if (g.halo) {
    // interior-first order: tile rows 1 .. tiles_y-2 of every image, then row 0 and row tiles_y-1 (the halo users)
    const int per_row = g.img_n * g.tiles_x;
    const int o = mt / per_row, r = mt - o * per_row;
    n = r / g.tiles_x;
    x0 = (r % g.tiles_x) * kConvTileW;
    const int ty = g.tiles_y <= 2 ? o : (o < g.tiles_y - 2 ? o + 1 : (o == g.tiles_y - 2 ? 0 : g.tiles_y - 1));
    y0 = ty * kConvTileH;
    return;
  }
  const int per_img = g.tiles_x * g.tiles_y;
  n = mt / per_img;
  const int r = mt - n * per_img;
  y0 = (r / g.tiles_x) * kConvTileH;
  x0 = (r % g.tiles_x) * kConvTileW;
}

// Bounded wait (one thread) until a flag written by another GPU reaches `epoch`.
// The rows that the flag announces were written by another GPU with generic-proxy stores and are read here by TMA
// (async proxy): after the acquire succeeds a proxy fence orders the two before the first bulk copy is issued.
__device__ __forceinline__ void fence_proxy_async_global() { asm volatile("fence.proxy.async.global;" ::: "memory"); }
__device__ __forceinline__ bool wait_remote_flag(const uint32_t* flag, uint32_t epoch, volatile int* abort_flag, int* err_word,
                                                 unsigned long long budget_ns) {
  uint32_t v;
  asm volatile("ld.acquire.sys.global.u32 %0, [%1];" : "=r"(v) : "l"(flag) : "memory");
  if (int32_t(v - epoch) >= 0) { fence_proxy_async_global(); return true; }
  const unsigned long long t0 = globaltimer_ns();
  uint32_t spins = 0;
  while (true) {
    asm volatile("ld.acquire.sys.global.u32 %0, [%1];" : "=r"(v) : "l"(flag) : "memory");
    if (int32_t(v - epoch) >= 0) { fence_proxy_async_global(); return true; }
    if ((++spins & 0xffu) == 0) {
      if (*abort_flag) return false;
      if (globaltimer_ns() - t0 > budget_ns) {
        atomicCAS(err_word, 0, ERR_WAIT_PEER);
        *abort_flag = 1;
        __threadfence_block();
        return false;
      }
    }
  }
}

constexpr int kBM = 128;
constexpr int kBK = 64;
constexpr int kChunkBytes = 32 * 128;  // 32 rows x 64 bf16

template <int BN, int MODE>
struct GemmCfg {
  static constexpr int EPI = BN / 16;         // epilogue warps: 4 lane quarters x (BN / 64) column blocks
  static constexpr int THREADS = 64 + 32 * EPI;
  // staging buffers of a warp: the auxiliary tile of the next block is prefetched while this one is worked on (128 columns: two
  // ahead); two outputs (128 columns only) alternate.  256 columns without an auxiliary tile leave the shared memory to the operand
  // stages.
  static_assert(BN == 128 || MODE != MODE_Z, "two outputs: 128-column tiles");
  static constexpr int NBUF = BN == 256 ? (MODE == MODE_AUX ? 2 : 1) : (MODE == MODE_AUX ? 3 : 2);
  static constexpr int STAGE_BYTES = kBM * kBK * 2 + BN * kBK * 2;
  static constexpr int STAGING = EPI * NBUF * kChunkBytes;
  static constexpr int BUDGET = 232448 - 1024 /*align*/ - 512 /*barriers*/;
  static constexpr int STAGES_RAW = (BUDGET - STAGING) / STAGE_BYTES;
  static constexpr int STAGES = STAGES_RAW > 6 ? 6 : STAGES_RAW;
  static constexpr int SMEM = 1024 + STAGES * STAGE_BYTES + STAGING + 512;
  static constexpr int TMEM_COLS = 2 * BN;  // 256 or 512: powers of two
  static_assert(STAGES >= 2, "not enough shared memory for a pipeline");
};

// The epilogues work on pairs of columns (f2_*, common.cuh): a row's values are an array of 32 pairs.
// 64 columns -> 64 bf16 = 8 chunks of 16 bytes, chunk j of row r lands at (j ^ (r & 7)).
__device__ __forceinline__ void stage_write16(uint8_t* buf, int lane, int k, const uint64_t* x) {
#pragma unroll
  for (int j = 0; j < 2; ++j)
    *reinterpret_cast<uint4*>(buf + lane * 128 + (((2 * k + j) ^ (lane & 7)) << 4)) =
        make_uint4(f2_to_bf16x2(x[4 * j]), f2_to_bf16x2(x[4 * j + 1]), f2_to_bf16x2(x[4 * j + 2]), f2_to_bf16x2(x[4 * j + 3]));
}
__device__ __forceinline__ void stage_write_row(uint8_t* buf, int lane, const uint64_t* v) {
#pragma unroll
  for (int k = 0; k < 4; ++k) stage_write16(buf, lane, k, v + 8 * k);
}
// columns [16 k, 16 k + 16) of a staged row
__device__ __forceinline__ void stage_read16(const uint8_t* buf, int lane, int k, uint64_t* a) {
#pragma unroll
  for (int j = 0; j < 2; ++j) {
    const uint4 u = *reinterpret_cast<const uint4*>(buf + lane * 128 + (((2 * k + j) ^ (lane & 7)) << 4));
    a[4 * j] = f2_from_bf16x2(u.x); a[4 * j + 1] = f2_from_bf16x2(u.y); a[4 * j + 2] = f2_from_bf16x2(u.z); a[4 * j + 3] = f2_from_bf16x2(u.w);
  }
}
// 32 columns of a row of the accumulator
__device__ __forceinline__ void tmem_ld_pairs(uint32_t taddr, uint64_t* v) {
  float t[32];
  tmem_ld32(taddr, t);
  tmem_ld_wait();
#pragma unroll
  for (int j = 0; j < 16; ++j) v[j] = f2_make(t[2 * j], t[2 * j + 1]);
}
// v <- v + p or v * p for the 2 NP columns from c0 on; p: vector of the columns (`vec`: whole and 16-byte aligned here), N of them
template <int NP, bool MUL>
__device__ __forceinline__ void epi_vector(uint64_t* v, const float* __restrict__ p, int c0, int N, bool vec) {
  if (vec) {
#pragma unroll
    for (int j = 0; j < NP / 2; ++j) {
      const float4 b = __ldg(reinterpret_cast<const float4*>(p + c0) + j);
      v[2 * j] = MUL ? f2_mul(v[2 * j], f2_make(b.x, b.y)) : f2_add(v[2 * j], f2_make(b.x, b.y));
      v[2 * j + 1] = MUL ? f2_mul(v[2 * j + 1], f2_make(b.z, b.w)) : f2_add(v[2 * j + 1], f2_make(b.z, b.w));
    }
  } else {
#pragma unroll
    for (int j = 0; j < NP; ++j) {
      const int c = c0 + 2 * j;
      const uint64_t b = f2_make(c < N ? __ldg(p + c) : 0.f, c + 1 < N ? __ldg(p + c + 1) : 0.f);
      v[j] = MUL ? f2_mul(v[j], b) : f2_add(v[j], b);
    }
  }
}
template <int NP>
__device__ __forceinline__ void epi_act(uint64_t* v, int act) {
  switch (act) {
    case ACT_GELU:
#pragma unroll
      for (int j = 0; j < NP; ++j) v[j] = gelu_f2(v[j]);
      break;
    case ACT_SILU:
#pragma unroll
      for (int j = 0; j < NP; ++j) v[j] = silu_f2(v[j]);
      break;
    case ACT_RELU:
#pragma unroll
      for (int j = 0; j < NP; ++j) {
        const float2 x = f2_get(v[j]);
        v[j] = f2_make(fmaxf(x.x, 0.f), fmaxf(x.y, 0.f));
      }
      break;
    default: break;
  }
}
// 16 columns with the auxiliary values of the same columns (all modes but the softmax backward; `ALL` false: those with arithmetic on
// the auxiliary values, the only ones that come to the 256-column tiles of one CTA)
template <bool ALL>
__device__ __forceinline__ void epi_aux16(uint64_t* v, const uint64_t* a, int mode) {
  switch (mode) {
    case AUX_ADD:
      if (ALL) {
#pragma unroll
        for (int j = 0; j < 8; ++j) v[j] = f2_add(v[j], a[j]);
      }
      break;
    case AUX_DGELU:
#pragma unroll
      for (int j = 0; j < 8; ++j) v[j] = f2_mul(v[j], gelu_grad_f2(a[j]));
      break;
    case AUX_DSILU:
#pragma unroll
      for (int j = 0; j < 8; ++j) v[j] = f2_mul(v[j], silu_grad_f2(a[j]));
      break;
    case AUX_DRELU:
      if (ALL) {
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          const float2 x = f2_get(v[j]), z = f2_get(a[j]);
          v[j] = f2_make(z.x > 0.f ? x.x : 0.f, z.y > 0.f ? x.y : 0.f);
        }
      }
      break;
    default: break;
  }
}
// softmax over a thread's 64 columns
__device__ __forceinline__ void epi_softmax64(uint64_t* v) {
  float m[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const float2 x = f2_get(v[i]);
    m[i] = fmaxf(x.x, x.y);
  }
#pragma unroll
  for (int j = 4; j < 32; ++j) {
    const float2 x = f2_get(v[j]);
    m[j & 3] = fmaxf(m[j & 3], fmaxf(x.x, x.y));
  }
  const uint64_t neg = f2_all(-fmaxf(fmaxf(m[0], m[1]), fmaxf(m[2], m[3]))), log2e = f2_all(1.4426950409f);
  uint64_t s[2] = {0, 0};
#pragma unroll
  for (int j = 0; j < 32; ++j) {
    const float2 x = f2_get(f2_mul(f2_add(v[j], neg), log2e));
    v[j] = f2_make(ex2_fast(x.x), ex2_fast(x.y));
    s[j & 1] = f2_add(s[j & 1], v[j]);
  }
  const float2 t = f2_get(f2_add(s[0], s[1]));
  const uint64_t inv = f2_all(__frcp_rn(t.x + t.y));
#pragma unroll
  for (int j = 0; j < 32; ++j) v[j] = f2_mul(v[j], inv);
}
// softmax backward of 16 columns: v <- a (v - dot); the sum of v log2(a) where a group's sum is wanted.  Where a is 0, so is v: the
// logarithm is that of the smallest normal number and the product 0.
template <bool SUM>
__device__ __forceinline__ void epi_dsoftmax16(uint64_t* v, const uint64_t* a, uint64_t neg_dot, uint64_t& sum) {
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    v[j] = f2_mul(a[j], f2_add(v[j], neg_dot));
    if (SUM) {
      const float2 p = f2_get(a[j]);
      sum = f2_fma(v[j], f2_make(lg2_fast(fmaxf(p.x, 1.17549435e-38f)), lg2_fast(fmaxf(p.y, 1.17549435e-38f))), sum);
    }
  }
}

template <int BN, int MODE>
__global__ void __launch_bounds__(GemmCfg<BN, MODE>::THREADS, 1)
gemm_tn_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmA2,
               const __grid_constant__ CUtensorMap tmA3, const __grid_constant__ CUtensorMap tmB, const __grid_constant__ CUtensorMap tmC,
               const __grid_constant__ CUtensorMap tmX /* Z (store) or aux (load) */, const GemmArgs g) {
  using Cfg = GemmCfg<BN, MODE>;
  constexpr int STAGES = Cfg::STAGES;
  constexpr int NBUF = Cfg::NBUF;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* base = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* staging = base + STAGES * Cfg::STAGE_BYTES;
  uint64_t* bars = reinterpret_cast<uint64_t*>(staging + Cfg::STAGING);
  uint64_t* full = bars;
  uint64_t* empty = bars + STAGES;
  uint64_t* tfull = bars + 2 * STAGES;
  uint64_t* tempty = tfull + 2;
  uint64_t* auxbar = tempty + 2;                      // [epilogue warps][NBUF]
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(auxbar + Cfg::EPI * NBUF);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int num_tiles = g.num_m_tiles * g.num_n_tiles;
  const int num_kb = (g.K + kBK - 1) / kBK;

  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) { mbar_init(&full[s], 1); mbar_init(&empty[s], 1); }
    for (int a = 0; a < 2; ++a) { mbar_init(&tfull[a], 1); mbar_init(&tempty[a], Cfg::EPI); }
    for (int i = 0; i < Cfg::EPI * NBUF; ++i) mbar_init(&auxbar[i], 1);
    *abort_flag = 0;
    mbar_fence_init();
    tma_prefetch_desc(&tmA); tma_prefetch_desc(&tmB); tma_prefetch_desc(&tmC);
  }
  if (warp == 1) { tmem_alloc(tmem_slot, Cfg::TMEM_COLS); tmem_relinquish(); }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;

  if (warp == 0) {
    // ------------------------------------------------------------ producer
    if (elect_one()) {
      uint32_t it = 0;
      bool ok = true;
      bool up_ready = false, down_ready = false;
      for (int tile = blockIdx.x; ok && tile < num_tiles; tile += gridDim.x) {
        const int mt = tile / g.num_n_tiles, nt = tile % g.num_n_tiles;
        for (int kb = 0; kb < num_kb; ++kb, ++it) {
          const int s = it % STAGES;
          const uint32_t ph = (it / STAGES) & 1;
          if (!mbar_wait(&empty[s], ph ^ 1, abort_flag, g.err, ERR_WAIT_EMPTY)) { ok = false; break; }
          uint8_t* sa = base + s * Cfg::STAGE_BYTES;
          uint8_t* sb = sa + kBM * kBK * 2;
          mbar_expect_tx(&full[s], Cfg::STAGE_BYTES);
          const int k = kb * kBK;
          auto load_a = [&](uint8_t* sa, int mt) -> bool {
            if (g.conv) {
              int n, y0, x0;
              conv_tile_origin(g, mt, n, y0, x0);
              const int tap = k / g.cin, c0 = k - tap * g.cin;
              const int xs = x0 + tap % g.ksize - g.pad, ys = y0 + tap / g.ksize - g.pad;
              if (g.halo && ys < 0 && g.has_up) {
                // box rows -1 .. 6: row -1 is the upper neighbour's bottom row, rows 0 .. 6 are local
                if (!up_ready) {
                  if (!wait_remote_flag(g.flag_up, g.halo_epoch, abort_flag, g.err, g.halo_budget_ns)) return false;
                  up_ready = true;
                }
                tma_load_4d(sa, &tmA3, &full[s], c0, xs, 0, n);
                tma_load_4d(sa + kConvTileW * 128, &tmA2, &full[s], c0, xs, 0, n);
              } else if (g.halo && ys + kConvTileH > g.img_h && g.has_down) {
                // box rows H-7 .. H: rows H-7 .. H-1 are local, row H is the lower neighbour's top row
                if (!down_ready) {
                  if (!wait_remote_flag(g.flag_down, g.halo_epoch, abort_flag, g.err, g.halo_budget_ns)) return false;
                  down_ready = true;
                }
                tma_load_4d(sa, &tmA2, &full[s], c0, xs, ys, n);
                tma_load_4d(sa + (kConvTileH - 1) * kConvTileW * 128, &tmX, &full[s], c0, xs, 0, n);
              } else {
                tma_load_4d(sa, &tmA, &full[s], c0, xs, ys, n);
              }
            } else if (k < g.K1) tma_load_2d(sa, &tmA, &full[s], k, mt * kBM);
            else if (k < g.K2) tma_load_2d(sa, &tmA2, &full[s], k - g.K1, mt * kBM);
            else tma_load_2d(sa, &tmA3, &full[s], k - g.K2, mt * kBM);
            return true;
          };
          if (BN == 256 && g.split_m) {
            if (!load_a(sa, 2 * mt) || !load_a(sa + kBM * kBK * 2, 2 * mt + 1)) { ok = false; break; }
            tma_load_2d(sa + 2 * kBM * kBK * 2, &tmB, &full[s], k, nt * 128);
            continue;
          }
          if (!load_a(sa, mt)) { ok = false; break; }
          tma_load_2d(sb, &tmB, &full[s], k, nt * BN + (g.batch_m_tiles ? (mt / g.batch_m_tiles) * g.N : 0));
        }
      }
      ring_drain(full, STAGES, it);
      if (!ok) abort_settle();                   // the loads of a stage that was only begun complete no phase
    }
  } else if (warp == 1) {
    // ---------------------------------------------------------- MMA issuer
    if (elect_one()) {
      constexpr uint32_t idesc = make_idesc_bf16(kBM, BN, false, false);
      uint32_t it = 0, tc = 0;
      bool ok = true;
      for (int tile = blockIdx.x; ok && tile < num_tiles; tile += gridDim.x, ++tc) {
        const int acc = tc & 1;
        const uint32_t aph = (tc >> 1) & 1;
        if (!mbar_wait(&tempty[acc], aph ^ 1, abort_flag, g.err, ERR_WAIT_TMEM_EMPTY)) break;
        tc_fence_after();
        const uint32_t d = tmem_base + acc * BN;
        for (int kb = 0; kb < num_kb; ++kb, ++it) {
          const int s = it % STAGES;
          const uint32_t ph = (it / STAGES) & 1;
          if (!mbar_wait(&full[s], ph, abort_flag, g.err, ERR_WAIT_FULL)) { ok = false; break; }
          tc_fence_after();
          uint8_t* sa = base + s * Cfg::STAGE_BYTES;
          const uint64_t ad = make_smem_desc(smem_u32(sa), 16, 1024, 2);
          if (BN == 256 && g.split_m) {
            constexpr uint32_t idesc_half = make_idesc_bf16(kBM, 128, false, false);
            const uint64_t ad1 = make_smem_desc(smem_u32(sa + kBM * kBK * 2), 16, 1024, 2);
            const uint64_t bdh = make_smem_desc(smem_u32(sa + 2 * kBM * kBK * 2), 16, 1024, 2);
#pragma unroll
            for (int k = 0; k < kBK / 16; ++k) {
              umma_f16(d, ad + 2 * k, bdh + 2 * k, idesc_half, (kb | k) != 0 ? 1u : 0u);
              umma_f16(d + 128, ad1 + 2 * k, bdh + 2 * k, idesc_half, (kb | k) != 0 ? 1u : 0u);
            }
            umma_commit(&empty[s]);
            continue;
          }
          const uint64_t bd = make_smem_desc(smem_u32(sa + kBM * kBK * 2), 16, 1024, 2);
#pragma unroll
          for (int k = 0; k < kBK / 16; ++k)
            umma_f16(d, ad + 2 * k, bd + 2 * k, idesc, (kb | k) != 0 ? 1u : 0u);
          umma_commit(&empty[s]);
        }
        if (ok) umma_commit(&tfull[acc]);
      }
    }
  } else {
    // ------------------------------------------------------------ epilogue
    const int e = warp - 2, q = warp & 3, h = e >> 2;   // lane quarter, 64-column block
    uint8_t* stg = staging + e * NBUF * kChunkBytes;
    uint64_t* mybar = auxbar + e * NBUF;
    uint32_t use = 0, tc = 0;
    bool ok = true;

    auto item_coords = [&](uint32_t item, int& r0, int& c0) -> bool {
      const int tile = blockIdx.x + int(item) * gridDim.x;
      if (tile >= num_tiles) return false;
      const int mt = tile / g.num_n_tiles, nt = tile % g.num_n_tiles;
      if (BN == 256 && g.split_m) {             // blocks 0, 1 are the columns of the first sub-tile, 2, 3 those of the second
        r0 = (2 * mt + (h >> 1)) * kBM + q * 32;
        c0 = nt * 128 + (h & 1) * 64;
        return true;
      }
      r0 = mt * kBM + q * 32;
      c0 = nt * BN + h * 64;
      return true;
    };
    auto issue_aux = [&](uint32_t item) {
      int r0, c0;
      if (!item_coords(item, r0, c0)) return;
      if (elect_one()) {
        tma_store_wait_read<NBUF - 2 < 0 ? 0 : NBUF - 2>();
        const int b = item % NBUF;
        mbar_expect_tx(&mybar[b], kChunkBytes);
        tma_load_2d(stg + b * kChunkBytes, &tmX, &mybar[b], c0, r0);
      }
    };
    if (MODE == MODE_AUX) issue_aux(0);
    auto add_group = [&](uint64_t sum, int c0, bool wanted) {      // of v log2(a), over the warp's 32 rows
      const float2 t = f2_get(sum);
      float gs = t.x + t.y;
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) gs += __shfl_xor_sync(0xffffffffu, gs, o);
      if (lane == 0 && c0 < g.N && wanted) atomicAdd(g.group_out + (c0 >> 6), gs * 0.6931471806f);
    };

    uint32_t item = 0;
    for (int tile = blockIdx.x; ok && tile < num_tiles; tile += gridDim.x, ++tc) {
      const int acc = tc & 1;
      const uint32_t aph = (tc >> 1) & 1;
      if (!mbar_wait_warp(&tfull[acc], aph, abort_flag, g.err, ERR_WAIT_TMEM_FULL)) break;
      tc_fence_after();
      {
        int r0, c0;
        item_coords(item, r0, c0);
        if (MODE == MODE_AUX) issue_aux(item + 1);
        const uint32_t taddr = tmem_base + acc * BN + h * 64 + (uint32_t(q * 32) << 16);
        if constexpr (BN == 256 && MODE == MODE_AUX) {
          // 16 columns at a time, straight from TMEM into the staged auxiliary tile (which the result replaces): a row of 64 and
          // its auxiliary values do not fit the 96 registers of a thread.  The softmax backward reads the accumulator twice.
          const bool store_ok = (r0 < g.M) && (c0 < g.N), full_cols = (c0 + 64 <= g.N);
          const bool bias_vec = full_cols && !(reinterpret_cast<uintptr_t>(g.bias) & 15);
          const bool scale_vec = full_cols && !(reinterpret_cast<uintptr_t>(g.scale) & 15);
          uint8_t* arow = stg + (item % NBUF) * kChunkBytes;
          auto load16 = [&](int k, uint64_t* x) {
            float t[16];
            tmem_ld16(taddr + 16 * k, t);
            tmem_ld_wait();
#pragma unroll
            for (int j = 0; j < 8; ++j) x[j] = f2_make(t[2 * j], t[2 * j + 1]);
            const int c = c0 + 16 * k;
            if (g.bias) epi_vector<8, false>(x, g.bias, c, g.N, bias_vec);
            if (g.scale && !g.scale_post) epi_vector<8, true>(x, g.scale, c, g.N, scale_vec);
            if (g.act) epi_act<8>(x, g.act);
          };
          if (!mbar_wait_warp(&mybar[item % NBUF], (item / NBUF) & 1, abort_flag, g.err, ERR_WAIT_AUX)) { ok = false; break; }
          uint64_t neg_dot = 0, gs = 0;
          if (g.aux_mode == AUX_DSOFTMAX) {
            uint64_t d[2] = {0, 0};
#pragma unroll 1
            for (int k = 0; k < 4; ++k) {
              uint64_t x[8], a[8];
              load16(k, x);
              stage_read16(arow, lane, k, a);
#pragma unroll
              for (int j = 0; j < 8; ++j) d[j & 1] = f2_fma(x[j], a[j], d[j & 1]);
            }
            const float2 t = f2_get(f2_add(d[0], d[1]));
            neg_dot = f2_all(-(t.x + t.y));
          }
#pragma unroll 1
          for (int k = 0; k < 4; ++k) {
            uint64_t x[8], a[8];
            load16(k, x);
            stage_read16(arow, lane, k, a);
            if (g.aux_mode != AUX_DSOFTMAX) epi_aux16<false>(x, a, g.aux_mode);
            else if (g.group_out) epi_dsoftmax16<true>(x, a, neg_dot, gs);
            else epi_dsoftmax16<false>(x, a, neg_dot, gs);
            if (g.scale && g.scale_post) epi_vector<8, true>(x, g.scale, c0 + 16 * k, g.N, scale_vec);
            stage_write16(arow, lane, k, x);
          }
          tc_fence_before();
          fence_async_smem();
          __syncwarp();
          if (elect_one()) {
            mbar_arrive(&tempty[acc]);
            if (store_ok) tma_store_2d(arow, &tmC, c0, r0);
            tma_store_commit();
          }
          if (g.group_out) add_group(gs, c0, g.aux_mode == AUX_DSOFTMAX);      // only the softmax backward has one
          ++item;
          continue;
        }
        const bool store_ok = (r0 < g.M) && (c0 < g.N);
        const bool full_cols = (c0 + 64 <= g.N);
        const int vo = g.batch_m_tiles ? (r0 / (kBM * g.batch_m_tiles)) * g.N : 0;   // offset of the problem's bias / scale
        // a vector may be a slice of a flat buffer that starts anywhere
        const bool bias_vec = full_cols && !(vo & 3) && !(reinterpret_cast<uintptr_t>(g.bias) & 15);
        const bool scale_vec = full_cols && !(vo & 3) && !(reinterpret_cast<uintptr_t>(g.scale) & 15);
        auto store = [&](uint8_t* buf) {          // the warp's block, written to `buf` by all lanes
          fence_async_smem();
          __syncwarp();
          if (elect_one()) {
            if (g.conv) {
              // this warp's 32 rows are two image rows of 16 pixels: one 4-D box; the copy engine clips at the image edge
              int n, y0, x0;
              conv_tile_origin(g, r0 / kBM, n, y0, x0);
              const int yy = y0 + 2 * q;
              if (r0 < g.M && c0 < g.N && yy < g.img_h) tma_store_4d(buf, &tmC, c0, x0, yy, n);
            } else if (store_ok) tma_store_2d(buf, &tmC, c0, r0);
            tma_store_commit();
          }
        };
        if (BN == 256 && MODE == MODE_PLAIN && g.act != ACT_SOFTMAX64) {
          // half a block at a time: with all 64 columns and the terms of an activation 96 registers spill
          if (elect_one()) tma_store_wait_read<0>();
          __syncwarp();
#pragma unroll 1
          for (int k = 0; k < 2; ++k) {
            uint64_t v[16];
            tmem_ld_pairs(taddr + 32 * k, v);
            if (g.bias) epi_vector<16, false>(v, g.bias + vo, c0 + 32 * k, g.N, bias_vec);
            if (g.scale && !g.scale_post) epi_vector<16, true>(v, g.scale + vo, c0 + 32 * k, g.N, scale_vec);
            if (g.act) epi_act<16>(v, g.act);
            if (g.scale && g.scale_post) epi_vector<16, true>(v, g.scale + vo, c0 + 32 * k, g.N, scale_vec);
            stage_write16(stg, lane, 2 * k, v);
            stage_write16(stg, lane, 2 * k + 1, v + 8);
          }
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(&tempty[acc]);
          store(stg);
          ++item;
          continue;
        }
        uint64_t v[32];
        tmem_ld_pairs(taddr, v);
        tmem_ld_pairs(taddr + 32, v + 16);
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&tempty[acc]);
        // ---- x = (acc + bias) * scale
        if (g.bias) epi_vector<32, false>(v, g.bias + vo, c0, g.N, bias_vec);
        if (g.scale && !g.scale_post) epi_vector<32, true>(v, g.scale + vo, c0, g.N, scale_vec);
        // ---- second output: pre-activation
        if (MODE == MODE_Z) {
          const int b = use % NBUF;
          if (elect_one()) tma_store_wait_read<NBUF - 1>();
          __syncwarp();
          stage_write_row(stg + b * kChunkBytes, lane, v);
          fence_async_smem();
          __syncwarp();
          if (elect_one()) {
            if (store_ok) tma_store_2d(stg + b * kChunkBytes, &tmX, c0, r0);
            tma_store_commit();
          }
          ++use;
        }
        // ---- activation
        if (g.act == ACT_SOFTMAX64) epi_softmax64(v);
        else if ((BN != 256 || MODE != MODE_PLAIN) && g.act) epi_act<32>(v, g.act);
        // ---- auxiliary operand
        int b = use % NBUF;
        if (MODE == MODE_AUX) {
          b = item % NBUF;
          const uint32_t bph = (item / NBUF) & 1;
          if (!mbar_wait_warp(&mybar[b], bph, abort_flag, g.err, ERR_WAIT_AUX)) { ok = false; break; }
          // read back 16 columns at a time: all 64 next to v would not fit the registers of a 16-warp epilogue
          const uint8_t* arow = stg + b * kChunkBytes;
          if (g.aux_mode != AUX_DSOFTMAX) {
#pragma unroll
            for (int k = 0; k < 4; ++k) {
              uint64_t a[8];
              stage_read16(arow, lane, k, a);
              epi_aux16<true>(v + 8 * k, a, g.aux_mode);
            }
          } else {
            uint64_t d[2] = {0, 0}, gs = 0;
#pragma unroll
            for (int k = 0; k < 4; ++k) {
              uint64_t a[8];
              stage_read16(arow, lane, k, a);
#pragma unroll
              for (int j = 0; j < 8; ++j) d[j & 1] = f2_fma(v[8 * k + j], a[j], d[j & 1]);
            }
            const float2 t = f2_get(f2_add(d[0], d[1]));
            const uint64_t neg_dot = f2_all(-(t.x + t.y));
#pragma unroll
            for (int k = 0; k < 4; ++k) {
              uint64_t a[8];
              stage_read16(arow, lane, k, a);
              if (g.group_out) epi_dsoftmax16<true>(v + 8 * k, a, neg_dot, gs);
              else epi_dsoftmax16<false>(v + 8 * k, a, neg_dot, gs);
            }
            if (g.group_out) add_group(gs, c0, true);
          }
        } else {
          if (elect_one()) tma_store_wait_read<NBUF - 1>();
          __syncwarp();
        }
        if (g.scale && g.scale_post) epi_vector<32, true>(v, g.scale + vo, c0, g.N, scale_vec);
        stage_write_row(stg + b * kChunkBytes, lane, v);
        store(stg + b * kChunkBytes);
        ++use;
        ++item;
      }
    }
    if (elect_one()) tma_store_wait_all<0>();
    __syncwarp();
  }
  // ------------------------------------------------------------- teardown
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base, Cfg::TMEM_COLS);
  }
}

// ---------------------------------------------------------------------- host
struct GemmCall {
  const void* A; int lda;
  const void* A2; int lda2;
  const void* A3; int lda3;
  const void* B; int ldb;
  void* C; int ldc;
  void* Z; int ldz;          // optional second output (pre-activation)
  const void* AUX; int ldaux; // optional auxiliary input [M,N]
  int M, N, K, K1, K2;
  const float* bias; const float* scale; float* group_out;
  int act, aux_mode, scale_post;
  int max_ctas;  // 0 = number of SMs
  int split_m = 0;  // BN = 256 instantiation as 256-row x 128-column tiles (see GemmArgs::split_m)
  int batch = 1; // > 1: `batch` stacked problems (see GemmArgs::batch_m_tiles); M is the total row count, M / batch % 128 == 0
  // convolution: A is an NHWC image [img_n, img_h, img_w, cin], B holds [N, ksize*ksize*cin] (tap-major), C is NHWC
  int conv = 0, img_n = 0, img_h = 0, img_w = 0, cin = 0, ksize = 0;
  // halo exchange fused into the convolution (see GemmArgs): boundary rows published by the neighbours [img_n, 1, img_w, cin]
  int halo = 0;
  const void* up_rows = nullptr; const void* down_rows = nullptr;
  const uint32_t* flag_up = nullptr; const uint32_t* flag_down = nullptr;
  uint32_t halo_epoch = 0;
  double halo_budget_s = 0.0;   // 0 = the library default
};

template <int BN, int MODE>
inline int launch_gemm_tn(const GemmCall& c, int num_sms, int* err_word, cudaStream_t stream) {
  using Cfg = GemmCfg<BN, MODE>;
  CUtensorMap tA, tA2, tA3, tB, tC, tX;
  if (c.conv) {
    if (MODE != MODE_PLAIN) return -19;
    if (make_tmap_nhwc_b16(&tA, c.A, c.img_n, c.img_h, c.img_w, c.cin, kConvTileH, kConvTileW)) return -10;
    if (c.halo) {
      if (c.ksize != 3 || (c.img_h % kConvTileH)) return -20;
      if (make_tmap_nhwc_b16(&tA2, c.A, c.img_n, c.img_h, c.img_w, c.cin, kConvTileH - 1, kConvTileW)) return -11;
      if (c.up_rows && make_tmap_nhwc_b16(&tA3, c.up_rows, c.img_n, 1, c.img_w, c.cin, 1, kConvTileW)) return -18;
      if (c.down_rows && make_tmap_nhwc_b16(&tX, c.down_rows, c.img_n, 1, c.img_w, c.cin, 1, kConvTileW)) return -15;
    }
  } else if (make_tmap_2d_b16(&tA, c.A, c.M, c.K1, c.lda, kBM, kBK)) return -10;
  const bool halo = c.conv && c.halo;
  if (c.K2 > c.K1) { if (make_tmap_2d_b16(&tA2, c.A2, c.M, c.K2 - c.K1, c.lda2, kBM, kBK)) return -11; }
  else if (!halo) tA2 = tA;
  if (c.K > c.K2) { if (make_tmap_2d_b16(&tA3, c.A3, c.M, c.K - c.K2, c.lda3, kBM, kBK)) return -18; }
  else if (!(halo && c.up_rows)) tA3 = tA;
  if (c.batch > 1 && (c.conv || c.M % (c.batch * kBM) || c.group_out)) return -21;
  const bool split = BN == 256 && MODE == MODE_PLAIN && c.split_m && c.batch <= 1;
  if (make_tmap_2d_b16(&tB, c.B, c.N * (c.batch > 1 ? c.batch : 1), c.K, c.ldb, split ? 128 : BN, kBK)) return -12;
  if (c.conv) { if (make_tmap_nhwc_b16(&tC, c.C, c.img_n, c.img_h, c.img_w, c.N, 2, kConvTileW)) return -13; }
  else if (make_tmap_2d_b16(&tC, c.C, c.M, c.N, c.ldc, 32, 64)) return -13;
  if (MODE == MODE_Z) { if (make_tmap_2d_b16(&tX, c.Z, c.M, c.N, c.ldz, 32, 64)) return -14; }
  else if (MODE == MODE_AUX) { if (make_tmap_2d_b16(&tX, c.AUX, c.M, c.N, c.ldaux, 32, 64)) return -15; }
  else if (!(halo && c.down_rows)) tX = tC;
  GemmArgs g;
  g.M = c.M; g.N = c.N; g.K = c.K; g.K1 = c.K1; g.K2 = c.K2;
  g.bias = c.bias; g.scale = c.scale; g.group_out = c.group_out;
  g.act = c.act; g.aux_mode = c.aux_mode; g.scale_post = c.scale_post;
  g.num_m_tiles = (c.M + kBM - 1) / kBM;
  g.num_n_tiles = (c.N + BN - 1) / BN;
  g.err = err_word;
  g.batch_m_tiles = c.batch > 1 ? c.M / c.batch / kBM : 0;
  g.split_m = split ? 1 : 0;
  g.conv = c.conv; g.cin = c.cin; g.ksize = c.ksize; g.pad = c.ksize / 2; g.img_h = c.img_h;
  g.tiles_x = g.tiles_y = 0;
  g.halo = c.conv ? c.halo : 0; g.has_up = c.up_rows != nullptr; g.has_down = c.down_rows != nullptr; g.img_n = c.img_n;
  g.flag_up = c.flag_up; g.flag_down = c.flag_down; g.halo_epoch = c.halo_epoch;
  g.halo_budget_ns = c.halo_budget_s > 0.0 ? (unsigned long long)(c.halo_budget_s * 1e9) : kWaitBudgetNs;
  if (c.conv) {
    g.tiles_x = (c.img_w + kConvTileW - 1) / kConvTileW;
    g.tiles_y = (c.img_h + kConvTileH - 1) / kConvTileH;
    g.num_m_tiles = c.img_n * g.tiles_x * g.tiles_y;
    g.M = g.num_m_tiles * kBM;            // every row of a tile is "in range"; the copy engine clips at image edges
  }
  static DeviceMask smem_set{0};
  if (!allow_smem(gemm_tn_kernel<BN, MODE>, Cfg::SMEM, smem_set)) return -16;
  if (split) {                                // 256-row tiles of 128 columns
    g.num_m_tiles = (g.num_m_tiles + 1) / 2;
    g.num_n_tiles = (c.N + 127) / 128;
  }
  int tiles = g.num_m_tiles * g.num_n_tiles;
  int cap = c.max_ctas > 0 ? c.max_ctas : num_sms;
  int grid = tiles < cap ? tiles : cap;
  gemm_tn_kernel<BN, MODE><<<grid, Cfg::THREADS, Cfg::SMEM, stream>>>(tA, tA2, tA3, tB, tC, tX, g);
  return cudaGetLastError() == cudaSuccess ? 0 : -17;
}

}  // namespace pnm

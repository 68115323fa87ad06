// Three-layer perceptron of 128-wide message-passing networks in one kernel:
//
//   h1 = act([s0[i0] | s1[i1] | s2[i2]] W1^T + b1)      up to three 128-wide sources, each read through an optional row index
//   h2 = act(h1 W2^T + b2)
//   y  = LayerNorm(h2 W3^T + b3) * gamma + beta (+ post)
//
// An edge row needs its own 256 bytes, two gathered node rows (mostly from L2) and 256 bytes of result; run layer by layer the
// same chain moves fifteen such rows through HBM.  Here everything between the sources and the result stays on the SM, and what
// is left is the latency of a tile's chain (product, epilogue, product, epilogue, product, normalisation):
// 1.4 M rows from three sources take 0.53 ms, where the rows' own traffic is worth 0.15 ms; with what the backward needs (five more
// rows each, 0.33 ms) 0.73 ms.  A MeshGraphNet step on 250 k nodes / 1.4 M edges, forward: 1.26 -> 0.70 ms.
//   * W1, W2, W3 (96 + 32 + 32 KB in bf16 for three sources) are loaded once per persistent CTA and stay in shared memory;
//   * gathered rows arrive by TMA gather4 (four indexed rows of 128 bytes per instruction, written in the same 128-byte
//     swizzle as a plain tile), so no gathered copy of the node features exists;
//   * accumulators are read back from TMEM by two threads per row (64 columns each), and the activations go back to TMEM as
//     the packed bf16 A operand of the next product (tcgen05.mma with A in tensor memory): hidden rows never use shared memory;
//   * the same two threads normalise the row (mean and squared deviations of each half, merged through two TMEM columns),
//     add `post` and store 32-byte vectors (whole sectors).
// Two row tiles of 128 are in flight, one per group of eight epilogue warps: the tensor cores
// work on one tile while the other is in its epilogue.  The only ring is that of the source tiles (64 columns each).
// One thread per row (half the warps) was no option: at 168 registers a thread the compiler spilled.
#pragma once
#include "common.cuh"
#include "tmap.cuh"
#include "pnm_internal.h"

namespace pnm {

constexpr int kMlpW = 128;                       // width of every layer
constexpr int kMlpRows = 128;                    // rows of a tile
constexpr int kMlpChunk = kMlpRows * 128;        // 128 rows x 64 bf16
constexpr int kMlpThreads = 640;                 // producer, MMA warp, 2 idle warps, 2 x 8 epilogue warps
constexpr int kMlpTmemCols = 512;                // per group of 256: accumulator 128, packed A operand 64, row statistics 8

enum { MLP_SILU = 2, MLP_RELU = 3, MLP_GELU = 1 };   // same codes as the GEMM epilogues

struct MlpArgs {
  long long M;
  const int* idx[3];                             // row index of a source, or null: row m itself
  const float *b1, *b2, *b3, *gamma, *beta;
  const __nv_bfloat16* post; long long ld_post;
  __nv_bfloat16* y; long long ld_y;
  // kept for the backward or null: pre-activations (whole tiles, see z_offset), their activations and the rows before the LayerNorm
  // (contiguous [M, 128]), the moments of the rounded rows.  ReLU keeps no pre-activations: the signs of the activations are all
  // that its derivative needs.
  __nv_bfloat16 *z1, *z2, *h1, *h2, *x3;
  float *mean, *rstd;
  float eps;
  int act;
  int* err;
};

// gather4: four rows of 64 columns, coordinates {x, r0, r1, r2, r3}
__device__ __forceinline__ void tma_gather4(void* smem_dst, const CUtensorMap* m, uint64_t* bar, int x, int r0, int r1, int r2, int r3) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cta.global.tile::gather4.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5, %6, %7}], [%2];"
      ::"r"(smem_u32(smem_dst)), "l"(reinterpret_cast<uint64_t>(m)), "r"(smem_u32(bar)), "r"(x), "r"(r0), "r"(r1), "r"(r2), "r"(r3)
      : "memory");
}
struct Vec32 { uint32_t w[8]; };                 // 16 bf16: one 32-byte sector
__device__ __forceinline__ Vec32 ldg32(const void* p) {
  Vec32 v;
  asm volatile("ld.global.v8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
               : "=r"(v.w[0]), "=r"(v.w[1]), "=r"(v.w[2]), "=r"(v.w[3]), "=r"(v.w[4]), "=r"(v.w[5]), "=r"(v.w[6]), "=r"(v.w[7])
               : "l"(p));
  return v;
}
__device__ __forceinline__ void stg32(void* p, const uint32_t* w) {
  asm volatile("st.global.v8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(p), "r"(w[0]), "r"(w[1]), "r"(w[2]), "r"(w[3]),
               "r"(w[4]), "r"(w[5]), "r"(w[6]), "r"(w[7])
               : "memory");
}
// 8 registers of bf16 pairs -> 32 lanes x 8 columns
__device__ __forceinline__ void tmem_st8(uint32_t taddr, const uint32_t* r) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]),
               "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7])
               : "memory");
}
// x[0..16) += 16 values in shared memory (the same for all lanes)
__device__ __forceinline__ void add_vec16(float* x, const float* v) {
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const float4 b = *reinterpret_cast<const float4*>(v + 4 * j);
    x[4 * j] += b.x; x[4 * j + 1] += b.y; x[4 * j + 2] += b.z; x[4 * j + 3] += b.w;
  }
}
__device__ __forceinline__ void tmem_st2(uint32_t taddr, float a, float b) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x2.b32 [%0], {%1, %2};" ::"r"(taddr), "r"(__float_as_uint(a)), "r"(__float_as_uint(b)) : "memory");
}
__device__ __forceinline__ float2 tmem_ld2(uint32_t taddr) {
  uint32_t a, b;
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x2.b32 {%0, %1}, [%2];" : "=r"(a), "=r"(b) : "r"(taddr) : "memory");
  tmem_ld_wait();
  return make_float2(__uint_as_float(a), __uint_as_float(b));
}
// barrier of the eight epilogue warps of a group
__device__ __forceinline__ void group_sync(int grp) { asm volatile("bar.sync %0, 256;" ::"r"(1 + grp) : "memory"); }
template <int ACT>
__device__ __forceinline__ float mlp_act(float x) {
  return ACT == MLP_SILU ? silu_f(x) : ACT == MLP_GELU ? gelu_f(x) : fmaxf(x, 0.f);
}

// Pre-activations lie as the threads hold them: vector c (16 columns) of lane l of a warp at (warp's block) + (32 c + l) * 16, so that a
// warp's 32-byte vectors are 1 KB in one piece, here and in the backward.  (With a row of its own per lane every access touches 32
// lines; the busiest unit of the kernel that keeps its rows is the one that handles those, at 61 %.)
__device__ __forceinline__ long long z_offset(long long tile, int q, int half, int lane) {
  return (((tile * 4 + q) * 2 + half) * 4 * 32 + lane) * 16;
}
constexpr int kZStep = 32 * 16;                  // elements from one vector of a thread to its next

template <int NSRC>
struct MlpCfg {
  static constexpr int WCHUNKS = 2 * NSRC + 4;                                    // 64-column blocks of W1 | W2 | W3
  static constexpr int SLOTS = NSRC == 3 ? 4 : 6;
  static constexpr int SMEM = (WCHUNKS + SLOTS) * kMlpChunk + 512 + 5 * kMlpW * 4;   // three sources: all 227 KB
};

template <int NSRC, int ACT, bool SAVE>
__global__ void __launch_bounds__(kMlpThreads, 1)
mlp3_ln_kernel(const __grid_constant__ CUtensorMap tm0, const __grid_constant__ CUtensorMap tm1, const __grid_constant__ CUtensorMap tm2,
               const __grid_constant__ CUtensorMap tmW1, const __grid_constant__ CUtensorMap tmW2, const __grid_constant__ CUtensorMap tmW3,
               const MlpArgs g) {
  using Cfg = MlpCfg<NSRC>;
  extern __shared__ __align__(1024) uint8_t smem_raw[];   // the only shared memory of the kernel: starts on a 1024-byte boundary
  uint8_t* wts = smem_raw;
  uint8_t* ring = wts + Cfg::WCHUNKS * kMlpChunk;
  float* vec = reinterpret_cast<float*>(ring + Cfg::SLOTS * kMlpChunk);      // b1, b2, b3, gamma, beta
  uint64_t* full = reinterpret_cast<uint64_t*>(vec + 5 * kMlpW);
  uint64_t* empty = full + Cfg::SLOTS;
  uint64_t* wfull = empty + Cfg::SLOTS;
  uint64_t* accfull = wfull + 1;                 // [2] an accumulator holds a finished product
  uint64_t* aready = accfull + 2;                // [2] the accumulator was read, the packed A operand (if any) is in place
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(aready + 2);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int tiles = int((g.M + kMlpRows - 1) / kMlpRows);
  constexpr int KB = 2 * NSRC;

  if (threadIdx.x == 0) {
    for (int s = 0; s < Cfg::SLOTS; ++s) { mbar_init(&full[s], 1); mbar_init(&empty[s], 1); }
    mbar_init(wfull, 1);
    for (int i = 0; i < 2; ++i) { mbar_init(&accfull[i], 1); mbar_init(&aready[i], 8); }
    *abort_flag = 0;
    mbar_fence_init();
    if (smem_u32(smem_raw) & 1023) { atomicCAS(g.err, 0, ERR_BAD_ARG); *abort_flag = 1; }
  }
  for (int i = threadIdx.x; i < 5 * kMlpW; i += kMlpThreads) {
    const float* src = i < kMlpW ? g.b1 : i < 2 * kMlpW ? g.b2 : i < 3 * kMlpW ? g.b3 : i < 4 * kMlpW ? g.gamma : g.beta;
    vec[i] = src ? src[i & (kMlpW - 1)] : 0.f;
  }
  if (warp == 1) { tmem_alloc(tmem_slot, kMlpTmemCols); tmem_relinquish(); }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;

  if (warp == 0) {
    // ------------------------------------------------------------------------------------------------ producer
    if (lane == 0) {
      mbar_expect_tx(wfull, Cfg::WCHUNKS * kMlpChunk);
      for (int k = 0; k < KB; ++k) tma_load_2d(wts + k * kMlpChunk, &tmW1, wfull, k * 64, 0);
      for (int k = 0; k < 2; ++k) tma_load_2d(wts + (KB + k) * kMlpChunk, &tmW2, wfull, k * 64, 0);
      for (int k = 0; k < 2; ++k) tma_load_2d(wts + (KB + 2 + k) * kMlpChunk, &tmW3, wfull, k * 64, 0);
    }
    uint32_t it = 0;
    bool ok = true;
    for (int tile = blockIdx.x; ok && tile < tiles; tile += gridDim.x) {
      const long long m0 = (long long)tile * kMlpRows;
#pragma unroll
      for (int j = 0; j < NSRC; ++j) {
        const CUtensorMap* tm = j == 0 ? &tm0 : (j == 1 ? &tm1 : &tm2);
        const int* ix = g.idx[j];
        int r[4] = {0, 0, 0, 0};
        if (ix) {
#pragma unroll
          for (int q = 0; q < 4; ++q) {          // rows past M repeat the last one: read, never stored
            const long long e = m0 + lane * 4 + q;
            r[q] = __ldg(ix + (e < g.M ? e : g.M - 1));
          }
        }
#pragma unroll
        for (int c = 0; c < 2; ++c, ++it) {
          const int s = it % Cfg::SLOTS;
          ok = mbar_wait(&empty[s], ((it / Cfg::SLOTS) & 1) ^ 1, abort_flag, g.err, ERR_WAIT_EMPTY);
          ok = __all_sync(0xffffffffu, ok);
          if (!ok) break;
          uint8_t* dst = ring + s * kMlpChunk;
          if (lane == 0) mbar_expect_tx(&full[s], kMlpChunk);
          __syncwarp();
          if (ix) tma_gather4(dst + lane * 512, tm, &full[s], c * 64, r[0], r[1], r[2], r[3]);
          else if (lane == 0) tma_load_2d(dst, tm, &full[s], c * 64, int(m0));
        }
        if (!ok) break;
      }
    }
    if (lane == 0) {                             // copies land before the CTA leaves, also after a wait that ran out
      mbar_drain(wfull, 0);
      ring_drain(full, Cfg::SLOTS, it);
    }
  } else if (warp == 1) {
    // -------------------------------------------------------------------------------- MMA issuer of both groups
    // One thread polls: a layer whose operand is in place goes first, then the next source chunk.  (An issuer per group would
    // wait on ring slots that it uses only every other tile: the parity of a slot two uses back looks like the next one.)
    if (lane == 0) {
      constexpr uint32_t idesc = make_idesc_bf16(kMlpRows, kMlpW, false, false);
      const int mine = tiles > int(blockIdx.x) ? (tiles - int(blockIdx.x) - 1) / int(gridDim.x) + 1 : 0;
      uint32_t arrivals[2] = {0, 0};             // phases of aready[grp] consumed so far
      int step[2] = {0, 0};                      // 0: first product not begun, 1: under way, 2 / 3: second / third product next
      uint32_t it = 0, kb = 0;
      int next = 0, finished = 0;
      unsigned long long t0 = 0;
      uint32_t spins = 0;
      bool ok = mbar_wait(wfull, 0, abort_flag, g.err, ERR_WAIT_FULL);
      while (ok && finished < mine) {
        bool any = false;
#pragma unroll
        for (int grp = 0; grp < 2; ++grp) {
          const uint32_t acc = tmem + grp * 256, aop = acc + 128;
          if (step[grp] >= 2 && mbar_try_wait(&aready[grp], arrivals[grp] & 1)) {
            ++arrivals[grp];
            tc_fence_after();
            const uint32_t w = smem_u32(wts + (KB + 2 * (step[grp] - 2)) * kMlpChunk);
#pragma unroll
            for (int k = 0; k < 8; ++k)
              umma_f16_ts(acc, aop + 8 * k, make_smem_desc(w + (k >> 2) * kMlpChunk, 16, 1024, 2) + 2 * (k & 3), idesc, k != 0 ? 1u : 0u);
            umma_commit(&accfull[grp]);
            if (step[grp] == 3) ++finished;
            step[grp] = step[grp] == 2 ? 3 : 0;
            any = true;
          }
          if (next < mine && (next & 1) == grp) {
            if (step[grp] == 0 && (next < 2 || mbar_try_wait(&aready[grp], arrivals[grp] & 1))) {   // the group's last tile was read
              if (next >= 2) ++arrivals[grp];
              step[grp] = 1;
              tc_fence_after();
            }
            const int s = it % Cfg::SLOTS;
            if (step[grp] == 1 && mbar_try_wait(&full[s], (it / Cfg::SLOTS) & 1)) {
              tc_fence_after();
              const uint64_t ad = make_smem_desc(smem_u32(ring + s * kMlpChunk), 16, 1024, 2);
              const uint64_t bd = make_smem_desc(smem_u32(wts + kb * kMlpChunk), 16, 1024, 2);
#pragma unroll
              for (int k = 0; k < 4; ++k) umma_f16(acc, ad + 2 * k, bd + 2 * k, idesc, (kb | k) != 0 ? 1u : 0u);
              umma_commit(&empty[s]);
              ++it;
              if (++kb == KB) {
                kb = 0;
                umma_commit(&accfull[grp]);
                step[grp] = 2;
                ++next;
              }
              any = true;
            }
          }
        }
        if (any) { spins = 0; t0 = 0; }
        else if ((++spins & 0x3ffu) == 0) {
          if (*abort_flag) break;
          const unsigned long long now = globaltimer_ns();
          if (t0 == 0) t0 = now;
          else if (now - t0 > kWaitBudgetNs) {
            atomicCAS(g.err, 0, ERR_WAIT_TMEM_EMPTY);
            *abort_flag = 1;
            __threadfence_block();
            break;
          }
        }
      }
    }
  } else if (warp >= 4) {
    // ----------------------------------------------------- epilogue: two threads per row, columns [64 half, 64 half + 64)
    const int grp = (warp - 4) >> 3, half = ((warp - 4) >> 2) & 1, q = warp & 3, col = half * 64;
    const uint32_t base = tmem + grp * 256 + (uint32_t(q * 32) << 16);
    const uint32_t acc = base + col, aop = base + 128 + half * 32, stat = base + 192;
    uint32_t n = 0, uses = 0;
    for (int tile = blockIdx.x; tile < tiles; tile += gridDim.x, ++n) {
      if ((n & 1) != uint32_t(grp)) continue;
      const long long row = (long long)tile * kMlpRows + q * 32 + lane;
      const bool live = row < g.M;
      bool ok = true;
#pragma unroll 1
      for (int layer = 0; layer < 2; ++layer) {
        const float* bias = vec + layer * kMlpW + col;
        __nv_bfloat16* z = (layer ? g.z2 : g.z1) + z_offset(tile, q, half, lane);
        __nv_bfloat16* h = (layer ? g.h2 : g.h1) + row * kMlpW + col;
        ok = mbar_wait(&accfull[grp], uses & 1, abort_flag, g.err, ERR_WAIT_TMEM_FULL);
        if (!__all_sync(0xffffffffu, ok)) { ok = false; break; }
        ++uses;
        tc_fence_after();
        float v[2][16];                          // two steps of 16 columns: one is read from TMEM while the other is worked on
        tmem_ld16(acc, v[0]);
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          tmem_ld_wait();
          if (c < 3) tmem_ld16(acc + (c + 1) * 16, v[(c + 1) & 1]);
          float* x = v[c & 1];
          add_vec16(x, bias + c * 16);
          uint32_t p[8];
          if (SAVE && ACT != MLP_RELU) {
#pragma unroll
            for (int j = 0; j < 8; ++j) p[j] = pack_bf16x2(x[2 * j], x[2 * j + 1]);
            stg32(z + c * kZStep, p);            // rows past M too: the buffer holds whole tiles
          }
#pragma unroll
          for (int j = 0; j < 8; ++j) p[j] = pack_bf16x2(mlp_act<ACT>(x[2 * j]), mlp_act<ACT>(x[2 * j + 1]));
          tmem_st8(aop + c * 8, p);
          if (SAVE && ACT == MLP_RELU && live) stg32(h + c * 16, p);
        }
        tmem_st_wait();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&aready[grp]);
        if (SAVE && ACT != MLP_RELU) {
          // The weight gradient's operand is this product's: recomputed from the rounded pre-activation it would be rounded twice (dW2
          // against 64 bits 0.0054 instead of 0.0049).  Read back and stored while the product runs (814 -> 778 us at 1.4 M rows; not
          // with ReLU, which stores nothing else: 631 -> 650 us).
#pragma unroll
          for (int c = 0; c < 2; ++c) {
            float p[16];
            tmem_ld16(aop + c * 16, p);
            tmem_ld_wait();
            if (live) {
              stg32(h + c * 32, reinterpret_cast<const uint32_t*>(p));
              stg32(h + c * 32 + 16, reinterpret_cast<const uint32_t*>(p) + 8);
            }
          }
        }
      }
      if (ok) {
        ok = mbar_wait(&accfull[grp], uses & 1, abort_flag, g.err, ERR_WAIT_TMEM_FULL);
        ok = __all_sync(0xffffffffu, ok);
      }
      ++uses;
      tc_fence_after();
      // moments of this half about its first element (a value of the row: no cancellation against a large mean)
      // (and, for the backward, those of the rounded rows that it will read: moments of other values would cost it precision)
      float pivot = 0.f, sum = 0.f, sq = 0.f, sum_k = 0.f, sq_k = 0.f;
      if (ok) {
        float v[2][16];
        tmem_ld16(acc, v[0]);
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          tmem_ld_wait();
          if (c < 3) tmem_ld16(acc + (c + 1) * 16, v[(c + 1) & 1]);
          float* x = v[c & 1];
          add_vec16(x, vec + 2 * kMlpW + col + c * 16);
          if (c == 0) pivot = x[0];
          if (SAVE) {
            uint32_t p[8];
#pragma unroll
            for (int j = 0; j < 8; ++j) {
              p[j] = pack_bf16x2(x[2 * j], x[2 * j + 1]);
              const float2 k = unpack_bf16x2(p[j]);
              const float d0 = k.x - pivot, d1 = k.y - pivot;
              sum_k += d0 + d1;
              sq_k = fmaf(d0, d0, fmaf(d1, d1, sq_k));
            }
            if (live) stg32(g.x3 + row * kMlpW + col + c * 16, p);
          }
#pragma unroll
          for (int j = 0; j < 16; ++j) { const float d = x[j] - pivot; sum += d; sq += d * d; }
        }
      }
      const float shift = sum * (1.f / 64), mean_h = pivot + shift, dev_h = fmaxf(sq - sum * shift, 0.f);
      const float shift_k = sum_k * (1.f / 64), mean_k = pivot + shift_k, dev_k = fmaxf(sq_k - sum_k * shift_k, 0.f);
      if (ok) {
        tmem_st2(stat + 2 * half, mean_h, dev_h);
        if (SAVE) tmem_st2(stat + 4 + 2 * half, mean_k, dev_k);
        tmem_st_wait();
      }
      Vec32 res = {};
      const __nv_bfloat16* post = g.post && live ? g.post + row * g.ld_post + col : nullptr;
      if (post) res = ldg32(post);
      tc_fence_before();
      __syncwarp();
      group_sync(grp);
      tc_fence_after();
      if (!__all_sync(0xffffffffu, ok && !*abort_flag)) continue;   // no warp leaves the loop early: a group's barriers need all
      // the halves' moments: mean = (a + b) / 2, squared deviations add up with 64 * 64 / 128 times the squared difference
      const float2 other = tmem_ld2(stat + 2 * (half ^ 1));
      const float mean = 0.5f * (mean_h + other.x), gap = mean_h - other.x;
      const float rstd = rsqrtf((dev_h + other.y + 32.f * gap * gap) * (1.f / kMlpW) + g.eps);
      if (SAVE) {
        const float2 other_k = tmem_ld2(stat + 4 + 2 * (half ^ 1));
        const float gap_k = mean_k - other_k.x;
        if (live && half == 0) {
          g.mean[row] = 0.5f * (mean_k + other_k.x);
          g.rstd[row] = rsqrtf((dev_k + other_k.y + 32.f * gap_k * gap_k) * (1.f / kMlpW) + g.eps);
        }
      }
#pragma unroll 1
      for (int c = 0; c < 4; ++c) {
        float v[16];
        tmem_ld16(acc + c * 16, v);
        Vec32 next = {};
        if (post && c < 3) next = ldg32(post + (c + 1) * 16);
        tmem_ld_wait();
        if (c == 3) {                            // the accumulator may be overwritten by the group's next tile
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(&aready[grp]);
        }
        uint32_t p[8];
        const float4* vb = reinterpret_cast<const float4*>(vec + 2 * kMlpW + col + c * 16);    // b3; gamma and beta follow
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const float4 b = vb[j], ga = vb[j + kMlpW / 4], be = vb[j + kMlpW / 2];
          const float2 r0 = unpack_bf16x2(res.w[2 * j]), r1 = unpack_bf16x2(res.w[2 * j + 1]);   // zeros without a residual
          const float h0 = (v[4 * j] + b.x - mean) * rstd, h1 = (v[4 * j + 1] + b.y - mean) * rstd, h2 = (v[4 * j + 2] + b.z - mean) * rstd,
                      h3 = (v[4 * j + 3] + b.w - mean) * rstd;
          p[2 * j] = pack_bf16x2(fmaf(h0, ga.x, be.x) + r0.x, fmaf(h1, ga.y, be.y) + r0.y);
          p[2 * j + 1] = pack_bf16x2(fmaf(h2, ga.z, be.z) + r1.x, fmaf(h3, ga.w, be.w) + r1.y);
        }
        if (live) stg32(g.y + row * g.ld_y + col + c * 16, p);
        res = next;
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    if (*abort_flag) abort_settle();
    tc_fence_after();
    tmem_dealloc(tmem, kMlpTmemCols);
  }
}

}  // namespace pnm

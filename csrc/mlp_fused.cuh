// Three-layer perceptron of 128-wide message-passing networks in one kernel:
//
//   h1 = act([s0[i0] | s1[i1] | s2[i2]] W1^T + b1)      up to three 128-wide sources, each read through an optional row index
//   h2 = act(h1 W2^T + b2)
//   y  = LayerNorm(h2 W3^T + b3) * gamma + beta (+ post)
//
// An edge row needs its own 256 bytes, two gathered node rows (mostly from L2) and 256 bytes of result; run layer by layer the
// same chain moves fifteen such rows through HBM.  Here everything between the sources and the result stays on the SM, and what
// is left is the chain of a tile (product, epilogue, product, epilogue, product, normalisation) and its instructions: 1.4 M rows from
// three sources take 0.31 ms (0.55 ms before the points marked * below), where its own traffic (row in and out, node rows once, indices:
// 0.80 GB at the 6.57 TB/s of a copy) is worth 0.12 ms; with what the backward needs (five more rows each, 1.82 GB, 0.28 ms) 0.59 ms (0.76).
//   * W1, W2, W3 (96 + 32 + 32 KB in bf16 for three sources) are loaded once per persistent CTA and stay in shared memory;
// * * gathered rows are copied 16 bytes at a time (cp.async), eight lanes to a row of 128 bytes, in the 128-byte swizzle of a plain
//     tile, so no gathered copy of the node features exists;
//   * accumulators are read back from TMEM by two threads per row (64 columns each), and the activations go back to TMEM as
//     the packed bf16 A operand of the next product (tcgen05.mma with A in tensor memory): hidden rows never use shared memory;
//   * the same two threads normalise the row (mean and squared deviations of each half, merged through two TMEM columns) and add `post`;
// * * rows pass through TMEM on their way to and from global memory, so that an access covers eight lines and not 32 rows (tmem_ld_rows):
//     with a row per thread the unit that handles lines was busy 4 000 cycles of a tile, and 10 000 where rows are kept.  Kept
//     activations go through the accumulator's columns that their thread has just read, before the next product overwrites them: the
//     A operand keeps the order of the columns, so that every product adds its terms in the order of the plain matrix products.
// * Three row tiles of 128 are in flight: one per group of eight epilogue warps, and a third accumulator takes the next tile's first
// product, so that neither its source rows nor its product are waited for (both took 13 000 of a tile's 26 000 cycles).
// The products are issued by two threads: an issue costs about 75 cycles, and the operands of one thread for all did not fit its registers.
// One thread per row (half the warps) was no option: at 168 registers a thread the compiler spilled.
#pragma once
#include "common.cuh"
#include "tmap.cuh"
#include "pnm_internal.h"

namespace pnm {

constexpr int kMlpW = 128;                       // width of every layer
constexpr int kMlpRows = 128;                    // rows of a tile
constexpr int kMlpChunk = kMlpRows * 128;        // 128 rows x 64 bf16
constexpr int kMlpProducers = 2;                 // warps that issue loads
constexpr int kMlpHelpers = kMlpProducers + 2;   // and two that issue products: one warpgroup
constexpr int kMlpThreads = 32 * (kMlpHelpers + 16);   // two groups of eight epilogue warps
constexpr int kMlpTmemCols = 512;                // three accumulators of 128 columns, a packed A operand of 64 per group

enum { MLP_SILU = 2, MLP_RELU = 3, MLP_GELU = 1 };   // same codes as the GEMM epilogues

struct MlpArgs {
  long long M;
  const int* idx[3];                             // row index of a source, or null: row m itself
  const __nv_bfloat16* src[3]; int ld_src[3];    // used where there is an index, whose values are rows of the table
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

// 16 bytes from global to shared memory, and groups of such copies (of one thread)
__device__ __forceinline__ void copy16_async(uint32_t smem_dst, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_dst), "l"(src) : "memory");
}
__device__ __forceinline__ void copy_group_end() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void copy_group_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }
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
// x[0..16) += 16 values in shared memory (the same for all lanes)
__device__ __forceinline__ void add_vec16(float* x, const float* v) {
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const float4 b = *reinterpret_cast<const float4*>(v + 4 * j);
    x[4 * j] += b.x; x[4 * j + 1] += b.y; x[4 * j + 2] += b.z; x[4 * j + 3] += b.w;
  }
}
// Registers of a warp (32 rows x 32 words: thread = row) <-> four vectors of 8 words a thread: thread t holds words [8 (t & 3), ..) of rows
// t / 4 + {0, 8, 16, 24}, so that an access to global memory covers eight whole lines and not 32 rows.  The turn goes through 32 columns
// of tensor memory: word 8 j + 2 g + e lies in column 8 g + 2 j + e, and shape 16x256b hands columns 8 g + 2 j + {0, 1} to thread j of four.
__device__ __forceinline__ void tmem_st32_turned(uint32_t taddr, const uint32_t* w) {
  float r[32];
#pragma unroll
  for (int i = 0; i < 32; ++i) r[i] = __uint_as_float(w[8 * ((i >> 1) & 3) + 2 * (i >> 3) + (i & 1)]);
  tmem_st32(taddr, r);
}
__device__ __forceinline__ void tmem_ld32_turned(uint32_t taddr, uint32_t* w) {
  float r[32];
  tmem_ld32(taddr, r);
  tmem_ld_wait();
#pragma unroll
  for (int i = 0; i < 32; ++i) w[8 * ((i >> 1) & 3) + 2 * (i >> 3) + (i & 1)] = __float_as_uint(r[i]);
}
// 16 rows from lane `taddr` on, 32 columns: a = row t / 4, b = row t / 4 + 8
__device__ __forceinline__ void tmem_ld_rows(uint32_t taddr, uint32_t* a, uint32_t* b) {
  asm volatile(
      "tcgen05.ld.sync.aligned.16x256b.x4.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
      : "=r"(a[0]), "=r"(a[1]), "=r"(b[0]), "=r"(b[1]), "=r"(a[2]), "=r"(a[3]), "=r"(b[2]), "=r"(b[3]), "=r"(a[4]), "=r"(a[5]), "=r"(b[4]),
        "=r"(b[5]), "=r"(a[6]), "=r"(a[7]), "=r"(b[6]), "=r"(b[7])
      : "r"(taddr)
      : "memory");
}
__device__ __forceinline__ void tmem_st_rows(uint32_t taddr, const uint32_t* a, const uint32_t* b) {
  asm volatile(
      "tcgen05.st.sync.aligned.16x256b.x4.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};" ::"r"(taddr),
      "r"(a[0]), "r"(a[1]), "r"(b[0]), "r"(b[1]), "r"(a[2]), "r"(a[3]), "r"(b[2]), "r"(b[3]), "r"(a[4]), "r"(a[5]), "r"(b[4]), "r"(b[5]),
      "r"(a[6]), "r"(a[7]), "r"(b[6]), "r"(b[7])
      : "memory");
}
// Registers of a warp -> the vectors of the turn, and those of the rows from row0 on -> global memory (row stride ld, in elements), rows
// past M left out
__device__ __forceinline__ void turn_rows(uint32_t taddr, const uint32_t* w, uint32_t (*v)[8]) {
  tmem_st32_turned(taddr, w);
  tmem_st_wait();
  tmem_ld_rows(taddr, v[0], v[1]);
  tmem_ld_rows(taddr + (16u << 16), v[2], v[3]);
  tmem_ld_wait();
}
__device__ __forceinline__ void store_turned(const uint32_t (*v)[8], __nv_bfloat16* dst, long long ld, long long row0, long long M, int lane) {
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const long long r = row0 + 8 * i + (lane >> 2);
    if (r < M) stg32(dst + r * ld + 16 * (lane & 3), v[i]);
  }
}
__device__ __forceinline__ void store_rows(uint32_t taddr, const uint32_t* w, __nv_bfloat16* dst, long long ld, long long row0, long long M,
                                           int lane) {
  uint32_t v[4][8];
  turn_rows(taddr, w, v);
  store_turned(v, dst, ld, row0, M, lane);
}
// 8 registers of bf16 pairs -> 32 lanes x 8 columns
__device__ __forceinline__ void tmem_st8(uint32_t taddr, const uint32_t* r) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]),
               "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7])
               : "memory");
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
// barrier of the two warps that share the rows of lane quarter q in a group
__device__ __forceinline__ void pair_sync(int grp, int q) { asm volatile("bar.sync %0, 64;" ::"r"(1 + 4 * grp + q) : "memory"); }
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

// The products of this kernel with K-major operands in 128-byte swizzle: of a descriptor only the low word (make_smem_desc) varies.
__device__ __forceinline__ uint32_t desc_lo(uint32_t saddr) { return ((saddr & 0x3ffff) >> 4) | (1u << 16); }
constexpr uint32_t kDescHi = (1024 >> 4) | (1u << 14) | (2u << 29);
__device__ __forceinline__ void umma_f16_k128(uint32_t d, uint32_t alo, uint32_t blo, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t.reg .b64 a, b;\n\t"
      "setp.ne.b32 p, %4, 0;\n\tmov.b64 a, {%1, %5};\n\tmov.b64 b, {%2, %5};\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], a, b, %3, p;\n\t}"
      ::"r"(d), "r"(alo), "r"(blo), "r"(idesc), "r"(accumulate), "n"(kDescHi)
      : "memory");
}
__device__ __forceinline__ void umma_f16_ts_k128(uint32_t d, uint32_t a_tmem, uint32_t blo, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t.reg .b64 b;\n\t"
      "setp.ne.b32 p, %4, 0;\n\tmov.b64 b, {%2, %5};\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], b, %3, p;\n\t}"
      ::"r"(d), "r"(a_tmem), "r"(blo), "r"(idesc), "r"(accumulate), "n"(kDescHi)
      : "memory");
}

template <int NSRC>
struct MlpCfg {
  static constexpr int WCHUNKS = 2 * NSRC + 4;                                    // 64-column blocks of W1 | W2 | W3
  static constexpr int STAGES = NSRC == 3 ? 2 : 3;                                // tiles of one source (two chunks)
  static constexpr int SMEM = (WCHUNKS + 2 * STAGES) * kMlpChunk + 512 + 5 * kMlpW * 4;   // three sources: all 227 KB
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
  float* vec = reinterpret_cast<float*>(ring + 2 * Cfg::STAGES * kMlpChunk);      // b1, b2, b3, gamma, beta
  uint64_t* full = reinterpret_cast<uint64_t*>(vec + 5 * kMlpW);
  uint64_t* empty = full + Cfg::STAGES;
  uint64_t* wfull = empty + Cfg::STAGES;
  uint64_t* first = wfull + 1;                   // [3] an accumulator holds a finished first product
  uint64_t* accfree = first + 3;                 // [3] its tile is finished
  uint64_t* accfull = accfree + 3;               // [2] the group's second or third product is finished
  uint64_t* aready = accfull + 2;                // [2] the accumulator was read, the packed A operand is in place
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(aready + 2);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int tiles = int((g.M + kMlpRows - 1) / kMlpRows);
  constexpr int KB = 2 * NSRC;
  constexpr int kStage = 2 * kMlpChunk;

  if (threadIdx.x == 0) {
    for (int s = 0; s < Cfg::STAGES; ++s) { mbar_init(&full[s], kMlpProducers); mbar_init(&empty[s], 1); }
    mbar_init(wfull, 1);
    for (int i = 0; i < 3; ++i) { mbar_init(&first[i], 1); mbar_init(&accfree[i], 8); }
    for (int i = 0; i < 2; ++i) { mbar_init(&accfull[i], 1); mbar_init(&aready[i], 8); }
    *abort_flag = 0;
    mbar_fence_init();
    if (smem_u32(smem_raw) & 1023) { atomicCAS(g.err, 0, ERR_BAD_ARG); *abort_flag = 1; }
  }
  for (int i = threadIdx.x; i < 5 * kMlpW; i += kMlpThreads) {
    const float* src = i < kMlpW ? g.b1 : i < 2 * kMlpW ? g.b2 : i < 3 * kMlpW ? g.b3 : i < 4 * kMlpW ? g.gamma : g.beta;
    vec[i] = src ? src[i & (kMlpW - 1)] : 0.f;
  }
  if (warp == 0) { tmem_alloc(tmem_slot, kMlpTmemCols); tmem_relinquish(); }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;
  // 640 threads are launched with 96 registers each: 128 x 64 + 512 x 104 is the same
  if (warp < kMlpHelpers) {                      // the first warpgroup
    asm volatile("setmaxnreg.dec.sync.aligned.u32 64;");
    if (warp < kMlpProducers) {
      // ---------------------------------------------------------------------------------------------- producers
      if (threadIdx.x == 0) {
        mbar_expect_tx(wfull, Cfg::WCHUNKS * kMlpChunk);
        for (int k = 0; k < KB; ++k) tma_load_2d(wts + k * kMlpChunk, &tmW1, wfull, k * 64, 0);
        for (int k = 0; k < 2; ++k) tma_load_2d(wts + (KB + k) * kMlpChunk, &tmW2, wfull, k * 64, 0);
        for (int k = 0; k < 2; ++k) tma_load_2d(wts + (KB + 2 + k) * kMlpChunk, &tmW3, wfull, k * 64, 0);
      }
      // Rows named by an index come by 16-byte copies, eight lanes to a row of 128 bytes, in the swizzle that a TMA tile would have: half
      // the rows of a tile per warp.  (TMA gathers of four rows take a warp 90 cycles each to issue, since their operands go through
      // uniform registers lane by lane: 128 of them to a tile were what the tile waited for.)  A stage is announced once its copies
      // have landed and are visible to the tensor cores' proxy: after the next one's copies are on their way, at once where the ring
      // is full.  Both warps announce every stage, also one that is a single TMA copy: a warp that could fall behind would meet the
      // phase of a stage two uses back.
      const uint32_t last = uint32_t(g.M) - 1, first_row = 64 * warp;
      const uint32_t my_row = first_row + (lane >> 3);       // of each set of four rows
      const uint32_t to[2] = {my_row * 128 + (((lane ^ my_row) & 7) << 4), my_row * 128 + (((lane ^ (my_row + 4)) & 7) << 4)};
      uint32_t slot = 0, phase = 1, told = 0, pending = 0;    // told: the oldest stage that is not announced
      int next[2] = {0, 0};                      // row numbers, read one source ahead: lane l has rows l and 32 + l of the warp's
      auto indices = [&](int tile, int j) {
        const int* ix = g.idx[j];
        if (ix && tile < tiles) {
#pragma unroll
          for (uint32_t q = 0; q < 2; ++q)       // rows past M repeat the last one: read, never stored
            next[q] = __ldg(ix + min(uint32_t(tile) * kMlpRows + first_row + 32 * q + lane, last));
        }
      };
      auto announce = [&]() {
        fence_async_smem();
        __syncwarp();
        if (lane == 0) mbar_arrive(&full[told]);
        if (++told == Cfg::STAGES) told = 0;
        --pending;
      };
      indices(blockIdx.x, 0);
      bool ok = true;
      for (int tile = blockIdx.x; ok && tile < tiles; tile += gridDim.x) {
#pragma unroll 1
        for (int j = 0; ok && j < NSRC; ++j) {
          const int r[2] = {next[0], next[1]};
          indices(j + 1 < NSRC ? tile : tile + int(gridDim.x), j + 1 < NSRC ? j + 1 : 0);
          if (!__all_sync(0xffffffffu, mbar_test(&empty[slot], phase))) {
            copy_group_wait<0>();
            while (pending) announce();
            ok = mbar_wait(&empty[slot], phase, abort_flag, g.err, ERR_WAIT_EMPTY);
            ok = __all_sync(0xffffffffu, ok);
            if (!ok) break;
          }
          uint8_t* dst = ring + slot * kStage;
          if (g.idx[j]) {
            const char* src = reinterpret_cast<const char*>(g.src[j]) + (lane & 7) * 16;
            const uint32_t dst0 = smem_u32(dst);
#pragma unroll
            for (int i = 0; i < 16; ++i) {
              const int row = __shfl_sync(0xffffffffu, r[i >> 3], (4 * i + (lane >> 3)) & 31);
              const char* from = src + (long long)row * (2 * g.ld_src[j]);
              copy16_async(dst0 + i * 512 + to[i & 1], from);
              copy16_async(dst0 + kMlpChunk + i * 512 + to[i & 1], from + 128);
            }
          } else if (threadIdx.x == 0) {
            const CUtensorMap* tm = j == 0 ? &tm0 : (j == 1 ? &tm1 : &tm2);
            mbar_expect_more(&full[slot], kStage);
            tma_load_2d(dst, tm, &full[slot], 0, tile * kMlpRows);
            tma_load_2d(dst + kMlpChunk, tm, &full[slot], 64, tile * kMlpRows);
          }
          copy_group_end();
          if (++pending == 2) {
            copy_group_wait<1>();
            announce();
          }
          if (++slot == Cfg::STAGES) { slot = 0; phase ^= 1; }
        }
      }
      copy_group_wait<0>();
      while (pending) announce();
      // tiles land before the CTA leaves; after a wait that ran out a stage that not both producers announced completes no phase
      if (!ok) abort_settle();
      else if (threadIdx.x == 0) {
        mbar_drain(wfull, 0);
        ring_drain(full, Cfg::STAGES, NSRC * (tiles > int(blockIdx.x) ? (tiles - int(blockIdx.x) - 1) / int(gridDim.x) + 1 : 0));
      }
    } else if (warp == kMlpProducers) {
      // ------------------------------------------------------------------------------------- first products, in order
      if (elect_one()) {
        constexpr uint32_t idesc = make_idesc_bf16(kMlpRows, kMlpW, false, false);
        const uint32_t wlo = desc_lo(smem_u32(wts)), rlo = desc_lo(smem_u32(ring));
        uint32_t slot = 0, phase = 0, a = 0, turn = 0;
        bool ok = mbar_wait(wfull, 0, abort_flag, g.err, ERR_WAIT_FULL);
        for (int tile = blockIdx.x; ok && tile < tiles; tile += gridDim.x) {
          if (turn) ok = mbar_wait(&accfree[a], (turn - 1) & 1, abort_flag, g.err, ERR_WAIT_TMEM_EMPTY);
#pragma unroll 1
          for (uint32_t j = 0; ok && j < NSRC; ++j) {
            ok = mbar_wait(&full[slot], phase, abort_flag, g.err, ERR_WAIT_FULL);
            if (!ok) break;
            tc_fence_after();
#pragma unroll
            for (uint32_t k = 0; k < 8; ++k) {
              const uint32_t at = (k >> 2) * (kMlpChunk >> 4) + 2 * (k & 3);
              umma_f16_k128(tmem + a * kMlpW, rlo + slot * (kStage >> 4) + at, wlo + j * (kStage >> 4) + at, idesc, j | k);
            }
            umma_commit(&empty[slot]);
            if (++slot == Cfg::STAGES) { slot = 0; phase ^= 1; }
          }
          if (!ok) break;
          umma_commit(&first[a]);
          if (++a == 3) { a = 0; ++turn; }
        }
      }
    } else {
      // ----------------------------------------------------- second and third products of both groups, as they become ready
      if (elect_one()) {
        constexpr uint32_t idesc = make_idesc_bf16(kMlpRows, kMlpW, false, false);
        int left = 2 * (tiles > int(blockIdx.x) ? (tiles - int(blockIdx.x) - 1) / int(gridDim.x) + 1 : 0);
        uint32_t arrivals[2] = {0, 0};           // phases of aready[grp] consumed so far: two per tile
        uint32_t acc[2] = {tmem, tmem + kMlpW};  // of the group's tile
        const uint32_t wlo = desc_lo(smem_u32(wts + KB * kMlpChunk));
        unsigned long long t0 = 0;
        uint32_t spins = 0;
        bool ok = mbar_wait(wfull, 0, abort_flag, g.err, ERR_WAIT_FULL);
        while (ok && left) {
          bool any = false;
#pragma unroll
          for (int grp = 0; grp < 2; ++grp) {
            if (!mbar_test(&aready[grp], arrivals[grp] & 1)) continue;
            const uint32_t layer = arrivals[grp] & 1;        // 0: second product, 1: third
            ++arrivals[grp];
            tc_fence_after();
            const uint32_t aop = tmem + 3 * kMlpW + grp * 64;
#pragma unroll
            for (uint32_t k = 0; k < 8; ++k)
              umma_f16_ts_k128(acc[grp], aop + 8 * k, wlo + (2 * layer + (k >> 2)) * (kMlpChunk >> 4) + 2 * (k & 3), idesc, k);
            umma_commit(&accfull[grp]);
            if (layer) acc[grp] = acc[grp] == tmem ? tmem + 2 * kMlpW : acc[grp] - kMlpW;   // two tiles on, modulo three
            --left;
            any = true;
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
    }
  } else {
    asm volatile("setmaxnreg.inc.sync.aligned.u32 104;");
    // ----------------------------------------------------- epilogue: two threads per row, columns [64 half, 64 half + 64)
    const int grp = (warp - kMlpHelpers) >> 3, half = ((warp - kMlpHelpers) >> 2) & 1, q = warp & 3, col = half * 64;
    const uint32_t base = tmem + (uint32_t(q * 32) << 16);
    // the moments of a half row lie in its own part of the A operand, whose last reader is the third product
    const uint32_t aop = base + 3 * kMlpW + grp * 64 + half * 32, other_aop = base + 3 * kMlpW + grp * 64 + (half ^ 1) * 32;
    // A group meets accumulator `a` every other turn, always with the parity of `turn`: a wait for turn t + 2 would be over at once if
    // turn t + 1 (the other group's tile n + 3) were not.  It is: one thread issues and commits the first products in the order of the
    // tiles, so that of tile n + 3 has finished before that of n + 4, which this group has waited for before it comes to n + 6.
    uint32_t n = 0, uses = 0, a = 0, turn = 0;   // n = 3 turn + a
    for (int tile = blockIdx.x; tile < tiles; tile += gridDim.x, ++n, turn += a == 2, a = a == 2 ? 0 : a + 1) {
      if ((n & 1) != uint32_t(grp)) continue;
      const uint32_t acc = base + a * kMlpW + col;
      const long long row0 = (long long)tile * kMlpRows + q * 32, row = row0 + lane;
      const bool live = row < g.M;
      bool ok = true;
#pragma unroll 1
      for (int layer = 0; layer < 2; ++layer) {
        const float* bias = vec + layer * kMlpW + col;
        __nv_bfloat16* z = (layer ? g.z2 : g.z1) + z_offset(tile, q, half, lane);
        __nv_bfloat16* h = (layer ? g.h2 : g.h1) + col;
        ok = mbar_wait(layer ? &accfull[grp] : &first[a], (layer ? uses : turn) & 1, abort_flag, g.err, ERR_WAIT_TMEM_FULL);
        if (!__all_sync(0xffffffffu, ok)) { ok = false; break; }
        uses += layer;
        tc_fence_after();
        uint32_t act[32];
        float v[2][16];                          // two steps of 16 columns: one is read from TMEM while the other is worked on
        tmem_ld16(acc, v[0]);
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          tmem_ld_wait();
          if (c < 3) tmem_ld16(acc + (c + 1) * 16, v[(c + 1) & 1]);
          float* x = v[c & 1];
          add_vec16(x, bias + c * 16);
          if (SAVE && ACT != MLP_RELU) {
            uint32_t p[8];
#pragma unroll
            for (int j = 0; j < 8; ++j) p[j] = pack_bf16x2(x[2 * j], x[2 * j + 1]);
            stg32(z + c * kZStep, p);            // rows past M too: the buffer holds whole tiles
          }
#pragma unroll
          for (int j = 0; j < 8; ++j) act[8 * c + j] = pack_bf16x2(mlp_act<ACT>(x[2 * j]), mlp_act<ACT>(x[2 * j + 1]));
          tmem_st8(aop + 8 * c, act + 8 * c);
        }
        // The weight gradient's operand is this product's: recomputed from the rounded pre-activation it would be rounded twice (dW2
        // against 64 bits 0.0054 instead of 0.0049).  Stored while the product runs.
        uint32_t rows[4][8];
        if (SAVE) turn_rows(acc, act, rows);
        else tmem_st_wait();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&aready[grp]);
        if (SAVE) store_turned(rows, h, kMlpW, row0, g.M, lane);
      }
      Vec32 res[4] = {};
      auto load_post = [&]() {
        if (!g.post) return;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const long long r = row0 + 8 * i + (lane >> 2);
          if (r < g.M) res[i] = ldg32(g.post + r * g.ld_post + col + 16 * (lane & 3));
        }
      };
      if (!SAVE) load_post();                    // on their way while the third product runs (with what is kept: no registers left)
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
        uint32_t kept[SAVE ? 32 : 1];
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
#pragma unroll
            for (int j = 0; j < 8; ++j) {
              kept[8 * c + j] = pack_bf16x2(x[2 * j], x[2 * j + 1]);
              const float2 k = unpack_bf16x2(kept[8 * c + j]);
              const float d0 = k.x - pivot, d1 = k.y - pivot;
              sum_k += d0 + d1;
              sq_k = fmaf(d0, d0, fmaf(d1, d1, sq_k));
            }
          }
#pragma unroll
          for (int j = 0; j < 16; ++j) { const float d = x[j] - pivot; sum += d; sq += d * d; }
        }
        if (SAVE) store_rows(aop, kept, g.x3 + col, kMlpW, row0, g.M, lane);
      }
      if (SAVE) load_post();
      const float shift = sum * (1.f / 64), mean_h = pivot + shift, dev_h = fmaxf(sq - sum * shift, 0.f);
      const float shift_k = sum_k * (1.f / 64), mean_k = pivot + shift_k, dev_k = fmaxf(sq_k - sum_k * shift_k, 0.f);
      if (ok) {
        tmem_st2(aop, mean_h, dev_h);
        if (SAVE) tmem_st2(aop + 2, mean_k, dev_k);
        tmem_st_wait();
      }
      tc_fence_before();
      __syncwarp();
      pair_sync(grp, q);
      tc_fence_after();
      const bool whole = __all_sync(0xffffffffu, ok && !*abort_flag);
      // the halves' moments: mean = (a + b) / 2, squared deviations add up with 64 * 64 / 128 times the squared difference
      const float2 other = tmem_ld2(other_aop);
      const float mean = 0.5f * (mean_h + other.x), gap = mean_h - other.x;
      const float rstd = rsqrtf((dev_h + other.y + 32.f * gap * gap) * (1.f / kMlpW) + g.eps);
      if (SAVE) {
        const float2 other_k = tmem_ld2(other_aop + 2);
        const float gap_k = mean_k - other_k.x;
        if (whole && live && half == 0) {
          g.mean[row] = 0.5f * (mean_k + other_k.x);
          g.rstd[row] = rsqrtf((dev_k + other_k.y + 32.f * gap_k * gap_k) * (1.f / kMlpW) + g.eps);
        }
      }
      tc_fence_before();
      pair_sync(grp, q);                         // both have read: the columns of the moments may be overwritten
      tc_fence_after();
      if (!whole) continue;                      // no warp leaves the loop early: a pair's barriers need both
      uint32_t out[32];
      if (g.post) {                              // zeros without a residual
        tmem_st_rows(aop, res[0].w, res[1].w);
        tmem_st_rows(aop + (16u << 16), res[2].w, res[3].w);
        tmem_st_wait();
        tmem_ld32_turned(aop, out);
      } else {
#pragma unroll
        for (int i = 0; i < 32; ++i) out[i] = 0;
      }
      float v[2][16];
      tmem_ld16(acc, v[0]);
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        tmem_ld_wait();
        if (c < 3) tmem_ld16(acc + (c + 1) * 16, v[(c + 1) & 1]);
        else {                                   // the accumulator may be overwritten
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(&accfree[a]);
        }
        const float* x = v[c & 1];
        uint32_t* p = out + 8 * c;
        const float4* vb = reinterpret_cast<const float4*>(vec + 2 * kMlpW + col + c * 16);    // b3; gamma and beta follow
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const float4 b = vb[j], ga = vb[j + kMlpW / 4], be = vb[j + kMlpW / 2];
          const float2 r0 = unpack_bf16x2(p[2 * j]), r1 = unpack_bf16x2(p[2 * j + 1]);
          const float h0 = (x[4 * j] + b.x - mean) * rstd, h1 = (x[4 * j + 1] + b.y - mean) * rstd, h2 = (x[4 * j + 2] + b.z - mean) * rstd,
                      h3 = (x[4 * j + 3] + b.w - mean) * rstd;
          p[2 * j] = pack_bf16x2(fmaf(h0, ga.x, be.x) + r0.x, fmaf(h1, ga.y, be.y) + r0.y);
          p[2 * j + 1] = pack_bf16x2(fmaf(h2, ga.z, be.z) + r1.x, fmaf(h3, ga.w, be.w) + r1.y);
        }
      }
      store_rows(aop, out, g.y + col, g.ld_y, row0, g.M, lane);
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 0) {
    if (*abort_flag) abort_settle();
    tc_fence_after();
    tmem_dealloc(tmem, kMlpTmemCols);
  }
}

}  // namespace pnm

// Backward of the fused three-layer perceptron (mlp_fused.cuh) from the gradient of its last linear layer down to the first
// pre-activation, in one kernel:
//
//   g2 = (dx3 W3) * act'(z2)      dW3 += dx3^T act(z2), db3 += dx3
//   g1 = (g2 W2) * act'(z1)       dW2 += g2^T act(z1),  db2 += g2
//
// Layer by layer these are two data-gradient and two weight-gradient products that move ten 256-byte rows per row of M; here
// a row tile is read once (dx3, z2, act(z2), z1, act(z1)) and only g1 is written: six rows (1.7 M rows: 0.47 ms, the rows are
// worth 0.39 ms; with the activations recomputed from z in the same threads 0.62 ms).  (The LayerNorm backward before it stays a
// kernel of its own: its column sums are free when a warp works along a row, but cost eight instructions per element when, as
// here, a thread owns a row; with it inside, this kernel was bound by instruction issue at 1.41 ms for 1.5 M rows.)
// dx3 and act(z2) arrive by TMA; g2 overwrites dx3 and act(z1) takes the place of act(z2).  A gradient tile lies in shared memory
// once, in the 128-byte-swizzled layout that tcgen05 reads both ways: as the K-major A operand of the data gradient and, with the
// row index as the reduction, as the MN-major A operand of the weight gradient.  (The activations are the forward's own operands:
// recomputed from the rounded z they would be rounded twice.)  Both weight gradients accumulate in TMEM over all tiles of a
// persistent CTA and are added to memory once at its end.
// Two tiles are in flight, one per group of eight warps (two threads per row); ONE thread issues all products, since products
// that accumulate into the same TMEM columns are only ordered within a thread.  A further warp per group sums the columns
// of the gradient tile while the tensor cores read it.
#pragma once
#include "mlp_fused.cuh"

namespace pnm {

struct MlpBwdArgs {
  long long M;
  const __nv_bfloat16 *z2, *z1;                  // whole tiles (z_offset); ReLU: the activations, contiguous [M, 128]
  __nv_bfloat16* g1;                             // [M, 128]
  float *dW3, *dW2, *db3, *db2;                  // added to
  int* err;
};

constexpr int kMlpBwdThreads = 640;              // issuer, 2 warps of column sums, producer, 2 x 8 warps of the tiles
constexpr int kMlpBwdSmem = 12 * kMlpChunk + 256;

// v act'(z); ReLU selects, so that an infinite v beside a negative z is 0 and not NaN
template <int ACT>
__device__ __forceinline__ float mlp_dact(float v, float z) {
  return ACT == MLP_SILU ? v * silu_grad_f(z) : ACT == MLP_GELU ? v * gelu_grad_f(z) : (z > 0.f ? v : 0.f);
}
// 16 packed columns [16 c, 16 c + 16) of tile row r -> the swizzled tile of two 64-column chunks
__device__ __forceinline__ void tile_put16(uint8_t* tile, int r, int c, const uint32_t* p) {
  uint8_t* row = tile + (c >> 2) * kMlpChunk + r * 128;
  const int u = (2 * c) & 7;
  *reinterpret_cast<uint4*>(row + ((u ^ (r & 7)) << 4)) = make_uint4(p[0], p[1], p[2], p[3]);
  *reinterpret_cast<uint4*>(row + (((u + 1) ^ (r & 7)) << 4)) = make_uint4(p[4], p[5], p[6], p[7]);
}

template <int ACT>
__global__ void __launch_bounds__(kMlpBwdThreads, 1)
mlp3_bwd_kernel(const __grid_constant__ CUtensorMap tmD, const __grid_constant__ CUtensorMap tmH2, const __grid_constant__ CUtensorMap tmH1,
                const __grid_constant__ CUtensorMap tmW3t, const __grid_constant__ CUtensorMap tmW2t, const MlpBwdArgs g) {
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  uint8_t* wts = smem_raw;
  uint8_t* tiles_smem = wts + 4 * kMlpChunk;     // per group: gradient tile (2 chunks), activation tile (2 chunks)
  uint64_t* wfull = reinterpret_cast<uint64_t*>(tiles_smem + 8 * kMlpChunk);
  uint64_t* dfull = wfull + 1;                   // [2] dx3 and act(z2) of a tile have arrived
  uint64_t* hfull = dfull + 2;                   // [2] act(z1) has arrived
  uint64_t* dfree = hfull + 2;                   // [2] both tiles were read for the last time
  uint64_t* ready = dfree + 2;                   // [2] the accumulator was read (second phase: and g2 is written)
  uint64_t* done = ready + 2;                    // [2] the phase's products and column sums are finished
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(done + 2);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int tiles = int((g.M + kMlpRows - 1) / kMlpRows);
  const int mine = tiles > int(blockIdx.x) ? (tiles - int(blockIdx.x) - 1) / int(gridDim.x) + 1 : 0;   // tiles of this CTA

  if (threadIdx.x == 0) {
    mbar_init(wfull, 1);
    for (int i = 0; i < 2; ++i) {
      mbar_init(&dfull[i], 1); mbar_init(&hfull[i], 1); mbar_init(&dfree[i], 2); mbar_init(&ready[i], 8); mbar_init(&done[i], 2);
    }
    *abort_flag = 0;
    mbar_fence_init();
    if (smem_u32(smem_raw) & 1023) { atomicCAS(g.err, 0, ERR_BAD_ARG); *abort_flag = 1; }
  }
  if (warp == 0) { tmem_alloc(tmem_slot, kMlpTmemCols); tmem_relinquish(); }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;              // accumulators of the groups at 0 and 128, dW3 at 256, dW2 at 384

  if (warp == 0) {
    if (elect_one()) {
      mbar_expect_tx(wfull, 4 * kMlpChunk);
      for (int k = 0; k < 2; ++k) tma_load_2d(wts + k * kMlpChunk, &tmW3t, wfull, k * 64, 0);
      for (int k = 0; k < 2; ++k) tma_load_2d(wts + (2 + k) * kMlpChunk, &tmW2t, wfull, k * 64, 0);
      constexpr uint32_t idesc = make_idesc_bf16(kMlpRows, kMlpW, false, false);
      constexpr uint32_t idesc_t = make_idesc_bf16(kMlpW, kMlpW, true, true);
      bool ok = mbar_wait(wfull, 0, abort_flag, g.err, ERR_WAIT_FULL);
      // phases of a group: two per tile; whichever group is ready first goes first
      int left[2] = {2 * ((mine + 1) / 2), 2 * (mine / 2)}, at[2] = {0, 0};
      uint32_t started = 0;                      // bit l: the weight gradient of phase l holds a value
      unsigned long long t0 = 0;
      uint32_t spins = 0;
      while (ok && (left[0] || left[1])) {
        bool any = false;
#pragma unroll
        for (int grp = 0; grp < 2; ++grp) {
          const int layer = at[grp] & 1;
          if (!left[grp] || !mbar_test(&ready[grp], layer)) continue;
          if (!mbar_test(layer ? &hfull[grp] : &dfull[grp], (at[grp] >> 1) & 1)) continue;
          any = true;
          tc_fence_after();
          const uint32_t xs = smem_u32(tiles_smem + grp * 4 * kMlpChunk), ws = smem_u32(wts + layer * 2 * kMlpChunk);
          const uint32_t acc = tmem + grp * 128, dw = tmem + 256 + layer * 128;
#pragma unroll
          for (int k = 0; k < 8; ++k)
            umma_f16(acc, make_smem_desc(xs + (k >> 2) * kMlpChunk, 16, 1024, 2) + 2 * (k & 3),
                     make_smem_desc(ws + (k >> 2) * kMlpChunk, 16, 1024, 2) + 2 * (k & 3), idesc, k != 0 ? 1u : 0u);
          const uint64_t gd = make_smem_desc(xs, kMlpChunk, 1024, 2), hd = make_smem_desc(xs + 2 * kMlpChunk, kMlpChunk, 1024, 2);
#pragma unroll
          for (int k = 0; k < 8; ++k)            // 16 rows of the tile = 2048 bytes per step
            umma_f16(dw, gd + 128 * k, hd + 128 * k, idesc_t, (((started >> layer) & 1) || k != 0) ? 1u : 0u);
          started |= 1u << layer;
          umma_commit(&done[grp]);
          if (layer == 1) umma_commit(&dfree[grp]);
          ++at[grp];
          --left[grp];
        }
        if (any) { spins = 0; t0 = 0; }
        else if ((++spins & 0x3ffu) == 0) {
          if (*abort_flag) break;
          const unsigned long long now = globaltimer_ns();
          if (t0 == 0) t0 = now;
          else if (now - t0 > kWaitBudgetNs) {
            atomicCAS(g.err, 0, ERR_WAIT_FULL);
            *abort_flag = 1;
            __threadfence_block();
            break;
          }
        }
      }
    }
  } else if (warp <= 2) {
    // ------------------------------- column sums of group warp - 1: lane l owns four columns; between them the load of act(z1)
    const int grp = warp - 1;
    const uint8_t* x = tiles_smem + grp * 4 * kMlpChunk + (lane >> 4) * kMlpChunk;
    const int u = (lane & 15) >> 1, low = (lane & 1) * 8;
    float s[2][4] = {};
    uint32_t issued = 0;
    const int phases = 2 * (grp == 0 ? (mine + 1) / 2 : mine / 2);
    uint8_t* ht = tiles_smem + (grp * 4 + 2) * kMlpChunk;
    for (int ph = 0; ph < phases; ++ph) {
      const bool second = ph & 1;
      // first phase: dx3 from TMA; second: g2 from the group's warps
      bool ok = second ? mbar_wait(&ready[grp], 1, abort_flag, g.err, ERR_WAIT_AUX)
                       : mbar_wait(&dfull[grp], (ph >> 1) & 1, abort_flag, g.err, ERR_WAIT_AUX);
      if (!__all_sync(0xffffffffu, ok)) break;
      float t[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll 16
      for (int r = 0; r < kMlpRows; ++r) {
        const uint2 v = *reinterpret_cast<const uint2*>(x + r * 128 + ((u ^ (r & 7)) << 4) + low);
        const float2 a = unpack_bf16x2(v.x), b = unpack_bf16x2(v.y);
        t[0] += a.x; t[1] += a.y; t[2] += b.x; t[3] += b.y;
      }
      __syncwarp();
      if (lane == 0) {
        mbar_arrive(&done[grp]);
        if (second) mbar_arrive(&dfree[grp]);
      }
      // Every phase of `done` is awaited here; each needs this warp's own arrival, so none is missed.  `ready` has completed its phase of
      // the same number by then and cannot complete the one after the next without `done`: no wait here can meet a phase of the same
      // parity two further on, however slow this warp is.
      ok = mbar_wait(&done[grp], ph & 1, abort_flag, g.err, ERR_WAIT_AUX);
      if (!__all_sync(0xffffffffu, ok)) break;
      if (!second && lane == 0) {                // act(z2) was read by the first phase's products: act(z1) takes its place
        const int m0 = (int(blockIdx.x) + (ph + grp) * int(gridDim.x)) * kMlpRows;      // tile ph / 2 of the group
        mbar_expect_tx(&hfull[grp], 2 * kMlpChunk);
        tma_load_2d(ht, &tmH1, &hfull[grp], 0, m0);
        tma_load_2d(ht + kMlpChunk, &tmH1, &hfull[grp], 64, m0);
        ++issued;
      }
#pragma unroll
      for (int i = 0; i < 4; ++i) { s[0][i] += second ? 0.f : t[i]; s[1][i] += second ? t[i] : 0.f; }
    }
    if (issued) mbar_drain(&hfull[grp], (issued - 1) & 1);
    const int col = (lane >> 4) * 64 + u * 8 + (lane & 1) * 4;
    if (phases)
#pragma unroll
      for (int i = 0; i < 4; ++i) { atomicAdd(g.db3 + col + i, s[0][i]); atomicAdd(g.db2 + col + i, s[1][i]); }
  } else if (warp == 3) {
    // --------------------------------------------------------------------------------------- dx3 and act(z2) tiles
    if (elect_one()) {
      uint32_t issued[2] = {0, 0};
#pragma unroll 1
      for (int n = 0; n < mine; ++n) {
        const int grp = n & 1, k = n >> 1;       // k-th tile of the group
        if (k && !mbar_wait(&dfree[grp], (k - 1) & 1, abort_flag, g.err, ERR_WAIT_EMPTY)) break;
        uint8_t* dst = tiles_smem + grp * 4 * kMlpChunk;
        const int m0 = (int(blockIdx.x) + n * int(gridDim.x)) * kMlpRows;
        mbar_expect_tx(&dfull[grp], 4 * kMlpChunk);
        for (int c = 0; c < 2; ++c) {
          tma_load_2d(dst + c * kMlpChunk, &tmD, &dfull[grp], 64 * c, m0);
          tma_load_2d(dst + (2 + c) * kMlpChunk, &tmH2, &dfull[grp], 64 * c, m0);
        }
        ++issued[grp];
      }
      for (int grp = 0; grp < 2; ++grp)          // copies land before the CTA leaves, also after a wait that ran out
        if (issued[grp]) mbar_drain(&dfull[grp], (issued[grp] - 1) & 1);
    }
  } else {
    // ------------------------------------------------- two threads per row of a tile, columns [64 half, 64 half + 64)
    const int grp = (warp - 4) >> 3, half = ((warp - 4) >> 2) & 1, q = warp & 3, r = q * 32 + lane, col = half * 64;
    const uint32_t lanes = uint32_t(q * 32) << 16;
    const uint32_t acc = tmem + grp * 128 + lanes + col;
    uint8_t* gt = tiles_smem + grp * 4 * kMlpChunk;
    uint32_t phase = 0;
    bool ok = true;
    constexpr int step = ACT == MLP_RELU ? 16 : kZStep;
    auto offset = [&](int n) {                   // rows past M: their dx3 is zero and their g1 not stored
      const long long tile = (long long)blockIdx.x + (long long)n * gridDim.x, row = tile * kMlpRows + r;
      return ACT == MLP_RELU ? (row < g.M ? row : g.M - 1) * kMlpW + col : z_offset(tile, q, half, lane);
    };
    Vec32 z[4];
    if (grp < mine) {
#pragma unroll
      for (int c = 0; c < 4; ++c) z[c] = ldg32(g.z2 + offset(grp) + c * step);
    }
    for (int n = grp; n < mine; n += 2) {
      const long long o = offset(n);
      tc_fence_before();                         // the accumulator was read: the last tile's g1 is on its way
      __syncwarp();
      if (lane == 0) mbar_arrive(&ready[grp]);
      // ---- g2 = (dx3 W3) act'(z2); each vector of z1 is requested where one of z2 is used up
      ok = mbar_wait(&done[grp], phase & 1, abort_flag, g.err, ERR_WAIT_TMEM_FULL) && ok;
      ++phase;
      tc_fence_after();
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        float v[16];
        tmem_ld16(acc + c * 16, v);
        tmem_ld_wait();
        uint32_t p[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          const float2 zv = unpack_bf16x2(z[c].w[j]);
          p[j] = pack_bf16x2(mlp_dact<ACT>(v[2 * j], zv.x), mlp_dact<ACT>(v[2 * j + 1], zv.y));
        }
        tile_put16(gt, r, half * 4 + c, p);
        z[c] = ldg32(g.z1 + o + c * step);
      }
      fence_async_smem();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&ready[grp]);
      // ---- g1 = (g2 W2) act'(z1); the next tile's z2 takes the place of z1
      const long long on = offset(n + 2 < mine ? n + 2 : n);
      ok = mbar_wait(&done[grp], phase & 1, abort_flag, g.err, ERR_WAIT_TMEM_FULL) && ok;
      ++phase;
      tc_fence_after();
      uint32_t out[32];
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        float v[16];
        tmem_ld16(acc + c * 16, v);
        tmem_ld_wait();
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          const float2 zv = unpack_bf16x2(z[c].w[j]);
          out[8 * c + j] = pack_bf16x2(mlp_dact<ACT>(v[2 * j], zv.x), mlp_dact<ACT>(v[2 * j + 1], zv.y));
        }
        z[c] = ldg32(g.z2 + on + c * step);
      }
      // through the columns of the accumulator that this thread has just read: eight lines an access instead of 32 rows
      store_rows(acc, out, g.g1 + col, kMlpW, ((long long)blockIdx.x + (long long)n * gridDim.x) * kMlpRows + q * 32, g.M, lane);
    }
    // A wait that ran out leaves wrong values behind (the error word says so); the loop ends all the same, since every later
    // wait gives up at once.  Otherwise every product of the CTA has been waited for by the warps that used its result, so the
    // weight gradients are complete.
    tc_fence_before();
    __syncwarp();
    asm volatile("bar.sync 3, 512;" ::: "memory");
    tc_fence_after();
    if (__all_sync(0xffffffffu, ok && !*abort_flag)) {
      float* dst = (grp ? g.dW2 : g.dW3) + r * kMlpW + col;
      const uint32_t src = tmem + 256 + grp * 128 + lanes + col;
#pragma unroll 1
      for (int c = 0; c < 2; ++c) {
        float v[32];
        tmem_ld32(src + c * 32, v);
        tmem_ld_wait();
#pragma unroll
        for (int j = 0; j < 8; ++j)
          asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(dst + c * 32 + 4 * j), "f"(v[4 * j]), "f"(v[4 * j + 1]),
                       "f"(v[4 * j + 2]), "f"(v[4 * j + 3])
                       : "memory");
      }
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

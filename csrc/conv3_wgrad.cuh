// Weight gradient of a 3 x 3 "same" convolution, channels-last bf16: dW[co, tap, ci] += sum over pixels p of dY[p, co] X[p + tap, ci]
// (fp32), optionally db[co] += sum of dY[p, co].  The reduction GEMM of gemm_nt.cuh in convolution mode brings one shifted box of X per
// tap and a box of dY for every 256 columns, 96 to 128 bytes from L2 for each cycle of its products; L2 delivers about 40 to an SM.
// Here a tile of the output is one COLUMN of taps (kx; ky = 0, 1, 2) x 128 input channels x 128 output channels:
//   * a reduction block is a patch of 4 x 16 pixels.  The windows of X of the three taps differ by whole rows of 16 pixels = 2048 bytes,
//     so one box of 6 x 16 pixels holds all of them, and one MN-major descriptor of N = 192 columns with 2048 bytes between
//     its groups of 64 columns reads the three taps of 64 channels at once;
//   * a box of dY serves all 384 columns of the tile, which accumulate in TMEM over the CTA's share of the patches.
// 40 KB per 64 pixels and 768 cycles of products: 52 bytes a cycle.  One image 512 x 512, 128 -> 128 / 256 -> 128 channels: 63 / 111 us
// (1.22 / 1.40 PFLOP/s; by the reduction GEMM 156 / 223 us), 2 x 128 x 128, 512 -> 512: 109 us (pair tiles of the reduction GEMM 170).
// Patches of 8 x 16 pixels (47 bytes a cycle, three stages instead of five): the same to 2 %.
#pragma once
#include "gemm_nt.cuh"

namespace pnm {

constexpr int kWg3Threads = 320;            // warp 0 producer, warp 1 products, warps 2 .. 9 epilogue
constexpr int kWg3Row = 272;                // bytes between the rows of 64 sums that an epilogue warp hands to the copy engine

struct Wg3Cfg {
  static constexpr int TH = kWgTileH, ROWS = TH * kWgTileW;        // pixels of a reduction block
  static constexpr int A_BOX = ROWS * 128, B_BOX = (TH + 2) * kWgTileW * 128;      // 64 channels of dY / of X
  static constexpr int STAGE_BYTES = 2 * A_BOX + 2 * B_BOX;
  static constexpr int STAGES = 5;
  static constexpr int ONES_BYTES = 2048;
  static constexpr int SMEM = 1024 + STAGES * STAGE_BYTES + ONES_BYTES + 256;
  static_assert(SMEM <= 232448, "shared memory budget");
};

struct Wg3Args {
  int cout, cin, tiles_x, tiles_y, patches, per_split;
  int tiles_a, tiles_c;                    // blocks of 128 output / input channels
  float* out; float* colsum;               // [cout, 9 cin], [cout] or null; added to
  int* err;
};

__global__ void __launch_bounds__(kWg3Threads, 1)
conv3_wgrad_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB, const Wg3Args g) {
  using Cfg = Wg3Cfg;
  constexpr int STAGES = Cfg::STAGES, TH = Cfg::TH;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* base = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* ones = base + STAGES * Cfg::STAGE_BYTES;
  uint64_t* full = reinterpret_cast<uint64_t*>(ones + Cfg::ONES_BYTES);
  uint64_t* empty = full + STAGES;
  uint64_t* tfull = empty + STAGES;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(tfull + 1);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int tiles = g.tiles_a * g.tiles_c * 3;
  const int tile = blockIdx.x % tiles, split = blockIdx.x / tiles;
  const int kx = tile % 3, tc = (tile / 3) % g.tiles_c, ta = tile / 3 / g.tiles_c;
  const int boxes = g.cin - tc * 128 >= 128 ? 2 : 1;               // of 64 input channels
  const int p_begin = split * g.per_split, p_end = min(p_begin + g.per_split, g.patches);
  const int num_kb = p_end > p_begin ? p_end - p_begin : 0;
  const bool sums = g.colsum && kx == 0 && tc == 0;

  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) { mbar_init(&full[s], 1); mbar_init(&empty[s], 1); }
    mbar_init(tfull, 1);
    *abort_flag = 0;
    mbar_fence_init();
    tma_prefetch_desc(&tmA); tma_prefetch_desc(&tmB);
  }
  for (int i = threadIdx.x; i < Cfg::ONES_BYTES / 4; i += kWg3Threads) reinterpret_cast<uint32_t*>(ones)[i] = 0x3f803f80u;
  fence_async_smem();
  if (warp == 1) { tmem_alloc(tmem_slot, 512); tmem_relinquish(); }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;                           // 2 x 192 columns of dW, then 16 of db

  if (warp == 0) {
    if (elect_one()) {
      int kb = 0;
      for (; kb < num_kb; ++kb) {
        const int s = kb % STAGES;
        if (!mbar_wait(&empty[s], ((kb / STAGES) & 1) ^ 1, abort_flag, g.err, ERR_WAIT_EMPTY)) break;
        uint8_t* sa = base + s * Cfg::STAGE_BYTES;
        const int patch = p_begin + kb, per_img = g.tiles_x * g.tiles_y;
        const int n = patch / per_img, r = patch - n * per_img;
        const int y0 = (r / g.tiles_x) * TH, x0 = (r % g.tiles_x) * kWgTileW;
        mbar_expect_tx(&full[s], 2 * Cfg::A_BOX + boxes * Cfg::B_BOX);
        for (int i = 0; i < 2; ++i) tma_load_4d(sa + i * Cfg::A_BOX, &tmA, &full[s], ta * 128 + i * 64, x0, y0, n);
        for (int i = 0; i < boxes; ++i)
          tma_load_4d(sa + 2 * Cfg::A_BOX + i * Cfg::B_BOX, &tmB, &full[s], tc * 128 + i * 64, x0 + kx - 1, y0 - 1, n);
      }
      ring_drain(full, STAGES, kb);
    }
  } else if (warp == 1) {
    if (elect_one()) {
      constexpr uint32_t idesc = make_idesc_bf16(128, 192, true, true);
      constexpr uint32_t idesc1 = make_idesc_bf16(128, 16, true, false);
      const uint64_t od = make_smem_desc(smem_u32(ones), 128, 256, 0);     // K-major, unswizzled: every element is 1.0
      bool ok = true;
      for (int kb = 0; kb < num_kb; ++kb) {
        const int s = kb % STAGES;
        if (!mbar_wait(&full[s], (kb / STAGES) & 1, abort_flag, g.err, ERR_WAIT_FULL)) { ok = false; break; }
        tc_fence_after();
        const uint32_t sa = smem_u32(base + s * Cfg::STAGE_BYTES), sb = sa + 2 * Cfg::A_BOX;
        const uint64_t ad = make_smem_desc(sa, Cfg::A_BOX, 1024, 2);
        const uint64_t bd0 = make_smem_desc(sb, 2048, 1024, 2), bd1 = make_smem_desc(sb + Cfg::B_BOX, 2048, 1024, 2);
#pragma unroll
        for (int k = 0; k < TH; ++k) {                             // a row of 16 pixels = 128 sixteen-byte units
          umma_f16(tmem_base, ad + 128 * k, bd0 + 128 * k, idesc, (kb | k) != 0 ? 1u : 0u);
          if (boxes == 2) umma_f16(tmem_base + 192, ad + 128 * k, bd1 + 128 * k, idesc, (kb | k) != 0 ? 1u : 0u);
          if (sums) umma_f16(tmem_base + 384, ad + 128 * k, od, idesc1, (kb | k) != 0 ? 1u : 0u);
        }
        umma_commit(&empty[s]);
      }
      if (ok) umma_commit(tfull);
    }
  } else if (num_kb > 0) {
    // Two warps per lane quarter, every second tap each; a lane's 64 sums leave as one bulk reduction of 256 bytes from the shared
    // memory of the finished stages (a warp's red instructions touch 32 rows each: 16 bytes of a sector at a time).
    const int q = warp & 3, half = (warp - 2) >> 2;
    if (mbar_wait_warp(tfull, 0, abort_flag, g.err, ERR_WAIT_TMEM_FULL)) {
      tc_fence_after();
      const int row = ta * 128 + q * 32 + lane;                    // output channel
      const uint32_t lanes = tmem_base + (uint32_t(q * 32) << 16);
      uint8_t* rows = base + (warp - 2) * (2 * 32 * kWg3Row);
#pragma unroll 1
      for (int it = half, n = 0; it < 3 * boxes; it += 2, ++n) {
        uint8_t* mine = rows + (n & 1) * (32 * kWg3Row) + lane * kWg3Row;
        tma_store_wait_read<1>();                                       // the buffer's last contents have left
#pragma unroll
        for (int c = 0; c < 2; ++c) {
          float v[32];
          tmem_ld32(lanes + it * 64 + c * 32, v);
          tmem_ld_wait();
#pragma unroll
          for (int j = 0; j < 8; ++j)
            *reinterpret_cast<float4*>(mine + c * 128 + 16 * j) = make_float4(v[4 * j], v[4 * j + 1], v[4 * j + 2], v[4 * j + 3]);
        }
        fence_async_smem();
        const int tap = 3 * (it % 3) + kx, ch = tc * 128 + it / 3 * 64;
        if (row < g.cout) bulk_add_f32(g.out + size_t(row) * (9 * g.cin) + tap * g.cin + ch, mine, 256);
        tma_store_commit();
      }
      if (sums && half) {
        float v[16];
        tmem_ld16(lanes + 384, v);
        tmem_ld_wait();
        if (row < g.cout) atomicAdd(g.colsum + row, v[0]);
      }
      tma_store_wait_read<0>();
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    if (*abort_flag) abort_settle();
    tc_fence_after();
    tmem_dealloc(tmem_base, 512);
  }
}

// The result leaves in 3 x 64 columns per box whatever the number of patches is: below about 256 units of work (patches x tiles) the
// reduction GEMM's smaller tiles are done sooner (16 x 16 pixels, 128 -> 128 channels, 12 units: 10.2 against 14.3 us; 33 x 17, 192 -> 136,
// 216: 12.3 against 14.3; 2 x 32 x 32, 256 -> 256, 384: 18.4 against 14.3).
inline bool conv3_wgrad_applicable(const NtCall& c) {
  const long long patches = (long long)c.img_n * ((c.img_h + kWgTileH - 1) / kWgTileH) * ((c.img_w + kWgTileW - 1) / kWgTileW);
  return !c.halo && !c.max_ctas && patches * (3 * ((c.Na + 127) / 128) * ((c.cin + 127) / 128)) >= 256;
}

inline int launch_conv3_wgrad(const NtCall& c, int num_sms, int* err_word, cudaStream_t stream) {
  using Cfg = Wg3Cfg;
  constexpr int TH = Cfg::TH;
  if (!c.conv || c.halo || c.cin % 64 || c.Na < 64 || (reinterpret_cast<uintptr_t>(c.out) & 15)) return -24;
  CUtensorMap tA, tB;
  if (make_tmap_nhwc_b16(&tA, c.A, c.img_n, c.img_h, c.img_w, c.Na, TH, kWgTileW)) return -20;
  if (make_tmap_nhwc_b16(&tB, c.B, c.img_n, c.img_h, c.img_w, c.cin, TH + 2, kWgTileW)) return -21;
  Wg3Args g;
  g.cout = c.Na; g.cin = c.cin; g.out = c.out; g.colsum = c.colsum; g.err = err_word;
  g.tiles_x = (c.img_w + kWgTileW - 1) / kWgTileW;
  g.tiles_y = (c.img_h + TH - 1) / TH;
  g.patches = c.img_n * g.tiles_x * g.tiles_y;
  g.tiles_a = (c.Na + 127) / 128;
  g.tiles_c = (c.cin + 127) / 128;
  const int tiles = g.tiles_a * g.tiles_c * 3;
  // Whole parts only: 75 to 147 tiles leave SMs idle, 149 and more make rounds of whole tiles.  It is still the sooner kernel there (us,
  // reduction GEMM / this; 16 x 16, 64 x 64, 128 x 128 pixels): 640 -> 640 channels, 75 tiles, 24 / 16, 114 / 49, 323 / 150; 512 -> 896, 84
  // tiles, 24 / 16, 85 / 49, 221 / 150; 896 -> 896, 147 tiles, 34 / 21, 171 / 55, 636 / 156; 1024 -> 1024, 192 tiles, 40 / 29, 163 / 94,
  // 431 / 289; 1280 -> 1280, 300 tiles, 54 / 37, 298 / 135, 833 / 442.
  int splits = num_sms / tiles;            // also few patches: 64 in 24 parts 16.4 us, in 8 18.4 us (256 -> 128 channels, 64 x 64 pixels)
  if (splits < 1) splits = 1;
  if (splits > g.patches) splits = g.patches;
  g.per_split = (g.patches + splits - 1) / splits;
  splits = (g.patches + g.per_split - 1) / g.per_split;
  static DeviceMask smem_set{0};
  if (!allow_smem(conv3_wgrad_kernel, Cfg::SMEM, smem_set)) return -22;
  conv3_wgrad_kernel<<<tiles * splits, kWg3Threads, Cfg::SMEM, stream>>>(tA, tB, g);
  return cudaGetLastError() == cudaSuccess ? 0 : -23;
}

}  // namespace pnm

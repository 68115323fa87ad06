// LayerNorm forward / backward over the last dimension, bf16 activations, fp32 statistics
// and parameters.  One or two rows per warp, 16-byte vectors; the backward's CTAs write partial
// column sums to scratch, which a second tiny kernel folds.
#pragma once
#include "common.cuh"
#include "pnm_internal.h"

namespace pnm {

constexpr int kLnWarps = 8;
constexpr int kLnMaxVec = 4;  // supports C up to 32 lanes * 8 elems * 4 = 1024

// y = (x - mean) * rstd * gamma + beta (+ post); optional second input r: normalises (x + r)
// and writes the sum to `sum_out` (fused residual add before the normalisation).
// LPR lanes share a row: 32 (one row per warp) or 16 (two rows per warp, C <= 256).  With a whole warp on a 256-wide row
// the kernel is bound by instruction issue, not by memory (ncu: warps stall "not selected" / on the shuffle chains while
// DRAM is ~50 % busy); two rows per warp halve the instructions per row.  This form is for the fused residual add; without
// `r` the streaming kernel below runs.
template <int VEC, int LPR>
__global__ void __launch_bounds__(kLnWarps * 32, VEC == 1 ? 3 : 2)
layernorm_fwd_kernel(const __nv_bfloat16* __restrict__ x, const __nv_bfloat16* __restrict__ r,
                     const float* __restrict__ gamma, const float* __restrict__ beta, __nv_bfloat16* __restrict__ y,
                     __nv_bfloat16* __restrict__ sum_out, float* __restrict__ mean_out, float* __restrict__ rstd_out,
                     const __nv_bfloat16* __restrict__ post, long long M, int C, float eps) {
  constexpr int RW = 32 / LPR;                            // rows per warp and step
  const int lane = threadIdx.x & 31, l = lane % LPR, sub = lane / LPR;
  const long long first = ((long long)blockIdx.x * kLnWarps + (threadIdx.x >> 5)) * RW + sub;
  const long long stride = (long long)gridDim.x * kLnWarps * RW;
  float gam[VEC][8], bet[VEC][8];
#pragma unroll
  for (int v = 0; v < VEC; ++v) {
    const int c = (v * LPR + l) * 8;
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      gam[v][j] = (c + j < C) ? gamma[c + j] : 0.f;
      bet[v][j] = (c + j < C && beta) ? beta[c + j] : 0.f;
    }
  }
  // A ring of D steps per warp is kept in flight: the loads of step i + D are issued before step i is processed.
  constexpr int D = (VEC <= 2) ? 2 : 1;                  // wider rows: the ring would spill
  uint4 nx[D][VEC], nr[D][VEC];
  auto fetch = [&](int slot, long long row) {
#pragma unroll
    for (int v = 0; v < VEC; ++v) {
      const int c = (v * LPR + l) * 8;
      const bool live = row < M && c < C;
      nx[slot][v] = live ? *reinterpret_cast<const uint4*>(x + row * C + c) : make_uint4(0u, 0u, 0u, 0u);
      nr[slot][v] = live ? *reinterpret_cast<const uint4*>(r + row * C + c) : make_uint4(0u, 0u, 0u, 0u);
    }
  };
#pragma unroll
  for (int d = 0; d < D; ++d) fetch(d, first + d * stride);
  // the loop bound is the same for all lanes of a warp (the shuffles below need every lane): rows past M are masked
  for (long long row0 = first - sub; row0 < M; row0 += D * stride) {
#pragma unroll
    for (int d = 0; d < D; ++d) {
      const long long row = row0 + sub + d * stride;
      const bool in = row < M;
      if (row0 + d * stride >= M) break;
      float val[VEC][8];
      float s = 0.f;
      uint4 cx[VEC], cr[VEC];
#pragma unroll
      for (int v = 0; v < VEC; ++v) { cx[v] = nx[d][v]; cr[v] = nr[d][v]; }
      fetch(d, row + D * stride);
#pragma unroll
      for (int v = 0; v < VEC; ++v) {
        const int c = (v * LPR + l) * 8;
        if (c < C) {
          const uint4 u = cx[v];
          const uint32_t w[4] = {u.x, u.y, u.z, u.w};
          const uint4 ur = cr[v];
          const uint32_t rw[4] = {ur.x, ur.y, ur.z, ur.w};
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            float2 f = unpack_bf16x2(w[j]);
            const float2 fr = unpack_bf16x2(rw[j]);
            f.x += fr.x; f.y += fr.y;
            val[v][2 * j] = f.x; val[v][2 * j + 1] = f.y;
            s += f.x + f.y;
          }
          if (sum_out && in) {
            uint4 o;
            o.x = pack_bf16x2(val[v][0], val[v][1]); o.y = pack_bf16x2(val[v][2], val[v][3]);
            o.z = pack_bf16x2(val[v][4], val[v][5]); o.w = pack_bf16x2(val[v][6], val[v][7]);
            *reinterpret_cast<uint4*>(sum_out + row * C + c) = o;
          }
        } else {
#pragma unroll
          for (int j = 0; j < 8; ++j) val[v][j] = 0.f;
        }
      }
#pragma unroll
      for (int o = LPR / 2; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
      const float mean = s / C;
      float sq = 0.f;
#pragma unroll
      for (int v = 0; v < VEC; ++v) {
        const int c = (v * LPR + l) * 8;
        if (c < C) {
#pragma unroll
          for (int j = 0; j < 8; ++j) { const float dd = val[v][j] - mean; sq += dd * dd; }
        }
      }
#pragma unroll
      for (int o = LPR / 2; o > 0; o >>= 1) sq += __shfl_xor_sync(0xffffffffu, sq, o);
      const float rstd = rsqrtf(sq / C + eps);
      if (l == 0 && in) {
        if (mean_out) mean_out[row] = mean;
        if (rstd_out) rstd_out[row] = rstd;
      }
#pragma unroll
      for (int v = 0; v < VEC; ++v) {
        const int c = (v * LPR + l) * 8;
        if (c < C && in) {
          float o[8];
#pragma unroll
          for (int j = 0; j < 8; ++j) o[j] = (val[v][j] - mean) * rstd * gam[v][j] + bet[v][j];
          if (post) {  // y = LN(x) + post  (residual added after the normalisation)
            const uint4 up = *reinterpret_cast<const uint4*>(post + row * C + c);
            float2 f;
            f = unpack_bf16x2(up.x); o[0] += f.x; o[1] += f.y;
            f = unpack_bf16x2(up.y); o[2] += f.x; o[3] += f.y;
            f = unpack_bf16x2(up.z); o[4] += f.x; o[5] += f.y;
            f = unpack_bf16x2(up.w); o[6] += f.x; o[7] += f.y;
          }
          uint4 u;
          u.x = pack_bf16x2(o[0], o[1]); u.y = pack_bf16x2(o[2], o[3]);
          u.z = pack_bf16x2(o[4], o[5]); u.w = pack_bf16x2(o[6], o[7]);
          *reinterpret_cast<uint4*>(y + row * C + c) = u;
        }
      }
    }
  }
}

// ---- streaming variants: rows arrive in shared memory through bulk copies, several stages ahead of their use -------------
// A LayerNorm moves 2 (forward) to 4 (backward) rows per row of input and computes little, so its time is set by how many
// bytes are in flight per SM.  Loads into registers hold at most a row or two per warp (36 KB per SM at C = 256, which is
// worth 60 % of the HBM rate); a ring of bulk copies holds 190 KB whatever the registers do.  One producer warp, eight
// consumer warps; a stage is a run of whole rows, i.e. ONE contiguous copy per tensor (rows are C * 2 bytes, a multiple of 16).
constexpr int kLnStreamThreads = (kLnWarps + 1) * 32;
constexpr int kLnFoldBytes = kLnWarps * 2 * 264 * 4;   // column sums of the warps of a backward CTA
__device__ __forceinline__ void bulk_load(void* smem_dst, const void* src, uint32_t bytes, uint64_t* bar) {
  asm volatile("cp.async.bulk.shared::cta.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
               ::"r"(smem_u32(smem_dst)), "l"(src), "r"(bytes), "r"(smem_u32(bar))
               : "memory");
}

template <int VEC, int LPR>
__global__ void __launch_bounds__(kLnStreamThreads, VEC <= 2 ? 3 : 2)
layernorm_fwd_stream_kernel(const __nv_bfloat16* __restrict__ x, const float* __restrict__ gamma, const float* __restrict__ beta,
                            __nv_bfloat16* __restrict__ y, float* __restrict__ mean_out, float* __restrict__ rstd_out,
                            const __nv_bfloat16* __restrict__ post, long long M, int C, float eps, int stage_rows, int stages, int* err) {
  constexpr int RW = 32 / LPR;
  extern __shared__ __align__(128) uint8_t ln_smem[];
  const uint32_t tile_bytes = uint32_t(stage_rows) * C * 2, stage_bytes = tile_bytes * (post ? 2 : 1);
  uint64_t* full = reinterpret_cast<uint64_t*>(ln_smem + size_t(stages) * stage_bytes);
  uint64_t* empty = full + stages;
  volatile int* abort_flag = reinterpret_cast<volatile int*>(empty + stages);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, l = lane % LPR, sub = lane / LPR;
  const long long tiles = (M + stage_rows - 1) / stage_rows;
  if (threadIdx.x == 0) {
    for (int s = 0; s < stages; ++s) { mbar_init(&full[s], 1); mbar_init(&empty[s], kLnWarps); }
    *abort_flag = 0;
    mbar_fence_init();
  }
  __syncthreads();
  if (warp == kLnWarps) {
    if (elect_one()) {
      int s = 0;
      uint32_t ph = 1, issued = 0;
      for (long long t = blockIdx.x; t < tiles; t += gridDim.x) {
        if (!mbar_wait(&empty[s], ph, abort_flag, err, ERR_WAIT_EMPTY)) break;
        const long long row = t * stage_rows;
        const uint32_t bytes = uint32_t(M - row < stage_rows ? M - row : stage_rows) * C * 2;
        mbar_expect_tx(&full[s], post ? 2 * bytes : bytes);
        bulk_load(ln_smem + size_t(s) * stage_bytes, x + row * C, bytes, &full[s]);
        if (post) bulk_load(ln_smem + size_t(s) * stage_bytes + tile_bytes, post + row * C, bytes, &full[s]);
        if (++s == stages) { s = 0; ph ^= 1; }
        ++issued;
      }
      ring_drain(full, stages, issued);          // copies land before the CTA leaves, also after a wait that ran out
    }
    return;
  }
  float gam[VEC][8], bet[VEC][8];
#pragma unroll
  for (int v = 0; v < VEC; ++v) {
    const int c = (v * LPR + l) * 8;
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      gam[v][j] = (c + j < C) ? gamma[c + j] : 0.f;
      bet[v][j] = (c + j < C && beta) ? beta[c + j] : 0.f;
    }
  }
  int s = 0;
  uint32_t ph = 0;
  for (long long t = blockIdx.x; t < tiles; t += gridDim.x) {
    if (!mbar_wait(&full[s], ph, abort_flag, err, ERR_WAIT_FULL)) break;
    const __nv_bfloat16* tx = reinterpret_cast<const __nv_bfloat16*>(ln_smem + size_t(s) * stage_bytes);
    const __nv_bfloat16* tp = reinterpret_cast<const __nv_bfloat16*>(ln_smem + size_t(s) * stage_bytes + tile_bytes);
    for (int r0 = warp * RW; r0 < stage_rows; r0 += kLnWarps * RW) {
      const int r = r0 + sub;
      const long long row = t * stage_rows + r;
      if (row - sub >= M) break;                  // the same for all lanes of the warp
      const bool in = row < M;
      float val[VEC][8];
      float sum = 0.f;
#pragma unroll
      for (int v = 0; v < VEC; ++v) {
        const int c = (v * LPR + l) * 8;
        const uint4 u = c < C ? *reinterpret_cast<const uint4*>(tx + r * C + c) : make_uint4(0u, 0u, 0u, 0u);
        const uint32_t w[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const float2 f = unpack_bf16x2(w[j]);
          val[v][2 * j] = f.x; val[v][2 * j + 1] = f.y;
          sum += f.x + f.y;
        }
      }
#pragma unroll
      for (int o = LPR / 2; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
      const float mean = sum / C;
      float sq = 0.f;
#pragma unroll
      for (int v = 0; v < VEC; ++v)
        if ((v * LPR + l) * 8 < C) {
#pragma unroll
          for (int j = 0; j < 8; ++j) { const float dd = val[v][j] - mean; sq += dd * dd; }
        }
#pragma unroll
      for (int o = LPR / 2; o > 0; o >>= 1) sq += __shfl_xor_sync(0xffffffffu, sq, o);
      const float rstd = rsqrtf(sq / C + eps);
      if (l == 0 && in) {
        if (mean_out) mean_out[row] = mean;
        if (rstd_out) rstd_out[row] = rstd;
      }
#pragma unroll
      for (int v = 0; v < VEC; ++v) {
        const int c = (v * LPR + l) * 8;
        if (c < C && in) {
          float o[8];
#pragma unroll
          for (int j = 0; j < 8; ++j) o[j] = (val[v][j] - mean) * rstd * gam[v][j] + bet[v][j];
          if (post) {  // y = LN(x) + post  (residual added after the normalisation)
            const uint4 up = *reinterpret_cast<const uint4*>(tp + r * C + c);
            const uint32_t w[4] = {up.x, up.y, up.z, up.w};
#pragma unroll
            for (int j = 0; j < 4; ++j) { const float2 f = unpack_bf16x2(w[j]); o[2 * j] += f.x; o[2 * j + 1] += f.y; }
          }
          *reinterpret_cast<uint4*>(y + row * C + c) =
              make_uint4(pack_bf16x2(o[0], o[1]), pack_bf16x2(o[2], o[3]), pack_bf16x2(o[4], o[5]), pack_bf16x2(o[6], o[7]));
        }
      }
    }
    __syncwarp();
    if (lane == 0) mbar_arrive(&empty[s]);
    if (++s == stages) { s = 0; ph ^= 1; }
  }
}

// dx = rstd * (g*dy - mean_c(g*dy) - xhat * mean_c(g*dy*xhat)) (+ dres); partial dgamma / dbeta rows go to
// scratch[blockIdx.x][2][C], so that the column sums stay in registers until a CTA is done.
// Measured against one row per warp from registers: 1 M x 256 forward 0.213 -> 0.191 ms (0.82 of 6544 GB/s), backward with a residual
// gradient 0.420 -> 0.336 ms (0.93); 1.4 M x 128 forward 0.177 -> 0.159 ms, backward 0.507 -> 0.256 ms (two rows per warp);
// 32 400 x 768 27.2 -> 25.6 us, 56.1 -> 50.3 us.
template <int VEC, int LPR>
__global__ void __launch_bounds__(kLnStreamThreads, VEC == 1 ? 3 : (VEC == 2 ? 2 : 1))
layernorm_bwd_stream_kernel(const __nv_bfloat16* __restrict__ dy, const __nv_bfloat16* __restrict__ x, const float* __restrict__ gamma,
                            const float* __restrict__ mean_in, const float* __restrict__ rstd_in, const __nv_bfloat16* __restrict__ dres,
                            __nv_bfloat16* __restrict__ dx, float* __restrict__ scratch, long long M, int C, int stage_rows, int stages,
                            int* err) {
  constexpr int RW = 32 / LPR;                   // rows per warp and step (two for C <= 128: half a warp would idle)
  extern __shared__ __align__(128) uint8_t ln_smem[];
  const uint32_t tile_bytes = uint32_t(stage_rows) * C * 2, stage_bytes = tile_bytes * (dres ? 3 : 2);
  // the barriers and the flag lie behind the ring AND behind the fold, which is the larger of the two for C <= 32
  const size_t ring_bytes = size_t(stages) * stage_bytes;
  uint64_t* full = reinterpret_cast<uint64_t*>(ln_smem + (ring_bytes > kLnFoldBytes ? ring_bytes : kLnFoldBytes));
  uint64_t* empty = full + stages;
  volatile int* abort_flag = reinterpret_cast<volatile int*>(empty + stages);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, l = lane % LPR, sub = lane / LPR;
  const long long tiles = (M + stage_rows - 1) / stage_rows;
  if (threadIdx.x == 0) {
    for (int s = 0; s < stages; ++s) { mbar_init(&full[s], 1); mbar_init(&empty[s], kLnWarps); }
    *abort_flag = 0;
    mbar_fence_init();
  }
  __syncthreads();
  float dg[VEC][8], db[VEC][8];
#pragma unroll
  for (int v = 0; v < VEC; ++v)
#pragma unroll
    for (int j = 0; j < 8; ++j) dg[v][j] = db[v][j] = 0.f;
  if (warp == kLnWarps) {
    if (elect_one()) {
      int s = 0;
      uint32_t ph = 1, issued = 0;
      for (long long t = blockIdx.x; t < tiles; t += gridDim.x) {
        if (!mbar_wait(&empty[s], ph, abort_flag, err, ERR_WAIT_EMPTY)) break;
        const long long row = t * stage_rows;
        const uint32_t bytes = uint32_t(M - row < stage_rows ? M - row : stage_rows) * C * 2;
        uint8_t* st = ln_smem + size_t(s) * stage_bytes;
        mbar_expect_tx(&full[s], dres ? 3 * bytes : 2 * bytes);
        bulk_load(st, x + row * C, bytes, &full[s]);
        bulk_load(st + tile_bytes, dy + row * C, bytes, &full[s]);
        if (dres) bulk_load(st + 2 * tile_bytes, dres + row * C, bytes, &full[s]);
        if (++s == stages) { s = 0; ph ^= 1; }
        ++issued;
      }
      ring_drain(full, stages, issued);          // copies land before the CTA leaves, also after a wait that ran out
    }
  } else {
    float gam[VEC][8];
#pragma unroll
    for (int v = 0; v < VEC; ++v) {
      const int c = (v * LPR + l) * 8;
#pragma unroll
      for (int j = 0; j < 8; ++j) gam[v][j] = (c + j < C) ? gamma[c + j] : 0.f;
    }
    int s = 0;
    uint32_t ph = 0;
    // the statistics of the row after the next one are requested while a row is processed
    auto stat_row = [&](long long t, int r) { const long long row = t * stage_rows + r; return row < M ? row : M - 1; };
    const int r_first = warp * RW + sub;
    float nmean = mean_in[stat_row(blockIdx.x, r_first)], nrstd = rstd_in[stat_row(blockIdx.x, r_first)];
    for (long long t = blockIdx.x; t < tiles; t += gridDim.x) {
      if (!mbar_wait(&full[s], ph, abort_flag, err, ERR_WAIT_FULL)) break;
      const __nv_bfloat16* tx = reinterpret_cast<const __nv_bfloat16*>(ln_smem + size_t(s) * stage_bytes);
      const __nv_bfloat16* td = tx + size_t(stage_rows) * C;
      const __nv_bfloat16* tr = td + size_t(stage_rows) * C;
      for (int r = r_first; r < stage_rows; r += kLnWarps * RW) {
        const long long row = t * stage_rows + r;
        const bool in = row < M;
        const float mean = in ? nmean : 0.f, rstd = in ? nrstd : 0.f;
        const bool wrap = r + kLnWarps * RW >= stage_rows;
        const long long nrow = wrap ? stat_row(t + gridDim.x, r_first) : stat_row(t, r + kLnWarps * RW);
        nmean = mean_in[nrow];
        nrstd = rstd_in[nrow];
        if (row - sub >= M) continue;               // the same for all lanes of the warp
        float xh[VEC][8], gy[VEC][8];
        float s1 = 0.f, s2 = 0.f;
#pragma unroll
        for (int v = 0; v < VEC; ++v) {
          const int c = (v * LPR + l) * 8;
          const bool live = c < C && in;
          const uint4 ux = live ? *reinterpret_cast<const uint4*>(tx + r * C + c) : make_uint4(0u, 0u, 0u, 0u);
          const uint4 ud = live ? *reinterpret_cast<const uint4*>(td + r * C + c) : make_uint4(0u, 0u, 0u, 0u);
          const uint32_t wx[4] = {ux.x, ux.y, ux.z, ux.w}, wd[4] = {ud.x, ud.y, ud.z, ud.w};
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            const float2 fx = unpack_bf16x2(wx[j]), fd = unpack_bf16x2(wd[j]);
            const float h0 = (fx.x - mean) * rstd, h1 = (fx.y - mean) * rstd;
            xh[v][2 * j] = h0; xh[v][2 * j + 1] = h1;
            dg[v][2 * j] += fd.x * h0; dg[v][2 * j + 1] += fd.y * h1;
            db[v][2 * j] += fd.x; db[v][2 * j + 1] += fd.y;
            const float g0 = fd.x * gam[v][2 * j], g1 = fd.y * gam[v][2 * j + 1];
            gy[v][2 * j] = g0; gy[v][2 * j + 1] = g1;
            s1 += g0 + g1; s2 += g0 * h0 + g1 * h1;
          }
        }
#pragma unroll
        for (int o = LPR / 2; o > 0; o >>= 1) {
          s1 += __shfl_xor_sync(0xffffffffu, s1, o);
          s2 += __shfl_xor_sync(0xffffffffu, s2, o);
        }
        const float m1 = s1 / C, m2 = s2 / C;
#pragma unroll
        for (int v = 0; v < VEC; ++v) {
          const int c = (v * LPR + l) * 8;
          if (c < C && in) {
            float o[8];
#pragma unroll
            for (int j = 0; j < 8; ++j) o[j] = rstd * (gy[v][j] - m1 - xh[v][j] * m2);
            if (dres) {
              const uint4 ur = *reinterpret_cast<const uint4*>(tr + r * C + c);
              const uint32_t wr[4] = {ur.x, ur.y, ur.z, ur.w};
#pragma unroll
              for (int j = 0; j < 4; ++j) { const float2 f = unpack_bf16x2(wr[j]); o[2 * j] += f.x; o[2 * j + 1] += f.y; }
            }
            *reinterpret_cast<uint4*>(dx + row * C + c) =
                make_uint4(pack_bf16x2(o[0], o[1]), pack_bf16x2(o[2], o[3]), pack_bf16x2(o[4], o[5]), pack_bf16x2(o[6], o[7]));
          }
        }
      }
      __syncwarp();
      if (lane == 0) mbar_arrive(&empty[s]);
      if (++s == stages) { s = 0; ph ^= 1; }
    }
  }
  // fold the warps of this CTA, one vector slot at a time, in the ring's memory: every copy into it has been waited for by all
  // consumers (after a wait that ran out the results are void)
  __syncthreads();
  if (*abort_flag) return;
  float* red = reinterpret_cast<float*>(ln_smem);   // kLnFoldBytes: [warps][2][264]
  constexpr int COLS = LPR * 8;                     // columns one vector slot covers
#pragma unroll
  for (int v = 0; v < VEC; ++v) {
    if (warp < kLnWarps) {
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        float a = dg[v][j], b = db[v][j];
        if (LPR == 16) { a += __shfl_xor_sync(0xffffffffu, a, 16); b += __shfl_xor_sync(0xffffffffu, b, 16); }
        if (sub == 0) { red[(warp * 2 + 0) * 264 + l * 8 + j] = a; red[(warp * 2 + 1) * 264 + l * 8 + j] = b; }
      }
    }
    __syncthreads();
    for (int i = threadIdx.x; i < 2 * COLS; i += kLnStreamThreads) {
      const int which = i / COLS, col = i % COLS, c = v * COLS + col;
      float sum = 0.f;
#pragma unroll
      for (int w = 0; w < kLnWarps; ++w) sum += red[(w * 2 + which) * 264 + col];
      if (c < C) scratch[((size_t)blockIdx.x * 2 + which) * C + c] = sum;
    }
    __syncthreads();
  }
}

// dgamma[c] = sum_b scratch[b][0][c], dbeta[c] = sum_b scratch[b][1][c].  A CTA owns 32 consecutive entries of the
// 2 C-wide scratch row; its 16 row groups walk the nblocks rows in parallel (coalesced 128-byte reads) and are folded
// through shared memory, so the dependent chain is nblocks / 16 loads instead of nblocks.
constexpr int kLnFoldRows = 16;
static __global__ void __launch_bounds__(32 * kLnFoldRows)
layernorm_bwd_finalize_kernel(const float* __restrict__ scratch, int nblocks, int C, float* __restrict__ dgamma,
                              float* __restrict__ dbeta) {
  __shared__ float part[kLnFoldRows][33];
  const int lane = threadIdx.x & 31, grp = threadIdx.x >> 5;
  const int i = blockIdx.x * 32 + lane;                       // entry of the [2][C] row
  float s = 0.f;
  if (i < 2 * C)
    for (int b = grp; b < nblocks; b += kLnFoldRows) s += scratch[(size_t)b * 2 * C + i];
  part[grp][lane] = s;
  __syncthreads();
  if (grp == 0 && i < 2 * C) {
    float t = 0.f;
#pragma unroll
    for (int g = 0; g < kLnFoldRows; ++g) t += part[g][lane];
    const int which = i / C, c = i % C;
    if (which == 0) { if (dgamma) dgamma[c] = t; }
    else { if (dbeta) dbeta[c] = t; }
  }
}

// Rows of a stage, stages and CTAs per SM of the streaming kernels: stages of about 16 KB per tensor (more rows where they are
// short) of which two fit a ring, `per_sm` rings that together fill the shared memory; with few rows in all, the smallest stage that
// still gives every warp a row, so that the rows spread over more SMs.  (Three tensors of 16 KB, twice, fill half the shared memory: a
// third of the CTAs then ran as a second wave.  1 M x 256 backward with a residual gradient 398 -> 339 us, 0.92 of the copy rate;
// 1.4 M x 128 296 -> 259 us; 100 003 x 256 64 -> 50 us.)
struct LnStream { int rows, stages, grid, smem; };
inline LnStream ln_stream_plan(long long M, int C, int tensors, int least_rows, int per_sm, int num_sms) {
  LnStream p;
  const int budget = 220 * 1024 / per_sm - 256, fits = budget / (4 * C * tensors);      // rows of each of two stages
  int rows = 16384 / (2 * C);
  if (rows > fits) rows = fits;
  if (rows > 256) rows = 256;
  rows = rows / least_rows * least_rows;
  if (rows < least_rows || M < (long long)num_sms * per_sm * rows) rows = least_rows;
  const int stage = rows * C * 2 * tensors;
  p.rows = rows;
  p.stages = budget / stage > 8 ? 8 : budget / stage;
  const int ring = p.stages * stage;             // the backward folds its warps in the ring's place
  p.smem = (ring > kLnFoldBytes ? ring : kLnFoldBytes) + p.stages * 16 + 16;
  const long long tiles = (M + rows - 1) / rows, cap = (long long)num_sms * per_sm;
  p.grid = int(tiles < cap ? tiles : cap);
  return p;
}
constexpr int kLnSmemMax = 225 * 1024;

template <int VEC, int LPR>
inline int launch_ln_fwd_stream(const __nv_bfloat16* x, const float* gamma, const float* beta, __nv_bfloat16* y, float* mean, float* rstd,
                                const __nv_bfloat16* post, long long M, int C, float eps, int num_sms, int* err, cudaStream_t st) {
  static DeviceMask smem_set{0};
  if (!allow_smem(layernorm_fwd_stream_kernel<VEC, LPR>, kLnSmemMax, smem_set)) return -31;
  const LnStream p = ln_stream_plan(M, C, post ? 2 : 1, kLnWarps * (32 / LPR), VEC <= 2 ? 3 : 2, num_sms);
  layernorm_fwd_stream_kernel<VEC, LPR><<<p.grid, kLnStreamThreads, p.smem, st>>>(x, gamma, beta, y, mean, rstd, post, M, C, eps, p.rows,
                                                                                  p.stages, err);
  return cudaGetLastError() == cudaSuccess ? 0 : -31;
}

inline int launch_layernorm_fwd(const void* x, const void* r, const float* gamma, const float* beta, void* y,
                                void* sum_out, float* mean, float* rstd, const void* post, long long M, int C,
                                float eps, int num_sms, int* err, cudaStream_t st) {
  if (C % 8 || C > 1024) return -30;
  auto X = (const __nv_bfloat16*)x; auto R = (const __nv_bfloat16*)r; auto Y = (__nv_bfloat16*)y; auto S = (__nv_bfloat16*)sum_out; auto P = (const __nv_bfloat16*)post;
  if (!R) {
    if (M <= 0) return 0;
    if (C <= 128) return launch_ln_fwd_stream<1, 16>(X, gamma, beta, Y, mean, rstd, P, M, C, eps, num_sms, err, st);
    if (C <= 256) return launch_ln_fwd_stream<2, 16>(X, gamma, beta, Y, mean, rstd, P, M, C, eps, num_sms, err, st);
    if (C <= 512) return launch_ln_fwd_stream<2, 32>(X, gamma, beta, Y, mean, rstd, P, M, C, eps, num_sms, err, st);
    if (C <= 768) return launch_ln_fwd_stream<3, 32>(X, gamma, beta, Y, mean, rstd, P, M, C, eps, num_sms, err, st);
    return launch_ln_fwd_stream<4, 32>(X, gamma, beta, Y, mean, rstd, P, M, C, eps, num_sms, err, st);
  }
  long long want = (M + kLnWarps - 1) / kLnWarps;
  // whole waves of resident CTAs (3 per SM for C <= 128, 2 above): a partial last wave would idle part of the SMs
  const long long resident = (long long)num_sms * (C <= 128 ? 3 : 2);
  int grid = (int)(want < resident * 2 ? want : resident * 2);
  if (grid < 1) grid = 1;
#define PNM_LN_FWD(V, L) layernorm_fwd_kernel<V, L><<<grid, kLnWarps * 32, 0, st>>>(X, R, gamma, beta, Y, S, mean, rstd, P, M, C, eps)
  if (C <= 128) { PNM_LN_FWD(1, 16); }
  else if (C <= 256) { PNM_LN_FWD(2, 16); }
  else if (C <= 512) { PNM_LN_FWD(2, 32); }
  else if (C <= 768) { PNM_LN_FWD(3, 32); }
  else { PNM_LN_FWD(4, 32); }
#undef PNM_LN_FWD
  return cudaGetLastError() == cudaSuccess ? 0 : -31;
}

// CTAs of the backward = rows of scratch needed (2 * C floats each), for the case with the most of them.
inline int ln_bwd_rows(int C) { return C <= 128 ? 2 * kLnWarps : kLnWarps; }
inline int ln_bwd_per_sm(int C) { return C <= 256 ? 3 : (C <= 512 ? 2 : 1); }
inline int layernorm_bwd_grid(long long M, int num_sms, int C) {
  if (M <= 0) return 1;
  const int a = ln_stream_plan(M, C, 2, ln_bwd_rows(C), ln_bwd_per_sm(C), num_sms).grid;
  const int b = ln_stream_plan(M, C, 3, ln_bwd_rows(C), ln_bwd_per_sm(C), num_sms).grid;
  return a > b ? a : b;
}

template <int VEC, int LPR>
inline int launch_ln_bwd_stream(const __nv_bfloat16* dy, const __nv_bfloat16* x, const float* gamma, const float* mean, const float* rstd,
                                const __nv_bfloat16* dres, __nv_bfloat16* dx, float* scratch, long long M, int C, const LnStream& p, int* err,
                                cudaStream_t st) {
  static DeviceMask smem_set{0};
  if (!allow_smem(layernorm_bwd_stream_kernel<VEC, LPR>, kLnSmemMax, smem_set)) return -33;
  layernorm_bwd_stream_kernel<VEC, LPR><<<p.grid, kLnStreamThreads, p.smem, st>>>(dy, x, gamma, mean, rstd, dres, dx, scratch, M, C, p.rows,
                                                                             p.stages, err);
  return cudaGetLastError() == cudaSuccess ? 0 : -33;
}

// dx and the partial dgamma / dbeta rows of every CTA (at most `max_ctas`); `p` tells how many there are.
inline int launch_layernorm_bwd_rows(const void* dy, const void* x, const float* gamma, const float* mean, const float* rstd,
                                     const void* dres, void* dx, float* scratch, long long M, int C, int max_ctas, int num_sms, int* err,
                                     cudaStream_t st, LnStream& p) {
  auto DY = (const __nv_bfloat16*)dy; auto X = (const __nv_bfloat16*)x; auto DR = (const __nv_bfloat16*)dres; auto DX = (__nv_bfloat16*)dx;
  p = ln_stream_plan(M, C, dres ? 3 : 2, ln_bwd_rows(C), ln_bwd_per_sm(C), num_sms);
  if (p.grid > max_ctas) p.grid = max_ctas;
  if (C <= 128) return launch_ln_bwd_stream<1, 16>(DY, X, gamma, mean, rstd, DR, DX, scratch, M, C, p, err, st);
  if (C <= 256) return launch_ln_bwd_stream<1, 32>(DY, X, gamma, mean, rstd, DR, DX, scratch, M, C, p, err, st);
  if (C <= 512) return launch_ln_bwd_stream<2, 32>(DY, X, gamma, mean, rstd, DR, DX, scratch, M, C, p, err, st);
  if (C <= 768) return launch_ln_bwd_stream<3, 32>(DY, X, gamma, mean, rstd, DR, DX, scratch, M, C, p, err, st);
  return launch_ln_bwd_stream<4, 32>(DY, X, gamma, mean, rstd, DR, DX, scratch, M, C, p, err, st);
}

inline int launch_layernorm_bwd(const void* dy, const void* x, const float* gamma, const float* mean,
                                const float* rstd, const void* dres, void* dx, float* dgamma, float* dbeta,
                                float* scratch, long long M, int C, int num_sms, int* err, cudaStream_t st) {
  if (C % 8 || C > 1024) return -32;
  LnStream p{};
  if (M > 0)
    if (const int rc = launch_layernorm_bwd_rows(dy, x, gamma, mean, rstd, dres, dx, scratch, M, C, 1 << 30, num_sms, err, st, p)) return rc;
  layernorm_bwd_finalize_kernel<<<(2 * C + 31) / 32, 32 * kLnFoldRows, 0, st>>>(scratch, p.grid, C, dgamma, dbeta);
  return cudaGetLastError() == cudaSuccess ? 0 : -34;
}

}  // namespace pnm

// Host side of the fused three-layer perceptron (kernels in mlp_fused.cuh).
#include "mlp_fused.cuh"
#include "mlp_fused_bwd.cuh"
#include "pnm_api.h"

namespace pnm {

template <int NSRC, int ACT, bool SAVE>
static int launch_mlp3(const CUtensorMap* tm, const CUtensorMap* tw, const MlpArgs& g, int grid, cudaStream_t st) {
  using Cfg = MlpCfg<NSRC>;
  static DeviceMask smem_set{0};
  if (!allow_smem(mlp3_ln_kernel<NSRC, ACT, SAVE>, Cfg::SMEM, smem_set)) return -16;
  mlp3_ln_kernel<NSRC, ACT, SAVE><<<grid, kMlpThreads, Cfg::SMEM, st>>>(tm[0], tm[1], tm[2], tw[0], tw[1], tw[2], g);
  return cudaGetLastError() == cudaSuccess ? 0 : -17;
}
template <int NSRC, int ACT>
static int launch_mlp3_save(const CUtensorMap* tm, const CUtensorMap* tw, const MlpArgs& g, int grid, cudaStream_t st) {
  return g.h1 ? launch_mlp3<NSRC, ACT, true>(tm, tw, g, grid, st) : launch_mlp3<NSRC, ACT, false>(tm, tw, g, grid, st);
}
template <int NSRC>
static int launch_mlp3_act(const CUtensorMap* tm, const CUtensorMap* tw, const MlpArgs& g, int grid, cudaStream_t st) {
  switch (g.act) {
    case MLP_SILU: return launch_mlp3_save<NSRC, MLP_SILU>(tm, tw, g, grid, st);
    case MLP_RELU: return launch_mlp3_save<NSRC, MLP_RELU>(tm, tw, g, grid, st);
    case MLP_GELU: return launch_mlp3_save<NSRC, MLP_GELU>(tm, tw, g, grid, st);
  }
  return -7;
}

template <int ACT>
static int launch_mlp3_bwd(const CUtensorMap& td, const CUtensorMap& th2, const CUtensorMap& th1, const CUtensorMap& t3,
                           const CUtensorMap& t2, const MlpBwdArgs& g, int grid, cudaStream_t st) {
  static DeviceMask smem_set{0};
  if (!allow_smem(mlp3_bwd_kernel<ACT>, kMlpBwdSmem, smem_set)) return -16;
  mlp3_bwd_kernel<ACT><<<grid, kMlpBwdThreads, kMlpBwdSmem, st>>>(td, th2, th1, t3, t2, g);
  return cudaGetLastError() == cudaSuccess ? 0 : -17;
}

// out[n] = [hi(s) | lo(s)], s = sum over k in [off[n], off[n+1]) of in[perm[k]] in fp32: two bf16 rows whose sum carries 16
// bits of s.  Against 64 bits dW1 of an edge MLP errs 0.9975 +- 0.0008 (601 nodes), 0.998 (4 001), 0.997 (30 011) times as much as with
// one product per row, and the gradients of the table, which that path rounds row by row, 0.934 times as much.  One thread per 16-byte chunk of a row, as the plain sum.
__global__ void __launch_bounds__(256)
segment_sum_split_kernel(const __nv_bfloat16* __restrict__ in, const int* __restrict__ perm, const int* __restrict__ offsets,
                         __nv_bfloat16* __restrict__ out, long long ldo, long long N, int C) {
  const int cpr = C >> 3;
  const long long total = N * cpr;
  for (long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x; t < total; t += (long long)gridDim.x * blockDim.x) {
    const long long n = t / cpr;
    const int c = int(t - n * cpr) << 3;
    const int k0 = __ldg(offsets + n), k1 = __ldg(offsets + n + 1);
    float acc[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
#pragma unroll 4
    for (int k = k0; k < k1; ++k) {
      const uint4 v = *reinterpret_cast<const uint4*>(in + (long long)__ldg(perm + k) * C + c);
      float2 f;
      f = unpack_bf16x2(v.x); acc[0] += f.x; acc[1] += f.y;
      f = unpack_bf16x2(v.y); acc[2] += f.x; acc[3] += f.y;
      f = unpack_bf16x2(v.z); acc[4] += f.x; acc[5] += f.y;
      f = unpack_bf16x2(v.w); acc[6] += f.x; acc[7] += f.y;
    }
    uint32_t hi[4], lo[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      hi[j] = pack_bf16x2(acc[2 * j], acc[2 * j + 1]);
      const float2 f = unpack_bf16x2(hi[j]);
      // a sum that is not finite in bf16 stays what it is: inf - inf must not make it NaN
      lo[j] = pack_bf16x2(fabsf(f.x) < 3.4e38f ? acc[2 * j] - f.x : 0.f, fabsf(f.y) < 3.4e38f ? acc[2 * j + 1] - f.y : 0.f);
    }
    __nv_bfloat16* dst = out + n * ldo + c;
    *reinterpret_cast<uint4*>(dst) = make_uint4(hi[0], hi[1], hi[2], hi[3]);
    *reinterpret_cast<uint4*>(dst + C) = make_uint4(lo[0], lo[1], lo[2], lo[3]);
  }
}

}  // namespace pnm

extern "C" int pnm_mlp3_bwd(const void* dx3, const void* z2, const void* z1, const void* h2, const void* h1, const void* W3t, const void* W2t,
                            int act, void* g1, float* dW3, float* dW2, float* db3, float* db2, long long M, void* stream) {
  using namespace pnm;
  int* err = error_word_ptr();
  if (!err) return -1;
  if (M <= 0 || M > 0x7fffff00LL) return -2;
  if (((reinterpret_cast<uintptr_t>(z2) | reinterpret_cast<uintptr_t>(z1) | reinterpret_cast<uintptr_t>(g1)) & 31) ||
      ((reinterpret_cast<uintptr_t>(dW3) | reinterpret_cast<uintptr_t>(dW2)) & 15))
    return -3;
  CUtensorMap td, th2, th1, t3, t2;
  if (make_tmap_2d_b16(&td, dx3, M, kMlpW, kMlpW, kMlpRows, 64)) return -9;
  if (make_tmap_2d_b16(&th2, h2, M, kMlpW, kMlpW, kMlpRows, 64)) return -12;
  if (make_tmap_2d_b16(&th1, h1, M, kMlpW, kMlpW, kMlpRows, 64)) return -13;
  if (make_tmap_2d_b16(&t3, W3t, kMlpW, kMlpW, kMlpW, kMlpW, 64)) return -10;
  if (make_tmap_2d_b16(&t2, W2t, kMlpW, kMlpW, kMlpW, kMlpW, 64)) return -11;
  MlpBwdArgs g{};
  g.M = M; g.z2 = reinterpret_cast<const __nv_bfloat16*>(z2); g.z1 = reinterpret_cast<const __nv_bfloat16*>(z1);
  g.g1 = reinterpret_cast<__nv_bfloat16*>(g1);
  g.dW3 = dW3; g.dW2 = dW2; g.db3 = db3; g.db2 = db2; g.err = err;
  const long long tiles = (M + kMlpRows - 1) / kMlpRows;
  const int sms = num_sms();
  const int grid = int(tiles < sms ? tiles : sms);
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  switch (act) {
    case MLP_SILU: return launch_mlp3_bwd<MLP_SILU>(td, th2, th1, t3, t2, g, grid, st);
    case MLP_RELU: return launch_mlp3_bwd<MLP_RELU>(td, th2, th1, t3, t2, g, grid, st);
    case MLP_GELU: return launch_mlp3_bwd<MLP_GELU>(td, th2, th1, t3, t2, g, grid, st);
  }
  return -7;
}

extern "C" int pnm_segment_sum_split(const void* in, const int* perm, const int* offsets, void* out, long long ldo, long long N, int C,
                                     void* stream) {
  using namespace pnm;
  if (C % 8 || ldo % 8 || N < 0 || ((reinterpret_cast<uintptr_t>(in) | reinterpret_cast<uintptr_t>(out)) & 15)) return -42;
  if (N == 0) return 0;
  const long long want = (N * (C >> 3) + 255) / 256, cap = (long long)num_sms() * 16;
  segment_sum_split_kernel<<<int(want < cap ? want : cap), 256, 0, reinterpret_cast<cudaStream_t>(stream)>>>(
      reinterpret_cast<const __nv_bfloat16*>(in), perm, offsets, reinterpret_cast<__nv_bfloat16*>(out), ldo, N, C);
  return cudaGetLastError() == cudaSuccess ? 0 : -43;
}

extern "C" int pnm_mlp3_ln_fwd(int nsrc, const void* const* src, const long long* rows, const int* ld, const int* const* idx, const void* W1,
                               const void* W2, const void* W3, const float* b1, const float* b2, const float* b3, const float* gamma,
                               const float* beta, float eps, int act, const void* post, long long ld_post, void* y, long long ld_y, void* z1,
                               void* z2, void* h1, void* h2, void* x3, float* mean, float* rstd, long long M, void* stream) {
  using namespace pnm;
  int* err = error_word_ptr();
  if (!err) return -1;
  if (nsrc < 1 || nsrc > 3 || M <= 0 || M > 0x7fffff00LL || !gamma || !y) return -2;
  const bool save = h1 != nullptr;
  if (save && (!h1 || !h2 || !x3 || !mean || !rstd || (act != MLP_RELU && (!z1 || !z2)))) return -5;
  const uintptr_t sectors = reinterpret_cast<uintptr_t>(post) | reinterpret_cast<uintptr_t>(y) | reinterpret_cast<uintptr_t>(z1) |
                            reinterpret_cast<uintptr_t>(z2) | reinterpret_cast<uintptr_t>(h1) | reinterpret_cast<uintptr_t>(h2) |
                            reinterpret_cast<uintptr_t>(x3) | uintptr_t((post ? ld_post : 0) * 2) |
                            uintptr_t(ld_y * 2);
  if (sectors & 31) return -3;                   // rows are read and written as 32-byte vectors
  const uintptr_t vec = reinterpret_cast<uintptr_t>(b1) | reinterpret_cast<uintptr_t>(b2) | reinterpret_cast<uintptr_t>(b3) |
                        reinterpret_cast<uintptr_t>(gamma) | reinterpret_cast<uintptr_t>(beta);
  if (vec & 15) return -3;
  CUtensorMap tm[3], tw[3];
  MlpArgs g{};
  for (int j = 0; j < nsrc; ++j) {
    if (rows[j] <= 0 || (!idx[j] && rows[j] < M)) return -2;
    g.idx[j] = idx[j];
    g.src[j] = reinterpret_cast<const __nv_bfloat16*>(src[j]); g.ld_src[j] = ld[j];
    if ((reinterpret_cast<uintptr_t>(src[j]) & 15) || (ld[j] & 7)) return -10 - j;
    if (idx[j]) tm[j] = CUtensorMap{};           // rows are copied one by one
    else if (make_tmap_2d_b16(&tm[j], src[j], M, kMlpW, ld[j], kMlpRows, 64)) return -10 - j;
  }
  for (int j = nsrc; j < 3; ++j) { tm[j] = tm[0]; g.idx[j] = nullptr; }
  if (make_tmap_2d_b16(&tw[0], W1, kMlpW, nsrc * kMlpW, nsrc * kMlpW, kMlpW, 64)) return -13;
  if (make_tmap_2d_b16(&tw[1], W2, kMlpW, kMlpW, kMlpW, kMlpW, 64)) return -14;
  if (make_tmap_2d_b16(&tw[2], W3, kMlpW, kMlpW, kMlpW, kMlpW, 64)) return -15;
  g.M = M; g.b1 = b1; g.b2 = b2; g.b3 = b3; g.gamma = gamma; g.beta = beta;
  g.post = reinterpret_cast<const __nv_bfloat16*>(post); g.ld_post = ld_post;
  g.y = reinterpret_cast<__nv_bfloat16*>(y); g.ld_y = ld_y;
  g.z1 = reinterpret_cast<__nv_bfloat16*>(z1); g.z2 = reinterpret_cast<__nv_bfloat16*>(z2); g.x3 = reinterpret_cast<__nv_bfloat16*>(x3);
  g.h1 = reinterpret_cast<__nv_bfloat16*>(h1); g.h2 = reinterpret_cast<__nv_bfloat16*>(h2);
  g.mean = mean; g.rstd = rstd; g.eps = eps; g.act = act; g.err = err;
  const long long tiles = (M + kMlpRows - 1) / kMlpRows;
  const int sms = num_sms();
  const int grid = int(tiles < sms ? tiles : sms);
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  if (nsrc == 3) return launch_mlp3_act<3>(tm, tw, g, grid, st);
  if (nsrc == 2) return launch_mlp3_act<2>(tm, tw, g, grid, st);
  return launch_mlp3_act<1>(tm, tw, g, grid, st);
}

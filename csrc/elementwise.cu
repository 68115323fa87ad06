// Elementwise kernels that have no producer to fuse into.
//
// pnm_silu_derivative: out = silu^(k)(x) [* g], k = 0..4, one pass, 16-byte vectors.  The k-th derivative is evaluated
// in closed form from s = sigmoid(x):  s' = s(1-s), s'' = s'(1-2s), s''' = s''(1-2s) - 2 s'^2,
// s'''' = s'''(1-2s) - 6 s' s'', and silu^(k) = k s^(k-1) + x s^(k).  Used for higher-order derivatives of
// physics-informed networks, where autograd would otherwise build a chain of ~10 elementwise launches per order.
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>
#include <type_traits>

#include "common.cuh"
#include "pnm_api.h"
#include "pnm_internal.h"

namespace pnm {

template <int K>
__device__ __forceinline__ float silu_d(float x) {
  const float s = 1.f / (1.f + __expf(-x));
  if (K == 0) return x * s;
  const float d1 = s * (1.f - s);
  if (K == 1) return s + x * d1;
  const float t = 1.f - 2.f * s;
  const float d2 = d1 * t;
  if (K == 2) return 2.f * d1 + x * d2;
  const float d3 = d2 * t - 2.f * d1 * d1;
  if (K == 3) return 3.f * d2 + x * d3;
  const float d4 = d3 * t - 6.f * d1 * d2;
  return 4.f * d3 + x * d4;
}

template <typename T> struct EVec;
template <> struct EVec<float> {
  static constexpr int N = 4;
  static __device__ __forceinline__ void load(const float* p, float* f) {
    const float4 u = *reinterpret_cast<const float4*>(p); f[0] = u.x; f[1] = u.y; f[2] = u.z; f[3] = u.w;
  }
  static __device__ __forceinline__ void store(float* p, const float* f) { *reinterpret_cast<float4*>(p) = make_float4(f[0], f[1], f[2], f[3]); }
  static __device__ __forceinline__ float get(const float* p) { return *p; }
  static __device__ __forceinline__ void put(float* p, float v) { *p = v; }
};
template <> struct EVec<__nv_bfloat16> {
  static constexpr int N = 8;
  static __device__ __forceinline__ void load(const __nv_bfloat16* p, float* f) {
    const uint4 u = *reinterpret_cast<const uint4*>(p);
    const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&u);
#pragma unroll
    for (int i = 0; i < 4; ++i) { const float2 v = __bfloat1622float2(h[i]); f[2 * i] = v.x; f[2 * i + 1] = v.y; }
  }
  static __device__ __forceinline__ void store(__nv_bfloat16* p, const float* f) {
    uint4 u;
    __nv_bfloat162* h = reinterpret_cast<__nv_bfloat162*>(&u);
#pragma unroll
    for (int i = 0; i < 4; ++i) h[i] = __floats2bfloat162_rn(f[2 * i], f[2 * i + 1]);
    *reinterpret_cast<uint4*>(p) = u;
  }
  static __device__ __forceinline__ float get(const __nv_bfloat16* p) { return __bfloat162float(*p); }
  static __device__ __forceinline__ void put(__nv_bfloat16* p, float v) { *p = __float2bfloat16(v); }
};

template <typename T, int K>
__global__ void __launch_bounds__(256) silu_derivative_kernel(const T* __restrict__ x, const T* __restrict__ g, T* __restrict__ out,
                                                               long long n) {
  constexpr int V = EVec<T>::N;
  const long long nvec = n / V, stride = (long long)gridDim.x * blockDim.x;
  float f[V], m[V];
  for (long long v = blockIdx.x * (long long)blockDim.x + threadIdx.x; v < nvec; v += stride) {
    EVec<T>::load(x + v * V, f);
    if (g) EVec<T>::load(g + v * V, m);
#pragma unroll
    for (int i = 0; i < V; ++i) f[i] = silu_d<K>(f[i]) * (g ? m[i] : 1.f);
    EVec<T>::store(out + v * V, f);
  }
  // ragged tail (n not a multiple of the vector width)
  for (long long i = nvec * V + blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += stride)
    EVec<T>::put(out + i, silu_d<K>(EVec<T>::get(x + i)) * (g ? EVec<T>::get(g + i) : 1.f));
}

template <typename T>
int launch_silu(const void* x, const void* g, void* out, long long n, int order, cudaStream_t st) {
  const T* xi = static_cast<const T*>(x);
  const T* gi = static_cast<const T*>(g);
  T* o = static_cast<T*>(out);
  const long long nvec = n / EVec<T>::N + 1;
  const unsigned grid = (unsigned)min((long long)148 * 16, (nvec + 255) / 256);
  switch (order) {
    case 0: silu_derivative_kernel<T, 0><<<grid, 256, 0, st>>>(xi, gi, o, n); break;
    case 1: silu_derivative_kernel<T, 1><<<grid, 256, 0, st>>>(xi, gi, o, n); break;
    case 2: silu_derivative_kernel<T, 2><<<grid, 256, 0, st>>>(xi, gi, o, n); break;
    case 3: silu_derivative_kernel<T, 3><<<grid, 256, 0, st>>>(xi, gi, o, n); break;
    case 4: silu_derivative_kernel<T, 4><<<grid, 256, 0, st>>>(xi, gi, o, n); break;
    default: return -1;
  }
  return (int)cudaGetLastError();
}

}  // namespace pnm

extern "C" int pnm_silu_derivative(const void* x, const void* g, void* out, long long n, int order, int dtype, void* stream) {
  if (n <= 0) return 0;
  if ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(out) | reinterpret_cast<uintptr_t>(g)) & 15) return -2;
  cudaStream_t st = (cudaStream_t)stream;
  return dtype == 0 ? pnm::launch_silu<__nv_bfloat16>(x, g, out, n, order, st) : pnm::launch_silu<float>(x, g, out, n, order, st);
}

// ---------------------------------------------------------------------------------------------------------------------
// EDM noise conditioning in one launch: sinusoidal embedding of the noise level (sin half first, then cos half: the
// "swapped" order the U-Net uses), optional additive term (class / augmentation embedding), then two Linear + SiLU
// layers.  out[b, :] = silu(W1 silu(W0 (emb(noise[b]) + extra[b]) + b0) + b1).
//
// One CTA per batch row.  A warp owns one output channel at a time: its lanes stride over the input channels (coalesced
// reads of one weight row) and reduce by shuffles; the hidden vector lives in shared memory between the two layers.  The
// weights (fp32 or bf16) are a megabyte or two and stay in L2 across the CTAs.
namespace pnm {

template <typename T> __device__ __forceinline__ float cond_ld(const T* p);
template <> __device__ __forceinline__ float cond_ld<float>(const float* p) { return *p; }
template <> __device__ __forceinline__ float cond_ld<__nv_bfloat16>(const __nv_bfloat16* p) { return __bfloat162float(*p); }

template <typename T>
__global__ void __launch_bounds__(512) edm_conditioning_kernel(const float* __restrict__ noise, const float* __restrict__ freqs,
                                                               const float* __restrict__ extra, const T* __restrict__ w0,
                                                               const T* __restrict__ b0, const T* __restrict__ w1,
                                                               const T* __restrict__ b1, float* __restrict__ out, int C, int E) {
  extern __shared__ float cond_smem[];
  float* emb = cond_smem;      // [C]
  float* hid = cond_smem + C;  // [E]
  const int b = blockIdx.x, half = C / 2;
  const float sigma = noise[b];
  for (int c = threadIdx.x; c < C; c += blockDim.x) {
    const float a = sigma * freqs[c < half ? c : c - half];
    float v = c < half ? sinf(a) : cosf(a);
    if (extra) v += extra[(size_t)b * C + c];
    emb[c] = v;
  }
  __syncthreads();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nwarps = blockDim.x >> 5;
  for (int e = warp; e < E; e += nwarps) {
    const T* row = w0 + (size_t)e * C;
    float acc = 0.f;
    for (int c = lane; c < C; c += 32) acc = fmaf(cond_ld(row + c), emb[c], acc);
    for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
    if (lane == 0) {
      const float z = acc + (b0 ? cond_ld(b0 + e) : 0.f);
      hid[e] = z / (1.f + __expf(-z));
    }
  }
  __syncthreads();
  for (int e = warp; e < E; e += nwarps) {
    const T* row = w1 + (size_t)e * E;
    float acc = 0.f;
    for (int c = lane; c < E; c += 32) acc = fmaf(cond_ld(row + c), hid[c], acc);
    for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
    if (lane == 0) {
      const float z = acc + (b1 ? cond_ld(b1 + e) : 0.f);
      out[(size_t)b * E + e] = z / (1.f + __expf(-z));
    }
  }
}

}  // namespace pnm

extern "C" int pnm_edm_conditioning(const float* noise, const float* freqs, const float* extra, const void* w0, const void* b0,
                                    const void* w1, const void* b1, float* out, int B, int C, int E, int weight_dtype,
                                    void* stream) {
  if (!noise || !freqs || !w0 || !w1 || !out || B <= 0 || C <= 0 || (C & 1) || E <= 0) return -1;
  const size_t smem = size_t(C + E) * sizeof(float);
  if (smem > 48 * 1024) return -1;
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  if (weight_dtype == 1) {
    pnm::edm_conditioning_kernel<float><<<B, 512, smem, st>>>(noise, freqs, extra, (const float*)w0, (const float*)b0, (const float*)w1,
                                                             (const float*)b1, out, C, E);
  } else if (weight_dtype == 0) {
    using bf = __nv_bfloat16;
    pnm::edm_conditioning_kernel<bf><<<B, 512, smem, st>>>(noise, freqs, extra, (const bf*)w0, (const bf*)b0, (const bf*)w1, (const bf*)b1,
                                                          out, C, E);
  } else {
    return -1;
  }
  return cudaGetLastError() == cudaSuccess ? 0 : -4;
}

// out = (a + b) * scale on bf16 tensors of n elements (n % 8 == 0, 16-byte aligned): the residual join of the diffusion
// U-Net blocks, one pass instead of an add and a multiply.  b may be null (out = a * scale).
namespace pnm {
__global__ void __launch_bounds__(256) add_scale_bf16_kernel(const uint4* __restrict__ a, const uint4* __restrict__ b, uint4* __restrict__ out,
                                                             long long nvec, float scale) {
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < nvec; i += (long long)gridDim.x * blockDim.x) {
    const uint4 ua = a[i];
    const uint32_t wa[4] = {ua.x, ua.y, ua.z, ua.w};
    uint32_t wo[4];
    if (b) {
      const uint4 ub = b[i];
      const uint32_t wb[4] = {ub.x, ub.y, ub.z, ub.w};
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const float2 x = unpack_bf16x2(wa[k]), y = unpack_bf16x2(wb[k]);
        wo[k] = pack_bf16x2((x.x + y.x) * scale, (x.y + y.y) * scale);
      }
    } else {
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const float2 x = unpack_bf16x2(wa[k]);
        wo[k] = pack_bf16x2(x.x * scale, x.y * scale);
      }
    }
    out[i] = make_uint4(wo[0], wo[1], wo[2], wo[3]);
  }
}
}  // namespace pnm

extern "C" int pnm_add_scale_bf16(const void* a, const void* b, void* out, long long n, float scale, void* stream) {
  if (!a || !out || n <= 0 || (n & 7)) return -2;
  const long long nvec = n >> 3;
  const long long blocks = (nvec + 255) / 256;
  pnm::add_scale_bf16_kernel<<<(unsigned)(blocks < 148 * 16 ? blocks : 148 * 16), 256, 0, (cudaStream_t)stream>>>(
      (const uint4*)a, (const uint4*)b, (uint4*)out, nvec, scale);
  return cudaGetLastError() == cudaSuccess ? 0 : -3;
}

// ------------------------------------------------------------------------------------------------ convolution weights
namespace pnm {

// w [cout, cin, k, k] (fp32 or bf16) -> out [rows_p, k * k, cols_p] bf16, tap-major and zero-padded: rows are output channels, or,
// with `flip`, input channels of the mirrored filter (the operand of the input gradient).  Tensor operations take a padded,
// permuted copy, a cast and, for the gradient, two flips: up to four launches per use of a weight that is a few hundred KB.  A
// block moves RT rows x 64 columns through shared memory: both sides are read and written in runs.
// KK = 0: any filter size; 1 and 9 are compiled in (the index arithmetic is most of the kernel's instructions).
template <typename T, int KK>
__global__ void __launch_bounds__(256) conv_pack_weight_kernel(const T* __restrict__ w, __nv_bfloat16* __restrict__ out, int cout, int cin,
                                                               int kk_any, int rows_p, int cols_p, int flip, int rt_any) {
  extern __shared__ float cw[];                  // [rt][64][kk]
  const int kk = KK ? KK : kk_any, rt = KK ? 8 : rt_any;
  const int r0 = blockIdx.x * rt, c0 = blockIdx.y * 64;
  const int rows = flip ? cin : cout, cols = flip ? cout : cin;
  const int n = rt * 64 * kk;
#pragma unroll 6
  for (int i = threadIdx.x; i < n; i += 256) {
    int r, c, t;                                 // the fastest index is the one that is contiguous in w
    t = i % kk;
    if (flip) { r = (i / kk) % rt; c = i / (kk * rt); }
    else { c = (i / kk) % 64; r = i / (kk * 64); }
    const int R = r0 + r, C = c0 + c;
    float v = 0.f;
    if (R < rows && C < cols) v = static_cast<float>(w[((size_t)(flip ? C : R) * cin + (flip ? R : C)) * kk + t]);
    cw[(r * 64 + c) * kk + (flip ? kk - 1 - t : t)] = v;
  }
  __syncthreads();
  for (int i = threadIdx.x; i < n; i += 256) {
    const int c = i % 64, t = (i / 64) % kk, r = i / (64 * kk);
    if (r0 + r < rows_p && c0 + c < cols_p)
      out[((size_t)(r0 + r) * kk + t) * cols_p + c0 + c] = __float2bfloat16(cw[(r * 64 + c) * kk + t]);
  }
}

// The same for 3 x 3 filters in fp32 whose rows of nine start on 16-byte boundaries every four channels: 4 rows x 64 columns per block, read by
// 16-byte vectors as they lie in w and written eight channels at a time, so that a thread has two or three accesses of either kind, all under
// way together.  (Element by element a thread went through 18 loads in three rounds and 18 stores of 2 bytes.  Event to event, of
// which 8 us are the two events': 512 x 512 channels 20.5 -> 10.2 us, 512 x 1024 34.8 -> 12.3, 128 x 256 18.4 -> 8.2.)
constexpr int kPack3Rows = 4, kPack3Run = kPack3Rows * 9;
template <bool FLIP>
__global__ void __launch_bounds__(256) conv_pack3_kernel(const float* __restrict__ w, __nv_bfloat16* __restrict__ out, int cout, int cin, int rows_p,
                                                         int cols_p) {
  constexpr int kLd = FLIP ? kPack3Run + 1 : 64 * 9 + 1;         // runs of w that are contiguous: one per column / per row
  constexpr int kRuns = FLIP ? 64 : kPack3Rows, kVecs = (FLIP ? kPack3Run : 64 * 9) / 4;
  __shared__ float cw[kRuns * kLd];
  const int r0 = blockIdx.x * kPack3Rows, c0 = blockIdx.y * 64;
  const int rows = FLIP ? cin : cout, cols = FLIP ? cout : cin;
  // channels of a run that exist
  const int inside = FLIP ? min(rows - r0, kPack3Rows) : min(cols - c0, 64), runs = FLIP ? min(cols - c0, 64) : min(rows - r0, kPack3Rows);
#pragma unroll 3
  for (int i = threadIdx.x; i < kRuns * kVecs; i += 256) {
    const int run = i / kVecs, v = i - run * kVecs;
    float4 x = make_float4(0.f, 0.f, 0.f, 0.f);
    // cin is a multiple of 4, and so is `inside` where it is one of cin's ends: a vector is inside or outside as a whole
    if (run < runs && 4 * v < inside * 9) x = __ldg(reinterpret_cast<const float4*>(w + ((size_t)(FLIP ? c0 + run : r0 + run) * cin + (FLIP ? r0 : c0)) * 9) + v);
    float* dst = cw + run * kLd + 4 * v;
    dst[0] = x.x; dst[1] = x.y; dst[2] = x.z; dst[3] = x.w;
  }
  __syncthreads();
#pragma unroll 2
  for (int i = threadIdx.x; i < kPack3Rows * 9 * 8; i += 256) {
    const int c = (i & 7) * 8, t = (i >> 3) % 9, r = (i >> 3) / 9;
    if (r0 + r >= rows_p || c0 + c >= cols_p) continue;
    uint32_t u[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      float x[2];
#pragma unroll
      for (int e = 0; e < 2; ++e) x[e] = FLIP ? cw[(c + 2 * q + e) * kLd + r * 9 + 8 - t] : cw[r * kLd + (c + 2 * q + e) * 9 + t];
      u[q] = pack_bf16x2(x[0], x[1]);
    }
    *reinterpret_cast<uint4*>(out + ((size_t)(r0 + r) * 9 + t) * cols_p + c0 + c) = make_uint4(u[0], u[1], u[2], u[3]);
  }
}

}  // namespace pnm

extern "C" int pnm_conv_pack_weight(const void* w, int is_bf16, void* out, int cout, int cin, int ksize, int rows_p, int cols_p, int flip,
                                    void* stream) {
  const int kk = ksize * ksize;
  if (cout <= 0 || cin <= 0 || ksize < 1 || ksize > 7 || rows_p < (flip ? cin : cout) || cols_p < (flip ? cout : cin)) return -2;
  if (kk == 9 && !is_bf16 && cin % 4 == 0 && cols_p % 8 == 0 && !((reinterpret_cast<uintptr_t>(w) | reinterpret_cast<uintptr_t>(out)) & 15)) {
    const dim3 blocks((rows_p + pnm::kPack3Rows - 1) / pnm::kPack3Rows, (cols_p + 63) / 64);
    cudaStream_t str = reinterpret_cast<cudaStream_t>(stream);
    const float* src = reinterpret_cast<const float*>(w);
    __nv_bfloat16* dst = reinterpret_cast<__nv_bfloat16*>(out);
    if (flip) pnm::conv_pack3_kernel<true><<<blocks, 256, 0, str>>>(src, dst, cout, cin, rows_p, cols_p);
    else pnm::conv_pack3_kernel<false><<<blocks, 256, 0, str>>>(src, dst, cout, cin, rows_p, cols_p);
    return cudaGetLastError() == cudaSuccess ? 0 : -17;
  }
  const int rt = kk <= 9 ? 8 : 1;                // 64 columns of an 8-row tile of a 3 x 3 filter: 18 KB
  const dim3 grid((rows_p + rt - 1) / rt, (cols_p + 63) / 64);
  const size_t smem = (size_t)rt * 64 * kk * sizeof(float);
  cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
  __nv_bfloat16* o = reinterpret_cast<__nv_bfloat16*>(out);
  const auto launch = [&](auto* src) {
    using T = std::remove_const_t<std::remove_pointer_t<decltype(src)>>;
    if (kk == 9) pnm::conv_pack_weight_kernel<T, 9><<<grid, 256, smem, st>>>(src, o, cout, cin, kk, rows_p, cols_p, flip, rt);
    else if (kk == 1) pnm::conv_pack_weight_kernel<T, 1><<<grid, 256, smem, st>>>(src, o, cout, cin, kk, rows_p, cols_p, flip, rt);
    else pnm::conv_pack_weight_kernel<T, 0><<<grid, 256, smem, st>>>(src, o, cout, cin, kk, rows_p, cols_p, flip, rt);
  };
  if (is_bf16) launch(reinterpret_cast<const __nv_bfloat16*>(w));
  else launch(reinterpret_cast<const float*>(w));
  return cudaGetLastError() == cudaSuccess ? 0 : -17;
}

// ------------------------------------------------------------------------------------- per-image channel vectors (channels-last)
namespace pnm {

// y[b, p, c] = x[b, p, c] + v[b, c]: the injection of an embedding into a feature map.  As a broadcast tensor addition on a
// channels-last map this ran at a quarter of the copy rate, and its gradient (the sum over the pixels) at a tenth: 512 x 512 x 128
// 79 -> 22 us and 182 -> 32 us.
__global__ void __launch_bounds__(256) add_channel_kernel(const uint4* __restrict__ x, const uint4* __restrict__ v, uint4* __restrict__ y,
                                                          long long per_image, int tpp, long long nvec) {
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < nvec; i += (long long)gridDim.x * blockDim.x) {
    const long long b = i / per_image;
    const uint4 a = x[i], s = __ldg(v + b * tpp + i % tpp);
    const uint32_t wa[4] = {a.x, a.y, a.z, a.w}, ws[4] = {s.x, s.y, s.z, s.w};
    uint32_t wo[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const float2 p = unpack_bf16x2(wa[k]), q = unpack_bf16x2(ws[k]);
      wo[k] = pack_bf16x2(p.x + q.x, p.y + q.y);
    }
    y[i] = make_uint4(wo[0], wo[1], wo[2], wo[3]);
  }
}

// part[b][s][c] = sum of g[b, p, c] over the pixels of slice s; grid (S, B).  A thread owns 8 channels of every ppi-th pixel.
__global__ void __launch_bounds__(256) channel_sum_kernel(const uint4* __restrict__ g, float* __restrict__ part, long long hw, int C) {
  __shared__ float stage[256 * 8];
  const int tpp = C / 8, ppi = 256 / tpp, chunk = threadIdx.x % tpp, lane = threadIdx.x / tpp;
  const bool active = (int)threadIdx.x < tpp * ppi;
  const long long per = (hw + gridDim.x - 1) / gridDim.x, p0 = blockIdx.x * per, p1 = p0 + per < hw ? p0 + per : hw;
  float a[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
  if (active) {
    const uint4* base = g + (long long)blockIdx.y * hw * tpp + chunk;
#pragma unroll 4
    for (long long p = p0 + lane; p < p1; p += ppi) {
      const uint4 u = base[p * tpp];
      const uint32_t w[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
      for (int k = 0; k < 4; ++k) { const float2 f = unpack_bf16x2(w[k]); a[2 * k] += f.x; a[2 * k + 1] += f.y; }
    }
  }
#pragma unroll
  for (int k = 0; k < 8; ++k) stage[threadIdx.x * 8 + k] = a[k];
  __syncthreads();
  for (int c = threadIdx.x; c < C; c += 256) {
    float s = 0.f;
    for (int l = 0; l < ppi; ++l) s += stage[l * C + c];
    part[((long long)blockIdx.y * gridDim.x + blockIdx.x) * C + c] = s;
  }
}

// out[b][c] = sum over the slices, bf16; grid (ceil(C / 32), B), block (32, 8)
__global__ void __launch_bounds__(256) channel_fold_kernel(const float* __restrict__ part, __nv_bfloat16* __restrict__ out, int S, int C) {
  __shared__ float red[8][32];
  const int c = blockIdx.x * 32 + threadIdx.x;
  float s = 0.f;
  if (c < C)
    for (int k = threadIdx.y; k < S; k += 8) s += part[((long long)blockIdx.y * S + k) * C + c];
  red[threadIdx.y][threadIdx.x] = s;
  __syncthreads();
  if (threadIdx.y == 0 && c < C) {
    for (int k = 1; k < 8; ++k) s += red[k][threadIdx.x];
    out[(long long)blockIdx.y * C + c] = __float2bfloat16(s);
  }
}

}  // namespace pnm

extern "C" int pnm_add_channel_bf16(const void* x, const void* v, void* y, int B, long long hw, int C, void* stream) {
  if (B <= 0 || hw <= 0 || C <= 0 || (C & 7)) return -2;
  const long long nvec = (long long)B * hw * (C / 8), blocks = (nvec + 255) / 256;
  const long long most = (long long)pnm::num_sms() * 16;
  if (most <= 0) return -1;
  pnm::add_channel_kernel<<<(unsigned)(blocks < most ? blocks : most), 256, 0, (cudaStream_t)stream>>>(
      (const uint4*)x, (const uint4*)v, (uint4*)y, hw * (C / 8), C / 8, nvec);
  return cudaGetLastError() == cudaSuccess ? 0 : -3;
}

// part: at least B * slices * C floats
extern "C" int pnm_channel_sum_bf16(const void* g, void* out, float* part, int B, long long hw, int C, int slices, void* stream) {
  if (B <= 0 || B > 65535 || hw <= 0 || C <= 0 || (C & 7) || C > 2048 || slices <= 0) return -2;
  cudaStream_t st = (cudaStream_t)stream;
  pnm::channel_sum_kernel<<<dim3(slices, B), 256, 0, st>>>((const uint4*)g, part, hw, C);
  pnm::channel_fold_kernel<<<dim3((C + 31) / 32, B), dim3(32, 8), 0, st>>>(part, (__nv_bfloat16*)out, slices, C);
  return cudaGetLastError() == cudaSuccess ? 0 : -3;
}

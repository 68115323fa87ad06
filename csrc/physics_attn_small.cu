// The small (parameter- and slice-token-sized) algebra of the fused Transolver physics attention, forward and backward,
// as four kernels.  The large passes over the N points are tcgen05 GEMMs (gemm_tn / gemm_nt); what is left per block is
// a chain of ~130 tiny tensor operations on matrices of at most 512 x 512 values, whose launch overhead does not shrink
// when the points are sharded.  Notation: H heads, S = 64 slices, D = head width, inner = H * D, C = channels of x.
//
//   pa_prepare_fwd   Wc = blockdiag_H(Ws) Wx (bf16), bc, 1 / clamp(T), bf16 copy of Wfx, Wback = [Wc^T | Wfx^T] (bf16)
//   pa_tokens_fwd    slice tokens (sum over ranks by peer loads in the prologue) -> normalise -> q k v -> 64 x 64
//                    attention per head -> Wcomb = Wo blockdiag(out_tokens)^T (bf16 + fp32)
//   pa_tokens_bwd    dWcomb (sum over ranks in the prologue) -> d out_tokens, dWo -> attention backward -> d tokens,
//                    dWqkv -> the operands of the point-sized backward GEMMs: Bcat = [Wcomb^T | blockdiag(d_tok)],
//                    BdT = blockdiag(d_tok)^T (bf16), d_norm
//   pa_prepare_bwd   dWx, dbx, dWs, dbs, dT from dWc, dbc and the per-head temperature sums; dWfx, dbfx out of the rows behind dWc, dbc
//
// Cross-rank sums: the producers (gemm_nt) write into a region of this rank's symmetric buffer, a signal kernel raises
// the flags, and the token kernels add the P copies with direct peer loads after a bounded wait -- there is no
// stand-alone all-reduce.  With world == 1 the source is an ordinary local buffer and no flag is touched.
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include <type_traits>

#include "pnm_api.h"
#include "pnm_internal.h"

namespace pnm {

constexpr int kPaS = 64;
constexpr int kPaMaxD = 64;
constexpr int kPaTokenThreads = 512;    // 4 x 4 outputs per thread: a product of a head has 128 to 384 tiles

struct PaSrc {
  const float* p[kPeerMaxRanks];  // per rank: base of the partial-sum matrix (peer-mapped for r != rank)
  int world;
  int use_flags;                  // wait for the ranks' "small" flags of the call before reading
};

__device__ __forceinline__ float pa_sum(const PaSrc& s, long long i) {
  float a = 0.f;
  for (int r = 0; r < s.world; ++r) a += __ldcg(s.p[r] + i);
  return a;
}

__device__ __forceinline__ bool pa_wait(const PaSrc& s, const PeerArgs& peer, int* err, int* sh_ok) {
  if (!s.use_flags) return true;
  return peer_small_wait(peer, peer_epoch(peer), err, sh_ok);
}

// grid H*S + inner, 256 threads
__global__ void __launch_bounds__(256)
pa_prepare_fwd_kernel(const float* __restrict__ Wx, const float* __restrict__ bx, const float* __restrict__ Wfx,
                      const float* __restrict__ Ws, const float* __restrict__ bs, const float* __restrict__ temp,
                      __nv_bfloat16* __restrict__ Wc, float* __restrict__ bc, float* __restrict__ inv_t,
                      __nv_bfloat16* __restrict__ Wfx16, __nv_bfloat16* __restrict__ Wback, int H, int D, int C) {
  __shared__ float ws[kPaMaxD];
  const int HS = H * kPaS, inner = H * D, ldb = HS + inner;
  const int r = blockIdx.x;
  if (r < HS) {
    const int h = r / kPaS, s = r % kPaS;
    if (threadIdx.x < D) ws[threadIdx.x] = Ws[s * D + threadIdx.x];
    __syncthreads();
    for (int c = threadIdx.x; c < C; c += blockDim.x) {
      float acc = 0.f;
      for (int d = 0; d < D; ++d) acc += ws[d] * Wx[(size_t)(h * D + d) * C + c];
      const __nv_bfloat16 v = __float2bfloat16(acc);
      Wc[(size_t)r * C + c] = v;
      Wback[(size_t)c * ldb + r] = v;
    }
    if (threadIdx.x == 0) {
      float acc = bs[s];
      for (int d = 0; d < D; ++d) acc += ws[d] * bx[h * D + d];
      bc[r] = acc;
      inv_t[r] = 1.f / fminf(fmaxf(temp[h], 0.5f), 5.f);
    }
  } else {
    const int j = r - HS;
    for (int c = threadIdx.x; c < C; c += blockDim.x) {
      const __nv_bfloat16 v = __float2bfloat16(Wfx[(size_t)j * C + c]);
      Wfx16[(size_t)j * C + c] = v;
      Wback[(size_t)c * ldb + HS + j] = v;
    }
  }
}

struct PaSaved {        // per block, fp32, all [H][S][...]
  float* token;         // [H][S][D]
  float* normp;         // [H][S]      norm + 0.01
  float* q; float* k; float* v;   // [H][S][D]
  float* prob;          // [H][S][S]
  float* out;           // [H][S][D]
  float* wcomb;         // [Cout][H*S]
};

// The token kernels: grid (H, slices).  Per head the work is a chain of products of 64 rows; every CTA of a head runs the chain and the
// CTAs share what hangs at its ends, the rows of Wo (forward: Wcomb; backward: dWo, Bcat, BdT) in chunks of 64.  What bounds a product is
// its reads of shared memory: with one output per thread two words per multiply-add (8 heads of width 32, Cout = 256: 43.5 us forward,
// 101 us backward on 8 CTAs), so a thread computes 4 x 4 outputs from 16-byte vectors, half a word per multiply-add or less, and a head
// has four CTAs: 17.7 / 44.3 us.  Every output is one sum in the order of k, as before, but for the sums along rows.
// With P ranks every CTA adds the P copies of its head's sums for itself, four times the peer reads of one CTA per head: backward, at the
// sizes above, (P - 1) x 2 MB per rank, by the link's 770 GB/s 2.7 us a peer (estimated; not measured on several GPUs).
constexpr int kPaChunk = 64;
constexpr int kPaLp = kPaS + 4;          // row length of S x S matrices: 16-byte vectors of eight rows fall on different banks

__device__ __forceinline__ float4 pa_ld4(const float* p) { return *reinterpret_cast<const float4*>(p); }
__device__ __forceinline__ void pa_fma4(float (&acc)[4], float a, const float4& b) {
  acc[0] = fmaf(a, b.x, acc[0]); acc[1] = fmaf(a, b.y, acc[1]); acc[2] = fmaf(a, b.z, acc[2]); acc[3] = fmaf(a, b.w, acc[3]);
}
// Tile t of out(i, j), i < I, j < J (multiples of 4, as is K):
//   nt  sum_k A[i][k] B[j][k]     rows i = ib + r I / 4, j = jb + c J / 4
//   nn  sum_k A[i][k] B[k][j]     rows i = ib + r I / 4, columns j = 4 jb + c
//   tn  sum_k A[k][i] B[k][j]     columns i = 4 ib + r, j = 4 jb + c
template <int I, int J, int K, int lda, int ldb>
__device__ __forceinline__ void pa_nt(float (&acc)[4][4], const float* A, const float* B, int t) {
  constexpr int ni = I >> 2, nj = J >> 2;
  const int ib = t / nj, jb = t - ib * nj;
  for (int k = 0; k < K; k += 4) {
    float4 a[4], b[4];
#pragma unroll
    for (int r = 0; r < 4; ++r) { a[r] = pa_ld4(A + (ib + r * ni) * lda + k); b[r] = pa_ld4(B + (jb + r * nj) * ldb + k); }
#pragma unroll
    for (int r = 0; r < 4; ++r)
#pragma unroll
      for (int c = 0; c < 4; ++c)
        acc[r][c] = fmaf(a[r].w, b[c].w, fmaf(a[r].z, b[c].z, fmaf(a[r].y, b[c].y, fmaf(a[r].x, b[c].x, acc[r][c]))));
  }
}
template <int I, int J, int K, int lda, int ldb>
__device__ __forceinline__ void pa_nn(float (&acc)[4][4], const float* A, const float* B, int t) {
  constexpr int ni = I >> 2, nj = J >> 2;
  const int ib = t / nj, jb = t - ib * nj;
  for (int k = 0; k < K; k += 4) {
    float4 a[4];
#pragma unroll
    for (int r = 0; r < 4; ++r) a[r] = pa_ld4(A + (ib + r * ni) * lda + k);
    const float4 b0 = pa_ld4(B + k * ldb + 4 * jb), b1 = pa_ld4(B + (k + 1) * ldb + 4 * jb), b2 = pa_ld4(B + (k + 2) * ldb + 4 * jb),
                 b3 = pa_ld4(B + (k + 3) * ldb + 4 * jb);
#pragma unroll
    for (int r = 0; r < 4; ++r) {
      pa_fma4(acc[r], a[r].x, b0); pa_fma4(acc[r], a[r].y, b1); pa_fma4(acc[r], a[r].z, b2); pa_fma4(acc[r], a[r].w, b3);
    }
  }
}
template <int J, int K, int lda, int ldb>
__device__ __forceinline__ void pa_tn(float (&acc)[4][4], const float* A, const float* B, int t) {
  constexpr int nj = J >> 2;
  const int ib = t / nj, jb = t - ib * nj;
#pragma unroll 4
  for (int k = 0; k < K; ++k) {
    const float4 a = pa_ld4(A + k * lda + 4 * ib), b = pa_ld4(B + k * ldb + 4 * jb);
    pa_fma4(acc[0], a.x, b); pa_fma4(acc[1], a.y, b); pa_fma4(acc[2], a.z, b); pa_fma4(acc[3], a.w, b);
  }
}
// f(i, j, value) for the outputs of a tile
template <int I, int J, class F>
__device__ __forceinline__ void pa_each_nt(const float (&acc)[4][4], int t, F f) {
  constexpr int ni = I >> 2, nj = J >> 2;
  const int ib = t / nj, jb = t - ib * nj;
#pragma unroll
  for (int r = 0; r < 4; ++r)
#pragma unroll
    for (int c = 0; c < 4; ++c) f(ib + r * ni, jb + c * nj, acc[r][c]);
}
template <int I, int J, class F>
__device__ __forceinline__ void pa_each_nn(const float (&acc)[4][4], int t, F f) {
  constexpr int ni = I >> 2, nj = J >> 2;
  const int ib = t / nj, jb = t - ib * nj;
#pragma unroll
  for (int r = 0; r < 4; ++r)
#pragma unroll
    for (int c = 0; c < 4; ++c) f(ib + r * ni, 4 * jb + c, acc[r][c]);
}
template <int J, class F>
__device__ __forceinline__ void pa_each_tn(const float (&acc)[4][4], int t, F f) {
  constexpr int nj = J >> 2;
  const int ib = t / nj, jb = t - ib * nj;
#pragma unroll
  for (int r = 0; r < 4; ++r)
#pragma unroll
    for (int c = 0; c < 4; ++c) f(4 * ib + r, 4 * jb + c, acc[r][c]);
}
__device__ __forceinline__ float pa_warp_sum(float v) {
#pragma unroll
  for (int x = 16; x > 0; x >>= 1) v += __shfl_xor_sync(0xffffffffu, v, x);
  return v;
}

template <int Dp>                        // padded head width: loops and indexes are the compiler's
__global__ void __launch_bounds__(kPaTokenThreads)
pa_tokens_fwd_kernel(PaSrc src, long long norm_off, int ld_tok, const float* __restrict__ Wqkv, const float* __restrict__ Wo,
                     __nv_bfloat16* __restrict__ wcomb16, PaSaved sv, int H, int D, int Cout, float scale, PeerArgs peer, int* err) {
  extern __shared__ __align__(16) float sm[];
  __shared__ int sh_ok;
  constexpr int S = kPaS, L = Dp + 4, nt = kPaTokenThreads;
  float* tok = sm;                 // [S][L]
  float* q = tok + S * L;          // q, k, v follow one another
  float* k = q + S * L;
  float* v = k + S * L;
  float* o = v + S * L;
  float* pr = o + S * L;           // [S][kPaLp]
  float* wq = pr + S * kPaLp;      // [3][Dp][L]
  float* wo = wq + 3 * Dp * L;     // [kPaChunk][L]  rows of Wo, this head's columns
  const int h = blockIdx.x, slice = blockIdx.y, slices = gridDim.y, tid = threadIdx.x;
  const int HS = H * S, inner = H * D;
  const bool ok = pa_wait(src, peer, err, &sh_ok), first = slice == 0;
  const float nanv = __int_as_float(0x7fc00000);
  auto load_wo = [&](int chunk) {
#pragma unroll 4
    for (int i = tid; i < kPaChunk * Dp; i += nt) {
      const int r = i / Dp, d = i - r * Dp, c = chunk * kPaChunk + r;
      wo[r * L + d] = c < Cout && d < D ? Wo[(size_t)c * inner + h * D + d] : 0.f;
    }
  };
#pragma unroll 6
  for (int i = tid; i < 3 * Dp * Dp; i += nt) {
    const int j = i / Dp, d = i - j * Dp, part = j / Dp, r = j - part * Dp;
    wq[j * L + d] = r < D && d < D ? Wqkv[(part * D + r) * D + d] : 0.f;
  }
  load_wo(slice);
#pragma unroll 4
  for (int i = tid; i < S * Dp; i += nt) {
    const int s = i / Dp, d = i - s * Dp;
    float tk = 0.f;
    if (d < D) {
      const float nrm = ok ? pa_sum(src, norm_off + h * S + s) + 1e-2f : nanv;
      tk = (ok ? pa_sum(src, (long long)(h * S + s) * ld_tok + h * D + d) : nanv) / nrm;
      if (first) sv.token[(size_t)(h * S + s) * D + d] = tk;
      if (first && d == 0) sv.normp[h * S + s] = nrm;
    }
    tok[s * L + d] = tk;
  }
  __syncthreads();
  for (int t = tid; t < S * 3 * Dp / 16; t += nt) {
    float acc[4][4] = {};
    pa_nt<S, 3 * Dp, Dp, L, L>(acc, tok, wq, t);
    pa_each_nt<S, 3 * Dp>(acc, t, [&](int s, int j, float x) {
      const int part = j / Dp, d = j - part * Dp;
      q[(part * S + s) * L + d] = x;
      if (first && d < D) (part == 0 ? sv.q : part == 1 ? sv.k : sv.v)[(size_t)(h * S + s) * D + d] = x;
    });
  }
  __syncthreads();
  for (int t = tid; t < S * S / 16; t += nt) {
    float acc[4][4] = {};
    pa_nt<S, S, Dp, L, L>(acc, q, k, t);
    pa_each_nt<S, S>(acc, t, [&](int s, int u, float x) { pr[s * kPaLp + u] = x * scale; });
  }
  __syncthreads();
  {  // softmax over t: one warp per row, two columns per lane
    const int warp = tid >> 5, lane = tid & 31, nw = nt >> 5;
    for (int s = warp; s < S; s += nw) {
      float a = pr[s * kPaLp + lane], b = pr[s * kPaLp + lane + 32];
      float m = fmaxf(a, b);
      for (int x = 16; x > 0; x >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, x));
      a = __expf(a - m); b = __expf(b - m);
      const float inv = 1.f / pa_warp_sum(a + b);
      pr[s * kPaLp + lane] = a * inv;
      pr[s * kPaLp + lane + 32] = b * inv;
      if (first) {
        sv.prob[(size_t)(h * S + s) * S + lane] = a * inv;
        sv.prob[(size_t)(h * S + s) * S + lane + 32] = b * inv;
      }
    }
  }
  __syncthreads();
  for (int t = tid; t < S * Dp / 16; t += nt) {
    float acc[4][4] = {};
    pa_nn<S, Dp, S, kPaLp, L>(acc, pr, v, t);
    pa_each_nn<S, Dp>(acc, t, [&](int s, int d, float x) {
      o[s * L + d] = x;
      if (first && d < D) sv.out[(size_t)(h * S + s) * D + d] = x;
    });
  }
  __syncthreads();
  for (int chunk = slice; chunk * kPaChunk < Cout; chunk += slices) {
    if (chunk != slice) {
      __syncthreads();
      load_wo(chunk);
      __syncthreads();
    }
    for (int t = tid; t < kPaChunk * S / 16; t += nt) {
      float acc[4][4] = {};
      pa_nt<kPaChunk, S, Dp, L, L>(acc, wo, o, t);
      pa_each_nt<kPaChunk, S>(acc, t, [&](int r, int s, float x) {
        const int c = chunk * kPaChunk + r;
        if (c < Cout) {
          wcomb16[(size_t)c * HS + h * S + s] = __float2bfloat16(x);
          sv.wcomb[(size_t)c * HS + h * S + s] = x;
        }
      });
    }
  }
}

// Heads wider than 32 would want 255 KB in the backward: there Wqkv, which is read after the last chunk of dWcomb and Wo and before the
// chunks of Wcomb, takes their place (221 KB).  4 heads of width 64, Cout = 256: 39 / 77 us event to event, 8 heads, Cout = 512: 43 / 108 us.
__host__ __device__ constexpr bool pa_bwd_shares(int Dp) { return Dp > 32; }
// floats of Wqkv and of a chunk of dWcomb and Wo
__host__ __device__ constexpr int pa_bwd_weights(int Dp) {
  const int wq = 3 * Dp * (Dp + 4), chunk = kPaChunk * (kPaLp + Dp + 4);
  return pa_bwd_shares(Dp) ? (wq > chunk ? wq : chunk) : wq + chunk;
}

template <int Dp>
__global__ void __launch_bounds__(kPaTokenThreads)
pa_tokens_bwd_kernel(PaSrc src, const float* __restrict__ Wqkv, const float* __restrict__ Wo, PaSaved sv,
                     float* __restrict__ dWo, float* __restrict__ dWqkv, float* __restrict__ d_norm,
                     __nv_bfloat16* __restrict__ Bcat, __nv_bfloat16* __restrict__ BdT, int H, int D, int Cout, float scale,
                     float share, PeerArgs peer, int* err) {
  extern __shared__ __align__(16) float sm[];
  __shared__ int sh_ok;
  constexpr int S = kPaS, L = Dp + 4, nt = kPaTokenThreads;
  float* q = sm;                   // [S][L] each
  float* k = q + S * L;
  float* v = k + S * L;
  float* tok = v + S * L;
  float* dq = tok + S * L;         // dq, dk, dv follow one another; the attention output until dq takes its place
  float* dk = dq + S * L;
  float* dv = dk + S * L;
  float* dout = dv + S * L;        // later: d token
  float* pr = dout + S * L;        // [S][kPaLp]
  float* ds = pr + S * kPaLp;
  float* wq = ds + S * kPaLp;      // [3][Dp][L]
  float* dwc = wq + (pa_bwd_shares(Dp) ? 0 : 3 * Dp * L);      // [kPaChunk][kPaLp]  rows of dWcomb, this head's columns; later: of Wcomb
  float* wo = dwc + kPaChunk * kPaLp;      // [kPaChunk][L]
  float* inv_np = ds + S * kPaLp + pa_bwd_weights(Dp);         // [S]
  const int h = blockIdx.x, slice = blockIdx.y, slices = gridDim.y, tid = threadIdx.x;
  const int warp = tid >> 5, lane = tid & 31, nw = nt >> 5;
  const int HS = H * S, inner = H * D, chunks = (Cout + kPaChunk - 1) / kPaChunk;
  const bool ok = pa_wait(src, peer, err, &sh_ok), first = slice == 0;
  const float nanv = __int_as_float(0x7fc00000);
  // the next chunk's values are on their way while this one is worked on
  constexpr int kPre = kPaChunk * kPaS / kPaTokenThreads;
  float pre[kPre], pre_o[kPre];
  auto fetch = [&](int chunk) {
#pragma unroll
    for (int n = 0; n < kPre; ++n) {
      const int i = tid + n * kPaTokenThreads, c = chunk * kPaChunk + i / S, r = i / Dp, d = i - r * Dp, co = chunk * kPaChunk + r;
      pre[n] = c >= Cout ? 0.f : ok ? pa_sum(src, (long long)c * HS + h * S + i % S) : nanv;
      pre_o[n] = r < kPaChunk && co < Cout && d < D ? Wo[(size_t)co * inner + h * D + d] : 0.f;
    }
  };
  fetch(0);
  auto load_wq = [&] {
#pragma unroll 6
    for (int i = tid; i < 3 * Dp * Dp; i += nt) {
      const int j = i / Dp, d = i - j * Dp, part = j / Dp, r = j - part * Dp;
      wq[j * L + d] = r < D && d < D ? Wqkv[(part * D + r) * D + d] : 0.f;
    }
  };
  if (!pa_bwd_shares(Dp)) load_wq();
#pragma unroll 4
  for (int i = tid; i < S * Dp; i += nt) {
    const int s = i / Dp, d = i - s * Dp, at = s * L + d;
    const size_t g = (size_t)(h * S + s) * D + d;
    const bool in = d < D;
    q[at] = in ? sv.q[g] : 0.f; k[at] = in ? sv.k[g] : 0.f; v[at] = in ? sv.v[g] : 0.f;
    tok[at] = in ? sv.token[g] : 0.f; dq[at] = in ? sv.out[g] : 0.f;
  }
#pragma unroll
  for (int i = tid; i < S * S; i += nt) pr[(i / S) * kPaLp + (i % S)] = sv.prob[(size_t)h * S * S + i];
  // d out_tokens[s][d] = sum_c dWcomb[c][s] Wo[c][h D + d];  dWo[c][h D + d] = sum_s dWcomb[c][s] out[s][d]
  constexpr int tiles_sd = S * Dp / 16;                                  // at most 256: one tile per thread
  float acc_o[4][4] = {};
  for (int chunk = 0; chunk < chunks; ++chunk) {
#pragma unroll
    for (int n = 0; n < kPre; ++n) {
      const int i = tid + n * kPaTokenThreads, r = i / Dp;
      dwc[(i / S) * kPaLp + i % S] = pre[n];
      if (r < kPaChunk) wo[r * L + i - r * Dp] = pre_o[n];
    }
    __syncthreads();
    if (chunk + 1 < chunks) fetch(chunk + 1);
    if (tid < tiles_sd) pa_tn<Dp, kPaChunk, kPaLp, L>(acc_o, dwc, wo, tid);
    if (chunk % slices == slice) {
      const int t = tid - (nt - kPaChunk * Dp / 16);                 // the last threads
      if (t >= 0) {
        float acc[4][4] = {};
        pa_nn<kPaChunk, Dp, S, kPaLp, L>(acc, dwc, dq, t);
        pa_each_nn<kPaChunk, Dp>(acc, t, [&](int r, int d, float x) {
          const int c = chunk * kPaChunk + r;
          if (c < Cout && d < D) dWo[(size_t)c * inner + h * D + d] = x * share;
        });
      }
    }
    __syncthreads();
  }
  if (pa_bwd_shares(Dp)) load_wq();                                      // the chunks are done with: all threads have met behind the last
  if (tid < tiles_sd) pa_each_tn<Dp>(acc_o, tid, [&](int s, int d, float x) { dout[s * L + d] = x; });
  __syncthreads();
  // dP = dout v^T ; dv = P^T dout
  for (int t = tid; t < S * S / 16 + tiles_sd; t += nt) {
    float acc[4][4] = {};
    if (t < S * S / 16) {
      pa_nt<S, S, Dp, L, L>(acc, dout, v, t);
      pa_each_nt<S, S>(acc, t, [&](int s, int u, float x) { ds[s * kPaLp + u] = x; });
    } else {
      pa_tn<Dp, S, kPaLp, L>(acc, pr, dout, t - S * S / 16);
      pa_each_tn<Dp>(acc, t - S * S / 16, [&](int u, int d, float x) { dv[u * L + d] = x; });
    }
  }
  __syncthreads();
  for (int s = warp; s < S; s += nw) {
    const float p0 = pr[s * kPaLp + lane], p1 = pr[s * kPaLp + lane + 32], g0 = ds[s * kPaLp + lane], g1 = ds[s * kPaLp + lane + 32];
    const float dot = pa_warp_sum(fmaf(g0, p0, g1 * p1));
    ds[s * kPaLp + lane] = p0 * (g0 - dot) * scale;
    ds[s * kPaLp + lane + 32] = p1 * (g1 - dot) * scale;
  }
  __syncthreads();
  // dq[s] = sum_t dS[s][t] k[t] ; dk[s] = sum_t dS[t][s] q[t]
  for (int t = tid; t < 2 * tiles_sd; t += nt) {
    float acc[4][4] = {};
    if (t < tiles_sd) {
      pa_nn<S, Dp, S, kPaLp, L>(acc, ds, k, t);
      pa_each_nn<S, Dp>(acc, t, [&](int s, int d, float x) { dq[s * L + d] = x; });
    } else {
      pa_tn<Dp, S, kPaLp, L>(acc, ds, q, t - tiles_sd);
      pa_each_tn<Dp>(acc, t - tiles_sd, [&](int s, int d, float x) { dk[s * L + d] = x; });
    }
  }
  __syncthreads();
  // d token[s][d] = sum_j dqkv[s][j] Wqkv[j][d] (in dout's place);  dWqkv[j][d] += share * sum_s dqkv[s][j] token[s][d]
  constexpr int tiles_w = Dp * Dp / 16;
  for (int t = tid; t < tiles_sd + (first ? 3 * tiles_w : 0); t += nt) {
    float acc[4][4] = {};
    if (t < tiles_sd) {
#pragma unroll 1
      for (int part = 0; part < 3; ++part) pa_nn<S, Dp, Dp, L, L>(acc, dq + part * S * L, wq + part * Dp * L, t);
      pa_each_nn<S, Dp>(acc, t, [&](int s, int d, float x) { dout[s * L + d] = x; });
    } else {
      const int part = (t - tiles_sd) / tiles_w, u = (t - tiles_sd) - part * tiles_w;
      pa_tn<Dp, S, L, L>(acc, dq + part * S * L, tok, u);
      pa_each_tn<Dp>(acc, u, [&](int j, int d, float x) {
        if (j < D && d < D) atomicAdd(dWqkv + (part * D + j) * D + d, x * share);
      });
    }
  }
  __syncthreads();
  for (int s = warp; s < S; s += nw) {
    float dot = lane < Dp ? dout[s * L + lane] * tok[s * L + lane] : 0.f;
    if (lane + 32 < Dp) dot = fmaf(dout[s * L + lane + 32], tok[s * L + lane + 32], dot);
    dot = pa_warp_sum(dot);
    const float np = sv.normp[h * S + s];
    if (lane == 0) {
      inv_np[s] = 1.f / np;
      if (first) d_norm[h * S + s] = -dot / np;
    }
  }
  __syncthreads();                         // also: Wqkv has been read where its memory is that of the chunks
  // Bcat rows h S + s: [Wcomb^T (Cout) | zeros ... d_tok[s][:] in block h ... zeros] ; BdT rows h D + d: d_tok[:, d] in block h
  const int ldc = Cout + inner;
  for (int chunk = slice; chunk < chunks; chunk += slices) {
#pragma unroll
    for (int i = tid; i < kPaChunk * S; i += nt) {
      const int c = chunk * kPaChunk + i / S;
      dwc[(i / S) * kPaLp + i % S] = c < Cout ? sv.wcomb[(size_t)c * HS + h * S + i % S] : 0.f;
    }
    __syncthreads();
#pragma unroll
    for (int i = tid; i < S * kPaChunk; i += nt) {
      const int s = i / kPaChunk, r = i % kPaChunk, c = chunk * kPaChunk + r;
      if (c < Cout) Bcat[(size_t)(h * S + s) * ldc + c] = __float2bfloat16(dwc[r * kPaLp + s]);
    }
    __syncthreads();
  }
  for (int s = slice; s < S; s += slices)
    for (int jd = tid; jd < inner; jd += nt)
      Bcat[(size_t)(h * S + s) * ldc + Cout + jd] = __float2bfloat16(jd / D == h ? dout[s * L + (jd % D)] * inv_np[s] : 0.f);
  for (int d = slice; d < D; d += slices)
    for (int col = tid; col < HS; col += nt)
      BdT[(size_t)(h * D + d) * HS + col] = __float2bfloat16(col / S == h ? dout[(col % S) * L + d] * inv_np[col % S] : 0.f);
}

// grid inner + S * D / 8 + 1, 256 threads
__global__ void __launch_bounds__(256)
pa_prepare_bwd_kernel(const float* __restrict__ dWc, const float* __restrict__ dbc, const float* __restrict__ grp,
                      const float* __restrict__ Wx, const float* __restrict__ bx, const float* __restrict__ Ws,
                      const float* __restrict__ temp, float* __restrict__ dWx, float* __restrict__ dbx, float* __restrict__ dWfx,
                      float* __restrict__ dbfx, float* __restrict__ dWs, float* __restrict__ dbs, float* __restrict__ dtemp, int H, int D, int C) {
  const int S = kPaS, inner = H * D, HS = H * S;
  const int b = blockIdx.x, tid = threadIdx.x;
  if (b < inner) {
    const int h = b / D, d = b % D;
    for (int c = tid; c < C; c += blockDim.x) {
      dWfx[(size_t)b * C + c] = dWc[(size_t)(HS + b) * C + c];
      float acc = 0.f;
      for (int s = 0; s < S; ++s) acc += Ws[s * D + d] * dWc[(size_t)(h * S + s) * C + c];
      dWx[(size_t)b * C + c] = acc;
    }
    if (tid == 0) {
      float acc = 0.f;
      for (int s = 0; s < S; ++s) acc += Ws[s * D + d] * dbc[h * S + s];
      dbx[b] = acc;
      dbfx[b] = dbc[HS + b];
    }
  } else if (b < inner + (S * D) / 8) {
    // dWs[s][d] = sum_h ( sum_c dWc[h S + s][c] Wx[h D + d][c] + dbc[h S + s] bx[h D + d] ): one warp per (s, d), lanes over c
    const int warp = tid >> 5, lane = tid & 31;
    const int e = (b - inner) * 8 + warp;
    const int s = e / D, d = e % D;
    float acc = 0.f;
    for (int h = 0; h < H; ++h) {
      const float* a = dWc + (size_t)(h * S + s) * C;
      const float* w = Wx + (size_t)(h * D + d) * C;
      for (int c = lane; c < C; c += 32) acc += a[c] * w[c];
    }
    for (int x = 16; x > 0; x >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, x);
    if (lane == 0) {
      float t = acc, bsum = 0.f;
      for (int h = 0; h < H; ++h) {
        t += dbc[h * S + s] * bx[h * D + d];
        bsum += dbc[h * S + s];
      }
      dWs[s * D + d] = t;
      if (d == 0) dbs[s] = bsum;
    }
  } else {
    for (int h = tid; h < H; h += blockDim.x) {
      const float T = temp[h];
      dtemp[h] = (T >= 0.5f && T <= 5.f) ? -grp[h] / T : 0.f;      // torch.clamp passes the gradient at its ends; 0.5 is the initial value
    }
  }
}

static constexpr size_t pa_fwd_smem(size_t Dp) {
  const size_t L = Dp + 4;
  return sizeof(float) * (5 * kPaS * L + kPaS * kPaLp + 3 * Dp * L + kPaChunk * L);
}
static constexpr size_t pa_bwd_smem(size_t Dp) {
  const size_t L = Dp + 4;
  return sizeof(float) * (8 * kPaS * L + 2 * kPaS * kPaLp + pa_bwd_weights(int(Dp)) + kPaS);
}
static_assert(pa_bwd_smem(kPaMaxD) <= 226 * 1024, "the widest head that is accepted fits");
// f(width) with the padded head width as a constant
template <class F>
static int pa_by_width(int D, F f) {
  if (D <= 4) return f(std::integral_constant<int, 4>{});
  if (D <= 8) return f(std::integral_constant<int, 8>{});
  if (D <= 16) return f(std::integral_constant<int, 16>{});
  if (D <= 32) return f(std::integral_constant<int, 32>{});
  return f(std::integral_constant<int, 64>{});
}
// CTAs per head: one per chunk of Wo's rows, four at most (each repeats the head's chain)
static int pa_slices(int Cout) {
  const int chunks = (Cout + kPaChunk - 1) / kPaChunk;
  return chunks < 4 ? chunks : 4;
}

static PaSrc make_src(const void* const* srcs, int world, int use_flags) {
  PaSrc s;
  for (int r = 0; r < kPeerMaxRanks; ++r) s.p[r] = r < world ? reinterpret_cast<const float*>(srcs[r]) : nullptr;
  s.world = world;
  s.use_flags = use_flags;
  return s;
}

static PaSaved make_saved(void* const* p) {
  PaSaved s;
  s.token = (float*)p[0]; s.normp = (float*)p[1]; s.q = (float*)p[2]; s.k = (float*)p[3]; s.v = (float*)p[4];
  s.prob = (float*)p[5]; s.out = (float*)p[6]; s.wcomb = (float*)p[7];
  return s;
}

}  // namespace pnm

extern "C" {

int pnm_pa_prepare_fwd(const float* Wx, const float* bx, const float* Wfx, const float* Ws, const float* bs, const float* temp,
                       void* Wc16, float* bc, float* inv_t, void* Wfx16, void* Wback16, int H, int D, int C, void* stream) {
  if (H <= 0 || D <= 0 || D > pnm::kPaMaxD || C <= 0) return -2;
  pnm::pa_prepare_fwd_kernel<<<H * pnm::kPaS + H * D, 256, 0, (cudaStream_t)stream>>>(
      Wx, bx, Wfx, Ws, bs, temp, (__nv_bfloat16*)Wc16, bc, inv_t, (__nv_bfloat16*)Wfx16, (__nv_bfloat16*)Wback16, H, D, C);
  return cudaGetLastError() == cudaSuccess ? 0 : -3;
}

// srcs: host array of `world` pointers to the [H*S, ld_tok] token-sum matrices (own first ... in rank order), whose
// element norm_off + h*S + s holds the slice norms.  saved: host array of 8 device pointers (token, normp, q, k, v,
// prob, out, wcomb).  use_flags != 0: wait for the peers' flags of call `epoch` (peer arguments as in pnm_peer_allreduce).
int pnm_pa_tokens_fwd(const void* const* srcs, int world, int use_flags, long long norm_off, int ld_tok, const float* Wqkv,
                      const float* Wo, void* wcomb16, void* const* saved, int H, int D, int Cout, float scale,
                      const void* const* bases, int rank, unsigned int epoch, long long capacity_floats, double budget_s,
                      const void* epoch_base, void* stream) {
  if (H <= 0 || D <= 0 || D > pnm::kPaMaxD || Cout <= 0 || world < 1 || world > pnm::kPeerMaxRanks) return -2;
  int* err = pnm::error_word_ptr();
  if (!err) return -1;
  pnm::PeerArgs p{};
  if (use_flags) p = pnm::make_peer_args(bases, rank, world, epoch, capacity_floats, budget_s, epoch_base);
  auto launch = [&](auto width) {
    constexpr int Dp = decltype(width)::value;
    constexpr size_t smem = pnm::pa_fwd_smem(Dp);
    static pnm::DeviceMask smem_set{0};
    if (!pnm::allow_smem(pnm::pa_tokens_fwd_kernel<Dp>, smem, smem_set)) return -4;
    pnm::pa_tokens_fwd_kernel<Dp><<<dim3(H, pnm::pa_slices(Cout)), pnm::kPaTokenThreads, smem, (cudaStream_t)stream>>>(
        pnm::make_src(srcs, world, use_flags), norm_off, ld_tok, Wqkv, Wo, (__nv_bfloat16*)wcomb16, pnm::make_saved(saved), H, D, Cout, scale, p, err);
    return 0;
  };
  const int code = pnm::pa_by_width(D, launch);
  if (code) return code;
  return cudaGetLastError() == cudaSuccess ? 0 : -3;
}

// srcs: per rank the [Cout, H*S] matrix dWcomb (partial sums).  dWqkv must be zero on entry (accumulated with atomics).
int pnm_pa_tokens_bwd(const void* const* srcs, int world, int use_flags, const float* Wqkv, const float* Wo, void* const* saved,
                      float* dWo, float* dWqkv, float* d_norm, void* Bcat16, void* BdT16, int H, int D, int Cout, float scale,
                      float share, const void* const* bases, int rank, unsigned int epoch, long long capacity_floats,
                      double budget_s, const void* epoch_base, void* stream) {
  if (H <= 0 || D <= 0 || D > pnm::kPaMaxD || Cout <= 0 || world < 1 || world > pnm::kPeerMaxRanks) return -2;
  int* err = pnm::error_word_ptr();
  if (!err) return -1;
  pnm::PeerArgs p{};
  if (use_flags) p = pnm::make_peer_args(bases, rank, world, epoch, capacity_floats, budget_s, epoch_base);
  auto launch = [&](auto width) {
    constexpr int Dp = decltype(width)::value;
    constexpr size_t smem = pnm::pa_bwd_smem(Dp);
    static pnm::DeviceMask smem_set{0};
    if (!pnm::allow_smem(pnm::pa_tokens_bwd_kernel<Dp>, smem, smem_set)) return -4;
    pnm::pa_tokens_bwd_kernel<Dp><<<dim3(H, pnm::pa_slices(Cout)), pnm::kPaTokenThreads, smem, (cudaStream_t)stream>>>(
        pnm::make_src(srcs, world, use_flags), Wqkv, Wo, pnm::make_saved(saved), dWo, dWqkv, d_norm, (__nv_bfloat16*)Bcat16, (__nv_bfloat16*)BdT16,
        H, D, Cout, scale, share, p, err);
    return 0;
  };
  const int code = pnm::pa_by_width(D, launch);
  if (code) return code;
  return cudaGetLastError() == cudaSuccess ? 0 : -3;
}

// dWc [H*S + H*D, C], dbc [H*S + H*D]: gradients of the combined projection, then those of the values' projection, which are copied out
// (a parameter's gradient is a buffer of its own).
int pnm_pa_prepare_bwd(const float* dWc, const float* dbc, const float* grp, const float* Wx, const float* bx, const float* Ws,
                       const float* temp, float* dWx, float* dbx, float* dWfx, float* dbfx, float* dWs, float* dbs, float* dtemp, int H, int D,
                       int C, void* stream) {
  if (H <= 0 || D <= 0 || D > pnm::kPaMaxD || C <= 0) return -2;
  pnm::pa_prepare_bwd_kernel<<<H * D + (pnm::kPaS * D) / 8 + 1, 256, 0, (cudaStream_t)stream>>>(dWc, dbc, grp, Wx, bx, Ws, temp, dWx, dbx, dWfx,
                                                                                      dbfx, dWs, dbs, dtemp, H, D, C);
  return cudaGetLastError() == cudaSuccess ? 0 : -3;
}

}  // extern "C"

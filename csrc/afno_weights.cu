// Parameters of the AFNO filter's complex block MLP: to the real bf16 matrices that the GEMMs take, and the gradients back.
//
//   E[n] = [[wr^T, -wi^T], [wi^T, wr^T]]   for w = wr + i wi of block n ([in, out]); both layers and their biases in one launch
//   dwr = (a + d)^T, dwi = (c - b)^T       for dE[n] = [[a, b], [c, d]]
//
// The matrices are a few hundred KB: what they cost is launches (twelve tensor operations forward, as many backward, a third of
// all launches of a small block's prediction).  32 x 32 tiles are transposed through shared memory, so both sides are coalesced.
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "pnm_api.h"

namespace pnm {

struct AfnoPair { const float* w; const float* b; __nv_bfloat16* e; float* be; };
struct AfnoFold { const float* de; const float* dbe; float* dw; float* db; };

// grid (ceil(Cb / 32), ceil(Cb / 32), 2 * nblk), block (32, 8)
__global__ void __launch_bounds__(256) afno_expand_kernel(AfnoPair p1, AfnoPair p2, int nb, int blk0, int nblk, int cb) {
  __shared__ float tr[32][33], ti[32][33];
  const AfnoPair p = blockIdx.z < (unsigned)nblk ? p1 : p2;
  const int n = blockIdx.z % nblk, o0 = blockIdx.x * 32, i0 = blockIdx.y * 32, tx = threadIdx.x;
  const size_t im = (size_t)nb * cb * cb;        // imaginary parts follow the real ones
  const float* w = p.w + (size_t)(blk0 + n) * cb * cb;
  for (int r = threadIdx.y; r < 32; r += 8)
    if (i0 + r < cb && o0 + tx < cb) {
      tr[r][tx] = w[(size_t)(i0 + r) * cb + o0 + tx];
      ti[r][tx] = w[im + (size_t)(i0 + r) * cb + o0 + tx];
    }
  __syncthreads();
  __nv_bfloat16* e = p.e + (size_t)n * 4 * cb * cb;
  for (int r = threadIdx.y; r < 32; r += 8)
    if (o0 + r < cb && i0 + tx < cb) {
      const int o = o0 + r, i = i0 + tx;
      const __nv_bfloat16 re = __float2bfloat16(tr[tx][r]), mi = __float2bfloat16(-ti[tx][r]), pi = __float2bfloat16(ti[tx][r]);
      e[(size_t)o * 2 * cb + i] = re;
      e[(size_t)o * 2 * cb + cb + i] = mi;
      e[(size_t)(cb + o) * 2 * cb + i] = pi;
      e[(size_t)(cb + o) * 2 * cb + cb + i] = re;
    }
  if (blockIdx.x == 0 && blockIdx.y == 0)
    for (int k = threadIdx.y * 32 + tx; k < 2 * cb; k += 256)
      p.be[n * 2 * cb + k] = p.b[((size_t)(k / cb) * nb + blk0 + n) * cb + k % cb];
}

// all blocks; same grid
__global__ void __launch_bounds__(256) afno_fold_kernel(AfnoFold p1, AfnoFold p2, int nb, int cb) {
  __shared__ float tr[32][33], ti[32][33];
  const AfnoFold p = blockIdx.z < (unsigned)nb ? p1 : p2;
  const int n = blockIdx.z % nb, o0 = blockIdx.x * 32, i0 = blockIdx.y * 32, tx = threadIdx.x;
  const float* de = p.de + (size_t)n * 4 * cb * cb;
  for (int r = threadIdx.y; r < 32; r += 8)
    if (o0 + r < cb && i0 + tx < cb) {
      const int o = o0 + r, i = i0 + tx;
      tr[r][tx] = de[(size_t)o * 2 * cb + i] + de[(size_t)(cb + o) * 2 * cb + cb + i];
      ti[r][tx] = de[(size_t)(cb + o) * 2 * cb + i] - de[(size_t)o * 2 * cb + cb + i];
    }
  __syncthreads();
  const size_t im = (size_t)nb * cb * cb;
  float* dw = p.dw + (size_t)n * cb * cb;
  for (int r = threadIdx.y; r < 32; r += 8)
    if (i0 + r < cb && o0 + tx < cb) {
      dw[(size_t)(i0 + r) * cb + o0 + tx] = tr[tx][r];
      dw[im + (size_t)(i0 + r) * cb + o0 + tx] = ti[tx][r];
    }
  if (blockIdx.x == 0 && blockIdx.y == 0)
    for (int k = threadIdx.y * 32 + tx; k < 2 * cb; k += 256)
      p.db[((size_t)(k / cb) * nb + n) * cb + k % cb] = p.dbe[n * 2 * cb + k];
}

}  // namespace pnm

extern "C" int pnm_afno_expand_weights(const float* w1, const float* b1, const float* w2, const float* b2, void* e1, float* be1, void* e2,
                                       float* be2, int nb, int blk0, int nblk, int cb, void* stream) {
  if (nb <= 0 || nblk <= 0 || blk0 < 0 || blk0 + nblk > nb || cb <= 0) return -2;
  const dim3 grid((cb + 31) / 32, (cb + 31) / 32, 2 * nblk);
  const pnm::AfnoPair p1{w1, b1, reinterpret_cast<__nv_bfloat16*>(e1), be1}, p2{w2, b2, reinterpret_cast<__nv_bfloat16*>(e2), be2};
  pnm::afno_expand_kernel<<<grid, dim3(32, 8), 0, reinterpret_cast<cudaStream_t>(stream)>>>(p1, p2, nb, blk0, nblk, cb);
  return cudaGetLastError() == cudaSuccess ? 0 : -17;
}

extern "C" int pnm_afno_fold_grads(const float* de1, const float* dbe1, const float* de2, const float* dbe2, float* dw1, float* db1, float* dw2,
                                   float* db2, int nb, int cb, void* stream) {
  if (nb <= 0 || cb <= 0) return -2;
  const dim3 grid((cb + 31) / 32, (cb + 31) / 32, 2 * nb);
  const pnm::AfnoFold p1{de1, dbe1, dw1, db1}, p2{de2, dbe2, dw2, db2};
  pnm::afno_fold_kernel<<<grid, dim3(32, 8), 0, reinterpret_cast<cudaStream_t>(stream)>>>(p1, p2, nb, cb);
  return cudaGetLastError() == cudaSuccess ? 0 : -17;
}

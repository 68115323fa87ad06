// Shared device helpers for the sm_100a kernel library: mbarrier, TMA (bulk tensor
// copies, never with cluster multicast), tcgen05 (TMEM allocation, MMA issue, commit,
// TMEM loads), bounded waits and the library-wide error word.
//
// Every wait in this library is bounded: when the budget runs out the waiting thread
// records a code in `pnm_error_word`, raises the CTA-local abort flag and returns
// false; callers unwind to the common teardown which frees TMEM and exits.
#pragma once
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

namespace pnm {

// Error codes written to the error word (first error wins).
enum : int {
  ERR_NONE = 0,
  ERR_WAIT_FULL = 1,      // consumer gave up waiting for a TMA stage
  ERR_WAIT_EMPTY = 2,     // producer gave up waiting for a free stage
  ERR_WAIT_TMEM_FULL = 3, // epilogue gave up waiting for an accumulator
  ERR_WAIT_TMEM_EMPTY = 4,
  ERR_WAIT_AUX = 5,
  ERR_WAIT_PEER = 6,      // bounded wait on a peer / signal flag ran out
  ERR_BAD_ARG = 7,
};

// Budget of one bounded wait, in nanoseconds of %globaltimer.
constexpr unsigned long long kWaitBudgetNs = 2000000000ull;  // 2 s
static_assert(kWaitBudgetNs < (1ull << 31), "mbar_wait compares it with the low word of the timer; the rest is for a thread that looks late");

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}
__device__ __forceinline__ unsigned long long globaltimer_ns() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}
__device__ __forceinline__ uint32_t globaltimer_lo() {
  uint32_t t;
  asm volatile("mov.u32 %0, %%globaltimer_lo;" : "=r"(t));
  return t;
}

// One lane of a converged warp, the same one at every call.  For the branches in which a single thread issues tensor-core products or
// bulk copies: their operands live in uniform registers, and after elect.sync the compiler knows that one thread is active, where under
// `lane == 0` it provides for several.  Four products of 128 x 64 x 16, a commit and a wait on a ready barrier took a thread 505 cycles
// under `lane == 0` and take 260 here; the tensor cores need 256 for four of 128 x 128 x 16.
__device__ __forceinline__ bool elect_one() {
  uint32_t p;
  asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.b32 %0, 1, 0, p;\n\t}" : "=r"(p));
  return p != 0;
}

// ---------------------------------------------------------------- mbarrier
__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count));
}
__device__ __forceinline__ void mbar_fence_init() {
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint64_t* bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes)
               : "memory");
}
// Bytes to come, without an arrival.
__device__ __forceinline__ void mbar_expect_more(uint64_t* bar, uint32_t bytes) {
  asm volatile("mbarrier.expect_tx.relaxed.cta.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes) : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint64_t* bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.b32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(smem_u32(bar)), "r"(parity)
      : "memory");
  return ok != 0;
}

// The same without suspending the thread (try_wait may, up to a time limit of the hardware): for a thread that polls several barriers.
__device__ __forceinline__ bool mbar_test(uint64_t* bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.b32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(smem_u32(bar)), "r"(parity)
      : "memory");
  return ok != 0;
}

// Bounded wait. `abort_flag` is a CTA-shared int; once any thread of the CTA times
// out every other waiter leaves promptly. Returns false when the wait was abandoned.
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t parity, volatile int* abort_flag,
                                          int* err_word, int code) {
  if (mbar_try_wait(bar, parity)) return true;
  uint32_t t0 = 0, spins = 0;
  while (true) {
    if (mbar_try_wait(bar, parity)) return true;
    if ((++spins & 0x3ffu) == 0) {
      if (*abort_flag) return false;
      const uint32_t now = globaltimer_lo();     // wraps after 4.3 s, more than the budget
      if (spins == 0x400u) t0 = now;
      else if (now - t0 > uint32_t(kWaitBudgetNs)) {
        atomicCAS(err_word, 0, code);
        *abort_flag = 1;
        __threadfence_block();
        return false;
      }
    }
  }
}

// The wait of a whole warp, one answer for all its lanes: what follows needs the warp together (elect.sync, TMEM loads, shuffles), and
// where a wait runs out one lane may still have seen the phase end and another not.
__device__ __forceinline__ bool mbar_wait_warp(uint64_t* bar, uint32_t parity, volatile int* abort_flag, int* err_word, int code) {
  return __all_sync(0xffffffffu, mbar_wait(bar, parity, abort_flag, err_word, code));
}

// Bounded wait that never raises the abort flag: lets a copy in flight land before the CTA leaves.  `parity` is that of the phase
// that the copy completes and must be the barrier's last: any wait for the other parity is over at once.
__device__ __forceinline__ void mbar_drain(uint64_t* bar, uint32_t parity) {
  const unsigned long long t0 = globaltimer_ns();
  while (!mbar_try_wait(bar, parity)) {
    if (globaltimer_ns() - t0 > kWaitBudgetNs) break;
  }
}
// The same for a ring of which `issued` stages were filled so far, one after the other.
__device__ __forceinline__ void ring_drain(uint64_t* full, uint32_t stages, uint32_t issued) {
  for (uint32_t i = issued > stages ? issued - stages : 0; i < issued; ++i) mbar_drain(&full[i % stages], (i / stages) & 1);
}
// After a wait that ran out: time for products in flight (a microsecond each) to retire before their TMEM is freed.
__device__ __forceinline__ void abort_settle() {
  const unsigned long long t0 = globaltimer_ns();
  while (globaltimer_ns() - t0 < 200000ull) {}
}

// --------------------------------------------------------------------- TMA
__device__ __forceinline__ void tma_prefetch_desc(const CUtensorMap* m) {
  asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(m)) : "memory");
}
// 2-D tiled load global -> this CTA's shared memory, completion on an mbarrier.
__device__ __forceinline__ void tma_load_2d(void* smem_dst, const CUtensorMap* m, uint64_t* bar, int x, int y) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cta.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
      ::"r"(smem_u32(smem_dst)), "l"(reinterpret_cast<uint64_t>(m)), "r"(smem_u32(bar)), "r"(x), "r"(y)
      : "memory");
}
// 2-D tiled store shared -> global (bulk async group).
__device__ __forceinline__ void tma_store_2d(const void* smem_src, const CUtensorMap* m, int x, int y) {
  asm volatile("cp.async.bulk.tensor.2d.global.shared::cta.tile.bulk_group [%0, {%2, %3}], [%1];"
               ::"l"(reinterpret_cast<uint64_t>(m)), "r"(smem_u32(smem_src)), "r"(x), "r"(y)
               : "memory");
}
// 3-D tiled load (x, y, z); coordinates outside the tensor read as zero.
__device__ __forceinline__ void tma_load_3d(void* smem_dst, const CUtensorMap* m, uint64_t* bar, int x, int y, int z) {
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cta.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];"
      ::"r"(smem_u32(smem_dst)), "l"(reinterpret_cast<uint64_t>(m)), "r"(smem_u32(bar)), "r"(x), "r"(y), "r"(z)
      : "memory");
}
// 4-D tiled load / store (channels, x, y, image): used by the implicit-GEMM convolution, where a tile of output pixels
// reads its shifted input window straight from the NHWC tensor; coordinates outside the tensor read as zero.
__device__ __forceinline__ void tma_load_4d(void* smem_dst, const CUtensorMap* m, uint64_t* bar, int c, int x, int y, int n) {
  asm volatile(
      "cp.async.bulk.tensor.4d.shared::cta.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5, %6}], [%2];"
      ::"r"(smem_u32(smem_dst)), "l"(reinterpret_cast<uint64_t>(m)), "r"(smem_u32(bar)), "r"(c), "r"(x), "r"(y), "r"(n)
      : "memory");
}
__device__ __forceinline__ void tma_store_4d(const void* smem_src, const CUtensorMap* m, int c, int x, int y, int n) {
  asm volatile("cp.async.bulk.tensor.4d.global.shared::cta.tile.bulk_group [%0, {%2, %3, %4, %5}], [%1];"
               ::"l"(reinterpret_cast<uint64_t>(m)), "r"(smem_u32(smem_src)), "r"(c), "r"(x), "r"(y), "r"(n)
               : "memory");
}
__device__ __forceinline__ void tma_store_commit() { asm volatile("cp.async.bulk.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void tma_store_wait_read() {
  asm volatile("cp.async.bulk.wait_group.read %0;" ::"n"(N) : "memory");
}
template <int N>
__device__ __forceinline__ void tma_store_wait_all() {
  asm volatile("cp.async.bulk.wait_group %0;" ::"n"(N) : "memory");
}
// global[i] += shared[i], fp32; both 16-byte aligned, a multiple of 16 bytes (bulk async group of the thread).
__device__ __forceinline__ void bulk_add_f32(float* dst, const void* smem_src, uint32_t bytes) {
  asm volatile("cp.reduce.async.bulk.global.shared::cta.bulk_group.add.f32 [%0], [%1], %2;" ::"l"(dst), "r"(smem_u32(smem_src)), "r"(bytes) : "memory");
}
// Make generic-proxy writes to shared memory visible to the async proxy (TMA store).
__device__ __forceinline__ void fence_async_smem() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }

// ----------------------------------------------------------------- tcgen05
__device__ __forceinline__ void tmem_alloc(uint32_t* smem_slot, uint32_t ncols) {
  asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(smem_slot)),
               "r"(ncols)
               : "memory");
}
__device__ __forceinline__ void tmem_relinquish() {
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc(uint32_t taddr, uint32_t ncols) {
  asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
// D[tmem] (+)= A[smem desc] * B[smem desc], bf16/fp16 inputs, fp32 accumulate.
__device__ __forceinline__ void umma_f16(uint32_t d_tmem, uint64_t adesc, uint64_t bdesc, uint32_t idesc,
                                         uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
      ::"r"(d_tmem), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
      : "memory");
}
// Same with the A operand read from tensor memory: lane = row of A, 16-bit elements packed two per 32-bit column
// (K = 16 elements occupy 8 columns).
__device__ __forceinline__ void umma_f16_ts(uint32_t d_tmem, uint32_t a_tmem, uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
      ::"r"(d_tmem), "r"(a_tmem), "l"(bdesc), "r"(idesc), "r"(accumulate)
      : "memory");
}
// Arrive on an mbarrier once all previously issued tcgen05 operations of this thread retire.
__device__ __forceinline__ void umma_commit(uint64_t* bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar))
               : "memory");
}
// 32 lanes x 32 consecutive 32-bit columns -> 32 registers per thread.
__device__ __forceinline__ void tmem_ld32(uint32_t taddr, float* v) {
  uint32_t* r = reinterpret_cast<uint32_t*>(v);
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
      "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
        "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]),
        "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]),
        "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
      : "r"(taddr)
      : "memory");
}
// 32 lanes x 16 consecutive 32-bit columns -> 16 registers per thread
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, float* v) {
  uint32_t* r = reinterpret_cast<uint32_t*>(v);
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]),
        "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr)
      : "memory");
}
// Registers -> 32 lanes x 32 consecutive 32-bit columns.
__device__ __forceinline__ void tmem_st32(uint32_t taddr, const float* v) {
  const uint32_t* r = reinterpret_cast<const uint32_t*>(v);
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], "
      "{%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16, "
      "%17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31, %32};"
      ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]),
        "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]), "r"(r[16]), "r"(r[17]),
        "r"(r[18]), "r"(r[19]), "r"(r[20]), "r"(r[21]), "r"(r[22]), "r"(r[23]), "r"(r[24]), "r"(r[25]), "r"(r[26]),
        "r"(r[27]), "r"(r[28]), "r"(r[29]), "r"(r[30]), "r"(r[31])
      : "memory");
}
__device__ __forceinline__ void tmem_st_wait() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void tmem_ld_wait() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }

// Instruction descriptor of tcgen05.mma kind::f16: bf16 x bf16 -> fp32.
// bits [4,6) D format (1 = f32); [7,10) A format (1 = bf16); [10,13) B format;
// bit 15 / 16: A / B are MN-major; [17,23) N >> 3; [24,29) M >> 4.
__host__ __device__ constexpr uint32_t make_idesc_bf16(int M, int N, bool a_mn_major, bool b_mn_major) {
  return (1u << 4) | (1u << 7) | (1u << 10) | (uint32_t(a_mn_major) << 15) | (uint32_t(b_mn_major) << 16) |
         (uint32_t(N >> 3) << 17) | (uint32_t(M >> 4) << 24);
}
// Shared-memory matrix descriptor: start address, leading / stride byte offsets (16-byte
// units), descriptor version 1 (bit 46), swizzle mode in bits [61,64): 0 none, 2 = 128 B.
__device__ __forceinline__ uint64_t make_smem_desc(uint32_t saddr, uint32_t lbo_bytes, uint32_t sbo_bytes,
                                                   uint32_t layout_type) {
  uint64_t d = 0;
  d |= uint64_t((saddr & 0x3ffff) >> 4);
  d |= uint64_t((lbo_bytes >> 4) & 0x3fff) << 16;
  d |= uint64_t((sbo_bytes >> 4) & 0x3fff) << 32;
  d |= uint64_t(1) << 46;
  d |= uint64_t(layout_type & 7) << 61;
  return d;
}

// -------------------------------------------------------------- math bits
__device__ __forceinline__ float tanh_fast(float x) {
  float y;
  asm("tanh.approx.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ float ex2_fast(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ float lg2_fast(float x) {
  float y;
  asm("lg2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
// 2^x on the FMA / ALU pipes (no special-function unit): round-to-nearest split x = n + f, f in [-0.5, 0.5], cubic for 2^f
// (relative error 1e-4, below bf16 resolution), then n is added to the exponent field.  Inputs below -126 give 0.
__device__ __forceinline__ float ex2_poly(float x) {
  const float xc = fmaxf(x, -126.f);
  const float t = xc + 12582912.f;   // 1.5 * 2^23: the integer part lands in the low mantissa bits
  const float f = xc - (t - 12582912.f);
  float p = fmaf(f, 0.05592204f, 0.24264008f);
  p = fmaf(p, f, 0.69312103f);
  p = fmaf(p, f, 0.99992448f);
  const float r = __int_as_float(__float_as_int(p) + (__float_as_int(t) << 23));
  return x < -126.f ? 0.f : r;
}
// Two fp32 values per instruction (add / mul / fma.rn.f32x2, the same roundings as one by one).
__device__ __forceinline__ uint64_t f2_make(float a, float b) {
  uint64_t r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ float2 f2_get(uint64_t v) {
  float2 r;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
  return r;
}
__device__ __forceinline__ uint64_t f2_add(uint64_t a, uint64_t b) {
  uint64_t r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ uint64_t f2_mul(uint64_t a, uint64_t b) {
  uint64_t r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ uint64_t f2_fma(uint64_t a, uint64_t b, uint64_t c) {
  uint64_t r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}
__device__ __forceinline__ uint64_t f2_all(float a) { return f2_make(a, a); }
__device__ __forceinline__ uint64_t f2_tanh(uint64_t v) {
  const float2 x = f2_get(v);
  return f2_make(tanh_fast(x.x), tanh_fast(x.y));
}

// GELU in its tanh form (|gelu_tanh - gelu_erf| < 1e-3, below bf16 resolution for O(1) values).
__device__ __forceinline__ float gelu_f(float x) {
  const float u = x * (0.7978845608f + 0.0356774081f * x * x), h = 0.5f * x;
  return fmaf(h, tanh_fast(u), h);
}
__device__ __forceinline__ float gelu_grad_f(float x) {
  float x2 = x * x;
  float u = x * (0.7978845608f + 0.0356774081f * x2);
  float t = tanh_fast(u);
  float du = 0.7978845608f + 0.1070322243f * x2;
  return 0.5f * (1.f + t) + 0.5f * x * (1.f - t * t) * du;
}
__device__ __forceinline__ float silu_f(float x) {
  const float h = 0.5f * x;
  return fmaf(h, tanh_fast(h), h);
}
__device__ __forceinline__ float silu_grad_f(float x) {
  float s = 0.5f + 0.5f * tanh_fast(0.5f * x);
  return s * (1.f + x * (1.f - s));
}

// The four for two values: as above, operation by operation.
__device__ __forceinline__ uint64_t gelu_f2(uint64_t x) {
  const uint64_t x2 = f2_mul(x, x), h = f2_mul(x, f2_all(0.5f));
  const uint64_t u = f2_mul(x, f2_fma(f2_all(0.0356774081f), x2, f2_all(0.7978845608f)));
  return f2_fma(h, f2_tanh(u), h);
}
__device__ __forceinline__ uint64_t silu_f2(uint64_t x) {
  const uint64_t h = f2_mul(x, f2_all(0.5f));
  return f2_fma(h, f2_tanh(h), h);
}
// 0.5 (1 + t) + 0.5 x (1 - t^2) u'
__device__ __forceinline__ uint64_t gelu_grad_f2(uint64_t x) {
  const uint64_t x2 = f2_mul(x, x);
  const uint64_t t = f2_tanh(f2_mul(x, f2_fma(f2_all(0.0356774081f), x2, f2_all(0.7978845608f))));
  const uint64_t du = f2_fma(f2_all(0.1070322243f), x2, f2_all(0.7978845608f));
  const uint64_t p = f2_fma(f2_mul(t, f2_all(-1.f)), t, f2_all(1.f));
  return f2_fma(f2_mul(f2_mul(x, f2_all(0.5f)), p), du, f2_fma(t, f2_all(0.5f), f2_all(0.5f)));
}
// s (1 + x (1 - s))
__device__ __forceinline__ uint64_t silu_grad_f2(uint64_t x) {
  const uint64_t s = f2_fma(f2_tanh(f2_mul(x, f2_all(0.5f))), f2_all(0.5f), f2_all(0.5f));
  return f2_mul(s, f2_fma(x, f2_fma(s, f2_all(-1.f), f2_all(1.f)), f2_all(1.f)));
}

__device__ __forceinline__ uint32_t pack_bf16x2(float a, float b) {
  __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
  return *reinterpret_cast<uint32_t*>(&h);
}
__device__ __forceinline__ float2 unpack_bf16x2(uint32_t u) {
  __nv_bfloat162 h = *reinterpret_cast<__nv_bfloat162*>(&u);
  return __bfloat1622float2(h);
}

__device__ __forceinline__ uint32_t f2_to_bf16x2(uint64_t v) {
  const float2 f = f2_get(v);
  return pack_bf16x2(f.x, f.y);
}
__device__ __forceinline__ uint64_t f2_from_bf16x2(uint32_t u) {      // the upper halves of two floats
  uint32_t a, b;
  a = u << 16; b = u & 0xffff0000u;
  return f2_make(__uint_as_float(a), __uint_as_float(b));
}

}  // namespace pnm

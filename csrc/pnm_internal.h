// Declarations shared by the translation units of the kernel library (not part of the C ABI).
#pragma once
#include <atomic>
#include "peer.cuh"

namespace pnm {

constexpr int kMaxDevices = 64;

int current_device();          // index of the current CUDA device (0 when it cannot be read)
int* error_word_ptr();         // device address of the library's error word on the current device (null on failure)
int num_sms();                 // SM count of the current device
PeerArgs make_peer_args(const void* const* bases, int rank, int world, unsigned int epoch, long long capacity_floats,
                        double budget_s, const void* epoch_base);

// Which devices a kernel's attributes have been set on, one bit each (they belong to the device's context).
using DeviceMask = std::atomic<unsigned long long>;

// Allows `kernel` `bytes` of dynamic shared memory on the current device, once per device and kernel.  The bit follows the
// attribute: a thread that sees it may launch, and threads that make the first call together all set it.
template <typename K>
inline bool allow_smem(K* kernel, size_t bytes, DeviceMask& done) {
  const unsigned long long bit = 1ull << (current_device() & 63);
  if (done.load(std::memory_order_acquire) & bit) return true;
  if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, int(bytes)) != cudaSuccess) return false;
  done.fetch_or(bit, std::memory_order_release);
  return true;
}

}  // namespace pnm

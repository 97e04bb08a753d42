// Internal launch helpers shared by the kernel translation units.
#pragma once

#include <cstdio>
#include <mutex>
#include <stdexcept>
#include <string>

#include "hz_kernels.cuh"

namespace hz {

static inline void check_launch(const char* name) {
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) {
    char buf[256];
    snprintf(buf, sizeof(buf), "kernel %s launch failed: %s", name, cudaGetErrorString(e));
    throw std::runtime_error(buf);
  }
}

// bytes: the launch's algorithmic DRAM bytes (each input read once, each
// output written once), the numerator of its roofline fraction.
#define HZ_LAUNCH(ctx, name, bytes, kern, grid, block, smem, ...) \
  do {                                                          \
    static thread_local int _id = -1;                           \
    const char* _nm = (name);                                   \
    if (_id < 0 || (size_t)_id >= (ctx).names.size() ||         \
        (ctx).names[_id] != _nm)                                \
      _id = (ctx).name_id(_nm);                                 \
    cudaEvent_t _a = nullptr;                                   \
    (ctx).before(_id, &_a);                                     \
    kern<<<grid, block, smem, (ctx).stream>>>(__VA_ARGS__);     \
    check_launch(_nm);                                          \
    (ctx).after(_id, _a, (double)(bytes));                      \
  } while (0)

static constexpr int kSMs = 152;

// A kernel's limit of dynamic shared memory belongs to the kernel on its device, not to a
// launch or a thread.  So it is raised once per device, to the most that any launch takes: a
// launch that set its own size could find it lowered by another thread's before it starts.
struct SmemLimit {
  std::mutex mu;
  bool raised[kMaxDevices] = {};
};
static inline void raise_smem_limit(SmemLimit& limit, const void* kernel, size_t bytes, const char* name,
                                    bool large_clusters = false) {
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev < 0 || dev >= kMaxDevices) throw std::runtime_error(std::string(name) + ": device ordinal out of range");
  std::lock_guard<std::mutex> lk(limit.mu);
  if (limit.raised[dev]) return;
  cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
  if (e == cudaSuccess && large_clusters)
    e = cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
  if (e != cudaSuccess) {
    cudaGetLastError();
    throw std::runtime_error(std::string(name) + ": shared memory attribute: " + cudaGetErrorString(e));
  }
  limit.raised[dev] = true;
}

// Column chunking: enough CTAs in flight for 152 SMs while each CTA reuses
// its per-node coefficients across as many right-hand sides as possible.
static inline int chunks_for(long long nblk_x, int ncols, int target = 8 * kSMs) {
  long long ch = (target + nblk_x - 1) / nblk_x;
  if (ch < 1) ch = 1;
  if (ch > ncols) ch = ncols;
  return (int)ch;
}

}  // namespace hz

// Shared helpers of the sm_100a kernels: error plumbing, device-wide barrier
// with a bounded wait, timers and exact-rounding arithmetic.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>
#include <string>

#include "../../include/ks_b200.h"

namespace ks {

// Message of the last failure on the calling host thread.
void set_error(const std::string& msg);
int fail(int code, const std::string& msg);
int cuda_fail(cudaError_t e, const char* what);

#define KS_CUDA(call)                                        \
  do {                                                       \
    cudaError_t _e = (call);                                 \
    if (_e != cudaSuccess) return ::ks::cuda_fail(_e, #call); \
  } while (0)

// Arrays that the kernels read and write 16 bytes at a time.
inline bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; }
inline int64_t round_up(int64_t x, int64_t m) { return (x + m - 1) / m * m; }
inline size_t align256(size_t x) { return (x + 255) & ~size_t(255); }

// Per-device properties cached on first use.
struct DeviceInfo {
  int device = -1;
  int sm_count = 0;
  int cc_major = 0, cc_minor = 0;
  size_t smem_optin = 0;
};
int device_info(DeviceInfo* out);

// Simple bump allocator over a caller workspace.
struct Carve {
  char* base;
  size_t used = 0;
  explicit Carve(void* p) : base(static_cast<char*>(p)) {}
  template <typename T>
  T* take(size_t n) {
    T* p = reinterpret_cast<T*>(base ? base + used : nullptr);
    used = align256(used + n * sizeof(T));
    return p;
  }
};

// Default limit of every device-side wait (ns of %globaltimer).
constexpr unsigned long long kWaitLimitNs = 2000000000ull;
// kWaitLimitNs, or KS_B200_WAIT_LIMIT_NS from the environment when set.
unsigned long long wait_limit_ns();
// Stage marks of ks_trace_stages: record the calling thread's event `slot`
// on the stream when tracing is on (no-op otherwise).
constexpr int kTraceMarks = 5;
void trace_mark(int slot, cudaStream_t stream);

}  // namespace ks

// ---------------------------------------------------------------- device side

__device__ __forceinline__ unsigned long long ks_globaltimer() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

__device__ __forceinline__ unsigned ks_ld_acquire(const unsigned* p) {
  unsigned v;
  asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}

__device__ __forceinline__ int ks_ld_volatile(const int* p) {
  return *reinterpret_cast<const volatile int*>(p);
}

// Control word of a team of co-resident blocks: arrivals at its barriers in the
// low 56 bits, the first error's code above them.  Every access while the team
// runs is 64 bits wide (memory-model ordering holds between accesses of one width
// to one word, not between a word and its halves).
constexpr int kCtlErrShift = 56;

__device__ __forceinline__ unsigned long long ks_ctl_load(const unsigned long long* ctl) {
  unsigned long long v;
  asm volatile("ld.acquire.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(ctl) : "memory");
  return v;
}
__device__ __forceinline__ int ks_ctl_error(const unsigned long long* ctl) {
  return (int)(ks_ctl_load(ctl) >> kCtlErrShift);
}
// Record an error; the first one stays.  A lost exchange means that another
// block arrived or failed in between, so the loop ends after as many rounds as
// there are blocks.
__device__ __forceinline__ void ks_ctl_fail(unsigned long long* ctl, int code) {
  unsigned long long v = ks_ctl_load(ctl);
  while (!(v >> kCtlErrShift)) {
    const unsigned long long seen = atomicCAS(ctl, v, v | (unsigned long long)code << kCtlErrShift);
    if (seen == v) break;
    v = seen;
  }
}

// Device-wide barrier for a cooperative (co-resident) grid over a control word
// that starts at zero.  The count only grows: barrier number `epoch` (1, 2, ...)
// completes when it reaches epoch * nblocks, so arriving is a single atomic and
// there is no reset to order.  Every block passes the same sequence of barriers
// and keeps its own epoch.  A wait that exceeds limit_ns records KS_ERR_TIMEOUT
// and returns; every caller then sees the error and leaves its loop, so no block
// waits without bound.  Returns true when no error is recorded; the answer is the
// same for every thread of the block (thread 0 reads the word and the closing
// barrier broadcasts it), so callers may branch on it around further block
// barriers.  A wait is round trips to L2, whatever the number of blocks (20 to
// 296 the same): one release and one acquire that reads the count and the error
// together, so that no fence and no second load follow the last arrival: a peel
// of 46 iterations at C=384, K=600, L=60122 1519 -> 1423 us against fences on
// both sides, a sleep before every poll and the error read at the end.
__device__ __forceinline__ bool ks_grid_sync(unsigned long long* ctl, unsigned nblocks,
                                             unsigned& epoch, unsigned long long limit_ns) {
  __syncthreads();
  ++epoch;
  int bad = 0;
  if (threadIdx.x == 0) {
    const unsigned long long target = (unsigned long long)epoch * nblocks;
    asm volatile("red.release.gpu.global.add.u64 [%0], %1;" ::"l"(ctl), "l"(1ull) : "memory");
    unsigned long long t0 = 0;
    for (unsigned spin = 0;; ++spin) {
      const unsigned long long v = ks_ctl_load(ctl);
      bad = (v >> kCtlErrShift) != 0;
      if ((v & ((1ull << kCtlErrShift) - 1)) >= target) break;
      if (spin >= 16) {
        __nanosleep(20);
        if (t0 == 0) t0 = ks_globaltimer();
        if (ks_globaltimer() - t0 > limit_ns) {
          ks_ctl_fail(ctl, KS_ERR_TIMEOUT);
          bad = 1;
          break;
        }
      }
    }
  }
  return __syncthreads_or(bad) == 0;
}

// xfp_sweep_util.cuh -- device helpers of the wavefront kernel (xfp_wave.cu):
// payload <-> 32-bit word conversion, stamped 64-bit hand-off words and bounded
// waits with error reporting.
#pragma once

#include <climits>
#include <type_traits>

#include "xfp_common.cuh"
#include "xfp_kernels.h"

namespace xfp {

template <typename T>
struct Pair {
  T a, b;
};

// ---- payload <-> 32-bit words ----
template <typename T>
struct Words {
  static constexpr int P = sizeof(T) / 4;
};
template <typename T>
__device__ __forceinline__ void to_words(const T& v, uint32_t* w) {
  union {
    T v;
    uint32_t w[sizeof(T) / 4];
  } u;
  u.v = v;
#pragma unroll
  for (int p = 0; p < (int)(sizeof(T) / 4); ++p) w[p] = u.w[p];
}
template <typename T>
__device__ __forceinline__ T from_words(const uint32_t* w) {
  union {
    T v;
    uint32_t w[sizeof(T) / 4];
  } u;
#pragma unroll
  for (int p = 0; p < (int)(sizeof(T) / 4); ++p) u.w[p] = w[p];
  return u.v;
}
__device__ __forceinline__ unsigned long long stamped(uint32_t stamp, uint32_t word) {
  return ((unsigned long long)stamp << 32) | word;
}
__device__ __forceinline__ unsigned long long ld_gpu64(const unsigned long long* p) {
  unsigned long long v;
  asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p));
  return v;
}

// Turns of a wait: false after `limit`, and with ctl once another wait has run out.
struct Spin {
  long long n = 0;
  __device__ __forceinline__ bool step(long long limit) {
    ++n;
    if (n > 256) __nanosleep(n > 8192 ? 256 : 20);
    return n < limit;
  }
  __device__ __forceinline__ bool step(const SweepCtl* ctl, long long limit) {
    if (!step(limit)) return false;
    return (n & 255) != 0 || ld_volatile_u32(&ctl->err) == 0;
  }
};

// Records the first wait that ran out (site, tile, step, thread) and raises
// the error flag every other wait checks.
__device__ __forceinline__ void raise_timeout(SweepCtl* ctl, unsigned where, int tile = -1, int tau = -1,
                                              int op = -1, unsigned long long seen = 0, unsigned expect = 0) {
  if (atomicCAS(&ctl->err, 0u, 1u) == 0u) {
    ctl->err_word = seen;
    ctl->err_expect = expect;
    ctl->err_where = where;
    ctl->err_tile = tile;
    ctl->err_tau = tau;
    ctl->err_thread = (int)(blockIdx.x * blockDim.x + threadIdx.x);
    ctl->err_op = op;
  }
}

}  // namespace xfp

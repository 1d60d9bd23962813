// xfp_warp_wait.h -- a warp's wait, ended by all its lanes together.
//
// A lane's own look at a mbarrier or at a word in shared memory promises nothing
// about what the other lanes see in the same turn.  A lane that left by its own
// answer would meet the warp's next shuffle while others still vote here, so the
// turn is decided by votes: every lane takes every turn, and all leave in the same
// one.  Plain C++ with the vote passed in, so that it also runs on the host.
#pragma once

#ifdef __CUDACC__
#define XFP_WARP_FN __device__ __forceinline__
#else
#define XFP_WARP_FN inline
#endif

namespace xfp {

// attempt(): this lane's look; step(): counts a turn, false once the lane has waited
// long enough; all(v): true if v is true in every lane.  False: given up.
template <typename Attempt, typename All, typename Step>
XFP_WARP_FN bool warp_wait(Attempt&& attempt, All&& all, Step&& step) {
  while (!all(attempt()))
    if (!all(step())) return false;
  return true;
}

}  // namespace xfp

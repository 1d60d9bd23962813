// xfp_edges.h -- which groups of edge values pass between two neighbouring blocks.
//
// A block (WBlk) has ng groups from the global group g0 on, numbered from 0 in sweep
// order.  It takes its groups as u = q + 1: to work on group q it needs its producer's
// values of the same global group, and of the one before it for the first step, so u
// runs from 0 (only the producer's group before its first) to ng.  What a producer
// sends to a consumer has to be exactly what the consumer waits for; the functions are
// plain C++, so that a test can hold one against the other.
#pragma once

#include <climits>

#ifdef __CUDACC__
#define XFP_EDGE_FN __host__ __device__ __forceinline__
#else
#define XFP_EDGE_FN inline
#endif

namespace xfp {

// The producer's number of the consumer's group u is u + edge_shift.
XFP_EDGE_FN int edge_shift(bool rev, int p_g0, int p_ng, int c_g0, int c_ng) {
  return (rev ? p_g0 + p_ng - c_g0 - c_ng : c_g0 - p_g0) - 1;
}
// The consumer gets values for u (u <= ng) from a producer with p_ng groups.
XFP_EDGE_FN bool edge_comes(int u, int shift, int p_ng) { return (unsigned)(u + shift) < (unsigned)p_ng; }
// ... the first and the last such u (none: first > last).
XFP_EDGE_FN int first_edge(int shift) { return shift < 0 ? -shift : 0; }
XFP_EDGE_FN int last_edge(int shift, int p_ng, int c_ng) {
  return p_ng == 0 ? -1 : (p_ng - 1 - shift < c_ng ? p_ng - 1 - shift : c_ng);
}
// The producer sends its groups q, shift <= q <= last_sent, as the consumer's u = q - shift.
XFP_EDGE_FN int last_sent(int shift, int p_ng, int c_ng) {
  return c_ng == 0 ? INT_MIN : (shift + c_ng < p_ng - 1 ? shift + c_ng : p_ng - 1);
}

}  // namespace xfp

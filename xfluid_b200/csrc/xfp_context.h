// xfp_context.h -- the context behind xfp_ctx* and the host helpers shared by
// the single-scene driver (xfp_capi.cu) and the batch driver (xfp_batch.cu).
// Internal to libxfp.
#pragma once

#include <algorithm>
#include <climits>
#include <string>
#include <vector>

#include "../../include/xfp.h"
#include "xfp_common.cuh"
#include "xfp_kernels.h"

namespace xfp_host {

constexpr int NBLK_MAX = 148 * 8;   // blocks of the reduction kernels (partials slots)

// A device allocation that only grows; given back with its owner (on the owner's
// device, which the caller has made the current one).
struct DevBuf {
  void* p = nullptr;
  size_t cap = 0;
  DevBuf() = default;
  DevBuf(const DevBuf&) = delete;
  DevBuf& operator=(const DevBuf&) = delete;
  ~DevBuf() {
    if (p) cudaFree(p);
  }
  cudaError_t ensure(size_t bytes) {
    if (bytes <= cap && p) return cudaSuccess;
    if (p) cudaFree(p);
    p = nullptr;
    cap = 0;
    size_t want = std::max<size_t>(bytes, 256);
    cudaError_t e = cudaMalloc(&p, want);
    if (e == cudaSuccess) cap = want;
    return e;
  }
  template <typename T>
  T* as() const { return reinterpret_cast<T*>(p); }
};

struct BatchState;                      // xfp_batch.cu
void batch_state_free(BatchState* b);

}  // namespace xfp_host

struct xfp_ctx {
  xfp_options opt;
  int device = 0;
  cudaStream_t stream = nullptr;
  bool own_stream = false;
  std::string err;
  using DevBuf = xfp_host::DevBuf;
  // I/O staging (host-pointer mode)
  DevBuf io_mat, io_u, io_v, io_w, io_wu, io_wv, io_ww, io_p, io_gu, io_gv, io_gw;
  // layout
  DevBuf lines, line_sums, blks, tiles, counters, group_nb;
  // compact arrays
  DevBuf A64[5];                  // diag, ax, ay, az, b (FP64)
  DevBuf A32[5];                  // same in FP32
  DevBuf x64, r64, x32, r32, s32, z32, s64, z64, dense;
  // control
  DevBuf ctl, scal2, partials, tpartials;   // ctl: LoopWords
  // particle steps (xfp_particles.cu): staged particles and field, bin keys,
  // indices, boxes, positions, bin starts, box spans, sort/scan scratch
  DevBuf part_io, phi_io, part_key, part_idx, part_spos, part_start, part_span,
      part_tmp;
  // sweep layout (WBlk), Gsw groups: the factorisation's operands, the factor,
  // r and y/z, the line-group -> element map, and the block-edge words (zeroed
  // when (re)allocated so no stale word can carry a live generation)
  DevBuf sw_sys, sw, gperm, edge;
  // host-pointer mode: fluid span per x-line and the two byte counters of
  // the sparse face transfer; bytes moved by the current call; whether its
  // velocities went face-sparse; XFP_HOST_FACES=full turns the sparse
  // transfer off
  DevBuf hio_span, hio_bytes;
  // host-pointer mode: a second stream for the transfers that can run beside
  // the compute stream (the face gather beside the layout build, the dense
  // pressure download beside the apply), and its events; io_pending: the
  // compute stream has still to wait for io_in before it reads the faces
  cudaStream_t io_stream = nullptr;
  cudaEvent_t ev_io_mat = nullptr, ev_io_in = nullptr, ev_io_p = nullptr;
  bool io_pending = false;
  long long h2d_bytes = 0, d2h_bytes = 0;
  int host_faces = 0;
  int host_sparse_ok = 1;
  // xfp_project_step_*: body force fused into assembly and apply, and the
  // extrapolation layers run after the apply (zero outside such a call);
  // xmarker is the extrapolation's layer bits
  xfp::Force3 force;
  int step_layers = 0;
  DevBuf xmarker;
  long long Gsw = 0, nlines_all = 0;   // groups and x-lines (one scene, or the whole batch)
  // block cap of the PCG loop's SpMV: 148 x 4 measured best at 256^3 (24.8 us per
  // launch with its event pair, against 27.7 at 148 x 8 and 29.3 at 148 x 2; 128^3
  // FP64: 16.7, 13.3 at 148; no difference at 48^3 and below).  XFP_VEC_BLOCKS
  // overrides, within [148, NBLK_MAX]; the dot's reduction order follows it.
  int vec_blocks = 148 * 4;
  // block cap of the x/r update (two groups in flight per thread): 148 x 2
  // measured best at 256^3 (21.1 us, against 26.3 at 148, 26.2 at 148 x 4 and 27.4
  // at 148 x 8).  Its |r|_inf is a max, the same in any order.  XFP_XR_BLOCKS
  // overrides, within [148, NBLK_MAX].
  int xr_blocks = 148 * 2;
  // CUDA events around the PCG loop's solve and vector-kernel launches
  // (xfp_stats.ms_sweeps, ms_vec), on every event_every-th iteration; 0 (the
  // default) records none.  An event between two launches serialises them:
  // events on every launch cost 1.3 ms of a 21.8 ms projection at 256^3.
  // XFP_KERNEL_EVENTS=N sets it.
  int event_every = 0;
  int sweep_ord = 0;              // triangular-solve launches of the current PCG loop
  std::vector<int> sweep_ord_of;  // per timed sweep entry: its launch ordinal
  // block cap of the PCG loop's s update: 148 x 8 at 256^3 (14.7 us per launch,
  // against 13.8 at 148 x 4, 16.8 at 148 x 16 and 21.2 at 148, with two groups in
  // flight per thread).  XFP_S_BLOCKS overrides, within [148, 148 x 32].
  int s_blocks = 148 * 8;
  // sizes of the current layout
  int ni = 0, nj = 0, nk = 0, NJB = 0, NKB = 0;
  int nw = 8;                     // options.tile_k as reported in the stats
  long long M = 0, rows = 0, nlines_act = 0, ntiles = 0;
  xfp::PcgScalars host_sc{};
  // The PCG loop's iterations as a graph (launch_iterations), re-captured for every
  // loop on a stream of the context's own: whatever else a program puts on its
  // stream meanwhile stays out.  The executable graph is updated, not rebuilt.
  cudaStream_t cap_stream = nullptr;
  cudaGraphExec_t loop_exec = nullptr;
  cudaEvent_t loop_ev[2] = {};
  bool loop_cooperative = false;  // the executable graph's sweeps are cooperative launches
  bool loop_graph = false;        // this call's loop ran as a graph
  // The sweeps' control block and the loop's scalars, on the device (ctl), and as a
  // loop last read them: one copy, into ordinary memory (a page-locked allocation
  // takes 2.4 ms, more than all else that a new context does).
  struct LoopWords {
    xfp::SweepCtl ctl;
    alignas(128) xfp::PcgScalars sc;
  };
  LoopWords loop_read_here{}, *loop_read = &loop_read_here;
  // stats
  double ms_setup = 0, ms_factor = 0, ms_solve = 0, ms_apply = 0;
  int iters = 0, refinements = 0;
  double res = 0, bnorm = 0;
  cudaEvent_t ev[8] = {};
  // device timing of the triangular-solve sweeps (pairs of events, read at the end)
  std::vector<cudaEvent_t> sweep_ev;
  int sweep_ev_used = 0;
  // per timed sweep launch (event pair): 1 when it did work, 0 for the
  // launches a PCG loop issues after convergence (they return at once)
  std::vector<char> sweep_work;
  // the PCG loop's vector kernels, timed the same way: event pairs with the
  // kernel kind (0 SpMV + dot, 1 x/r update, 2 s update) and its PCG iteration
  // (launches after the converged iteration return at once and are dropped)
  std::vector<cudaEvent_t> kern_ev;
  std::vector<int> kern_kind, kern_iter;
  int kern_ev_used = 0;
  long long launches = 0;
  // batched scenes (xfp_project_batch_*): buffers, tables and tuning cache
  xfp_host::BatchState* batch = nullptr;
  // xfp_debug_expire_next_sweep: in the n-th sweep launch from here on (0: none) the
  // waits for other clusters' edge words run out
  int expire_sweep = 0;
};

namespace xfp_host {

inline int fail(xfp_ctx* ctx, int code, const std::string& msg) {
  if (ctx) ctx->err = msg;
  return code;
}

#define XFP_CUDA(ctx, call)                                                                    \
  do {                                                                                         \
    cudaError_t _e = (call);                                                                   \
    if (_e != cudaSuccess) {                                                                   \
      return ::xfp_host::fail(ctx, _e == cudaErrorMemoryAllocation ? XFP_ERR_NOMEM : XFP_ERR_CUDA, \
                              std::string(#call) + ": " + cudaGetErrorString(_e));             \
    }                                                                                          \
  } while (0)

// Stage an input array on the device (or use it in place).
template <typename T>
int stage_in(xfp_ctx* ctx, DevBuf& buf, const T* src, size_t n, const T** dev) {
  if (src == nullptr) { *dev = nullptr; return XFP_OK; }
  if (ctx->opt.device_pointers) { *dev = src; return XFP_OK; }
  XFP_CUDA(ctx, buf.ensure(n * sizeof(T)));
  XFP_CUDA(ctx, cudaMemcpyAsync(buf.p, src, n * sizeof(T), cudaMemcpyHostToDevice, ctx->stream));
  ctx->h2d_bytes += (long long)(n * sizeof(T));
  *dev = buf.as<T>();
  return XFP_OK;
}

// xfp_capi.cu
size_t ncells(int ni, int nj, int nk);
size_t nu(int ni, int nj, int nk);
size_t nv(int ni, int nj, int nk);
size_t nw_(int ni, int nj, int nk);
long long spin_limit(const xfp_ctx* ctx);
int check_dims(xfp_ctx* ctx, int ni, int nj, int nk, const void* mat);
int ensure_compact(xfp_ctx* ctx, int prec);
int check_sweep_error(xfp_ctx* ctx);
int sweep_error(xfp_ctx* ctx, const xfp::SweepCtl& c);

}  // namespace xfp_host

#include "xfp_loop.h"

namespace xfp_host {

// Sweep-layout buffers of the current layout: the factorisation's operands
// (zeroed: cells that lines do not have stay zero), the factor, r (zeroed) and
// y in 8 bytes a value, and the block-edge words.
inline int ensure_sweep(xfp_ctx* ctx, size_t sys_bytes) {
  if (ctx->ntiles == 0) return XFP_OK;
  const size_t n = (size_t)ctx->Gsw * 256;
  XFP_CUDA(ctx, ctx->sw_sys.ensure(n * 4 * 8));
  XFP_CUDA(ctx, ctx->sw.ensure((size_t)ctx->Gsw * xfp::WAVE_ROW * 8));
  XFP_CUDA(ctx, cudaMemsetAsync(ctx->sw_sys.p, 0, n * 4 * sys_bytes, ctx->stream));
  const size_t words = (size_t)ctx->Gsw * 2 * xfp::WAVE_EDGE;
  if (ctx->edge.cap < words * 8 || !ctx->edge.p) {
    XFP_CUDA(ctx, ctx->edge.ensure(words * 8));
    XFP_CUDA(ctx, cudaMemsetAsync(ctx->edge.p, 0, ctx->edge.cap, ctx->stream));
  }
  return XFP_OK;
}

// r into the sweep layout, ready for the solves.
template <typename VT>
int sweep_rhs(xfp_ctx* ctx, const VT* r) {
  if (ctx->ntiles == 0) return XFP_OK;
  VT* const sr = ctx->sw.as<VT>() + xfp::WAVE_R;
  XFP_CUDA(ctx, cudaMemset2DAsync(sr, xfp::WAVE_ROW * sizeof(VT), 0, 256 * sizeof(VT), (size_t)ctx->Gsw, ctx->stream));
  XFP_CUDA(ctx, xfp::sw_permute<VT>(const_cast<VT*>(r), sr, ctx->gperm.as<int>(), ctx->M, 0,
                                    ctx->stream));
  return XFP_OK;
}

// Line-layout copy of the sweep-ordered solve result (z, or y after a
// forward solve alone).
template <typename VT>
int sweep_result(xfp_ctx* ctx, VT* out) {
  if (ctx->ntiles == 0) return XFP_OK;
  XFP_CUDA(ctx, xfp::sw_permute<VT>(out, ctx->sw.as<VT>() + xfp::WAVE_Y, ctx->gperm.as<int>(), ctx->M, 1, ctx->stream));
  return XFP_OK;
}

// The operands every sweep of the current layout shares.
inline xfp::WaveArgs wave_args(xfp_ctx* ctx) {
  xfp::WaveArgs g;
  g.nj = ctx->nj;
  g.nk = ctx->nk;
  g.NJB = ctx->NJB;
  g.NKB = ctx->NKB;
  g.ntiles = (int)ctx->ntiles;
  g.tiles = ctx->tiles.as<int2>();
  g.blks = ctx->blks.as<xfp::WBlk>();
  g.ctl = ctx->ctl.as<xfp::SweepCtl>();
  g.spin_limit = spin_limit(ctx);
  g.omega = ctx->opt.omega;
  g.ratio = ctx->opt.min_diag_ratio;
  g.sys = ctx->sw_sys.p;
  g.sw = ctx->sw.p;
  g.partials = ctx->tpartials.as<double>();
  g.bj = ctx->edge.as<unsigned long long>();
  g.bk = g.bj + (size_t)ctx->Gsw * xfp::WAVE_EDGE;
  return g;
}

}  // namespace xfp_host

// xfp_loop.h -- the PCG loop's iterations as a CUDA graph: capture, replay and the
// host's reads.  Plain host code over the CUDA runtime's C interface; xfp_ctx, fail,
// XFP_CUDA and sweep_error are the including file's (xfp_context.h).
#pragma once

#include <cuda_runtime_api.h>

namespace xfp {
extern thread_local long long g_kernel_launches;
}

namespace xfp_host {

// Iterations of a PCG loop's graph; its scalars are read after every launch of it.
// options.check_every bounds them.  Since the read runs beside the next launch, more
// than four only add launches past the end (two launches of the graph are on their
// way when the last one is known), and fewer, or one of an odd check_every, a read an
// iteration.
inline int loop_iterations(const xfp_ctx* ctx) {
  const int K = ctx->opt.check_every > 0 ? ctx->opt.check_every : 8;
  return K < 4 ? K : 4;
}

// Captures n iterations of a PCG loop (iteration(stream) launches one) into
// ctx->loop_exec.  False if a graph is refused: the loop then launches directly.
// A kernel of a graph starts 0.2 us after the one before it, one launched on a
// stream 2.3 us; capturing 20 launches and updating the executable graph takes
// 90 us on the host, while the device still works on what comes before the loop.  An
// update is not asked to change whether launches are cooperative: those of one cluster
// are not (wave_launch), and a graph of the other kind is given back first.
template <typename F>
bool capture_iterations(xfp_ctx* ctx, int n, bool cooperative, F&& iteration) {
  for (cudaEvent_t& e : ctx->loop_ev)
    if (!e && cudaEventCreateWithFlags(&e, cudaEventDisableTiming) != cudaSuccess) {
      e = nullptr;
      cudaGetLastError();
      return false;
    }
  if (!ctx->cap_stream && cudaStreamCreateWithFlags(&ctx->cap_stream, cudaStreamNonBlocking) != cudaSuccess) {
    ctx->cap_stream = nullptr;
    cudaGetLastError();
    return false;
  }
  cudaGraph_t graph = nullptr;
  const long long before = xfp::g_kernel_launches;
  cudaError_t e = cudaStreamBeginCapture(ctx->cap_stream, cudaStreamCaptureModeThreadLocal);
  if (e == cudaSuccess) {
    cudaError_t le = cudaSuccess;
    for (int q = 0; q < n && le == cudaSuccess; ++q) le = iteration(ctx->cap_stream);
    e = cudaStreamEndCapture(ctx->cap_stream, &graph);
    if (le != cudaSuccess) e = le;
  }
  xfp::g_kernel_launches = before;   // counted per launch of the graph
  if (e == cudaSuccess && graph) {
    if (ctx->loop_exec && ctx->loop_cooperative != cooperative) {
      cudaGraphExecDestroy(ctx->loop_exec);
      ctx->loop_exec = nullptr;
    }
    ctx->loop_cooperative = cooperative;
    cudaGraphExecUpdateResultInfo info;
    if (ctx->loop_exec && cudaGraphExecUpdate(ctx->loop_exec, graph, &info) != cudaSuccess) {
      cudaGetLastError();
      cudaGraphExecDestroy(ctx->loop_exec);
      ctx->loop_exec = nullptr;
    }
    if (!ctx->loop_exec) e = cudaGraphInstantiate(&ctx->loop_exec, graph, 0);
  }
  if (graph) cudaGraphDestroy(graph);
  if (e == cudaSuccess) return ctx->loop_exec != nullptr;
  if (ctx->loop_exec) cudaGraphExecDestroy(ctx->loop_exec);   // (an earlier call's)
  ctx->loop_exec = nullptr;
  cudaGetLastError();
  return false;
}

// Launches the captured graph (n iterations of per_iter kernels) until done() says
// that everything has ended: read(stream) enqueues the copy of what done looks at and
// of the sweeps' error word (ctx->loop_read->ctl).  The scalars of one launch are read
// while the next one runs, so the device does not wait for the host (30 us a read);
// once everything has ended, kernels return at once.
//
// Such a read may meet an update half-way.  The kernels write `done` last, behind a
// fence (end_solve), so it tells that all has ended, and a second read, begun after
// it, brings what the flag stands for.  The record of a wait that ran out is whole
// once its launch is over.
template <typename Read, typename Done>
int replay_iterations(xfp_ctx* ctx, int n, int per_iter, long long limit, Read&& read, Done&& done) {
  cudaStream_t st = ctx->stream, side = ctx->cap_stream;
  int rc = XFP_OK;
  auto launch = [&](int q) -> int {
    XFP_CUDA(ctx, cudaGraphLaunch(ctx->loop_exec, st));
    XFP_CUDA(ctx, cudaEventRecord(ctx->loop_ev[q & 1], st));
    xfp::g_kernel_launches += (long long)n * per_iter;
    return XFP_OK;
  };
  auto look = [&](cudaStream_t from) -> int {
    XFP_CUDA(ctx, read(from));
    XFP_CUDA(ctx, cudaStreamSynchronize(from));
    return XFP_OK;
  };
  const auto& failed = ctx->loop_read->ctl.err;
  if ((rc = launch(0)) != XFP_OK) return rc;
  for (int q = 1;; ++q) {
    if ((rc = launch(q)) != XFP_OK) return rc;
    XFP_CUDA(ctx, cudaStreamWaitEvent(side, ctx->loop_ev[(q - 1) & 1], 0));
    if ((rc = look(side)) != XFP_OK) return rc;
    if (failed || done()) break;
    if ((long long)q * n > limit) return fail(ctx, XFP_ERR_CUDA, "PCG loop did not terminate");
  }
  if (!failed && (rc = look(side)) != XFP_OK) return rc;
  if (failed && (rc = look(st)) != XFP_OK) return rc;
  return sweep_error(ctx, ctx->loop_read->ctl);
}

}  // namespace xfp_host

// The PCG loop's host side (xfluid_b200/csrc/xfp_loop.h) against a CUDA runtime of
// the test's own: a device that ends a solve, or reports an expired wait, while the
// host reads.
#include <cstdio>
#include <cstdlib>
#include <cuda_runtime_api.h>
#include <functional>
#include <string>

struct Scalars {
  double res = 0;
  int done = 0, iters = 0;
};
struct Ctl {
  unsigned err = 0, err_where = 0;
};
struct xfp_ctx {
  struct {
    int check_every = 0;
  } opt;
  cudaStream_t stream = (cudaStream_t)1, cap_stream = nullptr;
  cudaGraphExec_t loop_exec = nullptr;
  cudaEvent_t loop_ev[2] = {};
  bool loop_cooperative = false;
  struct Read {
    Scalars sc;
    Ctl ctl;
  } read, *loop_read = &read;
  std::string err;
};
enum { XFP_OK = 0, XFP_ERR_CUDA = -2, XFP_ERR_TIMEOUT = -4 };
namespace xfp_host {
int fail(xfp_ctx* ctx, int code, const std::string& msg) {
  ctx->err = msg;
  return code;
}
int sweep_error(xfp_ctx* ctx, const Ctl& c) {
  return c.err ? fail(ctx, XFP_ERR_TIMEOUT, "site " + std::to_string(c.err_where)) : XFP_OK;
}
}  // namespace xfp_host
#define XFP_CUDA(ctx, call) \
  do { \
    if ((call) != cudaSuccess) return xfp_host::fail(ctx, XFP_ERR_CUDA, #call); \
  } while (0)
#include "../../xfluid_b200/csrc/xfp_loop.h"
namespace xfp {
thread_local long long g_kernel_launches = 0;
}

// ---- the runtime ----
static int instances = 0, execs = 0, launches = 0, drained = 0;   // live executables, graph launches, how many of them the host has waited for
static cudaError_t capture_result = cudaSuccess, instantiate_result = cudaSuccess, update_result = cudaSuccess;
extern "C" {
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) { *e = (cudaEvent_t)8; return cudaSuccess; }
cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned) { *s = (cudaStream_t)2; return cudaSuccess; }
cudaError_t cudaGetLastError() { return cudaSuccess; }
cudaError_t cudaStreamBeginCapture(cudaStream_t, cudaStreamCaptureMode) { return cudaSuccess; }
cudaError_t cudaStreamEndCapture(cudaStream_t, cudaGraph_t* g) {
  *g = capture_result == cudaSuccess ? (cudaGraph_t)16 : nullptr;
  return capture_result;
}
cudaError_t cudaGraphExecUpdate(cudaGraphExec_t, cudaGraph_t, cudaGraphExecUpdateResultInfo*) { return update_result; }
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t) { --execs; return cudaSuccess; }
cudaError_t cudaGraphInstantiate(cudaGraphExec_t* e, cudaGraph_t, unsigned long long) {
  if (instantiate_result != cudaSuccess) return instantiate_result;
  ++execs;
  ++instances;
  *e = (cudaGraphExec_t)32;
  return cudaSuccess;
}
cudaError_t cudaGraphDestroy(cudaGraph_t) { return cudaSuccess; }
cudaError_t cudaGraphLaunch(cudaGraphExec_t, cudaStream_t) { ++launches; return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamWaitEvent(cudaStream_t, cudaEvent_t, unsigned) { return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t s) {
  drained = s == (cudaStream_t)1 ? launches : launches - 1;
  return cudaSuccess;
}
const char* cudaGetErrorString(cudaError_t) { return ""; }
}

static void check(bool ok, const char* what) {
  if (ok) return;
  std::fprintf(stderr, "failed: %s\n", what);
  std::exit(1);
}

// a loop whose n-th read brings what `device` says (reads count from 1; `over`: the
// last launch had ended when the read was enqueued)
static int loop(xfp_ctx& ctx, const std::function<void(int, bool, xfp_ctx::Read&)>& device) {
  ctx.read = {};
  launches = drained = 0;
  int reads = 0;
  auto read = [&](cudaStream_t from) -> cudaError_t {
    device(++reads, from == ctx.stream, ctx.read);
    return cudaSuccess;
  };
  return xfp_host::replay_iterations(&ctx, 4, 5, 100, read, [&] { return ctx.read.sc.done != 0; });
}

int main(int argc, char** argv) {
  const std::string what = argc > 1 ? argv[1] : "";
  xfp_ctx ctx;
  check(xfp_host::capture_iterations(&ctx, 4, true, [](cudaStream_t) { return cudaSuccess; }), "capture");
  if (what == "half") {
    // the third read meets the end of the solve half-way: the flag is there, the
    // count and the residual are an older iteration's
    const int rc = loop(ctx, [](int n, bool, xfp_ctx::Read& r) {
      r.sc = n < 3 ? Scalars{5.0, 0, 4 * n} : n == 3 ? Scalars{5.0, 1, 8} : Scalars{1.0, 1, 10};
    });
    check(rc == XFP_OK && ctx.read.sc.iters == 10 && ctx.read.sc.res == 1.0, "scalars of the iteration that ended the solve");
  } else if (what == "expired") {
    // the record of an expired wait is whole once the launch is over
    const int rc = loop(ctx, [](int n, bool over, xfp_ctx::Read& r) {
      if (n >= 2) r.ctl = {1, over ? 8u : 0u};
    });
    check(rc == XFP_ERR_TIMEOUT && ctx.err == "site 8", "the site of the expired wait");
    check(drained == launches, "no launch under way after an error");
  } else if (what == "both") {
    // an expired wait that a breakdown follows
    const int rc = loop(ctx, [](int n, bool over, xfp_ctx::Read& r) {
      if (n >= 2) r.sc.done = 1;
      if (n >= 3) r.ctl = {1, over ? 8u : 0u};
    });
    check(rc == XFP_ERR_TIMEOUT && ctx.err == "site 8", "the expired wait before the breakdown");
  } else if (what == "endless") {
    check(loop(ctx, [](int, bool, xfp_ctx::Read&) {}) == XFP_ERR_CUDA, "a loop that does not end");
  } else if (what == "check_every") {
    // at most check_every iterations between reads, whether it is even or odd
    for (int k : {0, 1, 2, 3, 4, 5, 6, 7, 8, 25, 32}) {
      ctx.opt.check_every = k;
      check(xfp_host::loop_iterations(&ctx) == (k == 0 || k > 4 ? 4 : k), "iterations of a graph");
    }
  } else if (what == "kinds") {
    // a graph of cooperative launches is not updated into one of plain launches
    check(instances == 1 && xfp_host::capture_iterations(&ctx, 4, true, [](cudaStream_t) { return cudaSuccess; }), "updated");
    check(instances == 1, "the same kind is updated");
    check(xfp_host::capture_iterations(&ctx, 4, false, [](cudaStream_t) { return cudaSuccess; }), "the other kind");
    check(instances == 2 && execs == 1, "the other kind is instantiated, and the first given back");
  } else if (what == "refused") {
    // a capture that fails after one that did not leaves no executable graph behind
    capture_result = cudaErrorStreamCaptureInvalidated;
    check(!xfp_host::capture_iterations(&ctx, 4, true, [](cudaStream_t) { return cudaSuccess; }), "a refused capture");
    check(execs == 0 && ctx.loop_exec == nullptr, "the earlier graph given back");
    capture_result = cudaSuccess;
    check(!xfp_host::capture_iterations(&ctx, 4, true, [](cudaStream_t) { return cudaErrorInvalidValue; }), "a refused launch");
    check(execs == 0 && ctx.loop_exec == nullptr, "nothing kept");
    check(xfp_host::capture_iterations(&ctx, 4, true, [](cudaStream_t) { return cudaSuccess; }) && execs == 1, "a new graph");
    update_result = cudaErrorGraphExecUpdateFailure;
    check(xfp_host::capture_iterations(&ctx, 4, true, [](cudaStream_t) { return cudaSuccess; }) && execs == 1, "one in its place");
    instantiate_result = cudaErrorMemoryAllocation;
    check(!xfp_host::capture_iterations(&ctx, 4, true, [](cudaStream_t) { return cudaSuccess; }) && execs == 0, "no instance");
  } else {
    return 2;
  }
  std::printf("ok\n");
  return 0;
}

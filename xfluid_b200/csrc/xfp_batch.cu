// xfp_batch.cu -- xfp_project_batch_{f32,f64}: many independent scenes of
// different sizes projected together.
//
// Every scene gets its own line table, compact slice [base, base+M) of the
// shared compact arrays and its own PCG scalars, so each is solved exactly as
// a single-scene call solves it.  What is shared:
//   * the MIC(0) sweeps: the active tiles of all scenes form one list, merged
//     by wavefront level (J+K), and one persistent launch walks it.  A lone
//     256^3 wavefront leaves most SMs waiting on its dependency chain; the
//     tiles of other scenes fill them.
//   * the vector kernels: one launch per kernel covers all scenes, each scene
//     running the same block decomposition (and so the same reduction order)
//     as its single-scene launch would.
//   * a PCG loop's iterations (SpMV+dot, x/r update, forward, backward, rho/beta,
//     s update) are captured as a CUDA graph of min(check_every, 4) of them and
//     replayed until every scene has converged or hit its cap.
#include <algorithm>
#include <cmath>
#include <cstdio>
#include <cstring>
#include <string>
#include <type_traits>
#include <vector>

#include "xfp_context.h"

using namespace xfp;

namespace xfp_host {

struct BatchState {
  DevBuf lines, scene_tile_lists, counters;
  DevBuf segs, tile_scene, scal, scal2, part, tols, maxits;
  DevBuf io, pdense;
  std::vector<BatchSeg> hsegs;
  std::vector<long long> rows, nlines_act;
  int n = 0, ntiles = 0, blocks_cells = 0, blocks_groups = 0;
  long long M = 0;
};

void batch_state_free(BatchState* b) { delete b; }

namespace {

// One scene with its arrays on the device.
template <typename T>
struct DevScene {
  int ni, nj, nk;
  const uint8_t* mat;
  T *u, *v, *w;
  const T *wu, *wv, *ww;
  T* p;
};

// Line and block tables, compact and sweep slices, and the merged tile list.
template <typename T>
int batch_layout(xfp_ctx* ctx, BatchState* B, const std::vector<DevScene<T>>& S) {
  cudaStream_t st = ctx->stream;
  const int n = (int)S.size();
  std::vector<long long> line_base(n + 1, 0), blk_base(n + 1, 0);
  for (int s = 0; s < n; ++s) {
    line_base[s + 1] = line_base[s] + (long long)S[s].nj * S[s].nk;
    blk_base[s + 1] = blk_base[s] + (long long)((S[s].nj + 7) / 8) * ((S[s].nk + 7) / 8);
  }
  const long long nlines = line_base[n], nblk = blk_base[n];
  XFP_CUDA(ctx, B->lines.ensure(nlines * sizeof(Line)));
  XFP_CUDA(ctx, ctx->line_sums.ensure((size_t)std::min(n, LAYOUT_SCENES) * 3 * LINE_CHUNKS * sizeof(long long)));
  XFP_CUDA(ctx, ctx->blks.ensure((size_t)nblk * sizeof(WBlk)));
  XFP_CUDA(ctx, B->scene_tile_lists.ensure((size_t)nblk * sizeof(int2)));
  XFP_CUDA(ctx, B->counters.ensure((size_t)n * 5 * sizeof(long long)));
  Line* lines = B->lines.as<Line>();
  std::vector<LayoutScene> layouts(n);
  for (int s = 0; s < n; ++s)   // (the scratch is a launch's own)
    layouts[s] = {S[s].mat, S[s].ni, S[s].nj, S[s].nk, lines + line_base[s],
                  ctx->line_sums.as<long long>() + (size_t)(s % LAYOUT_SCENES) * 3 * LINE_CHUNKS,
                  ctx->blks.as<WBlk>() + blk_base[s], B->scene_tile_lists.as<int2>() + blk_base[s],
                  B->counters.as<long long>() + 5 * s};
  XFP_CUDA(ctx, layout_build(layouts.data(), n, st));
  std::vector<long long> cnt((size_t)n * 5);
  std::vector<int2> all_tiles((size_t)nblk);
  XFP_CUDA(ctx, cudaMemcpyAsync(cnt.data(), B->counters.p, cnt.size() * sizeof(long long), cudaMemcpyDeviceToHost,
                                st));
  XFP_CUDA(ctx, cudaMemcpyAsync(all_tiles.data(), B->scene_tile_lists.p, (size_t)nblk * sizeof(int2),
                                cudaMemcpyDeviceToHost, st));
  XFP_CUDA(ctx, cudaStreamSynchronize(st));
  // compact slices: scene s occupies [base_s, base_s + M_s); line offsets made
  // global.  Sweep slices: groups [group_base_s, ...).
  std::vector<long long> base(n + 1, 0), group_base(n + 1, 0);
  B->rows.assign(n, 0);
  B->nlines_act.assign(n, 0);
  for (int s = 0; s < n; ++s) {
    base[s + 1] = base[s] + cnt[5 * s];
    B->rows[s] = cnt[5 * s + 1];
    B->nlines_act[s] = cnt[5 * s + 2];
    group_base[s + 1] = group_base[s] + cnt[5 * s + 4];
  }
  if (base[n] >= (1LL << 31)) return fail(ctx, XFP_ERR_ARGS, "batch too large: more than 2^31 stored cells");
  if (group_base[n] * 256 >= (1LL << 31)) return fail(ctx, XFP_ERR_ARGS, "batch too large for the sweep layout");
  // group -> its neighbours (cells global) and group -> sweep element
  XFP_CUDA(ctx, ctx->gperm.ensure((std::max<long long>(base[n], 4) / 4 + 8) * sizeof(int)));
  XFP_CUDA(ctx, ctx->group_nb.ensure((std::max<long long>(base[n], 4) / 4 + 8) * sizeof(GroupNb)));
  std::vector<TableScene> tables(n);
  for (int s = 0; s < n; ++s)
    tables[s] = {lines + line_base[s], ctx->blks.as<WBlk>() + blk_base[s], S[s].nj, S[s].nk, base[s], group_base[s]};
  XFP_CUDA(ctx, layout_tables(tables.data(), n, ctx->group_nb.as<GroupNb>(), ctx->gperm.as<int>(), st));
  // merge the scenes' block lists by wavefront level (each list is already in
  // its own topological order, which the merge keeps)
  long long ntl = 0;
  for (int s = 0; s < n; ++s) ntl += cnt[5 * s + 3];
  const int nt = (int)ntl;
  std::vector<int2> tiles;
  std::vector<int> tscene;
  tiles.reserve(std::max(nt, 1));
  tscene.reserve(std::max(nt, 1));
  std::vector<long long> at(n, 0);
  for (int level = 0; (int)tiles.size() < nt; ++level)
    for (int s = 0; s < n; ++s)
      for (; at[s] < cnt[5 * s + 3]; ++at[s]) {
        const int2 t = all_tiles[blk_base[s] + at[s]];
        if (t.x + t.y != level) break;
        tiles.push_back(t);
        tscene.push_back(s);
      }
  if (nt == 0) {
    tiles.push_back(int2{0, 0});
    tscene.push_back(0);
  }
  // per-scene block decomposition of the vector kernels (as a single launch)
  B->hsegs.assign(n, BatchSeg{});
  XFP_CUDA(ctx, B->part.ensure((size_t)n * NBLK_MAX * sizeof(double)));
  int bc = 0, bg = 0;
  for (int s = 0; s < n; ++s) {
    BatchSeg& g = B->hsegs[s];
    const long long Ms = cnt[5 * s];
    g.ni = S[s].ni; g.nj = S[s].nj; g.nk = S[s].nk;
    // the cell-based kernels run one thread per 4-cell group (absmax_init strides
    // over single cells with the same blocks)
    g.blk_cells = (int)std::max<long long>(1, std::min<long long>((Ms / 4 + 255) / 256, NBLK_MAX));
    g.blk_cells_start = bc;
    // the SpMV's dot is summed over blocks: as many as a single scene's has
    g.blk_groups = (int)spmv_block_count(Ms, ctx->vec_blocks);
    g.blk_groups_start = bg;
    g.blk_base = blk_base[s];
    g.line_base = line_base[s];
    g.group_base = group_base[s];
    g.base = base[s];
    g.M = Ms;
    g.lines = lines + line_base[s];
    g.partials = B->part.as<double>() + (size_t)s * NBLK_MAX;
    bc += g.blk_cells;
    bg += g.blk_groups;
  }
  B->blocks_cells = bc;
  B->blocks_groups = bg;
  XFP_CUDA(ctx, B->segs.ensure(n * sizeof(BatchSeg)));
  XFP_CUDA(ctx, ctx->tiles.ensure(tiles.size() * sizeof(int2)));
  XFP_CUDA(ctx, B->tile_scene.ensure(tscene.size() * sizeof(int)));
  XFP_CUDA(ctx, cudaMemcpyAsync(B->segs.p, B->hsegs.data(), n * sizeof(BatchSeg), cudaMemcpyHostToDevice, st));
  XFP_CUDA(ctx, cudaMemcpyAsync(ctx->tiles.p, tiles.data(), tiles.size() * sizeof(int2), cudaMemcpyHostToDevice, st));
  XFP_CUDA(ctx, cudaMemcpyAsync(B->tile_scene.p, tscene.data(), tscene.size() * sizeof(int),
                                cudaMemcpyHostToDevice, st));
  // the host vectors above go out of scope: make the copies complete first
  XFP_CUDA(ctx, cudaStreamSynchronize(st));
  B->n = n;
  B->ntiles = nt;
  B->M = base[n];
  ctx->M = B->M;
  ctx->ntiles = nt;
  ctx->Gsw = group_base[n];
  ctx->nlines_all = line_base[n];
  return XFP_OK;
}

WaveArgs batch_args(xfp_ctx* ctx, BatchState* B, PcgScalars* sc) {
  WaveArgs g = wave_args(ctx);
  g.tile_scene = B->tile_scene.as<int>();
  g.segs = B->segs.as<BatchSeg>();
  g.scal_batch = sc;
  return g;
}

// Assembly of every scene into the shared compact arrays and sweep layout.
template <typename FT, typename AT>
int batch_assemble(xfp_ctx* ctx, BatchState* B, const std::vector<DevScene<FT>>& S, AT* const A[5]) {
  for (size_t s = 0; s < S.size(); ++s) {
    const BatchSeg& g = B->hsegs[s];
    XFP_CUDA(ctx, (assemble<FT, AT>(S[s].mat, S[s].u, S[s].v, S[s].w, S[s].wu, S[s].wv, S[s].ww, S[s].ni, S[s].nj,
                                    S[s].nk, g.lines, A[0], A[1], A[2], A[3], A[4], ctx->stream,
                                    XFP_MATRIX_VARIATIONAL, Force3(), nullptr, ctx->sw_sys.as<AT>(),
                                    ctx->blks.as<WBlk>() + g.blk_base, g.group_base)));
  }
  return XFP_OK;
}

// PCG (pcg_solver.h:243-285) on every scene at once.  Per-scene tolerance and
// cap come from tol/maxit, or from the device arrays tols/maxits when given.
// On return hsc holds each scene's final scalars.
template <typename VT, typename DT>
int batch_pcg(xfp_ctx* ctx, BatchState* B, const VT* const A[4], const VT* b, VT* x, VT* r, VT* s, VT* z, double tol,
              int maxit, const double* tols, const int* maxits, PcgScalars* dsc, std::vector<PcgScalars>& hsc, int maxit_all) {
  cudaStream_t st = ctx->stream;
  const int n = B->n;
  const size_t M = (size_t)std::max<long long>(B->M, 1);
  const BatchSeg* segs = B->segs.as<BatchSeg>();
  int rc0;
  if (tol < 1e-30) tol = 1e-30;
  XFP_CUDA(ctx, cudaMemsetAsync(x, 0, M * sizeof(VT), st));
  XFP_CUDA(ctx, cudaMemsetAsync(dsc, 0, n * sizeof(PcgScalars), st));
  XFP_CUDA(ctx, copy_vec<VT>(b, r, (long long)M, st));
  XFP_CUDA(ctx, batch_absmax_init<VT>(segs, n, B->blocks_cells, r, dsc, tol, maxit, tols, maxits, st));
  // the solves stream the sweep layout (as single scenes do): r copied in, z
  // gathered back through gperm
  if ((rc0 = sweep_rhs<VT>(ctx, r)) != XFP_OK) return rc0;
  const WaveArgs g = batch_args(ctx, B, dsc);
  const bool swl = B->ntiles > 0;
  VT* rsw = swl ? ctx->sw.as<VT>() + WAVE_R : nullptr;
  const VT* zsw = swl ? ctx->sw.as<VT>() + WAVE_Y : nullptr;
  const int* gperm = swl ? ctx->gperm.as<int>() : nullptr;
  const double* lpart = ctx->tpartials.as<double>();
  // lines of blocks without cells are never written: their partials stay zero
  XFP_CUDA(ctx, cudaMemsetAsync(ctx->tpartials.p, 0, std::max<long long>(ctx->nlines_all, 1) * sizeof(double), st));
  XFP_CUDA(ctx, (wave_launch<VT, DT>(SWEEP_FWD, g, st)));
  XFP_CUDA(ctx, (wave_launch<VT, DT>(SWEEP_BWD, g, st)));
  XFP_CUDA(ctx, batch_bwd_reduce<DT>(segs, n, lpart, dsc, 0, st));
  if ((rc0 = sweep_result<VT>(ctx, s)) != XFP_OK) return rc0;
  auto iteration = [&](cudaStream_t cs) -> cudaError_t {
    cudaError_t e;
    if ((e = batch_spmv_dot<VT, VT, DT>(segs, n, B->blocks_groups, A[0], A[1], A[2], A[3], s, z,
                                        ctx->group_nb.as<GroupNb>(), dsc, 0, cs)))
      return e;
    if ((e = batch_update_xr<VT>(segs, n, B->blocks_cells, x, r, s, z, dsc, cs, rsw, gperm))) return e;
    if ((e = wave_launch<VT, DT>(SWEEP_FWD, g, cs))) return e;
    if ((e = wave_launch<VT, DT>(SWEEP_BWD, g, cs))) return e;
    if ((e = batch_bwd_reduce<DT>(segs, n, lpart, dsc, 1, cs))) return e;
    return batch_update_s<VT>(segs, n, B->blocks_cells, s, z, dsc, cs, zsw, gperm);
  };
  const int K = ctx->opt.check_every > 0 ? ctx->opt.check_every : 8;
  const int per_iter = B->ntiles > 0 ? 6 : 4;
  // iterations as a graph, read after every launch of it; if that is refused,
  // launch directly
  const int per = loop_iterations(ctx);
  const bool graph = capture_iterations(ctx, per, B->ntiles > 1, iteration);
  ctx->loop_graph = graph;
  hsc.assign(n, PcgScalars{});
  int rc = XFP_OK;
  auto read = [&](cudaStream_t cs) -> cudaError_t {
    const cudaError_t e = cudaMemcpyAsync(hsc.data(), dsc, n * sizeof(PcgScalars), cudaMemcpyDeviceToHost, cs);
    if (e != cudaSuccess) return e;
    return cudaMemcpyAsync(&ctx->loop_read->ctl, ctx->ctl.p, sizeof(SweepCtl), cudaMemcpyDeviceToHost, cs);
  };
  auto done = [&] {
    bool all = true;
    for (int q = 0; q < n; ++q) all &= hsc[q].done != 0;
    return all;
  };
  if (graph) return replay_iterations(ctx, per, per_iter, maxit_all + 2 * K, read, done);
  for (int done_iters = 0;;) {
    for (int q = 0; q < K; ++q) XFP_CUDA(ctx, iteration(st));
    done_iters += K;
    XFP_CUDA(ctx, read(st));
    XFP_CUDA(ctx, cudaStreamSynchronize(st));
    if ((rc = sweep_error(ctx, ctx->loop_read->ctl)) != XFP_OK || done()) break;
    if (done_iters > maxit_all + 2 * K) return fail(ctx, XFP_ERR_CUDA, "batch PCG loop did not terminate");
  }
  return rc;
}

struct SceneResult {
  int status = XFP_OK, iters = 0, refinements = 0;
  double res = 0, bnorm = 0;
};

// Solve of every scene; the solution ends in x64 (F64, MIXED) or x32 (F32).
template <typename IOT>
int batch_solve(xfp_ctx* ctx, BatchState* B, const std::vector<DevScene<IOT>>& S, std::vector<SceneResult>& out) {
  const int prec = ctx->opt.precision, n = B->n;
  cudaStream_t st = ctx->stream;
  const double tol = ctx->opt.tol;
  const int maxit = ctx->opt.max_iter;
  const long long M = std::max<long long>(B->M, 1);
  XFP_CUDA(ctx, B->scal.ensure(n * sizeof(PcgScalars)));
  XFP_CUDA(ctx, B->scal2.ensure(n * sizeof(PcgScalars)));
  PcgScalars* dsc = B->scal.as<PcgScalars>();
  std::vector<PcgScalars> hsc;
  out.assign(n, SceneResult{});
  int rc;
  if (prec == XFP_PREC_F64 || prec == XFP_PREC_F32) {
    if (prec == XFP_PREC_F64) {
      double* A[5];
      for (int q = 0; q < 5; ++q) A[q] = ctx->A64[q].as<double>();
      if ((rc = batch_assemble<IOT, double>(ctx, B, S, A))) return rc;
      const double* Ac[4] = {A[0], A[1], A[2], A[3]};
      XFP_CUDA(ctx, (wave_launch<double, double>(SWEEP_FACTOR, batch_args(ctx, B, nullptr), st)));
      rc = batch_pcg<double, double>(ctx, B, Ac, A[4], ctx->x64.as<double>(), ctx->r64.as<double>(),
                                     ctx->s64.as<double>(), ctx->z64.as<double>(), tol, maxit, nullptr, nullptr, dsc,
                                     hsc, maxit);
    } else {
      float* A[5];
      for (int q = 0; q < 5; ++q) A[q] = ctx->A32[q].as<float>();
      if ((rc = batch_assemble<IOT, float>(ctx, B, S, A))) return rc;
      const float* Ac[4] = {A[0], A[1], A[2], A[3]};
      XFP_CUDA(ctx, (wave_launch<float, float>(SWEEP_FACTOR, batch_args(ctx, B, nullptr), st)));
      rc = batch_pcg<float, float>(ctx, B, Ac, A[4], ctx->x32.as<float>(), ctx->r32.as<float>(),
                                   ctx->s32.as<float>(), ctx->z32.as<float>(), tol, maxit, nullptr, nullptr, dsc, hsc,
                                   maxit);
    }
    if (rc < 0) return rc;
    for (int q = 0; q < n; ++q) {
      out[q].iters = hsc[q].iters;
      out[q].res = hsc[q].res;
      out[q].bnorm = hsc[q].bnorm;
      out[q].status = hsc[q].status == XFP_ERR_BREAKDOWN ? XFP_ERR_BREAKDOWN
                      : hsc[q].status == 0               ? XFP_OK
                                                         : XFP_NOT_CONVERGED;
    }
    return XFP_OK;
  }
  // ---- mixed: FP64 system and refinement per scene, FP32 inner PCG ----
  double* A[5];
  for (int q = 0; q < 5; ++q) A[q] = ctx->A64[q].as<double>();
  if ((rc = batch_assemble<IOT, double>(ctx, B, S, A))) return rc;
  float* A32[4];
  for (int q = 0; q < 4; ++q) {
    A32[q] = ctx->A32[q].as<float>();
    XFP_CUDA(ctx, (convert<double, float>(A[q], A32[q], M, st)));
  }
  // FP64 factor, streamed by the FP32 solves rounded to FP32 (as a single scene's mixed solve)
  XFP_CUDA(ctx, (wave_launch<float, double>(SWEEP_FACTOR, batch_args(ctx, B, nullptr), st)));
  const float* A32c[4] = {A32[0], A32[1], A32[2], A32[3]};
  double* x64 = ctx->x64.as<double>();
  double* r64 = ctx->r64.as<double>();
  PcgScalars* osc = B->scal2.as<PcgScalars>();
  const BatchSeg* segs = B->segs.as<BatchSeg>();
  std::vector<PcgScalars> ho(n);
  XFP_CUDA(ctx, cudaMemsetAsync(x64, 0, M * sizeof(double), st));
  XFP_CUDA(ctx, cudaMemsetAsync(osc, 0, n * sizeof(PcgScalars), st));
  XFP_CUDA(ctx, batch_absmax_init<double>(segs, n, B->blocks_cells, A[4], osc, tol, 1, nullptr, nullptr, st));
  XFP_CUDA(ctx, cudaMemcpyAsync(ho.data(), osc, n * sizeof(PcgScalars), cudaMemcpyDeviceToHost, st));
  XFP_CUDA(ctx, cudaStreamSynchronize(st));
  const double t0 = tol < 1e-30 ? 1e-30 : tol;
  std::vector<double> target(n), res(n), tols(n);
  std::vector<int> total(n, 0), cycles(n, 0), maxits(n);
  std::vector<char> fin(n, 0);
  for (int q = 0; q < n; ++q) {
    out[q].bnorm = ho[q].bnorm;
    target[q] = t0 * ho[q].bnorm;
    res[q] = ho[q].bnorm;
    fin[q] = ho[q].bnorm == 0.0;
    out[q].status = fin[q] ? XFP_OK : XFP_NOT_CONVERGED;
  }
  const int max_ref = ctx->opt.max_refine > 0 ? ctx->opt.max_refine : 20;
  const double floor_tol = ctx->opt.inner_tol > 0 ? ctx->opt.inner_tol : 1e-6;
  XFP_CUDA(ctx, B->tols.ensure(n * sizeof(double)));
  XFP_CUDA(ctx, B->maxits.ensure(n * sizeof(int)));
  for (int cyc = 0; cyc < max_ref; ++cyc) {
    if (cyc > 0) {
      XFP_CUDA(ctx, batch_residual64(segs, n, B->blocks_groups, A[0], A[1], A[2], A[3], A[4], x64, r64,
                                   ctx->group_nb.as<GroupNb>(), osc, st));
      XFP_CUDA(ctx, cudaMemcpyAsync(ho.data(), osc, n * sizeof(PcgScalars), cudaMemcpyDeviceToHost, st));
      XFP_CUDA(ctx, cudaStreamSynchronize(st));
      for (int q = 0; q < n; ++q) {
        if (fin[q]) continue;
        res[q] = ho[q].res;
        if (res[q] <= target[q]) { fin[q] = 1; out[q].status = XFP_OK; }
      }
      XFP_CUDA(ctx, (convert<double, float>(r64, ctx->r32.as<float>(), M, st)));
    } else {
      XFP_CUDA(ctx, (convert<double, float>(A[4], ctx->r32.as<float>(), M, st)));
    }
    bool any = false;
    for (int q = 0; q < n; ++q) {
      const bool run = !fin[q] && total[q] < maxit;
      any |= run;
      tols[q] = run ? std::min(0.5, std::max(floor_tol, 0.5 * target[q] / res[q])) : 0.5;
      maxits[q] = run ? maxit - total[q] : 0;
    }
    if (!any) break;
    XFP_CUDA(ctx, cudaMemcpyAsync(B->tols.p, tols.data(), n * sizeof(double), cudaMemcpyHostToDevice, st));
    XFP_CUDA(ctx, cudaMemcpyAsync(B->maxits.p, maxits.data(), n * sizeof(int), cudaMemcpyHostToDevice, st));
    float* b32 = ctx->A32[4].as<float>();
    XFP_CUDA(ctx, copy_vec<float>(ctx->r32.as<float>(), b32, M, st));
    std::vector<PcgScalars> hin;
    rc = batch_pcg<float, double>(ctx, B, A32c, b32, ctx->x32.as<float>(), ctx->r32.as<float>(),
                                  ctx->s32.as<float>(), ctx->z32.as<float>(), 0.5, maxit, B->tols.as<double>(), B->maxits.as<int>(), dsc, hin, maxit);
    if (rc < 0) return rc;
    for (int q = 0; q < n; ++q)
      if (maxits[q] > 0) {
        total[q] += hin[q].iters;
        cycles[q] += 1;
        if (hin[q].status == XFP_ERR_BREAKDOWN) { fin[q] = 1; out[q].status = XFP_ERR_BREAKDOWN; }
      }
    XFP_CUDA(ctx, refine_update(x64, ctx->x32.as<float>(), M, st));
  }
  // scenes that ran out of cycles or iterations: final residual decides
  bool open = false;
  for (int q = 0; q < n; ++q) open |= !fin[q];
  if (open) {
    XFP_CUDA(ctx, batch_residual64(segs, n, B->blocks_groups, A[0], A[1], A[2], A[3], A[4], x64, r64,
                                   ctx->group_nb.as<GroupNb>(), osc, st));
    XFP_CUDA(ctx, cudaMemcpyAsync(ho.data(), osc, n * sizeof(PcgScalars), cudaMemcpyDeviceToHost, st));
    XFP_CUDA(ctx, cudaStreamSynchronize(st));
    for (int q = 0; q < n; ++q)
      if (!fin[q]) {
        res[q] = ho[q].res;
        if (res[q] <= target[q]) out[q].status = XFP_OK;
      }
  }
  for (int q = 0; q < n; ++q) {
    out[q].iters = total[q];
    out[q].refinements = cycles[q];
    out[q].res = res[q];
  }
  return XFP_OK;
}

template <typename IOT>
int project_batch(xfp_ctx* ctx, int n, const xfp_scene* scenes, xfp_stats* stats) {
  if (!ctx) return XFP_ERR_ARGS;
  if (n < 1 || !scenes) return fail(ctx, XFP_ERR_ARGS, "batch needs n >= 1 scenes");
  if (ctx->opt.matrix != XFP_MATRIX_VARIATIONAL)
    return fail(ctx, XFP_ERR_UNSUPPORTED, "batched projection supports the variational matrix only");
  for (int s = 0; s < n; ++s) {
    const xfp_scene& c = scenes[s];
    int rc = check_dims(ctx, c.ni, c.nj, c.nk, c.material);
    if (rc) return fail(ctx, rc, "scene " + std::to_string(s) + ": " + ctx->err);
    if (!c.u || !c.v || !c.w) return fail(ctx, XFP_ERR_ARGS, "scene " + std::to_string(s) + ": velocity is NULL");
    if ((c.wu == nullptr) != (c.wv == nullptr) || (c.wu == nullptr) != (c.ww == nullptr))
      return fail(ctx, XFP_ERR_ARGS, "scene " + std::to_string(s) + ": face weights: pass all three or none");
  }
  XFP_CUDA(ctx, cudaSetDevice(ctx->device));
  if (!ctx->batch) ctx->batch = new BatchState();
  BatchState* B = ctx->batch;
  cudaStream_t st = ctx->stream;
  const long long launches0 = g_kernel_launches;
  cudaEvent_t ev[5];
  for (auto& e : ev) cudaEventCreate(&e);
  cudaEventRecord(ev[0], st);

  // ---- inputs on the device (staged into one buffer in host-pointer mode) ----
  std::vector<DevScene<IOT>> S(n);
  const bool host = !ctx->opt.device_pointers;
  size_t io_bytes = 0;
  auto al = [](size_t b) { return (b + 255) & ~(size_t)255; };
  for (int s = 0; s < n; ++s) {
    const xfp_scene& c = scenes[s];
    const size_t cells = (size_t)c.ni * c.nj * c.nk;
    const size_t fu = (size_t)(c.ni + 1) * c.nj * c.nk, fv = (size_t)c.ni * (c.nj + 1) * c.nk,
                 fw = (size_t)c.ni * c.nj * (c.nk + 1);
    io_bytes += al(cells) + 2 * al(fu * sizeof(IOT)) + 2 * al(fv * sizeof(IOT)) + 2 * al(fw * sizeof(IOT)) +
                al(cells * sizeof(IOT));
  }
  if (host) XFP_CUDA(ctx, B->io.ensure(io_bytes));
  {
    size_t off = 0;
    auto place = [&](const void* src, size_t bytes) -> void* {
      char* dst = B->io.as<char>() + off;
      off += al(bytes);
      if (src) cudaMemcpyAsync(dst, src, bytes, cudaMemcpyHostToDevice, st);
      return dst;
    };
    for (int s = 0; s < n; ++s) {
      const xfp_scene& c = scenes[s];
      DevScene<IOT>& d = S[s];
      d.ni = c.ni; d.nj = c.nj; d.nk = c.nk;
      const size_t cells = (size_t)c.ni * c.nj * c.nk;
      const size_t fu = (size_t)(c.ni + 1) * c.nj * c.nk, fv = (size_t)c.ni * (c.nj + 1) * c.nk,
                   fw = (size_t)c.ni * c.nj * (c.nk + 1);
      if (host) {
        d.mat = (const uint8_t*)place(c.material, cells);
        d.u = (IOT*)place(c.u, fu * sizeof(IOT));
        d.v = (IOT*)place(c.v, fv * sizeof(IOT));
        d.w = (IOT*)place(c.w, fw * sizeof(IOT));
        d.wu = c.wu ? (const IOT*)place(c.wu, fu * sizeof(IOT)) : nullptr;
        d.wv = c.wv ? (const IOT*)place(c.wv, fv * sizeof(IOT)) : nullptr;
        d.ww = c.ww ? (const IOT*)place(c.ww, fw * sizeof(IOT)) : nullptr;
        if (!c.wu) off += al(fu * sizeof(IOT)) + al(fv * sizeof(IOT)) + al(fw * sizeof(IOT));
        d.p = (IOT*)place(nullptr, cells * sizeof(IOT));
      } else {
        d.mat = c.material;
        d.u = (IOT*)c.u; d.v = (IOT*)c.v; d.w = (IOT*)c.w;
        d.wu = (const IOT*)c.wu; d.wv = (const IOT*)c.wv; d.ww = (const IOT*)c.ww;
        d.p = (IOT*)c.pressure;
      }
    }
  }
  // device-pointer mode without a pressure output: a scratch grid per scene
  if (!host) {
    size_t need = 0;
    for (int s = 0; s < n; ++s)
      if (!S[s].p) need += al((size_t)S[s].ni * S[s].nj * S[s].nk * sizeof(IOT));
    if (need) {
      XFP_CUDA(ctx, B->pdense.ensure(need));
      size_t off = 0;
      for (int s = 0; s < n; ++s)
        if (!S[s].p) {
          S[s].p = (IOT*)(B->pdense.as<char>() + off);
          off += al((size_t)S[s].ni * S[s].nj * S[s].nk * sizeof(IOT));
        }
    }
  }

  // ---- layout ----
  const int prec = ctx->opt.precision;
  int rc;
  if ((rc = batch_layout<IOT>(ctx, B, S))) return rc;
  if ((rc = ensure_compact(ctx, prec))) return rc;
  cudaEventRecord(ev[1], st);

  // ---- solve ----
  std::vector<SceneResult> res;
  if ((rc = batch_solve<IOT>(ctx, B, S, res)) < 0) return rc;
  cudaEventRecord(ev[2], st);

  // ---- pressure on the dense grids, velocity update ----
  const long long M = std::max<long long>(B->M, 1);
  const bool sol64 = prec != XFP_PREC_F32;
  const void* xsol = sol64 ? (const void*)ctx->x64.p : (const void*)ctx->x32.p;
  if (sol64 != std::is_same<IOT, double>::value) {
    if (sol64) {
      XFP_CUDA(ctx, (convert<double, float>(ctx->x64.as<double>(), ctx->s32.as<float>(), M, st)));
      xsol = ctx->s32.p;
    } else {
      XFP_CUDA(ctx, ctx->r64.ensure(M * 8 + 64));
      XFP_CUDA(ctx, (convert<float, double>(ctx->x32.as<float>(), ctx->r64.as<double>(), M, st)));
      xsol = ctx->r64.p;
    }
  }
  for (int s = 0; s < n; ++s) {
    const DevScene<IOT>& d = S[s];
    XFP_CUDA(ctx, scatter_dense<IOT>((const IOT*)xsol, B->hsegs[s].lines, d.ni, d.nj, d.nk, d.p, st));
    XFP_CUDA(ctx, (apply_pressure<IOT, IOT>(d.mat, d.wu, d.wv, d.ww, d.p, d.ni, d.nj, d.nk, d.u, d.v, d.w, st)));
  }
  cudaEventRecord(ev[3], st);
  if (host) {
    for (int s = 0; s < n; ++s) {
      const xfp_scene& c = scenes[s];
      const DevScene<IOT>& d = S[s];
      const size_t cells = (size_t)c.ni * c.nj * c.nk;
      const size_t fu = (size_t)(c.ni + 1) * c.nj * c.nk, fv = (size_t)c.ni * (c.nj + 1) * c.nk,
                   fw = (size_t)c.ni * c.nj * (c.nk + 1);
      XFP_CUDA(ctx, cudaMemcpyAsync(c.u, d.u, fu * sizeof(IOT), cudaMemcpyDeviceToHost, st));
      XFP_CUDA(ctx, cudaMemcpyAsync(c.v, d.v, fv * sizeof(IOT), cudaMemcpyDeviceToHost, st));
      XFP_CUDA(ctx, cudaMemcpyAsync(c.w, d.w, fw * sizeof(IOT), cudaMemcpyDeviceToHost, st));
      if (c.pressure)
        XFP_CUDA(ctx, cudaMemcpyAsync(c.pressure, d.p, cells * sizeof(IOT), cudaMemcpyDeviceToHost, st));
    }
  }
  cudaEventRecord(ev[4], st);
  XFP_CUDA(ctx, cudaStreamSynchronize(st));
  float ms[4] = {0, 0, 0, 0};
  for (int q = 0; q < 4; ++q) cudaEventElapsedTime(&ms[q], ev[q], ev[q + 1]);
  for (auto& e : ev) cudaEventDestroy(e);

  int status = XFP_OK;
  for (int s = 0; s < n; ++s) {
    if (res[s].status == XFP_ERR_BREAKDOWN && status == XFP_OK) status = XFP_NOT_CONVERGED;
    if (res[s].status == XFP_NOT_CONVERGED) status = XFP_NOT_CONVERGED;
  }
  if (stats) {
    const long long launches = g_kernel_launches - launches0;
    for (int s = 0; s < n; ++s) {
      xfp_stats& o = stats[s];
      memset(&o, 0, sizeof(o));
      o.status = res[s].status;
      o.iterations = res[s].iters;
      o.refinements = res[s].refinements;
      o.residual = res[s].res;
      o.b_inf = res[s].bnorm;
      o.rel_residual = res[s].bnorm > 0 ? res[s].res / res[s].bnorm : 0.0;
      o.rows = B->rows[s];
      o.stored = B->hsegs[s].M;
      o.lines = B->nlines_act[s];
      // batch-wide timings (the scenes share every launch)
      o.ms_setup = ms[0];
      o.ms_solve = ms[1];
      o.ms_apply = ms[2];
      o.ms_total = ms[0] + ms[1] + ms[2] + ms[3];
      const double bpr = prec == XFP_PREC_F64 ? 224.0 : 112.0;   // FP32 pivots in the mixed solves
      const double cells = (double)scenes[s].ni * scenes[s].nj * scenes[s].nk;
      o.bytes = bpr * (double)o.rows * o.iterations + 33.0 * cells + 24.0 * (double)o.rows + 29.0 * cells;
      o.launches = launches;
      o.tile_k = ctx->nw;
      o.graph = ctx->loop_graph ? 1 : 0;
    }
  }
  return status;
}

}  // namespace
}  // namespace xfp_host

extern "C" int xfp_project_batch_f32(xfp_ctx* ctx, int n, const xfp_scene* scenes, xfp_stats* stats) {
  return xfp_host::project_batch<float>(ctx, n, scenes, stats);
}
extern "C" int xfp_project_batch_f64(xfp_ctx* ctx, int n, const xfp_scene* scenes, xfp_stats* stats) {
  return xfp_host::project_batch<double>(ctx, n, scenes, stats);
}

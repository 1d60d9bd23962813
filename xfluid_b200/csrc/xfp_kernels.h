// xfp_kernels.h -- host-side launchers of libxfp's device kernels (internal).
#pragma once

#include <cstdint>
#include <cuda_runtime.h>

#include "xfp_common.cuh"

namespace xfp {

enum { SWEEP_FACTOR = 0, SWEEP_FWD = 1, SWEEP_BWD = 2 };

// Kernels launched by this library in this thread (every launcher adds its
// launches); a call reports the difference across its own work.
extern thread_local long long g_kernel_launches;

// A launch of one of the PCG loop's kernels (start_next, wait_previous).
template <typename... P, typename... A>
cudaError_t launch_next(void (*kernel)(P...), unsigned blocks, unsigned threads, cudaStream_t st, A... args) {
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.gridDim = dim3(blocks);
  cfg.blockDim = dim3(threads);
  cfg.stream = st;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  ++g_kernel_launches;
  return cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(args)...);
}

// One launch of the wavefront kernel (xfp_wave.cu): blocks, control, operands.
struct WaveArgs {
  int nj = 0, nk = 0;           // lines along j and k (one scene)
  int NJB = 0, NKB = 0;         // 8 x 8-line blocks along j and k (one scene)
  int ntiles = 0;
  const int2* tiles = nullptr;  // active tiles (J, K), topological order
  const WBlk* blks = nullptr;   // block table(s), [K * NJB + J]
  SweepCtl* ctl = nullptr;
  long long spin_limit = 0;
  PcgScalars* scal = nullptr;   // forward/backward: skip when done; backward: rho/beta
  int bwd_mode = 0;             // backward: 0 = initial rho, 1 = beta update
  // Batch of scenes (null for one scene): scene of each tile, per-scene
  // geometry and scalars.  Tiles of a converged scene are skipped, and the
  // backward dot partials are reduced per scene by batch_bwd_reduce.
  const int* tile_scene = nullptr;
  const BatchSeg* segs = nullptr;
  PcgScalars* scal_batch = nullptr;
  // Diagnostic (xfp_debug_expire_next_sweep): edge words are expected with
  // generation + expect_bias, which no producer writes, so the bounded waits
  // run out.  0 in normal operation.
  unsigned expect_bias = 0;
  double omega = 0.97, ratio = 0.25;
  // sweep-layout arrays; the factor and the system keep four values per cell
  // (wave_cell_slot): (px, py, pz, inv) and (diag, A(c+1,c), A(c+ni,c), A(c+nn,c))
  const void* sys = nullptr;    // factor: the system, arithmetic type
  void* sw = nullptr;           // rows of WAVE_ROW values, solve type: the factor; r (backward: for
                                // z.r); y (backward: in y, out z)
  double* partials = nullptr;   // backward: z.r per line, [k * nj + j]
  unsigned long long* bj = nullptr;   // block-edge words of the J and K neighbours
  unsigned long long* bk = nullptr;
};
// VT: the solves' value type and the stored factor's; CT: the factorisation's
// arithmetic and the dot type of the backward solve.
template <typename VT, typename CT>
cudaError_t wave_launch(int op, const WaveArgs& g, cudaStream_t st);
// What a first launch of the solves looks up, ahead of it (outside a capture).
template <typename VT, typename CT>
cudaError_t wave_prepare();
// 64-bit words of the J and K edges per group: 4 steps x 8 lines of up to 16
// bytes (the factorisation's FP64 pair), 32 payload bits a word
constexpr size_t WAVE_EDGE = 4 * 8 * 4;

// dir 0: sw[wave_value(gperm)] = line; dir 1: the way back, for the M stored cells.
template <typename T>
cudaError_t sw_permute(T* line, T* sw, const int* gperm, long long M, int dir, cudaStream_t st);
// The factor back in the line layout: F = lx, ly, lz (keyed by the higher cell), inv.
template <typename T>
cudaError_t factor_lines(const T* fac, const Line* lines, int nj, int nk, const WBlk* blks, int NJB, T* const F[4],
                         cudaStream_t st);

// ---- layout (xfp_layout.cu) ----
// Builds the line table, the block table and the active-tile list for a
// material grid.  counters (device): stored cells M, unknown rows, active
// lines, active tiles, sweep-layout groups.
constexpr int LINE_CHUNKS = 1024;
constexpr int LAYOUT_SCENES = 16;   // grids a launch of the layout kernels takes
struct LayoutScene {
  const uint8_t* mat;
  int ni, nj, nk;
  Line* lines;               // [nk*nj]
  long long* sums;           // scratch [3 * LINE_CHUNKS]
  WBlk* blks;                // [ceil(nk/8) * ceil(nj/8)]
  int2* tiles;               // active tiles (at most as many as blocks)
  long long* counters;       // [5]
};
cudaError_t layout_build(const LayoutScene* scenes, int n, cudaStream_t st);
// Per aligned 4-cell group: its neighbours and its place in the sweep layout.  The
// grids' cells follow one another from `base` on, their groups of the sweep layout
// from group_base on.  Line offsets are made global.
struct TableScene {
  Line* lines;
  const WBlk* blks;
  int nj, nk;
  long long base, group_base;
};
cudaError_t layout_tables(const TableScene* scenes, int n, GroupNb* group_nb, int* gperm, cudaStream_t st);

// ---- assembly / apply / vector kernels (xfp_ops.cu) ----
template <typename FT, typename AT>
cudaError_t assemble(const uint8_t* mat, const FT* u, const FT* v, const FT* w, const FT* wu,
                     const FT* wv, const FT* ww, int ni, int nj, int nk, const Line* lines,
                     AT* diag, AT* ax, AT* ay, AT* az, AT* b, cudaStream_t st,
                     int matrix = XFP_MATRIX_VARIATIONAL, Force3 frc = Force3(),
                     float* const A32[4] = nullptr,    // also write diag..az as FP32 (mixed form)
                     AT* sys = nullptr, const WBlk* blks = nullptr, long long group_base = 0);
// sys: the factorisation's operands in the sweep layout (zeroed by the caller)

template <typename T>
cudaError_t scatter_dense(const T* x, const Line* lines, int ni, int nj, int nk, T* dense,
                          cudaStream_t st);
// Host-pointer mode, sparse face transfer (xfp_hostio.cu): fluid span of
// every x-line ({first, last + 1}, or {0, 0}), and the copy of every face
// row's fluid-bordering span of u, v, w from src to dst (either side may be
// page-locked host memory addressed in place); *bytes accumulates the bytes.
cudaError_t fluid_spans(const uint8_t* mat, int ni, int nj, int nk, int2* span, cudaStream_t st);
template <typename T>
cudaError_t face_rows_copy(const int2* span, int ni, int nj, int nk, const T* const src[3], T* const dst[3],
                           unsigned long long* bytes, cudaStream_t st);

template <typename FT, typename PT>
cudaError_t apply_pressure(const uint8_t* mat, const FT* wu, const FT* wv, const FT* ww,
                           const PT* p, int ni, int nj, int nk, FT* u, FT* v, FT* w,
                           cudaStream_t st, int matrix = XFP_MATRIX_VARIATIONAL, Force3 frc = Force3());
// FluidSimulator::_applyForces (FluidSimulator.cpp:429-499) as one pass.
template <typename FT>
cudaError_t apply_forces(const uint8_t* mat, int ni, int nj, int nk, FT* u, FT* v, FT* w, Force3 frc,
                         cudaStream_t st);
// FluidSimulator::_expolateVelocity(layers, axis) for the three axes
// (FluidSimulator.cpp:521-650); scratch: extrapolate_scratch bytes.
size_t extrapolate_scratch(int ni, int nj, int nk);
template <typename FT>
cudaError_t extrapolate(const uint8_t* mat, int ni, int nj, int nk, FT* u, FT* v, FT* w, int layers,
                        unsigned* scratch, cudaStream_t st);
template <typename FT>
cudaError_t divergence(const uint8_t* mat, int ni, int nj, int nk, const FT* u, const FT* v, const FT* w, FT* div,
                       cudaStream_t st);
template <typename FT, typename PT>
cudaError_t apply_pressure_T(const uint8_t* mat, const FT* wu, const FT* wv, const FT* ww,
                             const FT* gu, const FT* gv, const FT* gw, int ni, int nj, int nk,
                             const Line* lines, PT* q, cudaStream_t st);
template <typename FT, typename PT>
cudaError_t rhs_T(const uint8_t* mat, const FT* wu, const FT* wv, const FT* ww, const PT* lam,
                  const Line* lines, int ni, int nj, int nk, const FT* gu, const FT* gv,
                  const FT* gw, FT* du, FT* dv, FT* dw, cudaStream_t st);

// PCG vector kernels over the compact arrays (length M).
// z = A s with the fused dot s.z; one thread per aligned 4-cell group.
template <typename VT, typename AT, typename DT>
cudaError_t spmv_dot(const AT* diag, const AT* ax, const AT* ay, const AT* az, const VT* s, VT* z,
                     const GroupNb* group_nb, long long M, PcgScalars* sc, DT* partials, int nblk_max, int mode,
                     cudaStream_t st);
// SpMV blocks for M stored cells (the batch gives each scene the same count).
long long spmv_block_count(long long M, int nblk_max);
// rsw/gperm (optional): the updated r is also stored at rsw[wave_value(gperm[c / 4])].
template <typename VT, typename DT>
cudaError_t update_xr(VT* x, VT* r, const VT* s, const VT* z, long long M, PcgScalars* sc,
                      double* partials, int nblk_max, cudaStream_t st, VT* rsw = nullptr,
                      const int* gperm = nullptr);
// zsw/gperm (optional): z is read from zsw[wave_value(gperm[c / 4])] instead of z[c].
template <typename VT>
cudaError_t update_s(VT* s, const VT* z, long long M, PcgScalars* sc, cudaStream_t st, const VT* zsw = nullptr,
                     const int* gperm = nullptr, int nblk_max = 148 * 16);
template <typename VT>
cudaError_t absmax_init(const VT* b, long long M, PcgScalars* sc, double* partials, int nblk_max,
                        double tol, int maxit, cudaStream_t st);
template <typename A, typename B>
cudaError_t convert(const A* in, B* out, long long n, cudaStream_t st);
template <typename T>
cudaError_t gather_compact(const T* dense, const Line* lines, int ni, int nj, int nk, T* x,
                           cudaStream_t st);
template <typename T>
cudaError_t copy_vec(const T* in, T* out, long long n, cudaStream_t st);

// ---- batch forms: one launch covers every scene of a batch (BatchSeg table,
// nseg scenes, per-scene scalars sc[nseg]); grid = the table's total blocks ----
template <typename VT, typename AT, typename DT>
cudaError_t batch_spmv_dot(const BatchSeg* segs, int nseg, int blocks, const AT* diag, const AT* ax,
                           const AT* ay, const AT* az, const VT* s, VT* z, const GroupNb* group_nb, PcgScalars* sc,
                           int mode, cudaStream_t st);
// rsw/gperm, zsw/gperm (optional): as update_xr / update_s, gperm indexed by global group
template <typename VT>
cudaError_t batch_update_xr(const BatchSeg* segs, int nseg, int blocks, VT* x, VT* r, const VT* s,
                            const VT* z, PcgScalars* sc, cudaStream_t st, VT* rsw = nullptr,
                            const int* gperm = nullptr);
template <typename VT>
cudaError_t batch_update_s(const BatchSeg* segs, int nseg, int blocks, VT* s, const VT* z, PcgScalars* sc,
                           cudaStream_t st, const VT* zsw = nullptr, const int* gperm = nullptr);
// tols/maxits: optional per-scene tolerance and iteration cap (else tol, maxit)
template <typename VT>
cudaError_t batch_absmax_init(const BatchSeg* segs, int nseg, int blocks, const VT* b, PcgScalars* sc,
                              double tol, int maxit, const double* tols, const int* maxits, cudaStream_t st);
cudaError_t batch_residual64(const BatchSeg* segs, int nseg, int blocks, const double* diag, const double* ax,
                             const double* ay, const double* az, const double* b, const double* x, double* r,
                             const GroupNb* group_nb, PcgScalars* sc, cudaStream_t st);
// Per-scene z.r from the backward sweep's line partials, in the single-scene
// order; mode 0: rho, mode 1: beta and rho.
template <typename DT>
cudaError_t batch_bwd_reduce(const BatchSeg* segs, int nseg, const double* line_partials, PcgScalars* sc, int mode,
                             cudaStream_t st);
// ---- semi-Lagrangian MAC self-advection and its adjoint (xfp_advect.cu) ----
template <typename T>
cudaError_t advect(const T* u, const T* v, const T* w, T* ou, T* ov, T* ow, int ni, int nj, int nk, T c,
                   cudaStream_t st);
template <typename T>
cudaError_t advect_adjoint(const T* u, const T* v, const T* w, const T* gu, const T* gv, const T* gw, T* du,
                           T* dv, T* dw, int ni, int nj, int nk, T c, cudaStream_t st);
template <typename T>
cudaError_t box_loss(const T* u, const T* v, const T* w, T* gu, T* gv, T* gw, int ni, int nj, int nk,
                     const double box[6], double* loss, cudaStream_t st);

// Mixed precision: r64 = b64 - A64 x64, |r|_inf and r32 = (float) r64 / scale.
cudaError_t residual64(const double* diag, const double* ax, const double* ay, const double* az, const double* b,
                       const double* x, double* r, const GroupNb* group_nb, long long M, PcgScalars* sc,
                       double* partials, int nblk_max, cudaStream_t st);
cudaError_t refine_update(double* x64, const float* e32, long long M, cudaStream_t st);

}  // namespace xfp

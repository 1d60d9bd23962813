// xfp_common.cuh -- shared device helpers and layout structures for libxfp.
//
// Storage layout ("line-compacted"): the grid is cut into x-lines, one per
// (j,k).  Each line that holds an unknown stores the cells [lo, lo+len)
// contiguously at offset `off` in every per-cell array: lo is the first
// unknown moved down by 0..3 cells so that lo + j + k = 0 (mod XFP_ALIGN), len
// is rounded up to a multiple of XFP_ALIGN, and off is a multiple of
// XFP_ALIGN.  Cell (i,j,k) therefore sits at an address = i + j + k (mod
// XFP_ALIGN): every cell of one wavefront hyperplane i+j+k = t has the same
// position inside its aligned group of XFP_ALIGN cells, which is what lets
// the triangular-solve sweeps move whole groups with one vector access.  lo
// may be negative and lo+len may pass ni; cells inside a span that are not
// unknowns (air, uncoupled solid, outside the grid) are padding: zero
// coefficients, zero vectors, null rows.
#pragma once

#include <cstdint>
#include <cuda_runtime.h>

#define XFP_ALIGN 4
#define XFP_FULL 0xffffffffu
#ifndef XFP_MATRIX_NORMAL   // the same values as include/xfp.h
#define XFP_MATRIX_VARIATIONAL 0
#define XFP_MATRIX_NORMAL 1
#endif

namespace xfp {

enum : uint8_t { MAT_AIR = 0, MAT_FLUID = 1, MAT_SOLID = 2 };

// Per-line record: off (start in compact arrays), lo (first stored i), len
// (stored cells, 0 = line has no unknown), nrows (unknowns on the line).
struct __align__(16) Line {
  int off, lo, len, nrows;
};

// Constant body-force velocity increment (force * dt per axis), added to every
// face that borders a fluid cell, as xFluid's FluidSimulator::_applyForces does
// (FluidSimulator.cpp:429-499): an axis whose |dv| is not above 1e-10 is left
// alone.  on = 0: no force.
struct Force3 {
  double d[3] = {0.0, 0.0, 0.0};
  int on = 0;
  __host__ __device__ bool axis_on(int a) const { return on && (d[a] > 1e-10 || d[a] < -1e-10); }
};

// Sweep layout: the arrays the MIC(0) sweeps stream, in the order they use
// them.  The lines are cut into blocks of 8 x 8 (j, k); a block's cells are kept
// by groups of 4 wavefront steps t = i+j+k, group g holding steps 4g..4g+3.
// Element [(goff + g - g0)*256 + wave_line_slot(j, k) + (t & 3)] is line (j,k)'s
// cell of step t, zero where the line has none.  g0/ng: the block's first
// group and group count; goff: its first group in the arrays (scene-relative
// in a batch: BatchSeg::group_base).  ng = 0: no cells.
struct __align__(16) WBlk {
  int goff, g0, ng, pad;
};
// The factor (px, py, pz, inv) and the factorisation's system (diag and the
// couplings to the higher cells) keep four values per cell, 1024 per group:
// value a of line (j,k)'s cell of step 4g+e, so that a warp's step reads whole
// 16-byte units of consecutive cells and each half of a block (k & 4) is contiguous.
template <typename T>
__host__ __device__ __forceinline__ int wave_cell_slot(int j, int k, int e, int a) {
  constexpr int V = 16 / (int)sizeof(T), U = 4 / V;   // values per unit, units per cell
  return (((((k & 7) >> 2) * 4 + e) * U + a / V) * 32 + (k & 3) * 8 + (j & 7)) * V + a % V;
}
// The wavefront kernel's clusters: WAVE_TJ x 2 CTAs of two blocks along k, a tile
// of WAVE_TJ x WAVE_TK blocks (32 x 32 lines)
constexpr int WAVE_TJ = 4, WAVE_TK = 4, WAVE_CLUSTER = 8;
// A group's row of the solves' array: the factor's four values of its 256 cells,
// then r, then y (the backward solve's z).
constexpr int WAVE_R = 4 * 256, WAVE_Y = 5 * 256, WAVE_ROW = 6 * 256;
// element p = group * 256 + wave_line_slot of r or y, from the array's WAVE_R or WAVE_Y on
__host__ __device__ __forceinline__ size_t wave_value(int p) { return (size_t)(p >> 8) * WAVE_ROW + (p & 255); }
__host__ __device__ __forceinline__ int wave_line_slot(int j, int k) {
  return (k & 1) * 128 + (((k & 7) >> 1) * 8 + (j & 7)) * 4;
}

// Where the y and z neighbours (j -+ 1, k -+ 1) of a 4-cell group are stored: a
// neighbour line holds the first of them in the quad before quad q and the last in
// quad q, (q << 2) | (1: it stores the first quad) | (2: it stores the second).
struct __align__(16) GroupNb {
  unsigned ym, yp, zm, zp;
};

// The PCG loop's kernels start while the one before them ends (programmatic
// dependent launch): each waits, in all its threads and before it touches what
// another kernel writes, until its predecessors are complete and their writes
// visible.  The vector kernels let the next one start as soon as all their own CTAs
// run; the sweeps do not, since CTAs that wait beside them take their places on the
// SMs (a half-full 256^3 projection took 11.0 ms so, 10.3 without).
__device__ __forceinline__ void start_next() { asm volatile("griddepcontrol.launch_dependents;"); }
__device__ __forceinline__ void wait_previous() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

// Control block of the persistent sweep kernels (one per context).
struct SweepCtl {
  unsigned int gen;        // launch generation; stamped words carry it in their high half
  unsigned int finished;   // CTAs finished in the current launch
  unsigned int err;        // nonzero: a bounded wait ran out (XFP_ERR_TIMEOUT)
  unsigned int err_where;  // which wait ran out first (diagnostics)
  int err_tile, err_tau, err_thread, err_op;
  unsigned long long err_word;   // the word the failed wait last saw
  unsigned int err_expect;
  unsigned int ticket;           // tiles handed out in the current launch
};

// One scene of a batch: its grid, its slice [base, base+M) of the compact
// arrays, its line table (offsets already global) and the blocks the vector
// kernels give it (line-based and cell-based grids, consecutive per scene).
struct BatchSeg {
  int ni, nj, nk;
  int blk_cells, blk_cells_start;   // cell-based kernels (updates, norms)
  int blk_groups, blk_groups_start; // the SpMV and the residual (one thread per 4-cell group)
  long long blk_base, group_base;   // first entry of this scene's block table, first group of its sweep slice
  long long line_base;              // its first line among all scenes'
  long long base, M;
  const Line* lines;
  double* partials;                 // this scene's reduction slots
};

// The sum of n per-line partials, in a fixed order: 256 chunks of C consecutive
// lines, each summed in line order, then a fixed tree.  A lane's chain of C
// additions is what it costs, so the chunks go to as many warps as there are:
// a warp takes NCH chunks from `first` on (lane q's sum in lane q), P lines of
// each at a time through buf, NCH * (P + 1) words of its own.
template <bool F32, int NCH, int P>
__device__ __forceinline__ double chunk_sums(const double* __restrict__ part, long long n, int first, double* buf) {
  const int lane = threadIdx.x & 31;
  const long long C = (n + 255) / 256;
  double acc = 0.0;
  float accf = 0.f;
  for (long long o = 0; o < C; o += P) {
    double v[NCH * P / 32];
#pragma unroll
    for (int i = 0; i < NCH * P / 32; ++i) {
      const int e = i * 32 + lane;
      const long long w = o + e % P, q = (first + e / P) * C + w;
      v[i] = w < C && q < n ? __ldcg(part + q) : 0.0;
    }
    __syncwarp();
#pragma unroll
    for (int i = 0; i < NCH * P / 32; ++i) {
      const int e = i * 32 + lane;
      buf[(e / P) * (P + 1) + e % P] = v[i];
    }
    __syncwarp();
    if (lane < NCH) {
      const int m = C - o < P ? (int)(C - o) : P;
#pragma unroll 8
      for (int w = 0; w < m; ++w) {
        const double x = buf[lane * (P + 1) + w];
        if (F32) accf = __fadd_rn(accf, (float)x); else acc = __dadd_rn(acc, x);
      }
    }
  }
  return F32 ? (double)accf : acc;
}
// the tree over the 256 chunk sums, by one warp; returned to lane 0
template <bool F32>
__device__ __forceinline__ double chunk_tree(const double* s) {
  auto add = [](double a, double b) { return F32 ? (double)__fadd_rn((float)a, (float)b) : __dadd_rn(a, b); };
  double v[8];
#pragma unroll
  for (int m = 0; m < 8; ++m) v[m] = s[(threadIdx.x & 31) + 32 * m];
#pragma unroll
  for (int h = 4; h > 0; h >>= 1)
#pragma unroll
    for (int m = 0; m < h; ++m) v[m] = add(v[m], v[m + h]);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v[0] = add(v[0], __shfl_down_sync(XFP_FULL, v[0], o));
  return v[0];
}

// Scalars of one PCG solve, resident on the device.
struct PcgScalars {
  double rho, alpha, beta, res, tolabs, bnorm, dot_tmp;
  int done, iters, status, maxit;
  unsigned int red_count;  // last-block-done counter of the reductions
  unsigned int pad;
};

// Ends a solve.  The host may read the scalars beside the kernel that does: `done`
// goes last, behind a fence, so that whoever sees it finds the others in place.
__device__ __forceinline__ void end_solve(PcgScalars* sc, int status) {
  sc->status = status;
  __threadfence_system();
  *(volatile int*)&sc->done = 1;
}

__device__ __forceinline__ unsigned int ld_volatile_u32(const unsigned int* p) {
  return *(const volatile unsigned int*)p;
}

// Rounded arithmetic without contraction: the FP64 path follows xFluid's
// operation order exactly, so no multiply-add may be fused.
__device__ __forceinline__ double mul_rn(double a, double b) { return __dmul_rn(a, b); }
__device__ __forceinline__ float mul_rn(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ double add_rn(double a, double b) { return __dadd_rn(a, b); }
__device__ __forceinline__ float add_rn(float a, float b) { return __fadd_rn(a, b); }
__device__ __forceinline__ double sub_rn(double a, double b) { return __dsub_rn(a, b); }
__device__ __forceinline__ float sub_rn(float a, float b) { return __fsub_rn(a, b); }
__device__ __forceinline__ double div_rn(double a, double b) { return __ddiv_rn(a, b); }
__device__ __forceinline__ float div_rn(float a, float b) { return __fdiv_rn(a, b); }
// 1 / sqrt(x), both rounded as the reference rounds them: the reciprocal is the
// correctly rounded quotient 1 / y, in fewer steps than a division
__device__ __forceinline__ double rsqrt_ref(double x) { return __drcp_rn(__dsqrt_rn(x)); }
__device__ __forceinline__ float rsqrt_ref(float x) { return __frcp_rn(__fsqrt_rn(x)); }

// One group of XFP_ALIGN (4) consecutive cells of an array, from/to a
// group-aligned index: one 16-byte access (FP32) or two (FP64).  Groups of 8
// with 32-byte accesses were measured too in the sweeps: faster on long full
// lines, slower on the 256^3 blob scene (more padding steps, more registers).
__device__ __forceinline__ void ldg(float (&v)[4], const float* p) {
  const float4 t = *reinterpret_cast<const float4*>(p);
  v[0] = t.x; v[1] = t.y; v[2] = t.z; v[3] = t.w;
}
__device__ __forceinline__ void ldg(double (&v)[4], const double* p) {
  const double2 a = reinterpret_cast<const double2*>(p)[0], b = reinterpret_cast<const double2*>(p)[1];
  v[0] = a.x; v[1] = a.y; v[2] = b.x; v[3] = b.y;
}
__device__ __forceinline__ void stg(float* p, const float (&v)[4]) {
  *reinterpret_cast<float4*>(p) = make_float4(v[0], v[1], v[2], v[3]);
}
__device__ __forceinline__ void stg(double* p, const double (&v)[4]) {
  reinterpret_cast<double2*>(p)[0] = make_double2(v[0], v[1]);
  reinterpret_cast<double2*>(p)[1] = make_double2(v[2], v[3]);
}
}  // namespace xfp

// xfp_layout.cu -- line-compacted storage layout for one material grid.
//
// Unknown rows are xFluid's: fluid cells and solid cells with a fluid
// neighbour (variational_pressuresolver.cpp:245-321: only fluid cells assemble,
// and each solid neighbour of a fluid cell receives a row).  Every (j,k) x-line
// stores its active span, rounded out to whole groups of XFP_ALIGN cells that
// are aligned to the wavefront (see xfp_common.cuh).
#include <algorithm>
#include <climits>

#include "xfp_common.cuh"
#include "xfp_kernels.h"

namespace xfp {

__device__ __forceinline__ bool is_unknown(const uint8_t* mat, int ni, int nj, int nk, int i, int j,
                                           int k) {
  const size_t nn = (size_t)ni * nj;
  const size_t c = (size_t)k * nn + (size_t)j * ni + i;
  const uint8_t m = mat[c];
  if (m == MAT_FLUID) return true;
  if (m != MAT_SOLID) return false;
  if (i > 0 && mat[c - 1] == MAT_FLUID) return true;
  if (i + 1 < ni && mat[c + 1] == MAT_FLUID) return true;
  if (j > 0 && mat[c - ni] == MAT_FLUID) return true;
  if (j + 1 < nj && mat[c + ni] == MAT_FLUID) return true;
  if (k > 0 && mat[c - nn] == MAT_FLUID) return true;
  if (k + 1 < nk && mat[c + nn] == MAT_FLUID) return true;
  return false;
}

// The layout kernels take up to LAYOUT_SCENES grids a launch, blockIdx.y being the
// grid: a batch of 12 took 60 launches of 2 to 6 us for its line and block tables, and
// 36 for its group tables.
struct LayoutSet {
  LayoutScene s[LAYOUT_SCENES];
};

// One warp per x-line: span of unknowns and their count.
__global__ void line_span_kernel(const __grid_constant__ LayoutSet set) {
  const LayoutScene& G = set.s[blockIdx.y];
  const uint8_t* __restrict__ mat = G.mat;
  const int ni = G.ni, nj = G.nj, nk = G.nk;
  Line* __restrict__ lines = G.lines;
  const int lane = threadIdx.x & 31;
  const long long line = (long long)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  if (line >= (long long)nj * nk) return;
  const int j = (int)(line % nj), k = (int)(line / nj);
  int lo = INT_MAX, hi = -1, cnt = 0;
  for (int i = lane; i < ni; i += 32) {
    if (is_unknown(mat, ni, nj, nk, i, j, k)) {
      lo = min(lo, i);
      hi = max(hi, i);
      ++cnt;
    }
  }
  lo = __reduce_min_sync(XFP_FULL, lo);
  hi = __reduce_max_sync(XFP_FULL, hi);
  cnt = __reduce_add_sync(XFP_FULL, cnt);
  if (lane == 0) {
    Line L = {0, 0, 0, 0};
    if (cnt > 0) {
      // first stored cell S <= lo with S + j + k = 0 (mod XFP_ALIGN): cell i
      // then sits at an address = i + j + k (mod XFP_ALIGN); S may be < 0
      L.lo = lo - ((lo + j + k) & (XFP_ALIGN - 1));
      L.len = ((hi + 1 - L.lo) + XFP_ALIGN - 1) & ~(XFP_ALIGN - 1);
      L.nrows = cnt;
    }
    lines[line] = L;
  }
}

// Inclusive scan of one value per thread over a block of 1024 threads.
__device__ __forceinline__ long long scan1024(long long v, long long* sh) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const long long t = __shfl_up_sync(XFP_FULL, v, o);
    if (lane >= o) v += t;
  }
  if (lane == 31) sh[w] = v;
  __syncthreads();
  if (w == 0) {
    long long t = sh[lane];
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const long long u = __shfl_up_sync(XFP_FULL, t, o);
      if (lane >= o) t += u;
    }
    sh[lane] = t;
  }
  __syncthreads();
  const long long r = v + (w > 0 ? sh[w - 1] : 0);
  __syncthreads();
  return r;
}

// Offsets of the lines (exclusive scan of their lengths) and the totals, in two
// launches of at most LINE_CHUNKS CTAs with a chunk of lines each: every chunk's
// sums, then the scan, each CTA adding up the chunks before its own.  (One CTA
// alone took 65 us for the 16,384 lines of 128^3 and 155 us at 256^3; now 8 us.)
__device__ __forceinline__ long long line_chunk(long long nlines) {
  return max(1024LL, (nlines + LINE_CHUNKS - 1) / LINE_CHUNKS);
}
__global__ void __launch_bounds__(1024) line_sum_kernel(const __grid_constant__ LayoutSet set) {
  __shared__ long long sh[32];
  const LayoutScene& G = set.s[blockIdx.y];
  const Line* __restrict__ lines = G.lines;
  long long* __restrict__ sums = G.sums;
  const long long nlines = (long long)G.nj * G.nk, chunk = line_chunk(nlines);
  const long long a = blockIdx.x * chunk, b = min(a + chunk, nlines);
  if (a >= nlines) return;
  long long v[3] = {0, 0, 0};   // cells, rows, active lines
  for (long long l = a + threadIdx.x; l < b; l += 1024) {
    const Line L = lines[l];
    v[0] += L.len;
    v[1] += L.nrows;
    v[2] += L.len > 0;
  }
#pragma unroll
  for (int n = 0; n < 3; ++n) {
    const long long t = scan1024(v[n], sh);
    if (threadIdx.x == 1023) sums[n * LINE_CHUNKS + blockIdx.x] = t;
  }
}
__global__ void __launch_bounds__(1024) line_scan_kernel(const __grid_constant__ LayoutSet set) {
  __shared__ long long sh[32];
  __shared__ long long s_tot;
  const LayoutScene& G = set.s[blockIdx.y];
  Line* __restrict__ lines = G.lines;
  const long long* __restrict__ sums = G.sums;
  long long* __restrict__ counters = G.counters;
  const long long nlines = (long long)G.nj * G.nk, chunk = line_chunk(nlines);
  const unsigned chunks = (unsigned)((nlines + chunk - 1) / chunk);
  const long long a = blockIdx.x * chunk, b = min(a + chunk, nlines);
  if (a >= nlines) return;
  auto total = [&](int n, unsigned first) {   // of the first chunks (at most 1024)
    const long long t = scan1024(threadIdx.x < first ? sums[n * LINE_CHUNKS + threadIdx.x] : 0, sh);
    if (threadIdx.x == 1023) s_tot = t;
    __syncthreads();
    const long long r = s_tot;
    __syncthreads();
    return r;
  };
  long long carry = total(0, blockIdx.x);
  for (long long base = a; base < b; base += 1024) {
    const long long l = base + threadIdx.x;
    const long long v = l < b ? lines[l].len : 0;
    const long long inc = scan1024(v, sh);
    if (l < b) lines[l].off = (int)(carry + inc - v);
    if (threadIdx.x == 1023) s_tot = inc;
    __syncthreads();
    carry += s_tot;
    __syncthreads();
  }
  if (blockIdx.x + 1 != chunks) return;
  const long long rows = total(1, chunks), act = total(2, chunks);
  if (threadIdx.x == 0) {
    counters[0] = carry;
    counters[1] = rows;
    counters[2] = act;
  }
}

// Sweep-layout blocks: one warp per block of 8 x 8 lines finds the span of
// wavefront groups its cells cover (goff is scanned afterwards).
__global__ void blk_span_kernel(const __grid_constant__ LayoutSet set) {
  const LayoutScene& G = set.s[blockIdx.y];
  const Line* __restrict__ lines = G.lines;
  WBlk* __restrict__ blks = G.blks;
  const int nj = G.nj, nk = G.nk, NJB = (nj + 7) / 8;
  const long long nblk = (long long)NJB * ((nk + 7) / 8);
  const int lane = threadIdx.x & 31;
  const long long b = (long long)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  if (b >= nblk) return;
  const int jb = (int)(b % NJB), kb = (int)(b / NJB);
  int lo = INT_MAX, hi = INT_MIN;
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    const int j = jb * 8 + (lane & 7), k = kb * 8 + (lane >> 3) * 2 + h;
    if (j < nj && k < nk) {
      const Line L = lines[(size_t)k * nj + j];
      if (L.len > 0) {
        lo = min(lo, L.lo + j + k);
        hi = max(hi, L.lo + L.len - 1 + j + k);
      }
    }
  }
  lo = __reduce_min_sync(XFP_FULL, lo);
  hi = __reduce_max_sync(XFP_FULL, hi);
  if (lane == 0) {
    WBlk w = {0, 0, 0, 0};
    if (lo != INT_MAX) {
      w.g0 = lo >> 2;   // lo may be negative (group padding): arithmetic shift
      w.ng = (hi >> 2) - (lo >> 2) + 1;
    }
    blks[b] = w;
  }
}

// Block offsets (scan in block order) and the active tiles in topological
// order of the lower sweep: (J+K) ascending, then J.  One CTA per grid.
__global__ void __launch_bounds__(1024) blk_scan_kernel(const __grid_constant__ LayoutSet set) {
  __shared__ long long sh[32];
  __shared__ long long s_tot;
  const LayoutScene& G = set.s[blockIdx.y];
  WBlk* __restrict__ blks = G.blks;
  int2* __restrict__ tiles = G.tiles;
  long long* __restrict__ counters = G.counters;
  const int NJB = (G.nj + 7) / 8, NKB = (G.nk + 7) / 8;
  const int NJT = (NJB + WAVE_TJ - 1) / WAVE_TJ, NKT = (NKB + WAVE_TK - 1) / WAVE_TK;
  const long long nblk = (long long)NJB * NKB, ntile = (long long)NJT * NKT;
  long long carry = 0;
  for (long long base = 0; base < nblk; base += 1024) {
    const long long b = base + threadIdx.x;
    const long long v = b < nblk ? blks[b].ng : 0;
    const long long inc = scan1024(v, sh);
    if (b < nblk) blks[b].goff = (int)(carry + inc - v);
    if (threadIdx.x == 1023) s_tot = inc;
    __syncthreads();
    carry += s_tot;
    __syncthreads();
  }
  if (threadIdx.x == 0) counters[4] = carry;
  // tiles before diagonal d of an NJT x NKT grid
  auto before = [&](long long d) -> long long {
    const long long m = min(NJT, NKT), M = max(NJT, NKT);
    if (d <= m) return d * (d + 1) / 2;
    if (d <= M) return m * (m + 1) / 2 + (d - m) * m;
    const long long left = m + M - 1 - d;   // diagonals from d on
    return ntile - left * (left + 1) / 2;
  };
  carry = 0;
  for (long long base = 0; base < ntile; base += 1024) {
    const long long q = base + threadIdx.x;
    int2 t = make_int2(0, 0);
    long long act = 0;
    if (q < ntile) {
      long long lo = 0, hi = (long long)NJT + NKT - 2;   // the diagonal holding the q-th tile
      while (lo < hi) {
        const long long mid = (lo + hi + 1) >> 1;
        if (before(mid) <= q) lo = mid; else hi = mid - 1;
      }
      const int J = (int)(max(0LL, lo - (NKT - 1)) + (q - before(lo)));
      t = make_int2(J, (int)lo - J);
      for (int a = 0; a < WAVE_TJ * WAVE_TK; ++a) {
        const int jb = t.x * WAVE_TJ + a % WAVE_TJ, kb = t.y * WAVE_TK + a / WAVE_TJ;
        if (jb < NJB && kb < NKB && blks[(long long)kb * NJB + jb].ng > 0) act = 1;
      }
    }
    const long long inc = scan1024(act, sh);
    if (act) tiles[carry + inc - 1] = t;
    if (threadIdx.x == 1023) s_tot = inc;
    __syncthreads();
    carry += s_tot;
    __syncthreads();
  }
  if (threadIdx.x == 0) counters[3] = carry;
}

// For the aligned 4-cell group of cell c, at c / 4 (cells counted over all grids;
// lines start at multiples of 4 and hold multiples of 4 cells): where its y and z
// neighbours are, and the sweep element of its first cell (its four cells are four
// consecutive elements).
struct TableSet {
  TableScene s[LAYOUT_SCENES];
};
__global__ void group_tables_kernel(const __grid_constant__ TableSet set, GroupNb* __restrict__ group_nb,
                                    int* __restrict__ gperm) {
  const TableScene& G = set.s[blockIdx.y];
  const Line* __restrict__ lines = G.lines;
  const int nj = G.nj, nk = G.nk;
  const int lane = threadIdx.x & 31;
  const long long nlines = (long long)nj * nk;
  for (long long line = (long long)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); line < nlines;
       line += (long long)gridDim.x * (blockDim.x >> 5)) {
    const Line L = lines[line];
    if (L.len == 0) continue;
    const int j = (int)(line % nj), k = (int)(line / nj);
    const Line Z = {0, 0, 0, 0};
    const Line N[4] = {j > 0 ? lines[line - 1] : Z, j + 1 < nj ? lines[line + 1] : Z, k > 0 ? lines[line - nj] : Z,
                       k + 1 < nk ? lines[line + nj] : Z};
    const WBlk b = G.blks[(size_t)(k >> 3) * ((nj + 7) / 8) + (j >> 3)];
    for (int q = lane; q < (L.len >> 2); q += 32) {
      const size_t at = ((size_t)(G.base + L.off) >> 2) + q;
      unsigned nb[4];
#pragma unroll
      for (int n = 0; n < 4; ++n) {
        // the neighbour of the group's first cell; the quad after the one that
        // holds it, and whether the line stores either
        const int r = L.lo + 4 * q - N[n].lo;
        const int quad = (r >> 2) + 1;
        nb[n] = ((unsigned)(((G.base + N[n].off) >> 2) + quad) << 2) |
                ((unsigned)(r & ~3) < (unsigned)N[n].len ? 1u : 0u) | ((unsigned)(4 * quad) < (unsigned)N[n].len ? 2u : 0u);
      }
      const int t = L.lo + 4 * q + j + k;
      group_nb[at] = {nb[0], nb[1], nb[2], nb[3]};
      gperm[at] = (int)((G.group_base + b.goff + (t >> 2) - b.g0) * 256 + wave_line_slot(j, k));
    }
  }
}
// Adds every grid's base to the offsets of its lines.
__global__ void offset_lines_kernel(const __grid_constant__ TableSet set) {
  const TableScene& G = set.s[blockIdx.y];
  const long long nlines = (long long)G.nj * G.nk;
  for (long long q = (long long)blockIdx.x * blockDim.x + threadIdx.x; q < nlines; q += (long long)gridDim.x * blockDim.x)
    G.lines[q].off += (int)G.base;
}

cudaError_t layout_build(const LayoutScene* scenes, int n, cudaStream_t st) {
  for (int first = 0; first < n; first += LAYOUT_SCENES) {
    LayoutSet set = {};
    const unsigned m = (unsigned)std::min(LAYOUT_SCENES, n - first);
    long long nlines = 0, nblk = 0, chunks = 0;
    for (unsigned q = 0; q < m; ++q) {
      const LayoutScene& G = set.s[q] = scenes[first + q];
      const long long l = (long long)G.nj * G.nk, chunk = std::max<long long>(1024, (l + LINE_CHUNKS - 1) / LINE_CHUNKS);
      nlines = std::max(nlines, l);
      chunks = std::max(chunks, (l + chunk - 1) / chunk);
      nblk = std::max(nblk, (long long)((G.nj + 7) / 8) * ((G.nk + 7) / 8));
    }
    const int wpb = 8;
    g_kernel_launches += 5;
    line_span_kernel<<<dim3((unsigned)((nlines + wpb - 1) / wpb), m), wpb * 32, 0, st>>>(set);
    line_sum_kernel<<<dim3((unsigned)chunks, m), 1024, 0, st>>>(set);
    line_scan_kernel<<<dim3((unsigned)chunks, m), 1024, 0, st>>>(set);
    blk_span_kernel<<<dim3((unsigned)((nblk + wpb - 1) / wpb), m), wpb * 32, 0, st>>>(set);
    blk_scan_kernel<<<dim3(1, m), 1024, 0, st>>>(set);
    const cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
  }
  return cudaSuccess;
}

cudaError_t layout_tables(const TableScene* scenes, int n, GroupNb* group_nb, int* gperm, cudaStream_t st) {
  for (int first = 0; first < n; first += LAYOUT_SCENES) {
    TableSet set = {};
    const unsigned m = (unsigned)std::min(LAYOUT_SCENES, n - first);
    long long nlines = 0;
    bool offset = false;
    for (unsigned q = 0; q < m; ++q) {
      set.s[q] = scenes[first + q];
      nlines = std::max(nlines, (long long)set.s[q].nj * set.s[q].nk);
      offset |= set.s[q].base != 0;
    }
    ++g_kernel_launches;
    group_tables_kernel<<<dim3((unsigned)std::min<long long>((nlines + 7) / 8, 65535LL * 8), m), 256, 0, st>>>(
        set, group_nb, gperm);
    if (offset) {
      ++g_kernel_launches;
      offset_lines_kernel<<<dim3((unsigned)std::min<long long>((nlines + 255) / 256, 148LL * 8), m), 256, 0, st>>>(set);
    }
    const cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
  }
  return cudaSuccess;
}

}  // namespace xfp

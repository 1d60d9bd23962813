// xfp_steps.cu -- the simulator steps either side of the projection, on the
// device: the constant body force before it and the velocity extrapolation
// after it (xFluid/xFluid/FluidSimulator.cpp).
//
//   apply_forces  FluidSimulator::_applyForces              :429-499
//   extrapolate   FluidSimulator::_expolateVelocity(layers) :511-650
//
// The extrapolation is a breadth-first walk over the face grid of each axis,
// layer by layer.  A face of layer L takes the average of its neighbours of
// layer L-1, in the reference's neighbour order (+i,-i,+j,-j,+k,-k,
// xfluidutil.cpp:33-41), and the unmarked neighbours of layer L become layer
// L+1.  No face reads a value written in its own layer and a face's layer does
// not depend on the order a layer is visited in, so each layer is one
// data-parallel pass and the FP64 result is bit-identical to the sequential
// reference.
#include <algorithm>

#include "xfp_common.cuh"
#include "xfp_kernels.h"

namespace xfp {
namespace {

__device__ __forceinline__ bool fluid_at(const uint8_t* __restrict__ mat, int ni, int nj, int nk, int i, int j, int k) {
  return i >= 0 && j >= 0 && k >= 0 && i < ni && j < nj && k < nk &&
         mat[(size_t)k * ni * nj + (size_t)j * ni + i] == MAT_FLUID;
}

// a face of `axis` at (i,j,k) lies between cells (i,j,k) and (i,j,k) - e_axis
__device__ __forceinline__ bool borders_fluid(const uint8_t* __restrict__ mat, int ni, int nj, int nk, int axis, int i,
                                              int j, int k) {
  return fluid_at(mat, ni, nj, nk, i, j, k) ||
         fluid_at(mat, ni, nj, nk, i - (axis == 0), j - (axis == 1), k - (axis == 2));
}

template <typename FT>
__global__ void forces_kernel(const uint8_t* __restrict__ mat, int ni, int nj, int nk, int axis, FT* __restrict__ f,
                              FT dv) {
  const int si = ni + (axis == 0), sj = nj + (axis == 1), sk = nk + (axis == 2);
  const size_t n = (size_t)si * sj * sk;
  for (size_t idx = (size_t)blockIdx.x * blockDim.x + threadIdx.x; idx < n; idx += (size_t)gridDim.x * blockDim.x) {
    const int i = (int)(idx % si), j = (int)((idx / si) % sj), k = (int)(idx / ((size_t)si * sj));
    if (borders_fluid(mat, ni, nj, nk, axis, i, j, k)) f[idx] = add_rn(f[idx], dv);
  }
}

// The layers are sets of bits, 32 faces of a row along x to a word; all three
// axes use the row layout of the (ni+1) x (nj+1) x (nk+1) corner grid.
struct LayerBits {
  unsigned WX, J, K;   // words of a row, rows along j and k
  unsigned *seen, *front[2];   // per axis `stride` words: the layers so far; the last layer and the one before
  unsigned stride;   // (a grid has fewer than 2^31 cells, so words fit 32 bits)
};

// The fluid cells as bits (in front[1], read by layer0_kernel), WORDS words a warp:
// a byte per cell is all that is read of the material.
constexpr int WORDS = 8;
__global__ void fluid_bits_kernel(const uint8_t* __restrict__ mat, int ni, int nj, int nk, LayerBits B) {
  const int lane = threadIdx.x & 31;
  const unsigned w0 = (blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5)) * WORDS;
  bool c[WORDS];
#pragma unroll
  for (int n = 0; n < WORDS; ++n) {
    const unsigned w = w0 + n, r = w / B.WX, k = r / B.J;
    c[n] = w < B.stride && fluid_at(mat, ni, nj, nk, (int)(w - r * B.WX) * 32 + lane, (int)(r - k * B.J), (int)k);
  }
  unsigned mine = 0;
#pragma unroll
  for (int n = 0; n < WORDS; ++n) {
    const unsigned b = __ballot_sync(0xffffffffu, c[n]);
    if (lane == n) mine = b;
  }
  if (lane < WORDS && w0 + lane < B.stride) B.front[1][w0 + lane] = mine;
}

// layer 0: the faces of fluid cells (:547-560), a thread per word for the three axes
__global__ void layer0_kernel(LayerBits B) {
  const unsigned* __restrict__ cells = B.front[1];
  for (unsigned w = blockIdx.x * blockDim.x + threadIdx.x; w < B.stride; w += gridDim.x * blockDim.x) {
    const unsigned r = w / B.WX, k = r / B.J, c = cells[w];
    const unsigned low[3] = {c << 1 | (w != r * B.WX ? cells[w - 1] >> 31 : 0u), r != k * B.J ? cells[w - B.WX] : 0u,
                             k > 0 ? cells[w - B.WX * B.J] : 0u};
#pragma unroll
    for (int axis = 0; axis < 3; ++axis) {
      const size_t at = (size_t)axis * B.stride + w;
      B.seen[at] = B.front[0][at] = c | low[axis];
    }
  }
}

// Layer L (1, 2, ...): the unmarked faces next to layer L-1 (:565-590, :628-637)
// take the average of their neighbours there (:599-625).  A thread finds the new
// bits of a word, then its warp takes the words that have any, a lane per face.
//
// What bounds it is the instructions for the words that hold new faces (a division
// and up to six loads a face); finding them takes seven 4-byte loads from L2 for 32
// faces.  A pass over 16-bit markers per layer and axis took 87 us at 192^3 (blobs,
// FP32), three of them a layer; the three axes' layer now takes 30 us, and layer 0
// 24 us (71 with a byte load per axis and cell).  Four words at a time, for more
// loads under way, took 48 us.
template <typename FT>
__global__ void layer_kernel(FT* __restrict__ u, FT* __restrict__ v, FT* __restrict__ w_, int ni, int nj, int nk,
                             LayerBits B, int L) {
  const int lane = threadIdx.x & 31, axis = blockIdx.y;
  const int si = ni + (axis == 0), sj = nj + (axis == 1), sk = nk + (axis == 2);
  FT* __restrict__ f = axis == 0 ? u : axis == 1 ? v : w_;
  unsigned* __restrict__ seen = B.seen + (size_t)axis * B.stride;
  const unsigned* __restrict__ last = B.front[(L - 1) & 1] + (size_t)axis * B.stride;
  unsigned* __restrict__ next = B.front[L & 1] + (size_t)axis * B.stride;
  const unsigned row = B.WX, plane = row * B.J;
  for (unsigned w0 = (blockIdx.x * blockDim.x + threadIdx.x) & ~31u; w0 < B.stride; w0 += gridDim.x * blockDim.x) {
    const unsigned w = w0 + lane;
    unsigned x = 0, line = 0;   // first face / 32, k * sj + j
    unsigned own = 0, xm = 0, xp = 0, ym = 0, yp = 0, zm = 0, zp = 0, add = 0;
    if (w < B.stride) {
      const unsigned r = w / row, k = r / B.J, j = r - k * B.J;
      x = w - r * row;
      line = k * sj + j;
      const unsigned s = seen[w];
      own = last[w];
      if (x > 0) xm = last[w - 1];
      if (x + 1 < B.WX) xp = last[w + 1];
      if (j > 0) ym = last[w - row];
      if (j + 1 < B.J) yp = last[w + row];
      if (k > 0) zm = last[w - plane];
      if (k + 1 < B.K) zp = last[w + plane];
      xm = own << 1 | xm >> 31;   // from here on: by the bit of the face they are a neighbour of
      xp = own >> 1 | xp << 31;
      const int n = si - (int)x * 32;
      const unsigned face = (int)j < sj && (int)k < sk && n > 0 ? (n >= 32 ? 0xffffffffu : (1u << n) - 1u) : 0u;
      add = (xm | xp | ym | yp | zm | zp) & ~s & face;
      next[w] = add;
      if (add) seen[w] = s | add;
    }
    for (unsigned live = __ballot_sync(0xffffffffu, add != 0); live != 0; live &= live - 1) {
      const int src = __ffs(live) - 1;
      auto bit = [&](unsigned m) { return (__shfl_sync(0xffffffffu, m, src) >> lane) & 1u; };
      const unsigned me = bit(add), nb[6] = {bit(xp), bit(xm), bit(yp), bit(ym), bit(zp), bit(zm)};
      const unsigned r = __shfl_sync(0xffffffffu, line, src), c = __shfl_sync(0xffffffffu, x, src) * 32 + lane;
      if (!me) continue;
      const size_t q = (size_t)r * si + c;
      FT sum = FT(0);
      int count = 0;
#pragma unroll
      for (int n = 0; n < 6; ++n)
        if (nb[n]) {
          const size_t step = n < 2 ? (size_t)1 : n < 4 ? (size_t)si : (size_t)si * sj;
          sum = add_rn(sum, f[n & 1 ? q - step : q + step]);
          ++count;
        }
      f[q] = div_rn(sum, FT(count));
    }
  }
}

// VariationalPressureSolver::_calculate_divergience
// (variationalpressure/variational_pressuresolver.cpp:526-597): per fluid cell
// the sum of +u(low face) - u(high face) over the axes, a face counted only when
// the cell across it is not solid (outside the grid counts as solid); 0 for
// other cells.  Six additions from 0 in the reference's order.
template <typename FT>
__global__ void divergence_kernel(const uint8_t* __restrict__ mat, int ni, int nj, int nk, const FT* __restrict__ u,
                                  const FT* __restrict__ v, const FT* __restrict__ w, FT* __restrict__ div) {
  const size_t n = (size_t)ni * nj * nk;
  auto solid_at = [&](int i, int j, int k) {
    return !(i >= 0 && j >= 0 && k >= 0 && i < ni && j < nj && k < nk) ||
           mat[(size_t)k * ni * nj + (size_t)j * ni + i] == MAT_SOLID;
  };
  for (size_t c = (size_t)blockIdx.x * blockDim.x + threadIdx.x; c < n; c += (size_t)gridDim.x * blockDim.x) {
    const int i = (int)(c % ni), j = (int)((c / ni) % nj), k = (int)(c / ((size_t)ni * nj));
    FT d = FT(0);
    if (mat[c] == MAT_FLUID) {
      const size_t uu = (size_t)k * (ni + 1) * nj + (size_t)j * (ni + 1) + i;
      const size_t vv = (size_t)k * ni * (nj + 1) + (size_t)j * ni + i;
      const size_t ww = c;
      if (!solid_at(i - 1, j, k)) d = add_rn(d, u[uu]);
      if (!solid_at(i + 1, j, k)) d = sub_rn(d, u[uu + 1]);
      if (!solid_at(i, j - 1, k)) d = add_rn(d, v[vv]);
      if (!solid_at(i, j + 1, k)) d = sub_rn(d, v[vv + ni]);
      if (!solid_at(i, j, k - 1)) d = add_rn(d, w[ww]);
      if (!solid_at(i, j, k + 1)) d = sub_rn(d, w[ww + (size_t)ni * nj]);
    }
    div[c] = d;
  }
}

unsigned grid_for(size_t n) { return (unsigned)std::min<size_t>((n + 255) / 256, 148 * 32); }

}  // namespace

template <typename FT>
cudaError_t divergence(const uint8_t* mat, int ni, int nj, int nk, const FT* u, const FT* v, const FT* w, FT* div,
                       cudaStream_t st) {
  ++g_kernel_launches;
  divergence_kernel<FT><<<grid_for((size_t)ni * nj * nk), 256, 0, st>>>(mat, ni, nj, nk, u, v, w, div);
  return cudaGetLastError();
}
template cudaError_t divergence<double>(const uint8_t*, int, int, int, const double*, const double*, const double*,
                                        double*, cudaStream_t);
template cudaError_t divergence<float>(const uint8_t*, int, int, int, const float*, const float*, const float*, float*,
                                       cudaStream_t);

template <typename FT>
cudaError_t apply_forces(const uint8_t* mat, int ni, int nj, int nk, FT* u, FT* v, FT* w, Force3 frc,
                         cudaStream_t st) {
  FT* f[3] = {u, v, w};
  for (int axis = 0; axis < 3; ++axis) {
    if (!frc.axis_on(axis)) continue;
    const size_t n = (size_t)(ni + (axis == 0)) * (nj + (axis == 1)) * (nk + (axis == 2));
    ++g_kernel_launches;
    forces_kernel<FT><<<grid_for(n), 256, 0, st>>>(mat, ni, nj, nk, axis, f[axis], (FT)frc.d[axis]);
  }
  return cudaGetLastError();
}

size_t extrapolate_scratch(int ni, int nj, int nk) {
  return (size_t)((ni + 1 + 31) / 32) * (nj + 1) * (nk + 1) * 9 * sizeof(unsigned);
}

template <typename FT>
cudaError_t extrapolate(const uint8_t* mat, int ni, int nj, int nk, FT* u, FT* v, FT* w, int layers,
                        unsigned* scratch, cudaStream_t st) {
  if (layers <= 0) return cudaSuccess;
  LayerBits B;
  B.WX = (ni + 1 + 31) / 32;
  B.J = nj + 1;
  B.K = nk + 1;
  B.stride = B.WX * B.J * B.K;
  B.seen = scratch;
  B.front[0] = scratch + 3 * (size_t)B.stride;
  B.front[1] = scratch + 6 * (size_t)B.stride;
  ++g_kernel_launches;
  fluid_bits_kernel<<<(unsigned)((B.stride + 8 * WORDS - 1) / (8 * WORDS)), 256, 0, st>>>(mat, ni, nj, nk, B);
  ++g_kernel_launches;
  layer0_kernel<<<grid_for(B.stride), 256, 0, st>>>(B);
  const dim3 grid((unsigned)std::min<size_t>((B.stride + 127) / 128, 148 * 32), 3);
  for (int L = 1; L <= layers; ++L) {
    ++g_kernel_launches;
    layer_kernel<FT><<<grid, 128, 0, st>>>(u, v, w, ni, nj, nk, B, L);
  }
  return cudaGetLastError();
}

template cudaError_t apply_forces<double>(const uint8_t*, int, int, int, double*, double*, double*, Force3,
                                          cudaStream_t);
template cudaError_t apply_forces<float>(const uint8_t*, int, int, int, float*, float*, float*, Force3, cudaStream_t);
template cudaError_t extrapolate<double>(const uint8_t*, int, int, int, double*, double*, double*, int, unsigned*,
                                         cudaStream_t);
template cudaError_t extrapolate<float>(const uint8_t*, int, int, int, float*, float*, float*, int, unsigned*,
                                        cudaStream_t);

}  // namespace xfp

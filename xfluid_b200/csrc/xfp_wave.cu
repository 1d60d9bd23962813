// xfp_wave.cu -- the MIC(0) factorisation and both triangular solves in
// xFluid's natural (lexicographic) order, as one dataflow wavefront kernel.
//
// Reference semantics (xFluid/xFluid/variationalpressure/pcg_solver.h):
//   factor   factor_modified_incomplete_cholesky0         :85-186
//   forward  solve_lower (column-scatter L y = r)          :192-204
//   backward solve_lower_transpose_in_place                :207-220
// Every update is applied in the reference's column order with separately
// rounded multiplies and subtractions, so the FP64 path is bit-identical to
// the reference.
//
// What bounds it: the dependency chain.  Cell (i,j,k) is processed at step
// t = i+j+k and needs its three lower neighbours of step t-1, so a sweep is as
// long as its hyperplanes, and each holds a few thousand cells; the data (20 to
// 28 bytes a cell in FP32) would stream in a tenth of the time.  So a step has
// to be short, a hand-off between warps has to cost little more than a step,
// and the work has to be spread thinly over the SMs: 128 lines moving at 60
// cycles a step already ask 45 of the 64 bytes a cycle an SM gets from L2.
//
// Work decomposition.  A compute warp owns a block of 8 x 8 x-lines (j, k): lane
// (kl, jl) holds the lines k = 2*kl and 2*kl + 1 of column jl.  At each step a
// lane advances both its lines by one cell (two independent chains):
//   x-neighbour  the line's own previous step                 (register)
//   y-neighbour  lane -1's previous step                      (shuffle)
//   z-neighbour  the lane's other line, or lane -8's          (register / shuffle)
// so inside a block a step costs one shuffle and the row's arithmetic.  (The
// factorisation, whose step is a division and a square root, gives every line
// a lane of its own: half a block a warp.)
// A cluster of 8 CTAs with two blocks each covers 32 x 32 lines.  A block hands
// its edge values on by groups of 4 steps, to a block of its cluster straight
// into that block's ring of group slots in distributed shared memory (st.async),
// to a block of another cluster through global memory, as 64-bit words of 32
// bits payload and the launch generation (single-copy atomic, so no fence or
// flag is needed: the reader polls the words themselves).
// A slot of the ring holds all that a block needs for one group -- its own
// operands and its lower neighbours' edge values -- and one mbarrier counts
// their bytes, so a compute warp waits once per group and then runs four steps
// on registers and shuffles.  Three more warps keep the rest off its chain: a
// sender takes the results from the slot to global memory and hands on the edges,
// a helper refills the slots (bulk copies, S groups ahead) and reports the free
// ones, without which no one writes to them, and a courier fetches the edge values
// that come through global memory.  (The factorisation's step is long enough for
// its compute warp to hand on its results itself.)
//
// Data.  Every block's cells lie in its own stream of groups of 4 steps (WBlk,
// wave_line_slot, wave_cell_slot), a group's factor, r and y side by side, so
// that one bulk copy of a few KB fills a slot (issuing two or three took the
// helper warp longer than the steps take).  Cells that are absent hold zero in every
// array, which makes their results zero without masks.
//
// Tiles are taken in topological order (J+K ascending): the first ones by
// cluster index (a cooperative launch, so all clusters are resident), the
// others from a ticket counter, so a tile only ever waits on tiles that
// resident clusters hold.
//
// Waits are bounded.  The one wait that depends on other clusters, a courier's for
// edge words, runs out after spin_limit polls, or once another has: it records
// SweepCtl::err and from there on hands over whatever the words hold.  The results
// are void, but every group is still sent, waited for and freed, so that the tile
// runs to its end as it always does, no copy is left under way, and the host reports
// XFP_ERR_TIMEOUT.  The waits inside a cluster depend on nothing but that; they
// outlast it eight times, and one that runs out all the same (give_up) ends the
// cluster after its tile, once the copies to its slots have landed.
//
// z.r is summed as the solves always did: every lane its lines in cell order,
// the lines in 256 chunks, a fixed tree; the last cluster's eight CTAs share the
// chunks (one CTA alone reads 65,536 partials at 256^3).
//
// Measured (device time of a launch, full box of 128^3 / 256^3 cells): a solve
// takes 64 / 171 us in FP32 and 94 / 301 us in FP64, the factorisation 0.24 / 0.67
// ms; a launch costs 12 (FP64 14) us to start and end, a group of four steps of a
// lone block 0.28 (0.41) us, of which the steps are 0.13 (0.2) and the rest is
// waiting for a slot, reading it and handing it on.  Before waits were votes and
// refills fenced: 62 / 159 and 90 / 285 us, 0.25 (0.36) us a group.  (The fence in the
// sender instead, or one for two or four groups: the same within 2 %; waits that one
// lane makes for its warp: 69 / 176 us.)
// With the compute warp sending its edges and storing its results, as the
// factorisation's does: 0.31 (0.39) us a group, 74 / 190 and 102 / 330 us.  With an
// mbarrier each for operands and edge values, acknowledgements by the compute warp
// and two or three copies a group: 0.43 (0.50) us, 83 / 214 and 114 / 365 us.
// Before (one CTA per 32 x 15 lines, a CTA-wide barrier per step, tiles through
// global memory): 263 us for the FP64 128^3 solve, 180 us for a half-full FP32
// 256^3 one (now 65), 0.65 to 1.0 ms for the factorisation.  Tried on the way:
// lockstep CTAs of 2 x 2 blocks (143 us where the first form took 81), blocks that
// hand over through L2 words only (117 to 134), per-step instead of per-group
// hand-over in the cluster (367 cycles a step), one warp as helper and courier with
// 4 slots a block (207).
#include <algorithm>
#include <atomic>
#include <climits>

#include "xfp_edges.h"
#include "xfp_sweep_util.cuh"
#include "xfp_warp_wait.h"

namespace xfp {
namespace {

constexpr int GE = 256;   // cells of one block's group: 64 lines x 4 steps
// Groups of edge words a courier has under way per far edge.  Two cover a load's
// way to L2 and back at a group's pace; every further one only lengthens a poll
// and the queue of all couriers' polls.  Whole projections in ms with 1 / 2 / 3 / 4 /
// 6: 128^3 FP64 8.60 8.51 8.63 8.72 9.11, 256^3 mixed 11.1 9.98 9.94 10.1 10.3,
// 150 x 97 x 131 mixed 9.64 8.82 8.84 8.90 9.01.
constexpr int FB = 2;

// What a block hands to a neighbour per line and step (X): the factorisation
// sends L(m,c) and the sum of the column's other two entries (the dropped
// fill), the forward solve the product L(m,c) y[c], the backward solve z[c].
// HL: lines per lane; IN: operands per group; S: slots of the rings (a power of two).
template <int OP, typename VT, typename CT>
struct WaveOp {
  using X = VT;
  using ST = VT;
  static constexpr int HL = 2, IN = (OP == SWEEP_BWD ? 6 : 5) * GE, S = 8;
};
template <typename VT, typename CT>
struct WaveOp<SWEEP_FACTOR, VT, CT> {
  using X = Pair<CT>;
  using ST = CT;
  static constexpr int HL = 1, IN = 2 * GE, S = 4;
};
// Warps for a unit: compute, helper, courier and, for the solves, sender.
template <int OP>
constexpr int roles_of() { return OP == SWEEP_FACTOR ? 3 : 4; }
template <int OP>
constexpr int warps_of() { return OP == SWEEP_FACTOR ? 4 : 2; }   // compute warps per CTA (two blocks)

// One group of a block: its operands, and the edge values of its j and k
// producers' same group, [line][step in sweep order].
template <int OP, typename VT, typename CT>
struct __align__(128) Slot {
  using W = WaveOp<OP, VT, CT>;
  typename W::ST ops[W::IN];
  typename W::X ej[4 * W::HL][4], ek[8][4];
};
// Shared memory of one compute warp, its helper and its courier.
template <int OP, typename VT, typename CT>
struct __align__(128) UnitShared {
  static constexpr int S = WaveOp<OP, VT, CT>::S;
  Slot<OP, VT, CT> slot[S];
  unsigned long long full[S];    // mbarriers: a slot's operands and edge values have landed
  unsigned long long ready[S];   // mbarriers: a slot holds the group's results (solves)
  unsigned long long empty[S];   // mbarriers: a slot can be filled again
  int limit[2];                  // the j / k consumer has room for this block's groups below
  int freed;                     // slots given back (kept for a courier at work)
};

// One value as stamped words.
template <typename X>
struct EdgeWords {
  static constexpr int P = Words<X>::P;
  unsigned long long w[P];
  __device__ __forceinline__ bool ready(unsigned stamp) const {
    bool ok = true;
#pragma unroll
    for (int p = 0; p < P; ++p) ok &= (unsigned)(w[p] >> 32) == stamp;
    return ok;
  }
  __device__ __forceinline__ X value() const {
    uint32_t v[P];
#pragma unroll
    for (int p = 0; p < P; ++p) v[p] = (uint32_t)w[p];
    return from_words<X>(v);
  }
  __device__ __forceinline__ void load(const unsigned long long* a) {
    if constexpr (P == 1) {
      w[0] = ld_gpu64(a);
    } else {
#pragma unroll
      for (int p = 0; p < P; p += 2)
        asm volatile("ld.relaxed.gpu.global.v2.u64 {%0, %1}, [%2];" : "=l"(w[p]), "=l"(w[p + 1]) : "l"(a + p));
    }
  }
};
// four steps' values of a line as stamped words (32-byte stores; every word counts by itself)
template <typename X>
__device__ __forceinline__ void publish(unsigned long long* a, unsigned stamp, const X (&v)[4]) {
  constexpr int N = 4 * Words<X>::P;
  uint32_t w[N];
#pragma unroll
  for (int s = 0; s < 4; ++s) to_words(v[s], w + s * Words<X>::P);
#pragma unroll
  for (int q = 0; q < N; q += 4)
    asm volatile("st.relaxed.gpu.global.v4.u64 [%0], {%1, %2, %3, %4};"
                 ::"l"(a + q), "l"(stamped(stamp, w[q])), "l"(stamped(stamp, w[q + 1])),
                 "l"(stamped(stamp, w[q + 2])), "l"(stamped(stamp, w[q + 3])) : "memory");
}
// N 32-bit words to a slot in this cluster, counted by its mbarrier (both
// shared::cluster addresses, the slot's aligned to the store)
template <int N>
__device__ __forceinline__ void send(unsigned a, unsigned bar, const uint32_t (&w)[N]) {
  if constexpr (N == 1) {
    asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.b32 [%0], %1, [%2];"
                 ::"r"(a), "r"(w[0]), "r"(bar) : "memory");
  } else if constexpr (N == 2) {
    asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.v2.b32 [%0], {%1, %2}, [%3];"
                 ::"r"(a), "r"(w[0]), "r"(w[1]), "r"(bar) : "memory");
  } else {
#pragma unroll
    for (int q = 0; q < N; q += 4)
      asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.v4.b32 [%0], {%1, %2, %3, %4}, [%5];"
                   ::"r"(a + 4 * q), "r"(w[q]), "r"(w[q + 1]), "r"(w[q + 2]), "r"(w[q + 3]), "r"(bar) : "memory");
  }
}

__device__ __forceinline__ unsigned smem_u32(const void* p) { return (unsigned)__cvta_generic_to_shared(p); }
__device__ __forceinline__ unsigned cluster_addr(unsigned a, int rank) {
  unsigned r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(rank));
  return r;
}
__device__ __forceinline__ void st_cluster_u32(unsigned a, unsigned v) {
  asm volatile("st.relaxed.cluster.shared::cluster.u32 [%0], %1;" ::"r"(a), "r"(v) : "memory");
}
// A count of free slots, for another warp of the cluster (shared::cluster address), and
// that warp's look: what was read from a slot before it was given back comes before
// what is sent to it after.  The release is this CTA's: shared memory has one copy, so
// its accesses are over for the cluster once they are for the CTA.  (One of the
// cluster's scope holds the helper up for 0.2 us a group: 128^3 99 us against 64 in
// FP32, 131 against 97 in FP64; the acquire and this release cost nothing measurable.)
__device__ __forceinline__ void st_release_s32(unsigned a, int v) {
  asm volatile("st.release.cta.shared::cluster.s32 [%0], %1;" ::"r"(a), "r"(v) : "memory");
}
__device__ __forceinline__ int ld_acquire_s32(const int* p) {
  int v;
  asm volatile("ld.acquire.cluster.shared.s32 %0, [%1];" : "=r"(v) : "r"(smem_u32(p)) : "memory");
  return v;
}
__device__ __forceinline__ void cluster_sync() {
  asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ void mbar_init(unsigned long long* b) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(b)) : "memory");
}
__device__ __forceinline__ void mbar_expect(unsigned long long* b, unsigned bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(b)), "r"(bytes) : "memory");
}
__device__ __forceinline__ bool mbar_try(unsigned b, unsigned parity) {
  unsigned ok;
  asm volatile(
      "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.b32 %0, 1, 0, p;\n}"
      : "=r"(ok) : "r"(b), "r"(parity) : "memory");
  return ok != 0;
}
// size and both addresses are multiples of 16 bytes (whole groups)
__device__ __forceinline__ void bulk_load(void* dst, const void* src, unsigned bytes, unsigned long long* b) {
  asm volatile("cp.async.bulk.shared::cta.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
               ::"r"(smem_u32(dst)), "l"(src), "r"(bytes), "r"(smem_u32(b)) : "memory");
}

__device__ __forceinline__ unsigned long long now_ns() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
  return t;
}
// orders what this thread knows of ordinary accesses to shared memory before its bulk copies
__device__ __forceinline__ void fence_bulk() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }

__device__ __forceinline__ void mbar_arrive(unsigned long long* b) {
  asm volatile("mbarrier.arrive.release.cta.shared::cta.b64 _, [%0];" ::"r"(smem_u32(b)) : "memory");
}

template <typename T>
__device__ __forceinline__ T shfl_up_any(const T& v, int d) {
  uint32_t w[sizeof(T) / 4];
  to_words(v, w);
#pragma unroll
  for (int p = 0; p < (int)(sizeof(T) / 4); ++p) w[p] = __shfl_up_sync(XFP_FULL, w[p], d);
  return from_words<T>(w);
}
template <typename T>
__device__ __forceinline__ T shfl_down_any(const T& v, int d) {
  uint32_t w[sizeof(T) / 4];
  to_words(v, w);
#pragma unroll
  for (int p = 0; p < (int)(sizeof(T) / 4); ++p) w[p] = __shfl_down_sync(XFP_FULL, w[p], d);
  return from_words<T>(w);
}
// the four values of one cell of a group in the ring (wave_cell_slot's order; c: the cell's slot for e = 0, a = 0)
__device__ __forceinline__ void cell_values(float (&v)[4], const float* ring, int c, int e) { ldg(v, ring + c + e * 128); }
__device__ __forceinline__ void cell_values(double (&v)[4], const double* ring, int c, int e) {
  const double2 a = *reinterpret_cast<const double2*>(ring + c + e * 128);
  const double2 b = *reinterpret_cast<const double2*>(ring + c + e * 128 + 64);
  v[0] = a.x; v[1] = a.y; v[2] = b.x; v[3] = b.y;
}
__device__ __forceinline__ void put_cell(float* p, int c, int e, const float (&v)[4]) { stg(p + c + e * 128, v); }
__device__ __forceinline__ void put_cell(double* p, int c, int e, const double (&v)[4]) {
  *reinterpret_cast<double2*>(p + c + e * 128) = make_double2(v[0], v[1]);
  *reinterpret_cast<double2*>(p + c + e * 128 + 64) = make_double2(v[2], v[3]);
}

// z.r of a line in cell order (a backward group is taken from its last cell on),
// in FP32 or in FP64
template <typename VT, bool F32>
struct LineDot {
  float f = 0.f;
  double d = 0.0;
  __device__ __forceinline__ void add(const VT (&z)[4], const VT (&r)[4]) {
#pragma unroll
    for (int s = 3; s >= 0; --s) {
      if (F32) f = __fadd_rn(f, __fmul_rn((float)z[s], (float)r[s]));
      else if (sizeof(VT) == 4) d = __fma_rn((double)z[s], (double)r[s], d);   // (the product is exact)
      else d = __dadd_rn(d, __dmul_rn((double)z[s], (double)r[s]));
    }
  }
  __device__ __forceinline__ double sum() const { return F32 ? (double)f : d; }
};

template <int OP, typename VT, typename CT>
__global__ void __launch_bounds__(roles_of<OP>() * 32 * warps_of<OP>(), OP != SWEEP_FACTOR && sizeof(VT) == 4 ? 2 : 1)
    wave_kernel(WaveArgs g) {
  using W = WaveOp<OP, VT, CT>;
  using X = typename W::X;
  using ST = typename W::ST;
  using U = UnitShared<OP, VT, CT>;
  using SL = Slot<OP, VT, CT>;
  constexpr bool REV = OP == SWEEP_BWD, FACTOR = OP == SWEEP_FACTOR;
  constexpr int P = Words<X>::P, HL = W::HL, S = W::S, LS = S == 8 ? 3 : 2;
  static_assert(S == 1 << LS, "slots are a power of two");
  constexpr bool DOT32 = std::is_same<CT, float>::value;   // plain FP32: a lane's z.r in FP32
  constexpr int DIR = REV ? -1 : 1;
  constexpr int OUT = REV ? WAVE_Y : WAVE_R;               // a slot's results
  constexpr int NW = warps_of<OP>(), PER = NW / 2;         // compute warps per CTA, per block
  extern __shared__ __align__(128) unsigned char wave_smem[];
  U* const units = reinterpret_cast<U*>(wave_smem);
  // the next tile, by tile parity: a CTA may still read one while the leader
  // already writes the other
  __shared__ int s_next[2];
  __shared__ int s_broken;   // a wait inside the cluster ran out

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int unit = warp % NW;
  const bool compute = warp < NW, helper = warp / NW == 1, courier = warp / NW == 2;
  U& sh = units[unit];
  const int jl = lane & 7, kl = lane >> 3;
  const int rank = blockIdx.x % WAVE_CLUSTER;
  const int cj = rank % WAVE_TJ, ck = rank / WAVE_TJ;
  const int kt = ck * NW + unit;           // unit along k in the tile
  const int nclusters = gridDim.x / WAVE_CLUSTER;
  // producers and consumers in this cluster (near) or in another (far)
  const bool near_pj = cj - DIR >= 0 && cj - DIR < WAVE_TJ, near_nj = cj + DIR >= 0 && cj + DIR < WAVE_TJ;
  const bool near_pk = kt - DIR >= 0 && kt - DIR < 2 * NW, near_nk = kt + DIR >= 0 && kt + DIR < 2 * NW;
  auto unit_at = [&](int kk) -> U* { return &units[kk % NW]; };
  auto rank_at = [&](int c, int kk) { return (kk / NW) * WAVE_TJ + c; };
  if (threadIdx.x == 0) s_broken = 0;
  if (helper && lane == 0) {
    for (int q = 0; q < S; ++q) {
      mbar_init(&sh.full[q]);
      mbar_init(&sh.ready[q]);
      mbar_init(&sh.empty[q]);
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  // per slot: the parity of its mbarriers' next phase at the start of a tile
  // (ready and empty: one per group q; full: one per u)
  unsigned phase_q = 0, phase_u = 0;
  unsigned gen = 0;
  bool first = true;

  for (int pos = blockIdx.x / WAVE_CLUSTER, turn = 0; pos < g.ntiles; turn ^= 1) {
    const int tpos = REV ? g.ntiles - 1 - pos : pos;
    if (helper && lane == 0) sh.freed = 0;
    int NJB = g.NJB, NKB = g.NKB, lj = g.nj, lk = g.nk;
    long long gbase = 0, bbase = 0, lbase = 0;
    int sid = -1;
    if (g.tile_scene != nullptr) {
      sid = g.tile_scene[tpos];
      const BatchSeg& B = g.segs[sid];
      lj = B.nj;
      lk = B.nk;
      lbase = B.line_base;
      NJB = (lj + 7) >> 3;
      NKB = (lk + 7) >> 3;
      gbase = B.group_base;
      bbase = B.blk_base;
    }
    const int2 tile = g.tiles[tpos];
    const int jb = tile.x * WAVE_TJ + cj, ku = tile.y * 2 * NW + kt;
    const int kb = ku / PER, half = ku % PER;
    auto block_at = [&](int j, int u) -> WBlk {
      WBlk b = {0, 0, 0, 0};
      const int k = u / PER;
      if (j >= 0 && u >= 0 && j < NJB && k < NKB) b = g.blks[bbase + (long long)k * NJB + j];
      return b;
    };
    const WBlk me = block_at(jb, ku);
    const WBlk pj = block_at(jb - DIR, ku), pk = block_at(jb, ku - DIR);
    const long long mybase = gbase + me.goff;
    auto shift = [&](const WBlk& p, const WBlk& c) { return edge_shift(REV, p.g0, p.ng, c.g0, c.ng); };
    const int aj = shift(pj, me), ak = shift(pk, me);   // producer's group at u: u + aj, u + ak
    // the consumers' u of this block's group q is q - uj, q - uk
    const WBlk nj = block_at(jb + DIR, ku), nk = block_at(jb, ku + DIR);
    const int uj = shift(me, nj), uk = shift(me, nk);
    // the tables are the layout's; from here on, what the kernel before this one wrote
    if (first) {
      wait_previous();
      if (g.scal != nullptr && *(volatile int*)&g.scal->done != 0) return;   // (changes between launches only)
      gen = ld_volatile_u32(&g.ctl->gen);
    }
    // a converged scene's tiles are skipped (its scalars only change between
    // launches, so every warp of this launch decides the same way)
    const bool skip = sid >= 0 && g.scal_batch != nullptr && *(volatile int*)&g.scal_batch[sid].done != 0;
    first = false;
    if (helper && lane == 0) {
      sh.limit[0] = near_nj && nj.ng > 0 ? S + uj : INT_MAX;
      sh.limit[1] = near_nk && nk.ng > 0 ? S + uk : INT_MAX;
    }
    __syncwarp();
    // every CTA of the cluster runs, and its slots are free (no other shared
    // memory is touched before this)
    cluster_sync();
    if (rank == 0 && threadIdx.x == 0) {
      int nx = nclusters + (int)atomicAdd(&g.ctl->ticket, 1u);
      if (ld_volatile_u32(&g.ctl->err)) nx = INT_MAX;   // the results are void: no more tiles
      for (int r = 0; r < WAVE_CLUSTER; ++r) st_cluster_u32(cluster_addr(smem_u32(&s_next[turn]), r), (unsigned)nx);
    }
    __syncwarp();

    auto parity_q = [&](int q) { return ((phase_q >> (q & (S - 1))) ^ (unsigned)(q >> LS)) & 1u; };
    auto parity_u = [&](int u) { return ((phase_u >> (u & (S - 1))) ^ (unsigned)(u >> LS)) & 1u; };
    // a wait inside the cluster ran out
    auto give_up = [&](unsigned site, int n, unsigned expect) {
      raise_timeout(g.ctl, site, tpos, n, OP, 0ull, expect);
      for (int r = 0; r < WAVE_CLUSTER; ++r) st_cluster_u32(cluster_addr(smem_u32(&s_broken), r), 1u);
    };
    const long long near_limit = 8 * g.spin_limit;
    // waits for a mbarrier's phase, all lanes together (a lane's own look may be
    // ahead of another's, and full-warp shuffles follow); false: it gave up
    auto vote = [](bool v) { return __all_sync(XFP_FULL, v) != 0; };
    auto await = [&](unsigned long long* bar, unsigned parity, int n, unsigned site) -> bool {
      const unsigned b = smem_u32(bar);
      Spin sp;
      if (warp_wait([&] { return mbar_try(b, parity); }, vote, [&] { return sp.step(near_limit); })) return true;
      give_up(site, n, parity);
      return false;
    };
    // z.r of this lane's line h of the block
    auto put_dot = [&](int h, const LineDot<VT, DOT32>& d) {
      const int j = jb * 8 + jl, k = kb * 8 + 2 * kl + h;
      if (j < lj && k < lk) g.partials[lbase + (long long)k * lj + j] = d.sum();
    };
    int armed = 0;   // (the helper's) slots filled in this tile
    // the range of own groups that each consumer takes
    const int lo_j = uj, hi_j = last_sent(uj, me.ng, nj.ng);
    const int lo_k = uk, hi_k = last_sent(uk, me.ng, nk.ng);
    if (!skip && me.ng > 0 && compute) {
      // ======================= compute warp =======================
      const bool edge_j = jl == (REV ? 0 : 7), edge_k = kl == (REV ? 0 : 3);
      const bool in_j = jl == (REV ? 7 : 0), in_k = kl == (REV ? 3 : 0);
      unsigned to_j = 0, bar_j = 0, to_k = 0, bar_k = 0;   // near consumers: slot 0
      if (near_nj) {
        to_j = cluster_addr(smem_u32(unit_at(kt)->slot[0].ej[HL * kl]), rank_at(cj + DIR, kt));
        bar_j = cluster_addr(smem_u32(&unit_at(kt)->full[0]), rank_at(cj + DIR, kt));
      }
      if (near_nk) {
        to_k = cluster_addr(smem_u32(unit_at(kt + DIR)->slot[0].ek[jl]), rank_at(cj, kt + DIR));
        bar_k = cluster_addr(smem_u32(&unit_at(kt + DIR)->full[0]), rank_at(cj, kt + DIR));
      }
      // this lane's cells in a group: factor/system values (r/y: lane * 4)
      const int cell = wave_cell_slot<ST>(jl, FACTOR ? half * 4 + kl : 2 * kl, 0, 0) - (FACTOR ? half * 2 * GE : 0);
      constexpr int CELL_H = 8 * (16 / (int)sizeof(ST));   // from line h = 0 to h = 1

      const bool far = (!near_nj && nj.ng > 0) || (!near_nk && nk.ng > 0);
      // ... as a lane's own count of groups it sends from lo on (0: none)
      const unsigned near_j = near_nj && edge_j && hi_j >= lo_j ? (unsigned)(hi_j - lo_j) + 1u : 0u;
      const unsigned near_k = near_nk && edge_k && hi_k >= lo_k ? (unsigned)(hi_k - lo_k) + 1u : 0u;
      VT* res = static_cast<VT*>(g.sw) + mybase * WAVE_ROW + wave_cell_slot<VT>(jl, half * 4 + kl, 0, 0);   // (the factor)

      bool bad = false;
      X ej[HL][4], ek[4];        // the producers' values of the group, in sweep order
      auto take_edges = [&](int u) {   // (zero where a producer has no such group: the helper's work)
        const int sl = u & (S - 1);
        bad |= !await(&sh.full[sl], parity_u(u), u, 3);
        const SL& in = sh.slot[sl];
#pragma unroll
        for (int s = 0; s < 4; ++s) {
#pragma unroll
          for (int h = 0; h < HL; ++h) ej[h][s] = in.ej[HL * kl + h][s];
          ek[s] = in.ek[jl][s];
        }
      };
      ST v[4][HL][4];            // operands: [step in sweep order][line][value]
      VT rhs[HL][4];
      auto load_step = [&](const SL& in, int s) {
#pragma unroll
        for (int h = 0; h < HL; ++h) cell_values(v[s][h], in.ops, cell + h * CELL_H, REV ? 3 - s : s);
      };
      auto load_rhs = [&](const SL& in) {
        if constexpr (!FACTOR) {
#pragma unroll
          for (int h = 0; h < HL; ++h) ldg(rhs[h], reinterpret_cast<const VT*>(in.ops) + (REV ? WAVE_Y : WAVE_R) + h * 128 + lane * 4);
        }
      };
      X ox[HL] = {}, oz_own = X{};               // this lane's previous step: x, and z for its other line
      X sy[HL] = {}, sz = X{};                   // the neighbour lanes' previous step
      X cj_[HL], ck_;                            // the producers' step before the group
      take_edges(0);
#pragma unroll
      for (int s = 0; s < 4; ++s) load_step(sh.slot[0], s);
      load_rhs(sh.slot[0]);
#pragma unroll
      for (int h = 0; h < HL; ++h) cj_[h] = ej[h][3];
      ck_ = ek[3];
      int room = 0;                              // (as last looked up)
      for (int q = 0; q < me.ng && !bad; ++q) {
        // Four steps.  What the chain waits for (the shuffles of a step's
        // results) is issued before what it does not (the next group's operands,
        // which take the registers of the step just done; stores).
        const SL& nx = sh.slot[(q + 1) & (S - 1)];   // (after the last group: whatever it holds)
        VT out[HL][4];
        X outj[HL][4], outk[4];
#pragma unroll
        for (int s = 0; s < 4; ++s) {
          const int e = REV ? 3 - s : s;
          X vy[HL], vz[HL], oy[HL], oz[HL];
          constexpr int inl = REV ? HL - 1 : 0, up = REV ? 0 : HL - 1;   // the line fed from lane -8, and that lane's line
#pragma unroll
          for (int h = 0; h < HL; ++h) vy[h] = in_j ? (s == 0 ? cj_[h] : ej[h][s == 0 ? 0 : s - 1]) : sy[h];
          if constexpr (HL == 2) vz[up] = oz_own;
          vz[inl] = in_k ? (s == 0 ? ck_ : ek[s == 0 ? 0 : s - 1]) : sz;
          CT pivot = CT(0);   // the factorisation's 1 / sqrt(d)
#pragma unroll
          for (int h = 0; h < HL; ++h) {
            if constexpr (FACTOR) {
              // column c: updates from columns c-nn, c-ni, c-1 in that order
              // (:137-184), each d -= L*L then d -= omega*L*missing; pivot
              // safeguard (:126-131)
              const CT dg = v[s][h][0], ux = v[s][h][1], uy = v[s][h][2], uz = v[s][h][3];
              CT dd = dg;
              const X src[3] = {vz[h], vy[h], ox[h]};
#pragma unroll
              for (int n = 0; n < 3; ++n) {
                dd = sub_rn(dd, mul_rn(src[n].a, src[n].a));
                dd = sub_rn(dd, mul_rn(mul_rn((CT)g.omega, src[n].a), src[n].b));
              }
              const CT piv = dd < mul_rn((CT)g.ratio, dg) ? dg : dd;
              const CT iv = dg != CT(0) ? rsqrt_ref(piv) : CT(0);
              const CT px = ux != CT(0) ? mul_rn(ux, iv) : CT(0), py = mul_rn(uy, iv), pz = mul_rn(uz, iv);
              pivot = iv;
              ox[h] = {px, add_rn(py, pz)};
              oy[h] = {py, add_rn(px, pz)};
              oz[h] = {pz, add_rn(px, py)};
            } else if constexpr (!REV) {
              // solve_lower: columns c-nn, c-ni, c-1 scatter into row c in that
              // order, then result[c] *= invdiag[c] (:198-203); this column's
              // products go to its three upper neighbours
              VT t = sub_rn(rhs[h][e], vz[h]);
              t = sub_rn(t, vy[h]);
              t = sub_rn(t, ox[h]);
              const VT y = mul_rn(t, v[s][h][3]);
              ox[h] = mul_rn(v[s][h][0], y);
              oy[h] = mul_rn(v[s][h][1], y);
              oz[h] = mul_rn(v[s][h][2], y);
              out[h][e] = y;
            } else {
              // solve_lower_transpose_in_place: x[c] -= L(m,c) x[m] for m =
              // c+1, c+ni, c+nn in that order, then x[c] *= invdiag[c] (:215-218)
              VT t = sub_rn(rhs[h][e], mul_rn(v[s][h][0], ox[h]));
              t = sub_rn(t, mul_rn(v[s][h][1], vy[h]));
              t = sub_rn(t, mul_rn(v[s][h][2], vz[h]));
              const VT z = mul_rn(t, v[s][h][3]);
              ox[h] = oy[h] = oz[h] = z;
              out[h][e] = z;
            }
            outj[h][s] = oy[h];
          }
          oz_own = oz[inl];
          outk[s] = oz[up];
#pragma unroll
          for (int h = 0; h < HL; ++h) sy[h] = REV ? shfl_down_any(oy[h], 1) : shfl_up_any(oy[h], 1);
          sz = REV ? shfl_down_any(oz[up], 8) : shfl_up_any(oz[up], 8);
          if (s == 0) take_edges(q + 1);   // (the first step needs the last group's)
          load_step(nx, s);
          if constexpr (FACTOR) {
            const VT f[4] = {(VT)ox[0].a, (VT)oy[0].a, (VT)oz[0].a, (VT)pivot};
            put_cell(res, 0, e, f);
          }
        }
#pragma unroll
        for (int h = 0; h < HL; ++h) cj_[h] = ej[h][3];
        ck_ = ek[3];
        if constexpr (FACTOR) {
          // ---- edge values to the upper neighbours ----
          if (q >= room) {
            // a consumer's slot may not be free yet (one lane's look, so that all
            // lanes agree)
            Spin sp;
            if (!warp_wait(
                    [&] {
                      room = __shfl_sync(XFP_FULL, min(ld_acquire_s32(&sh.limit[0]), ld_acquire_s32(&sh.limit[1])), 0);
                      return q < room;
                    },
                    vote, [&] { return sp.step(near_limit); })) {
              give_up(4, q, (unsigned)room);
              break;
            }
          }
          const bool to_near_j = (unsigned)(q - lo_j) < near_j, to_near_k = (unsigned)(q - lo_k) < near_k;
          if (to_near_j || to_near_k) {
            if (to_near_j) {
              const unsigned d = (unsigned)(q - uj) & (S - 1);
#pragma unroll
              for (int h = 0; h < HL; ++h) {
                uint32_t w[4 * P];
#pragma unroll
                for (int s = 0; s < 4; ++s) to_words(outj[h][s], w + s * P);
                send(to_j + d * (unsigned)sizeof(SL) + h * 4 * (unsigned)sizeof(X), bar_j + d * 8, w);
              }
            }
            if (to_near_k) {
              const unsigned d = (unsigned)(q - uk) & (S - 1);
              uint32_t w[4 * P];
#pragma unroll
              for (int s = 0; s < 4; ++s) to_words(outk[s], w + s * P);
              send(to_k + d * (unsigned)sizeof(SL), bar_k + d * 8, w);
            }
          }
          if (far) {
            if (!near_nj && edge_j && q >= lo_j && q <= hi_j) {
#pragma unroll
              for (int h = 0; h < HL; ++h)
                publish<X>(g.bj + ((size_t)(mybase + q) * 32 + (half * 4 + HL * kl + h) * 4) * P, gen, outj[h]);
            }
            if (!near_nk && edge_k && q >= lo_k && q <= hi_k)
              publish<X>(g.bk + ((size_t)(mybase + q) * 32 + jl * 4) * P, gen, outk);
          }
          res += WAVE_ROW;
        } else {
          // the results to the slot, for the sender (forward: over r)
#pragma unroll
          for (int h = 0; h < HL; ++h)
            stg(reinterpret_cast<VT*>(sh.slot[q & (S - 1)].ops) + OUT + h * 128 + lane * 4, out[h]);
        }
        load_rhs(nx);
        __syncwarp();
        if (lane == 0) mbar_arrive(FACTOR ? &sh.empty[q & (S - 1)] : &sh.ready[q & (S - 1)]);
      }
    } else if (!skip && me.ng > 0 && helper) {
      // ======================= helper warp =======================
      // operands of the next group to load
      const long long e0 = mybase + (REV ? me.ng - 1 : 0);
      const ST* src = FACTOR ? static_cast<const ST*>(g.sys) + e0 * 4 * GE + half * 2 * GE : static_cast<const ST*>(g.sw) + e0 * WAVE_ROW;
      auto arm = [&](int n) {   // slot of group n, edge values u = n (the whole warp, n = 0, 1, ...)
        SL& d = sh.slot[n & (S - 1)];
        const bool have_j = edge_comes(n, aj, pj.ng), have_k = edge_comes(n, ak, pk.ng);
        // a producer without such a group sends nothing: its edge values are zero
        // (and stay so, unless the slot's last use had some)
        const bool clear_j = !have_j && (n < S || edge_comes(n - S, aj, pj.ng));
        const bool clear_k = !have_k && (n < S || edge_comes(n - S, ak, pk.ng));
        if (clear_j || clear_k) {
          if (clear_j)
            for (int q = lane; q < (int)(sizeof(d.ej) / 16); q += 32) reinterpret_cast<uint4*>(&d.ej[0][0])[q] = make_uint4(0, 0, 0, 0);
          if (clear_k)
            for (int q = lane; q < (int)(sizeof(d.ek) / 16); q += 32) reinterpret_cast<uint4*>(&d.ek[0][0])[q] = make_uint4(0, 0, 0, 0);
        }
        __syncwarp();
        if (lane == 0) {
          unsigned long long* b = &sh.full[n & (S - 1)];
          // The compute warp wrote its results over r or y here with ordinary stores,
          // which reached this lane through `ready`, `empty` and the warp's barrier;
          // without the fence the copy, of another proxy, would not be ordered after them
          fence_bulk();
          mbar_expect(b, (have_j ? (unsigned)sizeof(d.ej) : 0u) + (have_k ? (unsigned)sizeof(d.ek) : 0u) +
                             (n < me.ng ? W::IN * (unsigned)sizeof(ST) : 0u));
          if (n < me.ng) bulk_load(d.ops, src, W::IN * sizeof(ST), b);
        }
        src += DIR * (FACTOR ? 4 * GE : WAVE_ROW);
      };
      const unsigned ack_j = near_pj ? cluster_addr(smem_u32(&unit_at(kt)->limit[0]), rank_at(cj - DIR, kt)) : 0u;
      const unsigned ack_k = near_pk ? cluster_addr(smem_u32(&unit_at(kt - DIR)->limit[1]), rank_at(cj, kt - DIR)) : 0u;
      // who is told of a slot given back, a lane each: the producers in this
      // cluster (in their numbering) and the courier
      const bool far_in = (!near_pj && pj.ng > 0) || (!near_pk && pk.ng > 0);
      const unsigned tell = lane == 0 ? ack_j : lane == 1 ? ack_k : cluster_addr(smem_u32(&sh.freed), rank);
      const int tell_ahead = lane == 0 ? S + aj : lane == 1 ? S + ak : 0;
      const bool told = (lane == 0 && near_pj) || (lane == 1 && near_pk) || (lane == 2 && far_in);
      for (; armed < S && armed <= me.ng; ++armed) arm(armed);
      LineDot<VT, DOT32> dot;   // of the lines h = 1
      for (int q = 0; q < me.ng; ++q) {
        const int sl = q & (S - 1);
        if (!await(&sh.empty[sl], parity_q(q), q, 7)) break;
        VT z[4], rr[4];
        if constexpr (REV) {
          ldg(z, reinterpret_cast<const VT*>(sh.slot[sl].ops) + WAVE_Y + 128 + lane * 4);
          ldg(rr, reinterpret_cast<const VT*>(sh.slot[sl].ops) + WAVE_R + 128 + lane * 4);
          __syncwarp();
        }
        if (q + S <= me.ng) {
          arm(q + S);
          ++armed;
        }
        // the slot is the producers' again (all the rest at the end)
        if (told) st_release_s32(tell, (q + 1 == me.ng ? INT_MAX / 2 : q + 1) + tell_ahead);
        if constexpr (REV) dot.add(z, rr);
      }
      if constexpr (REV) put_dot(1, dot);
    } else if (!skip && me.ng > 0 && courier) {
      // ======================= courier warp =======================
      // far producers: this block's u .. last, FB under way; lane = line * 4 + step
      const unsigned want = gen + g.expect_bias;   // bias != 0 only in the expired-wait diagnostic
      constexpr int LJ = HL * 4;                   // lines of this unit's j edge
      const bool use_j = lane < 4 * LJ;
      struct Far {
        int u, last;
        EdgeWords<X> w[FB];
      };
      Far fj, fk;
      auto range = [&](Far& f, bool near, int a, const WBlk& p) {
        f.u = first_edge(a);
        f.last = near ? -1 : last_edge(a, p.ng, me.ng);
#pragma unroll
        for (int d = 0; d < FB; ++d)
#pragma unroll
          for (int q = 0; q < P; ++q) f.w[d].w[q] = 0ull;
      };
      range(fj, near_pj, aj, pj);
      range(fk, near_pk, ak, pk);
      const unsigned long long* src_j =
          g.bj + ((size_t)(gbase + pj.goff) * 32 + half * 16 + lane) * P;
      const unsigned long long* src_k = g.bk + ((size_t)(gbase + pk.goff) * 32 + lane) * P;
      const unsigned to_j = cluster_addr(smem_u32(&sh.slot[0].ej[(lane >> 2) % LJ][lane & 3]), rank);
      const unsigned to_k = cluster_addr(smem_u32(&sh.slot[0].ek[lane >> 2][lane & 3]), rank);
      const unsigned bar = cluster_addr(smem_u32(&sh.full[0]), rank);
      auto request = [&](Far& f, const unsigned long long* src, int a, bool use) {
#pragma unroll
        for (int d = 0; d < FB; ++d)
          if (use && f.u + d <= f.last && !f.w[d].ready(want)) f.w[d].load(src + (size_t)(f.u + d + a) * 32 * P);
      };
      bool late = false;   // a wait ran out: what the words hold will do
      int room = S;   // (with a look at `freed` for every group: 128^3 FP64 8.43 ms against 8.35)
      auto forward = [&](Far& f, unsigned to, bool use) -> bool {
        bool moved = false;
#pragma unroll
        for (int d = 0; d < FB; ++d) {
          if (f.u > f.last || !__all_sync(XFP_FULL, late || !use || f.w[0].ready(want))) break;
          const unsigned at = (unsigned)f.u & (S - 1);
          // its slot is free once group u - S is done with (one lane's look, so
          // that all lanes agree; a count, since the courier may be any number
          // of groups ahead, where a parity would be ambiguous); looked at again only
          // when the last count is used up
          if (f.u >= room) room = __shfl_sync(XFP_FULL, ld_acquire_s32(&sh.freed), 0) + S;
          if (f.u >= room) break;
          if (use) {
            uint32_t w[P];
            to_words(f.w[0].value(), w);
            send(to + at * (unsigned)sizeof(SL), bar + at * 8, w);
          }
#pragma unroll
          for (int e = 0; e + 1 < FB; ++e) f.w[e] = f.w[e + 1];
          f.w[FB - 1].w[0] = 0ull;
          ++f.u;
          moved = true;
        }
        return moved;
      };
      Spin sp;
      while (fj.u <= fj.last || fk.u <= fk.last) {
        request(fj, src_j, aj, use_j);
        request(fk, src_k, ak, true);
        bool moved = forward(fj, to_j, use_j);
        moved |= forward(fk, to_k, true);
        if (moved) {
          sp = Spin();
          continue;
        }
        if (late) {   // only a slot is waited for
          if (vote(sp.step(near_limit))) continue;
          give_up(8, fj.u, want);
          break;
        }
        const bool go = sp.step(g.ctl, g.spin_limit);
        if (!vote(go)) {
          if (!go) raise_timeout(g.ctl, 8, tpos, fj.u, OP, fj.w[0].w[0], want);
          late = true;
          sp = Spin();
        }
      }
    }
    if constexpr (!FACTOR) {
      if (!skip && me.ng > 0 && warp >= 3 * NW) {
        // ======================= sender warp =======================
        // A lane each for the 8 lines of the j edge and the 8 of the k edge: the
        // group's four values go to the consumer's slot or to global memory.
        const bool is_j = lane < 8, is_edge = lane < 16;
        const int line_j = is_j ? (REV ? 0 : 7) : lane & 7, line_k = is_j ? lane : (REV ? 0 : 7);
        const int lo = is_j ? lo_j : lo_k, hi = is_j ? hi_j : hi_k;
        const bool near = is_j ? near_nj : near_nk;
        unsigned count = is_edge && hi >= lo ? (unsigned)(hi - lo) + 1u : 0u;   // groups from lo on
        unsigned to = 0, bar = 0;   // near: slot 0
        if (near) {
          SL& d = unit_at(is_j ? kt : kt + DIR)->slot[0];
          const int r = is_j ? rank_at(cj + DIR, kt) : rank_at(cj, kt + DIR);
          to = cluster_addr(smem_u32(is_j ? d.ej[lane & 7] : d.ek[lane & 7]), r);
          bar = cluster_addr(smem_u32(&unit_at(is_j ? kt : kt + DIR)->full[0]), r);
        }
        unsigned long long* const pub = (is_j ? g.bj : g.bk) + ((size_t)mybase * 32 + (lane & 7) * 4) * P;
        const int* const limit = &sh.limit[is_j ? 0 : 1];
        const int coef = wave_cell_slot<VT>(line_j, line_k, 0, is_j ? 1 : 2);
        constexpr int CELL_E = 128;              // from one step's cells to the next's
        const int edge_at = OUT + wave_line_slot(line_j, line_k);
        VT* res = static_cast<VT*>(g.sw) + (mybase + (REV ? me.ng - 1 : 0)) * WAVE_ROW + WAVE_Y + lane * 4;
        int room = 0;
        LineDot<VT, DOT32> dot;   // of the lines h = 0 (the helper has h = 1)
        for (int q = 0; q < me.ng; ++q) {
          const int sl = q & (S - 1);
          if (!await(&sh.ready[sl], parity_q(q), q, 9)) break;
          const VT* const ops = reinterpret_cast<const VT*>(sh.slot[sl].ops);
          if ((unsigned)(q - lo) < count) {
            VT y[4], w[4];
            ldg(y, ops + edge_at);
#pragma unroll
            for (int s = 0; s < 4; ++s) {
              if (REV) w[s] = y[3 - s];
              else w[s] = mul_rn(ops[coef + s * CELL_E], y[s]);   // L(m,c) y[c], as in the block
            }
            if (near) {
              if (q >= room) {
                // the consumer's slot may not be free yet
                room = ld_acquire_s32(limit);
                for (Spin sp; q >= room; room = ld_acquire_s32(limit)) {
                  if (!sp.step(near_limit)) {
                    give_up(4, q, (unsigned)room);
                    count = 0;   // it is not free: nothing more goes there
                    break;
                  }
                }
              }
              if (count != 0) {
                const unsigned d = (unsigned)(q - lo) & (S - 1);
                uint32_t m[4 * P];
#pragma unroll
                for (int s = 0; s < 4; ++s) to_words(w[s], m + s * P);
                send(to + d * (unsigned)sizeof(SL), bar + d * 8, m);
              }
            } else {
              publish<X>(pub + (size_t)q * 32 * P, gen, w);
            }
          }
          __syncwarp();
          VT z[2][4], rr[4];
#pragma unroll
          for (int h = 0; h < 2; ++h) ldg(z[h], ops + OUT + h * 128 + lane * 4);
          if constexpr (REV) ldg(rr, ops + WAVE_R + lane * 4);
          __syncwarp();
          if (lane == 0) mbar_arrive(&sh.empty[sl]);
#pragma unroll
          for (int h = 0; h < 2; ++h) stg(res + h * 128, z[h]);
          res += DIR * WAVE_ROW;
          if constexpr (REV) dot.add(z[0], rr);
        }
        if constexpr (REV) put_dot(0, dot);
      }
    }
    __syncwarp();
    cluster_sync();   // every slot has been read; s_next and s_broken are set
    if (*(volatile int*)&s_broken != 0) {
      // Nothing more is sent.  What is under way to this CTA's slots lands before
      // any CTA of the cluster leaves: a slot's mbarrier tells, unless a value that
      // was never sent is missing from it too, for which 10 ms have to do.
      if (helper) {
        const unsigned long long t0 = now_ns();
        for (int u = max(0, armed - S); u < armed; ++u)
          (void)warp_wait([&] { return mbar_try(smem_u32(&sh.full[u & (S - 1)]), parity_u(u)); }, vote,
                          [&] { return now_ns() - t0 < 10000000ull; });
      }
      __syncwarp();
      cluster_sync();
      break;
    }
    // slot n has carried the groups q = n, n + S, ... < ng and the edges u = n, n + S, ... <= ng
    if (!skip && me.ng > 0)
#pragma unroll
      for (int n = 0; n < S; ++n) {
        phase_q ^= (unsigned)(((me.ng - 1 - n + S) >> LS) & 1) << n;
        phase_u ^= (unsigned)(((me.ng - n + S) >> LS) & 1) << n;
      }
    pos = *(volatile int*)&s_next[turn];
  }

  // ---------------- launch epilogue: the last cluster closes the generation ----------------
  unsigned last = 0;
  if (rank == 0 && threadIdx.x == 0) {
    __threadfence();
    last = atomicAdd(&g.ctl->finished, 1u) == (unsigned)nclusters - 1;
    __threadfence();
  }
  if (REV && g.scal != nullptr) {
    // z.r: every CTA of the last cluster sums its share of the chunks
    if constexpr (REV) {
      constexpr int NCH = 8, P = 64, SUMS = 256 / WAVE_CLUSTER / NCH;   // the first SUMS warps
      static_assert(SUMS * NCH * (P + 1) * sizeof(double) <= WaveOp<OP, VT, CT>::S * sizeof(SL) && SUMS <= 2 * NW, "");
      __shared__ unsigned s_last;
      __shared__ double s_sum[256];
      if (rank == 0 && threadIdx.x == 0)
        for (int r = 0; r < WAVE_CLUSTER; ++r) st_cluster_u32(cluster_addr(smem_u32(&s_last), r), last);
      __syncwarp();
      cluster_sync();
      if (*(volatile unsigned*)&s_last == 0u) return;
      if (warp < SUMS) {
        const int first = (rank * SUMS + warp) * NCH;
        double* const buf = reinterpret_cast<double*>(wave_smem) + warp * NCH * (P + 1);
        const double c = chunk_sums<DOT32, NCH, P>(g.partials, (long long)g.nj * g.nk, first, buf);
        if (lane < NCH)
          asm volatile("st.relaxed.cluster.shared::cluster.f64 [%0], %1;"
                       ::"r"(cluster_addr(smem_u32(&s_sum[first + lane]), 0)), "d"(c) : "memory");
      }
      __syncwarp();
      cluster_sync();
      if (rank != 0 || warp != 0) return;
      const double rho_new = chunk_tree<DOT32>(s_sum);
      if (lane != 0) return;
      PcgScalars* sc = g.scal;
      if (g.bwd_mode == 0) {
        sc->rho = rho_new;
        if (rho_new == 0.0 || rho_new != rho_new) end_solve(sc, -5);
      } else {
        sc->beta = DOT32 ? (double)__fdiv_rn((float)rho_new, (float)sc->rho) : __ddiv_rn(rho_new, sc->rho);
        sc->rho = rho_new;
      }
    }
  } else if (!last) {
    return;
  }
  g.ctl->finished = 0;
  g.ctl->ticket = 0;
  __threadfence();
  atomicExch(&g.ctl->gen, gen + 1);
}

// A launch's configuration but for its grid and stream, and the clusters that the
// current device holds at once (the kernel's attribute is per device too).
template <int OP, typename VT, typename CT>
struct WaveLaunch {
  static constexpr int smem = warps_of<OP>() * (int)sizeof(UnitShared<OP, VT, CT>);
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute attr[3];
  int resident = 0;
  cudaError_t prepare() {
    static std::atomic<int> known[64];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = WAVE_CLUSTER;
    attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    attr[2].id = cudaLaunchAttributeCooperative;
    attr[2].val.cooperative = 1;
    cfg.blockDim = dim3(roles_of<OP>() * 32 * warps_of<OP>());
    cfg.gridDim = dim3(WAVE_CLUSTER);
    cfg.dynamicSmemBytes = smem;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    resident = known[dev & 63].load();
    if (resident == 0) {
      int n = 0;
      e = cudaFuncSetAttribute(wave_kernel<OP, VT, CT>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
      if (e == cudaSuccess) e = cudaOccupancyMaxActiveClusters(&n, wave_kernel<OP, VT, CT>, &cfg);
      if (e != cudaSuccess) return e;
      if (n < 1) return cudaErrorLaunchOutOfResources;
      known[dev & 63] = resident = n;
    }
    return cudaSuccess;
  }
};
template <int OP, typename VT, typename CT>
cudaError_t launch(const WaveArgs& g, cudaStream_t st) {
  WaveLaunch<OP, VT, CT> L;
  const cudaError_t e = L.prepare();
  if (e != cudaSuccess) return e;
  const int clusters = std::min(L.resident, g.ntiles);
  L.cfg.gridDim = dim3(WAVE_CLUSTER * clusters);
  // Clusters that wait for one another have to be resident together; a lone one
  // waits for none.  (ncu refuses cooperative cluster launches, "LaunchFailed", so grids
  // of up to 32 x 32 lines are the ones that can be profiled.)
  L.cfg.numAttrs = clusters > 1 ? 3 : 2;
  L.cfg.stream = st;
  ++g_kernel_launches;
  return cudaLaunchKernelEx(&L.cfg, wave_kernel<OP, VT, CT>, g);
}

// one thread per group of 4 cells: dir 0 line -> sweep, dir 1 sweep -> line
template <typename T>
__global__ void sw_permute_kernel(T* __restrict__ line, T* __restrict__ sw, const int* __restrict__ gperm,
                                  long long ngroups, int dir) {
  for (long long q = blockIdx.x * (long long)blockDim.x + threadIdx.x; q < ngroups;
       q += (long long)gridDim.x * blockDim.x) {
    T v[4];
    if (dir == 0) {
      ldg(v, line + 4 * q);
      stg(sw + wave_value(gperm[q]), v);
    } else {
      ldg(v, sw + wave_value(gperm[q]));
      stg(line + 4 * q, v);
    }
  }
}

// The factor in the line layout, keyed by the higher cell (lx[c] = L(c,c-1) and
// so on), for the stage dumps.
template <typename T>
__global__ void factor_lines_kernel(const T* __restrict__ fac, const Line* __restrict__ lines, int nj, int nk,
                                    const WBlk* __restrict__ blks, int NJB, T* __restrict__ lx, T* __restrict__ ly,
                                    T* __restrict__ lz, T* __restrict__ inv) {
  const int lane = threadIdx.x & 31;
  const long long nlines = (long long)nj * nk;
  auto at = [&](int i, int j, int k, int a) -> T {
    if (j < 0 || k < 0) return T(0);
    const Line L = lines[(size_t)k * nj + j];
    if ((unsigned)(i - L.lo) >= (unsigned)L.len) return T(0);
    const int t = i + j + k;
    const WBlk b = blks[(size_t)(k >> 3) * NJB + (j >> 3)];
    return fac[(size_t)(b.goff + (t >> 2) - b.g0) * WAVE_ROW + wave_cell_slot<T>(j, k, t & 3, a)];
  };
  for (long long line = (long long)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); line < nlines;
       line += (long long)gridDim.x * (blockDim.x >> 5)) {
    const Line L = lines[line];
    const int j = (int)(line % nj), k = (int)(line / nj);
    for (int q = lane; q < L.len; q += 32) {
      const int i = L.lo + q;
      const size_t c = (size_t)L.off + q;
      lx[c] = at(i - 1, j, k, 0);
      ly[c] = at(i, j - 1, k, 1);
      lz[c] = at(i, j, k - 1, 2);
      inv[c] = at(i, j, k, 3);
    }
  }
}

unsigned cap_blocks(long long n) { return (unsigned)std::max<long long>(1, std::min<long long>((n + 255) / 256, 148LL * 16)); }

}  // namespace

template <typename VT, typename CT>
cudaError_t wave_launch(int op, const WaveArgs& g, cudaStream_t st) {
  if (g.ntiles <= 0) return cudaSuccess;
  switch (op) {
    case SWEEP_FACTOR: return launch<SWEEP_FACTOR, VT, CT>(g, st);
    case SWEEP_FWD: return launch<SWEEP_FWD, VT, CT>(g, st);
    default: return launch<SWEEP_BWD, VT, CT>(g, st);
  }
}
template <typename VT, typename CT>
cudaError_t wave_prepare() {
  const cudaError_t e = WaveLaunch<SWEEP_FWD, VT, CT>().prepare();
  return e != cudaSuccess ? e : WaveLaunch<SWEEP_BWD, VT, CT>().prepare();
}
template cudaError_t wave_prepare<double, double>();
template cudaError_t wave_prepare<float, float>();
template cudaError_t wave_prepare<float, double>();
template cudaError_t wave_launch<double, double>(int, const WaveArgs&, cudaStream_t);
template cudaError_t wave_launch<float, float>(int, const WaveArgs&, cudaStream_t);
template cudaError_t wave_launch<float, double>(int, const WaveArgs&, cudaStream_t);

template <typename T>
cudaError_t sw_permute(T* line, T* sw, const int* gperm, long long M, int dir, cudaStream_t st) {
  if (M <= 0) return cudaSuccess;
  ++g_kernel_launches;
  sw_permute_kernel<T><<<cap_blocks(M / 4), 256, 0, st>>>(line, sw, gperm, M / 4, dir);
  return cudaGetLastError();
}
template cudaError_t sw_permute<float>(float*, float*, const int*, long long, int, cudaStream_t);
template cudaError_t sw_permute<double>(double*, double*, const int*, long long, int, cudaStream_t);

template <typename T>
cudaError_t factor_lines(const T* fac, const Line* lines, int nj, int nk, const WBlk* blks, int NJB, T* const F[4],
                         cudaStream_t st) {
  ++g_kernel_launches;
  factor_lines_kernel<T><<<cap_blocks((long long)nj * nk * 32), 256, 0, st>>>(fac, lines, nj, nk, blks, NJB, F[0], F[1],
                                                                           F[2], F[3]);
  return cudaGetLastError();
}
template cudaError_t factor_lines<float>(const float*, const Line*, int, int, const WBlk*, int, float* const[4],
                                         cudaStream_t);
template cudaError_t factor_lines<double>(const double*, const Line*, int, int, const WBlk*, int, double* const[4],
                                          cudaStream_t);

}  // namespace xfp

// ggem_cells.cu -- Kernel A: the sorted cell list and the cached pair list.
//
// Replaces PointMesh::reinit (point_mesh.C:245-289): the element-point
// containing list (:573-648) becomes a counting sort of particles by cell,
// and the per-particle neighbour lists (:652-848) with their stored
// displacement vectors (:220-241) become fixed-width rows of (source slot,
// stencil code) entries, built in one pass per configuration, in both
// precisions (an FP64 context without a list sweeps the cell stencil).
//
// Bound: HBM.  Algorithmic bytes per particle of the cell build: 24 (read
// xyz) + 4 (cell id) + 4 (order) + 4 (rank) + 32 (pos64) + 16 (pos32) plus
// the scatter re-reads; the list build writes 4 B per listed pair once.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <vector>

#include "ggem_internal.cuh"

namespace ggem {
namespace {

__device__ __forceinline__ int wrap_index(int k, int n) {
  k %= n;
  return k < 0 ? k + n : k;
}

// cell coordinate along one axis, as the oracle and the reference's element
// search would compute it: floor((x - lo) / h), periodic axes wrapped first
__device__ __forceinline__ void assign_one(int64_t i, const double *__restrict__ xyz,
                                           const Grid &g, int32_t *__restrict__ cell_of,
                                           int32_t *__restrict__ count,
                                           double4_32a *__restrict__ wrapped,
                                           int *__restrict__ err) {
  double p[3];
  int c[3];
  bool bad = false, nonfinite = false;
  for (int d = 0; d < 3; ++d) {
    double x = xyz[3 * i + d];
    // common case without FP64 arithmetic (GB300 issues FP64 at a small
    // fraction of the FP32 rate): inside the box away from its faces and
    // away from the cell faces, the FP32 index is the FP64 one
    {
      const float t = d2f_bits(x) - g.lo32[d];  // NaN and infinities fail below
      if (t > g.margin32[d] && t < g.L32[d] - g.margin32[d]) {
        const float q = t * g.inv_h32[d];
        const float fq = floorf(q);
        if (q - fq > g.band32[d] && (fq + 1.f) - q > g.band32[d]) {
          const int k = (int)fq;
          p[d] = x;
          c[d] = k < 0 ? 0 : (k >= g.nc[d] ? g.nc[d] - 1 : k);
          continue;
        }
      }
    }
    if (!isfinite(x)) {  // reported as a bad argument; the cell index stays in range
      nonfinite = true;
      x = g.lo[d];
    }
    double t = x - g.lo[d];
    // (FP64 runs at a small fraction of the FP32 rate: fmod and the division
    // are taken only where they can change the result)
    if (g.periodic[d]) {
      // inside, fmod(t, L) == t; a bead inside the box whose x - lo rounded
      // up to L keeps t = L and so the last cell (the element search's
      // closed upper face, point_mesh.C) instead of wrapping to cell 0
      if (!(t >= 0.0 && t < g.L[d]) && !(x >= g.lo[d] && x < g.lo[d] + g.L[d])) {
        t = fmod(t, g.L[d]);
        if (t < 0) t += g.L[d];
        if (t >= g.L[d]) t = 0.0;
        x = g.lo[d] + t;  // a caller's value inside the box is kept as it is
      }
    } else if (!(t >= 0.0 && t <= g.L[d])) {
      bad = true;
    }
    p[d] = x;
    // floor(t / h): t * (1/h) is within a few ulps of t / h, so its floor is
    // the same unless it lies within 1e-9 of an integer (|t / h| < 1e6)
    const double q = t * g.inv_h[d];
    double fq = floor(q);
    if (q - fq < 1e-9 || (fq + 1.0) - q < 1e-9 || !(fabs(q) < 1e6)) fq = floor(t / g.h[d]);
    int k = (int)fq;
    c[d] = k < 0 ? 0 : (k >= g.nc[d] ? g.nc[d] - 1 : k);
  }
  if (bad) atomicOr(err, kErrOutOfDomain);
  if (nonfinite) atomicOr(err, kErrNonFinite);
  const int32_t id = c[0] + g.nc[0] * (c[1] + g.nc[1] * c[2]);
  cell_of[i] = id;
  atomicAdd(&count[id], 1);
  wrapped[i] = make_double4_32a(p[0], p[1], p[2], 0.0);
}

__global__ void k_assign(int64_t n, const double *__restrict__ xyz, Grid g,
                         int32_t *__restrict__ cell_of, int32_t *__restrict__ count,
                         double4_32a *__restrict__ wrapped, int *__restrict__ err) {
  wait_prior_grid();
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i < n) assign_one(i, xyz, g, cell_of, count, wrapped, err);
}

// ---- exclusive scan (warp shuffles, 1024-element blocks) ----------------
template <typename T>
__global__ void k_scan_block(const T *__restrict__ in, T *__restrict__ out,
                             int64_t *__restrict__ block_sums, int64_t n) {
  __shared__ T warp_tot[32];
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  T v = (i < n) ? in[i] : T(0);
  T x = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    T y = __shfl_up_sync(0xffffffffu, x, o);
    if (lane >= o) x += y;
  }
  if (lane == 31) warp_tot[warp] = x;
  __syncthreads();
  if (warp == 0) {
    const int nw = blockDim.x >> 5;
    T w = (lane < nw) ? warp_tot[lane] : T(0);
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      T y = __shfl_up_sync(0xffffffffu, w, o);
      if (lane >= o) w += y;
    }
    if (lane < nw) warp_tot[lane] = w;  // inclusive warp prefix
  }
  __syncthreads();
  const T base = warp ? warp_tot[warp - 1] : T(0);
  if (i < n) out[i] = base + x - v;
  if (threadIdx.x == blockDim.x - 1 && block_sums) block_sums[blockIdx.x] = (int64_t)(base + x);
}

template <typename T>
__global__ void k_scan_add(T *__restrict__ out, const int64_t *__restrict__ block_off, int64_t n,
                           const T *__restrict__ in, T *__restrict__ total_slot) {
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i < n) {
    out[i] += (T)block_off[blockIdx.x];
    if (i == n - 1 && total_slot) *total_slot = out[i] + in[i];
  }
}

template <typename T>
__global__ void k_scan_total(T *__restrict__ out, const T *__restrict__ in, int64_t n) {
  if (threadIdx.x == 0 && blockIdx.x == 0) out[n] = (n > 0) ? out[n - 1] + in[n - 1] : T(0);
}

template <typename T>
int scan_impl(ggem_ctx *c, const T *in, T *out, int64_t n, int level) {
  const int B = 1024;
  const int64_t nb = (n + B - 1) / B;
  if (n <= 0) {
    k_scan_total<T><<<1, 1, 0, c->stream>>>(out, in, 0);
    return check_launch(c, "scan");
  }
  if ((int)c->scan_scratch.size() <= 2 * level + 1) {
    c->scan_scratch.resize(2 * level + 2, nullptr);
  }
  for (int k = 0; k < 2; ++k)
    if (!c->scan_scratch[2 * level + k]) c->scan_scratch[2 * level + k] = new DevBuf<int64_t>();
  DevBuf<int64_t> &sums = *c->scan_scratch[2 * level];
  DevBuf<int64_t> &offs = *c->scan_scratch[2 * level + 1];
  cudaError_t e = sums.ensure(nb + 1);
  if (e == cudaSuccess) e = offs.ensure(nb + 1);
  if (e != cudaSuccess) return cuda_fail(c, e, "scan scratch");
  k_scan_block<T><<<(unsigned)nb, B, 0, c->stream>>>(in, out, sums.p, n);
  int rc = check_launch(c, "scan block");
  if (rc) return rc;
  if (nb > 1) {
    rc = scan_impl<int64_t>(c, sums.p, offs.p, nb, level + 1);
    if (rc) return rc;
    k_scan_add<T><<<(unsigned)nb, B, 0, c->stream>>>(out, offs.p, n, in, out + n);
    return check_launch(c, "scan add");
  }
  k_scan_total<T><<<1, 1, 0, c->stream>>>(out, in, n);
  return check_launch(c, "scan total");
}

// barrier of all threads of the cluster (shared memory written before it is
// visible to the cluster after it)
__device__ __forceinline__ void cluster_barrier() {
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}

// the value of another block's copy of a shared variable
__device__ __forceinline__ int32_t cluster_read(const int32_t *p, int rank) {
  const uint32_t a = (uint32_t)__cvta_generic_to_shared(p);
  uint32_t r;
  int32_t v;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(rank));
  asm volatile("ld.shared::cluster.s32 %0, [%1];" : "=r"(v) : "r"(r) : "memory");
  return v;
}

// the cell list's exclusive scan in one launch of one cluster of up to eight
// blocks: each takes a consecutive run of tiles of 4096 counts (four
// consecutive counts per thread, a running carry over its tiles), tells the
// others its total through distributed shared memory and adds the totals of
// the blocks before it; start[0..ncell].  The counts are zeroed as they are
// read, ready for the next build's k_assign, and so are the pair-list
// statistics (stat, when given) that the list build of the same
// configuration accumulates.  Latency-bound: one block takes 15 us for 24389
// counts, and the scan for any size four launches and two clears.  FP32
// matvec with its list at N = 400k (48778 cells) 353 -> 335 us, FP32 step at
// N = 200k 565 -> 557 us.  Beyond 131072 cells the blocks of one cluster
// would be the bottleneck and device_exclusive_scan_i32 runs.
constexpr int kScanTiles = 4;    // tiles per block
constexpr int kScanCluster = 8;  // blocks
constexpr int64_t kScanCellsMax = 4096 * kScanTiles * kScanCluster;

__global__ void __launch_bounds__(1024) k_scan_cells(int32_t *__restrict__ count,
                                                     int32_t *__restrict__ start, int64_t n,
                                                     int tiles,
                                                     unsigned long long *__restrict__ stat) {
  wait_prior_grid();
  __shared__ int32_t warp_tot[2][32];
  __shared__ int32_t s_total, s_before;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int rank = blockIdx.x;  // (one cluster)
  if (rank == 0 && stat && threadIdx.x < 2) stat[threadIdx.x] = 0ull;
  const int64_t c0 = (int64_t)rank * tiles * 4096 + 4 * threadIdx.x;
  int32_t v[kScanTiles][4], run[kScanTiles];
#pragma unroll
  for (int k = 0; k < kScanTiles; ++k)
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int64_t i = c0 + k * 4096 + j;
      v[k][j] = (k < tiles && i < n) ? count[i] : 0;
    }
#pragma unroll
  for (int k = 0; k < kScanTiles; ++k)
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int64_t i = c0 + k * 4096 + j;
      if (k < tiles && i < n) count[i] = 0;
    }
  int32_t carry = 0;
#pragma unroll
  for (int k = 0; k < kScanTiles; ++k) {
    if (k < tiles) {
      const int32_t tsum = (v[k][0] + v[k][1]) + (v[k][2] + v[k][3]);
      int32_t x = tsum;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int32_t y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
      }
      int32_t *wt = warp_tot[k & 1];  // alternate buffers: one barrier per tile
      if (lane == 31) wt[warp] = x;
      __syncthreads();
      int32_t w = wt[lane];
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int32_t y = __shfl_up_sync(0xffffffffu, w, o);
        if (lane >= o) w += y;
      }
      // every warp scans the 32 warp totals itself (no second barrier)
      const int32_t before = __shfl_sync(0xffffffffu, w, (warp + 31) & 31);
      run[k] = carry + (warp ? before : 0) + x - tsum;
      carry += __shfl_sync(0xffffffffu, w, 31);
    }
  }
  int32_t base = 0;
  if (gridDim.x > 1) {
    if (threadIdx.x == 0) s_total = carry;
    cluster_barrier();
    if (warp == 0) {  // lane r reads block r's total
      int32_t t = lane < rank ? cluster_read(&s_total, lane) : 0;
      t = __reduce_add_sync(0xffffffffu, t);
      if (lane == 0) s_before = t;
    }
    cluster_barrier();  // no block leaves while its total is read
    base = s_before;
  }
#pragma unroll
  for (int k = 0; k < kScanTiles; ++k) {
    if (k < tiles) {
      int32_t r = base + run[k];
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const int64_t i = c0 + k * 4096 + j;
        if (i < n) start[i] = r;
        r += v[k][j];
      }
    }
  }
  if (rank == (int)gridDim.x - 1 && threadIdx.x == 0) start[n] = base + carry;
}

__global__ void k_scatter(int64_t n, const int32_t *__restrict__ cell_of,
                          const int32_t *__restrict__ start, int32_t *__restrict__ fill,
                          int32_t *__restrict__ order) {
  wait_prior_grid();
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i >= n) return;
  const int32_t cid = cell_of[i];
  const int32_t slot = start[cid] + atomicAdd(&fill[cid], 1);
  order[slot] = (int32_t)i;
}

// ascending particle id inside each cell (deterministic slot order, and the
// order of build_elem_point_containing_list, point_mesh.C:585-631): cells of
// up to 16 particles are sorted in registers by an odd-even transposition
// network, larger ones by insertion in place.  The cell's fill counter is
// zeroed for the next build.
__global__ void k_sort_cells(int64_t ncell, const int32_t *__restrict__ start,
                             int32_t *__restrict__ order, int32_t *__restrict__ fill) {
  wait_prior_grid();
  const int64_t cidx = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (cidx >= ncell) return;
  fill[cidx] = 0;  // scattered; ready for the next build
  const int32_t b = start[cidx], e = start[cidx + 1];
  const int32_t m = e - b;
  if (m <= 1) return;
  if (m <= 16) {
    int32_t v[16];
#pragma unroll
    for (int k = 0; k < 16; ++k) v[k] = k < m ? order[b + k] : 0x7fffffff;
#pragma unroll
    for (int r = 0; r < 16; ++r) {
#pragma unroll
      for (int k = r & 1; k + 1 < 16; k += 2) {
        const int32_t lo = min(v[k], v[k + 1]), hi = max(v[k], v[k + 1]);
        v[k] = lo;
        v[k + 1] = hi;
      }
    }
#pragma unroll
    for (int k = 0; k < 16; ++k)
      if (k < m) order[b + k] = v[k];
    return;
  }
  for (int32_t k = b + 1; k < e; ++k) {
    const int32_t v = order[k];
    int32_t m = k - 1;
    while (m >= b && order[m] > v) {
      order[m + 1] = order[m];
      --m;
    }
    order[m + 1] = v;
  }
}

__device__ __forceinline__ void gather_one(int64_t s, const Grid &g,
                                           const int32_t *__restrict__ order,
                                           const int32_t *__restrict__ cell_of,
                                           const double4_32a *__restrict__ wrapped,
                                           double4_32a *__restrict__ pos64,
                                           float4 *__restrict__ pos32) {
  const int32_t i = order[s];
  const double4_32a p = wrapped[i];
  pos64[s] = p;
  const int32_t cid = cell_of[i];
  const int cx = cid % g.nc[0], cy = (cid / g.nc[0]) % g.nc[1], cz = cid / (g.nc[0] * g.nc[1]);
  // position relative to the cell centre: |rel| <= h/2 keeps FP32 exact to
  // ~1e-7 of h whatever the box size
  const double rx = p.x - (g.lo[0] + (cx + 0.5) * g.h[0]);
  const double ry = p.y - (g.lo[1] + (cy + 0.5) * g.h[1]);
  const double rz = p.z - (g.lo[2] + (cz + 0.5) * g.h[2]);
  pos32[s] = make_float4((float)rx, (float)ry, (float)rz, __int_as_float(cid));
}

__global__ void k_gather_sorted(int64_t n, Grid g, const int32_t *__restrict__ order,
                                const int32_t *__restrict__ cell_of,
                                const double4_32a *__restrict__ wrapped,
                                int32_t *__restrict__ rank, double4_32a *__restrict__ pos64,
                                float4 *__restrict__ pos32) {
  wait_prior_grid();
  const int64_t s = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (s >= n) return;
  rank[order[s]] = (int32_t)s;
  gather_one(s, g, order, cell_of, wrapped, pos64, pos32);
}

// neighbour cell of cell coordinate (cx,cy,cz) shifted by o; -1 if outside a
// non-periodic axis
__device__ __forceinline__ int32_t shifted_cell(const Grid &g, int cx, int cy, int cz, int4 o) {
  int c[3] = {cx + o.x, cy + o.y, cz + o.z};
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    if (c[d] < 0 || c[d] >= g.nc[d]) {
      if (!g.periodic[d]) return -1;
      c[d] = wrap_index(c[d], g.nc[d]);
    }
  }
  return c[0] + g.nc[0] * (c[1] + g.nc[1] * c[2]);
}

// exact FP64 cut-off decision, the oracle's predicate: minimum-image vector
// (pm_periodic_boundary.C:350-374) and (dx*dx + dy*dy) + dz*dz < rc^2
// without contraction
__device__ __forceinline__ bool exact_within(const Grid &g, double4_32a a, double4_32a b, double rc2) {
  double d[3] = {b.x - a.x, b.y - a.y, b.z - a.z};
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    if (g.periodic[k]) {
      const double xs = g.L[k];
      if (d[k] <= -xs / 2.0) d[k] += xs;
      if (d[k] > xs / 2.0) d[k] -= xs;
    }
  }
  const double r2 = __dadd_rn(__dadd_rn(__dmul_rn(d[0], d[0]), __dmul_rn(d[1], d[1])),
                              __dmul_rn(d[2], d[2]));
  return r2 < rc2;
}

// Warp-per-cell pair list, one pass into fixed-width rows.  The candidates
// of a target cell are the concatenation of its stencil cells (stencil
// order, slot order inside a cell).  For each chunk of up to 32 targets the
// lanes, one stencil cell each, write the candidates' entries to shared
// memory in that order; 64 of them at a time are then loaded, and those
// within reach of the chunk's bounding box queue in shared memory, still in
// order.  A full queue is tested against the chunk's targets, four at a time
// (list_targets); a ballot prefix places each accepted candidate.  Entries
// therefore come out in exactly the per-target order of a sequential sweep.
// Row s holds entries [s*W, s*W + cnt[s]); a row longer than W is counted
// but not stored: the kernel records the longest row and sets
// kErrListCapacity, and the host rebuilds with a wider W.
//
// The instruction issue bounds it (58 M warp instructions at N = 200k, phi =
// 0.1, 78% of the issue slots, DRAM 1%), so the work is in instructions per
// test.  One target at a time with its count in a lane took 83.5 M and 92 us;
// four targets' coordinates, row pointers and counts held in registers over
// a whole queue, two targets per packed instruction, 82 us; the stencil
// lanes writing the entries, instead of a marked scan that looks up each
// candidate's cell, 73 us; two loads in flight per lane 68 us; the box by
// warp-wide reductions 67 us (N = 400k: 167 -> 121 us).  Eight targets at a
// time spilled (75 us), a queue of 128 went over the targets too often (86 us
// where 256 took 82), three or four loads in flight 69 us.
// One warp per block, one block per cell: cells hold different numbers of
// targets, and a block of several cell-warps holds its resources until its
// longest cell is done; with the cell no longer block-uniform its row
// addresses also leave the uniform registers (two warps per block: 90 us).
// Resident blocks that stride over the cells balance worse (91 to 102 us
// where the former kernel took 92).
constexpr int kMaxStencil = 128;  // stencil cells per target cell
constexpr int kListIndex = 256;   // candidates per round: their entries in order
constexpr int kListLoads = 2;     // candidates in flight per lane
constexpr int kListQueue = 160 + 32 * kListLoads;  // kept candidates: tested once past 160

// FP32 distance of a candidate from the targets' box, formed like the pair
// test's r2 below (the same subtractions, squares and fused adds, each
// monotone in its operands), so that it never exceeds the r2 of any target
// inside the box: a candidate whose box distance is above rc2_hi is above it
// for every target and would be rejected there without the exact test
__device__ __forceinline__ float box_r2(float qx, float qy, float qz, float3 lo, float3 hi) {
  const float bx = qx > hi.x ? qx - hi.x : (qx < lo.x ? lo.x - qx : 0.f);
  const float by = qy > hi.y ? qy - hi.y : (qy < lo.y ? lo.y - qy : 0.f);
  const float bz = qz > hi.z ? qz - hi.z : (qz < lo.z ? lo.z - qz : 0.f);
  return fmaf(bz, bz, fmaf(by, by, bx * bx));
}

// a warp's minimum and maximum (NaN ignored, as fminf and fmaxf do)
__device__ __forceinline__ float warp_min(float x) {
  float r;
  asm volatile("redux.sync.min.f32 %0, %1, 0xffffffff;" : "=f"(r) : "f"(x));
  return r;
}
__device__ __forceinline__ float warp_max(float x) {
  float r;
  asm volatile("redux.sync.max.f32 %0, %1, 0xffffffff;" : "=f"(r) : "f"(x));
  return r;
}

// A queue of candidates against GT of the chunk's ntc targets, i0 and on (slot
// t0 + i0 and on; past the last target s_pi is far from everything).  The
// targets and their rows stay in registers over all batches of 32, two
// targets per packed instruction (each half rounds as the scalar form does).
template <int GT, bool HALF>
__device__ __forceinline__ void list_targets(int i0, int ntc, int32_t t0, int queued, bool last,
                                             const float4 *s_q, const float4 *s_pi, const Grid &g,
                                             const double4_32a *__restrict__ pos64, float rc2_lo,
                                             float rc2_hi, double rc2, int W,
                                             uint32_t *__restrict__ list,
                                             uint32_t *__restrict__ list_h, int32_t &own_cnt,
                                             int32_t &own_cnt_h) {
  const int lane = threadIdx.x & 31;
  const unsigned lt_mask = (1u << lane) - 1u;
  float2 px[GT / 2], py[GT / 2], pz[GT / 2];
  int32_t at[GT], at_h[GT];
  uint32_t *row[GT];
#pragma unroll
  for (int q = 0; q < GT; q += 2) {
    const float4 a = s_pi[i0 + q], b = s_pi[i0 + q + 1];
    px[q / 2] = make_float2(-a.x, -b.x);
    py[q / 2] = make_float2(-a.y, -b.y);
    pz[q / 2] = make_float2(-a.z, -b.z);
  }
#pragma unroll
  for (int q = 0; q < GT; ++q) {
    at[q] = __shfl_sync(0xffffffffu, own_cnt, i0 + q);
    at_h[q] = HALF ? __shfl_sync(0xffffffffu, own_cnt_h, i0 + q) : 0;
    row[q] = list + (int64_t)(t0 + i0 + q) * W;
  }
  // a partial batch only after the last candidates
  const int stop = last ? queued : queued & ~31;
  for (int b = 0; b < stop; b += 32) {
    // lanes past the queue carry a far point: r2 overflows, never accepted
    const float4 c = b + lane < queued ? s_q[b + lane] : make_float4(1e30f, 1e30f, 1e30f, 0.f);
    const uint32_t en = __float_as_uint(c.w);
    const int32_t tj = (int32_t)(en >> kCodeBits);
    const float2 cx = make_float2(c.x, c.x), cy = make_float2(c.y, c.y), cz = make_float2(c.z, c.z);
    bool in[GT];
    bool band = false;
#pragma unroll
    for (int q = 0; q < GT; q += 2) {
      const float2 dx = __fadd2_rn(cx, px[q / 2]), dy = __fadd2_rn(cy, py[q / 2]),
                   dz = __fadd2_rn(cz, pz[q / 2]);
      const float2 r2 = __ffma2_rn(dz, dz, __ffma2_rn(dy, dy, __fmul2_rn(dx, dx)));
      // accepted below rc2_lo, rejected above rc2_hi; in between (FP32
      // rounding of |r| = rc) the exact FP64 test decides, behind a
      // warp-uniform branch so that the common case carries none of it
      in[q] = tj != t0 + i0 + q && !(r2.x > rc2_hi);
      in[q + 1] = tj != t0 + i0 + q + 1 && !(r2.y > rc2_hi);
      band |= in[q] && !(r2.x < rc2_lo);
      band |= in[q + 1] && !(r2.y < rc2_lo);
    }
    if (__any_sync(0xffffffffu, band)) {
#pragma unroll
      for (int q = 0; q < GT; ++q) {
        const float4 pi = s_pi[i0 + q];
        const float dx = c.x - pi.x, dy = c.y - pi.y, dz = c.z - pi.z;
        const float r2 = fmaf(dz, dz, fmaf(dy, dy, dx * dx));
        if (in[q] && !(r2 < rc2_lo))
          in[q] = i0 + q < ntc && exact_within(g, pos64[t0 + i0 + q], pos64[tj], rc2);
      }
    }
#pragma unroll
    for (int q = 0; q < GT; ++q) {
      const unsigned bal = __ballot_sync(0xffffffffu, in[q]);
      const int32_t k = at[q] + __popc(bal & lt_mask);
      if (in[q] && k < W) row[q][k] = en;
      at[q] += __popc(bal);
      if (HALF) {
        // the half list: each unordered pair once, in the row of its
        // smaller slot (the full list is symmetric, its predicate exact)
        const bool in_h = in[q] && tj > t0 + i0 + q;
        const unsigned bal_h = __ballot_sync(0xffffffffu, in_h);
        const int32_t kh = at_h[q] + __popc(bal_h & lt_mask);
        if (in_h && kh < W) list_h[(int64_t)(t0 + i0 + q) * W + kh] = en;
        at_h[q] += __popc(bal_h);
      }
    }
  }
#pragma unroll
  for (int q = 0; q < GT; ++q) {
    if (lane == i0 + q) {
      own_cnt = at[q];
      if (HALF) own_cnt_h = at_h[q];
    }
  }
}

template <bool HALF>
__device__ __forceinline__ void pair_list_cell(
    int C, const Grid &g, const int4 *__restrict__ stencil, int nst,
    const float4 *__restrict__ shift, const int32_t *__restrict__ start, const float4 *__restrict__ pos32,
    const double4_32a *__restrict__ pos64, float rc2_lo, float rc2_hi, double rc2, int W,
    int32_t *__restrict__ count, uint32_t *__restrict__ list,
    unsigned long long *__restrict__ stat, int *__restrict__ err,
    int32_t *__restrict__ count_h, uint32_t *__restrict__ list_h) {
  __shared__ float4 s_pi[32];             // the targets of the current chunk
  __shared__ float4 s_q[kListQueue];      // kept candidates: frame position, entry
  __shared__ uint32_t s_idx[kListIndex];  // entries of the current round's candidates
  const int lane = threadIdx.x;
  const int32_t tb = start[C], te = start[C + 1];
  if (te <= tb) return;
  const int cx = C % g.nc[0], cy = (C / g.nc[0]) % g.nc[1], cz = C / (g.nc[0] * g.nc[1]);
  const unsigned lt_mask = (1u << lane) - 1u;
  unsigned long long cell_total = 0;
  int32_t cell_max = 0;
  for (int32_t t0 = tb; t0 < te; t0 += 32) {
    const int ntc = min(32, te - t0);
    const int32_t own = t0 + lane;
    const bool own_ok = lane < ntc;
    __syncwarp();  // the previous chunk's targets are no longer read
    // slots past the chunk's targets are as far from every candidate as the
    // padding candidates are on the other side: r2 overflows
    const float4 mine = own_ok ? pos32[own] : make_float4(-1e30f, -1e30f, -1e30f, 0.f);
    s_pi[lane] = mine;
    // the chunk's bounding box (FP32 min / max of the targets' own values)
    float3 blo = own_ok ? make_float3(mine.x, mine.y, mine.z)
                        : make_float3(INFINITY, INFINITY, INFINITY);
    float3 bhi = own_ok ? make_float3(mine.x, mine.y, mine.z)
                        : make_float3(-INFINITY, -INFINITY, -INFINITY);
    blo = make_float3(warp_min(blo.x), warp_min(blo.y), warp_min(blo.z));
    bhi = make_float3(warp_max(bhi.x), warp_max(bhi.y), warp_max(bhi.z));
    __syncwarp();
    int32_t own_cnt = 0, own_cnt_h = 0;
    int queued = 0;  // warp-uniform
    for (int k0 = 0; k0 < nst; k0 += 32) {
      // one stencil cell per lane: its slots and where they go in the order
      const int k = k0 + lane;
      int32_t cnt = 0, base = 0;
      uint32_t code = 0;
      if (k < nst) {
        const int4 o = stencil[k];
        const int32_t nc = shifted_cell(g, cx, cy, cz, o);
        code = (uint32_t)o.w;
        if (nc >= 0) {
          base = start[nc];
          cnt = start[nc + 1] - base;
        }
      }
      int32_t incl = cnt;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int32_t y = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += y;
      }
      const int32_t V = __shfl_sync(0xffffffffu, incl, 31);
      const int32_t first = incl - cnt;
      for (int32_t r0 = 0; r0 == 0 || r0 < V; r0 += kListIndex) {
        const int32_t Vr = min(V - r0, kListIndex);
        __syncwarp();  // the previous round's candidates are read
        for (int32_t v = max(first, r0); v < min(incl, r0 + kListIndex); ++v)
          s_idx[v - r0] = ((uint32_t)(base + v - first) << kCodeBits) | code;
        __syncwarp();
        for (int32_t v0 = 0; v0 == 0 || v0 < Vr; v0 += 32 * kListLoads) {
          uint32_t en[kListLoads];
          float4 sh[kListLoads], pj[kListLoads];
#pragma unroll
          for (int h = 0; h < kListLoads; ++h) {
            const int32_t v = v0 + 32 * h + lane;
            en[h] = v < Vr ? s_idx[v] : 0u;
            sh[h] = shift[en[h] & ((1u << kCodeBits) - 1u)];
            pj[h] = v < Vr ? pos32[en[h] >> kCodeBits] : make_float4(0.f, 0.f, 0.f, 0.f);
          }
#pragma unroll
          for (int h = 0; h < kListLoads; ++h) {
            // the candidate in the target cell's frame (the shift added once
            // per candidate; the filter's band absorbs the different rounding)
            const float qx = pj[h].x + sh[h].x, qy = pj[h].y + sh[h].y, qz = pj[h].z + sh[h].z;
            const bool keep =
                v0 + 32 * h + lane < Vr && !(box_r2(qx, qy, qz, blo, bhi) > rc2_hi);
            const unsigned kb = __ballot_sync(0xffffffffu, keep);
            if (keep)
              s_q[queued + __popc(kb & lt_mask)] = make_float4(qx, qy, qz, __uint_as_float(en[h]));
            queued += __popc(kb);
          }
          const bool last =
              k0 + 32 >= nst && r0 + kListIndex >= V && v0 + 32 * kListLoads >= Vr;
          if (queued <= kListQueue - 32 * kListLoads && !last) continue;
          // the queue against every target: whole batches, the rest moves to
          // its front, or all of it after the last candidates
          __syncwarp();
          for (int i = 0; i < ntc;) {
            if (ntc - i > 2) {
              list_targets<4, HALF>(i, ntc, t0, queued, last, s_q, s_pi, g, pos64, rc2_lo, rc2_hi,
                                    rc2, W, list, list_h, own_cnt, own_cnt_h);
              i += 4;
            } else {
              list_targets<2, HALF>(i, ntc, t0, queued, last, s_q, s_pi, g, pos64, rc2_lo, rc2_hi,
                                    rc2, W, list, list_h, own_cnt, own_cnt_h);
              i += 2;
            }
          }
          const int done = queued & ~31;
          queued -= done;
          const float4 r = lane < queued ? s_q[done + lane] : make_float4(0.f, 0.f, 0.f, 0.f);
          __syncwarp();
          if (lane < queued) s_q[lane] = r;
        }
      }
    }
    if (own_ok) {
      if (HALF) count_h[own] = min(own_cnt_h, W);
      count[own] = min(own_cnt, W);  // the stored entries; the full length goes to stat
    }
    cell_total += __reduce_add_sync(0xffffffffu, (unsigned)own_cnt);
    cell_max = max(cell_max, __reduce_max_sync(0xffffffffu, own_cnt));
  }
  // one pair of atomics per cell for the list statistics
  if (lane == 0) {
    atomicAdd(&stat[0], cell_total);
    atomicMax(&stat[1], (unsigned long long)cell_max);
    if (cell_max > W) atomicOr(err, kErrListCapacity);
  }
}

// One block per cell, or (SLOT) per slot, of which those with the first slot
// of their cell take it: where cells outnumber the particles, the blocks of
// empty ones are the cost (FP64 matvec with its list, N = 2000 in 1e6 cells:
// 589 -> 87 us).
template <bool HALF, bool SLOT>
__global__ void __launch_bounds__(32, 32) k_pair_list_warp(
    Grid g, const int4 *__restrict__ stencil, int nst, const float4 *__restrict__ shift,
    const int32_t *__restrict__ start, const float4 *__restrict__ pos32,
    const double4_32a *__restrict__ pos64, float rc2_lo, float rc2_hi, double rc2, int W,
    int32_t *__restrict__ count, uint32_t *__restrict__ list,
    unsigned long long *__restrict__ stat, int *__restrict__ err,
    int32_t *__restrict__ count_h, uint32_t *__restrict__ list_h) {
  wait_prior_grid();
  int C = (int)blockIdx.x;
  if (SLOT) {
    C = __float_as_int(pos32[blockIdx.x].w);
    if (start[C] != (int32_t)blockIdx.x) return;
  }
  pair_list_cell<HALF>(C, g, stencil, nst, shift, start, pos32, pos64, rc2_lo, rc2_hi, rc2, W,
                       count, list, stat, err, count_h, list_h);
}

// ---- many suspensions at once ----------------------------------------------
// The same build over the concatenated cells and slots of K suspensions
// (BatchGeo: each one's grid, stencil and first cell and slot), so that an
// ensemble's configuration takes one launch per phase instead of one per
// phase and suspension: the launches and host waits of 64 separate builds
// were ~7 ms, their kernels a few microseconds each.
__global__ void k_batch_susp(int64_t ntot, int K, const int64_t *__restrict__ off,
                             int32_t *__restrict__ susp) {
  const int64_t s = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (s >= ntot) return;
  int lo = 0, hi = K - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (off[mid] <= s) lo = mid;
    else hi = mid - 1;
  }
  susp[s] = lo;
}

__global__ void k_batch_assign(int64_t ntot, const double *__restrict__ xyz,
                               const BatchGeo *__restrict__ geo, const int32_t *__restrict__ susp,
                               int32_t *__restrict__ cell_of, int32_t *__restrict__ count,
                               double4_32a *__restrict__ wrapped, int *__restrict__ err) {
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i >= ntot) return;
  const BatchGeo &b = geo[susp[i]];
  assign_one(i, xyz, b.g, cell_of, count + b.cell0, wrapped, err);
}

// one block per suspension: its cells' counts (zeroed as they are read)
// scanned from its first slot on
__global__ void __launch_bounds__(1024) k_batch_scan(int K, const BatchGeo *__restrict__ geo,
                                                     const int64_t *__restrict__ off,
                                                     int32_t *__restrict__ count,
                                                     int32_t *__restrict__ start,
                                                     unsigned long long *__restrict__ stat) {
  __shared__ int32_t warp_tot[2][32];
  const int b = blockIdx.x;
  if (b == 0 && threadIdx.x < 2) stat[threadIdx.x] = 0ull;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int64_t c0 = geo[b].cell0, n = geo[b].g.ncell;
  int32_t carry = (int32_t)off[b];
  int buf = 0;
  for (int64_t t0 = 0; t0 < n; t0 += 4096, buf ^= 1) {
    int32_t v[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int64_t i = t0 + 4 * threadIdx.x + j;
      v[j] = i < n ? count[c0 + i] : 0;
      if (i < n) count[c0 + i] = 0;
    }
    const int32_t tsum = (v[0] + v[1]) + (v[2] + v[3]);
    int32_t x = tsum;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int32_t y = __shfl_up_sync(0xffffffffu, x, o);
      if (lane >= o) x += y;
    }
    int32_t *wt = warp_tot[buf];  // alternate buffers: one barrier per tile
    if (lane == 31) wt[warp] = x;
    __syncthreads();
    int32_t w = wt[lane];
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int32_t y = __shfl_up_sync(0xffffffffu, w, o);
      if (lane >= o) w += y;
    }
    const int32_t before = __shfl_sync(0xffffffffu, w, (warp + 31) & 31);
    const int32_t total = __shfl_sync(0xffffffffu, w, 31);
    int32_t run = carry + (warp ? before : 0) + x - tsum;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int64_t i = t0 + 4 * threadIdx.x + j;
      if (i < n) start[c0 + i] = run;
      run += v[j];
    }
    carry += total;
  }
  if (b == K - 1 && threadIdx.x == 0) start[c0 + n] = carry;
}

__global__ void k_batch_scatter(int64_t ntot, const BatchGeo *__restrict__ geo,
                                const int32_t *__restrict__ susp,
                                const int32_t *__restrict__ cell_of,
                                const int32_t *__restrict__ start, int32_t *__restrict__ fill,
                                int32_t *__restrict__ order) {
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i >= ntot) return;
  const int64_t cid = geo[susp[i]].cell0 + cell_of[i];
  order[start[cid] + atomicAdd(&fill[cid], 1)] = (int32_t)i;
}

__global__ void k_batch_gather(int64_t ntot, const BatchGeo *__restrict__ geo,
                               const int32_t *__restrict__ susp,
                               const int32_t *__restrict__ order,
                               const int32_t *__restrict__ cell_of,
                               const double4_32a *__restrict__ wrapped,
                               double4_32a *__restrict__ pos64, float4 *__restrict__ pos32) {
  const int64_t s = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (s >= ntot) return;
  gather_one(s, geo[susp[s]].g, order, cell_of, wrapped, pos64, pos32);
}

__global__ void __launch_bounds__(32, 32) k_batch_list(
    const BatchGeo *__restrict__ geo, const int32_t *__restrict__ cell_susp,
    const int32_t *__restrict__ start, const float4 *__restrict__ pos32,
    const double4_32a *__restrict__ pos64, float rc2_lo, float rc2_hi, double rc2, int W,
    int32_t *__restrict__ count, uint32_t *__restrict__ list,
    unsigned long long *__restrict__ stat, int *__restrict__ err) {
  const BatchGeo &b = geo[cell_susp[blockIdx.x]];
  pair_list_cell<false>((int)((int64_t)blockIdx.x - b.cell0), b.g, b.stencil, b.nst, b.shift, start + b.cell0,
                 pos32, pos64, rc2_lo, rc2_hi, rc2, W, count, list, stat, err, nullptr, nullptr);
}

// Element lists (reference mode) as pair-list rows: one warp per target slot,
// one lane per run of stencil elements along x.  The particles of a run are
// one or (across a periodic face) two ranges of consecutive slots, every one
// of them a neighbour (the list has no distance test), so a lane's count is
// two subtractions, a warp scan places the runs and each lane writes its own.
// ~110 runs instead of ~1000 elements per target at the h <= 1.414 mesh rule,
// and once per configuration instead of once per operator application.
constexpr int kRunWarps = 8;

__global__ void __launch_bounds__(32 * kRunWarps) k_run_list(
    int64_t n, Grid g, const int4 *__restrict__ runs, int nruns,
    const int32_t *__restrict__ start, const float4 *__restrict__ pos32, int W,
    int32_t *__restrict__ count, uint32_t *__restrict__ list,
    unsigned long long *__restrict__ stat, int *__restrict__ err) {
  wait_prior_grid();
  __shared__ int s_tot[kRunWarps];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int64_t s = blockIdx.x * (int64_t)kRunWarps + warp;
  int total = 0;
  if (s < n) {
    const int32_t cid = __float_as_int(pos32[s].w);
    const int cx = cid % g.nc[0], cy = (cid / g.nc[0]) % g.nc[1], cz = cid / (g.nc[0] * g.nc[1]);
    uint32_t *row = list + s * (int64_t)W;
    for (int r0 = 0; r0 < nruns; r0 += 32) {
      const int r = r0 + lane;
      int32_t b0 = 0, e0 = 0, b1 = 0, e1 = 0;
      bool own = false;
      if (r < nruns) {
        const int4 o = runs[r];
        own = o.x == 0 && o.y == 0;
        int y = cy + o.x, z = cz + o.y;
        bool ok = true;
        if (y < 0 || y >= g.nc[1]) {
          if (g.periodic[1]) y += y < 0 ? g.nc[1] : -g.nc[1];
          else ok = false;
        }
        if (z < 0 || z >= g.nc[2]) {
          if (g.periodic[2]) z += z < 0 ? g.nc[2] : -g.nc[2];
          else ok = false;
        }
        if (ok) {
          const int nx = g.nc[0];
          const int32_t *st = start + (int64_t)nx * (y + (int64_t)g.nc[1] * z);
          int a = cx + o.z, b = cx + o.w;
          if (!g.periodic[0]) {
            a = max(a, 0);
            b = min(b, nx - 1);
            if (a <= b) {
              b0 = st[a];
              e0 = st[b + 1];
            }
          } else {
            // offsets lie in (-nx, nx) and a run has at most nx elements
            if (b < 0) a += nx, b += nx;
            else if (a >= nx) a -= nx, b -= nx;
            const int lo = max(a, 0), hi = min(b, nx - 1);
            b0 = st[lo];
            e0 = st[hi + 1];
            if (a < 0) {
              b1 = st[a + nx];
              e1 = st[nx];
            } else if (b >= nx) {
              b1 = st[0];
              e1 = st[b - nx + 1];
            }
          }
        }
      }
      // the own run holds the target itself, which is no neighbour
      const int cnt = (e0 - b0) + (e1 - b1) - (own ? 1 : 0);
      int incl = cnt;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += y;
      }
      int at = total + incl - cnt;
      for (int32_t t = b0; t < e0; ++t)
        if (t != s) {
          if (at < W) row[at] = (uint32_t)t << kCodeBits;
          ++at;
        }
      for (int32_t t = b1; t < e1; ++t)
        if (t != s) {
          if (at < W) row[at] = (uint32_t)t << kCodeBits;
          ++at;
        }
      total += __shfl_sync(0xffffffffu, incl, 31);
    }
    if (lane == 0) count[s] = min(total, W);  // the full length goes to stat
  }
  if (lane == 0) s_tot[warp] = total;
  __syncthreads();
  if (threadIdx.x == 0) {
    unsigned long long sum = 0;
    int longest = 0;
    for (int w = 0; w < kRunWarps; ++w) {
      sum += (unsigned long long)s_tot[w];
      longest = max(longest, s_tot[w]);
    }
    atomicAdd(&stat[0], sum);
    atomicMax(&stat[1], (unsigned long long)longest);
    if (longest > W) atomicOr(err, kErrListCapacity);
  }
}

}  // namespace

int device_exclusive_scan_i32(ggem_ctx *c, const int32_t *in, int32_t *out, int64_t n) {
  return scan_impl<int32_t>(c, in, out, n, 0);
}
int device_exclusive_scan_i64(ggem_ctx *c, const int64_t *in, int64_t *out, int64_t n) {
  return scan_impl<int64_t>(c, in, out, n, 0);
}

int build_cells(ggem_ctx *c, bool defer_flags) {
  const int64_t n = c->n;
  const Grid &g = c->grid;
  cudaError_t e = cudaSuccess;
  if ((e = c->cell_of.ensure(n)) || (e = c->cell_count.ensure(g.ncell)) ||
      (e = c->cell_fill.ensure(g.ncell)) || (e = c->cell_start.ensure(g.ncell + 1)) ||
      (e = c->order.ensure(n)) || (e = c->rank.ensure(n)) || (e = c->wrapped.ensure(n)) ||
      (e = c->pos64.ensure(n)) || (e = c->pos32.ensure(n)))
    return cuda_fail(c, e, "cell buffers");
  cudaStream_t st = c->stream;
  // the cell counters are left at zero by the previous build (the
  // one-launch scan zeroes the counts, k_sort_cells the fills); they are
  // cleared here only after a reallocation, an interrupted build or on
  // grids too large for the one-launch scan
  const bool small = g.ncell <= kScanCellsMax;
  const bool clean = small && c->cell_counters_zero && c->cell_count.p == c->cell_counters_at;
  c->cell_counters_zero = false;
  if ((!clean && ((e = cudaMemsetAsync(c->cell_count.p, 0, sizeof(int32_t) * g.ncell, st)) ||
                  (e = cudaMemsetAsync(c->cell_fill.p, 0, sizeof(int32_t) * g.ncell, st)))) ||
      (e = cudaMemsetAsync(c->err.p, 0, sizeof(int), st)))
    return cuda_fail(c, e, "cell memset");
  const int T = 256;
  const unsigned bn = (unsigned)((n + T - 1) / T);
  if (n > 0) {
    launch_dependent(k_assign, dim3(bn), T, 0, st,
                   n, c->xyz_in.p, g, c->cell_of.p, c->cell_count.p, c->wrapped.p,
                               c->err.p);
    if (int rc = check_launch(c, "assign")) return rc;
  }
  c->list_stat_zero = false;
  if (small) {
    // blocks: a power of two with a tile each, then more tiles per block
    const int nt = (int)((g.ncell + 4095) / 4096);
    int blocks = 1;
    while (blocks < nt && blocks < kScanCluster) blocks *= 2;
    launch_dependent_cluster(k_scan_cells, dim3(blocks), 1024, 0, st, (unsigned)blocks,
                             c->cell_count.p, c->cell_start.p, g.ncell,
                             (nt + blocks - 1) / blocks, c->nb_stat.p);
    if (int rc = check_launch(c, "scan cells")) return rc;
    c->list_stat_zero = c->nb_stat.p != nullptr;
  } else if (int rc = device_exclusive_scan_i32(c, c->cell_count.p, c->cell_start.p, g.ncell)) {
    return rc;
  }
  if (n > 0) {
    launch_dependent(k_scatter, dim3(bn), T, 0, st,
                   n, c->cell_of.p, c->cell_start.p, c->cell_fill.p, c->order.p);
    if (int rc = check_launch(c, "scatter")) return rc;
  }
  // (for n = 0 only the fill counters are cleared)
  launch_dependent(k_sort_cells, dim3((unsigned)((g.ncell + T - 1) / T)), T, 0, st,
                   g.ncell, c->cell_start.p,
                                                                 c->order.p, c->cell_fill.p);
  if (int rc = check_launch(c, "sort cells")) return rc;
  if (n > 0) {
    launch_dependent(k_gather_sorted, dim3(bn), T, 0, st,
                   n, g, c->order.p, c->cell_of.p, c->wrapped.p, c->rank.p,
                                      c->pos64.p, c->pos32.p);
    if (int rc = check_launch(c, "gather sorted")) return rc;
  }
  c->cell_counters_zero = small;
  c->cell_counters_at = c->cell_count.p;
  c->cells_built = false;
  c->list_built = false;
  c->pretensor_ok = false;
  if (!defer_flags) {
    int flags = 0;
    if (int rc = read_error_flags(c, &flags)) return rc;
    if (int rc = cell_flag_error(c, flags)) return rc;
  }
  c->cells_built = true;
  return GGEM_OK;
}

int cell_flag_error(ggem_ctx *c, int flags) {
  if (flags & kErrNonFinite) {
    c->cells_built = false;
    return fail(c, GGEM_ERR_BAD_ARG, "non-finite position");
  }
  if (flags & kErrOutOfDomain) {
    c->cells_built = false;
    return fail(c, GGEM_ERR_OUT_OF_DOMAIN,
                "a particle lies outside the box on a non-periodic axis "
                "(point_mesh.C:602-613: no element contains it)");
  }
  return GGEM_OK;
}

void launch_pair_list(ggem_ctx *c, int nst, int W, cudaStream_t st) {
  if (c->prm.nb_mode == GGEM_NB_REFERENCE) {
    launch_dependent(k_run_list, dim3((unsigned)((c->n + kRunWarps - 1) / kRunWarps)), 32 * kRunWarps, 0, st,
                   c->n, c->grid, c->d_runs, c->n_runs, c->cell_start.p, c->pos32.p, W, c->nb_cnt.p,
        c->nb_list.p, c->nb_stat.p, c->err.p);
    return;
  }
  const bool slot = c->n < c->grid.ncell;
  launch_dependent(c->sym_pairs ? (slot ? k_pair_list_warp<true, true> : k_pair_list_warp<true, false>)
                                : (slot ? k_pair_list_warp<false, true> : k_pair_list_warp<false, false>),
                   dim3((unsigned)std::min(c->n, c->grid.ncell)), 32, 0, st, c->grid, c->d_stencil.p, nst,
                   c->d_shift.p, c->cell_start.p, c->pos32.p, c->pos64.p, c->rc2_lo, c->rc2_hi, c->rc2,
                   W, c->nb_cnt.p, c->nb_list.p, c->nb_stat.p, c->err.p,
                   c->sym_pairs ? c->nb_cnt_h.p : nullptr, c->sym_pairs ? c->nb_list_h.p : nullptr);
}

int build_pair_list(ggem_ctx *c) {
  const int64_t n = c->n;
  cudaError_t e = cudaSuccess;
  if ((e = c->nb_cnt.ensure(n)) || (e = c->nb_stat.ensure(2)))
    return cuda_fail(c, e, "pair list buffers");
  cudaStream_t st = c->stream;
  if (c->nb_w <= 0) {
    // first build: twice the mean row length of a uniform suspension plus slack
    const Grid &g = c->grid;
    const double vol = g.L[0] * g.L[1] * g.L[2];
    const double r = c->prm.nb_mode == GGEM_NB_REFERENCE ? c->search_radius_e : std::sqrt(c->rc2);
    double mean = vol > 0 ? (double)n / vol * 4.18879020478639 * r * r * r : 0.0;
    if (c->f64_list_is_own()) mean = std::min(mean, 0.5 * n);  // (a pair is listed once)
    c->nb_w = (int)std::min<double>(((int64_t)(2.0 * mean) + 16 + 7) / 8 * 8, 1 << 20);
  }
  if (n == 0) {
    c->n_pairs = 0;
    c->cells_built = true;
    c->list_built = true;
    return GGEM_OK;
  }
  const int nst = (int)c->stencil.size();
  if (nst > kMaxStencil && c->prm.nb_mode != GGEM_NB_REFERENCE)
    return fail(c, GGEM_ERR_BAD_ARG, "stencil too large for the list builder");
  if (c->defer_checks && c->list_checked_once) {
    // keep the width of the previous build; a longer row is stored clipped
    // (counts never exceed W) and found when the statistics are read
    if ((e = c->nb_list.ensure((size_t)n * c->nb_w))) return cuda_fail(c, e, "pair list");
    // (the statistics were zeroed by this configuration's cell scan)
    if (!c->list_stat_zero &&
        (e = cudaMemsetAsync(c->nb_stat.p, 0, 2 * sizeof(unsigned long long), st)))
      return cuda_fail(c, e, "memset");
    c->list_stat_zero = false;
    kt_start(c, kKListBuild);
    if (c->sym_pairs && ((e = c->nb_list_h.ensure((size_t)n * c->nb_w)) ||
                         (e = c->nb_cnt_h.ensure(n))))
      return cuda_fail(c, e, "half pair list");
    launch_pair_list(c, nst, c->nb_w, st);
    kt_stop(c, kKListBuild);
    if (int rc = check_launch(c, "pair list")) return rc;
    c->cells_built = true;
    c->list_built = true;
    c->list_unchecked = true;
    c->n_pairs = -1;
    return GGEM_OK;
  }
  // The error word still holds the cell build's flags; they come back with
  // the list statistics in one host synchronisation.  A row longer than the
  // current width makes the host widen the rows and fill once more.
  unsigned long long *h = reinterpret_cast<unsigned long long *>(c->h_red);
  c->list_stat_zero = false;
  for (int attempt = 0; attempt < 2; ++attempt) {
    const int W = c->nb_w;
    // a list that only saves time leaves most of the memory to the caller
    if (c->f64_list_is_own() && (size_t)n * W > c->nb_list.count) {
      size_t avail = 0, all = 0;
      if ((e = cudaMemGetInfo(&avail, &all))) return cuda_fail(c, e, "pair list");
      if ((size_t)n * W * sizeof(uint32_t) > avail / 4)
        return fail(c, GGEM_ERR_OOM, "pair list larger than a quarter of the free memory");
    }
    if ((e = c->nb_list.ensure((size_t)n * W))) return cuda_fail(c, e, "pair list");
    if ((e = cudaMemsetAsync(c->nb_stat.p, 0, 2 * sizeof(unsigned long long), st)))
      return cuda_fail(c, e, "memset");
    if (c->sym_pairs && ((e = c->nb_list_h.ensure((size_t)n * W)) || (e = c->nb_cnt_h.ensure(n))))
      return cuda_fail(c, e, "half pair list");
    if (attempt == 0) kt_start(c, kKListBuild);
    launch_pair_list(c, nst, W, st);
    if (attempt == 0) kt_stop(c, kKListBuild);  // a widened refill is left out
    if (int rc = check_launch(c, "pair list")) return rc;
    h[2] = 0;
    if ((e = cudaMemcpyAsync(h, c->nb_stat.p, 2 * sizeof(unsigned long long),
                             cudaMemcpyDeviceToHost, st)) ||
        (e = cudaMemcpyAsync(&h[2], c->err.p, sizeof(int), cudaMemcpyDeviceToHost, st)) ||
        (e = cudaStreamSynchronize(st)))
      return cuda_fail(c, e, "list statistics");
    const int flags = (int)h[2];
    if (int rc = cell_flag_error(c, flags)) return rc;
    c->cells_built = true;
    if (!(flags & kErrListCapacity)) {
      c->n_pairs = (int64_t)h[0];
      c->list_built = true;
      c->list_checked_once = true;
      return GGEM_OK;
    }
    const unsigned long long longest = h[1];
    c->nb_w = (int)std::min<unsigned long long>((longest + longest / 8 + 8 + 7) / 8 * 8, 1u << 24);
    if ((e = cudaMemsetAsync(c->err.p, 0, sizeof(int), st))) return cuda_fail(c, e, "memset");
  }
  return fail(c, GGEM_ERR_CELL_OVERFLOW, "pair list rows exceeded their width twice");
}

bool stream_capturing(const ggem_ctx *c) {
  cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
  if (cudaStreamIsCapturing(c->stream, &cap) != cudaSuccess) {
    cudaGetLastError();
    return true;
  }
  return cap != cudaStreamCaptureStatusNone;
}

// Does an FP64 context in the default mode use a list?  On very dilute grids
// the sweep of a few empty cells costs less than a list that holds almost no
// pairs (us for cells, list and one product against cells and sweep: N =
// 200k, 6.3e6 cells 451 / 412, 25e6 694 / 504, 1.6e6 413 / 601; N = 20k,
// 10e6 cells 211 / 195, 0.6e6 125 / 130).
bool f64_list_fits(const ggem_ctx *c) {
  const int64_t m = c->grid.ncell;
  return c->f64_list_exact &&
         (c->prm.nb_mode == GGEM_NB_REFERENCE || m <= 1 << 21 || m <= 8 * c->n);
}

int ensure_f64_list(ggem_ctx *c, bool flags_pending) {
  // (a product asks: the next configuration's list comes with its cells)
  if (!flags_pending) c->f64_wanted = true;
  if (c->prm.precision != GGEM_FP64 || c->f64_list >= 0 || c->list_built || c->f64_skip ||
      !f64_list_fits(c) || c->n == 0)
    return GGEM_OK;
  cudaError_t e;
  if (!flags_pending) {
    // a list build waits for the device, which a capture cannot
    if (stream_capturing(c)) return GGEM_OK;
    // (the error word may hold bits of a point sum that have been reported)
    if ((e = cudaMemsetAsync(c->err.p, 0, sizeof(int), c->stream)))
      return cuda_fail(c, e, "memset");
  }
  const bool defer = c->defer_checks;
  c->defer_checks = false;
  const int rc = build_pair_list(c);
  c->defer_checks = defer;
  if (rc != GGEM_ERR_OOM && rc != GGEM_ERR_CELL_OVERFLOW) return rc;
  // no room for this configuration's list: sweep its cells
  c->f64_skip = true;
  c->list_built = false;
  c->nb_w = 0;
  if (flags_pending) {
    int flags = 0;
    if (int frc = read_error_flags(c, &flags)) return frc;
    if (int frc = cell_flag_error(c, flags)) return frc;
  }
  c->cells_built = true;
  return GGEM_OK;
}

void batch_susp(const BatchBuild &b, const int64_t *off, int32_t *susp, cudaStream_t st) {
  k_batch_susp<<<(unsigned)((b.ntot + 255) / 256), 256, 0, st>>>(b.ntot, b.K, off, susp);
}

void batch_cells(const BatchBuild &b, const double *xyz, const int64_t *off, cudaStream_t st) {
  const unsigned bn = (unsigned)((b.ntot + 255) / 256);
  k_batch_assign<<<bn, 256, 0, st>>>(b.ntot, xyz, b.geo, b.susp, b.cell_of, b.cell_count,
                                     b.wrapped, b.err);
  k_batch_scan<<<b.K, 1024, 0, st>>>(b.K, b.geo, off, b.cell_count, b.cell_start, b.stat);
  k_batch_scatter<<<bn, 256, 0, st>>>(b.ntot, b.geo, b.susp, b.cell_of, b.cell_start, b.cell_fill,
                                      b.order);
  k_sort_cells<<<(unsigned)((b.ncell + 255) / 256), 256, 0, st>>>(b.ncell, b.cell_start, b.order,
                                                                   b.cell_fill);
  k_batch_gather<<<bn, 256, 0, st>>>(b.ntot, b.geo, b.susp, b.order, b.cell_of, b.wrapped,
                                     b.pos64, b.pos32);
}

void batch_list(const BatchBuild &b, const ggem_ctx *like, cudaStream_t st) {
  k_batch_list<<<(unsigned)b.ncell, 32, 0, st>>>(b.geo, b.cell_susp, b.cell_start, b.pos32, b.pos64,
                                                 like->rc2_lo, like->rc2_hi, like->rc2, b.W, b.cnt,
                                                 b.list, b.stat, b.err);
}

int enqueue_list_check(ggem_ctx *c) {
  if (!c->list_unchecked) return GGEM_OK;
  unsigned long long *h = reinterpret_cast<unsigned long long *>(c->h_red + kListStatSlot);
  h[2] = 0;
  cudaError_t e = cudaMemcpyAsync(h, c->nb_stat.p, 2 * sizeof(unsigned long long),
                                  cudaMemcpyDeviceToHost, c->stream);
  if (e == cudaSuccess)
    e = cudaMemcpyAsync(&h[2], c->err.p, sizeof(int), cudaMemcpyDeviceToHost, c->stream);
  if (e) return cuda_fail(c, e, "list statistics");
  return GGEM_OK;
}

int finish_list_check(ggem_ctx *c, unsigned long long total, unsigned long long longest, int flags,
                      bool *rebuilt) {
  if (rebuilt) *rebuilt = false;
  if (!c->list_unchecked) return GGEM_OK;
  c->list_unchecked = false;
  if (int rc = cell_flag_error(c, flags)) {
    c->list_built = false;
    return rc;
  }
  if (!(flags & kErrListCapacity)) {
    c->n_pairs = (int64_t)total;
    return GGEM_OK;
  }
  // rows overflowed: widen them and rebuild with the synchronous path
  c->nb_w = (int)std::min<unsigned long long>((longest + longest / 8 + 8 + 7) / 8 * 8, 1u << 24);
  cudaError_t e = cudaMemsetAsync(c->err.p, 0, sizeof(int), c->stream);
  if (e) return cuda_fail(c, e, "memset");
  const bool defer = c->defer_checks;
  c->defer_checks = false;
  int rc = build_pair_list(c);
  c->defer_checks = defer;
  if (rc) return rc;
  if ((rc = build_pair_tensors(c))) return rc;
  if (rebuilt) *rebuilt = true;
  return GGEM_OK;
}

int settle_list(ggem_ctx *c) {
  if (!c->list_unchecked) return GGEM_OK;
  if (int rc = enqueue_list_check(c)) return rc;
  cudaError_t e = cudaStreamSynchronize(c->stream);
  if (e) return cuda_fail(c, e, "list statistics");
  const unsigned long long *h = reinterpret_cast<unsigned long long *>(c->h_red + kListStatSlot);
  return finish_list_check(c, h[0], h[1], (int)h[2], nullptr);
}

}  // namespace ggem

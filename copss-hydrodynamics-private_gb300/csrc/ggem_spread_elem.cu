// ggem_spread_elem.cu -- the Gaussian force spreading onto the quadrature
// points of every element of the mesh, brick by brick.
//
// rho(q) = sum_j g_alpha(q - x_j) f_j with
// g_alpha(r) = alpha^3 pi^{-3/2} e^{-alpha^2 r^2} (2.5 - alpha^2 r^2)
// (GGEMStokes::smoothed_force_exp, ggem_stokes.C:117-128), summed for each
// quadrature point of element e over the particles of e's element
// neighbour list (AssembleStokes::compute_element_rhs,
// assemble_stokes.C:645-662; the list of point_mesh.C:652-799: the
// particles of every element whose centroid lies within search_radius_e of
// e's centroid, e itself included).
//
// Reference mode only: elements are the cells of the context's grid and a
// particle belongs to e's list exactly when the offset between its element
// and e lies in the element stencil (the host's centroid test), so the
// list test is integer arithmetic on element coordinates.
//
// One CTA takes a brick of B x B x B elements.  It stages every particle of
// the brick's stencil-dilated region (contiguous slot ranges, one per row of
// elements along x) into shared memory once; each warp then takes one
// element at a time: its lanes test the staged particles' element offsets
// against the stencil bitmap and compact the members into a per-warp list,
// then 32 / nq lanes per quadrature point sum g f over the members.  The
// gathers of a particle are shared by the brick's 64 elements instead of
// being repeated per element, and the ~1000 stencil elements of each
// element (most of them empty) are never visited one by one.
//
// Two arithmetic paths over the same lists:
//  * FP64: the oracle's arithmetic (minimum-image point_vector in FP64,
//    exp in FP64), factorised per axis where the points form a tensor grid;
//  * FP32: positions relative to the element centres (|x| <= h/2), the
//    element offset as an exact FP32 shift, e^{-alpha^2 s} on the
//    special-function unit with the exponent split into hi + lo parts,
//    block-Kahan sums per lane and a float-float combine of the lanes.
// Algorithmic work per (quadrature point, listed particle): 20 flops + 1 exp.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <vector>

#include "ggem_ff.cuh"
#include "ggem_internal.cuh"

namespace ggem {
namespace {

constexpr int kSpThreads = 256;
constexpr int kSpWarps = kSpThreads / 32;
constexpr int kSpCap32 = 512;    // staged particles per pass (FP32 records, 32 B)
constexpr int kSpCap64 = 256;    // staged particles per pass (FP64 records, 64 B)
constexpr int kSpMaxSeg = 2048;  // contiguous slot ranges of one dilated brick
constexpr int kSpMaxExt = 32;    // dilated brick extent per axis (5-bit coordinates)
constexpr size_t kSpRecBytes = 16384;
constexpr int kSpMaxWords = 1024;  // stencil bitmap words (32768 element offsets)
constexpr int kSpQueue = 96;      // queued members per warp (< 32 left + 64 new)
constexpr int kSpBatch = 6 * 32;  // floats of a staged batch of 32 members (FP32)
constexpr int kSpReachWords = 1024;  // union bitmap of a brick's elements
constexpr size_t kSpShared =
    kSpRecBytes + kSpCap32 * sizeof(uint32_t) +
    kSpWarps * (kSpBatch * sizeof(float) + kSpQueue * sizeof(uint32_t)) +
    2 * (kSpMaxSeg + 1) * sizeof(int32_t) + (kSpMaxWords + kSpReachWords) * sizeof(uint32_t);

struct SpreadGeo {
  Grid g;
  int lo[3], hi[3], dim[3];  // element-offset range of the stencil bitmap
  int nwords;                // 32-bit words of the bitmap
  int pad;                   // padded bitmap: bit (i + B - 1) + 32 (j + B - 1) + 1024 (k + B - 1)
                             // for the stencil offset index (i, j, k), read with the packed
                             // frame coordinates of a particle minus one value per element
  int B;                     // brick edge in elements
  int nb[3];                 // bricks per axis
  int nq;                    // quadrature points per element (<= 32)
  int lq;                    // lanes per quadrature point (32 / next power of two >= nq)
  float shift[3][kSpMaxExt]; // (float)(d h) for d in [lo, hi], per axis
  float L32[3];
  // FP32 constants: e^{-alpha^2 s} = 2^{s (e_hi + e_lo)}, g = E (c25 - c1 s)
  float e_hi, e_lo, c25, c1;
};

__device__ __forceinline__ float ex2_approx(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

__device__ __forceinline__ void kahan_acc(float &sum, float &comp, float v) {
  const float y = v - comp;
  const float t = sum + y;
  comp = (t - sum) - y;
  sum = t;
}

// the brick's dilated frame along one axis: start F (unwrapped) and extent E;
// full = the frame covers the whole periodic axis (coordinates absolute,
// offsets wrapped)
struct Frame {
  int F, E, full;
};

__device__ __forceinline__ Frame brick_frame(const SpreadGeo &sg, int d, int b0, int b1) {
  Frame f;
  const int nc = sg.g.nc[d];
  const int ext = (b1 - b0) + (sg.hi[d] - sg.lo[d]);
  if (sg.g.periodic[d] && ext >= nc) {
    f.F = 0;
    f.E = nc;
    f.full = 1;
  } else if (sg.g.periodic[d]) {
    f.F = b0 + sg.lo[d];
    f.E = ext;
    f.full = 0;
  } else {
    const int a = max(0, b0 + sg.lo[d]), z = min(nc - 1, b1 - 1 + sg.hi[d]);
    f.F = a;
    f.E = z - a + 1;
    f.full = 0;
  }
  return f;
}

__device__ __forceinline__ int wrap_cell(int k, int n) {
  k %= n;
  return k < 0 ? k + n : k;
}

// offset d (frame coordinates) of a staged particle from the element, or
// a value outside [lo, hi] when it is no stencil offset
__device__ __forceinline__ int axis_offset(const SpreadGeo &sg, int d, int us, int ue, int full) {
  int o = us - ue;
  if (full) {
    const int nc = sg.g.nc[d];
    if (o > nc / 2) o -= nc;
    else if (o < -((nc - 1) / 2)) o += nc;
  }
  return o;
}

// ANYFULL: some brick frame spans a whole periodic axis (small meshes);
// without it the wrapped-offset and minimum-image code is compiled out.
//
// The FP32 form is bound by instruction issue (81%) and shared-memory data
// (66% of its cycles): 144^3 elements x 8 points, N = 200k took 4.09 G warp
// instructions and 3.90 ms, then 3.68 G and 3.72 ms, and 3.53 ms with the four
// lanes per point known when compiling (LQ).  Two members of a lane
// share packed arithmetic up to the block sums, their positions and forces
// staged together (6 words a member instead of a position and a gathered
// record, 8); a point's four lanes reduce-scatter, so each converts and
// writes one component; the lanes decode 32 elements at once; two windows of
// candidates per pass.
// A lane's two members need not come through shared memory with 16 lanes per
// point (a shuffle) or 32 (one member).  N = 20k, us with one member
// at a time -> two: 27 points 923 -> 694, 12 points 632 -> 521, 4 points 433
// -> 424, 2 points 405 -> 398.
// LQ: the lanes per point, 4 or, read from sg, any (0)
template <bool F32, bool ANYFULL, bool PAD, int LQ>
__global__ void __launch_bounds__(kSpThreads, F32 ? 4 : 1) k_spread_brick(
    SpreadGeo sg, DevConsts K, const int32_t *__restrict__ start,
    const float4 *__restrict__ pos32, const double4_32a *__restrict__ pos64,
    const double *__restrict__ f_slot, const float4 *__restrict__ q_rel,
    const double *__restrict__ q_xyz, const uint32_t *__restrict__ bits,
    double *__restrict__ rho, unsigned long long *__restrict__ pairs) {
  extern __shared__ __align__(16) unsigned char sp_smem[];
  constexpr int CAP = F32 ? kSpCap32 : kSpCap64;
  // FP32 records as two arrays, positions [CAP] then forces [CAP]: the 16-byte
  // stride spreads the four members a warp reads at once over more banks
  // than 32-byte records would
  float4 *rec32 = reinterpret_cast<float4 *>(sp_smem);        // [2][CAP]
  double4_32a *rec64 = reinterpret_cast<double4_32a *>(sp_smem);  // [CAP][2]
  float *batch = reinterpret_cast<float *>(sp_smem + kSpRecBytes);  // [warps][kSpBatch]
  // FP32: the staged particles' frame coordinates once more, for the
  // membership pass (a 16-byte stride would take four times the banks)
  uint32_t *rec_u = reinterpret_cast<uint32_t *>(batch + kSpWarps * kSpBatch);  // [CAP]
  uint32_t *queue = rec_u + kSpCap32;                                // [warps][kSpQueue]
  int32_t *seg_begin = reinterpret_cast<int32_t *>(queue + kSpWarps * kSpQueue);
  int32_t *seg_pre = seg_begin + kSpMaxSeg + 1;
  uint32_t *s_bits = reinterpret_cast<uint32_t *>(seg_pre + kSpMaxSeg + 1);
  // the element-offset shifts and the stencil bitmap in shared memory: lanes
  // index them with different offsets (divergent constant-bank reads would
  // serialise)
  __shared__ float s_shift[3][kSpMaxExt];
  __shared__ int s_total;
  for (int k = threadIdx.x; k < 3 * kSpMaxExt; k += kSpThreads)
    s_shift[k / kSpMaxExt][k % kSpMaxExt] = sg.shift[k / kSpMaxExt][k % kSpMaxExt];
  for (int k = threadIdx.x; k < sg.nwords; k += kSpThreads) s_bits[k] = bits[k];
  uint32_t *s_reach = s_bits + kSpMaxWords;
  if (F32 && PAD)
    for (int k = threadIdx.x; k < kSpReachWords; k += kSpThreads) s_reach[k] = bits[sg.nwords + k];

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int B = sg.B;
  int bid = blockIdx.x;
  const int bx = bid % sg.nb[0];
  bid /= sg.nb[0];
  const int by = bid % sg.nb[1];
  const int bz = bid / sg.nb[1];
  const int e0[3] = {bx * B, by * B, bz * B};
  const int e1[3] = {min(e0[0] + B, sg.g.nc[0]), min(e0[1] + B, sg.g.nc[1]),
                     min(e0[2] + B, sg.g.nc[2])};
  Frame fr[3];
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    fr[d] = brick_frame(sg, d, e0[d], e1[d]);
    if (!ANYFULL) fr[d].full = 0;  // the host found no frame that spans an axis
  }
  // x segments per row: a periodic frame that is not the whole axis may
  // wrap once; others are one range
  const int xa = fr[0].F, xz = fr[0].F + fr[0].E - 1;
  const int nseg_x = (!fr[0].full && sg.g.periodic[0] && (xa < 0 || xz >= sg.g.nc[0])) ? 2 : 1;
  const int nrow = fr[1].E * fr[2].E;
  const int nseg = nrow * nseg_x;  // <= kSpMaxSeg (checked on the host)
  // slot range of every segment and the running prefix (block scan)
  for (int s0 = 0; s0 < nseg; s0 += kSpThreads) {
    const int s = s0 + threadIdx.x;
    int b = 0, cnt = 0;
    if (s < nseg) {
      const int row = s / nseg_x, k = s - row * nseg_x;
      const int uy = row % fr[1].E, uz = row / fr[1].E;
      const int cy = fr[1].full ? uy : (sg.g.periodic[1] ? wrap_cell(fr[1].F + uy, sg.g.nc[1])
                                                          : fr[1].F + uy);
      const int cz = fr[2].full ? uz : (sg.g.periodic[2] ? wrap_cell(fr[2].F + uz, sg.g.nc[2])
                                                          : fr[2].F + uz);
      int x0, x1;  // absolute cells [x0, x1]
      if (nseg_x == 1) {
        x0 = fr[0].full ? 0 : (sg.g.periodic[0] ? wrap_cell(xa, sg.g.nc[0]) : xa);
        x1 = x0 + fr[0].E - 1;
      } else if (k == 0) {
        x0 = wrap_cell(xa, sg.g.nc[0]);
        x1 = sg.g.nc[0] - 1;
      } else {
        x0 = 0;
        x1 = wrap_cell(xz, sg.g.nc[0]);
      }
      const int64_t rowc = (int64_t)sg.g.nc[0] * (cy + (int64_t)sg.g.nc[1] * cz);
      b = start[rowc + x0];
      cnt = start[rowc + x1 + 1] - b;
    }
    // block exclusive scan of cnt
    int incl = cnt;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int y = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += y;
    }
    __shared__ int wsum[kSpWarps];
    const int carry = (s0 == 0) ? 0 : seg_pre[s0];  // written before the last barrier
    if (lane == 31) wsum[warp] = incl;
    __syncthreads();
    int before = carry;
    for (int w = 0; w < warp; ++w) before += wsum[w];
    if (s < nseg) {
      seg_begin[s] = b;
      seg_pre[s] = before + incl - cnt;
    }
    if (threadIdx.x == kSpThreads - 1) seg_pre[min(s0 + kSpThreads, nseg)] = before + incl;
    __syncthreads();
  }
  if (threadIdx.x == 0) s_total = seg_pre[nseg];
  __syncthreads();
  const int total = s_total;
  // elements of this brick, one warp at a time
  const int ebx = e1[0] - e0[0], eby = e1[1] - e0[1], ebz = e1[2] - e0[2];
  const int nel = ebx * eby * ebz;
  const int nq = sg.nq, lq = LQ ? LQ : sg.lq;
  const int qi = lane / lq, sub = lane - qi * lq;
  const int llq = 31 - __clz(lq);
  unsigned long long my_pairs = 0;
  // the warp's member queue: per member its staged index (10 bits) and its
  // element offset (the padded bitmap index, or three 5-bit offsets); each
  // batch of 32 becomes positions in the element's frame (FP32: the staged
  // position plus the offset's shift, formed once per member instead of
  // once per point, one member per lane) with the staged index in .w
  uint32_t *mq = queue + warp * kSpQueue;
  float *mb = batch + warp * kSpBatch;
  // FP32, up to eight lanes per point: the two members that a lane takes one
  // after the other share a pair slot, i.e. member j of a batch (the t-th of
  // lane j % lq of a point) lies in slot (t / 2, j % lq), half t % 2
  float *mine = mb + 12 * ((qi >> 1) * lq + sub) + (qi & 1);
  const unsigned lt_mask = (1u << lane) - 1u;
  // with the padded bitmap, a particle at frame coordinates u is listed by
  // some element of the brick when the union bitmap holds u (shifted where
  // an open face clips the frame)
  int clip = 0;
  if (PAD)
    clip = (fr[0].F - (e0[0] + sg.lo[0])) + 32 * (fr[1].F - (e0[1] + sg.lo[1])) +
           1024 * (fr[2].F - (e0[2] + sg.lo[2]));
  __shared__ int s_kept[kSpWarps];
  // (a brick without particles in reach makes one empty pass: its sums are 0)
  for (int c0 = 0; c0 == 0 || c0 < total; c0 += CAP) {
    const int cw = min(CAP, total - c0);
    // stage particles [c0, c0 + cw), in order; the FP32 kernel drops those
    // that no element of the brick lists (about half of the dilated box), so
    // that every element's membership pass is as much shorter: 144^3 elements
    // x 8 points, N = 200k 4.22 -> 3.90 ms
    int cn = 0;
    for (int k0 = 0; k0 < cw; k0 += kSpThreads) {
      const int k = k0 + threadIdx.x;
      const int v = c0 + k;
      bool keep = k < cw;
      int slot = 0;
      uint32_t u = 0;
      float4 p = make_float4(0.f, 0.f, 0.f, 0.f);
      if (keep) {  // segment by binary search
        int lo = 0, hi = nseg - 1;
        while (lo < hi) {
          const int mid = (lo + hi + 1) >> 1;
          if (seg_pre[mid] <= v) lo = mid;
          else hi = mid - 1;
        }
        slot = seg_begin[lo] + (v - seg_pre[lo]);
        const int row = lo / nseg_x, kk = lo - row * nseg_x;
        const int uy = row % fr[1].E, uz = row / fr[1].E;
        p = pos32[slot];
        const int cid = __float_as_int(p.w);
        const int cx = cid % sg.g.nc[0];
        int ux;
        if (fr[0].full) ux = cx;
        else if (!sg.g.periodic[0]) ux = cx - fr[0].F;
        else if (nseg_x == 1) ux = cx - wrap_cell(xa, sg.g.nc[0]);
        else ux = kk == 0 ? cx - wrap_cell(xa, sg.g.nc[0]) : cx + (sg.g.nc[0] - wrap_cell(xa, sg.g.nc[0]));
        u = (uint32_t)ux | ((uint32_t)uy << 5) | ((uint32_t)uz << 10);
        if (F32 && PAD) {
          const int idx = (int)u + clip;
          keep = (s_reach[idx >> 5] >> (idx & 31)) & 1u;
        }
      }
      int at = k;
      if (F32 && PAD) {  // position among the kept ones
        const unsigned bal = __ballot_sync(0xffffffffu, keep);
        if (lane == 0) s_kept[warp] = __popc(bal);
        __syncthreads();
        at = cn + __popc(bal & lt_mask);
        for (int w = 0; w < kSpWarps; ++w) {
          if (w < warp) at += s_kept[w];
          cn += s_kept[w];
        }
        __syncthreads();
      }
      if (keep) {
        const double *fp = f_slot + 3 * (int64_t)slot;
        if (F32) {
          rec32[at] = make_float4(p.x, p.y, p.z, 0.f);
          rec_u[at] = u;
          rec32[kSpCap32 + at] =
              make_float4(d2f_bits(fp[0]), d2f_bits(fp[1]), d2f_bits(fp[2]), 0.f);
        } else {
          const double4_32a q = pos64[slot];
          rec64[2 * at] = make_double4_32a(q.x, q.y, q.z, __longlong_as_double((long long)u));
          rec64[2 * at + 1] = make_double4_32a(fp[0], fp[1], fp[2], 0.0);
        }
      }
    }
    if (!(F32 && PAD)) cn = cw;
    __syncthreads();
    // each lane decodes one of the warp's next 32 elements
    int64_t my_e = 0;
    int my_u = 0, my_q = 0;
    for (int it = 0; warp + kSpWarps * it < nel; ++it) {
      if ((it & 31) == 0) {
        const int le = min(warp + kSpWarps * (it + lane), nel - 1);
        const int lx = le % ebx, ly = (le / ebx) % eby, lz = le / (ebx * eby);
        const int ex = e0[0] + lx, ey = e0[1] + ly, ez = e0[2] + lz;
        my_e = ex + (int64_t)sg.g.nc[0] * (ey + (int64_t)sg.g.nc[1] * ez);
        const int ux = fr[0].full ? ex : ex - fr[0].F;
        const int uy = fr[1].full ? ey : ey - fr[1].F;
        const int uz = fr[2].full ? ez : ez - fr[2].F;
        my_u = ux | (uy << 10) | (uz << 20);
        // with the padded bitmap, the packed frame coordinates u of a staged
        // particle minus qe index the bitmap directly (each 5-bit field stays
        // in [0, 32) for every particle of the brick's frame)
        my_q = (ux + sg.lo[0] - B + 1) + 32 * (uy + sg.lo[1] - B + 1) +
               1024 * (uz + sg.lo[2] - B + 1);
      }
      const int64_t e = __shfl_sync(0xffffffffu, my_e, it & 31);
      const int ue = __shfl_sync(0xffffffffu, my_u, it & 31);
      const int uex = ue & 1023, uey = (ue >> 10) & 1023, uez = ue >> 20;
      const int qe = __shfl_sync(0xffffffffu, my_q, it & 31);
      const bool qok = qi < nq;
      const int64_t qg = e * nq + (qok ? qi : 0);
      float4 qr = make_float4(0.f, 0.f, 0.f, 0.f);
      double q0 = 0.0, q1 = 0.0, q2 = 0.0;
      if (F32) {
        qr = q_rel[qg];
      } else {
        q0 = q_xyz[3 * qg];
        q1 = q_xyz[3 * qg + 1];
        q2 = q_xyz[3 * qg + 2];
      }
      float sx = 0.f, sy = 0.f, sz = 0.f, cx = 0.f, cy = 0.f, cz = 0.f;
      float bx_ = 0.f, by_ = 0.f, bz_ = 0.f;
      int blk = 0, elem_pairs = 0;
      // minimum image (pm_periodic_boundary.C:350-374); only an axis whose
      // frame is the whole box can produce |d| > L/2
      auto axis32 = [&](int k, float d) {
        if (ANYFULL && fr[k].full) {
          if (d <= -0.5f * sg.L32[k]) d += sg.L32[k];
          if (d > 0.5f * sg.L32[k]) d -= sg.L32[k];
        }
        return d;
      };
      double ax = 0.0, ay = 0.0, az = 0.0;
      // members: staged particles whose element offset is a stencil offset,
      // queued in staging order and summed 32 at a time; lane (qi, sub)
      // takes members sub, sub + lq, ... of each batch, so every lane sees its
      // members in the order of one pass over the whole member list
      int queued = 0;  // warp-uniform
      for (int k0 = 0; k0 < cn; k0 += 64) {
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const int k = k0 + 32 * h + lane;
          bool in = false;
          uint32_t item = 0;
          if (k < cn) {
            const uint32_t u = F32 ? rec_u[k] : (uint32_t)__double_as_longlong(rec64[2 * k].w);
            if (PAD) {
              const int idx = (int)u - qe;
              in = (s_bits[idx >> 5] >> (idx & 31)) & 1u;
              item = (uint32_t)k | ((uint32_t)idx << 10);
            } else {
              const int ix =
                  axis_offset(sg, 0, (int)(u & 31u), uex, ANYFULL && fr[0].full) - sg.lo[0];
              const int iy =
                  axis_offset(sg, 1, (int)((u >> 5) & 31u), uey, ANYFULL && fr[1].full) - sg.lo[1];
              const int iz =
                  axis_offset(sg, 2, (int)(u >> 10), uez, ANYFULL && fr[2].full) - sg.lo[2];
              if ((unsigned)ix < (unsigned)sg.dim[0] && (unsigned)iy < (unsigned)sg.dim[1] &&
                  (unsigned)iz < (unsigned)sg.dim[2]) {
                const int idx = (iz * sg.dim[1] + iy) * sg.dim[0] + ix;
                in = (s_bits[idx >> 5] >> (idx & 31)) & 1u;
                item = (uint32_t)k | ((uint32_t)ix << 10) | ((uint32_t)iy << 15) |
                       ((uint32_t)iz << 20);
              }
            }
          }
          const unsigned bal = __ballot_sync(0xffffffffu, in);
          if (in) mq[queued + __popc(bal & lt_mask)] = item;
          queued += __popc(bal);
        }
        const bool last = k0 + 64 >= cn;
        int head = 0;  // warp-uniform: members of the queue that are done
        while (queued - head >= 32 || (last && queued > head)) {
          __syncwarp();
          const int m = min(queued - head, 32);
          // (FP32: position and force of member `lane`; past the last member
          // zeros, whose terms are exact zeros)
          float4 v = make_float4(0.f, 0.f, 0.f, 0.f), fv = v;
          if (F32) {
            if (lane < m) {
              const uint32_t en = mq[head + lane];
              const int kk = (int)(en & 1023u);
              int ix, iy, iz;
              if (PAD) {
                const int idx = (int)(en >> 10);
                ix = (idx & 31) - (B - 1);
                iy = ((idx >> 5) & 31) - (B - 1);
                iz = (idx >> 10) - (B - 1);
              } else {
                ix = (int)((en >> 10) & 31u);
                iy = (int)((en >> 15) & 31u);
                iz = (int)(en >> 20);
              }
              v = rec32[kk];
              fv = rec32[kSpCap32 + kk];
              v.x += s_shift[0][ix];
              v.y += s_shift[1][iy];
              v.z += s_shift[2][iz];
            }
            if (lq < 16) {
              mine[0] = v.x;
              mine[2] = v.y;
              mine[4] = v.z;
              mine[6] = fv.x;
              mine[8] = fv.y;
              mine[10] = fv.z;
            }
          }
          __syncwarp();
          // this lane's own member into the block sums
          auto term32 = [&]() {
            const float dx = axis32(0, v.x - qr.x);
            const float dy = axis32(1, v.y - qr.y);
            const float dz = axis32(2, v.z - qr.z);
            const float s2 = fmaf(dz, dz, fmaf(dy, dy, dx * dx));
            const float p = s2 * sg.e_hi;
            const float r = fmaf(s2, sg.e_lo, fmaf(s2, sg.e_hi, -p));
            const float E0 = ex2_approx(p);
            const float E = fmaf(E0, r * 0.6931471805599453f, E0);
            const float gv = E * fmaf(-sg.c1, s2, sg.c25);
            bx_ = fmaf(gv, fv.x, bx_);
            by_ = fmaf(gv, fv.y, by_);
            bz_ = fmaf(gv, fv.z, bz_);
          };
          // two members, one after the other into the block sums; what
          // precedes the sums in packed arithmetic (each half rounds as the
          // scalar form does)
          auto pair_terms = [&](const float4 &a, const float4 &b, const float4 &c) {
            float2 dx = __fadd2_rn(make_float2(a.x, a.y), make_float2(-qr.x, -qr.x));
            float2 dy = __fadd2_rn(make_float2(a.z, a.w), make_float2(-qr.y, -qr.y));
            float2 dz = __fadd2_rn(make_float2(b.x, b.y), make_float2(-qr.z, -qr.z));
            if (ANYFULL) {
              dx = make_float2(axis32(0, dx.x), axis32(0, dx.y));
              dy = make_float2(axis32(1, dy.x), axis32(1, dy.y));
              dz = make_float2(axis32(2, dz.x), axis32(2, dz.y));
            }
            const float2 s2 = __ffma2_rn(dz, dz, __ffma2_rn(dy, dy, __fmul2_rn(dx, dx)));
            const float2 pn = __fmul2_rn(s2, make_float2(-sg.e_hi, -sg.e_hi));
            const float2 r = __ffma2_rn(s2, make_float2(sg.e_lo, sg.e_lo),
                                        __ffma2_rn(s2, make_float2(sg.e_hi, sg.e_hi), pn));
            const float2 E0 = make_float2(ex2_approx(-pn.x), ex2_approx(-pn.y));
            const float2 E = __ffma2_rn(
                E0, __fmul2_rn(r, make_float2(0.6931471805599453f, 0.6931471805599453f)), E0);
            const float2 gv = __fmul2_rn(E, __ffma2_rn(make_float2(-sg.c1, -sg.c1), s2,
                                                       make_float2(sg.c25, sg.c25)));
            bx_ = fmaf(gv.y, b.w, fmaf(gv.x, b.z, bx_));
            by_ = fmaf(gv.y, c.y, fmaf(gv.x, c.x, by_));
            bz_ = fmaf(gv.y, c.w, fmaf(gv.x, c.z, bz_));
          };
          auto pair32 = [&](const float4 *o) { pair_terms(o[0], o[1], o[2]); };
          auto flush32 = [&]() {  // the block sums into the compensated sums
            kahan_acc(sx, cx, bx_);
            kahan_acc(sy, cy, by_);
            kahan_acc(sz, cz, bz_);
            bx_ = by_ = bz_ = 0.f;
            blk = 0;
          };
          if (F32) {
            // this lane's members of the batch, eight of them into the
            // compensated sums at a time (every earlier batch was full)
            const float4 *o = reinterpret_cast<const float4 *>(mb) + 3 * sub;
            const int cnt = (m - sub + lq - 1) >> llq, step = 3 * lq;
            if (LQ == 4) {
              if (m == 32) {
#pragma unroll
                for (int t = 0; t < 4; ++t) pair32(o + 12 * t);
                flush32();
              } else {
                for (int t = 0; 8 * t < m; ++t) pair32(o + 12 * t);
                if (cnt == 8) flush32();
              }
            } else if (lq < 4) {
              int t = 0;
              for (; 2 * t + 8 <= cnt; t += 4, o += 4 * step) {
#pragma unroll
                for (int u = 0; u < 4; ++u) pair32(o + u * step);
                flush32();
              }
              for (; 2 * t < cnt; ++t, o += step) pair32(o);
            } else if (lq == 8) {
              for (int t = 0; 2 * t < cnt; ++t) pair32(o + t * step);
              blk += cnt;
              if (blk == 8) flush32();
            } else if (lq == 16) {  // the lane's own member and that of the lane 16 from it
              const bool up = lane & 16;
              auto both = [&](float w) {
                const float other = __shfl_xor_sync(0xffffffffu, w, 16);
                return up ? make_float2(other, w) : make_float2(w, other);
              };
              const float2 x = both(v.x), y = both(v.y), z = both(v.z);
              const float2 fx = both(fv.x), fy = both(fv.y), fz = both(fv.z);
              pair_terms(make_float4(x.x, x.y, y.x, y.y), make_float4(z.x, z.y, fx.x, fx.y),
                         make_float4(fy.x, fy.y, fz.x, fz.y));
              blk += cnt;
              if (blk == 8) flush32();
            } else if (sub < m) {
              term32();
              if (++blk == 8) flush32();
            }
          } else {
            for (int j = sub; j < m && qok; j += lq) {
              const int kk = (int)(mq[head + j] & 1023u);
              const double4_32a a = rec64[2 * kk], fb = rec64[2 * kk + 1];
              // point_vector(q, x_j) with the minimum image (pm_periodic_boundary.C:350-374)
              double x[3] = {a.x - q0, a.y - q1, a.z - q2};
#pragma unroll
              for (int d = 0; d < 3; ++d) {
                if (sg.g.periodic[d]) {
                  const double xs = sg.g.L[d];
                  if (x[d] <= -xs / 2.0) x[d] += xs;
                  if (x[d] > xs / 2.0) x[d] -= xs;
                }
              }
              // smoothed_force_exp (ggem_stokes.C:117-128)
              const double r2 = x[0] * x[0] + x[1] * x[1] + x[2] * x[2];
              const double a2r2 = K.alpha2 * r2;
              const double gv = K.alpha3_pi_23 * exp(-a2r2) * (2.5 - a2r2);
              ax += gv * fb.x;
              ay += gv * fb.y;
              az += gv * fb.z;
            }
          }
          head += m;
        }
        elem_pairs += head;
        // the rest of the queue to its front
        if (head) {
          queued -= head;
          const uint32_t rv = lane < queued ? mq[head + lane] : 0u;
          __syncwarp();
          if (lane < queued) mq[lane] = rv;
        }
      }
      my_pairs += (unsigned)elem_pairs;
      __syncwarp();
      double out[3];
      if (F32) {
        kahan_acc(sx, cx, bx_);
        kahan_acc(sy, cy, by_);
        kahan_acc(sz, cz, bz_);
        float h[3] = {sx, sy, sz}, l[3] = {-cx, -cy, -cz};
        if (lq == 4) {
          // reduce-scatter over the point's four lanes, (0 + 1) + (2 + 3):
          // lane 0 ends with x, 1 and 3 with y, 2 with z
          const bool odd = sub & 1, high = sub & 2;
          float kh = odd ? h[1] : h[0], kl = odd ? l[1] : l[0];
          ff_add(kh, kl, __shfl_xor_sync(0xffffffffu, odd ? h[0] : h[1], 1),
                 __shfl_xor_sync(0xffffffffu, odd ? l[0] : l[1], 1));
          ff_add(h[2], l[2], __shfl_xor_sync(0xffffffffu, h[2], 1),
                 __shfl_xor_sync(0xffffffffu, l[2], 1));
          const bool z = !odd && high;  // keeps z, sends x; lane 0 the other way, odd lanes y
          float oh = z ? h[2] : kh, ol = z ? l[2] : kl;
          ff_add(oh, ol, __shfl_xor_sync(0xffffffffu, odd || z ? kh : h[2], 2),
                 __shfl_xor_sync(0xffffffffu, odd || z ? kl : l[2], 2));
          if (qok && sub < 3) {
            const double v = f2d_bits(oh) + f2d_bits(ol);
            double *dst = rho + 3 * qg + sub;
            // a brick staged in several passes adds each pass's sums
            *dst = c0 == 0 ? v : *dst + v;
          }
          __syncwarp();  // the member list is rebuilt for the next element
          continue;
        }
        for (int o = 1; o < lq; o <<= 1) {
#pragma unroll
          for (int c = 0; c < 3; ++c) {
            const float h2 = __shfl_xor_sync(0xffffffffu, h[c], o);
            const float l2 = __shfl_xor_sync(0xffffffffu, l[c], o);
            ff_add(h[c], l[c], h2, l2);
          }
        }
#pragma unroll
        for (int c = 0; c < 3; ++c) out[c] = f2d_bits(h[c]) + f2d_bits(l[c]);
      } else {
        out[0] = ax;
        out[1] = ay;
        out[2] = az;
        for (int o = 1; o < lq; o <<= 1) {
#pragma unroll
          for (int c = 0; c < 3; ++c) out[c] += __shfl_xor_sync(0xffffffffu, out[c], o);
        }
      }
      if (qok && sub == 0) {
        double *dst = rho + 3 * qg;
        if (c0 == 0) {
          dst[0] = out[0];
          dst[1] = out[1];
          dst[2] = out[2];
        } else {  // a brick staged in several passes adds each pass's sums
          dst[0] += out[0];
          dst[1] += out[1];
          dst[2] += out[2];
        }
      }
      __syncwarp();  // the member list is rebuilt for the next element
    }
    __syncthreads();  // the staged particles are replaced
  }
  if (pairs) {
    if (lane == 0 && my_pairs) atomicAdd(pairs, my_pairs * (unsigned long long)nq);
  }
}

// ---- separable FP64 spread -------------------------------------------------
// On a mesh whose quadrature points form a tensor grid (every point's x
// depends on its element column and an index alone, likewise y and z;
// checked bit for bit when the points are set), the Gaussian factorises:
// with h_d = alpha^2 d^2 and g_d = e^{-h_d} per axis,
//   g_alpha = alpha^3 pi^{-3/2} g_x g_y g_z (2.5 - h_x - h_y - h_z).
// k_axis_factors forms (g, h) of every particle at every axis coordinate of
// its stencil window once (~80 exponentials per particle instead of one per
// pair); k_spread_sep combines them: for a row of PX points along x,
// F = (g_y g_z) f, w = (2.5 - h_y) - h_z and, per point, v = w g_x - g_x h_x
// and three fused multiply-adds, i.e. 5 + 4 PX FP64 instructions per row and
// member (6.5 per pair at 2 x 2 x 2 points) against ~50 with the minimum
// image, r^2 and exp per pair.  GB300's FP64 pipe (two lanes per SM and
// clock) bounds both; the products of three factors carry the rounding that
// alpha^2 r^2 carried before.
//
// A brick of B^3 elements stages the particles that any of its elements
// lists, each with its factors at the brick's B p coordinates per axis and
// its force.  A lane owns one row of one element (E = 32 / R elements per
// warp, R rows each) and walks the set bits of the element's member mask:
// neighbouring elements list nearly the same particles, so the lanes stay
// level without a reduction at the end.
struct SepGeo {
  int p[3];       // points per element and axis
  int R, E;       // rows per element, elements per warp
  int aoff[3];    // offset of an axis inside a particle's factors
  int nfac;       // factors per particle (double2 each)
  int stride;     // staged double2 per particle: B (px + py + pz) + 2
  int cap, nw;    // staged particles per pass (a multiple of 32), mask words
  signed char qmap[32];  // point index of (row, a)
  signed char rep[3][32];  // a point with each axis index
};

// window[slot][axis][offset - lo][a] = (g, g h) on x, (g, 2.5 - h) on y,
// (alpha^3 pi^{-3/2} g, h) on z; the offset is the particle's element minus
// the point's, zero where that element lies outside an open axis
__global__ void __launch_bounds__(256) k_axis_factors(
    int64_t n, SpreadGeo sg, SepGeo sp, DevConsts K, const double *__restrict__ qp,
    const float4 *__restrict__ pos32, const double4_32a *__restrict__ pos64,
    double2 *__restrict__ fac) {
  const int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (t >= n * sp.nfac) return;
  const int64_t s = t / sp.nfac;
  const int r = (int)(t - s * sp.nfac);
  const int d = r >= sp.aoff[2] ? 2 : (r >= sp.aoff[1] ? 1 : 0);
  const int k = r - sp.aoff[d];
  const int off = sg.lo[d] + k / sp.p[d], a = k % sp.p[d];
  const int cid = __float_as_int(pos32[s].w);
  const int nc0 = sg.g.nc[0], nc1 = sg.g.nc[1], nc = sg.g.nc[d];
  int e = (d == 0 ? cid % nc0 : (d == 1 ? (cid / nc0) % nc1 : cid / (nc0 * nc1))) - off;
  double2 v = make_double2(0.0, 0.0);
  if (sg.g.periodic[d]) e = wrap_cell(e, nc);
  if (e >= 0 && e < nc) {
    const double4_32a P = pos64[s];
    const int64_t el = d == 0 ? e : (d == 1 ? e * (int64_t)nc0 : e * (int64_t)nc0 * nc1);
    const double q = qp[3 * (el * sg.nq + sp.rep[d][a]) + d];
    double x = (d == 0 ? P.x : (d == 1 ? P.y : P.z)) - q;
    if (sg.g.periodic[d]) {  // minimum image (pm_periodic_boundary.C:350-374)
      const double xs = sg.g.L[d];
      if (x <= -xs / 2.0) x += xs;
      if (x > xs / 2.0) x -= xs;
    }
    // h as a double and its remainder: e^{-h} would carry h times the
    // rounding of h, and three factors make one Gaussian
    const double x2 = x * x, h = K.alpha2 * x2;
    const double lo = fma(K.alpha2, fma(x, x, -x2), fma(K.alpha2, x2, -h));
    const double g0 = exp(-h), g = fma(-lo, g0, g0);
    v = d == 0 ? make_double2(g, g * h)
               : (d == 1 ? make_double2(g, 2.5 - h) : make_double2(K.alpha3_pi_23 * g, h));
  }
  fac[t] = v;
}

template <int PX, bool ANYFULL>
__global__ void __launch_bounds__(kSpThreads, 2) k_spread_sep(
    SpreadGeo sg, SepGeo sp, const int32_t *__restrict__ start, const float4 *__restrict__ pos32,
    const double *__restrict__ f_slot, const double2 *__restrict__ fac,
    const uint32_t *__restrict__ bits, double *__restrict__ rho,
    unsigned long long *__restrict__ pairs) {
  extern __shared__ __align__(16) unsigned char sp_smem[];
  double2 *stage = reinterpret_cast<double2 *>(sp_smem);  // [cap][stride]
  uint32_t *mask = reinterpret_cast<uint32_t *>(stage + (size_t)sp.cap * sp.stride);  // [B^3][nw]
  int2 *item = reinterpret_cast<int2 *>(mask + 64 * sp.nw);  // [cap] (slot, frame coordinates)
  int32_t *seg_begin = reinterpret_cast<int32_t *>(item + sp.cap);
  int32_t *seg_pre = seg_begin + kSpMaxSeg + 1;
  uint32_t *s_bits = reinterpret_cast<uint32_t *>(seg_pre + kSpMaxSeg + 1);
  __shared__ int wsum[kSpWarps];
  __shared__ int s_next;
  for (int k = threadIdx.x; k < sg.nwords; k += kSpThreads) s_bits[k] = bits[k];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const unsigned lt_mask = (1u << lane) - 1u;
  const int B = sg.B;
  int bid = blockIdx.x;
  const int bx = bid % sg.nb[0];
  bid /= sg.nb[0];
  const int e0[3] = {bx * B, (bid % sg.nb[1]) * B, (bid / sg.nb[1]) * B};
  const int e1[3] = {min(e0[0] + B, sg.g.nc[0]), min(e0[1] + B, sg.g.nc[1]),
                     min(e0[2] + B, sg.g.nc[2])};
  Frame fr[3];
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    fr[d] = brick_frame(sg, d, e0[d], e1[d]);
    if (!ANYFULL) fr[d].full = 0;
  }
  // slot ranges of the dilated brick's rows along x (as in k_spread_brick)
  const int nx = sg.g.nc[0];
  const int xa = fr[0].F, xz = fr[0].F + fr[0].E - 1;
  const int xaw = sg.g.periodic[0] ? wrap_cell(xa, nx) : xa;
  const int nseg_x = (!fr[0].full && sg.g.periodic[0] && (xa < 0 || xz >= nx)) ? 2 : 1;
  const int nseg = fr[1].E * fr[2].E * nseg_x;  // <= kSpMaxSeg (checked on the host)
  int total = 0;
  for (int s0 = 0; s0 < nseg; s0 += kSpThreads) {
    const int s = s0 + threadIdx.x;
    int b = 0, cnt = 0;
    if (s < nseg) {
      const int row = s / nseg_x, k = s - row * nseg_x;
      int cy = fr[1].F + row % fr[1].E, cz = fr[2].F + row / fr[1].E;
      if (sg.g.periodic[1]) cy = wrap_cell(cy, sg.g.nc[1]);
      if (sg.g.periodic[2]) cz = wrap_cell(cz, sg.g.nc[2]);
      int x0 = fr[0].full ? 0 : xaw, x1 = x0 + fr[0].E - 1;
      if (nseg_x == 2) {
        if (k == 0) x1 = nx - 1;
        else x0 = 0, x1 = wrap_cell(xz, nx);
      }
      const int64_t rowc = (int64_t)nx * (cy + (int64_t)sg.g.nc[1] * cz);
      b = start[rowc + x0];
      cnt = start[rowc + x1 + 1] - b;
    }
    int incl = cnt;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int y = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += y;
    }
    if (lane == 31) wsum[warp] = incl;
    __syncthreads();
    int before = total;
    for (int w = 0; w < kSpWarps; ++w) {
      if (w < warp) before += wsum[w];
      total += wsum[w];
    }
    if (s < nseg) {
      seg_begin[s] = b;
      seg_pre[s] = before + incl - cnt;
    }
    __syncthreads();
  }
  const int ebx = e1[0] - e0[0], eby = e1[1] - e0[1], ebz = e1[2] - e0[2];
  const int nel = ebx * eby * ebz;
  const int u0[3] = {fr[0].full ? e0[0] : e0[0] - fr[0].F, fr[1].full ? e0[1] : e0[1] - fr[1].F,
                     fr[2].full ? e0[2] : e0[2] - fr[2].F};
  // is a particle (frame coordinates u) listed by the element at frame
  // coordinates (x, y, z)?
  auto lists = [&](uint32_t u, int x, int y, int z) -> bool {
    if (sg.pad) {
      const int idx = (int)u - ((x + sg.lo[0] - B + 1) + 32 * (y + sg.lo[1] - B + 1) +
                                1024 * (z + sg.lo[2] - B + 1));
      return (s_bits[idx >> 5] >> (idx & 31)) & 1u;
    }
    const int ix = axis_offset(sg, 0, (int)(u & 31u), x, ANYFULL && fr[0].full) - sg.lo[0];
    const int iy = axis_offset(sg, 1, (int)((u >> 5) & 31u), y, ANYFULL && fr[1].full) - sg.lo[1];
    const int iz = axis_offset(sg, 2, (int)(u >> 10), z, ANYFULL && fr[2].full) - sg.lo[2];
    if ((unsigned)ix >= (unsigned)sg.dim[0] || (unsigned)iy >= (unsigned)sg.dim[1] ||
        (unsigned)iz >= (unsigned)sg.dim[2])
      return false;
    const int idx = (iz * sg.dim[1] + iy) * sg.dim[0] + ix;
    return (s_bits[idx >> 5] >> (idx & 31)) & 1u;
  };
  unsigned long long my_pairs = 0;
  bool first = true;
  int c0 = 0;
  do {
    // the next particles that some element of the brick lists, in order, up
    // to cap of them; s_next: the candidate where the next pass resumes
    int kept = 0;
    while (c0 < total && kept < sp.cap) {
      const int v = c0 + threadIdx.x;
      bool in = v < total;
      int2 it = make_int2(0, 0);
      if (in) {
        int lo = 0, hi = nseg - 1;
        while (lo < hi) {
          const int mid = (lo + hi + 1) >> 1;
          if (seg_pre[mid] <= v) lo = mid;
          else hi = mid - 1;
        }
        const int slot = seg_begin[lo] + (v - seg_pre[lo]);
        const int row = lo / nseg_x, kk = lo - row * nseg_x;
        const int cx = __float_as_int(pos32[slot].w) % nx;
        int ux = cx;
        if (!fr[0].full) ux = cx - xaw + (kk == 1 ? nx : 0);
        it = make_int2(slot, ux | ((row % fr[1].E) << 5) | ((row / fr[1].E) << 10));
        in = false;
        for (int z = 0; z < ebz && !in; ++z)
          for (int y = 0; y < eby && !in; ++y)
            for (int x = 0; x < ebx && !in; ++x)
              in = lists((uint32_t)it.y, u0[0] + x, u0[1] + y, u0[2] + z);
      }
      const unsigned bal = __ballot_sync(0xffffffffu, in);
      if (lane == 0) wsum[warp] = __popc(bal);
      if (threadIdx.x == 0) s_next = min(c0 + kSpThreads, total);
      __syncthreads();
      int at = kept, found = kept;
      for (int w = 0; w < kSpWarps; ++w) {
        if (w < warp) at += wsum[w];
        found += wsum[w];
      }
      at += __popc(bal & lt_mask);
      if (in && at < sp.cap) item[at] = it;
      if (in && at == sp.cap) s_next = v;  // the first one without room
      __syncthreads();
      kept = min(found, sp.cap);
      c0 = s_next;
      __syncthreads();
    }
    // stage the kept particles: one warp per particle, one lane per factor
    for (int r = lane; r < sp.stride; r += 32) {
      const int nfx = B * sp.p[0], nfy = nfx + B * sp.p[1], nfz = nfy + B * sp.p[2];
      const int d = r >= nfz ? 3 : (r >= nfy ? 2 : (r >= nfx ? 1 : 0));
      const int k = r - (d == 3 ? nfz : (d == 2 ? nfy : (d == 1 ? nfx : 0)));
      const int pd = d < 3 ? sp.p[d] : 1;
      const int a = k % pd, ue = d < 3 ? u0[d] + k / pd : 0;
      for (int p = warp; p < kept; p += kSpWarps) {
        const int2 it = item[p];
        double2 v = make_double2(0.0, 0.0);
        if (d == 3) {
          const double *fp = f_slot + 3 * (int64_t)it.x;
          v = k == 0 ? make_double2(fp[0], fp[1]) : make_double2(fp[2], 0.0);
        } else {
          const int i =
              axis_offset(sg, d, (it.y >> (5 * d)) & 31, ue, ANYFULL && fr[d].full) - sg.lo[d];
          if ((unsigned)i < (unsigned)sg.dim[d])
            v = fac[(int64_t)it.x * sp.nfac + sp.aoff[d] + i * pd + a];
        }
        stage[p * sp.stride + r] = v;
      }
    }
    __syncthreads();
    const int nw = (kept + 31) >> 5;
    for (int g = warp; g * sp.E < nel; g += kSpWarps) {
      const int el0 = g * sp.E, ne = min(sp.E, nel - el0);
      for (int q = 0; q < ne; ++q) {
        const int le = el0 + q;
        const int x = u0[0] + le % ebx, y = u0[1] + (le / ebx) % eby, z = u0[2] + le / (ebx * eby);
        for (int w = 0; w < nw; ++w) {
          const int k = 32 * w + lane;
          const unsigned m = __ballot_sync(
              0xffffffffu, k < kept && lists((uint32_t)item[min(k, kept - 1)].y, x, y, z));
          if (lane == 0) mask[le * sp.nw + w] = m;
          my_pairs += (unsigned long long)__popc(m);
        }
      }
      __syncwarp();
      const int q = lane / sp.R, row = lane - q * sp.R;
      const bool act = q < ne;
      const int le = el0 + (act ? q : 0);
      const int lx = le % ebx, ly = (le / ebx) % eby, lz = le / (ebx * eby);
      const int b = row % sp.p[1], c = row / sp.p[1];
      const double2 *X = stage + lx * PX;
      const double2 *Y = stage + B * PX + ly * sp.p[1] + b;
      const double2 *Z = stage + B * (PX + sp.p[1]) + lz * sp.p[2] + c;
      const double2 *Fp = stage + sp.stride - 2;
      const uint32_t *mrow = mask + le * sp.nw;
      // kAcc sums per point, members in turn: one sum over ~70 members
      // rounds three times as much as the lanes of k_spread_brick did
      constexpr int kAcc = PX == 1 ? 8 : (PX == 2 ? 6 : 3);
      double acc[kAcc][PX][3];
#pragma unroll
      for (int u = 0; u < kAcc; ++u)
#pragma unroll
        for (int a = 0; a < PX; ++a) acc[u][a][0] = acc[u][a][1] = acc[u][a][2] = 0.0;
      int w = 0;
      uint32_t m = act && nw > 0 ? mrow[0] : 0u;
      const int wend = act ? nw : 0;
      bool more = true;
      while (more) {
#pragma unroll
        for (int u = 0; u < kAcc; ++u) {
          while (m == 0u && w + 1 < wend) m = mrow[++w];
          const bool has = m != 0u;
          more = __any_sync(0xffffffffu, has);
          if (!more) break;
          if (has) {
            const int o = (32 * w + __ffs(m) - 1) * sp.stride;
            m &= m - 1u;
            const double2 gy = Y[o], gz = Z[o], f01 = Fp[o], f2 = Fp[o + 1];
            const double gyz = gy.x * gz.x, wv = gy.y - gz.y;
            const double F0 = gyz * f01.x, F1 = gyz * f01.y, F2 = gyz * f2.x;
#pragma unroll
            for (int a = 0; a < PX; ++a) {
              const double2 gx = X[o + a];
              const double v = fma(wv, gx.x, -gx.y);
              acc[u][a][0] = fma(v, F0, acc[u][a][0]);
              acc[u][a][1] = fma(v, F1, acc[u][a][1]);
              acc[u][a][2] = fma(v, F2, acc[u][a][2]);
            }
          }
        }
      }
#pragma unroll
      for (int u = 1; u < kAcc; ++u)
#pragma unroll
        for (int a = 0; a < PX; ++a)
#pragma unroll
          for (int d = 0; d < 3; ++d) acc[0][a][d] += acc[u][a][d];
      if (act) {
        const int64_t e = (e0[0] + lx) + (int64_t)nx * ((e0[1] + ly) +
                                                        (int64_t)sg.g.nc[1] * (e0[2] + lz));
#pragma unroll
        for (int a = 0; a < PX; ++a) {
          double *dst = rho + 3 * (e * sg.nq + sp.qmap[row * PX + a]);
#pragma unroll
          for (int d = 0; d < 3; ++d) dst[d] = first ? acc[0][a][d] : dst[d] + acc[0][a][d];
        }
      }
      __syncwarp();  // the warp's masks are rebuilt
    }
    first = false;
    __syncthreads();  // the staged particles are replaced
  } while (c0 < total);
  if (pairs && lane == 0 && my_pairs)
    atomicAdd(pairs, my_pairs * (unsigned long long)sg.nq);
}

// Do the points form a tensor grid?  The first element gives the indices (a
// point's coordinate among the distinct ones of its axis, -0 and 0 alike) and
// a point with each index, whose copies in the elements along the axis give
// the coordinates; every point of the mesh is compared with those.
struct AxisMap {
  int off;                  // a point differs from the grid
  int p[3];                 // distinct coordinates per element and axis
  signed char idx[3][32];   // the axis index of each point
  signed char rep[3][32];   // a point with each index
};

// quadrature points relative to their element centre (FP64 difference,
// rounded once to FP32; w = 0), and the axis map to the host's pinned copy,
// which costs a set of points 2 us and no other wait
__global__ void __launch_bounds__(256) k_qp_rel(int64_t nqt, int nq, Grid g,
                                                const double *__restrict__ q,
                                                volatile AxisMap *host, float4 *__restrict__ rel) {
  __shared__ int s_p[3], s_idx[3][32], s_rep[3][32];
  if (threadIdx.x < 96) {
    const int d = threadIdx.x >> 5, k = threadIdx.x & 31;
    const double v = (k < nq ? q[3 * k + d] : 0.0) + 0.0;  // (-0 becomes 0)
    const unsigned in = __ballot_sync(0xffffffffu, k < nq);
    const unsigned same =
        in & __match_any_sync(0xffffffffu, (unsigned long long)__double_as_longlong(v));
    const int first = same ? __ffs(same) - 1 : 0;
    const unsigned firsts = __ballot_sync(0xffffffffu, k < nq && first == k);
    const int a = __popc(firsts & ((1u << first) - 1u));
    s_idx[d][k] = a;
    if (k < nq && first == k) s_rep[d][a] = k;
    if (k == 0) s_p[d] = __popc(firsts);
    if (blockIdx.x == 0) {
      host->idx[d][k] = (signed char)a;
      if (k < nq && first == k) host->rep[d][a] = (signed char)k;
      if (k == 0) host->p[d] = __popc(firsts);
    }
  }
  __syncthreads();
  const int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  bool off = false;
  if (t < nqt) {
    const int64_t e = t / nq;
    const int k = (int)(t - e * nq);
    const int nx = g.nc[0];
    const int64_t nxy = (int64_t)nx * g.nc[1];
    const int ex = (int)(e % nx), ey = (int)((e / nx) % g.nc[1]), ez = (int)(e / nxy);
    const double cx = g.lo[0] + (ex + 0.5) * g.h[0];
    const double cy = g.lo[1] + (ey + 0.5) * g.h[1];
    const double cz = g.lo[2] + (ez + 0.5) * g.h[2];
    const double x = q[3 * t], y = q[3 * t + 1], z = q[3 * t + 2];
    rel[t] = make_float4((float)(x - cx), (float)(y - cy), (float)(z - cz), 0.f);
    if (s_p[0] * s_p[1] * s_p[2] == nq)  // (the host sees that too)
      off = x != q[3 * (ex * (int64_t)nq + s_rep[0][s_idx[0][k]])] ||
            y != q[3 * (ey * (int64_t)nx * nq + s_rep[1][s_idx[1][k]]) + 1] ||
            z != q[3 * (ez * nxy * nq + s_rep[2][s_idx[2][k]]) + 2];
  }
  if (__syncthreads_or(off) && threadIdx.x == 0) host->off = 1;
}

struct DeviceGuard {
  int prev = -1;
  explicit DeviceGuard(int dev) {
    cudaGetDevice(&prev);
    if (prev != dev) cudaSetDevice(dev);
  }
  ~DeviceGuard() {
    if (prev >= 0) cudaSetDevice(prev);
  }
};

// the stencil bitmap (own element included) and, padded, its union over a brick
int upload_bitmap(ggem_ctx *c, const SpreadGeo &sg) {
  const int B = sg.B;
  std::vector<uint32_t> &bits = c->sp_bits_h;  // (a captured copy reads it when replayed)
  bits.assign(sg.nwords, 0u);
  auto set = [&](int x, int y, int z) {
    const int i = x - sg.lo[0], j = y - sg.lo[1], k = z - sg.lo[2];
    const int idx = sg.pad ? (i + B - 1) + 32 * (j + B - 1) + 1024 * (k + B - 1)
                            : (k * sg.dim[1] + j) * sg.dim[0] + i;
    bits[idx >> 5] |= 1u << (idx & 31);
  };
  set(0, 0, 0);  // the element's own particles come first in its list
  for (const int4 &o : c->stencil) set(o.x, o.y, o.z);
  if (sg.pad) {
    // the particles that some element of a brick lists: bit u is the union of
    // the stencil bits u + (jx, jy, jz), 0 <= j < B (the elements of a brick
    // read the bitmap at u + B - 1 - l); one word per (y, z), x in its bits
    std::vector<uint32_t> x(kSpReachWords, 0u), y(kSpReachWords, 0u), z(kSpReachWords, 0u);
    for (int k = 0; k < sg.nwords; ++k)
      for (int j = 0; j < B; ++j) x[k] |= bits[k] >> j;
    for (int k = 0; k < kSpReachWords; ++k)
      for (int j = 0; j < B && (k & 31) + j < 32; ++j) y[k] |= x[k + j];
    for (int k = 0; k < kSpReachWords; ++k)
      for (int j = 0; j < B && k + 32 * j < kSpReachWords; ++j) z[k] |= y[k + 32 * j];
    bits.insert(bits.end(), z.begin(), z.end());
  }
  cudaError_t e = c->sp_bits.ensure(bits.size());
  if (e) return cuda_fail(c, e, "spread stencil");
  if ((e = cudaMemcpyAsync(c->sp_bits.p, bits.data(), sizeof(uint32_t) * bits.size(),
                           cudaMemcpyHostToDevice, c->stream)))
    return cuda_fail(c, e, "spread stencil");
  c->sp_bits_up = !stream_capturing(c);
  return GGEM_OK;
}

// the stencil bitmap (own element included) and the brick geometry
int spread_geometry(ggem_ctx *c, SpreadGeo *sg) {
  std::memset(sg, 0, sizeof(*sg));
  sg->g = c->grid;
  const Grid &g = c->grid;
  for (int d = 0; d < 3; ++d) sg->lo[d] = sg->hi[d] = 0;
  for (const int4 &o : c->stencil) {
    const int v[3] = {o.x, o.y, o.z};
    for (int d = 0; d < 3; ++d) {
      sg->lo[d] = std::min(sg->lo[d], v[d]);
      sg->hi[d] = std::max(sg->hi[d], v[d]);
    }
  }
  int B = 4;
  for (; B >= 1; B /= 2) {
    bool ok = true;
    int rows = 1, xs = 1;
    for (int d = 0; d < 3; ++d) {
      int ext = B + sg->hi[d] - sg->lo[d];
      if (g.periodic[d] && ext >= g.nc[d]) ext = g.nc[d];
      if (ext > kSpMaxExt) ok = false;
      if (d > 0) rows *= std::min(ext, g.nc[d]);
      else xs = (g.periodic[0] && ext < g.nc[0]) ? 2 : 1;
    }
    if (ok && rows * xs <= kSpMaxSeg) break;
  }
  if (B < 1)
    return fail(c, GGEM_ERR_BAD_ARG,
                "element stencil too wide for the brick spread (more than 28 elements across)");
  sg->B = B;
  for (int d = 0; d < 3; ++d) {
    sg->dim[d] = sg->hi[d] - sg->lo[d] + 1;
    sg->nb[d] = (g.nc[d] + B - 1) / B;
    for (int k = 0; k < kSpMaxExt; ++k) {
      const int off = sg->lo[d] + k;
      sg->shift[d][k] = off <= sg->hi[d] ? (float)(off * g.h[d]) : 0.f;
    }
    sg->L32[d] = (float)g.L[d];
  }
  // the padded layout needs every frame offset field in [0, 32): offsets
  // run over [-(B - 1), dim + B - 2] per axis, so dim + 2B - 2 <= 32; a
  // frame spanning a whole periodic axis wraps its offsets and keeps the
  // compact layout
  bool any_full = false;
  sg->pad = 1;
  for (int d = 0; d < 3; ++d) {
    any_full = any_full || (g.periodic[d] && B + sg->hi[d] - sg->lo[d] >= g.nc[d]);
    if (sg->dim[d] + 2 * B - 2 > 32) sg->pad = 0;
  }
  if (any_full) sg->pad = 0;
  const int nbits = sg->pad ? 1024 * (sg->dim[2] + 2 * B - 2)
                            : sg->dim[0] * sg->dim[1] * sg->dim[2];
  sg->nwords = (nbits + 31) / 32;
  if (sg->nwords > kSpMaxWords)
    return fail(c, GGEM_ERR_BAD_ARG, "element stencil bitmap too large for the brick spread");
  // (the stencil belongs to the context: its bitmap goes up once)
  if (!c->sp_bits_up)
    if (int rc = upload_bitmap(c, *sg)) return rc;
  // e^{-alpha^2 s} = 2^{s k}, k = -alpha^2 log2(e) split into hi + lo floats
  const double k = -c->cst.alpha2 * 1.4426950408889634;
  sg->e_hi = (float)k;
  sg->e_lo = (float)(k - (double)sg->e_hi);
  sg->c25 = (float)(2.5 * c->cst.alpha3_pi_23);
  sg->c1 = (float)(c->cst.alpha2 * c->cst.alpha3_pi_23);
  sg->nq = c->q_per_elem;
  int p2 = 1;
  while (p2 < sg->nq) p2 <<= 1;
  sg->lq = 32 / p2;
  return GGEM_OK;
}

// the separable FP64 spread; *done = false where the points are no tensor
// grid that it takes, or its factors do not fit (the caller sums per pair)
int spread_separable(ggem_ctx *c, const SpreadGeo &sg, bool any_full, const double *d_f_slot,
                     double *d_rho, unsigned long long *d_pairs, bool *done) {
  *done = false;
  if (!c->q_grid) return GGEM_OK;
  SepGeo sp;
  std::memset(&sp, 0, sizeof(sp));
  int at = 0;
  sp.stride = 2;
  for (int d = 0; d < 3; ++d) {
    sp.p[d] = c->q_p[d];
    sp.aoff[d] = at;
    at += sp.p[d] * sg.dim[d];
    sp.stride += sg.B * sp.p[d];
  }
  sp.nfac = at;
  sp.R = sp.p[1] * sp.p[2];
  sp.E = 32 / sp.R;
  std::memcpy(sp.qmap, c->q_map, sizeof(sp.qmap));
  std::memcpy(sp.rep, c->q_rep, sizeof(sp.rep));
  // 80 KB of staged particles: with the tables, two blocks per SM
  sp.cap = (int)std::min<size_t>(256, 80 * 1024 / (sp.stride * sizeof(double2))) / 32 * 32;
  if (sp.cap < 32) return GGEM_OK;
  sp.nw = sp.cap / 32;
  cudaError_t e;
  const size_t nf = (size_t)c->n * sp.nfac;
  if (nf > c->sp_fac.count) {
    size_t avail = 0, all = 0;
    if ((e = cudaMemGetInfo(&avail, &all))) return cuda_fail(c, e, "spread factors");
    if (nf * sizeof(double2) > avail / 4) return GGEM_OK;
  }
  if ((e = c->sp_fac.ensure(nf))) {
    if (e != cudaErrorMemoryAllocation) return cuda_fail(c, e, "spread factors");
    cudaGetLastError();
    return GGEM_OK;
  }
  if (nf) {
    k_axis_factors<<<(unsigned)((nf + 255) / 256), 256, 0, c->stream>>>(
        c->n, sg, sp, c->dc, c->q_xyz.p, c->pos32.p, c->pos64.p,
        c->sp_fac.p);
    if (int rc = check_launch(c, "spread factors")) return rc;
  }
  const size_t smem = (size_t)sp.cap * sp.stride * sizeof(double2) +
                      64 * sp.nw * sizeof(uint32_t) + sp.cap * sizeof(int2) +
                      2 * (kSpMaxSeg + 1) * sizeof(int32_t) + sg.nwords * sizeof(uint32_t);
  const unsigned nblk = (unsigned)((int64_t)sg.nb[0] * sg.nb[1] * sg.nb[2]);
  auto launch = [&](auto kernel) -> int {
    if ((e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  (int)smem)))
      return cuda_fail(c, e, "spread attributes");
    kernel<<<nblk, kSpThreads, smem, c->stream>>>(sg, sp, c->cell_start.p, c->pos32.p, d_f_slot,
                                                  c->sp_fac.p, c->sp_bits.p, d_rho, d_pairs);
    return GGEM_OK;
  };
  int rc;
  switch (sp.p[0]) {
    case 1: rc = any_full ? launch(k_spread_sep<1, true>) : launch(k_spread_sep<1, false>); break;
    case 2: rc = any_full ? launch(k_spread_sep<2, true>) : launch(k_spread_sep<2, false>); break;
    default: rc = any_full ? launch(k_spread_sep<3, true>) : launch(k_spread_sep<3, false>);
  }
  if (rc) return rc;
  *done = true;
  return check_launch(c, "spread bricks (separable)");
}

int spread_elements(ggem_ctx *c, int precision, const double *d_f_slot, double *d_rho,
                    unsigned long long *d_pairs) {
  SpreadGeo sg;
  if (int rc = spread_geometry(c, &sg)) return rc;
  const unsigned nblk = (unsigned)((int64_t)sg.nb[0] * sg.nb[1] * sg.nb[2]);
  cudaError_t e;
  // does any brick frame span a whole periodic axis? (brick_frame: the
  // frame of a brick of at most B elements spans B + hi - lo)
  bool any_full = false;
  for (int d = 0; d < 3; ++d)
    any_full = any_full || (sg.g.periodic[d] && sg.B + sg.hi[d] - sg.lo[d] >= sg.g.nc[d]);
  if (precision == GGEM_FP64) {
    bool done = false;
    if (int rc = spread_separable(c, sg, any_full, d_f_slot, d_rho, d_pairs, &done)) return rc;
    if (done) return GGEM_OK;
  }
  auto launch = [&](auto kernel) -> int {
    // (the attribute is per device; setting it costs microseconds)
    if ((e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  (int)kSpShared)))
      return cuda_fail(c, e, "spread attributes");
    kernel<<<nblk, kSpThreads, kSpShared, c->stream>>>(
        sg, c->dc, c->cell_start.p, c->pos32.p, c->pos64.p, d_f_slot, c->q_rel.p, c->q_xyz.p,
        c->sp_bits.p, d_rho, d_pairs);
    return GGEM_OK;
  };
  int rc;
  if (precision == GGEM_FP64)
    rc = any_full   ? launch(k_spread_brick<false, true, false, 0>)
         : sg.pad   ? launch(k_spread_brick<false, false, true, 0>)
                    : launch(k_spread_brick<false, false, false, 0>);
  else if (sg.lq == 4)
    rc = any_full   ? launch(k_spread_brick<true, true, false, 4>)
         : sg.pad   ? launch(k_spread_brick<true, false, true, 4>)
                    : launch(k_spread_brick<true, false, false, 4>);
  else
    rc = any_full   ? launch(k_spread_brick<true, true, false, 0>)
         : sg.pad   ? launch(k_spread_brick<true, false, true, 0>)
                    : launch(k_spread_brick<true, false, false, 0>);
  if (rc) return rc;
  return check_launch(c, "spread bricks");
}

int quadrature_common(ggem_ctx *c, int nq) {
  if (c->prm.nb_mode != GGEM_NB_REFERENCE)
    return fail(c, GGEM_ERR_BAD_ARG, "the element spread needs reference mode (elements = cells)");
  if (nq < 1 || nq > 32)
    return fail(c, GGEM_ERR_BAD_ARG, "quadrature points per element must be in [1, 32]");
  const int64_t nqt = c->grid.ncell * nq;
  cudaError_t e;
  if ((e = c->q_xyz.ensure(3 * nqt)) || (e = c->q_rel.ensure(nqt)))
    return cuda_fail(c, e, "quadrature buffers");
  c->q_per_elem = 0;
  c->q_grid = false;
  return GGEM_OK;
}

int quadrature_finish(ggem_ctx *c, int nq) {
  const int64_t nqt = c->grid.ncell * nq;
  AxisMap *m = reinterpret_cast<AxisMap *>(c->h_red);
  m->off = 0;
  k_qp_rel<<<(unsigned)((nqt + 255) / 256), 256, 0, c->stream>>>(nqt, nq, c->grid, c->q_xyz.p, m,
                                                                 c->q_rel.p);
  if (int rc = check_launch(c, "quadrature")) return rc;
  if (cudaError_t e = cudaStreamSynchronize(c->stream)) return cuda_fail(c, e, "quadrature");
  c->q_per_elem = nq;
  // a tensor grid of at most 3 points per element along x?
  if (m->off || m->p[0] > 3 || m->p[0] * m->p[1] * m->p[2] != nq) return GGEM_OK;
  for (int k = 0; k < nq; ++k) c->q_map[k] = -1;
  for (int k = 0; k < nq; ++k)
    c->q_map[(m->idx[2][k] * m->p[1] + m->idx[1][k]) * m->p[0] + m->idx[0][k]] = (signed char)k;
  for (int k = 0; k < nq; ++k)
    if (c->q_map[k] < 0) return GGEM_OK;  // a point twice, another missing
  for (int d = 0; d < 3; ++d) c->q_p[d] = m->p[d];
  std::memcpy(c->q_rep, m->rep, sizeof(c->q_rep));
  c->q_grid = true;
  return GGEM_OK;
}

}  // namespace
}  // namespace ggem

using namespace ggem;

extern "C" int ggem_set_quadrature(ggem_ctx *ctx, int nq_per_elem, const double *qxyz) {
  if (!ctx || (!qxyz && ctx->grid.ncell > 0)) return GGEM_ERR_BAD_ARG;
  DeviceGuard dg(ctx->device);
  if (int rc = quadrature_common(ctx, nq_per_elem)) return rc;
  const int64_t nqt = ctx->grid.ncell * nq_per_elem;
  cudaError_t e = cudaMemcpyAsync(ctx->q_xyz.p, qxyz, sizeof(double) * 3 * nqt,
                                  cudaMemcpyHostToDevice, ctx->stream);
  if (e) return cuda_fail(ctx, e, "quadrature h2d");
  return quadrature_finish(ctx, nq_per_elem);
}

extern "C" int ggem_set_quadrature_dev(ggem_ctx *ctx, int nq_per_elem, const double *d_qxyz) {
  if (!ctx || (!d_qxyz && ctx->grid.ncell > 0)) return GGEM_ERR_BAD_ARG;
  DeviceGuard dg(ctx->device);
  if (int rc = quadrature_common(ctx, nq_per_elem)) return rc;
  const int64_t nqt = ctx->grid.ncell * nq_per_elem;
  cudaError_t e = cudaMemcpyAsync(ctx->q_xyz.p, d_qxyz, sizeof(double) * 3 * nqt,
                                  cudaMemcpyDeviceToDevice, ctx->stream);
  if (e) return cuda_fail(ctx, e, "quadrature copy");
  return quadrature_finish(ctx, nq_per_elem);
}

extern "C" int ggem_spread_elements_dev(ggem_ctx *ctx, int precision, const double *d_f,
                                        double *d_rho, int64_t *pairs) {
  if (!ctx || (precision != GGEM_FP32 && precision != GGEM_FP64) || !d_rho ||
      (ctx->n > 0 && !d_f))
    return GGEM_ERR_BAD_ARG;
  if (!ctx->cells_built) return fail(ctx, GGEM_ERR_BAD_ARG, "call ggem_build_cells first");
  if (ctx->q_per_elem < 1) return fail(ctx, GGEM_ERR_BAD_ARG, "call ggem_set_quadrature first");
  DeviceGuard dg(ctx->device);
  const size_t n3 = (size_t)ctx->n * 3;
  cudaError_t e;
  if ((e = ctx->w_in.ensure(std::max<size_t>(n3, 1))) || (e = ctx->sp_pairs.ensure(1)))
    return cuda_fail(ctx, e, "spread buffers");
  if (n3) {
    if (int rc = permute_to_slots(ctx, 1, d_f, ctx->w_in.p)) return rc;
  }
  unsigned long long *d_pairs = nullptr;
  if (pairs) {
    d_pairs = ctx->sp_pairs.p;
    if ((e = cudaMemsetAsync(d_pairs, 0, sizeof(unsigned long long), ctx->stream)))
      return cuda_fail(ctx, e, "memset");
  }
  if (int rc = spread_elements(ctx, precision, ctx->w_in.p, d_rho, d_pairs)) return rc;
  if (pairs) {
    unsigned long long h = 0;
    if ((e = cudaMemcpyAsync(&h, d_pairs, sizeof(h), cudaMemcpyDeviceToHost, ctx->stream)) ||
        (e = cudaStreamSynchronize(ctx->stream)))
      return cuda_fail(ctx, e, "spread pairs");
    *pairs = (int64_t)h;
  }
  return GGEM_OK;
}

extern "C" int ggem_spread_elements(ggem_ctx *ctx, int precision, const double *f, double *rho) {
  if (!ctx || !rho || (ctx->n > 0 && !f)) return GGEM_ERR_BAD_ARG;
  if (ctx->q_per_elem < 1) return fail(ctx, GGEM_ERR_BAD_ARG, "call ggem_set_quadrature first");
  DeviceGuard dg(ctx->device);
  const size_t n3 = (size_t)ctx->n * 3;
  const size_t nr = (size_t)ctx->grid.ncell * ctx->q_per_elem * 3;
  cudaError_t e;
  if ((e = ctx->w_a.ensure(std::max<size_t>(n3, 1))) || (e = ctx->w_d.ensure(std::max<size_t>(nr, 1))))
    return cuda_fail(ctx, e, "spread buffers");
  if (n3 && (e = cudaMemcpyAsync(ctx->w_a.p, f, 8 * n3, cudaMemcpyHostToDevice, ctx->stream)))
    return cuda_fail(ctx, e, "forces h2d");
  if (int rc = ggem_spread_elements_dev(ctx, precision, ctx->w_a.p, ctx->w_d.p, nullptr)) return rc;
  if ((e = cudaMemcpyAsync(rho, ctx->w_d.p, 8 * nr, cudaMemcpyDeviceToHost, ctx->stream)) ||
      (e = cudaStreamSynchronize(ctx->stream)))
    return cuda_fail(ctx, e, "rho d2h");
  return GGEM_OK;
}

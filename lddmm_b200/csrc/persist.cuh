// Persistent multi-step sweep: all T time steps of the forward (shooting) or the
// backward (adjoint) recursion in one cooperative launch.
//
// The steps are sequential (step t + 1 reads the positions / adjoint state step t
// finalised) and, for one registration of a few thousand landmarks, one step is only
// a few microseconds of arithmetic.  Per-step launches then spend most of their time
// ramping CTAs up and down.  Here:
//
//   * every CTA stays resident for the whole recursion; steps are separated by a
//     grid barrier;
//   * the work of a step is the list of 64-row tiles times their j ranges, cut into one
//     share per CTA of equal cost (plan.h): no SM idles at the barrier while another runs a
//     second tile.  A CTA's share is a list of segments (tile, j range);
//   * each warp sums a contiguous part of the segment's j range for all 64 rows
//     (persistent_sweep_kernel); the 8 warps' FP64 sums are added in warp order, and a tile
//     cut over several CTAs stores one FP64 partial per part: the CTA that completes the
//     tile's arrival count (whichever it is) adds the parts in part order and finalises, so
//     results are bit-reproducible for a given plan.
//
// The cluster form (persistent_cluster_kernel) works on row groups of kGroup = 16 rows in
// rounds of two segments (persist_round), the group form (persistent_group_kernel) on one such
// group per CTA, the small form on whole pairs of a few hundred points.
//
// Grid barrier: a monotonically increasing arrival count (fire-and-forget atomic
// add) that the CTAs poll against (step + 1) x grid.  When a launch ends, each CTA
// counts its departure after its last wait; the last one to leave zeroes both counts,
// so the next launch starts from zero without a memset.  Every wait is bounded: after
// kSpinLimit polls the CTA records the step in the error word and leaves the kernel,
// so a launch that is not fully co-resident ends with an error instead of hanging (the
// host then clears the words).  The launch uses the cooperative attribute, with which
// the runtime refuses a grid that cannot be co-resident.
#pragma once

#include "common.cuh"
#include "layout.h"
#include "sweep.cuh"

namespace lddmm {

constexpr int kGroup = 16;                // rows per work unit of the cluster form
constexpr int kRowPairs = kGroup / 2;     // lanes sharing a j entry (2 rows each)
constexpr int kLaneGroups = 32 / kRowPairs;  // j interleave inside a warp
constexpr int kPersistWarps = 8;          // warps per persistent CTA

struct StepSync {
  unsigned int arrive;  // grid barrier arrivals since the launch began
  unsigned int error;   // nonzero: a barrier wait timed out (1 + step index)
  unsigned int depart;  // CTAs past their last wait (resets arrive at launch end)
  unsigned int pad_;
  // timeline of the cooperative kernels of the last cycle (%globaltimer, ns):
  // [slot][0] entry of CTA 0, [slot][1] latest CTA exit; slots: 0 forward sweep,
  // 1 backward sweep, 2 optimiser update
  unsigned long long stamp[4][2];
};

__device__ __forceinline__ unsigned long long global_ns() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

__device__ __forceinline__ void stamp_entry(StepSync *sy, int slot) {
  if (blockIdx.x == 0 && threadIdx.x == 0) sy->stamp[slot][0] = global_ns();
}

__device__ __forceinline__ void stamp_exit(StepSync *sy, int slot) {
  if (threadIdx.x == 0) atomicMax(&sy->stamp[slot][1], global_ns());
}

constexpr unsigned int kSpinLimit = 1u << 23;  // polls: a few seconds at most

__device__ __forceinline__ unsigned int ld_acquire(const unsigned int *p) {
  unsigned int v;
  asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}

// Arrival count with release semantics (orders this thread's writes, and those of
// threads synchronised with it, before the increment) and no return value.
__device__ __forceinline__ void red_add_release_gpu(unsigned int *p, unsigned int v) {
  asm volatile("red.release.gpu.global.add.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}

// Atomic add at GPU scope with release and acquire semantics; returns the old value.
__device__ __forceinline__ unsigned int atom_add_acq_rel_gpu(unsigned int *p, unsigned int v) {
  unsigned int old;
  asm volatile("atom.acq_rel.gpu.global.add.u32 %0, [%1], %2;" : "=r"(old) : "l"(p), "r"(v)
               : "memory");
  return old;
}

__device__ __forceinline__ unsigned int ld_relaxed(const unsigned int *p) {
  unsigned int v;
  asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}

// Waits until `target` arrivals (this CTA's included) have been counted.  Returns
// false when the wait timed out (the caller must leave the kernel without departing).
// `tag` identifies the wait in the error word.  The arrival is a release reduction
// (the CTA's writes, ordered before it by __syncthreads, become visible with it); the
// poll is one acquire load per iteration (the error word is read every 64th), so the
// load that sees the count complete also orders the CTA's later reads after the
// arrivals, with no further round trip to L2.
__device__ __forceinline__ bool grid_barrier(StepSync *sy, unsigned int target,
                                             unsigned int tag,
                                             unsigned int spin = kSpinLimit) {
  __shared__ int s_ok;
  __syncthreads();
  if (threadIdx.x == 0) {
    int ok = 1;
    red_add_release_gpu(&sy->arrive, 1u);
    unsigned int n = 0;
    while (ld_acquire(&sy->arrive) < target) {
      if ((++n & 63u) == 0u) {
        if (ld_relaxed(&sy->error) != 0u || n > spin) {
          atomicCAS(&sy->error, 0u, 1u + tag);
          ok = 0;
          break;
        }
        if (n > 4096u) __nanosleep(64);
      }
    }
    // the acquire load that read the complete count read the end of the release
    // sequence of every CTA's arrival (each arrival is a read-modify-write), so their
    // writes are visible to this thread, and through the __syncthreads to the CTA
    s_ok = ok;
  }
  __syncthreads();
  return s_ok != 0;
}

// After a CTA's last grid_barrier: the last CTA to depart zeroes the counts.  Every
// CTA has stopped polling `arrive` by then.
__device__ __forceinline__ void grid_depart(StepSync *sy) {
  if (threadIdx.x == 0) {
    const unsigned int old = atomicAdd(&sy->depart, 1u);
    if (old == gridDim.x - 1) {
      sy->arrive = 0u;
      sy->depart = 0u;
    }
  }
}

// Work plan of the persistent sweeps (built on the host when the context is created).
struct SweepPlan {
  const int2 *units;      // (pair, 64-row tile) per unit
  const int4 *segs;       // (unit, j begin, j end, part) in CTA order
  const int *cta_seg;     // CTA k owns segs[cta_seg[k] .. cta_seg[k + 1])
  const int2 *unit_parts; // (parts, first partial slot) per unit
  double *part;           // FP64 partials [slot][kPartNA][kTile]
  unsigned int *cnt;      // per-unit arrival count of split tiles (self-resetting)
};

constexpr int kPartNA = 6;  // accumulators per row in a partial slot (>= every Op::NA)

// One round of a persistent CTA: the entries of its (one or two) segments, laid end
// to end, cut into NW equal contiguous warp shares (a share that straddles the two
// segments is processed as two pieces); every warp leaves its FP64 row sums of
// segment g in s_red[g][warp] (zeros where it has no entries of g).  `o` has the step
// set; o.pd is redirected to the round's descriptors in shared memory.
template <class Op>
__device__ __forceinline__ void persist_round(
    Op &o, int nseg, const int4 *s_seg, const int (*s_uinf)[2], const PairDesc *s_pd,
    float4 (*s_j)[Op::JW][kSub], double (*s_red)[kPersistWarps][kGroup][Op::NA]) {
  constexpr int JW = Op::JW;
  constexpr int NA = Op::NA;
  constexpr int NW = kPersistWarps;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int lrow = lane % kRowPairs, lg = lane / kRowPairs;
  const int la = s_seg[0].z - s_seg[0].y, lb = nseg > 1 ? s_seg[1].z - s_seg[1].y : 0;
  const int wb = (int)((long long)(la + lb) * warp / NW);
  const int we = (int)((long long)(la + lb) * (warp + 1) / NW);
#pragma unroll 1
  for (int g = 0; g < nseg; ++g) {
    const int off = g ? la : 0, len = g ? lb : la;
    const int lo = max(wb, off), hi = min(we, off + len);
    if (hi <= lo || !s_uinf[g][1]) {
      // no entries of this segment: a zero contribution to its warp-order sum
      if (lane < kGroup) {
#pragma unroll
        for (int a = 0; a < NA; ++a) s_red[g][warp][lane][a] = 0.0;
      }
      continue;
    }
    const int4 sg = s_seg[g];
    const int grp = s_uinf[g][0] >> 16;
    o.pd = &s_pd[g];  // the op reads descriptor 0 from shared memory from here on
    const int p = 0;
    typename Op::IData I0, I1;
    o.load_i(p, grp * kGroup + lrow, I0);
    o.load_i(p, grp * kGroup + kRowPairs + lrow, I1);
    float hi0[NA], lo0[NA], hi1[NA], lo1[NA];
#pragma unroll
    for (int a = 0; a < NA; ++a) hi0[a] = lo0[a] = hi1[a] = lo1[a] = 0.0f;
    const int jb = sg.y + (lo - off);
    const int je = sg.y + (hi - off);
    const int split = Op::kTwoSets ? o.set_boundary(p) : sg.z;
    float4 nxt[JW];
    float acc0[NA], acc1[NA];
    if (jb + lane < je) o.load_j(p, jb + lane, nxt);
    for (int j0 = jb; j0 < je; j0 += kSub) {
      __syncwarp();
#pragma unroll
      for (int x = 0; x < JW; ++x) s_j[warp][x][lane] = nxt[x];
      __syncwarp();
      const int cnt = min(kSub, je - j0);
      const int jn = j0 + kSub;
      if (jn + lane < je) o.load_j(p, jn + lane, nxt);
      const bool fresh = ((j0 - jb) & (4 * kSub - 1)) == 0;
      if (fresh) {
#pragma unroll
        for (int a = 0; a < NA; ++a) acc0[a] = acc1[a] = 0.0f;
      }
      const int b = Op::kTwoSets ? min(max(split - j0, 0), cnt) : cnt;
#pragma unroll 4
      for (int jj = lg; jj < b; jj += kLaneGroups) {
        float4 w[JW];
#pragma unroll
        for (int x = 0; x < JW; ++x) w[x] = s_j[warp][x][jj];
        o.template pair<0>(I0, w, acc0);
        o.template pair<0>(I1, w, acc1);
      }
      if (Op::kTwoSets) {
        // first entry >= b that belongs to this lane group
        const int b1 = b + ((lg - b) % kLaneGroups + kLaneGroups) % kLaneGroups;
#pragma unroll 4
        for (int jj = b1; jj < cnt; jj += kLaneGroups) {
          float4 w[JW];
#pragma unroll
          for (int x = 0; x < JW; ++x) w[x] = s_j[warp][x][jj];
          o.template pair<1>(I0, w, acc0);
          o.template pair<1>(I1, w, acc1);
        }
      }
      // fold into the compensated sum every 4 sub-tiles (<= 32 plain FP32 terms
      // per lane) and after the last one
      if (((j0 - jb) & (4 * kSub - 1)) == 3 * kSub || j0 + kSub >= je) {
#pragma unroll
        for (int a = 0; a < NA; ++a) {
          two_sum_acc(hi0[a], lo0[a], acc0[a]);
          two_sum_acc(hi1[a], lo1[a], acc1[a]);
        }
      }
    }
    // lane groups -> lanes 0..7 (fixed butterfly)
#pragma unroll
    for (int a = 0; a < NA; ++a) {
      double v0 = (double)hi0[a] + (double)lo0[a];
      double v1 = (double)hi1[a] + (double)lo1[a];
#pragma unroll
      for (int off2 = kRowPairs; off2 < 32; off2 <<= 1) {
        v0 += __shfl_xor_sync(0xffffffffu, v0, off2);
        v1 += __shfl_xor_sync(0xffffffffu, v1, off2);
      }
      if (lg == 0) {
        s_red[g][warp][lrow][a] = v0;
        s_red[g][warp][kRowPairs + lrow][a] = v1;
      }
    }
  }
}

// Loads the descriptors of the round starting at segment k (nseg segments) into the
// round slots.  Called by the whole CTA.
template <class Op>
__device__ __forceinline__ void persist_load_round(const Op &op, const int4 *segs,
                                                   const int2 *units, int k, int nseg,
                                                   int4 *s_seg, int (*s_uinf)[2],
                                                   PairDesc *s_pd) {
  __syncthreads();  // the previous round's epilogue is done with the round slots
  if (threadIdx.x < nseg) {
    const int4 sg = segs[k + threadIdx.x];
    const int2 un = units[sg.x];
    s_seg[threadIdx.x] = sg;
    s_uinf[threadIdx.x][0] = un.x | (un.y << 16);
    s_uinf[threadIdx.x][1] = op.active(un.x);
    s_pd[threadIdx.x] = op.pd[un.x];
  }
  __syncthreads();
}

__device__ __forceinline__ void cluster_sync_all() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n\t"
               "barrier.cluster.wait.acquire.aligned;" ::: "memory");
}

// Op: the sweep interface of sweep.cuh plus set_step(t) (pointers of time step t) and
// write_group(p, k, v) (row-group partial of a kTileSum op).
// dir = +1 runs t = 0..T-1, dir = -1 runs t = T-1..0.
// Two CTAs per SM (<= 128 registers), 16 warps per SM.
// Rows are taken 64 at a time (kTile), four per lane: lanes l and l + 16 hold the same rows
// and take the even and the odd j points of a staged 32-point sub-tile, so that one staged
// point serves four pairs per lane (with two, the 128 bytes per clock that shared memory
// returns bound the loop, not the arithmetic).  A segment's j range is cut into 8 warp
// shares; a warp keeps at most 32 plain FP32 terms per sum before it adds them to its FP64
// sums in shared memory.  Bound at 2562 points by the chain around the pair loop (first loads,
// combine of about 7 parts per tile, grid barrier: about half of the step), beyond by FP32
// issue.  Us per step (3D Matern of order 1), 16-row groups cut over CTAs and 4 lane groups ->
// this: 642 points shooting 4.7 -> 4.5, adjoint 6.6 -> 5.6; 1200 points 5.8 -> 5.1, 8.9 -> 6.5;
// 2562 points 10.5 -> 8.6, 15.1 -> 12.3; 5000 points 26.1 -> 20.4, 41.2 -> 31.9.
struct SegDesc {
  int4 seg;      // unit, j begin, j end, part
  int row0, active;
  int2 up;       // parts, first partial slot
  PairDesc pd;
};

template <class Op>
__global__ void __launch_bounds__(kPersistWarps * 32, 2)
    persistent_sweep_kernel(Op op, SweepPlan plan, int T, int dir, StepSync *sy) {
  constexpr int JW = Op::JW, NA = Op::NA;
  constexpr int NW = kPersistWarps, NT = NW * 32, NS = NA * kTile;
  static_assert(NA <= kPartNA && !Op::kTwoSets && kTile == 64 && NS <= 2 * NT, "shape");
  __shared__ float4 s_j[NW][JW][kSub];
  __shared__ double s_red[NW][NS];
  __shared__ SegDesc s_d[2];
  __shared__ int s_last;
  pdl_wait();
  stamp_entry(sy, dir > 0 ? 0 : 1);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int l16 = lane & 15, lg = lane >> 4;
  const int s0 = plan.cta_seg[blockIdx.x], s1 = plan.cta_seg[blockIdx.x + 1];
  // descriptors of segment k: read once for the whole launch when the CTA has at most two
  // (a grid barrier's acquire empties L1, and the reads depend on one another)
  auto describe = [&](int k, SegDesc &d) {
    const int4 sg = plan.segs[k];
    const int2 un = plan.units[sg.x];
    d.seg = sg;
    d.row0 = un.y * kTile;
    d.active = op.active(un.x);
    d.up = plan.unit_parts[sg.x];
    d.pd = op.pd[un.x];
  };
  const bool once = s1 - s0 <= 2;
  if (once) {
    if (tid < s1 - s0) describe(s0 + tid, s_d[tid]);
    __syncthreads();
  }
  for (int s = 0; s < T; ++s) {
    Op o = op;
    o.set_step(dir > 0 ? s : T - 1 - s);
    for (int k = s0; k < s1; ++k) {
      if (k > s0) __syncthreads();  // the segment before is done with shared memory
      if (!once) {
        if (tid == 0) describe(k, s_d[0]);
        __syncthreads();
      }
      const SegDesc &d = s_d[once ? k - s0 : 0];
      if (!d.active) continue;  // uniform over the CTA
      o.pd = &d.pd;             // the op reads descriptor 0 from shared memory
      const int row0 = d.row0;
      {
        const int jb0 = d.seg.y, len = d.seg.z - jb0, chunk = (len + 2 * NW - 1) / (2 * NW) * 2;
        const int jb = jb0 + min(len, chunk * warp), je = jb0 + min(len, chunk * (warp + 1));
        float4 nxt[JW];
        if (jb + lane < je) o.load_j(0, jb + lane, nxt);
        typename Op::IData I[4];  // rows l16 + 16 r
#pragma unroll
        for (int r = 0; r < 4; ++r) o.load_i(0, row0 + 16 * r + l16, I[r]);
        bool first = true;
#pragma unroll 1
        for (int c0 = jb; c0 < je || first; c0 += 2 * kSub) {
          float acc[4][NA];
#pragma unroll
          for (int r = 0; r < 4; ++r)
#pragma unroll
            for (int a = 0; a < NA; ++a) acc[r][a] = 0.0f;
          const int ce = min(je, c0 + 2 * kSub);
#pragma unroll 1
          for (int j0 = c0; j0 < ce; j0 += kSub) {
            __syncwarp();
#pragma unroll
            for (int x = 0; x < JW; ++x) s_j[warp][x][lane] = nxt[x];
            __syncwarp();
            const int cnt = min(kSub, je - j0);
            if (j0 + kSub + lane < je) o.load_j(0, j0 + kSub + lane, nxt);
#pragma unroll Op::kUnroll
            for (int jj = lg; jj < cnt; jj += 2) {
              float4 w[JW];
#pragma unroll
              for (int x = 0; x < JW; ++x) w[x] = s_j[warp][x][jj];
#pragma unroll
              for (int r = 0; r < 4; ++r) o.template pair<0>(I[r], w, acc[r]);
            }
          }
          // the two lane halves: each keeps two of its rows and receives the other's sums
#pragma unroll
          for (int r = 0; r < 2; ++r)
#pragma unroll
            for (int a = 0; a < NA; ++a) {
              const float keep = lg ? acc[2 + r][a] : acc[r][a],
                          give = lg ? acc[r][a] : acc[2 + r][a];
              double x = (double)keep + (double)__shfl_xor_sync(0xffffffffu, give, 16);
              double *y = &s_red[warp][a * kTile + 32 * lg + 16 * r + l16];
              if (!first) x += *y;
              *y = x;
            }
          first = false;
        }
      }
      typename Op::FData F;  // finalize operands, in flight during the combine
      if (tid < kTile) o.fin_load(0, row0 + tid, F);
      __syncthreads();
      // the 8 warps in warp order; thread i takes sums i and i + 256
      const int parts = d.up.x;
      double *part = plan.part + (size_t)d.up.y * kTile * kPartNA;
      double x[2] = {0.0, 0.0};
#pragma unroll
      for (int w = 0; w < NW; ++w)
#pragma unroll
        for (int h = 0; h < 2; ++h)
          if (tid + h * NT < NS) x[h] += s_red[w][tid + h * NT];
      bool fin = true;
      if (parts > 1) {
        // tile cut over several CTAs: the CTA that completes the count adds all parts in
        // part order
#pragma unroll
        for (int h = 0; h < 2; ++h)
          if (tid + h * NT < NS) part[(size_t)d.seg.w * kTile * kPartNA + tid + h * NT] = x[h];
        __syncthreads();  // the parts are written before thread 0's release
        if (tid == 0) {
          unsigned int *cnt = &plan.cnt[d.seg.x];
          s_last = atom_add_acq_rel_gpu(cnt, 1u) == (unsigned int)parts - 1u;
          if (s_last) *cnt = 0u;  // next step's arrivals come after the barrier
        }
        __syncthreads();
        fin = s_last != 0;
        if (fin) {
          x[0] = x[1] = 0.0;
          for (int q0 = 0; q0 < parts; q0 += 10) {  // 10 parts' loads in flight at once
            double y[2][10];
#pragma unroll
            for (int q = 0; q < 10; ++q)
#pragma unroll
              for (int h = 0; h < 2; ++h)
                y[h][q] = q0 + q < parts && tid + h * NT < NS
                              ? __ldcg(part + (size_t)(q0 + q) * kTile * kPartNA + tid + h * NT)
                              : 0.0;
#pragma unroll
            for (int q = 0; q < 10; ++q)
#pragma unroll
              for (int h = 0; h < 2; ++h) x[h] += y[h][q];
          }
        }
      }
      if (fin) {
#pragma unroll
        for (int h = 0; h < 2; ++h)  // (sum i of warp 0 was read by this thread alone)
          if (tid + h * NT < NS) s_red[0][tid + h * NT] = x[h];
        __syncthreads();
        if (tid < kTile) {
          double v[NA];
#pragma unroll
          for (int a = 0; a < NA; ++a) v[a] = s_red[0][a * kTile + tid];
          double en = o.finalize(0, row0 + tid, v, F);
          if (Op::kTileSum) {
            // energy partials in the places of the tile's 16-row groups
#pragma unroll
            for (int off = 16; off > 0; off >>= 1) en += __shfl_xor_sync(0xffffffffu, en, off);
            if (lane < 2) o.write_group(0, row0 / kGroup + 2 * warp + lane, lane ? 0.0 : en);
          }
        }
      }
    }
    if (!grid_barrier(sy, (unsigned)(s + 1) * gridDim.x, (unsigned)s)) return;
  }
  grid_depart(sy);
  stamp_exit(sy, dir > 0 ? 0 : 1);
  pdl_trigger();
}

// ---------------------------------------------------------------------------------
// Group form: one whole 16-row group per CTA, no group cut, so that a step ends with the
// warps' sums, the finalisation and the grid barrier.  For a few hundred to a few thousand
// points of a cheap kernel, where a step is its latency and the combine of the 64-row tiles'
// parts a third of it: 2D Gaussian, us per shooting / adjoint step, 64-row tiles -> this: 400
// points 4.25 / 4.40 -> 3.16 / 3.80, 640 points 4.28 / 4.48 -> 3.53 / 4.21, 8 pairs of 500
// 4.97 / 5.73 -> 3.89 / 5.05.
// Beyond one group per resident CTA, or with a costlier pair, the tiles are faster (2D Matern
// at 500 points: 5.8 / 6.2 us on tiles, 9.9 / 10.4 in whole groups).

template <class Op>
__global__ void __launch_bounds__(kPersistWarps * 32, 2)
    persistent_group_kernel(Op op, const int2 *units, int T, int dir, StepSync *sy) {
  constexpr int JW = Op::JW, NA = Op::NA, NW = kPersistWarps;
  __shared__ float4 s_j[NW][JW][kSub];
  __shared__ double s_red[1][NW][kGroup][NA];
  __shared__ PairDesc s_pd[1];
  __shared__ int s_uinf[1][2];
  __shared__ int4 s_seg[1];
  pdl_wait();
  stamp_entry(sy, dir > 0 ? 0 : 1);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int2 un = units[blockIdx.x];
  if (threadIdx.x == 0) {
    s_uinf[0][0] = un.x | (un.y << 16);
    s_uinf[0][1] = op.active(un.x);
    s_pd[0] = op.pd[un.x];
    s_seg[0] = make_int4(0, 0, op.pd[un.x].Npad, 0);
  }
  __syncthreads();
  const int row = un.y * kGroup + lane;
  for (int s = 0; s < T; ++s) {
    Op o = op;
    o.set_step(dir > 0 ? s : T - 1 - s);
    persist_round(o, 1, s_seg, s_uinf, s_pd, s_j, s_red);
    o.pd = s_pd;
    const bool fin = warp == 0 && lane < kGroup && s_uinf[0][1];
    typename Op::FData F;  // finalize operands, in flight during the barrier
    if (fin) o.fin_load(0, row, F);
    __syncthreads();
    if (fin) {
      double v[NA];
#pragma unroll
      for (int a = 0; a < NA; ++a) {
        double x = 0.0;
#pragma unroll
        for (int w = 0; w < NW; ++w) x += s_red[0][w][lane][a];
        v[a] = x;
      }
      double en = o.finalize(0, row, v, F);
      if (Op::kTileSum) {
#pragma unroll
        for (int off = kGroup / 2; off > 0; off >>= 1)
          en += __shfl_xor_sync(0xffffu, en, off);
        if (lane == 0) o.write_group(0, un.y, en);
      }
    }
    if (!grid_barrier(sy, (unsigned)(s + 1) * gridDim.x, (unsigned)s)) return;
  }
  grid_depart(sy);
  stamp_exit(sy, dir > 0 ? 0 : 1);
  pdl_trigger();
}

// ---------------------------------------------------------------------------------
// Cluster form of the persistent sweep.  The same rounds and pair arithmetic, but a
// row group is never cut across thread-block clusters: the host plan gives each
// cluster of C CTAs a contiguous range of whole row groups (balanced by work), and
// cuts only inside a cluster.  The parts of a row group split between CTAs of one
// cluster meet in distributed shared memory instead of L2:
//   * a CTA keeps the FP64 partial of a split segment in one of two shared slots (its
//     share's first and last segment are the only ones that can be split);
//   * after its rounds every CTA arrives (release, cluster scope) on the mbarrier of
//     every CTA of its cluster;
//   * the CTA holding a split row group's first part (its "job", at most one per CTA)
//     polls its mbarrier's phase (non-blocking test, acquire; bounded), reads the
//     parts from the owners' slots in part order and finalises the row group.
// A step's slots are rewritten only after the grid barrier, which every CTA reaches
// after its reads.  No L2 round trip, fence at GPU scope or arrival count remains
// between the pair arithmetic and the grid barrier.  All mbarrier waits are bounded
// (timeout: the error word, as for the grid barrier); the only unbounded waits are
// the hardware cluster barriers at entry (mbarriers initialised before any remote
// arrival) and exit (no CTA leaves while a peer may still read its slots), which
// every CTA executes exactly once on every path.

constexpr int kMaxJobParts = 8;  // parts of a row group: at most the cluster size

struct ClusterSweepPlan {
  const int2 *units;    // (pair, row group) per unit
  const int4 *segs;     // (unit, j begin, j end, kind) in CTA order; kind 0: a whole row
                        // group (finalised by its CTA), 1 / 2: a part kept in slot 0 / 1
  const int *cta_seg;   // CTA k owns segs[cta_seg[k] .. cta_seg[k + 1])
  const int2 *job;      // per CTA: (unit whose first part it holds, or -1; parts)
  const int *job_src;   // per CTA, kMaxJobParts entries: cluster rank << 1 | slot of part q
};

__device__ __forceinline__ unsigned int cluster_nctas() {
  unsigned int n;
  asm volatile("mov.u32 %0, %%cluster_nctarank;" : "=r"(n));
  return n;
}

__device__ __forceinline__ void mbar_init(unsigned long long *bar, unsigned int count) {
  const unsigned int a = (unsigned int)__cvta_generic_to_shared(bar);
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(a), "r"(count) : "memory");
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}

// Arrival on the mbarrier at the same shared address in cluster CTA `rank`.
__device__ __forceinline__ void mbar_arrive_cluster(unsigned long long *bar, unsigned int rank) {
  const unsigned int a = (unsigned int)__cvta_generic_to_shared(bar);
  unsigned int ra;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(ra) : "r"(a), "r"(rank));
  asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(ra)
               : "memory");
}

// Non-blocking test of the completion of the mbarrier phase with the given parity.
__device__ __forceinline__ bool mbar_test_parity(unsigned long long *bar, unsigned int parity) {
  const unsigned int a = (unsigned int)__cvta_generic_to_shared(bar);
  unsigned int ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.test_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(a), "r"(parity)
      : "memory");
  return ok != 0u;
}

template <class Op>
__global__ void __launch_bounds__(kPersistWarps * 32, 2)
    persistent_cluster_kernel(Op op, ClusterSweepPlan plan, int T, int dir, StepSync *sy) {
  constexpr int JW = Op::JW;
  constexpr int NA = Op::NA;
  constexpr int NW = kPersistWarps;
  __shared__ float4 s_j[NW][JW][kSub];
  __shared__ double s_red[2][NW][kGroup][NA];
  __shared__ double s_slot[2][kGroup][NA];  // partials of this CTA's split segments
  __shared__ PairDesc s_pd[2];
  __shared__ int s_uinf[2][2];
  __shared__ int4 s_seg[2];
  __shared__ __align__(8) unsigned long long s_bar;
  pdl_wait();
  stamp_entry(sy, dir > 0 ? 0 : 1);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (threadIdx.x == 0) mbar_init(&s_bar, cluster_nctas());
  cluster_sync_all();  // every mbarrier initialised before the first remote arrival
  const int s0 = plan.cta_seg[blockIdx.x], s1 = plan.cta_seg[blockIdx.x + 1];
  const bool one_round = s1 - s0 <= 2;
  for (int s = 0; s < T; ++s) {
    const int t = dir > 0 ? s : T - 1 - s;
    Op o = op;
    o.set_step(t);
    for (int k = s0; k < s1; k += 2) {
      const int nseg = min(2, s1 - k);
      if (!one_round || s == 0)
        persist_load_round(op, plan.segs, plan.units, k, nseg, s_seg, s_uinf, s_pd);
      persist_round(o, nseg, s_seg, s_uinf, s_pd, s_j, s_red);
      __syncthreads();
      // epilogue: segment e on lanes 0-15 of warp e; a whole row group is finalised
      // here, a part goes to its slot
      const int e = warp;
      if (e < nseg && lane < kGroup && s_uinf[e][1]) {
        const int4 se = s_seg[e];
        const int grp_e = s_uinf[e][0] >> 16;
        Op oe = o;
        oe.pd = &s_pd[e];
        double v[NA];
#pragma unroll
        for (int a = 0; a < NA; ++a) {
          double x = 0.0;
#pragma unroll
          for (int w = 0; w < NW; ++w) x += s_red[e][w][lane][a];
          v[a] = x;
        }
        if (se.w == 0) {
          double en = oe.finalize(0, grp_e * kGroup + lane, v);
          if (Op::kTileSum) {
#pragma unroll
            for (int off = kGroup / 2; off > 0; off >>= 1)
              en += __shfl_xor_sync(0xffffu, en, off);
            if (lane == 0) oe.write_group(0, grp_e, en);
          }
        } else {
#pragma unroll
          for (int a = 0; a < NA; ++a) s_slot[se.w - 1][lane][a] = v[a];
        }
      }
    }
    __syncthreads();  // this CTA's slots are written
    if (threadIdx.x < cluster_nctas()) {
      asm volatile("fence.acq_rel.cluster;" ::: "memory");
      mbar_arrive_cluster(&s_bar, threadIdx.x);
    }
    // the job (if any) is re-read here rather than kept in registers through the rounds
    const int2 job = warp == 0 ? plan.job[blockIdx.x] : make_int2(-1, 0);
    if (job.x >= 0) {
      // the parts of the split row group whose first part this CTA holds
      const int2 un = plan.units[job.x];
      const int job_pair = un.x, job_grp = un.y, row = job_grp * kGroup + lane;
      Op &oj = o;
      oj.pd = op.pd;  // global descriptors (the rounds pointed o.pd at the round slots)
      typename Op::FData F;  // finalize operands, in flight during the wait
      if (lane < kGroup) oj.fin_load(job_pair, row, F);
      unsigned int n = 0;
      bool ok = true;
      while (!mbar_test_parity(&s_bar, (unsigned int)(s & 1))) {
        if ((++n & 63u) == 0u) {
          if (ld_relaxed(&sy->error) != 0u || n > kSpinLimit) {
            atomicCAS(&sy->error, 0u, 3000u + (unsigned int)s);
            ok = false;
            break;
          }
          if (n > 4096u) __nanosleep(64);
        }
      }
      ok = __all_sync(0xffffffffu, ok);
      if (ok && lane < kGroup && oj.active(job_pair)) {
        double v[NA];
#pragma unroll
        for (int a = 0; a < NA; ++a) v[a] = 0.0;
        for (int q = 0; q < job.y; ++q) {
          const int src = plan.job_src[blockIdx.x * kMaxJobParts + q];
          const double *rem =
              cg::this_cluster().map_shared_rank(&s_slot[src & 1][lane][0], src >> 1);
#pragma unroll
          for (int a = 0; a < NA; ++a) v[a] += rem[a];
        }
        double en = oj.finalize(job_pair, row, v, F);
        if (Op::kTileSum) {
#pragma unroll
          for (int off = kGroup / 2; off > 0; off >>= 1)
            en += __shfl_xor_sync(0xffffu, en, off);
          if (lane == 0) oj.write_group(job_pair, job_grp, en);
        }
      }
    }
    if (!grid_barrier(sy, (unsigned)(s + 1) * gridDim.x, (unsigned)s)) break;
  }
  cluster_sync_all();  // no CTA leaves while a peer may still read its slots
  grid_depart(sy);
  stamp_exit(sy, dir > 0 ? 0 : 1);
  pdl_trigger();
}

// ---------------------------------------------------------------------------------
// Small form of the persistent sweeps, for pairs of at most 512 (padded) points: one
// thread-block cluster per pair.  Every CTA holds all points' raw operands in shared
// memory (two buffers, by step parity) and owns a range of rows, 16 lanes per row; a
// finalised row's new operands go straight into every CTA's buffer of the next step
// (distributed shared memory), and the hardware cluster barrier ends the step: no operand
// of the recursion passes through L2 between steps, and there is no atomic to poll.
// The row's FP64 state stays in registers, a step's global results are stored after its
// barrier (whose release would wait for them), and operands that do not depend on the step
// before (a; q and r in the adjoint) are loaded two steps ahead.  The cluster barrier waits without a bound, but a cluster is co-resident
// by definition and every CTA of it reaches every barrier.
// Bound by the step's own latency (a chain of shared loads, exponential, shuffles, FP64
// finalise and cluster barrier); 16 lanes per row is the most that a block of 512 threads
// gives 512 points in 16 CTAs.  200 points (2D, Gaussian), us per step against 16-row groups
// combined through L2: shooting 3.30 -> 2.42, adjoint 3.66 -> 2.76.  500 points (2D, Matern of
// order 3) are bound by the Bessel functions instead: an evaluation takes 350 us with this
// form and 303 on the 64-row tiles, which autotuning then picks.

constexpr int kSmallMax = 512;      // padded points of a pair; threads per CTA
constexpr int kSmallCtas = 16;      // CTAs per cluster
constexpr int kSmallLanes = 16;     // lanes per row

template <class Op>
__host__ __device__ constexpr size_t small_smem(int npad) {
  return sizeof(float4) * 2 * Op::NRAW * npad;
}

template <class Op>
__global__ void __launch_bounds__(kSmallMax, 1)
    small_sweep_kernel(Op op, int C, int npmax, int T, int dir, StepSync *sy) {
  constexpr int NA = Op::NA, NR = Op::NRAW, ND = Op::RAW_DYN, L = kSmallLanes;
  static_assert(Op::RAW_DYN0 == 0, "dynamic operands first");
  extern __shared__ __align__(16) unsigned char s_raw[];
  float4 *sj = reinterpret_cast<float4 *>(s_raw);  // [buffer][operand][point]
  __shared__ double s_e[2][kSmallMax / L];
  pdl_wait();
  stamp_entry(sy, dir > 0 ? 0 : 1);
  const int p = blockIdx.x / C, rank = blockIdx.x - p * C;
  if (!op.active(p)) return;  // uniform over the cluster
  const int tid = threadIdx.x, sub = tid % L, nth = blockDim.x;
  const PairDesc P = op.pd[p];
  const int N = P.N, npad = P.Npad, ngrp = npad / kGroup;
  const int R = (N + C - 1) / C, r0 = rank * R;  // this CTA's rows
  const int rows = max(0, min(R, N - r0)), lrow = tid / L;
  const bool mine = lrow < rows, owner = mine && sub == 0;
  const int row = r0 + lrow;
  auto step_of = [&](int s) { return dir > 0 ? s : T - 1 - s; };
  Op o = op;
  float4 st[2][NR - ND];  // independent operands of points tid and tid + nth (npad <= 2 nth)
  auto fetch = [&](int s) {
    o.set_step(step_of(s));
#pragma unroll
    for (int k = ND; k < NR; ++k) {
      if (tid < npad) o.load_raw(p, tid, k, st[0][k - ND]);
      if (tid + nth < npad) o.load_raw(p, tid + nth, k, st[1][k - ND]);
    }
  };
  auto put = [&](float4 *buf) {
#pragma unroll
    for (int k = ND; k < NR; ++k) {
      if (tid < npad) buf[k * npmax + tid] = st[0][k - ND];
      if (tid + nth < npad) buf[k * npmax + tid + nth] = st[1][k - ND];
    }
  };
  fetch(0);
  for (int j = tid; j < npad; j += nth)
#pragma unroll
    for (int k = 0; k < ND; ++k) {
      float4 x;
      o.load_raw(p, j, k, x);
      sj[k * npmax + j] = x;
      // padding keeps its (zero) operands in both buffers
      if (j >= N) sj[(NR + k) * npmax + j] = x;
    }
  put(sj);
  typename Op::Small S;
  double a[3] = {0.0, 0.0, 0.0}, an[3] = {0.0, 0.0, 0.0};
  if (mine) {
    o.small_init(p, row, S);
    o.small_a(p, row, a);
  }
  if (T > 1) fetch(1);
  float4 nx[ND];
#pragma unroll
  for (int k = 0; k < ND; ++k) nx[k] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
  // results of the step before: its energy partial in the place of one of the pair's
  // 16-row groups (one per CTA), and the rows' stores
  auto flush = [&](int s) {
    o.set_step(step_of(s));
    if (owner) o.small_flush(P, row, S, nx, s == T - 1);
    if (Op::kTileSum && tid == 0) {
      double e = 0.0;
      for (int k = 0; k < rows; ++k) e += s_e[s & 1][k];
      o.write_group(p, rank, e);
      if (rank == 0)
        for (int k = C; k < ngrp; ++k) o.write_group(p, k, 0.0);
    }
  };
  cluster_sync_all();  // every CTA of the cluster runs before the first remote store
  for (int s = 0; s < T; ++s) {
    const int cur = s & 1;
    const float4 *c = sj + (size_t)cur * NR * npmax;
    float4 *nxt = sj + (size_t)(cur ^ 1) * NR * npmax;
    if (s > 0) flush(s - 1);
    if (s + 1 < T) {
      put(nxt);
      o.set_step(step_of(s + 1));
      if (mine) o.small_a(p, row, an);
      if (s + 2 < T) fetch(s + 2);
    }
    double v[NA];
    {
      typename Op::IData I;
      float4 x[NR];
#pragma unroll
      for (int k = 0; k < NR; ++k) x[k] = c[k * npmax + (mine ? row : 0)];
      Op::raw_i(x, I);
      float acc[NA];  // npad / 16 <= 32 plain FP32 terms
#pragma unroll
      for (int q = 0; q < NA; ++q) acc[q] = 0.0f;
      if (mine)
#pragma unroll 4
        for (int j = sub; j < npad; j += L) {
          float4 w[Op::JW];
#pragma unroll
          for (int k = 0; k < NR; ++k) x[k] = c[k * npmax + j];
          Op::raw_j(x, w);
          o.template pair<0>(I, w, acc);
        }
#pragma unroll
      for (int q = 0; q < NA; ++q) {
        v[q] = acc[q];
#pragma unroll
        for (int off = L / 2; off > 0; off >>= 1) v[q] += __shfl_xor_sync(0xffffffffu, v[q], off);
      }
    }
    if (mine) {  // the same in every lane of the row, so that each can serve one CTA
      const double e = o.small_step(P, v, a, S, nx);
      if (Op::kTileSum && owner) s_e[cur][lrow] = e;
    }
    if (s + 1 < T) {
#pragma unroll
      for (int k = 0; k < ND; ++k)
        if (mine && sub < C)  // lane `sub` serves cluster CTA `sub`
          *cg::this_cluster().map_shared_rank(&nxt[k * npmax + row], sub) = nx[k];
#pragma unroll
      for (int d = 0; d < 3; ++d) a[d] = an[d];
    }
    cluster_sync_all();
  }
  flush(T - 1);
  stamp_exit(sy, dir > 0 ? 0 : 1);
  pdl_trigger();
}

}  // namespace lddmm

// GB300 kernels of the sphere-DEM timestep.
//
// One step = k_particle (force gather of the previous step + walls + gravity +
// nve/sphere final and initial half-kicks + skin check) -> k_decide ->
// [rebuild kernels, no-ops unless ctrl->rebuild] -> k_pair.  All decisions
// live in device memory (Ctrl), so many steps are queued without a host sync.
//
// Determinism: every force is the sum of per-pair results in a fixed order
// (owner row ascending, then partner list ascending); no floating-point
// atomics anywhere.  Integer atomics are only used for counting; each
// resulting order is made canonical by a per-cell / per-atom sort.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdlib>
#include <stdint.h>

#include "bond_law.cuh"
#include "contact_law.cuh"
#include "dem_device.cuh"
#include "dem_kernels.h"
#include "mesh_device.cuh"
#include "step_device.cuh"

namespace gb300 {

// ----------------------------------------------------------------------------
// step control
// ----------------------------------------------------------------------------

// Neighbor::decide (src/neighbor.cpp:1362-1376): a fix that forces a
// rebuild at this step (FixMesh::next_reneighbor) comes before the
// ago/every/delay/check logic.  A moving mesh that travelled more than skin/2
// on a step without rebuild forces one at the next step.
// An ensemble decides per system, as each system running alone would; the
// rebuild stage runs when any system rebuilds, and the others keep their
// atom order, list and histories.  Called by every thread of a single
// block (one thread per system at a time); the result is the block's.  The
// displacement flags are read past L1 (the last block of k_particle decides
// while the flags other blocks set may sit stale in its SM's L1).
__device__ __forceinline__ int decide_rebuild(const Sys &s, Ctrl *c) {
  const int force = c->force_rebuild;
  int r_any = 0;
  for (int k = threadIdx.x; k < s.nsys; k += blockDim.x) {
    int r = 1;
    if (!force) {
      const int ago = ++s.sys_ago[k];
      r = (ago >= s.neigh_delay && ago % s.neigh_every == 0) ? (s.neigh_check ? __ldcg(&s.sys_moved[k]) : 1)
                                                             : 0;
    }
    s.sys_reb[k] = r;
    s.sys_moved[k] = 0;
    r_any |= r;
  }
  int reb = __syncthreads_or(r_any);
  if (threadIdx.x == 0) {
    if (force) {
      reb = 1;
    } else if (!s.nsys) {
      c->ago++;
      if (c->ago >= s.neigh_delay && c->ago % s.neigh_every == 0) reb = s.neigh_check ? __ldcg(&c->moved) : 1;
    }
    c->force_rebuild = reb ? 0 : c->mesh_moved;
    c->mesh_moved = 0;
    c->rebuild = reb;
    c->moved = 0;
  }
  return reb;
}

// this atom's system rebuilds at the current rebuild stage
__device__ __forceinline__ bool sys_rebuilds(const Sys &s, int type) { return s.nsys == 0 || s.sys_reb[type - 1]; }

__global__ void k_decide(Sys s) {
  Ctrl *c = s.ctrl;
  if (c->halt) return;
  if (threadIdx.x == 0) c->ntimestep++;
  decide_rebuild(s, c);
}

// The conditionals of the graph-resident step loop.  on: the last block of
// k_particle takes the decision (else k_decide_loop); gate: a step of the
// unrolled loop, which may be held.
struct LoopCond {
  int on, gate;
  cudaGraphConditionalHandle hreb, hloop;
};

// whether the loop's kernels are no-ops: halted, or held; ends the loop when
// halted or out of steps (called by every thread, `lead` by one of them)
__device__ __forceinline__ bool loop_held(const Ctrl *c, const LoopCond &lp, bool lead) {
  const int hold = lp.gate ? c->hold : kHoldNone;
  if (!c->halt && hold == kHoldNone) return false;
  if (lead && (c->halt || hold == kHoldDone)) {
    cudaGraphSetConditional(lp.hreb, 0);
    cudaGraphSetConditional(lp.hloop, 0);
  }
  return true;
}

// the decision of a loop step, by one thread behind decide_rebuild
__device__ __forceinline__ void loop_decided(Ctrl *c, const LoopCond &lp, int reb) {
  const int left = --c->loop_left;
  c->hold = reb ? kHoldRebuild : (left > 0 ? kHoldNone : kHoldDone);
  cudaGraphSetConditional(lp.hreb, reb ? 1u : 0u);
  cudaGraphSetConditional(lp.hloop, reb || left > 0 ? 1u : 0u);
}

// k_decide for the step loop: also drives the IF node around the rebuild and
// the WHILE node around the steps
__global__ void k_decide_loop(Sys s, LoopCond lp) {
  Ctrl *c = s.ctrl;
  if (loop_held(c, lp, threadIdx.x == 0)) return;
  __syncthreads();  // every thread has read the hold before it changes
  if (threadIdx.x == 0) c->ntimestep++;
  const int reb = decide_rebuild(s, c);
  if (threadIdx.x == 0) loop_decided(c, lp, reb);
}

__global__ void k_set_loop(Ctrl *c, int n, int phase, int turn) {
  c->loop_left = n;
  c->turn = turn;
  c->step_phase = phase;
}

__global__ void k_set_rebuild(Sys s, int v) {
  if (s.ctrl->halt) return;
  if (threadIdx.x == 0) {
    s.ctrl->rebuild = v;
    s.ctrl->moved = 0;
  }
  for (int k = threadIdx.x; k < s.nsys; k += blockDim.x) {
    s.sys_reb[k] = v;
    s.sys_moved[k] = 0;
  }
}

__global__ void k_zero_gated(Sys s, int *a, int n) {
  if (gated(s.ctrl)) return;
  GRID_STRIDE(i, n) a[i] = 0;
}

// ----------------------------------------------------------------------------
// exclusive scan (warp-shuffle prefix sums), 4096 items per block
// ----------------------------------------------------------------------------

// out[k] = sum(in[0..k-1]) within the block's 4096 items; bsum[block] = total.
// gate: 0 always runs; 1 only while the system rebuilds; 2 also not in an
// ensemble rebuild that keeps the other systems in place (Ctrl::pmode)
__device__ __forceinline__ bool scan_gated(const Ctrl *c, int gate) {
  return gate && (gated(c) || (gate == 2 && c->pmode));
}

__global__ void __launch_bounds__(1024) k_scan_blocks(Sys s, const int *__restrict__ in, int *out,
                                                      int len, int *bsum, int gate) {
  if (scan_gated(s.ctrl, gate)) return;
  __shared__ int wsum[32];
  const int t = threadIdx.x, lane = t & 31, w = t >> 5;
  const long base = (long)blockIdx.x * 4096 + 4 * t;
  int v[4], tot = 0;
#pragma unroll
  for (int k = 0; k < 4; k++) {
    v[k] = (base + k < len) ? in[base + k] : 0;
    tot += v[k];
  }
  int incl = warp_incl_scan(tot);
  if (lane == 31) wsum[w] = incl;
  __syncthreads();
  if (w == 0) wsum[lane] = warp_incl_scan(wsum[lane]);
  __syncthreads();
  int run = incl - tot + (w ? wsum[w - 1] : 0);
#pragma unroll
  for (int k = 0; k < 4; k++) {
    if (base + k < len) out[base + k] = run;
    run += v[k];
  }
  if (t == 1023 && bsum) bsum[blockIdx.x] = run;
}

// The same in one launch, for short arrays: a block sums the items before its
// chunk itself instead of waiting for the others' totals.
__global__ void __launch_bounds__(1024) k_scan_flat(Sys s, const int *__restrict__ in, int *out, int len, int gate) {
  if (scan_gated(s.ctrl, gate)) return;
  __shared__ int wsum[32], wbase[32];
  const int t = threadIdx.x, lane = t & 31, w = t >> 5;
  const int base = blockIdx.x * 4096 + 4 * t;
  int v[4], tot = 0, before = 0;
#pragma unroll
  for (int k = 0; k < 4; k++) {
    v[k] = (base + k < len) ? in[base + k] : 0;
    tot += v[k];
  }
#pragma unroll 8
  for (int k = t; k < (int)blockIdx.x * 4096; k += 1024) before += in[k];
  before = __reduce_add_sync(0xffffffffu, before);
  const int incl = warp_incl_scan(tot);
  if (lane == 31) wsum[w] = incl;
  if (lane == 0) wbase[w] = before;
  __syncthreads();
  if (w == 0) {
    wsum[lane] = warp_incl_scan(wsum[lane]);
    wbase[lane] = __reduce_add_sync(0xffffffffu, wbase[lane]);
  }
  __syncthreads();
  int run = wbase[0] + incl - tot + (w ? wsum[w - 1] : 0);
#pragma unroll
  for (int k = 0; k < 4; k++) {
    if (base + k < len) out[base + k] = run;
    run += v[k];
  }
}

__global__ void k_scan_add(Sys s, int *out, int len, const int *__restrict__ bsum, int gate) {
  if (scan_gated(s.ctrl, gate)) return;
  const int add = bsum[blockIdx.x];
  const long base = (long)blockIdx.x * 4096;
  for (int k = threadIdx.x; k < 4096; k += blockDim.x)
    if (base + k < len) out[base + k] += add;
}

// ----------------------------------------------------------------------------
// ensemble rebuilds that keep the other systems in place
// ----------------------------------------------------------------------------
//
// A rebuild of an ensemble where only some systems rebuild (Ctrl::pmode)
// runs the rebuild kernels over those systems' atoms, cells and list
// segments alone, through compact indices: atom t of the rebuilding systems
// (prefix sums rpre over rlist), cell u (ens_ncell per system), segment
// entry u (prefix sums cpre of the segments' capacities).  Every other
// system keeps its atoms, cells, list entries, histories and holds where
// they are.  The whole-list path runs instead when a rebuilding system loses
// atoms (the systems behind it would move), and its list layout (Ctrl::lmode
// 0) when a rebuilding system's entries outgrow its segment.  Both paths
// give the same atom order, entries and values for every system.

// largest q in [0, n) with pre[q] <= t (pre ascending from 0, pre[n] > t)
__device__ __forceinline__ int seg_find(const int *pre, int n, int t) {
  int lo = 0, hi = n - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (pre[mid] <= t) lo = mid;
    else hi = mid - 1;
  }
  return lo;
}

// atom of compact index t (t < nra); systems keep their ranges in pmode
__device__ __forceinline__ int ens_atom(const Sys &s, const Ctrl *c, int t) {
  const int q = seg_find(s.rpre, c->nR, t);
  return s.sys_start[s.rlist[q]] + (t - s.rpre[q]);
}

// list entry of compact segment index u (u < ncr)
__device__ __forceinline__ int ens_entry(const Sys &s, const Ctrl *c, int u) {
  const int q = seg_find(s.cpre, c->nR, u);
  return s.seg_start[s.rlist[q]] + (u - s.cpre[q]);
}

// cell of compact index u (u < nR * ens_ncell)
__device__ __forceinline__ int ens_cell(const Sys &s, int u) {
  return s.rlist[u / s.ens_ncell] * s.ens_ncell + u % s.ens_ncell;
}

__device__ __forceinline__ bool ens_partial(const Sys &s, const Ctrl *c) { return s.nsys && c->pmode; }
__device__ __forceinline__ bool ens_list_partial(const Sys &s, const Ctrl *c) { return s.nsys && c->lmode; }

// exclusive block-wide prefix sum of one int per thread (blockDim.x a
// multiple of 32); *tot = the block's total
__device__ int block_excl_scan(int v, int *tot) {
  __shared__ int ws[32];
  __shared__ int wt;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = blockDim.x >> 5;
  const int incl = warp_incl_scan(v);
  if (lane == 31) ws[w] = incl;
  __syncthreads();
  if (w == 0) {
    const int y = warp_incl_scan(lane < nw ? ws[lane] : 0);
    if (lane < nw) ws[lane] = y;
    if (lane == 31) wt = y;
  }
  __syncthreads();
  const int ex = incl - v + (w ? ws[w - 1] : 0);
  *tot = wt;
  __syncthreads();  // ws and wt are reused by the next call
  return ex;
}

// out[i] = base + sum(in[b..i)) for i in [b, e), and out_end[i] = out[i] +
// in[i] when out_end is set, by one block of 1024 threads in chunks of 8192
// (256 items per warp, eight per lane), the next chunk's items on their way
// while one is summed; returns the range's total (every thread).  One block per
// rebuilding system of an ensemble: its 30,000 cells took 18.5 us in chunks of
// 4096 loaded one after the other, and take 11.4.
__device__ int block_range_scan(const int *__restrict__ in, int b, int e, int base, int *out, int *out_end) {
  __shared__ int wsum[32];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  int carry = base, v[8];
  const int o = w * 256 + lane;
#pragma unroll
  for (int k = 0; k < 8; k++) v[k] = b + o + 32 * k < e ? in[b + o + 32 * k] : 0;
  for (int c0 = b; c0 < e; c0 += 8192) {
    int x[8], u[8], tot = 0;
#pragma unroll
    for (int k = 0; k < 8; k++) {
      const int i = c0 + 8192 + o + 32 * k;
      u[k] = i < e ? in[i] : 0;
    }
#pragma unroll
    for (int k = 0; k < 8; k++) {
      const int inc = warp_incl_scan(v[k]);
      x[k] = tot + inc - v[k];
      tot += __shfl_sync(0xffffffffu, inc, 31);
    }
    if (lane == 0) wsum[w] = tot;
    __syncthreads();
    const int sums = warp_incl_scan(wsum[lane]);  // (every warp for itself)
    const int before = carry + (w ? __shfl_sync(0xffffffffu, sums, w - 1) : 0);
    carry += __shfl_sync(0xffffffffu, sums, 31);
#pragma unroll
    for (int k = 0; k < 8; k++) {
      const int i = c0 + o + 32 * k;
      if (i < e) {
        out[i] = before + x[k];
        if (out_end) out_end[i] = before + x[k] + v[k];
      }
      v[k] = u[k];
    }
    __syncthreads();  // every warp has read wsum
  }
  return carry - base;
}

// Domain::pbc (src/domain.cpp:550-600) of one atom's position, in place;
// true when the atom is then outside the box in any dimension, which
// CommBrick::exchange deletes (src/comm_brick.cpp:784-808)
__device__ __forceinline__ bool pbc_wrap(const Sys &s, double xv[3]) {
  bool lost = false;
#pragma unroll
  for (int d = 0; d < 3; d++) {
    if (s.periodic[d]) {
      if (xv[d] < s.boxlo[d]) xv[d] = __dadd_rn(xv[d], s.prd[d]);
      if (xv[d] >= s.boxhi[d]) {
        xv[d] = __dadd_rn(xv[d], -s.prd[d]);
        if (xv[d] < s.boxlo[d]) xv[d] = s.boxlo[d];
      }
    }
    if (xv[d] < s.boxlo[d] || xv[d] >= s.boxhi[d]) lost = true;
  }
  return lost;
}

// Compacts the rebuilding systems and picks the path: in place (pmode 1)
// when the list is in segments, some system does not rebuild and the
// whole-list path is not forced.  One block.
__global__ void k_ens_plan(Sys s) {
  Ctrl *c = s.ctrl;
  if (gated(c)) return;
  __shared__ int cr, ca, cc;
  if (threadIdx.x == 0) cr = ca = cc = 0;
  __syncthreads();
  for (int b = 0; b < s.nsys; b += blockDim.x) {
    const int k = b + threadIdx.x;
    const int r = k < s.nsys ? s.sys_reb[k] : 0;
    const int na = r ? s.sys_start[k + 1] - s.sys_start[k] : 0;
    const int ne = r ? s.seg_start[k + 1] - s.seg_start[k] : 0;
    int tr, ta, te;
    const int xr = block_excl_scan(r, &tr);
    const int xa = block_excl_scan(na, &ta);
    const int xe = block_excl_scan(ne, &te);
    if (r) {
      s.rlist[cr + xr] = k;
      s.rpre[cr + xr] = ca + xa;
      s.cpre[cr + xr] = cc + xe;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
      cr += tr;
      ca += ta;
      cc += te;
    }
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    s.rpre[cr] = ca;
    s.cpre[cr] = cc;
    c->nR = cr;
    c->nra = ca;
    c->ncr = cc;
    const int part = (c->seg_ok && !s.ens_full && cr < s.nsys) ? 1 : 0;
    c->pmode = part;
    c->lmode = part;
    c->np_new = c->np;
  }
}

// in-place path: a rebuilding system that loses an atom moves every system
// behind it, so the whole-list path takes this rebuild
__global__ void k_ens_lost(Sys s) {
  Ctrl *c = s.ctrl;
  if (gated(c) || !c->pmode) return;
  const AtomArrays &A = s.atoms[0];
  GRID_STRIDE(t, c->nra) {
    const int i = ens_atom(s, c, t);
    double xv[3] = {A.x[i], A.y[i], A.z[i]};
    if (pbc_wrap(s, xv)) {
      c->pmode = 0;
      c->lmode = 0;
    }
  }
}

__global__ void k_ens_zero_cells(Sys s) {
  Ctrl *c = s.ctrl;
  if (gated(c)) return;
  if (c->pmode) {
    const int tot = c->nR * s.ens_ncell;
    GRID_STRIDE(u, tot) {
      const int cell = ens_cell(s, u);
      s.cell_count[cell] = 0;
      s.cell_fill[cell] = 0;
    }
  } else {
    GRID_STRIDE(u, s.ncell + 2) {
      s.cell_count[u] = 0;
      s.cell_fill[u] = 0;
    }
  }
}

// the in-place path's block-per-system prefix sums
enum { kEnsScanCells = 0, kEnsScanRowsPartial = 1, kEnsScanRowsFull = 2, kEnsScanRev = 3 };

// atoms of system k after this rebuild's cell sort: [lo, hi)
__device__ __forceinline__ void ens_range(const Sys &s, int k, int &lo, int &hi) {
  lo = s.cell_start[k * s.ens_ncell];
  hi = s.cell_start[(k + 1) * s.ens_ncell];
}

__global__ void __launch_bounds__(1024) k_ens_scan(Sys s, int what) {
  Ctrl *c = s.ctrl;
  if (gated(c)) return;
  const PairArrays &M = s.pairs[1];
  bool all = false;
  if (what == kEnsScanCells || what == kEnsScanRowsPartial) {
    if (!(what == kEnsScanCells ? c->pmode : c->lmode)) return;
  } else if (what == kEnsScanRowsFull) {
    if (c->lmode) return;
    all = true;
  } else {
    all = !c->lmode;
  }
  const int nlist = all ? s.nsys : c->nR;
  for (int q = blockIdx.x; q < nlist; q += gridDim.x) {
    const int k = all ? q : s.rlist[q];
    int lo, hi;
    if (what == kEnsScanCells) {
      // the system's cells, from its first atom (its range is unchanged)
      block_range_scan(s.cell_count, k * s.ens_ncell, (k + 1) * s.ens_ncell, s.sys_start[k], s.cell_start, nullptr);
      continue;
    }
    ens_range(s, k, lo, hi);
    if (what == kEnsScanRev) {
      block_range_scan(s.rev_count, lo, hi, s.seg_start[k], M.rev_start, M.reve);
      continue;
    }
    // owner rows: into the system's own segment, or relative (the layout
    // kernel places the segments) on the whole-list path
    const int base = what == kEnsScanRowsPartial ? s.seg_start[k] : 0;
    const int used = block_range_scan(s.pcount, lo, hi, base, M.row, M.rowe);
    if (threadIdx.x == 0) {
      s.seg_used[k] = used;
      if (what == kEnsScanRowsPartial && used > s.seg_start[k + 1] - s.seg_start[k]) c->lmode = 0;
    }
  }
}

// in place for the atoms, whole list for the entries: the systems that do
// not rebuild keep their atoms where they are (perm = identity) and count
// their current rows
__global__ void k_ens_kept(Sys s) {
  Ctrl *c = s.ctrl;
  if (gated(c) || !c->pmode || c->lmode) return;
  const AtomArrays &A = s.atoms[0];
  const PairArrays &L = s.pairs[0];
  GRID_STRIDE(i, c->n) {
    if (s.sys_reb[A.type[i] - 1]) continue;
    s.pcount[i] = L.rowe[i] - L.row[i];
    s.perm[i] = i;
  }
}

// whole-list path: every system gets a segment of its entries plus slack
// (ens_slack percent and 64 more; none with ens_slack 0), so that later
// rebuilds of it alone stay in place while it grows.  One block.
__global__ void k_ens_layout(Sys s) {
  Ctrl *c = s.ctrl;
  if (gated(c) || c->lmode) return;
  __shared__ int run;
  if (threadIdx.x == 0) run = 0;
  __syncthreads();
  for (int b = 0; b < s.nsys; b += blockDim.x) {
    const int k = b + threadIdx.x;
    int cap = 0;
    if (k < s.nsys) {
      const long u = s.seg_used[k];
      cap = (int)(u + (u * s.ens_slack) / 100 + (s.ens_slack ? 64 : 0));
    }
    int tot;
    const int x = block_excl_scan(cap, &tot);
    if (k < s.nsys) s.seg_start[k] = run + x;
    __syncthreads();
    if (threadIdx.x == 0) run += tot;
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    s.seg_start[s.nsys] = run;
    c->np_new = run;
  }
}

// whole-list path: relative rows into the system's segment
__global__ void k_ens_rows_base(Sys s) {
  Ctrl *c = s.ctrl;
  if (gated(c) || c->lmode) return;
  const AtomArrays &A = s.atoms[0];
  const PairArrays &M = s.pairs[1];
  GRID_STRIDE(i, c->n_new) {
    const int b = s.seg_start[A.type[i] - 1];
    M.row[i] += b;
    M.rowe[i] += b;
  }
}

__global__ void k_ens_zero_rev(Sys s) {
  Ctrl *c = s.ctrl;
  if (gated(c)) return;
  if (c->lmode) {
    GRID_STRIDE(t, c->nra) {
      const int i = ens_atom(s, c, t);
      s.rev_count[i] = 0;
      s.rev_fill[i] = 0;
    }
  } else {
    GRID_STRIDE(i, s.nmax + 1) {
      s.rev_count[i] = 0;
      s.rev_fill[i] = 0;
    }
  }
}

// unused entries at the end of each (rebuilt) segment
__global__ void k_ens_holes(Sys s) {
  Ctrl *c = s.ctrl;
  if (gated(c)) return;
  const PairArrays &M = s.pairs[1];
  const bool part = c->lmode;
  const int nlist = part ? c->nR : s.nsys;
  for (int q = blockIdx.x; q < nlist; q += gridDim.x) {
    const int k = part ? s.rlist[q] : q;
    for (int p = s.seg_start[k] + s.seg_used[k] + threadIdx.x; p < s.seg_start[k + 1]; p += blockDim.x) {
      M.i[p] = -1;
      M.j[p] = -1;
      M.sh[p] = (uint8_t)kHole;
      M.flag[p] = 0;
    }
  }
}

// ----------------------------------------------------------------------------
// rebuild: pbc wrap, cell sort, permutation
// ----------------------------------------------------------------------------

// Domain::pbc then CommBrick::exchange deletion of atoms outside the box
// (pbc_wrap), and the atoms' neighbour cells.
__device__ __forceinline__ void cell_count_atom(const Sys &s, const AtomArrays &A, int i) {
  double xv[3] = {A.x[i], A.y[i], A.z[i]};
  const bool lost = pbc_wrap(s, xv);
  A.x[i] = xv[0];
  A.y[i] = xv[1];
  A.z[i] = xv[2];
  int cell = s.ncell;
  if (!lost) {
    const int cx = cell_coord(s, xv[0], 0), cy = cell_coord(s, xv[1], 1), cz = cell_coord(s, xv[2], 2);
    cell = cx + s.nc[0] * (cy + s.nc[1] * cz) + (s.ens_ncell ? (A.type[i] - 1) * s.ens_ncell : 0);
  }
  s.pcount[i] = cell;  // reused as per-atom cell id until the pair count
  atomicAdd(&s.cell_count[cell], 1);
}

__global__ void k_cell_count(Sys s) {
  Ctrl *c = s.ctrl;
  if (gated(c)) return;
  const AtomArrays &A = s.atoms[0];
  if (ens_partial(s, c)) {
    GRID_STRIDE(t, c->nra) cell_count_atom(s, A, ens_atom(s, c, t));
    return;
  }
  const int n = c->n;
  // a system that does not rebuild keeps its atoms in order in its first
  // cell: its count is set once, not added per atom
  GRID_STRIDE(k, s.nsys)
    if (!s.sys_reb[k]) s.cell_count[k * s.ens_ncell] = s.sys_start[k + 1] - s.sys_start[k];
  GRID_STRIDE(i, n) {
    if (!sys_rebuilds(s, A.type[i])) {
      s.pcount[i] = (A.type[i] - 1) * s.ens_ncell;
      continue;
    }
    cell_count_atom(s, A, i);
  }
}

__global__ void k_cell_scatter(Sys s) {
  Ctrl *c = s.ctrl;
  if (gated(c)) return;
  const AtomArrays &A = s.atoms[0];
  if (ens_partial(s, c)) {
    GRID_STRIDE(t, c->nra) {
      const int i = ens_atom(s, c, t);
      const int cell = s.pcount[i];
      s.order[s.cell_start[cell] + atomicAdd(&s.cell_fill[cell], 1)] = i;
    }
    return;
  }
  const int n = c->n;
  GRID_STRIDE(i, n) {
    const int cell = s.pcount[i];
    int slot;
    if (!sys_rebuilds(s, A.type[i])) slot = s.cell_start[cell] + (i - s.sys_start[A.type[i] - 1]);
    else slot = s.cell_start[cell] + atomicAdd(&s.cell_fill[cell], 1);
    s.order[slot] = i;
  }
}

// canonical order inside every cell: ascending previous index
__device__ __forceinline__ void cell_sort_one(const Sys &s, int cell) {
  const int b = s.cell_start[cell], e = s.cell_start[cell + 1];
  for (int k = b + 1; k < e; k++) {
    const int v = s.order[k];
    int m = k - 1;
    while (m >= b && s.order[m] > v) {
      s.order[m + 1] = s.order[m];
      m--;
    }
    s.order[m + 1] = v;
  }
}

__global__ void k_cell_sort(Sys s) {
  Ctrl *c = s.ctrl;
  if (gated(c)) return;
  if (ens_partial(s, c)) {
    const int tot = c->nR * s.ens_ncell;
    GRID_STRIDE(u, tot) cell_sort_one(s, ens_cell(s, u));
  } else {
    GRID_STRIDE(cell, s.ncell) {
      if (s.nsys && !s.sys_reb[cell / s.ens_ncell]) continue;  // already in order
      cell_sort_one(s, cell);
    }
  }
  // (in place, cell_start[ncell] is the atom count of the last whole build
  // and no atom is lost)
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    c->n_new = s.cell_start[s.ncell];
    c->nmlist = 0;
    c->lost_step = c->n - c->n_new;
  }
}

// The copies of a rebuild load an item's values before they store the first:
// a store may alias the loads behind it, so that a copy value by value waits
// for every load in turn (526,000 atoms: k_permute 61 -> 46 us, k_copy_atoms 44 ->
// 27, k_copy_pairs 69 -> 35).
template <int N, class T>
__device__ __forceinline__ void copy_values(T *const (&to)[N], const T *const (&from)[N], size_t i, size_t o) {
  T v[N];
#pragma unroll
  for (int k = 0; k < N; k++) v[k] = from[k][o];
#pragma unroll
  for (int k = 0; k < N; k++) to[k][i] = v[k];
}

// gather atoms into the new order (buffer 1), xhold = x, primitive-wall
// neighbour lists (PrimitiveWall::buildNeighList, src/primitive_wall.h:129-138)
__device__ __forceinline__ void permute_atom(const Sys &s, const AtomArrays &A, const AtomArrays &B, int i) {
  {
    const int o = s.order[i];
    s.perm[i] = o;
    const int type = A.type[o], tag = A.tag[o], lidx = A.lidx[o];
    const uint8_t old_bits = A.wbits[o];
    const double x = A.x[o], y = A.y[o], z = A.z[o], r = A.r[o];
    // f and torque are not moved: a rebuild comes after the step's initial
    // integration, and the step's gather writes them again before they are
    // read (they are live only between dem_step calls)
    double *const to[9] = {B.vx, B.vy, B.vz, B.wx, B.wy, B.wz, B.m, B.dtfm, B.dtir};
    const double *const from[9] = {A.vx, A.vy, A.vz, A.wx, A.wy, A.wz, A.m, A.dtfm, A.dtir};
    copy_values(to, from, i, o);
    const bool reb = sys_rebuilds(s, type);
    double xh[3] = {x, y, z};
    if (!reb) {  // a system that does not rebuild keeps its holds
      xh[0] = A.xh[o];
      xh[1] = A.yh[o];
      xh[2] = A.zh[o];
    }
    B.x[i] = x; B.y[i] = y; B.z[i] = z;
    B.xh[i] = xh[0]; B.yh[i] = xh[1]; B.zh[i] = xh[2];
    B.r[i] = r;
    B.type[i] = type; B.tag[i] = tag; B.lidx[i] = lidx;
    uint8_t bits = 0;
    for (int w = 0; w < s.nplanes; w++) {
      double *const bw = B.whist + (size_t)w * 3 * s.nmax;
      const double *const aw = A.whist + (size_t)w * 3 * s.nmax;
      double *const wto[3] = {bw, bw + s.nmax, bw + 2 * (size_t)s.nmax};
      const double *const wfrom[3] = {aw, aw + s.nmax, aw + 2 * (size_t)s.nmax};
      copy_values(wto, wfrom, i, o);
      const Plane &pl = s.planes[w];
      const double dMax = __dadd_rn(r, s.skin);
      if (pl.kind == 1) {
        // Cylinder<dim>::resolveNeighlist (src/primitive_wall_definitions.h:192-198)
        const double xo[3] = {x, y, z};
        const double dy = __dadd_rn(xo[(pl.axis + 1) % 3], -pl.c1), dz = __dadd_rn(xo[(pl.axis + 2) % 3], -pl.c2);
        const double dist = __dadd_rn(__dsqrt_rn(__dadd_rn(__dmul_rn(dy, dy), __dmul_rn(dz, dz))), -pl.pos);
        if (dMax < dist || -dMax < dist) bits |= (uint8_t)(1u << w);
        continue;
      }
      const double pos = pl.axis == 0 ? x : (pl.axis == 1 ? y : z);
      const double dist = pos - plane_pos(pl, type);
      const double absdist = (dist > 0.0) ? dist : -dist;
      if (absdist <= dMax) bits |= (uint8_t)(1u << w);
    }
    B.wbits[i] = reb ? bits : old_bits;
    for (int k = 0; k < s.nmeshes; k++) {  // FixContactHistoryMesh per-atom slots travel too
      const MeshDev &M = s.meshes[k];
      const int ns = M.nslot[0][o];
      M.nslot[1][i] = ns;
      M.npart[1][i] = M.npart[0][o];
      for (int q = 0; q < ns; q++) {
        M.slot_tri[1][(size_t)q * s.nmax + i] = M.slot_tri[0][(size_t)q * s.nmax + o];
        for (int d = 0; d < 3; d++)
          M.slot_hist[1][(size_t)(3 * q + d) * s.nmax + i] = M.slot_hist[0][(size_t)(3 * q + d) * s.nmax + o];
      }
    }
  }
}

__global__ void k_permute(Sys s) {
  Ctrl *c = s.ctrl;
  if (gated(c)) return;
  const AtomArrays &A = s.atoms[0];
  const AtomArrays &B = s.atoms[1];
  if (ens_partial(s, c)) {
    GRID_STRIDE(t, c->nra) permute_atom(s, A, B, ens_atom(s, c, t));
    return;
  }
  const int n = c->n_new;
  GRID_STRIDE(i, n) permute_atom(s, A, B, i);
}

__device__ __forceinline__ void copy_atom(const Sys &s, const AtomArrays &A, const AtomArrays &B, int i) {
  {
    const double x = B.x[i], y = B.y[i], z = B.z[i], xh = B.xh[i], yh = B.yh[i], zh = B.zh[i], r = B.r[i];
    const int type = B.type[i], tag = B.tag[i], lidx = B.lidx[i];
    const uint8_t bits = B.wbits[i];
    double *const to[9] = {A.vx, A.vy, A.vz, A.wx, A.wy, A.wz, A.m, A.dtfm, A.dtir};
    const double *const from[9] = {B.vx, B.vy, B.vz, B.wx, B.wy, B.wz, B.m, B.dtfm, B.dtir};
    copy_values(to, from, i, i);
    A.x[i] = x; A.y[i] = y; A.z[i] = z;
    A.xh[i] = xh; A.yh[i] = yh; A.zh[i] = zh;
    A.r[i] = r;
    A.type[i] = type; A.tag[i] = tag; A.lidx[i] = lidx;
    A.wbits[i] = bits;
    const float4 xf = make_float4((float)x, (float)y, (float)z, (float)r);
    s.xf[i] = xf;
    // xhold = x at this build (k_permute), or kept by a system that did not rebuild
    s.xhf[i] = sys_rebuilds(s, type) ? xf : make_float4((float)xh, (float)yh, (float)zh, xf.w);
    for (int w = 0; w < s.nplanes; w++) {
      double *const aw = A.whist + (size_t)w * 3 * s.nmax;
      const double *const bw = B.whist + (size_t)w * 3 * s.nmax;
      double *const wto[3] = {aw, aw + s.nmax, aw + 2 * (size_t)s.nmax};
      const double *const wfrom[3] = {bw, bw + s.nmax, bw + 2 * (size_t)s.nmax};
      copy_values(wto, wfrom, i, i);
    }
    for (int k = 0; k < s.nmeshes; k++) {
      const MeshDev &M = s.meshes[k];
      const int ns = M.nslot[1][i];
      M.nslot[0][i] = ns;
      M.npart[0][i] = M.npart[1][i];
      for (int q = 0; q < ns; q++) {
        M.slot_tri[0][(size_t)q * s.nmax + i] = M.slot_tri[1][(size_t)q * s.nmax + i];
        for (int d = 0; d < 3; d++)
          M.slot_hist[0][(size_t)(3 * q + d) * s.nmax + i] = M.slot_hist[1][(size_t)(3 * q + d) * s.nmax + i];
      }
    }
  }
}

__global__ void k_copy_atoms(Sys s) {
  Ctrl *c = s.ctrl;
  if (gated(c)) return;
  const AtomArrays &A = s.atoms[0];
  const AtomArrays &B = s.atoms[1];
  if (ens_partial(s, c)) {
    GRID_STRIDE(t, c->nra) copy_atom(s, A, B, ens_atom(s, c, t));
    return;
  }
  const int n = c->n_new;
  GRID_STRIDE(i, n) copy_atom(s, A, B, i);
}

// ----------------------------------------------------------------------------
// rebuild: triangle-mesh candidate lists (FixNeighlistMesh::pre_force) and
// history slot maintenance (FixContactHistoryMesh::pre_exchange/pre_force)
// ----------------------------------------------------------------------------

__device__ __forceinline__ void mslot_swap(const MeshDev &M, size_t nmax, int i, int a, int b) {
  const int t = M.slot_tri[0][a * nmax + i];
  M.slot_tri[0][a * nmax + i] = M.slot_tri[0][b * nmax + i];
  M.slot_tri[0][b * nmax + i] = t;
  for (int d = 0; d < 3; d++) {
    const double h = M.slot_hist[0][(3 * a + d) * nmax + i];
    M.slot_hist[0][(3 * a + d) * nmax + i] = M.slot_hist[0][(3 * b + d) * nmax + i];
    M.slot_hist[0][(3 * b + d) * nmax + i] = h;
  }
}

__global__ void k_mesh_move(Sys s, int k, int gate) {
  Ctrl *c = s.ctrl;
  if (c->halt || (gate && c->hold)) return;
  const MeshDev &M = s.meshes[k];
  bool moved = false;
  const int per = (gridDim.x * blockDim.x) / 16;
  // whole warps iterate together (mesh_move_part synchronises the warp)
  for (int t0 = (blockIdx.x * blockDim.x + (threadIdx.x & ~31)) / 16; t0 < M.ntri; t0 += per)
    moved |= mesh_move_part(s, M, t0 + ((threadIdx.x & 31) >> 4), threadIdx.x & 15);
  if (__any_sync(0xffffffffu, moved) && (threadIdx.x & 31) == 0) atomicOr(&c->mesh_moved, 1);
}

// sort_contacts: move filled slots forward (swap first empty <-> last filled)
__global__ void k_mesh_sort(Sys s, int k) {
  Ctrl *c = s.ctrl;
  if (gated(c)) return;
  const MeshDev &M = s.meshes[k];
  const int n = c->n_new;
  const size_t nmax = s.nmax;
  GRID_STRIDE(i, n) {
    const int nn = M.nslot[0][i];
    int fe, lf;
    do {
      fe = lf = -1;
      for (int j = 0; j < nn; j++) {
        const int p = M.slot_tri[0][j * nmax + i];
        if (fe == -1 && p == -1) fe = j;
        if (p >= 0) lf = j;
      }
      if (fe > -1 && lf > -1 && fe < lf) mslot_swap(M, nmax, i, fe, lf);
    } while (fe > -1 && lf > -1 && fe < lf);
  }
}

__device__ __forceinline__ void tri_cell_range(const Sys &s, const MeshDev &M, int t, int lo[3], int hi[3]) {
  const double *g = M.tri + (size_t)t * kTriStride;
  for (int d = 0; d < 3; d++) {
    double a = g[d], b = g[d];
    for (int q = 1; q < 3; q++) {
      a = fmin(a, g[3 * q + d]);
      b = fmax(b, g[3 * q + d]);
    }
    lo[d] = cell_coord(s, a - M.distmax, d);
    hi[d] = cell_coord(s, b + M.distmax, d);
  }
}

__global__ void k_tri_count(Sys s, int k) {
  if (gated(s.ctrl)) return;
  const MeshDev &M = s.meshes[k];
  GRID_STRIDE(t, M.ntri) {
    if (M.moving)  // FixMesh::pre_force on a rebuild step: storeNodePosRebuild
      for (int q = 0; q < 9; q++) M.node_last[(size_t)t * 9 + q] = M.tri[(size_t)t * kTriStride + q];
    int lo[3], hi[3];
    tri_cell_range(s, M, t, lo, hi);
    for (int z = lo[2]; z <= hi[2]; z++)
      for (int y = lo[1]; y <= hi[1]; y++)
        for (int x = lo[0]; x <= hi[0]; x++) atomicAdd(&M.tc_count[x + s.nc[0] * (y + s.nc[1] * z)], 1);
  }
}

__global__ void k_tri_fill(Sys s, int k) {
  Ctrl *c = s.ctrl;
  if (gated(c)) return;
  const MeshDev &M = s.meshes[k];
  if (M.tc_start[s.ncell] > M.tc_cap) {  // the host grows tc_list to tc_start[ncell] and resumes
    if (blockIdx.x == 0 && threadIdx.x == 0) {
      c->status = kStatMeshReg;
      c->halt = 1;
    }
    return;
  }
  GRID_STRIDE(t, M.ntri) {
    int lo[3], hi[3];
    tri_cell_range(s, M, t, lo, hi);
    for (int z = lo[2]; z <= hi[2]; z++)
      for (int y = lo[1]; y <= hi[1]; y++)
        for (int x = lo[0]; x <= hi[0]; x++) {
          const int cell = x + s.nc[0] * (y + s.nc[1] * z);
          M.tc_list[M.tc_start[cell] + atomicAdd(&M.tc_fill[cell], 1)] = t;
        }
  }
}

// per atom: candidate triangles of its cell that pass resolveTriSphereNeighbuild,
// ascending; then cleanUpContactJumps and the re-paging of the slots
__global__ void k_mesh_cand(Sys s, int k) {
  Ctrl *c = s.ctrl;
  if (gated(c)) return;
  const MeshDev &M = s.meshes[k];
  const AtomArrays &A = s.atoms[0];
  const int n = c->n_new;
  const size_t nmax = s.nmax;
  const int cap = M.ccap;
  bool over = false;
  GRID_STRIDE(i, n) {
    const double xv[3] = {A.x[i], A.y[i], A.z[i]};
    const int cell = cell_coord(s, xv[0], 0) + s.nc[0] * (cell_coord(s, xv[1], 1) + s.nc[1] * cell_coord(s, xv[2], 2));
    const double rS = __dmul_rn(A.r[i], s.cdf);
    int *cand = M.cand + i;  // [q*nmax]
    int nc = 0, need = 0;
    for (int q = M.tc_start[cell]; q < M.tc_start[cell + 1]; q++) {
      const int t = M.tc_list[q];
      if (!tri_sphere_neighbuild(M.tri + (size_t)t * kTriStride, rS, xv, M.tskin)) continue;
      need++;
      if (nc == cap) continue;  // counted only: the host grows the capacity
      int m = nc++;
      while (m > 0 && cand[(size_t)(m - 1) * nmax] > t) {
        cand[(size_t)m * nmax] = cand[(size_t)(m - 1) * nmax];
        m--;
      }
      cand[(size_t)m * nmax] = t;
    }
    if (need > cap) {  // leave this atom's slots untouched; the rebuild resumes here after growth
      over = true;
      atomicMax(&c->mesh_need, need);
      continue;
    }
    M.cand_n[i] = nc;
    // cleanUpContactJumps: drop partners whose triangle no longer lists the atom
    int np = M.npart[0][i];
    int ip = 0;
    while (ip < np) {
      const int t = M.slot_tri[0][ip * nmax + i];
      bool listed = false;
      for (int q = 0; q < nc; q++) listed |= (cand[(size_t)q * nmax] == t);
      if (!listed) {
        M.slot_tri[0][ip * nmax + i] = -1;
        for (int d = 0; d < 3; d++) M.slot_hist[0][(3 * ip + d) * nmax + i] = 0.0;
        mslot_swap(M, nmax, i, ip, np - 1);
        np--;
      } else {
        ip++;
      }
    }
    for (int q = np; q < nc; q++) {
      M.slot_tri[0][q * nmax + i] = -1;
      for (int d = 0; d < 3; d++) M.slot_hist[0][(3 * q + d) * nmax + i] = 0.0;
    }
    M.npart[0][i] = np;
    M.nslot[0][i] = nc;
  }
  if (over) {
    c->status = kStatMeshCand;
    c->halt = 1;
  }
}

// Entry of the old list for the atom pair (owner o, partner q) in old
// indices: o's own row first, then the entries where o was the partner
// (flip = true).  Only flagged entries carry history (pre_exchange keeps
// those).  Returns -1 when none.
__device__ __forceinline__ int find_old(const Sys &s, const PairArrays &L, int o, int q, bool &flip) {
  flip = false;
  for (int k = L.row[o]; k < row_end(s, L, o); k++)
    if (L.j[k] == q && L.flag[k] != 0) return k;
  for (int k = L.rev_start[o]; k < rev_end(s, L, o); k++) {
    const int e = L.rev[k];
    if (L.i[e] == q && L.flag[e] != 0) {
      flip = true;
      return e;
    }
  }
  return -1;
}

// The contact constants of atom i with the walls that it is near (bits: its
// primitive walls); whether there are any.  Bit 7 is the eighth plane's behind
// k_permute and the list mark behind k_wall_list (of a system that does not
// rebuild, the mark of the build before): a reason to be listed either way.
__device__ __forceinline__ bool wall_consts_form(const Sys &s, int i, unsigned bits) {
  const AtomArrays &A = s.atoms[0];
  bool has = bits != 0;
  for (int w = 0; w < s.nplanes + s.nmeshes; w++) {
    const bool mesh = w >= s.nplanes;
    // (plane 7 shares its bit with the list mark, so that the wall tiles
    // look at it for every listed atom)
    const bool near = mesh ? s.meshes[w - s.nplanes].cand_n[i] > 0 : (w == 7 || ((bits >> w) & 1u));
    has |= mesh && near;
    if (!near) continue;
    const int wt = mesh ? s.meshes[w - s.nplanes].wall_type : s.planes[w].wall_type;
    const TypePair tp = load_typepair(s.params, s.ntypes, A.type[i], wt ? wt : A.type[i]);
    double c0, c1;
    if (s.normal == kHertz) contact_consts<kHertz>(tp, A.m[i], A.r[i], s.charVel, s.tdamp, c0, c1);
    else contact_consts<kHooke>(tp, A.m[i], A.r[i], s.charVel, s.tdamp, c0, c1);
    s.wcon[(size_t)(2 * w) * s.nmax + i] = c0;
    s.wcon[(size_t)(2 * w + 1) * s.nmax + i] = c1;
  }
  return has;
}

// new pair parameters between two builds: the walls' contacts take them at the
// next step (the pairs' constants belong to the list and stay until its build)
__global__ void k_wall_consts(Sys s) {
  GRID_STRIDE(i, s.ctrl->n) wall_consts_form(s, i, s.atoms[0].wbits[i]);
}

// atoms in a primitive wall's neighbour list or with candidate triangles on
// any mesh: bit 7 of wbits and the compact list the wall kernel walks (its
// order does not matter: one thread computes all of an atom's wall forces)
__global__ void __launch_bounds__(256) k_wall_list(Sys s) {
  __shared__ int wc[8], wbase;
  Ctrl *c = s.ctrl;
  if (gated(c)) return;
  const AtomArrays &A = s.atoms[0];
  const int n = c->n_new;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  // one reservation per block keeps each block's atoms ascending and
  // contiguous in the list (coalesced per-atom loads in the wall kernel)
  for (int base = blockIdx.x * blockDim.x; base < n; base += gridDim.x * blockDim.x) {
    const int i = base + threadIdx.x;
    bool has = false;
    if (i < n) {
      has = wall_consts_form(s, i, A.wbits[i]);
      A.wbits[i] = has ? (uint8_t)(A.wbits[i] | 0x80u) : (uint8_t)(A.wbits[i] & 0x7fu);
    }
    const unsigned m = __ballot_sync(0xffffffffu, has);
    if (lane == 0) wc[warp] = __popc(m);
    __syncthreads();
    if (threadIdx.x == 0) {
      int tot = 0;
      for (int w = 0; w < 8; w++) tot += wc[w];
      wbase = tot ? atomicAdd(&c->nmlist, tot) : 0;
    }
    __syncthreads();
    int off = wbase;
    for (int w = 0; w < warp; w++) off += wc[w];
    if (has) s.mlist[off + __popc(m & ((1u << lane) - 1u))] = i;
    __syncthreads();
  }
}

// ----------------------------------------------------------------------------
// rebuild: granular half list (Neighbor::granular_bin_no_newton,
// src/neigh_gran.cpp:485-644), 27-cell stencil with periodic images.  The
// count pass keeps each atom's first kStash entries (partner and image code
// in one int); the fill pass copies them into the atom's row, and searches
// again only for atoms with more.
// ----------------------------------------------------------------------------

// One run of candidates [jb, je) of the cell-sorted order, all with image
// code `code` (shift sv): FP32 prefilter of rsq <= (radsum*cdf + skin)^2;
// candidates clearly outside (or clearly inside) by more than the bound of
// the FP32 rounding are decided without FP64; the rest, and every entry the
// fill pass writes, use the exact FP64 test.  The next candidate is loaded while
// one is tested (526,000 atoms: 139 -> 102 us; nine lanes per atom, one per row
// of cells, took 256: the search is bound by its instructions, not its trips).
template <bool FILL>
__device__ __forceinline__ void pairs_scan(const Sys &s, const AtomArrays &A, const PairArrays &M, int i,
                                           const float4 &pi, double xi, double yi, double zi, double radi,
                                           float cdff, float skinf, float hi_f, float lo_f, int jb, int je,
                                           int code, const int sv[3], int &cnt, int &out, int out_end) {
  // image shifts by selection: an int-to-float conversion would issue on the FP64 pipe
  const float sxf = fshift(sv[0], s.prdf[0]), syf = fshift(sv[1], s.prdf[1]), szf = fshift(sv[2], s.prdf[2]);
  if (code == kNoShift) jb = max(jb, i + 1);
  float4 next = jb < je ? s.xf[jb] : pi;
  for (int j = jb; j < je; j++) {
    const float4 pj = next;
    if (j + 1 < je) next = s.xf[j + 1];  // on its way while this one is tested
    const float fx = pi.x - (pj.x + sxf), fy = pi.y - (pj.y + syf), fz = pi.z - (pj.z + szf);
    const float rsqf = fx * fx + fy * fy + fz * fz;
    const float csf = (pi.w + pj.w) * cdff + skinf;
    const float cs2f = csf * csf;
    if (rsqf > cs2f * hi_f) continue;
    if (code != kNoShift && !ghost_exists(s, A, j, sv)) continue;
    const bool clear_in = rsqf < cs2f * lo_f;
    if (!FILL && clear_in) {
      if (cnt < kStash) s.stash[(size_t)cnt * s.nmax + i] = j | (code << 24);
      cnt++;
      continue;
    }
    double xj = A.x[j], yj = A.y[j], zj = A.z[j];
    image(s, code, xj, yj, zj);
    const double delx = __dadd_rn(xi, -xj);
    const double dely = __dadd_rn(yi, -yj);
    const double delz = __dadd_rn(zi, -zj);
    const double rsq = rsq_rn(delx, dely, delz);
    const double radj = A.r[j];
    const double radsum = __dmul_rn(__dadd_rn(radi, radj), s.cdf);
    const double cs = __dadd_rn(radsum, s.skin);
    if (!(rsq <= __dmul_rn(cs, cs))) continue;
    if (!FILL) {
      if (cnt < kStash) s.stash[(size_t)cnt * s.nmax + i] = j | (code << 24);
      cnt++;
      continue;
    }
    if (out >= out_end) continue;  // count and fill passes agree; guard only
    const int p = out++;
    M.i[p] = i;
    M.j[p] = j;
    M.sh[p] = (uint8_t)code;
    if (s.nsys) M.rev[p] = -1;  // a fresh entry (source of copied ones: see pairs_atom)
  }
}

template <bool FILL>
__device__ __forceinline__ void pairs_atom(const Sys &s, const AtomArrays &A, const PairArrays &L,
                                           const PairArrays &M, int i) {
  {
    if (!sys_rebuilds(s, A.type[i])) {
      // a system that does not rebuild keeps its entries, in their order,
      // with partners renumbered by its block's shift (pairs never cross
      // systems); k_pair_init copies their history from the source entry
      const int sy = A.type[i] - 1;
      const int o = s.perm[i];
      const int eb = L.row[o], ee = row_end(s, L, o);
      if (!FILL) {
        s.pcount[i] = ee - eb;
        return;
      }
      const int shift = s.cell_start[sy * s.ens_ncell] - s.sys_start[sy];
      int out = M.row[i];
      for (int e = eb; e < ee; e++, out++) {
        M.i[out] = i;
        M.j[out] = L.j[e] + shift;
        M.sh[out] = L.sh[e];
        M.rev[out] = e;
      }
      return;
    }
    if (FILL) {  // the count pass kept the atom's entries unless it had more than kStash
      const int beg = M.row[i], ne = row_end(s, M, i) - beg;
      if (ne <= kStash) {
        for (int e = 0; e < ne; e++) {
          const int v = s.stash[(size_t)e * s.nmax + i];
          M.i[beg + e] = i;
          M.j[beg + e] = v & 0xffffff;
          M.sh[beg + e] = (uint8_t)(v >> 24);
          if (s.nsys) M.rev[beg + e] = -1;  // a fresh entry (source of copied ones: see above)
        }
        return;
      }
    }
    const double xi = A.x[i], yi = A.y[i], zi = A.z[i];
    const double radi = A.r[i];
    const int ci[3] = {cell_coord(s, xi, 0), cell_coord(s, yi, 1), cell_coord(s, zi, 2)};
    const float4 pi = s.xf[i];
    const int cell_base = s.ens_ncell ? (A.type[i] - 1) * s.ens_ncell : 0;
    const float cdff = s.cdff, skinf = s.skinf;
    const float hi_f = 1.0f + s.pf_margin, lo_f = 1.0f - s.pf_margin;
    int cnt = 0;
    int out = FILL ? M.row[i] : 0;
    const int out_end = FILL ? row_end(s, M, i) : 0;
    // per dimension: the neighbour coordinate, image shift and validity of
    // the offsets -1, 0, +1
    int nb[3][3], sv3[3][3];
    bool ok3[3][3];
#pragma unroll
    for (int d = 0; d < 3; d++) {
#pragma unroll
      for (int k = 0; k < 3; k++) {
        const int o = k - 1;
        int cc = ci[d] + o, sv = 0;
        bool ok = !(s.nc[d] == 1 && o != 0);
        if (cc < 0) {
          ok = ok && s.periodic[d];
          cc += s.nc[d];
          sv = -1;
        } else if (cc >= s.nc[d]) {
          ok = ok && s.periodic[d];
          cc -= s.nc[d];
          sv = 1;
        }
        nb[d][k] = cc;
        sv3[d][k] = sv;
        ok3[d][k] = ok;
      }
    }
    // the 27 cells in the stencil's order (z, then y, then x offsets): along
    // x the unwrapped cells of a row are consecutive, so their atoms are one
    // contiguous run of the cell-sorted order, scanned in one loop (the same
    // candidates in the same order as cell by cell); a cell that wraps
    // around a periodic x boundary is scanned alone, with its image shift
    const bool lwrap = ok3[0][0] && sv3[0][0] != 0, rwrap = ok3[0][2] && sv3[0][2] != 0;
    const int x0 = (ok3[0][0] && !lwrap) ? nb[0][0] : nb[0][1];
    const int x1 = (ok3[0][2] && !rwrap) ? nb[0][2] : nb[0][1];
#pragma unroll
    for (int kz = 0; kz < 3; kz++) {
#pragma unroll
      for (int ky = 0; ky < 3; ky++) {
        if (!ok3[2][kz] || !ok3[1][ky]) continue;
        const int rowb = s.nc[0] * (nb[1][ky] + s.nc[1] * nb[2][kz]) + cell_base;
        const int syz = 3 * (sv3[1][ky] + 1) + 9 * (sv3[2][kz] + 1);
        if (lwrap) {
          const int sv[3] = {-1, sv3[1][ky], sv3[2][kz]};
          pairs_scan<FILL>(s, A, M, i, pi, xi, yi, zi, radi, cdff, skinf, hi_f, lo_f, s.cell_start[rowb + nb[0][0]],
                           s.cell_start[rowb + nb[0][0] + 1], syz, sv, cnt, out, out_end);
        }
        {
          const int sv[3] = {0, sv3[1][ky], sv3[2][kz]};
          pairs_scan<FILL>(s, A, M, i, pi, xi, yi, zi, radi, cdff, skinf, hi_f, lo_f, s.cell_start[rowb + x0],
                           s.cell_start[rowb + x1 + 1], 1 + syz, sv, cnt, out, out_end);
        }
        if (rwrap) {
          const int sv[3] = {1, sv3[1][ky], sv3[2][kz]};
          pairs_scan<FILL>(s, A, M, i, pi, xi, yi, zi, radi, cdff, skinf, hi_f, lo_f, s.cell_start[rowb + nb[0][2]],
                           s.cell_start[rowb + nb[0][2] + 1], 2 + syz, sv, cnt, out, out_end);
        }
      }
    }
    if (!FILL) s.pcount[i] = cnt;
  }
}

template <bool FILL>
__global__ void k_pairs(Sys s) {
  Ctrl *c = s.ctrl;
  if (gated(c)) return;
  const AtomArrays &A = s.atoms[0];
  const PairArrays &L = s.pairs[0];  // old list (old atom order)
  const PairArrays &M = s.pairs[1];  // new list
  // count: in place for the rebuilding systems' atoms (pmode); fill: also
  // in place for their segments (lmode)
  if (FILL ? ens_list_partial(s, c) : ens_partial(s, c)) {
    GRID_STRIDE(t, c->nra) pairs_atom<FILL>(s, A, L, M, ens_atom(s, c, t));
    return;
  }
  const int n = c->n_new;
  const int total = FILL ? n : s.nmax + 1;
  GRID_STRIDE(i, total) {
    if (!FILL && i >= n) {
      s.pcount[i] = 0;
      continue;
    }
    pairs_atom<FILL>(s, A, L, M, i);
  }
}

// Per new list entry (one thread each, dense): exact distance, history
// carry-over, per-pair contact constants, reverse-list count.  The carry-over
// is the reference's (pre_exchange partner lists + the lookup of
// src/neigh_gran.cpp:590-620): the new entry's reference owner R (lower lidx
// of an owned pair, else i) takes its partner-list entry for the other atom:
// its own old entry, or the partner copy of an old owned pair, in which the
// values registered with newtonflag 1 change sign.  The shear is then
// expressed in the list's own orientation; history is carried only when the
// pair is within radsum*cdf at the build.
__device__ __forceinline__ void pair_init_entry(const Sys &s, const AtomArrays &A, const PairArrays &L,
                                                const PairArrays &M, int p) {
  {
    const int code = M.sh[p];
    if (code == kHole) return;  // an unused entry of an ensemble segment
    const int i = M.i[p], j = M.j[p];
    const int src = s.nsys ? M.rev[p] : -1;
    if (src >= 0) {  // kept entry of a system that does not rebuild: as it was
      M.flag[p] = L.flag[src];
      for (int d = 0; d < s.dnum; d++) M.hist[(size_t)d * s.pcap + p] = L.hist[(size_t)d * s.pcap + src];
      M.reff[p] = L.reff[src];
      M.c0[p] = L.c0[src];
      M.c1[p] = L.c1[src];
      if (code == kNoShift) atomicAdd(&s.rev_count[j], 1);
      return;
    }
    double xj = A.x[j], yj = A.y[j], zj = A.z[j];
    image(s, code, xj, yj, zj);
    const double rsq = rsq_rn(__dadd_rn(A.x[i], -xj), __dadd_rn(A.y[i], -yj), __dadd_rn(A.z[i], -zj));
    const double radi = A.r[i], radj = A.r[j];
    const double radsum = __dmul_rn(__dadd_rn(radi, radj), s.cdf);
    int e = -1;
    double ssign = 1.0;
    bool quirk = false;
    if (rsq < __dmul_rn(radsum, radsum)) {
      const bool rj = s.bond && code == kNoShift && A.lidx[i] > A.lidx[j];
      bool fl;
      e = rj ? find_old(s, L, s.perm[j], s.perm[i], fl) : find_old(s, L, s.perm[i], s.perm[j], fl);
      ssign = (fl ? -1.0 : 1.0) * (rj ? -1.0 : 1.0);
      quirk = s.bond && e >= 0 && !rj && code != kNoShift && L.sh[e] == kNoShift && A.lidx[i] > A.lidx[j];
    }
    M.flag[p] = e >= 0 ? 1 : 0;
    double sh[kDnumShear];
    for (int d = 0; d < kDnumShear; d++) sh[d] = e >= 0 ? ssign * L.hist[(size_t)d * s.pcap + e] : 0.0;
    for (int d = 0; d < kDnumShear; d++) M.hist[(size_t)d * s.pcap + p] = sh[d];
    for (int d = kDnumShear; d < s.dnum; d++) {
      double hv = e >= 0 ? L.hist[(size_t)d * s.pcap + e] : 0.0;
      if (quirk && d >= kDnumShear + 5 && d <= kDnumShear + 13) hv = -hv;
      M.hist[(size_t)d * s.pcap + p] = hv;
    }
    const double mi = A.m[i], mj = A.m[j];
    const double meff = mi * mj / (mi + mj);
    const double reff = radi * radj / (radi + radj);
    const TypePair tp = load_typepair(s.params, s.ntypes, A.type[i], A.type[j]);
    double c0, c1;
    if (s.normal == kHertz) contact_consts<kHertz>(tp, meff, reff, s.charVel, s.tdamp, c0, c1);
    else contact_consts<kHooke>(tp, meff, reff, s.charVel, s.tdamp, c0, c1);
    M.reff[p] = reff;
    M.c0[p] = c0;
    M.c1[p] = c1;
    if (code == kNoShift) atomicAdd(&s.rev_count[j], 1);
  }
}

__global__ void k_pair_init(Sys s) {
  Ctrl *c = s.ctrl;
  if (gated(c)) return;
  const AtomArrays &A = s.atoms[0];
  const PairArrays &L = s.pairs[0];  // old list (old atom order)
  const PairArrays &M = s.pairs[1];  // new list
  if (ens_list_partial(s, c)) {
    GRID_STRIDE(u, c->ncr) pair_init_entry(s, A, L, M, ens_entry(s, c, u));
    return;
  }
  const int np = c->np_new;
  GRID_STRIDE(p, np) pair_init_entry(s, A, L, M, p);
}

// after the pair-count scan: capacity check; halts on overflow
__global__ void k_pairs_total(Sys s) {
  Ctrl *c = s.ctrl;
  if (gated(c)) return;
  // ensembles: the segments' extent (k_ens_plan or k_ens_layout)
  const int np = s.nsys ? c->np_new : s.pairs[1].row[s.nmax];
  c->np_new = np;
  if (np > s.pcap) {
    c->status = kStatPairOverflow;
    c->halt = 1;
    c->halt_step = 1;
  }
}

__device__ __forceinline__ void rev_fill_entry(const Sys &s, const PairArrays &M, int p) {
  if (M.sh[p] != kNoShift) return;  // image entries and unused ones
  const int j = M.j[p];
  M.rev[M.rev_start[j] + atomicAdd(&s.rev_fill[j], 1)] = p;
}

__global__ void k_rev_fill(Sys s) {
  Ctrl *c = s.ctrl;
  if (gated(c)) return;
  const PairArrays &M = s.pairs[1];
  if (ens_list_partial(s, c)) {
    GRID_STRIDE(u, c->ncr) rev_fill_entry(s, M, ens_entry(s, c, u));
    return;
  }
  const int np = c->np_new;
  GRID_STRIDE(p, np) rev_fill_entry(s, M, p);
}

__device__ __forceinline__ void rev_sort_atom(const Sys &s, const PairArrays &M, int i) {
  const int b = M.rev_start[i], e = rev_end(s, M, i);
  if (e - b <= 8) {  // in registers: one load's wait instead of one per comparison
    int v[8];
#pragma unroll
    for (int k = 0; k < 8; k++) v[k] = b + k < e ? M.rev[b + k] : 0x7fffffff;
#pragma unroll
    for (int k = 0; k < 8; k++)
#pragma unroll
      for (int m = k & 1; m < 7; m += 2) {
        const int lo = min(v[m], v[m + 1]), hi = max(v[m], v[m + 1]);
        v[m] = lo;
        v[m + 1] = hi;
      }
#pragma unroll
    for (int k = 0; k < 8; k++)
      if (b + k < e) M.rev[b + k] = v[k];
    return;
  }
  for (int k = b + 1; k < e; k++) {
    const int v = M.rev[k];
    int m = k - 1;
    while (m >= b && M.rev[m] > v) {
      M.rev[m + 1] = M.rev[m];
      m--;
    }
    M.rev[m + 1] = v;
  }
}

__global__ void k_rev_sort(Sys s) {
  Ctrl *c = s.ctrl;
  if (gated(c)) return;
  const PairArrays &M = s.pairs[1];
  if (ens_list_partial(s, c)) {
    GRID_STRIDE(t, c->nra) rev_sort_atom(s, M, ens_atom(s, c, t));
    return;
  }
  const int n = c->n_new;
  GRID_STRIDE(i, n) rev_sort_atom(s, M, i);
}

__device__ __forceinline__ void copy_entry(const Sys &s, const PairArrays &L, const PairArrays &M, int p) {
  const int i = M.i[p], j = M.j[p], flag = M.flag[p], rev = M.rev[p];
  const uint8_t sh = M.sh[p];
  const size_t P = s.pcap;
  double *const to[6] = {L.reff, L.c0, L.c1, L.hist, L.hist + P, L.hist + 2 * P};
  const double *const from[6] = {M.reff, M.c0, M.c1, M.hist, M.hist + P, M.hist + 2 * P};
  copy_values(to, from, p, p);
  L.i[p] = i;
  L.j[p] = j;
  L.sh[p] = sh;
  L.flag[p] = flag;
  L.rev[p] = rev;
  // the bond's values (dnum - 3: none or a multiple of four)
  for (int d = kDnumShear; d < s.dnum; d += 4) {
    double *const h = L.hist + (size_t)d * P;
    const double *const m = M.hist + (size_t)d * P;
    double *const hto[4] = {h, h + P, h + 2 * P, h + 3 * P};
    const double *const hfrom[4] = {m, m + P, m + 2 * P, m + 3 * P};
    copy_values(hto, hfrom, p, p);
  }
}

__device__ __forceinline__ void copy_rows(const Sys &s, const PairArrays &L, const PairArrays &M, int i) {
  L.row[i] = M.row[i];
  L.rev_start[i] = M.rev_start[i];
  if (s.nsys) {
    L.rowe[i] = M.rowe[i];
    L.reve[i] = M.reve[i];
  }
}

__global__ void k_copy_pairs(Sys s) {
  Ctrl *c = s.ctrl;
  if (gated(c)) return;
  const PairArrays &L = s.pairs[0];
  const PairArrays &M = s.pairs[1];
  if (ens_list_partial(s, c)) {  // the rebuilt segments (with their unused entries) and rows
    GRID_STRIDE(u, c->ncr) copy_entry(s, L, M, ens_entry(s, c, u));
    GRID_STRIDE(t, c->nra) copy_rows(s, L, M, ens_atom(s, c, t));
    return;
  }
  const int np = c->np_new;
  const int nrow = s.nmax + 1;
  const int tot = np > nrow ? np : nrow;
  GRID_STRIDE(p, tot) {
    if (p < np) copy_entry(s, L, M, p);
    if (p < nrow) copy_rows(s, L, M, p);
  }
}

__global__ void k_finish_rebuild(Sys s) {
  Ctrl *c = s.ctrl;
  if (gated(c)) return;
  int live = 0;
  for (int k = threadIdx.x; k < s.nsys; k += blockDim.x) {
    if (s.sys_reb[k]) {
      s.sys_nreb[k]++;
      s.sys_ago[k] = 0;
    }
    s.sys_start[k] = s.cell_start[k * s.ens_ncell];
    live += s.seg_used[k];
  }
  int tot = 0;
  if (s.nsys) block_excl_scan(live, &tot);
  __syncthreads();  // every thread has read the gate before it changes
  if (threadIdx.x == 0) {
    if (s.nsys) {
      s.sys_start[s.nsys] = s.cell_start[s.ncell];
      c->seg_ok = 1;
      c->np_live = tot;
      if (c->pmode) {
        if (c->lmode) c->ens_inplace++;
        else c->ens_relayout++;
      }
    }
    c->lost += c->lost_step;
    c->n = c->n_new;
    c->np = c->np_new;
    if (!s.nsys) c->np_live = c->np_new;
    c->nrebuilds++;
    c->ago = 0;
    c->hold = c->loop_left > 0 ? kHoldNone : kHoldDone;
  }
}

// entries of a grid-stride walk over the list, 32 per warp
struct GridTiles {
  long base, stride;
  __device__ __forceinline__ GridTiles(int block) {
    base = (long)blockIdx.x * block + (threadIdx.x & ~31);
    stride = (long)gridDim.x * block;
    base -= stride;
  }
  __device__ __forceinline__ int operator()() {
    base += stride;
    return base < 0x7fffffffL ? (int)base : 0x7fffffff;
  }
};

template <int NORMAL, bool ROLL, bool BOND>
__global__ void __launch_bounds__(kBandTile, 4) k_pair(Sys s, int shearupdate, int gate) {
  __shared__ BandQueue q[kBandTile / 32];
  __shared__ BandRest<kBandTile> rest;
  Ctrl *c = s.ctrl;
  if (c->halt || (gate && c->hold)) return;
  const long long ntimestep = BOND ? c->ntimestep : 0;
  BandQueue &mine = q[threadIdx.x >> 5];
  const int qn = band_tiles<NORMAL, ROLL, BOND>(s, c->np, shearupdate, ntimestep, mine, GridTiles(kBandTile));
  band_rest<NORMAL, ROLL, BOND, kBandTile>(s, qn, shearupdate, ntimestep, mine, rest);
}

template <int NORMAL, bool ROLL, int MINB>
__global__ void __launch_bounds__(kPairTile, MINB) k_pair_pf(Sys s, int shearupdate, int gate) {
  __shared__ int qbuf[kPairTile / 32][64];
  __shared__ PfRest rest;
  Ctrl *c = s.ctrl;
  if (c->halt || (gate && c->hold)) return;
  int *q = qbuf[threadIdx.x >> 5];
  const int qn = pf_tiles<NORMAL, ROLL>(s, c->np, shearupdate, q, GridTiles(kPairTile));
  pf_rest<NORMAL, ROLL>(s, qn, shearupdate, q, rest);
}

template <int NORMAL>
__global__ void __launch_bounds__(kWallTile *kWallWarps) k_wall_force(Sys s, int shearupdate, int cap, int gate) {
  extern __shared__ double wshared[];  // per warp: res [cap * kWallRes]; then st, qa, qq of every warp
  Ctrl *c = s.ctrl;
  if (c->halt || (gate && c->hold)) return;
  const int warp = threadIdx.x >> 5;
  WallQueue w;
  w.res = wshared + (size_t)warp * cap * kWallRes;
  w.st = reinterpret_cast<int *>(wshared + (size_t)kWallWarps * cap * kWallRes) + warp * cap;
  w.qa = reinterpret_cast<unsigned char *>(wshared + (size_t)kWallWarps * cap * kWallRes) +
         (size_t)kWallWarps * cap * 4 + (size_t)warp * 2 * cap;
  w.qq = w.qa + cap;
  const int nl = c->nmlist;
  bool meshbad = false;
  for (int base = (blockIdx.x * kWallWarps + warp) * kWallTile; base < nl;
       base += gridDim.x * kWallWarps * kWallTile)
    wall_tile<NORMAL>(s, s.atoms[0], base, nl, shearupdate, cap, w, meshbad);
  if (__any_sync(0xffffffffu, meshbad) && (threadIdx.x & 31) == 0) atomicExch(&c->status, kStatMeshSlots);
}

// Graph steps without moving meshes: the last block of k_particle to finish
// takes the step's rebuild decision (LoopCond::on), as k_decide_loop does after
// it otherwise (one node and one dependency fewer per step).
// the flags of a block's atoms, and (lp.on) the decision by the last block
__device__ __forceinline__ void particle_end(const Sys &s, Ctrl *c, bool moved, bool bad, const LoopCond &lp) {
  __shared__ int last_block;
  if (__any_sync(0xffffffffu, moved) && (threadIdx.x & 31) == 0) atomicOr(&c->moved, 1);
  if (__any_sync(0xffffffffu, bad) && (threadIdx.x & 31) == 0) {
    atomicExch(&c->status, kStatNan);
  }
  if (lp.on) {  // the last block to finish decides (k_decide_loop's work)
    __syncthreads();
    if (threadIdx.x == 0) {
      __threadfence();
      last_block = atomicAdd(&c->pdone, 1) == (int)gridDim.x - 1;
    }
    __syncthreads();
    if (last_block) {
      __threadfence();
      if (threadIdx.x == 0) {
        c->pdone = 0;
        c->ntimestep++;
      }
      const int reb = decide_rebuild(s, c);
      if (threadIdx.x == 0) loop_decided(c, lp, reb);
    }
  }
}

template <bool GATHER, bool FINAL, bool INITIAL>
__global__ void __launch_bounds__(kParticleMaxThreads, 4) k_particle(Sys s, LoopCond lp) {
  __shared__ ParticleShared<kParticleMaxThreads> sm;
  Ctrl *c = s.ctrl;
  if (loop_held(c, lp, (lp.on || lp.gate) && blockIdx.x == 0 && threadIdx.x == 0)) return;
  const int n = c->n;
  bool moved = false, bad = false;
  for (int base = blockIdx.x * blockDim.x; base < n; base += gridDim.x * blockDim.x) {
    const int i = base + threadIdx.x;
    particle_tile(s, sm, i, i < n, GATHER, FINAL, INITIAL, moved, bad);
  }
  particle_end(s, c, moved, bad, lp);
}

// The first step of a graph launch: from stored forces (a call's first step),
// or gathering the previous step's (continuing a call after a capacity grew
// or atoms were inserted), as Ctrl::step_phase says.
__global__ void __launch_bounds__(kParticleMaxThreads, 4) k_particle_start(Sys s, LoopCond lp) {
  __shared__ ParticleShared<kParticleMaxThreads> sm;
  Ctrl *c = s.ctrl;
  if (loop_held(c, lp, (lp.on || lp.gate) && blockIdx.x == 0 && threadIdx.x == 0)) return;
  const int n = c->n;
  const bool gather = c->step_phase != kStepFirst;
  bool moved = false, bad = false;
  for (int base = blockIdx.x * blockDim.x; base < n; base += gridDim.x * blockDim.x) {
    const int i = base + threadIdx.x;
    particle_tile(s, sm, i, i < n, gather, gather, true, moved, bad);
  }
  particle_end(s, c, moved, bad, lp);
}

// ----------------------------------------------------------------------------
// insertion (dem_insert_atoms): new atoms are staged into the unused slots
// [first, first + k) of atom buffer 0 between steps and join the system at
// the next step after its initial integration, with a forced rebuild, as
// FixInsert::pre_exchange adds them in the reference (src/fix_insert.cpp,
// pre_exchange with next_reneighbor = the insertion step)
// ----------------------------------------------------------------------------

__global__ void k_insert_stage(Sys s, InsertStage in, int first, int k, int lidx0) {
  const AtomArrays &A = s.atoms[0];
  const size_t nmax = s.nmax;
  GRID_STRIDE(q, k) {
    const int i = first + q;
    A.x[i] = in.x[3 * q]; A.y[i] = in.x[3 * q + 1]; A.z[i] = in.x[3 * q + 2];
    A.vx[i] = in.v[3 * q]; A.vy[i] = in.v[3 * q + 1]; A.vz[i] = in.v[3 * q + 2];
    A.wx[i] = in.w[3 * q]; A.wy[i] = in.w[3 * q + 1]; A.wz[i] = in.w[3 * q + 2];
    A.fx[i] = A.fy[i] = A.fz[i] = 0.0;
    A.tx[i] = A.ty[i] = A.tz[i] = 0.0;
    A.xh[i] = A.x[i]; A.yh[i] = A.y[i]; A.zh[i] = A.z[i];
    A.r[i] = in.r[q]; A.m[i] = in.m[q];
    A.dtfm[i] = in.dtfm[q]; A.dtir[i] = in.dtir[q];
    A.type[i] = in.type[q]; A.tag[i] = in.tag[q]; A.lidx[i] = lidx0 + q;
    for (int w = 0; w < s.nplanes; w++)
      for (int d = 0; d < 3; d++) A.whist[(size_t)(w * 3 + d) * nmax + i] = 0.0;
    A.wbits[i] = 0;
    A.fmx[i] = A.fmy[i] = A.fmz[i] = A.tmx[i] = A.tmy[i] = A.tmz[i] = 0.0;
    const float4 f = make_float4((float)A.x[i], (float)A.y[i], (float)A.z[i], (float)A.r[i]);
    s.xf[i] = f;
    s.xhf[i] = f;
    for (int m = 0; m < s.nmeshes; m++) {
      const MeshDev &M = s.meshes[m];
      M.cand_n[i] = 0;
      M.nslot[0][i] = 0;
      M.npart[0][i] = 0;
      for (int u = 0; u < M.ccap; u++) {
        M.slot_tri[0][(size_t)u * nmax + i] = -1;
        for (int d = 0; d < 3; d++) M.slot_hist[0][(size_t)(3 * u + d) * nmax + i] = 0.0;
      }
    }
  }
}

// the new atoms get empty rows in the current (old) list, so that the
// rebuild's history carry-over finds nothing for them
__global__ void k_insert_commit(Sys s, int k) {
  __shared__ int n_old;
  Ctrl *c = s.ctrl;
  if (c->halt) return;
  if (threadIdx.x == 0) n_old = c->n;
  __syncthreads();
  const PairArrays &L = s.pairs[0];
  const int r = L.row[n_old], rv = L.rev_start[n_old];
  for (int q = threadIdx.x; q < k; q += blockDim.x) {
    L.row[n_old + 1 + q] = r;
    L.rev_start[n_old + 1 + q] = rv;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    c->n = n_old + k;
    c->force_rebuild = 1;
  }
}

// ----------------------------------------------------------------------------
// atom transfer: caller AoS <-> device SoA (dem_upload_atoms, dem_download_atoms)
// ----------------------------------------------------------------------------

__global__ void k_upload_atoms(Sys s, AtomsIn in, int n, double dtf, double dtfrotate, UploadCheck *chk) {
  const AtomArrays &A = s.atoms[0];
  const size_t nmax = s.nmax;
  unsigned long long rmin = ~0ull, rmax = 0ull;
  int bad_type = 0, bad_value = 0, nonfinite = 0;
  GRID_STRIDE(i, n) {
    const double x0 = in.x[3 * i], x1 = in.x[3 * i + 1], x2 = in.x[3 * i + 2];
    const double v0 = in.v[3 * i], v1 = in.v[3 * i + 1], v2 = in.v[3 * i + 2];
    const double w0 = in.w[3 * i], w1 = in.w[3 * i + 1], w2 = in.w[3 * i + 2];
    const double r = in.r[i], m = in.m[i];
    const int t = in.type[i];
    bad_type += (t < 1 || t > s.ntypes) ? 1 : 0;
    const bool okv = r > 0.0 && m > 0.0 && isfinite(r) && isfinite(m);
    bad_value += okv ? 0 : 1;
    const bool fin = isfinite(x0) && isfinite(x1) && isfinite(x2) && isfinite(v0) && isfinite(v1) &&
                     isfinite(v2) && isfinite(w0) && isfinite(w1) && isfinite(w2);
    nonfinite += fin ? 0 : 1;
    A.x[i] = x0; A.y[i] = x1; A.z[i] = x2;
    A.vx[i] = v0; A.vy[i] = v1; A.vz[i] = v2;
    A.wx[i] = w0; A.wy[i] = w1; A.wz[i] = w2;
    A.r[i] = r; A.m[i] = m;
    A.type[i] = t; A.tag[i] = in.tag[i]; A.lidx[i] = i;
    // FixNVESphere per-atom factors, as its init/initial_integrate form them
    // (src/fix_nve_sphere.cpp:150-178): dtf/(m*(1+CAdd/rho)) with no added
    // mass, dtfrotate/(r*r*m)
    A.dtfm[i] = dtf / (m * (1. + 0.0));
    A.dtir[i] = dtfrotate / (r * r * m);
    A.fx[i] = A.fy[i] = A.fz[i] = 0.0;
    A.tx[i] = A.ty[i] = A.tz[i] = 0.0;
    A.xh[i] = A.yh[i] = A.zh[i] = 0.0;
    for (int k = 0; k < 3 * s.nplanes; k++) A.whist[(size_t)k * nmax + i] = 0.0;
    A.wbits[i] = 0;
    A.fmx[i] = A.fmy[i] = A.fmz[i] = A.tmx[i] = A.tmy[i] = A.tmz[i] = 0.0;
    if (okv) {
      const unsigned long long b = (unsigned long long)__double_as_longlong(r);
      rmin = b < rmin ? b : rmin;
      rmax = b > rmax ? b : rmax;
    }
  }
  // positive doubles order as their bit patterns
  for (int o = 16; o > 0; o >>= 1) {
    const unsigned long long a = __shfl_down_sync(0xffffffffu, rmin, o);
    const unsigned long long b = __shfl_down_sync(0xffffffffu, rmax, o);
    rmin = a < rmin ? a : rmin;
    rmax = b > rmax ? b : rmax;
    bad_type += __shfl_down_sync(0xffffffffu, bad_type, o);
    bad_value += __shfl_down_sync(0xffffffffu, bad_value, o);
    nonfinite += __shfl_down_sync(0xffffffffu, nonfinite, o);
  }
  if ((threadIdx.x & 31) == 0) {
    if (rmin != ~0ull) atomicMin(&chk->rmin, rmin);
    if (rmax) atomicMax(&chk->rmax, rmax);
    if (bad_type) atomicAdd(&chk->bad_type, bad_type);
    if (bad_value) atomicAdd(&chk->bad_value, bad_value);
    if (nonfinite) atomicAdd(&chk->nonfinite, nonfinite);
  }
}

// One block writes a tile of kDownTile atoms. Each 3-vector goes through
// shared memory so that a warp's stores cover 256 contiguous bytes of the
// caller's array: strided stores (one component per instruction) left two
// thirds of every line they touched for later instructions, which over the
// host link took 2.9 ms for 1M atoms against 0.8 ms this way.
constexpr int kDownTile = 256;

__global__ void __launch_bounds__(kDownTile) k_download_atoms(Sys s, AtomsOut out, int n) {
  const AtomArrays &A = s.atoms[0];
  __shared__ double tile[3 * kDownTile];
  double *dst[5] = {out.x, out.v, out.w, out.f, out.t};
  const double *src[5][3] = {{A.x, A.y, A.z}, {A.vx, A.vy, A.vz}, {A.wx, A.wy, A.wz},
                             {A.fx, A.fy, A.fz}, {A.tx, A.ty, A.tz}};
  for (int b = blockIdx.x; (long)b * kDownTile < n; b += gridDim.x) {
    const int a0 = b * kDownTile, cnt = min(kDownTile, n - a0);
    const int t = threadIdx.x, i = a0 + t;
    for (int k = 0; k < 5; k++) {
      if (!dst[k]) continue;  // the same for the whole block
      if (t < cnt) {
        tile[3 * t] = src[k][0][i];
        tile[3 * t + 1] = src[k][1][i];
        tile[3 * t + 2] = src[k][2][i];
      }
      __syncthreads();
      double *base = dst[k] + 3 * (size_t)a0;
      for (int q = t; q < 3 * cnt; q += kDownTile) base[q] = tile[q];
      __syncthreads();
    }
    if (t < cnt) {
      if (out.r) out.r[i] = A.r[i];
      if (out.m) out.m[i] = A.m[i];
      if (out.tag) out.tag[i] = A.tag[i];
      if (out.type) out.type[i] = A.type[i];
    }
  }
}

int launch_upload_atoms(const Sys &s, const AtomsIn &in, int n, double dtf, double dtfrotate, UploadCheck *chk,
                        cudaStream_t st) {
  if (n <= 0) return 0;
  k_upload_atoms<<<std::min((n + 255) / 256, 152 * 16), 256, 0, st>>>(s, in, n, dtf, dtfrotate, chk);
  return 1;
}

int launch_download_atoms(const Sys &s, const AtomsOut &out, int n, cudaStream_t st) {
  if (n <= 0) return 0;
  k_download_atoms<<<std::min((n + kDownTile - 1) / kDownTile, 152 * 8), kDownTile, 0, st>>>(s, out, n);
  return 1;
}

int launch_insert_stage(const Sys &s, const InsertStage &in, int first, int k, int lidx0, cudaStream_t st) {
  k_insert_stage<<<(k + 127) / 128, 128, 0, st>>>(s, in, first, k, lidx0);
  return 1;
}

int launch_insert_commit(const Sys &s, int k, cudaStream_t st) {
  k_insert_commit<<<1, 256, 0, st>>>(s, k);
  return 1;
}

// ----------------------------------------------------------------------------
// diagnostics (dem_get_diagnostics): deterministic per-block partial sums,
// added in block order by the host
// ----------------------------------------------------------------------------

constexpr int kDiagBlock = 256;

__device__ __forceinline__ double block_sum(double v, double *sm) {
  sm[threadIdx.x] = v;
  __syncthreads();
  for (int st = kDiagBlock / 2; st > 0; st >>= 1) {
    if (threadIdx.x < st) sm[threadIdx.x] += sm[threadIdx.x + st];
    __syncthreads();
  }
  const double r = sm[0];
  __syncthreads();
  return r;
}

// ComputeKE (sum m v^2), ComputeERotateSphere (sum w^2 r^2 m) and the solid
// volume (sum r^3) of the atoms whose centre lies in [lo, hi)
__global__ void __launch_bounds__(kDiagBlock) k_diag_atoms(Sys s, double3 lo, double3 hi, double *part) {
  __shared__ double sm[kDiagBlock];
  const AtomArrays &A = s.atoms[0];
  const int n = s.ctrl->n;
  double ke = 0.0, er = 0.0, vol = 0.0;
  GRID_STRIDE(i, n) {
    const double m = A.m[i], r = A.r[i];
    ke += m * (A.vx[i] * A.vx[i] + A.vy[i] * A.vy[i] + A.vz[i] * A.vz[i]);
    er += (A.wx[i] * A.wx[i] + A.wy[i] * A.wy[i] + A.wz[i] * A.wz[i]) * r * r * m;
    const double x = A.x[i], y = A.y[i], z = A.z[i];
    if (x >= lo.x && x < hi.x && y >= lo.y && y < hi.y && z >= lo.z && z < hi.z) vol += r * r * r;
  }
  ke = block_sum(ke, sm);
  er = block_sum(er, sm);
  vol = block_sum(vol, sm);
  if (threadIdx.x == 0) {
    part[3 * blockIdx.x] = ke;
    part[3 * blockIdx.x + 1] = er;
    part[3 * blockIdx.x + 2] = vol;
  }
}

// per-wall force sums over the listed wall atoms: part[(blk*nw + w)*3 + d]
__global__ void __launch_bounds__(kDiagBlock) k_diag_walls(Sys s, int nw, double *part) {
  __shared__ double sm[kDiagBlock];
  const int nl = s.ctrl->nmlist;
  for (int w = 0; w < nw; w++)
    for (int d = 0; d < 3; d++) {
      const double *wf = s.wforce + (size_t)(3 * w + d) * s.nmax;
      double acc = 0.0;
      GRID_STRIDE(q, nl) acc += wf[s.mlist[q]];
      acc = block_sum(acc, sm);
      if (threadIdx.x == 0) part[((size_t)blockIdx.x * nw + w) * 3 + d] = acc;
    }
}

// list entries with a contact force in the last force evaluation
__global__ void k_diag_contacts(Sys s, unsigned long long *cnt) {
  const int np = s.ctrl->np;
  unsigned long long c = 0;
  GRID_STRIDE(p, np) c += s.active[p] ? 1ull : 0ull;
  for (int o = 16; o > 0; o >>= 1) c += __shfl_down_sync(0xffffffffu, c, o);
  if ((threadIdx.x & 31) == 0 && c) atomicAdd(cnt, c);
}

int launch_diagnostics(const Sys &s, const LaunchCfg &lc, const double lo[3], const double hi[3], double *part_atoms,
                       double *part_walls, unsigned long long *contacts, int nblocks, cudaStream_t st) {
  const int nw = s.nplanes + s.nmeshes;
  k_diag_atoms<<<nblocks, kDiagBlock, 0, st>>>(s, make_double3(lo[0], lo[1], lo[2]),
                                               make_double3(hi[0], hi[1], hi[2]), part_atoms);
  if (nw > 0) k_diag_walls<<<nblocks, kDiagBlock, 0, st>>>(s, nw, part_walls);
  cudaMemsetAsync(contacts, 0, sizeof(unsigned long long), st);
  const int gc = (int)std::max<long>(1, std::min<long>(((long)s.pcap + 255) / 256, lc.max_grid));
  k_diag_contacts<<<gc, 256, 0, st>>>(s, contacts);
  return nw > 0 ? 3 : 2;
}

// ----------------------------------------------------------------------------
// launchers
// ----------------------------------------------------------------------------

static inline int grid_for(long n, int block, int cap) {
  long g = (n + block - 1) / block;
  if (g < 1) g = 1;
  if (g > cap) g = cap;
  return (int)g;
}

// chunks of 4096 items up to which k_scan_flat scans; its last block reads the
// whole array, a cost that grows with the chunks (1: 3.5 us, 9: 5.4, 29: 9.0),
// while the three launches take 18 us at 37 chunks (4.6 + 2.5 + 10.9)
constexpr int kScanFlat = 32;

// in and out do not overlap
int scan_exclusive(const Sys &s, const int *in, int *out, int len, int *tmp, int gate,
                   cudaStream_t st) {
  const int nb = (len + 4095) / 4096;
  if (nb <= kScanFlat) {
    k_scan_flat<<<nb, 1024, 0, st>>>(s, in, out, len, gate);
    return 1;
  }
  k_scan_blocks<<<nb, 1024, 0, st>>>(s, in, out, len, tmp, gate);
  // nb <= 4096: one block scans the block totals in place
  k_scan_blocks<<<1, 1024, 0, st>>>(s, tmp, tmp, nb, nullptr, gate);
  k_scan_add<<<nb, 256, 0, st>>>(s, out, len, tmp, gate);
  return 3;
}

int launch_wall_consts(const Sys &s, const LaunchCfg &lc, cudaStream_t st) {
  if (s.nplanes == 0 && s.nmeshes == 0) return 0;
  k_wall_consts<<<grid_for(s.nmax, 256, lc.max_grid), 256, 0, st>>>(s);
  return 1;
}

// one block: one thread per ensemble system (up to 256 at a time)
static inline int sys_threads(const Sys &s) { return s.nsys > 32 ? 256 : 32; }

// Ensemble rebuild: in place for the rebuilding systems where that is
// possible (see k_ens_plan), else the whole list; the kernels of both paths
// are launched and each runs the path that Ctrl selects.  Stage 1 resumes
// after a pair-capacity overflow (whole-list path only).
static int launch_rebuild_ens(const Sys &s, const LaunchCfg &lc, cudaStream_t st, int stage) {
  int nl = 0;
  const int B = 256;
  const int gN = grid_for(s.nmax + 1, B, lc.max_grid);
  const int gC = grid_for(s.ncell + 2, B, lc.max_grid);
  const int gP = grid_for(s.pcap, B, lc.max_grid);
  const int gS = std::max(1, std::min(s.nsys, 2 * lc.sms));  // a block per system
  const int T = sys_threads(s);
  if (stage <= 0) {
    k_ens_plan<<<1, T, 0, st>>>(s);
    k_ens_lost<<<gN, B, 0, st>>>(s);
    k_ens_zero_cells<<<gC, B, 0, st>>>(s);
    k_cell_count<<<gN, B, 0, st>>>(s);
    nl += 4 + scan_exclusive(s, s.cell_count, s.cell_start, s.ncell + 2, s.scan_tmp, 2, st);
    k_ens_scan<<<gS, 1024, 0, st>>>(s, kEnsScanCells);
    k_cell_scatter<<<gN, B, 0, st>>>(s);
    k_cell_sort<<<gC, B, 0, st>>>(s);
    k_permute<<<gN, B, 0, st>>>(s);
    k_copy_atoms<<<gN, B, 0, st>>>(s);
    k_pairs<false><<<gN, B, 0, st>>>(s);
    k_ens_scan<<<gS, 1024, 0, st>>>(s, kEnsScanRowsPartial);
    k_ens_kept<<<gN, B, 0, st>>>(s);
    k_ens_scan<<<gS, 1024, 0, st>>>(s, kEnsScanRowsFull);
    k_ens_layout<<<1, T, 0, st>>>(s);
    k_ens_rows_base<<<gN, B, 0, st>>>(s);
    k_pairs_total<<<1, 1, 0, st>>>(s);
    nl += 13;
  }
  if (stage <= 1) {
    k_ens_zero_rev<<<gN, B, 0, st>>>(s);
    k_ens_holes<<<gS, B, 0, st>>>(s);
    k_pairs<true><<<gN, B, 0, st>>>(s);
    k_pair_init<<<gP, B, 0, st>>>(s);
    k_ens_scan<<<gS, 1024, 0, st>>>(s, kEnsScanRev);
    k_rev_fill<<<gP, B, 0, st>>>(s);
    k_rev_sort<<<gN, B, 0, st>>>(s);
    k_copy_pairs<<<grid_for((long)s.pcap > s.nmax + 1 ? s.pcap : s.nmax + 1, B, lc.max_grid), B, 0, st>>>(s);
    nl += 8;
  }
  if (s.nplanes > 0) {
    k_wall_list<<<gN, B, 0, st>>>(s);
    nl++;
  }
  k_finish_rebuild<<<1, T, 0, st>>>(s);
  return nl + 1;
}

int launch_rebuild(const Sys &s, const LaunchCfg &lc, cudaStream_t st, int stage) {
  if (s.nsys) return launch_rebuild_ens(s, lc, st, stage);
  int nl = 0;
  const int B = 256;
  const int gN = grid_for(s.nmax + 1, B, lc.max_grid);
  const int gC = grid_for(s.ncell + 2, B, lc.max_grid);
  const int gP = grid_for(s.pcap, B, lc.max_grid);
  // stage 0: the whole rebuild; stage 1: from the pair fill (after the host
  // grew the pair list); stage 2: from the mesh stages (after it grew mesh
  // slots or registrations).  Every resumed stage is idempotent.
  if (stage <= 0) {
    k_zero_gated<<<gC, B, 0, st>>>(s, s.cell_count, s.ncell + 2);
    k_zero_gated<<<gC, B, 0, st>>>(s, s.cell_fill, s.ncell + 2);
    k_cell_count<<<gN, B, 0, st>>>(s);
    nl += 3 + scan_exclusive(s, s.cell_count, s.cell_start, s.ncell + 2, s.scan_tmp, true, st);
    k_cell_scatter<<<gN, B, 0, st>>>(s);
    k_cell_sort<<<gC, B, 0, st>>>(s);
    k_permute<<<gN, B, 0, st>>>(s);
    k_copy_atoms<<<gN, B, 0, st>>>(s);
    k_pairs<false><<<gN, B, 0, st>>>(s);
    nl += 5 + scan_exclusive(s, s.pcount, s.pairs[1].row, s.nmax + 1, s.scan_tmp, true, st);
    k_pairs_total<<<1, 1, 0, st>>>(s);
    nl += 1;
  }
  if (stage <= 1) {
    k_zero_gated<<<gN, B, 0, st>>>(s, s.rev_count, s.nmax + 1);
    k_zero_gated<<<gN, B, 0, st>>>(s, s.rev_fill, s.nmax + 1);
    k_pairs<true><<<gN, B, 0, st>>>(s);
    k_pair_init<<<gP, B, 0, st>>>(s);
    nl += 4 + scan_exclusive(s, s.rev_count, s.pairs[1].rev_start, s.nmax + 1, s.scan_tmp, true, st);
    k_rev_fill<<<gP, B, 0, st>>>(s);
    k_rev_sort<<<gN, B, 0, st>>>(s);
    k_copy_pairs<<<grid_for((long)s.pcap > s.nmax + 1 ? s.pcap : s.nmax + 1, B, lc.max_grid), B, 0, st>>>(s);
  }
  for (int k = 0; k < s.nmeshes; k++) {
    const MeshDev &M = s.meshes[k];
    const int gT = grid_for(M.ntri, B, lc.max_grid);
    k_mesh_sort<<<gN, B, 0, st>>>(s, k);
    k_zero_gated<<<gC, B, 0, st>>>(s, M.tc_count, s.ncell + 2);
    k_zero_gated<<<gC, B, 0, st>>>(s, M.tc_fill, s.ncell + 2);
    k_tri_count<<<gT, B, 0, st>>>(s, k);
    nl += 6 + scan_exclusive(s, M.tc_count, M.tc_start, s.ncell + 2, s.scan_tmp, true, st);
    k_tri_fill<<<gT, B, 0, st>>>(s, k);
    k_mesh_cand<<<gN, B, 0, st>>>(s, k);
  }
  if (s.nmeshes > 0 || s.nplanes > 0) {
    k_wall_list<<<gN, B, 0, st>>>(s);
    nl++;
  }
  k_finish_rebuild<<<1, sys_threads(s), 0, st>>>(s);
  return nl + 4;
}

// Builds the executable graph of one dem_step call; launch_set_loop sets the
// number of steps and the phase it starts in before each launch.
//
// Fused (k_steps runs all steps up to the next rebuild):
//   WHILE(loop) { k_steps -> IF(rebuild) { rebuild kernels } }
// Separate kernels (ensembles, large systems):
//   k_particle_start ->
//   WHILE(loop) { IF(rebuild) { rebuild kernels } ->
//                 kUnroll x (pair || wall -> k_particle(gather+final+initial)) } ->
//   pair || wall -> k_particle(gather+final)
// A step that decides to rebuild, and the last one, hold the rest of the loop's
// kernels (Ctrl::hold): they are no-ops until the next iteration's rebuild, or
// to the end.
// Without moving meshes the last block of the per-atom kernel takes the
// decision, else k_decide_loop does after the mesh has moved.  The first
// step's rebuild sits behind an IF node too: launched from the host its some
// thirty kernels cost 67-150 us of each call while doing nothing.
static int launch_particle_lp(const Sys &s, const LaunchCfg &lc, int mode, const LoopCond &lp, cudaStream_t st);

// steps per iteration: the WHILE and IF nodes cost some 10 us an iteration, a
// held step's kernels 4 (they matter to ensembles, which rebuild every few
// steps).  50 steps at 1, 4, 8: 1,000,000 in a hopper 13693, 13331, 13407 us;
// 400,000 packed 24596, 24306, 24230; 100 steps of an ensemble of 48 14655,
// 13872, 14076.
constexpr int kUnroll = 4;

// Captures into one graph at a time on two streams and cleans up on failure.
struct GraphBuilder {
  const Sys &s;
  const LaunchCfg &lc;
  cudaStream_t st, st2;
  cudaGraph_t g = nullptr;
  cudaEvent_t fork = nullptr, join = nullptr;
  int kpr = 0;  // kernels of a rebuild

  // ends a capture still open on either stream (its graph belongs to g),
  // destroys the events and the graph
  cudaError_t fail(cudaError_t err) {
    const cudaStream_t qs[2] = {st, st2};
    for (cudaStream_t q : qs) {
      cudaStreamCaptureStatus cs0 = cudaStreamCaptureStatusNone;
      if (cudaStreamIsCapturing(q, &cs0) == cudaSuccess && cs0 != cudaStreamCaptureStatusNone) {
        cudaGraph_t part = nullptr;
        cudaStreamEndCapture(q, &part);
      }
    }
    done();
    if (g) cudaGraphDestroy(g);
    g = nullptr;
    return err;
  }
  void done() {
    if (fork) cudaEventDestroy(fork);
    if (join) cudaEventDestroy(join);
    fork = join = nullptr;
  }
  cudaError_t begin(cudaGraph_t into) {
    return cudaStreamBeginCaptureToGraph(st, into, nullptr, nullptr, 0, cudaStreamCaptureModeThreadLocal);
  }
  cudaError_t end() {
    cudaGraph_t out = nullptr;
    return cudaStreamEndCapture(st, &out);
  }
  // a conditional node behind what st has captured so far; its body in *body
  cudaError_t conditional(cudaGraphConditionalHandle h, cudaGraphConditionalNodeType type, cudaGraph_t *body) {
    cudaStreamCaptureStatus cs;
    const cudaGraphNode_t *deps = nullptr;
    size_t nd = 0;
    cudaGraph_t cg;
    cudaError_t e = cudaStreamGetCaptureInfo(st, &cs, nullptr, &cg, &deps, nullptr, &nd);
    if (e != cudaSuccess) return e;
    cudaGraphNodeParams p = {};
    p.type = cudaGraphNodeTypeConditional;
    p.conditional.handle = h;
    p.conditional.type = type;
    p.conditional.size = 1;
    cudaGraphNode_t node;
    if ((e = cudaGraphAddNode(&node, cg, deps, nullptr, nd, &p)) != cudaSuccess) return e;
    *body = p.conditional.phGraph_out[0];
    return cudaStreamUpdateCaptureDependencies(st, &node, nullptr, 1, cudaStreamSetCaptureDependencies);
  }
  // IF(h) { rebuild kernels }
  cudaError_t rebuild_if(cudaGraphConditionalHandle h) {
    cudaGraph_t body, out = nullptr;
    cudaError_t e = conditional(h, cudaGraphCondTypeIf, &body);
    if (e != cudaSuccess) return e;
    if ((e = cudaStreamBeginCaptureToGraph(st2, body, nullptr, nullptr, 0, cudaStreamCaptureModeThreadLocal)) !=
        cudaSuccess)
      return e;
    kpr = launch_rebuild(s, lc, st2, 0);
    return cudaStreamEndCapture(st2, &out);
  }
  // the pair kernel and the wall kernel of a step, side by side
  cudaError_t forces(int gate, int *k) {
    cudaError_t e;
    const bool walls = s.nmeshes > 0 || s.nplanes > 0;
    if (walls) {
      if (!fork && (e = cudaEventCreateWithFlags(&fork, cudaEventDisableTiming)) != cudaSuccess) return e;
      if (!join && (e = cudaEventCreateWithFlags(&join, cudaEventDisableTiming)) != cudaSuccess) return e;
      if ((e = cudaEventRecord(fork, st)) != cudaSuccess) return e;
      if ((e = cudaStreamWaitEvent(st2, fork, 0)) != cudaSuccess) return e;
      *k += launch_wall_force(s, lc, 1, st2, gate);
      if ((e = cudaEventRecord(join, st2)) != cudaSuccess) return e;
    }
    *k += launch_pair(s, lc, 1, st, gate);
    return walls ? cudaStreamWaitEvent(st, join, 0) : cudaSuccess;
  }
  // the per-atom kernel (start: the call's first step) with the decision
  cudaError_t particle(bool start, cudaGraphConditionalHandle hreb, cudaGraphConditionalHandle hloop, int *k) {
    bool moving = false;
    for (int m = 0; m < s.nmeshes; m++) moving |= s.meshes[m].moving != 0;
    const LoopCond lp{moving ? 0 : 1, start ? 0 : 1, hreb, hloop};
    const int mode = start ? kModeStart : kModeGatherFinalInitial;
    *k += launch_particle_lp(s, lc, mode, lp, st);
    if (moving) {  // the mesh moves between the per-atom kernel and the decision
      *k += launch_mesh_move(s, lc, st, lp.gate);
      k_decide_loop<<<1, sys_threads(s), 0, st>>>(s, lp);
      (*k)++;
    }
    return cudaGetLastError();
  }
};

cudaError_t build_step_graph(const Sys &s, const LaunchCfg &lc, cudaStream_t st, cudaStream_t st2,
                             cudaGraphExec_t *exec, StepCounts *counts) {
  GraphBuilder b{s, lc, st, st2};
  cudaError_t e = cudaGraphCreate(&b.g, 0);
  if (e != cudaSuccess) return b.fail(e);
  cudaGraphConditionalHandle hloop, hreb;
  for (cudaGraphConditionalHandle *h : {&hloop, &hreb})
    if ((e = cudaGraphConditionalHandleCreate(h, b.g, h == &hloop ? 1 : 0, cudaGraphCondAssignDefault)) != cudaSuccess)
      return b.fail(e);
  *counts = StepCounts{};
  cudaGraph_t body;
  if ((e = b.begin(b.g)) != cudaSuccess) return b.fail(e);
  if (lc.fused) {
    if ((e = b.conditional(hloop, cudaGraphCondTypeWhile, &body)) != cudaSuccess) return b.fail(e);
    if ((e = b.end()) != cudaSuccess) return b.fail(e);
    if ((e = b.begin(body)) != cudaSuccess) return b.fail(e);
    if ((e = launch_steps(s, lc, hreb, hloop, st)) != cudaSuccess) return b.fail(e);
    if ((e = b.rebuild_if(hreb)) != cudaSuccess) return b.fail(e);
    if ((e = b.end()) != cudaSuccess) return b.fail(e);
    counts->call = 1;  // and one more launch per rebuild
    counts->rebuild = b.kpr + 1;
  } else {
    if ((e = b.particle(true, hreb, hloop, &counts->call)) != cudaSuccess) return b.fail(e);
    if ((e = b.conditional(hloop, cudaGraphCondTypeWhile, &body)) != cudaSuccess) return b.fail(e);
    if ((e = b.forces(0, &counts->call)) != cudaSuccess) return b.fail(e);
    counts->call += launch_particle(s, lc, kModeGatherFinal, st);
    if ((e = b.end()) != cudaSuccess) return b.fail(e);
    if ((e = b.begin(body)) != cudaSuccess) return b.fail(e);
    if ((e = b.rebuild_if(hreb)) != cudaSuccess) return b.fail(e);
    for (int u = 0; u < kUnroll; u++) {
      counts->step = 0;
      if ((e = b.forces(1, &counts->step)) != cudaSuccess) return b.fail(e);
      if ((e = b.particle(false, hreb, hloop, &counts->step)) != cudaSuccess) return b.fail(e);
    }
    if ((e = b.end()) != cudaSuccess) return b.fail(e);
    counts->rebuild = b.kpr;
  }
  e = cudaGraphInstantiate(exec, b.g, 0);
  b.done();
  cudaGraphDestroy(b.g);
  return e;
}

int wall_cap_per_atom() {
  static const int cap = [] {
    const char *e = getenv("LIGGGHTS_GB300_WALL_CAP");
    return e ? std::max(1, std::min(16, atoi(e))) : kWallCapDefault;
  }();
  return cap;
}

// The wall kernel walks a short list (atoms near walls) with long per-atom
// dependency chains; it is launched with the device's highest priority so
// that its blocks start before those of the pair kernel beside it.
int launch_wall_force(const Sys &s, const LaunchCfg &lc, int shearupdate, cudaStream_t st, int gate) {
  if (s.nmeshes == 0 && s.nplanes == 0) return 0;
  int lo = 0, hi = 0;
  cudaDeviceGetStreamPriorityRange(&lo, &hi);
  const int cap_per_atom = wall_cap_per_atom();
  const size_t bytes = (size_t)kWallWarps * cap_per_atom * kWallTile * kWallQ;
  cudaFuncSetAttribute(k_wall_force<kHertz>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
  cudaFuncSetAttribute(k_wall_force<kHooke>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
  const int cap = cap_per_atom * kWallTile;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(grid_for(s.nmax, kWallWarps * kWallTile, 2 * lc.max_grid));
  cfg.blockDim = dim3(kWallWarps * kWallTile);
  cfg.dynamicSmemBytes = bytes;
  cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributePriority;
  attr[0].val.priority = hi;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  if (s.normal == kHertz) cudaLaunchKernelEx(&cfg, k_wall_force<kHertz>, s, shearupdate, cap, gate);
  else cudaLaunchKernelEx(&cfg, k_wall_force<kHooke>, s, shearupdate, cap, gate);
  return 1;
}

int launch_mesh_move(const Sys &s, const LaunchCfg &lc, cudaStream_t st, int gate) {
  int nl = 0;
  for (int k = 0; k < s.nmeshes; k++) {
    if (!s.meshes[k].moving) continue;
    k_mesh_move<<<grid_for(16L * s.meshes[k].ntri, 256, lc.max_grid), 256, 0, st>>>(s, k, gate);
    nl++;
  }
  return nl;
}

// Steps of a graph launch after which k_steps returns and the host looks whether
// the system is still alone on the device (see DeviceCall): 20 us, 0.1 % of the
// smallest systems' turn; LIGGGHTS_GB300_TURN sets it (tests)
constexpr int kTurn = 2048;

int launch_set_loop(const Sys &s, int n, int phase, cudaStream_t st) {
  const char *turn = getenv("LIGGGHTS_GB300_TURN");
  k_set_loop<<<1, 1, 0, st>>>(s.ctrl, n, phase, turn ? std::max(1, atoi(turn)) : kTurn);
  return 1;
}

int launch_decide(const Sys &s, cudaStream_t st) {
  k_decide<<<1, sys_threads(s), 0, st>>>(s);
  return 1;
}
int launch_set_rebuild(const Sys &s, int v, cudaStream_t st) {
  k_set_rebuild<<<1, sys_threads(s), 0, st>>>(s, v);
  return 1;
}

int launch_pair(const Sys &s, const LaunchCfg &lc, int shearupdate, cudaStream_t st, int gate) {
  const int B = 256;
  const int g = grid_for(s.pcap, B, lc.max_grid);
  const int Bb = kBandTile;
  const int gb = grid_for(s.pcap, Bb, 2 * lc.max_grid);
  if (s.bond) {
    if (s.normal == kHertz) {
      if (s.rolling) k_pair<kHertz, true, true><<<gb, Bb, 0, st>>>(s, shearupdate, gate);
      else k_pair<kHertz, false, true><<<gb, Bb, 0, st>>>(s, shearupdate, gate);
    } else {
      if (s.rolling) k_pair<kHooke, true, true><<<gb, Bb, 0, st>>>(s, shearupdate, gate);
      else k_pair<kHooke, false, true><<<gb, Bb, 0, st>>>(s, shearupdate, gate);
    }
    return 1;
  }
  if (s.cdf == 1.0) {
    // blocks per SM the kernel is compiled for (registers: 80 at 3, 64 at
    // 4 with some spilling): 3 with mesh walls, whose wall kernel runs
    // beside this one (the 1M hopper's graph step 2 % faster than at 4),
    // else 4 (the 256-system ensemble 12 % faster than at 3; the dense bed
    // 1.6 % slower); LIGGGHTS_GB300_PAIR_MINB 3 or 4 sets it.  The grid:
    // LIGGGHTS_GB300_PAIR_GRID (0: up to 8 blocks per SM, the default, which
    // leaves room for the wall kernel beside it; 1: one resident wave, the
    // tiles taken grid-stride: the pair kernel alone runs faster, the step
    // slower).  Results do not depend on either.
    static int env_minb = -1, wave = 0;
    if (env_minb < 0) {
      const char *e = getenv("LIGGGHTS_GB300_PAIR_MINB");
      env_minb = (e && (atoi(e) == 3 || atoi(e) == 4)) ? atoi(e) : 0;
      const char *w = getenv("LIGGGHTS_GB300_PAIR_GRID");
      wave = (w && atoi(w) == 1) ? 1 : 0;
    }
    const int minb = env_minb ? env_minb : (s.nmeshes > 0 ? 3 : 4);
    const int gp = wave ? std::min(g, lc.sms * minb) : g;
    if (minb == 4) {
      if (s.normal == kHertz) {
        if (s.rolling) k_pair_pf<kHertz, true, 4><<<gp, B, 0, st>>>(s, shearupdate, gate);
        else k_pair_pf<kHertz, false, 4><<<gp, B, 0, st>>>(s, shearupdate, gate);
      } else {
        if (s.rolling) k_pair_pf<kHooke, true, 4><<<gp, B, 0, st>>>(s, shearupdate, gate);
        else k_pair_pf<kHooke, false, 4><<<gp, B, 0, st>>>(s, shearupdate, gate);
      }
    } else {
      if (s.normal == kHertz) {
        if (s.rolling) k_pair_pf<kHertz, true, 3><<<gp, B, 0, st>>>(s, shearupdate, gate);
        else k_pair_pf<kHertz, false, 3><<<gp, B, 0, st>>>(s, shearupdate, gate);
      } else {
        if (s.rolling) k_pair_pf<kHooke, true, 3><<<gp, B, 0, st>>>(s, shearupdate, gate);
        else k_pair_pf<kHooke, false, 3><<<gp, B, 0, st>>>(s, shearupdate, gate);
      }
    }
    return 1;
  }
  if (s.normal == kHertz) {
    if (s.rolling) k_pair<kHertz, true, false><<<gb, Bb, 0, st>>>(s, shearupdate, gate);
    else k_pair<kHertz, false, false><<<gb, Bb, 0, st>>>(s, shearupdate, gate);
  } else {
    if (s.rolling) k_pair<kHooke, true, false><<<gb, Bb, 0, st>>>(s, shearupdate, gate);
    else k_pair<kHooke, false, false><<<gb, Bb, 0, st>>>(s, shearupdate, gate);
  }
  return 1;
}

static int launch_particle_lp(const Sys &s, const LaunchCfg &lc, int mode, const LoopCond &lp, cudaStream_t st) {
  // one particle per thread; smaller blocks give the same number of threads
  // in more, smaller blocks (each particle's sums do not depend on it)
  const int B = lc.particle_threads;
  const int g = grid_for(s.nmax, B, lc.max_grid * (256 / B));
  switch (mode) {
    case kModeInitial: k_particle<false, false, true><<<g, B, 0, st>>>(s, lp); break;
    case kModeGather: k_particle<true, false, false><<<g, B, 0, st>>>(s, lp); break;
    case kModeGatherFinal: k_particle<true, true, false><<<g, B, 0, st>>>(s, lp); break;
    case kModeGatherFinalInitial: k_particle<true, true, true><<<g, B, 0, st>>>(s, lp); break;
    case kModeStart: k_particle_start<<<g, B, 0, st>>>(s, lp); break;
  }
  return 1;
}

int launch_particle(const Sys &s, const LaunchCfg &lc, int mode, cudaStream_t st) {
  return launch_particle_lp(s, lc, mode, LoopCond{0, 0, 0, 0}, st);
}

}  // namespace gb300

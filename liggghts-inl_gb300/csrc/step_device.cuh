// Device code of one timestep, shared by the kernels of dem_kernels.cu and the
// fused step kernel of dem_steps.cu: exact predicates and image shifts, the
// moving meshes, the pair and wall force tiles, the per-atom tile.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include "bond_law.cuh"
#include "contact_law.cuh"
#include "dem_device.cuh"
#include "mesh_device.cuh"

namespace gb300 {

#define GRID_STRIDE(i, n) for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < (n); i += gridDim.x * blockDim.x)

__device__ __forceinline__ bool gated(const Ctrl *c) { return c->halt != 0 || c->rebuild == 0; }

// Exact reference arithmetic (no contraction) for everything that decides
// membership of the pair set.
__device__ __forceinline__ double rsq_rn(double dx, double dy, double dz) {
  return __dadd_rn(__dadd_rn(__dmul_rn(dx, dx), __dmul_rn(dy, dy)), __dmul_rn(dz, dz));
}

__device__ __forceinline__ void shift_decode(int c, int &sx, int &sy, int &sz) {
  sx = c % 3 - 1;
  sy = (c / 3) % 3 - 1;
  sz = c / 9 - 1;
}

// ghost image x_j + pbc*prd exactly as CommBrick::borders/forward_comm
// (src/atom_vec_sphere.cpp:213-223): fl(x + (+-prd)) per shifted dimension.
__device__ __forceinline__ void image(const Sys &s, int code, double &xj, double &yj, double &zj) {
  if (code == kNoShift) return;
  int sx, sy, sz;
  shift_decode(code, sx, sy, sz);
  // +-prd by selection: sx * prd would convert sx to FP64 and multiply on
  // the FP64 pipe (and the compiler hoists that out of candidate loops)
  if (sx) xj = __dadd_rn(xj, sx > 0 ? s.prd[0] : -s.prd[0]);
  if (sy) yj = __dadd_rn(yj, sy > 0 ? s.prd[1] : -s.prd[1]);
  if (sz) zj = __dadd_rn(zj, sz > 0 ? s.prd[2] : -s.prd[2]);
}

// Whether the periodic image of j (shift sv) exists as a ghost atom:
// CommBrick::borders sends an atom across a periodic boundary only when it
// lies within slab_offset + its radius of that boundary (the granular
// criterion of CommBrick::decide, src/comm_brick.cpp:443,1613-1624).  With a
// contact distance factor above 1 this band is narrower than the pair cutoff
// and some periodic pairs near the cutoff do not exist in the reference.
__device__ __forceinline__ bool ghost_exists(const Sys &s, const AtomArrays &A, int j, const int sv[3]) {
  const double rad = A.r[j];
  const double pos[3] = {A.x[j], A.y[j], A.z[j]};
#pragma unroll
  for (int d = 0; d < 3; d++) {
    if (sv[d] > 0 && !(pos[d] <= __dadd_rn(__dadd_rn(s.boxlo[d], s.ghost_slab), rad))) return false;
    if (sv[d] < 0 && !(pos[d] >= __dadd_rn(__dadd_rn(s.boxhi[d], -s.ghost_slab), -rad))) return false;
  }
  return true;
}

// The cells are wider than the neighbour cutoff by a relative 1e-9 at least,
// far above the rounding of this product, so atoms within the cutoff are
// never more than one cell apart; every kernel bins through this function.
// FP32 image shift -1, 0 or +1 times the period, by selection (no conversion)
__device__ __forceinline__ float fshift(int sv, float prd) { return sv == 0 ? 0.0f : (sv > 0 ? prd : -prd); }

__device__ __forceinline__ int cell_coord(const Sys &s, double x, int d) {
  int c = (int)((x - s.boxlo[d]) * s.icsz[d]);
  c = c < 0 ? 0 : c;
  c = c >= s.nc[d] ? s.nc[d] - 1 : c;
  return c;
}

__device__ __forceinline__ int warp_incl_scan(int x) {
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int off = 1; off < 32; off <<= 1) {
    int y = __shfl_up_sync(0xffffffffu, x, off);
    if (lane >= off) x += y;
  }
  return x;
}

// MathExtra::quatquat (src/math_extra.h:596-602) and
// MathExtraLiggghts::vec_quat_rotate (src/math_extra_liggghts.h:455-471) in
// the reference's operation order, exactly rounded: rotated nodes are
// bit-identical to the reference's
__device__ __forceinline__ void quatquat_rn(const double *a, const double *b, double *c) {
  c[0] = __dsub_rn(__dsub_rn(__dsub_rn(__dmul_rn(a[0], b[0]), __dmul_rn(a[1], b[1])), __dmul_rn(a[2], b[2])),
                   __dmul_rn(a[3], b[3]));
  c[1] = __dsub_rn(__dadd_rn(__dadd_rn(__dmul_rn(a[0], b[1]), __dmul_rn(b[0], a[1])), __dmul_rn(a[2], b[3])),
                   __dmul_rn(a[3], b[2]));
  c[2] = __dsub_rn(__dadd_rn(__dadd_rn(__dmul_rn(a[0], b[2]), __dmul_rn(b[0], a[2])), __dmul_rn(a[3], b[1])),
                   __dmul_rn(a[1], b[3]));
  c[3] = __dsub_rn(__dadd_rn(__dadd_rn(__dmul_rn(a[0], b[3]), __dmul_rn(b[0], a[3])), __dmul_rn(a[1], b[2])),
                   __dmul_rn(a[2], b[1]));
}
__device__ __forceinline__ void vec_quat_rotate_rn(double *v, const double *q) {
  const double vq[4] = {0., v[0], v[1], v[2]};
  const double qc[4] = {q[0], -q[1], -q[2], -q[3]};
  double t[4], r[4];
  quatquat_rn(q, vq, t);
  quatquat_rn(t, qc, r);
  v[0] = r[1];
  v[1] = r[2];
  v[2] = r[3];
}

// One step of a moving mesh: 16 lanes per triangle, lane q taking one of its
// vectors (nodes 0..2, edgeVec 3..5, edgeNorm 6..8, surfaceNorm 9), lane 10
// the centre.  A quaternion rotation is a chain of some fifty FP64
// instructions and most moving meshes have few triangles, so one thread per
// triangle made ten such chains one after the other (a two-triangle paddle:
// 23 us per step; one per lane: 6 us).  Returns whether a node moved more
// than skin/2 since the last build.
//   linear: MeshMoverLinear::initial_integrate + MultiNodeMesh::move (nodes and
//     centres += dx, src/multi_node_mesh_I.h:502-520);
//   rotating: MeshMoverRotate::initial_integrate
//     (src/mesh_mover_rotation.cpp:105-131): nodes and centres
//     (MultiNodeMesh::rotate(dQ, origin), src/multi_node_mesh_I.h:643-668), the
//     rotating element vectors edgeVec, edgeNorm, surfaceNorm
//     (CustomValueTracker::rotate), node velocities 0 + w x (node - O);
// then the node-travel test of MultiNodeMesh::decideRebuild
// (src/multi_node_mesh_I.h:792-823).
__device__ __forceinline__ bool mesh_move_part(const Sys &s, const MeshDev &M, int t, int q) {
  const double trigger = __dmul_rn(__dmul_rn(0.25, s.skin), s.skin);
  double *g = M.tri + (size_t)t * kTriStride;
  const bool on = t < M.ntri && q < 11;
  bool moved = false;
  double out[3] = {0., 0., 0.};
  int at = -1;  // where this lane's vector goes in the triangle's record
  if (on && !M.rotating) {
    if (q < 3 || q == 10) {
      at = q < 3 ? 3 * q : 33;
      for (int d = 0; d < 3; d++) out[d] = __dadd_rn(g[at + d], M.dx[d]);
    }
  } else if (M.rotating) {
    const double *o = M.rorig, *rq = M.rq;
    const bool trans =
        __dadd_rn(__dadd_rn(__dmul_rn(o[0], o[0]), __dmul_rn(o[1], o[1])), __dmul_rn(o[2], o[2])) > 0.;
    if (on && q < 10) {
      at = 3 * q + (q == 9 ? 3 : 0);
      for (int d = 0; d < 3; d++) out[d] = g[at + d];
      if (q < 3 && trans)
        for (int d = 0; d < 3; d++) out[d] = __dsub_rn(out[d], o[d]);
      vec_quat_rotate_rn(out, rq);
      if (q < 3 && trans)
        for (int d = 0; d < 3; d++) out[d] = __dadd_rn(out[d], o[d]);
    }
    // the centre from the turned nodes of lanes 0..2
    const double third = 1. / 3.;
    for (int d = 0; d < 3; d++) {
      double cen = 0.;
      for (int j = 0; j < 3; j++) cen = __dadd_rn(__shfl_sync(0xffffffffu, out[d], j, 16), cen);
      if (on && q == 10) out[d] = __dmul_rn(third, cen);
    }
    if (on && q == 10) at = 33;
  }
  __syncwarp();  // every lane has read the record before any writes it
  if (at >= 0) {
    for (int d = 0; d < 3; d++) g[at + d] = out[d];
    if (q < 3) {
      double dsq = 0.0;
      for (int d = 0; d < 3; d++) {
        const double e = __dadd_rn(out[d], -M.node_last[(size_t)t * 9 + 3 * q + d]);
        dsq = d == 0 ? __dmul_rn(e, e) : __dadd_rn(dsq, __dmul_rn(e, e));
      }
      moved = dsq > trigger;
      if (M.rotating) {
        const double *o = M.rorig, *w = M.romega;
        const double r[3] = {__dsub_rn(out[0], o[0]), __dsub_rn(out[1], o[1]), __dsub_rn(out[2], o[2])};
        double *v = M.nodev + (size_t)t * 9 + 3 * q;
        v[0] = __dadd_rn(0.0, __dsub_rn(__dmul_rn(w[1], r[2]), __dmul_rn(w[2], r[1])));
        v[1] = __dadd_rn(0.0, __dsub_rn(__dmul_rn(w[2], r[0]), __dmul_rn(w[0], r[2])));
        v[2] = __dadd_rn(0.0, __dsub_rn(__dmul_rn(w[0], r[1]), __dmul_rn(w[1], r[0])));
      }
    }
    // the FP32 copies: node 0, surface normal, edge normals (all zero where
    // the triangle is too thin for the edge bounds, see tri_floats)
    float4 *T = M.trif + kTrif * (size_t)t;
    const int slot = q == 0 ? 0 : (q == 9 ? 1 : (q >= 6 && q < 9 ? q - 4 : -1));
    if (slot >= 0) {
      const float4 old = T[slot];
      if (slot < 2 || old.x != 0.f || old.y != 0.f || old.z != 0.f)
        T[slot] = make_float4((float)out[0], (float)out[1], (float)out[2], old.w);
    }
  }
  return moved;
}

// end of atom i's owner row and of its partner list
__device__ __forceinline__ int row_end(const Sys &s, const PairArrays &L, int i) {
  return s.nsys ? L.rowe[i] : L.row[i + 1];
}
__device__ __forceinline__ int rev_end(const Sys &s, const PairArrays &L, int i) {
  return s.nsys ? L.reve[i] : L.rev_start[i + 1];
}

// ----------------------------------------------------------------------------
// pair forces: one thread per half-list entry, results to the pair buffer
// ----------------------------------------------------------------------------

// The pair kernels test list entries per lane (phase 1) and queue the ones
// that need the FP64 laws in a per-warp shared-memory queue (warp ballots),
// so phase 2 runs on full warps: entries that need nothing cost no FP64
// issue slots.  Results go to the entry's own slot, so the processing order
// never changes a value.  kPairTile is k_pair_pf's block size.
constexpr int kPairTile = 256;

// The general kernel carries the bond law.  Blocks of 128 threads capped at
// 128 registers (a few spilled) let four blocks share an SM (measured on the
// 200k bonded fibre bed with one queue per tile: 0.55 ms with one 256-thread
// block per SM, 0.41 ms with three 128-thread blocks, 0.35 ms with four;
// 64-thread tiles 0.40 ms; with per-warp queues 0.27 ms).
constexpr int kBandTile = 128;

// the entry's result record: three whole 32-byte sectors in one go
__device__ __forceinline__ void store_result(const Sys &s, int q, const ContactOut &o) {
  double2 *r = reinterpret_cast<double2 *>(s.res + (size_t)kResStride * q);
  r[0] = make_double2(o.F[0], o.F[1]);
  r[1] = make_double2(o.F[2], o.Ti[0]);
  r[2] = make_double2(o.Ti[1], o.Ti[2]);
  r[3] = make_double2(o.Tj[0], o.Tj[1]);
  r[4] = make_double2(o.Tj[2], 0.0);
  r[5] = make_double2(0.0, 0.0);
}

// x with its sign bit flipped where `sign` has it (a variable: a constant one
// would become a negation, which issues on the FP64 pipe, as a product does)
__device__ __forceinline__ double with_sign(double x, int sign) {
  return __hiloint2double(__double2hiint(x) ^ sign, __double2loint(x));
}

// Phase 2 of k_pair for one queued entry q (delx, dely, delz, rsq_q from
// its exact test): the bond law, the contact law, the result record
template <int NORMAL, bool ROLL, bool BOND>
__device__ __forceinline__ void band_entry(const Sys &s, int q, double delx, double dely, double delz,
                                           double rsq_q, int shearupdate, long long ntimestep) {
  const AtomArrays &A = s.atoms[0];
  const PairArrays &L = s.pairs[0];
  const size_t P = s.pcap;
  const int i = L.i[q], j = L.j[q];
  ContactIn ci;
  ci.d[0] = delx;
  ci.d[1] = dely;
  ci.d[2] = delz;
  ci.radi = A.r[i];
  ci.radj = A.r[j];
  ci.radsum = __dadd_rn(ci.radi, ci.radj);
  ci.vr[0] = A.vx[i] - A.vx[j];
  ci.vr[1] = A.vy[i] - A.vy[j];
  ci.vr[2] = A.vz[i] - A.vz[j];
  ci.wi[0] = A.wx[i]; ci.wi[1] = A.wy[i]; ci.wi[2] = A.wz[i];
  ci.wj[0] = A.wx[j]; ci.wj[1] = A.wy[j]; ci.wj[2] = A.wz[j];
  const bool touch = !BOND || gt_nonneg(__dmul_rn(ci.radsum, ci.radsum), rsq_q);
  ContactOut bo;
  bool bonded = false;
  if (BOND) {
    // evaluated in the reference's orientation: owner = lower lidx
    // (periodic entries are directed and always owned by i)
    const bool rev = L.sh[q] == kNoShift && A.lidx[i] > A.lidx[j];
    const int a = rev ? j : i, b = rev ? i : j;
    const int sg = rev ? (int)0x80000000 : 0;  // turns a vector round
    BondIn bi;
    for (int k = 0; k < 3; k++) bi.d[k] = with_sign(ci.d[k], sg);
    bi.rsq = rsq_q;
    bi.radi = A.r[a];
    bi.radj = A.r[b];
    bi.vi[0] = A.vx[a]; bi.vi[1] = A.vy[a]; bi.vi[2] = A.vz[a];
    bi.vj[0] = A.vx[b]; bi.vj[1] = A.vy[b]; bi.vj[2] = A.vz[b];
    bi.wi[0] = A.wx[a]; bi.wi[1] = A.wy[a]; bi.wi[2] = A.wz[a];
    bi.wj[0] = A.wx[b]; bi.wj[1] = A.wy[b]; bi.wj[2] = A.wz[b];
    bi.xi[0] = A.x[a]; bi.xi[1] = A.y[a]; bi.xi[2] = A.z[a];
    bi.tp = A.type[a] * (s.ntypes + 1) + A.type[b];
    ContactOut bc;
    bonded = bond_nonlinear(s, bi, L.hist + 3 * P + q, P, L.flag + q, shearupdate != 0, ntimestep, bc);
    if (bonded) {  // back to the list's orientation (i owns the entry)
      for (int k = 0; k < 3; k++) {
        bo.F[k] = with_sign(bc.F[k], sg);
        bo.Ti[k] = rev ? bc.Tj[k] : bc.Ti[k];
        bo.Tj[k] = rev ? bc.Ti[k] : bc.Tj[k];
      }
    }
  }
  ContactOut o;
  if (touch) {
    // r from 1/r: within an ulp of sqrt(rsq), which moves the overlap
    // radsum - r by ~1e-13 of itself
    ci.rinv = rsqrt(rsq_q);
    ci.r = rsq_q * ci.rinv;
    ci.reff = L.reff[q];
    ci.c0 = L.c0[q];
    ci.c1 = L.c1[q];
    ci.en[0] = ci.d[0] * ci.rinv;
    ci.en[1] = ci.d[1] * ci.rinv;
    ci.en[2] = ci.d[2] * ci.rinv;
    ci.deltan_wall = 0.0;
    const TypePair tp = load_typepair(s.params, s.ntypes, A.type[i], A.type[j]);
    double sh3[3] = {L.hist[q], L.hist[P + q], L.hist[2 * P + q]};
    contact_law<NORMAL, false>(ci, tp, s.dt, s.tdamp, s.limitf, ROLL, shearupdate != 0, sh3, o,
                               (BOND && bonded) ? &bo : nullptr);
    if (shearupdate) {
      L.hist[q] = sh3[0];
      L.hist[P + q] = sh3[1];
      L.hist[2 * P + q] = sh3[2];
    }
    L.flag[q] |= (kContactNormal | kContactTangential);
  } else {
    for (int k = 0; k < 3; k++) {
      o.F[k] = bo.F[k];
      o.Ti[k] = bo.Ti[k];
      o.Tj[k] = bo.Tj[k];
    }
  }
  if (touch || bonded) {
    store_result(s, q, o);
    s.active[q] = 1;
  }
}

// one warp's queue of the general kernel, and the block's last batch
struct BandQueue {
  int p[64];
  double d[4][64];
};
template <int TILE>
struct BandRest {
  int p[TILE];
  double d[4][TILE];
  int n;
};

// entry p of the list; code kHole: none
__device__ __forceinline__ void pf_load(const Sys &s, int np, int p, int &i, int &j, int &code) {
  const PairArrays &L = s.pairs[0];
  const bool on = p < np;
  code = on ? L.sh[p] : kHole;
  i = on ? L.i[p] : 0;
  j = on ? L.j[p] : 0;
}
// Phase 1 of the general kernel for entry p: the exact distance, the flags and
// histories of an entry that does not touch; true when phase 2 has to see it.
template <bool BOND>
__device__ __forceinline__ bool band_near(const Sys &s, int np, int p, int i, int j, int code, double cdm,
                                          bool may_create, double &delx, double &dely, double &delz, double &rsq) {
  const AtomArrays &A = s.atoms[0];
  const PairArrays &L = s.pairs[0];
  const size_t P = s.pcap;
  bool queue = false;
  if (code == kHole && p < np) s.active[p] = 0;  // an unused entry of an ensemble segment
  if (code != kHole) {
    double xj = A.x[j], yj = A.y[j], zj = A.z[j];
    image(s, code, xj, yj, zj);
    delx = __dadd_rn(A.x[i], -xj);
    dely = __dadd_rn(A.y[i], -yj);
    delz = __dadd_rn(A.z[i], -zj);
    rsq = rsq_rn(delx, dely, delz);
    const double radsum = __dadd_rn(A.r[i], A.r[j]);
    queue = gt_nonneg(__dmul_rn(radsum, radsum), rsq);
    if (!queue) {
      s.active[p] = 0;
      if (gt_nonneg(__dmul_rn(__dmul_rn(cdm, radsum), radsum), rsq)) {
        // TangentialModel<TANGENTIAL_HISTORY>::surfacesClose
        L.flag[p] &= ~kContactTangential;
        L.hist[p] = 0.0;
        L.hist[P + p] = 0.0;
        L.hist[2 * P + p] = 0.0;
        // CohesionModel::surfacesClose: bonded pairs (and pairs that may
        // bond in this pass) are evaluated in phase 2
        const long long tiny = order_key(1.e-15);
        if (BOND && (may_create || order_key(L.hist[3 * P + p]) >= tiny)) {
          const int tp = A.type[i] * (s.ntypes + 1) + A.type[j];
          queue = order_key(__ldg(s.bondp + tp)) >= tiny;
        }
      }
    }
  }
  return queue;
}

template <bool BOND>
__device__ __forceinline__ bool band_test(const Sys &s, int np, int p, double cdm, bool may_create, double &delx,
                                          double &dely, double &delz, double &rsq) {
  int i, j, code;
  pf_load(s, np, p, i, j, code);
  return band_near<BOND>(s, np, p, i, j, code, cdm, may_create, delx, dely, delz, rsq);
}

// cohesion bond/nonlinear: a bond can be created in this pass
template <bool BOND>
__device__ __forceinline__ bool band_may_create(const Sys &s, int shearupdate, long long ntimestep) {
  return BOND && shearupdate && ((s.bond_flags & kBondCreateAlways) || ntimestep == s.bond_ts_create);
}

// Phase 1 runs per lane on 32 consecutive entries of a warp at a time; the
// entries that need phase 2 wait in the warp's shared-memory queue (with
// their exact test's delta and rsq) until 32 have gathered, so the bond and
// contact laws run on full warps.  The warps' remainders merge into one
// block batch at the end (band_rest).  Each entry's result goes to its own slot
// and depends on no other entry, so the order changes no value.
// next() gives the first entry of the warp's next 32 (np or more: none left).
template <int NORMAL, bool ROLL, bool BOND, class Next>
__device__ __forceinline__ int band_tiles(const Sys &s, int np, int shearupdate, long long ntimestep, BandQueue &q,
                                          Next next) {
  int *qp = q.p;
  double(*qd)[64] = q.d;
  const double cdm = s.cdf * s.cdf;
  const int lane = threadIdx.x & 31;
  const unsigned below = (1u << lane) - 1u;
  const bool may_create = band_may_create<BOND>(s, shearupdate, ntimestep);
  int qn = 0;  // the same in every lane
  int base = next(), i = 0, j = 0, code = kHole;
  if (base < np) pf_load(s, np, base + lane, i, j, code);
  while (base < np) {
    const int p = base + lane, pi = i, pj = j, pc = code;
    base = next();
    if (base < np) pf_load(s, np, base + lane, i, j, code);  // on its way during this tile's test
    double delx = 0., dely = 0., delz = 0., rsq = 0.;
    const bool queue = band_near<BOND>(s, np, p, pi, pj, pc, cdm, may_create, delx, dely, delz, rsq);
    const unsigned m = __ballot_sync(0xffffffffu, queue);
    if (queue) {
      const int slot = qn + __popc(m & below);
      qp[slot] = p;
      qd[0][slot] = delx;
      qd[1][slot] = dely;
      qd[2][slot] = delz;
      qd[3][slot] = rsq;
    }
    qn += __popc(m);
    __syncwarp();
    if (qn >= 32) {
      band_entry<NORMAL, ROLL, BOND>(s, qp[lane], qd[0][lane], qd[1][lane], qd[2][lane], qd[3][lane], shearupdate,
                                     ntimestep);
      const int rem = qn - 32;
      __syncwarp();
      int vp = 0;
      double v0 = 0., v1 = 0., v2 = 0., v3 = 0.;
      if (lane < rem) {
        vp = qp[32 + lane];
        v0 = qd[0][32 + lane];
        v1 = qd[1][32 + lane];
        v2 = qd[2][32 + lane];
        v3 = qd[3][32 + lane];
      }
      __syncwarp();
      if (lane < rem) {
        qp[lane] = vp;
        qd[0][lane] = v0;
        qd[1][lane] = v1;
        qd[2][lane] = v2;
        qd[3][lane] = v3;
      }
      qn = rem;
      __syncwarp();
    }
  }
  return qn;
}

// the warps' remainders (at most 31 each) as one block batch
template <int NORMAL, bool ROLL, bool BOND, int TILE>
__device__ __forceinline__ void band_rest(const Sys &s, int qn, int shearupdate, long long ntimestep,
                                          const BandQueue &q, BandRest<TILE> &r) {
  const int lane = threadIdx.x & 31;
  if (threadIdx.x == 0) r.n = 0;
  __syncthreads();
  int at = 0;
  if (lane == 0 && qn) at = atomicAdd(&r.n, qn);
  at = __shfl_sync(0xffffffffu, at, 0);
  if (lane < qn) {
    r.p[at + lane] = q.p[lane];
    for (int k = 0; k < 4; k++) r.d[k][at + lane] = q.d[k][lane];
  }
  __syncthreads();
  if (threadIdx.x < r.n)
    band_entry<NORMAL, ROLL, BOND>(s, r.p[threadIdx.x], r.d[0][threadIdx.x], r.d[1][threadIdx.x],
                                   r.d[2][threadIdx.x], r.d[3][threadIdx.x], shearupdate, ntimestep);
}

// Pair forces without cohesion and with contact distance factor 1 (an entry
// that is not touching needs no work).  A warp tests 32 consecutive entries
// at a time in FP32 (x, y, z, r refreshed by every drift): entries apart by
// more than the bound of the FP32 rounding (pf_margin_touch) only clear
// their active flag.  The rest are queued in the warp's shared-memory queue;
// whenever 32 have gathered, the warp runs the exact test and the FP64
// contact law on all its lanes (the FP64 pipe issues per warp, so idle lanes
// would waste it).  No block-wide barrier inside the loop: the warps of a
// block reach their FP64 phases at different times (a block-wide queue
// of 256 held all eight warps at three barriers per tile; the pair kernel
// took 0.143 ms on the 1M-atom hopper that way, 0.136 ms this way).
template <int NORMAL, bool ROLL>
__device__ __forceinline__ void pair_entry(const Sys &s, int q, int i, int j, int code, int shearupdate) {
  const AtomArrays &A = s.atoms[0];
  const PairArrays &L = s.pairs[0];
  const size_t P = s.pcap;
  double xj = A.x[j], yj = A.y[j], zj = A.z[j];
  image(s, code, xj, yj, zj);
  ContactIn ci;
  ci.d[0] = __dadd_rn(A.x[i], -xj);
  ci.d[1] = __dadd_rn(A.y[i], -yj);
  ci.d[2] = __dadd_rn(A.z[i], -zj);
  const double rsq = rsq_rn(ci.d[0], ci.d[1], ci.d[2]);
  ci.radi = A.r[i];
  ci.radj = A.r[j];
  ci.radsum = __dadd_rn(ci.radi, ci.radj);
  if (!gt_nonneg(__dmul_rn(ci.radsum, ci.radsum), rsq)) {
    s.active[q] = 0;
    return;
  }
  ci.vr[0] = A.vx[i] - A.vx[j];
  ci.vr[1] = A.vy[i] - A.vy[j];
  ci.vr[2] = A.vz[i] - A.vz[j];
  ci.wi[0] = A.wx[i]; ci.wi[1] = A.wy[i]; ci.wi[2] = A.wz[i];
  ci.wj[0] = A.wx[j]; ci.wj[1] = A.wy[j]; ci.wj[2] = A.wz[j];
  // r from 1/r: within an ulp of sqrt(rsq), which moves the overlap
  // radsum - r by ~1e-13 of itself
  ci.rinv = rsqrt(rsq);
  ci.r = rsq * ci.rinv;
  ci.reff = L.reff[q];
  ci.c0 = L.c0[q];
  ci.c1 = L.c1[q];
  ci.en[0] = ci.d[0] * ci.rinv;
  ci.en[1] = ci.d[1] * ci.rinv;
  ci.en[2] = ci.d[2] * ci.rinv;
  ci.deltan_wall = 0.0;
  const TypePair tp = load_typepair(s.params, s.ntypes, A.type[i], A.type[j]);
  double sh3[3] = {L.hist[q], L.hist[P + q], L.hist[2 * P + q]};
  ContactOut o;
  if (ROLL) contact_law<NORMAL, false>(ci, tp, s.dt, s.tdamp, s.limitf, true, shearupdate != 0, sh3, o);
  else pair_law<NORMAL>(ci, tp, s.dt, s.tdamp, s.limitf, shearupdate != 0, sh3, o);
  if (shearupdate) {
    L.hist[q] = sh3[0];
    L.hist[P + q] = sh3[1];
    L.hist[2 * P + q] = sh3[2];
  }
  L.flag[q] |= (kContactNormal | kContactTangential);
  store_result(s, q, o);
  s.active[q] = 1;
}

// FP32 touching test of entry p between i and j (x, y, z, r refreshed by every
// drift): false when the pair is apart by more than the bound of the FP32
// rounding; code kHole: no entry.
__device__ __forceinline__ bool pf_near(const Sys &s, int np, int p, int i, int j, int code) {
  const float hi_f = 1.0f + s.pf_margin_touch;
  bool maybe = false;
  if (code != kHole) {
    const float4 a = s.xf[i], b = s.xf[j];
    float sx = 0.f, sy = 0.f, sz = 0.f;
    if (code != kNoShift) {
      sx = fshift(code % 3 - 1, s.prdf[0]);
      sy = fshift((code / 3) % 3 - 1, s.prdf[1]);
      sz = fshift(code / 9 - 1, s.prdf[2]);
    }
    const float fx = a.x - (b.x + sx), fy = a.y - (b.y + sy), fz = a.z - (b.z + sz);
    const float rs = a.w + b.w;
    maybe = !(fx * fx + fy * fy + fz * fz > rs * rs * hi_f);
  }
  if (!maybe && p < np) s.active[p] = 0;
  return maybe;
}
__device__ __forceinline__ bool pf_test(const Sys &s, int np, int p, int &i, int &j, int &code) {
  pf_load(s, np, p, i, j, code);
  return pf_near(s, np, p, i, j, code);
}

template <int NORMAL, bool ROLL>
__device__ __forceinline__ void pair_entry(const Sys &s, int q, int shearupdate) {
  const PairArrays &L = s.pairs[0];
  pair_entry<NORMAL, ROLL>(s, q, L.i[q], L.j[q], L.sh[q], shearupdate);
}

// The warps' loop of k_pair_pf over 32 entries at a time (next() as in
// band_tiles), the remainder of at most 31 left in q.
template <int NORMAL, bool ROLL, class Next>
__device__ __forceinline__ int pf_tiles(const Sys &s, int np, int shearupdate, int *q, Next next) {
  const int lane = threadIdx.x & 31;
  const unsigned below = (1u << lane) - 1u;
  int qn = 0;  // the same in every lane
  int base = next(), i = 0, j = 0, code = kHole;
  if (base < np) pf_load(s, np, base + lane, i, j, code);
  while (base < np) {
    const int p = base + lane, pi = i, pj = j, pc = code;
    base = next();
    if (base < np) pf_load(s, np, base + lane, i, j, code);  // on its way during this tile's test
    const bool maybe = pf_near(s, np, p, pi, pj, pc);
    const unsigned m = __ballot_sync(0xffffffffu, maybe);
    if (maybe) q[qn + __popc(m & below)] = p;
    qn += __popc(m);
    __syncwarp();
    if (qn >= 32) {
      pair_entry<NORMAL, ROLL>(s, q[lane], shearupdate);
      const int rem = qn - 32;
      __syncwarp();
      const int v = lane < rem ? q[32 + lane] : 0;
      __syncwarp();
      if (lane < rem) q[lane] = v;
      qn = rem;
      __syncwarp();
    }
  }
  return qn;
}

// the warps' remainders (at most 31 each) as one block batch, so that a block
// ends with one partial batch instead of one per warp
struct PfRest {
  int p[kPairTile];
  int n;
};
template <int NORMAL, bool ROLL>
__device__ __forceinline__ void pf_rest(const Sys &s, int qn, int shearupdate, const int *q, PfRest &r) {
  const int lane = threadIdx.x & 31;
  if (threadIdx.x == 0) r.n = 0;
  __syncthreads();
  int at = 0;
  if (lane == 0 && qn) at = atomicAdd(&r.n, qn);
  at = __shfl_sync(0xffffffffu, at, 0);
  if (lane < qn) r.p[at + lane] = q[lane];
  __syncthreads();
  if (threadIdx.x < r.n) pair_entry<NORMAL, ROLL>(s, r.p[threadIdx.x], shearupdate);
}

// ----------------------------------------------------------------------------
// per-atom kernel: force gather + gravity + primitive walls + nve/sphere
// ----------------------------------------------------------------------------

// Walls::Granular::compute_force (src/fix_wall_gran_base.h:159-372) for one
// wall contact: overlap -deltan, delta = closest wall point - centre, wall
// velocity vwall; c0, c1: the contact's constants (wall_consts); h points at
// the history (stride hs between components)
template <int NORMAL>
__device__ __forceinline__ void wall_force(const Sys &s, const AtomArrays &A, int i, double deltan,
                                           const double delta[3], const double vwall[3],
                                           int wall_type, bool rolling, double c0, double c1, double *h,
                                           size_t hs, int shearupdate, const double v[3], const double om[3],
                                           double &fx, double &fy, double &fz, double &tx,
                                           double &ty, double &tz) {
  const double radi = A.r[i];
  if (deltan <= 0) {
    ContactIn ci;
    ci.radi = radi;
    ci.radj = 0.0;
    ci.deltan_wall = -deltan;
    ci.d[0] = -delta[0];
    ci.d[1] = -delta[1];
    ci.d[2] = -delta[2];
    ci.r = radi - ci.deltan_wall;
    ci.rinv = 1.0 / ci.r;
    ci.en[0] = ci.d[0] * ci.rinv;
    ci.en[1] = ci.d[1] * ci.rinv;
    ci.en[2] = ci.d[2] * ci.rinv;
    ci.radsum = radi;
    ci.reff = radi;
    ci.vr[0] = v[0] - vwall[0];
    ci.vr[1] = v[1] - vwall[1];
    ci.vr[2] = v[2] - vwall[2];
    ci.wi[0] = om[0]; ci.wi[1] = om[1]; ci.wi[2] = om[2];
    ci.wj[0] = ci.wj[1] = ci.wj[2] = 0.0;
    const TypePair tp = load_typepair(s.params, s.ntypes, A.type[i], wall_type);
    ci.c0 = c0;
    ci.c1 = c1;
    double sh3[3] = {h[0], h[hs], h[2 * hs]};
    ContactOut o;
    contact_law<NORMAL, true>(ci, tp, s.dt, s.tdamp, s.limitf, rolling, shearupdate != 0, sh3, o);
    if (shearupdate) {
      h[0] = sh3[0];
      h[hs] = sh3[1];
      h[2 * hs] = sh3[2];
    }
    fx += o.F[0]; fy += o.F[1]; fz += o.F[2];
    tx += o.Ti[0]; ty += o.Ti[1]; tz += o.Ti[2];
  } else {
    h[0] = 0.0; h[hs] = 0.0; h[2 * hs] = 0.0;  // surfacesClose
  }
}

// Constants of atom i's contacts with wall w (planes, then meshes), formed at
// the neighbour build (k_wall_list): two square roots fewer per contact and
// step.
__device__ __forceinline__ void wall_consts(const Sys &s, int w, int i, double &c0, double &c1) {
  c0 = s.wcon[(size_t)(2 * w) * s.nmax + i];
  c1 = s.wcon[(size_t)(2 * w + 1) * s.nmax + i];
}

// component d of a vector in registers (d is the same for the whole warp)
__device__ __forceinline__ double comp(const double v[3], int d) { return d == 0 ? v[0] : (d == 1 ? v[1] : v[2]); }
__device__ __forceinline__ void put(double v[3], int d, double x) {
  if (d == 0) v[0] = x;
  else if (d == 1) v[1] = x;
  else v[2] = x;
}

// plane_contact through plane_law; false (nothing done) where the general law
// has to take it: cylinders, a centre exactly on the plane.  Systems with
// bonds or rolling friction keep the general law throughout, and with it their
// bits: both amplify a changed rounding of any force (the bond stiffness is
// unbounded at zero elongation; CDT's torque has a fixed size along the
// direction of a spin that may be rounding itself: on the 1M hopper a changed
// last bit grew to 2e-8 of the torques in 100 steps).
template <int NORMAL>
__device__ __forceinline__ bool plane_contact_fast(const Sys &s, const AtomArrays &A, int i, int w, int shearupdate,
                                                   const double v[3], const double om[3], const double xv[3],
                                                   double f[3], double t[3]) {
  const Plane &pl = s.planes[w];
  const int n = pl.axis, t1 = n == 2 ? 0 : n + 1, t2 = n == 0 ? 2 : n - 1;
  const double d = comp(xv, n) - plane_pos(pl, A.type[i]);
  if (s.bond || s.rolling || pl.rolling || pl.kind != 0 || (__double_as_longlong(d) << 1) == 0) return false;
  const double radi = A.r[i];
  const double deltan = radi - fabs(d);
  if (-deltan > s.cutneighmax) return true;
  double *h = A.whist + (size_t)(w * 3) * s.nmax + i;
  const size_t hs = s.nmax;
  // a restart's history may have a normal part, which counts until the first update
  if (!shearupdate && (__double_as_longlong(h[n * hs]) << 1) != 0) return false;
  if (!(deltan >= 0)) {  // not touching: the history ends (surfacesClose)
    h[0] = 0.0; h[hs] = 0.0; h[2 * hs] = 0.0;
    return true;
  }
  const int wt = pl.wall_type ? pl.wall_type : A.type[i];
  const TypePair tp = load_typepair(s.params, s.ntypes, A.type[i], wt);
  double c0, c1;
  wall_consts(s, w, i, c0, c1);
  const double vf[3] = {comp(v, n), comp(v, t1), comp(v, t2)};
  const double wf[3] = {comp(om, n), comp(om, t1), comp(om, t2)};
  double s1 = h[t1 * hs], s2 = h[t2 * hs], F[3], T[3];
  plane_law<NORMAL>(d > 0 ? 1.0 : -1.0, radi, deltan, vf, wf, c0, c1, tp, s.dt, s.tdamp, s.limitf,
                    shearupdate != 0, s1, s2, F, T);
  if (shearupdate) {
    h[n * hs] = 0.0;
    h[t1 * hs] = s1;
    h[t2 * hs] = s2;
  }
  put(f, n, F[0]); put(f, t1, F[1]); put(f, t2, F[2]);
  put(t, n, T[0]); put(t, t1, T[1]); put(t, t2, T[2]);
  return true;
}

template <int NORMAL>
__device__ __forceinline__ void plane_contact(const Sys &s, const AtomArrays &A, int i, int w,
                                              int shearupdate, double v[3], double om[3],
                                              double xv[3], double &fx, double &fy, double &fz,
                                              double &tx, double &ty, double &tz) {
  const Plane &pl = s.planes[w];
  const int ax = pl.axis, ay = (ax + 1) % 3, az = (ax + 2) % 3;
  const double radi = A.r[i];
  const double ppos = plane_pos(pl, A.type[i]);
  double delta[3];
  double deltan;
  if (pl.kind == 1) {
    // Cylinder<dim>::resolveContact, src/primitive_wall_definitions.h:170-190,
    // in the reference's operations and order
    const double dy = __dadd_rn(xv[ay], -pl.c1), dz = __dadd_rn(xv[az], -pl.c2);
    const double dist = __dsqrt_rn(__dadd_rn(__dmul_rn(dy, dy), __dmul_rn(dz, dz)));
    if (dist < 1e-13 && dist > -1e-13) {  // compDouble(dist, 0.0)
      delta[0] = delta[1] = delta[2] = 0.;
      deltan = 0.0;
    } else if (dist > ppos) {
      deltan = __dadd_rn(__dadd_rn(dist, -ppos), -radi);
      const double fact = __ddiv_rn(__dadd_rn(dist, -ppos), dist);
      delta[ax] = 0.;
      delta[ay] = __dmul_rn(-dy, fact);
      delta[az] = __dmul_rn(-dz, fact);
    } else {
      deltan = __dadd_rn(__dadd_rn(ppos, -dist), -radi);
      const double fact = __ddiv_rn(__dadd_rn(ppos, -dist), dist);
      delta[ax] = 0.;
      delta[ay] = __dmul_rn(dy, fact);
      delta[az] = __dmul_rn(dz, fact);
    }
  } else if (xv[ax] > ppos) {  // Plane<dim>::resolveContact, src/primitive_wall_definitions.h:123-140
    delta[ax] = ppos - xv[ax];
    deltan = xv[ax] - ppos - radi;
  } else {
    delta[ax] = ppos - xv[ax];
    deltan = ppos - xv[ax] - radi;
  }
  if (pl.kind == 0) {
    delta[ay] = 0.;
    delta[az] = 0.;
  }
  if (deltan > s.cutneighmax) return;
  double *h = A.whist + (size_t)(w * 3) * s.nmax + i;
  const size_t hs = s.nmax;
  const double cdm1 = s.cdf - 1.0;
  if (deltan <= 0 || deltan < cdm1 * radi) {
    const double vwall[3] = {0., 0., 0.};
    double c0, c1;
    wall_consts(s, w, i, c0, c1);
    wall_force<NORMAL>(s, A, i, deltan, delta, vwall, pl.wall_type ? pl.wall_type : A.type[i],
                       pl.rolling != 0, c0, c1, h, hs, shearupdate, v, om, fx, fy, fz, tx, ty, tz);
  } else {
    h[0] = 0.0; h[hs] = 0.0; h[2 * hs] = 0.0;
  }
}

// barycentric node velocity at the contact point (src/fix_wall_gran.cpp:929-934):
// the linear mover's node velocities are all vel, the rotating mover's nodev
__device__ __forceinline__ void mesh_vwall(const MeshDev &M, int t, const double bary[3], double vwall[3]) {
  if (M.rotating) {
    const double *vn = M.nodev + (size_t)t * 9;
    for (int d = 0; d < 3; d++) vwall[d] = (bary[0] * vn[d] + bary[1] * vn[3 + d] + bary[2] * vn[6 + d]);
  } else {
    for (int d = 0; d < 3; d++) vwall[d] = (bary[0] * M.vel[d] + bary[1] * M.vel[d] + bary[2] * M.vel[d]);
  }
}

// SurfaceMesh::areCoplanarNodeNeighs from the precomputed lists
__device__ __forceinline__ bool mesh_coplanar(const MeshDev &M, int a, int b) {
  for (int q = M.cn_start[a]; q < M.cn_start[a + 1]; q++)
    if (M.cn_list[q] == b) return true;
  return false;
}

// triangle id of a slot entry (-1: empty), without the kept mark
__device__ __forceinline__ int slot_tri_of(int v) { return v < 0 ? -1 : (v & ~kSlotKept); }

// FP32 test of candidate triangle t against an atom at xa within reach_f:
// false only when the sphere is beyond the triangle.  Two bounds:
//   plane  |sn.(x - n0)| > reach;
//   edges  the triangle lies behind each of its edge planes (outward in-plane
//          normal en_q), and a contact lies within sqrt(reach^2 - dn^2) of
//          the centre's foot point, so en_q.(x - n_q) beyond that is none.
// The margins cover the FP32 rounding of the copies and of this arithmetic (a
// difference of coordinates is within 5*2^-24 of the sum of their magnitudes;
// 2^-21 is four times that and more), and, for the edges, the 1e-8 by which
// the reference widens its face region.  A rejected candidate would resolve
// to deltan > 0, so leaving it out changes nothing.
struct TriF {
  float4 v[kTrif];
  __device__ __forceinline__ void load(const MeshDev &M, int t) {
#pragma unroll
    for (int k = 0; k < kTrif; k++) v[k] = M.trif[kTrif * (size_t)t + k];
  }
};
__device__ __forceinline__ bool tri_candidate_f(const TriF &T, const float4 &xa, float reach_f) {
  const float4 n0 = T.v[0], sn = T.v[1];
  const float wx = xa.x - n0.x, wy = xa.y - n0.y, wz = xa.z - n0.z;
  const float dn = fabsf(sn.x * wx + sn.y * wy + sn.z * wz);
  const float mag = fabsf(xa.x) + fabsf(xa.y) + fabsf(xa.z) + fabsf(n0.x) + fabsf(n0.y) + fabsf(n0.z);
  const float hi = reach_f + mag * 0x1p-21f;
  if (dn > hi) return false;
  const float lo = fmaxf(0.0f, dn - mag * 0x1p-21f);
  const float rho2 = (hi * hi - lo * lo) * (1.0f + 0x1p-20f) + hi * hi * 0x1p-20f;
#pragma unroll
  for (int q = 0; q < 3; q++) {
    const float4 e = T.v[2 + q];
    const float d = e.x * wx + e.y * wy + e.z * wz - e.w;
    const float m = (mag + fabsf(wx) + fabsf(wy) + fabsf(wz) + fabsf(e.w)) * 0x1p-21f + 4e-8f;
    const float a = d - m;
    if (a > 0.0f && a * a > rho2) return false;
  }
  return true;
}

// The closest-feature contacts of atom i with mesh k, one candidate at a
// time in ascending triangle order (FixWallGran::post_force_mesh with
// FixContactHistoryMesh::handleContact, coplanarContactAlready,
// checkCoplanarContactHistory and cleanUpContacts).  A slot touched in this
// evaluation carries kSlotKept in slot_tri until the clean-up, so the number
// of candidates has no fixed bound.
// acc: the atom's force and torque so far, added to, and the mesh's force.
// Not inlined: a rare path (its code between the tiled path's would cost that
// one instruction fetches, a quarter of its stalls).
template <int NORMAL>
__device__ __noinline__ bool mesh_contacts(const Sys &s, int i, int k, int shearupdate, double acc[9]) {
  const MeshDev &M = s.meshes[k];
  const AtomArrays &A = s.atoms[0];
  const int nc = M.cand_n[i];
  if (nc == 0) return false;
  bool bad = false;
  const double v[3] = {A.vx[i], A.vy[i], A.vz[i]}, om[3] = {A.wx[i], A.wy[i], A.wz[i]};
  const double xv[3] = {A.x[i], A.y[i], A.z[i]};
  const size_t nmax = s.nmax;
  int *st = M.slot_tri[0];
  double *sh = M.slot_hist[0];
  int np = M.npart[0][i];
  const double radi = A.r[i];
  const double cdm1 = s.cdf - 1.0;
  // a triangle is at least as far as its plane: candidates whose plane is
  // clearly beyond the contact range (relative margin 1e-9, far above the
  // rounding of either side) skip the closest-feature resolution; the
  // resolution would return deltan > 0 and skip them as well
  const double reach = __dmul_rn(__dadd_rn(radi, fmax(0.0, __dmul_rn(cdm1, radi))), 1.0 + 1e-9);
  // FP32 bounds first (tri_candidate_f); the rest take the FP64 path below
  const float4 xa = s.xf[i];
  const float reach_f = (float)reach * (1.0f + 0x1p-20f);
  for (int q = 0; q < nc; q++) {
    const int t = M.cand[(size_t)q * nmax + i];
    TriF T;
    T.load(M, t);
    if (!tri_candidate_f(T, xa, reach_f)) continue;
    const double *g = M.tri + (size_t)t * kTriStride;
    {
      const double *sn = tri_sn(g), *n0 = tri_node(g, 0);
      const double dn = sn[0] * (xv[0] - n0[0]) + sn[1] * (xv[1] - n0[1]) + sn[2] * (xv[2] - n0[2]);
      if (fabs(dn) > reach) continue;
    }
    double delta[3], bary[3];
    int bs;
    const double deltan = resolve_tri_sphere(g, M.meta[t], radi, xv, delta, bary, bs);
    if (deltan > s.cutneighmax) continue;
    if (!(deltan <= 0 || deltan < cdm1 * radi)) continue;
    int slot = -1;
    for (int u = 0; u < nc; u++)
      if (slot_tri_of(st[u * nmax + i]) == t) { slot = u; break; }
    if (slot >= 0) {
      st[slot * nmax + i] |= kSlotKept;
    } else {
      const bool face = bs == 7;
      if (face) {  // coplanarContactAlready
        bool already = false;
        for (int u = 0; u < nc; u++) {
          const int sv = st[u * nmax + i];
          const int p = slot_tri_of(sv);
          if (p >= 0 && p != t && (sv & kSlotKept) && mesh_coplanar(M, p, t)) already = true;
        }
        if (already) continue;
      }
      if (np >= nc) { bad = true; continue; }
      for (int u = 0; u < nc; u++)
        if (st[u * nmax + i] == -1) { slot = u; break; }
      st[slot * nmax + i] = t | kSlotKept;
      for (int d = 0; d < 3; d++) sh[(3 * slot + d) * nmax + i] = 0.0;
      np++;
      if (face)  // checkCoplanarContactHistory
        for (int u = 0; u < nc; u++) {
          const int p = slot_tri_of(st[u * nmax + i]);
          if (p >= 0 && p != t && mesh_coplanar(M, p, t))
            for (int d = 0; d < 3; d++) sh[(3 * slot + d) * nmax + i] = sh[(3 * u + d) * nmax + i];
        }
    }
    double vwall[3] = {0., 0., 0.};
    if (M.moving && M.vel_on) mesh_vwall(M, t, bary, vwall);
    double cfx = 0., cfy = 0., cfz = 0., ctx = 0., cty = 0., ctz = 0.;
    double c0, c1;
    wall_consts(s, s.nplanes + k, i, c0, c1);
    wall_force<NORMAL>(s, A, i, deltan, delta, vwall, M.wall_type, M.rolling != 0, c0, c1,
                         sh + (size_t)(3 * slot) * nmax + i, nmax, shearupdate, v, om, cfx, cfy, cfz, ctx, cty, ctz);
    acc[0] += cfx; acc[1] += cfy; acc[2] += cfz;
    acc[3] += ctx; acc[4] += cty; acc[5] += ctz;
    acc[6] += cfx; acc[7] += cfy; acc[8] += cfz;
  }
  for (int u = 0; u < nc; u++) {  // cleanUpContacts
    const int sv = st[u * nmax + i];
    if (sv >= 0 && (sv & kSlotKept)) {
      st[u * nmax + i] = sv & ~kSlotKept;
    } else {
      if (sv > -1) np--;
      st[u * nmax + i] = -1;
      for (int d = 0; d < 3; d++) sh[(3 * u + d) * nmax + i] = 0.0;
    }
  }
  M.npart[0][i] = np;
  return bad;
}

// FixWallGran::post_force_primitive / post_force_mesh for the atoms near a
// wall (the compact list of k_wall_list): wall forces and torques of the
// current state, planes then meshes in order, into fm/tm.  Independent of
// the pair kernel of the same step (it reads positions and velocities and
// writes only the wall histories, mesh slots and fm/tm), so the two run side
// by side; the per-atom kernel adds fm/tm.
//
// A warp takes a tile of 32 listed atoms (one lane each) and, per mesh, runs
// the FP64-heavy parts densely over the tile's work instead of per atom (the
// FP64 pipe issues per warp instruction, and atoms differ in their number of
// candidates and contacts):
//   A  per atom, FP32: the candidates the triangle bounds cannot reject
//      (tri_candidate_f), queued in ascending order;
//   B  per queued candidate: closest feature
//      (TriMesh::resolveTriSphereContactBary), kept when touching;
//   C  per atom, integer work in candidate order: FixContactHistoryMesh's
//      slot semantics (handleContact, coplanarContactAlready); an atom whose
//      new face contact would copy a coplanar neighbour's history
//      (checkCoplanarContactHistory) takes the sequential path instead,
//      since that copy depends on the order of the contact updates;
//   D  per contact: the contact law with the slot's history;
//   E  per atom: contact forces summed in candidate order, slot clean-up.
// Atoms without a touching candidate and without an occupied slot do nothing
// after B (their slots are empty, with zero history).  A tile whose queue
// would exceed its capacity (cap entries, a launch parameter) runs the
// sequential path for all its atoms.  Both paths give the same result.
//
// The launch is bound by latency: the phases are one dependent chain, a few
// warps per SM.  A warp per tile keeps the phases free of block barriers, and
// the edge bounds leave B about one candidate per contact (with the plane
// bound alone the conical mesh's tiles queued several per atom, three to five
// FP64 passes of B).  A runs over the tile's (atom, candidate) pairs, 32 at a
// time, the next ones' triangles on their way, and sends for the records that B
// will read; an atom at a time, it took 14 candidates' trips to L2 in a row.  C
// and E walk the slots in use instead of all of them, and the sequential path is
// a function of its own (instruction fetches were a quarter of the stalls):
// 100,000 spheres' wall kernel 42 -> 35 us.  Against 64-atom tiles with block barriers and the plane
// bound: the 100,000-sphere hopper's step 84 -> 67 us, the 1M one's 0.318 ->
// 0.309 ms (50 steps per call).
constexpr int kWallTile = 32;
constexpr int kWallWarps = 2;       // tiles (warps) per block
constexpr int kWallCapDefault = 4;  // queue entries per tile atom (LIGGGHTS_GB300_WALL_CAP)
constexpr int kWallRes = 7;  // doubles per queued candidate: deltan, delta[3], vwall[3]; then F[3], T[3]
constexpr int kWallQ = kWallRes * 8 + 4 + 2;  // result doubles, state int, atom and candidate bytes

// one warp's queue of `cap` entries in shared memory
struct WallQueue {
  double *res;             // [cap * kWallRes]
  int *st;                 // bit 0 touching, bit 1 face, bits 8+: contact slot + 1
  unsigned char *qa, *qq;  // tile atom, candidate index
};

template <int NORMAL>
__device__ __forceinline__ void wall_tile(const Sys &s, const AtomArrays &A, int base, int nl, int shearupdate,
                                          int cap, const WallQueue &w, bool &meshbad) {
  const size_t nmax = s.nmax;
  const double cdm1 = s.cdf - 1.0;
  const int a = threadIdx.x & 31;
  const bool valid = base + a < nl;
  const int i = valid ? s.mlist[base + a] : 0;
  double v[3] = {0., 0., 0.}, om[3] = {0., 0., 0.}, xv[3] = {0., 0., 0.};
  double fx = 0., fy = 0., fz = 0., tx = 0., ty = 0., tz = 0.;
  if (valid) {
    v[0] = A.vx[i]; v[1] = A.vy[i]; v[2] = A.vz[i];
    om[0] = A.wx[i]; om[1] = A.wy[i]; om[2] = A.wz[i];
    xv[0] = A.x[i]; xv[1] = A.y[i]; xv[2] = A.z[i];
    const uint8_t bits = A.wbits[i];
    for (int k = 0; k < s.nplanes; k++) {
      double pf[3] = {0., 0., 0.}, pt[3] = {0., 0., 0.};
      if ((bits & (1u << k)) && !plane_contact_fast<NORMAL>(s, A, i, k, shearupdate, v, om, xv, pf, pt))
        plane_contact<NORMAL>(s, A, i, k, shearupdate, v, om, xv, pf[0], pf[1], pf[2], pt[0], pt[1], pt[2]);
      fx += pf[0]; fy += pf[1]; fz += pf[2];
      tx += pt[0]; ty += pt[1]; tz += pt[2];
      for (int d = 0; d < 3; d++) s.wforce[(size_t)(3 * k + d) * nmax + i] = pf[d];
    }
  }
  for (int k = 0; k < s.nmeshes; k++) {
    const MeshDev &M = s.meshes[k];
    int *st = M.slot_tri[0];
    double *sh = M.slot_hist[0];
    const auto sequential = [&](double sum[3]) {
      double acc[9] = {fx, fy, fz, tx, ty, tz, 0., 0., 0.};
      meshbad |= mesh_contacts<NORMAL>(s, i, k, shearupdate, acc);
      fx = acc[0]; fy = acc[1]; fz = acc[2];
      tx = acc[3]; ty = acc[4]; tz = acc[5];
      for (int d = 0; d < 3; d++) sum[d] = acc[6 + d];
    };
    // ---- A: FP32 candidate pass
    const int nc = valid ? M.cand_n[i] : 0;
    unsigned todo = 0u;
    int np = 0;
    const bool big = nc > kMeshFastCand;  // beyond the 32-bit masks: sequential path
    const int na = big ? 0 : nc;
    if (na > 0) np = M.npart[0][i];
    {
      const int last = warp_incl_scan(na), pairs = __shfl_sync(0xffffffffu, last, 31), beg = last - na;
      const float4 xa = na > 0 ? s.xf[i] : make_float4(0.f, 0.f, 0.f, 0.f);
      const float reach_f = xa.w * fmaxf(1.0f, s.cdff) * (1.0f + 0x1p-19f);
      // a pair's atom (the first whose pairs end behind it), its candidate
      const auto pair_of = [&](int f, int &o) {
        o = 0;
#pragma unroll
        for (int h = 16; h > 0; h >>= 1)
          if (__shfl_sync(0xffffffffu, last, o + h - 1) <= f) o += h;
        const int io = __shfl_sync(0xffffffffu, i, o), q = f - __shfl_sync(0xffffffffu, beg, o);
        return f < pairs ? M.cand[(size_t)q * nmax + io] : 0;
      };
      // lane a tests pair f0 + a; the next round's candidates are on their way
      int on, tn = pair_of(a, on);
      for (int f0 = 0; f0 < pairs; f0 += 32) {
        const int o = on, t = tn;
        TriF T;
        T.load(M, t);
        if (f0 + 32 < pairs) tn = pair_of(f0 + 32 + a, on);
        const float4 xo = make_float4(__shfl_sync(0xffffffffu, xa.x, o), __shfl_sync(0xffffffffu, xa.y, o),
                                      __shfl_sync(0xffffffffu, xa.z, o), 0.f);
        const float ro = __shfl_sync(0xffffffffu, reach_f, o);
        const bool pass = f0 + a < pairs && tri_candidate_f(T, xo, ro);
        if (pass) {  // phase B reads its record
          const char *g = reinterpret_cast<const char *>(M.tri + (size_t)t * kTriStride);
          for (int k = 0; k < 3; k++) asm volatile("prefetch.global.L1 [%0];" ::"l"(g + 128 * k));
          asm volatile("prefetch.global.L1 [%0];" ::"l"(M.meta + t));
        }
        const unsigned b = __ballot_sync(0xffffffffu, pass);
        const int at = beg - f0;  // this lane's first pair in the ballot
        if (at > -32 && at < 32) todo |= at >= 0 ? b >> at : b << -at;
      }
      todo &= na >= 32 ? 0xffffffffu : (1u << na) - 1u;
    }
    const int cnt = __popc(todo);
    const int inc = warp_incl_scan(cnt);
    const int total = __shfl_sync(0xffffffffu, inc, 31);
    const int off = inc - cnt;
    double msum[3] = {0., 0., 0.};
    double *const wf = s.wforce + (size_t)(3 * (s.nplanes + k)) * nmax;
    if (total > cap) {  // sequential path for this tile
      if (nc > 0) sequential(msum);
      if (valid)
        for (int d = 0; d < 3; d++) wf[(size_t)d * nmax + i] = msum[d];
      __syncwarp();
      continue;
    }
    {
      unsigned m = todo;
      for (int e = off; m; e++) {
        w.qa[e] = (unsigned char)a;
        w.qq[e] = (unsigned char)(__ffs(m) - 1);
        m &= m - 1u;
      }
    }
    __syncwarp();
    // ---- B: closest feature per queued candidate
    for (int e = a; e < total; e += kWallTile) {
      const int ie = s.mlist[base + w.qa[e]];
      const int t = M.cand[(size_t)w.qq[e] * nmax + ie];
      const double *g = M.tri + (size_t)t * kTriStride;
      const double xe[3] = {A.x[ie], A.y[ie], A.z[ie]};
      const double re = A.r[ie];
      int state = 0;
      {
        double delta[3], bary[3];
        int bs;
        const double deltan = resolve_tri_sphere(g, M.meta[t], re, xe, delta, bary, bs);
        if (!(deltan > s.cutneighmax) && (deltan <= 0 || deltan < cdm1 * re)) {
          state = 1 | (bs == 7 ? 2 : 0);
          double *r = w.res + (size_t)e * kWallRes;
          r[0] = deltan;
          r[1] = delta[0]; r[2] = delta[1]; r[3] = delta[2];
          double vwall[3] = {0., 0., 0.};
          if (M.moving && M.vel_on) mesh_vwall(M, t, bary, vwall);
          r[4] = vwall[0]; r[5] = vwall[1]; r[6] = vwall[2];
        }
      }
      w.st[e] = state;
    }
    __syncwarp();
    // ---- C: slot semantics per atom, in candidate order
    bool fallback = big;
    unsigned keep = 0u;
    unsigned occ = 0u;  // slots in use
    int stl[kMeshFastCand];
    bool work = np > 0 && !big;
    for (int e = off; e < off + cnt; e++) work |= (w.st[e] & 1) != 0;
    if (work) {
      unsigned fresh = 0u;
#pragma unroll 4
      for (int u = 0; u < nc; u++) {
        const int v = st[u * nmax + i];
        stl[u] = v;
        occ |= (v >= 0 ? 1u : 0u) << u;
      }
      for (int e = off; e < off + cnt && !fallback; e++) {
        if (!(w.st[e] & 1)) continue;
        const int t = M.cand[(size_t)w.qq[e] * nmax + i];
        int slot = -1;
        for (unsigned m = occ; m; m &= m - 1u)
          if (stl[__ffs(m) - 1] == t) { slot = __ffs(m) - 1; break; }
        if (slot >= 0) {
          keep |= 1u << slot;
        } else {
          const bool face = (w.st[e] & 2) != 0;
          if (face) {  // coplanarContactAlready
            bool already = false;
            for (unsigned m = occ & keep; m; m &= m - 1u) already |= mesh_coplanar(M, stl[__ffs(m) - 1], t);
            if (already) continue;
          }
          slot = __ffs(~occ) - 1;
          if (np >= nc || slot < 0 || slot >= nc) { meshbad = true; continue; }
          if (face)  // checkCoplanarContactHistory would copy: order-dependent
            for (unsigned m = occ; m; m &= m - 1u) fallback |= mesh_coplanar(M, stl[__ffs(m) - 1], t);
          if (fallback) break;
          stl[slot] = t;
          occ |= 1u << slot;
          keep |= 1u << slot;
          fresh |= 1u << slot;
          np++;
        }
        w.st[e] |= (slot + 1) << 8;
      }
      if (fallback) {
        for (int e = off; e < off + cnt; e++) w.st[e] &= 0xff;
      } else {
        for (unsigned m = fresh; m; m &= m - 1u) {
          const int u = __ffs(m) - 1;
          st[u * nmax + i] = stl[u];
          for (int d = 0; d < 3; d++) sh[(3 * u + d) * nmax + i] = 0.0;
        }
      }
    }
    __syncwarp();
    // ---- D: contact law per contact
    for (int e = a; e < total; e += kWallTile) {
      const int slot = (w.st[e] >> 8) - 1;
      if (slot < 0) continue;
      const int ie = s.mlist[base + w.qa[e]];
      double *r = w.res + (size_t)e * kWallRes;
      const double delta[3] = {r[1], r[2], r[3]};
      const double vwall[3] = {r[4], r[5], r[6]};
      double ve[3] = {A.vx[ie], A.vy[ie], A.vz[ie]};
      double oe[3] = {A.wx[ie], A.wy[ie], A.wz[ie]};
      double cfx = 0., cfy = 0., cfz = 0., ctx = 0., cty = 0., ctz = 0.;
      double c0, c1;
      wall_consts(s, s.nplanes + k, ie, c0, c1);
      wall_force<NORMAL>(s, A, ie, r[0], delta, vwall, M.wall_type, M.rolling != 0, c0, c1,
                         sh + (size_t)(3 * slot) * nmax + ie, nmax, shearupdate, ve, oe, cfx, cfy, cfz, ctx, cty,
                         ctz);
      r[0] = cfx; r[1] = cfy; r[2] = cfz;
      r[3] = ctx; r[4] = cty; r[5] = ctz;
    }
    __syncwarp();
    // ---- E: sums in candidate order, clean-up (or the sequential path)
    if (fallback) {
      sequential(msum);
    } else if (work) {
      for (int e = off; e < off + cnt; e++) {
        if ((w.st[e] >> 8) == 0) continue;
        const double *r = w.res + (size_t)e * kWallRes;
        fx += r[0]; fy += r[1]; fz += r[2];
        tx += r[3]; ty += r[4]; tz += r[5];
        msum[0] += r[0]; msum[1] += r[1]; msum[2] += r[2];
      }
      for (unsigned m = occ & ~keep; m; m &= m - 1u) {  // cleanUpContacts
        const int u = __ffs(m) - 1;
        np--;
        st[u * nmax + i] = -1;
        for (int d = 0; d < 3; d++) sh[(3 * u + d) * nmax + i] = 0.0;
      }
      M.npart[0][i] = np;
    }
    if (valid)
      for (int d = 0; d < 3; d++) wf[(size_t)d * nmax + i] = msum[d];
    __syncwarp();
  }
  if (valid) {
    A.fmx[i] = fx; A.fmy[i] = fy; A.fmz[i] = fz;
    A.tmx[i] = tx; A.tmy[i] = ty; A.tmz[i] = tz;
  }
}

// Force gather of one atom: its own row (ascending), then its reverse list
// (ascending), the reference's per-atom order.  The FP64 pipe issues per warp
// instruction, so additions inside a loop over all list entries cost one
// issue per entry of the warp's longest row, active or not.  Here a first,
// integer-only pass collects the active entries of up to 32 entries per list
// as bit masks (gather_masks); one loop over the set bits then does the FP64
// additions (gather_sum).  A reverse contribution adds the negated force
// (sign bit flipped on the integer pipe: a + (-b) is exactly a - b) and Tj
// instead of Ti.  (particle_tile spreads the components over the lanes.)
template <int GROUP>
__device__ __forceinline__ bool gather_masks(const Sys &s, const PairArrays &L, int i, int &pb, int &rb,
                                             unsigned &om, unsigned &rm) {
  pb = L.row[i];
  rb = L.rev_start[i];
  const int pe = row_end(s, L, i), re = rev_end(s, L, i);
  if (pe - pb > 32 || re - rb > 32) return false;
  om = 0u;
  rm = 0u;
  // the flags in groups of loads that do not wait for one another
  const int no = pe - pb, nr = re - rb;
  for (int k0 = 0; k0 < max(no, nr); k0 += GROUP) {
    int e[GROUP];
    uint8_t ao[GROUP], ar[GROUP];
#pragma unroll
    for (int k = 0; k < GROUP; k++) {
      e[k] = k0 + k < nr ? L.rev[rb + k0 + k] : -1;
      ao[k] = k0 + k < no ? s.active[pb + k0 + k] : 0;
    }
#pragma unroll
    for (int k = 0; k < GROUP; k++) ar[k] = e[k] >= 0 ? s.active[e[k]] : 0;
#pragma unroll
    for (int k = 0; k < GROUP; k++) {
      om |= (ao[k] ? 1u : 0u) << (k0 + k);
      rm |= (ar[k] ? 1u : 0u) << (k0 + k);
    }
  }
  return true;
}

// takes the next set bit of om, then rm: the entry, the sign bit of its force
// and the offset of its torque in the record (Ti: own row, Tj: partner)
__device__ __forceinline__ const double *gather_next(const Sys &s, const PairArrays &L, int pb, int rb, unsigned &om,
                                                     unsigned &rm, unsigned long long &sg, int &to) {
  int p;
  if (om) {
    p = pb + __ffs(om) - 1;
    om &= om - 1u;
    sg = 0ull;
    to = 3;
  } else {
    p = L.rev[rb + __ffs(rm) - 1];
    rm &= rm - 1u;
    sg = 0x8000000000000000ull;
    to = 6;
  }
  return s.res + (size_t)kResStride * p;
}

// the next record is loaded while this one is added (a record's loads take
// twice as long as its six additions)
__device__ __forceinline__ void gather_sum(const Sys &s, const PairArrays &L, int pb, int rb, unsigned om,
                                           unsigned rm, double &fx, double &fy, double &fz, double &tx, double &ty,
                                           double &tz) {
  const int cnt = __popc(om) + __popc(rm);
  unsigned long long sg = 0ull;
  int to = 3;
  double r[6];
  if (cnt > 0) {
    const double *q = gather_next(s, L, pb, rb, om, rm, sg, to);
    for (int k = 0; k < 3; k++) {
      r[k] = q[k];
      r[3 + k] = q[to + k];
    }
  }
  for (int t = 0; t < cnt; t++) {
    double n[6];
    const unsigned long long su = sg;
    if (t + 1 < cnt) {
      const double *q = gather_next(s, L, pb, rb, om, rm, sg, to);
      for (int k = 0; k < 3; k++) {
        n[k] = q[k];
        n[3 + k] = q[to + k];
      }
    }
    fx += __longlong_as_double(__double_as_longlong(r[0]) ^ su);
    fy += __longlong_as_double(__double_as_longlong(r[1]) ^ su);
    fz += __longlong_as_double(__double_as_longlong(r[2]) ^ su);
    tx += r[3];
    ty += r[4];
    tz += r[5];
    for (int k = 0; k < 6; k++) r[k] = n[k];
  }
}

// lists that fit neither form: one pass over every entry
__device__ __forceinline__ void gather_long(const Sys &s, const PairArrays &L, int i, double &fx, double &fy,
                                            double &fz, double &tx, double &ty, double &tz) {
  const int pb = L.row[i], pe = row_end(s, L, i);
  const int rb = L.rev_start[i], re = rev_end(s, L, i);
  for (int p = pb; p < pe; p++) {
    if (!s.active[p]) continue;
    const double *r = s.res + (size_t)kResStride * p;
    fx += r[0]; fy += r[1]; fz += r[2];
    tx += r[3]; ty += r[4]; tz += r[5];
  }
  for (int k = rb; k < re; k++) {
    const int p = L.rev[k];
    if (!s.active[p]) continue;
    const double *r = s.res + (size_t)kResStride * p;
    fx -= r[0]; fy -= r[1]; fz -= r[2];
    tx += r[6]; ty += r[7]; tz += r[8];
  }
}

// shared memory of particle_tile's gather, per warp: the atoms' contacts (own
// entries from the front, the partner list's from the back), their sums, and
// the atoms in the order of their contact counts
constexpr int kGatherList = 16;
constexpr int kGatherBatch = 4;  // records in flight per lane
constexpr int kGatherSum = 7;  // doubles per atom: six and one that spreads the banks
constexpr int kParticleMaxThreads = 256;
template <int T>
struct ParticleShared {
  int list[T / 32][kGatherList][32];
  double sum[T / 32][32 * kGatherSum];
  unsigned char order[T / 32][32];
};

// the active entries of atom i into `list` (this lane's column, see above):
// own count | total << 8, or -1 when they do not fit
__device__ __forceinline__ int gather_list(const Sys &s, const PairArrays &L, int i, int (*list)[32], int lane) {
  constexpr int kGroup = 4;
  const int pb = L.row[i], rb = L.rev_start[i];
  const int no = row_end(s, L, i) - pb, nr = rev_end(s, L, i) - rb;
  int co = 0, cr = 0;
  // the flags in groups of loads that do not wait for one another
  for (int k0 = 0; k0 < max(no, nr); k0 += kGroup) {
    int e[kGroup];
    uint8_t ao[kGroup], ar[kGroup];
#pragma unroll
    for (int k = 0; k < kGroup; k++) {
      e[k] = k0 + k < nr ? L.rev[rb + k0 + k] : -1;
      ao[k] = k0 + k < no ? s.active[pb + k0 + k] : 0;
    }
#pragma unroll
    for (int k = 0; k < kGroup; k++) ar[k] = e[k] >= 0 ? s.active[e[k]] : 0;
#pragma unroll
    for (int k = 0; k < kGroup; k++) {
      if (ao[k]) {
        if (co + cr == kGatherList) return -1;
        list[co++][lane] = pb + k0 + k;
      }
      if (ar[k]) {
        if (co + cr == kGatherList) return -1;
        list[kGatherList - 1 - cr++][lane] = e[k];
      }
    }
  }
  return co | (co + cr) << 8;
}

// v += r where the program says so: left to itself the compiler adds first and
// selects the result after, and an addition that is not needed holds the FP64
// pipe as long as one that is
__device__ __forceinline__ void add_now(double &v, double r) {
  asm volatile("add.rn.f64 %0, %0, %1;" : "+d"(v) : "d"(r));
}

// the sums of a warp's atoms over their lists, started from and left in `sum`;
// cnt: gather_list's result of this lane's atom
__device__ __forceinline__ void gather_warp(const Sys &s, const int (*list)[32], double *sum, unsigned char *order,
                                            int cnt, int lane) {
  const int key = cnt < 0 ? 0 : cnt >> 8;
  const int top = __reduce_max_sync(0xffffffffu, key);
  if (top == 0) return;
  unsigned more = 0u, same = 0u;  // lanes with a larger, with the same count
  int nq = 0;
  for (int k = 1; k <= top; k++) {
    const unsigned b = __ballot_sync(0xffffffffu, key >= k);
    if (k == 1) nq = __popc(b);
    if (k == key) same = b;
    if (k == key + 1) more = b;
  }
  if (key) order[__popc(more) + __popc(same & ~more & ((1u << lane) - 1u))] = (unsigned char)lane;
  __syncwarp();
  // one batch of records is loaded while the one before it is added
  const int slot = lane / 6, comp = lane % 6;
  // of a partner's entry the negated force, the other torque
  const int torque = comp < 3 ? 0 : 3, flip = comp < 3 ? (int)0x80000000 : 0;
  int a = 0, co = 0, n = 0, m = 0;  // the atom, its own count and total, the group's largest total
  auto group = [&](int g) {
    const bool on = lane < 30 && g + slot < nq;
    a = on ? order[g + slot] : 0;
    const int ca = __shfl_sync(0xffffffffu, cnt, a);
    co = ca & 0xff;
    n = on ? ca >> 8 : 0;
    m = __shfl_sync(0xffffffffu, n, 0);
  };
  auto load = [&](double (&r)[kGatherBatch], int k0) {
#pragma unroll
    for (int k = 0; k < kGatherBatch; k++) {
      const int t = k0 + k;
      r[k] = -0.0;  // changes no sum
      if (t < n) {
        const bool own = t < co;
        const int p = list[own ? t : kGatherList - 1 - (t - co)][a];
        const double x = s.res[(size_t)kResStride * p + comp + (own ? 0 : torque)];
        // (a constant sign bit would become a negation, which issues on the FP64 pipe)
        r[k] = __hiloint2double(__double2hiint(x) ^ (own ? 0 : flip), __double2loint(x));
      }
    }
  };
  int g = 0, k0 = 0;
  double r[kGatherBatch];
  group(0);
  load(r, 0);
  double v = sum[a * kGatherSum + comp];
  while (g < nq) {
    const int left = m - k0, ga = a, gn = n;
    const bool done = left <= kGatherBatch;
    double q[kGatherBatch];
    if (!done) {
      k0 += kGatherBatch;
      load(q, k0);
    } else {
      g += 5;
      k0 = 0;
      if (g < nq) {
        group(g);
        load(q, 0);
      }
    }
#pragma unroll
    for (int k = 0; k < kGatherBatch; k++) {
      if (k >= left) break;
      add_now(v, r[k]);
    }
    if (done) {
      if (gn) sum[ga * kGatherSum + comp] = v;
      if (g < nq) v = sum[a * kGatherSum + comp];
    }
#pragma unroll
    for (int k = 0; k < kGatherBatch; k++) r[k] = q[k];
  }
  __syncwarp();
}

// 2x by the bits (exact; a multiplication, even one that is predicated off,
// holds the FP64 pipe): the exponent up by one, a denormal's mantissa (or zero)
// to the left, infinity from the top binade on
__device__ __forceinline__ double twice(double x) {
  const unsigned hi = (unsigned)__double2hiint(x), lo = (unsigned)__double2loint(x), e = hi & 0x7ff00000u;
  unsigned h = hi + 0x00100000u, l = lo;
  if (e == 0u) {
    h = (hi & 0x80000000u) | (__funnelshift_l(lo, hi, 1) & 0x7fffffffu);
    l = lo << 1;
  } else if (e == 0x7fe00000u) {
    h = (hi & 0x80000000u) | 0x7ff00000u;
    l = 0u;
  } else if (e == 0x7ff00000u) {
    h = hi;
  }
  return __hiloint2double((int)h, (int)l);
}

// (float)x on the integer pipe, for the FP32 copies of coordinates (the
// conversion issues on the FP64 pipe, also predicated off): round to nearest
// even, the top 24 bits of the mantissa and one unit more where the rest says
// so; a carry runs into the exponent as it should.  Below 2^-126 zero; from
// 2^128 on infinity, NaN included (a non-finite copy is what the check of the
// coordinates looks for).
__device__ __forceinline__ float to_float(double x) {
  const unsigned hi = (unsigned)__double2hiint(x), lo = (unsigned)__double2loint(x);
  const unsigned mag = hi & 0x7fffffffu;
  unsigned f = __funnelshift_l(lo, mag, 3) - (0x380u << 23);
  const unsigned rest = lo & 0x1fffffffu;
  f += (rest + 0x0fffffffu + (f & 1u)) >> 29;
  if (mag < 0x38100000u) f = 0u;
  if (mag >= 0x47f00000u) f = 0x7f800000u;
  return __uint_as_float(f | (hi & 0x80000000u));
}

// FixGravity::post_force (src/fix_gravity.cpp:329-337) adds m*g after the pair
// forces; starting the sum from it instead changes only the rounding order and
// saves three FP64 additions.  A component of +0 gives +0 without a product.
// The components that are not +0 come first in s.gaxis: a loop, not three
// conditions, whose products would issue predicated off.
__device__ __forceinline__ void gravity_force(const Sys &s, double m, double &fx, double &fy, double &fz) {
#pragma unroll 1
  for (int k = 0; k < s.gcount; k++) {
    const int d = s.gaxis[k];
    const double f = __dmul_rn(m, s.g[d]);
    if (d == 0) fx = f;
    if (d == 1) fy = f;
    if (d == 2) fz = f;
  }
}

// nve/sphere, FP32 copy and displacement check of atom i with its summed force
// and torque (hf: the FP32 position at the last build, in w the FP32 radius)
__device__ __forceinline__ void particle_finish(const Sys &s, int i, bool gather, bool final, bool initial, double fx,
                                                double fy, double fz, double tx, double ty, double tz, double v[3],
                                                double om[3], double xv[3], double dtfm, double dtir,
                                                const float4 &hf, bool &moved, bool &bad) {
  const AtomArrays &A = s.atoms[0];
  // the sums are kept for the download and the next call's first
  // step; inside a run (final && initial) nothing reads them
  if (gather && !(final && initial)) {
    A.fx[i] = fx; A.fy[i] = fy; A.fz[i] = fz;
    A.tx[i] = tx; A.ty[i] = ty; A.tz[i] = tz;
  }
  if (!(final || initial)) return;
  // FixNVESphere half-kicks and drift as fused multiply-adds: one FP64
  // instruction each (the FP64 pipe bounds this kernel on GB300); the
  // single rounding moves positions by at most an ulp from the reference.
  // The final half-kick of step n and the initial one of step n+1 use
  // the same force: fused into one FMA with 2*dtfm (2*dtir), exact
  // scalings, one rounding instead of two.
  if (final && initial) {
    const double kf = twice(dtfm), kt = twice(dtir);
    v[0] = fma(kf, fx, v[0]);
    v[1] = fma(kf, fy, v[1]);
    v[2] = fma(kf, fz, v[2]);
    om[0] = fma(kt, tx, om[0]);
    om[1] = fma(kt, ty, om[1]);
    om[2] = fma(kt, tz, om[2]);
  } else if (final || initial) {
    v[0] = fma(dtfm, fx, v[0]);
    v[1] = fma(dtfm, fy, v[1]);
    v[2] = fma(dtfm, fz, v[2]);
    om[0] = fma(dtir, tx, om[0]);
    om[1] = fma(dtir, ty, om[1]);
    om[2] = fma(dtir, tz, om[2]);
  }
  if (initial) {
    xv[0] = fma(s.dt, v[0], xv[0]);
    xv[1] = fma(s.dt, v[1], xv[1]);
    xv[2] = fma(s.dt, v[2], xv[2]);
    A.x[i] = xv[0]; A.y[i] = xv[1]; A.z[i] = xv[2];
    // the FP32 radius of the copy does not change: no conversion
    const float4 nf = make_float4(to_float(xv[0]), to_float(xv[1]), to_float(xv[2]), hf.w);
    s.xf[i] = nf;
    // Neighbor::check_distance (src/neighbor.cpp:1426-1466) with an FP32
    // prefilter: only displacements within the rounding band of skin/2
    // take the exact FP64 test, so the decision is the reference's
    const float ex = nf.x - hf.x, ey = nf.y - hf.y, ez = nf.z - hf.z;
    const float rf2 = ex * ex + ey * ey + ez * ez;
    bool mv = false;
    if (rf2 > s.skin_hi2) {
      mv = true;
    } else if (rf2 > s.skin_lo2) {
      const double dx = __dadd_rn(xv[0], -A.xh[i]);
      const double dy = __dadd_rn(xv[1], -A.yh[i]);
      const double dz = __dadd_rn(xv[2], -A.zh[i]);
      if (rsq_rn(dx, dy, dz) > 0.25 * s.skin * s.skin) mv = true;
    }
    if (mv && s.nsys) s.sys_moved[A.type[i] - 1] = 1;  // this atom's system (ensembles)
    moved |= mv;
    // a non-finite coordinate converts to a non-finite float (so does one
    // beyond the FP32 range, which no granular box reaches)
    if (!(isfinite(nf.x) && isfinite(nf.y) && isfinite(nf.z))) bad = true;
  }
  A.vx[i] = v[0]; A.vy[i] = v[1]; A.vz[i] = v[2];
  A.wx[i] = om[0]; A.wy[i] = om[1]; A.wz[i] = om[2];
}

// Per atom: force gather, gravity, wall totals, nve/sphere, FP32 copy,
// displacement check.  The FP64 pipe issues per warp instruction, so that a
// gather with one lane per atom costs six additions per contact of the warp's
// busiest atom.  Here a lane adds one of the six components of one atom: five
// atoms at a time, taken in the order of their contact counts, so that the
// lanes of a warp run loops of nearly equal length and a record is read by
// neighbouring lanes.  Warps work on their own: they reach the FP64 pipe at
// different times.  Each sum keeps its order, so the result does not depend on
// any of this.  Bound by the latency of its four dependent loads (FP64 pipe 44 %
// busy on the hopper, 48 % on the packed bed); measured against one lane per
// atom sorted over a block of 256 (pipe 42-50 % busy, its warps all waiting for
// the same phase): 1,000,000 atoms in a hopper 101 -> 77 us, 400,000 packed 81 ->
// 71, 526,000 of an ensemble 46 -> 39; and with no conversion, doubling or product
// issued in vain (a quarter of its FP64 instructions were predicated off) 74, 70
// and 36.  More blocks per SM (48 registers), larger batches and prefetches of
// the atom's state were slower.
// Called by all lanes of a warp, each with its atom i (valid or none).
template <int T>
__device__ __forceinline__ void particle_tile(const Sys &s, ParticleShared<T> &sm, int i, bool valid, bool gather,
                                              bool final, bool initial, bool &moved, bool &bad) {
  const AtomArrays &A = s.atoms[0];
  const PairArrays &L = s.pairs[0];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  double fx = 0.0, fy = 0.0, fz = 0.0, tx = 0.0, ty = 0.0, tz = 0.0;
  if (gather) {
    if (valid && s.gravity_on) gravity_force(s, A.m[i], fx, fy, fz);
    const int cnt = valid ? gather_list(s, L, i, sm.list[w], lane) : 0;
    double *sum = &sm.sum[w][lane * kGatherSum];
    if (cnt > 0) {
      sum[0] = fx; sum[1] = fy; sum[2] = fz;
      sum[3] = tx; sum[4] = ty; sum[5] = tz;
    }
    __syncwarp();
    gather_warp(s, sm.list[w], sm.sum[w], sm.order[w], cnt, lane);
    if (cnt > 0) {
      fx = sum[0]; fy = sum[1]; fz = sum[2];
      tx = sum[3]; ty = sum[4]; tz = sum[5];
    }
    if (cnt < 0) gather_long(s, L, i, fx, fy, fz, tx, ty, tz);
    __syncwarp();
  }
  if (!valid) return;
  double v[3] = {A.vx[i], A.vy[i], A.vz[i]}, om[3] = {A.wx[i], A.wy[i], A.wz[i]};
  double xv[3] = {A.x[i], A.y[i], A.z[i]};
  if (gather) {
    if (A.wbits[i] & 0x80u) {  // walls, computed by the wall tiles for this step
      fx += A.fmx[i]; fy += A.fmy[i]; fz += A.fmz[i];
      tx += A.tmx[i]; ty += A.tmy[i]; tz += A.tmz[i];
    }
  } else {
    fx = A.fx[i]; fy = A.fy[i]; fz = A.fz[i];
    tx = A.tx[i]; ty = A.ty[i]; tz = A.tz[i];
  }
  double dtfm = 0.0, dtir = 0.0;
  float4 hf = make_float4(0.f, 0.f, 0.f, 0.f);
  if (final || initial) {
    dtfm = A.dtfm[i];
    dtir = A.dtir[i];
  }
  if (initial) {
    hf = s.xhf[i];
    hf.w = s.xf[i].w;
  }
  particle_finish(s, i, gather, final, initial, fx, fy, fz, tx, ty, tz, v, om, xv, dtfm, dtir, hf, moved, bad);
}

// What one lane of k_steps keeps of its atom's list between two builds (one
// atom per thread and launch): the row, the partner list's first entries.
constexpr int kCachedRev = 8;
template <int T>
struct ListCache {
  int pb[T];
  int cnt[T];  // own entries | partner entries << 8 | near a wall << 16; -1: too many for the cache
  int rev[kCachedRev][T];
};

template <int T>
__device__ __forceinline__ void list_cache_load(const Sys &s, ListCache<T> &lc, int i, bool valid) {
  const PairArrays &L = s.pairs[0];
  const int tid = threadIdx.x;
  int cnt = 0, pb = 0;
  if (valid) {
    pb = L.row[i];
    const int rb = L.rev_start[i], no = row_end(s, L, i) - pb, nr = rev_end(s, L, i) - rb;
    cnt = no <= kCachedRev && nr <= kCachedRev ? (no | nr << 8 | (s.atoms[0].wbits[i] & 0x80u ? 1 << 16 : 0)) : -1;
    for (int k = 0; k < kCachedRev; k++) lc.rev[k][tid] = cnt >= 0 && k < nr ? L.rev[rb + k] : -1;
  }
  lc.pb[tid] = pb;
  lc.cnt[tid] = cnt;
}

// particle_tile for k_steps.  With few warps per SM the shared-memory round
// trips of particle_tile cost more than the additions that they save, and each load that waits for another costs a trip to L2 (the
// barriers leave nothing in L1): the list's indices come from the cache, what
// does not depend on them is loaded together, and a contact's record is loaded
// while the one before it is added.  Same sums in the same order.
template <int T>
__device__ __forceinline__ void particle_warp(const Sys &s, const ListCache<T> *lc, int i, bool valid, bool gather,
                                              bool final, bool initial, bool &moved, bool &bad) {
  if (!valid) return;
  const AtomArrays &A = s.atoms[0];
  const PairArrays &L = s.pairs[0];
  const int tid = threadIdx.x;
  double f[6] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0}, fm[6] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
  const int cnt = lc ? lc->cnt[tid] : -1;
  uint8_t ao[kCachedRev], ar[kCachedRev];
  if (gather && cnt >= 0) {
    const int pb = lc->pb[tid], no = cnt & 0xff, nr = (cnt >> 8) & 0xff;
#pragma unroll
    for (int k = 0; k < kCachedRev; k++) {
      ao[k] = k < no ? s.active[pb + k] : 0;
      ar[k] = k < nr ? s.active[lc->rev[k][tid]] : 0;
    }
  }
  double v[3] = {A.vx[i], A.vy[i], A.vz[i]}, om[3] = {A.wx[i], A.wy[i], A.wz[i]};
  double xv[3] = {A.x[i], A.y[i], A.z[i]};
  const double dtfm = A.dtfm[i], dtir = A.dtir[i];
  float4 hf = s.xhf[i];
  hf.w = s.xf[i].w;
  if (gather) {
    const double m = s.gravity_on ? A.m[i] : 0.0;
    const bool wall = cnt >= 0 ? (cnt >> 16) & 1 : (A.wbits[i] & 0x80u) != 0;
    if (wall) {
      fm[0] = A.fmx[i]; fm[1] = A.fmy[i]; fm[2] = A.fmz[i];
      fm[3] = A.tmx[i]; fm[4] = A.tmy[i]; fm[5] = A.tmz[i];
    }
    if (s.gravity_on) gravity_force(s, m, f[0], f[1], f[2]);
    if (cnt >= 0) {
      const int pb = lc->pb[tid];
      unsigned act = 0u;  // active entries, own then partner's
#pragma unroll
      for (int k = 0; k < kCachedRev; k++) act |= (ao[k] ? 1u : 0u) << k | (ar[k] ? 1u : 0u) << (kCachedRev + k);
      double r[6];
      unsigned long long sg = 0ull;
      auto load = [&](double *d, unsigned long long &sign) {
        const int b = __ffs(act) - 1;
        act &= act - 1u;
        const bool own = b < kCachedRev;
        const double *q = s.res + (size_t)kResStride * (own ? pb + b : lc->rev[b - kCachedRev][tid]);
        sign = own ? 0ull : 0x8000000000000000ull;
        for (int k = 0; k < 3; k++) {
          d[k] = q[k];
          d[3 + k] = q[(own ? 3 : 6) + k];
        }
      };
      int left = __popc(act);
      if (left) load(r, sg);
      while (left--) {
        double n[6] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
        unsigned long long sn = 0ull;
        if (left) load(n, sn);
        for (int k = 0; k < 3; k++) {
          f[k] += __longlong_as_double(__double_as_longlong(r[k]) ^ sg);
          f[3 + k] += r[3 + k];
        }
        sg = sn;
        for (int k = 0; k < 6; k++) r[k] = n[k];
      }
    } else {
      int pb, rb;
      unsigned mo, mr;
      if (gather_masks<4>(s, L, i, pb, rb, mo, mr)) gather_sum(s, L, pb, rb, mo, mr, f[0], f[1], f[2], f[3], f[4], f[5]);
      else gather_long(s, L, i, f[0], f[1], f[2], f[3], f[4], f[5]);
    }
    if (wall)
      for (int k = 0; k < 6; k++) f[k] += fm[k];
  } else {
    f[0] = A.fx[i]; f[1] = A.fy[i]; f[2] = A.fz[i];
    f[3] = A.tx[i]; f[4] = A.ty[i]; f[5] = A.tz[i];
  }
  particle_finish(s, i, gather, final, initial, f[0], f[1], f[2], f[3], f[4], f[5], v, om, xv, dtfm, dtir, hf, moved,
                  bad);
}

}  // namespace gb300

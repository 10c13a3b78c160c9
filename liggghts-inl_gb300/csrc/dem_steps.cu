// The fused step kernel: whole timesteps in one cooperative launch.
//
// A step of a small or middle-sized system is a chain of latencies: as
// separate graph nodes (per-atom kernel, rebuild decision, IF node, pair and
// wall kernels side by side, WHILE iteration) about 14 us of every step pass
// between the kernels, and each kernel fetches its parameters, its code and
// its atoms anew.  k_steps keeps one block resident on every SM (fewer blocks
// for systems of fewer warps) and runs step after step, with a grid barrier
// where a kernel boundary was:
//
//   A  per atom: gather, gravity, wall totals, nve/sphere, displacement test
//      (particle_warp); moving meshes advance on the grid's last warps
//   -- barrier; every block takes the same rebuild decision; a rebuild ends
//      the launch (the graph's IF node rebuilds, the WHILE node comes back,
//      and the launch resumes with B)
//   B  by warps, the tests of the block's list tiles (pf_test, band_test), then
//      its wall tiles (wall_tile) and the laws of the entries that passed
//   -- barrier; after a call's last step, and every 2,048, the launch ends
//
// The tiles are those of the separate kernels, and every atom's and entry's
// result goes to its own slot, so the results are the same bits.
//
// The blocks wait for one another, so the launch is cooperative (the runtime
// launches it only when all its blocks are resident together); every wait has
// an iteration limit, after which the block sets kStatTimeout and returns.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdlib>
#include <mutex>

#include "barrier_count.cuh"
#include "dem_kernels.h"
#include "step_device.cuh"

namespace gb300 {

constexpr int kStepThreads = 512;
// polls of one grid barrier before it gives up (each is a round trip to L2,
// 0.5 us and more: several seconds, where a phase takes milliseconds at
// most); LIGGGHTS_GB300_BARRIER_POLLS sets it (test of the give-up path)
constexpr int kBarrierPolls = 1 << 23;

// pair force path: entries need no work unless touching; contact distance
// factor above 1; cohesion bond/nonlinear
enum { kPathTouch = 0, kPathBand = 1, kPathBond = 2 };

// The block's queue of entries that need the FP64 laws (band and bond: with
// their exact test's delta and rsq), filled from up to kQueue / 32 tiles.
template <int PATH>
struct StepQueue {
  static constexpr int kQueue = 1024;
  int p[kQueue];
  double d[4][kQueue];
};
template <>
struct StepQueue<kPathTouch> {
  static constexpr int kQueue = 2048;
  int p[kQueue], i[kQueue], j[kQueue];
  uint8_t code[kQueue];
};

template <int PATH>
struct StepShared {
  StepQueue<PATH> queue;
  ListCache<kStepThreads> list;
};

struct StepFlags {  // what thread 0 read behind the barrier
  int ok, moved, mesh_moved;
  unsigned long long seen;
};

// Grid barrier: every block adds to one 64-bit count and polls it (one trip to
// L2 to arrive, one to see the last arrival: 2.3k cycles with 152 blocks; a
// separate release flag took 3.2k, a flag per block that all blocks poll
// 5.8k).  MOVEMENT: the barrier behind phase A, whose arrivals bring the
// movement flags (see barrier_count.cuh).  `seen` is the same in every block.
// False when a wait gave up.
template <bool MOVEMENT>
__device__ __forceinline__ bool grid_barrier(Ctrl *c, int blocks, int limit, unsigned long long &seen, int flags,
                                             StepFlags &fl) {
  if (MOVEMENT) flags = __syncthreads_or(flags & 1) | (__syncthreads_or(flags & 2) ? 2 : 0);
  else __syncthreads();
  if (threadIdx.x == 0) {
    const unsigned long long add = barrier_arrival(MOVEMENT ? flags : 0);
    unsigned long long now;
    int ok = 1, polls = 0;
    asm volatile("red.release.gpu.global.add.u64 [%0], %1;" ::"l"(&c->bar), "l"(add) : "memory");
    for (;;) {
      asm volatile("ld.acquire.gpu.global.u64 %0, [%1];" : "=l"(now) : "l"(&c->bar) : "memory");
      if (barrier_full(now, seen, blocks)) break;
      if (++polls >= limit || *(volatile int *)&c->bar_abort) {
        *(volatile int *)&c->bar_abort = 1;
        ok = 0;
        break;
      }
    }
    const BarrierPass p = barrier_pass(now, seen, blocks, MOVEMENT);
    fl.ok = ok;
    fl.moved = p.moved;
    fl.mesh_moved = p.mesh_moved;
    fl.seen = p.seen;
  }
  __syncthreads();
  seen = fl.seen;
  return fl.ok != 0;
}

__device__ __forceinline__ void queue_put(StepQueue<kPathTouch> &q, int at, const double *, int i, int j, int code) {
  q.i[at] = i;
  q.j[at] = j;
  q.code[at] = (uint8_t)code;
}
template <int PATH>
__device__ __forceinline__ void queue_put(StepQueue<PATH> &q, int at, const double *d, int, int, int) {
  for (int k = 0; k < 4; k++) q.d[k][at] = d[k];
}
template <int NORMAL, bool ROLL>
__device__ __forceinline__ void queue_entry(const Sys &s, const StepQueue<kPathTouch> &q, int e, long long) {
  pair_entry<NORMAL, ROLL>(s, q.p[e], q.i[e], q.j[e], q.code[e], 1);
}
// How a launch of k_steps is driven: by a graph's conditionals (in_graph), or
// from the host; n >= 0: steps and phase to start with, else Ctrl's.
struct StepCall {
  int in_graph, n, phase;
  cudaGraphConditionalHandle hreb, hloop;
};

// the launch ended with a rebuild due (reb), or done
__device__ __forceinline__ void step_conditionals(const StepCall &call, int reb) {
  if (!call.in_graph) return;
  cudaGraphSetConditional(call.hreb, reb ? 1u : 0u);
  cudaGraphSetConditional(call.hloop, reb ? 1u : 0u);
}

template <int NORMAL, bool ROLL, int PATH>
__device__ __forceinline__ void queue_entry(const Sys &s, const StepQueue<PATH> &q, int e, long long ts) {
  band_entry<NORMAL, ROLL, PATH == kPathBond>(s, q.p[e], q.d[0][e], q.d[1][e], q.d[2][e], q.d[3][e], 1, ts);
}

template <int NORMAL, bool ROLL, int PATH>
__global__ void __launch_bounds__(kStepThreads, 1)
    k_steps(const __grid_constant__ Sys s, int wall_cap, int limit, StepCall call) {
  constexpr int kStepWarps = kStepThreads / 32;
  extern __shared__ __align__(16) unsigned char dyn[];
  __shared__ StepFlags fl;
  __shared__ int next_tile, next_item, nqueue;
  Ctrl *c = s.ctrl;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, G = gridDim.x;
  if (c->halt) {
    if (blockIdx.x == 0 && tid == 0) step_conditionals(call, 0);
    return;
  }
  StepShared<PATH> &sh = *reinterpret_cast<StepShared<PATH> *>(dyn);
  WallQueue wq;  // this warp's wall queue, behind the union
  {
    unsigned char *w = dyn + ((sizeof(StepShared<PATH>) + 15) & ~(size_t)15);
    wq.res = reinterpret_cast<double *>(w) + (size_t)warp * wall_cap * kWallRes;
    wq.st = reinterpret_cast<int *>(w + (size_t)kStepWarps * wall_cap * kWallRes * 8) + warp * wall_cap;
    wq.qa = w + (size_t)kStepWarps * wall_cap * (kWallRes * 8 + 4) + (size_t)warp * 2 * wall_cap;
    wq.qq = wq.qa + wall_cap;
  }
  // the launch's constants, and the decision's state: the same in every block
  const int n = c->n, np = c->np, nl = c->nmlist;
  int left = call.n >= 0 ? call.n : c->loop_left, phase = call.n >= 0 ? call.phase : c->step_phase, turn = c->turn;
  int ago = c->ago, force = c->force_rebuild;
  long long ts = c->ntimestep;
  int reb = 0;
  unsigned long long seen = 0;  // the barrier's count behind the last one
  bool ok = true, moved = false, bad = false, meshbad = false;
  // a warp's tiles of 32 atoms: neighbouring tiles on different SMs, so that
  // small systems reach every SM
  const int warp_id = warp * G + blockIdx.x, atom_tiles = (n + 31) / 32;
  const bool cached = atom_tiles <= G * kStepWarps;
  if (cached) list_cache_load(s, sh.list, warp_id * 32 + lane, warp_id < atom_tiles && warp_id * 32 + lane < n);
  const int ntiles = (np + 31) / 32;
  const int chunk = max(1, min(8, (ntiles + G - 1) / G));
  const int my_tiles = (ntiles + G * chunk - 1) / (G * chunk) * chunk;  // some may lie past the list's end
  const double cdm = s.cdf * s.cdf;
  const bool walls = s.nplanes > 0 || s.nmeshes > 0;
  for (;;) {
    if (phase != kStepForces) {
      // ---- A
      const bool last = left == 0;
      const bool gather = phase != kStepFirst;
      moved = false;
      for (int t = warp_id; t < atom_tiles; t += G * kStepWarps)
        particle_warp(s, cached ? &sh.list : nullptr, t * 32 + lane, t * 32 + lane < n, gather, gather, !last, moved, bad);
      if (last) break;
      bool mm = false;
      for (int k = 0; k < s.nmeshes; k++) {
        const MeshDev &M = s.meshes[k];
        if (!M.moving) continue;
        const int w = G * kStepWarps - 1 - warp_id;
        for (int t0 = 2 * w; t0 < M.ntri; t0 += 2 * G * kStepWarps) mm |= mesh_move_part(s, M, t0 + (lane >> 4), lane & 15);
      }
      if (!(ok = grid_barrier<true>(c, G, limit, seen, (moved ? 1 : 0) | (mm ? 2 : 0), fl))) break;
      // Neighbor::decide (see decide_rebuild)
      ts++;
      if (force) {
        reb = 1;
      } else {
        ago++;
        reb = (ago >= s.neigh_delay && ago % s.neigh_every == 0) ? (s.neigh_check ? fl.moved : 1) : 0;
      }
      force = reb ? 0 : fl.mesh_moved;
      if (reb) break;
    }
    phase = kStepGather;
    const bool may_create = band_may_create<PATH == kPathBond>(s, 1, ts);
    // ---- B: the block's tiles of the list, then its wall tiles and batches of 32 queued entries
    StepQueue<PATH> &q = sh.queue;
    const int nwt = walls ? (max(0, nl - (int)blockIdx.x * kWallTile) + G * kWallTile - 1) / (G * kWallTile) : 0;
    for (int t0 = 0; t0 == 0 || t0 < my_tiles; t0 += StepQueue<PATH>::kQueue / 32) {
      if (tid == 0) next_tile = next_item = nqueue = 0;
      __syncthreads();
      const int nt = min(my_tiles - t0, StepQueue<PATH>::kQueue / 32);
      for (;;) {
        int u = 0;
        if (lane == 0) u = atomicAdd(&next_tile, 1);
        u = __shfl_sync(0xffffffffu, u, 0);
        if (u >= nt) break;
        u += t0;
        const long tile = (long)(u / chunk) * G * chunk + (long)blockIdx.x * chunk + u % chunk;
        if (tile >= ntiles) continue;
        const int p = (int)tile * 32 + lane;
        double d[4] = {0., 0., 0., 0.};
        bool want;
        int ti = 0, tj = 0, code = 0;
        if (PATH == kPathTouch) want = pf_test(s, np, p, ti, tj, code);
        else want = band_test<PATH == kPathBond>(s, np, p, cdm, may_create, d[0], d[1], d[2], d[3]);
        const unsigned m = __ballot_sync(0xffffffffu, want);
        int at = 0;
        if (lane == 0 && m) at = atomicAdd(&nqueue, __popc(m));
        at = __shfl_sync(0xffffffffu, at, 0) + __popc(m & ((1u << lane) - 1u));
        if (want) {
          q.p[at] = p;
          queue_put(q, at, d, ti, tj, code);
        }
      }
      __syncthreads();
      // wall tiles first: they are the longest items
      const int nw = t0 == 0 ? nwt : 0, nq = nqueue, items = nw + (nq + 31) / 32;
      for (;;) {
        int u = 0;
        if (lane == 0) u = atomicAdd(&next_item, 1);
        u = __shfl_sync(0xffffffffu, u, 0);
        if (u >= items) break;
        if (u < nw) {
          wall_tile<NORMAL>(s, s.atoms[0], (blockIdx.x + G * u) * kWallTile, nl, 1, wall_cap, wq, meshbad);
        } else {
          const int e = (u - nw) * 32 + lane;
          if (e < nq) queue_entry<NORMAL, ROLL>(s, q, e, ts);
        }
      }
      __syncthreads();
    }
    if (!(ok = grid_barrier<false>(c, G, limit, seen, 0, fl))) break;
    left--;
    if (call.in_graph && left > 0 && --turn <= 0) break;
  }
  if (__any_sync(0xffffffffu, bad) && lane == 0) atomicExch(&c->status, kStatNan);
  if (__any_sync(0xffffffffu, meshbad) && lane == 0) atomicExch(&c->status, kStatMeshSlots);
  __syncthreads();
  if (tid != 0) return;
  if (!ok) {  // a wait gave up: the host reads the status (the counts stay as they are until the next upload)
    atomicExch(&c->status, kStatTimeout);
    c->halt = 1;
    step_conditionals(call, 0);
    return;
  }
  // the last block to leave: every other one has read and passed everything
  __threadfence();
  if (atomicAdd(&c->bar_exit, 1) != G - 1) return;
  c->bar = 0;
  c->bar_exit = 0;
  c->ntimestep = ts;
  c->ago = ago;
  c->force_rebuild = force;
  c->rebuild = reb;
  c->moved = 0;
  c->mesh_moved = 0;
  c->loop_left = left;
  c->turn = turn;
  c->step_phase = reb ? kStepForces : (left > 0 ? kStepGather : kStepDone);
  step_conditionals(call, reb);
}

namespace {

typedef void (*StepKernel)(Sys, int, int, StepCall);

StepKernel step_kernel(const Sys &s, size_t *shared) {
  const int path = s.bond ? kPathBond : (s.cdf == 1.0 ? kPathTouch : kPathBand);
#define STEP_PICK(P)                                                                                              \
  if (path == P) {                                                                                                \
    *shared = (sizeof(StepShared<P>) + 15) & ~(size_t)15;                                                      \
    if (s.normal == kHertz)                                                                                       \
      return s.rolling ? (StepKernel)k_steps<kHertz, true, P> : (StepKernel)k_steps<kHertz, false, P>;      \
    return s.rolling ? (StepKernel)k_steps<kHooke, true, P> : (StepKernel)k_steps<kHooke, false, P>;        \
  }
  STEP_PICK(kPathTouch)
  STEP_PICK(kPathBand)
  STEP_PICK(kPathBond)
#undef STEP_PICK
  return nullptr;
}

}  // namespace

// Up to 330,000 list entries (about 115,000 spheres of a loose packing, 57,000
// of a dense one), with mesh walls and no bonds up to 160,000.  Us per step,
// fused against separate kernels, on one GB300:
//   loose column   80k spheres 39 / 44   100k 45 / 48   120k 53 / 52   200k 74 / 73
//   dense bed      15k 46 / 50           35k 66 / 65    50k 81 / 81    100k 150 / 127
//   hooke          60k 24 / 32           99k 37 / 37    200k 65 / 58
//   bonded fibres  30k 50 / 73           60k 93 / 113
//   hopper mesh    20k 35 / 42           60k 42 / 42    80k 53 / 45    200k 105 / 80
//   mixer mesh     40k 27 / 35           80k 38 / 39
// Above it the separate kernels win: each is compiled for its own registers,
// with twice the warps per SM to hide loads and fill the FP64 pipes, and the
// nodes' latency is small beside them; a mesh's wall kernel runs beside the pair
// kernel, while here its tiles hold up the blocks that have them.  (With bonds
// the pair law is the longer one.)  Ensembles decide per system
// (decide_rebuild) and keep the separate kernels.  Asked at every call.
// LIGGGHTS_GB300_FUSED_STEPS=0|1: never, always (tests).
bool fused_steps(const Sys &s, const LaunchCfg &lc) {
  if (s.nsys || !lc.coop) return false;
  if (const char *e = getenv("LIGGGHTS_GB300_FUSED_STEPS")) return atoi(e) != 0;
  return lc.np <= (s.nmeshes > 0 && !s.bond ? 160000 : 330000);
}

// one block per SM; fewer for systems of fewer warps
int steps_grid(const Sys &s, const LaunchCfg &lc) { return std::max(1, std::min((s.nmax + 31) / 32, lc.sms)); }

static int barrier_polls() {
  const char *polls = getenv("LIGGGHTS_GB300_BARRIER_POLLS");
  return polls ? std::max(1, atoi(polls)) : kBarrierPolls;
}

int step_loop_key(const LaunchCfg &lc) { return lc.fused ? barrier_polls() : 0; }

// Us per step of 1, 2 and 4 handles in as many threads, 50 steps a call: the
// separate kernels; k_steps in turns; by DeviceCall's rule:
//   2,000 spheres   21  23  24    16  16  30    16  16  24
//   10,000          22  24  27    18  34  68    18  26  28
//   50,000          31  40  56    26  50  99    25  40  57
//   100,000         42  59 104    45  89 177    44  60 105
namespace {
struct DeviceLoad {
  std::mutex m;
  int calls = 0, fused = 0, blocks = 0;  // in flight; those that run k_steps, and their blocks
};
constexpr int kMaxDevices = 64;
DeviceLoad &device_load(int device) {
  static DeviceLoad loads[kMaxDevices];
  return loads[device >= 0 ? device % kMaxDevices : 0];
}
}  // namespace

DeviceCall::DeviceCall(int device) : device_(device) {
  DeviceLoad &d = device_load(device_);
  std::lock_guard<std::mutex> lock(d.m);
  d.calls++;
}

DeviceCall::~DeviceCall() {
  DeviceLoad &d = device_load(device_);
  std::lock_guard<std::mutex> lock(d.m);
  give_back();
  d.calls--;
}

void DeviceCall::give_back() {
  DeviceLoad &d = device_load(device_);
  d.fused -= blocks_ > 0 ? 1 : 0;
  d.blocks -= blocks_;
  blocks_ = 0;
}

bool DeviceCall::ask(int blocks, int room) {
  DeviceLoad &d = device_load(device_);
  std::lock_guard<std::mutex> lock(d.m);
  give_back();
  // (this call is one of those that run no k_steps)
  if (blocks <= 0 || d.calls - d.fused > 1 || d.blocks + blocks > room) return false;
  blocks_ = blocks;
  d.fused++;
  d.blocks += blocks;
  return true;
}

bool coop_refused(int what) {
  const char *e = getenv("LIGGGHTS_GB300_COOP_REFUSE");
  return e && (atoi(e) & what);
}

namespace {

struct StepLaunch {
  StepKernel kernel = nullptr;
  int grid = 0, wall_cap = 0;
  size_t shared = 0;
};

cudaError_t step_launch(const Sys &s, const LaunchCfg &lc, StepLaunch *l) {
  size_t shared = 0;
  l->kernel = step_kernel(s, &shared);
  // wall queues as long as asked for, or as fit (a fuller tile takes the
  // sequential path, with the same result; 1 KB is for the static part)
  const size_t queue = (size_t)(kStepThreads / 32) * kWallTile * kWallQ;  // per entry of a tile's atom
  const int most = (int)std::min<size_t>(wall_cap_per_atom(), (226 * 1024 - shared) / queue);
  l->wall_cap = s.nmeshes > 0 ? most * kWallTile : 0;
  l->shared = shared + (size_t)(kStepThreads / 32) * kWallQ * l->wall_cap;
  l->grid = steps_grid(s, lc);
  // the limit belongs to the function, not to the launch: the same for every
  // system, so that threads that step different ones do not undercut each other
  return cudaFuncSetAttribute((const void *)l->kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                              (int)(shared + queue * most));
}

}  // namespace

bool steps_resident(const Sys &s, const LaunchCfg &lc) {
  if (coop_refused(kCoopGrid)) return false;
  StepLaunch l;
  int device = 0, coop = 0, blocks = 0;
  const bool ok = cudaGetDevice(&device) == cudaSuccess &&
                  cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, device) == cudaSuccess &&
                  step_launch(s, lc, &l) == cudaSuccess &&
                  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&blocks, (const void *)l.kernel, kStepThreads,
                                                                l.shared) == cudaSuccess;
  if (!ok) cudaGetLastError();
  return ok && coop && (long)blocks * lc.sms >= l.grid;
}

static cudaError_t launch_call(const Sys &s, const LaunchCfg &lc, const StepCall &call, cudaStream_t st) {
  if (coop_refused(call.in_graph ? kCoopInGraph : (call.n < 0 ? kCoopResume : kCoopDirect)))
    return cudaErrorCooperativeLaunchTooLarge;
  StepLaunch l;
  cudaError_t e = step_launch(s, lc, &l);
  if (e != cudaSuccess) return e;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(l.grid);
  cfg.blockDim = dim3(kStepThreads);
  cfg.dynamicSmemBytes = l.shared;
  cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeCooperative;
  attr[0].val.cooperative = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, l.kernel, s, l.wall_cap, barrier_polls(), call);
}

cudaError_t launch_steps(const Sys &s, const LaunchCfg &lc, cudaGraphConditionalHandle hreb,
                         cudaGraphConditionalHandle hloop, cudaStream_t st) {
  return launch_call(s, lc, StepCall{1, -1, 0, hreb, hloop}, st);
}

cudaError_t launch_steps_direct(const Sys &s, const LaunchCfg &lc, int n, int phase, cudaStream_t st) {
  return launch_call(s, lc, StepCall{0, n, phase, 0, 0}, st);
}

}  // namespace gb300

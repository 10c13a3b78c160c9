// Host-side launchers of the sphere-DEM kernels (dem_kernels.cu).
#pragma once
#include <cuda_runtime.h>

#include <mutex>

#include "dem_device.cuh"

namespace gb300 {

struct LaunchCfg {
  int max_grid;              // grid-stride kernels never launch more blocks of 256 than this
  int particle_threads = 256;  // threads per block of the per-particle kernel (64, 128, 256)
  int sms = 152;               // multiprocessors of the device
  int np = 0;                  // list entries at the last build (what fused_steps goes by)
  bool coop = true;            // k_steps' grid can be resident, and no launch of it was refused
  bool fused = false;          // the call runs in k_steps (dem_step's choice by fused_steps)
};

enum {
  kModeInitial = 0,             // nve/sphere initial_integrate only (first step of a call)
  kModeGather = 1,              // sum forces only (setup)
  kModeGatherFinal = 2,         // sum forces + final_integrate (last step of a call)
  kModeGatherFinalInitial = 3,  // sum forces + final(n) + initial(n+1) (steady state)
  kModeStart = 4,               // first step of a graph launch: kModeInitial or kModeGatherFinalInitial, by
                                // Ctrl::step_phase
};

struct InsertStage {  // new atoms, device arrays: x, v, w [3k], the rest [k]
  const double *x, *v, *w, *r, *m, *dtfm, *dtir;
  const int *type, *tag;
};
int launch_insert_stage(const Sys &s, const InsertStage &in, int first, int k, int lidx0, cudaStream_t st);
// Atom transfer between the caller's per-atom AoS arrays (atom->x[i][d] as
// x[3*i+d]) and the device's SoA arrays.  The pointers are either the
// caller's host arrays (read and written by the kernels themselves where the
// device reaches pageable host memory through the host's page tables) or
// device staging copies of them.
struct AtomsIn {
  const int *tag, *type;
  const double *x, *v, *w, *r, *m;
};
struct AtomsOut {  // null members are skipped
  int *tag, *type;
  double *x, *v, *w, *f, *t, *r, *m;
};
struct UploadCheck {         // filled by k_upload_atoms (zero-initialise rmax, counts; rmin = ~0)
  unsigned long long rmin;   // bit pattern of the smallest positive radius
  unsigned long long rmax;   // bit pattern of the largest radius
  int bad_type;              // atoms with a type outside 1..ntypes
  int bad_value;             // atoms with radius or rmass not finite and > 0
  int nonfinite;             // atoms with a non-finite position, velocity or angular velocity
  int pad;
};
// SoA state of the first n atoms (buffer 0) from `in`, the nve/sphere
// per-atom constants dtf/m and dtfrotate/(r^2 m), caller-order indices, and
// cleared forces, holds, wall histories and mesh slots; `chk` collects the
// checks and the radius range.
int launch_upload_atoms(const Sys &s, const AtomsIn &in, int n, double dtf, double dtfrotate, UploadCheck *chk,
                        cudaStream_t st);
int launch_download_atoms(const Sys &s, const AtomsOut &out, int n, cudaStream_t st);
int launch_insert_commit(const Sys &s, int k, cudaStream_t st);
int launch_diagnostics(const Sys &s, const LaunchCfg &lc, const double lo[3], const double hi[3], double *part_atoms,
                       double *part_walls, unsigned long long *contacts, int nblocks, cudaStream_t st);
// exclusive prefix sum of len ints (len <= 4096*4096 - 1); tmp holds
// (len+4095)/4096 + 1 ints; gate 0: always; 1: only while the system
// rebuilds; 2: not in an ensemble rebuild that keeps other systems in place
int scan_exclusive(const Sys &s, const int *in, int *out, int len, int *tmp, int gate,
                   cudaStream_t st);
int launch_decide(const Sys &s, cudaStream_t st);
int launch_set_rebuild(const Sys &s, int v, cudaStream_t st);
// stage 0: full rebuild; stage 1: resume after a pair-capacity overflow;
// stage 2: resume after a mesh slot or registration overflow
int launch_rebuild(const Sys &s, const LaunchCfg &lc, cudaStream_t st, int stage);
int launch_pair(const Sys &s, const LaunchCfg &lc, int shearupdate, cudaStream_t st, int gate = 0);
int launch_particle(const Sys &s, const LaunchCfg &lc, int mode, cudaStream_t st);
// the graph's next launch: n steps from `phase` (k_steps returns after some 2,000, see Ctrl::turn)
int launch_set_loop(const Sys &s, int n, int phase, cudaStream_t st);
// wall (plane and mesh) forces of the current state, before the particle
// kernel that gathers the step's forces; none without walls
int launch_wall_force(const Sys &s, const LaunchCfg &lc, int shearupdate, cudaStream_t st, int gate = 0);
// the wall contacts' constants anew (the pair parameters changed since the build)
int launch_wall_consts(const Sys &s, const LaunchCfg &lc, cudaStream_t st);
// fix move/mesh: moves the moving meshes by one step (after the drift)
int launch_mesh_move(const Sys &s, const LaunchCfg &lc, cudaStream_t st, int gate = 0);
// queue entries of the wall kernel per tile atom (LIGGGHTS_GB300_WALL_CAP)
int wall_cap_per_atom();
// Whether a system runs its steps in k_steps (dem_steps.cu) rather than as
// separate kernels, its grid, and its launch inside the step graph.
bool fused_steps(const Sys &s, const LaunchCfg &lc);
int steps_grid(const Sys &s, const LaunchCfg &lc);
// whether all blocks of k_steps can be resident together, which its cooperative launch needs
bool steps_resident(const Sys &s, const LaunchCfg &lc);

// A call that keeps the device busy, for as long as it lives.  k_steps holds
// its SMs until its launch ends, so calls from several threads would take turns
// where the separate kernels overlap: it is granted only beside other k_steps,
// and only up to `room` blocks of all together (the SMs: all are resident).
class DeviceCall {
 public:
  explicit DeviceCall(int device);
  ~DeviceCall();
  DeviceCall(const DeviceCall &) = delete;
  DeviceCall &operator=(const DeviceCall &) = delete;
  bool ask(int blocks, int room);  // k_steps with so many blocks (0: none); gives back what was granted before

 private:
  void give_back();
  int device_, blocks_ = 0;  // blocks_: granted
};
// Refusals as CUDA gives them (under MPS, say), for tests:
// LIGGGHTS_GB300_COOP_REFUSE adds up what is refused.
enum { kCoopGrid = 1, kCoopInGraph = 2, kCoopDirect = 4, kCoopResume = 8, kCoopGraphLaunch = 16 };
bool coop_refused(int what);
// what else the step graph depends on: 0 for the separate kernels, else k_steps' limit
int step_loop_key(const LaunchCfg &lc);
cudaError_t launch_steps(const Sys &s, const LaunchCfg &lc, cudaGraphConditionalHandle hreb,
                         cudaGraphConditionalHandle hloop, cudaStream_t st);
// the same from the host, without a graph: n steps from `phase`, or (n < 0) on from where Ctrl says
cudaError_t launch_steps_direct(const Sys &s, const LaunchCfg &lc, int n, int phase, cudaStream_t st);
// Executable graph of the step loop (WHILE node over steps, IF node around
// the rebuild); see dem_kernels.cu.  launch_set_loop sets what it runs.
struct StepCounts {  // kernels of a graph launch: per call, per further step, per rebuild
  int call = 0, step = 0, rebuild = 0;
};
cudaError_t build_step_graph(const Sys &s, const LaunchCfg &lc, cudaStream_t st, cudaStream_t st2,
                             cudaGraphExec_t *exec, StepCounts *counts);

}  // namespace gb300

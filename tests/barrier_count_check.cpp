// Host build of the arithmetic of the fused step kernel's grid barrier
// (liggghts-inl_gb300/csrc/barrier_count.cuh).  Every block runs steps of two
// barriers, behind the movement (with its flags) and behind the forces
// (without); a block's next action is either to arrive or to poll a full count,
// and check_barrier walks every interleaving of all blocks.  Built and called by
// tests/test_barrier_count.py.
#include <stdint.h>

#include <set>
#include <vector>

#include "barrier_count.cuh"

using namespace gb300;

namespace {

struct Block {
  int at = 0;  // barriers passed
  bool arrived = false;
  unsigned long long seen = 0;
  unsigned taken = 0;  // flags taken so far, two bits per step
};

struct Walk {
  int nb, steps;
  const int *flags;  // [step * nb + block]
  unsigned want;     // the flags that every block has to take
  long states = 0, wrong = 0;
  std::set<std::vector<unsigned long long>> done;

  void go(unsigned long long now, unsigned long long start, const std::vector<Block> &b) {
    std::vector<unsigned long long> key{now};
    for (const Block &k : b) {
      key.push_back((unsigned long long)k.at * 2 + k.arrived);
      key.push_back(k.seen);
      key.push_back(k.taken);
    }
    if (!done.insert(key).second) return;
    states++;
    bool any = false, end = true;
    for (int k = 0; k < nb; k++) {
      if (b[k].at == 2 * steps) continue;
      end = false;
      const bool movement = b[k].at % 2 == 0;
      const int step = b[k].at / 2;
      std::vector<Block> c = b;
      if (!b[k].arrived) {
        c[k].arrived = true;
        any = true;
        go(now + barrier_arrival(movement ? flags[step * nb + k] : 0), start, c);
      } else if (barrier_full(now, b[k].seen, nb)) {
        const BarrierPass p = barrier_pass(now, b[k].seen, nb, movement);
        c[k].arrived = false;
        c[k].at++;
        c[k].seen = p.seen;
        if (movement) c[k].taken |= (unsigned)((p.moved ? 1 : 0) | (p.mesh_moved ? 2 : 0)) << (2 * step);
        else if (p.moved || p.mesh_moved) wrong++;
        any = true;
        go(now, start, c);
      }
    }
    if (end) {  // every block has taken every flag, each once, and the whole count
      for (int k = 0; k < nb; k++) wrong += b[k].taken != want || b[k].seen != now;
    } else if (!any) {
      wrong++;  // no block can go on
    }
  }
};

}  // namespace

// Every interleaving of nb blocks over `steps` steps, for every combination of
// movement flags; the count starts at `start`.  Returns the number of wrong
// states (flags lost or taken twice, counts that differ, no way on).
extern "C" long check_barrier(int nb, int steps, unsigned long long start, long *states) {
  long wrong = 0;
  *states = 0;
  std::vector<int> flags(nb * steps);
  for (long combo = 0; combo < 1l << (2 * nb * steps); combo++) {
    for (int q = 0; q < nb * steps; q++) flags[q] = (combo >> (2 * q)) & 3;
    Walk w{nb, steps, flags.data(), 0};
    for (int q = 0; q < nb * steps; q++) w.want |= (unsigned)flags[q] << (2 * (q / nb));
    std::vector<Block> b(nb);
    for (Block &k : b) k.seen = start;
    w.go(start, start, b);
    wrong += w.wrong;
    *states += w.states;
  }
  return wrong;
}

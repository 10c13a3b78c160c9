// The arithmetic of k_steps' grid barrier (dem_steps.cu), for the device and
// for the host.
//
// All barriers of a launch share one 64-bit count.  A block arrives by adding 1;
// at the barrier behind the movement (phase A) a block with an atom that moved
// more than skin/2 adds 2^32 as well, one with such a mesh node 2^48, so that
// the wait also brings the movement flags.  `seen` is what a block has taken of
// the count at the barriers that it has passed; the rest is what has arrived
// since.
//
// A block that polls late may find the arrivals of the next barrier in the
// count already, never those of the one after that (no block passes the next
// barrier before this one has arrived there).  So a barrier takes exactly
// `blocks` arrivals, and the flags only where they belong:
//   behind the movement every flag of the step has come with its arrival, and
//     the barrier behind the forces, whose arrivals may be in the count too,
//     adds none: all flags found are the step's, and every block finds the same;
//   behind the forces the flags found are early ones of the next step's
//     movement: they stay for the barrier there.
// Either way `seen` ends up the same in every block.  The fields cannot run into
// one another: a difference holds less than twice `blocks` arrivals and at most
// `blocks` of either flag.
#pragma once

namespace gb300 {

struct BarrierPass {
  int moved, mesh_moved;
  unsigned long long seen;
};

// flags: 1 an atom of the block has moved, 2 a mesh node
__host__ __device__ inline unsigned long long barrier_arrival(int flags) {
  return 1ull + ((flags & 1) ? 1ull << 32 : 0ull) + ((flags & 2) ? 1ull << 48 : 0ull);
}

__host__ __device__ inline bool barrier_full(unsigned long long now, unsigned long long seen, int blocks) {
  return (unsigned)(now - seen) >= (unsigned)blocks;
}

// what a block takes from a full count; movement: the barrier behind phase A
__host__ __device__ inline BarrierPass barrier_pass(unsigned long long now, unsigned long long seen, int blocks,
                                                    bool movement) {
  const unsigned up = movement ? (unsigned)((now - seen) >> 32) : 0u;
  BarrierPass p;
  p.moved = (up & 0xffffu) != 0;
  p.mesh_moved = (up >> 16) != 0;
  p.seen = seen + (unsigned long long)blocks + ((unsigned long long)up << 32);
  return p;
}

}  // namespace gb300

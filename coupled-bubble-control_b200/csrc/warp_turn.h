// warp_turn.h -- what a persistent warp whose lanes hold one system each does
// next, from its lanes' votes.  A function of the votes alone, without device
// code, so that the host can check that every warp ends.
#pragma once

#if defined(__CUDACC__)
#define CBC_TURN_HD __host__ __device__ __forceinline__
#else
#define CBC_TURN_HD inline
#endif

namespace cbc {

enum class Turn { exit, refill, step };

// Votes, one bit per lane: `active` holds a system that is being integrated,
// `held` holds a system (active, or finished and not yet written back),
// `drained` takes no more systems (work list empty, time slice over, or a lane
// kept idle by the launch).  A finished system is written back and an empty lane
// filled before the next step; a warp steps only while some lane is active and
// ends when nothing is held and every lane is drained, also when that is so at
// its first turn (a block that starts after the end of its time slice).
CBC_TURN_HD Turn next_turn(unsigned active, unsigned held, unsigned drained) {
  if ((held & ~active) | ~(held | drained)) return Turn::refill;
  return active ? Turn::step : Turn::exit;
}

}  // namespace cbc

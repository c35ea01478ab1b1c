// Bounded waits of a warp on values that other warps write (ilu_trsv).  Plain
// C++, so that the rules can be run on the host with lanes that see a value at
// different polls.
//
// Lanes of a warp need not run in step, and one that polls may see a value
// before its neighbour does.  So nothing that every lane has to take part in (a
// vote, a shuffle) stands in a loop that a lane leaves on what it alone has seen:
// there each lane counts its own polls and gives up on its own, and the lanes
// meet again after it.  A loop whose exit is the result of a vote may vote again.
#pragma once

#ifdef __CUDACC__
#define CFDGPU_HD __host__ __device__ __forceinline__
#else
#define CFDGPU_HD inline
#endif

namespace cfdgpu {

// One lane's count of polls.  Every PERIOD polls it looks whether another wait
// of the group has given up, and at the clock: after LIMIT_NS it gives up itself.
// ENV: gave_up(), give_up(), now() in nanoseconds.
template <typename ENV>
struct LaneWait {
  static constexpr int PERIOD = 1024;
  static constexpr unsigned long long LIMIT_NS = 2000000000ull;
  ENV env;
  int it = 0;
  unsigned long long t0 = 0;
  CFDGPU_HD bool go_on()
  {
    if (++it & (PERIOD - 1)) return true;
    if (env.gave_up()) return false;
    const unsigned long long t = env.now();
    if (it == PERIOD) t0 = t;
    if (t - t0 < LIMIT_NS) return true;
    env.give_up();
    return false;
  }
};

// Every lane polls ready() until it is true or its wait runs out; all lanes leave together.
template <typename Ready, typename Wait, typename Sync>
CFDGPU_HD void wait_lanes(Ready ready, Wait &wait, Sync sync)
{
  while (!ready() && wait.go_on()) {}
  sync();
}

// attempt() (the same result in every lane: a vote) is repeated while it says
// "again" and no lane's wait has run out.  all(x): true in every lane if x is in every one.
template <typename Attempt, typename Wait, typename All>
CFDGPU_HD void retry_warp(Attempt attempt, Wait &wait, All all)
{
  while (attempt() && all(wait.go_on())) {}
}

}  // namespace cfdgpu

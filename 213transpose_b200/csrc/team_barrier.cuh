// The barrier word of a team of CTAs: a generation above an arrival count.
//
// The last arrival raises the generation and clears the count in one store, so
// the word needs no clearing between launches.  A CTA whose wait runs out
// withdraws its arrival, so that the word is clear for later launches, unless
// the barrier ended meanwhile.  Both are in one word because the withdrawal
// must not touch another generation's count: with the count in a word of its
// own, a barrier that ended between the withdrawal's last look at the
// generation and its exchange would lose an arrival at the next one.
//
// Word: load (acquire), add1 (acquire and release, the old value), store
// (release), cas (the old value).
#pragma once

#include <stdint.h>

namespace t213 {

constexpr uint32_t kTeamGen = 1u << 10;  // a generation; counts stay below (a team has at most two CTAs an SM)
constexpr uint32_t kTeamCount = kTeamGen - 1;

__host__ __device__ __forceinline__ uint32_t team_gen(uint32_t v) { return v & ~kTeamCount; }

#pragma nv_exec_check_disable
template <typename Word>
__host__ __device__ __forceinline__ bool team_arrive(const Word &w, uint32_t need, uint32_t gen) {
  if ((w.add1() & kTeamCount) != need - 1) return false;
  w.store(gen + kTeamGen);
  return true;
}

// True when the arrival was taken back, false when the barrier has ended.
#pragma nv_exec_check_disable
template <typename Word>
__host__ __device__ __forceinline__ bool team_withdraw(const Word &w, uint32_t need, uint32_t gen) {
  for (uint32_t v = w.load(), i = 0; team_gen(v) == gen && i < 1u << 20; i++) {
    if ((v & kTeamCount) == need) {  // the last arrival is about to end it
      v = w.load();
      continue;
    }
    const uint32_t was = w.cas(v, v - 1);
    if (was == v) return true;
    v = was;
  }
  return team_gen(w.load()) == gen;
}

}  // namespace t213

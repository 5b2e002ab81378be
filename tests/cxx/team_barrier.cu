// The team barrier's word (csrc/team_barrier.cuh) on the host: between any two
// of the withdrawal's accesses the rest of the team may arrive, end the
// barrier and arrive at the next one; whatever the moment, no arrival of the
// next generation is lost and the answer tells whether the barrier ended.
#include <cstdio>
#include <functional>

#include "team_barrier.cuh"

using namespace t213;

struct HostWord {
  uint32_t *p;
  std::function<void()> *before;  // what other CTAs do before the next access
  void other() const {
    if (*before) {
      auto f = *before;
      f();
    }
  }
  uint32_t load() const {
    other();
    return *p;
  }
  uint32_t add1() const {
    other();
    return (*p)++;
  }
  void store(uint32_t v) const {
    other();
    *p = v;
  }
  uint32_t cas(uint32_t old, uint32_t v) const {
    other();
    const uint32_t was = *p;
    if (was == old) *p = v;
    return was;
  }
};

int main() {
  int bad = 0, runs = 0;
  for (uint32_t gen : {0u, 5 * kTeamGen, ~kTeamCount})       // the last one wraps
    for (uint32_t ctas : {2u, 3u, 4u, 17u, 296u})
      for (uint32_t here : {1u, (ctas + 1) / 2, ctas - 1})   // arrivals when the wait runs out, this CTA's among them
        for (uint32_t next : {0u, 1u, ctas / 2, ctas - 1})   // arrivals at the next generation: this CTA makes none
          for (int at = 0; at < 4; at++)                     // before which access the others go on
            for (int half = 0; half < 2; half++) {           // 1: the last arrival is seen before its store
              uint32_t word = gen + here;
              int access = 0;
              bool ended = false;
              std::function<void()> none, script;
              HostWord plain{&word, &none};
              script = [&] {
                if (access++ == at && team_gen(word) == gen && (word & kTeamCount) == here) {
                  for (uint32_t i = here; i + 1 < ctas; i++) team_arrive(plain, ctas, gen);
                  plain.add1();  // the last arrival
                  ended = true;
                  if (half) return;
                  plain.store(gen + kTeamGen);
                  for (uint32_t i = 0; i < next; i++) team_arrive(plain, ctas, gen + kTeamGen);
                } else if (ended && half && team_gen(word) == gen) {
                  plain.store(gen + kTeamGen);
                  for (uint32_t i = 0; i < next; i++) team_arrive(plain, ctas, gen + kTeamGen);
                }
              };
              HostWord w{&word, &script};
              const bool withdrawn = team_withdraw(w, ctas, gen);
              runs++;
              const uint32_t want = withdrawn ? gen + here - 1 : gen + kTeamGen + next;
              if (withdrawn == ended || word != want) {
                if (bad++ < 5)
                  printf("gen %u ctas %u here %u next %u at %d half %d: withdrawn %d ended %d word %x want %x\n", gen, ctas,
                         here, next, at, half, withdrawn, ended, word, want);
              }
            }
  printf(bad ? "%d of %d runs wrong\n" : "ok (%d wrong of %d)\n", bad, runs);
  return bad != 0;
}

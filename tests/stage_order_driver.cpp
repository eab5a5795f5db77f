// Every interleaving of the apply engine's ring of stages for the first items, with
// barriers that know their phases by parity only: the producer stages an item when the
// stage's last one has been worked off, its bytes land at any later time, the groups
// wait by stage_landed.  Exit 1 when a group can take an item that has not landed, 2
// when everything can come to a halt, else 0.
#include <array>
#include <cstdio>
#include <set>
#include <vector>

#include "stage_order.h"

using namespace rschol::solvedev;

constexpr int ITEMS = 3 * NSTAGE * NGRP;

struct State {
  int issued = 0;                       // items staged by the producer
  unsigned long long landed = 0;        // bit k: item k's bytes are there
  std::array<int, NSTAGE> full{}, empty{};   // completed phases of the barriers
  std::array<int, NGRP> next{};         // a group's next item
  std::array<int, NGRP> busy{};         // 1 while it works on it
  bool operator<(const State& o) const {
    if (issued != o.issued) return issued < o.issued;
    if (landed != o.landed) return landed < o.landed;
    if (full != o.full) return full < o.full;
    if (empty != o.empty) return empty < o.empty;
    if (next != o.next) return next < o.next;
    return busy < o.busy;
  }
};

// a wait on a parity returns once the phase of that parity is the last one completed
static bool passes(int completed, int parity) { return (completed & 1) != parity; }

int main() {
  State first;
  for (int g = 0; g < NGRP; ++g) first.next[g] = g;
  std::set<State> seen{first};
  std::vector<State> todo{first};
  while (!todo.empty()) {
    const State st = todo.back();
    todo.pop_back();
    bool moved = false, done = true;
    auto go = [&](const State& n) {
      moved = true;
      if (seen.insert(n).second) todo.push_back(n);
    };
    if (st.issued < ITEMS) {
      const int s = st.issued % NSTAGE, use = st.issued / NSTAGE;
      if (use == 0 || passes(st.empty[s], (use - 1) & 1)) {
        State n = st;
        ++n.issued;
        go(n);
      }
    }
    for (int k = 0; k < st.issued; ++k)
      if (!(st.landed >> k & 1)) {
        State n = st;
        n.landed |= 1ull << k;
        ++n.full[k % NSTAGE];
        go(n);
      }
    for (int g = 0; g < NGRP; ++g) {
      const int k = st.next[g];
      if (k >= ITEMS) continue;
      done = false;
      State n = st;
      if (st.busy[g]) {
        ++n.empty[k % NSTAGE];
        n.busy[g] = 0;
        n.next[g] += NGRP;
        go(n);
      } else if (stage_landed(
                     k, [&](int s, int p) { return passes(st.full[s], p); },
                     [&](int s, int p) { return passes(st.empty[s], p); })) {
        if (!(st.landed >> k & 1)) {
          std::printf("group %d takes item %d before it has landed\n", g, k);
          return 1;
        }
        n.busy[g] = 1;
        go(n);
      }
    }
    if (!moved && !done) {
      std::printf("halt after %d items\n", st.issued);
      return 2;
    }
  }
  std::printf("%zu states\n", seen.size());
  return 0;
}

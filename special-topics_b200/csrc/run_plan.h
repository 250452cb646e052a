// run_plan.h -- the CUDA graphs that a run replays, and which of them are kept
// for the next run.  Host code without CUDA calls, so that it can be tested
// without a device.
#pragma once
#include <algorithm>
#include <cstddef>
#include <vector>

namespace fdtd {

constexpr int kGraphSteps = 64;         // shortest cap of a graph's steps
constexpr int kMaxGraphNodes = 40000;   // kernel launches held by one graph at most
constexpr int kWholeNodes = 1024;       // a run of at most so many launches is one graph from any start
constexpr size_t kMinCachedGraphs = 8, kMaxCachedGraphs = 256;
constexpr long long kMaxCachedNodes = kMaxGraphNodes;  // launches held by more than kMinCachedGraphs graphs

// What the launches of a graph depend on beyond how many steps they are: the
// path, and on the one-pass path the copy of the state that it starts from and
// its place in a time block of the surface DFT, as a flush is queued where a
// block closes.
struct RunStart {
  bool one_pass = false;
  int copy = 0;
  int phase = 0, block = 0;  // steps into a block; steps of one, 0: no blocks

  RunStart after(int steps) const {
    RunStart s = *this;
    s.copy ^= steps & 1;
    if (block > 0) s.phase = (phase + steps) % block;
    return s;
  }
  // Steps after which copy and phase are as before.
  int period() const { return !one_pass ? 1 : block <= 0 ? 2 : block % 2 ? 2 * block : block; }
  // The start, as far as `steps` steps depend on it: without a block that closes
  // in them the phase is of no account.
  long long tag(int steps) const {
    if (!one_pass) return 0;
    return 1 + copy + (block > 0 && phase + steps >= block ? 2LL * (phase + 1) : 0);
  }
  long long key(int steps) const { return (long long)steps << 16 | tag(steps); }
};

// One graph of a run: its first step, counted from the run's, and its steps.
struct RunPiece {
  int at, steps;
};

// The pieces of a run of `count` steps of `launches` launches each: graphs of at
// most `cap` steps (0: as many as kMaxGraphNodes allows), whole periods where it
// holds any, else none across a block's end.  A run that starts inside a block
// and is too long to be captured once for each place in it goes to the block's
// end first, then takes whole periods, whose number depends on `count` alone,
// then the rest: its one long graph serves it from any place.
// (Runs of 50 steps at a block of 16 start at eight places.  With six graphs kept
// each run was captured anew: 10.0 ms a run, 9.0 with its graph there, and a
// single step 0.81 ms, 0.35 with, on the 78x272x272 antenna at 64 frequencies.)
inline std::vector<RunPiece> run_pieces(int count, const RunStart& s, int launches, int cap) {
  std::vector<RunPiece> out;
  const int period = s.period();
  launches = std::max(1, launches);
  if (cap <= 0) cap = std::max(kGraphSteps, kMaxGraphNodes / launches);
  const bool periods = cap >= period;
  if (periods) cap = cap / period * period;
  int at = 0;
  auto take = [&](int steps) {
    for (const int end = at + steps; at < end; at += out.back().steps)
      out.push_back({at, std::min({cap, end - at, periods ? cap : s.block - s.after(at).phase})});
  };
  if (periods && s.phase > 0 && count >= 2 * period && (long long)count * launches > kWholeNodes) {
    take(s.block - s.phase);
    take((count - (s.block - 1)) / period * period);
  }
  take(count - at);
  return out;
}

// Graphs by key, the most recently used last.  A plan finds or adds its graphs
// one after another and launches them when it has all: fewer than
// kMinCachedGraphs of them, so that none of them is the one that makes room for
// the next.
template <class Exec>
struct GraphCache {
  struct Entry {
    long long key, nodes;
    Exec exec;
  };
  std::vector<Entry> g;

  // The graph of `key`, or NULL.
  Exec* find(long long key) {
    for (size_t q = 0; q < g.size(); q++)
      if (g[q].key == key) {
        const Entry e = g[q];
        g.erase(g.begin() + q);
        g.push_back(e);
        return &g.back().exec;
      }
    return nullptr;
  }
  // Adds a graph that is not there; `destroy` takes those that make room.
  template <class D>
  void add(long long key, long long nodes, Exec e, D destroy) {
    long long held = nodes;
    for (const Entry& q : g) held += q.nodes;
    while (g.size() >= kMaxCachedGraphs || (g.size() >= kMinCachedGraphs && held > kMaxCachedNodes)) {
      held -= g.front().nodes;
      destroy(g.front().exec);
      g.erase(g.begin());
    }
    g.push_back({key, nodes, e});
  }
};

}  // namespace fdtd

// run_plan.h -- the CUDA graphs that a run replays, and which of them are kept
// for the next run.  Host code without CUDA calls, so that it can be tested
// without a device.
#pragma once
#include <cstddef>
#include <vector>

namespace fdtd {

constexpr size_t kMaxCachedGraphs = 6;

// Graphs by key, the most recently used last.  A plan finds or adds its graphs
// one after another and launches them when it has all: fewer than
// kMaxCachedGraphs of them, so that none of them is the one that makes room for
// the next.
template <class Exec>
struct GraphCache {
  struct Entry {
    long long key;
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
  void add(long long key, Exec e, D destroy) {
    while (g.size() >= kMaxCachedGraphs) {
      destroy(g.front().exec);
      g.erase(g.begin());
    }
    g.push_back({key, e});
  }
};

}  // namespace fdtd

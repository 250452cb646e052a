"""The graphs that a run replays (csrc/run_plan.h), without a device: the header
is compiled into small programs whose "graphs" are numbers."""
import os
import shutil
import subprocess

import pytest

from conftest import ROOT

CSRC = os.path.join(ROOT, "special-topics_b200", "csrc")


def _run(tmp_path, body):
    src = tmp_path / "t.cpp"
    src.write_text('#include <cstdio>\n#include <cstdlib>\n#include <map>\n#include <set>\n#include "run_plan.h"\n'
                   '#define REQUIRE(x) do { if (!(x)) { printf("%s: line %d\\n", #x, __LINE__); exit(1); } } while (0)\n'
                   "using namespace fdtd;\n" + body)
    exe = tmp_path / "t"
    subprocess.run([shutil.which("g++"), "-std=c++17", "-O1", f"-I{CSRC}", "-o", str(exe), str(src)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0, r.stdout


def test_a_plans_graphs_outlive_the_plans_own_captures(tmp_path):
    """Runs of one full graph and a remainder that differs each time: the full
    graph, found and not captured again, is not the one that makes room."""
    _run(tmp_path, """
int main() {
  GraphCache<int> c;
  std::set<int> dead;
  int made = 0, captures = 0;
  auto get = [&](long long key) {
    if (int* e = c.find(key)) return *e;
    captures++;
    c.add(key, 10000, ++made, [&](int old) { dead.insert(old); });
    return made;
  };
  for (int run = 0; run < 40; run++) {
    const int full = get(32), rest = get(1000 + run);
    REQUIRE(!dead.count(full) && !dead.count(rest));
  }
  REQUIRE(captures == 41 && c.g.size() == kMinCachedGraphs);
}
""")


SIM = """
// A graph as what was captured: for each step the copy read, and whether a flush follows.
struct Sim {
  GraphCache<int> cache;
  std::map<int, std::vector<int>> graphs;
  int made = 0, captures = 0;
  int copy = 0, ts = 0, block = 0, launches = 3, cap = 0;
  bool one_pass = true;
  RunStart start() const {
    RunStart s;
    s.one_pass = one_pass, s.copy = copy, s.block = block, s.phase = block ? ts % block : 0;
    return s;
  }
  std::vector<int> steps(int copy0, int ts0, int n) const {
    std::vector<int> v;
    for (int q = 0; q < n && one_pass; q++) v.push_back(((copy0 + q) & 1) + 2 * (block > 0 && (ts0 + q + 1) % block == 0));
    return v;
  }
  int run(int count) {
    const RunStart s = start();
    int at = 0, pieces = 0;
    std::vector<int> plan, at_of;
    const int graph_cap = cap ? cap : kMaxGraphNodes / launches;
    for (const RunPiece& p : run_pieces(count, s, launches, cap)) {
      REQUIRE(p.at == at && p.steps > 0 && p.steps <= graph_cap);
      at += p.steps;
      const long long key = s.after(p.at).key(p.steps);
      int* have = cache.find(key);
      if (!have) {
        captures++;
        graphs[++made] = steps(copy ^ (p.at & 1), ts + p.at, p.steps);
        cache.add(key, (long long)p.steps * launches, made, [&](int e) { graphs.erase(e); });
        have = cache.find(key);
      }
      plan.push_back(*have);
      at_of.push_back(p.at);
    }
    REQUIRE(at == count);
    for (size_t q = 0; q < plan.size(); q++) {   // every graph is still there, and does what its steps need
      REQUIRE(graphs.count(plan[q]));
      const int n = (q + 1 < plan.size() ? at_of[q + 1] : count) - at_of[q];
      REQUIRE(!one_pass || graphs[plan[q]] == steps(copy ^ (at_of[q] & 1), ts + at_of[q], n));
    }
    copy ^= count & 1;
    ts += count;
    long long held = 0;
    for (auto& e : cache.g) held += e.nodes;
    REQUIRE(cache.g.size() <= kMinCachedGraphs || (cache.g.size() <= kMaxCachedGraphs && held <= kMaxCachedNodes));
    return captures;
  }
};
"""


@pytest.mark.parametrize("block", [0, 2, 3, 7, 16, 33, 1024])
def test_every_graph_does_what_its_place_needs(tmp_path, block):
    """Runs of all lengths, a block's and a graph's limits among them, alone (3
    launches a step) and as 32 chains of a batch (160 launches, 25 steps a graph):
    a graph from the cache has the copies and flushes of the steps that it is
    launched for, and a block longer than a graph does not lengthen the graph."""
    _run(tmp_path, SIM + """
int main() {
  srand(5);
  for (int kind = 0; kind < 2; kind++) {
    Sim s;
    s.block = %d;
    if (kind) s.launches = 160, s.cap = 25;
    const int lengths[] = {1, 2, 15, 16, 17, 23, 24, 25, 26, 31, 32, 33, 50, 64, 341, 342, 1023, 1024, 1025, 2049, 5000, 15000};
    for (int q = 0; q < 3000; q++) s.run(q %% 3 ? lengths[rand() %% 22] : 1 + rand() %% 700);
  }
}
""" % block)


@pytest.mark.parametrize("count,launches,cap", [(1, 3, 0), (7, 3, 0), (50, 3, 0), (500, 3, 0), (50, 160, 25), (3, 160, 25)])
@pytest.mark.parametrize("block", [0, 3, 16])
def test_equal_runs_stop_capturing(tmp_path, block, count, launches, cap):
    """Runs of one length from every place in a block: after two rounds of the
    places all graphs are there."""
    _run(tmp_path, SIM + """
int main() {
  Sim s;
  s.block = %d, s.launches = %d, s.cap = %d;
  int warm = 0;
  for (int q = 0; q < 400; q++) {
    const int n = s.run(%d);
    if (q == 4 * (s.block ? s.block : 1)) warm = n;
    REQUIRE(!warm || n == warm);
  }
}
""" % (block, launches, cap, count))

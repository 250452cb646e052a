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
    c.add(key, ++made, [&](int old) { dead.insert(old); });
    return made;
  };
  for (int run = 0; run < 40; run++) {
    const int full = get(32), rest = get(1000 + run);
    REQUIRE(!dead.count(full) && !dead.count(rest));
  }
  REQUIRE(captures == 41 && c.g.size() == kMaxCachedGraphs);
}
""")

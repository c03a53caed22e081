"""The serving engine's plan cache (csrc/plan_cache.h), compiled for the host:
a plan that a run holds is never destroyed, whatever the run's other jobs
bring in, and the cache is back at its capacity once the run is over."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
DRIVER = r"""
#include "plan_cache.h"
#include <cstdio>
#include <set>
#include <vector>

static std::set<int *> live;
static void destroy(int *p) { live.erase(p); delete p; }
using Cache = subby::PlanCache<int *, void (*)(int *)>;

#define CHECK(x) do { if (!(x)) { std::printf("line %d: %s\n", __LINE__, #x); return 1; } } while (0)

static int *take(Cache &c, uint64_t key, size_t capacity) {
  int *p = c.take(key);
  if (!p) {
    p = new int((int)key);
    live.insert(p);
    c.add(key, p, capacity);
  }
  return p;
}

int main() {
  for (size_t cap : {1, 8, 64}) {
    for (int batch : {1, 7, 8, 40, 85}) {
      Cache c(destroy);
      for (int round = 0; round < 3; ++round) {
        // a batch of distinct trees beside one that the run before left behind
        std::vector<int *> held;
        for (int i = 0; i < batch; ++i) held.push_back(take(c, 1000 * round + i, cap));
        CHECK(take(c, 1000 * round, cap) == held[0]);   // a second job on the first tree
        for (int i = 0; i < batch; ++i) {
          CHECK(live.count(held[i]) && *held[i] == 1000 * round + i && c.pinned(1000 * round + i));
        }
        CHECK(c.size() <= cap + batch);
        for (int i = 0; i < batch; ++i) CHECK(c.drop(1000 * round + i) == held[i]);
        c.trim(cap);
        CHECK(c.pinned(1000 * round) && live.count(held[0]));   // its second job still runs
        CHECK(c.drop(1000 * round) == held[0] && !c.pinned(1000 * round));
        CHECK(c.drop(1000 * round) == nullptr && c.drop(77777) == nullptr);
        c.trim(cap);
        CHECK(c.size() <= cap && c.size() == live.size());
      }
      c.clear();
      CHECK(c.size() == 0 && live.empty());
    }
  }
  // least recently used first out
  Cache c(destroy);
  for (uint64_t k : {1, 2, 3}) take(c, k, 3), c.drop(k);
  take(c, 1, 3), c.drop(1);
  take(c, 4, 3), c.drop(4);
  CHECK(c.size() == 3 && !c.take(2) && c.take(1) && c.take(3) && c.take(4));
  c.clear();
  CHECK(live.empty());
  return 0;
}
"""


@pytest.mark.skipif(shutil.which("g++") is None, reason="needs a host compiler")
def test_plans_of_a_run_outlive_the_cache_limit(tmp_path):
    src, exe = tmp_path / "cache.cpp", tmp_path / "cache"
    src.write_text(DRIVER)
    subprocess.run(["g++", "-std=c++17", "-O1", "-Wall", "-Werror",
                    "-I", os.path.join(ROOT, "subby_gb300", "csrc"), str(src), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True, timeout=120)
    assert r.returncode == 0, r.stdout

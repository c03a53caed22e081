"""Plans of different sizes run by several host threads of a native program at
once: the launches of one kernel ask for different amounts of shared memory,
and none of them may take away what another one needs."""
import os
import subprocess

import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():  # pragma: no cover
    pytest.skip("needs a CUDA GPU", allow_module_level=True)

from subby_gb300 import _build, _lib  # noqa: E402

DRIVER = r"""
#include <atomic>
#include <cstdio>
#include <cstdlib>
#include <random>
#include <thread>
#include <vector>
#include <cuda_runtime.h>
#include "subby_gb300.h"

int main(int argc, char **argv) {
  const int A = std::atoi(argv[1]), mode = std::atoi(argv[2]), runs = std::atoi(argv[3]);
  std::atomic<int> bad{0}, ready{0};
  std::vector<std::thread> th;
  const int leaves[4] = {4, A == 4 && mode < 2 ? 500 : 90, 40, 150}, C[4] = {40, 300, 2000, 500};
  for (int k = 0; k < 4; ++k)
    th.emplace_back([&, k] {
      std::mt19937 r(k);
      const int R = 2 * leaves[k] - 1;
      std::vector<int> par(R, -1);
      std::vector<double> t(R, 0.1), ev(A, -1.1), V(A * A), pi(A, 1.0 / A);
      int cur = 0;
      for (int n = 1; n < R; n += 2) par[n] = par[n + 1] = cur, cur = n + (r() & 1);
      ev[0] = 0.0;   // Jukes-Cantor: the Householder basis of (1, ..., 1)
      for (int i = 0; i < A; ++i)
        for (int j = 0; j < A; ++j) {
          const double u = 1.0 / std::sqrt((double)A), w = 1.0 / (1.0 - u);
          const double a = u - (i == 0), b = u - (j == 0);
          V[i * A + j] = (i == j) - w * a * b;
        }
      subby_plan *p = nullptr;
      int rc = subby_plan_create(par.data(), t.data(), ev.data(), V.data(), pi.data(), R, A, &p);
      int *d;
      float *out;
      cudaMalloc(&d, 4ull * R * C[k]);
      cudaMemset(d, 0, 4ull * R * C[k]);
      cudaMalloc(&out, 4ull * A * A * C[k] * (mode == 2 ? R : 1));
      cudaStream_t s;
      cudaStreamCreateWithFlags(&s, cudaStreamNonBlocking);
      cudaDeviceSynchronize();
      ++ready;
      while (ready < 4) std::this_thread::yield();
      for (int i = 0; i < runs && !rc && !bad; ++i) {
        if (mode == 0) rc = subby_plan_run(p, d, C[k], nullptr, out, nullptr, 0, 1, nullptr, SUBBY_DEVICE_PTRS, s);
        if (mode == 1) rc = subby_plan_run(p, d, C[k], out, nullptr, nullptr, 0, 0, nullptr, SUBBY_DEVICE_PTRS, s);
        if (mode == 2) rc = subby_plan_branch_counts(p, d, C[k], out, 0, 0, nullptr, SUBBY_DEVICE_PTRS, s);
        if (i % 64 == 0) cudaStreamSynchronize(s);
      }
      if (rc) std::printf("thread %d: %s\n", k, subby_last_error()), ++bad;
      cudaStreamSynchronize(s);
      subby_plan_destroy(p);
    });
  for (auto &x : th) x.join();
  if (cudaDeviceSynchronize() != cudaSuccess) std::printf("device error\n"), ++bad;
  return bad.load() != 0;
}
"""


@pytest.fixture(scope="module")
def driver(tmp_path_factory):
    lib = _lib.library_path()
    _lib.load()
    tmp = tmp_path_factory.mktemp("threads")
    src, exe = tmp / "threads.cu", tmp / "threads"
    src.write_text("#include <cmath>\n" + DRIVER)
    subprocess.run([_build.nvcc(), "-O2", "-std=c++17", "-I", _build.INCLUDE, str(src), lib, "-o", str(exe),
                    "-Xlinker", "-rpath", "-Xlinker", os.path.dirname(lib)], check=True)
    return str(exe)


# counts, LogLike, per-branch counts
@pytest.mark.parametrize("A,mode,runs", [(4, 0, 6000), (4, 1, 6000), (4, 2, 3000), (8, 0, 3000)])
def test_plans_of_different_sizes_in_threads(driver, A, mode, runs):
    r = subprocess.run([driver, str(A), str(mode), str(runs)], stdout=subprocess.PIPE, stderr=subprocess.STDOUT,
                       text=True, timeout=300)
    assert r.returncode == 0, r.stdout

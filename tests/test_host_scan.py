"""The host scan for non-finite values (``csrc/krr_finite.h``) when threads cannot be started (CPU).

The header is compiled into a program whose ``pthread_create`` succeeds a given number of times and
then reports that no more threads are to be had.
"""

from __future__ import annotations

import subprocess

import pytest

from conftest import ROOT

PROGRAM = r"""
#include <dlfcn.h>
#include <errno.h>
#include <pthread.h>
#include <atomic>
#include <cstdio>
#include <cstdlib>
#include <limits>
#include "krr_finite.h"

static std::atomic<int> left{0};
extern "C" int pthread_create(pthread_t* t, const pthread_attr_t* a, void* (*f)(void*), void* p) {
  if (left.fetch_sub(1) <= 0) return EAGAIN;
  using Fn = int (*)(pthread_t*, const pthread_attr_t*, void* (*)(void*), void*);
  return reinterpret_cast<Fn>(dlsym(RTLD_NEXT, "pthread_create"))(t, a, f, p);
}

int main(int, char** argv) {
  const int threads = std::atoi(argv[1]);
  const size_t n = std::strtoull(argv[2], nullptr, 10);
  std::vector<double> x(n, 1.0e308);
  const double values[] = {0.0, std::numeric_limits<double>::infinity(), -std::numeric_limits<double>::infinity(),
                           std::numeric_limits<double>::quiet_NaN()};
  for (size_t at : {(size_t)0, n / 2, n - 1})
    for (double v : values) {
      x[at] = v;
      left = threads;
      std::printf("%d", (int)krr_host::all_finite_parallel(x.data(), n));
      x[at] = -0.0;
    }
  return 0;
}
"""


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    folder = tmp_path_factory.mktemp("scan")
    (folder / "scan.cpp").write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-O2", "-I", str(ROOT / "kerrray_b200" / "csrc"), str(folder / "scan.cpp"), "-o",
                    str(folder / "scan"), "-pthread", "-ldl"], check=True)
    return folder / "scan"


@pytest.mark.parametrize("n", [1, (1 << 22) - 1, 1 << 22, (1 << 22) + 7])
@pytest.mark.parametrize("threads", [0, 1, 3, 1000])
def test_every_value_is_seen_however_many_threads_start(program, threads, n):
    run = subprocess.run([str(program), str(threads), str(n)], capture_output=True, text=True, timeout=120)
    assert run.returncode == 0, run.stderr
    assert run.stdout == "1000" * 3

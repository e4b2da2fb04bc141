"""The pinned staging memory's host side (``csrc/krr_staging.h``) against a CUDA runtime of the test's own (CPU).

The header is compiled with a ``cuda_runtime.h`` whose copies are immediate, whose pinned
allocations and event creations succeed a given number of times, and whose stream can be held (a
kernel running ahead of the copies): events then complete when it is let go.
"""

from __future__ import annotations

import subprocess

import pytest

from conftest import ROOT

RUNTIME = r"""
#pragma once
#include <atomic>
#include <chrono>
#include <cmath>
#include <cstdlib>
#include <cstring>
#include <thread>
#include <vector>
enum cudaError_t { cudaSuccess = 0, cudaErrorMemoryAllocation = 2, cudaErrorUnknown = 999 };
enum cudaMemcpyKind { cudaMemcpyHostToDevice = 1, cudaMemcpyDeviceToHost = 2 };
enum cudaMemoryType { cudaMemoryTypeUnregistered = 0, cudaMemoryTypeHost = 1 };
struct cudaPointerAttributes { cudaMemoryType type; };
using cudaStream_t = int;
struct FakeEvent { std::atomic<bool> recorded{false}; };
using cudaEvent_t = FakeEvent*;
constexpr unsigned cudaHostAllocDefault = 0, cudaEventDisableTiming = 2;
namespace fake {
inline std::atomic<int> allocs{1 << 30}, events{1 << 30}, made{0}, freed{0}, direct{0}, waiting{0}, most_waiting{0};
inline std::atomic<bool> held{false};
inline std::vector<char*> blocks;
inline std::vector<double>* poisoned = nullptr;  // another thread's array: it turns to NaN when the first copy is queued
inline bool pinned(const void* p) {
  for (char* b : blocks)
    if (p >= b && p < b + ((size_t)4 << 20)) return true;
  return false;
}
inline void wait() {
  const int n = ++waiting;
  int seen = most_waiting;
  while (n > seen && !most_waiting.compare_exchange_weak(seen, n)) {}
  while (held) std::this_thread::sleep_for(std::chrono::milliseconds(1));
  --waiting;
}
}  // namespace fake
inline cudaError_t cudaHostAlloc(void** p, size_t n, unsigned) {
  if (fake::allocs.fetch_sub(1) <= 0) return cudaErrorMemoryAllocation;
  *p = std::malloc(n);
  fake::blocks.push_back(static_cast<char*>(*p));
  ++fake::made;
  return cudaSuccess;
}
inline cudaError_t cudaFreeHost(void*) { return ++fake::freed, cudaSuccess; }
inline cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) {
  return fake::events.fetch_sub(1) <= 0 ? cudaErrorMemoryAllocation : (*e = new FakeEvent, cudaSuccess);
}
inline cudaError_t cudaEventDestroy(cudaEvent_t e) { return delete e, cudaSuccess; }
inline cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t) { return e->recorded = true, cudaSuccess; }
inline cudaError_t cudaEventSynchronize(cudaEvent_t e) {
  if (e->recorded) fake::wait();
  return cudaSuccess;
}
inline cudaError_t cudaStreamSynchronize(cudaStream_t) { return fake::wait(), cudaSuccess; }
inline cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind, cudaStream_t) {
  if (fake::poisoned)
    for (double& x : *fake::poisoned) x = NAN;
  if (!fake::pinned(d) && !fake::pinned(s)) ++fake::direct;
  std::memcpy(d, s, n);
  return cudaSuccess;
}
inline cudaError_t cudaPointerGetAttributes(cudaPointerAttributes* a, const void*) {
  a->type = cudaMemoryTypeUnregistered;
  return cudaSuccess;
}
inline cudaError_t cudaGetLastError() { return cudaSuccess; }
inline cudaError_t cudaSetDevice(int) { return cudaSuccess; }
"""

PROGRAM = r"""
#include <cstdio>
#include <limits>
#include "krr_staging.h"

// Arrays of the sizes given (in doubles) through `staging`, out and in; prints what arrived.
static void both_ways(krr_host::Staging& staging, const std::vector<size_t>& sizes) {
  std::vector<std::vector<double>> a, b, c;
  std::vector<krr_host::CopySpan> out, in;
  for (size_t n : sizes) {
    a.emplace_back(n);
    for (size_t i = 0; i < n; ++i) a.back()[i] = 1.0 + (double)(i * 2654435761u % 1000003);
    b.emplace_back(n, -1.0);
    c.emplace_back(n, -1.0);
  }
  for (size_t k = 0; k < sizes.size(); ++k) {
    out.push_back({b[k].data(), a[k].data(), sizes[k] * 8});
    in.push_back({c[k].data(), a[k].data(), sizes[k] * 8});
  }
  std::atomic<bool> bad{false};
  bool ok = staging.out(0, out, 0) == cudaSuccess && staging.in(0, in, 0, &bad) == cudaSuccess && a == b && a == c && !bad;
  a.back().back() = std::numeric_limits<double>::infinity();
  ok = ok && staging.in(0, in, 0, &bad) == cudaSuccess && bad;
  std::printf("ok %d made %d freed %d direct %d\n", (int)ok, (int)fake::made, (int)fake::freed, (int)fake::direct);
}

int main(int argc, char** argv) {
  krr_host::Staging staging;
  const std::vector<size_t> sizes = {100000, 131072, 131073, 1, 900000, 4500000};
  if (argc > 4) {  // one checked array, written to while it is copied
    fake::allocs = std::atoi(argv[4]);
    std::vector<double> a(std::atoll(argv[3]), 1.0), b(a.size(), 0.0);
    fake::poisoned = &a;
    std::atomic<bool> bad{false};
    const bool ok = staging.in(0, {{b.data(), a.data(), a.size() * 8}}, 0, &bad) == cudaSuccess;
    bool finite = true;
    for (double x : b) finite = finite && std::isfinite(x);
    std::printf("ok %d sound %d\n", (int)ok, (int)(bad || finite));
  } else if (argc > 2) {
    fake::allocs = std::atoi(argv[1]);
    fake::events = std::atoi(argv[2]);
    both_ways(staging, sizes);
  } else {
    fake::held = true;
    std::thread kernel([] {
      std::this_thread::sleep_for(std::chrono::milliseconds(300));
      std::printf("waiting %d\n", (int)fake::most_waiting);
      fake::held = false;
    });
    std::vector<double> from(4000000, 2.5), to(4000000, 0.0);
    const bool ok = staging.out(0, {{to.data(), from.data(), from.size() * 8}}, 0) == cudaSuccess && to == from;
    kernel.join();
    std::printf("ok %d\n", (int)ok);
  }
  return 0;
}
"""


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    folder = tmp_path_factory.mktemp("staging")
    (folder / "cuda_runtime.h").write_text(RUNTIME)
    (folder / "staging.cpp").write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-O1", "-I", str(folder), "-I", str(ROOT / "kerrray_b200" / "csrc"),
                    str(folder / "staging.cpp"), "-o", str(folder / "staging"), "-pthread"], check=True)
    return folder / "staging"


def _run(program, *args):
    run = subprocess.run([str(program), *map(str, args)], capture_output=True, text=True, timeout=120)
    assert run.returncode == 0, run.stderr
    return run.stdout.split()


@pytest.mark.parametrize("allocs,events,direct", [
    (1000, 1000, False),
    (3, 1000, False),   # 12 slots of 32
    (1, 1000, False),
    (0, 1000, True),    # no pinned memory at all
    (1000, 6, False),   # the second group's events fail
    (1000, 2, True),
])
def test_transfers_do_with_the_pinned_memory_there_is(program, allocs, events, direct):
    words = _run(program, allocs, events)
    assert words[:2] == ["ok", "1"]
    assert (int(words[words.index("direct") + 1]) > 0) == direct


def test_one_thread_waits_for_the_trace(program):
    """A 32 MB result behind a kernel: twelve threads may copy, one may wait for the kernel's end."""
    assert _run(program) == ["waiting", "1", "ok", "1"]


@pytest.mark.parametrize("doubles", [1000, 131072])
@pytest.mark.parametrize("allocs", [0, 1000])
def test_values_copied_are_the_ones_checked(program, doubles, allocs):
    """With and without pinned memory the caller's array is read once."""
    assert _run(program, 2, 1, doubles, allocs) == ["ok", "1", "sound", "1"]

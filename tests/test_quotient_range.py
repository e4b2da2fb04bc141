"""``quotient_any`` (``csrc/krr_quotient.cuh``) against IEEE division for operands of any size (CPU).

The header is compiled for the host, with a reciprocal of 19 correct bits in the place of the
hardware's.
"""

from __future__ import annotations

import subprocess

import pytest

from conftest import ROOT

RUNTIME = r"""
#pragma once
#include <cmath>
#include <cstdint>
#include <cstdio>
#include <cstring>
#include <limits>
#include <random>
#define __device__
#define __forceinline__ inline
#define __noinline__
using std::fma;
inline int __double2hiint(double x) { int64_t b; std::memcpy(&b, &x, 8); return (int)(b >> 32); }
inline double seed(double b) {
  double y = 1.0 / b;
  int64_t bits;
  std::memcpy(&bits, &y, 8);
  bits &= ~((1ll << 33) - 1);
  std::memcpy(&y, &bits, 8);
  return y;
}
#define asm(...) y = seed(b)
"""

PROGRAM = r"""
#include "krr_quotient.cuh"
#undef asm

int main() {
  std::mt19937_64 rng(5);
  auto number = [&](int lo, int hi) {  // a random fraction, or one next to a power of two
    const int e = lo + (int)(rng() % (unsigned)(hi - lo + 1));
    double f = 1.0 + (double)(rng() >> 12) * 0x1p-52;
    if (rng() % 4 == 0) f = rng() % 2 ? 1.0 + (double)(rng() % 4) * 0x1p-52 : 2.0 - (double)(1 + rng() % 4) * 0x1p-52;
    return std::ldexp(rng() % 2 ? f : -f, e);
  };
  const double inf = std::numeric_limits<double>::infinity();
  const double special[] = {0.0, -0.0, inf, -inf, std::nan(""), 0x1p-1074, 0x1p-1022, 0x1.fffffffffffffp1023};
  long wrong = 0;
  auto check = [&](double a, double b) {
    const double got = krr::quotient_any(a, b), want = a / b;
    if (got == want || (got != got && want != want)) return;
    if (wrong++ < 5) std::printf("%a / %a: %a, not %a\n", a, b, got, want);
  };
  for (int k = 0; k < 2000000; ++k) {
    check(number(-1074, 1023), number(-1074, 1023));
    check(number(-1074, 1023), number(-420, 420));
    check(number(-560, 560), number(-420, 420));
    check(number(-30, 30), number(-30, 30));
  }
  for (int e = -1074; e <= 1023; ++e)  // the ends of the ranges
    for (int f : {-401, -400, -399, 399, 400, 401}) {
      check(number(e, e), number(f, f));
      check(std::ldexp(1.0, e), std::ldexp(1.0, f));
    }
  for (double a : special)
    for (double b : special) {
      check(a, b);
      check(a, number(-500, 500));
      check(number(-500, 500), b);
    }
  std::printf("wrong %ld\n", wrong);
  return 0;
}
"""


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    folder = tmp_path_factory.mktemp("quotient")
    (folder / "cuda_runtime.h").write_text(RUNTIME)
    (folder / "q.cpp").write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-O2", "-ffp-contract=off", "-I", str(folder), "-I",
                    str(ROOT / "kerrray_b200" / "csrc"), str(folder / "q.cpp"), "-o", str(folder / "q")], check=True)
    return folder / "q"


def test_any_operands_give_the_ieee_quotient(program):
    run = subprocess.run([str(program)], capture_output=True, text=True, timeout=300)
    assert run.returncode == 0 and run.stdout == "wrong 0\n", run.stdout

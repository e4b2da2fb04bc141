"""The branch-free divisions (``csrc/krr_quotient.cuh``) and operands of extreme size.

On the CPU ``quotient_any`` against IEEE division, the header compiled for the host with a reciprocal of
19 correct bits in the place of the hardware's, and the metric terms' sizes over the scales that the
kernels' tests let through; on the GPU scales inside and outside that range against each other.
"""

from __future__ import annotations

import math
import random
import subprocess

import numpy as np
import pytest

import kerrray_b200 as K
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


def _terms(m, a, r, s, c, sin2th):
    """Denominators and numerators of the metric terms, as the kernel forms them (every operation rounded)."""
    a2, two_a2 = a * a, 2.0 * (a * a)
    s2, r2 = s * s, r * r
    sig = r2 + a2 * (c * c)
    dlt = r2 - 2.0 * m * r + a2
    r2a2 = r2 + a2
    big_a = r2a2 * r2a2 - a2 * dlt * s2
    sd = sig * dlt
    sig_r, sig_th, dlt_r = 2.0 * r, (-a2) * sin2th, 2.0 * (r - m)
    a_r = 4.0 * r * r2a2 - two_a2 * (r - m) * s2
    a_th = (-a2) * dlt * sin2th
    sd_r, sd_th = sig_r * dlt + sig * dlt_r, sig_th * dlt
    sd2, sig2 = sd * sd, sig * sig
    neg, pos = (-2.0 * m) * a, (2.0 * m) * a
    quotients = [(-big_a, sd), (neg * r, sd), (dlt, sig), (1.0, sig), (dlt - a2 * s2, sd * s2),
                 (-(a_r * sd - big_a * sd_r), sd2), (neg * (sd - r * sd_r), sd2), (dlt_r * sig - dlt * sig_r, sig2),
                 (-sig_r, sig2), (-sig_r, sig2 * s2), (a2 * sd_r, sd2), (-(a_th * sd - big_a * sd_th), sd2),
                 (pos * r * sd_th, sd2), (-dlt * sig_th, sig2), (-sig_th, sig2),
                 (-(sig_th * s2 + sig * sin2th), sig2 * (s2 * s2)), (a2 * sd_th, sd2)]
    return s2, r2, sd, quotients


def _within(x, lo, hi):
    return math.isfinite(x) and 2.0**lo <= abs(x) < 2.0**hi


def test_range_of_the_metric_terms():
    """Wherever the kernel's tests let a state through, no quotient of the metric can overflow, underflow or
    lose its residual: numerators 0 or in [2^-960, 2^960], quotients in [2^-960, 2^960]."""
    rng = random.Random(7)
    seen = 0

    def extreme(lo, hi):
        return 2.0 ** (rng.choice([lo, hi, rng.uniform(lo, hi)]) + rng.choice([0.0, 0.0, 2.0**-40]))

    for _ in range(60000):
        m = min(extreme(-50.0, 60.0), 2.0**60)
        a = rng.choice([0.0, m * rng.uniform(-1.0, 1.0), m * (1.0 - 2.0**-53), -2.0**-120, 2.0**-120,
                        rng.choice([-1.0, 1.0]) * 2.0 ** rng.uniform(-120.0, math.log2(m))])
        if abs(a) >= m:
            continue
        r_plus = m + math.sqrt(m * m - a * a)
        r = rng.choice([m, math.nextafter(m, math.inf), r_plus, math.nextafter(r_plus, math.inf), r_plus * (1.0 + 2.0**-30),
                        m * rng.uniform(1.0, 3.0), extreme(-50.0, 60.0), -extreme(-50.0, 60.0), m * 2.0 ** rng.uniform(0, 40)])
        th = rng.choice([rng.uniform(0.0, math.pi), 0.5 * math.pi, math.pi, 2.0 ** rng.uniform(-60.0, 0.0),
                         math.pi - 2.0 ** rng.uniform(-52.0, 0.0), 0.5 * math.pi + 2.0 ** rng.uniform(-53.0, -1.0),
                         rng.randrange(1, 636) * 0.5 * math.pi])
        s2, r2, sd, quotients = _terms(m, a, r, math.sin(th), math.cos(th), math.sin(2.0 * th))
        if not (_within(s2, -120, 120) and _within(r2, -100, 120) and _within(sd, -200, 240)):
            continue
        seen += 1
        for num, den in quotients:
            assert _within(den, -480, 485)
            if num != 0.0:
                assert _within(num, -960, 960) and _within(num / den, -960, 960), (m, a, r, th, num, den)
    assert seen > 20000


LENGTHS = [0, 1, 6, 7]  # t, r, p_theta, p_phi scale with the mass; theta, phi, p_t, p_r do not


def _run(mass, spin, atol, n):
    cam = K.Camera(radius=1000.0, inclination_deg=77.0, fov=9.0, resolution=n)
    y0 = K.initial_states(cam, K.Spacetime(1.0, spin))
    y0[:, LENGTHS] *= mass
    integ = K.IntegratorOptions(rtol=1e-7, atol=atol, step_size=2.0**-7 * mass, lambda_max=8192.0 * mass,
                                h_min=2.0**-40 * mass)
    term = K.TerminationOptions(horizon_epsilon=2.0**-20 * mass, escape_radius=1000.0 * mass)
    res = K.CudaBackend().integrate_batch(K.Spacetime(mass, spin), y0, integ, term)
    res.Y[:, LENGTHS] /= mass
    return res


@pytest.mark.gpu
@pytest.mark.parametrize("n", [18, 132])  # four lanes per ray, and one
@pytest.mark.parametrize("spin", [0.0, 0.9, 2.0**-60, 2.0**-119, 2.0**-125])
def test_scales_inside_and_outside_the_range_agree(n, spin):
    """Scaling every length by a power of two is exact in every operation: masses within the branch-free
    range, at its ends and beyond, and absolute tolerances below 2^-400 give the same bits."""
    base = _run(1.0, spin, 2.0**-300, n)
    assert np.any(base.state == 1) and np.any(base.state == 2)
    for mass, atol in ((2.0**-50, 2.0**-300), (2.0**-51, 2.0**-300), (2.0**33, 2.0**-300), (2.0**50, 2.0**-300),
                       (2.0**61, 2.0**-300), (1.0, 2.0**-450), (1.0, 2.0**-1070)):
        res = _run(mass, spin, atol, n)
        for name in ("state", "n_steps", "n_rejected", "Y", "max_carter_drift", "max_null_error"):
            assert np.array_equal(getattr(res, name), getattr(base, name)), (mass, atol, name)


@pytest.mark.gpu
def test_a_drift_beyond_the_largest_number_is_infinite():
    y0 = np.tile([0.0, 50.0, 1.2, 0.0, -1e-50, -1e115, 0.0, 3e-50], (3, 1))
    res = K.CudaBackend().integrate_batch(K.Spacetime(1.0, 0.5), y0, K.IntegratorOptions(max_steps=2), K.TerminationOptions())
    assert np.all(np.isposinf(res.max_null_error))

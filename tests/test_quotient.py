"""The reference order's branch-free divisions (``csrc/krr_quotient.cuh``).

On the CPU the algorithm in exact rational arithmetic, every operation rounded once to FP64, against
Python's IEEE division; on the GPU the kernels' branch-free path against their IEEE path through the
backend: scaling every length by a power of two is exact in every operation, and puts the mass
outside the range of the branch-free path.
"""

from __future__ import annotations

import math
import random
from fractions import Fraction

import numpy as np
import pytest

import kerrray_b200 as K


def _fma(a: float, b: float, c: float) -> float:
    return float(Fraction(a) * Fraction(b) + Fraction(c))  # Fraction -> float rounds to nearest even


def _recip(b: float, seed_error: float) -> float:
    y = float(Fraction(1) / Fraction(b) * (1 + Fraction(seed_error)))
    for _ in range(2):
        y = _fma(_fma(-b, y, 1.0), y, y)
    return y


def _shared(a: float, b: float, seed_error: float) -> float:
    y = _recip(b, seed_error)
    e = _fma(-b, y, 1.0)
    q0 = _fma(a, y, a * (e * y))
    return _fma(_fma(-b, q0, a), y, q0)


def _own(a: float, b: float, seed_error: float) -> float:
    y = _recip(b, seed_error)
    q0 = a * y
    q1 = _fma(_fma(-b, q0, a), y, q0)
    return _fma(_fma(-b, q1, a), y, q1)


def _denominators(rng: random.Random):
    for _ in range(60):
        yield rng.uniform(1.0, 2.0)
    for k in range(20):  # next to 1, and the largest fractions the kernels' test lets through
        yield 1.0 + k * 2.0**-52
        yield 2.0 - 2.0**-20 - (k + 1) * 2.0**-52
    yield from (1.0, 1.5, math.sqrt(2.0))


@pytest.mark.parametrize("seed_error", [2.0**-19, -(2.0**-19), 0.0])
def test_quotients_are_correctly_rounded(seed_error):
    rng = random.Random(11)
    for b in _denominators(rng):
        inv = 1.0 / b
        assert _recip(b, seed_error) in (inv, math.nextafter(inv, 0.0), math.nextafter(inv, 2.0))
        numerators = [rng.uniform(1.0, 2.0) for _ in range(6)] + [1.0, math.nextafter(b, 1.0), b, math.nextafter(2.0, 1.0)]
        # numerators that put a/b next to a rounding boundary: a = RN(b m) of a midpoint m
        for _ in range(6):
            m = Fraction(2 * rng.randrange(2**52, 2**53) + 1, 2**53)
            numerators.append(float(Fraction(b) * m))
        for a in numerators:
            for sign in (1.0, -1.0):
                for f in (_shared, _own):
                    assert f(sign * a, b, seed_error) == sign * a / b, (f.__name__, a.hex(), b.hex())
                    assert f(a, sign * b, seed_error) == a / (sign * b)


LENGTHS = [0, 1, 6, 7]  # t, r, p_theta, p_phi scale with the mass; theta, phi, p_t, p_r do not


def _run(mass: float, spin: float, atol: float, events: bool):
    cam = K.Camera(radius=1000.0, inclination_deg=77.0, fov=9.0, resolution=18)
    y0 = K.initial_states(cam, K.Spacetime(1.0, spin))
    y0[:, LENGTHS] *= mass
    integ = K.IntegratorOptions(rtol=1e-7, atol=atol, step_size=2.0**-7 * mass, lambda_max=8192.0 * mass,
                                h_min=2.0**-40 * mass)
    term = K.TerminationOptions(horizon_epsilon=2.0**-20 * mass, escape_radius=1000.0 * mass)
    ev = K.EventOptions(disk_plane=True, r_in=6.0 * mass, r_out=20.0 * mass) if events else None
    res = K.CudaBackend().integrate_batch(K.Spacetime(mass, spin), y0, integ, term, events=ev)
    res.Y[:, LENGTHS] /= mass
    return res


@pytest.mark.gpu
@pytest.mark.parametrize("events", [False, True])
@pytest.mark.parametrize("spin", [0.0, 0.5, 0.998])
def test_branch_free_path_equals_the_ieee_path(spin, events):
    base = _run(1.0, spin, 2.0**-300, events)
    assert np.any(base.state == 1) and np.any(base.state == 2)
    for mass, atol in ((2.0**70, 2.0**-300), (2.0**-70, 2.0**-300), (1.0, 2.0**-450)):
        res = _run(mass, spin, atol, events)
        assert np.array_equal(res.state, base.state) and np.array_equal(res.n_steps, base.n_steps)
        assert np.array_equal(res.n_rejected, base.n_rejected)
        assert np.array_equal(res.Y, base.Y), (mass, atol)
        assert np.array_equal(res.max_carter_drift, base.max_carter_drift)

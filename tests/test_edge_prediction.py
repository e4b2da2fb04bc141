"""The edge bisection's predicted path and spread queue: whatever the prediction, the brackets and
lost-photon counts are the sequential bisection's, bit for bit."""

from __future__ import annotations

import numpy as np
import pytest

import kerrray_b200 as K
from tests.test_gpu_parity import _sequential_bisection

pytestmark = pytest.mark.gpu


def _case(spin, incl, r_o, rtol, n, lo, hi, turn=0.1):
    angles = turn + 2 * np.pi * np.arange(n) / n
    return K.EdgeCase(K.Spacetime(1.0, spin), incl, r_o, rtol, (2 * spin * np.sin(np.deg2rad(incl)), 0.0), angles,
                      np.full(n, lo), np.full(n, hi))


def _check(cases, iterations, precision):
    res, stats = K.bisect_edges(cases, iterations, precision=precision, item_failures=True)
    assert stats["retired"] == sum(c.angles.size for c in cases)
    backend = K.CudaBackend(precision=precision)
    for case, (r_mid, width, fails) in zip(cases, res):
        r2, w2, f2 = _sequential_bisection(case, iterations, backend)
        assert np.array_equal(r2, r_mid) and np.array_equal(w2, width) and np.array_equal(f2, fails)


@pytest.mark.parametrize("precision", ["reference", "fast64", "mixed"])
@pytest.mark.parametrize("lo,hi", [(2.0, 8.0), (6.0, 8.0), (2.0, 3.0), (8.0, 2.0)])
def test_right_and_wrong_predictions(precision, lo, hi):
    """The edge inside the bracket, every photon on one side, and a bracket upside down; beside a case
    whose directions cross the axis (lost photons, never classified)."""
    rtol = 1e-6 if precision == "mixed" else 1e-8
    cases = [_case(0.9, 60.0, 1.0e3, rtol, 7, lo, hi), _case(0.0, 17.0, 1.0e3, 1e-6, 4, lo, hi, turn=np.pi / 2),
             _case(0.99, 85.0, 1.0e3, 1e-5, 5, lo, hi)]
    _check(cases, 36, precision)


@pytest.mark.parametrize("rtol,iterations", [(1e-3, 30), (1e-10, 40), (1e-6, 1), (1e-6, 0)])
def test_short_and_long_chains(rtol, iterations):
    """A prediction too coarse for any chain, chains as long as a path holds, and no halving to look ahead to."""
    _check([_case(0.7, 40.0, 1.0e3, rtol, 3, 2.0, 8.0)], iterations, "fast64")


@pytest.mark.parametrize("n", [1, 2, 1183, 1185, 4736, 4737, 9000])
def test_items_around_the_warps_shares(n):
    """1184 warps at two blocks per SM, 1776 at three: a share of one item, of more, and the other build (above 4736)."""
    half = n // 2
    cases = [_case(0.9, 60.0, 1.0e3, 1e-5, n - half, 2.0, 8.0)]
    if half:
        cases.append(_case(0.5, 17.0, 1.0e3, 1e-6, half, 2.0, 8.0))
    _check(cases, 6, "fast64")


@pytest.mark.parametrize("r_o,lo,hi", [(1.0e3, 2.0, 8.0), (6.0, 0.5, 4.0), (3.0, 0.1, 1.4), (1.0e3, 0.0, 200.0)])
@pytest.mark.parametrize("n", [1, 33, 180])
def test_outcomes_told_ahead(r_o, lo, hi, n):
    """Few items, so that lanes start below photons that still run: from far, from beside the photon orbits
    and inside them (where the radial momentum tells little or the wrong side), and in a wide bracket."""
    for precision, rtol in (("reference", 1e-6), ("fast64", 1e-10), ("mixed", 1e-6)):
        _check([_case(0.9, 60.0, r_o, rtol, n, lo, hi)], 36, precision)

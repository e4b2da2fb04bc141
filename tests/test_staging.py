"""Pageable host arrays through the pinned staging memory: the same bytes as through pinned arrays, at
sizes around its 1 MB slots and beyond its 32 of them."""

from __future__ import annotations

import numpy as np
import pytest
import torch

import kerrray_b200 as K

pytestmark = pytest.mark.gpu

NAMES = ("state", "n_steps", "n_rejected", "lam", "max_null_error", "max_energy_drift", "max_lz_drift", "max_carter_drift")


def _pinned(n):
    t = {"Y": torch.full((n, 8), -7.0, dtype=torch.float64, pin_memory=True)}
    for k in NAMES:
        dtype = torch.int64 if k in ("state", "n_steps", "n_rejected") else torch.float64
        t[k] = torch.full((n,), -7, dtype=dtype, pin_memory=True)
    return {k: v.numpy() for k, v in t.items()} | {"event_Y": None, "event_hit": None}


def _spec(n):
    res = 2 * int(np.ceil(np.sqrt(n) / 2 + 1))
    return K.ImageSpec(K.Spacetime(1.0, 0.9), K.Camera(radius=1000.0, inclination_deg=60.0, fov=8.0, resolution=res),
                       K.IntegratorOptions(rtol=1e-5, atol=1e-7, max_steps=3), K.TerminationOptions(), pixels=(1, n))


# 16,384 rows of Y are one slot; 131,072 values of the other arrays; 600,001 rows take more than 32 slots
# (37 for Y alone) and, above 1.4M, several ranges with copies in both directions.
@pytest.mark.parametrize("n", [1, 16_384, 16_385, 131_073, 600_001, 1_400_003])
def test_pageable_arrays_equal_pinned_ones(n):
    spec = _spec(n)
    y0 = K.initial_states(spec.camera, spec.spacetime)[1:n + 1]
    pinned_y0 = torch.empty((n, 8), dtype=torch.float64, pin_memory=True).numpy()
    pinned_y0[:] = y0
    pageable = K.trace_images([spec], Y0=y0.copy())
    pinned = K.trace_images([spec], Y0=pinned_y0, out=_pinned(n))
    for k in ("Y",) + NAMES:
        assert np.array_equal(pageable.arrays[k], pinned.arrays[k]), k
    assert np.all(pageable.arrays["n_steps"] == 3)
    batch = K.CudaBackend(precision="fast64").integrate_batch(spec.spacetime, y0, spec.integ, spec.term)
    assert np.array_equal(batch.Y, pinned.arrays["Y"]) and np.array_equal(batch.lam, pinned.arrays["lam"])
    for source in (y0.copy(), pinned_y0):  # the last value of the last range
        source[-1, 7] = np.inf
        with pytest.raises(ValueError, match="finite"):
            K.trace_images([spec], Y0=source)
    with pytest.raises(ValueError, match="finite"):
        K.CudaBackend().integrate_batch(spec.spacetime, source, spec.integ, spec.term)

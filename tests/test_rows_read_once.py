"""A host batch whose array is written to by another thread: the rows traced are rows that were checked."""

from __future__ import annotations

import threading

import numpy as np
import pytest
import torch

import kerrray_b200 as K

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("pinned", [False, True])
def test_no_row_is_traced_that_was_not_checked(pinned):
    spec = K.ImageSpec(K.Spacetime(1.0, 0.9), K.Camera(radius=1000.0, inclination_deg=60.0, fov=8.0, resolution=250),
                       K.IntegratorOptions(rtol=1e-5, atol=1e-7, max_steps=2), K.TerminationOptions())
    rows = K.initial_states(spec.camera, spec.spacetime)
    y0 = torch.empty(rows.shape, dtype=torch.float64, pin_memory=pinned).numpy()
    y0[:] = rows
    stop = threading.Event()

    def write():
        while not stop.is_set():
            y0[-1, 1] = np.nan
            y0[-1, 1] = 1000.0

    writer = threading.Thread(target=write)
    writer.start()
    backend = K.CudaBackend(precision="fast64")
    refused = 0
    try:
        for _ in range(80):
            try:
                res = backend.integrate_batch(spec.spacetime, y0, spec.integ, spec.term)
            except ValueError as exc:
                assert "finite" in str(exc)
                refused += 1
            else:
                assert np.all(np.isfinite(res.Y)) and not np.any(res.state == int(K.TerminationState.NUMERICAL_FAILURE))
    finally:
        stop.set()
        writer.join()
    assert np.array_equal(y0[:-1], rows[:-1]) and refused <= 80

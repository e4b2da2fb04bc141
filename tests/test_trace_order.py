"""Host batches traced long photons first: every row is traced once, to the bits of a batch in its own order."""

from __future__ import annotations

import numpy as np
import pytest
import torch

import kerrray_b200 as K

pytestmark = pytest.mark.gpu

NAMES = ("Y", "state", "n_steps", "n_rejected", "lam", "max_null_error", "max_carter_drift")
INTEG = K.IntegratorOptions(rtol=1e-5, atol=1e-7)


def _rows(n, spin=0.9):
    """Random image points, with some rows of other kinds: outgoing, at the axis, and inside the capture radius."""
    st = K.Spacetime(1.0, spin)
    p = np.random.default_rng(n).uniform(-9.0, 9.0, (2, n))
    y = K.initial_states_at(st, 1000.0, 60.0, p[0], p[1])
    y[::97, 5] *= -1.0
    y[1::101, 7] = 0.0
    y[2::103, 1] = 1.2
    return st, y


@pytest.mark.parametrize("precision,blocks", [("fast64", 2), ("mixed", 3), ("reference", 2)])
def test_ordered_batches_equal_their_pieces(precision, blocks):
    """One ray beyond the resident lanes of variant 0 (ordered, one thread per ray), and beyond the rule for that
    (ordered, from the queue); the pieces are small enough to be traced in their own order."""
    lanes = torch.cuda.get_device_properties(0).multi_processor_count * 128 * blocks
    backend = K.CudaBackend(precision=precision)
    for n in (lanes + 1, (3 * lanes // 2 if precision == "reference" else 4 * lanes) + 1):
        st, y = _rows(n)
        whole = backend.integrate_batch(st, y, INTEG, K.TerminationOptions())
        assert set(np.unique(whole.state)) >= {1, 2}
        for lo in range(0, n, lanes):
            part = backend.integrate_batch(st, y[lo:lo + lanes], INTEG, K.TerminationOptions())
            for k in NAMES:
                assert np.array_equal(getattr(whole, k)[lo:lo + lanes], getattr(part, k), equal_nan=True), (n, lo, k)


def test_ordered_images_equal_the_device_sweep():
    specs = [K.ImageSpec(K.Spacetime(1.0, s), K.Camera(radius=1000.0, inclination_deg=i, fov=8.0, resolution=130), INTEG,
                         K.TerminationOptions()) for s, i in ((0.9, 60.0), (0.0, 17.0), (0.99, 85.0))]
    sweep = K.DeviceSweep(specs)  # in the images' order
    sweep.run()
    rows = np.concatenate([K.initial_states(s.camera, s.spacetime) for s in specs])
    for y0 in (None, rows):
        host = K.trace_images(specs, Y0=y0)
        assert host.stats["retired"] == 3 * 130 * 130
        for k in NAMES:
            assert np.array_equal(host.arrays[k], sweep.tensors[k].cpu().numpy()), k
    sweep.close()

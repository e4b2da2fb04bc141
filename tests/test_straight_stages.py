"""The fast64 stages without branches, used at tight tolerances, against the general ones: the same bits,
also where a step turns too far for them and is done over."""

from __future__ import annotations

import numpy as np
import pytest
import torch

import kerrray_b200 as K

pytestmark = pytest.mark.gpu

NAMES = ("Y", "state", "n_steps", "n_rejected", "lam", "max_null_error", "max_carter_drift")


@pytest.mark.parametrize("spin,incl,step", [(0.0, 60.0, 0.01), (0.99, 85.0, 0.01), (0.9, 0.5, 40.0)])
def test_plain_and_queue_agree_at_tight_tolerance(spin, incl, step):
    """One photon per thread takes the straight stages at rtol <= 2e-9, the work queue never does. A
    first step of 40 M and an observer next to the axis make steps of large angles, most of them rejected."""
    spec = K.ImageSpec(K.Spacetime(1.0, spin), K.Camera(radius=30.0, inclination_deg=incl, fov=8.0, resolution=32),
                       K.IntegratorOptions(rtol=2e-9, atol=2e-11, step_size=step), K.TerminationOptions(escape_radius=30.0))
    out = []
    for launch in (K.LaunchConfig(), K.LaunchConfig(refill_threshold=1)):
        sweep = K.DeviceSweep([spec], precision="fast64", launch=launch)
        sweep.run()
        out.append({k: sweep.tensors[k].clone() for k in NAMES})
        sweep.close()
    assert all(torch.equal(out[0][k], out[1][k]) for k in NAMES)
    y0 = K.initial_states(spec.camera, spec.spacetime)
    batch = K.CudaBackend(precision="fast64").integrate_batch(spec.spacetime, y0, spec.integ, spec.term)
    assert np.array_equal(batch.Y, out[0]["Y"].cpu().numpy())


def test_lensing_steps_at_both_sides_of_the_rule():
    """The map's step counts and final angles at the tolerance of the rule equal the trace's, whose queue takes
    the general stages; and so do they just above it."""
    res = 24
    cam = K.Camera(radius=1000.0, inclination_deg=60.0, fov=12.0, resolution=res)
    a, b = (torch.tensor(np.asarray(x).ravel(), device="cuda") for x in cam.pixel_coordinates())
    for rtol in (2e-9, 2.001e-9):
        integ = K.IntegratorOptions(rtol=rtol, atol=1e-2 * rtol)
        m = K.lensing_map(a, b, 0.8, 60.0, integ=integ)
        sweep = K.DeviceSweep([K.ImageSpec(K.Spacetime(1.0, 0.8), cam, integ, K.TerminationOptions())],
                              launch=K.LaunchConfig(refill_threshold=1))
        sweep.run()
        same = m.n_steps == sweep.tensors["n_steps"]  # the camera of the map rounds otherwise: a few rays part
        assert same.double().mean() > 0.98 and torch.equal(m.state, sweep.tensors["state"])
        sweep.close()

"""Four lanes per ray in reference order against one lane per ray: the same bits, with rays missing from
the last groups, rays of every ending, and steps that leave the branch-free range."""

from __future__ import annotations

import numpy as np
import pytest
import torch

import kerrray_b200 as K

pytestmark = pytest.mark.gpu

NAMES = ("Y", "state", "n_steps", "n_rejected", "lam", "max_null_error", "max_energy_drift", "max_lz_drift",
         "max_carter_drift")


def _both(specs, y0=None):
    """The library's launch (four lanes), and one photon per thread as asked for."""
    out = []
    for launch in (K.LaunchConfig(), K.LaunchConfig(plain=True, block=64)):
        sweep = K.DeviceSweep(specs, precision="reference", launch=launch,
                              Y0=None if y0 is None else torch.from_numpy(y0).cuda())
        stats = sweep.run()
        out.append(({k: sweep.tensors[k].cpu().numpy() for k in NAMES}, stats))
        sweep.close()
    for k in NAMES:
        assert np.array_equal(out[0][0][k], out[1][0][k], equal_nan=True), k
    for k in ("retired", "attempts", "accepted", "busy_slots"):
        assert out[0][1][k] == out[1][1][k], k
    return out[0][0]


@pytest.mark.parametrize("n", [1, 7, 8, 9, 31, 33, 2049])
@pytest.mark.parametrize("spin,incl,rtol", [(0.0, 60.0, 1e-6), (0.99, 85.0, 1e-8)])
def test_pixels(n, spin, incl, rtol):
    spec = K.ImageSpec(K.Spacetime(1.0, spin), K.Camera(radius=1000.0, inclination_deg=incl, fov=8.0, resolution=46),
                       K.IntegratorOptions(rtol=rtol, atol=1e-2 * rtol), K.TerminationOptions(), pixels=(40, n))
    _both([spec])


def test_endings_and_careful_steps():
    """Budgets, step caps and minima, axis crossings, outgoing rays, starts inside the capture radius, and first
    steps of 500 M that jump through the horizon."""
    st = K.Spacetime(1.0, 0.9)
    cam = K.Camera(radius=1000.0, inclination_deg=60.0, fov=8.0, resolution=24)
    y0 = K.initial_states(cam, st)
    y0[::7, 5] *= -1.0
    y0[1::11, 7] = 0.0
    y0[2::13, 1] = 1.3
    y0[3::17, 2] = 1e-7
    seen = set()
    for integ in (K.IntegratorOptions(rtol=1e-6, atol=1e-8), K.IntegratorOptions(rtol=1e-6, atol=1e-8, max_steps=30),
                  K.IntegratorOptions(rtol=1e-6, atol=1e-8, lambda_max=990.0), K.IntegratorOptions(rtol=1e-6, atol=1e-8, h_max=3.0),
                  K.IntegratorOptions(rtol=1e-6, atol=1e-8, h_min=1e-2), K.IntegratorOptions(rtol=1e-3, atol=1e-5, step_size=500.0)):
        seen |= set(np.unique(_both([K.ImageSpec(st, cam, integ, K.TerminationOptions())], y0)["state"]))
    assert seen >= {1, 2, 3, 4, 5}
    # out of the branch-free range altogether
    huge = K.Spacetime(2.0**70, 0.9)
    big = y0.copy()
    big[:, [0, 1, 6, 7]] *= 2.0**70
    cam70 = K.Camera(radius=1000.0 * 2.0**70, inclination_deg=60.0, fov=8.0 * 2.0**70, resolution=24)
    integ = K.IntegratorOptions(rtol=1e-6, atol=1e-8, step_size=2.0**64, lambda_max=2.0**84)
    _both([K.ImageSpec(huge, cam70, integ, K.TerminationOptions(escape_radius=1000.0 * 2.0**70))], big)


def test_several_images_and_the_host_batch():
    """Two images of different holes in one warp, and the limit of the rule through the backend."""
    specs = [K.ImageSpec(K.Spacetime(1.0, s), K.Camera(radius=1000.0, inclination_deg=i, fov=8.0, resolution=10),
                         K.IntegratorOptions(rtol=r, atol=1e-2 * r), K.TerminationOptions())
             for s, i, r in ((0.9, 60.0, 1e-6), (0.0, 17.0, 1e-8), (0.99, 85.0, 1e-5))]
    _both(specs)
    limit = torch.cuda.get_device_properties(0).multi_processor_count * 64
    st = K.Spacetime(1.0, 0.9)
    p = np.random.default_rng(3).uniform(-9.0, 9.0, (2, limit + 1))
    y0 = K.initial_states_at(st, 1000.0, 60.0, p[0], p[1])
    integ, term = K.IntegratorOptions(rtol=1e-5, atol=1e-7), K.TerminationOptions()
    whole, at_limit = (K.CudaBackend().integrate_batch(st, y0[:m], integ, term) for m in (limit + 1, limit))
    for k in NAMES:
        assert np.array_equal(getattr(whole, k)[:limit], getattr(at_limit, k)), k

"""The library's own launch shapes: around the photon counts where the rule changes, every photon is
traced once and to the same bits as by the plain kernel."""

from __future__ import annotations

import pytest
import torch

import kerrray_b200 as K

pytestmark = pytest.mark.gpu

NAMES = ("Y", "state", "n_steps", "n_rejected", "lam", "max_null_error", "max_carter_drift")


@pytest.mark.parametrize("precision,layers", [("fast64", 2), ("mixed", 3), ("reference", 2)])
def test_shapes_at_the_rule_s_borders(precision, layers):
    """One block per SM holds SMs x 128 photons; ``layers`` blocks are what variant 0 keeps resident."""
    layer = torch.cuda.get_device_properties(0).multi_processor_count * 128
    for n in (1, layer, layer + 1, layers * layer, layers * layer + 1, layers * layer * 3 // 2, layers * layer * 3 // 2 + 1,
              4 * layers * layer, 4 * layers * layer + 1):
        specs = [K.ImageSpec(K.Spacetime(1.0, 0.9),
                             K.Camera(radius=1000.0, inclination_deg=60.0, fov=8.0, resolution=480),
                             K.IntegratorOptions(rtol=1e-5, atol=1e-7), K.TerminationOptions(), pixels=(3, n))]
        out = []
        for launch in (K.LaunchConfig(), K.LaunchConfig(plain=True, block=64), K.LaunchConfig(refill_threshold=1)):
            sweep = K.DeviceSweep(specs, precision=precision, launch=launch)
            stats = sweep.run()
            assert stats["retired"] == n
            out.append({k: sweep.tensors[k].clone() for k in NAMES})
            sweep.close()
        assert all(torch.equal(out[0][k], other[k]) for k in NAMES for other in out[1:]), n

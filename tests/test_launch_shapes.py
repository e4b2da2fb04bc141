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


@pytest.mark.parametrize("res,retrace,other", [
    (1024, 2, dict(variant=2, refill_threshold=4)),  # three overflowed photons: resumed in place, or by a later kernel
    (1024, 3, dict(variant=2, refill_threshold=4)),
    (300, 2, dict(critical_sms=4)),                  # one critical warp per scheduler, or two
    (300, 3, dict(critical_sms=4, variant=4)),
])
def test_mixed_pipeline_shapes_agree(res, retrace, other):
    spec = K.ImageSpec(K.Spacetime(1.0, 0.99), K.Camera(radius=1000.0, inclination_deg=85.0, fov=8.0, resolution=res),
                       K.IntegratorOptions(rtol=1e-6, atol=1e-8), K.TerminationOptions())
    out = []
    for launch in (K.LaunchConfig(retrace=retrace), K.LaunchConfig(retrace=retrace, **other)):
        sweep = K.DeviceSweep([spec], precision="mixed", launch=launch)
        stats = sweep.run()
        assert stats["retraced"] == stats["critical"] + stats["rechecked"]
        out.append(({k: sweep.tensors[k].clone() for k in NAMES}, stats))
        sweep.close()
    assert all(torch.equal(out[0][0][k], out[1][0][k]) for k in NAMES)
    assert out[0][1]["critical"] == out[1][1]["critical"] and out[0][1]["rechecked"] == out[1][1]["rechecked"]
    if res == 1024 and retrace == 2:  # with the near-edge band the three are traced in FP64
        assert out[0][1]["rechecked"] > 0

"""The work queue's kernels against the plain one, in every form that a launch rule can choose: the same bits."""

from __future__ import annotations

import numpy as np
import pytest
import torch

import kerrray_b200 as K

pytestmark = pytest.mark.gpu

NAMES = ("Y", "state", "n_steps", "n_rejected", "lam", "max_null_error", "max_carter_drift", "event_Y", "event_hit")
DISK = K.EventOptions(disk_plane=True, r_in=6.0, r_out=18.0)


def _spec(res, dtype, method, events, fov=20.0):
    integ = K.IntegratorOptions(method=method, rtol=1e-5, atol=1e-7, dtype=dtype, step_size=2.0 if method == "rk4" else 1e-2,
                                max_steps=700 if method == "rk4" else 100_000)
    term = K.TerminationOptions(horizon_epsilon=1e-3 if dtype == "float32" else 1e-6)
    cam = K.Camera(radius=1000.0, inclination_deg=80.0, fov=fov, resolution=res)
    return K.ImageSpec(K.Spacetime(1.0, 0.9), cam, integ, term, DISK if events else None)


def _assert_same(got, want):
    for name in NAMES:
        a, b = got[name], want[name]
        assert (a is None) == (b is None) and (a is None or np.array_equal(a, b)), name


FORMS = [(p, "float64", m, e) for p in ("reference", "fast64", "mixed") for m in ("rk45", "rk4") for e in (False, True)
         if not (p == "mixed" and m == "rk4")] + [("reference", "float32", m, e) for m in ("rk45", "rk4") for e in (False, True)]


@pytest.mark.parametrize("precision,dtype,method,events", FORMS)
def test_queue_variants_equal_the_plain_kernel(precision, dtype, method, events):
    spec = _spec(48, dtype, method, events)
    plain = K.trace_images([spec], precision=precision, launch=K.LaunchConfig(plain=True)).arrays
    if method == "rk45":
        assert {1, 2} <= set(plain["state"]) and (not events or 0 < plain["event_hit"].sum() < plain["event_hit"].size)
    _assert_same(K.trace_images([spec], precision=precision).arrays, plain)
    for v in K.list_variants(precision, spec.integ, spec.term):
        for launch in (dict(refill_threshold=1), dict(refill_threshold=8), dict(refill_threshold=32, blocks_per_sm=1)):
            cfg = K.LaunchConfig(variant=v["variant"], **launch)
            _assert_same(K.trace_images([spec], precision=precision, launch=cfg).arrays, plain)


@pytest.mark.parametrize("dtype,method,events", [("float32", "rk45", True), ("float32", "rk45", False),
                                                 ("float64", "rk45", True), ("float32", "rk4", False)])
def test_host_batches_beyond_the_plain_limit(dtype, method, events):
    """Reference order, one photon more than one and a half per resident lane: the queue, long photons first."""
    spec = _spec(300, dtype, method, events)
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    v = K.list_variants("reference", spec.integ, spec.term)[0]
    lanes = sms * v["blocks_per_sm"] * v["block"]
    n = lanes + lanes // 2 + 1
    rows = K.initial_states(spec.camera, spec.spacetime)
    assert lanes < n <= len(rows)
    rows = rows[np.random.default_rng(1).permutation(len(rows))[:n]]
    piece = K.ImageSpec(spec.spacetime, spec.camera, spec.integ, spec.term, spec.events, pixels=(0, n))
    plain = K.trace_images([piece], precision="reference", Y0=rows, launch=K.LaunchConfig(plain=True)).arrays
    got = K.CudaBackend().integrate_batch(spec.spacetime, rows, spec.integ, spec.term, events=spec.events)
    for name in NAMES:
        a, b = getattr(got, name), plain[name]
        assert (a is None) == (b is None) and (a is None or np.array_equal(a, b.astype(a.dtype))), name


@pytest.mark.parametrize("method", ["rk45", "rk4"])
@pytest.mark.parametrize("events", [False, True])
@pytest.mark.parametrize("dtype,inside,outside", [
    ("float64", (1.0, 0.5), (2.0**70, 0.5)),              # lengths scaled by 2^70, exact in every operation
    ("float64", (1.0, 2.0**-119), (2.0**70, 2.0**-119)),
    ("float32", (1.0, 2.0**-110), (1.0, 2.0**-125)),      # float32 cannot hold such lengths; a spin below any rounding
])
def test_steps_outside_the_branch_free_range(dtype, inside, outside, method, events):
    """Every step by IEEE division: the same bits."""
    lengths = [0, 1, 6, 7]  # t, r, p_theta, p_phi

    def run(mass, spin):
        y0 = K.initial_states(K.Camera(radius=256.0, inclination_deg=80.0, fov=20.0, resolution=24), K.Spacetime(1.0, inside[1]))
        y0[:, lengths] *= mass
        integ = K.IntegratorOptions(method=method, rtol=2.0**-17, atol=2.0**-120, dtype=dtype, max_steps=2000,
                                    step_size=(0.5 if method == "rk4" else 2.0**-7) * mass, lambda_max=8192.0 * mass,
                                    h_min=2.0**-40 * mass)
        term = K.TerminationOptions(horizon_epsilon=2.0**-10 * mass, escape_radius=256.0 * mass)
        ev = K.EventOptions(disk_plane=True, r_in=6.0 * mass, r_out=18.0 * mass) if events else None
        res = K.CudaBackend().integrate_batch(K.Spacetime(mass, spin), y0, integ, term, events=ev)
        for Y in (res.Y, res.event_Y):
            if Y is not None:
                Y[:, lengths] /= mass
        return res

    base, other = run(*inside), run(*outside)
    assert len(set(base.state)) > 1
    for name in ("Y", "state", "n_steps", "n_rejected", "max_null_error", "max_carter_drift", "event_Y", "event_hit"):
        a, b = getattr(base, name), getattr(other, name)
        assert (a is None) == (b is None) and (a is None or np.array_equal(a, b)), name

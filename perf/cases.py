"""Timed cases of the ray tracer's public entry points, with what each returns in plain 64-bit torch.

A case is a dict of plain values; ``kind`` names the entry point it goes through:

``shadow``   ``compute_shadow`` on the cuda backend: one image, host results (the everyday call);
``rays``     ``trace_rays`` of a host batch of initial states (random image points);
``disk``     ``render_disk``: an image with the disk-plane event, shaded on the device;
``sweep``    ``trace_images`` of many images, host ``Y0`` in and host results out;
``device``   ``DeviceSweep``: many images, or the mixed-precision pipelines, from a captured plan;
``edges``    ``bisect_edges``: the shadow edge by bisection along polar directions;
``lens``     ``LensingFunction``: the lensing map forward, and its gradients backward.

Spins and inclinations are the studies' {0, 0.5, 0.9, 0.99} x {17, 60, 85} degrees and their
neighbourhood: the seed moves both a little and turns the observer in azimuth. The observer stands
at 1000 M (the edge study: 1e5 M), ``atol`` is ``1e-2 rtol`` and the other options are the defaults.
"""

from __future__ import annotations

import math
import random

import numpy as np
import torch

import kerrray_b200 as K

DEG = math.pi / 180.0
R_O, R_EDGE = 1000.0, 1.0e5
SPINS, INCLINATIONS = (0.0, 0.5, 0.9, 0.99), (17.0, 60.0, 85.0)


# ---------------------------------------------------------------------------------------------
# The cases
# ---------------------------------------------------------------------------------------------
def listed() -> list[dict]:
    return [
        # The first thing a user runs: a 64 x 64 shadow at the backend's default precision.
        {"name": "shadow-64", "kind": "shadow", "res": 64, "spin": 0.9, "incl": 60.0, "rtol": 1e-6,
         "precision": "reference", "dtype": "float64"},
        # A publication image at the default precision, tighter tolerance, near-extremal hole seen from the side.
        {"name": "shadow-300-tight", "kind": "shadow", "res": 300, "spin": 0.99, "incl": 85.0, "rtol": 1e-8,
         "precision": "reference", "dtype": "float64"},
        # The reference's throughput benchmark: random image-plane rays at the default rtol 1e-9.
        {"name": "rays-20k", "kind": "rays", "n": 20011, "spin": 0.9, "incl": 60.0, "rtol": 1e-9,
         "precision": "reference", "dtype": "float64"},
        # The float32 working precision, chosen for quick looks at larger batches.
        {"name": "rays-100k-f32", "kind": "rays", "n": 100003, "spin": 0.9, "incl": 60.0, "rtol": 1e-5,
         "precision": "reference", "dtype": "float32"},
        # An accretion disk seen nearly edge-on.
        {"name": "disk-200", "kind": "disk", "res": 200, "spin": 0.9, "incl": 80.0, "rtol": 1e-8,
         "precision": "reference"},
        # A parameter sweep called with host buffers end to end.
        {"name": "sweep-host", "kind": "sweep", "res": 256, "levels": 2, "rtols": 3, "precision": "fast64"},
        # The full sweep with its results kept on the device: 108 images, 12.4M photons.
        {"name": "sweep-device", "kind": "device", "res": 512, "levels": 3, "rtols": 3, "precision": "fast64",
         "retrace": 0},
        # The mixed-precision image whose mask equals the FP64 kernel's ...
        {"name": "mixed-1024", "kind": "device", "res": 1024, "levels": 1, "rtols": 0, "spin": 0.99, "incl": 85.0,
         "precision": "mixed", "retrace": 2},
        # ... and with the near-edge photons' exit directions at FP64 accuracy as well.
        {"name": "mixed-near-640", "kind": "device", "res": 640, "levels": 1, "rtols": 0, "spin": 0.9, "incl": 60.0,
         "precision": "mixed", "retrace": 3},
        # One shadow edge at the default precision: few directions, long chains of halvings.
        {"name": "edge-90", "kind": "edges", "cases": 1, "angles": 90, "rtols": 1, "iterations": 36,
         "precision": "reference"},
        # The edge study's twelve holes at three tolerances in fast64.
        {"name": "edges-study", "kind": "edges", "cases": 12, "angles": 241, "rtols": 3, "iterations": 36,
         "precision": "fast64"},
        # The differentiable lensing map of a 256 x 256 image and its gradients.
        {"name": "lens-256", "kind": "lens", "res": 256, "spin": 0.8, "incl": 60.0, "rtol": 1e-10},
    ]


def _log(rng: random.Random, lo: float, hi: float) -> float:
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng: random.Random) -> dict:
    """One more case of the listed ranges."""
    kind = rng.choice(["shadow", "shadow", "rays", "rays", "disk", "sweep", "device", "mixed", "edges", "edges", "lens"])
    spin = round(rng.choice([0.0, rng.uniform(-0.95, 0.99), rng.uniform(0.5, 0.99)]), 4)
    incl = round(rng.uniform(10.0, 170.0), 2)
    rtol = float("%.3g" % _log(rng, 1e-10, 1e-6))
    precision = rng.choice(["reference", "reference", "fast64", "mixed"])
    if kind == "shadow":
        return {"kind": kind, "res": 2 * round(_log(rng, 16, 200)), "spin": spin, "incl": incl, "rtol": rtol,
                "precision": precision if rtol >= 1e-8 or precision != "mixed" else "fast64", "dtype": "float64"}
    if kind == "rays":
        f32 = rng.random() < 0.25
        return {"kind": kind, "n": int(_log(rng, 100, 150000)), "spin": spin, "incl": incl,
                "rtol": float("%.3g" % _log(rng, 1e-6, 1e-5)) if f32 else rtol,
                "precision": "reference" if f32 or precision == "mixed" else precision,
                "dtype": "float32" if f32 else "float64"}
    if kind == "disk":
        return {"kind": kind, "res": 2 * round(_log(rng, 24, 150)), "spin": spin, "incl": round(rng.uniform(15.0, 85.0), 2),
                "rtol": rtol, "precision": rng.choice(["reference", "fast64"])}
    if kind == "sweep":
        return {"kind": kind, "res": 8 * round(_log(rng, 8, 40)), "levels": rng.choice([1, 2, 3]),
                "rtols": rng.choice([1, 2, 3]), "precision": "fast64"}
    if kind == "device":
        return {"kind": kind, "res": 8 * round(_log(rng, 10, 60)), "levels": rng.choice([1, 2, 3]),
                "rtols": rng.choice([1, 2, 3]), "precision": "fast64", "retrace": 0}
    if kind == "mixed":
        return {"kind": "device", "res": 2 * round(_log(rng, 96, 700)), "levels": 1, "rtols": 0,
                "spin": round(rng.uniform(0.3, 0.99), 4), "incl": incl, "precision": "mixed",
                "retrace": rng.choice([0, 1, 2, 2, 3, 3])}
    if kind == "edges":
        if rng.random() < 0.5:
            return {"kind": kind, "cases": rng.choice([1, 1, 3]), "angles": round(_log(rng, 16, 120)),
                    "rtols": rng.choice([1, 2]), "iterations": rng.choice([20, 24, 30]), "precision": "reference"}
        return {"kind": kind, "cases": rng.choice([1, 3, 12]), "angles": round(_log(rng, 16, 240)),
                "rtols": rng.choice([1, 2, 3]), "iterations": rng.choice([20, 30, 36]), "precision": "fast64"}
    return {"kind": "lens", "res": 2 * round(_log(rng, 16, 120)), "spin": round(rng.uniform(0.1, 0.95), 4),
            "incl": round(rng.uniform(20.0, 80.0), 2), "rtol": rng.choice([1e-8, 1e-9, 1e-10])}


# ---------------------------------------------------------------------------------------------
# What a program holds before the call
# ---------------------------------------------------------------------------------------------
def _near(rng: random.Random, spin: float, incl: float) -> tuple[float, float, float]:
    """Spin, inclination and azimuth of the seed's observer: a little off the case's (0 stays 0)."""
    s = 0.0 if spin == 0.0 else max(-0.995, min(0.995, spin + rng.uniform(-0.004, 0.004)))
    return s, incl + rng.uniform(-0.5, 0.5), rng.uniform(0.0, 360.0)


def _options(case: dict, rtol: float):
    integ = K.IntegratorOptions(method="rk45", rtol=rtol, atol=1e-2 * rtol, dtype=case.get("dtype", "float64"))
    # float32 cannot resolve the default capture margin next to the horizon
    eps = 1e-3 if case.get("dtype") == "float32" else 1e-6
    return integ, K.TerminationOptions(horizon_epsilon=eps)


def _rtols(case: dict) -> list[float]:
    return [1e-6, 1e-8, 1e-10][: case["rtols"]] or [1e-6]


def _observers(case: dict, seed: int) -> list[dict]:
    """The images (or edge cases) of a case: spin, inclination, azimuth, tolerance, pixels a side."""
    rng = random.Random("%s observers" % seed)
    if case["kind"] in ("sweep", "device") and "spin" not in case:
        combos = [(s, i) for s in SPINS for i in INCLINATIONS]
    elif case["kind"] == "edges":
        combos = {1: [(0.9, 60.0)], 3: [(0.5, 17.0), (0.9, 60.0), (0.99, 85.0)],
                  12: [(s, i) for s in SPINS for i in INCLINATIONS]}[case["cases"]]
    else:
        combos = [(case["spin"], case["incl"])]
    out = []
    for level in range(case.get("levels", 1)):
        for s, i in combos:
            for rtol in (_rtols(case) if "rtols" in case else [case["rtol"]]):
                spin, incl, phi = _near(rng, s, i)
                out.append({"spin": spin, "incl": incl, "phi": phi, "rtol": rtol, "res": case.get("res", 0) >> level & ~1})
    return out


def _centre(x: dict) -> tuple[float, float]:
    """Near the shadow's centre: frame dragging displaces it by about 2 s sin(i)."""
    return 2.0 * x["spin"] * math.sin(x["incl"] * DEG), 0.0


def _angles(case: dict, seed: int) -> np.ndarray:
    """Uniformly spaced polar directions, turned by the seed."""
    n = case["angles"]
    return (np.arange(n) + random.Random("%s angles" % seed).random()) * (2.0 * math.pi / n)


def _grid(res: int, fov: float, device) -> tuple[torch.Tensor, torch.Tensor]:
    c = fov * (2.0 * torch.arange(res, dtype=torch.float64, device=device) + 1.0 - res) / res
    return c.repeat(res), (-c).repeat_interleave(res)


def _points(case: dict, seed: int) -> tuple[torch.Tensor, torch.Tensor]:
    """Random image points of a ray batch, uniform over +-12 M."""
    g = torch.Generator(device="cuda").manual_seed(int(seed))
    p = 24.0 * torch.rand((2, case["n"]), dtype=torch.float64, device="cuda", generator=g) - 12.0
    return p[0], p[1]


def _lens_points(case: dict, seed: int) -> tuple[torch.Tensor, torch.Tensor]:
    """Pixels of a +-12 M image that lie outside the shadow, moved within their cells by the seed."""
    a, b = _grid(case["res"], 12.0, "cuda")
    cell = 24.0 / case["res"]
    keep = torch.hypot(a - _centre(case)[0], b) > 5.6 + 0.75 * cell  # the shadow reaches 5.2 M from its centre
    a, b = a[keep], b[keep]
    g = torch.Generator(device="cuda").manual_seed(int(seed))
    move = cell * (torch.rand((2, a.numel()), dtype=a.dtype, device="cuda", generator=g) - 0.5)
    return a + move[0], b + move[1]


def prepare(case: dict, seed: int) -> dict:
    kind, obs = case["kind"], _observers(case, seed)
    o = obs[0]
    state: dict = {"case": case}
    if kind in ("shadow", "rays", "disk"):
        state["st"] = K.Spacetime(1.0, o["spin"])
        state["backend"] = K.CudaBackend(precision=case["precision"])
        state["options"] = _options(case, o["rtol"])
        if kind == "rays":
            y0, _, _ = _camera(o["spin"], o["incl"] * DEG, R_O, o["phi"] * DEG, *_points(case, seed))
            state["Y0"] = y0.t().contiguous().cpu().numpy()
        else:
            fov = 8.0 if kind == "shadow" else 20.0
            state["cam"] = K.Camera(radius=R_O, inclination_deg=o["incl"], phi_deg=o["phi"], fov=fov,
                                    resolution=case["res"])
        if kind == "disk":
            state["disk"] = K.DiskModel.for_spacetime(state["st"], r_out=18.0)
    elif kind in ("sweep", "device"):
        specs = [K.ImageSpec(K.Spacetime(1.0, x["spin"]),
                             K.Camera(radius=R_O, inclination_deg=x["incl"], phi_deg=x["phi"], fov=8.0,
                                      resolution=x["res"]), *_options(case, x["rtol"])) for x in obs]
        specs = [specs[k] for k in K.order_by_cost(specs)]
        if kind == "sweep":
            state["specs"] = specs
            state["Y0"] = np.concatenate([K.initial_states(s.camera, s.spacetime) for s in specs])
        else:
            state["sweep"] = K.DeviceSweep(specs, precision=case["precision"],
                                           launch=K.LaunchConfig(retrace=case["retrace"]))
    elif kind == "edges":
        angles = _angles(case, seed)
        lo, hi = np.full(angles.size, 2.0), np.full(angles.size, 8.0)
        state["cases"] = [K.EdgeCase(K.Spacetime(1.0, x["spin"]), x["incl"], R_EDGE, x["rtol"], _centre(x), angles, lo, hi)
                          for x in obs]
    else:
        state["alpha"], state["beta"] = _lens_points(case, seed)
        for name in ("alpha", "beta"):
            state[name].requires_grad_(True)
        state["spin"] = torch.tensor(o["spin"], dtype=torch.float64, device="cuda", requires_grad=True)
        state["incl"] = torch.tensor(o["incl"], dtype=torch.float64, device="cuda", requires_grad=True)
        state["integ"] = _options(case, o["rtol"])[0]
        g = torch.Generator(device="cuda").manual_seed(int(seed) + 1)
        n = state["alpha"].numel()
        state["weights"] = [torch.randn(n, dtype=torch.float64, device="cuda", generator=g) for _ in range(2)]
    return state


_FIELDS = ("Y", "state", "n_steps", "n_rejected", "lam", "max_null_error", "max_energy_drift", "max_lz_drift",
           "max_carter_drift")


def run(state: dict):
    case = state["case"]
    kind = case["kind"]
    if kind == "shadow":
        image = K.compute_shadow(state["st"], state["cam"], *state["options"], backend=state["backend"])
        return {n: getattr(image.result, n) for n in _FIELDS}
    if kind == "rays":
        res = K.trace_rays(state["st"], state["Y0"], *state["options"], backend=state["backend"])
        return {n: getattr(res, n) for n in _FIELDS}
    if kind == "disk":
        image = K.render_disk(state["st"], state["cam"], *state["options"], state["disk"], backend=state["backend"])
        out = {n: getattr(image.result, n) for n in _FIELDS}
        return out | {n: getattr(image, n) for n in ("intensity", "g", "hit", "r_hit", "hit_states")}
    if kind == "sweep":
        return {n: v for n, v in K.trace_images(state["specs"], precision=case["precision"], Y0=state["Y0"]).arrays.items()
                if v is not None}
    if kind == "device":
        state["sweep"].run(stats=False)
        return dict(state["sweep"].tensors)
    if kind == "edges":
        results, _ = K.bisect_edges(state["cases"], case["iterations"], precision=case["precision"])
        return {"r_mid": np.concatenate([r[0] for r in results]), "width": np.concatenate([r[1] for r in results]),
                "failures": np.array([r[2] for r in results])}
    theta, phi = K.LensingFunction.apply(state["alpha"], state["beta"], state["spin"], state["incl"], integ=state["integ"])
    wt, wp = state["weights"]
    grads = torch.autograd.grad([theta, phi], [state["alpha"], state["beta"], state["spin"], state["incl"]], [wt, wp])
    return {"theta": theta, "phi": phi, "d_alpha": grads[0], "d_beta": grads[1], "d_spin": grads[2], "d_incl": grads[3]}


def _photons(case: dict) -> int:
    if case["kind"] == "rays":
        return case["n"]
    if case["kind"] == "edges":
        return case["cases"] * case["rtols"] * case["angles"] * case["iterations"]
    images = sum((case["res"] >> k & ~1) ** 2 for k in range(case.get("levels", 1)))
    if case["kind"] in ("sweep", "device") and "spin" not in case:
        images *= len(SPINS) * len(INCLINATIONS) * len(_rtols(case))
    return int(0.72 * images) if case["kind"] == "lens" else images


def work(case: dict) -> dict:
    """Result rows written (and host states read); 1210 operations per Dormand-Prince attempt, whose
    number per photon grows by about 1.76 for each two decades of tolerance."""
    n = _photons(case)
    rtols = _rtols(case) if "rtols" in case else [case["rtol"]]
    attempts = sum(140.0 * 1.76 ** (math.log10(1e-6 / r) / 2.0) for r in rtols) / len(rtols)
    if case["kind"] == "edges":  # results per direction, not per photon; rays from 1e5 M, all next to the edge
        return {"bytes": 24.0 * n / case["iterations"], "flops": 1210.0 * n * 1.3 * attempts}
    if case["kind"] == "lens":  # the map and its Jacobian; the reverse sweep is twice the forward step
        return {"bytes": (16.0 + 16.0 + 64.0) * n, "flops": 1210.0 * n * (attempts + 2.0 * 0.7 * attempts)}
    per = 128 + (64 if case["kind"] in ("rays", "sweep") else 0) + (105 if case["kind"] == "disk" else 0)
    return {"bytes": float(per) * n, "flops": 1210.0 * n * attempts}


# ---------------------------------------------------------------------------------------------
# The same results in plain 64-bit torch
# ---------------------------------------------------------------------------------------------
def _camera(spin, incl, r, phi, alpha, beta):
    """Backward null states (8, n) at image points, mass 1: the projected local momentum, reversed.

    Returns the states and sin, cos of the observer's polar angle. All arguments may be complex."""
    one = alpha * 0.0 + 1.0
    a, th = spin * one, incl * one
    s, c = torch.sin(th), torch.cos(th)
    s2 = s * s
    sig, dlt = r * r + a * a * c * c, r * r - 2.0 * r + a * a
    g_tt, g_tp = -(1.0 - 2.0 * r / sig), -2.0 * a * r * s2 / sig
    g_rr, g_pp = sig / dlt, (r * r + a * a + 2.0 * a * a * r * s2 / sig) * s2
    omega, lapse = -g_tp / g_pp, torch.sqrt(g_tp * g_tp / g_pp - g_tt)
    p1 = torch.sqrt(1.0 - (alpha * alpha + beta * beta) / (r * r))
    u0, u3 = 1.0 / lapse, omega / lapse - alpha / r / torch.sqrt(g_pp)
    y = [0.0 * one, r * one, th, phi * one, -(u0 * g_tt + u3 * g_tp), -p1 * torch.sqrt(g_rr),
         -(beta / r) * torch.sqrt(sig), -(u0 * g_tp + u3 * g_pp)]
    return torch.stack(y), s, c


def _rhs(y, pt, pph, a, axis):
    """Hamilton's equations for (t, r, theta, phi, p_r, p_theta) in Carter's separated form."""
    r, th, pr, pth = y[1], y[2], y[4], y[5]
    s, c = torch.sin(th), torch.cos(th)
    e, r2a2 = -pt, r * r + a * a
    dlt, sig = r * r - 2.0 * r + a * a, r * r + a * a * c * c
    k = r2a2 * e - a * pph
    kd = k / dlt
    inv = torch.where(axis, torch.zeros_like(s), 1.0 / s)
    lis = pph * inv
    v = lis - a * e * s
    two_h = (v * v - k * kd + dlt * pr * pr + pth * pth) / sig
    return torch.stack([(a * s * v + kd * r2a2) / sig, dlt * pr / sig, pth / sig, (a * kd + lis * inv - a * e) / sig,
                        (r * two_h - (r - 1.0) * pr * pr - kd * (kd * (r - 1.0) - 2.0 * e * r)) / sig,
                        c * (v * (lis * inv + a * e) - a * a * s * two_h) / sig])


_A = ((1 / 5,), (3 / 40, 9 / 40), (44 / 45, -56 / 15, 32 / 9),
      (19372 / 6561, -25360 / 2187, 64448 / 6561, -212 / 729),
      (9017 / 3168, -355 / 33, 46732 / 5247, 49 / 176, -5103 / 18656))
_B = (35 / 384, 0.0, 500 / 1113, 125 / 192, -2187 / 6784, 11 / 84)
_BH = (5179 / 57600, 0.0, 7571 / 16695, 393 / 640, -92097 / 339200, 187 / 2100, 1 / 40)


def _step(y, f, h, pt, pph, a, axis):
    """One Dormand-Prince step: the new state, its right-hand side, the embedded error."""
    ks = [f]
    for row in _A:
        ks.append(_rhs(y + h * sum(w * k for w, k in zip(row, ks)), pt, pph, a, axis))
    yn = y + h * sum(w * k for w, k in zip(_B, ks) if w)
    ks.append(_rhs(yn, pt, pph, a, axis))
    err = h * sum((_BH[j] - (_B[j] if j < 6 else 0.0)) * ks[j] for j in (0, 2, 3, 4, 5, 6))
    return yn, ks[-1], err


def _trace(y0, a, rtol, r_cap, r_esc, lam_max=1.0e4, max_steps=100_000, disk=None, record=None):
    """Adaptive integration of the states y0 (8, n) with per-ray a, rtol, r_cap; (Y, state, lam, events).

    ``record`` (a list) receives each accepted step of the batch as (rays, state before, length)."""
    n, dev = y0.shape[1], y0.device
    full = lambda x: x if torch.is_tensor(x) else torch.full((n,), float(x), dtype=torch.float64, device=dev)  # noqa: E731
    Y, lam_out = y0.clone(), torch.zeros(n, dtype=torch.float64, device=dev)
    code_out = torch.zeros(n, dtype=torch.int64, device=dev)
    ev_Y, ev_hit = torch.zeros_like(y0), torch.zeros(n, dtype=torch.bool, device=dev)
    idx = torch.arange(n, device=dev)
    y, pt, pph = y0[[0, 1, 2, 3, 5, 6]].clone(), y0[4], y0[7]
    a, rtol, r_cap = full(a), full(rtol), full(r_cap)
    axis = pph == 0.0
    f = _rhs(y, pt, pph, a, axis)
    h, lam = torch.full_like(pt, 0.01), torch.zeros_like(pt)
    steps, after_rejection = torch.zeros_like(idx), torch.zeros_like(axis)
    code = torch.zeros_like(idx)
    tries = 0
    while idx.numel():
        remaining = lam_max - lam
        last = h >= remaining
        he = torch.where(last, remaining, h)
        yn, fn, err = _step(y, f, he, pt, pph, a, axis)
        scale = 1e-2 * rtol + rtol * torch.maximum(y.abs(), yn.abs())
        en2 = (err / scale).square().sum(0) / 8.0
        finite = torch.isfinite(en2) & torch.isfinite(yn).all(0) & torch.isfinite(fn).all(0)
        ok = finite & (en2 <= 1.0) & (code == 0)
        factor = torch.where(en2 == 0.0, torch.full_like(en2, 5.0), (0.9 * en2 ** -0.1).clamp(0.2, 5.0))
        factor = torch.where(after_rejection, factor.clamp(max=1.0), factor)
        if record is not None:
            rays = ok.nonzero()[:, 0]
            record.append((idx[rays], y[:, rays], he[rays]))
        h = torch.where(ok & last, h, he * factor)
        after_rejection = ~ok
        y_old, lam_old = y, lam
        y, f = torch.where(ok, yn, y), torch.where(ok, fn, f)
        lam = torch.where(ok, torch.where(last, torch.full_like(lam, lam_max), lam + he), lam)
        steps = steps + ok
        # the classification in its order of priority, lowest first
        new = torch.zeros_like(code)
        new = torch.where(ok & ((lam >= lam_max) | (steps >= max_steps)), 3, new)
        new = torch.where(ok & (y[1] >= r_esc) & (f[1] > 0.0), 1, new)
        new = torch.where(ok & (y[1] <= r_cap), 2, new)
        off = (y[1] < 0.0) | (y[2] < -1e-9) | (y[2] > math.pi + 1e-9) | (~axis & (torch.sin(y[2]).abs() < 1e-12))
        new = torch.where(ok & off, 5, new)
        new = torch.where(~finite | (h < 1e-12), 4, new)
        if disk is not None:
            lo, hi = y_old[2] - 0.5 * math.pi, y[2] - 0.5 * math.pi
            w = torch.where(ok, -lo / (hi - lo), torch.zeros_like(lo))
            at = y_old + w * (y - y_old)
            at[2] = 0.5 * math.pi
            hit = ok & (code == 0) & (lo * hi < 0.0) & (at[1] >= disk[0]) & (at[1] <= disk[1])
            y, lam = torch.where(hit, at, y), torch.where(hit, lam_old + w * he, lam)
            new = torch.where(hit, 6, new)
            rays = hit.nonzero()[:, 0]
            if rays.numel():
                ev_hit[idx[rays]] = True
                ev_Y[:, idx[rays]] = torch.stack([at[0], at[1], at[2], at[3], pt, at[4], at[5], pph])[:, rays]
        code = torch.where(code == 0, new, code)
        tries += 1
        if tries % 16 == 0 or record is not None:  # write out the rays that ended, go on with the others
            done = code != 0
            if bool(done.any()):
                rays = done.nonzero()[:, 0]
                Y[:, idx[rays]] = torch.stack([y[0], y[1], y[2], y[3], pt, y[4], y[5], pph])[:, rays]
                lam_out[idx[rays]], code_out[idx[rays]] = lam[rays], code[rays]
                go = (~done).nonzero()[:, 0]
                idx, pt, pph, a, rtol, r_cap, axis, h, lam, steps, after_rejection, code = (
                    x[go] for x in (idx, pt, pph, a, rtol, r_cap, axis, h, lam, steps, after_rejection, code))
                y, f = y[:, go], f[:, go]
        ended = code != 0  # an ended ray waits unchanged for the next write-out
        h = torch.where(ended, torch.full_like(h, 1e-3), h)
    return Y, code_out, lam_out, ev_Y, ev_hit


def _capture(spin: float, eps: float = 1e-6) -> float:
    return 1.0 + math.sqrt(1.0 - spin * spin) + eps


def _rows(Y, code, lam) -> dict:
    """Outputs in the order of a batch result; whole numbers and round-off maxima have no exact value."""
    del code
    return {n: None for n in _FIELDS} | {"Y": Y.t().contiguous(), "lam": lam}


def _exact_images(case: dict, seed: int):
    obs = _observers(case, seed)
    eps = 1e-3 if case.get("dtype") == "float32" else 1e-6
    if case["kind"] in ("sweep", "device"):
        obs = sorted(obs, key=lambda x: -(x["res"] ** 2 * (1.0 / x["rtol"]) ** 0.2))
    parts, a, rtol, cap = [], [], [], []
    for x in obs:
        pts = _points(case, seed) if case["kind"] == "rays" else _grid(x["res"], 20.0 if case["kind"] == "disk" else 8.0, "cuda")
        y0 = _camera(x["spin"], x["incl"] * DEG, R_O, x["phi"] * DEG, *pts)[0]
        parts.append(y0)
        for to, v in ((a, x["spin"]), (rtol, x["rtol"]), (cap, _capture(x["spin"], eps))):
            to.append(torch.full((y0.shape[1],), v, dtype=torch.float64, device="cuda"))
    disk = None
    if case["kind"] == "disk":
        st = obs[0]["spin"]
        disk = (_isco(st), 18.0)
    Y, code, lam, ev_Y, hit = _trace(torch.cat(parts, 1), torch.cat(a), torch.cat(rtol), torch.cat(cap), R_O, disk=disk)
    out = _rows(Y, code, lam)
    if case["kind"] == "disk":
        out |= _shade(obs[0]["spin"], disk[0], ev_Y, hit, case["res"])
    return out


def _isco(spin: float) -> float:
    """Bardeen, Press & Teukolsky 1972, prograde with the hole's own sense of rotation."""
    s = abs(spin)
    z1 = 1.0 + (1.0 - s * s) ** (1 / 3) * ((1.0 + s) ** (1 / 3) + (1.0 - s) ** (1 / 3))
    z2 = math.sqrt(3.0 * s * s + z1 * z1)
    return 3.0 + z2 - math.sqrt((3.0 - z1) * (3.0 + z1 + 2.0 * z2))


def _shade(spin: float, r_in: float, ev_Y, hit, res: int) -> dict:
    r, a = ev_Y[1].clamp(min=1.0), spin
    om = (-1.0 if a < 0.0 else 1.0) / (r * torch.sqrt(r) + abs(a))
    norm = (1.0 - 2.0 / r) + 4.0 * a / r * om - om * om * (r * r + a * a + 2.0 * a * a / r)
    ut = 1.0 / torch.sqrt(norm)
    g = ev_Y[4] / (ev_Y[4] * ut + ev_Y[7] * om * ut)
    nan = torch.full_like(g, math.nan)
    shape = lambda x: torch.where(hit, x, nan).reshape(res, res)  # noqa: E731
    intensity = torch.where(hit, (r / r_in) ** -3.0 * g**4, torch.zeros_like(g)).reshape(res, res)
    states = torch.where(hit, ev_Y, torch.full_like(ev_Y, math.nan)).t().reshape(res, res, 8)
    return {"intensity": intensity, "g": shape(g), "hit": None, "r_hit": shape(ev_Y[1]), "hit_states": states}


def _exact_edges(case: dict, seed: int):
    """Bisection five halvings at a time: the 31 midpoints any outcome could lead to, traced together."""
    obs, angles = _observers(case, seed), torch.tensor(_angles(case, seed), device="cuda")
    per = angles.numel()
    each = lambda v: torch.tensor([x[v] for x in obs], dtype=torch.float64, device="cuda").repeat_interleave(per)  # noqa: E731
    spin, rtol, incl = each("spin"), each("rtol"), each("incl") * DEG
    cap = torch.tensor([_capture(x["spin"]) for x in obs], dtype=torch.float64, device="cuda").repeat_interleave(per)
    ca, cb = (torch.tensor([_centre(x)[k] for x in obs], dtype=torch.float64, device="cuda").repeat_interleave(per)
              for k in (0, 1))
    cos, sin = torch.cos(angles).repeat(len(obs)), torch.sin(angles).repeat(len(obs))
    lo, hi = torch.full_like(spin, 2.0), torch.full_like(spin, 8.0)
    left = case["iterations"]
    while left:
        depth = min(5, left)
        los, his, mids = [lo], [hi], []
        for node in range(2**depth - 1):  # heap order: children 2k+1 (captured) and 2k+2 (escaped)
            mids.append(0.5 * (los[node] + his[node]))
            los += [mids[node], los[node]]
            his += [his[node], mids[node]]
        mid = torch.stack(mids)
        al, be = ca + mid * cos, cb + mid * sin
        wide = lambda v: v.expand(mid.shape).reshape(-1)  # noqa: E731
        y0 = _camera(wide(spin), wide(incl), R_EDGE, 0.0, al.reshape(-1), be.reshape(-1))[0]
        code = _trace(y0, wide(spin), wide(rtol), wide(cap), R_EDGE, 4.0 * R_EDGE, 2_000_000)[1]
        out = (code == 1).reshape(mid.shape)
        node = torch.zeros_like(lo, dtype=torch.int64)
        for _ in range(depth):
            node = 2 * node + 1 + out.gather(0, node[None])[0].to(torch.int64)
        lo, hi = torch.stack(los).gather(0, node[None])[0], torch.stack(his).gather(0, node[None])[0]
        left -= depth
    return {"r_mid": 0.5 * (lo + hi), "width": None, "failures": None}


def _exact_lens(case: dict, seed: int):
    """The recorded step sequence in complex arithmetic: derivatives as Im / eps, to machine precision."""
    o = _observers(case, seed)[0]
    alpha, beta = _lens_points(case, seed)
    n, eps = alpha.numel(), 1e-40
    y0 = _camera(o["spin"], o["incl"] * DEG, R_O, 0.0, alpha, beta)[0]
    record: list = []
    cap = _capture(o["spin"])
    _, code, _, _, _ = _trace(y0, o["spin"], o["rtol"], cap, R_O, record=record)
    # The steps of ray i in order; its last one is shortened to end on the surface.
    count = torch.zeros(n, dtype=torch.int64, device="cuda")
    for rays, _, _ in record:
        count[rays] += 1
    H = torch.zeros((int(count.max()), n), dtype=torch.float64, device="cuda")
    before, filled = torch.zeros((6, n), dtype=torch.float64, device="cuda"), torch.zeros_like(count)
    for rays, y, h in record:
        H[filled[rays], rays] = h
        before[:, rays] = y
        filled[rays] += 1
    rs = torch.where(code == 1, R_O, cap)
    pt, pph, spin = y0[4], y0[7], torch.full_like(alpha, o["spin"])
    axis = pph == 0.0
    h_last = H.gather(0, (count - 1).clamp(min=0)[None])[0]
    f0 = _rhs(before, pt, pph, spin, axis)
    yn, fn, _ = _step(before, f0, h_last, pt, pph, spin, axis)
    h = h_last - (yn[1] - rs) / fn[1]
    for it in range(4):
        yn, fn, _ = _step(before, f0, h, pt, pph, spin, axis)
        if it < 3:
            h = h - (yn[1] - rs) / fn[1]
    H.scatter_(0, (count - 1).clamp(min=0)[None], h[None])
    tilt = lambda x, k: torch.stack([x + (1j * eps if j == k else 0j) for j in range(4)]).reshape(-1)  # noqa: E731
    al, be, sp = tilt(alpha, 0), tilt(beta, 1), tilt(spin, 2)
    y8 = _camera(sp, tilt(torch.full_like(alpha, o["incl"] * DEG), 3), R_O, 0.0, al, be)[0]
    y, pt, pph, axis = y8[[0, 1, 2, 3, 5, 6]], y8[4], y8[7], axis.repeat(4)
    f = _rhs(y, pt, pph, sp, axis)
    for k in range(H.shape[0]):
        live = (k < count).repeat(4)
        yn, fn, _ = _step(y, f, H[k].repeat(4), pt, pph, sp, axis)
        y, f = torch.where(live, yn, y), torch.where(live, fn, f)
    surface = rs.repeat(4).to(y.dtype)
    dr = (y[1] - surface) / f[1]
    th, ph = (y[2] - f[2] * dr).reshape(4, n), (y[3] - f[3] * dr).reshape(4, n)
    g = torch.Generator(device="cuda").manual_seed(int(seed) + 1)
    wt, wp = (torch.randn(n, dtype=torch.float64, device="cuda", generator=g) for _ in range(2))
    grad = wt * th.imag / eps + wp * ph.imag / eps
    return {"theta": th[0].real, "phi": ph[0].real, "d_alpha": grad[0], "d_beta": grad[1], "d_spin": grad[2].sum(),
            "d_incl": grad[3].sum() * DEG}


def exact(case: dict, seed: int):
    """What :func:`run` returns, by the same adaptive scheme in plain 64-bit torch (no code of the package).

    A float32 run has no such value: its rounding decides which trial steps are rejected, so it ends its
    rays at other points of the same orbits."""
    if case.get("dtype") == "float32":
        return None
    if case["kind"] == "lens":
        return _exact_lens(case, seed)
    if case["kind"] == "edges":
        return _exact_edges(case, seed) if _photons(case) <= 400_000 else None
    return _exact_images(case, seed) if _photons(case) <= 2_500_000 else None

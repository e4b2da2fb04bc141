"""``krr_trace_images_noalloc`` rejects what is wrong with its arguments before it looks for a device (CPU)."""

from __future__ import annotations

import ctypes

import pytest

import kerrray_b200 as K
from kerrray_b200 import _lib
from kerrray_b200.build import build


@pytest.mark.parametrize("precision", ["reference", "fast64", "mixed"])
@pytest.mark.parametrize("device", [0, 977])
def test_variant_is_checked_before_the_device(precision, device):
    build()
    spec = K.ImageSpec(K.Spacetime(1.0, 0.9), K.Camera(radius=1000.0, inclination_deg=60.0, fov=8.0, resolution=2),
                       K.IntegratorOptions(), K.TerminationOptions())
    images = (_lib.KrrImage * 1)(spec.as_struct())
    out = _lib.KrrResult(Y=8, state=8)  # not looked at
    launch = _lib.KrrLaunch(precision=_lib.PRECISIONS[precision], variant=99)
    rc = _lib.lib().krr_trace_images_noalloc(device, images, 1, None, ctypes.byref(launch), ctypes.byref(out), None, None)
    assert rc == _lib.KRR_ERR_INVALID and "variant 99 out of range" in _lib.last_error()

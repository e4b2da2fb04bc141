"""``krr_integrate_batch_device`` around the counts where its launch changes: the host entry point's results."""

from __future__ import annotations

import ctypes

import numpy as np
import pytest
import torch

import kerrray_b200 as K
from kerrray_b200 import _lib

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["reference", "fast64", "mixed"])
def test_device_entry_point_equals_the_host_one(precision):
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    spec = K.ImageSpec(K.Spacetime(1.0, 0.9), K.Camera(radius=1000.0, inclination_deg=60.0, fov=8.0, resolution=200),
                       K.IntegratorOptions(rtol=1e-5, atol=1e-7), K.TerminationOptions())
    rows = K.initial_states(spec.camera, spec.spacetime)
    assert len(rows) > 256 * sms
    host = K.CudaBackend(precision=precision).integrate_batch(spec.spacetime, rows, spec.integ, spec.term)
    y0 = torch.as_tensor(rows).cuda()
    options = _lib.options_struct(spec.integ, spec.term, None)
    for n in (1, 64 * sms, 64 * sms + 1, 256 * sms, 256 * sms + 1):
        out = {"Y": torch.full((n, 8), -1.0, dtype=torch.float64, device="cuda"),
               "max_null_error": torch.full((n,), -1.0, dtype=torch.float64, device="cuda")}
        for name in ("state", "n_steps", "n_rejected"):
            out[name] = torch.full((n,), -1, dtype=torch.int64, device="cuda")
        _lib.check(_lib.lib().krr_integrate_batch_device(
            0, 1.0, 0.9, y0.data_ptr(), None, n, ctypes.byref(options), _lib.PRECISIONS[precision],
            ctypes.byref(_lib.result_struct(out, device=True)), torch.cuda.current_stream().cuda_stream))
        for name, got in out.items():
            assert np.array_equal(got.cpu().numpy(), getattr(host, name)[:n]), (n, name)

"""The backend integrates a snapshot of the caller's rows (CPU; the library's call is replaced)."""

from __future__ import annotations

import ctypes
from types import SimpleNamespace

import numpy as np
import pytest

import kerrray_b200 as K
from kerrray_b200 import _lib


@pytest.mark.parametrize("layout", ["C", "F", "strided", "readonly"])
def test_rows_are_the_ones_of_the_call(monkeypatch, layout):
    rows = np.random.default_rng(3).uniform(1.0, 2.0, (37, 8))
    y0 = {"C": rows.copy(), "F": np.asfortranarray(rows), "strided": np.repeat(rows, 2, axis=0)[::2],
          "readonly": rows.copy()}[layout]
    seen = {}

    def integrate(device, mass, spin, p, n, *rest):
        """Another thread writes to the caller's array while the library runs."""
        if layout != "readonly":
            y0[:] = np.nan
        address = p.value if isinstance(p, ctypes.c_void_p) else p
        seen["shared"] = address == y0.ctypes.data
        seen["rows"] = np.frombuffer((ctypes.c_double * (8 * n)).from_address(address)).reshape(n, 8).copy()
        return 0

    if layout == "readonly":
        y0.setflags(write=False)
    monkeypatch.setattr(_lib, "lib", lambda: SimpleNamespace(krr_integrate_batch=integrate))
    backend = object.__new__(K.CudaBackend)
    backend.device, backend.precision = 0, "reference"
    backend.integrate_batch(K.Spacetime(1.0, 0.5), y0, K.IntegratorOptions(), K.TerminationOptions())
    assert np.array_equal(seen["rows"], rows) and not seen["shared"]

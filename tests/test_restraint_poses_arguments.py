"""gisapr_restraint_poses visits only what an atom reaches, so it refuses a threshold below zero (where
gisapr_restraint_eval counts every voxel of the bounds), and names what it asks of apix, rp and kn. On the host: the
checks come before the device is touched."""
import ctypes as C

import numpy as np
import pytest


def _call(lib, threshold=1.0, apix=1.5, rp=1.0, kn=1.0):
    from gisapr_gb300 import _native as nat
    fn = lib.gisapr_restraint_poses
    fn.argtypes = nat.SIGNATURES["gisapr_restraint_poses"]
    room = C.create_string_buffer(1 << 16)  # stands for the context and for device arrays; none is read
    bounds = np.array([0, 0, 0, 8, 8, 8], np.int32)
    p = C.addressof(room)
    rc = fn(p, None, p, p, 4, 1, bounds.ctypes.data, p, p, 32, 6, apix, rp, kn, threshold, p)
    return rc, lib.gisapr_last_error().decode()


@pytest.mark.parametrize("threshold", [-1.0, -1e-30, float("-inf")])
def test_a_threshold_below_zero_is_refused(native_lib, threshold):
    rc, message = _call(native_lib, threshold)
    assert rc == 1 and "threshold below zero" in message


@pytest.mark.parametrize("bad", [dict(apix=0.0), dict(apix=-1.0), dict(apix=float("inf")), dict(rp=float("nan")),
                                 dict(kn=float("inf"))])
def test_parameters_are_named_as_they_are_checked(native_lib, bad):
    rc, message = _call(native_lib, **bad)
    assert rc == 1 and message == "apix must be positive and finite, rp and kn finite"

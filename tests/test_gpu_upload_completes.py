"""uc_upload_fields returns when the fields are on the device, whatever their number of cells (up to 512 they pass
through pinned staging rows, beyond through copies): only uc_upload_fields_device is asynchronous. The context's
stream is idle then, although work queued before the upload was still running, and another stream that knows
nothing of it reads the new fields."""
import ctypes

import numpy as np
import pytest

from conftest import random_state

pytestmark = pytest.mark.gpu


class View(ctypes.Structure):
    """uc_device_view"""
    _fields_ = [(k, ctypes.c_void_p) for k in ("tk", "rho", "fsp", "fsp_old", "stmf", "stnd", "rc", "qdsp", "qdot",
                                               "domega_dy", "vmu", "vtc", "vdf", "cp", "h")] + \
               [("n", ctypes.c_int), ("npad", ctypes.c_int), ("stream", ctypes.c_void_p)]


@pytest.mark.parametrize("n", [1, 512, 513])
def test_fields_are_on_the_device_when_the_upload_returns(oracle, n):
    import torch
    from unicorn_b200 import unichem
    tk, rho, y = random_state(oracle, n, 9)
    tk2, rho2, y2 = random_state(oracle, n, 10)
    with unichem.UniChem(n) as u:
        u.upload(tk, rho, y)
        u.ckrates()
        v = View()
        u.lib.uc_device_view_get.argtypes = [ctypes.c_void_p, ctypes.POINTER(View)]
        u._ck(u.lib.uc_device_view_get(u._h, ctypes.byref(v)))
        stream = torch.cuda.ExternalStream(v.stream)
        # some ten milliseconds of work that the call does not wait for (no pass count asked for)
        u._ck(u.lib.uc_species_update(u._h, 1e-3, 4000, 0.99, -1.0, 0.0, None, None, None))
        assert not stream.query()
        u.upload(tk2, rho2, y2)
        assert stream.query()
        other = torch.cuda.Stream()
        host = torch.empty(52, v.npad, dtype=torch.float64, pin_memory=True)
        dev = _tensor(torch, v.fsp, 52 * v.npad)
        with torch.cuda.stream(other):
            host.view(-1).copy_(dev, non_blocking=True)
        other.synchronize()
        assert np.array_equal(host.numpy()[:, :n], y2)


def _tensor(torch, ptr, count):
    class Holder:
        __cuda_array_interface__ = {"shape": (count,), "typestr": "<f8", "data": (ptr, False), "version": 2}
    return torch.as_tensor(Holder(), device="cuda")

"""Where a batch's magnitudes may go: pageable, page-locked and device memory give the same bits (SFH batches and weights
over ages and metallicities), and so do batches whose magnitudes come down in more than one piece of 4 Mi doubles."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _mags(c, params, n, ptr, wz=None):
    from libopensps_gb300 import capi
    k, names, vals, keep = capi._names_values(params, n)
    st = C.c_int(0)
    p = C.cast(C.c_void_p(ptr), C.POINTER(C.c_double))
    if wz is None:
        c.lib.opensps_context_compute_csp_batch(c.handle, n, k, names, vals, None, p, None, None, None, None, None, None,
                                                None, C.byref(st))
    else:
        c.lib.opensps_context_compute_csp_batch_grad(c.handle, n, k, names, vals, None, capi._ptr(wz), None, None, None,
                                                     None, None, p, None, None, None, None, None, None, None, None, None,
                                                     None, C.byref(st))
    capi._check(st, c.lib)
    del keep


def _params(n):
    rng = np.random.default_rng(n)
    return {"tau": 10.0 ** rng.uniform(-1.0, 1.0, n), "tage": rng.uniform(1.0, 13.7, n),
            "logzsol": rng.uniform(-2.0, 0.5, n), "dust2": rng.uniform(0.0, 2.0, n)}


@pytest.mark.parametrize("weights", [False, True])
def test_any_memory(data, built_lib, weights):
    import torch
    from conftest import config3_inputs
    from libopensps_gb300.capi import Context
    n = 33
    wz, params = config3_inputs(n, seed=4)
    if not weights:
        wz, params = None, _params(n)
    c = Context()
    c.set_int("sfh", 4)
    host = np.zeros((n, c.nbands))
    pinned = torch.zeros((n, c.nbands), dtype=torch.float64).pin_memory()
    dev = torch.zeros((n, c.nbands), dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    for ptr in (host.ctypes.data, pinned.data_ptr(), dev.data_ptr()):
        _mags(c, params, n, ptr, wz)
    c.close()
    assert np.isfinite(host).all() and host.all()
    assert np.array_equal(host, pinned.numpy()) and np.array_equal(host, dev.cpu().numpy())


def test_magnitudes_in_pieces(data, built_lib):
    import torch
    from libopensps_gb300.capi import Context
    c = Context()
    c.set_int("sfh", 4)
    n = (4 << 20) // c.nbands + 1000
    params = _params(n)
    host = np.zeros((n, c.nbands))
    pinned = torch.zeros((n, c.nbands), dtype=torch.float64).pin_memory()
    for ptr in (host.ctypes.data, pinned.data_ptr()):
        _mags(c, params, n, ptr)
    c.close()
    assert np.isfinite(host).all() and host.all()
    assert np.array_equal(host, pinned.numpy())

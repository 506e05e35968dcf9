"""Grids whose pixel tiles (120 pixels each) come in an odd count, so that the second CTA of the contraction's last
pair has no pixels, and of odd pixel counts: batches that single CTAs and CTA pairs take, against the FP64 oracle on
some of their models (spectra 1e-4 relative, magnitudes 1e-3 mag)."""
import os

import numpy as np
import pytest

from conftest import config3_inputs, rel_err_spec
from data_roots import cut_root

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ns", [5875, 5880, 5761])
def test_odd_pixel_tiles(data, built_lib, tmp_path, ns):
    from libopensps_gb300.capi import Context
    from oracle.oracle import Oracle
    assert -(-ns // 120) % 2 == 1
    root, cut = cut_root(tmp_path, data, ns=ns)
    old = os.environ["OPENSPS_DATA_HOME"]
    try:
        c = Context(data_root=root)
        c.set_int("add_neb_emission", 1)
        c.set_int("add_igm_absorption", 1)
        for n in (1, 300, 400, 1500):                     # (from 400 on but for 700: pairs)
            wz, params = config3_inputs(n, seed=n)
            got = c.csp_batch(params, ssp_weights_z=wz)
            m = np.unique(np.linspace(0, n - 1, 12).astype(int))
            ora = Oracle(cut, nbands=40).csp_batch({k: v[m] for k, v in params.items()}, wz[m])
            assert rel_err_spec(got["spec"][m], ora["spec"]) <= 1e-4
            assert np.array_equal(np.isnan(got["mags"][m]), np.isnan(ora["mags"]))
            assert float(np.nanmax(np.abs(got["mags"][m] - ora["mags"]))) <= 1e-3
        c.close()
    finally:
        os.environ["OPENSPS_DATA_HOME"] = old

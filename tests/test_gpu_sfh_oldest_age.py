"""A truncation at the grid's oldest age: star formation ended tq = tage - sf_trunc years ago, on that age or just above
it, so that no age of the grid holds any weight. The window's ends are compared in years by the kernel that forms the
moments and in log10 years by the one that takes their differences, and log10 of the oldest age may round below the
grid's own log age: on grids of every count of ages the weights have to be none, as the oracle's are."""
import os

import numpy as np
import pytest

from data_roots import cut_root

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sfh", [1, 4, 5])
@pytest.mark.parametrize("nt", [33, 35, 37, 41, 44, 48, 55])
def test_truncation_at_the_oldest_age(data, built_lib, tmp_path, sfh, nt):
    from libopensps_gb300.capi import Context
    root, cut = cut_root(tmp_path, data, nt=nt)
    oldest = 10.0 ** cut["log_age"][-1]
    tage = 3.0 * oldest / 1e9
    # sf_trunc over the doubles around tage - oldest; those whose tq is the oldest age or above it, as the device forms it
    # (a few ulps above: the context's own power of ten may differ by one)
    trunc = (tage * 1e9 - oldest) / 1e9
    trunc = trunc + np.arange(-60, 61) * np.spacing(trunc)
    trunc = trunc[tage * 1e9 - trunc * 1e9 >= oldest * (1.0 + 4e-16)]
    n = trunc.size
    assert n >= 20
    old = os.environ["OPENSPS_DATA_HOME"]
    try:
        c = Context(data_root=root)
        c.set_int("sfh", sfh)
        params = {"tau": np.full(n, tage), "tage": np.full(n, tage), "sf_trunc": trunc}
        if sfh == 5:
            params["sf_slope"] = np.full(n, -20.0 / tage)     # (a ramp that ends at once: at tq - tage / 20)
        got = c.csp_batch(params)
        c.close()
    finally:
        os.environ["OPENSPS_DATA_HOME"] = old
    if sfh == 5:                                              # (the ramp's own weights are the oracle's business)
        from oracle.oracle import blend_at_logzsol, sfh_weights
        w, _ = sfh_weights(cut["log_age"], 5, params, n)
        wz, _ = blend_at_logzsol(cut, w, np.zeros(n))
        want = np.einsum("mzt,zt->m", wz, cut["ssp_mass"])
        np.testing.assert_allclose(got["mass"], want, rtol=1e-9)
        return
    assert not got["mass"].any() and not got["spec"].any()

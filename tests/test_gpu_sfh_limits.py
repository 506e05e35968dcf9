"""The SFH weights where their moments change form: Ei's series by its count of terms and beyond 40 (tau from a
hundredth of the age), ages at, between and beyond the grid's, windows that a truncation closes early. Against the FP64
oracle within tests/test_gpu_sfh.py's gates. (Models with tau above 20 ages are left out: the moments' differences over
the whole age then cancel by (tau / age)^2 ulps on the device and in the oracle alike.)"""
import numpy as np
import pytest

from conftest import oracle_sfh_csp
from test_gpu_sfh import _check, _ctx, _forward

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sfh", [1, 4, 5])
def test_sfh_limits(data, built_lib, sfh):
    from oracle.oracle import Oracle
    node = 10.0 ** (data["log_age"][60] - 9.0)
    rows = [(tau, tage, trunc)
            for tau in (0.02, 0.1, 0.3424, 0.3426, 1.0, 10.0)
            for tage in (0.01, node, 0.5, 13.7, 14.2)
            for trunc in (0.0, 0.3)
            if tau <= 20.0 * tage]
    n = len(rows)
    tau, tage, trunc = np.array(rows).T
    params = {"tau": tau, "tage": tage, "sf_trunc": trunc * tage, "logzsol": np.linspace(-1.9, 0.4, n),
              "dust2": np.linspace(0.0, 1.0, n)}
    if sfh == 5:
        params["sf_slope"] = np.full(n, -0.5)
    c = _ctx(sfh, nbands=20)
    got = _forward(c, params, n)
    c.close()
    ora = oracle_sfh_csp(Oracle(data, nbands=20, add_neb=False, add_igm=False), data, sfh, params)
    # (e^(tage / tau) overflows from tage / tau = 709.8 on: the oracle's weights are then none, and so are the device's)
    some = ora["spec"].max(axis=1) > 0.0
    assert some[tage / tau < 700.0].all() and not got["spec"][~some].any()
    _check({k: v[some] for k, v in got.items()}, {k: v[some] for k, v in ora.items() if k in got})

"""The operator's fold for weights blended at logzsol (models sorted by metallicity, only their two slabs' columns
multiplied) against the fold over every slab, which takes the same weights from the caller: the mass and L_bol sums keep
their bits (1e-12), the spectra the split-BF16 sums' order (2^-17 of a term: 2e-5)."""
import numpy as np
import pytest

from conftest import rel_err_spec

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx(data, built_lib):
    from libopensps_gb300.capi import Context
    c = Context()
    c.set_int("add_igm_absorption", 1)
    c.build_ssp_ops()
    yield c
    c.close()


@pytest.mark.parametrize("n", [1, 2, 127, 130, 1409, 4200])
@pytest.mark.parametrize("one_metallicity", [False, True])
def test_slabs_match_every_slab(ctx, data, n, one_metallicity):
    from conftest import blend_at_logzsol
    rng = np.random.default_rng(n)
    w = rng.dirichlet(np.ones(data["log_age"].size), size=n)
    # beyond both ends of the grid and on its nodes too (extrapolated weights below zero count as none)
    logz = np.full(n, -0.31) if one_metallicity else rng.uniform(-2.1, 0.6, n)
    if not one_metallicity and n > 100:
        logz[:12] = np.log10(data["zlegend"] / 0.0142)
    params = {"imf1": rng.uniform(0.3, 1.8, n), "imf2": rng.uniform(1.3, 2.8, n), "imf3": rng.uniform(1.8, 3.3, n),
              "dust2": rng.uniform(0.0, 1.0, n), "zred": rng.uniform(0.0, 2.0, n)}
    got = ctx.csp_batch(dict(params, logzsol=logz), ssp_weights=w)
    assert ctx.ops_last_interpolated()
    wz, _ = blend_at_logzsol(data, w, logz)
    ref = ctx.csp_batch(params, ssp_weights_z=wz)
    assert ctx.ops_last_interpolated()
    np.testing.assert_allclose(got["mass"], ref["mass"], rtol=1e-12)
    np.testing.assert_allclose(got["lbol"], ref["lbol"], rtol=1e-12)
    assert rel_err_spec(got["spec"], ref["spec"]) <= 2e-5

"""The per-model epilogue without dust emission at the batch sizes where its CTAs change (512 threads a model up to 304
models, then 256), for both forms of the dust curve: a batch's spectra against the same models in batches of 100.

Tolerance, fixed before the first run: the models' own arithmetic does not change, the operator's sums before it may take
another split-BF16 order with the batch's size (2e-5, as between the operator's folds)."""
import numpy as np
import pytest

from conftest import rel_err_spec

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", params=[0, 1])
def ctx(request, data, built_lib):
    from libopensps_gb300.capi import Context
    c = Context()
    c.set_int("add_igm_absorption", 1)
    c.set_int("dust_type", request.param)
    c.build_ssp_ops()
    yield c
    c.close()


@pytest.mark.parametrize("n", [101, 304, 305, 1217])
def test_sizes_match_batches_of_100(ctx, data, n):
    rng = np.random.default_rng(n)
    w = rng.dirichlet(np.ones(data["log_age"].size), size=n)
    params = {"imf1": rng.uniform(0.3, 1.8, n), "dust1": rng.uniform(0.0, 1.0, n), "dust2": rng.uniform(0.0, 1.0, n),
              "dust_index": rng.uniform(-1.2, -0.3, n), "mwr": rng.uniform(2.5, 4.0, n), "uvb": rng.uniform(0.5, 1.5, n),
              "zred": rng.uniform(0.0, 2.0, n), "sigma_smooth": rng.uniform(0.0, 300.0, n), "logzsol": rng.uniform(-1.5, 0.3, n)}
    got = ctx.csp_batch(params, ssp_weights=w)
    for i in range(0, n, 100):
        sl = slice(i, min(i + 100, n))
        ref = ctx.csp_batch({k: v[sl] for k, v in params.items()}, ssp_weights=w[sl])
        assert rel_err_spec(got["spec"][sl], ref["spec"]) <= 2e-5
        np.testing.assert_allclose(got["mass"][sl], ref["mass"], rtol=1e-12)

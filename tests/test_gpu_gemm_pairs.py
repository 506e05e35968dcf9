"""The three-product GEMM by single CTAs and by CTA pairs: the operator's template sums and the reverse pass's weight
cotangents at model counts on both sides of the rule (one 128-row tile, a ragged pair, an odd count of tiles), against
the same models in batches of 32, which single CTAs take.

Tolerance, fixed before the first run: the split-BF16 sums in another order, 2e-5 of the spectra and of the cotangents'
norm (as between the operator's folds)."""
import numpy as np
import pytest

from conftest import rel_err_spec

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [64, 65, 129, 321, 833])
def test_template_sums(data, built_lib, n):
    from libopensps_gb300.capi import Context
    rng = np.random.default_rng(n)
    w = rng.dirichlet(np.ones(data["log_age"].size), size=n)
    params = {"imf1": rng.uniform(0.3, 1.8, n), "dust2": rng.uniform(0.0, 1.0, n), "logzsol": rng.uniform(-1.5, 0.3, n)}
    c = Context()
    c.build_ssp_ops()
    got = c.csp_batch(params, ssp_weights=w)["spec"]
    for i in range(0, n, 32):
        sl = slice(i, min(i + 32, n))
        assert rel_err_spec(got[sl], c.csp_batch({k: v[sl] for k, v in params.items()}, ssp_weights=w[sl])["spec"]) <= 2e-5
    c.close()


@pytest.mark.parametrize("n", [129, 321, 833])
def test_weight_cotangents(data, built_lib, n):
    from conftest import config3_inputs
    from libopensps_gb300.capi import Context
    from libopensps_gb300 import workloads
    wz, params = config3_inputs(n, seed=n)
    c = Context()
    mb, sb = workloads.adjoint_cotangents(n, c.nspec, c.nbands, seed=n)
    got = c.csp_batch_grad(params, ssp_weights_z=wz, mags_bar=mb, spec_bar=sb)["weights_z_bar"]
    for i in range(0, n, 32):
        sl = slice(i, min(i + 32, n))
        ref = c.csp_batch_grad({k: v[sl] for k, v in params.items()}, ssp_weights_z=wz[sl], mags_bar=mb[sl], spec_bar=sb[sl])["weights_z_bar"]
        for a, b in zip(got[sl], ref):
            assert np.linalg.norm(a - b) <= 2e-5 * np.linalg.norm(b)
    c.close()

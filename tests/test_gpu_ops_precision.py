"""The operator's fold over two slabs rounds no more than the fold over every slab. The tensor core's accumulator drops
what lies below its last place at each step of 16 columns, so that a longer chain of steps per split leaves sums of
positive terms lower: the mean signed difference of the two folds' spectra, over pixels and models, shows a longer chain
where its scatter (the split-BF16 rounding of the template sums, the same in both) hides it.

Tolerance, fixed before the first run: one step's three products, a last place each at most, 3 x 2^-24 of the sum."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx(data, built_lib):
    from libopensps_gb300.capi import Context
    c = Context()
    c.build_ssp_ops()
    yield c
    c.close()


@pytest.mark.parametrize("n", [1, 2, 4, 16, 64, 128, 129, 256, 513, 1024, 1500])
def test_two_slabs_round_no_more(ctx, data, n):
    from conftest import blend_at_logzsol
    rng = np.random.default_rng(n)
    w = rng.dirichlet(np.ones(data["log_age"].size), size=n)
    logz = rng.uniform(-2.0, 0.5, n)
    params = {"imf1": rng.uniform(0.3, 1.8, n), "imf2": rng.uniform(1.3, 2.8, n), "imf3": rng.uniform(1.8, 3.3, n)}
    got = ctx.csp_batch(dict(params, logzsol=logz), ssp_weights=w)["spec"]
    assert ctx.ops_last_interpolated()
    ref = ctx.csp_batch(params, ssp_weights_z=blend_at_logzsol(data, w, logz)[0])["spec"]
    some = ref > 1e-6 * ref.max(axis=1, keepdims=True)
    mean = np.mean(got[some] / ref[some] - 1.0)
    assert mean >= -3.0 * 2.0 ** -24, mean

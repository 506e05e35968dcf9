"""The reverse passes' GEMMs at batch sizes that split their K range differently: the same models' gradients from a batch
of their own, a middling one and one whose tiles fill the GPU. The split changes the order of the FP32 sums, whose
products carry the split-BF16 representation (2^-17 of a term): 5e-5 of each row's largest value."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SIZES = (1, 130, 1300, 10240)


@pytest.mark.parametrize("ops", [False, True])
def test_gradients_do_not_depend_on_the_batch(data, built_lib, ops):
    from libopensps_gb300 import workloads
    from libopensps_gb300.capi import Context
    ctx = Context()
    ctx.set_int("add_igm_absorption", 1)
    if ops:
        ctx.build_ssp_ops()
    else:
        ctx.set_int("add_neb_emission", 1)
    sizes = SIZES[:3] if ops else SIZES
    n = sizes[-1]
    wz, params = workloads.mixed_csp(n, seed=77)
    rng = np.random.default_rng(78)
    if ops:
        params.update(imf1=rng.uniform(0.3, 1.8, n), imf2=rng.uniform(1.3, 2.8, n), imf3=rng.uniform(1.8, 3.3, n))
    params["zred"] = rng.uniform(0.1, 2.0, n)
    bar = rng.standard_normal((n, ctx.nbands))
    got = {}
    for k in sizes:
        r = ctx.csp_batch_grad({p: v[:k] for p, v in params.items()}, wz[:k], mags_bar=bar[:k], spec=False)
        # (what the split GEMMs feed: the weights' cotangent, and with the operator the slopes' rows; the other rows come
        # from the per-model adjoint alone)
        got[k] = {"weights_z_bar": r["weights_z_bar"][:130].copy()}
        if ops:
            got[k]["imf rows"] = r["params_bar"][:130, 26:29].copy()
    ctx.close()
    for k in sizes[:-1]:
        m = min(k, 130)
        for q in got[k]:
            a, b = got[k][q][:m].reshape(m, -1), got[n][q][:m].reshape(m, -1)
            scale = np.abs(b).max(axis=1 if q == "weights_z_bar" else 0, keepdims=True)
            assert np.all(np.abs(a - b) <= 5e-5 * scale), (k, q, np.max(np.abs(a - b) / np.where(scale > 0, scale, 1)))

"""The three-product GEMM by single CTAs and by CTA pairs, each against FP64: the reverse pass's weight cotangents of
a plain spectrum (the basis times the cotangent) and the operator's sums. The sizes lie on both sides of the rule that
chooses between them (restated here for 152 SMs: pairs where 147 x their waves are below 200 x the single CTAs').

Tolerances, fixed before the first run: each cotangent within 4e-5 of the sum of its terms' magnitudes (three products of
operands in two BF16 parts: 3 x 2^-18; at most 226 steps of an accumulator that drops what lies below its last place,
2^-23 each), where a wrong half of a tile is off by 1e-2 of it; the spectra 1e-4, as the operator's tests hold them."""
import numpy as np
import pytest

from conftest import config3_inputs, rel_err_spec

pytestmark = pytest.mark.gpu
SMS = 152


def _ceil(a, b):
    return -(-a // b)


def _splits(tiles, nkb):
    best, best_eff = 1, -1.0
    for ks in range(1, max(1, min(64, nkb // 8)) + 1):
        eff = tiles * ks / (_ceil(tiles * ks, SMS) * SMS)
        if tiles * ks >= 2 * SMS and eff >= 0.85:
            return ks
        if eff > best_eff + 1e-9:
            best, best_eff = ks, eff
    return best


def _pairs(m, n, nkb):
    rest = _ceil(n, 256) * _splits(_ceil(m, 128) * _ceil(n, 256), nkb)
    return _ceil(_ceil(m, 256) * rest, SMS // 2) * 147 < _ceil(_ceil(m, 128) * rest, SMS) * 200


@pytest.fixture(scope="module", autouse=True)
def _chip():
    import torch
    if torch.cuda.get_device_properties(0).multi_processor_count != SMS:
        pytest.skip("the sizes are those of 152 SMs")


# (young columns, old columns by pairs)
@pytest.mark.parametrize("n,arms", [(65, (True, True)), (129, (True, True)), (321, (True, False)), (833, (False, False)),
                                    (1000, (True, True))])
def test_weight_cotangents_against_fp64(data, built_lib, n, arms):
    from libopensps_gb300.capi import Context
    nz, nt, ns = data["ssp_spec"].shape
    young = int(np.sum(data["log_age"] <= 7.0))
    pad = lambda k: _ceil(k, 64) * 64  # noqa: E731
    cols = pad(young * nz), pad((nt - young) * nz)
    assert tuple(_pairs(n, k, _ceil(ns, 64)) for k in cols) == arms
    rng = np.random.default_rng(n)
    wz, _ = config3_inputs(n, seed=n)
    bar = rng.standard_normal((n, ns))
    c = Context()
    got = c.csp_batch_grad({"dust2": np.zeros(n)}, ssp_weights_z=wz, spec_bar=bar, spec=False)["weights_z_bar"]
    c.close()
    want = (bar @ data["ssp_spec"].reshape(nz * nt, ns).T).reshape(n, nz, nt)
    terms = (np.abs(bar) @ data["ssp_spec"].reshape(nz * nt, ns).T).reshape(n, nz, nt)
    assert (np.abs(got - want) / terms).max() <= 4e-5


@pytest.mark.parametrize("n,pairs", [(100, False), (200, True), (321, True)])
def test_operator_sums_against_fp64(data, built_lib, n, pairs):
    """The fold over every slab (single CTAs up to 128 models) and the template sums (pairs at every size)."""
    from libopensps_gb300 import synth_ops
    from libopensps_gb300.capi import Context
    from oracle.oracle import OpsOracle
    assert all(_pairs(n, 2000, k) == pairs for k in (525, 1080))
    rng = np.random.default_rng(n)
    wz, _ = config3_inputs(n, seed=n)
    alpha = np.stack([rng.uniform(0.3, 1.8, n), rng.uniform(1.3, 2.8, n), rng.uniform(1.8, 3.3, n)], axis=1)
    c = Context()
    c.build_ssp_ops()
    got = c.csp_batch({"imf1": alpha[:, 0], "imf2": alpha[:, 1], "imf3": alpha[:, 2]}, ssp_weights_z=wz)
    assert c.ops_last_interpolated()
    c.close()
    m = np.unique(np.concatenate([np.linspace(0, n - 1, 8).astype(int), [63, 64, 127 % n, 128 % n, n - 2]]))
    y, o, mass, _ = OpsOracle(synth_ops.load()).parts(alpha[m], wz[m], int(np.sum(data["log_age"] <= 7.0)))
    assert rel_err_spec(got["spec"][m], y + o) <= 1e-4
    np.testing.assert_allclose(got["mass"][m], mass, rtol=1e-5)

"""The mixed batch at the sizes where its kernels change their split: models per CTA of the parameter kernel, a CTA or
a warp per model in the weight operand, the contraction's model tiles. A strided sample (the last model included)
against the FP64 oracle, within the gates of the batch's other parity tests (magnitudes 1e-3 mag, spectra 1e-4, FP64
mass sums 1e-12)."""
import numpy as np
import pytest

from conftest import config3_inputs, rel_err_spec

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def setup(data, built_lib):
    from libopensps_gb300.capi import Context
    from oracle.oracle import Oracle
    ctx = Context()
    ctx.set_int("add_neb_emission", 1)
    ctx.set_int("add_igm_absorption", 1)
    yield ctx, Oracle(data, nbands=ctx.nbands)
    ctx.close()


@pytest.mark.parametrize("n", [1, 2, 31, 33, 65, 153, 305, 609, 1217, 3011, 8192, 8193])
@pytest.mark.parametrize("birth_cloud", [False, True])
def test_batch_sizes(setup, n, birth_cloud):
    ctx, oracle = setup
    wz, params = config3_inputs(n, seed=n)
    if birth_cloud:
        rng = np.random.default_rng(n)
        params = dict(params, dust1=rng.uniform(0.1, 1.0, n), dust3=rng.uniform(0.0, 0.4, n))
    got = ctx.csp_batch(params, ssp_weights_z=wz)
    pick = np.unique(np.concatenate([np.linspace(0, n - 1, min(n, 12)).astype(int), [n - 1]]))
    ref = oracle.csp_batch({k: v[pick] for k, v in params.items()}, wz[pick])
    assert rel_err_spec(got["spec"][pick], ref["spec"]) <= 1e-4
    assert np.nanmax(np.abs(got["mags"][pick] - ref["mags"])) <= 1e-3
    assert np.max(np.abs(got["mass"][pick] / ref["mass"] - 1.0)) <= 1e-12


@pytest.mark.parametrize("n", [1, 33, 8192, 8193])
@pytest.mark.parametrize("fesc", [0.0, 0.4])
def test_device_inputs(setup, n, fesc):
    """Device inputs form the weight operand without the sums: the magnitudes of the same batch from host inputs, to
    FP32 rounding (1e-4 mag)."""
    import torch
    from libopensps_gb300 import workloads
    ctx, _ = setup
    wz, params = config3_inputs(n, seed=n)
    if fesc:
        params = dict(params, frac_obrun=np.full(n, fesc))
    want = ctx.csp_batch(params, ssp_weights_z=wz, spec=False)
    d_wz = torch.from_numpy(wz).cuda()
    d_par = torch.from_numpy(workloads.device_param_table(params, n)).cuda()
    d_mags = torch.empty((n, ctx.nbands), dtype=torch.float64, device="cuda")
    ctx.batch_device(n, d_par.data_ptr(), d_wz.data_ptr(), d_mags.data_ptr(), sync=True)
    np.testing.assert_allclose(d_mags.cpu().numpy(), want["mags"], rtol=0, atol=1e-4)

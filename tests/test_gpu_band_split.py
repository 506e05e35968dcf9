"""The band GEMM at the batch sizes where its split of the pixels over a cluster changes (few tiles and many, ragged
last tiles), from spectra at addresses of every alignment.

Tolerance, fixed before the first run: FP32 sums of a few thousand positive terms in another order, 1e-4 mag, as the
magnitudes of batches of different sizes are held to elsewhere."""
import pytest

from conftest import config3_inputs

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx(data, built_lib):
    from libopensps_gb300.capi import Context
    c = Context()
    c.set_int("add_igm_absorption", 1)
    yield c
    c.close()


@pytest.mark.parametrize("n", [1, 127, 129, 641, 2433, 2561, 4096, 4097, 9729, 19457, 20001])
@pytest.mark.parametrize("shift", [0, 1, 2, 3])
def test_split_and_alignment(ctx, n, shift):
    """spec_mags_noalloc of n spectra that begin `shift` floats into a buffer: the same magnitudes, model by model, as
    the same spectra give in batches of 97 (another split, and other alignments of each row)."""
    import torch
    if shift and n > 5000:
        pytest.skip("the alignments at the smaller sizes")
    base = 97
    wz, params = config3_inputs(base, seed=5)
    spec = torch.from_numpy(ctx.csp_batch(params, ssp_weights_z=wz)["spec"]).float().cuda()
    ns = spec.shape[1]
    z = torch.linspace(0.0, 4.0, base, dtype=torch.float64, device="cuda")
    z[1] = 0.0
    idx = torch.arange(n, device="cuda") % base
    buf = torch.full((shift + n * ns + 64,), float("nan"), device="cuda")
    buf[shift:shift + n * ns].view(n, ns).copy_(spec[idx])
    mags = torch.empty((n, ctx.nbands), dtype=torch.float64, device="cuda")
    zz = z[idx].contiguous()
    torch.cuda.synchronize()      # (the call runs on the context's stream)
    ctx.spec_mags_noalloc(n, buf.data_ptr() + 4 * shift, zz.data_ptr(), mags.data_ptr(), sync=True)
    ref = torch.empty((base, ctx.nbands), dtype=torch.float64, device="cuda")
    ctx.spec_mags_noalloc(base, spec.data_ptr(), z.data_ptr(), ref.data_ptr(), sync=True)
    want = ref[idx]
    assert torch.equal(torch.isnan(mags), torch.isnan(want))
    ok = ~torch.isnan(want)
    assert float((mags[ok] - want[ok]).abs().max()) <= 1e-4

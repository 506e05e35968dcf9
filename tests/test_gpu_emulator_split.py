"""The emulator's small batches (one member of a tile per CTA, then a reduction) against the fused kernel's results of the
same models in a batch that fills the GPU. Both run the same members' MMAs; only the order in which the five members'
outputs are summed differs: 5 x 2^-24 of values up to 150 (magnitudes, PCA coefficients), so 5e-5 absolute."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

FULL = 2 * 152 * 128 + 4096       # more than two tiles per SM: always the fused kernel


@pytest.fixture(scope="module")
def emu(built_lib):
    import torch
    from libopensps_gb300.emulator import WEIGHTS, training_context
    ctx = training_context()
    ctx.emulator_load(WEIGHTS)
    lo = np.array([0.1, 1.0, -2.0, 0.0, -1.0, 0.0, 50.0, 0.3, 1.3, 1.8])
    hi = np.array([10.0, 13.7, 0.5, 3.0, -0.4, 6.0, 300.0, 1.8, 2.8, 3.3])
    x = lo + (hi - lo) * np.random.default_rng(5).uniform(size=(FULL, 10))
    x[7, 3] = 4.0                  # outside the box
    x[11, 1] = np.nan              # not finite
    d_x = torch.from_numpy(x.astype(np.float32)).cuda()

    def predict(n):
        out = {k: torch.zeros((n, w), device="cuda") for k, w in (("mags", ctx.nbands), ("pca", 64), ("spread", 1))}
        flag, flagged = (torch.zeros(n, dtype=torch.int32, device="cuda") for _ in range(2))
        k = ctx.emulator_predict_device(n, d_x.data_ptr(), out["mags"].data_ptr(), flag.data_ptr(), flagged.data_ptr(),
                                        out["pca"].data_ptr(), out["spread"].data_ptr())
        got = {k2: v.cpu().numpy() for k2, v in out.items()}
        got["flag"], got["flagged"] = flag.cpu().numpy(), np.sort(flagged.cpu().numpy()[:k])
        return got

    yield predict, predict(FULL)
    ctx.close()


@pytest.mark.parametrize("n", [1, 127, 128, 129, 3891, 19457, 38912])
def test_split_matches_fused(emu, n):
    predict, full = emu
    got = predict(n)
    for k in ("mags", "pca", "spread"):
        np.testing.assert_allclose(got[k], full[k][:n], rtol=0, atol=5e-5)
    # flags: the box and the finite check exactly, the spread's threshold where it is not within rounding of it
    clear = np.abs(full["spread"][:n, 0] - 0.01) > 5e-5
    np.testing.assert_array_equal(got["flag"][clear], full["flag"][:n][clear])
    np.testing.assert_array_equal(got["flagged"], np.nonzero(got["flag"])[0])

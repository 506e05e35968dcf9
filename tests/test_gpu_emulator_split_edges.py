"""The emulator on both sides of its rule for small batches: members on CTAs of their own while that takes fewer rounds
over the SMs than whole tiles (up to 121 tiles of 128 models on 152 SMs, and from 153 to 273), the fused kernel between
and beyond. Each size against the fused kernel's results of the same models in a batch of more than two tiles per SM.

Tolerance: the five members' outputs summed in another order, 5 x 2^-24 of values up to 150, so 5e-5 absolute."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def emu(built_lib):
    import torch
    from libopensps_gb300.emulator import WEIGHTS, training_context
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    full = 2 * sms * 128 + 4096
    ctx = training_context()
    ctx.emulator_load(WEIGHTS)
    lo = np.array([0.1, 1.0, -2.0, 0.0, -1.0, 0.0, 50.0, 0.3, 1.3, 1.8])
    hi = np.array([10.0, 13.7, 0.5, 3.0, -0.4, 6.0, 300.0, 1.8, 2.8, 3.3])
    x = lo + (hi - lo) * np.random.default_rng(6).uniform(size=(full, 10))
    d_x = torch.from_numpy(x.astype(np.float32)).cuda()

    def predict(n):
        out = {k: torch.zeros((n, w), device="cuda") for k, w in (("mags", ctx.nbands), ("pca", 64), ("spread", 1))}
        flag, flagged = (torch.zeros(n, dtype=torch.int32, device="cuda") for _ in range(2))
        torch.cuda.synchronize()
        ctx.emulator_predict_device(n, d_x.data_ptr(), out["mags"].data_ptr(), flag.data_ptr(), flagged.data_ptr(),
                                    out["pca"].data_ptr(), out["spread"].data_ptr())
        return {k2: v.cpu().numpy() for k2, v in out.items()}

    def split(tiles):
        return tiles <= 2 * sms and -(-tiles * 5 // sms) < -(-tiles // sms) * 5

    edges = [t for t in range(1, 2 * sms + 1) if split(t) != split(t + 1)]
    assert len(edges) >= 3
    yield predict, predict(full), edges
    ctx.close()


@pytest.mark.parametrize("edge", [0, 1, 2])
@pytest.mark.parametrize("more", [-1, 0, 1])
def test_edges_of_the_split(emu, edge, more):
    predict, full, edges = emu
    n = 128 * edges[edge] + more
    got = predict(n)
    for k in ("mags", "pca", "spread"):
        np.testing.assert_allclose(got[k], full[k][:n], rtol=0, atol=5e-5)

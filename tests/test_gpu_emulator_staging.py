"""Host predictions of any size stage through a bounded page-locked buffer, and give what the same models give in
batches of one slice or less."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _shared_mb() -> int:
    """Resident shared memory of the process: page-locked host memory counts here."""
    for line in open("/proc/self/status"):
        if line.startswith("RssShmem:"):
            return int(line.split()[1]) // 1024
    pytest.skip("no RssShmem")


def test_staging_is_bounded(built_lib):
    from libopensps_gb300.emulator import WEIGHTS, training_context
    lo = np.array([0.1, 1.0, -2.0, 0.0, -1.0, 0.0, 50.0, 0.3, 1.3, 1.8])
    hi = np.array([10.0, 13.7, 0.5, 3.0, -0.4, 6.0, 300.0, 1.8, 2.8, 3.3])
    n = 3 * 65536 + 77
    x = lo + (hi - lo) * np.random.default_rng(9).uniform(size=(n, 10))
    x[65536 + 5, 3] = 4.0          # outside the box, in the second slice
    x[n - 1, 1] = np.nan           # and in the last (a NaN lies in no box)
    ctx = training_context()
    ctx.emulator_load(WEIGHTS)
    ctx.emulator_predict(x[:1000], fallback=False, pca=True)
    before = _shared_mb()
    got = ctx.emulator_predict(x, fallback=False, pca=True)
    assert _shared_mb() - before <= 64                    # (496 bytes a model: 98 MB for these)
    assert got["source"][65536 + 5] == 1 and got["source"][n - 1] == 1
    assert got["n_fallback"] == np.count_nonzero(got["source"])
    for m0 in range(0, n, 50000):
        m = slice(m0, min(n, m0 + 50000))
        part = ctx.emulator_predict(x[m], fallback=False, pca=True)
        for k in ("mags", "spread", "pca"):               # (the members' sum in another order: 5 x 2^-24 of 150)
            np.testing.assert_allclose(got[k][m], part[k], rtol=0, atol=5e-5)
        clear = np.abs(part["spread"] - 0.01) > 5e-5
        np.testing.assert_array_equal(got["source"][m][clear], part["source"][clear])
    ctx.close()

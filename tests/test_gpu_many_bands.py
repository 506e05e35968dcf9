"""Magnitudes in more than 80 bands (up to the 256 the band GEMM takes): there one CTA fits an SM, with two or three
slots of the band matrix, and a cluster holds at most eight. Against the same filters in sets of 40.

Tolerance, fixed before the first run: FP32 sums of a few thousand positive terms in another order, 1e-4 mag, as the
magnitudes of batches of different sizes are held to elsewhere."""
import os

import numpy as np
import pytest

from conftest import config3_inputs

pytestmark = pytest.mark.gpu
BASE = 97


@pytest.fixture(scope="module")
def bands(data, built_lib, tmp_path_factory):
    """A context, spectra and redshifts on the GPU, and their magnitudes in 256 bands, 40 at a time."""
    import torch
    from libopensps_gb300 import stdformat
    from libopensps_gb300.capi import Context
    root = tmp_path_factory.mktemp("many_bands")
    stdformat.convert_synthetic(root, dust=False, agn=False)
    centres = np.sort(10.0 ** np.random.default_rng(17).uniform(np.log10(1500.0), np.log10(50000.0), 256))
    sets = {f"many{nb}": np.arange(256)[:nb] for nb in (81, 128, 176, 200, 256)}
    sets.update({f"part{i}": np.arange(40 * i, min(40 * i + 40, 256)) for i in range(7)})
    for name, idx in sets.items():
        npts, lam, tr = stdformat.gaussian_curves(centres[idx])
        flt = [{"name": f"M{i:03d}", "description": "Gaussian, R = 5"} for i in idx]
        stdformat.write_library(root, "filters", name,
                                axes={"filter": {"units": "", "labels": [f["name"] for f in flt]}},
                                arrays={"npoints": (npts, "<i4", ["filter"], "count"),
                                        "wavelength": (lam, "<f8", None, "angstrom"),
                                        "transmission": (tr, "<f8", None, "relative throughput")},
                                metadata={"filters": flt}, title=name)
    stdformat.write_root_index(root)
    old = os.environ["OPENSPS_DATA_HOME"]
    c = Context(data_root=root)
    c.set_int("add_igm_absorption", 1)
    wz, params = config3_inputs(BASE, seed=6)
    spec = torch.from_numpy(c.csp_batch(params, ssp_weights_z=wz)["spec"]).float().cuda()
    z = torch.linspace(0.0, 4.0, BASE, dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    parts = []
    for i in range(7):
        c.set_filters_library(f"part{i}")
        parts.append(_mags(c, spec, z))
    yield c, spec, z, torch.cat(parts, 1)
    c.close()
    os.environ["OPENSPS_DATA_HOME"] = old


def _mags(c, spec, z):
    import torch
    mags = torch.empty((spec.shape[0], c.nbands), dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    c.spec_mags_noalloc(spec.shape[0], spec.data_ptr(), z.data_ptr(), mags.data_ptr(), sync=True)
    return mags


@pytest.mark.parametrize("nb", [81, 128, 176, 200, 256])
@pytest.mark.parametrize("n", [1, 129, 1500, 4097, 9729])
def test_many_bands(bands, nb, n):
    import torch
    c, spec, z, want = bands
    c.set_filters_library(f"many{nb}")
    assert c.nbands == nb
    idx = torch.arange(n, device="cuda") % BASE
    got, ref = _mags(c, spec[idx].contiguous(), z[idx].contiguous()), want[idx][:, :nb]
    assert torch.equal(torch.isnan(got), torch.isnan(ref))
    ok = ~torch.isnan(ref)
    assert float((got[ok] - ref[ok]).abs().max()) <= 1e-4

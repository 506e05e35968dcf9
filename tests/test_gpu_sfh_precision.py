"""The SFH weights stand as near the exact ones as the FP64 oracle's: masses of exponential and delayed-tau histories with
tau of 1 to 100 ages (the moments' differences cancel by the square of that), against the same closed forms in extended
precision. The ages are those whose logarithm, in years, rounds by more than 0.4 of its last place: a moment formed with
an age and a logarithm that do not belong together shows there.

Tolerance, fixed before the first run: the root mean square error over 1500 models at most 1.1 times the oracle's (three
times the sampling error of the two, 1 / sqrt(3000) each, and 0.02 for the functions' last places)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
LD = np.longdouble
GAMMA = LD("0.577215664901532860606512090082402431042159")


def _ei(x):
    """Ei by its power series (x up to 1)."""
    t, s = x.copy(), x.copy()
    for k in range(2, 40):
        t = t * x / k
        s = s + t / k
    return GAMMA + np.log(x) + s


def _masses(data, sfh, p):
    """The mass of the blended weights, in extended precision."""
    if np.finfo(LD).eps > 2e-19:
        pytest.skip("no extended precision")
    tf = data["log_age"].astype(LD)
    ten, log_e = LD(10), LD(1) / np.log(LD(10))
    tage, tau, trunc = (p[k].astype(LD) * LD(1e9) for k in ("tage", "tau", "sf_trunc"))
    tq = np.where((trunc <= 0) | (trunc > tage), LD(0), tage - trunc)
    lo, hi = np.maximum(tq, LD(1))[:, None], np.maximum(tage, LD(1))[:, None]
    t = np.minimum(np.maximum(ten ** tf[None], lo), hi)          # (n, nt) limits
    lt = np.minimum(np.maximum(tf[None], np.log10(lo)), np.log10(hi))
    x = t / tau[:, None]
    e, ei = np.exp(x), _ei(x)
    if sfh == 1:
        m0, m1 = e, lt * e - log_e * ei
        first = e[:, 0] - np.exp(lo[:, 0] / tau)
    else:
        q = t - tage[:, None] - tau[:, None]
        m0 = -(q * e)
        m1 = -((q * lt - tau[:, None] * log_e) * e) - (tage + tau)[:, None] * log_e * ei
        first = m0[:, 0] + (lo[:, 0] - tage - tau) * np.exp(lo[:, 0] / tau)
    d0, d1 = m0[:, 1:] - m0[:, :-1], m1[:, 1:] - m1[:, :-1]
    w = np.zeros_like(t)
    w[:, :-1] += (tf[1:] * d0 - d1) / (tf[1:] - tf[:-1])
    w[:, 1:] += (d1 - tf[:-1] * d0) / (tf[1:] - tf[:-1])
    w[:, 0] += np.where(lo[:, 0] < t[:, 0], first, LD(0))
    w /= w.sum(1, keepdims=True)
    return w


def _blended_mass(data, w, logzsol):
    lz = np.log10(data["zlegend"] / 0.0142)
    z = np.clip(np.searchsorted(lz, logzsol, side="right") - 1, 0, lz.size - 2)
    dz = ((logzsol - lz[z]) / (lz[z + 1] - lz[z])).astype(w.dtype)[:, None]
    m = data["ssp_mass"].astype(w.dtype)
    return (w * ((1 - dz) * m[z] + dz * m[z + 1])).sum(1)


@pytest.mark.parametrize("sfh", [1, 4])
@pytest.mark.parametrize("ratio", [(1.0, 10.0), (10.0, 100.0)])
def test_masses_against_extended_precision(data, built_lib, sfh, ratio):
    from libopensps_gb300.capi import Context
    from oracle.oracle import blend_at_logzsol, sfh_weights
    n = 1500
    rng = np.random.default_rng(sfh)
    tage = 10.0 ** rng.uniform(-2.0, 1.14, 20 * n)
    log_t = np.log10((tage * 1e9).astype(LD))
    off = np.abs(log_t.astype(np.float64).astype(LD) - log_t) / np.spacing(log_t.astype(np.float64))
    tage = tage[off > 0.4][:n]
    assert tage.size == n
    p = {"tage": tage, "tau": tage * 10.0 ** rng.uniform(*np.log10(ratio), n), "sf_trunc": np.zeros(n)}
    logz = rng.uniform(-1.9, 0.4, n)
    true = _blended_mass(data, _masses(data, sfh, p), logz)
    w, _ = sfh_weights(data["log_age"], sfh, p, n)
    plain = _blended_mass(data, w, logz)
    c = Context()
    c.set_int("sfh", sfh)
    got = c.csp_batch(dict(p, logzsol=logz), spec=False)["mass"]
    c.close()
    rms = [float(np.sqrt(np.mean((m.astype(LD) / true - 1) ** 2))) for m in (got, plain)]
    assert rms[0] <= 1.1 * rms[1], rms

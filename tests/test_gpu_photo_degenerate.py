"""Degenerate angles and units in the flux kernels: quotients by zero and by
infinity are the reference's (0 / 0 is NaN, 0 / inf is 0) in the tiled kernels
(32 and 16 bins) and in the thread-per-bin kernel alike, so the same call does
not depend on whether its tile fits shared memory. Finite values within the
photochemistry tests' 1e-11 of the oracle, relative per bin; NaN and infinities
where the oracle has them."""
import numpy as np
import pytest

from conftest import load_pkg
from oracle import photo as orc

pytestmark = pytest.mark.gpu

photo = load_pkg("photo")


def tables(rng, nz, nbin, ni):
    cross = lambda *s: 10.0 ** rng.uniform(-24.0, -18.0, s)   # noqa: E731
    return dict(absp_idx=np.arange(4), absp_cross=cross(4, nbin), absp_T_idx=np.arange(4, 6),
                absp_T_cross=cross(2, nz, nbin), scat_idx=np.arange(6, 8), scat_cross=cross(2, nbin),
                din12_indx=nbin // 3, dbin1=0.125, dbin2=0.5, bins=2.0 + np.arange(nbin) * 0.5,
                sflux_top=10.0 ** rng.uniform(0.0, 3.0, nbin), mu_zenith=0.67, edd=0.5, ag0=0.0, hc=1.98644582e-9)


@pytest.mark.parametrize("nz", [17, 130, 500])
@pytest.mark.parametrize("change", [dict(mu_zenith=0.0), dict(mu_zenith=np.inf), dict(edd=np.inf), dict(hc=0.0),
                                    dict(hc=np.inf), dict(bin=0.0), dict(bin=np.inf)], ids=str)
def test_degenerate(nz, change):
    rng = np.random.default_rng(nz)
    nbin, ni = 33, 10
    ph = tables(rng, nz, nbin, ni)
    if "bin" in change:
        ph["bins"][1] = change["bin"]
    else:
        ph.update(change)
    y = 10.0 ** rng.uniform(8.0, 16.0, (nz, ni))
    y[nz // 2:] = 0.0       # transparent layers: no optical depth, no scattering
    ph["sflux_top"][2] = 0.0
    ymix = y / np.maximum(y.sum(axis=1, keepdims=True), 1e-300)
    dz = 10.0 ** rng.uniform(5.5, 6.5, nz)
    prev = np.zeros((nz + 1, nbin))
    dev = photo.PhotoDevice(ph, nz)
    tau = photo.compute_tau_jax(y, dz, dev)
    got = photo.compute_flux_jax(tau, ymix, dev, prev)
    with np.errstate(all="ignore"):
        # (NumPy scalars: Python's floats raise on a division by zero)
        ph = {k: np.float64(v) if isinstance(v, float) else v for k, v in ph.items()}
        ref = orc.compute_flux(tau.cpu().numpy(), ymix, ph, prev)
    for a, b, name in zip(got, ref, ("aflux", "sflux", "dflux_d", "dflux_u")):
        a, b = a.cpu().numpy(), np.asarray(b)
        fin = np.isfinite(b)
        np.testing.assert_array_equal(np.where(fin, 0.0, a), np.where(fin, 0.0, b), err_msg=name)
        scale = np.abs(np.where(fin, b, 0.0)).max(axis=0, keepdims=True)
        err = np.abs(np.where(fin, a, 0.0) - np.where(fin, b, 0.0))
        assert np.isfinite(a[fin]).all() and np.all(err <= 1e-11 * scale), name

"""The tiled photochemistry kernels at the edges of their tiles: layer counts
around the layers in flight and on both sides of the shared-memory limits of
the flux tile (32 bins, 16 bins, a thread per column), bin counts off the tile,
batches either side of the J kernel's atmosphere tiles, missing absorber kinds,
and a mask of due atmospheres; against the oracle within the bounds of the
photochemistry tests (1e-12 tau, direct beam and J, 1e-11 diffuse and actinic
flux, relative per bin)."""
import numpy as np
import pytest
import torch

from conftest import load_pkg
from oracle import photo as orc

pytestmark = pytest.mark.gpu

photo = load_pkg("photo")


def tables(rng, nz, nbin, n_abs, n_T, n_scat, ni):
    sp = rng.permutation(ni)
    cross = lambda *s: 10.0 ** rng.uniform(-24.0, -18.0, s)   # noqa: E731
    bins = 2.0 + np.arange(nbin) * 0.5
    return dict(absp_idx=sp[:n_abs], absp_cross=cross(n_abs, nbin), absp_T_idx=sp[n_abs:n_abs + n_T],
                absp_T_cross=cross(n_T, nz, nbin), scat_idx=sp[n_abs + n_T:n_abs + n_T + n_scat],
                scat_cross=cross(n_scat, nbin), cross_J=cross(7, nbin), cross_J_T=cross(3, nz, nbin),
                branch_re_idx=np.arange(1, 8), branch_T_re_idx=np.arange(8, 11), din12_indx=nbin // 3, dbin1=0.125,
                dbin2=0.5, bins=bins, sflux_top=10.0 ** rng.uniform(0.0, 3.0, nbin), mu_zenith=0.67, edd=0.5, ag0=0.0,
                hc=1.98644582e-9, f_diurnal=1.0)


def close(a, b, tol):
    a, b = a.cpu().numpy(), np.asarray(b)
    assert a.shape == b.shape
    scale = np.abs(b).max(axis=0, keepdims=True)
    assert np.all(np.abs(a - b) <= tol * np.maximum(scale, 1e-300))


@pytest.mark.parametrize("nz,nbin,batch,kinds", [
    (2, 3, 1, (4, 2, 1)), (15, 17, 2, (5, 0, 2)), (16, 31, 3, (0, 3, 1)), (17, 33, 1, (6, 2, 0)), (33, 64, 4, (4, 1, 1)),
    (64, 100, 5, (9, 4, 2)), (120, 70, 10, (15, 4, 2)), (125, 40, 1, (15, 4, 2)), (130, 40, 2, (15, 4, 2)),
    (240, 20, 1, (4, 2, 1)), (260, 20, 1, (4, 2, 1)), (40, 40, 1, (40, 20, 9))])
def test_update_at_tile_edges(nz, nbin, batch, kinds):
    rng = np.random.default_rng(nz + nbin)
    ni = 70
    ph = tables(rng, nz, nbin, *kinds, ni)
    dev = photo.PhotoDevice(ph, nz)
    y = 10.0 ** rng.uniform(8.0, 16.0, (batch, nz, ni))
    ymix = y / y.sum(axis=2, keepdims=True)
    dz = 10.0 ** rng.uniform(5.5, 6.5, (batch, nz))
    prev = rng.uniform(0.0, 0.1, (batch, nz + 1, nbin)) * ph["sflux_top"]
    k = rng.uniform(0.0, 1.0, (batch, 12, nz))
    tau = photo.compute_tau_jax(y, dz, dev)
    af, sf, dd, du = photo.compute_flux_jax(tau, ymix, dev, prev)
    J, JT = photo.compute_J_jax_flat(af, dev)
    carry = photo.PhotoCarry(dev, batch, nz, dflux_u=prev)
    due = torch.as_tensor(np.arange(batch) % 3 != 1, dtype=torch.int32, device="cuda")
    kd = torch.as_tensor(k, device="cuda")
    yd, xd = torch.as_tensor(y, device="cuda"), torch.as_tensor(ymix, device="cuda")
    photo.photo_branch(carry, yd, xd, dz, kd, dev, due=due)
    for b in range(batch):
        close(tau[b], orc.compute_tau(y[b], dz[b], ph), 1e-12)
        # each later kernel against the oracle on the GPU's own input
        r = orc.compute_flux(tau[b].cpu().numpy(), ymix[b], ph, prev[b])
        for got, ref, tol in zip((af[b], sf[b], dd[b], du[b]), r, (1e-11, 1e-12, 1e-11, 1e-11)):
            close(got, ref, tol)
        rJ, rJT = orc.compute_J(af[b].cpu().numpy(), ph)
        assert np.allclose(J[b].cpu().numpy(), rJ, rtol=1e-12, atol=0.0)
        assert np.allclose(JT[b].cpu().numpy(), rJT, rtol=1e-12, atol=0.0)
        if due[b]:
            assert torch.equal(carry.tau[b], tau[b]) and torch.equal(carry.aflux[b], af[b])
            assert torch.equal(carry.dflux_u[b], du[b]) and torch.equal(carry.J_br[b], J[b])
            assert torch.equal(kd[b, 1:8], J[b]) and torch.equal(kd[b, 8:11], JT[b])
        else:
            assert np.array_equal(kd[b].cpu().numpy(), k[b]) and not bool(carry.tau[b].any())
            assert np.array_equal(carry.dflux_u[b].cpu().numpy(), prev[b])

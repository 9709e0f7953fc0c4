"""The shapes a batch of columns takes in the optical-depth and flux kernels:
tiles of 32 and 16 bins with 512, 256 and 128 threads, and a thread per bin for
many short columns. The arithmetic of a value is the same in all of them, so
every atmosphere of a batch equals its own call on a batch of one bit for bit
(that call against the oracle: test_gpu_photo_tiles)."""
import numpy as np
import pytest
import torch

from conftest import load_pkg

pytestmark = pytest.mark.gpu

photo = load_pkg("photo")


@pytest.mark.parametrize("nz,batch", [
    (2, 9), (2, 300), (3, 620), (5, 601), (9, 2400),        # tiles of 128 threads, then a thread per bin
    (13, 600), (20, 150), (20, 601), (43, 90), (43, 301),   # 32 bins by 128 and 256 threads
    (64, 160), (120, 90),                                   # by 512 (one tile per SM)
    (126, 160), (150, 90), (240, 90)])                      # 16 bins by 256 and 512
def test_batch_equals_single(nz, batch):
    rng = np.random.default_rng(nz)
    nbin, ni = 70, 24
    cross = lambda *s: 10.0 ** rng.uniform(-24.0, -18.0, s)   # noqa: E731
    ph = dict(absp_idx=np.arange(15), absp_cross=cross(15, nbin), absp_T_idx=np.arange(15, 17),
              absp_T_cross=cross(2, nz, nbin), scat_idx=np.arange(17, 19), scat_cross=cross(2, nbin), din12_indx=20,
              dbin1=0.125, dbin2=0.5, bins=2.0 + np.arange(nbin) * 0.5, sflux_top=10.0 ** rng.uniform(0.0, 3.0, nbin),
              mu_zenith=0.67, edd=0.5, ag0=0.0, hc=1.98644582e-9)
    dev = photo.PhotoDevice(ph, nz)
    cuda = lambda a: torch.as_tensor(a, device="cuda")        # noqa: E731
    y = cuda(10.0 ** rng.uniform(8.0, 16.0, (3, nz, ni)))
    ymix = y / y.sum(dim=2, keepdim=True)
    dz = cuda(10.0 ** rng.uniform(5.5, 6.5, (3, nz)))
    prev = cuda(rng.uniform(0.0, 0.1, (3, nz + 1, nbin)) * ph["sflux_top"])
    pick = torch.arange(batch, device="cuda") % 3
    tau = photo.compute_tau_jax(y[pick], dz[pick], dev)
    out = (tau,) + photo.compute_flux_jax(tau, ymix[pick], dev, prev[pick])
    for b in range(3):
        t1 = photo.compute_tau_jax(y[b], dz[b], dev)
        one = (t1,) + photo.compute_flux_jax(t1, ymix[b], dev, prev[b])
        for a, e in zip(out, one):
            assert torch.equal(a[b::3], e.expand_as(a[b::3]))

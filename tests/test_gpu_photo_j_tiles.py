"""The J kernel's tiles of layers: batches that fill the GPU and do not take
tiles of atmospheres, because each atmosphere has its own temperature-dependent
cross sections, or because four flux rows exceed shared memory (tiles of three
and two layers); against the oracle within the photochemistry tests' 1e-12."""
import numpy as np
import pytest
import torch

from conftest import load_pkg
from oracle import photo as orc

pytestmark = pytest.mark.gpu

photo = load_pkg("photo")


@pytest.mark.parametrize("batch,nz,nbin,own", [
    (30, 41, 60, True), (30, 40, 60, True),      # four layers, a part tile and none
    (30, 41, 7000, False),                       # three
    (30, 41, 9000, True), (30, 41, 9000, False)])   # two
def test_layer_tiles(batch, nz, nbin, own):
    rng = np.random.default_rng(nbin)
    cross = lambda *s: 10.0 ** rng.uniform(-24.0, -18.0, s)   # noqa: E731
    tabs = cross(batch if own else 1, 3, nz, nbin)
    ph = dict(absp_idx=np.arange(2), absp_cross=cross(2, nbin), absp_T_idx=np.zeros(0, int),
              absp_T_cross=np.zeros((0, nz, nbin)), scat_idx=np.arange(2, 3), scat_cross=cross(1, nbin),
              cross_J=cross(7, nbin), cross_J_T=tabs[0], branch_re_idx=np.arange(1, 8),
              branch_T_re_idx=np.arange(8, 11), din12_indx=nbin // 3, dbin1=0.125, dbin2=0.5,
              bins=2.0 + np.arange(nbin) * 0.5, sflux_top=np.ones(nbin), mu_zenith=0.67, edd=0.5, ag0=0.0,
              hc=1.98644582e-9, f_diurnal=1.0)
    dev = photo.PhotoDevice(ph, nz)
    if own:
        dev.keep["cross_J_T"] = torch.as_tensor(tabs, device="cuda")
        dev.struct.cross_J_T = dev.keep["cross_J_T"].data_ptr()
        dev.struct.T_stride_J = 3 * nz * nbin
    aflux = torch.as_tensor(10.0 ** rng.uniform(0.0, 12.0, (batch, nz, nbin)), device="cuda")
    J, JT = photo.compute_J_jax_flat(aflux, dev)
    for b in (0, 1, batch - 1):
        rJ, rJT = orc.compute_J(aflux[b].cpu().numpy(), dict(ph, cross_J_T=tabs[b if own else 0]))
        assert np.allclose(J[b].cpu().numpy(), rJ, rtol=1e-12, atol=0.0)
        assert np.allclose(JT[b].cpu().numpy(), rJT, rtol=1e-12, atol=0.0)

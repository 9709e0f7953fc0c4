"""J rates of a batch whose atmospheres are due at different times: the tiles of
four atmospheres hold due ones only, whatever their places and number (batches
below, at and above the block's 256 threads, part tiles, one, none or all due).
Due atmospheres equal an update of all of them bit for bit, the others keep
their rows."""
import numpy as np
import pytest
import torch

from conftest import load_pkg

pytestmark = pytest.mark.gpu

photo = load_pkg("photo")


def update(batch, nz, nbin, n_br=7, n_br_T=3):
    rng = np.random.default_rng(batch)
    ni = 12
    cross = lambda *s: 10.0 ** rng.uniform(-24.0, -18.0, s)   # noqa: E731
    ph = dict(absp_idx=np.arange(4), absp_cross=cross(4, nbin), absp_T_idx=np.arange(4, 5),
              absp_T_cross=cross(1, nz, nbin), scat_idx=np.arange(5, 6), scat_cross=cross(1, nbin),
              cross_J=cross(n_br, nbin), cross_J_T=cross(n_br_T, nz, nbin), branch_re_idx=np.arange(1, 1 + n_br),
              branch_T_re_idx=np.arange(1 + n_br, 1 + n_br + n_br_T), din12_indx=nbin // 3, dbin1=0.125, dbin2=0.5,
              bins=2.0 + np.arange(nbin) * 0.5, sflux_top=10.0 ** rng.uniform(0.0, 3.0, nbin), mu_zenith=0.67, edd=0.5,
              ag0=0.0, hc=1.98644582e-9, f_diurnal=1.0)
    dev = photo.PhotoDevice(ph, nz)
    y = torch.as_tensor(10.0 ** rng.uniform(8.0, 16.0, (batch, nz, ni)), device="cuda")
    ymix = y / y.sum(dim=2, keepdim=True)
    dz = torch.as_tensor(10.0 ** rng.uniform(5.5, 6.5, (batch, nz)), device="cuda")
    k0 = torch.as_tensor(rng.uniform(0.0, 1.0, (batch, n_br + n_br_T + 2, nz)), device="cuda")
    carry = photo.PhotoCarry(dev, batch, nz)

    def run(due):
        k = k0.clone()
        carry.J_br.zero_()
        carry.J_br_T.zero_()
        carry.dflux_u.zero_()
        photo.photo_branch(carry, y, ymix, dz, k, dev, due=due)
        return k, carry.J_br.clone(), carry.J_br_T.clone()

    return run, k0


@pytest.mark.parametrize("batch,nz", [(4, 300), (7, 300), (30, 40), (255, 5), (256, 5), (257, 5), (1100, 5)])
def test_due_atmospheres(batch, nz):
    run, k0 = update(batch, nz, 33)
    full = run(None)
    rng = np.random.default_rng(1)
    masks = [np.zeros(batch), np.ones(batch), np.arange(batch) == batch - 1, np.arange(batch) % 4 == 2,
             rng.random(batch) < 0.3, rng.random(batch) < 0.9]
    for m in masks:
        due = torch.as_tensor(np.asarray(m, np.int32) * 5, device="cuda")   # any nonzero word is due
        on = due != 0
        k, J, JT = run(due)
        assert torch.equal(k[on], full[0][on]) and torch.equal(k[~on], k0[~on])
        assert torch.equal(J[on], full[1][on]) and torch.equal(JT[on], full[2][on])
        assert not bool(J[~on].any()) and not bool(JT[~on].any())

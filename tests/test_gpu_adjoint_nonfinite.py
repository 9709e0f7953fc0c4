"""A lambda that is not finite shows in every transport-leaf cotangent, those of
the boundary fluxes and the deposition velocity too when the atmosphere has
none (their derivative is then 0 lambda, as in the reference's products)."""
import numpy as np
import pytest
import torch

from conftest import load_pkg

pytestmark = pytest.mark.gpu

chem = load_pkg("chem")
jstep = load_pkg("jax_step")
ssg = load_pkg("steady_state_grad")
syn = load_pkg("synthetic")


@pytest.mark.parametrize("fluxes", [False, True])
def test_nan_state_gives_nan_leaves(fluxes):
    net = syn.make_network(7, 12, 72)
    c = syn.make_case(seed=8, net=net, nz=9, mild=True, k_range=(-12.0, 4.0), fluxes=fluxes)
    atm, dn = jstep.atm_from_dict(c.atm), chem.to_device(net.tables)
    v = np.ones_like(c.y)
    good = ssg.implicit_cotangents(c.y, c.k, atm, dn, v)
    y = np.array(c.y)
    y[4, 3] = np.nan
    bad = ssg.implicit_cotangents(y, c.k, atm, dn, v)
    for name in ("top_flux", "bot_flux", "bot_vdep"):
        assert bool(torch.isfinite(good[name]).all())
        assert bool(good[name].any()) == fluxes
        assert bool(torch.isnan(bad[name]).all()), name

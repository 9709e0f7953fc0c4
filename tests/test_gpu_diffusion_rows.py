"""The step's diffusion rows (fields staged per block of layers) with zero
numerators and layers of no gas, against the layer-by-layer diffusion kernel,
which reads them in place: without reactions the residual is the diffusion
term, so the two are equal value for value, NaN for NaN. Layer counts around
the rows kernel's blocks of eight."""
import numpy as np
import pytest
import torch

from conftest import load_pkg

pytestmark = pytest.mark.gpu

chem = load_pkg("chem")
jstep = load_pkg("jax_step")
ssg = load_pkg("steady_state_grad")
syn = load_pkg("synthetic")


@pytest.mark.parametrize("empty_layer", [False, True])
@pytest.mark.parametrize("share", [0.0, 0.5, 1.0])
@pytest.mark.parametrize("nz", [2, 8, 9, 17])
def test_rows_equal_layer_kernel(nz, share, empty_layer):
    net = syn.make_network(3, 21, 60)
    c = syn.make_case(seed=4, net=net, nz=nz, mild=True, k_range=(-12.0, 4.0), dt=1e-5, moldiff=True, advection=True,
                      fluxes=True)
    g = np.random.default_rng(5)
    atm = dict(c.atm)
    for f in ("Dzz", "vm", "vs", "alpha", "vz"):
        a = np.array(atm[f], float)
        a *= g.choice([-1.0, 1.0], a.shape) if f in ("vm", "vs", "vz") else 1.0
        a[g.random(a.shape) < share] = 0.0
        atm[f] = a
    y = np.array(c.y)
    if empty_layer:
        y[nz // 2] = 0.0
    a = jstep.atm_from_dict(atm)
    rows = ssg.residual(y, np.zeros_like(c.k), a, chem.to_device(net.tables))
    diff = jstep.diffusion(y, a)[0]
    np.testing.assert_array_equal(rows.cpu().numpy(), diff.cpu().numpy())
    assert bool(torch.isfinite(rows).all()) != empty_layer

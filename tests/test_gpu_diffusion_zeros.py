"""Zero numerators in the diffusion stencil (no wind, settling or molecular
diffusion in part of the entries) take a product in place of the quotient:
value for value as the oracle's, with a layer of no gas (quotients by zero) too."""
import numpy as np
import pytest

from conftest import load_pkg
from oracle import ros2 as oracle

pytestmark = pytest.mark.gpu

jstep = load_pkg("jax_step")
syn = load_pkg("synthetic")


@pytest.mark.parametrize("empty_layer", [None, 0, 4, 10])
@pytest.mark.parametrize("share", [0.0, 0.5, 1.0])
def test_zero_numerators(share, empty_layer):
    net = syn.make_network(3, 21, 60)
    c = syn.make_case(seed=4, net=net, nz=11, mild=True, k_range=(-12.0, 4.0), dt=1e-5, moldiff=True, advection=True,
                      fluxes=True)
    g = np.random.default_rng(5)
    atm = dict(c.atm)
    for f in ("Dzz", "vm", "vs", "alpha", "vz"):
        a = np.array(atm[f], float)
        a *= g.choice([-1.0, 1.0], a.shape) if f in ("vm", "vs", "vz") else 1.0
        a[g.random(a.shape) < share] = 0.0
        atm[f] = a
    y = np.array(c.y)
    if empty_layer is not None:
        y[empty_layer] = 0.0
    with np.errstate(all="ignore"):
        co = oracle.build_diff_coeffs(y, atm, oracle.compute_diff_grav(atm))
        ref = oracle.apply_diffusion(y, *co[:6], atm)
    diff, _, sup, sub = jstep.diffusion(y, jstep.atm_from_dict(atm))
    A_e, B_e, C_e, A_m, B_m, C_m, _ = co
    np.testing.assert_array_equal(diff.cpu().numpy(), ref)
    np.testing.assert_array_equal(sup.cpu().numpy(), B_e[:-1, None] + B_m[:-1])
    np.testing.assert_array_equal(sub.cpu().numpy(), C_e[1:, None] + C_m[1:])

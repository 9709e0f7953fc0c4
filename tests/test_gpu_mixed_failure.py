"""The mixed step's sweeps when their waits on the bulk copies give up at once
(``set_wait_limit(0)``): every atmosphere gets VB_STATUS_WATCHDOG, the kernels
return after draining their copies, and with the limit restored the next step
equals the first bit for bit. Blocks small and large enough for rings of many
stages and of two."""
import numpy as np
import pytest

from conftest import load_pkg

pytestmark = pytest.mark.gpu

chem = load_pkg("chem")
jstep = load_pkg("jax_step")
syn = load_pkg("synthetic")

WATCHDOG = 8


@pytest.mark.parametrize("ni", [12, 69, 96])
def test_wait_limit_gives_watchdog_status_and_recovers(ni):
    net = syn.make_network(41, ni, 6 * ni, elements=("C", "H", "O", "N", "S") if ni > 77 else ("C", "H", "O", "N"))
    cases = [syn.make_case(seed=500 + b, net=net, nz=12, mild=True, k_range=(-12.0, 4.0)) for b in range(3)]
    A = {k: (v if isinstance(v, bool) else np.stack([c.atm[k] for c in cases])) for k, v in cases[0].atm.items()}
    step = jstep.Ros2Step(chem.to_device(net.tables), jstep.atm_from_dict(A), mixed=True)
    args = np.stack([c.y for c in cases]), np.stack([c.k for c in cases]), np.full(3, 1e-6)

    def run():
        return [t.cpu().numpy().copy() for t in step(*args)]

    sol0, delta0, st0 = run()
    assert not st0.any()
    try:
        jstep.set_wait_limit(0)
        st = run()[2]
    finally:
        jstep.set_wait_limit(None)
    assert (st & WATCHDOG).all(), st
    sol, delta, st2 = run()
    assert not st2.any()
    assert np.array_equal(sol, sol0) and np.array_equal(delta, delta0)

"""The adjoint's assembly with one and with two layers per CTA (two is the
automatic choice for large batches): its block stores, deposition term and
right-hand-side copy give the same bits, for odd and even layer counts, bottom
fluxes on and off, and for the batch against its atmospheres alone."""
import numpy as np
import pytest
import torch

from conftest import load_pkg

pytestmark = pytest.mark.gpu

at = load_pkg("autotune")
chem = load_pkg("chem")
jstep = load_pkg("jax_step")
ssg = load_pkg("steady_state_grad")
syn = load_pkg("synthetic")


@pytest.mark.parametrize("fluxes", [False, True])
@pytest.mark.parametrize("ni,nz", [(12, 2), (12, 9), (33, 8), (69, 11)])
def test_layers_per_cta(ni, nz, fluxes):
    net = syn.make_network(7 + ni, ni, 5 * ni)
    cases = [syn.make_case(seed=(40, b), net=net, nz=nz, mild=True, k_range=(-12.0, 4.0), moldiff=True, fluxes=fluxes)
             for b in range(3)]
    A = {k: (v if isinstance(v, bool) else np.stack([c.atm[k] for c in cases])) for k, v in cases[0].atm.items()}
    y, k = np.stack([c.y for c in cases]), np.stack([c.k for c in cases])
    v = np.random.default_rng(ni).standard_normal(y.shape) / y
    dn = chem.to_device(net.tables)
    got = []
    for layers in (1, 2):
        at.set_tuning(dn, dict(stage1_layers=layers))
        got.append(ssg.implicit_cotangents(y, k, jstep.atm_from_dict(A), dn, v))
    at.set_tuning(dn, {})
    assert not bool(got[0]["status"].any())
    for name in got[0]:
        assert torch.equal(got[0][name], got[1][name]), name
    one = ssg.implicit_cotangents(cases[1].y, cases[1].k, jstep.atm_from_dict(cases[1].atm), dn, v[1])
    for name in ("lambda", "k_arr", "Dzz", "bot_vdep"):
        assert torch.equal(one[name], got[1][name][1]), name

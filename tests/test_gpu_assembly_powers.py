"""The thread-per-layer stage 2 of networks whose slots need pow here and there,
everywhere, nowhere, or at the ends of the reaction chunks: the same bits as the
per-layer kernel, for few and for up to eight terms, one chunk and many."""
import types

import numpy as np
import pytest
import torch

from conftest import load_pkg

pytestmark = pytest.mark.gpu

chem = load_pkg("chem")
jstep = load_pkg("jax_step")
syn = load_pkg("synthetic")


@pytest.mark.parametrize("share", [0.0, 0.02, 1.0])
@pytest.mark.parametrize("ni,nr,T", [(5, 7, 1), (20, 40, 2), (33, 900, 4), (33, 901, 7), (20, 300, 8)])
def test_thread_per_layer_equals_per_layer(ni, nr, T, share):
    g = np.random.default_rng(nr + T)
    shape = (nr + 1, T)
    idx = [g.integers(0, ni, shape) for _ in range(2)]
    st = [g.choice((1.0, 2.0), shape) for _ in range(2)]
    pw = g.random(nr + 1) < share
    pw[[1, nr]] = share > 0.0
    st[0][pw, 0] = g.choice((0.5, 3.0), int(pw.sum()))
    for i, s in zip(idx, st):
        off = g.random(shape) < 0.4
        off[:, 0], off[0] = False, True
        i[off], s[off] = ni, 0.0
    net = types.SimpleNamespace(ni=ni, nr=nr, reactant_idx=idx[0], product_idx=idx[1], reactant_stoich=st[0],
                                product_stoich=st[1], is_three_body=g.random(nr + 1) < 0.3)
    dn = chem.to_device(net)
    b, nz = 2, 13
    a0, _ = syn.make_atmosphere(0, syn.make_network(0, 12, 60), nz=nz)
    atm = {k: (v if isinstance(v, bool) else np.asarray(v, float)) for k, v in a0.items()
           if k in jstep.AtmStatic._fields}
    for k, shp in (("Dzz", (nz - 1, ni)), ("vm", (nz, ni)), ("vs", (nz - 1, ni)), ("alpha", (ni,)), ("top_flux", (ni,)),
                   ("bot_flux", (ni,)), ("bot_vdep", (ni,))):
        atm[k] = np.zeros(shp)
    atm["ms"], atm["gas_indx_mask"], atm["M"] = np.ones(ni), np.ones(ni, bool), np.ones(nz)
    A = jstep.atm_from_dict({k: (v if isinstance(v, bool) else np.stack([v] * b)) for k, v in atm.items()})
    y, k = g.uniform(0.2, 3.0, (b, nz, ni)), g.uniform(0.1, 1.0, (b, nr + 1, nz)) * 1e-3
    dt = np.full(b, 1e-12)   # the second stage stays positive: pow of a negative number is NaN
    lv, pl = ([t.clone() for t in jstep.Ros2Step(dn, A, assembly=on)(y, k, dt)] for on in (True, False))
    for p, q in zip(lv, pl):
        assert torch.equal(p, q)
    assert bool(torch.isfinite(lv[0]).all()) and not bool(lv[2].any())

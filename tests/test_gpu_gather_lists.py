"""The gather lists of the chemistry kernels: packed coefficients and the
coefficient table, packed reaction words (up to six terms) and the wide tables,
lists from empty to longer than the words held ahead, and species counts
around the groups of 32.

Networks of stoichiometries 0, 1 and 2 involve no pow on the device and equal
the oracle bit for bit once it squares by a product too (NumPy's y ** 2.0 of an
array of exponents is y * y only to the last place). Others differ by pow: at most 3 units in the last place per power
between the device's and NumPy's, T powers in a term, which changes a term by
at most 6 T eps with the roundings of its products, so a sum of n terms moves
by at most n (6 T + n) eps times its largest term."""
import functools
import types

import numpy as np
import pytest
import torch

from conftest import load_pkg
from oracle import ros2 as oracle

pytestmark = pytest.mark.gpu

_at = load_pkg("autotune")
chem = load_pkg("chem")
jstep = load_pkg("jax_step")
syn = load_pkg("synthetic")

WHOLE = (1.0, 2.0)
OTHER = (1.0, 2.0, 3.0, 0.5, 1.0 / 3.0)


def squared_factors(y, net, plain):
    """The oracle's factors with squares as products."""
    y_r, f = plain(y, net)
    return y_r, np.where(net.reactant_stoich[None] == 2.0, y_r * y_r, f)


def random_net(ni, nr, T, values, seed):
    g = np.random.default_rng(seed)
    shape = (nr + 1, T)
    hub = lambda: np.where(g.random(shape) < 0.3, g.integers(0, min(ni, 3), shape), g.integers(0, ni, shape))
    r, p = hub(), hub()
    rs, ps = g.choice(values, shape), g.choice(values, shape)
    for idx, st in ((r, rs), (p, ps)):
        off = g.random(shape) < 0.4
        off[0] = True   # the padding reaction
        idx[off], st[off] = ni, 0.0
    return types.SimpleNamespace(ni=ni, nr=nr, reactant_idx=r, product_idx=p, reactant_stoich=rs, product_stoich=ps,
                                 is_three_body=g.random(nr + 1) < 0.3)


def term_bounds(y, M, k, net):
    """Largest terms of the sums and of the Jacobian entries, per layer."""
    T = net.reactant_idx.shape[1]
    y_r, f = oracle._factors(y, net)
    st = net.reactant_stoich[None]
    lo = np.stack([np.prod(np.where(np.arange(T) == s, 1.0, f), axis=2) for s in range(T)], axis=2)
    d = np.abs(st * np.where(st > 0, y_r ** (st - 1.0), 0.0) * lo * k.T[:, :, None])
    d = np.where(net.is_three_body[None, :, None], d * M[:, None, None], d)
    c = max(net.reactant_stoich.max(), net.product_stoich.max())
    return c * oracle.rates(y, M, k, net).max(axis=1), c * d.max(axis=(1, 2))


@pytest.mark.parametrize("ni,nr,T,values", [
    (1, 3, 1, WHOLE), (5, 40, 2, WHOLE), (16, 30, 3, WHOLE), (33, 200, 3, WHOLE), (69, 1400, 3, WHOLE),
    (40, 60, 6, WHOLE), (40, 60, 7, WHOLE), (128, 500, 8, WHOLE), (5, 40, 2, OTHER), (33, 200, 3, OTHER),
    (64, 300, 6, OTHER), (40, 60, 7, OTHER)])
def test_rhs_and_jacobian(ni, nr, T, values, monkeypatch):
    net = random_net(ni, nr, T, values, seed=ni + T)
    g = np.random.default_rng(1)
    nz = 5
    y, M, k = g.uniform(0.2, 3.0, (nz, ni)), g.uniform(0.5, 2.0, nz), g.uniform(0.1, 1.0, (nr + 1, nz))
    dn = chem.to_device(net)
    got = chem.chem_rhs(y, M, k, dn).cpu().numpy(), chem.chem_jac_analytical(y, M, k, dn).cpu().numpy()
    b_rhs, b_jac = term_bounds(y, M, k, net)
    monkeypatch.setattr(oracle, "_factors", functools.partial(squared_factors, plain=oracle._factors))
    want = oracle.chem_rhs(y, M, k, net), oracle.chem_jac(y, M, k, net)
    if values is WHOLE:
        assert np.array_equal(got[0], want[0]) and np.array_equal(got[1], want[1])
        return
    eps, n = 2.0 ** -52, nr * T
    assert np.all(np.abs(got[0] - want[0]) <= n * (6 * T + n) * eps * b_rhs[:, None])
    assert np.all(np.abs(got[1] - want[1]) <= n * T * (6 * T + n * T) * eps * b_jac[:, None, None])


@pytest.mark.parametrize("third", [False, True])
@pytest.mark.parametrize("ni", [12, 33, 69])
def test_step_layers_per_block(ni, third):
    """One and two layers per CTA give the same bits, packed coefficients or
    not (a third product coefficient makes a network's table unpackable), and
    the step equals the oracle's."""
    net = syn.make_network(7 + ni, ni, 5 * ni)
    c = syn.make_case(seed=8, net=net, nz=9, mild=True, k_range=(-12.0, 4.0), dt=1e-5)
    if third:
        net.tables.product_stoich[1, 0] = 1.0 / 3.0
    dn = chem.to_device(net.tables)
    step = jstep.Ros2Step(dn, jstep.atm_from_dict(c.atm))
    one = [t.clone() for t in step(c.y, c.k, c.dt)]
    _at.set_tuning(dn, dict(stage1_layers=2))
    two = step(c.y, c.k, c.dt)
    assert all(torch.equal(a, b) for a, b in zip(one, two))
    sol, _ = oracle.ros2_step(c.y, c.k, c.dt, c.atm, net.tables)[:2]
    assert np.allclose(one[0].cpu().numpy().reshape(sol.shape), sol, rtol=1e-9, atol=1e-9 * np.abs(sol).max())


@pytest.mark.parametrize("ni,change", [(12, None), (33, "coefficient"), (33, "power"), (69, "power")])
def test_stage2_tiles(ni, change):
    """A batch of enough layers takes the tiled stage 2 (whole and part tiles of
    eight layers); every atmosphere equals its own step, which does not."""
    net = syn.make_network(11 + ni, ni, 5 * ni)
    if change == "coefficient":
        net.tables.product_stoich[1, 0] = 1.0 / 3.0
    if change == "power":
        net.tables.reactant_stoich[2, 0] = 3.0
        net.tables.reactant_stoich[4, 0] = 0.5
    dn = chem.to_device(net.tables)
    cases = [syn.make_case(seed=20 + nz, net=net, nz=nz, mild=True, k_range=(-12.0, 4.0), dt=1e-5)
             for nz in (3, 7, 8, 9, 16, 17)]
    many = cases * 50
    step = jstep.RaggedRos2Step(dn, [jstep.atm_from_dict(c.atm) for c in many])
    y, k = step.pack([c.y for c in many], [c.k for c in many])
    sol, delta, _ = step(y, k, torch.full((len(many),), 1e-5, dtype=torch.float64, device="cuda"))
    alone = [[t.clone() for t in jstep.jax_ros2_step(c.y, c.k, 1e-5, jstep.atm_from_dict(c.atm), dn)] for c in cases]
    for b, (s, d) in enumerate(zip(step.unpack(sol), step.unpack(delta))):
        s1, d1 = alone[b % len(cases)]
        assert torch.equal(s, s1) and torch.equal(d, d1), b

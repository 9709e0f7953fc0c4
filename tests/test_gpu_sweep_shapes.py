"""The sweeps at the edges of their eight-row warps and of the copy ring: the
mixed-precision step's first and refinement passes against the FP64 step's
solves, from two layers up (the forward stream turns into the backward one
after nz - 1 blocks), and the FP64 step with every ring depth, bit for bit.
Bound of the mixed solves: refinement stops at corrections of 1e-12 of the
solution and these systems are well conditioned, 1e-10 normwise. The block
solver's own shapes, up to rings of one stage, are in
test_gpu_panel_factor.py."""
import numpy as np
import pytest
import torch

from conftest import load_pkg

pytestmark = pytest.mark.gpu

_at = load_pkg("autotune")
chem = load_pkg("chem")
jstep = load_pkg("jax_step")
syn = load_pkg("synthetic")


def case_of(ni, nz):
    net = syn.make_network(90 + ni, ni, 5 * ni)
    return net, syn.make_case(seed=91, net=net, nz=nz, mild=True, k_range=(-12.0, 4.0), dt=1e-5)


@pytest.mark.parametrize("ni,nz", [(12, 2), (12, 3), (12, 4), (15, 5), (16, 6), (17, 7), (31, 8), (33, 3), (40, 9),
                                   (41, 2), (64, 4), (65, 12), (72, 5), (73, 3)])
def test_mixed_sweeps(ni, nz):
    net, c = case_of(ni, nz)
    dn = chem.to_device(net.tables)
    atm = jstep.atm_from_dict(c.atm)
    ref, mix = jstep.Ros2Step(dn, atm), jstep.Ros2Step(dn, atm, mixed=True)
    ref(c.y, c.k, c.dt)
    _, _, status = mix(c.y, c.k, c.dt)
    assert int(status[0]) == 0
    for a, b in zip(ref.stages(), mix.stages()):
        assert float((a - b).abs().max()) <= 1e-10 * float(a.abs().max())


@pytest.mark.parametrize("ni,nz", [(15, 2), (24, 5), (69, 3), (69, 20), (72, 9)])
def test_ring_depths_bit_for_bit(ni, nz):
    net, c = case_of(ni, nz)
    dn = chem.to_device(net.tables)
    step = jstep.Ros2Step(dn, jstep.atm_from_dict(c.atm))
    want = [t.clone() for t in step(c.y, c.k, c.dt)]
    for stages in (1, 2, 3):
        _at.set_tuning(dn, dict(sweep_stages=stages))
        got = step(c.y, c.k, c.dt)
        assert all(torch.equal(a, b) for a, b in zip(want, got)), stages

"""The rate region of the stage-2 assembly is allocated only where it is read:
not for batches whose stage 2 goes by tiles, also as two halves on two streams,
and still for those whose halves are too small for tiles. The results do not
depend on it."""
import numpy as np
import pytest
import torch

from conftest import load_pkg

pytestmark = pytest.mark.gpu

_lib = load_pkg("_lib")
at = load_pkg("autotune")
chem = load_pkg("chem")
jstep = load_pkg("jax_step")
syn = load_pkg("synthetic")

NI, NZ = 20, 24   # three tiles of eight layers per atmosphere


@pytest.fixture(scope="module")
def net():
    return syn.make_network(5, NI, 120)


def inputs(net, batch):
    cases = [syn.make_case(seed=(30, b), net=net, nz=NZ, mild=True, k_range=(-12.0, 4.0), dt=1e-5) for b in range(4)]
    pick = [cases[b % 4] for b in range(batch)]
    A = {k: (v if isinstance(v, bool) else np.stack([c.atm[k] for c in pick])) for k, v in cases[0].atm.items()}
    dev = lambda f: torch.as_tensor(np.stack([getattr(c, f) for c in pick]), device="cuda")   # noqa: E731
    return jstep.atm_from_dict(A), dev("y"), dev("k"), torch.full((batch,), 1e-5, dtype=torch.float64, device="cuda")


def sms():
    return torch.cuda.get_device_properties(0).multi_processor_count


@pytest.mark.parametrize("mixed", [False, True])
@pytest.mark.parametrize("size", ["below", "whole", "halves"])
def test_region_only_where_used(net, size, mixed):
    tiles = 2 * sms()   # a stage 2 by tiles needs this many
    batch = {"below": tiles // 3 // 2, "whole": tiles // 3 + 2, "halves": 2 * (tiles // 3 + 2) + 1}[size]
    atm, y, k, dt = inputs(net, batch)
    dn = chem.to_device(net.tables)
    L = _lib.lib()
    own = int((L.vb_ros2_mixed_workspace_bytes if mixed else L.vb_ros2_workspace_bytes)(batch, NZ, NI, None))
    region = batch * NZ * (dn.nr + 1) * 8
    step = jstep.Ros2Step(dn, atm, mixed=mixed)
    assert step.ws_bytes == (own if size == "halves" else ((own + 255) & ~255) + region)
    plain = jstep.Ros2Step(dn, atm, mixed=mixed, assembly=False)
    ref = [t.clone() for t in plain(y, k, dt)]
    for streams in (1, 2):
        at.set_tuning(dn, dict(streams=streams))
        assert all(torch.equal(a, b) for a, b in zip(step(y, k, dt), ref))


def test_ragged_workspace_is_packed(net):
    batch = 2 * (2 * sms() // 3 + 2)
    cases = [syn.make_case(seed=(31, nz), net=net, nz=nz, mild=True, k_range=(-12.0, 4.0), dt=1e-5) for nz in (9, 24)]
    many = [cases[b % 2] for b in range(batch)]
    dn = chem.to_device(net.tables)
    step = jstep.RaggedRos2Step(dn, [jstep.atm_from_dict(c.atm) for c in many])
    assert step.ws_bytes == int(_lib.lib().vb_ros2_workspace_bytes(batch, NZ, NI, step.zoff_host.ctypes.data))
    y, k = step.pack([c.y for c in many], [c.k for c in many])
    sol, delta, _ = step(y, k, np.full(batch, 1e-5))
    for c, s, d in list(zip(many, step.unpack(sol), step.unpack(delta)))[:2]:
        s1, d1 = jstep.jax_ros2_step(c.y, c.k, 1e-5, jstep.atm_from_dict(c.atm), dn)[:2]
        assert torch.equal(s, s1) and torch.equal(d, d1)

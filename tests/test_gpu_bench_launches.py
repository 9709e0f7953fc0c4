"""The benchmark's launch count is the step's own, on every path of its stage 2:
by tiles, with a thread per layer (two kernels), per layer, for halves of an odd
batch that go different ways, and for a network whose rates exceed a tile's
shared memory."""
import numpy as np
import pytest
import torch

import bench
from conftest import load_pkg

pytestmark = pytest.mark.gpu

at = load_pkg("autotune")
chem = load_pkg("chem")
jstep = load_pkg("jax_step")
syn = load_pkg("synthetic")

NZ = 8   # one tile of eight layers per atmosphere


def launches(dn, case, batch, tuning=None, **kw):
    A = {k: (v if isinstance(v, bool) else np.stack([v] * batch)) for k, v in case.atm.items()}
    step = jstep.Ros2Step(dn, jstep.atm_from_dict(A), **kw)
    y, k = (torch.as_tensor(np.stack([v] * batch), device="cuda") for v in (case.y, case.k))
    dt = torch.full((batch,), 1e-5, dtype=torch.float64, device="cuda")
    out = torch.empty_like(y), torch.empty_like(y)
    at.set_tuning(dn, tuning or {})
    step(y, k, dt, out=out)
    n = bench.kernel_launches(torch, lambda: step(y, k, dt, out=out))
    at.set_tuning(dn, {})
    return n


def test_step_launches():
    net = syn.make_network(5, 20, 120)
    dn = chem.to_device(net.tables)
    case = syn.make_case(seed=30, net=net, nz=NZ, mild=True, k_range=(-12.0, 4.0), dt=1e-5)
    full = 2 * torch.cuda.get_device_properties(0).multi_processor_count   # tiles of a stage 2 that goes by tiles
    assert launches(dn, case, 3) == 9
    assert launches(dn, case, 3, assembly=False) == 8
    assert launches(dn, case, full - 1) == 9 and launches(dn, case, full) == 8
    two = dict(streams=2)
    assert launches(dn, case, full, two) == 18
    assert launches(dn, case, 2 * full - 1, two) == 17
    assert launches(dn, case, 2 * full, two) == 16


def test_large_network_launches():
    net = syn.make_network(0, 40, 1760)   # 3,521 slots of 64 bytes: above 220 KB
    dn = chem.to_device(net.tables)
    case = syn.make_case(seed=30, net=net, nz=NZ, mild=True, k_range=(-12.0, 4.0), dt=1e-5)
    full = 2 * torch.cuda.get_device_properties(0).multi_processor_count
    assert launches(dn, case, full) == 9

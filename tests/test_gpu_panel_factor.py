"""The panel Gauss-Jordan factor at the edges of its tiles: block sizes either
side of every panel (8 columns) and of every instantiated panel count, on
blocks that need pivoting, in both orientations (plain and transposed solves).
Each system is compared bit for bit with the pipelined kernel
(``vb_set_factor_kernel(2)``: the same elimination, scalar updates, its own
synchronisation) and, normwise, with NumPy's dense solve within
64 n eps cond(A)."""
import numpy as np
import pytest
import torch

from conftest import load_pkg

pytestmark = pytest.mark.gpu

_lib = load_pkg("_lib")
solver = load_pkg("solver")


def system(rng, batch, nz, ni):
    diag = rng.standard_normal((batch, nz, ni, ni)) + 3.0 * np.eye(ni)
    sup, sub = (0.3 * rng.standard_normal((batch, nz - 1, ni)) for _ in range(2))
    return diag, sup, sub, rng.standard_normal((batch, nz, ni))


def dense(diag, sup, sub):
    nz, ni, _ = diag.shape
    A = np.zeros((nz * ni, nz * ni))
    for j in range(nz):
        A[j * ni:(j + 1) * ni, j * ni:(j + 1) * ni] = diag[j]
    i = np.arange((nz - 1) * ni)
    A[i, i + ni] = sup.reshape(-1)
    A[i + ni, i] = sub.reshape(-1)
    return A


def solve_both(d, su, sb, r, kernel):
    _lib.check(_lib.lib().vb_set_factor_kernel(kernel), "vb_set_factor_kernel")
    try:
        f = solver.factor_block_thomas_diag_offdiag(d, su, sb)
        x = solver.solve_block_thomas_diag_offdiag(f, r)
        xt = solver.solve_block_thomas_diag_offdiag_T(f, r)
    finally:
        _lib.check(_lib.lib().vb_set_factor_kernel(1), "vb_set_factor_kernel")
    return x, xt, f.status


@pytest.mark.parametrize("ni", [1, 2, 7, 8, 9, 16, 17, 23, 24, 25, 31, 32, 33, 47, 48, 49, 63, 64, 65, 69, 71, 72, 73,
                                79, 80, 81, 88, 89, 95, 96, 97, 120, 121, 127, 128])
def test_tile_edges(ni):
    rng = np.random.default_rng(ni)
    d, su, sb, r = system(rng, 2, 3, ni)
    x, xt, st = solve_both(d, su, sb, r, 1)
    y, yt, _ = solve_both(d, su, sb, r, 2)
    assert int(st.abs().sum()) == 0
    assert torch.equal(x, y) and torch.equal(xt, yt)
    for b in range(2):
        A = dense(d[b], su[b], sb[b])
        bound = 64 * ni * np.finfo(float).eps * np.linalg.cond(A)
        for got, M in ((x, A), (xt, A.T)):
            ref = np.linalg.solve(M, r[b].reshape(-1))
            assert np.linalg.norm(got[b].cpu().numpy().reshape(-1) - ref) <= bound * np.linalg.norm(ref)


@pytest.mark.parametrize("ni,batch", [(69, 149), (72, 300), (30, 600), (64, 300)])
def test_more_atmospheres_than_sms(ni, batch):
    """The shapes with several CTAs per SM, a partial last wave."""
    rng = np.random.default_rng(ni)
    d, su, sb, r = (torch.as_tensor(a, device="cuda") for a in system(rng, 3, 4, ni))
    pick = torch.arange(batch, device="cuda") % 3
    x, xt, st = solve_both(d[pick].contiguous(), su[pick].contiguous(), sb[pick].contiguous(), r[pick].contiguous(), 1)
    y, yt, _ = solve_both(d, su, sb, r, 2)
    assert int(st.abs().sum()) == 0
    assert torch.equal(x, y[pick]) and torch.equal(xt, yt[pick])

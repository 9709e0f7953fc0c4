"""Infinite and NaN entries of the diagonal blocks, for every factor kernel.

An infinite diagonal entry (a time step of zero, an infinite deposition
velocity) holds its unknown at zero: the entry is the largest of its column, so
it is the pivot, its row and column of the block's inverse are zero, and the
other unknowns solve the system without it, which NumPy's dense solve gives
within 64 n eps cond(A). A NaN counts as magnitude 0, as a zero does: the
lowest row is taken, and the status is the result's, not a zero pivot's."""
import numpy as np
import pytest
import torch

from conftest import load_pkg

pytestmark = pytest.mark.gpu

_lib = load_pkg("_lib")
chem = load_pkg("chem")
jstep = load_pkg("jax_step")
solver = load_pkg("solver")
syn = load_pkg("synthetic")

ZERO_PIVOT, NONFINITE, REFINE_STALL = 1, 2, 4


def dense(diag, sup, sub):
    nz, ni, _ = diag.shape
    A = np.zeros((nz * ni, nz * ni))
    for j in range(nz):
        A[j * ni:(j + 1) * ni, j * ni:(j + 1) * ni] = diag[j]
    i = np.arange((nz - 1) * ni)
    A[i, i + ni] = sup.reshape(-1)
    A[i + ni, i] = sub.reshape(-1)
    return A


def solve_both(arrays, kernel):
    d, su, sb, r = (torch.as_tensor(a, device="cuda") for a in arrays)
    _lib.check(_lib.lib().vb_set_factor_kernel(kernel), "vb_set_factor_kernel")
    try:
        f = solver.factor_block_thomas_diag_offdiag(d, su, sb)
        return (solver.solve_block_thomas_diag_offdiag(f, r), solver.solve_block_thomas_diag_offdiag_T(f, r),
                f.status.cpu().numpy())
    finally:
        _lib.check(_lib.lib().vb_set_factor_kernel(1), "vb_set_factor_kernel")


@pytest.mark.parametrize("rows", ["one", "all"])
@pytest.mark.parametrize("ni,kernel", [(3, 1), (24, 1), (30, 1), (69, 0), (69, 1), (69, 2), (69, 3), (89, 1), (128, 1)])
def test_infinite_diagonal(ni, kernel, rows):
    rng = np.random.default_rng(ni)
    nz = 3
    diag = 0.1 * rng.standard_normal((2, nz, ni, ni)) / np.sqrt(ni) + 2.0 * np.eye(ni)
    sup, sub = (0.3 * rng.standard_normal((2, nz - 1, ni)) for _ in range(2))
    rhs = rng.standard_normal((2, nz, ni))
    held = [ni // 2] if rows == "one" else list(range(ni))
    diag[0, 1, held, held] = np.where(np.arange(len(held)) % 2 == 0, np.inf, -np.inf)
    x, xt, st = solve_both((diag, sup, sub, rhs), kernel)
    assert not st.any()
    free = np.ones((nz, ni), bool)
    free[1, held] = False
    for b in range(2):
        on = free.reshape(-1) if b == 0 else np.ones(nz * ni, bool)
        A = dense(np.where(np.isinf(diag[b]), 0.0, diag[b]), sup[b], sub[b])
        bound = 64 * ni * np.finfo(float).eps * np.linalg.cond(A[np.ix_(on, on)])
        for got, M in ((x, A), (xt, A.T)):
            g = got[b].cpu().numpy().reshape(-1)
            ref = np.linalg.solve(M[np.ix_(on, on)], rhs[b].reshape(-1)[on])
            assert not g[~on].any()
            assert np.linalg.norm(g[on] - ref) <= bound * np.linalg.norm(ref)


@pytest.mark.parametrize("ni,kernel", [(12, 1), (69, 0), (69, 1), (69, 2), (69, 3), (100, 1)])
def test_nan_is_no_zero_pivot(ni, kernel):
    diag = np.stack([np.full((2, ni), np.nan), np.ones((2, ni))])[..., None] * np.eye(ni)
    diag = np.where(np.eye(ni, dtype=bool), diag, 0.0)
    z = np.zeros((2, 1, ni))
    _, _, st = solve_both((diag, z, z, np.ones((2, 2, ni))), kernel)
    assert st.tolist() == [NONFINITE, 0]


@pytest.mark.parametrize("mixed", [False, True])
@pytest.mark.parametrize("ni", [12, 69])
def test_step_of_no_time(ni, mixed):
    """dt = 0: the blocks' diagonals are infinite, the first stage is zero and
    the second is 0/0: a non-finite result (the mixed step's refinement, which
    cannot reach it, stalls), not a singular matrix."""
    net = syn.make_network(7, ni, 6 * ni)
    c = syn.make_case(seed=8, net=net, nz=9, mild=True, k_range=(-12.0, 4.0), dt=1e-5)
    step = jstep.Ros2Step(chem.to_device(net.tables), jstep.atm_from_dict(c.atm), mixed=mixed)
    _, _, status = step(c.y, c.k, np.zeros(1))
    assert status.tolist() == [NONFINITE | (REFINE_STALL if mixed else 0)]
    if not mixed:
        assert not bool(step.stages()[0].any())

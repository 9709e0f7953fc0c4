"""The transport-leaf cotangents (``vb_adjoint_atm``) at the edges of their
blocks of 8 layers and of their 32-lane species passes, from the two-layer
column up, with gravity and with advection, against autograd of the oracle's
residual at a given lambda. Bound: each cotangent is a sum of at most
3 rows x 40 species (layer fields) or 33 rows (species fields) of terms of ~40
operations each, 1e-10 normwise as for the leaves of the other adjoint tests."""
import numpy as np
import pytest
import torch

from conftest import load_pkg
from oracle import adjoint as oa

pytestmark = pytest.mark.gpu

_lib = load_pkg("_lib")
jstep = load_pkg("jax_step")
ssg = load_pkg("steady_state_grad")
syn = load_pkg("synthetic")


@pytest.mark.parametrize("advection", [False, True], ids=["gravity", "advection"])
@pytest.mark.parametrize("nz,ni", [(2, 12), (3, 12), (7, 31), (8, 32), (9, 33), (16, 40), (17, 12), (33, 12)])
def test_leaves_at_block_edges(nz, ni, advection):
    net = syn.make_network(60 + ni, ni, 4 * ni)
    cases = [syn.make_case(seed=(80, b), net=net, nz=nz, mild=True, k_range=(-40.0, 4.0), moldiff=True, fluxes=True,
                           advection=advection) for b in range(2)]
    A = {kk: (np.stack([c.atm[kk] for c in cases]) if not isinstance(v, bool) else v)
         for kk, v in cases[0].atm.items()}
    atm = jstep.atm_from_dict(A)
    y = torch.as_tensor(np.stack([c.y for c in cases]), device="cuda")
    lam = torch.as_tensor(np.random.default_rng(nz).normal(0.0, 1.0, y.shape), device="cuda") / y
    blob = jstep.pack_atm(atm)
    g = torch.empty_like(blob)
    _lib.check(_lib.lib().vb_adjoint_atm(2, nz, ni, None, _lib.ptr(y), _lib.ptr(blob), jstep.atm_flags(atm),
                                         _lib.ptr(lam), _lib.ptr(g), _lib.stream_handle(None)), "vb_adjoint_atm")
    got = ssg.unpack_atm_cotangents(g, nz, ni)
    for b, c in enumerate(cases):
        ref = oa.vjp_from_lambda(c.y, c.k, c.atm, net.tables, lam[b].cpu().numpy())
        for leaf in oa.LEAVES:
            if leaf in ("k_arr", "M"):
                continue
            v = got["Kzz_transport" if leaf == "Kzz" else leaf][b].cpu().numpy()
            assert v.shape == np.shape(ref[leaf]), leaf
            assert np.abs(v - ref[leaf]).max() <= 1e-10 * np.abs(ref[leaf]).max(), leaf

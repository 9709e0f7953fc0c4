"""Rounding of the transport-leaf cotangents (``vb_adjoint_atm``) where lambda
is nearly the same in neighbouring layers, so the two rows an interface enters
nearly cancel: two layers, whose lambdas differ by 1e-5 of their size (their dz
is the same, so lambda_0/dz_0 - lambda_1/dz_1 is the difference over dz without
any cancellation of its own).

Each leaf of one interface and species is then a product of that difference and
of terms that do not cancel with it, at most 40 roundings: within 64 units of
2^-53 of the sum of its terms' magnitudes, evaluated in NumPy's long double from
the same lambda. A difference of the two rows' rounded products is off by about
1e5 units."""
import numpy as np
import pytest
import torch

from conftest import load_pkg

pytestmark = pytest.mark.gpu

_lib = load_pkg("_lib")
jstep = load_pkg("jax_step")
ssg = load_pkg("steady_state_grad")
syn = load_pkg("synthetic")

L = np.longdouble
BOUND = 64 * L(2.0) ** -53


def leaves(y, atm, lam):
    """{leaf: (value, sum of its terms' magnitudes)} of a two-layer column."""
    f = {k: np.asarray(v, L) for k, v in atm.items() if not isinstance(v, bool)}
    y, lam = np.asarray(y, L), np.asarray(lam, L)
    n = np.where(np.asarray(atm["gas_indx_mask"], bool), y, 0).sum(axis=1)
    d, T, H, g = f["dzi"][0], f["Ti"][0], f["Hpi"][0], f["g"]
    w, w0, w1 = (lam[0] - lam[1]) / d, lam[0] / d, lam[1] / d
    c = L(0.0 if atm["use_vm_mol"] else 0.5)
    S, s = (n[0] + n[1]) / 2, y[0] + y[1]
    mk = f["ms"] / (L(6.02214086e23) * L(1.38064852e-16)) / T
    dT = f["Tco"][1] - f["Tco"][0]
    wind = lambda v: np.where(v > 0, y[0], np.where(v < 0, y[1], 0))   # noqa: E731
    # the end rows use their own gravity in both terms
    e0, e1 = mk * (g[0] - g[1]) * y[1], mk * (g[1] - g[0]) * y[0]
    end = w0 * e0 - w1 * e1
    th, gr = f["alpha"] / T * dT / d * s, mk * (g[0] * y[0] + g[1] * y[1])
    D = f["Dzz"][0]
    out = {}
    out["Dzz"] = (-(w * (S * (y[1] / n[1] - y[0] / n[0]) / d + c * (th - s / H + gr)) + c * end),
                  np.abs(w) * (S * (y[1] / n[1] + y[0] / n[0]) / d + c * (np.abs(th) + s / H + gr))
                  + c * (np.abs(w0 * e0) + np.abs(w1 * e1)))
    out["alpha"] = (-(w * c * D / T * dT / d * s), np.abs(w * c * D / T * dT / d * s))
    out["ms"] = (-(c * D * (w * gr + end)) * T / f["ms"] / T,
                 c * D * (np.abs(w) * gr + np.abs(w0 * e0) + np.abs(w1 * e1)) / f["ms"])
    if atm["use_settling"]:
        out["vs"] = (w * wind(f["vs"][0]), np.abs(w * wind(f["vs"][0])))
    return out


@pytest.mark.parametrize("seed", range(6))
@pytest.mark.parametrize("advection", [False, True], ids=["gravity", "advection"])
def test_nearly_conserved_lambda(seed, advection):
    ni = 40
    net = syn.make_network(60 + ni, ni, 4 * ni)
    c = syn.make_case(seed=(81, seed), net=net, nz=2, mild=True, k_range=(-40.0, 4.0), moldiff=True, fluxes=True,
                      advection=advection)
    atm = jstep.atm_from_dict(c.atm)
    rng = np.random.default_rng(seed)
    lam = rng.normal(0.0, 1.0, ni) * (1.0 + 1e-5 * rng.normal(0.0, 1.0, (2, ni)))
    y, ld = (torch.as_tensor(v, device="cuda").contiguous() for v in (np.asarray(c.y)[None], lam[None]))
    blob = jstep.pack_atm(atm)
    g = torch.empty_like(blob)
    _lib.check(_lib.lib().vb_adjoint_atm(1, 2, ni, None, _lib.ptr(y), _lib.ptr(blob), jstep.atm_flags(atm),
                                         _lib.ptr(ld), _lib.ptr(g), _lib.stream_handle(None)), "vb_adjoint_atm")
    got = ssg.unpack_atm_cotangents(g, 2, ni)
    for leaf, (ref, scale) in leaves(c.y, c.atm, lam).items():
        v = got[leaf][0].cpu().numpy().reshape(-1).astype(L)
        assert np.all(np.abs(v - ref) <= BOUND * scale), (leaf, float((np.abs(v - ref) / scale).max()))

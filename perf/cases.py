"""The workloads whose speed this framework is judged by.

Every case is one pass through a public entry point with the plan, tables and
device tensors a program would hold before the call:

* ``step``     one Ros2 step of a uniform batch (``jax_step.Ros2Step``), in
               FP64 or with the mixed-precision factor, with or without
               molecular diffusion, advection, boundary fluxes and fixed cells;
* ``ragged``   one Ros2 step of atmospheres with uneven layer counts
               (``jax_step.RaggedRos2Step``);
* ``solve``    the block-Thomas solver on its own: factor, solve, transposed
               solve (``solver``);
* ``photo``    one photochemistry update (``photo.photo_update``);
* ``adjoint``  the implicit steady-state cotangents
               (``steady_state_grad.implicit_cotangents``);
* ``loop``     the start of an adaptive integration with photochemistry
               (``outer_loop.AdaptiveRunner``).

Networks are seeded and fixed per size, as the reaction file of a program is;
states, rates, atmospheres and time steps come from the case's seed. Rate
constants are order-scaled (pseudo-first-order 1e-12 .. 1e4 /s), so a step is
determined to working precision and its outputs can be compared.
"""
from __future__ import annotations

import functools
import importlib

import numpy as np
import torch


def _pkg(name):
    return importlib.import_module("jax-vulcan_b200." + name)


# ------------------------------------------------------------------ the cases
def listed():
    return [
        # the smallest call: one shallow column of a reduced network, stepped
        # by an interactive or one-dimensional run; launches and latency count
        dict(name="step_small", kind="step", batch=1, ni=30, n_fwd=185, nz=43),
        # one hot-Jupiter column with the C/H/O/N network: what a single
        # reference run does at every step
        dict(name="step_one", kind="step", batch=1, ni=69, n_fwd=700, nz=120),
        # a parameter study of a few dozen columns with every transport term
        # on and some cells held fixed; an odd count and an odd layer number
        dict(name="step_transport", kind="step", batch=33, ni=69, n_fwd=700, nz=97, transport=True, fixed=True),
        # the headline batch: two atmospheres per SM
        dict(name="step_batch", kind="step", batch=296, ni=69, n_fwd=700, nz=120),
        # the largest network (C/H/O/N/S) on deep columns
        dict(name="step_sncho", kind="step", batch=128, ni=89, n_fwd=1000, nz=150),
        # a survey whose columns have their own layer counts
        dict(name="step_ragged", kind="ragged", batch=85, ni=69, n_fwd=700, nz_min=60, nz_max=200),
        # the mixed-precision step on a batch of one atmosphere per SM
        dict(name="step_mixed", kind="step", batch=148, ni=69, n_fwd=700, nz=120, mixed=True),
        # the block solver used by itself (a Newton iteration with its adjoint)
        dict(name="solve_block", kind="solve", batch=64, ni=69, n_fwd=700, nz=120),
        # photolysis rates of one column: the photo branch of a single run
        dict(name="photo_one", kind="photo", batch=1, ni=69, n_fwd=700, n_photo=40, nz=120),
        # and of a batch
        dict(name="photo_batch", kind="photo", batch=64, ni=69, n_fwd=700, n_photo=40, nz=120),
        # gradients of a retrieval: every cotangent of the steady state
        dict(name="adjoint_batch", kind="adjoint", batch=64, ni=69, n_fwd=700, nz=120),
        # a whole call: the first attempts of an adaptive run with photochemistry
        dict(name="loop_photo", kind="loop", batch=16, ni=69, n_fwd=700, n_photo=40, nz=120, attempts=8),
    ]


def draw(rng):
    """One more case: block sizes 12 .. 96, 20 .. 200 layers, batches of 1 to
    296, spread over the logarithm, capped at the work and the serial length
    of the largest listed cases."""
    def logint(lo, hi):
        return max(lo, min(hi, int(round(lo * (hi / lo) ** rng.random()))))

    kind = rng.choice(["step", "step", "step", "step", "ragged", "mixed", "solve", "photo", "adjoint", "loop"])
    ni = logint(12, 96) if rng.random() < 0.7 else rng.randint(61, 77)
    nz = logint(20, 200)
    cap = 128 * 150 * 89 ** 3 // max(1, nz * ni ** 3)
    batch = logint(1, max(1, min(296, cap)))
    n_fwd = int(ni * rng.uniform(4.0, 11.0))
    if kind == "photo":
        return dict(kind="photo", batch=logint(1, 60), ni=69, n_fwd=700, n_photo=40, nz=logint(20, 120))
    if kind == "loop":
        return dict(kind="loop", batch=logint(1, 16), ni=69, n_fwd=700, n_photo=40, nz=logint(20, 120),
                    attempts=rng.randint(2, 8))
    if kind == "ragged":
        return dict(kind="ragged", batch=max(2, min(batch, 85)), ni=min(ni, 89), n_fwd=int(min(ni, 89) * 8),
                    nz_min=rng.randint(20, 60), nz_max=rng.randint(61, 200))
    if kind in ("solve", "adjoint"):
        return dict(kind=kind, batch=min(batch, 64), ni=min(ni, 77), n_fwd=n_fwd, nz=min(nz, 150))
    c = dict(kind="step", batch=batch, ni=ni, n_fwd=n_fwd, nz=nz)
    if kind == "mixed":
        c.update(mixed=True, batch=min(batch, 148))
    elif rng.random() < 0.4:
        c.update(transport=True, fixed=rng.random() < 0.5)
    return c


# ------------------------------------------------------------------ inputs
@functools.lru_cache(maxsize=None)
def _network(ni, n_fwd, n_photo=0):
    """The seeded network of a size (the reaction file of a program)."""
    el = ("C", "H", "O", "N", "S") if ni > 77 else ("C", "H", "O", "N")
    return _pkg("synthetic").make_network(0, ni, n_fwd, elements=el, n_photo=n_photo)


def _net_of(case):
    return _network(case["ni"], case["n_fwd"], case.get("n_photo", 0))


def _stack(atms):
    return {k: (v if isinstance(v, bool) else np.stack([a[k] for a in atms])) for k, v in atms[0].items()}


def _atmospheres(case, seed, nzs, transport=False):
    syn = _pkg("synthetic")
    net = _net_of(case)
    rng = np.random.default_rng([int(seed), 1])
    return zip(*[syn.make_atmosphere((int(seed), b), net, nz=nz, T_offset=float(rng.uniform(-300.0, 300.0)),
                                     kzz_scale=float(10.0 ** rng.uniform(-1.0, 1.0)), moldiff=transport,
                                     advection=False, fluxes=transport) for b, nz in enumerate(nzs)])


def _rates(case, seed, b, nz, n_max):
    """Order-scaled rate constants k [b, nr+1, nz]: pseudo-first-order rates
    log-uniform in [1e-12, 1e4] /s at each column's densest layer."""
    t = _net_of(case).tables
    gen = torch.Generator(device="cuda").manual_seed(1000003 * (int(seed) + 1) + nz)
    u = torch.rand((b, t.nr + 1, nz), dtype=torch.float64, device="cuda", generator=gen)
    k = 10.0 ** (16.0 * u - 12.0)
    order = torch.as_tensor(t.reactant_stoich.sum(axis=1) + t.is_three_body, device="cuda")
    n_ref = torch.as_tensor(np.asarray(n_max, np.float64), device="cuda").reshape(b, 1, 1)
    k = k / n_ref ** torch.clamp(order - 1.0, min=0.0)[None, :, None]
    k[:, 0] = 0.0
    k[:, torch.as_tensor(np.asarray(t.is_photo, bool), device="cuda")] = 0.0
    return k.contiguous()


def _uniform_inputs(case, seed):
    """(atmosphere dict of stacked arrays, extras, y, k, dt, fix_mask) of a batch."""
    b, nz = case["batch"], case["nz"]
    transport = bool(case.get("transport")) or case["kind"] == "adjoint"
    atms, extras = _atmospheres(case, seed, [nz] * b, transport)
    rng = np.random.default_rng([int(seed), 2])
    y = torch.as_tensor(np.stack([e["y"] for e in extras]), device="cuda")
    k = _rates(case, seed, b, nz, [e["n"].max() for e in extras])
    dt = torch.as_tensor(10.0 ** rng.uniform(-8.0, -2.0, b), device="cuda")
    fix = None
    if case.get("fixed"):
        fix = torch.as_tensor((rng.random((b, nz, case["ni"])) < 0.02).astype(np.uint8), device="cuda")
    return _stack(atms), extras, y, k, dt, fix


def _ragged_inputs(case, seed):
    # the layer counts are the plan's, the same for every seed
    lay = np.random.default_rng([case["batch"], case["nz_min"], case["nz_max"]])
    nzs = [int(v) for v in lay.integers(case["nz_min"], case["nz_max"] + 1, case["batch"])]
    rng = np.random.default_rng([int(seed), 3])
    atms, extras = _atmospheres(case, seed, nzs)
    ks = [_rates(case, int(seed) * 1009 + b, 1, nz, [e["n"].max()])[0] for b, (nz, e) in enumerate(zip(nzs, extras))]
    dt = torch.as_tensor(10.0 ** rng.uniform(-8.0, -2.0, case["batch"]), device="cuda")
    return atms, [torch.as_tensor(e["y"], device="cuda") for e in extras], ks, dt


def _photo_inputs(case, seed):
    syn = _pkg("synthetic")
    net = _net_of(case)
    bins, din12 = syn.make_bins()
    atms, extras = _atmospheres(case, seed, [case["nz"]] * case["batch"])
    # the cross sections are per network and temperature grid: one table for the batch
    ph = syn.make_photo(int(seed), net, syn.make_atmosphere(0, net, nz=case["nz"])[0]["Tco"], bins, din12)
    gen = torch.Generator(device="cuda").manual_seed(77 + int(seed))
    prev = torch.rand((case["batch"], case["nz"] + 1, len(bins)), dtype=torch.float64, device="cuda", generator=gen)
    prev = prev * torch.as_tensor(0.1 * ph["sflux_top"], device="cuda")

    def dev(name):
        return torch.as_tensor(np.stack([e[name] for e in extras]), device="cuda")

    return ph, dev("y"), dev("ymix"), dev("dz"), _rates(case, seed, case["batch"], case["nz"],
                                                        [e["n"].max() for e in extras]), prev


def prepare(case, seed):
    jstep, chem = _pkg("jax_step"), _pkg("chem")
    kind = case["kind"]
    if kind == "step":
        A, _, y, k, dt, fix = _uniform_inputs(case, seed)
        step = jstep.Ros2Step(chem.to_device(_net_of(case).tables), jstep.atm_from_dict(A),
                              mixed=bool(case.get("mixed")))
        return dict(kind=kind, step=step, y=y, k=k, dt=dt, fix=fix)
    if kind == "ragged":
        atms, ys, ks, dt = _ragged_inputs(case, seed)
        step = jstep.RaggedRos2Step(chem.to_device(_net_of(case).tables), [jstep.atm_from_dict(a) for a in atms])
        y, k = step.pack(ys, ks)
        return dict(kind="step", step=step, y=y, k=k, dt=dt, fix=None)
    if kind == "solve":
        return dict(kind=kind, sys=_block_system(case, seed))
    if kind == "photo":
        ph, y, ymix, dz, k, prev = _photo_inputs(case, seed)
        return dict(kind=kind, photo=_pkg("photo").PhotoDevice(ph, case["nz"]), y=y, ymix=ymix, dz=dz, k=k, prev=prev)
    if kind == "adjoint":
        A, _, y, k, _, _ = _uniform_inputs(case, seed)
        atm = jstep.AtmStatic(**{f: (torch.as_tensor(A[f], device="cuda") if isinstance(A[f], np.ndarray) else A[f])
                                 for f in jstep.AtmStatic._fields})
        return dict(kind=kind, net=chem.to_device(_net_of(case).tables), atm=atm, y=y, k=k, v=_loss_gradient(case, seed, y))
    return _prepare_loop(case, seed)


def _prepare_loop(case, seed):
    syn, loop, photo, jstep, chem = (_pkg("synthetic"), _pkg("outer_loop"), _pkg("photo"), _pkg("jax_step"),
                                     _pkg("chem"))
    net = _net_of(case)
    b, nz = case["batch"], case["nz"]
    atms, extras = _atmospheres(case, seed, [nz] * b)
    # rates in detailed balance with a composition near the initial one, as in
    # a run restarted from a neighbouring state
    k0, eq = syn.make_balanced_rates((int(seed),), net, nz, extras[0]["n"], -12.0, 4.0, M=atms[0]["M"])
    rng = np.random.default_rng([int(seed), 5])
    ymix = eq[None] * 10.0 ** rng.uniform(-0.3, 0.3, (b, net.tables.ni))
    ymix = ymix / ymix.sum(axis=1, keepdims=True)
    y0 = ymix[:, None, :] * np.stack([e["n"] for e in extras])[:, :, None]
    atom_ini = np.einsum("bzi,ia->ba", y0, net.compo)
    bins, din12 = syn.make_bins()
    ph = photo.PhotoDevice(syn.make_photo(int(seed), net, atms[0]["Tco"], bins, din12), nz)
    runner = loop.AdaptiveRunner(
        chem.to_device(net.tables), jstep.atm_from_dict(_stack(atms)), loop.LoopStatics(dt_max=1e17), net.compo,
        atom_ini, batch=b, conv=loop.ConvStatics(use_photo=True, conv_step=50),
        slope_min=np.concatenate([loop.slope_min_of(a["Kzz"], e["Hp"]) for a, e in zip(atms, extras)]),
        photo=ph, dz=np.stack([e["dz"] for e in extras]), flux_atol=1.0)
    return dict(kind="loop", runner=runner, attempts=case["attempts"], photo=ph, batch=b, nz=nz,
                y0=torch.as_tensor(y0, device="cuda"), loss0=torch.zeros(atom_ini.shape, dtype=torch.float64, device="cuda"),
                ymix0=torch.as_tensor(np.broadcast_to(ymix[:, None, :], y0.shape).copy(), device="cuda"),
                k=torch.as_tensor(np.broadcast_to(k0, (b,) + k0.shape).copy(), device="cuda"))


def _loss_gradient(case, seed, y):
    """dL/dy of seeded weights times log ymix at some layers."""
    rng = np.random.default_rng([int(seed), 4])
    nz = case["nz"]
    layers = torch.as_tensor(rng.choice(nz, min(10, nz), replace=False), device="cuda")
    w = torch.as_tensor(rng.normal(0.0, 1.0, (case["batch"], layers.numel(), case["ni"])), device="cuda")
    v = torch.zeros_like(y)
    ys = y[:, layers]
    v[:, layers] = w / ys - w.sum(dim=2, keepdim=True) / ys.sum(dim=2, keepdim=True)
    return v


# ------------------------------------------------------------------ one pass
def run(state):
    kind = state["kind"]
    if kind == "step":
        return state["step"](state["y"], state["k"], state["dt"], fix_mask=state["fix"])
    if kind == "solve":
        solver = _pkg("solver")
        diag, sup, sub, rhs = state["sys"]
        f = solver.factor_block_thomas_diag_offdiag(diag, sup, sub)
        return (solver.solve_block_thomas_diag_offdiag(f, rhs), solver.solve_block_thomas_diag_offdiag_T(f, rhs),
                f.status)
    if kind == "photo":
        aflux, du = _pkg("photo").photo_update(state["y"], state["ymix"], state["dz"], state["k"], state["photo"],
                                               state["prev"])
        return state["k"], aflux, du
    if kind == "adjoint":
        return _pkg("steady_state_grad").implicit_cotangents(state["y"], state["k"], state["atm"], state["net"],
                                                             state["v"])
    loop, photo, runner = _pkg("outer_loop"), _pkg("photo"), state["runner"]
    runner.photo_carry = photo.PhotoCarry(state["photo"], state["batch"], state["nz"])
    s = loop.LoopState(state["y0"], state["ymix0"], 1e-10, state["loss0"], rtol=0.2)
    runner.start(s)
    k = state["k"].clone()
    runner.run(s, k, state["attempts"])
    return s.y, s.ymix, s.dt, k


# ------------------------------------------------------------------ the work of a pass
def work(case):
    kind, b, ni = case["kind"], case["batch"], case["ni"]
    nr = 2 * case["n_fwd"] + 2 * case.get("n_photo", 0)
    if kind == "ragged":
        layers = b * (case["nz_min"] + case["nz_max"]) // 2
    else:
        layers = b * case["nz"]
    factor = 2 * ni ** 3 * layers
    sweep = 2 * ni * ni * layers
    chem = 12 * nr * layers
    atm = 8 * layers * (8 + 3 * ni)
    step = dict(bytes=8 * layers * (3 * ni + nr + 1) + atm, flops=factor + 4 * sweep + 3 * chem)
    if kind in ("step", "ragged"):
        return step
    if kind == "solve":
        return dict(bytes=8 * layers * (ni * ni + 5 * ni), flops=factor + 4 * sweep)
    nbin, br = 2500, case.get("n_photo", 0)
    photo = dict(bytes=8 * layers * (2 * ni + 3 * nbin + br) + 8 * nbin * (4 * case.get("nz", 0) + br),
                 flops=layers * nbin * (2 * 21 * 2 + 100 + 2 * br))
    if kind == "photo":
        return photo
    if kind == "adjoint":
        return dict(bytes=8 * layers * (3 * ni + 2 * (nr + 1)) + 2 * atm, flops=factor + 2 * sweep + 4 * chem)
    return dict(bytes=case["attempts"] * step["bytes"] + photo["bytes"],
                flops=case["attempts"] * step["flops"] + photo["flops"])


# ------------------------------------------------------------------ the same results in plain torch, 64 bits
_KB, _NAVO = 1.38064852e-16, 6.02214086e23


def _flags(A):
    return {f: bool(A[f]) for f in ("use_vm_mol", "use_settling", "use_topflux", "use_botflux")}


def _t64(A):
    return {k: torch.as_tensor(np.asarray(v, np.float64) if k != "gas_indx_mask" else np.asarray(v, bool),
                               device="cuda") for k, v in A.items() if not isinstance(v, bool)}


def _transport(y, P, flags):
    """(A, B, C) of d y_j/dt = A_j y_j + B_j y_{j+1} + C_j y_{j-1} from eddy and
    molecular diffusion (no advection), [b, nz, ni] with B[-1] = C[0] = 0."""
    if flags["use_vm_mol"] or flags["use_settling"]:
        raise NotImplementedError
    lay = lambda x: x[..., None]                               # noqa: E731
    Kzz, Dzz, dzi, Hpi, Ti, Tco, g = (P[n] for n in ("Kzz", "Dzz", "dzi", "Hpi", "Ti", "Tco", "g"))
    ms, alpha = P["ms"][:, None, :], P["alpha"][:, None, :]
    n = torch.where(P["gas_indx_mask"][:, None, :], y, torch.zeros_like(y)).sum(-1)       # [b, nz]
    face = 0.5 * (n[:, 1:] + n[:, :-1])                                                   # [b, nz-1]
    # layer thickness a flux difference is divided by: the half sums inside, the edge spacing at the ends
    dz = torch.cat([dzi[:, :1], 0.5 * (dzi[:, 1:] + dzi[:, :-1]), dzi[:, -1:]], 1)        # [b, nz]
    D = (lay(Kzz) + Dzz) * lay(face / dzi)                                                # eddy + molecular
    # molecular drift of the interface, with the gravity of the layer it acts on
    slope = alpha / lay(Ti) * lay((Tco[:, 1:] - Tco[:, :-1]) / dzi)

    def drift(gl):
        return Dzz * (-1.0 / lay(Hpi) + ms * lay(gl) / (_NAVO * _KB * lay(Ti)) + slope) / 2.0

    lo, hi = drift(g[:, :-1]), drift(g[:, 1:])       # interface j seen with the gravity of layer j, j + 1
    z = torch.zeros_like(y[:, :1])
    up_A, up_B = -D / lay(n[:, :-1]) + lo, D / lay(n[:, 1:]) + hi      # flux through the upper face, times +1
    dn_A, dn_C = -D / lay(n[:, 1:]) - hi, D / lay(n[:, :-1]) - lo      # through the lower face
    # the end layers use their own gravity for both terms
    up_B = torch.cat([up_B[:, :1] - hi[:, :1] + lo[:, :1], up_B[:, 1:]], 1)
    dn_C = torch.cat([dn_C[:, :-1], dn_C[:, -1:] + lo[:, -1:] - hi[:, -1:]], 1)
    vz = P["vz"]
    wp, wm = lay(torch.where(vz > 0, vz, 0.0 * vz)), lay(torch.where(vz < 0, vz, 0.0 * vz))
    A = (torch.cat([up_A - wp, z], 1) + torch.cat([z, dn_A + wm], 1)) / lay(dz)
    B = torch.cat([up_B - wm, z], 1) / lay(dz)
    C = torch.cat([z, dn_C + wp], 1) / lay(dz)
    return A, B, C


def _tables(t):
    dev = lambda a, d: torch.as_tensor(np.asarray(a, d), device="cuda")   # noqa: E731
    return (dev(t.reactant_idx, np.int64), dev(t.product_idx, np.int64), dev(t.reactant_stoich, np.float64),
            dev(t.product_stoich, np.float64), dev(t.is_three_body, bool))


def _powers(y, tab):
    ridx, _, rst, _, _ = tab
    yr = torch.cat([y, torch.ones_like(y[..., :1])], -1)[..., ridx]                        # [b, nz, nr+1, T]
    return yr, torch.where(rst > 0, yr ** rst, torch.ones_like(yr))


def _chem(y, M, k, tab):
    ridx, pidx, rst, pst, three = tab
    rate = k.transpose(1, 2) * _powers(y, tab)[1].prod(-1)
    rate = torch.where(three, rate * M[..., None], rate)
    net = torch.zeros((ridx.shape[0], y.shape[2] + 1), dtype=torch.float64, device=y.device)
    rows = torch.arange(ridx.shape[0], device=y.device)
    for s in range(ridx.shape[1]):
        net[rows, pidx[:, s]] += pst[:, s]
        net[rows, ridx[:, s]] -= rst[:, s]
    return (rate @ net)[..., :-1]


def _chem_jac(y, M, k, tab):
    ridx, pidx, rst, pst, three = tab
    b, nz, ni = y.shape
    yr, f = _powers(y, tab)
    T = ridx.shape[1]
    J = torch.zeros((b * nz, (ni + 1) * (ni + 1)), dtype=torch.float64, device=y.device)
    rows = torch.arange(ridx.shape[0], device=y.device)
    kk = k.transpose(1, 2)
    kk = torch.where(three, kk * M[..., None], kk)
    for s in range(T):
        d = torch.where(rst[:, s] > 0, rst[:, s] * yr[..., s] ** (rst[:, s] - 1.0), torch.zeros_like(kk))
        for o in range(T):
            if o != s:
                d = d * f[..., o]
        d = (d * kk).reshape(b * nz, -1)
        net = torch.zeros((ridx.shape[0], (ni + 1) * (ni + 1)), dtype=torch.float64, device=y.device)
        for o in range(T):
            net[rows, pidx[:, o] * (ni + 1) + ridx[:, s]] += pst[:, o]
            net[rows, ridx[:, o] * (ni + 1) + ridx[:, s]] -= rst[:, o]
        J.addmm_(d, net)
    return J.reshape(b, nz, ni + 1, ni + 1)[:, :, :ni, :ni]


def _rhs(y, P, flags, k, tab):
    A, B, C = _transport(y, P, flags)
    d = A * y
    d = d + torch.cat([B[:, :-1] * y[:, 1:], torch.zeros_like(y[:, :1])], 1)
    d = d + torch.cat([torch.zeros_like(y[:, :1]), C[:, 1:] * y[:, :-1]], 1)
    edge = torch.zeros_like(y)
    if flags["use_botflux"]:
        bot = (P["bot_flux"] - y[:, 0] * P["bot_vdep"]) / P["dzi"][:, :1]
        edge = torch.cat([edge[:, :1] + bot[:, None], edge[:, 1:]], 1)
    if flags["use_topflux"]:
        edge = torch.cat([edge[:, :-1], edge[:, -1:] + (P["top_flux"] / P["dzi"][:, -1:])[:, None]], 1)
    return _chem(y, P["M"], k, tab) + d + edge


def _jacobian(y, P, flags, k, tab):
    """Blocks of the Jacobian with the transport coefficients held: (diag, sup, sub)."""
    A, B, C = _transport(y, P, flags)
    if flags["use_botflux"]:
        A = torch.cat([A[:, :1] - (P["bot_vdep"] / P["dzi"][:, :1])[:, None], A[:, 1:]], 1)
    return _chem_jac(y, P["M"], k, tab) + torch.diag_embed(A), B[:, :-1], C[:, 1:]


def _thomas(diag, sup, sub):
    """A solver of the block-tridiagonal system with diagonal off-diagonal blocks."""
    nz = diag.shape[1]
    eye = torch.eye(diag.shape[2], dtype=torch.float64, device=diag.device).expand(diag.shape[0], -1, -1)
    lus = []
    for j in range(nz):
        a = diag[:, j]
        if j:
            a = a - sub[:, j - 1, :, None] * sup[:, j - 1, None, :] * torch.linalg.lu_solve(*lus[-1], eye)
        lus.append(torch.linalg.lu_factor(a))

    def solve(rhs):
        f = [rhs[:, 0]]
        one = lambda j, r: torch.linalg.lu_solve(*lus[j], r[..., None])[..., 0]   # noqa: E731
        for j in range(1, nz):
            f.append(rhs[:, j] - sub[:, j - 1] * one(j - 1, f[-1]))
        x = [one(nz - 1, f[-1])]
        for j in range(nz - 2, -1, -1):
            x.append(one(j, f[j] - sup[:, j] * x[-1]))
        return torch.stack(x[::-1], 1)

    return solve


def _step_matrix(y, P, flags, k, dt, tab, fix=None):
    r = 1.0 + 0.5 ** 0.5
    diag, sup, sub = _jacobian(y, P, flags, k, tab)
    c0 = (1.0 / (r * dt))[:, None, None]
    diag = torch.diag_embed(c0.expand(y.shape)) - diag
    sup, sub = -sup, -sub
    if fix is not None:
        diag = torch.where(fix[..., None], torch.diag_embed(c0.expand(y.shape)), diag)
        sup = torch.where(fix[:, :-1], torch.zeros_like(sup), sup)
        sub = torch.where(fix[:, 1:], torch.zeros_like(sub), sub)
    return diag, sup, sub


def _ros2(y, P, flags, k, dt, tab, fix=None):
    r = 1.0 + 0.5 ** 0.5
    fix = None if fix is None else fix.bool()
    hold = (lambda x: x) if fix is None else (lambda x: torch.where(fix, torch.zeros_like(x), x))
    solve = _thomas(*_step_matrix(y, P, flags, k, dt, tab, fix))
    k1 = solve(hold(_rhs(y, P, flags, k, tab)))
    y2 = y + k1 / r
    k2 = solve(hold(_rhs(y2, P, flags, k, tab)) - (2.0 / (r * dt))[:, None, None] * k1)
    sol = y + 1.5 / r * k1 + 0.5 / r * k2
    return sol, (sol - y2).abs()


def _block_system(case, seed):
    """The linear system of a Ros2 step and a right-hand side of its scale."""
    A, _, y, k, dt, _ = _uniform_inputs(case, seed)
    P, flags, tab = _t64(A), _flags(A), _tables(_net_of(case).tables)
    diag, sup, sub = _step_matrix(y, P, flags, k, dt, tab)
    return diag.contiguous(), sup.contiguous(), sub.contiguous(), _rhs(y, P, flags, k, tab).contiguous()


def _batch_chunks(b, size):
    return [slice(i, min(b, i + size)) for i in range(0, b, size)]


def exact(case, seed):
    kind = case["kind"]
    tab = _tables(_net_of(case).tables)
    if kind == "step":
        A, _, y, k, dt, fix = _uniform_inputs(case, seed)
        P, flags = _t64(A), _flags(A)
        parts = []
        for s in _batch_chunks(case["batch"], 148):
            parts.append(_ros2(y[s], {n: v[s] for n, v in P.items()}, flags, k[s], dt[s], tab,
                               None if fix is None else fix[s]))
        return torch.cat([p[0] for p in parts]), torch.cat([p[1] for p in parts]), None
    if kind == "ragged":
        atms, ys, ks, dt = _ragged_inputs(case, seed)
        out = [_ros2(y[None], _t64(_stack([a])), _flags(a), k[None], dt[b:b + 1], tab)
               for b, (a, y, k) in enumerate(zip(atms, ys, ks))]
        return torch.cat([o[0][0] for o in out]), torch.cat([o[1][0] for o in out]), None
    if kind == "solve":
        diag, sup, sub, rhs = _block_system(case, seed)
        return _thomas(diag, sup, sub)(rhs), _thomas(diag.transpose(2, 3).contiguous(), sub, sup)(rhs), None
    if kind == "photo":
        return _exact_photo(case, seed)
    if kind == "adjoint":
        return _exact_adjoint(case, seed, tab)
    # the loop takes its own accept / reject decisions and steps: no value
    # outside the loop itself
    return None


def _exact_photo(case, seed):
    ph, y, ymix, dz, k, prev = _photo_inputs(case, seed)
    P = {n: torch.as_tensor(v, device="cuda") for n, v in ph.items() if isinstance(v, np.ndarray)}
    mu, edd = -ph["mu_zenith"], ph["edd"]
    afs, dus = [], []
    for s in _batch_chunks(case["batch"], 16):
        def columns(x):
            a = x[..., P["absp_idx"]] @ P["absp_cross"]
            a = a + torch.einsum("bzs,szw->bzw", x[..., P["absp_T_idx"]], P["absp_T_cross"])
            return a, x[..., P["scat_idx"]] @ P["scat_cross"]

        a, sc = columns(y[s])
        dtau = (a + sc) * dz[s][..., None]
        tau = torch.cat([dtau.flip(1).cumsum(1).flip(1), torch.zeros_like(dtau[:, :1])], 1)
        dtau = tau[:, :-1] - tau[:, 1:]
        a, sc = columns(ymix[s])
        w0 = (sc / (a + sc).clamp(min=1e-300)).clamp(max=1.0 - 1e-8)
        root = (1.0 - w0).sqrt()
        tran = torch.exp(-root * dtau / edd)
        zp, zm = 0.5 * (1.0 + root), 0.5 * (1.0 - root)
        part = -w0 / (1.0 / mu ** 2 - (1.0 - w0) / edd ** 2)
        gp, gm = 0.5 * part * (1.0 / edd + 1.0 / mu), 0.5 * part * (1.0 / edd - 1.0 / mu)
        chi = zm ** 2 * tran ** 2 - zp ** 2
        xi = zp * zm * (1.0 - tran ** 2)
        phi = (zm ** 2 - zp ** 2) * tran
        direct = P["sflux_top"] * torch.exp(tau / mu)
        df = -mu * direct
        iu = phi * gp * df[:, :-1] - (xi * gm + chi * gp) * df[:, 1:]
        idn = phi * gm * df[:, 1:] - (chi * gm + xi * gp) * df[:, :-1]
        down = [torch.zeros_like(tau[:, 0])]
        for j in range(case["nz"] - 1, -1, -1):
            down.append((phi[:, j] * down[-1] - xi[:, j] * prev[s][:, j] + idn[:, j] / mu) / chi[:, j])
        down = torch.stack(down[::-1], 1)
        up = [torch.zeros_like(tau[:, 0])]
        for j in range(case["nz"]):
            up.append((phi[:, j] * up[-1] - xi[:, j] * down[:, j + 1] + iu[:, j] / mu) / chi[:, j])
        up = torch.stack(up, 1)
        tot = 0.5 * (direct[:, 1:] + direct[:, :-1]) + 0.5 * (up[:, 1:] + up[:, :-1] + down[:, 1:] + down[:, :-1]) / edd
        afs.append(tot * P["bins"] / ph["hc"])
        dus.append(up)
    aflux, du = torch.cat(afs), torch.cat(dus)
    d = ph["din12_indx"]
    w = torch.full((len(ph["bins"]),), ph["dbin2"], dtype=torch.float64, device="cuda")
    w[:d] = ph["dbin1"]
    for e in (0, d - 1, d, -1):
        w[e] = 0.5 * w[e]
    k = k.clone()
    if len(ph["branch_re_idx"]):
        k[:, P["branch_re_idx"]] = torch.einsum("bzw,nw->bnz", aflux * w, P["cross_J"]) * ph["f_diurnal"]
    if len(ph["branch_T_re_idx"]):
        k[:, P["branch_T_re_idx"]] = torch.einsum("bzw,nzw->bnz", aflux * w, P["cross_J_T"]) * ph["f_diurnal"]
    return k, aflux, du


def _exact_adjoint(case, seed, tab):
    A, _, y, k, _, _ = _uniform_inputs(case, seed)
    flags = _flags(A)
    v = _loss_gradient(case, seed, y)
    names = ("Kzz", "dzi", "vz", "Hpi", "Ti", "Tco", "g", "M", "Dzz", "ms", "alpha", "top_flux", "bot_flux", "bot_vdep")
    out = {}
    for s in _batch_chunks(case["batch"], 16):
        P = {n: t[s] for n, t in _t64(A).items()}
        diag, sup, sub = _jacobian(y[s], P, flags, k[s], tab)
        lam = _thomas(diag.transpose(2, 3).contiguous(), sub, sup)(v[s])
        leaves = {n: P[n].detach().clone().requires_grad_(True) for n in names}
        kk = k[s].clone().requires_grad_(True)
        f = _rhs(y[s], {**P, **leaves}, flags, kk, tab)
        grads = torch.autograd.grad(f, [kk] + [leaves[n] for n in names], grad_outputs=lam)
        part = dict(zip(("k_arr",) + names, [-g for g in grads]))
        part["lambda"] = lam
        part["Kzz_transport"] = part["Kzz"]
        for n, g in part.items():
            out.setdefault(n, []).append(g)
    out = {n: torch.cat(g) for n, g in out.items()}
    # the advection speeds are off: their terms do not enter the residual
    b, nz, ni = y.shape
    out["vm"] = torch.zeros((b, nz, ni), dtype=torch.float64, device="cuda")
    out["vs"] = torch.zeros((b, nz - 1, ni), dtype=torch.float64, device="cuda")
    out["status"] = None
    return out

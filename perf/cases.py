"""What a run of this package spends its time in: the cases whose speed counts.

A case names a kind of call, a size and options:

  host      the drop-in time step of a host program that keeps its own arrays (wt_rk4_step_host)
  rk4       the single-level stepper on the device, `steps` RK4 steps between two outputs of the state
  tree      the adaptive run on its partially refined patch tree, `steps` time steps between two outputs
  dense     the same with every patch present
  split     the mode-split adaptive run (implicit free surface), `steps` time steps between two outputs
  solve     the free-surface solve alone, new right-hand side to solution
  learned   the learned preconditioner: one application, or one loss and parameter gradient

Inputs come from a seed: a zonal jet, Gaussian bumps of the layers' thickness and a noisy free surface over a
flat bottom or a seamount; a random bathymetry and right-hand side for the solves.  The adaptive and single-level
states step on from pass to pass, as a model does between two outputs; a patch tree grows as its flow spreads, so
those passes take many steps.
"""
from __future__ import annotations

import functools
import math

import numpy as np
import torch

from wavetrisk_hydrostatic_b200 import Grid, OceanParams, _native, halo_nodes, jet_state
from wavetrisk_hydrostatic_b200.adaptive import AdaptiveOcean, ModeSplitOcean
from wavetrisk_hydrostatic_b200.cases import bathymetry, elliptic_rhs, seamount_topography
from wavetrisk_hydrostatic_b200.model import EllipticSolver, TriskModel, solver_opts

RADIUS = 6371e3
RHO_BOTTOM, RHO_TOP = 1027.0, 1024.0
TOL = 5e-3                      # wavelet threshold of the adaptive runs
RT, DG, UP = 0, 1, 2
TAPS = ((0, 0), (1, 0), (1, 1), (0, 1), (-1, 0), (-1, -1), (0, -1))


def listed():
    return [
        # one time step of a small host program through its own arrays: copies, launches and latency
        {"name": "host_J4x4", "kind": "host", "level": 4, "nz": 4, "steps": 1, "bits": 64},
        # the reference's CPU-sized case, 100 steps between outputs: launch-bound
        {"name": "rk4_J5x8", "kind": "rk4", "level": 5, "nz": 8, "steps": 100, "bits": 64},
        # ordinary and large single-level runs
        {"name": "rk4_J7x16", "kind": "rk4", "level": 7, "nz": 16, "steps": 25, "bits": 64},
        {"name": "rk4_J8x32", "kind": "rk4", "level": 8, "nz": 32, "steps": 15, "bits": 64},
        # the FP32 flux option of the single-level stepper, an odd number of layers
        {"name": "rk4_J7x15_flux32", "kind": "rk4", "level": 7, "nz": 15, "steps": 25, "bits": 32},
        # the adaptive run: the small configuration, and the largest one that sets up in seconds
        {"name": "tree_J4-J7x16", "kind": "tree", "lo": 4, "hi": 7, "nz": 16, "steps": 80},
        {"name": "tree_J5-J8x32", "kind": "tree", "lo": 5, "hi": 8, "nz": 32, "steps": 40},
        # every patch present: a flow that is active everywhere
        {"name": "dense_J5-J7x16", "kind": "dense", "lo": 5, "hi": 7, "nz": 16, "steps": 80},
        # a member of the mode-split ensemble
        {"name": "split_J5-J7x16", "kind": "split", "lo": 5, "hi": 7, "nz": 16, "steps": 45},
        # the free-surface solve: the reference's multigrid at a small size, the mixed-precision one at a large
        {"name": "solve_fmg_J6", "kind": "solve", "lo": 4, "hi": 6, "dt": 600, "method": "fmg"},
        {"name": "solve_mixed_J8", "kind": "solve", "lo": 5, "hi": 8, "dt": 600, "method": "mixed"},
        # one training pair of the learned preconditioner, forward and backward
        {"name": "learned_grad_J7", "kind": "learned", "lo": 5, "hi": 7, "dt": 600, "grad": True},
    ]


def draw(rng):
    kind = rng.choice(["host", "rk4", "rk4", "tree", "tree", "dense", "split", "solve", "solve", "learned"])
    if kind == "host":
        return {"kind": kind, "level": rng.randint(4, 6), "nz": rng.randint(2, 12), "steps": rng.randint(1, 4),
                "bits": 64}
    if kind == "rk4":
        level = rng.randint(4, 8)
        most = 31 if level == 8 else 40
        nz = int(round(math.exp(rng.uniform(math.log(3), math.log(most)))))
        return {"kind": kind, "level": level, "nz": nz, "steps": rng.randint(8, 14) if level == 8 else
                rng.randint(15, 60), "bits": rng.choice([64, 64, 32])}
    if kind == "tree":
        lo, hi = rng.choice([(4, 6), (4, 7), (5, 7), (5, 8)])
        steps = {6: (100, 160), 7: (60, 79), 8: (20, 39)}[hi]
        return {"kind": kind, "lo": lo, "hi": hi, "nz": rng.randint(5, 30), "steps": rng.randint(*steps)}
    if kind == "dense":
        lo, hi = rng.choice([(4, 6), (4, 7), (5, 7)])
        return {"kind": kind, "lo": lo, "hi": hi, "nz": rng.randint(4, 20), "steps": rng.randint(50, 79)}
    if kind == "split":
        lo, hi = rng.choice([(4, 6), (5, 7)])
        return {"kind": kind, "lo": lo, "hi": hi, "nz": rng.randint(4, 20), "steps": rng.randint(30, 45)}
    if kind == "solve":
        hi = rng.randint(6, 8)
        return {"kind": kind, "lo": rng.choice([4, 5]) if hi < 8 else 5, "hi": hi, "dt": rng.randint(300, 900),
                "method": rng.choice(["fmg", "srj", "mixed", "mixed", "mg64", "fcg", "fcg_mg"])}
    return {"kind": kind, "lo": 5, "hi": rng.randint(6, 8), "dt": rng.randint(300, 900), "grad": rng.choice([True, False])}


# ------------------------------------------------------------------ inputs


@functools.lru_cache(maxsize=None)
def _grid(lo, hi):
    return Grid(lo, hi, radius=RADIUS)


def _geom(case):
    """The levels of a case, coarsest first."""
    lo, hi = case.get("lo", case.get("level")), case.get("hi", case.get("level"))
    G = _grid(lo, hi)
    return [G.level(l) for l in range(lo, hi + 1)]


@functools.lru_cache(maxsize=None)
def _jet(lo, hi, level):
    """The zonal jet (1 m/s at 45N) on the level's edges, and the unit vectors of its nodes."""
    g = _grid(lo, hi).level(level)
    nrm = np.linalg.norm(g.node, axis=0)
    return jet_state(g, 2, eta_amp=0.0)["velo"][1], g.node / np.where(nrm > 0, nrm, 1.0), nrm > 0


def _water(key, level, nz, seed, seamount):
    """Layered state of one level: linear layer densities, the jet decaying to the bottom, 8 bumps of 300 km and
    0.05 m in every layer's thickness, a free surface with 1 mm of noise."""
    g = _grid(*key).level(level)
    ph = OceanParams()
    jet, x, ok = _jet(*key, level)
    topo = seamount_topography(g, seed=seed) if seamount else np.full(g.NN, -ph.depth)
    rng = np.random.default_rng(seed)
    c = rng.standard_normal((8, 3))
    c /= np.linalg.norm(c, axis=1, keepdims=True)
    ang = (torch.as_tensor(c) @ torch.as_tensor(x)).clamp_(-1.0, 1.0).acos_()
    dz = (0.05 * torch.exp(-((RADIUS / 300e3 * ang) ** 2))).sum(0).numpy()
    eta = 1e-3 * np.random.default_rng((seed, level)).standard_normal(g.NN)
    for f in (dz, eta):
        f[~ok] = 0.0
        halo_nodes(g, f)
    rho = torch.linspace(RHO_BOTTOM, RHO_TOP, nz, dtype=torch.double)[:, None]
    theta = 1.0 - rho / ph.ref_density
    one = torch.ones_like(theta)
    dz, mean = torch.as_tensor(ph.ref_density * dz), torch.as_tensor(ph.ref_density / nz * -topo)
    st = {"mass": one * dz, "temp": theta * dz, "mean_m": one * mean, "mean_t": theta * mean,
          "velo": torch.linspace(0.0, 1.0, nz, dtype=torch.double)[:, None] * torch.as_tensor(jet)}
    st["mass"][-1] += torch.as_tensor(ph.ref_density * eta)
    return {**{k: a.numpy() for k, a in st.items()}, "topo": topo}


def _dt(case):
    """Explicit time step: 150 s at J7, scaled with the grid spacing, at most 300 s; half of that in the long
    adaptive runs, four times that where the free surface is implicit."""
    dt = min(300.0, 150.0 * 2.0 ** (7 - case.get("hi", case.get("level"))))
    return dt * {"tree": 0.5, "dense": 0.5, "split": 4.0}.get(case["kind"], 1.0)


def _pinned(shape, dtype=torch.float64):
    return torch.empty(shape, dtype=dtype, pin_memory=True).numpy()


def _network(seed):
    """Parameters of the 2 -> 32 -> 32 -> 1 network."""
    rng = np.random.default_rng((seed, 7))
    return np.concatenate([(rng.standard_normal(7 * i * o) * s / math.sqrt(7 * i)) for i, o, s in
                           ((2, 32, 1.0), (32, 32, 1.0), (32, 1, 0.1))]).astype(np.float32)


def _solver(levels, seed, dt):
    return EllipticSolver(levels, [bathymetry(g, seed=seed, nterms=24) for g in levels], dt=float(dt))


def _nodes(levels):
    """Owned slots and poles of the finest level, in storage order."""
    g = levels[-1]
    src = np.arange(g.NN)
    src[g.halo_node[:, 0]] = g.halo_node[:, 1]
    _, i, j = g.ij()
    return np.nonzero((i >= 0) & (j >= 0) & (i <= g.n) & (j <= g.n) & (src == np.arange(g.NN)))[0]


def _pair(levels, seed):
    """A residual and an error of the solve, as a training pair."""
    ns = _nodes(levels).size
    rng = np.random.default_rng((seed, 8))
    return rng.standard_normal(ns), 0.3 * rng.standard_normal(ns)


def _opts(case):
    if case["method"] == "fmg":
        return solver_opts("fmg", 1e-10, max_vcycle=50, coarse_iter=300)
    if case["method"] == "srj":
        return solver_opts("srj", 1e-10, max_srj_iter=4000, coarse_iter=300)
    return solver_opts(case["method"], 1e-10, down_iter=2, up_iter=2, coarse_iter=6, ir_max=2000)


def prepare(case, seed):
    kind, dt = case["kind"], _dt(case) if case["kind"] not in ("solve", "learned") else 0.0
    levels = _geom(case)
    g = levels[-1]
    s = {"case": case, "dt": dt, "levels": levels}
    if kind in ("host", "rk4"):
        nz = case["nz"]
        st = _water((case["level"],) * 2, case["level"], nz, seed, False)
        s["model"] = m = TriskModel(g, nz, st["topo"])
        m.upload(st)
        if case["bits"] == 32:
            m.flux_precision(32)
        s["out"] = [_pinned((nz, g.NN)), _pinned((nz, g.NN)), _pinned((nz, 3 * g.NN))]
        if kind == "host":
            for a, name in zip(s["out"], ("mass", "temp", "velo")):
                a[:] = st[name]
    elif kind in ("tree", "dense", "split"):
        lo, hi, nz = case["lo"], case["hi"], case["nz"]
        states = [_water((lo, hi), l, nz, seed, True) for l in range(lo - 1, hi + 1)]
        how = {"tol": TOL, "root_state": states[0]} if kind != "dense" else {"tol": TOL, "init": "dense"}
        if kind == "split":
            s["model"] = ModeSplitOcean(_grid(lo, hi), lo, hi, nz, states[1:], dt, OceanParams(), **how)
        else:
            s["model"] = AdaptiveOcean(_grid(lo, hi), lo, hi, nz, states[1:], OceanParams(), **how)
        if kind == "dense":
            s["out"] = [_pinned((nz, g.NN)), _pinned((nz, g.NN)), _pinned((nz, 3 * g.NN))]
        else:
            s["out"] = s["model"].dev.tree_state_buffers(alloc=_pinned)
            for a in s["out"]:      # rows past the patches that exist stay 0
                torch.as_tensor(a).zero_()
            for _ in range(4):      # the tree reaches the top level in the first steps
                s["model"].step(dt)
        s["masks"] = [(l.level, name, _pinned(k * l.NN, torch.int32)) for l in levels
                      for name, k in (("mask_n", 1), ("mask_e", 3))]
    elif kind == "solve":
        s["model"] = S = _solver(levels, seed, case["dt"])
        f = S.field()
        f[S.offsets[-2]:] = elliptic_rhs(g, seed=seed)
        S.upload(f=f)
        S.restrict()
        _, s["f"] = S.download()
        s["u0"], s["u"], s["opts"] = S.field(), _pinned(int(S.offsets[-1])), _opts(case)
    else:
        s["model"] = S = _solver(levels, seed, case["dt"])
        S.learned_setup(1)
        S.learned_params(_network(seed))
        s["r"], s["e"] = _pair(levels, seed)
    return s


def run(s):
    case, m = s["case"], s["model"]
    kind, g = case["kind"], s["levels"][-1]
    n = g.n
    if kind == "host":
        m.rk4_host(s["dt"], case["steps"], *s["out"])
    elif kind == "rk4":
        m.rk4(s["dt"], case["steps"])
        _native.check("wt_download_state", _native.lib().wt_download_state(m.h, *[_native.dptr(a) for a in s["out"]]))
    elif kind in ("tree", "dense", "split"):
        for _ in range(case["steps"]):
            m.step(s["dt"])
        if kind == "dense":
            m.dev.download_many([(g.level, name, a) for name, a in zip(("mass", "temp", "velo"), s["out"])])
        m.dev.download_many(s["masks"])
        masks = [a for _, _, a in s["masks"]]
        if kind != "dense":
            count = m.dev.download_tree_state(s["out"])
            got = [count, *s["out"]] + masks + [m.dev.tree(g.level, m.patch_size)[0]]
            if kind == "split":
                got.append(m.dev.free_surface(g.level).reshape(10, g.P, g.P)[:, 2:n + 2, 2:n + 2])
            return got
    elif kind == "solve":
        m.upload(u=s["u0"], f=s["f"])
        m.solve(s["opts"])
        _native.check("wt_elliptic_download",
                      _native.lib().wt_elliptic_download(m.h, _native.dptr(s["u"]), None))
        return s["u"][m.offsets[-2]:].reshape(10, g.P, g.P)[:, 2:n + 2, 2:n + 2]
    elif case["grad"]:
        return m.learned_grad(s["r"], s["e"])
    else:
        return m.learned_infer(s["r"])
    mass, temp, velo = s["out"]     # the nodes [0, n]^2 (with the poles) and the owned edges
    nz = case["nz"]
    state = [a.reshape(nz, 10, g.P, g.P)[:, :, 2:n + 3, 2:n + 3] for a in (mass, temp)]
    state.append(velo.reshape(nz, 3, 10, g.P, g.P)[:, :, :, 2:n + 2, 2:n + 2])
    return state + masks if kind == "dense" else state


# -------------------------------------------------------------------- work

# Node-layers of one RK stage read the stage state, the base state and the layer means and write the new state
# (17 words); the operators cost about 330 operations each.
_STAGE_BYTES, _STAGE_FLOPS = 17 * 8, 330
# Share of the nodes above the coarsest level that the patch trees of these flows hold after a few steps.
_TREE_SHARE = 0.15


def work(case):
    kind = case["kind"]
    nodes = [10 * 4 ** l for l in range(case.get("lo", case.get("level")), case.get("hi", case.get("level")) + 1)]
    if kind in ("host", "rk4"):
        k = nodes[0] * case["nz"]
        return {"bytes": case["steps"] * 4 * (k * _STAGE_BYTES + nodes[0] * 23 * 8) + 5 * 8 * k,
                "flops": case["steps"] * 4 * k * _STAGE_FLOPS}
    if kind in ("tree", "dense", "split"):
        share = 1.0 if kind == "dense" else _TREE_SHARE
        k = (nodes[0] + share * sum(nodes[1:])) * case["nz"]
        # beside the stage: wavelets of 5 fields written and read, the state rebuilt (15 words)
        return {"bytes": case["steps"] * k * (4 * (_STAGE_BYTES + 15 * 8) + 15 * 8),
                "flops": case["steps"] * k * 4 * (_STAGE_FLOPS + 150)}
    if kind == "solve":
        # about ten multigrid cycles: 5 operator passes of 8 words on 4/3 of the finest level's nodes
        return {"bytes": 10 * 5 * sum(nodes) * 8 * (4 if case["method"] == "mixed" else 8),
                "flops": 10 * 5 * sum(nodes) * 20}
    weights = 7 * (2 * 32 + 32 * 32 + 32)
    passes = 3 if case["grad"] else 1
    return {"bytes": passes * nodes[-1] * (16 + 4 * 64 + 28), "flops": passes * 2 * weights * nodes[-1]}


# ------------------------------------------------------------- exact values


def _dev():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _t(a):
    return torch.as_tensor(np.ascontiguousarray(a)).to(_dev())


class _Ghosts:
    def __init__(self, g):
        hn, he = _t(g.halo_node), _t(g.halo_edge)
        self.nd, self.ns, self.ed, self.es = hn[:, 0], hn[:, 1], he[:, 0], he[:, 1]
        self.sign = torch.where(he[:, 2] < 0, -1.0, 1.0).double()

    def nodes(self, f):
        f[..., self.nd] = f[..., self.ns]
        return f

    def edges(self, f):
        """f: (..., 3, NN)"""
        flat = f.view(*f.shape[:-2], -1)
        flat[..., self.ed] = flat[..., self.es] * self.sign
        return f


def _shifts(P):
    """Readers of the neighbours of every node."""
    off = {"E": 1, "W": -1, "N": P, "S": -P, "NE": P + 1, "SW": -P - 1, "SE": 1 - P, "NW": P - 1}
    return {k: functools.partial(torch.roll, shifts=-o, dims=-1) for k, o in off.items()}


def _corner_pv(g, r, up, part, cor, qe):
    """Potential vorticity at the pentagon corners of every lozenge, where two triangles merge into one."""
    n, P = g.n, g.P
    d = torch.arange(10, device=r.device) * P * P

    def at(i, j):
        return d + (j + 2) * P + i + 2

    def R(x, *parts):
        return sum(r[:, x] * part[k - 1, x] for k in parts)

    def mean(a, b):
        return 0.5 * (a + b)

    u = lambda e, x: up[:, e, x]  # noqa: E731
    x, N, E, S, W = at(n, n), at(n, n + 1), at(n + 1, n), at(n, n - 1), at(n - 1, n)
    pv = (cor[0, x] + u(RT, x) - u(RT, N) - u(UP, x)) / (R(E, 3) + R(x, 1, 2) + R(N, 6))
    pw = (cor[0, W] + u(RT, W) + u(UP, x) + u(DG, W)) / (R(W, 1) + R(x, 3) + R(N, 5))
    ps = (cor[1, S] - u(DG, S) - u(UP, S) - u(RT, x)) / (R(S, 2) + R(E, 4) + R(x, 6))
    new = [(RT, x, mean(pv, ps)), (UP, x, mean(pv, pw))]
    x, E, S, W, NE, SW = at(n, 0), at(n + 1, 0), at(n, -1), at(n - 1, 0), at(n + 1, 1), at(n - 1, -1)
    pv = (cor[0, SW] - u(RT, x) + u(RT, SW) + u(DG, SW)) / (R(SW, 1) + R(S, 3) + R(x, 5, 6))
    pl = (cor[0, x] + u(RT, x) + u(UP, E) + u(DG, x)) / (R(x, 1) + R(E, 3) + R(NE, 5))
    pu = (cor[1, SW] - u(RT, W) - u(DG, SW) - u(UP, SW)) / (R(SW, 2) + R(x, 4) + R(W, 6))
    new += [(RT, x, mean(pv, pl)), (DG, SW, mean(pv, pu))]
    x, N, E, S, W, SW = at(0, 0), at(0, 1), at(1, 0), at(0, -1), at(-1, 0), at(-1, -1)
    pw = (cor[0, W] + u(RT, W) + u(UP, x) + u(DG, W)) / (R(W, 6) + R(x, 4, 5) + R(S, 3))
    pv = (cor[0, SW] + u(UP, S) - u(RT, W) + u(RT, SW)) / (R(W, 1) + R(x, 3) + R(N, 5))
    ps = (cor[1, S] - u(RT, x) - u(DG, S) - u(UP, S)) / (R(S, 2) + R(E, 4) + R(x, 6))
    new += [(RT, W, mean(pw, pv)), (UP, S, mean(ps, pv))]
    x, N, S, W, NE, SW = at(0, n), at(0, n + 1), at(0, n - 1), at(-1, n), at(1, n + 1), at(-1, n - 1)
    pv = (cor[1, SW] + u(UP, x) - u(DG, SW) - u(UP, SW)) / (R(SW, 2) + R(x, 3, 4) + R(W, 6))
    pu = (cor[1, x] - u(DG, x) - u(UP, x) - u(RT, N)) / (R(x, 2) + R(NE, 4) + R(N, 6))
    pl = (cor[0, SW] + u(RT, SW) + u(UP, S) + u(DG, SW)) / (R(SW, 1) + R(S, 3) + R(x, 5))
    new += [(UP, x, mean(pv, pu)), (DG, SW, mean(pl, pv))]
    for e, x, q in new:
        qe[:, e, x] = q


def _exact_rk4(case, seed):
    g, nz, dt = _geom(case)[-1], case["nz"], _dt(case)
    ph, n, NN = OceanParams(), g.n, g.NN
    st = {k: _t(v) for k, v in _water((g.level,) * 2, g.level, nz, seed, False).items()}
    gh, sh = _Ghosts(g), _shifts(g.P)
    E, W, N, S, NE, SW, SE, NW = (sh[k] for k in ("E", "W", "N", "S", "NE", "SW", "SE", "NW"))
    ln, ped, part, hinv, cor = _t(g.len), _t(g.pedlen), _t(g.part), _t(g.hex_inv), _t(g.coriolis)
    _, i, j = (_t(a) for a in g.ij())
    scal = (i >= 0) & (j >= 0) & (i <= n) & (j <= n)
    own = (i >= 0) & (j >= 0) & (i < n) & (j < n)

    def weights(offs):
        acc, w = part[offs], []
        for q in range(5):
            if q:
                acc = acc + part[(q + offs) % 6]
            w.append((0.5 - acc * hinv) * (-1.0 if q % 2 else 1.0))
        return w

    wgt = [weights(k) for k in range(6)]

    def trend(m, t, v):
        gh.nodes(m), gh.nodes(t), gh.edges(v)
        r, th = m + st["mean_m"], t + st["mean_t"]
        weight = ph.grav * (r - th)
        upper = weight.sum(0) + ph.p_top - weight.cumsum(0)
        pressure = upper + 0.5 * weight
        thick = ph.grav * r / ph.ref_density
        phi = ph.grav * st["topo"] + thick.cumsum(0) - 0.5 * thick
        up, ud = v * ln, v * ped
        ur, ug, uu = up.unbind(1)
        low = (cor[0] + ur + E(uu) + ug) / (r * part[0] + E(r * part[2]) + NE(r * part[4]))
        upl = (cor[1] - ug - uu - N(ur)) / (r * part[1] + NE(r * part[3]) + N(r * part[5]))
        qe = 0.5 * torch.stack([S(upl) + low, upl + low, upl + W(low)], 1)
        _corner_pv(g, r, up, part, cor, qe)
        e = (up * ud).unbind(1)
        ke = (e[0] + e[1] + e[2] + W(e[0]) + SW(e[1]) + S(e[2])) * hinv / 4.0
        bern = ke + phi + pressure / ph.ref_density
        fm, ft = (gh.edges(torch.stack([ud[:, 0] * 0.5 * (a + E(a)), ud[:, 1] * 0.5 * (a + NE(a)),
                                        ud[:, 2] * 0.5 * (a + N(a))], 1)) for a in (r, th))
        out = []
        for f in (fm, ft):
            div = (f[:, 0] - W(f[:, 0]) + SW(f[:, 1]) - f[:, 1] + f[:, 2] - S(f[:, 2])) * hinv
            out.append(torch.where(scal, -div, 0.0))
        theta = th / r
        dv = torch.zeros_like(v)
        same = lambda x: x  # noqa: E731
        around = (  # the ten edges each edge's Coriolis term averages over: five about each end
            (E, 0, 3, ((DG, same), (UP, same), (RT, W), (DG, SW), (UP, S)),
             ((DG, S), (UP, SE), (RT, E), (DG, E), (UP, E))),
            (NE, 1, 4, ((UP, same), (RT, W), (DG, SW), (UP, S), (RT, same)),
             ((UP, E), (RT, NE), (DG, NE), (UP, NE), (RT, N))),
            (N, 2, 5, ((RT, W), (DG, SW), (UP, S), (RT, same), (DG, same)),
             ((RT, N), (DG, N), (UP, N), (RT, NW), (DG, W))))
        for k, (nb, o1, o2, first, second) in enumerate(around):
            q = 0.0
            for ws, es, mv in ((wgt[o1], first, same), (wgt[o2], second, nb)):
                for w, (e1, at) in zip(ws, es):
                    q = q + at(fm[:, e1]) * 0.5 * (at(qe[:, e1]) + qe[:, k]) * mv(w)
            sign = -1.0 if k == DG else 1.0     # DG points from the north-east node to this one
            grad = sign * ((nb(bern) - bern) - 0.5 * (theta + nb(theta)) * (nb(phi) - phi))
            dv[:, k] = torch.where(own, (-q - grad) / ln[k], 0.0)
        return out[0], out[1], dv

    q = [st["mass"].clone(), st["temp"].clone(), st["velo"].reshape(nz, 3, NN).clone()]
    for _ in range(case["steps"]):
        x = [a.clone() for a in q]
        for h in (dt / 4, dt / 3, dt / 2, dt):
            x = [a + h * b for a, b in zip(q, trend(*x))]
        q = x
    gh.nodes(q[0]), gh.nodes(q[1]), gh.edges(q[2])
    state = [a.reshape(nz, 10, g.P, g.P)[:, :, 2:n + 3, 2:n + 3] for a in q[:2]]
    return state + [q[2].reshape(nz, 3, 10, g.P, g.P)[:, :, :, 2:n + 2, 2:n + 2]]


def _operator(g, topo, dt):
    """L(u) = dt^2 div(g |H| grad u) - u of one level, on arrays whose ghosts it fills itself."""
    gh, sh, ph = _Ghosts(g), _shifts(g.P), OceanParams()
    csq, ln, ped, hinv = ph.grav * _t(topo).abs(), _t(g.len), _t(g.pedlen), _t(g.hex_inv)
    K = [0.5 * (csq + sh[k](csq)) * torch.where(ln[e] > 0, ped[e] / ln[e], 0.0)
         for e, k in ((RT, "E"), (DG, "NE"), (UP, "N"))]

    def apply(u):
        u = gh.nodes(u.clone())
        f = gh.edges(torch.stack([K[0] * (sh["E"](u) - u), K[1] * (u - sh["NE"](u)), K[2] * (sh["N"](u) - u)]))
        div = f[0] - sh["W"](f[0]) + sh["SW"](f[1]) - f[1] + f[2] - sh["S"](f[2])
        return dt * dt * div * hinv - u

    return apply


def _exact_solve(case, seed):
    levels = _geom(case)
    g = levels[-1]
    L = _operator(g, bathymetry(g, seed=seed, nterms=24), case["dt"])
    sel = torch.zeros(g.NN, dtype=torch.double, device=_dev())
    sel[_t(_nodes(levels))] = 1.0
    f = _t(elliptic_rhs(g, seed=seed)) * sel
    A = lambda x: L(x) * sel  # noqa: E731
    u, goal = torch.zeros_like(f), 1e-14 * float(f.norm())
    for _ in range(8):      # BiCGSTAB, restarted from the true residual
        r = f - A(u)
        if float(r.norm()) <= goal:
            break
        r0, p = r.clone(), r.clone()
        rho = r0 @ r
        for _ in range(600):
            ap = A(p)
            alpha = rho / (r0 @ ap)
            t = r - alpha * ap
            at = A(t)
            omega = (at @ t) / (at @ at)
            u = u + alpha * p + omega * t
            r = t - omega * at
            if float(r.norm()) <= 0.1 * goal:
                break
            rho, old = r0 @ r, rho
            p = r + (rho / old) * (alpha / omega) * (p - omega * ap)
    n = g.n
    return u.reshape(10, g.P, g.P)[:, 2:n + 2, 2:n + 2]


def _exact_learned(case, seed):
    levels = _geom(case)
    g = levels[-1]
    n, P = g.n, g.P
    slot = _nodes(levels)
    src = np.arange(g.NN)
    src[g.halo_node[:, 0]] = g.halo_node[:, 1]
    where = np.full(g.NN, slot.size)
    where[slot] = np.arange(slot.size)
    tap = [_t(where[src[slot + dj * P + di]]) for di, dj in TAPS]
    topo = bathymetry(g, seed=seed, nterms=24)
    r, e = (_t(a) for a in _pair(levels, seed))
    rs = r.square().mean().sqrt()
    depth = _t(np.abs(topo[slot]) / 2750.0 - 1.0)
    theta = _t(_network(seed).astype(np.float64))
    W, o = [], 0
    for ci, co in ((2, 32), (32, 32), (32, 1)):
        W.append(theta[o:o + 7 * ci * co].reshape(7, ci, co).clone().requires_grad_(True))
        o += 7 * ci * co
    with torch.enable_grad():
        h = torch.stack([r / rs, r / rs * depth], 1)
        for w in W:
            pad = torch.cat([h, torch.zeros_like(h[:1])])
            h = sum(pad[tap[k]] @ w[k] for k in range(7))
        y = h[:, 0]
    i, j = slot % P - 2, slot // P % P - 2
    own = _t(((i < n) & (j < n)).astype(np.float64))
    if not case["grad"]:
        return (rs * y * own).detach()
    full = torch.zeros(g.NN, dtype=torch.double, device=_dev())
    full[_t(slot)] = (own * y - e / rs).detach()
    area = 1.0 / _t(g.hex_inv[slot])
    a = -_operator(g, topo, case["dt"])(full)[_t(slot)] * area / area.sum()
    loss = float((full[_t(slot)] * a).sum())
    y.backward(2.0 * own * a)
    return loss, torch.cat([w.grad.reshape(-1) for w in W])


def exact(case, seed):
    """The results in 64 bits from the formulas; None for the adaptive runs, whose masks, tree and transforms
    would take minutes in plain array code."""
    if case["kind"] in ("host", "rk4"):
        return _exact_rk4(case, seed)
    if case["kind"] == "solve":
        return _exact_solve(case, seed)
    if case["kind"] == "learned":
        return _exact_learned(case, seed)
    return None

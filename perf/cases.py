"""The chemistry engine's work as a flow solver's program has it done, for timing.

listed() and draw() give cases, prepare() what the program holds before the call, run() one pass through
the public entry points, work() what a pass cannot do without, and exact() the same results in plain
64-bit torch, written from the published equations of the update.

Mechanisms are the repository's own pre-processor outputs (tests/golden/mech), cells its seeded workloads.
A pass that updates cells in place starts from a copy of the prepared state, as a solver's stage would, so
that it can be repeated.  Intervals run from 1e-7 to 1e-6 s, the flow time steps of the workloads; fresh cells
(dt_chem = -1) and cells that carry a step size both occur.  The Runge-Kutta mechanisms (air) take 1e-7 to
2e-7 s: over longer intervals the step size that their nearly steady cells hand on is a difference of rounding errors.
"""
import math
import os
import re

import numpy as np
import torch

from gdtk_gb300.cells import ReactorCells, ReactorCells2T
from gdtk_gb300.gas import GasModel, GasState, ThermochemicalReactor
from gdtk_gb300 import workloads

MECH = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "tests", "golden", "mech")
PARK5 = ["N2", "O2", "NO", "N", "O"]
METHANE_AIR = {"CH4": 1.0, "O2": 2.0, "N2": 7.52}
EXACT_CELLS = 24000            # above this the plain update takes too long


def listed():
    return [
        # one cell through the per-state binding: a script's constant-volume reactor, latency only
        dict(name="state-h2air", kind="state", mech="j92", dt=1.0e-7),
        # a small block of Park air behind a shock (RKF), fresh step sizes
        dict(name="air5-4096", kind="cells", mech="park5", n=4096, dt=2.0e-7),
        # the smallest block of the H2-air batch, an odd number of cells
        dict(name="h2air-2053", kind="cells", mech="j92", n=2053, dt=1.0e-6),
        # a solver that keeps its cells on the host: copies in, update, copies out
        dict(name="h2air-host-20011", kind="host", mech="j92", n=20011, dt=1.0e-7),
        # a mixing layer within its time loop: step sizes carried, the cold fuel stream frozen
        dict(name="layer-131072", kind="layer", mech="j92", nx=512, ny=256, dt=5.0e-7),
        # uneven blocks of a multi-block grid in one launch, each with its own interval
        dict(name="h2air-blocks-9", kind="blocks", mech="j92", nblocks=9, n_min=1500, n_max=24000),
        # the ordinary batch at size: half cold, half igniting
        dict(name="h2air-262147", kind="cells", mech="j92", n=262147, dt=1.0e-6),
        # methane-air with pressure-dependent (Troe) rates, 21 species
        dict(name="drm19-9001", kind="cells", mech="drm19", n=9001, dt=1.0e-6),
        # the 75-species acetylene mechanism on shock-tube states
        dict(name="c2h2-6007", kind="cells", mech="c2h2", n=6007, dt=1.0e-6),
        # two-temperature air: the multi-temperature reactor
        dict(name="air2t-65536", kind="air2t", mech="park2t", n=65536, dt=2.0e-7),
        # source terms of every cell, for a solver that integrates the chemistry itself
        dict(name="source-h2air-600011", kind="source", mech="j92", n=600011),
        # the surrogate network's increments for a block of cells
        dict(name="surrogate-262147", kind="surrogate", mech="j92", n=262147),
    ]


def draw(rng):
    def log(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    def dt(mech="j92"):
        most = 2.0e-7 if mech.startswith("park") else 1.0e-6
        return float("%.3g" % math.exp(rng.uniform(math.log(1.0e-7), math.log(most))))

    kind = rng.choice(["state", "air5", "h2air", "h2air", "host", "layer", "blocks", "drm19", "c2h2", "air2t", "source",
                       "surrogate"])
    if kind == "state":
        mech = rng.choice(["j92", "park5", "drm19"])
        return dict(kind="state", mech=mech, dt=dt(mech))
    if kind == "air5":
        return dict(kind="cells", mech="park5", n=log(256, 65536), dt=dt("park5"))
    if kind == "h2air":
        return dict(kind="cells", mech="j92", n=log(300, 200000), dt=dt())
    if kind == "host":
        mech = rng.choice(["j92", "park5"])
        return dict(kind="host", mech=mech, n=log(500, 24000), dt=dt(mech))
    if kind == "layer":
        return dict(kind="layer", mech="j92", nx=log(32, 512), ny=log(64, 400), dt=5.0e-7)
    if kind == "blocks":
        return dict(kind="blocks", mech="j92", nblocks=rng.randrange(2, 14), n_min=log(500, 2000), n_max=log(4000, 24000))
    if kind == "drm19":
        return dict(kind="cells", mech="drm19", n=log(300, 12000), dt=dt())
    if kind == "c2h2":
        return dict(kind="cells", mech="c2h2", n=log(200, 8000), dt=dt())
    if kind == "air2t":
        return dict(kind="air2t", mech=rng.choice(["park2t", "park2tmt"]), n=log(500, 100000), dt=dt("park2t"))
    if kind == "source":
        return dict(kind="source", mech=rng.choice(["j92", "park5", "drm19"]), n=log(2000, 600000))
    return dict(kind="surrogate", mech="j92", n=log(2000, 400000))


# ------------------------------------------------------------------------------------- prepare and run
_KEPT = {}


def _path(name):
    return os.path.join(MECH, name + ".lua")


def _reactor(mech):
    """The reactor that a program makes once from its mechanism files."""
    if mech not in _KEPT:
        if mech.startswith("park2t"):
            _KEPT[mech] = ReactorCells2T(_path(mech + "-gas"), _path(mech + "-chem"), _path(mech + "-eem"))
        else:
            _KEPT[mech] = ReactorCells(_path(mech + "-gas"), _path(mech + "-chem"))
    return _KEPT[mech]


def _species(mech):
    """Species names and molar masses of a mechanism's gas file."""
    g = _lua(mech + "-gas")
    names = _list(g["species"])
    return names, np.array([g["db"][s]["M"] for s in names])


def _host_cells(case, seed):
    """Seeded T, p (n,) and Y (nsp, n) of a case, on the host."""
    mech, n = case["mech"], case.get("n", 1)
    names, M = _species(mech)
    if mech == "park5":
        return workloads.air5_cells(n, seed=seed)
    if mech == "c2h2":
        return workloads.acetylene_cells(names, M, n, seed=seed)
    if mech == "drm19":   # premixed methane-air with a share of the other species, hot enough to react
        rng = np.random.Generator(np.random.PCG64(seed))
        x = np.array([METHANE_AIR.get(s, 0.0) for s in names])
        y0 = x * M / (x * M).sum()
        minor = [i for i, s in enumerate(names) if s not in METHANE_AIR]
        share = 10.0 ** rng.uniform(-6.0, -2.0, n)
        Y = np.repeat(y0[None, :], n, axis=0) * (1.0 - share)[:, None]
        Y[:, minor] += share[:, None] * rng.dirichlet(np.full(len(minor), 0.5), n)
        return rng.uniform(1100.0, 2400.0, n), 10.0 ** rng.uniform(4.3, 5.7, n), np.ascontiguousarray(Y.T)
    if case["kind"] == "layer":
        return workloads.h2air_mixing_layer(names, M, nx=case["nx"], ny=case["ny"], seed=seed)
    if case["kind"] in ("source", "surrogate"):
        # a field of burnt, unburnt and mixing cells: the mixing layer's streams at many temperatures
        rng = np.random.Generator(np.random.PCG64(seed))
        w = rng.dirichlet(np.full(len(names), 0.3), 4096)[rng.integers(0, 4096, n)]
        Y = 0.8 * w
        Y[:, names.index("N2")] += 0.2
        return rng.uniform(600.0, 3000.0, n), 10.0 ** rng.uniform(4.3, 5.7, n), np.ascontiguousarray(Y.T)
    hot = (1100.0, 2800.0) if case["kind"] != "state" else (1300.0, 2200.0)
    return workloads.h2air_cells(names, M, n, seed=seed, gas_file=_path(mech + "-gas"), T_hot=hot,
                                 frozen_fraction=0.0 if case["kind"] == "state" else 0.5)


def _dev(a):
    return torch.tensor(np.ascontiguousarray(a), dtype=torch.float64, device="cuda")


def _block(rc, T, p, Y, dt, dt_chem=None):
    T, p, Y = _dev(T), _dev(p), _dev(Y)
    rho, u = rc.thermo_from_pT(p, T, Y)
    n = T.shape[0]
    return dict(rho=rho, u=u, T=T, p=p, massf=Y, t_interval=dt,
                dt_chem=_dev(dt_chem) if dt_chem is not None else torch.full((n,), -1.0, dtype=torch.float64, device="cuda"),
                status=torch.zeros(n, dtype=torch.int32, device="cuda"))


def _sizes(case):
    """Cells of each block: from n_min to n_max in equal ratios, large and small ones in turn."""
    k, r = case["nblocks"], case["n_max"] / case["n_min"]
    n = [int(round(case["n_min"] * r ** (i / (k - 1)))) for i in range(k)]
    return n[::2] + n[1::2][::-1]


def _grid(case, seed):
    """Blocks of a grid, each with its own cold share, ranges of T and p, and interval."""
    names, M = _species(case["mech"])
    rng = np.random.Generator(np.random.PCG64(seed))
    out = []
    for b, n in enumerate(_sizes(case)):
        cold, hot = np.sort(rng.uniform(300.0, 600.0, 2)), np.sort(rng.uniform(1100.0, 2800.0, 2))
        lp = np.sort(rng.uniform(math.log10(2.0e4), math.log10(5.0e5), 2))
        T, p, Y = workloads.h2air_cells(names, M, n, seed=1000 * seed + b, frozen_fraction=float(rng.uniform()), T_cold=tuple(cold),
                                        T_hot=tuple(hot), p_range=tuple(10.0 ** lp), gas_file=_path(case["mech"] + "-gas"))
        out.append(dict(T=T, p=p, Y=Y, dt=(1.0e-7, 1.0e-6)[b % 2]))
    return out


def _views(nsp, flat):
    """The blocks of a grid whose fields lie one block after the other."""
    blocks, at = [], 0
    for n, dt in zip(flat["sizes"], flat["dts"]):
        b = {k: flat[k][at:at + n] for k in ("rho", "u", "T", "p", "dt_chem", "status")}
        blocks.append(dict(b, massf=flat["massf"][nsp * at:nsp * (at + n)].view(nsp, n), t_interval=dt))
        at += n
    return blocks


def _layer_steps(n, seed):
    """The step sizes that cells carry from one flow step to the next."""
    rng = np.random.Generator(np.random.PCG64(seed + 77))
    return 10.0 ** rng.uniform(-9.0, -6.5, n)


def _network(case, seed):
    """Network parameters and normalisation as training leaves them in size: [16, 256 x 4, 16] for J92."""
    rng = np.random.Generator(np.random.PCG64(seed + 5))
    dims = [16, 256, 256, 256, 256, 16]
    W = [rng.normal(0.0, 1.2 / math.sqrt(a), (b, a)).astype(np.float32) for a, b in zip(dims[:-1], dims[1:])]
    b = [rng.normal(0.0, 0.1, d).astype(np.float32) for d in dims[1:]]
    norm = dict(x_shift=rng.normal(0.0, 0.3, 16).astype(np.float32), x_scale=rng.uniform(0.5, 2.0, 16).astype(np.float32),
                y_shift=rng.normal(0.0, 0.01, 16).astype(np.float32), y_scale=rng.uniform(0.5, 2.0, 16).astype(np.float32),
                x_min=np.full(16, -1e30), x_max=np.full(16, 1e30))
    return W, b, norm


def _features(case, seed):
    """Raw features (n, 16) float32: ln T, ln p, Y, ln dt, brought to the scale of the normalisation above."""
    T, p, Y = _host_cells(case, seed)
    X = np.concatenate([np.log(T / 1500.0)[None], np.log(p / 1.0e5)[None], Y, np.zeros((1, len(T)))]).T
    return np.ascontiguousarray(X, np.float32)


def prepare(case, seed):
    kind = case["kind"]
    if kind == "state":
        T, p, Y = _host_cells(case, seed)
        key = ("state", case["mech"])
        if key not in _KEPT:
            gm = GasModel(_path(case["mech"] + "-gas"))
            _KEPT[key] = gm, ThermochemicalReactor(gm, _path(case["mech"] + "-chem"))
        gm, reactor = _KEPT[key]
        # gas states are never given back by the C ABI: as a script does, the two are made once and filled again
        if ("gs", seed) not in _KEPT:
            _KEPT["gs", seed] = {}
        made = _KEPT["gs", seed]
        if case["mech"] not in made:
            made[case["mech"]] = GasState(gm), GasState(gm)
        start, gs = made[case["mech"]]
        start.p, start.T, start.massf = float(p[0]), float(T[0]), [float(y) for y in Y[:, 0]]
        start.update_thermo_from_pT()
        return dict(case=case, reactor=reactor, start=start, gs=gs)
    rc = _reactor(case["mech"])
    if kind in ("cells", "layer"):
        T, p, Y = _host_cells(case, seed)
        s = _block(rc, T, p, Y, case["dt"], _layer_steps(len(T), seed) if kind == "layer" else None)
        return dict(case=case, rc=rc, T_frozen=300.0 if kind == "layer" else 0.0, **s)
    if kind == "blocks":
        raw = _grid(case, seed)
        made = [_block(rc, b["T"], b["p"], b["Y"], b["dt"]) for b in raw]
        flat = {k: torch.cat([b[k].reshape(-1) for b in made]) for k in ("rho", "u", "T", "p", "massf", "dt_chem", "status")}
        return dict(case=case, rc=rc, sizes=[len(b["T"]) for b in raw], dts=[b["dt"] for b in raw], **flat)
    if kind == "host":
        T, p, Y = _host_cells(case, seed)
        s = _block(rc, T, p, Y, case["dt"])
        pin = lambda t: t.cpu().pin_memory()   # noqa: E731
        start = {k: pin(s[k]) for k in ("rho", "u", "T", "p", "massf", "dt_chem", "status")}
        work = {k: v.clone().pin_memory() for k, v in start.items()}
        return dict(case=case, rc=rc, start={k: v.numpy() for k, v in start.items()}, work={k: v.numpy() for k, v in work.items()},
                    keep=(start, work))
    if kind == "air2t":
        T, Tve, p, Y = workloads.air2t_cells(case["n"], seed=seed)
        T, Tve, p, Y = _dev(T), _dev(Tve), _dev(p), _dev(Y)
        rho, u, uve = rc.thermo_from_pT(p, T, Tve, Y)
        return dict(case=case, rc=rc, rho=rho, T=T, Tve=Tve, p=p, massf=Y, u=u, u_ve=uve,
                    dt_chem=torch.full_like(T, -1.0), status=torch.zeros(T.shape[0], dtype=torch.int32, device="cuda"))
    if kind == "source":
        T, p, Y = _host_cells(case, seed)
        T, p, Y = _dev(T), _dev(p), _dev(Y)
        rho, _ = rc.thermo_from_pT(p, T, Y)
        return dict(case=case, rc=rc, rho=rho, T=T, massf=Y)
    from gdtk_gb300.surrogate import ChemSurrogate
    sg = ChemSurrogate(rc, width=256, depth=4)
    W, b, norm = _network(case, seed)
    sg.set_params(np.concatenate([w.ravel() for w in W] + b))
    sg.set_normalisation(**norm)
    return dict(case=case, sg=sg, X=torch.tensor(_features(case, seed), device="cuda"))


def run(state):
    kind = state["case"]["kind"]
    if kind == "state":
        gs = state["gs"]
        gs.copy_values(state["start"])
        dt_chem = state["reactor"].update_state(gs, state["case"]["dt"])
        gs.update_thermo_from_rhou()
        return dict(T=np.float64(gs.T), p=np.float64(gs.p), massf=np.array(gs.massf), dt_chem=np.float64(dt_chem))
    rc = state.get("rc")
    if kind in ("cells", "layer"):
        out = {k: state[k].clone() for k in ("T", "p", "massf", "dt_chem", "status")}
        rc.update(state["rho"], state["u"], out["T"], out["p"], out["massf"], out["dt_chem"], state["case"]["dt"],
                  status=out["status"], T_frozen=state["T_frozen"])
        return out
    if kind == "blocks":
        out = {k: state[k].clone() for k in ("T", "p", "massf", "dt_chem", "status")}
        rc.update_blocks(_views(rc.nsp, dict(state, **out)))
        return out
    if kind == "host":
        w, s = state["work"], state["start"]
        for k in ("T", "p", "massf", "dt_chem"):
            np.copyto(w[k], s[k])
        rc.update_host(w["rho"], w["u"], w["T"], w["p"], w["massf"], w["dt_chem"], state["case"]["dt"], status=w["status"])
        return {k: w[k] for k in ("T", "p", "massf", "dt_chem", "status")}
    if kind == "air2t":
        out = {k: state[k].clone() for k in ("T", "Tve", "p", "massf", "u", "u_ve", "dt_chem", "status")}
        rc.update(state["rho"], out["T"], out["Tve"], out["p"], out["massf"], out["dt_chem"], state["case"]["dt"],
                  status=out["status"], u=out["u"], u_ve=out["u_ve"])
        return out
    if kind == "source":
        return rc.source_terms(state["rho"], state["T"], state["massf"])
    return state["sg"].predict(state["X"])


# FP64 operations that an update of one cell over 1e-6 s takes (adds, multiplies, two for each fused one), as counted
# on the cells of these workloads; an update over dt takes about (dt / 1e-6)^0.45 of it.
_OPS = {"park5": 6.0e4, "j92": 1.0e6, "drm19": 2.0e6, "c2h2": 7.0e6, "park2t": 5.3e5, "park2tmt": 5.3e5}
_NSP = {"park5": 5, "j92": 13, "drm19": 21, "c2h2": 75, "park2t": 5, "park2tmt": 5}


def work(case):
    kind, mech = case["kind"], case["mech"]
    nsp = _NSP[mech]
    if kind == "surrogate":
        return dict(bytes=case["n"] * 32 * 4 + 4 * 205000, flops=2.0 * case["n"] * (2 * 16 * 256 + 3 * 256 * 256))
    if kind == "source":
        return dict(bytes=8.0 * case["n"] * (2 + 2 * nsp), flops=case["n"] * {"park5": 1.0e3, "j92": 4.0e3, "drm19": 1.0e4}[mech])
    if kind == "blocks":   # half the blocks take 1e-7 s, half 1e-6 s
        n = sum(_sizes(case))
        ops = 0.68 * _OPS[mech]
    else:
        n = case["nx"] * case["ny"] if kind == "layer" else case.get("n", 1)
        ops = _OPS[mech] * (case["dt"] / 1.0e-6) ** 0.45 * (0.05 if kind == "layer" else 1.0)
    fields = (4, 6) if kind == "air2t" else (5, 3)
    return dict(bytes=n * (8.0 * (sum(fields) + 2 * nsp) + 4), flops=n * ops)


# ------------------------------------------------------------------------------------- plain 64-bit results
R_U, P_ATM = 8.31451, 101.325e3


def _lua(name):
    """The assignments of a pre-processor's output file: nested dicts, numbers, texts and truth values."""
    if ("lua", name) in _KEPT:
        return _KEPT["lua", name]
    with open(_path(name)) as f:
        text = re.sub(r"--[^\n]*", "", f.read())
    tok = re.findall(r"'[^']*'|\"[^\"]*\"|[-+]?(?:\d+\.?\d*|\.\d+)(?:[eE][-+]?\d+)?|[A-Za-z_]\w*|[{}\[\]=,.;]", text)
    at = 0

    def value():
        nonlocal at
        t = tok[at]
        at += 1
        if t == "{":
            d, k = {}, 1
            while tok[at] != "}":
                if tok[at] == "[":
                    at += 1
                    key = value()
                    at += 2            # ] =
                    d[key] = value()
                elif tok[at + 1] == "=":
                    key = tok[at]
                    at += 2
                    d[key] = value()
                else:
                    d[k] = value()
                    k += 1
                if tok[at] in ",;":
                    at += 1
            at += 1
            return d
        if t[0] in "'\"":
            return t[1:-1]
        if t in ("true", "false"):
            return t == "true"
        return int(t) if re.fullmatch(r"[-+]?\d+", t) else float(t)

    out = {}
    while at < len(tok):
        path = [tok[at]]
        at += 1
        while tok[at] != "=":
            if tok[at] == "[":
                at += 1
                path.append(value())
                at += 1
            else:
                path.append(tok[at + 1])
                at += 2
        at += 1
        d = out
        for k in path[:-1]:
            d = d.setdefault(k, {})
        d[path[-1]] = value()
    _KEPT["lua", name] = out
    return out


def _list(d):
    return [d[k] for k in sorted(k for k in d if isinstance(k, int))]


class _Plain:
    """A thermally perfect gas (NASA-9 curves) with a finite-rate mechanism, in plain torch, cells in the last axis."""

    def __init__(self, mech):
        self.dev = torch.device("cuda" if torch.cuda.is_available() else "cpu")
        gas, chem = _lua(mech + "-gas"), _lua(mech + "-chem")
        names = _list(gas["species"])
        self.nsp = n = len(names)
        t = lambda a: torch.tensor(np.asarray(a, dtype=np.float64), device=self.dev)   # noqa: E731
        self.t = t
        self.M = t([gas["db"][s]["M"] for s in names])
        self.R = R_U / self.M
        curves = [gas["db"][s]["thermoCoeffs"] for s in names]
        nseg = max(c["nsegments"] for c in curves)
        A, lo, wd = np.zeros((nseg, 9, n)), np.full((nseg - 1, n), 1e30), np.ones((nseg - 1, n))
        for i, c in enumerate(curves):
            brk, bld = _list(c["T_break_points"]), _list(c["T_blend_ranges"])
            for s in range(c["nsegments"]):
                A[s, :, i] = _list(c["segment%d" % s])
            for s in range(1, c["nsegments"]):
                lo[s - 1, i], wd[s - 1, i] = brk[s] - 0.5 * bld[s - 1], bld[s - 1]
        self.A, self.lo, self.wd = t(A)[..., None], t(lo)[..., None], t(wd)[..., None]
        cfg = chem["config"]
        self.T_lo, self.T_hi = float(cfg["tempLimits"]["lower"]), float(cfg["tempLimits"]["upper"])
        self.step, self.tight, self.attempts = cfg["odeStep"], cfg["tightTempCoupling"], cfg["maxAttempts"]
        rx = _list(chem["reaction"])
        self.nr = m = len(rx)
        self.plain = all(r["frc"]["model"] in ("Arrhenius", "Troe") and r["brc"]["model"] == "fromEqConst" for r in rx)
        if not self.plain:
            return
        k1 = [r["frc"].get("kInf", r["frc"]) for r in rx]
        self.kA, self.kn, self.kC = (t([float(k[x]) for k in k1])[:, None] for x in "AnC")
        nu, re_, pr_, eff = np.zeros((m, n)), np.full((3, m), n), np.full((3, m), n), np.zeros((m, n))
        collider, troe = np.zeros(m, bool), []
        for j, r in enumerate(rx):
            for side, slots, sign in (("reac", re_, -1), ("prod", pr_, 1)):
                k = 0
                for i, c in zip(_list(r[side + "Idx"]), _list(r[side + "Coeffs"])):
                    nu[j, i] += sign * c
                    for _ in range(int(c)):
                        slots[k, j] = i
                        k += 1
            for i, e in r.get("efficiencies", {}).items():
                eff[j, i] = e
            collider[j] = r["type"] == "anonymous_collider"
            if r["frc"]["model"] == "Troe":
                troe.append(j)
        self.nu, self.eff = t(nu), t(eff)
        self.up, self.down = t(np.maximum(nu, 0.0).T), t(np.maximum(-nu, 0.0).T)
        ix = lambda a: torch.tensor(np.asarray(a), device=self.dev)   # noqa: E731
        self.re, self.pr, self.collider, self.troe = ix(re_), ix(pr_), ix(collider)[:, None], troe
        if troe:
            f = [rx[j]["frc"] for j in troe]
            self.k0 = [t([float(x["k0"][y]) for x in f])[:, None] for y in "AnC"]
            col = lambda y, d: t([float(x.get(y, d)) for x in f])[:, None]   # noqa: E731
            self.Fc, self.ta, self.t1, self.t2, self.t3 = (col(y, d) for y, d in (("F_cent", 0.0), ("a", 0.0), ("T1", 0.0),
                                                                                  ("T2", 0.0), ("T3", 1.0)))

    def curve(self, T):
        """The nine coefficients of every species at T, blended between segments."""
        a = self.A[0].expand(9, self.nsp, T.shape[0])
        for s in range(self.lo.shape[0]):
            w = ((T - self.lo[s]) / self.wd[s]).clamp(0.0, 1.0)
            a = a + w * (self.A[s + 1] - a)
        return a

    def h(self, T):     # J/kg
        a, L = self.curve(T), torch.log(T)
        return self.R[:, None] * (-a[0] / T + a[1] * L + T * (a[2] + T * (a[3] / 2 + T * (a[4] / 3 + T * (a[5] / 4 + T * a[6] / 5)))) + a[7])

    def cp(self, T):
        a = self.curve(T)
        return self.R[:, None] * (a[0] / T ** 2 + a[1] / T + a[2] + T * (a[3] + T * (a[4] + T * (a[5] + T * a[6]))))

    def rho_u(self, p, T, Y):
        return p / ((self.R[:, None] * Y).sum(0) * T), (Y * (self.h(T) - self.R[:, None] * T)).sum(0)

    def T_from_u(self, u, Y, T):
        T, live = T.clone(), torch.ones_like(T, dtype=torch.bool)
        R = self.R[:, None]
        for _ in range(10):
            d = -((Y * (self.h(T) - R * T)).sum(0) - u) / (Y * (self.cp(T) - R)).sum(0)
            T = torch.where(live, T + d, T)
            live = live & (d.abs() / T >= 1e-10)
            if not bool(live.any()):
                break
        return T

    def rates(self, T, c):
        T = T.clamp(self.T_lo, self.T_hi)
        a, L = self.curve(T), torch.log(T)
        g = (-a[0] / T ** 2 / 2 + a[1] * (L + 1) / T + a[2] * (1 - L) - T * (a[3] / 2 + T * (a[4] / 6 + T * (a[5] / 12 + T * a[6] / 20)))
             + a[7] / T - a[8])
        kf = self.kA * torch.exp(self.kn * L - self.kC / T)
        if self.troe:
            j = self.troe
            Mb = self.eff[j] @ c
            k0, ki = self.k0[0] * torch.exp(self.k0[1] * L - self.k0[2] / T), kf[j]
            lp = torch.log10((k0 * Mb / ki).clamp(min=1e-30))
            F = torch.where(self.Fc > 0, self.Fc, (1 - self.ta) * torch.exp(-T / self.t3) + torch.where(self.t1 > 0, self.ta * torch.exp(
                -T / self.t1.clamp(min=1e-30)), 0.0) + torch.where(self.t2 > 0, torch.exp(-self.t2 / T), 0.0))
            lF = torch.log10(F.clamp(min=1e-30))
            x = lp - 0.4 - 0.67 * lF
            x = x / (0.75 - 1.27 * lF - 0.14 * x)
            kf[j] = 10.0 ** (lF / (1 + x * x)) * k0 * ki * Mb / (k0 * Mb + ki)
        lnK = -(self.nu @ g) + self.nu.sum(1, keepdim=True) * torch.log(P_ATM / (R_U * T))
        return kf, kf / torch.exp(lnK)

    def qL(self, c, kf, kb):
        c1 = torch.cat([c, torch.ones_like(c[:1])])
        m = torch.where(self.collider, self.eff @ c, 1.0)
        wf = kf * m * c1[self.re[0]] * c1[self.re[1]] * c1[self.re[2]]
        wb = kb * m * c1[self.pr[0]] * c1[self.pr[1]] * c1[self.pr[2]]
        return self.up @ wf + self.down @ wb, self.up @ wb + self.down @ wf

    def first_step(self, c, q, L):
        net = (q - L).abs()
        d = torch.where(q > 1e4 * L, c / (L + 1e-50), c / net)
        d = torch.where((c > 0) & (net > 1e-30), d, 1e6).amin(0).clamp(max=1e6)
        return (1e-3 * d).clamp(1e-15, 1e-10)

    def rkf(self, y, h, kf, kb, k1):
        a = [[1 / 5], [3 / 40, 9 / 40], [3 / 10, -9 / 10, 6 / 5], [-11 / 54, 5 / 2, -70 / 27, 35 / 27],
             [1631 / 55296, 175 / 512, 575 / 13824, 44275 / 110592, 253 / 4096]]
        k = [k1]
        for row in a:
            q, L = self.qL(y + h * sum(x * v for x, v in zip(row, k)), kf, kb)
            k.append(q - L)
        b5, b4 = [37 / 378, 0, 250 / 621, 125 / 594, 0, 512 / 1771], [2825 / 27648, 0, 18575 / 48384, 13525 / 55296, 277 / 14336, 1 / 4]
        o = y + h * sum(x * v for x, v in zip(b5, k))
        e = o - (y + h * sum(x * v for x, v in zip(b4, k)))
        tol = self.step["errTol"]
        err = ((e / (tol + tol * torch.maximum(y.abs(), o.abs()))) ** 2).mean(0).sqrt()
        s = torch.where(err == 0, 10.0, 0.9 * err ** -0.2)
        return o, torch.where(err <= 1, s.clamp(0.2, 10.0), s.clamp(min=0.2)) * h, err <= 1

    def qss(self, y, h, kf, kb, q0, L0):
        eps1, eps2, delta = (self.step[k] for k in ("eps1", "eps2", "delta"))

        def alpha(p):
            s = (p * h).clamp(max=1e50)
            return (180 + s * (60 + s * (11 + s))) / (360 + s * (60 + s * (12 + s)))

        p0 = L0 / (y + 1e-50)
        yp = y + h * (q0 - p0 * y) / (1 + alpha(p0) * h * p0)
        first, out = yp, yp.clone()
        open_ = torch.ones_like(h, dtype=torch.bool)
        for _ in range(self.step["maxIters"]):
            q, L = self.qL(yp, kf, kb)
            p = L / (yp + 1e-50)
            al, pb = alpha(p), 0.5 * (p0 + p)
            yc = y + h * (al * q + (1 - al) * q0 - pb * y) / (1 + al * h * pb)
            out = torch.where(open_, yc, out)
            miss = (((yc - first).abs() >= eps1 * (yc + delta)) & ~(yc < 1e-50)).any(0)
            open_ = open_ & miss
            if not bool(open_.any()):
                break
            yp = yc
        sig = torch.where(out < 1e-50, 0.0, (out - first).abs() / (eps2 * (out + delta))).amax(0)
        x = sig
        for _ in range(3):
            x = x - 0.5 * (x * x - sig) / x
        return out, torch.where(sig <= 0, 10 * h, h * (1 / x + 0.005)), ~open_

    def massf(self, c, rho):
        y = c * self.M[:, None] / rho
        return torch.where(y < 1e-30, 0.0, y)

    def update(self, rho, u, T, p, Y, dt_chem, dt, T_frozen):
        """The operator-split update of every cell; returns T, p, Y, dt_chem (failed and frozen cells unchanged)."""
        out = [T.clone(), p.clone(), Y.clone(), dt_chem.clone()]
        at = torch.nonzero(T > T_frozen).flatten()
        c0 = Y[:, at] * rho[at] / self.M[:, None]
        c0 = torch.where(c0 < 1e-30, 0.0, c0)
        z = torch.zeros_like(T[at])
        s = dict(at=at, c=c0, T=T[at].clone(), h=z.clone(), t=z.clone(), dtS=dt_chem[at].clone(), save=dt_chem[at].clone(), att=z.clone(),
                 cyc=z.clone(), again=z.clone(), new=z + 1)
        kf, kb = self.rates(s["T"], s["c"])
        while s["at"].numel():
            r, U = rho[s["at"]], u[s["at"]]
            if self.tight:
                kf, kb = self.rates(s["T"], s["c"])
            q, L = self.qL(s["c"], kf, kb)
            new = s["new"] > 0
            if bool(new.any()):
                s["h"] = torch.where(new, torch.where(s["dtS"] > dt, z[0] + dt if z.numel() else z, torch.where(
                    s["dtS"] <= 0, self.first_step(s["c"], q, L), s["dtS"])), s["h"])
            begin = s["att"] == 0
            s["save"] = torch.where(begin, s["dtS"], s["save"])
            h = torch.where(begin, torch.minimum(s["h"], dt - s["t"]), s["h"])
            y, hs, ok = self.rkf(s["c"], h, kf, kb, q - L) if self.step["method"] == "rkf" else self.qss(s["c"], h, kf, kb, q, L)
            mf = self.massf(y, r)
            ok = ok & ~((mf.sum(0) - 1).abs() > 1e-3)
            s["new"], s["dtS"] = torch.zeros_like(h), hs
            s["t"] = torch.where(ok, s["t"] + h, s["t"])
            s["c"] = torch.where(ok, y, s["c"])
            grow = torch.where(hs > h, torch.minimum(hs, 1.1 * h), h)
            s["h"] = torch.where(ok, grow, h / 10)
            s["att"] = torch.where(ok, 0.0, s["att"] + 1)
            if self.tight:
                s["T"] = torch.where(ok, self.T_from_u(U, mf, s["T"]), s["T"])
            done = ok & (s["t"] >= dt)
            s["save"] = torch.where(done & (s["cyc"] == 0), hs, s["save"])
            s["cyc"] = torch.where(ok, s["cyc"] + 1, s["cyc"])
            bad = ~ok & ((s["h"] < 1e-15) | (s["att"] >= self.attempts))
            if bool(done.any()):
                i = s["at"][done]
                Yn = self.massf(s["c"][:, done], r[done])
                Yn = Yn / Yn.sum(0)
                Tn = self.T_from_u(U[done], Yn, s["T"][done])
                out[0][i], out[1][i], out[2][:, i], out[3][i] = Tn, r[done] * (self.R[:, None] * Yn).sum(0) * Tn, Yn, s["save"][done]
            if bool(bad.any()):   # once more from the start with a fresh step size
                i, b = s["at"][bad], bad
                cb = Y[:, i] * rho[i] / self.M[:, None]
                s["c"][:, b] = torch.where(cb < 1e-30, 0.0, cb)
                s["T"][b], s["dtS"][b], s["t"][b], s["att"][b], s["cyc"][b], s["new"][b] = T[i], -1.0, 0.0, 0.0, 0.0, 1.0
                s["again"][b] += 1
            keep = ~done & (s["again"] < 2)
            if not bool(keep.all()):
                s = {k: v[..., keep] for k, v in s.items()}
                kf, kb = kf[:, keep], kb[:, keep]
        return dict(T=out[0], p=out[1], massf=out[2], dt_chem=out[3])


def exact(case, seed):
    kind = case["kind"]
    if kind == "surrogate":
        W, b, nm = _network(case, seed)
        dev = torch.device("cuda" if torch.cuda.is_available() else "cpu")
        t = lambda a: torch.tensor(np.asarray(a, np.float64), device=dev)   # noqa: E731
        x = (t(_features(case, seed)) - t(nm["x_shift"])) / t(nm["x_scale"])
        for k, (w, c) in enumerate(zip(W, b)):
            x = x @ t(w).T + t(c)
            if k < len(W) - 1:
                x = 0.5 * x * (1 + torch.tanh(math.sqrt(2 / math.pi) * (x + 0.044715 * x ** 3)))
        return x * t(nm["y_scale"]) + t(nm["y_shift"])
    # the two-temperature reactor's plain form, and plain updates of many cells, take far longer than the others
    if kind == "air2t" or case["mech"] == "c2h2" or (kind in ("cells", "host") and case["n"] > EXACT_CELLS):
        return None
    if kind in ("blocks", "layer"):
        cells = case["nx"] * case["ny"] if kind == "layer" else sum(_sizes(case))
        if cells > 160000:
            return None
    m = _Plain(case["mech"])

    def one(T, p, Y, dt, dtc=None, T_frozen=0.0):
        T, p, Y = m.t(T), m.t(p), m.t(Y)
        rho, u = m.rho_u(p, T, Y)
        return m.update(rho, u, T, p, Y, m.t(dtc) if dtc is not None else torch.full_like(T, -1.0), dt, T_frozen)

    if kind == "source":
        T, p, Y = (m.t(v) for v in _host_cells(case, seed))
        rho, _ = m.rho_u(p, T, Y)
        parts = []
        for k in range(0, T.shape[0], 1 << 16):
            c = Y[:, k:k + (1 << 16)] * rho[k:k + (1 << 16)] / m.M[:, None]
            q, L = m.qL(c, *m.rates(T[k:k + (1 << 16)], c))
            parts.append((q - L) * m.M[:, None])
        return torch.cat(parts, 1)
    if kind == "blocks":
        raw = _grid(case, seed)
        got = [one(b["T"], b["p"], b["Y"], b["dt"]) for b in raw]
        return dict({k: torch.cat([g[k].reshape(-1) for g in got]) for k in ("T", "p", "massf", "dt_chem")}, status=None)
    T, p, Y = _host_cells(case, seed)
    layer = kind == "layer"
    got = one(T, p, Y, case["dt"], _layer_steps(len(T), seed) if layer else None, 300.0 if layer else 0.0)
    if kind == "state":
        return dict(T=got["T"][0], p=got["p"][0], massf=got["massf"][:, 0], dt_chem=got["dt_chem"][0])
    return dict(got, status=None)

"""Timed cases of the surface Green's-function path, through its public Python entry points.

A case solves (k, omega) points of seeded Hermitian tight-binding models in the surface-cell
form the library takes (Num_wann x Num_wann blocks over R vectors, Hartree).  Kinds:

  kpath   Model.surface_spectrum over a k list x omega list (surfstat: dos.dat of a k path)
  arc     Model.surface_spectrum at one omega, sums divided by pi (SurfaceDOSkk: an arc map)
  spin    Model.surface_spectrum_spin with the arc map's spin texture
  engine  Engine.run: points of several models of uneven Ndim, one broadening per point
  single  surfgreen_1985: one decimation with its full GLL / GRR / GB matrices

Host arrays in, host arrays out, as the library's callers have them.
"""
import math

import numpy as np
import torch

from wannier_tools_gb300 import api

EV = 1.0 / 27.211385                  # Hartree
PI_REF = 3.14159265358979             # the reference's literal (arc sums are divided by it)
TOL = float(np.float32(1e-16))        # the reference's convergence threshold and cap
ITERMAX = 100
FORMS = {"fp64": api.PREC_FP64, "mixed": api.PREC_MIXED}

# Num_wann and Np of the engine cases' models: the Ndim 16 / 40 / 112 / 264 batch, and the
# serving mix's Ndim 8 / 32 / 60 / 120 / 112 / 150
SETS = {
    "four": [(8, 2), (20, 2), (56, 2), (88, 3)],
    "six": [(8, 1), (16, 2), (30, 2), (40, 3), (56, 2), (75, 2)],
    "three": [(7, 1), (13, 3), (33, 2)],
    "five": [(2, 2), (9, 3), (24, 2), (31, 2), (45, 2)],
}


def listed():
    return [
        # one (k, omega) point of a small model: the latency of a call
        {"name": "point_n16_fp64", "kind": "kpath", "nw": 8, "np": 2, "nk": 1, "nomega": 1,
         "eta_ev": 1e-2, "rmax": 3, "form": "fp64"},
        # a two-band model on its k path x omega grid: tiny matrices, very many points
        {"name": "kpath_n4_fp64", "kind": "kpath", "nw": 2, "np": 2, "nk": 101, "nomega": 200,
         "eta_ev": 1e-2, "rmax": 1, "form": "fp64"},
        # the k-path spectrum at Ndim 40, in both forms
        {"name": "kpath_n40_fp64", "kind": "kpath", "nw": 20, "np": 2, "nk": 51, "nomega": 101,
         "eta_ev": 1e-2, "rmax": 3, "form": "fp64"},
        {"name": "kpath_n40_mixed", "kind": "kpath", "nw": 20, "np": 2, "nk": 51, "nomega": 101,
         "eta_ev": 1e-2, "rmax": 3, "form": "mixed"},
        # the Fermi-arc map of the Num_wann = 56 model, part of the plane, in both forms
        {"name": "arc_n112_fp64", "kind": "arc", "nw": 56, "np": 2, "nk": 304, "nomega": 1,
         "eta_ev": 4e-3, "rmax": 3, "form": "fp64"},
        {"name": "arc_n112_mixed", "kind": "arc", "nw": 56, "np": 2, "nk": 912, "nomega": 1,
         "eta_ev": 1e-3, "rmax": 3, "form": "mixed"},
        # spectra of large cells: Ndim 150 and 264 (surfstat's broadening for 500 omegas in 1 eV)
        {"name": "kpath_n150_fp64", "kind": "kpath", "nw": 75, "np": 2, "nk": 3, "nomega": 50,
         "eta_ev": 6e-3, "rmax": 3, "form": "fp64"},
        {"name": "kpath_n264_mixed", "kind": "kpath", "nw": 88, "np": 3, "nk": 3, "nomega": 50,
         "eta_ev": 1e-3, "rmax": 3, "form": "mixed"},
        # the spin texture of an arc map, Ndim 60
        {"name": "spin_n60_fp64", "kind": "spin", "nw": 30, "np": 2, "nk": 1001, "nomega": 1,
         "eta_ev": 6e-3, "rmax": 3, "form": "fp64"},
        # uneven batches of several models in one launch, as the request loop makes them
        {"name": "uneven4_mixed", "kind": "engine", "set": "four", "points": 301,
         "eta_ev": 1e-3, "rmax": 3, "form": "mixed"},
        {"name": "uneven6_fp64", "kind": "engine", "set": "six", "points": 250,
         "eta_ev": 4e-3, "rmax": 3, "form": "fp64"},
        # one decimation with its full matrices, as a caller that replaces surfgreen_1985 makes it
        {"name": "single_n112_fp64", "kind": "single", "nw": 56, "np": 2, "nk": 1, "nomega": 1,
         "eta_ev": 1e-2, "rmax": 3, "form": "fp64"},
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng):
    kind = rng.choice(["kpath", "kpath", "arc", "spin", "engine", "single"])
    form = "fp64" if kind == "single" else rng.choice(["fp64", "mixed"])
    eta = _log(rng, 4e-3, 3e-2) if form == "fp64" else _log(rng, 1e-3, 2e-2)
    case = {"kind": kind, "eta_ev": eta, "rmax": rng.choice([1, 2, 3]), "form": form}
    if kind == "engine":
        case["set"] = rng.choice(sorted(SETS) if form == "mixed" else ["six", "three", "five"])
        case["points"] = round(_log(rng, 20, 290 if form == "mixed" else 230))
        return case
    n = _log(rng, 4, 264 if form == "mixed" else 150)
    case["np"] = rng.choice([1, 2, 2, 3])
    case["nw"] = max(2, round(n / case["np"]))
    if case["nw"] * case["np"] > (264 if form == "mixed" else 150):
        case["nw"] -= 1
    if kind == "spin":
        case["nw"] += case["nw"] % 2 * (1 if case["nw"] < 40 else -1)
    ndim = case["nw"] * case["np"]
    # no more work than the largest listed case of the form
    most = min(20000.0, max(1.0, (900.0 if form == "mixed" else 280.0) * (112.0 / ndim) ** 3))
    if ndim > 112:
        most = min(most, 150.0)
    points = 1 if kind == "single" else max(1, round(_log(rng, min(4.0, most), most)))
    if kind == "kpath":
        case["nk"] = max(1, round(math.sqrt(points) * rng.uniform(0.3, 1.0)))
        case["nomega"] = max(1, points // case["nk"])
    else:
        case["nk"], case["nomega"] = points, 1
    return case


def _model(nw, np_, rmax, seed):
    """Hermitian H(R) over R in [-rmax, rmax]^3, decaying with |R| (the decay length 1.2 cells,
    0.5 eV on-cell width, on-site energies in [-1, 1] eV): (irvec, hmnr[R, i, j])."""
    rng = np.random.default_rng(seed)
    g = np.arange(-rmax, rmax + 1)
    r3, r2, r1 = np.meshgrid(g, g, g, indexing="ij")
    irvec = np.stack([r1.ravel(), r2.ravel(), r3.ravel()], 1).astype(np.int32)
    a = rng.standard_normal((len(irvec), nw, nw, 2)).view(np.complex128)[..., 0]
    a *= (0.5 / math.sqrt(2.0) * np.exp(-np.linalg.norm(irvec, axis=1) / 1.2))[:, None, None]
    h = (a + a[::-1].conj().transpose(0, 2, 1)) / math.sqrt(2.0)     # H(-R) = H(R)^dagger
    i = np.arange(nw)
    h[len(irvec) // 2, i, i] = rng.uniform(-1.0, 1.0, nw)
    return irvec, h * EV


def _orbitals(nw):
    """Top and bottom lists: the whole layer, and every orbital but the first where there are more."""
    return list(range(1, nw + 1)), list(range(2 if nw > 2 else 1, nw + 1))


def _points(case, seed):
    """k list and omega list of the per-model kinds."""
    rng = np.random.default_rng(seed + 77)
    if case["kind"] == "kpath":
        a, b = rng.uniform(-0.5, 0.5, (2, 2))
        t = np.linspace(0.0, 1.0, case["nk"])[:, None]
        om = np.linspace(-1.0, 1.0, case["nomega"]) if case["nomega"] > 1 else rng.uniform(-1, 1, 1)
        return a + (b - a) * t, om * EV
    return rng.uniform(-0.5, 0.5, (case["nk"], 2)), rng.uniform(-0.2, 0.2, case["nomega"]) * EV


def _engine_points(case, seed):
    """model index, k, omega, eta of an engine case: the models' points interleaved."""
    rng = np.random.default_rng(seed + 78)
    n, m = case["points"], len(SETS[case["set"]])
    eta = np.exp(rng.uniform(np.log(case["eta_ev"]), np.log(10.0 * case["eta_ev"]), n))
    return (np.arange(n, dtype=np.int32) % m, rng.uniform(-0.5, 0.5, (n, 2)),
            rng.uniform(-1.0, 1.0, n) * EV, eta * EV)


def prepare(case, seed):
    form = FORMS[case["form"]]
    if case["kind"] == "engine":
        shapes = SETS[case["set"]]
        models = []
        for i, (nw, np_) in enumerate(shapes):
            irvec, h = _model(nw, np_, case["rmax"], seed * 16 + i)
            models.append(api.Model(h, irvec, None, np_))
        lists = [_orbitals(nw) for nw, _ in shapes]
        engine = api.Engine(models, [t for t, _ in lists], [b for _, b in lists], precision=form,
                            max_points=max(64, case["points"]))
        return {"kind": "engine", "engine": engine, "models": models,
                "points": _engine_points(case, seed)}
    irvec, h = _model(case["nw"], case["np"], case["rmax"], seed * 16)
    kpts, omega = _points(case, seed)
    state = {"kind": case["kind"], "kpts": kpts, "omega": omega, "eta": case["eta_ev"] * EV,
             "form": form, "lists": _orbitals(case["nw"])}
    if case["kind"] == "single":
        state["h00"], state["h01"] = _layers(irvec, h, case["np"], kpts)
        state["h00"], state["h01"] = state["h00"][0], state["h01"][0]
    else:
        state["model"] = api.Model(h, irvec, None, case["np"])
    return state


def run(state):
    kind = state["kind"]
    if kind == "engine":
        pm, k, om, eta = state["points"]
        return state["engine"].run(pm, k, om, eta)
    if kind == "single":
        g = api.surfgreen_1985(float(state["omega"][0]), state["h00"], state["h01"], state["eta"])
        return {"gll": g[0], "grr": g[1], "gb": g[2], "iters": g[3], "status": g[4]}
    top, bot = state["lists"]
    if kind == "spin":
        return state["model"].surface_spectrum_spin(state["kpts"], state["omega"], state["eta"],
                                                    top, bot, arc=True, precision=state["form"])
    return state["model"].surface_spectrum(state["kpts"], state["omega"], state["eta"], top, bot,
                                           divide_by_pi=kind == "arc", precision=state["form"])


def _solve_work(nw, np_, rmax, eta_ev):
    """(bytes, flops) of one solve: its decimation (six products and an inverse an iteration, three
    inverses at the end, 8 Ndim^3 each; iterations grow as log2 of 1 / eta), its three sums."""
    iters = 6.0 + max(0.0, math.log2(1.0 / eta_ev))
    return 24.0, (56.0 * iters + 24.0) * float(nw * np_) ** 3


def _model_bytes(nw, np_, rmax):
    return 16.0 * nw * nw * (2 * rmax + 1) ** 2 * min(2 * rmax + 1, 3 * np_ - 1)


def work(case):
    if case["kind"] == "engine":
        shapes = SETS[case["set"]]
        each = case["points"] / len(shapes)
        out = {"bytes": 40.0 * case["points"], "flops": 0.0}
        for nw, np_ in shapes:
            b, f = _solve_work(nw, np_, case["rmax"], 3.0 * case["eta_ev"])
            out["bytes"] += _model_bytes(nw, np_, case["rmax"]) + each * b
            out["flops"] += each * f
        return out
    n = case["nk"] * case["nomega"]
    b, f = _solve_work(case["nw"], case["np"], case["rmax"], case["eta_ev"])
    ndim = case["nw"] * case["np"]
    if case["kind"] == "single":
        return {"bytes": 5 * 16.0 * ndim * ndim, "flops": f}
    extra = 72.0 if case["kind"] == "spin" else 0.0
    return {"bytes": _model_bytes(case["nw"], case["np"], case["rmax"])
            + 16.0 * case["nk"] + 8.0 * case["nomega"] + n * (b + 5.0 + extra), "flops": n * f}


# --- the same path in plain 64-bit numpy / torch --------------------------------------------


def _layers(irvec, h, np_, kpts):
    """H00 and H01 of each k: (nk, Ndim, Ndim) arrays."""
    nw = h.shape[1]
    ph = np.exp(2j * PI_REF * (kpts @ irvec[:, :2].T.astype(float)))            # (nk, nR)
    lo, hi = -(np_ - 1), 2 * np_ - 1
    blocks = {}
    for r3 in range(lo, hi + 1):
        sel = np.flatnonzero(irvec[:, 2] == r3)
        blocks[r3] = (ph[:, sel] @ h[sel].reshape(-1, nw * nw)).reshape(-1, nw, nw)
    h00 = np.zeros((len(kpts), nw * np_, nw * np_), complex)
    h01 = np.zeros_like(h00)
    for i in range(np_):
        for j in range(np_):
            at = (slice(None), slice(i * nw, (i + 1) * nw), slice(j * nw, (j + 1) * nw))
            h00[at] = blocks[j - i]
            h01[at] = blocks[j - i + np_]
    return h00, h01


def _decimate(h00, h01, omega, eta):
    """GLL, GRR, GB of a batch; a point's matrices stop changing once it has converged."""
    n = h00.shape[-1]
    w = (omega + 1j * eta)[:, None, None] * torch.eye(n, dtype=h00.dtype, device=h00.device)
    e, es, et = h00.clone(), h00.clone(), h00.clone()
    al, be = h01.clone(), h01.mH.clone()
    live = torch.arange(len(h00), device=h00.device)
    for _ in range(ITERMAX):
        if not len(live):
            break
        a, b = al[live], be[live]
        g = torch.linalg.inv(w[live] - e[live])
        m1, m2 = a @ g, b @ g
        t = m1 @ b
        e[live] += t
        es[live] += t
        t = m2 @ a
        e[live] += t
        et[live] += t
        al[live], be[live] = m1 @ a, m2 @ b
        live = live[al[live].abs().sum((1, 2)) > TOL]
    return torch.linalg.inv(w - es), torch.linalg.inv(w - et), torch.linalg.inv(w - e)


def _sums(gll, grr, gb, nw, top, bot, spin):
    """The spectral sums of a batch (and the spin sums of an arc map)."""
    n = gll.shape[-1]
    it = torch.tensor(top, device=gll.device) - 1
    ib = torch.tensor(bot, device=gll.device) - 1 + n - nw
    diag = lambda g: g.diagonal(dim1=1, dim2=2)  # noqa: E731
    out = {"dos_l": -diag(gll)[:, it].imag.sum(1), "dos_r": -diag(grr)[:, ib].imag.sum(1),
           "dos_bulk": -diag(gb).imag.sum(1)}
    if spin:
        half = nw // 2
        for tag, g, io in (("l", gll, it), ("r", grr, ib)):
            up = (io % nw) < half
            part = torch.where(up, io + half, io - half)
            sgn = torch.where(up, 1.0, -1.0).to(torch.float64)
            gp = g[:, io, part]
            out["sx_" + tag] = -gp.imag.sum(1)
            out["sy_" + tag] = -(sgn * gp.real).sum(1)
            out["sz_" + tag] = -(sgn * diag(g)[:, io].imag).sum(1)
    return out


def _solve(h00, h01, omega, eta, nw, lists, spin):
    """_sums over a list of points, in batches that fit the device."""
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    n, parts = h00.shape[-1], []
    step = max(1, int(2e9 / (16.0 * n * n * 14)))
    for p in range(0, len(omega), step):
        s = slice(p, p + step)
        t = [torch.from_numpy(np.ascontiguousarray(x[s])).to(dev) for x in (h00, h01, omega, eta)]
        part = _sums(*_decimate(*t), nw, *lists, spin)
        parts.append({k: v.cpu().numpy() for k, v in part.items()})
    return {k: np.concatenate([q[k] for q in parts]) for k in parts[0]}


def exact(case, seed):
    if case["kind"] == "engine":
        pm, k, om, eta = _engine_points(case, seed)
        out = {name: np.empty(len(pm)) for name in ("dos_l", "dos_r", "dos_bulk")}
        for i, (nw, np_) in enumerate(SETS[case["set"]]):
            at = np.flatnonzero(pm == i)
            if len(at):
                h00, h01 = _layers(*_model(nw, np_, case["rmax"], seed * 16 + i), np_, k[at])
                got = _solve(h00, h01, om[at], eta[at], nw, _orbitals(nw), False)
                for name in out:
                    out[name][at] = got[name]
        return {**out, "iters": None, "status": None}
    kpts, omega = _points(case, seed)
    h00, h01 = _layers(*_model(case["nw"], case["np"], case["rmax"], seed * 16), case["np"], kpts)
    eta = case["eta_ev"] * EV
    if case["kind"] == "single":
        t = [torch.from_numpy(x) for x in (h00, h01, omega, np.full(1, eta))]
        g = [x[0].numpy() for x in _decimate(*t)]
        return {"gll": g[0], "grr": g[1], "gb": g[2], "iters": None, "status": None}
    nk, nw_ = len(kpts), len(omega)
    parts = []
    for p in range(0, nk, 64):                       # H00 / H01 repeat over a k's omegas
        q = slice(p, min(nk, p + 64))
        rep = lambda x: np.repeat(x[q], nw_, 0)      # noqa: E731
        m = q.stop - q.start
        parts.append(_solve(rep(h00), rep(h01), np.tile(omega, m), np.full(m * nw_, eta),
                            case["nw"], _orbitals(case["nw"]), case["kind"] == "spin"))
    scale = 1.0 if case["kind"] == "kpath" else 1.0 / PI_REF
    out = {k: scale * np.concatenate([x[k] for x in parts]).reshape(nk, nw_) for k in parts[0]}
    return {**out, "iters": None, "status": None}

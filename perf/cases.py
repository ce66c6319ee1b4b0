"""Workloads whose speed is measured: what users of the framework have it compute.

A case is a dict of plain values; ``prepare`` makes what a program holds before
the call (structures, form-factor tables, a plan), ``run`` is one pass through
the public entry points, ``exact`` the same outputs from plain torch in 64
bits. The sizes are those of the benchmark's workloads and of its serving
stream (500 to 50,000 atoms, 100 to 1,000 grid points up to q = 1/Angstrom),
with small and odd ones between them.

The kinds of call:

  solve       pripps_b200.debye.solve: host arrays in, the six profiles out
  model       the facade: Pripps.debye_model, then its intensity
  plan        a plan kept by the program, coordinates and result on the GPU
              (structures of one topology scored one after another)
  trajectory  one solve over a batch of frames with frame weights
  stream      debye.TrajectoryStream: frames pushed as a reader delivers them
  serve       serving.Server: a burst of requests submitted at once
  grid        excluded volume and hydration shell as grid dummies at their own
              positions (lattice sets)
  direct      direct.amplitudes: a periodic box of molecules at reciprocal-
              lattice vectors

The "fp32" form is a single-precision calculation (the library states 1e-5 for
it) whose sums come back in float64 arrays; a program that chooses it keeps
its profiles in single precision, and so do these cases. The "fp64" form's
profiles, and the direct transform's rows, stay in float64.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from pripps_b200 import _lib
from pripps_b200.debye import DebyeRequest, Pripps, TrajectoryStream, solve, union_request
from pripps_b200.direct import amplitudes
from pripps_b200.dummies import DummySet
from pripps_b200.formfactor import AtomKind, FormFactorMap, Gaussian
from pripps_b200.serving import Server
from pripps_b200.shard import ShardedPlan
from pripps_b200.solvent import ExcludedVolume, Hydration, SolventConfig
from pripps_b200.structure import Structure

# Four scatterer kinds in protein-like proportions, and water: Gaussian sums
# sum a exp(-b s^2) + c with s^2 = q^2 / (16 pi^2), a radius and a displaced
# volume.
KINDS = (
    ("C", 1.58, 16.44, ((2.31, 20.8439), (1.02, 10.2075), (1.5886, 0.5687), (0.865, 51.6512)),
     0.2156, 0.63),
    ("N", 0.84, 2.49, ((12.2126, 0.0057), (3.1322, 9.8933), (2.0125, 28.9975),
                       (1.1663, 0.5826)), -11.529, 0.17),
    ("O", 1.30, 9.13, ((3.0485, 13.2771), (2.2868, 5.7011), (1.5463, 0.3239),
                       (0.867, 32.9089)), 0.2508, 0.19),
    ("S", 1.68, 19.86, ((6.9053, 1.4679), (5.2034, 22.2151), (1.4379, 0.2536),
                        (1.5863, 56.172)), 0.8669, 0.01),
)
WATER = (1.93, 30.0, ((4.2, 11.3), (2.9, 7.4), (1.8, 0.9), (0.9, 40.0)), 0.2)
BULK = 0.334         # electrons per cubic Angstrom
PROBE, SHELL = 1.8, 3.0
VOLUME = 17.2        # cubic Angstrom per atom of a globule


def listed():
    return [
        # the smallest call: a peptide in vacuum, double precision
        dict(name="peptide_300_fp64", kind="solve", precision="fp64", n=300, nq=100, qmin=0.0,
             qmax=0.5, solvent="none", ratio=1.0),
        # an interactive user: one small protein through the facade
        dict(name="model_1500", kind="model", precision="fp32", n=1500, nq=200, qmin=0.0,
             qmax=0.5, solvent="shell", ratio=1.0),
        # an ordinary request of the serving stream, alone
        dict(name="request_3000", kind="solve", precision="fp32", n=3000, nq=300, qmin=0.0,
             qmax=0.6, solvent="shell", ratio=1.0),
        # a double-precision reference of a medium protein; odd sizes
        dict(name="protein_6001_fp64", kind="solve", precision="fp64", n=6001, nq=301, qmin=0.01,
             qmax=0.5, solvent="shell", ratio=1.3),
        # structures of 10,000 atoms scored on the GPU
        dict(name="sphere_10000", kind="plan", precision="fp32", n=10000, nq=500, qmin=0.0,
             qmax=0.5, solvent="shell", ratio=1.0),
        # a large complex: 100,000 atoms in an 80 x 40 x 40 Angstrom ellipsoid
        dict(name="ellipsoid_100000", kind="plan", precision="fp32", n=100000, nq=1000, qmin=0.0,
             qmax=1.0, solvent="shell", ratio=2.0, volume=5.36),
        # accessible-surface hydration: a weight of its own for each atom
        dict(name="sasa_20000", kind="solve", precision="fp32", n=20000, nq=512, qmin=0.0,
             qmax=1.0, solvent="sasa", ratio=2.0, volume=5.36),
        # an ensemble average over a batch of frames in memory
        dict(name="trajectory_64x5000", kind="trajectory", precision="fp32", n=5000, nq=300,
             qmin=0.0, qmax=0.5, solvent="none", ratio=1.0, frames=64),
        # the same from a reader, in pushes that do not fall on batch ends
        dict(name="stream_150x2003", kind="stream", precision="fp32", n=2003, nq=200, qmin=0.0,
             qmax=0.5, solvent="shell", ratio=1.2, frames=150, batch=32),
        # a server that meets a burst of requests of mixed sizes
        dict(name="serve_32", kind="serve", precision="fp32", n=20000, nq=600, qmin=0.0,
             qmax=0.8, solvent="shell", ratio=1.0, requests=32),
        # explicit solvent dummies on grids: cells of 1.5 Angstrom, water shell
        dict(name="grid_2500", kind="grid", precision="fp32", n=2500, nq=250, qmin=0.0, qmax=0.5,
             solvent="grid", ratio=1.0, spacing=1.5),
        # a simulation box: 64 molecules of 2,000 atoms, 1,300 Miller vectors
        dict(name="direct_64x2000", kind="direct", precision="fp64", n=2000, nq=100, qmin=0.0,
             qmax=0.0, solvent="none", ratio=1.0, copies=64, box=320.0),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case of the same kinds and ranges, never dearer than the
    100,000-atom solve."""
    kind = rng.choice(["solve", "solve", "model", "plan", "plan", "trajectory", "stream", "serve",
                       "grid", "direct"])
    c = dict(kind=kind, precision="fp32", n=_log(rng, 200, 20000), nq=_log(rng, 60, 1000),
             qmin=rng.choice([0.0, 0.0, 0.01, 0.05]), qmax=round(rng.uniform(0.3, 1.0), 3),
             solvent=rng.choice(["none", "shell", "shell", "sasa"]),
             ratio=round(rng.uniform(1.0, 2.5), 2))
    if kind in ("solve", "plan") and rng.random() < 0.4:
        c.update(precision="fp64", n=_log(rng, 100, 8000), nq=_log(rng, 60, 500))
    elif kind == "plan":
        c.update(n=_log(rng, 1000, 60000))
    elif kind == "model":
        c.update(n=_log(rng, 200, 6000), nq=_log(rng, 50, 400),
                 solvent=rng.choice(["none", "shell", "sasa"]))
    elif kind == "trajectory":
        c.update(n=_log(rng, 200, 5000), nq=_log(rng, 60, 400), frames=_log(rng, 3, 96))
    elif kind == "stream":
        c.update(n=_log(rng, 200, 3000), nq=_log(rng, 60, 300), frames=_log(rng, 20, 200),
                 batch=rng.choice([8, 16, 32, 64]))
    elif kind == "serve":
        c.update(n=_log(rng, 2000, 20000), nq=_log(rng, 200, 800), requests=_log(rng, 4, 40),
                 qmin=0.0,
                 solvent=rng.choice(["none", "shell"]))
    elif kind == "grid":
        c.update(n=_log(rng, 300, 3000), nq=_log(rng, 60, 300), solvent="grid",
                 qmax=round(rng.uniform(0.3, 0.6), 3), ratio=1.0,
                 spacing=round(rng.uniform(1.3, 2.0), 2))
    elif kind == "direct":
        c.update(precision="fp64", n=_log(rng, 50, 2000), nq=_log(rng, 6, 100), qmin=0.0,
                 qmax=0.0, solvent="none", ratio=1.0, copies=_log(rng, 1, 64),
                 box=round(rng.uniform(120.0, 320.0), 1))
    return c


# ------------------------------------------------------------------- inputs
def _gauss(ab, c, q):
    s2 = np.asarray(q) ** 2 / (16.0 * math.pi ** 2)
    return sum(a * np.exp(-b * s2) for a, b in ab) + c


def _tables(q):
    """Per kind: F(q), the excluded-volume Gaussian, and water's F(q)."""
    ff = np.stack([_gauss(k[3], k[4], q) for k in KINDS])
    ex = np.stack([BULK * k[2] * np.exp(-k[2] ** (2.0 / 3.0) / (16.0 * math.pi) * q ** 2)
                   for k in KINDS])
    return ff, ex, _gauss(WATER[2], WATER[3], q)


def _grid(case):
    k = np.arange(case["nq"], dtype=np.float64)
    return case["qmin"] + (case["qmax"] - case["qmin"]) * k / max(case["nq"] - 1, 1)


def _globule(n, ratio, volume, rng):
    """n atoms at the given volume each in a prolate ellipsoid (semi-axes
    ratio : 1 : 1): a cubic packing with random displacements, so that no two
    atoms are closer than about 0.6 of its spacing. Positions, kinds, and which atoms
    lie in the outer 3 Angstrom."""
    a = volume ** (1.0 / 3.0)
    b = (n * volume * 3.0 / (4.0 * math.pi * ratio)) ** (1.0 / 3.0)
    ext = [np.arange(-int(s / a) - 2, int(s / a) + 3) * a for s in (b * ratio, b, b)]
    p = np.stack(np.meshgrid(*ext, indexing="ij"), axis=-1).reshape(-1, 3)
    p = p + rng.uniform(-0.5 * a, 0.5 * a, 3)
    d = np.sqrt(np.sum((p / (b * ratio, b, b)) ** 2, axis=1))
    keep = np.argpartition(d, n - 1)[:n]
    p, d = p[keep], d[keep]
    p = p + rng.uniform(-0.2 * a, 0.2 * a, p.shape)
    order = rng.permutation(n)
    kinds = rng.choice(len(KINDS), size=n, p=[k[5] for k in KINDS])
    return p[order], kinds, (d[order] > 1.0 - SHELL / b)


def _shell_weights(kinds, outer, solvent, rng):
    if solvent == "none":
        return None
    full = np.array([4.0 * math.pi * (k[1] + PROBE) ** 2 * SHELL / 30.0 for k in KINDS])[kinds]
    w = np.where(outer & (rng.random(len(kinds)) < 0.35), full, 0.0)
    if solvent == "sasa":  # partly exposed: a value of its own for each atom
        w = w * rng.uniform(0.05, 1.0, len(kinds))
    return w


def _inputs(case, seed):
    """Structures, weights and frames from the seed alone, as numpy arrays."""
    rng = np.random.default_rng([seed, 17])
    kind = case["kind"]
    if kind == "serve":
        sizes = np.random.default_rng([case["requests"], case["n"], case["nq"]])
        out = []
        for _ in range(case["requests"]):  # the sizes belong to the case, the atoms to the seed
            n = int(math.exp(sizes.uniform(math.log(500), math.log(case["n"]))))
            nq = int(sizes.integers(100, case["nq"] + 1))
            one = dict(case, kind="solve", n=n, nq=nq,
                       qmax=case["qmax"] * float(sizes.uniform(0.4, 1.0)))
            out.append((one, _inputs(one, int(rng.integers(1 << 30)))))
        return out
    pos, kinds, outer = _globule(case["n"], case["ratio"], case.get("volume", VOLUME), rng)
    got = dict(pos=pos, kinds=kinds,
               weights=_shell_weights(kinds, outer, case["solvent"], rng)
               if kind != "grid" else None)
    if kind in ("trajectory", "stream"):
        f = case["frames"]
        got["frames"] = pos[None] + rng.normal(0.0, 0.5, (f,) + pos.shape)
        e = rng.exponential(1.0, f)
        got["frame_weights"] = e / e.sum()
    if kind == "grid":
        got["cells"], got["waters"] = _dummies(pos, kinds, case["spacing"])
    if kind == "direct":
        m, box = case["copies"], case["box"]
        turn = np.linalg.qr(rng.normal(size=(m, 3, 3)))[0]
        centres = rng.uniform(0.0, box, (m, 3))
        pts = np.einsum("mab,nb->mna", turn, pos - pos.mean(axis=0)) + centres[:, None]
        got["points"] = np.ascontiguousarray(pts.reshape(-1, 3))
        got["kinds"] = np.tile(kinds, m)
    return got


def _dummies(pos, kinds, spacing):
    """Grid points inside the atoms' spheres, and those 1.8 to 4.8 Angstrom
    off them on a water-sized grid: (points, (origin, spacing, extent)) each."""
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    at = torch.tensor(pos, device=dev)
    rad = torch.tensor([k[1] for k in KINDS], dtype=torch.float64, device=dev)[
        torch.tensor(kinds, device=dev)]
    out = []
    for h, lo, hi in ((spacing, -math.inf, 0.0), (3.10516, PROBE, PROBE + SHELL)):
        margin = float(rad.max()) + max(hi, 0.0) + h
        o = pos.min(axis=0) - margin
        ext = tuple(int(math.ceil((pos[:, a].max() + margin - o[a]) / h)) + 1 for a in range(3))
        axes = [torch.arange(ext[a], dtype=torch.float64, device=dev) * h + float(o[a])
                for a in range(3)]
        g = torch.stack(torch.meshgrid(*axes, indexing="ij"), dim=-1).reshape(-1, 3)
        d = torch.cat([(torch.cdist(p, at) - rad).amin(dim=1) for p in g.split(16384)])
        keep = (d > lo) & (d < hi)
        out.append((g[keep].cpu().numpy(), (tuple(float(v) for v in o), float(h), ext)))
    return out


def _request(case, got, frames=None):
    q = _grid(case)
    ff, ex, fw = _tables(q)
    w = got["weights"]
    return DebyeRequest(got["pos"] if frames is None else frames, got["kinds"], ff,
                        None if w is None else ex, w, None if w is None else fw, case["qmin"],
                        case["qmax"], case["nq"],
                        None if frames is None else got["frame_weights"], case["precision"])


def _formfactors():
    entries = [(AtomKind(k[0], 2.0 * k[1], k[2]), Gaussian((0.0, 6.0), list(k[3]), k[4]))
               for k in KINDS]
    return FormFactorMap.from_entries(
        entries + [(AtomKind("H2O", 2.0 * WATER[0], WATER[1]),
                    Gaussian((0.0, 6.0), list(WATER[2]), WATER[3]))])


class _Plan:
    """A plan the program keeps, given back with the state."""

    def __init__(self, req):
        self.plan = ShardedPlan(req, _lib.default_context(), 0, 1)

    def __del__(self):
        try:
            self.plan.close()
        except Exception:
            pass


def _miller(p_max):
    d = [(1, 0, 0), (0, 1, 0), (0, 0, 1), (1, 1, 0), (0, 1, 1), (1, 0, 1), (-1, 1, 0), (-1, 0, 1),
         (0, -1, 1), (1, 1, 1), (-1, 1, 1), (1, -1, 1), (1, 1, -1)]
    return np.array([[p * a for a in v] for v in d for p in range(1, p_max + 1)], dtype=np.int64)


def prepare(case, seed):
    kind = case["kind"]
    got = _inputs(case, seed)
    st = dict(kind=kind, single=case["precision"] == "fp32", case=case)
    if kind == "solve":
        st["request"] = _request(case, got)
    elif kind == "model":
        w = got["weights"]
        st["pripps"] = Pripps(_formfactors(), precision=case["precision"])
        st["structure"] = Structure(got["pos"], got["kinds"])
        st["solvent"] = None if w is None else SolventConfig(
            ExcludedVolume.fraser_foxs(1.0), Hydration.sasa(0.03, weights=w))
    elif kind == "plan":
        st["plan"] = _Plan(_request(case, got))
        st["xyz"] = torch.tensor(got["pos"], device="cuda")
    elif kind == "trajectory":
        st["request"] = _request(case, got, got["frames"])
    elif kind == "stream":
        st["request"] = _request(case, got)
        st["frames"], st["frame_weights"] = got["frames"], got["frame_weights"]
    elif kind == "serve":
        st["requests"] = [_request(one, g) for one, g in got]
        st["server"] = Server(_lib.default_context())
    elif kind == "grid":
        q = _grid(case)
        ff, _, _ = _tables(q)
        (cells, lc), (waters, lw) = got["cells"], got["waters"]
        v = case["spacing"] ** 3
        cell = Gaussian((0.0, 6.0), [(BULK * v, v ** (2.0 / 3.0) * 4.0 * math.pi)], 0.0)
        water = Gaussian((0.0, 6.0), list(WATER[2]), WATER[3])
        st["request"] = union_request(
            got["pos"], got["kinds"], ff, None, None, None,
            DummySet.weighted(cells, cell, np.ones(len(cells)), lc),
            DummySet.weighted(waters, water, np.ones(len(waters)), lw), q, case["qmin"],
            case["qmax"], case["precision"])
    elif kind == "direct":
        hkl = _miller(case["nq"])
        qn = 2.0 * math.pi / case["box"] * np.sqrt(np.sum(hkl.astype(float) ** 2, axis=1))
        st.update(xyz=got["points"], kinds=got["kinds"], ff=_tables(qn)[0], hkl=hkl,
                  box=np.full(3, case["box"]), molecules=case["copies"])
    return st


def run(state):
    kind = state["kind"]
    if kind in ("solve", "trajectory", "grid"):
        out = solve(state["request"])
    elif kind == "model":
        c = state["case"]
        m = state["pripps"].debye_model(state["structure"], c["qmin"], c["qmax"], c["nq"],
                                        state["solvent"])
        out = np.vstack([m.intensity(1.0, 0.03).total, m.terms])
    elif kind == "plan":
        out = state["plan"].plan.execute(state["xyz"])
    elif kind == "stream":
        s = TrajectoryStream(state["request"], state["case"]["batch"])
        for k in range(0, len(state["frames"]), 50):
            s.push(state["frames"][k:k + 50], state["frame_weights"][k:k + 50])
        out = s.finish()
    elif kind == "serve":
        srv = state["server"]
        tickets = [srv.submit(r) for r in state["requests"]]
        return [srv.wait(t).astype(np.float32) for t in tickets]
    else:
        return amplitudes(state["xyz"], state["kinds"], state["ff"], None, state["molecules"],
                          hkl=state["hkl"], box=state["box"])
    if state["single"]:
        return out.float() if isinstance(out, torch.Tensor) else out.astype(np.float32)
    return out


def work(case):
    """Inputs read once and outputs written once; every distance once (three
    subtractions, three multiply-adds' worth of squares and sums: 8), and for
    the direct transform a complex product and sum per vector and point. Grid
    dummies: about as many points as the globule's volume holds cells."""
    n, nq = case["n"], case["nq"]
    if case["kind"] == "serve":
        mean = (case["n"] - 500) / math.log(case["n"] / 500)
        mean_sq = (case["n"] ** 2 - 500 ** 2) / (2 * math.log(case["n"] / 500))
        return {"bytes": case["requests"] * (36.0 * mean + 7.5 * 8 * (100 + nq)),
                "flops": case["requests"] * mean_sq / 2 * 8.0}
    if case["kind"] == "direct":
        p, v = float(n * case["copies"]), 13.0 * nq
        return {"bytes": p * 28 + v * (12 + 32 + 32), "flops": p * v * 8}
    frames = case.get("frames", 1)
    if case["kind"] == "grid":
        n = int(n * (1.0 + 0.9 * VOLUME / case["spacing"] ** 3))
    tables = (4 if case["solvent"] == "none" else 9) * nq * 8.0
    per_atom = 4.0 + (0.0 if case["solvent"] == "none" else 8.0)
    return {"bytes": 24.0 * n * frames + per_atom * n + tables + 48.0 * nq,
            "flops": frames * (n * (n - 1) / 2.0) * 8.0}


# -------------------------------------------------------------------- exact
def _sums(xyz, rows, q):
    """[R, R, nq] sums over all i, j of rows_a[i] rows_b[j] sinc(q r_ij), in
    64 bits; rows is [R, classes, nq] by the points' class."""
    pts, cls, fac = xyz
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    x = torch.tensor(np.ascontiguousarray(pts), device=dev)
    x = x - x.mean(dim=0)
    n, nq = len(x), len(q)
    cls = torch.tensor(np.asarray(cls, dtype=np.int64), device=dev)
    rows = torch.tensor(rows, device=dev)
    fac = [torch.ones(n, dtype=torch.float64, device=dev) if f is None
           else torch.tensor(f, device=dev) for f in fac]
    out = torch.zeros((len(rows), len(rows), nq), dtype=torch.float64, device=dev)
    step = max(1, min(n, int(4e7 // n)))
    for i in range(0, n, step):
        d = x[i:i + step, None, :] - x[None, :, :]
        r = torch.sqrt((d * d).sum(dim=2))
        for k in range(nq):
            a = torch.stack([rows[m, cls, k] * fac[m] for m in range(len(rows))])
            s = torch.sinc(r * (float(q[k]) / math.pi))
            out[:, :, k] += a[:, i:i + step] @ (s @ a.T)
    return out.cpu().numpy()


def _six(pos, kinds, weights, q):
    ff, ex, fw = _tables(q)
    if weights is None:
        out = np.zeros((6, len(q)))
        out[0] = _sums((pos, kinds, [None]), ff[None], q)[0, 0]
        return out
    rows = np.stack([ff, ex, np.tile(fw, (len(KINDS), 1))])
    s = _sums((pos, kinds, [None, None, weights]), rows, q)
    return np.stack([s[0, 0], s[1, 1], s[2, 2], s[0, 1], s[0, 2], s[1, 2]])


def exact(case, seed):
    kind, n, nq = case["kind"], float(case["n"]), case["nq"]
    if kind == "serve":
        cost = case["requests"] * (n * n / (2 * math.log(n / 500))) * (100 + nq) / 2
    elif kind == "grid":
        cost = (n * (1.0 + 2.0 * VOLUME / case["spacing"] ** 3)) ** 2 * nq
    elif kind == "direct":
        cost = n * case["copies"] * 13 * nq * 4
    else:
        cost = n * n * nq * case.get("frames", 1)
    if cost > 7e11:
        return None
    got = _inputs(case, seed)
    if kind == "serve":
        return [_six(g["pos"], g["kinds"], g["weights"], _grid(one)) for one, g in got]
    if kind == "direct":
        return _direct_rows(case, got)
    q = _grid(case)
    if kind in ("trajectory", "stream"):
        w = got["frame_weights"]
        return sum(w[f] * _six(got["frames"][f], got["kinds"], got["weights"], q)
                   for f in range(len(w))) / w.sum()
    if kind == "grid":
        cells, waters = got["cells"][0], got["waters"][0]
        ff, _, fw = _tables(q)
        v = case["spacing"] ** 3
        cell = _gauss([(BULK * v, v ** (2.0 / 3.0) * 4.0 * math.pi)], 0.0, q)
        z = np.zeros_like(q)
        rows = np.stack([np.vstack([ff, z, z]), np.vstack([0 * ff, cell, z]),
                         np.vstack([0 * ff, z, fw])])
        m = len(KINDS)
        cls = np.concatenate([got["kinds"], np.full(len(cells), m), np.full(len(waters), m + 1)])
        s = _sums((np.vstack([got["pos"], cells, waters]), cls, [None] * 3), rows, q)
        return np.stack([s[0, 0], s[1, 1], s[2, 2], s[0, 1], s[0, 2], s[1, 2]])
    six = _six(got["pos"], got["kinds"], got["weights"], q)
    if kind == "model":
        c = 0.03 if got["weights"] is not None else 0.0
        v = 1.0 if got["weights"] is not None else 0.0
        total = (six[0] + v * six[1] + c * c * six[2] - 2 * v * six[3] + 2 * c * six[4]
                 - 2 * v * c * six[5])
        return np.vstack([total, six])
    return six


def _direct_rows(case, got):
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    hkl = torch.tensor(_miller(case["nq"]), dtype=torch.float64, device=dev)
    qv = 2.0 * math.pi * hkl / case["box"]
    ff = torch.tensor(_tables(torch.linalg.norm(qv, dim=1).cpu().numpy())[0], device=dev)
    x = torch.tensor(got["points"], device=dev)
    kinds = torch.tensor(got["kinds"], dtype=torch.int64, device=dev)
    m = case["copies"]
    mol = torch.zeros((m, len(qv)), dtype=torch.complex128, device=dev)
    for k, (p, c) in enumerate(zip(x.reshape(m, -1, 3), kinds.reshape(m, -1))):
        ph = p @ qv.T
        mol[k] = (ff[c] * torch.complex(torch.cos(ph), torch.sin(ph))).sum(dim=0)
    a = mol.sum(dim=0)
    return torch.stack([a.real, a.imag, a.abs() ** 2, (mol.abs() ** 2).sum(dim=0)],
                       dim=1).cpu().numpy()

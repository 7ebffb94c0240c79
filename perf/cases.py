"""Performance cases of the time-stepping paths, through the public Python entry points.

`listed()` names the cases, `draw(rng)` gives more of the same ranges,
`prepare` builds what a program holds before it steps (script and mesh files,
the prepared simulation or batch, advanced until the wave has entered the
domain), `run` is one pass, `work` the bytes and operations it cannot do
without, `exact` the same outputs in 64 bits from plain torch and numpy.

Three kinds of pass:

* a simulation or batch advances `steps` leapfrog steps and hands the field
  back: the whole state (`readout` "state": U, B, F) or, one streamed step
  later, the sample of every probe point (`readout` "probes").  This is how
  the reference's loop is driven from a host program that looks at the field
  now and then; a probe sample is recorded every step, as in the reference's
  own outputs (`SET period 0`);
* a batch does the same for many uneven meshes at once;
* `pcg` solves one sparse SPD system on the caller's CSR.

FP32 simulations return their values as 32-bit numbers (the library widens
them to double on the way out).
"""
from __future__ import annotations

import math
import os
import tempfile

import numpy as np
import torch

import tetfit_b200 as tb
from tetfit_b200 import cases as gen

MU0 = 4 * math.pi * 1e-7
EPS0 = 8.854187817e-12
C0 = 1 / math.sqrt(MU0 * EPS0)
_TMP = tempfile.TemporaryDirectory(prefix="tetfit_perf_")
_FILES: dict = {}


# ------------------------------------------------------------------- the cases
def listed():
    return [
        # the smallest Cartesian run: a parameter sweep's coarse cavity; launches count
        dict(name="fit_small_f64", kind="fit", nx=24, ny=24, nz=24, precision="fp64", spheres=0, steps=256),
        # the plain FP64 cavity the reference is quoted on
        dict(name="fit_cavity64_f64", kind="fit", nx=64, ny=64, nz=64, precision="fp64", spheres=0, steps=256),
        # an ordinary lossy scene with ragged sides in FP32
        dict(name="fit_ragged_f32", kind="fit", nx=43, ny=31, nz=47, precision="fp32", spheres=12, steps=128),
        # ten million cells in FP64, ragged, lossy spheres
        dict(name="fit_wide_f64", kind="fit", nx=261, ny=187, nz=214, precision="fp64", spheres=40, steps=16),
        # the large FP32 scene with 200 lossy spheres: beyond L2
        dict(name="fit_large_f32", kind="fit", nx=256, ny=256, nz=256, precision="fp32", spheres=200, steps=16),
        # the explicit method on the jittered 24^3 Kuhn box
        dict(name="dga24_f64", kind="tet", method="dga", n=24, precision="fp64", material="uniform", warm="previous",
             steps=64, readout="state"),
        # a larger two-material box, explicit, FP32
        dict(name="dga36_f32", kind="tet", method="dga", n=36, precision="fp32", material="split", warm="previous",
             steps=48, readout="probes"),
        # the smallest implicit-mass run: a CG of a few thousand unknowns every step, latency bound
        dict(name="gfdtd9_f64", kind="tet", method="gfdtd", n=9, precision="fp64", material="split", warm="previous",
             steps=48, readout="state"),
        # the implicit-mass method as the reference runs it (FP64, previous solution as guess)
        dict(name="gfdtd24_f64", kind="tet", method="gfdtd", n=24, precision="fp64", material="uniform",
             warm="previous", steps=16, readout="state"),
        # a heterogeneous box with the extrapolated guess, FP32
        dict(name="gfdtd40_f32", kind="tet", method="gfdtd", n=40, precision="fp32", material="grf",
             warm="extrapolate", steps=16, readout="probes"),
        # many uneven members in one group with the learned guess, FP32
        dict(name="batch16_learned_f32", kind="batch", count=16, n_lo=8, n_hi=36, precision="fp32", warm="learned",
             steps=16),
        # a caller's own SPD system on the standalone solver
        dict(name="pcg_grid", kind="pcg", nx=61, ny=50, nz=43, contrast=2.0, tol=1e-9),
    ]


def draw(rng):
    kind = rng.choice(["fit", "fit", "fit", "tet", "tet", "tet", "batch", "pcg"])
    log = lambda a, b: int(round(math.exp(rng.uniform(math.log(a), math.log(b)))))
    precision = rng.choice(["fp64", "fp32"])
    if kind == "fit":
        # between the two ranges the library estimates the time step of a Cartesian grid on the host for many seconds
        lo, hi, top = (16, 64, 8e4) if rng.random() < 0.5 else (150, 330, 1.65e7)
        while True:
            nx, ny, nz = (log(lo, hi) for _ in range(3))
            if (8e3 if lo == 16 else 1.02e7) <= nx * ny * nz <= top:
                break
        return dict(kind=kind, nx=nx, ny=ny, nz=nz, precision=precision, spheres=rng.choice([0, 5, 40, 150]),
                    steps=rng.choice([64, 100, 192, 256]) if lo == 16 else rng.choice([12, 16]))
    if kind == "tet":
        method = rng.choice(["dga", "gfdtd", "gfdtd", "fem"])
        n = log(7, 36 if method == "dga" else (40 if precision == "fp32" else 28))
        warm = "previous" if method == "dga" else rng.choice(["previous", "extrapolate"])
        return dict(kind=kind, method=method, n=n, precision=precision,
                    material=rng.choice(["uniform", "split", "grf"]), warm=warm,
                    steps=rng.choice([32, 48, 64]) if method == "dga" or n < 14 else rng.choice([12, 16, 24]),
                    readout="state" if n < 26 else "probes")
    if kind == "batch":
        lo = rng.randint(7, 12)
        return dict(kind=kind, count=rng.randint(3, 14), n_lo=lo, n_hi=rng.randint(lo + 4, 32), precision=precision,
                    warm=rng.choice(["previous", "extrapolate", "learned"]), steps=rng.choice([12, 16]))
    n = rng.uniform(math.log(3e3), math.log(1.3e5))
    nx = rng.randint(11, 60)
    ny = max(5, int(math.sqrt(math.exp(n) / nx)) + rng.randint(-3, 3))
    return dict(kind=kind, nx=nx, ny=ny, nz=max(5, int(math.exp(n) / nx / ny)),
                contrast=rng.choice([0.5, 1.0, 2.0]), tol=rng.choice([1e-8, 1e-9, 1e-10]))


# ------------------------------------------------------------- scripts and files
# probe points as fractions of the box, off the planes of any regular mesh
_GRID = ((0.131, 0.173, 0.9), (0.317, 0.411, 0.8), (0.0713, 0.0507, 0.95))


def _probe_axis(a, extent):
    lo, st, hi = (float(np.float32(v * extent)) for v in _GRID[a])
    out, v = [], lo
    while v <= hi:
        out.append(v)
        v += st
    return out


def _probe_points(extent):
    X, Y, Z = (_probe_axis(a, extent[a]) for a in range(3))
    return np.array([(x, y, z) for z in Z for y in Y for x in X])


def _source(seed):
    r = np.random.default_rng([seed, 11])
    return float(r.uniform(1.5e8, 3.5e8)), float(r.uniform(0.5, 2.0))


def _tail(extent, freq, amp, pec=(2, 3, 4, 5, 6)):
    """bc, source and output blocks shared by every script."""
    L = ["DEFINE bc 1"] + [f"   SET surface {s}" for s in pec] + ["   SET type pec", "END bc 1"]
    L += gen.source_lines(gen.FitCase(frequency=freq, amplitude=amp))
    L += ["DEFINE output 1", "   SET name out", "   SET mode probepoint"]
    for a, ax in enumerate("xyz"):
        L += ["   SET %sgrid {%r, %r, %r}" % ((ax,) + tuple(float(np.float32(v * extent[a])) for v in _GRID[a]))]
    return L + ["   SET grid on", "   SET period 0", "END output 1"]


def _write(path, lines):
    with open(path, "w") as f:
        f.write("\n".join(lines) + "\n")
    return path


def _fit_scene(case, seed):
    n = (case["nx"], case["ny"], case["nz"])
    h = 2.0 ** -math.ceil(math.log2(max(n)))  # exact in binary: cell counts come out as asked
    ext = tuple(v * h for v in n)
    r = np.random.default_rng([seed, 7])
    sph = []  # clear of the source wall z = 0
    for _ in range(case["spheres"]):
        rad = float(r.uniform(0.02, 0.1) * min(ext))
        centre = tuple(float(r.uniform(lo, e)) for lo, e in zip((0.0, 0.0, rad + 2 * h), ext))
        sph.append((centre, rad, float(r.uniform(1, 10)), float(10 ** r.uniform(-4, 0))))
    return n, h, ext, sph, 0.95 * 0.98 * h / (C0 * math.sqrt(3.0))


def _fit_script(case, seed, steps):
    n, h, ext, sph, dt = _fit_scene(case, seed)
    base = os.path.join(_TMP.name, "fit_%d_%d_%d_%d_%d" % (n + (len(sph), seed)))
    ns = len(sph)
    L = []
    for i, (c, rad, _, _) in enumerate(sph):
        L += [f"DEFINE solid {i + 1}", f"   SET material {i + 1}", "   SET type sphere",
              "   SET center {%r,%r,%r}" % c, f"   SET radius {rad!r}", f"END solid {i + 1}"]
    L += [f"DEFINE solid {ns + 1}", f"   SET material {ns + 1}", "   SET type box", "   SET corner {0,0,0}",
          "   SET size {%r,%r,%r}" % ext, f"END solid {ns + 1}"]
    _write(base + "_solids.txt", L)
    L = ["DEFINE mesh 1", "   SET type cartesian"]
    L += ["   SET %sgrid {0,%r,%r}" % (ax, h, e) for ax, e in zip("xyz", ext)]
    L += [f"   SET file {os.path.basename(base)}_solids.txt", "   SET name scene", "END mesh 1"]
    for i, (_, _, e, s) in enumerate(sph + [(0, 0, 1.0, 0.0)]):
        L += [f"DEFINE material {i + 1}", f"   SET epsilon {e!r}", "   SET mu 1", f"   SET sigma {s!r}",
              f"END material {i + 1}"]
    L += _tail(ext, *_source(seed))
    L += ["DEFINE simulation 1", "   SET method fdtd", "   SET mesh 1", "   SET source 1",
          f"   SET duration {(steps - 1) * dt!r}", f"   SET step {dt!r}", "   SET courant 0.98", "   SET output 1",
          "END simulation 1"]
    return _write(base + ".fdtd", L)


def _tet_materials(case, seed):
    """(centroids -> labels, {label: eps_r}): the mesh file holds the labels, the seed the permittivities."""
    r = np.random.default_rng([seed, 5])
    if case["material"] == "grf":
        hi = float(r.uniform(8, 12))
        field, table, _ = gen.grf_materials(hi=12.0)
        return field, {q: 1 + (e - 1) * (hi - 1) / 11 for q, e in table.items()}
    if case["material"] == "split":
        return (lambda c: np.where(c[:, 0] < 0.5, 1, 2)), {q + 1: float(v) for q, v in enumerate(r.uniform(1, 4, 2))}
    return (lambda c: np.ones(len(c), dtype=int)), {1: 1.0}


def _mesh(n, mesh_seed, material, field):
    """A jittered Kuhn box and its netgen file, written once per process."""
    key = (n, mesh_seed, material)
    if key not in _FILES:
        geo = gen.kuhn_mesh(n, 0.15, mesh_seed, field)
        path = os.path.join(_TMP.name, "mesh_%d_%d_%s.mesh" % key)
        _FILES[key] = (gen.write_netgen(path, *geo), geo)
    return _FILES[key]


def _tet_dt(method, n):
    return (0.15 if method == "fem" else 0.25) / n / C0


def _tet_script(case, seed, steps, mesh_seed=77):
    field, eps = _tet_materials(case, seed)
    path, _ = _mesh(case["n"], mesh_seed, case["material"], field)
    dt = _tet_dt(case["method"], case["n"])
    L = ["DEFINE mesh 1", "   SET type tetrahedral", "   SET mesher netgen", f"   SET file {os.path.basename(path)}",
         "   SET name box", "   SET scalefactor 1", "END mesh 1"]
    for m, e in eps.items():
        L += [f"DEFINE material {m}", f"   SET epsilon {float(e)!r}", "   SET mu 1", "   SET sigma 0",
              f"END material {m}"]
    L += _tail((1.0, 1.0, 1.0), *_source(seed))
    L += ["DEFINE simulation 1", f"   SET method {case['method']}", "   SET solver cg", "   SET tolerance 1e-8",
          "   SET mesh 1", "   SET source 1", f"   SET duration {(steps + 0.5) * dt!r}", f"   SET step {dt!r}",
          "   SET courant 0.98", "   SET output 1", "END simulation 1"]
    return _write(os.path.join(_TMP.name, "tet_%s_%d_%s_%d_%d.fdtd" % (case["method"], case["n"], case["material"],
                                                                     mesh_seed, seed)), L)


def _members(case, seed):
    """The members of a batch: sizes and meshes of the case, materials and sources of the seed."""
    r = np.random.default_rng([case["count"], case["n_lo"], case["n_hi"]])
    sizes = [case["n_lo"], case["n_hi"]] + [int(v) for v in r.integers(case["n_lo"], case["n_hi"] + 1,
                                                                        case["count"] - 2)]
    return [(dict(method="gfdtd", n=n, material="split"), 1000 * seed + i, 500 + i) for i, n in enumerate(sizes)]


# ------------------------------------------------------------------ preparation
def _counts(n):
    return 7 * n ** 3 + 9 * n ** 2 + 3 * n, 12 * n ** 3 + 6 * n ** 2  # edges, faces of the Kuhn box


def _warm(case):
    """Steps before the first pass: the wave has entered the domain; a learned guess has been trained."""
    if case["kind"] == "fit":
        return 32 + 3 * max(case["nx"], case["ny"], case["nz"]) // 2
    if case["kind"] == "batch":
        return 100
    return 24 + 4 * case["n"]


_LEARN = 60  # steps the network is trained on


def _total_steps(case):
    """Loop length of the script: seconds of stepping, within a few GB of probe samples."""
    w = work(case)["bytes"] / (case["steps"] + 1)
    probes = 180 * (case["count"] if case["kind"] == "batch" else 1)
    return int(min(6.0 / max(3.5e-6, w / 12e12), 6e9 / (48 * probes))) + _warm(case) + 1000


def prepare(case, seed):
    if case["kind"] == "pcg":
        ptr, col, val, b = _pcg_system(case, seed)
        dev = torch.device("cuda:0")
        return dict(kind="pcg", ptr=torch.from_numpy(ptr).to(dev), col=torch.from_numpy(col).to(dev),
                    val=torch.from_numpy(val).to(dev), b=torch.from_numpy(b).to(dev), tol=case["tol"])
    total = _total_steps(case)
    opts = dict(precision=case["precision"], device=0)
    if case["kind"] == "fit":
        sim = tb.Discretization(_fit_script(case, seed, total))
        probes = sim.prepare(1, **opts)["n_probes"]
    elif case["kind"] == "tet":
        sim = tb.Discretization(_tet_script(case, seed, total))
        if case["method"] != "dga":
            opts.update(warm_start=case["warm"], cg_criterion="reference" if case["warm"] == "previous" else "rhs")
        probes = sim.prepare(1, **opts)["n_probes"]
    else:
        opts.update(warm_start=case["warm"], cg_criterion="rhs", learn_steps=_LEARN)
        sim = tb.Batch([(_tet_script(c, s, total, m), 1) for c, s, m in _members(case, seed)], **opts)
        probes = sum(sim.info(m)["n_probes"] for m in range(sim.size))
    sim.step(_warm(case))
    return dict(kind=case["kind"], sim=sim, steps=case["steps"], readout=case.get("readout", "probes"),
                out=np.zeros((probes, 6)), dtype=np.float32 if case["precision"] == "fp32" else np.float64)


def run(state):
    if state["kind"] == "pcg":
        x = torch.zeros_like(state["b"])
        rc, iterations, _ = tb.pcg_solve(state["ptr"], state["col"], state["val"], state["b"], x, tol=state["tol"],
                                         maxiter=2000, criterion=1)
        if rc != tb.TF_OK:
            raise RuntimeError(tb.last_thread_error())
        return {"x": x, "iterations": iterations}
    sim = state["sim"]
    if sim.step(state["steps"]) != state["steps"]:
        raise RuntimeError("the simulation has reached its duration")
    if state["readout"] == "state":
        return {k: v.astype(state["dtype"], copy=False) for k, v in zip("UBF", sim.state())}
    if sim.step_io(None, state["out"]) != 1:
        raise RuntimeError("the simulation has reached its duration")
    return state["out"].astype(state["dtype"])


# ------------------------------------------------------------------------- work
_ITER = {"previous": 20, "extrapolate": 11, "learned": 10}  # CG iterations a step, as measured on such scenes


def _tet_work(case, n, warm):
    E, F = _counts(n)
    s = 4 if case["precision"] == "fp32" else 8
    method = case.get("method", "gfdtd")
    nnz_n = F + 72 * n ** 3
    nnz_e = E + 6 * F + (36 * n ** 3 if method == "fem" else 0)
    curl = 12 * F
    if method == "dga":  # curls, N and the node-star inverses once, the fields in and out
        nnz_h = 190 * n ** 3
        return 2 * curl + (nnz_n + nnz_h) * (4 + s) + s * (2 * E + 4 * F), 2 * (nnz_n + nnz_h) + 12 * F
    it = _ITER[warm]
    step = 2 * curl + nnz_n * (4 + s) + nnz_e * (4 + s) + s * (4 * E + 4 * F)
    return step + it * (nnz_e * (4 + s) + 9 * s * E), 2 * (nnz_n + nnz_e) + 12 * F + it * (2 * nnz_e + 12 * E)


def work(case):
    """Per step: every operator entry once and every field value in and out once (a field must be read and written
    each half step); per CG iteration the matrix and the iteration's vectors once."""
    if case["kind"] == "pcg":
        n = case["nx"] * case["ny"] * case["nz"]
        it = 110
        return {"bytes": it * (7 * 12 + 9 * 8) * n, "flops": it * 26 * n}
    k = case["steps"] + (case.get("readout") != "state")
    if case["kind"] == "fit":
        cells = case["nx"] * case["ny"] * case["nz"]
        s = 4 if case["precision"] == "fp32" else 8
        return {"bytes": k * 6 * 3 * cells * s, "flops": k * 45 * cells}
    if case["kind"] == "tet":
        b, f = _tet_work(case, case["n"], case["warm"])
    else:
        parts = [_tet_work(case, c["n"], case["warm"]) for c, _, _ in _members(case, 0)]
        b, f = (sum(p[q] for p in parts) for q in range(2))
    return {"bytes": k * b, "flops": k * f}


# ------------------------------------------------ the same outputs in 64 bits
def _device():
    return torch.device("cuda:0" if torch.cuda.is_available() else "cpu")


def _carrier(freq, amp, t):
    return amp * math.sin(2 * math.pi * freq * t) if t >= 0 else 0.0


def exact(case, seed):
    if case["kind"] == "pcg":
        return {"x": _exact_pcg(case, seed), "iterations": None}
    if case["kind"] == "fit":
        return _exact_fit(case, seed)
    if case["kind"] == "tet":
        return _exact_tets(case, [(case, seed, 77)])
    return _exact_tets(case, _members(case, seed))


def _exact_fit(case, seed):
    dev = _device()
    (nx, ny, nz), h, ext, sph, dt = _fit_scene(case, seed)
    freq, amp = _source(seed)
    f64 = dict(dtype=torch.float64, device=dev)
    ax = [(torch.arange(m, **f64) + 0.5) * h for m in (nz, ny, nx)]
    Z, Y, X = ax[0][:, None, None], ax[1][None, :, None], ax[2][None, None, :]
    eps = torch.full((nz, ny, nx), EPS0, **f64)
    sig = torch.zeros((nz, ny, nx), **f64)
    for (cx, cy, cz), rad, e, s in reversed(sph):  # the first solid in the file wins
        inside = (X - cx) ** 2 + (Y - cy) ** 2 + (Z - cz) ** 2 <= rad ** 2
        eps[inside] = EPS0 * e
        sig[inside] = s
    area, quarter = h * h, h * h / 4
    pad = lambda a: torch.nn.functional.pad(a, (1, 1, 1, 1, 1, 1))

    def edge(a, q):  # sum over the cells around each edge of axis q (0 x, 1 y, 2 z), array index [k, j, i]
        p = pad(a * quarter)
        for d in (0, 1, 2):
            if d != 2 - q:
                p = p.narrow(d, 0, p.shape[d] - 1) + p.narrow(d, 1, p.shape[d] - 1)
            else:
                p = p.narrow(d, 1, p.shape[d] - 2)
        return p

    coef = []
    for q in range(3):
        e, s = edge(eps, q), edge(sig, q)
        coef.append((h / (e + 0.5 * dt * s), (e - 0.5 * dt * s) / h))
    # mask: edges on the PEC walls (x, y walls and the top) are held at zero; the z = 0 wall carries the source
    mask = []
    for q in range(3):
        m = torch.ones_like(coef[q][0])
        for d, first in ((2, True), (1, True), (0, False)):
            if d != 2 - q:
                m.narrow(d, m.shape[d] - 1, 1).zero_()
                if first:
                    m.narrow(d, 0, 1).zero_()
        mask.append(m)
    mh = [c[0] * m for c, m in zip(coef, mask)]
    mq = [c[1] for c in coef]
    # faces lie between two half cells of mu0 (one on the boundary): M_nu = (sum of half lengths / mu) / area
    half = h / 2 / MU0
    nu = []
    for q in range(3):
        shape = [nz, ny, nx]
        shape[2 - q] += 1
        v = torch.full(shape, 2 * half / area, **f64)
        for at in (0, shape[2 - q] - 1):
            v.narrow(2 - q, at, 1).fill_(half / area)
        nu.append(v)
    U = [torch.zeros_like(m) for m in mask]
    F = [torch.zeros_like(v) for v in nu]

    def below(a, d):  # a[index - 1] along d with zero outside, one longer than a
        z = torch.zeros_like(a.narrow(d, 0, 1))
        return torch.cat([z, a], d) - torch.cat([a, z], d)  # lower neighbour minus own

    # source: the dual edge of a y edge on z = 0 points along -x
    xs = torch.arange(nx + 1, **f64) * h
    prof = -h * torch.sin(2 * math.pi * 0.5 * xs)
    count = _warm(case) + case["steps"] + 1
    B = None
    for i in range(count):
        Fx, Fy, Fz = F
        # C^T F per edge, as in the curl of the magnetomotive force
        cx = below(Fy, 0) - below(Fz, 1)
        cy = -(below(Fx, 0) - below(Fz, 2))
        cz = below(Fx, 1) - below(Fy, 2)
        cy[0] += _carrier(freq, amp, i * dt - 0.5 * dt) * prof[None, :]
        for q, c in enumerate((cx, cy, cz)):
            U[q] = mh[q] * (mq[q] * U[q] + dt * c)
        Ux, Uy, Uz = U
        curl = (Uy[:-1] - Uy[1:] + Uz[:, 1:] - Uz[:, :-1], Ux[1:] - Ux[:-1] + Uz[:, :, :-1] - Uz[:, :, 1:],
                Ux[:, :-1] - Ux[:, 1:] + Uy[:, :, 1:] - Uy[:, :, :-1])
        if i == count - 1:
            B = [F[q] / nu[q] - dt * curl[q] for q in range(3)]
        F = [nu[q] * (F[q] / nu[q] - dt * curl[q]) for q in range(3)]
    pts = _probe_points(ext)
    i, j, k = (torch.from_numpy(np.floor(pts[:, a] / h).astype(np.int64)).to(dev) for a in range(3))
    Ux, Uy, Uz = U
    vol = h ** 3
    E = [sum(Ux[k + a, j + b, i] for a in (0, 1) for b in (0, 1)) * quarter / vol,
         sum(Uy[k + a, j, i + b] for a in (0, 1) for b in (0, 1)) * quarter / vol,
         sum(Uz[k, j + a, i + b] for a in (0, 1) for b in (0, 1)) * quarter / vol]
    H = [(B[0][k, j, i] + B[0][k, j, i + 1]), (B[1][k, j, i] + B[1][k, j + 1, i]), (B[2][k, j, i] + B[2][k + 1, j, i])]
    H = [v * (0.5 * h) / MU0 / vol for v in H]
    return torch.stack(E + H, 1).cpu().numpy()


_EDGE = ((0, 1), (1, 2), (0, 2), (0, 3), (1, 3), (2, 3))   # local edges, and those at each node
_AT = ((0, 2, 3), (0, 1, 4), (1, 2, 5), (3, 4, 5))


class _Box:
    """One tetrahedral member in numpy: numbering, operators as (rows, columns, values), sources and probes."""

    def __init__(self, case, seed, mesh_seed):
        field, eps = _tet_materials(case, seed)
        _, (pts, tets, mats, tris, labels) = _mesh(case["n"], mesh_seed, case["material"], field)
        method, n = case["method"], len(pts)
        T = np.sort(tets, 1)
        order = np.lexsort((T[:, 3], T[:, 2], T[:, 1], T[:, 0]))
        T, mats = T[order], np.asarray(mats)[order]
        eps = EPS0 * np.vectorize(lambda m: eps[m])(mats)
        P = pts[T]
        V = np.einsum("ij,ij->i", P[:, 1] - P[:, 0], np.cross(P[:, 2] - P[:, 0], P[:, 3] - P[:, 0])) / 6
        tri = np.stack([T[:, [1, 2, 3]], T[:, [0, 2, 3]], T[:, [0, 1, 3]], T[:, [0, 1, 2]]], 1)  # opposite node 0..3
        key3 = lambda t: (t[..., 0].astype(np.int64) * n + t[..., 1]) * n + t[..., 2]
        fk, first, inv, cnt = np.unique(key3(tri).ravel(), return_index=True, return_inverse=True, return_counts=True)
        vtf = inv.reshape(-1, 4)
        faces = tri.reshape(-1, 3)[first]
        ends = np.stack([T[:, list(e)] for e in _EDGE], 1)
        ek, fe, inv = np.unique((ends[..., 0].astype(np.int64) * n + ends[..., 1]).ravel(), return_index=True,
                                return_inverse=True)
        vte = inv.reshape(-1, 6)
        edges = ends.reshape(-1, 2)[fe]
        eid = lambda a, b: np.searchsorted(ek, a.astype(np.int64) * n + b)
        fte = np.stack([eid(faces[:, 0], faces[:, 1]), eid(faces[:, 0], faces[:, 2]), eid(faces[:, 1], faces[:, 2])], 1)
        self.nE, self.nF = len(edges), len(faces)
        bf = np.searchsorted(fk, key3(np.sort(tris, 1)))
        pec = np.zeros(self.nE, bool)
        pec[fte[bf[labels != 1]]] = True
        self.free = np.flatnonzero(~pec)
        # source: dual edges on surface 1 (z = 0) of the free edges, oriented with the outward normal
        sf = bf[labels == 1]
        bar = pts[faces].mean(1)
        dual = np.zeros((self.nE, 3))
        pair = {}
        for f in np.sort(sf):
            for e in fte[f]:
                pair.setdefault(int(e), []).append(int(f))
        self.src = np.array([e for e, fs in sorted(pair.items()) if len(fs) == 2 and not pec[e]], dtype=np.int64)
        two = np.array([pair[int(e)] for e in self.src])
        d = bar[two[:, 1]] - bar[two[:, 0]]
        ev = pts[edges[self.src, 1]] - pts[edges[self.src, 0]]
        d *= np.where(np.einsum("ij,ij->i", np.cross(ev, [0.0, 0.0, -1.0]), d) >= 0, 1, -1)[:, None]
        mid = pts[edges[self.src]].mean(1)
        self.profile = d[:, 0] * np.sin(2 * math.pi * 0.5 * mid[:, 0])
        self.freq, self.amp = _source(seed)
        self.dt = _tet_dt(method, case["n"])
        r = np.repeat(np.arange(self.nF), 3)
        self.C = (r, fte.ravel(), np.tile([1.0, -1.0, 1.0], self.nF))
        # N: the inverse of each tet's magnetic mass from its dual area vectors
        eb = np.stack([P[:, list(e)].mean(1) for e in _EDGE], 1)
        fb = np.stack([P[:, [1, 2, 3]].mean(1), P[:, [0, 2, 3]].mean(1), P[:, [0, 1, 3]].mean(1),
                       P[:, [0, 1, 2]].mean(1)], 1)
        vb = P.mean(1)
        fpair = ((2, 3), (0, 3), (3, 1), (1, 2), (2, 0), (0, 1))
        g = np.stack([np.cross(vb - eb[:, q], fb[:, a] - fb[:, b]) for q, (a, b) in enumerate(fpair)], 1)
        g *= np.where(V < 0, -0.5, 0.5)[:, None, None]
        D = np.einsum("tax,tbx->tab", g, g) * (MU0 * 36 / np.abs(V))[:, None, None]
        M = np.empty((len(T), 4, 4))
        M[:, 0, 0] = D[:, 0, 0] + D[:, 2, 2] + D[:, 3, 3]
        M[:, 1, 1] = D[:, 0, 0] + D[:, 1, 1] + D[:, 4, 4]
        M[:, 2, 2] = D[:, 1, 1] + D[:, 2, 2] + D[:, 5, 5]
        M[:, 3, 3] = D[:, 3, 3] + D[:, 4, 4] + D[:, 5, 5]
        M[:, 0, 1] = -D[:, 1, 2] - D[:, 3, 4]
        M[:, 0, 2] = -D[:, 0, 1] + D[:, 3, 5]
        M[:, 0, 3] = D[:, 0, 4] + D[:, 2, 5]
        M[:, 1, 2] = -D[:, 0, 2] - D[:, 4, 5]
        M[:, 1, 3] = D[:, 0, 3] - D[:, 1, 5]
        M[:, 2, 3] = -D[:, 2, 3] - D[:, 1, 4]
        for a in range(4):
            for b in range(a):
                M[:, a, b] = M[:, b, a]
        self.N = (np.repeat(vtf, 4, 1).ravel(), np.tile(vtf, (1, 4)).ravel(), np.linalg.inv(M).ravel())
        lam = np.concatenate([P, np.ones((len(T), 4, 1))], 2)
        grad = np.linalg.inv(lam)  # [t, axis (3: constant), node]
        rows, cols, vals = [], [], []
        if method == "fem":
            # Whitney mass by the quadrature with weights 1/40 at the nodes and 9/40 at the face barycentres
            mass = np.zeros((len(T), 6, 6))
            for pos, wt in ((P, 1.0), (fb, 9.0)):
                for q in range(4):
                    l = np.einsum("tx,txn->tn", pos[:, q], grad[:, :3]) + grad[:, 3]
                    w = np.stack([l[:, a, None] * grad[:, :3, b] - l[:, b, None] * grad[:, :3, a] for a, b in _EDGE], 1)
                    mass += wt * np.einsum("tax,tbx->tab", w, w)
            mass *= (np.abs(V) * eps / 40)[:, None, None]
            rows, cols, vals = [np.repeat(vte, 6, 1).ravel()], [np.tile(vte, (1, 6)).ravel()], [mass.ravel()]
        elif method == "gfdtd":
            # the reference's node dual basis on the half edges that leave the node
            for k in range(4):
                a = eb[:, list(_AT[k])] - P[:, k, None]
                x = np.stack([np.cross(a[:, 1], a[:, 2]), np.cross(a[:, 2], a[:, 0]), np.cross(a[:, 0], a[:, 1])], 1)
                x /= np.einsum("ti,ti->t", a[:, 0], x[:, 0])[:, None, None]
                blk = np.einsum("tax,tbx->tab", x, x) * (np.abs(V) / 4 * eps)[:, None, None]
                e = vte[:, list(_AT[k])]
                rows.append(np.repeat(e, 3, 1).ravel())
                cols.append(np.tile(e, (1, 3)).ravel())
                vals.append(blk.ravel())
        else:
            # node stars: masked inverses of the star's mass
            star = np.concatenate([np.stack([edges[:, s], np.arange(self.nE)], 1) for s in (0, 1)])
            star = star[np.lexsort((star[:, 1], star[:, 0]))]
            start = np.searchsorted(star[:, 0], np.arange(n + 1))
            rank = np.arange(len(star)) - start[star[:, 0]]
            m = int(rank.max()) + 1
            slot = np.zeros((self.nE, 2), dtype=np.int64)
            slot[star[:, 1], (edges[star[:, 1], 1] == star[:, 0]).astype(int)] = rank
            S = np.zeros((n, m, m))
            pe = (P[:, 1] - P[:, 0], P[:, 2] - P[:, 1], P[:, 2] - P[:, 0], P[:, 3] - P[:, 0], P[:, 3] - P[:, 1])
            av = np.stack([np.cross(pe[1], pe[4]), np.cross(pe[2], pe[3]), np.cross(pe[0], pe[3]),
                           np.cross(pe[0], pe[2])], 1) * 0.5
            av *= np.array([1.0, -1.0, 1.0, -1.0])[None, :, None]
            fv = ((1, 2, 3), (0, 2, 3), (1, 0, 3), (0, 1, 2))
            sg = ((-1, -1, -1), (1, -1, -1), (1, 1, -1), (1, 1, 1))
            for k in range(4):
                w = av[:, list(fv[k])] * (np.array(sg[k])[None] * (2.0 / 3.0 / np.abs(V))[:, None])[..., None]
                blk = np.einsum("tax,tbx->tab", w, w) * (np.abs(V) / 4 * eps)[:, None, None]
                e = vte[:, list(_AT[k])]
                loc = slot[e, (edges[e, 1] == T[:, k, None]).astype(int)]
                np.add.at(S, (T[:, k, None, None], loc[:, :, None], loc[:, None, :]), blk)
            hole = np.ones((n, m), bool)
            ids = np.full((n, m), -1)
            ids[star[:, 0], rank] = star[:, 1]
            hole[star[:, 0], rank] = pec[star[:, 1]]
            S[hole[:, :, None] | hole[:, None, :]] = 0
            S[hole[:, :, None] & np.eye(m, dtype=bool)[None]] = EPS0  # masked rows stay apart
            Hs = torch.linalg.inv(torch.from_numpy(S).to(_device())).cpu().numpy()
            keep = ~(hole[:, :, None] | hole[:, None, :])
            rows = [np.broadcast_to(ids[:, :, None], S.shape)[keep]]
            cols = [np.broadcast_to(ids[:, None, :], S.shape)[keep]]
            vals = [Hs[keep]]
        self.E = (np.concatenate(rows), np.concatenate(cols), np.concatenate(vals))
        # probes: the tet that holds each point, E by Whitney functions, H from the face fluxes
        q = _probe_points((1.0, 1.0, 1.0))
        lo, hi = P.min(1), P.max(1)
        self.pE, self.pF, rE, rF = [], [], [], []
        for x in q:
            cand = np.flatnonzero(np.all((lo <= x) & (x <= hi), 1))
            l = np.einsum("x,txn->tn", x, grad[cand, :3]) + grad[cand, 3]
            best = int(np.argmax(l.min(1)))
            t, l = cand[best], l[best]
            if l.min() < -1e-9:
                continue
            G = grad[t, :3]
            rE.append(np.stack([l[a] * G[:, b] - l[b] * G[:, a] for a, b in _EDGE]))
            p = P[t]
            ab, bc, ac, ad, bd, cd = (p[j] - p[i] for i, j in _EDGE)
            w = np.stack([ab + ac + ad, ab - bc - bd, cd - ac - bc, ad + bd + cd])
            rF.append(w * (0.25 / MU0 / (3 * V[t])))
            self.pE.append(vte[t])
            self.pF.append(vtf[t])
        self.pE, self.pF, self.wE, self.wF = (np.array(v) for v in (self.pE, self.pF, rE, rF))


def _exact_tets(case, members):
    dev = _device()
    boxes = [_Box(c, s, m) for c, s, m in members]
    method = members[0][0]["method"]
    eo = np.cumsum([0] + [b.nE for b in boxes])
    fo = np.cumsum([0] + [b.nF for b in boxes])
    nE, nF = int(eo[-1]), int(fo[-1])
    t64 = lambda a: torch.from_numpy(np.ascontiguousarray(a, dtype=np.float64)).to(dev)
    idx = lambda a: torch.from_numpy(np.ascontiguousarray(a, dtype=np.int64)).to(dev)

    def sparse(parts, ro, co, shape):
        r = np.concatenate([p[0] + o for p, o in zip(parts, ro)])
        c = np.concatenate([p[1] + o for p, o in zip(parts, co)])
        v = np.concatenate([p[2] for p in parts])
        return torch.sparse_coo_tensor(torch.stack([idx(r), idx(c)]), t64(v), shape).coalesce().to_sparse_csr()

    C = sparse([b.C for b in boxes], fo, eo, (nF, nE))
    Ct = sparse([(b.C[1], b.C[0], b.C[2]) for b in boxes], eo, fo, (nE, nF))
    N = sparse([b.N for b in boxes], fo, fo, (nF, nF))
    E = sparse([b.E for b in boxes], eo, eo, (nE, nE))
    mul = lambda A, x: torch.mv(A, x)
    dt_e = t64(np.concatenate([np.full(b.nE, b.dt) for b in boxes]))
    dt_f = t64(np.concatenate([np.full(b.nF, b.dt) for b in boxes]))
    src = idx(np.concatenate([b.src + o for b, o in zip(boxes, eo)]))
    prof = [t64(b.profile) for b in boxes]
    free = torch.zeros(nE, dtype=torch.float64, device=dev)
    free[idx(np.concatenate([b.free + o for b, o in zip(boxes, eo)]))] = 1.0
    seg = idx(np.concatenate([np.full(b.nE, i) for i, b in enumerate(boxes)]))
    dot = lambda a, b: torch.zeros(len(boxes), dtype=torch.float64, device=dev).index_add_(0, seg, a * b)
    U, B, F = (t64(np.zeros(m)) for m in (nE, nF, nF))
    Uo, x, fb_old = U.clone(), U.clone(), t64(np.zeros(len(src)))
    if method != "dga":
        r, c = E.crow_indices(), E.col_indices()
        row = torch.repeat_interleave(torch.arange(nE, device=dev), r[1:] - r[:-1])
        diag = torch.zeros(nE, dtype=torch.float64, device=dev)
        diag[row[row == c]] = E.values()[row == c]
        pre = free / diag

    def solve(b, x):  # block-wise Jacobi-PCG far below the tolerance of the runs
        r = free * (b - mul(E, x))
        z = pre * r
        p, rz, bb = z.clone(), dot(r, z), dot(free * b, free * b)
        for it in range(400):
            q = free * mul(E, p)
            alpha = rz / dot(p, q).clamp_min(1e-300)
            a = alpha[seg]
            x = x + a * p
            r = r - a * q
            if it % 8 == 7 and bool((dot(r, r) <= 1e-26 * bb).all()):
                break
            z = pre * r
            new = dot(r, z)
            p = z + (new / rz.clamp_min(1e-300))[seg] * p
            rz = new
        return x

    sample = None
    last = _warm(case) + case["steps"] + (case.get("readout", "probes") != "state")
    for i in range(1, last + 1):
        fb = torch.cat([_carrier(b.freq, b.amp, i * b.dt - 0.5 * b.dt) * w for b, w in zip(boxes, prof)])
        if method == "dga":
            cf = mul(Ct, F)
            cf[src] += fb
            U = U + dt_e * mul(E, cf)
            cu = mul(C, U)
            B = B - dt_f * cu
            F = F - dt_f * mul(N, cu)
            sample = (U, B)
            continue
        cu = mul(C, U)
        B = B - dt_f * cu
        F = mul(N, cu if method == "fem" else B)
        sample = (U, B)
        cb = torch.zeros_like(U)
        if method == "fem":
            cb[src] = fb - fb_old
            rhs = mul(E, 2 * U - Uo) - dt_e ** 2 * mul(Ct, F) + dt_e * cb
        else:
            cb[src] = fb
            rhs = mul(E, U) + dt_e * mul(Ct, F) + dt_e * cb
        fb_old = fb
        new = solve(rhs, 2 * x - Uo if i > 2 else x)
        Uo, U, x = U, new * free, new
    if case.get("readout") == "state":
        return {"U": U.cpu().numpy(), "B": B.cpu().numpy(), "F": F.cpu().numpy()}
    U, B = (v.cpu().numpy() for v in sample)
    out = []
    for b, a, o in zip(boxes, eo, fo):
        out.append(np.concatenate([np.einsum("pq,pqx->px", U[b.pE + a], b.wE),
                                   np.einsum("pq,pqx->px", B[b.pF + o], b.wF)], 1))
    return np.concatenate(out)


def _pcg_system(case, seed):
    """A cell-centred diffusion operator on a grid, harmonic means of a log-normal coefficient plus an implicit time
    term, as CSR with sorted columns, and a smooth-plus-noise right-hand side."""
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    n = nx * ny * nz
    r = np.random.default_rng([seed, 3])
    k = np.exp(case["contrast"] * r.standard_normal((nz, ny, nx)))
    own = np.arange(n).reshape(nz, ny, nx)
    rows, cols, vals = [], [], []
    diag = 0.5 * np.exp(0.3 * r.standard_normal((nz, ny, nx)))
    for d in range(3):
        a = [slice(None)] * 3
        b = [slice(None)] * 3
        a[d], b[d] = slice(None, -1), slice(1, None)
        a, b = tuple(a), tuple(b)
        t = 2 * k[a] * k[b] / (k[a] + k[b])
        diag[a] += t
        diag[b] += t
        rows += [own[a].ravel(), own[b].ravel()]
        cols += [own[b].ravel(), own[a].ravel()]
        vals += [-t.ravel(), -t.ravel()]
    rows = np.concatenate(rows + [own.ravel()])
    cols = np.concatenate(cols + [own.ravel()])
    vals = np.concatenate(vals + [diag.ravel()])
    order = np.lexsort((cols, rows))
    ptr = np.zeros(n + 1, dtype=np.int64)
    ptr[1:] = np.cumsum(np.bincount(rows, minlength=n))
    z = np.arange(n) / n
    return ptr, cols[order].astype(np.int32), vals[order], np.sin(9 * z) + 0.1 * r.standard_normal(n)


def _exact_pcg(case, seed):
    dev = _device()
    ptr, col, val, b = (torch.from_numpy(np.ascontiguousarray(v)).to(dev) for v in _pcg_system(case, seed))
    n = len(b)
    A = torch.sparse_csr_tensor(ptr, col.long(), val, (n, n))
    row = torch.repeat_interleave(torch.arange(n, device=dev), ptr[1:] - ptr[:-1])
    diag = torch.zeros(n, dtype=torch.float64, device=dev)
    diag[row[row == col]] = val[row == col]
    x = torch.zeros_like(b)
    for _ in range(3):  # restarted on the true residual, down to rounding
        r = b - torch.mv(A, x)
        z = r / diag
        p, rz = z, torch.dot(r, z)
        stop = 1e-12 * torch.linalg.vector_norm(r)
        for it in range(3000):
            q = torch.mv(A, p)
            a = rz / torch.dot(p, q)
            x = x + a * p
            r = r - a * q
            if it % 16 == 15 and bool(torch.linalg.vector_norm(r) <= stop):
                break
            z = r / diag
            new = torch.dot(r, z)
            p = z + new / rz * p
            rz = new
    return x.cpu().numpy()

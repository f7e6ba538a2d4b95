"""What a user of this framework has it do, as cases that can be timed.

A case is one H-matrix (or a batch of them) of the point kernel 1 / (4 pi r),
built by HACApK's rules, resident on the GPU as a plan, and one call of the
public API on it: a single-vector product in each precision, a captured
product, a block of right-hand sides, a batch, a Krylov solve.

``prepare`` makes what a program holds before the call, ``run`` is the call,
``work`` what it cannot do without, ``exact`` its result in FP64 with numpy.
"""
import numpy as np
import torch

from hacapk_hmvm_b200 import Batch, HMatrix, Plan

GEOMETRIES = ("sphere", "cube", "plate")
# Bytes of a stored element.  Mixed plans: FP8 / FP16 / FP32 low-rank columns,
# FP32 dense and FP64 diagonal leaves, on average.
ELEMENT_BYTES = {"fp64": 8.0, "fp32": 4.0, "mixed": 2.65}


def listed():
    return [
        # one product per solver step at the size the benchmark is quoted on
        {"name": "apply fp64 262144", "kind": "apply", "precision": "fp64", "geometry": "sphere", "n": 262144},
        # the same in single precision, an odd number of unknowns, another mesh
        {"name": "apply fp32 100003", "kind": "apply", "precision": "fp32", "geometry": "cube", "n": 100003},
        # and in compressed storage
        {"name": "apply mixed 131072", "kind": "apply", "precision": "mixed", "geometry": "sphere", "n": 131072},
        # the smallest problem: launches and their latency are all there is
        {"name": "apply fp64 1536", "kind": "apply", "precision": "fp64", "geometry": "sphere", "n": 1536},
        # a small mesh (as many unknowns as the 216h model), its product captured once and replayed
        {"name": "replay fp64 21600", "kind": "replay", "precision": "fp64", "geometry": "plate", "n": 21600},
        # blocks of right-hand sides: block Krylov methods, several excitations of one structure
        {"name": "multi fp64 65536x8", "kind": "multi", "precision": "fp64", "geometry": "sphere", "n": 65536,
         "nrhs": 8},
        {"name": "multi fp32 100003x8", "kind": "multi", "precision": "fp32", "geometry": "cube", "n": 100003,
         "nrhs": 8},
        {"name": "multi fp64 30001x13", "kind": "multi", "precision": "fp64", "geometry": "plate", "n": 30001,
         "nrhs": 13},
        # many excitations: monostatic sweeps
        {"name": "multi fp32 65536x128", "kind": "multi", "precision": "fp32", "geometry": "sphere", "n": 65536,
         "nrhs": 128},
        {"name": "multi mixed 65536x16", "kind": "multi", "precision": "mixed", "geometry": "sphere", "n": 65536,
         "nrhs": 16},
        # independent matrices of uneven size, a few right-hand sides each, replayed as one graph
        {"name": "batch fp32 16", "kind": "batch", "precision": "fp32", "count": 16, "nmin": 2048, "nmax": 32768,
         "rhs": 16, "shapes": 5},
        # a whole solve: BiCGSTAB on a well-conditioned system
        {"name": "bicgstab fp64 12000", "kind": "solve", "precision": "fp64", "geometry": "sphere", "n": 12000},
    ]


def _between(rng, lo, hi):
    """A whole number in [lo, hi], its logarithm uniform."""
    return int(round(lo * (hi / lo) ** rng.random()))


def draw(rng):
    kind = rng.choice(("apply", "apply", "replay", "multi", "multi", "multi", "batch", "solve"))
    precision = rng.choice(("fp64", "fp32", "mixed"))
    if kind == "batch":
        return {"kind": kind, "precision": rng.choice(("fp64", "fp32")), "count": rng.randint(6, 16), "nmin": 2048,
                "nmax": _between(rng, 8192, 32768), "rhs": rng.randint(1, 16), "shapes": rng.randint(0, 999)}
    case = {"kind": kind, "precision": precision, "geometry": rng.choice(GEOMETRIES)}
    if kind == "apply":
        case["n"] = _between(rng, 1000, 150000)
    elif kind == "replay":
        case["n"] = _between(rng, 1000, 60000)
    elif kind == "solve":
        case["precision"] = "fp64"
        case["n"] = _between(rng, 2000, 12000)
    else:
        case["n"] = _between(rng, 3000, 65536)
        case["nrhs"] = _between(rng, 2, 24 if precision == "fp64" else 128)
    return case


# ---- matrices and right-hand sides -------------------------------------------

def _matrix(case, seed):
    """The case's H-matrix over points drawn from the seed."""
    hm = HMatrix.generate(case["n"], case["geometry"], leaf_size=32, eta=2.0, eps=1e-4, seed=seed + 1)
    if case["kind"] == "solve":
        # the single-layer matrix alone is indefinite: its diagonal raised to
        # the order of its norm, as the mass term of a second-kind equation
        rowmat = hm.rowmat.copy()
        diagonal = np.flatnonzero((hm.ltmtx == 2) & (hm.nstrtl == hm.nstrtt) & (hm.ndl == hm.ndt))
        for i in diagonal:
            n = int(hm.ndt[i])
            rowmat[int(hm.a1[i]) + np.arange(n) * (n + 1)] += 0.1 * case["n"]
        hm = HMatrix.from_arrays(hm.nd, hm.ktmax, hm.ltmtx, hm.kt, hm.ndl, hm.ndt, hm.nstrtl, hm.nstrtt, hm.a1,
                                 hm.a2, rowmat)
    return hm


def _instances(case):
    """The sizes of a batch, the same for every seed."""
    rng = np.random.default_rng(case["shapes"])
    for _ in range(case["count"]):
        n = int(round(case["nmin"] * (case["nmax"] / case["nmin"]) ** rng.random()))
        yield {"kind": "batch", "n": n, "geometry": GEOMETRIES[int(rng.integers(3))],
               "nrhs": int(rng.integers(1, case["rhs"] + 1))}


def _vectors(case, seed, nrhs=None):
    """Right-hand sides in [-1, 1), as numpy rows of the plan's element type."""
    rng = np.random.default_rng(seed + 1000)
    shape = (case["n"],) if nrhs is None else (nrhs, case["n"])
    return rng.uniform(-1.0, 1.0, shape).astype(np.float32 if case["precision"] == "fp32" else np.float64)


def _plan_width(precision, nrhs):
    """The plan's pass width for so many right-hand sides: the wide tensor-core
    form from 32, the 16-wide pass of mixed plans from 16, else up to 8."""
    if precision != "fp64" and nrhs >= 32:
        return 128
    if precision == "mixed" and nrhs >= 16:
        return 16
    return min(nrhs, 8)


def prepare(case, seed):
    kind, precision = case["kind"], case["precision"]
    if kind == "batch":
        insts = [dict(c, precision=precision) for c in _instances(case)]
        mats = [_matrix(c, seed + 31 * i) for i, c in enumerate(insts)]
        if precision == "fp32":
            mats = [m.to_float() for m in mats]
        X = [torch.from_numpy(_vectors(c, seed + 31 * i, c["nrhs"])).cuda() for i, c in enumerate(insts)]
        Y = [torch.empty_like(x) for x in X]
        batch = Batch(mats, precision, nrhs=[c["nrhs"] for c in insts])
        batch.capture(X, Y)
        return {"kind": kind, "batch": batch, "X": X, "Y": Y}
    hm = _matrix(case, seed)
    nrhs = case.get("nrhs")
    x = torch.from_numpy(_vectors(case, seed, nrhs)).cuda()
    y = torch.empty_like(x)
    plan = Plan(hm, precision, nrhs_max=1 if nrhs is None else _plan_width(precision, nrhs))
    if kind == "replay":
        plan.capture(x, y)
    return {"kind": kind, "plan": plan, "x": x, "y": y}


def run(state):
    kind = state["kind"]
    if kind == "batch":
        state["batch"].launch()
        return state["Y"]
    plan, x, y = state["plan"], state["x"], state["y"]
    if kind == "apply":
        plan.apply(x, y)
    elif kind == "replay":
        plan.replay()
    elif kind == "multi":
        plan.apply_multi(x, y)
    else:  # solve H y = x from a zero guess
        y.zero_()
        steps, _ = plan.bicgstab(x, y, eps=1e-8, max_steps=100)
        return {"u": y, "steps": steps}
    return y


def work(case):
    """The stored elements and each vector once per pass over the matrix; a pass
    takes any number of right-hand sides.  A solve counts its products."""
    e = ELEMENT_BYTES[case["precision"]]
    ev = 4 if case["precision"] == "fp32" else 8
    if case["kind"] == "batch":
        parts = [(_matrix(c, 0).stored_elements(), c["n"], c["nrhs"]) for c in _instances(case)]
    else:
        parts = [(_matrix(case, 0).stored_elements(), case["n"], case.get("nrhs", 1))]
    products = 12 if case["kind"] == "solve" else 1
    return {"bytes": products * sum(m * e + 2 * n * r * ev for m, n, r in parts),
            "flops": products * sum(2 * m * r for m, _, r in parts)}


# ---- the same in FP64 with numpy -----------------------------------------------

def _product(hm, x):
    """H x, leaf by leaf; x of shape (N,) or (nrhs, N)."""
    cols = np.ascontiguousarray(x.T, dtype=np.float64)
    y = np.zeros_like(cols)
    rowmat = hm.rowmat
    table = zip(*(a.tolist() for a in (hm.ltmtx, hm.kt, hm.ndl, hm.ndt, hm.nstrtl, hm.nstrtt, hm.a1, hm.a2)))
    for kind, k, ndl, ndt, row, col, a1, a2 in table:
        xs = cols[col - 1:col - 1 + ndt]
        if kind == 1:
            t = rowmat[a1:a1 + k * ndt].reshape(k, ndt) @ xs
            y[row - 1:row - 1 + ndl] += rowmat[a2:a2 + k * ndl].reshape(k, ndl).T @ t
        else:
            y[row - 1:row - 1 + ndl] += rowmat[a1:a1 + ndl * ndt].reshape(ndl, ndt) @ xs
    return np.ascontiguousarray(y.T)


def _bicgstab(product, b, eps, max_steps):
    """HACApK's iteration from a zero guess."""
    u, r = np.zeros_like(b), b.copy()
    shadow, p, hp = r.copy(), np.zeros_like(b), np.zeros_like(b)
    beta = zeta = 0.0
    for step in range(1, max_steps + 1):
        p = r + beta * (p - zeta * hp)
        hp = product(p)
        nom = shadow @ r
        alpha = nom / (shadow @ hp)
        t = r - alpha * hp
        ht = product(t)
        zeta = (ht @ t) / (ht @ ht)
        u = u + alpha * p + zeta * t
        r = t - zeta * ht
        beta = alpha / zeta * (shadow @ r) / nom
        if np.linalg.norm(r) < eps * np.linalg.norm(b):
            break
    return u, step


def exact(case, seed):
    if case["kind"] == "batch":
        out = []
        for i, c in enumerate(_instances(case)):
            c = dict(c, precision=case["precision"])
            out.append(_product(_matrix(c, seed + 31 * i), _vectors(c, seed + 31 * i, c["nrhs"])))
        return out
    hm = _matrix(case, seed)
    x = _vectors(case, seed, case.get("nrhs"))
    if case["kind"] == "solve":
        u, steps = _bicgstab(lambda v: _product(hm, v), x, 1e-8, 100)
        return {"u": u, "steps": steps}
    return _product(hm, x)

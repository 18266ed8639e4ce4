"""Timed cases of the GMRES-IR path: what a program that uses this package has it do.

A case is one call, or the few calls that belong together, on a quasi-definite
KKT system of :mod:`mpir_b200.kkt`: a 2-D or 3-D Laplacian H (``grid`` points a
side), about a quarter as many constraint rows with 4 (2-D) or 6 (3-D) entries
each, and b = K x_true.  ``kind`` says which calls:

* ``refactor``  new values on an analysed pattern, then one right-hand side
  (``factor`` + ``Solve``): a step of an interior-point or time-stepping loop;
* ``rhs``       a new right-hand side on a resident factor (``Solve``);
* ``batch``     ``nrhs`` right-hand sides on a resident factor in lockstep
  (``SolveBatch``);
* ``group``     ``members`` value sets on one pattern, refactorized together
  (``FactorGroup.factor``), then ``nrhs`` right-hand sides on each;
* ``compute``   a system seen for the first time: ``Compute`` (analysis and
  factor) + ``Solve``, as the example driver does;
* ``qdldl``     the QDLDL functions by themselves, natural order:
  ``QDLDL_etree``, ``QDLDL_factor``, ``QDLDL_solve`` (one pattern a size, the
  values and the right-hand side from the seed);
* ``serve``     ``requests`` requests queued at once on a serving engine whose
  patterns are resident: for each pattern one new value set and, on it, the
  new right-hand sides that follow it.

The systems are host arrays, as the entry points take them and return them.
The analysed solver, the resident factor and the engine are made in
``prepare``: a program that uses them keeps them.
"""
import math

import numpy as np

import mpir_b200 as mp
from mpir_b200 import kkt

# Lower bound of a diagonal entry of H and of |delta|, as the generators of
# mpir_b200.kkt and the benchmark have them.
SHIFT = 1e-2
DELTA = {2: 1e-4, 3: 1e-6}
PER_ROW = {2: 4, 3: 6}


def listed():
    return [
        # The smallest configured system (n = 1,280), one refactorization and
        # one solve: launches and latency.
        {"name": "refactor_2d32", "kind": "refactor", "dim": 2, "grid": 32, "uf": "f32", "ur": "f64"},
        # An odd mid-size grid (n = 24,603) with the double-double residual.
        {"name": "refactor_3d27_dd", "kind": "refactor", "dim": 3, "grid": 27, "uf": "f32", "ur": "dd"},
        # The configured drop-in at scale (n = 138,240).
        {"name": "refactor_3d48", "kind": "refactor", "dim": 3, "grid": 48, "uf": "f32", "ur": "f64"},
        # The bfloat16 tier (n = 14,045): a cheap factor and more iterations.
        {"name": "refactor_2d106_bf16", "kind": "refactor", "dim": 2, "grid": 106, "uf": "bf16", "ur": "f64"},
        # New right-hand sides on a resident factor, the commonest request of a
        # served stream: a small system (n = 2,160) and a larger one (n = 40,960).
        {"name": "rhs_3d12", "kind": "rhs", "dim": 3, "grid": 12, "uf": "f32", "ur": "f64"},
        {"name": "rhs_3d32", "kind": "rhs", "dim": 3, "grid": 32, "uf": "f32", "ur": "f64"},
        # Lockstep solves: a full batch of 16 (n = 20,480) and the ragged
        # batch of three that a served stream has on average (n = 40,951).
        {"name": "batch16_2d128", "kind": "batch", "dim": 2, "grid": 128, "nrhs": 16, "uf": "f32", "ur": "f64"},
        {"name": "batch3_2d181", "kind": "batch", "dim": 2, "grid": 181, "nrhs": 3, "uf": "f32", "ur": "f64"},
        # The same-pattern batch of an interior-point sweep (n = 5,120 each).
        {"name": "group8_2d64", "kind": "group", "dim": 2, "grid": 64, "members": 8, "nrhs": 4, "uf": "f32",
         "ur": "f64"},
        # A pattern seen for the first time (n = 11,576).
        {"name": "compute_3d21", "kind": "compute", "dim": 3, "grid": 21, "uf": "f32", "ur": "f64"},
        # The QDLDL functions, natural order, on the smallest configured system.
        {"name": "qdldl_2d32", "kind": "qdldl", "dim": 2, "grid": 32},
        # The serving engine: 18 requests on 3 resident patterns of unlike
        # sizes (n = 14,045, 5,120 and 24,603).
        {"name": "serve_18", "kind": "serve", "dim": 2, "grid": 106, "patterns": 3, "requests": 18, "uf": "f32",
         "ur": "f64"},
    ]


def _grid(rng, dim, lo, hi):
    """A grid whose system has n log-uniform in [lo, hi] unknowns (n = 1.25 grid^dim)."""
    n = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    return max(5, round((n / 1.25) ** (1.0 / dim)))


def draw(rng):
    kind = rng.choice(["refactor", "refactor", "rhs", "rhs", "batch", "batch", "group", "compute"])
    dim = rng.choice([2, 3])
    hi = {"refactor": 80e3, "rhs": 80e3, "batch": 40e3, "group": 12e3, "compute": 30e3}[kind]
    c = {"kind": kind, "dim": dim, "grid": _grid(rng, dim, 1e3, hi), "rows": rng.randint(20, 29), "uf": "f32",
         "ur": rng.choice(["f64", "f64", "dd"])}
    if kind in ("refactor", "rhs") and c["dim"] == 2 and rng.random() < 0.3:
        c["uf"] = "bf16"
    if kind == "batch":
        c["nrhs"] = rng.randint(2, 16)
    if kind == "group":
        c["members"] = rng.randint(2, 8)
        c["nrhs"] = rng.randint(1, 8)
    return c


def _system(case, seed, nrhs=1, dim=None, grid=None):
    """One system; x_true and b are (nrhs, n) arrays when nrhs > 1."""
    dim, grid = dim or case["dim"], grid or case["grid"]
    fixed = case["kind"] == "qdldl"
    m = max(1, grid ** dim * case.get("rows", 25) // 100)
    s = kkt.make(grid, dim, m, PER_ROW[dim], DELTA[dim], shift=SHIFT, seed=0 if fixed else int(seed), nrhs=nrhs)
    if fixed:
        rng = np.random.default_rng(int(seed))
        s.Ax = _values(s, rng)
        s.x_true = rng.uniform(-1.0, 1.0, size=s.n)
        s.b = kkt.symmetric_matvec(s.n, s.Ap, s.Ai, s.Ax, s.x_true)
    return s


def _rows(v):
    """A system's x_true or b as one row a vector."""
    return np.atleast_2d(v)


def _values(s, rng):
    """New values on the pattern of s: a larger diagonal of H, other constraint rows (K stays quasi-definite)."""
    Ax = s.Ax.copy()
    cols = np.repeat(np.arange(s.n, dtype=np.int64), np.diff(s.Ap))
    diag_h = (s.Ai == cols) & (cols < s.n1)
    Ax[diag_h] += np.exp(rng.uniform(math.log(1e-6), 0.0, size=int(diag_h.sum())))
    cons = (cols >= s.n1) & (s.Ai < s.n1)
    Ax[cons] = rng.standard_normal(int(cons.sum()))
    return Ax


def _member_sets(case, seed):
    """The pattern of a group, its members' values, solutions and right-hand sides."""
    s = _system(case, seed)
    out = []
    for k in range(case["members"]):
        rng = np.random.default_rng((int(seed), k))
        Ax = _values(s, rng)
        X = rng.uniform(-1.0, 1.0, size=(case["nrhs"], s.n))
        out.append((Ax, X, np.stack([kkt.symmetric_matvec(s.n, s.Ap, s.Ai, Ax, x) for x in X])))
    return s, out


def _request_sets(case, seed):
    """The patterns of a serving case and its requests: (pattern, value set, b, x_true), each pattern's value
    set used by requests / patterns right-hand sides."""
    shapes = [(2, case["grid"]), (2, max(8, case["grid"] * 3 // 5)), (3, max(5, case["grid"] // 4 + 1))][: case["patterns"]]
    systems = [_system(case, int(seed) + i, dim=d, grid=g) for i, (d, g) in enumerate(shapes)]
    reqs = []
    for r in range(case["requests"]):
        p = r % len(systems)
        s = systems[p]
        x = np.random.default_rng((int(seed), r)).uniform(-1.0, 1.0, size=s.n)
        reqs.append((p, kkt.symmetric_matvec(s.n, s.Ap, s.Ai, s.Ax, x), x))
    return systems, reqs


def _solver(case, s):
    solver = mp.GmresLDLIR(uf=case["uf"], uw="f64", ur=case["ur"])
    if case["uf"] != "f32":  # a 16-bit factor refines in more, longer steps
        solver.SetMaxIRIterations(30)
        solver.SetMaxGmresIterations(50)
    solver.analyze(s.Ap, s.Ai, s.Ax)
    return solver


def prepare(case, seed):
    kind = case["kind"]
    if kind == "group":
        s, sets = _member_sets(case, seed)
        solver = _solver(case, s)
        return {"case": case, "solver": solver, "group": mp.FactorGroup(solver, case["members"]),
                "values": [m[0] for m in sets], "b": [m[2] for m in sets]}
    if kind == "serve":
        systems, reqs = _request_sets(case, seed)
        # Room for the factors of a few passes: an engine at work holds as many
        # as its budget allows and evicts the least recently used.
        server = mp.Server(uf=case["uf"], ur=case["ur"], budget_bytes=4 * 10 ** 9)
        state = {"case": case, "server": server, "systems": systems, "b": [(p, b) for p, b, _ in reqs], "pass": 0}
        for _ in range(4):  # the patterns are resident and the budget is in use
            run(state)
        return state
    s = _system(case, seed, nrhs=case.get("nrhs", 1))
    state = {"case": case, "s": s, "b": np.ascontiguousarray(_rows(s.b))}
    if kind in ("refactor", "rhs", "batch"):
        state["solver"] = _solver(case, s)
    if kind in ("rhs", "batch"):
        state["solver"].factor(s.Ax)
    return state


def run(state):
    case = state["case"]
    kind, s = case["kind"], state.get("s")
    if kind == "refactor":
        state["solver"].factor(s.Ax)
        return state["solver"].Solve(state["b"][0])
    if kind == "rhs":
        return state["solver"].Solve(state["b"][0])
    if kind == "batch":
        return state["solver"].SolveBatch(state["b"])
    if kind == "group":
        state["group"].factor(state["values"])
        return [state["group"].SolveBatch(k, b) for k, b in enumerate(state["b"])]
    if kind == "compute":
        solver = mp.GmresLDLIR(uf=case["uf"], uw="f64", ur=case["ur"])
        solver.Compute(s.Ap, s.Ai, s.Ax)
        return solver.Solve(state["b"][0])
    if kind == "qdldl":
        _, Lnz, etree = mp.QDLDL_etree(s.n, s.Ap, s.Ai)
        npos, Lp, Li, Lx, D, Dinv = mp.QDLDL_factor(s.n, s.Ap, s.Ai, s.Ax, Lnz, etree)
        x = mp.QDLDL_solve(s.n, Lp, Li, Lx, Dinv, state["b"][0].copy())
        return {"npos": npos, "Lp": Lp, "Li": Li, "Lx": Lx, "D": D, "Dinv": Dinv, "x": x}
    # serve: this pass's value sets are new to the engine.
    server, systems = state["server"], state["systems"]
    state["pass"] += 1
    ids = [server.submit(p + 1, state["pass"] * len(systems) + p, systems[p].Ap, systems[p].Ai, systems[p].Ax, b)
           for p, b in state["b"]]
    return [server.wait(i)[0] for i in ids]


def exact(case, seed):
    """The solutions that the right-hand sides were made from (b = K x_true in float64); for the QDLDL functions
    the dense float64 factor."""
    kind = case["kind"]
    if kind == "group":
        return [m[1] for m in _member_sets(case, seed)[1]]
    if kind == "serve":
        return [x for _, _, x in _request_sets(case, seed)[1]]
    s = _system(case, seed, nrhs=case.get("nrhs", 1))
    if kind != "qdldl":
        return s.x_true
    if s.n > 3000:
        return None
    K = np.zeros((s.n, s.n))
    cols = np.repeat(np.arange(s.n), np.diff(s.Ap))
    K[s.Ai, cols] = s.Ax
    K[cols, s.Ai] = s.Ax
    # Dense LDL^T, column by column; L's pattern is that of QDLDL_etree.
    L, D = K.copy(), np.zeros(s.n)
    for j in range(s.n):
        D[j] = L[j, j]
        below = np.flatnonzero(L[j + 1:, j]) + j + 1
        l = L[below, j] / D[j]
        L[np.ix_(below, below)] -= np.outer(l, L[below, j])
        L[below, j] = l
    _, Lnz, etree = mp.QDLDL_etree(s.n, s.Ap, s.Ai)
    rows = _factor_rows(s, etree)
    Lx = np.concatenate([L[r, j] for j, r in enumerate(rows)] or [np.zeros(0)])
    return {"npos": None, "Lp": None, "Li": None, "Lx": Lx, "D": D, "Dinv": 1.0 / D, "x": s.x_true}


def _factor_rows(s, etree):
    """Row indices of each column of L: row k holds the tree paths from the entries of column k of K up to k."""
    rows, mark = [[] for _ in range(s.n)], np.full(s.n, -1)
    for k in range(s.n):
        mark[k] = k
        for i in s.Ai[s.Ap[k]:s.Ap[k + 1]]:
            while mark[i] != k:
                rows[i].append(k)
                mark[i] = k
                i = etree[i]
    return [np.array(r, dtype=np.int64) for r in rows]


def work(case):
    """Bytes: the values (and the factor, where it is resident) and right-hand sides in, the solutions out.
    Flops: the factor's, and L and L^T applied twice a right-hand side (the first solve and one correction)."""
    kind = case["kind"]

    def one(s, factors, solves, order=mp.ORDER_AUTO):
        info = mp.analyze_host(s.Ap, s.Ai, s.Ax, ordering=order)["info"]
        resident = 0 if factors else 4.0 * info["nnz_L"]
        return (factors * 8.0 * s.nnz + resident + 16.0 * s.n * solves,
                factors * info["factor_flops"] + solves * 2 * 4.0 * info["nnz_L"])

    if kind == "group":
        got = [one(_system(case, 0), case["members"], case["members"] * case["nrhs"])]
    elif kind == "serve":
        systems, reqs = _request_sets(case, 0)
        got = [one(s, 1, sum(1 for r in reqs if r[0] == p)) for p, s in enumerate(systems)]
    elif kind == "qdldl":
        s = _system(case, 0)
        got = [one(s, 1, 0.5, mp.ORDER_NATURAL)]
        got.append((12.0 * mp.QDLDL_etree(s.n, s.Ap, s.Ai)[0], 0.0))  # L itself comes back
    else:
        got = [one(_system(case, 0), 0 if kind in ("rhs", "batch") else 1, case.get("nrhs", 1))]
    return {"bytes": sum(g[0] for g in got), "flops": sum(g[1] for g in got)}

"""The work a detector tomography has this package do, as cases to time.

A case names a path through the public entry points (pqdts_gb300.Solver and
solve_batch) and its sizes: M photon numbers, N outcomes, D probes, as in
pqdts_gb300.synth.CONFIGS and make_batch.  Inputs follow the same generator
(coherent probes, an ideal detector of efficiency eta, sampled frequencies),
evaluated on the GPU so that many instances can be made.

  project   simplexproj of `rows` vectors of length N: the projection on its
            own, as a host program calls it row by row or for a whole POVM
  gradient  a host-driven optimiser's step: set_x, L, dL
  hessian   BF (FP64) or BF32 (mixed) of one direction, full or reduced space
  solve     a tomography from the data: set_problem, solve, get_x on a handle
            that the program keeps for its stream of data sets
  resume    set_x, solve, get_x on a problem that is already loaded: restarts
            and comparisons of starting points
  batch     solve_batch over detectors of uneven sizes with resampled data

`late` iterates carry the exact zeros that the projections leave after the
first iterations; early ones are dense.  Capped solves (maxiter) are the
bounded runs of a scan over gamma or of a scheduler's time slice.  The mixed
ones run with the timed launch schedules off, as a program does that wants
the same bits from one process to the next, and for one iteration a stage:
every later one multiplies what the FP32 iterations round differently.
"""
import math

import numpy as np
import torch

import pqdts_gb300 as pq
from pqdts_gb300.synth import Instance

PRECISION = {"fp64": pq.FP64, "mixed": pq.MIXED}


def listed():
    return [
        # one detector row: the drop-in projection at its smallest, all latency
        dict(name="project_one", kind="project", rows=1, N=20),
        # the whole POVM of the 10^4 x 10^3 configuration projected at once
        dict(name="project_povm", kind="project", rows=10000, N=1000),
        # objective and gradient of the benchmark configuration at an iterate
        # with its zeros
        dict(name="gradient_fp64", kind="gradient", precision="fp64", M=2000, N=200, D=4000, eta=0.9, late=True),
        # ... of the 10^4 x 10^3 configuration in mixed precision
        dict(name="gradient_mixed", kind="gradient", precision="mixed", M=10000, N=1000, D=20000, eta=0.75, late=True),
        # one Hessian product of each precision, as an outer Krylov method takes it
        dict(name="hessian_fp64", kind="hessian", precision="fp64", M=2000, N=200, D=4000, eta=0.9, late=True),
        dict(name="hessian_mixed", kind="hessian", precision="mixed", M=10000, N=1000, D=20000, eta=0.75, late=True),
        # whole tomographies in FP64: the smallest configuration to the
        # reference's stopping rule, the benchmark configuration capped
        dict(name="solve_small", kind="solve", precision="fp64", M=200, N=20, D=400, eta=0.9, gamma=1e-4, maxiter=100),
        dict(name="solve_fp64", kind="solve", precision="fp64", M=2000, N=200, D=4000, eta=0.9, gamma=1e-5, maxiter=30),
        # a mixed one at odd sizes, from the data: the set-up counts too
        dict(name="solve_mixed", kind="solve", precision="mixed", M=5003, N=501, D=9501, eta=0.8, gamma=1e-6,
             maxiter=1),
        # restarts at large sizes in both precisions
        dict(name="resume_fp64", kind="resume", precision="fp64", M=5000, N=500, D=10000, eta=0.8, gamma=1e-6,
             maxiter=3),
        dict(name="resume_mixed", kind="resume", precision="mixed", M=10000, N=1000, D=20000, eta=0.75, gamma=1e-6,
             maxiter=1),
        # resampled data of uneven detectors, one call
        dict(name="batch", kind="batch", precision="fp64", M=1201, N=151, D=2399, eta=0.8, count=6, maxiter=6),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["project", "gradient", "gradient", "hessian", "hessian", "solve", "resume", "batch"])
    if kind == "project":
        return dict(kind=kind, rows=_log(rng, 1, 10000), N=_log(rng, 20, 1000))
    precision = "fp64" if kind == "batch" else rng.choice(["fp64", "mixed"])
    largest = 10000
    if precision == "fp64":
        largest = {"gradient": 10000, "hessian": 10000, "solve": 1500, "resume": 4000, "batch": 1000}[kind]
    M = _log(rng, 200, min(largest, 5000) if kind == "solve" else largest)
    case = dict(kind=kind, precision=precision, M=M, N=max(3, round(M * rng.uniform(0.08, 0.1))),
                D=round(M * rng.uniform(1.7, 2.0)), eta=round(rng.uniform(0.6, 0.95), 3))
    if kind in ("gradient", "hessian"):
        case.update(late=rng.random() < 0.6)
        return case
    case.update(maxiter={"solve": rng.randint(5, 30), "resume": rng.randint(1, 3), "batch": rng.randint(2, 6)}[kind])
    if precision == "mixed":
        case.update(maxiter=1)
    if kind == "batch":
        case.update(count=rng.randint(3, 6))
    else:
        case.update(gamma=10.0 ** rng.uniform(-7, -2))
    return case


# -- inputs ------------------------------------------------------------------


def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def _bands(M, D, xmax):
    """Poisson windows F[d, i] >= 1e-16 of coherent probes: lo, hi (D,) and
    the concatenated values, on the GPU."""
    x = torch.linspace(0.01, xmax, D, dtype=torch.float64, device="cuda")
    half = 12.0 * math.sqrt(xmax) + 40.0
    width = int(2 * half) + 3
    i = torch.floor(x - half).long()[:, None] + torch.arange(width, device="cuda")[None, :]
    inside = (i >= 0) & (i < M)
    ii = i.clamp(0, M - 1).double()
    p = torch.exp(ii * torch.log(x)[:, None] - x[:, None] - torch.lgamma(ii + 1.0))
    keep = inside & (p >= 1e-16)
    big = torch.iinfo(torch.int64).max
    lo = torch.where(keep, i, big).amin(1)
    hi = torch.where(keep, i, -1).amax(1)
    lo = torch.where(hi >= 0, lo, -1)
    return lo, hi, p[keep]


def _povm(M, N, eta):
    """The ideal detector: binomial columns, the tail mass in the last one."""
    i = torch.arange(M, dtype=torch.float64, device="cuda")[:, None]
    n = torch.arange(N - 1, dtype=torch.float64, device="cuda")[None, :]
    logp = (torch.lgamma(i + 1) - torch.lgamma(n + 1) - torch.lgamma((i - n).clamp(min=0) + 1)
            + n * math.log(eta) + (i - n) * math.log(1.0 - eta))
    pi = torch.where(n <= i, torch.exp(logp), torch.zeros((), dtype=torch.float64, device="cuda"))
    return torch.cat([pi, (1.0 - pi.sum(1, keepdim=True)).clamp(min=0.0)], 1)


def _block_rows(lo, hi, val):
    """F in dense blocks of 256 rows: (row slice, column slice, block)."""
    w = torch.where(lo >= 0, hi - lo + 1, 0)
    off = torch.cumsum(w, 0) - w
    for d0 in range(0, lo.numel(), 256):
        d1 = min(lo.numel(), d0 + 256)
        rows = torch.nonzero(w[d0:d1] > 0).flatten() + d0
        if not rows.numel():
            continue
        a, b = int(lo[rows].min()), int(hi[rows].max()) + 1
        j = torch.arange(a, b, device=lo.device)[None, :] - lo[d0:d1, None]
        on = (j >= 0) & (j < w[d0:d1, None])
        block = torch.where(on, val[(off[d0:d1, None] + j).clamp(0, val.numel() - 1)], 0.0)
        yield slice(d0, d1), slice(a, b), block


def _forward(lo, hi, val, X):
    out = torch.zeros((lo.numel(), X.shape[1]), dtype=X.dtype, device=X.device)
    for rows, cols, block in _block_rows(lo, hi, val):
        out[rows] = block @ X[cols]
    return out


def _transposed(lo, hi, val, R, M):
    out = torch.zeros((M, R.shape[1]), dtype=R.dtype, device=R.device)
    for rows, cols, block in _block_rows(lo, hi, val):
        out[cols] += block.T @ R[rows]
    return out


def _data(M, N, D, eta, seed, count=1):
    """Bands of F, the detector's POVM, and `count` samples of P with about
    10^7 shots a probe."""
    g = _generator(seed)
    lo, hi, val = _bands(M, D, 0.9 * M)
    pi = _povm(M, N, eta)
    rate = _forward(lo, hi, val, pi).clamp(min=0.0)
    rate *= 1e7 / rate.sum(1, keepdim=True).clamp(min=1e-300)
    P = []
    for _ in range(count):
        counts = torch.poisson(rate, generator=g)
        P.append((counts / counts.sum(1, keepdim=True).clamp(min=1.0)).cpu().numpy())
    return lo, hi, val, pi, P


def _instances(case, seed, gammas):
    lo, hi, val, pi, P = _data(case["M"], case["N"], case["D"], case["eta"], seed, len(gammas))
    lo, hi, val = lo.cpu().numpy(), hi.cpu().numpy(), val.cpu().numpy()
    return [Instance(case["M"], case["N"], case["D"], g, 1e-6, lo, hi, val, p) for g, p in zip(gammas, P)], pi


def _project(Y):
    """Rows of Y onto the unit simplex, by sorting."""
    s = torch.sort(Y, dim=1, descending=True).values
    k = torch.arange(1, Y.shape[1] + 1, dtype=Y.dtype, device=Y.device)
    tau = (torch.cumsum(s, 1) - 1.0) / k
    rho = (s > tau).sum(1, keepdim=True)
    return (Y - torch.gather(tau, 1, rho - 1)).clamp(min=0.0)


def _iterate(pi, late, g):
    """A feasible iterate: the detector plus noise, projected (late: noise
    that leaves most entries at exactly zero; early: every entry positive)."""
    noise = torch.rand(pi.shape, dtype=torch.float64, device="cuda", generator=g)
    if late:
        return _project(pi + 0.02 * (noise - 0.8))
    X = 0.3 * pi + 0.7 / pi.shape[1] * (0.5 + noise)
    return X / X.sum(1, keepdim=True)


def _fortran(X):
    return np.asfortranarray(X.cpu().numpy())


def _direction(case, pi, X, g):
    """A CG direction: noise on the detector's scale, zero on the active set."""
    V = torch.randn(pi.shape, dtype=torch.float64, device="cuda", generator=g) * (0.01 + pi)
    return torch.where(X > 0, V, 0.0) if case["late"] else V


def _inputs(case, seed):
    """The raw inputs of a gradient or hessian case, on the GPU."""
    g = _generator(seed + 1)
    inst, pi = _instances(case, seed, [1e-6])
    X = _iterate(pi, case["late"], g)
    return inst[0], X, _direction(case, pi, X, g)


def _vectors(case, seed):
    g = _generator(seed)
    pi = _povm(max(case["rows"], 2), case["N"], 0.9)[: case["rows"]]
    return pi + 0.02 * (torch.rand(pi.shape, dtype=torch.float64, device="cuda", generator=g) - 0.5)


def prepare(case, seed):
    kind = case["kind"]
    if kind == "project":
        return dict(kind=kind, solver=pq.Solver(0), Y=_vectors(case, seed).cpu().numpy())
    if kind == "batch":
        # uneven members of one family, each resampled with its own gamma
        members = []
        for k in range(case["count"]):
            f = 0.5 + 0.5 * (k + 1) / case["count"]
            sub = dict(case, M=int(case["M"] * f), N=max(3, int(case["N"] * f)), D=int(case["D"] * f))
            inst, _ = _instances(sub, seed + 17 * k, [10.0 ** (-7 + 5 * k / case["count"])])
            members += inst
        return dict(kind=kind, members=members, precision=PRECISION[case["precision"]], maxiter=case["maxiter"])
    s = pq.Solver(0)
    precision = PRECISION[case["precision"]]
    if precision == pq.MIXED and kind in ("solve", "resume"):
        s.set_option("autotune", 0)
    if kind in ("gradient", "hessian"):
        inst, X, V = _inputs(case, seed)
        s.set_instance(inst, precision)
        if kind == "gradient":
            return dict(kind=kind, solver=s, X=_fortran(X))
        # the reduced space of a late iterate, the full one of an early one
        s.set_space(not case["late"], X.argmax(1).int().cpu().numpy() if case["late"] else None)
        return dict(kind=kind, solver=s, V=_fortran(V), mixed=case["precision"] == "mixed")
    inst, pi = _instances(case, seed, [case["gamma"]])
    state = dict(kind=kind, solver=s, inst=inst[0], precision=precision, maxiter=case["maxiter"])
    if kind == "resume":
        s.set_instance(inst[0], precision)
        state["X"] = _fortran(_iterate(pi, False, _generator(seed + 1)))
    return state


def run(state):
    kind = state["kind"]
    if kind == "project":
        return state["solver"].simplexproj(state["Y"])
    if kind == "batch":
        X, stats = pq.solve_batch(state["members"], precision=state["precision"], maxiter=state["maxiter"])
        return dict(X=X, L=[st["L"] for st in stats], cg=[int(st["cg"]) for st in stats])
    s = state["solver"]
    if kind == "gradient":
        s.set_x(state["X"])
        return dict(L=s.L(), G=s.dL())
    if kind == "hessian":
        # BF32's products are FP32 numbers, handed out widened
        return s.BF32(state["V"]).astype(np.float32) if state["mixed"] else s.BF(state["V"])
    if kind == "solve":
        s.set_instance(state["inst"], state["precision"])
    else:
        s.set_x(state["X"])
    st = s.solve(mode=2, maxiter=state["maxiter"], eps=1e-6)
    return dict(X=s.get_x(), L=st["L"], conv=st["conv"], outer=int(st["outer"]), cg=int(st["cg"]))


# -- what a pass cannot do without ---------------------------------------------


def _nnz(M, D):
    """Entries of F: windows of +-8.3 standard deviations (pmf >= 1e-16)."""
    x = np.linspace(0.01, 0.9 * M, D)
    lo = np.clip(x - 8.3 * np.sqrt(x), 0, M)
    hi = np.clip(x + 8.3 * np.sqrt(x) + 10, 0, M)
    return float((hi - lo).sum())


def work(case):
    kind = case["kind"]
    if kind == "project":
        n = case["rows"] * case["N"]
        return dict(bytes=16 * n, flops=3 * n)
    if kind == "batch":
        total = dict(bytes=0.0, flops=0.0)
        for k in range(case["count"]):
            f = 0.5 + 0.5 * (k + 1) / case["count"]
            w = work(dict(case, kind="solve", M=int(case["M"] * f), N=max(3, int(case["N"] * f)), D=int(case["D"] * f)))
            total = {key: total[key] + w[key] for key in total}
        return total
    M, N, D = case["M"], case["N"], case["D"]
    nnz = _nnz(M, D)
    # F's values and P read once, X read and the result written
    size = 8 * nnz + 8 * D * N + 16 * M * N
    if kind == "gradient":
        return dict(bytes=size, flops=4 * nnz * N)
    if kind == "hessian":
        return dict(bytes=size - 8 * D * N, flops=4 * nnz * N)
    # a solve: at least one gradient, one Hessian product and one step's
    # objective in each outer iteration of its two stages
    return dict(bytes=size, flops=2 * case["maxiter"] * 10 * nnz * N)


# -- the same results in plain 64-bit torch -------------------------------------


def exact(case, seed):
    kind = case["kind"]
    if kind == "project":
        return _project(_vectors(case, seed))
    if kind not in ("gradient", "hessian"):
        return None  # a solve's iterations have no closed form
    inst, X, V = _inputs(case, seed)
    lo, hi = torch.from_numpy(inst.band_lo).cuda(), torch.from_numpy(inst.band_hi).cuda()
    val = torch.from_numpy(inst.band_val).cuda()
    gam, M = inst.gamma, inst.M

    def products(A, B):
        """F^T (2 (F A - B)) and the gamma stencil on A."""
        r = _forward(lo, hi, val, A) - B
        G = _transposed(lo, hi, val, 2.0 * r, M)
        d = A[:-1] - A[1:]
        G[:-1] += 2.0 * gam * d
        G[1:] -= 2.0 * gam * d
        return r, d, G

    if kind == "gradient":
        r, d, G = products(X, torch.from_numpy(inst.P).cuda())
        banded = (lo >= 0)[:, None]
        return dict(L=float((r * r * banded).sum() + gam * (d * d).sum()), G=G)
    if not case["late"]:
        return products(V, torch.zeros((), dtype=torch.float64, device="cuda"))[2]
    # reduced space: the max column follows from the others
    m = X.argmax(1, keepdim=True)
    full = V.scatter(1, m, 0.0)
    full = full.scatter(1, m, -full.sum(1, keepdim=True))
    H = products(full, torch.zeros((), dtype=torch.float64, device="cuda"))[2]
    return H - torch.gather(H, 1, m)

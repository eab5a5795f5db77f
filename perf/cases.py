"""The workloads this framework's speed is judged on, through its public entry points.

A case is one call that a program makes again and again with matrices of one
pattern (``call``):

* ``step``   new values, then PCG: rschol_refactor_device + rschol_pcg_device
             (a time step or a Newton step; the benchmark's unit of work);
* ``solve``  PCG on a factor that is kept (implicit time stepping with a fixed
             operator, many load cases), one right-hand side or a batch;
* ``apply``  one application of the preconditioner inside the caller's own
             iteration; here with every separator below max_dense_block, where
             nothing is compressed and the application is the direct solve;
* ``serve``  a PCG session (continuous batching) fed requests of several
             right-hand sides from host buffers until all are done;
* ``new``    a matrix seen for the first time: ordering, symbolic analysis,
             factorisation and PCG from host arrays through the Python classes.

Matrices are the repository's own synthetic problems (variable-coefficient
5-point / 7-point diffusion, Q1 elasticity) with values from the seed.
"""
import functools
import math

import numpy as np
import torch

import rank_structured_cholesky_gb300 as rs

# c1 of the benchmark: a small grid with every kind of compressed block
COMPRESSING = dict(nd_leaf=64, max_dense_block=16, max_diag_block=32, rank_cap=32, oversampling=10)


def _case(name, call, grid, nx, ny=1, nz=1, *, sigma=1.0, precision="mixed", nrhs=1, eps=1e-8, **params):
    c = dict(call=call, grid=grid, nx=nx, ny=ny, nz=nz, sigma=sigma, precision=precision, nrhs=nrhs, eps=eps)
    for k, v in params.items():
        c["p_" + k] = v
    return dict(name=name, **c) if name else c


def listed():
    return [
        # the smallest systems: launches and latency are all there is
        _case("apply_2d_40x37_fp64", "apply", "diffusion", 40, 37, precision="fp64"),
        _case("step_2d_61x53_fp64", "step", "diffusion", 61, 53, precision="fp64"),
        # the benchmark's small compressing grid
        _case("step_2d_128x128_mixed", "step", "diffusion", 128, 128, sigma=0.0, eps=1e-10, **COMPRESSING),
        # a direct solve of an ordinary size: the largest grid below the default compression threshold
        _case("apply_2d_193x187_fp64", "apply", "diffusion", 193, 187, precision="fp64"),
        # a first call on a new matrix, from host arrays
        _case("new_2d_150x131_fp64", "new", "diffusion", 150, 131, precision="fp64"),
        # the default precision on an odd 3D grid
        _case("step_3d_37x41x35_fp64", "step", "diffusion", 37, 41, 35, precision="fp64"),
        # many solves on one factor, double precision, a few right-hand sides
        _case("solve8_3d_44x40x47_fp64", "solve", "diffusion", 44, 40, 47, precision="fp64", nrhs=8),
        # the headline workload: factor + PCG, 262,144 unknowns
        _case("step_3d_64x64x64_mixed", "step", "diffusion", 64, 64, 64),
        # vector unknowns: 3 per node, denser rows, many iterations
        _case("step_elasticity_30_mixed", "step", "elasticity", 30, sigma=0.0, rank_cap=64),
        # serving: a session with 40 right-hand sides arriving in requests of mixed widths
        _case("serve40_3d_40x40x40_mixed", "serve", "diffusion", 40, 40, 40, nrhs=40),
        # a wide block of right-hand sides on a large 2D grid with strong contrasts
        _case("solve64_2d_1024x1024_mixed", "solve", "diffusion", 1024, 1024, sigma=2.0, nrhs=64, eps=1e-10),
        # the largest system of the serving pool
        _case("step_3d_96x96x96_mixed", "step", "diffusion", 96, 96, 96),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """A case of the same ranges: any call, odd sizes, both precisions and their options."""
    call = rng.choice(["step", "step", "step", "solve", "solve", "apply", "serve", "new"])
    precision = rng.choice(["mixed", "mixed", "fp64"])
    opts = {}
    if call == "apply":
        return _case(None, call, "diffusion", _log(rng, 24, 195), _log(rng, 24, 195), sigma=round(rng.uniform(0, 1.5), 2),
                     precision="fp64", nrhs=rng.choice([1, 1, 1, 4, 16]))
    if call == "new":
        return _case(None, call, "diffusion", _log(rng, 40, 180), _log(rng, 40, 180), sigma=round(rng.uniform(0, 1.5), 2),
                     precision=precision)
    grid = rng.choice(["2d", "3d", "3d", "elasticity"])
    nrhs = {"step": 1, "solve": rng.choice([1, 1, 2, 5, 8, 16]), "serve": _log(rng, 6, 40)}[call]
    if precision == "mixed":
        if rng.random() < 0.1:
            opts["root_fp64"] = 1
        if rng.random() < 0.1:
            opts["schur_bf16"] = 1
    if grid == "2d":
        if rng.random() < 0.3:   # small and compressing, as c1
            s = _log(rng, 60, 200)
            return _case(None, call, "diffusion", s, max(40, int(s * rng.uniform(0.7, 1.0))), sigma=round(rng.uniform(0, 1), 2),
                         precision=precision, nrhs=nrhs, eps=1e-10, **COMPRESSING, **opts)
        s = _log(rng, 60, 900 if precision == "mixed" else 500)
        return _case(None, call, "diffusion", s, max(40, int(s * rng.uniform(0.6, 1.0))), sigma=round(rng.uniform(0, 2), 2),
                     precision=precision, nrhs=nrhs, eps=1e-10, **opts)
    if grid == "3d":
        s = _log(rng, 16, 72 if precision == "mixed" else 44)
        ny, nz = (max(12, int(s * rng.uniform(0.7, 1.1))) for _ in range(2))
        return _case(None, call, "diffusion", s, ny, nz, sigma=round(rng.uniform(0, 1.5), 2), precision=precision, nrhs=nrhs,
                     **opts)
    ne = _log(rng, 8, 28 if precision == "mixed" else 16)
    return _case(None, call, "elasticity", ne, sigma=0.0, precision=precision, nrhs=nrhs, rank_cap=64, **opts)


def _problem(case, seed):
    if case["grid"] == "elasticity":
        return rs.elasticity(case["nx"], seed=seed % 65521 + 1)
    dim = 3 if case["nz"] > 1 else 2
    return rs.diffusion(dim, case["nx"], case["ny"], case["nz"], sigma=case["sigma"], seed=seed % 65521 + 1)


def _rhs(case, n, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    return torch.randn(case["nrhs"], n, dtype=torch.float64, device="cuda", generator=g)


def _params(case):
    return {k[2:]: v for k, v in case.items() if k.startswith("p_")}


def prepare(case, seed):
    prob = _problem(case, seed)
    b = _rhs(case, prob.n, seed)
    s = dict(case=case, n=prob.n, nrhs=case["nrhs"])
    if case["call"] == "new":   # everything from host arrays
        s.update(prob=prob, b=b[0].cpu().numpy(), params=dict(_params(case), precision=case["precision"]))
        return s
    ctx = rs.Context(precision=case["precision"], **_params(case))
    s["ctx"] = ctx
    s["F"] = rs.GpuFactor(ctx, prob.colptr, prob.rowind, prob.vals, prob.xyz)
    if case["call"] == "serve":
        s["session"] = rs.Session(s["F"], 64)
        h, k, s["requests"] = b.cpu().numpy(), 0, []
        while k < case["nrhs"]:   # requests of 1, 2, 4, ... 8, 1, 2, ... right-hand sides
            w = min(case["nrhs"] - k, 1 << (len(s["requests"]) % 4))
            s["requests"].append(np.ascontiguousarray(h[k:k + w]))
            k += w
        return s
    s.update(vals=torch.from_numpy(prob.vals).cuda(), b=b, x=torch.zeros_like(b), infos=(rs.PcgInfo * case["nrhs"])())
    return s


def _check(status, ctx):
    if status != rs.RSCHOL_OK:
        raise rs.RscholError(status, ctx.last_error())


def run(state):
    case, lib = state["case"], rs.load_library()
    call = case["call"]
    if call == "new":
        prob, prm = state["prob"], state["params"]
        M = rs.FactorPreconditioner(**prm)
        M.initialize((prob.colptr, prob.rowind, prob.vals), prob.xyz)
        x = rs.PCGSolver(None, case["eps"]).solve_pcg(state["b"], M)
        M.factor.close()
        M.ctx.close()
        return x
    F, ctx = state["F"], state["ctx"]
    if call == "serve":   # two requests arrive before every iteration of the block
        ses, todo, xs = state["session"], list(enumerate(state["requests"])), {}
        while len(xs) < len(state["requests"]):
            for tag, b in todo[:2]:
                ses.add(tag, b, eps=case["eps"])
            todo = todo[2:]
            for tag, (st, x, _) in ses.step().items():
                _check(st, ctx)
                xs[tag] = x
        return [xs[t] for t in sorted(xs)]
    b, x = state["b"].data_ptr(), state["x"].data_ptr()
    if call == "apply":
        _check(lib.rschol_precond_apply_device(F.h, b, x, case["nrhs"]), ctx)
        return state["x"]
    if call == "step":
        _check(lib.rschol_refactor_device(F.h, state["vals"].data_ptr()), ctx)
    _check(lib.rschol_pcg_device(F.h, b, x, case["nrhs"], case["eps"], 10000, state["infos"]), ctx)
    return state["x"]


# --------------------------------------------------------------------------
# The solution in 64 bits: conjugate gradients with the diagonal as
# preconditioner, all right-hand sides together, until the residual stops
# falling near the rounding level.
def exact(case, seed):
    unknowns = case["nx"] * case["ny"] * case["nz"]
    if case["sigma"] > 1.0 and unknowns > 60000 or case["nz"] == 1 and unknowns > 300000 or unknowns * case["nrhs"] > 8000000:
        return None   # ten thousand iterations and more, or very wide
    prob = _problem(case, seed)
    A = torch.sparse_csr_tensor(torch.from_numpy(prob.colptr.astype(np.int64)), torch.from_numpy(prob.rowind.astype(np.int64)),
                                torch.from_numpy(prob.vals), size=(prob.n, prob.n), dtype=torch.float64).cuda()
    rows = np.repeat(np.arange(prob.n), np.diff(prob.colptr))
    dinv = torch.from_numpy(1.0 / prob.vals[rows == prob.rowind]).cuda()[:, None]
    b = _rhs(case, prob.n, seed).T.contiguous()
    x = torch.zeros_like(b)
    norm = b.norm(dim=0)
    for _ in range(4):   # restarted on the true residual
        r = b - A @ x
        if float((r.norm(dim=0) / norm).max()) < 1e-14:
            break
        z = dinv * r
        p, rz, goal = z.clone(), (r * z).sum(0), r.norm(dim=0) * 1e-7
        for it in range(20000):
            q = A @ p
            a = rz / (p * q).sum(0).clamp_min(1e-300)
            x += a * p
            r -= a * q
            if it % 25 == 24 and bool((r.norm(dim=0) <= goal).all()):
                break
            z = dinv * r
            rz, old = (r * z).sum(0), rz
            p = z + (rz / old.clamp_min(1e-300)) * p
    x = x.T.contiguous()
    if case["call"] == "new":
        return x[0]
    if case["call"] == "serve":
        out, k = [], 0
        while k < case["nrhs"]:
            w = min(case["nrhs"] - k, 1 << (len(out) % 4))
            out.append(x[k:k + w])
            k += w
        return out
    return x


# --------------------------------------------------------------------------
@functools.lru_cache(maxsize=None)
def _dissect(dims, faces, dof, dense, cap):
    """(factor entries, factor operations) of nested dissection of a box of
    grid points with ``faces`` sides on earlier separators: dense diagonal
    blocks, and off-diagonal blocks of the rank of the reference's rule for
    separators above ``dense`` columns."""
    n = math.prod(dims) * dof
    area = sum(n / d for d in dims if d > 1) / max(1, sum(d > 1 for d in dims))   # mean cross-section
    m = faces * area
    if n <= 64 or max(dims) < 3:
        return n * n / 2 + n * m, n ** 3 / 3 + n * n * m + n * m * m
    k = max(range(len(dims)), key=lambda i: dims[i])
    s = n / dims[k]
    if s > dense:
        r = min(max(16, int(0.4 * math.sqrt(s) * math.log2(s))) + 5, s, cap or s)
        entries, ops = s * s / 2 + r * (s + m), s ** 3 / 3 + 2 * r * s * (s + m)
    else:
        entries, ops = s * s / 2 + s * m, s ** 3 / 3 + s * s * m + s * m * m
    for part in ((dims[k] - 1) // 2, dims[k] - 1 - (dims[k] - 1) // 2):
        sub = list(dims)
        sub[k] = part
        e, o = _dissect(tuple(sorted(sub)), min(faces + 1, 6 if dims[0] > 1 else 4), dof, dense, cap)
        entries, ops = entries + e, ops + o
    return entries, ops


def work(case):
    """The factor read twice (forward, backward) in every application, the
    matrix and four vectors in every iteration, the values and the factor
    written once by a factorisation; iterations as these problems take."""
    el = case["grid"] == "elasticity"
    dims = tuple(sorted([case["nx"] + 1] * 3 if el else [case["nx"], case["ny"], case["nz"]]))
    dof, dim = (3, 3) if el else (1, 3 if case["nz"] > 1 else 2)
    n = math.prod(dims) * dof
    nnz = n * (81 if el else 2 * dim + 1)
    entries, ops = _dissect(dims, 0, dof, case.get("p_max_dense_block", 200), case.get("p_rank_cap", 0))
    size, k = (8 if case["precision"] == "fp64" else 4), case["nrhs"]
    its = 1 if case["call"] == "apply" else 50 if el else 16 if dim == 3 else 3
    bytes_, flops = 16.0 * n * k, 0.0
    if case["call"] in ("step", "new"):
        bytes_ += 8.0 * nnz + size * entries
        flops += ops
    bytes_ += its * (2 * size * entries + 12.0 * nnz * (case["call"] != "apply") + 32.0 * n * k)
    flops += its * k * (4.0 * entries + 2.0 * nnz + 10.0 * n)
    return {"bytes": bytes_, "flops": flops}

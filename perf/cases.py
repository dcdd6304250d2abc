"""Performance cases of the ILU(k) + GMRES framework: the work its users have it do, each
through the public entry points, over the range of matrices, options and value types that
the tests and the benchmark use.

Kinds of a case:

* ``apply``   one preconditioner application x = U^-1 L^-1 b on device vectors (FP64);
* ``factor``  new matrix values on a known pattern: numeric factorisation (optionally with
              the learned diagonal shift), then one application of the new factors;
* ``solve``   one GMRES solve to the tolerance with factors in hand;
* ``step``    new matrix values: factorisation and solve (one step of an outer iteration);
* ``batch``   many small systems with several right-hand sides, one launch, host vectors;
* ``train``   one optimiser step of the learned-shift network.

Matrices (natural order, x fastest): ``pt5`` / ``pt7`` variable-coefficient upwind
convection-diffusion on a full box, ``pt27`` the 27-point operator, ``holes`` the 7-point
operator on a box with cells cut out (an irregular domain: no full stencil).
"""
from __future__ import annotations

import ctypes
import functools
import math

import numpy as np
import torch

from par_ilu0_cpp_gb300 import api, learned_shift
from par_ilu0_cpp_gb300.generators import Csr

RTOL = 1e-8
MAXIT = 1000
WIND = (1.0, 0.5, 0.25)


# --------------------------------------------------------------------------------------
# Cases
# --------------------------------------------------------------------------------------
def listed():
    return [
        # the smallest call: a coarse 2-D level, where launches and latency count
        dict(name="apply_2d_small", kind="apply", matrix="pt5", nx=63, ny=65, nz=1, lof=0),
        # an application on the benchmark's 3-D grid (what a Krylov method of the user's
        # own does once per iteration)
        dict(name="apply_3d_128", kind="apply", matrix="pt7", nx=128, ny=128, nz=128, lof=0),
        # a nonlinear or time-dependent 3-D run: new coefficients every step, ragged grid
        dict(name="factor_3d", kind="factor", matrix="pt7", nx=101, ny=90, nz=75, lof=0, learned=False),
        # the densest factors of the test set: 27-point ILU(2), ragged grid
        dict(name="factor_27pt_ilu2", kind="factor", matrix="pt27", nx=30, ny=27, nz=25, lof=2, learned=False),
        # the learned diagonal shift inferred in the factorisation (2-D, as it was trained)
        dict(name="factor_2d_learned", kind="factor", matrix="pt5", nx=384, ny=301, nz=1, lof=0, learned=True),
        # a small solve on an irregular domain, FP64 throughout, on host arrays as the
        # drop-in C interface has it
        dict(name="solve_holes_small", kind="solve", matrix="holes", nx=21, ny=20, nz=19, lof=0, mode=0, restart=30,
             host=True),
        # the 2-D benchmark configuration, FP64 throughout
        dict(name="solve_2d_256", kind="solve", matrix="pt5", nx=256, ny=256, nz=1, lof=0, mode=0, restart=30),
        # a mid-size 3-D solve, FP64 throughout
        dict(name="solve_3d_plain", kind="solve", matrix="pt7", nx=100, ny=96, nz=90, lof=0, mode=0, restart=50),
        # the headline: factorisation and mixed-precision solve on the benchmark's 3-D grid
        dict(name="step_3d_128_mixed", kind="step", matrix="pt7", nx=128, ny=128, nz=128, lof=0, mode=1, restart=50),
        # the 27-point configuration with fill, mixed precision
        dict(name="solve_27pt_ilu1_mixed", kind="solve", matrix="pt27", nx=44, ny=40, nz=42, lof=1, mode=1, restart=30),
        # many systems of uneven size with several right-hand sides
        dict(name="batch", kind="batch", systems=128, side_lo=32, side_hi=128, nrhs=4, restart=30),
        # training of the learned shift at its configured batch size
        dict(name="train_step", kind="train", samples=500000, batch=65536),
    ]


def draw(rng):
    def log_int(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["apply", "apply", "factor", "factor", "solve", "solve", "solve", "step", "batch", "train"])
    if kind == "batch":
        lo = rng.randint(16, 48)
        return dict(kind=kind, systems=log_int(8, 128), side_lo=lo, side_hi=rng.randint(lo + 8, 112),
                    nrhs=rng.choice([1, 2, 3, 4]), restart=rng.choice([20, 30, 40]))
    if kind == "train":
        batch = log_int(4096, 65536)
        return dict(kind=kind, samples=log_int(batch, 500000), batch=batch)
    matrix = rng.choice(["pt5", "pt7", "pt7", "pt27", "holes"])
    lof = rng.choice([0, 1, 2]) if matrix == "pt27" else 0
    if matrix == "pt5":
        nx, ny, nz = log_int(40, 400), log_int(40, 400), 1
    elif matrix == "pt27":
        nx, ny, nz = rng.randint(12, 30), rng.randint(12, 30), rng.randint(12, 30)
    else:
        hi = 110 if kind in ("apply", "factor") else 80
        hi = min(hi, 64) if matrix == "holes" else hi
        nx, ny, nz = log_int(12, hi), log_int(12, hi), log_int(12, hi)
    c = dict(kind=kind, matrix=matrix, nx=nx, ny=ny, nz=nz, lof=lof)
    if kind == "factor":
        c["learned"] = matrix == "pt5" and rng.random() < 0.5
    if kind in ("solve", "step"):
        c["mode"] = rng.choice([0, 1])
        c["restart"] = rng.choice([30, 40, 50])
        c["host"] = kind == "solve" and rng.random() < 0.3
    return c


# --------------------------------------------------------------------------------------
# Matrices
# --------------------------------------------------------------------------------------
def _field(nx, ny, nz, sigma, rng):
    """exp(sigma g), g a smooth unit-variance random field (a few cosine modes)."""
    modes = 12
    k = rng.uniform(0.5, 4.0, size=(modes, 3)) * 2.0 * np.pi
    ph = rng.uniform(0.0, 2.0 * np.pi, size=modes)
    x, y, z = (torch.arange(m, device="cuda", dtype=torch.float64) / max(m, 32) for m in (nx, ny, nz))
    g = torch.zeros(nz, ny, nx, device="cuda", dtype=torch.float64)
    for (kx, ky, kz), p in zip(k, ph):
        g += torch.cos(float(kz) * z[:, None, None] + float(ky) * y[None, :, None] + float(kx) * x[None, None, :] + float(p))
    return torch.exp(sigma * g * math.sqrt(2.0 / modes))


@functools.lru_cache(maxsize=16)
def _holes(nx, ny, nz):
    """Active cells of a box with a few balls cut out (fixed by the box's sides)."""
    rng = np.random.default_rng(nx * 1000003 + ny * 1009 + nz)
    z, y, x = np.meshgrid(np.arange(nz), np.arange(ny), np.arange(nx), indexing="ij")
    keep = np.ones((nz, ny, nx), dtype=bool)
    for _ in range(5):
        c = rng.uniform(0.0, 1.0, 3) * (nx, ny, nz)
        r = rng.uniform(0.08, 0.2) * min(nx, ny, nz)
        keep &= (x - c[0]) ** 2 + (y - c[1]) ** 2 + (z - c[2]) ** 2 > r * r
    return torch.from_numpy(keep).cuda()


def _offsets(matrix):
    if matrix == "pt27":
        return [(dx, dy, dz) for dz in (-1, 0, 1) for dy in (-1, 0, 1) for dx in (-1, 0, 1)]
    o = [(0, 0, -1), (0, -1, 0), (-1, 0, 0), (0, 0, 0), (1, 0, 0), (0, 1, 0), (0, 0, 1)]
    return [d for d in o if d[2] == 0] if matrix == "pt5" else o


def _matrix(case, rng):
    """(row_ptr, col_idx, values) of the case's matrix, on the device (int32, int32, float64),
    and the product A x as a function."""
    m, nx, ny, nz = case["matrix"], case["nx"], case["ny"], case["nz"]
    k = _field(nx, ny, nz, 1.0 if m == "pt27" else 0.5, rng)
    peclet = rng.uniform(0.3, 0.5)
    keep = _holes(nx, ny, nz) if m == "holes" else torch.ones(nz, ny, nx, dtype=torch.bool, device="cuda")
    index = torch.where(keep, torch.cumsum(keep.reshape(-1).long(), 0).reshape(keep.shape) - 1, -1)
    pad = lambda t, v: torch.nn.functional.pad(t, (1, 1, 1, 1, 1, 1), value=v)  # noqa: E731
    kp, ip = pad(k, 0.0), pad(index, -1)
    offs = _offsets(m)
    cols, vals = [], []
    diag = torch.full_like(k, 1e-3 if m == "pt27" else 0.0)
    for dx, dy, dz in offs:
        sl = (slice(1 + dz, 1 + dz + nz), slice(1 + dy, 1 + dy + ny), slice(1 + dx, 1 + dx + nx))
        q, kq = ip[sl], kp[sl]
        cols.append(q)
        if (dx, dy, dz) == (0, 0, 0):
            vals.append(None)
            continue
        if m == "pt27":
            coef = torch.where(q >= 0, 2.0 * k * kq / (k + kq) / float(dx * dx + dy * dy + dz * dz), torch.zeros_like(k))
            diag += coef
        else:  # Dirichlet walls: a face without a neighbour still adds to the diagonal
            coef = torch.where(q >= 0, 2.0 * k * kq / (k + kq), k)
            diag += coef
            w = WIND[0] * abs(dx) + WIND[1] * abs(dy) + WIND[2] * abs(dz)
            if dx + dy + dz < 0:  # first-order upwind, wind along +x, +y, +z
                coef = coef + 2.0 * peclet * w
                diag += 2.0 * peclet * w
        vals.append(-coef)
    vals = [diag if v is None else v for v in vals]
    cols = torch.stack([c.reshape(-1) for c in cols], 1)[keep.reshape(-1)]
    vals = torch.stack([v.reshape(-1) for v in vals], 1)[keep.reshape(-1)]
    here = cols >= 0
    row_ptr = torch.zeros(cols.shape[0] + 1, dtype=torch.int64, device="cuda")
    row_ptr[1:] = torch.cumsum(here.sum(1), 0)
    matvec = lambda x: torch.where(here, vals * x[cols.clamp(min=0)], 0.0).sum(1)  # noqa: E731
    return row_ptr.int(), cols[here].int(), vals[here].contiguous(), matvec


@functools.lru_cache(maxsize=4)
def _fill_pattern(matrix, nx, ny, nz, lof):
    """ILU(k) pattern and value map (fixed by the grid: a program computes it once)."""
    case = dict(matrix=matrix, nx=nx, ny=ny, nz=nz)
    rp, ci, v, _ = _matrix(case, np.random.default_rng(0))
    f, nzmap = api.iluk_symbolic(Csr(rp.numel() - 1, rp.cpu().numpy(), ci.cpu().numpy(), v.cpu().numpy()), lof)
    return f, torch.from_numpy(nzmap).cuda().long()


def _system(case, seed):
    """Matrix, known solution and right-hand side of a case, from the seed alone."""
    rng = np.random.default_rng(seed)
    rp, ci, v, matvec = _matrix(case, rng)
    x_true = torch.from_numpy(rng.uniform(-1.0, 1.0, rp.numel() - 1)).cuda()
    return rp, ci, v, x_true, matvec(x_true)


def _batch_inputs(case, seed):
    sides = np.random.default_rng(case["systems"]).integers(case["side_lo"], case["side_hi"] + 1, size=case["systems"])
    rng = np.random.default_rng(seed)
    systems, xs, bs = [], [], []
    for s in sides:
        rp, ci, v, matvec = _matrix(dict(matrix="pt5", nx=int(s), ny=int(s), nz=1), rng)
        x = torch.from_numpy(rng.uniform(-1.0, 1.0, (case["nrhs"], rp.numel() - 1))).cuda()
        bs.append(torch.stack([matvec(xi) for xi in x]).reshape(-1).cpu().numpy())
        xs.append(x.reshape(-1).cpu().numpy())
        systems.append(Csr(rp.numel() - 1, rp.cpu().numpy(), ci.cpu().numpy(), v.cpu().numpy()))
    return systems, np.concatenate(xs), np.concatenate(bs)


def _train_inputs(case, seed):
    """Features with the spread the pre-pass gives on 2-D operators, smooth targets."""
    rng = np.random.default_rng(seed)
    n = case["samples"]
    X = np.empty((n, 4), dtype=np.float32)
    X[:, 0] = rng.normal(-0.3, 0.8, n)
    X[:, 1] = X[:, 0] - rng.uniform(0.3, 1.0, n)
    X[:, 2] = np.clip(rng.normal(1.0, 0.2, n), 0.0, 4.0)
    X[:, 3] = rng.uniform(0.0, 1.0, n)
    T = (np.maximum(0.0, 1.0 - X[:, 2]) + 0.05 * (X[:, 3] > 0.5)).astype(np.float32)
    p = rng.uniform(-0.5, 0.5, 369).astype(np.float32)  # a network in the middle of its training
    return X, T, rng.permutation(n)[: case["batch"]].astype(np.int32), p


# --------------------------------------------------------------------------------------
# The program around a pass
# --------------------------------------------------------------------------------------
def prepare(case, seed):
    kind = case["kind"]
    if kind == "batch":
        systems, _, b = _batch_inputs(case, seed)
        solver = api.BatchSolver(systems, case["nrhs"], restart=case["restart"], rtol=RTOL, maxit=MAXIT)
        solver.set_shape(2, True, 4 if case["nrhs"] > 1 else 1)
        return dict(kind=kind, solver=solver, b=b)
    if kind == "train":
        X, T, idx, params = _train_inputs(case, seed)
        trainer = api.ShiftTrainer()
        trainer.params = params
        trainer.set_data(X, T)
        return dict(kind=kind, trainer=trainer, idx=idx)
    rp, ci, v, _, b = _system(case, seed)
    n = rp.numel() - 1
    if case["lof"] == 0:
        f, fv = Csr(n, rp.cpu().numpy(), ci.cpu().numpy(), v.cpu().numpy()), v
    else:
        f, nzmap = _fill_pattern(case["matrix"], case["nx"], case["ny"], case["nz"], case["lof"])
        fv = torch.zeros(f.nnz, dtype=torch.float64, device="cuda")
        fv[nzmap] = v
        f = Csr(n, f.row_ptr, f.col_idx, fv.cpu().numpy())
    ilu = api.IluSolver()
    ilu.set_matrix(f)
    if ilu.setup() != 0:
        raise RuntimeError(api.last_error())
    if case.get("learned"):
        params, meta = learned_shift.load_model()
        ilu.set_shift_model(params, meta.get("min_shift", 0.0))
    st = dict(kind=kind, ilu=ilu, n=n, fv=fv, b=b, x=torch.zeros(n, dtype=torch.float64, device="cuda"))
    torch.cuda.current_stream().synchronize()
    if ilu.factorize_device(fv.data_ptr()) != 0:
        raise RuntimeError(api.last_error())
    if kind in ("solve", "step"):
        gm = api.Gmres(RTOL * float(torch.linalg.norm(b)), case["restart"], MAXIT)
        gm.set_preconditioner(ilu)
        gm.set_option(api.GMRES_OPT_MODE, case["mode"])
        st.update(gm=gm, rp=rp, ci=ci, av=v)
        if case.get("host"):
            st.update(a=Csr(n, rp.cpu().numpy(), ci.cpu().numpy(), v.cpu().numpy()), b_host=b.cpu().numpy())
    return st


def _apply(st):
    rc = st["ilu"].lib.LLJBASH_IluSolverSubstituteDeviceNoAlloc(
        st["ilu"].h, ctypes.c_void_p(st["b"].data_ptr()), ctypes.c_void_p(st["x"].data_ptr()))
    if rc != 0:
        raise RuntimeError(api.last_error())
    return st["x"]


def run(st):
    kind = st["kind"]
    if kind == "batch":
        out = st["solver"].solve(st["b"])
        return dict(x=out["x"], converged=out["converged"].astype(np.int32))
    if kind == "train":
        loss = st["trainer"].step(st["idx"], 3e-3)
        return dict(loss=loss, params=st["trainer"].params)
    if kind != "solve" and kind != "apply" and st["ilu"].factorize_device(st["fv"].data_ptr()) != 0:
        raise RuntimeError(api.last_error())
    if kind in ("apply", "factor"):
        return dict(x=_apply(st))
    if "a" in st:
        res = st["gm"].solve(st["a"], st["b_host"])
        return dict(x=res.x, ok=int(res.ok))
    st["x"].zero_()
    torch.cuda.current_stream().synchronize()  # operands are ready when the solve is called
    ok, _ = st["gm"].solve_device(st["n"], st["rp"].data_ptr(), st["ci"].data_ptr(), st["av"].data_ptr(),
                                  st["b"].data_ptr(), st["x"].data_ptr())
    return dict(x=st["x"], ok=int(ok))


# --------------------------------------------------------------------------------------
# What a pass cannot do without, and what it gives in exact arithmetic
# --------------------------------------------------------------------------------------
def _cells(case):
    n = case["nx"] * case["ny"] * case["nz"]
    return int(n * 0.9) if case["matrix"] == "holes" else n


def work(case):
    kind = case["kind"]
    if kind == "batch":
        mean = (case["side_lo"] ** 2 + case["side_lo"] * case["side_hi"] + case["side_hi"] ** 2) / 3.0
        rows = case["systems"] * mean
        return {"bytes": rows * (5 * 12 + 16 * case["nrhs"]), "flops": rows * (2 * 5 * case["nrhs"])}
    if kind == "train":
        return {"bytes": case["batch"] * 24.0 + 369 * 16.0, "flops": case["batch"] * 6.0 * 352}
    n = _cells(case)
    entries = {"pt5": 5, "pt7": 7, "holes": 7, "pt27": 27}[case["matrix"]]
    fill = entries * {0: 1.0, 1: 2.2, 2: 3.4}[case["lof"]]  # stored entries per factor row
    factors, vectors = n * fill * 12.0, n * 16.0
    if kind == "apply":
        return {"bytes": factors + vectors, "flops": 2.0 * n * fill}
    if kind == "factor":  # values in, factors out, factors in again for the application
        return {"bytes": 2 * factors + n * fill * 8.0 + vectors, "flops": n * (2.0 * fill + fill * fill / 4.0)}
    a = n * entries * 12.0
    extra = n * fill * 8.0 if kind == "step" else 0.0
    return {"bytes": a + factors + extra + vectors, "flops": 2.0 * n * (fill + entries)}


def _ilu0_apply(case, v, rp, shift, b):
    """x = U^-1 L^-1 b for the ILU(0) factors of a full 5- / 7-point stencil, in FP64 by
    wavefronts x + y + z = const (there the elimination changes only the diagonal:
    d_i = a_ii - sum over lower neighbours j of (a_ij / d_j) a_ji)."""
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    n = nx * ny * nz
    offs = _offsets(case["matrix"])
    i = torch.arange(n, device="cuda")
    x, y, z = i % nx, (i // nx) % ny, i // (nx * ny)
    coef, nbr, p = [], [], rp[:-1].long()
    for dx, dy, dz in offs:
        ok = (x + dx >= 0) & (x + dx < nx) & (y + dy >= 0) & (y + dy < ny) & (z + dz >= 0) & (z + dz < nz)
        coef.append(torch.where(ok, v[torch.clamp(p, max=v.numel() - 1)], torch.zeros_like(b)))
        nbr.append(torch.where(ok, i + dx + nx * (dy + ny * dz), i))
        p = p + ok.long()
    c, nb = torch.stack(coef), torch.stack(nbr)
    h = len(offs) // 2
    d = c[h] + shift if shift is not None else c[h].clone()
    level = x + y + z
    order = torch.argsort(level, stable=True)
    bounds = [0] + torch.cumsum(torch.bincount(level), 0).tolist()
    sol = b.clone()
    planes = [order[a:e] for a, e in zip(bounds[:-1], bounds[1:])]
    for r in planes:
        dr, sr = d[r], sol[r]
        for t in range(h):
            l = c[t][r] / d[nb[t][r]]  # 0 where there is no neighbour
            dr = dr - l * c[2 * h - t][nb[t][r]]
            sr = sr - l * sol[nb[t][r]]
        d[r], sol[r] = dr, sr
    for r in reversed(planes):
        sr = sol[r]
        for t in range(2 * h, h, -1):
            sr = sr - c[t][r] * sol[nb[t][r]]
        sol[r] = sr / d[r]
    return sol


def _learned_shift(case, rp, ci, v):
    """The learned shift's features and network in FP64 (a model's parameters are FP32)."""
    params, meta = learned_shift.load_model()
    w = torch.from_numpy(np.asarray(params, dtype=np.float64)).cuda()
    n = rp.numel() - 1
    rows = torch.repeat_interleave(torch.arange(n, device="cuda"), (rp[1:] - rp[:-1]).long())
    off = ci.long() != rows
    a = torch.zeros(n, dtype=torch.float64, device="cuda").index_add_(0, rows[~off], v[~off])
    s1 = torch.zeros_like(a).index_add_(0, rows[off], v[off].abs())
    s2 = torch.zeros_like(a).index_add_(0, rows[off], v[off] ** 2).sqrt()
    md = a.abs().mean()
    i = torch.arange(n, device="cuda")
    depth = (i % case["nx"] + i // case["nx"]).double() / (case["nx"] + case["ny"] - 2)
    X = torch.stack([torch.log(a.abs() / md), torch.log(s2 / md), torch.clamp(a.abs() / s1, max=4.0), depth], 1)
    h1 = torch.tanh(X @ w[:64].reshape(16, 4).T + w[64:80])
    h2 = torch.tanh(h1 @ w[80:336].reshape(16, 16).T + w[336:352])
    y = torch.nn.functional.softplus(h2 @ w[352:368] + w[368])
    return torch.where(y >= meta.get("min_shift", 0.0), torch.sign(a) * y * s1, torch.zeros_like(a))


def _train_exact(case, seed):
    X, T, idx, params = _train_inputs(case, seed)
    w = torch.from_numpy(params.astype(np.float64)).requires_grad_()
    X, T = torch.from_numpy(X[idx].astype(np.float64)), torch.from_numpy(T[idx].astype(np.float64))
    h1 = torch.tanh(X @ w[:64].reshape(16, 4).T + w[64:80])
    h2 = torch.tanh(h1 @ w[80:336].reshape(16, 16).T + w[336:352])
    loss = ((torch.nn.functional.softplus(h2 @ w[352:368] + w[368]) - T) ** 2).mean()
    loss.backward()
    g = w.grad  # first Adam step: m / (1 - b1) = g, v / (1 - b2) = g^2
    return dict(loss=float(loss.detach()), params=(w.detach() - 3e-3 * g / (g.abs() + 1e-8)).numpy())


def exact(case, seed):
    kind = case["kind"]
    if kind == "batch":
        return dict(x=_batch_inputs(case, seed)[1], converged=None)
    if kind == "train":
        return _train_exact(case, seed)
    rp, ci, v, x_true, b = _system(case, seed)
    if kind in ("solve", "step"):
        return dict(x=x_true, ok=None)
    if case["matrix"] not in ("pt5", "pt7"):
        return None  # a general elimination with fill takes minutes without a library
    shift = _learned_shift(case, rp, ci, v) if case.get("learned") else None
    return dict(x=_ilu0_apply(case, v, rp, shift, b))

"""The workloads this framework's speed is judged on: one pass each through the public entry points.

Every case is what a program that calls the framework does again and again: solve a dense or sparse
SPD system, apply a matrix function, find leading eigenpairs, take a Gaussian-process gradient step,
or solve a family of systems.  Sizes follow the repository's configurations, tests and benchmark;
the inputs are synthetic with the spectra and structure those problems have.  FP32 problems have
condition numbers (1e2 .. 1e3) that single precision resolves, and solves refined in FP64 go to
1e-11, the tolerance of the parity tests, so that outputs can be compared closely.

    listed()         the cases by name
    draw(rng)        one more case of the same ranges
    prepare(c, seed) inputs, operators and weights as a program would hold them before the call
    run(state)       one pass, all of its outputs
    work(c)          bytes (inputs once, outputs once) and operations of one pass
    exact(c, seed)   the same outputs in 64-bit torch
"""
import math

import torch

import cola_gb300 as cola
from cola_gb300.linalg import BatchedCSR, CG, Lanczos, cg, solve_batched, solve_dense_batched, stochastic_lanczos_quad
from cola_gb300.linalg.batched import FsaiPattern
from cola_gb300.precond import learned_fsai

DEV = "cuda"
_DT = {"float32": torch.float32, "float64": torch.float64, "bfloat16": torch.bfloat16}


def listed():
    return [
        # the smallest calls: a few hundred unknowns in double precision, where latency is everything
        {"name": "dense-cg-200-f64", "kind": "dense_cg", "n": 200, "k": 1, "dtype": "float64", "lo": 1e-1, "hi": 1e1,
         "jacobi": False, "tol": 1e-11},
        # the dense 2048 x 2048 FP32 solve, one right-hand side
        {"name": "dense-cg-2048", "kind": "dense_cg", "n": 2048, "k": 1, "dtype": "float32", "lo": 1e-1, "hi": 1e2,
         "jacobi": False, "tol": 1e-6},
        # BF16 storage, an odd size and a few right-hand sides with a diagonal preconditioner
        {"name": "dense-cg-3001x3-bf16", "kind": "dense_cg", "n": 3001, "k": 3, "dtype": "bfloat16", "lo": 1e-1,
         "hi": 1e1, "jacobi": True, "tol": 1e-6},
        # a block of right-hand sides at once (predictive variances, probe solves)
        {"name": "dense-cg-4096x32", "kind": "dense_cg", "n": 4096, "k": 32, "dtype": "float32", "lo": 1e-1, "hi": 1e1,
         "jacobi": False, "tol": 1e-6},
        # one FP64 diffusion solve with Jacobi through the reference's solve() call
        {"name": "sparse-cg-256x256-f64", "kind": "sparse_cg", "m": 256, "dtype": "float64", "shift": 0.0,
         "tol": 1e-12},
        # Gaussian process on a grid: Kronecker kernel plus noise, the general operator loop
        {"name": "kron-cg-96x80", "kind": "kron_cg", "m1": 96, "m2": 80, "m3": 0, "k": 8, "dtype": "float32",
         "noise": 1.0, "tol": 1e-6},
        # log-determinant quadratic forms of a block of Rademacher probes: batched Lanczos, three factors
        {"name": "kron-slq-48^3x16", "kind": "kron_fun", "m1": 48, "m2": 48, "m3": 48, "k": 16, "steps": 40,
         "fun": "log", "dtype": "float32", "noise": 1.0},
        # leading eigenpairs of Kronecker + graph Laplacian (512^2 unknowns)
        {"name": "eig-kron512+laplacian", "kind": "eig", "m1": 512, "m2": 512, "k": 8, "steps": 96},
        # a marginal-likelihood step: solve, log-determinant and both backward passes
        {"name": "gp-grad-1500", "kind": "gp_grad", "n": 1500, "k": 16, "steps": 40, "noise": 0.5},
        # the headline family: learned factor build and the batched solve, 512 x 512 grids
        {"name": "family-512x512x16", "kind": "family", "m": 512, "systems": 16, "precond": "learned"},
        # dense systems of uneven sizes in one launch
        {"name": "uneven-dense-24", "kind": "uneven", "systems": 24, "n_lo": 300, "n_hi": 3000},
        # many right-hand sides of one 3-D diffusion matrix
        {"name": "diffusion3d-64^3x16", "kind": "block3d", "m": 64, "k": 16},
    ]


def _loguni(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["dense_cg", "dense_cg", "dense_cg", "sparse_cg", "kron_cg", "kron_fun", "eig", "gp_grad", "family",
                       "uneven", "block3d"])
    if kind == "dense_cg":
        dtype = rng.choice(["float32", "float32", "float64", "bfloat16"])
        k = rng.choice([1, 1, 1, rng.randint(2, 8), rng.randint(9, 48)])
        top = 6000 if k == 1 else 4000
        if dtype == "float64":
            top = 3000 if k <= 8 else 1200
        return {"kind": kind, "n": _loguni(rng, 64, top), "k": k, "dtype": dtype, "lo": 1e-1,
                "hi": rng.choice([1e1, 1e2]) if dtype != "bfloat16" else 1e1, "jacobi": rng.random() < 0.3,
                "tol": 1e-11 if dtype == "float64" else 1e-6}
    if kind == "sparse_cg":
        dtype = rng.choice(["float64", "float32"])
        return {"kind": kind, "m": _loguni(rng, 24, 300), "dtype": dtype, "shift": 0.0 if dtype == "float64" else 0.5,
                "tol": 1e-12 if dtype == "float64" else 1e-6}
    if kind == "kron_cg":
        dtype = rng.choice(["float32", "float32", "float64"])
        three = rng.random() < 0.3
        hi = 28 if three else 128
        return {"kind": kind, "m1": rng.randint(12, hi), "m2": rng.randint(12, hi), "m3": rng.randint(8, 24) if three else 0,
                "k": rng.choice([1, 1, rng.randint(2, 16)]), "dtype": dtype, "noise": round(rng.uniform(0.7, 2.0), 3),
                "tol": 1e-11 if dtype == "float64" else 1e-6}
    if kind == "kron_fun":
        dtype = rng.choice(["float32", "float32", "float64"])  # FP64: the matrix function times the probes
        return {"kind": kind, "m1": rng.randint(12, 48), "m2": rng.randint(12, 48),
                "m3": rng.choice([0, rng.randint(8, 48 if dtype == "float32" else 20)]),
                "k": rng.choice([1, 4, rng.randint(2, 16), 16]), "steps": rng.randint(20, 40),
                "fun": rng.choice(["sqrt", "log"]), "dtype": dtype, "noise": round(rng.uniform(0.7, 2.0), 3)}
    if kind == "eig":
        return {"kind": kind, "m1": _loguni(rng, 48, 512), "m2": _loguni(rng, 48, 512), "k": rng.randint(3, 8),
                "steps": rng.randint(72, 96)}
    if kind == "gp_grad":
        return {"kind": kind, "n": _loguni(rng, 200, 2500), "k": rng.randint(4, 24), "steps": rng.randint(25, 40),
                "noise": round(rng.uniform(0.5, 1.5), 3)}
    if kind == "family":
        m = 2 * _loguni(rng, 16, 190)
        return {"kind": kind, "m": m, "systems": rng.randint(2, 24), "precond": rng.choice(["learned", "learned", "jacobi"])}
    if kind == "uneven":
        return {"kind": kind, "systems": rng.randint(2, 24), "n_lo": rng.randint(64, 300), "n_hi": rng.randint(400, 2800)}
    return {"kind": kind, "m": 2 * rng.randint(6, 32), "k": rng.randint(4, 16)}


# ---- inputs -----------------------------------------------------------------------------------------


def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(int(seed))


def _rand(g, *shape, dtype=torch.float64):
    return torch.rand(*shape, generator=g, device=DEV, dtype=dtype)


def _randn(g, *shape, dtype=torch.float64):
    return torch.randn(*shape, generator=g, device=DEV, dtype=dtype)


def _spd(n, lo, hi, g):
    """Q diag(lam) Q^T with lam log-uniform in [lo, hi]."""
    Q, _ = torch.linalg.qr(_randn(g, n, n, dtype=torch.float32))
    lam = torch.exp(_rand(g, n, dtype=torch.float32) * math.log(hi / lo) + math.log(lo))
    A = (Q * lam) @ Q.T
    return 0.5 * (A + A.T)


def _grid2d(m):
    """CSR pattern of the 5-point stencil, and which of the five neighbours exist."""
    p = torch.arange(m * m, device=DEV)
    i, j = p // m, p % m
    ok = torch.stack([i > 0, j > 0, torch.ones_like(i, dtype=torch.bool), j < m - 1, i < m - 1], 1)
    cols = torch.stack([p - m, p - 1, p, p + 1, p + m], 1)
    indptr = torch.zeros(m * m + 1, dtype=torch.int64, device=DEV)
    indptr[1:] = torch.cumsum(ok.sum(1), 0)
    return indptr.to(torch.int32), cols[ok].to(torch.int32), ok


def _diffusion2d(m, systems, g):
    """FP64 values (systems, nnz) of finite-volume diffusion with harmonic-mean faces and Dirichlet
    walls, cell coefficients the exponential of a smooth random field of variance about 1."""
    k = torch.fft.fftfreq(2 * m, d=1.0 / m, device=DEV, dtype=torch.float64)
    filt = (3.0 / 0.12 ** 2 + 4 * math.pi ** 2 * (k[:, None] ** 2 + k[None, :] ** 2)) ** -1.25
    indptr, indices, ok = _grid2d(m)
    vals = torch.empty(systems, indices.numel(), dtype=torch.float64, device=DEV)
    for s in range(systems):
        f = torch.fft.ifft2(torch.fft.fft2(_randn(g, 2 * m, 2 * m)) * (filt / filt.square().mean().sqrt())).real
        a = torch.exp(f[:m, :m])
        face = 2 * a[1:] * a[:-1] / (a[1:] + a[:-1])
        tN, tS = torch.cat([2 * a[:1], face]), torch.cat([face, 2 * a[-1:]])
        face = 2 * a[:, 1:] * a[:, :-1] / (a[:, 1:] + a[:, :-1])
        tW, tE = torch.cat([2 * a[:, :1], face], 1), torch.cat([face, 2 * a[:, -1:]], 1)
        vals[s] = torch.stack([-tN, -tW, tN + tS + tW + tE, -tE, -tS], -1).reshape(m * m, 5)[ok]
    return indptr, indices, vals


def _diffusion3d(m, g):
    """CSR of the 7-point variable-coefficient diffusion on m^3 cells plus 1e-3 I (FP32 values)."""
    n = m ** 3
    a = torch.exp(_randn(g, n))
    p = torch.arange(n, device=DEV)
    z, y, x = p // (m * m), (p // m) % m, p % m
    diag = torch.full((n,), 1e-3, dtype=torch.float64, device=DEV)
    cols, vals, oks = [], [], []
    for off, valid in ((-m * m, z > 0), (-m, y > 0), (-1, x > 0), (0, None), (1, x < m - 1), (m, y < m - 1), (m * m, z < m - 1)):
        if off == 0:
            cols.append(p), vals.append(diag), oks.append(torch.ones_like(p, dtype=torch.bool))
            continue
        nb = a[(p + off).clamp(0, n - 1)]
        t = torch.where(valid, 2 * a * nb / (a + nb), 2 * a)
        diag += t
        cols.append(p + off), vals.append(-t), oks.append(valid)
    ok = torch.stack(oks, 1)
    indptr = torch.zeros(n + 1, dtype=torch.int64, device=DEV)
    indptr[1:] = torch.cumsum(ok.sum(1), 0)
    return indptr.to(torch.int32), torch.stack(cols, 1)[ok].to(torch.int32), torch.stack(vals, 1)[ok].float()


def _rbf_grid(m, ell):
    x = torch.linspace(0, 1, m, dtype=torch.float64, device=DEV)
    return torch.exp(-((x[:, None] - x[None, :]) ** 2) / (2 * ell * ell))


def _rbf_points(n, dim, ell, g):
    pts = _rand(g, n, dim)
    return torch.exp(-torch.cdist(pts, pts).square() / (2 * ell * ell))


def _kron_factors(c, g):
    """1-D RBF kernels, scaled so that the product's largest eigenvalue is a few hundred."""
    ms = [m for m in (c["m1"], c["m2"], c["m3"]) if m]
    Ks = [_rbf_grid(m, 0.05 + 0.1 * float(_rand(g, 1))) for m in ms]
    return [K * (200.0 ** (1.0 / len(ms)) / float(K.sum(1).max())) for K in Ks]


def _laplacian(n, g):
    """0.05 (D - W) of a graph with about six neighbours per vertex, mostly near in the numbering."""
    r = torch.arange(n, device=DEV).repeat(3)
    hop = 1 + (_rand(g, 3 * n) ** 4 * (n / 4)).long()
    c = (r + hop) % n
    key = torch.unique(torch.cat([r * n + c, c * n + r]))
    r, c = key // n, key % n
    deg = torch.bincount(r, minlength=n).double()
    r, c, v = torch.cat([r, torch.arange(n, device=DEV)]), torch.cat([c, torch.arange(n, device=DEV)]), \
        torch.cat([-torch.ones(r.numel(), dtype=torch.float64, device=DEV), deg])
    o = torch.argsort(r * n + c)
    indptr = torch.zeros(n + 1, dtype=torch.int64, device=DEV)
    indptr[1:] = torch.cumsum(torch.bincount(r, minlength=n), 0)
    return indptr.to(torch.int32), c[o].to(torch.int32), (0.05 * v[o]).float()


def _inputs(c, seed):
    """The plain tensors of a case."""
    g, kind = _gen(seed), c["kind"]
    if kind == "dense_cg":
        dt = _DT[c["dtype"]]
        A = _spd(c["n"], c["lo"], c["hi"], g).to(dt)
        b = _randn(g, c["n"], c["k"]).to(torch.float64 if dt == torch.float64 else torch.float32)
        return {"A": A, "b": b[:, 0].contiguous() if c["k"] == 1 else b}
    if kind == "sparse_cg":
        ip, ix, v = _diffusion2d(c["m"], 1, g)
        v = v[0].to(_DT[c["dtype"]])
        rows = torch.repeat_interleave(torch.arange(c["m"] ** 2, device=DEV), (ip[1:] - ip[:-1]).long())
        v = torch.where(rows == ix, v + c["shift"], v)
        return {"ip": ip, "ix": ix, "v": v, "d": v[rows == ix].clone(), "b": _randn(g, c["m"] ** 2).to(v.dtype)}
    if kind in ("kron_cg", "kron_fun"):
        dt = _DT[c["dtype"]]
        Ks = [K.to(dt) for K in _kron_factors(c, g)]
        n = math.prod(K.shape[0] for K in Ks)
        b = _randn(g, n, c["k"])
        return {"Ks": Ks, "b": (torch.sign(b) if kind == "kron_fun" else b).to(dt)}
    if kind == "eig":
        Ks = [40.0 * _rbf_grid(m, e + 0.02 * float(_rand(g, 1))) / m for m, e in ((c["m1"], 0.11), (c["m2"], 0.17))]
        n = c["m1"] * c["m2"]
        return {"Ks": [K.float() for K in Ks], "L": _laplacian(n, g), "b": _randn(g, n).float()}
    if kind == "gp_grad":
        K = _rbf_points(c["n"], 3, 0.1, g).float()
        return {"K": K, "y": _randn(g, c["n"]).float(), "Z": torch.sign(_randn(g, c["n"], c["k"])).float()}
    if kind == "family":
        ip, ix, v = _diffusion2d(c["m"], c["systems"], g)
        return {"ip": ip, "ix": ix, "v": v.float(), "b": _randn(g, c["systems"], c["m"] ** 2)}
    if kind == "uneven":
        mats, rhs = [], []
        for s in range(c["systems"]):  # sizes spread over the range by the golden ratio
            n = c["n_lo"] + int((0.618034 * (s + 1)) % 1.0 * (c["n_hi"] - c["n_lo"] + 1))
            K = _rbf_points(n, 3, 0.05 + 0.25 * float(_rand(g, 1)), g)
            K.diagonal().add_(10 ** (-2 + float(_rand(g, 1))))
            mats.append(K.float())
            rhs.append(_randn(g, n).float())
        return {"mats": mats, "rhs": rhs}
    ip, ix, v = _diffusion3d(c["m"], g)
    return {"ip": ip, "ix": ix, "v": v[None], "b": _randn(g, c["k"], c["m"] ** 3)}


def prepare(c, seed):
    t, kind = _inputs(c, seed), c["kind"]
    if kind == "dense_cg":
        t["op"] = cola.PSD(cola.Dense(t["A"]))
        t["P"] = cola.Diagonal(1.0 / t["A"].diagonal().to(t["b"].dtype)) if c["jacobi"] else None
    elif kind == "sparse_cg":
        n = c["m"] ** 2
        t["op"] = cola.PSD(cola.Sparse.from_csr(t["ip"], t["ix"], t["v"], (n, n)))
        t["P"] = cola.Diagonal(1.0 / t["d"])
    elif kind in ("kron_cg", "kron_fun"):
        K = cola.Kronecker(*[cola.Dense(K) for K in t["Ks"]])
        t["op"] = cola.PSD(K + c["noise"] * cola.I_like(K))
    elif kind == "eig":
        n = t["b"].numel()
        K = cola.Kronecker(*[cola.Dense(K) for K in t["Ks"]])
        t["op"] = cola.SelfAdjoint(K + cola.Sparse.from_csr(*t["L"], (n, n)))
    elif kind == "gp_grad":
        t["K"].requires_grad_(True)
        t["y"].requires_grad_(True)
    elif kind in ("family", "block3d"):
        t["fam"] = BatchedCSR(t["ip"], t["ix"], t["v"], shared=kind == "block3d")
        if c.get("precond") == "learned":
            t["net"] = learned_fsai.FsaiNet.load(learned_fsai.WEIGHTS, device=DEV)
            t["pat"] = FsaiPattern(t["ip"], t["ix"])
    t["case"] = dict(c)
    return t


def run(t):
    c = t["case"]
    kind = c["kind"]
    if kind in ("dense_cg", "sparse_cg"):
        return cola.linalg.solve(t["op"], t["b"], CG(tol=c["tol"], max_iters=2000, P=t["P"]))
    if kind == "kron_cg":
        return cola.linalg.solve(t["op"], t["b"], CG(tol=c["tol"], max_iters=1000))
    if kind == "kron_fun":
        fA = (cola.linalg.sqrt if c["fun"] == "sqrt" else cola.linalg.log)(t["op"], Lanczos(max_iters=c["steps"], tol=1e-12))
        return fA @ t["b"] if c["dtype"] == "float64" else fA.quadratic_forms(t["b"])
    if kind == "eig":
        vals, vecs = cola.linalg.eig(t["op"], c["k"], "LM", Lanczos(start_vector=t["b"], max_iters=c["steps"], tol=1e-12))
        return {"vals": vals, "vecs": vecs}
    if kind == "gp_grad":  # the operator is rebuilt in every step, as its kernel matrix is new in every step
        K = cola.Dense(t["K"])
        A = cola.PSD(K + c["noise"] * cola.I_like(K))
        x, _ = cg(A, t["y"], tol=1e-6, max_iters=1000)
        ld = stochastic_lanczos_quad(A, torch.log, max_iters=c["steps"], tol=1e-12, probes=t["Z"])
        loss = 0.5 * (t["y"] @ x) + 0.5 * ld
        dK, dy = torch.autograd.grad(loss, [t["K"], t["y"]])
        return {"loss": loss.detach(), "dK": dK, "dy": dy}
    if kind == "family":
        fsai = learned_fsai.g_values(t["fam"], t["net"], t["pat"]) if c["precond"] == "learned" else None
        X, _ = solve_batched(t["fam"], t["b"], precond="fsai" if fsai else "jacobi", fsai=fsai, tol=1e-11)
        return X
    if kind == "uneven":
        return solve_dense_batched(t["mats"], t["rhs"], tol=1e-11, max_iters=1000, refine=True)[0]
    X, _ = solve_batched(t["fam"], t["b"], precond="jacobi", tol=1e-11)
    return X


# ---- the work of a pass -------------------------------------------------------------------------------


def _steps(kappa, tol):
    """CG steps to a relative residual of tol at condition number kappa (Chebyshev estimate)."""
    return 0.5 * math.sqrt(kappa) * math.log(2.0 / tol)


def work(c):
    kind = c["kind"]
    if kind == "dense_cg":
        n, k = c["n"], c["k"]
        e = {"float32": 4, "float64": 8, "bfloat16": 2}[c["dtype"]]
        return {"bytes": n * n * e + 2 * n * k * max(e, 4), "flops": _steps(c["hi"] / c["lo"], c["tol"]) * 2 * n * n * k}
    if kind == "sparse_cg":
        n, e = c["m"] ** 2, 8 if c["dtype"] == "float64" else 4
        kappa = 4 * c["m"] ** 2 / math.pi ** 2 if not c["shift"] else 16 / c["shift"]
        return {"bytes": n * (5 * (e + 4) + 4 + 3 * e), "flops": _steps(kappa, c["tol"]) * n * 22}
    if kind in ("kron_cg", "kron_fun", "eig"):
        ms = [m for m in (c["m1"], c["m2"], c.get("m3", 0)) if m]
        n = math.prod(ms)
        e = 8 if c.get("dtype", "float32") == "float64" else 4
        if kind == "eig":
            mv, s = n * (2 * sum(ms) + 14), c["steps"]
            return {"bytes": n * (7 * 8 + 4 + 4) + 4 * c["k"] * n, "flops": s * mv + 8 * n * s * s / 2}
        mv = 2 * n * c["k"] * sum(ms)
        s = c["steps"] if kind == "kron_fun" else _steps(200 / c["noise"], c["tol"])
        extra = 8 * n * c["k"] * s * s / 2 if kind == "kron_fun" else 10 * n * c["k"] * s
        return {"bytes": 2 * n * c["k"] * e + e * sum(m * m for m in ms), "flops": s * mv + extra}
    if kind == "gp_grad":
        n, k, s = c["n"], c["k"], c["steps"]
        it = _steps(1 + 25 / c["noise"], 1e-6)
        flops = 2 * n * n * (2 * it + k * s + k * it + k + 1) + 8 * n * k * s * s / 2
        return {"bytes": 2 * 4 * n * n + 4 * n * (k + 2), "flops": flops}
    if kind == "family":
        n, S = c["m"] ** 2, c["systems"]
        per = 2 * (5 + 7 * (c["precond"] == "learned")) + 11
        its = (1.1 if c["precond"] == "learned" else 2.2) * 2.2 * c["m"]
        return {"bytes": S * n * (5 * 4 + 8 + 8), "flops": S * n * per * its}
    if kind == "uneven":
        mid = (c["n_lo"] + c["n_hi"]) / 2
        sq = mid * mid + (c["n_hi"] - c["n_lo"]) ** 2 / 12
        return {"bytes": c["systems"] * (4 * sq + 12 * mid), "flops": c["systems"] * 2 * sq * 300}
    n = c["m"] ** 3
    return {"bytes": n * (7 * 8 + 4 + 16 * c["k"]), "flops": n * c["k"] * 25 * 4 * c["m"]}


# ---- 64-bit values --------------------------------------------------------------------------------------


def _kron_apply(Ks, V):
    """(K1 x K2 x ...) V for an (n, k) block."""
    dims = [K.shape[0] for K in Ks]
    Y = V.reshape(*dims, V.shape[1])
    for i, K in enumerate(Ks):
        Y = torch.movedim(torch.tensordot(K, Y, dims=([1], [i])), 0, i)
    return Y.reshape(V.shape)


def _kron_fun(Ks, noise, f, V):
    """f(K1 x K2 x ... + noise I) V through the factors' eigendecompositions."""
    lam, Us = torch.ones(1, dtype=torch.float64, device=DEV), []
    for K in Ks:
        w, U = torch.linalg.eigh(K)
        Us.append(U)
        lam = torch.kron(lam, w)
    return _kron_apply(Us, f(lam + noise)[:, None] * _kron_apply([U.T for U in Us], V))


def _pcg(ip, ix, vals, B, tol=1e-14, most=12000):
    """FP64 Jacobi-CG of a block-diagonal system (vals (S, nnz), B (S, n)) or of one matrix with many
    right-hand sides (vals (1, nnz)), in torch tensor operations."""
    S, n = B.shape
    rows = torch.repeat_interleave(torch.arange(n, device=DEV), (ip[1:] - ip[:-1]).long())
    dinv = 1.0 / vals.double()[:, rows == ix]
    if vals.shape[0] == 1:
        A = torch.sparse_csr_tensor(ip.long(), ix.long(), vals[0].double(), (n, n))
        mv = lambda P: (A @ P.T).T  # noqa: E731
    else:
        off = torch.arange(S, device=DEV)[:, None]
        nnz = ix.numel()
        A = torch.sparse_csr_tensor(torch.cat([(ip[:-1].long() + off * nnz).reshape(-1), torch.tensor([S * nnz], device=DEV)]),
                                    (ix.long() + off * n).reshape(-1), vals.double().reshape(-1), (S * n, S * n))
        mv = lambda P: (A @ P.reshape(-1)).reshape(S, n)  # noqa: E731
    X, R = torch.zeros_like(B), B.clone()
    Z = dinv * R
    P, rz, bn = Z.clone(), (R * Z).sum(1, keepdim=True), B.norm(dim=1)
    for it in range(most):
        AP = mv(P)
        al = rz / (P * AP).sum(1, keepdim=True).clamp_min(1e-300)
        X += al * P
        R -= al * AP
        if it % 50 == 49 and bool(((R.norm(dim=1) / bn) < tol).all()):
            break
        Z = dinv * R
        new = (R * Z).sum(1, keepdim=True)
        P = Z + (new / rz.clamp_min(1e-300)) * P
        rz = new
    return X


def exact(c, seed):
    t, kind = _inputs(c, seed), c["kind"]
    if kind == "dense_cg":
        b = t["b"].double()
        x = torch.linalg.solve(t["A"].double(), b[:, None] if c["k"] == 1 else b)
        return x[:, 0] if c["k"] == 1 else x
    if kind == "sparse_cg":
        return _pcg(t["ip"], t["ix"], t["v"][None], t["b"].double()[None])[0]
    if kind in ("kron_cg", "kron_fun"):
        f = {"kron_cg": torch.reciprocal, "sqrt": torch.sqrt, "log": torch.log}[c.get("fun", kind)]
        b = t["b"].double()
        y = _kron_fun([K.double() for K in t["Ks"]], c["noise"], f, b)
        return (b * y).sum(0) if kind == "kron_fun" and c["dtype"] == "float32" else y
    if kind == "eig":  # eigenvalues by long FP64 Lanczos; the vectors' signs are the caller's own
        Ks, (ip, ix, v), n = [K.double() for K in t["Ks"]], t["L"], t["b"].numel()
        A = torch.sparse_csr_tensor(ip.long(), ix.long(), v.double(), (n, n))
        V, al, be = [t["b"].double() / t["b"].double().norm()], [], []
        for i in range(min(140, n)):
            w = _kron_apply(Ks, V[-1][:, None])[:, 0] + A @ V[-1]
            al.append(w @ V[-1])
            Q = torch.stack(V)
            for _ in range(2):
                w = w - Q.T @ (Q @ w)
            be.append(w.norm())
            V.append(w / be[-1])
        T = torch.diag(torch.stack(al)) + torch.diag(torch.stack(be[:-1]), 1) + torch.diag(torch.stack(be[:-1]), -1)
        return {"vals": torch.linalg.eigvalsh(T)[-c["k"]:], "vecs": None}
    if kind == "gp_grad":
        K, y, Z = t["K"].double(), t["y"].double(), t["Z"].double()
        w, U = torch.linalg.eigh(K)
        w = w + c["noise"]
        x = U @ ((U.T @ y) / w)
        UZ = U.T @ Z
        ld = (torch.log(w)[:, None] * UZ.square()).sum() / Z.shape[1]
        S = U @ (UZ / w[:, None])
        return {"loss": 0.5 * (y @ x) + 0.5 * ld, "dK": 0.5 * (S @ Z.T) / Z.shape[1] - 0.5 * torch.outer(x, x), "dy": x}
    if kind == "family":
        return _pcg(t["ip"], t["ix"], t["v"], t["b"], tol=1e-13)
    if kind == "uneven":
        return [torch.linalg.solve(A.double(), b.double()) for A, b in zip(t["mats"], t["rhs"])]
    return _pcg(t["ip"], t["ix"], t["v"], t["b"], tol=1e-13)

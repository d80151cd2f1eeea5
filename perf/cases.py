"""The workloads whose speed is followed: whole time loops and history sums through the public API.

Sizes are those of this repository's configurations (config1..config5 and sf3d of
fpde_hpc_gb300.problems, the Sum-contract workloads of bench.py) and ragged ones beside them.
Every case is one of seven kinds:
  line      one 1D Caputo column, a whole solve from an initial state (Line.solve_host)
  do        the same for the distributed-order equation in Crank-Nicolson form
  richards  a Richards column whose coefficients follow the solution
  lod       a 3D LOD run on device-resident grids (Lod3D.reset / run / state)
  batch     an ensemble of independent columns (Batch.solve_host)
  sum       one call of the Sum kernel's contract (Context.sum_alg), as a step loop of a host
            program issues it
  sf        a 3D LOD run with implicit space-fractional line solves
"""
import math

import numpy as np
import torch

import fpde_hpc_gb300 as fp

FP64, SPLIT = 0, 3          # fpde_precision: plain FP64, exact three-slice bf16 far history
PREC = {"fp64": FP64, "split": SPLIT}


def listed():
    return [
        # the smallest run in use: a 1,000-interval column, 1,000 steps; launches and latency count
        {"name": "line_small", "kind": "line", "N": 1000, "steps": 1000, "alpha": 0.8, "tau": 1e-3, "prec": "fp64"},
        # the plain FP64 method on the benchmark's fine grid
        {"name": "line_fp64", "kind": "line", "N": 65536, "steps": 2048, "alpha": 0.7, "tau": 1e-4, "prec": "fp64"},
        # the benchmark's headline run
        {"name": "line_split", "kind": "line", "N": 65536, "steps": 8192, "alpha": 0.7, "tau": 1e-4,
         "prec": "split"},
        # a distributed-order run, 16 orders fused into one lag-weight vector
        {"name": "do_split", "kind": "do", "N": 16384, "steps": 4096, "orders": 16, "tau": 1e-4, "prec": "split"},
        # soil water transport: a 3 m column with van Genuchten-Mualem closures, 900 s steps
        {"name": "richards", "kind": "richards", "N": 4001, "steps": 400, "alpha": 0.8, "k_form": 1,
         "prec": "fp64"},
        # the benchmark's 3D run: zero-flux sides, Dirichlet top and bottom
        {"name": "lod_split", "kind": "lod", "sN": 128, "M": 128, "K": 128, "steps": 1024, "alpha": 0.85,
         "tau": 1e-3, "prec": "split"},
        # a ragged 3D grid in FP64
        {"name": "lod_fp64", "kind": "lod", "sN": 61, "M": 47, "K": 90, "steps": 300, "alpha": 0.8, "tau": 1e-3,
         "prec": "fp64"},
        # the benchmark's ensemble of uneven columns
        {"name": "batch_split", "kind": "batch", "cols": 512, "n_min": 256, "n_max": 16384, "steps": 2048,
         "sizes": 6, "tau": 1e-3, "prec": "split"},
        # a parameter study on a smaller ensemble in FP64
        {"name": "batch_fp64", "kind": "batch", "cols": 96, "n_min": 200, "n_max": 5000, "steps": 300, "sizes": 6,
         "tau": 1e-3, "prec": "fp64"},
        # restricted summing of a host program's step loop: newest 256 lags on a 130^3 grid
        {"name": "sum_window", "kind": "sum", "alg": 1, "nodes": 2197000, "rows": 320, "terms": 256, "alpha": 0.8},
        # the series history of the same loop: 16 moments per point
        {"name": "sum_series", "kind": "sum", "alg": 2, "nodes": 2197000, "rows": 2, "terms": 16, "alpha": 0.8},
        # implicit space-fractional line solves, the reference's default solver threshold
        {"name": "sf_lod", "kind": "sf", "n": 64, "steps": 8, "gamma": 0.7, "two_sided": False},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["line", "line", "do", "richards", "lod", "lod", "batch", "batch", "sum", "sum", "sf"])
    prec = rng.choice(["fp64", "split"])
    alpha = round(rng.uniform(0.5, 0.95), 3)
    if kind == "line":
        N, steps = _log_int(rng, 300, 65536), _log_int(rng, 100, 8192 if prec == "split" else 2048)
        return {"kind": kind, "N": N, "steps": steps, "alpha": alpha, "tau": rng.choice([1e-4, 1e-3]), "prec": prec}
    if kind == "do":
        steps = _log_int(rng, 100, 4096 if prec == "split" else 2048)
        return {"kind": kind, "N": _log_int(rng, 300, 16384), "steps": steps, "orders": rng.randint(4, 32),
                "tau": 1e-4, "prec": prec}
    if kind == "richards":
        return {"kind": kind, "N": _log_int(rng, 300, 16384), "steps": _log_int(rng, 50, 400), "alpha": alpha,
                "k_form": rng.choice([1, 2]), "prec": prec}
    if kind == "lod":
        return {"kind": kind, "sN": _log_int(rng, 20, 128), "M": _log_int(rng, 20, 128), "K": _log_int(rng, 20, 128),
                "steps": _log_int(rng, 64, 1024 if prec == "split" else 300), "alpha": alpha, "tau": 1e-3,
                "prec": prec}
    if kind == "batch":
        n_min = _log_int(rng, 64, 1000)
        return {"kind": kind, "cols": _log_int(rng, 8, 256), "n_min": n_min,
                "n_max": min(16384, n_min * rng.randint(2, 60)),
                "steps": _log_int(rng, 100, 1024 if prec == "split" else 300), "sizes": rng.randint(0, 1 << 20),
                "tau": 1e-3, "prec": prec}
    if kind == "sum":
        alg = rng.choice([1, 2])
        terms = _log_int(rng, 16, 300) if alg == 1 else rng.randint(4, 32)
        return {"kind": kind, "alg": alg, "nodes": _log_int(rng, 1000, 2197000),
                "rows": terms + rng.randint(2, 40) if alg == 1 else 2, "terms": terms, "alpha": alpha}
    return {"kind": kind, "n": rng.randint(16, 64), "steps": rng.randint(3, 8),
            "gamma": round(rng.uniform(0.6, 0.9), 3), "two_sided": False}


# ------------------------------------------------------------------ inputs

def _field(n, sigma, ell, rng):
    """Lognormal conductivity on n uniform nodes of [0, 1]: filtered noise of correlation length ell."""
    f = np.fft.rfftfreq(n, d=1.0 / (n - 1))
    g = np.fft.irfft(np.fft.rfft(rng.standard_normal(n)) * np.exp(-0.5 * (2 * np.pi * f * ell) ** 2), n=n)
    return np.exp(sigma * (g - g.mean()) / g.std())


def _mixture(x, rng):
    """Sum of 8 Gaussians, zero at both ends."""
    c, w, a = rng.uniform(0.1, 0.9, 8), rng.uniform(0.01, 0.1, 8), rng.uniform(0.5, 1.0, 8)
    u = (a * np.exp(-0.5 * ((x[:, None] - c) / w) ** 2)).sum(axis=1) * np.sin(np.pi * x)
    u[0] = u[-1] = 0.0
    return u


def _column(N, rng):
    """A, B, Rlap of a lognormal column of N intervals and its initial state."""
    k, u0 = _field(N + 1, 0.5, 0.01, rng), _mixture(np.arange(N + 1) / N, rng)
    A, B, R = np.zeros(N + 1), np.zeros(N + 1), np.zeros(N + 1)
    A[1:N], B[1:N] = k[:N - 1] * (N * N), k[1:N] * (N * N)
    R[1:N] = A[1:N] + B[1:N]
    return A, B, R, u0


def _do_orders(n):
    x, w = np.polynomial.legendre.leggauss(n)
    a = 0.5 * (x + 1.0)
    return a, 0.5 * w * 6.0 * a * (1.0 - a)


def _field_3d(shape, sigma, ell, h, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    g = torch.fft.rfftn(torch.randn(shape, generator=gen, device="cuda", dtype=torch.float64))
    for axis, n in enumerate(shape):
        f = (torch.fft.rfftfreq if axis == 2 else torch.fft.fftfreq)(n, d=h[axis], device="cuda", dtype=torch.float64)
        g = g * torch.exp(-0.5 * (2 * math.pi * ell * f) ** 2).reshape([-1 if q == axis else 1 for q in range(3)])
    g = torch.fft.irfftn(g, s=shape)
    return torch.exp(sigma * (g - g.mean()) / g.std())


def _grid(case, seed):
    """Coefficients (3 passes of A, B, Rlap), initial grid, line-end kinds and steps of a 3D run."""
    dims = (case["sN"], case["M"], case["K"]) if "sN" in case else (case["n"],) * 3
    sN, M, K = dims
    shape, h = (K + 2, M + 2, sN + 2), (1.0 / K, 1.0 / M, 1.0 / sN)
    k = _field_3d(shape, 0.4, 0.05, h, seed)
    rng = np.random.default_rng(seed)
    c = rng.uniform(0.35, 0.65, 3)
    z, y, x = (torch.arange(s, device="cuda", dtype=torch.float64) * d for s, d in zip(shape, h))
    u0 = (torch.exp(-(z - c[0]) ** 2 / 0.02)[:, None, None] * torch.exp(-(y - c[1]) ** 2 / 0.02)[:, None]
          * torch.exp(-(x - c[2]) ** 2 / 0.02))
    u0[0] = 0.0
    u0[K:] = 0.0
    return dims, shape, h, k, u0


def _lod_coefs(k, h):
    cA, cB = (torch.empty((3,) + tuple(k.shape), dtype=torch.float64, device="cuda") for _ in range(2))
    for pss, axis in ((0, 2), (1, 1), (2, 0)):
        cA[pss] = torch.roll(k, 1, dims=axis) / (h[axis] * h[axis])
        cB[pss] = k / (h[axis] * h[axis])
    return cA, cB, cA + cB


def _batch_sizes(case):
    """Intervals of every column, log-uniform; part of the workload, the same for every input."""
    u = np.random.default_rng(case["sizes"]).uniform(math.log(case["n_min"]), math.log(case["n_max"]), case["cols"])
    return [int(n) for n in np.rint(np.exp(u))]


def _batch_columns(case, seed):
    rng = np.random.default_rng(seed)
    alphas = rng.uniform(0.5, 0.95, case["cols"])
    return [(N, float(a)) + _column(N, rng) for N, a in zip(_batch_sizes(case), alphas)]


def _sum_inputs(case, seed):
    """Snapshots of a decaying field (rows x nodes), steps, weights and, for the series, moments."""
    gen = torch.Generator(device="cuda").manual_seed(seed)
    nodes, rows = case["nodes"], case["rows"]
    base = torch.rand(nodes, generator=gen, device="cuda", dtype=torch.float64)
    rate = 0.5 + torch.rand(nodes, generator=gen, device="cuda", dtype=torch.float64)
    old = torch.empty((rows, nodes), device="cuda", dtype=torch.float64)
    for t in range(rows):
        torch.mul(base, torch.exp(rate * (-0.01 * t)), out=old[t])
    tau = 1e-3
    if case["alg"] == 1:
        lag = np.arange(rows - 1, 0, -1, dtype=np.float64)          # term t has lag rows-1-t
        p = 1 - case["alpha"]
        kb = tau ** p * ((lag + 1) ** p - lag ** p) / p
        kept, cut = rows - 1 - case["terms"], rows - 2 - case["terms"]
        return old, np.full(rows - 1, tau), kb, 0.5 * (kb[kept] + kb[cut])
    H = torch.rand((nodes, case["terms"]), generator=gen, device="cuda", dtype=torch.float64) * 1e-3
    n = 500
    t0, t1 = n * tau, (n + 1) * tau
    j = np.arange(case["terms"])
    row2 = (t1 ** (j + 1) - t0 ** (j + 1)) / ((j + 1) * t1 ** (j + 1))
    return old, np.full(n + 2, tau), row2, (t1 + tau, t1, n, H)


def _dev(x):
    return torch.from_numpy(np.ascontiguousarray(x)).cuda()


_context = []


def _ctx():
    if not _context:
        _context.append(fp.Context(0))
    return _context[0]


class _State(dict):
    """A case's handle, inputs and output buffers; the handle's device memory goes with it."""

    def __del__(self):
        if self.get("handle") is not None:
            self["handle"].close()


def prepare(case, seed):
    ctx, kind, s = _ctx(), case["kind"], _State(case=case)
    steps = case.get("steps")
    if kind in ("line", "do"):
        A, B, R, u0 = _column(case["N"], np.random.default_rng(seed))
        if kind == "line":
            Da = 1.0 / math.gamma(1.0 - case["alpha"])
            s["handle"] = fp.Line(ctx, case["N"], case["alpha"], case["tau"], Da, A, B, R, u0, steps,
                                  precision=PREC[case["prec"]])
        else:
            a, qw = _do_orders(case["orders"])
            c = fp.do_weights(a, qw, case["tau"], steps + 1)
            s["handle"] = fp.Line(ctx, case["N"], 0.5, case["tau"], 1.0, 0.5 * A, 0.5 * B, 0.5 * R, u0, steps,
                                  precision=PREC[case["prec"]], lag_weights=c / case["tau"], theta=1.0)
        s["u0"], s["out"] = u0, np.empty_like(u0)
    elif kind == "richards":
        N = case["N"]
        rng = np.random.default_rng(seed)
        Z = np.arange(N + 1) * 3.0 / N
        u0 = -rng.uniform(0.7, 0.9) - Z
        E = 2.3e-8 * (1.0 + 0.3 * np.sin(np.arange(steps) * 0.05) + 0.05 * rng.random(steps))
        rich = dict(k_form=case["k_form"], k_sat=2e-6, Z=Z, dL=np.full(N + 1, 3.0 / N), evaporation=E)
        s["handle"] = fp.Line(ctx, N, case["alpha"], 900.0, 1.0 / math.gamma(1.0 - case["alpha"]), None, None, None,
                              u0, steps, right=(0, u0[-1]), precision=PREC[case["prec"]], richards=rich)
        s["u0"], s["out"] = u0, np.empty_like(u0)
    elif kind == "lod":
        dims, shape, h, k, u0 = _grid(case, seed)
        cA, cB, cR = (c.cpu().numpy() for c in _lod_coefs(k, h))
        s["handle"] = fp.Lod3D(ctx, dims, case["alpha"], case["tau"], 1.0 / math.gamma(1.0 - case["alpha"]), cA, cB,
                               cR, u0.cpu().numpy(), steps, left_kind=(1, 1, 0), right_kind=(1, 1, 0),
                               dLN=(h[2], h[1], h[0]), precision=PREC[case["prec"]])
        s["u0"], s["out"] = u0, torch.empty_like(u0)
    elif kind == "sf":
        dims, shape, h, k, u0 = _grid(case, seed)
        n, gamma = case["n"], case["gamma"]
        for axis in (1, 2):                                   # Dirichlet 0 at every line end
            u0.select(axis, 0).zero_()
            u0.narrow(axis, n, 2).zero_()
        z = torch.arange(n + 2, device="cuda", dtype=torch.float64) / n
        iw = (1.5 + torch.sin(z / 4.0))[:, None, None].expand(shape).contiguous()
        w = h[0] ** (1.0 - gamma) / math.gamma(2.0 - gamma)
        mA, mB, mR = _lod_coefs(k, h)
        cA, cB, cR = ((c * iw * w).cpu().numpy() for c in (mA, mB, mR))
        mc = torch.stack([mA, -mR, mB], dim=1).cpu().numpy()
        Tm = np.tile(fp.sf_toeplitz_row(gamma, np.arange(n + 2) / n, n), (3, 1))
        src = (5.0 * torch.exp(-(z - 0.5) ** 2 / 0.045)[:, None, None] * torch.exp(-(z - 0.5) ** 2 / 0.045)[:, None]
               * torch.exp(-(z - 0.4) ** 2 / 0.045))
        s["handle"] = fp.Lod3D(ctx, dims, 0.8, 1e-3, 1.0 / math.gamma(0.2), cA, cB, cR, u0.cpu().numpy(), steps,
                               source=src.cpu().numpy(),
                               space_frac=dict(space_der=int(case["two_sided"]), tol=1e-9, max_iter=5000, Tm=Tm, mc=mc,
                                               iw=np.stack([iw.cpu().numpy()] * 3)))
        s["u0"], s["out"] = u0, torch.empty_like(u0)
    elif kind == "batch":
        cols = [dict(N=N, alpha=a, tau=case["tau"], Da=1.0 / math.gamma(1.0 - a), A=A, B=B, Rlap=R, u0=u0)
                for N, a, A, B, R, u0 in _batch_columns(case, seed)]
        b = fp.Batch(ctx, cols, steps, precision=PREC[case["prec"]])
        s["handle"] = b
        s["u0"] = b.pack([c["u0"] for c in cols])
        s["out"] = np.zeros_like(s["u0"])
    else:
        old, taus, w, more = _sum_inputs(case, seed)
        s.update(old=old, tau=_dev(taus), w=_dev(w), S=torch.zeros(case["nodes"], device="cuda", dtype=torch.float64))
        if case["alg"] == 1:
            s["param"] = more
        else:
            s["gtj"], s["gt"], s["tstep"], s["H"] = more
    return s


def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind in ("line", "do", "richards", "batch"):
        return s["handle"].solve_host(s["u0"], case["steps"], s["out"])
    if kind in ("lod", "sf"):
        s["handle"].reset(s["u0"])
        s["handle"].run(case["steps"])
        return s["handle"].state(s["out"])
    if case["alg"] == 1:
        return _ctx().sum_alg(1, s["old"], s["tau"], kb=s["w"], sum_param=s["param"], out=s["S"])
    _ctx().sum_alg(2, s["old"], s["tau"], sum_param=case["terms"], Htmp=s["H"], row2=s["w"], gtj=s["gtj"], gt=s["gt"],
                   alpha=case["alpha"], tstep=s["tstep"], out=s["S"])
    return {"S": s["S"], "moments": s["H"]}


def work(case):
    """Bytes: inputs (coefficients, states, snapshots) once and results once. Operations: two per
    history term of the method (every earlier step, every node), nine per node and step for the
    right-hand side, the Thomas sweeps and the increment; per space-fractional line solve one
    Toeplitz product per step."""
    kind = case["kind"]
    if kind == "sum":
        n, p = case["nodes"], case["terms"]
        if case["alg"] == 1:
            return {"bytes": 8.0 * n * (p + 2), "flops": 3.0 * n * p}
        return {"bytes": 8.0 * n * (2 * p + 3), "flops": (4.0 * p + 2) * n}
    S = case["steps"]
    if kind in ("line", "do", "richards"):
        nodes, passes, arrays = case["N"], 1, 5 if kind != "richards" else 4
    elif kind == "batch":
        nodes, passes, arrays = sum(_batch_sizes(case)), 1, 5
    elif kind == "lod":
        nodes, passes, arrays = (case["sN"] + 2) * (case["M"] + 2) * (case["K"] + 2), 3, 11
    else:
        nodes, passes, arrays = (case["n"] + 2) ** 3, 3, 24
    flops = nodes * (S * (S - 1.0) + 9.0 * passes * S)
    if kind == "richards":
        flops += 60.0 * nodes * S
    if kind == "sf":
        flops += nodes * S * 3.0 * case["n"]
    return {"bytes": 8.0 * nodes * arrays, "flops": flops}


# ------------------------------------------------------------------ the same in 64 bits, in torch

class _Tridiag:
    """A U_{i-1} - R U_i + B U_{i+1} = r along dimension 0 (rows 1..N-1), by cyclic reduction on all
    rows at once."""

    def __init__(self, A, B, R):
        a, c, b = A.clone(), B.clone(), -R
        a[0], c[-1] = 0.0, 0.0
        n, self.levels, st = A.shape[0], [], 1
        while st < n:
            al, ga = torch.zeros_like(a), torch.zeros_like(a)
            al[st:] = -a[st:] / b[:-st]
            ga[:-st] = -c[:-st] / b[st:]
            b2, a2, c2 = b.clone(), torch.zeros_like(a), torch.zeros_like(a)
            b2[st:] += al[st:] * c[:-st]
            b2[:-st] += ga[:-st] * a[st:]
            a2[st:] = al[st:] * a[:-st]
            c2[:-st] = ga[:-st] * c[st:]
            self.levels.append((st, al[st:].contiguous(), ga[:-st].contiguous()))
            a, b, c = a2, b2, c2
            st *= 2
        self.b = b

    def solve(self, r):
        for st, al, ga in self.levels:
            q = r.clone()
            q[st:].addcmul_(al, r[:-st])
            q[:-st].addcmul_(ga, r[st:])
            r = q
        return r / self.b


def _lags(alpha, n):
    j = np.arange(1, n, dtype=np.float64)
    return np.concatenate([[1.0], np.exp((1 - alpha) * np.log(j)) * np.expm1((1 - alpha) * np.log1p(1.0 / j))])


def _caputo(alpha, tau, n):
    """Lag weights Da kkk0 b_l / tau, l = 0..n-1."""
    return _lags(alpha, n) * tau ** -alpha / ((1.0 - alpha) * math.gamma(1.0 - alpha))


def _march(A, B, R, u0, w, steps, theta=0.0):
    """The line scheme on interior rows (Dirichlet 0 ends). A, B, R, u0: (rows,); w: (lags,) or,
    for decoupled columns side by side, (lags, rows)."""
    T = _Tridiag(A, B, R + w[0])
    u, hist = u0.clone(), torch.zeros((steps,) + tuple(u0.shape), dtype=torch.float64, device="cuda")
    rev = w.flip(0)
    for n in range(steps):
        om = -w[0] * u
        if n:
            ww = rev[rev.shape[0] - 1 - n:rev.shape[0] - 1]          # w[n], ..., w[1] for t = 0..n-1
            om += torch.mv(hist[:n].t(), ww) if w.dim() == 1 else (hist[:n] * ww).sum(0)
        if theta:
            lap = -R * u
            lap[1:] += A[1:] * u[:-1]
            lap[:-1] += B[:-1] * u[1:]
            om -= theta * lap
        x = T.solve(om)
        hist[n] = x - u
        u = x
    return u


def _exact_line(case, seed):
    A, B, R, u0 = _column(case["N"], np.random.default_rng(seed))
    f = 1.0
    if case["kind"] == "line":
        w = _caputo(case["alpha"], case["tau"], case["steps"] + 1)
    else:
        a, qw = _do_orders(case["orders"])
        f, w = 0.5, sum(q * case["tau"] ** (-x) * _lags(x, case["steps"] + 1) / math.gamma(2.0 - x)
                        for x, q in zip(a, qw))
    inner = [_dev(f * v[1:-1]) for v in (A, B, R)]
    u = _march(*inner, _dev(u0[1:-1]), _dev(w), case["steps"], 1.0 if f == 0.5 else 0.0)
    out = torch.zeros(case["N"] + 1, dtype=torch.float64, device="cuda")
    out[1:-1] = u
    return out


def _exact_batch(case, seed):
    cols = _batch_columns(case, seed)
    S, total = case["steps"], sum(c[0] for c in cols)
    if S * S * float(total) > 5e11 or S * float(total) > 2e9:
        return None
    cat = lambda k: _dev(np.concatenate([np.concatenate([c[k][1:-1], [0.0]]) for c in cols]))  # noqa: E731
    A, B, R, u0 = cat(2), cat(3), cat(4), cat(5)
    at, first = 0, []
    for c in cols:                                              # decouple neighbouring columns
        A[at], B[at + c[0] - 2], R[at + c[0] - 1] = 0.0, 0.0, 1.0
        first.append(at)
        at += c[0]
    reps = torch.tensor([c[0] for c in cols], device="cuda")
    w = _dev(np.stack([_caputo(c[1], case["tau"], S + 1) for c in cols], axis=1)).repeat_interleave(reps, dim=1)
    u = _march(A, B, R, u0, w, S).cpu().numpy()
    parts = []
    for c, f in zip(cols, first):                               # the padded layout of Batch.pack
        v = np.concatenate([[0.0], u[f:f + c[0] - 1], [0.0]])
        parts.append(np.concatenate([v, np.zeros(-len(v) % 512)]))
    return np.concatenate(parts)


def _exact_lod(case, seed):
    dims, shape, h, k, u0 = _grid(case, seed)
    sN, M, K = dims
    S, G = case["steps"], u0.numel()
    if G * 8.0 * S > 6e10 or G * float(S) * S > 4e12:
        return None
    cA, cB, cR = _lod_coefs(k, h)
    w = _dev(_caputo(case["alpha"], case["tau"], S + 1))
    rev, lam = w.flip(0), w[0]
    axis_of, N, i, j, k_ = (2, 1, 0), dims, slice(1, sN), slice(1, M), slice(1, K)
    rest = {0: (k_, j), 1: (k_, i), 2: (j, i)}

    def line_view(g, pss, lo, hi):
        v = torch.movedim(g, axis_of[pss], 0)
        return v[(slice(lo, hi),) + rest[pss]]

    T = {}
    for pss in (0, 1, 2):
        A, B, R = (line_view(c[pss], pss, 1, N[pss]).contiguous() for c in (cA, cB, cR))
        R = R + lam
        if pss != 2:                                            # zero flux: U_0 = U_1 and U_N = U_{N-1}
            R[0] -= A[0]
            R[-1] -= B[-1]
        T[pss] = _Tridiag(A, B, R)
    u, hist = u0.clone(), torch.zeros((S, G), dtype=torch.float64, device="cuda")
    for n in range(S):
        before = u.clone()
        for pss in (2, 1, 0):
            om = -lam * line_view(u, pss, 1, N[pss])
            if pss == 2 and n:
                s = torch.mv(hist[:n].t(), rev[S - n:S]).view(shape)
                om = om + line_view(s, pss, 1, N[pss])
            x = T[pss].solve(om.contiguous())
            line_view(u, pss, 1, N[pss]).copy_(x)
            zero = pss == 2
            line_view(u, pss, 0, 1).copy_(torch.zeros_like(x[:1]) if zero else x[:1])
            end = torch.zeros_like(x[:1]) if zero else x[-1:]
            line_view(u, pss, N[pss], N[pss] + 2).copy_(end.expand((2,) + tuple(x.shape[1:])))
        hist[n] = (u - before).reshape(-1)
    return u


def _exact_sum(case, seed):
    old, taus, w, more = _sum_inputs(case, seed)
    if case["alg"] == 1:
        S = torch.zeros(case["nodes"], dtype=torch.float64, device="cuda")
        for t in range(case["rows"] - 2, -1, -1):
            if abs(w[t]) < more:
                break
            S += float(w[t]) * (old[t + 1] - old[t]) / float(taus[t])
        return S
    gtj, gt, n, H = more
    d = old[1] - old[0]
    j = np.arange(case["terms"])
    v = np.empty(case["terms"])
    v[0] = gtj ** -case["alpha"]
    for q in range(1, case["terms"]):
        v[q] = v[q - 1] * (case["alpha"] + q - 1) / (q * gtj)
    H = H + d[:, None] * _dev(gt ** (j + 1) * w)
    return {"S": torch.mv(H, _dev(v)) / float(taus[n]), "moments": H}


def exact(case, seed):
    kind = case["kind"]
    if kind in ("line", "do"):
        return _exact_line(case, seed)
    if kind == "batch":
        return _exact_batch(case, seed)
    if kind == "lod":
        return _exact_lod(case, seed)
    if kind == "sum":
        return _exact_sum(case, seed)
    return None                 # richards: closures far from a torch form; sf: iterates up to a threshold

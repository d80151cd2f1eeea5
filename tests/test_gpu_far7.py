"""The FP64 far history on the tensor cores (seven bf16 slices, k_far_tc7) inside the FP64 time loops: columns
whose node counts sit beside the 128-row tiles, histories of 1, 2 and many 64-step blocks and cut short by
a window, K splits, ensembles with a weight table per column, a 3D grid; states of magnitude 1e-150
to 1e120 (the slices' exponents) and a transient that falls by six orders inside one block.

Tolerance against the oracle: 1e-12, or four times its response to a one-ulp change of coefficients and
weights. The far sums are also compared with exact sums: no further off than the FP64 multiply-add chain of
the plain per-step form (ratio of the largest errors at most 1.5, both relative to the largest value)."""
import math

import numpy as np
import pytest

from conftest import relmax

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    import fpde_hpc_gb300 as fp
    c = fp.Context(0)
    yield c
    c.close()


def _problem(N, steps, alpha=0.7, tau=1e-3, scale=1.0, rough=0.3):
    rng = np.random.default_rng(N + steps)
    k = np.exp(rough * rng.standard_normal(N + 1))
    A, B, R = np.zeros(N + 1), np.zeros(N + 1), np.zeros(N + 1)
    A[1:N], B[1:N] = k[:N - 1] * N * N, k[1:N] * N * N
    R[1:N] = A[1:N] + B[1:N]
    u0 = scale * (np.sin(np.pi * np.arange(N + 1) / N) + 0.3 * rng.random(N + 1))
    Da = 1.0 / math.gamma(1.0 - alpha)
    j = np.arange(1, steps + 1, dtype=np.float64)
    b = np.concatenate([[1.0], np.exp((1 - alpha) * np.log(j)) * np.expm1((1 - alpha) * np.log1p(1.0 / j))])
    return A, B, R, u0, alpha, tau, Da, Da * tau ** -alpha / (1.0 - alpha) * b, rng


@pytest.mark.parametrize("N,steps,scale,alpha,lags", [
    (126, 65, 1.0, 0.7, 0), (127, 129, 1.0, 0.5, 0), (128, 200, 1.0, 0.95, 0), (300, 1000, 1.0, 0.7, 0),
    (300, 500, 1e-150, 0.6, 0), (300, 500, 1e120, 0.8, 0), (2000, 700, 1.0, 0.7, 70), (2000, 700, 1.0, 0.7, 200),
    (20000, 260, 1.0, 0.6, 0)])
def test_line_vs_oracle(ctx, N, steps, scale, alpha, lags):
    import fpde_hpc_gb300 as fp
    import oracle
    A, B, R, u0, alpha, tau, Da, w, rng = _problem(N, steps, alpha, scale=scale)
    eps = 0.0
    if lags:
        eps = 0.5 * (w[lags] + w[lags + 1]) * tau / Da
        w = w.copy()
        w[lags + 1:] = 0.0
    line = fp.Line(ctx, N, alpha, tau, Da, A, B, R, u0, steps, restrict_eps=eps)
    line.run(steps)
    u = line.state()
    line.close()
    ref, _ = oracle.line_run_general(u0, steps, w, 0.0, A, B, R)
    pert = lambda v: v * (1 + 2.2e-16 * rng.choice([-1, 1], size=v.shape))
    env = relmax(oracle.line_run_general(u0, steps, pert(w), 0.0, pert(A), pert(B), pert(R))[0], ref)
    err = relmax(u, ref)
    print(f"far7 line N={N} steps={steps} scale {scale:g} alpha {alpha} lags {lags}: {err:.2e} (envelope {env:.2e})")
    assert err <= max(1e-12, 4 * env)


def test_far_sums_against_exact(ctx):
    """The history sum of one step, isolated: all nodes uncoupled (A = B = tiny), so the new state is the
    right-hand side over the local weight; increments of seven decades within a block. Exact: the same
    recurrence in extended precision."""
    import fpde_hpc_gb300 as fp
    N, steps = 383, 640
    rng = np.random.default_rng(7)
    A = np.full(N + 1, 1e-300)
    u0 = rng.standard_normal(N + 1)
    w = np.concatenate([[1.0], 0.9 * np.arange(1, steps + 1) ** -1.3])
    src = (rng.standard_normal((steps, N + 1)) * 10.0 ** rng.uniform(-6, 1, (steps, 1)))
    src[:, 0] = src[:, -1] = 0.0
    u0[0] = u0[-1] = 0.0
    # exact: u_{n+1} = u_n - (src_n + sum w D)/w0, the Om / R of the scheme with A = B = 0
    ld = np.longdouble
    u, D = u0.astype(ld), np.zeros((steps, N + 1), dtype=ld)
    wl = w.astype(ld)
    for n in range(steps):
        S = (wl[n:0:-1, None] * D[:n]).sum(axis=0) if n else np.zeros(N + 1, dtype=ld)
        un = u - (src[n].astype(ld) + S) / wl[0]
        un[0] = un[-1] = 0
        D[n] = un - u
        u = un
    errs = []
    for tuning in (None, fp.LineTuning(gemv_splits=1)):
        line = fp.Line(ctx, N, 0.5, 1.0, 1.0, A, A, 2 * A, u0, steps, lag_weights=w, source=src, tuning=tuning)
        line.run(steps)
        errs.append(float(np.max(np.abs(line.state() - u)) / np.max(np.abs(u))))
        line.close()
    print(f"history sums against extended-precision sums: blocks {errs[0]:.2e}, plain per-step form {errs[1]:.2e}")
    assert errs[0] <= 1.5 * errs[1]


def test_batch_and_lod_vs_oracle(ctx):
    import fpde_hpc_gb300 as fp
    import oracle
    from fpde_hpc_gb300 import problems
    cols, steps = [], 150
    for i, N in enumerate((5, 127, 511, 700, 3000)):
        A, B, R, u0, alpha, tau, Da, w, rng = _problem(N, steps, 0.5 + 0.1 * i)
        cols.append(dict(N=N, alpha=alpha, tau=tau, Da=Da, A=A, B=B, Rlap=R, u0=u0))
    b = fp.Batch(ctx, cols, steps)
    b.run(100)
    b.run(50)
    for k, c in enumerate(cols):
        ref = oracle.line_run(c["u0"], steps, c["tau"], c["alpha"], c["Da"], c["A"], c["B"], c["Rlap"])[0]
        pert = lambda v: v * (1 + 2.2e-16 * rng.choice([-1, 1], size=v.shape))
        env = relmax(oracle.line_run(c["u0"], steps, c["tau"], c["alpha"], c["Da"], pert(c["A"]), pert(c["B"]), pert(c["Rlap"]))[0], ref)
        err = relmax(b.state(k), ref)
        print(f"far7 ensemble N={c['N']}: {err:.2e} (envelope {env:.2e})")
        assert err <= max(1e-12, 4 * env)
    b.close()
    p = problems.config4(n=14, steps=steps)
    cA, cB, cR = p.coefs()
    kw = dict(left_kind=p.left_kind, right_kind=p.right_kind, dLN=p.dLN)
    lod = fp.Lod3D(ctx, p.dims, p.alpha, p.tau, p.Da, cA, cB, cR, p.u0, steps, **kw)
    lod.run(70)
    lod.run(80)
    u = lod.state()
    lod.close()
    ok = dict(lkind=p.left_kind, rkind=p.right_kind, dLN=p.dLN)
    ref = oracle.lod_run(p.dims, p.u0, steps, p.tau, p.alpha, p.Da, cA, cB, cR, **ok)
    env = relmax(oracle.lod_run(p.dims, p.u0, steps, p.tau, p.alpha, p.Da, pert(cA), pert(cB), pert(cR), **ok), ref)
    print(f"far7 LOD 14^3: {relmax(u, ref):.2e} (envelope {env:.2e})")
    assert relmax(u, ref) <= max(1e-12, 4 * env)

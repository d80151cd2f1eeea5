"""FP64 histories whose sums the digit slices of k_far_tc7 cannot hold, because old increments far above the
current ones carry no weight: windows (restricted summing) and lag weights that fall steeply. The state falls
by up to a hundred orders over the run and every step stays accurate to its own magnitude.

Tolerance against the oracle, relative to the final state: 1e-12, or four times its response to a one-ulp
change of coefficients and weights."""
import numpy as np
import pytest

from conftest import relmax
from test_gpu_far7 import _problem

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    import fpde_hpc_gb300 as fp
    c = fp.Context(0)
    yield c
    c.close()


def _case(N, steps, tau, lags):
    A, B, R, u0, alpha, tau, Da, w, rng = _problem(N, steps, tau=tau)
    u0[0] = u0[-1] = 0.0
    eps = 0.5 * (w[lags] + w[lags + 1]) * tau / Da
    w = w.copy()
    w[lags + 1:] = 0.0
    return A, B, R, u0, alpha, tau, Da, w, eps, rng


def _check(name, u, u0, steps, w, A, B, R, rng):
    import oracle
    ref, _ = oracle.line_run_general(u0, steps, w, 0.0, A, B, R)
    pert = lambda v: v * (1 + 2.2e-16 * rng.choice([-1, 1], size=v.shape))
    env = relmax(oracle.line_run_general(u0, steps, pert(w), 0.0, pert(A), pert(B), pert(R))[0], ref)
    err = relmax(u, ref)
    print(f"{name}: last state {np.abs(ref).max():.1e}, error {err:.2e} (envelope {env:.2e})")
    assert err <= max(1e-12, 4 * env)


@pytest.mark.parametrize("N,steps,tau,lags", [
    (64, 4000, 1e-3, 5), (64, 3000, 1e-3, 20), (64, 400, 0.1, 5), (64, 260, 1.0, 3), (300, 260, 1.0, 70), (129, 130, 0.02, 64)])
def test_windowed_line(ctx, N, steps, tau, lags):
    import fpde_hpc_gb300 as fp
    A, B, R, u0, alpha, tau, Da, w, eps, rng = _case(N, steps, tau, lags)
    line = fp.Line(ctx, N, alpha, tau, Da, A, B, R, u0, steps, restrict_eps=eps)
    line.run(steps)
    u = line.state()
    line.close()
    _check(f"line N={N}, tau {tau}, {lags} lags", u, u0, steps, w, A, B, R, rng)


@pytest.mark.parametrize("c,f,w0", [(1.0, 0.5, 10.0), (1.0, 0.1, 20.0), (0.25, 0.3, 60.0)])
def test_falling_weights(ctx, c, f, w0):
    """w_l = w_0 f 2^-cl: a lag weight spans 64 c binary orders within one 64-step block."""
    import fpde_hpc_gb300 as fp
    N, steps = 64, 260
    A, B, R, u0, alpha, tau, Da, _, rng = _problem(N, steps)
    u0[0] = u0[-1] = 0.0
    w = np.concatenate([[1.0], f * np.exp2(-c * np.arange(1, steps + 1))]) * w0
    line = fp.Line(ctx, N, 0.5, 1.0, 1.0, A, B, R, u0, steps, lag_weights=w)
    line.run(steps)
    u = line.state()
    line.close()
    _check(f"line, weights falling {c} binary orders per lag", u, u0, steps, w, A, B, R, rng)


def test_windowed_ensemble(ctx):
    """One windowed column beside an unrestricted one."""
    import fpde_hpc_gb300 as fp
    steps, cols, parts = 400, [], []
    for N, lags in ((64, 5), (600, None)):
        A, B, R, u0, alpha, tau, Da, w, eps, rng = _case(N, steps, 0.1, lags or steps - 1)
        cols.append(dict(N=N, alpha=alpha, tau=tau, Da=Da, A=A, B=B, Rlap=R, u0=u0, restrict_eps=eps if lags else 0.0))
        parts.append((f"column N={N}, {lags} lags", u0, steps, w, A, B, R, rng))
    b = fp.Batch(ctx, cols, steps)
    b.run(steps)
    states = [b.state(k).copy() for k in range(2)]
    b.close()
    for u, (name, *rest) in zip(states, parts):
        _check(name, u, *rest)


def test_windowed_grid(ctx):
    """Also the per-step FP64 sum over more than 64 rows under the staged K pass: two partial rows, which the pass
    adds (100 lags), and three, which are added before it (150)."""
    import fpde_hpc_gb300 as fp
    import oracle
    from fpde_hpc_gb300 import problems
    for tau, lags, steps in ((0.05, 5, 260), (0.5, 100, 200), (0.5, 150, 220)):
        base = problems.config4(n=9, steps=steps)
        cA, cB, cR = base.coefs()
        Da, alpha = base.Da, base.alpha
        time = oracle.time_points(np.full(steps + 1, tau))
        full = oracle.l1_weights(alpha, time, steps - 1)[0]            # term t of the last step: lag steps - 1 - t
        eps = 0.5 * (full[steps - 1 - lags] + full[steps - 2 - lags])
        kinds = dict(left_kind=(0, 0, 0), right_kind=(0, 0, 0), dLN=base.dLN)
        u0 = base.u0.copy()
        u0[0] = u0[-1] = 0.0
        lod = fp.Lod3D(ctx, base.dims, alpha, tau, Da, cA, cB, cR, u0, steps, restrict_eps=eps, **kinds)
        lod.run(steps)
        u = lod.state()
        lod.close()

        def run(f):
            U, hist, taus = u0.copy(), np.zeros((steps,) + u0.shape), np.full(steps + 1, tau)
            A, B, R = f(cA), f(cB), f(cR)
            for n in range(steps):
                kb, k0 = oracle.l1_weights(alpha, time, n)
                if n:
                    kb = kb.copy()
                    kb[:max(n - lags, 0)] = 0.0
                oracle.lod_step(base.dims, U, hist, n, kb if n else np.zeros(1), taus, Da, k0, A, B, R, None,
                                np.zeros(u0.shape), dLN=base.dLN)
            return U[1:base.dims[2], 1:base.dims[1], 1:base.dims[0]]       # the unknowns (line ends hold u0)

        rng = np.random.default_rng(0)
        ref = run(lambda v: v)
        env = relmax(run(lambda v: v * (1 + 2.2e-16 * rng.choice([-1, 1], size=v.shape))), ref)
        err = relmax(u[1:base.dims[2], 1:base.dims[1], 1:base.dims[0]], ref)
        print(f"grid 9^3, tau {tau}, {lags} lags: last state {np.abs(ref).max():.1e}, error {err:.2e} (envelope {env:.2e})")
        assert err <= max(1e-12, 4 * env)

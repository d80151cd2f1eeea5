"""FP64 near history of grids and ensembles in sub-blocks of 8 steps (k_near64_pre, k_near64): a run cut
anywhere (inside and at the edges of sub-blocks and 64-step blocks) gives the state of one run bit for
bit, with the full history and with windows shorter than a sub-block, than a block and than the run; the
windowed ensemble equals the oracle's run with the dropped weights zeroed (1e-12, or four times its
response to a one-ulp change of the coefficients)."""
import numpy as np
import pytest

from conftest import relmax
from test_gpu_far7 import _problem

pytestmark = pytest.mark.gpu
CUTS = [(1,), (7, 8, 9), (13, 63), (64, 65), (3, 60, 72, 127, 129)]


@pytest.fixture(scope="module")
def ctx():
    import fpde_hpc_gb300 as fp
    c = fp.Context(0)
    yield c
    c.close()


def _run(obj, steps, cuts):
    for a, b in zip((0,) + tuple(cuts), tuple(cuts) + (steps,)):
        obj.run(b - a)


def _eps(w, lag, tau, Da):
    """restrict_eps that keeps the first `lag` lags: between kb of lag and of lag + 1 (kb = w tau / Da)."""
    kb = w * tau / Da
    return 0.0 if lag is None else 0.5 * (kb[lag] + kb[lag + 1])


@pytest.mark.parametrize("lag", [None, 3, 20, 100])
def test_ensemble(ctx, lag):
    import fpde_hpc_gb300 as fp
    import oracle
    steps, cols, ws = 140, [], []
    for i, N in enumerate((5, 511, 512, 1500)):
        A, B, R, u0, alpha, tau, Da, w, rng = _problem(N, steps, 0.5 + 0.1 * i)
        cols.append(dict(N=N, alpha=alpha, tau=tau, Da=Da, A=A, B=B, Rlap=R, u0=u0,
                         restrict_eps=_eps(w, lag, tau, Da)))
        ws.append(w)
    states = []
    for cuts in [()] + CUTS:
        b = fp.Batch(ctx, cols, steps)
        _run(b, steps, cuts)
        states.append([b.state(k).copy() for k in range(len(cols))])
        b.close()
    for s in states[1:]:
        assert all(np.array_equal(x, y) for x, y in zip(s, states[0]))
    for k, c in enumerate(cols):
        w = ws[k].copy()
        if lag is not None:
            w[lag + 1:] = 0.0
        args = lambda f: (c["u0"], steps, w, 0.0, f(c["A"]), f(c["B"]), f(c["Rlap"]))
        ref = oracle.line_run_general(*args(lambda v: v))[0]
        pert = lambda v: v * (1 + 2.2e-16 * rng.choice([-1, 1], size=v.shape))
        env = relmax(oracle.line_run_general(*args(pert))[0], ref)
        err = relmax(states[0][k], ref)
        print(f"ensemble N={c['N']} lag {lag}: {err:.2e} (envelope {env:.2e})")
        assert err <= max(1e-12, 4 * env)


def test_grid_pieces(ctx):
    import fpde_hpc_gb300 as fp
    from fpde_hpc_gb300 import problems
    steps = 140
    p = problems.config4(n=11, steps=steps)
    cA, cB, cR = p.coefs()
    kw = dict(left_kind=p.left_kind, right_kind=p.right_kind, dLN=p.dLN)
    for eps in (0.0, 0.3, 0.05):
        states = []
        for cuts in [()] + CUTS:
            lod = fp.Lod3D(ctx, p.dims, p.alpha, p.tau, p.Da, cA, cB, cR, p.u0, steps, restrict_eps=eps, **kw)
            _run(lod, steps, cuts)
            states.append(lod.state().copy())
            lod.close()
        for s in states[1:]:
            assert np.array_equal(s, states[0])

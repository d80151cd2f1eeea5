"""FP64 lines under restricted summing on each side of the rule that takes them to 64-step blocks or to the
per-step form (512 nodes per SM, 32 lags), with windows that begin inside a block, inside the far sum's groups of
16 steps and before the block: each against the same line forced to the per-step form. Tolerance: 1e-12, or
four times the default form's response to a one-ulp change of the coefficients (long fine lines)."""
import numpy as np
import pytest

from conftest import relmax
from test_gpu_far7 import _problem

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N", [700, 77824, 77825])
@pytest.mark.parametrize("lags", [1, 2, 3, 15, 16, 17, 31, 32, 63, 64, 65, 100])
def test_windows(N, lags):
    import fpde_hpc_gb300 as fp
    steps = 200
    A, B, R, u0, alpha, tau, Da, w, rng = _problem(N, steps)
    u0[0] = u0[-1] = 0.0
    eps = 0.5 * (w[lags] + w[lags + 1]) * tau / Da
    pert = lambda v: v * (1 + 2.2e-16 * rng.choice([-1, 1], size=v.shape))
    with fp.Context(0) as ctx:
        def run(tuning, f=lambda v: v, pieces=(steps,)):
            line = fp.Line(ctx, N, alpha, tau, Da, f(A), f(B), f(R), u0, steps, restrict_eps=eps, tuning=tuning)
            for n in pieces:
                line.run(n)
            u = line.state()
            line.close()
            return u
        u = run(None)
        np.testing.assert_array_equal(run(None, pieces=(1, 40, 30, 60, steps - 131)), u)
        env = relmax(run(None, pert), u)
        err = relmax(u, run(fp.LineTuning(gemv_splits=1)))
    print(f"N={N}, {lags} lags: {err:.2e} from the per-step form (envelope {env:.2e})")
    assert err <= max(1e-12, 4 * env)

"""Increments that the digit slices of k_far_tc7 represent by special cases: states below FP64's normal range."""
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


def test_below_the_normal_range(ctx):
    """States of about 1e-310 (spacing 5e-324, 5e-14 of them). Tolerance 1e-9: N = 40 roundings of that size per
    solve and 200 steps come to 4e-10."""
    import fpde_hpc_gb300 as fp
    N, steps = 40, 200
    A, B, R, u0, alpha, tau, Da, w, rng = _problem(N, steps)
    u0 = u0 * 1e-310
    out = []
    for tuning in (fp.LineTuning(gemv_splits=1), None):
        line = fp.Line(ctx, N, alpha, tau, Da, A, B, R, u0, steps, tuning=tuning)
        line.run(steps)
        out.append(line.state() * 1e300)
        line.close()
    err = relmax(out[1], out[0])
    print(f"subnormal line: {err:.2e} from the sum over rows, last state {np.abs(out[0]).max():.1e}e-300")
    assert err <= 1e-9

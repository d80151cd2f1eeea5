"""Increments that the digit slices of k_far_tc7 represent by special cases: values that are not finite, which
every later sum keeps as the FP64 sum over rows does, and states below FP64's normal range."""
import ctypes as C

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


def _write(line, u):
    rt = C.CDLL("libcudart.so")                # the context's stream does not wait for this copy's, nor the reverse
    assert rt.cudaDeviceSynchronize() == 0
    assert rt.cudaMemcpy(C.c_void_p(line.state_ptr()), u.ctypes.data_as(C.c_void_p), C.c_size_t(u.nbytes), 1) == 0
    assert rt.cudaDeviceSynchronize() == 0


@pytest.mark.parametrize("tau", [1e-3, 1e20])
@pytest.mark.parametrize("bad", [np.nan, np.inf, -np.inf])
def test_not_finite(ctx, bad, tau):
    """A state spoilt in the first 64-step block and mended by the caller at its end: the history keeps the
    increments that were not finite, so no later value is finite, in blocks as step by step; with large weights
    and with small ones (a stand-in of 2^1025 for such an increment would come out finite)."""
    import fpde_hpc_gb300 as fp
    N, steps = 200, 140
    A, B, R, u0, alpha, tau, Da, w, rng = _problem(N, steps, tau=tau)
    for tuning in (fp.LineTuning(gemv_splits=1), None):
        line = fp.Line(ctx, N, alpha, tau, Da, A, B, R, u0, steps, tuning=tuning)
        line.run(30)
        u = line.state()
        u[77] = bad
        _write(line, u)
        line.run(34)
        _write(line, np.ascontiguousarray(u0))
        for n in (1, 1, 64):
            line.run(n)
            assert not np.isfinite(line.state()[1:-1]).any(), (tuning is None, n)
        line.reset(u0)                         # an empty history again
        line.run(steps)
        assert np.isfinite(line.state()).all()
        line.close()


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

"""Lines whose inputs hold a NaN, whatever its bits (a 64-bit pattern of ones marks an empty exchange slot of
the block solve and of the Richards step): the result is NaN, not an error. A Richards line whose state the
caller writes between runs: the increment of the next step counts from the last computed state."""
import ctypes as C

import numpy as np
import pytest

from conftest import relmax
from test_gpu_far7 import _problem
from test_gpu_richards_step import _case

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    import fpde_hpc_gb300 as fp
    c = fp.Context(0)
    yield c
    c.close()


ONES = np.array([~np.uint64(0)]).view(np.float64)[0]


@pytest.mark.parametrize("precision,N", [(0, 100), (0, 1000), (3, 1000)])
def test_nan_of_all_ones(ctx, precision, N):
    import fpde_hpc_gb300 as fp
    A, B, R, u0, alpha, tau, Da, w, rng = _problem(N, 3)
    u0 = u0.copy()
    u0.view(np.uint64)[N // 2] = ~np.uint64(0)
    line = fp.Line(ctx, N, alpha, tau, Da, A, B, R, u0, 3, precision=precision)
    line.run(3)
    u = line.state()
    line.close()
    assert np.isnan(u[1:N]).all()


def test_nan_of_all_ones_richards(ctx):
    import fpde_hpc_gb300 as fp
    N, steps = 300, 2
    c = _case(N, steps, False)
    u0 = c["u0"].copy()
    u0.view(np.uint64)[N // 2] = ~np.uint64(0)
    rich = dict(k_form=1, k_sat=2e-6, Z=c["Z"], dL=c["dL"], evaporation=c["E"])
    line = fp.Line(ctx, N, c["alpha"], c["tau"], c["Da"], None, None, None, u0, steps, right=(0, c["u0"][-1]),
                   richards=rich)
    line.run(steps)
    u = line.state()
    line.close()
    assert np.isnan(u[1:N]).all()


def test_richards_state_written_between_runs(ctx):
    """u0 -> u1, the caller writes v, v -> u2 and u2 -> u3: the sum of the third step holds D_0 = u1 - u0 and
    D_1 = u2 - u1. Reference: a line started at u2 whose source is that sum. Tolerance 1e-12 (rounding)."""
    import fpde_hpc_gb300 as fp
    from fpde_hpc_gb300 import weights_l1_lags
    N = 400
    c = _case(N, 3, False)
    rich = lambda E: dict(k_form=1, k_sat=2e-6, Z=c["Z"], dL=c["dL"], evaporation=E)
    mk = lambda u0, steps, E, **kw: fp.Line(ctx, N, c["alpha"], c["tau"], c["Da"], None, None, None, u0, steps,
                                            right=(0, c["u0"][-1]), richards=rich(E), **kw)
    rt = C.CDLL("libcudart.so")
    line = mk(c["u0"], 3, c["E"])
    line.run(1)
    u1 = line.state()
    v = u1.copy()
    v[100:200] *= 1.01
    assert rt.cudaMemcpy(C.c_void_p(line.state_ptr()), v.ctypes.data_as(C.c_void_p), C.c_size_t(v.nbytes), 1) == 0
    assert rt.cudaDeviceSynchronize() == 0
    line.run(1)
    u2 = line.state()
    line.run(1)
    u3 = line.state()
    line.close()
    b = weights_l1_lags(c["alpha"], 3)
    w = c["Da"] * c["tau"] ** -c["alpha"] / (1.0 - c["alpha"]) * b
    S = w[2] * (u1 - c["u0"]) + w[1] * (u2 - u1)
    ref = mk(u2, 1, c["E"][2:], source=S[None, :])
    ref.run(1)
    err = relmax(u3, ref.state())
    ref.close()
    print(f"Richards line after a written state: {err:.2e}")
    assert err <= 1e-12

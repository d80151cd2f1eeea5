"""The FP64 line in 64-step blocks (k_far64 and the persistent block solve with an FP64 near history):
against the oracle at the sizes where its chunks and row slices change (one node, one thread block and
one more, one per SM and one more, the longest line and one more, which takes the per-step form), with
flux ends, sources and restricted summing; runs cut anywhere equal one run bit for bit, also after the
caller has changed the state between runs.

Tolerance: 1e-12, or four times the oracle's response to a one-ulp change of its coefficients and
weights (long fine lines are ill-conditioned)."""
import ctypes as C
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


def _problem(N, steps):
    rng = np.random.default_rng(N)
    k = np.exp(0.3 * rng.standard_normal(N + 1))
    A, B, R = np.zeros(N + 1), np.zeros(N + 1), np.zeros(N + 1)
    A[1:N], B[1:N] = k[:N - 1] * N * N, k[1:N] * N * N
    R[1:N] = A[1:N] + B[1:N]
    x = np.arange(N + 1) / N
    u0 = np.sin(np.pi * x) + 0.3 * rng.random(N + 1)
    alpha, tau = 0.7, 1e-3
    Da = 1.0 / math.gamma(1.0 - alpha)
    j = np.arange(1, steps + 1, dtype=np.float64)
    b = np.concatenate([[1.0], np.exp((1 - alpha) * np.log(j)) * np.expm1((1 - alpha) * np.log1p(1.0 / j))])
    w = Da * tau ** -alpha / (1.0 - alpha) * b
    return A, B, R, u0, alpha, tau, Da, w, rng


@pytest.mark.parametrize("N,steps,left,right,src,lags", [
    (2, 150, (0, 0.3), (0, -0.2), True, 0), (3, 70, (1, 0.1), (1, 0.2), False, 0), (127, 150, (0, 0.0), (0, 0.0), False, 0),
    (128, 200, (1, 0.02), (1, -0.5), True, 0), (129, 200, (0, 0.1), (1, 0.3), False, 0), (1024, 130, (1, 0.0), (0, 0.0), True, 0),
    (1025, 130, (0, 0.0), (1, 0.0), False, 0), (3000, 200, (0, 0.0), (0, 0.0), False, 5), (3000, 260, (0, 0.0), (0, 0.0), True, 90),
    (19456, 80, (0, 0.0), (0, 0.0), False, 0), (19457, 80, (0, 0.0), (0, 0.0), False, 0), (155648, 66, (0, 0.0), (0, 0.0), False, 0),
    (155649, 66, (0, 0.0), (0, 0.0), False, 0)])
def test_blocks_vs_oracle(ctx, N, steps, left, right, src, lags):
    import fpde_hpc_gb300 as fp
    import oracle
    A, B, R, u0, alpha, tau, Da, w, rng = _problem(N, steps)
    S = rng.standard_normal((min(steps, 7), N + 1)) if src else None
    eps = 0.0
    if lags:                                   # keep lags 1 .. lags (kb = w tau / Da falls with the lag)
        eps = 0.5 * (w[lags] + w[lags + 1]) * tau / Da
        w = w.copy()
        w[lags + 1:] = 0.0
    line = fp.Line(ctx, N, alpha, tau, Da, A, B, R, u0, steps, left=left, right=right, dLN=1.0 / N, source=S,
                   restrict_eps=eps)
    out = np.empty(N + 1)
    line.solve_host(u0, steps, out)
    line.reset(u0)
    done = 0
    for n in (1, 1, 34, 28, 3, steps):
        n = min(n, steps - done)
        line.run(n)
        done += n
    pieces = line.state()
    line.close()
    np.testing.assert_array_equal(out, pieces)
    kw = dict(src=S, ltype=left[0], g0=left[1], rtype=right[0], gN=right[1], dLN=1.0 / N)
    ref, _ = oracle.line_run_general(u0, steps, w, 0.0, A, B, R, **kw)
    pert = lambda v: v * (1 + 2.2e-16 * rng.choice([-1, 1], size=v.shape))
    env = relmax(oracle.line_run_general(u0, steps, pert(w), 0.0, pert(A), pert(B), pert(R), **kw)[0], ref)
    err = relmax(out, ref)
    print(f"FP64 blocks N={N} steps={steps} ends {left}{right} src {src} lags {lags}: {err:.2e} (envelope {env:.2e})")
    assert err <= max(1e-12, 4 * env)


def test_state_changed_between_runs(ctx):
    """A caller that writes to the state between two runs inside a block (state_ptr): the next step starts
    from what it wrote, as the per-step form does (tolerance 1e-12 as above)."""
    import fpde_hpc_gb300 as fp
    N, steps = 700, 100
    A, B, R, u0, alpha, tau, Da, w, rng = _problem(N, steps)
    rt = C.CDLL("libcudart.so")
    got = []
    for tuning in (None, fp.LineTuning(gemv_splits=1)):
        line = fp.Line(ctx, N, alpha, tau, Da, A, B, R, u0, steps, tuning=tuning)
        line.run(40)
        u = line.state()
        u[100:300] *= 1.5
        assert rt.cudaMemcpy(C.c_void_p(line.state_ptr()), u.ctypes.data_as(C.c_void_p), C.c_size_t(u.nbytes), 1) == 0
        line.run(steps - 40)
        got.append(line.state())
        line.close()
    assert relmax(got[0], got[1]) <= 1e-12

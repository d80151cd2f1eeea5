"""Kernel probes of FP64 lines in 64-step blocks: every block's far sum (digit slices as the tensor-core
contraction, a window's FP64 rows as the sum over rows) and solve are reported with their bytes and operations;
the run itself is unchanged."""
import numpy as np
import pytest

from test_gpu_far7 import _problem

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("lags", [0, 100])
def test_fp64_block_probes(lags):
    import fpde_hpc_gb300 as fp
    N, steps = 5000, 230
    A, B, R, u0, alpha, tau, Da, w, rng = _problem(N, steps)
    eps = 0.5 * (w[lags] + w[lags + 1]) * tau / Da if lags else 0.0
    with fp.Context(0) as ctx:
        line = fp.Line(ctx, N, alpha, tau, Da, A, B, R, u0, steps, restrict_eps=eps)
        line.run(steps)
        plain = line.state()
        line.set_probe(7)
        line.reset(u0)
        line.run(steps)
        np.testing.assert_array_equal(line.state(), plain)
        got = {k: line.probe_stats(k) for k in (0, 1, 2)}
        line.close()
    far = [n - max(0, n - lags) if lags else n for n in (64, 128, 192)]       # rows of each block's far sum
    kind, size, ops, count = (0, 8, 2 * 64, 3 * 64) if lags else (1, 14, 28 * 2 * 64, 3)
    assert got[1 - kind]["count"] == 0
    assert got[kind]["count"] == count and got[kind]["ms"] > 0
    assert got[kind]["bytes"] == size * sum(far) * (N + 1) and got[kind]["flops"] == ops * sum(far) * (N + 1)
    assert got[2]["count"] == steps and got[2]["ms"] > 0
    near = sum(8 * (N + 1) * (n % 64 + 2) for n in range(steps))               # and the far partials
    assert near <= got[2]["bytes"] <= near + 4 * 8 * (N + 1) * steps and got[2]["flops"] > 0

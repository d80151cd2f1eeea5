"""FP64 ensembles of more than 65,535 columns (a limit of two of a grid's axes): every column's state is that of
the same column in an ensemble of two, bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_many_columns():
    import fpde_hpc_gb300 as fp
    N, n_cols, steps = 6, 65540, 70
    x = np.arange(N + 1) / N
    A, B, R = np.zeros(N + 1), np.zeros(N + 1), np.zeros(N + 1)
    A[1:N] = B[1:N] = 1e3 * (1.0 + 0.5 * np.sin(9 * x[1:N]))
    R[1:N] = 2 * A[1:N]
    col = dict(N=N, alpha=0.7, tau=1e-3, Da=0.3, A=A, B=B, Rlap=R, u0=np.sin(np.pi * x))
    with fp.Context(0) as ctx:
        few = fp.Batch(ctx, [col, col], steps)
        few.run(steps)
        want = few.state(0).copy()
        few.close()
        b = fp.Batch(ctx, [col] * n_cols, steps)
        b.run(steps)
        for k in (0, 32768, 65535, 65536, n_cols - 1):
            np.testing.assert_array_equal(b.state(k), want)
        b.close()

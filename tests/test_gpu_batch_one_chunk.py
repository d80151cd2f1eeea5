"""Ensembles whose columns are all one chunk (at most 1,024 intervals): the sweep finishes the step itself. Their
states equal, bit for bit, those of the same columns beside a longer one, which take the sweep and the join: at
the sizes where a thread's, a warp's and the chunk's nodes end, with both kinds of ends, in FP64 (digit slices,
and rows where a column has a window) and on the split path, in one run and in pieces."""
import numpy as np
import pytest

from test_gpu_batch_chunks import _column

pytestmark = pytest.mark.gpu
KINDS = [((0, 0.0), (0, 0.0)), ((1, 0.05), (1, -0.3)), ((0, 0.2), (1, 0.1)), ((1, 0.0), (0, 0.4))]


@pytest.mark.parametrize("prec,eps", [(0, 0.0), (0, 1e-2), (3, 0.0)])
def test_one_chunk_columns(prec, eps):
    import fpde_hpc_gb300 as fp
    steps = 140
    sizes = (2, 3, 7, 8, 9, 16, 255, 256, 257, 511, 512, 513, 1000, 1023, 1024)
    cols = [_column(N, *KINDS[i % 4], seed=N + i) for i, N in enumerate(sizes)]
    cols[4]["restrict_eps"] = eps
    long = _column(1025, *KINDS[1], seed=5)
    with fp.Context(0) as ctx:
        states = []
        for extra, cuts in (([long], (steps,)), ([], (steps,)), ([], (1, 62, 3, steps - 66))):
            b = fp.Batch(ctx, cols + extra, steps, precision=prec)
            for n in cuts:
                b.run(n)
            states.append([b.state(k).copy() for k in range(len(cols))])
            b.close()
    for s in states[1:]:
        for x, y in zip(s, states[0]):
            np.testing.assert_array_equal(x, y)
    assert all(np.isfinite(x).all() for x in states[0])

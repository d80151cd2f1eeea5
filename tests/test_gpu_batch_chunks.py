"""The ensemble's chunked solve (k_batch_sweep, k_batch_join) against the oracle where its tiling can go
wrong: columns of 1 unknown, of exactly one thread's, one warp's and one chunk's nodes and one more or
less, of 33 chunks and more (several chunks per lane of the joining warp), with both kinds of ends.

Tolerance: 1e-12, or four times the oracle's response to a one-ulp change of a column's coefficients."""
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


def _column(N, left, right, seed):
    rng = np.random.default_rng(seed)
    k = np.exp(0.3 * rng.standard_normal(N + 1))
    A, B, R = np.zeros(N + 1), np.zeros(N + 1), np.zeros(N + 1)
    A[1:N], B[1:N] = k[:N - 1] * N * N, k[1:N] * N * N
    R[1:N] = A[1:N] + B[1:N]
    alpha = float(rng.uniform(0.5, 0.95))
    return dict(N=N, alpha=alpha, tau=1e-3, Da=1.0 / math.gamma(1.0 - alpha), A=A, B=B, Rlap=R, u0=rng.random(N + 1),
                left=left, right=right, dLN=1.0 / N)


@pytest.mark.parametrize("sizes,steps,prec", [
    ((2, 3, 7, 8, 9, 255, 256, 257), 30, 0), ((511, 512, 1023, 1024, 1025, 1031, 1032), 20, 0),
    ((2048, 2049, 4097, 511), 12, 0), ((33 * 1024, 33 * 1024 + 1, 70001, 2), 4, 0), ((300, 1500, 1024, 5000), 64, 3)])
def test_chunks_vs_oracle(ctx, sizes, steps, prec):
    import fpde_hpc_gb300 as fp
    import oracle
    kinds = [((0, 0.0), (0, 0.0)), ((1, 0.05), (1, -0.3)), ((0, 0.2), (1, 0.1)), ((1, 0.0), (0, 0.4))]
    cols = [_column(N, *kinds[i % 4], seed=N + i) for i, N in enumerate(sizes)]
    b = fp.Batch(ctx, cols, steps, precision=prec)
    b.run(1)
    b.run(steps - 1)
    got = [b.state(c) for c in range(len(cols))]
    out = np.zeros(b.total)
    b.solve_host(b.pack([c["u0"] for c in cols]), steps, out)
    for x, y in zip(b.unpack(out), got):
        np.testing.assert_array_equal(x, y)
    b.close()
    rng = np.random.default_rng(1)
    pert = lambda v: v * (1 + 2.2e-16 * rng.choice([-1, 1], size=v.shape))
    for c, u in zip(cols, got):
        run = lambda A, B, R: oracle.line_run(c["u0"], steps, c["tau"], c["alpha"], c["Da"], A, B, R, c["left"][0], c["left"][1],
                                              c["right"][0], c["right"][1], c["dLN"])[0]
        ref = run(c["A"], c["B"], c["Rlap"])
        env = relmax(run(pert(c["A"]), pert(c["B"]), pert(c["Rlap"])), ref)
        err = relmax(u, ref)
        print(f"ensemble column N={c['N']} ends {c['left']}{c['right']} prec {prec}: {err:.2e} (envelope {env:.2e})")
        assert err <= max(1e-12, 4 * env)

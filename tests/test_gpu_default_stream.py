"""Objects created while the default stream is busy (as in any program that queues torch work): the context
runs on a stream of its own that does not wait for the default one, so every clear and copy of a creation has
to be on the context's stream. FP64 lines, ensembles and grids of several 64-step blocks equal, bit for bit,
the same runs on an idle GPU."""
import numpy as np
import pytest

from test_gpu_far7 import _problem

pytestmark = pytest.mark.gpu
STEPS = 200


def _line(ctx):
    import fpde_hpc_gb300 as fp
    A, B, R, u0, alpha, tau, Da, w, rng = _problem(500, STEPS)
    line = fp.Line(ctx, 500, alpha, tau, Da, A, B, R, u0, STEPS)
    line.run(STEPS)
    return line, line.state


def _ensemble(ctx):
    import fpde_hpc_gb300 as fp
    cols = []
    for N in (300, 700):
        A, B, R, u0, alpha, tau, Da, w, rng = _problem(N, STEPS)
        cols.append(dict(N=N, alpha=alpha, tau=tau, Da=Da, A=A, B=B, Rlap=R, u0=u0))
    b = fp.Batch(ctx, cols, STEPS)
    b.run(STEPS)
    return b, lambda: np.concatenate([b.state(k) for k in range(2)])


def _grid(ctx):
    import fpde_hpc_gb300 as fp
    from fpde_hpc_gb300 import problems
    p = problems.config4(n=10, steps=STEPS)
    cA, cB, cR = p.coefs()
    lod = fp.Lod3D(ctx, p.dims, p.alpha, p.tau, p.Da, cA, cB, cR, p.u0, STEPS, left_kind=p.left_kind,
                   right_kind=p.right_kind, dLN=p.dLN)
    lod.run(STEPS)
    return lod, lod.state


@pytest.mark.parametrize("make", [_line, _ensemble, _grid])
def test_busy_default_stream(make):
    torch = pytest.importorskip("torch")
    import fpde_hpc_gb300 as fp
    with fp.Context(0) as ctx:
        obj, state = make(ctx)
        idle = np.array(state())
        obj.close()
        x = torch.rand(4096, 4096, device="cuda")
        torch.cuda.synchronize()
        for _ in range(200):                       # some tenths of a second queued on the default stream
            x = (x @ x).clamp_(0.0, 1.0)
        obj, state = make(ctx)
        busy = np.array(state())
        obj.close()
        torch.cuda.synchronize()
    np.testing.assert_array_equal(busy, idle)

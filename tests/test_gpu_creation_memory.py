"""FP64 objects where the digit slices of the far history do not fit beside everything else: creation falls
back to FP64 rows as long as those fit, and the runs agree with the sliced form to 1e-12 (rounding of the
sums)."""
import numpy as np
import pytest

from conftest import relmax

pytestmark = pytest.mark.gpu
STEPS = 128


@pytest.fixture(scope="module")
def ctx():
    import fpde_hpc_gb300 as fp
    c = fp.Context(0)
    yield c
    c.close()


def _column(N):
    x = np.arange(N + 1) / N
    A, B, R = np.zeros(N + 1), np.zeros(N + 1), np.zeros(N + 1)
    A[1:N] = B[1:N] = 1e3 * (1.0 + 0.5 * np.sin(9 * x[1:N]))
    R[1:N] = 2 * A[1:N]
    return A, B, R, np.sin(np.pi * x)


def _line(ctx):
    import fpde_hpc_gb300 as fp
    N = 150000
    return fp.Line(ctx, N, 0.7, 1e-3, 0.3, *_column(N), STEPS)


def _ensemble(ctx):
    import fpde_hpc_gb300 as fp
    A, B, R, u0 = _column(2000)
    return fp.Batch(ctx, [dict(N=2000, alpha=0.7, tau=1e-3, Da=0.3, A=A, B=B, Rlap=R, u0=u0)] * 300, STEPS)


def _grid(ctx):
    import fpde_hpc_gb300 as fp
    from fpde_hpc_gb300 import problems
    p = problems.config4(n=96, steps=STEPS)
    cA, cB, cR = p.coefs()
    return fp.Lod3D(ctx, p.dims, p.alpha, p.tau, p.Da, cA, cB, cR, p.u0, STEPS, left_kind=p.left_kind,
                    right_kind=p.right_kind, dLN=p.dLN)


def _state(obj):
    obj.run(STEPS)
    s = obj.state()
    return np.concatenate([np.ravel(x) for x in s]) if isinstance(s, (list, tuple)) else np.array(s)


# Per node, for 128 steps: slices 896 bytes and rings of 2,560 (line) or 1,024 bytes; rows 1,024 bytes and 512 of
# far sums or partial sums. The shares of the sliced form's memory that are left lie between the two forms.
@pytest.mark.parametrize("make,shares", [(_line, (0.9, 0.75, 0.6)), (_ensemble, (0.95, 0.88)), (_grid, (0.95, 0.88))])
def test_rows_where_the_slices_do_not_fit(ctx, make, shares):
    torch = pytest.importorskip("torch")
    obj = make(ctx)
    free_with, total = torch.cuda.mem_get_info()
    want = _state(obj)
    obj.close()
    torch.cuda.synchronize()
    free_all = torch.cuda.mem_get_info()[0]
    sliced = free_all - free_with                     # what the sliced form takes
    for share in shares:
        hold = torch.empty(int(free_all - share * sliced), dtype=torch.uint8, device="cuda")
        try:
            obj = make(ctx)
            err = relmax(_state(obj), want)
            obj.close()
            print(f"{make.__name__} with {share:.2f} of {sliced / 1e6:.0f} MB free: {err:.2e}")
            assert err <= 1e-12
        finally:
            del hold
            torch.cuda.empty_cache()

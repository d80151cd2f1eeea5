"""The one-launch Richards step (k_rich_step) at the sizes where its chunking changes: one node, one
warp and one more, the largest lines of 1, 2, 4 and 8 warps per SM (152 SMs) and one interval more
(the last of them on the two-kernel step), Dirichlet and flux right ends, dry and partly saturated
columns, FP64 and split history; against the oracle's sequential restatement.

Tolerance: 1e-12, or four times the oracle's response to a one-ulp change of its node coordinates and
steps where that is larger (the bar of the other Richards line tests)."""
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


def _case(N, steps, wet):
    Z = np.arange(N + 1) * 3.0 / N
    u0 = -0.8 - Z
    if wet:                                    # suction below zero (saturated) over the lower third
        u0 = np.where(Z > 2.0, Z + 0.05, u0)
    E = 2.3e-8 * (1.0 + 0.3 * np.sin(np.arange(steps) * 0.05))
    return dict(Z=Z, dL=np.full(N + 1, 3.0 / N), u0=u0, E=E, alpha=0.8, Da=1.0 / math.gamma(0.2), tau=900.0)


def _oracle(c, steps, kform, rkind, pert=None):
    import oracle
    f = pert or (lambda x: x)
    gN = c["u0"][-1] if rkind == 0 else 0.0
    return oracle.line_run_richards(c["u0"], steps, c["tau"], c["alpha"], c["Da"], f(c["Z"]), f(c["dL"]), kform, 2e-6,
                                    c["E"], rtype=rkind, gN=gN, dLN=c["dL"][-1])[0]


@pytest.mark.parametrize("N,kform,rkind,wet,prec", [
    (2, 1, 0, False, 0), (3, 2, 1, False, 0), (33, 1, 1, False, 0), (34, 1, 0, False, 0), (65, 2, 0, True, 0),
    (200, 1, 1, True, 0), (4865, 1, 0, False, 0), (4866, 2, 1, False, 0), (9729, 1, 0, False, 0),
    (9730, 1, 1, False, 0), (19457, 2, 0, False, 0), (38913, 1, 0, False, 0), (38914, 1, 0, False, 0),
    (1000, 1, 0, False, 3), (10000, 1, 1, False, 3)])
def test_step_sizes_vs_oracle(ctx, N, kform, rkind, wet, prec):
    import fpde_hpc_gb300 as fp
    steps = 20 if N > 9000 else 40
    c = _case(N, steps, wet)
    rich = dict(k_form=kform, k_sat=2e-6, Z=c["Z"], dL=c["dL"], evaporation=c["E"])
    right = (rkind, c["u0"][-1] if rkind == 0 else 0.0)
    line = fp.Line(ctx, N, c["alpha"], c["tau"], c["Da"], None, None, None, c["u0"], steps, right=right,
                   dLN=c["dL"][-1], precision=prec, richards=rich)
    out = np.empty(N + 1)
    line.solve_host(c["u0"], steps, out)
    line.reset(c["u0"])                        # the same again in uneven pieces (slot parity, odd launches)
    line.run(3)
    line.run(steps - 3)
    pieces = line.state()
    line.close()
    np.testing.assert_array_equal(out, pieces)
    ref = _oracle(c, steps, kform, rkind)
    rng = np.random.default_rng(0)
    env = relmax(_oracle(c, steps, kform, rkind, lambda x: x * (1 + 2.2e-16 * rng.choice([-1, 1], size=x.shape))), ref)
    err = relmax(out, ref)
    print(f"Richards step N={N} k_form {kform} right {rkind} wet {wet} prec {prec}: {err:.2e} (envelope {env:.2e})")
    assert err <= max(1e-12, 4 * env)

"""The staged LOD passes (k_lod_pass_st) against the oracle where their tiling can go wrong: line counts
beside multiples of 32, node counts beside multiples of the 4-node groups, lines of 1 and 2 unknowns,
lines near and past the longest that is staged, every mix of line ends, boundary grids and sources; short
grids whose history sum leaves more partial rows than the staged K pass takes; split history.

Tolerance: 1e-12, or four times the oracle's response to a one-ulp change of its coefficients."""
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


@pytest.mark.parametrize("dims,steps,lkind,rkind,bc,src,prec", [
    ((2, 2, 2), 6, (0, 0, 0), (0, 0, 0), True, True, 0), ((3, 2, 4), 30, (1, 0, 1), (0, 1, 1), True, False, 0),
    ((33, 33, 5), 12, (1, 1, 0), (1, 1, 0), False, False, 0), ((34, 9, 6), 12, (0, 1, 0), (1, 0, 0), True, True, 0),
    ((9, 34, 33), 20, (0, 0, 1), (1, 1, 1), True, True, 0), ((12, 12, 12), 40, (1, 1, 1), (0, 0, 0), False, True, 0),
    ((389, 5, 6), 8, (1, 1, 0), (1, 1, 0), False, False, 0), ((4, 5, 420), 8, (0, 0, 1), (0, 0, 1), True, True, 0),
    ((6, 830, 4), 6, (1, 1, 0), (1, 1, 0), False, True, 0), ((900, 4, 5), 6, (0, 1, 0), (1, 1, 0), False, False, 0),
    ((130, 66, 67), 5, (1, 1, 0), (1, 1, 0), True, True, 0), ((17, 22, 35), 60, (1, 1, 0), (1, 1, 0), True, True, 3)])
def test_staged_passes_vs_oracle(ctx, dims, steps, lkind, rkind, bc, src, prec):
    import fpde_hpc_gb300 as fp
    import oracle
    sN, M, K = dims
    rng = np.random.default_rng(sN * 10000 + M * 100 + K)
    shape = (K + 2, M + 2, sN + 2)
    k = np.exp(0.4 * rng.standard_normal(shape))
    h = (1.0 / sN, 1.0 / M, 1.0 / K)
    cA, cB = np.zeros((3,) + shape), np.zeros((3,) + shape)
    for pss, axis in ((0, 2), (1, 1), (2, 0)):
        cA[pss], cB[pss] = np.roll(k, 1, axis=axis) / h[pss] ** 2, k / h[pss] ** 2
    cR = cA + cB
    u0 = rng.random(shape)
    bcg = rng.standard_normal(shape) if bc else None
    rp = rng.standard_normal(shape) if src else None
    alpha, tau = 0.8, 1e-3
    Da = 1.0 / math.gamma(1.0 - alpha)
    lod = fp.Lod3D(ctx, dims, alpha, tau, Da, cA, cB, cR, u0, steps, left_kind=lkind, right_kind=rkind, dLN=h,
                   source=rp, bc=bcg, precision=prec)
    lod.run(steps)
    u = lod.state()
    lod.close()
    args = (dims, u0, steps, tau, alpha, Da)
    kw = dict(rp=rp, bc=bcg, lkind=lkind, rkind=rkind, dLN=h)
    ref = oracle.lod_run(*args, cA, cB, cR, **kw)
    pert = lambda x: x * (1 + 2.2e-16 * rng.choice([-1, 1], size=x.shape))
    env = relmax(oracle.lod_run(*args, pert(cA), pert(cB), pert(cR), **kw), ref)
    err = relmax(u, ref)
    print(f"staged LOD {dims} kinds {lkind}{rkind} bc {bc} src {src} prec {prec}: {err:.2e} (envelope {env:.2e})")
    assert err <= max(1e-12, 4 * env)


@pytest.mark.parametrize("dims,steps,prec", [((128, 128, 128), 64, 3), ((128, 128, 128), 12, 0), ((127, 100, 128), 12, 3)])
def test_staged_passes_on_a_full_chip(ctx, dims, steps, prec):
    """Every SM holds several tiles, so the tiles' warps and copies contend: the same run with the
    segmented passes (another kernel on the same system) gives the same grids. Tolerance: the passes
    differ by rounding, 1e-12 (split runs within their first 64-step block, before the far history
    rounds increments to 24 bits of a block's largest)."""
    import fpde_hpc_gb300 as fp
    from fpde_hpc_gb300 import problems
    sN, M, K = dims
    base = problems.config4(n=128, steps=steps)
    p = problems.LodProblem("lod", dims, base.alpha, base.tau, steps, base.k[:K + 2, :M + 2, :sN + 2].copy(),
                            base.u0[:K + 2, :M + 2, :sN + 2].copy(), base.left_kind, base.right_kind)
    cA, cB, cR = p.coefs()
    out = []
    for seg in ((0, 0, 0), (8, 8, 8)):
        lod = fp.Lod3D(ctx, p.dims, p.alpha, p.tau, p.Da, cA, cB, cR, p.u0, steps, left_kind=p.left_kind,
                       right_kind=p.right_kind, dLN=p.dLN, precision=prec, segments=seg)
        states = []
        for n in (1, 2, steps - 3):
            lod.run(n)
            states.append(lod.state())
        out.append(states)
        lod.close()
    errs = [relmax(x, y) for x, y in zip(*out)]
    print(f"staged against segmented passes, {dims}, precision {prec}: {max(errs):.2e}")
    assert max(errs) <= 1e-12

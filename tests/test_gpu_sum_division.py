"""The series sum's division by tau (fpde_sum, sum_alg 2), which multiplies by a reciprocal and corrects:
with one moment, an unchanged state and gtj = 1 the sum is the moment divided by tau, so every value must be
the FP64 quotient itself (the corrected quotient differs from it only within 2^-52 ulp of the middle of two
doubles). Moments over the whole FP64 range, zeros, infinities; taus with round, random and all-ones
significands, tiny and huge ones, infinity; node counts that leave a partial CTA."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tau", [1.0, 900.0, 1e-3, 0.1, 1.0 / 3.0, np.nextafter(2.0, 0.0), 1.5e-200, 3.1e250, np.inf])
@pytest.mark.parametrize("nodes", [1, 127, 128, 20_003])
def test_quotients(tau, nodes):
    import torch

    import fpde_hpc_gb300 as fp
    rng = np.random.default_rng(nodes)
    h = rng.standard_normal(nodes) * 10.0 ** rng.uniform(-300, 300, nodes)
    h[::7] = rng.standard_normal(len(h[::7]))
    h[5::91] = 0.0
    h[6::97] = np.inf
    ctx = fp.Context(0)
    old = torch.zeros((2, nodes), dtype=torch.float64, device="cuda")
    H = torch.from_numpy(h.reshape(nodes, 1).copy()).cuda()
    S = ctx.sum_alg(2, old, torch.tensor([tau], dtype=torch.float64, device="cuda"), sum_param=1, Htmp=H,
                    row2=torch.ones(1, dtype=torch.float64, device="cuda"), gtj=1.0, gt=1.0, alpha=0.8).cpu().numpy()
    with np.errstate(all="ignore"):
        want = h / tau
    assert np.array_equal(S, want, equal_nan=True)
    ctx.close()

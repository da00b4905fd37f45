"""The mixed VJP at the edges of its tiles (512 targets), chunks (128 sources), chains of
the centre (256) and splits, equal and unequal masses, against the FP64 VJP.  Tolerance of
every mixed VJP: 1e-5 of the gradient's norm."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 2, 31, 128, 129, 255, 257, 512, 513, 2047, 2049, 5000, 16384, 20001])
@pytest.mark.parametrize("equal", [True, False])
def test_sizes(lib, cuda, n, equal):
    import torch

    from gravhopper_gb300 import engine
    rng = np.random.default_rng(n)
    x, lam = (torch.from_numpy(rng.normal(size=(n, 3))).to(cuda) for _ in range(2))
    x += 3.0  # a centre to subtract
    m = torch.full((n,), 0.3, dtype=torch.float64, device=cuda)
    if not equal:
        m = m * torch.from_numpy(rng.uniform(0.5, 2.0, n)).to(cuda)
    got = engine.direct_vjp(x, m, 0.05, lam, precision="mixed")
    ref = engine.direct_vjp(x, m, 0.05, lam)
    for a, b in zip(got, ref):
        assert float((a - b).norm()) <= 1e-5 * float(b.norm()) + 1e-300
    again = engine.direct_vjp(x, m, 0.05, lam, precision="mixed")
    assert torch.equal(again[0], got[0]) and torch.equal(again[1], got[1])

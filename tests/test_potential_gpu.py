"""The potential's pair kernel where its blocks of 128 particles end, against plain
PyTorch FP64.  Tolerance: each of up to n terms of one sign is rounded to 1.25 * 2^-53, and
sums of n terms in any order err by at most n 2^-53 of their magnitude; both sides do, so
rel <= (2 n + 3) 2^-53 bounds the difference (4e-12 at the largest size here)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def dense(torch, x, m, eps):
    out = torch.empty_like(m)
    for a in range(0, len(m), 1024):
        d = x[None] - x[a:a + 1024, None]
        s = (d * d).sum(2) + eps * eps
        y = torch.where(s > 0, s, torch.ones_like(s)).rsqrt() * (s > 0)
        k = torch.arange(s.shape[0], device=x.device)
        y[k, a + k] = 0.0
        out[a:a + 1024] = -(y * m).sum(1)
    return out


# 1 block; 2 (even, d = 1 for the lower row only), 3, 4; a last block of 1 particle; many
@pytest.mark.parametrize("n", [1, 2, 127, 128, 129, 256, 257, 384, 385, 512, 1000, 17001])
@pytest.mark.parametrize("eps", [0.0, 0.03])
def test_sizes(lib, cuda, n, eps):
    import torch

    from gravhopper_gb300 import engine
    rng = np.random.default_rng(n)
    x = torch.from_numpy(rng.normal(size=(n, 3))).to(cuda)
    m = torch.from_numpy(rng.uniform(0.1, 10.0, n)).to(cuda)
    if n > 200:
        x[3] = x[150]  # a coincident pair in one block, and one across blocks
        x[n - 1] = x[5]
    got = engine.potential(x, m, eps)
    ref = dense(torch, x, m, eps)
    torch.testing.assert_close(got, ref, rtol=(2 * n + 3) * 2.0 ** -53, atol=0.0)
    assert torch.equal(engine.potential(x, m, eps), got)


@pytest.mark.parametrize("scale", [1e-60, 1e60, 1e170])
def test_scales(lib, cuda, scale):
    """Inside and outside the fixed-point range; 1e170: the squared distance overflows
    and the result is not finite, as in FP64 arithmetic throughout."""
    import torch

    from gravhopper_gb300 import engine
    rng = np.random.default_rng(3)
    x = torch.from_numpy(rng.normal(size=(300, 3))).to(cuda)
    m = torch.from_numpy(rng.uniform(0.1, 10.0, 300)).to(cuda)
    got = engine.potential(x * scale, m, 0.1 * scale)
    if scale > 1e150:
        assert not torch.isfinite(got).any()
    else:
        torch.testing.assert_close(got * scale, dense(torch, x, m, 0.1), rtol=700 * 2.0 ** -53, atol=0.0)

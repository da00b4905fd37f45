"""The potential of small systems: two launches for one block of particles, as few as the
sum over ordered pairs took (its largest coordinate is found by the pair kernel itself),
and shares of a pair of blocks at the sizes where their number changes, against NumPy sums
in long double.  Tolerance: terms of one sign within 1.25 * 2^-53 each, n - 1 additions."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def potential(x, m, eps):
    import torch

    from gravhopper_gb300 import engine
    return engine.potential(torch.from_numpy(x).cuda(), torch.from_numpy(m).cuda(), eps).cpu().numpy()


@pytest.mark.parametrize("n,launches", [(1, 2), (30, 2), (128, 2), (129, 3)])
def test_launches(lib, cuda, n, launches):
    from gravhopper_gb300 import _capi
    rng = np.random.default_rng(n)
    x, m = rng.normal(size=(n, 3)), rng.uniform(1, 2, n)
    potential(x, m, 0.1)
    before = _capi.launch_count()
    potential(x, m, 0.1)
    assert _capi.launch_count() - before == launches


# one block in 32 shares; blocks: 2, 3 (32 shares), 4 and 24 (8 shares), 25 (whole)
@pytest.mark.parametrize("n", [1, 2, 5, 96, 127, 128, 129, 384, 385, 3072, 3073])
@pytest.mark.parametrize("scale,eps", [(1.0, 0.0), (1.0, 0.03), (1e-60, 0.0)])
def test_shares(lib, cuda, n, scale, eps):
    rng = np.random.default_rng(n)
    x, m = rng.normal(size=(n, 3)) * scale, rng.uniform(0.1, 10.0, n)
    got = potential(x, m, eps)
    rows = rng.permutation(n)[:200]
    d = x[None].astype(np.longdouble) - x[rows, None]
    s = (d * d).sum(2) + np.longdouble(eps * eps)
    s[np.arange(len(rows)), rows] = 1
    y = 1 / np.sqrt(s)
    y[np.arange(len(rows)), rows] = 0
    ref = -(y * m).sum(1)
    assert np.all(np.abs(got[rows] - ref) <= (n + 3) * 2.0 ** -53 * np.abs(ref))

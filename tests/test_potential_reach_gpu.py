"""The potential of a compact system with one particle so far away that ordinary separations
and softenings lie near 2^-31 of the box, where the fixed-point pair distance ends, against
plain NumPy sums in long double.  Tolerance: each of the n - 1 terms of one sign is within
1.25 * 2^-53 (1.5 * 2^-52 where FP64 operations form it: differences, three products, the
root), and their sum errs by at most n 2^-53 of its magnitude."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


# |x| < 2^E with E = 32: the fixed-point pairs end at sqrt(d^2 + eps^2) = 2
@pytest.mark.parametrize("eps", [0.0, 1e-9, 0.9, 1.0, 1.5, 2.0, 2.5])
@pytest.mark.parametrize("n", [100, 300])
def test_far_particle(lib, cuda, n, eps):
    import torch

    from gravhopper_gb300 import engine
    rng = np.random.default_rng(n)
    x = rng.normal(size=(n, 3)) * np.exp(rng.uniform(np.log(0.2), np.log(8.0), (n, 1)))
    x[n // 2] = [1.0, 2.0 ** 31, -3.0]
    m = rng.uniform(0.1, 10.0, n)
    got = engine.potential(torch.from_numpy(x).to(cuda), torch.from_numpy(m).to(cuda), eps).cpu().numpy()
    d = x[None].astype(np.longdouble) - x[:, None]
    s = (d * d).sum(2) + np.longdouble(eps * eps)
    np.fill_diagonal(s, 1)
    y = 1 / np.sqrt(s)
    np.fill_diagonal(y, 0)
    ref = -(y * m).sum(1)
    assert np.max(np.abs((got - ref) / ref)) <= (n + 3) * 2.0 ** -53

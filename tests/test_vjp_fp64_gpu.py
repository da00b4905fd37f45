"""The FP64 VJP where its blocks of 128 particles are one, whole, ragged, odd and even in
number, and where the shares of a pair of blocks change, against NumPy sums of the same
formula.  Tolerance: some 40 roundings of 2^-53 per term and those of n sums, of the sum of
the terms' magnitudes: (40 + n) 2^-53."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


# blocks: 1, 2, 3, 4 (32 shares below 3), 8, 9; 48 and 49 (1200 pairs of blocks and more: whole)
@pytest.mark.parametrize("n", [1, 2, 127, 128, 129, 255, 256, 257, 384, 385, 512, 1000, 1025, 6016, 6145])
@pytest.mark.parametrize("eps", [0.0, 0.05])
def test_blocks(lib, cuda, n, eps):
    import torch
    from gravhopper_gb300 import engine, ics
    ic = ics.plummer(n, b=1.0, totmass=1.0, seed=21)
    rng = np.random.default_rng(22)
    x, m, lam = ic["pos"], rng.uniform(0.5, 2.0, n) / n, rng.normal(size=(n, 3))
    t = lambda a: torch.from_numpy(a).cuda()
    gp, gm = (a.cpu().numpy() for a in engine.direct_vjp(t(x), t(m), eps, t(lam), precision="fp64"))
    rows = rng.permutation(n)[:512]
    g, gs, w, ws = np.zeros((n, 3)), np.zeros((n, 3)), np.zeros(n), np.zeros(n)
    tol = (40 + n) * 2.0 ** -53
    for k in rows:
        d = x - x[k]
        s = (d * d).sum(1) + eps * eps
        s[k] = 1.0
        q = s ** -1.5
        q[k] = 0.0
        u = m[k] * lam - m[:, None] * lam[k]
        size = m[k] * np.abs(lam) + m[:, None] * np.abs(lam[k])
        p = 3 * q / s
        g[k] = (q[:, None] * u - (p * (d * u).sum(1))[:, None] * d).sum(0)
        gs[k] = (q[:, None] * size + (p * (np.abs(d) * size).sum(1))[:, None] * np.abs(d)).sum(0)
        w[k] = -(q * (lam * d).sum(1)).sum()
        ws[k] = (q * (np.abs(lam) * np.abs(d)).sum(1)).sum()
    assert np.all(np.abs(gp - g)[rows] <= tol * gs[rows])
    assert np.all(np.abs(gm - w)[rows] <= tol * ws[rows])

"""The mixed tree walk where its loop of 32 steps per fold ends early, exactly and late:
systems of one particle up to some folds, against the oracle tree.  Tolerance: an
interaction's eight FP32 roundings and the 31 of a fold's partial sums, each 2^-24 of the
sum of the magnitudes, so 2^-18.7 of it at most."""
import numpy as np
import pytest

from oracle import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 2, 16, 17, 31, 32, 33, 48, 64, 65, 129])
@pytest.mark.parametrize("theta", [0.0, 0.7, 1.0])
def test_folds(lib, cuda, n, theta):
    import torch
    from gravhopper_gb300 import engine, ics
    ic = ics.plummer(n, b=1.0, totmass=1.0, seed=12)
    pos, mass, eps = ic["pos"], ic["mass"], 0.05
    got = engine.tree_force(torch.from_numpy(pos).cuda(), torch.from_numpy(mass).cuda(), eps, theta,
                            precision="mixed").cpu().numpy()
    ref = oracle.tree_force(pos, mass, eps, theta)
    r = np.linalg.norm(pos[:, None] - pos[None], axis=2)
    scale = (mass[None] * r / (r * r + eps * eps) ** 1.5).sum(1)
    assert np.all(np.linalg.norm(got - ref, axis=1) <= 2.0 ** -18.6 * scale)

"""The ensemble's default tiles (one warp, chunks of 128 sources) against the 128-thread
tiles whose chunks they share: the same bits, at the ends of tiles and chunks, with equal
and unequal masses and with no softening."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("eps", [0.05, 0.0])
@pytest.mark.parametrize("equal", [True, False])
def test_same_bits_as_128_thread_tiles(lib, cuda, eps, equal):
    import torch

    from gravhopper_gb300.ensemble import Ensemble
    rng = np.random.default_rng(11)
    systems = []
    for n in (1, 2, 31, 127, 128, 129, 255, 256, 257, 511, 513, 1000, 2049):
        m = np.full(n, 2.0) if equal else rng.uniform(0.5, 2.0, n)
        systems.append({"pos": rng.normal(size=(n, 3)) + 5.0, "vel": rng.normal(size=(n, 3)), "mass": m, "eps": eps,
                        "dt": 1e-3})
    a, b = Ensemble(systems, device=cuda), Ensemble(systems, device=cuda)
    a.run(5, config=0)
    b.run(5)
    assert torch.equal(a.pos, b.pos) and torch.equal(a.vel, b.vel)
    assert torch.isfinite(a.pos).all()

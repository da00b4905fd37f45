"""Which build small systems get after ties beyond two key words, by the kernels launched:
every count of particles has its own memory of them, and loses it."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def force_launches(pos):
    import torch

    from gravhopper_gb300 import _capi, engine
    x = torch.from_numpy(pos).cuda()
    m = torch.ones(len(pos), dtype=torch.float64, device="cuda")
    before = _capi.launch_count()
    engine.tree_force(x, m, 1e-3, 0.7)
    return _capi.launch_count() - before


def tied(rng, n):
    base = rng.uniform(-1, 1, size=(n // 2, 3))
    return np.concatenate([base, base + 1e-13 * rng.normal(size=base.shape)])


def test_two_counts_that_tie_take_turns(lib, cuda):
    rng = np.random.default_rng(1)
    a, b = tied(rng, 612), tied(rng, 614)
    for p in (a, b):
        force_launches(p)
        force_launches(p)
    alone = {len(p): force_launches(p) for p in (b, a)}
    for p in (b, a, b, a):
        assert force_launches(p) == alone[len(p)]


def test_ordinary_systems_get_the_small_build_back(lib, cuda):
    rng = np.random.default_rng(2)
    small = force_launches(rng.normal(size=(621, 3)))
    force_launches(tied(rng, 620))
    assert force_launches(tied(rng, 620)) > small
    x = rng.normal(size=(620, 3))
    for _ in range(8):
        last = force_launches(x)
    assert last == small


def test_tied_and_ordinary_of_one_count_take_turns(lib, cuda):
    """The general build throughout: none is made in vain."""
    rng = np.random.default_rng(3)
    t, x = tied(rng, 630), rng.normal(size=(630, 3))
    force_launches(t)
    general = force_launches(t)
    for _ in range(4):
        force_launches(x)
        assert force_launches(t) == general

"""The fixed-point pair factors of the FP64 tree walk and the potential as the GPU forms them
(its own FP32 reciprocal square root as the seed, whose range nothing checks there) against
long double, over the inputs of the host checks and where the factors end.  Bound as on the
host: 1.25 half-ulps (2^-53 of the value each)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
N = 400_000
MASS_INV_CUBE, INV_DISTANCE, FIX96 = range(3)


def worst(kind, rows, want):
    """(largest error in half-ulps, refused) of the device's factors."""
    import torch

    from gravhopper_gb300 import _capi
    got = _capi.check_pair_factor(kind, torch.from_numpy(np.ascontiguousarray(rows)).cuda()).cpu().numpy()
    took = ~np.isnan(got)
    err = np.abs((got[took].astype(np.longdouble) - want[took]) / want[took]) * 2.0 ** 53
    return (float(err.max()) if took.any() else 0.0), ~took


def binades(rng, shape, lo, hi):
    return rng.choice([-1.0, 1.0], shape) * np.ldexp(1.0 + rng.random(shape), rng.integers(lo, hi + 1, shape))


# ordinary offsets; components far apart; softening from far below to far above them; zero
# components; zero offset; the edges of the range
@pytest.mark.parametrize("mode", range(6))
@pytest.mark.parametrize("kind", [MASS_INV_CUBE, INV_DISTANCE])
def test_differences(lib, cuda, kind, mode):
    rng = np.random.default_rng(10 * kind + mode)
    d, eps = binades(rng, (N, 3), 0, 5), np.where(rng.random(N) < 0.3, 0.0, np.abs(binades(rng, N, -3, -3)))
    m = binades(rng, N, -30, 30)
    if mode == 1:
        d = binades(rng, (N, 3), -100, 100)
    if mode == 2:
        eps = np.abs(binades(rng, N, -100, 100))
    if mode == 3:
        d[np.arange(N), rng.integers(0, 3, N)] = rng.choice([0.0, -0.0], N)
    if mode == 4:
        d[:] = 0.0
        eps = np.abs(binades(rng, N, -100, 100))
    if mode == 5:
        d = np.where(rng.random((N, 1)) < 0.5, binades(rng, (N, 3), -150, -149), binades(rng, (N, 3), 149, 150))
        m = np.where(rng.random(N) < 0.5, binades(rng, N, -500, -500), binades(rng, N, 500, 500))
        eps = np.where(rng.random(N) < 0.5, 0.0, 2.0 ** -149)
    s = (d.astype(np.longdouble) ** 2).sum(1) + (eps * eps).astype(np.longdouble)
    rows = np.concatenate([d, (eps * eps)[:, None]] + ([m[:, None]] if kind == MASS_INV_CUBE else []), axis=1)
    err, refused = worst(kind, rows, m / (s * np.sqrt(s)) if kind == MASS_INV_CUBE else 1 / np.sqrt(s))
    assert not refused.any() and err < 1.25


def test_out_of_range_is_refused(lib, cuda):
    bad = [np.nan, np.inf, -np.inf, 2.0 ** 152, 1e300]
    d = np.tile([1.0, -2.0, 3.0], (15, 1))
    for k, v in enumerate(bad):
        for c in range(3):
            d[3 * k + c, c] = v
    for kind, rows in ((MASS_INV_CUBE, np.concatenate([d, np.full((15, 1), 0.01), np.ones((15, 1))], 1)),
                       (INV_DISTANCE, np.concatenate([d, np.full((15, 1), 0.01)], 1))):
        assert worst(kind, rows, np.ones(15))[1].all()
    masses = np.array([0.0, -0.0, 1e-310, 1e200, np.nan, np.inf])
    rows = np.concatenate([np.tile([1.0, 2.0, 3.0, 0.01], (6, 1)), masses[:, None]], 1)
    assert worst(MASS_INV_CUBE, rows, np.ones(6))[1].all()


# positions over the box; softening as large as the box; sqrt(d^2 + eps^2) from 2^-33 to
# 2^-29 of the box, without softening and with
@pytest.mark.parametrize("mode", range(4))
def test_fixed_point_positions(lib, cuda, mode):
    rng = np.random.default_rng(30 + mode)
    E = rng.integers(-60, 121, N)
    box = np.ldexp(1.0, E)
    a, b = (box[:, None] * rng.uniform(-0.99, 0.99, (N, 3)) for _ in range(2))
    eps = box * np.ldexp(1.0 + rng.random(N), -1 - rng.integers(0, 29, N))
    if mode == 1:
        eps = box * rng.uniform(0.5, 0.99, N)
    if mode > 1:
        reach = box * np.exp2(rng.uniform(-33.0, -29.0, N))
        share = np.ones(N) if mode == 2 else rng.uniform(0.0, 0.999, N)
        u = rng.normal(size=(N, 3))
        a = 2.0 ** -20 * a
        b = a + (reach * np.sqrt(share) / np.linalg.norm(u, axis=1))[:, None] * u
        eps = reach * np.sqrt(1.0 - share)
    s = ((a.astype(np.longdouble) - b) ** 2).sum(1) + (eps * eps).astype(np.longdouble)
    err, refused = worst(FIX96, np.concatenate([a, b, (eps * eps)[:, None], E[:, None]], 1), 1 / np.sqrt(s))
    assert err < 1.25
    assert abs(int(refused.sum()) - int((np.sqrt(s) < box * np.longdouble(2.0) ** -31).sum())) <= N // 100_000

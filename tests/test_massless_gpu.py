"""Tree forces of systems with massless particles (tracers), in the FP64 walk's integer
factor and outside its range, against the oracle tree.  Tolerance as for every FP64 tree
force: rms <= 1e-12, max <= 1e-9 per particle; a cell of massless particles alone has no
centre of mass, and forces that accept one are NaN in both."""
import numpy as np
import pytest

from oracle import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("scale", [1.0, 1e-50])
@pytest.mark.parametrize("eps", [0.0, 0.03])
@pytest.mark.parametrize("n,share", [(700, 0.01), (700, 0.5), (9000, 0.2), (9000, 1.0)])
def test_massless(lib, cuda, n, share, eps, scale):
    from gravhopper_gb300 import _jbgrav, ics
    ic = ics.plummer(n, b=1.0, totmass=1.0, seed=n)
    rng = np.random.default_rng(4)
    mass = np.where(rng.random(n) < share, rng.choice([0.0, -0.0], n), ic["mass"])
    pos = ic["pos"] * scale
    got = _jbgrav.tree_force(pos, mass, eps * scale, 0.6)
    ref = oracle.tree_force(pos, mass, eps * scale, 0.6)
    np.testing.assert_array_equal(np.isnan(got), np.isnan(ref))
    ok = np.isfinite(ref).all(axis=1)
    got, ref = got[ok] * scale ** 2, ref[ok] * scale ** 2
    num, den = np.linalg.norm(got - ref, axis=1), np.linalg.norm(ref, axis=1)
    assert np.all(num[den == 0] == 0)
    if np.any(den > 0):
        r = num[den > 0] / den[den > 0]
        assert np.sqrt(np.mean(r * r)) <= 1e-12 and r.max() <= 1e-9

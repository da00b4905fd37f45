"""The FP64 tree walk where its interaction changes form (scales inside and outside the
fixed-point factor's range, with and without softening) and where its split over warps
does (numbers of target groups, sorted and unsorted points), against the oracle tree.
Tolerance as for every FP64 tree force: rms <= 1e-12, max <= 1e-9 per particle."""
import numpy as np
import pytest

from oracle import oracle

pytestmark = pytest.mark.gpu


def check(got, ref):
    num, den = np.linalg.norm(got - ref, axis=1), np.linalg.norm(ref, axis=1)
    assert np.all(num[den == 0] == 0)
    if not np.any(den > 0):
        return
    r = num[den > 0] / den[den > 0]
    assert float(np.sqrt(np.mean(r * r))) <= 1e-12 and r.max() <= 1e-9, (np.sqrt(np.mean(r * r)), r.max())


# 1e-50, 1e44: differences below 2^-150 and near 2^147, where some pairs leave the range
@pytest.mark.parametrize("scale", [1e-50, 1e-45, 1e-3, 1.0, 1e44])
@pytest.mark.parametrize("eps", [0.0, 0.05])
def test_scales(lib, cuda, scale, eps):
    from gravhopper_gb300 import _jbgrav, ics
    ic = ics.plummer(700, b=1.0, totmass=1.0, seed=4)
    pos = ic["pos"] * scale
    got = _jbgrav.tree_force(pos, ic["mass"], eps * scale, 0.6)
    check(got * scale * scale, oracle.tree_force(pos, ic["mass"], eps * scale, 0.6) * scale * scale)


def test_signs_and_sizes_of_masses(lib, cuda):
    from gravhopper_gb300 import _jbgrav, ics
    ic = ics.plummer(500, b=1.0, totmass=1.0, seed=5)
    rng = np.random.default_rng(6)
    mass = ic["mass"] * 10.0 ** rng.uniform(-170, 150, 500)  # beyond 2^+-500 at both ends
    check(_jbgrav.tree_force(ic["pos"], mass, 0.05, 0.0), oracle.tree_force(ic["pos"], mass, 0.05, 0.0))


# 8193: no small build, 8704 and 8705: tiles of 512 in the moments' sums
# groups of 32 targets: 1, 2, 5, 63, 1024, 1025, 2048, 2816 (11 warps each), 2817 (two)
@pytest.mark.parametrize("n", [1, 2, 32, 33, 129, 2000, 8193, 8704, 8705, 32768, 32769, 65536, 90112, 90113])
def test_particles(lib, cuda, n):
    from gravhopper_gb300 import _jbgrav, ics
    ic = ics.hernquist_disk(n, seed=7)
    got = _jbgrav.tree_force(ic["pos"], ic["mass"], 0.1, 0.7)
    check(got, oracle.tree_force(ic["pos"], ic["mass"], 0.1, 0.7))
    np.testing.assert_array_equal(_jbgrav.tree_force(ic["pos"], ic["mass"], 0.1, 0.7), got)


# 8191 points keep their order, from 8192 they are sorted; 1 and 2 particles: every range
# but one is empty
@pytest.mark.parametrize("n,points", [(3000, 1), (3000, 31), (3000, 33), (3000, 8191), (3000, 8192), (3000, 33000), (3000, 90113),
                                      (1, 40), (2, 9000)])
def test_points(lib, cuda, n, points):
    from gravhopper_gb300 import _jbgrav, ics
    ic = ics.plummer(n, b=1.0, totmass=1.0, seed=8)
    rng = np.random.default_rng(9)
    fp = ic["pos"][rng.integers(0, n, points)] * rng.uniform(0.5, 3.0, (points, 1)) + rng.normal(0, 0.1, (points, 3))
    fp[::7] *= 50.0  # some outside the root cell
    got = _jbgrav.tree_force_position(ic["pos"], ic["mass"], fp, 0.01, 0.5)
    check(got, oracle.tree_force_position(ic["pos"], ic["mass"], fp, 0.01, 0.5))
    np.testing.assert_array_equal(_jbgrav.tree_force_position(ic["pos"], ic["mass"], fp, 0.01, 0.5), got)

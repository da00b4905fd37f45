"""The ordered FP64 direct sum with each number of targets per block it uses (2, 4, 5, 7, 8,
by the number of targets), whole and partial blocks and chunks: bit for bit the oracle."""
import numpy as np
import pytest

from oracle import oracle

pytestmark = pytest.mark.gpu


# 152 SMs: 2 targets up to ~300, 4 to ~600, 5 and 7 between, 8 from ~2200 with gaps
@pytest.mark.parametrize("nt", [1, 2, 5, 303, 305, 607, 609, 700, 761, 1063, 1065, 1500, 1520, 2000, 2127, 2129, 4001])
@pytest.mark.parametrize("np_", [1, 55, 57, 64, 65, 90, 300])
def test_points(lib, cuda, nt, np_):
    from gravhopper_gb300 import _jbgrav
    rng = np.random.default_rng(nt * 1000 + np_)
    pos, mass, fp = rng.normal(size=(np_, 3)), rng.uniform(0.5, 2.0, np_), rng.normal(size=(nt, 3))
    np.testing.assert_array_equal(_jbgrav.direct_summation_position(pos, mass, fp, 0.05),
                                  oracle.direct_summation_position(pos, mass, fp, 0.05))


@pytest.mark.parametrize("n", [3, 300, 609, 1500, 2000, 2999])
def test_self(lib, cuda, n):
    from gravhopper_gb300 import _jbgrav
    rng = np.random.default_rng(n)
    pos, mass = rng.normal(size=(n, 3)), rng.uniform(0.5, 2.0, n)
    np.testing.assert_array_equal(_jbgrav.direct_summation(pos, mass, 0.0), oracle.direct_summation(pos, mass, 0.0))

"""The build of small systems (up to 8192 particles) at the edges of its blocks, its size
range and its ways out: the reference tree's cell count, the tree's invariants, and
forces by the tolerance of every FP64 tree force (rms <= 1e-12, max <= 1e-9)."""
import numpy as np
import pytest

from oracle import oracle

pytestmark = pytest.mark.gpu


def same_tree(pos, mass, eps, forces=True):
    import torch

    from gravhopper_gb300 import _capi, _jbgrav
    d = torch.device("cuda:0")
    v = _capi.tree_validate(torch.from_numpy(pos).to(d), torch.from_numpy(mass).to(d), eps)
    ref, cells = oracle.tree_force(pos, mass, eps, 0.6, return_nodes=True)
    assert v["leaves"] == len(mass) and v["cells"] == cells, v
    assert all(v[k] == 0 for k in v if k not in ("cells", "leaves")), v
    if not forces:
        return
    got = _jbgrav.tree_force(pos, mass, eps, 0.6)
    num, den = np.linalg.norm(got - ref, axis=1), np.linalg.norm(ref, axis=1)
    assert np.all(num[den == 0] == 0)
    if np.any(den > 0):
        r = num[den > 0] / den[den > 0]
        assert np.sqrt(np.mean(r * r)) <= 1e-12 and r.max() <= 1e-9


# blocks of 64 (cells), 256 (keys, moments), 1024 (rank, layout); 8193: the general build
@pytest.mark.parametrize("n", [1, 2, 3, 63, 64, 65, 255, 257, 1023, 1024, 1025, 2049, 8191, 8192, 8193])
def test_sizes(lib, cuda, n):
    from gravhopper_gb300 import ics
    ic = ics.plummer(n, b=1.0, totmass=1.0, seed=n)
    rng = np.random.default_rng(n)
    same_tree(ic["pos"], ic["mass"] * rng.uniform(0.5, 2.0, n), 0.02)


def test_far_from_the_origin(lib, cuda):
    """Every key by the recurrence: the system is 4000 times its size off the origin.
    The reference's centres of mass are rounded sums of m x there, 2^-53 of |x| each, so
    its forces (3e-12 from exact sums' here) say nothing at this tolerance; its cells do."""
    rng = np.random.default_rng(1)
    same_tree(rng.normal(size=(3000, 3)) + [1e4, -2e4, 3e4], rng.uniform(1, 2, 3000), 0.02, forces=False)


def test_more_nodes_than_room(lib, cuda):
    """Pairs 2^-36 of the box apart: chains of some 30 cells each, more nodes than the
    build first makes room for; then an ordinary system of the same size."""
    rng = np.random.default_rng(2)
    base = rng.uniform(-1, 1, size=(1500, 3))
    pos = np.concatenate([base, base + 2.0 ** -35 * rng.uniform(0.5, 1.0, size=base.shape)])
    same_tree(pos, np.ones(3000), 1e-3)
    same_tree(rng.normal(size=(3000, 3)), np.ones(3000), 1e-3)


def test_ties_then_ordinary(lib, cuda):
    """Pairs below the 42nd level need wider keys (the general build); then a system of
    the same size, and one of another."""
    rng = np.random.default_rng(3)
    base = rng.uniform(-1, 1, size=(200, 3))
    same_tree(np.concatenate([base, base + 1e-13 * rng.normal(size=base.shape)]), np.ones(400), 1e-3)
    same_tree(rng.normal(size=(400, 3)), np.ones(400), 1e-3)
    same_tree(rng.normal(size=(401, 3)), np.ones(401), 1e-3)


def test_run_stops_at_a_bad_step(lib, cuda):
    """A step whose build is refused leaves the state of the steps before it."""
    import torch

    from gravhopper_gb300 import _capi, engine, ics
    ic = ics.plummer(500, seed=4)
    x, v, m = (torch.from_numpy(ic[k]).to(cuda) for k in ("pos", "vel", "mass"))
    v[7] = 1e308  # finite; the second half-drift overflows
    x0, v0 = x.clone(), v.clone()
    with pytest.raises(_capi.EngineError) as err:
        engine.run_dkd(x, v, m, 3, 1e10, 5e-5, algorithm="tree")
    assert err.value.code == _capi.GH_ERR_ARG
    torch.cuda.synchronize()
    assert torch.equal(x, x0) and torch.equal(v, v0)

"""Sums over unordered pairs whose column sums do not fit the scratch at once (several
launches that add to one result), at the sizes where that begins and where memory is
short, and the FP64 tree walk when the scratch that splits it cannot be had.

Reference: sampled rows in long double.  Tolerances: potential, terms of one sign within
1.25 * 2^-53 each and n additions; VJP, some 40 roundings per term and n additions, of the
sum of the terms' magnitudes; tree, rms <= 1e-12 and max <= 1e-9 per particle."""
import numpy as np
import pytest

from oracle import oracle

pytestmark = pytest.mark.gpu


@pytest.fixture
def fail_after():
    """fail_after(passed, failed): the next reservations pass, then some run out of memory."""
    from gravhopper_gb300 import _capi

    def arm(passed, failed):
        _capi.inject(_capi.GH_INJECT_ALLOC_PASS, passed)
        _capi.inject(_capi.GH_INJECT_ALLOC, failed)

    yield arm
    arm(0, 0)


def system(n):
    from gravhopper_gb300 import ics
    rng = np.random.default_rng(n)
    ic = ics.plummer(n, b=1.0, totmass=1.0, seed=n)
    return ic["pos"], ic["mass"] * rng.uniform(0.5, 2.0, n), rng.normal(size=(n, 3)), rng.permutation(n)[:48]


def check_potential(x, m, rows, eps=0.01):
    import torch

    from gravhopper_gb300 import engine
    n = len(m)
    got = engine.potential(torch.from_numpy(x).cuda(), torch.from_numpy(m).cuda(), eps).cpu().numpy()
    assert np.isfinite(got).all()
    for k in rows:
        d = x.astype(np.longdouble) - x[k]
        y = 1 / np.sqrt((d * d).sum(1) + np.longdouble(eps * eps))
        y[k] = 0
        ref = -(y * m).sum()
        assert abs(got[k] - ref) <= (n + 3) * 2.0 ** -53 * abs(ref)


def check_vjp(x, m, lam, rows, eps=0.01):
    import torch

    from gravhopper_gb300 import engine
    n = len(m)
    t = lambda a: torch.from_numpy(a).cuda()
    gp, gm = (a.cpu().numpy() for a in engine.direct_vjp(t(x), t(m), eps, t(lam)))
    assert np.isfinite(gp).all() and np.isfinite(gm).all()
    tol = (40 + n) * 2.0 ** -53
    for k in rows:
        d = x.astype(np.longdouble) - x[k]
        s = (d * d).sum(1) + np.longdouble(eps * eps)
        q = 1 / (s * np.sqrt(s))
        q[k] = 0
        p = 3 * q / s
        u = m[k] * lam - m[:, None] * lam[k].astype(np.longdouble)
        size = m[k] * np.abs(lam) + m[:, None] * np.abs(lam[k])
        g = (q[:, None] * u - (p * (d * u).sum(1))[:, None] * d).sum(0)
        gs = (q[:, None] * size + (p * (np.abs(d) * size).sum(1))[:, None] * np.abs(d)).sum(0)
        w, ws = -(q * (lam * d).sum(1)).sum(), (q * (np.abs(lam) * np.abs(d)).sum(1)).sum()
        assert np.all(np.abs(gp[k] - g) <= tol * gs) and abs(gm[k] - w) <= tol * ws


# the last size of one launch, the first of two, and an odd number of blocks in two
@pytest.mark.parametrize("n", [92672, 92673, 100001])
def test_potential_in_several_launches(lib, cuda, n):
    x, m, _, rows = system(n)
    check_potential(x, m, np.concatenate([rows, [0, 127, 128, n - 129, n - 1]]))


@pytest.mark.parametrize("n", [46336, 46337])
def test_fp64_vjp_in_several_launches(lib, cuda, n):
    x, m, lam, rows = system(n)
    check_vjp(x, m, lam, np.concatenate([rows, [0, 127, 128, n - 129, n - 1]]))


# the column sums' reservation fails once (16 or 17 rows at a time -> 2 or 3), twice (-> 1)
@pytest.mark.parametrize("failed", [1, 2])
@pytest.mark.parametrize("n", [2048, 2049])
def test_fewer_rows_when_memory_is_short(lib, cuda, fail_after, n, failed):
    x, m, lam, rows = system(n)
    fail_after(1, failed)
    check_potential(x, m, rows)
    fail_after(1, failed)
    check_vjp(x, m, lam, rows)


def test_out_of_memory_with_one_row(lib, cuda, fail_after):
    from gravhopper_gb300 import _capi
    x, m, _, rows = system(2048)
    fail_after(0, 3)
    with pytest.raises(_capi.EngineError) as err:
        check_potential(x, m, rows)
    assert err.value.code == _capi.GH_ERR_OOM
    fail_after(0, 0)
    check_potential(x, m, rows)


@pytest.mark.parametrize("n", [2000, 20000])
def test_walk_without_scratch_is_not_split(lib, cuda, fail_after, n):
    """Every reservation before the walk's ends the call; the walk's own two do not, and
    leave it unsplit: other bits, since its sums are grouped otherwise."""
    from gravhopper_gb300 import _capi, _jbgrav
    x, m, _, _ = system(n)
    split = _jbgrav.tree_force(x, m, 0.02, 0.7)
    ref = oracle.tree_force(x, m, 0.02, 0.7)
    survived = []
    for k in range(40):
        fail_after(k, 1)
        try:
            survived.append(_jbgrav.tree_force(x, m, 0.02, 0.7))
        except _capi.EngineError as e:
            assert e.code == _capi.GH_ERR_OOM and not survived
        fail_after(0, 0)
    unsplit = [a for a in survived if not np.array_equal(a, split)]
    assert len(unsplit) == 2
    for a in unsplit + [_jbgrav.tree_force(x, m, 0.02, 0.7)]:
        r = np.linalg.norm(a - ref, axis=1) / np.linalg.norm(ref, axis=1)
        assert np.sqrt(np.mean(r * r)) <= 1e-12 and r.max() <= 1e-9
    np.testing.assert_array_equal(a, split)

"""Arguments that the device-level API settles on the host, without a GPU: empty target
points, buffers that are too short or missing."""
import pytest
import torch

from gravhopper_gb300 import _capi, engine


@pytest.fixture
def calls(monkeypatch):
    """The library calls that the API makes, with CPU tensors taken for device tensors."""
    made = []
    monkeypatch.setattr(engine, "_check", lambda *a: None)
    monkeypatch.setattr(_capi, "call", lambda name, *a: made.append((name, a)))
    monkeypatch.setattr(_capi, "stream_handle", lambda s=None: None)
    return made


def f64(*shape):
    return torch.zeros(shape, dtype=torch.float64)


@pytest.mark.parametrize("fn", [engine.direct_force, engine.tree_force])
def test_no_points_is_no_work(calls, fn):
    """An empty tensor's pointer is null, which would ask for the self-force instead."""
    assert fn(f64(5, 3), f64(5), 0.1, force_pos=f64(0, 3)).shape == (0, 3)
    points, count = calls[-1][1][3:5]
    assert points and count == 0
    assert fn(f64(5, 3), f64(5), 0.1).shape == (5, 3)
    assert not calls[-1][1][3]


def test_short_buffers_are_refused(calls):
    x, m = f64(5, 3), f64(5)
    for bad in (lambda: engine.potential(x, f64(4), 0.1),
                lambda: engine.potential(x, m, 0.1, out=f64(4)),
                lambda: engine.direct_vjp(x, f64(4), 0.1, x),
                lambda: engine.direct_vjp(x, m, 0.1, f64(4, 3)),
                lambda: engine.direct_vjp(x, m, 0.1, x, grad_pos=f64(4, 3)),
                lambda: engine.direct_vjp(x, m, 0.1, x, grad_mass=f64(4)),
                lambda: engine.direct_force(x, m, 0.1, out=f64(4, 3)),
                lambda: engine.tree_force(x, m, 0.1, force_pos=f64(6, 3), out=f64(5, 3))):
        with pytest.raises(ValueError):
            bad()
    with pytest.raises(ValueError):
        _capi.tree_validate(x, f64(4), 0.1)
    assert calls == []


def test_ensemble_refuses_ragged_systems():
    from gravhopper_gb300.ensemble import Ensemble
    good = {"pos": f64(4, 3), "vel": f64(4, 3), "mass": f64(4), "eps": 0.1, "dt": 0.1}
    assert Ensemble([good], device="cpu").nsys == 1
    for k, v in (("pos", f64(3, 3)), ("vel", f64(5, 3)), ("pos", f64(4, 2)), ("mass", f64(4, 2))):
        with pytest.raises(ValueError):
            Ensemble([good, dict(good, **{k: v})], device="cpu")


@pytest.mark.parametrize("entry", ["gh_tree_dev", "gh_direct_dev"])
def test_null_result_is_refused_before_the_device(lib, entry):
    """Addresses are never read: the call ends on the host."""
    x = torch.zeros((5, 3), dtype=torch.float64)
    m = torch.zeros(5, dtype=torch.float64)
    theta = (0.7,) if entry == "gh_tree_dev" else ()
    fn = getattr(lib, entry)
    assert fn(x.data_ptr(), m.data_ptr(), 5, None, 0, 0.1, *theta, 0, None, None) == _capi.GH_ERR_ARG
    assert fn(x.data_ptr(), m.data_ptr(), 5, x.data_ptr(), 0, 0.1, *theta, 0, None, None) == _capi.GH_OK  # no points
    assert fn(x.data_ptr(), m.data_ptr(), 5, x.data_ptr(), 0, -0.1, *theta, 0, None, None) == _capi.GH_ERR_ARG
    assert fn(None, m.data_ptr(), 5, None, 0, 0.1, *theta, 0, x.data_ptr(), None) == _capi.GH_ERR_ARG
    assert fn(x.data_ptr(), None, 5, None, 0, 0.1, *theta, 0, x.data_ptr(), None) == _capi.GH_ERR_ARG

"""The mixed direct sum at target points where its tile shape changes (4096 points or 2048
sources beside a long other side) and where tiles of 128 end, against the FP64 form.
Tolerance of every mixed force: rms <= 1e-6, max <= 1e-3 of the FP64 force."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,points", [(30000, 1), (30000, 128), (30000, 129), (30000, 4096), (30000, 4097), (1, 30000),
                                      (512, 30000), (513, 30000), (2048, 30000), (2049, 30000)])
@pytest.mark.parametrize("equal", [True, False])
def test_points(lib, cuda, n, points, equal):
    import torch

    from gravhopper_gb300 import engine
    rng = np.random.default_rng(n + points)
    x, f = (torch.from_numpy(rng.normal(size=(k, 3))).to(cuda) for k in (n, points))
    m = torch.ones(n, dtype=torch.float64, device=cuda) * 0.7
    if not equal:
        m = m * torch.from_numpy(rng.uniform(0.5, 2.0, n)).to(cuda)
    got = engine.direct_force(x, m, 0.02, force_pos=f, precision="mixed")
    ref = engine.direct_force(x, m, 0.02, force_pos=f)
    r = ((got - ref).norm(dim=1) / ref.norm(dim=1)).cpu().numpy()
    assert np.sqrt(np.mean(r * r)) <= 1e-6 and r.max() <= 1e-3

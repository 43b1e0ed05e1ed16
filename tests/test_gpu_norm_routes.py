"""The norms fused into a step against the separate pass over the same state."""
import pytest
import torch

from cvfes_b200.solver import GPUSolidSolver, LocalComm
from test_gpu_step_shapes import Cfg, wall

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision,state", [(32, "velocity"), (32, "previous"), (64, "previous")])
@pytest.mark.parametrize("kind,samples", [("tube", 1), ("tube", 6), ("tube", 8), ("tube", 33),
                                          ("tube", 64), ("tube", 100), ("tube", 516),
                                          ("irregular", 40), ("irregular", 132)])
def test_separate_norms_of_a_fused_step(lib, cuda, precision, state, kind, samples):
    """The node terms have the same bits on both routes; their FP64 sums, of at most 2,000
    non-negative terms, are taken in another order (2e-13 relative a side)."""
    s = GPUSolidSolver(LocalComm(), wall(kind, samples), Cfg(1e-8, samples, precision, state, 1))
    s.pressure = 1e5
    for _ in range(3):
        s.Solve(None, 1e-8)
    assert s._norms_step == s.step_count
    fused = torch.from_numpy(s.Norms().copy())
    s._norms_step = -1  # the next call runs the separate pass
    separate = torch.from_numpy(s.Norms().copy())
    assert (fused[:, :3] > 0).all() and (fused[:, 3] == 0).all()
    torch.testing.assert_close(separate, fused, rtol=4e-13, atol=0)


@pytest.mark.parametrize("samples", [8, 64])
def test_non_finite_values_are_counted_alike(lib, cuda, samples):
    s = GPUSolidSolver(LocalComm(), wall("tube", samples), Cfg(1e-8, samples, 32, "velocity", 1))
    s.pressure = 1e5
    s.Solve(None, 1e-8)
    s.bufs[s.cur][300, samples // 2] = float("inf")
    s.Solve(None, 1e-8)
    fused = s.Norms(check_finite=False).copy()
    s._norms_step = -1
    separate = s.Norms(check_finite=False).copy()
    assert fused[samples // 2, 3] > 0 and (fused[:, 3] == separate[:, 3]).all()
    assert (fused[:samples // 2, 3] == 0).all()

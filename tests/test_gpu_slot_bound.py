"""Descriptors whose max_degree is below some nodes' number of elements: the kernels whose
shared-memory stages are sized by it form those nodes' rows from global memory, with the bits
of the true descriptor."""
import numpy as np
import pytest
import torch

from cvfes_b200 import _lib
from cvfes_b200.solver import GPUSolidSolver, LocalComm
from test_gpu_step_shapes import Cfg, wall

pytestmark = pytest.mark.gpu


def advance(mesh, precision, state, interval, degree, norms_every=0):
    cfg = Cfg(1e-8, mesh.nSmp, precision, state, norms_every)
    cfg.update_interval = interval
    s = GPUSolidSolver(LocalComm(), mesh, cfg)
    if degree:
        assert degree < s.plan.max_degree
        s._desc.max_degree = degree
    s.Advance(1e4 * (1.0 + np.arange(7)))
    s.plan.check_status()
    out = [s.bufs[s.cur].clone(), s.bufs[s.prev].clone()]
    if norms_every:
        s.pressure = 1e5
        s.Solve(None, 1e-8)
        out.append(torch.from_numpy(s.Norms().copy()))
    s.release_graphs()
    return out


@pytest.mark.parametrize("precision,state,interval", [(32, "velocity", 0), (32, "previous", 0),
                                                      (64, "previous", 0), (32, "previous", 1),
                                                      (64, "previous", 1), (32, "previous", 2),
                                                      (64, "previous", 2)])
@pytest.mark.parametrize("kind,samples,degree", [
    ("tube", 8, 5), ("tube", 3, 2), ("tube", 64, 5), ("tube", 100, 2), ("irregular", 2, 4),
    ("irregular", 16, 7), ("irregular", 40, 6), ("irregular", 128, 1)])
def test_understated_degree_gives_the_same_bits(lib, cuda, precision, state, interval, kind,
                                                samples, degree):
    mesh = wall(kind, samples)
    fused = 1 if interval == 0 else 0
    want = advance(mesh, precision, state, interval, 0, fused)
    got = advance(mesh, precision, state, interval, degree, fused)
    assert torch.isfinite(want[0]).all() and want[0].abs().max() > 0
    assert torch.equal(got[0], want[0]) and torch.equal(got[1], want[1])
    # the norms' node terms have the same bits too, but max_degree decides which kernel adds
    # them and in which order: sums of at most 2,000 non-negative FP64 terms, 2e-13 relative
    for g, w in zip(got[2:], want[2:]):
        torch.testing.assert_close(g, w, rtol=4e-13, atol=0)


@pytest.mark.parametrize("precision,samples", [(32, 24), (32, 64), (64, 33)])
@pytest.mark.parametrize("degree", [1, 5])
def test_understated_degree_in_the_reverse_step(lib, cuda, precision, samples, degree):
    from cvfes_b200.cases import TubeCase, adjoint_setup
    case = TubeCase("bound", 16, 12, 1.5, n_samples=samples, dt=None, n_steps=30,
                    extra=dict(n_obs=24, obs_every=10, ckpt_every=15))
    p, logE, logh, _ = adjoint_setup(case, precision=precision, device=cuda, grad_logh=True)
    outs = []
    for d in (p.plan.max_degree, degree):
        p._desc.mesh.max_degree = p._desc_rec.mesh.max_degree = d
        p.release_graphs()
        J = p.objective(logE, logh).clone()
        outs.append((J, *p.gradient()))
    assert outs[0][1].abs().max() > 0
    for a, b in zip(*outs):
        assert torch.equal(a, b)

"""Long runs of overlapped launches on small walls (a step may be resident while the one before
it writes the rows that it reads): the same bits as steps launched one by one."""
import numpy as np
import pytest
import torch

from cvfes_b200 import _lib
from cvfes_b200.mesh import SolidMesh, TubeGeometry, tube_mesh
from cvfes_b200.solver import GPUSolidSolver, LocalComm

pytestmark = pytest.mark.gpu


class Cfg:
    def __init__(self, dt, nSmp, precision, interval):
        self.dt, self.nSmp, self.update_interval = dt, nSmp, interval
        self.gpu = type("G", (), dict(precision=precision, use_graph=True, graph_chunk=48,
                                      watchdog=True, device=0))()
        self.pressure_ramp = "linear"


def wall(nc, na, S):
    rng = np.random.default_rng(3)
    nodes, elems, i, o = tube_mesh(TubeGeometry(nc, na, 1.0, 0.3))
    bdy = np.concatenate([i, o])
    u0 = 1e-3 * rng.standard_normal((len(nodes), 3))
    u0[bdy] = 0.0
    E = len(elems)
    return SolidMesh(nodes, elems, bdy, S, density=1.0, v=0.49, damp=100.0,
                     elmE=7e6 * np.exp(0.2 * rng.standard_normal((E, S))),
                     elmThick=0.04 * np.exp(0.1 * rng.standard_normal((E, S))),
                     iniU=u0.ravel(), iniDu=rng.standard_normal((len(nodes), 3)).ravel())


@pytest.mark.parametrize("precision", [32, 64])
@pytest.mark.parametrize("nc,na,samples", [(12, 9, 4), (24, 20, 8), (24, 20, 16), (16, 12, 64),
                                           (40, 60, 33), (40, 60, 128)])
@pytest.mark.parametrize("interval,steps", [(0, 600), (1, 300)])
def test_overlapped_steps_give_the_bits_of_single_steps(lib, cuda, precision, nc, na, samples,
                                                        interval, steps):
    mesh = wall(nc, na, samples)
    pres = 1e4 * (1.0 + np.arange(steps) / steps)
    one, many = [GPUSolidSolver(LocalComm(), mesh, Cfg(1e-8, samples, precision, interval))
                 for _ in range(2)]
    many.Advance(pres)
    for p in pres:  # one launch a call, none overlapped
        one.pressure = float(p)
        one.Solve(None, 1e-8)
    a, b = many.local_displacement(), one.local_displacement()
    assert torch.isfinite(a).all() and a.abs().max() > 0 and torch.equal(a, b)
    assert torch.equal(many.bufs[many.prev], one.bufs[one.prev])


@pytest.mark.parametrize("precision", [32, 64])
def test_overlapped_reverse_steps_give_the_row_gather_bits(lib, cuda, precision):
    from cvfes_b200.cases import TubeCase, adjoint_setup
    case = TubeCase("overlap", 16, 14, 1.0, n_samples=40, dt=None, n_steps=400,
                    extra=dict(n_obs=24, obs_every=50, ckpt_every=200))
    p, logE, logh, _ = adjoint_setup(case, precision=precision, device=cuda, grad_logh=True)
    saved, outs = _lib.get_adjoint_tuning(precision), []
    try:
        for variant in (0, 2):
            _lib.set_adjoint_tuning(precision, 1, 4, variant, 2)
            p.release_graphs()
            p.objective(logE, logh)
            outs.append(p.gradient())
    finally:
        _lib.set_adjoint_tuning(precision, **saved)
    assert torch.isfinite(outs[0][0]).all() and outs[0][0].abs().max() > 0
    assert torch.equal(outs[0][0], outs[1][0]) and torch.equal(outs[0][1], outs[1][1])

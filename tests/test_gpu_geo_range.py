"""The geometric step in FP32 on walls whose edges are so small or large that the squared area of
an element leaves FP32's range (the fourth power of an edge): the results of FP64 to the FP32
step's accuracy."""
import numpy as np
import pytest
import torch

from cvfes_b200.mesh import SolidMesh
from cvfes_b200.solver import GPUSolidSolver, LocalComm
from test_gpu_step_shapes import Cfg, wall

pytestmark = pytest.mark.gpu


def scaled(mesh, L):
    """The same wall with lengths in another unit: mass and pressure follow, so the motion is the
    same in that unit."""
    return SolidMesh(mesh.nodes * L, mesh.elementNodeIds, mesh.boundary, mesh.nSmp,
                     density=mesh.density / L ** 2, v=mesh.v, damp=mesh.damp, elmE=mesh.elmE,
                     elmThick=mesh.elmThick, iniU=mesh.iniU * L, iniDu=mesh.iniDu * L)


@pytest.mark.parametrize("interval", [1, 2])
@pytest.mark.parametrize("kind,samples", [("tube", 5), ("tube", 64), ("irregular", 62)])
@pytest.mark.parametrize("L", [2e-10, 1e-9, 1.0, 1e11])
def test_small_and_large_edges(lib, cuda, L, kind, samples, interval):
    mesh = scaled(wall(kind, samples), L)
    out = []
    for precision in (32, 64):
        cfg = Cfg(1e-8, samples, precision, "auto")
        cfg.update_interval = interval
        s = GPUSolidSolver(LocalComm(), mesh, cfg)
        s.Advance(1e4 / L * (1.0 + np.arange(4)))
        out.append(s.local_displacement().double())
    assert torch.isfinite(out[0]).all() and out[1].abs().max() > 0
    assert torch.linalg.norm(out[0] - out[1]) <= 1e-5 * torch.linalg.norm(out[1])

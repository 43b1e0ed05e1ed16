"""The batch's routes: mesh by mesh (small meshes on side streams, the others on the caller's),
and the table's fan and row-gather kernels, each mesh with the bits of the same mesh alone."""
import numpy as np
import pytest
import torch

from cvfes_b200.batched import SMALL_MESH, BatchedSolidSolver
from cvfes_b200.solver import GPUSolidSolver, LocalComm
from test_gpu_overlap import wall
from test_gpu_step_shapes import Cfg

pytestmark = pytest.mark.gpu
SHAPES = [(24, 20, 16), (96, 40, 64), (16, 30, 32), (40, 60, 128), (12, 9, 16)]


@pytest.mark.parametrize("precision", [32, 64])
@pytest.mark.parametrize("variant,grid,grouped,concurrent,by_mesh", [
    (1, 0, True, False, True), (1, 592, True, False, False), (1, 592, False, False, False),
    (0, 0, True, False, False), (1, 0, True, True, False)])
def test_every_route_gives_the_bits_of_the_mesh_alone(lib, cuda, precision, variant, grid, grouped,
                                                      concurrent, by_mesh):
    meshes = [wall(*s) for s in SHAPES]
    sizes = [m.nNodes * m.nSmp for m in meshes]
    assert sum(x >= SMALL_MESH for x in sizes) == 2 and sum(x < SMALL_MESH for x in sizes) == 3
    dts = [1e-8 * (1 + 0.1 * i) for i in range(len(meshes))]
    batch = BatchedSolidSolver(meshes, dts, precision=precision, device=cuda, graph_chunk=12,
                               variant=variant, grid=grid, grouped=grouped, concurrent=concurrent)
    assert batch.by_mesh == by_mesh
    pres = 1e4 * (1.0 + np.arange(70) / 70)
    side = torch.cuda.Stream(device=cuda)
    batch.Advance(pres[:31])  # graph chunks and a remainder
    side.wait_stream(torch.cuda.current_stream(cuda))
    with torch.cuda.stream(side):
        batch.Advance(pres[31:66])  # lead steps first; another stream
    torch.cuda.current_stream(cuda).wait_stream(side)
    batch.Advance(pres[66:], use_graph=False)
    for m, (mesh, dt) in enumerate(zip(meshes, dts)):
        s = GPUSolidSolver(LocalComm(), mesh, Cfg(dt, mesh.nSmp, precision, "auto"))
        s.Advance(pres, dt=dt)
        b = batch.solvers[m]
        assert torch.equal(s.local_displacement(), b.local_displacement()), m
        assert torch.equal(s.bufs[s.prev], b.bufs[b.prev]), m

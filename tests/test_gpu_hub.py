"""A tube closed by a cap whose apex joins a whole ring of elements: nodes of many more
elements than six, up to what the step kernels' stages hold for the block they launch, and
beyond."""
import numpy as np
import pytest
import torch

from cvfes_b200.mesh import SolidMesh, TubeGeometry, tube_mesh
from test_gpu_step_shapes import run

pytestmark = pytest.mark.gpu


def capped(nc, na, S):
    rng = np.random.default_rng(7)
    nodes, elems, i, o = tube_mesh(TubeGeometry(nc, na, 1.0, 0.3))
    ring = nodes[o]
    apex = len(nodes)
    order = np.asarray(o)[np.argsort(np.arctan2(ring[:, 1], ring[:, 0]))]
    cap = np.stack([order, np.roll(order, -1), np.full(nc, apex)], 1)
    nodes = np.vstack([nodes, [0.0, 0.0, 1.1 * nodes[:, 2].max() + 0.05]])
    elems = np.vstack([elems, cap])
    u0 = 1e-3 * rng.standard_normal((len(nodes), 3))
    u0[i] = 0.0
    E = len(elems)
    return SolidMesh(nodes, elems, i, S, density=1.0, v=0.49, damp=100.0,
                     elmE=7e6 * np.exp(0.2 * rng.standard_normal((E, S))),
                     elmThick=0.04 * np.exp(0.1 * rng.standard_normal((E, S))),
                     iniU=u0.ravel(), iniDu=rng.standard_normal((len(nodes), 3)).ravel())


@pytest.mark.parametrize("precision", [32, 64])
@pytest.mark.parametrize("nc,samples", [(16, 64), (17, 64), (29, 33), (29, 128), (30, 40), (31, 64),
                                        (42, 48), (53, 128), (54, 128),
                                        (9, 8), (24, 1), (24, 8), (30, 16), (60, 3), (200, 16)])
def test_a_node_of_many_elements(lib, cuda, precision, nc, samples):
    mesh = capped(nc, 12, samples)
    want = run(mesh, precision, "auto", 0)
    got = run(mesh, precision, "auto", 6)
    assert torch.isfinite(want[0]).all() and want[0].abs().max() > 0
    assert torch.equal(got[0], want[0]) and torch.equal(got[1], want[1])

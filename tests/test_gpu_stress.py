"""Stresses on the undeformed wall at the sizes where the dispatch has edges (one sample vector,
a few, many; blocks of 32 and 128 elements, partly filled; the vectors of one block in parts)."""
import numpy as np
import pytest
import torch

from cvfes_b200.solver import GPUSolidSolver, LocalComm
from test_gpu_step_shapes import Cfg, wall

pytestmark = pytest.mark.gpu


def matrices(nodes, elems, nu):
    """(E, 5, 6) from the local frame of each element: the five global stresses per unit E of
    unit displacements of nodes 1 and 2 relative to node 0.  In extended precision: in FP64 the
    frame of a thin triangle itself loses three digits."""
    P = nodes[elems].astype(np.longdouble)
    ex = P[:, 2] - P[:, 1]
    ex /= np.linalg.norm(ex, axis=1, keepdims=True)
    ey = P[:, 0] - P[:, 2]
    ey -= (ex * ey).sum(1, keepdims=True) * ex
    ey /= np.linalg.norm(ey, axis=1, keepdims=True)
    R = np.stack([ex, ey, np.cross(ex, ey)], 1)
    x, y = (P * ex[:, None]).sum(2), (P * ey[:, None]).sum(2)
    area2 = (x[:, 1] - x[:, 0]) * (y[:, 2] - y[:, 0]) - (x[:, 2] - x[:, 0]) * (y[:, 1] - y[:, 0])
    M = np.zeros((len(elems), 5, 6), dtype=P.dtype)
    nu, k = np.longdouble(nu), np.longdouble(5) / 6
    q = 1 - nu * nu
    for a in (1, 2):
        b = (y[:, (a + 1) % 3] - y[:, (a + 2) % 3]) / area2
        c = (x[:, (a + 2) % 3] - x[:, (a + 1) % 3]) / area2
        for d in range(3):
            lu, lv, lw = R[:, 0, d], R[:, 1, d], R[:, 2, d]
            L = np.zeros((len(elems), 3, 3), dtype=P.dtype)
            L[:, 0, 0] = (b * lu + nu * c * lv) / q
            L[:, 1, 1] = (nu * b * lu + c * lv) / q
            L[:, 0, 1] = L[:, 1, 0] = 0.5 * (1 - nu) / q * (c * lu + b * lv)
            L[:, 0, 2] = L[:, 2, 0] = 0.5 * k * (1 - nu) / q * b * lw
            L[:, 1, 2] = L[:, 2, 1] = 0.5 * k * (1 - nu) / q * c * lw
            G = np.einsum("epi,epq,eqj->eij", R, L, R)
            M[:, :, 3 * (a - 1) + d] = np.stack([G[:, 0, 0], G[:, 1, 1], G[:, 0, 1], G[:, 0, 2],
                                                 G[:, 1, 2]], 1)
    return M


@pytest.mark.parametrize("precision", [32, 64])
@pytest.mark.parametrize("kind", ["tube", "short", "irregular"])
@pytest.mark.parametrize("samples", [1, 2, 3, 4, 5, 6, 8, 12, 16, 20, 37, 64, 130, 256])
def test_stress_against_the_local_frame(lib, cuda, precision, kind, samples):
    """Bound: the FP64 matrix rounded once, a difference, six fused products, E and the product
    with it, 10 roundings of the summed magnitudes (FP64: 40, the matrix itself takes about 30
    on either side)."""
    mesh = wall(kind, samples)
    s = GPUSolidSolver(LocalComm(), mesh, Cfg(1e-8, samples, precision, "auto"))
    got = s.Stress().double().cpu().numpy()
    elems, nodes = s.plan.elems.cpu().numpy(), s.plan.nodes.cpu().numpy()
    M = matrices(nodes, elems, mesh.v)
    u = s.bufs[s.cur].double().cpu().numpy().reshape(-1, 3, samples)[elems]
    d = np.concatenate([u[:, 1] - u[:, 0], u[:, 2] - u[:, 0]], 1)
    E = mesh.element_moduli()
    want = np.einsum("eqk,eks->esq", M, d) * E[:, :, None]
    size = np.einsum("eqk,eks->esq", np.abs(M).max(1, keepdims=True).repeat(5, 1),
                     np.abs(d)) * E[:, :, None]
    eps = 2.0 ** -24 if precision == 32 else 2.0 ** -53
    # a triangle whose height is a fraction of its sides loses that factor in the frame
    thin = np.linalg.cond(np.stack([nodes[elems][:, 1] - nodes[elems][:, 0],
                                    nodes[elems][:, 2] - nodes[elems][:, 0]], 2))
    bound = eps * size * (10.0 if precision == 32 else 40.0 * thin[:, None, None])
    assert np.abs(want).max() > 0 and (np.abs(got - want) <= bound).all()


@pytest.mark.parametrize("precision", [32, 64])
@pytest.mark.parametrize("samples", [3, 4, 5, 16, 37, 130])
def test_stress_of_a_sample_does_not_depend_on_the_ensemble(lib, cuda, precision, samples):
    from cvfes_b200.mesh import SolidMesh
    mesh = wall("tube", samples)
    last = SolidMesh(mesh.nodes, mesh.elementNodeIds, mesh.boundary, 1, density=1.0, v=0.49,
                     damp=100.0, elmE=mesh.elmE[:, -1:], elmThick=mesh.elmThick[:, -1:],
                     iniU=mesh.iniU, iniDu=mesh.iniDu)
    got, want = [GPUSolidSolver(LocalComm(), m, Cfg(1e-8, m.nSmp, precision, "auto")).Stress()
                 for m in (mesh, last)]
    assert torch.equal(got[:, -1:], want)

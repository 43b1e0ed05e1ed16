"""The default step kernels (patch and group, solid_patch.cu and solid_group.cu) at the sizes
where their dispatch, lanes and patches have edges: the same bits as the row-gather kernel
(every step kernel forms the same products and sums in the same order), and the norms of
the new state against FP64 sums of it."""
import numpy as np
import pytest
import torch

from cvfes_b200 import _lib
from cvfes_b200.mesh import SolidMesh, TubeGeometry, tube_mesh
from cvfes_b200.solver import GPUSolidSolver, LocalComm

pytestmark = pytest.mark.gpu


class Cfg:
    def __init__(self, dt, nSmp, precision, state, norms_every=0):
        self.dt, self.nSmp = dt, nSmp
        self.gpu = type("G", (), dict(precision=precision, use_graph=True, graph_chunk=6,
                                      watchdog=True, device=0, state=state,
                                      norms_every=norms_every))()
        self.pressure_ramp = "linear"


def wall(kind, S, seed=5):
    """``tube``: ragged rows of 37 nodes; ``short``: too few rows for 4 x 4 patches;
    ``shuffled``: a random numbering (no rows at all); ``irregular``: a Delaunay sheet, nodes
    of 3 to 9 and more elements, open fans."""
    rng = np.random.default_rng(seed)
    if kind == "irregular":
        from scipy.spatial import Delaunay
        p = rng.random((400, 2))
        tri = Delaunay(p).simplices.astype(np.int64)
        a, b, c = p[tri[:, 0]], p[tri[:, 1]], p[tri[:, 2]]
        area = (b[:, 0] - a[:, 0]) * (c[:, 1] - a[:, 1]) - (b[:, 1] - a[:, 1]) * (c[:, 0] - a[:, 0])
        tri[area < 0] = tri[area < 0][:, [0, 2, 1]]
        tri = tri[np.abs(area) > 1e-5]
        nodes = np.column_stack([p, 0.05 * np.sin(3.0 * p[:, 0])])
        used = np.unique(tri)
        new = np.full(len(nodes), -1)
        new[used] = np.arange(len(used))
        nodes, elems = nodes[used], new[tri]
        bdy = np.where(nodes[:, 0] < 0.1)[0]
    else:
        nc, na = {"tube": (37, 41), "short": (12, 7), "shuffled": (16, 20)}[kind]
        nodes, elems, i, o = tube_mesh(TubeGeometry(nc, na, 1.0, 0.3))
        bdy = np.concatenate([i, o])
        if kind == "shuffled":
            perm = rng.permutation(len(nodes))
            inv = np.argsort(perm)
            nodes, elems, bdy = nodes[perm], inv[elems], inv[bdy]
    E, N = len(elems), len(nodes)
    u0 = 1e-3 * rng.standard_normal((N, 3))
    u0[bdy] = 0.0
    return SolidMesh(nodes, elems, bdy, S, density=1.0, v=0.49, damp=100.0,
                     elmE=7e6 * np.exp(0.2 * rng.standard_normal((E, S))),
                     elmThick=0.04 * np.exp(0.1 * rng.standard_normal((E, S))),
                     iniU=u0.ravel(), iniDu=rng.standard_normal((N, 3)).ravel())


def run(mesh, precision, state, variant, steps=13):
    saved = _lib.get_step_tuning(precision)
    try:
        _lib.set_step_tuning(precision, 4 if precision == 32 else 2, 4, variant, 2)
        s = GPUSolidSolver(LocalComm(), mesh, Cfg(1e-8, mesh.nSmp, precision, state))
        s.Advance(1e4 * (1.0 + np.arange(steps)))
        s.plan.check_status()
        out = s.bufs[s.cur].clone(), s.bufs[s.prev].clone()
        s.release_graphs()
    finally:
        _lib.set_step_tuning(precision, **saved)
    return out


@pytest.mark.parametrize("precision,state", [(32, "velocity"), (32, "previous"), (64, "previous"),
                                             (64, "velocity")])
@pytest.mark.parametrize("kind,samples", [
    ("tube", 1), ("tube", 3), ("tube", 8), ("tube", 16), ("tube", 20), ("tube", 21),
    ("tube", 32), ("tube", 34), ("tube", 64), ("tube", 100), ("tube", 129), ("tube", 132),
    ("tube", 260), ("short", 5), ("short", 64), ("shuffled", 12), ("shuffled", 66),
    ("irregular", 2), ("irregular", 40), ("irregular", 128)])
def test_default_kernels_give_the_row_gather_bits(lib, cuda, precision, state, kind, samples):
    mesh = wall(kind, samples)
    want = run(mesh, precision, state, 0)
    got = run(mesh, precision, state, 6)
    assert torch.isfinite(want[0]).all() and want[0].abs().max() > 0
    assert torch.equal(got[0], want[0]) and torch.equal(got[1], want[1])


@pytest.mark.parametrize("precision", [32, 64])
@pytest.mark.parametrize("kind,samples", [("tube", 1), ("tube", 8), ("tube", 33), ("tube", 100),
                                          ("short", 64), ("irregular", 40), ("irregular", 132)])
def test_step_norms_against_sums_of_the_state(lib, cuda, precision, kind, samples):
    """Node terms carry at most three roundings of the state's type and the FP32 mass term
    a reciprocal and a product more (<= 4e-7 relative, all terms positive); FP64 <= 1e-14."""
    mesh = wall(kind, samples)
    s = GPUSolidSolver(LocalComm(), mesh, Cfg(1e-8, samples, precision, "velocity", 1))
    s.pressure = 1e5
    for _ in range(2):
        s.Solve(None, 1e-8)
    got = s.Norms()
    u, v = s.bufs[s.cur].double(), s.bufs[s.prev].double()
    m = s.plan.lm
    v2 = v.square().reshape(-1, 3, samples).sum(1)
    want = torch.stack([u.square().sum(0), v.square().sum(0), (m * v2).sum(0)], 1).cpu().numpy()
    tol = 6e-7 if precision == 32 else 1e-13
    assert np.all(got[:, 3] == 0) and np.all(want > 0)
    np.testing.assert_allclose(got[:, :3], want, rtol=tol, atol=0)
    np.testing.assert_allclose(got, s.__class__.Norms(s), rtol=0, atol=0)


def run_geo(mesh, precision, interval, vec, steps=5):
    saved = [_lib.C.c_int32(), _lib.C.c_int32()]
    _lib.call("cvfes_get_geo_tuning", precision, _lib.C.byref(saved[0]), _lib.C.byref(saved[1]))
    try:
        _lib.call("cvfes_set_geo_tuning", precision, vec, 128)
        cfg = Cfg(1e-8, mesh.nSmp, precision, "auto")
        cfg.update_interval = interval
        s = GPUSolidSolver(LocalComm(), mesh, cfg)
        s.Advance(1e4 * (1.0 + np.arange(steps)))
        return s.bufs[s.cur].clone()
    finally:
        _lib.call("cvfes_set_geo_tuning", precision, saved[0].value, saved[1].value)


@pytest.mark.parametrize("precision", [32, 64])
@pytest.mark.parametrize("interval", [1, 2])
@pytest.mark.parametrize("kind,samples", [("tube", 30), ("tube", 64), ("tube", 96), ("short", 64),
                                          ("shuffled", 64), ("irregular", 62), ("irregular", 130)])
def test_geometric_step_alone_or_in_an_ensemble(lib, cuda, precision, interval, kind, samples):
    """Samples never interact and every width and kernel rounds alike: the first three
    samples of an ensemble (patch kernel where its lanes are filled) and the same three
    alone (plain kernel, one a thread) have the same bits."""
    mesh = wall(kind, samples)
    few = SolidMesh(mesh.nodes, mesh.elementNodeIds, mesh.boundary, 3, density=1.0, v=0.49,
                    damp=100.0, elmE=mesh.elmE[:, :3], elmThick=mesh.elmThick[:, :3],
                    iniU=mesh.iniU, iniDu=mesh.iniDu)
    got = run_geo(mesh, precision, interval, 2 if precision == 32 else 1)
    want = run_geo(few, precision, interval, 1)
    assert torch.isfinite(got).all() and torch.equal(got[:, :3], want)


@pytest.mark.parametrize("precision", [32, 64])
@pytest.mark.parametrize("kind,samples", [("tube", 2), ("tube", 6), ("tube", 64), ("tube", 129),
                                          ("irregular", 36)])
def test_stress_alone_or_in_an_ensemble(lib, cuda, precision, kind, samples):
    """The stresses of an ensemble's first sample are those of that sample alone (one sample a
    thread, the ensemble up to four), bit for bit."""
    mesh = wall(kind, samples)
    one = SolidMesh(mesh.nodes, mesh.elementNodeIds, mesh.boundary, 1, density=1.0, v=0.49,
                    damp=100.0, elmE=mesh.elmE[:, :1], elmThick=mesh.elmThick[:, :1],
                    iniU=mesh.iniU, iniDu=mesh.iniDu)
    got, want = [GPUSolidSolver(LocalComm(), m, Cfg(1e-8, m.nSmp, precision, "auto")).Stress()
                 for m in (mesh, one)]
    assert torch.isfinite(got).all() and want.abs().max() > 0
    assert torch.equal(got[:, :1], want)

"""FP64 rows as given (slot_form 0): a caller's slot rows need not annihilate translations --
here every self block carries an elastic support -- and all FP64 kernels apply them whole."""
import numpy as np
import pytest
import torch

from cvfes_b200 import _lib
from cvfes_b200._lib import call, ptr
from cvfes_b200.batched import BatchedSolidSolver
from cvfes_b200.solver import GPUSolidSolver, LocalComm
from test_gpu_step_shapes import Cfg, wall

pytestmark = pytest.mark.gpu
DT = 1e-8


def solver(mesh, state="previous", norms_every=0):
    return GPUSolidSolver(LocalComm(), mesh, Cfg(DT, mesh.nSmp, 64, state, norms_every))


def support(plan, share=0.3):
    """Add share of each self block's size to its diagonal (in place)."""
    K = plan.slot_k64.view(-1, 28)
    size = K[:, :9].abs().amax(1, keepdim=True)
    K[:, [0, 4, 8]] += share * size


def rows_times(plan, u):
    """sum over slots of c (K0 u_a + K1 u_b1 + K2 u_b2) with plain torch, FP64."""
    K = plan.slot_k64.view(-1, 28)[:, :27].reshape(-1, 3, 3, 3)
    ptr_, rec = plan.node_ptr.long(), plan.slot_rec.long()
    a = torch.repeat_interleave(torch.arange(plan.N, device=u.device), ptr_[1:] - ptr_[:-1])
    x = u.reshape(plan.N, 3, -1)
    r = sum(torch.einsum("kij,kjs->kis", K[:, q], x[n])
            for q, n in enumerate((a, rec[:, 1], rec[:, 2])))
    out = torch.zeros_like(x).index_add_(0, a, r * plan.coef64[rec[:, 0]][:, None])
    scale = torch.zeros_like(x).index_add_(0, a, (r * plan.coef64[rec[:, 0]][:, None]).abs())
    return out.reshape(u.shape), scale.reshape(u.shape)


@pytest.mark.parametrize("kind,samples", [("tube", 3), ("tube", 8), ("tube", 64), ("irregular", 5),
                                          ("irregular", 40)])
def test_product_of_given_rows(lib, cuda, kind, samples):
    s = solver(wall(kind, samples))
    support(s.plan)
    desc = s.plan.desc(64)
    desc.slot_form = 0
    u = s.bufs[s.cur]
    got = torch.empty_like(u)
    call("cvfes_solid_kmul_f64", _lib.C.byref(desc), ptr(s.plan.coef64), ptr(u), ptr(got), 0,
         s._stream())
    want, scale = rows_times(s.plan, u)
    # at most 18 elements of 9 terms a row: 200 roundings of the summed magnitudes
    assert scale.max() > 0 and ((got - want).abs() <= 2.3e-14 * 3 * scale.max()).all()
    desc.slot_form = 1  # the difference form does not see the support
    call("cvfes_solid_kmul_f64", _lib.C.byref(desc), ptr(s.plan.coef64), ptr(u), ptr(got), 0,
         s._stream())
    assert (got - want).abs().max() > 1e-3 * scale.max()


@pytest.mark.parametrize("state", ["previous", "velocity"])
@pytest.mark.parametrize("kind,samples", [("tube", 1), ("tube", 8), ("tube", 16), ("tube", 33),
                                          ("tube", 64), ("irregular", 4), ("irregular", 40),
                                          ("irregular", 66)])
@pytest.mark.parametrize("degree", [None, 5])
def test_steps_of_given_rows(lib, cuda, state, kind, samples, degree):
    """Default kernels and the staged, fan and tiled variants against the row gather, bit for
    bit, and one step of it against plain torch."""
    mesh = wall(kind, samples)
    outs, saved = [], _lib.get_step_tuning(64)
    try:
        for variant in (0, 6, 3, 1, 7):
            _lib.set_step_tuning(64, 2, 4, variant, 2)
            s = solver(mesh, state, norms_every=1 if variant == 6 else 0)
            support(s.plan)
            s._desc.slot_form = 0
            if degree and variant:
                s._desc.max_degree = degree
            u, v = [s.bufs[i].clone() for i in (s.cur, s.prev)]
            s.pressure = 1e5
            s.Solve(None, DT)
            first = s.local_displacement().clone()
            for _ in range(4):
                s.Solve(None, DT)
            outs.append((first, s.local_displacement().clone(), s.bufs[s.prev].clone()))
            s.Norms()
            s.plan.check_status()
    finally:
        _lib.set_step_tuning(64, **saved)
    for o in outs[1:]:
        for x, y in zip(o, outs[0]):
            assert torch.equal(x, y)
    p, S = s.plan, samples
    ku, _ = rows_times(p, u)
    g = 0.5 * DT * mesh.damp
    im = p.invm64.reshape(p.N, 1, S)
    inc = (v if state == "velocity" else u - v).reshape(p.N, 3, S)
    f = 1e5 * p.fhat64[:, :3, None] - ku.reshape(p.N, 3, S)
    step = inc * (1 - DT * mesh.damp / (1 + g)) + DT * DT / (1 + g) * im * f
    want = (u.reshape(p.N, 3, S) + step)
    want[: p.n_clamped] = p.clamp_value
    torch.testing.assert_close(outs[0][0].reshape(p.N, 3, S), want, rtol=1e-12,
                               atol=1e-13 * float(want.abs().max()))


@pytest.mark.parametrize("variant", [0, 1])
def test_batch_of_given_rows(lib, cuda, variant):
    meshes = [wall("tube", 16), wall("irregular", 64)]
    b = BatchedSolidSolver(meshes, [DT, DT], precision=64, device=cuda, variant=variant, grid=64)
    alone = [solver(m) for m in meshes]
    for s in b.solvers + alone:
        support(s.plan)
        s._desc.slot_form = 0
    b._pack()
    pres = 1e4 * (1.0 + np.arange(7))
    b.Advance(pres)
    for s, t in zip(b.solvers, alone):
        t.Advance(pres)
        assert torch.equal(s.local_displacement(), t.local_displacement())


@pytest.mark.parametrize("samples", [8, 33, 64])
@pytest.mark.parametrize("degree", [None, 4])
def test_reverse_step_of_given_rows(lib, cuda, samples, degree):
    """The patch kernel (and the fan variant, which takes it) against the row gather, bit for
    bit; the library's own rows give the difference form's results to rounding."""
    from cvfes_b200.cases import TubeCase, adjoint_setup
    case = TubeCase("given", 10, 8, 1.5, n_samples=samples, dt=None, n_steps=30,
                    extra=dict(n_obs=12, obs_every=10, ckpt_every=15))
    p, logE, logh, _ = adjoint_setup(case, precision=64, device=cuda, grad_logh=True)
    want = p.objective(logE, logh).clone(), *[g.clone() for g in p.gradient()]
    for d in (p._desc, p._desc_rec):
        d.mesh.slot_form = 0
    outs, saved = [], _lib.get_adjoint_tuning(64)
    try:
        for variant in (0, 2, 1):
            _lib.set_adjoint_tuning(64, 1, 4, variant, 2)
            if degree and variant:
                p._desc.mesh.max_degree = p._desc_rec.mesh.max_degree = degree
            p.release_graphs()
            outs.append((p.objective(logE, logh).clone(), *p.gradient()))
    finally:
        _lib.set_adjoint_tuning(64, **saved)
    for o in outs[1:]:
        for x, y in zip(o, outs[0]):
            assert torch.equal(x, y)
    for x, y in zip(outs[0], want):
        torch.testing.assert_close(x, y, rtol=0, atol=1e-9 * float(y.abs().max()))

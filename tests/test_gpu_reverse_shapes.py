"""The reverse step's patch kernel at the sizes where its lanes, chunks and fans have edges: the
bits of the row gather (every reverse kernel forms the same products and sums in the same
order)."""
import numpy as np
import pytest
import torch

from cvfes_b200 import _lib
from cvfes_b200.adjoint import MismatchProblem
from test_gpu_step_shapes import wall

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [32, 64])
@pytest.mark.parametrize("logh", [False, True])
@pytest.mark.parametrize("kind,samples", [
    ("tube", 19), ("tube", 20), ("tube", 24), ("tube", 31), ("tube", 33), ("tube", 37),
    ("tube", 64), ("tube", 100), ("tube", 129), ("tube", 130), ("short", 20), ("short", 66),
    ("shuffled", 40), ("irregular", 20), ("irregular", 37), ("irregular", 100)])
def test_patch_reverse_gives_the_row_gather_bits(lib, cuda, precision, logh, kind, samples):
    mesh = wall(kind, samples)
    free = np.setdiff1d(np.arange(mesh.nNodes), mesh.boundary)
    p = MismatchProblem(mesh, 1e-8, 1e5 * np.ones(24), free[::7], obs_every=6, ckpt_every=9,
                        precision=precision, device=cuda, grad_logh=logh)
    g = torch.Generator(device=cuda).manual_seed(1)
    p.set_observations(1e-4 * torch.randn(4, len(free[::7]), 3, samples, generator=g,
                                          device=cuda, dtype=torch.float64))
    logE = torch.from_numpy(np.log(mesh.elmE)).to(cuda)
    logh_ = torch.from_numpy(np.log(mesh.elmThick)).to(cuda)
    saved, outs = _lib.get_adjoint_tuning(precision), []
    try:
        for vec, variant in ((1, 0), (saved["vec"], 2)):
            _lib.set_adjoint_tuning(precision, vec, 4, variant, 2)
            p.release_graphs()
            J = p.objective(logE, logh_).clone()
            outs.append((J, *[x for x in p.gradient() if x is not None]))
    finally:
        _lib.set_adjoint_tuning(precision, **saved)
    assert outs[0][1].abs().max() > 0
    for a, b in zip(*outs):
        assert torch.isfinite(a).all() and torch.equal(a, b)

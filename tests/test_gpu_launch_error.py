"""A launch that the runtime refuses on the host is reported by the call that made it and leaves
nothing behind for the next launch check, the library's or the caller's."""
import pytest
import torch

from cvfes_b200 import _lib
from cvfes_b200._lib import call, ptr

pytestmark = pytest.mark.gpu


def test_a_refused_launch_is_reported_once(lib, cuda):
    S = 1 << 26  # one node: more sample vectors than a grid has rows of blocks for
    u = torch.zeros(3, S, device=cuda)
    im = torch.ones(1, S, device=cuda)
    work = torch.empty(int(lib.cvfes_norms_work_size(1, S)), dtype=torch.float64, device=cuda)
    out = torch.empty(S, 4, dtype=torch.float64, device=cuda)
    st = torch.cuda.current_stream().cuda_stream
    with pytest.raises(_lib.CvfesError):
        call("cvfes_solid_norms_f32", 1, S, ptr(u), ptr(u), ptr(im), ptr(work), ptr(out), 0, st)
    assert "k_norms_partial" in _lib.last_error()
    x = torch.arange(5, device=cuda) + 1  # torch checks the last error after its launches
    call("cvfes_solid_norms_f32", 1, 64, ptr(u), ptr(u), ptr(im), ptr(work), ptr(out), 1, st)
    assert int(x.sum()) == 15 and float(out[:64].abs().sum()) == 0.0

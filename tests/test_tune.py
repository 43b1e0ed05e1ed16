"""The autotuner's cache keys and candidate lists (no GPU)."""
import hashlib
import json

import torch

from cvfes_b200 import tune


def test_a_choice_measured_with_other_kernels_is_not_found(tmp_path, monkeypatch):
    monkeypatch.setenv("CVFES_CACHE", str(tmp_path))
    monkeypatch.setattr(torch.cuda, "get_device_name", lambda d=None: "gpu")
    shape = ("step", 32, 100, 180, 8, 6, "velocity")
    before = "step|gpu|" + hashlib.sha1(repr(shape).encode()).hexdigest()[:16]
    (tmp_path / "tuning.json").write_text(json.dumps({before: dict(staged=3)}))
    key = tune._key("step", "cuda:0", shape)
    assert key not in tune._load_cache()
    tune._store(key, dict(staged=6))
    assert tune._load_cache()[tune._key("step", "cuda:0", shape)]["staged"] == 6
    monkeypatch.setattr(tune, "KERNELS", tune.KERNELS + 1)
    assert tune._key("step", "cuda:0", shape) not in tune._load_cache()


def test_the_mesh_by_mesh_route_is_timed_once():
    grids = {0: [0, 4], 1: [0, 4]}
    got = tune.batch_candidates([1, 0], [4, 2, 1], grids, True)
    assert len(set(got)) == len(got) == 10
    assert [c for c in got if c[0] == 1 and c[2] == 0] == [(1, 4, 0)]
    assert {(1, x, 4) for x in (4, 2, 1)} <= set(got)
    assert len(tune.batch_candidates([1, 0], [4, 2, 1], grids, False)) == 12

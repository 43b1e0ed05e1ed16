"""Kernels that may start while the step before them still runs (programmatic dependent
launch) read state rows with plain loads: the read-only path (__ldg, const __restrict__) is
defined only for data that nothing writes while the kernel is resident."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(__file__)), "cvfes_b200", "csrc")
STATIC = re.compile(r"\b(coef|cf|invm|node_ptr|rec|geo|fhat|trac|nodes|elems)\b")


def source(name):
    text = open(os.path.join(CSRC, name)).read()
    return re.sub(r"//[^\n]*", "", text)


def closing(text, start, pair):
    depth = 0
    for i in range(start, len(text)):
        depth += (text[i] == pair[0]) - (text[i] == pair[1])
        if depth == 0:
            return i
    raise AssertionError("unbalanced " + pair)


def function(text, name):
    """Head and body of the (template) function of this name."""
    at = re.search(r"\b%s\s*\(" % name, text).start()
    return text[at:closing(text, text.index("{", at), "{}") + 1]


def read_only_loads(text):
    for m in re.finditer(r"\b(__ldg|ldg\s*<[^>]*>)\s*\(", text):
        yield text[m.end():closing(text, m.end() - 1, "()")]


def bodies():
    for name in ("solid_patch.cu", "solid_group.cu", "solid_geo.cu"):
        yield name, source(name)
    adjoint, core = source("solid_adjoint.cu"), source("step_core.cuh")
    for f in ("k_reverse_patch", "rev_rows", "rev_update", "owner_form", "slot_fma2"):
        yield f, function(adjoint, f)
    for f in ("clamp_store", "slot_fma", "to_diff", "step_pressure"):
        yield f, function(core, f)


def test_streaming_loads_of_state_rows_keep_their_place():
    """ldcs may be moved over the wait; it is for the inverse mass alone."""
    for name, text in bodies():
        for m in re.finditer(r"\bldcs\s*<[^>]*>\s*\(", text):
            assert "invm" in text[m.end():closing(text, m.end() - 1, "()")], name


@pytest.mark.parametrize("name,text", list(bodies()), ids=lambda v: v if len(v) < 40 else "")
def test_only_static_data_goes_through_the_read_only_path(name, text):
    for arg in read_only_loads(text):
        assert STATIC.search(arg), (name, arg)


@pytest.mark.parametrize("kernel", ["k_norms_partial", "k_norms_final"])
def test_norm_kernels_do_not_declare_their_input_read_only(kernel):
    text = function(source("solid_step.cu"), kernel)
    assert "__restrict__" not in text and not list(read_only_loads(text))


@pytest.mark.parametrize("kernel,name", [("k_step_patch", "solid_patch.cu"),
                                         ("k_step_geo_patch", "solid_geo.cu"),
                                         ("k_reverse_patch", "solid_adjoint.cu")])
def test_state_rows_follow_the_wait(kernel, name):
    text = function(source(name), kernel)
    first = re.search(r"\bld(_state)?\s*<", text)
    assert first and text.index("grid_dependency_wait()") < first.start()

"""Launches that overlap the one before them (programmatic dependent launch) read what that launch writes with
coherent loads: the read-only path (__ldg) is defined only for memory that stays as it is while the kernel runs,
and a block may be resident while the launch before is still storing."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "geopvi_gb300", "csrc")

# What each file may read through __ldg: tables and inputs that are constant through a call, and the level before
# the previous one (p0, lam2), whose writer had finished when the previous launch began.
READ_ONLY = {
    "fwi2d_exact_adjoint.cuh": {"ab", "vdt", "b.cells", "tz", "tx", "lam2"},
    "fwi2d_step.cuh": {"c", "c.c->bl", "cz->bl", "cz", "p", "p0", "vdt", "w.vdt", "pc.rik"},
    "fwi3d_engine.cu": {"p0", "b.w", "b.omw", "src"},
}


def operands(text):
    """The base name of every __ldg operand."""
    return [re.match(r"\s*(?:reinterpret_cast<[^>]*>\()?[&(*]*([A-Za-z_][\w.]*(?:->\w+)?)", a).group(1)
            for a in re.split(r"__ldg\(", text)[1:]]


@pytest.mark.parametrize("name", sorted(READ_ONLY))
def test_read_only_loads_are_of_finished_memory(name):
    text = re.sub(r"//[^\n]*", "", open(os.path.join(CSRC, name)).read())
    assert set(operands(text)) <= READ_ONLY[name]


def test_a_stage_is_released_after_the_whole_warp_has_read_it():
    """Lane 0's arrival lets the copy engine overwrite the stage; a vote orders no memory, a warp barrier does."""
    lines = [ln.split("//")[0].strip() for ln in open(os.path.join(CSRC, "fwi3d_engine.cu"))]
    at = [i for i, ln in enumerate(lines) if re.search(r"mbar_arrive\(empty", ln)]
    assert at and all(lines[i - 1] == "__syncwarp();" for i in at)

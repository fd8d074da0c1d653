"""Kernels of the backward that may start before the one ahead of them has ended: a grid launched that way sees another grid's writes only
behind `griddepcontrol.wait`.  In every role of such a kernel that reads what the preprocess kernel wrote (dA, the row
statistics), the wait has to come first.  Read off the source: a missing wait gives right results nearly always."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "triton_diff_attn_b200", "csrc")


def _kernel(name, function):
    text = re.sub(r"//[^\n]*", "", open(os.path.join(CSRC, name)).read())
    text = text[text.index(function + "("):]
    end = text.find("__global__")
    return text[:end] if end > 0 else text


# kernel, reads of the preprocess kernel's results (QSIDE: which instantiation reads it there)
@pytest.mark.parametrize("name,function,reads", [
    ("bwd.cuh", "diffattn_bwd_dkdv64_kernel", r"&tm_da|args\.stats"),
    ("bwd.cuh", "diffattn_bwd_dq64_kernel", r"load_da\(|stat_row\("),
    ("bwd128.cuh", "diffattn_bwd_dv128_kernel", r"&tm_da|args\.stats|stat_row\("),
    ("bwd128.cuh", "diffattn_bwd_side128_kernel<QSIDE>", r"&tm_y,|args\.stats|stat_row\("),
    ("bwd128.cuh", "diffattn_bwd_side128_kernel<!QSIDE>", r"&tm_w,|args\.stats"),
])
def test_waits_before_it_reads(name, function, reads):
    function, _, form = function.partition("<")
    text = _kernel(name, function)
    if form:
        other = r"\(!QSIDE\)" if form == "QSIDE>" else r"\(QSIDE\)"
        text = re.sub(r"if %s griddep_wait\(\);" % other, "", text)
    text = text.replace("auto load_da = ", "")
    setup, *roles = re.split(r"\} else if \(warp ==|\} else \{\n    const int g|\n  if \(warp == WARP_TMA\) \{", text)
    setup = setup[setup.index("if (warp == WARP_TMA && lane == 0)"):]
    assert not re.search(reads, setup)
    readers = 0
    for role in roles:
        first = re.search(reads, role)
        if first:
            readers += 1
            assert "griddep_wait();" in role[:first.start()], role[:200]
    assert readers

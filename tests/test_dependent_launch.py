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


def _roles(name, function):
    """(text before the roles, texts of the roles); "<QSIDE>" and "<!QSIDE>" leave only that form's code in."""
    function, _, form = function.partition("<")
    text = _kernel(name, function)
    if form:
        text = re.sub(r"if \(%s\) griddep_wait\(\);" % ("!QSIDE" if form == "QSIDE>" else "QSIDE"), "", text)
        if form == "!QSIDE>":
            text = re.sub(r"\n    if \(QSIDE\) \{.*?\n    \}", "", text, flags=re.S)
    text = text.replace("auto load_da = ", "")
    setup, *roles = re.split(r"\} else if \(warp ==|\} else \{\n    const int g|\n  if \(warp == WARP_TMA\) \{", text)
    return setup[setup.index("if (warp == WARP_TMA && lane == 0)"):], roles


KERNELS = [   # kernel (and form), reads of the preprocess kernel's results, barriers that complete without the grid ahead
    ("bwd.cuh", "diffattn_bwd_dkdv64_kernel", r"&tm_da|args\.stats", "kv_empty|"),       # (kv_empty: for the second tile on)
    ("bwd.cuh", "diffattn_bwd_dq64_kernel", r"load_da\(|stat_row\(", "q_empty|"),         # (q_empty likewise)
    ("bwd128.cuh", "diffattn_bwd_dv128_kernel", r"&tm_da|args\.stats|stat_row\(", "bar_kv|k_ready|"),
    ("bwd128.cuh", "diffattn_bwd_side128_kernel<QSIDE>", r"&tm_y,|args\.stats|stat_row\(", ""),
    ("bwd128.cuh", "diffattn_bwd_side128_kernel<!QSIDE>", r"&tm_w,|args\.stats", "bar_xy|y_ready|"),
]


@pytest.mark.parametrize("name,function,reads,own", KERNELS)
def test_waits_before_it_reads(name, function, reads, own):
    setup, roles = _roles(name, function)
    assert not re.search(reads, setup)
    readers = 0
    for role in roles:
        first = re.search(reads, role)
        if first:
            readers += 1
            assert "griddep_wait();" in role[:first.start()], role[:200]
    assert readers


@pytest.mark.parametrize("name,function,reads,own", KERNELS)
def test_bounded_waits_do_not_count_the_grid_ahead(name, function, reads, own):
    """griddepcontrol.wait has no time limit, the other waits have one: whatever can only come once the grid ahead has completed is waited
    for behind it, in every role, or a long kernel ahead would look like a lost load."""
    setup, roles = _roles(name, function)
    assert "mbar_wait" not in setup
    waits = 0
    for role in roles:
        first = re.search(r"mbar_wait\w*\(&misc->(?!%s\d)\w+" % own, role)
        if first:
            waits += 1
            assert "griddep_wait();" in role[:first.start()], first.group(0)
    assert waits >= 3

"""What the kernels' error paths must hold, read from their sources (a wait that gives up cannot be
provoked on a healthy device)."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "pyscfad_b200", "csrc")


def _source(name):
    with open(os.path.join(CSRC, name)) as f:
        return re.sub(r"//[^\n]*", "", f.read())


def _body(src, start):
    """The braces' content from the first { behind `start`."""
    at = src.index("{", src.index(start))
    depth, end = 0, at
    while True:
        depth += {"{": 1, "}": -1}.get(src[end], 0)
        end += 1
        if depth == 0:
            return src[at:end]


# A block that retires with a bulk copy in flight leaves it writing into the next block's shared memory
@pytest.mark.parametrize("name,kernel", [("tc_f1.cuh", "k_f1_tc("), ("tc_b1.cuh", "k_b1_tc("), ("f2m.cuh", "k_f2m(")])
def test_copies_in_flight_are_waited_for_after_a_timeout(name, kernel):
    src = _source(name)
    body = _body(src, kernel)
    assert ("pend_phase[s]" in body and "kSpinLimit" in body) or "f2m_drain(" in body.rsplit("break;", 1)[1]


def test_mixed_epilogue_loads_nothing_more_after_a_timeout():
    src = _source("f2m.cuh")
    # a stage is refilled by its eighth reader; a wait that gives up puts every count out of reach
    body = _body(src, "k_f2m(")
    assert "if (seen == 7u)" in body
    slow = _body(src, "void f2m_wait_slow(")
    assert slow.index("*abortp = 1") < slow.index("atomicAdd((int *)abortp - s, 1 << 16)")
    tables = [line for line in body.split("\n") if "issue_tables(" in line and "auto issue_tables" not in line]
    assert len(tables) == 2                                     # the first item's and the next one's
    assert "s_read[kF2mStages] == 0u" in tables[1]             # the abort flag


def test_error_bits_name_one_place():
    seen = {}
    for name in sorted(os.listdir(CSRC)):
        for bit in re.findall(r"atomicOr\([^;]*?err, (\d+)\)", _source(name)):
            seen.setdefault(int(bit), []).append(name)
    assert sorted(seen) == [1, 2, 4, 8, 16, 32, 64, 128]
    assert all(len(places) == 1 for places in seen.values()), seen

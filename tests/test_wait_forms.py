"""CPU: the form of the waits inside the GEMM kernels, read from their sources.

Every role of these kernels is a whole warp: it waits on an mbarrier and then elects the issuing lane, loads from tensor
memory or meets (`elect.sync`, `tcgen05.ld.sync.aligned`, `bar.warp.sync`: all name the full warp).  A wait that runs out in
some lanes only must therefore not let those lanes leave alone - the others would wait for them without a limit.  The voted
forms (`mbar_wait_warp`, `mbar_wait_both`) give one answer to the warp; `mbar_wait` answers per lane.  Running out of a limit
inside a kernel cannot be provoked on a GPU from the host, so the rule is held here."""
import os
import re

import pytest

import util

CSRC = os.path.join(util.ROOT, "justgoal_b200", "csrc")


def _code(name):
    src = open(os.path.join(CSRC, name)).read()
    return re.sub(r"//[^\n]*", "", src)


@pytest.mark.parametrize("name", ["gemm.cuh", "gemm_pair.cuh"])
def test_warp_wide_roles_wait_with_a_vote(name):
    code = _code(name)
    assert re.search(r"\bmbar_wait_warp\s*\(", code)
    assert not re.search(r"\bmbar_wait\s*\(", code) and not re.search(r"\bmbar_try_wait\s*\(", code)


def test_voted_forms_vote():
    code = _code("common.cuh")
    for fn in ("mbar_wait_warp", "mbar_wait_both"):
        body = code[code.index("bool " + fn):]
        body = body[:body.index("\n}")]
        assert body.rstrip().endswith("return merged(ok);")
        slow = body[body.rindex("if (!ok)"):]
        assert "__all_sync(0xFFFFFFFFu" in slow

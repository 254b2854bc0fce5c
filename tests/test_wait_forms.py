"""CPU: the form of the waits and hand-outs inside the GEMM kernels, read from their sources.

Every role of these kernels is a whole warp: it waits on an mbarrier and then elects the issuing lane, loads from tensor
memory or meets (`elect.sync`, `tcgen05.ld.sync.aligned`, `bar.warp.sync`: all name the full warp).  A wait that runs out in
some lanes only must therefore not let those lanes leave alone - the others would wait for them without a limit.  The voted
forms (`mbar_wait_warp`, `mbar_wait_both`) give one answer to the warp; `mbar_wait` answers per lane.  Running out of a limit
inside a kernel, or a warp's lanes apart in time, cannot be provoked from the host, so the rules are held here."""
import os
import re

import pytest

import util

CSRC = os.path.join(util.ROOT, "justgoal_b200", "csrc")


def _code(name):
    src = open(os.path.join(CSRC, name)).read()
    return re.sub(r"//[^\n]*", "", src)


VOTED = {"mbar_wait_warp", "mbar_wait_both"}


def _waits(code):
    """Every call that looks at an mbarrier, whatever it is named."""
    return set(re.findall(r"\b(mbar_\w*(?:wait|test)\w*)\s*\(", code))


def _promotion_loop(code):
    """The tokens-on-M branch of the promotion warps: (before the block loop, the loop, behind it up to the other branch)."""
    branch = code[code.index("auto qload ="):]
    branch = branch[:branch.index("} else\n")]
    head, rest = branch.split("for (int n = ge - gb; n > 0; --n) {")
    end = rest.index("\n                }\n")
    return head, rest[:end], rest[end:]


@pytest.mark.parametrize("name", ["gemm.cuh", "gemm_pair.cuh"])
def test_warp_wide_roles_wait_with_a_vote(name):
    code = _code(name)
    assert "mbar_wait_warp" in _waits(code)
    if name == "gemm.cuh":
        for part in _promotion_loop(code):
            assert code.count(part) == 1
            code = code.replace(part, "")
    assert _waits(code) <= VOTED
    assert "try_wait" not in code and "test_wait" not in code          # no barrier is polled by hand either


def test_lanes_that_waited_alone_meet_before_they_load():
    head, loop, behind = _promotion_loop(_code("gemm.cuh"))
    for part in (head, loop, behind):
        assert _waits(part) <= {"mbar_wait_flag", "mbar_test"}
    assert not re.search(r"\b(break|continue|return)\b", loop) and "qload(0)" not in head.split("};")[-1]
    before_load = loop[:loop.index("qload(")]
    assert before_load.rindex("mbar_wait_flag(") < before_load.rindex("__syncwarp();") < before_load.rindex("tc_fence_after();")
    assert _waits(loop[loop.index("qload("):]) == {"mbar_test"}        # a look; what it says is acted on in front of the meeting
    assert "mbar_test" not in _waits(before_load)
    hand_backs = re.findall(r"if \(([^)]*)\) mbar_arrive\(bar_tempty", loop)
    assert hand_backs == ["lane == 0 && landed"]
    vote = behind.index("__all_sync(0xFFFFFFFFu, landed != 0)")
    assert "ok = false; break;" in behind[vote:]


def test_voted_forms_vote():
    code = _code("common.cuh")
    for fn in ("mbar_wait_warp", "mbar_wait_both"):
        body = code[code.index("bool " + fn):]
        body = body[:body.index("\n}")]
        assert body.rstrip().endswith("return merged(ok);")
        slow = body[body.rindex("if (!ok)"):]
        assert "__all_sync(0xFFFFFFFFu" in slow


def test_what_one_lane_learns_about_other_ctas_orders_the_whole_warp():
    """One lane acquires (or counts in with an atomic) and hands the answer out by a shuffle or a vote, which order no memory;
    all lanes then load what other CTAs stored.  A `__syncwarp` has to stand between: static pieces, claimed chunks, fused
    combine."""
    code = _code("gemm.cuh")
    for answer in ("here = __shfl_sync(0xFFFFFFFFu, here, 0);", "seen_pieces = __shfl_sync(0xFFFFFFFFu, seen_pieces, 0);",
                   "unsigned todo = __ballot_sync(0xFFFFFFFFu, last);"):
        assert code.count(answer) == 1
        after = code[code.index(answer) + len(answer):].lstrip()
        assert after.startswith("__syncwarp();"), answer


def test_routed_front_end_keeps_nothing_in_the_handle():
    """Calls of b200moe_forward_routed on two streams share a handle and nothing else: what GEMM1 watches of their front end lies in the
    workspace.  The handle's count belongs to the routing front end's meeting; every CTA clears its own word before GEMM1 can look."""
    front, host = _code("front.cuh"), _code("b200moe.cu")
    body = front[front.index("void front_body("):front.index("front_route_kernel(")]
    assert "fp.sync" not in body
    small = front[front.index("front_small_kernel("):front.index("template <int VPT")]
    clear = small.index("(fp.copied)[blockIdx.x] = 0;")
    assert "pdl_launch" not in small[:clear]
    zero, nobody_looks, rest = small[clear:].split("pdl_launch();")[:3]
    assert "__threadfence();" in zero and nobody_looks.endswith("else if (!fp.copied) {\n        ")
    assert rest.index("threadIdx.x >= clears - 31") < rest.index("fence.acq_rel.gpu;") < rest.index("__syncwarp();")
    assert "g1.copied = ntok < 128 ? front_copied(" in host and "d_sync" not in host[host.index("int* front_copied("):host.index("int front_grid(")]
    assert re.findall(r"met = (\w+) \? h->d_sync", host) == ["route_in_front"] * 2


def test_meeting_count_is_cleared_whatever_happened():
    """The count of the front end's meeting is cleared by the last kernel of a forward, also after a wait that ran out (the next call
    would not wait for its routing otherwise), and only when nobody watches it any more.  Where one launch does both GEMMs and the
    combine, that is behind the last CTA of the launch, whose warps have all come back; never at a claim, which a CTA that gave up does
    not take and which, in a call without rows, need not wait for the front end."""
    code = _code("gemm.cuh")
    roles = code[code.index("void gemm_roles("):code.index("gemm_kernel(const __grid_constant__")]
    assert re.findall(r"\*p\.met = |p\.met\[", roles) == ["*p.met = "]
    line = next(s for s in roles.splitlines() if "*p.met = 0;" in s)
    assert "FUSE && !BOTH" in line and "pdl_wait();" in roles[:roles.index(line)].splitlines()[-1]
    both = code[code.index("gemm_both_kernel(const __grid_constant__"):]
    tail = both[both.index("gemm_teardown<C>(x);"):]
    assert "p2.met" not in both[:both.index("gemm_teardown<C>(x);")] and "x.ok" not in tail
    assert tail.index("__threadfence();") < tail.index("atomicAdd(p2.met + 1, 1) == (int)gridDim.x - 1") < tail.index("p2.met[0] = 0; p2.met[1] = 0;")

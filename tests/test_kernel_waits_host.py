"""The tensor-core kernels promise bounded waits: on expiry a warp sets the status word and leaves, so no other warp may be left
waiting for it without a limit.  Read from the sources, where the warps have parted into roles."""
import os
import re

import pytest

KERNELS = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "orion_b200", "csrc", "kernels")


def _roles(name):
    """The part of the kernel in which its warps have different roles: from the abort flag's pointer to the barrier of the teardown."""
    text = open(os.path.join(KERNELS, name)).read()
    text = re.sub(r"//[^\n]*", "", text)
    body = text[text.index("volatile int* abort_flag = &ctl->abort_flag"):]
    return body[:body[:body.index("tmem_dealloc")].index("__syncthreads()")]


@pytest.mark.parametrize("name", ["igemm_fprop.cu", "gemm_bf16.cu", "attention.cu"])
def test_no_unbounded_barrier_between_roles(name):
    """... except the implicit GEMM's one named barrier, which the next test is about."""
    roles = _roles(name)
    assert "mbar_wait" in roles
    found = re.findall(r"bar\.sync|barrier\.sync|barrier\.cluster|__syncthreads|cluster_sync_all", roles)
    assert found == (["bar.sync"] if name == "igemm_fprop.cu" else [])


def _block(text, start):
    """The braces' contents that open at or behind `start`."""
    i = j = text.index("{", start)
    depth = 0
    while True:
        depth += {"{": 1, "}": -1}.get(text[j], 0)
        j += 1
        if depth == 0:
            return text[i + 1:j - 1]


def test_an_epilogue_warp_that_gives_up_keeps_meeting_the_others():
    """The implicit GEMM's epilogue warps meet at a named barrier around every piece of a cut tile.  The barrier is whole only if
    no warp leaves the walk over the pieces early, and a warp that has given up meets the others as often as one that has not."""
    roles = _roles("igemm_fprop.cu")
    epilogue = _block(roles, roles.index("if (epi_id >= 0)"))
    head = re.search(r"for \(; ([^;]*); local\+\+\)", epilogue)
    assert head.group(1) == "ok && work.next(seg)"
    walk = _block(epilogue, head.end())
    behind = epilogue[epilogue.index(walk) + len(walk):]
    given_up = _block(behind, behind.index("if (!ok && p.mode == 0)"))
    assert re.match(r"\s*do \{\s*if \(seg\.nseg > 1\)", given_up) and given_up.rstrip().endswith("while (work.next(seg));")
    assert given_up.count("meet()") == walk.count("meet()") == 3 and "return" not in walk
    # left with the piece's own three meetings behind it only where it says so
    assert walk.index("seg.nseg = 0;") > walk.rindex("meet()")
    for m in re.finditer(r"\bbreak;", walk):
        opened = []   # the headers of the blocks around it
        for i, ch in enumerate(walk[:m.start()]):
            if ch == "{":
                opened.append(re.split(r"[;{}]\s*\n", walk[:i])[-1])
            elif ch == "}":
                opened.pop()
        assert any("for (" in h for h in opened) or walk[:m.start()].rstrip().endswith("ok = false;")

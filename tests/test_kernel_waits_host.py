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
    assert head.group(1) == "__builtin_expect(ok, 1) && work.next(seg)"
    walk = _block(epilogue, head.end())
    behind = epilogue[epilogue.index(walk) + len(walk):]
    given_up = _block(behind, behind.index("if (__builtin_expect(!ok, 0) && p.mode == 0)"))
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


SHIM = """
#include <cstdint>
static int waited[64][2], waits;
static inline void mbar_wait_landed(uint64_t* bar, uint32_t parity, long long) { waited[waits][0] = (int)*bar; waited[waits++][1] = (int)parity; }
static inline void __syncwarp() {}
static inline long long clock64() { return 0; }
#define __device__
#define __forceinline__ inline
%s
extern "C" int settle(int stages, int used, int back, int* out) {
    uint64_t bars[16];
    for (int i = 0; i < stages; i++) bars[i] = i;
    waits = 0;
    ring_settle(bars, stages, used %% stages, (uint32_t)(used / stages) & 1u, back);
    for (int i = 0; i < waits; i++) { out[2 * i] = waited[i][0]; out[2 * i + 1] = waited[i][1]; }
    return waits;
}
"""


@pytest.fixture(scope="module")
def settle(tmp_path_factory):
    import ctypes
    import subprocess
    text = open(os.path.join(KERNELS, "sm100_primitives.cuh")).read()
    start = text.index("__device__ __forceinline__ void ring_settle")
    func = text[start:text.index("{", start)] + "{" + _block(text, start) + "}"
    d = tmp_path_factory.mktemp("settle")
    (d / "settle.cpp").write_text(SHIM % func)
    subprocess.run(["g++", "-shared", "-fPIC", "-std=c++17", "-o", str(d / "settle.so"), str(d / "settle.cpp")], check=True)
    fn = ctypes.CDLL(str(d / "settle.so")).settle

    def call(stages, used, back):
        out = (ctypes.c_int * 128)()
        n = fn(stages, used, back, out)
        return [(out[2 * i], out[2 * i + 1]) for i in range(n)]
    return call


@pytest.mark.parametrize("stages", [1, 2, 3, 4, 6, 8])
def test_a_role_that_leaves_waits_for_the_last_lap_of_its_ring(settle, stages):
    """After `used` uses of the ring: the newest phase of every stage (use n of a stage is its barrier's phase n // stages), and for a
    stage never used the phase before the first, which counts as complete."""
    for used in range(0, 4 * stages + 1):
        want = {s: (max(n // stages for n in range(used) if n % stages == s) & 1 if used > s else 1) for s in range(stages)}
        assert dict(settle(stages, used, stages)) == want and len(settle(stages, used, stages)) == stages
        last = (used - 1) % stages
        assert settle(stages, used, 1) == [(last, want[last])]


@pytest.mark.parametrize("name,copies,products", [("igemm_fprop.cu", ["ctl->raw_full"], ["ctl->empty"]), ("gemm_bf16.cu", ["ctl->full"], ["ctl->empty"]),
                                                  ("attention.cu", ["&ctl->k_full", "&ctl->v_full", "&ctl->q_full"], ["&ctl->s_full", "&ctl->o_full"])])
def test_roles_leave_with_no_copy_and_no_product_under_way(name, copies, products):
    """On every way out of a role, given up or not, what it set off has landed (or a bounded wait for it has run out) before the CTA's
    shared and tensor memory go."""
    roles = _roles(name)
    for bar in copies + products:
        assert re.search(r"(ring_settle|mbar_wait_landed)\(" + re.escape(bar), roles), bar
    # a warp-wide instruction behind a wait needs the same answer in all lanes
    assert not re.search(r"if \(!(dead && !)?mbar_wait\(|!timed_wait\(&ctl->(raw_full|tmem)", roles)

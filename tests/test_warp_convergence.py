"""Warp-wide instructions of the learned strip's tensor-core kernel, read from
csrc/learned.cu: between a poll (each lane leaves it by itself) or a block of
one thread's own (the MMA issue, the barrier set-up) and the next warp-wide
instruction (tcgen05.ld, alloc, dealloc, bar.sync, bar.red) stands a point
where the whole warp meets."""
import os
import re

from conftest import PKG

SRC = os.path.join(PKG, "csrc", "learned.cu")


def code():
    with open(SRC) as f:
        s = f.read()
    return re.sub(r"//[^\n]*", "", s)


def body(s, head):
    """The braces' content of the definition that starts with `head`."""
    i = s.index("{", re.search(head, s).end())
    depth = 0
    for j in range(i, len(s)):
        depth += (s[j] == "{") - (s[j] == "}")
        if depth == 0:
            return s[i:j + 1]
    raise AssertionError(head)


DIVERGES = r"mbar_wait_bounded\(|mbar_init1\(|mma_commit\("
MEETS = r"__syncwarp\(\)|__syncthreads\(\)|wait_commit\(|wg_sync_or\(|wg_sync\("
WARP_WIDE = r"tmem_ld16\(|hidden_half\(|tcgen05\.alloc|tcgen05\.dealloc|bar\.sync|bar\.red"


def unmet(text):
    """Warp-wide instructions that a diverged warp can reach, in source order."""
    diverged, bad = None, []
    for m in re.finditer("(?P<d>%s)|(?P<m>%s)|(?P<w>%s)" % (DIVERGES, MEETS, WARP_WIDE), text):
        if m.group("d"):
            diverged = m.group("d")
        elif m.group("m"):
            diverged = None
        elif diverged:
            bad.append((diverged, m.group("w")))
    return bad


def test_the_kernel_meets_before_warp_wide_instructions():
    assert unmet(body(code(), r"k_strip_tc\(Model")) == []


def test_the_helpers_meet():
    """The helpers that count as meeting points above are ones: they meet first
    (the group barriers) or after their poll (wait_commit)."""
    s = code()
    for head in (r"bool wg_sync_or\(int g", r"void wg_sync\(int g"):
        b = body(s, head)
        assert b.index("__syncwarp()") < re.search(r"bar\.(sync|red)", b).start()
    b = body(s, r"bool wait_commit\(uint64_t")
    assert b.index("mbar_wait_bounded(") < b.index("__syncwarp()") < b.index("tc_after()")

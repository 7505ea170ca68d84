"""The tall kernel's tensor-memory instructions are .sync.aligned: all lanes of a
warp must arrive at each together, and nothing but a barrier makes lanes that took
different branches do so.  Checked on the source: between each of them and the last
branch or loop that can part a warp's lanes stands a barrier -- on the path with
the clusters' exchanges and on the one without."""
import os
import re

from conftest import REPO

EVENTS = re.compile(r"(?P<join>__syncwarp\(|__syncthreads\(|\.sync\(\))"
                    r"|(?P<part>if \(tid\b|if \(lane\b|= tid;|mbar_wait|c\.xindex >=|issue_copies\()"
                    r"|(?P<all>\btmem_\w+\(|\bpiv_store\()")


def block_end(s, at):
    """Past the brace that closes the first one at or after `at`."""
    depth = 0
    for i in range(s.index("{", at), len(s)):
        depth += {"{": 1, "}": -1}.get(s[i], 0)
        if depth == 0:
            return i + 1
    raise AssertionError("unbalanced braces")


def without(s, opening):
    """s without the blocks that start with `opening`."""
    while opening in s:
        at = s.index(opening)
        s = s[:at] + s[block_end(s, at):]
    return s


def test_lanes_are_together_at_every_tensor_memory_instruction():
    src = open(os.path.join(REPO, "futhark-benchmarks_b200", "csrc", "lvc_tall.cuh")).read()
    src = re.sub(r"//[^\n]*", "", src)
    src = src[src.index("lvc_line_tall_kernel(RollbackArgs"):]
    at = src.index("auto issue_copies =")
    copies = src[at:block_end(src, at)]
    joined = re.search(r"__syncwarp\(\);\s*}$", copies) is not None
    for opening in ("auto issue_copies =", "auto piv_load =", "auto piv_store ="):
        src = without(src, opening)
    checked = 0
    for view in (src, without(src, "if (clustered) {")):
        parted = None
        for e in EVENTS.finditer(view):
            if e["join"]:
                parted = None
            elif e["part"]:
                parted = None if e["part"] == "issue_copies(" and joined else e[0]
            else:
                checked += 1
                assert parted is None, f"{e[0]}...) follows {parted}...) with no barrier between"
    assert checked >= 20

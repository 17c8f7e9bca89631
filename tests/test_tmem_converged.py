"""tcgen05.ld is one instruction of a converged warp (.sync.aligned).  Epilogues reach it from branches that split the lanes, and no
run shows whether they are together again, so the text is read: a join of the warp (__syncwarp, or a vote) stands between every such branch and
the load that comes next, round the loop included, and the wait that lane 0 polls alone ends with one."""
import re

import pytest

from test_cluster_order import kernel_body

JOIN = r"__syncwarp\(\);|__any_sync\(|__all_sync\(|wait_acc\(\d|mbar_wait_warp\(|load_acc\(t"  # wait_acc ends with a vote, load_acc begins with a join
SPLIT = r"if \(row_ok\)|if \(row < p\.M|\) continue;|finish_cols<|finish\(b0|mbar_wait\(|if \(i < p\.len\)|if \(threadIdx\.x == \d+\)|if \(lane == 0\)"
LOAD = r"tmem_ld\w*\("


def closing(text, at, pair):
    """Position behind the bracket that closes the one at `at`."""
    depth = 0
    for i in range(at, len(text)):
        depth += (text[i] == pair[0]) - (text[i] == pair[1])
        if depth == 0:
            return i + 1


def block_of(body, at, head):
    """The innermost braced block behind a match of `head` (which ends with an open round bracket) that holds position `at`."""
    best = None
    for m in re.finditer(head, body[:at]):
        behind = closing(body, m.end() - 1, "()")
        if body[behind:].lstrip().startswith("{"):
            start = body.index("{", behind)
            end = closing(body, start, "{}")
            if start < at < end:
                best = (start, end)
    return best


@pytest.mark.parametrize("path,name", [("gemm_tc.cu", "gemm_tc_kernel"), ("gemm_smallm.cu", "gemm_smallm_kernel"), ("gemm_wide.cu", "gemm_wide_kernel"),
                                       ("gemm_mid.cu", "gemm_mid_kernel"), ("attn_prefill.cu", "attn_prefill_kernel")])
def test_loads_come_after_a_join(path, name):
    body = kernel_body("llm.cu_b200/csrc/" + path, name)
    events = sorted([(m.start(), "join") for m in re.finditer(JOIN, body)] + [(m.start(), "split") for m in re.finditer(SPLIT, body)])
    loads = [m.start() for m in re.finditer(LOAD, body)]
    assert loads

    def last(lo, hi):
        seen = [kind for pos, kind in events if lo <= pos < hi]
        return seen[-1] if seen else None
    while loads:
        at = loads.pop()
        function = block_of(body, at, r"= \[&\]\(")
        if function and last(function[0], at) is None:  # a local function without a join of its own: its calls count
            loads += [m.start() for m in re.finditer(r"\b%s\(" % re.findall(r"auto (\w+) = \[&\]", body[:at])[-1], body)]
            continue
        assert last(function[0] if function else 0, at) == "join", body[at - 300:at + 40]
        loop = block_of(body, at, r"\bfor \(")
        if loop:  # once round the loop
            assert (last(loop[0], at) or last(at, loop[1])) in ("join", None), body[at - 300:at + 40]


def test_warp_wait_ends_converged():
    body = kernel_body("llm.cu_b200/csrc/common.cuh", "bool mbar_wait_warp")
    assert body.rstrip().endswith("return __all_sync(0xffffffffu, ok != 0);")

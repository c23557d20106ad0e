"""Waits that can run out, as the kernels' sources have them: a bounded wait gives each lane an answer of its own, so in a
branch with warp-collective instructions (shuffles, votes, reductions, tcgen05.ld) the lanes have to agree before they act
on it; lanes that leave such a branch alone hang the CTA.  The sources are read, nothing is run: a wait that runs out on
some lanes only cannot be provoked on a GPU without hanging it where the vote is missing."""
import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "sgl_analytic_gb300" / "csrc"
WAIT = re.compile(r"\b(?:mbar_wait_bounded|mbar_wait_sleep|wait_consumed)\s*\(")
COLLECTIVE = re.compile(r"__shfl\w*_sync|__reduce_\w+_sync|__syncwarp|\btmem_ld16|\bmf_ld8\b|\bxf_ld4\b")
VOTE = re.compile(r"\bwarp_all\s*\(|__any_sync|__all_sync|__syncthreads_and")
SINGLE = re.compile(r"lane\s*==\s*0|tid\s*==\s*\d+")


def _code(path):
    """The source without comments and string literals."""
    s = path.read_text()
    s = re.sub(r"//[^\n]*|/\*.*?\*/", "", s, flags=re.S)
    return re.sub(r'"(?:\\.|[^"\\])*"', '""', s)


def _blocks(s):
    """(header, start, end) of every braced block; the header is the text since the last ; { or }."""
    stack, out = [], []
    for i, c in enumerate(s):
        if c == "{":
            h = max(s.rfind(x, 0, i) for x in ";{}") + 1
            p = s.rfind("(", 0, i)                         # a for header holds semicolons
            while p >= 0 and s[p:i].count("(") != s[p:i].count(")"):
                p = s.rfind("(", 0, p)
            if re.search(r"\bfor\s*$", s[:p]):
                h = min(h, s.rfind("for", 0, p))
            stack.append((s[h:i], i))
        elif c == "}":
            head, start = stack.pop()
            out.append((head, start, i))
    return out


def _unvoted(path):
    s = _code(path)
    blocks = _blocks(s)
    bad = []
    for m in WAIT.finditer(s):
        around = sorted((b for b in blocks if b[1] < m.start() < b[2]), key=lambda b: b[2] - b[1])
        # the wait's own definition, and lambdas that return its answer to a caller
        stmt0 = max(s.rfind(x, 0, m.start()) for x in ";{}") + 1
        stmt = s[stmt0:s.find(";", m.start())]
        if not around or re.match(r"\s*(?:__device__|return\b|template)", stmt):
            continue
        if any(SINGLE.search(h) for h, _, _ in around) or SINGLE.search(stmt):
            continue
        # the vote: in the same statement, or in the next one
        after = s[s.find(";", m.start()) + 1:]
        if VOTE.search(stmt) or VOTE.search(after[:after.find(";")]):
            continue
        # the role: the widest block around the wait that is a branch on the warp or on lanes, or a loop in one
        role = [b for b in around if re.search(r"\bwarp\b|\belse\s*$|\bfor\b", b[0])]
        if any(COLLECTIVE.search(s[a:e]) for _, a, e in role):
            bad.append((path.name, s.count("\n", 0, m.start()) + 1, " ".join(stmt.split())))
    return bad


@pytest.mark.parametrize("name", ["xi_fused.cu", "mlp_fused.cu", "oz_gemm.cu", "tc_gemm.cu"])
def test_lanes_of_a_warp_agree_on_a_wait_that_ran_out(name):
    assert _unvoted(CSRC / name) == []


def test_a_cta_that_gave_up_waits_for_its_bulk_copies():
    """A bulk copy that lands after its CTA has ended writes into the next one's shared memory.  Every kernel that issues
    them has a loop of waits over those issued but not taken, after the roles (mlp_fused: at the end of the copy role)."""
    wait = re.compile(r"for \([^{;]*;[^{;]*(?:\bissued\b|\bj >= 0\b)[^{;]*;[^{;]*\)\s*(?:if \(!)?mbar_wait_(?:bounded|sleep)\(")
    for name in ("xi_fused.cu", "mlp_fused.cu", "oz_gemm.cu", "tc_gemm.cu"):
        s = _code(CSRC / name)
        for kernel in re.split(r"__global__", s)[1:]:
            if "bulk_g2s(" in kernel:
                assert wait.search(kernel, kernel.rindex("bulk_g2s(")), (name, " ".join(kernel[:120].split()))

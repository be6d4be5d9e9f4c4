"""CPU: the Gram kernel's warps that wait as a whole vote on the outcome.

A bounded wait ends for each lane by itself: one lane may see the phase complete while
another gives up.  Warp-wide operations with a full mask follow (elect.sync, ballots,
aligned tensor-memory loads), so lanes that disagreed would block there without limit.
Only the copy producer waits in a single lane; every other wait is the argument of a
vote, or reaches one before any branch on it."""
import os
import re

from conftest import ROOT


def gram_kernel():
    src = open(os.path.join(ROOT, "tensor_bf_main_gb300", "csrc", "k_umma.cu")).read()
    src = re.sub(r"//[^\n]*", "", src)
    body = src[src.index("gram_kernel(const __grid_constant__"):]
    return body[: body.index("uint64_t gram_queue_slack")]


def outcomes(text):
    """(variable, statement) of every wait: the variable that a statement assigns, or
    None where the statement assigns none."""
    out = []
    for m in re.finditer(r"ptx::mbar_(?:test_)?wait\(", text):
        start = max(text.rfind(c, 0, m.start()) for c in ";{}") + 1
        stmt = text[start: text.index(";", m.end())]
        a = re.match(r"\s*(?:const\s+)?(?:bool\s+)?(\w+)\s*=", stmt)
        out.append((a.group(1) if a else None, " ".join(stmt.split()), text[text.index(";", m.end()):]))
    return out


def test_every_wait_of_a_whole_warp_is_voted_on():
    body = gram_kernel()
    issuer = body[body.index("} else if (warp == 1) {"):]
    waits = outcomes(issuer)
    assert len(waits) >= 5
    for var, stmt, rest in waits:
        if "__all_sync(FULL" in stmt or "= take(" in stmt:
            continue
        # otherwise the variable reaches the vote that its function returns, and nothing
        # but further waits lies between
        assert var is not None, stmt
        vote = re.search(r"__all_sync\(FULL, %s\)" % var, rest)
        assert vote, stmt
        between = rest[: vote.start()]
        assert "elect_one" not in between and "__syncwarp" not in between, stmt
        assert not re.search(r"\b(for|while|break|continue)\b", between), stmt
        for cond in re.findall(r"if \(([^)]*)\)", between):
            assert cond == "SPLIT", stmt

"""Waits of the tensor-memory kernel, by its source.  An mbarrier wait answers
each lane for itself, and lanes of a warp may be answered differently.  Behind
the waits stand instructions that a whole warp has to reach together
(``tcgen05.ld.sync.aligned``, ``elect.sync``), so the lanes meet first, and
whether they do is never up to a lane's own answer.  A lane that goes its own
way could hang the GPU, so this is read here and not tried there."""
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                    "beampower_b200", "csrc")
MEET = ("__syncwarp()", "__all_sync(0xFFFFFFFFu, ok)")


def _struct():
    with open(os.path.join(CSRC, "bp_tmem.cuh")) as fh:
        text = re.sub(r"//[^\n]*", "", fh.read())
    return text[text.index("struct Tm {"):]


def test_lanes_meet_after_a_wait():
    text = _struct()
    waits = [m.end() for m in re.finditer(r"\bmbar_wait_spin\(", text)]
    assert len(waits) >= 3
    for at in waits:
        rest = text[at:]
        meet = min(rest.index(x) for x in MEET if x in rest)
        together = re.search(r"tm_fence_after|tm_cp\(|elect_one|\bload\(|bulk_g2s|__shfl|return true",
                             rest)
        assert meet < together.start(), rest[:120]


def test_a_lane_s_answer_is_voted_on():
    text = _struct()
    answer = re.findall(r"(\w+) = mbar_try_wait_at\(", text)
    assert answer == ["ready"] and text.count("mbar_try_wait_at(") == 1
    uses = re.findall(r"[^\n]*\bready\b[^\n]*", text)
    assert [u.strip() for u in uses if "mbar_try_wait_at" not in u and "false" not in u] == \
        ["tm_take(sm, u.n, status, ready);"]
    take = text[text.index("void tm_take("):]
    take = re.sub(r"\s+", " ", take[:take.index("\n  }")])
    assert re.search(r"if \(!__all_sync\(0xFFFFFFFFu, seen\)\) { mbar_wait_spin\([^;]*; "
                     r"__syncwarp\(\); } tm_fence_after\(\);$", take.strip())

"""The barriers of the streaming kernel (tcec_gemm_stream.cu), as its source declares them.

A wait on a barrier tells phases apart by one bit, so it is safe only where the waiter has looked at the
phase before (a barrier that is still in it looks like one that has ended the phase waited for), and
where the phase after cannot have ended yet (that looks like the one waited for is still open).
Checked here on the order in which every waiter uses its barriers: arrivals on different barriers (a
commit's on the other CTA of a pair among them) have no order of their own."""
import re
from pathlib import Path

import pytest

SOURCE = (Path(__file__).resolve().parent.parent / "cumpsgemm_b200" / "csrc" /
          "tcec_gemm_stream.cu").read_text()


def _constants(bn, cg):
    """StreamCfg's integer constants for one pair of template arguments."""
    body = SOURCE[SOURCE.index("struct StreamCfg {"):]
    body = re.sub(r"//[^\n]*", "", body[:body.index("\n};")])
    known = {"BN": bn, "CG": cg, "BM_CTA": 128, "ROW_BYTES": 128, "SLOT_K": 32, "CVT_TEAMS": 2,
             "TEAM_WARPS": 8}
    for name, expr in re.findall(r"static constexpr (?:int|uint32_t|bool) (\w+) = ([^;,]+);", body):
        expr = expr.replace("/", "//")
        while "?" in expr:                        # C's conditional, innermost last
            cond, rest = expr.split("?", 1)
            yes, no = rest.split(":", 1)
            expr = no if not eval(cond, {}, known) else yes
        try:
            known[name] = eval(expr, {}, known)
        except NameError:                         # (needs something that is not a number)
            pass
    return known


def _phases_are_told_apart(waits, bars):
    """waits: (event, own) in the order one waiter waits, where event number u is the (u // bars)-th phase
    of barrier u % bars and cannot end before the waiter has come past every wait with own <= u."""
    seen = {}
    for event, own in waits:
        if event < 0:
            continue                              # nothing to wait for yet
        barrier, phase = event % bars, event // bars
        if phase != seen.get(barrier, -1) + 1:
            return False                          # passed over a phase
        if event + bars < own:
            return False                          # the phase after it may have ended too
        seen[barrier] = phase
    return True


CONFIGS = [(256, 2), (128, 2), (128, 1)]


@pytest.mark.parametrize("bn,cg", CONFIGS)
def test_epilogue_halves_tell_the_phases_of_their_accumulators_apart(bn, cg):
    c = _constants(bn, cg)
    bars = c.get("D_FULL_BARS", c["D_BUFS"])
    for half in (0, 1):                           # the halves of the columns are filled in turn
        # (fill f + D_BUFS of an accumulator comes after the drain of fill f)
        assert _phases_are_told_apart([(f, f + c["D_BUFS"]) for f in range(half, 64, 2)], bars)
    # the accumulator of a fill follows from its barrier
    assert all(f % c["D_BUFS"] == (f % bars) % c["D_BUFS"] for f in range(64))


@pytest.mark.parametrize("bn,cg", CONFIGS)
@pytest.mark.parametrize("kind", ["fp16", "tf32"])
def test_converter_teams_tell_the_phases_of_their_stages_apart(bn, cg, kind):
    c = _constants(bn, cg)
    stages, bars = c["STAGES"], c.get("EMPTY_BARS", c["STAGES"])
    # all warps fill every stage; or, TF32 with slots that the teams take in turn, one of two teams does
    step = 1 if kind == "fp16" or c["SLOT_TEAMS"] == 1 else 2
    for total in ([1, 2, 3, 64, 65] if kind == "fp16" else [2, 4, 6, 8, 64]):
        last = set()
        for team in (0, 1):
            # use u of the ring waits for the release of use u - stages; the last ones are waited for too
            uses = range(0 if step == 1 else team, total + stages, step)
            assert _phases_are_told_apart([(u - stages, u) for u in uses], bars)
            last |= {u - stages for u in uses if u >= max(total, stages)}
        assert last == set(range(max(total, stages) - stages, total))
    # the stage of a use follows from the barrier it waits on
    assert all((u + stages) % bars % stages == u % stages for u in range(64))


@pytest.mark.parametrize("bn,cg", CONFIGS)
def test_a_raw_slot_belongs_to_one_team_or_to_all_warps(bn, cg):
    c = _constants(bn, cg)
    assert c["SLOT_TEAMS"] in (1, 2) and c["RAW_SLOTS"] % c["SLOT_TEAMS"] == 0
    # slot u of the stream is refilled once its u-th use has been given back: each of its phases is seen
    for team in range(c["SLOT_TEAMS"]):
        uses = range(team, 64, c["SLOT_TEAMS"])
        assert _phases_are_told_apart([(u, u + c["RAW_SLOTS"]) for u in uses], c["RAW_SLOTS"])

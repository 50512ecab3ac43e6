"""How a warp of the tcgen05 kernels ends when a bounded wait runs out (csrc/sm100.cuh, csrc/chunkwise_sm100.cu), on the
CPU: a lane-level model of a warp whose lanes poll for themselves, and a check that the kernels' warp-wide waits have the
form that the model shows to be sound.  No GPU wait is made to expire: the failure is an interleaving of the model."""

import os
import random
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "mlstm_kernels_b200", "csrc")
LANES, POLLS, ROUNDS = 4, 6, 3


def lane(i, state, on_failure):
    """One lane: rounds of (bounded wait, warp-wide operation, arrival of lane 0).  Yields "operation" where the whole
    warp has to come together; the polls of the lanes interleave freely.  After a failed wait the lane leaves, or goes on
    without waits and arrivals ("flag"), or without the arrival that follows the wait ("answer"), or without arrivals
    once any wait has run out ("abort flag"), or only meets the others in the operations that are left ("stand by")."""
    ok = True
    for round_ in range(ROUNDS):
        if ok or on_failure in ("answer", "abort flag"):
            ok = False
            for poll in range(POLLS):
                yield "poll"                            # another lane, or the barrier, may move here
                if state["complete"] > round_:
                    ok = True
                    break
                if poll % 2 == 1 and state["abort"]:
                    break
            else:
                state["abort"] = True
            if on_failure == "leave" and not ok:
                return
            if on_failure == "stand by" and not ok:
                for _ in range(round_, ROUNDS):
                    yield "operation"
                return
        yield "operation"                               # elect, shuffle, tensor-memory access
        if i == 0 and (not state["abort"] if on_failure == "abort flag" else ok):
            assert state["complete"] > round_, "arrival without the phase that it follows"
            state["arrivals"] += 1


def run(seed, on_failure):
    rnd = random.Random(seed)
    state = {"complete": 0, "abort": False, "arrivals": 0}
    lanes = [lane(i, state, on_failure) for i in range(LANES)]
    at = [next(x) for x in lanes]
    alive = set(range(LANES))

    def advance(i):
        try:
            at[i] = next(lanes[i])
        except StopIteration:
            alive.discard(i)

    while alive:
        # a phase completes at any time, or too late, and needs this warp's arrival of the round before
        if rnd.random() < 0.05 and state["complete"] <= state["arrivals"]:
            state["complete"] += 1
        movable = [i for i in alive if at[i] == "poll"]
        if movable:
            advance(rnd.choice(movable))
        else:
            assert len(alive) == LANES, "lanes wait in a warp-wide operation for others that have left"
            for i in range(LANES):
                advance(i)
    return state


@pytest.mark.parametrize("on_failure", ["flag", "answer", "abort flag", "stand by"])
def test_lanes_that_go_on_end_together(on_failure):
    expired = 0
    for seed in range(4000):
        expired += run(seed, on_failure)["abort"]
    assert 400 < expired < 3600      # both kinds of run were seen


def test_lanes_that_leave_alone_would_block_the_others():
    with pytest.raises(AssertionError, match="others that have left"):
        for seed in range(5000):
            run(seed, "leave")


# The waits of single threads, by their status code: the MMA thread, the store thread, the intra-chunk producer, the
# expiry self-test; code 0 lets copies in flight land on the error path.  Every other wait is a whole warp's.
ONE_THREAD = {"102", "103", "108", "201", "202", "203", "204", "212", "213", "215", "216", "217", "0", "code"}


def test_no_lane_leaves_a_warp_alone():
    with open(os.path.join(CSRC, "chunkwise_sm100.cu")) as f:
        src = f.read()
    calls = re.findall(r"^([^\n]*)\bmbar_wait\(&[^;\n]*?, (?:&g_sm100_status|nullptr), (\w+)(?:, limit)?\)([^\n]*)\n([^\n]*)",
                       src, re.M)
    assert len(calls) >= 25
    for before, code, after, next_line in calls:
        if code in ONE_THREAD:
            continue
        left = "break" in after or "return" in after or "break" in next_line or "return" in next_line
        stands_by = "stand_by(h, " in after or "__syncwarp();" in next_line
        assert stands_by or (not left and "if (!" not in before), f"wait with status code {code}"
    # hand-overs to other roles depend on the wait before them
    for bar, flag in (("gated", "acc_ok"), ("accfree", r"!aborted\(smem_u32\(&sh\.abort\)\)"), (r"done\[sub & 1\]", r"!aborted\(smem_u32\(&sh\.abort\)\)")):
        assert re.findall(rf"(.*)mbar_arrive\(&sh\.bar_{bar}\)", src) == [re.search(rf" *if \({flag}\) (?=mbar_arrive\(&sh\.bar_{bar}\))", src).group(0)]
    for bar in ("out_full", "acc_free"):
        assert re.search(rf"warp_arrive\(&bar_{bar}\[\w+\], ok\)", src)


# the same of the roles that the shipped recurrence and the intra-chunk backward have: the recurrence's producers, and producer,
# MMA and E-tile thread of the backward
ONE_THREAD_OF_RINGS = ONE_THREAD | {"101", "110", "111", "113", "301", "302", "303", "304", "305", "306", "307"}


@pytest.mark.parametrize("name,status,least", [("chunkwise_sm100.cu", "g_sm100_status", 25), ("chunkwise_bw_sm100.cu", "g_par_bw_status", 11)])
def test_no_lane_leaves_a_warp_alone_in_any_wait(name, status, least):
    with open(os.path.join(CSRC, name)) as f:
        src = f.read()
    pattern = rf"\bmbar_wait(?:<true>)?\(&[^;\n]*?, (?:&{status}|nullptr), (\w+)(?:, limit)?\)"
    calls = re.findall(rf"^([^\n]*){pattern}([^\n]*)\n([^\n]*)", src, re.M)
    assert len(re.findall(pattern, src)) == len(re.findall(r"\bmbar_wait(?:<true>)?\(", src)) >= least    # none is overlooked
    for before, code, after, next_line in calls:
        if code in ONE_THREAD_OF_RINGS:
            continue
        left = "break" in after or "return" in after or "break" in next_line or "return" in next_line
        assert "__syncwarp();" in next_line or (not left and "if (!" not in before), f"wait with status code {code}"

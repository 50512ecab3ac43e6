"""Model of the recurrence kernel's protocol (csrc/chunkwise_sm100.cu, rec_body) with its two operand rings and the ring of
gated tiles in tensor memory, run on the CPU.

Its roles hand work around rings whose barriers run on over the whole sequence (thousands of phases), every wait seeing only
the phase PARITY: two TMA producers (the left and the right operand; one for both with 64-column tiles), two groups of four
gating warps, the MMA thread, eight state warps, and the warp that stores the states and keeps n.  The order of waits,
arrivals, copy issues and MMA commits of each is restated here and run under random interleavings - copies land in any order,
commits fire in order - with every wait checked against the true phase count (a waiter two phases away from its barrier,
early or late, is a hang or a corruption), every barrier against over-arrival, the run against deadlock, tensor-memory tiles
and operand slots against being overwritten under a reader, and the ring of chunk decays against races: every thread
carries a vector clock, handed on by arrivals and taken up by waits, and a read of a decay must be ordered after its write,
the write that overwrites it after all its reads.  The depths are read from the source; the order of operations is kept next
to the kernel by hand."""

import os
import random
import re

import pytest

from test_rec_protocol_model import Bar, join

SRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "mlstm_kernels_b200", "csrc", "chunkwise_sm100.cu")


def depths():
    """(left ring, right ring) with 128-column and with 64-column tiles, which have one ring for both; gated tiles; decays."""
    with open(SRC) as f:
        src = f.read()
    pair = [re.search(rf"int {n}\(int TN\) \{{ return TN == 128 \? (\d+) : (\d+); \}}", src).groups() for n in ("rec_stages", "rec_right_stages")]
    one = [int(re.search(rf"constexpr int {n} = (\d+);", src).group(1)) for n in ("REC_LBUF", "G_RING")]
    assert "constexpr bool JOINT = TN == 64;" in src
    return [(int(pair[0][0]), int(pair[1][0]), *one, False), (int(pair[0][1]), int(pair[1][1]), *one, True)]


def run(NC, do_n, store_states, seed, rings, slow=None, decay_writer="left"):
    """slow: a role that gets its turn late.  decay_writer: the lane that writes the decays, "left" being the one that arrives
    on the stage's barrier."""
    left, right, lbuf, g_ring, joint = rings
    rnd = random.Random(seed)
    NH2 = 2 * NC
    count = {f"full{s}": 1 for s in range(left)}
    count.update({f"empty{s}": 4 for s in range(left)})
    count.update({f"rfull{s}": 1 for s in range(right)})
    count.update({f"{n}{s}": c for s in range(lbuf) for n, c in (("scaled", 4), ("done", 1))})
    count.update({f"{n}{s}": c for s in range(2) for n, c in (("acc_free", 8), ("nsum", 8), ("nread", 1), ("out_full", 8),
                                                              ("out_free", 1))})
    B = {n: Bar(n, c) for n, c in count.items()}
    loads, commits, clocks = [], [], {}
    written, reads = [None] * g_ring, [[] for _ in range(g_ring)]
    multiplied = [0] * lbuf          # products in flight that read a gated tile
    landed = [s - right for s in range(right)]   # half chunk in each slot of the right ring

    def tick(a):
        clocks[a][a] = clocks[a].get(a, 0) + 1
        return clocks[a][a]

    def arrive(a, name):
        tick(a)
        B[name].arrive(clocks[a])

    def read_decay(a, s):
        w, t, chunk = written[s % g_ring]
        assert chunk == s, f"{a} reads the decay of chunk {chunk} for that of {s}"
        assert clocks[a].get(w, 0) >= t, f"{a} reads the decay of chunk {s} unordered"
        reads[s % g_ring].append((a, tick(a)))

    def left_producer():
        for h in range(NH2):
            s = h >> 1
            if not joint:
                yield f"empty{h % left}", h // left - 1
            elif h >= left:
                yield f"done{(h - left) % lbuf}", (h - left) // lbuf
            if h % 2 == 0:
                for r, t in reads[s % g_ring]:
                    assert clocks[decay_writer].get(r, 0) >= t, f"decay of chunk {s - g_ring} overwritten before {r} is known to have read it"
                if s >= g_ring:
                    assert len(reads[s % g_ring]) == 8 + do_n, "decay overwritten before it is read"
                reads[s % g_ring].clear()
                written[s % g_ring] = (decay_writer, tick(decay_writer), s)
            tick("left")
            assert not joint or landed[h % right] == h - right
            loads.append((f"full{h % left}", dict(clocks["left"])))

    def right_producer():
        for h in range(NH2):
            if h >= right:
                yield f"done{(h - right) % lbuf}", (h - right) // lbuf
            assert landed[h % right] == h - right, "load over an operand that has not been used"
            loads.append((f"rfull{h % right}", dict(clocks["right"])))

    def mma():
        for h in range(NH2):
            s, lb = h >> 1, h % lbuf
            if h % 2 == 0:
                yield f"acc_free{s & 1}", (s >> 1) - 1
            if not joint:
                yield f"rfull{h % right}", h // right
            yield f"scaled{lb}", h // lbuf
            tick("mma")
            multiplied[lb] += 1
            commits.append((("product", lb), None))
            assert landed[h % right] == h, "product of an operand that has not landed"
            commits.append((f"done{lb}", dict(clocks["mma"])))

    def gating(w, group):
        for h in range(group, NH2, 2):
            s, lb = h >> 1, h % lbuf
            yield f"full{h % left}", h // left
            if not joint:
                arrive(w, f"empty{h % left}")
                yield f"done{lb}", h // lbuf - 1
            assert multiplied[lb] == 0, "gated over a tile that a product reads"
            arrive(w, f"scaled{lb}")
            if do_n:
                yield f"nread{s & 1}", (s >> 1) - 1
                arrive(w, f"nsum{s & 1}")

    def store_and_n():
        for n in range(NC + 1):
            if store_states:
                yield f"out_full{n & 1}", n >> 1
                if n >= 1:
                    arrive("store", f"out_free{(n & 1) ^ 1}")
            if do_n and n < NC:
                yield f"nsum{n & 1}", n >> 1
                read_decay("store", n)
                arrive("store", f"nread{n & 1}")

    def state(w):
        for n in range(NC + 1):
            if n > 0:
                s = n - 1
                yield f"done{(2 * s + 1) % lbuf}", (2 * s + 1) // lbuf
                read_decay(w, s)
                arrive(w, f"acc_free{s & 1}")
            if store_states:
                yield f"out_free{n & 1}", (n >> 1) - 1
                arrive(w, f"out_full{n & 1}")

    agents = {"left": left_producer(), "mma": mma(), "store": store_and_n()}
    if not joint:
        agents["right"] = right_producer()
    for w in range(8):
        agents[f"gate{w}"] = gating(f"gate{w}", w >> 2)
        agents[f"state{w}"] = state(f"state{w}")
    clocks.update({a: {} for a in [*agents, decay_writer]})
    blocked = {}

    def acquire(a, bar, phase):
        if phase >= 0:
            for lane in {a, decay_writer} if a == "left" else (a,):
                join(clocks[lane], B[bar].released.get(phase, {}))

    while agents:
        choices = list(agents) + (["land"] if loads else []) + (["commit"] if commits else [])
        rnd.shuffle(choices)
        if slow is not None and rnd.random() < 0.95:
            choices.sort(key=lambda c: c == slow)
        for c in choices:
            if c == "land":
                bar, clock = loads.pop(rnd.randrange(len(loads)))
                B[bar].arrive(clock)
                if bar.startswith("full" if joint else "rfull"):
                    landed[int(bar.lstrip("rful"))] += right
                break
            if c == "commit":
                bar, clock = commits.pop(0)
                if isinstance(bar, tuple):
                    multiplied[bar[1]] -= 1
                else:
                    B[bar].arrive(clock)
                break
            if c in blocked:
                bar, phase = blocked[c]
                if not B[bar].test(phase):
                    continue
                del blocked[c]
                acquire(c, bar, phase)
            try:
                bar, phase = next(agents[c])
            except StopIteration:
                del agents[c]
                break
            if phase < 0 or B[bar].test(phase):
                acquire(c, bar, phase)
            else:
                blocked[c] = (bar, phase)
            break
        else:
            raise AssertionError(f"DEADLOCK: {blocked}")


DEPTHS = depths()


@pytest.mark.parametrize("NC", [1, 2, 3, 5, 8, 17, 40])
@pytest.mark.parametrize("do_n,store_states", [(True, True), (False, True), (False, False), (True, False)])
@pytest.mark.parametrize("rings", DEPTHS)
def test_no_aliasing_deadlock_or_race(NC, do_n, store_states, rings):
    for seed in range(12):
        run(NC, do_n, store_states, seed, rings)


@pytest.mark.parametrize("slow", ["left", "right", "mma", "gate0", "gate5", "state0", "state7", "store", "land", "commit"])
@pytest.mark.parametrize("rings", DEPTHS)
def test_a_role_that_falls_behind_meets_no_barrier_two_phases_on(rings, slow):
    for seed in range(10):
        for do_n, store_states in ((True, True), (False, True), (False, False)):
            run(24, do_n, store_states, seed, rings, slow=slow)


def test_a_shorter_ring_of_decays_would_race():
    left, right, lbuf, _, joint = DEPTHS[0]
    with pytest.raises(AssertionError, match="decay"):
        for seed in range(50):
            run(40, False, True, seed, (left, right, lbuf, 8, joint), slow="state0")


@pytest.mark.parametrize("left", [3, 5])
def test_odd_left_ring_would_alias(left):
    """With an odd number of stages a gating group returns to a stage two phases later, and its wait passes on the load before
    the one it wants."""
    _, right, lbuf, g_ring, _ = DEPTHS[0]
    with pytest.raises(AssertionError, match="ALIAS early pass on full"):
        for seed in range(400):
            run(16, False, True, seed, (left, right, lbuf, g_ring, False), slow=("gate0", "gate5", None)[seed % 3])


def test_decay_written_by_another_lane_than_the_arriving_one_would_race():
    """Nothing orders another lane's write before the readers."""
    with pytest.raises(AssertionError, match="unordered"):
        run(4, True, True, 0, DEPTHS[0], decay_writer="another lane")

"""Model of the barrier protocol of the recurrence kernel (csrc/chunkwise_sm100.cu, rec_body), run on the CPU.

Six roles hand work around two rings whose barriers run on over the whole sequence (thousands of phases), every wait
seeing only the phase PARITY: the TMA producer (operand ring of half-chunk stages), two groups of four gating warps, the
MMA thread (two accumulator buffers), the state warps, the store warp (two staging buffers) and the n warp (two buffers
of partial sums, each filled by both halves of a chunk).  The order of waits, arrivals, copy issues and MMA commits of
each role is restated here and run under random interleavings - copies land in any order, commits fire in order - with
every wait checked against the true phase count (a waiter two phases away from its barrier, early or late, is a hang or
a corruption), every barrier against over-arrival, the run against deadlock, and the eight-entry ring of chunk decays
against races: every thread carries a vector clock, handed on by arrivals and taken up by waits, and a read of a decay
must be ordered after its write, the write that overwrites it after all its reads.  The ring depths are read from the kernel's source; the order of
operations is a model, kept next to the kernel by hand."""

import os
import random
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "mlstm_kernels_b200", "csrc")


def ring_depths():
    """Stages of the operand ring with 128-column and with 64-column tiles."""
    with open(os.path.join(CSRC, "chunkwise_sm100.cu")) as f:
        m = re.search(r"int rec_stages\(int TN\) \{ return TN == 128 \? (\d+) : (\d+); \}", f.read())
    return tuple(int(x) for x in m.groups())


def join(into, other):
    for a, t in other.items():
        if into.get(a, 0) < t:
            into[a] = t


class Bar:
    def __init__(self, name, count):
        self.name, self.count, self.pending, self.phase = name, count, count, 0
        self.clock, self.released = {}, {}    # of the arrivals of the current phase; per completed phase

    def arrive(self, clock):
        self.pending -= 1
        assert self.pending >= 0, f"over-arrival on {self.name}"
        join(self.clock, clock)
        if self.pending == 0:
            self.released = {self.phase: self.clock, self.phase - 1: self.released.get(self.phase - 1, {})}
            self.phase += 1
            self.pending = self.count
            self.clock = {}

    def test(self, want):
        passes = (self.phase & 1) != (want & 1)      # what the hardware sees
        truth = self.phase > want
        if passes and not truth:
            raise AssertionError(f"ALIAS early pass on {self.name}: want {want} at {self.phase}")
        if truth and not passes:
            raise AssertionError(f"ALIAS late wait on {self.name}: want {want} at {self.phase}")
        return passes


def run(NC, do_n, store_states, seed, stages, decay_writer="issuing lane", slow=None):
    """slow: a role that gets its turn late."""
    rnd = random.Random(seed)
    NH2 = 2 * NC
    B = {}
    for s in range(stages):
        B[f"full{s}"], B[f"empty{s}"], B[f"scaled{s}"] = Bar(f"full{s}", 1), Bar(f"empty{s}", 1), Bar(f"scaled{s}", 4)
    for s in range(2):
        B[f"acc_full{s}"], B[f"acc_free{s}"] = Bar(f"acc_full{s}", 1), Bar(f"acc_free{s}", 8)
        B[f"nsum{s}"], B[f"nread{s}"] = Bar(f"nsum{s}", 8), Bar(f"nread{s}", 1)
        B[f"out_full{s}"], B[f"out_free{s}"] = Bar(f"out_full{s}", 8), Bar(f"out_free{s}", 1)
    loads, commits = [], []          # copies in flight (land in any order), MMA commits (fire in order)
    clocks = {}                      # per agent: what it knows of every agent's operations
    written = [None] * 8             # slot of the decay ring: (writer, its time, chunk)
    reads = [[] for _ in range(8)]   # (reader, its time) since the last write

    def tick(a):
        clocks[a][a] = clocks[a].get(a, 0) + 1
        return clocks[a][a]

    def arrive(a, name):
        tick(a)
        B[name].arrive(clocks[a])

    def write_decay(a, s):
        for r, t in reads[s & 7]:
            assert clocks[a].get(r, 0) >= t, f"decay of chunk {s - 8} overwritten before {r} is known to have read it"
        reads[s & 7].clear()
        written[s & 7] = (a, tick(a), s)

    def read_decay(a, s):
        w, t, chunk = written[s & 7]
        assert chunk == s, f"{a} reads the decay of chunk {chunk} for that of {s}"
        assert clocks[a].get(w, 0) >= t, f"{a} reads the decay of chunk {s}, whose write by {w} nothing orders before it"
        reads[s & 7].append((a, tick(a)))

    def producer():
        for h in range(NH2):
            st, s = h % stages, h >> 1
            if h % 2 == 0 and decay_writer != "issuing lane":
                write_decay("prod other lane", s)
            yield ("wait", f"empty{st}", h // stages - 1)
            if h % 2 == 0 and decay_writer == "issuing lane":
                write_decay("prod", s)
            tick("prod")
            loads.append((st, dict(clocks["prod"])))   # (the copy's completion; the arrival that expects it)
            yield ("step",)

    def mma():
        for h in range(NH2):
            st, s = h % stages, h >> 1
            buf = s & 1
            yield ("wait", f"scaled{st}", h // stages)
            if h % 2 == 0:
                yield ("wait", f"acc_free{buf}", (s >> 1) - 1)
            tick("mma")
            commits.append((f"empty{st}", dict(clocks["mma"])))
            if h % 2 == 1:
                commits.append((f"acc_full{buf}", dict(clocks["mma"])))

    def gating(w, group):
        for h in range(group, NH2, 2):
            st, s = h % stages, h >> 1
            nb = s & 1
            yield ("wait", f"full{st}", h // stages)
            arrive(w, f"scaled{st}")
            if do_n:
                yield ("step",)
                if s >= 2:
                    yield ("wait", f"nread{nb}", (s >> 1) - 1)
                arrive(w, f"nsum{nb}")

    def store_warp():
        for n in range(NC + 1):
            ob = n & 1
            yield ("wait", f"out_full{ob}", n >> 1)
            if n >= 1:
                arrive("store", f"out_free{ob ^ 1}")

    def n_warp():
        for s in range(NC):
            nb = s & 1
            yield ("wait", f"nsum{nb}", s >> 1)
            arrive("n", f"nread{nb}")
            yield ("step",)
            read_decay("n", s)

    def state_warp(w):
        n_out = 0

        def store_c():
            nonlocal n_out
            if store_states:
                ob = n_out & 1
                if n_out >= 2:
                    yield ("wait", f"out_free{ob}", (n_out >> 1) - 1)
                arrive(w, f"out_full{ob}")
            n_out += 1
        yield from store_c()
        for s in range(NC):
            buf = s & 1
            yield ("wait", f"acc_full{buf}", s >> 1)
            read_decay(w, s)
            arrive(w, f"acc_free{buf}")
            yield from store_c()

    agents = {"prod": producer(), "mma": mma()}
    for w in range(8):
        agents[f"gate{w}"] = gating(f"gate{w}", w >> 2)
        agents[f"state{w}"] = state_warp(f"state{w}")
    if store_states:
        agents["store"] = store_warp()
    if do_n:
        agents["n"] = n_warp()
    clocks.update({a: {} for a in [*agents, "prod other lane"]})
    blocked, alive = {}, dict.fromkeys(agents)    # (in a fixed order: a run depends on its seed alone)

    def acquire(a, bar, phase):
        if phase < 0:
            return
        for lane in (a, "prod other lane") if a == "prod" else (a,):
            join(clocks[lane], B[bar].released.get(phase, {}))

    while alive:
        choices = [("agent", a) for a in alive]
        if loads:
            choices.append(("load", None))
        if commits:
            choices.append(("commit", None))
        rnd.shuffle(choices)
        if slow is not None and rnd.random() < 0.95:
            choices.sort(key=lambda c: c[1] == slow)
        progressed = False
        for kind, a in choices:
            if kind == "load":
                st, clock = loads.pop(rnd.randrange(len(loads)))
                B[f"full{st}"].arrive(clock)
                progressed = True
                break
            if kind == "commit":
                bar, clock = commits.pop(0)
                B[bar].arrive(clock)
                progressed = True
                break
            if a in blocked:
                _, bn, ph = blocked[a]
                if not B[bn].test(ph):
                    continue
                del blocked[a]
                acquire(a, bn, ph)
            try:
                op = next(agents[a])
            except StopIteration:
                del alive[a]
                progressed = True
                break
            if op[0] == "wait":
                if B[op[1]].test(op[2]):
                    acquire(a, op[1], op[2])
                else:
                    blocked[a] = op
            progressed = True
            break
        if not progressed:
            raise AssertionError(f"DEADLOCK: {blocked}")


DEPTHS = ring_depths()


@pytest.mark.parametrize("NC", [1, 2, 3, 5, 8, 17, 40])
@pytest.mark.parametrize("do_n,store_states", [(True, True), (False, True), (False, False), (True, False)])
@pytest.mark.parametrize("stages", DEPTHS)
def test_recurrence_protocol_has_no_aliasing_deadlock_or_over_arrival(NC, do_n, store_states, stages):
    for seed in range(25):
        run(NC, do_n, store_states, seed, stages)


@pytest.mark.parametrize("slow", ["prod", "mma", "gate0", "gate5", "state0", "state7", "store", "n"])
@pytest.mark.parametrize("stages", DEPTHS)
def test_a_role_that_falls_behind_meets_no_barrier_two_phases_on(stages, slow):
    for seed in range(20):
        run(12, True, True, seed, stages, slow=slow)
        run(12, False, True, seed, stages, slow=slow)


@pytest.mark.parametrize("stages", [5, 7])
def test_odd_ring_would_alias(stages):
    """With an odd number of stages a gating group returns to a stage two phases later, and its wait passes on the load
    before the one it wants."""
    for seed in range(400):
        try:
            run(16, False, True, seed, stages)
        except AssertionError as e:
            assert "ALIAS early pass on full" in str(e)
            return
    raise AssertionError("no interleaving out of 400 showed the hazard")


def test_decay_written_by_another_lane_than_the_arriving_one_would_race():
    """The decay has to be written by the lane that arrives on the stage's barrier: nothing orders another lane's write
    before the readers."""
    with pytest.raises(AssertionError, match="nothing orders"):
        run(4, True, True, 0, DEPTHS[0], decay_writer="another lane")

"""Model of the barrier protocol of the intra-chunk backward (csrc/chunkwise_bw_sm100.cu), run on the CPU.

One CTA goes through many work items with all rings and barriers running on, and a wait sees only the parity of a phase: no
waiter may ever be two phases away from its barrier, early or late.  The order of waits, arrivals, copies and MMA commits
of each role is restated here and run under random interleavings (copies land in any order, commits fire in order), with
every wait checked against the true phase count, every barrier against over-arrival and the run against deadlock.  Kept
next to the kernel by hand; the depth of the operand ring is read from its source."""

import os
import random
import re

import pytest

SRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "mlstm_kernels_b200", "csrc", "chunkwise_bw_sm100.cu")


def ring_depth():
    with open(SRC) as f:
        return int(re.search(r"constexpr int NST = (\d+);", f.read()).group(1))


class Bar:
    def __init__(self, name, count):
        self.name, self.count, self.pending, self.phase = name, count, count, 0

    def arrive(self):
        self.pending -= 1
        assert self.pending >= 0, f"over-arrival on {self.name}"
        if self.pending == 0:
            self.phase += 1
            self.pending = self.count

    def test(self, want):
        passes, truth = (self.phase & 1) != (want & 1), self.phase > want
        if passes != truth and (passes or self.phase >= want + 2):
            raise AssertionError(f"ALIAS on {self.name}: want {want} at {self.phase}")
        return passes


def run(items, seed, slow=None, gated=2, sread=True):
    """items: (slices, tiles, has an E tile) of each.  slow: a role that gets its turn late.  gated: buffers of the gated
    tile, which are reused without a wait of their own; without sread a score is issued while the one before it may still
    be read: the run checks that nothing is overwritten under a reader."""
    rnd = random.Random(seed)
    stages = ring_depth()
    count = {"sfull": 1, "sread": 8}
    count.update({f"{n}{i}": c for i in range(2) for n, c in (("gready", 8), ("afull", 1), ("accfree", 8), ("scaled", 8), ("hfull", 1),
                                                              ("ready", 1), ("staged", 8))})
    count.update({f"{n}{s}": 1 for n in ("full", "empty") for s in range(stages)})
    B = {n: Bar(n, c) for n, c in count.items()}
    loads, commits = [], []
    reads = {"S": 0, "G0": 0, "G1": 0, "acc0": 0, "acc1": 0, "tile0": 0, "tile1": 0}   # who still reads what another role will overwrite
    tiles = [e for _, nsub, e in items for _ in range(nsub)]
    n_loads = sum(nd + nsub * (nd + 1) for nd, nsub, _ in items)

    def producer():
        for k in range(n_loads):
            if k >= stages:
                yield f"empty{k % stages}", k // stages - 1
            loads.append(f"full{k % stages}")

    def mma():
        k = t = 0

        def product_x(n, first):
            nonlocal k
            yield f"full{k % stages}", k // stages
            if first:
                yield f"gready{n & 1}", n >> 1
            yield f"scaled{(t - 1) & 1}", (t - 1) >> 1
            reads[f"G{n % gated}"] += 1
            commits.extend([("product", f"G{n % gated}"), f"empty{k % stages}", f"hfull{(t - 1) & 1}"])
            k += 1

        before = 0
        for n, (nd, nsub, _) in enumerate(items):
            if n > 0 and sread:
                yield "sread", n - 1
            for _ in range(nd):
                yield f"full{k % stages}", k // stages
                assert reads["S"] == 0, "score written while it is read"
                commits.append(f"empty{k % stages}")
                k += 1
            commits.append("sfull")
            for s in range(nsub):
                if s == 0 and t > 0:
                    yield from product_x(n - 1, before == 1)
                if t >= 2:
                    yield f"accfree{t & 1}", (t >> 1) - 1
                for _ in range(nd):
                    yield f"full{k % stages}", k // stages
                    assert reads[f"acc{t & 1}"] == 0, "product written while the accumulator is read"
                    commits.append(f"empty{k % stages}")
                    k += 1
                commits.append(f"afull{t & 1}")
                if s > 0:
                    yield from product_x(n, s == 1)
                t += 1
            before = nsub
        yield from product_x(len(items) - 1, before == 1)

    def tile_warp():
        def fill(t):
            if t < len(tiles):
                assert reads[f"tile{t & 1}"] == 0, "E loaded over a tile that is being stored"
                if tiles[t]:
                    loads.append(f"ready{t & 1}")
                else:
                    B[f"ready{t & 1}"].arrive()
        fill(0)
        fill(1)
        for t in range(len(tiles)):
            yield f"staged{t & 1}", t >> 1
            reads[f"tile{t & 1}"] += 1
            yield None, None                       # the store reads its buffer
            reads[f"tile{t & 1}"] -= 1
            fill(t + 2)

    def gating(_):
        t = 0
        for n, (_, nsub, _) in enumerate(items):
            yield "sfull", n
            reads["S"] += 1
            yield None, None
            assert reads[f"G{n % gated}"] == 0, "gated over a tile that a product reads"
            reads["S"] -= 1
            B["sread"].arrive()
            B[f"gready{n & 1}"].arrive()
            for _ in range(nsub):
                yield f"afull{t & 1}", t >> 1
                B[f"scaled{t & 1}"].arrive()
                t += 1

    def output(_):
        for t in range(len(tiles)):
            yield f"ready{t & 1}", t >> 1
            yield f"hfull{t & 1}", t >> 1
            reads[f"acc{t & 1}"] += 1
            yield None, None
            reads[f"acc{t & 1}"] -= 1
            B[f"accfree{t & 1}"].arrive()
            assert reads[f"tile{t & 1}"] == 0, "staging under a store"
            B[f"staged{t & 1}"].arrive()

    agents = {"producer": producer(), "mma": mma(), "tile": tile_warp()}
    agents.update({f"gating{w}": gating(w) for w in range(8)})
    agents.update({f"output{w}": output(w) for w in range(8)})
    blocked = {}
    while agents:
        choices = list(agents) + (["land"] if loads else []) + (["commit"] if commits else [])
        rnd.shuffle(choices)
        if slow is not None and rnd.random() < 0.95:
            choices.sort(key=lambda c: c == slow)
        for c in choices:
            if c == "land":
                B[loads.pop(rnd.randrange(len(loads)))].arrive()
                break
            if c == "commit":
                what = commits.pop(0)
                if isinstance(what, tuple):
                    reads[what[1]] -= 1
                else:
                    B[what].arrive()
                break
            if c in blocked and not B[blocked[c][0]].test(blocked[c][1]):
                continue
            blocked.pop(c, None)
            try:
                bar, phase = next(agents[c])
            except StopIteration:
                del agents[c]
                break
            if bar is not None and not B[bar].test(phase):
                blocked[c] = (bar, phase)
            break
        else:
            raise AssertionError(f"DEADLOCK {blocked}")
    assert not loads, "copies in flight when the CTA retires"


SHAPES = [   # slices, tiles, E: of a chunk's three modes
    [(4, 2, False), (4, 2, True), (4, 2, True)], [(2, 2, False), (4, 1, True), (4, 1, True)], [(1, 1, False), (1, 1, True), (1, 1, True)],
    [(4, 4, False), (8, 2, True), (8, 2, True)], [(1, 3, False), (5, 1, True), (5, 1, True)], [(8, 4, False), (16, 4, True), (16, 4, True)]]


@pytest.mark.parametrize("shape", SHAPES)
@pytest.mark.parametrize("n", [1, 2, 3, 7])
def test_rings_run_on_across_items(shape, n):
    for seed in range(20):
        run((shape * 4)[seed % 3:seed % 3 + n], seed)


@pytest.mark.parametrize("shape", SHAPES)
@pytest.mark.parametrize("slow", ["producer", "mma", "tile", "gating0", "output7", "land", "commit"])
def test_a_role_that_falls_behind_meets_no_barrier_two_phases_on(shape, slow):
    for seed in range(8):
        run((shape * 3)[seed % 3:seed % 3 + 6], seed, slow=slow)


@pytest.mark.parametrize("kw,message", [({"gated": 1}, "gated over a tile"), ({"sread": False}, "ALIAS on sfull|score written while")])
def test_what_the_second_gated_tile_and_the_wait_before_a_score_are_for(kw, message):
    with pytest.raises(AssertionError, match=message):
        for seed in range(2000):
            run([(1, 1, False)] * 7, seed, slow=("commit", "gating0")[seed & 1], **kw)

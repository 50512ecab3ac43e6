"""How the intra-chunk backward's work items are dealt out to its CTAs (csrc/par_bw_items.h, plain integers): the header itself,
compiled with the host compiler, over launches of every size."""

import os
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "mlstm_kernels_b200", "csrc")
SMS = 148
PROGRAM = r"""
#include <cstdio>
#include "par_bw_items.h"
using namespace mlstm;
int main() {
  int units, bh0, NC, DHQK, DHHV, sms;
  while (scanf("%d %d %d %d %d %d", &units, &bh0, &NC, &DHQK, &DHHV, &sms) == 6) {
    const BwItems w = bw_plan(units, bh0, NC, DHQK, DHHV, sms);
    printf("launch %u %u\n", w.stride, bw_grid(w));
    for (unsigned b = 0; b < bw_grid(w); ++b)
      for (BwRun it(w, b, bw_grid(w)); it.left > 0; it.next(w))
        printf("%u %d %d %d %d %d %d\n", b, it.bh, it.ck, it.mode(w), it.tile0(w), it.tiles(w), it.slices(w));
  }
}
"""
SIZES = [(units, 3, NC, DHQK, DHHV) for DHQK, DHHV in [(256, 512), (128, 256), (192, 384), (256, 256), (96, 192), (8, 24), (256, 1024), (128, 640),
                                                       (512, 1024), (264, 136)]
         for units, NC in [(1, 1), (8, 3), (8, 4), (8, 5), (8, 6), (16, 3), (7, 7), (8, 9), (8, 12), (3, 33), (8, 25), (8, 111), (149, 1), (16, 64)]]


@pytest.fixture(scope="module")
def launches(tmp_path_factory):
    d = tmp_path_factory.mktemp("items")
    with open(d / "items.cpp", "w") as f:
        f.write(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-O1", "-Wall", "-Werror", f"-I{CSRC}", str(d / "items.cpp"), "-o", str(d / "items")], check=True)
    out = subprocess.run([str(d / "items")], input="".join(f"{' '.join(map(str, s))} {SMS}\n" for s in SIZES), capture_output=True, text=True,
                         check=True).stdout
    runs = []
    for line in out.splitlines():
        if line.startswith("launch"):
            runs.append((int(line.split()[1]), int(line.split()[2]), []))
        else:
            runs[-1][2].append(tuple(map(int, line.split())))
    assert len(runs) == len(SIZES)
    return dict(zip(SIZES, runs))


def ring_stages(tiles, slices):
    """Operands of an item: the score's slices, and of every output tile the inter-chunk product's and X."""
    return slices + tiles * (slices + 1)


@pytest.mark.parametrize("size", SIZES)
def test_every_tile_once_and_bounded_runs(launches, size):
    units, bh0, NC, DHQK, DHHV = size
    stride, grid, items = launches[size]
    assert 1 <= stride <= SMS and grid % stride == 0
    done, taken = set(), {}
    for b, bh, ck, mode, tile0, tiles, slices in items:
        assert slices == -(-(DHQK if mode == 0 else DHHV) // 64) and 1 <= tiles <= 4
        taken[b] = taken.get(b, 0) + 1
        for t in range(tile0, tile0 + tiles):
            assert (bh, ck, mode, t) not in done
            done.add((bh, ck, mode, t))
    assert done == {(bh, ck, mode, t) for bh in range(bh0, bh0 + units) for ck in range(NC) for mode in range(3)
                    for t in range(-(-(DHHV if mode == 0 else DHQK) // 128))}
    assert max(taken.values()) <= 24


@pytest.mark.parametrize("size", SIZES)
def test_no_cta_has_more_to_do_than_whole_items_in_turn_would_give(launches, size):
    """Splitting items never leaves the busiest CTA of a small launch more than the whole ones, dealt out one by one, would; in a
    large one every CTA meets all kinds of items, so that none is further above the mean than two items."""
    units, _, NC, DHQK, DHHV = size
    stride, grid, items = launches[size]
    load = [0] * grid
    for b, _, _, _, _, tiles, slices in items:
        load[b] += ring_stages(tiles, slices)
    T = {0: -(-DHHV // 128), 1: -(-DHQK // 128), 2: -(-DHQK // 128)}
    whole = [ring_stages(min(4, T[mode] - t), -(-(DHQK if mode == 0 else DHHV) // 64)) for _ in range(units * NC) for mode in range(3)
             for t in range(0, T[mode], 4)]
    if len(whole) < 2 * SMS:
        assert max(load) <= max(sum(whole[b::SMS]) for b in range(SMS))
    if grid == stride:
        assert max(load) <= sum(load) / SMS + 2 * max(whole)

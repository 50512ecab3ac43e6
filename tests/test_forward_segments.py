"""The rule that cuts a long sequence of few (batch, head) units into segments (csrc/segments.h, plain numbers), compiled with
the host compiler: against sizes that were timed in segments and in one piece on a GPU of 148 SMs."""

import os
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "mlstm_kernels_b200", "csrc")
PROGRAM = r"""
#include <cstdio>
#include "segments.h"
int main() {
  int units, S, DHQK, DHHV;
  while (scanf("%d %d %d %d", &units, &S, &DHQK, &DHHV) == 4) {
    const long c = (long)((DHHV + 127) / 128) * ((DHQK + 127) / 128) * units;
    printf("%d\n", mlstm::forward_segments(c, (S + 127) / 128, units, DHQK, DHHV, 148));
  }
}
"""
# units, DHQK, DHHV: us per call at 65536, 131072 and 262144 tokens, in segments and in one piece (None: not timed, or not cut by the older rule)
FASTER_IN_SEGMENTS = [
    (8, 256, 512, (935, 1023), (1973, 2154), (3625, 4356)),
    (16, 256, 256, (1135, 1179), (2201, 2385), (4256, 4759)),
    (16, 64, 512, (1009, 1060), (2040, 2229), (3955, 4461)),
    (8, 64, 1024, (983, 1031), (1943, 2158), (3816, 4391)),
    (2, 512, 1024, (851, 898), (1693, 1844), (3305, 3711)),
    (4, 256, 1024, (950, 1062), (1843, 2073), (3430, 4234)),
    (4, 256, 512, (606, 714), (1140, 1398), (2185, 2780)),
    (16, 128, 256, (763, 873), (1466, 1733), (2823, 3713)),
    (32, 64, 128, (862, 937), (1647, 1827), (3196, 3605)),
    (24, 128, 256, None, None, (4106, 4813)),
    (6, 128, 1024, None, None, (3353, 4352)),
]
NOT_FASTER_IN_SEGMENTS = [
    (64, 64, 128, (1658, 1439), (3277, 2812), (6495, 5577)),
    (64, 64, 64, (1493, 1327), (2905, 2591), (5746, 5130)),
    (32, 128, 256, (1518, 1410), (3029, 2841), (6024, 5544)),
    (36, 128, 256, (1645, 1430), (3294, 2855), None),
    (16, 128, 512, (1339, 1286), (2613, 2559), (5148, 5093)),
    (32, 64, 256, (1195, 1153), (2422, 2439), (4786, 4825)),     # (both the same from 98304 tokens on)
    (8, 128, 1024, (1255, 1220), (2508, 2512), (4948, 4996)),
]


@pytest.fixture(scope="module")
def segments(tmp_path_factory):
    d = tmp_path_factory.mktemp("segments")
    with open(d / "segments.cpp", "w") as f:
        f.write(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-O1", "-Wall", "-Werror", f"-I{CSRC}", str(d / "segments.cpp"), "-o", str(d / "segments")], check=True)

    def ask(*sizes):
        text = "".join(f"{u} {S} {k} {v}\n" for u, S, k, v in sizes)
        return [int(x) for x in subprocess.run([str(d / "segments")], input=text, capture_output=True, text=True, check=True).stdout.split()]

    return ask


@pytest.mark.parametrize("cut,table", [(True, FASTER_IN_SEGMENTS), (False, NOT_FASTER_IN_SEGMENTS)])
def test_cut_where_segments_were_faster(segments, cut, table):
    sizes = [(units, S, DHQK, DHHV) for units, DHQK, DHHV, *times in table for S, t in zip((65536, 131072, 262144), times) if t is not None]
    for size, n in zip(sizes, segments(*sizes)):
        assert 1 <= n <= 16
        assert (n > 1) == cut, size


def test_one_piece_where_the_recurrence_has_more_than_half_of_the_sms_or_the_sequence_is_short(segments):
    sizes = [(u, S, 256, 512) for u in (1, 2, 4, 8, 9, 16, 128, 4096) for S in (1, 128, 500, 8192, 16384)]
    sizes += [(u, 131072, 256, 512) for u in (10, 16, 128)]
    assert set(segments(*sizes)) == {1}

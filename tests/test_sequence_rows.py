"""Which register form of the sequence kernel (csrc/step.cu, step_seq_rows) a DHQK takes: the rows that its token loop goes
through without a look at DHQK must exist, all rows must have a place, and above 128 no more than two rows beyond DHQK, or
tested in the loop, are left."""

import os
import re

import pytest

SRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "mlstm_kernels_b200", "csrc", "step.cu")


def forms():
    """(condition in front, rows, rows without a test, columns, CTAs per SM) in the order of the dispatch."""
    with open(SRC) as f:
        src = f.read()
    body = src[src.index("int step_seq_rows("):]
    body = body[:body.index("#undef SEQ_CASE")]
    body = body[body.index("if (narrow) {"):]
    out, conditions = [], []
    for m in re.finditer(r"if \(((?:[^()]|\((?:[^()]|\([^()]*\))*\))*)\) \{|(\})|SEQ_CASE\((\d+), (\d+), (\d+), (\d+)\)", body):
        if m[1] is not None:
            conditions.append(m[1])
        elif m[2] is not None:
            conditions.pop()
        else:
            out.append((tuple(conditions), *(int(x) for x in m.groups()[2:])))
    return out


@pytest.mark.parametrize("one_wave", [False, True])
@pytest.mark.parametrize("narrow", [False, True])
def test_rows_of_every_size(narrow, one_wave):
    table = forms()
    assert len(table) == 15
    for DHQK in range(1, 513):
        for conditions, rows, full, tv, ctas in table:
            value = {"narrow": narrow or DHQK > 128, "DHQK == 256": DHQK == 256, "DHQK == 512": DHQK == 512,
                     "(long)ceil_div(DHHV, 32) * B * NH <= sm_count()": one_wave}
            rg = 256 // (tv // 4)
            if all(value[c] for c in conditions) and -(-DHQK // rg) <= rows:
                break
        else:
            raise AssertionError(f"no form for {DHQK}")
        assert full * rg <= DHQK <= rows * rg
        if DHQK > 128:
            assert tv == 32 and (rows * rg == DHQK or rows - full <= 4 and rows * rg - DHQK < 4 * rg)
        assert ctas == (1 if DHQK > 256 and one_wave else 2)

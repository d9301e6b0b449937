"""bench.py's count of the work of phase A against the library's rules for it."""
import os
import re

import pytest

import bench

SRC = open(os.path.join(os.path.dirname(bench.__file__), "vkzg_b200", "csrc", "proof_kernels.cu")).read()


@pytest.mark.parametrize("blobs,points,threads", [(1, 96, 32), (9, 96, 32), (10, 24, 8), (37, 24, 8), (38, 10, 2),
                                                  (256, 10, 2)])
def test_tail_of_phase_a_lists(blobs, points, threads):
    assert bench.phase_a_tail(blobs, 148) == (points, threads)


def test_tail_rule_is_the_launchers():
    names = dict(re.findall(r"(kTreeTail\d*) = (\d+)", SRC))
    assert {k: int(v) for k, v in names.items()} == {"kTreeTail": 10, "kTreeTail8": 24, "kTreeTail32": 96}
    assert "return lists <= 8 * sms ? 32 : lists <= 32 * sms ? 8 : 2;" in SRC


def test_executed_products():
    """23 windows: lists of 1472 points; 736 + 368 + 184 + 92 pairs down to 92 points
    for few blobs, whose 32 chains make 60 mixed additions and 31 tree additions."""
    adds = 736 + 368 + 184 + 92
    assert bench.phase_a_executed_products_per_output(23, 6, 148) == 6 * adds + 11 * 60 + 16 * 31
    adds += 46 + 23 + 11  # 46, 23, 12 points
    assert bench.phase_a_executed_products_per_output(23, 37, 148) == 6 * (adds - 11) + 11 * 15 + 16 * 7
    adds += 6  # 6 points
    assert bench.phase_a_executed_products_per_output(23, 256, 148) == 6 * adds + 11 * 4 + 16
    assert (bench.phase_a_executed_imad_per_output(23, 256, 148) ==
            adds * (5 * bench.IMAD_FP_MUL_TM + bench.IMAD_FP_SQR_TM) +
            (7 * 4 + 11) * bench.IMAD_FP_MUL_KS + (4 * 4 + 5) * bench.IMAD_FP_SQR_KS)

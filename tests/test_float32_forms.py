"""The forms in which a float32 product of many rows runs, as the library itself chooses them, without a GPU."""
import pytest

from infurnace_b200.kernels.build import load_library
from test_kernels_gpu import LONGER, MANY_ROWS, MANY_ROWS_OF

F32, BF16 = 0, 1
ALL = {2 * rows + alone for rows in range(2, 9) for alone in (0, 1)} - {2 * 6 + 1}      # six rows per thread alone: never the quickest


def form(n, o, k, epilogue=0, vec=1, out=F32, sms=148):
    return load_library("core").ifb_linear_float32_form(n, o, k, epilogue, vec, out, sms)


def test_every_form_is_among_the_products_that_are_tested():
    reached = {form(n, o, k, e) for n in range(17, 700, 5) for o in range(64, 12000, 192) for k in (16, 256, 1024, 4096) for e in (0, 1)}
    tested = {form(n, o, k, e) for n, o, k in [(n, *of) for n in MANY_ROWS for of in MANY_ROWS_OF] + LONGER for e in (0, 1)}
    assert reached == tested == ALL
    assert {form(n, o, k, e, 0) for n, o, k in [(49, 2500, 1041), (41, 9600, 37)] for e in (0, 1)} == {16, 17}
    assert {form(n, o, k, e, 1, BF16) for n, o, k in [(49, 2500, 1040), (41, 9600, 36)] for e in (0, 1)} == {16, 17}


# Where eight rows per thread are the only choice, whether a CTA takes a tile alone is chosen for eight: 38 to 49 tiles for 74 pairs are one
# round of the pairs, whatever another number of rows would have done.
@pytest.mark.parametrize("n,tiles", [(41, 38), (48, 49), (336, 7)])
@pytest.mark.parametrize("vec,out", [(0, F32), (1, BF16), (0, BF16)])
def test_eight_rows_per_thread_are_judged_as_eight(n, tiles, vec, out):
    assert form(n, 64 * tiles, 1024, 0, vec, out) == 16
    assert form(n, 32 * tiles, 1024, 1, vec, out) == 16


def test_a_lone_cta_is_for_a_short_k():
    """Five tiles of rows times 40 of features: three rounds of 74 pairs against two of 148 CTAs, of which one takes 1.54 times as long at a k of
    512 and 1.8 at 4,096."""
    assert [form(300, 2500, k, 0, 1, BF16) for k in (256, 512, 1024, 2048, 4096)] == [17, 16, 16, 16, 16]
    assert [form(300, 2500, k) for k in (256, 4096)] == [15, 16]
    assert form(200, 2500, 4096, 0, 1, F32, 74) != form(200, 2500, 4096)              # by the SMs that there are

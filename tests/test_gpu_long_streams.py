"""Entropy-coded segments longer than 32-bit bit positions reach: what lies within reach decodes, the rest counts as cut off.
Before the limit was kept, the restart decoder addressed shared memory with wrapped positions; the case below must not
run on such a build."""
import numpy as np
import pytest

import datago_b200 as dg
import oracle
from gpu_common import assert_same, jpeg

pytestmark = pytest.mark.gpu

LONG = (1 << 29) + (1 << 22)


def _process(items):
    c = dg.Context(0, None)  # (not the other tests' context: its blocks would stay this large)
    try:
        return c.process(items)
    finally:
        c.close()


def test_an_early_end_of_image_counts_however_much_follows():
    good = jpeg(np.random.default_rng(601), 200, 120)
    (st, out, _), (st2, out2, _) = _process([good + b"\x11" * LONG, good])
    assert st == st2 == 0
    assert_same(out, oracle.jpeg_decode(good))
    assert_same(out2, oracle.jpeg_decode(good))


def test_segments_out_of_reach_count_as_cut_off():
    rng = np.random.default_rng(602)
    good = jpeg(rng, 320, 240, rst=1)  # 300 segments: three CTAs
    first = good.index(b"\xff\xd0")
    (st, out, _), (st2, out2, _) = _process([good[:first] + b"\x11" * LONG + good[first:], good])
    assert (st, out) == (3, None)
    assert st2 == 0
    assert_same(out2, oracle.jpeg_decode(good))
    # within reach, data between the end of a segment's last block and its marker is skipped
    (st, out, _), = _process([good[:first] + b"\x11" * 100000 + good[first:]])
    assert st == 0
    assert_same(out, oracle.jpeg_decode(good))

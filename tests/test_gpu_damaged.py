"""Slots of damaged images: what the stream holds, mid-gray behind it, whatever the context decoded before."""
import numpy as np
import pytest

import datago_b200 as dg
import oracle
from gpu_common import assert_same, jpeg

pytestmark = pytest.mark.gpu

W, H = 336, 272


def _entropy_start(data):
    sos = data.index(b"\xff\xda")
    return sos + 2 + int.from_bytes(data[sos + 2:sos + 4], "big")


def _without_restart_markers(data, from_byte):
    out, i = bytearray(data[:from_byte]), from_byte
    while i < len(data):
        if data[i] == 0xFF and 0xD0 <= data[i + 1] <= 0xD7:
            i += 2
            continue
        out.append(data[i])
        i += 1
    return bytes(out)


def _slots(items, junk):
    c = dg.Context(0, None)
    try:
        for x in junk:
            c.process([x] * 3)
        with c.batch(items, None, dg.BATCH_COLLATE) as b:
            b.upload()
            b.run()
            host = np.zeros(b.packed_bytes(), np.uint8)
            b.download_packed(host)
            b.sync()
            k, = b.buckets()
            assert k["items"] == list(range(len(items)))
            return [b.result(i).status for i in range(len(items))], host[k["packed_offset"]:k["packed_offset"] + k["nbytes"]].reshape(k["shape"])
    finally:
        c.close()


@pytest.mark.parametrize("rst", [0, 1, 40])
@pytest.mark.parametrize("sub", ["4:2:0", "4:2:2", "4:4:4", None])
def test_what_a_damaged_stream_does_not_hold_is_gray(sub, rst):
    rng = np.random.default_rng(501)
    good = jpeg(rng, W, H, sub or "4:2:0", 90, rst, gray=sub is None)
    want = oracle.jpeg_decode(good).reshape(H, W, -1)
    start, n = _entropy_start(good), len(good)
    cuts = [start + int(f * (n - start)) for f in (0.0, 0.02, 0.35, 0.8)]
    items = [good[:cut] for cut in cuts] + [good[:start] + b"\xff\xd9", good]
    if rst:
        items.insert(0, _without_restart_markers(good, cuts[2]))
    junk = [jpeg(np.random.default_rng(s), 640, 480, s2, 98, r, noise=60.0) for s, s2, r in ((1, "4:2:0", 0), (2, "4:4:4", 0), (3, "4:2:0", 2))]
    status, slots = _slots(items, junk)
    again, other = _slots(items, junk[::-1] + [jpeg(np.random.default_rng(9), 900, 700, "4:2:2", 95, 0, noise=30.0)])
    assert status == again and status[-1] == 0 and all(s in (3, 4, 7) for s in status[:-1])
    assert np.array_equal(slots, other)
    assert_same(slots[-1], want)
    mcu = 16 if sub == "4:2:0" else 8
    first = 1 if rst else 0
    for i, cut in enumerate(cuts):
        rows = [bool((slots[first + i][y] == want[y]).all()) for y in range(H)]
        whole = rows.index(False)  # rows that are there in full, then at most the MCU row the cut falls into (and the chroma filter's reach)
        gray = min(H, (whole // mcu + 2) * mcu + 1)
        assert (slots[first + i][gray:] == 128).all(), (i, whole)
        if i > 1:
            assert whole >= mcu
        elif i == 0:
            assert (slots[first] == 128).all()
    assert (slots[-2] == 128).all()
    if rst == 1:  # behind the first missing marker everything is gray but what is left of its segment
        assert (slots[0][-mcu:] == 128).all()

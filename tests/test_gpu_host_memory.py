"""Payloads in the library's page-locked blocks: what they hold, which block they lie in, and how long it stays in use."""
import gc

import numpy as np
import pytest

import datago_b200 as dg
import oracle
from gpu_common import assert_same, ctx, jpeg

pytestmark = pytest.mark.gpu

BLOCK = 8 << 20  # payloads share a block up to this size


def _block(a):
    while not hasattr(a, "_block"):
        a = a.base
    return a._block.value


def _lent(address, nbytes, tries):
    """Whether the pool lends the block at `address` to another caller: its idle blocks of that size come first."""
    taken = []
    while len(taken) < tries:
        taken.append(dg.host_block(nbytes))
        if taken[-1].ctypes.data == address:
            return True
    return False


@pytest.mark.parametrize("end", ["sync", "close"])
def test_a_block_is_not_lent_on_while_a_copy_into_it_may_be_queued(end):
    rng = np.random.default_rng(401)
    x = rng.integers(0, 256, (700, 900, 3), dtype=np.uint8)
    b = ctx().batch([x])
    b.upload()
    b.run()
    first = b.download()[0].ctypes.data  # (the result itself is dropped)
    second = b.download()
    gc.collect()
    assert not _lent(first, x.nbytes, 3)
    getattr(b, end)()
    assert _lent(first, x.nbytes, 60)
    assert np.array_equal(second[0], x)
    b.close()


@pytest.mark.parametrize("shape", [(40, 50, 3), (400, 500, 3)])  # copied, handed on as a view
def test_what_a_ticket_returns_is_the_callers_own(shape):
    rng = np.random.default_rng(403)
    x = rng.integers(0, 256, shape, dtype=np.uint8)
    with dg.Feeder(0, None, max_batch=4, max_wait_us=500) as f:
        for order in ("ffpp", "pfpf", "fpf"):
            t, other = f.submit(x), f.submit(x)
            r = f.wait(t)
            got = [f.fetch(t, r) if c == "f" else f.peek(t, r) for c in order]
            for c, a in zip(order, got):
                assert np.array_equal(a, x), order
                if c == "f":
                    a[:] = 0  # nobody else's pixels change
            for c, a in zip(order, got):
                assert np.array_equal(a, x) == (c == "p"), order
            kept = f.fetch(t, r)
            f.release(t)
            assert np.array_equal(f.fetch(other, f.wait(other)), x)
            f.release(other)
        landing = np.zeros(shape, np.uint8)  # a buffer given at submit is filled by wait, after a fetch as well
        t = f.submit(x, host_out=landing)
        while f.stats()["completed"] < f.stats()["submitted"]:
            pass
        r = dg.Result()
        r.nbytes, r.height, r.width, r.channels = x.nbytes, *shape
        f.fetch(t, r)[:] = 0
        f.wait(t)
        assert np.array_equal(landing, x)
        f.release(t)
    assert np.array_equal(kept, x)


@pytest.mark.parametrize("collate", [0, dg.BATCH_COLLATE])
def test_payloads_are_whole_and_share_small_blocks_only(collate):
    rng = np.random.default_rng(402)
    items, want = [], []
    for i, (w, h) in enumerate([(1300, 1200), (900, 700), (64, 48), (1300, 1200), (2000, 1700), (333, 555), (900, 700), (64, 48)]):
        if i % 2:
            items.append(rng.integers(0, 256, (h, w, 3), dtype=np.uint8))
            want.append(items[-1])
        else:
            items.append(jpeg(rng, w, h))
            want.append(oracle.jpeg_decode(items[-1]))
    items.insert(3, b"not an image")
    want.insert(3, None)
    with ctx().batch(items, None, collate) as b:
        b.upload()
        b.run()
        outs = b.download()
        assert b.counters()["d2h_bytes"] == sum(w.nbytes for w in want if w is not None)
        b.sync()
    per_block = {}
    for i, (out, w) in enumerate(zip(outs, want)):
        if w is None:
            assert out is None
            continue
        assert out.flags.writeable
        assert_same(out, w, str(i))
        per_block.setdefault(_block(out), []).append(out)
    for arrays in per_block.values():
        assert len(arrays) == 1 or sum(a.nbytes for a in arrays) <= BLOCK
    assert any(len(a) > 1 for a in per_block.values())
    kept, address = outs[4].copy(), outs[4].ctypes.data  # one payload outlives the others, unharmed by what follows
    keep = outs[4]
    del outs, out, arrays, per_block
    gc.collect()
    for st, out, _ in ctx().process(items[:3] * 4):
        assert st == 0
        out[:] = 0
    assert keep.ctypes.data == address and np.array_equal(keep, kept)

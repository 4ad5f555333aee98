"""Who keeps host memory alive, and for how long, without a GPU: the Python side runs on a stand-in for the library that
counts references to page-locked blocks."""
import ctypes as C
import gc

import numpy as np
import pytest

import datago_b200 as dg


class FakeLibrary:
    """Batches of one 4 x 4 payload whose copies are queued and run by dg_batch_sync / dg_batch_destroy; blocks with counts."""

    def __init__(self):
        self.blocks = {}   # address -> [buffer, references]
        self.queued, self.held, self.scarce = [], [], False

    def in_use(self):
        return {a for a, (_, refs) in self.blocks.items() if refs}

    def dg_host_alloc(self, nbytes, out):
        buf = (C.c_uint8 * nbytes)()
        self.blocks[C.addressof(buf)] = [buf, 1]
        out._obj.value = C.addressof(buf)
        return 0

    def dg_host_release(self, block):
        self.blocks[getattr(block, "value", block)][1] -= 1

    def dg_batch_create(self, ctx, items, n, flags, out):
        out._obj.value = 1
        return 0

    def dg_batch_packed_bytes(self, b):
        return 48

    def dg_batch_results(self, b, out):
        out[0].status, out[0].width, out[0].height, out[0].channels, out[0].nbytes = 0, 4, 4, 3, 48
        return 0

    def dg_batch_download_packed(self, b, dst, capacity):
        self.queued.append(dst)
        return 0

    def dg_batch_download_views(self, b, host, blocks):
        if self.scarce:
            return dg.E_TOO_LARGE
        p = C.c_void_p()
        self.dg_host_alloc(48, C.byref(p))
        self.blocks[p.value][1] += 1  # the batch's own reference, until the copy has run
        self.held.append(p.value)
        host[0] = blocks[0] = p.value
        self.queued.append(p.value)
        return 0

    def dg_batch_download(self, b, ptrs):
        self.queued.append(ptrs[0])
        return 0

    def dg_batch_sync(self, b):
        self.queued.clear()
        for p in self.held:
            self.dg_host_release(p)
        self.held.clear()
        return 0

    def dg_batch_destroy(self, b):
        self.dg_batch_sync(b)


@pytest.fixture
def fake(monkeypatch):
    lib = FakeLibrary()
    monkeypatch.setattr(dg, "_lib", lib)
    yield lib
    gc.collect()


class _Ctx:
    _h = C.c_void_p(1)
    image_config = None


@pytest.mark.parametrize("end", ["sync", "close"])
def test_a_block_stays_in_use_while_a_copy_into_it_is_queued(fake, end):
    b = dg.Batch(_Ctx(), [np.zeros((4, 4, 3), np.uint8)])
    first = b.download()[0].ctypes.data  # (the result itself is dropped)
    second = b.download()
    gc.collect()
    assert first in fake.queued and first in fake.in_use()
    getattr(b, end)()
    gc.collect()
    assert fake.in_use() == {second[0].ctypes.data}
    del second
    b.close()
    gc.collect()
    assert not fake.in_use()


def test_a_landing_buffer_stays_alive_while_a_copy_into_it_is_queued(fake):
    b = dg.Batch(_Ctx(), [np.zeros((4, 4, 3), np.uint8)])
    for _ in range(2):
        b.download_packed(dg.host_block(48))
    gc.collect()
    assert len(fake.in_use()) == 2
    b.sync()
    gc.collect()
    assert not fake.in_use()
    b.close()


def test_payloads_arrive_in_ordinary_memory_while_blocks_are_scarce(fake):
    fake.scarce = True
    b = dg.Batch(_Ctx(), [np.zeros((4, 4, 3), np.uint8)])
    out, = b.download()
    assert fake.queued == [out.ctypes.data] and out.flags.owndata and out.shape == (4, 4, 3)
    b.close()

"""The batch scheduler's host side (csrc/api.cu), built against a stand-in for the CUDA runtime and the kernels: what is copied and
when, what a call returns, and what happens while the caller's stream is being captured."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

import datago_b200 as dg
from datago_b200 import synth

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "datago_b200", "csrc")
CFG = dict(crop_and_resize=True, default_image_size=512, downsampling_ratio=16, min_aspect_ratio=0.5, max_aspect_ratio=2.0)


@pytest.fixture(scope="module")
def library(tmp_path_factory):
    out = str(tmp_path_factory.mktemp("fake") / "libbatch.so")
    cuda = os.environ.get("CUDA_HOME", "/usr/local/cuda")
    sources = [os.path.join(ROOT, "tests", "fake_device.cpp")] + [os.path.join(CSRC, f) for f in ("api.cu", "feeder.cpp", "host_blocks.cpp", "host_logic.cpp", "jpeg_header.cpp")]
    subprocess.run(["g++", "-std=c++17", "-O1", "-shared", "-fPIC", "-pthread", "-Wl,-Bsymbolic", "-I", os.path.join(cuda, "include"), "-x", "c++", *sources, "-o", out], check=True)
    return out


@pytest.fixture
def fake(library, monkeypatch):
    monkeypatch.setattr(dg, "library_path", lambda: library)
    monkeypatch.setattr(dg, "_lib", None)
    monkeypatch.delenv("DATAGO_B200_REBUILD", raising=False)
    L = dg.lib()
    L.fake_capture.argtypes, L.fake_timeouts.argtypes = [C.c_void_p, C.c_int], [C.c_uint]
    L.fake_to_device.restype = L.fake_to_host.restype = C.c_uint64
    return L


def raw(shape):
    return np.zeros(shape, np.uint8)


@pytest.mark.parametrize("n", [1, 3])  # 0.4 MB of inputs: copied by upload; 3.2: queued by the time the batch exists
@pytest.mark.parametrize("upload_inside", [False, True])
def test_a_captured_stream_waits_for_no_event_from_outside(fake, n, upload_inside):
    c = dg.Context(0, CFG)
    with c.batch([raw((300 * n, 400 * n, 3))]) as b:
        if not upload_inside:
            b.upload()
        fake.fake_capture(c.stream, 1)
        before = fake.fake_to_device()
        if upload_inside:
            b.upload()
            assert fake.fake_to_device() - before == b.counters()["h2d_bytes"]  # a graph holds the copies
        b.run()
        fake.fake_capture(c.stream, 0)
        b.sync()
    c.close()


def test_intermediates_of_a_batch_in_two_waves(fake):
    # 168 MiB of coefficients: two waves, which keep what they made in a scratch block each
    data = synth.encode_jpeg(np.full((2048, 2048, 3), 90, np.uint8), 90, "4:4:4", 0)
    c = dg.Context(0, CFG)
    with c.batch([data] * 7) as b:
        spans = []
        for i in range(len(b)):
            coef, blocks, decoded = C.c_void_p(), C.c_uint64(), C.c_void_p()
            assert fake.dg_batch_debug(b._h, i, C.byref(coef), C.byref(blocks), C.byref(decoded)) == 0, i
            assert blocks.value == 3 * 256 * 256
            spans += [(coef.value, coef.value + blocks.value * 128), (decoded.value, decoded.value + 2048 * 2048 * 3)]
        spans.sort()
        assert all(a[1] <= b[0] for a, b in zip(spans, spans[1:]))
    c.close()


def test_a_resize_that_gave_up_waiting_is_reported(fake):
    c = dg.Context(0, CFG)
    x = raw((1104, 1408, 3))
    dst = np.zeros((2048, 2048, 3), np.uint8)

    def static():
        c.resize_device_static(x.ctypes.data, x.shape[1], x.shape[0], 3, dst.ctypes.data)

    static()
    fake.fake_timeouts(2)
    with pytest.raises(dg.DatagoB200Error, match="CTAs gave up"):
        static()
    with c.batch([x]) as b:
        b.upload(); b.run()
        with pytest.raises(dg.DatagoB200Error, match="CTAs gave up"):
            b.sync()
    fake.fake_timeouts(0)
    static()
    c.close()


def test_what_the_static_resize_needs_is_made_once_per_device(fake):
    # page-locking takes longer than the rest of making a context
    x, dst = raw((300, 400, 3)), np.zeros((2048, 2048, 3), np.uint8)
    made = []
    for _ in range(3):
        c = dg.Context(0, CFG)
        before = fake.fake_host_allocations()
        c.resize_device_static(x.ctypes.data, 400, 300, 3, dst.ctypes.data)
        made.append((before, fake.fake_host_allocations()))
        c.close()
    assert made[0][1] == made[1][0] == made[1][1] == made[2][0] == made[2][1]


@pytest.mark.parametrize("n", [1, 4, 5])
def test_counters_hold_what_was_copied(fake, n):
    c = dg.Context(0, CFG)
    with c.batch([raw((300, 400, 3))] * n) as b:
        before = fake.fake_to_device(), fake.fake_to_host()
        b.upload(); b.run()
        b.download_packed(np.empty(b.packed_bytes(), np.uint8))
        b.sync()
        k = b.counters()
        # (small batches: larger ones are copied before upload is called)
        assert (k["h2d_bytes"], k["d2h_bytes"]) == (fake.fake_to_device() - before[0], fake.fake_to_host() - before[1])
    c.close()


@pytest.mark.parametrize("n", [1, 3])
def test_decoder_counters_of_a_batch_that_has_not_run(fake, n):
    # zeros, as uploaded, also while the inputs of a larger batch are on their way
    c = dg.Context(0, CFG)
    with c.batch([raw((300 * n, 400 * n, 3))]) as b:
        b.upload()
        assert set(b.huffman_stats().values()) == {0}
        b.run()
        b.sync()
    c.close()

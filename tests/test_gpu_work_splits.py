"""Kernels whose split of the work depends on sizes, at the sizes where a split changes or a tile ends.  Everything is integer
arithmetic on 8-bit samples, so results equal the oracle's exactly."""
import io

import numpy as np
import pytest

import datago_b200 as dg
import oracle
from datago_b200 import synth
from gpu_common import assert_same, ctx, jpeg

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("w", [3, 5, 6, 7, 8, 9, 15, 16, 17, 31, 33, 255, 256, 257, 263, 264])
def test_horizontal_chroma_filter_at_the_edges(w):
    # 4:2:2: eight pixels per thread; the last chroma column is replicated, also inside a word
    rng = np.random.default_rng(300 + w)
    datas = [synth.encode_jpeg(rng.integers(0, 256, (h, w, 3), dtype=np.uint8), 92, "4:2:2", 0) for h in (1, 9, 40)]
    for data, (st, out, _) in zip(datas, ctx().process(datas)):
        assert st == 0
        assert_same(out, oracle.jpeg_decode(data), str(w))


@pytest.mark.parametrize("shape", [(1, 1), (1, 3, 3), (5, 3, 3), (7, 11), (37, 41, 3), (64, 64, 4), (127, 129, 3)])
def test_raw_pixels_handed_through_at_every_alignment(shape):
    # collated payloads lie back to back, so those of an odd size start at every byte alignment
    rng = np.random.default_rng(310)
    items = [rng.integers(0, 256, shape, dtype=np.uint8) for _ in range(20)]
    with ctx().batch(items, None, dg.BATCH_COLLATE) as b:
        b.upload(); b.run()
        host = np.empty(max(1, b.packed_bytes()), np.uint8)
        b.download_packed(host); b.sync()
        k, = b.buckets()
        got = host[k["packed_offset"]:k["packed_offset"] + k["nbytes"]].reshape(len(items), -1)
        for i, x in enumerate(items):
            assert np.array_equal(got[i], x.reshape(-1)), i


def test_integral_crop_of_a_pitched_source():
    # an aspect ratio between two buckets at the bucket's own scale: rows of the source are cut, nothing is filtered
    cfg = dict(crop_and_resize=True, default_image_size=224, downsampling_ratio=16, min_aspect_ratio=0.5, max_aspect_ratio=2.0)
    rng = np.random.default_rng(311)
    base = ctx(cfg).plan_geometry(224, 224, 3)
    for dw in (2, 6, 8):
        x = rng.integers(0, 256, (base.target_h, base.target_w + dw, 3), dtype=np.uint8)
        (st, out, _), = ctx(cfg).process([x])
        want, _ = oracle.crop_and_resize(cfg, x)
        assert st == 0
        assert_same(out, want, str(dw))


def _noisy(rng, w, h, sub, q, optimize=False):
    b = io.BytesIO()
    from PIL import Image, ImageFile
    ImageFile.MAXBLOCK = 1 << 24  # the encoder's buffer: it cannot suspend while it optimises its tables
    a = rng.integers(0, 256, (h, w, 3), dtype=np.uint8)
    a[: h // 3] //= 8  # a quieter part: other code lengths, more blocks per cell
    if sub is None:
        Image.fromarray(a[:, :, 0]).save(b, "JPEG", quality=q, optimize=optimize)
    else:
        Image.fromarray(a).save(b, "JPEG", quality=q, subsampling=sub, optimize=optimize)
    return b.getvalue()


@pytest.mark.parametrize("copies", [1, 6, 30, 130])
def test_entropy_cells_and_spans(copies):
    # one file per sampling, with the standard and with its own code tables; more of them pass through short cells, long
    # cells, spans of cells and the smaller linking CTAs
    rng = np.random.default_rng(320)
    distinct = [_noisy(rng, w, h, sub, q, opt) for (w, h, sub, q, opt) in
                [(700, 500, "4:2:0", 95, False), (640, 640, "4:2:0", 75, True), (500, 301, "4:4:4", 98, True), (400, 333, "4:2:2", 90, False),
                 (611, 400, None, 97, True), (33, 17, "4:2:0", 90, False)]]
    distinct.append(jpeg(rng, 512, 480, q=40, noise=0.0))  # many blocks per cell
    want = [oracle.jpeg_decode(d) for d in distinct]
    with ctx().batch(distinct * copies) as b:
        b.upload(); b.run()
        outs = b.download(); b.sync()
        for i, out in enumerate(outs):
            assert b.result(i).status == 0, i
            assert_same(out, want[i % len(distinct)], str(i))


@pytest.mark.parametrize("copies", [1, 30])
def test_restart_segments_per_cta(copies):
    # 3 106 segments of one MCU, or 93 180: CTAs of 128 threads, or of 224
    rng = np.random.default_rng(322)
    distinct = [jpeg(rng, w, h, q=92, rst=1) for w, h in [(640, 480), (1201, 400), (17, 33)]]
    want = [oracle.jpeg_decode(d) for d in distinct]
    with ctx().batch(distinct * copies) as b:
        b.upload(); b.run()
        outs = b.download(); b.sync()
        for i, out in enumerate(outs):
            assert b.result(i).status == 0, i
            assert_same(out, want[i % len(distinct)], str(i))


def test_decoder_counters():
    # cells of 512 bits with this little work: each is decoded by one candidate at least, by one per block of the MCU at most,
    # and once for the values; where no candidate was right once more or oftener
    rng = np.random.default_rng(321)
    data = _noisy(rng, 600, 400, "4:2:0", 90)
    stream = data[data.index(b"\xff\xda") + 14:-2].replace(b"\xff\x00", b"\xff")
    cells = (len(stream) * 8 + 511) // 512
    for copies in (1, 3):
        with ctx().batch([data] * copies) as b:
            b.upload(); b.run(); b.sync()
            st = b.huffman_stats()
        assert st["chunks"] == copies * cells
        assert copies <= st["rounds"] <= copies * 200
        assert 2 * copies * (cells - 2) <= st["subsequence_decodes"] <= 8 * copies * cells


@pytest.mark.parametrize("h", [1, 40, 700, 2300])
def test_resize_pass_cuts(h):
    # one image (CTAs of two chunks) and forty (longer ones), as tall and as flat as a pass gets
    cfg = dict(crop_and_resize=True, default_image_size=512, downsampling_ratio=16, min_aspect_ratio=0.5, max_aspect_ratio=2.0)
    rng = np.random.default_rng(330 + h)
    x = rng.integers(0, 256, (h, 600, 3), dtype=np.uint8)
    want, _ = oracle.crop_and_resize(cfg, x)
    for n in (1, 40):
        for st, out, _ in ctx(cfg).process([x] * n):
            assert st == 0
            assert_same(out, want, str((h, n)))


@pytest.mark.parametrize("sub", ["4:2:0", "4:4:4"])
def test_colour_rows_at_every_alignment(sub):
    # rows of odd-sized images start at any byte; tiles of 256 pixels end at, before and behind the right edge
    rng = np.random.default_rng(340)
    datas = [synth.encode_jpeg(rng.integers(0, 256, (21, w, 3), dtype=np.uint8), 90, sub, 0)
             for w in list(range(5, 26)) + list(range(249, 273)) + [511, 513, 519]]
    for data, (st, out, _) in zip(datas, ctx().process(datas)):
        assert st == 0
        assert_same(out, oracle.jpeg_decode(data), str(out.shape))


@pytest.mark.parametrize("n", [1, 3, 40])
def test_inputs_copied_while_they_are_staged(n, monkeypatch):
    # about 0.4 to 16 MB of files and re-pitched raw pixels in one wave and in many: below 2 MB the upload copies, above it
    # the pieces are queued as they are staged.  A batch may be dropped before its upload, uploaded again, and run again.
    cfg = dict(crop_and_resize=True, default_image_size=224, downsampling_ratio=16, min_aspect_ratio=0.5, max_aspect_ratio=2.0)
    rng = np.random.default_rng(350)
    files = [jpeg(rng, w, h, q=95, noise=8.0) for w, h in [(640, 480), (333, 222)]]
    raw = rng.integers(0, 256, (301, 401, 3), dtype=np.uint8)
    want = [oracle.crop_and_resize(cfg, oracle.jpeg_decode(f))[0] for f in files] + [oracle.crop_and_resize(cfg, raw)[0]]
    items = (files + [raw]) * n
    monkeypatch.setenv("DATAGO_B200_WAVE_MB", "16")
    c = dg.Context(0, cfg)
    try:
        c.batch(items).close()
        with c.batch(items) as b, c.batch(items[::-1]) as other:
            b.upload(); other.upload(); b.run(); other.run()
            outs, others = b.download(), other.download()
            b.sync(); other.sync()
            for i in range(len(items)):
                assert_same(outs[i], want[i % 3], str(i))
                assert_same(others[i], want[2 - i % 3], str(i))
            b.upload(); b.run(); b.run()
            outs = b.download(); b.sync()
            for i in range(len(items)):
                assert_same(outs[i], want[i % 3], str(i))
    finally:
        c.close()


@pytest.mark.parametrize("n", [1, 40])
@pytest.mark.parametrize("upload_inside", [False, True])
def test_calls_recorded_into_a_graph(n, upload_inside, monkeypatch):
    # the caller's stream is being captured when a batch is run, or uploaded and run: also a batch whose inputs are still on
    # their way, on a stream that is not captured
    import torch
    rng = np.random.default_rng(351)
    items = [jpeg(rng, w, h, q=95, rst=rst, noise=8.0) for w, h, rst in [(640, 480, 0), (333, 222, 4), (480, 640, 0)]] * n
    want = [oracle.jpeg_decode(d) for d in items[:3]]
    monkeypatch.setenv("DATAGO_B200_WAVE_MB", "16")
    stream = torch.cuda.Stream()
    c = dg.Context(0, None, stream=stream.cuda_stream)
    try:
        with c.batch(items) as b:
            if not upload_inside:
                b.upload()
            graph = torch.cuda.CUDAGraph()
            with torch.cuda.graph(graph, stream=stream, capture_error_mode="thread_local"):
                if upload_inside:
                    b.upload()
                b.run()
            with torch.cuda.stream(stream):
                graph.replay()
                graph.replay()
            outs = b.download(); b.sync()
            for i, out in enumerate(outs):
                assert b.result(i).status == 0, i
                assert_same(out, want[i % 3], str(i))
            del graph
    finally:
        c.close()


def test_intermediates_of_a_batch_in_two_waves():
    # 168 MiB of coefficients: two waves
    cfg = dict(crop_and_resize=True, default_image_size=512, downsampling_ratio=16, min_aspect_ratio=0.5, max_aspect_ratio=2.0)
    rng = np.random.default_rng(352)
    datas = [jpeg(rng, 2048, 2048, "4:4:4", noise=2.0)] * 4 + [jpeg(rng, 2041, 2047, "4:4:4", noise=2.0)] * 3
    with ctx(cfg).batch(datas) as b:
        b.upload(); b.run(); b.sync()
        for i in (0, 6):
            assert_same(b.debug_decoded(i), oracle.jpeg_decode(datas[i]), str(i))

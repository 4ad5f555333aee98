"""What a user of datago_b200 has it do, as measurable cases.

A case is one call pattern on one kind of data:

  process   Context.process on a list of samples: host bytes in, host arrays out, in one call
  host      a batch with one packed download into page-locked memory (a loader that hands pixels to host code)
  device    a collated batch whose payloads stay on the GPU (a training loop that consumes device tensors)
  feeder    single samples submitted to the Feeder, waited for and fetched (per-sample workers)
  client    one epoch of DatagoClient over a directory of files
  resident  Batch.run on an uploaded batch: the kernels alone, inputs and outputs in device memory
  static    Context.resize_device_static on an image the caller holds in device memory

Image sizes are a function of the case, pixel content of the seed.  Sizes, qualities, noise levels, restart intervals and
image_config values are those of datago_b200/synth.py and the tests.  All outputs are 8-bit pixels and therefore exact.
"""
import io
import json
import math
import os
import random
import shutil
import tempfile
from concurrent.futures import ThreadPoolExecutor

import numpy as np
import torch
from PIL import Image

import datago_b200 as dg
from datago_b200.client import DatagoClient

MAX_OUTPUTS = 48  # payloads handed back one by one; larger batches come back bucket by bucket


def listed():
    return [
        # one small file, decoded: an interactive request, or the first sample of a job; all latency
        dict(name="process_one_thumbnail", path="process", data="jpeg420", n=1, lo=256, hi=256, step=8, quality=90, noise=8.0, rst=0, size=0),
        # one photo of a few megapixels decoded and put into its bucket: what datago does per sample
        dict(name="process_one_photo", path="process", data="jpeg420", n=1, lo=1200, hi=1800, step=1, quality=90, noise=4.0, rst=0, size=1024),
        # a handful of web images of every kind (samplings, gray, RGBA and masks as raw pixels), odd sizes, converted to RGB
        dict(name="process_mixed", path="process", data="mixed", n=32, lo=300, hi=640, step=1, quality=85, noise=4.0, rst=0, size=512),
        # per-sample workers through the submit / wait front end
        dict(name="feeder_samples", path="feeder", data="jpeg420", n=48, lo=512, hi=1024, step=16, quality=85, noise=4.0, rst=0, size=512),
        # a training loop that keeps the payloads on the GPU: the local-file set, decoded and bucketed
        dict(name="device_buckets", path="device", data="jpeg420", n=192, lo=256, hi=2048, step=8, quality=90, noise=8.0, rst=0, size=1024),
        # a loader that wants full-size host pixels of odd-sized files
        dict(name="host_decode", path="host", data="jpeg420", n=96, lo=375, hi=1201, step=1, quality=85, noise=2.0, rst=0, size=0),
        # one epoch of the client over a directory, payloads bucketed, samples taken one by one
        dict(name="client_epoch", path="client", data="jpeg420", n=48, lo=512, hi=1536, step=16, quality=85, noise=4.0, rst=0, size=512),
        # the decode-throughput set: half of the files with a restart interval of four MCUs
        dict(name="resident_decode", path="resident", data="jpeg420", n=1024, lo=512, hi=1536, step=16, quality=85, noise=0.0, rst=4, size=0),
        # the local-file set again, kernels alone: entropy-heavy files, decode + bucket
        dict(name="resident_buckets", path="resident", data="jpeg420", n=256, lo=256, hi=2048, step=8, quality=90, noise=8.0, rst=0, size=1024),
        # raw pixels into small buckets: the resize kernels alone
        dict(name="resident_resize", path="resident", data="raw", n=48, lo=512, hi=4096, step=1, quality=0, noise=0.0, rst=0, size=512),
        # large 4:4:4 images, each with a same-size mask that goes into the image's bucket
        dict(name="resident_pairs", path="resident", data="pairs444", n=8, lo=1024, hi=4096, step=1, quality=90, noise=4.0, rst=0, size=2048),
        # one device-resident image, no allocation: latency of the resize chain
        dict(name="static_resize", path="static", data="raw", n=1, lo=900, hi=1600, step=1, quality=0, noise=0.0, rst=0, size=512),
    ]


RATIO = {512: 16, 1024: 32, 2048: 64}


def draw(rng):
    def log_int(a, b):
        return int(round(math.exp(rng.uniform(math.log(a), math.log(b)))))

    path = rng.choice(["process", "process", "host", "device", "feeder", "client", "resident", "resident", "resident", "static"])
    data = {"static": "raw", "client": "jpeg420", "feeder": rng.choice(["jpeg420", "mixed"])}.get(
        path, rng.choice(["jpeg420", "jpeg420", "jpeg422", "jpeg444", "gray", "mixed", "raw", "pairs444"]))
    if path == "host" and data in ("mixed", "pairs444"):
        data = "jpeg420"
    lo = log_int(160, 1024)
    hi = min(4096, log_int(lo, 4 * lo))
    if path == "static":
        hi = min(hi, 3000)
    size = rng.choice([512, 512, 1024, 2048]) if data in ("raw", "pairs444", "mixed") else rng.choice([0, 0, 512, 1024])
    if path in ("client", "static"):
        size = rng.choice([512, 1024])
    if data == "pairs444":
        size = rng.choice([1024, 2048])
    if path == "host":
        size = rng.choice([0, 512, 1024])
        data = "jpeg420" if data == "raw" and size == 0 else data
    # how many images: up to the pixels (decoded and produced) of the largest listed case of the same path
    per = (((lo + hi) / 2) ** 2 + (size or (lo + hi) / 2) ** 2) * (1.5 if data in ("jpeg444", "pairs444", "raw") else 1.0) / 1e6
    cap = {"process": 40.0, "feeder": 40.0, "client": 60.0, "host": 90.0, "device": 300.0, "resident": 350.0, "static": 1.0}[path]
    most = {"process": 48, "feeder": 48, "client": 48, "host": 128, "device": 256, "resident": 512, "static": 1}[path]
    n = 1 if path == "static" else log_int(1, max(1, min(most // 2 if data == "pairs444" else most, int(cap / per))))
    return dict(path=path, data=data, n=n, lo=lo, hi=hi, step=rng.choice([1, 1, 8, 16]), quality=rng.randint(75, 95), noise=round(rng.uniform(0.0, 8.0), 2),
                rst=rng.choice([0, 0, 4, 8]) if data.startswith("jpeg") else 0, size=size)


# ---- what a case holds ---------------------------------------------------------------------------------------------------
def image_config(case):
    if not case["size"]:
        return None
    return dict(crop_and_resize=True, default_image_size=case["size"], downsampling_ratio=RATIO[case["size"]], min_aspect_ratio=0.5, max_aspect_ratio=2.0)


def _shapes(case):
    """(width, height) per image.  Decode-only batches too large to come back one by one hold a few distinct shapes (the
    formats of a camera set), so that their payloads form dense buckets."""
    rng = random.Random(json.dumps({k: v for k, v in case.items() if k != "name"}, sort_keys=True))
    lo, hi, step = case["lo"], case["hi"], case["step"]

    def side():
        return max(8, rng.randint(lo, hi) // step * step)

    def shape():
        if case["data"] == "pairs444":  # the long side from the range, the aspect ratio from the bucket range and beyond
            long_side, ar = side(), rng.uniform(0.33, 3.0)
            return (long_side, max(8, round(long_side / ar))) if ar >= 1 else (max(8, round(long_side * ar)), long_side)
        return side(), side()

    n = case["n"]
    if case["size"] == 0 and n > MAX_OUTPUTS // 2:
        formats = [shape() for _ in range(24)]
        return [formats[rng.randrange(len(formats))] for _ in range(n)]
    return [shape() for _ in range(n)]


MIXED = ("jpeg420", "jpeg420", "jpeg422", "jpeg444", "gray", "rgba", "mask", "jpeg420")


def _kinds(case):
    if case["data"] == "mixed":
        return [MIXED[i % len(MIXED)] for i in range(case["n"])]
    if case["data"] == "pairs444":
        return ["jpeg444"] * case["n"]
    return [case["data"]] * case["n"]


CHANNELS = {"gray": 1, "mask": 1, "rgba": 4}


def _bits_per_pixel(kind, case):
    """Compressed size of the synthetic images, roughly: measured at 0 and 8 levels of noise, quality 75 to 95."""
    q = (case["quality"] - 75) / 20.0
    quiet, noisy = 0.3 + 0.35 * q, 1.1 + 2.4 * q * q
    return (quiet + (noisy - quiet) * (case["noise"] / 8.0) ** 1.5) * {"jpeg444": 1.5, "jpeg422": 1.15}.get(kind, 1.0)


def work(case):
    cfg = image_config(case)
    planner = dg.Context(dg.DG_DEVICE_NONE, cfg) if cfg else None
    total = 0.0
    for (w, h), kind in zip(_shapes(case), _kinds(case)):
        c = CHANNELS.get(kind, 3)
        c_out = 3 if case["data"] == "mixed" else c
        parts = [(kind, c, c_out)] + ([("mask", 1, 1)] if case["data"] == "pairs444" else [])
        for k, ci, co in parts:
            if cfg:
                p = planner.plan_geometry(w, h, ci)
                scale = max(p.target_w / w, p.target_h / h)
                used = min(w, math.ceil(p.target_w / scale)) * min(h, math.ceil(p.target_h / scale))
                out = p.target_w * p.target_h
            else:
                used = out = w * h
            total += (w * h * _bits_per_pixel(k, case) / 8.0 if k.startswith("jpeg") or k == "gray" else used * ci) + out * co
    return {"bytes": total, "flops": 0.0}


def tolerance(case):
    return "exact"


# ---- inputs ---------------------------------------------------------------------------------------------------------------
def _device():
    return "cuda" if torch.cuda.is_available() else "cpu"


def _picture(gen, rng, w, h, noise, channels=3):
    """Octaves of smooth noise, a gradient, hard-edged rectangles and pixel noise, as in datago_b200/synth.py, made on the GPU."""
    dev = gen.device
    acc = torch.zeros((1, channels, h, w), device=dev)
    amp, total, cells = 1.0, 0.0, 2
    while cells <= 256 and cells < max(w, h):
        gw, gh = max(2, round(cells * w / max(w, h)) + 1), max(2, round(cells * h / max(w, h)) + 1)
        grid = torch.rand((1, channels, gh, gw), device=dev, generator=gen)
        acc += amp * torch.nn.functional.interpolate(grid, size=(h, w), mode="bicubic", align_corners=True)
        total += amp
        amp *= 0.6
        cells *= 2
    img = acc[0] * (255.0 / max(total, 1.0))
    img += torch.linspace(0, rng.uniform(-60, 60), w, device=dev)[None, None, :] + torch.linspace(0, rng.uniform(-60, 60), h, device=dev)[None, :, None]
    for _ in range(rng.randint(4, 11)):
        x0, x1 = sorted(rng.randrange(w) for _ in range(2))
        y0, y1 = sorted(rng.randrange(h) for _ in range(2))
        img[:, y0:y1 + 1, x0:x1 + 1] = torch.tensor([rng.randrange(256) for _ in range(channels)], dtype=torch.float32, device=dev)[:, None, None]
    if noise > 0:
        img += torch.randn(img.shape, device=dev, generator=gen) * noise
    return img.clamp_(0, 255).to(torch.uint8).permute(1, 2, 0).contiguous()


def _mask(rng, w, h, dev):
    """A segmentation mask: filled ellipses of 255 on 0."""
    m = torch.zeros((h, w), dtype=torch.uint8, device=dev)
    yy, xx = torch.arange(h, device=dev)[:, None], torch.arange(w, device=dev)[None, :]
    for _ in range(rng.randint(4, 8)):
        cx, cy, rx, ry = rng.uniform(0, w), rng.uniform(0, h), rng.uniform(0.02, 0.25) * w + 1, rng.uniform(0.02, 0.25) * h + 1
        m[((xx - cx) / rx) ** 2 + ((yy - cy) / ry) ** 2 <= 1.0] = 255
    return m


def _encode(args):
    arr, kind, quality, rst = args
    kw = dict(quality=quality, optimize=False, progressive=False)
    if rst:
        kw["restart_marker_blocks"] = rst
    if kind != "gray":
        kw["subsampling"] = {"jpeg420": "4:2:0", "jpeg422": "4:2:2", "jpeg444": "4:4:4"}[kind]
    b = io.BytesIO()
    Image.fromarray(arr).save(b, "JPEG", **kw)
    return b.getvalue()


_ENCODERS = ThreadPoolExecutor(min(16, os.cpu_count() or 4))
DISTINCT = 192  # files of a larger batch repeat: encoding more of them would only make the preparation longer


def _samples(case, seed):
    """Inputs in order (bytes of a JPEG file, or an array of raw pixels) and the bucket key to force per input, or None."""
    rng = random.Random(seed)
    gen = torch.Generator(device=_device())
    gen.manual_seed(seed & 0x7FFFFFFF)
    out, jobs, made = [], [], {}
    for i, ((w, h), kind) in enumerate(zip(_shapes(case), _kinds(case))):
        rst = case["rst"] if i % 2 else 0
        again = made.get((w, h, kind, rst))
        if again and i >= DISTINCT:
            out.append(again[rng.randrange(len(again))])
            continue
        if kind == "raw":
            x = torch.randint(0, 256, (h, w, 3), dtype=torch.uint8, device=gen.device, generator=gen).cpu().numpy()
        elif kind == "mask":
            x = _mask(rng, w, h, gen.device).cpu().numpy()
        else:
            x = _picture(gen, rng, w, h, case["noise"], CHANNELS.get(kind, 3)).cpu().numpy()
            if kind != "rgba":
                x = _ENCODERS.submit(_encode, (x[:, :, 0] if kind == "gray" else x, kind, case["quality"], rst))
        made.setdefault((w, h, kind, rst), []).append(x)
        out.append(x)
        if case["data"] == "pairs444":
            out.append(_mask(rng, w, h, gen.device).cpu().numpy())
    return [x.result() if hasattr(x, "result") else x for x in out]


_KEPT = {}


def _kept(what, case):
    """Contexts and feeders: a program makes one and keeps it."""
    key = (what, case["size"])
    if key not in _KEPT:
        if what == "feeder":
            _KEPT[key] = dg.Feeder(0, image_config(case), max_batch=32, max_wait_us=500)
        else:
            _KEPT[key] = dg.Context(0, image_config(case))
    return _KEPT[key]


class State:
    """What the program has in hand."""

    def __init__(self, **kw):
        self.batch = self.outputs = None
        self.__dict__.update(kw)


class Folder:
    """A directory of files that goes away with the state."""

    def __init__(self, files):
        self.path = tempfile.mkdtemp(prefix="cases_", dir="/dev/shm" if os.path.isdir("/dev/shm") else None)
        for i, data in enumerate(files):
            with open(os.path.join(self.path, "%05d.jpg" % i), "wb") as f:
                f.write(data)

    def __del__(self, remove=shutil.rmtree):
        remove(self.path, ignore_errors=True)


def prepare(case, seed):
    path = case["path"]
    items = _samples(case, seed)
    cfg = image_config(case)
    if path == "client":
        folder = Folder(items)
        conf = dict(source_type="file", source_config=dict(root_path=folder.path, rank=0, world_size=1), limit=len(items), samples_buffer_size=64, image_config=cfg)
        return State(path=path, folder=folder, client=DatagoClient(json.dumps(conf)))
    if path == "feeder":
        return State(path=path, feeder=_kept("feeder", case), items=items, to_rgb8=case["data"] == "mixed")
    ctx = _kept("context", case)
    if path == "static":
        src = torch.from_numpy(items[0]).cuda()
        h, w = items[0].shape[:2]
        plan = ctx.plan_geometry(w, h, 3)
        return State(path=path, ctx=ctx, src=src, w=w, h=h, dst=torch.empty((plan.target_h, plan.target_w, 3), dtype=torch.uint8, device="cuda"))
    forced = None
    if case["data"] == "pairs444":  # the mask goes where its image goes
        forced = [k for jpg in items[::2] for k in (None, _key(ctx, jpg))]
    s = State(path=path, ctx=ctx, items=items, forced=forced, to_rgb8=True if case["data"] == "mixed" else None, collate=len(items) > MAX_OUTPUTS // 2)
    flags = dg.BATCH_COLLATE if s.collate else 0
    if path == "resident":
        s.batch = ctx.batch(items, forced, flags, s.to_rgb8)
        s.batch.upload()
        s.batch.run()
        s.batch.sync()
        _all_ok(s.batch)
        s.outputs = _on_device(s.batch, s.collate)
    elif path == "host":
        with ctx.batch(items, forced, flags, s.to_rgb8) as b:
            s.landing = torch.empty(b.packed_bytes(), dtype=torch.uint8).pin_memory().numpy()
    return s


def _key(ctx, jpg):
    info = dg.jpeg_probe(jpg)
    return ctx.plan_geometry(info.width, info.height, 3).key.decode()


def _all_ok(batch):
    for i in range(len(batch)):
        status = batch.result(i).status
        if status:
            raise RuntimeError("item %d: status %d" % (i, status))


def _on_device(batch, collate):
    """The payloads as tensors over the batch's device memory."""
    if collate:
        return [torch.as_tensor(b["array"], device="cuda") for b in batch.buckets()]
    got = [batch.result(i) for i in range(len(batch))]
    return [torch.as_tensor(dg.DeviceArray(r.device_data, (r.height, r.width, r.channels), batch), device="cuda") for r in got]


# ---- one pass -------------------------------------------------------------------------------------------------------------
def run(state):
    return _PASS[state.path](state)


def _run_process(s):
    got = s.ctx.process(s.items, s.forced, 0, s.to_rgb8)
    return [pixels for _, pixels, _ in got]


def _run_host(s):
    with s.ctx.batch(s.items, s.forced, dg.BATCH_COLLATE if s.collate else 0, s.to_rgb8) as b:
        b.upload()
        b.run()
        b.download_packed(s.landing)
        b.sync()
        if s.collate:
            places = [(k["packed_offset"], k["nbytes"], k["shape"]) for k in b.buckets()]
        else:
            places = [(r.packed_offset, r.nbytes, (r.height, r.width, r.channels)) for r in (b.result(i) for i in range(len(b)))]
    return [s.landing[o:o + n].reshape(shape) for o, n, shape in places]


def _run_device(s):
    s.batch = s.outputs = None  # the last batch has been consumed
    s.batch = b = s.ctx.batch(s.items, s.forced, dg.BATCH_COLLATE if s.collate else 0, s.to_rgb8)
    b.upload()
    b.run()
    b.sync()  # statuses of the samples
    s.outputs = _on_device(b, s.collate)
    return s.outputs


def _run_feeder(s):
    tickets = [s.feeder.submit(x, to_rgb8=s.to_rgb8) for x in s.items]
    out = []
    for t in tickets:
        r = s.feeder.wait(t)
        out.append(s.feeder.fetch(t, r))
        s.feeder.release(t)
    return out


def _run_client(s):
    samples = {}
    while True:
        sample = s.client.get_sample()
        if sample is None:
            break
        samples[sample.id] = sample.image.to_numpy_array()
    return [samples[k] for k in sorted(samples)]


def _run_resident(s):
    s.batch.run()
    return s.outputs


def _run_static(s):
    s.ctx.resize_device_static(s.src.data_ptr(), s.w, s.h, 3, s.dst.data_ptr())
    return s.dst


_PASS = dict(process=_run_process, host=_run_host, device=_run_device, feeder=_run_feeder, client=_run_client, resident=_run_resident, static=_run_static)

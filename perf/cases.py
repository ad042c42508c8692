"""The work this library is used for, as cases that can be timed through its public entry points.

A case is a dict of plain values; ``kind`` says which entry point it goes through:

* ``gops``    Engine.analyse_gops_device: the pictures of several streams, sources on the device, one
              persistent launch, the records copied to pinned memory for the bitstream writers (and, with
              ``recon``, the last reconstructions) -- in the plain, full-search or learned form;
* ``group``   Engine.analyse_gops_group: the same for engines of several picture sizes at once;
* ``wave``    H264Encoder.submit / collect: host frames in, access units out;
* ``frame``   H264Encoder.encode_frame: one picture per call, as ragdoll's own encoder is called;
* ``hints``   CandidateNet.predict_hints: the network and the coarse motion pass of the learned form;
* ``grads``   CandidateNet.forward_backward: the pass of a training step that yields the gradients;
* ``ssim``    ssim_batch_device: SSIM and MS-SSIM of many plane pairs;
* ``ssim1``   ssim_plane_device_noalloc: one plane pair, no allocation.

Sources are the library's seeded test pictures (ragdoll_b200.synth.grating_clip: four gratings and
blurred noise under a global motion, moving textured rectangles), drawn here on the device.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from ragdoll_b200.encoder import H264Encoder
from ragdoll_b200.engine import (HINT_DTYPE, PROFILES, RECORD_DTYPE, RG_FORM_FULLSEARCH, RG_FORM_LEARNED, RG_FORM_PLAIN,
                                 RG_FRAME_IDR, RG_FRAME_P, Engine, RgError, lib, ssim_batch_device,
                                 ssim_plane_device_noalloc)
from ragdoll_b200.learned import CandidateNet

FORMS = {"plain": RG_FORM_PLAIN, "fullsearch": RG_FORM_FULLSEARCH, "learned": RG_FORM_LEARNED}
# the picture sizes of the batched workload
MIXED_SIZES = ((320, 240), (640, 360), (1280, 720), (1920, 1080))


def listed():
    return [
        # a live or interactive source: one small picture per call (an IDR picture and three P pictures)
        {"name": "frame_320x180", "kind": "frame", "width": 320, "height": 180, "profile": "main", "qp": 26,
         "frames": 4, "motion": 4.0, "rects": 2},
        # one 720p stream, Constrained Baseline, a GOP of 30 in one launch: a transcode that cannot be cut up
        {"name": "stream_720p", "kind": "gops", "form": "plain", "width": 1280, "height": 720, "profile": "baseline",
         "qp": 30, "streams": 1, "frames": 30, "motion": 8.0, "rects": 6, "recon": True},
        # the headline workload: 120 pictures of 1080p High as eight GOPs side by side
        {"name": "gops_1080p", "kind": "gops", "form": "plain", "width": 1920, "height": 1080, "profile": "high",
         "qp": 26, "streams": 8, "frames": 15, "motion": 24.0, "rects": 12, "recon": False},
        # the whole encode, host frames to access units
        {"name": "wave_1080p", "kind": "wave", "width": 1920, "height": 1080, "profile": "high", "qp": 26,
         "streams": 4, "frames": 10, "motion": 24.0, "rects": 12},
        # a batched transcode: streams of four sizes and their own QPs in one launch
        {"name": "mixed_sizes", "kind": "group", "profile": "main", "qp": 28, "streams": 4, "frames": 10,
         "motion": 8.0, "rects": 6, "sizes": 4},
        # the training labels' generator: exhaustive search over eight clips of three pictures
        {"name": "fullsearch_720p", "kind": "gops", "form": "fullsearch", "range": 32, "width": 1280, "height": 720,
         "profile": "high", "qp": 22, "streams": 8, "frames": 3, "motion": 24.0, "rects": 12, "recon": False},
        # the learned form at 1080p: network, coarse motion and restricted search
        {"name": "learned_1080p", "kind": "gops", "form": "learned", "range": 32, "width": 1920, "height": 1080,
         "profile": "high", "qp": 26, "streams": 8, "frames": 8, "motion": 24.0, "rects": 12, "recon": False},
        # the learned form at 4K with its wide fallback
        {"name": "learned_4k", "kind": "gops", "form": "learned", "range": 64, "width": 3840, "height": 2160,
         "profile": "high", "qp": 28, "streams": 4, "frames": 3, "motion": 48.0, "rects": 24, "recon": False},
        # the candidate network and the coarse motion pass alone, eight pictures
        {"name": "hints_1080p", "kind": "hints", "width": 1920, "height": 1080, "frames": 8, "coarse": 32,
         "motion": 24.0, "rects": 12},
        # the gradients of one training batch
        {"name": "grads_256", "kind": "grads", "batch": 256, "motion": 24.0, "rects": 12},
        # the quality of a job's reconstructions: sixty 1080p pairs, SSIM and MS-SSIM
        {"name": "ssim_1080p", "kind": "ssim", "width": 1920, "height": 1080, "pairs": 60, "ms": True,
         "motion": 8.0, "rects": 6},
        # the quality of one small picture inside a frame loop that may not allocate
        {"name": "ssim_360p", "kind": "ssim1", "width": 640, "height": 360, "motion": 8.0, "rects": 6},
    ]


def _size(rng, lo, hi):
    """A picture size between lo and hi samples wide, odd ones among them."""
    w = int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
    h = int(round(w * rng.choice((9 / 16, 3 / 4, 10 / 16, 1.0))))
    return max(32, w), max(32, h)


def _pictures(rng, w, h, most, top=64):
    """How many pictures of w x h are taken at once: at most `most` samples of luma in all."""
    return max(1, min(top, int(math.exp(rng.uniform(0.0, math.log(max(2.0, most / (w * h))))))))


def draw(rng):
    kind = rng.choice(("gops", "gops", "gops", "group", "wave", "frame", "hints", "grads", "ssim", "ssim1"))
    motion, rects = round(rng.uniform(0.0, 24.0), 2), rng.randint(0, 12)
    qp, profile = rng.randint(20, 36), rng.choice(("baseline", "main", "high"))
    c = {"kind": kind, "motion": motion, "rects": rects}
    if kind == "gops":
        form = rng.choice(("plain", "plain", "learned", "fullsearch"))
        w, h = _size(rng, 160, 2560 if form == "plain" else 1920)
        most = {"plain": 100e6, "learned": 60e6, "fullsearch": 12e6}[form]
        n = _pictures(rng, w, h, most, 240)
        frames = max(1, min(30, int(round(math.exp(rng.uniform(0.0, math.log(n + 1)))))))
        c.update(form=form, width=w, height=h, qp=qp, streams=max(1, min(16, n // frames)), frames=frames,
                 recon=rng.random() < 0.3, profile=profile if form == "plain" else rng.choice(("main", "high")))
        if form != "plain":
            c["range"] = rng.choice((8, 16, 24, 32))
    elif kind == "group":
        c.update(profile=profile, qp=qp, streams=rng.randint(1, 4), frames=rng.randint(2, 10), sizes=rng.randint(2, 4))
    elif kind == "wave":
        w, h = _size(rng, 160, 1920)
        n = _pictures(rng, w, h, 60e6, 120)
        frames = max(1, min(15, n))
        c.update(width=w, height=h, profile=profile, qp=qp, streams=max(1, min(8, n // frames)), frames=frames)
    elif kind == "frame":
        w, h = _size(rng, 96, 1920)
        c.update(width=w, height=h, profile=profile, qp=qp, frames=rng.randint(1, 6))
    elif kind == "hints":
        w, h = _size(rng, 160, 3840)
        c.update(width=w, height=h, frames=_pictures(rng, w, h, 30e6, 32), coarse=rng.choice((0, 16, 32, 32, 64)))
    elif kind == "grads":
        c.update(batch=int(round(math.exp(rng.uniform(math.log(16), math.log(512))))))
    elif kind == "ssim":
        w, h = _size(rng, 64, 3840)
        c.update(width=w, height=h, pairs=_pictures(rng, w, h, 120e6, 120), ms=rng.random() < 0.75)
    else:
        w, h = _size(rng, 64, 1920)
        c.update(width=w, height=min(h, 1088))
    return c


# ---- sources ------------------------------------------------------------------------------------
def _blurred_noise(h, w, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    x = torch.rand((h + 10, w + 10), generator=g, device="cuda") * 40.0 - 20.0
    k = [math.exp(-0.5 * (i / 1.5) ** 2) for i in range(-5, 6)]
    k = [v / sum(k) for v in k]
    x = sum(k[i] * x[i:i + h] for i in range(11))
    return sum(k[i] * x[:, i:i + w] for i in range(11))


def _clip(w, h, frames, seed, motion, rects):
    """A seeded clip on the device: [frames, w h + 2 (w/2)(h/2)] bytes, Y | U | V of each picture."""
    rng = np.random.default_rng(seed)
    periods, angles = rng.uniform(8, 64, 4), rng.uniform(0, np.pi, 4)
    phases, amps = rng.uniform(0, 2 * np.pi, 4), rng.uniform(12, 28, 4)
    steps = np.round(rng.uniform(-motion, motion, (frames, 2)) * 4) / 4
    steps[0] = 0
    pos = np.cumsum(steps, axis=0)
    boxes = []
    for _ in range(rects):
        rw, rh = (int(v) for v in rng.integers(64, 257, 2))
        boxes.append((rw, rh, rng.uniform(0, max(1, w - rw)), rng.uniform(0, max(1, h - rh)),
                      *rng.uniform(-motion, motion, 2), rng.uniform(6, 24), rng.uniform(0, np.pi), rng.uniform(40, 215)))
    lo = np.floor(pos.min(axis=0)).astype(int)
    span = np.ceil(pos.max(axis=0)).astype(int) - lo + 2
    noise = _blurred_noise(h + int(span[1]), w + int(span[0]), seed)
    ys = torch.arange(h, device="cuda", dtype=torch.float32)[:, None]
    xs = torch.arange(w, device="cuda", dtype=torch.float32)[None, :]
    cw, ch = (w + 1) // 2, (h + 1) // 2
    out = torch.empty((frames, w * h + 2 * cw * ch), dtype=torch.uint8, device="cuda")
    for f in range(frames):
        gx, gy = pos[f]
        x0, y0 = int(np.floor(gx)) - int(lo[0]), int(np.floor(gy)) - int(lo[1])
        fx, fy = float(gx - np.floor(gx)), float(gy - np.floor(gy))
        field = 126.0 + (1 - fx) * (1 - fy) * noise[y0:y0 + h, x0:x0 + w] + fx * (1 - fy) * noise[y0:y0 + h, x0 + 1:x0 + 1 + w] \
            + (1 - fx) * fy * noise[y0 + 1:y0 + 1 + h, x0:x0 + w] + fx * fy * noise[y0 + 1:y0 + 1 + h, x0 + 1:x0 + 1 + w]
        for p, a, ph, am in zip(periods, angles, phases, amps):
            k = 2 * np.pi / p
            field += float(am) * torch.sin(float(k * np.cos(a)) * xs + float(k * np.sin(a)) * ys
                                           + float(k * (gx * np.cos(a) + gy * np.sin(a)) + ph))
        for rw, rh, rx, ry, vx, vy, tp, ta, base in boxes:
            xr, yr = int(round(rx + vx * f)), int(round(ry + vy * f))
            xa, xb, ya, yb = max(0, xr), min(w, xr + rw), max(0, yr), min(h, yr + rh)
            if xa < xb and ya < yb:
                k = 2 * np.pi / tp
                field[ya:yb, xa:xb] = base + 30 * torch.sin(float(k * np.cos(ta)) * (xs[:, xa:xb] - xr)
                                                            + float(k * np.sin(ta)) * (ys[ya:yb] - yr))
        out[f, :w * h] = field.round().clamp(16, 235).to(torch.uint8).reshape(-1)
        c = torch.nn.functional.pad(field[None, None], (0, 2 * cw - w, 0, 2 * ch - h), mode="replicate")[0, 0]
        c = c.reshape(ch, 2, cw, 2).mean(dim=(1, 3)) - 126.0
        out[f, w * h:w * h + cw * ch] = (c * 0.5 + 128).round().clamp(16, 240).to(torch.uint8).reshape(-1)
        out[f, w * h + cw * ch:] = (c * -0.4 + 128).round().clamp(16, 240).to(torch.uint8).reshape(-1)
    return out


def _clips(w, h, streams, frames, seed, motion, rects):
    """[streams, frames, picture bytes], an independent clip per stream."""
    return torch.stack([_clip(w, h, frames, seed * 1000 + s, motion, rects) for s in range(streams)])


def _pointers(clips, w, h):
    """Device pointers of the clips' planes in the order of the calls: picture, stream, plane."""
    cw, ch = (w + 1) // 2, (h + 1) // 2
    streams, frames, fb = clips.shape
    base = clips.data_ptr()
    return [base + (s * frames + f) * fb + o for f in range(frames) for s in range(streams)
            for o in (0, w * h, w * h + cw * ch)]


def _host_frames(clips, w, h):
    """(pinned tensor, frames[f][s] = (y, u, v) views of it)."""
    cw, ch = (w + 1) // 2, (h + 1) // 2
    pinned = torch.empty(clips.shape, dtype=torch.uint8, pin_memory=True)
    pinned.copy_(clips)
    a = pinned.numpy()
    frames = [[(a[s, f, :w * h].reshape(h, w), a[s, f, w * h:w * h + cw * ch].reshape(ch, cw),
                a[s, f, w * h + cw * ch:].reshape(ch, cw)) for s in range(clips.shape[0])] for f in range(clips.shape[1])]
    return pinned, frames


def _kinds(streams, frames):
    return [RG_FRAME_IDR if f == 0 else RG_FRAME_P for f in range(frames) for _ in range(streams)]


def _records(eng, frames):
    """Pinned memory for the records of `frames` pictures of every stream, as 64-bit words."""
    return torch.empty((frames * eng.num_streams * eng.n_mb, RECORD_DTYPE.itemsize // 8), dtype=torch.int64, pin_memory=True)


def _fetch(eng, frames, records):
    rc = lib().rg_copy_records_gops(eng.h, frames, records.data_ptr())
    if rc:
        raise RgError(rc, lib().rg_last_error().decode())


def _stream_qps(qp, streams, seed):
    """QPs of a batched job's streams, drawn around the case's."""
    rng = np.random.default_rng(seed)
    return [int(v) for v in np.clip(rng.integers(qp - 8, qp + 9, streams), 1, 51)]


# ---- cases --------------------------------------------------------------------------------------
def prepare(case, seed):
    kind, motion, rects = case["kind"], case["motion"], case["rects"]
    s = {"kind": kind}
    if kind == "gops":
        w, h, S, F = case["width"], case["height"], case["streams"], case["frames"]
        s["src"] = _clips(w, h, S, F, seed, motion, rects)
        s["ptrs"], s["kinds"], s["frames"], s["recon"] = _pointers(s["src"], w, h), _kinds(S, F), F, case["recon"]
        s["eng"] = Engine(w, h, case["qp"], profile=PROFILES[case["profile"]], num_streams=S, max_frames=F)
        if case["form"] != "plain":
            s["eng"].set_analysis_form(FORMS[case["form"]], case["range"])
        if case["form"] == "learned":
            s["net"] = CandidateNet.trained()
            s["eng"].set_hint_net(s["net"])
        s["records"] = _records(s["eng"], F)
    elif kind == "group":
        S, F = case["streams"], case["frames"]
        s["frames"], s["engs"], s["src"], s["ptrs"], s["kinds"], s["records"] = F, [], [], [], [], []
        for k, (w, h) in enumerate(MIXED_SIZES[-case["sizes"]:]):
            eng = Engine(w, h, case["qp"], profile=PROFILES[case["profile"]], num_streams=S, max_frames=F)
            for i, qp in enumerate(_stream_qps(case["qp"], S, seed * 10 + k)):
                eng.set_stream_qp(i, qp)
            clips = _clips(w, h, S, F, seed * 10 + k, motion, rects)
            s["engs"].append(eng)
            s["src"].append(clips)
            s["ptrs"].append(_pointers(clips, w, h))
            s["kinds"].append(_kinds(S, F))
            s["records"].append(_records(eng, F))
        s["sy"] = [e.width for e in s["engs"]]
        s["suv"] = [(e.width + 1) // 2 for e in s["engs"]]
    elif kind in ("wave", "frame"):
        w, h, S, F = case["width"], case["height"], case.get("streams", 1), case["frames"]
        s["pinned"], s["frames"] = _host_frames(_clips(w, h, S, F, seed, motion, rects), w, h)
        s["enc"] = H264Encoder(w, h, case["qp"], profile=PROFILES[case["profile"]], keyint=max(F, 2), streams=S,
                               max_frames=F if kind == "wave" else 1)
    elif kind == "hints":
        w, h, F = case["width"], case["height"], case["frames"]
        s["src"] = _clip(w, h, F + 1, seed, motion, rects)
        s["size"] = (w, h)
        s["cur"] = [s["src"][f + 1].data_ptr() for f in range(F)]
        s["prev"] = [s["src"][f].data_ptr() for f in range(F)]
        n_mb = ((w + 15) // 16) * ((h + 15) // 16)
        s["hints"] = torch.zeros((F, n_mb * HINT_DTYPE.itemsize), dtype=torch.uint8, device="cuda")
        s["dst"] = [s["hints"][f].data_ptr() for f in range(F)]
        s["net"] = CandidateNet.trained()
        s["net"].set_coarse_range(case["coarse"])
    elif kind == "grads":
        s.update(_batch(case["batch"], seed, motion, rects))
        s["net"] = CandidateNet(seed=1 + seed % 1000)
        s["batch"] = case["batch"]
    else:
        w, h, n = case["width"], case["height"], case.get("pairs", 1)
        s["size"], s["ms"] = (w, h), case.get("ms", True)
        s["a"] = _clip(w, h, n, seed, motion, rects)[:, :w * h].contiguous()
        g = torch.Generator(device="cuda").manual_seed(seed + 1)
        # a reconstruction differs from its source by a few levels
        d = torch.randn(s["a"].shape, generator=g, device="cuda") * 2.5
        s["b"] = (s["a"].float() + d).round().clamp(0, 255).to(torch.uint8)
        s["pa"] = [s["a"][i].data_ptr() for i in range(n)]
        s["pb"] = [s["b"][i].data_ptr() for i in range(n)]
        s["out"] = torch.zeros(2, dtype=torch.float64, device="cuda")
    return s


def _batch(n, seed, motion, rects):
    """Crops of a clip and labels as the full search's decisions give them: a third of the samples
    from IDR pictures (intra 4x4 modes, where the macroblock was coded so), the rest from P pictures
    (partition types, the 16x16 vectors' offsets)."""
    w, h = 640, 360
    luma = _clip(w, h, 3, seed, motion, rects)[:, :w * h].reshape(3, h, w)
    rng = np.random.default_rng(seed + 7)
    f = rng.integers(0, 3, n)
    x, y = rng.integers(0, w - 24, n), rng.integers(0, h - 24, n)
    crops = torch.stack([torch.stack([luma[k, b:b + 24, a:a + 24], luma[max(k - 1, 0), b:b + 24, a:a + 24]])
                         for k, a, b in zip(f.tolist(), x.tolist(), y.tolist())]).contiguous()
    part = np.where(f > 0, rng.choice(4, n, p=(0.55, 0.18, 0.17, 0.10)), -1).astype(np.int32)
    i4 = np.where(((f == 0) & (rng.random(n) < 0.8))[:, None], rng.integers(0, 9, (n, 16)), -1).astype(np.int32)
    mv = np.clip(rng.normal(0, 0.5, (n, 2)), -3, 3).astype(np.float32)
    mvv = ((part == 0) & (rng.random(n) < 0.9)).astype(np.int32)
    dev = {k: torch.from_numpy(v).cuda() for k, v in (("part", part), ("i4", i4), ("mv", mv), ("mvv", mvv))}
    return {"crops": crops, **dev}


def run(s):
    kind = s["kind"]
    if kind == "gops":
        eng = s["eng"]
        eng.analyse_gops_device(s["ptrs"], eng.width, (eng.width + 1) // 2, s["kinds"], s["frames"])
        _fetch(eng, s["frames"], s["records"])
        if s["recon"]:
            return [s["records"], [list(eng.recon(k)) for k in range(eng.num_streams)]]
        return s["records"]
    if kind == "group":
        Engine.analyse_gops_group(s["engs"], s["ptrs"], s["sy"], s["suv"], s["kinds"], s["frames"])
        for eng, records in zip(s["engs"], s["records"]):
            _fetch(eng, s["frames"], records)
        return s["records"]
    if kind == "wave":
        s["enc"].new_gops()
        s["enc"].submit(s["frames"])
        return _units([u for row in s["enc"].collect() for u in row], s["enc"])
    if kind == "frame":
        s["enc"].new_gops()
        return _units([s["enc"].encode_frame(row[0]) for row in s["frames"]], s["enc"])
    if kind == "hints":
        w, h = s["size"]
        s["net"].predict_hints(s["cur"], s["prev"], w, h, w, s["dst"], stream=torch.cuda.current_stream().cuda_stream)
        return s["hints"]
    if kind == "grads":
        loss, grads = s["net"].forward_backward(s["crops"].data_ptr(), s["batch"], s["part"].data_ptr(), s["i4"].data_ptr(),
                                                s["mv"].data_ptr(), s["mvv"].data_ptr(), want_grads=True)
        return {"loss": loss, "grads": grads}
    w, h = s["size"]
    if kind == "ssim":
        ssim, ms = ssim_batch_device(s["pa"], s["pb"], w, h, w, w, stream=torch.cuda.current_stream().cuda_stream, ms=s["ms"])
        return {"ssim": ssim, "ms": ms}
    ssim_plane_device_noalloc(s["pa"][0], w, s["pb"][0], w, w, h, s["out"].data_ptr(),
                              stream=torch.cuda.current_stream().cuda_stream)
    return s["out"]


def _units(units, enc):
    """Access units back to back in a buffer that holds four bits a sample (zeros behind them), and their sizes."""
    data = b"".join(units)
    out = np.zeros(len(units) * (enc.width * enc.height // 2 + 4096), np.uint8)
    out[:len(data)] = np.frombuffer(data, np.uint8)
    return {"bytes": out, "sizes": np.array([len(u) for u in units], np.int64)}


def work(case):
    kind = case["kind"]
    if kind == "grads":
        # three 3x3 convolutions of 32 channels forward, their input gradients (not the first's) and weight gradients
        conv = [2 * 9 * 32 * c * p for c, p in ((2, 22 * 22), (32, 20 * 20), (32, 18 * 18))]
        return {"bytes": case["batch"] * (1152 + 4 + 64 + 8 + 4) + 2 * 4 * 19599, "flops": case["batch"] * (2 * sum(conv) + conv[1] + conv[2])}
    if kind == "group":
        sizes = MIXED_SIZES[-case["sizes"]:]
    else:
        sizes = ((case["width"], case["height"]),)
    nbytes = flops = 0
    for w, h in sizes:
        n_mb, yuv = ((w + 15) // 16) * ((h + 15) // 16), w * h + 2 * ((w + 1) // 2) * ((h + 1) // 2)
        if kind == "hints":
            # each picture's luma once (a picture is the next one's previous), its hints; 13.9 MFLOP a macroblock
            nbytes += (case["frames"] + 1) * w * h + case["frames"] * n_mb * HINT_DTYPE.itemsize
            flops += case["frames"] * n_mb * 2 * 9 * 32 * (2 * 22 * 22 + 32 * 20 * 20 + 32 * 18 * 18)
        elif kind in ("ssim", "ssim1"):
            nbytes += case.get("pairs", 1) * (2 * w * h + 16)
        else:
            # per picture: source in, reference in (P pictures), reconstruction and records out
            n = case.get("streams", 1)
            nbytes += n * case["frames"] * (2 * yuv + n_mb * RECORD_DTYPE.itemsize) + n * (case["frames"] - 1) * yuv
            if case.get("form") == "learned":
                flops += n * case["frames"] * n_mb * 2 * 9 * 32 * (2 * 22 * 22 + 32 * 20 * 20 + 32 * 18 * 18)
    return {"bytes": nbytes, "flops": flops}


# ---- the computed numbers in 64 bits --------------------------------------------------------------
def exact(case, seed):
    if case["kind"] == "grads":
        return _exact_grads(case, seed)
    if case["kind"] in ("ssim", "ssim1"):
        s = prepare(case, seed)
        w, h = s["size"]
        got = [_exact_ssim(a.reshape(h, w), b.reshape(h, w), s["ms"]) for a, b in zip(s["a"], s["b"])]
        if case["kind"] == "ssim1":
            return torch.tensor(got[0], dtype=torch.float64)
        return {"ssim": np.array([g[0] for g in got]), "ms": np.array([g[1] for g in got]) if s["ms"] else None}
    return None  # records, hints and access units are whole numbers


def _ssim64(a, b):
    """Mean SSIM over the 8x8 windows at every fourth sample (sums of 4x4 blocks)."""
    bh, bw = a.shape[0] // 4, a.shape[1] // 4
    a, b = a[:4 * bh, :4 * bw], b[:4 * bh, :4 * bw]
    blocks = [v.reshape(bh, 4, bw, 4).sum(dim=(1, 3)) for v in (a, b, a * a + b * b, a * b)]
    s1, s2, ss, s12 = ((v[:-1, :-1] + v[1:, :-1] + v[:-1, 1:] + v[1:, 1:]) if bh > 1 and bw > 1 else v for v in blocks)
    var, cov = ss * 64 - s1 * s1 - s2 * s2, s12 * 64 - s1 * s2
    return float(((2 * s1 * s2 + 416) * (2 * cov + 235963) / ((s1 * s1 + s2 * s2 + 416) * (var + 235963))).mean())


def _exact_ssim(a, b, ms):
    a, b = a.double(), b.double()
    weights, scores = (0.0448, 0.2856, 0.3001, 0.2363, 0.1333), []
    for level in range(5 if ms else 1):
        scores.append(_ssim64(a, b))
        h, w = a.shape[0] // 2, a.shape[1] // 2
        if w < 8 or h < 8:
            break
        a, b = (((v[:2 * h:2, :2 * w:2] + v[:2 * h:2, 1:2 * w:2] + v[1:2 * h:2, :2 * w:2] + v[1:2 * h:2, 1:2 * w:2] + 2) / 4).floor()
                for v in (a, b))
    total = sum(weights[:len(scores)])
    prod = 1.0
    for wt, v in zip(weights, scores):
        prod *= max(min(max(v, 0.0), 1.0), 1e-9) ** (wt / total)
    return scores[0], min(max(prod, 0.0), 1.0)


def _exact_grads(case, seed):
    s = prepare(case, seed)
    n, F = case["batch"], torch.nn.functional
    flat = torch.from_numpy(s["net"].params()).double().cuda().requires_grad_()
    shapes = ((32, 2, 3, 3), (32,), (32, 32, 3, 3), (32,), (32, 32, 3, 3), (32,), (4, 32), (4,), (2, 32), (2,), (9, 32), (9,))
    p = [v.reshape(sh) for v, sh in zip(flat.split([math.prod(sh) for sh in shapes]), shapes)]

    def conv(x, weight, bias):  # valid 3x3 convolution as one product
        cols = F.unfold(x, 3)
        return torch.relu(weight.reshape(32, -1) @ cols + bias[:, None]).reshape(len(x), 32, x.shape[2] - 2, x.shape[3] - 2)

    total = 0.0
    counts = [max(1, int((s["part"] >= 0).sum())), max(1, int((s["i4"] >= 0).sum())), max(1, int((s["mvv"] != 0).sum()))]
    for i in range(0, n, 64):
        part, i4, mv, mvv = (s[k][i:i + 64].long() if k != "mv" else s[k][i:i + 64].double() for k in ("part", "i4", "mv", "mvv"))
        x = (s["crops"][i:i + 64].double() - 128) / 64
        a = conv(conv(conv(x, p[0], p[1]), p[2], p[3]), p[4], p[5])
        g = a.mean(dim=(2, 3))
        blocks = F.avg_pool2d(a[:, :, 1:17, 1:17], 4).flatten(2).transpose(1, 2)
        loss = F.cross_entropy(g @ p[6].T + p[7], part, ignore_index=-1, reduction="sum") / counts[0]
        loss = loss + F.cross_entropy((blocks @ p[10].T + p[11]).flatten(0, 1), i4.flatten(), ignore_index=-1, reduction="sum") / counts[1]
        off = F.huber_loss(g @ p[8].T + p[9], mv, reduction="none").sum(dim=1)
        loss = loss + 0.25 * (off * (mvv != 0)).sum() / counts[2]
        loss.backward(retain_graph=i + 64 < n)
        total += float(loss.detach())
    return {"loss": total, "grads": flat.grad.cpu().numpy()}

"""The encoder's work as its users have it done: the cases, their inputs and one pass of each.

Kinds:

* ``live``: a camera or a call.  One encoder at pipeline depth 0 (``EncoderConfig.new``'s
  default), one ``encode_frame`` per pass from a host RGB buffer; the pass returns the record
  that reached the writer.  Key frames every 30 frames, as the default configuration has them.
* ``clip``: a recording cut into segments.  One encoder with frames in flight; a pass encodes
  one segment (a key frame, then P-frames), flushes it with ``finish`` and takes the
  segment's records.  RGB frames in pinned host memory or already on the device.
* ``batch``: many independent clips of mixed size encoded together, one frame per clip and
  step, flushed at the end of each segment.
* ``decode``: playing a stream back, a segment of frames per pass, as planes or as RGB.
* ``train``: one training step of the proposal network.

Inputs are made on the GPU from the seed: gratings that pan, textured rectangles that move
by half-pixel steps over them, and noise -- the scene model of the repository's synthetic
clips.
"""
from __future__ import annotations

import math
import os

import numpy as np
import torch
import torch.nn.functional as F

import riv2_b200
from riv2_b200 import batch as B
from riv2_b200 import decoder as D
from riv2_b200 import encoder as E
from riv2_b200 import proposal as P

HEADER = 36  # bytes of a stream's header
WEIGHTS = os.path.join(os.path.dirname(os.path.abspath(riv2_b200.__file__)), "weights", "proposal.bin")
FORMS = {"plain": 0, "learned": 1, "parallel": 2}
# the sizes of the multi-clip workload, taken in turn by a batch's clips
BATCH_SIZES = ((352, 288), (640, 360), (1280, 720), (1920, 1080))


def _clip(name, w, h, frames, depth, iq, pq, sr, form="plain", source="host"):
    return {"name": name, "kind": "clip", "w": w, "h": h, "frames": frames, "depth": depth, "iq": iq, "pq": pq,
            "sr": sr, "form": form, "source": source}


def listed():
    return [
        # a video call at CIF: the smallest call, where latency counts
        {"name": "live_cif", "kind": "live", "w": 352, "h": 288, "iq": 85, "pq": 80, "sr": 12, "form": "plain"},
        # a camera at 1080p with the default, synchronous configuration
        {"name": "live_1080p", "kind": "live", "w": 1920, "h": 1080, "iq": 85, "pq": 80, "sr": 12, "form": "plain"},
        # an odd display size (storage 864x480) at a lower quality, frames decoded on the device
        _clip("clip_odd_480p", 853, 479, 16, 8, 75, 70, 12, source="device"),
        # the headline workload: 1080p, quality 85/80, 16 frames in flight, host frames
        _clip("clip_1080p", 1920, 1080, 16, 16, 85, 80, 12),
        # the same size at the wide search range and the high quality
        _clip("clip_1080p_sr31_q95", 1920, 1080, 12, 16, 95, 90, 31),
        # the largest frames
        _clip("clip_4k", 3840, 2160, 6, 8, 75, 70, 12, source="device"),
        # the learned-proposal form at 1080p, device frames, as the headline metric compares it
        _clip("learned_1080p", 1920, 1080, 16, 16, 85, 80, 12, form="learned", source="device"),
        # 24 mixed clips on one GPU (an encoding service)
        {"name": "batch_24", "kind": "batch", "clips": 24, "steps": 8, "depth": 4, "iq": 85, "pq": 80, "sr": 12,
         "source": "device"},
        # 32 small streams at the default quality (a wall of thumbnails), host frames
        {"name": "batch_small", "kind": "batch", "clips": 32, "steps": 8, "depth": 4, "iq": 90, "pq": 35, "sr": 12,
         "source": "host", "w": 320, "h": 180},
        # verification playback at 1080p: YUV planes
        {"name": "decode_1080p", "kind": "decode", "w": 1920, "h": 1080, "frames": 12, "iq": 85, "pq": 80, "sr": 12,
         "out": "yuv"},
        # thumbnails of a CIF stream: RGB
        {"name": "decode_cif_rgb", "kind": "decode", "w": 352, "h": 288, "frames": 12, "iq": 85, "pq": 80, "sr": 12,
         "out": "rgb"},
        # the proposal network's training at its default batch
        {"name": "train_4096", "kind": "train", "n": 4096},
    ]


def _logint(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _size(rng, wmin, wmax):
    w = _logint(rng, wmin, wmax)
    h = max(64, int(w * rng.choice((9 / 16, 3 / 4, 1.0, 16 / 9) if w < 1000 else (9 / 16, 9 / 16, 3 / 4))) + rng.randrange(-8, 9))
    return w, h


def draw(rng):
    kind = rng.choice(("live", "clip", "clip", "clip", "batch", "decode", "train"))
    iq, pq = rng.choice(((85, 80), (95, 90), (75, 70), (90, 35)))
    sr = rng.choice((7, 12, 12, 12, 15, 16, 24, 31))
    if kind == "live":
        w, h = _size(rng, 128, 1920)
        return {"kind": "live", "w": w, "h": h, "iq": iq, "pq": pq, "sr": sr, "form": rng.choice(("plain", "plain", "learned"))}
    if kind == "clip":
        w, h = _size(rng, 160, 2560)
        c = _clip("", w, h, rng.randrange(4, 9) if sr > 15 or w > 1920 else rng.randrange(6, 13), rng.choice((4, 8, 16)), iq, pq, sr,
                  rng.choice(("plain", "plain", "learned", "parallel")), rng.choice(("host", "device")))
        del c["name"]
        return c
    if kind == "batch":
        c = {"kind": "batch", "clips": rng.randrange(5, 21), "steps": rng.randrange(4, 8), "depth": rng.choice((2, 4)),
             "iq": iq, "pq": pq, "sr": min(sr, 16), "source": rng.choice(("host", "device"))}
        if rng.random() < 0.5:
            c["w"], c["h"] = _size(rng, 160, 640)
        return c
    if kind == "decode":
        w, h = _size(rng, 160, 1920)
        return {"kind": "decode", "w": w, "h": h, "frames": rng.randrange(6, 13), "iq": iq, "pq": pq, "sr": sr,
                "out": rng.choice(("yuv", "rgb"))}
    return {"kind": "train", "n": 64 * _logint(rng, 8, 96)}


# ---------------------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------------------

def _frames(w, h, n, seed):
    """n RGB24 frames (n, h, w, 3) uint8 on the GPU."""
    dev = torch.device("cuda")
    r = np.random.default_rng(seed)
    g = torch.Generator(device=dev).manual_seed(int(r.integers(1 << 31)))
    scale = w / 1920.0
    yy = torch.arange(h, device=dev, dtype=torch.float32)[:, None]
    xx = torch.arange(w, device=dev, dtype=torch.float32)[None, :]
    gr = [(r.uniform(0.01, 0.1), r.uniform(0, math.pi), r.uniform(0, 2 * math.pi), r.uniform(20, 60, 3)) for _ in range(3)]
    pan = r.uniform(-4, 4, 2)
    vmax = max(3.0, min(16.0, 16.0 * scale))
    rects = []
    for _ in range(14):
        rw, rh = (int(v) for v in r.integers(max(16, int(64 * scale)), max(32, int(384 * scale)), 2))
        cell = max(8, int(16 * scale))
        lat = torch.rand((1, 3, rh // cell + 3, rw // cell + 3), device=dev, generator=g) * 255.0
        tex = F.interpolate(lat, size=(2 * (rh + 1), 2 * (rw + 1)), mode="bilinear", align_corners=True)[0]
        rects.append((rw, rh, tex, r.integers(-rw // 2, w, 1)[0], r.integers(-rh // 2, h, 1)[0],
                      np.round(r.uniform(-vmax, vmax, 2) * 2)))
    out = torch.empty((n, h, w, 3), dtype=torch.uint8, device=dev)
    for t in range(n):
        v = torch.full((3, h, w), 128.0, device=dev)
        for f, th, ph, amp in gr:
            s = torch.sin(2 * math.pi * f * ((xx + pan[0] * t) * math.cos(th) + (yy + pan[1] * t) * math.sin(th)) + ph)
            for c in range(3):
                v[c] += float(amp[c]) * s
        for rw, rh, tex, x0, y0, vel in rects:  # positions and velocities in half pixels
            hx, hy = int(2 * x0 + vel[0] * t), int(2 * y0 + vel[1] * t)
            hx = (hx + 2 * rw) % (2 * (w + rw)) - 2 * rw
            hy = (hy + 2 * rh) % (2 * (h + rh)) - 2 * rh
            px, py = -(-hx // 2), -(-hy // 2)  # first covered pixel
            xa, xb, ya, yb = max(px, 0), min(px + rw, w), max(py, 0), min(py + rh, h)
            if xa < xb and ya < yb:
                sx, sy = 2 * xa - hx, 2 * ya - hy
                v[:, ya:yb, xa:xb] = tex[:, sy:sy + 2 * (yb - ya):2, sx:sx + 2 * (xb - xa):2]
        v += 2.0 * torch.randn((3, h, w), device=dev, generator=g)
        out[t] = v.round_().clamp_(0, 255).to(torch.uint8).permute(1, 2, 0)
    return out


def _host(t):
    """The frames in pinned host memory, as arrays."""
    p = torch.empty(t.shape, dtype=t.dtype, pin_memory=True)
    p.copy_(t)
    return list(p.numpy())


class _Segments(E.VideoWriter):
    """A writer over one buffer of fixed size; a segment's records are taken together, the header
    stays in front."""

    def __init__(self, cap):
        self.buf = np.zeros(HEADER + cap, np.uint8)
        self.view = memoryview(self.buf)
        self.pos = 0
        self.end = HEADER   # of what was written since the last take
        self.last = HEADER  # of what the last take returned

    def write(self, data):
        self.view[self.pos:self.pos + len(data)] = data
        self.pos += len(data)
        self.end = max(self.end, self.pos)

    def position(self):
        return self.pos

    def seek(self, pos):
        self.pos = pos

    def flush(self):
        pass

    def take(self):
        """The records and their length, zeros behind them (valid until the next frame)."""
        n = self.end
        self.buf[n:max(n, self.last)] = 0
        self.pos = self.end = HEADER
        self.last = n
        return [self.buf[HEADER:], n - HEADER]


def _writer(w, h, frames):
    return _Segments(w * h * 2 + frames * (w * h // 4) + 4096)


def _config(case, w, h, depth, gop):
    return (E.EncoderConfig.new(w, h, 30).with_intra_quality(case["iq"]).with_inter_quality(case["pq"])
            .with_search_range(case["sr"]).with_keyframe_interval(E.KeyframeInterval.fixed(gop))
            .with_pipeline_depth(depth).with_encode_form(FORMS[case.get("form", "plain")]))


def _encoder(case, w, h, depth, gop, writer):
    enc = E.Encoder.new(_config(case, w, h, depth, gop), writer)
    if case.get("form") == "learned":
        enc.set_proposal(P.load_params(WEIGHTS))
    return enc


def _batch_sizes(case):
    if "w" in case:
        return [(case["w"], case["h"])] * case["clips"]
    return [BATCH_SIZES[i % 4] for i in range(case["clips"])]


# ---------------------------------------------------------------------------------------
# the proposal network's training inputs
# ---------------------------------------------------------------------------------------

def _params(seed):
    """He-initialised parameters whose weights are bf16 values, so that the device's bf16 copy
    is the parameters themselves."""
    r = np.random.default_rng(seed)
    p = np.zeros(P.NW + P.NB, np.float32)
    o = 0
    for _, rows, cols, fan in P.WEIGHTS:
        w = np.zeros((rows, cols), np.float32)
        w[:, :fan] = r.normal(0.0, math.sqrt(2.0 / fan), (rows, fan))
        p[o:o + rows * cols] = torch.from_numpy(w).to(torch.bfloat16).float().numpy().reshape(-1)
        o += rows * cols
    p[o:] = r.normal(0.0, 0.05, P.NB)
    return p


def _records(n, seed):
    """n records as the trainer logs them: network inputs of consecutive frames' luma, target
    MVs (half pixels) and skip flags."""
    dev = torch.device("cuda")
    r = np.random.default_rng(seed + 1)
    w, h = 1280, 720
    per = (w // 16) * (h // 16)
    feats, x1s, tmvs = [], [], []
    got = 0
    fr = _frames(w, h, -(-n // per) + 1, seed).float()
    luma = (16.0 + 0.1826 * fr[..., 0] + 0.6142 * fr[..., 1] + 0.0620 * fr[..., 2]).round().to(torch.uint8).contiguous()
    for t in range(1, luma.shape[0]):
        mv = np.zeros((per, 4), np.int8)
        mv[:, :2] = np.clip(np.repeat(r.normal(0, 5, (per // 4, 2)), 4, axis=0), -12, 12)
        mv[:, 2:] = r.integers(0, 2, (per, 2))
        pc = torch.from_numpy(mv).to(dev)
        f = torch.empty((per, 24, 24, 2), dtype=torch.bfloat16, device=dev)
        x = torch.zeros((per, 320), dtype=torch.bfloat16, device=dev)
        rc = P.lib().riv_nn_features(luma[t].data_ptr(), luma[t - 1].data_ptr(), w, h, pc.data_ptr(), 0, per, f.data_ptr(),
                                     x.data_ptr(), None)
        if rc:
            raise RuntimeError(f"riv_nn_features failed ({rc})")
        torch.cuda.synchronize()
        feats.append(f)
        x1s.append(x)
        tmvs.append(torch.from_numpy((2 * mv[:, :2] + mv[:, 2:] + r.integers(-3, 4, (per, 2))).astype(np.int16)))
        got += per
    idx = torch.from_numpy(r.permutation(got)[:n].astype(np.int64))
    skip = torch.from_numpy((r.random(n) < 0.15).astype(np.uint8))
    return (torch.cat(feats)[idx.to(dev)].contiguous(), torch.cat(x1s)[idx.to(dev)].contiguous(),
            torch.cat(tmvs)[idx].contiguous().to(dev), skip.to(dev))


# ---------------------------------------------------------------------------------------
# state and passes
# ---------------------------------------------------------------------------------------

def prepare(case, seed):
    kind = case["kind"]
    if kind == "train":
        feat, x1, tmv, tskip = _records(case["n"], seed)
        return {"case": case, "net": P.ProposalNet(_params(seed + 2)), "data": (feat, x1, tmv, tskip)}
    if kind == "batch":
        writers, cfgs, frames = [], [], []
        for i, (w, h) in enumerate(_batch_sizes(case)):
            f = _frames(w, h, case["steps"], seed + 7919 * i)
            frames.append(f if case["source"] == "device" else _host(f))
            writers.append(_writer(w, h, case["steps"]))
            cfgs.append(_config(case, w, h, case["depth"], 30))
        torch.cuda.synchronize()
        return {"case": case, "batch": B.Batch.new(cfgs, writers), "writers": writers, "frames": frames, "t": 0}
    w, h = case["w"], case["h"]
    if kind == "live":
        frames = _host(_frames(w, h, 8, seed))
        writer = _writer(w, h, 1)
        return {"case": case, "enc": _encoder(case, w, h, 0, 30, writer), "writer": writer, "frames": frames, "t": 0}
    frames = _frames(w, h, case["frames"], seed)
    if kind == "clip":
        frames = _host(frames) if case["source"] == "host" else frames
        torch.cuda.synchronize()
        writer = _writer(w, h, case["frames"])
        enc = _encoder(case, w, h, case["depth"], case["frames"], writer)
        return {"case": case, "enc": enc, "writer": writer, "frames": frames, "t": 0}
    # decode: a stream of many segments, played from the start again at its end
    torch.cuda.synchronize()
    vec = E.VecWriter()
    enc = _encoder(case, w, h, 8, case["frames"], vec)
    for t in range(case["frames"] * 24):
        enc.encode_frame_device(frames[t % case["frames"]].data_ptr(), 33 * t)
    enc.finish()
    stream = vec.into_inner()
    enc.close()
    return {"case": case, "stream": stream, "dec": D.Decoder.new(stream)}


def _run_live(s):
    case, t = s["case"], s["t"]
    s["t"] = t + 1
    k = t % 14  # to the last of the eight frames and back
    s["enc"].encode_frame(E.Frame(s["frames"][k if k < 8 else 14 - k], case["w"], case["h"], 33 * t))
    return s["writer"].take()


def _run_clip(s):
    case, enc, t = s["case"], s["enc"], s["t"]
    s["t"] = t + case["frames"]
    for k, f in enumerate(s["frames"]):
        if case["source"] == "host":
            enc.encode_frame(E.Frame(f, case["w"], case["h"], 33 * (t + k)))
        else:
            enc.encode_frame_device(f.data_ptr(), 33 * (t + k))
    enc.finish()
    return s["writer"].take()


def _run_batch(s):
    case, b, t = s["case"], s["batch"], s["t"]
    s["t"] = t + case["steps"]
    for k in range(case["steps"]):
        ts = [33 * (t + k)] * case["clips"]
        if case["source"] == "host":
            b.encode_step([f[k] for f in s["frames"]], ts)
        else:
            b.encode_step_device([f[k].data_ptr() for f in s["frames"]], ts)
    b.finish()
    return [w.take() for w in s["writers"]]


def _run_decode(s):
    case = s["case"]
    if not s["dec"].has_more_frames():
        s["dec"].close()
        s["dec"] = D.Decoder.new(s["stream"])
    if case["out"] == "rgb":
        return [s["dec"].decode_frame_rgb().rgb for _ in range(case["frames"])]
    got = [s["dec"].decode_frame() for _ in range(case["frames"])]
    return [[f.y, f.u, f.v] for f in got]


def _run_train(s):
    # learning rate 0, as a warm-up schedule begins: the weights stay, so every pass computes the
    # same gradients
    net = s["net"]
    loss = net.train_step(*s["data"], lr=0.0)
    return {"loss": loss, "grad": net.g}


def run(state):
    return {"live": _run_live, "clip": _run_clip, "batch": _run_batch, "decode": _run_decode,
            "train": _run_train}[state["case"]["kind"]](state)


# ---------------------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------------------

# integer multiply-adds of a macroblock's separable 16x16 and two 8x8 transforms, one direction
_TRANSFORM = 2 * (2 * 16 * 256 + 2 * 2 * 8 * 64)


def work(case):
    """Encoders: RGB read once (the records written are about a hundredth of it), the forward and
    inverse transforms of every macroblock.  Decoder: the frames written, the inverse
    transforms.  Training: records and weights read, gradients written; three products per
    multiply-add of the network."""
    kind = case["kind"]
    if kind == "train":
        n = case["n"]
        return {"bytes": n * (2 * 1152 + 2 * 32 + 5) + (P.NW * 2 + P.NB * 4) + (P.NW + P.NB) * 4,
                "flops": 3 * 2 * 888832 * n}
    sizes = _batch_sizes(case) if kind == "batch" else [(case["w"], case["h"])]
    reps = case["steps"] if kind == "batch" else case.get("frames", 1)
    mbs = sum(-(-w // 16) * -(-h // 16) for w, h in sizes)
    pixels = sum(w * h for w, h in sizes)
    if kind == "decode":
        out = 3 * pixels if case["out"] == "rgb" else 384 * mbs
        return {"bytes": reps * out, "flops": reps * mbs * _TRANSFORM}
    return {"bytes": reps * 3 * pixels, "flops": reps * 2 * mbs * _TRANSFORM}


# ---------------------------------------------------------------------------------------
# the training step in 64 bits
# ---------------------------------------------------------------------------------------

def exact(case, seed):
    """Encoders and decoders give bytes.  The training step: loss (summed over the records) and
    gradients of the mean loss by autograd in float64, in the parameters' layout."""
    if case["kind"] != "train":
        return None
    feat, x1, tmv, tskip = (t.double() for t in _records(case["n"], seed))
    n = case["n"]
    dev = feat.device
    p = torch.from_numpy(_params(seed + 2)).to(dev).double()
    par, o = {}, 0
    for name, rows, cols, _ in P.WEIGHTS:
        par[name] = p[o:o + rows * cols].reshape(rows, cols).clone().requires_grad_(True)
        o += rows * cols
    for name, k in P.BIASES:
        par[name] = p[o:o + k].clone().requires_grad_(True)
        o += k
    def conv(x, layer, stride):  # weights [out][tap][channel]
        cin = x.shape[1]
        pad = F.pad(x, (1, 1, 1, 1))
        ho = (x.shape[2] - 1) // stride + 1
        cols = [pad[:, :, ky:ky + stride * ho:stride, kx:kx + stride * ho:stride][:, :, :ho, :ho]
                for ky in range(3) for kx in range(3)]
        a = torch.stack(cols, 1).permute(0, 3, 4, 1, 2).reshape(n * ho * ho, 9 * cin)
        z = torch.relu(a @ par[f"w{layer}"][:, :9 * cin].T + par[f"b{layer}"])
        return z.reshape(n, ho, ho, 32).permute(0, 3, 1, 2)

    x = feat.permute(0, 3, 1, 2)
    for layer, stride in ((1, 2), (2, 2), (3, 1), (4, 2)):
        x = conv(x, layer, stride)
    f = torch.cat([x.permute(0, 2, 3, 1).reshape(n, 288), x1[:, 288:320]], 1)
    h1 = torch.relu(f @ par["f1"].T + par["bf1"])
    h2 = torch.relu(h1 @ par["f2"].T + par["bf2"])
    out = h2 @ par["f3"].T + par["bf3"]
    d = 1.0 / 32.0
    e = (out[:, :8].reshape(n, 4, 2) - (tmv / 32.0)[:, None]).abs()
    hub = torch.where(e < d, 0.5 * e * e / d, e - 0.5 * d).sum(2)
    best = F.one_hot(hub.argmin(1), 4).double()
    wgt = best + 0.05 * (1.0 - best)
    loss = (wgt * hub).sum() + 0.5 * F.binary_cross_entropy_with_logits(out[:, 8], tskip, reduction="sum")
    (loss / n).backward()
    names = [w[0] for w in P.WEIGHTS] + [b[0] for b in P.BIASES]
    grad = torch.cat([(par[k].grad if par[k].grad is not None else torch.zeros_like(par[k])).reshape(-1) for k in names])
    return {"loss": loss.detach().reshape(1), "grad": grad}

"""The work this framework is measured on: one case per way a program uses it.

The kinds follow the public entry points.

* ``deblock`` / ``sao`` / ``mc``: the standalone frame kernels
  (``tcb_deblock_frames``, ``tcb_sao_frames``, ``tcb_mc_frames``) on frames
  that are in device memory, as a pixel pipeline of its own calls them.
* ``frame``: one frame through the CTU engine (``tcb_ctu_encode_frame``),
  for programs that keep their own reference frames on the device.  Its
  references are the engine's own reconstructions of the frames before.
* ``clip``: a whole short clip from host memory to packets
  (``api.encode_sequence``): create the encoder, encode, drain, close.
  ``version`` 2 is the quadtree syntax, 0 and 1 the 8x8 block syntax that
  ``tc_config_defaults`` selects.
* ``batch``: one step of many streams that share every engine launch
  (``api.BatchEncoder.encode``), sources in device memory.  A step encodes
  the next frame of every stream, so passes on one state go on in time.
* ``decode``: a whole short clip of packets to pictures
  (``api.decode_sequence``).

Sizes are the benchmark's (320x240, 640x360, 1280x720, 1920x1080), qualities
its QPs 22 to 37; content is its generator's: sinusoids under a global
motion, moving rectangles of noise texture, and Gaussian noise.
"""
import ctypes
import math

import numpy as np
import torch

from tcodec_b200 import api

KEY, P, B = 0, 1, 2


def listed():
    return [
        # one small picture filtered: the smallest call, latency counts
        dict(name="deblock_1x320x240", kind="deblock", width=320, height=240, frames=1, qp=32),
        # in-loop filtering of many full-size pictures at once
        dict(name="sao_64x1920x1080", kind="sao", width=1920, height=1080, frames=64, qp=32),
        # prediction of a stack of pictures with a vector per block
        dict(name="mc_16x1280x720", kind="mc", width=1280, height=720, frames=16, field="random"),
        # a key frame: intra only
        dict(name="key_1280x720", kind="frame", width=1280, height=720, type=KEY, qp=27, preset=2, profile=1),
        # the two inter frame kinds of the headline configuration
        dict(name="p_1920x1080", kind="frame", width=1920, height=1080, type=P, qp=32, preset=2, profile=1),
        dict(name="b_1920x1080", kind="frame", width=1920, height=1080, type=B, qp=34, preset=2, profile=1),
        # short clips as a command-line encoder runs them: the small default,
        # a fast preset at an odd size, and hierarchical B frames
        dict(name="clip_320x240", kind="clip", width=320, height=240, frames=8, qp=32, preset=2, profile=0,
             b_frames=False, version=2),
        dict(name="clip_fast_1272x712", kind="clip", width=1272, height=712, frames=4, qp=37, preset=1, profile=0,
             b_frames=False, version=2),
        dict(name="clip_gop4b_640x360", kind="clip", width=640, height=360, frames=5, qp=22, preset=2, profile=1,
             b_frames=True, version=2),
        # the 8x8 block syntax, the library's default configuration
        dict(name="clip_v1_640x360", kind="clip", width=640, height=360, frames=4, qp=32, preset=2, profile=0,
             b_frames=False, version=1),
        # many full-size streams that advance together: the throughput form
        dict(name="batch_32x1920x1080", kind="batch", width=1920, height=1080, streams=32, qp=32, preset=2, profile=1),
        # playback
        dict(name="decode_1280x720", kind="decode", width=1280, height=720, frames=6, qp=27, preset=1, profile=0,
             b_frames=False, version=2),
    ]


def draw(rng):
    def size(lo, hi, step):
        return step * max(1, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi))) / step)))

    kind = rng.choice(["deblock", "sao", "mc", "frame", "frame", "clip", "clip", "clip", "batch", "decode"])
    qp = rng.randint(22, 37)
    if kind in ("deblock", "sao", "mc"):
        w = size(64, 1920, 2)
        h = size(max(64, w // 4), min(1080, w), 2)
        frames = max(1, min(64, int(64 * math.exp(rng.uniform(-4.2, 0.0)) * 1920 * 1080 / (w * h) / 4)))
        c = dict(kind=kind, width=w, height=h, frames=frames)
        c.update(dict(field=rng.choice(["global", "integer", "random"])) if kind == "mc" else dict(qp=qp))
        return c
    preset = rng.choice([0, 1, 2, 2, 2, 3])
    profile = rng.choice([0, 1])
    # whole 8x8 blocks, the unit every encoder form codes in
    w = size(96, 1920 if kind == "frame" else 960, 8)
    h = size(max(64, w // 3), min(1080, max(72, w * 2 // 3)), 8)
    if kind == "frame":
        return dict(kind=kind, width=w, height=h, type=rng.choice([KEY, P, P, B]), qp=qp, preset=preset,
                    profile=profile)
    if kind == "batch":
        streams = max(2, min(32, int(1920 * 1080 * 4 / (w * h) * rng.uniform(0.5, 2.0))))
        return dict(kind=kind, width=w, height=h, streams=streams, qp=qp, preset=preset, profile=profile)
    frames = max(2, min(8, int(640 * 360 * 6 / (w * h) * rng.uniform(0.5, 2.0))))
    return dict(kind=kind, width=w, height=h, frames=frames, qp=qp, preset=preset, profile=profile,
                b_frames=rng.random() < 0.4, version=rng.choice([2, 2, 1, 0]))


# ---------------------------------------------------------------- content

def _clip(width, height, n, seed):
    """n frames (y, cb, cr) of uint8 CUDA tensors: a sum of eight sinusoids
    moving by a global vector, 16 rectangles of noise texture with their own
    motion, and noise of standard deviation 3."""
    g = torch.Generator(device="cuda").manual_seed(int(seed))
    r = np.random.default_rng(int(seed))
    vx, vy = r.uniform(-4.0, 4.0), r.uniform(-2.0, 2.0)

    def waves():
        period, amp = r.uniform(8.0, 64.0, 8), r.uniform(10.0, 40.0, 8)
        theta, phase = r.uniform(0.0, math.pi, 8), r.uniform(0.0, 2 * math.pi, 8)
        k = 2 * math.pi / period
        return list(zip(k * np.cos(theta), k * np.sin(theta), phase, amp))

    planes = [(height, width, 1.0, waves()), (height // 2, width // 2, 0.5, waves()),
              (height // 2, width // 2, 0.5, waves())]
    rects = []
    for _ in range(16):
        rw, rh = (2 * (int(v) // 2) for v in r.integers(32, 161, 2))
        rw, rh = min(rw, width), min(rh, height)
        tex = [torch.randint(0, 256, (rh, rw), device="cuda", generator=g).float(),
               torch.randint(0, 256, (rh // 2, rw // 2), device="cuda", generator=g).float(),
               torch.randint(0, 256, (rh // 2, rw // 2), device="cuda", generator=g).float()]
        rects.append((rw, rh, r.uniform(0, width), r.uniform(0, height), r.uniform(-6, 6), r.uniform(-6, 6), tex))
    out = []
    for t in range(n):
        frame = []
        for i, (h, w, scale, ws) in enumerate(planes):
            y = (torch.arange(h, device="cuda", dtype=torch.float32) - vy * scale * t)[:, None]
            x = (torch.arange(w, device="cuda", dtype=torch.float32) - vx * scale * t)[None, :]
            p = torch.full((h, w), 128.0, device="cuda")
            for kx, ky, phase, amp in ws:
                p += float(amp) * torch.sin(float(kx) * x + float(ky) * y + float(phase))
            for rw, rh, x0, y0, rvx, rvy, tex in rects:
                px = int(x0 + rvx * t) % (width - rw + 1) // 2 * 2
                py = int(y0 + rvy * t) % (height - rh + 1) // 2 * 2
                q, s = tex[i], 1 if i == 0 else 2
                p[py // s:py // s + q.shape[0], px // s:px // s + q.shape[1]] = q
            p += 3.0 * torch.randn(h, w, device="cuda", generator=g)
            frame.append(p.round_().clamp_(0, 255).to(torch.uint8))
        out.append(tuple(frame))
    return out


def _host(clip):
    return [tuple(p.cpu().numpy() for p in f) for f in clip]


def _blocky(h, w, n, g):
    """Smooth content with steps at multiples of 4 samples and mild noise:
    what a block codec's reconstruction looks like before the loop filters."""
    cells = torch.randn(n, 1, -(-h // 32) + 2, -(-w // 32) + 2, device="cuda", generator=g)
    smooth = torch.nn.functional.interpolate(cells, size=(-(-h // 4), -(-w // 4)), mode="bilinear")
    p = 128 + 45 * smooth.repeat_interleave(4, 2).repeat_interleave(4, 3)[:, 0, :h, :w]
    p += 1.5 * torch.randn(n, h, w, device="cuda", generator=g)
    return p.round_().clamp_(0, 255).to(torch.uint8)


def _stream():
    return torch.cuda.current_stream().cuda_stream


# ---------------------------------------------------------------- kinds

def _prepare_filter(c, seed, lib):
    w, h, n = c["width"], c["height"], c["frames"]
    g = torch.Generator(device="cuda").manual_seed(int(seed))
    y, cb, cr = _blocky(h, w, n, g), _blocky(h // 2, w // 2, n, g), _blocky(h // 2, w // 2, n, g)
    src = (y.to(torch.int16) + torch.randint(-2, 5, (n, h, w), device="cuda", generator=g, dtype=torch.int16))
    src = src.clamp_(0, 255).to(torch.uint8)
    nctu = -(-w // 64) * -(-h // 64)
    params = torch.zeros(n, nctu, 3, dtype=torch.int16, device="cuda")
    desc = (api.FilterFrame * n)()
    for i, f in enumerate(desc):
        f.width, f.height, f.stride_y, f.stride_c, f.stride_src, f.qp = w, h, w, w // 2, w, c["qp"]
        f.y, f.cb, f.cr, f.src_y = y[i].data_ptr(), cb[i].data_ptr(), cr[i].data_ptr(), src[i].data_ptr()
        f.sao_params = params[i].data_ptr()
    fn = lib.tcb_deblock_frames if c["kind"] == "deblock" else lib.tcb_sao_frames
    out = (y, cb, cr) if c["kind"] == "deblock" else (y, params)
    return dict(fn=fn, desc=desc, n=n, out=out, keep=(cb, cr, src))


def _prepare_mc(c, seed, lib):
    w, h, n = c["width"], c["height"], c["frames"]
    g = torch.Generator(device="cuda").manual_seed(int(seed))
    base = _clip(w, h, 1, seed)[0]
    ref = [torch.stack([torch.roll(p, i, 1) for i in range(n)]) for p in base]
    pred = [torch.zeros_like(p) for p in ref]
    gw, gh = -(-w // 8), -(-h // 8)
    if c["field"] == "random":       # vectors within 24 samples, some far outside the picture
        mv = torch.randint(-96, 97, (n, gh, gw, 2), device="cuda", generator=g, dtype=torch.int16)
        far = torch.rand(n, gh, gw, 1, device="cuda", generator=g) < 0.01
        mv = torch.where(far, mv * 40, mv).to(torch.int16)
    elif c["field"] == "integer":    # whole samples
        mv = torch.randint(-16, 17, (n, gh, gw, 2), device="cuda", generator=g, dtype=torch.int16) * 4
    else:                            # one vector a picture
        mv = torch.randint(-32, 33, (n, 1, 1, 2), device="cuda", generator=g, dtype=torch.int16)
        mv = mv.expand(n, gh, gw, 2).contiguous()
    desc = (api.McFrame * n)()
    for i, f in enumerate(desc):
        f.width, f.height, f.stride_y, f.stride_c = w, h, w, w // 2
        f.ref_y, f.ref_cb, f.ref_cr = (p[i].data_ptr() for p in ref)
        f.pred_y, f.pred_cb, f.pred_cr = (p[i].data_ptr() for p in pred)
        f.mv = mv[i].data_ptr()
    return dict(fn=lib.tcb_mc_frames, desc=desc, n=n, out=tuple(pred), keep=(ref, mv))


class _Frame:
    """A caller's own frame loop on tcb_ctu_encode_frame: picture buffers,
    MV grids, decision records and scratch on the device."""

    def __init__(self, lib, c):
        self.lib, self.c = lib, c
        w, h = c["width"], c["height"]
        self.cells = -(-w // 8) * -(-h // 8)
        self.nctu = -(-w // 64) * -(-h // 64)
        self.scratch = torch.zeros(lib.tcb_ctu_scratch_bytes(w, h), dtype=torch.uint8, device="cuda")

    def describe(self, src, ftype, poc, refs, prev_grid):
        c, lib = self.c, self.lib
        w, h = c["width"], c["height"]
        rec = tuple(torch.zeros_like(p) for p in src)
        grid = torch.zeros(self.cells, lib.tcb_mv_cell_bytes(), dtype=torch.uint8, device="cuda")
        records = torch.zeros(self.nctu, lib.tcb_ctu_record_bytes(), dtype=torch.uint8, device="cuda")
        d = api.FrameDesc()
        d.width, d.height, d.stride_y, d.stride_c = w, h, w, w // 2
        d.src_y, d.src_cb, d.src_cr = (p.data_ptr() for p in src)
        d.rec_y, d.rec_cb, d.rec_cr = (p.data_ptr() for p in rec)
        for i, (r, ref_poc) in enumerate(refs):
            d.ref_y[i], d.ref_cb[i], d.ref_cr[i] = (p.data_ptr() for p in r)
            d.ref_poc[i] = ref_poc
        d.prev_mv_grid = None if prev_grid is None else prev_grid.data_ptr()
        d.cur_mv_grid, d.ctu_records = grid.data_ptr(), records.data_ptr()
        d.frame_type, d.poc, d.qp, d.preset, d.profile = ftype, poc, c["qp"], c["preset"], c["profile"]
        return dict(desc=d, rec=rec, grid=grid, records=records, keep=(src, refs, prev_grid))

    def encode(self, f):
        r = self.lib.tcb_ctu_encode_frame(ctypes.byref(f["desc"]), self.scratch.data_ptr(), self.scratch.numel(),
                                          _stream())
        if r != api.TC_OK:
            raise RuntimeError(f"tcb_ctu_encode_frame -> {r}")


def _prepare_frame(c, seed, lib):
    run = _Frame(lib, c)
    if c["type"] == KEY:
        clip = _clip(c["width"], c["height"], 1, seed)
        return dict(run=run, frame=run.describe(clip[0], KEY, 0, [], None))
    # P: frame 2 after the key frame and a P frame; B: frame 2 between the
    # key frame and the P frame of poc 4
    order = [0, 1, 2] if c["type"] == P else [0, 4, 2]
    clip = _clip(c["width"], c["height"], max(order) + 1, seed)
    refs, grid = [], None
    for i, poc in enumerate(order):
        f = run.describe(clip[poc], (KEY, P, c["type"])[i], poc, refs, grid)
        if i < 2:
            run.encode(f)
            refs, grid = [(f["rec"], poc)] + refs, f["grid"]
    return dict(run=run, frame=f)


def _config(lib, c):
    return api.make_config(lib, c["width"], c["height"], qp=c["qp"], preset=c["preset"], profile=c["profile"],
                           keyframe_interval=1000, b_frames=c.get("b_frames", False), version=c.get("version", 2))


def _prepare_batch(c, seed, lib):
    n, depth = c["streams"], 6
    clip = _clip(c["width"], c["height"], depth + n, seed)   # stream s shows the clip from frame s on
    enc = api.BatchEncoder(lib, [_config(lib, c) for _ in range(n)])
    w = c["width"]
    state = dict(enc=enc, n=n, depth=depth, t=0, clip=clip,
                 planes=[tuple((p.data_ptr(), w if i == 0 else w // 2) for i, p in enumerate(f)) for f in clip])
    torch.cuda.synchronize()    # the encoder works on a stream of its own
    _step(state)                # the key frames
    return state


def _step(s):
    k = s["t"] % (2 * s["depth"])
    k = min(k, 2 * s["depth"] - k)      # forwards, then backwards through the clip
    s["t"] += 1
    return s["enc"].encode([s["planes"][k + i] for i in range(s["n"])], on_device=True)


def prepare(case, seed):
    lib = api.bind_b200(api.load_library())
    kind = case["kind"]
    if kind in ("deblock", "sao"):
        s = _prepare_filter(case, seed, lib)
    elif kind == "mc":
        s = _prepare_mc(case, seed, lib)
    elif kind == "frame":
        s = _prepare_frame(case, seed, lib)
    elif kind == "batch":
        s = _prepare_batch(case, seed, lib)
    else:
        frames = _host(_clip(case["width"], case["height"], case["frames"], seed))
        s = dict(lib=lib, cfg=_config(lib, case), frames=frames)
        if kind == "decode":
            s = dict(lib=lib, packets=api.encode_sequence(lib, s["cfg"], frames))
    s["kind"] = kind
    if kind in ("batch", "clip"):       # room for a byte per sample, above what these qualities give
        pictures = case["streams"] if kind == "batch" else case["frames"]
        s["bytes"], s["used"] = np.zeros(3 * case["width"] * case["height"] // 2 * pictures, dtype=np.uint8), 0
    return s


def _packets(s, packets):
    """The packets one after the other in the state's buffer (zeros after the
    last), and their sizes."""
    at, sizes = 0, []
    for p in packets:
        n = len(p or b"")
        if n:
            s["bytes"][at:at + n] = np.frombuffer(p, dtype=np.uint8)
        at += n
        sizes.append(n)
    s["bytes"][at:s["used"]] = 0
    s["used"] = at
    return s["bytes"], np.array(sizes, dtype=np.int64)


def run(s):
    kind = s["kind"]
    if kind in ("deblock", "sao", "mc"):
        if s["fn"](s["desc"], s["n"], _stream()) != api.TC_OK:
            raise RuntimeError(kind)
        return s["out"]
    if kind == "frame":
        f = s["frame"]
        s["run"].encode(f)
        return dict(rec=f["rec"], grid=f["grid"], records=f["records"])
    if kind == "batch":
        return _packets(s, _step(s))
    if kind == "clip":
        return _packets(s, api.encode_sequence(s["lib"], s["cfg"], s["frames"]))
    return [p for f in api.decode_sequence(s["lib"], s["packets"]) for p in f]


def exact(case, seed):
    """Every output is whole numbers or bytes that the format fixes: there
    is no rounding to compare with a 64-bit value."""
    return None


# Integer operations per luma sample of one encoded frame, by what its
# preset scores: the transforms of every candidate (multiply-adds counted
# twice) and the searches' absolute differences (three operations each).
_CODED = {KEY: 7000.0, P: 10000.0, B: 8000.0}
_FAST = {KEY: 900.0, P: 1500.0, B: 1800.0}


def work(case):
    kind, px = case["kind"], case["width"] * case["height"]
    n = case.get("frames", 1)
    if kind == "deblock":     # every plane in and out; 30 operations per edge sample, every fourth sample each way
        return dict(bytes=3.0 * px * n, flops=20.0 * px * n)
    if kind == "sao":         # luma in and out and the source
        return dict(bytes=3.0 * px * n, flops=12.0 * px * n)
    if kind == "mc":          # reference in, prediction out, a vector per 8x8 block
        return dict(bytes=(3.0 + 4.0 / 64) * px * n, flops=40.0 * px * n)
    frame = 3.0 * px          # source in and reconstruction out, both 4:2:0
    if kind == "frame":
        ops = (_CODED if case["preset"] >= 2 else _FAST)[case["type"]]
        return dict(bytes=frame + (0, 1, 2)[case["type"]] * 1.5 * px, flops=ops * px)
    if kind == "batch":
        ops = (_CODED if case["preset"] >= 2 else _FAST)[P]
        return dict(bytes=(frame + 1.5 * px) * case["streams"], flops=ops * px * case["streams"])
    if kind == "decode":      # one reference in, the picture out, one inverse transform per sample
        return dict(bytes=frame * n, flops=40.0 * px * n)
    if case["version"] < 2:   # 18 modes, two searches of some 50 points, two transforms
        return dict(bytes=(frame + 1.5 * px) * n, flops=700.0 * px * n)
    table = _CODED if case["preset"] >= 2 else _FAST
    inter = B if case["b_frames"] else P
    return dict(bytes=(frame + 1.5 * px) * n, flops=(table[KEY] + table[inter] * (n - 1)) * px)

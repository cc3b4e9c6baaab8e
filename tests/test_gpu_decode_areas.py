"""Decoder reconstruction area by area: hand-written streams (raw Exp-Golomb
syntax, one 8x8 leaf) whose dequantised levels lie inside, at and far beyond
the range of the matrix form, against the transform's definition in 64-bit
integers; and clips whose leaves wait for one another in every way, against
the encoder's reconstruction.  Integers throughout: equality."""
import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

QSCALE = {10: 4, 11: 4, 32: 85, 33: 98, 50: 1024, 51: 1196}        # quantiser step by QP
JND = (6, 7, 8, 10)
ZIGZAG4 = [0, 1, 4, 8, 5, 2, 3, 6, 9, 12, 13, 10, 7, 11, 14, 15]


def zigzag(n):
    if n == 4:
        return ZIGZAG4
    order = sorted(((i, j) for i in range(8) for j in range(8)),
                   key=lambda p: (p[0] + p[1], p[0] if (p[0] + p[1]) % 2 else p[1]))
    return [8 * i + j for i, j in order]


class Bits:
    def __init__(self):
        self.s = ""

    def u(self, v, n):
        self.s += format(v, "0%db" % n)

    def ue(self, v):
        b = format(v + 1, "b")
        self.s += "0" * (len(b) - 1) + b

    def levels(self, lv, n):
        zz = zigzag(n)
        last = max((i for i in range(n * n) if lv.flat[zz[i]]), default=-1)
        self.ue(last + 1)
        for i in range(last, -1, -1):
            v = int(lv.flat[zz[i]])
            self.ue(abs(v))
            if v:
                self.u(v < 0, 1)

    def bytes(self):
        s = self.s + "0" * (-len(self.s) % 8) + "0" * 16
        return bytes(int(s[i:i + 8], 2) for i in range(0, len(s), 8))


def packet(size, qp, tu8, luma, chroma):
    b = Bits()
    for v, n in ((0x544356, 24), (2, 8), (size, 16), (size, 16), (0x80, 8), ((qp - 32) & 0xFF, 8), (1, 8), (0, 8),
                 (0, 16)):
        b.u(v, n)
    b.u(0, 1)                     # 8x8 leaf: not split, intra, DC, chroma DC
    b.u(1, 1)
    b.u(1, 5)
    b.u(0, 1)
    b.u(tu8, 1)
    if tu8:
        b.levels(luma, 8)
    else:
        for q in range(4):
            b.u(0, 1)
            b.levels(luma[4 * (q >> 1):4 * (q >> 1) + 4, 4 * (q & 1):4 * (q & 1) + 4], 4)
    for c in chroma:
        b.levels(c, 4)
    return b.bytes()


def int16(v):
    return (v + 32768) % 65536 - 32768


def picture(lv, qp):
    """Flat 128 plus the inverse transform of the levels."""
    n = lv.shape[0]
    m = np.array([[round(16384 * math.sqrt((1 if k == 0 else 2) / n) * math.cos((2 * x + 1) * k * math.pi / (2 * n)))
                   for x in range(n)] for k in range(n)], dtype=np.int64)
    pos = np.arange(n * n).reshape(n, n)
    band = (pos > 0).astype(int) + (pos >= n * n // 4) + (pos >= n * n // 2)
    eff = np.maximum((QSCALE[qp] * np.array(JND)[band] + 4) >> 3, 1)
    dq = int16(lv * eff + np.sign(lv) * (eff // 6))
    rows = (dq @ m + 8192) >> 14
    res = int16((m.T @ rows + 8192) >> 14)
    return np.clip(128 + res, 0, 255), np.abs(dq).max()


@pytest.mark.parametrize("size", [8, 10])
@pytest.mark.parametrize("tu8", [0, 1])
@pytest.mark.parametrize("qp,top", [(32, 40), (10, 900), (10, 1100), (10, 32767), (50, 32767)])
def test_levels_of_any_size(size, tu8, qp, top):
    from tcodec_b200 import api
    lib = api.bind_b200(api.load_library())
    assert zigzag(8)[:6] == [0, 1, 8, 16, 9, 2]
    rng = np.random.default_rng(qp + top + tu8)
    dec = api.Decoder(lib)
    peaks = []
    try:
        for _ in range(24):
            def draw(n):
                v = rng.integers(-top, top + 1, (n, n)) * (rng.random((n, n)) < rng.choice([0.05, 0.3, 1.0]))
                return v.astype(np.int64)
            luma, chroma = draw(8), [draw(4), draw(4)]
            got = dec.decode(packet(size, qp, tu8, luma, chroma))
            want = np.zeros((size, size), np.int64)          # beyond the last whole leaf: the frame's zeros
            if tu8:
                want[:8, :8], peak = picture(luma, qp)
                peaks.append(peak)
            else:
                for q in range(4):
                    s = np.s_[4 * (q >> 1):4 * (q >> 1) + 4, 4 * (q & 1):4 * (q & 1) + 4]
                    want[:8, :8][s], peak = picture(luma[s], qp)
                    peaks.append(peak)
            assert np.array_equal(got[0], want)
            for k in range(2):
                want = np.zeros((size // 2, size // 2), np.int64)
                want[:4, :4], _ = picture(chroma[k], qp + 1)
                assert np.array_equal(got[1 + k], want)
    finally:
        dec.close()
    assert (min(peaks) <= 4095) if top <= 900 else (max(peaks) > 4095)


@pytest.mark.parametrize("w,h", [(8, 8), (64, 64), (72, 136), (200, 120)])
@pytest.mark.parametrize("preset", [1, 3])
def test_clips_decode_to_the_encoders_pictures(w, h, preset):
    from tcodec_b200 import api, synth
    lib = api.load_library()
    rng = np.random.default_rng(w + h)
    frames = [tuple(np.clip(p.astype(int) + rng.integers(-20, 21, p.shape), 0, 255).astype(np.uint8) for p in f)
              for f in synth.moving_rects_clip(w, h, 5)]
    cfg = api.make_config(lib, w, h, qp=24, preset=preset, profile=1, keyframe_interval=1000)
    packets, recons = api.encode_sequence(lib, cfg, frames, with_recon=True)
    decoded = api.decode_sequence(lib, packets)
    assert len(decoded) == len(recons)
    for got, want in zip(decoded, recons):
        for k in range(3):
            assert np.array_equal(got[k], want[k]), k

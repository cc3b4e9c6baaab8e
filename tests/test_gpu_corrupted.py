"""Corrupted v2 and legacy streams without a build of the reference: flipped
bits, garbage, cut packets, pictures that change size and packets of other
streams in between.  Every call returns (a picture, a wait for reordering, or
an error code), the decoder stays usable, and the clean stream decodes to the
encoder's pictures on it afterwards.  (Each mutation's exact outcome is
compared with the reference decoder in test_gpu_fuzz.py; which memory the
kernel may touch is checked on the CPU in test_decoder_host.py.)"""
import random

import numpy as np
import pytest

from tests.test_gpu_fuzz import mutate

pytestmark = pytest.mark.gpu

SPECS = [dict(w=96, h=80, n=4, qp=32, preset=2, profile=1), dict(w=128, h=64, n=4, qp=24, preset=2, profile=0, entropy=False, crc=True),
         dict(w=128, h=96, n=6, qp=32, preset=2, profile=1, b_frames=True), dict(w=72, h=136, n=4, qp=20, preset=0, profile=0),
         dict(w=100, h=60, n=4, qp=30, preset=3, profile=1, keyframe_interval=2),
         dict(w=96, h=80, n=4, qp=30, preset=2, profile=1, version=1, entropy=True),
         dict(w=96, h=80, n=4, qp=30, preset=2, profile=1, version=0, entropy=False)]
OTHER = (48, 16, 200, 136)       # sizes a mutated header may announce: all allocations stay small
TRIALS = 60


@pytest.fixture(scope="module")
def lib():
    from tcodec_b200 import api
    return api.load_library()


def _streams(lib):
    from tcodec_b200 import api, synth
    out = []
    for s in SPECS:
        kw = {k: v for k, v in s.items() if k not in ("w", "h", "n")}
        kw.setdefault("keyframe_interval", 1000)
        out.append(api.encode_sequence(lib, api.make_config(lib, s["w"], s["h"], **kw),
                                       synth.moving_rects_clip(s["w"], s["h"], s["n"])))
    return out


def _feed(dec, packet):
    try:
        dec.decode(packet)
    except RuntimeError as e:
        assert e.args[0] == "tc_decoder_decode" and e.args[1] < 0
        return False
    return True


@pytest.mark.parametrize("si", range(len(SPECS)))
def test_every_call_returns_and_the_decoder_stays_usable(lib, si):
    from tcodec_b200 import api
    streams = _streams(lib)
    packets = streams[si]
    want = api.decode_sequence(lib, packets)
    rng = random.Random(si)
    dec = api.Decoder(lib)
    errors = pictures = 0
    try:
        for trial in range(TRIALS):
            k = rng.randrange(len(packets))
            for t, p in enumerate(packets):
                if t == k:
                    p, _ = mutate(rng, p)
                    p = bytearray(p)
                    if len(p) > 8:      # version and magic stay; sizes are the stream's or one of a few others
                        p[:4] = packets[t][:4]
                        p[4:8] = packets[t][4:8]
                        if rng.random() < 0.25:
                            a, b = rng.choice(OTHER), rng.choice(OTHER)
                            p[4:8] = bytes([a >> 8, a & 255, b >> 8, b & 255])
                    p = bytes(p)
                elif rng.random() < 0.05:       # a packet of another stream
                    _feed(dec, rng.choice(rng.choice(streams)))
                ok = _feed(dec, p)
                errors, pictures = errors + (not ok), pictures + ok
        dec.flush()
        assert pictures > TRIALS
        if SPECS[si].get("version", 2) == 2:      # (a legacy frame's blocks parse whatever the bits are)
            assert errors > 0
    finally:
        dec.close()
    # a fresh decoder, and the context, are sound
    got = api.decode_sequence(lib, packets)
    assert len(got) == len(want)
    for a, b in zip(got, want):
        for c in range(3):
            assert np.array_equal(a[c], b[c])


def test_the_used_decoder_still_decodes_the_clean_stream(lib):
    """From a key frame that clears the references on, a decoder that has seen
    corrupted packets gives the same pictures as a fresh one."""
    from tcodec_b200 import api, synth
    w, h = 96, 80
    packets = api.encode_sequence(lib, api.make_config(lib, w, h, qp=28, preset=2, profile=1, keyframe_interval=4),
                                  synth.moving_rects_clip(w, h, 8))
    want = api.decode_sequence(lib, packets)
    rng = random.Random(9)
    for _ in range(20):
        dec = api.Decoder(lib)
        try:
            for p in packets[:4]:
                bad = bytearray(mutate(rng, p)[0])
                if len(bad) > 8:
                    bad[:8] = p[:8]
                _feed(dec, bytes(bad))
            for t in range(4, 8):
                got = dec.decode(packets[t])
                for c in range(3):
                    assert np.array_equal(got[c], want[t][c]), (t, c)
        finally:
            dec.close()

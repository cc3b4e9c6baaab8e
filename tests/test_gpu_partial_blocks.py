"""Frame sizes that are not multiples of 8.  Samples outside whole 8x8 blocks
are never coded: encoder and decoder keep the previous picture's there (zero
before the first) and apply SAO to them, and searches and predictions of later
frames read them.  So the same input must give the same packets every time,
alone and in a batch, and the decoder's pictures must equal the encoder's
reconstructions in every sample."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _clip(w, h, n):
    from tcodec_b200 import synth
    rng = np.random.default_rng(w * h)
    return [tuple(np.clip(p.astype(int) + rng.integers(-8, 9, p.shape), 0, 255).astype(np.uint8) for p in f)
            for f in synth.moving_rects_clip(w, h, n)]


def _encode(lib, cfg, frames):
    """Packets, and the reconstruction by picture number."""
    from tcodec_b200 import api
    enc = api.Encoder(lib, cfg)
    packets, recon = [], {}
    try:
        for f in frames:
            p = enc.encode(*f)
            if p is not None:
                packets.append(p)
                recon[p[10]] = enc.recon()
        packets.extend(enc.flush())
    finally:
        enc.close()
    return packets, recon


@pytest.mark.parametrize("w,h", [(100, 60), (66, 130), (70, 64), (64, 78), (334, 190)])
@pytest.mark.parametrize("preset,b_frames,interval", [(0, False, 1000), (1, False, 1000), (2, False, 1000), (2, True, 1000),
                                                      (3, False, 2)])
def test_partial_blocks_are_kept_alike(w, h, preset, b_frames, interval):
    from tcodec_b200 import api
    lib = api.load_library()
    frames = _clip(w, h, 6)
    cfg = lambda: api.make_config(lib, w, h, qp=26, preset=preset, profile=1, keyframe_interval=interval, b_frames=b_frames)
    packets, recon = _encode(lib, cfg(), frames)
    assert _encode(lib, cfg(), frames)[0] == packets
    decoded = api.decode_sequence(lib, packets)
    assert len(decoded) == 6
    for poc, want in recon.items():
        for k in range(3):
            assert np.array_equal(decoded[poc][k], want[k]), (poc, k)
    batch = api.BatchEncoder(lib, [cfg() for _ in range(3)])
    got = [[] for _ in range(3)]
    try:
        for f in frames:
            for g, p in zip(got, batch.encode([f] * 3)):
                if p is not None:
                    g.append(p)
        for g, t in zip(got, batch.flush()):
            g.extend(t)
    finally:
        batch.close()
    assert got == [packets] * 3

"""The GPU's legacy (v0 / v1) block encoder against its CPU restatement, which
test_legacy_cpu.py holds to the reference: every packet (modes, vectors,
levels) and every sample of the reconstruction, at sizes with missing and
partial blocks, extreme quantisers and content, two searched references and
hierarchical B frames.  Whole numbers: equality."""
import numpy as np
import pytest

from tests import legacy_restate as lr

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def restate(tmp_path_factory):
    return lr.build(tmp_path_factory.mktemp("restate"))


def _clip(kind, w, h, n):
    from tcodec_b200 import synth
    rng = np.random.default_rng(w * h + n)
    if kind == "moving":
        return [tuple(np.clip(p.astype(int) + rng.integers(-10, 11, p.shape), 0, 255).astype(np.uint8) for p in f)
                for f in synth.moving_rects_clip(w, h, n)]
    shapes = ((h, w), (h // 2, w // 2), (h // 2, w // 2))
    if kind == "saturated":
        return [tuple(np.where(rng.random(s) < 0.5, 0, 255).astype(np.uint8) for s in shapes) for _ in range(n)]
    still = [rng.integers(60, 200, (-(-s[0] // 8), -(-s[1] // 8))).repeat(8, 0).repeat(8, 1)[:s[0], :s[1]] for s in shapes]
    return [tuple(np.clip(p + rng.integers(0, 2, p.shape), 0, 255).astype(np.uint8) for p in still) for _ in range(n)]


@pytest.mark.parametrize("w,h", [(8, 8), (64, 64), (100, 60), (72, 136), (202, 138)])
@pytest.mark.parametrize("version,preset,profile,qp,entropy,b_frames,kind", [
    (0, 2, 0, 28, False, False, "moving"), (1, 0, 0, 12, False, False, "moving"), (1, 1, 1, 40, True, False, "moving"),
    (1, 3, 1, 26, False, False, "moving"), (1, 2, 1, 30, True, True, "moving"), (1, 3, 1, 22, False, True, "moving"),
    (1, 2, 1, 10, False, False, "saturated"), (1, 2, 1, 51, True, True, "saturated"), (1, 2, 1, 63, False, False, "saturated"),
    (1, 2, 1, 24, False, True, "still"), (0, 3, 1, 45, False, False, "still")])
def test_packets_and_pictures_equal_the_restatement(restate, w, h, version, preset, profile, qp, entropy, b_frames, kind):
    from tcodec_b200 import api
    lib = api.load_library()
    frames = _clip(kind, w, h, 6)
    enc = api.Encoder(lib, api.make_config(lib, w, h, qp=qp, preset=preset, profile=profile, keyframe_interval=1000,
                                           version=version, entropy=entropy, b_frames=b_frames))
    ref = lr.Restated(restate, w, h, preset, profile, version, entropy)
    try:
        def check(packet, recon):
            frame_type, q, poc = lr.header(packet, b_frames)
            want, planes = ref.frame(frames[poc], frame_type, q, poc, b_frames)
            assert packet == want, (frame_type, poc)
            if recon is not None:
                for k in range(3):
                    assert np.array_equal(recon[k], planes[k]), (frame_type, poc, k)
        for f in frames:
            p = enc.encode(*f)
            if p is not None:
                check(p, enc.recon())
        for p in enc.flush():
            check(p, None)
    finally:
        enc.close()
        ref.close()

"""Legacy (v0 / v1) streams at the edges of their kernels: CTUs with missing
blocks, single blocks, extreme quantisers and every preset; the decoder's
pictures must equal the encoder's reconstructions, which come from another
kernel with other transforms (integers: equality)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("w,h", [(8, 8), (64, 64), (72, 40), (136, 200)])
@pytest.mark.parametrize("version,preset,qp", [(0, 2, 28), (1, 0, 40), (1, 1, 16), (1, 3, 30)])
def test_legacy_clips_decode_to_the_encoders_pictures(w, h, version, preset, qp):
    from tcodec_b200 import api, synth
    lib = api.load_library()
    rng = np.random.default_rng(w + h + qp)
    frames = [tuple(np.clip(p.astype(int) + rng.integers(-12, 13, p.shape), 0, 255).astype(np.uint8) for p in f)
              for f in synth.moving_rects_clip(w, h, 4)]
    cfg = api.make_config(lib, w, h, qp=qp, preset=preset, profile=1, keyframe_interval=1000, version=version,
                          entropy=version > 0)    # a v0 header cannot announce range coding
    packets, recons = api.encode_sequence(lib, cfg, frames, with_recon=True)
    decoded = api.decode_sequence(lib, packets)
    assert len(decoded) == len(recons) == 4
    for got, want in zip(decoded, recons):
        for k in range(3):
            assert np.array_equal(got[k], want[k]), k

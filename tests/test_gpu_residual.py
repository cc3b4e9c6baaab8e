"""The encoder's residual path at the ends of its ranges: saturated
residuals (0 against 255), flat pictures, and quantiser steps from 1 (level =
coefficient) to above every coefficient, with leaves of every size and both
TU sizes.  The decoder rebuilds every picture from the packets, so its pictures
must equal the encoder's reconstructions sample for sample (its transforms
are checked against 64-bit integers in test_gpu_decode_areas.py)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _content(kind, rng, h, w, t):
    yy, xx = np.mgrid[0:h, 0:w]
    if kind == "saturated":          # noise of the two extreme values
        return np.where(rng.random((h, w)) < 0.5, 0, 255).astype(np.uint8)
    if kind == "stripes":            # every transform basis' largest gain in one direction, moving
        return np.where(((xx + 3 * t) // 2 + yy // 4) % 2, 255, 0).astype(np.uint8)
    return np.full((h, w), 255 * (t & 1), np.uint8)     # flat, jumping between the extremes


QPS = [(0, 2), (5, 3), (22, 2), (37, 1), (51, 2), (63, 2)]
# (saturated noise at QP 0 codes to more than the encoder's packet buffer
# holds and is refused with TC_ERR_MEMORY)
CASES = [(kind, qp, preset) for kind in ("saturated", "stripes", "flat") for qp, preset in QPS
         if not (kind == "saturated" and qp == 0)]


@pytest.mark.parametrize("kind,qp,preset", CASES)
def test_residual_extremes_decode_to_the_encoders_picture(kind, qp, preset):
    from tcodec_b200 import api
    lib = api.load_library()
    rng = np.random.default_rng(qp)
    w, h = 136, 72                   # whole and partial CTUs
    frames = [tuple(_content(kind, rng, hh, ww, t) for hh, ww in ((h, w), (h // 2, w // 2), (h // 2, w // 2)))
              for t in range(3)]
    cfg = api.make_config(lib, w, h, qp=qp, preset=preset, profile=1, keyframe_interval=1000)
    packets, recons = api.encode_sequence(lib, cfg, frames, with_recon=True)
    decoded = api.decode_sequence(lib, packets)
    assert len(decoded) == len(recons) == 3
    for t, (got, want) in enumerate(zip(decoded, recons)):
        for k in range(3):
            assert np.array_equal(got[k], want[k]), (t, k)


@pytest.mark.parametrize("w,h", [(64, 64), (72, 72), (200, 136)])
def test_skipped_leaves_leave_no_gap_in_the_record(w, h):
    """Half of each picture is the previous reconstruction (exact skips), the
    other half changes: the levels of the coded leaves, placed in z-order,
    must close up over the skipped ones."""
    from tcodec_b200 import api, synth
    lib = api.load_library()
    frames = synth.moving_rects_clip(w, h, 4)
    enc = api.Encoder(lib, api.make_config(lib, w, h, qp=27, preset=2, profile=1, keyframe_interval=1000))
    packets, recons = [], []
    try:
        for t, f in enumerate(frames):
            if t:
                f = tuple(np.where(np.arange(p.shape[1])[None, :] < p.shape[1] // 2, r, p)
                          for p, r in zip(f, recons[-1]))
            packets.append(enc.encode(*f))
            recons.append(enc.recon())
    finally:
        enc.close()
    for t, (got, want) in enumerate(zip(api.decode_sequence(lib, packets), recons)):
        for k in range(3):
            assert np.array_equal(got[k], want[k]), (t, k)

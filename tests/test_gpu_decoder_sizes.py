"""Streams whose pictures change size, and decoders created for another size:
every picture equals that of a decoder which sees only that size (in the part
both have; a caller reads the size tc_decoder_get_info gives, and what lies
beyond a smaller picture is empty).  Which rows the kernel may touch is
checked on the CPU in test_decoder_host.py."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def clip(lib, w, h, version):
    from tcodec_b200 import api, synth
    cfg = api.make_config(lib, w, h, qp=26, preset=2, profile=1, keyframe_interval=1000, version=version)
    return api.encode_sequence(lib, cfg, synth.moving_rects_clip(w, h, 3))


@pytest.mark.parametrize("version", [2, 1])
@pytest.mark.parametrize("created", [(0, 0), (72, 40), (95, 79), (320, 200)])
def test_each_size_decodes_as_alone(created, version):
    from tcodec_b200 import api
    lib = api.load_library()
    dec = api.Decoder(lib, *created)
    W, H = None, None
    try:
        for w, h in ((96, 80), (96, 16), (200, 136), (64, 64), (96, 80)):
            packets = clip(lib, w, h, version)
            want = api.decode_sequence(lib, packets)
            assert len(want) == 3
            if W is None:
                W, H = created if created[0] else (w, h)
            for p, planes in zip(packets, want):
                got = dec.decode(p)
                for k, (g, full) in enumerate(zip(got, planes)):
                    exp = np.zeros((H, W) if k == 0 else (H // 2, W // 2), np.uint8)
                    part = full[:exp.shape[0], :exp.shape[1]]
                    exp[:part.shape[0], :part.shape[1]] = part
                    assert np.array_equal(g, exp), (w, h, k)
    finally:
        dec.close()

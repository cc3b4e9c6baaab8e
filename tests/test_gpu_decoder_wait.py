"""Failure detection in the decoder's kernel, without a GPU fault: with the
test hook the first area of every CTU never counts as done, so the intra areas
that read it give up waiting (bounded by tcb_set_neighbor_wait_limit).  The
packet is TC_ERR_INTERNAL and leaves no trace: given again it decodes, and so
does the rest of the stream.  What the host does with the status is checked
on the CPU in test_decoder_host.py."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("w,h", [(64, 64), (136, 72)])
@pytest.mark.parametrize("lost", [0, 1, 5])
def test_a_lost_area_is_reported_and_the_stream_goes_on(w, h, lost):
    from tcodec_b200 import api
    lib = api.bind_b200(api.load_library())
    rng = np.random.default_rng(w)
    # Dark and bright ramps in turn at the preset whose leaves are all 8x8: no
    # frame predicts the next, so every leaf is intra and reads the ones before.
    def plane(h, w, t):
        yy, xx = np.mgrid[0:h, 0:w]
        return (160 * (t & 1) + (xx + yy) * 60 // (w + h) + rng.integers(0, 5, (h, w))).astype(np.uint8)
    frames = [(plane(h, w, t), plane(h // 2, w // 2, t), plane(h // 2, w // 2, t)) for t in range(7)]
    packets = api.encode_sequence(lib, api.make_config(lib, w, h, qp=30, preset=0, profile=1, keyframe_interval=1000),
                                  frames)
    want = api.decode_sequence(lib, packets)
    default = ctypes.c_longlong()
    assert lib.tcb_get_neighbor_wait_limit(ctypes.byref(default)) == api.TC_OK
    assert lib.tcb_debug_decoder_lose_area(None) == api.TC_ERR_PARAM
    dec = api.Decoder(lib)
    try:
        for t, p in enumerate(packets):
            if t == lost:
                try:
                    assert lib.tcb_set_neighbor_wait_limit(1 << 10) == api.TC_OK
                    assert lib.tcb_debug_decoder_lose_area(dec.h) == api.TC_OK
                    with pytest.raises(RuntimeError) as e:
                        dec.decode(p)
                    assert e.value.args[1] == api.TC_ERR_INTERNAL
                finally:
                    assert lib.tcb_set_neighbor_wait_limit(default.value) == api.TC_OK
            got = dec.decode(p)
            for k in range(3):
                assert np.array_equal(got[k], want[t][k]), (t, k)
    finally:
        dec.close()

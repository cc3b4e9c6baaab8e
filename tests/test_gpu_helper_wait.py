"""Failure detection in a CTU's helper CTAs, without a GPU fault: with the test
hook one helper leaves at a given command without an answer (the CTU's own
command, the first leaf's, a later leaf's).  The wait for it is bounded by
tcb_set_neighbor_wait_limit and runs out once; the frame is finished without
helpers, tcb_ctu_frame_result reports TC_ERR_INTERNAL, and the same process
then encodes the same frames with the usual output."""
import ctypes
import time

import numpy as np
import pytest

from tests import ctu_frames

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("commands", [1, 2, 9])
@pytest.mark.parametrize("frame", [0, 1])                # intra only; four searches
def test_a_helper_that_leaves_is_reported_and_the_context_survives(commands, frame):
    import torch
    from tcodec_b200 import api
    lib = api.bind_b200(api.load_library())
    name, frames, qp, preset, profile = ctu_frames.clips()[1]
    assert preset >= 2
    frames = frames[:2]
    h, w = frames[0][0].shape
    nbytes = lib.tcb_ctu_scratch_bytes(w, h)
    scratch = torch.empty(nbytes, dtype=torch.uint8, device="cuda")
    st = torch.cuda.current_stream().cuda_stream

    def whole(desc):
        return lib.tcb_ctu_encode_frame(desc, scratch.data_ptr(), nbytes, st)

    def quitting(desc):
        return lib.tcb_debug_ctu_encode_frame_helper_quits(desc, scratch.data_ptr(), nbytes, st, commands)

    want = ctu_frames.FrameRun(lib, frames, qp, preset, profile, whole).run()
    default = ctypes.c_longlong()
    assert lib.tcb_get_neighbor_wait_limit(ctypes.byref(default)) == api.TC_OK
    run = ctu_frames.FrameRun(lib, frames, qp, preset, profile, whole)
    for t in range(frame):
        run.step(t)
    assert lib.tcb_debug_ctu_encode_frame_helper_quits(None, scratch.data_ptr(), nbytes, st, commands) == api.TC_ERR_PARAM
    try:
        # some milliseconds of polling, then 4,096 sleeps of at most 1,024 ns
        assert lib.tcb_set_neighbor_wait_limit(1 << 12) == api.TC_OK
        run.call = quitting
        t0 = time.perf_counter()
        run.step(frame)
        assert lib.tcb_ctu_frame_result(scratch.data_ptr(), st) == api.TC_ERR_INTERNAL
        elapsed = time.perf_counter() - t0
        print(f"lost helper reported after {elapsed * 1e3:.1f} ms")
        assert elapsed < 2.0
    finally:
        assert lib.tcb_set_neighbor_wait_limit(default.value) == api.TC_OK
    got = ctu_frames.FrameRun(lib, frames, qp, preset, profile, whole).run()
    assert lib.tcb_ctu_frame_result(scratch.data_ptr(), st) == api.TC_OK
    for t in range(2):
        for k, what in enumerate(("y", "cb", "cr", "records", "mv grid")):
            assert np.array_equal(got[t][k], want[t][k]), (t, what)

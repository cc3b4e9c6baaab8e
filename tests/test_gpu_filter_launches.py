"""Launch forms of the frame filters at their edges, bit-exact against the oracle: groups of one size (3D grid) and of mixed
sizes, one CTU up to more CTUs than SMs (the fine and the coarse deblocking
items), more frames than one launch holds, and planes at every byte offset
(the word loads and the store widths)."""
import numpy as np
import pytest

from tcodec_b200.api import FilterFrame
from tests import test_gpu_filters as tf

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def lib():
    from tcodec_b200 import api
    return api.bind_b200(api.load_library())


def check(lib, cases):
    got = tf.run(lib, lib.tcb_deblock_frames, cases)
    for c, g in zip(cases, got):
        y, cb, cr = tf.oracle_deblock(c)
        assert np.array_equal(g["y"], y) and np.array_equal(g["cb"], cb) and np.array_equal(g["cr"], cr)
    got = tf.run(lib, lib.tcb_sao_frames, cases)
    for c, g in zip(cases, got):
        y, params = tf.oracle_sao(c)
        assert np.array_equal(g["params"], params) and np.array_equal(g["y"], y)


@pytest.mark.parametrize("sizes", [[(64, 64)], [(832, 704)], [(832, 768)], [(64, 64), (128, 64)], [(130, 70)] * 3,
                                   [(64, 64)] * 65, [(64, 64)] * 64 + [(66, 130)]])
def test_groups(lib, sizes):
    rng = np.random.default_rng(len(sizes))
    check(lib, [tf.make_case(rng, w, h, 24 + i % 20, 0) for i, (w, h) in enumerate(sizes)])


@pytest.mark.parametrize("offset", [0, 1, 2, 3, 4, 7, 8, 13])
@pytest.mark.parametrize("pad", [0, 1, 2, 5])
def test_planes_at_any_offset(lib, offset, pad):
    import torch
    rng = np.random.default_rng(10 * offset + pad)
    w, h, qp = 192, 128, 36
    c = tf.make_case(rng, w, h, qp, 0)
    bufs, f = {}, (FilterFrame * 1)()
    for k in ("y", "cb", "cr", "src"):
        hh, ww = c[k].shape
        rows = np.full((hh, ww + pad), 77, np.uint8)
        rows[:, :ww] = c[k]
        bufs[k] = torch.full((offset + rows.size + 16,), 77, dtype=torch.uint8, device="cuda")
        bufs[k][offset:offset + rows.size] = torch.from_numpy(rows.ravel()).cuda()
    f[0].width, f[0].height, f[0].qp = w, h, qp
    f[0].stride_y, f[0].stride_c, f[0].stride_src = w + pad, w // 2 + pad, w + pad
    f[0].y, f[0].cb, f[0].cr, f[0].src_y = (bufs[k].data_ptr() + offset for k in ("y", "cb", "cr", "src"))
    st = torch.cuda.current_stream().cuda_stream
    assert lib.tcb_deblock_frames(f, 1, st) == 0 and lib.tcb_sao_frames(f, 1, st) == 0
    torch.cuda.synchronize()
    c["y"], c["cb"], c["cr"] = tf.oracle_deblock(c)
    c["y"], _ = tf.oracle_sao(c)
    for k in ("y", "cb", "cr"):
        hh, ww = c[k].shape
        want = np.full(bufs[k].numel(), 77, np.uint8)       # nothing outside the planes is written
        rows = np.full((hh, ww + pad), 77, np.uint8)
        rows[:, :ww] = c[k]
        want[offset:offset + rows.size] = rows.ravel()
        assert np.array_equal(bufs[k].cpu().numpy(), want), k

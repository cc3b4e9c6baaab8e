"""Motion compensation where its forms meet, bit-exact against the oracle:
vectors that put the six-tap and bilinear supports on, across and far beyond
every frame edge, few and many edge blocks per CTA (sample by sample, row by
row), every quarter phase, strides of every remainder, frames smaller than the
support, and more frames than one launch holds."""
import numpy as np
import pytest

from tests import test_gpu_mc as tm

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def lib():
    from tcodec_b200 import api
    return tm.bind(api.load_library())


def check(lib, cases):
    for c, got in zip(cases, tm.run_gpu(lib, cases)):
        for g, want, half in zip(got, tm.run_oracle(c), (1, 2, 2)):
            assert np.array_equal(g[:c["h"] // half, :c["w"] // half], want), (c["w"], c["h"], c["pad"])


@pytest.mark.parametrize("w,h", [(2, 2), (8, 8), (10, 12), (64, 8), (512, 16), (136, 72)])
@pytest.mark.parametrize("pad", [0, 1, 2, 3])
def test_edges_and_phases(lib, w, h, pad):
    rng = np.random.default_rng(w + h + pad)
    cases = []
    for reach in (16, 4 * max(w, h)):
        c = tm.make_case(rng, w, h, pad, "random")
        c["mv"] = rng.integers(-reach, reach + 1, c["mv"].shape).astype(np.int16)
        for k in ("y", "cb", "cr"):
            c[k] = rng.integers(0, 256, c[k].shape).astype(np.uint8)
        cases.append(c)
    check(lib, cases)


@pytest.mark.parametrize("phase", range(16))
def test_one_phase_everywhere(lib, phase):
    rng = np.random.default_rng(phase)
    c = tm.make_case(rng, 272, 48, phase & 3, "global")
    c["mv"][:] = (phase & 3, phase >> 2)
    check(lib, [c])


def test_more_frames_than_a_launch(lib):
    rng = np.random.default_rng(3)
    check(lib, [tm.make_case(rng, 24, 16, i & 3, "random") for i in range(67)])

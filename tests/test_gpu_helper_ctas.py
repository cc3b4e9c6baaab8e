"""The CTU engine with and without helper CTAs: the same streams encoded alone
(a cluster of four CTAs per CTU), in batches whose CTUs in work leave room for
one helper each, and in batches that fill the GPU (single CTAs) must give the
same packets, whatever the picture's shape, preset and GOP; and a batch in
which only some streams make use of helpers."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _clip(w, h, n, seed):
    from tcodec_b200 import synth
    rng = np.random.default_rng(seed)
    return [tuple(np.clip(p.astype(int) + rng.integers(-6, 7, p.shape), 0, 255).astype(np.uint8) for p in f)
            for f in synth.moving_rects_clip(w, h, n)]


def _batch(lib, cfgs, clips):
    from tcodec_b200 import api
    batch = api.BatchEncoder(lib, cfgs)
    got = [[] for _ in cfgs]
    try:
        for frames in zip(*clips):
            for g, p in zip(got, batch.encode(list(frames))):
                if p is not None:
                    g.append(p)
        for g, t in zip(got, batch.flush()):
            g.extend(t)
    finally:
        batch.close()
    return got


# (streams x CTUs in work): 148 SMs hold clusters of four up to 37, of two up to 74
@pytest.mark.parametrize("w,h,many", [(320, 256, (10, 20)), (328, 200, (10, 20)), (64, 192, (38, 75)), (192, 72, (19, 38))])
@pytest.mark.parametrize("preset,b_frames", [(2, True), (3, False)])
def test_batches_of_any_size_give_the_single_streams_packets(w, h, many, preset, b_frames):
    from tcodec_b200 import api
    lib = api.load_library()
    clip = _clip(w, h, 4, w + h)
    cfg = lambda: api.make_config(lib, w, h, qp=28, preset=preset, profile=1, keyframe_interval=1000, b_frames=b_frames)
    want = api.encode_sequence(lib, cfg(), clip)
    for n in many:
        for got in _batch(lib, [cfg() for _ in range(n)], [clip] * n):
            assert got == want


def test_mixed_presets_share_a_clustered_launch():
    from tcodec_b200 import api
    lib = api.load_library()
    shapes = [(128, 128, 2), (192, 72, 0), (72, 136, 3), (136, 64, 1)]
    clips = [_clip(w, h, 3, w) for w, h, _ in shapes]
    cfgs = [api.make_config(lib, w, h, qp=30, preset=p, profile=1, keyframe_interval=1000) for w, h, p in shapes]
    for got, cfg, clip in zip(_batch(lib, cfgs, clips), cfgs, clips):
        assert got == api.encode_sequence(lib, cfg, clip)


def test_replayed_graphs_follow_the_cluster_size():
    """Steps with the same nodes whose streams ask for clusters in one step and
    for single CTAs in the next."""
    from tcodec_b200 import api
    lib = api.load_library()
    shapes = [(128, 128, 2), (128, 128, 0), (320, 256, 2)]
    clips = [_clip(w, h, 4, w) for w, h, _ in shapes]
    cfgs = [api.make_config(lib, w, h, qp=30, preset=p, profile=0, keyframe_interval=1) for w, h, p in shapes]
    batch = api.BatchEncoder(lib, cfgs)
    batch.set_graphs(True)
    got = [[] for _ in cfgs]
    try:
        for t in range(4):
            for turn in range(3):
                packets = batch.encode([clips[i][t] if i == turn else None for i in range(3)])
                got[turn].append(packets[turn])
    finally:
        batch.close()
    for g, cfg, clip in zip(got, cfgs, clips):
        assert g == api.encode_sequence(lib, cfg, clip)

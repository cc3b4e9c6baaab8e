"""The legacy encoder's CPU restatement against the reference's 72 v0 / v1 /
v1e conformance hashes, without a build of the reference (test_legacy_cpu.py
compares whole sequences where there is one; test_gpu_legacy_blocks.py holds
the GPU encoder to it)."""
import hashlib
import struct

import numpy as np

from tests import legacy_restate as lr
from tests.golden import make_golden as golden


def test_golden_streams(tmp_path):
    lib = lr.build(tmp_path)
    rows = golden.load(golden.OUT_LEGACY)
    assert len(rows) == 72
    bad = []
    for (digest, name, pat, w, h, qp, var) in rows:
        y, cb, cr = golden.clip(pat, w, h)
        planes = (np.frombuffer(y, np.uint8).reshape(h, w),) + tuple(
            np.frombuffer(p, np.uint8).reshape(h // 2, w // 2) for p in (cb, cr))
        kw = golden.LEGACY_VARIANTS[var]
        e = lr.Restated(lib, w, h, 2, 0, kw["version"], kw["entropy"])
        packet, _ = e.frame(planes, 0, qp, 0, False)
        e.close()
        if hashlib.sha256(struct.pack("<I", len(packet)) + packet).hexdigest() != digest:
            bad.append(name)
    assert not bad, bad

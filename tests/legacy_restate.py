"""ctypes binding of tests/legacy_restate.cpp.  Test-only."""
import ctypes
import os
import subprocess

import numpy as np

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)


def build(tmp_dir):
    out = os.path.join(str(tmp_dir), "liblegacy_restate.so")
    subprocess.run(["g++", "-O2", "-std=c++17", "-w", "-shared", "-fPIC", "-o", out,
                    os.path.join(HERE, "legacy_restate.cpp"),
                    os.path.join(ROOT, "tcodec_b200", "csrc", "tcb_entropy.cpp")], check=True, timeout=300)
    lib = ctypes.CDLL(out)
    vp, i = ctypes.c_void_p, ctypes.c_int
    lib.lr_create.argtypes = [i] * 8
    lib.lr_create.restype = vp
    lib.lr_destroy.argtypes = [vp]
    lib.lr_frame.argtypes = [vp, vp, vp, vp, i, i, i, i, vp, ctypes.c_size_t, vp, vp, vp]
    lib.lr_frame.restype = ctypes.c_size_t
    return lib


class Restated:
    def __init__(self, lib, w, h, preset, profile, version, entropy, crc=False, threads=0):
        self.lib, self.w, self.h = lib, w, h
        self.handle = lib.lr_create(w, h, preset, profile, version, int(entropy), int(crc), threads)
        self.buf = np.zeros(3 * w * h + 4096, np.uint8)

    def frame(self, planes, frame_type, qp, poc, b_mode):
        """(packet, reconstruction)"""
        planes = [np.ascontiguousarray(p, dtype=np.uint8) for p in planes]
        rec = [np.empty_like(p) for p in planes]
        n = self.lib.lr_frame(self.handle, *(p.ctypes.data for p in planes), frame_type, qp, poc, int(b_mode),
                              self.buf.ctypes.data, self.buf.size, *(p.ctypes.data for p in rec))
        return self.buf[:n].tobytes(), rec

    def close(self):
        self.lib.lr_destroy(self.handle)


def header(packet, b_mode):
    """(frame type, QP, picture number) of a legacy packet."""
    qp = 32 + (packet[9] - 256 if packet[9] > 127 else packet[9])
    key = packet[8] & 0x80
    if packet[3] and b_mode:
        return {0: 0, 2: 2}.get(packet[14], 1), qp, packet[10]
    return (0 if key else 1), qp, packet[10]

"""Key frames of the CTU engine against the integer oracle, decision by
decision: for every leaf of the coded tree the oracle scores all 18 modes and
both TU sizes from its own reconstruction, chooses as the reference does (first
minimum of distortion + lambda * bits), and its mode, TU size, chroma choice
and levels must be the record's; after the CTU's filters its picture must be
the engine's.  Content and quantisers at the ends of their ranges: saturated
residuals, steps from 1 to above every coefficient.  Whole numbers: equality."""
import ctypes

import numpy as np
import pytest

from tests import orabind
from tests.ctu_frames import FrameRun
from tests.test_gpu_residual import _content

pytestmark = pytest.mark.gpu

NODE = np.dtype([(n, "u1") for n in ("split", "skip", "merge", "intra", "bi", "dct_size", "intra_mode", "intra_cmode",
                                     "ref_sel", "ch_intra")] + [("mvd_x", "<i2"), ("mvd_y", "<i2")])
RECORD = np.dtype([("nodes", NODE, 85), ("pad0", "u1", 2), ("ncoef", "<i4"), ("sao", "<i2", 4), ("pad1", "u1", 4),
                   ("tu8mask", "<u8"), ("coef", "<i2", 6144)])
BASE = (0, 1, 5, 21)


class Oracle:
    """One key frame as the oracle codes it, driven by the engine's trees."""

    def __init__(self, planes, qp):
        self.o = orabind.port()
        self.o.or_sao_decide.restype = ctypes.c_int
        self.org = [np.ascontiguousarray(p) for p in planes]
        self.rec = [np.zeros_like(p) for p in self.org]
        self.h, self.w = self.org[0].shape
        self.qp, self.qp_c = qp, min(qp + 1, 63)
        self.lam, self.lam_c = self.o.or_lambda(qp) * 3 // 4, self.o.or_lambda(self.qp_c)

    def tu(self, n, plane, x, y, pred, px, py, rec):
        """One TU at (x, y) of the plane: (sse, bits, levels); reconstruction into rec."""
        org, lv, bits = self.org[plane], np.zeros(64, np.int16), ctypes.c_int()
        luma = plane == 0
        sse = self.o.or_code_tu(n, orabind.PO(org, y * org.shape[1] + x), org.shape[1], orabind.PO(pred, py * pred.shape[1] + px),
                                pred.shape[1], self.qp if luma else self.qp_c, self.lam if luma else self.lam_c,
                                orabind.P(lv), orabind.PO(rec, py * rec.shape[1] + px), rec.shape[1], ctypes.byref(bits))
        return sse, bits.value, lv[:n * n]

    def luma(self, x, y, cu, pred, n):
        """(distortion, bits, levels, reconstruction) of a leaf with n x n TUs."""
        rec, levels, d, b = np.zeros((cu, cu), np.uint8), [], 0, 0
        for ay in range(0, cu, 8):
            for ax in range(0, cu, 8):
                b += n == 4
                for q in range(64 // (n * n)):
                    tx, ty = ax + 4 * (q & 1), ay + 4 * (q >> 1)
                    s, k, lv = self.tu(n, 0, x + tx, y + ty, pred, tx, ty, rec)
                    d, b = d + s, b + k
                    levels.append(lv)
        return d, b, np.concatenate(levels), rec

    def chroma(self, cx, cy, cs, preds):
        d, b, levels, recs = 0, 0, [], []
        for c in (1, 2):
            rec = np.zeros((cs, cs), np.uint8)
            for ty in range(0, cs, 4):
                for tx in range(0, cs, 4):
                    s, k, lv = self.tu(4, c, cx + tx, cy + ty, preds[c - 1], tx, ty, rec)
                    d, b = d + s, b + k
                    levels.append(lv)
            recs.append(rec)
        return d, b, np.concatenate(levels), recs

    def leaf(self, x, y, cu):
        """The leaf's decision: (mode, dct_size, ch_intra, levels); its reconstruction is kept."""
        o, rec = self.o, self.rec
        ra, rl = np.zeros(2 * cu + 4, np.uint8), np.zeros(2 * cu + 4, np.uint8)
        o.or_intra_refs(orabind.P(rec[0]), self.w, x, y, cu, self.w, self.h, orabind.P(ra), orabind.P(rl))
        best = None
        for mode in range(18):
            pred = np.zeros((cu, cu), np.uint8)
            o.or_intra_pred(orabind.P(pred), cu, orabind.P(ra), orabind.P(rl), cu, mode)
            d, b, lv, r = self.luma(x, y, cu, pred, 8)
            dct = 1
            if cu <= 32:
                d4, b4, lv4, r4 = self.luma(x, y, cu, pred, 4)
                if d4 + self.lam * b4 < d + self.lam * b:
                    d, b, lv, r, dct = d4, b4, lv4, r4, 0
            cost = d + self.lam * (8 + b)
            if best is None or cost < best[0]:
                best = (cost, mode, dct, lv, r)
        _, mode, dct, levels, r = best
        rec[0][y:y + cu, x:x + cu] = r
        cs, cx, cy = cu // 2, x // 2, y // 2
        options = []
        for cfl in (0, 1):
            preds = []
            for c in (1, 2):
                p = np.zeros((cs, cs), np.uint8)
                o.or_chroma_dc(orabind.P(rec[c]), self.w // 2, cx, cy, cs, orabind.P(p), cs)
                if cfl:
                    o.or_cfl_blend(orabind.P(p), cs, orabind.P(rec[0]), self.w, orabind.P(rec[c]), self.w // 2, x, y, cx, cy,
                                   cs, cs)
                preds.append(p)
            d, b, lv, rr = self.chroma(cx, cy, cs, preds)
            options.append((d + self.lam * (b + (4 if cfl else 1)), lv, rr))
        cfl = int(options[1][0] < options[0][0])
        for c in (1, 2):
            rec[c][cy:cy + cs, cx:cx + cs] = options[cfl][2][c - 1]
        return mode, dct, cfl, np.concatenate([levels, options[cfl][1]])

    def filters(self, x, y):
        """Deblocking of a whole CTU and SAO; its (present, band, offset)."""
        o, rec, w, h = self.o, self.rec, min(64, self.w - x), min(64, self.h - y)
        if w == 64 and h == 64:
            o.or_deblock_ctu(orabind.P(rec[0]), self.w, orabind.P(rec[1]), self.w // 2, orabind.P(rec[2]), self.w // 2, x, y,
                             self.qp)
        band, off = ctypes.c_int(), ctypes.c_int()
        has = o.or_sao_decide(orabind.P(self.org[0]), self.w, orabind.P(rec[0]), self.w, x, y, self.w, self.h,
                              self.qp, ctypes.byref(band), ctypes.byref(off))
        if has:
            o.or_sao_apply(orabind.P(rec[0]), self.w, x, y, self.w, self.h, band.value, off.value)
        return (int(has != 0), band.value, off.value) if has else (0, 0, 0)


CASES = [(kind, qp, size) for size in ((64, 64), (72, 40), (104, 88))
         for kind, qp in (("saturated", 5), ("saturated", 37), ("saturated", 63), ("stripes", 0), ("stripes", 22),
                          ("stripes", 51), ("flat", 30), ("texture", 0), ("texture", 18), ("texture", 32), ("texture", 45))]


@pytest.mark.parametrize("kind,qp,size", CASES)
def test_every_decision_and_level_is_the_oracles(kind, qp, size):
    import torch
    from tcodec_b200 import api
    lib = api.bind_b200(api.load_library())
    assert RECORD.itemsize == lib.tcb_ctu_record_bytes()
    w, h = size
    rng = np.random.default_rng(qp + w)

    def plane(hh, ww, t):
        if kind != "texture":
            return _content(kind, rng, hh, ww, t)
        yy, xx = np.mgrid[0:hh, 0:ww]
        v = 128 + 70 * np.sin(xx / 5.0 + t) * np.cos(yy / 7.0) + rng.normal(0, 6, (hh, ww))
        return np.clip(v, 0, 255).astype(np.uint8)
    planes = (plane(h, w, 1), plane(h // 2, w // 2, 2), plane(h // 2, w // 2, 3))
    nbytes = lib.tcb_ctu_scratch_bytes(w, h)
    scratch = torch.zeros(nbytes, dtype=torch.uint8, device="cuda")
    st = torch.cuda.current_stream().cuda_stream
    run = FrameRun(lib, [planes], qp, 2, 1, lambda d: lib.tcb_ctu_encode_frame(d, scratch.data_ptr(), nbytes, st))
    *got, records, _ = run.step(0)
    records = np.frombuffer(records.tobytes(), RECORD)
    ora = Oracle(planes, qp)
    cols = (w + 63) // 64
    for k, r in enumerate(records):
        x0, y0 = k % cols * 64, k // cols * 64
        at = 0

        def visit(d, x, y):
            nonlocal at
            cu = 64 >> d
            inside = x + cu <= w and y + cu <= h
            if d == 3 and not inside:
                return
            cx, cy = (x - x0) // 8 >> (3 - d), (y - y0) // 8 >> (3 - d)
            node = r["nodes"][BASE[d] + (cy << d) + cx]
            if d < 3 and (not inside or node["split"]):
                for q in range(4):
                    visit(d + 1, x + (q & 1) * cu // 2, y + (q >> 1) * cu // 2)
                return
            mode, dct, cfl, levels = ora.leaf(x, y, cu)
            where = (x, y, cu)
            assert node["intra"] == 1, where
            assert (node["intra_mode"], node["dct_size"], node["ch_intra"]) == (mode, dct, cfl), where
            assert np.array_equal(r["coef"][at:at + len(levels)], levels), where
            at += len(levels)
        visit(0, x0, y0)
        assert r["ncoef"] == at
        assert tuple(int(v) for v in r["sao"][:3]) == ora.filters(x0, y0)
    for c in range(3):
        assert np.array_equal(got[c], ora.rec[c]), c

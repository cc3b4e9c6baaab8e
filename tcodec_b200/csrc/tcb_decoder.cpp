// tcb_decoder.cpp — tc_decoder_* (reference include/tcodec.h:64-111): the
// serial syntax parse (range decoder / Exp-Golomb) runs on the host and
// fills the same per-CTU records the encoder emits; the reconstruction
// (prediction, dequantisation, inverse transform, deblocking, SAO) runs on
// the device as the CTU wavefront of decode_kernel (v2 streams) or of the
// legacy block kernel (v0 / v1 streams, tcb_legacy.cu).
//
// Mirrors reference src/decoder.c: header checks (102-225), frame-level
// flow (2541-2925), entry-point tables (2096-2190), syntax parse
// (1302-1520), display reorder for B-frame streams (2880-2956).
#include <stdlib.h>
#include <string.h>
#include <time.h>

#include <algorithm>
#include <new>
#include <thread>
#include <vector>

#include <cuda_runtime.h>

#include "../../include/tcodec.h"
#include "../../include/tcodec_b200.h"
#include "tcb_encoder.h"
#include "tcb_entropy.h"
#include "tcb_launch.h"
#include "tcb_parse.h"

using namespace tcb;
using namespace tcb::parse;

namespace {

uint64_t now_ns() {
    timespec t;
    clock_gettime(CLOCK_MONOTONIC, &t);
    return (uint64_t)t.tv_sec * 1000000000ull + (uint64_t)t.tv_nsec;
}

// Replaces the coded vector differences of a CTU's leaves by absolute
// quarter-sample vectors (16-bit, wrapping as in reference
// src/decoder.c:1560-1600): the predictor is the shortest of the left, above
// and above-right neighbours' vectors (src/motion.c:119-170), which chains
// every leaf to the one before, so it is done here, where the leaves are in
// order anyway, and the device takes them in any order.
void resolve_vectors(CtuOut &o, int ctu_x, int ctu_y, int W, int H) {
    struct Cell { int dx, dy; bool ok; } grid[64];
    for (Cell &g : grid) g.ok = false;
    for (int z = 0; z < 64;) {
        const int cx = (z & 1) | (z >> 1 & 2) | (z >> 2 & 4), cy = (z >> 1 & 1) | (z >> 2 & 2) | (z >> 3 & 4);
        int d = 0;
        for (; d < 3; ++d) {   // the largest node that starts here, is inside the frame and not split
            const int gc = 8 >> d, m = gc - 1;
            if (!(cx & m) && !(cy & m) && ctu_x + 8 * (cx + gc) <= W && ctu_y + 8 * (cy + gc) <= H &&
                !o.nodes[qt_index(d, cx, cy)].split)
                break;
        }
        const int gc = 8 >> d;
        if (ctu_x + 8 * (cx + gc) <= W && ctu_y + 8 * (cy + gc) <= H) {
            Node &nd = o.nodes[qt_index(d, cx, cy)];
            Cell a = {0, 0, false}, b = a, c = a;
            if (cx > 0) a = grid[cy * 8 + cx - 1];
            if (cy > 0) b = grid[cy * 8 + cx - 8];
            if (cy > 0 && cx < 7) c = grid[cy * 8 + cx - 7];
            int mx = 0, my = 0;
            if (a.ok || b.ok || c.ok) {
                if (!a.ok) a = b.ok ? b : c;
                if (!b.ok) b = a;
                if (!c.ok) c = a;
                auto len = [](const Cell &g) { return (uint32_t)(g.dx * g.dx) + (uint32_t)(g.dy * g.dy); };
                const uint32_t qa = len(a), qb = len(b), qc = len(c);
                const Cell &p = qb < qa && qb <= qc ? b : qc < qa && qc < qb ? c : a;
                mx = p.dx; my = p.dy;
            }
            const bool own = !(nd.skip || nd.merge);
            const Cell g = {(int16_t)(mx + (own ? nd.mvd_x : 0)), (int16_t)(my + (own ? nd.mvd_y : 0)), !nd.intra};
            for (int y = 0; y < gc; ++y)
                for (int x = 0; x < gc; ++x) grid[(cy + y) * 8 + cx + x] = g;
            const bool add = own && !nd.intra;
            nd.mvd_x = (int16_t)(mx + (ctu_x + cx * 8) * 4 + (add ? nd.mvd_x : 0));
            nd.mvd_y = (int16_t)(my + (ctu_y + cy * 8) * 4 + (add ? nd.mvd_y : 0));
        }
        z += 64 >> (2 * d);
    }
}

}  // namespace

namespace tcb {

struct DecImpl {
    // The size callers are told (tc_decoder_get_info): the one given at
    // creation, else the first packet's.  It does not follow later packets.
    int W = 0, H = 0;
    // The size of the packet at hand, which the buffers, the parser and the
    // kernels all go by.
    int fw = 0, fh = 0, sy = 0, sc = 0, cols = 0, rows = 0;
    int device = 0;
    cudaStream_t st = nullptr;
    DevFrame cur;                     // persistent reconstruction target
    DevFrame dpb[TC_REF_FRAMES];
    int dpb_ok[TC_REF_FRAMES] = {0, 0, 0, 0};
    int dpb_poc[TC_REF_FRAMES] = {-1, -1, -1, -1};
    std::vector<DevFrame> spare;      // free device frames
    CtuOut *d_rec = nullptr, *h_rec = nullptr;
    int *h_status = nullptr;          // the kernels' status word, behind h_rec
    // Legacy (v0 / v1) streams: block records and the wavefront of
    // diagonals c + 2r (see tcb_legacy.cu).
    legacy::LBlock *d_lblk = nullptr, *h_lblk = nullptr;
    int *d_litems = nullptr;
    std::vector<int> ldiag_off, ldiag_cnt;
    FrameParams *d_params = nullptr;
    int *d_items = nullptr;
    std::vector<int> diag_off, diag_cnt;
    tc_frame_buf_t *out = nullptr;    // host output (pinned)
    std::vector<tc_frame_buf_t *> disp_frames;
    std::vector<int> disp_pocs;
    int disp_active = 0, disp_next = 0;
    tc_frame_buf_t *disp_out = nullptr;
    int crc_valid = 1, entropy = 0, threads = 4, profile = 0;
    int lose_area = 0;                // test hook, for the next v2 packet
    uint64_t prof[7] = {0, 0, 0, 0, 0, 0, 0};

    // All three planes or none: a partly allocated frame is freed again.
    bool alloc_frame(DevFrame &f) {
        const size_t yb = (size_t)sy * fh + 64, cb = (size_t)sc * (fh / 2) + 64;
        if (dev_alloc(&f.y, yb) != cudaSuccess || dev_alloc(&f.cb, cb) != cudaSuccess ||
            dev_alloc(&f.cr, cb) != cudaSuccess) {
            free_frame(f);
            return false;
        }
        cudaMemset(f.y, 0, yb); cudaMemset(f.cb, 0, cb); cudaMemset(f.cr, 0, cb);
        return true;
    }
    void free_frame(DevFrame &f) { cudaFree(f.y); cudaFree(f.cb); cudaFree(f.cr); f = DevFrame(); }
    void release_geometry() {
        if (st) cudaStreamSynchronize(st);
        free_frame(cur);
        for (int i = 0; i < TC_REF_FRAMES; ++i) if (dpb_ok[i]) free_frame(dpb[i]);
        for (auto &f : spare) free_frame(f);
        spare.clear();
        for (int i = 0; i < TC_REF_FRAMES; ++i) { dpb_ok[i] = 0; dpb_poc[i] = -1; }
        release_v2_records();
        release_legacy_records();
        tcb_host_frame_free(out);
        out = nullptr;
    }
    // Geometry-dependent buffers for w x h.  On failure everything is
    // released and the size forgotten, so the next frame starts over
    // instead of decoding into a partly allocated set.
    bool setup(int w, int h) {
        if (setup_buffers(w, h)) return true;
        release_geometry();
        fw = fh = 0;
        return false;
    }
    bool setup_buffers(int w, int h) {
        release_geometry();
        fw = w; fh = h;
        sy = ((w + 63) / 64) * 64;
        sc = ((w / 2 + 63) / 64) * 64;
        cols = (w + 63) / 64;
        rows = (h + 63) / 64;
        if (!alloc_frame(cur)) return false;
        // room for the size callers are told: a smaller picture lies in its
        // upper left corner
        out = tcb_host_frame_alloc(std::max(w, std::min(W, TC_MAX_WIDTH)), std::max(h, std::min(H, TC_MAX_HEIGHT)), 1);
        return out != nullptr;
    }
    // Records and work lists of the kind of stream at hand, on its first packet:
    // a stream is v2 or legacy, and the records' pinned host copy is what
    // setting up costs most (1.8 ms for 3.2 MB at 1280x720, each kind).  Buffers
    // that are there are kept, and a failed call leaves none.
    bool setup_records(bool legacy_stream) { return legacy_stream ? setup_legacy_records() : setup_v2_records(); }
    bool setup_v2_records() {
        if (h_rec) return true;
        if (dev_alloc(&d_rec, sizeof(CtuOut) * cols * rows) != cudaSuccess) return release_v2_records();
        if (pinned_alloc(&h_rec, sizeof(CtuOut) * (cols * rows + 1)) != cudaSuccess) return release_v2_records();
        h_status = (int *)(h_rec + cols * rows);
        std::vector<int> items;
        diag_off.clear(); diag_cnt.clear();
        for (int d = 0; d < rows + cols - 1; ++d) {
            diag_off.push_back((int)items.size());
            for (int r = 0; r < rows; ++r) {
                const int c = d - r;
                if (c >= 0 && c < cols) items.push_back((r << 10) | c);
            }
            diag_cnt.push_back((int)items.size() - diag_off.back());
        }
        items.push_back(0);   // the kernels' status word
        if (dev_alloc(&d_items, sizeof(int) * items.size()) != cudaSuccess) return release_v2_records();
        cudaMemcpy(d_items, items.data(), sizeof(int) * items.size(), cudaMemcpyHostToDevice);
        return true;
    }
    bool setup_legacy_records() {
        if (h_lblk) return true;
        std::vector<int> litems;
        ldiag_off.clear(); ldiag_cnt.clear();
        for (int d = 0; d < cols + 2 * (rows - 1); ++d) {
            ldiag_off.push_back((int)litems.size());
            for (int r = 0; r < rows; ++r) {
                const int c = d - 2 * r;
                if (c >= 0 && c < cols) litems.push_back((r << 10) | c);
            }
            ldiag_cnt.push_back((int)litems.size() - ldiag_off.back());
        }
        if (dev_alloc(&d_litems, sizeof(int) * litems.size()) != cudaSuccess) return release_legacy_records();
        cudaMemcpy(d_litems, litems.data(), sizeof(int) * litems.size(), cudaMemcpyHostToDevice);
        const size_t nblk = (size_t)cols * rows * legacy::BLOCKS;
        if (dev_alloc(&d_lblk, sizeof(legacy::LBlock) * nblk) != cudaSuccess) return release_legacy_records();
        if (pinned_alloc(&h_lblk, sizeof(legacy::LBlock) * nblk) != cudaSuccess) return release_legacy_records();
        return true;
    }
    bool release_v2_records() {
        cudaFree(d_rec); cudaFreeHost(h_rec); cudaFree(d_items);
        d_rec = nullptr; h_rec = nullptr; d_items = nullptr;
        return false;
    }
    bool release_legacy_records() {
        cudaFree(d_lblk); cudaFreeHost(h_lblk); cudaFree(d_litems);
        d_lblk = nullptr; h_lblk = nullptr; d_litems = nullptr;
        return false;
    }
    DevFrame take_frame() {
        if (!spare.empty()) { DevFrame f = spare.back(); spare.pop_back(); return f; }
        DevFrame f;
        if (!alloc_frame(f)) f = DevFrame();
        return f;
    }
    bool copy_frame(const DevFrame &dst, const DevFrame &src) {
        return cudaMemcpyAsync(dst.y, src.y, (size_t)sy * fh, cudaMemcpyDeviceToDevice, st) == cudaSuccess &&
               cudaMemcpyAsync(dst.cb, src.cb, (size_t)sc * (fh / 2), cudaMemcpyDeviceToDevice, st) == cudaSuccess &&
               cudaMemcpyAsync(dst.cr, src.cr, (size_t)sc * (fh / 2), cudaMemcpyDeviceToDevice, st) == cudaSuccess;
    }
    void clear_frame(const DevFrame &f) {
        cudaMemsetAsync(f.y, 0, (size_t)sy * fh, st);
        cudaMemsetAsync(f.cb, 0, (size_t)sc * (fh / 2), st);
        cudaMemsetAsync(f.cr, 0, (size_t)sc * (fh / 2), st);
    }
    bool d2h(tc_frame_buf_t *dst, const DevFrame &src) {
        return cudaMemcpy2DAsync(dst->y, dst->stride_y, src.y, sy, fw, fh, cudaMemcpyDeviceToHost, st) == cudaSuccess &&
               cudaMemcpy2DAsync(dst->cb, dst->stride_c, src.cb, sc, fw / 2, fh / 2, cudaMemcpyDeviceToHost, st) == cudaSuccess &&
               cudaMemcpy2DAsync(dst->cr, dst->stride_c, src.cr, sc, fw / 2, fh / 2, cudaMemcpyDeviceToHost, st) == cudaSuccess &&
               cudaStreamSynchronize(st) == cudaSuccess;
    }
    tc_error_t decode(const uint8_t *data, size_t size, const tc_pixel_t **y, int *ys, const tc_pixel_t **cb,
                      int *cbs, const tc_pixel_t **cr, int *crs);
    tc_error_t legacy_body(const uint8_t *data, size_t size, Reader &bs, const Header &hdr);
    tc_error_t emit(tc_frame_buf_t *f, const tc_pixel_t **y, int *ys, const tc_pixel_t **cb, int *cbs,
                    const tc_pixel_t **cr, int *crs) {
        if (y) *y = f->y;
        if (ys) *ys = f->stride_y;
        if (cb) *cb = f->cb;
        if (cbs) *cbs = f->stride_c;
        if (cr) *cr = f->cr;
        if (crs) *crs = f->stride_c;
        return TC_OK;
    }
    tc_error_t pop_display(const tc_pixel_t **y, int *ys, const tc_pixel_t **cb, int *cbs,
                           const tc_pixel_t **cr, int *crs) {
        for (size_t i = 0; i < disp_pocs.size(); ++i)
            if (disp_pocs[i] == disp_next) {
                if (!disp_out) disp_out = tcb_host_frame_alloc(W, H, 1);
                if (!disp_out) return TC_ERR_MEMORY;
                tc_frame_buf_t *f = disp_frames[i];
                const int cw = (disp_out->width < f->width ? disp_out->width : f->width);
                const int chh = (disp_out->height < f->height ? disp_out->height : f->height);
                if (cw < disp_out->width || chh < disp_out->height) {   // nothing of an earlier, larger picture
                    memset(disp_out->y, 0, (size_t)disp_out->stride_y * disp_out->height);
                    memset(disp_out->cb, 0, (size_t)disp_out->stride_c * (disp_out->height / 2));
                    memset(disp_out->cr, 0, (size_t)disp_out->stride_c * (disp_out->height / 2));
                }
                for (int r = 0; r < chh; ++r) memcpy(disp_out->y + (size_t)r * disp_out->stride_y, f->y + (size_t)r * f->stride_y, cw);
                for (int r = 0; r < chh / 2; ++r) {
                    memcpy(disp_out->cb + (size_t)r * disp_out->stride_c, f->cb + (size_t)r * f->stride_c, cw / 2);
                    memcpy(disp_out->cr + (size_t)r * disp_out->stride_c, f->cr + (size_t)r * f->stride_c, cw / 2);
                }
                tcb_host_frame_free(f);
                disp_frames.erase(disp_frames.begin() + i);
                disp_pocs.erase(disp_pocs.begin() + i);
                disp_next++;
                return emit(disp_out, y, ys, cb, cbs, cr, crs);
            }
        return TC_ERR_NEED_MORE;
    }
};

tc_error_t DecImpl::decode(const uint8_t *data, size_t size, const tc_pixel_t **y, int *ys,
                           const tc_pixel_t **cb, int *cbs, const tc_pixel_t **cr, int *crs) {
    const uint64_t t_parse0 = now_ns();
    Reader bs;
    bs.init(data, size);
    Header hdr;
    tc_error_t err = read_header(bs, hdr);
    if (err != TC_OK) return err;
    const bool legacy_stream = hdr.version != TC_VERSION_V2;
    if ((hdr.W & 1) || (hdr.H & 1)) return TC_ERR_BITSTREAM;
    if (legacy_stream && (hdr.tools & TC_TOOL_ENTRY_POINTS)) return TC_ERR_BITSTREAM;
    if (W == 0 || H == 0) { W = hdr.W; H = hdr.H; }
    if (!cur.y || fw != hdr.W || fh != hdr.H)
        if (!setup(hdr.W, hdr.H)) return TC_ERR_MEMORY;
    if (!setup_records(legacy_stream)) return TC_ERR_MEMORY;
    crc_valid = 1;
    if (hdr.has_crc) {
        if (size >= 2) {
            const size_t p = size - 2;
            if (crc16_ccitt(data, p) != (uint16_t)((data[p] << 8) | data[p + 1])) crc_valid = 0;
        } else {
            crc_valid = 0;
        }
    }
    if (!legacy_stream && (hdr.flags & TC_FLAG_WPP)) return TC_ERR_BITSTREAM;
    entropy = (hdr.version != TC_VERSION_V0 && (hdr.tools & TC_TOOL_ENTROPY_CODED)) ? 1 : 0;
    bs.align();
    if (hdr.frame_type == 0 && hdr.frame_num > 0)
        for (int i = 0; i < TC_REF_FRAMES; ++i) {
            if (dpb_ok[i]) spare.push_back(dpb[i]);
            dpb_ok[i] = 0; dpb_poc[i] = -1; dpb[i] = DevFrame();
        }
    uint64_t t_parse1 = 0;
    if (legacy_stream) {
        const tc_error_t le = legacy_body(data, size, bs, hdr);
        if (le != TC_OK) return le;
        t_parse1 = now_ns();
    } else {
    // ---- parse every CTU into its record ------------------------------
    const int multiref_tool = (hdr.tools & TC_TOOL_MULTI_REF) != 0;
    const int sao_tool = (hdr.tools & TC_TOOL_SAO) != 0;
    auto parse_rows = [&](Reader &r, RDec *rc, uint8_t *ctx, int row0, int row1) -> bool {
        Parser p{&r, rc, ctx, fw, fh, hdr.frame_type, multiref_tool, sao_tool, dpb_ok, nullptr, 0, 0, 0};
        for (int row = row0; row < row1; ++row)
            for (int col = 0; col < cols; ++col) {
                p.o = h_rec + row * cols + col;
                p.ctu(row, col);
                if (r.error) return false;
                resolve_vectors(*p.o, col * 64, row * 64, fw, fh);
            }
        return true;
    };
    if (hdr.tools & TC_TOOL_ENTRY_POINTS) {
        // Entry-point table (reference src/decoder.c:2096-2190).
        if (rows < 1 || rows > 64 || cols < 1) return TC_ERR_BITSTREAM;
        if (bs.pos >= bs.size) return TC_ERR_BITSTREAM;
        const uint32_t nrows = bs.bits(16);
        if (bs.error || nrows != (uint32_t)rows) return TC_ERR_BITSTREAM;
        uint32_t off[64];
        for (int i = 0; i < rows; ++i) {
            off[i] = bs.bits(32);
            if (bs.error) return TC_ERR_BITSTREAM;
        }
        const size_t payload = bs.pos;
        size_t data_end = size;
        if (hdr.has_crc) {
            if (data_end < 2) return TC_ERR_BITSTREAM;
            data_end -= 2;
        }
        if (data_end < payload) return TC_ERR_BITSTREAM;
        const size_t datalen = data_end - payload;
        if (off[0] != 0) return TC_ERR_BITSTREAM;
        for (int i = 1; i < rows; ++i)
            if (off[i] < off[i - 1] || off[i] > datalen) return TC_ERR_BITSTREAM;
        for (int r = 0; r < rows; ++r) {
            const size_t start = payload + off[r];
            const size_t end = r + 1 < rows ? payload + off[r + 1] : data_end;
            if (end < start || end > size) return TC_ERR_BITSTREAM;
        }
        // Every row is its own substream with fresh contexts and writes
        // only its own CTU records, so the rows parse on up to `threads`
        // host threads (tc_decoder_set_threads); any bad row fails the frame.
        bool row_bad[64];
        auto parse_part = [&](int first, int step) {
            for (int r = first; r < rows; r += step) {
                const size_t start = payload + off[r];
                const size_t end = r + 1 < rows ? payload + off[r + 1] : data_end;
                Reader rr;
                rr.init(data + start, end - start);
                RDec rc;
                uint8_t ctx[TC_NUM_CONTEXTS_RC];
                memset(ctx, 0, sizeof(ctx));
                if (entropy) rc.init(&rr);
                row_bad[r] = !parse_rows(rr, entropy ? &rc : nullptr, ctx, r, r + 1);
            }
        };
        const int nth = std::max(1, std::min(threads, rows));
        if (nth > 1) {
            std::vector<std::thread> th;
            for (int t = 1; t < nth; ++t) th.emplace_back(parse_part, t, nth);
            parse_part(0, nth);
            for (auto &x : th) x.join();
        } else {
            parse_part(0, 1);
        }
        for (int r = 0; r < rows; ++r)
            if (row_bad[r]) return TC_ERR_BITSTREAM;
    } else {
        RDec rc;
        uint8_t ctx[TC_NUM_CONTEXTS_RC];
        memset(ctx, 0, sizeof(ctx));
        if (entropy) rc.init(&bs);
        if (!parse_rows(bs, entropy ? &rc : nullptr, ctx, 0, rows)) return TC_ERR_BITSTREAM;
    }
    t_parse1 = now_ns();
    // ---- device reconstruction ------------------------------------------
    FrameParams P;
    memset(&P, 0, sizeof(P));
    P.W = fw; P.H = fh; P.stride_y = sy; P.stride_c = sc; P.ctu_cols = cols; P.ctu_rows = rows;
    P.rec_y = cur.y; P.rec_cb = cur.cb; P.rec_cr = cur.cr;
    for (int i = 0; i < MAX_REFS; ++i) {
        P.ref_valid[i] = dpb_ok[i];
        P.ref_poc[i] = dpb_poc[i];
        const DevFrame &f = dpb_ok[i] ? dpb[i] : cur;
        P.ref_y[i] = f.y; P.ref_cb[i] = f.cb; P.ref_cr[i] = f.cr;
    }
    P.out = d_rec;
    P.frame_type = hdr.frame_type;
    P.poc = hdr.frame_num;
    P.qp = hdr.qp;
    P.qp_c = clampi(hdr.qp + 1, 0, 63);
    P.fresh_skip = (hdr.tools & TC_TOOL_FRESH_SKIP) != 0;
    P.lose_area = lose_area;
    lose_area = 0;
    static const int qs[64] = TCB_QSCALE_INIT;
    static const int jw[4] = TCB_JND_INIT;
    for (int b = 0; b < 4; ++b) {
        P.eff_l[b] = maxi((qs[P.qp] * jw[b] + 4) >> 3, 1);
        P.eff_c[b] = maxi((qs[P.qp_c] * jw[b] + 4) >> 3, 1);
    }
    if (!d_params && dev_alloc(&d_params, sizeof(FrameParams)) != cudaSuccess) return TC_ERR_MEMORY;
    const int nctu = rows * cols;
    if (cudaMemcpyAsync(d_params, &P, sizeof(P), cudaMemcpyHostToDevice, st) != cudaSuccess ||
        cudaMemcpyAsync(d_rec, h_rec, sizeof(CtuOut) * nctu, cudaMemcpyHostToDevice, st) != cudaSuccess)
        return TC_ERR_INTERNAL;
    for (size_t d = 0; d < diag_off.size(); ++d)
        if (launch_decode_items(d_params, d_items + diag_off[d], diag_cnt[d], d_items + nctu, st) != cudaSuccess)
            return TC_ERR_INTERNAL;
    if (cudaMemcpyAsync(h_status, d_items + nctu, sizeof(int), cudaMemcpyDeviceToHost, st) != cudaSuccess)
        return TC_ERR_INTERNAL;
    }   // v2 stream
    // DPB: slot 3 falls out and its buffer takes a copy of the reconstruction
    // into slot 0 (another buffer when slot 3 is empty, taken here, while the
    // kernels run).  Nothing moves before the picture is known to be good: a
    // packet that fails from here on leaves the DPB, and the reconstruction
    // that later packets build on, as they were.
    const bool reuse = dpb_ok[TC_REF_FRAMES - 1] != 0;
    const DevFrame nf = reuse ? dpb[TC_REF_FRAMES - 1] : take_frame();
    auto undo = [&](tc_error_t e) {
        if (!reuse && nf.y) spare.push_back(nf);
        if (dpb_ok[0]) copy_frame(cur, dpb[0]);
        else clear_frame(cur);
        return e;
    };
    if (!nf.y) return undo(TC_ERR_MEMORY);
    if (!d2h(out, cur)) return undo(TC_ERR_INTERNAL);
    if (!legacy_stream && *h_status != 0) {   // an area gave up waiting
        cudaMemsetAsync(d_items + rows * cols, 0, sizeof(int), st);
        return undo(TC_ERR_INTERNAL);
    }
    // (ordered before the next packet's kernels on the stream)
    if (!copy_frame(nf, cur)) return undo(TC_ERR_INTERNAL);
    for (int i = TC_REF_FRAMES - 1; i > 0; --i) { dpb[i] = dpb[i - 1]; dpb_ok[i] = dpb_ok[i - 1]; dpb_poc[i] = dpb_poc[i - 1]; }
    dpb[0] = nf; dpb_ok[0] = 1; dpb_poc[0] = hdr.frame_num;
    const uint64_t t_rec = now_ns();
    if (profile) { prof[0] += t_parse1 - t_parse0; prof[2] += t_rec - t_parse1; }
    if (hdr.has_ext) {
        // Display reorder (reference src/decoder.c:2880-2925).
        const int is_rap = (hdr.flags & TC_FLAG_RAP) != 0;
        if (is_rap && disp_active) {
            for (auto *f : disp_frames) tcb_host_frame_free(f);
            disp_frames.clear(); disp_pocs.clear();
            disp_next = hdr.frame_num;
        }
        disp_active = 1;
        if ((int)disp_frames.size() < TC_REF_FRAMES + 1) {
            tc_frame_buf_t *f = tcb_host_frame_alloc(fw, fh, 0);
            if (!f) return TC_ERR_MEMORY;
            for (int r = 0; r < fh; ++r) memcpy(f->y + (size_t)r * f->stride_y, out->y + (size_t)r * out->stride_y, fw);
            for (int r = 0; r < fh / 2; ++r) {
                memcpy(f->cb + (size_t)r * f->stride_c, out->cb + (size_t)r * out->stride_c, fw / 2);
                memcpy(f->cr + (size_t)r * f->stride_c, out->cr + (size_t)r * out->stride_c, fw / 2);
            }
            disp_frames.push_back(f);
            disp_pocs.push_back(hdr.frame_num);
        }
        return pop_display(y, ys, cb, cbs, cr, crs);
    }
    return emit(out, y, ys, cb, cbs, cr, crs);
}

// Legacy stream body: rows as per-row runs behind a 16-bit entry table
// (TC_FLAG_WPP) or one run, raw or range coded; parse on the host, then
// the legacy CTU wavefront reconstructs into `cur`, whose previous contents
// (the last decoded frame) stand in for samples not yet decoded, as in the
// reference decoder (src/decoder.c:2620-2770, 652-683).
tc_error_t DecImpl::legacy_body(const uint8_t *data, size_t size, Reader &bs, const Header &hdr) {
    if (upload_legacy_tables() != cudaSuccess) return TC_ERR_INTERNAL;
    const int ft = hdr.frame_type;
    const size_t nblk = (size_t)cols * rows * legacy::BLOCKS;
    const tc_error_t pe = parse_legacy_frame(data, size, bs, hdr, entropy, fw, fh, cols, rows, h_lblk);
    if (pe != TC_OK) return pe;
    legacy::LFrame F;
    memset(&F, 0, sizeof(F));
    F.W = fw; F.H = fh; F.sy = sy; F.sc = sc; F.ctu_cols = cols; F.ctu_rows = rows;
    F.rec_y = cur.y; F.rec_cb = cur.cb; F.rec_cr = cur.cr;
    int fp = -1, bp = 0x7FFFFFFF;
    for (int i = 0; i < TC_REF_FRAMES; ++i) {
        F.dpb_y[i] = dpb_ok[i] ? dpb[i].y : nullptr;
        if (!dpb_ok[i] || dpb_poc[i] < 0) continue;
        if (dpb_poc[i] < hdr.frame_num && dpb_poc[i] > fp) { fp = dpb_poc[i]; F.fwd_y = dpb[i].y; }
        if (dpb_poc[i] > hdr.frame_num && dpb_poc[i] < bp) { bp = dpb_poc[i]; F.bwd_y = dpb[i].y; }
    }
    F.frame_type = ft;
    F.qp = hdr.qp;
    F.blocks = d_lblk;
    if (cudaMemcpyAsync(d_lblk, h_lblk, sizeof(legacy::LBlock) * nblk, cudaMemcpyHostToDevice, st) != cudaSuccess)
        return TC_ERR_INTERNAL;
    for (size_t d = 0; d < ldiag_off.size(); ++d)
        if (launch_legacy_decode(F, d_litems + ldiag_off[d], ldiag_cnt[d], st) != cudaSuccess)
            return TC_ERR_INTERNAL;
    return TC_OK;
}

}  // namespace tcb

struct tc_decoder {
    tcb::DecImpl *impl;
};

extern "C" {

tc_decoder_t *tc_decoder_create(int32_t width, int32_t height) {
    int ndev = 0;
    if (cudaGetDeviceCount(&ndev) != cudaSuccess || ndev == 0) return nullptr;
    if (init_device_tables() != cudaSuccess) return nullptr;
    tc_decoder_t *d = (tc_decoder_t *)calloc(1, sizeof(tc_decoder_t));
    if (!d) return nullptr;
    d->impl = new (std::nothrow) DecImpl();
    if (!d->impl) { free(d); return nullptr; }
    DecImpl &e = *d->impl;
    cudaGetDevice(&e.device);
    if (cudaStreamCreateWithFlags(&e.st, cudaStreamNonBlocking) != cudaSuccess) {
        delete d->impl; free(d); return nullptr;
    }
    e.W = width > 0 && height > 0 ? width : 0;
    e.H = width > 0 && height > 0 ? height : 0;
    return d;
}

void tc_decoder_destroy(tc_decoder_t *dec) {
    if (!dec) return;
    if (dec->impl) {
        DecImpl &e = *dec->impl;
        e.release_geometry();
        for (auto *f : e.disp_frames) tcb_host_frame_free(f);
        tcb_host_frame_free(e.disp_out);
        cudaFree(e.d_params);
        if (e.st) cudaStreamDestroy(e.st);
        delete dec->impl;
    }
    free(dec);
}

tc_error_t tc_decoder_decode(tc_decoder_t *dec, const uint8_t *data, size_t size, const tc_pixel_t **y,
                             int *stride_y, const tc_pixel_t **cb, int *stride_cb, const tc_pixel_t **cr,
                             int *stride_cr) {
    // no frame unless one is output: callers that ignore the status read
    // NULL planes rather than stale pointers
    if (y) *y = nullptr;
    if (cb) *cb = nullptr;
    if (cr) *cr = nullptr;
    if (stride_y) *stride_y = 0;
    if (stride_cb) *stride_cb = 0;
    if (stride_cr) *stride_cr = 0;
    if (!dec || !dec->impl || !data || size == 0) return TC_ERR_PARAM;
    if (cudaSetDevice(dec->impl->device) != cudaSuccess) return TC_ERR_INTERNAL;
    return dec->impl->decode(data, size, y, stride_y, cb, stride_cb, cr, stride_cr);
}

void tc_decoder_get_info(tc_decoder_t *dec, int32_t *width, int32_t *height) {
    if (!dec || !dec->impl) return;
    if (width) *width = dec->impl->W;
    if (height) *height = dec->impl->H;
}

tc_error_t tc_decoder_flush_tail(tc_decoder_t *dec, const tc_pixel_t **y, int *stride_y, const tc_pixel_t **cb,
                                 int *stride_cb, const tc_pixel_t **cr, int *stride_cr) {
    if (!dec || !dec->impl || !dec->impl->disp_active) return TC_ERR_EOF;
    const tc_error_t r = dec->impl->pop_display(y, stride_y, cb, stride_cb, cr, stride_cr);
    return r == TC_ERR_NEED_MORE ? TC_ERR_EOF : r;
}

int tc_decoder_crc_valid(tc_decoder_t *dec) { return dec && dec->impl ? dec->impl->crc_valid : 0; }
int tc_decoder_entropy_coded(tc_decoder_t *dec) { return dec && dec->impl ? dec->impl->entropy : 0; }
void tc_decoder_set_profile(tc_decoder_t *dec, int enabled) { if (dec && dec->impl) dec->impl->profile = enabled; }
void tc_decoder_reset_profile(tc_decoder_t *dec) {
    if (dec && dec->impl) memset(dec->impl->prof, 0, sizeof(dec->impl->prof));
}
void tc_decoder_get_profile(tc_decoder_t *dec, uint64_t *parse_ns, uint64_t *coeff_ns, uint64_t *transform_ns,
                            uint64_t *motion_ns, uint64_t *chroma_ns, uint64_t *deblock_ns, uint64_t *copy_ns) {
    if (!dec || !dec->impl) return;
    const uint64_t *p = dec->impl->prof;
    if (parse_ns) *parse_ns = p[0];
    if (coeff_ns) *coeff_ns = p[1];
    if (transform_ns) *transform_ns = p[2];
    if (motion_ns) *motion_ns = p[3];
    if (chroma_ns) *chroma_ns = p[4];
    if (deblock_ns) *deblock_ns = p[5];
    if (copy_ns) *copy_ns = p[6];
}
void tc_decoder_set_threads(tc_decoder_t *dec, int nthreads) {
    if (!dec || !dec->impl) return;
    dec->impl->threads = nthreads < 1 ? 1 : (nthreads > 16 ? 16 : nthreads);
}

tc_error_t tcb_debug_decoder_lose_area(tc_decoder_t *dec) {
    if (!dec || !dec->impl) return TC_ERR_PARAM;
    dec->impl->lose_area = 1;
    return TC_OK;
}

}  // extern "C"

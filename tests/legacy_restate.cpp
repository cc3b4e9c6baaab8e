// legacy_restate.cpp — the legacy (v0 / v1) encoder's CPU restatement
// (tcodec_b200/csrc/tcb_legacy.cuh as plain C++, a team of one lane) behind a
// C interface, for the tests that hold the GPU's block encoder to it.  A handle
// keeps what an encoder keeps between frames: the reconstruction, which is
// coded in place, and the DPB.  Frame type, QP and picture number are the
// caller's; packets are written by the library's host syntax writer.
#include <math.h>
#include <stdint.h>
#include <string.h>

#include <vector>

#include "../include/tcodec.h"

#define __device__
#define __forceinline__ inline
#define __constant__
#define __noinline__
static inline int __ffs(int x) { return __builtin_ffs(x); }

namespace tcb {
namespace legacy {
static int g_dct[9][8][8];
inline int ldct4(int k, int n) { return g_dct[4][k][n]; }
inline int ldct8(int k, int n) { return g_dct[8][k][n]; }
}  // namespace legacy
}  // namespace tcb

#include "../tcodec_b200/csrc/tcb_entropy.h"
#include "../tcodec_b200/csrc/tcb_legacy.cuh"

using namespace tcb;
using namespace tcb::legacy;

namespace {

struct Picture {
    std::vector<uint8_t> y, cb, cr;
    int poc;
};
struct Restated {
    tc_config_t cfg;
    int W, H, sy, sc, cols, rows;
    Picture cur, rec;
    std::vector<Picture> dpb;              // newest first
    std::vector<LBlock> blocks;
    std::vector<uint8_t> scratch;
    LState S;
};

void rows_in(std::vector<uint8_t> &d, int s, const uint8_t *src, int w, int h) {
    for (int r = 0; r < h; ++r) memcpy(&d[(size_t)r * s], src + (size_t)r * w, w);
}
void rows_out(uint8_t *dst, const std::vector<uint8_t> &s, int stride, int w, int h) {
    for (int r = 0; r < h; ++r) memcpy(dst + (size_t)r * w, &s[(size_t)r * stride], w);
}

}  // namespace

extern "C" {

void *lr_create(int W, int H, int preset, int profile, int version, int entropy, int crc, int threads) {
    for (int N = 4; N <= 8; N += 4)
        for (int k = 0; k < N; ++k)
            for (int n = 0; n < N; ++n)
                g_dct[N][k][n] = (int)lround(16384.0 * sqrt((k ? 2.0 : 1.0) / N) * cos((2 * n + 1) * k * M_PI / (2.0 * N)));
    Restated *e = new Restated();
    memset(&e->cfg, 0, sizeof(e->cfg));
    e->cfg.width = W; e->cfg.height = H;
    e->cfg.preset = (tc_preset_t)preset;
    e->cfg.profile = (uint8_t)profile;
    e->cfg.bitstream_version = (uint8_t)version;
    e->cfg.enable_entropy_coded = entropy;
    e->cfg.enable_crc = crc;
    e->cfg.threads = threads;
    e->W = W; e->H = H;
    e->sy = (W + 63) / 64 * 64; e->sc = (W / 2 + 63) / 64 * 64;
    e->cols = (W + 63) / 64; e->rows = (H + 63) / 64;
    for (Picture *p : {&e->cur, &e->rec}) {
        p->y.assign((size_t)e->sy * H + 64, 0);
        p->cb.assign((size_t)e->sc * (H / 2) + 64, 0);
        p->cr.assign((size_t)e->sc * (H / 2) + 64, 0);
    }
    e->blocks.resize((size_t)e->cols * e->rows * BLOCKS);
    return e;
}

void lr_destroy(void *h) { delete (Restated *)h; }

// Encodes one picture; planes are tight.  Returns the packet's size.
size_t lr_frame(void *h, const uint8_t *y, const uint8_t *cb, const uint8_t *cr, int frame_type, int qp, int poc,
                int b_mode, uint8_t *out, size_t cap, uint8_t *ry, uint8_t *rcb, uint8_t *rcr) {
    Restated &e = *(Restated *)h;
    const int W = e.W, H = e.H;
    rows_in(e.cur.y, e.sy, y, W, H);
    rows_in(e.cur.cb, e.sc, cb, W / 2, H / 2);
    rows_in(e.cur.cr, e.sc, cr, W / 2, H / 2);
    if (frame_type == 0 && poc > 0) e.dpb.clear();
    LFrame F;
    memset(&F, 0, sizeof(F));
    F.W = W; F.H = H; F.sy = e.sy; F.sc = e.sc; F.ctu_cols = e.cols; F.ctu_rows = e.rows;
    F.cur_y = e.cur.y.data(); F.cur_cb = e.cur.cb.data(); F.cur_cr = e.cur.cr.data();
    F.rec_y = e.rec.y.data(); F.rec_cb = e.rec.cb.data(); F.rec_cr = e.rec.cr.data();
    for (size_t i = 0; i < e.dpb.size(); ++i) F.dpb_y[i] = e.dpb[i].y.data();
    if (frame_type == 2) {
        int fp = -1, bp = 0x7FFFFFFF;
        for (Picture &p : e.dpb) {
            if (p.poc < poc && p.poc > fp) { fp = p.poc; F.fwd_y = p.y.data(); }
            if (p.poc > poc && p.poc < bp) { bp = p.poc; F.bwd_y = p.y.data(); }
        }
        const uint8_t *two[2] = {F.fwd_y, F.bwd_y};
        for (int k = 0; k < 2; ++k)
            if (two[k]) { F.cand_y[F.n_cand] = two[k]; F.cand_sel[F.n_cand++] = k; }
    } else if (frame_type == 1) {
        const size_t most = e.cfg.preset == TC_PRESET_SLOW && e.cfg.profile >= TC_PROFILE_STREAMING_MAIN ? TC_REF_FRAMES : 1;
        for (size_t i = 0; i < most && i < e.dpb.size() && F.n_cand < 2; ++i) {
            F.cand_y[F.n_cand] = F.dpb_y[i];
            F.cand_sel[F.n_cand++] = (int)i;
        }
    }
    F.frame_type = frame_type;
    F.qp = qp;
    F.search_range = e.cfg.preset == TC_PRESET_ULTRAFAST ? 16 : e.cfg.preset == TC_PRESET_SLOW ? 64 : 32;
    const long long s = qscale_of(qp), l = (s * s * 200) >> 10;
    F.lambda = l < 1 ? 1 : l > (1ll << 30) ? 1ll << 30 : l;
    F.blocks = e.blocks.data();
    for (int r = 0; r < e.rows; ++r)
        for (int c = 0; c < e.cols; ++c) code_ctu(e.S, F, r, c, true);
    const int threads = e.cfg.threads > 0 ? e.cfg.threads : 4;
    const bool wpp = e.rows > 1 && threads > 1 && !e.cfg.enable_entropy_coded;
    const size_t n = write_legacy_frame(out, cap, legacy_frame_syntax(e.cfg, frame_type == 0, frame_type, qp, poc, b_mode, wpp),
                                        e.blocks.data(), e.cols, e.rows, e.scratch);
    rows_out(ry, e.rec.y, e.sy, W, H);
    rows_out(rcb, e.rec.cb, e.sc, W / 2, H / 2);
    rows_out(rcr, e.rec.cr, e.sc, W / 2, H / 2);
    e.dpb.insert(e.dpb.begin(), e.rec);
    e.dpb[0].poc = poc;
    if (e.dpb.size() > TC_REF_FRAMES) e.dpb.pop_back();
    return n;
}

}  // extern "C"

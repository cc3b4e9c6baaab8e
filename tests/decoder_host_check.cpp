// decoder_host_check.cpp — the v2 decoder's host side (tcb_decoder.cpp) on
// the CPU, against a CUDA runtime whose device memory is host memory with
// known bounds.
//
// Every copy is checked against the allocations it touches.  In the kernel's
// place, the launch checks the frame parameters it is handed: that every
// sample the reconstruction reads or writes for this work list (its
// CTU's border, interior and export, and references clamped to the frame)
// lies in its plane's allocation, and that every leaf of the parsed tree
// carries the vector of its own position.  Packets are raw Exp-Golomb key and
// P frames without levels, written here.
//
// Usage: decoder_host_check sizes|reorder W0 H0 W H [W H ...]: a decoder created
// for W0 x H0 (0 0: from the stream) is fed two packets per size; or
// decoder_host_check status|status_key W0 H0 W H n lost: n packets, of which
// one (a key frame in status_key) fails in the kernel.  Exit code 0 when every
// check holds.
#include <stdint.h>
#include <stdio.h>
#include <stdlib.h>
#include <string.h>

#include <map>
#include <string>
#include <vector>

#include "../tcodec_b200/csrc/tcb_decoder.cpp"

// ---------------------------------------------------------------- runtime

static std::map<const uint8_t *, size_t> g_mem;    // live allocations
static std::vector<std::string> g_bad;

static void bad(const std::string &s) {
    if (g_bad.size() < 20) g_bad.push_back(s);
}
// Bytes from p to the end of its allocation; -1 when it lies in none.
static long long room(const void *q) {
    const uint8_t *p = (const uint8_t *)q;
    auto it = g_mem.upper_bound(p);
    if (it == g_mem.begin()) return -1;
    --it;
    return p <= it->first + it->second ? (long long)(it->first + it->second - p) : -1;
}
static bool is_device(const void *p) { return room(p) >= 0; }
static void check_2d(const void *p, size_t pitch, size_t w, size_t h, const char *what) {
    if (!w || !h || !is_device(p)) return;
    if (room(p) < (long long)(pitch * (h - 1) + w)) bad(std::string(what) + " past its allocation");
}

extern "C" {
cudaError_t cudaMalloc(void **p, size_t n) {
    *p = malloc(n ? n : 1);
    g_mem[(const uint8_t *)*p] = n;
    return cudaSuccess;
}
cudaError_t cudaMallocHost(void **p, size_t n) { return cudaMalloc(p, n); }
cudaError_t cudaFree(void *p) {
    if (p && !g_mem.erase((const uint8_t *)p)) bad("free of an unknown pointer");
    free(p);
    return cudaSuccess;
}
cudaError_t cudaFreeHost(void *p) { return cudaFree(p); }
cudaError_t cudaMemset(void *p, int v, size_t n) {
    check_2d(p, n, n, 1, "memset");
    memset(p, v, n);
    return cudaSuccess;
}
cudaError_t cudaMemsetAsync(void *p, int v, size_t n, cudaStream_t) { return cudaMemset(p, v, n); }
cudaError_t cudaMemcpy(void *d, const void *s, size_t n, cudaMemcpyKind) {
    check_2d(d, n, n, 1, "copy destination");
    check_2d(s, n, n, 1, "copy source");
    memcpy(d, s, n);
    return cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void *d, const void *s, size_t n, cudaMemcpyKind k, cudaStream_t) {
    return cudaMemcpy(d, s, n, k);
}
cudaError_t cudaMemcpy2DAsync(void *d, size_t dp, const void *s, size_t sp, size_t w, size_t h, cudaMemcpyKind,
                              cudaStream_t) {
    check_2d(d, dp, w, h, "2D copy destination");
    check_2d(s, sp, w, h, "2D copy source");
    for (size_t y = 0; y < h; ++y) memcpy((uint8_t *)d + y * dp, (const uint8_t *)s + y * sp, w);
    return cudaSuccess;
}
cudaError_t cudaStreamCreateWithFlags(cudaStream_t *s, unsigned) { *s = (cudaStream_t)1; return cudaSuccess; }
cudaError_t cudaStreamDestroy(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaGetDevice(int *d) { *d = 0; return cudaSuccess; }
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaGetDeviceCount(int *n) { *n = 1; return cudaSuccess; }

tc_frame_buf_t *tcb_host_frame_alloc(int width, int height, int) {
    tc_frame_buf_t *f = (tc_frame_buf_t *)calloc(1, sizeof(tc_frame_buf_t));
    f->width = width;
    f->height = height;
    f->stride_y = ((width + 63) / 64) * 64;
    f->stride_c = ((width / 2 + 63) / 64) * 64;
    cudaMalloc((void **)&f->y, (size_t)f->stride_y * height);
    cudaMalloc((void **)&f->cb, (size_t)f->stride_c * (height / 2));
    cudaMalloc((void **)&f->cr, (size_t)f->stride_c * (height / 2));
    memset(f->y, 0, (size_t)f->stride_y * height);
    memset(f->cb, 0, (size_t)f->stride_c * (height / 2));
    memset(f->cr, 0, (size_t)f->stride_c * (height / 2));
    return f;
}
void tcb_host_frame_free(tc_frame_buf_t *f) {
    if (!f) return;
    cudaFree(f->y); cudaFree(f->cb); cudaFree(f->cr);
    free(f);
}
}

// ----------------------------------------------------------------- kernel

static FrameParams g_last;            // parameters of the last launch
static int g_fill = -1;               // luma value the fake reconstruction writes
static bool g_give_up = false;        // it reports a wait that ran out
static int g_before = -1, g_ref = -1; // luma of the reconstruction and of the first reference at the launch

namespace tcb {
std::atomic<long long> g_alloc_countdown{-1};
cudaError_t init_device_tables() { return cudaSuccess; }
cudaError_t upload_legacy_tables() { return cudaSuccess; }
cudaError_t launch_legacy_decode(const legacy::LFrame &, const int *, int, cudaStream_t) { return cudaSuccess; }

static void check_plane(const uint8_t *p, int stride, int w, int h, const char *what) {
    if (!p || w <= 0 || h <= 0) { bad(std::string(what) + ": no samples"); return; }
    if (room(p) < (long long)(h - 1) * stride + w) bad(std::string(what) + ": rows past the plane's end");
    if (w > stride) bad(std::string(what) + ": wider than a row");
}
// The parsed tree of a CTU as the kernel walks it.
static void check_tree(const FrameParams &P, const CtuOut &o, int d, int ctu_x, int ctu_y, int cx, int cy) {
    const int cu = 64 >> d, px = ctu_x + cx * 8, py = ctu_y + cy * 8, h = 4 >> d;
    const bool in = px + cu <= P.W && py + cu <= P.H;
    if (d == 3 && !in) return;
    const Node &nd = o.nodes[qt_index(d, cx, cy)];
    if (d < 3 && (!in || nd.split)) {
        for (int q = 0; q < 4; ++q) check_tree(P, o, d + 1, ctu_x, ctu_y, cx + (q & 1) * h, cy + (q >> 1) * h);
        return;
    }
    if (nd.mvd_x != px * 4 || nd.mvd_y != py * 4) bad("a leaf without its position's vector");
}
cudaError_t launch_decode_items(const FrameParams *d_params, const int *d_items, int n, int *d_status, cudaStream_t) {
    const FrameParams &P = *d_params;
    if (d_items[0] == 0) {            // the picture's first diagonal
        g_before = P.rec_y[0];
        g_ref = P.ref_valid[0] ? P.ref_y[0][0] : -1;
    }
    g_last = P;
    for (int i = 0; i < n; ++i) {
        const int row = (d_items[i] >> 10) & 1023, col = d_items[i] & 1023, x = col * 64, y = row * 64;
        const int w = P.W - x < 64 ? P.W - x : 64, h = P.H - y < 64 ? P.H - y : 64;
        if (w <= 0 || h <= 0) { bad("a CTU outside the frame"); continue; }
        check_plane(P.rec_y, P.stride_y, (x + w + 3) & ~3, y + h, "luma");
        check_plane(P.rec_cb, P.stride_c, (x / 2 + w / 2 + 3) & ~3, (y + h) / 2, "Cb");
        check_plane(P.rec_cr, P.stride_c, (x / 2 + w / 2 + 3) & ~3, (y + h) / 2, "Cr");
        if (row >= P.ctu_rows || col >= P.ctu_cols) bad("a CTU outside the records");
        check_tree(P, P.out[row * P.ctu_cols + col], 0, x, y, 0, 0);
    }
    for (int r = 0; r < MAX_REFS; ++r) {      // vectors clamp to the frame
        check_plane(P.ref_y[r], P.stride_y, P.W, P.H, "reference luma");
        check_plane(P.ref_cb[r], P.stride_c, P.W / 2, P.H / 2, "reference Cb");
        check_plane(P.ref_cr[r], P.stride_c, P.W / 2, P.H / 2, "reference Cr");
    }
    if (g_fill >= 0 && room(P.rec_y) >= (long long)P.stride_y * (P.H - 1) + P.W)
        for (int y = 0; y < P.H; ++y) memset(P.rec_y + (size_t)y * P.stride_y, g_fill, P.W);
    if (g_give_up) *d_status = 1;
    return cudaSuccess;
}
}  // namespace tcb

// ---------------------------------------------------------------- packets

struct Bits {
    std::vector<uint8_t> out;
    int n = 0;
    void put(uint32_t v, int bits) {
        for (int i = bits - 1; i >= 0; --i, ++n) {
            if ((n & 7) == 0) out.push_back(0);
            out.back() |= (uint8_t)((v >> i & 1) << (7 - (n & 7)));
        }
    }
};
static void put_node(Bits &b, int W, int H, int frame_type, int d, int px, int py) {
    const int cu = 64 >> d;
    const bool in = px + cu <= W && py + cu <= H;
    if (!in) {
        if (d < 3)
            for (int q = 0; q < 4; ++q) put_node(b, W, H, frame_type, d + 1, px + (q & 1) * cu / 2, py + (q >> 1) * cu / 2);
        return;
    }
    b.put(0, 1);                       // not split
    if (frame_type) {                  // skipped inter leaf
        b.put(0, 1);
        b.put(1, 1);
        return;
    }
    b.put(1, 1);                       // intra, DC, chroma DC, no levels
    b.put(1, 5);
    b.put(0, 1);
    for (int i = 0; i < (cu / 8) * (cu / 8); ++i) b.put(3, 2);      // 8x8 TU, empty
    for (int i = 0; i < 2 * (cu / 8) * (cu / 8); ++i) b.put(1, 1);
}
static std::vector<uint8_t> packet(int W, int H, int frame_type, int poc, bool reorder = false) {
    Bits b;
    const int flags = (frame_type ? 0 : TC_FLAG_KEY_FRAME | TC_FLAG_RAP) | (reorder ? TC_FLAG_EXT_HEADER : 0);
    b.put(0x544356, 24); b.put(2, 8); b.put(W, 16); b.put(H, 16);
    b.put(flags, 8); b.put(0, 8); b.put(poc, 8); b.put(0, 8); b.put(0, 16);
    if (reorder) b.put(frame_type, 8);
    for (int y = 0; y < H; y += 64)
        for (int x = 0; x < W; x += 64) put_node(b, W, H, frame_type, 0, x, y);
    b.put(0, 24);
    return b.out;
}

static tc_error_t feed(tc_decoder_t *dec, const std::vector<uint8_t> &p, const tc_pixel_t **y, int *ys) {
    const tc_pixel_t *cb, *cr;
    int cbs, crs;
    const tc_error_t e = tc_decoder_decode(dec, p.data(), p.size(), y, ys, &cb, &cbs, &cr, &crs);
    if (e == TC_OK) {     // a caller reads the size that tc_decoder_get_info gives
        int w, h;
        tc_decoder_get_info(dec, &w, &h);
        check_2d(*y, *ys, w, h, "output luma");
        check_2d(cb, cbs, w / 2, h / 2, "output Cb");
        check_2d(cr, crs, w / 2, h / 2, "output Cr");
        if (*ys < w || cbs < w / 2) bad("output rows narrower than the frame");
    }
    return e;
}

// Pictures of the given sizes in turn, a key frame and a P frame each
// (`reorder`: through the display reorder of B-frame streams).  What a caller
// reads beyond a smaller picture is empty.
static void sizes(tc_decoder_t *dec, const std::vector<int> &wh, bool reorder) {
    const tc_pixel_t *y;
    int ys, W, H;
    for (size_t i = 0; i + 1 < wh.size(); i += 2)
        for (int t = 0; t < 2; ++t) {
            g_fill = 10 + (int)i + t;
            if (feed(dec, packet(wh[i], wh[i + 1], t, t, reorder), &y, &ys) != TC_OK) { bad("a packet was refused"); continue; }
            if (g_last.W != wh[i] || g_last.H != wh[i + 1]) bad("the kernel's frame is not the packet's");
            tc_decoder_get_info(dec, &W, &H);
            for (int r = 0; r < H; ++r)
                for (int c = 0; c < W && c < ys; ++c)
                    if (y[(size_t)r * ys + c] != (r < wh[i + 1] && c < wh[i] ? g_fill : 0)) {
                        bad("not the picture just decoded");
                        r = H;
                        break;
                    }
        }
}

// Pictures 0 .. n-1, one of them (`lost`) with a wait that runs out: it is an
// error, and the packets after it find references, picture order and base
// picture as if it had not come.
static void status(tc_decoder_t *dec, int W, int H, int n, int lost, bool key) {
    const tc_pixel_t *y;
    int ys, last = -1;
    std::vector<int> pocs;
    for (int t = 0; t < n; ++t) {
        g_fill = 20 + t;
        g_give_up = t == lost;
        const bool k = t == 0 || (key && t == lost);
        const tc_error_t e = feed(dec, packet(W, H, !k, t), &y, &ys);
        if (e != (t == lost ? TC_ERR_INTERNAL : TC_OK)) bad("status not as expected");
        if (k) pocs.clear();
        const bool cleared = key && lost > 0 && t > lost && pocs.empty();
        if (g_before != (last >= 0 && !cleared ? last : 0)) bad("the picture built on is not the last good one");
        for (int i = 0; i < MAX_REFS; ++i) {
            const bool have = i < (int)pocs.size();
            if (g_last.ref_valid[i] != have) bad("references not those of the good pictures");
            else if (have && g_last.ref_poc[i] != pocs[pocs.size() - 1 - i]) bad("picture order not that of the good pictures");
        }
        if (!pocs.empty() && g_ref != last) bad("the reference is not the last good picture");
        if (t != lost) {
            last = g_fill;
            pocs.push_back(t);
        }
    }
}

int main(int argc, char **argv) {
    if (argc < 6) { fprintf(stderr, "usage\n"); return 2; }
    const std::string what = argv[1];
    std::vector<int> wh;
    for (int i = 4; i < argc; ++i) wh.push_back(atoi(argv[i]));
    tc_decoder_t *dec = tc_decoder_create(atoi(argv[2]), atoi(argv[3]));
    if (!dec) { printf("no decoder\n"); return 2; }
    if (what == "sizes" || what == "reorder") sizes(dec, wh, what == "reorder");
    else if (what == "status" || what == "status_key") status(dec, wh[0], wh[1], wh[2], wh[3], what == "status_key");
    else bad("no such case");
    tc_decoder_destroy(dec);
    if (!g_mem.empty()) bad("memory left behind");
    for (const std::string &s : g_bad) printf("%s\n", s.c_str());
    return g_bad.empty() ? 0 : 1;
}

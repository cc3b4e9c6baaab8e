// tcb_legacy_enc.cuh — encoder of the legacy (v0 / v1) 8x8 block path on the
// CTU engine's parts (included by tcb_engine.cu).
//
// One 512-thread CTA codes one CTU, its blocks in raster order.  The CTU's
// source and reconstruction live in shared memory for the whole CTU; a block
// is a handful of barrier-separated steps in which independent work runs side
// by side on different warps:
//
//   1  reference samples, source variance, source pairs for the search;
//   2  SAD of the 18 intra modes (a warp per mode), the merge SADs, and the
//      previous block's chroma on one more warp;
//   3  inter: the motion searches, one 256-thread team per reference (the
//      engine's me_integer / me_qpel with 8x8 blocks, which leave the
//      prediction);
//   4  the two transform candidates (WHT, DCT), one warp each, on the matrix
//      units;
//   5  decision, reconstruction, record.
//
// What it computes is the block path of tcb_legacy.cuh (reference
// src/encoder.c:1526-2361), which the CPU tests check against the reference;
// tests/test_gpu_legacy.py holds this kernel to the reference's hashes.
//
// Bound: the serial chain of a block (the search's dependent steps), 64 blocks
// a CTU, at most ctu_rows CTUs at a time.  One warp per CTU with every sample
// read from global memory took 55k cycles per inter block.
#pragma once

namespace tcb {
namespace legacy {

__device__ __forceinline__ int ldct4(int k, int n) { return c_dct4[k][n]; }
__device__ __forceinline__ int ldct8(int k, int n) { return c_dct8[k][n]; }

}  // namespace legacy
}  // namespace tcb

#include "tcb_legacy.cuh"

namespace tcb {
namespace legacy {

struct EncCtu {
    uint8_t right[8][8];          // rows 8 by - 1, columns 64..71 of the reconstruction (uncoded: previous frame's)
    uint8_t below[8][8];          // columns 8 bx - 1, rows 64..71
    uint8_t ra[20], rl[20];       // reference runs: samples 0..15, 15 again
    int sad[18], merge_sad[2];
    int var;
    int16_t lev[2][64];           // levels in write order, per transform
    uint8_t rec[2][64];           // reconstructions
    int sse[2], nz[2];
    uint8_t bi[2][64];            // bi-predictions at the searched and the merge vector
    int bi_sad[2];
    uint8_t inter[64];
    int mvx[64], mvy[64];
    uint2 wht[2][32];             // fragments of the 8x8 and 4x4 WHT
    float4 quant[3][3][32];       // luma 8x8, luma 4x4, chroma (QuantLane parts)
};

// Fragment of the Walsh-Hadamard matrix (8, or two 4s on the diagonal) in the
// Cl rows: its sums need no split.
__device__ inline uint2 wht_fragment(int N, int lane) {
    const int m = lane >> 2;
    float v[2];
    for (int e = 0; e < 2; ++e) {
        const int k = 2 * (lane & 3) + e;
        v[e] = N == 4 && (k >> 2) != (m >> 2) ? 0.0f : (float)tmat(0, N, m & (N - 1), k & (N - 1));
    }
    return make_uint2(0u, pack_h2(v[0], v[1]));
}

// Quantiser of a position: dead zone eff / 3, reconstruction offset eff / 2,
// no RDOQ (reference src/quantize.c:101-147).
__device__ inline QuantPos legacy_quant(int eff) {
    QuantPos q(eff, 0);
    q.bias = (float)(eff >> 1);
    return q;
}

// A pass's two results from the MMA sums: DCT by the 14-bit rounding shift,
// WHT rows exactly, WHT columns by (x + N / 2) >> log2 N.
__device__ __forceinline__ void pass_result(const MmaSums &d, bool dct, bool cols, int N, float &a, float &b) {
    if (dct) {
        a = shift14(d.h0, d.l0) - RND;
        b = shift14(d.h1, d.l1) - RND;
    } else if (!cols) {
        a = d.l0 - 8192.0f;
        b = d.l1 - 8192.0f;
    } else {
        const float off = 8192.0f - (float)(N >> 1), k = N == 8 ? 0.125f : 0.25f;
        a = __fmaf_rd(d.l0 - off, k, RND) - RND;
        b = __fmaf_rd(d.l1 - off, k, RND) - RND;
    }
}

// One transform candidate of an 8x8 area (or 4x4 WHTs of chroma) on a warp,
// with code_area's layout.  A level dequantises to at most 2.25 |c| (q eff +
// eff / 2), so row-inverse WHT results stay below 2.25 * 2040 * sqrt(8) < 2^14
// and split into f16 values and remainders of at most 4.
__device__ __forceinline__ AreaCode code_legacy(uint32_t cv, uint32_t pv, bool dct, int N, const uint2 f, const uint2 i,
                                                const QuantLane &q) {
    AreaCode r;
    float a, b;
    MmaSums d = mma_k8(f, h2_sub(bytes_h2(cv), bytes_h2(pv)));
    pass_result(d, dct, false, N, a, b);
    d = mma_k8(f, pack_h2(a, b));
    pass_result(d, dct, true, N, r.c0, r.c1);
    const float a0 = fabsf(r.c0), a1 = fabsf(r.c1);
    r.z0 = a0 >= q.a.z ? 1.0f : 0.0f;
    r.z1 = a1 >= q.b.z ? 1.0f : 0.0f;
    r.q0 = (__fadd_rd(__fmaf_rn(a0, q.a.x, q.a.y), RND) - RND) * r.z0;
    r.q1 = (__fadd_rd(__fmaf_rn(a1, q.b.x, q.b.y), RND) - RND) * r.z1;
    uint32_t hi, lo;
    split_h2(__fmaf_rn(r.q0, q.a.w, q.c.x) * copysignf(r.z0, r.c0), __fmaf_rn(r.q1, q.b.w, q.c.y) * copysignf(r.z1, r.c1),
             hi, lo);
    d = mma_k16(i, hi, lo);
    pass_result(d, dct, false, N, a, b);
    split_h2(a, b, hi, lo);
    d = mma_k16(i, hi, lo);
    pass_result(d, dct, true, N, a, b);
    const int v0 = clampi((int)(pv & 0xFF) + (int)a, 0, 255), v1 = clampi((int)(pv >> 8) + (int)b, 0, 255);
    r.e0 = (int)(cv & 0xFF) - v0;
    r.e1 = (int)(cv >> 8) - v1;
    r.rec = (uint32_t)v0 | (uint32_t)v1 << 8;
    return r;
}

__device__ __forceinline__ QuantLane quant_of(const EncCtu &E, int k, int lane) {
    return {E.quant[k][0][lane], E.quant[k][1][lane], E.quant[k][2][lane]};
}

// Chroma of the block at CTU position (lx, ly) (reference
// src/encoder.c:2192-2268) on one warp: Cb on the first quarter of the area's
// lanes, Cr on the second (the others repeat them).
__device__ __noinline__ void encode_chroma(EncCtu &E, int lx, int ly, int fx, int fy, bool intra, LBlock *out) {
    Smem &S = smem_state();
    const int lane = threadIdx.x & 31, r = (lane >> 2) & 3, cc = 2 * (lane & 1), c = (lane >> 1) & 1;
    const int cx = lx >> 1, cy = ly >> 1;
    uint32_t pv = 128u * 0x101u;
    if (intra) {
        // luma average of the block's top-left 4x4 samples, this lane's two
        const int l0 = RY(S, lx + cc, ly + r), l1 = RY(S, lx + cc + 1, ly + r);
        const int i = (lane & 1) | ((lane >> 1) & 6);     // lane of the quarter: bits 0, 2, 3
        const bool up = fy > 0, left = fx > 0;
        int m = l0 + l1, s = 0;
        if (i < 4) { if (up) s = RC(S, c, cx + i, cy - 1); }
        else if (left) s = RC(S, c, cx - 1, cy + i - 4);
        for (int k = 1; k < 16; k = k == 1 ? 4 : 2 * k) {
            m += __shfl_xor_sync(0xffffffffu, m, k);
            s += __shfl_xor_sync(0xffffffffu, s, k);
        }
        m >>= 4;
        const int dc = up && left ? (s + 4) >> 3 : up || left ? (s + 2) >> 2 : 128;
        pv = (uint32_t)clampi(dc + ((l0 - m) >> 3), 0, 255) | (uint32_t)clampi(dc + ((l1 - m) >> 3), 0, 255) << 8;
    }
    const uint32_t cv = *(const uint16_t *)(S.cur_c[c] + (cy + r) * 32 + cx + cc);
    const uint2 w = E.wht[1][lane];
    const AreaCode a = code_legacy(cv, pv, false, 4, w, w, quant_of(E, 2, lane));
    __syncwarp();
    if (lane < 16) {
        *(uint16_t *)&RC(S, c, cx + cc, cy + r) = (uint16_t)a.rec;
        *(uint32_t *)(out->chroma + c * 16 + r * 4 + cc) = a.levels();
    }
}

// Bi-prediction sample at absolute vector (mvx, mvy) (reference
// src/encoder.c:1688-1706), or the single prediction when b is null.
__device__ __noinline__ int pred_sample(const uint8_t *a, const uint8_t *b, int mvx, int mvy, int x, int y) {
    LumaMC m;
    m.init(a, g_fp.stride_y, g_fp.W, g_fp.H, mvx, mvy, 8);
    int v = m.at(x, y);
    if (b) {
        m.init(b, g_fp.stride_y, g_fp.W, g_fp.H, -mvx, -mvy, 8);
        v = (v + m.at(x, y) + 1) >> 1;
    }
    return v;
}

__device__ __forceinline__ bool median_of(const EncCtu &E, int bi, int &px, int &py) {
    const int bx = bi & 7, by = bi >> 3;
    int ax = 0, ay = 0, bxv = 0, byv = 0, cxv = 0, cyv = 0;
    bool ha = false, hb = false, hc = false;
    if (bx > 0 && E.inter[bi - 1]) { ax = E.mvx[bi - 1]; ay = E.mvy[bi - 1]; ha = true; }
    if (by > 0 && E.inter[bi - 8]) { bxv = E.mvx[bi - 8]; byv = E.mvy[bi - 8]; hb = true; }
    if (by > 0 && bx < 7 && E.inter[bi - 7]) { cxv = E.mvx[bi - 7]; cyv = E.mvy[bi - 7]; hc = true; }
    if (!(ha || hb || hc)) return false;
    if (!ha) { ax = hb ? bxv : cxv; ay = hb ? byv : cyv; }
    if (!hb) { bxv = ha ? ax : cxv; byv = ha ? ay : cyv; }
    if (!hc) { cxv = ha ? ax : bxv; cyv = ha ? ay : byv; }
    px = maxi(mini(ax, bxv), mini(maxi(ax, bxv), cxv));
    py = maxi(mini(ay, byv), mini(maxi(ay, byv), cyv));
    return true;
}

__global__ void __launch_bounds__(NT, 1) legacy_encode_kernel(const LFrame F, const int *__restrict__ items) {
    extern __shared__ __align__(16) uint8_t smem_raw[];
    Smem &S = *reinterpret_cast<Smem *>(smem_raw);
    __shared__ __align__(16) EncCtu E;
    const int item = items[blockIdx.x], row = item >> 10, col = item & 1023;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int ox = col * 64, oy = row * 64, W = F.W, H = F.H;
    const int w = mini(64, W - ox), h = mini(64, H - oy), wc = w >> 1, hc = h >> 1;
    if (tid == 0) { g_fp.W = W; g_fp.H = H; g_fp.stride_y = F.sy; g_fp.search_window = 0; }
    init_fragments(S);
    init_windows(S);
    if (tid >= 128 && tid < 192) E.wht[(tid - 128) >> 5][lane] = wht_fragment(tid < 160 ? 8 : 4, lane);
    if (tid >= NT - 96) {
        const int k = (tid - (NT - 96)) >> 5, r = lane >> 2, c = 2 * (lane & 3);
        const int scale = qscale_of(k == 2 ? clampi(F.qp + 1, 0, 63) : F.qp);
        const int b0 = k == 2 ? 0 : k ? band_rc(4, r & 3, c & 3) : band_rc(8, r, c);
        const int b1 = k == 2 ? 0 : k ? band_rc(4, r & 3, (c & 3) + 1) : band_rc(8, r, c + 1);
        const QuantLane q = QuantLane::make(legacy_quant(eff_of(scale, b0)), legacy_quant(eff_of(scale, b1)));
        E.quant[k][0][lane] = q.a;
        E.quant[k][1][lane] = q.b;
        E.quant[k][2][lane] = q.c;
    }
    // source, and the reconstruction with its borders (samples coded later
    // hold the previous frame's, as the reference reads them)
    for (int i = tid; i < 64 * 64; i += NT) {
        const int y = i >> 6, x = i & 63;
        S.cur_y[i] = (x < w && y < h) ? F.cur_y[(size_t)(oy + y) * F.sy + ox + x] : 0;
    }
    for (int i = tid; i < 2 * 32 * 32; i += NT) {
        const int c = i >> 10, p = i & 1023, y = p >> 5, x = p & 31;
        const uint8_t *src = c ? F.cur_cr : F.cur_cb;
        S.cur_c[c][p] = (x < wc && y < hc) ? src[(size_t)((oy >> 1) + y) * F.sc + (ox >> 1) + x] : 0;
    }
    for (int i = tid; i < 65 * 65; i += NT) {
        const int y = i / 65 - 1, x = i % 65 - 1;
        if (oy + y >= 0 && ox + x >= 0 && y < h && x < w) RY(S, x, y) = F.rec_y[(size_t)(oy + y) * F.sy + ox + x];
    }
    for (int i = tid; i < 2 * 33 * 33; i += NT) {
        const int c = i / (33 * 33), p = i - c * 33 * 33, y = p / 33 - 1, x = p % 33 - 1;
        const uint8_t *src = c ? F.rec_cr : F.rec_cb;
        if ((oy >> 1) + y >= 0 && (ox >> 1) + x >= 0 && y < hc && x < wc)
            RC(S, c, x, y) = src[(size_t)((oy >> 1) + y) * F.sc + (ox >> 1) + x];
    }
    if (tid < 64) {
        const int k = tid & 7, yr = oy + (tid >> 3) * 8 - 1, xr = ox + 64 + k, yb = oy + 64 + k, xb = ox + (tid >> 3) * 8 - 1;
        E.right[tid >> 3][k] = (yr >= 0 && yr < H && xr < W) ? F.rec_y[(size_t)yr * F.sy + xr] : 0;
        E.below[tid >> 3][k] = (xb >= 0 && xb < W && yb < H) ? F.rec_y[(size_t)yb * F.sy + xb] : 0;
        // blocks outside the frame keep the reference's zeroed block info:
        // not intra, motion vector (0, 0)
        E.inter[tid] = 1;
        E.mvx[tid] = 0;
        E.mvy[tid] = 0;
    }
    LBlock *blk = F.blocks + (size_t)(row * F.ctu_cols + col) * BLOCKS;
    if (tid >= 64 && tid < 128) blk[tid - 64].coded = 0;
    SYNC();

    int prev = -1;              // block whose chroma is still to be coded
    bool prev_intra = false;
    for (int b = 0; b < BLOCKS; ++b) {
        const int lx = (b & 7) * 8, ly = (b >> 3) * 8, fx = ox + lx, fy = oy + ly;
        if (fx + 8 > W || fy + 8 > H) continue;
        // ---- 1: references (reference src/predict.c:23-110), variance, pairs
        if (tid < 34) {
            const bool left = tid >= 17, ha = fy > 0, hl = fx > 0;
            const int i = mini(left ? tid - 17 : tid, 15);
            int v = 128;
            if (left && hl) {
                const int y = mini(fy + i, H - 1) - oy;
                v = y < 64 ? RY(S, lx - 1, y) : E.below[b & 7][y - 64];
            } else if (!left && ha) {
                const int x = mini(fx + i, W - 1) - ox;
                v = x < 64 ? RY(S, x, ly - 1) : E.right[b >> 3][x - 64];
            }
            (left ? E.rl : E.ra)[left ? tid - 17 : tid] = (uint8_t)v;
        }
        if (warp == 2) {
            const uint32_t c = *(const uint16_t *)(S.cur_y + (ly + (lane >> 2)) * 64 + lx + 2 * (lane & 3));
            const int o0 = c & 0xFF, o1 = c >> 8;
            const int sum = (int)__reduce_add_sync(0xffffffffu, (unsigned)(o0 + o1)) / 64;
            const int sq = (int)__reduce_add_sync(0xffffffffu, (unsigned)(o0 * o0 + o1 * o1));
            if (lane == 0) E.var = sq / 64 - sum * sum;
        }
        if (warp == 3) {
            const uint8_t *c = S.cur_y + (ly + (lane >> 2)) * 64 + lx + (lane & 3);
            S.cur_pair[lane] = (uint32_t)c[0] | (uint32_t)c[4] << 16;
        }
        const int ftype = F.frame_type;
        int mgx = fx * 4, mgy = fy * 4;
        const bool merge_ok = ftype != 0 && b > 0 && median_of(E, b, mgx, mgy);
        SYNC();
        // ---- 2: intra and merge SADs, the previous block's chroma
        const int px = 2 * (lane & 3), py = lane >> 2;
        const uint32_t cv = *(const uint16_t *)(S.cur_y + (ly + py) * 64 + lx + px);
        const int dc = ((int)__reduce_add_sync(0xffffffffu, lane < 8 ? E.ra[1 + lane] : lane < 16 ? E.rl[lane - 7] : 0u) + 8) >> 4;
        if (warp < 9) {
            for (int m = warp; m < 18; m += 9) {
                const uint32_t pv = (uint32_t)intra_at(E.ra, E.rl, 8, m, dc, px, py) |
                                    (uint32_t)intra_at(E.ra, E.rl, 8, m, dc, px + 1, py) << 8;
                const int v = (int)__reduce_add_sync(0xffffffffu, __vsadu4(cv, pv));
                if (lane == 0) E.sad[m] = v;
            }
        } else if (warp < 11 && merge_ok && warp - 9 < F.n_cand) {
            const int x = mgx >> 2, y = mgy >> 2;
            int v = 0x7FFFFFFF;
            if (x >= 0 && y >= 0 && x + 8 <= W && y + 8 <= H) {
                const uint8_t *p = F.cand_y[warp - 9] + (size_t)(y + py) * F.sy + x + px;
                v = (int)__reduce_add_sync(0xffffffffu, __vsadu4(cv, (uint32_t)p[0] | (uint32_t)p[1] << 8));
            }
            if (lane == 0) E.merge_sad[warp - 9] = v;
        } else if (warp == 15 && prev >= 0) {
            encode_chroma(E, (prev & 7) * 8, (prev >> 3) * 8, ox + (prev & 7) * 8, oy + (prev >> 3) * 8, prev_intra, blk + prev);
        }
        SYNC();
        // Eight fast modes in their order, the other ten when none of them is
        // below 257; the first minimum wins (reference src/encoder.c:1563-1600).
        constexpr uint32_t FAST = 1u << 0 | 1u << 1 | 1u << 2 | 1u << 5 | 1u << 8 | 1u << 9 | 1u << 13 | 1u << 17;
        const bool fast = lane < 18 && (FAST >> lane & 1u);
        const unsigned key = lane < 18 ? (unsigned)E.sad[lane] << 6 | (fast ? 0u : 32u) | (unsigned)lane : 0xFFFFFFFFu;
        unsigned best = __reduce_min_sync(0xffffffffu, fast ? key : 0xFFFFFFFFu);
        if ((best >> 6) > 256) best = __reduce_min_sync(0xffffffffu, key);
        const int best_isad = (int)(best >> 6), best_intra = (int)(best & 31u);
        // ---- 3: motion searches
        int best_sad = SAD_MAX, bmx = 0, bmy = 0, bref = 0, merge_sad = SAD_MAX, merge_sel = 0;
        const uint8_t *pred = nullptr;      // inter prediction of the best candidate
        const bool search = ftype != 0 && best_isad > 32;
        if (search) {
            const MeTeam T(8);
            if (T.g < F.n_cand) {
                me_integer(T, T.g, F.cand_y[T.g], lx, ly, 8, mgx / 4, mgy / 4, F.search_range);
                T.sync();
                me_qpel(T, T.g, S.plane + T.g * plane_words(8), F.cand_y[T.g], 8);
            }
            SYNC();
            for (int ci = 0; ci < F.n_cand; ++ci) {
                if (S.me[ci].best < best_sad) {
                    best_sad = S.me[ci].best; bmx = S.me[ci].mvx; bmy = S.me[ci].mvy; bref = F.cand_sel[ci];
                    pred = S.pred[ci];
                }
                if (merge_ok && E.merge_sad[ci] < merge_sad) { merge_sad = E.merge_sad[ci]; merge_sel = F.cand_sel[ci]; }
            }
            if (ftype == 2 && F.n_cand == 2) {
                if (tid < 128) {
                    const int k = tid >> 6, p = tid & 63;
                    if (!k || merge_ok)
                        E.bi[k][p] = (uint8_t)pred_sample(F.cand_y[0], F.cand_y[1], k ? mgx : bmx, k ? mgy : bmy, p & 7, p >> 3);
                }
                SYNC();
                if (warp < 2) {
                    const int v = (int)__reduce_add_sync(0xffffffffu, __vsadu4(cv, *(const uint16_t *)(E.bi[warp] + 2 * lane)));
                    if (lane == 0) E.bi_sad[warp] = v;
                }
                SYNC();
                if (E.bi_sad[0] < best_sad) { best_sad = E.bi_sad[0]; bref = 2; pred = E.bi[0]; }
                if (merge_ok && E.bi_sad[1] < merge_sad) { merge_sad = E.bi_sad[1]; merge_sel = 2; }
            }
        }
        if (!search) { mgx = fx * 4; mgy = fy * 4; }
        const bool inter = best_sad < best_isad;
        // ---- 4: transform size by variance, WHT and DCT
        const int N = E.var > 512 ? 4 : 8;
        if (warp < 2) {
            const uint32_t pv = inter ? *(const uint16_t *)(pred + 2 * lane)
                                      : (uint32_t)intra_at(E.ra, E.rl, 8, best_intra, dc, px, py) |
                                            (uint32_t)intra_at(E.ra, E.rl, 8, best_intra, dc, px + 1, py) << 8;
            const uint2 f = warp ? S.frag[N == 8 ? 0 : 2][lane] : E.wht[N == 8 ? 0 : 1][lane];
            const uint2 i = warp ? S.frag[N == 8 ? 1 : 3][lane] : f;
            const AreaCode a = code_legacy(cv, pv, warp != 0, N, f, i, quant_of(E, N == 8 ? 0 : 1, lane));
            const int e = N == 8 ? 2 * lane : (py >> 2) * 32 + (px >> 2) * 16 + (py & 3) * 4 + (px & 3);
            *(uint32_t *)(E.lev[warp] + e) = a.levels();
            *(uint16_t *)(E.rec[warp] + 2 * lane) = (uint16_t)a.rec;
            const int sse = (int)__reduce_add_sync(0xffffffffu, (unsigned)(a.e0 * a.e0 + a.e1 * a.e1));
            const int nz = __popc(__ballot_sync(0xffffffffu, a.z0 != 0.0f)) + __popc(__ballot_sync(0xffffffffu, a.z1 != 0.0f));
            if (lane == 0) { E.sse[warp] = sse; E.nz[warp] = nz; }
        }
        SYNC();
        // ---- 5: RD-lite choice, mode decision (merge > skip > inter > intra)
        const long long c0 = E.sse[0] + F.lambda * (4LL * E.nz[0] + 2), c1 = E.sse[1] + F.lambda * (4LL * E.nz[1] + 2);
        const int tt = c1 < c0;
        const bool all_zero = E.nz[tt] == 0;
        const bool is_merge = inter && all_zero && merge_ok && merge_sad < F.qp * F.qp;
        const bool is_skip = inter && !is_merge && (all_zero || best_sad < F.qp * F.qp / 2);
        const bool zero_res = is_merge || is_skip;
        if (tid < 64) {
            uint8_t v;
            if (is_merge) {
                const uint8_t *src = ftype == 2 ? (merge_sel == 1 ? F.bwd_y : F.fwd_y) : F.dpb_y[0];
                const bool bi = ftype == 2 && merge_sel == 2;
                v = (bi ? F.fwd_y && F.bwd_y : src != nullptr)
                        ? (uint8_t)pred_sample(src, bi ? F.bwd_y : nullptr, mgx, mgy, tid & 7, tid >> 3) : 128;
            } else {
                v = zero_res ? pred[tid] : E.rec[tt][tid];
            }
            RY(S, lx + (tid & 7), ly + (tid >> 3)) = v;
        } else if (tid < 96) {
            ((uint32_t *)blk[b].luma)[lane] = zero_res ? 0u : ((const uint32_t *)E.lev[tt])[lane];
        } else if (tid == 96) {
            LBlock &o = blk[b];
            const int mvx = is_merge ? mgx : inter ? bmx : 0, mvy = is_merge ? mgy : inter ? bmy : 0;
            o.coded = 1;
            o.mode = is_merge ? 3 : is_skip ? 0 : inter ? 1 : 2;
            o.intra_mode = (uint8_t)best_intra;
            o.ref = (uint8_t)(is_merge ? merge_sel : inter ? bref : 0);
            o.tid = (uint8_t)((N == 8 ? 2 : 0) | tt);
            o.mvd_x = mvx - mgx;
            o.mvd_y = mvy - mgy;
            E.inter[b] = inter;
            E.mvx[b] = mvx;
            E.mvy[b] = mvy;
        }
        prev = b;
        prev_intra = !inter;
        SYNC();
    }
    if (warp == 15 && prev >= 0)
        encode_chroma(E, (prev & 7) * 8, (prev >> 3) * 8, ox + (prev & 7) * 8, oy + (prev >> 3) * 8, prev_intra, blk + prev);
    SYNC();
    if (w == 64 && h == 64) deblock_tile(S, F.qp);
    for (int i = tid; i < w * h; i += NT) {
        const int y = div_p2(i, w), x = i - y * w;
        F.rec_y[(size_t)(oy + y) * F.sy + ox + x] = RY(S, x, y);
    }
    for (int i = tid; i < 2 * wc * hc; i += NT) {
        const int c = div_p2(i, wc * hc), p = i - c * wc * hc, y = div_p2(p, wc), x = p - y * wc;
        uint8_t *dst = c ? F.rec_cr : F.rec_cb;
        dst[(size_t)((oy >> 1) + y) * F.sc + (ox >> 1) + x] = RC(S, c, x, y);
    }
}

}  // namespace legacy

cudaError_t launch_legacy_encode(const legacy::LFrame &F, const int *d_items, int n, cudaStream_t st) {
    if (n <= 0) return cudaSuccess;
    legacy::legacy_encode_kernel<<<n, NT, sizeof(Smem), st>>>(F, d_items);
    return cudaGetLastError();
}

}  // namespace tcb

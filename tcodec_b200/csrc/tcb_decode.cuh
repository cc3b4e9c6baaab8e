// tcb_decode.cuh — decoder reconstruction of v2 streams (reference
// src/decoder.c:1521-1816): CTUs rebuilt from their parsed records, one launch
// per anti-diagonal (included by tcb_engine.cu).
//
// A CTU is 64 areas of 8x8 luma samples with their two 4x4 chroma blocks.  The
// 16 warps of a CTA take them in z-order; an area of an inter leaf depends on
// nothing in the CTU (the parser has resolved the vectors), one of an intra
// leaf waits until the cells left of and above its leaf are done (references
// beyond them are replicated).  A warp predicts in registers, inverts the
// transform on the matrix units and writes the reconstruction, so an inter CTU
// takes four areas' time a warp and an all-intra one the 15 steps of its inner
// wavefront, without a barrier of the CTA in between.
//
// Bound: latency of an area (a few thousand cycles, most of it the sample-by-
// sample interpolation and the dependent steps of the transform passes), times
// the 31 launches of a 1280x720 picture.  Leaf by leaf with the whole CTA and a
// barrier per step, a packet of a 1280x720 clip took 10.0 ms with four parser
// threads, in this form 4.1 ms.
//
// Levels come from an arbitrary bitstream: the second inverse pass accumulates
// in 64 bits in the reference.  Dequantised levels within +-4095 keep every
// matrix sum below 2^22 and every result inside 16 bits (row results
// <= 4095 * 43284 / 2^14 = 10,818, column results <= 28,580), where the matrix
// form is exact; other areas take plain 64-bit sums.
#pragma once

namespace tcb {

constexpr int NO_LEAF = 0xFFFF;

struct DecSmem {
    alignas(16) uint8_t rec_y[RY_H * RY_W];
    alignas(16) uint8_t rec_c[2][RC_H * RC_W];
    Node nodes[QT_NODES];
    uint16_t leaf[64];           // per cell: depth << 6 | origin cell (8 cy + cx), or NO_LEAF
    uint16_t at[64];             // per cell in z-order: levels before it, / 96
    uint8_t order[64];           // coded cells in z-order (8 cy + cx)
    volatile uint8_t done[64];   // per cell
    int ncell, next, skip_mask[2];
    int eff[2][4];
    unsigned long long tu8mask;
    uint2 frag[2][32];           // inverse 8x8, inverse 4x4
    uint8_t edge[NW][2][EDGE_LEN];
    int scratch[NW][64];
};

// Waits until the cells [x0, x1) x [y0, y1) (a row or a column, at most 8) are
// done.  They come earlier in z-order, so their warps are already running; the
// bound (g_neighbor_wait_limit short sleeps after WAIT_POLLS polls) only guards
// against a fault elsewhere, and the caller then reports it.
__device__ __forceinline__ bool cells_done(const DecSmem &S, int x0, int x1, int y0, int y1, int lane) {
    const int k = lane & 7, n = x1 - x0 + y1 - y0 - 1;
    const int c = (y0 + (y1 - y0 > 1 ? mini(k, n - 1) : 0)) * 8 + x0 + (x1 - x0 > 1 ? mini(k, n - 1) : 0);
    auto done = [&] { return __all_sync(0xffffffffu, S.done[c] || S.leaf[c] == NO_LEAF); };
    for (int i = 0; i < WAIT_POLLS; ++i)
        if (done()) return true;
    const long long limit = g_neighbor_wait_limit;
    for (long long i = 0; i < limit; ++i) {
        __nanosleep(128);
        if (done()) return true;
    }
    return false;
}

// Two luma prediction samples (x, y), (x + 1, y) of the CTU from references r1
// (and r2 at the mirrored vector, averaged) at the absolute vector (mvx, mvy)
// of the leaf at (lx, ly); sample by sample with the reference's edge
// fallbacks (see mc_samples).
__device__ __forceinline__ uint32_t dec_luma_mc(const uint8_t *r1, const uint8_t *r2, int mvx, int mvy, int x, int y) {
    const int s = g_fp.stride_y, W = g_fp.W, H = g_fp.H;
    uint32_t out = 0;
#pragma unroll 1
    for (int e = 0; e < 2; ++e) {
        int v = 0;
#pragma unroll 1
        for (int h = 0; h < (r2 ? 2 : 1); ++h) {
            const uint8_t *ref = h ? r2 : r1;
            const int mx = h ? -mvx : mvx, my = h ? -mvy : mvy;
            const int u = mc_sample(ref, s, W, H, (mx >> 2) + x + e, (my >> 2) + y, mx & 3, my & 3);
            v = h ? (v + u + 1) >> 1 : u;
        }
        out |= (uint32_t)v << (8 * e);
    }
    return out;
}

// Residual of this lane's two positions from their levels: matrix form, or
// 64-bit sums through the warp's scratch when a level is too large.  N = 4:
// four (or two) 4x4 transforms side by side.
__device__ __forceinline__ void dec_residual(DecSmem &S, int warp, int lane, int N, const uint2 f, uint32_t levels,
                                             int eff0, int eff1, int &r0, int &r1) {
    const int d0 = (int16_t)dequant_coeff((int16_t)levels, eff0), d1 = (int16_t)dequant_coeff((int16_t)(levels >> 16), eff1);
    if (__all_sync(0xffffffffu, absi(d0) <= 4095 && absi(d1) <= 4095)) {
        uint32_t hi, lo;
        split_h2((float)d0, (float)d1, hi, lo);
        MmaSums d = mma_k16(f, hi, lo);
        split_h2(shift14(d.h0, d.l0) - RND, shift14(d.h1, d.l1) - RND, hi, lo);
        d = mma_k16(f, hi, lo);
        r0 = (int)(shift14(d.h0, d.l0) - RND);
        r1 = (int)(shift14(d.h1, d.l1) - RND);
        return;
    }
    int *scr = S.scratch[warp];
    const int row = lane >> 2, col = 2 * (lane & 3), cb = N == 8 ? 0 : col & 4, rb = N == 8 ? 0 : row & 4;
    scr[row * 8 + col] = d0;
    scr[row * 8 + col + 1] = d1;
    __syncwarp();
    int t[2];
    for (int e = 0; e < 2; ++e) {
        int acc = 0;
        for (int n = 0; n < N; ++n)
            acc += (N == 8 ? c_dct8[n][col + e] : c_dct4[n][(col + e) & 3]) * scr[row * 8 + cb + n];
        t[e] = (acc + 8192) >> 14;
    }
    __syncwarp();
    scr[row * 8 + col] = t[0];
    scr[row * 8 + col + 1] = t[1];
    __syncwarp();
    int r[2];
    for (int e = 0; e < 2; ++e) {
        long long acc = 0;
        for (int n = 0; n < N; ++n)
            acc += (long long)(N == 8 ? c_dct8[n][row] : c_dct4[n][row & 3]) * scr[(rb + n) * 8 + col + e];
        r[e] = (int16_t)(int)((acc + 8192) >> 14);
    }
    __syncwarp();
    r0 = r[0];
    r1 = r[1];
}

__device__ __forceinline__ uint32_t add_clamp2(uint32_t pv, int r0, int r1) {
    return (uint32_t)clampi((int)(pv & 0xFF) + r0, 0, 255) | (uint32_t)clampi((int)(pv >> 8) + r1, 0, 255) << 8;
}

// One 8x8 area on a warp.
__device__ __forceinline__ void dec_area(DecSmem &S, const CtuOut *rec, int ctu_x, int ctu_y, int cell, int warp,
                                         int *status) {
    const FrameParams &P = g_fp;
    const int lane = threadIdx.x & 31, row = lane >> 2, col = 2 * (lane & 3);
    const int info = S.leaf[cell], depth = info >> 6, ocx = info & 7, ocy = (info >> 3) & 7;
    const int cu = 64 >> depth, gc = cu >> 3, lx = ocx * 8, ly = ocy * 8;
    const int ax = (cell & 7) * 8 - lx, ay = (cell >> 3) * 8 - ly;      // area in the leaf
    const Node nd = S.nodes[qt_index(depth, ocx, ocy)];
    const int px = ctu_x + lx, py = ctu_y + ly, mvx = nd.mvd_x, mvy = nd.mvd_y;   // absolute vector (parser)
    const bool bidir = P.frame_type == 2;
    const int16_t *el = rec->coef + 96 * S.at[ocy * 8 + ocx];
    // ---- references (reference src/decoder.c:1628-1664, 1697-1750)
    const int rf = bidir ? dpb_fwd(P) : -1, rb = bidir ? dpb_bwd(P) : -1;
    int r1 = -1, r2 = -1, kind = CH_DC, c1 = 0, c2 = -1;
    if (nd.intra) {
        if (nd.ch_intra) kind = CH_CFL;
        else if (P.ref_valid[0]) kind = CH_MC;
    } else {
        const int sel = nd.ref_sel < MAX_REFS && P.ref_valid[nd.ref_sel & 3] ? nd.ref_sel : -1;
        if (bidir) {
            if ((nd.bi || nd.skip) && rf >= 0 && rb >= 0) { r1 = rf; r2 = rb; }
            else {
                r1 = nd.bi ? rf : (nd.ref_sel ? rb : rf);
                if (r1 < 0) r1 = rf >= 0 ? rf : rb;
            }
        } else {
            r1 = sel;
        }
        if (bidir && nd.bi) {
            if (rf >= 0 && rb >= 0) { kind = CH_MC; c1 = rf; c2 = rb; }
            else if (rf >= 0 || rb >= 0) { kind = CH_MC; c1 = rf >= 0 ? rf : rb; }
        } else {
            const int r = bidir ? (nd.ref_sel ? rb : rf) : sel;
            if (r >= 0) { kind = CH_MC; c1 = r; }
        }
    }
    const bool fresh = P.fresh_skip && P.frame_type == 1 && P.ref_valid[0];
    if (nd.skip) { kind = CH_MC; c1 = 0; c2 = -1; }
    // ---- wait for the neighbours that are read
    const bool ha = py > 0, hl = px > 0;
    if (nd.intra || (kind != CH_MC && !nd.skip)) {
        bool ok = ocx == 0 || cells_done(S, ocx - 1, ocx, ocy, ocy + gc, lane);
        if (ocy > 0) ok = cells_done(S, ocx, ocx + gc, ocy - 1, ocy, lane) && ok;
        if (!ok && lane == 0) atomicExch(status, 1);
        __threadfence_block();
    }
    // ---- luma prediction
    uint32_t pv = 128u * 0x101u;
    if (nd.intra) {
        // the leaf's reference samples, as build_refs lays them out
        const int n = 4 * cu + 3;
        auto sample = [&](bool left, int i) -> int {
            const int j = mini(i, cu - 1);
            if (left) return hl ? RY(S, lx - 1, ly + j) : (ha ? RY(S, lx, ly - 1) : 128);
            return ha ? RY(S, lx + j, ly - 1) : (hl ? RY(S, lx - 1, ly) : 128);
        };
        for (int i = lane; i < 2 * n; i += 32) {
            const bool horiz = i >= n;
            const int j = (horiz ? i - n : i) - 3 * cu / 2;
            S.edge[warp][horiz][EDGE_BASE + j] = (uint8_t)sample(horiz == (j > 0), j > 0 ? j : 1 - j);
        }
        int sum = 0;
        for (int i = lane + 1; i <= cu; i += 32) sum += sample(false, i) + sample(true, i);
        sum = __reduce_add_sync(0xffffffffu, sum);
        const int above0 = sample(false, 0);
        __syncwarp();
        const int m = nd.intra_mode;
        pv = intra2(S.edge[warp], above0, (sum + cu) >> __ffs(cu), cu, m, m > 1 && m < 18 ? c_ang_disp[m] : 0, ax + col,
                    ay + row);
    } else if (r1 >= 0) {
        pv = dec_luma_mc(P.ref_y[r1], r2 >= 0 ? P.ref_y[r2] : nullptr, mvx, mvy, ax + col, ay + row);
    }
    // ---- luma residual
    if (!nd.skip) {
        const bool t8 = S.tu8mask >> cell & 1ull;
        const int16_t *lv = el + ((ay >> 3) * gc + (ax >> 3)) * 64;
        const int r = row & 3, c = col & 3;
        const uint32_t l = *(const uint32_t *)(lv + (t8 ? 2 * lane : (row >> 2) * 32 + (col >> 2) * 16 + r * 4 + c));
        const int b0 = t8 ? band_rc(8, row, col) : band_rc(4, r, c), b1 = t8 ? band_rc(8, row, col + 1) : band_rc(4, r, c + 1);
        int r0, r1_;
        dec_residual(S, warp, lane, t8 ? 8 : 4, S.frag[t8 ? 0 : 1][lane], l, S.eff[0][b0], S.eff[0][b1], r0, r1_);
        pv = add_clamp2(pv, r0, r1_);
    }
    *(uint16_t *)&RY(S, lx + ax + col, ly + ay + row) = (uint16_t)pv;
    __syncwarp();
    // ---- chroma: Cb on the first quarter of the lanes, Cr on the second
    if (!nd.skip || fresh) {
        const int cs = cu >> 1, r = row & 3, c = (lane >> 1) & 1;
        const int lxc = lx >> 1, lyc = ly >> 1, x = (ax >> 1) + (lane & 1) * 2, y = (ay >> 1) + r;
        uint32_t cv;
        if (kind == CH_MC) {
            const int Wc = P.W >> 1, Hc = P.H >> 1;
            cv = 0;
#pragma unroll 1
            for (int e = 0; e < 2; ++e) {
                int v = chroma_mc_at(c ? P.ref_cr[c1] : P.ref_cb[c1], P.stride_c, Wc, Hc, mvx, mvy, x + e, y);
                if (c2 >= 0)
                    v = (v + chroma_mc_at(c ? P.ref_cr[c2] : P.ref_cb[c2], P.stride_c, Wc, Hc, -mvx, -mvy, x + e, y) + 1) >> 1;
                cv |= (uint32_t)v << (8 * e);
            }
        } else {
            const Leaf L(P, ctu_x, ctu_y, depth, ocx, ocy);
            ChromaModel M;
#pragma unroll 1
            for (int k = 0; k < 2; ++k) {
                const ChromaModel m = chroma_stats(S, L, k);
                if (k == c) M = m;
            }
            cv = (uint32_t)M.dc * 0x101u;
            if (kind == CH_CFL) cv = cfl_pair(S, L, M, x, y);
        }
        __syncwarp();
        if (!nd.skip) {
            const int nt = cs >> 2, t = (ay >> 3) * nt + (ax >> 3);
            const uint32_t l = *(const uint32_t *)(el + cu * cu + c * cs * cs + t * 16 + r * 4 + (lane & 1) * 2);
            const int b0 = band_rc(4, r, (lane & 1) * 2), b1 = band_rc(4, r, (lane & 1) * 2 + 1);
            int r0, r1_;
            dec_residual(S, warp, lane, 4, S.frag[1][lane], l, S.eff[1][b0], S.eff[1][b1], r0, r1_);
            cv = add_clamp2(cv, r0, r1_);
        }
        if (lane < 16) *(uint16_t *)&RC(S, c, lxc + x, lyc + y) = (uint16_t)cv;
    }
    __syncwarp();
    __threadfence_block();
    if (lane == 0 && !(P.lose_area && cell == S.order[0])) S.done[cell] = 1;
}

__global__ void __launch_bounds__(NT, 1)
decode_kernel(const FrameParams *__restrict__ params, const int *__restrict__ items, int *status) {
    __shared__ DecSmem S;
    FrameParams &P = g_fp;   // the shared helpers read the frame from g_fp
    const int item = items[blockIdx.x];
    const int sid = item >> 20, row = (item >> 10) & 1023, col = item & 1023;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    if (tid == 0) P = params[sid];
    if (tid < 64) S.frag[tid >> 5][lane] = dct_fragment(tid < 32 ? 8 : 4, 1, lane);
    SYNC();
    const int ctu_x = col * 64, ctu_y = row * 64;
    const int w = mini(64, P.W - ctu_x), h = mini(64, P.H - ctu_y);
    const int wc = w >> 1, hc = h >> 1;
    const CtuOut *rec = P.out + row * P.ctu_cols + col;
    // Border from the frame being rebuilt; the interior starts from the
    // persistent reconstruction buffer (stale samples are only ever read by
    // streams that skip with stale chroma, as in the reference).  Whole words:
    // strides are multiples of 64, so the words of the last columns lie in
    // their row's padding and those left of x = 0 are skipped.
    for (int i = tid; i < 65 * 17; i += NT) {
        const int y = i / 17 - 1, x = 4 * (i % 17) - 4;
        if (ctu_y + y >= 0 && ctu_x + x >= 0 && y < h && x < w)
            *(uint32_t *)&RY(S, x, y) = *(const uint32_t *)(P.rec_y + (size_t)(ctu_y + y) * P.stride_y + ctu_x + x);
    }
    for (int i = tid; i < 2 * 33 * 9; i += NT) {
        const int c = i >= 33 * 9, p = i - c * 33 * 9, y = p / 9 - 1, x = 4 * (p % 9) - 4;
        if ((ctu_y >> 1) + y >= 0 && (ctu_x >> 1) + x >= 0 && y < hc && x < wc)
            *(uint32_t *)&RC(S, c, x, y) =
                *(const uint32_t *)((c ? P.rec_cr : P.rec_cb) + (size_t)((ctu_y >> 1) + y) * P.stride_c + (ctu_x >> 1) + x);
    }
    for (int i = tid; i < QT_NODES; i += NT) S.nodes[i] = rec->nodes[i];
    if (tid < 8) S.eff[tid >> 2][tid & 3] = tid < 4 ? P.eff_l[tid] : P.eff_c[tid & 3];
    if (tid == 0) { S.tu8mask = rec->tu8mask; S.next = 0; }
    SYNC();
    // ---- the tree's leaves, cells in z-order (thread z < 64)
    if (tid < 64) {
        auto bits = [](int z, int b) { return (z >> b & 1) | (z >> (b + 1) & 2) | (z >> (b + 2) & 4); };
        const int cx = bits(tid, 0), cy = bits(tid, 1), cell = cy * 8 + cx;
        int info = NO_LEAF;
        bool skip = false;
        if (ctu_x + cx * 8 + 8 <= P.W && ctu_y + cy * 8 + 8 <= P.H)
            for (int d = 0; d < 4; ++d) {
                const int m = ~((8 >> d) - 1), nx = cx & m, ny = cy & m, cu = 64 >> d;
                const bool in = ctu_x + nx * 8 + cu <= P.W && ctu_y + ny * 8 + cu <= P.H;
                const Node &nd = S.nodes[qt_index(d, nx, ny)];
                if (d < 3 && (!in || nd.split)) continue;
                info = d << 6 | (ny << 3 | nx);
                skip = nd.skip;
                break;
            }
        S.leaf[cell] = (uint16_t)info;
        S.done[cell] = 0;
        const unsigned coded = __ballot_sync(0xffffffffu, info != NO_LEAF), sk = __ballot_sync(0xffffffffu, skip);
        if (lane == 0) { S.skip_mask[warp] = (int)(coded & ~sk); S.scratch[0][warp] = (int)coded; }
        asm volatile("bar.sync 1, 64;" ::: "memory");
        const unsigned lt = (1u << lane) - 1u;
        const int nl = __popc((unsigned)S.skip_mask[warp] & lt) + (warp ? __popc((unsigned)S.skip_mask[0]) : 0);
        const int nc = __popc(coded & lt) + (warp ? __popc((unsigned)S.scratch[0][0]) : 0);
        S.at[cell] = (uint16_t)nl;
        if (info != NO_LEAF) S.order[nc] = (uint8_t)cell;
        if (tid == 63) S.ncell = nc + (info != NO_LEAF);
    }
    SYNC();
    const int n = S.ncell;
    for (;;) {
        int k = 0;
        if (lane == 0) k = atomicAdd(&S.next, 1);
        k = __shfl_sync(0xffffffffu, k, 0);
        if (k >= n) break;
        dec_area(S, rec, ctu_x, ctu_y, S.order[k], warp, status);
    }
    SYNC();
    if (w == 64 && h == 64) deblock_on(S, P.qp);
    const bool sao = rec->sao_has;
    const int band = clampi(rec->sao_band, 0, 31), off = clampi(rec->sao_offset, -7, 7);
    for (int i = tid; i < 16 * h; i += NT) {
        const int y = i >> 4, x = 4 * (i & 15);
        if (x >= w) continue;
        uint32_t v = *(const uint32_t *)&RY(S, x, y);
        if (sao) {
            uint32_t u = 0;
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                const int p = (int)(v >> (8 * k) & 0xFF);
                u |= (uint32_t)((p >> 3) == band ? clampi(p + off, 0, 255) : p) << (8 * k);
            }
            v = u;
        }
        uint8_t *d = P.rec_y + (size_t)(ctu_y + y) * P.stride_y + ctu_x + x;
        if (x + 4 <= w) *(uint32_t *)d = v;
        else *(uint16_t *)d = (uint16_t)v;     // even sizes
    }
    for (int i = tid; i < 16 * hc; i += NT) {
        const int c = i & 1, y = i >> 4, x = 4 * (i >> 1 & 7);
        if (x >= wc) continue;
        uint8_t *d = (c ? P.rec_cr : P.rec_cb) + (size_t)((ctu_y >> 1) + y) * P.stride_c + (ctu_x >> 1) + x;
        if (x + 4 <= wc) *(uint32_t *)d = *(const uint32_t *)&RC(S, c, x, y);
        else for (int k = 0; x + k < wc; ++k) d[k] = RC(S, c, x + k, y);
    }
}

cudaError_t launch_decode_items(const FrameParams *d_params, const int *d_items, int n, int *d_status,
                                cudaStream_t st) {
    if (n <= 0) return cudaSuccess;
    decode_kernel<<<n, NT, 0, st>>>(d_params, d_items, d_status);
    return cudaGetLastError();
}

}  // namespace tcb

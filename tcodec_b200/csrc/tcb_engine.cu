// tcb_engine.cu — the v2 CTU rate-distortion engine on sm_100a.
//
// One 512-thread CTA encodes one 64x64 CTU end to end, keeping the CTU's
// source, reconstruction, quadtree snapshots and candidate predictions in
// shared memory:
//
//   decide pass  recursive quadtree RDO (reference src/encoder.c:1292-1397
//                qt_split) over leaves (src/encoder.c:562-1290 qt_leaf):
//                inside a leaf the motion searches run on warp groups while
//                the other warps score the intra modes, an 8x8 area a warp on
//                the matrix instructions; then an in-order strict-< scan
//                reproduces the reference's first-minimum tie rule, and the
//                winner is coded into the tile and the CTU's record
//                (src/encoder.c:1450-1456);
//   filters      deblocking of the CTU's inner edges (src/filter.c:175-237)
//                and the luma SAO band-offset choice, rate gate and
//                application (src/filter.c:245-319, src/encoder.c:1463-1506);
//   exports      reconstruction, MV grid (src/encoder.c:1508-1521) and the
//                CTU record the host range coder consumes.
//
// CTUs of one frame run as an anti-diagonal wavefront: CTU (r, c) reads the
// filtered reconstruction of (r, c-1), (r-1, c) and (r-1, c-1) only.  Where that
// leaves SMs idle, helper CTAs share the large leaves of a CTU (see below).
#include <mutex>

#include "tcb_engine.cuh"
#include "tcb_pair16.cuh"
#include "tcb_pixel.cuh"
#include "tcb_launch.h"
#include "tcb_encoder.h"

namespace tcb {

#define SYNC() __syncthreads()

// Code size: what a leaf runs through once stays in the instruction cache only
// if all of it fits (straight-line code costs 2 cycles an instruction below
// 32 KB, 3 below 128 KB and 9 beyond), so loops of a few iterations are kept
// rolled: the compiler's unrolling by four had the functions of a leaf decision
// at 170 KB, now 125 KB (a key frame of 1280x720 22.7 -> 22.0 ms, a P frame of
// 1920x1080 61.0 -> 59.5).

// Optional per-phase cycle counters (build with -DTCB_PHASE_PROFILE); thread
// 0 of each CTA accumulates clock64() deltas into tcb_phase_cycles[].
#ifdef TCB_PHASE_PROFILE
// Slots 0..14 as listed by the profiling reader (2 and 6 are not used);
// 16 + 8 * depth + k: leaf phase k (0..7) of leaves at that quadtree depth;
// 48 + depth: leaf decisions at that depth; 52 + 2 * depth + {0, 1}: integer
// stages and quarter-pel refinement of group 0's searches at that depth.
constexpr int PHASE_SLOTS = 60;
__device__ unsigned long long tcb_phase_cycles[PHASE_SLOTS];
#define PHASE_T0() long long _ph_t = clock64()
#define PHASE(k) do { if (threadIdx.x == 0) { const long long _n = clock64(); \
    atomicAdd(&tcb_phase_cycles[k], (unsigned long long)(_n - _ph_t)); _ph_t = _n; } } while (0)
#define PHASE_D(k, d) do { if (threadIdx.x == 0) { const long long _n = clock64(); \
    atomicAdd(&tcb_phase_cycles[k], (unsigned long long)(_n - _ph_t)); \
    atomicAdd(&tcb_phase_cycles[16 + 8 * (d) + (k)], (unsigned long long)(_n - _ph_t)); _ph_t = _n; } } while (0)
#define COUNT_D(d) do { if (threadIdx.x == 0) atomicAdd(&tcb_phase_cycles[48 + (d)], 1ull); } while (0)
// Inside a motion search, thread 0 of group 0 splits its time into the
// integer stages (slot 11) and the quarter-pel refinement (slot 12).
#define ME_T0() long long _me_t = clock64()
#define ME_MARK(k) do { if (g == 0 && gt == 0) { const long long _n = clock64(); \
    const int _d = blk == 64 ? 0 : blk == 32 ? 1 : blk == 16 ? 2 : 3; \
    atomicAdd(&tcb_phase_cycles[k], (unsigned long long)(_n - _me_t)); \
    atomicAdd(&tcb_phase_cycles[52 + 2 * _d + (k) - 11], (unsigned long long)(_n - _me_t)); _me_t = _n; } } while (0)
// Work counts (thread 0 of the calling group, one atomic per call):
// [0] integer-search SAD pixel differences, [1] quarter-pel SAD pixels,
// [2] 8x8 and [3] 4x4 transform units coded (luma and chroma).
__device__ unsigned long long tcb_op_counts[4];
#define OPCOUNT(k, v) atomicAdd(&tcb_op_counts[k], (unsigned long long)(v))
#else
#define PHASE_T0() do {} while (0)
#define PHASE(k) do {} while (0)
#define PHASE_D(k, d) do {} while (0)
#define COUNT_D(d) do {} while (0)
#define ME_T0() do {} while (0)
#define ME_MARK(k) do {} while (0)
#define OPCOUNT(k, v) do {} while (0)
#endif

// A motion-search group: index, thread in it, log2 of its threads (7 or 8).
struct MeTeam {
    int g, gt, lth;
    __device__ __forceinline__ MeTeam(int lth_) : g(threadIdx.x >> lth_), gt(threadIdx.x & ((1 << lth_) - 1)), lth(lth_) {}
    // the group's barrier (named barrier g + 1)
    __device__ __forceinline__ void sync() const {
        asm volatile("bar.sync %0, %1;" ::"r"(g + 1), "r"(1 << lth) : "memory");
    }
};

// Four bytes from any address.  Reads only the aligned words that hold
// p[0..3], so a plane whose last row ends exactly at the end of its
// allocation (no padding) is never read past.
__device__ __forceinline__ uint32_t ld4u(const uint8_t *p) {
    const uintptr_t a = (uintptr_t)p;
    const uint32_t *w = (const uint32_t *)(a & ~(uintptr_t)3);
    const uint32_t lo = __ldg(w);
    if ((a & 3) == 0) return lo;
    return __funnelshift_r(lo, __ldg(w + 1), (uint32_t)(a & 3) * 8);
}

template <class T>
__device__ __forceinline__ uint8_t &RY(T &S, int x, int y) {
    return S.rec_y[(y + RY_OY) * RY_W + x + RY_OX];
}
template <class T>
__device__ __forceinline__ uint8_t &RC(T &S, int c, int x, int y) {
    return S.rec_c[c][(y + RC_OY) * RC_W + x + RC_OX];
}

// The CTU state lives in the kernels' one dynamic shared buffer, and the
// frame parameters of the CTU being encoded or decoded in g_fp (every
// kernel that calls the helpers below fills g_fp first).  Functions compiled
// once (__noinline__, so the kernel keeps a single copy of each: the whole
// engine is far larger than the SM's instruction cache) take them from here
// rather than through their reference parameters, so their accesses stay
// shared-memory accesses instead of generic ones.
__device__ __forceinline__ Smem &smem_state() {
    extern __shared__ __align__(16) uint8_t smem_raw[];
    return *reinterpret_cast<Smem *>(smem_raw);
}
__shared__ FrameParams g_fp;

struct Leaf {
    int depth, cx, cy, cu, lx, ly, px, py;
    __device__ Leaf(const FrameParams &P, int ctu_x, int ctu_y, int d, int x, int y) {
        depth = d; cx = x; cy = y; cu = 8 << (3 - d);
        lx = x * 8; ly = y * 8; px = ctu_x + lx; py = ctu_y + ly;
    }
};

// Minimum-magnitude MV predictor over left / above / above-right cells
// (reference src/encoder.c:405-427 qt_mvp).
__device__ void mvp_at(const MvCell *grid, int cx, int cy, int &mx, int &my) {
    int ax = 0, ay = 0, bx = 0, by = 0, cxv = 0, cyv = 0;
    bool ha = false, hb = false, hc = false;
    if (cx > 0) { const MvCell m = grid[cy * 8 + cx - 1]; if (!m.intra) { ax = m.dx; ay = m.dy; ha = true; } }
    if (cy > 0) { const MvCell m = grid[(cy - 1) * 8 + cx]; if (!m.intra) { bx = m.dx; by = m.dy; hb = true; } }
    if (cy > 0 && cx < 7) { const MvCell m = grid[(cy - 1) * 8 + cx + 1]; if (!m.intra) { cxv = m.dx; cyv = m.dy; hc = true; } }
    if (!ha && !hb && !hc) { mx = 0; my = 0; return; }
    if (!ha) { ax = hb ? bx : cxv; ay = hb ? by : cyv; }
    if (!hb) { bx = ha ? ax : cxv; by = ha ? ay : cyv; }
    if (!hc) { cxv = ha ? ax : bx; cyv = ha ? ay : by; }
    // squared lengths of 16-bit vectors: at most 2^31
    const uint32_t qa = (uint32_t)(ax * ax) + (uint32_t)(ay * ay);
    const uint32_t qb = (uint32_t)(bx * bx) + (uint32_t)(by * by);
    const uint32_t qc = (uint32_t)(cxv * cxv) + (uint32_t)(cyv * cyv);
    if (qb < qa && qb <= qc) { mx = bx; my = by; }
    else if (qc < qa && qc < qb) { mx = cxv; my = cyv; }
    else { mx = ax; my = ay; }
}

// ====================================================================
// Helper CTAs.  One stream's wavefront keeps at most min(columns, rows) CTUs
// going, a fraction of the SMs.  Launches that leave SMs idle run clusters of
// two or four CTAs: the first encodes the CTU, and for every leaf decision the
// others take their share of the motion searches and of the scoring of the
// intra modes.  They work on their own copy of the source tile, are sent the
// leaf and its intra reference samples, claim scoring items from the first
// CTA's queue, add to its sums and write predictions and vectors into its
// shared memory; nothing else crosses.  What is computed, and from what, does
// not depend on who computes it.
//
// Protocol: the first CTA writes cmd (and the samples) into a helper's shared
// memory, then its cmd_seq, one more than the command before; the helper
// answers by adding 1 to the first CTA's acks once its results are written.
// The first CTA waits for all acks of a command before it sends the next, so a
// helper never reads a command that is being written.  CMD_LEAVE in cmd_seq
// ends a helper; no other word goes with it.
//
// Waits are bounded.  If the first CTA's gives up it reports an error (ctrl[1])
// and is without helpers from then on: it sends no command any more, only
// CMD_LEAVE at its end, because a late helper may still be at the last one
// (its results land in bounds, in a frame that is an error by then).  A helper
// whose wait gives up, or that finds anything but the next command, leaves.
// Every CTA ends at a barrier of the cluster, so no shared memory is released
// while another CTA may still write to it.
//
// Leaves from 32x32 on only (at 16x16 the round trip, about 3,000 cycles, takes
// what the shares give).  A 64x64 / 32x32 leaf of a P frame with four searches
// takes 199,000 / 86,000 cycles alone and 98,000 / 60,000 with three helpers,
// bound by the longest search.
// ====================================================================
enum HelpCmd { HELP_CTU, HELP_LEAF };
constexpr int CMD_LEAVE = 0x7FFFFFFF;

// Bound of a neighbour wait, in back-off iterations (sleeps of 32 ns
// doubling to 2,048 ns): the default 2^22 is about 8.6 s, far above a
// CTU's encode time even when the GPU is time-shared.  Per device; set by
// tcb_set_neighbor_wait_limit.
__device__ long long g_neighbor_wait_limit = 1ll << 22;
// Waits inside a CTU or a cluster poll this often before they begin to sleep
// and count towards that limit (some milliseconds; the longest share of a leaf
// takes 0.1 ms).
constexpr int WAIT_POLLS = 1 << 16;

__device__ __forceinline__ Smem *peer_smem(int rank) {
    uint64_t p;
    asm("mapa.u64 %0, %1, %2;" : "=l"(p) : "l"(&smem_state()), "r"(rank));
    return (Smem *)p;
}
__device__ __forceinline__ int cluster_rank() {
    int r;
    asm("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
__device__ __forceinline__ int cluster_size() {
    int r;
    asm("mov.u32 %0, %%cluster_nctarank;" : "=r"(r));
    return r;
}
__device__ __forceinline__ void cluster_barrier() {
    SYNC();
    asm volatile("barrier.cluster.arrive.aligned;\n\tbarrier.cluster.wait.aligned;" ::: "memory");
}
__device__ __forceinline__ void cluster_fence() { asm volatile("fence.acq_rel.cluster;" ::: "memory"); }
__device__ __forceinline__ int ld_acquire_cluster(const int *p) {
    int v;
    asm volatile("ld.acquire.cluster.s32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}

// The last warp sends a command (c0: HelpCmd) to every helper; a leaf's with
// its intra reference samples.  The caller has seen all earlier acks.
__device__ __noinline__ void send_command(int c0, int c1, int c2, int c3, int c4, int c5) {
    Smem &S = smem_state();
    const int lane = threadIdx.x & 31;
    if (threadIdx.x == 0) S.ack_goal += S.helpers;
    if (threadIdx.x < NT - 32) return;
    const int seq = S.cmd_sent + 1, n = S.helpers;
    __syncwarp();
#pragma unroll 1
    for (int r = 1; r <= n; ++r) {
        Smem *H = peer_smem(r);
        if (c0 == HELP_LEAF) {
#pragma unroll 1
            for (int i = lane; i < 2 * EDGE_LEN / 4; i += 32) ((uint32_t *)H->edge)[i] = ((const uint32_t *)S.edge)[i];
            if (lane == 0) { H->dc = S.dc; H->above0 = S.above0; }
        }
        if (lane < 6) H->cmd[lane] = lane == 0 ? c0 : lane == 1 ? c1 : lane == 2 ? c2 : lane == 3 ? c3 : lane == 4 ? c4 : c5;
    }
    cluster_fence();
    __syncwarp();
    if (lane == 0) {
        S.cmd_sent = seq;
#pragma unroll 1
        for (int r = 1; r <= n; ++r)
            asm volatile("st.release.cluster.s32 [%0], %1;" ::"l"(&peer_smem(r)->cmd_seq), "r"(seq) : "memory");
    }
}
// The helpers' end.  By the last warp.
__device__ __noinline__ void send_leave() {
    if (threadIdx.x < NT - 32) return;
    const int r = threadIdx.x & 31;
    if (r > 0 && r < cluster_size())
        asm volatile("st.release.cluster.s32 [%0], %1;" ::"l"(&peer_smem(r)->cmd_seq), "r"(CMD_LEAVE) : "memory");
}
// Thread 0 waits for the helpers' acks; a barrier of the CTA follows.
__device__ __noinline__ void wait_helpers_slowly(Smem &S, int goal) {
    const long long limit = g_neighbor_wait_limit;
    unsigned ns = 32;
    for (long long i = 0; i < limit; ++i) {
        if (ld_acquire_cluster(&S.acks) >= goal) return;
        __nanosleep(ns);
        if (ns < 1024) ns <<= 1;
    }
    atomicExch(S.error, 1);
    S.helpers = 0;
}
__device__ __forceinline__ void wait_helpers(Smem &S) {
    if (threadIdx.x != 0 || S.helpers == 0) return;
    const int goal = S.ack_goal;
    for (int i = 0; i < WAIT_POLLS; ++i)
        if (ld_acquire_cluster(&S.acks) >= goal) return;
    wait_helpers_slowly(S, goal);
}
// A helper's answer: everything its threads have written is the first CTA's
// to read.
__device__ __forceinline__ void acknowledge() {
    cluster_fence();
    SYNC();
    if (threadIdx.x == 0) {
        cluster_fence();
        atomicAdd(&peer_smem(0)->acks, 1);
    }
}

// ====================================================================
// Motion search on one warp group (reference src/motion.c:384-485): the
// integer stages (me_integer), then, once every search of the leaf is done
// with them, the quarter-sample refinement (me_qpel).  A group is 128
// threads, or 256 when a leaf has at most two searches.
// ====================================================================

// Search patterns (reference src/motion.c:347-367), one nibble (value + 8)
// per point: large hexagon, small hexagon, diamond.  Point 0 is the centre.
__host__ __device__ constexpr uint32_t nib7(int a, int b, int c, int d, int e, int f, int g) {
    return (uint32_t)(a + 8) | (uint32_t)(b + 8) << 4 | (uint32_t)(c + 8) << 8 | (uint32_t)(d + 8) << 12 |
           (uint32_t)(e + 8) << 16 | (uint32_t)(f + 8) << 20 | (uint32_t)(g + 8) << 24;
}
__device__ __forceinline__ void pat_point(int pat, int p, int &dx, int &dy) {
    const uint32_t px = pat == 0 ? nib7(0, -2, 2, -4, 4, -2, 2) : pat == 1 ? nib7(0, -1, 1, -2, 2, -1, 1)
                                                                          : nib7(0, 0, -1, 1, 0, 0, 0);
    const uint32_t py = pat == 0 ? nib7(0, -4, -4, 0, 0, 4, 4) : pat == 1 ? nib7(0, -2, -2, 0, 0, 2, 2)
                                                                         : nib7(0, -1, 0, 0, 1, 0, 0);
    dx = (int)(px >> (4 * p) & 15u) - 8;
    dy = (int)(py >> (4 * p) & 15u) - 8;
}

__device__ __forceinline__ int lg2i(int v) { return 31 - __clz(v); }
// i / d for d > 0, by a shift when d is a power of two (full CTU rows and
// tiles: 64, 32), else by division (partial CTUs at the frame edge).
__device__ __forceinline__ int div_p2(int i, int d) { return (d & (d - 1)) == 0 ? i >> lg2i(d) : i / d; }

// SAD of 16 samples at any address against 16 aligned ones.  Reads only the
// aligned words that hold p[0..15] (see ld4u).
__device__ __forceinline__ unsigned sad16(const uint8_t *p, const uint4 c, unsigned acc) {
    const uintptr_t a = (uintptr_t)p;
    const uint32_t *w = (const uint32_t *)(a & ~(uintptr_t)3), sh = (uint32_t)(a & 3) * 8;
    const uint32_t w0 = __ldg(w), w1 = __ldg(w + 1), w2 = __ldg(w + 2), w3 = __ldg(w + 3);
    const uint32_t w4 = sh ? __ldg(w + 4) : 0u;
    acc += __vsadu4(__funnelshift_r(w0, w1, sh), c.x);
    acc += __vsadu4(__funnelshift_r(w1, w2, sh), c.y);
    acc += __vsadu4(__funnelshift_r(w2, w3, sh), c.z);
    return acc + __vsadu4(__funnelshift_r(w3, w4, sh), c.w);
}
__device__ __forceinline__ unsigned sad8(const uint8_t *p, const uint2 c, unsigned acc) {
    const uintptr_t a = (uintptr_t)p;
    const uint32_t *w = (const uint32_t *)(a & ~(uintptr_t)3), sh = (uint32_t)(a & 3) * 8;
    const uint32_t w0 = __ldg(w), w1 = __ldg(w + 1), w2 = sh ? __ldg(w + 2) : 0u;
    acc += __vsadu4(__funnelshift_r(w0, w1, sh), c.x);
    return acc + __vsadu4(__funnelshift_r(w1, w2, sh), c.y);
}

// The frame plane and block a search works on.
struct MeBlock {
    const uint8_t *ref, *cur;   // reference plane, block in S.cur_y
    int s, W, H, blk;
    __device__ __forceinline__ bool inside(int x, int y) const {
        return x >= 0 && y >= 0 && x + blk <= W && y + blk <= H;
    }
};

// SADs of pattern points p0 .. p0 + K - 1 (K <= 7) around (bx, by), each on
// an eighth of the group (16 or 32 lanes); out-of-frame points get 0x7FFFFFFF
// (reference sad_at).  Lane k of every warp returns point p0 + k's SAD.  The
// results go through part[par], which flips per call: a thread only gets to
// the next call's barrier after all have read this one's.
__device__ __forceinline__ int batch_sads(Smem &S, const MeTeam &T, int &par, const MeBlock &M, int pat, int p0, int K,
                                          int bx, int by, int scale) {
    const int gt = T.gt, lpc = 1 << (T.lth - 3), k = gt >> (T.lth - 3), l = gt & (lpc - 1), lane = gt & 31;
    unsigned v = 0;
    bool in = false;
    if (gt == 0) OPCOUNT(0, K * M.blk * M.blk);
    if (k < K) {
        int dx, dy;
        pat_point(pat, p0 + k, dx, dy);
        const int x = bx + dx * scale, y = by + dy * scale;
        in = M.inside(x, y);
        if (in) {
            const uint8_t *r = M.ref + (size_t)y * M.s + x;
            if (M.blk == 8) {
                if (l < 8) v = sad8(r + (size_t)l * M.s, *(const uint2 *)(M.cur + l * 64), 0);
            } else {
                const int lc = lg2i(M.blk) - 4, n = M.blk << lc;
#pragma unroll 4
                for (int c = l; c < n; c += lpc) {
                    const int row = c >> lc, xo = (c & ((1 << lc) - 1)) * 16;
                    v = sad16(r + (size_t)row * M.s + xo, *(const uint4 *)(M.cur + row * 64 + xo), v);
                }
            }
        }
    }
    v += __shfl_xor_sync(0xffffffffu, v, 8);
    v += __shfl_xor_sync(0xffffffffu, v, 4);
    v += __shfl_xor_sync(0xffffffffu, v, 2);
    v += __shfl_xor_sync(0xffffffffu, v, 1);
    if (lpc == 32) v += __shfl_xor_sync(0xffffffffu, v, 16);
    int *part = S.me[T.g].part[par];
    if (l == 0) part[k] = in ? (int)v : 0x7FFFFFFF;
    T.sync();
    par ^= 1;
    return lane < K ? part[lane] : 0x7FFFFFFF;
}

// ---- small hexagon and diamond of blocks up to 16x16 from a SAD table ----
// Both stages move the running best by at most 2 samples per commit, so
// their candidates are looked up in a table of the (2R+1)^2 integer
// positions around a window centre (R = FrameParams::search_window, 2..5,
// chosen per frame size by the engine tuning; 4 by default): one position
// per thread (two threads, half the rows each, in a group of 256), one
// barrier per table, instead of one barrier round per batch of candidates.
// The table is refilled around the running best when a candidate falls
// outside it (R >= 2 keeps every pattern point of the new centre inside); the
// walk (order of candidates, first-improvement commits) is that of the
// batched stages, on the same SAD values, so R changes the speed and never
// the result.  Two tables alternate, so refilling one never races with a
// lagging thread still reading the other.  The first one, around the start,
// is filled along with the first batch.
//
// A walk is a chain of look-ups, about a dozen a search, and that chain is
// what a small block's search takes: one minimum over (point, SAD + 1) keys
// finds the next event, with "off the table" stored as 0 so that it passes
// the same comparison, and a ring of such entries instead of bounds checks.
__device__ __forceinline__ int window_radius(int r) { return r >= 2 && r <= WIN_RMAX ? r : 4; }
__device__ __forceinline__ int win_index(int dx, int dy, int R) { return (dy + R + 2) * WIN_SIDE + dx + R + 2; }

// "Off the table" everywhere; once per CTU (a fill writes the positions of its
// radius, the same for the whole CTU).
__device__ void init_windows(Smem &S) {
    for (int i = threadIdx.x; i < NGROUP * 2 * WIN_WORDS; i += NT)
        S.me[i / (2 * WIN_WORDS)].win[0][i % (2 * WIN_WORDS)] = 0;
}

__device__ __forceinline__ void fill_sad_window(const MeTeam &T, uint16_t *tab, const MeBlock &M, int wx, int wy, int R) {
    const int N = 2 * R + 1, two = T.lth - 7, gt = T.gt, pos = gt >> two;
    if (gt == 0) OPCOUNT(0, N * N * M.blk * M.blk);
    // pos / N for pos < 128, N = 5, 7, 9, 11
    const int py = pos * (N == 9 ? 7282 : N == 7 ? 9363 : N == 11 ? 5958 : 13108) >> 16, px = pos - py * N;
    const int x = wx + px - R, y = wy + py - R;
    const int rows = M.blk >> two, r0 = (gt & two) * rows;
    const bool in = pos < N * N && M.inside(x, y);
    unsigned v = 0;
    if (in) {
        const uint8_t *r = M.ref + (size_t)(y + r0) * M.s + x, *c = M.cur + r0 * 64;
        if (M.blk == 16) {
#pragma unroll 4
            for (int i = 0; i < rows; ++i) v = sad16(r + (size_t)i * M.s, *(const uint4 *)(c + i * 64), v);
        } else {
#pragma unroll 4
            for (int i = 0; i < rows; ++i) v = sad8(r + (size_t)i * M.s, *(const uint2 *)(c + i * 64), v);
        }
    }
    if (two) v += __shfl_xor_sync(0xffffffffu, v, 1);
    if (pos < N * N) tab[(py + 2) * WIN_SIDE + px + 2] = in ? (uint16_t)(v + 1) : (uint16_t)0xFFFF;
}

// The integer stages of one search: large hexagon (6 points, 2 passes,
// scaled), small hexagon (6, 3), diamond (4, 4); each pass takes its points
// relative to the running best and commits the first improvement
// (reference src/motion.c:398-448).  A pass scores all its remaining points
// at once, one lane per point; the first one that improves is the sequential
// walk's next commit, and the points after it are scored again around it.
// The first batch also takes the centre, whose SAD the search starts from.
__device__ __noinline__ void me_integer(const MeTeam T, int id, const uint8_t *ref, int lx, int ly, int blk, int center_x,
                                        int center_y, int sr) {
    Smem &S = smem_state();
    ME_T0();
    const int g = T.g, gt = T.gt;
    const MeBlock M = {ref, S.cur_y + ly * 64 + lx, g_fp.stride_y, g_fp.W, g_fp.H, blk};
    const int lane = gt & 31;
    int par = 0;
    int bx = clampi(center_x, 0, M.W - blk), by = clampi(center_y, 0, M.H - blk);
    int wx = bx, wy = by;               // table around (wx, wy)
    uint16_t *const tab0 = S.me[g].win[0], *tab = tab0;
    const int R = window_radius(g_fp.search_window);
    if (blk <= 16) fill_sad_window(T, tab, M, wx, wy, R);
    int bsad = 0x7FFFFFFF;
    bool centre = true;
    // batched stages: the large hexagon, from 32x32 on all three
#pragma unroll 1
    for (int pat = 0; pat < (blk <= 16 ? 1 : 3); ++pat) {
        const int npts = pat == 2 ? 4 : 6, scale = pat == 0 ? maxi(1, sr / 4) : 1;
#pragma unroll 1
        for (int it = 0; it < pat + 2; ++it) {
            bool improved = false;
            int p0 = 1;
            while (p0 <= npts) {
                const int base = centre ? 0 : p0;                  // lane k: point base + k
                const int v = batch_sads(S, T, par, M, pat, base, npts + 1 - base, bx, by, scale);
                if (centre) bsad = __shfl_sync(0xffffffffu, v, 0);
                centre = false;
                // SADs are below 2^20: the first improving point has the smallest key
                const unsigned k = __reduce_min_sync(0xffffffffu, v < bsad ? (unsigned)lane << 20 | (unsigned)v : 0xFFFFFFFFu);
                if (k == 0xFFFFFFFFu) break;                       // no point of this pass improves
                const int f = base + (int)(k >> 20);
                int dx, dy;
                pat_point(pat, f, dx, dy);
                bsad = (int)(k & 0xFFFFFu);
                bx += dx * scale;
                by += dy * scale;
                improved = true;
                p0 = f + 1;
            }
            if (!improved) break;
        }
    }
    if (blk <= 16) {
        int c = win_index(bx - wx, by - wy, R), b1 = bsad + 1;
        if (bx - wx > R || bx - wx < -R || by - wy > R || by - wy < -R) {
            tab = tab0 + WIN_WORDS;
            wx = bx; wy = by;
            c = win_index(0, 0, R);
            fill_sad_window(T, tab, M, wx, wy, R);
            T.sync();
        }
#pragma unroll 1
        for (int pat = 1; pat < 3; ++pat) {
            const int npts = pat == 1 ? 6 : 4;
            int ldx, ldy;               // this lane's pattern point (lanes 1..npts)
            pat_point(pat, mini(lane, 6), ldx, ldy);
            const int loff = ldy * WIN_SIDE + ldx;
#pragma unroll 1
            for (int it = 0; it < pat + 2; ++it) {
                bool improved = false;
                int p0 = 1;
                while (p0 <= npts) {
                    unsigned key = 0xFFFFFFFFu;
                    if (lane >= p0 && lane <= npts) {
                        const int v = tab[c + loff];
                        if (v < b1) key = (unsigned)lane << 16 | (unsigned)v;
                    }
                    key = __reduce_min_sync(0xffffffffu, key);
                    if (key == 0xFFFFFFFFu) break;
                    const int f = (int)(key >> 16), v = (int)(key & 0xFFFFu);
                    if (v == 0) {
                        // off the table: refill it around the running best, as
                        // the sequential walk does on reaching this point
                        tab = tab == tab0 ? tab0 + WIN_WORDS : tab0;
                        wx = bx; wy = by;
                        c = win_index(0, 0, R);
                        fill_sad_window(T, tab, M, wx, wy, R);
                        T.sync();
                        p0 = f;
                        continue;
                    }
                    int dx, dy;
                    pat_point(pat, f, dx, dy);
                    b1 = v;
                    bx += dx; by += dy;
                    c += dy * WIN_SIDE + dx;
                    improved = true;
                    p0 = f + 1;
                }
                if (!improved) break;
            }
        }
        bsad = b1 - 1;
    }
    ME_MARK(11);
    if (gt == 0) { S.me[id].bx = bx; S.me[id].by = by; S.me[id].best = bsad; }
}

// ---- quarter-sample refinement from half-sample planes -------------------
// The eight points of reference src/motion.c:450-481, each taken around the
// running best with first-improvement commits, stay within 3 quarter samples
// of the integer best (bx, by).  The group forms once, in the planes of its
// search, the integer samples and the horizontal, vertical and centre half
// samples around the block (unclipped six-tap values biased by 208,
// reference src/motion.c:70-107); a point's sample is then the average of two
// columns of the half-sample grid averaged over two of its rows (a position
// on the grid averages a value with itself, which returns it), clamped, as
// the nine-anchor form of src/motion.c:190-260 has it.  Points whose six-tap
// support leaves the frame take the bilinear form from the integer samples
// (src/motion.c:308-341).
//
// A word holds the samples at x and x + B / 2, so every whole-sample shift is
// an index and every operation works on two samples.  All points still to be
// tried are scored together, a warp per point (per quarter of a point from
// 32x32 on), and their SADs kept per position: after a commit most points
// around the new best are already known.  Bound: shared-memory loads and
// packed integer operations, 9 to 18 instructions per two samples and point
// where one point at a time from bytes took about 70 per sample.
__device__ __forceinline__ int plane_div(int i, int blk) {   // i / plane_stride(blk), i < 5000
    const uint32_t m = blk == 64 ? 65536 / 38 + 1 : blk == 32 ? 65536 / 22 + 1 : blk == 16 ? 65536 / 14 + 1
                                                                                      : 65536 / 10 + 1;
    return (int)((uint32_t)i * m >> 16);
}

// The planes of a block around its integer position (bx, by), every sample
// biased by 208 (integer samples too: 208..463 are in the range the six-tap
// is exact for, see pair_six_tap).
struct Planes {
    uint32_t *I, *H, *V, *D;
    int B, ST;
    __device__ __forceinline__ Planes(uint32_t *area, int blk) : B(blk), ST((blk >> 1) + 6) {
        I = area;
        H = I + (B + 6) * ST;
        V = H + (B + 6) * ST;
        D = V + (B + 1) * ST;
    }
    // Integer samples of rows by - 3 .., columns bx - 3 .. (clamped: samples
    // outside the frame are never part of a point that is used); then, as
    // asked for, horizontal halves at columns bx - 1 .. (word j reads columns
    // j .. j + 5) of every row, vertical halves of rows by - 1 .. at columns
    // bx - 1 .., and centre halves.  All threads of the team.
    __device__ __forceinline__ void build(const MeTeam &T, const uint8_t *ref, int bx, int by, bool h, bool v,
                                          bool d) const {
        const int nthr = 1 << T.lth, half = B >> 1, s = g_fp.stride_y, W = g_fp.W, Hh = g_fp.H;
#pragma unroll 2
        for (int i = T.gt; i < (B + 6) * ST; i += nthr) {
            const int r = plane_div(i, B), x = bx - 3 + i - r * ST;
            const uint8_t *row = ref + (size_t)clampi(by - 3 + r, 0, Hh - 1) * s;
            I[i] = ((uint32_t)__ldg(row + clampi(x, 0, W - 1)) | (uint32_t)__ldg(row + clampi(x + half, 0, W - 1)) << 16) + PAIR_B;
        }
        T.sync();
        if (h)
#pragma unroll 2
            for (int i = T.gt; i < (B + 6) * ST - 5; i += nthr)
                H[i] = pair_six_tap(I[i], I[i + 1], I[i + 2], I[i + 3], I[i + 4], I[i + 5], PAIR_K_HALF);
        if (v)
#pragma unroll 2
            for (int i = T.gt; i < (B + 1) * ST - 2; i += nthr) {
                const uint32_t *q = I + i + 2;
                V[i] = pair_six_tap(q[0], q[ST], q[2 * ST], q[3 * ST], q[4 * ST], q[5 * ST], PAIR_K_HALF);
            }
        T.sync();
        if (d) {
#pragma unroll 2
            for (int i = T.gt; i < (B + 1) * ST - 5; i += nthr) {
                const uint32_t *q = H + i;
                D[i] = pair_six_tap(q[0], q[ST], q[2 * ST], q[3 * ST], q[4 * ST], q[5 * ST], PAIR_K_HALF);
            }
            T.sync();
        }
    }
};
// Position (X, Y) in quarter samples (0..7) from (bx - 1, by - 1): the two
// columns h0, h1 and rows v0, v1 of the half-sample grid it averages.  Even
// ones lie on samples (planes I, V), odd ones between (H, D); rows likewise
// (I, H / V, D).
struct PlanePoint {
    const uint32_t *q00, *q01, *q10, *q11;
    bool four;               // both directions average two values; else q00 and q11 do
    __device__ __forceinline__ PlanePoint(const Planes &A, int X, int Y, int y0) {
        const int h0 = X >> 1, h1 = (X + 1) >> 1, v0 = Y >> 1, v1 = (Y + 1) >> 1;
        auto at = [&](int v, int h) {
            const uint32_t *q = (v & 1) ? ((h & 1) ? A.D : A.V) : ((h & 1) ? A.H + 2 * A.ST : A.I + 2 * A.ST + 2);
            return q + ((v >> 1) + y0) * A.ST + (h >> 1);
        };
        q00 = at(v0, h0); q01 = at(v0, h1); q10 = at(v1, h0); q11 = at(v1, h1);
        four = X & Y & 1;
    }
    __device__ __forceinline__ static uint32_t finish(uint32_t v) {   // clamped, bias removed
        return pair_min(pair_max(v, PAIR_B), PAIR_B + 255u * 0x00010001u) - PAIR_B;
    }
    // the samples of word o
    __device__ __forceinline__ uint32_t value4(int o) const {
        return finish(pair_avg(pair_avg(q00[o], q01[o]), pair_avg(q10[o], q11[o])));
    }
    __device__ __forceinline__ uint32_t value2(int o) const { return finish(pair_avg(q00[o], q11[o])); }
};

// The prediction at (X, Y) into dst (stride B), averaged with what is there
// when `avg`.  All threads of the team.
__device__ __forceinline__ void plane_pred(const MeTeam &T, const Planes &A, int X, int Y, uint8_t *dst, bool avg) {
    const PlanePoint P(A, X, Y, 0);
    const int half = A.B >> 1, lgh = lg2i(half);
#pragma unroll 2
    for (int i = T.gt; i < A.B * half; i += 1 << T.lth) {
        const int y = i >> lgh, x = i & (half - 1);
        uint8_t *d = dst + y * A.B + x;
        uint32_t v = P.four ? P.value4(y * A.ST + x) : P.value2(y * A.ST + x);
        if (avg) v = pair_avg(v, (uint32_t)d[0] | (uint32_t)d[half] << 16);
        d[0] = (uint8_t)v;
        d[half] = (uint8_t)(v >> 16);
    }
}

// One interpolated luma sample (reference src/motion.c:269-304).
__device__ __forceinline__ int mc_sample(const uint8_t *ref, int s, int W, int H, int fx, int fy, int dx, int dy) {
    if (fx >= 2 && fx + 3 < W && fy >= 2 && fy + 3 < H) return luma_hv(ref, s, fx, fy, dx, dy);
    if (fx >= 0 && fy >= 0 && fx + 1 < W && fy + 1 < H) {
        const uint8_t *p = ref + (size_t)fy * s + fx;
        return interp_qpel(interp_qpel(p[0], p[1], dx), interp_qpel(p[s], p[s + 1], dx), dy);
    }
    const int nx = clampi(fx + (dx >= 2 ? 1 : 0), 0, W - 1), ny = clampi(fy + (dy >= 2 ? 1 : 0), 0, H - 1);
    return ref[(size_t)ny * s + nx];
}

// Luma prediction of a B x B block at the absolute quarter-sample vector
// (mvx, mvy), sample by sample, by `nthr` threads (reference
// src/motion.c:493-584); `avg` as in plane_pred.  The per-sample form with its
// edge fallbacks covers the block forms too: samples whose six-tap support is
// inside the frame take the nine-anchor combination, which for a whole-sample
// or one-direction phase gives the copy's and the one-direction filters'
// values (their truncating division differs on negative sums only, which the
// clamp maps to 0), and a whole-sample phase gives the copy everywhere.
__device__ __noinline__ void mc_samples(int t, int nthr, const uint8_t *ref, int mvx, int mvy, int B, uint8_t *dst,
                                        bool avg) {
    const int s = g_fp.stride_y, W = g_fp.W, H = g_fp.H, dx = mvx & 3, dy = mvy & 3, lg = lg2i(B);
#pragma unroll 1
    for (int i = t; i < B * B; i += nthr) {
        const int fx = (mvx >> 2) + (i & (B - 1)), fy = (mvy >> 2) + (i >> lg);
        const int v = mc_sample(ref, s, W, H, fx, fy, dx, dy);
        dst[i] = (uint8_t)(avg ? (v + dst[i] + 1) >> 1 : v);
    }
}

// The same by a team with a plane area of its own: from planes where the
// six-tap support lies inside the frame and the block is large enough to pay
// for them.
__device__ __noinline__ void mc_team(const MeTeam T, uint32_t *area, const uint8_t *ref, int mvx, int mvy, int B,
                                     uint8_t *dst, bool avg) {
    const int fx = mvx >> 2, fy = mvy >> 2, dx = mvx & 3, dy = mvy & 3;
    if (area && B >= 16 && (dx | dy) && fx >= 2 && fy >= 2 && fx + B + 2 < g_fp.W && fy + B + 2 < g_fp.H) {
        const Planes A(area, B);
        A.build(T, ref, fx + 1, fy + 1, dx, dy, dx && dy);
        plane_pred(T, A, dx, dy, dst, avg);
    } else {
        mc_samples(T.gt, 1 << T.lth, ref, mvx, mvy, B, dst, avg);
    }
    T.sync();
}

// Refines search `id` and leaves its prediction in S.pred[id].
__device__ __noinline__ void me_qpel(const MeTeam T, int id, uint32_t *area, const uint8_t *ref, int blk) {
    Smem &S = smem_state();
    ME_T0();
    MeGroup &E = S.me[id];
    const int g = T.g, gt = T.gt;
    const int W = g_fp.W, H = g_fp.H, B = blk, half = B >> 1;
    const int bx = E.bx, by = E.by, lane = gt & 31, warp = gt >> 5, gw = 1 << (T.lth - 5);
    const Planes A(area, B);
    const int ST = A.ST;
    if (gt < QPOS * QPOS) E.tab[gt] = make_int4(0, 0, 0, 0);
    A.build(T, ref, bx, by, true, true, true);

    // Lane p (1..8) holds point p; the points' offsets a nibble each (value +
    // 8): (+-1, 0), (0, +-1), then the corners.
    constexpr uint32_t PX = 0x79798879u, PY = 0x77997988u;
    const bool point = lane >= 1 && lane <= 8;
    const int sh = 4 * (lane - 1) & 31;
    const int ox = (int)(PX >> sh & 15u) - 8, oy = (int)(PY >> sh & 15u) - 8;
    int ux = 3, uy = 3, bsad = E.best, p0 = 1;     // running best: quarter-sample offset + 3
    // Positions scored so far.  Kept in registers, the same in every warp: a
    // warp that looked at the table instead could already see what a faster
    // one has written for the next round, and their barriers would not match.
    unsigned long long known = 0;
    const bool inner = bx >= 3 && by >= 3 && bx + B + 2 < W && by + B + 2 < H;   // every point is a plane point
#pragma unroll 1
    for (;;) {
        const int cx = ux + ox, cy = uy + oy, fx = (4 * bx + cx - 3) >> 2, fy = (4 * by + cy - 3) >> 2;
        const bool act = point && lane >= p0 && (inner || (fx >= 0 && fy >= 0 && fx + B + 1 <= W && fy + B + 1 <= H));
        const int idx = act ? cy * QPOS + cx : 0;
        const unsigned need = __ballot_sync(0xffffffffu, act && !(known >> idx & 1ull));
        if (need) {
            const unsigned long long mine = act ? 1ull << idx : 0ull;
            known |= (unsigned long long)__reduce_or_sync(0xffffffffu, (unsigned)(mine >> 32)) << 32 |
                     __reduce_or_sync(0xffffffffu, (unsigned)mine);
            const int K = __popc(need), lsp = B >= 32 ? 2 : 0, n = (B * half) >> lsp, lgh = lg2i(half);
            if (gt == 0) OPCOUNT(1, K * B * B);
#pragma unroll 1
            for (int it = warp; it < K << lsp; it += gw) {
                unsigned m = need;
                for (int j = it >> lsp; j > 0; --j) m &= m - 1;
                const int fs = 4 * (__ffs((int)m) - 2), part = it & ((1 << lsp) - 1);
                // position in quarter samples from (bx - 1, by - 1): 1..7
                const int X = ux + (int)(PX >> fs & 15u) - 7, Y = uy + (int)(PY >> fs & 15u) - 7;
                const int qfx = bx - 1 + (X >> 2), qfy = by - 1 + (Y >> 2);
                const uint32_t *cur = S.cur_pair + part * n;
                const int y0 = (part * n) >> lgh;
                unsigned acc = 0;
                if (inner || (qfx >= 2 && qfy >= 2 && qfx + B + 2 < W && qfy + B + 2 < H)) {
                    const PlanePoint P(A, X, Y, y0);
                    if (P.four) {
#pragma unroll 4
                        for (int i = lane; i < n; i += 32)
                            acc += __vsadu4(P.value4((i >> lgh) * ST + (i & (half - 1))), cur[i]);
                    } else {
#pragma unroll 4
                        for (int i = lane; i < n; i += 32)
                            acc += __vsadu4(P.value2((i >> lgh) * ST + (i & (half - 1))), cur[i]);
                    }
                } else {
                    const uint32_t *q = A.I + (2 + (Y >> 2) + y0) * ST + 2 + (X >> 2);
                    const uint32_t dx = X & 3, dy = Y & 3, k2 = 0x00020002u;
#pragma unroll 1
                    for (int i = lane; i < n; i += 32) {
                        const int o = (i >> lgh) * ST + (i & (half - 1));
                        const uint32_t t = (((q[o] - PAIR_B) * (4 - dx) + (q[o + 1] - PAIR_B) * dx + k2) >> 2) & 0x00FF00FFu;
                        const uint32_t b = (((q[o + ST] - PAIR_B) * (4 - dx) + (q[o + ST + 1] - PAIR_B) * dx + k2) >> 2) & 0x00FF00FFu;
                        acc += __vsadu4(((t * (4 - dy) + b * dy + k2) >> 2) & 0x00FF00FFu, cur[i]);
                    }
                }
                acc = __reduce_add_sync(0xffffffffu, acc);
                if (lane == 0) ((int *)&E.tab[(Y - 1) * QPOS + X - 1])[part] = (int)acc;
            }
            T.sync();
        }
        const int4 e = E.tab[idx];
        const int v = e.x + e.y + e.z + e.w;       // below 2^20
        const unsigned k = __reduce_min_sync(0xffffffffu, act && v < bsad ? (unsigned)lane << 20 | (unsigned)v : 0xFFFFFFFFu);
        if (k == 0xFFFFFFFFu) break;
        const int f = (int)(k >> 20), fs = 4 * (f - 1);
        bsad = (int)(k & 0xFFFFFu);
        ux += (int)(PX >> fs & 15u) - 8;
        uy += (int)(PY >> fs & 15u) - 8;
        p0 = f + 1;
    }
    ME_MARK(12);
    // the prediction at the refined vector (an integer one, or one whose
    // six-tap support is inside, is a plane point; else sample by sample)
    const int mvx = 4 * bx + ux - 3, mvy = 4 * by + uy - 3, fx = mvx >> 2, fy = mvy >> 2;
    if (!((mvx | mvy) & 3) || (fx >= 2 && fy >= 2 && fx + B + 2 < W && fy + B + 2 < H))
        plane_pred(T, A, ux + 1, uy + 1, S.pred[id], false);
    else
        mc_samples(gt, 1 << T.lth, ref, mvx, mvy, B, S.pred[id], false);
    if (gt == 0) { E.mvx = mvx; E.mvy = mvy; E.best = bsad; S.cand_mvx[id] = mvx; S.cand_mvy[id] = mvy; }
}

// The leaf's searches (bits of `mask`, search k on plane r_k from centre
// (x_k, y_k)), one warp group each: integer stages, refinement, prediction.
// Two groups' planes fit for a 64x64 leaf, so there a third and fourth group
// wait for the first and second to be done with theirs.  The merge
// predictions at vector (mx, my) go to the groups without a search, or
// follow one: P (slot 4): from r0; B: slot 3 from r0, slot 4 from r1, slot 2
// their average with r1 at the mirrored vector (reference
// src/encoder.c:642-647, 855-859); null planes are left out.  No barrier of
// the whole CTA: the other warps score the intra modes meanwhile.
struct MeStart {
    const uint8_t *r0, *r1, *r2, *r3;
    int x0, y0, x1, y1, x2, y2, x3, y3;
    int mx, my;
};
__device__ __noinline__ void me_searches(const Leaf L, uint32_t mask, const MeStart J, int sr, int lth, bool merges,
                                         bool is_b) {
    Smem &S = smem_state();
    const int cu = L.cu, n = __popc(mask);
    const MeTeam T(lth);
    const int teams = NT >> lth;
    uint32_t *area = cu == 64 ? (T.g < PLANES64 ? S.plane + T.g * plane_words(64) : nullptr)
                              : S.plane + T.g * plane_words(cu);
    if (T.g < n) {
        unsigned m = mask;          // the group's search
        if (T.g > 0) m &= m - 1;
        if (T.g > 1) m &= m - 1;
        if (T.g > 2) m &= m - 1;
        const int id = __ffs((int)m) - 1;
        const uint8_t *ref = id == 0 ? J.r0 : id == 1 ? J.r1 : id == 2 ? J.r2 : J.r3;
        me_integer(T, id, ref, L.lx, L.ly, cu, id == 0 ? J.x0 : id == 1 ? J.x1 : id == 2 ? J.x2 : J.x3,
                   id == 0 ? J.y0 : id == 1 ? J.y1 : id == 2 ? J.y2 : J.y3, sr);
        T.sync();                   // S.me[id] is written by one thread
        if (cu == 64 && T.g >= PLANES64)
            asm volatile("bar.sync %0, %1;" ::"r"(NGROUP + 1 + T.g - PLANES64), "r"(2 << lth) : "memory");
        me_qpel(T, id, S.plane + (cu == 64 ? T.g & (PLANES64 - 1) : T.g) * plane_words(cu), ref, cu);
        if (cu == 64 && T.g + PLANES64 < n) {
            T.sync();
            asm volatile("bar.arrive %0, %1;" ::"r"(NGROUP + 1 + T.g), "r"(2 << lth) : "memory");
        }
        if (n < teams) return;      // free groups take the merges
        if (cu == 64) area = nullptr;   // another group may be using it
    }
    if (!merges) return;
    const int g0 = n < teams ? n : 0, ng = teams - g0;   // groups taking merges
    for (int k = T.g - g0; k < (is_b ? 3 : 1); k += ng) {
        T.sync();
        if (!is_b) {
            mc_team(T, area, J.r0, J.mx, J.my, cu, S.pred[K_MRG], false);
        } else if (k == 0) {
            if (J.r0 && J.r1) {
                mc_team(T, area, J.r0, J.mx, J.my, cu, S.pred[K_B0 + 2], false);
                mc_team(T, area, J.r1, -J.mx, -J.my, cu, S.pred[K_B0 + 2], true);
            }
        } else if (k == 1) {
            if (J.r0) mc_team(T, area, J.r0, J.mx, J.my, cu, S.pred[K_B0 + 3], false);
        } else if (J.r1) {
            mc_team(T, area, J.r1, J.mx, J.my, cu, S.pred[K_B0 + 4], false);
        }
    }
}

// ====================================================================
// Reference selection for B-frames (reference src/encoder.c:204-228):
// forward = largest POC below the current one, backward = smallest above.
// ====================================================================
__device__ __forceinline__ int dpb_fwd(const FrameParams &P) {
    int best = -1, bp = -1;
    for (int i = 0; i < MAX_REFS; ++i)
        if (P.ref_valid[i] && P.ref_poc[i] >= 0 && P.ref_poc[i] < P.poc && P.ref_poc[i] > bp) { bp = P.ref_poc[i]; best = i; }
    return best;
}
__device__ __forceinline__ int dpb_bwd(const FrameParams &P) {
    int best = -1, bp = 0x7FFFFFFF;
    for (int i = 0; i < MAX_REFS; ++i)
        if (P.ref_valid[i] && P.ref_poc[i] >= 0 && P.ref_poc[i] > P.poc && P.ref_poc[i] < bp) { bp = P.ref_poc[i]; best = i; }
    return best;
}

// The searches of a leaf (reference src/encoder.c:795-852, 862-933): bit k of
// `mask` is search k of `J`.
struct LeafSearch {
    uint32_t mask;
    int sr;
    MeStart J;
};
__device__ __forceinline__ LeafSearch leaf_searches(const Leaf &L, int mvpx, int mvpy) {
    const FrameParams &P = g_fp;
    const bool fast = P.preset <= 1;
    const int cx0 = (mvpx + L.px * 4) >> 2, cy0 = (mvpy + L.py * 4) >> 2, mx = mvpx + L.px * 4, my = mvpy + L.py * 4;
    if (P.frame_type == 2) {
        const int rf = dpb_fwd(P), rb = dpb_bwd(P);
        const uint8_t *f = rf >= 0 ? P.ref_y[rf] : nullptr, *b = rb >= 0 ? P.ref_y[rb] : nullptr;
        return {(uint32_t)(rf >= 0) | (uint32_t)(rb >= 0) << 1, fast ? 16 : 32,
                {f, b, f, b, cx0, cy0, cx0, cy0, cx0, cy0, cx0, cy0, mx, my}};
    }
    const bool me1 = !fast && P.multiref && P.ref_valid[1];
    const bool glb = !fast && P.glob_valid && (P.glob_x > 16 || P.glob_x < -16 || P.glob_y > 16 || P.glob_y < -16);
    bool tmp = false;
    int tdx = 0, tdy = 0;
    if (!fast && P.ref_valid[0] && P.prev_valid) {
        const int fx = L.px >> 3, fy = L.py >> 3;
        if (fx < P.grid_w && fy < P.grid_h) {
            const MvCell pg = P.prev_grid[fy * P.grid_w + fx];
            if (!pg.intra) { tmp = true; tdx = pg.dx; tdy = pg.dy; }
        }
    }
    return {1u | (uint32_t)me1 << 1 | (uint32_t)glb << 2 | (uint32_t)tmp << 3, fast ? 16 : 24,
            {P.ref_y[0], P.ref_y[1], P.ref_y[0], P.ref_y[0], cx0, cy0, cx0, cy0, (L.px * 4 + P.glob_x) >> 2,
             (L.py * 4 + P.glob_y) >> 2, (L.px * 4 + tdx) >> 2, (L.py * 4 + tdy) >> 2, mx, my}};
}
// The searches CTA `rank` of n takes, in turn.
__device__ __forceinline__ uint32_t search_share(uint32_t mask, int rank, int n) {
    uint32_t mine = 0;
    for (int j = 0; mask; mask &= mask - 1, j = j + 1 == n ? 0 : j + 1)
        if (j == rank) mine |= mask & -mask;
    return mine;
}
// log2 of a team's threads for a CTA's share.
__device__ __forceinline__ int search_team(uint32_t share, int helpers) {
    return g_fp.preset <= 1 || (helpers && __popc(share) <= 2) ? 8 : 7;
}
// The leaf's source samples as pairs, for the searches.
__device__ __forceinline__ void pair_source(Smem &S, const Leaf &L) {
    const int half = L.cu >> 1, lgh = lg2i(half);
#pragma unroll 1
    for (int i = threadIdx.x; i < L.cu * half; i += NT) {
        const uint8_t *c = S.cur_y + (L.ly + (i >> lgh)) * 64 + L.lx + (i & (half - 1));
        S.cur_pair[i] = (uint32_t)c[0] | (uint32_t)c[half] << 16;
    }
}

// ====================================================================
// Leaf helpers
// ====================================================================

// v2 intra reference samples (reference src/predict.c:480-520): sample i of
// the above (left) run, i >= 0, those past the block replicating the last.
//
// An angular mode interpolates at p = 32 (position along its primary run) +
// displacement between samples p / 32 + 1 and p / 32 + 2 of that run, or, for
// p < 0, at -p of the other run (intra_at).  Both cases read one array per
// direction (0: vertical modes, primary run above; 1: horizontal modes):
// entry j > 0 is primary sample j, entry j <= 0 is secondary sample 1 - j, and
// with P = floor(p / 32), f = p mod 32 the prediction is
// (32 E[k] + (E[k + 1] - E[k]) f + 16) >> 5 at k = P + 1 (p >= 0) or
// k = P (p < 0), since -p = 32 (-P - 1) + (32 - f).
__device__ __noinline__ void build_refs(const Leaf L) {
    Smem &S = smem_state();
    const int N = L.cu, n = 4 * N + 3;
    const bool ha = L.py > 0, hl = L.px > 0;
    auto sample = [&](bool left, int i) -> int {
        const int j = mini(i, N - 1);
        if (left) return hl ? RY(S, L.lx - 1, L.ly + j) : (ha ? RY(S, L.lx, L.ly - 1) : 128);
        return ha ? RY(S, L.lx + j, L.ly - 1) : (hl ? RY(S, L.lx - 1, L.ly) : 128);
    };
#pragma unroll 1
    for (int i = threadIdx.x; i < 2 * n; i += NT) {
        const bool horiz = i >= n;
        const int j = (horiz ? i - n : i) - 3 * N / 2;
        S.edge[horiz][EDGE_BASE + j] = (uint8_t)sample(horiz == (j > 0), j > 0 ? j : 1 - j);
    }
    if (threadIdx.x == 0) S.above0 = sample(false, 0);
    if (threadIdx.x >= NT - 96 && threadIdx.x < NT - 64) {
        // DC value (reference src/predict.c:140-161): samples 1..N of each run.
        int sum = 0;
#pragma unroll 1
        for (int i = (threadIdx.x & 31) + 1; i <= N; i += 32) sum += sample(false, i) + sample(true, i);
        sum = __reduce_add_sync(0xffffffffu, sum);
        if ((threadIdx.x & 31) == 0) S.dc = (sum + N) >> __ffs(N);   // / (2 N)
    }
    SYNC();
}

// Intra prediction samples (x, y) and (x + 1, y) of an N x N leaf in the low
// two bytes; disp is the mode's angular displacement (the per-sample form is
// intra_at; reference src/predict.c:117-340).
__device__ __forceinline__ uint32_t intra2(const uint8_t (*edge)[EDGE_LEN], int above0, int dc, int N, int mode, int disp,
                                           int x, int y) {
    if (mode == 0) {
        const uint8_t *ra = edge[0] + EDGE_BASE;
        const int sh = __ffs(N), l = edge[1][EDGE_BASE + y + 1], c = above0;
        const int v0 = (ra[x + 1] * (N - 1 - y) + l * (N - 1 - x) + c * (x + y) + N) >> sh;
        const int v1 = (ra[x + 2] * (N - 1 - y) + l * (N - 2 - x) + c * (x + 1 + y) + N) >> sh;
        return (uint32_t)mini(v0, 255) | (uint32_t)mini(v1, 255) << 8;
    }
    if (mode == 1 || mode > 17) return (uint32_t)dc * 0x101u;
    const bool vert = mode < 9;
    const uint8_t *E = edge[vert ? 0 : 1] + EDGE_BASE + 1;
    const int p0 = vert ? (x << 5) + y * disp : (y << 5) + x * disp, p1 = p0 + (vert ? 32 : disp);
    const uint8_t *e0 = E + (p0 >> 5) + (p0 >> 31), *e1 = E + (p1 >> 5) + (p1 >> 31);
    const int a0 = e0[0], b0 = e0[1], a1 = e1[0], b1 = e1[1];
    const uint32_t v0 = (uint32_t)(32 * a0 + 16 + (b0 - a0) * (p0 & 31)) >> 5;
    const uint32_t v1 = (uint32_t)(32 * a1 + 16 + (b1 - a1) * (p1 & 31)) >> 5;
    return v0 | v1 << 8;
}

// Entry of a candidate list for slot `slot` with the TU sizes `sizes`.
__device__ __forceinline__ int cl_entry(int slot, int sizes) {
    const int m = slot - K_INTRA;
    return slot | sizes | (m > 1 && m < 18 ? (int)c_ang_disp[m] * 65536 : 0);
}
// The intra modes a preset tries, as the first entries of the candidate list.
__device__ __forceinline__ uint32_t intra_modes(int preset) {
    return preset == 0 ? 0x1041u : preset == 1 ? 0x9249u : 0x3FFFFu;
}
__device__ __forceinline__ void list_intra(Smem &S, uint32_t modes, bool use4) {
    const int tid = threadIdx.x;
    if (tid < 18 && (modes >> tid & 1u))
        S.cl[__popc(modes & ((1u << tid) - 1u))] = cl_entry(K_INTRA + tid, CL_8 | (use4 ? CL_4 : 0));
}
// Prediction samples (x, y) and (x + 1, y), x even, of a candidate (list entry e).
__device__ __forceinline__ uint32_t pred2(const Smem &S, int cu, int e, int x, int y) {
    const int slot = e & CL_SLOT;
    if (slot < NPRED) return *(const uint16_t *)(S.pred[slot] + y * cu + x);
    return intra2(S.edge, S.above0, S.dc, cu, slot - K_INTRA, e >> 16, x, y);
}

__device__ __forceinline__ QuantLane quant_lane(const Smem &S, int type, int lane) {
    return {S.quant[type][0][lane], S.quant[type][1][lane], S.quant[type][2][lane]};
}

// Scores the listed candidates: distortion and bits of one 8x8 TU, of four
// 4x4 TUs, or of both per 8x8 area, added to the slots' sums (reference
// src/encoder.c:476-560; the four-TU form has an outer flag bit).
//
// Warps take (candidate, group of areas) items from queue `queue` until it is
// empty: on inter frames the intra modes are scored by the warps that no
// search occupies, and by the others as their searches end.  Bound: issue
// slots (four warps a scheduler).  Both TU sizes share one prediction and run
// interleaved; what a lane adds up over its group's areas is reduced once per
// item.  Slots not in `mask` are left out.  Groups of 4, 2, 2, 1 areas for 64x64 .. 8x8 leaves; an 8x8 leaf's
// single area is split by TU size instead.
template <bool HELP>
__device__ __noinline__ void luma_score(const Leaf L, const int *cl, int ncl, int queue, uint32_t mask) {
    Smem &S = smem_state();
    Smem *const M = HELP ? peer_smem(0) : nullptr;      // a helper's queue and sums are the first CTA's
    // the next item: a helper asks for it one item ahead
    const int lane = threadIdx.x & 31;
    auto claim = [&] { return lane == 0 ? HELP ? atomicAdd(&M->next[queue], 1) : atomicAdd(&S.next[queue], 1) : 0; };
    int ahead = HELP ? claim() : 0;
    const int cu = L.cu, lt = lg2i(cu) - 3, la = 2 * lt;
    const int row = lane >> 2, col = 2 * (lane & 3);
    const uint2 f8 = S.frag[0][lane], i8 = S.frag[1][lane], f4 = S.frag[2][lane], i4 = S.frag[3][lane];
    const QuantLane q8 = quant_lane(S, 0, lane), q4 = quant_lane(S, 1, lane);
#ifdef TCB_PHASE_PROFILE
    if (threadIdx.x < ncl) { OPCOUNT(2, cl[threadIdx.x] & CL_8 ? 1 << la : 0); OPCOUNT(3, cl[threadIdx.x] & CL_4 ? 4 << la : 0); }
#endif
    const int lG = la == 6 ? 2 : la == 0 ? 0 : 1;            // log2 of a group's areas
    const int lg = la == 0 ? 1 : la - lG;                    // log2 of the groups (8x8: TU sizes)
    for (;;) {
        const int it = __shfl_sync(0xffffffffu, HELP ? ahead : claim(), 0);
        if (it >= ncl << lg) break;
        if (HELP) ahead = claim();
        const int group = it & ((1 << lg) - 1);
        const int e = cl[it >> lg], slot = e & CL_SLOT, do_sizes = e & (la == 0 ? (group ? CL_4 : CL_8) : CL_8 | CL_4);
        if (!do_sizes || !(mask >> slot & 1u)) continue;
        const int t0 = la == 0 ? 0 : group << lG;
        AreaSums s8, s4;
        int n8 = 0, n4 = 0;      // last positions' bits
        bool differs = false;
        for (int t = t0; t < t0 + (1 << lG); ++t) {
            const int x = (t & ((1 << lt) - 1)) * 8 + col, y = (t >> lt) * 8 + row;
            const uint32_t cv = *(const uint16_t *)(S.cur_y + (L.ly + y) * 64 + L.lx + x);
            const uint32_t pv = pred2(S, cu, e, x, y);
            differs |= pv != cv;
            auto add8 = [&](const AreaCode &c) {
                s8.add(c);
                const int b = S.last_bits[last8(c, lane)];
                if (lane == 0) n8 += b;
            };
            auto add4 = [&](const AreaCode &c) {
                s4.add(c);
                const int b = S.last_bits[last4(c, lane)];
                if ((lane & 13) == 0) n4 += b;
            };
            if (do_sizes == (CL_8 | CL_4)) {
                const AreaCode c8 = code_area(cv, pv, f8, i8, q8);
                const AreaCode c4 = code_area(cv, pv, f4, i4, q4);
                add8(c8);
                add4(c4);
            } else if (do_sizes == CL_8) {
                add8(code_area(cv, pv, f8, i8, q8));
            } else {
                add4(code_area(cv, pv, f4, i4, q4));
            }
        }
        if ((e & CL_EXACT) && __any_sync(0xffffffffu, differs)) S.inexact = 1;
        int v = 0;   // lanes 0..3: the four sums of the slot
        if (do_sizes & CL_8) {
            const int a = (int)__reduce_add_sync(0xffffffffu, (unsigned)s8.sse);
            const int b = (int)__reduce_add_sync(0xffffffffu, (unsigned)(n8 + s8.bits()));
            v = lane == 0 ? a : lane == 1 ? b : 0;
        }
        if (do_sizes & CL_4) {
            const int a = (int)__reduce_add_sync(0xffffffffu, (unsigned)s4.sse);
            const int b = (int)__reduce_add_sync(0xffffffffu, (unsigned)(n4 + s4.bits()));
            v = lane == 2 ? a : lane == 3 ? b + (1 << lG) : v;
        }
        if (lane < 4) atomicAdd((HELP ? M : &S)->acc[slot][0] + lane, v);
    }
}

// Codes the luma of a leaf with one candidate and TU size (list entry e) into
// the reconstruction tile; `emit` takes the levels in syntax order.  A warp
// per 8x8 area.
__device__ __noinline__ void luma_replay(const Leaf L, int e, int16_t *emit) {
    Smem &S = smem_state();
    const int cu = L.cu, lt = lg2i(cu) - 3;
    const int lane = threadIdx.x & 31, row = lane >> 2, col = 2 * (lane & 3);
    int t = threadIdx.x >> 5;
    if (t >= 1 << (2 * lt)) return;
    const bool d8 = e & CL_8;
    const uint2 f = S.frag[d8 ? 0 : 2][lane], i = S.frag[d8 ? 1 : 3][lane];
    const QuantLane q = quant_lane(S, d8 ? 0 : 1, lane);
    const int pos = d8 ? 2 * lane : (row >> 2) * 32 + (col >> 2) * 16 + (row & 3) * 4 + (col & 3);
    for (; t < 1 << (2 * lt); t += NW) {
        const int x = (t & ((1 << lt) - 1)) * 8 + col, y = (t >> lt) * 8 + row;
        const uint32_t cv = *(const uint16_t *)(S.cur_y + (L.ly + y) * 64 + L.lx + x);
        const AreaCode c = code_area(cv, pred2(S, cu, e, x, y), f, i, q);
        *(uint16_t *)&RY(S, L.lx + x, L.ly + y) = (uint16_t)c.rec;
        *(uint32_t *)(emit + t * 64 + pos) = c.levels();
    }
}

// Chroma DC value and chroma-from-luma model of component c of a leaf, by one
// warp, from its reconstructed neighbours (reference src/predict.c:364-462).
// At most 64 neighbour pairs of 8-bit samples: every sum and product stays
// under 2^29 (n * sum(la * cv) <= 64 * 64 * 255^2), so 32-bit integers give
// the reference's int64 values.
template <class T>
__device__ __forceinline__ ChromaModel chroma_stats(T &S, const Leaf L, int c) {
    const int cs = L.cu >> 1, lxc = L.lx >> 1, lyc = L.ly >> 1, lane = threadIdx.x & 31;
    const bool up = L.py > 0, left = L.px > 0;
    int sl = 0, sc = 0, slc = 0, sl2 = 0;
#pragma unroll 1
    for (int i = lane; i < cs; i += 32) {
        if (up) {
            const int la = (RY(S, L.lx + 2 * i, L.ly - 1) + RY(S, L.lx + 2 * i + 1, L.ly - 1) + 1) >> 1;
            const int cv = RC(S, c, lxc + i, lyc - 1);
            sl += la; sc += cv; slc += la * cv; sl2 += la * la;
        }
        if (left) {
            const int la = (RY(S, L.lx - 2, L.ly + 2 * i) + RY(S, L.lx - 1, L.ly + 2 * i) +
                            RY(S, L.lx - 2, L.ly + 2 * i + 1) + RY(S, L.lx - 1, L.ly + 2 * i + 1) + 2) >> 2;
            const int cv = RC(S, c, lxc - 1, lyc + i);
            sl += la; sc += cv; slc += la * cv; sl2 += la * la;
        }
    }
    const int n = (up ? cs : 0) + (left ? cs : 0);
    sl = (int)__reduce_add_sync(0xffffffffu, (unsigned)sl);
    sc = (int)__reduce_add_sync(0xffffffffu, (unsigned)sc);
    slc = (int)__reduce_add_sync(0xffffffffu, (unsigned)slc);
    sl2 = (int)__reduce_add_sync(0xffffffffu, (unsigned)sl2);
    const int cov = n * slc - sl * sc, vl = n * sl2 - sl * sl;
    int ash = 3;
    if (n > 0 && vl > 0 && cov != 0) {
        const unsigned q = (unsigned)vl / (unsigned)(cov < 0 ? -cov : cov);
        const int sh = q < 1 ? 2 : 31 - __clz((int)q);
        ash = sh < 2 ? 2 : (sh > 5 ? 5 : sh);
    }
    return {n ? (sc + n / 2) >> lg2i(n) : 128, cov >= 0 ? 1 : -1, ash};   // n: cs or 2 cs
}
__device__ __noinline__ void chroma_model(const Leaf L, int c) {
    Smem &S = smem_state();
    const ChromaModel m = chroma_stats(S, L, c);
    if ((threadIdx.x & 31) == 0) S.cmodel[c] = m;
}

// CfL prediction of chroma samples (x, y), (x + 1, y) of a leaf: the model's DC
// plus the scaled difference of the collocated luma from the mean of the 4x4
// tile, whose eight lanes (index bits 0, 2 and 3) call this together.
template <class T>
__device__ __forceinline__ uint32_t cfl_pair(T &S, const Leaf &L, const ChromaModel &M, int x, int y) {
    const uint32_t l0 = *(const uint32_t *)&RY(S, L.lx + 2 * x, L.ly + 2 * y);
    const uint32_t l1 = *(const uint32_t *)&RY(S, L.lx + 2 * x, L.ly + 2 * y + 1);
    const int a0 = (int)__dp4a(l0, 0x0101u, __dp4a(l1, 0x0101u, 2u)) >> 2;
    const int a1 = (int)__dp4a(l0, 0x01010000u, __dp4a(l1, 0x01010000u, 2u)) >> 2;
    int m = a0 + a1;
    m += __shfl_xor_sync(0xffffffffu, m, 1);
    m += __shfl_xor_sync(0xffffffffu, m, 4);
    m += __shfl_xor_sync(0xffffffffu, m, 8);
    m = (m + 8) >> 4;
    return (uint32_t)__viaddmin_s32_relu(M.dc, M.sign * ((a0 - m) >> M.shift), 255) |
           (uint32_t)__viaddmin_s32_relu(M.dc, M.sign * ((a1 - m) >> M.shift), 255) << 8;
}

// A leaf's chroma prediction: DC, CfL (DC plus the scaled difference of the
// collocated luma from its 4x4 mean), or motion compensation, bi-predictive
// with the mirrored vector when r2 >= 0 (reference src/encoder.c:673-699).
enum { CH_DC, CH_CFL, CH_MC };
struct ChromaPred {
    int kind, r1, r2, mvx, mvy;
};

// Chroma coding (reference src/encoder.c:429-475 qt_code_chroma): 4x4 TUs,
// four (option, component, TU) jobs per warp, one on each quarter of the
// area's lanes, from warp `woff` on; predictions are formed in registers (a
// TU is one 4x4 tile, so its CfL mean is a sum over the quarter's lanes).
// One option (nopt 1): prediction K, reconstruction into the tile, levels to
// `emit`.  Two: K and CfL, distortion and bits to S.cacc, reconstruction and
// levels of both to S.cpred / S.clev.
__device__ __noinline__ void chroma_areas(const Leaf L, int nopt, const ChromaPred K, int16_t *emit, int woff) {
    Smem &S = smem_state();
    const FrameParams &P = g_fp;
    const int cs = L.cu >> 1, ln = lg2i(cs) - 2, J = nopt << (2 * ln + 1);
    const int lxc = L.lx >> 1, lyc = L.ly >> 1;
    const int lane = threadIdx.x & 31, r = (lane >> 2) & 3, cc = 2 * (lane & 1);
    const int quarter = ((lane >> 3) & 2) | ((lane >> 1) & 1);
    if (threadIdx.x == 0) OPCOUNT(3, J);
    int base = 4 * (((threadIdx.x >> 5) + NW - woff) & (NW - 1));
    if (base >= J) return;
    const uint2 f4 = S.frag[2][lane], i4 = S.frag[3][lane];
    const QuantLane q = quant_lane(S, 2, lane);
    for (; base < J; base += 4 * NW) {
        const bool act = base + quarter < J;
        const int j = act ? base + quarter : 0;
        const int o = j >> (2 * ln + 1), c = (j >> (2 * ln)) & 1, t = j & ((1 << (2 * ln)) - 1);
        const int x = (t & ((1 << ln) - 1)) * 4 + cc, y = (t >> ln) * 4 + r;
        const uint32_t cv = *(const uint16_t *)(S.cur_c[c] + (lyc + y) * 32 + lxc + x);
        const ChromaModel M = S.cmodel[c];
        uint32_t pv = (uint32_t)M.dc * 0x101u;
        if (K.kind == CH_CFL || nopt == 2) {
            const uint32_t v = cfl_pair(S, L, M, x, y);
            if (K.kind == CH_CFL || o == 1) pv = v;
        }
        if (K.kind == CH_MC && o == 0) {
            const int Wc = P.W >> 1, Hc = P.H >> 1;
            pv = 0;
#pragma unroll 1
            for (int e = 0; e < 2; ++e) {
                int v = chroma_mc_at(c ? P.ref_cr[K.r1] : P.ref_cb[K.r1], P.stride_c, Wc, Hc, K.mvx, K.mvy, x + e, y);
                if (K.r2 >= 0)
                    v = (v + chroma_mc_at(c ? P.ref_cr[K.r2] : P.ref_cb[K.r2], P.stride_c, Wc, Hc, -K.mvx, -K.mvy, x + e, y) + 1) >> 1;
                pv |= (uint32_t)v << (8 * e);
            }
        }
        __syncwarp();
        const AreaCode a = code_area(cv, pv, f4, i4, q);
        if (nopt == 2) {
            AreaSums u;
            u.add(a);
            int d = u.sse, n = u.bits();    // of the quarter's eight lanes: index bits 0, 2 and 3
            for (int m = 1; m < 16; m = m == 1 ? 4 : 2 * m) {
                d += __shfl_xor_sync(0xffffffffu, d, m);
                n += __shfl_xor_sync(0xffffffffu, n, m);
            }
            n += S.last_bits[last4(a, lane)];
            if (act) {
                if ((lane & 13) == 0) {
                    atomicAdd(&S.cacc[o][0], d);
                    atomicAdd(&S.cacc[o][1], n);
                }
                *(uint16_t *)(S.cpred[2 * o + c] + y * cs + x) = (uint16_t)a.rec;
                *(uint32_t *)(S.clev[2 * o + c] + t * 16 + r * 4 + cc) = a.levels();
            }
        } else if (act) {
            *(uint16_t *)&RC(S, c, lxc + x, lyc + y) = (uint16_t)a.rec;
            *(uint32_t *)(emit + c * cs * cs + t * 16 + r * 4 + cc) = a.levels();
        }
    }
}

// Chroma MC of both components into cpred[dst+c] (or straight into the
// recon tile when to_rec).
__device__ __noinline__ void chroma_mc(Smem &, const FrameParams &, const Leaf L, int refi, int mvx, int mvy,
                          int dst, bool to_rec) {
    Smem &S = smem_state();
    const FrameParams &P = g_fp;
    const int cs = L.cu >> 1, Wc = P.W >> 1, Hc = P.H >> 1, lgs = lg2i(cs);
#pragma unroll 1
    for (int i = threadIdx.x; i < 2 * cs * cs; i += NT) {
        const int c = i >> (2 * lgs), p = i & ((1 << (2 * lgs)) - 1), y = p >> lgs, x = p & (cs - 1);
        const uint8_t *ref = c ? P.ref_cr[refi] : P.ref_cb[refi];
        const int v = chroma_mc_at(ref, P.stride_c, Wc, Hc, mvx, mvy, x, y);
        if (to_rec) RC(S, c, (L.lx >> 1) + x, (L.ly >> 1) + y) = (uint8_t)v;
        else S.cpred[dst + c][p] = (uint8_t)v;
    }
    SYNC();
}

// Luma prediction of a leaf into S.pred[0] from plane r1, averaged with r2 at
// the mirrored vector unless null (reference src/encoder.c:642-647, 855-859).
// By the whole CTA.
__device__ void luma_mc(Smem &S, const Leaf &L, const uint8_t *r1, const uint8_t *r2, int mvx, int mvy) {
    mc_samples(threadIdx.x, NT, r1, mvx, mvy, L.cu, S.pred[0], false);
    SYNC();
    if (r2) {
        mc_samples(threadIdx.x, NT, r2, -mvx, -mvy, L.cu, S.pred[0], true);
        SYNC();
    }
}
// A skipped leaf's luma: the prediction in S.pred[0].
__device__ void copy_pred(Smem &S, const Leaf &L) {
    const int lg = lg2i(L.cu);
#pragma unroll 1
    for (int i = threadIdx.x; i < L.cu * L.cu; i += NT) RY(S, L.lx + (i & (L.cu - 1)), L.ly + (i >> lg)) = S.pred[0][i];
}

__device__ void zero_acc(Smem &S) {
    for (int i = threadIdx.x; i < NCAND * 4; i += NT) (&S.acc[0][0][0])[i] = 0;
    if (threadIdx.x < 4) S.cacc[threadIdx.x >> 1][threadIdx.x & 1] = 0;
    if (threadIdx.x == 0) { S.acc64 = 0; S.inexact = 0; S.next[0] = 0; S.next[1] = 0; }
}

// Sum over the CU of |orig - pred| per listed slot into acc[slot][0][0]
// (fast-preset SAD proxy): one warp per (candidate, 8x8 area).
__device__ __noinline__ void sad_areas(const Leaf L, const int *cl, int ncl, uint32_t mask) {
    Smem &S = smem_state();
    const int cu = L.cu, lt = lg2i(cu) - 3, J = ncl << (2 * lt);
    const int lane = threadIdx.x & 31;
    for (int it = threadIdx.x >> 5; it < J; it += NW) {
        const int e = cl[it >> (2 * lt)];
        if (!(mask >> (e & CL_SLOT) & 1u)) continue;
        const int t = it & ((1 << (2 * lt)) - 1);
        const int x = (t & ((1 << lt) - 1)) * 8 + 2 * (lane & 3), y = (t >> lt) * 8 + (lane >> 2);
        const uint32_t cv = *(const uint16_t *)(S.cur_y + (L.ly + y) * 64 + L.lx + x);
        const unsigned s = __reduce_add_sync(0xffffffffu, __vsadu4(cv, pred2(S, cu, e, x, y)));
        if (lane == 0) atomicAdd(&S.acc[e & CL_SLOT][0][0], (int)s);
    }
}

__device__ __forceinline__ long long best_of(const Smem &S, int slot, bool use4, long long lambda,
                                             int &lb, int &dct) {
    const long long d8 = S.acc[slot][0][0];
    const int b8 = S.acc[slot][0][1];
    if (use4) {
        const long long d4 = S.acc[slot][1][0];
        const int b4 = S.acc[slot][1][1];
        if (d4 + lambda * b4 < d8 + lambda * b8) { lb = b4; dct = 0; return d4; }
    }
    lb = b8; dct = 1;
    return d8;
}

// Snapshot / restore of a node's reconstruction and grid cells (rows of a node
// start on 8-byte addresses in luma, on 4-byte ones in chroma).  Compiled once
// for all depths: the decide pass's code should stay in the instruction cache.
//  to, from: snapshot the node is saved to, and the one it is then restored
//  from (-1: none).
__device__ __noinline__ void snap(const Leaf L, int to, int from) {
    Smem &S = smem_state();
    const int cu = L.cu, cs = cu >> 1, gc = cu >> 3, lg = lg2i(cu), d = L.depth;
    const int size = 6 * cu * cu >> 2, step = d == 0 ? 0 : size;   // bytes; from snapshot 0 to 1
    uint8_t *base = d == 0 ? S.snap0[0] : d == 1 ? S.snap1[0] : S.snap2[0];
    const int ny = cu * cu >> 3, nc = cs * cs >> 2;
    if (threadIdx.x < ny) {
        const int i = threadIdx.x;
        uint2 *t = (uint2 *)&RY(S, L.lx + (8 * i & (cu - 1)), L.ly + (8 * i >> lg));
        if (to >= 0) *((uint2 *)(base + to * step) + i) = *t;
        if (from >= 0) *t = *((uint2 *)(base + from * step) + i);
    }
    if (threadIdx.x < 2 * nc) {
        const int i = threadIdx.x, c = i >= nc, p = 4 * (i - c * nc);
        uint32_t *t = (uint32_t *)&RC(S, c, (L.lx >> 1) + (p & (cs - 1)), (L.ly >> 1) + (p >> (lg - 1)));
        if (to >= 0) *((uint32_t *)(base + to * step + cu * cu) + i) = *t;
        if (from >= 0) *t = *((uint32_t *)(base + from * step + cu * cu) + i);
    }
    if (threadIdx.x >= NT - gc * gc) {
        const int i = threadIdx.x - (NT - gc * gc);
        MvCell *g = &S.grid[(L.cy + (i >> (lg - 3))) * 8 + L.cx + (i & (gc - 1))];
        if (to >= 0) S.snap_g[d][to][i] = *g;
        if (from >= 0) *g = S.snap_g[d][from][i];
    }
    SYNC();
}
static_assert(NT >= 64 * 64 / 8, "a thread per 8 luma samples of a snapshot");

// Grid update after a leaf (reference src/encoder.c:1279-1288 / 760-780).
__device__ void grid_update(Smem &S, const Leaf &L, const Node &nd, int mvpx, int mvpy) {
    const int gc = L.cu >> 3, lgg = lg2i(gc);
#pragma unroll 1
    for (int i = threadIdx.x; i < gc * gc; i += NT) {
        const int y = i >> lgg, x = i & (gc - 1);
        MvCell &g = S.grid[(L.cy + y) * 8 + L.cx + x];
        if (nd.intra) g.intra = 1;
        else {
            g.intra = 0;
            g.dx = (int16_t)(mvpx + ((nd.merge || nd.skip) ? 0 : nd.mvd_x));
            g.dy = (int16_t)(mvpy + ((nd.merge || nd.skip) ? 0 : nd.mvd_y));
        }
    }
    SYNC();
}

// ====================================================================
// Leaf coding of a decided node (reference src/encoder.c:587-781): its
// reconstruction into the tile and its levels into the CTU's record, where
// the leaf's place is 96 levels per coded 8x8 cell before it in z-order
// (close_gaps moves the levels up when skipped leaves leave gaps).  A 32x32 or
// 16x16 leaf's levels wait in shared memory until it has won against its
// split.  The last time a leaf of the final tree is coded leaves the record's
// values, so no pass over the final tree is needed.
// `decided`: the decision has just been made; its reference samples, chroma
// model and inter predictions are still in shared memory, and an intra leaf's
// chroma prediction is still to be chosen (src/encoder.c:1194-1221);
// (mvpx, mvpy) is its vector predictor.
// ====================================================================
__device__ __noinline__ void leaf_code(const Leaf L, bool decided, int mvpx, int mvpy) {
    Smem &S = smem_state();
    const FrameParams &P = g_fp;
    Node &node = S.nodes[qt_index(L.depth, L.cx, L.cy)];
    const Node nd = node;
    if (!decided) mvp_at(S.grid, L.cx, L.cy, mvpx, mvpy);
    const int cu = L.cu, cs = cu >> 1;
    int16_t *el = L.depth == 1 ? S.lev1 : L.depth == 2 ? S.lev2 : S.coef + 96 * S.zoff[L.cy * 8 + L.cx];
    int16_t *ec = el + cu * cu;
    const int cl_size = nd.dct_size ? CL_8 : CL_4;
    if (nd.intra) {
        if (!decided) {
            if (threadIdx.x >= NT - 64) chroma_model(L, (threadIdx.x >> 5) & 1);
            build_refs(L);
        }
        luma_replay(L, cl_entry(K_INTRA + nd.intra_mode, cl_size), el);
        SYNC();
        const ChromaPred mc = {P.ref_valid[0] ? CH_MC : CH_DC, 0, -1, mvpx + L.px * 4, mvpy + L.py * 4};
        if (decided && P.preset >= 2) {
            chroma_areas(L, 2, mc, nullptr, 0);
            SYNC();
            const long long lam = P.lambda;
            const int o = S.cacc[1][0] + lam * (S.cacc[1][1] + 4) < S.cacc[0][0] + lam * (S.cacc[0][1] + 1);
            if (threadIdx.x == 0) node.ch_intra = (uint8_t)o;
            const int lg = lg2i(cs);
#pragma unroll 1
            for (int i = threadIdx.x; i < cs * cs; i += NT) {   // two samples of one component
                const int c = i >> (2 * lg - 1), p = 2 * i & (cs * cs - 1), y = p >> lg, x = p & (cs - 1);
                *(uint16_t *)&RC(S, c, (L.lx >> 1) + x, (L.ly >> 1) + y) = *(const uint16_t *)(S.cpred[2 * o + c] + p);
                *(uint32_t *)(ec + 2 * i) = *(const uint32_t *)(S.clev[2 * o + c] + p);
            }
        } else {
            const ChromaPred cfl = {CH_CFL, 0, -1, 0, 0};
            chroma_areas(L, 1, nd.ch_intra ? cfl : mc, ec, 0);
        }
    } else {
        int mvx, mvy;
        if (nd.merge || nd.skip) { mvx = mvpx + L.px * 4; mvy = mvpy + L.py * 4; }
        else { mvx = mvpx + L.px * 4 + nd.mvd_x; mvy = mvpy + L.py * 4 + nd.mvd_y; }
        const bool bidir = P.frame_type == 2;
        // Luma / chroma reference choice.
        int r1 = 0, r2 = -1, cr1 = 0, cr2 = -1;
        bool flat = false, cflat = false;   // no reference at all: 128 / chroma DC
        if (bidir) {
            const int rf = dpb_fwd(P), rb = dpb_bwd(P);
            if (nd.bi) {
                if (rf >= 0 && rb >= 0) { r1 = rf; r2 = rb; }
                else if (rf >= 0) r1 = rf;
                else if (rb >= 0) r1 = rb;
                else flat = true;
                if (rf >= 0 && rb >= 0) { cr1 = rf; cr2 = rb; }
                else if (rf >= 0 || rb >= 0) cr1 = rf >= 0 ? rf : rb;
                else cflat = true;
            } else {
                int rr = nd.ref_sel ? rb : rf;
                if (rr < 0) rr = rf >= 0 ? rf : rb;
                if (rr >= 0) r1 = rr; else flat = true;
                int rc = nd.ref_sel ? rb : rf;
                if (rc < 0) rc = 0;
                cr1 = rc;
            }
        } else {
            const int ri = nd.ref_sel & 3;
            r1 = (ri < MAX_REFS && P.ref_valid[ri]) ? ri : 0;
            cr1 = r1;
        }
        if (!nd.skip) {
            const int src = decided ? S.win_slot : 0;   // the decision's prediction is still in its slot
            if (!decided) {
                if (cflat && threadIdx.x >= NT - 64) chroma_model(L, (threadIdx.x >> 5) & 1);
                if (flat) {
#pragma unroll 1
                    for (int i = threadIdx.x; i < cu * cu; i += NT) S.pred[0][i] = 128;
                    SYNC();
                } else {
                    luma_mc(S, L, P.ref_y[r1], r2 >= 0 ? P.ref_y[r2] : nullptr, mvx, mvy);
                }
            }
            // luma and chroma run side by side on different warps
            const ChromaPred mc = {cflat ? CH_DC : CH_MC, cr1, cr2, mvx, mvy};
            luma_replay(L, src | cl_size, el);
            chroma_areas(L, 1, mc, ec, mini(NW / 2, (cu * cu) >> 6));
        } else {
            luma_mc(S, L, P.ref_y[0], nullptr, mvx, mvy);
            copy_pred(S, L);
            if (P.fresh_skip && P.frame_type == 1 && P.ref_valid[0])
                chroma_mc(S, P, L, 0, mvx, mvy, 0, true);
        }
    }
    grid_update(S, L, nd, mvpx, mvpy);
}

// ====================================================================
// Leaf decision (reference src/encoder.c:784-1277).
// ====================================================================
__device__ __noinline__ long long leaf_decide(const Leaf L) {
    Smem &S = smem_state();
    const FrameParams &P = g_fp;
    const int cu = L.cu, tid = threadIdx.x, lane = tid & 31;
    const bool fast = P.preset <= 1;
    const bool medium = P.preset >= 2;
    const bool key = P.frame_type == 0;
    const bool is_p = P.frame_type == 1;
    const bool is_b = P.frame_type == 2;
    PHASE_T0();
    COUNT_D(L.depth);
    int mvpx, mvpy;
    mvp_at(S.grid, L.cx, L.cy, mvpx, mvpy);
    zero_acc(S);
    // Candidate list: intra modes first (they can be scored before the
    // searches are done), inter candidates after them.
    const bool try_intra = key || cu <= 16 || medium;
    const bool use4 = medium && cu <= 32;
    const uint32_t modes = !try_intra ? 0u : intra_modes(P.preset);
    const int nintra = __popc(modes);
    // slots 2..4 of a B leaf and the merge slot of a P leaf: 8x8 TUs only
    const uint32_t merges = is_b ? 0x1Cu : 1u << K_MRG;
    if (tid >= 32 && tid < 32 + NPRED) {
        const bool m8 = merges >> (tid - 32) & 1u;
        S.cl[nintra + tid - 32] = cl_entry(tid - 32, CL_8 | (use4 && !m8 ? CL_4 : 0) | (is_p && m8 ? CL_EXACT : 0));
    }
    list_intra(S, modes, use4);
    if (!key) pair_source(S, L);
    if (tid >= NT - 64) chroma_model(L, (tid >> 5) & 1);
    build_refs(L);
    const int helpers = fast || cu < 32 ? 0 : S.helpers;
    if (helpers) send_command(HELP_LEAF, L.depth, L.cx, L.cy, mvpx, mvpy);
    PHASE_D(0, L.depth);

    // ---- candidate set -------------------------------------------------
    // Present slots, one bit each: inter candidates 0..4, intra modes from
    // K_INTRA on.
    uint32_t cand = 0;
    if (!key) {
        const LeafSearch M = leaf_searches(L, mvpx, mvpy);
        const uint32_t share = helpers ? search_share(M.mask, 0, helpers + 1) : M.mask;
        me_searches(L, share, M.J, M.sr, search_team(share, helpers), medium, is_b);
        if (!fast) luma_score<false>(L, S.cl, nintra, 0, ~0u);
        if (helpers) wait_helpers(S);
        SYNC();
        PHASE_D(1, L.depth);
        cand = M.mask;
        if (is_p) {
            if (S.me[2].mvx == S.me[0].mvx && S.me[2].mvy == S.me[0].mvy) cand &= ~(1u << K_GLB);
            if (S.me[3].mvx == S.me[0].mvx && S.me[3].mvy == S.me[0].mvy) cand &= ~(1u << K_TMP);
            cand |= (uint32_t)medium << K_MRG;
        } else {
            const uint32_t mrg = medium, hf = M.mask & 1u, hb = M.mask >> 1;
            cand |= (mrg & hf & hb) << 2 | (mrg & hf) << 3 | (mrg & hb) << 4;
        }
    }

    // ---- residual coding / SAD proxies for every candidate --------------
    cand |= modes << K_INTRA;
    if (fast) {
        sad_areas(L, S.cl, nintra + (key ? 0 : NPRED), cand);
        SYNC();
    } else {
        if (key) {
            luma_score<false>(L, S.cl, nintra, 0, ~0u);
            if (helpers) wait_helpers(S);
        } else {
            luma_score<false>(L, S.cl + nintra, NPRED, 1, cand);
        }
        SYNC();
        PHASE_D(3, L.depth);
        if (is_p) {
            // Skip pre-check (src/encoder.c:1064-1142): the merge prediction
            // equals the source luma, then fresh chroma SSE.
            if (!S.inexact && P.ref_valid[0]) {
                chroma_mc(S, P, L, 0, mvpx + L.px * 4, mvpy + L.py * 4, 0, false);
                const int cs = cu >> 1;
                long long ac = 0;
#pragma unroll 1
                for (int p = tid; p < cs * cs; p += NT) {
                    const int y = p >> lg2i(cs), x = p & (cs - 1);
                    const int db = (int)S.cur_c[0][((L.ly >> 1) + y) * 32 + (L.lx >> 1) + x] - (int)S.cpred[0][p];
                    const int dr = (int)S.cur_c[1][((L.ly >> 1) + y) * 32 + (L.lx >> 1) + x] - (int)S.cpred[1][p];
                    ac += db * db + dr * dr;
                }
                ac = __reduce_add_sync(0xffffffffu, (unsigned)ac);
                if (lane == 0 && ac) atomicAdd((unsigned long long *)&S.acc64, (unsigned long long)ac);
                SYNC();
            }
        }
    }

    PHASE_D(4, L.depth);
    // ---- in-order candidate scan (strict <, first minimum wins) ---------
    // Lane k of warp 0 scores slot k (inter candidates, then the intra modes,
    // the order of a sequential scan); lane 23 the skip candidate of a P
    // leaf, which comes between them.  The smallest (cost, position) is the
    // first minimum, as a sequential scan with strict < leaves it.  The node
    // takes the winner's fields, the others keep their defaults (every
    // candidate sets all the fields later candidates could have changed).
    if (tid < 32) {
        constexpr int SKIP_LANE = NCAND;
        const long long lam = P.lambda;
        const bool inter = lane < NPRED, intra = lane >= K_INTRA && lane < NCAND, skip = lane == SKIP_LANE;
        const bool merge = merges >> lane & 1u;      // 8x8-only sums, the MVP's vector
        const int pos = lane < NPRED ? lane : (skip ? NPRED : lane + 1);
        const bool valid = (cand >> lane & 1u) ||
                           (skip && is_p && medium && P.ref_valid[0] && !S.inexact && S.acc64 == 0);
        // extra bits (a nibble per inter slot): 6, 8 for the second reference,
        // and the multiref syntax of a P leaf's searches; 8 for intra, 2 for skip
        const uint32_t ext = !is_p ? 0x66666u : P.multiref ? 0x68788u : 0x66686u;
        const int extra = inter ? (int)(ext >> (4 * lane) & 15u) : skip ? 2 : 8;
        const int f_ref = is_b ? (lane == K_B0 + 1 || lane == K_B0 + 4) : lane == K_ME1;
        int f_dct = 1, f_mx = 0, f_my = 0, bits = extra;
        uint32_t kh = 0xFFFFFFFFu, kl = 0xFFFFFFFFu;
        long long cost = (long long)1 << 58;         // no candidate
        if (valid) {
            if (inter && (!merge || is_p)) {
                // (a P merge carries the first search's vector difference)
                const int v = merge ? K_ME0 : lane;
                f_mx = S.cand_mvx[v] - mvpx - L.px * 4;
                f_my = S.cand_mvy[v] - mvpy - L.py * 4;
                if (!merge) bits += se_bits(f_mx) + se_bits(f_my);
            }
            long long d = 0;
            if (!skip) {
                if (fast) {
                    const long long sad = S.acc[lane][0][0];
                    d = (sad * sad) >> (2 * lg2i(cu));   // / (cu * cu), sad >= 0
                    bits += intra ? 8 : 3;
                } else {
                    int lb;
                    d = best_of(S, lane, use4 && !merge, lam, lb, f_dct);
                    bits += lb;
                }
            }
            cost = d + lam * bits;
        }
        // costs stay below 2^58: distortion < 2^28, lambda <= 2^30, bits < 2^18
        const unsigned long long k = (unsigned long long)cost << 5 | (unsigned)pos;
        kh = (uint32_t)(k >> 32);
        kl = (uint32_t)k;
        const uint32_t mh = __reduce_min_sync(0xffffffffu, kh);
        const uint32_t ml = __reduce_min_sync(0xffffffffu, kh == mh ? kl : 0xFFFFFFFFu);
        if (kh == mh && kl == ml) {
            S.win_slot = skip ? -1 : lane;
            Node &nd = S.nodes[qt_index(L.depth, L.cx, L.cy)];
            nd.intra = intra; nd.skip = skip; nd.merge = inter && merge;
            nd.bi = is_b && lane == K_B0 + 2;
            nd.intra_mode = (uint8_t)(intra ? lane - K_INTRA : 1); nd.intra_cmode = 0; nd.ch_intra = 0;
            nd.ref_sel = (uint8_t)f_ref; nd.dct_size = (uint8_t)f_dct;
            nd.mvd_x = (int16_t)f_mx; nd.mvd_y = (int16_t)f_my;
            nd.split = 0;
            S.best_cost = cost;
        }
    }
    SYNC();

    PHASE_D(5, L.depth);
    const long long best = S.best_cost;
    leaf_code(L, true, mvpx, mvpy);
    PHASE_D(7, L.depth);
    return best;
}

// ====================================================================
// Quadtree recursion (reference src/encoder.c:1292-1397).
// ====================================================================
// `cached`: this node was already evaluated as a leaf (in its parent's
// split test) from exactly the state it sees now — every earlier sibling
// kept the leaf decision it had then — so its decision (still in
// S.nodes) and cost (S.node_cost) are reused and only the replay runs.
__device__ __noinline__ long long leaf_eval(const Leaf L, bool cached) {
    Smem &S = smem_state();
    const int idx = qt_index(L.depth, L.cx, L.cy);
    if (cached) {
        const long long c = S.node_cost[idx];
        leaf_code(L, false, 0, 0);
        return c;
    }
    const long long c = leaf_decide(L);
    if (threadIdx.x == 0) S.node_cost[idx] = c;
    return c;
}

// One copy per depth, not inlined into each other: an unrolled tree would be
// code that runs once per CTU and misses the instruction cache every time.
template <int D>
__device__ __noinline__ void qt_decide(int ctu_x, int ctu_y, int cx, int cy, bool cached) {
    Smem &S = smem_state();
    const FrameParams &P = g_fp;
    constexpr int cu = 64 >> D;
    const int px = ctu_x + cx * 8, py = ctu_y + cy * 8;
    const bool in_frame = px + cu <= P.W && py + cu <= P.H;
    Node &nd = S.nodes[qt_index(D, cx, cy)];
    if constexpr (D < 3) {
        constexpr int h = 4 >> D;   // child offset in cells
        const int fast_leaf_depth = P.preset == 0 ? 3 : 2;
        const bool pass = in_frame && P.preset <= 1 && D < fast_leaf_depth;
        if (!in_frame || pass) {
            if (pass) {
                if (threadIdx.x == 0) nd.split = 1;
                SYNC();
            }
#pragma unroll 1
            for (int q = 0; q < 4; ++q)
                qt_decide<D + 1>(ctu_x, ctu_y, cx + (q & 1) * h, cy + (q >> 1) * h, false);
            return;
        }
        const Leaf L(P, ctu_x, ctu_y, D, cx, cy);
        snap(L, 0, -1);
        const long long parent = leaf_eval(L, cached);
        snap(L, D > 0 ? 1 : -1, 0);
        long long child = 0;
#pragma unroll 1
        for (int q = 0; q < 4; ++q)
            child += leaf_eval(Leaf(P, ctu_x, ctu_y, D + 1, cx + (q & 1) * h, cy + (q >> 1) * h), false);
        if (child <= parent) {
            if (threadIdx.x == 0) nd.split = 1;
            if constexpr (D == 2) {
                // 8x8 children split no further: the split test has left
                // their final reconstruction, grid and levels
                SYNC();
            } else {
                snap(L, -1, 0);
                // Children keep their split-test evaluation until one of them
                // splits (its region then differs from the split test's state).
                bool same_state = true;
#pragma unroll 1
                for (int q = 0; q < 4; ++q) {
                    const int qx = cx + (q & 1) * h, qy = cy + (q >> 1) * h;
                    qt_decide<D + 1>(ctu_x, ctu_y, qx, qy, same_state);
                    if (S.nodes[qt_index(D + 1, qx, qy)].split) same_state = false;
                }
            }
        } else {
            if (threadIdx.x == 0) nd.split = 0;
            if constexpr (D == 0) {
                snap(L, -1, 0);
                leaf_code(L, false, 0, 0);
            } else {
                const uint2 *lev = (const uint2 *)(D == 1 ? S.lev1 : S.lev2);
                uint2 *out = (uint2 *)(S.coef + 96 * S.zoff[cy * 8 + cx]);
#pragma unroll 1
                for (int i = threadIdx.x; i < 24 * (64 >> (2 * D)); i += NT) out[i] = lev[i];
                snap(L, -1, 1);
            }
        }
    } else {
        if (!in_frame) return;
        leaf_eval(Leaf(P, ctu_x, ctu_y, D, cx, cy), cached);
        if (threadIdx.x == 0) nd.split = 0;
        SYNC();
    }
}

// The final tree's 8x8-TU mask, and its levels without the gaps of skipped
// leaves (reference src/encoder.c:1450-1456 writes the leaves in z-order).
__device__ __noinline__ void close_gaps(int ctu_x, int ctu_y, CtuOut *out) {
    Smem &S = smem_state();
    const int t = threadIdx.x;
    const auto in_frame = [&](int cx, int cy, int cu) {
        return ctu_x + cx * 8 + cu <= g_fp.W && ctu_y + cy * 8 + cu <= g_fp.H;
    };
    bool skip = false, tu8 = false, cell = false;
    if (t < 64) {
        const int cx = t & 7, cy = t >> 3;
        cell = in_frame(cx, cy, 8);
        for (int d = 0; cell && d < 4; ++d) {
            const int m = ~((8 >> d) - 1), nx = cx & m, ny = cy & m;
            const Node &nd = S.nodes[qt_index(d, nx, ny)];
            if (d < 3 && (nd.split || !in_frame(nx, ny, 64 >> d))) continue;
            skip = nd.skip;
            tu8 = !skip && nd.dct_size;
            break;
        }
        S.leaf_skip[t] = skip;
    }
    const unsigned b8 = __ballot_sync(0xffffffffu, tu8);
    if (t == 0 || t == 32) ((unsigned *)&S.tu8mask)[t >> 5] = b8;
    const int ncells = __syncthreads_count(cell), nskip = __syncthreads_count(skip);
    if (t == 0) S.ncoef = 96 * (ncells - nskip);
    if (nskip) {
        // every thread holds its levels before any is moved; a cell's levels
        // move by the skipped cells before it
        constexpr int PER = CTU_COEF_MAX / 4 / NT;
        uint2 v[PER];
        int to[PER];
#pragma unroll
        for (int k = 0; k < PER; ++k) {
            const int u = t + k * NT, z = u / 24;      // 4 levels; cell in order of coding
            to[k] = -1;
            if (z < ncells) {
                v[k] = *(const uint2 *)(out->coef + 4 * u);
                int before = 0;
                for (int i = 0; i < 64; ++i) {
                    const int zi = S.zoff[i];
                    if (S.leaf_skip[i] && zi < z) ++before;
                    if (zi == z && in_frame(i & 7, i >> 3, 8) && !S.leaf_skip[i]) to[k] = 0;
                }
                if (to[k] == 0) to[k] = u - 24 * before;
            }
        }
        SYNC();
#pragma unroll
        for (int k = 0; k < PER; ++k) {
            const int u = t + k * NT;
            if (u >= 24 * (ncells - nskip) && u < 24 * ncells) *(uint2 *)(out->coef + 4 * u) = make_uint2(0, 0);
        }
        // (a cell never moves past the end of the kept ones)
#pragma unroll
        for (int k = 0; k < PER; ++k)
            if (to[k] >= 0) *(uint2 *)(out->coef + 4 * to[k]) = v[k];
    }
    SYNC();
}

// ====================================================================
// In-loop filters on the CTU tile.
// ====================================================================
template <class T>
__device__ __forceinline__ void deblock_on(T &S, int qp) {
    const int tc = clampi(qp / 3, 1, 10);
    const int cqp = clampi(qp - 1, 0, 63), ctc = clampi(cqp / 4, 1, 6);
    // Luma vertical edges x = 4..60 and chroma (Cb) vertical edges x = 4..28.
    for (int i = threadIdx.x; i < 15 * 64 + 7 * 32; i += NT) {
        if (i < 15 * 64) {
            const int e = i / 64 + 1, r = i - (e - 1) * 64, x = e * 4;
            const int p1 = RY(S, x - 2, r), p0 = RY(S, x - 1, r), q0 = RY(S, x, r), q1 = RY(S, x + 1, r);
            if (edge_strength(p0, q0, qp)) {
                RY(S, x - 1, r) = (uint8_t)weak_filter(p1, p0, q0, q1, tc);
                RY(S, x, r) = (uint8_t)weak_filter(q1, q0, p0, p1, tc);
            }
        } else {
            const int k = i - 15 * 64, e = k / 32 + 1, r = k - (e - 1) * 32, x = e * 4;
            const int p0 = RC(S, 0, x - 1, r), q0 = RC(S, 0, x, r);
            if (edge_strength(p0, q0, cqp)) {
                const int d = clampi((q0 - p0 + 1) >> 1, -ctc, ctc);
                RC(S, 0, x - 1, r) = (uint8_t)clampi(p0 + d, 0, 255);
                RC(S, 0, x, r) = (uint8_t)clampi(q0 - d, 0, 255);
            }
        }
    }
    SYNC();
    // Luma horizontal edges; chroma horizontal edges filter rows y, y+1
    // with the Cr strength for both planes (reference src/filter.c:212-236).
    for (int i = threadIdx.x; i < 15 * 64 + 7 * 32; i += NT) {
        if (i < 15 * 64) {
            const int e = i / 64 + 1, c = i - (e - 1) * 64, y = e * 4;
            const int p1 = RY(S, c, y - 2), p0 = RY(S, c, y - 1), q0 = RY(S, c, y), q1 = RY(S, c, y + 1);
            if (edge_strength(p0, q0, qp)) {
                RY(S, c, y - 1) = (uint8_t)weak_filter(p1, p0, q0, q1, tc);
                RY(S, c, y) = (uint8_t)weak_filter(q1, q0, p0, p1, tc);
            }
        } else {
            const int k = i - 15 * 64, e = k / 32 + 1, c = k - (e - 1) * 32, y = e * 4;
            const int p0 = RC(S, 1, c, y), q0 = RC(S, 1, c, y + 1);
            const int pb = RC(S, 0, c, y), qb = RC(S, 0, c, y + 1);
            if (edge_strength(p0, q0, cqp)) {
                int d = clampi((q0 - p0 + 1) >> 1, -ctc, ctc);
                RC(S, 1, c, y) = (uint8_t)clampi(p0 + d, 0, 255);
                RC(S, 1, c, y + 1) = (uint8_t)clampi(q0 - d, 0, 255);
                d = clampi((qb - pb + 1) >> 1, -ctc, ctc);
                RC(S, 0, c, y) = (uint8_t)clampi(pb + d, 0, 255);
                RC(S, 0, c, y + 1) = (uint8_t)clampi(qb - d, 0, 255);
            }
        }
    }
    SYNC();
}

__device__ __noinline__ void deblock_tile(Smem &, int qp) { deblock_on(smem_state(), qp); }

// Luma SAO band offset: choose (reference src/filter.c:269-319), rate gate
// (src/encoder.c:1473-1493) and apply (src/filter.c:251-266).
__device__ __noinline__ void sao_tile(Smem &, int w, int h, int lambda_sao) {
    Smem &S = smem_state();
    if (threadIdx.x < 32) {
        S.band_sum[threadIdx.x] = 0; S.band_cnt[threadIdx.x] = 0;
        S.band_sq[threadIdx.x] = 0; S.band_new[threadIdx.x] = 0;
    }
    SYNC();
    for (int i = threadIdx.x; i < w * h; i += NT) {
        const int y = div_p2(i, w), x = i - y * w;
        const int o = S.cur_y[y * 64 + x], r = RY(S, x, y), d = o - r, b = r >> 3;
        atomicAdd(&S.band_sum[b], d);
        atomicAdd(&S.band_cnt[b], 1);
        atomicAdd(&S.band_sq[b], d * d);
    }
    SYNC();
    // each band's candidate offset once (rounded mean of o - r, within +-7)
    if (threadIdx.x < 32) {
        const int cnt = S.band_cnt[threadIdx.x], sum = S.band_sum[threadIdx.x];
        S.band_cand[threadIdx.x] = cnt ? clampi((sum + (sum >= 0 ? cnt / 2 : -(cnt / 2))) / cnt, -7, 7) : 0;
    }
    SYNC();
    for (int i = threadIdx.x; i < w * h; i += NT) {
        const int y = div_p2(i, w), x = i - y * w;
        const int o = S.cur_y[y * 64 + x], r = RY(S, x, y), b = r >> 3;
        const int cand = S.band_cand[b];
        if (cand) {
            const int d = o - clampi(r + cand, 0, 255);
            atomicAdd(&S.band_new[b], d * d);
        }
    }
    SYNC();
    if (threadIdx.x == 0) {
        long long base = 0;
        for (int b = 0; b < 32; ++b) base += S.band_sq[b];
        long long best = base;
        int bb = 0, bo = 0;
        for (int b = 0; b < 32; ++b) {
            const int cand = S.band_cand[b];   // 0 for an empty band
            if (!cand) continue;
            const long long sse = base - S.band_sq[b] + S.band_new[b];
            if (sse < best) { best = sse; bb = b; bo = cand; }
        }
        int has = best < base;
        if (has && best + (long long)lambda_sao * 6 >= base) has = 0;
        S.sao[0] = has; S.sao[1] = has ? bb : 0; S.sao[2] = has ? bo : 0;
    }
    SYNC();
    if (S.sao[0]) {
        const int band = S.sao[1], off = S.sao[2];
        for (int i = threadIdx.x; i < w * h; i += NT) {
            const int y = div_p2(i, w), x = i - y * w;
            uint8_t &p = RY(S, x, y);
            if ((p >> 3) == band) p = (uint8_t)clampi(p + off, 0, 255);
        }
    }
    SYNC();
}

// What a CTU's searches and scoring work from: its source luma, every lane's
// quantisers, empty SAD tables.
__device__ void load_luma(Smem &S, const FrameParams &P, int ctu_x, int ctu_y) {
    const int w = mini(64, P.W - ctu_x), h = mini(64, P.H - ctu_y);
    for (int i = threadIdx.x; i < 64 * 64; i += NT) {
        const int y = i >> 6, x = i & 63;
        S.cur_y[i] = (x < w && y < h) ? P.cur_y[(size_t)(ctu_y + y) * P.stride_y + ctu_x + x] : 0;
    }
    if (threadIdx.x >= NT - 96) {
        const int t = threadIdx.x - (NT - 96), type = t >> 5, lane = t & 31, r = lane >> 2, c = 2 * (lane & 3);
        const int b0 = type ? band_rc(4, r & 3, c & 3) : band_rc(8, r, c);
        const int b1 = type ? band_rc(4, r & 3, (c & 3) + 1) : band_rc(8, r, c + 1);
        const int *eff = type == 2 ? P.eff_c : P.eff_l;
        const long long lambda = type == 2 ? (long long)P.lambda_c : P.lambda;
        const QuantLane q = QuantLane::make(QuantPos(eff[b0], lambda), QuantPos(eff[b1], lambda));
        S.quant[type][0][lane] = q.a;
        S.quant[type][1][lane] = q.b;
        S.quant[type][2][lane] = q.c;
    }
    init_windows(S);
}

// A helper's part of a leaf decision (see leaf_decide).
__device__ __noinline__ void help_leaf(const Leaf L, int mvpx, int mvpy) {
    Smem &S = smem_state();
    const FrameParams &P = g_fp;
    const int rank = cluster_rank(), n = cluster_size();
    const uint32_t modes = intra_modes(P.preset);
    list_intra(S, modes, L.cu <= 32);
    uint32_t share = 0;
    if (P.frame_type != 0) {
        const LeafSearch M = leaf_searches(L, mvpx, mvpy);
        share = search_share(M.mask, rank, n);
        if (share) {
            pair_source(S, L);
            SYNC();
            const int lth = search_team(share, n - 1);
            me_searches(L, share, M.J, M.sr, lth, false, false);
            // the team's search to the first CTA
            const MeTeam T(lth);
            if (T.g < __popc(share)) {
                uint32_t m = share;
                for (int i = 0; i < T.g; ++i) m &= m - 1;
                const int id = __ffs((int)m) - 1;
                T.sync();
                Smem *A = peer_smem(0);
                for (int i = T.gt; i < L.cu * L.cu / 16; i += 1 << lth)
                    ((uint4 *)A->pred[id])[i] = ((const uint4 *)S.pred[id])[i];
                if (T.gt == 0) {
                    A->me[id].mvx = S.me[id].mvx; A->me[id].mvy = S.me[id].mvy;
                    A->cand_mvx[id] = S.cand_mvx[id]; A->cand_mvy[id] = S.cand_mvy[id];
                }
            }
        }
    }
    if (!share) SYNC();
    luma_score<true>(L, S.cl, __popc(modes), 0, ~0u);
}

// A helper's life: commands until CMD_LEAVE.
__device__ void help(Smem &S, const FrameParams *__restrict__ params, int *ctrl) {
    int ctu_x = 0, ctu_y = 0;
    for (int seq = 1;; ++seq) {
        int got = 0;
        if (threadIdx.x == 0) {
            // far longer than the first CTA waits for its neighbours
            const long long w = g_neighbor_wait_limit, limit = w < 1ll << 60 ? 4 * w + (1ll << 24) : w;
            unsigned ns = 32;
            for (long long i = 0; i < limit && got < seq; ++i) {
                got = ld_acquire_cluster(&S.cmd_seq);
                if (got < seq && i > 4096) {
                    __nanosleep(ns);
                    if (ns < 1024) ns <<= 1;
                }
            }
            if (got < seq) atomicExch(&ctrl[1], 1);
        }
        if (!__syncthreads_or(got == seq)) return;
        const int c0 = S.cmd[0], c1 = S.cmd[1], c2 = S.cmd[2], c3 = S.cmd[3], c4 = S.cmd[4], c5 = S.cmd[5];
        if (c0 == HELP_CTU) {
            if (threadIdx.x == 0) g_fp = params[c1 >> 20];
            SYNC();
            ctu_x = (c1 & 1023) * 64;
            ctu_y = (c1 >> 10 & 1023) * 64;
            load_luma(S, g_fp, ctu_x, ctu_y);
        } else {
            help_leaf(Leaf(g_fp, ctu_x, ctu_y, c1, c2, c3), c4, c5);
        }
        // (test hook: the first helper leaves without an answer)
        if (g_fp.helper_quits && seq >= g_fp.helper_quits && cluster_rank() == 1) return;
        acknowledge();
    }
}

// ====================================================================
// The CTU kernel.  items[i] = (stream << 20) | (row << 10) | col.
// ====================================================================
__device__ void encode_ctu(Smem &S, const FrameParams &P, int row, int col) {
    const int ctu_x = col * 64, ctu_y = row * 64;
    const int w = mini(64, P.W - ctu_x), h = mini(64, P.H - ctu_y);
    const int wc = w >> 1, hc = h >> 1;
    // ---- load source and the filtered neighbour border ----------------
    load_luma(S, P, ctu_x, ctu_y);
    for (int i = threadIdx.x; i < 2 * 32 * 32; i += NT) {
        const int c = i >> 10, p = i & 1023, y = p >> 5, x = p & 31;
        const uint8_t *src = c ? P.cur_cr : P.cur_cb;
        S.cur_c[c][p] = (x < wc && y < hc) ? src[(size_t)((ctu_y >> 1) + y) * P.stride_c + (ctu_x >> 1) + x] : 0;
    }
    if (ctu_y > 0) {
        for (int x = threadIdx.x - 2; x < w; x += NT)
            if (ctu_x + x >= 0) RY(S, x, -1) = __ldcg(P.rec_y + (size_t)(ctu_y - 1) * P.stride_y + ctu_x + x);
        for (int i = threadIdx.x; i < 2 * 33; i += NT) {
            const int c = i / 33, x = i - c * 33 - 1;
            const uint8_t *src = c ? P.rec_cr : P.rec_cb;
            if (x < wc && ctu_x / 2 + x >= 0)
                RC(S, c, x, -1) = __ldcg(src + (size_t)((ctu_y >> 1) - 1) * P.stride_c + (ctu_x >> 1) + x);
        }
    }
    if (ctu_x > 0) {
        for (int i = threadIdx.x; i < 2 * h; i += NT) {
            const int y = i >> 1, x = (i & 1) - 2;
            RY(S, x, y) = __ldcg(P.rec_y + (size_t)(ctu_y + y) * P.stride_y + ctu_x + x);
        }
        for (int i = threadIdx.x; i < 2 * hc; i += NT) {
            const int c = i / hc, y = i - c * hc;
            const uint8_t *src = c ? P.rec_cr : P.rec_cb;
            RC(S, c, -1, y) = __ldcg(src + (size_t)((ctu_y >> 1) + y) * P.stride_c + (ctu_x >> 1) - 1);
        }
    }
    // Samples outside whole 8x8 blocks are never coded: they keep the picture
    // before's, as in the decoder, whose reconstruction buffer persists.
    if ((w | h) & 7) {
        const int w8 = w & ~7, h8 = h & ~7;
        for (int i = threadIdx.x; i < 64 * 64; i += NT) {
            const int y = i >> 6, x = i & 63;
            if (x < w && y < h && (x >= w8 || y >= h8))
                RY(S, x, y) = P.kept_y[(size_t)(ctu_y + y) * P.stride_y + ctu_x + x];
        }
        for (int i = threadIdx.x; i < 2 * 32 * 32; i += NT) {
            const int c = i >> 10, p = i & 1023, y = p >> 5, x = p & 31;
            if (x < wc && y < hc && (x >= w8 >> 1 || y >= h8 >> 1))
                RC(S, c, x, y) = (c ? P.kept_cr : P.kept_cb)[(size_t)((ctu_y >> 1) + y) * P.stride_c + (ctu_x >> 1) + x];
        }
    }
    for (int i = threadIdx.x; i < 64; i += NT) {
        S.grid[i].dx = 0; S.grid[i].dy = 0; S.grid[i].intra = 1; S.grid[i].pad = 0;
    }
    for (int i = threadIdx.x; i < QT_NODES; i += NT) {
        Node z = {};
        S.nodes[i] = z;
    }
    CtuOut *out = P.out + row * P.ctu_cols + col;
    if (threadIdx.x == 0) S.coef = out->coef;
    if (threadIdx.x < 64) {
        // coded cells (whole 8x8 blocks of the frame) before the z-th cell of
        // z-order, z = this thread
        auto at = [](int z, int b) { return (z >> b & 1) | (z >> (b + 1) & 2) | (z >> (b + 2) & 4); };
        int n = 0;
        for (int z = 0; z < (int)threadIdx.x; ++z)
            n += ctu_x + at(z, 0) * 8 + 8 <= P.W && ctu_y + at(z, 1) * 8 + 8 <= P.H;
        S.zoff[at(threadIdx.x, 1) * 8 + at(threadIdx.x, 0)] = (uint16_t)n;
    }
    wait_helpers(S);      // they have loaded the CTU too
    SYNC();

    // ---- decide and code -------------------------------------------------
    PHASE_T0();
    qt_decide<0>(ctu_x, ctu_y, 0, 0, false);
    PHASE(8);
    close_gaps(ctu_x, ctu_y, out);
    PHASE(9);
    // ---- in-loop filters ------------------------------------------------
    if (w == 64 && h == 64) deblock_tile(S, P.qp);
    sao_tile(S, w, h, P.lambda_sao);
    PHASE(10);
    // ---- exports --------------------------------------------------------
    for (int i = threadIdx.x; i < w * h; i += NT) {
        const int y = div_p2(i, w), x = i - y * w;
        P.rec_y[(size_t)(ctu_y + y) * P.stride_y + ctu_x + x] = RY(S, x, y);
    }
    for (int i = threadIdx.x; i < 2 * wc * hc; i += NT) {
        const int c = div_p2(i, wc * hc), p = i - c * wc * hc, y = div_p2(p, wc), x = p - y * wc;
        uint8_t *dst = c ? P.rec_cr : P.rec_cb;
        dst[(size_t)((ctu_y >> 1) + y) * P.stride_c + (ctu_x >> 1) + x] = RC(S, c, x, y);
    }
    for (int i = threadIdx.x; i < 64; i += NT) {
        const int gy = i >> 3, gx = i & 7;
        const int fy = row * 8 + gy, fx = col * 8 + gx;
        if (fy < P.grid_h && fx < P.grid_w) P.cur_grid[fy * P.grid_w + fx] = S.grid[i];
    }
    for (int i = threadIdx.x; i < QT_NODES; i += NT) out->nodes[i] = S.nodes[i];
    if (threadIdx.x == 0) {
        out->ncoef = S.ncoef;
        out->tu8mask = S.tu8mask;
        out->sao_has = (int16_t)S.sao[0];
        out->sao_band = (int16_t)S.sao[1];
        out->sao_offset = (int16_t)S.sao[2];
    }
}

// The transform fragments (forward and inverse, 8x8 and 4x4) of every lane and
// the last-position bits, once per CTA.
__device__ void init_fragments(Smem &S) {
    if (threadIdx.x < 128)
        S.frag[threadIdx.x >> 5][threadIdx.x & 31] =
            dct_fragment(threadIdx.x < 64 ? 8 : 4, (threadIdx.x >> 5) & 1, threadIdx.x & 31);
    else if (threadIdx.x < 128 + 65)
        S.last_bits[threadIdx.x - 128] = last_bits((int)threadIdx.x - 129);
}

// One CTA per CTU of one anti-diagonal (items[blockIdx.x]).
__global__ void __launch_bounds__(NT, CTAS_PER_SM)
ctu_kernel(const FrameParams *__restrict__ params, const int *__restrict__ items) {
    extern __shared__ __align__(16) uint8_t smem_raw[];
    Smem &S = *reinterpret_cast<Smem *>(smem_raw);
    FrameParams &P = g_fp;
    const int item = items[blockIdx.x];
    if (threadIdx.x == 0) P = params[item >> 20];
    init_fragments(S);
    if (threadIdx.x == 0) S.helpers = 0;
    SYNC();
    encode_ctu(S, P, (item >> 10) & 1023, item & 1023);
}

__device__ __forceinline__ int ld_acquire(const int *p) {
    int v;
    asm volatile("ld.acquire.gpu.global.s32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void st_release(int *p, int v) {
    asm volatile("st.release.gpu.global.s32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}

// Persistent wavefront: a resident grid pulls CTUs from a queue laid out in
// topological (anti-diagonal) order and starts each one as soon as its
// left and above neighbours are published.  A CTU only ever waits for
// items dequeued before it, by CTAs that are already running, so the queue
// always drains.  Waits are bounded: on expiry the CTA records an error in
// ctrl[1] and goes on, and the host reports TC_ERR_INTERNAL.
__global__ void __launch_bounds__(NT, CTAS_PER_SM)
ctu_persistent_kernel(const FrameParams *__restrict__ params, const int *__restrict__ items, int n_items,
                      int *ctrl) {
    extern __shared__ __align__(16) uint8_t smem_raw[];
    Smem &S = *reinterpret_cast<Smem *>(smem_raw);
    FrameParams &P = g_fp;
    __shared__ int s_item;
    init_fragments(S);    // visible to all after the first item's barrier
    const bool cluster = cluster_size() > 1;
    if (threadIdx.x == 0) {
        S.helpers = cluster_size() - 1;
        S.cmd_sent = S.cmd_seq = S.acks = S.ack_goal = 0;
        S.error = ctrl + 1;
    }
    if (cluster) {
        cluster_barrier();    // every CTA's counters are set
        if (cluster_rank() > 0) {
            help(S, params, ctrl);
            cluster_barrier();
            return;
        }
    }
#ifdef TCB_PHASE_PROFILE
    const long long k0 = clock64();   // residency of the CTA (slot 14); neighbour waits in slot 13
#endif
    for (;;) {
        if (threadIdx.x == 0) {
            const int i = atomicAdd(&ctrl[0], 1);
            s_item = i < n_items ? items[i] : -1;
        }
        SYNC();
        const int item = s_item;
        if (item < 0) {
#ifdef TCB_PHASE_PROFILE
            if (threadIdx.x == 0) atomicAdd(&tcb_phase_cycles[14], (unsigned long long)(clock64() - k0));
#endif
            break;
        }
        const int row = (item >> 10) & 1023, col = item & 1023;
        if (S.helpers) send_command(HELP_CTU, item, 0, 0, 0, 0);
        if (threadIdx.x == 0) {
            P = params[item >> 20];
            const int epoch = P.epoch;
            const int *dl = col > 0 ? P.done + row * P.ctu_cols + col - 1 : nullptr;
            const int *du = row > 0 ? P.done + (row - 1) * P.ctu_cols + col : nullptr;
            unsigned ns = 32;
            long long spins = 0;
            const long long limit = g_neighbor_wait_limit;
#ifdef TCB_PHASE_PROFILE
            const long long w0 = clock64();
#endif
            while ((dl && ld_acquire(dl) != epoch) || (du && ld_acquire(du) != epoch)) {
                __nanosleep(ns);
                if (ns < 2048) ns <<= 1;
                if (++spins > limit) { atomicExch(&ctrl[1], 1); break; }
            }
#ifdef TCB_PHASE_PROFILE
            atomicAdd(&tcb_phase_cycles[13], (unsigned long long)(clock64() - w0));
#endif
        }
        SYNC();
        encode_ctu(S, P, row, col);
        __threadfence();
        SYNC();
        if (threadIdx.x == 0) st_release(P.done + row * P.ctu_cols + col, P.epoch);
    }
    if (cluster) {
        send_leave();
        cluster_barrier();
    }
}

namespace legacy {
__global__ void legacy_encode_kernel(const LFrame F, const int *__restrict__ items);
}

cudaError_t init_engine_tables() {
    cudaError_t e = upload_dct_tables();
    if (e != cudaSuccess) return e;
    e = cudaFuncSetAttribute(ctu_persistent_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)sizeof(Smem));
    if (e != cudaSuccess) return e;
    e = cudaFuncSetAttribute(legacy::legacy_encode_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)sizeof(Smem));
    if (e != cudaSuccess) return e;
    if (CTAS_PER_SM > 1) {   // room for CTAS_PER_SM CTUs' shared memory per SM
        e = cudaFuncSetAttribute(ctu_persistent_kernel, cudaFuncAttributePreferredSharedMemoryCarveout,
                                 (int)cudaSharedmemCarveoutMaxShared);
        if (e != cudaSuccess) return e;
    }
    return cudaFuncSetAttribute(ctu_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                (int)sizeof(Smem));
}

// Layout of the CTU-engine scratch used by tcb_ctu_encode_frame: frame
// parameters, queue counter + error word, per-CTU publish flags, queue.
constexpr size_t SCR_PARAMS = 0, SCR_CTRL = 1024, SCR_DONE = 1280;
constexpr int MAX_DEVICES = 64;
inline size_t scratch_bytes_for(int nctu) { return SCR_DONE + 8 * (size_t)nctu; }

static_assert(sizeof(FrameParams) <= SCR_CTRL, "frame parameters overflow their scratch slot");

// Writes the frame parameters into the scratch, clears the queue counter,
// error word and publish flags, and lays out the queue in wavefront order:
// anti-diagonal d = r + c ascending, rows ascending within a diagonal, so
// every CTU's left / above / above-right neighbours are dequeued before it.
__global__ void frame_setup_kernel(FrameParams P, uint8_t *__restrict__ scratch) {
    const int nctu = P.ctu_cols * P.ctu_rows;
    int *ctrl = (int *)(scratch + SCR_CTRL), *done = (int *)(scratch + SCR_DONE), *items = done + nctu;
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t == 0) {
        *(FrameParams *)(scratch + SCR_PARAMS) = P;
        ctrl[0] = 0;
        ctrl[1] = 0;
    }
    if (t >= nctu) return;
    done[t] = 0;
    const int r = t / P.ctu_cols, c = t - r * P.ctu_cols, d = r + c;
    int pos = 0;
    for (int dd = 0; dd < d; ++dd) pos += min(dd, P.ctu_rows - 1) - max(0, dd - (P.ctu_cols - 1)) + 1;
    items[pos + r - max(0, d - (P.ctu_cols - 1))] = (r << 10) | c;
}

// Shared host half of the frame entry points: one set-up launch fills
// `scratch`, one persistent launch drains its queue.  Nothing is allocated
// and nothing is copied from host memory.  `first` > 0 leaves the queue's
// first items out (the wait-expiry test hook: their publish flags are
// never set, so their neighbours' bounded waits run out).
// `helper_quits`: see FrameParams.
cudaError_t encode_frame_with_scratch(const FrameParams &P0, uint8_t *scratch, cudaStream_t st, int first,
                                      int helper_quits = 0) {
    FrameParams P = P0;
    P.helper_quits = helper_quits;
    const int nctu = P.ctu_cols * P.ctu_rows;
    int *ctrl = (int *)(scratch + SCR_CTRL), *done = (int *)(scratch + SCR_DONE), *items = done + nctu;
    P.done = done;
    P.epoch = 1;
    P.err = ctrl + 1;
    frame_setup_kernel<<<(nctu + 255) / 256, 256, 0, st>>>(P, scratch);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    int dev = 0, sms = 0;
    if ((e = cudaGetDevice(&dev)) != cudaSuccess) return e;
    if ((e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev)) != cudaSuccess) return e;
    return launch_ctu_persistent((const FrameParams *)(scratch + SCR_PARAMS), items + first, nctu - first, ctrl,
                                 sms, P.preset >= 2 ? mini(P.ctu_cols, P.ctu_rows) : 0, st);
}

// Constant tables and kernel attributes, once per device.
cudaError_t ensure_device_tables() {
    static std::mutex mu;
    static bool ready[MAX_DEVICES] = {};
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    if (dev < 0 || dev >= MAX_DEVICES) return cudaErrorInvalidDevice;
    std::lock_guard<std::mutex> lk(mu);
    if (!ready[dev]) {
        if ((e = init_device_tables()) != cudaSuccess) return e;
        ready[dev] = true;
    }
    return cudaSuccess;
}

// `ready`: CTUs that can be in work at once, 0 if the frames' leaves leave
// nothing for helper CTAs.  Clusters of four where the CTUs in work leave SMs
// for them, of two where only for one helper each; up to twice as many clusters
// as CTUs in work, because a cluster that has dequeued a CTU waits with it
// for its neighbours, and no more, to leave the other SMs to other streams.  With 17 CTUs in work (1920x1080) a P frame takes 59.9 ms
// with single CTAs, 56.0 with clusters of two, 54.2 with four, 56.5 with six
// (then 24 clusters), and 56.4 with four but only 17 clusters; 32 such streams
// fill the SMs with single CTAs.
cudaError_t launch_ctu_persistent(const FrameParams *d_params, const int *d_items, int n, int *d_ctrl,
                                  int grid, int ready, cudaStream_t st) {
    if (n <= 0) return cudaSuccess;
    grid *= CTAS_PER_SM;
    const int size = ready <= 0 ? 1 : 4 * ready <= grid ? 4 : 2 * ready <= grid ? 2 : 1;
    if (size > 1) {
        cudaLaunchAttribute at;
        at.id = cudaLaunchAttributeClusterDimension;
        at.val.clusterDim = {(unsigned)size, 1, 1};
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3((unsigned)(size * mini(mini(grid / size, 2 * ready), n)));
        cfg.blockDim = dim3(NT);
        cfg.dynamicSmemBytes = sizeof(Smem);
        cfg.stream = st;
        cfg.attrs = &at;
        cfg.numAttrs = 1;
        if (cudaLaunchKernelEx(&cfg, ctu_persistent_kernel, d_params, d_items, n, d_ctrl) == cudaSuccess) return cudaSuccess;
        cudaGetLastError();    // no room for a cluster on this device or partition: single CTAs
    }
    ctu_persistent_kernel<<<grid < n ? grid : n, NT, sizeof(Smem), st>>>(d_params, d_items, n, d_ctrl);
    return cudaGetLastError();
}

size_t ctu_smem_bytes() { return sizeof(Smem); }

cudaError_t launch_ctu_items(const FrameParams *d_params, const int *d_items, int n,
                             cudaStream_t st) {
    if (n <= 0) return cudaSuccess;
    ctu_kernel<<<n, NT, sizeof(Smem), st>>>(d_params, d_items);
    return cudaGetLastError();
}

}  // namespace tcb

// --------------------------------------------------------------------
// Frame entry point that allocates nothing (tcb_ctu_encode_frame_static).
//
// Some callers cannot allocate device memory: an application whose own
// pool allocator reserves the GPU's memory up front and owns every byte of
// it, a plugin host that only lends out the frame buffers it manages, or a
// real-time loop in which cudaMalloc / cudaFree (and the device-wide
// synchronisation cudaFree implies) are not allowed.  For them the
// scratch that tcb_ctu_encode_frame takes from its caller -- frame
// parameters, queue counter and error word, per-CTU publish flags, work
// queue -- lives in this fixed device array instead.  Every GPU that loads
// the library holds it (17,664 bytes) until the process exits.  In host
// code the name below only identifies the symbol; its device address comes
// from cudaGetSymbolAddress.
// --------------------------------------------------------------------
static __device__ __align__(256) uint8_t g_ctu_static_scratch[tcb::SCR_DONE + 8 * TCB_CTU_STATIC_MAX_CTUS];

namespace tcb {

// Device address of g_ctu_static_scratch on the current device, looked up
// on the first call made with that device current and kept afterwards.
cudaError_t static_scratch_address(uint8_t **out) {
    static std::mutex mu;
    static uint8_t *addr[MAX_DEVICES] = {};
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    if (dev < 0 || dev >= MAX_DEVICES) return cudaErrorInvalidDevice;
    std::lock_guard<std::mutex> lk(mu);
    if (!addr[dev]) {
        void *p = nullptr;
        e = cudaGetSymbolAddress(&p, g_ctu_static_scratch);
        if (e != cudaSuccess) return e;
        addr[dev] = (uint8_t *)p;
    }
    *out = addr[dev];
    return cudaSuccess;
}

}  // namespace tcb

extern "C" {

size_t tcb_ctu_record_bytes(void) { return sizeof(tcb::CtuOut); }
size_t tcb_mv_cell_bytes(void) { return sizeof(tcb::MvCell); }
size_t tcb_ctu_scratch_bytes(int width, int height) {
    if (width <= 0 || height <= 0) return 0;
    return tcb::scratch_bytes_for(((width + 63) / 64) * ((height + 63) / 64));
}

tc_error_t tcb_ctu_encode_frame(const tcb_frame_desc_t *desc, void *scratch, size_t scratch_bytes, void *stream) {
    tcb::FrameParams P;
    if (!desc || !scratch || !tcb::frame_params_from_desc(*desc, P)) return TC_ERR_PARAM;
    if (scratch_bytes < tcb::scratch_bytes_for(P.ctu_cols * P.ctu_rows)) return TC_ERR_PARAM;
    if (tcb::ensure_device_tables() != cudaSuccess) return TC_ERR_INTERNAL;
    return tcb::encode_frame_with_scratch(P, (uint8_t *)scratch, (cudaStream_t)stream, 0) == cudaSuccess
               ? TC_OK : TC_ERR_INTERNAL;
}

tc_error_t tcb_ctu_encode_frame_static(const tcb_frame_desc_t *desc, void *stream) {
    tcb::FrameParams P;
    if (!desc || !tcb::frame_params_from_desc(*desc, P)) return TC_ERR_PARAM;
    if (P.ctu_cols * P.ctu_rows > TCB_CTU_STATIC_MAX_CTUS) return TC_ERR_MEMORY;
    if (tcb::ensure_device_tables() != cudaSuccess) return TC_ERR_INTERNAL;
    uint8_t *scratch = nullptr;
    if (tcb::static_scratch_address(&scratch) != cudaSuccess) return TC_ERR_INTERNAL;
    return tcb::encode_frame_with_scratch(P, scratch, (cudaStream_t)stream, 0) == cudaSuccess ? TC_OK
                                                                                              : TC_ERR_INTERNAL;
}

// The frame's error word (set when a neighbour wait ran out), read once the
// frame's work on `stream` has finished.
static tc_error_t frame_result(const uint8_t *scratch, void *stream) {
    int err = 0;
    if (cudaMemcpyAsync(&err, scratch + tcb::SCR_CTRL + sizeof(int), sizeof(int), cudaMemcpyDeviceToHost,
                        (cudaStream_t)stream) != cudaSuccess ||
        cudaStreamSynchronize((cudaStream_t)stream) != cudaSuccess)
        return TC_ERR_INTERNAL;
    return err ? TC_ERR_INTERNAL : TC_OK;
}

tc_error_t tcb_ctu_frame_result(const void *scratch, void *stream) {
    if (!scratch) return TC_ERR_PARAM;
    return frame_result((const uint8_t *)scratch, stream);
}

tc_error_t tcb_ctu_frame_result_static(void *stream) {
    uint8_t *scratch = nullptr;
    if (tcb::static_scratch_address(&scratch) != cudaSuccess) return TC_ERR_INTERNAL;
    return frame_result(scratch, stream);
}

tc_error_t tcb_set_neighbor_wait_limit(long long spins) {
    if (spins < 1) return TC_ERR_PARAM;
    return cudaMemcpyToSymbol(tcb::g_neighbor_wait_limit, &spins, sizeof(spins)) == cudaSuccess ? TC_OK
                                                                                                : TC_ERR_INTERNAL;
}

tc_error_t tcb_get_neighbor_wait_limit(long long *spins) {
    if (!spins) return TC_ERR_PARAM;
    return cudaMemcpyFromSymbol(spins, tcb::g_neighbor_wait_limit, sizeof(*spins)) == cudaSuccess
               ? TC_OK : TC_ERR_INTERNAL;
}

tc_error_t tcb_debug_ctu_encode_frame_helper_quits(const tcb_frame_desc_t *desc, void *scratch, size_t scratch_bytes,
                                                   void *stream, int commands) {
    tcb::FrameParams P;
    if (!desc || !scratch || commands < 1 || !tcb::frame_params_from_desc(*desc, P)) return TC_ERR_PARAM;
    if (scratch_bytes < tcb::scratch_bytes_for(P.ctu_cols * P.ctu_rows)) return TC_ERR_PARAM;
    if (tcb::ensure_device_tables() != cudaSuccess) return TC_ERR_INTERNAL;
    return tcb::encode_frame_with_scratch(P, (uint8_t *)scratch, (cudaStream_t)stream, 0, commands) == cudaSuccess
               ? TC_OK : TC_ERR_INTERNAL;
}

tc_error_t tcb_debug_ctu_encode_frame_without_first(const tcb_frame_desc_t *desc, void *scratch,
                                                    size_t scratch_bytes, void *stream) {
    tcb::FrameParams P;
    if (!desc || !scratch || !tcb::frame_params_from_desc(*desc, P)) return TC_ERR_PARAM;
    if (P.ctu_cols * P.ctu_rows < 2 || scratch_bytes < tcb::scratch_bytes_for(P.ctu_cols * P.ctu_rows))
        return TC_ERR_PARAM;
    if (tcb::ensure_device_tables() != cudaSuccess) return TC_ERR_INTERNAL;
    return tcb::encode_frame_with_scratch(P, (uint8_t *)scratch, (cudaStream_t)stream, 1) == cudaSuccess
               ? TC_OK : TC_ERR_INTERNAL;
}

}  // extern "C"

#include "tcb_decode.cuh"
#include "tcb_legacy_enc.cuh"

#ifdef TCB_PHASE_PROFILE
// Profiling builds only: read and reset the phase cycle counters.
extern "C" __attribute__((visibility("default"))) int tcb_debug_op_counts(unsigned long long *out4) {
    cudaDeviceSynchronize();
    if (cudaMemcpyFromSymbol(out4, tcb::tcb_op_counts, 4 * sizeof(unsigned long long)) != cudaSuccess) return -1;
    unsigned long long z[4] = {0};
    return cudaMemcpyToSymbol(tcb::tcb_op_counts, z, sizeof(z)) == cudaSuccess ? 0 : -1;
}
extern "C" __attribute__((visibility("default"))) int tcb_debug_phase_cycles(unsigned long long *out60) {
    cudaDeviceSynchronize();
    if (cudaMemcpyFromSymbol(out60, tcb::tcb_phase_cycles, tcb::PHASE_SLOTS * sizeof(unsigned long long)) != cudaSuccess)
        return -1;
    unsigned long long z[tcb::PHASE_SLOTS] = {0};
    return cudaMemcpyToSymbol(tcb::tcb_phase_cycles, z, sizeof(z)) == cudaSuccess ? 0 : -1;
}
#endif

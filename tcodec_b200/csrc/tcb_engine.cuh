// tcb_engine.cuh — shared-memory layout and launch constants of the CTU
// rate-distortion engine (one 512-thread CTA per 64x64 CTU).
#pragma once
#include <stddef.h>
#include "tcb_common.cuh"
#include "tcb_resid.cuh"

namespace tcb {

constexpr int NT = 512;             // threads per CTA (one CTU)
constexpr int CTAS_PER_SM = 1;      // CTUs resident per SM
constexpr int NW = NT / 32;         // warps per CTA
constexpr int NGROUP = 4;           // motion-search warp groups

// Recon tile: luma rows -1..63 and columns -8..63 of the CTU, chroma rows
// -1..31 and columns -4..31.  Column offsets keep the interior aligned.
constexpr int RY_W = 72, RY_OX = 8, RY_OY = 1, RY_H = 65;
constexpr int RC_W = 36, RC_OX = 4, RC_OY = 1, RC_H = 33;

// Candidate slots of one leaf.
enum {
    K_ME0 = 0,      // explicit inter, MVP-centred search on the first reference
    K_ME1 = 1,      // explicit inter on the second reference (multiref)
    K_GLB = 2,      // explicit inter, global-motion centre
    K_TMP = 3,      // explicit inter, temporal centre
    K_MRG = 4,      // merge at the MVP
    K_B0 = 0,       // B: forward / backward / average / single merges (0..4;
                    // B frames use no P slot, so the two sets share buffers)
    K_INTRA = 5,    // intra modes 0..17 -> slots 5..22
    NCAND = 23
};
constexpr int NPRED = 5;            // inter prediction buffers (slots 0..4)

// Entry of a leaf's candidate list: the slot, which TU sizes are scored, and
// from bit 16 on an angular mode's displacement.
enum {
    CL_SLOT = 0xFF,
    CL_8 = 0x100,       // one 8x8 TU per 8x8 area
    CL_4 = 0x200,       // four 4x4 TUs per 8x8 area
    CL_EXACT = 0x400    // note whether the prediction equals the source
};

constexpr int EDGE_BASE = 96, EDGE_LEN = 264;   // index 0 of S.edge; entries up to 2.5 * 64 + 2

// SAD tables of the integer stages of blocks up to 16x16: positions within R
// (2..WIN_RMAX) of the window's centre, and a ring of 2 around them that
// says "off the table".
constexpr int WIN_RMAX = 5, WIN_SIDE = 2 * WIN_RMAX + 5, WIN_WORDS = WIN_SIDE * WIN_SIDE;

constexpr int QPOS = 7;               // quarter-sample positions per axis around an integer best: -3..3
struct alignas(16) MeGroup {
    int part[2][8];         // SADs of a batch of candidates, double-buffered (see batch_sads)
    int4 tab[QPOS * QPOS];  // SADs of the quarter-sample positions scored, by quarters of the block
    uint16_t win[2][WIN_WORDS];   // two SAD tables: SAD + 1, 0 off the table, 0xFFFF outside the frame
    int bx, by;             // integer best
    int mvx, mvy, best;
};

// Sample planes of a quarter-sample refinement (me_qpel) of a B x B block, in
// 32-bit words that hold two columns B / 2 apart: integer samples and
// horizontal halves (B + 6 rows), vertical and centre halves (B + 1 rows).
__host__ __device__ constexpr int plane_stride(int B) { return B / 2 + 6; }
__host__ __device__ constexpr int plane_words(int B) { return (4 * B + 14) * plane_stride(B); }
constexpr int PLANES64 = 2;           // searches of a 64x64 leaf refined at a time
constexpr int PLANE_WORDS = PLANES64 * plane_words(64);
static_assert(NGROUP * plane_words(32) <= PLANE_WORDS && NGROUP * plane_words(16) <= PLANE_WORDS,
              "every group's planes fit below 64x64");

// Chroma DC value and chroma-from-luma model of a leaf's component.
struct ChromaModel {
    int dc, sign, shift;
};

struct Smem {
    alignas(16) uint8_t cur_y[64 * 64];
    uint8_t cur_c[2][32 * 32];
    alignas(16) uint8_t rec_y[RY_H * RY_W];
    alignas(16) uint8_t rec_c[2][RC_H * RC_W];
    // qt_split snapshots, per depth: luma, cb, cr, grid (pre / parent; a
    // 64x64 parent that wins is coded again instead).
    // [luma | cb | cr] of a node, 6 bytes per 4 luma samples
    alignas(16) uint8_t snap0[1][6144], snap1[2][1536], snap2[2][384];
    MvCell snap_g[3][2][64];
    MvCell grid[64];
    Node nodes[QT_NODES];
    long long node_cost[QT_NODES];
    alignas(16) uint8_t pred[NPRED][64 * 64];
    union {
        // after the searches of a leaf
        struct {
            // chroma predictions (skip check), or the two chroma
            // options of an intra leaf: reconstruction and levels of option o,
            // component c in [2 * o + c]
            alignas(16) uint8_t cpred[4][32 * 32];
            int16_t clev[4][32 * 32];
        };
        // during them: sample planes
        alignas(16) uint32_t plane[PLANE_WORDS];
    };
    uint32_t cur_pair[64 * 32];      // leaf's source samples (x, x + cu / 2) as 16-bit lanes, for the searches
    uint8_t edge[2][EDGE_LEN];       // intra reference samples per direction (see build_refs)
    uint2 frag[4][32];        // transform fragments per lane: forward 8x8, inverse 8x8, forward 4x4, inverse 4x4
    MeGroup me[NGROUP];
    float4 quant[3][3][32];   // QuantLane parts per lane: luma 8x8, luma 4x4, chroma 4x4
    int win_slot;              // candidate slot of the last scan's winner (-1: skip)
    int acc[NCAND][2][2];      // per slot and TU size (8x8, 4x4): distortion, bits
    int cacc[2][2];            // per chroma option: distortion, bits
    ChromaModel cmodel[2];     // chroma DC and CfL model of the current leaf, per component
    uint16_t zoff[64];         // coded 8x8 cells before each cell of the CTU in z-order
    uint8_t leaf_skip[64];     // the cell's leaf is skipped
    int last_bits[65];         // last_bits(last) by last + 1
    long long acc64;
    int cl[NCAND];             // candidate list for job loops
    int cand_mvx[NPRED], cand_mvy[NPRED];   // refined vectors of the searches
    int next[2];               // work queues of luma_score: next item
    int dc;
    int above0;                // first sample of the above run (the planar mode's corner)
    int inexact;               // the merge prediction of the current leaf differs from the source
    long long best_cost;
    int sao[3];
    int band_sum[32], band_cnt[32], band_sq[32], band_new[32], band_cand[32];
    int ncoef;
    int16_t *coef;             // the CTU record's levels
    // levels of a 32x32 / 16x16 leaf while its split is tried
    alignas(8) int16_t lev1[32 * 48], lev2[16 * 24];
    alignas(8) unsigned long long tu8mask;
    // helper CTAs (see HelpCmd): their number; commands sent, and (helper)
    // received; acknowledgements received and expected
    int helpers;
    int *error;                // set to 1 when a wait gives up
    int cmd_sent, cmd_seq, acks, ack_goal;
    int cmd[6];
};

}  // namespace tcb

// tcb_resid.cuh — fused residual path of one 8x8 luma area (one 8x8 TU or
// four 4x4 TUs) or of four 4x4 chroma TUs on one warp: forward DCT-II (14-bit,
// two rounded passes) -> JND-band dead-zone quantisation -> RDOQ-lite
// (keep-vs-zero of |level| == 1) -> bit-model estimate -> centroid
// dequantisation -> inverse DCT -> reconstruction and SSE.
//
// The four transform passes run on the tensor cores (mma.sync f16, f32
// accumulators) and give the reference's integers exactly:
//
//  * A matrix entry C (|C| <= 10703) is split as 128 Ch + Cl with
//    |Ch| <= 84, |Cl| <= 64; the 16 rows of the A operand are the 8 rows of
//    Ch and the 8 rows of Cl, so one MMA gives both partial sums.
//  * The first pass multiplies the residuals (|r| <= 255, exact in f16).  The
//    later passes multiply intermediates t, |t| < 8192, split as 64 th + tl
//    with 0 <= tl < 64: k = 16 holds [64 C | C] against [th; tl].
//  * Every product is an integer and every accumulator starts at 1.5 * 2^23,
//    so its bits are 0x4B400000 + sum as long as |sum| < 2^22.  Residuals of
//    8-bit pictures have norm <= 2040, a non-zero level dequantises to at
//    most 1.75 |c| (q eff + eff / 6 with q eff <= |c| + eff / 3 and
//    eff <= 1.5 |c|), so no intermediate exceeds 3571 and no partial sum
//    182 * 3571 < 2^20.
//
// Data layout: lane l owns row l >> 2, columns 2 (l & 3) and 2 (l & 3) + 1 of
// the 8x8 area.  That is the C fragment of an m16n8 MMA (rows 0..7: the Ch
// sums, rows 8..15: the Cl sums of the same positions), and read as the next
// pass's B fragment it is its transpose, so the row pass feeds the column
// pass without a shuffle or shared memory.  Four 4x4 TUs are the same code
// with block-diagonal matrices.
//
// Compared with eight (four) lanes per TU and rows exchanged through shared
// memory: 150 instructions per area and type instead of about 250 per 8x8 TU
// and 50 per 4x4 TU, in a serial chain of about 150 instead of 1000, and
// 3 KB of code instead of 38 KB.
//
// Arithmetic follows reference src/transform.c:331-439 (dct4_point,
// dct8_point2, tc_fdct*/tc_idct*_res), src/encoder.c:333-385 (rdoq_level1,
// count_siglevel_bits, lastpos_cost) and tcodec_common.h:226-246
// (quant/dequant).
#pragma once
#include <math.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include "tcb_common.cuh"

namespace tcb {

// DCT matrices: one copy per translation unit (no relocatable device
// code); each unit that launches kernels using them uploads its copy with
// upload_dct_tables() before its first launch.
static __constant__ int c_dct4[4][4];
static __constant__ int c_dct8[8][8];

// Orthonormal DCT-II matrix in 14-bit fixed point:
// m[k][n] = round(2^14 * s_k * cos((2n+1) k pi / 2N)), s_0 = sqrt(1/N),
// s_k = sqrt(2/N).  Equals the reference tables of src/transform.c:313-329.
inline void dct_matrix(int N, int *m) {
    const double pi = 3.14159265358979323846;
    for (int k = 0; k < N; ++k)
        for (int n = 0; n < N; ++n) {
            const double s = k == 0 ? sqrt(1.0 / N) : sqrt(2.0 / N);
            m[k * N + n] = (int)lround(16384.0 * s * cos((2 * n + 1) * k * pi / (2.0 * N)));
        }
}

static inline cudaError_t upload_dct_tables() {
    int d4[4][4], d8[8][8];
    dct_matrix(4, &d4[0][0]);
    dct_matrix(8, &d8[0][0]);
    cudaError_t e = cudaMemcpyToSymbol(c_dct4, d4, sizeof(d4));
    if (e != cudaSuccess) return e;
    return cudaMemcpyToSymbol(c_dct8, d8, sizeof(d8));
}

struct QuantParams {
    int eff[4];
    // Per band: {quant step | dequantiser bias (eff / 6) << 16, reciprocal,
    // quantiser offset (eff / 3) | (eff <= 1) << 16, RDOQ threshold}.  A level
    // of magnitude 1 dequantises to dq = eff + eff / 6 and is dropped when
    // c^2 + lambda < (|c| - dq)^2 + 2 lambda (reference
    // src/encoder.c:333-355), i.e. when dq (2 |c| - dq) < lambda: for the
    // |c| below ceil((dq + ceil(lambda / dq)) / 2).
    uint4 band[4];
    __host__ __device__ void set_band(int b, int e, uint32_t r, long long lambda) {
        const int dq = e + e / 6;
        const long long thr = ((lambda + dq - 1) / dq + dq + 1) >> 1;
        eff[b] = e;
        band[b].x = (uint32_t)e | (uint32_t)(e / 6) << 16;
        band[b].y = r;
        band[b].z = (uint32_t)(e / 3) | (e <= 1 ? 1u << 16 : 0u);
        band[b].w = (uint32_t)(thr < 0x7FFFFFFF ? thr : 0x7FFFFFFF);
    }
};

// Frequency band of coefficient (row r, column c) of an N x N TU in raster
// order: DC, first quarter, second quarter, rest (the raster-index bands of
// freq_band).
__device__ __forceinline__ int band_rc(int N, int r, int c) { return freq_band(r * N + c, N * N); }

// A fragments of the forward (inv 0) or inverse (inv 1) transform for this
// lane: {64 Ch, 64 Cl, Ch, Cl} of matrix row lane >> 2, columns
// 2 (lane & 3) + {0, 1}; N = 4: two 4x4 matrices on the diagonal.
__device__ inline uint4 dct_fragment(int N, int inv, int lane) {
    const int m = lane >> 2;
    float ch[2], cl[2];
    for (int e = 0; e < 2; ++e) {
        const int k = 2 * (lane & 3) + e;
        int c = 0;
        if (N == 8) c = inv ? c_dct8[k][m] : c_dct8[m][k];
        else if ((k >> 2) == (m >> 2)) c = inv ? c_dct4[k & 3][m & 3] : c_dct4[m & 3][k & 3];
        const int h = (c + 64) >> 7;
        ch[e] = (float)h;
        cl[e] = (float)(c - 128 * h);
    }
    auto pack = [](float a, float b) {
        const __half2 v = __floats2half2_rn(a, b);
        return *reinterpret_cast<const uint32_t *>(&v);
    };
    return make_uint4(pack(64.f * ch[0], 64.f * ch[1]), pack(64.f * cl[0], 64.f * cl[1]), pack(ch[0], ch[1]),
                      pack(cl[0], cl[1]));
}

constexpr float MMA_BIAS = 12582912.0f;                  // 1.5 * 2^23, bits 0x4B400000
// -(0x4B400000 * 129) mod 2^32 plus the rounding term of the 14-bit shift
constexpr uint32_t MMA_UNBIAS = 0u - 0x4B400000u * 129u + 8192u;

__device__ __forceinline__ void mma_k8(float d[4], uint32_t a0, uint32_t a1, uint32_t b0) {
    d[0] = d[1] = d[2] = d[3] = MMA_BIAS;
    asm("mma.sync.aligned.m16n8k8.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5}, {%6}, {%0,%1,%2,%3};"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3]) : "r"(a0), "r"(a1), "r"(b0));
}
__device__ __forceinline__ void mma_k16(float d[4], const uint4 a, uint32_t b0, uint32_t b1) {
    d[0] = d[1] = d[2] = d[3] = MMA_BIAS;
    asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
        : "r"(a.x), "r"(a.y), "r"(a.z), "r"(a.w), "r"(b0), "r"(b1));
}
// Rounded 14-bit result of one position from its two partial sums (+ bias).
template <int BIAS>
__device__ __forceinline__ int mma_round(float hi, float lo) {
    return (int)((__float_as_uint(hi) << 7) + __float_as_uint(lo) + (MMA_UNBIAS + (uint32_t)BIAS * 16384u)) >> 14;
}
__device__ __forceinline__ uint32_t h2_sub(uint32_t a, uint32_t b) {
    const __half2 r = __hsub2(*reinterpret_cast<const __half2 *>(&a), *reinterpret_cast<const __half2 *>(&b));
    return *reinterpret_cast<const uint32_t *>(&r);
}
// B fragment halves of two intermediates given as t + 8192 (0..16383):
// hi = half2(t >> 6), lo = half2(t & 63).  0x6400 | v is the half 1024 + v.
__device__ __forceinline__ void split_b(int t0, int t1, uint32_t &hi, uint32_t &lo) {
    const uint32_t pk = __byte_perm((uint32_t)t0, (uint32_t)t1, 0x5410);
    lo = h2_sub((pk & 0x003F003Fu) | 0x64006400u, 0x64006400u);            // - 1024
    hi = h2_sub(((pk >> 6) & 0x03FF03FFu) | 0x64006400u, 0x64806480u);     // - (1024 + 8192 / 64)
}
// Two 8-bit samples (low 16 bits of v) as half2(1024 + v0, 1024 + v1).
__device__ __forceinline__ uint32_t bytes_h2(uint32_t v) { return __byte_perm(v, 0x64u, 0x4140); }

// One coefficient: dead-zone quantiser with RDOQ-lite.  Returns the level's
// magnitude; dq is the signed dequantised value.
__device__ __forceinline__ int quant_one(int c, const uint4 b, int &dq) {
    const int a = absi(c);
    const uint32_t n = (uint32_t)a + (b.z & 0xFFFFu);
    int q = (int)(__umulhi(n, b.y) + n * (b.z >> 16));     // step <= 1: reciprocal 0, level n
    if (q == 1 && a < (int)b.w) q = 0;
    const int m = q ? q * (int)(b.x & 0xFFFFu) + (int)(b.x >> 16) : 0;
    dq = c < 0 ? -m : m;
    return q;
}

// What the warp knows of one coded area.
struct AreaCode {
    int q0, q1;        // this lane's signed levels
    uint32_t rec;      // this lane's two reconstructed samples (low 16 bits)
    uint32_t sums;     // this lane's SSE << 10 | bit lengths of its levels
};

// Codes the area whose samples this lane holds two of: cv (source) and pv
// (prediction), 16 bits each, with the transform fragments f / i and the
// quantiser bands b0 / b1 of the lane's two positions.  All 32 lanes.
__device__ __forceinline__ AreaCode code_area(uint32_t cv, uint32_t pv, const uint4 f, const uint4 i, const uint4 b0,
                                              const uint4 b1) {
    AreaCode r;
    float d[4];
    uint32_t hi, lo;
    mma_k8(d, f.z, f.w, h2_sub(bytes_h2(cv), bytes_h2(pv)));
    split_b(mma_round<8192>(d[0], d[2]), mma_round<8192>(d[1], d[3]), hi, lo);
    mma_k16(d, f, hi, lo);
    const int c0 = mma_round<0>(d[0], d[2]), c1 = mma_round<0>(d[1], d[3]);
    int dq0, dq1;
    const int m0 = quant_one(c0, b0, dq0), m1 = quant_one(c1, b1, dq1);
    r.q0 = c0 < 0 ? -m0 : m0;
    r.q1 = c1 < 0 ? -m1 : m1;
    split_b(dq0 + 8192, dq1 + 8192, hi, lo);
    mma_k16(d, i, hi, lo);
    split_b(mma_round<8192>(d[0], d[2]), mma_round<8192>(d[1], d[3]), hi, lo);
    mma_k16(d, i, hi, lo);
    const int v0 = clampi((int)(pv & 0xFF) + mma_round<0>(d[0], d[2]), 0, 255);
    const int v1 = clampi((int)(pv >> 8) + mma_round<0>(d[1], d[3]), 0, 255);
    const int e0 = (int)(cv & 0xFF) - v0, e1 = (int)(cv >> 8) - v1;
    r.rec = (uint32_t)v0 | (uint32_t)v1 << 8;
    r.sums = ((uint32_t)(e0 * e0 + e1 * e1) << 10) + (uint32_t)(bitlen((unsigned)m0) + bitlen((unsigned)m1));
    return r;
}

// Bit estimate of a TU without its levels' bit lengths.  The reference counts
// 1 + 2 nz, a level term (1 for a zero, 2 + 2 bitlen otherwise) for every
// position up to the last and the last position's cost
// (src/encoder.c:360-385): with B the sum of the bit lengths that is
// 2 B + 2 + 3 nz + last + lastpos_cost(last), last = -1 for an empty TU.
__device__ __forceinline__ int tu_base_bits(int nz, int last) { return 2 + 3 * nz + last + lastpos_cost(last); }

// The 8x8 TU of the area: raster position of (lane, e) is 2 lane + e.
__device__ __forceinline__ int base_bits8(const AreaCode &c) {
    const unsigned n0 = __ballot_sync(0xffffffffu, c.q0 != 0), n1 = __ballot_sync(0xffffffffu, c.q1 != 0);
    const unsigned any = n0 | n1;
    const int h = 31 - __clz((int)any);
    const int last = any ? 2 * h + (int)((n1 >> h) & 1u) : -1;
    return tu_base_bits(__popc(n0) + __popc(n1), last);
}

// The lane's 4x4 TU (lanes of a quarter share bits 4 and 1 of their index,
// and within it the raster position grows with the lane index).
__device__ __forceinline__ int base_bits4(const AreaCode &c, int lane) {
    const unsigned qm = ((lane & 2) ? 0xCCCCCCCCu : 0x33333333u) & ((lane & 16) ? 0xFFFF0000u : 0x0000FFFFu);
    const unsigned n0 = __ballot_sync(0xffffffffu, c.q0 != 0) & qm, n1 = __ballot_sync(0xffffffffu, c.q1 != 0) & qm;
    const unsigned any = n0 | n1;
    const int h = 31 - __clz((int)any);
    const int last = any ? ((h >> 2) & 3) * 4 + (h & 1) * 2 + (int)((n1 >> h) & 1u) : -1;
    return tu_base_bits(__popc(n0) + __popc(n1), last);
}

}  // namespace tcb

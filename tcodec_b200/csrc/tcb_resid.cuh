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
//  * Every product is an integer and the accumulators start at about
//    1.5 * 2^23, so their bits are a constant plus the sum while
//    |sum| < 2^20.3.  Residuals of 8-bit pictures have norm <= 2040, a
//    non-zero level dequantises to at most 1.75 |c| (q eff + eff / 6 with
//    q eff <= |c| + eff / 3 and eff <= 1.5 |c|), so no intermediate exceeds
//    3571 and no partial sum 182 * 3571 < 2^20.
//  * The start values are chosen so that 128 Hi + Lo, modulo 2^32 (or 2^28
//    where only bits 14..27 are used), is the rounded sum with no correction.
//
// Data layout: lane l owns row l >> 2, columns 2 (l & 3) and 2 (l & 3) + 1 of
// the 8x8 area.  That is the C fragment of an m16n8 MMA (rows 0..7: the Ch
// sums, rows 8..15: the Cl sums of the same positions), and read as the next
// pass's B fragment it is its transpose, so the row pass feeds the column
// pass without a shuffle or shared memory.  Four 4x4 TUs are the same code
// with block-diagonal matrices.
//
// Compared with eight (four) lanes per TU and rows exchanged through shared
// memory: about 110 instructions per area and type with its bit estimate
// instead of about 300 per 8x8 TU and 90 per 4x4 TU, in a serial chain of the
// same length instead of 1000, and 3 KB of code instead of 38 KB.
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
    // Per band: {reciprocal, quantiser offset times reciprocal, smallest |c|
    // with a level, quant step | dequantiser bias (eff / 6) << 16}.  The level
    // is (|c| + eff / 3) / eff, as the high word of |c| rcp + off rcp (a step
    // of 1: reciprocal 2^32 - 1 and offset 1, which give |c|).  A level of
    // magnitude 1 dequantises to dq = eff + eff / 6 and is dropped when
    // c^2 + lambda < (|c| - dq)^2 + 2 lambda (reference
    // src/encoder.c:333-355), i.e. when dq (2 |c| - dq) < lambda: below
    // ceil((dq + ceil(lambda / dq)) / 2), if that lies in level 1's range.
    uint4 band[4];
    __host__ __device__ void set_band(int b, int e, uint32_t r, long long lambda) {
        const int off = e / 3, dq = e + e / 6;
        long long thr = ((lambda + dq - 1) / dq + dq + 1) >> 1;
        if (thr > 2 * e - off) thr = 2 * e - off;
        if (thr < e - off) thr = e - off;
        eff[b] = e;
        band[b].x = e <= 1 ? 0xFFFFFFFFu : r;
        band[b].y = e <= 1 ? 0xFFFFFFFFu : (uint32_t)off * r;
        band[b].z = (uint32_t)thr;
        band[b].w = (uint32_t)e | (uint32_t)(e / 6) << 16;
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

// Accumulator start values.  With 0x4B400000 the bits of 1.5 * 2^23,
// (bits(Hi) << 7) + bits(Lo) = 0xEB400000 + 128 dH + dL + sum (mod 2^32) for
// starts 1.5 * 2^23 + dH and + dL; dL = 8192 rounds the 14-bit shift.
//   EXACT: 128 dH = 2^32 - 0xEB400000, the word is sum + 8192;
//   FIELD: 128 dH = 2^27 - 0xEB400000 (mod 2^28), bits 14..27 are the rounded
//          result + 8192 (results within +-8191).
constexpr float ACC_LO = 12582912.0f + 8192.0f;
constexpr float ACC_EXACT = 12582912.0f + 2719744.0f, ACC_FIELD = 12582912.0f - 425984.0f;

struct MmaSums {
    float h0, h1, l0, l1;
    __device__ __forceinline__ uint32_t x0() const { return (__float_as_uint(h0) << 7) + __float_as_uint(l0); }
    __device__ __forceinline__ uint32_t x1() const { return (__float_as_uint(h1) << 7) + __float_as_uint(l1); }
};
__device__ __forceinline__ MmaSums mma_k8(uint32_t a0, uint32_t a1, uint32_t b0, float start) {
    MmaSums d;
    asm("mma.sync.aligned.m16n8k8.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5}, {%6}, {%7,%7,%8,%8};"
        : "=f"(d.h0), "=f"(d.h1), "=f"(d.l0), "=f"(d.l1) : "r"(a0), "r"(a1), "r"(b0), "f"(start), "f"(ACC_LO));
    return d;
}
__device__ __forceinline__ MmaSums mma_k16(const uint4 a, uint32_t b0, uint32_t b1, float start) {
    MmaSums d;
    asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%11,%11};"
        : "=f"(d.h0), "=f"(d.h1), "=f"(d.l0), "=f"(d.l1)
        : "r"(a.x), "r"(a.y), "r"(a.z), "r"(a.w), "r"(b0), "r"(b1), "f"(start), "f"(ACC_LO));
    return d;
}
__device__ __forceinline__ uint32_t h2_sub(uint32_t a, uint32_t b) {
    const __half2 r = __hsub2(*reinterpret_cast<const __half2 *>(&a), *reinterpret_cast<const __half2 *>(&b));
    return *reinterpret_cast<const uint32_t *>(&r);
}
// B fragment halves of two intermediates, each t + 8192 in the low 14 bits of
// its 16-bit lane of pk (the two bits above are ignored): hi = half2(t >> 6),
// lo = half2(t & 63).  0x6400 | v is the half 1024 + v.
__device__ __forceinline__ void split_b(uint32_t pk, uint32_t &hi, uint32_t &lo) {
    lo = h2_sub((pk & 0x003F003Fu) | 0x64006400u, 0x64006400u);            // - 1024
    hi = h2_sub(((pk >> 6) & 0x00FF00FFu) | 0x64006400u, 0x64806480u);     // - (1024 + 8192 / 64)
}
__device__ __forceinline__ void split_sums(const MmaSums &d, uint32_t &hi, uint32_t &lo) {
    split_b(__byte_perm(d.x0() >> 14, d.x1() << 2, 0x7610), hi, lo);
}
// Two 8-bit samples (low 16 bits of v) as half2(1024 + v0, 1024 + v1).
__device__ __forceinline__ uint32_t bytes_h2(uint32_t v) { return __byte_perm(v, 0x64u, 0x4140); }

// One coefficient: dead-zone quantiser with RDOQ-lite.  Returns the level's
// magnitude; dq is the signed dequantised value + 8192.
__device__ __forceinline__ int quant_one(int c, const uint4 b, int &dq) {
    const int a = absi(c);
    const bool zero = a < (int)b.z;
    int q = (int)(((unsigned long long)(unsigned)a * b.x + b.y) >> 32);
    int m = q * (int)(b.w & 0xFFFFu) + (int)(b.w >> 16);
    q = zero ? 0 : q;
    m = zero ? 0 : m;
    dq = (c < 0 ? -m : m) + 8192;
    return q;
}

// What the warp knows of one coded area.
struct AreaCode {
    int m0, m1;        // magnitudes of this lane's levels
    int c0, c1;        // its coefficients (whose signs the levels have)
    uint32_t rec;      // its two reconstructed samples (low 16 bits)
    int sse, bits;     // its SSE; 2 bitlen + 3 summed over its non-zero levels
    __device__ __forceinline__ uint32_t levels() const {   // two int16 levels
        return __byte_perm((uint32_t)(c0 < 0 ? -m0 : m0), (uint32_t)(c1 < 0 ? -m1 : m1), 0x5410);
    }
};

// Codes the area whose samples this lane holds two of: cv (source) and pv
// (prediction), 16 bits each, with the transform fragments f / i and the
// quantiser bands b0 / b1 of the lane's two positions.  All 32 lanes.
__device__ __forceinline__ AreaCode code_area(uint32_t cv, uint32_t pv, const uint4 f, const uint4 i, const uint4 b0,
                                              const uint4 b1) {
    AreaCode r;
    uint32_t hi, lo;
    split_sums(mma_k8(f.z, f.w, h2_sub(bytes_h2(cv), bytes_h2(pv)), ACC_FIELD), hi, lo);
    MmaSums d = mma_k16(f, hi, lo, ACC_EXACT);
    r.c0 = (int)d.x0() >> 14;
    r.c1 = (int)d.x1() >> 14;
    int dq0, dq1;
    r.m0 = quant_one(r.c0, b0, dq0);
    r.m1 = quant_one(r.c1, b1, dq1);
    split_b(__byte_perm((uint32_t)dq0, (uint32_t)dq1, 0x5410), hi, lo);
    split_sums(mma_k16(i, hi, lo, ACC_FIELD), hi, lo);
    d = mma_k16(i, hi, lo, ACC_EXACT);
    const int v0 = __viaddmin_s32_relu((int)(pv & 0xFF), (int)d.x0() >> 14, 255);   // clamped to 0..255
    const int v1 = __viaddmin_s32_relu((int)(pv >> 8), (int)d.x1() >> 14, 255);
    const int e0 = (int)(cv & 0xFF) - v0, e1 = (int)(cv >> 8) - v1;
    r.rec = (uint32_t)v0 | (uint32_t)v1 << 8;
    r.sse = e0 * e0 + e1 * e1;
    r.bits = 2 * (bitlen((unsigned)r.m0) + bitlen((unsigned)r.m1)) + (r.m0 ? 3 : 0) + (r.m1 ? 3 : 0);
    return r;
}

// Rest of a TU's bit estimate.  The reference counts 1 + 2 nz, a level term (1
// for a zero, 2 + 2 bitlen otherwise) for every position up to the last and
// the last position's cost (src/encoder.c:360-385): over all levels that is
// the sum of 2 bitlen + 3 over the non-zero ones plus last_bits(last),
// last = -1 for an empty TU.
__host__ __device__ __forceinline__ int last_bits(int last) { return 2 + last + lastpos_cost(last); }

// Last position + 1 of the area's 8x8 TU (0: empty): the raster position of
// (lane, e) is 2 lane + e.
__device__ __forceinline__ int last8(const AreaCode &c, int lane) {
    return (int)__reduce_max_sync(0xffffffffu, c.m1 ? 2u * lane + 2u : c.m0 ? 2u * lane + 1u : 0u);
}

// Of the lane's 4x4 TU (lanes of a quarter share bits 4 and 1 of their index,
// and within it the raster position grows with the lane index).
__device__ __forceinline__ int last4(const AreaCode &c, int lane) {
    const unsigned qm = ((lane & 2) ? 0xCCCCCCCCu : 0x33333333u) & ((lane & 16) ? 0xFFFF0000u : 0x0000FFFFu);
    const unsigned any = __ballot_sync(0xffffffffu, (c.m0 | c.m1) != 0) & qm, n1 = __ballot_sync(0xffffffffu, c.m1 != 0);
    const int h = 31 - __clz((int)any);
    return any ? ((h >> 2) & 3) * 4 + (h & 1) * 2 + 1 + (int)((n1 >> h) & 1u) : 0;
}

}  // namespace tcb

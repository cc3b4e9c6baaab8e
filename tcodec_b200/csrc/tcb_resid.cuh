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
//    Ch and the 8 rows of Cl, so one MMA gives both partial sums Sh and Sl.
//  * B operands are integers exact in f16 (|v| <= 2048): residuals
//    (|r| <= 255), first-pass results (|t| <= 722), and dequantised levels
//    and row-inverse results as f16(v) plus the remainder v - f16(v) (at most
//    1 here, where |v| <= 3571), against [C | C] with k = 16.
//  * Every product and sum is an integer below 2^24, so f32 holds it exactly:
//    residuals of 8-bit pictures have norm <= 2040, a non-zero level
//    dequantises to at most 1.75 |c| (q eff + eff / 6 with q eff <= |c| +
//    eff / 3 and eff <= 1.5 |c|), so no intermediate exceeds 3571 and no
//    partial sum 182 * 3571 < 2^20.
//  * The 14-bit rounding shift, floor((128 Sh + Sl + 8192) / 2^14), is taken
//    in f32 with round-down adds of 1.5 * 2^23, whose last bit is 1 (the
//    8192 is the accumulator's start value).
//
// Everything up to the reconstruction stays in f32: the FMA pipe issues one
// instruction a cycle where the integer ALU issues one every two, and the
// integer form of the same steps was bound by the latter (142 cycles a
// scheduler per area and TU size; now 125).
//
// Data layout: lane l owns row l >> 2, columns 2 (l & 3) and 2 (l & 3) + 1 of
// the 8x8 area.  That is the C fragment of an m16n8 MMA (rows 0..7: the Ch
// sums, rows 8..15: the Cl sums of the same positions), and read as the next
// pass's B fragment it is its transpose, so the row pass feeds the column
// pass without a shuffle or shared memory.  Four 4x4 TUs are the same code
// with block-diagonal matrices.
//
// Compared with eight (four) lanes per TU and rows exchanged through shared
// memory: about 100 instructions per area and type instead of about 300 per
// 8x8 TU and 90 per 4x4 TU, in a serial chain of the same length instead of
// 1000, and 3 KB of code instead of 38 KB.
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

// Quantiser of one coefficient position: 1 / eff, (eff / 3 + 1/2) / eff, the
// smallest |c| with a level, eff, and eff / 6, the dequantiser's bias.  The
// level is floor((|c| + eff / 3) / eff) = floor(|c| / eff + (eff / 3 + 1/2) /
// eff): the half keeps the sum 1 / (2 eff) away from every integer, far more
// than its f32 rounding (below 2^-22 of it, for |c| + eff / 3 < 2^13).  A level
// of magnitude 1 dequantises to dq = eff + eff / 6 and is dropped when
// c^2 + lambda < (|c| - dq)^2 + 2 lambda (reference src/encoder.c:333-355), i.e.
// when dq (2 |c| - dq) < lambda: below ceil((dq + ceil(lambda / dq)) / 2), if
// that lies in level 1's range.
struct QuantPos {
    float r, off, thr, eff, bias;
    __host__ __device__ QuantPos() {}
    __host__ __device__ QuantPos(int e, long long lambda) {
        const int o = e / 3, dq = e + e / 6;
        long long t = ((lambda + dq - 1) / dq + dq + 1) >> 1;
        if (t > 2 * e - o) t = 2 * e - o;
        if (t < e - o) t = e - o;
        r = 1.0f / (float)e;
        off = ((float)o + 0.5f) / (float)e;
        thr = (float)t;
        eff = (float)e;
        bias = (float)(e / 6);
    }
};
// The quantisers of a lane's two positions, as laid out in shared memory.
struct QuantLane {
    float4 a, b, c;      // r, off, thr, eff of each position; both biases
    __device__ __forceinline__ static QuantLane make(const QuantPos &p, const QuantPos &q) {
        return {make_float4(p.r, p.off, p.thr, p.eff), make_float4(q.r, q.off, q.thr, q.eff),
                make_float4(p.bias, q.bias, 0.0f, 0.0f)};
    }
};

// Frequency band of coefficient (row r, column c) of an N x N TU in raster
// order: DC, first quarter, second quarter, rest (the raster-index bands of
// freq_band).
__device__ __forceinline__ int band_rc(int N, int r, int c) { return freq_band(r * N + c, N * N); }

// A fragments of the forward (inv 0) or inverse (inv 1) transform for this
// lane: {Ch, Cl} of matrix row lane >> 2, columns 2 (lane & 3) + {0, 1};
// N = 4: two 4x4 matrices on the diagonal.
__device__ inline uint2 dct_fragment(int N, int inv, int lane) {
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
    return make_uint2(pack(ch[0], ch[1]), pack(cl[0], cl[1]));
}

struct MmaSums {
    float h0, h1, l0, l1;    // Sh and Sl + 8192 of the lane's two positions
};
__device__ __forceinline__ MmaSums mma_k8(const uint2 a, uint32_t b0) {
    MmaSums d;
    asm("mma.sync.aligned.m16n8k8.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5}, {%6}, {%7,%7,%8,%8};"
        : "=f"(d.h0), "=f"(d.h1), "=f"(d.l0), "=f"(d.l1) : "r"(a.x), "r"(a.y), "r"(b0), "f"(0.0f), "f"(8192.0f));
    return d;
}
__device__ __forceinline__ MmaSums mma_k16(const uint2 a, uint32_t b0, uint32_t b1) {
    MmaSums d;
    asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%4,%5}, {%6,%7}, {%8,%8,%9,%9};"
        : "=f"(d.h0), "=f"(d.h1), "=f"(d.l0), "=f"(d.l1)
        : "r"(a.x), "r"(a.y), "r"(b0), "r"(b1), "f"(0.0f), "f"(8192.0f));
    return d;
}
constexpr float RND = 12582912.0f;     // 1.5 * 2^23, bits 0x4B400000
// RND + floor((128 h + l) / 2^14): any sums, or (first pass) 128 |h| + |l| < 2^24.
__device__ __forceinline__ float shift14(float h, float l) {
    return __fmaf_rd(__fmaf_rd(l, 1.0f / 128, RND) + h, 1.0f / 128, RND - RND / 128);
}
__device__ __forceinline__ float shift14_small(float h, float l) {
    return __fmaf_rd(__fmaf_rn(h, 128.0f, l), 1.0f / 16384, RND);
}
__device__ __forceinline__ uint32_t pack_h2(float a, float b) {
    const __half2 v = __floats2half2_rn(a, b);
    return *reinterpret_cast<const uint32_t *>(&v);
}
__device__ __forceinline__ uint32_t h2_sub(uint32_t a, uint32_t b) {
    const __half2 r = __hsub2(*reinterpret_cast<const __half2 *>(&a), *reinterpret_cast<const __half2 *>(&b));
    return *reinterpret_cast<const uint32_t *>(&r);
}
// B operands of two integers below 2^14: f16 values and remainders, both exact
// (remainders of at most 1 within +-4095, of at most 4 beyond: the decoder passes
// up to 10,818, the block path up to 2^14).
__device__ __forceinline__ void split_h2(float a, float b, uint32_t &hi, uint32_t &lo) {
    const __half2 h = __floats2half2_rn(a, b);
    hi = *reinterpret_cast<const uint32_t *>(&h);
    lo = pack_h2(a - __low2float(h), b - __high2float(h));
}
// Two 8-bit samples (low 16 bits of v) as half2(1024 + v0, 1024 + v1).
__device__ __forceinline__ uint32_t bytes_h2(uint32_t v) { return __byte_perm(v, 0x64u, 0x4140); }

// What the warp knows of one coded area.
struct AreaCode {
    float z0, z1;      // 1 where this lane's level is non-zero, else 0
    float q0, q1;      // magnitudes of its levels
    float c0, c1;      // its coefficients (whose signs the levels have)
    uint32_t rec;      // its two reconstructed samples (low 16 bits)
    int e0, e1;        // its reconstruction errors
    __device__ __forceinline__ uint32_t levels() const {   // two int16 levels
        return __byte_perm(__float_as_uint(copysignf(q0, c0) + RND), __float_as_uint(copysignf(q1, c1) + RND), 0x5410);
    }
};
// A lane's sums over areas: SSE, exponents and number of non-zero levels.
struct AreaSums {
    int sse = 0;
    unsigned exps = 0;
    float nz = 0.0f;
    __device__ __forceinline__ void add(const AreaCode &c) {
        sse += c.e0 * c.e0 + c.e1 * c.e1;
        exps += (__float_as_uint(c.q0) >> 23) + (__float_as_uint(c.q1) >> 23);
        nz += c.z0 + c.z1;
    }
    // 2 bitlen + 3 over the non-zero levels: the exponent field of a level of
    // bit length n is 126 + n, that of zero 0
    __device__ __forceinline__ int bits() const { return 2 * (int)exps - 249 * (int)nz; }
};

// Codes the area whose samples this lane holds two of: cv (source) and pv
// (prediction), 16 bits each, with the transform fragments f / i and the
// lane's quantisers.  All 32 lanes.
__device__ __forceinline__ AreaCode code_area(uint32_t cv, uint32_t pv, const uint2 f, const uint2 i,
                                              const QuantLane &q) {
    AreaCode r;
    MmaSums d = mma_k8(f, h2_sub(bytes_h2(cv), bytes_h2(pv)));
    d = mma_k8(f, pack_h2(shift14_small(d.h0, d.l0) - RND, shift14_small(d.h1, d.l1) - RND));
    r.c0 = shift14(d.h0, d.l0) - RND;
    r.c1 = shift14(d.h1, d.l1) - RND;
    // dead-zone quantiser with RDOQ-lite, centroid dequantiser
    const float a0 = fabsf(r.c0), a1 = fabsf(r.c1);
    r.z0 = a0 >= q.a.z ? 1.0f : 0.0f;
    r.z1 = a1 >= q.b.z ? 1.0f : 0.0f;
    r.q0 = (__fadd_rd(__fmaf_rn(a0, q.a.x, q.a.y), RND) - RND) * r.z0;
    r.q1 = (__fadd_rd(__fmaf_rn(a1, q.b.x, q.b.y), RND) - RND) * r.z1;
    uint32_t hi, lo;
    split_h2(__fmaf_rn(r.q0, q.a.w, q.c.x) * copysignf(r.z0, r.c0), __fmaf_rn(r.q1, q.b.w, q.c.y) * copysignf(r.z1, r.c1),
             hi, lo);
    d = mma_k16(i, hi, lo);
    split_h2(shift14(d.h0, d.l0) - RND, shift14(d.h1, d.l1) - RND, hi, lo);
    d = mma_k16(i, hi, lo);
    // prediction + residual, clamped: the prediction carries minus the bits of RND
    const uint32_t p0 = __byte_perm(pv, 0xB4C00000u, 0x7650), p1 = __byte_perm(pv, 0xB4C00000u, 0x7651);
    const int v0 = __viaddmin_s32_relu((int)p0, __float_as_int(shift14(d.h0, d.l0)), 255);
    const int v1 = __viaddmin_s32_relu((int)p1, __float_as_int(shift14(d.h1, d.l1)), 255);
    r.e0 = (int)(cv & 0xFF) - v0;
    r.e1 = (int)(cv >> 8) - v1;
    r.rec = (uint32_t)v0 | (uint32_t)v1 << 8;
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
    return (int)__reduce_max_sync(0xffffffffu, c.z1 != 0.0f ? 2u * lane + 2u : c.z0 != 0.0f ? 2u * lane + 1u : 0u);
}

// Of the lane's 4x4 TU (lanes of a quarter share bits 4 and 1 of their index,
// and within it the raster position grows with the lane index).
__device__ __forceinline__ int last4(const AreaCode &c, int lane) {
    const unsigned qm = ((lane & 2) ? 0xCCCCCCCCu : 0x33333333u) & ((lane & 16) ? 0xFFFF0000u : 0x0000FFFFu);
    const unsigned any = __ballot_sync(0xffffffffu, c.z0 + c.z1 != 0.0f) & qm,
                   n1 = __ballot_sync(0xffffffffu, c.z1 != 0.0f);
    const int h = 31 - __clz((int)any);
    return any ? ((h >> 2) & 3) * 4 + (h & 1) * 2 + 1 + (int)((n1 >> h) & 1u) : 0;
}

}  // namespace tcb

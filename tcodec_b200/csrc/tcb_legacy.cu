// tcb_legacy.cu — reconstruction of the legacy (v0 / v1) 8x8 block path from
// parsed records (reference src/decoder.c:260-683); the encoder runs on the
// CTU engine's parts (tcb_legacy_enc.cuh).
//
// A CTA per CTU: one warp decodes the luma of block after block, two the Cb and
// Cr of the block before (chroma reads its own plane and, in intra blocks, the
// block's luma; luma reads no chroma), all four deblock.  Bound: the latency of
// a block's chain (references, prediction, two transform passes), 64 blocks in
// a row.  One warp per CTU that also fetched its records from memory and its
// matrices from constant memory (a lane each at its own entry, which the
// constant cache serialises) took 9.2 ms for a frame of 832x456, now 3.8.
//
// A CTU reads the reconstruction of its left, above and
// above-right neighbours (intra references, including the above-right 8
// samples of a block) and, where the reference reads samples not yet coded
// in raster order, the previous frame's reconstruction that the caller
// leaves in the output planes.  The wavefront therefore runs CTU (r, c) on
// diagonal c + 2r: its left, above and above-right neighbours lie on
// earlier diagonals, and every CTU whose samples it may read before they
// are coded (right and below-left) on later ones.  One launch per diagonal
// keeps that order without any inter-CTA waiting.
#include <cuda_runtime.h>
#include <math.h>

namespace tcb {
namespace legacy {
static __constant__ int c_ldct4[4][4];
static __constant__ int c_ldct8[8][8];
static __shared__ int s_ldct4[16], s_ldct8[64];    // their copies, per CTA
__device__ __forceinline__ int ldct4(int k, int n) { return s_ldct4[k * 4 + n]; }
__device__ __forceinline__ int ldct8(int k, int n) { return s_ldct8[k * 8 + n]; }
}  // namespace legacy
}  // namespace tcb

#include "tcb_legacy.cuh"
#include "tcb_launch.h"

namespace tcb {
namespace legacy {

constexpr int DT = 128;
__global__ void __launch_bounds__(DT) legacy_decode_kernel(LFrame F, const int *items) {
    __shared__ LState S[3];
    __shared__ __align__(4) LBlock B[BLOCKS];
    const int v = items[blockIdx.x], row = v >> 10, col = v & 1023, ox = col * 64, oy = row * 64;
    const int t = threadIdx.x, warp = t >> 5;
    const uint32_t *src = (const uint32_t *)(F.blocks + (size_t)(row * F.ctu_cols + col) * BLOCKS);
    static_assert(sizeof(LBlock) % 4 == 0, "records are copied in words");
    for (int i = t; i < (int)(BLOCKS * sizeof(LBlock) / 4); i += DT) ((uint32_t *)B)[i] = src[i];
    if (t < 64) s_ldct8[t] = c_ldct8[t >> 3][t & 7];
    else if (t < 80) s_ldct4[t - 64] = c_ldct4[(t - 64) >> 2][t & 3];
    __syncthreads();
    for (int step = 0; step <= BLOCKS; ++step) {
        const int b = warp == 0 ? step : step - 1, fx = ox + (b & 7) * 8, fy = oy + (b >> 3) * 8;
        if (warp < 3 && b >= 0 && b < BLOCKS && fx + 8 <= F.W && fy + 8 <= F.H && B[b].coded) {
            if (warp == 0) decode_luma(S[0], F, fx, fy, B[b]);
            else decode_chroma(S[warp], F, warp - 1, fx, fy, B[b]);
        }
        __syncthreads();
    }
    if (ox + 64 <= F.W && oy + 64 <= F.H) deblock_ctu(F, ox, oy, t, DT, [] { __syncthreads(); });
}

}  // namespace legacy

// DCT-II matrices in 14-bit fixed point from their closed form
// (m[k][n] = round(2^14 s_k cos((2n+1) k pi / 2N))), equal to the reference
// tables of src/transform.c:313-329.
cudaError_t upload_legacy_tables() {
    static bool done[64] = {};
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    if (dev >= 0 && dev < 64 && done[dev]) return cudaSuccess;
    int d4[4][4], d8[8][8];
    const double pi = 3.14159265358979323846;
    for (int N = 4; N <= 8; N += 4)
        for (int k = 0; k < N; ++k)
            for (int m = 0; m < N; ++m) {
                const double s = k == 0 ? sqrt(1.0 / N) : sqrt(2.0 / N);
                const int v = (int)lround(16384.0 * s * cos((2 * m + 1) * k * pi / (2.0 * N)));
                if (N == 4) d4[k][m] = v; else d8[k][m] = v;
            }
    if ((e = cudaMemcpyToSymbol(legacy::c_ldct4, d4, sizeof(d4))) != cudaSuccess) return e;
    if ((e = cudaMemcpyToSymbol(legacy::c_ldct8, d8, sizeof(d8))) != cudaSuccess) return e;
    if (dev >= 0 && dev < 64) done[dev] = true;
    return cudaSuccess;
}

cudaError_t launch_legacy_decode(const legacy::LFrame &F, const int *d_items, int n, cudaStream_t st) {
    if (n <= 0) return cudaSuccess;
    legacy::legacy_decode_kernel<<<n, legacy::DT, 0, st>>>(F, d_items);
    return cudaGetLastError();
}

}  // namespace tcb

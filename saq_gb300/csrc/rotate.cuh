// Rotation of many rows by a segment's matrix, out[v][o] = sum_j x[v][j] P[j][o] in
// the order of Eigen's GEMV (GeneralMatrixVector.h:108-300): per output one FMA
// chain per block of 16 inputs (one chain when dim < 128), the blocks added in
// order.  Shared by the index build (vectors of a chunk) and the batched search
// (queries).
//
// Bound: FP32 FMAs (2 dim^2 per row, no tensor-core form rounds like this) and, next
// to them, shared memory filling registers.  Tile: 128 rows x 64 outputs per CTA of
// 128 threads, 8 x 8 per thread, the largest that leaves room for both sums (chain
// and folded) of every output: four 16-byte shared loads feed 64 FMAs.  Dims are
// multiples of 64, so no output column is padding.  Two rows share a packed FMA
// (fma.rn.f32x2, each half rounded as fmaf), which halves the issue slots.  The next
// 16 inputs are in registers while the current ones are multiplied.
#pragma once

#include <cstdint>

namespace saqg {

constexpr int kRotM = 128, kRotN = 64, kRotK = 16, kRotThreads = 128;
constexpr int kRotXs = kRotM + 4;  // row length of the transposed row tile

__device__ __forceinline__ uint64_t f2_pack(float lo, float hi) {
    return (uint64_t)__float_as_uint(lo) | ((uint64_t)__float_as_uint(hi) << 32);
}
__device__ __forceinline__ float f2_lo(uint64_t v) { return __uint_as_float((uint32_t)v); }
__device__ __forceinline__ float f2_hi(uint64_t v) { return __uint_as_float((uint32_t)(v >> 32)); }
__device__ __forceinline__ uint64_t f2_fma(uint64_t a, uint64_t b, uint64_t c) {
    uint64_t d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
    return d;
}
__device__ __forceinline__ uint64_t f2_add(uint64_t a, uint64_t b) {
    uint64_t d;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}

// The tile of rows [v0, v0 + 128) and outputs [o0, o0 + 64).  load4(v, j): inputs
// j .. j + 3 (j a multiple of 4) of row v, zeros past the end; store(v, o, r): the
// thread's outputs, r[i][b] of row v + i and output o + b (v a multiple of 8, o of
// 4; rows past the end included; called for either half of the outputs).  P is 16-byte aligned.
template <class Load, class Store>
__device__ __forceinline__ void rotate_tile(int dim, const float *__restrict__ P, int64_t v0, int o0, Load load4,
                                            Store store) {
    __shared__ __align__(16) float xs[2][kRotK][kRotXs];
    __shared__ __align__(16) float ps[2][kRotK][kRotN];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    // compute: warp w the rows 32 w .., lane (ly, lx) of 4 x 8
    const int vt = warp * 32 + (lane >> 3) * 8, ot = (lane & 7) * 4;  // outputs ot .. and 32 + ot ..
    // copy: rows xr + 32 i, inputs xk .. xk + 3; matrix rows pr + 8 i, columns pc .. pc + 3
    const int xr = tid >> 2, xk = (tid & 3) * 4, pr = tid >> 4, pc = (tid & 15) * 4;
    const bool fold16 = dim >= 128;
    uint64_t res[4][8], c[4][8];
#pragma unroll
    for (int a = 0; a < 4; ++a)
#pragma unroll
        for (int b = 0; b < 8; ++b) res[a][b] = c[a][b] = 0ull;
    float4 xv[4], pv[2];
    auto fetch = [&](int j0) {
#pragma unroll
        for (int i = 0; i < 4; ++i) xv[i] = load4(v0 + xr + 32 * i, j0 + xk);
#pragma unroll
        for (int i = 0; i < 2; ++i)
            pv[i] = *reinterpret_cast<const float4 *>(P + (size_t)(j0 + pr + 8 * i) * dim + o0 + pc);
    };
    auto put = [&](int s) {
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            xs[s][xk][xr + 32 * i] = xv[i].x;
            xs[s][xk + 1][xr + 32 * i] = xv[i].y;
            xs[s][xk + 2][xr + 32 * i] = xv[i].z;
            xs[s][xk + 3][xr + 32 * i] = xv[i].w;
        }
#pragma unroll
        for (int i = 0; i < 2; ++i) *reinterpret_cast<float4 *>(&ps[s][pr + 8 * i][pc]) = pv[i];
    };
    fetch(0);
    put(0);
    __syncthreads();
#pragma unroll 1
    for (int j0 = 0, s = 0; j0 < dim; j0 += kRotK, s ^= 1) {
        const bool more = j0 + kRotK < dim;
        if (more) fetch(j0 + kRotK);
        if (fold16 || j0 == 0) {  // a chain starts
#pragma unroll
            for (int a = 0; a < 4; ++a)
#pragma unroll
                for (int b = 0; b < 8; ++b) c[a][b] = 0ull;
        }
#pragma unroll
        for (int k = 0; k < kRotK; ++k) {
            const ulonglong2 x0 = *reinterpret_cast<const ulonglong2 *>(&xs[s][k][vt]);
            const ulonglong2 x1 = *reinterpret_cast<const ulonglong2 *>(&xs[s][k][vt + 4]);
            const float4 p0 = *reinterpret_cast<const float4 *>(&ps[s][k][ot]);
            const float4 p1 = *reinterpret_cast<const float4 *>(&ps[s][k][32 + ot]);
            const uint64_t x[4] = {x0.x, x0.y, x1.x, x1.y};
            const float p[8] = {p0.x, p0.y, p0.z, p0.w, p1.x, p1.y, p1.z, p1.w};
#pragma unroll
            for (int b = 0; b < 8; ++b) {
                const uint64_t pp = f2_pack(p[b], p[b]);
#pragma unroll
                for (int a = 0; a < 4; ++a) c[a][b] = f2_fma(pp, x[a], c[a][b]);
            }
        }
        if (fold16 || !more) {
#pragma unroll
            for (int a = 0; a < 4; ++a)
#pragma unroll
                for (int b = 0; b < 8; ++b) res[a][b] = f2_add(c[a][b], res[a][b]);
        }
        if (more) put(s ^ 1);
        __syncthreads();
    }
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        float r[8][4];
#pragma unroll
        for (int a = 0; a < 4; ++a)
#pragma unroll
            for (int b = 0; b < 4; ++b) {
                r[2 * a][b] = f2_lo(res[a][4 * h + b]);
                r[2 * a + 1][b] = f2_hi(res[a][4 * h + b]);
            }
        store(v0 + vt, o0 + 32 * h + ot, r);
    }
}

}  // namespace saqg

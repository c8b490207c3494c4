// Device primitives that reproduce the reference's floating-point order.
//
// The reference (saqlib/, compiled with -O3 -march=native -ffp-contract=off on
// an AVX-512 host) evaluates its float reductions in fixed SIMD orders.  A
// 32-lane warp maps onto them directly:
//   * Eigen's vectorised sum (Eigen/src/Core/Redux.h:227-283): two 16-lane
//     accumulators take the even and odd 16-float packets; lanes 0-15 of the
//     warp hold accumulator 0, lanes 16-31 accumulator 1.
//   * predux<Packet16f> and GCC's _mm512_reduce_add_ps: lane i + lane i+8,
//     then +4, +2, +1 -- exactly a 16-wide shfl_down tree.
//   * _mm512_reduce_min_ps(_mm512_min_ps(a, b)): the same tree with x86
//     min semantics ((a < b) ? a : b, second operand on NaN).
// This translation unit is compiled with --fmad=false; every FMA below is an
// explicit fmaf(), matching the reference's explicit _mm512_fmadd_ps calls.
#pragma once

#include <cstdint>

namespace saqg {

constexpr unsigned kFull = 0xffffffffu;

__device__ __forceinline__ float minps(float a, float b) { return a < b ? a : b; }
__device__ __forceinline__ float maxps(float a, float b) { return a > b ? a : b; }

// Eigen redux over n elements, one warp.  f(i) yields element i (already
// rounded on its own).  Result returned to every lane.
template <class F>
__device__ __forceinline__ float warp_eigen_sum(int n, F f) {
    const int lane = threadIdx.x & 31, l = lane & 15, half = lane >> 4;
    const int aligned = n & ~15, aligned2 = n & ~31;
    float r;
    if (aligned == 0) {
        r = 0.0f;
        if (lane == 0 && n > 0) {
            r = f(0);
            for (int i = 1; i < n; ++i) r = __fadd_rn(r, f(i));
        }
        return __shfl_sync(kFull, r, 0);
    }
    float acc;
    if (aligned > 16) {
        acc = f(16 * half + l);
        for (int p = half + 2; p < aligned2 / 16; p += 2) acc = __fadd_rn(acc, f(16 * p + l));
        const float other = __shfl_down_sync(kFull, acc, 16);
        acc = __fadd_rn(acc, other);
        if (aligned > aligned2 && lane < 16) acc = __fadd_rn(acc, f(aligned2 + l));
    } else {
        acc = lane < 16 ? f(l) : 0.0f;
    }
    acc = __fadd_rn(acc, __shfl_down_sync(kFull, acc, 8));
    acc = __fadd_rn(acc, __shfl_down_sync(kFull, acc, 4));
    acc = __fadd_rn(acc, __shfl_down_sync(kFull, acc, 2));
    acc = __fadd_rn(acc, __shfl_down_sync(kFull, acc, 1));
    r = acc;
    if (lane == 0)
        for (int i = aligned; i < n; ++i) r = __fadd_rn(r, f(i));
    return __shfl_sync(kFull, r, 0);
}

// 16-lane add tree inside a half-warp (lane l of the half holds lane l of the
// SIMD accumulator).  Result valid in the half's lane 0.
__device__ __forceinline__ float half_reduce16(float v, unsigned mask) {
    v = __fadd_rn(v, __shfl_down_sync(mask, v, 8, 16));
    v = __fadd_rn(v, __shfl_down_sync(mask, v, 4, 16));
    v = __fadd_rn(v, __shfl_down_sync(mask, v, 2, 16));
    v = __fadd_rn(v, __shfl_down_sync(mask, v, 1, 16));
    return v;
}

// _mm512_reduce_min_ps(_mm512_min_ps(d[0..15], d[16..31])) with lane j holding d[j].
__device__ __forceinline__ float warp_min_tree(float x) {
    float v = minps(x, __shfl_down_sync(kFull, x, 16));  // (a < b) ? a : b, a = lanes 0-15
    float o = __shfl_down_sync(kFull, v, 8);
    v = minps(o, v);                                     // T3 = min(upper, lower)
    o = __shfl_down_sync(kFull, v, 4);
    v = minps(o, v);                                     // T6
    o = __shfl_down_sync(kFull, v, 2);
    v = minps(v, o);                                     // T8 = min(T6, shuffled)
    o = __shfl_down_sync(kFull, v, 1);
    v = minps(v, o);                                     // T10
    return __shfl_sync(kFull, v, 0);
}

// --------------------------------------------------------------- ex-codes
// CodeHelper<B>::compute_ip (code_helper.hpp) by a half-warp: lane l accumulates
// dims l, l+16, l+32, ... in increasing order, as SIMD lane l does, reading the
// bytes that the reference's compacted layouts give that lane (the same positions
// in every 64 dims) straight from global memory, 16 consecutive bytes per half-warp
// load.  The query is in ex order: within every 64 dims, lane l's four values (dims
// l, 16+l, 32+l, 48+l) lie together at 4l, one 16-byte load.
__device__ __forceinline__ int ex_order(int d) { return (d & ~63) | ((d & 15) << 2) | ((d >> 4) & 3); }

// The integer in the bits of `field` at position SH and up, as a float: set under
// the mantissa of 2^(23-SH), whose last place then counts 2^-SH; the difference is
// exact.  No shift and no conversion instruction.
template <int SH>
__device__ __forceinline__ float bits_float(uint32_t field) {
    return __fsub_rn(__uint_as_float(field | (0x4b000000u - ((uint32_t)SH << 23))), __uint_as_float(0x4b000000u - ((uint32_t)SH << 23)));
}

// What lane l reads of 64 dims of a B-bit code, and its four values from that.
template <int B>
struct Ex64 {
    static constexpr int kLoads = B <= 2 ? 1 : B == 3 || B == 4 ? 2 : B == 6 ? 3 : 4;
    uint32_t r[kLoads];
    __device__ __forceinline__ void load(const uint8_t *__restrict__ g, int l) {
        if (B == 1) {  // bit d of the little-endian string: this lane's bits in the words' places
            const uint2 w = *reinterpret_cast<const uint2 *>(g);
            r[0] = ((w.x >> l) & 1u) | (((w.x >> (16 + l)) & 1u) << 1) | (((w.y >> l) & 1u) << 2) |
                   (((w.y >> (16 + l)) & 1u) << 3);
        } else {
            r[0] = g[l];
            if (B == 3) r[1] = g[16 + (l & 7)];  // top bit of dim 16k + l: bit 2k + (l >> 3)
            if (B >= 4) r[1] = g[16 + l];
            if (B >= 6) r[2] = g[32 + l];
            if (B == 7) r[3] = g[48 + (l & 7)];  // as for 3 bits
            if (B == 8) r[3] = g[48 + l];
        }
    }
    __device__ __forceinline__ void values(int l, float (&v)[4]) const {
        if (B == 2 || B == 3) {
            const uint32_t t = B == 3 ? (r[kLoads - 1] >> (l >> 3)) << 2 : 0u;
            v[0] = bits_float<0>((r[0] & 0x03u) | (t & 0x04u));
            v[1] = bits_float<2>((r[0] & 0x0cu) | (t & 0x10u));
            v[2] = bits_float<4>((r[0] & 0x30u) | (t & 0x40u));
            v[3] = bits_float<6>((r[0] & 0xc0u) | (t & 0x100u));
        } else if (B == 4) {
            v[0] = bits_float<0>(r[0] & 0x0fu);
            v[1] = bits_float<4>(r[0] & 0xf0u);
            v[2] = bits_float<0>(r[kLoads - 1] & 0x0fu);
            v[3] = bits_float<4>(r[kLoads - 1] & 0xf0u);
        } else if (B == 6 || B == 7) {
            const uint32_t b0 = r[0], b1 = r[1 % kLoads], b2 = r[2 % kLoads];
            const uint32_t t = B == 7 ? r[kLoads - 1] >> (l >> 3) : 0u;
            v[0] = bits_float<0>((b0 & 0x3fu) | ((t << 6) & 0x40u));
            v[1] = bits_float<0>((b1 & 0x3fu) | ((t << 4) & 0x40u));
            v[2] = bits_float<0>(((b0 >> 2) & 0x30u) | (b2 & 0x0fu) | ((t << 2) & 0x40u));
            v[3] = bits_float<4>((b2 & 0xf0u) | ((b1 << 2) & 0x300u) | ((t << 4) & 0x400u));
        } else if (B == 8) {
#pragma unroll
            for (int k = 0; k < 4; ++k) v[k] = bits_float<0>(r[k % kLoads]);
        }
    }
    __device__ __forceinline__ void add(int l, const float4 &q, float &acc) const {
        if (B == 1) {  // masked adds
            acc = __fadd_rn(acc, (r[0] & 1u) ? q.x : 0.0f);
            acc = __fadd_rn(acc, (r[0] & 2u) ? q.y : 0.0f);
            acc = __fadd_rn(acc, (r[0] & 4u) ? q.z : 0.0f);
            acc = __fadd_rn(acc, (r[0] & 8u) ? q.w : 0.0f);
        } else {
            float v[4];
            values(l, v);
            acc = fmaf(v[0], q.x, acc);
            acc = fmaf(v[1], q.y, acc);
            acc = fmaf(v[2], q.z, acc);
            acc = fmaf(v[3], q.w, acc);
        }
    }
};

// Every lane of the warp takes part (both halves with the same D); the half's
// result is valid in its lane 0.  Four groups' codes are loaded ahead of their
// chain: the chain of a lane is D / 16 FMAs, and a load per step would wait D / 64
// times.
template <int B>
__device__ __forceinline__ float ip16_bits(const float *__restrict__ q, const uint8_t *__restrict__ y, int D, int l) {
    const float4 *q4 = reinterpret_cast<const float4 *>(q) + l;
    const int G = D / 64;
    float acc = 0.0f;
    int g = 0;
    for (; g + 4 <= G; g += 4) {
        Ex64<B> e[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) e[u].load(y + (g + u) * 8 * B, l);
#pragma unroll
        for (int u = 0; u < 4; ++u) e[u].add(l, q4[(g + u) * 16], acc);
    }
    for (; g < G; ++g) {
        Ex64<B> e;
        e.load(y + g * 8 * B, l);
        e.add(l, q4[g * 16], acc);
    }
    return half_reduce16(acc, kFull);
}

__device__ __forceinline__ float ip16_8(const float *__restrict__ q, const uint8_t *__restrict__ y, int D, int bits, int l) {
    switch (bits) {
    case 1:
        return ip16_bits<1>(q, y, D, l);
    case 2:
        return ip16_bits<2>(q, y, D, l);
    case 3:
        return ip16_bits<3>(q, y, D, l);
    case 4:
        return ip16_bits<4>(q, y, D, l);
    case 5: {  // CodeHelper<5>::compute_ip = 2 * IP4(top 4 bits) + IP1(low bit)
        const float a = ip16_bits<4>(q, y, D, l);
        const float b = ip16_bits<1>(q, y + D / 2, D, l);
        return __fadd_rn(2.0f * a, b);
    }
    case 6:
        return ip16_bits<6>(q, y, D, l);
    case 7:
        return ip16_bits<7>(q, y, D, l);
    case 8:
        return ip16_bits<8>(q, y, D, l);
    default:
        return 0.0f;
    }
}

// get_IP_FUNC(ex_bits)(q, y, D) (code_helper.hpp:599-640) by half-warps, q in ex
// order.  One copy per kernel: the callers' loops are short beside it.
static __device__ __noinline__ float excode_ip16(const float *__restrict__ q, const uint8_t *__restrict__ y, int D, int exb) {
    const int l = threadIdx.x & 15;
    if (exb > 8)  // CodeHelper<B>::compute_ip, B > 8: IP8(low bytes) + 256 * IP(rest)
        return __fadd_rn(ip16_bits<8>(q, y, D, l), 256.0f * ip16_8(q, y + D, D, exb - 8, l));
    return ip16_8(q, y, D, exb, l);
}

// ---- the same inner products computed by ONE thread: the 16 SIMD lanes of
// CodeHelper<B>::compute_ip become 16 independent accumulators (lane l takes
// dims l, l+16, ... in increasing order), reduced with the same 16->1 tree.
// Bit-identical to the half-warp form, about half its instructions per vector (no
// reduction across lanes) but its whole length in one thread: used where many
// candidate vectors are re-ranked at once (one thread per vector and segment).
// The query is in ex order here too.
__device__ __forceinline__ float tree16(const float *a) {
    float x[8], y[4];
#pragma unroll
    for (int i = 0; i < 8; ++i) x[i] = __fadd_rn(a[i], a[i + 8]);
#pragma unroll
    for (int i = 0; i < 4; ++i) y[i] = __fadd_rn(x[i], x[i + 4]);
    return __fadd_rn(__fadd_rn(y[0], y[2]), __fadd_rn(y[1], y[3]));
}

template <int B>
__device__ __forceinline__ float ip_thread_bits(const float *__restrict__ q, const uint8_t *__restrict__ y, int D) {
    float acc[16];
#pragma unroll
    for (int l = 0; l < 16; ++l) acc[l] = 0.0f;
    uint32_t nxt[2 * B];  // a group's 8 B bytes (groups of odd widths are 8-byte aligned)
    auto fetch = [&](int g) {
        const uint8_t *gp = y + g * 8 * B;
        if (B % 2 == 0) {
#pragma unroll
            for (int i = 0; i < B / 2; ++i) {
                const uint4 v = reinterpret_cast<const uint4 *>(gp)[i];
                nxt[4 * i] = v.x, nxt[4 * i + 1] = v.y, nxt[4 * i + 2] = v.z, nxt[4 * i + 3] = v.w;
            }
        } else {
#pragma unroll
            for (int i = 0; i < B; ++i) {
                const uint2 v = reinterpret_cast<const uint2 *>(gp)[i];
                nxt[2 * i] = v.x, nxt[2 * i + 1] = v.y;
            }
        }
    };
    constexpr bool kAhead = B <= 4;  // the next group's words in flight (wider codes: too many registers)
    if (kAhead) fetch(0);
    for (int g = 0; g < D / 64; ++g) {
        if (!kAhead) fetch(g);
        uint32_t w[2 * B];
#pragma unroll
        for (int i = 0; i < 2 * B; ++i) w[i] = nxt[i];
        if (kAhead && g + 1 < D / 64) fetch(g + 1);
        auto byte = [&](int i) { return __byte_perm(w[(i >> 2) % (2 * B)], 0u, 0x4440u | (i & 3)); };
        const float4 *q4 = reinterpret_cast<const float4 *>(q + 64 * g);
#pragma unroll
        for (int l = 0; l < 16; ++l) {  // what SIMD lane l reads, as Ex64::load
            Ex64<B> e;
            if (B == 1) {
                e.r[0] = ((w[0] >> l) & 1u) | (((w[0] >> (16 + l)) & 1u) << 1) | (((w[1] >> l) & 1u) << 2) |
                         (((w[1] >> (16 + l)) & 1u) << 3);
            } else {
                e.r[0] = byte(l);
                if (B == 3) e.r[1] = byte(16 + (l & 7));
                if (B >= 4) e.r[1] = byte(16 + l);
                if (B >= 6) e.r[2] = byte(32 + l);
                if (B == 7) e.r[3] = byte(48 + (l & 7));
                if (B == 8) e.r[3] = byte(48 + l);
            }
            e.add(l, q4[l], acc[l]);
        }
    }
    return tree16(acc);
}

__device__ __forceinline__ float ip8_thread(const float *__restrict__ q, const uint8_t *__restrict__ y, int D, int bits) {
    switch (bits) {
    case 1:
        return ip_thread_bits<1>(q, y, D);
    case 2:
        return ip_thread_bits<2>(q, y, D);
    case 3:
        return ip_thread_bits<3>(q, y, D);
    case 4:
        return ip_thread_bits<4>(q, y, D);
    case 5:
        return __fadd_rn(2.0f * ip_thread_bits<4>(q, y, D), ip_thread_bits<1>(q, y + D / 2, D));
    case 6:
        return ip_thread_bits<6>(q, y, D);
    case 7:
        return ip_thread_bits<7>(q, y, D);
    case 8:
        return ip_thread_bits<8>(q, y, D);
    default:
        return 0.0f;
    }
}

// get_IP_FUNC(ex_bits)(q, y, D) by one thread.
static __device__ __noinline__ float excode_ip_thread(const float *__restrict__ q, const uint8_t *__restrict__ y, int D,
                                                      int exb) {
    if (exb == 0) return 0.0f;
    if (exb > 8) return __fadd_rn(ip8_thread(q, y, D, 8), 256.0f * ip8_thread(q, y + D, D, exb - 8));
    return ip8_thread(q, y, D, exb);
}

// CaqCluEstimator::compAccurateDist + Lut::getExtIP, L2 (caq_estimator.hpp:190-217, lut.hpp:121-126)
__device__ __forceinline__ float accurate_dist(float onorm, float ipx, float ex_ip, float rescale, int bits, float sum_q,
                                               float q_l2sqr) {
    const float o2 = __fmul_rn(onorm, onorm);
    if (bits == 0) return __fadd_rn(o2, q_l2sqr);
    const float dl = (float)(2.0 / (double)(1 << bits));
    const double e = __dadd_rn(__dadd_rn((double)ipx, __dmul_rn((double)ex_ip, (double)dl)),
                               __dmul_rn(__dadd_rn(-1.0, (double)(dl / 2)), (double)sum_q));
    const float ipoq = __fmul_rn(rescale, (float)e);
    return __fsub_rn(__fadd_rn(o2, q_l2sqr), __fmul_rn(2.0f, ipoq));
}

}  // namespace saqg

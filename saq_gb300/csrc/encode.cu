// Encode path: CAQEncoder (quantization/caq/caq_encoder.hpp) on the GPU.
//
// The code adjustment is a sequential coordinate descent in FP64 whose every
// accepted move changes the running <o,o_a> and |o_a|^2 read by the next
// dimension (caq_encoder.hpp:57-142); bit-exact codes need the reference's
// exact FP64 sums, so one thread owns one vector and walks its dimensions in
// order (caq_encode_one).  In index construction the 32 lanes of a warp encode
// 32 vectors whose residuals and codes are interleaved by dimension, so every
// step of the 32 chains is one coalesced access.  This file is compiled with
// --fmad=false: no multiply is fused into an add unless written as fma().
#include <cfloat>
#include <cmath>
#include <cstring>
#include <memory>
#include <type_traits>
#include <vector>

#include "device_common.cuh"
#include "rotate.cuh"
#include "saqg_internal.h"

namespace saqg {

namespace {

// Eigen's 16-lane two-accumulator float sum (Redux.h:227-283) in one thread.
template <class F>
__device__ float thread_eigen_sum(int n, F f) {
    const int aligned = n & ~15, aligned2 = n & ~31;
    if (aligned == 0) {
        float r = f(0);
        for (int i = 1; i < n; ++i) r = __fadd_rn(r, f(i));
        return r;
    }
    float r0[16], r1[16];
#pragma unroll
    for (int l = 0; l < 16; ++l) r0[l] = f(l);
    if (aligned > 16) {
#pragma unroll
        for (int l = 0; l < 16; ++l) r1[l] = f(16 + l);
        for (int idx = 32; idx < aligned2; idx += 32)
#pragma unroll
            for (int l = 0; l < 16; ++l) {
                r0[l] = __fadd_rn(r0[l], f(idx + l));
                r1[l] = __fadd_rn(r1[l], f(idx + 16 + l));
            }
#pragma unroll
        for (int l = 0; l < 16; ++l) r0[l] = __fadd_rn(r0[l], r1[l]);
        if (aligned > aligned2)
#pragma unroll
            for (int l = 0; l < 16; ++l) r0[l] = __fadd_rn(r0[l], f(aligned2 + l));
    }
    float x[8], y[4];
#pragma unroll
    for (int i = 0; i < 8; ++i) x[i] = __fadd_rn(r0[i], r0[i + 8]);
#pragma unroll
    for (int i = 0; i < 4; ++i) y[i] = __fadd_rn(x[i], x[i + 4]);
    float r = __fadd_rn(__fadd_rn(y[0], y[2]), __fadd_rn(y[1], y[3]));
    for (int i = aligned; i < n; ++i) r = __fadd_rn(r, f(i));
    return r;
}

// x as a double.  Normal floats take integer operations (widening the exponent,
// shifting the mantissa): FP64 and its conversions run at 1/64 of the FP32 rate here.
__device__ __forceinline__ double widen(float x) {
    const uint32_t u = __float_as_uint(x);
    if ((u & 0x7f800000u) - 0x00800000u >= 0x7f000000u) return (double)x;  // zero, denormal, inf, NaN
    return __hiloint2double((int)((u & 0x80000000u) | (((u & 0x7fffffffu) >> 3) + 0x38000000u)), (int)(u << 29));
}

// A double of magnitude in [2^-120, 2^120] truncated to float (within 2^-23 of it).
__device__ __forceinline__ float narrow(double x) {
    const uint32_t hi = (uint32_t)__double2hiint(x), lo = (uint32_t)__double2loint(x);
    return __uint_as_float((hi & 0x80000000u) | (__funnelshift_l(lo, hi - 0x38000000u, 3) & 0x7fffffffu));
}
__device__ __forceinline__ bool in_range(double x, double lo, double hi) { return x >= lo && x <= hi; }

__device__ __forceinline__ float rcp_approx(float x) {  // within 2^-23 of 1 / x
    float y;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

// FP32 view of the adjustment's state (ip = <o, o_a>, oa2 = |o_a|^2).  A code's
// value is oa = delta (m + 1/2) exactly, m = code - 2^(bits-1), so a move by one
// code step is accepted (caq_encoder.hpp:93, 108) exactly when
//   up:   g = a (a + 2) - Q (m + 1) - rho > 0
//   down: g = a (a - 2) + Q m - rho > 0
// with a = delta o_j / ip, Q = (1 + rho) 2 delta^2 / oa2, rho = re_eps / ip^2: both
// sides of the reference's comparison divided by ip^2 oa2, their common part
// taken off.  In FP32 g is within `margin` of its value: the factors are within
// 2^-21.3 of theirs (truncation, reciprocal, up to three roundings), the sums add
// three roundings, and 2^-19 (4 |a|max + Q (2^(bits-1) + 1) + |rho|) is over three
// times that for |a| <= 2 (beyond, the margin is infinite); 1e-12 (1 + |rho|)
// covers the rounding of the reference's own FP64 sides.  So a g outside the
// margin has the FP64 comparison's outcome; within it (about one test in 10^5)
// the FP64 comparison itself runs.
//
// init decides once whether the vector stays in float range: each |oa| lies in
// [delta / 2, v_mx], which bounds oa2; an accepted move never lowers ip^2 / oa2,
// so |ip| never falls below 2^-bits of its first value and stays below |o| |oa|.
// Otherwise (or with a NaN) every test runs in FP64 (k* infinite or NaN).
struct AdjView {
    float A2, Q, rho, margin;
    float df2, q1, ref, kv, kh;
    __device__ __forceinline__ void init(double ip, double oa2, double re_eps, double v_mx, double delta, double l2max,
                                         float half) {
        const bool ok = in_range(fabs(ip), 0x1p-80, 0x1p80) && in_range(oa2, 0x1p-100, 0x1p100) &&
                        in_range(v_mx, 0x1p-40, 0x1p40) && in_range(delta, 0x1p-44, 0x1p40) && l2max < 0x1p100 &&
                        (re_eps == 0 || in_range(re_eps, 0x1p-100, 0x1p100));
        const float vm = (float)v_mx, df = (float)delta;
        df2 = 2.0f * df;
        q1 = df2 * df;
        ref = ok ? (float)re_eps : 0.0f;
        kv = ok ? 3.8146973e-6f * vm : __int_as_float(0x7f800000);  // 2^-19 * 2 v_mx, on |A2| = 2 |A|
        kh = 1.9073486e-6f * (half + 1.0f);
        set(ip, oa2);
    }
    __device__ __forceinline__ void set(double ip, double oa2) {
        const float ri = rcp_approx(narrow(ip)), ro = rcp_approx(narrow(oa2));
        A2 = df2 * ri;
        rho = ref * ri * ri;
        Q = fmaf(rho, q1, q1) * ro;
        const float am = fabsf(A2) * kv;  // 2^-19 * 4 |a|max
        margin = am + fmaf(fabsf(Q), kh, fmaf(fabsf(rho), 1.9073496e-6f, 1e-12f));
        if (!(am <= 1.5258789e-5f)) margin = __int_as_float(0x7f800000);  // |a|max > 2
    }
    // g of either direction, -inf where the code is at its end (top = 2^(bits-1) - 1)
    __device__ __forceinline__ void test(float ov, float m, float top, float &gu, float &gd) const {
        const float a2 = A2 * ov, a = 0.5f * a2, p = fmaf(a, a, -rho), w = fmaf(-Q, m, a2);
        gu = m < top ? (p + w) - Q : __int_as_float(0xff800000);
        gd = m > -top - 1.0f ? p - w : __int_as_float(0xff800000);
    }
    __device__ __forceinline__ float best(float ov, float m, float top) const {
        float gu, gd;
        test(ov, m, top, gu, gd);
        return fmaxf(gu, gd);
    }
};

// The reference's comparison (caq_encoder.hpp:93, 108): whether the move to
// (ni, nl) is refused.  A call, so that its FP64 operations are not issued under a
// false predicate on every visit.
__device__ __noinline__ bool refused(double ip, double oa2, double re_eps, double ni, double nl) {
    return __dmul_rn(__dadd_rn(__dmul_rn(ip, ip), re_eps), nl) >= __dmul_rn(__dmul_rn(ni, ni), oa2);
}

constexpr int kEncTableBits = 6;  // codes of at most this many bits keep their values in shared memory
constexpr int kEncWin = 8;       // dimensions a warp visits together
constexpr int kEncThreads = 32;  // one warp a CTA: the last wave fills evenly
constexpr int kEncCtas = 21;     // resident CTAs per SM the register budget is sized for

// Bytes of shared memory per warp: (oa, oa^2) of the codes above the middle (the
// lower half mirrors them), one column per lane.
__host__ __device__ constexpr size_t enc_table_bytes(int bits) {
    return bits >= 1 && bits <= kEncTableBits ? (size_t)(1 << (bits - 1)) * 2 * 32 * 8 : 0;
}

// kN (4 or 8) consecutive dimensions of a vector, or of its codes.  STR = 1: a
// row-major vector (16-byte accesses when `vec`); 32: a vector of a
// warp-interleaved group.
template <int STR, int kN>
__device__ __forceinline__ void load_dims(const float *__restrict__ p, bool vec, float (&x)[kN]) {
    if (STR == 1 && vec) {
#pragma unroll
        for (int k = 0; k < kN; k += 4) {
            const float4 a = *reinterpret_cast<const float4 *>(p + k);
            x[k] = a.x, x[k + 1] = a.y, x[k + 2] = a.z, x[k + 3] = a.w;
        }
    } else {
#pragma unroll
        for (int k = 0; k < kN; ++k) x[k] = p[k * STR];
    }
}
template <int STR, int kN, class CodeT>
__device__ __forceinline__ void load_codes(const CodeT *p, bool vec, int (&x)[kN]) {
    if (STR == 1 && sizeof(CodeT) == 4 && vec) {
#pragma unroll
        for (int k = 0; k < kN; k += 4) {
            const int4 a = *reinterpret_cast<const int4 *>(p + k);
            x[k] = a.x, x[k + 1] = a.y, x[k + 2] = a.z, x[k + 3] = a.w;
        }
    } else {
#pragma unroll
        for (int k = 0; k < kN; ++k) x[k] = (int)p[k * STR];
    }
}

// encode + code_adjustment + encode_and_fac (caq_encoder.hpp:57-247) for one
// vector of D dimensions (a multiple of 32), dimension j at o_[j * STR] (its code
// at code_[j * STR]): STR = 1 for a row-major vector, 32 for a vector of a
// warp-interleaved group, where the 32 lanes of a warp encode 32 vectors and
// every load and store of the warp at dimension j is one contiguous line.
//
// The FP64 pipe bounds it (two lanes per SM and cycle).  With the adjustment as
// the reference writes it, about 190 FP64 operations per dimension, 100,000 x 960
// at 4 bits took 54 ms and 8,191 x 960 9.8 ms; now 5.6 and 1.7 ms, the FP64 pipe
// active 70% of the time with about 23 operations per dimension.  What stays FP64
// is what the codes and factors are made of, the running sums of accepted moves
// and the correction sums:
//   * the comparisons run in FP32 with a bound (AdjView): 54 to 12 ms;
//   * the code values and their squares come from a table;
//   * products that are exact in FP64 (24-bit operands: delta o_j, and oa o_j up to
//     5 bits) are fused into their sums, which rounds the same;
//   * the correction sums of a round accumulate while the round runs, since a
//     dimension's code is final once its window is done;
//   * a warp visits a window of kEncWin dimensions together, each lane at its own
//     next move, so one pass of the FP64 operations serves every lane that still has
//     a move: 3-4 passes per window instead of one or more per dimension (7.7 to
//     5.6 ms).
// Every sum rounds at the same places as the reference's.  kWidth: 0 up to 5 bits
// (table, fused products), 1 for 6 (table), 2 for more.
template <int STR, int kWidth, class CodeT>
__device__ void caq_encode_one(const float *__restrict__ o_, int D, int bits, const float *__restrict__ cent, int rdlmt,
                               float eps, CodeT *code_, float *__restrict__ fac, bool vec, float *win, double *tab) {
    auto code = [&](int j) -> CodeT & { return code_[(int64_t)j * STR]; };
    // Eigen's 16-lane two-accumulator sum (thread_eigen_sum), four dimensions per load
    auto eigen_sum = [&](auto f) {
        float r[32];
#pragma unroll
        for (int l = 0; l < 32; ++l) r[l] = 0.0f;
        for (int j = 0; j < D; j += 32)
#pragma unroll
            for (int h = 0; h < 32; h += 4) {
                float x[4];
                load_dims<STR>(o_ + (int64_t)(j + h) * STR, vec, x);
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    const float t = f(j + h + k, x[k]);
                    r[h + k] = j == 0 ? t : __fadd_rn(r[h + k], t);
                }
            }
#pragma unroll
        for (int l = 0; l < 16; ++l) r[l] = __fadd_rn(r[l], r[16 + l]);
        return tree16(r);
    };
    double v_mx = 0, v_mi = 0, delta = 0, ip = 0, oa2 = 0;
    if (bits > 0) {
        const int cmax = (1 << bits) - 1;
        float mx = o_[0], mn = o_[0];
        const double vec_sum = (double)eigen_sum([&](int, float x) {
            mx = fmaxf(mx, x);
            mn = fminf(mn, x);
            return x;
        });
        const float vmx_f = fmaxf(mx, -mn);
        v_mx = (double)vmx_f;
        v_mi = -v_mx;
        delta = __ddiv_rn(__dsub_rn(v_mx, v_mi), (double)(cmax + 1));
        double ip_o_code = 0;
        uint64_t code_l2 = 0;
        uint32_t code_sum = 0;
        const float vmi_f = (float)v_mi, d_f = (float)delta;
        for (int j = 0; j < D; j += 4) {
            float x[4];
            load_dims<STR>(o_ + (int64_t)j * STR, vec, x);
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                float cf = 0.0f;
                if (delta != 0) cf = fminf(floorf(__fdiv_rn(__fsub_rn(x[k], vmi_f), d_f)), (float)cmax);
                ip_o_code = __dadd_rn(ip_o_code, widen(__fmul_rn(cf, x[k])));
                const int c = (int)cf;
                code(j + k) = (CodeT)c;
                code_l2 += (uint64_t)(c * c);
                code_sum += (uint32_t)c;
            }
        }
        ip = __dadd_rn(__dmul_rn(ip_o_code, delta), __dmul_rn(__dadd_rn(v_mi, __dmul_rn(0.5, delta)), vec_sum));
        const double dd = __dmul_rn(delta, delta);
        oa2 = __dadd_rn(__dmul_rn(dd, (double)code_l2),
                        __dmul_rn(__dadd_rn(dd, __dmul_rn(__dmul_rn(2.0, delta), v_mi)), (double)code_sum));
        const double k3 = __dadd_rn(__dadd_rn(__dmul_rn(__dmul_rn(0.25, delta), delta), __dmul_rn(delta, v_mi)),
                                    __dmul_rn(v_mi, v_mi));
        oa2 = __dadd_rn(oa2, __dmul_rn(k3, (double)D));
        if (rdlmt && oa2 != 0) {
            const double re_eps = __dmul_rn((double)eps, oa2);
            const int half = 1 << (bits - 1);
            const float bias = 8388608.0f + (float)half;
            constexpr bool table = kWidth <= 1;
            // m and its float: code - 2^(bits-1), by the mantissa of 2^23 + code
            auto m_float = [&](int c) { return __int_as_float(0x4b000000 | c) - bias; };
            auto m_int = [](float mf) { return __float_as_int(mf + 12582912.0f) - 0x4b400000; };
            const float top = (float)(half - 1);
            // oa and oa^2 of code half + m; entry i of the table holds those of m = i
            // and, negated, of m = -i - 1
            auto value = [&](int m, double &oa, double &sq) {
                if (table) {
                    const double2 t = *reinterpret_cast<const double2 *>(tab + (m ^ (m >> 31)) * 64);
                    oa = __hiloint2double(__double2hiint(t.x) ^ (m & 0x80000000), __double2loint(t.x));
                    sq = t.y;
                } else {
                    oa = __dadd_rn(__dmul_rn(widen((float)(m + half) + 0.5f), delta), v_mi);
                    sq = __dmul_rn(oa, oa);
                }
            };
            if (table)
                for (int i = 0; i < half; ++i) {
                    const double t = __dadd_rn(__dmul_rn((double)(half + i) + 0.5, delta), v_mi);
                    *reinterpret_cast<double2 *>(tab + i * 64) = make_double2(t, __dmul_rn(t, t));
                }
            AdjView st;
            st.init(ip, oa2, re_eps, v_mx, delta, (double)vmx_f * vmx_f * D, (float)half);
            for (int adj = 1, round = 1; adj; round++) {
                adj = 0;
                const bool last = round >= rdlmt;  // the reference leaves before this round's correction
                double ci = 0, co = 0;
                float xn[kEncWin];
                int cn[kEncWin];
                load_dims<STR>(o_, vec, xn);
                load_codes<STR>(code_, vec, cn);
#pragma unroll 1
                for (int j0 = 0; j0 < D; j0 += kEncWin) {
                    float x[kEncWin];
                    int c0[kEncWin];
#pragma unroll
                    for (int k = 0; k < kEncWin; ++k) {
                        x[k] = xn[k];
                        c0[k] = cn[k];
                        win[k * 64] = x[k];
                        win[k * 64 + 32] = m_float(c0[k]);
                    }
                    if (j0 + kEncWin < D) {  // the next window, in flight while this one is visited
                        load_dims<STR>(o_ + (int64_t)(j0 + kEncWin) * STR, vec, xn);
                        load_codes<STR>(code_ + (int64_t)(j0 + kEncWin) * STR, vec, cn);
                    }
                    // one code step of one dimension per trip: each lane takes its own next
                    // dimension whose move is not surely refused, so the FP64 operations of a
                    // trip serve every lane that still has one
                    int k0 = 0, tj = -1;
                    double tmp = 0;  // of dimension tj: oa2 less its oa^2, fixed while its steps last
                    for (;;) {
                        uint32_t cand = 0;
#pragma unroll
                        for (int k = 0; k < kEncWin; ++k) cand |= (uint32_t)(!(st.best(x[k], win[k * 64 + 32], top) < -st.margin)) << k;
                        cand &= ~0u << k0;
                        if (!cand) break;
                        const int j = __ffs(cand) - 1;
                        const float ov = win[j * 64], mf = win[j * 64 + 32];
                        float gu, gd;
                        st.test(ov, mf, top, gu, gd);
                        int m = m_int(mf);
                        const double od = widen(ov);
                        double oa, sq, sqn;
                        value(m, oa, sq);
                        if (j != tj) tmp = __dsub_rn(oa2, sq);
                        tj = j;
                        const bool up = gu > st.margin;
                        if (up || (gu < -st.margin && gd > st.margin)) {  // surely accepted; tested again next trip
                            value(up ? m + 1 : m - 1, oa, sqn);
                            ip = fma(up ? delta : -delta, od, ip);
                            oa2 = __dadd_rn(tmp, sqn);
                            win[j * 64 + 32] = up ? mf + 1.0f : mf - 1.0f;
                            st.set(ip, oa2);
                            k0 = j;
                            continue;
                        }
                        // the reference's loops as written: upward steps until one is refused, then downward
                        for (int d = 1; d >= -1; d -= 2)
                            while (d > 0 ? m < half - 1 : m > -half) {
                                value(m + d, oa, sqn);
                                const double nl = __dadd_rn(tmp, sqn), ni = fma(d > 0 ? delta : -delta, od, ip);
                                if (refused(ip, oa2, re_eps, ni, nl)) break;
                                m += d;
                                ip = ni;
                                oa2 = nl;
                            }
                        win[j * 64 + 32] = (float)m;
                        st.set(ip, oa2);
                        k0 = j + 1;
                    }
#pragma unroll
                    for (int k = 0; k < kEncWin; ++k) {
                        const float mf = win[k * 64 + 32];
                        const int m = m_int(mf);
                        if (m + half != c0[k]) {
                            code(j0 + k) = (CodeT)(m + half);
                            adj = 1;
                        }
                        if (!last) {  // the correction sums over the round's final codes
                            double oa, sq;
                            value(m, oa, sq);
                            const double od = widen(x[k]);
                            ci = kWidth == 0 ? fma(oa, od, ci) : __dadd_rn(ci, __dmul_rn(oa, od));
                            co = __dadd_rn(co, sq);
                        }
                    }
                }
                if (last) break;
                oa2 = co;
                ip = ci;
                st.set(ip, oa2);
            }
        }
    } else {
        for (int j = 0; j < D; ++j) code(j) = 0;
    }
    const double o_l2sqr = (double)eigen_sum([&](int, float x) { return __fmul_rn(x, x); });
    const double o_l2norm = __dsqrt_rn(o_l2sqr);
    double rescale = ip != 0 ? __ddiv_rn(o_l2sqr, ip) : 0.0;
    const double err = __dmul_rn(
        __dmul_rn(o_l2sqr, (double)1.9f),
        __dsqrt_rn(__ddiv_rn(__dsub_rn(__ddiv_rn(__dmul_rn(o_l2sqr, oa2), __dmul_rn(ip, ip)), 1.0), (double)(D - 1))));
    if (v_mx != 0) {
        const double s = __ddiv_rn(1.0, v_mx);
        delta = __dmul_rn(delta, s);
        rescale = __dmul_rn(rescale, v_mx);
        v_mi = __dmul_rn(v_mi, s);
    }
    float ipc = 0.0f;
    if (bits > 1 && cent) {
        const float df = (float)delta, vf = (float)v_mi;
        ipc = thread_eigen_sum(
            D, [&](int i) { return __fmul_rn(cent[i], __fadd_rn(__fmul_rn((float)(int)code(i), df), vf)); });
    }
    fac[0] = (float)o_l2norm;
    fac[1] = ipc;
    fac[2] = (float)rescale;
    fac[3] = (float)err;
}

// Shared memory of an encoding warp: its window (kEncWin dimensions and their
// codes), then its table.
__device__ __forceinline__ float *enc_window() {
    extern __shared__ __align__(16) double enc_smem[];
    return reinterpret_cast<float *>(enc_smem) + (threadIdx.x & 31);
}
__device__ __forceinline__ double *enc_table() {
    extern __shared__ __align__(16) double enc_smem[];
    return enc_smem + kEncWin * 32 + 2 * (threadIdx.x & 31);
}

template <int kWidth>
__global__ void __launch_bounds__(kEncThreads, kEncCtas) k_caq_encode(const float *__restrict__ resid, int64_t n, int D, int bits,
                                                            const float *__restrict__ cent, int rdlmt, float eps,
                                                            int32_t *codes, float *__restrict__ facs, int vec) {
    const int64_t v = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (v >= n) return;
    caq_encode_one<1, kWidth>(resid + v * D, D, bits, cent, rdlmt, eps, codes + v * D, facs + v * 4, vec != 0,
                              enc_window(), enc_table());
}

// Shared memory of a CTA (one warp; at most 18 KB).
size_t enc_smem_bytes(int bits) { return kEncWin * 32 * 8 + enc_table_bytes(bits); }

// Calls f with the kernel's kWidth for codes of `bits` bits.
template <class F>
void by_width(int bits, F f) {
    if (bits <= 5) f(std::integral_constant<int, 0>());
    else if (bits <= kEncTableBits) f(std::integral_constant<int, 1>());
    else f(std::integral_constant<int, 2>());
}

}  // namespace

void run_caq_encode(const float *resid, int64_t n, int64_t dim, int bits, const float *cent, int rdlmt, float eps,
                    int32_t *codes, float *facs, int mem, cudaStream_t st) {
    if (n == 0) return;
    const float *dr = resid, *dc = cent;
    int32_t *dcodes = codes;
    float *dfacs = facs;
    void *buf = nullptr;
    if (mem == SAQG_MEM_HOST) {
        const size_t br = 4 * (size_t)n * dim, bc = cent ? 4 * (size_t)dim : 0, bo = 4 * (size_t)n * dim,
                     bf = 16 * (size_t)n;
        SAQG_CUDA_TRY(cudaMalloc(&buf, br + bc + bo + bf + 64));
        char *p = (char *)buf;
        SAQG_CUDA_TRY(cudaMemcpyAsync(p, resid, br, cudaMemcpyHostToDevice, st));
        dr = (const float *)p;
        if (cent) {
            SAQG_CUDA_TRY(cudaMemcpyAsync(p + br, cent, bc, cudaMemcpyHostToDevice, st));
            dc = (const float *)(p + br);
        }
        dcodes = (int32_t *)(p + br + bc);
        dfacs = (float *)(p + br + bc + bo);
    }
    // rows of a multiple of 32 floats: 16-byte accesses need only aligned bases
    const int vec = ((uintptr_t)dr & 15) == 0 && ((uintptr_t)dcodes & 15) == 0;
    by_width(bits, [&](auto w) {
        k_caq_encode<decltype(w)::value>
            <<<(unsigned)((n + kEncThreads - 1) / kEncThreads), kEncThreads, enc_smem_bytes(bits), st>>>(
                dr, n, (int)dim, bits, dc, rdlmt, eps, dcodes, dfacs, vec);
    });
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) {
        if (buf) cudaFree(buf);
        throw Error{SAQG_ERR_CUDA, std::string("k_caq_encode launch failed: ") + cudaGetErrorString(e)};
    }
    count_launch(1);
    if (mem == SAQG_MEM_HOST) {
        SAQG_CUDA_TRY(cudaMemcpyAsync(codes, dcodes, 4 * (size_t)n * dim, cudaMemcpyDeviceToHost, st));
        SAQG_CUDA_TRY(cudaMemcpyAsync(facs, dfacs, 16 * (size_t)n, cudaMemcpyDeviceToHost, st));
        SAQG_CUDA_TRY(cudaStreamSynchronize(st));
        cudaFree(buf);
    }
}

// ---------------------------------------------------------------- construct
namespace {

// SaqDataMaker::compute_variance (saq_data.hpp:95-100): column means by Eigen's
// packetwise reduction (PartialReduxEvaluator.h:102-128), variances of the
// rowwise() difference by a sequential column sum (that expression has no
// packet access); both divided by the row count.
//
// The order of the sums leaves one chain of n / 4 and one of n FP32 adds per
// column, so a column belongs to one thread and its time is the adds' latency if
// the rows arrive in time.  A CTA has 16 columns (64 bytes of a row; more CTAs than
// with 32 share the loading): warp 1 keeps 14 stages of 64 rows in flight by
// asynchronous copies while warp 0 adds one up.  Row 0 is taken apart, so that the
// groups of four rows of the mean start at a stage.  250,007 x 1,024: 36 ms with a
// thread per column loading its own rows (each group waited for memory), 3.4 with
// one warp copying and adding, 2.0 now.
constexpr int kVarCols = 16, kVarRows = 64, kVarStages = 16, kVarThreads = 64;
__global__ void __launch_bounds__(kVarThreads) k_colwise_var(const float *__restrict__ x, int64_t n, int D, int vec,
                                                             float *__restrict__ var) {
    extern __shared__ __align__(16) float var_ring[];  // [stage][row][kVarCols]
    const int lane = threadIdx.x & 31, c0 = blockIdx.x * kVarCols, col = lane & (kVarCols - 1);
    const bool copier = threadIdx.x >= 32;
    const int64_t rest = n - 1, nst = (rest + kVarRows - 1) / kVarRows;  // rows 1 .. n - 1 in stages
    auto issue = [&](int64_t st) {
        if (st < nst) {
            float *dst = var_ring + (int)(st & (kVarStages - 1)) * (kVarRows * kVarCols);
            const int rows = (int)min((int64_t)kVarRows, rest - st * kVarRows);
            const float *src = x + (1 + st * kVarRows) * D + c0;
            if (vec) {
                const int k = lane % (kVarCols / 4) * 4;
#pragma unroll
                for (int r = lane / (kVarCols / 4); r < kVarRows; r += 128 / kVarCols)
                    if (r < rows)
                        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(
                                         (unsigned)__cvta_generic_to_shared(dst + r * kVarCols + k)),
                                     "l"(src + (int64_t)r * D + k)
                                     : "memory");
            } else {
                for (int e = lane; e < rows * kVarCols; e += 32) {
                    const int r = e / kVarCols, k = e % kVarCols;
                    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(
                                     (unsigned)__cvta_generic_to_shared(dst + r * kVarCols + k)),
                                 "l"(src + (int64_t)r * D + k)
                                 : "memory");
                }
            }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    // f(rows of the stage, its column) of warp 0: the stages in order.  While it adds
    // stage st up, warp 1 refills the stage read before it and waits for the next.
    auto stream = [&](auto f) {
        if (copier) {
            for (int st = 0; st < kVarStages - 1; ++st) issue(st);
            asm volatile("cp.async.wait_group %0;" ::"n"(kVarStages - 2) : "memory");
        }
        __syncthreads();
        for (int64_t st = 0; st < nst; ++st) {
            if (copier) {
                issue(st + kVarStages - 1);
                asm volatile("cp.async.wait_group %0;" ::"n"(kVarStages - 2) : "memory");
            } else {
                f((int)min((int64_t)kVarRows, rest - st * kVarRows),
                  var_ring + (int)(st & (kVarStages - 1)) * (kVarRows * kVarCols) + col);
            }
            __syncthreads();
        }
    };
    const float first = x[c0 + col];
    float p = first;
    stream([&](int rows, const float *s) {
        if (rows == kVarRows) {
#pragma unroll
            for (int r = 0; r < kVarRows; r += 4) {
                const float a = __fadd_rn(s[r * kVarCols], s[(r + 1) * kVarCols]);
                const float b = __fadd_rn(s[(r + 2) * kVarCols], s[(r + 3) * kVarCols]);
                p = __fadd_rn(p, __fadd_rn(a, b));
            }
        } else {  // the last stage: groups of four while they fit, then single rows
            int r = 0;
            for (; r + 4 <= rows; r += 4) {
                const float a = __fadd_rn(s[r * kVarCols], s[(r + 1) * kVarCols]);
                const float b = __fadd_rn(s[(r + 2) * kVarCols], s[(r + 3) * kVarCols]);
                p = __fadd_rn(p, __fadd_rn(a, b));
            }
            for (; r < rows; ++r) p = __fadd_rn(p, s[r * kVarCols]);
        }
    });
    const float mean = __fdiv_rn(p, (float)n);
    const float d0 = __fsub_rn(first, mean);
    float v = __fmul_rn(d0, d0);
    stream([&](int rows, const float *s) {
        if (rows == kVarRows) {
#pragma unroll
            for (int r = 0; r < kVarRows; ++r) {
                const float d = __fsub_rn(s[r * kVarCols], mean);
                v = __fadd_rn(v, __fmul_rn(d, d));
            }
        } else {
            for (int r = 0; r < rows; ++r) {
                const float d = __fsub_rn(s[r * kVarCols], mean);
                v = __fadd_rn(v, __fmul_rn(d, d));
            }
        }
    });
    if (threadIdx.x < kVarCols) var[c0 + col] = __fdiv_rn(v, (float)n);
}

// Rotated residuals of one segment: out[v][i] = (x_v . P[:, i]) - rc[cid_v][i],
// where x_v is rows[v]'s slice [off, off + dim) of the data, zero-padded past D
// (rotate_tile; rc null: no centroid taken off).  `vec`: the data are 16-byte
// aligned (rows and slices start at multiples of 64 floats).  Output
// warp-interleaved ([v / 32][dim][v % 32], padded to whole groups) or row-major.
// 100,000 x 960 (184 GFLOP): 6.8 ms with 64 x 64
// tiles of scalar FMAs, 3.6 ms now (51 TFLOP/s; FMA pipe 70%, shared memory 73%).
__global__ void __launch_bounds__(kRotThreads, 2) k_rotate(const float *__restrict__ data, int D,
                                                           const int64_t *__restrict__ rows, int64_t nv, int off,
                                                           int dim, const float *__restrict__ P,
                                                           const float *__restrict__ rc,
                                                           const int32_t *__restrict__ cid, float *__restrict__ out,
                                                           int interleaved, int vec) {
    rotate_tile(
        dim, P, (int64_t)blockIdx.y * kRotM, blockIdx.x * kRotN,
        [&](int64_t v, int j) {
            float4 r = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            if (v < nv && off + j < D) {  // D is a multiple of 64: four inputs at once are in or out
                const float *x = data + rows[v] * D + off + j;
                if (vec) r = *reinterpret_cast<const float4 *>(x);
                else r = make_float4(x[0], x[1], x[2], x[3]);
            }
            return r;
        },
        [&](int64_t v, int o, float (&r)[8][4]) {
            if (v >= nv) return;
            if (rc)
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    const float4 c = *reinterpret_cast<const float4 *>(rc + (int64_t)cid[min(v + i, nv - 1)] * dim + o);
                    r[i][0] = __fsub_rn(r[i][0], c.x);
                    r[i][1] = __fsub_rn(r[i][1], c.y);
                    r[i][2] = __fsub_rn(r[i][2], c.z);
                    r[i][3] = __fsub_rn(r[i][3], c.w);
                }
            if (interleaved) {
#pragma unroll
                for (int b = 0; b < 4; ++b) {
                    float4 *d = reinterpret_cast<float4 *>(out + (v >> 5) * (int64_t)dim * 32 + (int64_t)(o + b) * 32 + (v & 31));
                    d[0] = make_float4(r[0][b], r[1][b], r[2][b], r[3][b]);
                    d[1] = make_float4(r[4][b], r[5][b], r[6][b], r[7][b]);
                }
            } else {
#pragma unroll
                for (int i = 0; i < 8; ++i)
                    if (v + i < nv)
                        *reinterpret_cast<float4 *>(out + (v + i) * dim + o) = make_float4(r[i][0], r[i][1], r[i][2], r[i][3]);
            }
        });
}

// Un-rotated centroid slice (zero-padded) of cluster c, as the reference passes
// it to encode_and_fac for ip_cent_oa (quantizer.hpp:64, saq_quantizer.hpp:51-54).
__global__ void k_centroid_slices(const float *__restrict__ cent, int64_t K, int D, int off, int dim,
                                  float *__restrict__ out) {
    const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= K * dim) return;
    const int64_t c = t / dim;
    const int i = (int)(t % dim);
    out[t] = off + i < D ? cent[c * D + off + i] : 0.0f;
}

// CAQEncoder::encode_and_fac for the vectors of a chunk, each with its own
// cluster's un-rotated centroid slice.  Residuals and codes are warp-interleaved
// ([v / 32][dim][v % 32]): lane l of a warp encodes vector 32 w + l, and each
// step of the 32 sequential FP64 chains reads one coalesced line.
__device__ __forceinline__ int64_t inter_at(int64_t v, int D) { return (v >> 5) * (int64_t)D * 32 + (v & 31); }

template <int kWidth>
__global__ void __launch_bounds__(kEncThreads, kEncCtas) k_caq_encode_clustered(const float *__restrict__ resid, int64_t n, int D,
                                                                      int bits, const float *__restrict__ cslices,
                                                                      const int32_t *__restrict__ cid, int rdlmt,
                                                                      float eps, uint16_t *codes,
                                                                      float *__restrict__ facs) {
    const int64_t v = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (v >= n) return;
    caq_encode_one<32, kWidth>(resid + inter_at(v, D), D, bits, cslices + (int64_t)cid[v] * D, rdlmt, eps,
                       codes + inter_at(v, D), facs + v * 4, false, enc_window(), enc_table());
}

// CodeHelper<B>::compacted_code8/16 (code_helper.hpp) for one vector (code of
// dimension d at v[d * STR]).
template <int STR>
__device__ void pack_bits8_dev(const uint16_t *__restrict__ v, int D, int bits, int shift, int mask,
                               uint8_t *__restrict__ y) {
    auto val = [&](int d) { return (uint32_t)((v[(int64_t)d * STR] >> shift) & mask); };
    switch (bits) {
    case 1:
        for (int i = 0; i < D / 8; ++i) {
            uint32_t b = 0;
            for (int j = 0; j < 8; ++j) b |= (val(i * 8 + j) & 1u) << j;
            y[i] = (uint8_t)b;
        }
        break;
    case 2:
    case 3:
        for (int g = 0; g < D / 64; ++g) {
            uint8_t *b = y + g * (bits == 2 ? 16 : 24);
            const int d0 = g * 64;
            for (int r = 0; r < 16; ++r)
                b[r] = (uint8_t)((val(d0 + r) & 3u) | ((val(d0 + 16 + r) & 3u) << 2) | ((val(d0 + 32 + r) & 3u) << 4) |
                                 ((val(d0 + 48 + r) & 3u) << 6));
            if (bits == 3)
                for (int k = 0; k < 8; ++k) {
                    uint32_t t = 0;
                    for (int m = 0; m < 8; ++m) t |= ((val(d0 + 8 * m + k) >> 2) & 1u) << m;
                    b[16 + k] = (uint8_t)t;
                }
        }
        break;
    case 4:
        for (int g = 0; g < D / 32; ++g)
            for (int r = 0; r < 16; ++r)
                y[g * 16 + r] = (uint8_t)((val(g * 32 + r) & 15u) | ((val(g * 32 + 16 + r) & 15u) << 4));
        break;
    case 6:
    case 7:
        for (int g = 0; g < D / 64; ++g) {
            uint8_t *b = y + g * (bits == 6 ? 48 : 56);
            const int d0 = g * 64;
            for (int r = 0; r < 16; ++r) {
                b[r] = (uint8_t)((val(d0 + r) & 63u) | (((val(d0 + 32 + r) >> 4) & 3u) << 6));
                b[16 + r] = (uint8_t)((val(d0 + 16 + r) & 63u) | (((val(d0 + 48 + r) >> 4) & 3u) << 6));
                b[32 + r] = (uint8_t)((val(d0 + 32 + r) & 15u) | ((val(d0 + 48 + r) & 15u) << 4));
            }
            if (bits == 7)
                for (int k = 0; k < 8; ++k) {
                    uint32_t t = 0;
                    for (int m = 0; m < 8; ++m) t |= ((val(d0 + 8 * m + k) >> 6) & 1u) << m;
                    b[48 + k] = (uint8_t)t;
                }
        }
        break;
    case 8:
        for (int d = 0; d < D; ++d) y[d] = (uint8_t)val(d);
        break;
    default:
        break;
    }
}

template <int STR>
__device__ void pack_excode_dev(const uint16_t *__restrict__ code, int D, int exb, uint8_t *__restrict__ y) {
    const int lowmask = (1 << exb) - 1;
    if (exb > 8) {  // compacted_code16: low bytes, then the remaining bits in their own layout
        for (int d = 0; d < D; ++d) y[d] = (uint8_t)(code[(int64_t)d * STR] & lowmask & 0xFF);
        const int hb = exb - 8;
        if (hb == 5) {
            pack_bits8_dev<STR>(code, D, 4, 9, 15, y + D);
            pack_bits8_dev<STR>(code, D, 1, 8, 1, y + D + D / 2);
        } else {
            pack_bits8_dev<STR>(code, D, hb, 8, (1 << hb) - 1, y + D);
        }
    } else if (exb == 5) {  // CodeHelper<5>: 4-bit layout of code>>1, then the low bit
        pack_bits8_dev<STR>(code, D, 4, 1, 15, y);
        pack_bits8_dev<STR>(code, D, 1, 0, 1, y + D / 2);
    } else {
        pack_bits8_dev<STR>(code, D, exb, 0, lowmask, y);
    }
}

// ClusterPacker::store_and_pack + finalize_and_store (cluster_packer.hpp:59-116)
// into the device layout (saqg_internal.h): one thread per vector.
__global__ void k_pack(const uint16_t *__restrict__ codes, const float *__restrict__ facs, int64_t n, int64_t vbase,
                       const int32_t *__restrict__ cid, const int64_t *__restrict__ blk_off,
                       const int64_t *__restrict__ vec_off, SegDev g) {
    const int64_t v = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (v >= n) return;
    const int64_t gv = vbase + v;
    const int c = cid[v];
    const int64_t pos = gv - vec_off[c];
    const int64_t gb = blk_off[c] + pos / 32;
    const int lane = (int)(pos % 32);
    const float *f = facs + v * 4;
    g.onorm[gb * 32 + lane] = f[0];
    if (g.bits == 0) return;
    g.ipcent[gb * 32 + lane] = f[1];
    g.exfac[gv] = make_float2(f[2], f[3]);
    const uint16_t *code = codes + inter_at(v, g.dim);  // warp-interleaved codes: dimension d at code[32 d]
    const int sb = 1 << (g.bits - 1);
    uint8_t *cb = reinterpret_cast<uint8_t *>(g.codes) + (size_t)gb * (g.dim / 8) * 32;
    for (int i = 0; i < g.dim / 8; ++i) {
        uint32_t byte = 0;
        for (int k = 0; k < 8; ++k) byte |= (code[(int64_t)(i * 8 + k) * 32] & sb) ? (0x80u >> k) : 0u;
        cb[((size_t)(i / 8) * 32 + lane) * 8 + (i % 8)] = (uint8_t)byte;
    }
    if (g.bits > 1) pack_excode_dev<32>(code, g.dim, g.bits - 1, g.lcode + (size_t)gv * g.lstride);
}

// Random orthogonal matrix (modified Gram-Schmidt on a Gaussian matrix, FP64,
// seeded) -- the stand-in for Rotator::orthogonalize (rotator.hpp:30-35) when
// the caller gives no rotation.  Returned row-major as P (rows orthonormal).
std::vector<float> random_orthogonal(int64_t d, uint64_t seed) {
    uint64_t st = seed * 0x9E3779B97F4A7C15ull + 0x1234567ull;
    auto next = [&]() {
        st += 0x9E3779B97F4A7C15ull;
        uint64_t z = st;
        z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
        z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
        return z ^ (z >> 31);
    };
    auto unif = [&]() { return ((next() >> 11) + 0.5) * (1.0 / 9007199254740992.0); };
    std::vector<double> A(d * d);
    for (int64_t i = 0; i < d * d; i += 2) {
        const double u1 = unif(), u2 = unif();
        const double r = std::sqrt(-2.0 * std::log(u1));
        A[i] = r * std::cos(6.283185307179586 * u2);
        if (i + 1 < d * d) A[i + 1] = r * std::sin(6.283185307179586 * u2);
    }
    for (int64_t i = 0; i < d; ++i) {  // rows of A become orthonormal
        double *ri = &A[i * d];
        for (int pass = 0; pass < 2; ++pass)
            for (int64_t k = 0; k < i; ++k) {
                const double *rk = &A[k * d];
                double dot = 0;
                for (int64_t t = 0; t < d; ++t) dot += ri[t] * rk[t];
                for (int64_t t = 0; t < d; ++t) ri[t] -= dot * rk[t];
            }
        double nrm = 0;
        for (int64_t t = 0; t < d; ++t) nrm += ri[t] * ri[t];
        nrm = 1.0 / std::sqrt(nrm);
        for (int64_t t = 0; t < d; ++t) ri[t] *= nrm;
    }
    return std::vector<float>(A.begin(), A.end());
}

void launch_check(const char *what) {
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) throw Error{SAQG_ERR_CUDA, std::string(what) + " launch failed: " + cudaGetErrorString(e)};
    count_launch(1);
}

int encoder_sms() {
    int dev = 0, sms = 0;
    SAQG_CUDA_TRY(cudaGetDevice(&dev));
    SAQG_CUDA_TRY(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    return std::max(1, sms);
}

struct DevBuf {
    void *p = nullptr;
    explicit DevBuf(size_t bytes) {
        cudaError_t e = cudaMalloc(&p, bytes ? bytes : 16);
        if (e != cudaSuccess) throw Error{SAQG_ERR_NOMEM, std::string("cudaMalloc failed: ") + cudaGetErrorString(e)};
    }
    ~DevBuf() {
        if (p) cudaFree(p);
    }
    template <class T>
    T *as() const {
        return static_cast<T *>(p);
    }
};

}  // namespace

// Vectors that the construction's encoder holds at once at this width: kEncCtas warps an
// SM, fewer where the table of code values takes more shared memory (12 at 6 bits).
int64_t encoder_vectors(int bits) {
    int per_sm = 0;
    by_width(bits, [&](auto w) {
        SAQG_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_caq_encode_clustered<decltype(w)::value>,
                                                                    kEncThreads, enc_smem_bytes(bits)));
    });
    return (int64_t)encoder_sms() * std::max(1, per_sm) * 32;
}

// Vectors of a chunk of the construction of n vectors: equal chunks of whole 32-vector
// groups (residuals and codes are warp-interleaved), each no more than the encoder holds
// at once, since a few warps left for a second wave would take as long as a full one
// (125,000 x 512 at 6 bits: 9.2 ms with chunks for 21 warps an SM, 8.4 for its 12).
int64_t encode_chunk(int64_t n, int bits, int64_t maxd) {
    const int64_t at_once =
        std::max<int64_t>(32, std::min<int64_t>((int64_t)(1u << 30) / (8 * maxd), encoder_vectors(bits)) / 32 * 32);
    const int64_t nchunk = std::max<int64_t>(1, (n + at_once - 1) / at_once);
    return std::max<int64_t>(32, ((n + nchunk - 1) / nchunk + 31) / 32 * 32);
}

// IVF::construct (index/ivf.hpp:130-184): group by cluster, plan, then per
// segment rotate / encode / pack on the GPU, in chunks of vectors.
Index *construct_index(const float *data, int64_t n, int64_t dim, const float *centroids, int64_t k,
                       const uint32_t *cids, const saqg_quantize_config &cfg, const float *variance,
                       const float *rotations, uint64_t seed, int data_mem) {
    SAQG_REQUIRE(dim % 64 == 0, "dimension must be a multiple of 64 (the reference's load requires it)");
    SAQG_REQUIRE(cfg.avg_bits >= 0 && cfg.avg_bits <= kMaxBits, "avg_bits out of range");
    auto I = std::make_unique<Index>();
    cudaGetDevice(&I->device);
    I->N = n;
    I->D = dim;
    I->K = k;
    // raw config structs as the reference writes them (config.h:12-27)
    uint8_t s20[20] = {0};
    {
        int32_t qt = 0, rd = cfg.caq_adj_rd_lmt, ori = 0;
        std::memcpy(s20, &qt, 4);
        s20[4] = (uint8_t)(cfg.random_rotation != 0);
        s20[5] = 1;
        std::memcpy(s20 + 8, &rd, 4);
        std::memcpy(s20 + 12, &cfg.caq_adj_eps, 4);
        std::memcpy(s20 + 16, &ori, 4);
        int32_t eq = cfg.seg_eqseg;
        std::memcpy(I->qcfg_raw, &cfg.avg_bits, 4);
        std::memcpy(I->qcfg_raw + 4, &eq, 4);
        I->qcfg_raw[8] = (uint8_t)(cfg.enable_segmentation != 0);
        I->qcfg_raw[9] = (uint8_t)(cfg.use_compact_layout != 0);
        std::memcpy(I->qcfg_raw + 12, s20, 20);
    }
    // data on the device
    const float *ddata = data;
    std::unique_ptr<DevBuf> data_buf;
    if (data_mem == SAQG_MEM_HOST) {
        data_buf = std::make_unique<DevBuf>(4 * (size_t)n * dim);
        SAQG_CUDA_TRY(cudaMemcpy(data_buf->p, data, 4 * (size_t)n * dim, cudaMemcpyHostToDevice));
        ddata = data_buf->as<float>();
    }
    // variance
    // variance and the segment plan (the planner runs on the device)
    I->var.resize(dim);
    std::vector<std::pair<int64_t, int64_t>> plan;
    if (variance) {
        std::memcpy(I->var.data(), variance, 4 * dim);
        plan = make_plan_gpu(variance, dim, cfg.avg_bits, cfg.enable_segmentation != 0, cfg.seg_eqseg, false, 0);
    } else {
        DevBuf dv(4 * dim);
        constexpr int ring = 4 * kVarStages * kVarRows * kVarCols;
        SAQG_CUDA_TRY(cudaFuncSetAttribute(k_colwise_var, cudaFuncAttributeMaxDynamicSharedMemorySize, ring));
        k_colwise_var<<<(unsigned)(dim / kVarCols), kVarThreads, ring>>>(ddata, n, (int)dim, ((uintptr_t)ddata & 15) == 0,
                                                               dv.as<float>());
        launch_check("k_colwise_var");
        plan = make_plan_gpu(dv.as<float>(), dim, cfg.avg_bits, cfg.enable_segmentation != 0, cfg.seg_eqseg, true, 0);
        SAQG_CUDA_TRY(cudaMemcpy(I->var.data(), dv.p, 4 * dim, cudaMemcpyDeviceToHost));
    }
    SAQG_REQUIRE(!plan.empty() && plan.size() <= (size_t)kMaxSeg, "planner produced an unsupported plan");
    int64_t roff = 0;
    for (auto &pr : plan) {
        Index::SegHost sg;
        sg.dim = pr.first;
        sg.bits = pr.second;
        std::memcpy(sg.cfg_raw, s20, 20);
        sg.rotated = cfg.random_rotation != 0;
        if (sg.rotated) {
            if (rotations) sg.P.assign(rotations + roff, rotations + roff + sg.dim * sg.dim);
            else sg.P = random_orthogonal(sg.dim, seed + (uint64_t)I->segs.size());
        }
        roff += sg.dim * sg.dim;
        I->segs.push_back(std::move(sg));
    }
    const size_t S = I->segs.size();
    I->compact = S == 1 || cfg.use_compact_layout;
    // group by cluster: ids ascending within each cluster (ivf.hpp:149-157)
    I->sizes.assign(k, 0);
    for (int64_t i = 0; i < n; ++i) {
        SAQG_REQUIRE(cids[i] < (uint64_t)k, "cluster id out of range");
        I->sizes[cids[i]]++;
    }
    I->blk_off.assign(k + 1, 0);
    I->vec_off.assign(k + 1, 0);
    for (int64_t c = 0; c < k; ++c) {
        I->blk_off[c + 1] = I->blk_off[c] + (I->sizes[c] + kBlock - 1) / kBlock;
        I->vec_off[c + 1] = I->vec_off[c] + I->sizes[c];
    }
    const int64_t NB = I->blk_off[k];
    I->total_blocks = NB;
    std::vector<int64_t> rows(n), fill(I->vec_off.begin(), I->vec_off.end() - 1);
    std::vector<int32_t> cid_sorted(n);
    std::vector<uint32_t> ids(n);
    for (int64_t i = 0; i < n; ++i) {
        const int64_t p = fill[cids[i]]++;
        rows[p] = i;
        cid_sorted[p] = (int32_t)cids[i];
        ids[p] = (uint32_t)i;
    }
    // device index arrays
    Index &X = *I;
    DevIndexView &v = X.view;
    float *dcent = (float *)X.dalloc(4 * k * dim);
    X.upload(dcent, centroids, 4 * k * dim);
    v.centroids = dcent;
    {
        float *dvar = (float *)X.dalloc(4 * dim);
        X.upload(dvar, X.var.data(), 4 * dim);
        v.var = dvar;
    }
    uint32_t *dids = (uint32_t *)X.dalloc(4 * n);
    X.upload(dids, ids.data(), 4 * n);
    v.ids = dids;
    int64_t *dbo = (int64_t *)X.dalloc(8 * (k + 1));
    X.upload(dbo, X.blk_off.data(), 8 * (k + 1));
    v.blk_off = dbo;
    int64_t *dvo = (int64_t *)X.dalloc(8 * (k + 1));
    X.upload(dvo, X.vec_off.data(), 8 * (k + 1));
    v.vec_off = dvo;
    DevBuf drows(8 * n), dcid(4 * n);
    SAQG_CUDA_TRY(cudaMemcpy(drows.p, rows.data(), 8 * n, cudaMemcpyHostToDevice));
    SAQG_CUDA_TRY(cudaMemcpy(dcid.p, cid_sorted.data(), 4 * n, cudaMemcpyHostToDevice));
    DevBuf didx(8 * k), dkc(4 * k);
    {
        std::vector<int64_t> ii(k);
        std::vector<int32_t> kc(k);
        for (int64_t c = 0; c < k; ++c) {
            ii[c] = c;
            kc[c] = (int32_t)c;
        }
        SAQG_CUDA_TRY(cudaMemcpy(didx.p, ii.data(), 8 * k, cudaMemcpyHostToDevice));
        SAQG_CUDA_TRY(cudaMemcpy(dkc.p, kc.data(), 4 * k, cudaMemcpyHostToDevice));
    }
    int64_t maxd = 0;
    for (auto &sg : X.segs) maxd = std::max(maxd, sg.dim);
    int64_t most = 0;
    for (auto &sg : X.segs) most = std::max(most, encode_chunk(n, (int)sg.bits, maxd));
    const int64_t chunk_pad = (std::min(most, n) + 31) / 32 * 32;
    DevBuf resid(4 * (size_t)chunk_pad * maxd), codes(2 * (size_t)chunk_pad * maxd), facs(16 * (size_t)chunk_pad);
    DevBuf cslice(4 * (size_t)k * maxd);
    int off = 0;
    for (size_t s = 0; s < S; ++s) {
        SegDev &g = v.seg[s];
        const int64_t d = X.segs[s].dim;
        g.dim = (int)d;
        g.bits = (int)X.segs[s].bits;
        g.pv = g.bits ? (int)(d * (g.bits - 1) / 8) : 0;
        g.lstride = (g.pv + 15) / 16 * 16;
        float *dP = nullptr;
        if (X.segs[s].rotated) {
            dP = (float *)X.dalloc(4 * d * d);
            X.upload(dP, X.segs[s].P.data(), 4 * d * d);
        }
        g.P = dP;
        g.codes = (uint2 *)X.dalloc(g.bits ? (size_t)NB * 32 * d / 8 : 0);
        g.onorm = (float *)X.dalloc(4 * (size_t)NB * 32);
        g.ipcent = (float *)X.dalloc(4 * (size_t)NB * 32);
        g.lcode = (uint8_t *)X.dalloc((size_t)n * g.lstride);
        g.exfac = (float2 *)X.dalloc(8 * (size_t)n);
        g.cent = (float *)X.dalloc(4 * (size_t)k * d);
        SAQG_CUDA_TRY(cudaMemset(g.codes, 0, g.bits ? (size_t)NB * 32 * d / 8 : 0));
        SAQG_CUDA_TRY(cudaMemset(g.onorm, 0, 4 * (size_t)NB * 32));
        SAQG_CUDA_TRY(cudaMemset(g.ipcent, 0, 4 * (size_t)NB * 32));
        SAQG_CUDA_TRY(cudaMemset(g.lcode, 0, (size_t)n * g.lstride));
        SAQG_CUDA_TRY(cudaMemset(g.exfac, 0, 8 * (size_t)n));
        // rotated centroids: clus.centroid() = centroid * P (quantizer.hpp:46)
        {
            dim3 grid((unsigned)(d / kRotN), (unsigned)((k + kRotM - 1) / kRotM));
            if (dP) {
                k_rotate<<<grid, kRotThreads>>>(dcent, (int)dim, didx.as<int64_t>(), k, off, (int)d, dP, nullptr, nullptr,
                                                g.cent, 0, 1);
                launch_check("k_rotate(centroids)");
            }
            k_centroid_slices<<<(unsigned)((k * d + 255) / 256), 256>>>(dcent, k, (int)dim, off, (int)d,
                                                                       cslice.as<float>());
            launch_check("k_centroid_slices");
            if (!dP) SAQG_CUDA_TRY(cudaMemcpy(g.cent, cslice.p, 4 * (size_t)k * d, cudaMemcpyDeviceToDevice));
        }
        std::vector<float> ident;
        DevBuf *idP = nullptr;
        std::unique_ptr<DevBuf> idbuf;
        if (!dP) {  // no rotation: residual = x - c, same kernel with an identity matrix
            ident.assign(d * d, 0.0f);
            for (int64_t i = 0; i < d; ++i) ident[i * d + i] = 1.0f;
            idbuf = std::make_unique<DevBuf>(4 * d * d);
            SAQG_CUDA_TRY(cudaMemcpy(idbuf->p, ident.data(), 4 * d * d, cudaMemcpyHostToDevice));
            idP = idbuf.get();
        }
        const int64_t chunk = encode_chunk(n, g.bits, maxd);
        for (int64_t v0 = 0; v0 < n; v0 += chunk) {
            const int64_t nv = std::min(chunk, n - v0);
            dim3 grid((unsigned)(d / kRotN), (unsigned)((nv + kRotM - 1) / kRotM));
            k_rotate<<<grid, kRotThreads>>>(ddata, (int)dim, drows.as<int64_t>() + v0, nv, off, (int)d,
                                            dP ? dP : idP->as<float>(), g.cent, dcid.as<int32_t>() + v0,
                                            resid.as<float>(), 1, ((uintptr_t)ddata & 15) == 0);
            launch_check("k_rotate");
            by_width(g.bits, [&](auto w) {
                k_caq_encode_clustered<decltype(w)::value>
                    <<<(unsigned)((nv + kEncThreads - 1) / kEncThreads), kEncThreads, enc_smem_bytes(g.bits)>>>(
                        resid.as<float>(), nv, (int)d, g.bits, cslice.as<float>(), dcid.as<int32_t>() + v0,
                        cfg.caq_adj_rd_lmt, cfg.caq_adj_eps, codes.as<uint16_t>(), facs.as<float>());
            });
            launch_check("k_caq_encode");
            k_pack<<<(unsigned)((nv + 127) / 128), 128>>>(codes.as<uint16_t>(), facs.as<float>(), nv, v0,
                                                          dcid.as<int32_t>() + v0, dbo, dvo, g);
            launch_check("k_pack");
        }
        SAQG_CUDA_TRY(cudaDeviceSynchronize());
        off += (int)d;
    }
    finalize_view(X);
    return I.release();
}

}  // namespace saqg

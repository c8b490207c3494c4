// Segment bit planner on the device: SaqDataMaker::dynamic_programming
// (quantization/saq_data.hpp:147-227).
//
// The reference's dynamic program pushes every state f[ns][i][bits] (least sum
// over ns segments of var_sum / 2^b covering the first i 64-dim blocks with
// `bits` total bits) forward to f[ns + 1][i + j][bits + b * 64 j + 64], keeping
// the first strict improvement in its visit order (ns, i, bits, then j, b),
// plus a 0-bit tail segment to the end.  Here each level ns + 1 is computed
// from level ns by one thread per target state (i', B'), which pulls its
// candidates in exactly the order the pushes would reach it: sources by i
// ascending, and for one i by bits ascending, i.e. b descending, the 0-bit tail
// (when i' is the end) last.  The same strict comparisons on the same double
// values give the same table, so the answer and the backtracked plan are the
// reference's.  The answer scan (the 1 % rule) runs in one warp, in order, and the
// backtrack in one thread.
#include <algorithm>
#include <cfloat>
#include <cstdint>
#include <string>
#include <vector>

#include "saqg_internal.h"

namespace saqg {

namespace {

constexpr double kLim = DBL_MAX;  // the reference's valid_lmt (numeric_limits<double>::max())

// Sum of one 64-float block in Eigen's 16-lane order (Redux.h:227-283):
// accumulators over packets {0, 2} and {1, 3}, then the 16 -> 1 tree.
__device__ float block_sum64(const float *x) {
    float r0[16];
#pragma unroll
    for (int l = 0; l < 16; ++l) {
        const float a = __fadd_rn(x[l], x[32 + l]);
        const float b = __fadd_rn(x[16 + l], x[48 + l]);
        r0[l] = __fadd_rn(a, b);
    }
    float a[8], b[4];
#pragma unroll
    for (int i = 0; i < 8; ++i) a[i] = __fadd_rn(r0[i], r0[i + 8]);
#pragma unroll
    for (int i = 0; i < 4; ++i) b[i] = __fadd_rn(a[i], a[i + 4]);
    return __fadd_rn(__fadd_rn(b[0], b[2]), __fadd_rn(b[1], b[3]));
}

// vsum[i * H + j] = sum of blocks i .. i + j - 1, accumulated in double from
// block i upward (the reference's var_sum for source i and length j).
__global__ void k_plan_vsum(const float *__restrict__ var, int i_end, int H, double *__restrict__ vsum) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= i_end) return;
    double s = 0.0;
    vsum[(size_t)i * H] = 0.0;
    for (int j = 1; i + j <= i_end; ++j) {
        s = __dadd_rn(s, (double)block_sum64(var + 64 * (size_t)(i + j - 1)));
        vsum[(size_t)i * H + j] = s;
    }
}

__global__ void k_plan_init(double *__restrict__ fv, uint32_t *__restrict__ fs, size_t total) {
    for (size_t t = blockIdx.x * (size_t)blockDim.x + threadIdx.x; t < total; t += (size_t)gridDim.x * blockDim.x) {
        fv[t] = t == 0 ? 0.0 : kLim;  // f[0][0][0] = 0
        fs[t] = 0;
    }
}

// x < DBL_MAX, as the comparison of doubles, on the words (FP64 comparisons run at
// 1/64 of the integer rate).
__device__ __forceinline__ bool below_lim(double x) {
    const uint32_t hi = (uint32_t)__double2hiint(x), lo = (uint32_t)__double2loint(x);
    return (hi & 0x7fffffffu) <= 0x7fefffffu && !(hi == 0x7fefffffu && lo == 0xffffffffu);
}

// Level ns + 1 from level ns (prev / next are one level's H x W slices).  FP64
// operations bound it; two per candidate remain, the sum and the comparison: the
// shares var_sum / 2^b (products with 2^-b, exact either way) are computed once per
// CTA, unreached states are seen on their words, and the states of one source's
// widths are loaded together.  960 dimensions at 4 bits: 80 us a level with a
// division per candidate, 38 us now.
constexpr int kPlanBits = kMaxBits, kPlanMaxBlocks = 256;
__global__ void __launch_bounds__(128) k_plan_level(const double *__restrict__ prev, double *__restrict__ next,
                                                    uint32_t *__restrict__ fs_next, const double *__restrict__ vsum,
                                                    int i_end, int H, int W, int nbf) {
    __shared__ double share[kPlanMaxBlocks][kPlanBits + 1];  // [source][b]; b = 0: var_sum itself
    const int Bp = blockIdx.x * blockDim.x + threadIdx.x;
    const int ip = blockIdx.y + 1;
    double val = kLim;
    uint32_t arg = 0;
    for (int i0 = 0; i0 < ip; i0 += kPlanMaxBlocks) {
        const int ni = min(kPlanMaxBlocks, ip - i0);
        __syncthreads();
        for (int e = threadIdx.x; e < ni * (kPlanBits + 1); e += blockDim.x) {
            const int i = e / (kPlanBits + 1), b = e % (kPlanBits + 1);
            share[i][b] = __dmul_rn(vsum[(size_t)(i0 + i) * H + ip - i0 - i], 1.0 / (double)(1 << b));
        }
        __syncthreads();
        if (Bp >= W) continue;
        for (int i = i0; i < i0 + ni; ++i) {
            const int j = ip - i;
            const double *row = prev + (size_t)i * W;
            double cur[kPlanBits + 1];
#pragma unroll
            for (int b = kPlanBits; b >= 1; --b) {
                const long long ub = (long long)Bp - (long long)b * j * 64 - nbf;
                cur[b] = ub < 0 ? kLim : row[ub];
            }
            cur[0] = ip == i_end ? row[Bp] : kLim;  // the 0-bit tail segment from source (i, Bp)
#pragma unroll
            for (int b = kPlanBits; b >= 0; --b) {
                if (!below_lim(cur[b])) continue;
                const double cand = __dadd_rn(cur[b], share[i - i0][b]);
                if (val > cand) {
                    val = cand;
                    arg = ((uint32_t)i << 4) + (uint32_t)b;
                }
            }
        }
    }
    if (Bp >= W) return;
    next[(size_t)ip * W + Bp] = val;
    fs_next[(size_t)ip * W + Bp] = arg;
}

// The answer (first end state, in (ns, bits) order, that beats the current one
// by 1 %) and the backtrack; out[0] = number of segments, then (length, bits).
// One warp: each lane holds kAnsRun end states of a run in order (state r * 32 +
// lane), loaded at once and a run ahead; of 32 states the first that beats the current one takes
// its place and the later ones are asked again, as the scan one by one would.  960
// dimensions at 4 bits: 2.9 ms with one thread waiting for each state, 0.09 ms now.
constexpr int kAnsRun = 16;
__global__ void __launch_bounds__(32) k_plan_answer(const double *__restrict__ fv, const uint32_t *__restrict__ fs,
                                                    int max_ns, int i_end, int H, int W, int tot_bits, int nbf,
                                                    long long *__restrict__ out, int cap) {
    const int lane = threadIdx.x;
    auto at = [&](int ns, int i, int b) { return ((size_t)ns * H + i) * W + b; };
    int ans_ns = 0, ans_b = tot_bits;
    double best = fv[at(0, i_end, tot_bits)], nxt[kAnsRun];
    auto load = [&](int ns, int u0) {
#pragma unroll
        for (int r = 0; r < kAnsRun; ++r) {
            const int ub = u0 + 32 * r + lane;
            nxt[r] = ns <= max_ns && ub <= tot_bits ? fv[at(ns, i_end, ub)] : kLim;
        }
    };
    load(0, 0);
    for (int ns = 0, u0 = 0; ns <= max_ns;) {
        double cur[kAnsRun];
#pragma unroll
        for (int r = 0; r < kAnsRun; ++r) cur[r] = nxt[r];
        const int at_ns = ns, at_u = u0;
        u0 += 32 * kAnsRun;
        if (u0 > tot_bits) {
            u0 = 0;
            ++ns;
        }
        load(ns, u0);
#pragma unroll
        for (int r = 0; r < kAnsRun; ++r) {
            const double lim = below_lim(cur[r]) ? __dmul_rn(cur[r], 1.01) : kLim;
            for (unsigned later = 0xffffffffu; later;) {
                const unsigned win = __ballot_sync(0xffffffffu, below_lim(cur[r]) && lim < best) & later;
                if (!win) break;
                const int l = __ffs(win) - 1;
                later = ~((2u << l) - 1u);
                best = __shfl_sync(0xffffffffu, cur[r], l);
                ans_ns = at_ns;
                ans_b = at_u + 32 * r + l;
            }
        }
    }
    if (lane) return;
    int ns = ans_ns, i = i_end, B = ans_b, n = 0;
    long long tmp[2 * 64];
    // (as the reference: with no segment possible the walk reads the table's
    // untouched state and yields one 0-bit segment; a corrupt table ends the
    // walk with out[0] = -1)
    while (i > 0 && n < 64 && ns >= 0 && B >= 0) {
        const uint32_t s = fs[at(ns, i, B)];
        const int pi = (int)(s >> 4), bits = (int)(s & 0xf);
        if (pi >= i) break;
        const int len = (i - pi) * 64;
        tmp[2 * n] = len;
        tmp[2 * n + 1] = bits;
        ++n;
        --ns;
        i = pi;
        if (bits) B -= bits * len + nbf;
    }
    out[0] = i == 0 ? n : -1;
    for (int k = 0; k < n && k < cap; ++k) {  // reversed: first segment first
        out[1 + 2 * k] = tmp[2 * (n - 1 - k)];
        out[2 + 2 * k] = tmp[2 * (n - 1 - k) + 1];
    }
}

struct DevMem {
    void *p = nullptr;
    explicit DevMem(size_t b) {
        const cudaError_t e = cudaMalloc(&p, b ? b : 16);
        if (e != cudaSuccess) throw Error{SAQG_ERR_NOMEM, std::string("cudaMalloc failed: ") + cudaGetErrorString(e)};
    }
    ~DevMem() {
        if (p) cudaFree(p);
    }
};

void launched(const char *what) {
    const cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) throw Error{SAQG_ERR_CUDA, std::string(what) + " launch failed: " + cudaGetErrorString(e)};
    count_launch(1);
}

}  // namespace

// The DP plan from a device-resident variance (dim_padded floats), on `st`.
std::vector<std::pair<int64_t, int64_t>> make_plan_device(const float *dvar, int64_t Dp, float avg_bits,
                                                          cudaStream_t st) {
    SAQG_REQUIRE(Dp > 0 && Dp % 64 == 0, "dim_padded must be a positive multiple of 64");
    const int nbf = 2 * (int)sizeof(float) * 8;
    const int tot_bits = (int)(size_t)(avg_bits * (float)Dp + (float)nbf);
    const int i_end = (int)(Dp / 64), H = i_end + 1, W = tot_bits + 1;
    const int max_ns = avg_bits < 2 ? i_end : i_end / 2;
    const size_t level = (size_t)H * W, total = (size_t)(max_ns + 1) * level;
    DevMem fv(8 * total), fs(4 * total), vs(8 * (size_t)H * H), out(8 * (1 + 2 * 64));
    double *dfv = static_cast<double *>(fv.p);
    uint32_t *dfs = static_cast<uint32_t *>(fs.p);
    double *dvs = static_cast<double *>(vs.p);
    long long *dout = static_cast<long long *>(out.p);
    k_plan_vsum<<<(i_end + 63) / 64, 64, 0, st>>>(dvar, i_end, H, dvs);
    launched("k_plan_vsum");
    k_plan_init<<<(unsigned)std::min<size_t>((total + 255) / 256, 4096), 256, 0, st>>>(dfv, dfs, total);
    launched("k_plan_init");
    for (int ns = 0; ns < max_ns; ++ns) {
        k_plan_level<<<dim3((unsigned)((W + 127) / 128), (unsigned)i_end), 128, 0, st>>>(
            dfv + ns * level, dfv + (ns + 1) * level, dfs + (ns + 1) * level, dvs, i_end, H, W, nbf);
        launched("k_plan_level");
    }
    k_plan_answer<<<1, 32, 0, st>>>(dfv, dfs, max_ns, i_end, H, W, tot_bits, nbf, dout, 64);
    launched("k_plan_answer");
    long long h[1 + 2 * 64];
    SAQG_CUDA_TRY(cudaMemcpyAsync(h, dout, sizeof(h), cudaMemcpyDeviceToHost, st));
    SAQG_CUDA_TRY(cudaStreamSynchronize(st));
    SAQG_REQUIRE(h[0] >= 1 && h[0] <= 64, "device planner produced no valid plan");
    std::vector<std::pair<int64_t, int64_t>> plan;
    for (long long k = 0; k < h[0]; ++k) plan.emplace_back((int64_t)h[1 + 2 * k], (int64_t)h[2 + 2 * k]);
    return plan;
}

// Equal segmentation needs no program; the DP runs on the device.
std::vector<std::pair<int64_t, int64_t>> make_plan_gpu(const float *var, int64_t Dp, float avg_bits, bool seg,
                                                       int eqseg, bool var_on_device, cudaStream_t st) {
    if (!seg || eqseg > 0) return make_plan(nullptr, Dp, avg_bits, seg, eqseg);
    if (var_on_device) return make_plan_device(var, Dp, avg_bits, st);
    DevMem dv(4 * (size_t)Dp);
    SAQG_CUDA_TRY(cudaMemcpyAsync(dv.p, var, 4 * (size_t)Dp, cudaMemcpyHostToDevice, st));
    return make_plan_device(static_cast<const float *>(dv.p), Dp, avg_bits, st);
}

}  // namespace saqg

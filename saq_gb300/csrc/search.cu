// Search hot path: IVF::search / IVF::estimate (index/ivf.hpp:275-362) on the GPU.
//
// Pipeline for a batch of nq independent queries (nq = 1 is the plain
// single-query drop-in):
//   k_probe_dist   L2 from every query to every centroid, in Eigen's order
//                  (FlatInitializer::centroids_distances, initializer.hpp:52-76)
//   k_probe_select the nprobe nearest in std::partial_sort order: radix select
//                  + sort; on any tie the exact libstdc++ heap algorithm runs
//   k_qprep_few / k_qprep_tiled + k_prune_bounds
//                  per segment: zero-padded query slice, prune bound
//                  sqrt(sum var*q^2)*m and the rotated query q_s*P_s in Eigen's
//                  GEMV order (saq_estimator.hpp:28-48, caq_estimator.hpp:56-68)
//   k_scan         one CTA per query walks its probes in order: 128 blocks at a
//                  time are filtered by the first pruning stage; of the rest, per
//                  cluster the LUTs (Lut::prepare, lut.hpp:60-87) and per tile of
//                  blocks (one warp = one 32-vector block) FastScan sums and fast /
//                  variance estimates, the block's pruning stages, accurate
//                  distances of every lane that can pass under the tile-start
//                  distk (distk only shrinks, so this is a superset), then one
//                  warp replays SAQSearcher::searchCluster / scanCluster
//                  (saq_searcher.hpp:68-214) and the ResultPool inserts
//                  (utils/pool.hpp:17-30) exactly in the reference's order.
#include <cfloat>
#include <climits>
#include <cstdio>
#include <cstdlib>
#include <functional>
#include <map>
#include <memory>
#include <string>
#include <tuple>

#include "device_common.cuh"
#include "rotate.cuh"
#include "saqg_internal.h"

namespace saqg {

namespace {

constexpr int kScanWarps = 8;
constexpr int kScanThreads = kScanWarps * 32;
constexpr int kBlocksPerWarp = 2;
constexpr int kTileB = kScanWarps * kBlocksPerWarp;  // blocks per tile
constexpr int kMaxTopK = 4096;
// Candidates of a tile up to which half-warps take the accurate distances, with one
// segment and with several (whose tasks spread over the warps by themselves).
constexpr int kItemCands = 16, kItemCandsSegs = 6;
constexpr int kPullDim = 1024;  // one segment from this width on: codes prefetched (tile_candidates)
constexpr int kScanMinCtas = 4;  // resident scan CTAs per SM the register budget is sized for

struct SegScal {
    float delta, vl, sum_vl, sum_q, q_l2sqr, q_l2norm, c1, c2, vfac;
    float rdelta;  // RN(1 / delta), for the LUT quantizer
};

// A u16 LUT entry (uint16_t)(int)(x / d), x >= 0, with the division rounded to
// nearest, without dividing.  n, the integer nearest to x * RN(1 / d), is within 0.52
// of x / d (x / d stays below 65,536), so the entry is n or n - 1: n when x / d rounds
// to n or above, i.e. when n - x / d is at most half the spacing u of the floats below n
// (n is the even neighbour of that tie).  x - n d, one FMA, decides: its sign is
// right, and where it is near -d u / 2 (below 2^-9 d) it is exact, a multiple of d's
// last place of less than 24 bits.  d must be a normal float with room below
// (lut_quant_ok); 16 entries take 11 operations each, where a check of the product
// and a division for 3% of the entries took 7 and a loop.
__device__ __forceinline__ bool lut_quant_ok(float d) { return d > 1e-30f && d < 1e30f; }
__device__ __forceinline__ uint32_t lut_quant(float x, float d, float r) {
    const float m = __fadd_rn(__fmul_rn(x, r), 8388608.0f);  // 2^23 + n: n in the low mantissa bits
    const float n = __fsub_rn(m, 8388608.0f);
    const float half_u = __uint_as_float(((__float_as_uint(n) - 1u) & 0x7f800000u) - (24u << 23));  // n = 0: huge
    const float rem = __fmaf_rn(-n, d, x);
    return (__float_as_uint(m) - (rem < -__fmul_rn(d, half_u) ? 1u : 0u)) & 0xffffu;
}

__device__ __forceinline__ uint32_t fkey(float f) {
    uint32_t u = __float_as_uint(f);
    return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}

__device__ __forceinline__ float key_to_float(uint32_t k) {
    return __uint_as_float((k & 0x80000000u) ? (k & 0x7fffffffu) : ~k);
}

// Per-query nprobe and k of a batch (null arrays: every query uses the
// maxima).  Probe rows are np_max long and result rows k_max long.
struct QueryShape {
    const int *np = nullptr, *k = nullptr;
    int np_max = 0, k_max = 0;
    __device__ __forceinline__ int np_of(int qi) const { return np ? np[qi] : np_max; }
    __device__ __forceinline__ int k_of(int qi) const { return k ? k[qi] : k_max; }
};

// ------------------------------------------------------------------ probe
__global__ void k_probe_dist(DevIndexView ix, const float *__restrict__ q, float *__restrict__ dist) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int c = blockIdx.x * (blockDim.x >> 5) + warp;
    const int qi = blockIdx.y;
    if (c >= ix.K) return;
    const float *cr = ix.centroids + (size_t)c * ix.D;
    const float *qq = q + (size_t)qi * ix.D;
    float d = warp_eigen_sum(ix.D, [&](int i) {
        const float t = __fsub_rn(cr[i], qq[i]);
        return __fmul_rn(t, t);
    });
    if (lane == 0) dist[(size_t)qi * ix.K + c] = d;
}

// Tiled form for batches: a CTA holds kProbeQT queries in shared memory; each
// warp keeps one centroid in registers (lane (h, l) holds the elements of the
// packets p = h, h+2, ... at offset l -- Eigen's two-accumulator assignment)
// and evaluates it against every query of the tile.  Same reduction order as
// k_probe_dist (dimension a multiple of 32, so no odd packet or scalar tail).
constexpr int kProbeQT = 16, kProbeWarps = 8, kProbeRegs = 64;  // up to 64 floats per lane: dim <= 2048
__global__ void __launch_bounds__(kProbeWarps * 32) k_probe_dist_tiled(DevIndexView ix, const float *__restrict__ q,
                                                                        int nq, float *__restrict__ dist) {
    extern __shared__ float qs[];  // kProbeQT x D
    const int D = ix.D, warp = threadIdx.x >> 5, lane = threadIdx.x & 31, l = lane & 15, h = lane >> 4;
    const int q0 = blockIdx.y * kProbeQT, nqt = min(kProbeQT, nq - q0);
    for (int i = threadIdx.x; i < nqt * D; i += blockDim.x) qs[i] = q[(size_t)q0 * D + i];
    __syncthreads();
    const int npk = D / 32;  // packets per lane
    for (int c = blockIdx.x * kProbeWarps + warp; c < ix.K; c += gridDim.x * kProbeWarps) {
        const float *cr = ix.centroids + (size_t)c * D;
        float cv[kProbeRegs];
#pragma unroll
        for (int k = 0; k < kProbeRegs; ++k)
            if (k < npk) cv[k] = cr[16 * (h + 2 * k) + l];
        for (int qi = 0; qi < nqt; ++qi) {
            const float *qq = qs + qi * D;
            float acc = 0.0f;
#pragma unroll
            for (int k = 0; k < kProbeRegs; ++k)
                if (k < npk) {
                    const float t = __fsub_rn(cv[k], qq[16 * (h + 2 * k) + l]);
                    acc = k == 0 ? __fmul_rn(t, t) : __fadd_rn(acc, __fmul_rn(t, t));
                }
            acc = __fadd_rn(acc, __shfl_down_sync(kFull, acc, 16));
            acc = __fadd_rn(acc, __shfl_down_sync(kFull, acc, 8));
            acc = __fadd_rn(acc, __shfl_down_sync(kFull, acc, 4));
            acc = __fadd_rn(acc, __shfl_down_sync(kFull, acc, 2));
            acc = __fadd_rn(acc, __shfl_down_sync(kFull, acc, 1));
            if (lane == 0) dist[(size_t)(q0 + qi) * ix.K + c] = acc;
        }
    }
}

struct Cand {
    uint32_t id;
    float d;
};

// libstdc++ std::partial_sort (stl_algo.h __heap_select + __sort_heap,
// stl_heap.h __adjust_heap / __push_heap / __pop_heap), comp = operator< on
// the distance (Candidate::operator<, defines.hpp:48).
__device__ void heap_adjust(Cand *a, long hole, long len, Cand val) {
    const long top = hole;
    long sc = hole;
    while (sc < (len - 1) / 2) {
        sc = 2 * (sc + 1);
        if (a[sc].d < a[sc - 1].d) sc--;
        a[hole] = a[sc];
        hole = sc;
    }
    if ((len & 1) == 0 && sc == (len - 2) / 2) {
        sc = 2 * (sc + 1);
        a[hole] = a[sc - 1];
        hole = sc - 1;
    }
    long parent = (hole - 1) / 2;
    while (hole > top && a[parent].d < val.d) {
        a[hole] = a[parent];
        hole = parent;
        parent = (hole - 1) / 2;
    }
    a[hole] = val;
}

__device__ void exact_partial_sort(Cand *a, long mid, long len) {
    if (mid >= 2)
        for (long parent = (mid - 2) / 2;; --parent) {
            heap_adjust(a, parent, mid, a[parent]);
            if (parent == 0) break;
        }
    for (long i = mid; i < len; ++i)
        if (a[i].d < a[0].d) {
            Cand v = a[i];
            a[i] = a[0];
            heap_adjust(a, 0, mid, v);
        }
    for (long last = mid; last > 1;) {
        --last;
        Cand v = a[last];
        a[last] = a[0];
        heap_adjust(a, 0, last, v);
    }
}

// One radix-select step, by a whole warp: the first bin b with
// hist[0] + ... + hist[b] > rem and the count of the bins before it (what a
// sequential scan of the 256 bins finds).
__device__ __forceinline__ void select_bin(const uint32_t *hist, uint32_t rem, int &b, uint32_t &below) {
    const int lane = threadIdx.x & 31;
    uint32_t h[8], sum = 0;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        h[i] = hist[lane * 8 + i];
        sum += h[i];
    }
    uint32_t incl = sum;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t v = __shfl_up_sync(kFull, incl, o);
        if (lane >= o) incl += v;
    }
    const uint32_t excl = incl - sum;
    const uint32_t m = __ballot_sync(kFull, excl <= rem && rem < incl);
    if (!m) {  // rem beyond every count: the scan runs off the end
        b = 256;
        below = __shfl_sync(kFull, incl, 31);
        return;
    }
    const int L = __ffs(m) - 1;
    int bb = 0;
    uint32_t cum = excl;
    if (lane == L) {
        int i = 0;
        for (; i < 8; ++i) {
            if (cum + h[i] > rem) break;
            cum += h[i];
        }
        bb = L * 8 + i;
    }
    b = __shfl_sync(kFull, bb, L);
    below = __shfl_sync(kFull, cum, L);
}

constexpr int kSelThreads = 1024;
constexpr int kSelMax = 1024;  // fast path handles nprobe <= 1024

__global__ void __launch_bounds__(kSelThreads) k_probe_select(const float *__restrict__ dist, int K, int nprobe_max,
                                                              uint32_t *__restrict__ probe, Cand *__restrict__ work,
                                                              int *__restrict__ fallback_count,
                                                              const uint8_t *__restrict__ only = nullptr,
                                                              const int *__restrict__ qnp = nullptr) {
    __shared__ uint32_t hist[256];
    __shared__ uint32_t s_prefix, s_mask, s_rem, s_eq, s_n;
    __shared__ unsigned long long sel[kSelMax];
    const int qi = blockIdx.x, tid = threadIdx.x;
    if (only && !only[qi]) return;  // ranked by the shortlist
    const int nprobe = qnp ? qnp[qi] : nprobe_max;  // this query's nprobe; rows are nprobe_max long
    const float *dq = dist + (size_t)qi * K;
    if (tid == 0) {
        s_prefix = 0;
        s_mask = 0;
        s_rem = (uint32_t)(nprobe - 1);
    }
    __syncthreads();
    for (int pass = 0; pass < 4; ++pass) {
        const int shift = 24 - 8 * pass;
        for (int i = tid; i < 256; i += kSelThreads) hist[i] = 0;
        __syncthreads();
        const uint32_t prefix = s_prefix, mask = s_mask;
        for (int i = tid; i < K; i += kSelThreads) {
            const uint32_t k = fkey(dq[i]);
            if ((k & mask) == prefix) atomicAdd(&hist[(k >> shift) & 255u], 1u);
        }
        __syncthreads();
        if (tid < 32) {
            int b;
            uint32_t cum;
            select_bin(hist, s_rem, b, cum);
            if (tid == 0) {
                s_rem = s_rem - cum;
                s_prefix = prefix | ((uint32_t)b << shift);
                s_mask = mask | (255u << shift);
                s_eq = b < 256 ? hist[b] : 0u;
                s_n = 0;
            }
        }
        __syncthreads();
    }
    const uint32_t T = s_prefix;
    const uint32_t count_lt = (uint32_t)(nprobe - 1) - s_rem;
    bool need_exact = (s_eq != 1) || nprobe > kSelMax;
    if (!need_exact) {
        for (int i = tid; i < K; i += kSelThreads) {
            const uint32_t k = fkey(dq[i]);
            if (k <= T) {
                const uint32_t pos = atomicAdd(&s_n, 1u);
                if (pos < kSelMax) sel[pos] = ((unsigned long long)k << 32) | (uint32_t)i;
            }
        }
        __syncthreads();
        const int n = (int)s_n;
        int P = 1;
        while (P < n) P <<= 1;
        for (int i = n + tid; i < P; i += kSelThreads) sel[i] = ~0ull;
        __syncthreads();
        for (int k = 2; k <= P; k <<= 1)
            for (int j = k >> 1; j > 0; j >>= 1) {
                for (int i = tid; i < P; i += kSelThreads) {
                    const int ixj = i ^ j;
                    if (ixj > i) {
                        const unsigned long long a = sel[i], b = sel[ixj];
                        const bool up = (i & k) == 0;
                        if ((a > b) == up) {
                            sel[i] = b;
                            sel[ixj] = a;
                        }
                    }
                }
                __syncthreads();
            }
        // equal keys inside the selection make the heap order matter
        __shared__ int s_dup;
        if (tid == 0) s_dup = (n != nprobe) || (count_lt + 1 != (uint32_t)nprobe);
        __syncthreads();
        for (int i = tid; i + 1 < n; i += kSelThreads)
            if ((sel[i] >> 32) == (sel[i + 1] >> 32)) s_dup = 1;
        __syncthreads();
        if (!s_dup) {
            for (int i = tid; i < nprobe; i += kSelThreads) probe[(size_t)qi * nprobe_max + i] = (uint32_t)(sel[i] & 0xffffffffu);
            return;
        }
        need_exact = true;
    }
    // exact fallback: the standard library's algorithm, sequentially
    if (nprobe > kSelMax) {
        if (tid == 0) {
            atomicAdd(fallback_count, 1);
            Cand *a = work + (size_t)qi * K;
            for (int i = 0; i < K; ++i) a[i] = Cand{(uint32_t)i, dq[i]};
            exact_partial_sort(a, nprobe, K);
            for (int i = 0; i < nprobe; ++i) probe[(size_t)qi * nprobe_max + i] = a[i].id;
        }
        return;
    }
    // the same steps with the heap (the first nprobe slots of the array) in
    // shared memory; the rest of the row is only ever compared against the
    // heap's top at its turn, so it streams through in coalesced chunks
    __shared__ float chunk[kSelThreads];
    Cand *heap = reinterpret_cast<Cand *>(sel);
    const int mid = nprobe;
    for (int i = tid; i < mid; i += kSelThreads) heap[i] = Cand{(uint32_t)i, dq[i]};
    __syncthreads();
    if (tid == 0) {
        atomicAdd(fallback_count, 1);
        if (mid >= 2)
            for (long parent = (mid - 2) / 2;; --parent) {
                heap_adjust(heap, parent, mid, heap[parent]);
                if (parent == 0) break;
            }
    }
    // the heap's top only shrinks, so an element not below the top at its
    // chunk's start is skipped at its own turn too: each chunk is filtered in
    // parallel against that top and thread 0 runs the steps on the rest, in order
    __shared__ int s_wcnt[kSelThreads / 32];
    __shared__ int s_list[kSelThreads];
    const int lane = tid & 31, wp = tid >> 5;
    for (int base = mid; base < K; base += kSelThreads) {
        __syncthreads();
        const float top = heap[0].d;
        const float v = base + tid < K ? dq[base + tid] : 0.0f;
        const bool in = base + tid < K && v < top;
        const uint32_t bal = __ballot_sync(kFull, in);
        if (lane == 0) s_wcnt[wp] = __popc(bal);
        chunk[tid] = v;
        __syncthreads();
        int off = 0, total = 0;
        for (int i = 0; i < kSelThreads / 32; ++i) {
            if (i < wp) off += s_wcnt[i];
            total += s_wcnt[i];
        }
        if (in) s_list[off + __popc(bal & ((1u << lane) - 1))] = tid;
        __syncthreads();
        if (tid == 0)
            for (int r = 0; r < total; ++r) {
                const int j = s_list[r];
                if (chunk[j] < heap[0].d) heap_adjust(heap, 0, mid, Cand{(uint32_t)(base + j), chunk[j]});
            }
    }
    if (tid == 0) {
        for (long last = mid; last > 1;) {
            --last;
            const Cand v = heap[last];
            heap[last] = heap[0];
            heap_adjust(heap, 0, last, v);
        }
        for (int i = 0; i < mid; ++i) probe[(size_t)qi * nprobe_max + i] = heap[i].id;
    }
}

// ------------------------------------------------------ probe: GEMM shortlist
// Batches rank centroids from inner products q.c computed by a BF16
// tensor-core GEMM (probe_gemm.cu).  Each approximate distance a = |q|^2 +
// |c|^2 - 2 q.c gets a rigorous bound b on its distance from the reference's
// float distance (operands rounded to BF16 are within 2^-9 of their FP32
// values, so |q.c error| <= (2^-8 + 2^-18 + accumulation) |q||c|; the norms and
// the reference's own sum add (2D + 32) * 2^-24 (|q| + |c|)^2).  Every centroid of the exact top-nprobe has
// a - b <= T, T the nprobe-th smallest a + b, so only those centroids get the
// exact Eigen-order distance and the ranking is the exact one.  A query with
// equal distances among its first nprobe + 1 (where the standard library's
// heap order decides), a non-finite value or more than kShortCap centroids on
// its shortlist is ranked by the full exact path instead.
constexpr int kShortThreads = 512;
constexpr int kShortCap = 1024;  // shortlist capacity (more: the full exact path); keeps 2 CTAs per SM
constexpr int kGemmMinQueries = 64;  // smaller calls rank with the exact kernels directly

constexpr int kShortKeys = 16384;    // clusters whose upper-bound keys the shortlist keeps in shared memory

// |c|^2 and |c| of every centroid (any summation order: only the bounds use them)
__global__ void k_cnorm2(DevIndexView ix, float2 *__restrict__ cn) {
    const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
    if (warp >= ix.K) return;
    const float *cr = ix.centroids + (size_t)warp * ix.D;
    float a = 0.0f;
    for (int i = lane; i < ix.D; i += 32) a += cr[i] * cr[i];
    for (int o = 16; o; o >>= 1) a += __shfl_xor_sync(kFull, a, o);
    if (lane == 0) cn[warp] = make_float2(a, sqrtf(a));
}

struct ShortBound {
    float e1, e2;  // b = e1 |q||c| + e2 (|q| + |c|)^2
};

__device__ __forceinline__ void approx_bounds(float qn2, float qn, float ip, float2 cnn, const ShortBound &sb, float &lo,
                                              float &hi) {
    const float cn2 = cnn.x, cn = cnn.y;
    const float a = (qn2 + cn2) - 2.0f * ip;
    const float s = qn + cn;
    const float b = (sb.e1 * qn * cn + sb.e2 * s * s) * 1.01f + 1e-30f;
    lo = a - b;
    hi = a + b;
}

__global__ void __launch_bounds__(kShortThreads) k_probe_shortlist(DevIndexView ix, const float *__restrict__ q,
                                                                   const float *__restrict__ ip,
                                                                   const float2 *__restrict__ cn2, ShortBound sb,
                                                                   int nprobe_max, const int *__restrict__ qnp,
                                                                   uint32_t *__restrict__ probe,
                                                                   uint8_t *__restrict__ full, int *__restrict__ fb_list,
                                                                   int *__restrict__ fb_count,
                                                                   unsigned long long *__restrict__ counters,
                                                                   const int *__restrict__ ip_err, int keep_keys) {
    extern __shared__ __align__(16) char smem_raw[];
    unsigned long long *keys = reinterpret_cast<unsigned long long *>(smem_raw);  // [kShortCap]
    uint32_t *cand = reinterpret_cast<uint32_t *>(keys + kShortCap);             // [kShortCap]
    float *qs = reinterpret_cast<float *>(cand + kShortCap);                      // [D]
    uint32_t *hk = reinterpret_cast<uint32_t *>(qs + ix.D);                       // [K] when keep_keys
    const bool keep = keep_keys != 0;
    __shared__ uint32_t hist[256];
    __shared__ uint32_t tmin[2 * kShortThreads];
    __shared__ uint32_t s_prefix, s_mask, s_rem, s_n;
    __shared__ int s_bad;
    __shared__ float s_red[kShortThreads / 32];
    const int qi = blockIdx.x, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int K = ix.K, D = ix.D;
    const int nprobe = qnp ? qnp[qi] : nprobe_max;
    const float *ipq = ip + (size_t)qi * K;
    float a = 0.0f;
    for (int i = tid; i < D; i += kShortThreads) {
        const float v = q[(size_t)qi * D + i];
        qs[i] = v;
        a += v * v;
    }
    for (int o = 16; o; o >>= 1) a += __shfl_xor_sync(kFull, a, o);
    if (lane == 0) s_red[warp] = a;
    if (tid == 0) {
        s_prefix = 0;
        s_mask = 0;
        s_rem = (uint32_t)(nprobe - 1);
        s_n = 0;
        s_bad = 0;
    }
    __syncthreads();
    float qn2 = 0.0f;
    for (int i = 0; i < kShortThreads / 32; ++i) qn2 += s_red[i];
    const float qn = sqrtf(qn2);
    // T: the nprobe-th smallest upper end (radix select on the order-preserving
    // keys).  For nprobe <= threads / 2, each thread contributes the two smallest
    // upper ends of its strided share of the centroids and T is the nprobe-th
    // smallest of those: the nprobe-th smallest of a subset of the upper ends is
    // at least the nprobe-th smallest of all, so the shortlist below still holds
    // every centroid of the exact top-nprobe (it may hold a few more).  With the
    // smallest alone nprobe = 256 of 16,384 gives the 355th: this kernel took 0.99 ms
    // for 4,096 queries with nprobe up to 256, with two 0.55.
    const bool by_thread = nprobe <= kShortThreads / 2;
    if (by_thread) {
        uint32_t m = 0xffffffffu, m2 = 0xffffffffu;
        for (int c = tid; c < K; c += kShortThreads) {
            float lo, hi;
            approx_bounds(qn2, qn, ipq[c], cn2[c], sb, lo, hi);
            if (!(isfinite(lo) && isfinite(hi))) s_bad = 1;
            const uint32_t k = fkey(hi);
            m2 = min(m2, max(m, k));
            m = min(m, k);
        }
        tmin[tid] = m;
        tmin[kShortThreads + tid] = m2;
    }
    for (int pass = 0; pass < 4; ++pass) {
        const int shift = 24 - 8 * pass;
        for (int i = tid; i < 256; i += kShortThreads) hist[i] = 0;
        __syncthreads();
        const uint32_t prefix = s_prefix, mask = s_mask;
        if (by_thread) {
            for (int i = tid; i < 2 * kShortThreads; i += kShortThreads) {
                const uint32_t k = tmin[i];
                if ((k & mask) == prefix) atomicAdd(&hist[(k >> shift) & 255u], 1u);
            }
        } else {
            for (int c = tid; c < K; c += kShortThreads) {
                uint32_t k;
                if (pass == 0 || !keep) {
                    float lo, hi;
                    approx_bounds(qn2, qn, ipq[c], cn2[c], sb, lo, hi);
                    if (pass == 0 && !(isfinite(lo) && isfinite(hi))) s_bad = 1;
                    k = fkey(hi);
                    if (keep) hk[c] = k;
                } else {
                    k = hk[c];
                }
                if ((k & mask) == prefix) atomicAdd(&hist[(k >> shift) & 255u], 1u);
            }
        }
        __syncthreads();
        if (tid < 32) {
            int b;
            uint32_t cum;
            select_bin(hist, s_rem, b, cum);
            if (tid == 0) {
                s_rem = s_rem - cum;
                s_prefix = prefix | ((uint32_t)b << shift);
                s_mask = mask | (255u << shift);
            }
        }
        __syncthreads();
    }
    const float T = key_to_float(s_prefix);
    if (*ip_err) s_bad = 1;  // the inner products are incomplete: the full exact path ranks every query
    // the shortlist: lower end not above T
    if (!s_bad)
        for (int c = tid; c < K; c += kShortThreads) {
            float lo, hi;
            approx_bounds(qn2, qn, ipq[c], cn2[c], sb, lo, hi);
            if (lo <= T) {
                const uint32_t pos = atomicAdd(&s_n, 1u);
                if (pos < kShortCap) cand[pos] = (uint32_t)c;
            }
        }
    __syncthreads();
    const int n = (int)s_n;
    if (s_bad || n > kShortCap) {
        if (tid == 0) {
            full[qi] = 1;
            fb_list[atomicAdd(fb_count, 1)] = qi;
            if (counters) atomicAdd(counters + 5, 1ull);
            if (counters) atomicAdd(counters + 4, (unsigned long long)K);
        }
        return;
    }
    // exact distances of the shortlist, in the reference's order (as k_probe_dist)
    for (int i = warp; i < n; i += kShortThreads / 32) {
        const uint32_t c = cand[i];
        const float *cr = ix.centroids + (size_t)c * D;
        const float d = warp_eigen_sum(D, [&](int e) {
            const float t = __fsub_rn(cr[e], qs[e]);
            return __fmul_rn(t, t);
        });
        if (lane == 0) {
            if (d != d) s_bad = 1;
            keys[i] = ((unsigned long long)fkey(d) << 32) | c;
        }
    }
    int P = 1;
    while (P < n) P <<= 1;
    for (int i = n + tid; i < P; i += kShortThreads) keys[i] = ~0ull;
    __syncthreads();
    for (int k = 2; k <= P; k <<= 1)
        for (int j = k >> 1; j > 0; j >>= 1) {
            for (int i = tid; i < P; i += kShortThreads) {
                const int ixj = i ^ j;
                if (ixj > i) {
                    const unsigned long long x = keys[i], y = keys[ixj];
                    if ((x > y) == ((i & k) == 0)) {
                        keys[i] = y;
                        keys[ixj] = x;
                    }
                }
            }
            __syncthreads();
        }
    // equal distances among the first nprobe + 1 leave the order to the heap
    const int m = min(n, nprobe + 1);
    for (int i = tid; i + 1 < m; i += kShortThreads)
        if ((keys[i] >> 32) == (keys[i + 1] >> 32)) s_bad = 1;
    __syncthreads();
    if (s_bad || n < nprobe) {
        if (tid == 0) {
            full[qi] = 1;
            fb_list[atomicAdd(fb_count, 1)] = qi;
            if (counters) atomicAdd(counters + 6, 1ull);
            if (counters) atomicAdd(counters + 4, (unsigned long long)K);
        }
        return;
    }
    for (int i = tid; i < nprobe; i += kShortThreads) probe[(size_t)qi * nprobe_max + i] = (uint32_t)(keys[i] & 0xffffffffu);
    if (tid == 0) {
        full[qi] = 0;
        if (counters) atomicAdd(counters + 4, (unsigned long long)n);
    }
}

// Exact distances to every centroid for the queries the shortlist handed back
// (a grid-stride loop over (query, group of 8 centroids)).
__global__ void k_probe_dist_list(DevIndexView ix, const float *__restrict__ q, float *__restrict__ dist,
                                  const int *__restrict__ fb_list, const int *__restrict__ fb_count) {
    const int nfb = *fb_count;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, wpb = blockDim.x >> 5;
    const int groups = (ix.K + wpb - 1) / wpb;
    for (long w = blockIdx.x; w < (long)nfb * groups; w += gridDim.x) {
        const int qi = fb_list[w / groups], c = (int)(w % groups) * wpb + warp;
        if (c >= ix.K) continue;
        const float *cr = ix.centroids + (size_t)c * ix.D;
        const float *qq = q + (size_t)qi * ix.D;
        const float d = warp_eigen_sum(ix.D, [&](int i) {
            const float t = __fsub_rn(cr[i], qq[i]);
            return __fmul_rn(t, t);
        });
        if (lane == 0) dist[(size_t)qi * ix.K + c] = d;
    }
}

// ------------------------------------------------------------------ query prep
// Prune bound sqrt(sum var * q^2) * m of segment s and query slice cq (zero-padded
// past the dimension), by one warp; valid in every lane.
template <class Q>
__device__ __forceinline__ float prune_bound(const DevIndexView &ix, const SegDev &g, float m, Q cq) {
    const float *var = ix.var + g.qoff;
    const float v2 = warp_eigen_sum(g.dim, [&](int i) {
        const float q = cq(i);
        return __fmul_rn(var[i], __fmul_rn(q, q));
    });
    return __fmul_rn(sqrtf(v2), m);
}

// ------------------------------------------------------------------ LUT

// 16 float LUT entries of one 4-dim codebook: fastscan::pack_lut (fastscan.hpp:236-248),
// entry j = entry[j - lowbit(j)] + q[kPos[j]].
__device__ __forceinline__ void lut_entries(const float *__restrict__ qq, float *t) {
    t[0] = 0.0f;
#pragma unroll
    for (int j = 1; j < 16; ++j) {
        const int lb = j & -j, pos = lb == 1 ? 3 : lb == 2 ? 2 : lb == 4 ? 1 : 0;  // kPos[j] (fastscan.hpp:22-39)
        t[j] = __fadd_rn(t[j - lb], qq[pos]);
    }
}

// Lut::compFastIP's float epilogue and the L2 form of CaqCluEstimator::compFastDist
// (caq_estimator.hpp:148-179) for a FastScan sum.
__device__ __forceinline__ float fast_of_sum(const SegScal &sc, int sum, float onorm, float &ipx) {
    float t = __fmul_rn((float)sum, sc.delta);
    t = __fadd_rn(t, sc.sum_vl);
    ipx = t;
    float f = __fmul_rn(__fsub_rn(t, sc.c1), sc.c2);
    f = __fmul_rn(f, onorm);
    return maxps(0.0f, __fadd_rn(__fmul_rn(onorm, onorm), __fsub_rn(sc.q_l2sqr, f)));
}

// FastScan sum of one vector (this lane) of block gb: sum over codebooks of
// LUT_u16[cb][nibble] (accumulate_hacc, fastscan_highacc.hpp:66-139, exact
// for dim <= 2048), then fast_of_sum.
__device__ __forceinline__ float fast_est(const SegDev &g, const uint16_t *__restrict__ lut, const SegScal &sc,
                                          int64_t gb, int lane, float onorm, float &ipx) {
    const int nc = g.dim / 64;
    const uint2 *cp = g.codes + (size_t)gb * nc * 32 + lane;
    int sum = 0;
#pragma unroll 4
    for (int c8 = 0; c8 < nc; ++c8) {
        const uint2 w = cp[(size_t)c8 * 32];
        const char *L = reinterpret_cast<const char *>(lut + c8 * 256);
        // byte k of these holds 2 x (high / low nibble of code byte k): the byte
        // offset of the entry within its 16-entry u16 table
        const uint32_t hx = (w.x >> 3) & 0x1E1E1E1Eu, lx = (w.x << 1) & 0x1E1E1E1Eu;
        const uint32_t hy = (w.y >> 3) & 0x1E1E1E1Eu, ly = (w.y << 1) & 0x1E1E1E1Eu;
#pragma unroll
        for (int j = 0; j < 4; ++j)
            sum += *reinterpret_cast<const uint16_t *>(L + (2 * j) * 32 + __byte_perm(hx, 0u, 0x4440u | j)) +
                   *reinterpret_cast<const uint16_t *>(L + (2 * j + 1) * 32 + __byte_perm(lx, 0u, 0x4440u | j));
#pragma unroll
        for (int j = 0; j < 4; ++j)
            sum += *reinterpret_cast<const uint16_t *>(L + (8 + 2 * j) * 32 + __byte_perm(hy, 0u, 0x4440u | j)) +
                   *reinterpret_cast<const uint16_t *>(L + (8 + 2 * j + 1) * 32 + __byte_perm(ly, 0u, 0x4440u | j));
    }
    return fast_of_sum(sc, sum, onorm, ipx);
}

__device__ __forceinline__ float vars_est(const SegScal &sc, float onorm) {
    return maxps(0.0f, __fadd_rn(__fmul_rn(onorm, onorm), sc.vfac));
}

// ResultPool::insert / distk (utils/pool.hpp:17-49), L2
__device__ __forceinline__ void pool_insert(uint32_t *ids, float *d, int &size, int cap, uint32_t u, float dist) {
    if (size == cap && dist > d[size - 1]) return;
    int lo = 0, len = size;
    while (len > 1) {
        const int half = len >> 1;
        len -= half;
        lo += (d[lo + half - 1] < dist) * half;
    }
    if (lo < size && d[lo] < dist) lo++;
    for (int i = size; i > lo; --i) {
        ids[i] = ids[i - 1];
        d[i] = d[i - 1];
    }
    ids[lo] = u;
    d[lo] = dist;
    size += (size < cap);
}

// Prune bounds and rotated queries (saq_estimator.hpp:28-48, caq_estimator.hpp:56-68)
// of a few queries, spread for latency: in Eigen's GEMV order the 16-input block
// sums of an output are independent (only their fold runs in block order), so a
// CTA takes 32 outputs of one segment for up to kQprepFewQ queries, its warps
// compute the block sums (lane = output; the block's 16 matrix elements are loaded
// at once and serve every query), and the sums are folded in order.  The prune
// bounds come from the CTA of the first 32 outputs.  Bound by one pass of load
// latency: one query of 960 dimensions 11.6 us (62 us with the block's elements
// loaded one after the other), 37 of segments (64, 320, 640) 11.2 us (88 us).
constexpr int kQprepOut = 32;
constexpr int kQprepFewQ = 8;
constexpr int kQprepFewThreads = 512;
__host__ __device__ inline size_t qprep_few_smem(int dim, int nq) {
    const int blocks = dim < 128 ? 1 : dim / 16;
    return 4 * (size_t)nq * (dim + (size_t)blocks * kQprepOut);
}
__global__ void __launch_bounds__(kQprepFewThreads) k_qprep_few(DevIndexView ix, const float *__restrict__ q, int nq,
                                                                float m, float *__restrict__ qrot,
                                                                float *__restrict__ prune) {
    extern __shared__ __align__(16) float qsm[];  // [queries][dim], then [block][queries][32] block sums
    const int s = blockIdx.y, q0 = blockIdx.z * kQprepFewQ, nqt = min(kQprepFewQ, nq - q0);
    const SegDev &g = ix.seg[s];
    const int dim = g.dim, qoff = g.qoff, o0 = blockIdx.x * kQprepOut;
    if (o0 >= dim) return;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nw = kQprepFewThreads / 32, i = o0 + lane;
    const int nbk = dim < 128 ? 1 : dim / 16;
    float *cq = qsm, *part = qsm + nqt * dim;
    for (int e = threadIdx.x; e < nqt * dim; e += kQprepFewThreads) {
        const int t = e / dim, gi = qoff + e - t * dim;
        cq[e] = gi < ix.D ? q[(size_t)(q0 + t) * ix.D + gi] : 0.0f;
    }
    __syncthreads();
    if (g.P) {
        if (dim < 128) {  // one chain of `dim` inputs: a warp per query
            for (int t = warp; t < nqt; t += nw) {
                float c = 0.0f;
#pragma unroll 16
                for (int j = 0; j < dim; ++j) c = fmaf(g.P[(size_t)j * dim + i], cq[t * dim + j], c);
                part[t * kQprepOut + lane] = c;
            }
        } else {
            for (int b = warp; b < nbk; b += nw) {
                float p[16];
#pragma unroll
                for (int j = 0; j < 16; ++j) p[j] = g.P[(size_t)(16 * b + j) * dim + i];
#pragma unroll 2
                for (int t = 0; t < nqt; ++t) {
                    const float4 *x = reinterpret_cast<const float4 *>(cq + t * dim + 16 * b);
                    float c = 0.0f;
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        const float4 v = x[j];
                        c = fmaf(p[4 * j], v.x, c);
                        c = fmaf(p[4 * j + 1], v.y, c);
                        c = fmaf(p[4 * j + 2], v.z, c);
                        c = fmaf(p[4 * j + 3], v.w, c);
                    }
                    part[(b * nqt + t) * kQprepOut + lane] = c;
                }
            }
        }
    }
    if (blockIdx.x == 0)
        for (int t = warp; t < nqt; t += nw) {
            const float v = prune_bound(ix, g, m, [&](int e) { return cq[t * dim + e]; });
            if (lane == 0) prune[(size_t)(q0 + t) * ix.S + s] = v;
        }
    __syncthreads();
    for (int t = warp; t < nqt; t += nw) {
        float res = 0.0f;
        if (g.P) {
#pragma unroll 8
            for (int b = 0; b < nbk; ++b) res = __fadd_rn(part[(b * nqt + t) * kQprepOut + lane], res);
        } else {
            res = cq[t * dim + i];
        }
        qrot[(size_t)(q0 + t) * ix.Dtot + qoff + i] = res;
    }
}

// The same for a batch: tiles of 128 queries x 64 outputs (rotate_tile), grid
// (outputs, segment, queries); the prune bounds in a kernel of their own (a warp
// per query and segment).  2,048 queries of 1,536 dimensions: 615 us with 16
// queries x 256 outputs per CTA, one thread per output; 226 us
// now, 16 us the bounds.
__global__ void __launch_bounds__(kRotThreads, 2) k_qprep_tiled(DevIndexView ix, const float *__restrict__ q, int nq,
                                                                int vec, float *__restrict__ qrot) {
    const SegDev &g = ix.seg[blockIdx.y];
    const int dim = g.dim, qoff = g.qoff;
    if ((int)blockIdx.x * kRotN >= dim) return;
    auto load4 = [&](int64_t v, int j) {
        float4 r = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        const int gi = qoff + j;
        if (v < nq) {
            const float *x = q + (size_t)v * ix.D + gi;
            if (vec && gi + 3 < ix.D) r = *reinterpret_cast<const float4 *>(x);
            else r = make_float4(gi < ix.D ? x[0] : 0.0f, gi + 1 < ix.D ? x[1] : 0.0f, gi + 2 < ix.D ? x[2] : 0.0f,
                                 gi + 3 < ix.D ? x[3] : 0.0f);
        }
        return r;
    };
    if (!g.P) {  // no rotation: the padded slice itself
        const int64_t v0 = (int64_t)blockIdx.z * kRotM;
        for (int e = threadIdx.x; e < kRotM * kRotN / 4; e += kRotThreads) {
            const int64_t v = v0 + e / (kRotN / 4);
            const int j = blockIdx.x * kRotN + e % (kRotN / 4) * 4;
            if (v < nq) *reinterpret_cast<float4 *>(qrot + v * ix.Dtot + qoff + j) = load4(v, j);
        }
        return;
    }
    rotate_tile(dim, g.P, (int64_t)blockIdx.z * kRotM, blockIdx.x * kRotN, load4,
                [&](int64_t v, int o, float (&r)[8][4]) {
#pragma unroll
                    for (int i = 0; i < 8; ++i)
                        if (v + i < nq)
                            *reinterpret_cast<float4 *>(qrot + (v + i) * ix.Dtot + qoff + o) =
                                make_float4(r[i][0], r[i][1], r[i][2], r[i][3]);
                });
}
__global__ void __launch_bounds__(256) k_prune_bounds(DevIndexView ix, const float *__restrict__ q, int nq, float m,
                                                      float *__restrict__ prune) {
    const int64_t w = (int64_t)blockIdx.x * 8 + (threadIdx.x >> 5);
    if (w >= (int64_t)nq * ix.S) return;
    const int64_t qi = w / ix.S;
    const int s = (int)(w - qi * ix.S);
    const SegDev &g = ix.seg[s];
    const float *x = q + qi * ix.D + g.qoff;
    const int n = ix.D - g.qoff;
    const float v = prune_bound(ix, g, m, [&](int i) { return i < n ? x[i] : 0.0f; });
    if ((threadIdx.x & 31) == 0) prune[w] = v;
}

// ------------------------------------------------------------------ scan
struct ScanSmem {
    // laid out in dynamic shared memory by scan_smem_layout()
    uint16_t *lut;
    float *qres;
    SegScal *scal;
    float *cd, *ipx, *part, *cur, *stage;
    uint32_t *cmask;
    int *nstage;
    int *sblk;        // block of the cluster in each slot of the tile
    uint32_t *pool_id;
    float *pool_d;
    uint32_t *mm;     // per segment LUT min / max keys
    uint8_t *xbuf;    // per half-warp ex-code staging
    int xstride;
};

__host__ __device__ inline size_t align16(size_t x) { return (x + 15) & ~size_t(15); }

__host__ __device__ inline size_t scan_smem_bytes(int Dtot, int S, int topk, int xstride) {
    size_t b = 0;
    b += align16(sizeof(uint32_t) * 2 * S);
    b += align16((size_t)2 * kScanWarps * xstride);
    b += align16(sizeof(uint16_t) * 4 * (size_t)Dtot);
    b += align16(sizeof(float) * Dtot);
    b += align16(sizeof(SegScal) * S);
    b += 2 * align16(sizeof(float) * kTileB * S * 32);  // cd (= part), ipx
    b += align16(sizeof(float) * kTileB * 32);          // cur
    b += align16(sizeof(float) * kTileB * (S + 1));     // stage minima
    b += align16(sizeof(uint32_t) * kTileB);
    b += 2 * align16(sizeof(int) * kTileB);             // nstage, sblk
    b += align16(sizeof(uint32_t) * (topk + 1));
    b += align16(sizeof(float) * (topk + 1));
    return b;
}

__device__ ScanSmem scan_smem_layout(char *base, int Dtot, int S, int topk, int xstride) {
    ScanSmem s;
    size_t o = 0;
    s.mm = (uint32_t *)(base + o);
    o += align16(sizeof(uint32_t) * 2 * S);
    s.xbuf = (uint8_t *)(base + o);
    s.xstride = xstride;
    o += align16((size_t)2 * kScanWarps * xstride);
    s.lut = (uint16_t *)(base + o);
    o += align16(sizeof(uint16_t) * 4 * (size_t)Dtot);
    s.qres = (float *)(base + o);
    o += align16(sizeof(float) * Dtot);
    s.scal = (SegScal *)(base + o);
    o += align16(sizeof(SegScal) * S);
    s.cd = (float *)(base + o);
    o += align16(sizeof(float) * kTileB * S * 32);
    s.ipx = (float *)(base + o);
    o += align16(sizeof(float) * kTileB * S * 32);
    // A candidate's partial replaces its estimate in place: the accurate pass
    // reads cd[i] and writes part[i] in the same thread, and nothing reads a
    // candidate's estimate afterwards (the replay and the split pass's records
    // read partials of candidate lanes only).
    s.part = s.cd;
    s.cur = (float *)(base + o);
    o += align16(sizeof(float) * kTileB * 32);
    s.stage = (float *)(base + o);
    o += align16(sizeof(float) * kTileB * (S + 1));
    s.cmask = (uint32_t *)(base + o);
    o += align16(sizeof(uint32_t) * kTileB);
    s.nstage = (int *)(base + o);
    o += align16(sizeof(int) * kTileB);
    s.sblk = (int *)(base + o);
    o += align16(sizeof(int) * kTileB);
    s.pool_id = (uint32_t *)(base + o);
    o += align16(sizeof(uint32_t) * (topk + 1));
    s.pool_d = (float *)(base + o);
    return s;
}

// ---- pieces of Lut::prepare (lut.hpp:60-87) shared by the in-CTA preparation
// (prepare_cluster) and the batched one (k_lut), so both give the same bits.
// The quantizer's scale from the segment's LUT min / max keys.
__device__ __forceinline__ void seg_quant_scalars(uint32_t kmin, uint32_t kmax, SegScal &sc) {
    const float vl = key_to_float(kmin), vr = key_to_float(kmax);
    const float delta = (float)__ddiv_rn((double)__fsub_rn(vr, vl), 65536.0 - 0.01);
    sc.delta = delta;
    sc.rdelta = __frcp_rn(delta);
    sc.vl = vl;
}

// compFastIP's epilogue constants (sum_q, q_l2sqr, vl and delta already set).
__device__ __forceinline__ void seg_epilogue_scalars(const SegDev &g, float prune_s, SegScal &sc) {
    const int ncb = g.dim / 4;
    sc.sum_vl = (float)__dmul_rn(__dadd_rn((double)sc.vl, __dmul_rn(0.5, (double)sc.delta)), (double)(float)ncb);
    sc.q_l2norm = sqrtf(sc.q_l2sqr);
    sc.c1 = (float)__dsub_rn(__dmul_rn(0.5, (double)sc.sum_q), (double)__fmul_rn(0.58f, sc.q_l2norm));
    sc.c2 = g.c2;
    sc.vfac = __fsub_rn(sc.q_l2sqr, __fmul_rn(2.0f, prune_s));
}

// The 16 u16 entries of one codebook (4 residual dims at qq), 32 bytes at dst.
__device__ __forceinline__ void quant_codebook(const float *qq, float vl, float delta, float rd, uint16_t *dst) {
    float t[16];
    lut_entries(qq, t);
    uint32_t packed[8];
    if (lut_quant_ok(delta)) {  // the segment's: uniform over most of a warp
#pragma unroll
        for (int j = 0; j < 16; j += 2)
            packed[j / 2] = lut_quant(__fsub_rn(t[j], vl), delta, rd) | lut_quant(__fsub_rn(t[j + 1], vl), delta, rd) << 16;
    } else {
#pragma unroll
        for (int j = 0; j < 16; j += 2) {
            const uint32_t a = (uint16_t)(int)__fdiv_rn(__fsub_rn(t[j], vl), delta);
            const uint32_t b = (uint16_t)(int)__fdiv_rn(__fsub_rn(t[j + 1], vl), delta);
            packed[j / 2] = a | (b << 16);
        }
    }
    uint4 *d = reinterpret_cast<uint4 *>(dst);
    d[0] = make_uint4(packed[0], packed[1], packed[2], packed[3]);
    d[1] = make_uint4(packed[4], packed[5], packed[6], packed[7]);
}

// Min and max keys of one codebook's float entries.  An entry adds its dims in a
// fixed order (lut_entries), and rounding is monotone: leaving out a dim that is not
// negative never raises the sum, adding a negative one never does either, so the
// smallest entry is the one of the negative dims and the largest that of the positive.
__device__ __forceinline__ void codebook_keys(const float4 &q, uint32_t &kmin, uint32_t &kmax) {
    float lo = 0.0f, hi = 0.0f;
    lo = __fadd_rn(lo, fminf(q.x, 0.0f));
    hi = __fadd_rn(hi, fmaxf(q.x, 0.0f));
    lo = __fadd_rn(lo, fminf(q.y, 0.0f));
    hi = __fadd_rn(hi, fmaxf(q.y, 0.0f));
    lo = __fadd_rn(lo, fminf(q.z, 0.0f));
    hi = __fadd_rn(hi, fmaxf(q.z, 0.0f));
    lo = __fadd_rn(lo, fminf(q.w, 0.0f));
    hi = __fadd_rn(hi, fmaxf(q.w, 0.0f));
    kmin = fkey(lo);
    kmax = fkey(hi);
}

// One group of 64 residuals into ex order, by a whole warp.
__device__ __forceinline__ void ex_reorder(float *x) {
    const int lane = threadIdx.x & 31;
    const float a = x[lane], b = x[lane + 32];
    __syncwarp();
    x[ex_order(lane)] = a;
    x[ex_order(lane + 32)] = b;
    __syncwarp();
}

// The first part of Lut::prepare (lut.hpp:60-87) for every segment of cluster c,
// spread over the whole CTA: the residual query (natural order, sm.qres), its
// Eigen-order sum and squared norm, the float LUT's min / max, and from them delta =
// (max-min)/(65536-0.01) in double and the epilogue constants of compFastIP (these
// are in place after the caller's next barrier).
// t_first > 0: only threads [t_first, blockDim.x) take part (whole warps),
// synchronising on named barrier `bar` instead of __syncthreads.
__device__ __forceinline__ void cta_sync(int bar, int nt) {
    if (bar) asm volatile("bar.sync %0, %1;" ::"r"(bar), "r"(nt) : "memory");
    else __syncthreads();
}
__device__ void prepare_scalars(const DevIndexView &ix, const float *__restrict__ qrot, const float *__restrict__ prune,
                                int c, ScanSmem &sm, int t_first = 0, int bar = 0) {
    const int tid = (int)threadIdx.x - t_first, nt = (int)blockDim.x - t_first, warp = tid >> 5, lane = tid & 31;
    const int S = ix.S;
    for (int i = tid; i < ix.Dtot; i += nt) {
        int s = 0;
        while (s + 1 < S && i >= ix.seg[s + 1].qoff) ++s;
        const SegDev &g = ix.seg[s];
        sm.qres[i] = __fsub_rn(qrot[i], g.cent[(size_t)c * g.dim + (i - g.qoff)]);
    }
    if (tid < S) {
        sm.mm[2 * tid] = 0xffffffffu;  // min key
        sm.mm[2 * tid + 1] = 0u;       // max key
    }
    cta_sync(bar, nt);
    for (int t = warp; t < 2 * S; t += nt / 32) {
        const int s = t >> 1;
        const float *qr = sm.qres + ix.seg[s].qoff;
        const float r = (t & 1) ? warp_eigen_sum(ix.seg[s].dim, [&](int i) { return __fmul_rn(qr[i], qr[i]); })
                                : warp_eigen_sum(ix.seg[s].dim, [&](int i) { return qr[i]; });
        if (lane == 0) {
            if (t & 1) sm.scal[s].q_l2sqr = r;
            else sm.scal[s].sum_q = r;
        }
    }
    const int ncb_all = ix.Dtot / 4;
    for (int cb0 = 0; cb0 < ncb_all; cb0 += nt) {  // warp-uniform trip count
        const int cb = cb0 + tid;
        int s = -1;
        uint32_t kmin = 0xffffffffu, kmax = 0u;
        if (cb < ncb_all) {
            s = 0;
            while (s + 1 < S && cb * 4 >= ix.seg[s + 1].qoff) ++s;
            codebook_keys(*reinterpret_cast<const float4 *>(sm.qres + cb * 4), kmin, kmax);
        }
        // one shared atomic per segment present in the warp
        const unsigned grp = __match_any_sync(kFull, s);
        kmin = __reduce_min_sync(grp, kmin);
        kmax = __reduce_max_sync(grp, kmax);
        if (s >= 0 && lane == __ffs(grp) - 1) {
            atomicMin(&sm.mm[2 * s], kmin);
            atomicMax(&sm.mm[2 * s + 1], kmax);
        }
    }
    cta_sync(bar, nt);
    if (tid < S) seg_quant_scalars(sm.mm[2 * tid], sm.mm[2 * tid + 1], sm.scal[tid]);  // what the quantizer needs
    cta_sync(bar, nt);
    if (tid >= nt - S) {  // the epilogue constants, beside what follows (the last warp's last lanes)
        const int s = tid - (nt - S);
        seg_epilogue_scalars(ix.seg[s], prune[s], sm.scal[s]);
    }
}

// Lut::prepare: prepare_scalars, then the u16 LUT trunc((entry-min)/delta); leaves the
// residual query in ex order (see excode_ip16).
__device__ void prepare_cluster(const DevIndexView &ix, const float *__restrict__ qrot, const float *__restrict__ prune,
                                int c, ScanSmem &sm, int t_first = 0, int bar = 0) {
    const int tid = (int)threadIdx.x - t_first, nt = (int)blockDim.x - t_first, warp = tid >> 5;
    const int S = ix.S, ncb_all = ix.Dtot / 4;
    prepare_scalars(ix, qrot, prune, c, sm, t_first, bar);
    for (int cb = tid; cb < ncb_all; cb += nt) {
        int s = 0;
        while (s + 1 < S && cb * 4 >= ix.seg[s + 1].qoff) ++s;
        const SegScal &sc = sm.scal[s];
        quant_codebook(sm.qres + cb * 4, sc.vl, sc.delta, sc.rdelta, sm.lut + cb * 16);
    }
    cta_sync(bar, nt);
    for (int g = warp; g < ix.Dtot / 64; g += nt / 32) ex_reorder(sm.qres + 64 * g);
    cta_sync(bar, nt);
}

// Output of the batched preparation (k_lut) for the first `slots` entries of the
// split list; other entries (and null members) build each cluster's state in
// the scan CTA.
struct Prepared {
    const uint16_t *lut = nullptr;
    const SegScal *scal = nullptr;
    int np_max = 0;
    int slots = 0;
    __device__ __forceinline__ bool has(int slot) const { return lut != nullptr && slot < slots; }
    __device__ __forceinline__ const uint16_t *lut_of(int slot, int p, int Dtot) const {
        return lut + ((size_t)slot * np_max + p) * 4 * Dtot;
    }
    __device__ __forceinline__ const SegScal *scal_of(int slot, int p, int S) const {
        return scal + ((size_t)slot * np_max + p) * S;
    }
};

// ---- batched preparation: the LUT and scalars of the (query, probe) pairs of
// the first `slots` entries of a list (the split pass's), one warp per pair.
// Pair i = slot * np_max + probe; its LUT is 4 * Dtot u16 at lut + i * 4 * Dtot
// (the layout of ScanSmem::lut), its scalars S SegScal at scal + i * S.  Work
// item w is list entry w / np_max (entries at or past *nlist are none) and
// probe w % np_max.  Pairs past a query's nprobe and pairs of empty clusters
// are not written (no scan reads them).
constexpr int kLutWarps = 8;
__global__ void __launch_bounds__(kLutWarps * 32) k_lut(DevIndexView ix, const uint32_t *__restrict__ probe,
                                                        QueryShape qsh, const int *__restrict__ qlist,
                                                        const int *__restrict__ nlist, int cap,
                                                        const uint8_t *__restrict__ skip,
                                                        const float *__restrict__ qrot_all,
                                                        const float *__restrict__ prune_all, uint16_t *__restrict__ lut,
                                                        SegScal *__restrict__ scal) {
    extern __shared__ __align__(16) float k_lut_qres[];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int64_t w = (int64_t)blockIdx.x * kLutWarps + warp;
    const int slot = (int)(w / qsh.np_max), p = (int)(w - (int64_t)slot * qsh.np_max);
    if (slot >= (qlist ? min(*nlist, cap) : cap)) return;  // whole warp
    const int qi = qlist ? qlist[slot] : slot;  // no list: every query, entry = query
    if (p >= qsh.np_of(qi) || (skip && skip[qi])) return;
    const int64_t pair = (int64_t)slot * qsh.np_max + p;
    const int c = (int)probe[(size_t)qi * qsh.np_max + p];
    if (ix.blk_off[c + 1] == ix.blk_off[c]) return;
    float *qres = k_lut_qres + (size_t)warp * ix.Dtot;
    const float *qrot = qrot_all + (size_t)qi * ix.Dtot;
    for (int s = 0; s < ix.S; ++s) {
        const SegDev &g = ix.seg[s];
        const float *cent = g.cent + (size_t)c * g.dim;
        for (int i = lane; i < g.dim; i += 32) qres[g.qoff + i] = __fsub_rn(qrot[g.qoff + i], cent[i]);
    }
    __syncwarp();
    uint16_t *L = lut + pair * 4 * ix.Dtot;
    // segment s's sums and LUT min / max keys end in lane s, so the scalar steps
    // (FP64) of all segments run at once, one lane each
    SegScal sc;
    uint32_t my_min = 0xffffffffu, my_max = 0u;
    for (int s = 0; s < ix.S; ++s) {
        const SegDev &g = ix.seg[s];
        const float *qr = qres + g.qoff;
        const float sq = warp_eigen_sum(g.dim, [&](int i) { return qr[i]; });
        const float l2 = warp_eigen_sum(g.dim, [&](int i) { return __fmul_rn(qr[i], qr[i]); });
        const int cb0 = g.qoff / 4, ncb = g.dim / 4;
        uint32_t kmin = 0xffffffffu, kmax = 0u;
        for (int k = lane; k < ncb; k += 32) {
            uint32_t a, b;
            codebook_keys(*reinterpret_cast<const float4 *>(qres + (cb0 + k) * 4), a, b);
            kmin = min(kmin, a);
            kmax = max(kmax, b);
        }
        kmin = __reduce_min_sync(kFull, kmin);
        kmax = __reduce_max_sync(kFull, kmax);
        if (lane == s) {
            sc.sum_q = sq;
            sc.q_l2sqr = l2;
            my_min = kmin;
            my_max = kmax;
        }
    }
    if (lane < ix.S) seg_quant_scalars(my_min, my_max, sc);
    for (int s = 0; s < ix.S; ++s) {
        const SegDev &g = ix.seg[s];
        const float vl = __shfl_sync(kFull, sc.vl, s), delta = __shfl_sync(kFull, sc.delta, s),
                    rd = __shfl_sync(kFull, sc.rdelta, s);
        const int cb0 = g.qoff / 4, ncb = g.dim / 4;
        for (int k = lane; k < ncb; k += 32) quant_codebook(qres + (cb0 + k) * 4, vl, delta, rd, L + (cb0 + k) * 16);
    }
    if (lane < ix.S) {
        seg_epilogue_scalars(ix.seg[lane], prune_all[(size_t)qi * ix.S + lane], sc);
        scal[pair * ix.S + lane] = sc;
    }
}

// The prepared state of cluster c from k_lut's output (lut / scal: this
// pair's), and the residual query in ex order, into the CTA's shared memory.
__device__ void load_cluster(const DevIndexView &ix, const float *__restrict__ qrot, const uint16_t *__restrict__ lut,
                             const SegScal *__restrict__ scal, int c, ScanSmem &sm) {
    const int tid = threadIdx.x, nt = blockDim.x;
    const uint4 *src = reinterpret_cast<const uint4 *>(lut);
    uint4 *dst = reinterpret_cast<uint4 *>(sm.lut);
    for (int i = tid; i < ix.Dtot / 2; i += nt) dst[i] = src[i];  // 8 * Dtot bytes
    if (tid < ix.S) sm.scal[tid] = scal[tid];
    for (int s = 0; s < ix.S; ++s) {
        const SegDev &g = ix.seg[s];
        const float *cent = g.cent + (size_t)c * g.dim;
        for (int i = tid; i < g.dim; i += nt) sm.qres[g.qoff + ex_order(i)] = __fsub_rn(qrot[g.qoff + i], cent[i]);
    }
    __syncthreads();
}

// The block's minimum estimate for a pruning stage.  Only its comparisons with
// distk / tau are ever used; without NaN lanes every reduction order gives the
// same minimum (up to the sign of a zero, which no comparison sees), so a
// single key reduction stands in for the reference's min tree.  With a NaN lane
// the tree's order decides the result, and the tree runs.
__device__ __forceinline__ float block_min(float cur) {
    if (!__any_sync(kFull, cur != cur)) return key_to_float(__reduce_min_sync(kFull, fkey(cur)));
    return warp_min_tree(cur);
}

// Stage 0 of SAQSearcher::searchCluster (saq_searcher.hpp:87-97) for four
// consecutive blocks at once, by a warp: lane l takes vectors 4 (l & 7) .. + 3 of
// block l >> 3, whose variance bounds sum in the same order as block_estimates'.
// A block whose smallest bound exceeds `tau` (>= every distk it will meet) stops at
// this stage and has no effect; the others come back as four bits.  Most blocks of a
// probed cluster stop here (88% of those a 10M batch probes, 60% at nprobe up to 256),
// and 16 bytes per lane and segment decide four of them, so the scans look at 128
// blocks ahead and spend their tiles, LUT copies and barriers on the rest.
// gb: first block of the four (global); nvalid: blocks of them that exist; vf: the
// segments' q_l2sqr - 2 prune.  A block with a NaN bound stays (its minimum depends
// on the reference's reduction order).  U groups of four at a time, for more loads in
// flight.
constexpr int kQuad = 4;
template <int U>
__device__ __forceinline__ void quad_filter(const DevIndexView &ix, const float *const (&vf)[U], const int64_t (&gb)[U],
                                            const int (&nvalid)[U], float tau, uint32_t (&left)[U]) {
    const int lane = threadIdx.x & 31;
    float4 cur[U];
#pragma unroll
    for (int i = 0; i < U; ++i) cur[i] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
#pragma unroll 4
    for (int s = 0; s < ix.S; ++s)
#pragma unroll
        for (int i = 0; i < U; ++i) {
            float4 on = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            if ((lane >> 3) < nvalid[i]) on = *reinterpret_cast<const float4 *>(ix.seg[s].onorm + gb[i] * 32 + 4 * lane);
            const float v = vf[i][s];
            cur[i].x = __fadd_rn(cur[i].x, maxps(0.0f, __fadd_rn(__fmul_rn(on.x, on.x), v)));
            cur[i].y = __fadd_rn(cur[i].y, maxps(0.0f, __fadd_rn(__fmul_rn(on.y, on.y), v)));
            cur[i].z = __fadd_rn(cur[i].z, maxps(0.0f, __fadd_rn(__fmul_rn(on.z, on.z), v)));
            cur[i].w = __fadd_rn(cur[i].w, maxps(0.0f, __fadd_rn(__fmul_rn(on.w, on.w), v)));
        }
#pragma unroll
    for (int i = 0; i < U; ++i) {
        // left: some vector's bound is not above tau (or is a NaN)
        const bool keep = (lane >> 3) < nvalid[i] &&
                          !(cur[i].x > tau && cur[i].y > tau && cur[i].z > tau && cur[i].w > tau);
        const uint32_t b = __ballot_sync(kFull, keep);
        left[i] = ((b & 0xffu) ? 1u : 0u) | ((b & 0xff00u) ? 2u : 0u) | ((b & 0xff0000u) ? 4u : 0u) | ((b >> 24) ? 8u : 0u);
    }
}

// q_l2sqr - 2 prune of segment s and cluster c (seg_epilogue_scalars' vfac), by a warp.
__device__ __forceinline__ float stage0_scalar(const DevIndexView &ix, int s, int c, const float *__restrict__ qrot,
                                               const float *__restrict__ prune) {
    const SegDev &g = ix.seg[s];
    const float *cent = g.cent + (size_t)c * g.dim, *q = qrot + g.qoff;
    const float q2 = warp_eigen_sum(g.dim, [&](int i) {
        const float r = __fsub_rn(q[i], cent[i]);
        return __fmul_rn(r, r);
    });
    return __fsub_rn(q2, __fmul_rn(2.0f, prune[s]));
}

// Position of the n-th (from 0) set bit of a warp-uniform mask.
__device__ __forceinline__ int nth_bit(uint32_t m, int n) {
    const int lane = threadIdx.x & 31;
    return __ffs(__ballot_sync(kFull, ((m >> lane) & 1u) && __popc(m & ((1u << lane) - 1u)) == n)) - 1;
}

// Estimates of one block (this warp, lane = vector).  Fills cd/ipx for every
// segment and, for several segments, the running sum and the pruning-stage
// minima of SAQSearcher::searchCluster steps 1-2 (saq_searcher.hpp:87-132).
// Like the reference, it stops at the first stage whose minimum exceeds the
// bound `tau` (>= every distk the block will meet): such a block has no
// candidate lanes, so the later segments' estimates would never be read.
__device__ void block_estimates(const DevIndexView &ix, int64_t gb, ScanSmem &sm, int w, int lane, float tau) {
    const int S = ix.S;
    if (S == 1) {
        const SegDev &g = ix.seg[0];
        const float on = g.onorm[gb * 32 + lane];
        float ipx = 0.0f, est;
        if (g.bits) est = fast_est(g, sm.lut, sm.scal[0], gb, lane, on, ipx);
        else est = vars_est(sm.scal[0], on);
        sm.cd[w * 32 + lane] = est;
        sm.ipx[w * 32 + lane] = ipx;
        sm.cur[w * 32 + lane] = est;
        return;
    }
    float cur = 0.0f;
    for (int s = 0; s < S; ++s) {
        const float v = vars_est(sm.scal[s], ix.seg[s].onorm[gb * 32 + lane]);
        sm.cd[(w * S + s) * 32 + lane] = v;
        sm.ipx[(w * S + s) * 32 + lane] = 0.0f;
        cur = __fadd_rn(cur, v);
    }
    int k = 0;
    float mi = block_min(cur);
    if (lane == 0) sm.stage[w * (S + 1) + k] = mi;
    ++k;
    for (int s = 0; s < S && !(mi > tau); ++s) {  // mi is warp-uniform
        const SegDev &g = ix.seg[s];
        if (!g.bits) continue;
        const float on = g.onorm[gb * 32 + lane];
        cur = __fsub_rn(cur, sm.cd[(w * S + s) * 32 + lane]);
        float ipx;
        const float f = fast_est(g, sm.lut + 4 * g.qoff, sm.scal[s], gb, lane, on, ipx);
        sm.cd[(w * S + s) * 32 + lane] = f;
        sm.ipx[(w * S + s) * 32 + lane] = ipx;
        cur = __fadd_rn(cur, f);
        mi = block_min(cur);
        if (lane == 0) sm.stage[w * (S + 1) + k] = mi;
        ++k;
    }
    if (lane == 0) sm.nstage[w] = k;
    sm.cur[w * 32 + lane] = cur;
}

// Largest stage minimum (NaN-free ones; NaN when all are NaN or n == 0):
// stages_pass(st, n, tau) == !(stage_max(st, n) > tau).
__device__ __forceinline__ float stage_max(const float *st, int n) {
    float m = __int_as_float(0x7fffffff);
    for (int i = 0; i < n; ++i) m = fmaxf(m, st[i]);
    return m;
}

__device__ __forceinline__ bool stages_pass(const float *st, int n, float tau) {
    for (int i = 0; i < n; ++i)
        if (st[i] > tau) return false;
    return true;
}

// Steps 1-3 of a tile of ng blocks of one cluster (at most kTileB): estimates,
// candidate masks under `tau`, and the accurate distances (multi-segment: accurate
// - estimate per segment) of every candidate lane.  Slot i holds block blk(i) of the
// cluster (called by whole warps, blk ascending; also left in sm.sblk).  Ends with the
// partials in sm.part and the masks in sm.cmask.
// The threads [tbase, tbase + nthr) take part (whole warps; a tile then has at
// most nthr / 32 * kBlocksPerWarp slots); they synchronise on __syncthreads when
// barid is 0, else on the named barrier barid.
// kOne: the index has one segment (a form of its own, so that neither holds the other's
// registers).
template <bool kOne = false, class Blk>
__device__ __forceinline__ void tile_candidates(const DevIndexView &ix, ScanSmem &sm, int64_t b0, int64_t v0, int nb, int n, int ng,
                                Blk blk, float tau, int tbase = 0, int nthr = kScanThreads, int barid = 0) {
    const int S = kOne ? 1 : ix.S, tid = (int)threadIdx.x - tbase, w = tid >> 5, lane = tid & 31;
    const int nwarps = nthr >> 5, nslots = nwarps * kBlocksPerWarp;
    auto sync = [&]() {
        if (barid) asm volatile("bar.sync %0, %1;" ::"r"(barid), "r"(nthr) : "memory");
        else __syncthreads();
    };
    // One wide segment: the next block's codes into L1 ahead of their use, a line of 128
    // bytes per lane (256 queries of 1,536 dimensions over equal clusters, L2 cold: 0.597 ms,
    // 0.622 without this and without the form of its own; 768 dimensions would lose 1-3% by
    // it, several segments up to 8%).
    const bool pull = kOne && ix.seg[0].dim >= kPullDim;
    auto pull_codes = [&](int b) {
        const SegDev &g = ix.seg[0];
        const int lines = g.bits ? g.dim / 64 * 2 : 0;
        const char *p = reinterpret_cast<const char *>(g.codes) + (size_t)(b0 + b) * lines * 128;
        for (int l = lane; l < lines; l += 32) asm volatile("prefetch.global.L1 [%0];" ::"l"(p + l * 128));
    };
    if (pull && w < ng) pull_codes(blk(w));
#pragma unroll 1
    for (int slot = w; slot < nslots; slot += nwarps) {
        if (slot >= ng) {
            if (lane == 0) sm.cmask[slot] = 0;
            continue;
        }
        const int b = blk(slot);
        if (pull && slot + nwarps < ng) pull_codes(blk(slot + nwarps));
        block_estimates(ix, b0 + b, sm, slot, lane, tau);
        // the mask reads only what this warp's estimates wrote (the slot's cd, cur,
        // stage and nstage rows): a warp barrier orders them
        __syncwarp();
        bool cand;
        if (S == 1) {
            const int cnp = (b == nb - 1) ? (n % 32) : 32;  // scanCluster's last-block count (saq_searcher.hpp:186)
            cand = lane < cnp && sm.cd[slot * 32 + lane] < tau;
        } else {
            cand = stages_pass(sm.stage + slot * (S + 1), sm.nstage[slot], tau) && sm.cur[slot * 32 + lane] < tau &&
                   (b * 32 + lane) < n;
        }
        const uint32_t m = __ballot_sync(kFull, cand);
        if (lane == 0) {
            sm.cmask[slot] = m;
            sm.sblk[slot] = b;
        }
        if (cand) {  // pull the candidate's ex-code rows, factors and id into L1 ahead of their use
            const int64_t gv = v0 + (int64_t)b * 32 + lane;
            asm volatile("prefetch.global.L1 [%0];" ::"l"(ix.ids + gv));
            for (int s = 0; s < S; ++s) {
                const SegDev &g = ix.seg[s];
                asm volatile("prefetch.global.L1 [%0];" ::"l"(g.exfac + gv));
                if (g.bits > 1) {
                    const uint8_t *row = g.lcode + (size_t)gv * g.lstride;
                    for (int o = 0; o < g.lstride; o += 128) asm volatile("prefetch.global.L1 [%0];" ::"l"(row + o));
                }
            }
        }
    }
    sync();
    // Accurate distances.  Few candidates (at most kItemCands, or kItemCandsSegs): work
    // items of two candidates of one segment, a half-warp each (excode_ip16), the widest
    // segments first; a warp takes every nwarps-th.  More: one thread per (candidate,
    // segment) (excode_ip_thread), the tasks of a segment from a warp boundary on, which
    // takes half the instructions.  The lines lie where the two cross.  One segment (a
    // single warp's tasks, each a chain over every dimension): 256 queries of 1,536
    // dimensions, about 13 candidates a tile, 1.20 ms with half-warps up to 16 candidates,
    // 1.34 up to 8, 1.63 without.  Several: 4,000 queries of an anisotropic 400,000 x 1024
    // index, many candidates, 11.8 / 12.0 / 12.1 / 12.3 / 12.6 ms with half-warps up to 0 /
    // 4 / 6 / 8 / 12, 1,500 of Zipf clusters of that size, few, 4.13 / 3.97 / 3.96 / 3.89 / 3.85.
    // The FP64 step of the distance (accurate_dist) would cost a warp's issue for two
    // lanes, so lane 2i, 2i + 1 keep the products of the warp's i-th item and up to 32
    // of them take that step together.
    const uint32_t my_mask = lane < nslots ? sm.cmask[lane] : 0u;  // lane i: slot i
    int incl = __popc(my_mask);
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(kFull, incl, o);
        if (lane >= o) incl += y;
    }
    const int ncand = __shfl_sync(kFull, incl, 31);
    // the r-th candidate of the tile, as slot * 32 + lane of its block
    auto locate = [&](int r) {
        const int slot = __popc(__ballot_sync(kFull, incl <= r));  // lanes past the last slot hold ncand > r
        const uint32_t m = __shfl_sync(kFull, my_mask, slot);
        const int nth = r - (__shfl_sync(kFull, incl, slot) - __popc(m));
        const uint32_t hit = __ballot_sync(kFull, ((m >> lane) & 1u) && __popc(m & ((1u << lane) - 1u)) == nth);
        return slot * 32 + __ffs(hit) - 1;
    };
    if (ncand == 0 && !barid) return;  // the callers' next barrier orders the rest
    auto vec_of = [&](int c) { return v0 + (int64_t)sm.sblk[c >> 5] * 32 + (c & 31); };
    int held = 0, my_seg = -1, my_cand = 0;
    float my_ex = 0.0f;
    auto finish = [&]() {
        if (my_seg >= 0) {
            const int ww = my_cand >> 5, j = my_cand & 31;
            const int64_t gb = b0 + sm.sblk[ww], gv = vec_of(my_cand);
            const SegDev &g = ix.seg[my_seg];
            const SegScal &sc = sm.scal[my_seg];
            const int at = (ww * S + my_seg) * 32 + j;
            const float acc = accurate_dist(g.onorm[gb * 32 + j], sm.ipx[at], my_ex, g.exfac[gv].x, g.bits, sc.sum_q,
                                            sc.q_l2sqr);
            sm.part[at] = S == 1 ? acc : __fsub_rn(acc, sm.cd[at]);
        }
        my_seg = -1;
        held = 0;
        __syncwarp();
    };
    if (ncand > (S > 1 ? kItemCandsSegs : kItemCands)) {
        const int P = (ncand + 31) >> 5;  // warps' worth of tasks per segment
        for (int t = w; t < S * P; t += nwarps) {
            const int si = t / P, r0 = (t - si * P) * 32, s = S - 1 - si;
            // the candidates [r0, r0 + 32) of the tile, one per lane: from the slots they span
            int c = 0;
            {
                const int r = min(r0 + lane, ncand - 1);
                int slot = 0;
#pragma unroll
                for (int o = 8; o; o >>= 1) {  // slot: how many have incl <= r (incl ascends)
                    const int v = __shfl_sync(kFull, incl, slot + o - 1);
                    if (v <= r) slot += o;
                }
                uint32_t m = __shfl_sync(kFull, my_mask, slot);
                for (int i = r - (__shfl_sync(kFull, incl, slot) - __popc(m)); i > 0; --i) m &= m - 1;
                c = slot * 32 + __ffs(m) - 1;
            }
            if (r0 + lane < ncand) {
                const SegDev &g = ix.seg[s];
                my_seg = s;
                my_cand = c;
                my_ex = g.bits > 1 ? excode_ip_thread(sm.qres + g.qoff, g.lcode + (size_t)vec_of(c) * g.lstride, g.dim, g.bits - 1)
                                   : 0.0f;
            }
            finish();
        }
        sync();
        return;
    }
    const int pairs = (ncand + 1) >> 1;
    for (int it = w; it < S * pairs; it += nwarps) {
        const int si = it / pairs, r0 = 2 * (it - si * pairs), s = S - 1 - si;
        const int c0 = locate(r0), c1 = locate(min(r0 + 1, ncand - 1)), c = lane < 16 ? c0 : c1;
        const SegDev &g = ix.seg[s];
        float ex = 0.0f;
        if (g.bits > 1)
            ex = excode_ip16(sm.qres + g.qoff, g.lcode + (size_t)vec_of(c) * g.lstride, g.dim, g.bits - 1);
        const float e0 = __shfl_sync(kFull, ex, 0), e1 = __shfl_sync(kFull, ex, 16);
        if (lane == 2 * held) {
            my_seg = s;
            my_cand = c0;
            my_ex = e0;
        } else if (lane == 2 * held + 1 && r0 + 1 < ncand) {
            my_seg = s;
            my_cand = c1;
            my_ex = e1;
        }
        if (++held == 16) finish();
    }
    if (held) finish();
    sync();
}

// The reference's sequential decisions for one block (single thread):
// scanCluster's mask-then-insert (saq_searcher.hpp:185-208) or
// searchCluster's stage checks and per-lane partial sums (saq_searcher.hpp:87-160).
// cur: fast estimate (one segment) or running sum; part: [S][32] partials.
__device__ __forceinline__ void replay_block(int S, int n, int nb, int bb, const float *cur, const float *stage,
                                             int nstage, const float *part, uint32_t cm, const uint32_t *ids_v0,
                                             uint32_t *pid, float *pd, int &sz, int topk, float &dk, int *err,
                                             unsigned long long &c_rr) {
    // Only candidate lanes (cm) can pass: every other lane's estimate is >= the
    // tile-start distk >= dk, or lies past the cluster's end.
    (void)n;
    (void)nb;
    (void)err;
    if (S == 1) {
        uint32_t mask = 0;  // scanCluster computes the mask once, at the block's start
        for (uint32_t m = cm; m; m &= m - 1) {
            const int j = __ffs(m) - 1;
            mask |= (uint32_t)(cur[j] < dk) << j;
        }
        while (mask) {
            const int j = __ffs(mask) - 1;
            mask &= mask - 1;
            ++c_rr;
            pool_insert(pid, pd, sz, topk, ids_v0[(int64_t)bb * 32 + j], part[j]);
            dk = sz == topk ? pd[sz - 1] : FLT_MAX;
        }
        return;
    }
    if (!cm || !stages_pass(stage, nstage, dk)) return;
    for (uint32_t m = cm; m; m &= m - 1) {
        const int j = __ffs(m) - 1;
        if (!(cur[j] < dk)) continue;
        ++c_rr;
        float acc = cur[j];
        for (int s = 0; s < S; ++s) {
            acc = __fadd_rn(acc, part[s * 32 + j]);
            if (acc >= dk) break;
        }
        pool_insert(pid, pd, sz, topk, ids_v0[(int64_t)bb * 32 + j], acc);
        dk = sz == topk ? pd[sz - 1] : FLT_MAX;
    }
}

// ResultPool::insert (utils/pool.hpp:17-49) by a whole warp on the pool in
// shared memory: the insert position is the number of entries below `dist`,
// which is what the reference's lower-bound search returns on a sorted pool;
// when `dist` or an entry is NaN (no order) lane 0 runs that search itself.
__device__ __forceinline__ void pool_insert_warp(uint32_t *ids, float *d, int &size, int cap, uint32_t u, float dist) {
    const int lane = threadIdx.x & 31;
    if (size == cap && dist > d[size - 1]) return;
    int lo = 0;
    bool nan = dist != dist;
    for (int i0 = 0; i0 < size; i0 += 32) {
        const int i = i0 + lane;
        const float v = i < size ? d[i] : 0.0f;
        lo += __popc(__ballot_sync(kFull, i < size && v < dist));
        nan = __any_sync(kFull, nan || v != v);
    }
    if (nan) {
        int sz = size;
        if (lane == 0) pool_insert(ids, d, sz, cap, u, dist);
        __syncwarp();
        size = __shfl_sync(kFull, sz, 0);
        return;
    }
    // entries [lo, size) move up one (entry size - 1 lands in the spare slot when full), top chunk first
    for (int i0 = (size >> 5) << 5; i0 >= ((lo + 1) >> 5) << 5; i0 -= 32) {
        const int i = i0 + lane;
        const bool mv = i > lo && i <= size;
        uint32_t pi = 0;
        float pv = 0.0f;
        if (mv) {
            pi = ids[i - 1];
            pv = d[i - 1];
        }
        __syncwarp();
        if (mv) {
            ids[i] = pi;
            d[i] = pv;
        }
        __syncwarp();
    }
    if (lane == 0) {
        ids[lo] = u;
        d[lo] = dist;
    }
    __syncwarp();
    size += size < cap;
}

// The reference's decisions for one block (saq_searcher.hpp:87-160 for several
// segments, scanCluster's mask-then-insert, saq_searcher.hpp:185-208, for one),
// taken by a whole warp.  distk changes only when an insert is accepted, so
// every lane evaluates its own insert under the current distk at once; the
// first accepted lane (in lane order) is inserted, the lanes before it were
// rejected under that same distk, and the lanes after it are evaluated again.
// Rejected inserts thus cost no serial steps.  c_rr counts the lanes whose
// accurate distance the reference computes.
// smax: stage_max of the block's stage minima (several segments).
__device__ __forceinline__ void replay_block_warp(int S, int bb, const float *cur, float smax, const float *part,
                                                  uint32_t cm, const uint32_t *ids_v0, uint32_t *pid, float *pd,
                                                  int &sz, int topk, float &dk, unsigned long long &c_rr) {
    const int lane = threadIdx.x & 31;
    if (!cm) return;
    if (S > 1 && smax > dk) return;
    const bool in = (cm >> lane) & 1u;
    const float c = in ? cur[lane] : FLT_MAX;
    if (S == 1) {
        uint32_t rest = __ballot_sync(kFull, in && c < dk);  // the mask, at the block's start
        c_rr += __popc(rest);
        const float a = in ? part[lane] : FLT_MAX;
        while (rest) {
            const uint32_t ok = rest & __ballot_sync(kFull, !(sz == topk && a > dk));
            if (!ok) break;
            const int j = __ffs(ok) - 1;
            pool_insert_warp(pid, pd, sz, topk, ids_v0[(int64_t)bb * 32 + j], __shfl_sync(kFull, a, j));
            dk = sz == topk ? pd[sz - 1] : FLT_MAX;
            rest &= ~((2u << j) - 1u);
        }
        return;
    }
    uint32_t rest = __ballot_sync(kFull, in);
    while (rest) {
        const uint32_t pass = rest & __ballot_sync(kFull, c < dk);
        float acc = c;
        if ((pass >> lane) & 1u)
            for (int s = 0; s < S; ++s) {
                acc = __fadd_rn(acc, part[s * 32 + lane]);
                if (acc >= dk) break;
            }
        const uint32_t ok = pass & __ballot_sync(kFull, !(sz == topk && acc > dk));
        if (!ok) {
            c_rr += __popc(pass);
            break;
        }
        const int j = __ffs(ok) - 1;
        c_rr += __popc(pass & ((2u << j) - 1u));
        pool_insert_warp(pid, pd, sz, topk, ids_v0[(int64_t)bb * 32 + j], __shfl_sync(kFull, acc, j));
        dk = sz == topk ? pd[sz - 1] : FLT_MAX;
        rest &= ~((2u << j) - 1u);
    }
}

// ResultPool (utils/pool.hpp:17-49) of at most 32 kPer entries in a warp's registers,
// entry kPer lane + r in d[r] / u[r]; past the size FLT_MAX, so that the k-th entry is
// distk whether the pool is full or not.  An insert is a shift by one entry under a
// comparison per entry: the two shuffles of the shift do not wait for the value, and
// the one of the new distk ends it: 240 cycles.  (With ballots for the position, the size as
// a counter and the entries spread row by row: 37 queries with k = 100 1.66 ms, now
// 1.54; in shared memory, pool_insert_warp, over a thousand cycles an insert.)
constexpr int kRegPool = 128;  // largest k whose pool is held so
template <int kPer>
struct RegPool {
    float d[kPer], dk;
    uint32_t u[kPer];
    int cap;
    bool odd;  // an entry is not finite: replay_block_warp takes over
    __device__ __forceinline__ float kth() const {
        float x = d[0];
#pragma unroll
        for (int r = 1; r < kPer; ++r)
            if (r == (cap - 1) % kPer) x = d[r];
        return __shfl_sync(kFull, x, (cap - 1) / kPer);
    }
    __device__ __forceinline__ void load(const uint32_t *pid, const float *pd, int size, int topk) {
        const int lane = threadIdx.x & 31;
        cap = topk;
        bool bad = false;
#pragma unroll
        for (int r = 0; r < kPer; ++r) {
            const int e = kPer * lane + r;
            d[r] = e < size ? pd[e] : FLT_MAX;
            u[r] = e < size ? pid[e] : 0u;
            bad |= e < size && !(fabsf(d[r]) < FLT_MAX);
        }
        odd = __any_sync(kFull, bad);
        dk = kth();
    }
    __device__ __forceinline__ void store(uint32_t *pid, float *pd, int &size) const {
        const int lane = threadIdx.x & 31;
        int n = 0;
#pragma unroll
        for (int r = 0; r < kPer; ++r) {
            const int e = kPer * lane + r;
            const bool have = e < cap && d[r] < FLT_MAX;
            if (have) {
                pd[e] = d[r];
                pid[e] = u[r];
            }
            n += __popc(__ballot_sync(kFull, have));
        }
        size = n;
        __syncwarp();
    }
    // Inserts v (uniform, finite, accepted under dk) and updates dk.
    __device__ __forceinline__ void insert(uint32_t id, float v) {
        float pv = __shfl_up_sync(kFull, d[kPer - 1], 1);
        const uint32_t pu = __shfl_up_sync(kFull, u[kPer - 1], 1);
        if ((threadIdx.x & 31) == 0) pv = __int_as_float(0xff800000);
#pragma unroll
        for (int r = kPer - 1; r >= 0; --r) {
            const float prev = r ? d[r > 0 ? r - 1 : 0] : pv;
            const uint32_t prevu = r ? u[r > 0 ? r - 1 : 0] : pu;
            const bool keep = d[r] < v, put = prev < v;  // equal entries move up: the later one goes first
            d[r] = keep ? d[r] : put ? v : prev;
            u[r] = keep ? u[r] : put ? id : prevu;
        }
        dk = kth();
    }
};

// replay_block_warp on a pool in registers, for at most kRegSegs segments (ids: the
// block's 32 ids).  A lane's running sums are formed once and stay in registers: while
// the largest is below dk the reference's loop runs to the last one, which is inserted;
// otherwise it ends at the first sum >= dk, which is refused unless it equals dk.  Returns
// the lanes not decided: those of a block with a NaN or an infinity, or from the first
// lane with a sum that equals dk on (for replay_block_warp).  seen(dk): called after each insert.
constexpr int kRegSegs = 4;
template <int kPer, class Seen>
__device__ __forceinline__ uint32_t replay_block_regs(int S, const float *cur, float smax, const float *part, uint32_t cm,
                                                      const uint32_t *ids, RegPool<kPer> &P, Seen seen) {
    const int lane = threadIdx.x & 31;
    if (P.odd) return cm;
    if (!cm || (S > 1 && smax > P.dk)) return 0u;
    const bool in = (cm >> lane) & 1u;
    const uint32_t id = in ? ids[lane] : 0u;
    const float c = in ? cur[lane] : FLT_MAX;
    float sum[kRegSegs], top = 0.0f, last = c;
#pragma unroll
    for (int s = 0; s < kRegSegs; ++s) {
        if (in && s < S) {
            const float x = part[s * 32 + lane];
            last = S == 1 ? x : __fadd_rn(last, x);
        }
        sum[s] = last;  // past the last segment: the last sum again
        top = s == 0 ? last : fmaxf(top, last);
    }
    const float gate = fmaxf(c, top);
    // (a NaN stays one in the later sums, and a -inf stays or becomes one)
    if (__any_sync(kFull, in && !(gate < FLT_MAX && fabsf(last) < FLT_MAX))) return cm;
    if (S == 1) {
        uint32_t rest = __ballot_sync(kFull, in && c < P.dk);  // the mask, at the block's start
        while (rest) {
            const uint32_t ok = rest & __ballot_sync(kFull, last <= P.dk);
            if (!ok) break;
            const int j = __ffs(ok) - 1;
            P.insert(__shfl_sync(kFull, id, j), __shfl_sync(kFull, last, j));
            seen(P.dk);
            rest &= ~((2u << j) - 1u);
        }
        return 0u;
    }
    uint32_t rest = cm;
    while (rest) {
        const float dk = P.dk;
        bool tie = false;
#pragma unroll
        for (int s = 0; s < kRegSegs; ++s) tie |= sum[s] == dk;
        const uint32_t less = __ballot_sync(kFull, gate < dk), ties = rest & __ballot_sync(kFull, tie && c < dk);
        const uint32_t hit = (rest & less) | ties;
        if (!hit) break;
        const int j = __ffs(hit) - 1;
        if ((ties >> j) & 1u) return rest & ~((1u << j) - 1u);
        P.insert(__shfl_sync(kFull, id, j), __shfl_sync(kFull, last, j));
        seen(P.dk);
        rest &= ~((2u << j) - 1u);
    }
    return 0u;
}

// The reference's decisions for the nblk (<= 32) blocks of a tile, in order, by
// one warp: lane i first reads block i's candidate mask and (several segments)
// the largest of its stage minima, and a ballot keeps the blocks that can
// change the pool under the distk at the tile's start.  distk only decreases,
// so a block dropped here (no candidate lane, or a stage minimum above distk)
// would be skipped by the replay as well; the rest are replayed in order.  Slot i is
// block sblk[i] of the cluster (sblk null: block t0 + i).
// Returns the tile's candidate lanes (for the tally).
__device__ __forceinline__ unsigned replay_tile_warp(int S, int t0, const int *sblk, int nblk, const ScanSmem &v,
                                                     const uint32_t *ids_v0, uint32_t *pid, float *pd, int &sz, int topk,
                                                     float &dk, bool counted, unsigned long long &c_rr) {
    const int lane = threadIdx.x & 31;
    uint32_t cm = 0;
    float smax = 0.0f;
    if (lane < nblk) {
        cm = v.cmask[lane];
        if (S > 1 && cm) smax = stage_max(v.stage + lane * (S + 1), v.nstage[lane]);
    }
    uint32_t live = __ballot_sync(kFull, cm != 0 && !(S > 1 && smax > dk));
    if (!live) return __reduce_add_sync(kFull, __popc(cm));
    const int bb = lane < nblk ? (sblk ? sblk[lane] : t0 + lane) : 0;
    // blocks from the first of live on, lane by lane (m: the lanes of the first one left)
    const auto one = [&](uint32_t m, float sx) {
        const int ww = __ffs(live) - 1;
        replay_block_warp(S, __shfl_sync(kFull, bb, ww), v.cur + ww * 32, sx, v.part + ww * S * 32, m, ids_v0, pid, pd, sz, topk,
                          dk, c_rr);
        live &= live - 1;
    };
    auto in_regs = [&](auto &P) {
        while (live) {
            P.load(pid, pd, sz, topk);
            uint32_t m = 0u, left = 0u;
            float sx = 0.0f;
            for (; live; live &= live - 1) {
                const int ww = __ffs(live) - 1;
                m = __shfl_sync(kFull, cm, ww);
                sx = __shfl_sync(kFull, smax, ww);
                left = replay_block_regs(S, v.cur + ww * 32, sx, v.part + ww * S * 32, m,
                                         ids_v0 + (int64_t)__shfl_sync(kFull, bb, ww) * 32, P, [](float) {});
                if (left) break;
            }
            if (!P.odd) {
                P.store(pid, pd, sz);
                dk = P.dk;
            }
            if (left) one(left, left == m ? sx : -FLT_MAX);  // after an insert of the block its stage minima have passed
        }
    };
    if (counted || S > kRegSegs) {
    } else if (topk <= 32) {
        RegPool<1> P;
        in_regs(P);
    } else if (topk <= kRegPool) {
        RegPool<kRegPool / 32> P;
        in_regs(P);
    }
    while (live) one(__shfl_sync(kFull, cm, __ffs(live) - 1), __shfl_sync(kFull, smax, __ffs(live) - 1));
    return __reduce_add_sync(kFull, __popc(cm));
}

struct ScanTally {
    unsigned long long blocks = 0, vecs = 0, rr = 0, spec = 0;
    bool counted = false;  // counters are kept: every evaluated lane is counted
};

// Exact sequential scan of the np probes of one query, continuing the pool held
// in shared memory (pool_size / distk in shared memory).  A probed cluster's LUT comes
// from the batched preparation when `lut` is set (this query's pairs: probe p's at
// lut + p * 4 * Dtot, scal + p * S), else it is built here, when a block first needs it.
//
// The blocks of up to kHdrProbes probes form one sequence of groups of four, in scan order.  A pass looks at kPassQuads groups (one or
// a few until the pool is full and bounds distk: their every vector is a candidate): several segments, all warps filter them
// by stage 0 (quad_filter) under the pass's distk, then the blocks left are taken in
// order, up to kTileB of one cluster per tile; a probe with none left is not touched
// any further, nor its LUT.
constexpr int kHdrProbes = 32, kPassQuads = 32;
struct ProbeHdr {
    int c, nb, n, quads;
    int64_t b0, v0;
};
template <bool kOne>
__device__ __forceinline__ void scan_probes(const DevIndexView &ix, const uint32_t *__restrict__ probe, int np,
                            const float *__restrict__ qrot, const float *__restrict__ prune, int topk, ScanSmem &sm,
                            int &pool_size, float &distk, ScanTally &tl, const uint16_t *__restrict__ lut,
                            const SegScal *__restrict__ scal) {
    __shared__ ProbeHdr hdr[kHdrProbes];
    __shared__ float vf[kHdrProbes * kMaxSeg];
    __shared__ uint8_t nib[2][kPassQuads];  // blocks of each group left by the filter (two passes' worth)
    const int S = kOne ? 1 : ix.S, tid = threadIdx.x, w = tid >> 5, lane = tid & 31;
    int par = 0;
    for (int p0 = 0; p0 < np; p0 += kHdrProbes) {
        const int m = min(kHdrProbes, np - p0);
        __syncthreads();  // every thread is done with the headers
        if (tid < kHdrProbes) {
            ProbeHdr h{0, 0, 0, 0, 0, 0};
            if (lane < m) {
                h.c = (int)probe[p0 + lane];
                h.b0 = ix.blk_off[h.c];
                h.v0 = ix.vec_off[h.c];
                h.nb = (int)(ix.blk_off[h.c + 1] - h.b0);
                h.n = (int)(ix.vec_off[h.c + 1] - h.v0);
                h.quads = (h.nb + kQuad - 1) / kQuad;
            }
            hdr[lane] = h;
            tl.blocks += __reduce_add_sync(kFull, (unsigned)h.nb);
            tl.vecs += __reduce_add_sync(kFull, (unsigned)h.n);
        }
        __syncthreads();
        if (S > 1) {  // stage 0's scalars of every probe: the batched preparation's, or (Lut::prepare's q_l2sqr, in
                      // its order) a warp per probe
            if (scal) {
                for (int i = tid; i < m * S; i += kScanThreads)
                    if (hdr[i / S].nb) vf[i] = scal[(size_t)p0 * S + i].vfac;
            } else {
                for (int i = w; i < m; i += kScanWarps) {
                    if (!hdr[i].nb) continue;
                    for (int s = 0; s < S; ++s) {
                        const float v = stage0_scalar(ix, s, hdr[i].c, qrot, prune);
                        if (lane == 0) vf[i * S + s] = v;
                    }
                }
            }
            __syncthreads();
        }
        int loaded = -1;  // probe whose LUT is in place
        // lane i: groups of probes 0 .. i
        int qincl = hdr[lane].quads;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int y = __shfl_up_sync(kFull, qincl, o);
            if (lane >= o) qincl += y;
        }
        const int total = __shfl_sync(kFull, qincl, 31);
        for (int q0 = 0; q0 < total;) {
            const float tau = distk;
            const int nqd = min(pool_size == topk ? kPassQuads : min(4, (topk + 63) >> 6), total - q0);
            for (int qd = w; qd < nqd; qd += 2 * kScanWarps) {  // this warp's groups, two at a time
                const float *fv[2];
                int64_t gb[2];
                int nv[2];
                uint32_t left[2];
#pragma unroll
                for (int i = 0; i < 2; ++i) {
                    const int q = min(qd + i * kScanWarps, nqd - 1);
                    const int pi = __popc(__ballot_sync(kFull, qincl <= q0 + q));
                    const ProbeHdr &h = hdr[pi];
                    const int bq = kQuad * (q0 + q - (__shfl_sync(kFull, qincl, pi) - h.quads));
                    nv[i] = min(kQuad, h.nb - bq);
                    gb[i] = h.b0 + bq;
                    fv[i] = vf + pi * S;
                    left[i] = (1u << nv[i]) - 1u;
                }
                if (S > 1) quad_filter(ix, fv, gb, nv, tau, left);
                if (lane == 0) {
                    nib[par][qd] = (uint8_t)left[0];
                    if (qd + kScanWarps < nqd) nib[par][qd + kScanWarps] = (uint8_t)left[1];
                }
            }
            __syncthreads();
            // lane i: the pass's i-th group, its probe, and the blocks left up to it
            const uint32_t mine = lane < nqd ? nib[par][lane] : 0u;
            par ^= 1;
            int my_pi = 0;
            {
                const int x = q0 + min(lane, nqd - 1);
#pragma unroll
                for (int o = 16; o; o >>= 1) {
                    const int v = __shfl_sync(kFull, qincl, my_pi + o - 1);
                    if (v <= x) my_pi += o;
                }
            }
            int sincl = __popc(mine);
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int y = __shfl_up_sync(kFull, sincl, o);
                if (lane >= o) sincl += y;
            }
            const int nleft = __shfl_sync(kFull, sincl, 31);
            for (int k = 0; k < nleft;) {
                const int pi = __shfl_sync(kFull, my_pi, __popc(__ballot_sync(kFull, sincl <= k)));
                const int same = 31 - __clz(__ballot_sync(kFull, lane < nqd && my_pi == pi));  // its last group
                const int ng = min(kTileB, __shfl_sync(kFull, sincl, same) - k);
                const ProbeHdr h = hdr[pi];
                if (loaded != pi) {
                    if (lut) load_cluster(ix, qrot, lut + (size_t)(p0 + pi) * 4 * ix.Dtot, scal + (size_t)(p0 + pi) * S, h.c, sm);
                    else prepare_cluster(ix, qrot, prune, h.c, sm);
                    loaded = pi;
                }
                const int first = q0 - (__shfl_sync(kFull, qincl, pi) - h.quads);  // group of the probe at lane 0
                auto blk = [&](int slot) {
                    const int r = k + slot, g = __popc(__ballot_sync(kFull, sincl <= r));
                    const uint32_t gm = __shfl_sync(kFull, mine, g);
                    return kQuad * (first + g) + nth_bit(gm, r - (__shfl_sync(kFull, sincl, g) - __popc(gm)));
                };
                tile_candidates<kOne>(ix, sm, h.b0, h.v0, h.nb, h.n, ng, blk, distk);
                if (tid < 32) {
                    float dk = distk;
                    int sz = pool_size;
                    const unsigned nc = replay_tile_warp(S, 0, sm.sblk, ng, sm, ix.ids + h.v0, sm.pool_id, sm.pool_d, sz,
                                                         topk, dk, tl.counted, tl.rr);
                    if (tid == 0) {
                        tl.spec += nc;
                        distk = dk;
                        pool_size = sz;
                    }
                }
                __syncthreads();
                k += ng;
            }
            q0 += nqd;
        }
    }
}

__device__ void init_pool(ScanSmem &sm, int topk, int &pool_size, float &distk) {
    for (int i = threadIdx.x; i <= topk; i += blockDim.x) {
        sm.pool_id[i] = 0;
        sm.pool_d[i] = 0.0f;
    }
    if (threadIdx.x == 0) {
        pool_size = 0;
        distk = FLT_MAX;
    }
    __syncthreads();
}

__device__ void flush_tally(const ScanTally &tl, unsigned long long *counters) {
    if (threadIdx.x == 0 && counters) {
        atomicAdd(counters + 0, tl.blocks);
        atomicAdd(counters + 1, tl.vecs);
        atomicAdd(counters + 2, tl.rr);
        atomicAdd(counters + 3, tl.spec);
    }
}

// The pool as the reference returns it (unfilled slots id 0), then, for a
// row longer than this query's k, id 0 / FLT_MAX up to k_max.
__device__ void write_results(const ScanSmem &sm, int pool_size, int topk, int k_max, uint32_t *out_ids, float *out_d) {
    for (int i = threadIdx.x; i < k_max; i += blockDim.x) {
        out_ids[i] = i < topk ? sm.pool_id[i] : 0u;
        if (out_d) out_d[i] = i < pool_size && i < topk ? sm.pool_d[i] : FLT_MAX;
    }
}

// ------------------------------------------------------------------ warp-specialised scan
// k_scan with the replay overlapped: warp 0 replays tile t (the reference's
// decisions, the pool, distk) while warps 1-7 compute the estimates, masks and
// accurate distances of tile t + 1 into the other of two tile buffers.  The
// workers' bound for a tile is the distk the replay had published when the tile
// began, which is at least every distk the tile will meet in the replay (distk
// only shrinks), so the candidate lanes remain a superset and the answers are
// k_scan's.  Named barriers: 1 among the workers (224 threads); 2 + b "tile in
// buffer b written" (workers arrive, warp 0 waits); 4 + b "buffer b replayed"
// (warp 0 arrives, the workers wait before they overwrite it).
constexpr int kWsWorkers = kScanThreads - 32;
constexpr int kWsSlots = (kWsWorkers / 32) * kBlocksPerWarp;  // blocks per tile

struct WsTile {
    int64_t v0;  // first vector of the tile's cluster
    int t0;      // first block of the tile within the cluster
};

__host__ __device__ inline size_t ws_tile_bytes(int S) {
    return 3 * align16(sizeof(float) * kTileB * S * 32) + align16(sizeof(float) * kTileB * 32) +
           align16(sizeof(float) * kTileB * (S + 1)) + align16(sizeof(uint32_t) * kTileB) +
           2 * align16(sizeof(int) * kTileB);
}

__host__ __device__ inline size_t ws_smem_bytes(int Dtot, int S, int topk, int xstride) {
    return scan_smem_bytes(Dtot, S, topk, xstride) + ws_tile_bytes(S);
}

// The tile buffer `b` of a warp-specialised layout: buffer 0 is the base
// layout's, buffer 1 the arrays appended at `extra`.
__device__ __forceinline__ ScanSmem ws_view(const ScanSmem &sm, char *extra, int S, int b) {
    if (!b) return sm;
    ScanSmem v = sm;
    size_t o = 0;
    v.cd = (float *)(extra + o);
    o += align16(sizeof(float) * kTileB * S * 32);
    v.ipx = (float *)(extra + o);
    o += align16(sizeof(float) * kTileB * S * 32);
    v.part = (float *)(extra + o);
    o += align16(sizeof(float) * kTileB * S * 32);
    v.cur = (float *)(extra + o);
    o += align16(sizeof(float) * kTileB * 32);
    v.stage = (float *)(extra + o);
    o += align16(sizeof(float) * kTileB * (S + 1));
    v.cmask = (uint32_t *)(extra + o);
    o += align16(sizeof(uint32_t) * kTileB);
    v.nstage = (int *)(extra + o);
    o += align16(sizeof(int) * kTileB);
    v.sblk = (int *)(extra + o);
    return v;
}

__device__ __forceinline__ void named_sync(int id, int n) { asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(n) : "memory"); }
__device__ __forceinline__ void named_arrive(int id, int n) {
    asm volatile("bar.arrive %0, %1;" ::"r"(id), "r"(n) : "memory");
}

__global__ void __launch_bounds__(kScanThreads, kScanMinCtas) k_scan_ws(DevIndexView ix, const uint32_t *__restrict__ probe,
                                                          QueryShape qsh, const float *__restrict__ qrot_all,
                                                          const float *__restrict__ prune_all,
                                                          uint32_t *__restrict__ out_ids, float *__restrict__ out_d,
                                                          unsigned long long *__restrict__ counters, int xstride,
                                                          const uint8_t *__restrict__ deferred,
                                                          const int *__restrict__ order) {
    extern __shared__ __align__(16) char smem_raw[];
    const int qi = order ? order[blockIdx.x] : (int)blockIdx.x;
    if (deferred && deferred[qi]) return;  // answered by the split pass
    const int np = qsh.np_of(qi), topk = qsh.k_of(qi), S = ix.S, tid = threadIdx.x;
    ScanSmem sm = scan_smem_layout(smem_raw, ix.Dtot, S, qsh.k_max, xstride);
    char *extra = smem_raw + scan_smem_bytes(ix.Dtot, S, qsh.k_max, xstride);
    __shared__ WsTile meta[2];
    __shared__ int pool_size;
    __shared__ float distk;
    volatile float *vdistk = &distk;
    init_pool(sm, topk, pool_size, distk);
    const uint32_t *pr = probe + (size_t)qi * qsh.np_max;
    const float *qrot = qrot_all + (size_t)qi * ix.Dtot, *prune = prune_all + (size_t)qi * ix.S;
    int ntiles = 0;
    if (tid >= 32) {
        // ---- workers: LUTs, estimates, masks, accurate distances
        unsigned long long blocks = 0, vecs = 0;
        for (int p = 0; p < np; ++p) {
            const int c = (int)pr[p];
            const int64_t b0 = ix.blk_off[c], v0 = ix.vec_off[c];
            const int nb = (int)(ix.blk_off[c + 1] - b0), n = (int)(ix.vec_off[c + 1] - v0);
            blocks += nb;
            vecs += n;
            if (nb == 0) continue;
            prepare_cluster(ix, qrot, prune, c, sm, 32, 1);
            for (int t0 = 0; t0 < nb; t0 += kWsSlots, ++ntiles) {
                const int b = ntiles & 1;
                if (ntiles >= 2) named_sync(4 + b, kScanThreads);  // the replay of tile ntiles - 2 is done
                ScanSmem v = ws_view(sm, extra, S, b);
                if (tid == 32) meta[b] = WsTile{v0, t0};
                const float tau = __shfl_sync(kFull, *vdistk, 0);  // warp-uniform, as block_estimates wants
                tile_candidates(ix, v, b0, v0, nb, n, min(kWsSlots, nb - t0), [&](int slot) { return t0 + slot; }, tau, 32,
                                kWsWorkers, 1);
                __threadfence_block();
                named_arrive(2 + b, kScanThreads);
            }
        }
        for (int t = max(0, ntiles - 2); t < ntiles; ++t) named_sync(4 + (t & 1), kScanThreads);  // the last replays
        if (tid == 32 && counters) {
            atomicAdd(counters + 0, blocks);
            atomicAdd(counters + 1, vecs);
        }
    } else {
        // ---- warp 0: the reference's decisions, in order
        unsigned long long rr = 0, spec = 0;
        float dk = distk;
        int sz = pool_size;
        for (int p = 0; p < np; ++p) {
            const int c = (int)pr[p];
            const int nb = (int)(ix.blk_off[c + 1] - ix.blk_off[c]);
            for (int t0 = 0; t0 < nb; t0 += kWsSlots, ++ntiles) {
                const int b = ntiles & 1;
                named_sync(2 + b, kScanThreads);  // tile ntiles written
                const ScanSmem v = ws_view(sm, extra, S, b);
                const WsTile mt = meta[b];
                const unsigned nc = replay_tile_warp(S, mt.t0, nullptr, min(kWsSlots, nb - mt.t0), v, ix.ids + mt.v0,
                                                     sm.pool_id, sm.pool_d, sz, topk, dk, counters != nullptr, rr);
                if (tid == 0) {
                    spec += nc;
                    *vdistk = dk;
                    pool_size = sz;
                }
                __threadfence_block();
                __syncwarp();
                named_arrive(4 + b, kScanThreads);  // buffer b may be overwritten
            }
        }
        if (tid == 0 && counters) {
            atomicAdd(counters + 2, rr);
            atomicAdd(counters + 3, spec);
        }
    }
    __syncthreads();
    write_results(sm, pool_size, topk, qsh.k_max, out_ids + (size_t)qi * qsh.k_max,
                  out_d ? out_d + (size_t)qi * qsh.k_max : nullptr);
}

// ------------------------------------------------------------------ warp scan
// Throughput form for batches: one WARP per query, no CTA barriers.  The warp
// walks its probes and blocks in the reference's order with the exact current
// distk (no speculation): lane v estimates vector v of the block, the lanes
// that pass re-rank themselves (thread-level chains, all segments), and lane 0
// applies the reference's insert sequence.  Each warp owns its LUTs and pool
// in shared memory.
constexpr int kWarpsPerCta = 4;

struct WarpSmem {
    uint16_t *lut;   // 4 * Dtot
    float *qres;     // Dtot
    SegScal *scal;   // S
    float *cd, *ipx, *part;  // S * 32 each
    float *cur;      // 32
    float *stage;    // S + 1
    uint32_t *pool_id;
    float *pool_d;   // topk + 1 each
};

__host__ __device__ inline size_t warp_smem_bytes(int Dtot, int S, int topk) {
    return align16(2 * 4 * (size_t)Dtot) + align16(4 * (size_t)Dtot) + align16(sizeof(SegScal) * S) +
           3 * align16(4 * 32 * (size_t)S) + align16(4 * 32) + align16(4 * (size_t)(S + 1)) +
           2 * align16(4 * (size_t)(topk + 1));
}

__device__ WarpSmem warp_smem_layout(char *base, int Dtot, int S, int topk) {
    WarpSmem w;
    size_t o = 0;
    w.lut = (uint16_t *)(base + o);
    o += align16(2 * 4 * (size_t)Dtot);
    w.qres = (float *)(base + o);
    o += align16(4 * (size_t)Dtot);
    w.scal = (SegScal *)(base + o);
    o += align16(sizeof(SegScal) * S);
    w.cd = (float *)(base + o);
    o += align16(4 * 32 * (size_t)S);
    w.ipx = (float *)(base + o);
    o += align16(4 * 32 * (size_t)S);
    w.part = (float *)(base + o);
    o += align16(4 * 32 * (size_t)S);
    w.cur = (float *)(base + o);
    o += align16(4 * 32);
    w.stage = (float *)(base + o);
    o += align16(4 * (size_t)(S + 1));
    w.pool_id = (uint32_t *)(base + o);
    o += align16(4 * (size_t)(topk + 1));
    w.pool_d = (float *)(base + o);
    return w;
}

// Lut::prepare for every segment of cluster c, by one warp.
__device__ void prepare_cluster_warp(const DevIndexView &ix, const float *__restrict__ qrot,
                                     const float *__restrict__ prune, int c, WarpSmem &ws) {
    const int lane = threadIdx.x & 31, S = ix.S;
    for (int i = lane; i < ix.Dtot; i += 32) {
        int s = 0;
        while (s + 1 < S && i >= ix.seg[s + 1].qoff) ++s;
        const SegDev &g = ix.seg[s];
        ws.qres[i] = __fsub_rn(qrot[i], g.cent[(size_t)c * g.dim + (i - g.qoff)]);
    }
    __syncwarp();
    for (int s = 0; s < S; ++s) {
        const SegDev &g = ix.seg[s];
        const float *qr = ws.qres + g.qoff;
        const float sum_q = warp_eigen_sum(g.dim, [&](int i) { return qr[i]; });
        const float q2 = warp_eigen_sum(g.dim, [&](int i) { return __fmul_rn(qr[i], qr[i]); });
        const int ncb = g.dim / 4;
        float lo = FLT_MAX, hi = -FLT_MAX;
        for (int cb = lane; cb < ncb; cb += 32) {
            float t[16];
            lut_entries(qr + cb * 4, t);
#pragma unroll
            for (int j = 0; j < 16; ++j) {
                lo = fminf(lo, t[j]);
                hi = fmaxf(hi, t[j]);
            }
        }
        for (int o = 16; o > 0; o >>= 1) {
            lo = fminf(lo, __shfl_xor_sync(kFull, lo, o));
            hi = fmaxf(hi, __shfl_xor_sync(kFull, hi, o));
        }
        const float delta = (float)__ddiv_rn((double)__fsub_rn(hi, lo), 65536.0 - 0.01);
        uint16_t *lut = ws.lut + 4 * g.qoff;
        for (int cb = lane; cb < ncb; cb += 32) {
            float t[16];
            lut_entries(qr + cb * 4, t);
            uint32_t packed[8];
#pragma unroll
            for (int j = 0; j < 16; j += 2) {
                const uint32_t a = (uint16_t)(int)__fdiv_rn(__fsub_rn(t[j], lo), delta);
                const uint32_t b = (uint16_t)(int)__fdiv_rn(__fsub_rn(t[j + 1], lo), delta);
                packed[j / 2] = a | (b << 16);
            }
            uint4 *dst = reinterpret_cast<uint4 *>(lut + cb * 16);
            dst[0] = make_uint4(packed[0], packed[1], packed[2], packed[3]);
            dst[1] = make_uint4(packed[4], packed[5], packed[6], packed[7]);
        }
        if (lane == 0) {
            SegScal &sc = ws.scal[s];
            sc.delta = delta;
            sc.vl = lo;
            sc.sum_vl = (float)__dmul_rn(__dadd_rn((double)lo, __dmul_rn(0.5, (double)delta)), (double)(float)ncb);
            sc.sum_q = sum_q;
            sc.q_l2sqr = q2;
            sc.q_l2norm = sqrtf(q2);
            sc.c1 = (float)__dsub_rn(__dmul_rn(0.5, (double)sum_q), (double)__fmul_rn(0.58f, sc.q_l2norm));
            const float one_over_sqrtD = (float)__ddiv_rn(1.0, (double)sqrtf((float)g.dim));
            sc.c2 = __fmul_rn(__fdiv_rn(4.0f, 0.8f), one_over_sqrtD);
            sc.vfac = __fsub_rn(q2, __fmul_rn(2.0f, prune[s]));
        }
    }
    __syncwarp();
    for (int g = 0; g < ix.Dtot / 64; ++g) ex_reorder(ws.qres + 64 * g);
}

__global__ void __launch_bounds__(kWarpsPerCta * 32) k_scan_warp(DevIndexView ix, const uint32_t *__restrict__ probe,
                                                                 int nprobe, int nq, const float *__restrict__ qrot_all,
                                                                 const float *__restrict__ prune_all, int topk,
                                                                 uint32_t *__restrict__ out_ids,
                                                                 float *__restrict__ out_d,
                                                                 unsigned long long *__restrict__ counters,
                                                                 size_t per_warp) {
    extern __shared__ __align__(16) char smem_raw[];
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31, S = ix.S;
    const int qi = blockIdx.x * kWarpsPerCta + w;
    if (qi >= nq) return;
    WarpSmem ws = warp_smem_layout(smem_raw + w * per_warp, ix.Dtot, S, topk);
    for (int i = lane; i <= topk; i += 32) {
        ws.pool_id[i] = 0;
        ws.pool_d[i] = 0.0f;
    }
    int sz = 0;
    float dk = FLT_MAX;
    unsigned long long c_blocks = 0, c_vecs = 0, c_rr = 0, c_spec = 0;
    const uint32_t *pr = probe + (size_t)qi * nprobe;
    const float *qrot = qrot_all + (size_t)qi * ix.Dtot, *prune = prune_all + (size_t)qi * S;
    for (int p = 0; p < nprobe; ++p) {
        const int c = (int)pr[p];
        prepare_cluster_warp(ix, qrot, prune, c, ws);
        const int64_t b0 = ix.blk_off[c], v0 = ix.vec_off[c];
        const int nb = (int)(ix.blk_off[c + 1] - b0), n = (int)(ix.vec_off[c + 1] - v0);
        c_blocks += nb;
        c_vecs += n;
        for (int b = 0; b < nb; ++b) {
            const int64_t gb = b0 + b;
            // estimates (saq_searcher.hpp:87-132 / 185-195), lane = vector
            float cur = 0.0f;
            int nst = 0;
            bool pass = true;
            if (S == 1) {
                const SegDev &g = ix.seg[0];
                const float on = g.onorm[gb * 32 + lane];
                float ipx = 0.0f;
                const float est = g.bits ? fast_est(g, ws.lut, ws.scal[0], gb, lane, on, ipx) : vars_est(ws.scal[0], on);
                ws.cd[lane] = est;
                ws.ipx[lane] = ipx;
                cur = est;
            } else {
                float cdv[kMaxSeg];
                for (int s = 0; s < S; ++s) {
                    cdv[s] = vars_est(ws.scal[s], ix.seg[s].onorm[gb * 32 + lane]);
                    cur = __fadd_rn(cur, cdv[s]);
                }
                float mi = warp_min_tree(cur);
                pass = !(mi > dk);
                ws.stage[0] = mi;  // all lanes write the same value
                nst = 1;
                for (int s = 0; s < S && pass; ++s) {
                    const SegDev &g = ix.seg[s];
                    if (!g.bits) continue;
                    const float on = g.onorm[gb * 32 + lane];
                    cur = __fsub_rn(cur, cdv[s]);
                    float ipx;
                    cdv[s] = fast_est(g, ws.lut + 4 * g.qoff, ws.scal[s], gb, lane, on, ipx);
                    ws.ipx[s * 32 + lane] = ipx;
                    cur = __fadd_rn(cur, cdv[s]);
                    mi = warp_min_tree(cur);
                    pass = !(mi > dk);
                    ++nst;
                }
                for (int s = 0; s < S; ++s) ws.cd[s * 32 + lane] = cdv[s];
            }
            // candidates under the exact distk at the block's start
            bool cand;
            if (S == 1) {
                const int cnp = (b == nb - 1) ? (n % 32) : 32;  // scanCluster's last-block count
                cand = lane < cnp && cur < dk;
            } else {
                cand = pass && cur < dk && (b * 32 + lane) < n;
            }
            const uint32_t cm = __ballot_sync(kFull, cand);
            if (!cm) continue;
            if (cand) {  // re-rank this lane's vector: every segment, thread-level chains
                const int64_t gv = v0 + (int64_t)b * 32 + lane;
                for (int s = 0; s < S; ++s) {
                    const SegDev &g = ix.seg[s];
                    const float ex = g.bits > 1 ? excode_ip_thread(ws.qres + g.qoff, g.lcode + (size_t)gv * g.lstride,
                                                                   g.dim, g.bits - 1)
                                                : 0.0f;
                    const float acc = accurate_dist(g.onorm[gb * 32 + lane], ws.ipx[s * 32 + lane], ex, g.exfac[gv].x,
                                                    g.bits, ws.scal[s].sum_q, ws.scal[s].q_l2sqr);
                    ws.part[s * 32 + lane] = S == 1 ? acc : __fsub_rn(acc, ws.cd[s * 32 + lane]);
                }
            }
            ws.cur[lane] = cur;
            __syncwarp();
            if (lane == 0) {
                c_spec += __popc(cm);
                replay_block(S, n, nb, b, ws.cur, ws.stage, 0, ws.part, cm, ix.ids + v0, ws.pool_id, ws.pool_d, sz,
                             topk, dk, nullptr, c_rr);
            }
            dk = __shfl_sync(kFull, dk, 0);
            sz = __shfl_sync(kFull, sz, 0);
            __syncwarp();
        }
    }
    if (lane == 0 && counters) {
        atomicAdd(counters + 0, c_blocks);
        atomicAdd(counters + 1, c_vecs);
        atomicAdd(counters + 2, c_rr);
        atomicAdd(counters + 3, c_spec);
    }
    __syncwarp();
    for (int i = lane; i < topk; i += 32) {
        out_ids[(size_t)qi * topk + i] = ws.pool_id[i];
        if (out_d) out_d[(size_t)qi * topk + i] = i < sz ? ws.pool_d[i] : FLT_MAX;
    }
}

// ------------------------------------------------------------------ split scan
// For latency-bound calls (one query, or a few).  The first tile of the
// nearest cluster is scanned exactly; the pool's distk afterwards, tau1, bounds
// distk for the rest of the scan (distk never grows).  Every remaining (probe,
// tile) is processed in parallel across the GPU under tau1; each block with a
// lane below tau1 leaves a record in a slot indexed by its position in scan
// order.  A final pass per query walks the positions in order and replays the
// reference's decisions on the records.  Blocks without a record cannot insert
// anything (none of their lanes is below tau1 >= distk), so the replay is exact.
// Blocks of a speculative tile (one warp's work): 16 for deferred queries, 4 when a few
// queries have the GPU alone.  One query over 32 probes of 3-4 blocks has 32 tiles
// either way, but over 32 x 31 blocks 64 tiles of 16 leave half of the SMs idle; tiles of 4
// and the ids in the records: 131 to 123 us (host call), 37 queries 1.74 to 1.59 ms.
constexpr int kTileBlocks = 16;
constexpr int kFewTileBlocks = 4;
static_assert(kTileBlocks <= kTileB && kFewTileBlocks <= kTileB, "tile_candidates has a slot per block");
constexpr int kFirstBlocks = 16;  // exact prefix of a deferred query (its distk bounds the first level)
// Levels of the speculation for deferred queries, in tiles after the split
// point: [0, 8), [8, 64), [64, end) by default; the autotuner may pick another
// set (each level's replay leaves the exact pool whose distk bounds the next
// level's speculation: more levels, tighter bounds, more launches).
constexpr int kMaxSpecLevels = 5;
constexpr int kSpecLevelSets[][kMaxSpecLevels] = {
    {0, 8, 64, -1, -1},
    {0, 4, 32, 256, -1},
    {0, 16, 128, -1, -1},
    {0, 8, 64, 512, -1},
    {0, 64, -1, -1, -1},
};
constexpr int kNumSpecLevelSets = (int)(sizeof(kSpecLevelSets) / sizeof(kSpecLevelSets[0]));
// A query probing more blocks than this takes the split pass (SAQG_DEFER_BLOCKS
// overrides it; 0 disables deferral).  The longest query on a single CTA ends the
// CTA scan, so the line lies low: 37 queries of 1,800 blocks 4.23 ms with 1,024
// and 1.73 with 256, 256 queries of 560 blocks 1.72 and 1.22, 4,096 queries over
// 10M vectors 2.90 and 2.15 (384: 2.13, 192: 2.21).
// With the built-in line the batch as a whole decides first, since the CTA scan of the
// queries below it holds SMs that the split pass's short kernels wait for:
//   * most queries above it: all of them take the split pass (600 queries of about 340
//     blocks, anisotropic 400,000 x 576: 2.42 ms at the line, 1.95 without deferral, 1.72
//     all deferred);
//   * else, where no query is longer than 1.25 times a resident CTA's share of the batch,
//     none does (4,000 queries of about 230 blocks, a third above the line, anisotropic
//     400,000 x 576 in 600-vector clusters: 5.33 / 4.78 / 5.19 ms);
//   * else, with three in ten above it, all (1,500 uneven queries of about 250 blocks,
//     anisotropic 647,483 x 576: 3.72 / 3.32 / 3.17 ms; 600 of about 275, Zipf 400,000 x
//     1024: 2.34 / 2.86 / 1.72; worst found, 4,000 of 281, Zipf: 2.49 / 3.49 / 2.72);
//   * else those above it (a tenth to a quarter: the batch of 4,096 over 10M vectors 1.84 /
//     8.76 / 2.32 ms).
constexpr int kDeferBlocks = 256;

struct SplitState {
    int *nlist;          // number of queries on the list (device)
    int *work_next;      // next chunk of the level's speculative tiles (reset by k_tile_prefix)
    int *qlist;          // [cap] slot -> query id
    int cap;             // slots
    uint32_t *pool_id;   // [cap][topk]
    float *pool_d;       // [cap][topk]
    int *pool_size;      // [cap]
    float *tau;          // [cap]
    int *tile_off;       // [cap][nprobe + 1] tiles before probe p
    int *blk_base;       // [cap][nprobe] scan-order position of the probe's first block
    int *split_p;        // [cap] probe where the speculative part starts (nprobe: none)
    int *split_b;        // [cap] block of that probe's cluster where it starts
    int *q_tile_off;     // [cap + 1]
    int *npos;           // [cap] scan positions (blocks) of the query
    int64_t *pos_off;    // [cap] first record position reserved for the slot
    unsigned long long *pos_used;  // record positions handed out so far
    // [pos_cap] per record (NaN: none): x the smallest candidate estimate, y the
    // largest stage minimum, z the smallest value a candidate lane's accept test
    // can see (its accurate distance; several segments: every running sum),
    // -inf when one of them is NaN
    float4 *summ;
    float *rec;          // [pos_cap][rec_words]
    int64_t pos_cap;
    int rec_words;
    QueryShape qsh;      // per-query nprobe and k (strides np_max, k_max)
    int first_blocks;    // exact prefix: at least this many blocks, and a full pool
    // the level being speculated and replayed: tiles [t_lo, t_hi) after the split
    // point of each query (distk at the level's start bounds its speculation)
    int t_lo, t_hi;
    int final_level;     // the last level writes the results, the others the pool
    // > 0: every query of the call is listed, in order, with room for this many blocks
    // each, so k_scan_first fills the list itself and k_defer does not run
    int64_t stride;
    int tile_blocks;     // blocks of a speculative tile (kFewTileBlocks or kTileBlocks)
    int replay_recs;     // records of a staged chunk of the replay (at most kReplayRecs)
};

// Scan-order position of the first block of tile t after a query's split
// point (npos when t is past its last tile).
__device__ __forceinline__ int tile_pos(const SplitState &st, int slot, int t) {
    const int npm = st.qsh.np_max;
    const int *to = st.tile_off + (size_t)slot * (npm + 1);
    if (t >= to[npm]) return st.npos[slot];
    int lo = 0, hi = npm;  // probe: last p with to[p] <= t
    while (hi - lo > 1) {
        const int mid = (lo + hi) >> 1;
        if (to[mid] <= t) lo = mid;
        else hi = mid;
    }
    const int first = lo == st.split_p[slot] ? st.split_b[slot] : 0;
    return st.blk_base[(size_t)slot * npm + lo] + first + (t - to[lo]) * st.tile_blocks;
}

// Words of a record: 8 of header, S + 1 stage minima, the 32 estimates, 32 partials per
// segment, the 32 ids (so that the replay reads nothing but staged records).
__host__ __device__ constexpr int rec_words_of(int S) { return (8 + (S + 1) + 32 + 32 * S + 32 + 3) & ~3; }
__device__ __forceinline__ const uint32_t *rec_ids(const float *rec, int S) {
    return reinterpret_cast<const uint32_t *>(rec) + 8 + (S + 1) + 32 + 32 * S;
}

__device__ __forceinline__ int list_len(const SplitState &st) { return st.stride ? st.cap : min(*st.nlist, st.cap); }

__global__ void __launch_bounds__(kScanThreads, kScanMinCtas) k_scan_first(DevIndexView ix, const uint32_t *__restrict__ probe,
                                                             const float *__restrict__ qrot_all,
                                                             const float *__restrict__ prune_all, SplitState st, int *__restrict__ err,
                                                             unsigned long long *__restrict__ counters, int xstride,
                                                             Prepared prep) {
    extern __shared__ __align__(16) char smem_raw[];
    const int S = ix.S, tid = threadIdx.x;
    // slots round-robin over a grid sized to the machine (the list length is known on the device only)
    for (int slot = blockIdx.x; slot < list_len(st); slot += gridDim.x) {
        const int qi = st.stride ? slot : st.qlist[slot];
        const int np_max = st.qsh.np_max, k_max = st.qsh.k_max;
        const int nprobe = st.qsh.np_of(qi), topk = st.qsh.k_of(qi);
        ScanSmem sm = scan_smem_layout(smem_raw, ix.Dtot, S, k_max, xstride);
        __shared__ int pool_size;
        __shared__ float distk;
        ScanTally tl;
        tl.counted = counters != nullptr;
        init_pool(sm, topk, pool_size, distk);
        const uint32_t *pr = probe + (size_t)qi * np_max;
        const float *qrot = qrot_all + (size_t)qi * ix.Dtot, *prune = prune_all + (size_t)qi * S;
        // the exact prefix, as scan_probes does: whole tiles in scan order until at
        // least kFirstBlocks blocks are done and the pool is full (its distk then
        // bounds every later distk, so it can serve as the speculation bound)
        int sp_p = nprobe, sp_b = 0;
        for (int p = 0; p < nprobe && sp_p == nprobe; ++p) {
            const int c = (int)pr[p];
            const int64_t b0 = ix.blk_off[c], v0 = ix.vec_off[c];
            const int nb = (int)(ix.blk_off[c + 1] - b0), n = (int)(ix.vec_off[c + 1] - v0);
            bool prepared = false;
            for (int t0 = 0; t0 < nb; t0 += kTileB) {
                if (tl.blocks >= st.first_blocks && pool_size == topk) {
                    sp_p = p;
                    sp_b = t0;
                    break;
                }
                if (!prepared) {
                    if (prep.has(slot)) load_cluster(ix, qrot, prep.lut_of(slot, p, ix.Dtot), prep.scal_of(slot, p, S), c, sm);
                    else prepare_cluster(ix, qrot, prune, c, sm);
                    prepared = true;
                }
                const int te = min(nb, t0 + kTileB);
                tl.blocks += te - t0;
                tl.vecs += min(n, te * 32) - t0 * 32;
                tile_candidates(ix, sm, b0, v0, nb, n, te - t0, [&](int slot) { return t0 + slot; }, distk);
                if (tid < 32) {
                    float dk = distk;
                    int sz = pool_size;
                    const unsigned nc = replay_tile_warp(S, t0, nullptr, te - t0, sm, ix.ids + v0, sm.pool_id, sm.pool_d, sz, topk, dk,
                                                         tl.counted, tl.rr);
                    if (tid == 0) {
                        tl.spec += nc;
                        distk = dk;
                        pool_size = sz;
                    }
                }
                __syncthreads();
            }
        }
        flush_tally(tl, counters);
        for (int i = tid; i < topk; i += blockDim.x) {
            st.pool_id[(size_t)slot * k_max + i] = sm.pool_id[i];
            st.pool_d[(size_t)slot * k_max + i] = sm.pool_d[i];
        }
        if (tid == 0) {
            st.pool_size[slot] = pool_size;
            st.tau[slot] = distk;
            st.split_p[slot] = sp_p;
            st.split_b[slot] = sp_b;
        }
        if (tid < 32) {  // tiles and blocks before each probe: prefix sums over the warp's lanes
            int tiles = 0;
            int64_t pos = 0;
            for (int p0 = 0; p0 < nprobe; p0 += 32) {
                const int p = p0 + tid;
                int nb = 0, nt = 0;
                if (p < nprobe) {
                    const int c = (int)pr[p];
                    nb = (int)(ix.blk_off[c + 1] - ix.blk_off[c]);
                    const int rest = p < sp_p ? 0 : p == sp_p ? nb - sp_b : nb;
                    nt = (rest + st.tile_blocks - 1) / st.tile_blocks;
                }
                int xt = nt;
                int64_t xb = nb;
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) {
                    const int yt = __shfl_up_sync(kFull, xt, o);
                    const int64_t yb = __shfl_up_sync(kFull, xb, o);
                    if (tid >= o) {
                        xt += yt;
                        xb += yb;
                    }
                }
                if (p < nprobe) {
                    st.tile_off[(size_t)slot * (np_max + 1) + p] = tiles + xt - nt;
                    st.blk_base[(size_t)slot * np_max + p] = (int)(pos + xb - nb);
                }
                tiles += __shfl_sync(kFull, xt, 31);
                pos += __shfl_sync(kFull, xb, 31);
            }
            for (int p = nprobe + tid; p <= np_max; p += 32) st.tile_off[(size_t)slot * (np_max + 1) + p] = tiles;
            if (st.stride) {
                if (tid == 0) {
                    st.qlist[slot] = slot;
                    st.npos[slot] = (int)pos;
                    st.pos_off[slot] = slot * st.stride;
                }
            } else if (tid == 0 && pos != st.npos[slot]) {
                *err = 2;
            }
        }
        __syncthreads();  // the next slot reuses the shared state
    }
}

// Work offsets of the level's tiles: slot q holds tiles [t_lo, t_hi) of its own.
// One CTA of kPrefixThreads: each thread sums a contiguous run of slots, a
// block-wide exclusive scan of the run sums, then each run is written.
constexpr int kPrefixThreads = 256;
__global__ void __launch_bounds__(kPrefixThreads) k_tile_prefix(SplitState st) {
    __shared__ int wsum[kPrefixThreads / 32];
    const int nprobe = st.qsh.np_max, tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
    const int n = list_len(st);
    const int per = (n + kPrefixThreads - 1) / kPrefixThreads, q0 = min(n, tid * per), q1 = min(n, q0 + per);
    auto count = [&](int q) {
        const int nt = st.tile_off[(size_t)q * (nprobe + 1) + nprobe];
        return max(0, min(nt, st.t_hi) - min(nt, st.t_lo));
    };
    int run = 0;
    for (int q = q0; q < q1; ++q) run += count(q);
    int x = run;  // inclusive scan within the warp
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
    }
    if (lane == 31) wsum[w] = x;
    __syncthreads();
    constexpr int kW = kPrefixThreads / 32;
    if (w == 0) {
        int v = lane < kW ? wsum[lane] : 0;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int y = __shfl_up_sync(0xffffffffu, v, o);
            if (lane >= o) v += y;
        }
        if (lane < kW) wsum[lane] = v;  // inclusive over warps
    }
    __syncthreads();
    int acc = x - run + (w ? wsum[w - 1] : 0);
    for (int q = q0; q < q1; ++q) {
        st.q_tile_off[q] = acc;
        acc += count(q);
    }
    if (tid == kPrefixThreads - 1) {
        st.q_tile_off[n] = wsum[kPrefixThreads / 32 - 1];
        *st.work_next = 0;
    }
}

// Last index i of a[0, n) (ascending, a[0] <= x) with a[i] <= x, by a warp.
__device__ __forceinline__ int warp_last_le(const int *__restrict__ a, int n, int x) {
    const int lane = threadIdx.x & 31;
    int lo = 0;
    while (n > 1) {
        const int step = (n + 31) >> 5, i = lane * step;
        const int hit = __popc(__ballot_sync(kFull, i < n && a[lo + min(i, n - 1)] <= x)) - 1;  // a prefix of the lanes
        lo += hit * step;
        n = min(step, n - hit * step);
    }
    return lo;
}

// One tile of a chunk of k_scan_spec.
struct SpecTile {
    int slot, q, p, c, n, nb, first, blocks;  // blocks [first, first + blocks) of cluster c, probe p of query q
    int64_t b0, v0, pos;                      // pos: record position of block 0 of the cluster (in the slot's)
    float tau;
    uint32_t left;  // its blocks that stage 0 leaves
};

__global__ void __launch_bounds__(kScanThreads, kScanMinCtas) k_scan_spec(DevIndexView ix, const uint32_t *__restrict__ probe,
                                                            int nprobe, const float *__restrict__ qrot_all,
                                                            const float *__restrict__ prune_all, SplitState st,
                                                            unsigned long long *__restrict__ counters, int xstride,
                                                            Prepared prep) {
    extern __shared__ __align__(16) char smem_raw[];
    __shared__ SpecTile tiles[kScanWarps];
    __shared__ float vf[kScanWarps * kMaxSeg];
    const int S = ix.S, tid = threadIdx.x, w = tid >> 5, lane = tid & 31;
    ScanSmem sm = scan_smem_layout(smem_raw, ix.Dtot, S, 1, xstride);
    ScanTally tl;
    const int nl = list_len(st);
    const int total = st.q_tile_off[nl];
    // chunks of consecutive tiles taken from a shared counter: tiles differ widely in
    // cost (candidates, pruning stages), so equal shares per CTA leave a long tail.  A
    // chunk has up to a tile per warp: each warp finds its tile and filters its blocks
    // by stage 0 when the LUT's scalars are prepared, then the CTA takes the tiles with
    // blocks left in order.  At least about four chunks per CTA, so that a small level
    // (few queries) still spreads over the whole grid.
    const int ct = max(1, min(kScanWarps, total / (4 * (int)gridDim.x)));
    __shared__ int chunk;
    int last_slot = -1, last_c = -1;
    for (;;) {
        if (tid == 0) chunk = atomicAdd(st.work_next, 1);
        __syncthreads();
        const int w_begin = chunk * ct, nt = min(total - w_begin, ct);
        if (nt <= 0) break;
        if (w < nt) {
            const int wi = w_begin + w, slot = warp_last_le(st.q_tile_off, nl, wi);
            const int local = st.t_lo + (wi - st.q_tile_off[slot]);
            const int *to = st.tile_off + (size_t)slot * (nprobe + 1);
            const int p = warp_last_le(to, nprobe, local), q = st.qlist[slot];
            SpecTile t;
            t.slot = slot;
            t.q = q;
            t.p = p;
            t.c = (int)probe[(size_t)q * nprobe + p];
            t.b0 = ix.blk_off[t.c];
            t.v0 = ix.vec_off[t.c];
            t.nb = (int)(ix.blk_off[t.c + 1] - t.b0);
            t.n = (int)(ix.vec_off[t.c + 1] - t.v0);
            t.first = (p == st.split_p[slot] ? st.split_b[slot] : 0) + (local - to[p]) * st.tile_blocks;
            t.blocks = min(st.tile_blocks, t.nb - t.first);
            t.tau = st.tau[slot];
            t.pos = st.blk_base[(size_t)slot * nprobe + p];
            t.left = (1u << t.blocks) - 1u;
            if (S > 1) {
                float *fv = vf + w * kMaxSeg;
                if (prep.has(slot)) {
                    if (lane < S) fv[lane] = prep.scal_of(slot, p, S)[lane].vfac;
                } else {
                    for (int s = 0; s < S; ++s) {
                        const float v = stage0_scalar(ix, s, t.c, qrot_all + (size_t)q * ix.Dtot, prune_all + (size_t)q * S);
                        if (lane == 0) fv[s] = v;
                    }
                }
                __syncwarp();
                uint32_t left = 0;
                for (int g = 0; kQuad * g < t.blocks; g += 2) {
                    const float *const fvs[2] = {fv, fv};
                    const int64_t gb[2] = {t.b0 + t.first + kQuad * g, t.b0 + t.first + kQuad * g + kQuad};
                    const int nv[2] = {t.blocks - kQuad * g, t.blocks - kQuad * g - kQuad};  // past the tile: none
                    uint32_t l2[2];
                    const int nvc[2] = {min(kQuad, nv[0]), min(kQuad, nv[1])};
                    quad_filter(ix, fvs, gb, nvc, t.tau, l2);
                    left |= (l2[0] | l2[1] << kQuad) << (kQuad * g);
                }
                t.left = left;
            }
            if (lane == 0) tiles[w] = t;
        }
        __syncthreads();
        for (int i = 0; i < nt; ++i) {
            const SpecTile &t = tiles[i];
            if (tid == 0) {
                tl.blocks += t.blocks;
                tl.vecs += min(t.n, (t.first + t.blocks) * 32) - t.first * 32;
            }
            const uint32_t left = t.left;
            const int ng = __popc(left), slot = t.slot;
            if (ng == 0) continue;
            if (slot != last_slot || t.c != last_c) {  // LUTs survive across tiles of one cluster
                if (prep.has(slot)) load_cluster(ix, qrot_all + (size_t)t.q * ix.Dtot, prep.lut_of(slot, t.p, ix.Dtot),
                                                 prep.scal_of(slot, t.p, S), t.c, sm);
                else prepare_cluster(ix, qrot_all + (size_t)t.q * ix.Dtot, prune_all + (size_t)t.q * S, t.c, sm);
                last_slot = slot;
                last_c = t.c;
            }
            tile_candidates(ix, sm, t.b0, t.v0, t.nb, t.n, ng, [&](int sl) { return t.first + nth_bit(left, sl); }, t.tau);
            for (int wslot = w; wslot < ng; wslot += kScanWarps) {
                const uint32_t cm = sm.cmask[wslot];
                const int b = sm.sblk[wslot];
                const int64_t pos = t.pos + b;
                if (cm && pos < st.npos[slot]) {
                    float *r = st.rec + (size_t)(st.pos_off[slot] + pos) * st.rec_words;
                    uint32_t *ri = reinterpret_cast<uint32_t *>(r);
                    // summary: a later distk below the minimum estimate, or below a stage minimum,
                    // leaves the block without effect
                    const bool in = (cm >> lane) & 1u;
                    float mn = in ? sm.cur[wslot * 32 + lane] : __int_as_float(0x7fffffff);
                    float mx = (S > 1 && lane < sm.nstage[wslot]) ? sm.stage[wslot * (S + 1) + lane] : __int_as_float(0x7fffffff);
                    // ... and a later distk below every value the lane's accept test can
                    // compare (replay_block_warp: the accurate distance, or each running sum)
                    float mz = __int_as_float(0x7f800000);
                    if (in) {
                        if (S == 1) {
                            mz = sm.part[wslot * 32 + lane];
                        } else {
                            float acc = sm.cur[wslot * 32 + lane];
                            for (int s2 = 0; s2 < S; ++s2) {
                                acc = __fadd_rn(acc, sm.part[(wslot * S + s2) * 32 + lane]);
                                mz = fminf(mz, acc);
                                if (acc != acc) mz = -__int_as_float(0x7f800000);
                            }
                        }
                        if (mz != mz) mz = -__int_as_float(0x7f800000);
                    }
#pragma unroll
                    for (int o = 16; o; o >>= 1) {
                        mn = fminf(mn, __shfl_xor_sync(kFull, mn, o));
                        mx = fmaxf(mx, __shfl_xor_sync(kFull, mx, o));
                        mz = fminf(mz, __shfl_xor_sync(kFull, mz, o));
                    }
                    if (lane == 0) {
                        ri[0] = (uint32_t)pos;
                        ri[1] = cm;
                        ri[2] = (uint32_t)(S == 1 ? 0 : sm.nstage[wslot]);
                        ri[3] = (uint32_t)t.c;
                        ri[4] = (uint32_t)b;
                        ri[5] = (uint32_t)(uint64_t)t.v0;
                        ri[6] = (uint32_t)((uint64_t)t.v0 >> 32);
                        ri[7] = __float_as_uint(mx);
                        st.summ[st.pos_off[slot] + pos] = make_float4(mn, mx, mz, 0.0f);
                        if (counters) atomicAdd(counters + 3, (unsigned long long)__popc(cm));
                    }
                    if (S > 1 && lane <= S) r[8 + lane] = sm.stage[wslot * (S + 1) + lane];
                    r[8 + (S + 1) + lane] = sm.cur[wslot * 32 + lane];
                    for (int s = 0; s < S; ++s) r[8 + (S + 1) + 32 + s * 32 + lane] = sm.part[(wslot * S + s) * 32 + lane];
                    ri[8 + (S + 1) + 32 + 32 * S + lane] = in ? ix.ids[t.v0 + (int64_t)b * 32 + lane] : 0u;
                }
            }
            __syncthreads();
        }
        __syncthreads();  // every thread is done with the chunk's tiles
    }
    if (tid == 0 && counters) {
        atomicAdd(counters + 0, tl.blocks);
        atomicAdd(counters + 1, tl.vecs);
    }
}

__device__ __forceinline__ void cp_async16(void *smem, const void *gmem) {
    const unsigned sa = (unsigned)__cvta_generic_to_shared(smem);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(sa), "l"(gmem) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() {
    asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

// Whether a staged record changes the pool under the current distk / pool
// size (some lane's insert would be accepted), and how many of its lanes the
// reference evaluates accurately when nothing earlier in the record changes
// distk.  Warp-uniform.
__device__ __forceinline__ bool record_effect(int S, const float *rec, float dk, int sz, int topk, int &count) {
    const int lane = threadIdx.x & 31;
    const uint32_t *ri = reinterpret_cast<const uint32_t *>(rec);
    const uint32_t cm = ri[1];
    count = 0;
    if (!cm || (S > 1 && __uint_as_float(ri[7]) > dk)) return false;
    const float *cur = rec + 8 + (S + 1), *part = cur + 32;
    const bool in = (cm >> lane) & 1u;
    const float c = in ? cur[lane] : FLT_MAX;
    const bool pass = in && c < dk;
    count = __popc(__ballot_sync(kFull, pass));
    float acc = c;
    if (S == 1) {
        acc = pass ? part[lane] : FLT_MAX;
    } else if (pass) {
        for (int s = 0; s < S; ++s) {
            acc = __fadd_rn(acc, part[s * 32 + lane]);
            if (acc >= dk) break;
        }
    }
    return __any_sync(kFull, pass && !(sz == topk && acc > dk));
}

// Records per staged chunk (double-buffered): 32 where they fit beside the scan's own
// shared memory, fewer for plans of many segments or a large k (16 segments of 64
// dimensions leave room for 29, and for 22 with k = 4,096), at the least 4.
constexpr int kReplayRecs = 32;
// Most shared memory of a scan (200 KB beside the tiles' block numbers, which a tile
// buffer has 64 bytes of), of the warp-specialised form's two buffers, and of a replay.
constexpr size_t kScanSmem = 200 * 1024 + sizeof(int) * kTileB;
constexpr size_t kScanWsSmem = 220 * 1024 + 2 * sizeof(int) * kTileB, kReplaySmem = 220 * 1024;
static_assert(kScanSmem + 2 * 4 * 4 * rec_words_of(kMaxSeg) <= kReplaySmem, "four records always fit");
constexpr int kReplayPer = 4;    // scan positions per thread in a window

// Per query on the list: walk its scan positions in order, kScanThreads at a
// time.  A record can matter only if a candidate estimate lies below distk and
// no stage minimum above it; distk only shrinks, so positions whose summary
// fails the distk at the window's start are dropped at once.  The rest are
// staged into shared memory by asynchronous copies, replay_recs at a time
// (the next chunk in flight while the current one is evaluated).  In a chunk,
// every warp evaluates records under the current distk; the first record with
// an accepted insert is replayed exactly by warp 0 (the records before it
// change nothing and only add their counts), and evaluation resumes after it.
// kPer > 0 (no counters kept, k at most 32 kPer, at most kRegSegs segments): warp 0 holds
// the pool in registers, and a chunk is evaluated once: the records marked under the distk at its
// start are replayed one after the other, without a barrier per record.  A record left
// unmarked can still matter to the reference where a running sum equals the distk of
// its turn (the sum is inserted); all warps look for that among the distk values that the
// chunk's inserts left, and a chunk with such a sum, or with more inserts than kSeen, is replayed again, every record.
constexpr int kSeen = 64;
template <int kPer>
__global__ void __launch_bounds__(kScanThreads) k_scan_replay(DevIndexView ix, SplitState st,
                                                              uint32_t *__restrict__ out_ids, float *__restrict__ out_d,
                                                              unsigned long long *__restrict__ counters, int xstride) {
    extern __shared__ __align__(16) char smem_raw[];
    const int S = ix.S;
    // slots round-robin over a grid sized to the machine (the list length is known on the device only)
    for (int slot = blockIdx.x; slot < list_len(st); slot += gridDim.x) {
        const int qi = st.qlist[slot];
        const int k_max = st.qsh.k_max, topk = st.qsh.k_of(qi);
        ScanSmem sm = scan_smem_layout(smem_raw, ix.Dtot, S, k_max, xstride);
        float *stage_buf = reinterpret_cast<float *>(smem_raw + scan_smem_bytes(ix.Dtot, S, k_max, xstride));
        __shared__ int pool_size;
        __shared__ float distk;
        __shared__ int list[kScanThreads * kReplayPer];
        __shared__ int warp_cnt[kScanWarps];
        __shared__ int eff[kReplayRecs], cnt[kReplayRecs];
        __shared__ int s_next, s_plo, s_phi;
        __shared__ int eff_pos[kReplayRecs], n_eff;  // records replayed in the current chunk
        __shared__ float eff_dk[kReplayRecs], c_dk0;
        const int tid = threadIdx.x, w = tid >> 5, lane = tid & 31;
        for (int i = tid; i < topk; i += blockDim.x) {
            sm.pool_id[i] = st.pool_id[(size_t)slot * k_max + i];
            sm.pool_d[i] = st.pool_d[(size_t)slot * k_max + i];
        }
        if (tid == 0) {
            pool_size = st.pool_size[slot];
            distk = st.tau[slot];
            s_plo = tile_pos(st, slot, st.t_lo);  // this level's scan positions
            s_phi = tile_pos(st, slot, st.t_hi);
        }
        const int np = st.npos[slot];
        const float4 *su = st.summ + st.pos_off[slot];
        const float *rq = st.rec + (size_t)st.pos_off[slot] * st.rec_words;
        const int RW = st.rec_words, R16 = RW / 4, RC = st.replay_recs;
        unsigned long long rr = 0;
        __syncthreads();
        __shared__ float old_d[kPer ? 32 * kPer : 1];  // the pool before a chunk
        __shared__ uint32_t old_id[kPer ? 32 * kPer : 1];
        __shared__ float seen[kSeen];  // distk after each insert of the chunk
        __shared__ int nseen;
        const int pos_end = min(np, s_phi);
        for (int base = s_plo, per; base < pos_end; base += kScanThreads * per) {
            // the first window is short: its inserts lower the distk that filters the next
            per = base == s_plo ? 1 : kReplayPer;
            // thread t tests positions base + per t .. + per - 1; a
            // block-wide prefix of the counts keeps the list in position order
            const int p0 = base + per * tid;
            const float dk0 = distk;
            // with a full pool a lane is accepted only at a value <= distk: a record whose
            // every such value exceeds distk (summary z) changes nothing and is not staged.
            // With counters kept, the lanes the reference evaluates in such a record are
            // counted after each chunk under the distk at its position (count_dropped).
            const bool zf = pool_size == topk;
            const int wend = min(pos_end, base + kScanThreads * per);
            bool f[kReplayPer];
            int mine = 0;
    #pragma unroll
            for (int r = 0; r < kReplayPer; ++r) {
                f[r] = false;
                if (r < per && p0 + r < pos_end) {
                    const float4 v = su[p0 + r];
                    f[r] = v.x < dk0 && !(v.y > dk0) && !(zf && v.z > dk0);
                }
                mine += f[r];
            }
            int incl = mine;
    #pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int v = __shfl_up_sync(kFull, incl, o);
                if (lane >= o) incl += v;
            }
            if (lane == 31) warp_cnt[w] = incl;
            __syncthreads();
            int off = incl - mine, total = 0;
            for (int i = 0; i < kScanWarps; ++i) {
                if (i < w) off += warp_cnt[i];
                total += warp_cnt[i];
            }
    #pragma unroll
            for (int r = 0; r < kReplayPer; ++r)
                if (f[r]) list[off++] = p0 + r;
            __syncthreads();
            const int nch = (total + RC - 1) / RC;
            // lanes with candidate estimate below the distk at their position in the
            // records of [lo, hi) that the accept bound dropped (distk: c_dk0, then after
            // each of the n_eff records replayed in this range, in position order)
            auto count_dropped = [&](int lo, int hi) {
                unsigned long long add = 0;
                for (int p = lo + tid; p < hi; p += kScanThreads) {
                    const float4 v = su[p];
                    if (!(v.x < dk0 && !(v.y > dk0) && v.z > dk0)) continue;
                    float dkp = c_dk0;
                    for (int e = 0; e < n_eff; ++e)
                        if (eff_pos[e] < p) dkp = eff_dk[e];
                    if (S > 1 && v.y > dkp) continue;  // a stage minimum above distk: no lane evaluated
                    const float *rec = rq + (size_t)p * RW;
                    const float *cur = rec + 8 + (S + 1);
                    for (uint32_t m = reinterpret_cast<const uint32_t *>(rec)[1]; m; m &= m - 1)
                        add += cur[__ffs(m) - 1] < dkp;
                }
                if (add) atomicAdd(counters + 2, add);
            };
            if (nch == 0 && counters && zf) {
                if (tid == 0) {
                    c_dk0 = dk0;
                    n_eff = 0;
                }
                __syncthreads();
                count_dropped(base, wend);
                __syncthreads();
            }
            auto issue = [&](int k) {
                const int c0 = k * RC, cn = min(RC, total - c0);
                float *buf = stage_buf + (size_t)(k & 1) * RC * RW;
                for (int i = tid; i < cn * R16; i += kScanThreads) {
                    const int r = i / R16, e = i - r * R16;
                    cp_async16(buf + (size_t)r * RW + 4 * e, rq + (size_t)list[c0 + r] * RW + 4 * e);
                }
                cp_async_commit();
            };
            if (nch) issue(0);
            for (int k = 0; k < nch; ++k) {
                if (k + 1 < nch) {
                    issue(k + 1);
                    cp_async_wait<1>();
                } else {
                    cp_async_wait<0>();
                }
                __syncthreads();
                const float *buf = stage_buf + (size_t)(k & 1) * RC * RW;
                const int c0 = k * RC, cn = min(RC, total - c0);
                if (kPer) {
                    // every warp marks the records with an accepted insert under the distk at the
                    // chunk's start (but for ties a superset of those that have one at their turn)
                    const float dk = distk;
                    const int sz = pool_size;
                    for (int r = w; r < cn; r += kScanWarps) {
                        int c;
                        const bool e = record_effect(S, buf + (size_t)r * RW, dk, sz, topk, c);
                        if (lane == 0) eff[r] = e;
                    }
                    if (tid == 0) nseen = 0;
                    __syncthreads();
                    const uint32_t marked = __ballot_sync(kFull, lane < cn && eff[lane]);
                    if (!marked) continue;  // uniform
                    // the records `live` in order, from the pool in shared memory
                    const auto replay_records = [&](uint32_t live) {
                        RegPool<kPer ? kPer : 1> P;
                        int szw = sz, n = 0;
                        float dkw = dk;
                        while (live) {
                            P.load(sm.pool_id, sm.pool_d, szw, topk);
                            uint32_t left = 0u, m = 0u;
                            const float *rec = buf;
                            for (; live; live &= live - 1) {
                                rec = buf + (size_t)(__ffs(live) - 1) * RW;
                                m = reinterpret_cast<const uint32_t *>(rec)[1];
                                left = replay_block_regs(S, rec + 8 + (S + 1), rec[7], rec + 8 + (S + 1) + 32, m,
                                                         rec_ids(rec, S), P, [&](float x) {
                                                             if (lane == 0 && n < kSeen) seen[n] = x;
                                                             ++n;
                                                         });
                                if (left) break;
                            }
                            if (!P.odd) {
                                P.store(sm.pool_id, sm.pool_d, szw);
                                dkw = P.dk;
                            }
                            if (left) {  // lane by lane
                                n = kSeen + 1;
                                replay_block_warp(S, 0, rec + 8 + (S + 1), left == m ? rec[7] : -FLT_MAX,
                                                  rec + 8 + (S + 1) + 32, left, rec_ids(rec, S), sm.pool_id, sm.pool_d, szw, topk,
                                                  dkw, rr);
                                live &= live - 1;
                            }
                        }
                        if (lane == 0) {
                            distk = dkw;
                            pool_size = szw;
                            nseen = n;
                        }
                        __syncwarp();
                    };
                    const uint32_t all = cn == 32 ? kFull : (1u << cn) - 1u;
                    if (w == 0) {
                        for (int i = lane; i < sz; i += 32) {
                            old_d[i] = sm.pool_d[i];
                            old_id[i] = sm.pool_id[i];
                        }
                        replay_records(marked);
                    }
                    __syncthreads();
                    if (S > 1 && marked != all) {
                        const int n = nseen;
                        bool tie = n > kSeen;
                        if (!tie)
                            for (int r = w; r < cn; r += kScanWarps) {
                                if ((marked >> r) & 1u) continue;
                                const float *rec = buf + (size_t)r * RW;
                                const bool in = (reinterpret_cast<const uint32_t *>(rec)[1] >> lane) & 1u;
                                const float *cur = rec + 8 + (S + 1), *part = cur + 32;
                                float acc = in ? cur[lane] : FLT_MAX;
                                if (in && acc < dk)
                                    for (int s = 0; s < S; ++s) {
                                        acc = __fadd_rn(acc, part[s * 32 + lane]);
                                        for (int e = 0; e < n; ++e) tie |= acc == seen[e];
                                    }
                            }
                        if (__syncthreads_or(tie)) {
                            if (w == 0) {
                                for (int i = lane; i < sz; i += 32) {
                                    sm.pool_d[i] = old_d[i];
                                    sm.pool_id[i] = old_id[i];
                                }
                                __syncwarp();
                                replay_records(all);
                            }
                            __syncthreads();
                        }
                    }
                    continue;
                }
                if (tid == 0) {  // read by warp 0 (thread 0 first) and, after the chunk, by count_dropped
                    c_dk0 = distk;
                    n_eff = 0;
                }
                int r0 = 0;
                while (r0 < cn) {
                    const float dk = distk;
                    const int sz = pool_size;
                    for (int r = r0 + w; r < cn; r += kScanWarps) {
                        int c;
                        const bool e = record_effect(S, buf + (size_t)r * RW, dk, sz, topk, c);
                        if (lane == 0) {
                            eff[r] = e;
                            cnt[r] = c;
                        }
                    }
                    __syncthreads();
                    if (w == 0) {
                        const bool mine = lane >= r0 && lane < cn;
                        const uint32_t hit = __ballot_sync(kFull, mine && eff[lane]);
                        const int rs = hit ? __ffs(hit) - 1 : cn;  // first record that changes the pool
                        int c = (lane >= r0 && lane < rs) ? cnt[lane] : 0;
                        for (int o = 16; o; o >>= 1) c += __shfl_xor_sync(kFull, c, o);
                        rr += (unsigned long long)c;
                        if (rs < cn) {
                            const float *rec = buf + (size_t)rs * RW;
                            const uint32_t *ri = reinterpret_cast<const uint32_t *>(rec);
                            float dkw = dk;
                            int szw = sz;
                            replay_block_warp(S, 0, rec + 8 + (S + 1), __uint_as_float(ri[7]), rec + 8 + (S + 1) + 32, ri[1],
                                              rec_ids(rec, S), sm.pool_id, sm.pool_d, szw, topk, dkw, rr);
                            if (lane == 0) {
                                distk = dkw;
                                pool_size = szw;
                                eff_pos[n_eff] = list[c0 + rs];
                                eff_dk[n_eff] = dkw;
                                ++n_eff;
                            }
                        }
                        if (lane == 0) s_next = rs + 1;
                    }
                    __syncthreads();
                    r0 = s_next;
                }
                if (counters && zf) {
                    count_dropped(k == 0 ? base : list[c0 - 1] + 1, k + 1 == nch ? wend : list[c0 + cn - 1] + 1);
                    __syncthreads();
                }
            }
        }
        __syncthreads();
        if (tid == 0 && counters) atomicAdd(counters + 2, rr);
        if (st.final_level) {
            write_results(sm, pool_size, topk, k_max, out_ids + (size_t)qi * k_max,
                          out_d ? out_d + (size_t)qi * k_max : nullptr);
        } else {  // the pool and its distk carry over to the next level
            for (int i = tid; i < topk; i += blockDim.x) {
                st.pool_id[(size_t)slot * k_max + i] = sm.pool_id[i];
                st.pool_d[(size_t)slot * k_max + i] = sm.pool_d[i];
            }
            if (tid == 0) {
                st.pool_size[slot] = pool_size;
                st.tau[slot] = distk;
            }
        }
        __syncthreads();  // the next slot reuses the shared state
    }
}

// One CTA per query: the whole probe list sequentially (queries deferred to
// the split pass are skipped).
template <bool kOne>
__global__ void __launch_bounds__(kScanThreads, kScanMinCtas) k_scan(DevIndexView ix, const uint32_t *__restrict__ probe,
                                                       QueryShape qsh, const float *__restrict__ qrot_all,
                                                       const float *__restrict__ prune_all,
                                                       uint32_t *__restrict__ out_ids, float *__restrict__ out_d,
                                                       unsigned long long *__restrict__ counters, int xstride,
                                                       const uint8_t *__restrict__ deferred,
                                                       const int *__restrict__ order, Prepared prep) {
    extern __shared__ __align__(16) char smem_raw[];
    const int qi = order ? order[blockIdx.x] : (int)blockIdx.x;
    if (deferred && deferred[qi]) return;  // answered by the split pass
    const int np = qsh.np_of(qi), topk = qsh.k_of(qi);
    ScanSmem sm = scan_smem_layout(smem_raw, ix.Dtot, ix.S, qsh.k_max, xstride);
    __shared__ int pool_size;
    __shared__ float distk;
    ScanTally tl;
    tl.counted = counters != nullptr;
    init_pool(sm, topk, pool_size, distk);
    scan_probes<kOne>(ix, probe + (size_t)qi * qsh.np_max, np, qrot_all + (size_t)qi * ix.Dtot,
                      prune_all + (size_t)qi * ix.S, topk, sm, pool_size, distk, tl,
                      prep.has(qi) ? prep.lut_of(qi, 0, ix.Dtot) : nullptr,
                      prep.has(qi) ? prep.scal_of(qi, 0, ix.S) : nullptr);
    flush_tally(tl, counters);
    write_results(sm, pool_size, topk, qsh.k_max, out_ids + (size_t)qi * qsh.k_max,
                  out_d ? out_d + (size_t)qi * qsh.k_max : nullptr);
}

// Launch order of the CTA scan, heaviest queries first (blocks of their probes,
// in power-of-two classes; the order inside a class is arbitrary), so that a
// long query does not start in the last wave; the split pass's queries (deferred)
// last, as their CTAs only return.  One CTA of kOrderThreads.
constexpr int kOrderThreads = 1024;
constexpr int kOrderMinQueries = 1024;  // batches from which the CTA scan is launched heaviest first
__global__ void __launch_bounds__(kOrderThreads) k_order(DevIndexView ix, const uint32_t *__restrict__ probe, QueryShape qsh,
                                                         int nq, const int *__restrict__ qblocks,
                                                         const uint8_t *__restrict__ deferred,
                                                         int *__restrict__ order) {
    __shared__ int cnt[33], cur[33];
    const int tid = threadIdx.x;
    if (tid < 33) cnt[tid] = 0;
    __syncthreads();
    auto cls = [&](int qi) {
        if (deferred && deferred[qi]) return 32;
        int64_t total = 0;
        if (qblocks) {
            total = qblocks[qi];
        } else {
            const int np = qsh.np_of(qi);
            for (int p = 0; p < np; ++p) {
                const int c = (int)probe[(size_t)qi * qsh.np_max + p];
                total += ix.blk_off[c + 1] - ix.blk_off[c];
            }
        }
        return 31 - min(31, 63 - __clzll((long long)total + 1));  // heavier: smaller class
    };
    for (int qi = tid; qi < nq; qi += kOrderThreads) atomicAdd(&cnt[cls(qi)], 1);
    __syncthreads();
    if (tid == 0) {
        int acc = 0;
        for (int k = 0; k < 33; ++k) {
            cur[k] = acc;
            acc += cnt[k];
        }
    }
    __syncthreads();
    for (int qi = tid; qi < nq; qi += kOrderThreads) order[atomicAdd(&cur[cls(qi)], 1)] = qi;
}

// Puts the queries whose probes hold more than `defer_blocks` blocks (giant Zipf
// clusters; every query when defer_blocks < 0) on the split list, each with
// record positions for all its blocks, heaviest first while the record space
// lasts: queries in power-of-two classes of their blocks, heavy classes first,
// in query order inside a class.  What does not fit is left to the CTA scan,
// which then holds the lighter queries.  Writes every query's block count
// (qblocks: the CTA scan's launch order) unless k_qblocks has (have_qblocks).
// One CTA of up to kDeferThreads (a multiple of 32); thread t owns the queries
// [t * per, (t + 1) * per).
constexpr int kDeferThreads = 1024;
constexpr int kQblocksMinQueries = 256;  // from this batch size the block counts come from k_qblocks

// Blocks of a query's probes (at most INT_MAX), by a warp.
__device__ __forceinline__ int query_blocks(const DevIndexView &ix, const uint32_t *__restrict__ probe,
                                            const QueryShape &qsh, int qi) {
    const int lane = threadIdx.x & 31, np = qsh.np_of(qi);
    long long total = 0;
    for (int p = lane; p < np; p += 32) {
        const int c = (int)probe[(size_t)qi * qsh.np_max + p];
        total += ix.blk_off[c + 1] - ix.blk_off[c];
    }
#pragma unroll
    for (int o = 16; o; o >>= 1) total += __shfl_xor_sync(kFull, total, o);
    return total < (long long)INT_MAX ? (int)total : INT_MAX;
}

// Blocks of each query's probes, one warp per query (k_defer's input for
// large batches, where its single CTA would sum them one after the other).
__global__ void __launch_bounds__(256) k_qblocks(DevIndexView ix, const uint32_t *__restrict__ probe, QueryShape qsh,
                                                 int nq, int *__restrict__ qblocks) {
    const int qi = blockIdx.x * 8 + (threadIdx.x >> 5);
    if (qi >= nq) return;
    const int total = query_blocks(ix, probe, qsh, qi);
    if ((threadIdx.x & 31) == 0) qblocks[qi] = total;
}

__global__ void __launch_bounds__(kDeferThreads) k_defer(DevIndexView ix, const uint32_t *__restrict__ probe, int nq,
                                                         int defer_blocks, int resident, SplitState st,
                                                         int *__restrict__ qblocks, int have_qblocks,
                                                         uint8_t *__restrict__ deferred) {
    __shared__ long long wsum_b[kDeferThreads / 32];
    __shared__ int wsum_n[kDeferThreads / 32], wmost[kDeferThreads / 32], hist[32];
    __shared__ long long s_base;  // record positions handed out
    __shared__ int s_slot;        // list entries handed out
    const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5, nt = blockDim.x, nw = nt >> 5;
    const int per = (nq + nt - 1) / nt, q0 = min(nq, tid * per), q1 = min(nq, q0 + per);
    if (!have_qblocks) {
        for (int qi = w; qi < nq; qi += nw) {
            const int total = query_blocks(ix, probe, st.qsh, qi);
            if (lane == 0) qblocks[qi] = total;
        }
        __syncthreads();
    }
    if (resident > 0) {  // the built-in line: the batch as a whole decides first (kDeferBlocks)
        long long sum = 0;
        int most = 0, over = 0;
        for (int qi = q0; qi < q1; ++qi) {
            sum += qblocks[qi];
            most = max(most, qblocks[qi]);
            over += qblocks[qi] > defer_blocks;
        }
#pragma unroll
        for (int o = 16; o; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
        most = __reduce_max_sync(0xffffffffu, most);
        over = __reduce_add_sync(0xffffffffu, over);
        if (lane == 0) {
            wsum_b[w] = sum;
            wsum_n[w] = over;
            wmost[w] = most;
        }
        __syncthreads();
        sum = over = 0;
        for (int i = 0; i < nw; ++i) {
            sum += wsum_b[i];
            over += wsum_n[i];
            most = max(most, wmost[i]);
        }
        const bool even = 4LL * most * resident <= 5 * sum;  // no query is much longer than a CTA's share
        if (2 * over > nq || (!even && 10LL * over >= 3LL * nq)) defer_blocks = -1;
        else if (even) defer_blocks = 0;
        __syncthreads();  // the sums are used again
    }
    auto eligible = [&](int qi) {
        return defer_blocks < 0 || (defer_blocks > 0 && qblocks[qi] > defer_blocks);
    };
    auto cls = [&](int qi) { return 31 - min(31, 31 - __clz(qblocks[qi] + 1)); };  // heavier: smaller class
    if (tid < 32) hist[tid] = 0;
    if (tid == 0) {
        s_base = 0;
        s_slot = 0;
    }
    __syncthreads();
    for (int qi = q0; qi < q1; ++qi) {
        deferred[qi] = 0;
        if (eligible(qi)) atomicAdd(&hist[cls(qi)], 1);
    }
    __syncthreads();
    for (int c = 0; c < 32; ++c) {
        if (hist[c] == 0) continue;  // uniform: read after a barrier
        long long mine = 0;
        int cnt = 0;
        for (int qi = q0; qi < q1; ++qi)
            if (eligible(qi) && cls(qi) == c) {
                mine += qblocks[qi];
                ++cnt;
            }
        // exclusive prefix of (blocks, count) over the threads, in thread order
        long long xb = mine;
        int xn = cnt;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const long long yb = __shfl_up_sync(0xffffffffu, xb, o);
            const int yn = __shfl_up_sync(0xffffffffu, xn, o);
            if (lane >= o) {
                xb += yb;
                xn += yn;
            }
        }
        if (lane == 31) {
            wsum_b[w] = xb;
            wsum_n[w] = xn;
        }
        __syncthreads();
        long long before_b = xb - mine;
        int before_n = xn - cnt;
        for (int i = 0; i < w; ++i) {  // the warps before this one
            before_b += wsum_b[i];
            before_n += wsum_n[i];
        }
        const long long base = s_base;
        const int slot0 = s_slot;
        __syncthreads();  // every thread has read s_base / s_slot and the warp sums
        // the accepted queries of the class are a prefix of its order: positions grow along it
        long long acc_b = 0;
        int acc_n = 0;
        long long pos = base + before_b;
        int k = before_n;
        for (int qi = q0; qi < q1; ++qi) {
            if (!eligible(qi) || cls(qi) != c) continue;
            const int t = qblocks[qi];
            if (pos + t > st.pos_cap) break;
            const int slot = slot0 + k;
            st.qlist[slot] = qi;
            st.pos_off[slot] = pos;
            st.npos[slot] = t;
            deferred[qi] = 1;
            pos += t;
            ++k;
            acc_b += t;
            ++acc_n;
        }
        // the class's accepted blocks and queries
#pragma unroll
        for (int o = 16; o; o >>= 1) {
            acc_b += __shfl_xor_sync(0xffffffffu, acc_b, o);
            acc_n += __shfl_xor_sync(0xffffffffu, acc_n, o);
        }
        if (lane == 0) {
            wsum_b[w] = acc_b;
            wsum_n[w] = acc_n;
        }
        __syncthreads();
        if (tid == 0) {
            for (int i = 0; i < nw; ++i) {
                s_base += wsum_b[i];
                s_slot += wsum_n[i];
            }
        }
        __syncthreads();
    }
    if (tid == 0) {
        *st.nlist = s_slot;
        *st.pos_used = (unsigned long long)s_base;
    }
}

// ------------------------------------------------------------------ estimate
// IVF::estimate: every vector of the probed clusters (no pruning); one CTA per
// kEstBlocks blocks of a probed cluster (tiles: probe and first block), outputs at the cluster's offset in
// probe order.  A CTA per cluster waited for the largest: 250,007 vectors in 1,024 clusters of
// Zipf sizes took 4.9 ms, now 0.15 with tiles of 16 blocks (two per warp, against the
// 4 us in which a CTA builds its cluster's LUT).
constexpr int kEstBlocks = 16;
__global__ void __launch_bounds__(kScanThreads) k_estimate(DevIndexView ix, const uint32_t *__restrict__ probe,
                                                           const int2 *__restrict__ tiles,
                                                           const int64_t *__restrict__ out_off,
                                                           const float *__restrict__ qrot,
                                                           const float *__restrict__ prune, uint32_t *__restrict__ o_ids,
                                                           float *__restrict__ o_acc, float *__restrict__ o_fast,
                                                           float *__restrict__ o_vars, int xstride) {
    extern __shared__ __align__(16) char smem_raw[];
    const int S = ix.S;
    ScanSmem sm = scan_smem_layout(smem_raw, ix.Dtot, S, 1, xstride);
    const int2 tile = tiles[blockIdx.x];
    const int p = tile.x, c = (int)probe[p];
    const int tid = threadIdx.x, w = tid >> 5, lane = tid & 31;
    prepare_cluster(ix, qrot, prune, c, sm);
    const int64_t b0 = ix.blk_off[c], v0 = ix.vec_off[c];
    const int nb = (int)(ix.blk_off[c + 1] - b0), n = (int)(ix.vec_off[c + 1] - v0);
    const int64_t base = out_off[p];
    for (int b = tile.y + w; b < min(nb, tile.y + kEstBlocks); b += kScanWarps) {
        const int64_t gb = b0 + b;
        float fsum = 0.0f, vsum = 0.0f;
        for (int s = 0; s < S; ++s) {
            const SegDev &g = ix.seg[s];
            const float on = g.onorm[gb * 32 + lane];
            const float v = vars_est(sm.scal[s], on);
            float ipx = 0.0f;
            const float f = g.bits ? fast_est(g, sm.lut + 4 * g.qoff, sm.scal[s], gb, lane, on, ipx) : v;
            sm.ipx[(w * S + s) * 32 + lane] = ipx;
            fsum = __fadd_rn(fsum, f);
            vsum = __fadd_rn(vsum, v);
        }
        __syncwarp();
        const int nv = min(32, n - b * 32);
        if (lane < nv) {  // one thread per vector, all segments in order
            const int64_t gv = v0 + (int64_t)b * 32 + lane;
            float acc = 0.0f;
            for (int s = 0; s < S; ++s) {
                const SegDev &g = ix.seg[s];
                const float ex = g.bits > 1 ? excode_ip_thread(sm.qres + g.qoff, g.lcode + (size_t)gv * g.lstride,
                                                               g.dim, g.bits - 1)
                                            : 0.0f;
                acc = __fadd_rn(acc, accurate_dist(g.onorm[gb * 32 + lane], sm.ipx[(w * S + s) * 32 + lane], ex,
                                                   g.exfac[gv].x, g.bits, sm.scal[s].sum_q, sm.scal[s].q_l2sqr));
            }
            const int64_t o = base + (int64_t)b * 32 + lane;
            o_ids[o] = ix.ids[gv];
            o_acc[o] = acc;
            o_fast[o] = fsum;
            o_vars[o] = vsum;
        }
        __syncwarp();
    }
}

struct Bump {
    char *base;
    size_t off = 0;
    template <class T>
    T *take(size_t count) {
        off = align16(off);
        T *p = reinterpret_cast<T *>(base + off);
        off += sizeof(T) * count;
        return p;
    }
};

// List entries of the split pass that get the batched preparation: as many as
// kPrepCap holds (nprobe pairs each), at most nq; 0 below kPrepMinQueries
// queries, where the scan CTAs build each cluster's state in the shorter latency
// (256 threads per LUT).  12 GB holds every query of a 4,096-query batch at
// nprobe 256 with D = 1024 (8.8 GB; the CTA scan's copy is as large
// again), a few percent of the device beside the index.
constexpr size_t kPrepCap = (size_t)12 << 30;
constexpr int64_t kPrepMinQueries = 64;
size_t prep_pair_bytes(const Index &I) { return 8 * (size_t)I.view.Dtot + sizeof(SegScal) * I.view.S; }
int64_t prep_slots(const Index &I, int64_t nq, int64_t nprobe) {
    if (nq < kPrepMinQueries) return 0;
    return std::min<int64_t>(nq, (int64_t)(kPrepCap / (prep_pair_bytes(I) * (size_t)nprobe)));
}
size_t prep_bytes(const Index &I, int64_t nq, int64_t nprobe) {
    const size_t pairs = (size_t)prep_slots(I, nq, nprobe) * nprobe;
    return pairs ? align16(pairs * 8 * (size_t)I.view.Dtot) + align16(pairs * sizeof(SegScal) * I.view.S) : 0;
}

size_t search_scratch_bytes(const Index &I, int64_t nq, int64_t topk, int64_t nprobe, bool host_io) {
    size_t b = 0;
    auto add = [&](size_t x) { b += align16(x); };
    add(4 * (size_t)nq * I.D);                 // queries (host io)
    add(4 * (size_t)nq * I.K);                 // centroid distances
    add(8 * (size_t)nq * I.K);                 // exact-select work (fallback)
    add(4 * (size_t)nq * nprobe);              // probe ids
    add(4 * (size_t)nq * I.view.Dtot);         // rotated queries
    add(4 * (size_t)nq * I.view.S);            // prune bounds
    add(2 * (size_t)nq * I.D);                 // BF16 queries (probe GEMM)
    add((size_t)nq);                           // shortlist: queries on the full exact path
    add(4 * (size_t)nq);                       // ... and their list
    add(4 * (size_t)nq);                       // CTA scan launch order
    add(4 * (size_t)nq * topk * 2);            // outputs (host io)
    add(4 * (size_t)nq * 2);                   // per-query nprobe / k
    add(64);                                   // flags
    add(64);                                   // counters
    add(prep_bytes(I, nq, nprobe));            // prepared LUTs of the split list
    if (prep_slots(I, nq, nprobe) == nq) add(prep_bytes(I, nq, nprobe));  // ... and of the CTA scan's
    (void)host_io;
    return b + 256;
}

size_t split_scratch_bytes(const Index &I, int64_t cap, int64_t topk, int64_t nprobe, int64_t pos_cap) {
    size_t b = 0;
    auto add = [&](size_t x) { b += align16(x); };
    add(4 * 16);                                 // nlist, pos_used, work_next
    add(4 * (size_t)cap);                        // qlist
    add(4 * (size_t)cap * topk);
    add(4 * (size_t)cap * topk);
    add(4 * (size_t)cap);
    add(4 * (size_t)cap);
    add(4 * (size_t)cap * (nprobe + 1));
    add(4 * (size_t)cap * nprobe);
    add(8 * (size_t)cap);                        // split_p, split_b
    add(4 * (size_t)(cap + 1));
    add(4 * (size_t)cap);                        // npos
    add(8 * (size_t)cap);                        // pos_off
    add(16 * (size_t)pos_cap);                   // record summaries
    add(4 * (size_t)pos_cap * rec_words_of(I.view.S));
    add((size_t)cap);                            // deferred flags, one per query
    add(4 * (size_t)cap);                        // blocks of each query's probes
    return b + 256;
}

// A record and its summary.
size_t record_bytes(const Index &I) { return 4 * (size_t)rec_words_of(I.view.S) + 16; }

// Record positions of the split pass for a batch: every block of every query
// (`want`), bounded by scratch memory.
int64_t split_positions(const Index &I, int64_t want) {
    const size_t per = record_bytes(I);
    // 12 GB: with 8 GB a batch of 4,096 queries with nprobe up to 256 over 10M vectors leaves
    // some of its heaviest queries to the CTA scan (43.9 ms a batch, 39.7 from 10 GB on)
    size_t budget = (size_t)12 << 30;
    if (const char *e = std::getenv("SAQG_SPLIT_RECORD_BYTES"))  // tests: a small budget forces the overflow path
        budget = std::max<size_t>(per, (size_t)std::atoll(e));
    const int64_t by_mem = (int64_t)(budget / per);
    return std::max<int64_t>(1, std::min(want, by_mem));
}

// The split pass's scratch in the context, for as many record positions of `want` (out:
// pos_cap) as the budget, the context's limit and the device have room for.  Queries that
// the records do not reach stay with the CTA scan, so a device short of memory answers a
// call more slowly instead of refusing it.  While `st` is captured, what the context holds
// is all there is.
char *split_scratch_take(const Index &I, SearchCtx &C, int64_t cap, int64_t topk, int64_t nprobe, int64_t want,
                         int64_t &pos_cap, cudaStream_t st) {
    auto bytes = [&] { return split_scratch_bytes(I, cap, topk, nprobe, pos_cap); };
    pos_cap = split_positions(I, want);
    if (bytes() > C.split_scratch_bytes) {
        cudaStreamCaptureStatus capture = cudaStreamCaptureStatusNone;
        if (cudaStreamIsCapturing(st, &capture) != cudaSuccess) cudaGetLastError();
        const bool fixed = capture != cudaStreamCaptureStatusNone && C.split_scratch;
        const size_t limit = fixed ? C.split_scratch_bytes : std::max(C.split_limit, C.split_scratch_bytes);
        if (bytes() > limit) {  // as many as fit below it
            const size_t over = bytes() - limit;
            pos_cap = std::max<int64_t>(1, pos_cap - (int64_t)(over / record_bytes(I)) - 1);
        }
        for (; pos_cap > 1; pos_cap /= 2)
            if (C.split_scratch_try(bytes())) break;
    }
    return static_cast<char *>(C.split_scratch_get(bytes()));
}

constexpr int64_t kFewQueries = 16;  // calls of up to so many take the split scan

// Which exact scan serves a call: the split scan for latency-bound calls (few
// queries), one CTA per query for batches, unless the tuned shape says
// otherwise.  SAQG_SCAN_MODE=seq|split|warp forces one (tests).
// 0: one CTA per query, 1: split scan, 2: one warp per query.
int scan_mode(int64_t nq, int64_t topk, const ScanTune &t) {
    const char *m = std::getenv("SAQG_SCAN_MODE");
    if (m && std::string(m) == "seq") return 0;
    if (m && std::string(m) == "split") return 1;
    if (m && std::string(m) == "warp") return topk <= 256 ? 2 : 0;
    if (m && std::string(m) == "ws") return 0;
    if (t.mode == 0 || t.mode == 1) return t.mode;
    if (t.mode == 3) return 0;
    if (t.mode == 2) return topk <= 256 ? 2 : 0;
    if (nq <= kFewQueries) return 1;
    return 0;
}

}  // namespace

// Blocks of a speculative tile: short ones for a few queries that have the GPU alone, so
// that they spread over it.  A batch on the split scan (tuned or forced) has tiles enough:
// 24 / 256 / 1,024 queries of an anisotropic 500,000 x 768 index 423 us / 2.45 / 8.91 ms
// with tiles of 4, 370 us / 1.75 / 5.86 ms with 16 (16 queries: 353 and 380 us).
int spec_tile_blocks(int mode, int64_t nq) {
    return mode == 1 && nq <= kFewQueries ? kFewTileBlocks : kTileBlocks;
}

namespace {

// Whether mode 0's CTA scan runs warp-specialised (scan mode 3).
bool scan_ws(const ScanTune &t) {
    if (const char *m = std::getenv("SAQG_SCAN_MODE")) return std::string(m) == "ws";
    return t.mode == 3;
}

// The deferral threshold of mode 0 (blocks of a query's probes above which it
// takes the split pass; 0: never), and whether it was given rather than built in.
bool defer_line_given(const ScanTune &t) { return t.defer_blocks >= 0 || std::getenv("SAQG_DEFER_BLOCKS"); }
int defer_threshold(const ScanTune &t) {
    int defer = t.defer_blocks >= 0 ? t.defer_blocks : kDeferBlocks;
    if (const char *e = std::getenv("SAQG_DEFER_BLOCKS")) defer = std::max(0, std::atoi(e));
    return defer;
}

// Whether no query of a mode-0 call is deferred: its nprobe largest clusters hold no more
// blocks than the threshold, or (built-in line, one nprobe for all: `even`) clusters of
// about one size give equally long queries that fill one wave of the CTA scan, which
// then ends everywhere at once (600 queries of 923 blocks, 400,000 x 576: 0.85 ms, 0.92
// with the split pass; 480 queries, three quarters of a wave: 0.88 and 0.85).
constexpr int kFullWave = 87, kEvenBlocks = 80;  // percent: of the resident CTAs; mean of the longest query
bool no_deferral(const Index &I, int64_t nq, int64_t nprobe, bool even, int resident, const ScanTune &t) {
    const int defer = defer_threshold(t);
    const int64_t most = I.max_blocks_of_probes(nprobe);
    if (defer == 0 || most <= defer) return true;
    return even && !defer_line_given(t) && nq <= resident && 100 * nq >= kFullWave * (int64_t)resident &&
           kEvenBlocks * most * I.K <= 100 * nprobe * I.blk_off[I.K];
}

// Per-query nprobe / k copies clamped to the call's maxima (graph launches read
// caller-written device arrays; an out-of-range value must not index past a row).
__global__ void k_clamp_shape(const int *__restrict__ np, const int *__restrict__ k, int nq, int np_max, int k_max,
                              int *__restrict__ np_out, int *__restrict__ k_out) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= nq) return;
    if (np) np_out[i] = min(max(np[i], 1), np_max);
    if (k) k_out[i] = min(max(k[i], 1), k_max);
}

int xstride_of(const DevIndexView &) { return 0; }  // re-rank reads ex-codes in place (no staging buffer)

void check_launch(const char *what) {
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) throw Error{SAQG_ERR_CUDA, std::string(what) + " launch failed: " + cudaGetErrorString(e)};
    count_launch(1);
}

// cudaFuncSetAttribute(MaxDynamicSharedMemorySize) once per (kernel, device)
// and size: a call's host time matters for single queries.
void ensure_smem(const void *fn, size_t bytes) {
    static std::mutex mu;
    static std::map<std::pair<const void *, int>, size_t> have;
    int dev = 0;
    SAQG_CUDA_TRY(cudaGetDevice(&dev));
    std::lock_guard<std::mutex> lk(mu);
    size_t &h = have[{fn, dev}];
    if (bytes <= h) return;
    SAQG_CUDA_TRY(cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes));
    h = bytes;
}

// The CTA scan for an index of S segments.
auto scan_kernel(int S) { return S == 1 ? k_scan<true> : k_scan<false>; }

// The CTA-per-query scan of `nq` queries (deferred ones skipped): k_scan, with
// the batched LUTs that prep_of(deferred) launches and returns (or none), or its
// warp-specialised form k_scan_ws, which gives the same answers.
void launch_cta_scan(bool ws, const DevIndexView &ix, const uint32_t *probe, const QueryShape &qsh, const float *qrot,
                     const float *prune, uint32_t *ids, float *d, unsigned long long *cnt, int xs,
                     const uint8_t *deferred, int64_t nq, int *order, const int *qblocks,
                     const std::function<Prepared(const uint8_t *)> &prep_of, cudaStream_t st) {
    if (order) {
        k_order<<<1, kOrderThreads, 0, st>>>(ix, probe, qsh, (int)nq, qblocks, deferred, order);
        check_launch("k_order");
    }
    if (ws) {
        const size_t smem = ws_smem_bytes(ix.Dtot, ix.S, qsh.k_max, xs);
        SAQG_REQUIRE(smem <= kScanWsSmem, "dimension / topk too large for the scan kernel's shared memory");
        ensure_smem((const void *)k_scan_ws, smem);
        k_scan_ws<<<(unsigned)nq, kScanThreads, smem, st>>>(ix, probe, qsh, qrot, prune, ids, d, cnt, xs, deferred,
                                                             order);
        check_launch("k_scan_ws");
        return;
    }
    const size_t smem = scan_smem_bytes(ix.Dtot, ix.S, qsh.k_max, xs);
    SAQG_REQUIRE(smem <= kScanSmem, "dimension / topk too large for the scan kernel's shared memory");
    const auto scan = scan_kernel(ix.S);
    ensure_smem((const void *)scan, smem);
    const Prepared prep = prep_of(deferred);
    scan<<<(unsigned)nq, kScanThreads, smem, st>>>(ix, probe, qsh, qrot, prune, ids, d, cnt, xs, deferred, order,
                                                      prep);
    check_launch("k_scan");
}

// SMs x resident CTAs of a kernel (per device and shared-memory size), cached.
// Streaming multiprocessors of the current device, cached.
int sm_count() {
    static std::mutex mu;
    static std::map<int, int> have;
    int dev = 0;
    SAQG_CUDA_TRY(cudaGetDevice(&dev));
    std::lock_guard<std::mutex> lk(mu);
    auto it = have.find(dev);
    if (it != have.end()) return it->second;
    int sms = 0;
    SAQG_CUDA_TRY(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    return have[dev] = std::max(1, sms);
}

int full_grid(const void *fn, int threads, size_t smem) {
    static std::mutex mu;
    static std::map<std::tuple<const void *, int, size_t>, int> have;
    int dev = 0;
    SAQG_CUDA_TRY(cudaGetDevice(&dev));
    std::lock_guard<std::mutex> lk(mu);
    auto it = have.find({fn, dev, smem});
    if (it != have.end()) return it->second;
    int sms = 0, per_sm = 0;
    SAQG_CUDA_TRY(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    SAQG_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, fn, threads, smem));
    const int g = std::max(1, sms * std::max(1, per_sm));
    have[{fn, dev, smem}] = g;
    return g;
}

// CTAs of the CTA scan that the GPU holds at once.
int resident_scans(int S, size_t smem) {
    const auto scan = scan_kernel(S);
    ensure_smem((const void *)scan, smem);
    return full_grid((const void *)scan, kScanThreads, smem);
}

// Prune bounds and rotated queries of a call on `st`.  k_qprep_few spreads over the
// GPU but reads the matrices once per 8 queries, k_qprep_tiled reads them once per
// 128 and needs a chain of the longest segment's length: up to kQprepFewWork
// query-matrix elements the former is faster.  Segments (64, 320, 640): 64 queries
// 12 against 49 us, 512: 45 against 50, 1,024: 80 against 75; one of 1,536: 128
// queries 68 against 106 us, 256: 124 against 108.
constexpr int64_t kQprepFewWork = 400000000;
void launch_qprep(const DevIndexView &ix, const float *q, int64_t nq, float m, float *qrot, float *prune,
                  cudaStream_t st) {
    int dmax = 0;
    int64_t elems = 0;
    for (int s = 0; s < ix.S; ++s) {
        dmax = std::max(dmax, ix.seg[s].dim);
        elems += (int64_t)ix.seg[s].dim * ix.seg[s].dim;
    }
    const int few = (int)std::min<int64_t>(nq, kQprepFewQ);
    const size_t smem = qprep_few_smem(dmax, few);
    if (nq <= kQprepFewWork / elems && smem <= 200 * 1024) {
        ensure_smem((const void *)k_qprep_few, smem);
        k_qprep_few<<<dim3((unsigned)(dmax / kQprepOut), (unsigned)ix.S, (unsigned)((nq + kQprepFewQ - 1) / kQprepFewQ)),
                      kQprepFewThreads, smem, st>>>(ix, q, (int)nq, m, qrot, prune);
        check_launch("k_qprep_few");
        return;
    }
    const int vec = ((uintptr_t)q & 15) == 0 && ix.D % 4 == 0;
    k_qprep_tiled<<<dim3((unsigned)(dmax / kRotN), (unsigned)ix.S, (unsigned)((nq + kRotM - 1) / kRotM)), kRotThreads, 0,
                    st>>>(ix, q, (int)nq, vec, qrot);
    check_launch("k_qprep_tiled");
    k_prune_bounds<<<(unsigned)((nq * ix.S + 7) / 8), 256, 0, st>>>(ix, q, (int)nq, m, prune);
    check_launch("k_prune_bounds");
}

}  // namespace

int64_t tune_bucket(int64_t nq) {
    int64_t b = 1;
    while (b < nq) b <<= 1;
    return b;
}

void clamp_shape(const int *np, const int *k, int64_t nq, int np_max, int k_max, int *np_out, int *k_out,
                 cudaStream_t st) {
    if (nq <= 0 || (!np && !k)) return;
    k_clamp_shape<<<(unsigned)((nq + 255) / 256), 256, 0, st>>>(np, k, (int)nq, np_max, k_max, np_out, k_out);
    check_launch("k_clamp_shape");
}

namespace {


// Centroid ranking of a batch: BF16 GEMM of inner products, the shortlist
// kernel, and the full exact path for the queries it hands back.
void probe_shortlist(const Index &I, SearchCtx &C, const float *q, int64_t nq, int64_t nprobe, const int *qnp,
                     float *dist, uint32_t *probe, uint8_t *full, int *fb_list, int *flags, Cand *work,
                     unsigned long long *cnt, void *qbf, cudaStream_t st,
                     const std::function<void()> &after_gemm = nullptr) {
    const DevIndexView &ix = I.view;
    // upper-end keys kept in shared memory for the full radix select, which only
    // a query with nprobe > kShortThreads / 2 runs
    const bool keep = I.K <= kShortKeys && nprobe > kShortThreads / 2;
    const size_t smem = 12 * (size_t)kShortCap + 4 * (size_t)I.D + (keep ? 4 * (size_t)I.K : 0);
    // refused before any work is under way on another stream
    SAQG_REQUIRE(smem <= 220 * 1024, "dimension too large for the probe shortlist's shared memory");
    {
        std::lock_guard<std::mutex> lk(I.init_mu);
        if (!I.cnorm2) {
            float *p = nullptr;
            SAQG_CUDA_TRY(cudaMalloc(&p, 8 * (size_t)I.K));
            k_cnorm2<<<(unsigned)((I.K * 32 + 255) / 256), 256, 0, st>>>(ix, reinterpret_cast<float2 *>(p));
            check_launch("k_cnorm2");
            SAQG_CUDA_TRY(cudaStreamSynchronize(st));  // other contexts read it on their own streams
            I.cnorm2 = p;
        }
    }
    {
        std::lock_guard<std::mutex> lk(I.init_mu);
        if (!I.cent_bf16) {
            void *p = nullptr;
            SAQG_CUDA_TRY(cudaMalloc(&p, 2 * (size_t)I.K * I.D));
            to_bf16(ix.centroids, I.K * I.D, p, st);
            SAQG_CUDA_TRY(cudaStreamSynchronize(st));  // other contexts read it on their own streams
            I.cent_bf16 = p;
        }
    }
    // dist (row-major nq x K) = Q C^T on the tensor cores (BF16 operands rounded
    // to nearest, FP32 accumulation); flags[3] is set if a GEMM wait timed out
    to_bf16(q, nq * I.D, qbf, st);
    probe_ip_gemm(qbf, nq, I.cent_bf16, I.K, I.D, dist, flags + 3, st);
    // Work that can run beside the shortlist and its select.  The caller's stream
    // has the device's least (default) priority, like that work's, so the shortlist
    // and the select then move to the context's greatest-priority stream: their CTAs
    // go first and the side work fills the gaps.
    cudaStream_t ps = st;
    if (after_gemm) {
        after_gemm();
        ps = C.aux_stream();
        SAQG_CUDA_TRY(cudaEventRecord(C.fork_event(), st));
        SAQG_CUDA_TRY(cudaStreamWaitEvent(ps, C.fork_event(), 0));
    }
    const double u = 1.0 / 16777216.0;
    ShortBound sb;
    // BF16 operands lie within 2^-9 of their values: |q.c error| <= (2^-8 + 2^-18) |q||c| + accumulation
    sb.e1 = (float)(2.0 * (1.0 / 256 + 1.0 / 262144 + (double)(I.D + 2) * u));
    sb.e2 = (float)((2.0 * (double)I.D + 32.0) * u);
    // (first touched after the rotation's kernel: with the attribute set at the check above,
    // the two run beside one another 50 us slower, 2,048 queries of 1M x 1536 0.50 ms ranking
    // and rotation instead of 0.45 in every process)
    ensure_smem((const void *)k_probe_shortlist, (size_t)smem);
    k_probe_shortlist<<<(unsigned)nq, kShortThreads, smem, ps>>>(ix, q, dist, reinterpret_cast<const float2 *>(I.cnorm2),
                                                                 sb, (int)nprobe, qnp, probe, full,
                                                                 fb_list, flags + 2, cnt, flags + 3, keep ? 1 : 0);
    check_launch("k_probe_shortlist");
    k_probe_dist_list<<<608, 256, 0, ps>>>(ix, q, dist, fb_list, flags + 2);
    check_launch("k_probe_dist_list");
    k_probe_select<<<(unsigned)nq, kSelThreads, 0, ps>>>(dist, (int)I.K, (int)nprobe, probe, work, flags, full, qnp);
    check_launch("k_probe_select");
    if (ps != st) {
        SAQG_CUDA_TRY(cudaEventRecord(C.join_event(), ps));
        SAQG_CUDA_TRY(cudaStreamWaitEvent(st, C.join_event(), 0));
    }
}

}  // namespace

void presize_ctx(const Index &I, SearchCtx &C, int64_t nq, int64_t topk, int64_t nprobe) {
    std::lock_guard<std::mutex> lock(C.mu);
    C.scratch_get(search_scratch_bytes(I, nq, topk, nprobe, false));
    int64_t pos_cap = 0;
    split_scratch_take(I, C, nq, topk, nprobe, nq * I.max_blocks_of_probes(nprobe), pos_cap, nullptr);
    C.create_streams();
}

// Records for two thirds of the blocks, and 8 GB at most, are enough to admit a batch (the
// heaviest queries come first, the CTA scan takes those that are left without); a few
// queries, which the split pass answers alone, need them all.  The call itself takes up
// to all of them where its budget has them (split_limit).
size_t search_bytes_estimate(const Index &I, int64_t nq, int64_t topk, int64_t nprobe) {
    const int64_t all = split_positions(I, nq * I.max_blocks_of_probes(nprobe));
    const int64_t of_8gb = (int64_t)(((size_t)8 << 30) / record_bytes(I));
    const int64_t least = nq <= kFewQueries ? all : std::max<int64_t>(1, std::min(2 * all / 3, of_8gb));
    return search_scratch_bytes(I, nq, topk, nprobe, false) + split_scratch_bytes(I, nq, topk, nprobe, least);
}
size_t search_arena1_bytes(const Index &I, int64_t nq, int64_t topk, int64_t nprobe) {
    return search_scratch_bytes(I, nq, topk, nprobe, false);
}

void run_search(const Index &I, const float *q, int64_t nq, int64_t topk, int64_t nprobe, float m, uint32_t *ids,
                float *dists, int mem, cudaStream_t st, saqg_search_stats *stats, uint32_t *probes_out,
                const int *np_host, const int *k_host, SearchCtx *ctx, const SearchOpts *opts) {
    std::unique_ptr<CtxLease> lease;
    if (!ctx) {
        lease = std::make_unique<CtxLease>(I, st);  // locked; ordered after its previous call
        ctx = lease->c;
    }
    SearchCtx &C = *ctx;
    // per-query nprobe / k (host arrays): the scalars become their maxima
    int64_t sum_np = nq * nprobe;
    if (np_host || k_host) {
        int64_t npm = 0, km = 0;
        sum_np = 0;
        for (int64_t i = 0; i < nq; ++i) {
            const int a = np_host ? np_host[i] : (int)nprobe, b = k_host ? k_host[i] : (int)topk;
            SAQG_REQUIRE(a >= 1 && a <= I.K, "every nprobe must be in [1, number of clusters]");
            SAQG_REQUIRE(b >= 1 && b <= kMaxTopK, "every topk must be in [1, 4096]");
            npm = std::max<int64_t>(npm, a);
            km = std::max<int64_t>(km, b);
            sum_np += a;
        }
        if (np_host) nprobe = npm;
        if (k_host) topk = km;
    }
    SAQG_REQUIRE(nq >= 0 && topk >= 1 && topk <= kMaxTopK, "topk must be in [1, 4096]");
    SAQG_REQUIRE(nprobe >= 1 && nprobe <= I.K, "nprobe must be in [1, number of clusters]");
    if (nq == 0) return;
    const DevIndexView &ix = I.view;
    std::unique_lock<std::mutex> lock(C.mu, std::defer_lock);
    if (!lease) lock.lock();  // a caller's own context (graph, serving slot)
    const bool host = mem == SAQG_MEM_HOST;
    Bump bp{(char *)C.scratch_get(search_scratch_bytes(I, nq, topk, nprobe, host))};
    QueryShape qsh;
    qsh.np_max = (int)nprobe;
    qsh.k_max = (int)topk;
    if (np_host) {
        int *d = bp.take<int>(nq);
        SAQG_CUDA_TRY(cudaMemcpyAsync(d, np_host, 4 * (size_t)nq, cudaMemcpyHostToDevice, st));
        qsh.np = d;
    }
    if (k_host) {
        int *d = bp.take<int>(nq);
        SAQG_CUDA_TRY(cudaMemcpyAsync(d, k_host, 4 * (size_t)nq, cudaMemcpyHostToDevice, st));
        qsh.k = d;
    }
    if (!np_host && !k_host && opts && (opts->np_dev || opts->k_dev)) {  // device arrays: clamped copies
        int *dn = opts->np_dev ? bp.take<int>(nq) : nullptr;
        int *dk = opts->k_dev ? bp.take<int>(nq) : nullptr;
        clamp_shape(opts->np_dev, opts->k_dev, nq, (int)nprobe, (int)topk, dn, dk, st);
        qsh.np = dn;
        qsh.k = dk;
    }
    // launch shapes: the caller's, else the autotuner's choice for this shape, else built-in
    ScanTune tune;
    if (opts && opts->tune) {
        tune = *opts->tune;
    } else {
        std::lock_guard<std::mutex> lk(I.tune_mu);
        const auto it = I.scan_tunes.find(TuneKey{0, tune_bucket(nq), topk, nprobe});
        if (it != I.scan_tunes.end()) tune = it->second;
    }
    float *dq = bp.take<float>((size_t)nq * I.D);
    float *dist = bp.take<float>((size_t)nq * I.K);
    Cand *work = bp.take<Cand>((size_t)nq * I.K);
    uint32_t *probe = bp.take<uint32_t>((size_t)nq * nprobe);
    float *qrot = bp.take<float>((size_t)nq * ix.Dtot);
    float *prune = bp.take<float>((size_t)nq * ix.S);
    void *qbf = bp.take<uint16_t>((size_t)nq * I.D);
    uint8_t *full = bp.take<uint8_t>((size_t)nq);
    int *fb_list = bp.take<int>((size_t)nq);
    // heaviest queries first once the CTA scan runs in several waves
    int *order = nq >= kOrderMinQueries ? bp.take<int>((size_t)nq) : nullptr;
    uint32_t *oid = bp.take<uint32_t>((size_t)nq * topk);
    float *od = bp.take<float>((size_t)nq * topk);
    int *flags = bp.take<int>(16);
    unsigned long long *counters = bp.take<unsigned long long>(8);
    const int64_t pslots = prep_slots(I, nq, nprobe);
    uint16_t *prep_lut = pslots ? bp.take<uint16_t>((size_t)pslots * nprobe * 4 * ix.Dtot) : nullptr;
    SegScal *prep_scal = pslots ? bp.take<SegScal>((size_t)pslots * nprobe * ix.S) : nullptr;
    const bool scan_prep_fits = pslots > 0 && pslots == nq;
    uint16_t *scan_lut = scan_prep_fits ? bp.take<uint16_t>((size_t)nq * nprobe * 4 * ix.Dtot) : nullptr;
    SegScal *scan_scal = scan_prep_fits ? bp.take<SegScal>((size_t)nq * nprobe * ix.S) : nullptr;
    cudaEvent_t ev[7] = {};
    bool shortlist = false;  // centroid ranking by the GEMM shortlist
    if (stats)
        for (auto &e : ev) SAQG_CUDA_TRY(cudaEventCreate(&e));
    struct EvGuard {
        cudaEvent_t *e;
        ~EvGuard() {
            for (int i = 0; i < 7; ++i)
                if (e[i]) cudaEventDestroy(e[i]);
        }
    } evg{ev};
    const float *qin = q;
    if (host) {
        SAQG_CUDA_TRY(cudaMemcpyAsync(dq, q, 4 * (size_t)nq * I.D, cudaMemcpyHostToDevice, st));
        qin = dq;
    }
    SAQG_CUDA_TRY(cudaMemsetAsync(flags, 0, 64, st));
    if (stats) SAQG_CUDA_TRY(cudaMemsetAsync(counters, 0, 64, st));
    {
        const int wpb = 8;
        dim3 grid((unsigned)((I.K + wpb - 1) / wpb), (unsigned)nq);
        if (stats) SAQG_CUDA_TRY(cudaEventRecord(ev[0], st));
        // query preparation (rotation, prune bounds) depends on the queries alone:
        // it runs on the context's least-priority stream beside the centroid ranking
        // (beside the shortlist and its select when the GEMM ranks the centroids:
        // the GEMM wants whole SMs; those two then run at the greatest priority,
        // so their CTAs go first)
        auto fork_qprep = [&]() {
            cudaStream_t qs = C.low_stream();
            SAQG_CUDA_TRY(cudaEventRecord(C.qfork_event(), st));
            SAQG_CUDA_TRY(cudaStreamWaitEvent(qs, C.qfork_event(), 0));
            launch_qprep(ix, qin, nq, m, qrot, prune, qs);
            SAQG_CUDA_TRY(cudaEventRecord(C.qjoin_event(), qs));
        };
        const char *pm = std::getenv("SAQG_PROBE");
        shortlist = nq >= kGemmMinQueries && nprobe <= kShortCap && !(pm && std::string(pm) == "exact");
        if (!shortlist) fork_qprep();
        if (shortlist) {
            probe_shortlist(I, C, qin, nq, nprobe, qsh.np, dist, probe, full, fb_list, flags, work,
                            stats ? counters : nullptr, qbf, st, fork_qprep);
        } else if (nq >= 8 && I.D % 32 == 0 && I.D <= 32 * kProbeRegs) {
            const size_t qsm = 4 * (size_t)kProbeQT * I.D;
            ensure_smem((const void *)k_probe_dist_tiled, (size_t)qsm);
            const unsigned gx = (unsigned)std::min<int64_t>((I.K + kProbeWarps - 1) / kProbeWarps, 304);
            k_probe_dist_tiled<<<dim3(gx, (unsigned)((nq + kProbeQT - 1) / kProbeQT)), kProbeWarps * 32, qsm, st>>>(
                ix, qin, (int)nq, dist);
            check_launch("k_probe_dist_tiled");
        } else {
            k_probe_dist<<<grid, wpb * 32, 0, st>>>(ix, qin, dist);
            check_launch("k_probe_dist");
        }
        if (!shortlist) {
            k_probe_select<<<(unsigned)nq, kSelThreads, 0, st>>>(dist, (int)I.K, (int)nprobe, probe, work, flags,
                                                                  nullptr, qsh.np);
            check_launch("k_probe_select");
        }
        if (stats) SAQG_CUDA_TRY(cudaEventRecord(ev[1], st));
        SAQG_CUDA_TRY(cudaStreamWaitEvent(st, C.qjoin_event(), 0));  // the rotated queries
        if (stats) SAQG_CUDA_TRY(cudaEventRecord(ev[2], st));
        const int xs = xstride_of(ix);
        const size_t smem = scan_smem_bytes(ix.Dtot, ix.S, (int)topk, xs);
        SAQG_REQUIRE(smem <= kScanSmem, "dimension / topk too large for the scan kernel's shared memory");
        uint32_t *ids_out = host ? oid : ids;
        float *d_out = host ? od : dists;
        unsigned long long *cnt = stats ? counters : nullptr;
        const int mode0 = scan_mode(nq, topk, tune);
        const int mode = (qsh.np || qsh.k) && mode0 == 2 ? 0 : mode0;
        // The CTA scan's queries get batched LUTs too (by query; on the caller's stream,
        // after the split pass has forked, so it overlaps the split pass's start) when
        // the budget holds every query's.  A CTA that builds the LUTs of the probes that
        // stage 0 leaves does less work where that is one in four (10M / 16,384 Zipf clusters,
        // 4,096 queries: 1.93 ms against 1.98) but loses where most are left: 647,483
        // vectors in 6,497 clusters, 1,088 queries, 3.21 ms against 2.85, 600 on an anisotropic set 2.46 against 2.12.
        const std::function<Prepared(const uint8_t *)> scan_prep = [&](const uint8_t *skip) {  // skip: queries left out
            Prepared pp;
            if (!scan_lut || scan_ws(tune)) return pp;
            const size_t lsm = 4 * (size_t)kLutWarps * ix.Dtot;
            SAQG_REQUIRE(lsm <= 200 * 1024, "dimension too large for the batched LUT preparation");
            ensure_smem((const void *)k_lut, lsm);
            const int64_t items = nq * nprobe;
            k_lut<<<(unsigned)((items + kLutWarps - 1) / kLutWarps), kLutWarps * 32, lsm, st>>>(
                ix, probe, qsh, nullptr, nullptr, (int)nq, skip, qrot, prune, scan_lut, scan_scal);
            check_launch("k_lut");
            pp.lut = scan_lut;
            pp.scal = scan_scal;
            pp.np_max = (int)nprobe;
            pp.slots = (int)nq;
            return pp;
        };

        if (mode == 2) {
            const size_t per_warp = align16(warp_smem_bytes(ix.Dtot, ix.S, (int)topk));
            const size_t wsm = per_warp * kWarpsPerCta;
            ensure_smem((const void *)k_scan_warp, (size_t)wsm);
            k_scan_warp<<<(unsigned)((nq + kWarpsPerCta - 1) / kWarpsPerCta), kWarpsPerCta * 32, wsm, st>>>(
                ix, probe, (int)nprobe, (int)nq, qrot, prune, (int)topk, ids_out, d_out, cnt, per_warp);
            check_launch("k_scan_warp");
        } else if (mode == 0 && no_deferral(I, nq, nprobe, !qsh.np, resident_scans(ix.S, smem), tune)) {
            // no query of this call can probe more blocks than the deferral
            // threshold: the CTA scan answers every query, no split pass
            launch_cta_scan(scan_ws(tune), ix, probe, qsh, qrot, prune, ids_out, d_out, cnt, xs, nullptr, nq, order,
                            nullptr, scan_prep, st);
        } else {
            // split-pass state: every query (mode 1), or the deferred giant-cluster queries (mode 0)
            const int64_t max_pos = I.max_blocks_of_probes(nprobe);
            const int64_t cap = nq;
            const int64_t want = nq * max_pos;
            int64_t pos_cap = 0;
            Bump sb{split_scratch_take(I, C, cap, topk, nprobe, want, pos_cap, st)};
            SplitState ss;
            ss.nlist = sb.take<int>(16);
            ss.pos_used = reinterpret_cast<unsigned long long *>(ss.nlist + 2);
            ss.work_next = ss.nlist + 4;
            ss.qlist = sb.take<int>(cap);
            ss.cap = (int)cap;
            ss.pool_id = sb.take<uint32_t>((size_t)cap * topk);
            ss.pool_d = sb.take<float>((size_t)cap * topk);
            ss.pool_size = sb.take<int>(cap);
            ss.tau = sb.take<float>(cap);
            ss.tile_off = sb.take<int>((size_t)cap * (nprobe + 1));
            ss.blk_base = sb.take<int>((size_t)cap * nprobe);
            ss.split_p = sb.take<int>(cap);
            ss.split_b = sb.take<int>(cap);
            ss.q_tile_off = sb.take<int>(cap + 1);
            ss.npos = sb.take<int>(cap);
            ss.pos_off = sb.take<int64_t>(cap);
            ss.pos_cap = pos_cap;
            ss.summ = sb.take<float4>((size_t)pos_cap);
            ss.rec_words = rec_words_of(ix.S);
            ss.rec = sb.take<float>((size_t)pos_cap * ss.rec_words);
            ss.qsh = qsh;
            // heavy queries beside a batch: a longer prefix for a tighter bound; a
            // few queries alone: the speculative part has the GPU, so only the pool must fill
            ss.first_blocks = tune.first_blocks > 0 ? tune.first_blocks : (mode == 0 ? kFirstBlocks : 1);
            ss.tile_blocks = spec_tile_blocks(mode, nq);
            ss.t_lo = 0;
            ss.t_hi = INT_MAX;
            ss.final_level = 1;
            if (const char *e = std::getenv("SAQG_FIRST_BLOCKS")) ss.first_blocks = std::max(1, std::atoi(e));
            uint8_t *deferred = sb.take<uint8_t>(nq);
            int *qblocks = sb.take<int>(nq);
            SAQG_CUDA_TRY(cudaMemsetAsync(ss.summ, 0xff, 16 * (size_t)pos_cap, st));  // NaN: no record
            // A few queries that all fit: nothing to choose, so k_scan_first fills the list (one
            // host query over 100k vectors: 121 us with k_defer, 113 without it).
            ss.stride = mode == 1 && pos_cap >= want && max_pos < INT_MAX && !prep_lut ? max_pos : 0;
            if (!ss.stride) {
                SAQG_CUDA_TRY(cudaMemsetAsync(ss.nlist, 0, 32, st));
                int defer = -1, resident = 0;  // mode 1: every query
                if (mode == 0) {
                    defer = defer_threshold(tune);
                    resident = defer_line_given(tune) ? 0 : resident_scans(ix.S, smem);
                }
                const int dthreads = (int)std::min<int64_t>(kDeferThreads, 32 * nq);  // a warp per query while they fit
                const bool par = nq >= kQblocksMinQueries;
                if (par) {
                    k_qblocks<<<(unsigned)((nq + 7) / 8), 256, 0, st>>>(ix, probe, qsh, (int)nq, qblocks);
                    check_launch("k_qblocks");
                }
                k_defer<<<1, dthreads, 0, st>>>(ix, probe, (int)nq, defer, resident, ss, qblocks, par ? 1 : 0, deferred);
                check_launch("k_defer");
            }
            cudaStream_t sp = st;  // stream of the split pass
            // the CTA scan serves what the split list does not hold: always in mode 0,
            // in mode 1 only when the record space cannot hold every query
            if (mode == 0 || pos_cap < want) {
                if (mode == 0) {  // the split pass runs beside the CTA scan on the index's auxiliary stream
                    sp = C.aux_stream();
                    SAQG_CUDA_TRY(cudaEventRecord(C.fork_event(), st));
                    SAQG_CUDA_TRY(cudaStreamWaitEvent(sp, C.fork_event(), 0));
                }
                launch_cta_scan(scan_ws(tune), ix, probe, qsh, qrot, prune, ids_out, d_out, cnt, xs, deferred, nq,
                                order, qblocks, scan_prep, st);
            }
            const size_t smem1 = scan_smem_bytes(ix.Dtot, ix.S, 1, xs);
            const size_t rec_smem = 2 * 4 * (size_t)ss.rec_words;
            ss.replay_recs = (int)std::min<size_t>(kReplayRecs, (kReplaySmem - smem) / rec_smem);
            const size_t smem_r = smem + ss.replay_recs * rec_smem;
            ensure_smem((const void *)k_scan_first, (size_t)smem);
            ensure_smem((const void *)k_scan_spec, (size_t)smem1);
            // counters need every record's count, and a longer pool shared memory
            const auto replay = cnt || topk > kRegPool || ix.S > kRegSegs ? k_scan_replay<0> : topk <= 32 ? k_scan_replay<1>
                                                                               : k_scan_replay<kRegPool / 32>;
            ensure_smem((const void *)replay, (size_t)smem_r);
            Prepared prep;  // the listed queries' LUTs, one batched kernel ahead of the split pass
            if (prep_lut) {
                const size_t lsm = 4 * (size_t)kLutWarps * ix.Dtot;
                SAQG_REQUIRE(lsm <= 200 * 1024, "dimension too large for the batched LUT preparation");
                ensure_smem((const void *)k_lut, lsm);
                const int64_t items = pslots * nprobe;
                k_lut<<<(unsigned)((items + kLutWarps - 1) / kLutWarps), kLutWarps * 32, lsm, sp>>>(
                    ix, probe, qsh, ss.qlist, ss.nlist, (int)pslots, nullptr, qrot, prune, prep_lut, prep_scal);
                check_launch("k_lut");
                prep.lut = prep_lut;
                prep.scal = prep_scal;
                prep.np_max = (int)nprobe;
                prep.slots = (int)pslots;
            }
            // the list holds at most cap slots; the per-slot kernels loop over them
            const unsigned slot_grid = (unsigned)std::min<int64_t>(cap, 4 * (int64_t)sm_count());
            k_scan_first<<<slot_grid, kScanThreads, smem, sp>>>(ix, probe, qrot, prune, ss, flags + 1, cnt, xs,
                                                                     prep);
            check_launch("k_scan_first");
            if (stats) SAQG_CUDA_TRY(cudaEventRecord(ev[5], sp));
            const unsigned grid = (unsigned)full_grid((const void *)k_scan_spec, kScanThreads, smem1);
            // levels of speculation (tiles after the split point): each level's
            // replay leaves the exact pool, whose distk bounds the next level
            const int *levels = kSpecLevelSets[tune.spec_levels >= 0 && tune.spec_levels < kNumSpecLevelSets
                                                   ? tune.spec_levels : 0];
            int nlev = 1;
            if (mode == 0)
                while (nlev < kMaxSpecLevels && levels[nlev] >= 0) ++nlev;
            // a last level that holds less than half of the tiles (of the largest query: a tile
            // per kTileBlocks blocks, and one per probe that they do not fill) costs its three
            // launches for little: the one before it takes them (400 queries of 70 probes over
            // 146,720 vectors: 710 us, 692 without that level)
            const int64_t max_tiles = max_pos / kTileBlocks + nprobe;
            while (nlev > 1 && 2 * (int64_t)levels[nlev - 1] > max_tiles) --nlev;
            for (int L = 0; L < nlev; ++L) {
                SplitState sl = ss;
                sl.t_lo = mode == 0 ? levels[L] : 0;
                sl.t_hi = L + 1 < nlev ? levels[L + 1] : INT_MAX;
                sl.final_level = L + 1 == nlev;
                k_tile_prefix<<<1, kPrefixThreads, 0, sp>>>(sl);
                check_launch("k_tile_prefix");
                k_scan_spec<<<grid, kScanThreads, smem1, sp>>>(ix, probe, (int)nprobe, qrot, prune, sl, cnt, xs, prep);
                check_launch("k_scan_spec");
                if (stats && sl.final_level) SAQG_CUDA_TRY(cudaEventRecord(ev[6], sp));
                replay<<<slot_grid, kScanThreads, smem_r, sp>>>(ix, sl, ids_out, d_out, cnt, xs);
                check_launch("k_scan_replay");
            }
            if (stats) SAQG_CUDA_TRY(cudaEventRecord(ev[4], sp));
            if (sp != st) {  // join
                SAQG_CUDA_TRY(cudaEventRecord(C.join_event(), sp));
                SAQG_CUDA_TRY(cudaStreamWaitEvent(st, C.join_event(), 0));
            }
        }
        if (stats) SAQG_CUDA_TRY(cudaEventRecord(ev[3], st));
    }
    if (probes_out)
        SAQG_CUDA_TRY(cudaMemcpyAsync(probes_out, probe, 4 * (size_t)nq * nprobe,
                                      host ? cudaMemcpyDeviceToHost : cudaMemcpyDeviceToDevice, st));
    if (host) {
        SAQG_CUDA_TRY(cudaMemcpyAsync(ids, oid, 4 * (size_t)nq * topk, cudaMemcpyDeviceToHost, st));
        if (dists) SAQG_CUDA_TRY(cudaMemcpyAsync(dists, od, 4 * (size_t)nq * topk, cudaMemcpyDeviceToHost, st));
        int hflags[2] = {0, 0};
        SAQG_CUDA_TRY(cudaMemcpyAsync(hflags, flags, 8, cudaMemcpyDeviceToHost, st));
        SAQG_CUDA_TRY(cudaStreamSynchronize(st));
        if (hflags[1]) throw Error{SAQG_ERR_INTERNAL, "scan replay met a lane without a precomputed distance"};
    }
    if (stats) {
        unsigned long long hc[8] = {0, 0, 0, 0, 0, 0, 0, 0};
        SAQG_CUDA_TRY(cudaMemcpyAsync(hc, counters, 64, cudaMemcpyDeviceToHost, st));
        SAQG_CUDA_TRY(cudaStreamSynchronize(st));
        float t01 = 0, t12 = 0, t23 = 0, t03 = 0;
        SAQG_CUDA_TRY(cudaEventElapsedTime(&t01, ev[0], ev[1]));
        SAQG_CUDA_TRY(cudaEventElapsedTime(&t12, ev[1], ev[2]));
        SAQG_CUDA_TRY(cudaEventElapsedTime(&t23, ev[2], ev[3]));
        SAQG_CUDA_TRY(cudaEventElapsedTime(&t03, ev[0], ev[3]));
        stats->ms_probe = t01;
        stats->ms_qprep = t12;
        stats->ms_scan = t23;
        stats->ms_total = t03;
        // split pass phases (0 when the call had no split pass)
        auto span = [&](int a, int b) {
            float t = 0.0f;
            if (cudaEventQuery(ev[a]) != cudaSuccess || cudaEventQuery(ev[b]) != cudaSuccess) return 0.0f;
            return cudaEventElapsedTime(&t, ev[a], ev[b]) == cudaSuccess ? t : 0.0f;
        };
        stats->ms_split = span(2, 4);
        stats->ms_split_first = span(2, 5);
        stats->ms_split_spec = span(5, 6);
        stats->ms_split_replay = span(6, 4);
        cudaGetLastError();
        stats->probes = sum_np;
        stats->blocks = (int64_t)hc[0];
        stats->vectors = (int64_t)hc[1];
        stats->reranked = (int64_t)hc[2];
        stats->speculative = (int64_t)hc[3];
        stats->probe_exact = shortlist ? (int64_t)hc[4] : nq * I.K;
        stats->probe_full = shortlist ? (int64_t)(hc[5] + hc[6]) : nq;
        stats->probe_full_ties = (int64_t)hc[6];
        // Algorithmic bytes: per block of a probed cluster 32 lanes of 1-bit codes of
        // every coded segment and |o| of every segment (also where the first pruning
        // stage leaves the codes unread); per probe the rotated centroid; per re-ranked
        // vector its ex-codes, ex factors and id.
        int64_t per_lane = 0, per_rr = 4;
        for (int s = 0; s < ix.S; ++s) {
            per_lane += 4 + (ix.seg[s].bits ? ix.seg[s].dim / 8 : 0);
            per_rr += ix.seg[s].pv + 8;
        }
        stats->fast_bytes = stats->blocks * 32 * per_lane + stats->probes * 4 * (int64_t)ix.Dtot;
        stats->rerank_bytes = stats->reranked * per_rr;
    }
}

int64_t run_estimate(const Index &I, const float *q_host, int64_t nprobe, float m, uint32_t *ids, float *acc,
                     float *fast, float *vars, int64_t cap) {
    SAQG_REQUIRE(nprobe >= 1 && nprobe <= I.K, "nprobe must be in [1, number of clusters]");
    const DevIndexView &ix = I.view;
    cudaStream_t st = 0;
    CtxLease lease(I, st);
    Bump bp{(char *)lease.c->scratch_get(search_scratch_bytes(I, 1, 1, nprobe, true))};
    float *dq = bp.take<float>(I.D);
    float *dist = bp.take<float>(I.K);
    Cand *work = bp.take<Cand>(I.K);
    uint32_t *probe = bp.take<uint32_t>(nprobe);
    float *qrot = bp.take<float>(ix.Dtot);
    float *prune = bp.take<float>(ix.S);
    bp.take<uint32_t>(2);
    bp.take<float>(2);
    int *flags = bp.take<int>(16);
    SAQG_CUDA_TRY(cudaMemcpy(dq, q_host, 4 * I.D, cudaMemcpyHostToDevice));
    SAQG_CUDA_TRY(cudaMemset(flags, 0, 64));
    const int wpb = 8;
    k_probe_dist<<<dim3((unsigned)((I.K + wpb - 1) / wpb), 1), wpb * 32, 0, st>>>(ix, dq, dist);
    check_launch("k_probe_dist");
    k_probe_select<<<1, kSelThreads, 0, st>>>(dist, (int)I.K, (int)nprobe, probe, work, flags);
    check_launch("k_probe_select");
    launch_qprep(ix, dq, 1, m, qrot, prune, st);
    std::vector<uint32_t> hprobe(nprobe);
    SAQG_CUDA_TRY(cudaMemcpy(hprobe.data(), probe, 4 * nprobe, cudaMemcpyDeviceToHost));
    std::vector<int64_t> off(nprobe + 1, 0);
    for (int64_t p = 0; p < nprobe; ++p) off[p + 1] = off[p] + I.sizes[hprobe[p]];
    const int64_t total = off[nprobe];
    if (total > 0) {
        std::vector<int2> tiles;
        for (int64_t p = 0; p < nprobe; ++p)
            for (int64_t b = 0; 32 * b < off[p + 1] - off[p]; b += kEstBlocks) tiles.push_back(make_int2((int)p, (int)b));
        const auto carve = [&](char *base, int64_t *&doff, int2 *&dtiles, uint32_t *&oids, float *&oacc, float *&ofast,
                               float *&ovars) {
            Bump b{base};
            doff = b.take<int64_t>(nprobe + 1);
            dtiles = b.take<int2>(tiles.size());
            oids = b.take<uint32_t>(total);
            oacc = b.take<float>(total);
            ofast = b.take<float>(total);
            ovars = b.take<float>(total);
            return b.off;
        };
        int64_t *doff;
        int2 *dtiles;
        uint32_t *oids;
        float *oacc, *ofast, *ovars;
        const size_t bytes = carve(nullptr, doff, dtiles, oids, oacc, ofast, ovars);
        // up to kEstKeep bytes from the context's scratch, which stays for the next call; more is freed after it
        constexpr size_t kEstKeep = (size_t)64 << 20;
        std::unique_ptr<char, void (*)(char *)> own(nullptr, [](char *x) { cudaFree(x); });
        char *base;
        if (bytes <= kEstKeep) {
            base = (char *)lease.c->split_scratch_get(bytes);
        } else {
            void *x = nullptr;
            SAQG_CUDA_TRY(cudaMalloc(&x, bytes));
            own.reset(base = (char *)x);
        }
        carve(base, doff, dtiles, oids, oacc, ofast, ovars);
        SAQG_CUDA_TRY(cudaMemcpy(doff, off.data(), 8 * (nprobe + 1), cudaMemcpyHostToDevice));
        SAQG_CUDA_TRY(cudaMemcpy(dtiles, tiles.data(), sizeof(int2) * tiles.size(), cudaMemcpyHostToDevice));
        const int xs = xstride_of(ix);
        const size_t smem = scan_smem_bytes(ix.Dtot, ix.S, 1, xs);
        ensure_smem((const void *)k_estimate, (size_t)smem);
        k_estimate<<<(unsigned)tiles.size(), kScanThreads, smem, st>>>(ix, probe, dtiles, doff, qrot, prune, oids, oacc, ofast,
                                                                       ovars, xs);
        check_launch("k_estimate");
        const int64_t nw = std::min(total, cap);
        SAQG_CUDA_TRY(cudaMemcpy(ids, oids, 4 * nw, cudaMemcpyDeviceToHost));
        SAQG_CUDA_TRY(cudaMemcpy(acc, oacc, 4 * nw, cudaMemcpyDeviceToHost));
        SAQG_CUDA_TRY(cudaMemcpy(fast, ofast, 4 * nw, cudaMemcpyDeviceToHost));
        SAQG_CUDA_TRY(cudaMemcpy(vars, ovars, 4 * nw, cudaMemcpyDeviceToHost));
    }
    return total;
}

// ------------------------------------------------- search with static scratch
// The scratch of saqg_search_static: one file-scope device array (one instance
// per device, placed by the driver when it loads this file's kernels), shared by
// every call on that device.  Nothing in it needs to start at zero except the
// 64-byte flag words, which each call clears on its stream before its kernels.
// Because it belongs to this file's module, every process that runs any search
// kernel of the library on a device holds these 16 MiB there until it exits,
// whether or not it calls saqg_search_static.
static __device__ __align__(256) unsigned char g_static_scratch[SAQG_STATIC_SCRATCH_BYTES];

namespace {

constexpr int kMaxStaticDevices = 64;
std::mutex g_static_mu;
void *g_static_ptr[kMaxStaticDevices] = {};

// Device address of the array on `dev` (current), looked up on the first call
// on that device.
void *static_scratch(int dev) {
    SAQG_REQUIRE(dev >= 0 && dev < kMaxStaticDevices, "device ordinal out of range for the static scratch");
    std::lock_guard<std::mutex> lock(g_static_mu);
    if (!g_static_ptr[dev]) {
        void *p = nullptr;
        const cudaError_t e = cudaGetSymbolAddress(&p, g_static_scratch);
        if (e != cudaSuccess || !p)
            throw Error{SAQG_ERR_CUDA, std::string("cudaGetSymbolAddress(static scratch) failed: ") +
                                           cudaGetErrorString(e)};
        g_static_ptr[dev] = p;
    }
    return g_static_ptr[dev];
}

}  // namespace

size_t static_search_scratch_bytes(const Index &I, int64_t nq, int64_t nprobe) {
    size_t b = 0;
    auto add = [&](size_t x) { b += align16(x); };
    add(4 * (size_t)nq * I.K);          // centroid distances
    add(8 * (size_t)nq * I.K);          // exact-select work (fallback)
    add(4 * (size_t)nq * nprobe);       // probe ids
    add(4 * (size_t)nq * I.view.Dtot);  // rotated queries
    add(4 * (size_t)nq * I.view.S);     // prune bounds
    add(64);                            // flags
    return b;
}

void run_search_static(const Index &I, const float *q, int64_t nq, int64_t topk, int64_t nprobe, float m,
                       uint32_t *ids, float *dists, cudaStream_t st) {
    SAQG_REQUIRE(nq >= 0 && topk >= 1 && topk <= kMaxTopK, "topk must be in [1, 4096]");
    SAQG_REQUIRE(nprobe >= 1 && nprobe <= I.K, "nprobe must be in [1, number of clusters]");
    if (nq == 0) return;
    const size_t need = static_search_scratch_bytes(I, nq, nprobe);
    SAQG_REQUIRE(need <= (size_t)SAQG_STATIC_SCRATCH_BYTES,
                 "saqg_search_static: " + std::to_string(nq) + " queries with " + std::to_string(I.K) +
                     " clusters and nprobe " + std::to_string(nprobe) + " need " + std::to_string(need) +
                     " bytes of scratch, above the static maximum of " +
                     std::to_string((size_t)SAQG_STATIC_SCRATCH_BYTES) + " bytes; split the batch");
    // The kernels would fault on a host pointer or one on another device; a
    // wrong pointer is reported instead (this call takes device memory only).
    auto require_device_ptr = [&](const void *p, const char *what) {
        cudaPointerAttributes a{};
        const cudaError_t e = cudaPointerGetAttributes(&a, p);
        if (e != cudaSuccess) {
            cudaGetLastError();
            throw Error{SAQG_ERR_INVALID, std::string("saqg_search_static: ") + what +
                                              " is not a pointer the CUDA runtime knows: " + cudaGetErrorString(e)};
        }
        if (a.type == cudaMemoryTypeManaged) return;
        if (a.type != cudaMemoryTypeDevice || a.device != I.device)
            throw Error{SAQG_ERR_INVALID, std::string("saqg_search_static: ") + what +
                                              " must be device memory on the index's device (" +
                                              std::to_string(I.device) + ")"};
    };
    require_device_ptr(q, "queries");
    require_device_ptr(ids, "ids");
    if (dists) require_device_ptr(dists, "dists");
    const DevIndexView &ix = I.view;
    const size_t smem = scan_smem_bytes(ix.Dtot, ix.S, (int)topk, xstride_of(ix));
    SAQG_REQUIRE(smem <= kScanSmem, "dimension / topk too large for the scan kernel's shared memory");
    int prev = 0;
    SAQG_CUDA_TRY(cudaGetDevice(&prev));
    struct DevGuard {
        int prev, cur;
        ~DevGuard() {
            if (prev != cur) cudaSetDevice(prev);
        }
    } dg{prev, I.device};
    if (prev != I.device) SAQG_CUDA_TRY(cudaSetDevice(I.device));
    Bump bp{(char *)static_scratch(I.device)};
    float *dist = bp.take<float>((size_t)nq * I.K);
    Cand *work = bp.take<Cand>((size_t)nq * I.K);
    uint32_t *probe = bp.take<uint32_t>((size_t)nq * nprobe);
    float *qrot = bp.take<float>((size_t)nq * ix.Dtot);
    float *prune = bp.take<float>((size_t)nq * ix.S);
    int *flags = bp.take<int>(16);
    SAQG_CUDA_TRY(cudaMemsetAsync(flags, 0, 64, st));
    if (nq >= 8 && I.D % 32 == 0 && I.D <= 32 * kProbeRegs) {
        const size_t qsm = 4 * (size_t)kProbeQT * I.D;
        ensure_smem((const void *)k_probe_dist_tiled, (size_t)qsm);
        const unsigned gx = (unsigned)std::min<int64_t>((I.K + kProbeWarps - 1) / kProbeWarps, 304);
        k_probe_dist_tiled<<<dim3(gx, (unsigned)((nq + kProbeQT - 1) / kProbeQT)), kProbeWarps * 32, qsm, st>>>(
            ix, q, (int)nq, dist);
        check_launch("k_probe_dist_tiled");
    } else {
        const int wpb = 8;
        k_probe_dist<<<dim3((unsigned)((I.K + wpb - 1) / wpb), (unsigned)nq), wpb * 32, 0, st>>>(ix, q, dist);
        check_launch("k_probe_dist");
    }
    k_probe_select<<<(unsigned)nq, kSelThreads, 0, st>>>(dist, (int)I.K, (int)nprobe, probe, work, flags);
    check_launch("k_probe_select");
    launch_qprep(ix, q, nq, m, qrot, prune, st);
    const size_t smem_k = scan_smem_bytes(ix.Dtot, ix.S, (int)topk, xstride_of(ix));
    SAQG_REQUIRE(smem_k <= kScanSmem, "dimension / topk too large for the scan kernel's shared memory");
    const auto scan = scan_kernel(ix.S);
    ensure_smem((const void *)scan, smem_k);
    QueryShape qsh;
    qsh.np_max = (int)nprobe;
    qsh.k_max = (int)topk;
    scan<<<(unsigned)nq, kScanThreads, smem_k, st>>>(ix, probe, qsh, qrot, prune, ids, dists, nullptr,
                                                      xstride_of(ix), nullptr, nullptr, Prepared{});
    check_launch("k_scan");
}

// ------------------------------------------ tensor-core form: probes and re-rank
namespace {

// A cluster's residual query (ex order, x) and the scalars of Lut::prepare, by one
// warp; lanes s and 16 + s return with segment s's scalars.
__device__ __forceinline__ SegScal warp_scalars(const DevIndexView &ix, const float *__restrict__ qrot,
                                                const float *__restrict__ prune, int c, float *x) {
    const int lane = threadIdx.x & 31, at0 = ex_order(lane), at1 = ex_order(lane + 32);
    SegScal sc;
    uint32_t my_min = 0xffffffffu, my_max = 0u;
    for (int s = 0; s < ix.S; ++s) {
        const SegDev &g = ix.seg[s];
        const float *cent = g.cent + (size_t)c * g.dim + lane, *q = qrot + g.qoff + lane;
        float *xs = x + g.qoff;
        // Eigen's sums (warp_eigen_sum): lane i of the two 16-lane accumulators takes the
        // dims i, i + 32, ...
        float sum = 0.0f, sq = 0.0f;
#pragma unroll 4
        for (int d = 0; d < g.dim; d += 64) {
            const float a = __fsub_rn(q[d], cent[d]), b = __fsub_rn(q[d + 32], cent[d + 32]);
            xs[d + at0] = a;
            xs[d + at1] = b;
            sum = d == 0 ? a : __fadd_rn(sum, a);
            sq = d == 0 ? __fmul_rn(a, a) : __fadd_rn(sq, __fmul_rn(a, a));
            sum = __fadd_rn(sum, b);
            sq = __fadd_rn(sq, __fmul_rn(b, b));
        }
#pragma unroll
        for (int o = 16; o; o >>= 1) {
            sum = __fadd_rn(sum, __shfl_down_sync(kFull, sum, o));
            sq = __fadd_rn(sq, __shfl_down_sync(kFull, sq, o));
        }
        sum = __shfl_sync(kFull, sum, 0);
        sq = __shfl_sync(kFull, sq, 0);
        __syncwarp();
        uint32_t kmin = 0xffffffffu, kmax = 0u;
        for (int k = lane; k < g.dim / 4; k += 32) {
            const float *p = xs + ex_order(4 * k);  // dims 4k .. 4k + 3 lie four apart
            uint32_t a, b;
            codebook_keys(make_float4(p[0], p[4], p[8], p[12]), a, b);
            kmin = min(kmin, a);
            kmax = max(kmax, b);
        }
        kmin = __reduce_min_sync(kFull, kmin);
        kmax = __reduce_max_sync(kFull, kmax);
        if ((lane & 15) == s) {
            sc.sum_q = sum;
            sc.q_l2sqr = sq;
            my_min = kmin;
            my_max = kmax;
        }
    }
    if ((lane & 15) < ix.S) {
        seg_quant_scalars(my_min, my_max, sc);
        seg_epilogue_scalars(ix.seg[lane & 15], prune[lane & 15], sc);
    }
    return sc;
}

// Distance the search inserts for a vector that passes every pruning stage
// (block_estimates + the accurate pass + the replay): one segment, the
// accurate distance; several, the running sum of variance bounds, each coded
// segment's bound replaced by its fast estimate, then every segment's
// estimate replaced by its accurate distance, in segment order.  Two vectors at a
// time, one per half-warp (gb, gv, ln: the half's own), without a LUT: of each codebook
// the one entry that the vector's nibble selects is formed and quantized.  x: the
// residual in ex order; sc: lanes s and 16 + s segment s's scalars.
__device__ float searched_dist(const DevIndexView &ix, const float *x, const SegScal &sc, int64_t gb, int64_t gv, int ln) {
    const int S = ix.S, lane = threadIdx.x & 31, l = lane & 15;
    float v = 0.0f, f = 0.0f, ipx = 0.0f, ex = 0.0f;  // lane l = s of the half: segment s
    for (int s = 0; s < S; ++s) {
        const SegDev &g = ix.seg[s];
        int sum = 0;
        float e = 0.0f;
        if (g.bits) {
            const float vl = __shfl_sync(kFull, sc.vl, s), delta = __shfl_sync(kFull, sc.delta, s),
                        rd = __shfl_sync(kFull, sc.rdelta, s);
            const bool quick = lut_quant_ok(delta);
            const int nc = g.dim / 64;
            // codebook l of every group: byte l / 2 of the vector's 8, high nibble first; its
            // dims at q[0, 4, 8, 12]
            const uint32_t *cp = reinterpret_cast<const uint32_t *>(g.codes + (size_t)gb * nc * 32 + ln) + (l >> 3);
            const int sh = 8 * ((l >> 1) & 3) + 4 * (~l & 1);
            const float *q = x + g.qoff + ex_order(4 * l);
#pragma unroll 4
            for (int c8 = 0; c8 < nc; ++c8) {
                const uint32_t nib = cp[(size_t)c8 * 64] >> sh;
                const float *p = q + 64 * c8;
                float t = (nib & 8u) ? __fadd_rn(0.0f, p[0]) : 0.0f;
                t = __fadd_rn(t, (nib & 4u) ? p[4] : 0.0f);
                t = __fadd_rn(t, (nib & 2u) ? p[8] : 0.0f);
                t = __fadd_rn(t, (nib & 1u) ? p[12] : 0.0f);
                const float y = __fsub_rn(t, vl);
                sum += quick ? (int)lut_quant(y, delta, rd) : (int)(uint16_t)(int)__fdiv_rn(y, delta);
            }
#pragma unroll
            for (int o = 8; o; o >>= 1) sum += __shfl_xor_sync(kFull, sum, o);
            if (g.bits > 1)
                e = __shfl_sync(kFull, excode_ip16(x + g.qoff, g.lcode + (size_t)gv * g.lstride, g.dim, g.bits - 1), 0, 16);
        }
        if (l == s) {
            const float on = g.onorm[gb * 32 + ln];
            v = vars_est(sc, on);
            f = g.bits ? fast_of_sum(sc, sum, on, ipx) : v;
            ex = e;
        }
    }
    float acc = 0.0f;
    if (l < S) {
        const SegDev &g = ix.seg[l];
        acc = accurate_dist(g.onorm[gb * 32 + ln], ipx, ex, g.exfac[gv].x, g.bits, sc.sum_q, sc.q_l2sqr);
    }
    if (S == 1) return __shfl_sync(kFull, acc, 0, 16);
    float cur = 0.0f;
    for (int s = 0; s < S; ++s) cur = __fadd_rn(cur, __shfl_sync(kFull, v, s, 16));
    for (int s = 0; s < S; ++s)
        if (ix.seg[s].bits)
            cur = __fadd_rn(__fsub_rn(cur, __shfl_sync(kFull, v, s, 16)), __shfl_sync(kFull, f, s, 16));
    const float part = __fsub_rn(acc, f);  // accurate less estimate (its bound when uncoded)
    for (int s = 0; s < S; ++s) cur = __fadd_rn(cur, __shfl_sync(kFull, part, s, 16));
    return cur;
}

// Re-rank of the tensor-core shortlist, one CTA per query: its positions ascend, so
// the vectors of one probed cluster lie together.  Work item: up to kRerankRun of them,
// by one warp, which forms the cluster's residual and scalars for itself and then each
// vector's distance (searched_dist).  A cluster holds a handful of the shortlist, and a
// vector needs one entry of each codebook, so no LUT is built and nothing waits for a
// barrier.  2,048 queries of 1,536 dimensions, 40 vectors each: 0.98 ms with a CTA and a
// LUT per (query, cluster), 0.34 now; 4,096 queries over 10M x 1,024: 1.02 and 0.50.
// Up to four warps, as many as their residuals (4 Dtot bytes each) fit beside the
// kernel's own 6 KB: four up to 14,080 dimensions, three above.
constexpr int kRerankThreads = 128, kRerankRun = 8, kRerankMax = 1024;  // at most kTcMaxShort entries
constexpr size_t kRerankSmem = 220 * 1024;
__global__ void __launch_bounds__(kRerankThreads) k_tc_rerank(DevIndexView ix, const uint32_t *__restrict__ probe,
                                                              int nprobe, const float *__restrict__ qrot_all,
                                                              const float *__restrict__ prune,
                                                              const int *__restrict__ lp, const int *__restrict__ sl_pos,
                                                              const int *__restrict__ sl_cnt, int L,
                                                              float *__restrict__ sl_dist) {
    extern __shared__ __align__(16) float rr_x[];  // a residual per warp
    __shared__ int pj[kRerankMax];                 // entry's probe
    __shared__ uint16_t first[kRerankMax + 1];     // items' first entries
    __shared__ int nitems, next;
    const int qi = blockIdx.x, n = sl_cnt[qi], tid = threadIdx.x, w = tid >> 5, lane = tid & 31;
    const int *pos = sl_pos + (size_t)qi * L, *lq = lp + (size_t)qi * (nprobe + 1);
    const float *qrot = qrot_all + (size_t)qi * ix.Dtot;
    for (int e = tid; e < n; e += (int)blockDim.x) {  // the last probe that starts at or before it (empty probes share an offset)
        int lo = 0, hi = nprobe - 1;
        const int x = pos[e];
        while (lo < hi) {
            const int mid = (lo + hi + 1) >> 1;
            if (lq[mid] <= x) lo = mid;
            else hi = mid - 1;
        }
        pj[e] = lo;
    }
    if (tid == 0) next = 0;
    __syncthreads();
    if (w == 0) {
        int cnt = 0;
        for (int e0 = 0; e0 < n; e0 += 32) {
            const int e = e0 + lane;
            const bool start = e < n && (e % kRerankRun == 0 || pj[e] != pj[e - 1]);
            const uint32_t b = __ballot_sync(kFull, start);
            if (start) first[cnt + __popc(b & ((1u << lane) - 1u))] = (uint16_t)e;
            cnt += __popc(b);
        }
        if (lane == 0) {
            nitems = cnt;
            first[cnt] = (uint16_t)n;
        }
    }
    __syncthreads();
    float *x = rr_x + (size_t)w * ix.Dtot;
    for (;;) {
        int it = 0;
        if (lane == 0) it = atomicAdd(&next, 1);
        it = __shfl_sync(kFull, it, 0);
        if (it >= nitems) break;
        const int e0 = first[it], e1 = first[it + 1], j = pj[e0], c = (int)probe[(size_t)qi * nprobe + j], base = lq[j];
        const int64_t b0 = ix.blk_off[c], v0 = ix.vec_off[c];
        for (int e = e0; e < e1; ++e) {  // pull every vector's codes, rows and factors in while the scalars are formed
            const int r = pos[e] - base;
            const int64_t gb = b0 + r / 32, gv = v0 + r;
            for (int s = 0; s < ix.S; ++s) {
                const SegDev &g = ix.seg[s];
                if (lane == 0) asm volatile("prefetch.global.L1 [%0];" ::"l"(g.onorm + gb * 32 + (r & 31)));
                if (lane == 1) asm volatile("prefetch.global.L1 [%0];" ::"l"(g.exfac + gv));
                if (!g.bits) continue;
                const int nc = g.dim / 64;
                for (int k = lane; k < nc; k += 32)
                    asm volatile("prefetch.global.L1 [%0];" ::"l"(g.codes + ((size_t)gb * nc + k) * 32 + (r & 31)));
                for (int o = 128 * lane; o < g.lstride; o += 128 * 32)
                    asm volatile("prefetch.global.L1 [%0];" ::"l"(g.lcode + (size_t)gv * g.lstride + o));
            }
        }
        __syncwarp();  // the previous item's residual is done with
        const SegScal sc = warp_scalars(ix, qrot, prune + (size_t)qi * ix.S, c, x);
        for (int e = e0; e < e1; e += 2) {
            const int me = min(e + (lane >> 4), e1 - 1), r = pos[me] - base;
            const float d = searched_dist(ix, x, sc, b0 + r / 32, v0 + r, r & 31);
            if ((lane & 15) == 0 && e + (lane >> 4) < e1) sl_dist[(size_t)qi * L + me] = d;
        }
    }
}

// Top-k of the re-ranked shortlist, one CTA per query: ordered by distance,
// equal distances the later-scanned first, which is where ResultPool::insert
// puts an equal distance (pool.hpp:17-30).
__global__ void __launch_bounds__(kScanThreads) k_tc_topk(DevIndexView ix, const uint32_t *__restrict__ probe,
                                                          int nprobe, const int *__restrict__ lp,
                                                          const int *__restrict__ sl_pos,
                                                          const float *__restrict__ sl_apx,
                                                          const int *__restrict__ sl_cnt,
                                                          const float *__restrict__ sl_dist, int L, int L2, int topk,
                                                          const int *__restrict__ qk, uint32_t *__restrict__ ids,
                                                          float *__restrict__ dists, float *__restrict__ apx_out) {
    extern __shared__ __align__(16) char smem_raw[];
    unsigned long long *key = reinterpret_cast<unsigned long long *>(smem_raw);
    const int qi = blockIdx.x, tid = threadIdx.x;
    const int n = sl_cnt[qi];
    const int *pos = sl_pos + (size_t)qi * L;
    const float *dist = sl_dist + (size_t)qi * L;
    const int *lq = lp + (size_t)qi * (nprobe + 1);
    for (int e = tid; e < L2; e += blockDim.x)
        key[e] = e < n ? ((unsigned long long)fkey(dist[e]) << 32) | (unsigned)(0x7fffffff - pos[e]) : ~0ull;
    __syncthreads();
    for (int k = 2; k <= L2; k <<= 1)
        for (int jj = k >> 1; jj > 0; jj >>= 1) {
            for (int e = tid; e < L2; e += blockDim.x) {
                const int o = e ^ jj;
                if (o > e) {
                    const unsigned long long a = key[e], b = key[o];
                    if ((a > b) == ((e & k) == 0)) {
                        key[e] = b;
                        key[o] = a;
                    }
                }
            }
            __syncthreads();
        }
    const int kq = qk ? qk[qi] : topk;  // this query's k; rows are topk long, padded with (0, FLT_MAX)
    for (int t = tid; t < topk; t += blockDim.x) {
        uint32_t id = 0;
        float d = FLT_MAX, a = FLT_MAX;
        if (t < n && t < kq) {
            const int p = 0x7fffffff - (int)(unsigned)(key[t] & 0xffffffffull);
            int lo = 0, hi = n - 1;  // the shortlist entry of position p
            while (lo < hi) {
                const int mid = (lo + hi) >> 1;
                if (pos[mid] < p) lo = mid + 1;
                else hi = mid;
            }
            int jlo = 0, jhi = nprobe - 1;  // its probe: the last j with lq[j] <= p
            while (jlo < jhi) {
                const int mid = (jlo + jhi + 1) >> 1;
                if (lq[mid] <= p) jlo = mid;
                else jhi = mid - 1;
            }
            const int c = (int)probe[(size_t)qi * nprobe + jlo];
            id = ix.ids[ix.vec_off[c] + (p - lq[jlo])];
            d = dist[lo];
            a = sl_apx[(size_t)qi * L + lo];
        }
        ids[(size_t)qi * topk + t] = id;
        if (dists) dists[(size_t)qi * topk + t] = d;
        if (apx_out) apx_out[(size_t)qi * topk + t] = a;
    }
}

}  // namespace

void tc_rank_rotate(const Index &I, SearchCtx &C, const float *q, int64_t nq, int64_t nprobe, const int *qnp, float m,
                    float *dist, void *work, uint32_t *probe, float *qrot, float *prune, uint8_t *full, int *fb_list,
                    int *flags, void *qbf, cudaStream_t st) {
    const DevIndexView &ix = I.view;
    SAQG_CUDA_TRY(cudaMemsetAsync(flags, 0, 64, st));
    Cand *wk = static_cast<Cand *>(work);
    // the rotation runs on the context's least-priority stream beside the ranking, as in run_search
    auto fork_qprep = [&]() {
        cudaStream_t qs = C.low_stream();
        SAQG_CUDA_TRY(cudaEventRecord(C.qfork_event(), st));
        SAQG_CUDA_TRY(cudaStreamWaitEvent(qs, C.qfork_event(), 0));
        launch_qprep(ix, q, nq, m, qrot, prune, qs);
        SAQG_CUDA_TRY(cudaEventRecord(C.qjoin_event(), qs));
    };
    const char *pm = std::getenv("SAQG_PROBE");
    const bool shortlist = nq >= kGemmMinQueries && nprobe <= kShortCap && !(pm && std::string(pm) == "exact");
    if (shortlist) {
        probe_shortlist(I, C, q, nq, nprobe, qnp, dist, probe, full, fb_list, flags, wk, nullptr, qbf, st, fork_qprep);
    } else {
        fork_qprep();
        k_probe_dist<<<dim3((unsigned)((I.K + 7) / 8), (unsigned)nq), 256, 0, st>>>(ix, q, dist);
        check_launch("k_probe_dist");
        k_probe_select<<<(unsigned)nq, kSelThreads, 0, st>>>(dist, (int)I.K, (int)nprobe, probe, wk, flags, nullptr,
                                                              qnp);
        check_launch("k_probe_select");
    }
    SAQG_CUDA_TRY(cudaStreamWaitEvent(st, C.qjoin_event(), 0));  // the rotated queries
}

size_t tc_probe_work_bytes(const Index &I, int64_t nq) { return sizeof(Cand) * (size_t)nq * I.K; }

void tc_rerank(const Index &I, const uint32_t *probe, int64_t nq, int64_t nprobe, const float *qrot,
               const float *prune, const int *lp, const int *sl_pos, const float *sl_apx, const int *sl_cnt, int L,
               int64_t topk, const int *qk, float *sl_dist, uint32_t *ids, float *dists, float *apx, cudaStream_t st) {
    const DevIndexView &ix = I.view;
    int L2 = 1;
    while (L2 < L) L2 <<= 1;
    const size_t per_warp = 4 * (size_t)ix.Dtot;
    SAQG_REQUIRE(scan_smem_bytes(ix.Dtot, ix.S, 1, 0) <= kScanSmem,
                 "dimension too large for the re-rank kernel's shared memory");
    const int warps = (int)std::min<size_t>(kRerankThreads / 32, kRerankSmem / per_warp);  // (3 at the check's limit)
    ensure_smem((const void *)k_tc_rerank, warps * per_warp);
    k_tc_rerank<<<(unsigned)nq, 32 * warps, warps * per_warp, st>>>(ix, probe, (int)nprobe, qrot, prune, lp, sl_pos,
                                                                   sl_cnt, L, sl_dist);
    check_launch("k_tc_rerank");
    k_tc_topk<<<(unsigned)nq, kScanThreads, 8 * (size_t)L2, st>>>(ix, probe, (int)nprobe, lp, sl_pos, sl_apx, sl_cnt,
                                                                  sl_dist, L, L2, (int)topk, qk, ids, dists, apx);
    check_launch("k_tc_topk");
}

}  // namespace saqg

// Estimation kernels for sm_103a: the dispersion scorer and the depth
// profiles of the focus search.
//
// Dispersion (octrecon/estimation/dispersion.py:66-107): the B-scans are
// k-linearised and Hann/rms-windowed once (X, real); every candidate beta
// then costs one phase multiply, one inverse FFT and |.| per A-scan
// (dispersion.py:88-102), and a sharpness metric per B-scan over the depth
// pixels z >= 20 (dispersion.py:46-63).
//   k_disp_mag    one launch for a whole list of betas: a warp per A-scan
//                 loads X and the beta's phase row straight into the registers
//                 of the first FFT stage (64 points a lane), one exchange
//                 through its own shared memory; |X| is averaged over the
//                 B-scan repeats (dispersion.py:101).
//   k_phase       the phase rows of a list of betas, in float64.
//   k_top_sum     top_percentile: 1 to 8 CTAs per (beta, B-scan) find the exact
//                 k-th largest magnitude by a three-digit radix select on the
//                 float bits (12 + 11 + 8 bits, histograms in shared memory),
//                 then sums I = float32(A^2) in float64 over the top k
//                 (elements above the threshold plus the ties needed), and
//                 returns log(sum / k).
//   k_moments     kurtosis, entropy, legacy_peak, one CTA per (beta, B-scan).
// Focus (octrecon/estimation/focus.py:146,156,255): k_xmedian takes the
// median over x of every depth column of (frames, nX, nZ) magnitudes, as
// float64, optionally ignoring NaN (nanmedian), by bisection on the float bits
// (one warp per column); or, in mean mode, the float64 mean of the column's
// non-NaN values.
#include <cooperative_groups.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "octgb_device.cuh"
#include "octgb_internal.h"

namespace octgb {
namespace {

// One warp an A-scan (ifft2048_low_mag_warp), four warps a CTA, three CTAs an
// SM (168 registers a thread: 64 complex points a lane).  Bound by latency and
// issue: 2 835 warp instructions an A-scan, issue active 56 %, FMA pipe 50 %,
// shared-memory path 54 %, DRAM 32 % (205 000 transforms, 41 betas).  There it
// takes 823 us; with 128 threads an A-scan, two exchanges and four group
// barriers the same arithmetic took 967 us.  The next line is prefetched into
// L2 (holding it in registers behind the last stage spilled), or into shared
// memory (below).
constexpr int kDispWarps = 4;
// Without pooling or repeats shared memory has room for each warp's next line:
// one CTA of twelve warps shares the twiddles, and a bulk copy brings the line in
// behind the transform before it, where the warps' loads took a fifth of their
// time (823 -> 726 us).  Taken from 24 A-scans a warp on (28 a warp: 24 us of a
// volume's last pass); below, the three smaller CTAs an SM run beside other
// streams' kernels and end less unevenly (16 a warp: 217 us a call of the
// precision form against 221).
constexpr int kLineWarps = 12;
constexpr int kLineItems = 24;

template <int kWarps, bool kLine>
struct DispSmem {
    alignas(16) float2 tw[kTwTable];                     // tw2, tw3
    alignas(16) float2 ex[kWarps][kWarpExchange];
    alignas(16) float line[kLine ? kWarps : 1][kLine ? kN : 4];
    uint64_t bar[kWarps];
    // followed by [kWarps][kHalf] floats (a line's magnitudes) with pooling or repeats
};
static_assert(sizeof(DispSmem<kLineWarps, true>) <= 232448, "k_disp_mag shared memory exceeds 227 KB");

// streamed once: keep L1 for the phase row
__device__ __forceinline__ float ld_stream(const float* p) {
    float v;
    asm volatile("ld.global.L1::no_allocate.f32 %0, [%1];" : "=f"(v) : "l"(p));
    return v;
}

// Pool: probe images; Db: dB of a depth crop; Rep: several B-scan repeats (a.rep > 1)
template <bool Pool, bool Db, bool Rep, bool kLine>
__global__ void __launch_bounds__((kLine ? kLineWarps : kDispWarps) * 32, kLine ? 1 : 3)
    k_disp_mag(const DispArgs a) {
    static_assert(!kLine || (!Pool && !Rep), "no room for the lines");
    constexpr int kWarps = kLine ? kLineWarps : kDispWarps;
    extern __shared__ __align__(128) unsigned char smem_raw[];
    using Smem = DispSmem<kWarps, kLine>;
    Smem& S = *reinterpret_cast<Smem*>(smem_raw);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    for (int k = tid; k < kTwTable / 2; k += kWarps * 32)
        reinterpret_cast<float4*>(S.tw)[k] = __ldg(reinterpret_cast<const float4*>(a.tw) + k);
    const float2 *tw2 = S.tw, *tw3 = S.tw + 256;
    if (kLine && lane == 0) {
        mbar_init(&S.bar[warp], 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();
    pdl_wait();                                          // the lines and phase rows
    // kLine: the kernel after this one starts when it ends (started early, the
    // next pass's lines kernel cost a precision volume's tile 1882 -> 2012 us)
    if (!kLine) pdl_launch();
    float run_min = __int_as_float(0x7f800000), run_max = -__int_as_float(0x7f800000);
    float2* ex = S.ex[warp];
    float* sums = reinterpret_cast<float*>(&S + 1) + warp * kHalf;
    // items < 2^32 - the grid's warps (the launcher checks): 32-bit item arithmetic
    const unsigned int nbx = static_cast<unsigned int>(a.nb) * static_cast<unsigned int>(a.nx);
    const unsigned int n_items = static_cast<unsigned int>(a.n_beta) * nbx, step = gridDim.x * kWarps;
    // repeat 0 of an item: B-scan b0 + bu, A-scan x; repeat rp is rp * nx lines further
    auto line_of = [&](unsigned int item) -> const float* {
        const unsigned int bx = item % nbx;
        const unsigned int bu = bx / static_cast<unsigned int>(a.nx);
        const unsigned int x = bx - bu * static_cast<unsigned int>(a.nx);
        return a.X + ((static_cast<int64_t>(a.b0 + static_cast<int>(bu)) * a.rep) * a.nx + x) * kN;
    };
    const unsigned int first = blockIdx.x * kWarps + warp;
    auto copy_line = [&](unsigned int item) {                // by lane 0
        mbar_expect_tx(&S.bar[warp], kN * sizeof(float));
        tma_bulk_g2s(S.line[warp], line_of(item), kN * sizeof(float), &S.bar[warp]);
    };
    if (kLine && lane == 0 && first < n_items) copy_line(first);
    uint32_t parity = 0;
    for (unsigned int item = first; item < n_items; item += step, parity ^= 1u) {
        const float2* ph = a.phase + static_cast<int64_t>(item / nbx) * kN + lane;
        const float* line = line_of(item) + lane;
        float* out = Pool ? sums : a.A + static_cast<int64_t>(item) * (Db ? a.nz : kHalf);
        // the warp's next line into L2 behind this one's transform
        if (!kLine && !Rep && lane == 0 && item + step < n_items) bulk_prefetch_l2(line_of(item + step), kN * sizeof(float));
        for (int rp = 0; rp < (Rep ? a.rep : 1); ++rp, line += static_cast<int64_t>(a.nx) * kN) {
            float2 v[64];
#pragma unroll
            for (int r = 0; r < 64; ++r)
                if (!kLine) v[r].x = ld_stream(line + 32 * r);
            if (kLine) {
                const bool ok = mbar_wait_bounded(&S.bar[warp], parity, a.status);
                if (!__all_sync(0xffffffffu, ok)) {
                    mbar_wait_bounded(&S.bar[warp], parity, a.status);   // the copy lands before the CTA ends
                    return;
                }
#pragma unroll
                for (int r = 0; r < 64; ++r) v[r].x = S.line[warp][lane + 32 * r];
                __syncwarp();
                if (lane == 0 && item + step < n_items) copy_line(item + step);
            }
#pragma unroll
            for (int r = 0; r < 64; ++r) {
                const float2 p = __ldg(ph + 32 * r);
                // complex64 (xv + 0i) * p, as numpy multiplies (dispersion.py:94)
                v[r] = make_float2(v[r].x * p.x, v[r].x * p.y);
            }
            ifft2048_low_mag_warp(v, ex, tw2, tw3, lane, [&](int k, float m) {
                if (Db) {
                    // (no branch around the few depths cropped)
                    const int z = k - a.z0;
                    const bool in = static_cast<unsigned int>(z) < static_cast<unsigned int>(a.nz);
                    const float db = 20.0f * log10f(m);
                    if (in) out[z] = db;
                    const bool use = in && isfinite(db);
                    run_min = fminf(run_min, use ? db : __int_as_float(0x7f800000));
                    run_max = fmaxf(run_max, use ? db : -__int_as_float(0x7f800000));
                    return;
                }
                if (!Rep) {
                    out[k] = m;
                    return;
                }
                // numpy's float32 mean over the repeats: sum, then divide
                const float t = (rp == 0 ? 0.f : sums[k]) + m;
                if (rp + 1 == a.rep)
                    out[k] = __fdiv_rn(t, static_cast<float>(a.rep));
                else
                    sums[k] = t;
            });
        }
        if (Pool) {
            // probe images: per image row zi the sum over depths
            // [zi z_keep / 256, ceil((zi + 1) z_keep / 256))
            __syncwarp();
            for (int zi = lane; zi < 256; zi += 32) {
                const int z0 = zi * a.z_keep / 256, z1 = ((zi + 1) * a.z_keep + 255) / 256;
                float sum = 0.f;
                for (int z = z0; z < z1; ++z) sum += sums[z];
                a.zcol[static_cast<int64_t>(item) * 256 + zi] = sum;
            }
            __syncwarp();
        }
    }
    if (Db && a.minmax != nullptr) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            run_min = fminf(run_min, __shfl_xor_sync(0xffffffffu, run_min, o));
            run_max = fmaxf(run_max, __shfl_xor_sync(0xffffffffu, run_max, o));
        }
        if (lane == 0 && run_min <= run_max) {
            atomicMin(&a.minmax[0], f2ord(run_min));
            atomicMax(&a.minmax[1], f2ord(run_max));
        }
    }
}

// Phase rows exp(-i beta dk^2), formed in float64, rounded to complex64
// (dispersion.py:88-89) and scaled by 1/N, one thread a sample.
__global__ void __launch_bounds__(256) k_phase(const double* __restrict__ betas, const double* __restrict__ dk2,
                                               int n, float2* __restrict__ phase) {
    const int i = blockIdx.x * 256 + threadIdx.x;
    if (i >= n * kN) return;
    double s, c;
    sincos(betas[i / kN] * dk2[i % kN], &s, &c);
    phase[i] = make_float2(static_cast<float>(c) * (1.0f / kN), static_cast<float>(-s) * (1.0f / kN));
}

// ---------------------------------------------------------------- block helpers
constexpr int kSelThreads = 1024;                // k_moments
constexpr int kTopThreads = 512;                 // k_top_sum

// Inclusive prefix sum of one value per thread over the block.
template <int kThr>
__device__ __forceinline__ unsigned int block_inclusive_scan(unsigned int v, unsigned int* warp_tot) {
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const unsigned int t = __shfl_up_sync(0xffffffffu, v, o);
        if (lane >= o) v += t;
    }
    if (lane == 31) warp_tot[w] = v;
    __syncthreads();
    if (w == 0) {
        unsigned int t = lane < kThr / 32 ? warp_tot[lane] : 0u;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const unsigned int u = __shfl_up_sync(0xffffffffu, t, o);
            if (lane >= o) t += u;
        }
        warp_tot[lane] = t;                     // inclusive over warps
    }
    __syncthreads();
    const unsigned int off = w > 0 ? warp_tot[w - 1] : 0u;
    __syncthreads();
    return v + off;
}

// The bin (counted from the top) holding the need-th largest element, and the
// number of elements in the bins above it.  hist has nbins entries.
template <int kThr>
__device__ __forceinline__ void find_from_top(const unsigned int* hist, int nbins, unsigned int need,
                                              unsigned int* warp_tot, int* bin_out, unsigned int* above_out) {
    const int chunk = (nbins + kThr - 1) / kThr;
    const int lo = threadIdx.x * chunk, hi = min(lo + chunk, nbins);
    unsigned int c = 0;
    for (int b = lo; b < hi; ++b) c += hist[b];
    const unsigned int incl = block_inclusive_scan<kThr>(c, warp_tot);
    __shared__ unsigned int total_s;
    if (threadIdx.x == kThr - 1) total_s = incl;
    __syncthreads();
    const unsigned int above = total_s - incl;     // elements in bins >= hi
    if (c > 0 && above < need && above + c >= need) {
        unsigned int ab = above;
        for (int b = hi - 1; b >= lo; --b) {
            if (ab + hist[b] >= need) {
                *bin_out = b;
                *above_out = ab;
                break;
            }
            ab += hist[b];
        }
    }
    __syncthreads();
}

__device__ __forceinline__ double block_sum_f64(double v, double* red) {
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    if (lane == 0) red[w] = v;
    __syncthreads();
    double t = 0.0;
    if (w == 0) {
        t = lane < static_cast<int>(blockDim.x >> 5) ? red[lane] : 0.0;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
        if (lane == 0) red[0] = t;
    }
    __syncthreads();
    t = red[0];
    __syncthreads();
    return t;
}

__device__ __forceinline__ double block_max_f64(double v, double* red) {
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = fmax(v, __shfl_xor_sync(0xffffffffu, v, o));
    if (lane == 0) red[w] = v;
    __syncthreads();
    double t = -__longlong_as_double(0x7ff0000000000000ll);
    if (w == 0) {
        t = red[lane];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) t = fmax(t, __shfl_xor_sync(0xffffffffu, t, o));
        if (lane == 0) red[0] = t;
    }
    __syncthreads();
    t = red[0];
    __syncthreads();
    return t;
}

// top_percentile of a segment (beta, B-scan) of A (nx rows of kHalf
// magnitudes): a cluster of C CTAs, each with its share of the rows, counts
// the first digit, collects the elements of the digit's bin (each thread its
// own, in its own slots, so that the order of every sum is fixed) while it sums
// the larger ones, and decides the other two digits among the collected ones:
// two passes over the magnitudes.  Rank 0's histogram gathers the cluster's
// through distributed shared memory.  C (set by the launcher) fills the GPU
// when there are few segments (the search's refinement rounds have 1 to 9).
// Bound by DRAM: 410 segments of 500 rows (840 MB, read twice) in 315 us =
// 5.3 TB/s; one CTA a segment reading four times, a float a load, took 1304 us.
constexpr int kTopSlots = 24;                     // collected elements of a thread; past them it reads A again

struct TopSmem {
    unsigned int hist[4096];
    unsigned int warp_tot[32];
    double red[32];
    int bin;
    unsigned int above;
    double part[8];                               // rank 0: the CTAs' sums
    unsigned int cand[kTopSlots][kTopThreads];
};

__global__ void __launch_bounds__(kTopThreads, 3) k_top_sum(const float* __restrict__ A, int nx, int z_min,
                                                            unsigned int k, double* __restrict__ score) {
    namespace cg = cooperative_groups;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    TopSmem& S = *reinterpret_cast<TopSmem*>(smem_raw);
    cg::cluster_group cl = cg::this_cluster();
    const int C = static_cast<int>(cl.num_blocks()), rank = static_cast<int>(cl.block_rank());
    TopSmem& S0 = *cl.map_shared_rank(&S, 0);
    const int tid = threadIdx.x;
    const int x0 = static_cast<int>(static_cast<int64_t>(nx) * rank / C);
    const int x1 = static_cast<int>(static_cast<int64_t>(nx) * (rank + 1) / C);
    const float* seg = A + (static_cast<int64_t>(blockIdx.x / C) * nx + x0) * kHalf;
    const bool vec = (reinterpret_cast<uintptr_t>(A) & 15u) == 0;   // a caller's buffer may be aligned to a float only
    // four depths a load: group q = i % 256 of row i / 256
    const int n4 = (x1 - x0) * (kHalf / 4);
    auto each = [&](auto&& f) {
        constexpr int kU = 4;                     // loads in flight
        for (int i0 = tid; i0 < n4; i0 += kU * kTopThreads) {
            float4 v[kU];
#pragma unroll
            for (int u = 0; u < kU; ++u) {
                const int i = i0 + u * kTopThreads;
                if (i >= n4) continue;
                const float* p = seg + 4 * static_cast<int64_t>(i);
                v[u] = vec ? __ldg(reinterpret_cast<const float4*>(p))
                           : make_float4(__ldg(p), __ldg(p + 1), __ldg(p + 2), __ldg(p + 3));
            }
#pragma unroll
            for (int u = 0; u < kU; ++u) {
                const int i = i0 + u * kTopThreads;
                const int z = 4 * (i & (kHalf / 4 - 1));
                if (i >= n4 || z + 3 < z_min) continue;
                if (z >= z_min) f(__float_as_uint(v[u].x) & 0x7fffffffu);
                if (z + 1 >= z_min) f(__float_as_uint(v[u].y) & 0x7fffffffu);
                if (z + 2 >= z_min) f(__float_as_uint(v[u].z) & 0x7fffffffu);
                f(__float_as_uint(v[u].w) & 0x7fffffffu);
            }
        }
    };
    // the digit's bin holding the need-th largest element of the cluster's
    // histograms, and the elements above it
    auto decide = [&](int nbins, unsigned int need, unsigned int& above) -> unsigned int {
        if (rank != 0) {
            __syncthreads();
            for (int b = tid; b < nbins; b += kTopThreads)
                if (S.hist[b] != 0u) atomicAdd(&S0.hist[b], S.hist[b]);
        }
        cl.sync();
        if (rank == 0) find_from_top<kTopThreads>(S.hist, nbins, need, S.warp_tot, &S.bin, &S.above);
        cl.sync();
        const unsigned int bin = static_cast<unsigned int>(S0.bin);
        above = S0.above;
        cl.sync();                                // read before the next digit's decision
        return bin;
    };
    auto clear = [&](int nbins) {
        for (int b = tid; b < nbins; b += kTopThreads) S.hist[b] = 0u;
        cl.sync();                                // rank 0's is clear before the others add to it
    };
    unsigned int above;
    clear(4096);
    each([&](unsigned int key) { atomicAdd(&S.hist[key >> 19], 1u); });
    const unsigned int p1 = decide(4096, k, above);        // bits 30..19
    unsigned int gt = above;
    // float64 sum of I = float32(A^2), in row order
    auto square = [](unsigned int key) {
        const float v = __uint_as_float(key);
        return static_cast<double>(__fmul_rn(v, v));
    };
    double s = 0.0;
    int n = 0;
    each([&](unsigned int key) {
        const unsigned int p = key >> 19;
        if (p < p1) return;
        if (p > p1) {
            s += square(key);
        } else {
            if (n < kTopSlots) S.cand[n][tid] = key;
            ++n;
        }
    });
    auto each_cand = [&](auto&& f) {
        if (n <= kTopSlots) {
            for (int i = 0; i < n; ++i) f(S.cand[i][tid]);
        } else {
            each([&](unsigned int key) {
                if ((key >> 19) == p1) f(key);
            });
        }
    };
    clear(2048);
    each_cand([&](unsigned int key) { atomicAdd(&S.hist[(key >> 8) & 0x7ffu], 1u); });
    const unsigned int p2 = (p1 << 11) | decide(2048, k - gt, above);
    gt += above;
    clear(256);
    each_cand([&](unsigned int key) {
        if ((key >> 8) == p2) atomicAdd(&S.hist[key & 0xffu], 1u);
    });
    const unsigned int thr = (p2 << 8) | decide(256, k - gt, above);
    gt += above;
    each_cand([&](unsigned int key) {
        if (key > thr) s += square(key);
    });
    s = block_sum_f64(s, S.red);
    if (tid == 0) S0.part[rank] = s;
    cl.sync();
    if (rank == 0 && tid == 0) {
        double top = static_cast<double>(k - gt) * square(thr);
        for (int r = 0; r < C; ++r) top += S.part[r];
        score[blockIdx.x / C] = log(top / static_cast<double>(k));
    }
}

// metric 2 kurtosis: sum(I^2) / sum(I)^2; 3 entropy: sum(p log(p + 1e-30)),
// p = I / sum(I); 4 legacy_peak: max_z mean_x log(A + 1e-12) (float32 as the
// reference's arrays).  I = float64(float32(A^2)).
__global__ void __launch_bounds__(kSelThreads, 1) k_moments(const float* __restrict__ A, int nx, int z_min,
                                                            int metric, double* __restrict__ score) {
    __shared__ double red[32];
    const float* seg = A + static_cast<int64_t>(blockIdx.x) * nx * kHalf;
    const int z = z_min + threadIdx.x;
    const bool act = z < kHalf;
    if (metric == 4) {
        float L = 0.f;
        if (act)
            for (int x = 0; x < nx; ++x) L += logf(seg[static_cast<int64_t>(x) * kHalf + z] + 1e-12f);
        const double mean = act ? static_cast<double>(__fdiv_rn(L, static_cast<float>(nx)))
                                : -__longlong_as_double(0x7ff0000000000000ll);
        const double m = block_max_f64(mean, red);
        if (threadIdx.x == 0) score[blockIdx.x] = m;
        return;
    }
    double s1 = 0.0, s2 = 0.0;
    if (act)
        for (int x = 0; x < nx; ++x) {
            const float v = seg[static_cast<int64_t>(x) * kHalf + z];
            const double I = static_cast<double>(__fmul_rn(v, v));
            s1 += I;
            s2 += I * I;
        }
    s1 = block_sum_f64(s1, red);
    if (metric == 2) {
        s2 = block_sum_f64(s2, red);
        if (threadIdx.x == 0) score[blockIdx.x] = s2 / (s1 * s1);
        return;
    }
    double e = 0.0;
    if (act)
        for (int x = 0; x < nx; ++x) {
            const float v = seg[static_cast<int64_t>(x) * kHalf + z];
            const double p = static_cast<double>(__fmul_rn(v, v)) / s1;
            e += p * log(p + 1e-30);
        }
    e = block_sum_f64(e, red);
    if (threadIdx.x == 0) score[blockIdx.x] = e;
}

// ---------------------------------------------------------------- x-median
constexpr int kMedThreads = 256;
constexpr int kMedMaxX = 4096;
constexpr int kMedMaxReg = 1024;                  // columns of up to this many A-scans are held in registers

// A block takes kCols depth columns of a frame: rows x read along depth into
// shared memory (pitch kCols + 1: a column's reads fall in distinct banks), a
// warp per column.  The median is found by bisection on the ordered float
// bits: 32 times the warp counts its keys below a candidate (kReg keys a lane
// in registers; kReg = 0 reads them from shared memory each time).  Issue-bound:
// ~2 instructions a key and bit.  9216 columns of 333 A-scans take 29 us; the
// bitonic sort of a column per warp in shared memory before it took 169 us.  Up
// to 32 A-scans a column is one key a lane and sorted by shuffles (a whole call of
// 200 frames of 32: 80 us, 264 by bisection, 162 before it).
// mean_mode: the float64 mean of the non-NaN values instead of the median.
template <int kCols, int kReg>
__global__ void __launch_bounds__(kMedThreads) k_xmedian(const float* __restrict__ mag, int nx, int nz,
                                                         int ignore_nan, int mean_mode, double* __restrict__ out) {
    extern __shared__ __align__(16) float tile[];  // [nx][kCols + 1]
    constexpr int kPitch = kCols + 1;
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int64_t f = blockIdx.y;
    const int z0 = blockIdx.x * kCols;
    for (int e = threadIdx.x; e < nx * kCols; e += kMedThreads) {
        const int x = e / kCols, c = e % kCols;
        if (z0 + c < nz) tile[x * kPitch + c] = mag[(f * nx + x) * nz + z0 + c];
    }
    __syncthreads();
    for (int c = w; c < kCols && z0 + c < nz; c += kMedThreads / 32) {
        const float* s = tile + c;
        double* o = out + f * nz + z0 + c;
        if (mean_mode) {
            double acc = 0.0;
            int nn = 0;
            for (int i = lane; i < nx; i += 32) {
                const float v = s[i * kPitch];
                nn += isnan(v);
                if (!isnan(v)) acc += static_cast<double>(v);
            }
            nn = __reduce_add_sync(0xffffffffu, nn);
            for (int d = 16; d > 0; d >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, d);
            if (lane == 0) *o = nx > nn ? acc / (nx - nn) : __longlong_as_double(0x7ff8000000000000ll);
            continue;
        }
        // ordered keys; NaN and padding above every value
        unsigned int key[kReg > 0 ? kReg : 1];
        int nn = 0;
        auto key_of = [&](int i) -> unsigned int {
            const float v = i < nx ? s[i * kPitch] : 0.f;
            return i >= nx || isnan(v) ? 0xffffffffu : f2ord(v + 0.0f);
        };
        if (kReg > 0) {
#pragma unroll
            for (int i = 0; i < kReg; ++i) key[i] = key_of(lane + 32 * i);
        }
        auto each = [&](auto&& g) {
            if (kReg > 0) {
#pragma unroll
                for (int i = 0; i < kReg; ++i) g(key[i]);
            } else {
                for (int i = lane; i < nx; i += 32) g(key_of(i));
            }
        };
        each([&](unsigned int k) { nn += k != 0xffffffffu; });
        const int n = __reduce_add_sync(0xffffffffu, nn);                  // values that are not NaN
        if (n == 0 || (n < nx && !ignore_nan)) {
            if (lane == 0) *o = __longlong_as_double(0x7ff8000000000000ll);
            continue;
        }
        // the key of rank k0 (the middle one, or the lower of the two)
        const int k0 = (n - 1) / 2;
        if (kReg == 1) {
            // one key a lane: sorted by a bitonic network of shuffles
            unsigned int v = key[0];
#pragma unroll
            for (int k = 2; k <= 32; k <<= 1)
#pragma unroll
                for (int j = k >> 1; j > 0; j >>= 1) {
                    const unsigned int u = __shfl_xor_sync(0xffffffffu, v, j);
                    v = ((lane & j) == 0) == ((lane & k) == 0) ? min(v, u) : max(v, u);
                }
            const double lo = static_cast<double>(ord2f(__shfl_sync(0xffffffffu, v, k0)));
            const double hi = static_cast<double>(ord2f(__shfl_sync(0xffffffffu, v, n / 2)));
            if (lane == 0) *o = (n & 1) ? lo : (lo + hi) / 2.0;
            continue;
        }
        unsigned int med = 0u;
#pragma unroll 1
        for (int bit = 31; bit >= 0; --bit) {
            const unsigned int cand = med | (1u << bit);
            int below = 0;
            each([&](unsigned int k) { below += k < cand; });
            if (__reduce_add_sync(0xffffffffu, below) <= k0) med = cand;
        }
        double m = static_cast<double>(ord2f(med));
        if ((n & 1) == 0) {
            // the upper of the two: the same key when it repeats past rank k0, else the next larger one
            int le = 0;
            unsigned int next = 0xffffffffu;
            each([&](unsigned int k) {
                if (k <= med) ++le; else next = k < next ? k : next;
            });
            le = __reduce_add_sync(0xffffffffu, le);
            next = __reduce_min_sync(0xffffffffu, next);
            m = (m + static_cast<double>(ord2f(le > k0 + 1 ? med : next))) / 2.0;
        }
        if (lane == 0) *o = m;
    }
}

template <int kCols, int kReg>
cudaError_t launch_xmedian_t(const float* mag, int n_frames, int nx, int nz, int ignore_nan, int mean_mode,
                             double* out, cudaStream_t st) {
    const size_t smem = static_cast<size_t>(nx) * (kCols + 1) * sizeof(float);
    cudaError_t e = cudaFuncSetAttribute(k_xmedian<kCols, kReg>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         static_cast<int>(smem));
    if (e != cudaSuccess) return e;
    const dim3 grid((nz + kCols - 1) / kCols, n_frames);
    k_xmedian<kCols, kReg><<<grid, kMedThreads, smem, st>>>(mag, nx, nz, ignore_nan, mean_mode, out);
    return cudaGetLastError();
}

}  // namespace

cudaError_t launch_disp_mag(const DispArgs& a, int num_sms, cudaStream_t st) {
    if (a.mode == kModeDb && (a.rep > 1 || a.zcol != nullptr)) return cudaErrorInvalidValue;
    const int64_t items = static_cast<int64_t>(a.n_beta) * a.nb * a.nx;
    if (items >= (int64_t(1) << 32) - 12 * num_sms) return cudaErrorInvalidValue;   // 32-bit item index
    const bool extra = a.zcol != nullptr || a.rep > 1;
    const bool line = !extra && items >= static_cast<int64_t>(kLineItems) * kLineWarps * num_sms;
    const int warps = line ? kLineWarps : kDispWarps, per_sm = line ? 1 : 3;
    const size_t smem = line ? sizeof(DispSmem<kLineWarps, true>)
                             : sizeof(DispSmem<kDispWarps, false>) + (extra ? kDispWarps * kHalf * sizeof(float) : 0);
    const auto kernel = a.mode == kModeDb   ? (line ? k_disp_mag<false, true, false, true>
                                                    : k_disp_mag<false, true, false, false>)
                        : a.zcol != nullptr ? (a.rep > 1 ? k_disp_mag<true, false, true, false>
                                                         : k_disp_mag<true, false, false, false>)
                        : a.rep > 1         ? k_disp_mag<false, false, true, false>
                        : line              ? k_disp_mag<false, false, false, true>
                                            : k_disp_mag<false, false, false, false>;
    const int bit = line                  ? (a.mode == kModeDb ? 6 : 5)
                    : a.mode == kModeDb ? 4
                                        : (a.zcol != nullptr ? 2 : 0) + (a.rep > 1 ? 1 : 0);
    const cudaError_t e = kernel_ready(a.ready, kReadyDisp + bit, kernel, smem);
    if (e != cudaSuccess) return e;
    const int64_t most = static_cast<int64_t>(per_sm) * num_sms, want = (items + warps - 1) / warps;
    const unsigned int grid = static_cast<unsigned int>(want < most ? want : most);
    return launch_dependent(kernel, dim3(grid), dim3(warps * 32), smem, st, a);
}

cudaError_t launch_phase(const double* betas, const double* dk2, int n, float2* phase, cudaStream_t st) {
    k_phase<<<n * (kN / 256), 256, 0, st>>>(betas, dk2, n, phase);
    return cudaGetLastError();
}

cudaError_t launch_disp_metric(const float* A, int n_seg, int nx, int z_min, int metric, unsigned int top_k,
                               double* score, int num_sms, cudaStream_t st) {
    if (metric == 1) {
        // three CTAs an SM: the widest cluster (1 to 8 CTAs a segment) that one wave holds
        int C = 8;
        while (C > 1 && (static_cast<int64_t>(n_seg) * C > 3 * num_sms || nx < C)) C >>= 1;
        cudaError_t e = cudaFuncSetAttribute(k_top_sum, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                             static_cast<int>(sizeof(TopSmem)));
        if (e != cudaSuccess) return e;
        cudaLaunchAttribute at{};
        at.id = cudaLaunchAttributeClusterDimension;
        at.val.clusterDim.x = static_cast<unsigned int>(C);
        at.val.clusterDim.y = at.val.clusterDim.z = 1;
        cudaLaunchConfig_t cfg{};
        cfg.gridDim = dim3(static_cast<unsigned int>(n_seg * C));
        cfg.blockDim = dim3(kTopThreads);
        cfg.dynamicSmemBytes = sizeof(TopSmem);
        cfg.stream = st;
        cfg.attrs = &at;
        cfg.numAttrs = 1;
        return cudaLaunchKernelEx(&cfg, k_top_sum, A, nx, z_min, top_k, score);
    } else
        k_moments<<<n_seg, kSelThreads, 0, st>>>(A, nx, z_min, metric, score);
    return cudaGetLastError();
}

cudaError_t launch_xmedian(const float* mag, int n_frames, int nx, int nz, int ignore_nan, int mean_mode,
                           double* out, cudaStream_t st) {
    if (nx > kMedMaxX) return cudaErrorInvalidValue;
    // 16 columns (64-byte rows) while their tile leaves several blocks an SM,
    // 8 for long columns (147 KB at 4096 A-scans) and where 16 would leave SMs idle
    // (one frame of 32 A-scans, a whole call: mean 27 -> 21 us)
    const bool few = static_cast<int64_t>(n_frames) * ((nz + 15) / 16) < 152;
    const auto f = nx <= 32           ? (few ? launch_xmedian_t<8, 1> : launch_xmedian_t<16, 1>)
                   : nx <= 256        ? (few ? launch_xmedian_t<8, 8> : launch_xmedian_t<16, 8>)
                   : nx <= 512        ? (few ? launch_xmedian_t<8, 16> : launch_xmedian_t<16, 16>)
                   : nx <= kMedMaxReg ? (few ? launch_xmedian_t<8, 32> : launch_xmedian_t<16, 32>)
                                      : launch_xmedian_t<8, 0>;
    return f(mag, n_frames, nx, nz, ignore_nan, mean_mode, out, st);
}

}  // namespace octgb

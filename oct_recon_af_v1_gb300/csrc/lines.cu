// Spectral stage up to the transform for sm_103a: raw camera counts ->
// background-free, k-linearised lines.
//
// Per A-scan (2048 samples):
//   d[j] = float(raw[j]) - apod[j] (float32 apodisation mean of the B-scan,
//     rounded from an exact sum as core/cpu_kernels.py:20-25 does), line mean
//     m removed (cpu_kernels.py:26-36);
//   v[i] = sum_t w[t,i] (d - m)[start_i + t] + m (banded sinc, cpu_kernels.py:
//     37-40, float32 accumulation), written as the real line that the
//     transform (estimate.cu) takes, times the complex window (the fused
//     pre-FFT operator's output, cpu_kernels.py:41) or times a float64 window
//     rounded once (the scorer's lines).
//
// k_lines is one persistent CTA an SM with two kinds of warps, joined by a
// ring of background-free lines in shared memory:
//   sinc warps (16)        thread t owns outputs 4t .. 4t + 3; its band weights
//                          stay in registers for the whole launch, in a dense
//                          form over its window of U source samples.  Step u
//                          reads the sample congruent to u (mod U): at one
//                          step a warp's threads read the same samples or
//                          samples U apart, which with gcd(U, 32) = 2 lie in
//                          distinct banks;
//   background warps       one A-scan each: the raw row arrives by a bulk copy
//                          two A-scans ahead, the apodisation-mean row when the
//                          B-scan changes; 64 samples a lane stay in registers
//                          until the line mean is known, so no two warps wait
//                          for one another except through the ring.
// A CTA takes a contiguous range of A-scans, so the apodisation row changes
// once a B-scan.
//
// Exact (integer raws; the precision form): the background without the float32
// form's rounding of the apodisation mean.  With S the integer sum of the
// apodisation lines and A their count, n = A raw - S is an exact integer, the
// line mean m = sum(n) / (2048 A) comes from integer sums, and
// d - m = fma(n, 1/A, -m) takes one rounding; then the same band.  30 000
// A-scans to magnitudes in 217 us, 1.2e-7 off float64 (2-norm); with a
// split-FP16 tensor-core product over 96-sample windows (1.5 x the outputs,
// three products, copies of 16-byte rows: 248 us of its 351) 2.2e-7.
// Bound by the shared-memory path: 471 wavefronts an A-scan, 67 % of its
// cycles, with 1718 warp instructions (issue active 52 %); 25 000 A-scans in
// 65 us (382 M/s, 12.4 kB read and written an A-scan = 4.7 TB/s).  With the
// transform after it (estimate.cu) they take 260 us to dB rows; one kernel for
// both, 512 threads in lock step through two block barriers per four A-scans
// (1619 wavefronts, 5880 instructions an A-scan), took 314 us, and 324 000
// A-scans stitched 3888 us against 2690 now (with the stitch's own changes).
#include <cuda_runtime.h>
#include <stdint.h>

#include "octgb_device.cuh"
#include "octgb_internal.h"

namespace octgb {
namespace {

constexpr int kSincWarps = 16;                   // 512 threads x 4 outputs
// Wide windows (U > 18): a sinc thread's 4 U weights do not fit its 96 registers
// (17 to 20 warps are five on a scheduler, so fewer background warps give it no
// more).  The compiler kept what did not fit in local memory, which the L1 beside
// 160 KB and more of shared memory does not hold either: 100 000 A-scans to
// magnitudes with U = 22 took 1622 us (uint16) and 1912 (float32).  The weights of
// the window's steps from kRegSteps on now lie in shared memory, eight bytes a
// thread and bank-conflict free: 797 and 827 us (U = 26: 1784 and 1857, now 904 and
// 1000).  Two background warps leave the room for them.
constexpr int kRegSteps = 16;
constexpr int bg_warps(int U) { return U <= 18 ? 4 : 2; }
constexpr int reg_steps(int U) { return U <= 18 ? U : kRegSteps; }
constexpr int lines_threads(int U) { return (kSincWarps + bg_warps(U)) * 32; }
constexpr int kRing = 8;                         // background-free lines in shared memory
constexpr int kDLine = kN + kTail;               // line incl. zero tail (16-byte rows)

// float32 values of four raw samples
template <typename RawT>
__device__ __forceinline__ void raw4(const RawT* p, float2& a, float2& b);
// 2^23 + u is exact in float32 with u in its low bits, so subtracting 2^23
// gives the 16-bit integer u exactly, two at a time (int16: u offset by 2^15)
__device__ __forceinline__ void raw4_u16(uint2 q, uint32_t flip, float2 off, float2& a, float2& b) {
    q.x ^= flip;
    q.y ^= flip;
    a = sub2(make_float2(__uint_as_float(__byte_perm(q.x, 0x4b000000u, 0x7610)),
                         __uint_as_float(__byte_perm(q.x, 0x4b000000u, 0x7632))),
             off);
    b = sub2(make_float2(__uint_as_float(__byte_perm(q.y, 0x4b000000u, 0x7610)),
                         __uint_as_float(__byte_perm(q.y, 0x4b000000u, 0x7632))),
             off);
}
template <>
__device__ __forceinline__ void raw4<uint16_t>(const uint16_t* p, float2& a, float2& b) {
    raw4_u16(*reinterpret_cast<const uint2*>(p), 0u, make_float2(8388608.f, 8388608.f), a, b);
}
template <>
__device__ __forceinline__ void raw4<int16_t>(const int16_t* p, float2& a, float2& b) {
    raw4_u16(*reinterpret_cast<const uint2*>(p), 0x80008000u, make_float2(8421376.f, 8421376.f), a, b);
}
template <>
__device__ __forceinline__ void raw4<float>(const float* p, float2& a, float2& b) {
    const float4 u = *reinterpret_cast<const float4*>(p);
    a = make_float2(u.x, u.y);
    b = make_float2(u.z, u.w);
}

// float32(float64(x) * h), two samples at a time, for float64 h given as float32
// hi + lo (the rest below 2^-48 |h|) without the FP64 pipe: p + e1 = x * hi
// exactly (fma), q = x lo + e1 (one rounding), o = p + q rounded once.  The
// exact product differs from p + q by < 2^-46 |o|; when p + q lies more than
// 2^-40 |o| from a float32 rounding boundary (r = (p + q) - o exactly, by
// Fast2Sum), both the product and its float64 rounding round to o.  |o| of
// exponent e has its boundaries 2^(e-24) away, a power of two the lower one half
// as far (hence the exponent of the bits - 1, for both), and 2^-15 of that
// covers 2^-40 |o|: safe when |r| < 2^(e-24) (1 - 2^-15).  Otherwise (about one
// sample in 33 000), and for tiny, infinite and NaN values, the float64 product is
// formed as the reference does: by the caller for the lanes whose `safe` is false,
// behind a warp vote, so the FP64 pipe only runs in the rare warps that need it.
// (One sample at a time, with the distance to the boundary formed per sample, the
// window was half of the sinc warps' instructions: 274 -> 235 us for 50 000 lines.)
__device__ __forceinline__ float2 mul_window2(float2 x, float2 hi, float2 lo, float2& p, bool& safe0, bool& safe1) {
    const float2 nx = make_float2(-x.x, -x.y), nz = make_float2(-0.f, -0.f);
    p = fma2(x, hi, nz);
    const float2 nq = fma2(nx, lo, fma2(nx, hi, p));
    const float2 o = sub2(p, nq);
    const float2 r = add2(nq, sub2(o, p));                    // -r
    constexpr float kEdge = 5.9602826e-08f;                   // 2^-24 (1 - 2^-15)
    const float e0 = __int_as_float((__float_as_int(o.x) - 1) & 0x7f800000) * kEdge;
    const float e1 = __int_as_float((__float_as_int(o.y) - 1) & 0x7f800000) * kEdge;
    safe0 = fabsf(r.x) < e0 && fabsf(o.x) > 1e-30f;
    safe1 = fabsf(r.y) < e1 && fabsf(o.y) > 1e-30f;
    return o;
}

template <typename RawT, int U>
struct LinesSmem {
    static constexpr int kBgWarps = bg_warps(U);
    uint64_t raw_full[kBgWarps][2], full[kRing], empty[kRing];
    int abort;
    float mval[kRing];
    alignas(16) RawT raw[kBgWarps][2][kN];
    alignas(16) float apod[kBgWarps][2][kN];
    alignas(16) float d[kRing][kDLine];
    float2 w[U > reg_steps(U) ? U - reg_steps(U) : 1][2][U > reg_steps(U) ? kSincWarps * 32 : 1];   // weights of steps reg_steps(U) .. U - 1
};
static_assert(sizeof(LinesSmem<float, 18>) <= 232448 && sizeof(LinesSmem<float, 26>) <= 232448, "k_lines shared memory exceeds 227 KB");

// the place of one A-scan: segment (or tile), B-scan, column
struct LinePos {
    unsigned int sg, b, x;
};

// sum of the two 16-bit integers of a word, added to c
template <typename RawT>
__device__ __forceinline__ int add_pair(uint32_t w, int c) {
    return static_cast<RawT>(-1) < 0 ? __dp2a_lo(static_cast<int>(w), 0x0101, c)
                                     : static_cast<int>(__dp2a_lo(w, 0x0101u, static_cast<uint32_t>(c)));
}

// With more apodisation lines than this A raw - S may not be exact in float32,
// and the sums are kept as integers.
constexpr int kExactFloat = 255;

template <typename RawT, int Mode, int U, bool Tiles, bool Exact>
__global__ void __launch_bounds__(lines_threads(U), 1) k_lines(const LinesArgs a) {
    constexpr int kBgWarps = bg_warps(U), kThr = lines_threads(U);
    extern __shared__ __align__(128) unsigned char smem_raw[];
    using Smem = LinesSmem<RawT, U>;
    Smem& S = *reinterpret_cast<Smem*>(smem_raw);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    // this CTA's A-scans
    const unsigned int n_all = a.l1 - a.l0;
    const unsigned int first = a.l0 + static_cast<unsigned int>(static_cast<uint64_t>(n_all) * blockIdx.x / gridDim.x);
    const int n = static_cast<int>(
        a.l0 + static_cast<unsigned int>(static_cast<uint64_t>(n_all) * (blockIdx.x + 1) / gridDim.x) - first);

    if (tid == 0) {
        for (int w = 0; w < kBgWarps; ++w)
            for (int s = 0; s < 2; ++s) mbar_init(&S.raw_full[w][s], 1);
        for (int s = 0; s < kRing; ++s) {
            mbar_init(&S.full[s], 1);
            mbar_init(&S.empty[s], kSincWarps);
        }
        S.abort = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    for (int k = tid; k < kRing * kTail; k += kThr) S.d[k / kTail][kN + k % kTail] = 0.f;
    // a wait that runs out ends every role of the CTA
    auto wait = [&](uint64_t* bar, uint32_t parity) -> bool {
        if (*reinterpret_cast<volatile int*>(&S.abort)) return false;
        if (mbar_wait_bounded(bar, parity, a.status)) return true;
        atomicExch(&S.abort, 1);
        return false;
    };

    if (warp >= kSincWarps) {
        // ------------------------------------------------ background
        const int w = warp - kSincWarps;
        __syncthreads();
        pdl_wait();                                          // the lines' readers, the apodisation means
        pdl_launch();
        if (w >= n) return;
        LinePos pos;
        auto dims = [&](unsigned int sg, unsigned int& B, unsigned int& nx) {
            if (Tiles) {
                B = static_cast<unsigned int>(a.qt[sg].B);
                nx = static_cast<unsigned int>(a.qt[sg].nx);
            } else {
                B = static_cast<unsigned int>(a.B);
                nx = static_cast<unsigned int>(a.nx);
            }
        };
        {
            unsigned int l = first + static_cast<unsigned int>(w);
            if (Tiles) {
                int lo = 0, hi = a.n_qt - 1;                 // last tile with line0 <= l
                while (lo < hi) {
                    const int mid = (lo + hi + 1) >> 1;
                    if (a.qt[mid].line0 <= l) lo = mid; else hi = mid - 1;
                }
                pos.sg = static_cast<unsigned int>(lo);
                l -= a.qt[lo].line0;
            } else {
                pos.sg = l / (static_cast<unsigned int>(a.B) * static_cast<unsigned int>(a.nx));
                l -= pos.sg * (static_cast<unsigned int>(a.B) * static_cast<unsigned int>(a.nx));
            }
            unsigned int B, nx;
            dims(pos.sg, B, nx);
            pos.b = l / nx;
            pos.x = l - pos.b * nx;
        }
        auto row_of = [&](const LinePos& p, unsigned int& apod_row) -> const RawT* {
            if (Tiles) {
                const QueueTile& t = a.qt[p.sg];
                apod_row = static_cast<unsigned int>(t.apod_row0) + p.b;
                return static_cast<const RawT*>(t.raw) +
                       (static_cast<int64_t>(p.b) * t.interf + t.apod + p.x) * kN;
            }
            apod_row = p.sg * static_cast<unsigned int>(a.B) + p.b;
            return static_cast<const RawT*>(a.seg[p.sg]) +
                   (static_cast<int64_t>(p.b) * a.interf + a.apod + p.x) * kN;
        };
        auto advance = [&](LinePos& p) {                     // kBgWarps A-scans on (tiles without A-scans are skipped)
            unsigned int B, nx;
            dims(p.sg, B, nx);
            p.x += kBgWarps;
            while (p.x >= nx) {
                p.x -= nx;
                if (++p.b == B) {
                    p.b = 0;
                    do {
                        ++p.sg;
                        dims(p.sg, B, nx);
                    } while (B == 0);
                }
            }
        };
        // A-scan k of this warp: raw row into stage k & 1, its apodisation row
        // into the other slot when it differs from the previous A-scan's
        unsigned int have_row = 0xffffffffu;
        int slot = 0;
        auto issue = [&](int k, const LinePos& p) -> bool {
            unsigned int ar;
            const RawT* row = row_of(p, ar);
            const bool load = ar != have_row;
            if (load) {
                have_row = ar;
                slot ^= 1;
            }
            if (lane == 0) {
                uint64_t* bar = &S.raw_full[w][k & 1];
                mbar_expect_tx(bar, kN * sizeof(RawT) + (load ? kN * sizeof(float) : 0) +
                                        starved_bytes(w == 0 && k == 0));
                tma_bulk_g2s(S.raw[w][k & 1], row, kN * sizeof(RawT), bar);
                if (load)
                    tma_bulk_g2s(S.apod[w][slot], a.apod_mean + static_cast<int64_t>(ar) * kN, kN * sizeof(float), bar);
            }
            return load;
        };
        const int mine = (n - w + kBgWarps - 1) / kBgWarps;    // A-scans of this warp
        issue(0, pos);
        int issued = 1;
        bool ok = true, fresh = true, fresh_next = false;    // the A-scan's apodisation row is new
        long long row_sum = 0;                               // Exact: sum of S over the row
        const bool exact_float = Exact && a.apod <= kExactFloat;
        const float apod_f = static_cast<float>(a.apod), inv_apod = 1.0f / apod_f;
        for (int k = 0; k < mine; ++k) {
            const int cur = slot;                            // the current A-scan's apodisation row
            if (k + 1 < mine) {
                advance(pos);
                __syncwarp();                                // stage (k + 1) & 1 was read by every lane
                fresh_next = issue(k + 1, pos);
                ++issued;
            }
            ok = wait(&S.raw_full[w][k & 1], static_cast<uint32_t>(k >> 1) & 1u);
            if (__any_sync(0xffffffffu, !ok)) break;
            float2 d[32];
            float m;
            const RawT* rw = S.raw[w][k & 1] + 4 * lane;
            const float* ap = S.apod[w][cur] + 4 * lane;
            if constexpr (Exact) {
                int tot = 0;
                if (fresh) {
                    row_sum = 0;
#pragma unroll
                    for (int i = 0; i < 16; ++i) {
                        const int4 q = *reinterpret_cast<const int4*>(ap + 128 * i);
                        row_sum += exact_float
                                       ? -static_cast<long long>(__int_as_float(q.x)) - static_cast<long long>(__int_as_float(q.y)) -
                                             static_cast<long long>(__int_as_float(q.z)) - static_cast<long long>(__int_as_float(q.w))
                                       : static_cast<long long>(q.x) + q.y + q.z + q.w;
                    }
#pragma unroll
                    for (int o = 16; o > 0; o >>= 1) row_sum += __shfl_xor_sync(0xffffffffu, row_sum, o);
                }
#pragma unroll
                for (int i = 0; i < 16; ++i) {
                    const uint2 q = *reinterpret_cast<const uint2*>(rw + 128 * i);
                    tot = add_pair<RawT>(q.y, add_pair<RawT>(q.x, tot));
                    if (exact_float) {
                        // the row holds -S; A raw - S exactly
                        float2 r01, r23;
                        raw4<RawT>(rw + 128 * i, r01, r23);
                        const float4 ns = *reinterpret_cast<const float4*>(ap + 128 * i);
                        const float2 a2 = make_float2(apod_f, apod_f);
                        d[2 * i] = fma2(r01, a2, make_float2(ns.x, ns.y));
                        d[2 * i + 1] = fma2(r23, a2, make_float2(ns.z, ns.w));
                    } else {
                        const int4 sv = *reinterpret_cast<const int4*>(ap + 128 * i);
                        d[2 * i].x = static_cast<float>(a.apod * static_cast<int>(static_cast<RawT>(q.x & 0xffffu)) - sv.x);
                        d[2 * i].y = static_cast<float>(a.apod * static_cast<int>(static_cast<RawT>(q.x >> 16)) - sv.y);
                        d[2 * i + 1].x = static_cast<float>(a.apod * static_cast<int>(static_cast<RawT>(q.y & 0xffffu)) - sv.z);
                        d[2 * i + 1].y = static_cast<float>(a.apod * static_cast<int>(static_cast<RawT>(q.y >> 16)) - sv.w);
                    }
                }
                const long long sum_n = static_cast<long long>(a.apod) * __reduce_add_sync(0xffffffffu, tot) - row_sum;
                m = static_cast<float>(sum_n) / (static_cast<float>(kN) * apod_f);
            } else {
                // lane holds samples 4 lane + 128 i .. + 3, i = 0 .. 15 (i = p + 4 q).
                // The sum keeps the order of the four partial sums of 128 threads
                // with 16 samples each: p = lt / 32 of thread lt's, q within it.
                float part[4];
#pragma unroll
                for (int p = 0; p < 4; ++p) {
                    float sum = 0.f;
#pragma unroll
                    for (int q = 0; q < 4; ++q) {
                        const int i = p + 4 * q;
                        float2 r01, r23;
                        raw4<RawT>(rw + 128 * i, r01, r23);
                        const float4 m = *reinterpret_cast<const float4*>(ap + 128 * i);
                        d[2 * i] = sub2(r01, make_float2(m.x, m.y));
                        d[2 * i + 1] = sub2(r23, make_float2(m.z, m.w));
                        sum += (d[2 * i].x + d[2 * i].y) + (d[2 * i + 1].x + d[2 * i + 1].y);
                    }
                    part[p] = sum;
                }
                // the four trees over 32 lanes (o = 16, 8, 4, 2, 1), two at a time
                // after the first two steps: lane bit 4 selects the pair, bit 3 the sum
                float s0, s1;
                {
                    const bool up = (lane & 16) != 0;
                    s0 = (up ? part[2] : part[0]) + __shfl_xor_sync(0xffffffffu, up ? part[0] : part[2], 16);
                    s1 = (up ? part[3] : part[1]) + __shfl_xor_sync(0xffffffffu, up ? part[1] : part[3], 16);
                    const bool up2 = (lane & 8) != 0;
                    s0 = (up2 ? s1 : s0) + __shfl_xor_sync(0xffffffffu, up2 ? s0 : s1, 8);
                }
#pragma unroll
                for (int o = 4; o > 0; o >>= 1) s0 += __shfl_xor_sync(0xffffffffu, s0, o);
                s0 += __shfl_xor_sync(0xffffffffu, s0, 8);       // part 0 + part 1, part 2 + part 3
                s0 += __shfl_xor_sync(0xffffffffu, s0, 16);
                m = s0 * (1.0f / kN);
            }
            const int i_line = w + kBgWarps * k, st = i_line % kRing;
            ok = wait(&S.empty[st], (static_cast<uint32_t>(i_line / kRing) & 1u) ^ 1u);
            if (__any_sync(0xffffffffu, !ok)) break;
            const float2 m2 = make_float2(m, m), nm2 = make_float2(-m, -m), ia2 = make_float2(inv_apod, inv_apod);
#pragma unroll
            for (int i = 0; i < 16; ++i) {
                const float2 e01 = Exact ? fma2(d[2 * i], ia2, nm2) : sub2(d[2 * i], m2);
                const float2 e23 = Exact ? fma2(d[2 * i + 1], ia2, nm2) : sub2(d[2 * i + 1], m2);
                *reinterpret_cast<float4*>(&S.d[st][4 * lane + 128 * i]) = make_float4(e01.x, e01.y, e23.x, e23.y);
            }
            if (lane == 0) S.mval[st] = m;
            __syncwarp();
            if (lane == 0) mbar_arrive(&S.full[st]);
            fresh = fresh_next;
        }
        // copies still in flight land before the CTA's memory is released
        if (!ok || issued < mine)
            for (int k = issued - 2 < 0 ? 0 : issued - 2; k < issued; ++k)
                mbar_wait_bounded(&S.raw_full[w][k & 1], static_cast<uint32_t>(k >> 1) & 1u, a.status);
        return;
    }

    // ---------------------------------------------------- sinc
    // the weights of outputs 4t, 4t + 1 (4t + 2, 4t + 3) at window step u form
    // one packed pair wp[0][u] (wp[1][u]): two outputs per f32x2 fma
    constexpr int kReg = reg_steps(U);
    float2 wp[2][kReg];
#pragma unroll
    for (int h = 0; h < 2; ++h)
        for (int u = kReg; u < U; ++u) S.w[u - kReg][h][tid] = __ldg(a.g.wsh + (h * U + u) * (kSincWarps * 32) + tid);
#pragma unroll
    for (int h = 0; h < 2; ++h)
#pragma unroll
        for (int u = 0; u < kReg; ++u) wp[h][u] = __ldg(a.g.wsh + (h * U + u) * (kSincWarps * 32) + tid);
    const int s0 = __ldg(a.g.s0 + tid);
    const int wrot = s0 % U;                                 // window samples before s0 wrap to the next period
    const int wbase = s0 - wrot;
    float4 wa{}, wb{};                                       // window of outputs 4t .. 4t + 3
    if (Mode == kModeSpec) {
        wa = __ldg(reinterpret_cast<const float4*>(a.g.win + 4 * tid));
        wb = __ldg(reinterpret_cast<const float4*>(a.g.win + 4 * tid + 2));
    }
    bool end0 = false, end3 = false;                         // kModeLinHann: window values of exactly zero
    if (Mode == kModeLinHann) {
        end0 = a.hann2[4 * tid] == 0.f && a.hann2[kN + 4 * tid] == 0.f;
        end3 = a.hann2[4 * tid + 3] == 0.f && a.hann2[kN + 4 * tid + 3] == 0.f;
    }
    __syncthreads();
    pdl_wait();                                              // the previous lines have been read
    pdl_launch();
    const int64_t out0 = static_cast<int64_t>(first - a.out_l0);
    // two A-scans an iteration (their ring stages are adjacent, so the window
    // addresses are formed once for both)
    for (int i = 0; i < n; i += 2) {
        const int st = i % kRing;
        const uint32_t ph = static_cast<uint32_t>(i / kRing) & 1u;
        const bool two = i + 1 < n;
        bool ok = wait(&S.full[st], ph);
        if (ok && two) ok = wait(&S.full[st + 1], ph);
        if (__any_sync(0xffffffffu, !ok)) return;
        const float* dk = S.d[st] + wbase;
        float2 acc[2][2] = {};
        // Exact: the window in two halves, their sums added last (each rounds
        // at about half the magnitude)
        constexpr int kHalfU = Exact ? (U / 2 + 1) / 2 * 2 : U;
        float2 first_half[2][2] = {};
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const float* p = dk + (u < wrot ? u + U : u);
            if (Exact && u == kHalfU) {
#pragma unroll
                for (int h = 0; h < 2; ++h)
#pragma unroll
                    for (int e = 0; e < 2; ++e) {
                        first_half[h][e] = acc[h][e];
                        acc[h][e] = make_float2(0.f, 0.f);
                    }
            }
            const float2 w0 = u < kReg ? wp[0][u < kReg ? u : 0] : S.w[u < kReg ? 0 : u - kReg][0][tid];
            const float2 w1 = u < kReg ? wp[1][u < kReg ? u : 0] : S.w[u < kReg ? 0 : u - kReg][1][tid];
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const float x = p[h * kDLine];
                acc[h][0] = fma2(w0, make_float2(x, x), acc[h][0]);
                acc[h][1] = fma2(w1, make_float2(x, x), acc[h][1]);
            }
        }
        if (Exact) {
#pragma unroll
            for (int h = 0; h < 2; ++h)
#pragma unroll
                for (int e = 0; e < 2; ++e) acc[h][e] = add2(first_half[h][e], acc[h][e]);
        }
        const float mk[2] = {S.mval[st], S.mval[st + 1]};
        __syncwarp();
        if (lane == 0) {
            mbar_arrive(&S.empty[st]);
            if (two) mbar_arrive(&S.empty[st + 1]);
        }
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            if (h == 1 && !two) break;
            const float2 m2 = make_float2(mk[h], mk[h]);
            const float2 v01 = add2(acc[h][0], m2), v23 = add2(acc[h][1], m2);
            if (Mode == kModeReal) {
                *reinterpret_cast<float4*>(a.out + (out0 + i + h) * kN + 4 * tid) = make_float4(v01.x, v01.y, v23.x, v23.y);
            } else if (Mode == kModeSpec) {
                // spec output undoes the 1/N ifft scaling folded into the window
                float4* o = reinterpret_cast<float4*>(a.out + ((out0 + i + h) * kN + 4 * tid) * 2);
                o[0] = make_float4(v01.x * wa.x * kN, v01.x * wa.y * kN, v01.y * wa.z * kN, v01.y * wa.w * kN);
                o[1] = make_float4(v23.x * wb.x * kN, v23.x * wb.y * kN, v23.y * wb.z * kN, v23.y * wb.w * kN);
            } else {
                // the plain line (its window is one) times the float64 window, one rounding to float32
                const float4 wh = __ldg(reinterpret_cast<const float4*>(a.hann2 + 4 * tid));
                const float4 wl = __ldg(reinterpret_cast<const float4*>(a.hann2 + kN + 4 * tid));
                float2 p01, p23;
                bool ok0, ok1, ok2, ok3;
                const float2 o01 = mul_window2(v01, make_float2(wh.x, wh.y), make_float2(wl.x, wl.y), p01, ok0, ok1);
                const float2 o23 = mul_window2(v23, make_float2(wh.z, wh.w), make_float2(wl.z, wl.w), p23, ok2, ok3);
                // an end point of the window that is exactly zero: x * 0 with x's
                // sign (or NaN), as the float64 product, for every A-scan
                float lh[4] = {end0 ? p01.x : o01.x, o01.y, o23.x, end3 ? p23.y : o23.y};
                ok0 = ok0 || end0;
                ok3 = ok3 || end3;
                if (__any_sync(0xffffffffu, !(ok0 && ok1 && ok2 && ok3))) {
                    const float lx[4] = {v01.x, v01.y, v23.x, v23.y};
                    const bool lsafe[4] = {ok0, ok1, ok2, ok3};
#pragma unroll
                    for (int r = 0; r < 4; ++r)
                        if (!lsafe[r])
                            lh[r] = static_cast<float>(static_cast<double>(lx[r]) * __ldg(a.hann + 4 * tid + r));
                }
                *reinterpret_cast<float4*>(a.out + (out0 + i + h) * kN + 4 * tid) = make_float4(lh[0], lh[1], lh[2], lh[3]);
            }
        }
    }
}

// apodisation mean (cpu_kernels.py:20-25): exact sum, divided in float64,
// stored float32.  Nine lines in flight: a call of few B-scans is one trip to
// memory per batch of lines (25 lines of three B-scans: five in flight 6.7 us,
// nine 5.6, thirteen 5.5 but 2 % slower for 30 B-scans).  Integers: four samples
// a thread.  Float32 raws: one, since their float64 sums are bound by the SM's
// FP64 rate and a row then spans four times the SMs (nine B-scans: 14.5 -> 7.0 us).
// Many lines take 24 in flight (10 B-scans of 400 A-scans and 700 lines to
// magnitudes: 77.5 -> 63.7 us; 2000 float32 lines: 346 -> 319, 700: 118 -> 121).
constexpr int kApodThreads = 128;
constexpr int kApodFlight = 9, kApodFlightMany = 24;
template <typename RawT>
constexpr int kApodMany = sizeof(RawT) == 2 ? 128 : 1024;
template <typename RawT>
constexpr int kApodPer = sizeof(RawT) == 2 ? 4 : 1;                          // samples a thread
template <typename RawT>
constexpr int kApodParts = kN / (kApodThreads * kApodPer<RawT>);             // CTAs a row
// Exact: the sums instead, as -S in float32 while that is exact, else as int32.
template <typename RawT, bool Tiles, bool Exact, int kFlight>
__global__ void __launch_bounds__(kApodThreads) k_apod_mean(const LinesArgs a, float* __restrict__ out) {
    pdl_launch();                                // the lines kernel loads its weights meanwhile
    const int row = blockIdx.x / kApodParts<RawT>;   // segment * B + b, or the tiles' apod_row0 + b
    const int j = (blockIdx.x % kApodParts<RawT> * kApodThreads + threadIdx.x) * kApodPer<RawT>;
    const RawT* p;
    int apod;
    if (Tiles) {
        int lo = 0, hi = a.n_qt - 1;             // last tile with apod_row0 <= row
        while (lo < hi) {
            const int mid = (lo + hi + 1) >> 1;
            if (a.qt[mid].apod_row0 <= row) lo = mid; else hi = mid - 1;
        }
        const QueueTile& t = a.qt[lo];
        apod = t.apod;
        p = static_cast<const RawT*>(t.raw) + static_cast<int64_t>(row - t.apod_row0) * t.interf * kN + j;
    } else {
        const int sg = row / a.B;
        apod = a.apod;
        p = static_cast<const RawT*>(a.seg[sg]) + static_cast<int64_t>(row - sg * a.B) * a.interf * kN + j;
    }
    if constexpr (sizeof(RawT) == 2) {
        int acc[4] = {0, 0, 0, 0};
        for (int k0 = 0; k0 < apod; k0 += kFlight) {
            uint2 q[kFlight];
#pragma unroll
            for (int i = 0; i < kFlight; ++i)
                q[i] = k0 + i < apod ? __ldg(reinterpret_cast<const uint2*>(p + static_cast<int64_t>(k0 + i) * kN))
                                     : make_uint2(0u, 0u);
#pragma unroll
            for (int i = 0; i < kFlight; ++i) {
                acc[0] += static_cast<int>(static_cast<RawT>(q[i].x & 0xffffu));
                acc[1] += static_cast<int>(static_cast<RawT>(q[i].x >> 16));
                acc[2] += static_cast<int>(static_cast<RawT>(q[i].y & 0xffffu));
                acc[3] += static_cast<int>(static_cast<RawT>(q[i].y >> 16));
            }
        }
        float4 o;
        if (Exact)
            o = apod <= kExactFloat ? make_float4(-static_cast<float>(acc[0]), -static_cast<float>(acc[1]),
                                                  -static_cast<float>(acc[2]), -static_cast<float>(acc[3]))
                                    : make_float4(__int_as_float(acc[0]), __int_as_float(acc[1]),
                                                  __int_as_float(acc[2]), __int_as_float(acc[3]));
        else
            o = make_float4(static_cast<float>(static_cast<double>(acc[0]) / apod),
                            static_cast<float>(static_cast<double>(acc[1]) / apod),
                            static_cast<float>(static_cast<double>(acc[2]) / apod),
                            static_cast<float>(static_cast<double>(acc[3]) / apod));
        *reinterpret_cast<float4*>(out + static_cast<int64_t>(row) * kN + j) = o;
    } else {
        double s = 0.0;
        for (int k0 = 0; k0 < apod; k0 += kFlight) {
            float q[kFlight];
#pragma unroll
            for (int i = 0; i < kFlight; ++i)
                q[i] = k0 + i < apod ? __ldg(p + static_cast<int64_t>(k0 + i) * kN) : 0.f;
#pragma unroll
            for (int i = 0; i < kFlight; ++i)
                if (k0 + i < apod) s += static_cast<double>(q[i]);
        }
        out[static_cast<int64_t>(row) * kN + j] = static_cast<float>(s / apod);
    }
}

template <typename RawT, int Mode, int U, bool Tiles, bool Exact>
cudaError_t launch_t(const LinesArgs& a, int num_sms, cudaStream_t st) {
    const size_t smem = sizeof(LinesSmem<RawT, U>);
    const auto kernel = k_lines<RawT, Mode, U, Tiles, Exact>;
    constexpr int kType = sizeof(RawT) == 4 ? 2 : static_cast<RawT>(-1) < 0 ? 1 : 0;
    constexpr int kBit = Exact ? kReadyExact + kType * 4 + (U - 14) / 4
                               : (kType * 4 + (Tiles ? 3 : Mode)) * 4 + (U - 14) / 4;
    static_assert(Exact ? kBit < 64 : kBit < kReadyDisp, "the bits of the kernels overlap");
    const cudaError_t e = kernel_ready(a.ready, kBit, kernel, smem);
    if (e != cudaSuccess) return e;
    const unsigned int n = a.l1 - a.l0;
    const unsigned int grid = n < static_cast<unsigned int>(num_sms) ? n : static_cast<unsigned int>(num_sms);
    return launch_dependent(kernel, dim3(grid), dim3(lines_threads(U)), smem, st, a);
}

// (five warps a scheduler have 96 registers a thread: windows of 18 spill a few weights)
template <typename RawT, int Mode, bool Tiles, bool Exact>
cudaError_t launch_u(const LinesArgs& a, int num_sms, cudaStream_t st) {
    switch (a.g.U) {
        case 14: return launch_t<RawT, Mode, 14, Tiles, Exact>(a, num_sms, st);
        case 18: return launch_t<RawT, Mode, 18, Tiles, Exact>(a, num_sms, st);
        case 22: return launch_t<RawT, Mode, 22, Tiles, Exact>(a, num_sms, st);
        case 26: return launch_t<RawT, Mode, 26, Tiles, Exact>(a, num_sms, st);
        default: return cudaErrorInvalidValue;
    }
}

template <typename RawT>
cudaError_t launch_mode(const LinesArgs& a, int mode, int num_sms, cudaStream_t st) {
    if constexpr (sizeof(RawT) == 2)
        if (a.exact) return launch_u<RawT, kModeReal, false, true>(a, num_sms, st);
    if (a.exact) return cudaErrorInvalidValue;
    if (a.qt != nullptr) return launch_u<RawT, kModeReal, true, false>(a, num_sms, st);
    switch (mode) {
        case kModeSpec: return launch_u<RawT, kModeSpec, false, false>(a, num_sms, st);
        case kModeLinHann: return launch_u<RawT, kModeLinHann, false, false>(a, num_sms, st);
        default: return launch_u<RawT, kModeReal, false, false>(a, num_sms, st);
    }
}

template <typename RawT, int kFlight>
void launch_apod_t(const LinesArgs& a, int rows, float* out, cudaStream_t st) {
    const auto kernel = a.exact           ? k_apod_mean<RawT, false, true, kFlight>
                        : a.qt != nullptr ? k_apod_mean<RawT, true, false, kFlight>
                                          : k_apod_mean<RawT, false, false, kFlight>;
    kernel<<<kApodParts<RawT> * rows, kApodThreads, 0, st>>>(a, out);
}

template <typename RawT>
void launch_apod_f(const LinesArgs& a, int rows, float* out, cudaStream_t st) {
    if (a.qt == nullptr && a.apod >= kApodMany<RawT>)
        launch_apod_t<RawT, kApodFlightMany>(a, rows, out, st);
    else
        launch_apod_t<RawT, kApodFlight>(a, rows, out, st);
}

}  // namespace

cudaError_t launch_apod_mean(const LinesArgs& a, int dtype, int rows, float* out, cudaStream_t st) {
    if (rows == 0) return cudaSuccess;
    if (dtype == 0)
        launch_apod_f<uint16_t>(a, rows, out, st);
    else if (dtype == 1)
        launch_apod_f<int16_t>(a, rows, out, st);
    else
        launch_apod_f<float>(a, rows, out, st);
    return cudaGetLastError();
}

cudaError_t launch_lines(const LinesArgs& a, int dtype, int mode, int num_sms, cudaStream_t st) {
    if (a.l1 == a.l0) return cudaSuccess;
    if (dtype == 0) return launch_mode<uint16_t>(a, mode, num_sms, st);
    if (dtype == 1) return launch_mode<int16_t>(a, mode, num_sms, st);
    return launch_mode<float>(a, mode, num_sms, st);
}

cudaError_t set_wait_test_spectral(unsigned long long limit_ns, int starve, cudaStream_t st) {
    return set_wait_test_here(limit_ns, starve, st);
}

}  // namespace octgb

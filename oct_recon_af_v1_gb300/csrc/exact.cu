// Float64 form of the spectral stage for sm_103a: the reference's
// SpectralProcessor at precision "float64" (octrecon/core/spectral.py:123-165,
// NumPy path), raw integer counts -> |ifft| rounded once to float32.
//
// GB300 executes float64 at two operations per clock per SM, a 64th of its
// float32 rate, so the arithmetic is on pairs of float32 (value = h + l,
// |l| <= ulp(h) / 2, 48 significant bits; the exact sum and product errors of
// Knuth's two-sum and of a fused multiply-add, Dekker 1971 / Ogita, Rump and
// Oishi 2005): an error of ~1e-13 of the line's scale, five decades below the
// one rounding of the result.  Re and im of a complex pair go through the packed
// f32x2 instructions together.
//
// Per A-scan (group of 128 threads, four A-scans per CTA):
//   background: with S_j the integer sum of the apodisation lines and A their
//     count, interf_j = raw_j - S_j / A = n_j / A for the integer n_j = A raw_j
//     - S_j; the line mean is sum(n) / (2048 A), summed in integers, and the
//     background-free sample d_j = N_j / (2048 A) with N_j = 2048 n_j - sum(n);
//   sinc: lin_i = (sum_t w[t,i] N[start_i + t] + sum(n)) / (2048 A), a
//     compensated dot product over the float64 band weights (split hi + lo) in
//     the reference's tap order (core/spectral.py:128-134);
//   window (Hann/rms x dispersion phase, 1/N folded in);
//   inverse FFT, Stockham radix 16, 16, 8 (last stage pruned to k < N/2), |X|
//     with its square root corrected by the low part, rounded to float32.
// Thread lt computes the sinc outputs its first FFT stage takes (samples
// lt + 128 r), so the line goes from the sinc to the FFT in registers; the
// band weights (tap-major, coalesced) are read through L1 for every A-scan.
// 3000 A-scans in 163 us (18 M/s), where float64 operations, at 86 % of their
// pipe, took 634; every output of 25 M voxels and of the timed case has the same
// bits.  Bound by the FP32 pipes and latency: 16 warps an SM at 128 registers.
#include <cuda_runtime.h>
#include <stdint.h>

#include "octgb_device.cuh"
#include "octgb_internal.h"

namespace octgb {
namespace {

constexpr int kXGroup = 128;                    // threads per A-scan
constexpr int kXPerCta = 4;                     // A-scans per CTA
constexpr int kXThreads = kXGroup * kXPerCta;
constexpr int kXStride = kN + (kN >> 4);        // padded complex line (one slot per 16)
constexpr int kXTail = 32;                      // zero tail of the integer line (padded taps)

__device__ __forceinline__ int xpad(int e) { return e + (e >> 4); }

__device__ __forceinline__ float2 mul2(float2 a, float2 b) {
    float2 r;
    asm("{\n\t.reg .b64 x, y, z;\n\tmov.b64 x, {%2, %3};\n\tmov.b64 y, {%4, %5};\n\t"
        "mul.rn.f32x2 z, x, y;\n\tmov.b64 {%0, %1}, z;\n\t}"
        : "=f"(r.x), "=f"(r.y)
        : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
    return r;
}
__device__ __forceinline__ float2 neg2(float2 a) { return make_float2(-a.x, -a.y); }
__device__ __forceinline__ float2 dup(float a) { return make_float2(a, a); }

// two values (re and im, or two outputs), each h + l
struct Pair {
    float2 h, l;
};
__device__ __forceinline__ Pair renorm(float2 s, float2 e) {
    Pair r;
    r.h = add2(s, e);
    r.l = sub2(e, sub2(r.h, s));
    return r;
}
// s = a + b rounded, and its exact error
__device__ __forceinline__ float2 two_sum(float2 a, float2 b, float2& err) {
    const float2 s = add2(a, b), bb = sub2(s, a);
    err = add2(sub2(a, sub2(s, bb)), sub2(b, bb));
    return s;
}
__device__ __forceinline__ Pair padd(Pair a, Pair b) {
    float2 e;
    const float2 s = two_sum(a.h, b.h, e);
    return renorm(s, add2(e, add2(a.l, b.l)));
}
__device__ __forceinline__ Pair psub(Pair a, Pair b) {
    const float2 s = sub2(a.h, b.h), bb = sub2(s, a.h);
    const float2 e = sub2(sub2(a.h, sub2(s, bb)), add2(b.h, bb));
    return renorm(s, add2(e, sub2(a.l, b.l)));
}
// a b to first order in the low parts: product p and the rest
__device__ __forceinline__ float2 two_prod(float2 ah, float2 al, float2 bh, float2 bl, float2& e) {
    const float2 p = mul2(ah, bh);
    e = fma2(ah, bh, neg2(p));
    e = fma2(ah, bl, e);
    e = fma2(al, bh, e);
    return p;
}
// lanewise product
__device__ __forceinline__ Pair pmul(Pair a, Pair b) {
    float2 e;
    const float2 p = two_prod(a.h, a.l, b.h, b.l, e);
    return renorm(p, e);
}
// complex product a w
__device__ __forceinline__ Pair cmulp(Pair a, Pair w) {
    float2 e1, e2, e;
    const float2 p1 = two_prod(dup(a.h.x), dup(a.l.x), w.h, w.l, e1);
    const float2 p2 = two_prod(dup(a.h.y), dup(a.l.y), make_float2(-w.h.y, w.h.x), make_float2(-w.l.y, w.l.x), e2);
    const float2 s = two_sum(p1, p2, e);
    return renorm(s, add2(e, add2(e1, e2)));
}
__device__ __forceinline__ Pair cmuli(Pair a) {
    return Pair{make_float2(-a.h.y, a.h.x), make_float2(-a.l.y, a.l.x)};
}
__device__ __forceinline__ Pair from4(float4 v) { return Pair{make_float2(v.x, v.y), make_float2(v.z, v.w)}; }
__device__ __forceinline__ float4 to4(Pair p) { return make_float4(p.h.x, p.h.y, p.l.x, p.l.y); }

// a float64 constant (re, im) as a pair
__device__ __forceinline__ Pair cpair(double re, double im) {
    const float hr = static_cast<float>(re), hi = static_cast<float>(im);
    return Pair{make_float2(hr, hi), make_float2(static_cast<float>(re - hr), static_cast<float>(im - hi))};
}

__device__ __forceinline__ void pdft4(Pair& x0, Pair& x1, Pair& x2, Pair& x3) {
    const Pair a = padd(x0, x2), b = psub(x0, x2), c = padd(x1, x3), d = cmuli(psub(x1, x3));
    x0 = padd(a, c);
    x2 = psub(a, c);
    x1 = padd(b, d);
    x3 = psub(b, d);
}

constexpr double kDC1 = 0.92387953251128675613;   // cos(pi/8)
constexpr double kDS1 = 0.38268343236508977173;   // sin(pi/8)
constexpr double kDC2 = 0.70710678118654752440;   // cos(pi/4)

// inverse DFT-16 as 4 x 4 (the float32 kernel's decomposition)
__device__ __forceinline__ void pdft16(Pair (&v)[16]) {
#pragma unroll
    for (int n1 = 0; n1 < 4; ++n1) pdft4(v[n1], v[n1 + 4], v[n1 + 8], v[n1 + 12]);
    v[1 + 4] = cmulp(v[1 + 4], cpair(kDC1, kDS1));
    v[1 + 8] = cmulp(v[1 + 8], cpair(kDC2, kDC2));
    v[1 + 12] = cmulp(v[1 + 12], cpair(kDS1, kDC1));
    v[2 + 4] = cmulp(v[2 + 4], cpair(kDC2, kDC2));
    v[2 + 8] = cmuli(v[2 + 8]);
    v[2 + 12] = cmulp(v[2 + 12], cpair(-kDC2, kDC2));
    v[3 + 4] = cmulp(v[3 + 4], cpair(kDS1, kDC1));
    v[3 + 8] = cmulp(v[3 + 8], cpair(-kDC2, kDC2));
    v[3 + 12] = cmulp(v[3 + 12], cpair(-kDC1, -kDS1));
#pragma unroll
    for (int k2 = 0; k2 < 4; ++k2) pdft4(v[4 * k2], v[4 * k2 + 1], v[4 * k2 + 2], v[4 * k2 + 3]);
    // X[4 k1 + k2] sits in v[k1 + 4 k2]
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = i + 1; j < 4; ++j) {
            const Pair t = v[i + 4 * j];
            v[i + 4 * j] = v[j + 4 * i];
            v[j + 4 * i] = t;
        }
}

__device__ __forceinline__ void pdft8_low(Pair (&v)[8], Pair (&X)[4]) {
    pdft4(v[0], v[2], v[4], v[6]);
    pdft4(v[1], v[3], v[5], v[7]);
    X[0] = padd(v[0], v[1]);
    X[1] = padd(v[2], cmulp(v[3], cpair(kDC2, kDC2)));
    X[2] = padd(v[4], cmuli(v[5]));
    X[3] = padd(v[6], cmulp(v[7], cpair(-kDC2, kDC2)));
}

// |X| of a pair, rounded to float32: the root of the high part of the squares'
// sum, corrected by its residual.  Values whose squares would leave float32's
// range are scaled by a power of two first.
__device__ __forceinline__ float pabs(Pair X) {
    const float big = fmaxf(fabsf(X.h.x), fabsf(X.h.y));
    const float up = big < 1e-12f ? 0x1p60f : big > 1e15f ? 0x1p-60f : 1.f;
    const float down = big < 1e-12f ? 0x1p-60f : big > 1e15f ? 0x1p60f : 1.f;
    const float2 h = mul2(X.h, dup(up)), l = mul2(X.l, dup(up));
    float2 e;
    const float2 p = two_prod(h, l, h, l, e);
    const float s = p.x + p.y, bb = s - p.x;
    const float err = ((p.x - (s - bb)) + (p.y - bb)) + (e.x + e.y);
    const float r = __fsqrt_rn(s);
    const float res = fmaf(-r, r, s) + err;
    return (r > 0.f ? fmaf(res, __fdividef(0.5f, r), r) : r) * down;
}

__device__ __forceinline__ void xgroup_sync(int g) {
    asm volatile("bar.sync %0, %1;" ::"r"(1 + g), "r"(kXGroup) : "memory");
}

// integer sums of the apodisation lines, (B, N)
template <typename RawT>
__global__ void k_exact_apod_sum(const RawT* __restrict__ raw, int interf, int apod, int* __restrict__ sums) {
    const int b = blockIdx.y;
    const int j = blockIdx.x * blockDim.x + threadIdx.x;
    if (j >= kN) return;
    const RawT* p = raw + static_cast<int64_t>(b) * interf * kN + j;
    int s = 0;
#pragma unroll 5
    for (int k = 0; k < apod; ++k) s += static_cast<int>(p[static_cast<int64_t>(k) * kN]);
    sums[static_cast<int64_t>(b) * kN + j] = s;
}

// an integer below 2^48 as h + l
__device__ __forceinline__ float2 split_int(long long n) {
    const float h = static_cast<float>(n);
    return make_float2(h, static_cast<float>(n - static_cast<long long>(h)));
}

struct ExactSmem {
    alignas(16) float4 line[kXPerCta][kXStride];         // N_j (float2 each) with its zero tail, then the FFT line
    alignas(16) float4 tw[kTwTable];                     // tw2[16 r + j], then tw3[256 (r - 1) + j]
    long long red[kXPerCta][4];
};
static_assert((kN + kXTail) * sizeof(float2) <= kXStride * sizeof(float4), "the integer line fits the FFT line");

template <typename RawT>
__global__ void __launch_bounds__(kXThreads, 1) k_exact(const ExactArgs a) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    ExactSmem& S = *reinterpret_cast<ExactSmem*>(smem_raw);
    const int tid = threadIdx.x, g = tid / kXGroup, lt = tid % kXGroup;
    const int warp = tid >> 5, lane = tid & 31;
    for (int k = tid; k < kTwTable; k += kXThreads) S.tw[k] = __ldg(a.tw + k);
    __syncthreads();

    float4* X = S.line[g];
    float2* D = reinterpret_cast<float2*>(X);
    for (int64_t as = static_cast<int64_t>(blockIdx.x) * kXPerCta + g; as < a.n_ascans;
         as += static_cast<int64_t>(gridDim.x) * kXPerCta) {
        const int64_t b = as / a.nx, x = as - b * a.nx;
        const RawT* row = static_cast<const RawT*>(a.raw) + ((b * a.interf + a.apod + x) * kN);
        const int* Sb = a.apod_sum + b * kN;
        // ---- background: integer n_j and their sum
        int nj[16];
        long long sum = 0;
#pragma unroll
        for (int r = 0; r < 16; ++r) {
            const int j = lt + 128 * r;
            nj[r] = a.apod * static_cast<int>(row[j]) - __ldg(Sb + j);
            sum += nj[r];
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
        if (lane == 0) S.red[g][warp & 3] = sum;
        xgroup_sync(g);                                  // (and the previous A-scan's line has been read)
        const long long sn = (S.red[g][0] + S.red[g][1]) + (S.red[g][2] + S.red[g][3]);
#pragma unroll
        for (int r = 0; r < 16; ++r) D[lt + 128 * r] = split_int(2048LL * nj[r] - sn);
        if (lt < kXTail) D[kN + lt] = make_float2(0.f, 0.f);
        xgroup_sync(g);
        // ---- sinc + window: the outputs lt + 128 r (this thread's first FFT
        // stage), two at a time
        Pair v[16];
        const float2 sf = split_int(sn);
        const Pair snp{dup(sf.x), dup(sf.y)}, inv{dup(a.inv_h), dup(a.inv_l)};
#pragma unroll
        for (int r = 0; r < 16; r += 2) {
            const int i0 = lt + 128 * r, i1 = i0 + 128;
            const float2* d0 = D + __ldg(a.start + i0);
            const float2* d1 = D + __ldg(a.start + i1);
            const float2* w0 = a.w + i0;
            float2 s = dup(0.f), c = dup(0.f);
            for (int t = 0; t < a.taps; ++t, w0 += kN) {
                const float2 wa = __ldg(w0), wb = __ldg(w0 + 128), da = d0[t], db = d1[t];
                float2 e, err;
                const float2 p = two_prod(make_float2(wa.x, wb.x), make_float2(wa.y, wb.y), make_float2(da.x, db.x),
                                          make_float2(da.y, db.y), e);
                s = two_sum(s, p, err);
                c = add2(c, add2(err, e));
            }
            const Pair lin = pmul(padd(renorm(s, c), snp), inv);
            v[r] = pmul(Pair{dup(lin.h.x), dup(lin.l.x)}, from4(__ldg(a.win + i0)));
            v[r + 1] = pmul(Pair{dup(lin.h.y), dup(lin.l.y)}, from4(__ldg(a.win + i1)));
        }
        // ---- inverse FFT in place
        pdft16(v);
        xgroup_sync(g);                                  // N_j has been read
#pragma unroll
        for (int r = 0; r < 16; ++r) X[xpad(16 * lt + r)] = to4(v[r]);
        xgroup_sync(g);
        {
            const int jm = lt & 15;
#pragma unroll
            for (int r = 0; r < 16; ++r) v[r] = from4(X[xpad(lt + 128 * r)]);
#pragma unroll
            for (int r = 1; r < 16; ++r) v[r] = cmulp(v[r], from4(S.tw[r * 16 + jm]));
            pdft16(v);
            const int idxD = (lt >> 4) * 256 + jm;
            xgroup_sync(g);
#pragma unroll
            for (int r = 0; r < 16; ++r) X[xpad(idxD + 16 * r)] = to4(v[r]);
        }
        xgroup_sync(g);
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int j = lt + 128 * h;
            Pair w8[8];
#pragma unroll
            for (int r = 0; r < 8; ++r) w8[r] = from4(X[xpad(j + 256 * r)]);
#pragma unroll
            for (int r = 1; r < 8; ++r) w8[r] = cmulp(w8[r], from4(S.tw[256 + (r - 1) * 256 + j]));
            Pair Xk[4];
            pdft8_low(w8, Xk);
#pragma unroll
            for (int r = 0; r < 4; ++r) a.mag[as * kHalf + j + 256 * r] = pabs(Xk[r]);
        }
    }
}

template <typename RawT>
cudaError_t launch_exact_t(const ExactArgs& a, int* sums, int num_sms, cudaStream_t st) {
    const dim3 sgrid(kN / 256, a.B);
    k_exact_apod_sum<RawT><<<sgrid, 256, 0, st>>>(static_cast<const RawT*>(a.raw), a.interf, a.apod, sums);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    e = cudaFuncSetAttribute(k_exact<RawT>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             static_cast<int>(sizeof(ExactSmem)));
    if (e != cudaSuccess) return e;
    const int64_t quads = (a.n_ascans + kXPerCta - 1) / kXPerCta;
    const int grid = static_cast<int>(quads < num_sms ? quads : num_sms);
    ExactArgs b = a;
    b.apod_sum = sums;
    const double inv = 1.0 / (2048.0 * a.apod);          // one rounding, as the mean's division
    b.inv_h = static_cast<float>(inv);
    b.inv_l = static_cast<float>(inv - b.inv_h);
    k_exact<RawT><<<grid, kXThreads, sizeof(ExactSmem), st>>>(b);
    return cudaGetLastError();
}

}  // namespace

cudaError_t launch_exact(const ExactArgs& a, int dtype, int* sums, int num_sms, cudaStream_t st) {
    if (dtype == 0) return launch_exact_t<uint16_t>(a, sums, num_sms, st);
    if (dtype == 1) return launch_exact_t<int16_t>(a, sums, num_sms, st);
    return cudaErrorInvalidValue;
}

}  // namespace octgb

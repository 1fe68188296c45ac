// Device helpers shared by the spectral and estimation kernels: complex
// arithmetic, the inverse DFT blocks of the 2048-point shared-memory FFT,
// bulk-copy/mbarrier primitives with a bounded wait, and the FFT itself.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include "octgb_internal.h"

namespace octgb {
namespace {

// Packed float32 pairs (sm_100 family f32x2 instructions): one instruction
// for both lanes, each lane rounded to nearest exactly as the scalar operation,
// so results are bit-identical to two scalar ops.  The explicit rounding mode
// also keeps ptxas from contracting them (as it would not contract the
// scalar forms here either).
__device__ __forceinline__ float2 add2(float2 a, float2 b) {
    float2 r;
    asm("{\n\t.reg .b64 x, y, z;\n\tmov.b64 x, {%2, %3};\n\tmov.b64 y, {%4, %5};\n\t"
        "add.rn.f32x2 z, x, y;\n\tmov.b64 {%0, %1}, z;\n\t}"
        : "=f"(r.x), "=f"(r.y)
        : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
    return r;
}
__device__ __forceinline__ float2 sub2(float2 a, float2 b) {
    float2 r;
    asm("{\n\t.reg .b64 x, y, z;\n\tmov.b64 x, {%2, %3};\n\tmov.b64 y, {%4, %5};\n\t"
        "sub.rn.f32x2 z, x, y;\n\tmov.b64 {%0, %1}, z;\n\t}"
        : "=f"(r.x), "=f"(r.y)
        : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
    return r;
}
// (a.x b.x + c.x, a.y b.y + c.y), each a single-rounding fma
__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) {
    float2 r;
    asm("{\n\t.reg .b64 x, y, z, w;\n\tmov.b64 x, {%2, %3};\n\tmov.b64 y, {%4, %5};\n\t"
        "mov.b64 z, {%6, %7};\n\tfma.rn.f32x2 w, x, y, z;\n\tmov.b64 {%0, %1}, w;\n\t}"
        : "=f"(r.x), "=f"(r.y)
        : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y), "f"(c.x), "f"(c.y));
    return r;
}

__device__ __forceinline__ float2 cadd(float2 a, float2 b) { return add2(a, b); }
__device__ __forceinline__ float2 csub(float2 a, float2 b) { return sub2(a, b); }
__device__ __forceinline__ float2 cmul(float2 a, float2 b) {
    return make_float2(fmaf(a.x, b.x, -a.y * b.y), fmaf(a.x, b.y, a.y * b.x));
}
__device__ __forceinline__ float2 muli(float2 a) { return make_float2(-a.y, a.x); }

// inverse DFT-4 (omega = +i), natural order in and out; b +- i e lane-crossed
// in scalar form (a packed form would need the swapped pair of e first)
__device__ __forceinline__ void dft4(float2& x0, float2& x1, float2& x2, float2& x3) {
    const float2 a = cadd(x0, x2), b = csub(x0, x2), c = cadd(x1, x3), e = csub(x1, x3);
    x0 = cadd(a, c);
    x2 = csub(a, c);
    x1 = make_float2(b.x - e.y, b.y + e.x);
    x3 = make_float2(b.x + e.y, b.y - e.x);
}

// cos/sin of multiples of pi/8 (float64 literals rounded to float32)
constexpr float kC1 = 0.92387953251128675613f;   // cos(pi/8)
constexpr float kS1 = 0.38268343236508977173f;   // sin(pi/8)
constexpr float kC2 = 0.70710678118654752440f;   // cos(pi/4)

// inverse DFT-16 as 4 x 4: X[4*k1 + k2] = sum_n1 w4^(n1 k1) w16^(n1 k2) sum_n2 x[n1 + 4 n2] w4^(n2 k2)
__device__ __forceinline__ void dft16(float2 (&v)[16]) {
#pragma unroll
    for (int n1 = 0; n1 < 4; ++n1) dft4(v[n1], v[n1 + 4], v[n1 + 8], v[n1 + 12]);
    // twiddles w16^(n1*k2) on element v[n1 + 4*k2]
    v[1 + 4] = cmul(v[1 + 4], make_float2(kC1, kS1));     // n1=1,k2=1: w^1
    v[1 + 8] = cmul(v[1 + 8], make_float2(kC2, kC2));     // n1=1,k2=2: w^2
    v[1 + 12] = cmul(v[1 + 12], make_float2(kS1, kC1));   // n1=1,k2=3: w^3
    v[2 + 4] = cmul(v[2 + 4], make_float2(kC2, kC2));     // n1=2,k2=1: w^2
    v[2 + 8] = muli(v[2 + 8]);                            // n1=2,k2=2: w^4 = i
    v[2 + 12] = cmul(v[2 + 12], make_float2(-kC2, kC2));  // n1=2,k2=3: w^6
    v[3 + 4] = cmul(v[3 + 4], make_float2(kS1, kC1));     // n1=3,k2=1: w^3
    v[3 + 8] = cmul(v[3 + 8], make_float2(-kC2, kC2));    // n1=3,k2=2: w^6
    v[3 + 12] = cmul(v[3 + 12], make_float2(-kC1, -kS1)); // n1=3,k2=3: w^9
#pragma unroll
    for (int k2 = 0; k2 < 4; ++k2) dft4(v[4 * k2], v[4 * k2 + 1], v[4 * k2 + 2], v[4 * k2 + 3]);
    // X[4*k1 + k2] sits in v[k1 + 4*k2]: transpose the 4x4 block
    float2 t;
    t = v[1]; v[1] = v[4]; v[4] = t;
    t = v[2]; v[2] = v[8]; v[8] = t;
    t = v[3]; v[3] = v[12]; v[12] = t;
    t = v[6]; v[6] = v[9]; v[9] = t;
    t = v[7]; v[7] = v[13]; v[13] = t;
    t = v[11]; v[11] = v[14]; v[14] = t;
}

// inverse DFT-8 as 2 x 4, returning only X[0..3] (the last stage keeps k < N/2)
__device__ __forceinline__ void dft8_low(float2 (&v)[8], float2 (&X)[4]) {
    dft4(v[0], v[2], v[4], v[6]);
    dft4(v[1], v[3], v[5], v[7]);
    const float2 y1 = cmul(v[3], make_float2(kC2, kC2));
    const float2 y2 = muli(v[5]);
    const float2 y3 = cmul(v[7], make_float2(-kC2, kC2));
    X[0] = cadd(v[0], v[1]);
    X[1] = cadd(v[2], y1);
    X[2] = cadd(v[4], y2);
    X[3] = cadd(v[6], y3);
}

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
    return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

// bytes from p to the next multiple of `to` (added to a shared pointer it stays
// one: through an integer cast the compiler would use generic accesses)
__device__ __forceinline__ uint32_t align_up_smem(const void* p, uint32_t to) {
    return (to - (smem_u32(p) & (to - 1u))) & (to - 1u);
}

__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}

__device__ __forceinline__ void mbar_expect_tx(uint64_t* bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes)
                 : "memory");
}

__device__ __forceinline__ void tma_bulk_g2s(void* dst, const void* src, uint32_t bytes, uint64_t* bar) {
    asm volatile(
        "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
            smem_u32(dst)),
        "l"(src), "r"(bytes), "r"(smem_u32(bar))
        : "memory");
}

// copy `bytes` (a multiple of 16) from a 16-byte aligned global address into L2
__device__ __forceinline__ void bulk_prefetch_l2(const void* src, uint32_t bytes) {
    asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(src), "r"(bytes) : "memory");
}

__device__ __forceinline__ bool mbar_test(uint64_t* bar, uint32_t parity) {
    uint32_t done;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(done)
        : "r"(smem_u32(bar)), "r"(parity)
        : "memory");
    return done != 0;
}

__device__ __forceinline__ uint64_t globaltimer_ns() {
    uint64_t t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

// try_wait suspends the thread in hardware until the phase completes or the
// hint (ns) runs out, so waiting warps issue (almost) no instructions
__device__ __forceinline__ bool mbar_try(uint64_t* bar, uint32_t parity) {
    uint32_t done;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(done)
        : "r"(smem_u32(bar)), "r"(parity), "r"(100000u)
        : "memory");
    return done != 0;
}

// Limit of the bounded waits (ns of wall time, 2 s) and the self-test switch
// that makes each CTA's first bulk-copy barrier expect 16 bytes more than its
// copies deliver, so that wait runs out while every copy still lands.  One
// copy per translation unit, written only by its set_wait_test_* function
// (octgb_selftest_wait_expiry); the product never changes them.
__device__ unsigned long long g_wait_limit_ns = 2000000000ull;
__device__ int g_starve_first_copy = 0;

// Programmatic dependent launch: a kernel started by launch_dependent() may
// begin while the one before it in the stream drains; pdl_wait() returns when
// that one has completed and its writes are visible, so a kernel calls it
// before it touches anything an earlier one wrote or reads.  pdl_launch() lets
// the next such kernel's blocks take the places of blocks that exit.
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void pdl_launch() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

template <typename... Params, typename... Args>
inline cudaError_t launch_dependent(void (*kernel)(Params...), dim3 grid, dim3 block, size_t smem, cudaStream_t st,
                                    Args&&... args) {
    cudaLaunchAttribute at{};
    at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cfg.attrs = &at;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kernel, args...);
}

// bytes a CTA's first bulk-copy barrier expects beyond its copies (0 outside the self-test)
__device__ __forceinline__ uint32_t starved_bytes(bool first) { return first && g_starve_first_copy ? 16u : 0u; }

// Bounded wait on an mbarrier phase: gives up after g_wait_limit_ns of wall
// time and reports it through the status word (the copies and MMAs waited
// for normally complete within microseconds).  The first try (it suspends the
// thread for up to 100 us) comes before the timer and the limit are read: those
// reads cost more than most waits.
__device__ __forceinline__ bool mbar_wait_bounded(uint64_t* bar, uint32_t parity, int* status) {
    if (mbar_test(bar, parity)) return true;
    if (mbar_try(bar, parity)) return true;
    const uint64_t t0 = globaltimer_ns();
    const uint64_t limit = g_wait_limit_ns;
    for (uint32_t it = 0; it < (1u << 30); ++it) {
        if (mbar_try(bar, parity)) return true;
        if (globaltimer_ns() - t0 > limit) break;
    }
    atomicExch(status, kStatusTimeout);
    return false;
}

// host side: set this translation unit's wait limit and self-test switch
inline cudaError_t set_wait_test_here(unsigned long long limit_ns, int starve, cudaStream_t st) {
    cudaError_t e = cudaMemcpyToSymbolAsync(g_wait_limit_ns, &limit_ns, sizeof(limit_ns), 0,
                                            cudaMemcpyHostToDevice, st);
    if (e != cudaSuccess) return e;
    e = cudaMemcpyToSymbolAsync(g_starve_first_copy, &starve, sizeof(starve), 0, cudaMemcpyHostToDevice, st);
    if (e != cudaSuccess) return e;
    return cudaStreamSynchronize(st);
}

// ---- tcgen05 (5th-generation tensor cores) helpers
// shared-memory matrix descriptor without swizzle: lbo = byte step between
// core matrices (8 rows x 16 bytes) along K, sbo = along M/N; without swizzle
// this holds for K-major operands (a core matrix row = 8 K values) and
// MN-major ones (a row = 8 M/N values) alike.  Bit 46 is the descriptor
// version of sm_100-family tensor cores.
__device__ __forceinline__ uint64_t smem_desc(const void* p, uint32_t lbo, uint32_t sbo) {
    const uint64_t a = smem_u32(p);
    return ((a >> 4) & 0x3fffull) | (static_cast<uint64_t>((lbo >> 4) & 0x3fff) << 16) |
           (static_cast<uint64_t>((sbo >> 4) & 0x3fff) << 32) | (1ull << 46);
}

// kind::f16 instruction descriptor: f16 x f16 -> f32 accumulate, K-major A and
// B, shape M x N (M = 64 or 128, N a multiple of 16 up to 256 for M = 128)
__host__ __device__ constexpr uint32_t mma_idesc_f16(int m, int n) {
    return (1u << 4) | (static_cast<uint32_t>(n >> 3) << 17) | (static_cast<uint32_t>(m >> 4) << 24);
}

__device__ __forceinline__ void mma_f16_id(uint32_t d_tmem, uint64_t a, uint64_t b, uint32_t idesc,
                                           uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(d_tmem),
        "l"(a), "l"(b), "r"(idesc), "r"(accumulate)
        : "memory");
}

// arrive on the mbarrier when every tcgen05 operation issued so far by this thread has completed
__device__ __forceinline__ void mma_commit(uint64_t* bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar))
                 : "memory");
}

// The same two issued by a converged warp (one elected lane, always the same):
// control flow and operands stay uniform, so the compiler keeps the descriptors
// in uniform registers.  Issued from a one-thread branch, every MMA first moves
// its operands there: measured 160-235 cycles an MMA, more than a 128 x 32 x 16
// one takes.
__device__ __forceinline__ void mma_f16_warp(uint32_t d_tmem, uint64_t a, uint64_t b, uint32_t idesc,
                                             uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p, q;\n\telect.sync _|q, 0xffffffff;\n\tsetp.ne.b32 p, %4, 0;\n\t"
        "@q tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(d_tmem),
        "l"(a), "l"(b), "r"(idesc), "r"(accumulate)
        : "memory");
}
__device__ __forceinline__ void mma_commit_warp(uint64_t* bar) {
    asm volatile(
        "{\n\t.reg .pred q;\n\telect.sync _|q, 0xffffffff;\n\t"
        "@q tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n\t}" ::"r"(smem_u32(bar))
        : "memory");
}

__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}

__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

// 32 consecutive TMEM columns of this warp's 32 lanes (one lane per thread)
__device__ __forceinline__ void tmem_ld32(uint32_t taddr, float (&v)[32]) {
    uint32_t r[32];
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, "
        "%15, %16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
          "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]),
          "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]),
          "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
        : "r"(taddr));
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int i = 0; i < 32; ++i) v[i] = __uint_as_float(r[i]);
}

// Inverse FFT of one 2048-point line by one warp, 64 points a lane, with one
// exchange through the warp's own shared memory and no block barrier.  The
// arithmetic is that of the radix 16, 16, 8 transform above, operation for
// operation (the same bits); only the grouping differs.  With n = a + 8 b +
// 128 n1 (a < 8, b = b1 + 4 b2 < 16, n1 < 16) lane a + 8 b1 holds every n1 and
// b2: the first radix-16 stage (over n1) and the first radix-4 layer of the
// second (over b2) need no exchange.  The result c = k0 + 16 k2 (< 64) then
// moves to lane c mod 32, which holds every a and b1: the second radix-4
// layer (over b1) and the radix-8 stage (over a) need none either.  The
// exchange runs in two halves (c < 32, c >= 32) through 32 x 33 complex
// values, the odd pitch keeping both sides free of bank conflicts, so the
// second half waits in registers while the first is read.
// v[r] = x[lane + 32 r] on entry; emit(k, |X[k]|) for the lane's 32 bins
// k < N/2.
// tw2[16 j + r] = w^(r j N/256), tw3[256 (r - 1) + j] = w^(r j) for r >= 1.
constexpr int kWarpPitch = 33;
constexpr int kWarpExchange = 32 * kWarpPitch;            // float2 of a warp's exchange buffer

template <typename Emit>
__device__ __forceinline__ void ifft2048_low_mag_warp(float2 (&v)[64], float2* ex, const float2* tw2,
                                                      const float2* tw3, int lane, Emit&& emit) {
    const int b1 = lane >> 3;
    // v[b2 + 4 n1] -> v[b2 + 4 k0]
#pragma unroll
    for (int b2 = 0; b2 < 4; ++b2) {
        float2 t[16];
#pragma unroll
        for (int i = 0; i < 16; ++i) t[i] = v[b2 + 4 * i];
        dft16(t);
        const float2* tw = tw2 + b1 + 4 * b2;             // four addresses a warp, in four banks
        v[b2] = t[0];
#pragma unroll
        for (int i = 1; i < 16; ++i) v[b2 + 4 * i] = cmul(t[i], tw[16 * i]);
    }
    // the inner twiddles w16^(b1 k2) of the second radix-16 stage, k2 = 1..3,
    // as dft16 has them (b1 = 0 and the exact i give the same values)
    const float2 wi1 = b1 == 0 ? make_float2(1.f, 0.f) : b1 == 1 ? make_float2(kC1, kS1)
                     : b1 == 2 ? make_float2(kC2, kC2) : make_float2(kS1, kC1);
    const float2 wi2 = b1 == 0 ? make_float2(1.f, 0.f) : b1 == 1 ? make_float2(kC2, kC2)
                     : b1 == 2 ? make_float2(0.f, 1.f) : make_float2(-kC2, kC2);
    const float2 wi3 = b1 == 0 ? make_float2(1.f, 0.f) : b1 == 1 ? make_float2(kS1, kC1)
                     : b1 == 2 ? make_float2(-kC2, kC2) : make_float2(-kC1, -kS1);
#pragma unroll
    for (int k0 = 0; k0 < 16; ++k0) {
        float2 (&q)[64] = v;
        dft4(q[4 * k0], q[4 * k0 + 1], q[4 * k0 + 2], q[4 * k0 + 3]);
        q[4 * k0 + 1] = cmul(q[4 * k0 + 1], wi1);
        q[4 * k0 + 2] = cmul(q[4 * k0 + 2], wi2);
        q[4 * k0 + 3] = cmul(q[4 * k0 + 3], wi3);
    }
    __syncwarp();                                         // the buffer's last readers are done
#pragma unroll
    for (int c = 0; c < 32; ++c) ex[c * kWarpPitch + lane] = v[4 * (c & 15) + (c >> 4)];
    __syncwarp();
    float2 u[32];                                         // u[a + 8 b1] of c = lane (then c = lane + 32)
#pragma unroll
    for (int i = 0; i < 32; ++i) u[i] = ex[lane * kWarpPitch + i];
    __syncwarp();
#pragma unroll
    for (int c = 0; c < 32; ++c) ex[c * kWarpPitch + lane] = v[4 * (c & 15) + (c >> 4) + 2];
    __syncwarp();
    // one copy of the code for both halves: the whole kernel stays near 32 KB
    // of instructions, which the warps at different points of it share
#pragma unroll 1
    for (int c = lane;; c += 32) {
#pragma unroll
        for (int a = 0; a < 8; ++a) dft4(u[a], u[a + 8], u[a + 16], u[a + 24]);
#pragma unroll
        for (int k1 = 0; k1 < 4; ++k1) {
            const int K = c + 64 * k1;
            float2 w[8];
            w[0] = u[8 * k1];
#pragma unroll
            for (int a = 1; a < 8; ++a) w[a] = cmul(u[8 * k1 + a], tw3[256 * (a - 1) + K]);
            float2 X[4];
            dft8_low(w, X);
#pragma unroll
            for (int p = 0; p < 4; ++p) emit(K + 256 * p, __fsqrt_rn(fmaf(X[p].x, X[p].x, X[p].y * X[p].y)));
        }
        if (c >= 32) break;
#pragma unroll
        for (int i = 0; i < 32; ++i) u[i] = ex[lane * kWarpPitch + i];
    }
}

}  // namespace
}  // namespace octgb

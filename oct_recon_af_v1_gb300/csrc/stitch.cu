// Focus-weighted tile stitching, row finalisation and the legacy uint16
// quantisation.
//
// Stitching (octrecon/core/stitching.py:122-139, pipeline.py:283-284): for
// one tile and one batch of B-scans,
//   a[f,x,r]  = mag[f, x, clip(r0 + r + shift)]   (optical-path gather)
//   F[f,x,r]  = valid * fz[r]
//   num[f, zo, c0+c] += sum_x WxT[x,c] sum_r Wz[zo,r] a F
//   den[f, zo, c0+c] += sum_x WxT[x,c] sum_r Wz[zo,r] F
// Wz / WxT are linear-interpolation operators with at most two adjacent
// non-zeros per output row / column, stored compactly.
//
// The work unit (k_stitch) is a block of 32 to 128 rows zo x 32 columns c of
// one frame.  The block reads a small patch of each tile's magnitudes (the
// A-scans feeding its columns x the depth rows feeding its rows) into shared
// memory with reads along depth (the magnitude layout) and writes along x (the
// output layout): a transpose through shared memory, so both global sides are
// coalesced.  For a frame batch every tile is summed in tile order with
// num/den in registers, then finalised (threshold -> NaN, 20 log10) with the
// plane / running clim: num/den never reach memory.  For the row interface one
// tile's contribution is added to num/den in memory.  In both the per-voxel
// floating-point operations and their order are those of the reference loop
// (tile contributions added one after the other); an A-scan whose lateral
// weight is zero is not read.
#include <cuda.h>
#include <cudaTypedefs.h>
#include <cuda_runtime.h>
#include <math.h>
#include <stdint.h>

#include "octgb_device.cuh"
#include "octgb_internal.h"

namespace octgb {
namespace {

constexpr int kStThreads = 256;          // 32 columns x 8 row groups

__device__ __forceinline__ void warp_minmax(float& mn, float& mx) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        mn = fminf(mn, __shfl_xor_sync(0xffffffffu, mn, o));
        mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
    }
}

// Folds [mn, mx] into an ordered-uint range in memory.  Most ranges add
// nothing: the current one is read first (an older, wider value only costs an
// atomic), since atomics of every warp on one address serialise in L2: 726 000 warps of a
// frame batch took ~1 ms, whatever else they did.
__device__ __forceinline__ void fold_range(unsigned int* mm, float mn, float mx) {
    if (!(mn <= mx)) return;
    const unsigned int lo = f2ord(mn), hi = f2ord(mx);
    const uint2 cur = __ldcg(reinterpret_cast<const uint2*>(mm));
    if (lo < cur.x) atomicMin(&mm[0], lo);
    if (hi > cur.y) atomicMax(&mm[1], hi);
}

// asynchronous global -> shared copy of one 8- or 16-byte element (both addresses aligned to its size)
template <int kBytes>
__device__ __forceinline__ void cp_async(void* dst, const void* src) {
    static_assert(kBytes == 8 || kBytes == 16, "cp.async element size");
    asm volatile("cp.async.ca.shared.global [%0], [%1], %2;" ::"r"(
                     static_cast<uint32_t>(__cvta_generic_to_shared(dst))),
                 "l"(src), "n"(kBytes)
                 : "memory");
}

// One CTA = one frame x kFZ output rows x 32 output columns.  The tiles
// touching each block and their patch extents come from a table built once per
// tile list on the host (StitchSlot); the CTA reads the table and each tile's
// plan fields in one round of loads, then stages every contributing patch and
// the tiles' per-row / per-column interpolation parameters (precomputed per
// plan) in shared memory by asynchronous copies: no load waits on another
// before the one barrier.  Then every voxel sums the tiles in order.
// kFZ output rows per CTA (the tile shape the autotuner picks: 32, 64 or 128).
// Where every column of a block takes one A-scan of a tile (kSlotSingle: the
// output grid and the tile's share their pixels, as a scan's do except in the
// first columns of a tile and between tiles at a fraction of a pixel) the
// second A-scan, its weight of zero and half of the reads fall away.
// kRow: one tile, its contribution added to num / den (the row interface);
// otherwise all tiles, finalised to dB with the plane and running range.
// Issue-bound (1776 warp instructions a warp of 256 voxels, a third of them
// staging): 183 M voxels of 6 tiles in ~1180 us; k_stitch_tma takes what it can.
template <int kFZ, bool kRow>
__global__ void __launch_bounds__(kStThreads) k_stitch(const StitchDev* __restrict__ plans, const StitchArgs a) {
    constexpr int kFRows = kFZ / 8;          // rows per thread
    // dynamic shared memory: row / column parameters of a round's slots, then the patches
    extern __shared__ __align__(16) float smem_all[];
    __shared__ StitchSlot slot[kMaxSeg];
    float4* rowp = reinterpret_cast<float4*>(smem_all);                 // [ns_round][kFZ] {zr, w0, w1, F interpolated}
    float2* rowf = reinterpret_cast<float2*>(rowp + a.ns_round * kFZ);  // [ns_round][kFZ] {F of the row's two taps}
    float4* colp = reinterpret_cast<float4*>(rowf + a.ns_round * kFZ);  // [ns_round][kBlk] {xr, wx0, wx1, single A-scan}
    float* sm = reinterpret_cast<float*>(colp + a.ns_round * kBlk);
    const int f = blockIdx.z;
    const int zb = blockIdx.y * kFZ;
    const int cb = (a.cblk0 + blockIdx.x) * kBlk;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int blk = blockIdx.y * gridDim.x + blockIdx.x;
    const int ns = a.slot_count[blk];
    if (kRow && ns == 0) return;
    if (tid < ns) slot[tid] = a.slots[static_cast<int64_t>(blk) * a.tiles.n + tid];
    __syncthreads();

    // 1. stage each contributing tile's interpolation parameters and its
    //    magnitude patch (F beside it when the optical-path correction makes it
    //    depend on the A-scan); depth fastest in the patch, one zero row after
    //    each A-scan's rows and (unless single) one zero A-scan after the last
    //    (stride s.rst), so every read below is in the patch.  Slots k0 .. k1 - 1
    //    of a round are spread over the warps (a warp deals with one slot, not
    //    each with all of them); the patch is copied as is (asynchronous 4-byte
    //    copies, 32 rows of an A-scan a warp); the focus weight multiplies it
    //    when it is read, the same single product a * F.
    auto stage = [&](int k, int kr, int part, int parts) {
        const StitchSlot s = slot[k];
        const StitchDev& p = plans[a.tiles.id[s.t]];
        const bool opc = (s.kind & kSlotOpc) != 0;
        const int na = (s.kind & kSlotSingle) ? s.xs : s.xs + 1;
        float* pa = sm + s.off;
        float* pf = pa + na * s.rst;
        const int r0 = p.r0 + s.r_lo;
        const float* mag_f = a.mag + s.t * a.mag_tile_stride + static_cast<int64_t>(f) * a.n_tile_x * kHalf;
        if (!opc) {
            const float* src = mag_f + static_cast<int64_t>(s.x_lo + part) * kHalf + r0 + lane;
            uint32_t dst = static_cast<uint32_t>(__cvta_generic_to_shared(pa + part * s.rst + lane));
            for (int xx = part; xx < s.xs; xx += parts) {
                for (int rr = 0; rr < s.rs; rr += 32)
                    if (rr + lane < s.rs)
                        asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(dst + 4 * rr), "l"(src + rr)
                                     : "memory");
                src += static_cast<int64_t>(parts) * kHalf;
                dst += static_cast<uint32_t>(parts * s.rst) * 4u;
            }
        } else {
            const int fy = kRow && a.frame_y != nullptr ? a.frame_y[f] : a.f0 + f;
            for (int xx = part; xx < s.xs; xx += parts) {
                const int x = s.x_lo + xx;
                const int64_t o = static_cast<int64_t>(fy) * p.n_tile_x + x;
                const int lo = p.lo[o], hi = p.hi[o], shift = p.shift[o];
                for (int rr = lane; rr < s.rs; rr += 32) {
                    const int i = xx * s.rst + rr;
                    const int ra = r0 + rr;
                    pf[i] = (ra < lo || ra > hi) ? 0.f : p.fz[s.r_lo + rr];
                    int src = ra + shift;
                    src = src < 0 ? 0 : (src > p.n_rows - 1 ? p.n_rows - 1 : src);
                    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(
                                     static_cast<uint32_t>(__cvta_generic_to_shared(pa + i))),
                                 "l"(mag_f + static_cast<int64_t>(x) * kHalf + src)
                                 : "memory");
                }
            }
        }
        if (part != 0) return;
        // without the optical-path correction F depends on the row only: its two
        // taps and the depth-interpolated F (the den term) per row.  The slot's
        // rows reach zr + 1 of every row, so the per-plan F[zr + 1] (0 past the
        // window) is the one the patch holds.
        for (int z = lane; z < kFZ; z += 32) {
            const int zo = zb + z;
            if (zo < p.n_out_z) {
                cp_async<16>(rowp + kr * kFZ + z, p.zrow + zo);
                cp_async<8>(rowf + kr * kFZ + z, p.zf + zo);
            } else {
                rowp[kr * kFZ + z] = make_float4(__int_as_float(-1), 0.f, 0.f, 0.f);
                rowf[kr * kFZ + z] = make_float2(0.f, 0.f);
            }
        }
        // the slot's A-scans reach every one a column of the block reads
        const int cc = cb + lane - p.c0;
        if (cc >= 0 && cc < p.C)
            cp_async<16>(colp + kr * kBlk + lane, p.xcol + cc);
        else
            colp[kr * kBlk + lane] = make_float4(__int_as_float(-1), 0.f, 0.f, __int_as_float(-1));
        // zero rows (rst - rs of them, 1 or 2) and the zero A-scan (plain stores, before the barrier)
        for (int xx = lane; xx < s.xs; xx += 32)
            for (int r = s.rs; r < s.rst; ++r) {
                pa[xx * s.rst + r] = 0.f;
                if (opc) pf[xx * s.rst + r] = 0.f;
            }
        if (na > s.xs)
            for (int r = lane; r < s.rst; r += 32) {
                pa[s.xs * s.rst + r] = 0.f;
                if (opc) pf[s.xs * s.rst + r] = 0.f;
            }
    };
    float an[kFRows], ad[kFRows];
#pragma unroll
    for (int q = 0; q < kFRows; ++q) an[q] = ad[q] = 0.f;
    const int tx = lane, ty = warp;
    const int c = cb + tx;
    // (most blocks take one round; those where many tiles meet take several, so
    // that they do not set the shared memory of all)
    for (int k0 = 0, k1; k0 < ns; k0 = k1) {
    k1 = k0;
    while (!slot[k1++].last) {
    }
    if (k0 > 0) __syncthreads();                             // the previous round's patches have been read
    {
        const int n = k1 - k0;
        constexpr int kWarps = kStThreads / 32;
        if (n <= kWarps) {
            const int kr = warp % n;
            stage(k0 + kr, kr, warp / n, (kWarps - 1 - kr) / n + 1);
        } else {
            for (int kr = warp; kr < n; kr += kWarps) stage(k0 + kr, kr, 0, 1);
        }
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
    __syncthreads();

    // 2. per voxel: tiles in order, depth (Wz) then lateral (WxT) interpolation.
    //    A tap outside the patch reads a zero, so a * F and F of it are the
    //    zeros the reference's operators give there.
    for (int k = k0; k < k1; ++k) {
        const float4 cp = colp[(k - k0) * kBlk + tx];
        const int kind = slot[k].kind;
        const int xr = __float_as_int((kind & kSlotSingle) ? cp.w : cp.x);
        if (xr < 0) continue;
        const int rst = slot[k].rst;
        // this thread's first A-scan of the patch, rows indexed by zr directly
        const float* pa = sm + slot[k].off + (xr - slot[k].x_lo) * rst - slot[k].r_lo;
        const float wx0 = cp.y, wx1 = cp.z;
        const float4* rpk = rowp + (k - k0) * kFZ + ty;
        const float2* rfk = rowf + (k - k0) * kFZ + ty;
        if (kind == kSlotSingle) {
            const float w = wx0 != 0.f ? wx0 : wx1;          // the other is zero
#pragma unroll
            for (int q = 0; q < kFRows; ++q) {
                const float4 rp = rpk[8 * q];
                const int zr = __float_as_int(rp.x);
                if (zr < 0) continue;
                const float2 ff = rfk[8 * q];
                // a = magnitude * F (TileStitcher.contribute, stitching.py:136)
                const float a0 = pa[zr] * ff.x, a1 = pa[zr + 1] * ff.y;
                const float u = fmaf(a1, rp.z, a0 * rp.y);
                an[q] += __fmul_rn(u, w);
                ad[q] += __fmul_rn(rp.w, w);
            }
        } else if (kind == 0) {
            // F depends on the row only: its two taps and the den term per row
#pragma unroll
            for (int q = 0; q < kFRows; ++q) {
                const float4 rp = rpk[8 * q];
                const int zr = __float_as_int(rp.x);
                if (zr < 0) continue;
                const float* p0 = pa + zr;
                const float* p1 = p0 + rst;
                const float w0 = rp.y, w1 = rp.z, d = rp.w;
                const float2 ff = rfk[8 * q];
                const float a00 = p0[0] * ff.x, a01 = p0[1] * ff.y;
                const float a10 = p1[0] * ff.x, a11 = p1[1] * ff.y;
                const float u0 = fmaf(a01, w1, a00 * w0), u1 = fmaf(a11, w1, a10 * w0);
                an[q] += fmaf(u1, wx1, u0 * wx0);
                ad[q] += fmaf(d, wx1, d * wx0);
            }
        } else if (kind & kSlotSingle) {
            // optical-path correction: F per A-scan and row, its patch after the magnitudes
            const float w = wx0 != 0.f ? wx0 : wx1;
            const float* pf = pa + slot[k].xs * rst;
#pragma unroll
            for (int q = 0; q < kFRows; ++q) {
                const float4 rp = rpk[8 * q];
                const int zr = __float_as_int(rp.x);
                if (zr < 0) continue;
                const float f0 = pf[zr], f1 = pf[zr + 1];
                const float a0 = pa[zr] * f0, a1 = pa[zr + 1] * f1;
                const float u = fmaf(a1, rp.z, a0 * rp.y), d = fmaf(f1, rp.z, f0 * rp.y);
                an[q] += __fmul_rn(u, w);
                ad[q] += __fmul_rn(d, w);
            }
        } else {
            const float* pf = pa + (slot[k].xs + 1) * rst;
#pragma unroll
            for (int q = 0; q < kFRows; ++q) {
                const float4 rp = rpk[8 * q];
                const int zr = __float_as_int(rp.x);
                if (zr < 0) continue;
                const float w0 = rp.y, w1 = rp.z;
                const float f00 = pf[zr], f01 = pf[zr + 1], f10 = pf[zr + rst], f11 = pf[zr + rst + 1];
                const float d0 = fmaf(f01, w1, f00 * w0), d1 = fmaf(f11, w1, f10 * w0);
                const float a00 = pa[zr] * f00, a01 = pa[zr + 1] * f01;
                const float a10 = pa[zr + rst] * f10, a11 = pa[zr + rst + 1] * f11;
                const float u0 = fmaf(a01, w1, a00 * w0), u1 = fmaf(a11, w1, a10 * w0);
                an[q] += fmaf(u1, wx1, u0 * wx0);
                ad[q] += fmaf(d1, wx1, d0 * wx0);
            }
        }
    }
    }

    if (kRow) {
        if (c >= a.n_out_x) return;
#pragma unroll
        for (int q = 0; q < kFRows; ++q) {
            const int zo = zb + ty + 8 * q;
            if (zo >= a.n_out_z || (an[q] == 0.f && ad[q] == 0.f)) continue;
            const int64_t o = (static_cast<int64_t>(a.frame_offset + f) * a.n_out_z + zo) * a.n_out_x + c;
            a.num[o] += an[q];
            a.den[o] += ad[q];
        }
        return;
    }
    // 3. finalise (pipeline.py:296-300) and clim (io/tiff_writer.py:48-50)
    float mn = __int_as_float(0x7f800000), mx = -__int_as_float(0x7f800000);
#pragma unroll
    for (int q = 0; q < kFRows; ++q) {
        const int zo = zb + ty + 8 * q;
        if (zo >= a.n_out_z || c >= a.n_out_x) continue;
        float v;
        if (ad[q] < a.thr || isnan(ad[q])) {
            v = __int_as_float(0x7fc00000);
        } else {
            v = 20.0f * log10f(__fdiv_rn(an[q], ad[q]));
        }
        a.db[(static_cast<int64_t>(f) * a.n_out_z + zo) * a.n_out_x + c] = v;
        if (isfinite(v)) {
            mn = fminf(mn, v);
            mx = fmaxf(mx, v);
        }
    }
    warp_minmax(mn, mx);
    if (lane == 0) {
        if (a.plane_mm) fold_range(a.plane_mm + 2 * f, mn, mx);
        if (a.run_mm) fold_range(a.run_mm, mn, mx);
    }
}

// k_stitch without the optical-path correction, its staging by tensor copies:
// per slot one thread issues a two-dimensional copy of the patch (an aligned
// window of pitch rows of xs A-scans) and bulk copies of the block's row and
// column parameters from the plan's tables (padded, so that a block never
// leaves them); the other threads only wait.  Rows past a tile's window carry
// weights of zero.  A copy starts at a row that is a multiple of four and its
// pitch is 4 x an odd number: a warp takes 8 columns x 4 rows, whose reads then
// fall in distinct banks (8 A-scans a pitch apart x 4 neighbouring rows), and
// writes whole 32-byte sectors.  Five blocks an SM (48 registers): 183 M voxels
// of 6 tiles in ~720 us, ~1180 with the copies spread over the threads
// (k_stitch); four blocks ~840, six (spills) ~815.
template <int kFZ, bool kRow>
__global__ void __launch_bounds__(kStThreads, kFZ == 128 ? 3 : 5) k_stitch_tma(const __grid_constant__ CUtensorMap map,
                                                           const StitchArgs a) {
    constexpr int kFRows = kFZ / 8;          // rows per thread
    extern __shared__ __align__(128) unsigned char smem_raw[];
    __shared__ uint64_t bar;
    __shared__ StitchTmaSlot slot[kMaxSeg];
    unsigned char* sm = smem_raw + align_up_smem(smem_raw, 128);   // tensor copies: 128-byte aligned
    const int f = blockIdx.z;
    const int zb = blockIdx.y * kFZ;
    const int cb = (a.cblk0 + blockIdx.x) * kBlk;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int blk = blockIdx.y * gridDim.x + blockIdx.x;
    const int ns = a.slot_count[blk];
    if (kRow && ns == 0) return;
    if (tid < ns) slot[tid] = a.tslots[static_cast<int64_t>(blk) * a.tiles.n + tid];
    if (tid == 0) {
        mbar_init(&bar, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();
    const int cl = 8 * (warp & 3) + (lane & 7);                      // column of the block
    const int zl = (warp >> 2) * (kFZ / 2) + (lane >> 3);            // first row; then every fourth
    const int c = cb + cl;
    const uint32_t row_off = a.patch_bytes, rowf_off = row_off + kFZ * 16, col_off = rowf_off + kFZ * 8;
    float an[kFRows], ad[kFRows];
#pragma unroll
    for (int q = 0; q < kFRows; ++q) an[q] = ad[q] = 0.f;
    for (int k0 = 0, round = 0; k0 < ns; k0 += a.ns_round, ++round) {
        const int n = min(a.ns_round, ns - k0);
        if (round > 0) __syncthreads();                              // the previous round has been read
        if (warp == 0) {
            if (lane == 0)
                mbar_expect_tx(&bar, static_cast<uint32_t>(n) * (a.pitch * a.box_lines * 4 + kFZ * 24 + kBlk * 16) +
                                         (round == 0 ? a.starve : 0u));
            __syncwarp();
            if (lane < n) {
                const StitchTmaSlot& s = slot[k0 + lane];
                unsigned char* d = sm + lane * a.slot_bytes;
                asm volatile(
                    "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], "
                    "[%1, {%2, %3}], [%4];" ::"r"(smem_u32(d)),
                    "l"(reinterpret_cast<uint64_t>(&map)), "r"(s.row0), "r"(s.t * a.tile_lines + f * a.n_tile_x + s.x_lo),
                    "r"(smem_u32(&bar))
                    : "memory");
                tma_bulk_g2s(d + row_off, s.zrow, kFZ * 16, &bar);
                tma_bulk_g2s(d + rowf_off, s.zf, kFZ * 8, &bar);
                tma_bulk_g2s(d + col_off, s.xcol, kBlk * 16, &bar);
            }
        }
        if (!__all_sync(0xffffffffu, mbar_wait_bounded(&bar, round & 1, a.status))) {
            mbar_wait_bounded(&bar, round & 1, a.status);    // the copies land before the CTA ends
            return;
        }
        for (int kr = 0; kr < n; ++kr) {
            const StitchTmaSlot& s = slot[k0 + kr];
            const unsigned char* d = sm + kr * a.slot_bytes;
            const float4 cp = reinterpret_cast<const float4*>(d + col_off)[cl];
            const int x = __float_as_int(s.single ? cp.w : cp.x);
            if (x < 0) continue;
            const int P = a.pitch;
            // this thread's first A-scan of the patch, rows indexed by zr directly
            const float* pa = reinterpret_cast<const float*>(d) + (x - s.x_lo) * P - s.r_lo;
            const float4* rpk = reinterpret_cast<const float4*>(d + row_off) + zl;
            const float2* rfk = reinterpret_cast<const float2*>(d + rowf_off) + zl;
            if (s.single) {
                const float w = cp.y != 0.f ? cp.y : cp.z;           // the other is zero
#pragma unroll
                for (int q = 0; q < kFRows; ++q) {
                    const float4 rp = rpk[4 * q];
                    const int zr = __float_as_int(rp.x);
                    if (zr < 0) continue;
                    const float2 ff = rfk[4 * q];
                    // a = magnitude * F (TileStitcher.contribute, stitching.py:136)
                    const float a0 = pa[zr] * ff.x, a1 = pa[zr + 1] * ff.y;
                    const float u = fmaf(a1, rp.z, a0 * rp.y);
                    an[q] += __fmul_rn(u, w);
                    ad[q] += __fmul_rn(rp.w, w);
                }
            } else {
                const float wx0 = cp.y, wx1 = cp.z;
#pragma unroll
                for (int q = 0; q < kFRows; ++q) {
                    const float4 rp = rpk[4 * q];
                    const int zr = __float_as_int(rp.x);
                    if (zr < 0) continue;
                    const float* p0 = pa + zr;
                    const float* p1 = p0 + P;
                    const float w0 = rp.y, w1 = rp.z, dd = rp.w;
                    const float2 ff = rfk[4 * q];
                    const float a00 = p0[0] * ff.x, a01 = p0[1] * ff.y;
                    const float a10 = p1[0] * ff.x, a11 = p1[1] * ff.y;
                    const float u0 = fmaf(a01, w1, a00 * w0), u1 = fmaf(a11, w1, a10 * w0);
                    an[q] += fmaf(u1, wx1, u0 * wx0);
                    ad[q] += fmaf(dd, wx1, dd * wx0);
                }
            }
        }
    }
    if (kRow) {
        if (c >= a.n_out_x) return;
#pragma unroll
        for (int q = 0; q < kFRows; ++q) {
            const int zo = zb + zl + 4 * q;
            if (zo >= a.n_out_z || (an[q] == 0.f && ad[q] == 0.f)) continue;
            const int64_t o = (static_cast<int64_t>(a.frame_offset + f) * a.n_out_z + zo) * a.n_out_x + c;
            a.num[o] += an[q];
            a.den[o] += ad[q];
        }
        return;
    }
    // finalise (pipeline.py:296-300) and clim (io/tiff_writer.py:48-50)
    float mn = __int_as_float(0x7f800000), mx = -__int_as_float(0x7f800000);
    float* out = a.db + (static_cast<int64_t>(f) * a.n_out_z + zb + zl) * a.n_out_x + c;
#pragma unroll
    for (int q = 0; q < kFRows; ++q) {
        if (zb + zl + 4 * q >= a.n_out_z || c >= a.n_out_x) continue;
        float v;
        if (ad[q] < a.thr || isnan(ad[q])) {
            v = __int_as_float(0x7fc00000);
        } else {
            v = 20.0f * log10f(__fdiv_rn(an[q], ad[q]));
        }
        out[static_cast<int64_t>(4 * q) * a.n_out_x] = v;
        if (isfinite(v)) {
            mn = fminf(mn, v);
            mx = fmaxf(mx, v);
        }
    }
    warp_minmax(mn, mx);
    if (lane == 0) {
        if (a.plane_mm) fold_range(a.plane_mm + 2 * f, mn, mx);
        if (a.run_mm) fold_range(a.run_mm, mn, mx);
    }
}

// Batched form, after the transform: each A-scan's depth operator and focus
// weight (u = Wz (a F)), the lateral operator between neighbouring A-scans
// (num = WxT u, den likewise) as TileStitcher.contribute for one tile
// (stitching.py:126-139), then finalise (pipeline.py:296-300).  The lateral
// operator of a single tile is the identity except for the reference's 1e-10
// widening of its end nodes, which blends a neighbour in with a weight ~1e-7
// (the host checks that it lies within four A-scans).  One block takes
// kResLines A-scans, a thread an output row of all of them: the row's
// parameters are read once, reads and writes run along depth.  12 tiles of
// 100 500 A-scans, 104 M rows: the whole call takes 939 us; as the epilogue of
// the spectral kernel (16 warps between block barriers) it took 2086 us.
constexpr int kResThreads = 256, kResLines = 8;
__global__ void __launch_bounds__(kResThreads) k_resample(const QueueTile* __restrict__ qt, int n_qt, unsigned int l0,
                                                          unsigned int l1, const float* __restrict__ mag, float thr,
                                                          unsigned int* __restrict__ run_mm) {
    struct Line {
        const float4* zrow;
        const float2* zf;
        const float* m0;                         // magnitudes (from row r0) of the first A-scan blended in
        float* out;
        float wx0, wx1;
        int nz, tile;                            // nz 0: no line
    };
    __shared__ Line L[kResLines];
    __shared__ unsigned int mm[2];
    const int tid = threadIdx.x;
    if (tid == 0) {
        mm[0] = 0xffffffffu;
        mm[1] = 0u;
    }
    if (tid < kResLines) {
        Line q{};
        const unsigned int l = l0 + blockIdx.x * kResLines + tid;
        if (l < l1) {
            int lo = 0, hi = n_qt - 1;           // last tile with line0 <= l
            while (lo < hi) {
                const int mid = (lo + hi + 1) >> 1;
                if (qt[mid].line0 <= l) lo = mid; else hi = mid - 1;
            }
            const QueueTile& t = qt[lo];
            const StitchDev& p = *t.plan;
            const unsigned int as = l - t.line0;
            const int x = static_cast<int>(as % static_cast<unsigned int>(t.nx));
            q.tile = lo;
            q.nz = t.nz;
            q.zrow = p.zrow;
            q.zf = p.zf;
            q.wx0 = p.wx0[x];
            q.wx1 = p.wx1[x];
            // A-scan xr + 1 is read only with a weight: it is then in this pass
            q.m0 = mag + static_cast<int64_t>(l - l0) * kHalf + static_cast<int64_t>(p.xr[x] - x) * kHalf + p.r0;
            q.out = t.out + static_cast<int64_t>(as) * t.nz;
        }
        L[tid] = q;
    }
    __syncthreads();
    int nz = 0;
#pragma unroll
    for (int j = 0; j < kResLines; ++j) nz = max(nz, L[j].nz);
    float mn = __int_as_float(0x7f800000), mx = -__int_as_float(0x7f800000);
    for (int zo = tid; zo < nz; zo += kResThreads) {
        int tile = -1, zr = -1;
        float4 rw = make_float4(0.f, 0.f, 0.f, 0.f);
        float2 ff = make_float2(0.f, 0.f);
#pragma unroll 4
        for (int j = 0; j < kResLines; ++j) {
            const Line& q = L[j];
            if (zo >= q.nz) continue;
            if (q.tile != tile) {
                tile = q.tile;
                rw = __ldg(q.zrow + zo);
                ff = __ldg(q.zf + zo);
                zr = __float_as_int(rw.x);
            }
            float v = __int_as_float(0x7fc00000);
            if (zr >= 0) {
                // a row without a second tap (F1 = 0) does not read it
                auto depth = [&](const float* m) {
                    const float a0 = m[zr] * ff.x;
                    const float a1 = ff.y != 0.f ? m[zr + 1] * ff.y : 0.f;
                    return fmaf(a1, rw.z, a0 * rw.y);
                };
                const float u0 = q.wx0 != 0.f ? depth(q.m0) : 0.f;
                const float u1 = q.wx1 != 0.f ? depth(q.m0 + kHalf) : 0.f;
                const float num = fmaf(u1, q.wx1, u0 * q.wx0);
                const float den = fmaf(rw.w, q.wx1, rw.w * q.wx0);
                if (!(den < thr) && !isnan(den)) v = 20.0f * log10f(__fdiv_rn(num, den));
            }
            q.out[zo] = v;
            if (isfinite(v)) {
                mn = fminf(mn, v);
                mx = fmaxf(mx, v);
            }
        }
    }
    warp_minmax(mn, mx);
    if ((tid & 31) == 0 && mn <= mx) {
        atomicMin(&mm[0], f2ord(mn));
        atomicMax(&mm[1], f2ord(mx));
    }
    __syncthreads();
    if (tid == 0 && mm[0] != 0xffffffffu) fold_range(run_mm, ord2f(mm[0]), ord2f(mm[1]));
}

// pipeline.py:296-300 plus plane_clim (io/tiff_writer.py:48-50)
__global__ void k_finalise(const float* __restrict__ num, const float* __restrict__ den, int64_t n_per_plane,
                           float thr, float* __restrict__ db, unsigned int* __restrict__ plane_mm) {
    const int plane = blockIdx.y;
    float mn = __int_as_float(0x7f800000), mx = -__int_as_float(0x7f800000);
    const int64_t base = static_cast<int64_t>(plane) * n_per_plane;
    for (int64_t i = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x; i < n_per_plane;
         i += static_cast<int64_t>(gridDim.x) * blockDim.x) {
        const float d = den[base + i];
        float v;
        if (d < thr || isnan(d)) {
            v = __int_as_float(0x7fc00000);
        } else {
            v = 20.0f * log10f(__fdiv_rn(num[base + i], d));
        }
        db[base + i] = v;
        if (isfinite(v)) {
            mn = fminf(mn, v);
            mx = fmaxf(mx, v);
        }
    }
    if (plane_mm == nullptr) return;
    warp_minmax(mn, mx);
    if ((threadIdx.x & 31) == 0 && mn <= mx) {
        atomicMin(&plane_mm[2 * plane], f2ord(mn));
        atomicMax(&plane_mm[2 * plane + 1], f2ord(mx));
    }
}

// MATLAB uint16() of (db - c1)/(c2 - c1) * 65534, then + 1 saturating, NaN -> 0
__device__ __forceinline__ uint16_t quantise_exact(float x, double c1, double span) {
    if (isnan(x)) return 0;
    const double v = (static_cast<double>(x) - c1) / span * 65534.0;
    double r = floor(fabs(v) + 0.5);
    if (v < 0) r = -r;
    if (!(r > 0.0)) r = 0.0;
    if (r > 65535.0) r = 65535.0;
    const unsigned int u = static_cast<unsigned int>(r) + 1u;
    return static_cast<uint16_t>(u > 65535u ? 65535u : u);
}

// The legacy code is a non-decreasing function of the float32 dB value
// (every float64 step is monotonic), so it is fully described by 65534
// thresholds T[k] = the smallest float32 x with code(x) >= k (k = 2..65535;
// T[1] = -inf, T[65536] = +inf).  k_quant_table finds each T[k] in float64:
// a float32 guess next to c1 + (k - 1.5) * span / 65534, then moved ulp by ulp
// until code(T[k]) >= k > code(prev(T[k])).  Per voxel a float32 estimate
// v32 = (x - c1f) * sf (error < 0.02 code) gives the code directly when v32
// is more than kGuard from a rounding boundary; otherwise two table
// comparisons decide.  Bit-exact, and no float64 work per voxel.
constexpr float kGuard = 0.05f;
constexpr int kTable = 65537;

__global__ void k_quant_table(const unsigned int* __restrict__ clim_mm, double c1_in, double c2_in,
                              float* __restrict__ T) {
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= kTable) return;
    double c1 = c1_in, c2 = c2_in;
    if (clim_mm != nullptr) {
        c1 = static_cast<double>(ord2f(clim_mm[0]));
        c2 = static_cast<double>(ord2f(clim_mm[1]));
    }
    const double span = c2 - c1;
    if (k <= 1) {
        T[k] = -__int_as_float(0x7f800000);
        return;
    }
    if (k == kTable - 1) {
        T[k] = __int_as_float(0x7f800000);
        return;
    }
    float y = static_cast<float>(c1 + (k - 1.5) * span / 65534.0);
    const float lo = -__int_as_float(0x7f800000), hi = __int_as_float(0x7f800000);
    for (int i = 0; i < 256 && quantise_exact(y, c1, span) >= k; ++i) y = nextafterf(y, lo);
    for (int i = 0; i < 256 && quantise_exact(y, c1, span) < k; ++i) y = nextafterf(y, hi);
    T[k] = y;
}

struct QuantParams {
    float c1f, sf;
    bool fast;
};

__host__ __device__ inline QuantParams quant_params(double c1, double c2) {
    QuantParams q;
    const double span = c2 - c1;
    q.c1f = static_cast<float>(c1);
    q.sf = static_cast<float>(65534.0 / span);
    // three float32 roundings of values <= ~65535 plus the offset error of c1f
    const double off = fabs(c1 - static_cast<double>(q.c1f)) * (65534.0 / span);
    q.fast = (4.0 * 65536.0 * 5.96e-8 + off) < 0.5 * kGuard && span > 0.0;
    return q;
}

__device__ __forceinline__ uint16_t quantise_one(float x, const QuantParams& q, const float* __restrict__ T) {
    if (isnan(x)) return 0;
    int n;       // estimated code
    if (q.fast) {
        const float v = (x - q.c1f) * q.sf;
        if (v < 0.5f - kGuard) return 1;              // rounds to <= 0: clipped to 0, + 1
        if (v > 65534.5f + kGuard) return 65535;      // rounds to >= 65535: + 1 saturates
        const float f = v + 0.5f;
        const float fl = floorf(f);
        const float fr = f - fl;
        n = static_cast<int>(fl) + 1;
        if (fr > kGuard && fr < 1.0f - kGuard) return static_cast<uint16_t>(n);
        n = n < 1 ? 1 : (n > 65535 ? 65535 : n);
        // within one code of the truth: settle with the thresholds
        if (n < 65535 && x >= T[n + 1]) return static_cast<uint16_t>(n + 1);
        if (x >= T[n]) return static_cast<uint16_t>(n);
        return static_cast<uint16_t>(n - 1);
    }
    // no usable estimate: binary search of the thresholds
    int a = 1, b = 65535;        // code in [a, b]
    while (a < b) {
        const int m = (a + b + 1) >> 1;
        if (x >= T[m]) a = m; else b = m - 1;
    }
    return static_cast<uint16_t>(a);
}

// Grid-stride quantisation of n voxels: 4 per thread and iteration (one
// 16-byte load, one 8-byte store) when db and bits are aligned for it, so the
// pass streams at HBM rate; scalar otherwise and for the tail.
__device__ __forceinline__ void quantise_span(const float* __restrict__ db, int64_t n, const QuantParams& q,
                                              const float* __restrict__ T, uint16_t* __restrict__ bits) {
    const int64_t tid = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x;
    const int64_t stride = static_cast<int64_t>(gridDim.x) * blockDim.x;
    int64_t done = 0;
    if ((reinterpret_cast<uintptr_t>(db) & 15u) == 0 && (reinterpret_cast<uintptr_t>(bits) & 7u) == 0) {
        const int64_t n4 = n >> 2;
        const float4* d4 = reinterpret_cast<const float4*>(db);
        uint2* b4 = reinterpret_cast<uint2*>(bits);
        // four independent 16-byte loads in flight per thread
        int64_t i = tid;
        for (; i + 3 * stride < n4; i += 4 * stride) {
            float4 v[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) v[u] = d4[i + u * stride];
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                const unsigned int c0 = quantise_one(v[u].x, q, T), c1 = quantise_one(v[u].y, q, T);
                const unsigned int c2 = quantise_one(v[u].z, q, T), c3 = quantise_one(v[u].w, q, T);
                b4[i + u * stride] = make_uint2(c0 | (c1 << 16), c2 | (c3 << 16));
            }
        }
        for (; i < n4; i += stride) {
            const float4 v = d4[i];
            const unsigned int c0 = quantise_one(v.x, q, T), c1 = quantise_one(v.y, q, T);
            const unsigned int c2 = quantise_one(v.z, q, T), c3 = quantise_one(v.w, q, T);
            b4[i] = make_uint2(c0 | (c1 << 16), c2 | (c3 << 16));
        }
        done = n4 << 2;
    }
    for (int64_t i = done + tid; i < n; i += stride) bits[i] = quantise_one(db[i], q, T);
}

// db_to_bits (io/tiff_writer.py:26-38), float64 semantics
__global__ void k_quantise(const float* __restrict__ db, int64_t n, double c1, double c2,
                           const float* __restrict__ T, uint16_t* __restrict__ bits) {
    quantise_span(db, n, quant_params(c1, c2), T, bits);
}

// same with the clim read from device memory (ordered-uint [min, max] of float32 dB)
__global__ void k_quantise_dev(const float* __restrict__ db, int64_t n, const unsigned int* __restrict__ clim_mm,
                               const float* __restrict__ T, uint16_t* __restrict__ bits) {
    quantise_span(db, n, quant_params(static_cast<double>(ord2f(clim_mm[0])), static_cast<double>(ord2f(clim_mm[1]))),
                  T, bits);
}

__global__ void k_minmax(const float* __restrict__ x, int64_t n, unsigned int* __restrict__ mm) {
    float mn = __int_as_float(0x7f800000), mx = -__int_as_float(0x7f800000);
    for (int64_t i = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x; i < n;
         i += static_cast<int64_t>(gridDim.x) * blockDim.x) {
        const float v = x[i];
        if (isfinite(v)) {
            mn = fminf(mn, v);
            mx = fmaxf(mx, v);
        }
    }
    warp_minmax(mn, mx);
    if ((threadIdx.x & 31) == 0) fold_range(mm, mn, mx);
}

__global__ void k_minmax_init(unsigned int* mm, int count) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < count) mm[i] = (i & 1) ? 0u : 0xffffffffu;
}

int grid_for(int64_t n, int threads) {
    int64_t b = (n + threads - 1) / threads;
    if (b > 152 * 32) b = 152 * 32;
    return static_cast<int>(b < 1 ? 1 : b);
}

}  // namespace

namespace {
// the magnitudes as lines of kHalf floats, boxes of `pitch` floats x `lines`
bool encode_mag_map(CUtensorMap* map, const float* mag, int64_t n_lines, int pitch, int lines) {
    static PFN_cuTensorMapEncodeTiled_v12000 encode = nullptr;
    if (encode == nullptr) {
        cudaDriverEntryPointQueryResult q;
        void* fn = nullptr;
        if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &fn, 12000, cudaEnableDefault, &q) !=
                cudaSuccess ||
            q != cudaDriverEntryPointSuccess || fn == nullptr)
            return false;
        encode = reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(fn);
    }
    const cuuint64_t dims[2] = {static_cast<cuuint64_t>(kHalf), static_cast<cuuint64_t>(n_lines)};
    const cuuint64_t strides[1] = {kHalf * sizeof(float)};
    const cuuint32_t box[2] = {static_cast<cuuint32_t>(pitch), static_cast<cuuint32_t>(lines)};
    const cuuint32_t estr[2] = {1, 1};
    return encode(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, const_cast<float*>(mag), dims, strides, box, estr,
                  CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                  CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}
}  // namespace

cudaError_t launch_stitch(const StitchDev* plans_dev, const StitchArgs& a, size_t patch_smem_bytes, int n_cblk, int B,
                          int rows, cudaStream_t st) {
    if (B == 0 || n_cblk == 0) return cudaSuccess;
    const bool row = a.num != nullptr;
    if (a.tslots != nullptr) {
        const auto kern = rows == 32   ? (row ? k_stitch_tma<32, true> : k_stitch_tma<32, false>)
                          : rows == 64 ? (row ? k_stitch_tma<64, true> : k_stitch_tma<64, false>)
                                       : (row ? k_stitch_tma<128, true> : k_stitch_tma<128, false>);
        const size_t smem = static_cast<size_t>(a.ns_round) * a.slot_bytes + 128;
        CUtensorMap map;
        if (!encode_mag_map(&map, a.mag, a.n_lines, a.pitch, a.box_lines)) return cudaErrorInvalidValue;
        cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem));
        if (e != cudaSuccess) return e;
        kern<<<dim3(n_cblk, (a.n_out_z + rows - 1) / rows, B), kStThreads, smem, st>>>(map, a);
        return cudaGetLastError();
    }
    const auto kern = rows == 32   ? (row ? k_stitch<32, true> : k_stitch<32, false>)
                      : rows == 64 ? (row ? k_stitch<64, true> : k_stitch<64, false>)
                                   : k_stitch<128, false>;
    if ((rows != 32 && rows != 64 && rows != 128) || (row && rows == 128)) return cudaErrorInvalidValue;
    const size_t smem = patch_smem_bytes +
                        static_cast<size_t>(a.ns_round) * sizeof(float) * (6 * rows + 4 * kBlk) + 16;
    if (smem > 200 * 1024) return cudaErrorInvalidValue;
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem));
    if (e != cudaSuccess) return e;
    kern<<<dim3(n_cblk, (a.n_out_z + rows - 1) / rows, B), kStThreads, smem, st>>>(plans_dev, a);
    return cudaGetLastError();
}

cudaError_t launch_finalise(const float* num, const float* den, int64_t n_per_plane, int n_planes, float thr,
                            float* db, unsigned int* plane_minmax, cudaStream_t st) {
    if (n_planes == 0 || n_per_plane == 0) return cudaSuccess;
    // enough blocks for every SM whatever the number of planes, eight values a thread at least
    int gx = grid_for((n_per_plane + 7) / 8, 256);
    const int most = n_planes < 16 ? 1024 / n_planes : 64;
    if (gx > most) gx = most;
    k_finalise<<<dim3(gx, n_planes), 256, 0, st>>>(num, den, n_per_plane, thr, db, plane_minmax);
    return cudaGetLastError();
}

cudaError_t launch_quantise(const float* db, int64_t n, double c1, double c2, float* table, uint16_t* bits,
                            cudaStream_t st) {
    if (n == 0) return cudaSuccess;
    k_quant_table<<<(kTable + 255) / 256, 256, 0, st>>>(nullptr, c1, c2, table);
    k_quantise<<<grid_for(n, 256), 256, 0, st>>>(db, n, c1, c2, table, bits);
    return cudaGetLastError();
}

cudaError_t launch_quantise_dev(const float* db, int64_t n, const unsigned int* clim_mm, float* table,
                                uint16_t* bits, cudaStream_t st) {
    if (n == 0) return cudaSuccess;
    k_quant_table<<<(kTable + 255) / 256, 256, 0, st>>>(clim_mm, 0.0, 0.0, table);
    k_quantise_dev<<<grid_for(n, 256), 256, 0, st>>>(db, n, clim_mm, table, bits);
    return cudaGetLastError();
}

cudaError_t launch_minmax(const float* x, int64_t n, unsigned int* mm, cudaStream_t st) {
    if (n == 0) return cudaSuccess;
    k_minmax<<<grid_for(n, 256), 256, 0, st>>>(x, n, mm);
    return cudaGetLastError();
}

cudaError_t launch_resample(const QueueTile* qt, int n_qt, unsigned int l0, unsigned int l1, const float* mag,
                            float thr, unsigned int* run_mm, cudaStream_t st) {
    if (l0 == l1) return cudaSuccess;
    k_resample<<<(l1 - l0 + kResLines - 1) / kResLines, kResThreads, 0, st>>>(qt, n_qt, l0, l1, mag, thr, run_mm);
    return cudaGetLastError();
}

cudaError_t set_wait_test_stitch(unsigned long long limit_ns, cudaStream_t st) {
    return set_wait_test_here(limit_ns, 0, st);
}

cudaError_t launch_minmax_init(unsigned int* mm, int count, cudaStream_t st) {
    if (count == 0) return cudaSuccess;
    k_minmax_init<<<(count + 255) / 256, 256, 0, st>>>(mm, count);
    return cudaGetLastError();
}

}  // namespace octgb

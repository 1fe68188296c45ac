// Tensor-core kernels of the learned estimator.
//
// k_conv3x3_tc: the 3x3 convolution (cnn.cu's k_conv3x3 on the tensor cores):
// stride 1, zero padding 1, + bias, NCHW float32 in and out, FP16 operands
// (BF16 for the data gradient) and float32 accumulation on the 5th-generation
// tensor cores (tcgen05.mma kind::f16, accumulator in TMEM).  Forward pass of
// training and inference, and the data gradient (the convolution of dy with
// the flipped kernel).  k_conv3x3_wgrad_tc (further down): the weight and
// bias gradients.
//
// Both are bound by the float32 planes they read and write, so both are built
// around that stream.  The unit of work is a band: R rows (of one column
// segment where whole rows would not fit) of one image.  Specialised warps
// hand a band on through mbarriers:
//   producer   copies the band's rows, eight channels at a time, into a ring of
//              raw slots (one tensor copy a slot);
//   converters pack a slot's rows to 16-bit operands in one of two staged blocks
//              (kDirect, rows off 16-byte boundaries: from memory, all channels at
//              once; a form of its own, since both in one kernel cost the slots'
//              form up to 18 %);
//   MMA        one warp issues the band's tcgen05.mma;
//   epilogue   (convolution) drains the accumulators to global memory.
// Copies of later bands are in flight throughout, so no phase waits for the
// memory latency.  Measured at 128 images, against kernels that staged each tile
// with plain loads between two block barriers (and summed the bias gradient in a
// pass of its own):
//   convolution       3 x 256 x 256: 516 -> 270 us (4.3 TB/s), 32 x 128 x 128: 370 -> 104 us (5.2 TB/s)
//     + ReLU + mean   280 -> 217 us, 265 -> 88 us
//   gradients of w, b 1100 -> 274 us (4.2 TB/s), 470 -> 180 us (3.0 TB/s)
// What bounds them now: the 1.1 GB stream of the first convolution and its nine
// MMAs a tile about equally; of the gradients the converters' instructions and
// the copies (168 us at 32 x 128 x 128 without MMAs).
//
// A staged block holds the band's input rows y0 - 1 .. y0 + R with a zero
// column before each row and zeros after it up to the row pitch Wp (W + 2
// rounded up to 4), as [channel group of 8][pixel][8 channels x 2 B].  Output
// pixel q = r * Wp + ox then meets input pixel q + ty * Wp + tx, so tap
// (ty, tx) is the staged block itself seen from that pixel on: a matrix
// descriptor offset of 16 bytes a pixel, no im2col copy.
//
// Every mbarrier wait is bounded; on expiry the CTA records the status, waits
// (bounded) for its copies and MMAs, frees its TMEM and returns.
#include <cuda.h>
#include <cudaTypedefs.h>
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "octgb_device.cuh"
#include "octgb_internal.h"

namespace octgb {
namespace {

constexpr int kCM = 128;                    // MMA M of the convolution: output pixels per tile
constexpr int kMaxSlots = 8;                // raw slots (3 at least: a copy in flight while two are converted)
constexpr int kMaxBox = 256;                // elements per dimension of a tensor copy
constexpr uint32_t kSmemBudget = 226u * 1024u;

// the bands of an image and the shape of a raw slot
struct Band {
    int C, H, W;
    int R;               // rows per band
    int Ws, Wp;          // columns per segment, staged row pitch
    int nseg, nband;     // per image
    int rp, rawp;        // raw slot of x: floats per row (W, or Ws + 8: from column x0 - 4), per channel (R + 2 rows)
    int vec;             // rows on 16-byte boundaries: tensor copies
    uint32_t wp_inv;     // ceil(2^32 / Wp)
    int64_t n_units;
};

struct BandAt {
    int img, y0, x0, rows;                  // rows: R, fewer in an image's last band
};

__device__ __forceinline__ int div_wp(const Band& g, int q) {
    return static_cast<int>(__umulhi(static_cast<uint32_t>(q), g.wp_inv));      // exact: q * Wp < 2^32
}

__device__ __forceinline__ BandAt band_at(const Band& g, int64_t u) {
    BandAt o;
    const int per_img = g.nband * g.nseg;
    o.img = static_cast<int>(u / per_img);
    const int i = static_cast<int>(u - static_cast<int64_t>(o.img) * per_img);
    const int band = i / g.nseg;
    o.y0 = band * g.R;
    o.x0 = (i - band * g.nseg) * g.Ws;
    o.rows = min(g.R, g.H - o.y0);
    return o;
}

// first column in a raw slot of x (4 before a segment: its halo column, on a 16-byte boundary)
__device__ __forceinline__ int slot_x0(const Band& g, const BandAt& o) { return g.nseg == 1 ? 0 : o.x0 - 4; }

__device__ __forceinline__ uint32_t pack_h2(float a, float b) {
    const __half2 h = __floats2half2_rn(a, b);
    return *reinterpret_cast<const uint32_t*>(&h);
}

__device__ __forceinline__ uint32_t pack_bf2(float a, float b) {
    const __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
    return *reinterpret_cast<const uint32_t*>(&h);
}

// two operand values in the kernel's 16-bit type, the first in the low half
template <bool kBf16>
__device__ __forceinline__ uint32_t pack2(float a, float b) {
    return kBf16 ? pack_bf2(a, b) : pack_h2(a, b);
}

// kind::f16 A and B formats: 0 = FP16, 1 = BF16 (both operands the same type)
constexpr uint32_t kIdescBf16 = (1u << 7) | (1u << 10);

// a bounded wait of a warp (all lanes go on, or none); false ends its role's loop
__device__ __forceinline__ bool role_wait(uint64_t* bar, uint32_t parity, int* abort, int* status) {
    bool ok = false;
    if (*reinterpret_cast<volatile int*>(abort) == 0) {
        ok = mbar_wait_bounded(bar, parity, status);
        if (!ok) atomicExch(abort, 1);
    }
    return __all_sync(0xffffffffu, ok);
}

__device__ __forceinline__ void tensor_copy(const CUtensorMap& map, int x0, int y0, int plane, float* dst,
                                            uint64_t* bar) {
    asm volatile(
        "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];" ::"r"(
            smem_u32(dst)),
        "l"(reinterpret_cast<uint64_t>(&map)), "r"(x0), "r"(y0), "r"(plane), "r"(smem_u32(bar))
        : "memory");
}

// Producer warp: a box of eight channels from plane `plane` on, of rows from y0
// and columns from x0 on, into a raw slot by one tensor copy (zeros outside the
// planes); the slot's barrier counts the 32 lanes.  (One bulk copy per channel and
// row of 512 bytes measured 100 cycles a copy: 751 us for 1.1 GB, copies alone.)
__device__ __forceinline__ void load_slot(const CUtensorMap& map, int plane, int y0, int x0, int box_floats, float* slot,
                                          uint64_t* bar) {
    if ((threadIdx.x & 31) == 0) {
        mbar_expect_tx(bar, static_cast<uint32_t>(box_floats) * 4u);
        tensor_copy(map, x0, y0, plane, slot, bar);
    } else {
        mbar_arrive(bar);
    }
    __syncwarp();
}

// converter thread t of nt, rows off 16-byte boundaries: nch channels, rows y0 ..
// y0 + rows - 1 and columns x0 .. x0 + cols - 1 into L2 (of the band after this one)
__device__ __forceinline__ void prefetch_planes(const float* src, int H, int W, int plane, int nch, int y0, int rows,
                                                int x0, int cols, int t, int nt) {
    const int r0 = max(0, -y0), r1 = min(rows, H - y0), c0 = max(0, -x0), c1 = min(cols, W - x0);
    const bool whole = c1 - c0 == W;                           // a channel's rows are one run
    const int runs = whole ? 1 : r1 - r0, lines = ((whole ? (r1 - r0) * W : c1 - c0) + 31) / 32;
    for (int k = t; k < nch * runs * lines; k += nt) {
        const int c = k / (runs * lines), m = k - c * (runs * lines), r = m / lines, l = m - r * lines;
        const float* p = src + (static_cast<int64_t>(plane + c) * H + y0 + r0 + r) * W + x0 + c0 + 32 * l;
        asm volatile("prefetch.global.L2 [%0];" ::"l"(p));
    }
}

// converter thread t of nt: a band's pixels from memory, as 16-byte groups of 8
// channels, zero outside the image.  (Rows off 16-byte boundaries: all warps' plain
// loads over all channels at once.  Taken through the raw slots by one warp's
// 4-byte copies, the gradients of 64 images of 32 -> 32 channels, 64 x 30, took
// 341 us, so 42.)
template <bool kBf16>
__device__ __forceinline__ void stage_planes(const Band& g, const BandAt& o, const float* __restrict__ x, int groups,
                                             uint4* dst, int xpix, int npix, int t, int nt) {
    const int64_t hw = static_cast<int64_t>(g.H) * g.W;
    const float* img = x + static_cast<int64_t>(o.img) * g.C * hw;
#pragma unroll 4
    for (int k = t; k < groups * npix; k += nt) {
        const int p = k / npix, i = k - p * npix;
        const int r = div_wp(g, i), cc = i - r * g.Wp;
        const int iy = o.y0 - 1 + r, ix = o.x0 - 1 + cc;
        const bool in = r < o.rows + 2 && cc < g.Ws + 2 && iy >= 0 && iy < g.H && ix >= 0 && ix < g.W;
        const float* q = img + (in ? 8 * p * hw + static_cast<int64_t>(iy) * g.W + ix : 0);
        const int nch = g.C - 8 * p;
        float v[8];
#pragma unroll
        for (int e = 0; e < 8; ++e) v[e] = in && e < nch ? __ldg(q + e * hw) : 0.f;
        dst[p * xpix + i] = make_uint4(pack2<kBf16>(v[0], v[1]), pack2<kBf16>(v[2], v[3]), pack2<kBf16>(v[4], v[5]),
                                       pack2<kBf16>(v[6], v[7]));
    }
}

// The same from a tensor copy's slot, whose rows and columns outside the image
// are zeros already: what is left of the bounds (the pitch's padding, and column
// -1 of a slot that holds whole rows) is the same in every band, so the slot
// offset of each of the thread's pixels is kept in registers (-1: zero).
// kMask: the slot holds pre-activations, and from float poff0 on the gradient of
// their ReLU + 2x2 mean (R / 2 + 2 rows from image row y0 / 2 - 1 on; whole rows,
// y0 even): the pixel is y > 0 ? dp / 4 : 0, k_relu_pool_bwd's value.
template <int kIt, bool kMask = false>
struct Pixels {
    int off[kIt], poff[kMask ? kIt : 1];
    __device__ __forceinline__ Pixels(const Band& g, int npix, int t, int nt, int poff0 = 0) {
        const int sx = g.nseg == 1 ? -1 : 3;               // slot column of staged column 0
#pragma unroll
        for (int k = 0; k < kIt; ++k) {
            const int i = t + k * nt;
            const int r = div_wp(g, i), cc = i - r * g.Wp;
            const bool in = i < npix && r < g.R + 2 && cc < g.Ws + 2 && cc + sx >= 0 && cc + sx < g.rp;
            off[k] = in ? r * g.rp + sx + cc : -1;
            if (kMask) poff[k] = poff0 + ((r + 1) >> 1) * (g.rp / 2) + ((sx + cc) >> 1);
        }
    }
    template <bool kBf16, bool kAll>
    __device__ __forceinline__ void stage(const float* raw, int rawp, int prawp, int nch, uint4* dst, int npix, int t,
                                          int nt) const {
#pragma unroll
        for (int k = 0; k < kIt; ++k) {
            const int i = t + k * nt;
            if (i >= npix) break;
            float v[8];
#pragma unroll
            for (int e = 0; e < 8; ++e) {
                const bool in = off[k] >= 0 && (kAll || e < nch);
                v[e] = in ? raw[off[k] + e * rawp] : 0.f;
                if (kMask) {
                    const float d = in ? raw[poff[k] + e * prawp] : 0.f;
                    v[e] = v[e] > 0.f ? 0.25f * d : 0.f;
                }
            }
            dst[i] = make_uint4(pack2<kBf16>(v[0], v[1]), pack2<kBf16>(v[2], v[3]), pack2<kBf16>(v[4], v[5]),
                                pack2<kBf16>(v[6], v[7]));
        }
    }
};

// the raw ring's place in the sequence of slots
struct Ring {
    int slot = 0;
    uint32_t use = 0;
    __device__ __forceinline__ void next(int slots) {
        if (++slot == slots) {
            slot = 0;
            ++use;
        }
    }
};

// ---------------------------------------------------------------- convolution
// Implicit GEMM: M = 128 staged pixels, N = the output channels, K = 3 x 3 taps
// x the input channels (chunks of 8, an even number of chunks).  W >= 128: a
// tile is 128 columns of a row (with ReLU + 2x2 mean fused a vertical pair of
// them, two accumulators); W < 128: 128 consecutive pixels of the staged pitch,
// whose padding columns are computed and not written.  Tile t's accumulator is
// drained by one of two sets of four warps (each warp its 32 TMEM lanes =
// pixels, + bias, coalesced along x) while the next tiles' MMAs run.
constexpr int kCEpi = 8, kCConv = 8;                       // epilogue and converter warps
constexpr int kCThreads = 32 * (kCEpi + kCConv + 2);
constexpr int kBandPix = 1024;                             // most pixels of a band (of more than two rows)
constexpr int kCPix = 7;                                   // staged pixels a converter thread: 1024 + 2 (256 + 4) of them

struct ConvGeom {
    Band b;
    int cout;
    int cin8, cin8r;   // channel chunks of 8, even (chunks past cin8r are zero)
    int xpix;          // pixels per chunk of a staged block
    int pool, wide;    // wide: W >= 128; pool: 1 = ReLU + mean only, 2 = beside the pre-activations
    int slots, nd;     // raw slots, accumulators
    int poff, prawp;   // kMask: floats from a slot to its pooled gradient, floats per channel of that
    uint32_t slotb, xbytes, off_x, off_b, smem;
    int tmem_cols;
};

struct ConvBars {
    uint64_t full[kMaxSlots], empty[kMaxSlots], sfull[2], sempty[2], dfull[4], dempty[4], drain;
    uint32_t tmem;
    int abort;
    float bias[128];
};

__device__ __forceinline__ int conv_tiles(const ConvGeom& g, const BandAt& o) {
    if (g.wide) return (g.pool ? o.rows / 2 : o.rows) * (g.b.Ws / kCM);
    return (o.rows * g.b.Wp + kCM - 1) / kCM;
}

__device__ __forceinline__ uint32_t uniform(uint32_t v) { return __shfl_sync(0xffffffffu, v, 0); }
__device__ __forceinline__ uint64_t uniform64(uint64_t v) { return __shfl_sync(0xffffffffu, v, 0); }

// a tile's MMAs: nine taps x kKs steps of 16 channels
template <int kKs>
__device__ __forceinline__ void conv_mmas(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc, int Wp, int xpix,
                                          int cout) {
    d = uniform(d);
    a = uniform64(a);
#pragma unroll
    for (int tap = 0; tap < 9; ++tap)
#pragma unroll
        for (int ks = 0; ks < kKs; ++ks)
            mma_f16_warp(d, a + static_cast<uint64_t>(tap / 3 * Wp + tap % 3 + 2 * ks * xpix),
                         b + static_cast<uint64_t>((2 * kKs * tap + 2 * ks) * cout), idesc, tap > 0 || ks > 0 ? 1u : 0u);
}

// kMask (the data gradient through ReLU + 2x2 mean): xmap is of the
// pre-activations, pmap of the pooled gradient, their product with the mask is
// formed while it is packed (32 x 128 x 128 at 128 images: 89 + 108 -> 124 us when it
// was made so; the three layers' data gradients of a training step take 182).
template <bool kBf16, bool kMask, bool kDirect>
__global__ void __launch_bounds__(kCThreads, 1)
    k_conv3x3_tc(const __grid_constant__ CUtensorMap xmap, const __grid_constant__ CUtensorMap pmap, const float* __restrict__ x, const float* __restrict__ w, const float* __restrict__ bias,
                 float* __restrict__ y, float* __restrict__ pooled, const ConvGeom g, int* status) {
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    __shared__ ConvBars S;
    uint8_t* base = smem_raw + align_up_smem(smem_raw, 1024);
    uint8_t* X = base + g.off_x;                         // two blocks [cin8][xpix][16 B]
    uint8_t* B = base + g.off_b;                         // [9 taps][cin8][cout][16 B]
    const int tid = threadIdx.x, lane = tid & 31;
    const int warp = __shfl_sync(0xffffffffu, tid >> 5, 0);          // uniform: the roles are warps
    const uint32_t b_chunk = static_cast<uint32_t>(g.cout) * 16;
    const int64_t hw = static_cast<int64_t>(g.b.H) * g.b.W;
    const int U = g.pool ? 2 : 1;                        // accumulators per tile

    if (tid == 0) {
        for (int i = 0; i < g.slots; ++i) {
            mbar_init(&S.full[i], 32);
            mbar_init(&S.empty[i], kCConv);
        }
        for (int i = 0; i < 2; ++i) {
            mbar_init(&S.sfull[i], kCConv);
            mbar_init(&S.sempty[i], 1);
        }
        for (int i = 0; i < g.nd; ++i) {
            mbar_init(&S.dfull[i], 1);
            mbar_init(&S.dempty[i], 4);
        }
        mbar_init(&S.drain, 1);
        S.abort = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&S.tmem)),
                     "r"(g.tmem_cols)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    for (int co = tid; co < g.cout; co += kCThreads) S.bias[co] = bias != nullptr ? bias[co] : 0.f;
    // weights: B[tap][c8][co] = 8 values of channels 8 c8 .. 8 c8 + 7 (zero past cin).
    // Where they fit in the L1 that the shared memory leaves, a thread gathers the
    // eight values of an operand row 36 bytes apart; else they are read along memory
    // (24 -> 128 channels, two rows of 128: 29 us a call gathered, 17 so; with
    // little shared memory, 16 x 16: 13.5 gathered, 15.3 so).
    if (static_cast<uint32_t>(9 * g.b.C * g.cout * 4) + g.smem <= 240 * 1024) {
        for (int i = tid; i < 9 * g.cin8 * g.cout; i += kCThreads) {
            const int kb = i / g.cout, co = i - kb * g.cout;
            const int tap = kb / g.cin8, c8 = kb - tap * g.cin8;
            float v[8];
#pragma unroll
            for (int e = 0; e < 8; ++e) {
                const int c = 8 * c8 + e;
                v[e] = c < g.b.C ? w[(static_cast<int64_t>(co) * g.b.C + c) * 9 + tap] : 0.f;
            }
            *reinterpret_cast<uint4*>(B + static_cast<uint32_t>(kb) * b_chunk + co * 16) =
                make_uint4(pack2<kBf16>(v[0], v[1]), pack2<kBf16>(v[2], v[3]), pack2<kBf16>(v[4], v[5]),
                           pack2<kBf16>(v[6], v[7]));
        }
    } else {
        const auto at = [&](int tap, int c, int co) {
            return reinterpret_cast<uint16_t*>(B + static_cast<uint32_t>(tap * g.cin8 + c / 8) * b_chunk + co * 16 + c % 8 * 2);
        };
        const int per_co = 9 * g.b.C;
#pragma unroll 8
        for (int i = tid; i < g.cout * per_co; i += kCThreads) {
            const int co = i / per_co, k = i - co * per_co, c = k / 9;
            *at(k - 9 * c, c, co) = static_cast<uint16_t>(pack2<kBf16>(w[i], 0.f));
        }
        for (int i = tid; i < 9 * (8 * g.cin8 - g.b.C) * g.cout; i += kCThreads) {
            const int k = i / g.cout, co = i - k * g.cout;
            *at(k % 9, g.b.C + k / 9, co) = 0;
        }
    }
    // the padding chunk of both staged blocks (never rewritten)
    if (g.cin8 > g.cin8r)
        for (int i = tid; i < 2 * g.xpix; i += kCThreads) {
            const int bb = i / g.xpix;
            reinterpret_cast<uint4*>(X + bb * g.xbytes)[g.cin8r * g.xpix + i - bb * g.xpix] = make_uint4(0, 0, 0, 0);
        }
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = __shfl_sync(0xffffffffu, S.tmem, 0);

    if (warp == kCEpi + kCConv) {
        // ---- producer
        Ring k;
        bool ok = !kDirect;                                // else nothing goes through the slots
        for (int64_t u = blockIdx.x; u < g.b.n_units && ok; u += gridDim.x) {
            const BandAt o = band_at(g.b, u);
            for (int c8 = 0; c8 < g.cin8r; ++c8, k.next(g.slots)) {
                if (k.use > 0 && !(ok = role_wait(&S.empty[k.slot], (k.use - 1) & 1u, &S.abort, status))) break;
                float* slot = reinterpret_cast<float*>(base + k.slot * g.slotb);
                if (kMask) {
                    const int plane = o.img * g.b.C + 8 * c8, nc = min(8, g.b.C);
                    if (lane == 0) {
                        mbar_expect_tx(&S.full[k.slot], static_cast<uint32_t>(nc * (g.b.rawp + g.prawp)) * 4u);
                        tensor_copy(xmap, 0, o.y0 - 1, plane, slot, &S.full[k.slot]);
                        tensor_copy(pmap, 0, o.y0 / 2 - 1, plane, slot + g.poff, &S.full[k.slot]);
                    } else {
                        mbar_arrive(&S.full[k.slot]);
                    }
                    __syncwarp();
                } else {
                    load_slot(xmap, o.img * g.b.C + 8 * c8, o.y0 - 1, slot_x0(g.b, o), min(8, g.b.C) * g.b.rawp, slot,
                              &S.full[k.slot]);
                }
            }
        }
        // no copy may be in flight when the block ends
        for (int i = 0; i < g.slots; ++i) {
            const uint32_t n = k.use + (i < k.slot ? 1u : 0u);            // copies into slot i
            if (n > 0) mbar_wait_bounded(&S.full[i], (n - 1) & 1u, status);
        }
    } else if (warp == kCEpi + kCConv + 1) {
        // ---- MMA issue
        const uint32_t idesc = mma_idesc_f16(kCM, g.cout) | (kBf16 ? kIdescBf16 : 0u);
        const uint32_t lbo = static_cast<uint32_t>(g.xpix) * 16;
        const int spr = g.b.Ws / kCM;                                     // tiles a row (wide)
        const uint64_t db0 = smem_desc(B, b_chunk, 128);
        uint32_t j = 0, d = 0, use = 0;
        bool ok = true;
        for (int64_t u = blockIdx.x; u < g.b.n_units && ok; u += gridDim.x, ++j) {
            const BandAt o = band_at(g.b, u);
            const int nt = conv_tiles(g, o);
            const uint32_t b = j & 1u;
            ok = role_wait(&S.sfull[b], (j >> 1) & 1u, &S.abort, status);
            if (!ok) break;
            const uint64_t da0 = uniform64(smem_desc(X + b * g.xbytes, lbo, 128));
            for (int t = 0; t < nt; ++t) {
                if (use > 0 && !(ok = role_wait(&S.dempty[d], (use - 1) & 1u, &S.abort, status))) break;
                tc_fence_after();
                const int pix = g.wide ? U * (t / spr) * g.b.Wp + kCM * (t % spr) : kCM * t;
                for (int h = 0; h < U; ++h) {
                    const uint64_t dah = da0 + static_cast<uint64_t>(pix + h * g.b.Wp);       // 16-byte units: pixels
                    if (g.cin8 == 2)
                        conv_mmas<1>(tmem + (d * U + h) * g.cout, dah, db0, idesc, g.b.Wp, g.xpix, g.cout);
                    else
                        conv_mmas<2>(tmem + (d * U + h) * g.cout, dah, db0, idesc, g.b.Wp, g.xpix, g.cout);
                }
                mma_commit_warp(&S.dfull[d]);
                if (++d == static_cast<uint32_t>(g.nd)) {
                    d = 0;
                    ++use;
                }
            }
            mma_commit_warp(&S.sempty[b]);
        }
        // every MMA this CTA issued has completed before its TMEM is released
        mma_commit_warp(&S.drain);
        mbar_wait_bounded(&S.drain, 0, status);
        __syncwarp();
    } else if (warp >= kCEpi) {
        // ---- converters
        const int t = tid - 32 * kCEpi;
        const Pixels<kDirect ? 1 : kCPix, kMask> px(g.b, (g.b.R + 2) * g.b.Wp, t, 32 * kCConv, g.poff);
        Ring k;
        uint32_t j = 0;
        bool ok = true;
        for (int64_t u = blockIdx.x; u < g.b.n_units && ok; u += gridDim.x, ++j) {
            const BandAt o = band_at(g.b, u);
            const uint32_t b = j & 1u;
            // the MMAs of the band two before have read block b
            if (j >= 2 && !(ok = role_wait(&S.sempty[b], ((j >> 1) - 1) & 1u, &S.abort, status))) break;
            const int npix = (o.rows + 2) * g.b.Wp;
            if (kDirect) {
                if (u + gridDim.x < g.b.n_units) {
                    const BandAt q = band_at(g.b, u + gridDim.x);
                    prefetch_planes(x, g.b.H, g.b.W, q.img * g.b.C, g.b.C, q.y0 - 1, g.b.R + 2, slot_x0(g.b, q), g.b.rp,
                                    t, 32 * kCConv);
                }
                stage_planes<kBf16>(g.b, o, x, g.cin8r, reinterpret_cast<uint4*>(X + b * g.xbytes), g.xpix, npix, t,
                                    32 * kCConv);
            }
            for (int c8 = 0; !kDirect && c8 < g.cin8r; ++c8, k.next(g.slots)) {
                ok = role_wait(&S.full[k.slot], k.use & 1u, &S.abort, status);
                if (!ok) break;
                const float* raw = reinterpret_cast<const float*>(base + k.slot * g.slotb);
                uint4* dst = reinterpret_cast<uint4*>(X + b * g.xbytes) + c8 * g.xpix;
                const int nch = min(8, g.b.C - 8 * c8);
                if (nch == 8)
                    px.template stage<kBf16, true>(raw, g.b.rawp, g.prawp, 8, dst, npix, t, 32 * kCConv);
                else
                    px.template stage<kBf16, false>(raw, g.b.rawp, g.prawp, nch, dst, npix, t, 32 * kCConv);
                __syncwarp();
                if (lane == 0) mbar_arrive(&S.empty[k.slot]);
            }
            if (!ok) break;
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            __syncwarp();
            if (lane == 0) mbar_arrive(&S.sfull[b]);
        }
    } else {
        // ---- epilogue: set e drains tiles e, e + 2, ...
        const uint32_t e = static_cast<uint32_t>(warp) >> 2;
        const int quarter = warp & 3;
        const int m = 32 * quarter + lane;
        const int spr = g.b.Ws / kCM;
        uint32_t T = 0;
        bool ok = true;
        for (int64_t u = blockIdx.x; u < g.b.n_units && ok; u += gridDim.x) {
            const BandAt o = band_at(g.b, u);
            const int nt = conv_tiles(g, o);
            for (int t = 0; t < nt; ++t, ++T) {
                if ((T & 1u) != e) continue;
                const uint32_t d = T % static_cast<uint32_t>(g.nd), use = T / static_cast<uint32_t>(g.nd);
                ok = role_wait(&S.dfull[d], use & 1u, &S.abort, status);
                if (!ok) break;
                tc_fence_after();
                const uint32_t taddr =
                    tmem + (static_cast<uint32_t>(32 * quarter) << 16) + d * static_cast<uint32_t>(U * g.cout);
                int r, ox;
                if (g.wide) {
                    r = U * (t / spr);
                    ox = o.x0 + kCM * (t % spr) + m;
                } else {
                    r = div_wp(g.b, kCM * t + m);
                    ox = kCM * t + m - r * g.b.Wp;
                }
                if (!g.pool) {
                    const bool in = r < o.rows && ox < g.b.W;
                    float* yo = y + static_cast<int64_t>(o.img) * g.cout * hw + static_cast<int64_t>(o.y0 + r) * g.b.W + ox;
                    for (int c0 = 0; c0 < g.cout; c0 += 32) {
                        float v[32];
                        tmem_ld32(taddr + static_cast<uint32_t>(c0), v);
                        if (in) {
#pragma unroll
                            for (int i = 0; i < 32; ++i) {
                                *yo = v[i] + S.bias[c0 + i];
                                yo += hw;
                            }
                        }
                    }
                } else {
                    // rows r (accumulator 0) and r + 1 (accumulator 1); lanes m, m + 1
                    // are the two columns.  Per pair of channels a lane swaps values
                    // with its neighbour and writes one mean: the even lane the first
                    // channel's, the odd lane the second's.  Alone, the mean sums
                    // columns first (one swap); beside the pre-activations it is
                    // k_relu_pool's, rows first, bit for bit (a backward pass and
                    // later layers see the same values as from the two kernels).
                    const int Ho = g.b.H / 2, Wo = g.b.W / 2;
                    const int64_t pw = static_cast<int64_t>(Ho) * Wo;
                    const int odd = lane & 1;
                    float* po = pooled + static_cast<int64_t>(o.img) * g.cout * pw +
                                static_cast<int64_t>((o.y0 + r) / 2) * Wo + ox / 2 + odd * pw;
                    float* yo = y + static_cast<int64_t>(o.img) * g.cout * hw + static_cast<int64_t>(o.y0 + r) * g.b.W + ox;
                    for (int c0 = 0; c0 < g.cout; c0 += 32) {
                        float v0[32], v1[32];
                        tmem_ld32(taddr + static_cast<uint32_t>(c0), v0);
                        tmem_ld32(taddr + static_cast<uint32_t>(g.cout + c0), v1);
                        if (g.pool == 1) {
#pragma unroll
                            for (int i = 0; i < 32; i += 2) {
                                const float b0 = S.bias[c0 + i], b1 = S.bias[c0 + i + 1];
                                const float t0 = fmaxf(v0[i] + b0, 0.f) + fmaxf(v1[i] + b0, 0.f);
                                const float t1 = fmaxf(v0[i + 1] + b1, 0.f) + fmaxf(v1[i + 1] + b1, 0.f);
                                const float other = __shfl_xor_sync(0xffffffffu, odd ? t0 : t1, 1);
                                *po = 0.25f * ((odd ? t1 : t0) + other);
                                po += 2 * pw;
                            }
                        } else {
#pragma unroll
                            for (int i = 0; i < 32; i += 2) {
                                float a[2][2];                         // [channel][row]
#pragma unroll
                                for (int e = 0; e < 2; ++e) {
                                    const float bb = S.bias[c0 + i + e];
                                    const float p0 = v0[i + e] + bb, p1 = v1[i + e] + bb;
                                    yo[0] = p0;
                                    yo[g.b.W] = p1;
                                    yo += hw;
                                    a[e][0] = fmaxf(p0, 0.f);
                                    a[e][1] = fmaxf(p1, 0.f);
                                }
                                const float s0 = __shfl_xor_sync(0xffffffffu, odd ? a[0][0] : a[1][0], 1);
                                const float s1 = __shfl_xor_sync(0xffffffffu, odd ? a[0][1] : a[1][1], 1);
                                *po = 0.25f * (((odd ? a[1][0] : a[0][0]) + s0) + ((odd ? a[1][1] : a[0][1]) + s1));
                                po += 2 * pw;
                            }
                        }
                    }
                }
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(&S.dempty[d]);
            }
        }
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    if (warp == 0)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(g.tmem_cols)
                     : "memory");
}

// ---------------------------------------------------------------- weight gradient
// dw[k][c][ty][tx] = sum over the images and output pixels (oy, ox) of
//   dy[k](oy, ox) * x[c](oy + ty - 1, ox + tx - 1)          (x zero outside the image)
// as nine GEMMs that contract over pixels: M = the output channels, 64 rows or 128
// (the MMA reads all M rows of A from shared memory, whatever their use: 32
// channels at M = 128 took 233 us at 32 x 128 x 128, 188 at M = 64 then; rows past cout
// read in-bounds data of the following chunks into accumulator rows that are
// never read), N = the input channels rounded up to
// 16, K = 16 pixels per MMA; BF16 operands (gradients span float32's exponent
// range), float32 accumulation.  x is staged as above (the MN-major B operand);
// dy on the same pitch pixel-contiguous ([8-pixel chunk][output channel][8
// pixels x 2 B], the K-major A operand) with zeros past each row's pixels.  The
// nine accumulators (9 x N TMEM columns) stay in TMEM over all the CTA's bands.
// The converters also sum each channel of dy (float32, before its rounding) for
// the bias gradient.  Each CTA then writes its partial sums, which
// k_sum_partials adds in an order that does not depend on timing.
constexpr int kWConv = 14;                                 // converter warps (2 ..)
constexpr int kWThreads = 32 * (kWConv + 2);
constexpr int kWPix = 4, kWDy = 5;                         // per converter thread: staged pixels, 32-pixel steps of dy

struct WgradGeom {
    Band b;
    int K, M;            // output channels, MMA M (64 or 128)
    int Q;               // pixels per band (R Wp rounded up to 32)
    int N;               // MMA N: C rounded up to 16
    int cgr, kg;         // channel groups of 8: of x (loaded), of dy
    int xpix;            // staged input pixels per channel group (Q + 2 Wp + 3, rounded up to 8)
    int rpd, rawd;       // raw slot of dy: floats per row, per channel
    int dvec;            // dy's rows on 16-byte boundaries
    int poff;            // floats from a slot of dy (pooled: of y) to dp
    int apitch;          // bytes from a staged 8-pixel chunk of dy to the next
    int fold;            // C <= 8: the column taps are one MMA (N = 32, its groups of 8 columns the one channel
                         // group seen 0 .. 3 pixels on, the last not read): 3 MMAs a K step, not 9
    int acc_cols;        // TMEM columns of the accumulators (9 N, or 3 x 32 folded)
    int slots;           // raw slots
    uint32_t slotb, xbytes, stage, smem;
    int tmem_cols;
};

struct WgradBars {
    uint64_t full[kMaxSlots], empty[kMaxSlots], sfull[2], sempty[2], drain;
    uint32_t tmem;
    int abort, drained;
    float bias[kWConv][128];
};

// kPool: dy is not in memory: dmap is then of the pre-activations y and pmap of the
// gradient dp of their ReLU + 2x2 mean, and dy = y > 0 ? dp / 4 : 0 is formed while
// it is packed (k_relu_pool_bwd's value).  That saves writing and reading dy, of
// the first layer's 1.1 GB each at 128 images: 339 + 307 us -> 297 us.
template <bool kPool, bool kDirect>
__global__ void __launch_bounds__(kWThreads, 1)
    k_conv3x3_wgrad_tc(const __grid_constant__ CUtensorMap xmap, const __grid_constant__ CUtensorMap dmap,
                       const __grid_constant__ CUtensorMap pmap, const float* __restrict__ x, const float* __restrict__ dy, float* __restrict__ part,
                       const WgradGeom g, int* status) {
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    __shared__ WgradBars S;
    uint8_t* base = smem_raw + align_up_smem(smem_raw, 1024);    // raw slots, then the staged blocks
    uint8_t* stages = base + g.slots * g.slotb;
    const bool xdirect = kDirect && !g.b.vec, ddirect = kDirect && !kPool && !g.dvec;
    const int tid = threadIdx.x, lane = tid & 31;
    const int warp = __shfl_sync(0xffffffffu, tid >> 5, 0);          // uniform: the roles are warps

    if (tid == 0) {
        for (int i = 0; i < g.slots; ++i) {
            mbar_init(&S.full[i], 32);
            mbar_init(&S.empty[i], kWConv);
        }
        for (int i = 0; i < 2; ++i) {
            mbar_init(&S.sfull[i], kWConv);
            mbar_init(&S.sempty[i], 1);
        }
        mbar_init(&S.drain, 1);
        S.abort = 0;
        S.drained = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&S.tmem)),
                     "r"(g.tmem_cols)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    for (int i = tid; i < kWConv * 128; i += kWThreads) (&S.bias[0][0])[i] = 0.f;
    {   // a channel group that no slot fills stays zero (the last one of an odd count)
        const int zg = g.cgr, ng = g.fold ? 0 : g.N / 8 - zg;
        for (int i = tid; i < 2 * ng * g.xpix; i += kWThreads) {
            const int bb = i / (ng * g.xpix), p = i - bb * ng * g.xpix;
            *reinterpret_cast<uint4*>(stages + bb * g.stage + (static_cast<uint32_t>(zg) * g.xpix + p) * 16u) =
                make_uint4(0, 0, 0, 0);
        }
    }
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = __shfl_sync(0xffffffffu, S.tmem, 0);

    if (warp == 0) {
        // ---- producer: per band the channel groups of x, then of dy (of those that
        // go through the slots)
        Ring k;
        bool ok = true;
        for (int64_t u = blockIdx.x; u < g.b.n_units && ok; u += gridDim.x) {
            const BandAt o = band_at(g.b, u);
            for (int p = xdirect ? g.cgr : 0; p < g.cgr + (ddirect ? 0 : g.kg); ++p, k.next(g.slots)) {
                if (k.use > 0 && !(ok = role_wait(&S.empty[k.slot], (k.use - 1) & 1u, &S.abort, status))) break;
                float* slot = reinterpret_cast<float*>(base + k.slot * g.slotb);
                if (p < g.cgr)
                    load_slot(xmap, o.img * g.b.C + 8 * p, o.y0 - 1, slot_x0(g.b, o), min(8, g.b.C) * g.b.rawp, slot,
                              &S.full[k.slot]);
                else if (kPool) {
                    const int plane = o.img * g.K + 8 * (p - g.cgr), nd = min(8, g.K);
                    if (lane == 0) {
                        mbar_expect_tx(&S.full[k.slot], static_cast<uint32_t>(nd * (g.rawd + g.rawd / 4)) * 4u);
                        tensor_copy(dmap, o.x0, o.y0, plane, slot, &S.full[k.slot]);
                        tensor_copy(pmap, o.x0 / 2, o.y0 / 2, plane, slot + g.poff, &S.full[k.slot]);
                    } else {
                        mbar_arrive(&S.full[k.slot]);
                    }
                    __syncwarp();
                } else
                    load_slot(dmap, o.img * g.K + 8 * (p - g.cgr), o.y0, o.x0, min(8, g.K) * g.rawd, slot,
                              &S.full[k.slot]);
            }
        }
        // no copy may be in flight when the block ends
        for (int i = 0; i < g.slots; ++i) {
            const uint32_t n = k.use + (i < k.slot ? 1u : 0u);            // copies into slot i
            if (n > 0) mbar_wait_bounded(&S.full[i], (n - 1) & 1u, status);
        }
    } else if (warp == 1) {
        // ---- MMA issue: BF16 A (K-major) and B (MN-major: bit 16)
        const uint32_t idesc = mma_idesc_f16(g.M, g.fold ? 32 : g.N) | kIdescBf16 | (1u << 16);
        const uint32_t lbo_a = static_cast<uint32_t>(g.apitch);         // next 8-pixel chunk of dy
        // B is MN-major without swizzle: there the descriptor's leading offset is
        // the step along K (the next 8 pixels, 128 bytes on) and the stride offset
        // the step along N (the next channel group; folded the next pixel)
        const uint32_t sbo_b = g.fold ? 16u : static_cast<uint32_t>(g.xpix) * 16;
        const int ksteps = g.Q / 16;
        uint32_t j = 0;
        bool ok = true;
        for (int64_t u = blockIdx.x; u < g.b.n_units; u += gridDim.x, ++j) {
            const uint32_t b = j & 1u, use = j >> 1;
            ok = role_wait(&S.sfull[b], use & 1u, &S.abort, status);
            if (!ok) break;
            tc_fence_after();
            const uint8_t* Xs = stages + b * g.stage;
            uint64_t da = uniform64(smem_desc(Xs + g.xbytes, lbo_a, 128));
            // descriptor addresses are in 16-byte units: one unit per staged pixel of x
            uint64_t db = uniform64(smem_desc(Xs, 128, sbo_b));
            // K steps outer, taps inner: consecutive MMAs go to different
            // accumulators, so no MMA waits for the previous one's sum
            for (int ks = 0; ks < ksteps; ++ks, da += 2u * lbo_a >> 4, db += 16) {
                const uint32_t acc = (j > 0 || ks > 0) ? 1u : 0u;
                if (g.fold) {
                    // one MMA per row tap: N = the column taps x 8 channels
#pragma unroll
                    for (int ty = 0; ty < 3; ++ty)
                        mma_f16_warp(tmem + static_cast<uint32_t>(32 * ty), da,
                                     db + static_cast<uint64_t>(ty * g.b.Wp), idesc, acc);
                } else {
#pragma unroll
                    for (int tap = 0; tap < 9; ++tap) {
                        const int ty = tap / 3, tx = tap - 3 * ty;
                        mma_f16_warp(tmem + static_cast<uint32_t>(tap * g.N), da,
                                     db + static_cast<uint64_t>(ty * g.b.Wp + tx), idesc, acc);
                    }
                }
            }
            mma_commit_warp(&S.sempty[b]);
        }
        // every MMA this CTA issued has completed before the accumulators are read
        mma_commit_warp(&S.drain);
        const bool drained = mbar_wait_bounded(&S.drain, 0, status) && ok;
        if (lane == 0) S.drained = drained ? 1 : 0;
        __syncwarp();
    } else {
        // ---- converters
        const int cw = warp - 2;
        const Pixels<kWPix> px(g.b, g.xpix, tid - 64, 32 * kWConv);
        // dy: a warp takes four channels of a group x 8 half chunks (of 4 pixels, one
        // row: the pitch is a multiple of 4) at a time, so that the eight lanes of a
        // 16-byte load phase read one channel's 128 bytes; the staged chunks lie 32
        // bytes off a multiple of 128, so that the stores of a phase (two channels x
        // four chunks) fall on different banks
        const int kk = 4 * (cw & 1) + (lane >> 3);             // this lane's channel of the group
        int doff[kWDy], poff[kWDy];
#pragma unroll
        for (int i = 0; i < kWDy; ++i) {
            const int q = 32 * ((cw >> 1) + kWConv / 2 * i) + 4 * (lane & 7);
            const int r = div_wp(g.b, q), ox = q - r * g.b.Wp;
            doff[i] = r < g.b.R && ox < g.rpd ? kk * g.rawd + r * g.rpd + ox : -1;
            poff[i] = g.poff + (kk * g.rawd / 2 + (r >> 1) * g.rpd + ox) / 2;
        }
        const uint32_t d0 = static_cast<uint32_t>((4 * (cw >> 1) + ((lane & 7) >> 1)) * g.apitch + kk * 16 + (lane & 1) * 8);
        Ring k;
        uint32_t j = 0;
        bool ok = true;
        for (int64_t u = blockIdx.x; u < g.b.n_units && ok; u += gridDim.x, ++j) {
            const BandAt o = band_at(g.b, u);
            const uint32_t b = j & 1u, use = j >> 1;
            uint8_t* Xs = stages + b * g.stage;
            uint8_t* Ds = Xs + g.xbytes;
            // the MMAs of the band staged in block b before have read it
            if (use > 0 && !(ok = role_wait(&S.sempty[b], (use - 1) & 1u, &S.abort, status))) break;
            const int t = tid - 64, nt = 32 * kWConv;
            if (kDirect && u + gridDim.x < g.b.n_units) {
                const BandAt q = band_at(g.b, u + gridDim.x);
                if (xdirect)
                    prefetch_planes(x, g.b.H, g.b.W, q.img * g.b.C, g.b.C, q.y0 - 1, g.b.R + 2, slot_x0(g.b, q), g.b.rp,
                                    t, nt);
                if (ddirect) prefetch_planes(dy, g.b.H, g.b.W, q.img * g.K, g.K, q.y0, g.b.R, q.x0, g.rpd, t, nt);
            }
            if (xdirect) stage_planes<true>(g.b, o, x, g.cgr, reinterpret_cast<uint4*>(Xs), g.xpix, g.xpix, t, nt);
            if (ddirect) {
                const int64_t hw = static_cast<int64_t>(g.b.H) * g.b.W;
                // dy from memory: the groups and steps of the band in one sequence
                const int steps = g.Q / 32;
                const float* img = dy + static_cast<int64_t>(o.img) * g.K * hw;
#pragma unroll 8
                for (int it = cw >> 1; it < g.kg * steps; it += kWConv / 2) {
                    const int p = it / steps, hb = it - p * steps, ch = 8 * p + kk;
                    const int q = 32 * hb + 4 * (lane & 7);
                    const int r = div_wp(g.b, q), ox = q - r * g.b.Wp;
                    const int nx = ch < g.K && r < o.rows ? min(g.b.Ws - ox, g.b.W - o.x0 - ox) : 0;
                    const float* pr = img + (nx > 0 ? ch * hw + static_cast<int64_t>(o.y0 + r) * g.b.W + o.x0 + ox : 0);
                    const float4 f = make_float4(nx > 0 ? __ldg(pr) : 0.f, nx > 1 ? __ldg(pr + 1) : 0.f,
                                                 nx > 2 ? __ldg(pr + 2) : 0.f, nx > 3 ? __ldg(pr + 3) : 0.f);
                    *reinterpret_cast<uint2*>(Ds + (4 * hb + ((lane & 7) >> 1)) * g.apitch + kk * 16 + (lane & 1) * 8 + p * 128) =
                        make_uint2(pack_bf2(f.x, f.y), pack_bf2(f.z, f.w));
                    float sum = (f.x + f.y) + (f.z + f.w);
                    sum += __shfl_xor_sync(0xffffffffu, sum, 1);
                    sum += __shfl_xor_sync(0xffffffffu, sum, 2);
                    sum += __shfl_xor_sync(0xffffffffu, sum, 4);
                    if ((lane & 7) == 0) S.bias[cw][ch] += sum;
                }
            }
            for (int p = xdirect ? g.cgr : 0; p < g.cgr + (ddirect ? 0 : g.kg); ++p, k.next(g.slots)) {
                ok = role_wait(&S.full[k.slot], k.use & 1u, &S.abort, status);
                if (!ok) break;
                const float* raw = reinterpret_cast<const float*>(base + k.slot * g.slotb);
                if (p < g.cgr) {
                    uint4* dst = reinterpret_cast<uint4*>(Xs) + p * g.xpix;
                    const int nch = min(8, g.b.C - 8 * p);
                    if (nch == 8)
                        px.template stage<true, true>(raw, g.b.rawp, 0, 8, dst, g.xpix, t, nt);
                    else
                        px.template stage<true, false>(raw, g.b.rawp, 0, nch, dst, g.xpix, t, nt);
                } else {
                    const int ch = 8 * (p - g.cgr) + kk;
                    uint8_t* dd = Ds + d0 + (p - g.cgr) * 128;
                    float sum = 0.f;
#pragma unroll
                    for (int i = 0; i < kWDy; ++i) {
                        const int hb = (cw >> 1) + kWConv / 2 * i;
                        if (hb >= g.Q / 32) break;
                        float4 f = make_float4(0.f, 0.f, 0.f, 0.f);
                        if (doff[i] >= 0 && ch < g.K) {
                            f = *reinterpret_cast<const float4*>(raw + doff[i]);
                            if (kPool) {
                                const float2 d = *reinterpret_cast<const float2*>(raw + poff[i]);
                                const float g0 = 0.25f * d.x, g1 = 0.25f * d.y;
                                f = make_float4(f.x > 0.f ? g0 : 0.f, f.y > 0.f ? g0 : 0.f, f.z > 0.f ? g1 : 0.f,
                                                f.w > 0.f ? g1 : 0.f);
                            }
                        }
                        *reinterpret_cast<uint2*>(dd + i * (2 * kWConv * g.apitch)) =
                            make_uint2(pack_bf2(f.x, f.y), pack_bf2(f.z, f.w));
                        sum += (f.x + f.y) + (f.z + f.w);
                    }
                    sum += __shfl_xor_sync(0xffffffffu, sum, 1);
                    sum += __shfl_xor_sync(0xffffffffu, sum, 2);
                    sum += __shfl_xor_sync(0xffffffffu, sum, 4);
                    if ((lane & 7) == 0) S.bias[cw][ch] += sum;
                }
                __syncwarp();
                if (lane == 0) mbar_arrive(&S.empty[k.slot]);
            }
            if (!ok) break;
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            __syncwarp();
            if (lane == 0) mbar_arrive(&S.sfull[b]);
        }
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    if (S.drained) {
        // warp w reads TMEM lanes 32 (w % 4) .. + 31 (output channels; M = 64: 16 a
        // warp, in its lanes 0 .. 15), 32-column chunks w / 4, w / 4 + 4, ...; column
        // t * N + c is tap t of channel c
        const int quarter = warp & 3, rows = g.M / 4;
        const int k = lane < rows ? rows * quarter + lane : g.K;
        const int cols = g.acc_cols;
        const int64_t kc9 = static_cast<int64_t>(g.K) * g.b.C * 9;
        float* mine = part + blockIdx.x * (kc9 + g.K);
        if (rows * quarter < g.K) {
            for (int ch = warp >> 2; 32 * ch < cols; ch += kWThreads / 128) {
                float v[32];
                tmem_ld32(tmem + (static_cast<uint32_t>(32 * quarter) << 16) + static_cast<uint32_t>(32 * ch), v);
                if (k < g.K) {
                    float* pk = mine + static_cast<int64_t>(k) * g.b.C * 9;
#pragma unroll
                    for (int i = 0; i < 32; ++i) {
                        const int col = 32 * ch + i;
                        int t, c;
                        if (g.fold) {              // column 32 ty + 8 tx + c
                            const int tx = (col & 31) >> 3;
                            t = tx < 3 ? 3 * (col >> 5) + tx : -1;
                            c = col & 7;
                        } else {
                            t = col / g.N;
                            c = col - t * g.N;
                        }
                        if (col < cols && t >= 0 && c < g.b.C) pk[c * 9 + t] = v[i];
                    }
                }
            }
        }
        for (int c = tid; c < g.K; c += kWThreads) {
            float s = 0.f;
            for (int i = 0; i < kWConv; ++i) s += S.bias[i][c];
            mine[kc9 + c] = s;
        }
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    if (warp == 0)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(g.tmem_cols)
                     : "memory");
}

// sums over the nb partials (rows of n0 + n1 values) of each value, the first n0
// into out0, the rest into out1: a CTA takes 32 values, its eight warps every
// eighth partial each, then adds the warps' sums in order
__global__ void __launch_bounds__(256) k_sum_partials(const float* __restrict__ part, int nb, int64_t n0, int n1,
                                                      float* __restrict__ out0, float* __restrict__ out1) {
    __shared__ float red[8][32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int64_t n = n0 + n1, i = blockIdx.x * 32ll + lane;
    float s = 0.f;
    if (i < n) {
#pragma unroll 4
        for (int b = warp; b < nb; b += 8) s += part[b * n + i];
    }
    red[warp][lane] = s;
    __syncthreads();
    if (warp == 0 && i < n) {
        for (int w = 1; w < 8; ++w) s += red[w][lane];
        if (i < n0) out0[i] = s;
        else out1[i - n0] = s;
    }
}

// ---------------------------------------------------------------- geometries
// bands of R rows and segments of Ws columns of n images (rows on 16-byte
// boundaries where vec)
void band_set(Band& b, int n, int R, int Ws) {
    b.R = R;
    b.Ws = Ws;
    b.nseg = (b.W + Ws - 1) / Ws;
    b.nband = (b.H + R - 1) / R;
    b.Wp = (Ws + 2 + 3) / 4 * 4;
    b.rp = b.nseg == 1 ? b.W : Ws + 8;
    b.rawp = (R + 2) * b.rp;
    b.wp_inv = static_cast<uint32_t>(((1ull << 32) + b.Wp - 1) / b.Wp);
    b.n_units = static_cast<int64_t>(n) * b.nband * b.nseg;
}

// Rows per band: as many as leave three raw slots beside the staged blocks (the
// halo rows are read and packed once per band), up to 1024 pixels (more brings
// nothing), and few enough that every SM has two bands where the work allows, but
// no fewer than `least` staged pixels (the convolution of narrow images: half an
// MMA tile; 16 images of 32 channels, 64 x 2: 12.7 us, 74 in bands of three rows).
// Columns: whole rows where a band of two of them fits, else the longest
// segment for which it does.  fits(R, Ws) lays the geometry out.
template <class Fits>
bool band_choose(Band& b, int n, int unit, int col_unit, int least, int num_sms, Fits fits) {
    for (int nseg = 1;; ++nseg) {
        const int Ws = (b.W + nseg - 1) / nseg;
        const int Wu = nseg == 1 ? b.W : (Ws + col_unit - 1) / col_unit * col_unit;
        const int need = b.H < 2 ? 1 : 2;
        if (fits(need, Wu)) {
            int R = need;
            for (int r = need + unit; r <= b.H && r * (Wu + 4) <= kBandPix; r += unit) {
                if (static_cast<int64_t>(n) * ((b.H + r - 1) / r) * nseg < 2ll * num_sms && R * (Wu + 4) >= least) break;
                if (!fits(r, Wu)) break;
                R = r;
            }
            const int nband = (b.H + R - 1) / R;
            R = (b.H + nband - 1) / nband;         // bands of one height
            R = (R + unit - 1) / unit * unit;
            return fits(R < need ? need : R, Wu);
        }
        if (Wu <= col_unit) return fits(1, Wu);
    }
}

int tmem_columns(int cols) { return cols <= 32 ? 32 : (cols <= 64 ? 64 : (cols <= 128 ? 128 : (cols <= 256 ? 256 : 512))); }

bool conv_geom(int n, int cin, int cout, int H, int W, int pool, bool mask, int num_sms, ConvGeom& g) {
    g = ConvGeom{};
    g.b.C = cin;
    g.b.H = H;
    g.b.W = W;
    g.cout = cout;
    g.pool = pool;
    g.wide = W >= kCM ? 1 : 0;
    g.cin8r = (cin + 7) / 8;
    g.cin8 = (g.cin8r + 1) / 2 * 2;
    const int cols = (pool ? 2 : 1) * cout;
    g.nd = 512 / cols < 4 ? 512 / cols : 4;
    g.tmem_cols = tmem_columns(g.nd * cols);
    const uint32_t bbytes = 9u * static_cast<uint32_t>(g.cin8) * static_cast<uint32_t>(cout) * 16u;
    return band_choose(g.b, n, pool || mask ? 2 : 1, kCM, g.wide ? 0 : kCM / 2, num_sms, [&](int R, int Ws) {
        if (g.wide && (Ws % kCM != 0 || W % Ws != 0)) return false;
        if (mask && (Ws != W || R % 2 != 0)) return false;
        band_set(g.b, n, R, Ws);
        // (a converter thread takes kCPix pixels of a block)
        if (g.b.rp > kMaxBox || (R + 2) * g.b.Wp > kCPix * 32 * kCConv) return false;
        // staged pixels; W < 128: the last tile reads on past them (rows that are not written)
        const int last = (R * g.b.Wp + kCM - 1) / kCM * kCM + 2 * g.b.Wp + 2;
        g.xpix = g.wide ? (R + 2) * g.b.Wp : (last > (R + 2) * g.b.Wp ? last : (R + 2) * g.b.Wp);
        g.xbytes = static_cast<uint32_t>(g.cin8) * g.xpix * 16u;
        const int nc = cin < 8 ? cin : 8;
        g.poff = (nc * g.b.rawp + 31) / 32 * 32;
        g.prawp = mask ? (R / 2 + 2) * (g.b.rp / 2) : 0;
        g.slotb = (static_cast<uint32_t>(mask ? g.poff + nc * g.prawp : nc * g.b.rawp) * 4u + 127u) & ~127u;
        const uint32_t rest = 2u * g.xbytes + bbytes + 1024u;
        if (rest + 3u * g.slotb + sizeof(ConvBars) > kSmemBudget) return false;
        const uint32_t s = (kSmemBudget - static_cast<uint32_t>(sizeof(ConvBars)) - rest) / g.slotb;
        g.slots = s < kMaxSlots ? static_cast<int>(s) : kMaxSlots;
        g.off_x = g.slots * g.slotb;
        g.off_b = g.off_x + 2u * g.xbytes;
        g.smem = g.off_b + bbytes + 1024u;
        return true;
    });
}

bool wgrad_geom(int n, int cin, int cout, int H, int W, bool pool, int num_sms, WgradGeom& g) {
    if (pool && (H % 2 != 0 || W % 8 != 0)) return false;
    if (n < 1 || cin < 1 || cin > 48 || cout < 1 || cout > 128 || H < 1 || W < 1) return false;
    g = WgradGeom{};
    g.b.C = cin;
    g.b.H = H;
    g.b.W = W;
    g.K = cout;
    g.M = cout <= 64 ? 64 : 128;
    g.N = (cin + 15) / 16 * 16;
    g.cgr = (cin + 7) / 8;
    g.kg = (cout + 7) / 8;
    g.fold = cin <= 8 ? 1 : 0;
    g.apitch = 128 * g.kg + 32;
    g.acc_cols = g.fold ? 3 * 32 : 9 * g.N;
    g.tmem_cols = tmem_columns(g.acc_cols < 128 ? 128 : g.acc_cols);
    const uint32_t xgroups = g.fold ? 1 : g.N / 8;          // staged channel groups of x
    auto stage_bytes = [&](int R, int Wp, int& Q, int& xpix, uint32_t& xbytes) {
        Q = (R * Wp + 31) / 32 * 32;
        xpix = (Q + 2 * Wp + 3 + 7) / 8 * 8;
        xbytes = xgroups * static_cast<uint32_t>(xpix) * 16u;
        return (xbytes + static_cast<uint32_t>(Q / 8 * g.apitch) + 127u) & ~127u;
    };
    {   // the widths taken: those of which one staged row of whole width fits (the rest go to the CUDA cores)
        if (W > (1 << 16)) return false;
        const uint32_t Wp = (W + 2 + 3) / 4 * 4, Q = (Wp + 31) / 32 * 32, xpix = (Q + 2 * Wp + 2 + 7) / 8 * 8;
        if ((((g.fold ? 4 : xgroups) * xpix * 16u + Q * g.kg * 16u + 127u) & ~127u) + 3072u > 227u * 1024u) return false;
    }
    return band_choose(g.b, n, pool ? 2 : 1, pool ? 8 : 4, 0, num_sms, [&](int R, int Ws) {
        if (pool && R % 2 != 0) return false;
        band_set(g.b, n, R, Ws);
        if (g.b.rp > kMaxBox) return false;
        g.stage = stage_bytes(R, g.b.Wp, g.Q, g.xpix, g.xbytes);
        // (a converter thread takes kWPix pixels of x and kWDy steps of dy; rows of
        // three pixels are staged eight apart, and 146 of them would be 37 steps of 32)
        if (g.xpix > kWPix * 32 * kWConv || g.Q > kWDy * 32 * (kWConv / 2)) return false;
        g.rpd = g.b.nseg == 1 ? W : Ws;
        g.rawd = R * g.rpd;
        const int xc = cin < 8 ? cin : 8, dc = cout < 8 ? cout : 8;
        g.poff = (dc * g.rawd + 31) / 32 * 32;
        const int df = pool ? g.poff + dc * g.rawd / 4 : dc * g.rawd;
        const int f = xc * g.b.rawp > df ? xc * g.b.rawp : df;
        g.slotb = (static_cast<uint32_t>(f) * 4u + 127u) & ~127u;
        // the blocks, 2 KB past the last one for the unused A rows, 1 KB alignment
        const uint32_t rest = 2u * g.stage + 2048u + 1024u;
        if (rest + 3u * g.slotb + sizeof(WgradBars) > kSmemBudget) return false;
        const uint32_t s = (kSmemBudget - static_cast<uint32_t>(sizeof(WgradBars)) - rest) / g.slotb;
        g.slots = s < kMaxSlots ? static_cast<int>(s) : kMaxSlots;
        g.smem = rest + static_cast<uint32_t>(g.slots) * g.slotb;
        return true;
    });
}

int units_grid(const Band& b, int num_sms) {
    return static_cast<int>(b.n_units < num_sms ? b.n_units : num_sms);
}

// n planes of H x W floats, boxes of bw x bh x bn
bool encode_planes(CUtensorMap* map, const float* p, int64_t n, int H, int W, int bw, int bh, int bn) {
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
    const cuuint64_t dims[3] = {static_cast<cuuint64_t>(W), static_cast<cuuint64_t>(H), static_cast<cuuint64_t>(n)};
    const cuuint64_t strides[2] = {static_cast<cuuint64_t>(W) * 4, static_cast<cuuint64_t>(W) * H * 4};
    const cuuint32_t box[3] = {static_cast<cuuint32_t>(bw), static_cast<cuuint32_t>(bh), static_cast<cuuint32_t>(bn)};
    const cuuint32_t estr[3] = {1, 1, 1};
    return encode(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 3, const_cast<float*>(p), dims, strides, box, estr,
                  CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                  CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// rows that tensor copies can take
int aligned_rows(const void* p, int W) { return W % 4 == 0 && reinterpret_cast<uintptr_t>(p) % 16 == 0 ? 1 : 0; }
}  // namespace

bool conv3x3_tc_supported(int cin, int cout, int H, int W) {
    if (cin < 1 || cin > 32 || cout < 32 || cout > 128 || cout % 32 != 0) return false;
    if (W >= kCM) return W % kCM == 0;
    return W >= 1 && kCM % W == 0 && H % (kCM / W) == 0;
}

bool conv3x3_tc_pool_supported(int cin, int cout, int H, int W) {
    return conv3x3_tc_supported(cin, cout, H, W) && W >= kCM && H % 2 == 0;
}

bool conv3x3_tc_mask_supported(int cin, int cout, int H, int W) {
    return conv3x3_tc_supported(cin, cout, H, W) && H % 2 == 0 && W % 8 == 0 && W <= kCM;
}

cudaError_t launch_conv3x3_tc(const float* x, const float* dp, const float* w, const float* b, float* y, float* pooled,
                              int n, int cin, int cout, int H, int W, int num_sms, int* status, cudaStream_t st,
                              bool bf16) {
    if (!conv3x3_tc_supported(cin, cout, H, W)) return cudaErrorInvalidValue;
    const int pool = pooled == nullptr ? 0 : (y == nullptr ? 1 : 2);
    const bool mask = dp != nullptr;
    if (pool && !conv3x3_tc_pool_supported(cin, cout, H, W)) return cudaErrorInvalidValue;
    if (mask && (!bf16 || !conv3x3_tc_mask_supported(cin, cout, H, W))) return cudaErrorInvalidValue;
    ConvGeom g;
    if (!conv_geom(n, cin, cout, H, W, pool, mask, num_sms, g)) return cudaErrorInvalidValue;
    if (g.b.n_units == 0) return cudaSuccess;
    CUtensorMap xmap{}, pmap{};
    const int nc = cin < 8 ? cin : 8;
    const int64_t planes = static_cast<int64_t>(n) * cin;
    g.b.vec = aligned_rows(x, W) && encode_planes(&xmap, x, planes, H, W, g.b.rp, g.b.R + 2, nc);
    if (mask && !(g.b.vec && aligned_rows(dp, W / 2) &&
                  encode_planes(&pmap, dp, planes, H / 2, W / 2, g.b.rp / 2, g.b.R / 2 + 2, nc)))
        return cudaErrorInvalidValue;
    const auto kern = mask      ? k_conv3x3_tc<true, true, false>
                      : g.b.vec ? (bf16 ? k_conv3x3_tc<true, false, false> : k_conv3x3_tc<false, false, false>)
                                : (bf16 ? k_conv3x3_tc<true, false, true> : k_conv3x3_tc<false, false, true>);
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(g.smem));
    if (e != cudaSuccess) return e;
    kern<<<units_grid(g.b, num_sms), kCThreads, g.smem, st>>>(xmap, pmap, x, w, b, y, pooled, g, status);
    return cudaGetLastError();
}

size_t conv3x3_wgrad_tc_partials(int n, int cin, int cout, int H, int W, bool pool, int num_sms) {
    WgradGeom g;
    if (!wgrad_geom(n, cin, cout, H, W, pool, num_sms, g)) return 0;
    return static_cast<size_t>(units_grid(g.b, num_sms)) * (static_cast<size_t>(cout) * cin * 9 + cout);
}

cudaError_t launch_conv3x3_wgrad_tc(const float* x, const float* dy, const float* dp, float* dw, float* db, int n,
                                    int cin, int cout, int H, int W, float* partials, int num_sms, int* status,
                                    cudaStream_t st) {
    WgradGeom g;
    const bool pool = dp != nullptr;
    if (!wgrad_geom(n, cin, cout, H, W, pool, num_sms, g) || partials == nullptr) return cudaErrorInvalidValue;
    const int dc = cout < 8 ? cout : 8;
    const int64_t planes = static_cast<int64_t>(n) * cout;
    CUtensorMap xmap{}, dmap{}, pmap{};
    g.b.vec = aligned_rows(x, W) &&
              encode_planes(&xmap, x, static_cast<int64_t>(n) * cin, H, W, g.b.rp, g.b.R + 2, cin < 8 ? cin : 8);
    g.dvec = aligned_rows(dy, W) && encode_planes(&dmap, dy, planes, H, W, g.rpd, g.b.R, dc);
    if (pool && !(g.dvec && aligned_rows(dp, W / 2) &&
                  encode_planes(&pmap, dp, planes, H / 2, W / 2, g.rpd / 2, g.b.R / 2, dc)))
        return cudaErrorInvalidValue;
    const auto kern = pool ? (g.b.vec ? k_conv3x3_wgrad_tc<true, false> : k_conv3x3_wgrad_tc<true, true>)
                           : (g.b.vec && g.dvec ? k_conv3x3_wgrad_tc<false, false> : k_conv3x3_wgrad_tc<false, true>);
    const int grid = units_grid(g.b, num_sms);
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(g.smem));
    if (e != cudaSuccess) return e;
    kern<<<grid, kWThreads, g.smem, st>>>(xmap, dmap, pmap, x, dy, partials, g, status);
    e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    const int64_t kc9 = static_cast<int64_t>(cout) * cin * 9;
    k_sum_partials<<<static_cast<unsigned int>((kc9 + cout + 31) / 32), 256, 0, st>>>(partials, grid, kc9, cout, dw, db);
    return cudaGetLastError();
}

cudaError_t set_wait_test_cnn(unsigned long long limit_ns, int starve, cudaStream_t st) {
    return set_wait_test_here(limit_ns, starve, st);
}

}  // namespace octgb

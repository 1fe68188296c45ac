// Output encoding of the legacy TIFF (octrecon/io/tiff_writer.py:53-71) on the
// device.
//
//   k_requant_lut   legacy double quantisation (tiff_writer.py:62-64): the
//                   re-quantised code of a plane depends only on its first
//                   code b = db_to_bits(db, plane clim), so one 65 536-entry
//                   table per plane, built in float64 with the reference's
//                   operations (bits_to_db then db_to_bits, :33-45), replaces
//                   the per-voxel float64 work; k_apply_lut maps the codes.
//   k_packbits_rows PackBits (TIFF compression 32773) of every image row on
//                   its own (TIFF 6.0 packs rows separately), one warp per
//                   row, little-endian sample bytes: a run of >= 3 equal bytes
//                   (up to 128) becomes a repeat packet, everything else
//                   literal packets of up to 128 bytes.  Each row is written to
//                   its own worst-case slot; its byte count goes to sizes[].
//   k_row_offsets, k_pack_rows   the rows' bytes without gaps, so that only
//                   they cross to the host.
#include <cuda_runtime.h>
#include <stdint.h>

#include "octgb_internal.h"

namespace octgb {
namespace {

__device__ __forceinline__ uint16_t quantise_f64(double x, double c1, double span) {
    if (isnan(x)) return 0;
    const double v = (x - c1) / span * 65534.0;
    double r = floor(fabs(v) + 0.5);
    if (v < 0) r = -r;
    if (!(r > 0.0)) r = 0.0;
    if (r > 65535.0) r = 65535.0;
    const unsigned int u = static_cast<unsigned int>(r) + 1u;
    return static_cast<uint16_t>(u > 65535u ? 65535u : u);
}

__global__ void k_requant_lut(double p1, double p2, double c1, double c2, uint16_t* __restrict__ lut) {
    const int b = blockIdx.x * blockDim.x + threadIdx.x;
    if (b >= 65536) return;
    if (b == 0) {
        lut[0] = 0;                                       // bits_to_db(0) is NaN -> 0
        return;
    }
    const double db = static_cast<double>(b - 1) * (p2 - p1) / 65534.0 + p1;
    lut[b] = quantise_f64(db, c1, c2 - c1);
}

__global__ void k_apply_lut(uint16_t* __restrict__ bits, int64_t n, const uint16_t* __restrict__ lut) {
    for (int64_t i = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x; i < n;
         i += static_cast<int64_t>(gridDim.x) * blockDim.x)
        bits[i] = lut[bits[i]];
}

// The row is a chain of packets, so a warp walks it packet by packet: lane l
// holds the bytes i + 4 l .. + 3 of the 128 that a packet starting at i can
// cover, and one ballot finds where the run or the literal ends.  Bound by the
// latency of that chain (about 35 packets of 128 bytes a row of 1900 codes);
// 1767 such rows take 32 us, and one thread a row (14 CTAs) took 1183.
constexpr int kPackWarps = 4;
__global__ void __launch_bounds__(kPackWarps * 32) k_packbits_rows(const uint16_t* __restrict__ img, int rows,
                                                                   int cols, uint8_t* __restrict__ out, int slot,
                                                                   int* __restrict__ sizes) {
    const int r = blockIdx.x * kPackWarps + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (r >= rows) return;
    const uint8_t* row = reinterpret_cast<const uint8_t*>(img + static_cast<int64_t>(r) * cols);   // little-endian
    uint8_t* o = out + static_cast<int64_t>(r) * slot;
    const int n = 2 * cols;
    int w = 0;
    for (int i = 0; i < n;) {
        const int j0 = i + 4 * lane;
        // bytes j0 .. j0 + 5; past the row: distinct values that equal nothing
        int c[6];
#pragma unroll
        for (int e = 0; e < 4; ++e) c[e] = j0 + e < n ? __ldg(row + j0 + e) : 256 + e;
#pragma unroll
        for (int e = 4; e < 6; ++e) {
            c[e] = __shfl_down_sync(0xffffffffu, c[e - 4], 1);
            if (lane == 31) c[e] = j0 + e < n ? __ldg(row + j0 + e) : 260 + e;
        }
        // first place of the lane's four where the run of b[i] ends, and where three equal bytes start
        int ends = 4, three = 4;
#pragma unroll
        for (int e = 3; e >= 0; --e) {
            if (c[e] != c[e + 1]) ends = e;
            if (c[e] == c[e + 1] && c[e] == c[e + 2]) three = e;
        }
        const bool repeat = __shfl_sync(0xffffffffu, three, 0) == 0;
        const int mine = repeat ? ends : three;
        const unsigned int found = __ballot_sync(0xffffffffu, mine < 4);
        const int at = found ? __ffs(static_cast<int>(found)) - 1 : 0;
        const int first = 4 * at + __shfl_sync(0xffffffffu, mine, at);
        if (repeat) {
            const int run = found && first < 127 ? first + 1 : 128;
            if (lane == 0) {
                o[w] = static_cast<uint8_t>(1 - run);     // -(run - 1)
                o[w + 1] = static_cast<uint8_t>(c[0]);
            }
            w += 2;
            i += run;
        } else {
            const int left = n - i < 128 ? n - i : 128;
            const int len = found && first < left ? first : left;
            if (lane == 0) o[w] = static_cast<uint8_t>(len - 1);
#pragma unroll
            for (int e = 0; e < 4; ++e)
                if (4 * lane + e < len) o[w + 1 + 4 * lane + e] = static_cast<uint8_t>(c[e]);
            w += 1 + len;
            i += len;
        }
    }
    if (lane == 0) sizes[r] = w;
}

// offsets[r] = bytes of the rows before r (offsets[rows]: of all); one CTA
__global__ void __launch_bounds__(1024) k_row_offsets(const int* __restrict__ sizes, int rows,
                                                      long long* __restrict__ offsets) {
    __shared__ long long tot[32];
    const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
    long long base = 0;
    for (int r0 = 0; r0 < rows; r0 += 1024) {
        const int r = r0 + tid;
        const long long v = r < rows ? sizes[r] : 0;
        long long t = v;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const long long u = __shfl_up_sync(0xffffffffu, t, o);
            if (lane >= o) t += u;
        }
        if (lane == 31) tot[w] = t;
        __syncthreads();
        long long before = 0, all = 0;
        for (int k = 0; k < 32; ++k) {
            if (k < w) before += tot[k];
            all += tot[k];
        }
        if (r < rows) offsets[r] = base + before + t - v;
        base += all;
        __syncthreads();
    }
    if (tid == 0) offsets[rows] = base;
}

// one CTA a row: whole destination words, each from two source words
__global__ void __launch_bounds__(128) k_pack_rows(const uint8_t* __restrict__ slots, int slot,
                                                   const int* __restrict__ sizes,
                                                   const long long* __restrict__ offsets, uint8_t* __restrict__ out) {
    const int r = blockIdx.x, n = sizes[r];
    const uint8_t* src = slots + static_cast<int64_t>(r) * slot;      // slot: a multiple of 4, with 4 bytes to spare
    uint8_t* dst = out + offsets[r];
    const int head = static_cast<int>((4 - (reinterpret_cast<uintptr_t>(dst) & 3u)) & 3u);
    const int h = head < n ? head : n, words = (n - h) / 4;
    const uint32_t* s4 = reinterpret_cast<const uint32_t*>(src);
    uint32_t* d4 = reinterpret_cast<uint32_t*>(dst + h);
    for (int i = threadIdx.x; i < words; i += 128) d4[i] = __funnelshift_r(s4[i], s4[i + 1], 8 * h);
    if (static_cast<int>(threadIdx.x) < h) dst[threadIdx.x] = src[threadIdx.x];
    const int tail = h + 4 * words;
    if (static_cast<int>(threadIdx.x) < n - tail) dst[tail + threadIdx.x] = src[tail + threadIdx.x];
}

int grid_n(int64_t n) {
    int64_t g = (n + 255) / 256;
    return static_cast<int>(g > 65536 ? 65536 : (g < 1 ? 1 : g));
}

}  // namespace

cudaError_t launch_requant(uint16_t* bits, int64_t n, double p1, double p2, double c1, double c2, uint16_t* lut,
                           cudaStream_t st) {
    k_requant_lut<<<65536 / 256, 256, 0, st>>>(p1, p2, c1, c2, lut);
    k_apply_lut<<<grid_n(n), 256, 0, st>>>(bits, n, lut);
    return cudaGetLastError();
}

// the worst case of a row (whole words, and one that k_pack_rows may read past the last byte)
int packbits_slot(int cols) { return ((2 * cols + (2 * cols + 127) / 128 + 1 + 3) & ~3) + 4; }

cudaError_t launch_packbits(const uint16_t* img, int rows, int cols, uint8_t* slots, int* sizes, long long* offsets,
                            uint8_t* out, cudaStream_t st) {
    const int slot = packbits_slot(cols);
    k_packbits_rows<<<(rows + kPackWarps - 1) / kPackWarps, kPackWarps * 32, 0, st>>>(img, rows, cols, slots, slot,
                                                                                      sizes);
    if (out == nullptr) return cudaGetLastError();
    k_row_offsets<<<1, 1024, 0, st>>>(sizes, rows, offsets);
    k_pack_rows<<<rows, 128, 0, st>>>(slots, slot, sizes, offsets, out);
    return cudaGetLastError();
}

}  // namespace octgb

// Internal declarations shared by the octgb CUDA translation units.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

namespace octgb {

constexpr int kN = 2048;          // spectral samples per A-scan (FFT length)
constexpr int kHalf = kN / 2;     // depth bins kept (core/spectral.py:153, nz = N/2)
constexpr int kMaxTaps = 32;      // sinc taps supported
constexpr int kTail = 32;         // zero tail after each line so padded taps stay in bounds
constexpr int kSincThreads = 512; // threads of the banded sinc, four outputs each
// A-scans of one pass (lines kernel, transform) through the linearised lines'
// scratch: at most 600 per SM (712 MiB).  A pass costs its two kernels' ramps
// and tails (~12 us) and longer ones win although their lines go through DRAM:
// 324 000 A-scans stitched took 4043, 3685, 3479, 3356 and 3290 us with 24,
// 48, 96, 192 and 600 per SM.  set_geometry makes room for kFirstPass (228
// MiB: a first call of up to 29 184 A-scans allocates nothing), longer calls
// grow it; the allocation-free entry point has its own of kMinPass.  A device
// short of memory holds less of each, down to kLeastPass: the calls then take
// more passes.
constexpr int kMaxPass = 152 * 600, kFirstPass = 152 * 192, kMinPass = 152 * 24, kLeastPass = 152;
constexpr int kTwTable = 256 + 7 * 256;   // the transform's twiddles tw2, tw3

// device-side status word values
constexpr int kStatusOk = 0;
constexpr int kStatusTimeout = 1;

// What k_lines writes per A-scan: the real linearised line; that times the
// complex window (the fused pre-FFT operator); or that times a float64 window,
// rounded once to float32 (the scorer's input, (eq * hann).astype(complex64)
// with a window of ones).
enum LineMode : int { kModeReal = 0, kModeSpec = 1, kModeLinHann = 2 };
// What follows the transform: |X|, dB of a depth crop with its range
enum OutMode : int { kModeMag = 0, kModeDb = 1 };

constexpr int kBlk = 32;          // output rows / columns per stitch block
constexpr int kMaxSeg = 32;       // tiles per multi-tile launch

struct DevGeometry {
    // [2][U][kSincThreads] shifted weights of outputs 4t, 4t + 1 (4t + 2, 4t + 3) at window step u
    const float2* wsh;
    const int* s0;        // [kSincThreads] source window base of thread t
    int U;                // window width (14, 18, 22 or 26)
    const float2* win;    // [kN] complex64 window scaled by 1/kN (ifft normalisation)
    const float2* tw;     // [kTwTable] twiddles of the transform, rounded from float64
};

struct StitchDev;

// One tile of the batched form: its raw B-scans, its depth operator (a stitch
// plan with the identity lateral operator) and its dB output (A-scan major).
struct QueueTile {
    const void* raw;          // (B, interf, kN) device
    float* out;               // (B * nx, nz) float32 dB
    const StitchDev* plan;    // device pointer into the context's plan table
    int B, interf, apod, nx, nz;
    int apod_row0;            // first row of the tile in the apodisation-mean buffer
    unsigned int line0;       // first global A-scan of the tile
    int pad_;
};
constexpr int kMaxQueueTiles = 256;
// a batched tile's lateral weights stay inside groups of this many A-scans (the
// last group of a B-scan ends on its last A-scan)
constexpr int kLateral = 4;

// float64 form of the spectral stage (exact.cu)
struct ExactArgs {
    const void* raw;          // (B, interf, kN) device, uint16 or int16
    int B, interf, apod, nx;
    int64_t n_ascans;         // B * nx
    const int* apod_sum;      // (B, kN) integer sums of the apodisation lines (filled by launch_exact)
    const int* start;         // [kN] first source sample of each output
    const double* w;          // [taps][kN] float64 band weights, tap-major (padding 0)
    int taps;
    const double2* win;       // [kN] window / kN, float64 complex
    const double2* tw;        // [kN] exp(+2 pi i k / kN), float64
    float* mag;               // (n_ascans, kHalf) |X| rounded to float32
};
cudaError_t launch_exact(const ExactArgs& a, int dtype, int* sums, int num_sms, cudaStream_t st);

// the raw batches of the precision form's kernels
struct SpectralArgs {
    const void* raw;          // (B, interf, kN)
    int B, interf, apod, nx;  // nx = interf - apod
    int64_t n_ascans;         // B * nx
};

// The context's device allows `kernel` its shared memory; the attribute is set
// on the kernel's first launch through a context (bit `bit` of its `ready`), not
// on every one (~1 us of host time each).
template <typename Kernel>
inline cudaError_t kernel_ready(uint64_t* ready, int bit, Kernel kernel, size_t smem) {
    if (*ready >> bit & 1u) return cudaSuccess;
    const cudaError_t e =
        cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem));
    if (e == cudaSuccess) *ready |= uint64_t(1) << bit;
    return e;
}
// bits 0 .. 47: k_lines, 48 .. 54: k_disp_mag, 55 .. 62: k_lines with the exact background
constexpr int kReadyDisp = 48, kReadyExact = 55;

// lines.cu: A-scans [l0, l1) of n_seg raw batches of one shape, or of tiles of
// uneven size (qt), numbered segment by segment, B-scan by B-scan
struct LinesArgs {
    const void* seg[kMaxSeg]; // raw batches, each (B, interf, kN)
    int B, interf, apod, nx;  // nx = interf - apod
    const QueueTile* qt;      // null: the batches above
    int n_qt;
    unsigned int l0, l1;
    const float* apod_mean;   // float32 apodisation mean (exact: sums), a row per B-scan
    bool exact;               // integer raws: the exact background (kModeReal, no tiles)
    DevGeometry g;
    float* out;               // line l at (l - out_l0) kN (kModeSpec: complex)
    unsigned int out_l0;
    const double* hann;       // kModeLinHann: the float64 window (kN)
    const float* hann2;       // kModeLinHann: the window split hi (kN), lo (kN) in float32
    int* status;              // device status word
    uint64_t* ready;          // host: bits of the caller's context, see kernel_ready
};
// apodisation mean (exact: sums) of every B-scan (`rows` of them) into out
cudaError_t launch_apod_mean(const LinesArgs& a, int dtype, int rows, float* out, cudaStream_t st);
// launched dependent on the kernel before it in the stream (as launch_disp_mag's)
cudaError_t launch_lines(const LinesArgs& a, int dtype, int mode, int num_sms, cudaStream_t st);

// stitch.cu
struct StitchDev {
    // compact 2-tap depth operator: for output row zo, rows zr[zo] and zr[zo]+1 (relative to r0)
    const int* zr;            // [n_out_z], -1 = no contribution
    const float* wz0;         // [n_out_z]
    const float* wz1;         // [n_out_z]
    // compact 2-tap lateral operator: output column c0+cc takes A-scans xr[cc], xr[cc]+1
    const int* xr;            // [C], -1 = none
    const float* wx0;         // [C]
    const float* wx1;         // [C]
    const float* fz;          // [R] focus weight of rows r0..r1-1
    const int* shift;         // [n_y, n_tile_x] optical-path row shift, or null
    const int* lo;            // [n_y, n_tile_x] smallest valid r (incl.), or null
    const int* hi;            // [n_y, n_tile_x] largest valid r (incl.), or null
    // per output row: {zr (int bits), wz0, wz1, d = fma(F1, wz1, F0 wz0)} and
    // {F0 = fz[zr], F1 = fz[zr + 1] or 0 past the window} (batched form)
    const float4* zrow;
    const float2* zf;
    // per output column c0 + cc: {xr (int bits), wx0, wx1, the one A-scan with a
    // weight (int bits; -1: two or none)}
    const float4* xcol;
    int r0, R, c0, C, n_out_z, n_tile_x, n_rows;
};

struct TileList {
    int n;
    int id[kMaxSeg];
};

constexpr int kStitchRows = 64;   // default output rows per stitch block (x 32 columns; 32, 64 or 128)
constexpr int kSlotOpc = 1;       // optical-path correction on (patch of F follows the magnitudes')
constexpr int kSlotSingle = 2;    // every column of the block takes one A-scan of the tile
struct StitchSlot {               // one tile touching one output block
    int t;                        // index into the TileList
    int x_lo, xs;                 // A-scans read
    int r_lo, rs;                 // rows (relative to r0) read
    int off;                      // float offset of the patch in shared memory
    int kind;                     // kSlotOpc | kSlotSingle
    int rst;                      // patch stride per A-scan: rs + a zero row, made odd (distinct banks)
    int last;                     // last slot of a round (the patches of a round are staged together)
};
struct StitchTmaSlot {            // one tile touching one output block, staged by tensor copies
    const float4* zrow;           // the block's row parameters in the plan's tables
    const float2* zf;
    const float4* xcol;           // the block's column parameters
    int t;                        // index into the TileList
    int row0;                     // first magnitude row copied (a multiple of 4)
    int x_lo, r_lo;               // A-scan and row (relative to r0; row0 is r0 + r_lo) at the patch's origin
    int single;                   // every column of the block takes one A-scan of the tile
    int pad_;
};
struct StitchArgs {
    TileList tiles;
    const StitchSlot* slots;      // [blocks][tiles.n], the first slot_count[block] used
    const int* slot_count;
    int ns_round;                 // most slots of a round
    const StitchTmaSlot* tslots;  // null: slots; else the same blocks' slots for tensor copies,
    uint32_t patch_bytes, slot_bytes;   // each with slot_bytes of shared memory, the patch (padded) first:
    int pitch, box_lines;         // box_lines lines of `pitch` floats
    int tile_lines;               // lines of `mag` per tile,
    int64_t n_lines;              // and in all
    int* status;                  // device status word (bounded waits)
    uint32_t starve;              // self-test: bytes the first round's barrier expects beyond its copies
    const float* mag;             // tile t, frame f, A-scan x at t mag_tile_stride + (f n_tile_x + x) kHalf
    int64_t mag_tile_stride;
    int n_tile_x, f0, n_out_z, n_out_x;
    int cblk0;                    // first 32-column block
    // frame batch: all tiles, dB and clim
    float thr;
    float* db;                    // (B, n_out_z, n_out_x)
    unsigned int* plane_mm;       // [B][2] or null
    unsigned int* run_mm;         // [2] or null
    // row interface: one tile added to num / den (frames, n_out_z, n_out_x); null otherwise
    float *num, *den;
    const int* frame_y;           // frame of the optical-path correction, null: f0 + f
    int frame_offset;
};
cudaError_t launch_stitch(const StitchDev* plans_dev, const StitchArgs& a, size_t patch_smem_bytes, int n_cblk, int B,
                          int rows, cudaStream_t st);
// batched form: dB rows of the A-scans [l0, l1) of tiles of uneven size from
// their magnitudes (A-scan l at (l - l0) kHalf), with the running range
cudaError_t launch_resample(const QueueTile* qt, int n_qt, unsigned int l0, unsigned int l1, const float* mag,
                            float thr, unsigned int* run_mm, cudaStream_t st);
cudaError_t launch_finalise(const float* num, const float* den, int64_t n_per_plane, int n_planes, float thr,
                            float* db, unsigned int* plane_minmax, cudaStream_t st);
// quantisation: `table` is scratch of kQuantTable floats (the code thresholds of the clim)
constexpr int kQuantTable = 65537;
cudaError_t launch_quantise(const float* db, int64_t n, double c1, double c2, float* table, uint16_t* bits,
                            cudaStream_t st);
cudaError_t launch_quantise_dev(const float* db, int64_t n, const unsigned int* clim_mm, float* table,
                                uint16_t* bits, cudaStream_t st);
cudaError_t launch_minmax(const float* x, int64_t n, unsigned int* minmax, cudaStream_t st);
cudaError_t launch_minmax_init(unsigned int* minmax, int count, cudaStream_t st);

// dispersion scorer: A[(gi * nb + bi) * nx + x][k] = mean over repeats of
// |ifft(X line * phase[gi])|[k], k < N/2, for B-scans b0 .. b0 + nb - 1
struct DispArgs {
    const float* X;        // (B, rep, nx, kN) linearised, windowed, real
    const float2* phase;   // (n_beta, kN) exp(-i beta dk^2) / N
    const float2* tw;      // kTwTable twiddles
    float* A;              // (n_beta, nb, nx, kHalf), or null with zcol; dB rows of nz with mode kModeDb
    int mode;              // kModeMag, or kModeDb: 20 log10 |X| of depths [z0, z0 + nz) (rep = 1)
    int z0, nz;
    unsigned int* minmax;  // kModeDb: [2] ordered-uint range of the finite dB, may be null
    float* zcol;           // (n_beta, nb, nx, 256) depth-pooled sums of |X| (probe images), or null
    int z_keep;            // depths pooled into the 256 image rows
    int n_beta, nb, b0, nx, rep;
    int* status;           // where a wait that runs out is recorded
    uint64_t* ready;       // host: bits of the caller's context, see kernel_ready
};
cudaError_t launch_disp_mag(const DispArgs& a, int num_sms, cudaStream_t st);
// per segment (n_seg rows of nx x kHalf magnitudes): metric 1 top_percentile
// (top_k elements), 2 kurtosis, 3 entropy, 4 legacy_peak, depths >= z_min
cudaError_t launch_disp_metric(const float* A, int n_seg, int nx, int z_min, int metric, unsigned int top_k,
                               double* score, int num_sms, cudaStream_t st);
// n phase rows exp(-i beta dk2) / N (complex64 of the float64 value)
cudaError_t launch_phase(const double* betas, const double* dk2, int n, float2* phase, cudaStream_t st);
// median over x of every (frame, z) column of (n_frames, nx, nz) float32, as float64
cudaError_t launch_xmedian(const float* mag, int n_frames, int nx, int nz, int ignore_nan, int mean_mode,
                           double* out, cudaStream_t st);

// rare raw formats (prepare.cu): AScanBinning, frame-mean apodisation, repeats
struct PrepArgs {
    const void* raw;      // (B, n_lines, kN)
    int B, n_lines;
    int a_out;            // apodisation lines of the output (apod_size, or 1 for frame mean)
    int n_kept;           // scan lines of the output
    int n_scan, scan0;    // scan lines of a file and the first one
    int s0, left;         // AScanBinning: first kept column, window lines before the column
    int binning, mode, group;   // mode 0: apodisation lines, 1: frame mean over `group` files
};
cudaError_t launch_prepare(const PrepArgs& p, int dtype, float* frame_apod, float* out, cudaStream_t st);
cudaError_t launch_srr_decode(const uint16_t* src, int64_t src_file, int a0, int na, int s0, int lines_out, int n,
                              int n_files, int16_t* out, cudaStream_t st);
cudaError_t launch_avg_repeats(const float* mag, int n_frames, int nb, int size_x, int na, int nz, float* out,
                               cudaStream_t st);

// legacy TIFF encoding (encode.cu)
cudaError_t launch_requant(uint16_t* bits, int64_t n, double p1, double p2, double c1, double c2, uint16_t* lut,
                           cudaStream_t st);
int packbits_slot(int cols);
// slots: rows x packbits_slot(cols) bytes of scratch; offsets: rows + 1; out: the rows' bytes, one after the other
// (NULL: slots and sizes only, offsets not used)
cudaError_t launch_packbits(const uint16_t* img, int rows, int cols, uint8_t* slots, int* sizes, long long* offsets,
                            uint8_t* out, cudaStream_t st);

// precision form of float32 raws (precision.cu): tensor-core sinc
constexpr int kPM = 128;                 // A-scans per tile (MMA M)
constexpr int kPN = 64;                  // output samples per block (MMA N)
constexpr int kPKW = 96;                 // source window per block (6 K-steps of 16)
constexpr int kPChunks = kPKW / 8;       // 8-sample column chunks of a window
constexpr int kPBlocks = kN / kPN;       // output blocks per A-scan
}  // namespace octgb
#include <cuda.h>
#include <cuda_fp16.h>
#include <vector>
namespace octgb {
// apod64: B x kN of scratch
cudaError_t launch_prec_split(const SpectralArgs& a, double* apod64, __half* hi, __half* lo, float* mline,
                              int num_sms, cudaStream_t st);
cudaError_t launch_prec_sinc(const CUtensorMap& tm_hi, const CUtensorMap& tm_lo, const uint8_t* wtiles,
                             const int* kb, const float* mline, float* X, int64_t n_ascans, int* status, int num_sms,
                             cudaStream_t st);
bool encode_prec_map(CUtensorMap* map, const void* base, int64_t n_ascans);
// W tiles (per output block: hi then lo, canonical K-major no-swizzle, W x 64)
// and window starts kb; false when a block's band exceeds the window
bool build_prec_tiles(const int* start, const int* len, const float* wt, std::vector<uint16_t>& tiles,
                      std::vector<int>& kb);

// learned beta/focus estimator (cnn.cu)
cudaError_t launch_image_pool(const float* A, int n_probe, int nb, int nx, int z_keep, float* img, cudaStream_t st);
// the same images from k_disp_mag's depth-pooled column sums (n_probe, nb, nx, 256)
cudaError_t launch_image_cols(const float* zcol, int n_probe, int nb, int nx, int z_keep, float* img,
                              cudaStream_t st);
cudaError_t launch_image_norm(float* img, int n_images, int64_t per_image, cudaStream_t st);
// tensor-core 3x3 convolution (cnn_tc.cu): same contract as launch_conv3x3 for
// the shapes conv3x3_tc_supported accepts; FP16 operands (BF16 with bf16: the
// data gradient, whose values span float32's exponent range), float32
// accumulation (with pooled (n, cout, H/2, W/2): its ReLU + 2x2 mean, y may be
// NULL; with dp (n, cin, H/2, W/2) and bf16, on shapes of
// conv3x3_tc_mask_supported with x and dp 16-byte aligned: of the gradient of
// x's ReLU + 2x2 mean whose pooled gradient is dp)
bool conv3x3_tc_supported(int cin, int cout, int H, int W);
bool conv3x3_tc_pool_supported(int cin, int cout, int H, int W);
bool conv3x3_tc_mask_supported(int cin, int cout, int H, int W);
cudaError_t launch_conv3x3_tc(const float* x, const float* dp, const float* w, const float* b, float* y, float* pooled,
                              int n, int cin, int cout, int H, int W, int num_sms, int* status, cudaStream_t st, bool bf16 = false);
// weight and bias gradients of the 3x3 convolution (cnn_tc.cu; dw on the tensor
// cores with BF16 operands and float32 accumulation, db from dy in float32):
// dw (cout, cin, 3, 3) and db (cout) from x (n, cin, H, W) and dy (n, cout, H, W).
// With dp (n, cout, H/2, W/2; H even, W a multiple of 8, dy and dp 16-byte
// aligned) dy is the pre-activation of a ReLU + 2x2 mean whose gradient is dp.
// conv3x3_wgrad_tc_partials: the float count of the per-CTA partial sums the
// launch needs (0: shape not supported).
size_t conv3x3_wgrad_tc_partials(int n, int cin, int cout, int H, int W, bool pool, int num_sms);
cudaError_t launch_conv3x3_wgrad_tc(const float* x, const float* dy, const float* dp, float* dw, float* db, int n,
                                    int cin, int cout, int H, int W, float* partials, int num_sms, int* status,
                                    cudaStream_t st);
cudaError_t launch_conv3x3(const float* x, const float* w, const float* b, float* y, int Nn, int C, int K, int H,
                           int W, cudaStream_t st);
cudaError_t launch_flip_weights(const float* w, int K, int C, float* wf, cudaStream_t st);
cudaError_t launch_conv3x3_wgrad(const float* x, const float* dy, float* dw, int Nn, int C, int K, int H, int W,
                                 cudaStream_t st);
cudaError_t launch_relu_pool(const float* y, int64_t nk, int H, int W, float* p, cudaStream_t st);
cudaError_t launch_relu_pool_bwd(const float* dp, const float* y, int64_t nk, int H, int W, float* dy,
                                 cudaStream_t st);
cudaError_t launch_gemm(const float* A, int64_t sa0, int64_t sa1, const float* B, int64_t sb0, int64_t sb1, float* C,
                        int64_t ldc, int M, int N, int K, int accumulate, cudaStream_t st);
// split-K form (S slices of K, partial: S x M x N floats of scratch); gemm_splits picks S
int gemm_splits(int M, int N, int K, int num_sms);
cudaError_t launch_gemm_split(const float* A, int64_t sa0, int64_t sa1, const float* B, int64_t sb0, int64_t sb1,
                              float* C, int64_t ldc, int M, int N, int K, int accumulate, int S, float* partial,
                              cudaStream_t st);
cudaError_t launch_bias_relu(float* y, const float* b, int M, int N, float* out, cudaStream_t st);
// db[k] = sum over n and inner of g[n][k][inner]; part (Nn * K floats, optional)
// takes the plane sums of the two-pass form used when inner is a multiple of 4
cudaError_t launch_bias_grad(const float* g, int Nn, int K, int64_t inner, float* db, float* part, cudaStream_t st);
cudaError_t launch_relu_bwd(float* g, const float* pre, int64_t n, cudaStream_t st);
cudaError_t launch_mse(const float* pred, const float* t, int n, float* grad, double* loss, cudaStream_t st);
// one Adam step on up to kAdamMost tensors
constexpr int kAdamMost = 16;
struct AdamTensor {
    float* p;
    const float* g;
    float *m, *v;
    int64_t n;
};
struct AdamList {
    AdamTensor t[kAdamMost];
};
cudaError_t launch_adam(const AdamList& a, int count, float lr, float b1, float b2, float eps, float c1, float c2,
                        cudaStream_t st);

// ordered-uint encoding of float32 for atomic min/max
__host__ __device__ inline unsigned int f2ord(float f) {
#ifdef __CUDA_ARCH__
    unsigned int u = __float_as_uint(f);
#else
    unsigned int u;
    __builtin_memcpy(&u, &f, 4);
#endif
    return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}
__host__ __device__ inline float ord2f(unsigned int u) {
    unsigned int v = (u & 0x80000000u) ? (u & 0x7fffffffu) : ~u;
#ifdef __CUDA_ARCH__
    return __uint_as_float(v);
#else
    float f;
    __builtin_memcpy(&f, &v, 4);
    return f;
#endif
}

// the bounded waits' limit and self-test switch of each kernel file (see
// octgb_device.cuh); only octgb_selftest_wait_expiry calls these
cudaError_t set_wait_test_spectral(unsigned long long limit_ns, int starve, cudaStream_t st);
cudaError_t set_wait_test_precision(unsigned long long limit_ns, int starve, cudaStream_t st);
cudaError_t set_wait_test_stitch(unsigned long long limit_ns, cudaStream_t st);
cudaError_t set_wait_test_cnn(unsigned long long limit_ns, int starve, cudaStream_t st);

}  // namespace octgb

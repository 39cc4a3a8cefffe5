// Finite-cone footprint and accumulation of the collapsed-cone scatter image
// (citrus/scatter_solver/scatter_image.py:897-1135, 1234-1323).
//
// The footprint of direction k is a box blur of its single-ray image with a width of hbar_k W_k / pitch pixels along
// the channels and the rows, hbar_k the emission-weighted mean panel height (from the emission kernel's sums). The
// reference applies it as dense [N, N] overlap matrices in batched products (box_matrix, :952-1007); here each output
// pixel sums only the input pixels its window overlaps, with the same overlap weights
// B[c, j] = |[j, j + 1] n W_c| / |W_c|, W_c = [c + 1/2 - w/2, c + 1/2 + w/2] n [0, N], so the cost is O(N w) instead of
// O(N^2). The width is computed in the kernel from the height sums, so no host round trip sits between the emission
// and the blur.
#include <math.h>

#include "common.cuh"

namespace citrus {
namespace {

struct WidthArgs {
  const float* fixed;        // [K] widths in pixels, or null
  const float* height_sums;  // [K, 2] (sum e, sum e h), with cell widths
  const float* cell_width;   // [K, 2] gnomonic widths (channels, rows)
  int axis;                  // 0: channels, 1: rows
  float inv_pitch;           // 1 / pixel pitch along the axis
  float center_height;       // mean height where the emission vanishes
};

__device__ __forceinline__ float blur_width(const WidthArgs& w, int k) {
  if (w.fixed) return w.fixed[k];
  const float den = w.height_sums[2 * k], num = w.height_sums[2 * k + 1];
  const float hbar = den > 0.f ? num / fmaxf(den, 1.17549435e-38f) : w.center_height;
  return hbar * w.cell_width[2 * k + w.axis] * w.inv_pitch;
}

// out[k, line, c] = sum_j B_k[c, j] in[k, line, j] along an axis of N pixels; lines and pixels through strides.
__global__ void box_blur_kernel(const float* __restrict__ in, float* __restrict__ out, int K, int64_t lines, int N,
                                int64_t is_k, int64_t is_l, int64_t is_p, int64_t os_k, int64_t os_l, int64_t os_p,
                                WidthArgs wa) {
  const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const int k = blockIdx.y;
  if (t >= lines * N || k >= K) return;
  const int64_t line = t / N;
  const int c = (int)(t - line * N);
  const float half = 0.5f * fmaxf(blur_width(wa, k), 1e-3f);
  const float nf = (float)N;
  const float center = (float)c + 0.5f;
  const float lo = fminf(fmaxf(center - half, 0.f), nf), hi = fminf(fmaxf(center + half, 0.f), nf);
  const float* src = in + k * is_k + line * is_l;
  const int j0 = max(0, (int)floorf(lo)), j1 = min(N - 1, (int)ceilf(hi) - 1);
  float acc = 0.f;
  for (int j = j0; j <= j1; ++j) {
    const float ov = fmaxf(fminf(hi, (float)j + 1.f) - fmaxf(lo, (float)j), 0.f);
    acc = fmaf(ov, src[j * is_p], acc);
  }
  out[k * os_k + line * os_l + (int64_t)c * os_p] = acc / (hi - lo);
}

// The same filter with O(1) work per output pixel (box_blur_warp_kernel below): a warp owns one line, stages its N
// pixels in shared memory with their prefix sums (a warp scan, float32 pairs), and each output pixel is its partial
// first pixel, the prefix-sum difference over the fully covered pixels and its partial last pixel, divided by the
// window length.
constexpr int kScanMaxN = 1024;

// A float32 pair (hi, lo) that carries a sum to about 2^-40 of its magnitude: the prefix sums of the scan below are
// kept this way instead of in float64, whose rate on this GPU is a small fraction of float32's.
struct F2 {
  float hi, lo;
};

// hi + lo of a + b exactly (Knuth's two-sum), then the pair renormalised
__device__ __forceinline__ F2 f2_add(F2 a, F2 b) {
  const float s = __fadd_rn(a.hi, b.hi);
  const float bp = __fsub_rn(s, a.hi);
  const float e = __fadd_rn(__fsub_rn(a.hi, __fsub_rn(s, bp)), __fsub_rn(b.hi, bp));
  const float t = __fadd_rn(e, __fadd_rn(a.lo, b.lo));
  const float hi = __fadd_rn(s, t);
  return F2{hi, __fsub_rn(t, __fsub_rn(hi, s))};
}

__device__ __forceinline__ F2 f2_neg(F2 a) { return F2{-a.hi, -a.lo}; }

// One warp per line and kBlurLines lines per block: a lane sums a contiguous run of ceil(N / 32) pixels, a
// warp-level scan of the run sums gives the prefix sums, and no block barrier is needed, so a block's eight lines
// proceed independently (a block of 256 threads per line, as before, left most of its threads waiting at the
// scan's barriers). Lines of strided pixels (the row blur) are adjacent in memory across the block's warps, so
// the eight warps share the sectors of their loads and stores.
constexpr int kBlurLines = 8;

// One line by one warp: the pixels x [N] are in shared memory, P_hi and P_lo [N + 1] receive their prefix sums, and
// emit(c, value) takes the output pixels.
template <typename Emit>
__device__ __forceinline__ void blur_line(const float* x, float* P_hi, float* P_lo, int N, float half, int lane,
                                          Emit emit) {
  const int per = (N + 31) / 32;
  const int j0 = min(N, lane * per), j1 = min(N, j0 + per);
  F2 run{0.f, 0.f};
  for (int j = j0; j < j1; ++j) run = f2_add(run, F2{x[j], 0.f});
  F2 incl = run;
#pragma unroll
  for (int off = 1; off < 32; off <<= 1) {
    const F2 y{__shfl_up_sync(0xffffffffu, incl.hi, off), __shfl_up_sync(0xffffffffu, incl.lo, off)};
    if (lane >= off) incl = f2_add(incl, y);
  }
  F2 acc = f2_add(incl, f2_neg(run));  // exclusive prefix of this lane's run
  if (lane == 0) {
    P_hi[0] = 0.f;
    P_lo[0] = 0.f;
  }
  for (int j = j0; j < j1; ++j) {
    acc = f2_add(acc, F2{x[j], 0.f});
    P_hi[j + 1] = acc.hi;
    P_lo[j + 1] = acc.lo;
  }
  __syncwarp();
  const float nf = (float)N;
  for (int c = lane; c < N; c += 32) {
    const float center = (float)c + 0.5f;
    const float lo = fminf(fmaxf(center - half, 0.f), nf), hi = fminf(fmaxf(center + half, 0.f), nf);
    const int a = max(0, (int)floorf(lo)), b = min(N - 1, (int)ceilf(hi) - 1);
    float sum;
    if (a >= b) {
      sum = fmaxf(hi - lo, 0.f) * x[a];
    } else {
      const float first = ((float)a + 1.f - lo) * x[a], last = (hi - (float)b) * x[b];
      const F2 interior = f2_add(F2{P_hi[b], P_lo[b]}, F2{-P_hi[a + 1], -P_lo[a + 1]});
      const F2 total = f2_add(f2_add(interior, F2{first, 0.f}), F2{last, 0.f});
      sum = total.hi + total.lo;
    }
    emit(c, sum / (hi - lo));
  }
}

__global__ void __launch_bounds__(32 * kBlurLines) box_blur_warp_kernel(const float* __restrict__ in,
                                                                        float* __restrict__ out, int64_t lines, int N,
                                                                        int64_t is_k, int64_t is_l, int64_t is_p,
                                                                        int64_t os_k, int64_t os_l, int64_t os_p,
                                                                        WidthArgs wa) {
  extern __shared__ float s_blur[];  // per warp: x [N], P_hi [N + 1], P_lo [N + 1]
  const int lane = threadIdx.x % 32, warp = threadIdx.x / 32;
  const int k = blockIdx.y;
  const int64_t line = (int64_t)blockIdx.x * kBlurLines + warp;
  if (line >= lines) return;  // the whole warp: no block barrier follows
  float* x = s_blur + (int64_t)warp * (3 * N + 2);
  float* P_hi = x + N;
  const float* src = in + k * is_k + line * is_l;
  for (int j = lane; j < N; j += 32) x[j] = src[j * is_p];
  __syncwarp();
  float* dst = out + k * os_k + line * os_l;
  blur_line(x, P_hi, P_hi + N + 1, N, 0.5f * fmaxf(blur_width(wa, k), 1e-3f), lane,
            [&](int c, float v) { dst[(int64_t)c * os_p] = v; });
}

// Lines that are adjacent in memory (the row blur: pixels a row apart). A line at a time, every lane's load and store is
// a sector of its own: 64 wavefronts per 32 pixels, twice the arithmetic. A block takes kTileLines adjacent lines through
// shared memory instead, read and written by rows of kTileLines floats (two whole sectors), two lines per warp: the rows
// of 512 images of 192 x 256 pixels 241 -> 175 us (the arithmetic remains), of 5 groups of 61 x 83 pixels 164 -> 150 us.
// Up to kTileMaxN pixels a line two blocks fit an SM; longer lines keep the form above. So do images of few pixels, whose
// tiles leave SMs idle (two lines per warp, one after the other; us, lines / tiles): 16 directions of 17 x 19 pixels 2.7 /
// 3.9, 4 of 192 x 256 5.0 / 6.9, 16 of 128 x 128 5.1 / 5.6, 32 of them 8.0 / 6.6, 16 of 192 x 256 10.4 / 8.3.
constexpr int kTileLines = 16, kTileMaxN = 440;
constexpr int64_t kTilePixels = 1 << 19;  // of all directions

__host__ __device__ constexpr int blur_tile_stride(int N) { return (4 * N + 2) | 1; }  // odd: no bank conflicts across lines

__global__ void __launch_bounds__(32 * kBlurLines) box_blur_tile_kernel(const float* __restrict__ in,
                                                                        float* __restrict__ out, int64_t lines, int N,
                                                                        int64_t is_k, int64_t is_p, int64_t os_k,
                                                                        int64_t os_p, WidthArgs wa) {
  extern __shared__ float s_blur[];  // per line: x [N], P_hi [N + 1], P_lo [N + 1], out [N]
  const int lane = threadIdx.x % 32, warp = threadIdx.x / 32, W = blur_tile_stride(N);
  const int k = blockIdx.y;
  const int64_t line0 = (int64_t)blockIdx.x * kTileLines;
  const int count = (int)min((int64_t)kTileLines, lines - line0);
  const int l = threadIdx.x % kTileLines;
  const float* src = in + k * is_k + line0 + l;
  if (l < count)
    for (int j = threadIdx.x / kTileLines; j < N; j += 32 * kBlurLines / kTileLines) s_blur[l * W + j] = src[j * is_p];
  __syncthreads();
  const float half = 0.5f * fmaxf(blur_width(wa, k), 1e-3f);
  for (int line = warp; line < count; line += kBlurLines) {
    float* x = s_blur + line * W;
    blur_line(x, x + N, x + 2 * N + 1, N, half, lane, [&](int c, float v) { x[3 * N + 2 + c] = v; });
  }
  __syncthreads();
  float* dst = out + k * os_k + line0 + l;
  if (l < count)
    for (int j = threadIdx.x / kTileLines; j < N; j += 32 * kBlurLines / kTileLines)
      dst[j * os_p] = s_blur[l * W + 3 * N + 2 + j];
}

// the dense overlap matrices of the same filter, [K, N, N] (scatter_image.py:952-981)
__global__ void box_matrix_kernel(const float* __restrict__ widths, int N, float* __restrict__ out) {
  const int k = blockIdx.y;
  const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= (int64_t)N * N) return;
  const int c = (int)(t / N), j = (int)(t - (int64_t)c * N);
  const float half = 0.5f * fmaxf(widths[k], 1e-3f);
  const float nf = (float)N, center = (float)c + 0.5f;
  const float lo = fminf(fmaxf(center - half, 0.f), nf), hi = fminf(fmaxf(center + half, 0.f), nf);
  out[(int64_t)k * N * N + t] = fmaxf(fminf(hi, (float)j + 1.f) - fmaxf(lo, (float)j), 0.f) / (hi - lo);
}

// out[k, r, c] = sum_g img[k, r, g, c] W[k, g, c or 0] for rows-outer images [K, R, G, C]
__global__ void weighted_group_sum_kernel(const float* __restrict__ img, const float* __restrict__ W, int K, int R,
                                          int G, int C, int w_channels, float* __restrict__ out) {
  const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const int k = blockIdx.y;
  if (t >= (int64_t)R * C) return;
  const int r = (int)(t / C), c = (int)(t - (int64_t)r * C);
  const float* src = img + (((int64_t)k * R + r) * G) * C + c;
  const float* w = W + (int64_t)k * G * w_channels + (w_channels > 1 ? c : 0);
  float acc = 0.f;
  for (int g = 0; g < G; ++g) acc = fmaf(src[(int64_t)g * C], w[(int64_t)g * w_channels], acc);
  out[((int64_t)k * R + r) * C + c] = acc;
}

// Sums over directions in blocks of kSumBlock, each added to the accumulator in order: the rounding is that of one call per
// block, so a sum over all 512 directions of an image is as accurate as eight over 64. A thread takes a pixel and walks all
// its directions; where there are several blocks and too few pixels to fill the SMs, a thread takes a pixel of one block
// and the first of the pixel's threads adds the sums up (kBlocks): a full image of 5 groups, 64 x 64 pixels 332 -> 59 us.
constexpr int kSumBlock = 64, kSumPixels = 64, kSumSlices = 8, kSumThreads = 256;

// sum over k of term(k, s) into acc; walk(first, last) gives a block's sum to a thread that takes the pixel alone
template <bool kBlocks, typename Term, typename Walk>
__device__ __forceinline__ void sum_directions(int K, bool inside, float* __restrict__ acc, int accumulate, Term term,
                                               Walk walk) {
  float total = inside && accumulate && threadIdx.y == 0 ? *acc : 0.f;
  bool have = accumulate != 0;
  if constexpr (!kBlocks) {
    if (!inside) return;
    int k0 = 0;
    do {
      const float s = walk(k0, min(k0 + kSumBlock, K));
      total = have ? total + s : s;
      have = true;
      k0 += kSumBlock;
    } while (k0 < K);
    *acc = total;
  } else {
    __shared__ float s_part[kSumSlices][kSumPixels];
    const int slices = blockDim.y;
    for (int k0 = 0; k0 < K; k0 += slices * kSumBlock) {
      const int first = k0 + threadIdx.y * kSumBlock, last = min(first + kSumBlock, K);
      float s = 0.f;
      if (inside) {
#pragma unroll 8
        for (int k = first; k < last; ++k) term(k, s);
      }
      s_part[threadIdx.y][threadIdx.x] = s;
      __syncthreads();
      if (threadIdx.y == 0)
        for (int j = 0; j < slices && k0 + j * kSumBlock < K; ++j) {
          total = have ? total + s_part[j][threadIdx.x] : s_part[j][threadIdx.x];
          have = true;
        }
      __syncthreads();
    }
    if (inside && threadIdx.y == 0) *acc = total;
  }
}

// The block of a sum over K directions of the given pixels; two dimensions: by blocks of directions. us, a thread per pixel / by
// blocks: 65 directions of 192 x 256 pixels 3.4 / 4.5, 256 of them 7.3 / 8.2, 512 of 384 x 512 64 / 69, of 64 x 64 13 / 4.7; weighted, 65
// directions of 192 x 256 pixels 10.9 / 8.4, of 384 x 512 9.9 / 20, 96 of them 14 / 26, 128 of them 51 / 35.
inline dim3 sum_threads(int64_t K, int64_t pixels, bool weighted) {
  const int64_t alone = weighted ? (pixels >= 131072 ? 96 : kSumBlock)
                                 : (pixels >= 131072 ? K : pixels >= 32768 ? 256 : 96);
  if (K <= alone) return dim3(kSumThreads);
  return dim3(kSumPixels, (unsigned)(cdiv(K, kSumBlock) < kSumSlices ? cdiv(K, kSumBlock) : kSumSlices));
}

// acc[p] (+)= sum_k img[k, p]
template <bool kBlocks>
__global__ void sum_directions_kernel(const float* __restrict__ img, int K, int64_t P, int64_t stride_k,
                                      float* __restrict__ acc, int accumulate) {
  const int64_t p = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  sum_directions<kBlocks>(
      K, p < P, acc + p, accumulate, [&](int k, float& s) { s += img[k * stride_k + p]; },
      [&](int first, int last) {
        float s = 0.f;
        for (int k = first; k < last; ++k) s += img[k * stride_k + p];
        return s;
      });
}

// acc[g, r, c] (+)= sum_k W[k, g, r | 0, c | 0] img[k, g, r, c], images through strides (the accumulation of the full
// images, DirectionSetContext.accumulate, scatter_image.py:340-371)
template <bool kBlocks>
__global__ void weighted_direction_sum_kernel(const float* __restrict__ img, int K, int G, int R, int C, int64_t is_k,
                                              int64_t is_g, int64_t is_r, int64_t is_c, const float* __restrict__ W,
                                              int w_rows, int w_cols, float* __restrict__ acc, int accumulate) {
  const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const int g = (int)(t / ((int64_t)R * C));
  const int64_t rc = t - (int64_t)g * R * C;
  const int r = (int)(rc / C), c = (int)(rc - (int64_t)r * C);
  const int64_t w_k = (int64_t)G * w_rows * w_cols;
  const float* w = W + ((int64_t)g * w_rows + (w_rows > 1 ? r : 0)) * w_cols + (w_cols > 1 ? c : 0);
  const float* src = img + g * is_g + r * is_r + c * is_c;
  sum_directions<kBlocks>(
      K, t < (int64_t)G * R * C, acc + t, accumulate, [&](int k, float& s) { s = fmaf(w[k * w_k], src[k * is_k], s); },
      [&](int first, int last) {
        const float *wk = w + first * w_k, *x = src + first * is_k;
        float s = 0.f;
#pragma unroll 4
        for (int k = first; k < last; ++k, wk += w_k, x += is_k) s = fmaf(*wk, *x, s);
        return s;
      });
}

}  // namespace
}  // namespace citrus

using namespace citrus;

extern "C" int citrus_weighted_direction_sum(const float* image, int64_t num_directions, int64_t groups,
                                             int64_t rows, int64_t cols, int64_t is_k, int64_t is_g, int64_t is_r,
                                             int64_t is_c, const float* weights, int64_t weight_rows,
                                             int64_t weight_cols, float* accumulator, int32_t accumulate,
                                             void* stream) {
  CITRUS_REQUIRE(image && weights && accumulator, "citrus_weighted_direction_sum: null pointer");
  CITRUS_REQUIRE((weight_rows == 1 || weight_rows == rows) && (weight_cols == 1 || weight_cols == cols),
                 "citrus_weighted_direction_sum: weights must be [K, G, rows | 1, cols | 1]");
  const int64_t total = groups * rows * cols;
  if (total == 0) return CITRUS_OK;
  const dim3 threads = sum_threads(num_directions, total, true);
  auto kernel = threads.y > 1 ? weighted_direction_sum_kernel<true> : weighted_direction_sum_kernel<false>;
  kernel<<<(unsigned)cdiv(total, threads.x), threads, 0, as_stream(stream)>>>(
      image, (int)num_directions, (int)groups, (int)rows, (int)cols, is_k, is_g, is_r, is_c, weights,
      (int)weight_rows, (int)weight_cols, accumulator, accumulate);
  note_launches();
  return launch_status("citrus_weighted_direction_sum");
}

extern "C" int citrus_box_blur(const float* in, float* out, int64_t num_directions, int64_t lines, int64_t length,
                               int64_t is_k, int64_t is_l, int64_t is_p, int64_t os_k, int64_t os_l, int64_t os_p,
                               const float* widths, const float* height_sums, const float* cell_width, int32_t axis,
                               double pitch, double center_height, void* stream) {
  CITRUS_REQUIRE(in && out, "citrus_box_blur: null pointer");
  CITRUS_REQUIRE(widths || (height_sums && cell_width && pitch > 0), "citrus_box_blur: give widths or height sums");
  CITRUS_REQUIRE(num_directions >= 0 && num_directions <= 65535 && lines >= 0 && length >= 1 && (axis == 0 || axis == 1),
                 "citrus_box_blur: bad sizes");
  CITRUS_REQUIRE(in != out, "citrus_box_blur: in and out must not alias");
  if (num_directions == 0 || lines == 0) return CITRUS_OK;
  WidthArgs wa{widths, height_sums, cell_width, axis, (float)(pitch > 0 ? 1.0 / pitch : 0.0), (float)center_height};
  if (length <= kTileMaxN && num_directions * lines * length >= kTilePixels && is_l == 1 && os_l == 1 && is_p != 1 &&
      cdiv(lines, kTileLines) <= 0x7fffffff) {
    const size_t smem = (size_t)kTileLines * blur_tile_stride((int)length) * sizeof(float);
    cudaError_t e = cudaFuncSetAttribute(box_blur_tile_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         (int)(kTileLines * blur_tile_stride(kTileMaxN) * sizeof(float)));
    if (e != cudaSuccess) return set_error(CITRUS_ECUDA, "citrus_box_blur: %s", cudaGetErrorString(e));
    dim3 grid((unsigned)cdiv(lines, kTileLines), (unsigned)num_directions);
    box_blur_tile_kernel<<<grid, 32 * kBlurLines, smem, as_stream(stream)>>>(in, out, lines, (int)length, is_k, is_p,
                                                                             os_k, os_p, wa);
  } else if (length <= kScanMaxN && cdiv(lines, kBlurLines) <= 0x7fffffff) {
    const size_t smem = (size_t)kBlurLines * (3 * length + 2) * sizeof(float);  // 96 KB at the longest lines
    cudaError_t e = cudaFuncSetAttribute(box_blur_warp_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         (int)((size_t)kBlurLines * (3 * kScanMaxN + 2) * sizeof(float)));
    if (e != cudaSuccess) return set_error(CITRUS_ECUDA, "citrus_box_blur: %s", cudaGetErrorString(e));
    dim3 grid((unsigned)cdiv(lines, kBlurLines), (unsigned)num_directions);
    box_blur_warp_kernel<<<grid, 32 * kBlurLines, smem, as_stream(stream)>>>(in, out, lines, (int)length, is_k, is_l,
                                                                             is_p, os_k, os_l, os_p, wa);
  } else {
    dim3 grid((unsigned)cdiv(lines * length, 256), (unsigned)num_directions);
    box_blur_kernel<<<grid, 256, 0, as_stream(stream)>>>(in, out, (int)num_directions, lines, (int)length, is_k,
                                                         is_l, is_p, os_k, os_l, os_p, wa);
  }
  note_launches();
  return launch_status("citrus_box_blur");
}

extern "C" int citrus_box_matrix(const float* widths, int64_t num_directions, int64_t length, float* out,
                                 void* stream) {
  CITRUS_REQUIRE(widths && out && num_directions >= 0 && num_directions <= 65535 && length >= 1,
                 "citrus_box_matrix: bad arguments");
  if (num_directions == 0) return CITRUS_OK;
  dim3 grid((unsigned)cdiv(length * length, 256), (unsigned)num_directions);
  box_matrix_kernel<<<grid, 256, 0, as_stream(stream)>>>(widths, (int)length, out);
  note_launches();
  return launch_status("citrus_box_matrix");
}

extern "C" int citrus_weighted_group_sum(const float* image, const float* weights, int64_t num_directions,
                                         int64_t rows, int64_t groups, int64_t cols, int64_t weight_cols, float* out,
                                         void* stream) {
  CITRUS_REQUIRE(image && weights && out, "citrus_weighted_group_sum: null pointer");
  CITRUS_REQUIRE(num_directions >= 0 && num_directions <= 65535 && (weight_cols == 1 || weight_cols == cols),
                 "citrus_weighted_group_sum: bad sizes");
  if (num_directions == 0) return CITRUS_OK;
  dim3 grid((unsigned)cdiv(rows * cols, 256), (unsigned)num_directions);
  weighted_group_sum_kernel<<<grid, 256, 0, as_stream(stream)>>>(image, weights, (int)num_directions, (int)rows,
                                                                 (int)groups, (int)cols, (int)weight_cols, out);
  note_launches();
  return launch_status("citrus_weighted_group_sum");
}

extern "C" int citrus_sum_directions(const float* image, int64_t num_directions, int64_t pixels, int64_t stride_k,
                                     float* accumulator, int32_t accumulate, void* stream) {
  CITRUS_REQUIRE(image && accumulator && num_directions >= 0 && pixels >= 0, "citrus_sum_directions: bad arguments");
  if (pixels == 0) return CITRUS_OK;
  const dim3 threads = sum_threads(num_directions, pixels, false);
  auto kernel = threads.y > 1 ? sum_directions_kernel<true> : sum_directions_kernel<false>;
  kernel<<<(unsigned)cdiv(pixels, threads.x), threads, 0, as_stream(stream)>>>(image, (int)num_directions, pixels, stride_k,
                                                                               accumulator, accumulate);
  note_launches();
  return launch_status("citrus_sum_directions");
}

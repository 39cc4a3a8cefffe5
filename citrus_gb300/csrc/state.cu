// Compact per-view storage of the CITRUS accumulator: the linear-discontinuous cell mean in scaled float16
// (citrus/citrus.py:620-720, StateStore.put / get).
//
// Encoding: for every (group, moment) the largest |cell mean| over the cells is mapped to 2^14, scale = max / 2^14
// (1 where the maximum is 0), and each cell mean is stored as float16(mean / scale) with IEEE division and
// round-to-nearest-even conversion, as the reference's float32 tensor arithmetic does. The maximum carries a NaN as
// the reference's abs().amax() does; "maximum > 0" is then false and that (group, moment) takes the scale 1, its
// other cells stored unscaled, exactly as the reference stores them. Decoding multiplies back in
// float32 and writes zero slopes. A maximum does not depend on the order it is taken in, so the codec is bit-exact and
// deterministic.
//
// Bound by HBM: in the sweep's cell-major storage the cell means are one float in four, every line of the accumulator
// holds some, and the encoder reads it twice (maximum, then values). Blocks therefore take a run of cells times a tile
// of groups, with the threads running over the groups first where those are the nearer neighbours in memory, and turn
// the tile in shared memory for the side whose cells are contiguous. One block per (group, moment) walking its
// cells at the stride of a whole cell uses a line per 4 bytes: at 64^3 cells, 8 groups, 36 moments (1.2 GB) storing an
// accumulator took 1.15 ms so and bringing it back 2.98 ms; by tiles the two with their host calls take 0.83 ms. A small
// accumulator, or one whose cells are adjacent, is encoded that way all the same (encode_by_lines).
#include <cuda_fp16.h>

#include "common.cuh"

namespace citrus {
namespace {

constexpr int kStateThreads = 256;
constexpr int kTileCells = 256;             // cells of a tile that is turned in shared memory
constexpr int kTileGroups = 32;             // groups of a tile at most
constexpr int kMaxCells = 16;               // cells of one thread of the maximum kernel
constexpr float kFloat16Target = 16384.0f;  // 2^14: |q| <= 16384 < 65504

// The work of a block: moment n, groups [g0, g0 + gt) and cells from x0; the threads run over the tile's groups first.
struct StateTile {
  int n, g0, gt;
  int64_t x0;
  int g, x, step;  // this thread's group, first cell and cell stride within the tile; g < 0: no work
};

__device__ __forceinline__ StateTile state_tile(int G, int N, int tile, int64_t cells_per_block, int64_t cells) {
  const int gtiles = (G + tile - 1) / tile;
  const int64_t chunks = (cells + cells_per_block - 1) / cells_per_block;
  const int64_t chunk = blockIdx.x % chunks, rest = blockIdx.x / chunks;
  StateTile t;
  t.n = (int)(rest / gtiles);
  t.g0 = (int)(rest % gtiles) * tile;
  t.gt = min(tile, G - t.g0);
  t.x0 = chunk * cells_per_block;
  t.step = kStateThreads / t.gt;
  t.x = threadIdx.x / t.gt;
  t.g = t.x < t.step ? (int)threadIdx.x % t.gt : -1;
  return t;
}

// The largest |cell mean| of every (group, moment), as the bits of a non-negative float (which order as the floats do,
// a NaN above infinity) taken by integer maxima into zeroed words.
__global__ void __launch_bounds__(kStateThreads) state_max_kernel(const float* __restrict__ acc, int G, int N,
                                                                  int tile, int64_t cells_per_block, int64_t cells,
                                                                  int64_t s_g, int64_t s_n, int64_t s_x,
                                                                  unsigned* __restrict__ bits) {
  __shared__ unsigned s_max[kTileGroups];
  const StateTile t = state_tile(G, N, tile, cells_per_block, cells);
  if (threadIdx.x < kTileGroups) s_max[threadIdx.x] = 0u;
  __syncthreads();
  if (t.g >= 0) {
    const float* src = acc + (t.g0 + t.g) * s_g + t.n * s_n;
    unsigned v[kMaxCells];
#pragma unroll
    for (int u = 0; u < kMaxCells; ++u) {
      const int64_t x = t.x0 + t.x + (int64_t)u * t.step;
      v[u] = u * t.step + t.x < cells_per_block && x < cells ? __float_as_uint(__ldg(src + x * s_x)) & 0x7fffffffu : 0u;
    }
    unsigned m = 0u;
#pragma unroll
    for (int u = 0; u < kMaxCells; ++u) m = max(m, v[u]);
    if (m != 0u) atomicMax(s_max + t.g, m);
  }
  __syncthreads();
  if (threadIdx.x < t.gt && s_max[threadIdx.x] != 0u)
    atomicMax(bits + (int64_t)(t.g0 + threadIdx.x) * N + t.n, s_max[threadIdx.x]);
}

// the maxima's bits turned into scales, in place
__global__ void __launch_bounds__(kStateThreads) state_scale_kernel(float* scale, int64_t count) {
  const int64_t i = (int64_t)blockIdx.x * kStateThreads + threadIdx.x;
  if (i < count) scale[i] = scale[i] > 0.f ? __fdiv_rn(scale[i], kFloat16Target) : 1.f;
}

// element (g, n, cell) of the cell-mean component at g * s_g + n * s_n + cell * s_x
__global__ void __launch_bounds__(kStateThreads) state_encode_kernel(const float* __restrict__ acc, int G, int N,
                                                                     int tile, int64_t cells, int64_t s_g,
                                                                     int64_t s_n, int64_t s_x,
                                                                     const float* __restrict__ scale,
                                                                     __half* __restrict__ data) {
  __shared__ __half s_val[kTileGroups][kTileCells + 2];  // two halves of padding: 32 groups of a cell in 32 banks
  const StateTile t = state_tile(G, N, tile, kTileCells, cells);
  const int count = (int)min((int64_t)kTileCells, cells - t.x0);
  if (t.g >= 0) {
    const float* src = acc + (t.g0 + t.g) * s_g + t.n * s_n + t.x0 * s_x;
    const float sc = __ldg(scale + (int64_t)(t.g0 + t.g) * N + t.n);
#pragma unroll 8
    for (int x = t.x; x < count; x += t.step) s_val[t.g][x] = __float2half_rn(__fdiv_rn(__ldg(src + x * s_x), sc));
  }
  __syncthreads();
  for (int g = 0; g < t.gt; ++g)
    if (threadIdx.x < count)
      data[((int64_t)(t.g0 + g) * N + t.n) * cells + t.x0 + threadIdx.x] = s_val[g][threadIdx.x];
}

// The accumulator's quadruple (decoded mean, 0, 0, 0) as one float4: o_k = 1, the other strides multiples of 4
__global__ void __launch_bounds__(kStateThreads) state_decode4_kernel(const __half* __restrict__ data,
                                                                      const float* __restrict__ scale, int G, int N,
                                                                      int tile, int64_t cells,
                                                                      float* __restrict__ out, int64_t o_g,
                                                                      int64_t o_n, int64_t o_x) {
  __shared__ __half s_val[kTileGroups][kTileCells + 2];
  const StateTile t = state_tile(G, N, tile, kTileCells, cells);
  const int count = (int)min((int64_t)kTileCells, cells - t.x0);
#pragma unroll 8
  for (int g = 0; g < t.gt; ++g)
    if (threadIdx.x < count)
      s_val[g][threadIdx.x] = data[((int64_t)(t.g0 + g) * N + t.n) * cells + t.x0 + threadIdx.x];
  __syncthreads();
  if (t.g < 0) return;
  const float sc = __ldg(scale + (int64_t)(t.g0 + t.g) * N + t.n);
  float* dst = out + (t.g0 + t.g) * o_g + t.n * o_n + t.x0 * o_x;
  for (int x = t.x; x < count; x += t.step)
    *reinterpret_cast<float4*>(dst + x * o_x) = make_float4(__half2float(s_val[t.g][x]) * sc, 0.f, 0.f, 0.f);
}

// groups of a tile: all of them (at most kTileGroups) where groups are nearer in memory than cells, else one
inline int state_tile_groups(int64_t groups, int64_t s_g, int64_t s_x) {
  return s_x <= s_g ? 1 : (int)(groups < kTileGroups ? groups : kTileGroups);
}

// The whole encoding of a (group, moment) in one block, which walks its cells twice with kLineLoads of them in flight per
// thread; the second time they come from L2.
constexpr int kLineLoads = 8;

template <int kThreads>
__global__ void __launch_bounds__(kThreads) state_encode_lines_kernel(const float* __restrict__ acc, int N,
                                                                      int64_t cells, int64_t s_g, int64_t s_n,
                                                                      int64_t s_x, __half* __restrict__ data,
                                                                      float* __restrict__ scale) {
  __shared__ unsigned s_max[kThreads / 32];
  const int gn = blockIdx.x;  // g * N + n
  const int g = gn / N, n = gn - g * N;
  const float* src = acc + g * s_g + n * s_n;
  unsigned m = 0u;
  for (int64_t x0 = threadIdx.x; x0 < cells; x0 += kLineLoads * kThreads) {
    unsigned v[kLineLoads];
#pragma unroll
    for (int u = 0; u < kLineLoads; ++u) {
      const int64_t x = x0 + u * kThreads;
      v[u] = x < cells ? __float_as_uint(__ldg(src + x * s_x)) & 0x7fffffffu : 0u;
    }
#pragma unroll
    for (int u = 0; u < kLineLoads; ++u) m = max(m, v[u]);
  }
  m = __reduce_max_sync(0xffffffffu, m);
  if (threadIdx.x % 32 == 0) s_max[threadIdx.x / 32] = m;
  __syncthreads();
#pragma unroll
  for (int w = 0; w < kThreads / 32; ++w) m = max(m, s_max[w]);
  const float maximum = __uint_as_float(m);
  const float sc = maximum > 0.f ? __fdiv_rn(maximum, kFloat16Target) : 1.f;
  if (threadIdx.x == 0) scale[gn] = sc;
  __half* dst = data + (int64_t)gn * cells;
  for (int64_t x0 = threadIdx.x; x0 < cells; x0 += kLineLoads * kThreads) {
    float v[kLineLoads];
#pragma unroll
    for (int u = 0; u < kLineLoads; ++u) {
      const int64_t x = x0 + u * kThreads;
      v[u] = x < cells ? __ldg(src + x * s_x) : 0.f;
    }
#pragma unroll
    for (int u = 0; u < kLineLoads; ++u) {
      const int64_t x = x0 + u * kThreads;
      if (x < cells) dst[x] = __float2half_rn(__fdiv_rn(v[u], sc));
    }
  }
}

int encode_lines(const float* acc, int64_t groups, int64_t moments, int64_t cells, int64_t s_g, int64_t s_n, int64_t s_x,
                 uint16_t* data, float* scale, cudaStream_t s) {
  const unsigned blocks = (unsigned)(groups * moments);
  __half* out = reinterpret_cast<__half*>(data);
  if (cells > 2048) {
    state_encode_lines_kernel<1024><<<blocks, 1024, 0, s>>>(acc, (int)moments, cells, s_g, s_n, s_x, out, scale);
  } else {
    state_encode_lines_kernel<256><<<blocks, 256, 0, s>>>(acc, (int)moments, cells, s_g, s_n, s_x, out, scale);
  }
  note_launches();
  return launch_status("citrus_state_encode");
}

int encode_tiles(const float* acc, int64_t groups, int64_t moments, int64_t cells, int64_t s_g, int64_t s_n, int64_t s_x,
                 uint16_t* data, float* scale, cudaStream_t s) {
  const int G = (int)groups, N = (int)moments, tile = state_tile_groups(groups, s_g, s_x);
  const int64_t gtiles = cdiv(groups, tile), count = groups * moments;
  const int64_t per_block = (int64_t)kStateThreads / tile * kMaxCells;
  CITRUS_REQUIRE(moments * gtiles * cdiv(cells, kTileCells < per_block ? kTileCells : per_block) < (1ll << 31),
                 "citrus_state_encode: the accumulator exceeds the launch grid");
  cudaError_t e = cudaMemsetAsync(scale, 0, count * sizeof(float), s);
  if (e != cudaSuccess) return set_error(CITRUS_ECUDA, "citrus_state_encode: %s", cudaGetErrorString(e));
  state_max_kernel<<<(unsigned)(moments * gtiles * cdiv(cells, per_block)), kStateThreads, 0, s>>>(
      acc, G, N, tile, per_block, cells, s_g, s_n, s_x, reinterpret_cast<unsigned*>(scale));
  state_scale_kernel<<<(unsigned)cdiv(count, kStateThreads), kStateThreads, 0, s>>>(scale, count);
  state_encode_kernel<<<(unsigned)(moments * gtiles * cdiv(cells, kTileCells)), kStateThreads, 0, s>>>(
      acc, G, N, tile, cells, s_g, s_n, s_x, scale, reinterpret_cast<__half*>(data));
  note_launches(3);
  return launch_status("citrus_state_encode");
}

// Whether one launch (lines) encodes the accumulator, or the tiles' memset and three launches, which read whole lines and
// spread a (group, moment) over many blocks but cost 10 us however small it is. us, lines / tiles, at 16^3, 32^3 and 64^3 cells:
//   cells next to one another (or one group): 16 (group, moment)s 4 / 10, 9 / 14, 49 / 47; 4 of them 4 / 10, 9 / 11,
//     49 / 19; 288 of them 6 / 19, 17 / 94, 171 / 690;
//   8 groups next to one another, 16 moments: 7 / 12, 39 / 27, 278 / 193; 36 moments 13 / 14, 189 / 66, 2113 / 410.
// From 20 blocks on adjacent cells are read as fast by lines, below that while a block's walk is short; adjacent groups
// while the walk is short and the accumulator stays well inside L2 between the uses of a sector (two of them share
// one, so that enough blocks of two groups lose nothing at any size).
inline bool encode_by_lines(int64_t groups, int64_t moments, int64_t cells, int64_t s_g, int64_t s_x) {
  const int64_t count = groups * moments;
  if (state_tile_groups(groups, s_g, s_x) == 1) return count >= 20 || cells <= 49152;
  return (groups == 2 && count >= 64) || (groups * cells <= 65536 && 16 * count * cells <= 25'000'000);
}

// full accumulator element (g, n, k, cell) at g * o_g + n * o_n + k * o_k + cell * o_x: k = 0 the decoded mean, else 0
__global__ void __launch_bounds__(kStateThreads) state_decode_kernel(const __half* __restrict__ data,
                                                                     const float* __restrict__ scale, int N,
                                                                     int64_t cells, float* __restrict__ out,
                                                                     int64_t o_g, int64_t o_n, int64_t o_k,
                                                                     int64_t o_x) {
  const int gn = blockIdx.y;
  const int g = gn / N, n = gn - g * N;
  const int64_t x = (int64_t)blockIdx.x * kStateThreads + threadIdx.x;
  if (x >= cells) return;
  const float v = __half2float(data[(int64_t)gn * cells + x]) * __ldg(scale + gn);
  float* o = out + g * o_g + n * o_n + x * o_x;
  o[0] = v;
  o[o_k] = 0.f;
  o[2 * o_k] = 0.f;
  o[3 * o_k] = 0.f;
}

}  // namespace
}  // namespace citrus

using namespace citrus;

extern "C" int citrus_state_encode(const float* accumulator, int64_t groups, int64_t moments, int64_t cells,
                                   int64_t s_g, int64_t s_n, int64_t s_x, uint16_t* data, float* scale,
                                   void* stream) {
  CITRUS_REQUIRE(accumulator && data && scale, "citrus_state_encode: null pointer argument");
  CITRUS_REQUIRE(groups >= 1 && moments >= 1 && cells >= 1 && groups * moments <= (1 << 30),
                 "citrus_state_encode: bad sizes (groups %lld, moments %lld, cells %lld)", (long long)groups,
                 (long long)moments, (long long)cells);
  const auto encode = encode_by_lines(groups, moments, cells, s_g, s_x) ? encode_lines : encode_tiles;
  return encode(accumulator, groups, moments, cells, s_g, s_n, s_x, data, scale, as_stream(stream));
}

extern "C" int citrus_state_decode(const uint16_t* data, const float* scale, int64_t groups, int64_t moments,
                                   int64_t cells, float* accumulator, int64_t o_g, int64_t o_n, int64_t o_k,
                                   int64_t o_x, void* stream) {
  CITRUS_REQUIRE(accumulator && data && scale, "citrus_state_decode: null pointer argument");
  CITRUS_REQUIRE(groups >= 1 && moments >= 1 && cells >= 1 && groups * moments <= 65535,
                 "citrus_state_decode: bad sizes (groups %lld, moments %lld, cells %lld)", (long long)groups,
                 (long long)moments, (long long)cells);
  const int tile = state_tile_groups(groups, o_g, o_x);
  // by tiles of groups; a single group is read and written in order without one (64 moments of 32^3 cells 7 us, 20 in tiles)
  if (tile > 1 && o_k == 1 && o_g % 4 == 0 && o_n % 4 == 0 && o_x % 4 == 0 && ((uintptr_t)accumulator % 16) == 0) {
    const int64_t blocks = moments * cdiv(groups, tile) * cdiv(cells, kTileCells);
    CITRUS_REQUIRE(blocks < (1ll << 31), "citrus_state_decode: the accumulator exceeds the launch grid");
    state_decode4_kernel<<<(unsigned)blocks, kStateThreads, 0, as_stream(stream)>>>(
        reinterpret_cast<const __half*>(data), scale, (int)groups, (int)moments, tile, cells, accumulator, o_g, o_n,
        o_x);
    note_launches();
    return launch_status("citrus_state_decode");
  }
  dim3 grid((unsigned)cdiv(cells, kStateThreads), (unsigned)(groups * moments));
  state_decode_kernel<<<grid, kStateThreads, 0, as_stream(stream)>>>(reinterpret_cast<const __half*>(data), scale,
                                                                     (int)moments, cells, accumulator, o_g, o_n,
                                                                     o_k, o_x);
  note_launches();
  return launch_status("citrus_state_decode");
}

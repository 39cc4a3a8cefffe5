// Spherical-harmonic moments of the scattering source, T[g, n, k, x] = sum_g' transfer[g', g, l(n), x] phi[g', n, k, x]
// (citrus/scatter_solver/angular_quadrature.py:600-677 and kernels/scattering_kernels.py:159-252), summed over the
// incoming groups in ascending order. Two kernels, by blocks of points and one degree (moments_kernel) or by points
// (moments_point_kernel), over values of float4 (layouts with the 4 linear-discontinuous moments contiguous, the sweep's
// cell-major storage) or float (any other strides: the image's cell means, moment-major).
#include "common.cuh"

namespace citrus {
namespace {

constexpr int kPts = 32;     // points per block: the lanes of each warp
constexpr int kStages = 3;   // moments of phi in flight in shared memory
constexpr int kMaxGroups = 32;
constexpr int kMaxWarps = 8;

__device__ __forceinline__ void copy_async(float4* dst, const float4* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src));
}
__device__ __forceinline__ void copy_async(float* dst, const float* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src));
}
__device__ __forceinline__ void add_product(float4& acc, float m, float4 p) {
  acc.x = fmaf(m, p.x, acc.x);
  acc.y = fmaf(m, p.y, acc.y);
  acc.z = fmaf(m, p.z, acc.z);
  acc.w = fmaf(m, p.w, acc.w);
}
__device__ __forceinline__ void add_product(float& acc, float m, float p) { acc = fmaf(m, p, acc); }
__device__ __forceinline__ void set_zero(float4& v) { v = make_float4(0.f, 0.f, 0.f, 0.f); }
__device__ __forceinline__ void set_zero(float& v) { v = 0.f; }

// A block takes 32 points and one degree l and walks its 2l + 1 moments: a warp holds the transfer of its kGT outgoing
// groups for its lanes' points in registers (read once per point, coalesced, and used for every moment of the degree),
// the moments of phi stream through a ring of kStages shared-memory tiles [point][group] filled by asynchronous copies
// that run along whichever of points and groups lies closer in memory, and the results leave the same way through a
// tile of their own. Bound by HBM: phi, T and the transfer move once. With the points' 16 G bytes read and written
// per thread instead (one thread per (moment, point), 32 lines per load) the lines left L1 before their other groups
// were used: 64 x 64 x 48 cells, 16 groups, 64 moments (8.1 GB) took 12.7 ms, now 1.9 ms; 64^3 cells, 8 groups, 36
// moments (2.8 GB) 0.88 ms, now 0.52 ms. The tiles' pitch is odd in values, so neither direction has bank conflicts.
template <int kGI, int kGT, typename V>
__global__ void __launch_bounds__(32 * kMaxWarps) moments_kernel(const float* __restrict__ transfer,
                                                                 const float* __restrict__ phi,
                                                                 float* __restrict__ out, int GI, int GO,
                                                                 int num_legendre, int num_degrees, int64_t X,
                                                                 int k_count, int64_t ps_g, int64_t ps_n, int64_t ps_k,
                                                                 int64_t ps_x, int64_t os_g, int64_t os_n,
                                                                 int64_t os_k, int64_t os_x) {
  extern __shared__ float4 smem4[];
  const int lane = threadIdx.x % 32, warp = threadIdx.x / 32, warps = blockDim.x / 32;
  const int tile_groups = warps * kGT;                  // outgoing groups of this block
  const int pitch = GI | 1, pitch_out = tile_groups | 1;
  V* s_phi = reinterpret_cast<V*>(smem4);               // [kStages][kPts][pitch]
  V* s_out = s_phi + kStages * kPts * pitch;            // [kPts][pitch_out]
  const int64_t x0 = (int64_t)blockIdx.x * kPts;
  const int points = (int)min((int64_t)kPts, X - x0);
  const int l = num_degrees - 1 - blockIdx.y;           // the longest walks first
  const int k = blockIdx.z % k_count, block_go = blockIdx.z / k_count * tile_groups, go0 = block_go + warp * kGT;
  const float* src = phi + k * ps_k + x0 * ps_x;
  float* dst = out + k * os_k + x0 * os_x;
  const bool points_in = ps_x < ps_g, points_out = os_x < os_g;  // neighbours in memory: points, else groups
  auto load = [&](int n, int stage) {
    V* tile = s_phi + stage * kPts * pitch;
    const float* row = src + n * ps_n;
    for (int i = threadIdx.x; i < GI * kPts; i += blockDim.x) {
      const int p = points_in ? i % kPts : i / GI, g = points_in ? i / kPts : i - p * GI;
      if (p < points) copy_async(tile + p * pitch + g, reinterpret_cast<const V*>(row + g * ps_g + p * ps_x));
    }
  };
  const int first = l * l, count = 2 * l + 1;
#pragma unroll
  for (int s = 0; s < kStages - 1; ++s) {
    if (s < count) load(first + s, s);
    asm volatile("cp.async.commit_group;");
  }
  float tr[kGI][kGT];
  {
    const float* t = transfer + (int64_t)l * X + x0 + lane;
    const int64_t pair = (int64_t)num_legendre * X;
#pragma unroll
    for (int gi = 0; gi < kGI; ++gi)
#pragma unroll
      for (int q = 0; q < kGT; ++q)
        tr[gi][q] = (gi < GI && go0 + q < GO && lane < points) ? __ldg(t + (int64_t)(gi * GO + go0 + q) * pair) : 0.f;
  }
  for (int j = 0; j < count; ++j) {
    asm volatile("cp.async.wait_group %0;" ::"n"(kStages - 2));
    __syncthreads();  // moment j is in its tile, and the tiles of moment j - 1 are free
    if (j + kStages - 1 < count) load(first + j + kStages - 1, (j + kStages - 1) % kStages);
    asm volatile("cp.async.commit_group;");
    const V* row = s_phi + (j % kStages * kPts + lane) * pitch;
    V acc[kGT];
#pragma unroll
    for (int q = 0; q < kGT; ++q) set_zero(acc[q]);
#pragma unroll
    for (int gi = 0; gi < kGI; ++gi) {
      if (gi < GI) {
        const V p = row[gi];
#pragma unroll
        for (int q = 0; q < kGT; ++q) add_product(acc[q], tr[gi][q], p);
      }
    }
    float* o = dst + (first + j) * os_n;
    if (points_out) {
#pragma unroll
      for (int q = 0; q < kGT; ++q)
        if (go0 + q < GO && lane < points)
          *reinterpret_cast<V*>(o + (go0 + q) * os_g + lane * os_x) = acc[q];
    } else {
#pragma unroll
      for (int q = 0; q < kGT; ++q) s_out[lane * pitch_out + warp * kGT + q] = acc[q];
      __syncthreads();
      const int groups = min(tile_groups, GO - block_go);
      for (int i = threadIdx.x; i < groups * kPts; i += blockDim.x) {
        const int p = i / groups, g = i - p * groups;
        if (p < points)
          *reinterpret_cast<V*>(o + (block_go + g) * os_g + p * os_x) = s_out[p * pitch_out + g];
      }
    }
  }
}

template <int kGI, int kGT, typename V>
void launch_moments(const float* transfer, const float* phi, float* out, int GI, int GO, int num_legendre,
                    int num_degrees, int64_t X, int k_count, int64_t ps_g, int64_t ps_n, int64_t ps_k, int64_t ps_x,
                    int64_t os_g, int64_t os_n, int64_t os_k, int64_t os_x, cudaStream_t s) {
  const int warps = (int)(cdiv(GO, kGT) < kMaxWarps ? cdiv(GO, kGT) : kMaxWarps);
  const size_t smem = (size_t)kPts * (kStages * (GI | 1) + ((warps * kGT) | 1)) * sizeof(V);
  if (smem > 48 * 1024)  // above 24 groups of float4
    cudaFuncSetAttribute(moments_kernel<kGI, kGT, V>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  dim3 grid((unsigned)cdiv(X, kPts), (unsigned)num_degrees, (unsigned)(k_count * cdiv(GO, warps * kGT)));
  moments_kernel<kGI, kGT, V><<<grid, 32 * warps, smem, s>>>(transfer, phi, out, GI, GO, num_legendre, num_degrees, X,
                                                             k_count, ps_g, ps_n, ps_k, ps_x, os_g, os_n, os_k, os_x);
}

// A thread per (moment, point) with all of its incoming groups in registers, the moments fastest over the blocks, so that the
// transfer rows of a degree, shared by its 2l + 1 moments, come from L2 after the first.
constexpr int kPointThreads = 256;

__device__ __forceinline__ int degree_of(int n) {
  int l = (int)sqrtf((float)n);
  while ((l + 1) * (l + 1) <= n) ++l;
  while (l * l > n) --l;
  return l;
}

template <int kGI, typename V>
__global__ void __launch_bounds__(kPointThreads) moments_point_kernel(const float* __restrict__ transfer,
                                                                      const float* __restrict__ phi,
                                                                      float* __restrict__ out, int GI, int GO,
                                                                      int num_legendre, int64_t X, int64_t ps_g,
                                                                      int64_t ps_n, int64_t ps_k, int64_t ps_x,
                                                                      int64_t os_g, int64_t os_n, int64_t os_k,
                                                                      int64_t os_x) {
  const int64_t x = (int64_t)blockIdx.y * kPointThreads + threadIdx.x;
  const int n = blockIdx.x, k = blockIdx.z;
  if (x >= X) return;
  const float* src = phi + n * ps_n + k * ps_k + x * ps_x;
  V ph[kGI];
#pragma unroll
  for (int gi = 0; gi < kGI; ++gi)
    if (gi < GI) ph[gi] = *reinterpret_cast<const V*>(src + gi * ps_g);
  const float* tr = transfer + (int64_t)degree_of(n) * X + x;
  const int64_t pair = (int64_t)num_legendre * X;
  float* dst = out + n * os_n + k * os_k + x * os_x;
  for (int go = 0; go < GO; ++go) {
    V acc;
    set_zero(acc);
#pragma unroll
    for (int gi = 0; gi < kGI; ++gi)
      if (gi < GI) add_product(acc, __ldg(tr + (int64_t)(gi * GO + go) * pair), ph[gi]);
    *reinterpret_cast<V*>(dst + go * os_g) = acc;
  }
}

template <int kGI, typename V>
void launch_moments_point(const float* transfer, const float* phi, float* out, int GI, int GO, int num_legendre,
                          int num_degrees, int64_t X, int k_count, int64_t ps_g, int64_t ps_n, int64_t ps_k, int64_t ps_x,
                          int64_t os_g, int64_t os_n, int64_t os_k, int64_t os_x, cudaStream_t s) {
  dim3 grid((unsigned)(num_degrees * num_degrees), (unsigned)cdiv(X, kPointThreads), (unsigned)k_count);
  moments_point_kernel<kGI, V><<<grid, kPointThreads, 0, s>>>(transfer, phi, out, GI, GO, num_legendre, X, ps_g, ps_n,
                                                              ps_k, ps_x, os_g, os_n, os_k, os_x);
}

// Whether the points' threads form the moments. The blocks above run a degree's moments one after the other with a warp
// per four outgoing groups: with few groups that is one warp and little to load at a time, and in a small volume most
// of the SMs wait. The points' threads run all moments at once, but read a point's groups from lines that have left the
// caches between the groups once phi and T do not fit L2. us, points / blocks, cell-major:
//   1 group, 16 moments: 32^3 cells 3.8 / 7.5, 64^3 24 / 44; 2 groups, 64 moments: 32^3 25 / 30, 64^3 186 / 208;
//   3 groups, 36 moments: 20^3 7.0 / 15 (28 MB), 32^3 29 / 24 (113 MB); 4 groups: 16^3 6.9 / 17 (19 MB), 24^3 17 / 20 (64), 32^3
//   54 / 33 (151); 5 groups: 24^3 19 / 26 (80), 32^3 63 / 52 (189); 8 groups: 16^3 14 / 21 (38), 24^3 60 / 33 (127).
// With the points adjacent (moment-major) the blocks' tiles pay from 14 MB on, except over so few moments that the
// transfers are most of what is read (4 moments of 5 groups, 64^3: 123 / 157). bytes: the lines of phi and T that are touched.
// From points adjacent to cells adjacent the blocks' tiles pay for two groups too (64^3, 36 moments, 604 MB: 499 / 409).
inline bool moments_by_points(int GI, int degrees, int64_t bytes, bool points_adjacent, bool out_adjacent) {
  if (GI == 1) return true;
  if (GI == 2) return !points_adjacent || out_adjacent || bytes <= 300'000'000;
  if (GI > 8 || (GI > 6 && degrees < 4)) return false;
  if (degrees == 1) return true;
  if (points_adjacent) return bytes <= 14'000'000 || (degrees == 2 && GI != 4);
  return bytes <= (GI == 4 ? 60'000'000 : GI == 5 ? 170'000'000 : GI <= 6 ? 100'000'000 : 40'000'000);
}

}  // namespace
}  // namespace citrus

using namespace citrus;

extern "C" int citrus_scattering_moments(const float* transfer, const float* phi, float* out, int64_t g_in,
                                         int64_t g_out, int64_t num_legendre, int64_t num_moments, int64_t k_count,
                                         int64_t num_points, int64_t ps_g, int64_t ps_n, int64_t ps_k, int64_t ps_x,
                                         int64_t os_g, int64_t os_n, int64_t os_k, int64_t os_x, void* stream) {
  CITRUS_REQUIRE(transfer && phi && out, "citrus_scattering_moments: null pointer argument");
  CITRUS_REQUIRE(g_in >= 1 && g_in <= kMaxGroups && g_out >= 1 && g_out <= 4096,
                 "citrus_scattering_moments: groups in %lld / out %lld outside [1, %d]", (long long)g_in,
                 (long long)g_out, kMaxGroups);
  CITRUS_REQUIRE(num_moments >= 1 && num_moments <= 65535 && num_points >= 0 && (k_count == 1 || k_count == 4),
                 "citrus_scattering_moments: bad sizes");
  int L = 0;
  while ((L + 1) * (L + 1) < num_moments) ++L;
  CITRUS_REQUIRE((L + 1) * (L + 1) == num_moments && L + 1 <= num_legendre,
                 "citrus_scattering_moments: %lld moments is not (L+1)^2 with L < %lld Legendre orders",
                 (long long)num_moments, (long long)num_legendre);
  if (num_points == 0) return CITRUS_OK;
  cudaStream_t s = as_stream(stream);
  const bool vec = k_count == 4 && ps_k == 1 && os_k == 1 && ps_g % 4 == 0 && ps_n % 4 == 0 && ps_x % 4 == 0 &&
                   os_g % 4 == 0 && os_n % 4 == 0 && os_x % 4 == 0 && ((uintptr_t)phi % 16) == 0 &&
                   ((uintptr_t)out % 16) == 0;
  CITRUS_REQUIRE(num_points <= 65535ll * 256, "citrus_scattering_moments: %lld points exceed the grid",
                 (long long)num_points);
  const int GI = (int)g_in, GO = (int)g_out, NL = (int)num_legendre;
  const bool points_adjacent = !vec && ps_x == 1;
  const int64_t bytes = 4 * (g_in + g_out) * num_moments * num_points * (points_adjacent ? k_count : 4);
#define CITRUS_MOMENTS_POINT(KGI)                                                                                     \
  if (vec)                                                                                                           \
    launch_moments_point<KGI, float4>(transfer, phi, out, GI, GO, NL, L + 1, num_points, 1, ps_g, ps_n, 0, ps_x, os_g, \
                                      os_n, 0, os_x, s);                                                             \
  else                                                                                                               \
    launch_moments_point<KGI, float>(transfer, phi, out, GI, GO, NL, L + 1, num_points, (int)k_count, ps_g, ps_n,    \
                                     ps_k, ps_x, os_g, os_n, os_k, os_x, s);
  if (moments_by_points(GI, L + 1, bytes, points_adjacent, os_x == 1)) {
    if (GI == 1) {
      CITRUS_MOMENTS_POINT(1)
    } else if (GI == 2) {
      CITRUS_MOMENTS_POINT(2)
    } else if (GI <= 4) {
      CITRUS_MOMENTS_POINT(4)
    } else {
      CITRUS_MOMENTS_POINT(8)
    }
    note_launches();
    return launch_status("citrus_scattering_moments");
  }
#undef CITRUS_MOMENTS_POINT
  // the incoming groups a thread's transfers are unrolled for: four outgoing groups each up to 16, two above, which
  // keeps the 64 transfers in registers
#define CITRUS_MOMENTS_LAUNCH(KGI, KGT)                                                                              \
  if (vec)                                                                                                           \
    launch_moments<KGI, KGT, float4>(transfer, phi, out, GI, GO, NL, L + 1, num_points, 1, ps_g, ps_n, 0, ps_x, os_g, \
                                     os_n, 0, os_x, s);                                                              \
  else                                                                                                               \
    launch_moments<KGI, KGT, float>(transfer, phi, out, GI, GO, NL, L + 1, num_points, (int)k_count, ps_g, ps_n,     \
                                    ps_k, ps_x, os_g, os_n, os_k, os_x, s);
  if (GI <= 4) {
    CITRUS_MOMENTS_LAUNCH(4, 4)
  } else if (GI <= 8) {
    CITRUS_MOMENTS_LAUNCH(8, 4)
  } else if (GI <= 12) {
    CITRUS_MOMENTS_LAUNCH(12, 4)
  } else if (GI <= 16) {
    CITRUS_MOMENTS_LAUNCH(16, 4)
  } else {
    CITRUS_MOMENTS_LAUNCH(32, 2)
  }
#undef CITRUS_MOMENTS_LAUNCH
  note_launches();
  return launch_status("citrus_scattering_moments");
}

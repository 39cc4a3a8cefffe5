// The attenuated total emission of the collapsed-cone image with per-block sums of its mean panel height
// (scatter_image.py:829-874, uncollided_kernels.py:712-795): a kernel with a thread per (point, direction) and all of its groups,
// and one with a thread per (point, group), which also forms the multiple-collision source from its moments.
#include <math.h>
#include <type_traits>
#include <stdlib.h>

#include "emission_warps.cuh"

namespace citrus {
namespace {

// ---- attenuated total emission of the image ---------------------------------------------------------------------
// e = (S_FC + S_MC,cell) exp(-max(0, tau_cell - mu_cell omega . (r - r_cell))), written voxel-major [k, V, G] (or the
// weighted group sum [k, V] with signal weights), and per block the sums of e and e h (h = panel height of the point).
//
// A block is 32 points by the G groups (a warp holds 32 / G points with their groups in adjacent lanes) by 16, 32 or
// 64 directions (emission_dirs): the [K, NC, G] loads of a warp are coalesced, the point's inputs are loaded once for
// all of the block's directions, and the transfer rows of the eta nodes that the block's points and directions touch are staged
// in shared memory (the window). S_MC is either read ([K, G, NC], the reference's interface) or formed from the
// scattering-source moments of the point's cell held in registers, T[n, g, cell] for n < N_sh, and the harmonics of
// the block's directions in shared memory. The per-block sums are a butterfly over the groups and one over the points:
// deterministic.
constexpr int kMaxMoments = 64;
constexpr int kRegMoments = 36;  // scattering-source moments held in registers (P5); more are read per direction

// window bytes of an emission block with kDirs directions (more directions span more table nodes)
__host__ __device__ constexpr int emission_window_bytes(int dirs) {
  return dirs > 32 ? 64 * 1024 : dirs > 16 ? 48 * 1024 : kWindowBytes;
}

template <int kGP, int kMM, bool kFused, int kDirs>
__global__ void __launch_bounds__(kEmitPoints * kGP) emission_kernel(
    FCInputs in, Table tb, PointGrid pg, const float* __restrict__ omegas, int K,
    const float* __restrict__ tau /*[K, NC, G], or [K, NC, TM] path lengths with tau_mu*/,
    const float* __restrict__ tau_mu /*[TM, G] or null*/, int TM, const float* __restrict__ mu /*[G, NC]*/,
    const float* __restrict__ multiple /*[K, NC, G], read when not fused*/,
    const float* __restrict__ harmonics /*[K, NS], fused*/, const float* __restrict__ moments /*[NS, NC, G], fused*/,
    int NS, const float* __restrict__ heights, const float* __restrict__ signal_weight /*[K, G] or null*/, float dx,
    float dy, float dz, float* __restrict__ out, float* __restrict__ partial /*[K, nblocks, 2]*/) {
  constexpr int kPW = 32 / kGP;                 // points per warp
  constexpr int kWarps = kEmitPoints / kPW;     // = kGP
  extern __shared__ float4 s_dyn4[];
  float* s_tab = reinterpret_cast<float*>(s_dyn4);  // the table window (dynamic, kWindowBytes)
  __shared__ float s_om[kDirs][3];
  __shared__ float s_sw[kDirs][kGP];          // signal weights of the block's directions
  __shared__ __align__(16) float s_y[kFused ? kDirs : 1][kFused ? kMaxMoments : 4];
  __shared__ float s_sum[kDirs][kWarps][2];   // per-direction, per-warp sums of e and e h
  __shared__ int s_range[2][32];
  __shared__ int s_window[2];
  const int G = tb.G;
  const int tid = threadIdx.x, warp = tid / 32, lane = tid % 32;
  const int g = lane % kGP, p = warp * kPW + lane / kGP;   // the thread's group and point of the block
  const bool gvalid = g < G;
  const int d0 = blockIdx.y * kDirs;
  const int nd = min(kDirs, K - d0);
  constexpr int nthreads = kEmitPoints * kGP;
  for (int i = tid; i < kDirs * 3; i += nthreads) s_om[i / 3][i % 3] = i < nd * 3 ? omegas[3 * d0 + i] : 0.f;
  if (signal_weight != nullptr)
    for (int i = tid; i < kDirs * kGP; i += nthreads) {
      const int dd = i / kGP, q = i % kGP;
      s_sw[dd][q] = (dd < nd && q < G) ? signal_weight[(int64_t)(d0 + dd) * G + q] : 0.f;
    }
  if (kFused)
    for (int i = tid; i < kDirs * NS; i += nthreads)
      s_y[i / NS][i % NS] = i < nd * NS ? harmonics[(int64_t)d0 * NS + i] : 0.f;

  const int64_t v = (int64_t)blockIdx.x * kEmitPoints + p;
  const bool valid = v < in.V;
  const int64_t NC = (int64_t)pg.Rc * pg.Cc * pg.Sc;
  float rho[kMM], phi[kGP];
  float ux = 0.f, uy = 0.f, uz = 0.f, h = 0.f, offx = 0.f, offy = 0.f, offz = 0.f, muc = 0.f;
  int64_t cell = 0;
#pragma unroll
  for (int q = 0; q < kGP; ++q) phi[q] = 0.f;
#pragma unroll
  for (int m = 0; m < kMM; ++m) rho[m] = 0.f;
  float tmom[kFused ? kRegMoments : 1];
  if (valid) {
    int i, j, k;
    point_rcs(v, pg, i, j, k);
    primary_direction(__ldg(in.ax_x + j), __ldg(in.ax_y + i), __ldg(in.ax_z + k), in.r0x, in.r0y, in.r0z, ux, uy, uz);
#pragma unroll
    for (int m = 0; m < kMM; ++m)
      if (m < tb.M) rho[m] = __ldg(in.rho + (int64_t)m * in.V + v);
#pragma unroll
    for (int q = 0; q < kGP; ++q)
      if (q < G) phi[q] = __ldg(in.phi + (int64_t)q * in.V + v);
    const int F = pg.f, ic = i / F, jc = j / F, kc = k / F;
    cell = ((int64_t)ic * pg.Cc + jc) * pg.Sc + kc;
    const float half = (F - 1) * 0.5f;
    offy = dy * ((float)(i - ic * F) - half);
    offx = dx * ((float)(j - jc * F) - half);
    offz = dz * ((float)(k - kc * F) - half);
    h = heights ? __ldg(heights + v) : 0.f;
    if (gvalid) muc = __ldg(mu + (int64_t)g * NC + cell);
  }
  float tmu[kMM];  // the group's attenuation per traced material, when tau holds material path lengths
#pragma unroll
  for (int m = 0; m < kMM; ++m) tmu[m] = (tau_mu != nullptr && m < TM && gvalid) ? __ldg(tau_mu + m * G + g) : 0.f;
  if (kFused) {
#pragma unroll
    for (int n = 0; n < (kFused ? kRegMoments : 1); ++n)
      tmom[n] = (valid && gvalid && n < NS) ? __ldg(moments + ((int64_t)n * NC + cell) * G + g) : 0.f;
  }
  __syncthreads();  // s_om and s_y are complete
  stage_window(tb, valid, ux, uy, uz, s_om, nd, g, kGP, warp, kWarps, tid, nthreads, s_range, s_window, s_tab,
               emission_window_bytes(kDirs));
  const int win_lo = s_window[0];

  // running pointers to this lane's element of direction d0 + dd (advanced once per direction)
  const float* mp = kFused ? nullptr : multiple + ((int64_t)d0 * NC + cell) * G + g;
  const float* tp = tau_mu != nullptr ? tau + ((int64_t)d0 * NC + cell) * TM : tau + ((int64_t)d0 * NC + cell) * G + g;
  const int64_t mp_step = NC * G, tp_step = tau_mu != nullptr ? NC * TM : NC * G;
  float* op = signal_weight != nullptr ? out + (int64_t)d0 * in.V + v : out + ((int64_t)d0 * in.V + v) * G + g;
  const int64_t op_step = signal_weight != nullptr ? in.V : in.V * G;
  // the table window (or, where a block's nodes do not fit it, the table in global memory) is fixed for the block:
  // the direction loop is compiled for each case, with no test of it per direction
  auto directions = [&](auto windowed) {
    constexpr bool kWin = decltype(windowed)::value;
    for (int dd = 0; dd < nd; ++dd) {
      float e = 0.f;
      if (valid && gvalid) {
        const float ox = s_om[dd][0], oy = s_om[dd][1], oz = s_om[dd][2];
        const float cosine = ux * ox + uy * oy + uz * oz;
        int i0;
        float w;
        table_position(tb, cosine, i0, w);
        const float offset = pg.f > 1 ? oy * offy + ox * offx + oz * offz : 0.f;  // one point per cell: its centre
        const float src = fc_group<kGP, kMM, kWin ? 1 : 2, true>(tb, s_tab, win_lo, i0, w, g, rho, phi);
        float smc = 0.f;
        if (kFused) {
#pragma unroll
          for (int n = 0; n < (kFused ? kRegMoments : 1); n += 4) {
            const float4 y = *reinterpret_cast<const float4*>(&s_y[kFused ? dd : 0][n]);
            smc = fmaf(y.x, tmom[n], smc);
            if (n + 1 < kRegMoments) smc = fmaf(y.y, tmom[n + 1], smc);
            if (n + 2 < kRegMoments) smc = fmaf(y.z, tmom[n + 2], smc);
            if (n + 3 < kRegMoments) smc = fmaf(y.w, tmom[n + 3], smc);
          }
          for (int n = kRegMoments; n < NS; ++n)
            smc = fmaf(s_y[kFused ? dd : 0][n], __ldg(moments + ((int64_t)n * NC + cell) * G + g), smc);
        } else {
          smc = __ldg(mp);
        }
        float t;
        if (tau_mu != nullptr) {  // sum_m mu[m, g] P_m, in material order
          t = 0.f;
#pragma unroll
          for (int m = 0; m < kMM; ++m)
            if (m < TM) t = fmaf(tmu[m], __ldg(tp + m), t);
        } else {
          t = __ldg(tp);
        }
        const float depth = pg.f > 1 ? fmaxf(t - muc * offset, 0.f) : fmaxf(t, 0.f);
        e = (src + smc) * __expf(-depth);  // the fast exponential: within a few ulp for these depths
      }
      // group sums over the kGP lanes of the point (in group order), then the warp's points
      float tot = e, sgl = signal_weight != nullptr ? s_sw[dd][g] * e : 0.f;
#pragma unroll
      for (int off = 1; off < kGP; off <<= 1) {
        tot += __shfl_xor_sync(0xffffffffu, tot, off);
        sgl += __shfl_xor_sync(0xffffffffu, sgl, off);
      }
      if (signal_weight != nullptr) {
        if (g == 0 && valid) *op = sgl;
      } else if (valid && gvalid) {
        *op = e;
      }
      float a = (g == 0) ? tot : 0.f, b = (g == 0) ? tot * h : 0.f;
#pragma unroll
      for (int off = kGP; off < 32; off <<= 1) {
        a += __shfl_xor_sync(0xffffffffu, a, off);
        b += __shfl_xor_sync(0xffffffffu, b, off);
      }
      if (lane == 0) {
        s_sum[dd][warp][0] = a;
        s_sum[dd][warp][1] = b;
      }
      if (!kFused) mp += mp_step;
      tp += tp_step;
      op += op_step;
    }
  };
  if (win_lo >= 0) directions(std::true_type{});
  else directions(std::false_type{});
  __syncthreads();
  for (int i = tid; i < 2 * nd; i += nthreads) {  // one or two groups have fewer threads than sums
    const int dd = i / 2, which = i % 2;
    float part[kWarps];
#pragma unroll
    for (int q = 0; q < kWarps; ++q) part[q] = s_sum[dd][q][which];
    partial[((int64_t)(d0 + dd) * gridDim.x + blockIdx.x) * 2 + which] = tree_sum<kWarps>(part);  // the butterfly goes on
  }
}

// sums over the blocks of the emission's partial sums, in block order: [K, nblocks, 2] -> [K, 2]
__global__ void reduce_partials_kernel(const float* __restrict__ partial, int64_t nblocks, int K,
                                       float* __restrict__ out) {
  const int d = blockIdx.x;
  const int which = threadIdx.y;
  __shared__ double s[2][256];
  double acc = 0.0;
  for (int64_t b = threadIdx.x; b < nblocks; b += blockDim.x) acc += partial[((int64_t)d * nblocks + b) * 2 + which];
  s[which][threadIdx.x] = acc;
  __syncthreads();
  for (int w = blockDim.x / 2; w > 0; w /= 2) {
    if (threadIdx.x < w) s[which][threadIdx.x] += s[which][threadIdx.x + w];
    __syncthreads();
  }
  if (threadIdx.x == 0) out[d * 2 + which] = (float)s[which][0];
}

}  // namespace
}  // namespace citrus

using namespace citrus;

namespace citrus {
namespace {

template <int kGP, int kMM, bool kFused, int kDirs>
int launch_emission_d(dim3 grid, cudaStream_t s, const FCInputs& in, const Table& tb, const PointGrid& pg,
                      const float* omegas, int K, const float* tau, const float* tau_mu, int TM, const float* mu,
                      const float* multiple, const float* harmonics, const float* moments, int NS,
                      const float* heights, const float* signal_weight, const double* deltas, float* out,
                      float* partial) {
  constexpr int bytes = emission_window_bytes(kDirs);
  cudaError_t e = cudaFuncSetAttribute(emission_kernel<kGP, kMM, kFused, kDirs>,
                                       cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
  if (e != cudaSuccess) return set_error(CITRUS_ECUDA, "emission window: %s", cudaGetErrorString(e));
  grid.y = (unsigned)cdiv(K, kDirs);
  emission_kernel<kGP, kMM, kFused, kDirs><<<grid, kEmitPoints * kGP, bytes, s>>>(
      in, tb, pg, omegas, K, tau, tau_mu, TM, mu, multiple, harmonics, moments, NS, heights, signal_weight, (float)deltas[0],
      (float)deltas[1], (float)deltas[2], out, partial);
  note_launches();
  return CITRUS_OK;
}

// directions per emission block: 32 amortise the block's set-up (point geometry, table window) over twice as many
// directions once there are enough of them; CITRUS_EMISSION_DIRS (16, 32 or 64) overrides, for measurements
inline int emission_dirs(int K) {
  static const int forced = [] {
    const char* v = getenv("CITRUS_EMISSION_DIRS");
    return v ? atoi(v) : 0;
  }();
  if (forced == 16 || forced == 32 || forced == 64) return forced;
  return K >= 64 ? 32 : 16;
}

template <int kGP, int kMM, bool kFused>
int launch_emission_m(dim3 grid, int G, cudaStream_t s, const FCInputs& in, const Table& tb, const PointGrid& pg,
                      const float* omegas, int K, const float* tau, const float* tau_mu, int TM, const float* mu,
                      const float* multiple, const float* harmonics, const float* moments, int NS,
                      const float* heights, const float* signal_weight, const double* deltas, float* out,
                      float* partial) {
  (void)G;
  const int dirs = emission_dirs(K);
  if (dirs == 64)
    return launch_emission_d<kGP, kMM, kFused, 64>(grid, s, in, tb, pg, omegas, K, tau, tau_mu, TM, mu, multiple,
                                                   harmonics, moments, NS, heights, signal_weight, deltas, out,
                                                   partial);
  if (dirs == 32)
    return launch_emission_d<kGP, kMM, kFused, 32>(grid, s, in, tb, pg, omegas, K, tau, tau_mu, TM, mu, multiple,
                                                   harmonics, moments, NS, heights, signal_weight, deltas, out,
                                                   partial);
  return launch_emission_d<kGP, kMM, kFused, 16>(grid, s, in, tb, pg, omegas, K, tau, tau_mu, TM, mu, multiple,
                                                 harmonics, moments, NS, heights, signal_weight, deltas, out, partial);
}

template <int kGP, bool kFused>
int launch_emission(dim3 grid, int G, cudaStream_t s, const FCInputs& in, const Table& tb, const PointGrid& pg,
                    const float* omegas, int K, const float* tau, const float* tau_mu, int TM, const float* mu,
                    const float* multiple, const float* harmonics, const float* moments, int NS,
                    const float* heights, const float* signal_weight, const double* deltas, float* out,
                    float* partial) {
  if (tb.M <= 2 && TM <= 2)
    return launch_emission_m<kGP, 2, kFused>(grid, G, s, in, tb, pg, omegas, K, tau, tau_mu, TM, mu, multiple,
                                             harmonics, moments, NS, heights, signal_weight, deltas, out, partial);
  return launch_emission_m<kGP, kMaxM, kFused>(grid, G, s, in, tb, pg, omegas, K, tau, tau_mu, TM, mu, multiple,
                                               harmonics, moments, NS, heights, signal_weight, deltas, out, partial);
}

// CITRUS_EMISSION_KERNEL=groups selects the group-lane kernel (emission_kernel) for the product form too; read at
// every call, for measurements and for the test that the two kernels agree
inline bool emission_by_groups() {
  const char* v = getenv("CITRUS_EMISSION_KERNEL");
  return v != nullptr && v[0] == 'g';
}

template <int kGP>
int emission_for(int64_t V, int K, cudaStream_t s, const FCInputs& in, const Table& tb, const PointGrid& pg,
                 const float* omegas, const float* tau, const float* tau_mu, int TM, const float* mu,
                 const float* multiple,
                 const float* harmonics, const float* moments, int NS, const float* heights,
                 const float* signal_weight, const double* deltas, float* out, float* partial,
                 float* height_sums) {
  const int64_t nblocks = cdiv(V, kEmitPoints);
  dim3 grid((unsigned)nblocks, 1u);  // grid.y: the direction blocks, set by the launcher
  int st;
  if (moments == nullptr && kGP <= 16 && !emission_by_groups()) {
    const EmissionCall c{in, tb, pg, K, TM, omegas, tau, tau_mu, mu, multiple, heights, signal_weight, deltas, out, partial, s};
    st = kGP <= 4 ? emission_warps_4(c) : kGP <= 8 ? emission_warps_8(c) : emission_warps_16(c);
  } else {
    st = moments != nullptr
             ? launch_emission<kGP, true>(grid, tb.G, s, in, tb, pg, omegas, K, tau, tau_mu, TM, mu, multiple,
                                          harmonics, moments, NS, heights, signal_weight, deltas, out, partial)
             : launch_emission<kGP, false>(grid, tb.G, s, in, tb, pg, omegas, K, tau, tau_mu, TM, mu, multiple,
                                           harmonics, moments, NS, heights, signal_weight, deltas, out, partial);
  }
  if (st) return st;
  reduce_partials_kernel<<<K, dim3(256, 2), 0, s>>>(partial, nblocks, K, height_sums);
  note_launches();
  return CITRUS_OK;
}

// shared by the two entry points: multiple [K, G, NC] (moments NULL), or harmonics [K, NS] and moments [NS, G, NC]
int attenuated_emission(const char* name, const float* rho, int64_t num_materials, const float* phi,
                        int64_t num_groups, const float* axes, const int64_t* point_dims, int64_t points_per_cell,
                        const double* point_deltas, const double* focal_spot, const float* table, int64_t num_eta,
                        double eta_lo, double eta_hi, const float* omegas, int64_t num_directions, const float* tau,
                        const float* tau_mu, int64_t tau_materials, const float* mu, const float* multiple,
                        const float* harmonics, const float* moments,
                        int64_t num_moments, const float* heights, const float* signal_weight, float* out,
                        float* partial, int64_t partial_capacity, float* height_sums, void* stream) {
  int st = check_table(table, num_materials, num_eta, num_groups);
  if (st) return st;
  CITRUS_REQUIRE(rho && phi && axes && point_dims && point_deltas && focal_spot && omegas && tau && mu && out &&
                     partial && height_sums && (multiple || (harmonics && moments)),
                 "%s: null pointer", name);
  CITRUS_REQUIRE(tau_mu == nullptr || (tau_materials >= 1 && tau_materials <= kMaxM),
                 "%s: %lld traced materials outside [1, %d]", name, (long long)tau_materials, kMaxM);
  CITRUS_REQUIRE(moments == nullptr || (num_moments >= 1 && num_moments <= kMaxMoments),
                 "%s: %lld moments outside [1, %d]", name, (long long)num_moments, kMaxMoments);
  const int64_t f = points_per_cell;
  CITRUS_REQUIRE(f >= 1 && point_dims[0] % f == 0 && point_dims[1] % f == 0 && point_dims[2] % f == 0,
                 "%s: the point grid is not cells x %lld", name, (long long)f);
  CITRUS_REQUIRE(num_directions >= 0 && num_directions <= 65535, "%s: bad direction count", name);
  if (num_groups % 4 == 0)
    CITRUS_REQUIRE(((uintptr_t)table % 16) == 0 && ((uintptr_t)out % 16) == 0,
                   "%s: table and out must be 16-byte aligned", name);
  const int64_t V = point_dims[0] * point_dims[1] * point_dims[2];
  const int64_t nblocks = cdiv(V, kEmitPoints);
  CITRUS_REQUIRE(partial_capacity >= nblocks * num_directions * 2, "%s: partial buffer holds %lld floats, needs %lld",
                 name, (long long)partial_capacity, (long long)(nblocks * num_directions * 2));
  if (V == 0 || num_directions == 0) return CITRUS_OK;
  const FCInputs in = make_inputs(rho, phi, axes, V, focal_spot, point_dims);
  const Table tb = make_table(table, num_materials, num_eta, num_groups, eta_lo, eta_hi);
  const PointGrid pg = make_grid(point_dims, f);
  const int G = (int)num_groups, K = (int)num_directions, NS = (int)num_moments;
  cudaStream_t s = as_stream(stream);
#define CITRUS_EMISSION(GP)                                                                                        \
  emission_for<GP>(V, K, s, in, tb, pg, omegas, tau, tau_mu, (int)tau_materials, mu, multiple, harmonics, moments,  \
                   NS, heights, signal_weight, \
                   point_deltas, out, partial, height_sums)
  if (G <= 1) st = CITRUS_EMISSION(1);
  else if (G <= 2) st = CITRUS_EMISSION(2);
  else if (G <= 4) st = CITRUS_EMISSION(4);
  else if (G <= 8) st = CITRUS_EMISSION(8);
  else if (G <= 16) st = CITRUS_EMISSION(16);
  else st = CITRUS_EMISSION(32);
#undef CITRUS_EMISSION
  if (st) return st;
  return launch_status(name);
}

}  // namespace
}  // namespace citrus

extern "C" int citrus_attenuated_emission(const float* rho, int64_t num_materials, const float* phi,
                                          int64_t num_groups, const float* axes, const int64_t* point_dims,
                                          int64_t points_per_cell, const double* point_deltas,
                                          const double* focal_spot, const float* table, int64_t num_eta,
                                          double eta_lo, double eta_hi, const float* omegas, int64_t num_directions,
                                          const float* tau, const float* tau_mu, int64_t tau_materials,
                                          const float* mu, const float* multiple, const float* heights,
                                          const float* signal_weight, float* out, float* partial,
                                          int64_t partial_capacity, float* height_sums, void* stream) {
  CITRUS_REQUIRE(multiple != nullptr, "citrus_attenuated_emission: null multiple-collision source");
  return attenuated_emission("citrus_attenuated_emission", rho, num_materials, phi, num_groups, axes, point_dims,
                             points_per_cell, point_deltas, focal_spot, table, num_eta, eta_lo, eta_hi, omegas,
                             num_directions, tau, tau_mu, tau_materials, mu, multiple, nullptr, nullptr, 0, heights,
                             signal_weight, out, partial, partial_capacity, height_sums, stream);
}

extern "C" int citrus_attenuated_emission_moments(const float* rho, int64_t num_materials, const float* phi,
                                                  int64_t num_groups, const float* axes, const int64_t* point_dims,
                                                  int64_t points_per_cell, const double* point_deltas,
                                                  const double* focal_spot, const float* table, int64_t num_eta,
                                                  double eta_lo, double eta_hi, const float* omegas,
                                                  int64_t num_directions, const float* tau, const float* tau_mu,
                                                  int64_t tau_materials, const float* mu, const float* harmonics,
                                                  const float* moments, int64_t num_moments,
                                                  const float* heights, const float* signal_weight, float* out,
                                                  float* partial, int64_t partial_capacity, float* height_sums,
                                                  void* stream) {
  CITRUS_REQUIRE(harmonics != nullptr && moments != nullptr,
                 "citrus_attenuated_emission_moments: null harmonics or moments");
  return attenuated_emission("citrus_attenuated_emission_moments", rho, num_materials, phi, num_groups, axes,
                             point_dims, points_per_cell, point_deltas, focal_spot, table, num_eta, eta_lo, eta_hi,
                             omegas, num_directions, tau, tau_mu, tau_materials, mu, nullptr, harmonics, moments,
                             num_moments, heights,
                             signal_weight, out, partial, partial_capacity, height_sums, stream);
}

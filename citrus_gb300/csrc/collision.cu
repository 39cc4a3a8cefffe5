// Uncollided fluence and first-collision source of one view.
//
//  * group transmission, T_g = sum_{e in g} w_e exp(-sum_m mu_m(e) P_m - mu_f(e) P_f)
//    (citrus/scatter_solver/cross_sections.py:797-883, kernels/transmission_kernels.py:187-226), optionally times a
//    per-point factor (the source weight b / |r - r0|^2 of uncollided.py:160-197);
//  * the focal-spot weight b(Omega) / |r - r0|^2 at points (source.py:289-382: 1 where the ray from the focal spot
//    meets the collimated field on the panel);
//  * the first-collision source S_FC,g(r, omega) = sum_m rho_m sum_{g' <= g} T_m^{g' -> g}(Omega_UC . omega) phi_g'
//    with the transfer interpolated linearly in eta (uncollided.py:200-308, cross_sections.py:905-1021), and three
//    fused forms of it: the LD moments of the corrected source per transport cell, written cell-major into the
//    sweep's store (uncollided.py:464-511, uncollided_kernels.py:552-634); the quadrature sums I0, I1, I2 with the
//    exact moments E0, E1 and the float64 correction factors (uncollided.py:357-461, 538-636); and the attenuated
//    total emission of the image (emission.cu).
//
// Thread layout of the point kernels: a block is 32 points (threadIdx.x) by the outgoing groups (threadIdx.y), so a
// warp reads and writes 32 consecutive points of one group. The transfer table is laid out [M, N_eta, G_out, G_in]
// (downscatter only, zero above the diagonal), so the 32 B row of one outgoing group at one node is one vector load.
#include <math.h>
#include <type_traits>
#include <stdlib.h>

#include "collision.cuh"
#include "panel_interpolate.cuh"

namespace citrus {
namespace {

constexpr int kPoints = 32;
// S_FC of group go at one point for one direction: sum_m rho_m [(1 - w) T_m[i0] + w T_m[i0 + 1]] . phi
template <int kG>
__device__ __forceinline__ float fc_value(const Table& tb, int i0, float w, int go, const float* rho,
                                          const float* phi) {
  const int G = kG > 0 ? kG : tb.G;
  float acc = 0.f;
  for (int m = 0; m < tb.M; ++m) {
    const float r = rho[m];
    if (r == 0.f) continue;
    const float* row0 = tb.t + (((int64_t)m * tb.N + i0) * G + go) * G;
    const float* row1 = row0 + (int64_t)G * G;
    float a0 = 0.f, a1 = 0.f;
#pragma unroll
    for (int gi = 0; gi < (kG > 0 ? kG : kMaxG); ++gi) {
      if (gi > go || gi >= G) break;
      a0 = fmaf(__ldg(row0 + gi), phi[gi], a0);
      a1 = fmaf(__ldg(row1 + gi), phi[gi], a1);
    }
    acc = fmaf(r, a0 + (a1 - a0) * w, acc);
  }
  return acc;
}

// ---- group transmission -------------------------------------------------------------------------------------
__global__ void transmission_kernel(const float* __restrict__ path, int Mp, int64_t P,
                                    const float* __restrict__ fine_mu /*[Mp, E]*/, const float* __restrict__ weight,
                                    const int* __restrict__ group, int E, int G, const float* __restrict__ filter_path,
                                    const float* __restrict__ filter_mu, const float* __restrict__ factor,
                                    float* __restrict__ out) {
  extern __shared__ float sm[];
  float* s_mu = sm;                        // [Mp, E]
  float* s_w = sm + Mp * E;                // [E]
  float* s_f = s_w + E;                    // [E]
  int* s_g = reinterpret_cast<int*>(s_f + E);
  for (int i = threadIdx.x; i < Mp * E; i += blockDim.x) s_mu[i] = fine_mu[i];
  for (int i = threadIdx.x; i < E; i += blockDim.x) {
    s_w[i] = weight[i];
    s_f[i] = filter_mu ? filter_mu[i] : 0.f;
    s_g[i] = group[i];
  }
  __syncthreads();
  const int64_t p = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= P) return;
  float pm[kMaxM];
#pragma unroll
  for (int m = 0; m < kMaxM; ++m) pm[m] = m < Mp ? path[(int64_t)m * P + p] : 0.f;
  const float pf = filter_path ? filter_path[p] : 0.f;
  float acc[kMaxG];
#pragma unroll
  for (int g = 0; g < kMaxG; ++g) acc[g] = 0.f;
  for (int e = 0; e < E; ++e) {
    float tau = s_mu[e] * pm[0];
    for (int m = 1; m < Mp; ++m) tau = fmaf(s_mu[m * E + e], pm[m], tau);
    if (filter_path) tau = fmaf(s_f[e], pf, tau);  // the filter after the materials, as the reference adds it
    const float t = s_w[e] * expf(-tau);
    const int g = s_g[e];
#pragma unroll
    for (int q = 0; q < kMaxG; ++q)
      if (q == g) acc[q] += t;
  }
  const float fac = factor ? factor[p] : 1.f;
#pragma unroll
  for (int g = 0; g < kMaxG; ++g)
    if (g < G) out[(int64_t)g * P + p] = acc[g] * fac;
}

// ---- focal-spot weight b / |r - r0|^2 -----------------------------------------------------------------------
struct Field {
  int curved;
  double r0[3];
  double center[3], u_hat[3], v_hat[3], n_hat[3];
  double sdd;
  double off_u, off_v, half_u, half_v, margin_u, margin_v;
};

// b(Omega) (/ |r - r0|^2) and the filter path rho_f t(Omega) of the ray from the focal spot through (x, y, z)
// (source.py:289-430)
__device__ __forceinline__ float source_field(const Field& fd, const SourceExtras& ex, float x, float y, float z,
                                              int squared, float* filter_path) {
  const double dx = x - fd.r0[0], dy = y - fd.r0[1], dz = z - fd.r0[2];
  double t;
  if (!fd.curved) {
    const double den = dx * fd.n_hat[0] + dy * fd.n_hat[1] + dz * fd.n_hat[2];
    const double num = (fd.center[0] - fd.r0[0]) * fd.n_hat[0] + (fd.center[1] - fd.r0[1]) * fd.n_hat[1] +
                       (fd.center[2] - fd.r0[2]) * fd.n_hat[2];
    t = num / den;
  } else {  // from the cylinder's axis: |h(t d)| = SDD -> t = SDD / |h(d)|
    const double a = dx * dx + dy * dy;
    t = a > 0 ? fd.sdd / sqrt(a) : INFINITY;
  }
  double w = 0.0, path = 0.0;
  if (isfinite(t) && t > 0) {
    const double hx = fd.r0[0] + t * dx, hy = fd.r0[1] + t * dy, hz = fd.r0[2] + t * dz;
    double u, v;
    if (!fd.curved) {
      u = (hx - fd.center[0]) * fd.u_hat[0] + (hy - fd.center[1]) * fd.u_hat[1] + (hz - fd.center[2]) * fd.u_hat[2];
      v = (hx - fd.center[0]) * fd.v_hat[0] + (hy - fd.center[1]) * fd.v_hat[1] + (hz - fd.center[2]) * fd.v_hat[2];
    } else {
      const double ex_ = hx - fd.r0[0], ey = hy - fd.r0[1], ez = hz - fd.r0[2];
      const double depth = -(ex_ * fd.n_hat[0] + ey * fd.n_hat[1] + ez * fd.n_hat[2]);
      u = fd.sdd * atan2(ex_ * fd.u_hat[0] + ey * fd.u_hat[1] + ez * fd.u_hat[2], depth);
      v = fd.sdd * (ex_ * fd.v_hat[0] + ey * fd.v_hat[1] + ez * fd.v_hat[2]) / depth;
    }
    const double edge_u = fd.half_u + fd.margin_u, edge_v = fd.half_v + fd.margin_v;
    const double au = fabs(u + fd.off_u), av = fabs(v + fd.off_v);
    if (au <= edge_u && av <= edge_v) {
      w = 1.0;
    } else if (ex.n_off > 0) {  // past the field edge: the off-focal fraction of the distance to the field rectangle
      const double pu = fmax(au - edge_u, 0.0), pv = fmax(av - edge_v, 0.0);
      const double dist = sqrt(pu * pu + pv * pv);
      if (dist <= ex.off_nodes[ex.n_off - 1]) {
        int above = 0;  // nodes <= dist
        while (above < ex.n_off && ex.off_nodes[above] <= dist) ++above;
        const int i0 = min(max(above - 1, 0), ex.n_off - 1), i1 = min(above, ex.n_off - 1);
        const double span = ex.off_nodes[i1] - ex.off_nodes[i0];
        const double f = span > 0 ? fmin(fmax((dist - ex.off_nodes[i0]) / span, 0.0), 1.0) : 0.0;
        w = ex.off_values[i0] + (ex.off_values[i1] - ex.off_values[i0]) * f;
      }
    }
    if (w != 0.0 && ex.profile) w *= panel_interpolate(ex.profile, ex.rows, ex, u, v);
    if (ex.thickness) path = panel_interpolate(ex.thickness, ex.t_rows, ex, u, v) * ex.filter_density;
  }
  if (filter_path) *filter_path = (float)path;
  if (!squared) return (float)w;
  const float fx = x - (float)fd.r0[0], fy = y - (float)fd.r0[1], fz = z - (float)fd.r0[2];
  return (float)w / (fx * fx + fy * fy + fz * fz);
}

__global__ void source_weight_kernel(Field fd, SourceExtras ex, const double* __restrict__ pts,
                                     const double* __restrict__ ax_x, const double* __restrict__ ax_y,
                                     const double* __restrict__ ax_z, int gc, int gs, int64_t P, int squared,
                                     float* __restrict__ out, float* __restrict__ filter_out) {
  const int64_t p = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= P) return;
  float x, y, z;
  if (pts) {
    x = (float)pts[3 * p];
    y = (float)pts[3 * p + 1];
    z = (float)pts[3 * p + 2];
  } else {
    const int64_t row = p / ((int64_t)gc * gs), rem = p - row * (int64_t)gc * gs, col = rem / gs;
    x = (float)ax_x[col];
    y = (float)ax_y[row];
    z = (float)ax_z[rem - col * gs];
  }
  float path;
  out[p] = source_field(fd, ex, x, y, z, squared, filter_out ? &path : nullptr);
  if (filter_out) filter_out[p] = path;
}

// ---- point inputs in registers ----------------------------------------------------------------------------------
template <int kG>
__device__ __forceinline__ void load_point(const FCInputs& in, const Table& tb, int64_t v, float* rho, float* phi) {
  const int G = kG > 0 ? kG : tb.G;
  for (int m = 0; m < tb.M; ++m) rho[m] = __ldg(in.rho + (int64_t)m * in.V + v);
#pragma unroll
  for (int g = 0; g < (kG > 0 ? kG : kMaxG); ++g)
    if (g < G) phi[g] = __ldg(in.phi + (int64_t)g * in.V + v);
}

// ---- first-collision source [K, G, V] ------------------------------------------------------------------------
template <int kG>
__global__ void fc_source_kernel(FCInputs in, Table tb, PointGrid pg, const float* __restrict__ omegas, int K,
                                 int KB, float* __restrict__ out) {
  const int64_t v = (int64_t)blockIdx.x * kPoints + threadIdx.x;
  const int go = threadIdx.y;
  if (v >= in.V) return;
  int i, j, k;
  point_rcs(v, pg, i, j, k);
  float ux, uy, uz;
  primary_direction(__ldg(in.ax_x + j), __ldg(in.ax_y + i), __ldg(in.ax_z + k), in.r0x, in.r0y, in.r0z, ux, uy, uz);
  float rho[kMaxM], phi[kG > 0 ? kG : kMaxG];
  load_point<kG>(in, tb, v, rho, phi);
  const int G = kG > 0 ? kG : tb.G;
  for (int kb = 0; kb < KB; ++kb) {
    const int d = blockIdx.y * KB + kb;
    if (d >= K) break;
    const float cosine = ux * __ldg(omegas + 3 * d) + uy * __ldg(omegas + 3 * d + 1) + uz * __ldg(omegas + 3 * d + 2);
    int i0;
    float w;
    table_position(tb, cosine, i0, w);
    out[((int64_t)d * G + go) * in.V + v] = fc_value<kG>(tb, i0, w, go, rho, phi);
  }
}

// ---- LD moments of the corrected source per transport cell, cell-major [K, NC, G, 4] ---------------------------
template <int kG>
__global__ void fc_moments_kernel(FCInputs in, Table tb, PointGrid pg, const float* __restrict__ omegas, int K,
                                  const float* __restrict__ scale, const float* __restrict__ beta, float slope_scale,
                                  float* __restrict__ out, int64_t out_k_stride) {
  const int64_t NC = (int64_t)pg.Rc * pg.Cc * pg.Sc;
  const int64_t c = (int64_t)blockIdx.x * kPoints + threadIdx.x;
  const int go = threadIdx.y;
  const int d = blockIdx.y;
  if (c >= NC || d >= K) return;
  const int G = kG > 0 ? kG : tb.G;
  const int64_t csc = (int64_t)pg.Cc * pg.Sc;
  const int ic = (int)(c / csc);
  const int jc = (int)((c - (int64_t)ic * csc) / pg.Sc);
  const int kc = (int)(c - (int64_t)ic * csc - (int64_t)jc * pg.Sc);
  const float ox = __ldg(omegas + 3 * d), oy = __ldg(omegas + 3 * d + 1), oz = __ldg(omegas + 3 * d + 2);
  const int F = pg.f;
  float m0 = 0.f, mx = 0.f, my = 0.f, mz = 0.f;
  for (int a = 0; a < F; ++a) {      // rows (y)
    for (int b = 0; b < F; ++b) {    // cols (x)
      for (int e = 0; e < F; ++e) {  // slices (z)
        const int i = ic * F + a, j = jc * F + b, k = kc * F + e;
        const int64_t v = ((int64_t)i * pg.C + j) * pg.S + k;
        float ux, uy, uz;
        primary_direction(__ldg(in.ax_x + j), __ldg(in.ax_y + i), __ldg(in.ax_z + k), in.r0x, in.r0y, in.r0z, ux, uy,
                          uz);
        float rho[kMaxM], phi[kG > 0 ? kG : kMaxG];
        load_point<kG>(in, tb, v, rho, phi);
        const float cosine = ux * ox + uy * oy + uz * oz;
        int i0;
        float w;
        table_position(tb, cosine, i0, w);
        const float src = fc_value<kG>(tb, i0, w, go, rho, phi);
        const int64_t gv = (int64_t)go * in.V + v;
        const float s = src * __ldg(scale + gv) * (1.f + __ldg(beta + gv) * cosine);
        m0 += s;
        mx += s * ((2.f * b + 1.f) / F - 1.f);
        my += s * ((2.f * a + 1.f) / F - 1.f);
        mz += s * ((2.f * e + 1.f) / F - 1.f);
      }
    }
  }
  const float inv = 1.f / (float)(F * F * F);
  float4 r;
  r.x = m0 * inv;
  r.y = mx * (inv * slope_scale);
  r.z = my * (inv * slope_scale);
  r.w = mz * (inv * slope_scale);
  *reinterpret_cast<float4*>(out + d * out_k_stride + (c * G + go) * 4) = r;
}

// ---- quadrature sums, exact moments and the float64 correction factors -----------------------------------------
template <int kG>
__global__ void fc_sums_kernel(FCInputs in, Table tb, PointGrid pg, const float* __restrict__ omegas,
                               const float* __restrict__ weights, int K, const float* __restrict__ moments /*[M,2,G,G]*/,
                               float* __restrict__ sums /*[5, G, V] or null*/, float* __restrict__ scale,
                               float* __restrict__ beta) {
  const int64_t v = (int64_t)blockIdx.x * kPoints + threadIdx.x;
  const int go = threadIdx.y;
  if (v >= in.V) return;
  const int G = kG > 0 ? kG : tb.G;
  int i, j, k;
  point_rcs(v, pg, i, j, k);
  float ux, uy, uz;
  primary_direction(__ldg(in.ax_x + j), __ldg(in.ax_y + i), __ldg(in.ax_z + k), in.r0x, in.r0y, in.r0z, ux, uy, uz);
  float rho[kMaxM], phi[kG > 0 ? kG : kMaxG];
  load_point<kG>(in, tb, v, rho, phi);
  float E0 = 0.f, E1 = 0.f;
  for (int m = 0; m < tb.M; ++m) {
    const float* r0 = moments + (((int64_t)m * 2 + 0) * G + go) * G;
    const float* r1 = moments + (((int64_t)m * 2 + 1) * G + go) * G;
    float a0 = 0.f, a1 = 0.f;
    for (int gi = 0; gi <= go; ++gi) {
      a0 = fmaf(__ldg(r0 + gi), phi[gi], a0);
      a1 = fmaf(__ldg(r1 + gi), phi[gi], a1);
    }
    E0 = fmaf(rho[m], a0, E0);
    E1 = fmaf(rho[m], a1, E1);
  }
  float I0 = 0.f, I1 = 0.f, I2 = 0.f;
  for (int d = 0; d < K; ++d) {
    const float cosine = ux * __ldg(omegas + 3 * d) + uy * __ldg(omegas + 3 * d + 1) + uz * __ldg(omegas + 3 * d + 2);
    int i0;
    float w;
    table_position(tb, cosine, i0, w);
    const float ws = fc_value<kG>(tb, i0, w, go, rho, phi) * __ldg(weights + d);
    I0 += ws;
    I1 += ws * cosine;
    I2 += ws * (cosine * cosine);
  }
  const int64_t gv = (int64_t)go * in.V + v;
  if (sums) {
    const int64_t GV = (int64_t)G * in.V;
    sums[gv] = I0;
    sums[GV + gv] = I1;
    sums[2 * GV + gv] = I2;
    sums[3 * GV + gv] = E0;
    sums[4 * GV + gv] = E1;
  }
  // factors in float64 (uncollided.py:611-636)
  const double i0d = I0, i1d = I1, i2d = I2, e0 = E0, e1 = E1;
  const bool pos = e0 > 0;
  const double c = pos ? e1 / e0 : 0.0;
  const double den = i2d - c * i1d;
  const bool ok = pos && fabs(den) > 1e-12 * fabs(i0d);
  double b = ok ? (c * i0d - i1d) / den : 0.0;
  b = fmin(fmax(b, -1.0), 1.0);
  const double d0 = i0d + b * i1d;
  scale[gv] = (float)(d0 > 0 ? e0 / d0 : 1.0);
  beta[gv] = (float)b;
}

// ---- sampling correction over the sweep directions, with the source values kept -----------------------------------
// A block is 32 points by the G groups and walks all K sweep directions, in the order of their cosine with the
// block's first point so that each batch of kFcBatch directions touches few table nodes (the window); it sums
// I0, I1, I2 per (point, group), stores S_FC(direction, group, point) in cache [K, G, V] when given (the LD moments
// of the sweep's source read it back instead of evaluating the table again), and forms E0, E1 and the float64
// factors as the reference does.
constexpr int kFcBatch = 16;
constexpr int kMaxSorted = 1024;

template <int kGP, int kMM>
__global__ void __launch_bounds__(kEmitPoints * kGP) fc_correction_kernel(
    FCInputs in, Table tb, PointGrid pg, const float* __restrict__ omegas, const float* __restrict__ weights, int K,
    const float* __restrict__ moments /*[M, 2, G, G]*/, float* __restrict__ sums /*[5, G, V] or null*/,
    float* __restrict__ scale, float* __restrict__ beta, float* __restrict__ cache /*[K, G, V] or null*/) {
  extern __shared__ float4 s_dyn4[];
  float* s_tab = reinterpret_cast<float*>(s_dyn4);
  __shared__ float s_key[kMaxSorted];
  __shared__ int s_order[kMaxSorted];
  __shared__ float s_om[kFcBatch][3];
  __shared__ float s_w[kFcBatch];
  __shared__ int s_d[kFcBatch];
  __shared__ int s_range[2][32];
  __shared__ int s_window[2];
  __shared__ float s_u0[3];
  const int G = tb.G;
  const int g = threadIdx.y, lane = threadIdx.x;
  const int nthreads = kEmitPoints * G, tid = g * kEmitPoints + lane;
  const int64_t v = (int64_t)blockIdx.x * kEmitPoints + lane;
  const bool valid = v < in.V;
  float rho[kMM], phi[kGP];
  float ux = 0.f, uy = 0.f, uz = 0.f;
#pragma unroll
  for (int q = 0; q < kGP; ++q) phi[q] = 0.f;
#pragma unroll
  for (int m = 0; m < kMM; ++m) rho[m] = 0.f;
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
  }
  // exact l = 0, 1 moments of the source (downscatter rows of the moment table)
  float E0 = 0.f, E1 = 0.f;
  for (int m = 0; m < tb.M; ++m) {
    const float* r0 = moments + (((int64_t)m * 2 + 0) * G + g) * G;
    const float* r1 = moments + (((int64_t)m * 2 + 1) * G + g) * G;
    float a0 = 0.f, a1 = 0.f;
    for (int gi = 0; gi <= g; ++gi) {
      a0 = fmaf(__ldg(r0 + gi), phi[gi < kGP ? gi : 0], a0);
      a1 = fmaf(__ldg(r1 + gi), phi[gi < kGP ? gi : 0], a1);
    }
    E0 = fmaf(rho[m], a0, E0);
    E1 = fmaf(rho[m], a1, E1);
  }
  // directions in the order of their cosine with the block's first point
  if (tid == 0) {
    s_u0[0] = ux;
    s_u0[1] = uy;
    s_u0[2] = uz;
  }
  __syncthreads();
  const bool sorted = K <= kMaxSorted;
  if (sorted) {
    for (int d = tid; d < K; d += nthreads)
      s_key[d] = s_u0[0] * __ldg(omegas + 3 * d) + s_u0[1] * __ldg(omegas + 3 * d + 1) +
                 s_u0[2] * __ldg(omegas + 3 * d + 2);
    __syncthreads();
    for (int d = tid; d < K; d += nthreads) {
      const float key = s_key[d];
      int rank = 0;
      for (int q = 0; q < K; ++q) {
        const float other = s_key[q];
        rank += (other < key) || (other == key && q < d);
      }
      s_order[rank] = d;
    }
    __syncthreads();
  }
  float I0 = 0.f, I1 = 0.f, I2 = 0.f;
  for (int b0 = 0; b0 < K; b0 += kFcBatch) {
    const int nb = min(kFcBatch, K - b0);
    if (tid < nb) {
      const int d = sorted ? s_order[b0 + tid] : b0 + tid;
      s_d[tid] = d;
      s_om[tid][0] = __ldg(omegas + 3 * d);
      s_om[tid][1] = __ldg(omegas + 3 * d + 1);
      s_om[tid][2] = __ldg(omegas + 3 * d + 2);
      s_w[tid] = __ldg(weights + d);
    }
    __syncthreads();
    stage_window(tb, valid, ux, uy, uz, s_om, nb, g, G, g, G, tid, nthreads, s_range, s_window, s_tab);
    const int win_lo = s_window[0];
    if (valid) {
      for (int i = 0; i < nb; ++i) {
        const float cosine = ux * s_om[i][0] + uy * s_om[i][1] + uz * s_om[i][2];
        int i0;
        float w;
        table_position(tb, cosine, i0, w);
        const float S = fc_group<kGP, kMM>(tb, s_tab, win_lo, i0, w, g, rho, phi);
        const float ws = S * s_w[i];
        I0 += ws;
        I1 += ws * cosine;
        I2 += ws * (cosine * cosine);
        if (cache != nullptr) cache[((int64_t)s_d[i] * G + g) * in.V + v] = S;
      }
    }
    __syncthreads();  // the batch's directions and window are replaced next
  }
  if (!valid) return;
  const int64_t gv = (int64_t)g * in.V + v;
  if (sums) {
    const int64_t GV = (int64_t)G * in.V;
    sums[gv] = I0;
    sums[GV + gv] = I1;
    sums[2 * GV + gv] = I2;
    sums[3 * GV + gv] = E0;
    sums[4 * GV + gv] = E1;
  }
  // factors in float64 (uncollided.py:611-636)
  const double i0d = I0, i1d = I1, i2d = I2, e0 = E0, e1 = E1;
  const bool pos = e0 > 0;
  const double c = pos ? e1 / e0 : 0.0;
  const double den = i2d - c * i1d;
  const bool ok = pos && fabs(den) > 1e-12 * fabs(i0d);
  double b = ok ? (c * i0d - i1d) / den : 0.0;
  b = fmin(fmax(b, -1.0), 1.0);
  const double d0 = i0d + b * i1d;
  scale[gv] = (float)(d0 > 0 ? e0 / d0 : 1.0);
  beta[gv] = (float)b;
}

// ---- sampling correction, one thread per (point, direction) with all of its groups --------------------------------
// The correction of fc_correction_kernel with the emission's thread layout: a block is 32 points (the lanes) by
// kFcWarps warps; per batch of kFcDirBatch directions (in the order of their cosine with the block's first point, so
// that a batch touches few table nodes) warp w takes the batch's directions w, w + kFcWarps, ... . A thread forms the
// cosine and the table position of its (point, direction) once and the source of every group from float4 rows
// (incoming groups at or above the outgoing one), adds the weighted source to its own partial sums I0, I1, I2 and
// writes the source values to the cache; the warps' partial sums are then added in warp order, and the float64
// factors formed as fc_correction_kernel forms them. The sums differ from fc_correction_kernel's at rounding level
// (another order of the same terms).
// 3 blocks of 256 threads per SM (80 registers): at 2 (128 registers) the table gathers' latency went unhidden
// Directions of a batch, and the bytes of its window: a batch of the sorted directions has to fit its window, or every
// row is gathered from global memory. 120 directions over the sphere take 401 nodes, 24 of them 80, and the points of
// a block spread a node over up to 28 more: 120 nodes of two materials and 8 groups are 64 KB. (32 directions in 48
// KB, 88 nodes, never fitted: 1.77 ms at 64^3 points, 8 groups and 120 directions, now 0.75.)
// kWindow: up to 8 groups the window is taken from 4 on, where kFcWindowNodes nodes of all materials fit it (8 directions of
// 120 take 27 of 401 nodes, and 32 points along a column 25.6 long spread them over up to 104 from a source at 60). With fewer
// groups filling it costs more than it saves, and a batch that does not fit after all gathers its rows without the L1 that the
// window holds; so a block whose batch does not fit goes on in batches of one direction per warp (and gathers those
// that don't fit either; going back to whole batches for them took registers, 246 -> 262 us below). us at 32^3 points, 120
// directions, the source at 100 / 60, without the window or with one of 24 directions or none -> now: two materials, 8
// groups 546 / 786 -> 246 / 722, 7 groups 525 / 1201 -> 179 / 469, 5 groups 208 / 443 -> 126 / 179, one group 82 / 43 -> 23 / 23;
// three materials and 7 groups, no window, 1322 / 2008 -> 805 / 904.
constexpr int kFcWarps = 8;
// Where the table has more than kFcNodesPerDirection nodes for each direction, the nodes of 8 directions are too many to copy for
// them, and the whole batch gathers: 11 groups, 32 directions 135 us, in batches of 8 219; 5 groups, 80 directions 278 / 309.
constexpr int kFcWindowNodes = 140, kFcNodesPerDirection = 4;
__host__ __device__ constexpr int fc_batch(int gp, bool window) { return window ? (gp > 8 ? 16 : 24) : 32; }
__host__ __device__ constexpr int fc_window_bytes(int gp) { return gp > 8 ? 176 * 1024 : 64 * 1024; }
__host__ __device__ constexpr int fc_sums_bytes(int gp) { return kFcWarps * 3 * gp * 32 * 4; }

template <int kGP, int kMM, bool kVec, bool kExact, bool kWindow>  // kExact: kGP groups and kMM materials
__global__ void __launch_bounds__(32 * kFcWarps, kGP > 8 ? 1 : 3) fc_correction_warps_kernel(
    FCInputs in, Table tb, PointGrid pg, const float* __restrict__ omegas, const float* __restrict__ weights, int K,
    const float* __restrict__ moments /*[M, 2, G, G]*/, float* __restrict__ sums /*[5, G, V] or null*/,
    float* __restrict__ scale, float* __restrict__ beta, float* __restrict__ cache /*[K, G, V] or null*/) {
  constexpr int nthreads = 32 * kFcWarps, kFcDirBatch = fc_batch(kGP, kWindow);
  extern __shared__ float4 s_dyn4[];
  float* s_tab = reinterpret_cast<float*>(s_dyn4);
  __shared__ float s_key[kMaxSorted];
  __shared__ int s_order[kMaxSorted];
  __shared__ float s_om[kFcDirBatch][3];
  __shared__ float s_w[kFcDirBatch];
  __shared__ int s_d[kFcDirBatch];
  __shared__ int s_range[2][32];
  __shared__ int s_window[2];
  __shared__ float s_u0[3];
  // after the direction loop the window's shared memory holds the warps' partial sums [kFcWarps][3][kGP][32]
  static_assert(fc_sums_bytes(kGP) <= fc_window_bytes(kGP), "partial sums exceed the window");
  const int G = kExact ? kGP : tb.G, M = kExact ? kMM : tb.M;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int64_t v = (int64_t)blockIdx.x * 32 + lane;
  const bool valid = v < in.V;
  float rho[kMM], phi[kGP];
  float ux = 0.f, uy = 0.f, uz = 0.f;
#pragma unroll
  for (int q = 0; q < kGP; ++q) phi[q] = 0.f;
#pragma unroll
  for (int m = 0; m < kMM; ++m) rho[m] = 0.f;
  if (valid) {
    int i, j, k;
    point_rcs(v, pg, i, j, k);
    primary_direction(__ldg(in.ax_x + j), __ldg(in.ax_y + i), __ldg(in.ax_z + k), in.r0x, in.r0y, in.r0z, ux, uy, uz);
#pragma unroll
    for (int m = 0; m < kMM; ++m)
      if (m < M) rho[m] = __ldg(in.rho + (int64_t)m * in.V + v);
#pragma unroll
    for (int q = 0; q < kGP; ++q)
      if (q < G) phi[q] = __ldg(in.phi + (int64_t)q * in.V + v);
  }
  if (tid == 0) {
    s_u0[0] = ux;
    s_u0[1] = uy;
    s_u0[2] = uz;
  }
  __syncthreads();
  const bool sorted = K <= kMaxSorted;
  if (sorted) {
    for (int d = tid; d < K; d += nthreads)
      s_key[d] = s_u0[0] * __ldg(omegas + 3 * d) + s_u0[1] * __ldg(omegas + 3 * d + 1) +
                 s_u0[2] * __ldg(omegas + 3 * d + 2);
    __syncthreads();
    for (int d = tid; d < K; d += nthreads) {
      const float key = s_key[d];
      int rank = 0;
      for (int q = 0; q < K; ++q) {
        const float other = s_key[q];
        rank += (other < key) || (other == key && q < d);
      }
      s_order[rank] = d;
    }
    __syncthreads();
  }
  float I0[kGP], I1[kGP], I2[kGP];
#pragma unroll
  for (int q = 0; q < kGP; ++q) I0[q] = I1[q] = I2[q] = 0.f;
  const int NS = window_node_stride(M, G);
  const int W = window_nodes(M, G, fc_window_bytes(kGP));
  int held = 0, held_end = 0;  // the nodes in the window
  int most = kFcDirBatch, nb;
  for (int b0 = 0; b0 < K; b0 += nb) {
    nb = min(most, K - b0);
    if (tid < nb) {
      const int d = sorted ? s_order[b0 + tid] : b0 + tid;
      s_d[tid] = d;
      s_om[tid][0] = __ldg(omegas + 3 * d);
      s_om[tid][1] = __ldg(omegas + 3 * d + 1);
      s_om[tid][2] = __ldg(omegas + 3 * d + 2);
      s_w[tid] = __ldg(weights + d);
    }
    __syncthreads();
    // the window's slots are a ring over the nodes, node n in slot n % W: the batches' nodes move up the table, and only
    // those that no batch before has brought are copied
    bool windowed = false;
    int first_node = 0, first_slot = 0;
    if constexpr (kWindow) {
      window_range(tb, valid, ux, uy, uz, s_om, nb, warp, kFcWarps, warp, kFcWarps, tid, s_range, s_window);
      first_node = s_window[0];
      const int end = first_node + s_window[1];  // all of it uniform over the block
      windowed = s_window[1] <= W;
      if (!windowed && nb > kFcWarps && tb.N <= kFcNodesPerDirection * K) {
        most = kFcWarps;
        nb = 0;
        continue;
      }
      if (windowed) {
        int from = held_end;
        if (first_node < held || first_node > held_end || max(end, held_end) - first_node > W) from = held = first_node;
        held_end = from == first_node ? end : max(end, held_end);
        held = max(held, held_end - W);
        first_slot = first_node % W;
        const int slot = from % W, n = held_end - from, straight = min(n, W - slot);
        if (n > 0) {
          copy_window<kExact ? kGP : 0>(tb, from, straight, warp, kFcWarps, tid, nthreads, s_tab + slot * NS);
          if (n > straight)
            copy_window<kExact ? kGP : 0>(tb, from + straight, n - straight, warp, kFcWarps, tid, nthreads, s_tab);
          __syncthreads();
        }
      }
    }
    // one body per place of the rows: a pointer to either is a generic one, whose loads are no shared-memory loads
    auto batch = [&](auto windowed) {
      constexpr bool kWin = decltype(windowed)::value;
      for (int i = warp; i < nb; i += kFcWarps) {
        const float cosine = ux * s_om[i][0] + uy * s_om[i][1] + uz * s_om[i][2];
        int i0;
        float w;
        table_position(tb, cosine, i0, w);
        int slot0 = i0 - first_node + first_slot;
        if (slot0 >= W) slot0 -= W;
        const int slot1 = slot0 + 1 == W ? 0 : slot0 + 1;
        float S[kGP];
#pragma unroll
        for (int q = 0; q < kGP; ++q) S[q] = 0.f;
#pragma unroll
        for (int m = 0; m < kMM; ++m) {
          const float r = rho[m];
          if (m >= M || r == 0.f) continue;
          const float* row0 = kWin ? s_tab + slot0 * NS + m * G * G : tb.t + ((int64_t)m * tb.N + i0) * G * G;
          const float* row1 = kWin ? s_tab + slot1 * NS + m * G * G : row0 + G * G;
#pragma unroll
          for (int g = 0; g < kGP; ++g) {
            if (g >= G) break;
            const float a0 = dot_lower<kGP, kVec, kWin>(row0 + g * G, phi, g);
            const float a1 = dot_lower<kGP, kVec, kWin>(row1 + g * G, phi, g);
            S[g] = fmaf(r, a0 + (a1 - a0) * w, S[g]);
          }
        }
        const float wt = s_w[i], c2 = cosine * cosine;
        const int64_t d = s_d[i];
#pragma unroll
        for (int g = 0; g < kGP; ++g) {
          if (g >= G) break;
          const float ws = S[g] * wt;
          I0[g] += ws;
          I1[g] += ws * cosine;
          I2[g] += ws * c2;
          if (cache != nullptr) cache[(d * G + g) * in.V + v] = S[g];
        }
      }
    };
    if (valid) {
      if (kWindow && windowed) batch(std::bool_constant<kWindow>{});
      else batch(std::false_type{});
    }
    __syncthreads();  // the batch's directions and window are replaced next
  }
  float* s_part = s_tab;  // free: the last batch's barrier above ended every read of the window
#pragma unroll
  for (int q = 0; q < kGP; ++q) {
    s_part[((warp * 3 + 0) * kGP + q) * 32 + lane] = I0[q];
    s_part[((warp * 3 + 1) * kGP + q) * 32 + lane] = I1[q];
    s_part[((warp * 3 + 2) * kGP + q) * 32 + lane] = I2[q];
  }
  __syncthreads();
  // warp g forms the factors of group g of its lane's point (every warp holds the point's densities and fluence)
  for (int g = warp; g < G && g < kGP; g += kFcWarps) {
    if (!valid) break;
    float i0s = 0.f, i1s = 0.f, i2s = 0.f;
#pragma unroll
    for (int q = 0; q < kFcWarps; ++q) {
      i0s += s_part[((q * 3 + 0) * kGP + g) * 32 + lane];
      i1s += s_part[((q * 3 + 1) * kGP + g) * 32 + lane];
      i2s += s_part[((q * 3 + 2) * kGP + g) * 32 + lane];
    }
    // exact l = 0, 1 moments of the source (downscatter rows of the moment table)
    float E0 = 0.f, E1 = 0.f;
    for (int m = 0; m < M && m < kMM; ++m) {
      const float* r0 = moments + (((int64_t)m * 2 + 0) * G + g) * G;
      const float* r1 = moments + (((int64_t)m * 2 + 1) * G + g) * G;
      float a0 = 0.f, a1 = 0.f;
      for (int gi = 0; gi <= g; ++gi) {
        a0 = fmaf(__ldg(r0 + gi), phi[gi], a0);
        a1 = fmaf(__ldg(r1 + gi), phi[gi], a1);
      }
      E0 = fmaf(rho[m], a0, E0);
      E1 = fmaf(rho[m], a1, E1);
    }
    const int64_t gv = (int64_t)g * in.V + v;
    if (sums) {
      const int64_t GV = (int64_t)G * in.V;
      sums[gv] = i0s;
      sums[GV + gv] = i1s;
      sums[2 * GV + gv] = i2s;
      sums[3 * GV + gv] = E0;
      sums[4 * GV + gv] = E1;
    }
    // factors in float64 (uncollided.py:611-636)
    const double i0d = i0s, i1d = i1s, i2d = i2s, e0 = E0, e1 = E1;
    const bool pos = e0 > 0;
    const double c = pos ? e1 / e0 : 0.0;
    const double den = i2d - c * i1d;
    const bool ok = pos && fabs(den) > 1e-12 * fabs(i0d);
    double b = ok ? (c * i0d - i1d) / den : 0.0;
    b = fmin(fmax(b, -1.0), 1.0);
    const double d0 = i0d + b * i1d;
    scale[gv] = (float)(d0 > 0 ? e0 / d0 : 1.0);
    beta[gv] = (float)b;
  }
}

// ---- LD moments of the corrected source from the kept source values ---------------------------------------------
// A block is 32 cells by the G groups by kFcBatch directions of the chunk: S_FC read from cache [K, G, V] at the
// chunk direction's cache_index, corrected (scale (1 + beta cos)) and restricted to the cell's LD moments; the
// block's [cells, G, 4] tile goes out through shared memory as contiguous float4 rows.
// kF: the points per cell axis (0: pg.f of them). A point's primary direction and correction factors are formed once for
// all directions where they fit registers (kF of 1 and 2), and with one point per cell eight directions' values are in
// flight before their stores: 1.85 -> 0.82 ms at 64^3 points, 8 groups and 120 directions, 90 % of a copy's bandwidth.
template <int kGP, int kF>
__global__ void __launch_bounds__(kEmitPoints * kGP) fc_moments_cached_kernel(
    FCInputs in, PointGrid pg, const float* __restrict__ omegas, int K, const float* __restrict__ cache,
    const int32_t* __restrict__ cache_index, const float* __restrict__ scale, const float* __restrict__ beta,
    float slope_scale, float* __restrict__ out, int64_t out_k_stride) {
  // thread (cell, group) with the group fastest: a warp's float4 outputs [cell, group, 4] are contiguous
  const int G = (int)(blockDim.y);
  const int tid = threadIdx.y * kEmitPoints + threadIdx.x;
  const int lane = tid / G, g = tid - lane * G;
  const int64_t NC = (int64_t)pg.Rc * pg.Cc * pg.Sc;
  const int64_t c0 = (int64_t)blockIdx.x * kEmitPoints;
  const int64_t c = c0 + lane;
  const bool valid = c < NC;
  const int F = kF > 0 ? kF : pg.f;
  int ic = 0, jc = 0, kc = 0;
  if (valid) {
    const int64_t csc = (int64_t)pg.Cc * pg.Sc;
    ic = (int)(c / csc);
    jc = (int)((c - (int64_t)ic * csc) / pg.Sc);
    kc = (int)(c - (int64_t)ic * csc - (int64_t)jc * pg.Sc);
  }
  const float inv = 1.f / (float)(F * F * F);
  const int dlast = min(K, (int)(blockIdx.y + 1) * kFcBatch);
  if constexpr (kF == 1) {
    float ux = 0.f, uy = 0.f, uz = 0.f, sc = 0.f, be = 0.f;
    const int64_t v = ((int64_t)ic * pg.C + jc) * pg.S + kc;
    if (valid) {
      primary_direction(__ldg(in.ax_x + jc), __ldg(in.ax_y + ic), __ldg(in.ax_z + kc), in.r0x, in.r0y, in.r0z, ux, uy, uz);
      sc = __ldg(scale + (int64_t)g * in.V + v);
      be = __ldg(beta + (int64_t)g * in.V + v);
    }
    constexpr int kU = 8;
    const float* src = cache + (int64_t)g * in.V + v;
    float4* dst = reinterpret_cast<float4*>(out) + c * G + g;
    for (int d0 = blockIdx.y * kFcBatch; d0 < dlast; d0 += kU) {
      float x[kU];
#pragma unroll
      for (int q = 0; q < kU; ++q)
        x[q] = valid && d0 + q < dlast ? __ldg(src + (int64_t)__ldg(cache_index + d0 + q) * G * in.V) : 0.f;
#pragma unroll
      for (int q = 0; q < kU; ++q) {
        const int d = d0 + q;
        if (!valid || d >= dlast) break;
        const float cosine = ux * __ldg(omegas + 3 * d) + uy * __ldg(omegas + 3 * d + 1) + uz * __ldg(omegas + 3 * d + 2);
        dst[d * (out_k_stride / 4)] = make_float4(x[q] * sc * (1.f + be * cosine) * inv, 0.f, 0.f, 0.f);
      }
    }
    return;
  }
  constexpr int kPoints3 = kF == 2 ? 8 : 1;
  float u[kPoints3][3], sc[kPoints3], be[kPoints3];
  if (kF == 2 && valid) {
#pragma unroll
    for (int p = 0; p < kPoints3; ++p) {
      const int i = ic * 2 + (p >> 2), j = jc * 2 + ((p >> 1) & 1), k = kc * 2 + (p & 1);
      const int64_t gv = (int64_t)g * in.V + ((int64_t)i * pg.C + j) * pg.S + k;
      primary_direction(__ldg(in.ax_x + j), __ldg(in.ax_y + i), __ldg(in.ax_z + k), in.r0x, in.r0y, in.r0z, u[p][0],
                        u[p][1], u[p][2]);
      sc[p] = __ldg(scale + gv);
      be[p] = __ldg(beta + gv);
    }
  }
  for (int d = blockIdx.y * kFcBatch; d < dlast; ++d) {
    if (!valid) break;
    float4 r = make_float4(0.f, 0.f, 0.f, 0.f);
    const float ox = __ldg(omegas + 3 * d), oy = __ldg(omegas + 3 * d + 1), oz = __ldg(omegas + 3 * d + 2);
    const float* src = cache + (int64_t)__ldg(cache_index + d) * G * in.V + (int64_t)g * in.V;
    {
      float m0 = 0.f, mx = 0.f, my = 0.f, mz = 0.f;
#pragma unroll
      for (int a = 0; a < F; ++a) {      // rows (y)
#pragma unroll
        for (int b = 0; b < F; ++b) {    // cols (x)
#pragma unroll
          for (int e = 0; e < F; ++e) {  // slices (z)
            const int i = ic * F + a, j = jc * F + b, k = kc * F + e;
            const int64_t v = ((int64_t)i * pg.C + j) * pg.S + k;
            float ux, uy, uz, scale_v, beta_v;
            if constexpr (kF == 2) {
              const int p = 4 * a + 2 * b + e;
              ux = u[p][0], uy = u[p][1], uz = u[p][2], scale_v = sc[p], beta_v = be[p];
            } else {
              primary_direction(__ldg(in.ax_x + j), __ldg(in.ax_y + i), __ldg(in.ax_z + k), in.r0x, in.r0y, in.r0z,
                                ux, uy, uz);
              scale_v = __ldg(scale + (int64_t)g * in.V + v);
              beta_v = __ldg(beta + (int64_t)g * in.V + v);
            }
            const float cosine = ux * ox + uy * oy + uz * oz;
            const float s = __ldg(src + v) * scale_v * (1.f + beta_v * cosine);
            m0 += s;
            mx += s * ((2.f * b + 1.f) / F - 1.f);
            my += s * ((2.f * a + 1.f) / F - 1.f);
            mz += s * ((2.f * e + 1.f) / F - 1.f);
          }
        }
      }
      r.x = m0 * inv;
      r.y = mx * (inv * slope_scale);
      r.z = my * (inv * slope_scale);
      r.w = mz * (inv * slope_scale);
    }
    reinterpret_cast<float4*>(out + d * out_k_stride)[c * G + g] = r;
  }
}

// The means alone, for one point per cell (whose LD slopes vanish): out [K, NC, G] with out_k_stride floats between
// directions. A block is 32 cells by the G groups and 16 directions: it reads the cached source rows [g][cells] whole
// (a warp per group) and writes each direction's [cells, G] run whole, through shared memory.
template <int kGP>
__global__ void __launch_bounds__(kEmitPoints * kGP) fc_means_kernel(
    FCInputs in, PointGrid pg, const float* __restrict__ omegas, int K, const float* __restrict__ cache,
    const int32_t* __restrict__ cache_index, const float* __restrict__ scale, const float* __restrict__ beta,
    float* __restrict__ out, int64_t out_k_stride) {
  constexpr int kPass = kGP >= 16 ? 128 / kGP : kFcBatch;  // directions per shared-memory pass (16 KB)
  __shared__ float s_out[kPass][kEmitPoints * kGP];
  const int G = (int)blockDim.y;
  const int x = threadIdx.x, g = threadIdx.y, tid = g * kEmitPoints + x;
  const int64_t c0 = (int64_t)blockIdx.x * kEmitPoints;
  const int64_t c = c0 + x;  // one point per cell: the cell is the point
  const int n = (int)min((int64_t)kEmitPoints, in.V - c0);  // cells of this block
  float ux = 0.f, uy = 0.f, uz = 0.f, sc = 0.f, be = 0.f;
  if (x < n) {
    int i, j, k;
    point_rcs(c, pg, i, j, k);
    primary_direction(__ldg(in.ax_x + j), __ldg(in.ax_y + i), __ldg(in.ax_z + k), in.r0x, in.r0y, in.r0z, ux, uy, uz);
    sc = __ldg(scale + (int64_t)g * in.V + c);
    be = __ldg(beta + (int64_t)g * in.V + c);
  }
  const int d0 = blockIdx.y * kFcBatch, dlast = min(K, d0 + kFcBatch);
  for (int p0 = d0; p0 < dlast; p0 += kPass) {
    const int np = min(kPass, dlast - p0);
    // eight directions' cache loads in flight per thread before their products and shared-memory stores
    constexpr int kU = 8;
    for (int q0 = 0; q0 < np; q0 += kU) {
      float v[kU];
#pragma unroll
      for (int u = 0; u < kU; ++u)
        v[u] = (x < n && q0 + u < np)
                   ? __ldg(cache + ((int64_t)__ldg(cache_index + p0 + q0 + u) * G + g) * in.V + c)
                   : 0.f;
#pragma unroll
      for (int u = 0; u < kU; ++u) {
        if (q0 + u >= np) break;
        const int d = p0 + q0 + u;
        float r = 0.f;
        if (x < n) {
          const float ox = __ldg(omegas + 3 * d), oy = __ldg(omegas + 3 * d + 1), oz = __ldg(omegas + 3 * d + 2);
          const float cosine = ux * ox + uy * oy + uz * oz;
          r = v[u] * sc * (1.f + be * cosine);
        }
        s_out[q0 + u][x * G + g] = r;
      }
    }
    __syncthreads();
    for (int q = 0; q < np; ++q)
      if (tid < n * G) out[(int64_t)(p0 + q) * out_k_stride + c0 * G + tid] = s_out[q][tid];
    __syncthreads();
  }
}

#define CITRUS_G_DISPATCH(G, KERNEL, GRID, BLOCK, SMEM, STREAM, ...)                         \
  switch (G) {                                                                                \
    case 1: KERNEL<1><<<GRID, BLOCK, SMEM, STREAM>>>(__VA_ARGS__); break;                    \
    case 4: KERNEL<4><<<GRID, BLOCK, SMEM, STREAM>>>(__VA_ARGS__); break;                    \
    case 8: KERNEL<8><<<GRID, BLOCK, SMEM, STREAM>>>(__VA_ARGS__); break;                    \
    case 16: KERNEL<16><<<GRID, BLOCK, SMEM, STREAM>>>(__VA_ARGS__); break;                  \
    default: KERNEL<0><<<GRID, BLOCK, SMEM, STREAM>>>(__VA_ARGS__); break;                   \
  }                                                                                           \
  note_launches();

}  // namespace
}  // namespace citrus

using namespace citrus;

extern "C" int citrus_group_transmission(const float* path, int64_t num_materials, int64_t num_points,
                                         const float* fine_mu, const float* fine_weight, const int32_t* fine_group,
                                         int64_t num_fine, int64_t num_groups, const float* filter_path,
                                         const float* filter_mu, const float* factor, float* out, void* stream) {
  CITRUS_REQUIRE(path && fine_mu && fine_weight && fine_group && out, "citrus_group_transmission: null pointer");
  CITRUS_REQUIRE(num_materials >= 1 && num_materials <= kMaxM && num_groups >= 1 && num_groups <= kMaxG &&
                     num_fine >= 1 && num_points >= 0,
                 "citrus_group_transmission: bad sizes (materials %lld, groups %lld, fine %lld)",
                 (long long)num_materials, (long long)num_groups, (long long)num_fine);
  CITRUS_REQUIRE((filter_path == nullptr) == (filter_mu == nullptr),
                 "citrus_group_transmission: filter_path and filter_mu go together");
  const size_t smem = (size_t)(num_materials * num_fine + 2 * num_fine) * sizeof(float) + num_fine * sizeof(int);
  CITRUS_REQUIRE(smem <= 96 * 1024, "citrus_group_transmission: %lld fine energies too many", (long long)num_fine);
  if (num_points == 0) return CITRUS_OK;
  if (smem > 48 * 1024)
    cudaFuncSetAttribute(transmission_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  transmission_kernel<<<(unsigned)cdiv(num_points, 128), 128, smem, as_stream(stream)>>>(
      path, (int)num_materials, num_points, fine_mu, fine_weight, fine_group, (int)num_fine, (int)num_groups,
      filter_path, filter_mu, factor, out);
  note_launches();
  return launch_status("citrus_group_transmission");
}

extern "C" int citrus_source_field(const double* field, const double* panel, const double* profile,
                                   const double* thickness, int64_t thickness_rows, double filter_density,
                                   const double* off_focal_nodes, const double* off_focal_values,
                                   int64_t num_off_focal, const double* points, const double* axis_x,
                                   const double* axis_y, const double* axis_z, const int64_t* point_dims,
                                   int64_t num_points, int32_t divide_by_distance_squared, float* out,
                                   float* filter_path_out, void* stream) {
  CITRUS_REQUIRE(field && out, "citrus_source_field: null pointer");
  CITRUS_REQUIRE(points || (axis_x && axis_y && axis_z && point_dims), "citrus_source_field: no points");
  CITRUS_REQUIRE(num_points >= 0 && num_off_focal >= 0, "citrus_source_field: negative size");
  CITRUS_REQUIRE((num_off_focal == 0) == (off_focal_nodes == nullptr) &&
                     (off_focal_nodes == nullptr) == (off_focal_values == nullptr),
                 "citrus_source_field: the off-focal nodes and values go together with their count");
  CITRUS_REQUIRE((thickness == nullptr) == (filter_path_out == nullptr),
                 "citrus_source_field: the filter thickness and the filter-path output go together");
  CITRUS_REQUIRE(!(profile || thickness) || panel, "citrus_source_field: a profile or a filter needs the panel");
  Field fd;
  fd.curved = field[0] != 0.0;
  for (int a = 0; a < 3; ++a) {
    fd.r0[a] = field[1 + a];
    fd.center[a] = field[4 + a];
    fd.u_hat[a] = field[7 + a];
    fd.v_hat[a] = field[10 + a];
    fd.n_hat[a] = field[13 + a];
  }
  fd.sdd = field[16];
  fd.off_u = field[17];
  fd.off_v = field[18];
  fd.half_u = field[19];
  fd.half_v = field[20];
  fd.margin_u = field[21];
  fd.margin_v = field[22];
  SourceExtras ex{};
  ex.profile = profile;
  ex.thickness = thickness;
  ex.off_nodes = off_focal_nodes;
  ex.off_values = off_focal_values;
  ex.n_off = (int)num_off_focal;
  ex.filter_density = filter_density;
  if (panel) {
    ex.rows = (int)panel[0];
    ex.channels = (int)panel[1];
    ex.d_row = panel[2];
    ex.d_ch = panel[3];
    ex.off_row = panel[4];
    ex.off_ch = panel[5];
    CITRUS_REQUIRE(ex.rows >= 1 && ex.channels >= 1 && ex.d_row > 0 && ex.d_ch > 0,
                   "citrus_source_field: bad panel");
  }
  ex.t_rows = (int)thickness_rows;
  CITRUS_REQUIRE(!thickness || thickness_rows == 1 || thickness_rows == ex.rows,
                 "citrus_source_field: the filter thickness must have 1 or all rows");
  int gc = 1, gs = 1;
  if (!points) {
    gc = (int)point_dims[1];
    gs = (int)point_dims[2];
  }
  if (num_points == 0) return CITRUS_OK;
  source_weight_kernel<<<(unsigned)cdiv(num_points, 128), 128, 0, as_stream(stream)>>>(
      fd, ex, points, axis_x, axis_y, axis_z, gc, gs, num_points, divide_by_distance_squared, out, filter_path_out);
  note_launches();
  return launch_status("citrus_source_field");
}

extern "C" int citrus_source_weight(const double* field, const double* points, const double* axis_x,
                                    const double* axis_y, const double* axis_z, const int64_t* point_dims,
                                    int64_t num_points, int32_t divide_by_distance_squared, float* out, void* stream) {
  return citrus_source_field(field, nullptr, nullptr, nullptr, 0, 0.0, nullptr, nullptr, 0, points, axis_x, axis_y,
                             axis_z, point_dims, num_points, divide_by_distance_squared, out, nullptr, stream);
}

extern "C" int citrus_first_collision_source(const float* rho, int64_t num_materials, const float* phi,
                                             int64_t num_groups, const float* axes, const int64_t* point_dims,
                                             const double* focal_spot, const float* table, int64_t num_eta,
                                             double eta_lo, double eta_hi, const float* omegas,
                                             int64_t num_directions, float* out, void* stream) {
  int st = check_table(table, num_materials, num_eta, num_groups);
  if (st) return st;
  CITRUS_REQUIRE(rho && phi && axes && point_dims && focal_spot && omegas && out,
                 "citrus_first_collision_source: null pointer");
  const int64_t V = point_dims[0] * point_dims[1] * point_dims[2];
  if (V == 0 || num_directions == 0) return CITRUS_OK;
  const FCInputs in = make_inputs(rho, phi, axes, V, focal_spot, point_dims);
  const Table tb = make_table(table, num_materials, num_eta, num_groups, eta_lo, eta_hi);
  const PointGrid pg = make_grid(point_dims, 1);
  const int G = (int)num_groups, K = (int)num_directions, KB = 4;
  dim3 grid((unsigned)cdiv(V, kPoints), (unsigned)cdiv(K, KB)), block(kPoints, G);
  CITRUS_G_DISPATCH(G, fc_source_kernel, grid, block, 0, as_stream(stream), in, tb, pg, omegas, K, KB, out)
  return launch_status("citrus_first_collision_source");
}

namespace citrus {
namespace {

template <int kGP, int kMM>
int launch_fc_correction_m(dim3 grid, int G, cudaStream_t s, const FCInputs& in, const Table& tb,
                           const PointGrid& pg, const float* omegas, const float* weights, int K,
                           const float* moments, float* sums, float* scale, float* beta, float* cache) {
  cudaError_t e = cudaFuncSetAttribute(fc_correction_kernel<kGP, kMM>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       kWindowBytes);
  if (e != cudaSuccess) return set_error(CITRUS_ECUDA, "first-collision window: %s", cudaGetErrorString(e));
  fc_correction_kernel<kGP, kMM><<<grid, dim3(kEmitPoints, G), kWindowBytes, s>>>(in, tb, pg, omegas, weights, K,
                                                                                 moments, sums, scale, beta, cache);
  note_launches();
  return CITRUS_OK;
}

template <int kGP, int kMM, bool kVec, bool kExact, bool kWindow>
int launch_fc_correction_warps_w(dim3 grid, cudaStream_t s, const FCInputs& in, const Table& tb, const PointGrid& pg,
                                 const float* omegas, const float* weights, int K, const float* moments, float* sums,
                                 float* scale, float* beta, float* cache) {
  constexpr int bytes = kWindow ? fc_window_bytes(kGP) : fc_sums_bytes(kGP);
  auto kernel = fc_correction_warps_kernel<kGP, kMM, kVec, kExact, kWindow>;
  cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
  if (e != cudaSuccess) return set_error(CITRUS_ECUDA, "first-collision window: %s", cudaGetErrorString(e));
  kernel<<<grid, 32 * kFcWarps, bytes, s>>>(in, tb, pg, omegas, weights, K, moments, sums, scale, beta, cache);
  note_launches();
  return CITRUS_OK;
}

template <int kGP, int kMM, bool kVec>
int launch_fc_correction_warps(dim3 grid, cudaStream_t s, const FCInputs& in, const Table& tb, const PointGrid& pg,
                               const float* omegas, const float* weights, int K, const float* moments, float* sums,
                               float* scale, float* beta, float* cache) {
#define CITRUS_FCW(EXACT, WINDOW)                                                                                        \
  launch_fc_correction_warps_w<kGP, kMM, kVec, EXACT, WINDOW>(grid, s, in, tb, pg, omegas, weights, K, moments, sums, \
                                                              scale, beta, cache)
  // two materials and the padded number of groups known to the compiler: us at 32^3 points and 120 directions, known / not: one
  // group 23 / 29, two 43 / 41, 8 groups 246 / 717 (not known, their window of 124 nodes is not taken), 16 groups 1438 / 1497
  constexpr bool kExact = kMM == 2 && (kVec || kGP < 4);
  const bool exact = kExact && tb.G == kGP && tb.M == kMM;
  if constexpr (kGP > 8) {
    return exact ? CITRUS_FCW(kExact, true) : CITRUS_FCW(false, true);
  } else {
    constexpr bool kWindow = kGP >= 4;
    // up to 33 directions on 401 nodes fit no window but that of the last batch, which costs the others the L1: 5 groups, 32
    // directions 50 us with it, 39 without; 48 directions pay
    if (kWindow && tb.G >= 4 && (exact || (window_nodes(tb.M, tb.G, fc_window_bytes(kGP)) >= kFcWindowNodes &&
                                           tb.N <= 3 * kFcNodesPerDirection * (int64_t)K)))
      return exact ? CITRUS_FCW(kExact, kWindow) : CITRUS_FCW(false, kWindow);
    return exact ? CITRUS_FCW(kExact, false) : CITRUS_FCW(false, false);
  }
#undef CITRUS_FCW
}

// CITRUS_FC_KERNEL=groups selects the group-lane correction kernel (fc_correction_kernel); read at every call
inline bool fc_by_groups() {
  const char* v = getenv("CITRUS_FC_KERNEL");
  return v != nullptr && v[0] == 'g';
}

// materials held in registers: two (the common water and bone case) or up to eight; G <= 16 takes the (point,
// direction) kernel
template <int kGP>
int launch_fc_correction(dim3 grid, int G, cudaStream_t s, const FCInputs& in, const Table& tb, const PointGrid& pg,
                         const float* omegas, const float* weights, int K, const float* moments, float* sums,
                         float* scale, float* beta, float* cache) {
  if constexpr (kGP <= 16) {
    if (!fc_by_groups()) {
      const bool vec = kGP >= 4 && G % 4 == 0 && ((uintptr_t)tb.t % 16) == 0;
      constexpr bool kCanVec = kGP >= 4;
      if (tb.M <= 2)
        return vec ? launch_fc_correction_warps<kGP, 2, kCanVec>(grid, s, in, tb, pg, omegas, weights, K, moments,
                                                                 sums, scale, beta, cache)
                   : launch_fc_correction_warps<kGP, 2, false>(grid, s, in, tb, pg, omegas, weights, K, moments,
                                                               sums, scale, beta, cache);
      return vec ? launch_fc_correction_warps<kGP, kMaxM, kCanVec>(grid, s, in, tb, pg, omegas, weights, K, moments,
                                                                   sums, scale, beta, cache)
                 : launch_fc_correction_warps<kGP, kMaxM, false>(grid, s, in, tb, pg, omegas, weights, K, moments,
                                                                 sums, scale, beta, cache);
    }
  }
  if (tb.M <= 2)
    return launch_fc_correction_m<kGP, 2>(grid, G, s, in, tb, pg, omegas, weights, K, moments, sums, scale, beta,
                                          cache);
  return launch_fc_correction_m<kGP, kMaxM>(grid, G, s, in, tb, pg, omegas, weights, K, moments, sums, scale, beta,
                                            cache);
}

template <int kGP>
void launch_fc_moments_cached(int64_t NC, int G, int K, cudaStream_t s, const FCInputs& in, const PointGrid& pg,
                              const float* omegas, const float* cache, const int32_t* cache_index,
                              const float* scale, const float* beta, float slope_scale, float* out,
                              int64_t out_k_stride) {
  dim3 grid((unsigned)cdiv(NC, kEmitPoints), (unsigned)cdiv(K, kFcBatch));
  // above 16 groups the block's 1024 threads leave 64 registers each: the eight points' factors would spill
  auto kernel = pg.f == 1                ? fc_moments_cached_kernel<kGP, 1>
                : pg.f == 2 && kGP <= 16 ? fc_moments_cached_kernel<kGP, kGP <= 16 ? 2 : 0>
                                         : fc_moments_cached_kernel<kGP, 0>;
  kernel<<<grid, dim3(kEmitPoints, G), 0, s>>>(in, pg, omegas, K, cache, cache_index, scale, beta, slope_scale, out,
                                               out_k_stride);
  note_launches();
}

template <int kGP>
void launch_fc_means(int G, int K, cudaStream_t s, const FCInputs& in, const PointGrid& pg, const float* omegas,
                     const float* cache, const int32_t* cache_index, const float* scale, const float* beta, float* out,
                     int64_t out_k_stride) {
  dim3 grid((unsigned)cdiv(in.V, kEmitPoints), (unsigned)cdiv(K, kFcBatch));
  fc_means_kernel<kGP><<<grid, dim3(kEmitPoints, G), 0, s>>>(in, pg, omegas, K, cache, cache_index, scale, beta, out,
                                                             out_k_stride);
  note_launches();
}

}  // namespace
}  // namespace citrus

#define CITRUS_GP_DISPATCH(G, CALL) \
  ((G) <= 1 ? CALL(1) : (G) <= 2 ? CALL(2) : (G) <= 4 ? CALL(4) : (G) <= 8 ? CALL(8) : (G) <= 16 ? CALL(16) : CALL(32))

extern "C" int citrus_first_collision_moments(const float* rho, int64_t num_materials, const float* phi,
                                              int64_t num_groups, const float* axes, const int64_t* point_dims,
                                              int64_t points_per_cell, const double* focal_spot, const float* table,
                                              int64_t num_eta, double eta_lo, double eta_hi, const float* omegas,
                                              int64_t num_directions, const float* scale, const float* beta,
                                              const float* cache, const int32_t* cache_index, float* out,
                                              int64_t out_direction_stride, void* stream) {
  int st = check_table(table, num_materials, num_eta, num_groups);
  if (st) return st;
  CITRUS_REQUIRE(rho && phi && axes && point_dims && focal_spot && omegas && scale && beta && out,
                 "citrus_first_collision_moments: null pointer");
  CITRUS_REQUIRE((cache == nullptr) == (cache_index == nullptr),
                 "citrus_first_collision_moments: cache and cache_index go together");
  const int64_t f = points_per_cell;
  CITRUS_REQUIRE(f >= 1 && point_dims[0] % f == 0 && point_dims[1] % f == 0 && point_dims[2] % f == 0,
                 "citrus_first_collision_moments: the point grid is not cells x %lld", (long long)f);
  CITRUS_REQUIRE(((uintptr_t)out % 16) == 0 && out_direction_stride % 4 == 0,
                 "citrus_first_collision_moments: out must be 16-byte aligned");
  CITRUS_REQUIRE(num_directions <= 65535, "citrus_first_collision_moments: too many directions");
  const int64_t V = point_dims[0] * point_dims[1] * point_dims[2];
  if (V == 0 || num_directions == 0) return CITRUS_OK;
  const FCInputs in = make_inputs(rho, phi, axes, V, focal_spot, point_dims);
  const Table tb = make_table(table, num_materials, num_eta, num_groups, eta_lo, eta_hi);
  const PointGrid pg = make_grid(point_dims, f);
  double mean_u2 = 0;
  for (int j = 0; j < f; ++j) {
    const double u = (2.0 * j + 1.0) / f - 1.0;
    mean_u2 += u * u / f;
  }
  const float slope_scale = f > 1 ? (float)(1.0 / mean_u2) : 0.f;
  const int64_t NC = V / (f * f * f);
  const int G = (int)num_groups, K = (int)num_directions;
  cudaStream_t s = as_stream(stream);
  if (cache != nullptr) {
#define CITRUS_FCM(GP) \
  (launch_fc_moments_cached<GP>(NC, G, K, s, in, pg, omegas, cache, cache_index, scale, beta, slope_scale, out, \
                                out_direction_stride), 0)
    (void)CITRUS_GP_DISPATCH(G, CITRUS_FCM);
#undef CITRUS_FCM
    return launch_status("citrus_first_collision_moments");
  }
  dim3 grid((unsigned)cdiv(NC, kPoints), (unsigned)K), block(kPoints, G);
  CITRUS_G_DISPATCH(G, fc_moments_kernel, grid, block, 0, s, in, tb, pg, omegas, K, scale, beta, slope_scale, out,
                    out_direction_stride)
  return launch_status("citrus_first_collision_moments");
}

extern "C" int citrus_first_collision_means(int64_t num_groups, const float* axes, const int64_t* point_dims,
                                            const double* focal_spot, const float* omegas, int64_t num_directions,
                                            const float* scale, const float* beta, const float* cache,
                                            const int32_t* cache_index, float* out, int64_t out_direction_stride,
                                            void* stream) {
  CITRUS_REQUIRE(axes && point_dims && focal_spot && omegas && scale && beta && cache && cache_index && out,
                 "citrus_first_collision_means: null pointer");
  CITRUS_REQUIRE(num_groups >= 1 && num_groups <= 32 && num_directions <= 65535,
                 "citrus_first_collision_means: bad sizes");
  const int64_t V = point_dims[0] * point_dims[1] * point_dims[2];
  CITRUS_REQUIRE(out_direction_stride >= V * num_groups, "citrus_first_collision_means: direction stride too small");
  if (V == 0 || num_directions == 0) return CITRUS_OK;
  const FCInputs in = make_inputs(nullptr, nullptr, axes, V, focal_spot, point_dims);  // points only
  const PointGrid pg = make_grid(point_dims, 1);
  const int G = (int)num_groups, K = (int)num_directions;
  cudaStream_t s = as_stream(stream);
#define CITRUS_FCM(GP) \
  (launch_fc_means<GP>(G, K, s, in, pg, omegas, cache, cache_index, scale, beta, out, out_direction_stride), 0)
  (void)CITRUS_GP_DISPATCH(G, CITRUS_FCM);
#undef CITRUS_FCM
  return launch_status("citrus_first_collision_means");
}

extern "C" int citrus_first_collision_correction(const float* rho, int64_t num_materials, const float* phi,
                                                 int64_t num_groups, const float* axes, const int64_t* point_dims,
                                                 const double* focal_spot, const float* table, int64_t num_eta,
                                                 double eta_lo, double eta_hi, const float* omegas,
                                                 const float* weights, int64_t num_directions, const float* moments,
                                                 float* sums, float* scale, float* beta, float* cache, void* stream) {
  int st = check_table(table, num_materials, num_eta, num_groups);
  if (st) return st;
  CITRUS_REQUIRE(rho && phi && axes && point_dims && focal_spot && omegas && weights && moments && scale && beta,
                 "citrus_first_collision_correction: null pointer");
  if (num_groups % 4 == 0)
    CITRUS_REQUIRE(((uintptr_t)table % 16) == 0, "citrus_first_collision_correction: table must be 16-byte aligned");
  const int64_t V = point_dims[0] * point_dims[1] * point_dims[2];
  if (V == 0) return CITRUS_OK;
  const FCInputs in = make_inputs(rho, phi, axes, V, focal_spot, point_dims);
  const Table tb = make_table(table, num_materials, num_eta, num_groups, eta_lo, eta_hi);
  const PointGrid pg = make_grid(point_dims, 1);
  const int G = (int)num_groups, K = (int)num_directions;
  dim3 grid((unsigned)cdiv(V, kEmitPoints));
  cudaStream_t s = as_stream(stream);
#define CITRUS_FCC(GP) launch_fc_correction<GP>(grid, G, s, in, tb, pg, omegas, weights, K, moments, sums, scale, beta, cache)
  st = CITRUS_GP_DISPATCH(G, CITRUS_FCC);
#undef CITRUS_FCC
  if (st) return st;
  return launch_status("citrus_first_collision_correction");
}

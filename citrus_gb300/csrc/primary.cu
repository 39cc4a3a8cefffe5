// The primary image of one view from its path lengths (citrus/scatter_solver/scatter_image.py:1395-1471): the
// fine-energy transmission of every pixel's n x n rays, their mean, and the pixel's factors, in one pass.
#include <math.h>

#include "common.cuh"
#include "panel_interpolate.cuh"

namespace citrus {
namespace {

constexpr int kThreads = 128;
constexpr int kMaxM = 8;
constexpr int kMaxG = 32;

struct PrimaryArgs {
  const float* path;      // [Mp, rows n, cols n] line integrals in g/cm^2
  const float* mu;        // [Mp, E]
  const float* weight;    // [E]
  const int* group;       // [E] ascending
  const float* filter_mu; // [E], or null without a beam filter
  const double* columns;  // [cols, 9]: position at v = 0 from the focal spot, direction of v, local normal
  const double* u;        // [cols] panel coordinate of the pixel columns
  const double* v;        // [rows] panel coordinate of the pixel rows
  const double* theta;    // [T] ascending incidence nodes of the detector table
  const double* response; // [G, T] detector response times grid transmission at the group energies
  float *fluence, *planar, *per_group, *signal;
  int Mp, rows, cols, n, E, G, T;
};

// A thread takes a pixel: kB of its rays at a time, so that an energy's coefficients, read from shared memory, serve
// kB exponentials; the energies are in group order, so a group's sum is one register and is finished when the group
// changes. The factors (inverse square, profile, cosine of incidence, detector response) are float64 and stay in
// registers; only what the caller asked for touches memory. Bound by the exponentials: a 384 x 512 panel with 2 x 2
// rays and 256 energies (201 million) takes 0.19 ms. The geometry and the responses used to be numpy arrays of
// the whole panel, formed and copied on every call: 99 ms of a call's 100 ms
// (the separate transmission took 0.53 ms of it); the call now takes 0.71 ms, the ray trace 0.42 ms of it.
template <int kB>
__global__ void __launch_bounds__(kThreads) primary_kernel(PrimaryArgs a, SourceExtras ex) {
  extern __shared__ float smem[];
  float* s_mu = smem;                                   // [Mp, E]
  float* s_w = s_mu + a.Mp * a.E;                       // [E]
  float* s_f = s_w + a.E;                               // [E]
  int* s_g = reinterpret_cast<int*>(s_f + a.E);         // [E]
  float* s_acc = reinterpret_cast<float*>(s_g + a.E);   // [G, kThreads], with more than kB rays per pixel
  for (int i = threadIdx.x; i < a.Mp * a.E; i += kThreads) s_mu[i] = a.mu[i];
  for (int i = threadIdx.x; i < a.E; i += kThreads) {
    s_w[i] = a.weight[i];
    s_f[i] = a.filter_mu ? a.filter_mu[i] : 0.f;
    s_g[i] = a.group[i];
  }
  __syncthreads();
  const int64_t P = (int64_t)a.rows * a.cols;
  const int64_t p = (int64_t)blockIdx.x * kThreads + threadIdx.x;
  if (p >= P) return;
  const int r = (int)(p / a.cols), c = (int)(p - (int64_t)r * a.cols);
  const double* col = a.columns + 9 * c;
  const double v = a.v[r];
  double d[3], dist2 = 0.0, dot = 0.0;
  for (int k = 0; k < 3; ++k) {
    d[k] = col[k] + v * col[3 + k];
    dist2 += d[k] * d[k];
    dot -= d[k] * col[6 + k];
  }
  const double cosine = fmin(fmax(dot / sqrt(dist2), -1.0), 1.0);
  const double weight = (ex.profile ? panel_interpolate(ex.profile, ex.rows, ex, a.u[c], v) : 1.0) / dist2;
  int t0 = 0, t1 = 0;
  double tw = 0.0;
  if (a.T > 1) {  // the detector's incidence nodes around theta, clamped to the end nodes
    const double theta = fmin(fmax(acos(cosine), a.theta[0]), a.theta[a.T - 1]);
    while (t1 < a.T && a.theta[t1] <= theta) ++t1;
    t1 = min(max(t1, 1), a.T - 1);
    t0 = t1 - 1;
    tw = fmin(fmax((theta - a.theta[t0]) / (a.theta[t1] - a.theta[t0]), 0.0), 1.0);
  }
  const float f_fluence = (float)weight, f_planar = (float)(weight * cosine);
  float signal = 0.f;
  auto write = [&](int g, float transmission) {
    const double* table = a.response + (int64_t)g * a.T;
    const double response = table[t0] + (table[t1] - table[t0]) * tw;
    const float s = transmission * (float)(weight * cosine * response);
    const int64_t at = g * P + p;
    a.fluence[at] = transmission * f_fluence;
    a.planar[at] = transmission * f_planar;
    a.per_group[at] = s;
    signal += s;
  };
  const int rays = a.n * a.n;
  const int64_t ray_cols = (int64_t)a.cols * a.n, plane = ray_cols * a.rows * a.n;
  for (int b0 = 0; b0 < rays; b0 += kB) {
    float pm[kB][kMaxM], pf[kB];
#pragma unroll
    for (int b = 0; b < kB; ++b) {
      const int ray = min(b0 + b, rays - 1), i = ray / a.n, j = ray - i * a.n;
      const int64_t at = ((int64_t)r * a.n + i) * ray_cols + (int64_t)c * a.n + j;
#pragma unroll
      for (int m = 0; m < kMaxM; ++m) pm[b][m] = m < a.Mp ? __ldg(a.path + m * plane + at) : 0.f;
      pf[b] = 0.f;
      if (a.filter_mu) {
        const double du = ((2 * j + 1) / (2.0 * a.n) - 0.5) * ex.d_ch, dv = ((2 * i + 1) / (2.0 * a.n) - 0.5) * ex.d_row;
        pf[b] = (float)(panel_interpolate(ex.thickness, ex.t_rows, ex, a.u[c] + du, v + dv) * ex.filter_density);
      }
    }
    const int live = min(kB, rays - b0);
    int e = 0;
    for (int g = 0; g < a.G; ++g) {
      float sum[kB];
#pragma unroll
      for (int b = 0; b < kB; ++b) sum[b] = 0.f;
      for (; e < a.E && s_g[e] == g; ++e) {
        float tau[kB];
#pragma unroll
        for (int b = 0; b < kB; ++b) tau[b] = s_mu[e] * pm[b][0];
#pragma unroll
        for (int m = 1; m < kMaxM; ++m) {
          if (m < a.Mp) {
            const float mu = s_mu[m * a.E + e];
#pragma unroll
            for (int b = 0; b < kB; ++b) tau[b] = fmaf(mu, pm[b][m], tau[b]);
          }
        }
        if (a.filter_mu) {  // the filter after the materials
#pragma unroll
          for (int b = 0; b < kB; ++b) tau[b] = fmaf(s_f[e], pf[b], tau[b]);
        }
#pragma unroll
        for (int b = 0; b < kB; ++b) sum[b] += s_w[e] * expf(-tau[b]);
      }
      float total = 0.f;
#pragma unroll
      for (int b = 0; b < kB; ++b)
        if (b < live) total += sum[b];
      if (rays > kB) {
        float* slot = s_acc + g * kThreads + threadIdx.x;
        *slot = b0 == 0 ? total : *slot + total;
      } else {
        write(g, rays == 1 ? total : total / (float)rays);
      }
    }
  }
  if (rays > kB)
    for (int g = 0; g < a.G; ++g) write(g, s_acc[g * kThreads + threadIdx.x] / (float)rays);
  a.signal[p] = signal;
}

}  // namespace
}  // namespace citrus

using namespace citrus;

extern "C" int citrus_primary_image(const float* path, int64_t num_materials, int64_t num_rows, int64_t num_cols,
                                    int64_t samples, const float* fine_mu, const float* fine_weight,
                                    const int32_t* fine_group, int64_t num_fine, int64_t num_groups,
                                    const double* columns, const double* u, const double* v, const double* theta_nodes,
                                    const double* response, int64_t num_theta, const double* panel,
                                    const double* profile, const double* thickness, int64_t thickness_rows,
                                    double filter_density, const float* filter_mu, float* fluence, float* planar,
                                    float* per_group, float* signal, void* stream) {
  CITRUS_REQUIRE(path && fine_mu && fine_weight && fine_group && columns && u && v && theta_nodes && response &&
                     panel && fluence && planar && per_group && signal, "citrus_primary_image: null pointer");
  CITRUS_REQUIRE(num_materials >= 1 && num_materials <= kMaxM && num_groups >= 1 && num_groups <= kMaxG &&
                     num_fine >= 1 && num_rows >= 0 && num_cols >= 0 && samples >= 1 && num_theta >= 1,
                 "citrus_primary_image: bad sizes (materials %lld, groups %lld, fine %lld, samples %lld)",
                 (long long)num_materials, (long long)num_groups, (long long)num_fine, (long long)samples);
  CITRUS_REQUIRE(num_rows * samples < (1 << 24) && num_cols * samples < (1 << 24) && samples < (1 << 12) &&
                     num_rows * num_cols < (1ll << 31),
                 "citrus_primary_image: panel too large");
  CITRUS_REQUIRE((thickness == nullptr) == (filter_mu == nullptr),
                 "citrus_primary_image: the filter's thickness and attenuation go together");
  CITRUS_REQUIRE(!thickness || thickness_rows == 1 || thickness_rows == num_rows,
                 "citrus_primary_image: the filter thickness must have 1 or all rows");
  const size_t tables = (size_t)(num_materials + 3) * num_fine * sizeof(float);
  CITRUS_REQUIRE(tables <= 96 * 1024, "citrus_primary_image: %lld fine energies too many", (long long)num_fine);
  if (num_rows == 0 || num_cols == 0) return CITRUS_OK;
  SourceExtras ex{};
  ex.profile = profile;
  ex.thickness = thickness;
  ex.t_rows = (int)thickness_rows;
  ex.filter_density = filter_density;
  ex.rows = (int)num_rows;
  ex.channels = (int)num_cols;
  ex.d_row = panel[0];
  ex.d_ch = panel[1];
  ex.off_row = panel[2];
  ex.off_ch = panel[3];
  CITRUS_REQUIRE(ex.d_row > 0 && ex.d_ch > 0, "citrus_primary_image: bad panel");
  const PrimaryArgs a{path, fine_mu, fine_weight, fine_group, filter_mu, columns, u, v, theta_nodes, response,
                      fluence, planar, per_group, signal, (int)num_materials, (int)num_rows, (int)num_cols,
                      (int)samples, (int)num_fine, (int)num_groups, (int)num_theta};
  const int64_t blocks = cdiv(num_rows * num_cols, kThreads);
  const bool one = samples == 1;
  const size_t smem = tables + (samples > 2 ? (size_t)num_groups * kThreads * sizeof(float) : 0);
  if (smem > 48 * 1024) {
    cudaError_t e = one ? cudaFuncSetAttribute(primary_kernel<1>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem)
                        : cudaFuncSetAttribute(primary_kernel<4>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return set_error(CITRUS_ECUDA, "citrus_primary_image: %s", cudaGetErrorString(e));
  }
  if (one) primary_kernel<1><<<(unsigned)blocks, kThreads, smem, as_stream(stream)>>>(a, ex);
  else primary_kernel<4><<<(unsigned)blocks, kThreads, smem, as_stream(stream)>>>(a, ex);
  note_launches();
  return launch_status("citrus_primary_image");
}

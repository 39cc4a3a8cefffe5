// What the first-collision kernels (collision.cu) and the emission of the image (emission*.cu) share: the points, the transfer
// table, its window in shared memory, and the sums over incoming groups.
#pragma once

#include <math.h>
#include <type_traits>

#include "common.cuh"

namespace citrus {

constexpr int kMaxG = 32;
constexpr int kMaxM = 8;
constexpr int kEmitPoints = 32;

struct PointGrid {
  int R, C, S;            // points of the quadrature grid
  int f;                  // points per cell axis (q)
  int Rc, Cc, Sc;         // transport cells
};

__device__ __forceinline__ void point_rcs(int64_t v, const PointGrid& g, int& i, int& j, int& k) {
  const int64_t cs = (int64_t)g.C * g.S;
  i = (int)(v / cs);
  const int64_t rem = v - (int64_t)i * cs;
  j = (int)(rem / g.S);
  k = (int)(rem - (int64_t)j * g.S);
}

// unit primary direction from the focal spot to point (x, y, z), IEEE sqrt and division
__device__ __forceinline__ void primary_direction(float x, float y, float z, float r0x, float r0y, float r0z,
                                                  float& ux, float& uy, float& uz) {
  const float dx = x - r0x, dy = y - r0y, dz = z - r0z;
  const float n = __fsqrt_rn(dx * dx + dy * dy + dz * dz);
  ux = __fdiv_rn(dx, n);
  uy = __fdiv_rn(dy, n);
  uz = __fdiv_rn(dz, n);
}

struct Table {
  const float* t;    // [M, N, G, G] transfer by (node, g_out, g_in)
  int M, N, G;
  float eta_lo, eta_hi;
  float inv_span;    // 1 / (eta_hi - eta_lo) when the span is a power of two (the product is then the quotient), else 0
};

inline Table make_table(const float* t, int64_t M, int64_t N, int64_t G, double eta_lo, double eta_hi) {
  Table tb{t, (int)M, (int)N, (int)G, (float)eta_lo, (float)eta_hi, 0.f};
  const float span = tb.eta_hi - tb.eta_lo;
  int e = 0;
  if (span > 0.f && frexpf(span, &e) == 0.5f) tb.inv_span = ldexpf(1.f, 1 - e);
  return tb;
}

// table position of a cosine (cross_sections.py:905-938, uniform table)
__device__ __forceinline__ void table_position(const Table& tb, float cosine, int& i0, float& w) {
  const float eta = fminf(fmaxf(cosine, tb.eta_lo), tb.eta_hi);
  const float q = tb.inv_span != 0.f ? (eta - tb.eta_lo) * tb.inv_span : __fdiv_rn(eta - tb.eta_lo, tb.eta_hi - tb.eta_lo);
  const float pos = q * (float)(tb.N - 1);
  float f0 = floorf(pos);
  f0 = fminf(fmaxf(f0, 0.f), (float)(tb.N - 2));
  i0 = (int)f0;
  w = fminf(fmaxf(pos - f0, 0.f), 1.f);
}

// ---- shared point inputs of the first-collision kernels ---------------------------------------------------------
struct FCInputs {
  const float* rho;   // [M, V]
  const float* phi;   // [G, V]
  const float* ax_x;  // [C] point coordinates (float32, as the reference's float32 path)
  const float* ax_y;  // [R]
  const float* ax_z;  // [S]
  float r0x, r0y, r0z;
  int64_t V;
};

// row . phi over the incoming groups (upscatter entries of the table are zero); the row in global memory (read-only
// path) or in shared memory
template <int kGP, bool kShared>
__device__ __forceinline__ float row_dot(const float* __restrict__ row, const float* phi, int G) {
  float a = 0.f;
  if (kGP % 4 == 0 && G == kGP) {
#pragma unroll
    for (int q = 0; q < kGP / 4; ++q) {
      const float4 t = kShared ? reinterpret_cast<const float4*>(row)[q] : __ldg(reinterpret_cast<const float4*>(row) + q);
      a = fmaf(t.x, phi[4 * q], a);
      a = fmaf(t.y, phi[4 * q + 1], a);
      a = fmaf(t.z, phi[4 * q + 2], a);
      a = fmaf(t.w, phi[4 * q + 3], a);
    }
  } else {
#pragma unroll
    for (int gi = 0; gi < kGP; ++gi)
      if (gi < G) a = fmaf(kShared ? row[gi] : __ldg(row + gi), phi[gi], a);
  }
  return a;
}

// The window of table nodes a block needs: its points' cosines with its directions span a few dozen of the eta nodes,
// so the rows of those nodes ([node][m][g][g']) are staged in shared memory once and every interpolation of the block
// reads them there. The lanes' nodes are neighbours: a node's stride is an odd number of 16-byte reads (of floats where rows
// are read as floats), so that neighbouring nodes are read without bank conflicts (16 bytes per (node, m) let four of them).
constexpr int kWindowBytes = 32 * 1024;

__host__ __device__ inline int window_node_stride(int M, int G) {
  return G % 4 == 0 ? (M * G * G / 4 | 1) * 4 : M * G * G | 1;
}
__host__ __device__ inline int window_nodes(int M, int G, int bytes = kWindowBytes) {
  const int n = bytes / (4 * window_node_stride(M, G));
  return n < 192 ? n : 192;
}


// The rows of the nodes [lo, lo + n) into a window, asynchronously and waited for by the thread that copied them. kG: the
// groups when they are known at compile time (else 0): the copy is then shifts and 16-byte copies, all in flight together.
template <int kG>
__device__ __forceinline__ void copy_window(const Table& tb, int lo, int n, int warp, int nwarps, int tid, int nthreads,
                                            float* s_tab) {
  const int G = tb.G, GG = G * G, NS = window_node_stride(tb.M, G), lane = tid & 31;
  const bool quads = G % 4 == 0 && ((uintptr_t)tb.t % 16) == 0;
  if (kG > 0 && kG % 4 == 0 && quads) {
    constexpr int GG4 = kG >= 4 ? kG * kG / 4 : 1;
    for (int m = 0; m < tb.M; ++m) {
      const float4* src = reinterpret_cast<const float4*>(tb.t + ((int64_t)m * tb.N + lo) * (kG * kG));
      const uint32_t dst = (uint32_t)__cvta_generic_to_shared(s_tab + m * kG * kG);
      for (int i = tid; i < n * GG4; i += nthreads)
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst + (i / GG4) * NS * 4 + (i % GG4) * 16),
                     "l"(src + i));
    }
  } else if (quads && GG <= 128) {  // a lane per quad of a node, as many nodes a warp as it holds
    const int per = 32 / (GG / 4), sub = lane / (GG / 4), r = lane - sub * (GG / 4);
    for (int m = 0; m < tb.M; ++m)
      for (int node = sub < per ? warp * per + sub : n; node < n; node += nwarps * per)
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(
                         (uint32_t)__cvta_generic_to_shared(s_tab + node * NS + m * GG + 4 * r)),
                     "l"(tb.t + ((int64_t)m * tb.N + lo + node) * GG + 4 * r));
  } else {  // a warp per node: no division per element here either
    for (int m = 0; m < tb.M; ++m)
      for (int node = warp; node < n; node += nwarps) {
        const float* src = tb.t + ((int64_t)m * tb.N + lo + node) * GG;
        const uint32_t dst = (uint32_t)__cvta_generic_to_shared(s_tab + node * NS + m * GG);
        if (quads) {
          for (int r = lane; r < GG / 4; r += 32)
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst + 16 * r), "l"(src + 4 * r));
        } else {
          for (int r = lane; r < GG; r += 32)
            asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(dst + 4 * r), "l"(src + r));
        }
      }
  }
  asm volatile("cp.async.wait_all;" ::: "memory");
}

// The eta nodes [lo, lo + n) that the valid points of a block read for the directions s_om[0..n): s_window = {lo, n}. Each
// thread evaluates the directions first_dir, first_dir + dir_step, ... for its point; s_range holds one (lo, hi) per warp. Ends
// with a block barrier; every thread of the block must call it.
__device__ __forceinline__ void window_range(const Table& tb, bool valid, float ux, float uy, float uz,
                                             const float (*s_om)[3], int n, int first_dir, int dir_step, int warp,
                                             int nwarps, int tid, int (*s_range)[32], int* s_window) {
  int lo = 1 << 30, hi = -1;
  if (valid) {
    for (int dd = first_dir; dd < n; dd += dir_step) {
      int i0;
      float w;
      table_position(tb, ux * s_om[dd][0] + uy * s_om[dd][1] + uz * s_om[dd][2], i0, w);
      lo = min(lo, i0);
      hi = max(hi, i0);
    }
  }
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) {
    lo = min(lo, __shfl_xor_sync(0xffffffffu, lo, off));
    hi = max(hi, __shfl_xor_sync(0xffffffffu, hi, off));
  }
  if ((tid & 31) == 0) {
    s_range[0][warp] = lo;
    s_range[1][warp] = hi;
  }
  __syncthreads();
  if (tid == 0) {
    for (int q = 1; q < nwarps; ++q) {
      lo = min(lo, s_range[0][q]);
      hi = max(hi, s_range[1][q]);
    }
    s_window[0] = lo;
    s_window[1] = hi + 2 - lo;
  }
  __syncthreads();
}

// Stages the table window of a block for the directions s_om[0..n) if its nodes fit, else s_window[0] = -1 (rows read from
// global memory); arguments and barrier as window_range.
__device__ __forceinline__ void stage_window(const Table& tb, bool valid, float ux, float uy, float uz,
                                             const float (*s_om)[3], int n, int first_dir, int dir_step, int warp,
                                             int nwarps, int tid, int nthreads, int (*s_range)[32], int* s_window,
                                             float* s_tab, int window_bytes = kWindowBytes) {
  window_range(tb, valid, ux, uy, uz, s_om, n, first_dir, dir_step, warp, nwarps, tid, s_range, s_window);
  const int lo = s_window[0], count = s_window[1];
  const bool fits = count >= 2 && count <= window_nodes(tb.M, tb.G, window_bytes);
  if (fits) copy_window<0>(tb, lo, count, warp, nwarps, tid, nthreads, s_tab);
  __syncthreads();  // s_window is read, the copies are complete
  if (!fits) {
    if (tid == 0) s_window[0] = -1;
    __syncthreads();
  }
}

// the source between two nodes whose sums over the materials are f0 and f1
__device__ __forceinline__ float interpolate_nodes(float f0, float f1, float w) {
  return fmaf(__fsub_rn(f1, f0), w, f0);
}

// S_FC of group g at one point for one direction, rows from the window (win_lo >= 0) or from global memory
// kWindow: 1 the rows are in the block's shared-memory window, 2 in global memory, 0 decided by win_lo >= 0. kNodes: the
// materials are summed at each node before the interpolation (as emission_warps_kernel's ring holds them), else after
template <int kGP, int kMM, int kWindow = 0, bool kNodes = false>
__device__ __forceinline__ float fc_group(const Table& tb, const float* s_tab, int win_lo, int i0, float w, int g,
                                          const float* rho, const float* phi) {
  const int G = tb.G, NS = window_node_stride(tb.M, G);
  float f0 = 0.f, f1 = 0.f;
#pragma unroll
  for (int m = 0; m < kMM; ++m) {
    const float r = rho[m];
    if (m >= tb.M || r == 0.f) continue;
    float a0, a1;
    if (kWindow == 1 || (kWindow == 0 && win_lo >= 0)) {
      const float* row0 = s_tab + (i0 - win_lo) * NS + (m * G + g) * G;
      a0 = row_dot<kGP, true>(row0, phi, G);
      a1 = row_dot<kGP, true>(row0 + NS, phi, G);
    } else {
      const float* row0 = tb.t + (((int64_t)m * tb.N + i0) * G + g) * G;
      a0 = row_dot<kGP, false>(row0, phi, G);
      a1 = row_dot<kGP, false>(row0 + (int64_t)G * G, phi, G);
    }
    if (kNodes) {
      f0 = fmaf(r, a0, f0);
      f1 = fmaf(r, a1, f1);
    } else {
      f0 = fmaf(r, a0 + (a1 - a0) * w, f0);
    }
  }
  return kNodes ? interpolate_nodes(f0, f1, w) : f0;
}

// sum_{gi <= g} row[gi] phi[gi], in incoming-group order; the row in shared or global memory, float4 reads when the
// rows are 16-byte aligned (kVec)
template <int kGP, bool kVec, bool kShared>
__device__ __forceinline__ float dot_lower(const float* __restrict__ row, const float* phi, int g) {
  float a = 0.f;
  if constexpr (kVec) {
#pragma unroll
    for (int q = 0; q < kGP / 4; ++q) {
      if (4 * q > g) break;
      const float4 t = kShared ? reinterpret_cast<const float4*>(row)[q]
                               : __ldg(reinterpret_cast<const float4*>(row) + q);
      a = fmaf(t.x, phi[4 * q], a);
      if (4 * q + 1 <= g) a = fmaf(t.y, phi[4 * q + 1], a);
      if (4 * q + 2 <= g) a = fmaf(t.z, phi[4 * q + 2], a);
      if (4 * q + 3 <= g) a = fmaf(t.w, phi[4 * q + 3], a);
    }
  } else {
#pragma unroll
    for (int gi = 0; gi < kGP; ++gi) {
      if (gi > g) break;
      a = fmaf(kShared ? row[gi] : __ldg(row + gi), phi[gi], a);
    }
  }
  return a;
}

inline int check_table(const float* table, int64_t M, int64_t N, int64_t G) {
  CITRUS_REQUIRE(table != nullptr, "first collision: null transfer table");
  CITRUS_REQUIRE(M >= 1 && M <= kMaxM, "first collision: %lld materials outside [1, %d]", (long long)M, kMaxM);
  CITRUS_REQUIRE(N >= 2 && G >= 1 && G <= kMaxG, "first collision: bad table (N %lld, G %lld)", (long long)N,
                 (long long)G);
  return CITRUS_OK;
}

inline FCInputs make_inputs(const float* rho, const float* phi, const float* ax, int64_t V, const double* r0,
                     const int64_t* pdims) {
  FCInputs in;
  in.rho = rho;
  in.phi = phi;
  in.ax_x = ax;                    // x [C] then y [R] then z [S]
  in.ax_y = ax + pdims[1];
  in.ax_z = ax + pdims[1] + pdims[0];
  in.r0x = (float)r0[0];
  in.r0y = (float)r0[1];
  in.r0z = (float)r0[2];
  in.V = V;
  return in;
}

inline PointGrid make_grid(const int64_t* pdims, int64_t f) {
  PointGrid pg;
  pg.R = (int)pdims[0];
  pg.C = (int)pdims[1];
  pg.S = (int)pdims[2];
  pg.f = (int)f;
  pg.Rc = pg.R / pg.f;
  pg.Cc = pg.C / pg.f;
  pg.Sc = pg.S / pg.f;
  return pg;
}

}  // namespace citrus

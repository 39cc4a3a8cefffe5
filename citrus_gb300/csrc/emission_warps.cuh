// The attenuated emission of the image with a thread per (point, direction): its kernel and launchers.
#pragma once

#include "collision.cuh"

namespace citrus {

// The arguments of one call of the kernel below
struct EmissionCall {
  FCInputs in;
  Table tb;
  PointGrid pg;
  int K, TM;
  const float *omegas, *tau, *tau_mu, *mu, *multiple, *heights, *signal_weight;
  const double* deltas;
  float *out, *partial;
  cudaStream_t stream;
};

// Per padded number of groups, in units of their own: emission_warps_4.cu (up to 4), _8.cu and _16.cu
int emission_warps_4(const EmissionCall& c);
int emission_warps_8(const EmissionCall& c);
int emission_warps_16(const EmissionCall& c);

namespace {

// x[0] + ... + x[n-1] in the order of an xor butterfly over n lanes read at lane 0: pairwise halves, each addition
// rounded on its own (a butterfly's shuffles keep a product from fusing into the next addition; here __fadd_rn does)
template <int n>
__device__ __forceinline__ float tree_sum(const float* x) {
  if constexpr (n == 1) {
    return x[0];
  } else {
    return __fadd_rn(tree_sum<n / 2>(x), tree_sum<n / 2>(x + n / 2));
  }
}

// ---- attenuated emission, one thread per (point, direction) with all of its groups ---------------------------------
// A block is 32 points (the lanes, consecutive points and, for one point per cell, consecutive cells) by kEmitWarps
// warps; a warp takes one direction at a time. The multiple-collision source (and per-group optical depths) of a cell
// are G contiguous floats, read as float4 and coalesced over the warp.
// A point's first-collision source depends on the direction through the scattering cosine alone, and the panel's directions
// see few of the table's nodes: the block forms F[node][group], the sum over materials and incoming groups, once per
// node and point (node_sums), and a direction only interpolates between two nodes. The directions run in the order of their
// cosine with the block's middle direction, and F is a ring of nodes in shared memory that moves with them, so
// that every node is formed once per block. A row of the table read for a whole warp costs four shared-memory or L1
// wavefronts per float4; with both rows read per direction that was 192 wavefronts for 8 groups and two materials, the
// kernel's bound, against 16 for the interpolation and 96 per node formed. 64^3 points, 8 groups,
// 512 directions: 3.46 -> 1.80 ms (2.56 with the numbers of groups and materials checked at run time, hence kExact); 32^3,
// one group: 213 -> 152 us.
// Only the transfer entries of incoming groups at or above the outgoing one enter the sum (the reference's
// first-collision table is downscatter only, uncollided_kernels.py:488-550). Every group value, the group sums and the
// per-block partial sums are formed in emission_kernel's order (its sequential incoming-group sums, its butterflies
// over groups and points), so the two kernels give the same bits on a table without upscatter entries.
constexpr int kEmitWarps = 8;
constexpr int kEmitDirs = 256;  // directions of a block
constexpr int kEmitBins = 512;  // bins of the sort by cosine

// nodes of the ring: a power of two, 64 KB of float[kGP][32] per node for up to 8 groups (3 blocks per SM), 128 KB for 16
__host__ __device__ constexpr int ring_nodes(int gp) { return gp > 8 ? 64 : 512 / gp; }

// floats of the ring and the warps' rows of the node that they form, and the blocks that an SM holds with them
__host__ __device__ constexpr int emission_rows(int gp, int mm) { return (mm * gp * gp + 31) / 32 * 32; }
__host__ __device__ constexpr int emission_floats(int gp, int mm) {
  return ring_nodes(gp) * gp * 32 + kEmitWarps * emission_rows(gp, mm);
}
__host__ __device__ constexpr int emission_blocks(int gp, int mm) { return gp > 8 ? 1 : emission_floats(gp, mm) > 18432 ? 2 : 3; }

template <int kGP, bool kVec>
__device__ __forceinline__ void load_groups(const float* __restrict__ p, int G, float* x) {
  if constexpr (kVec) {
#pragma unroll
    for (int q = 0; q < kGP / 4; ++q) {
      if (4 * q < G) {
        const float4 t = __ldg(reinterpret_cast<const float4*>(p) + q);
        x[4 * q] = t.x;
        x[4 * q + 1] = t.y;
        x[4 * q + 2] = t.z;
        x[4 * q + 3] = t.w;
      } else {
        x[4 * q] = x[4 * q + 1] = x[4 * q + 2] = x[4 * q + 3] = 0.f;
      }
    }
  } else {
#pragma unroll
    for (int q = 0; q < kGP; ++q) x[q] = q < G ? __ldg(p + q) : 0.f;
  }
}

// F of one node at this lane's point: sum_m rho_m sum_{g' <= g} T_m[node][g][g'] phi_g', materials without density left
// out, into f; the rows [material][G][G] in shared memory
template <int kGP, int kMM, bool kVec, int kExact>
__device__ __forceinline__ void node_sums(const Table& tb, const float* rows, const float* rho, const float* phi, float* f) {
  const int G = kExact > 0 ? kExact : tb.G;
#pragma unroll
  for (int g = 0; g < kGP; ++g) f[g] = 0.f;
#pragma unroll
  for (int m = 0; m < kMM; ++m) {
    if (!kExact && m >= tb.M) break;
    const float* row = rows + m * G * G;
#pragma unroll
    for (int g = 0; g < kGP; ++g) {
      if (g >= G) break;
      const float a = dot_lower<kGP, kVec, true>(row + g * G, phi, g);
      if (rho[m] != 0.f) f[g] = fmaf(rho[m], a, f[g]);
    }
  }
}

// The same sums of the groups q .. q + kN - 1 at two nodes, the rows of a material material_stride floats after the last
// one's, in shared memory or in the table
template <int kGP, int kMM, bool kVec, int kExact, bool kShared, int kN>
__device__ __forceinline__ void node_pair_sums(const Table& tb, const float* row0, const float* row1,
                                               int64_t material_stride, int q, const float* rho, const float* phi,
                                               float* f0, float* f1) {
  const int G = kExact > 0 ? kExact : tb.G;
#pragma unroll
  for (int i = 0; i < kN; ++i) f0[i] = f1[i] = 0.f;
#pragma unroll
  for (int m = 0; m < kMM; ++m) {
    if (!kExact && m >= tb.M) break;
    const float r = rho[m];
    if (r == 0.f) continue;
#pragma unroll
    for (int i = 0; i < kN; ++i) {
      if (q + i >= G) break;
      const int64_t at = m * material_stride + (q + i) * G;
      f0[i] = fmaf(r, dot_lower<kGP, kVec, kShared>(row0 + at, phi, q + i), f0[i]);
      f1[i] = fmaf(r, dot_lower<kGP, kVec, kShared>(row1 + at, phi, q + i), f1[i]);
    }
  }
}

// kN values of a ring slot at this lane from group g on: float4s of consecutive groups [group / 4][lane], or floats
// [group][lane] for 1 or 2 groups
template <int kN>
__device__ __forceinline__ void load_ring(const float* __restrict__ slot, int g, int lane, float* f) {
  if constexpr (kN == 4) {
    const float4 t = *reinterpret_cast<const float4*>(slot + (g * 32 + 4 * lane));
    f[0] = t.x;
    f[1] = t.y;
    f[2] = t.z;
    f[3] = t.w;
  } else {
#pragma unroll
    for (int q = 0; q < kN; ++q) f[q] = slot[(g + q) * 32 + lane];
  }
}

// kQ1: one point per cell (the point is the cell's centre: no in-cell offsets, no cell attenuation needed). A warp's
// loads of its next direction's multiple-collision source and path lengths are issued before the interpolation of the
// current one, so their latency hides behind that arithmetic; 3 blocks of 256 threads per SM (80 registers).
// kExact: the number of groups (0: at run time), with kMM materials and traced lengths of kMM materials: the group and
// material tests of every direction drop out (a third of the instructions), and so do the groups past
// G of a kGP: an image of 44 x 54 x 38 points and 5 groups 0.94 -> 0.57 ms.
template <int kGP, int kMM, bool kVec, bool kQ1, int kExact>
__global__ void __launch_bounds__(32 * kEmitWarps, emission_blocks(kGP, kMM)) emission_warps_kernel(
    FCInputs in, Table tb, PointGrid pg, const float* __restrict__ omegas, int K,
    const float* __restrict__ tau /*[K, NC, G], or [K, NC, TM] path lengths with tau_mu*/,
    const float* __restrict__ tau_mu /*[TM, G] or null*/, int traced_materials, const float* __restrict__ mu /*[G, NC]*/,
    const float* __restrict__ multiple /*[K, NC, G]*/, const float* __restrict__ heights,
    const float* __restrict__ signal_weight /*[K, G] or null*/, float dx, float dy, float dz,
    float* __restrict__ out, float* __restrict__ partial /*[K, nblocks, 2]*/) {
  constexpr int nthreads = 32 * kEmitWarps;
  constexpr int kRing = ring_nodes(kGP);
  extern __shared__ float4 s_dyn4[];
  float* s_ring = reinterpret_cast<float*>(s_dyn4);   // [kRing][kGP][32]
  __shared__ float s_om[kEmitDirs][3];
  __shared__ __align__(16) float s_tmu[kMM][kGP];
  __shared__ int s_first[kEmitBins + 1];              // directions before each bin
  __shared__ short s_order[kEmitDirs], s_bin[kEmitDirs];
  __shared__ int s_longest;                           // bits of the largest squared length of a direction
  const int G = kExact > 0 ? kExact : tb.G, TM = kExact ? kMM : traced_materials, M = kExact ? kMM : tb.M;
  const bool traced = kExact || tau_mu != nullptr;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int d0 = blockIdx.y * kEmitDirs;
  const int nd = min(kEmitDirs, K - d0);
  for (int i = tid; i < nd * 3; i += nthreads) s_om[i / 3][i % 3] = omegas[3 * d0 + i];
  for (int i = tid; i < kMM * kGP; i += nthreads) {
    const int m = i / kGP, q = i % kGP;
    s_tmu[m][q] = (traced && m < TM && q < G) ? tau_mu[m * G + q] : 0.f;
  }
  for (int i = tid; i <= kEmitBins; i += nthreads) s_first[i] = 0;
  if (tid == 0) s_longest = __float_as_int(1.f);

  const int64_t v = (int64_t)blockIdx.x * 32 + lane;
  const bool valid = v < in.V;
  const int64_t NC = (int64_t)pg.Rc * pg.Cc * pg.Sc;
  float muc[kGP];
  float ux = 0.f, uy = 0.f, uz = 0.f, h = 0.f, offx = 0.f, offy = 0.f, offz = 0.f;
  int64_t cell = 0;
#pragma unroll
  for (int q = 0; q < kGP; ++q) muc[q] = 0.f;
  if (valid) {
    int i, j, k;
    point_rcs(v, pg, i, j, k);
    primary_direction(__ldg(in.ax_x + j), __ldg(in.ax_y + i), __ldg(in.ax_z + k), in.r0x, in.r0y, in.r0z, ux, uy, uz);
    const int F = pg.f, ic = i / F, jc = j / F, kc = k / F;
    cell = ((int64_t)ic * pg.Cc + jc) * pg.Sc + kc;
    const float half = (F - 1) * 0.5f;
    offy = dy * ((float)(i - ic * F) - half);
    offx = dx * ((float)(j - jc * F) - half);
    offz = dz * ((float)(k - kc * F) - half);
    h = heights ? __ldg(heights + v) : 0.f;
    if (!kQ1) {
#pragma unroll
      for (int q = 0; q < kGP; ++q)
        if (q < G) muc[q] = __ldg(mu + (int64_t)q * NC + cell);
    }
  }
  // the middle of the block's primary directions, and the farthest of them in nodes of the table (every warp holds all
  // 32 points): a direction's nodes at the block's points lie that far around its node at the middle
  float c[3] = {ux, uy, uz}, margin = 0.f;
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    float lo = valid ? c[a] : INFINITY, hi = valid ? c[a] : -INFINITY;
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) {
      lo = fminf(lo, __shfl_xor_sync(0xffffffffu, lo, off));
      hi = fmaxf(hi, __shfl_xor_sync(0xffffffffu, hi, off));
    }
    const float mid = 0.5f * (lo + hi);
    if (valid) margin = fmaf(c[a] - mid, c[a] - mid, margin);
    c[a] = mid;
  }
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) margin = fmaxf(margin, __shfl_xor_sync(0xffffffffu, margin, off));
  int shift = 0;                                      // nodes per bin, as a power of two
  while (((tb.N - 1) >> shift) >= kEmitBins) ++shift;
  __syncthreads();  // s_om, s_tmu and the zeroed bins are complete
  for (int i = tid; i < nd; i += nthreads) {
    const float length2 = s_om[i][0] * s_om[i][0] + s_om[i][1] * s_om[i][1] + s_om[i][2] * s_om[i][2];
    if (!(length2 <= 1.005f)) atomicMax(&s_longest, __float_as_int(length2));
    int node;
    float w;
    table_position(tb, c[0] * s_om[i][0] + c[1] * s_om[i][1] + c[2] * s_om[i][2], node, w);
    s_bin[i] = (short)(node >> shift);
    atomicAdd(&s_first[(node >> shift) + 1], 1);
  }
  __syncthreads();
  // the directions' lengths (up to 1.0025 taken as 1) and the cosines are rounded: one node and 1.01 cover more than that
  const float nodes_away =
      1.01f * sqrtf(margin * __int_as_float(s_longest)) * (float)(tb.N - 1) / (tb.eta_hi - tb.eta_lo) + 1.f;
  const int reach = nodes_away < 4096.f ? (int)nodes_away + 1 : 4096;
  // nodes [first of a bin - reach, last of the bin + reach + 1] have to fit the ring, or the window of rows in its place
  constexpr int kFloats = emission_floats(kGP, kMM);
  const int bin_nodes = 2 * reach + 1 + (1 << shift);
  const bool ring = bin_nodes <= kRing;
  const int window = kFloats / window_node_stride(M, G);
  if (warp == 0) {  // running sums over the bins, 16 a lane
    constexpr int kPer = kEmitBins / 32;
    int count = 0;
    for (int q = 0; q < kPer; ++q) count += s_first[1 + lane * kPer + q];
    int before = count;
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
      const int other = __shfl_up_sync(0xffffffffu, before, off);
      if (lane >= off) before += other;
    }
    before -= count;
    for (int q = 0; q < kPer; ++q) {
      before += s_first[1 + lane * kPer + q];
      s_first[1 + lane * kPer + q] = before;
    }
  }
  __syncthreads();
  // directions by bin; their order within one changes nothing, every direction's result is its own. A bin's first
  // place moves up to the next bin's.
  for (int i = tid; i < nd; i += nthreads) s_order[atomicAdd(&s_first[s_bin[i]], 1)] = (short)i;
  __syncthreads();
  // the point's densities and fluence, read where nodes are formed (registers short in the direction loop)
  auto load_inputs = [&](float* rho, float* phi) {
#pragma unroll
    for (int m = 0; m < kMM; ++m) rho[m] = valid && m < M ? __ldg(in.rho + (int64_t)m * in.V + v) : 0.f;
#pragma unroll
    for (int q = 0; q < kGP; ++q) phi[q] = valid && q < G ? __ldg(in.phi + (int64_t)q * in.V + v) : 0.f;
  };

  const float* multiple_c = multiple + (d0 * NC + cell) * G;  // of the block's first direction
  const float* tau_c = tau + (d0 * NC + cell) * (traced ? TM : G);
  const int64_t multiple_step = NC * G, tau_step = NC * (traced ? TM : G);
  float* out_v = out + (d0 * in.V + v) * (signal_weight != nullptr ? 1 : G);
  const int64_t out_step = in.V * (signal_weight != nullptr ? 1 : G);
  // directions s_order[from .. to) of this warp: kPlace 0 the table's rows in global memory, 1 their nodes in the ring, 2 the
  // rows of the nodes [win_lo, win_lo + win_n) in the window
  auto directions = [&](auto place, int from, int to, int win_lo = 0, int win_n = 2) {
    constexpr int kPlace = decltype(place)::value;
    constexpr bool kRinged = kPlace == 1;
    float rho[kRinged ? 1 : kMM], phi[kRinged ? 1 : kGP];
    if constexpr (!kRinged) load_inputs(rho, phi);
    float smc_n[kGP], P_n[kMM];
    auto fetch = [&](int at) {
      if (valid && at < to) {
        const int dd = s_order[at];
        load_groups<kGP, kVec>(multiple_c + dd * multiple_step, G, smc_n);
        if (traced) {
#pragma unroll
          for (int m = 0; m < kMM; ++m) P_n[m] = m < TM ? __ldg(tau_c + dd * tau_step + m) : 0.f;
        }
      }
    };
    fetch(from + warp);
    for (int at = from + warp; at < to; at += kEmitWarps) {
      const int dd = s_order[at];
      const int64_t d = d0 + dd;
      float e[kGP];
#pragma unroll
      for (int q = 0; q < kGP; ++q) e[q] = 0.f;
      float smc[kGP], P[kMM];
#pragma unroll
      for (int q = 0; q < kGP; ++q) smc[q] = smc_n[q];
#pragma unroll
      for (int m = 0; m < kMM; ++m) P[m] = P_n[m];
      fetch(at + kEmitWarps);  // the next direction's loads in flight during this one's arithmetic
      if (valid) {
        const float ox = s_om[dd][0], oy = s_om[dd][1], oz = s_om[dd][2];
        const float cosine = ux * ox + uy * oy + uz * oz;
        int i0;
        float w;
        table_position(tb, cosine, i0, w);
        const float offset = kQ1 ? 0.f : oy * offy + ox * offx + oz * offz;
        const float *slot0, *slot1;  // in the ring, or the nodes' rows
        if constexpr (kRinged) {
          slot0 = s_ring + (i0 & (kRing - 1)) * kGP * 32;
          slot1 = s_ring + ((i0 + 1) & (kRing - 1)) * kGP * 32;
        } else if constexpr (kPlace == 2) {
          const int NS = window_node_stride(M, G);
          slot0 = s_ring + min(max(i0 - win_lo, 0), win_n - 2) * NS;  // within the window in any case
          slot1 = slot0 + NS;
        } else {
          slot0 = tb.t + (int64_t)i0 * G * G;
          slot1 = slot0 + G * G;
        }
        constexpr int kN = kGP < 4 ? kGP : 4;
#pragma unroll
        for (int q = 0; q < kGP; q += kN) {
          if (q >= G) break;
          float t[kN], f0[kN], f1[kN];
          if (traced) {  // sum_m mu[m, g] P_m, in material order
#pragma unroll
            for (int g = 0; g < kN; ++g) t[g] = 0.f;
#pragma unroll
            for (int m = 0; m < kMM; ++m) {  // materials past TM: zero lengths
              if (kMM <= 2 || m < TM) {
#pragma unroll
                for (int g = 0; g < kN; ++g) t[g] = fmaf(s_tmu[m][q + g], P[m], t[g]);
              }
            }
          } else {
            load_groups<kN, kVec>(tau_c + dd * tau_step + q, G - q, t);
          }
          if constexpr (kRinged) {
            load_ring<kN>(slot0, q, lane, f0);
            load_ring<kN>(slot1, q, lane, f1);
          } else {
            node_pair_sums<kGP, kMM, kVec, kExact, kPlace == 2, kN>(
                tb, slot0, slot1, kPlace == 2 ? G * G : (int64_t)tb.N * G * G, q, rho, phi, f0, f1);
          }
#pragma unroll
          for (int g = 0; g < kN; ++g) {  // groups past G: zero sources and depths
            const float depth = kQ1 ? fmaxf(t[g], 0.f) : fmaxf(t[g] - muc[q + g] * offset, 0.f);
            // the fast exponential: within a few ulp for these depths
            e[q + g] = (interpolate_nodes(f0[g], f1[g], w) + smc[q + g]) * __expf(-depth);
          }
        }
      }
      const float tot = tree_sum<kGP>(e);
      if (signal_weight != nullptr) {
        float sg[kGP];
        load_groups<kGP, kVec>(signal_weight + d * G, G, sg);
#pragma unroll
        for (int q = 0; q < kGP; ++q) sg[q] = __fmul_rn(sg[q], e[q]);
        if (valid) out_v[dd * out_step] = tree_sum<kGP>(sg);
      } else if (valid) {
        float* o = out_v + dd * out_step;
        if (kVec) {
#pragma unroll
          for (int q = 0; q < kGP / 4; ++q)
            if (4 * q < G) reinterpret_cast<float4*>(o)[q] = make_float4(e[4 * q], e[4 * q + 1], e[4 * q + 2], e[4 * q + 3]);
        } else {
#pragma unroll
          for (int q = 0; q < kGP; ++q)
            if (q < G) o[q] = e[q];
        }
      }
      // a butterfly over the block's points
      float a = tot, b = __fmul_rn(tot, h);
#pragma unroll
      for (int off = 1; off < 32; off <<= 1) {
        a += __shfl_xor_sync(0xffffffffu, a, off);
        b += __shfl_xor_sync(0xffffffffu, b, off);
      }
      if (lane == 0) {
        partial[(d * gridDim.x + blockIdx.x) * 2] = a;
        partial[(d * gridDim.x + blockIdx.x) * 2 + 1] = b;
      }
    }
  };
  if (!ring && bin_nodes > window) {  // points too far apart for either (uniform over the block)
    directions(std::integral_constant<int, 0>{}, 0, nd);
    return;
  }
  // the points' own sums between the rows of the next nodes of the table: 32^3 points, 8 groups, 512 directions, a source at 60
  // of a box 32 long 0.60 ms, from global memory 2.6
  if (!ring) {
    for (int from = 0; from < nd;) {
      const int first = (s_bin[s_order[from]] << shift) - reach;
      const int bins = min((first + window - 1 - reach) >> shift, kEmitBins);  // as below
      const int to = s_first[bins - 1];
      const int lo = max(first, 0), hi = min(tb.N - 1, (s_bin[s_order[to - 1]] << shift) + (1 << shift) + reach);
      copy_window<kExact>(tb, lo, hi + 1 - lo, warp, kEmitWarps, tid, nthreads, s_ring);
      __syncthreads();
      directions(std::integral_constant<int, 2>{}, from, to, lo, hi + 1 - lo);
      __syncthreads();
      from = to;
    }
    return;
  }
  // this warp's rows of one node, [material][G][G], and where its lanes find them in the table
  constexpr int kLoads = (kMM * kGP * kGP + 31) / 32;
  float* s_rows = s_ring + kRing * kGP * 32 + warp * kLoads * 32;
  int64_t row_at[kLoads];
#pragma unroll
  for (int q = 0; q < kLoads; ++q) {
    const int e = q * 32 + lane, m = e / (G * G);
    row_at[q] = m < M ? (int64_t)m * tb.N * G * G + (e - m * G * G) : -1;
  }
  int built = 0;  // nodes below this are in the ring or behind it
  for (int from = 0; from < nd;) {
    const int lo = (s_bin[s_order[from]] << shift) - reach;
    // the bins whose nodes all lie below lo + kRing: node + reach + 1 <= lo + kRing - 1 for the last node of the bin
    const int bins = min((lo + kRing - 1 - reach) >> shift, kEmitBins);
    const int to = s_first[bins - 1];
    const int hi = min(tb.N - 1, (s_bin[s_order[to - 1]] << shift) + (1 << shift) + reach);
    if (max(lo, built) <= hi) {
      float rho[kMM], phi[kGP];
      load_inputs(rho, phi);
      int node = max(max(lo, 0), built) + warp;
      // the warp's rows of its next node are loaded while it sums the current one's from its shared memory
      float next[kLoads];
      auto load_rows = [&](int n) {
#pragma unroll
        for (int q = 0; q < kLoads; ++q) next[q] = row_at[q] >= 0 && n <= hi ? __ldg(tb.t + (int64_t)n * G * G + row_at[q]) : 0.f;
      };
      load_rows(node);
      for (; node <= hi; node += kEmitWarps) {
        float f[kGP];
        __syncwarp();
#pragma unroll
        for (int q = 0; q < kLoads; ++q)
          if (row_at[q] >= 0) s_rows[q * 32 + lane] = next[q];
        __syncwarp();
        load_rows(node + kEmitWarps);
        node_sums<kGP, kMM, kVec, kExact>(tb, s_rows, rho, phi, f);
        float* slot = s_ring + (node & (kRing - 1)) * kGP * 32;
        if constexpr (kGP >= 4) {
#pragma unroll
          for (int q = 0; q < kGP; q += 4)
            *reinterpret_cast<float4*>(slot + q * 32 + 4 * lane) = make_float4(f[q], f[q + 1], f[q + 2], f[q + 3]);
        } else {
#pragma unroll
          for (int q = 0; q < kGP; ++q) slot[q * 32 + lane] = f[q];
        }
      }
    }
    built = hi + 1;
    __syncthreads();
    directions(std::integral_constant<int, 1>{}, from, to);
    __syncthreads();  // the ring moves on
    from = to;
  }
}

template <int kGP, int kMM, bool kVec, bool kQ1, int kExact>
int launch_emission_warps_q(const EmissionCall& c) {
  constexpr int bytes = emission_floats(kGP, kMM) * 4;
  auto kernel = emission_warps_kernel<kGP, kMM, kVec, kQ1, kExact>;
  cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
  if (e != cudaSuccess) return set_error(CITRUS_ECUDA, "emission ring: %s", cudaGetErrorString(e));
  const dim3 grid((unsigned)cdiv(c.in.V, kEmitPoints), (unsigned)cdiv(c.K, kEmitDirs));
  kernel<<<grid, 32 * kEmitWarps, bytes, c.stream>>>(c.in, c.tb, c.pg, c.omegas, c.K, c.tau, c.tau_mu, c.TM, c.mu,
                                                     c.multiple, c.heights, c.signal_weight, (float)c.deltas[0],
                                                     (float)c.deltas[1], (float)c.deltas[2], c.out, c.partial);
  note_launches();
  return CITRUS_OK;
}

template <int kGP, int kMM, bool kVec>
int launch_emission_warps_v(const EmissionCall& c) {
  const bool q1 = c.pg.f == 1;
  // Numbers of groups and materials known to the compiler, where the optical depths come by material: us at 32^3 points and
  // 512 directions, known / not: 1 group 151 / 163, 2 155 / 208, 5 282 / 402, 8 326 / 482, 12 688 / 886, 16 782 / 1021. Each number
  // costs two kernels a material count and their compile time, so 9 to 11, 13 to 15 and three materials have none.
  if (c.tau_mu != nullptr && c.tb.M == kMM && c.TM == kMM) {
#define CITRUS_EWE(EXACT)                                                                                     \
  if constexpr (kMM <= 2 && kVec == (EXACT % 4 == 0) && kGP >= EXACT && kGP < 2 * EXACT) {                    \
    if (c.tb.G == EXACT)                                                                                      \
      return q1 ? launch_emission_warps_q<kGP, kMM, kVec, true, EXACT>(c)                                     \
                : launch_emission_warps_q<kGP, kMM, kVec, false, EXACT>(c);                                   \
  }
    CITRUS_EWE(1) CITRUS_EWE(2) CITRUS_EWE(3) CITRUS_EWE(4) CITRUS_EWE(5) CITRUS_EWE(6) CITRUS_EWE(7) CITRUS_EWE(8)
    CITRUS_EWE(12) CITRUS_EWE(16)
#undef CITRUS_EWE
  }
  if constexpr (kMM == 1)
    return launch_emission_warps_v<kGP, 2, kVec>(c);
  else
    return q1 ? launch_emission_warps_q<kGP, kMM, kVec, true, 0>(c) : launch_emission_warps_q<kGP, kMM, kVec, false, 0>(c);
}

// float4 group rows when G is a multiple of 4 and the table, the per-group inputs and the output are 16-byte aligned
template <int kGP>
int launch_emission_warps(const EmissionCall& c) {
  const auto aligned = [](const void* p) { return ((uintptr_t)p % 16) == 0; };
  const bool vec = c.tb.G % 4 == 0 && aligned(c.tb.t) && aligned(c.multiple) && (c.tau_mu != nullptr || aligned(c.tau)) &&
                   (c.signal_weight != nullptr ? aligned(c.signal_weight) : aligned(c.out));
  constexpr bool kCanVec = kGP >= 4;  // G < 4 has no float4 rows
  // one material has exact kernels of its own up to 8 groups (32^3 points, 512 directions, 8 groups 0.38 -> 0.33 ms)
  if (kGP <= 8 && c.tb.M == 1 && c.TM == 1)
    return vec ? launch_emission_warps_v<kGP, kGP <= 8 ? 1 : 2, kCanVec>(c)
               : launch_emission_warps_v<kGP, kGP <= 8 ? 1 : 2, false>(c);
  if (c.tb.M <= 2 && c.TM <= 2)
    return vec ? launch_emission_warps_v<kGP, 2, kCanVec>(c) : launch_emission_warps_v<kGP, 2, false>(c);
  return vec ? launch_emission_warps_v<kGP, kMaxM, kCanVec>(c) : launch_emission_warps_v<kGP, kMaxM, false>(c);
}

}  // namespace
}  // namespace citrus

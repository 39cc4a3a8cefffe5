// Linear-discontinuous discrete-ordinates sweep: the closed-form cell solve of every (entry, direction, group) of a
// diagonal wavefront plane, in place in the chunk's cell-major store [views, 8, Dc, N, 4G].
//
// The cell equations are those of citrus/scatter_solver/linear_discontinuous_cell.py:14-87 (right-hand sides from the
// source and the three upstream neighbours, then the closed-form 4 x 4 solve), evaluated term by term in float32: the
// coefficients of a lane with IEEE division, the per-view quotients as products with correctly rounded reciprocals.
// Two drivers share the lane body: one launch per plane (the reference's plan, sweep_kernels.py:265-290) and one
// persistent cooperative launch that walks all planes with a bounded grid barrier between them, so a whole chunk is a
// single launch.
#include "common.cuh"
#include <mutex>

namespace citrus {
namespace {

constexpr int kThreads = 256;

template <bool kCoherent>
__device__ __forceinline__ float4 load4(const float4* p) {
  if (kCoherent) return __ldcg(p);  // L2 only: written by other SMs this launch
  return *p;
}

// The view-independent part of one lane (entry e of the plane, direction d of the chunk, group g): the octant signs,
// the direction's c_a, every coefficient of the 4 x 4 solve that depends on c and the cell's attenuation only, and
// the float4 positions within one view's store of the cell and of its three upstream neighbours (upstream neighbours
// lie on the previous plane, already swept; kVacuum marks a vacuum face, which reads zeros). The views of a launch
// share it: a thread computes it once and solves the lane in every view.
constexpr uint32_t kVacuum = 0xffffffffu;

struct LaneCoef {
  float sx, sy, sz, cx, cy, cz;
  float k3x, k3y, k3z;  // 3 s_a c_a
  float rdx, rdy, rdz;  // 1 / d_a, d_a = 3 c_a + sum_{b != a} c_b + m
  float qsx, qsy, qsz;  // s_a c_a / d_a
  float rden;           // 1 / (sum_a c_a + m + 3 sum_a c_a q_a)
  uint32_t at, ax, ay, az;
  bool plain;  // the direction's c_a are 0 or within [kPlainMin, kPlainMax]
};

// c_a and m between these (or 0) keep d_a, its reciprocal, c_a / d_a and the remainder of quotient() normal numbers
constexpr float kPlainMin = 1e-18f, kPlainMax = 1e18f;

__device__ __forceinline__ bool plain_c(float c) { return c == 0.f || (c >= kPlainMin && c <= kPlainMax); }

// a / b from the correctly rounded reciprocal r of b, which the lane needs as well: the product a r corrected once by its
// exact remainder (Markstein, Computation of elementary functions on the IBM RISC System/6000 processor, 1990), the
// rounding of an IEEE division for normal numbers (no other result in 6e8 random pairs). Three such quotients are nine
// instructions; three divisions were a quarter of a lane's.
__device__ __forceinline__ float quotient(float a, float b, float r) {
  const float q = __fmul_rn(a, r);
  return __fmaf_rn(__fmaf_rn(-q, b, a), r, q);
}

// The part of a lane that its octant and direction give. Every operation here and below is rounded on its own (no
// multiply-add contraction), so every kernel computes the same bits.
__device__ __forceinline__ void direction_coef(int o, float cx, float cy, float cz, LaneCoef& k) {
  const float sx = (o & 4) ? -1.f : 1.f, sy = (o & 2) ? -1.f : 1.f, sz = (o & 1) ? -1.f : 1.f;
  k.sx = sx, k.sy = sy, k.sz = sz, k.cx = cx, k.cy = cy, k.cz = cz;
  k.plain = plain_c(cx) && plain_c(cy) && plain_c(cz);
  k.k3x = __fmul_rn(__fmul_rn(3.f, sx), cx);
  k.k3y = __fmul_rn(__fmul_rn(3.f, sy), cy);
  k.k3z = __fmul_rn(__fmul_rn(3.f, sz), cz);
}

// The part that the cell's attenuation m gives for that direction
__device__ __forceinline__ void cell_coef(float m, LaneCoef& k) {
  const float cx = k.cx, cy = k.cy, cz = k.cz;
  const float csum = __fadd_rn(__fadd_rn(cx, cy), cz);
  const float dx = __fadd_rn(__fadd_rn(__fmul_rn(3.f, cx), __fsub_rn(csum, cx)), m);
  const float dy = __fadd_rn(__fadd_rn(__fmul_rn(3.f, cy), __fsub_rn(csum, cy)), m);
  const float dz = __fadd_rn(__fadd_rn(__fmul_rn(3.f, cz), __fsub_rn(csum, cz)), m);
  k.rdx = __frcp_rn(dx);
  k.rdy = __frcp_rn(dy);
  k.rdz = __frcp_rn(dz);
  float qx, qy, qz;
  if (k.plain && m >= 0.f && m <= kPlainMax) {
    qx = quotient(cx, dx, k.rdx), qy = quotient(cy, dy, k.rdy), qz = quotient(cz, dz, k.rdz);
  } else {
    qx = __fdiv_rn(cx, dx), qy = __fdiv_rn(cy, dy), qz = __fdiv_rn(cz, dz);
  }
  const float qsum = __fadd_rn(__fadd_rn(__fmul_rn(cx, qx), __fmul_rn(cy, qy)), __fmul_rn(cz, qz));
  k.rden = __frcp_rn(__fadd_rn(__fadd_rn(csum, m), __fmul_rn(3.f, qsum)));
  k.qsx = __fmul_rn(k.sx, qx);
  k.qsy = __fmul_rn(k.sy, qy);
  k.qsz = __fmul_rn(k.sz, qz);
}

// The lane of entry e, direction d and group g; every float4 position of a view is below 2^31 (checked on the host)
template <int kG>
__device__ __forceinline__ void lane_coef_edg(uint32_t e, uint32_t d, uint32_t g, LaneCoef& k,
                                              const float* __restrict__ mu, const float* __restrict__ c,
                                              const int* __restrict__ octant, const int* __restrict__ cell,
                                              const int* __restrict__ upstream, uint32_t N, int G_runtime,
                                              uint32_t Dc) {
  const uint32_t G = kG > 0 ? kG : G_runtime;
  const int o = __ldg(octant + e);
  const uint32_t n = __ldg(cell + e);
  const uint32_t ux = __ldg(upstream + 3 * e), uy = __ldg(upstream + 3 * e + 1), uz = __ldg(upstream + 3 * e + 2);
  const uint32_t od = (uint32_t)o * Dc + d;
  const float cx = __ldg(c + 3 * od), cy = __ldg(c + 3 * od + 1), cz = __ldg(c + 3 * od + 2);
  const float m = __ldg(mu + (size_t)n * G + g);
  const uint32_t base = od * N;
  k.at = (base + n) * G + g;
  k.ax = ux < N ? (base + ux) * G + g : kVacuum;
  k.ay = uy < N ? (base + uy) * G + g : kVacuum;
  k.az = uz < N ? (base + uz) * G + g : kVacuum;
  direction_coef(o, cx, cy, cz, k);
  cell_coef(m, k);
}

// lane = (e - start) Dc G + d G + g of a plane starting at entry start
template <int kG>
__device__ __forceinline__ void lane_coef(uint32_t lane, LaneCoef& k, const float* __restrict__ mu,
                                          const float* __restrict__ c, const int* __restrict__ octant,
                                          const int* __restrict__ cell, const int* __restrict__ upstream,
                                          uint32_t start, uint32_t N, int G_runtime, uint32_t Dc) {
  const uint32_t G = kG > 0 ? kG : G_runtime;
  const uint32_t g = lane % G, t = lane / G;
  lane_coef_edg<kG>(start + t / Dc, t % Dc, g, k, mu, c, octant, cell, upstream, N, G_runtime, Dc);
}

// The store moments a lane reads in one view: the source (s) and (psi0, psi_x, psi_y, psi_z) of the x, y, z upstream
// neighbours
struct LaneIn {
  float4 s, X, Y, Z;
};

template <bool kCoherent>
__device__ __forceinline__ void gather_view(const LaneCoef& k, const float4* view, LaneIn& in) {
  const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
  in.s = load4<kCoherent>(view + k.at);
  in.X = k.ax != kVacuum ? load4<kCoherent>(view + k.ax) : zero;
  in.Y = k.ay != kVacuum ? load4<kCoherent>(view + k.ay) : zero;
  in.Z = k.az != kVacuum ? load4<kCoherent>(view + k.az) : zero;
}

// The closed-form cell solve of the equations of linear_discontinuous_cell.py:14-87 in one view
__device__ __forceinline__ float4 solve_cell(const LaneCoef& k, const LaneIn& in) {
  const float4 s = in.s, X = in.X, Y = in.Y, Z = in.Z;
  // face-averaged inflow psibar_a = psi_0[N_a] + s_a psi_a[N_a]
  const float pbx = __fadd_rn(X.x, __fmul_rn(k.sx, X.y));
  const float pby = __fadd_rn(Y.x, __fmul_rn(k.sy, Y.z));
  const float pbz = __fadd_rn(Z.x, __fmul_rn(k.sz, Z.w));
  const float r0 =
      __fadd_rn(s.x, __fadd_rn(__fadd_rn(__fmul_rn(k.cx, pbx), __fmul_rn(k.cy, pby)), __fmul_rn(k.cz, pbz)));
  // R_a = S_a - 3 s_a c_a psibar_a + sum_{b != a} c_b psi_a[N_b]
  const float rx = __fadd_rn(__fsub_rn(s.y, __fmul_rn(k.k3x, pbx)), __fadd_rn(__fmul_rn(k.cy, Y.y), __fmul_rn(k.cz, Z.y)));
  const float ry = __fadd_rn(__fsub_rn(s.z, __fmul_rn(k.k3y, pby)), __fadd_rn(__fmul_rn(k.cx, X.z), __fmul_rn(k.cz, Z.z)));
  const float rz = __fadd_rn(__fsub_rn(s.w, __fmul_rn(k.k3z, pbz)), __fadd_rn(__fmul_rn(k.cx, X.w), __fmul_rn(k.cy, Y.w)));
  const float corr =
      __fadd_rn(__fadd_rn(__fmul_rn(k.qsx, rx), __fmul_rn(k.qsy, ry)), __fmul_rn(k.qsz, rz));
  // the per-view quotients as products with the lane's correctly rounded reciprocals (within 1.5 ulp of the quotient)
  const float p0 = __fmul_rn(__fsub_rn(r0, corr), k.rden);
  float4 out;
  out.x = p0;
  out.y = __fmul_rn(__fadd_rn(rx, __fmul_rn(k.k3x, p0)), k.rdx);
  out.z = __fmul_rn(__fadd_rn(ry, __fmul_rn(k.k3y, p0)), k.rdy);
  out.w = __fmul_rn(__fadd_rn(rz, __fmul_rn(k.k3z, p0)), k.rdz);
  return out;
}

// ... stored over the source
__device__ __forceinline__ void solve_view(const LaneCoef& k, const LaneIn& in, float4* view) {
  view[k.at] = solve_cell(k, in);
}

// One plane, one lane (view v, entry, direction, group) per thread: the reference's launch plan.
template <int kG>
__global__ void __launch_bounds__(kThreads) plane_kernel(float4* __restrict__ store, const float* __restrict__ mu,
                                                         const float* __restrict__ c, const int* __restrict__ octant,
                                                         const int* __restrict__ cell, const int* __restrict__ upstream,
                                                         uint32_t start, uint32_t per_view, uint32_t N, int G,
                                                         uint32_t Dc, int64_t views, int64_t view_stride) {
  const int64_t lane = (int64_t)blockIdx.x * kThreads + threadIdx.x;
  if (lane >= views * per_view) return;
  const int64_t v = lane / per_view;
  LaneCoef k;
  lane_coef<kG>((uint32_t)(lane - v * per_view), k, mu, c, octant, cell, upstream, start, N, G, Dc);
  LaneIn in;
  float4* view = store + v * view_stride;
  gather_view<false>(k, view, in);
  solve_view(k, in, view);
}

// All planes in one cooperative launch, with a bounded grid barrier between planes. A thread takes one lane (entry,
// direction, group) of a plane at a time and solves it in every view, kVB views at a time: the loads of kVB views are
// issued before their solves (which a plain loop cannot do: the stores might alias the next view's loads as far as
// the compiler knows; within a plane they never do).
template <int kG, int kVB, int kMinBlocks>
__global__ void __launch_bounds__(kThreads, kMinBlocks) persistent_kernel(
    float4* __restrict__ store, const float* __restrict__ mu, const float* __restrict__ c,
    const int* __restrict__ octant, const int* __restrict__ cell, const int* __restrict__ upstream,
    const int* __restrict__ offsets, int num_planes, uint32_t N, int G, uint32_t Dc, int views, int64_t view_stride,
    unsigned* sync, uint64_t timeout_ns, int skip) {
  const uint32_t stride = gridDim.x * kThreads;
  const uint32_t per_entry = Dc * (kG > 0 ? kG : G);
  for (int p = 0; p < num_planes; ++p) {
    const uint32_t start = __ldg(offsets + p);
    const uint32_t total = (__ldg(offsets + p + 1) - start) * per_entry;
    for (uint32_t lane = blockIdx.x * kThreads + threadIdx.x; lane < total; lane += stride) {
      LaneCoef k;
      lane_coef<kG>(lane, k, mu, c, octant, cell, upstream, start, N, G, Dc);
      float4* view = store;
      for (int v0 = 0; v0 < views; v0 += kVB, view += kVB * view_stride) {
        LaneIn in[kVB];
#pragma unroll
        for (int j = 0; j < kVB; ++j)
          if (v0 + j < views) gather_view<true>(k, view + j * view_stride, in[j]);
#pragma unroll
        for (int j = 0; j < kVB; ++j)
          if (v0 + j < views) solve_view(k, in[j], view + j * view_stride);
      }
    }
    if (p + 1 < num_planes && !grid_barrier(sync, gridDim.x, timeout_ns, skip)) return;
  }
}

// The tiled schedule: in each octant's sweep frame the cells are cut into tiles of T^3; the tiles with the same sum
// of tile coordinates (a tile diagonal) depend only on earlier diagonals, so the grid barrier runs once per tile
// diagonal instead of once per plane. A block takes one task (a tile of one octant and a block of up to dpb
// directions) and walks the tile's 3 T - 2 sub-planes (cells with the same sum of in-tile coordinates) with a block
// barrier between them: the upstream reads of a sub-plane are the block's own writes one sub-plane earlier (L2 hits),
// and only the reads across a tile face come from an earlier diagonal. Every lane is the per-plane kernel's lane with
// the same inputs, so the store comes out bit for bit the same.
//
// Tables (host-built, transport_sweep.build_tiled_plan): entries (octant, cell, upstream) ordered by task and
// sub-plane; sub_offsets [tasks, num_sub + 1] the entry range of each sub-plane of each task; diagonal_offsets
// [num_diagonals + 1] the task range of each diagonal.
template <int kG, int kVB, int kMinBlocks>
__global__ void __launch_bounds__(kThreads, kMinBlocks) tiled_kernel(
    float4* __restrict__ store, const float* __restrict__ mu, const float* __restrict__ c,
    const int* __restrict__ octant, const int* __restrict__ cell, const int* __restrict__ upstream,
    const int* __restrict__ diagonal_offsets, const int* __restrict__ sub_offsets, int num_diagonals, int num_sub,
    uint32_t N, int G_runtime, uint32_t Dc, uint32_t dpb, int views, int64_t view_stride, unsigned* sync,
    uint64_t timeout_ns, int skip) {
  const uint32_t G = kG > 0 ? kG : G_runtime;
  const uint32_t dir_blocks = (Dc + dpb - 1) / dpb;
  for (int D = 0; D < num_diagonals; ++D) {
    const uint32_t t0 = __ldg(diagonal_offsets + D);
    const uint32_t work = (__ldg(diagonal_offsets + D + 1) - t0) * dir_blocks;
    for (uint32_t w = blockIdx.x; w < work; w += gridDim.x) {
      const uint32_t task = t0 + w / dir_blocks, d0 = (w % dir_blocks) * dpb;
      const uint32_t nd = min(dpb, Dc - d0);
      const int* so = sub_offsets + (size_t)task * (num_sub + 1);
      for (int sp = 0; sp < num_sub; ++sp) {
        const uint32_t start = __ldg(so + sp), count = __ldg(so + sp + 1) - start;
        if (count == 0) continue;  // the same for every thread of the block
        const uint32_t total = count * nd * G;
        for (uint32_t lane = threadIdx.x; lane < total; lane += kThreads) {
          const uint32_t g = lane % G, t = lane / G;
          LaneCoef k;
          lane_coef_edg<kG>(start + t / nd, d0 + t % nd, g, k, mu, c, octant, cell, upstream, N, G_runtime, Dc);
          float4* view = store;
          for (int v0 = 0; v0 < views; v0 += kVB, view += kVB * view_stride) {
            LaneIn in[kVB];
#pragma unroll
            for (int j = 0; j < kVB; ++j)
              if (v0 + j < views) gather_view<true>(k, view + j * view_stride, in[j]);
#pragma unroll
            for (int j = 0; j < kVB; ++j)
              if (v0 + j < views) solve_view(k, in[j], view + j * view_stride);
          }
        }
        __syncthreads();  // the sub-plane's outputs are written before the next sub-plane reads them
      }
    }
    if (D + 1 < num_diagonals && !grid_barrier(sync, gridDim.x, timeout_ns, skip)) return;
  }
}

// ---- pencils ------------------------------------------------------------------------------------------------------
// The wavefront without grid barriers. In each octant's sweep frame the (row, column) plane is cut into tiles of T x T
// pencils; a task is one tile of one (octant, block of dpb directions, block of kVB views), and a block walks its pencils
// along the slices, a thread per (pencil, direction, group), pencil (i, j) of the tile i + j steps behind the first. A
// thread keeps its own last cell (the z inflow) in registers and hands its outputs to the pencils (i + 1, j) and
// (i, j + 1) of the tile through shared memory one step later; only the tile's faces read what another block wrote.
// Shared memory is a ring of kPencilSlots steps of (T + 1) x (T + 1) pencils, the first row and column being the inflow
// through the faces. The sources and face inflows of the next kPencilAhead steps are on their way to it (cp.async, each
// thread into places that it alone reads), and a step's output takes its source's place, so a step costs one block
// barrier, every inflow is read at the same offset, and no thread waits for memory.
// Tasks come from a counter, by views and then by tile diagonal over all octants and directions; a task waits, with a
// limit, for the flags of its two upstream tiles, which earlier tasks set. A block holds one task at a time and the
// earliest unfinished task never waits, so every wait ends, however many blocks are resident.
// Against the plane wavefront it reads a cell's source once and its own outputs not at all (three neighbours per cell
// came from L2), loads no entry tables, and needs no grid barrier: 64^3 cells, 8 groups, 120 directions 3.81 -> 2.31 ms,
// in pairs of views 2.92 -> 1.77 ms per view; 32^3, one group 0.57 -> 0.21 ms. Its issue slots are 70 % busy (about 250
// instructions per cell, half of them the coefficients that two views share); HBM's floor at 64^3 is 1.19 ms.
constexpr int kPencilSlots = 5;
constexpr int kPencilAhead = kPencilSlots - 2;  // a slot is refilled a barrier after the neighbours read its outputs
constexpr int kPencilThreads = 512;
constexpr int kPencilFlag = 4;  // the first flag among the sync words: 0 the task counter, 1 progress, 2 the error word
constexpr int kPencilBeat = 512 * kPencilSlots;  // steps between two signs of progress

struct Pencils {
  uint32_t R, C, S, G, Dc, dpb, T;  // grid, groups, directions of an octant and of a task, tile edge
  uint32_t tiles_r, tiles_c, dir_blocks, sequences, total;  // tiles along rows and columns; (octant, directions) pairs
};

// 16 bytes to shared memory if `issue`: those at src, or zeros if bytes is 0 (predicated: a branch per copy costs more)
__device__ __forceinline__ void cp_async16_if(bool issue, uint32_t dst, const void* src, int bytes = 16) {
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %0, 0;\n\t"
      "@p cp.async.cg.shared.global [%1], [%2], 16, %3;\n\t}" ::"r"((int)issue), "r"(dst), "l"(src), "r"(bytes) : "memory");
}

__device__ __forceinline__ float4 load_shared4(uint32_t at) {
  float4 v;
  asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(at));
  return v;
}

__device__ __forceinline__ void store_shared4(uint32_t at, float4 v) {
  asm volatile("st.shared.v4.f32 [%0], {%1, %2, %3, %4};" ::"r"(at), "f"(v.x), "f"(v.y), "f"(v.z), "f"(v.w) : "memory");
}

// The next task of the block as (sequence, tile row, tile column, flag index), its inflow complete; false when there is
// none or a wait ran out. One thread.
__device__ __forceinline__ bool next_pencil_task(const Pencils& p, unsigned* sync, uint64_t timeout_ns, uint32_t out[4]) {
  const uint32_t id = atomicAdd(&sync[0], 1u);
  if (id >= p.total) return false;
  const uint32_t tiles = p.tiles_r * p.tiles_c, per_view = p.sequences * tiles;
  const uint32_t v = id / per_view, rem = id - v * per_view;
  const uint32_t rank = rem / p.sequences;
  const uint32_t q = v * p.sequences + (rem - rank * p.sequences);
  // the tile of that rank by diagonals: they grow to n = min(tiles_r, tiles_c) tiles, stay so and shrink again
  const uint32_t n = min(p.tiles_r, p.tiles_c), wide = max(p.tiles_r, p.tiles_c) - n + 1;
  const uint32_t grow = (uint32_t)((uint64_t)n * (n - 1) / 2);
  uint32_t D, place;
  if (rank >= grow && rank - grow < n * wide) {
    D = n - 1 + (rank - grow) / n;
    place = (rank - grow) % n;
  } else {
    const bool shrinking = rank >= grow;
    const uint32_t r = shrinking ? tiles - 1 - rank : rank;
    uint32_t e = (uint32_t)((sqrt(8.0 * r + 1.0) - 1.0) * 0.5);  // the last e with e (e + 1) / 2 <= r
    while ((uint64_t)e * (e + 1) / 2 > r) --e;
    while ((uint64_t)(e + 1) * (e + 2) / 2 <= r) ++e;
    place = r - (uint32_t)((uint64_t)e * (e + 1) / 2);
    if (shrinking) place = e - place;
    D = shrinking ? p.tiles_r + p.tiles_c - 2 - e : e;
  }
  const uint32_t I = (D >= p.tiles_c ? D - p.tiles_c + 1 : 0) + place, J = D - I;
  const uint32_t flag = q * tiles + I * p.tiles_c + J;
  const unsigned* flags = sync + kPencilFlag;
  // the limit is on the time without progress of any block: upstream tasks may wait in turn, and a task of a long grid
  // may take longer than any sensible limit
  uint64_t t0 = global_timer_ns();
  unsigned seen = ld_acquire_u32(&sync[1]);
  for (int a = 0; a < 2; ++a) {
    if ((a == 0 ? I : J) == 0) continue;
    const unsigned* f = flags + flag - (a == 0 ? p.tiles_c : 1);
    while (ld_acquire_u32(f) == 0u) {
      if (ld_acquire_u32(&sync[2]) != 0u) return false;
      const unsigned now = ld_acquire_u32(&sync[1]);
      if (now != seen) {
        seen = now;
        t0 = global_timer_ns();
      } else if (global_timer_ns() - t0 > timeout_ns) {
        atomicExch(&sync[2], 1u);
        return false;
      }
      __nanosleep(64);
    }
  }
  __threadfence();
  out[0] = q, out[1] = I, out[2] = J, out[3] = flag;
  return true;
}

template <int kG, int kVB>
__global__ void __launch_bounds__(kPencilThreads, 2) pencil_kernel(float4* __restrict__ store,
                                                                   const float* __restrict__ mu,
                                                                   const float* __restrict__ c, Pencils p, int views,
                                                                   int64_t view_stride, unsigned* sync,
                                                                   uint64_t timeout_ns, int skip) {
  extern __shared__ float4 s_pencil[];  // [kPencilSlots][kVB][T + 1][T + 1][L]
  __shared__ uint32_t s_task[4];
  __shared__ int s_go;
  const uint32_t G = kG > 0 ? kG : p.G, L = p.dpb * G, T = p.T;
  const uint32_t tid = threadIdx.x, l = tid % L, col = tid / L, tj = col % T, ti = col / T, dd = l / G, g = l - dd * G;
  const uint32_t to_x = 16 * L, to_y = (T + 1) * to_x, view_bytes = (T + 1) * to_y, slot_bytes = kVB * view_bytes;
  const uint32_t mine = (uint32_t)__cvta_generic_to_shared(s_pencil) + (ti + 1) * to_y + (tj + 1) * to_x + 16 * l;
  const int lag = (int)(ti + tj);
  for (;;) {
    if (tid == 0) s_go = next_pencil_task(p, sync, timeout_ns, s_task);
    __syncthreads();
    if (!s_go) return;
    const uint32_t q = s_task[0], I = s_task[1], J = s_task[2];
    const uint32_t vb = q / p.sequences, od = q - vb * p.sequences, o = od / p.dir_blocks;
    const uint32_t d = (od - o * p.dir_blocks) * p.dpb + dd;
    const uint32_t ip = I * T + ti, jp = J * T + tj;  // the pencil in the octant's sweep frame
    const bool valid = ip < p.R && jp < p.C && d < p.Dc;
    const int v0 = (int)vb * kVB, nv = min(kVB, views - v0);
    const int steps = (int)(p.S + min(T, p.R - I * T) + min(T, p.C - J * T)) - 2;
    const uint32_t S = valid ? p.S : 0u;  // cells of this thread's pencil
    const int dk = (o & 1) ? -(int)G : (int)G;  // float4 (and attenuation) stride to the next cell of the pencil
    // ... and to the x and y upstream cells (0 at a vacuum face, which reads zeros)
    const int up_x = jp == 0 ? 0 : (o & 4) ? (int)(p.S * G) : -(int)(p.S * G);
    const int up_y = ip == 0 ? 0 : (o & 2) ? (int)(p.C * p.S * G) : -(int)(p.C * p.S * G);
    const bool at_face = __any_sync(__activemask(), tj == 0 || ti == 0);  // the warp's pencils at the tile's faces
    const int bytes_x = jp > 0 ? 16 : 0, bytes_y = ip > 0 ? 16 : 0;
    LaneCoef k;
    direction_coef((int)o, 0.f, 0.f, 0.f, k);
    k.at = 0;
    int64_t at = 0;  // the cell that is loaded, as a float4 position; kPencilAhead cells on from the one that is solved
    const float* m_next_at = mu;
    if (valid) {
      const uint32_t i = (o & 2) ? p.R - 1 - ip : ip, j = (o & 4) ? p.C - 1 - jp : jp, k0 = (o & 1) ? p.S - 1 : 0;
      const uint32_t n = (i * p.C + j) * p.S + k0, odir = o * p.Dc + d;
      direction_coef((int)o, __ldg(c + 3 * odir), __ldg(c + 3 * odir + 1), __ldg(c + 3 * odir + 2), k);
      at = v0 * view_stride + ((int64_t)odir * (p.R * p.C * p.S) + n) * G + g - (int64_t)lag * dk;
      m_next_at = mu + ((int64_t)n * G + g) - (int64_t)(lag + kPencilAhead - 1) * dk;
    }
    float4 Z[kVB];
#pragma unroll
    for (int v = 0; v < kVB; ++v) Z[v] = make_float4(0.f, 0.f, 0.f, 0.f);
    float m_next = 0.f;
    // Step t runs in slot (t + kPencilAhead) % kPencilSlots; the inflow of a step is in the slot before it
    for (int t0 = -kPencilAhead; t0 < steps; t0 += kPencilSlots) {
      if (tid == 0 && (uint32_t)(t0 + kPencilAhead) % kPencilBeat == kPencilBeat - kPencilSlots) atomicAdd(&sync[1], 1u);
#pragma unroll
      for (int q5 = 0; q5 < kPencilSlots; ++q5) {
        constexpr int kA = kPencilAhead, kP = kPencilSlots;
        const int t = t0 + q5, here = t - lag;
        if (t >= steps) break;
        const bool load = (uint32_t)(here + kA) < S;
#pragma unroll
        for (int v = 0; v < kVB; ++v) {
          const bool some = load && (kVB == 1 || v < nv);
          const float4* src = store + at + v * view_stride;
          const uint32_t to = mine + v * view_bytes, before = to + (q5 + kA - 1) % kP * slot_bytes;
          cp_async16_if(some, to + (q5 + kA) % kP * slot_bytes, src);
          if (at_face) {
            cp_async16_if(some && tj == 0, before - to_x, src + up_x, bytes_x);
            cp_async16_if(some && ti == 0, before - to_y, src + up_y, bytes_y);
          }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
        const float m = m_next;
        if ((uint32_t)(here + 1) < S) m_next = __ldg(m_next_at);
        m_next_at += dk;
        if (t >= 0) {
          asm volatile("cp.async.wait_group %0;" ::"n"(kA) : "memory");
          if ((uint32_t)here < S) {
            cell_coef(m, k);
            float4* out = store + at - kA * dk;
#pragma unroll
            for (int v = 0; v < kVB; ++v) {
              if (kVB > 1 && v >= nv) break;
              const uint32_t slot = mine + v * view_bytes + q5 * slot_bytes;
              const uint32_t last = mine + v * view_bytes + (q5 + kP - 1) % kP * slot_bytes;
              LaneIn in;
              in.s = load_shared4(slot);
              in.X = load_shared4(last - to_x);
              in.Y = load_shared4(last - to_y);
              in.Z = Z[v];
              Z[v] = solve_cell(k, in);
              out[v * view_stride] = Z[v];
              store_shared4(slot, Z[v]);
            }
          }
          __syncthreads();
        }
        at += dk;
      }
    }
    if (tid == 0) {  // the last step's barrier put the block's stores before this
      __threadfence();
      if ((int)blockIdx.x != skip) {
        st_release_u32(sync + kPencilFlag + s_task[3], 1u);
        atomicAdd(&sync[1], 1u);
      }
    }
  }
}

template <int kG>
int launch_planes(float* store, const float* mu, const float* c, const int* octant, const int* cell,
                  const int* upstream, const int64_t* offsets, int64_t num_planes, int64_t N, int G, int64_t Dc,
                  int64_t views, cudaStream_t stream) {
  const int64_t view_stride = 8 * Dc * N * (int64_t)G;  // float4 per view
  for (int64_t p = 0; p < num_planes; ++p) {
    const int64_t start = offsets[p], E = offsets[p + 1] - offsets[p];
    const int64_t per_view = E * Dc * G;
    if (per_view <= 0) continue;
    plane_kernel<kG><<<(unsigned)cdiv(views * per_view, kThreads), kThreads, 0, stream>>>(
        reinterpret_cast<float4*>(store), mu, c, octant, cell, upstream, (uint32_t)start, (uint32_t)per_view,
        (uint32_t)N, G, (uint32_t)Dc, views, view_stride);
    note_launches();
  }
  return launch_status("citrus_sweep_planes");
}

template <int kG, int kVB, int kMinBlocks = 1>
int launch_persistent_u(float* store, const float* mu, const float* c, const int* octant, const int* cell,
                        const int* upstream, const int* offsets, int num_planes, int64_t N, int G, int64_t Dc,
                        int64_t views, unsigned* sync, int64_t max_blocks, uint64_t timeout_ns, int skip,
                        cudaStream_t stream) {
  int per_sm = 0;
  cudaError_t e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, persistent_kernel<kG, kVB, kMinBlocks>,
                                                                kThreads, 0);
  if (e != cudaSuccess || per_sm < 1) return set_error(CITRUS_ECUDA, "citrus_sweep_persistent: occupancy query failed");
  int64_t blocks = (int64_t)per_sm * num_sms();
  if (max_blocks > 0 && max_blocks < blocks) blocks = max_blocks;
  if (skip >= blocks) skip = (int)blocks - 1;
  float4* store4 = reinterpret_cast<float4*>(store);
  uint32_t n32 = (uint32_t)N, dc32 = (uint32_t)Dc;
  int views32 = (int)views;
  int64_t view_stride = 8 * Dc * N * (int64_t)G;  // float4 per view
  cudaError_t z = cudaMemsetAsync(sync, 0, 4 * sizeof(unsigned), stream);
  if (z != cudaSuccess) return set_error(CITRUS_ECUDA, "citrus_sweep_persistent: %s", cudaGetErrorString(z));
  void* args[] = {&store4, &mu, &c, &octant, &cell, &upstream, &offsets, &num_planes, &n32, &G, &dc32, &views32,
                  &view_stride, &sync, &timeout_ns, &skip};
  e = cudaLaunchCooperativeKernel((const void*)persistent_kernel<kG, kVB, kMinBlocks>, dim3((unsigned)blocks),
                                  dim3(kThreads), args, 0, stream);
  if (e != cudaSuccess) return set_error(CITRUS_ELAUNCH, "citrus_sweep_persistent: %s", cudaGetErrorString(e));
  note_launches();
  return CITRUS_OK;
}

template <int kG, int kVB, int kMinBlocks>
int launch_tiled_u(float* store, const float* mu, const float* c, const int* octant, const int* cell,
                   const int* upstream, const int* diagonal_offsets, const int* sub_offsets, int num_diagonals,
                   int num_sub, int64_t N, int G, int64_t Dc, int64_t dpb, int64_t views, unsigned* sync,
                   int64_t max_blocks, uint64_t timeout_ns, int skip, cudaStream_t stream) {
  int per_sm = 0;
  cudaError_t e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, tiled_kernel<kG, kVB, kMinBlocks>, kThreads,
                                                                0);
  if (e != cudaSuccess || per_sm < 1) return set_error(CITRUS_ECUDA, "citrus_sweep_tiled: occupancy query failed");
  int64_t blocks = (int64_t)per_sm * num_sms();
  if (max_blocks > 0 && max_blocks < blocks) blocks = max_blocks;
  if (skip >= blocks) skip = (int)blocks - 1;
  float4* store4 = reinterpret_cast<float4*>(store);
  uint32_t n32 = (uint32_t)N, dc32 = (uint32_t)Dc, dpb32 = (uint32_t)dpb;
  int views32 = (int)views;
  int64_t view_stride = 8 * Dc * N * (int64_t)G;  // float4 per view
  cudaError_t z = cudaMemsetAsync(sync, 0, 4 * sizeof(unsigned), stream);
  if (z != cudaSuccess) return set_error(CITRUS_ECUDA, "citrus_sweep_tiled: %s", cudaGetErrorString(z));
  void* args[] = {&store4, &mu, &c, &octant, &cell, &upstream, &diagonal_offsets, &sub_offsets, &num_diagonals,
                  &num_sub, &n32, &G, &dc32, &dpb32, &views32, &view_stride, &sync, &timeout_ns, &skip};
  e = cudaLaunchCooperativeKernel((const void*)tiled_kernel<kG, kVB, kMinBlocks>, dim3((unsigned)blocks),
                                  dim3(kThreads), args, 0, stream);
  if (e != cudaSuccess) return set_error(CITRUS_ELAUNCH, "citrus_sweep_tiled: %s", cudaGetErrorString(e));
  note_launches();
  return CITRUS_OK;
}

// the thread forms of the tiled launch: one view at a time (four blocks per SM), or the loads of two views issued
// before their solves (three blocks per SM)
template <int kG>
int launch_tiled(float* store, const float* mu, const float* c, const int* octant, const int* cell,
                 const int* upstream, const int* diagonal_offsets, const int* sub_offsets, int num_diagonals,
                 int num_sub, int64_t N, int G, int64_t Dc, int64_t dpb, int64_t views, unsigned* sync,
                 int64_t max_blocks, uint64_t timeout_ns, int skip, cudaStream_t stream, int form) {
  if (form == 2)
    return launch_tiled_u<kG, 2, 3>(store, mu, c, octant, cell, upstream, diagonal_offsets, sub_offsets,
                                    num_diagonals, num_sub, N, G, Dc, dpb, views, sync, max_blocks, timeout_ns, skip,
                                    stream);
  if (form == 1)
    return launch_tiled_u<kG, 1, 4>(store, mu, c, octant, cell, upstream, diagonal_offsets, sub_offsets,
                                    num_diagonals, num_sub, N, G, Dc, dpb, views, sync, max_blocks, timeout_ns, skip,
                                    stream);
  return set_error(CITRUS_EINVAL, "citrus_sweep_tiled: thread form %d (1 or 2)", form);
}

template <int kG, int kVB>
int launch_pencils(float* store, const float* mu, const float* c, Pencils p, int64_t views, unsigned* sync,
                   int64_t sync_words, int64_t max_blocks, uint64_t timeout_ns, int skip, cudaStream_t stream) {
  const int64_t view_blocks = cdiv(views, kVB), tiles = (int64_t)p.tiles_r * p.tiles_c;
  const int64_t total = view_blocks * p.sequences * tiles;
  CITRUS_REQUIRE(total < (1ll << 30), "citrus_sweep_pencils: too many tasks (%lld)", (long long)total);
  CITRUS_REQUIRE(sync_words >= kPencilFlag + total, "citrus_sweep_pencils: %lld sync words for %lld tasks",
                 (long long)sync_words, (long long)total);
  p.total = (uint32_t)total;
  const int lanes = (int)(p.dpb * p.G), threads = (int)(p.T * p.T) * lanes;
  const int smem = kPencilSlots * kVB * (int)((p.T + 1) * (p.T + 1)) * lanes * (int)sizeof(float4);
  CITRUS_REQUIRE(smem <= 226 * 1024, "citrus_sweep_pencils: %d bytes of shared memory for tiles of %d^2 pencils of %d "
                 "lanes", smem, (int)p.T, lanes);
  cudaError_t e = cudaFuncSetAttribute(pencil_kernel<kG, kVB>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  int per_sm = 0;
  if (e == cudaSuccess)
    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, pencil_kernel<kG, kVB>, threads, smem);
  if (e != cudaSuccess || per_sm < 1) return set_error(CITRUS_ECUDA, "citrus_sweep_pencils: occupancy query failed");
  int64_t blocks = (int64_t)per_sm * num_sms();
  if (max_blocks > 0 && max_blocks < blocks) blocks = max_blocks;
  if (blocks > total) blocks = total;
  if (skip >= blocks) skip = (int)blocks - 1;
  e = cudaMemsetAsync(sync, 0, (kPencilFlag + total) * sizeof(unsigned), stream);
  if (e != cudaSuccess) return set_error(CITRUS_ECUDA, "citrus_sweep_pencils: %s", cudaGetErrorString(e));
  const int64_t view_stride = 8 * (int64_t)p.Dc * p.R * p.C * p.S * p.G;  // float4 per view
  pencil_kernel<kG, kVB><<<(unsigned)blocks, threads, smem, stream>>>(reinterpret_cast<float4*>(store), mu, c, p,
                                                                      (int)views, view_stride, sync, timeout_ns, skip);
  note_launches();
  return launch_status("citrus_sweep_pencils");
}

constexpr int kDefaultUnroll = 1;

// the forms of the persistent launch's threads, chosen per grid by the autotuner
template <int kG>
int launch_persistent(float* store, const float* mu, const float* c, const int* octant, const int* cell,
                      const int* upstream, const int* offsets, int num_planes, int64_t N, int G, int64_t Dc,
                      int64_t views, unsigned* sync, int64_t max_blocks, uint64_t timeout_ns, int skip,
                      cudaStream_t stream, int unroll = kDefaultUnroll) {
  switch (unroll) {
    case 1:  // one view at a time, five blocks of 256 threads per SM
      return launch_persistent_u<kG, 1, 5>(store, mu, c, octant, cell, upstream, offsets, num_planes, N, G, Dc,
                                           views, sync, max_blocks, timeout_ns, skip, stream);
    case 3:  // one view at a time, registers capped for six blocks of 256 threads per SM
      return launch_persistent_u<kG, 1, 6>(store, mu, c, octant, cell, upstream, offsets, num_planes, N, G, Dc,
                                           views, sync, max_blocks, timeout_ns, skip, stream);
    case 5:  // one view at a time, four blocks per SM
      return launch_persistent_u<kG, 1, 4>(store, mu, c, octant, cell, upstream, offsets, num_planes, N, G, Dc,
                                           views, sync, max_blocks, timeout_ns, skip, stream);
    case 2:  // the loads of two views before their solves, three blocks per SM
      return launch_persistent_u<kG, 2, 3>(store, mu, c, octant, cell, upstream, offsets, num_planes, N, G, Dc,
                                           views, sync, max_blocks, timeout_ns, skip, stream);
    case 4:  // the loads of four views before their solves, two blocks per SM
      return launch_persistent_u<kG, 4, 2>(store, mu, c, octant, cell, upstream, offsets, num_planes, N, G, Dc,
                                           views, sync, max_blocks, timeout_ns, skip, stream);
    default:
      return set_error(CITRUS_EINVAL, "citrus_sweep_persistent: thread form %d (1, 2, 3, 4 or 5)", unroll);
  }
}

int check_sweep_args(const float* store, const float* mu, const float* c, const int* octant, const int* cell,
                     const int* upstream, int64_t num_planes, int64_t N, int64_t G, int64_t Dc, int64_t views) {
  CITRUS_REQUIRE(store && mu && c && octant && cell && upstream, "sweep: null pointer argument");
  CITRUS_REQUIRE(num_planes >= 1 && N >= 1 && G >= 1 && Dc >= 1 && views >= 1,
                 "sweep: sizes must be positive (planes %lld, cells %lld, groups %lld, dc %lld, views %lld)",
                 (long long)num_planes, (long long)N, (long long)G, (long long)Dc, (long long)views);
  CITRUS_REQUIRE(N < (1ll << 31) / 8, "sweep: %lld cells exceed the int32 entry tables", (long long)N);
  CITRUS_REQUIRE(views < (1ll << 31), "sweep: too many views (%lld)", (long long)views);
  CITRUS_REQUIRE(8 * N * Dc * G < (1ll << 31),
                 "sweep: one view's store of %lld float4 exceeds the 32-bit lane positions; sweep fewer directions "
                 "per chunk", (long long)(8 * N * Dc * G));
  CITRUS_REQUIRE(G <= 4096, "sweep: too many groups (%lld)", (long long)G);
  CITRUS_REQUIRE(((uintptr_t)store % 16) == 0, "sweep: store must be 16-byte aligned");
  return CITRUS_OK;
}

}  // namespace
}  // namespace citrus

using namespace citrus;

extern "C" int citrus_sweep_planes(float* store, const float* mu_cells, const float* c, const int32_t* octant,
                                   const int32_t* cell, const int32_t* upstream, const int64_t* plane_offsets_host,
                                   int64_t num_planes, int64_t num_cells, int64_t num_groups, int64_t dc,
                                   int64_t views, void* stream) {
  int status = check_sweep_args(store, mu_cells, c, octant, cell, upstream, num_planes, num_cells, num_groups, dc,
                                views);
  if (status) return status;
  CITRUS_REQUIRE(plane_offsets_host != nullptr, "citrus_sweep_planes: null plane offsets");
  const int G = (int)num_groups;
  cudaStream_t s = as_stream(stream);
  switch (G) {
    case 1: return launch_planes<1>(store, mu_cells, c, octant, cell, upstream, plane_offsets_host, num_planes,
                                    num_cells, G, dc, views, s);
    case 2: return launch_planes<2>(store, mu_cells, c, octant, cell, upstream, plane_offsets_host, num_planes,
                                    num_cells, G, dc, views, s);
    case 4: return launch_planes<4>(store, mu_cells, c, octant, cell, upstream, plane_offsets_host, num_planes,
                                    num_cells, G, dc, views, s);
    case 8: return launch_planes<8>(store, mu_cells, c, octant, cell, upstream, plane_offsets_host, num_planes,
                                    num_cells, G, dc, views, s);
    case 16: return launch_planes<16>(store, mu_cells, c, octant, cell, upstream, plane_offsets_host, num_planes,
                                      num_cells, G, dc, views, s);
    default: return launch_planes<0>(store, mu_cells, c, octant, cell, upstream, plane_offsets_host, num_planes,
                                     num_cells, G, dc, views, s);
  }
}

extern "C" int citrus_sweep_persistent_config(float* store, const float* mu_cells, const float* c,
                                              const int32_t* octant, const int32_t* cell, const int32_t* upstream,
                                              const int32_t* plane_offsets_dev, int64_t num_planes, int64_t num_cells,
                                              int64_t num_groups, int64_t dc, int64_t views, uint32_t* sync,
                                              int64_t max_blocks, int32_t thread_form, int64_t timeout_ns,
                                              int64_t skip_block, void* stream) {
  int status = check_sweep_args(store, mu_cells, c, octant, cell, upstream, num_planes, num_cells, num_groups, dc,
                                views);
  if (status) return status;
  CITRUS_REQUIRE(plane_offsets_dev != nullptr && sync != nullptr, "citrus_sweep_persistent: null offsets or sync");
  CITRUS_REQUIRE(num_planes < (1ll << 30), "citrus_sweep_persistent: too many planes");
  CITRUS_REQUIRE(timeout_ns > 0, "citrus_sweep_persistent: timeout_ns must be positive");
  const int G = (int)num_groups, P = (int)num_planes, skip = skip_block < 0 ? -1 : (int)skip_block;
  const uint64_t t = (uint64_t)timeout_ns;
  const int u = thread_form <= 0 ? kDefaultUnroll : thread_form;
  unsigned* sy = reinterpret_cast<unsigned*>(sync);
  cudaStream_t s = as_stream(stream);
  switch (G) {
    case 1: return launch_persistent<1>(store, mu_cells, c, octant, cell, upstream, plane_offsets_dev, P, num_cells,
                                        G, dc, views, sy, max_blocks, t, skip, s, u);
    case 2: return launch_persistent<2>(store, mu_cells, c, octant, cell, upstream, plane_offsets_dev, P, num_cells,
                                        G, dc, views, sy, max_blocks, t, skip, s, u);
    case 4: return launch_persistent<4>(store, mu_cells, c, octant, cell, upstream, plane_offsets_dev, P, num_cells,
                                        G, dc, views, sy, max_blocks, t, skip, s, u);
    case 8: return launch_persistent<8>(store, mu_cells, c, octant, cell, upstream, plane_offsets_dev, P, num_cells,
                                        G, dc, views, sy, max_blocks, t, skip, s, u);
    case 16: return launch_persistent<16>(store, mu_cells, c, octant, cell, upstream, plane_offsets_dev, P,
                                          num_cells, G, dc, views, sy, max_blocks, t, skip, s, u);
    default: return launch_persistent<0>(store, mu_cells, c, octant, cell, upstream, plane_offsets_dev, P, num_cells,
                                         G, dc, views, sy, max_blocks, t, skip, s, u);
  }
}

extern "C" int citrus_sweep_persistent(float* store, const float* mu_cells, const float* c, const int32_t* octant,
                                       const int32_t* cell, const int32_t* upstream, const int32_t* plane_offsets_dev,
                                       int64_t num_planes, int64_t num_cells, int64_t num_groups, int64_t dc,
                                       int64_t views, uint32_t* sync, int64_t max_blocks, int64_t timeout_ns,
                                       int64_t skip_block, void* stream) {
  return citrus_sweep_persistent_config(store, mu_cells, c, octant, cell, upstream, plane_offsets_dev, num_planes,
                                        num_cells, num_groups, dc, views, sync, max_blocks, 0, timeout_ns, skip_block,
                                        stream);
}

extern "C" int citrus_sweep_tiled(float* store, const float* mu_cells, const float* c, const int32_t* octant,
                                  const int32_t* cell, const int32_t* upstream, const int32_t* diagonal_offsets,
                                  const int32_t* sub_offsets, int64_t num_diagonals, int64_t num_sub,
                                  int64_t num_cells, int64_t num_groups, int64_t dc, int64_t views,
                                  int64_t dirs_per_block, uint32_t* sync, int64_t max_blocks, int64_t thread_form,
                                  int64_t timeout_ns, int64_t skip_block, void* stream) {
  int status = check_sweep_args(store, mu_cells, c, octant, cell, upstream, num_diagonals, num_cells, num_groups, dc,
                                views);
  if (status) return status;
  CITRUS_REQUIRE(diagonal_offsets && sub_offsets && sync, "citrus_sweep_tiled: null tables or sync words");
  CITRUS_REQUIRE(num_sub >= 1 && num_sub <= 4096 && num_diagonals <= (1 << 20),
                 "citrus_sweep_tiled: bad table sizes (diagonals %lld, sub-planes %lld)", (long long)num_diagonals,
                 (long long)num_sub);
  CITRUS_REQUIRE(dirs_per_block >= 1 && dirs_per_block <= dc, "citrus_sweep_tiled: directions per block %lld outside "
                 "[1, %lld]", (long long)dirs_per_block, (long long)dc);
  CITRUS_REQUIRE(timeout_ns > 0, "citrus_sweep_tiled: timeout_ns must be positive");
  const int G = (int)num_groups, ND = (int)num_diagonals, NS = (int)num_sub, form = (int)thread_form;
  const uint64_t t = (uint64_t)timeout_ns;
  const int skip = (int)skip_block;
  unsigned* sy = reinterpret_cast<unsigned*>(sync);
  cudaStream_t s = as_stream(stream);
#define CITRUS_TILED(KG)                                                                                           \
  launch_tiled<KG>(store, mu_cells, c, octant, cell, upstream, diagonal_offsets, sub_offsets, ND, NS, num_cells, G, \
                   dc, dirs_per_block, views, sy, max_blocks, t, skip, s, form)
  switch (G) {
    case 1: status = CITRUS_TILED(1); break;
    case 2: status = CITRUS_TILED(2); break;
    case 4: status = CITRUS_TILED(4); break;
    case 8: status = CITRUS_TILED(8); break;
    case 16: status = CITRUS_TILED(16); break;
    default: status = CITRUS_TILED(0); break;
  }
#undef CITRUS_TILED
  if (status) return status;
  return launch_status("citrus_sweep_tiled");
}

extern "C" int citrus_sweep_pencils(float* store, const float* mu_cells, const float* c, int64_t rows, int64_t cols,
                                    int64_t slices, int64_t num_groups, int64_t dc, int64_t views, int64_t tile,
                                    int64_t dirs_per_block, int64_t views_per_thread, uint32_t* sync,
                                    int64_t sync_words, int64_t max_blocks, int64_t timeout_ns, int64_t skip_block,
                                    void* stream) {
  CITRUS_REQUIRE(store && mu_cells && c && sync, "citrus_sweep_pencils: null pointer argument");
  CITRUS_REQUIRE(rows >= 1 && cols >= 1 && slices >= 1 && num_groups >= 1 && dc >= 1 && views >= 1,
                 "citrus_sweep_pencils: sizes must be positive");
  const int64_t cells_max = (1ll << 31) / 8;
  CITRUS_REQUIRE(rows < cells_max && cols < cells_max && slices < cells_max && rows * cols < cells_max &&
                     rows * cols * slices < cells_max,
                 "citrus_sweep_pencils: the grid's cells exceed the 32-bit positions");
  const int64_t cells = rows * cols * slices;
  CITRUS_REQUIRE(views < (1ll << 31), "citrus_sweep_pencils: too many views (%lld)", (long long)views);
  CITRUS_REQUIRE(num_groups <= 4096 && dc < (1ll << 28) && 8 * cells * num_groups < (1ll << 31) &&
                     8 * cells * num_groups * dc < (1ll << 31),
                 "citrus_sweep_pencils: one view's store exceeds the 32-bit lane positions; sweep fewer directions per "
                 "chunk");
  CITRUS_REQUIRE(((uintptr_t)store % 16) == 0, "citrus_sweep_pencils: store must be 16-byte aligned");
  CITRUS_REQUIRE(dirs_per_block >= 1 && dirs_per_block <= dc, "citrus_sweep_pencils: directions per task %lld outside "
                 "[1, %lld]", (long long)dirs_per_block, (long long)dc);
  CITRUS_REQUIRE(tile >= 1 && tile <= 16 && tile * tile * dirs_per_block * num_groups <= kPencilThreads,
                 "citrus_sweep_pencils: a tile of %lld^2 pencils of %lld lanes exceeds %d threads", (long long)tile,
                 (long long)(dirs_per_block * num_groups), kPencilThreads);
  CITRUS_REQUIRE(views_per_thread == 1 || views_per_thread == 2,
                 "citrus_sweep_pencils: views per thread %lld (1 or 2)", (long long)views_per_thread);
  CITRUS_REQUIRE(timeout_ns > 0, "citrus_sweep_pencils: timeout_ns must be positive");
  Pencils p;
  p.R = (uint32_t)rows, p.C = (uint32_t)cols, p.S = (uint32_t)slices, p.G = (uint32_t)num_groups, p.Dc = (uint32_t)dc;
  p.dpb = (uint32_t)dirs_per_block, p.T = (uint32_t)tile;
  p.tiles_r = (uint32_t)cdiv(rows, tile), p.tiles_c = (uint32_t)cdiv(cols, tile);
  p.dir_blocks = (uint32_t)cdiv(dc, dirs_per_block), p.sequences = 8 * p.dir_blocks, p.total = 0;
  const uint64_t t = (uint64_t)timeout_ns;
  const int skip = skip_block < 0 ? -1 : (int)skip_block;
  unsigned* sy = reinterpret_cast<unsigned*>(sync);
  cudaStream_t s = as_stream(stream);
#define CITRUS_PENCILS(KG)                                                                                        \
  (views_per_thread == 2                                                                                          \
       ? launch_pencils<KG, 2>(store, mu_cells, c, p, views, sy, sync_words, max_blocks, t, skip, s)              \
       : launch_pencils<KG, 1>(store, mu_cells, c, p, views, sy, sync_words, max_blocks, t, skip, s))
  // the number of groups known to the compiler for the two commonest: us at 64^3 cells and 120 directions, with it / without,
  // one group 630 / 635, 8 groups 2242 / 2263 (32^3: 366 / 374); 16 groups have nothing more to gain
  switch (num_groups) {
    case 1: return CITRUS_PENCILS(1);
    case 8: return CITRUS_PENCILS(8);
    default: return CITRUS_PENCILS(0);
  }
#undef CITRUS_PENCILS
}

// ---- allocation-free persistent sweep ----------------------------------------------------------------------------
//
// The same persistent launch with its scratch in a file-scope device array instead of caller-provided device memory:
// the barrier words at [0, 4) and the int32 plane offsets from word 64 (byte 256) on. The call makes no device
// allocation of any kind; it only clears the barrier words and copies the offsets into the array, both on the stream.
namespace citrus {
namespace {

constexpr int64_t kStaticMaxPlanes = 8191;  // R + C + S - 2 <= 8191: every grid up to 2730^3 cells
constexpr int kStaticOffsetsWord = 64;
constexpr int kStaticWords = kStaticOffsetsWord + (int)kStaticMaxPlanes + 1;  // 8256 words, 33 KB per device
constexpr int kStaticMaxDevices = 64;

static __device__ __align__(256) uint32_t g_static_sweep_scratch[kStaticWords];

std::mutex g_static_mutex;
uint32_t* g_static_address[kStaticMaxDevices] = {};

// Device address of the scratch array on the current device, looked up once per device.
int static_scratch(uint32_t** out) {
  int dev = -1;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return set_error(CITRUS_ECUDA, "citrus_sweep_persistent_static: %s", cudaGetErrorString(e));
  if (dev < 0 || dev >= kStaticMaxDevices)
    return set_error(CITRUS_EINVAL, "citrus_sweep_persistent_static: device %d beyond the %d supported", dev,
                     kStaticMaxDevices);
  std::lock_guard<std::mutex> lock(g_static_mutex);
  if (g_static_address[dev] == nullptr) {
    void* p = nullptr;
    e = cudaGetSymbolAddress(&p, g_static_sweep_scratch);
    if (e != cudaSuccess || p == nullptr)
      return set_error(CITRUS_ECUDA, "citrus_sweep_persistent_static: scratch address on device %d: %s", dev,
                       cudaGetErrorString(e));
    g_static_address[dev] = static_cast<uint32_t*>(p);
  }
  *out = g_static_address[dev];
  return CITRUS_OK;
}

}  // namespace
}  // namespace citrus

extern "C" int citrus_sweep_persistent_static(float* store, const float* mu_cells, const float* c,
                                              const int32_t* octant, const int32_t* cell, const int32_t* upstream,
                                              const int32_t* plane_offsets_host, int64_t num_planes,
                                              int64_t num_cells, int64_t num_groups, int64_t dc, int64_t views,
                                              uint32_t* timeout_word, int64_t timeout_ns, void* stream) {
  int status = check_sweep_args(store, mu_cells, c, octant, cell, upstream, num_planes, num_cells, num_groups, dc,
                                views);
  if (status) return status;
  CITRUS_REQUIRE(plane_offsets_host != nullptr, "citrus_sweep_persistent_static: null plane offsets");
  CITRUS_REQUIRE(num_planes <= kStaticMaxPlanes,
                 "citrus_sweep_persistent_static: %lld planes exceed the static scratch (at most %lld planes, "
                 "R + C + S - 2 <= %lld); use citrus_sweep_persistent with caller scratch",
                 (long long)num_planes, (long long)kStaticMaxPlanes, (long long)kStaticMaxPlanes);
  CITRUS_REQUIRE(timeout_ns > 0, "citrus_sweep_persistent_static: timeout_ns must be positive");
  uint32_t* scratch = nullptr;
  status = static_scratch(&scratch);
  if (status) return status;
  cudaStream_t s = as_stream(stream);
  int32_t* offsets = reinterpret_cast<int32_t*>(scratch + kStaticOffsetsWord);
  cudaError_t e = cudaMemcpyAsync(offsets, plane_offsets_host, (size_t)(num_planes + 1) * sizeof(int32_t),
                                  cudaMemcpyHostToDevice, s);
  if (e != cudaSuccess)
    return set_error(CITRUS_ECUDA, "citrus_sweep_persistent_static: offsets copy: %s", cudaGetErrorString(e));
  // the barrier words are cleared by the launch below (cudaMemsetAsync on the stream)
  const int G = (int)num_groups, P = (int)num_planes;
  const uint64_t t = (uint64_t)timeout_ns;
  unsigned* sy = reinterpret_cast<unsigned*>(scratch);
  switch (G) {
    case 1: status = launch_persistent<1>(store, mu_cells, c, octant, cell, upstream, offsets, P, num_cells, G, dc,
                                          views, sy, 0, t, -1, s); break;
    case 2: status = launch_persistent<2>(store, mu_cells, c, octant, cell, upstream, offsets, P, num_cells, G, dc,
                                          views, sy, 0, t, -1, s); break;
    case 4: status = launch_persistent<4>(store, mu_cells, c, octant, cell, upstream, offsets, P, num_cells, G, dc,
                                          views, sy, 0, t, -1, s); break;
    case 8: status = launch_persistent<8>(store, mu_cells, c, octant, cell, upstream, offsets, P, num_cells, G, dc,
                                          views, sy, 0, t, -1, s); break;
    case 16: status = launch_persistent<16>(store, mu_cells, c, octant, cell, upstream, offsets, P, num_cells, G, dc,
                                            views, sy, 0, t, -1, s); break;
    default: status = launch_persistent<0>(store, mu_cells, c, octant, cell, upstream, offsets, P, num_cells, G, dc,
                                           views, sy, 0, t, -1, s); break;
  }
  if (status || timeout_word == nullptr) return status;
  e = cudaMemcpyAsync(timeout_word, scratch + 2, sizeof(uint32_t), cudaMemcpyDefault, s);
  if (e != cudaSuccess)
    return set_error(CITRUS_ECUDA, "citrus_sweep_persistent_static: timeout word copy: %s", cudaGetErrorString(e));
  return CITRUS_OK;
}

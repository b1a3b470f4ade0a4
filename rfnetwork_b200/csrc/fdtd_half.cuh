// Half-step kernels for sm_100a: one launch advances E of every cell, the next
// one H, in place in time buffer 0.
//
//   thread    one cell. No halo is recomputed, nothing is shared between
//             threads, so every warp runs on its own and 40 of them hide each
//             other's latency; the price is a second pass over the fields, which
//             stays in L2 for grids of a few million cells
//   static    a launch may start while the last blocks of the one before it
//             still run (programmatic dependent launch): the material index, the
//             table row, a split cell's pair offsets and the neighbours' rows
//             are read before the wait, the fields after it
//
// Measured on a B200, per step, against the streaming kernels' best shape:
// 96x96x64 cells with 10-cell layers 33.5 -> 16.1 us, 120x100x64 with 8-cell
// layers 32.1 -> 19.0 us, 128x128x96 with 10-cell layers 61.4 -> 35.4 us,
// 160x130x110 with 8-cell layers 74.6 -> 55.3 us; 150x130x90 without layers 26.8
// (streaming) against 31.2 us, 256x256x128 with 8-cell layers 169 against 245 us,
// so the autotuner picks by measurement. The streaming kernels lose where most
// tiles hold layer cells (their warps run both the split and the unsplit path
// behind one barrier per plane with 20 warps per SM); these lose where the
// second pass no longer comes from L2. Bound by latency and issue (173 and 184
// instructions per cell). Two or four cells of a row per thread (16-byte loads)
// need 80 to 128 registers and were slower up to 2.3 M cells (39 us on
// 128x128x96); a march along z with prefetch was slower everywhere.
//
// Same per-cell expressions as fdtd_step_kernel through the same rounding-fixed
// helpers, so all step kernels give the same bits.
#pragma once

#include "fdtd_adjoint.cuh"
#include "fdtd_kernels.cuh"

#include <climits>

namespace rfn {

__device__ __forceinline__ void pdl_launch_dependents() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

// The cells of a launch. A block takes, in one plane, `rows` rows of `seg`
// columns, or one piece of a long row.
//   blocks    (simulation, x0 | rows << 16, y0, z | seg << 16) per block: whole
//             grids of several simulations
//   boxes     else, when given: the cells within lo cells below and hi cells
//             above each simulation's box (x0 x1 y0 y1 z0 z1 per simulation);
//             blockIdx = (piece of a row, group of rows, simulation * planes + plane)
//   neither   one simulation's whole grid, blockIdx = (piece, group of rows, plane)
struct HalfLaunch {
  const int4* blocks;
  const int* boxes;
  int seg, rows, planes;
  int lo, hi;
  int n;                 // time step
  int deep;              // reverse step: planes per block
};

struct HalfPlace {
  int sim, x, y, z;
  bool region;
};

// This thread's cell (its column may lie outside the grid).
__device__ __forceinline__ HalfPlace half_place(const HalfLaunch& L) {
  HalfPlace p;
  int rows = L.rows, seg = L.seg;
  p.region = false;
  if (L.blocks) {
    const int4 b = __ldg(L.blocks + blockIdx.x);
    p.sim = b.x;
    p.x = b.y & 0xffff;
    rows = int(unsigned(b.y) >> 16);
    p.y = b.z;
    p.z = b.w & 0xffff;
    seg = int(unsigned(b.w) >> 16);
  } else {
    p.sim = L.boxes ? int(blockIdx.z) / L.planes : 0;
    p.x = blockIdx.x * seg;
    p.y = blockIdx.y * rows;
    p.z = L.boxes ? int(blockIdx.z) - p.sim * L.planes : int(blockIdx.z);
    p.region = L.boxes != nullptr;
  }
  // row of this thread: tid / seg by a reciprocal, exact for these small
  // integers (tid + 1/2 is at least 1/2 away from every multiple of seg)
  const int tid = threadIdx.x;
  const int q = rows > 1 ? int((float(tid) + 0.5f) * __fdividef(1.0f, float(seg))) : 0;
  p.x += tid - q * seg;
  p.y += q;
  if (q >= rows || tid - q * seg >= seg) p.z = INT_MAX;
  return p;
}

// Whether place p is a cell of the launch in a grid of nx x ny x nz; a region's
// place is moved to the grid.
__device__ __forceinline__ bool half_inside(const HalfLaunch& L, HalfPlace& p, int nx, int ny, int nz) {
  if (p.z == INT_MAX) return false;
  if (p.region) {
    const int* b = L.boxes + 6 * p.sim;
    p.x += max(__ldg(b) - L.lo, 0);
    p.y += max(__ldg(b + 2) - L.lo, 0);
    p.z += max(__ldg(b + 4) - L.lo, 0);
    nx = min(nx, __ldg(b + 1) + L.hi);
    ny = min(ny, __ldg(b + 3) + L.hi);
    nz = min(nz, __ldg(b + 5) + L.hi);
  }
  return p.x < nx && p.y < ny && p.z < nz;
}

// ------------------------------------------------------------------- forward

// Soft sources of one component m (0..5) of a probe cell (solver.cu:459-488,
// 515-541): s1 += v; s2 += v for every source probe on it (a sourced component
// is always stored as its split pair).
__device__ __forceinline__ void half_inject(const SimDev& S, int first, int np, int n, int m, float2& p) {
  for (int e = 0; e < np; ++e) {
    const int2 pe = __ldg(S.cell_probes + first + e);
    if (pe.y == m && __ldg(S.is_src + pe.x)) {
      const float v = __ldg(S.src + (size_t)pe.x * S.nt + n);
      p.x = __fadd_rn(p.x, v);
      p.y = __fadd_rn(p.y, v);
    }
  }
}

// Records this cell's probes of the E (first field 0) or H (3) group (solver.cu:467, 521).
__device__ __forceinline__ void half_record(const SimDev& S, int first, int np, int n, int field0, float a, float b,
                                            float c) {
  for (int e = 0; e < np; ++e) {
    const int2 pe = __ldg(S.cell_probes + first + e);
    const int f = pe.y - field0;
    if (f >= 0 && f < 3) S.rec[(size_t)pe.x * S.nt + n] = f == 0 ? a : f == 1 ? b : c;
  }
}

// The source amplitudes of a probe cell into L1 (no step writes them).
__device__ __forceinline__ void half_prefetch_sources(const SimDev& S, int first, int np, int n) {
  for (int e = 0; e < np; ++e) {
    const int2 pe = __ldg(S.cell_probes + first + e);
    if (__ldg(S.is_src + pe.x)) prefetch_l1(S.src + (size_t)pe.x * S.nt + n);
  }
}

// E of cell (x, y, z). hist: where the nine history values of a gradient-box
// cell go, `nb` apart (null: no box cell).
__device__ __forceinline__ void half_e(const SimDev& S, int x, int y, int z, int n, float* hist, int64_t nb) {
  const int plane = S.plane, pitch = S.pitch, i = z * plane + y * pitch + x;
  const float4* const row = S.rows + 8 * int(__ldg(S.mat + i));
  const float2 w = __ldg(reinterpret_cast<const float2*>(row + 7) + 1);  // flags, word 31
  const uint32_t flags = __float_as_uint(w.x);
  const int first = __float_as_int(w.y), np = int(flags >> 16);
  const float4 ra = __ldg(row), rb = __ldg(row + 1), rd = __ldg(row + 2);
  int cs = 0;
  int64_t so = 0;
  if (flags & kESplit) so = split_off(S.sp, split_store(S.sp, S.nx, S.ny, S.nz, x, y, z), x, y, z, first, cs);
  if (np) half_prefetch_sources(S, first, np, n);
  const bool xn = x + 1 < S.nx, yn = y + 1 < S.ny, zn = z + 1 < S.nz;
  const float* const Hx = S.H[0][0] + i;
  const float* const Hy = S.H[0][1] + i;
  const float* const Hz = S.H[0][2] + i;
  pdl_wait();
  const float hx = *Hx, hy = *Hy, hz = *Hz;
  const float hx_z = zn ? Hx[plane] : 0.f, hy_z = zn ? Hy[plane] : 0.f;
  const float hx_y = yn ? Hx[pitch] : 0.f, hz_y = yn ? Hz[pitch] : 0.f;
  const float hy_x = xn ? Hy[1] : 0.f, hz_x = xn ? Hz[1] : 0.f;
  float e[3];
  float2 p[3];
#pragma unroll
  for (int m = 0; m < 3; ++m) {
    e[m] = S.E[0][m][i];
    p[m] = (flags & (kCompSplit0 << m)) ? S.sp.base[0][so + m * int64_t(cs)] : make_float2(0.f, 0.f);
  }
  // ex: dhz_y, dhy_z; ey: dhx_z, dhz_x; ez: dhy_x, dhx_y
  const float d1[3] = {hz_y - hz, hx_z - hx, hy_x - hy}, d2[3] = {hy_z - hy, hz_x - hz, hx_y - hx};
  if (hist) {
#pragma unroll
    for (int m = 0; m < 3; ++m) {
      hist[m * nb] = e[m];
      hist[(3 + 2 * m) * nb] = d1[m];
      hist[(4 + 2 * m) * nb] = d2[m];
    }
  }
  float v[3];
#pragma unroll
  for (int m = 0; m < 3; ++m) {
    const float4 k = m == 0 ? ra : m == 1 ? rb : rd;
    v[m] = upd_e(k.x, e[m], k.y, d1[m], k.w, d2[m]);
    if (flags & (kCompSplit0 << m)) {
      p[m].x = upd_e_split(k.x, p[m].x, k.y, d1[m]);
      p[m].y = upd_e_split(k.z, p[m].y, k.w, d2[m]);
      if (np) half_inject(S, first, np, n, m, p[m]);
      v[m] = __fadd_rn(p[m].x, p[m].y);
      S.sp.base[0][so + m * int64_t(cs)] = p[m];
    }
    S.E[0][m][i] = v[m];
  }
  if (np) half_record(S, first, np, n, 0, v[0], v[1], v[2]);
}

// H of cell (x, y, z).
__device__ __forceinline__ void half_h(const SimDev& S, int x, int y, int z, int n) {
  const int plane = S.plane, pitch = S.pitch, i = z * plane + y * pitch + x;
  const float4* const row = S.rows + 8 * int(__ldg(S.mat + i));
  const float4 rp = __ldg(row + 3), rq = __ldg(row + 4), ru = __ldg(row + 5), rv = __ldg(row + 6), r7 = __ldg(row + 7);
  const uint32_t flags = __float_as_uint(r7.z);
  const int first = __float_as_int(r7.w), np = int(flags >> 16);
  int cs = 0;
  int64_t so = 0;
  if (flags & kHSplit) so = split_off(S.sp, split_store(S.sp, S.nx, S.ny, S.nz, x, y, z), x, y, z, first, cs);
  if (np) half_prefetch_sources(S, first, np, n);
  const float* const Ex = S.E[0][0] + i;
  const float* const Ey = S.E[0][1] + i;
  const float* const Ez = S.E[0][2] + i;
  pdl_wait();
  const float ex = *Ex, ey = *Ey, ez = *Ez;
  const float ex_z = z > 0 ? Ex[-plane] : 0.f, ey_z = z > 0 ? Ey[-plane] : 0.f;
  const float ex_y = y > 0 ? Ex[-pitch] : 0.f, ez_y = y > 0 ? Ez[-pitch] : 0.f;
  const float ey_x = x > 0 ? Ey[-1] : 0.f, ez_x = x > 0 ? Ez[-1] : 0.f;
  float h[3];
  float2 p[3];
#pragma unroll
  for (int m = 0; m < 3; ++m) {
    h[m] = S.H[0][m][i];
    p[m] = (flags & (kCompSplit0 << (3 + m))) ? S.sp.base[0][so + (3 + m) * int64_t(cs)] : make_float2(0.f, 0.f);
  }
  // slots 12..29: (Da, Db1, Db2) of hx_y, hx_z, hy_z, hy_x, hz_x, hz_y
  const float g1[3] = {h_term(rp.z, ez, rp.y, ez_y), h_term(ru.x, ex, rq.w, ex_z), h_term(rv.z, ey, rv.y, ey_x)};
  const float g2[3] = {h_term(rq.y, ey, rq.x, ey_z), h_term(ru.w, ez, ru.z, ez_x), h_term(r7.y, ex, r7.x, ex_y)};
  const float da1[3] = {rp.x, rq.z, rv.x}, da2[3] = {rp.w, ru.y, rv.w};
  float v[3];
#pragma unroll
  for (int m = 0; m < 3; ++m) {
    v[m] = upd_h(da1[m], h[m], g1[m], g2[m]);
    if (flags & (kCompSplit0 << (3 + m))) {
      p[m].x = upd_h_split(da1[m], p[m].x, g1[m]);
      p[m].y = upd_h_split(da2[m], p[m].y, g2[m]);
      if (np) half_inject(S, first, np, n, 3 + m, p[m]);
      v[m] = __fadd_rn(p[m].x, p[m].y);
      S.sp.base[0][so + (3 + m) * int64_t(cs)] = p[m];
    }
    S.H[0][m][i] = v[m];
  }
  if (np) half_record(S, first, np, n, 3, v[0], v[1], v[2]);
}

constexpr int kHalfThreads = 256;  // most threads of a block
constexpr int kHalfBlocks = 5;     // resident blocks per SM the registers are sized for (48)

// One half step: E (H_SIDE false) or H. ONE: a single simulation, whose
// descriptor is a kernel parameter (constant memory). CAP: the E side also
// writes the history of step n of the gradient boxes, caps[simulation], at slot
// n - n0.
template <bool H_SIDE, bool ONE, bool CAP>
__global__ void __launch_bounds__(kHalfThreads, kHalfBlocks)
half_step_kernel(const __grid_constant__ SimDev one, const __grid_constant__ HalfLaunch L,
                 const SimDev* __restrict__ sims, const CapSim* __restrict__ caps, int n0) {
  pdl_launch_dependents();
  HalfPlace p = half_place(L);
  const SimDev& S = ONE ? one : sims[p.sim];
  if (!half_inside(L, p, S.nx, S.ny, S.nz)) return;
  if constexpr (H_SIDE) {
    half_h(S, p.x, p.y, p.z, L.n);
  } else {
    float* hist = nullptr;
    int64_t nb = 0;
    if (CAP) {
      const CapSim& C = caps[p.sim];
      if (C.hist && p.x >= C.bx0 && p.x < C.bx1 && p.y >= C.by0 && p.y < C.by1 && p.z >= C.bz0 && p.z < C.bz1) {
        nb = C.nb;
        hist = C.hist + int64_t(L.n - n0) * 9 * nb +
               box_cell(p.x - C.bx0, p.y - C.by0, p.z - C.bz0, C.bx1 - C.bx0, C.by1 - C.by0);
      }
    }
    half_e(S, p.x, p.y, p.z, L.n, hist, nb);
  }
}

}  // namespace rfn

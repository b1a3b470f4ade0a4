// The reverse time step (fdtd_adjoint.cuh) as two launches, in place in buffer 0
// of the adjoint state:
//   E side    mu = lamE + (own Db2 lamH) - (Db1 lamH of the +1 neighbours) for
//             every cell, with the gradient of the box cells. mu takes lamE's
//             place in the state: the next E side forms lamE = Ca mu (and adds
//             the records' adjoints) before it uses it, so the H side can read mu
//   H side    lamH' = Da lamH + (Cb mu of the -1 neighbours - own Cb mu), with
//             the adjoints of the records of the step before
// One thread per column of a few cells along z, no halo, no barrier; what no step
// writes (the index, the rows of the first cell and of its neighbours) is read
// before the wait for the launch before. A neighbour's coefficient is this cell's
// own where both use one table row. With one cell per thread the row quads, eight
// per cell and up to nine more words of other rows, kept the L1 pipe 70 % busy;
// along z they change only at the model's and the z layers' boundaries, so a
// thread keeps them while the four ids stay the same. 128x128x96 cells with
// 10-cell layers, per step: one launch 89 us, halves of one cell per thread 71,
// of four 65; small grids need every thread. 80 registers and 24 warps
// per SM instead of 64 and 32 lose 5 %; halves kept per component instead of per
// cell move a third less in the layers and were slower (more branches per
// access). The arithmetic and its roundings are those of adj_e_part and
// adj_h_part, so all reverse steps give the same bits.
#pragma once

#include "fdtd_adjoint.cuh"
#include "fdtd_half.cuh"

namespace rfn {

// Adds the records' adjoints of step `step` to the E (first field 0) or H (3)
// adjoints l of a probe cell: totals in l[0..2], or six halves.
__device__ __forceinline__ void adj_add_records(const AdjSim& A, const float4& r7, int step, int field0, bool halves,
                                                float (&l)[6]) {
  const int np = int(__float_as_uint(r7.z) >> 16), first = __float_as_int(r7.w);
  for (int e = 0; e < np; ++e) {
    const int2 pe = __ldg(A.cell_probes + first + e);
    const int c = pe.y - field0;
    if (c < 0 || c > 2) continue;
    const float rv = __ldg(A.radj + size_t(pe.x) * A.nt + step);
#pragma unroll
    for (int k = 0; k < 6; ++k)
      if (halves ? k / 2 == c : k == c) l[k] = __fadd_rn(l[k], rv);
  }
}

// Whether the cell with table row `row` keeps halves of the E or H group.
__device__ __forceinline__ bool adj_halves(const float4* row, uint32_t group) {
  return (__float_as_uint(__ldg(&row[7].z)) & group) != 0;
}

// E side of the cells (x, y, z0 .. z1-1).
__device__ __forceinline__ void adj_half_e(const AdjSim& A, int x, int y, int z0, int z1, int n, int hist_n0) {
  const int plane = A.plane, pitch = A.pitch;
  const int64_t N = A.N;
  const float4* const rows = A.rows;
  const bool xn = x + 1 < A.nx, yn = y + 1 < A.ny;
  int i = z0 * plane + y * pitch + x;
  // ids of the cell and its neighbours whose coefficients are held
  int id = -1, ix = -1, iy = -1, iz = -1, id_up = __ldg(A.mat + i);
  float ca[6], db[6], bx_hy, bx_hz, by_hx, by_hz, bz_hx, bz_hy;
  float4 r7;
  bool sx, sy, sz;
#pragma unroll 1
  for (int z = z0; z < z1; ++z, i += plane) {
    const bool zn = z + 1 < A.nz;
    const int jd = id_up, jx = xn ? int(__ldg(A.mat + i + 1)) : jd, jy = yn ? int(__ldg(A.mat + i + pitch)) : jd;
    const int jz = zn ? int(__ldg(A.mat + i + plane)) : jd;
    id_up = jz;
    if (jd != id || jx != ix || jy != iy || jz != iz) {
      id = jd; ix = jx; iy = jy; iz = jz;
      const float4* const row = rows + 8 * id;
      const float4 ra = __ldg(row), rb = __ldg(row + 1), rd = __ldg(row + 2);
      const float4 p = __ldg(row + 3), q = __ldg(row + 4), u = __ldg(row + 5), v = __ldg(row + 6);
      r7 = __ldg(row + 7);
      ca[0] = ra.x; ca[1] = ra.z; ca[2] = rb.x; ca[3] = rb.z; ca[4] = rd.x; ca[5] = rd.z;
      db[0] = p.z; db[1] = q.y; db[2] = u.x; db[3] = u.w; db[4] = v.z; db[5] = r7.y;
      // Db1 of the neighbours' terms and whether they keep halves of H
      bx_hy = u.z; bx_hz = v.y; by_hx = p.y; by_hz = r7.x; bz_hx = q.x; bz_hy = q.w;
      sx = sy = sz = __float_as_uint(r7.z) & kHSplit;
      if (ix != id) {
        const float4* const r = rows + 8 * ix;
        bx_hy = __ldg(&r[5].z); bx_hz = __ldg(&r[6].y); sx = adj_halves(r, kHSplit);
      }
      if (iy != id) {
        const float4* const r = rows + 8 * iy;
        by_hx = __ldg(&r[3].y); by_hz = __ldg(&r[7].x); sy = adj_halves(r, kHSplit);
      }
      if (iz != id) {
        const float4* const r = rows + 8 * iz;
        bz_hx = __ldg(&r[4].x); bz_hy = __ldg(&r[4].w); sz = adj_halves(r, kHSplit);
      }
    }
    const uint32_t fl = __float_as_uint(r7.z);
    const bool hs = fl & kHSplit, es = fl & kESplit;
    float* const E = A.lam + i;              // totals (mu of the unsplit cells)
    const float* const H = A.lam + 3 * N + i;
    float* const Es = A.lams + i;            // halves
    const float* const Hs = A.lams + 6 * N + i;
    pdl_wait();
    float h[6], l[6];
    if (hs) {
#pragma unroll
      for (int k = 0; k < 6; ++k) h[k] = Hs[k * N];
    } else {
#pragma unroll
      for (int c = 0; c < 3; ++c) h[2 * c] = h[2 * c + 1] = H[c * N];
    }
    // hy, hz of the cell at x + 1; hx, hz at y + 1; hx, hy at z + 1
    const float hx_hy = !xn ? 0.f : sx ? Hs[3 * N + 1] : H[N + 1], hx_hz = !xn ? 0.f : sx ? Hs[4 * N + 1] : H[2 * N + 1];
    const float hy_hx = !yn ? 0.f : sy ? Hs[pitch] : H[pitch], hy_hz = !yn ? 0.f : sy ? Hs[5 * N + pitch] : H[2 * N + pitch];
    const float hz_hx = !zn ? 0.f : sz ? Hs[N + plane] : H[plane], hz_hy = !zn ? 0.f : sz ? Hs[2 * N + plane] : H[N + plane];
    if (es) {
#pragma unroll
      for (int k = 0; k < 6; ++k) l[k] = Es[k * N];
    } else {
#pragma unroll
      for (int c = 0; c < 3; ++c) l[c] = E[c * N];
    }
    // lamE of step n: Ca mu, and the adjoints of its records
    if (es) {
#pragma unroll
      for (int k = 0; k < 6; ++k) l[k] = __fmul_rn(ca[k], l[k]);
    } else {
#pragma unroll
      for (int c = 0; c < 3; ++c) l[c] = __fmul_rn(ca[2 * c], l[c]);
    }
    if (fl >> 16) adj_add_records(A, r7, n, 0, es, l);
    const float qx_hy = __fmul_rn(bx_hy, hx_hy), qx_hz = __fmul_rn(bx_hz, hx_hz);
    const float qy_hx = __fmul_rn(by_hx, hy_hx), qy_hz = __fmul_rn(by_hz, hy_hz);
    const float qz_hx = __fmul_rn(bz_hx, hz_hx), qz_hy = __fmul_rn(bz_hy, hz_hy);
    const float a[3] = {__fadd_rn(__fmaf_rn(db[2], h[2], -qz_hy), __fmaf_rn(db[5], h[5], -qy_hz)),
                        __fadd_rn(__fmaf_rn(db[1], h[1], -qz_hx), __fmaf_rn(db[4], h[4], -qx_hz)),
                        __fadd_rn(__fmaf_rn(db[0], h[0], -qy_hx), __fmaf_rn(db[3], h[3], -qx_hy))};
    if (es) {  // (a gradient box holds no split cells)
#pragma unroll
      for (int k = 0; k < 6; ++k) Es[k * N] = __fadd_rn(l[k], a[k / 2]);
      continue;
    }
    float mu[6];
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      mu[2 * c] = mu[2 * c + 1] = __fadd_rn(l[c], a[c]);
      E[c * N] = mu[2 * c];
    }
    if (A.hist && x >= A.bx0 && x < A.bx1 && y >= A.by0 && y < A.by1 && z >= A.bz0 && z < A.bz1) {
      const int64_t bi = box_cell(x - A.bx0, y - A.by0, z - A.bz0, A.bx1 - A.bx0, A.by1 - A.by0);
      adj_grad_cell(A.grad, A.nb, bi, A.hist + int64_t(n - hist_n0) * 9 * A.nb, mu);
    }
  }
}

// H side of the cells (x, y, z0 .. z1-1).
__device__ __forceinline__ void adj_half_h(const AdjSim& A, int x, int y, int z0, int z1, int n) {
  const int plane = A.plane, pitch = A.pitch;
  const int64_t N = A.N;
  const float4* const rows = A.rows;
  int i = z0 * plane + y * pitch + x;
  int id = -1, ix = -1, iy = -1, iz = -1, id_down = z0 > 0 ? int(__ldg(A.mat + i - plane)) : -1;
  float4 ra, rb, rd, p, q, u, v, r7;
  float c0, c1, c2, c3, c4, c5;
  bool sx, sy, sz;
#pragma unroll 1
  for (int z = z0; z < z1; ++z, i += plane) {
    const int jd = __ldg(A.mat + i), jx = x > 0 ? int(__ldg(A.mat + i - 1)) : jd,
              jy = y > 0 ? int(__ldg(A.mat + i - pitch)) : jd, jz = z > 0 ? id_down : jd;
    id_down = jd;
    if (jd != id || jx != ix || jy != iy || jz != iz) {
      id = jd; ix = jx; iy = jy; iz = jz;
      const float4* const row = rows + 8 * id;
      ra = __ldg(row); rb = __ldg(row + 1); rd = __ldg(row + 2);
      p = __ldg(row + 3); q = __ldg(row + 4); u = __ldg(row + 5); v = __ldg(row + 6); r7 = __ldg(row + 7);
      // Cb of the neighbours' terms and whether they keep halves of E
      c3 = rb.w; c4 = rd.y; c0 = ra.y; c5 = rd.w; c1 = ra.w; c2 = rb.y;
      sx = sy = sz = __float_as_uint(r7.z) & kESplit;
      if (ix != id) {
        const float4* const r = rows + 8 * ix;
        c3 = __ldg(&r[1].w); c4 = __ldg(&r[2].y); sx = adj_halves(r, kESplit);
      }
      if (iy != id) {
        const float4* const r = rows + 8 * iy;
        c0 = __ldg(&r[0].y); c5 = __ldg(&r[2].w); sy = adj_halves(r, kESplit);
      }
      if (iz != id) {
        const float4* const r = rows + 8 * iz;
        c1 = __ldg(&r[0].w); c2 = __ldg(&r[1].y); sz = adj_halves(r, kESplit);
      }
    }
    const uint32_t fl = __float_as_uint(r7.z);
    const float* const E = A.lam + i;
    float* const H = A.lam + 3 * N + i;
    const float* const Es = A.lams + i;
    float* const Hs = A.lams + 6 * N + i;
    pdl_wait();
    float h[6], m[6];
    const bool hs = fl & kHSplit, es = fl & kESplit;
    if (hs) {
#pragma unroll
      for (int k = 0; k < 6; ++k) h[k] = Hs[k * N];
    } else {
#pragma unroll
      for (int c = 0; c < 3; ++c) h[2 * c] = h[2 * c + 1] = H[c * N];
    }
    if (es) {
#pragma unroll
      for (int k = 0; k < 6; ++k) m[k] = Es[k * N];
    } else {
#pragma unroll
      for (int c = 0; c < 3; ++c) m[2 * c] = m[2 * c + 1] = E[c * N];
    }
    // mu of the -1 neighbours: x: dB_y (3), dA_z (4); y: dA_x (0), dB_z (5); z: dB_x (1), dA_y (2)
    const float m3 = x == 0 ? 0.f : sx ? Es[3 * N - 1] : E[N - 1], m4 = x == 0 ? 0.f : sx ? Es[4 * N - 1] : E[2 * N - 1];
    const float m0 = y == 0 ? 0.f : sy ? Es[-pitch] : E[-pitch], m5 = y == 0 ? 0.f : sy ? Es[5 * N - pitch] : E[2 * N - pitch];
    const float m1 = z == 0 ? 0.f : sz ? Es[N - plane] : E[-plane], m2 = z == 0 ? 0.f : sz ? Es[2 * N - plane] : E[N - plane];
    const float cb[6] = {ra.y, ra.w, rb.y, rb.w, rd.y, rd.w};
    float ad[6], lh[6] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
#pragma unroll
    for (int k = 0; k < 6; ++k) ad[k] = __fmul_rn(cb[k], m[k]);
    adj_h_part(p, q, u, v, fl, h, ad, __fmul_rn(c0, m0), __fmul_rn(c5, m5), __fmul_rn(c3, m3), __fmul_rn(c4, m4),
               __fmul_rn(c1, m1), __fmul_rn(c2, m2), lh);
    if ((fl >> 16) && n >= 1) adj_add_records(A, r7, n - 1, 3, hs, lh);
    if (hs) {
#pragma unroll
      for (int k = 0; k < 6; ++k) Hs[k * N] = lh[k];
    } else {
#pragma unroll
      for (int c = 0; c < 3; ++c) H[c * N] = lh[c];
    }
  }
}

constexpr int kAdjHalfBlocks = 4;  // resident blocks per SM the registers are sized for (64)

// One half of reverse step n of every cell. ONE: a single simulation, whose
// descriptor is a kernel parameter.
template <bool H_SIDE, bool ONE>
__global__ void __launch_bounds__(kHalfThreads, kAdjHalfBlocks)
adj_half_kernel(const __grid_constant__ AdjSim one, const __grid_constant__ HalfLaunch L,
                const AdjSim* __restrict__ sims, int hist_n0) {
  pdl_launch_dependents();
  HalfPlace p = half_place(L);
  const AdjSim& A = ONE ? one : sims[p.sim];
  if (!L.blocks && p.z != INT_MAX) p.z *= L.deep;
  if (!half_inside(L, p, A.nx, A.ny, A.nz)) return;
  const int z1 = min(p.z + L.deep, A.nz);
  if constexpr (H_SIDE)
    adj_half_h(A, p.x, p.y, p.z, z1, L.n);
  else
    adj_half_e(A, p.x, p.y, p.z, z1, L.n, hist_n0);
}

}  // namespace rfn

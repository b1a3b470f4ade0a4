// Resident step kernel for sm_100a: one cooperative launch advances many time
// steps of a grid whose whole state fits in the shared memory of the GPU.
//
// A small grid's step is bound by latency, not by bandwidth: with one launch
// per step every block pays its launch, the chain index -> table row -> fields
// from L2, and a pipeline that fills for a handful of planes. Here each SM
// keeps one brick of the grid in shared memory for the whole launch, so a step
// is shared-memory arithmetic plus the exchange of the brick's faces.
//
//   brick     the grid is cut into px x py x pz bricks (thinner ones in the
//             absorbing layers where that pays), one block each, all
//             resident at once (cooperative launch). E and H of the brick's
//             cells and one halo layer (H above, E below) and the split pairs
//             of its split cells live in shared memory; where these do not all
//             fit the last of them stay in global memory (FAR)
//   cells     two lists per brick, one in the order of the E phase and one in
//             that of the H phase (built on the device once per simulation):
//             first the cells whose results a neighbour waits for, then the
//             others, each grouped by which components are stored split and by
//             table row, so that a warp's cells take the same path and mostly
//             one row
//   rows      the brick's distinct table rows in shared memory, as many as fit
//             beside the state (24 words each: rows with two Db per split and
//             probe cells' rows stay in global memory)
//   faces     a face value travels as one 8-byte word (value, step tag), so
//             the reader polls the word itself: no flag, no fence and no second
//             round trip. A word is written again only after its reader has
//             answered with its own faces of the same step, so one buffer is
//             enough
//   monitors  a plane monitor's elements in a brick are a list of the brick
//             (res_monitor_kernel); after a sampled step one more barrier, then
//             every thread adds its elements. The phasor sums stay in shared
//             memory for the launch as far as they fit beside the rest (in
//             global memory a 36-plane far-field box on 72x64x64 cells took 9 us
//             per step, a chain of L2 round trips per element)
//   waits     every poll is bounded; a block whose poll expires votes at the
//             next barrier, records an error code and returns
//
// Measured on a B200, per step, against the streaming kernels' best shape (one
// or two launches per step): 24x20x16 cells, 4-cell layers 9.0 -> 2.9 us;
// 64x64x48, 10-cell layers 17.2 -> 5.6 us; 91x71x53 graded, 7-cell layers 20.6
// -> 7.7 us; 100x80x64, 5-cell layers 25.8 -> 9.5 us; 133x44x88, 8-cell layers
// 11.4 us, half steps 15.5; 120x110x80 without layers 22.3 -> 16.0 us. With some
// pairs in global memory, against half steps: 139x49x93, 8-cell layers 17.2 -> 12.9
// us, 120x100x64 18.7 -> 14.5; 110x100x90, 6-cell layers 22.2 us is about the most. What bounds it now is a
// warp's chain of about a hundred dependent instructions per cell and phase
// (about 700 cycles, two or three cells per thread), shared-memory wavefronts,
// and two exchanges per step of about 0.6 us each, partly hidden. Two cells per
// thread loaded side by side spilled (64x64x48: 10.6 us); a barrier and a pass
// of their own for the face values cost 0.3 us more than sending from the
// cells' threads; rows read through L1 took 9.7 us (a gather of 32 rows is 32
// tag lookups).
//
// Same per-cell expressions as fdtd_step_kernel (fdtd_kernels.cuh) through the
// same rounding-fixed helpers, so all step kernels give the same bits. State
// between launches is time buffer 0.
#pragma once

#include "fdtd_kernels.cuh"

namespace rfn {

constexpr int kResThreads = 1024;   // most threads of a block
constexpr uint32_t kResNone = 0xffffu;
constexpr int kResMonitors = 50;    // most plane monitors of a simulation
// flags of a list entry beside the six bits of its split components
constexpr uint32_t kResProbe = 1u << 6;   // the cell holds probes
constexpr uint32_t kResGlobal = 1u << 7;  // its table row is read from global memory

// Soft sources of one field group of a cell (solver.cu:459-488, 515-541):
// s1 += v; s2 += v for every source probe on a component of that group (a
// sourced component is always stored as its split pair).
__device__ __forceinline__ void res_inject(const SimDev& S, const float4& r7, int n, bool e_side, float2 (&p)[3]) {
  const int np = int(__float_as_uint(r7.z) >> 16);
  const int first = __float_as_int(r7.w);
  for (int e = 0; e < np; ++e) {
    const int2 pe = __ldg(S.cell_probes + first + e);
    const bool mine = e_side ? pe.y < 3 : pe.y >= 3;
    if (mine && __ldg(S.is_src + pe.x)) {
      const float v = __ldg(S.src + (size_t)pe.x * S.nt + n);
      const int c = e_side ? pe.y : pe.y - 3;
#pragma unroll
      for (int k = 0; k < 3; ++k)
        if (c == k) {
          p[k].x = __fadd_rn(p[k].x, v);
          p[k].y = __fadd_rn(p[k].y, v);
        }
    }
  }
}

// Records this cell's probes of one field group (solver.cu:467, 521).
__device__ __forceinline__ void res_record(const SimDev& S, const float4& r7, int n, bool e_side, float a, float b,
                                           float c) {
  const int np = int(__float_as_uint(r7.z) >> 16);
  const int first = __float_as_int(r7.w);
  for (int e = 0; e < np; ++e) {
    const int2 pe = __ldg(S.cell_probes + first + e);
    const int f = e_side ? pe.y : pe.y - 3;
    if (f >= 0 && f < 3) S.rec[(size_t)pe.x * S.nt + n] = f == 0 ? a : f == 1 ? b : c;
  }
}

// How a grid is cut: bricks along each axis and the first cells of each. Layer
// cells cost more time (two values and an addition per component) and memory
// (up to 72 bytes instead of 24), so bricks in the layers may be thinner.
constexpr int kResCuts = 152;       // most bricks along an axis, and one
struct ResPart {
  int px, py, pz;
  int most[3];                     // cells of the longest brick along each axis
  uint16_t cut[3][kResCuts];
};

// The partition and the lists of one simulation.
struct ResGrid {
  SimDev s;
  ResPart part;
  int cap;                 // list entries per brick
  int row_cap;             // most table rows a brick keeps in shared memory
  const uint2* e_list;     // [brick][cap]: cell | row << 16, pair slot | (split components, flags) << 16
  const uint2* h_list;
  const uint2* e_words;    // [brick][cap]: the face words of the lists' face cells (x | y << 16, z; kResNone: none)
  const uint2* h_words;
  const int4* count;       // per brick: E-phase face cells, H-phase face cells, pairs, distinct rows
  const uint16_t* row_ids; // [brick][row_cap]: table rows of the brick's local row numbers
  const uint16_t* stride;  // [brick][64]: pairs between the components of the cells with a given set of split ones
  unsigned long long* e_face;  // [brick][face_cap] (value, tag)
  unsigned long long* h_face;
  int face_cap;
  const MonDev* mons;      // plane monitors
  int n_mon, mon_cap;
  const uint2* mon_list;   // [brick][mon_cap]: field word | monitor << 16 | H side << 31, element
  const int* mon_count;    // per brick
  uint32_t state;          // shared bytes for a brick's fields and pairs
  float2* far;             // [brick][far_cap]: the pairs that do not fit there
  int far_cap;
  int acc_f, acc_cap;      // phasor sums in shared memory: frequencies, elements per brick (the first of its list)
  int* err;
  uint32_t wait_limit;     // polls per face word
};

struct ResBox {
  int x0, y0, z0, bx, by, bz, ix, iy, iz;
  // strides of the brick's field arrays, which have one halo layer: odd, so that
  // cells along any axis lie in different banks
  __host__ __device__ int sy() const { return (bx + 1) | 1; }
  __host__ __device__ int sz() const { return (sy() * (by + 1)) | 1; }
  __host__ __device__ int size() const { return sz() * (bz + 1); }
};

__host__ __device__ __forceinline__ ResBox res_box(const ResPart& P, int b) {
  ResBox r;
  r.ix = b % P.px;
  r.iy = (b / P.px) % P.py;
  r.iz = b / (P.px * P.py);
  r.x0 = P.cut[0][r.ix];
  r.y0 = P.cut[1][r.iy];
  r.z0 = P.cut[2][r.iz];
  r.bx = P.cut[0][r.ix + 1] - r.x0;
  r.by = P.cut[1][r.iy + 1] - r.y0;
  r.bz = P.cut[2][r.iz + 1] - r.z0;
  return r;
}

// A row may go to a brick's local table: its H terms use one Db per split (a
// PEC edge correction makes two) and no probe list hangs on it.
__device__ __forceinline__ bool res_row_local(const float4* row) {
  const float4 p = row[3], q = row[4], u = row[5], v = row[6], r7 = row[7];
  auto same = [](float a, float b) { return __float_as_uint(a) == __float_as_uint(b); };
  return (__float_as_uint(r7.z) >> 16) == 0 && same(p.y, p.z) && same(q.x, q.y) && same(q.w, u.x) && same(u.z, u.w) &&
         same(v.y, v.z) && same(r7.x, r7.y);
}

// Scratch of the list building, per brick: map[table row]: its number in the
// brick (-1 unseen); then per number (cap entries each): the table row |
// position in the local table << 16, list positions (E face cells, E others, H
// face cells, H others), pair slots, and the numbers in list order.
struct ResScratch {
  int* map;
  int* num;
  int n_rows, cap;
  __device__ int* of(int b, int k) const { return num + (size_t(b) * 7 + k) * cap; }
};
constexpr int kResScratch = 7;

// A cell's sides in the exchange and its table row.
struct ResCell {
  int id, k;
  uint32_t flags;
  bool ex, ey, ez, hx, hy, hz;  // E sent up along x, y, z; H sent down
  int lx, ly, lz;
};

__device__ __forceinline__ ResCell res_cell(const SimDev& s, const ResPart& P, const ResBox& r, int c) {
  ResCell q;
  q.lx = c % r.bx;
  q.ly = (c / r.bx) % r.by;
  q.lz = c / (r.bx * r.by);
  q.id = s.mat[(r.z0 + q.lz) * s.plane + (r.y0 + q.ly) * s.pitch + r.x0 + q.lx];
  q.flags = __float_as_uint(s.rows[8 * q.id + 7].z);
  q.k = q.lz * r.sz() + q.ly * r.sy() + q.lx;
  q.ex = q.lx == r.bx - 1 && r.ix + 1 < P.px;
  q.ey = q.ly == r.by - 1 && r.iy + 1 < P.py;
  q.ez = q.lz == r.bz - 1 && r.iz + 1 < P.pz;
  q.hx = q.lx == 0 && r.ix > 0;
  q.hy = q.ly == 0 && r.iy > 0;
  q.hz = q.lz == 0 && r.iz > 0;
  return q;
}

// Adds the lanes' cells to the counters of their keys, one lane per distinct
// key; returns each lane's place.
__device__ __forceinline__ int res_take(int* n, int key, unsigned on) {
  const int lane = threadIdx.x & 31;
  const unsigned m = __match_any_sync(on, key);
  const int first = __ffs(int(m)) - 1;
  int at = 0;
  if (lane == first) {
    at = n[key];
    n[key] = at + __popc(m);
  }
  return __shfl_sync(m, at, first) + __popc(m & ((1u << lane) - 1u));
}

// First pass over one brick's cells (one warp): numbers the distinct table rows
// in the order they appear, gives those that may be local a place in the local
// table, and counts the cells of each row, the pairs and the face cells.
__global__ void __launch_bounds__(32)
res_count_kernel(const SimDev s, const __grid_constant__ ResPart P, const ResScratch X, int4* __restrict__ count,
                 int* __restrict__ n_nums) {
  const int lane = threadIdx.x, b = blockIdx.x;
  const ResBox r = res_box(P, b);
  const int cells = r.bx * r.by * r.bz;
  int* const mp = X.map + size_t(b) * X.n_rows;
  int* const info = X.of(b, 0);
  int fe = 0, fh = 0, pairs = 0, nums = 0;
  for (int c0 = 0; c0 < cells; c0 += 32) {
    const int c = c0 + lane;
    const unsigned on = __ballot_sync(0xffffffffu, c < cells);
    if (c < cells) {
      const ResCell q = res_cell(s, P, r, c);
      const bool ef = q.ex || q.ey || q.ez, hf = q.hx || q.hy || q.hz;
      fe += ef;
      fh += hf;
      pairs += __popc((q.flags >> 8) & 63u);
      const unsigned m = __match_any_sync(on, q.id);
      const bool first = __ffs(int(m)) - 1 == lane && mp[q.id] == -1;
      const unsigned f = __ballot_sync(on, first);
      if (first) {
        const int k = nums + __popc(f & ((1u << lane) - 1u));
        mp[q.id] = k;
        info[k] = q.id;
        for (int j = 1; j < 6; ++j) X.of(b, j)[k] = 0;
      }
      nums += __popc(f);
      __syncwarp(on);
      const int k = mp[q.id];
      res_take(X.of(b, ef ? 1 : 2), k, __match_any_sync(on, int(ef)));
      __syncwarp(on);
      res_take(X.of(b, hf ? 3 : 4), k, __match_any_sync(on, int(hf)));
      __syncwarp(on);
    }
    nums = __shfl_sync(0xffffffffu, nums, 0);  // (lane 0 always has a cell)
  }
  int n_local = 0;
  for (int k0 = 0; k0 < nums; k0 += 32) {
    const int k = k0 + lane, id = k < nums ? info[k] : 0;
    const bool local = k < nums && res_row_local(s.rows + 8 * id);
    const unsigned f = __ballot_sync(0xffffffffu, local);
    if (k < nums) info[k] = id | (local ? n_local + __popc(f & ((1u << lane) - 1u)) : int(kResNone)) << 16;
    n_local += __popc(f);
  }
  for (int o = 16; o > 0; o >>= 1) {
    fe += __shfl_down_sync(0xffffffffu, fe, o);
    fh += __shfl_down_sync(0xffffffffu, fh, o);
    pairs += __shfl_down_sync(0xffffffffu, pairs, o);
  }
  if (lane == 0) {
    count[b] = make_int4(fe, fh, pairs, n_local);
    n_nums[b] = nums;
  }
}

// Second pass: the lists of one brick (one warp), ordered by face cell or not,
// then by set of split components, then by table row.
__global__ void __launch_bounds__(32)
res_build_kernel(const SimDev s, const __grid_constant__ ResPart P, const ResScratch X, const int* __restrict__ n_nums, int cap,
                 int row_cap, uint2* __restrict__ e_list, uint2* __restrict__ h_list, uint2* __restrict__ e_words,
                 uint2* __restrict__ h_words, uint16_t* __restrict__ row_ids, uint16_t* __restrict__ stride) {
  __shared__ int n_m[64];
  const int lane = threadIdx.x, b = blockIdx.x;
  const ResBox r = res_box(P, b);
  const int cells = r.bx * r.by * r.bz, nums = n_nums[b];
  const int* const mp = X.map + size_t(b) * X.n_rows;
  const int* const info = X.of(b, 0);
  int* const order = X.of(b, 6);
  // first words of the y and z faces (laid out for the largest brick, so that
  // a face has the same words in both bricks' buffers)
  const int mx = P.most[0], my = P.most[1], mz = P.most[2];
  const int wy = 2 * my * mz, wz = wy + 2 * mx * mz;
  auto split_set = [&](int k) { return int((__float_as_uint(s.rows[8 * (info[k] & 0xffff) + 7].z) >> 8) & 63u); };
  // the numbers in order of their split sets (most components first)
  for (int i = lane; i < 64; i += 32) n_m[i] = 0;
  __syncwarp();
  for (int pass = 0; pass < 2; ++pass) {
    for (int k0 = 0; k0 < nums; k0 += 32) {
      const int k = k0 + lane;
      const unsigned on = __ballot_sync(0xffffffffu, k < nums);
      if (k < nums) {
        const int at = res_take(n_m, split_set(k), on);
        if (pass == 1) order[at] = k;
      }
      __syncwarp();
    }
    if (pass == 0 && lane == 0)
      for (int m = 63, at = 0; m >= 0; --m) {
        const int c = n_m[m];
        n_m[m] = at;
        at += c;
      }
    __syncwarp();
  }
  // cells per row to first list positions, in that order; pair slots of the
  // rows of one split set lie side by side, the set's components `stride` apart
  int at[5] = {0, 0, 0, 0, 0};  // E face, E others, H face, H others, pairs
  for (int pass = 0; pass < 2; ++pass) {  // pass 0 sums the face cells, which go first
    if (pass == 1) {
      at[1] = at[0];
      at[3] = at[2];
      at[0] = at[2] = 0;
    }
    int set_now = -1, set_first = 0, set_cells = 0;  // the running set's first slot and cells so far
    for (int k0 = 0; k0 < nums; k0 += 32) {
      const int o = k0 + lane < nums ? order[k0 + lane] : -1;
      int n[4], set = -2;
      for (int j = 0; j < 4; ++j) n[j] = o >= 0 ? X.of(b, 1 + j)[o] : 0;
      if (o >= 0) set = split_set(o);
      for (int l = 0; l < 32; ++l) {  // (the rows of a brick are few: a serial scan)
        const int sl = __shfl_sync(0xffffffffu, set, l), ol = __shfl_sync(0xffffffffu, o, l);
        int nl[4];
        for (int j = 0; j < 4; ++j) nl[j] = __shfl_sync(0xffffffffu, n[j], l);
        if (ol < 0) break;
        if (pass == 1) {
          if (sl != set_now) {
            if (set_now >= 0) {
              if (lane == 0) stride[size_t(b) * 64 + set_now] = uint16_t(set_cells);
              set_first += set_cells * __popc(unsigned(set_now));
            }
            set_now = sl;
            set_cells = 0;
          }
          if (lane == 0) {
            for (int j = 0; j < 4; ++j) X.of(b, 1 + j)[ol] = at[j];
            X.of(b, 5)[ol] = set_first + set_cells;
          }
          set_cells += nl[0] + nl[1];
        }
        if (pass == 0) {
          at[0] += nl[0];
          at[2] += nl[2];
        } else {
          for (int j = 0; j < 4; ++j) at[j] += nl[j];
        }
      }
    }
    if (pass == 1 && set_now >= 0 && lane == 0) stride[size_t(b) * 64 + set_now] = uint16_t(set_cells);
    __syncwarp();
  }
  for (int k = lane; k < nums; k += 32) {
    const int tab = int(unsigned(info[k]) >> 16);
    if (tab < row_cap) row_ids[size_t(b) * row_cap + tab] = uint16_t(info[k] & 0xffff);
  }
  __syncwarp();
  for (int c0 = 0; c0 < cells; c0 += 32) {
    const int c = c0 + lane;
    const unsigned on = __ballot_sync(0xffffffffu, c < cells);
    if (c < cells) {
      const ResCell q = res_cell(s, P, r, c);
      const bool ef = q.ex || q.ey || q.ez, hf = q.hx || q.hy || q.hz;
      const int k = mp[q.id];
      const int tab = int(unsigned(info[k]) >> 16);
      const bool glob = tab >= row_cap;
      const int at_e = res_take(X.of(b, ef ? 1 : 2), k, __match_any_sync(on, int(ef)));
      __syncwarp(on);
      const int at_h = res_take(X.of(b, hf ? 3 : 4), k, __match_any_sync(on, int(hf)));
      __syncwarp(on);
      const int slot = res_take(X.of(b, 5), k, on);
      __syncwarp(on);
      const uint32_t fl = ((q.flags >> 8) & 63u) | ((q.flags >> 16) ? kResProbe : 0u) | (glob ? kResGlobal : 0u);
      const uint2 d = make_uint2(uint32_t(q.k) | uint32_t(glob ? q.id : tab) << 16, (uint32_t(slot) & 0xffffu) | fl << 16);
      e_list[size_t(b) * cap + at_e] = d;
      h_list[size_t(b) * cap + at_h] = d;
      const uint32_t fx = uint32_t(q.lz * r.by + q.ly), fy = uint32_t(wy + q.lz * r.bx + q.lx),
                     fz = uint32_t(wz + q.ly * r.bx + q.lx);
      if (ef)
        e_words[size_t(b) * cap + at_e] =
            make_uint2((q.ex ? fx : kResNone) | (q.ey ? fy : kResNone) << 16, q.ez ? fz : kResNone);
      if (hf)
        h_words[size_t(b) * cap + at_h] =
            make_uint2((q.hx ? fx : kResNone) | (q.hy ? fy : kResNone) << 16, q.hz ? fz : kResNone);
    }
    __syncwarp();
  }
}

// The part of [0, n) of a monitor's in-plane axis, or its position, that lies
// in a brick's [c0, c0 + cn).
__host__ __device__ __forceinline__ int res_mon_elements(const MonDev& M, const ResBox& r) {
  const int lo[3] = {r.x0, r.y0, r.z0}, n[3] = {r.bx, r.by, r.bz};
  if (M.position < lo[M.axis] || M.position >= lo[M.axis] + n[M.axis]) return 0;
  return n[M.axis == 0 ? 1 : 0] * n[M.axis == 2 ? 1 : 2];
}

// Lists the monitor elements of one brick (one block), monitor by monitor, in
// the order of the monitor's output.
__global__ void __launch_bounds__(128)
res_monitor_kernel(const __grid_constant__ ResPart P, const MonDev* __restrict__ mons, int n_mon, int cap,
                   uint2* __restrict__ list, int* __restrict__ count) {
  const ResBox r = res_box(P, blockIdx.x);
  const int e0 = 1 + r.sy() + r.sz();
  int base = 0;
  for (int m = 0; m < n_mon; ++m) {
    const MonDev M = mons[m];
    const int n = res_mon_elements(M, r), n2 = M.axis == 2 ? r.by : r.bz;
    for (int i = threadIdx.x; i < n; i += blockDim.x) {
      const int a = i / n2, b = i - a * n2;
      const int lx = M.axis == 0 ? M.position - r.x0 : a;
      const int ly = M.axis == 0 ? a : M.axis == 1 ? M.position - r.y0 : b;
      const int lz = M.axis == 2 ? M.position - r.z0 : b;
      const int k = lz * r.sz() + ly * r.sy() + lx;
      const int ga = M.axis == 0 ? r.y0 + ly : r.x0 + lx, gb = M.axis == 2 ? r.y0 + ly : r.z0 + lz;
      const uint32_t word = M.field < 3 ? uint32_t(3 * (k + e0) + M.field) : uint32_t(3 * k + M.field - 3);
      list[size_t(blockIdx.x) * cap + base + i] =
          make_uint2(word | uint32_t(m) << 16 | (M.field < 3 ? 0u : 1u << 31), uint32_t(ga * M.n2 + gb));
    }
    base += n;
  }
  if (threadIdx.x == 0) count[blockIdx.x] = base;
}

// Shared bytes of a brick: its local rows (12 E words, 12 H words: Da, Db of
// each split), six field arrays with one halo layer, its pairs.
constexpr uint32_t kResRowBytes = 96;
__host__ __device__ __forceinline__ uint32_t res_smem(int bx, int by, int bz, int pairs) {
  const ResBox r{0, 0, 0, bx, by, bz, 0, 0, 0};
  return ((6u * uint32_t(r.size()) + 1u) & ~1u) * 4u + uint32_t(pairs) * 8u;
}

__device__ __forceinline__ void res_put(unsigned long long* p, float v, uint32_t tag) {
  const unsigned long long w = (static_cast<unsigned long long>(tag) << 32) | __float_as_uint(v);
  asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(p), "l"(w) : "memory");
}
__device__ __forceinline__ unsigned long long res_get(const unsigned long long* p) {
  unsigned long long w;
  asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(w) : "l"(p) : "memory");
  return w;
}

// Pairs of a brick that fit in `state` bytes beside its fields.
__host__ __device__ __forceinline__ int res_pair_cap(const ResBox& r, uint32_t state) {
  return int((state - res_smem(r.bx, r.by, r.bz, 0)) / 8u);
}

// Advances steps n0 .. n1-1 of the grid. FACES: face values of one side per
// thread (at least a brick's face values / threads). MON: with plane monitors.
// FAR: the last pairs of a brick lie in global memory (each belongs to one thread
// per phase, so nothing is shared through it); the addresses of all pairs are then
// generic ones.
template <int FACES, int THREADS, bool MON, bool FAR>
__global__ void __launch_bounds__(THREADS, 1)
res_step_kernel(const __grid_constant__ ResGrid G, int n0, int n1) {
  // E quads, H quads of the local rows, then fields, pairs, phasor sums
  extern __shared__ __align__(16) float4 s_rows[];
  __shared__ int s_stride[64];
  __shared__ MonDev s_mon[MON ? kResMonitors : 1];
  __shared__ int s_sample[MON ? kResMonitors : 1];  // this step's sample of each monitor, -1: none
  const SimDev& S = G.s;
  const int T = blockDim.x, tid = threadIdx.x;
  const ResBox r = res_box(G.part, blockIdx.x);
  // Position k = (lz, ly, lx) of own cell (lx, ly, lz). The three components of
  // a position lie side by side: the three words' odd stride keeps a warp's
  // accesses free of bank conflicts and a neighbour costs one address. H has
  // its halo above (lx = bx, ...); E its halo below, so E of cell k lies e0
  // positions further.
  const int sy = r.sy(), sz = r.sz(), V = r.size(), e0 = 1 + sy + sz;
  const float4* const e_rows = s_rows;
  const float4* const h_rows = s_rows + 3 * G.row_cap;
  float* const H = reinterpret_cast<float*>(s_rows + 6 * G.row_cap);
  float* const E = H + 3 * V;
  float2* const P = reinterpret_cast<float2*>(H + ((6 * V + 1) & ~1));
  const int4 cnt = G.count[blockIdx.x];
  const int cells = r.bx * r.by * r.bz;
  const uint2* const el = G.e_list + size_t(blockIdx.x) * G.cap;
  const uint2* const hl = G.h_list + size_t(blockIdx.x) * G.cap;
  const float4* const rows = S.rows;
  // the monitor elements whose sums stay here: nm_in of the brick's nm, sum of
  // frequency f of element i at acc[f * acc_cap + i]
  const int near = FAR ? min(cnt.z, res_pair_cap(r, G.state)) : cnt.z;
  float2* const far = FAR ? G.far + size_t(blockIdx.x) * G.far_cap : nullptr;
  auto pair = [&](int q) -> float2& { return FAR && q >= near ? far[q - near] : P[q]; };
  float2* const acc = P + near;
  const uint2* const ml = G.mon_list + size_t(blockIdx.x) * G.mon_cap;
  const int nm = MON ? G.mon_count[blockIdx.x] : 0, nm_in = MON ? min(nm, G.acc_cap) : 0;
  if (MON)
    for (int m = tid; m < G.n_mon; m += T) s_mon[m] = G.mons[m];
  for (int i = tid; i < nm_in; i += T) {
    const uint2 d = ml[i];
    const MonDev M = G.mons[(d.x >> 16) & 0x7fffu];
    for (int f = 0; f < G.acc_f; ++f)
      acc[f * G.acc_cap + i] = static_cast<const float2*>(M.out)[size_t(f) * M.n1 * M.n2 + d.y];
  }
  for (int k = tid; k < 64; k += T) s_stride[k] = G.stride[size_t(blockIdx.x) * 64 + k];
  for (int k = tid; k < min(cnt.w, G.row_cap); k += T) {
    const float4* const row = rows + 8 * int(G.row_ids[size_t(blockIdx.x) * G.row_cap + k]);
    const float4 p = row[3], q = row[4], u = row[5], v = row[6];
    for (int j = 0; j < 3; ++j) s_rows[3 * k + j] = row[j];
    float4* const h = s_rows + 3 * G.row_cap + 3 * k;
    h[0] = make_float4(p.x, p.y, p.w, q.x);
    h[1] = make_float4(q.z, q.w, u.y, u.z);
    h[2] = make_float4(v.x, v.y, v.w, row[7].x);
  }

  // ---- load the brick: H with its halo (zero outside the grid), E, pairs
  for (int k = tid; k < V; k += T) {
    const int lz = k / sz, ly = (k - lz * sz) / sy, lx = k - lz * sz - ly * sy;
    const int x = r.x0 + lx, y = r.y0 + ly, z = r.z0 + lz;
    const bool in = lx <= r.bx && ly <= r.by && x < S.nx && y < S.ny && z < S.nz;
    const int i = z * S.plane + y * S.pitch + x;
    for (int c = 0; c < 3; ++c) {
      H[3 * k + c] = in ? S.H[0][c][i] : 0.f;
      E[3 * k + c] = 0.f;
    }
  }
  __syncthreads();
  // a list entry's cell offset in the field arrays, and where its pairs lie in
  // the split stores
  auto cell_of = [&](const uint2& d, int& x, int& y, int& z) {
    const int k = int(d.x & 0xffffu);
    const int lz = k / sz, ly = (k - lz * sz) / sy;
    x = r.x0 + k - lz * sz - ly * sy;
    y = r.y0 + ly;
    z = r.z0 + lz;
    return z * S.plane + y * S.pitch + x;
  };
  auto store_of = [&](int x, int y, int z, int i, int& cs) {
    const int slot = __float_as_int(__ldg(&rows[8 * int(S.mat[i]) + 7].w));
    return S.sp.base[0] + split_off(S.sp, split_store(S.sp, S.nx, S.ny, S.nz, x, y, z), x, y, z, slot, cs);
  };
  for (int c = tid; c < cells; c += T) {
    const uint2 d = el[c];
    const uint32_t f = d.y >> 16;
    int x, y, z;
    const int i = cell_of(d, x, y, z);
    float* const e = E + 3 * (int(d.x & 0xffffu) + e0);
    for (int m = 0; m < 3; ++m)
      if (!(f >> m & 1u)) e[m] = S.E[0][m][i];
    if (f & 63u) {
      int cs;
      const float2* const g = store_of(x, y, z, i, cs);
      int p = int(d.y & 0xffffu);
      const int st = s_stride[f & 63u];
      for (int m = 0; m < 6; ++m)
        if (f >> m & 1u) {
          pair(p) = g[m * cs];
          p += st;
        }
    }
  }

  // ---- the face values this thread receives: H from above (hi), E from below
  // (lo); along x components 1, 2, along y 0, 2, along z 0, 1. Face value q of
  // a brick lies at word q of its buffers. hi / lo: the halo cell's word in H
  // and E (kResNone: no neighbour), step: distance to the neighbour's buffer.
  uint32_t hi[FACES], lo[FACES];
  int step[FACES];
  {
    const int fx = r.by * r.bz, fy = r.bx * r.bz, fz = r.bx * r.by;
    // words of the x, y and z faces, laid out for the largest brick so that a
    // face has the same words in both bricks' buffers
    const int mx = G.part.most[0], my = G.part.most[1], mz = G.part.most[2];
    const int wy = 2 * my * mz, wz = wy + 2 * mx * mz;
#pragma unroll
    for (int j = 0; j < FACES; ++j) {
      const int q = tid + j * T;
      hi[j] = lo[j] = kResNone;
      step[j] = 0;
      const int axis = q < wy ? 0 : q < wz ? 1 : 2;
      const int e = q - (axis == 0 ? 0 : axis == 1 ? wy : wz), n = axis == 0 ? fx : axis == 1 ? fy : fz;
      if (e >= 2 * n) continue;
      const int second = e >= n ? 1 : 0, pos = e - second * n;
      const int comp = axis == 0 ? 1 + second : axis == 1 ? 2 * second : second;
      const int na = axis == 0 ? r.by : r.bx, a = pos % na, b = pos / na;
      // the face's cell at layer l along the axis
      auto cell = [&](int l) {
        return axis == 0 ? b * sz + a * sy + l : axis == 1 ? b * sz + l * sy + a : l * sz + b * sy + a;
      };
      const int len = axis == 0 ? r.bx : axis == 1 ? r.by : r.bz;
      const bool up = axis == 0 ? r.ix + 1 < G.part.px : axis == 1 ? r.iy + 1 < G.part.py : r.iz + 1 < G.part.pz;
      const bool down = axis == 0 ? r.ix > 0 : axis == 1 ? r.iy > 0 : r.iz > 0;
      step[j] = (axis == 0 ? 1 : axis == 1 ? G.part.px : G.part.px * G.part.py) * G.face_cap;
      if (up) hi[j] = uint32_t(3 * cell(len) + comp);
      if (down) lo[j] = uint32_t(3 * (cell(-1) + e0) + comp);
    }
  }
  unsigned long long* const e_face = G.e_face + size_t(blockIdx.x) * G.face_cap;
  unsigned long long* const h_face = G.h_face + size_t(blockIdx.x) * G.face_cap;
  const uint2* const ew = G.e_words + size_t(blockIdx.x) * G.cap;
  const uint2* const hw = G.h_words + size_t(blockIdx.x) * G.cap;
  // sends a face cell's values to the bricks that wait for them
  auto send = [&](unsigned long long* face, const uint2& w, float vx, float vy, float vz, uint32_t tag) {
    const uint32_t wx = w.x & 0xffffu, wy = w.x >> 16, wz = w.y;
    if (wx != kResNone) {
      res_put(face + wx, vy, tag);
      res_put(face + wx + r.by * r.bz, vz, tag);
    }
    if (wy != kResNone) {
      res_put(face + wy, vx, tag);
      res_put(face + wy + r.bx * r.bz, vz, tag);
    }
    if (wz != kResNone) {
      res_put(face + wz, vx, tag);
      res_put(face + wz + r.bx * r.by, vy, tag);
    }
  };
  __syncthreads();

  // polls one face word for tag `want`
  auto receive = [&](const unsigned long long* p, uint32_t want, float& v) -> bool {
    unsigned long long w = res_get(p);
    for (uint32_t i = 0; uint32_t(w >> 32) != want; ++i) {
      if (i >= G.wait_limit) return false;
      w = res_get(p);
    }
    v = __uint_as_float(uint32_t(w));
    return true;
  };

  for (int n = n0; n < n1; ++n) {
    // ------------------------------------------------------------ E phase
    bool bad = false;
    uint2 next = tid < cells ? __ldg(el + tid) : make_uint2(0u, 0u);
    if (n > n0) {
#pragma unroll
      for (int j = 0; j < FACES; ++j)
        if (hi[j] != kResNone) bad |= !receive(h_face + tid + j * T + step[j], uint32_t(n), H[hi[j]]);
    }
    if (__syncthreads_or(bad)) {
      if (tid == 0) atomicExch(G.err, kErrFaceExpired);
      return;
    }
#pragma unroll 1
    for (int c = tid; c < cells; c += T) {
      const uint2 d = next;
      if (c + T < cells) next = __ldg(el + c + T);
      const uint32_t f = d.y >> 16;
      float4 ra, rb, rd;
      if (!(f & kResGlobal)) {
        const float4* const row = e_rows + 3 * (d.x >> 16);
        ra = row[0]; rb = row[1]; rd = row[2];
      } else {
        const float4* const row = rows + 8 * (d.x >> 16);
        ra = __ldg(row); rb = __ldg(row + 1); rd = __ldg(row + 2);
      }
      const int k = 3 * int(d.x & 0xffffu);
      const float* const h = H + k;
      const float* const hy_p = h + 3 * sy;
      const float* const hz_p = h + 3 * sz;
      float* const e = E + k + 3 * e0;
      const float hx = h[0], hy = h[1], hz = h[2];
      const float dhz_y = hy_p[2] - hz, dhy_z = hz_p[1] - hy;
      const float dhx_z = hz_p[0] - hx, dhz_x = h[5] - hz;
      const float dhy_x = h[4] - hy, dhx_y = hy_p[0] - hx;
      float vx = upd_e(ra.x, e[0], ra.y, dhz_y, ra.w, dhy_z);
      float vy = upd_e(rb.x, e[1], rb.y, dhx_z, rb.w, dhz_x);
      float vz = upd_e(rd.x, e[2], rd.y, dhy_x, rd.w, dhx_y);
      if (f & 7u) {
        const int st = s_stride[f & 63u];
        const int q0 = int(d.y & 0xffffu), q1 = q0 + ((f & 1u) ? st : 0), q2 = q1 + ((f & 2u) ? st : 0);
        float2 p[3];
        p[0] = (f & 1u) ? pair(q0) : make_float2(0.f, 0.f);
        p[1] = (f & 2u) ? pair(q1) : make_float2(0.f, 0.f);
        p[2] = (f & 4u) ? pair(q2) : make_float2(0.f, 0.f);
        p[0].x = upd_e_split(ra.x, p[0].x, ra.y, dhz_y);  // ex_y
        p[0].y = upd_e_split(ra.z, p[0].y, ra.w, dhy_z);  // ex_z
        p[1].x = upd_e_split(rb.x, p[1].x, rb.y, dhx_z);  // ey_z
        p[1].y = upd_e_split(rb.z, p[1].y, rb.w, dhz_x);  // ey_x
        p[2].x = upd_e_split(rd.x, p[2].x, rd.y, dhy_x);  // ez_x
        p[2].y = upd_e_split(rd.z, p[2].y, rd.w, dhx_y);  // ez_y
        if (f & kResProbe) res_inject(S, __ldg(rows + 8 * (d.x >> 16) + 7), n, true, p);
        if (f & 1u) { vx = __fadd_rn(p[0].x, p[0].y); pair(q0) = p[0]; }
        if (f & 2u) { vy = __fadd_rn(p[1].x, p[1].y); pair(q1) = p[1]; }
        if (f & 4u) { vz = __fadd_rn(p[2].x, p[2].y); pair(q2) = p[2]; }
      }
      if (c < cnt.x) send(e_face, __ldg(ew + c), vx, vy, vz, uint32_t(n) + 1u);
      e[0] = vx;
      e[1] = vy;
      e[2] = vz;
      if (f & kResProbe) res_record(S, __ldg(rows + 8 * (d.x >> 16) + 7), n, true, vx, vy, vz);
    }
    // ------------------------------------------------------------ H phase
    if (tid < cells) next = __ldg(hl + tid);
#pragma unroll
    for (int j = 0; j < FACES; ++j)
      if (lo[j] != kResNone) bad |= !receive(e_face + tid + j * T - step[j], uint32_t(n) + 1u, E[lo[j]]);
    if (__syncthreads_or(bad)) {
      if (tid == 0) atomicExch(G.err, kErrFaceExpired);
      return;
    }
#pragma unroll 1
    for (int c = tid; c < cells; c += T) {
      const uint2 d = next;
      if (c + T < cells) next = __ldg(hl + c + T);
      const uint32_t f = d.y >> 16;
      // (Da, Db) of both splits of each component; Db of the own and of the
      // neighbour's E differ only in rows read from global memory
      float4 kx, ky, kz;
      float bxy, bxz, byz, byx, bzx, bzy;
      if (!(f & kResGlobal)) {
        const float4* const row = h_rows + 3 * (d.x >> 16);
        kx = row[0]; ky = row[1]; kz = row[2];
        bxy = kx.y; bxz = kx.w; byz = ky.y; byx = ky.w; bzx = kz.y; bzy = kz.w;
      } else {
        const float4* const row = rows + 8 * (d.x >> 16);
        const float4 p = __ldg(row + 3), q = __ldg(row + 4), u = __ldg(row + 5), v = __ldg(row + 6), w = __ldg(row + 7);
        kx = make_float4(p.x, p.y, p.w, q.x);
        ky = make_float4(q.z, q.w, u.y, u.z);
        kz = make_float4(v.x, v.y, v.w, w.x);
        bxy = p.z; bxz = q.y; byz = u.x; byx = u.w; bzx = v.z; bzy = w.y;
      }
      const int k = 3 * int(d.x & 0xffffu);
      float* const h = H + k;
      const float* const e = E + k + 3 * e0;
      const float* const ey_m = e - 3 * sy;
      const float* const ez_m = e - 3 * sz;
      const float ex = e[0], ey = e[1], ez = e[2];
      const float gxy = h_term(bxy, ez, kx.y, ey_m[2]);
      const float gxz = h_term(bxz, ey, kx.w, ez_m[1]);
      const float gyz = h_term(byz, ex, ky.y, ez_m[0]);
      const float gyx = h_term(byx, ez, ky.w, e[-1]);
      const float gzx = h_term(bzx, ey, kz.y, e[-2]);
      const float gzy = h_term(bzy, ex, kz.w, ey_m[0]);
      float vx = upd_h(kx.x, h[0], gxy, gxz);
      float vy = upd_h(ky.x, h[1], gyz, gyx);
      float vz = upd_h(kz.x, h[2], gzx, gzy);
      if (f & 56u) {
        const int st = s_stride[f & 63u];
        const int q0 = int(d.y & 0xffffu) + __popc(f & 7u) * st, q1 = q0 + ((f & 8u) ? st : 0),
                  q2 = q1 + ((f & 16u) ? st : 0);
        float2 p[3];
        p[0] = (f & 8u) ? pair(q0) : make_float2(0.f, 0.f);
        p[1] = (f & 16u) ? pair(q1) : make_float2(0.f, 0.f);
        p[2] = (f & 32u) ? pair(q2) : make_float2(0.f, 0.f);
        p[0].x = upd_h_split(kx.x, p[0].x, gxy);
        p[0].y = upd_h_split(kx.z, p[0].y, gxz);
        p[1].x = upd_h_split(ky.x, p[1].x, gyz);
        p[1].y = upd_h_split(ky.z, p[1].y, gyx);
        p[2].x = upd_h_split(kz.x, p[2].x, gzx);
        p[2].y = upd_h_split(kz.z, p[2].y, gzy);
        if (f & kResProbe) res_inject(S, __ldg(rows + 8 * (d.x >> 16) + 7), n, false, p);
        if (f & 8u) { vx = __fadd_rn(p[0].x, p[0].y); pair(q0) = p[0]; }
        if (f & 16u) { vy = __fadd_rn(p[1].x, p[1].y); pair(q1) = p[1]; }
        if (f & 32u) { vz = __fadd_rn(p[2].x, p[2].y); pair(q2) = p[2]; }
      }
      if (c < cnt.y) send(h_face, __ldg(hw + c), vx, vy, vz, uint32_t(n) + 1u);
      h[0] = vx;
      h[1] = vy;
      h[2] = vz;
      if (f & kResProbe) res_record(S, __ldg(rows + 8 * (d.x >> 16) + 7), n, false, vx, vy, vz);
    }
    if (MON) {
      for (int m = tid; m < G.n_mon; m += T)
        s_sample[m] = monitor_samples(n, s_mon[m].n_step) ? n / s_mon[m].n_step : -1;
      __syncthreads();
      for (int i = tid; i < nm; i += T) {
        const uint2 d = __ldg(ml + i);
        const int m = int((d.x >> 16) & 0x7fffu), mn = s_sample[m];
        if (mn < 0) continue;
        const MonDev& M = s_mon[m];
        const float v = ((d.x >> 31) ? H : E)[d.x & 0xffffu];
        if (i < nm_in) {
          const float2* const ph = M.phase + size_t(mn) * G.acc_f;
          for (int f = 0; f < G.acc_f; ++f) {
            const float2 p = __ldg(ph + f);
            float2 a = acc[f * G.acc_cap + i];
            a.x = __fmaf_rn(v, p.x, a.x);
            a.y = __fmaf_rn(v, p.y, a.y);
            acc[f * G.acc_cap + i] = a;
          }
        } else {
          monitor_add(M, M.n1 * M.n2, int(d.y), mn, v);
        }
      }
    }
  }
  __syncthreads();

  // ---- the sums and the state after the last step
  for (int i = tid; i < nm_in; i += T) {
    const uint2 d = ml[i];
    const MonDev M = G.mons[(d.x >> 16) & 0x7fffu];
    for (int f = 0; f < G.acc_f; ++f)
      static_cast<float2*>(M.out)[size_t(f) * M.n1 * M.n2 + d.y] = acc[f * G.acc_cap + i];
  }
  for (int c = tid; c < cells; c += T) {
    const uint2 d = el[c];
    const uint32_t f = d.y >> 16;
    int x, y, z;
    const int i = cell_of(d, x, y, z);
    const float* const h = H + 3 * int(d.x & 0xffffu);
    const float* const e = E + 3 * (int(d.x & 0xffffu) + e0);
    for (int m = 0; m < 3; ++m) {
      S.H[0][m][i] = h[m];
      if (!(f >> m & 1u)) S.E[0][m][i] = e[m];
    }
    if (f & 63u) {
      int cs;
      float2* const g = store_of(x, y, z, i, cs);
      int p = int(d.y & 0xffffu);
      const int st = s_stride[f & 63u];
      for (int m = 0; m < 6; ++m)
        if (f >> m & 1u) {
          g[m * cs] = pair(p);
          p += st;
        }
    }
  }
}

}  // namespace rfn

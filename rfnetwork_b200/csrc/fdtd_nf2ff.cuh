// Near-field to far-field transform of equivalent surface currents
// (rfnetwork/core/src/postprocess.cpp:130-505, postprocess_nf2ff).
//
// For every frequency f and direction (theta, phi), with r^ = (u, v, w) =
// (sin th cos ph, sin th sin ph, cos th):
//   S_J = sum over the surface cells c of ds_c J_c exp(j beta r^ . r_c), S_M alike
//   N_theta = S_Jx cos th cos ph + S_Jy cos th sin ph - S_Jz sin th,  N_phi = -S_Jx sin ph + S_Jy cos ph
//   L_theta, L_phi from S_M the same way
//   E_theta = (-j beta / 4 pi) (L_phi + eta0 N_theta),  E_phi = (j beta / 4 pi) (L_theta - eta0 N_phi)
// The reference loops frequency x theta x phi x faces on one CPU thread and
// forms the four sums per face. Here one thread owns one direction of one
// frequency and accumulates the six current moments S_J, S_M; the cells of all
// faces are cut into parts, one row of blocks each, so that a pattern of a few
// hundred directions still fills the GPU, and a second kernel adds the parts in
// order and forms the fields. A block stages its cells through shared memory.
// Phases and products are FP32 (as the reference), the running sums FP64 across
// chunks and parts.
//
// Bound by FP32 issue: one sincosf and twelve packed multiply-adds (two FP32
// lanes each) per cell and direction. 17,400 cells x 1,729 directions x 2
// frequencies: with one part (28 blocks on 148 SMs, unpacked arithmetic, the
// cells packed on the host) the call took 2.93 ms; with 43 parts the kernels
// take 0.19 + 0.03 ms and the call 0.52 ms. The error against 64 bits went from
// 2.2e-7 to 1.7e-7 (runs of 128 cells in FP32: 2.8e-7).
#pragma once

#include <cstdint>

namespace rfn {

constexpr double kEta0 = 376.730313;  // free-space impedance used by the reference (postprocess.cpp:39)
constexpr int kNf2ffThreads = 128;
constexpr int kNf2ffRun = 32;  // cells summed in FP32 before they join the FP64 sums

// One face of the surface: its arrays as offsets (floats) into the call's data.
struct Nf2ffFaceDev {
  int axis, cells, first;  // first: cells of the faces before it
  float pos;
  int64_t r0, r1, ds, J, M;  // J, M: [3][frequency][cell] complex
};

// One surface cell at one frequency: position (m) and ds J, ds M (complex), each
// real and imaginary part twice, as the packed multiply-adds take them.
struct Nf2ffCell {
  float4 pos;
  float4 cur[6];  // re, re, im, im
};

// a * b + c on two FP32 lanes (fma.rn.f32x2).
__device__ __forceinline__ unsigned long long ffma2(unsigned long long a, unsigned long long b, unsigned long long c) {
  unsigned long long d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
  return d;
}
__device__ __forceinline__ unsigned long long pack2(float lo, float hi) {
  unsigned long long d;
  asm("mov.b64 %0, {%1, %2};" : "=l"(d) : "f"(lo), "f"(hi));
  return d;
}
__device__ __forceinline__ void unpack2(unsigned long long v, float& lo, float& hi) {
  asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v));
}

// Far field of the moments acc (Jx Jy Jz Mx My Mz, each re, im) in one
// direction: E_theta to out[o], E_phi to out[half + o].
__device__ __forceinline__ void nf2ff_field(const double (&acc)[12], float beta, float theta, float phi, float2* out,
                                            size_t o, size_t half) {
  float sin_th, cos_th, sin_ph, cos_ph;
  sincosf(theta, &sin_th, &cos_th);
  sincosf(phi, &sin_ph, &cos_ph);
  const double ct = cos_th, st = sin_th, cp = cos_ph, sp = sin_ph;
  // N and L: (re, im)
  const double nt_r = acc[0] * ct * cp + acc[2] * ct * sp - acc[4] * st, nt_i = acc[1] * ct * cp + acc[3] * ct * sp - acc[5] * st;
  const double np_r = -acc[0] * sp + acc[2] * cp, np_i = -acc[1] * sp + acc[3] * cp;
  const double lt_r = acc[6] * ct * cp + acc[8] * ct * sp - acc[10] * st, lt_i = acc[7] * ct * cp + acc[9] * ct * sp - acc[11] * st;
  const double lp_r = -acc[6] * sp + acc[8] * cp, lp_i = -acc[7] * sp + acc[9] * cp;
  const double k = double(beta) / (4.0 * 3.14159265358979323846);
  // E_theta = -j k (L_phi + eta0 N_theta); E_phi = j k (L_theta - eta0 N_phi)
  const double et_r = lp_r + kEta0 * nt_r, et_i = lp_i + kEta0 * nt_i;
  const double ep_r = lt_r - kEta0 * np_r, ep_i = lt_i - kEta0 * np_i;
  out[o] = make_float2(float(k * et_i), float(-k * et_r));
  out[half + o] = make_float2(float(-k * ep_i), float(k * ep_r));
}

// The moments of the cells of part blockIdx.z (cells part * per .. + per) for
// 128 directions of frequency blockIdx.y: sums[f][part][12][directions], or
// with one part the far field itself.
__global__ void __launch_bounds__(kNf2ffThreads)
nf2ff_kernel(const float* __restrict__ data, const Nf2ffFaceDev* __restrict__ faces, int n_faces, int n_cells, int per,
             const float* __restrict__ beta, const float* __restrict__ theta, int n_theta,
             const float* __restrict__ phi, int n_phi, double* __restrict__ sums, float2* __restrict__ out) {
  __shared__ __align__(16) Nf2ffCell s_cells[kNf2ffThreads];
  const int f = blockIdx.y, n_freq = gridDim.y, n_dir = n_theta * n_phi;
  const int a = blockIdx.x * kNf2ffThreads + threadIdx.x;
  const bool live = a < n_dir;
  const int th = live ? a / n_phi : 0, ph = live ? a % n_phi : 0;
  float sin_th, cos_th, sin_ph, cos_ph;
  sincosf(theta[th], &sin_th, &cos_th);
  sincosf(phi[ph], &sin_ph, &cos_ph);
  const float u = sin_th * cos_ph, v = sin_th * sin_ph, w = cos_th;
  const float b = beta[f];
  double acc[12] = {0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0};  // Jx Jy Jz Mx My Mz, (re, im)
  const int c_end = min(n_cells, (int(blockIdx.z) + 1) * per);
  for (int c0 = int(blockIdx.z) * per; c0 < c_end; c0 += kNf2ffThreads) {
    const int nc = min(kNf2ffThreads, c_end - c0);
    __syncthreads();
    if (int(threadIdx.x) < nc) {
      const int c = c0 + threadIdx.x;
      int k = 0;
      while (k + 1 < n_faces && c >= faces[k + 1].first) ++k;
      const Nf2ffFaceDev F = faces[k];
      const int i = c - F.first;
      const float r0 = data[F.r0 + i], r1 = data[F.r1 + i], ds = data[F.ds + i];
      Nf2ffCell& s = s_cells[threadIdx.x];
      s.pos = F.axis == 0 ? make_float4(F.pos, r0, r1, 0.f)
              : F.axis == 1 ? make_float4(r0, F.pos, r1, 0.f) : make_float4(r0, r1, F.pos, 0.f);
#pragma unroll
      for (int q = 0; q < 6; ++q) {
        const int64_t o = (q < 3 ? F.J : F.M) + 2 * ((int64_t(q % 3) * n_freq + f) * F.cells + i);
        const float re = ds * data[o], im = ds * data[o + 1];
        s.cur[q] = make_float4(re, re, im, im);
      }
    }
    __syncthreads();
    for (int k0 = 0; k0 < nc; k0 += kNf2ffRun) {
      unsigned long long part[6] = {0, 0, 0, 0, 0, 0};
      for (int k = k0; k < min(nc, k0 + kNf2ffRun); ++k) {
        const Nf2ffCell& c = s_cells[k];
        float s, co;
        sincosf(b * (u * c.pos.x + v * c.pos.y + w * c.pos.z), &s, &co);
        const unsigned long long e = pack2(co, s), je = pack2(-s, co);  // exp and j exp
#pragma unroll
        for (int q = 0; q < 6; ++q) {  // (re + j im) exp
          const ulonglong2 z = *reinterpret_cast<const ulonglong2*>(&c.cur[q]);
          part[q] = ffma2(z.y, je, ffma2(z.x, e, part[q]));
        }
      }
#pragma unroll
      for (int q = 0; q < 6; ++q) {
        float re, im;
        unpack2(part[q], re, im);
        acc[2 * q] += double(re);
        acc[2 * q + 1] += double(im);
      }
    }
  }
  if (!live) return;
  if (gridDim.z == 1) {
    nf2ff_field(acc, b, theta[th], phi[ph], out, size_t(f) * n_dir + a, size_t(n_freq) * n_dir);
    return;
  }
  double* const o = sums + (int64_t(f) * gridDim.z + blockIdx.z) * 12 * n_dir + a;
#pragma unroll
  for (int q = 0; q < 12; ++q) o[int64_t(q) * n_dir] = acc[q];
}

// Adds the parts and forms the far field: a block takes 16 directions of one
// frequency, eight threads each, thread g the parts g, g + 8, ... (one thread
// per direction took 99 us for 43 parts of 1,729 directions).
constexpr int kNf2ffGroups = 8;

__global__ void __launch_bounds__(kNf2ffThreads)
nf2ff_field_kernel(const double* __restrict__ sums, int n_parts, const float* __restrict__ beta,
                   const float* __restrict__ theta, int n_theta, const float* __restrict__ phi, int n_phi,
                   float2* __restrict__ out) {
  constexpr int kDirs = kNf2ffThreads / kNf2ffGroups;
  __shared__ double s_acc[kNf2ffGroups][12][kDirs];
  const int f = blockIdx.y, n_freq = gridDim.y, n_dir = n_theta * n_phi;
  const int d = threadIdx.x % kDirs, g = threadIdx.x / kDirs;
  const int a = blockIdx.x * kDirs + d;
  double acc[12] = {0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0, 0};
  if (a < n_dir)
    for (int p = g; p < n_parts; p += kNf2ffGroups) {
      const double* const o = sums + (int64_t(f) * n_parts + p) * 12 * n_dir + a;
#pragma unroll
      for (int q = 0; q < 12; ++q) acc[q] += o[int64_t(q) * n_dir];
    }
#pragma unroll
  for (int q = 0; q < 12; ++q) s_acc[g][q][d] = acc[q];
  __syncthreads();
  if (g > 0 || a >= n_dir) return;
  for (int k = 1; k < kNf2ffGroups; ++k)
#pragma unroll
    for (int q = 0; q < 12; ++q) acc[q] += s_acc[k][q][d];
  nf2ff_field(acc, beta[f], theta[a / n_phi], phi[a % n_phi], out, size_t(f) * n_dir + a, size_t(n_freq) * n_dir);
}

}  // namespace rfn

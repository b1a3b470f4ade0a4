// C ABI and runtime of the B200 FDTD engine (declarations in include/fdtd.h).
//
// Replaces SolverFDTD::solver_run_cu (rfnetwork/core/src/solver.cu:546-1143):
// instead of 48 device arrays and four kernel launches per step on the
// default stream, each simulation keeps its fields double-buffered in an
// x-fastest layout, its coefficients as a 16-bit material index plus a row
// table, and the whole time loop is one kernel launch per step (plus a DFT
// pass every kDftChunk steps), captured once into a CUDA graph and replayed.
#include <cuda_runtime.h>

#include <algorithm>
#include <array>
#include <chrono>
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <map>
#include <memory>
#include <mutex>
#include <shared_mutex>
#include <string>
#include <thread>
#include <unordered_set>
#include <utility>
#include <vector>

#include "../../include/fdtd.h"
#include "fdtd_compile.h"
#include "fdtd_kernels.cuh"
#include "fdtd_adjoint.cuh"
#include "fdtd_nf2ff.cuh"
#include "fdtd_step_stream.cuh"
#include "fdtd_half.cuh"
#include "fdtd_adjoint_half.cuh"
#include "fdtd_resident.cuh"
#include "fdtd_adjoint_stream.cuh"
#include <cudaTypedefs.h>

using namespace rfn;

namespace {

constexpr int kDftChunk = 256;  // steps between DFT accumulation passes
constexpr int kResidentSteps = 16 * kDftChunk;  // most steps of one launch of the resident kernel
constexpr int kMaxProbes = 1 << 20;
constexpr int kMaxMonitors = 50;  // MAX_MONITORS, rfnetwork/core/inc/solver.h:15
static_assert(kMaxMonitors <= kResMonitors, "monitor table of the resident kernel");

// error text of the calls without a handle, kept per calling thread
thread_local std::string g_error;

struct CudaError {
  cudaError_t code;
  std::string where;
};

#define CK(call)                                                   \
  do {                                                             \
    cudaError_t e_ = (call);                                       \
    if (e_ != cudaSuccess) throw CudaError{e_, #call};             \
  } while (0)

struct ArgError {
  int code;
  std::string msg;
};

// The engine's device memory comes from a stream-ordered pool of its own per
// device that keeps freed blocks (release threshold: never), so the ~1 GB of
// one solve is reused by the next instead of being unmapped and mapped again
// (which otherwise adds a few hundred ms to some solves).
cudaMemPool_t engine_pool() {
  static std::mutex mu;
  static cudaMemPool_t pools[64] = {};
  int dev = 0;
  CK(cudaGetDevice(&dev));
  if (dev < 0 || dev >= 64) throw ArgError{FDTD_ERR_CUDA, "device index out of range"};
  std::lock_guard<std::mutex> lock(mu);
  if (!pools[dev]) {
    cudaMemPoolProps props{};
    props.allocType = cudaMemAllocationTypePinned;
    props.location.type = cudaMemLocationTypeDevice;
    props.location.id = dev;
    CK(cudaMemPoolCreate(&pools[dev], &props));
    uint64_t keep = UINT64_MAX;
    CK(cudaMemPoolSetAttribute(pools[dev], cudaMemPoolAttrReleaseThreshold, &keep));
  }
  return pools[dev];
}

// A wait for the whole device and a capture in another thread spoil each other:
// the wait is refused and the capture ends invalid. Captures share this lock, waits
// take it alone.
std::shared_mutex& capture_mutex() {
  static std::shared_mutex m;
  return m;
}

cudaError_t device_wait() {
  std::unique_lock<std::shared_mutex> lock(capture_mutex());
  const cudaError_t e = cudaDeviceSynchronize();
  if (e != cudaSuccess) cudaGetLastError();  // (the next launch's check is not to find it)
  return e;
}

// An instantiated graph (null: none).
struct Graph {
  cudaGraphExec_t exec = nullptr;
  Graph() = default;
  explicit Graph(cudaGraphExec_t e) : exec(e) {}
  Graph(Graph&& o) noexcept : exec(std::exchange(o.exec, nullptr)) {}
  Graph& operator=(Graph&& o) noexcept {
    std::swap(exec, o.exec);
    return *this;
  }
  ~Graph() {
    if (exec) cudaGraphExecDestroy(exec);
  }
};

// What f launches on the stream it is given, as a graph; none when the capture was
// ended by a wait for the device outside this library.
template <typename F>
Graph capture(F&& f) {
  cudaStream_t cap;
  cudaGraph_t g = nullptr;
  CK(cudaStreamCreateWithFlags(&cap, cudaStreamNonBlocking));
  std::shared_lock<std::shared_mutex> lock(capture_mutex());
  try {
    CK(cudaStreamBeginCapture(cap, cudaStreamCaptureModeThreadLocal));
    f(cap);
    CK(cudaStreamEndCapture(cap, &g));
  } catch (...) {
    // (an ended capture shows as different errors in what is captured after it)
    cudaStreamCaptureStatus status = cudaStreamCaptureStatusNone;
    cudaStreamIsCapturing(cap, &status);
    const cudaError_t end = cudaStreamEndCapture(cap, &g);
    if (g) cudaGraphDestroy(g);
    cudaStreamDestroy(cap);
    cudaGetLastError();
    if (status == cudaStreamCaptureStatusInvalidated || end == cudaErrorStreamCaptureInvalidated) return Graph();
    throw;
  }
  lock.unlock();
  cudaStreamDestroy(cap);
  cudaGraphExec_t exec = nullptr;
  const cudaError_t e = cudaGraphInstantiate(&exec, g, 0);
  cudaGraphDestroy(g);
  CK(e);
  return Graph(exec);
}

template <typename T>
struct DevBuf {
  T* p = nullptr;
  size_t n = 0;    // elements in use
  size_t cap = 0;  // elements allocated
  void alloc(size_t count) {
    free();
    if (count) {
      CK(cudaMallocFromPoolAsync(reinterpret_cast<void**>(&p), count * sizeof(T), engine_pool(), 0));
      CK(cudaStreamSynchronize(0));  // usable on every stream from here
    }
    n = cap = count;
  }
  // Like alloc, but keeps the allocation when it already holds `count`.
  void reserve(size_t count) {
    if (count > cap) alloc(count);
    n = count;
  }
  void free() {
    // no stream may still use it (cudaFree would wait the same way); where the wait is
    // refused, because code outside this library captures a stream, the block stays out
    // of use
    if (p && device_wait() == cudaSuccess) {
      cudaFreeAsync(p, 0);
      cudaStreamSynchronize(0);
    }
    p = nullptr;
    n = cap = 0;
  }
  ~DevBuf() { free(); }
  DevBuf() = default;
  DevBuf(const DevBuf&) = delete;
  DevBuf& operator=(const DevBuf&) = delete;
};

struct Monitor {
  int field, axis, position, n_step, n_freq;
  std::vector<float> phase;  // interleaved complex64 rows
  int n_phase_rows;
  int n1, n2;
  size_t out_bytes(int nt) const {
    const size_t plane = size_t(n1) * n2;
    return n_freq ? plane * n_freq * 8 : plane * size_t(nt / n_step + 1) * 4;
  }
};

int threads_for_host() {
  unsigned h = std::thread::hardware_concurrency();
  return int(std::max(1u, std::min(h, 32u)));
}

}  // namespace

// Kernel selection of an engine: the plain-load kernel (one cell per thread)
// or the TMA-pipelined streaming kernel (tile height, plane slots), and the z chunk.
struct KernelConfig {
  int variant = 1;  // 0 plain loads, 1 TMA streaming, 2 resident, 3 half steps (the engine's own choice)
  int ty = 0;       // tile height; 0 (with variant 1): autotuned (ty, stages, zchunk); resident: bricks along x;
                    // half steps: threads per block
  int stages = 6;   // streaming: shared-memory plane slots; resident: bricks along y
  int zchunk = 0;   // 0: pick from the grid size; resident: bricks along z
  int one_list = 0; // streaming: every tile through the general instantiation (no plain-tile kernel beside it);
                    // resident: weight of a layer's plane, percent of another's
};

// Step-kernel shapes the autotuner times, (variant, tile height, plane slots,
// z chunk, one tile list), and its choices per set of grid sizes
// (process-wide). With one list the plain tiles run in the general kernel's
// interior path: one launch per step instead of two side by side, which can
// pay on grids whose step time is mostly launch and pipeline latency.
constexpr int kTuneCandidates[][5] = {{1, 8, 6, 0, 0}, {1, 8, 8, 0, 0},  {1, 8, 4, 0, 0}, {1, 8, 6, 32, 0},
                                      {1, 12, 4, 0, 0}, {1, 6, 6, 0, 0}, {1, 4, 6, 0, 0}, {1, 4, 6, 16, 0},
                                      {1, 8, 6, 4, 0}, {1, 4, 6, 4, 0},  {1, 8, 6, 0, 1}, {1, 8, 6, 4, 1},
                                      {1, 4, 6, 4, 1}, {3, 256, 0, 0, 0}, {3, 128, 0, 0, 0}};
using TuneChoice = std::array<int, 5>;
std::mutex g_tune_mutex;
std::map<std::vector<int>, TuneChoice> g_tune_cache;

// RFN_FDTD_ONE_LIST=1: explicit streaming shapes run every tile through the
// general kernel (the autotuner decides this by itself).
int one_list_env() {
  const char* v = std::getenv("RFN_FDTD_ONE_LIST");
  return v && std::atoi(v) != 0 ? 1 : 0;
}

KernelConfig default_config() {
  KernelConfig c;
  if (const char* v = std::getenv("RFN_FDTD_KERNEL"))
    c.variant = std::string(v) == "plain" ? 0 : std::string(v) == "half" ? 3 : 1;
  if (const char* v = std::getenv("RFN_FDTD_TY")) c.ty = std::atoi(v);
  if (const char* v = std::getenv("RFN_FDTD_STAGES")) c.stages = std::atoi(v);
  if (const char* v = std::getenv("RFN_FDTD_ZCHUNK")) c.zchunk = std::atoi(v);
  c.one_list = one_list_env();
  return c;
}

struct Engine;

struct fdtd_sim {
  int nx, ny, nz;
  std::vector<float> coef[kNumCoef];
  // borrowed caller arrays (fdtd_set_coefficient_view); null: coef[i] holds a copy
  const float* coef_view[kNumCoef] = {};
  bool have_coef[kNumCoef] = {};
  std::vector<ProbeSpec> probes;
  std::vector<std::vector<float>> probe_values;
  std::vector<Monitor> monitors;
  // DFT specification
  int n_series = 0, n_freq = 0;
  std::vector<int> series_start, term_probe;
  std::vector<double> term_weight, omega;

  // device state (valid when prepared)
  bool compiled = false;
  bool prepared = false;
  int prepared_nt = -1;
  int pitch = 0;
  size_t cells_padded = 0;
  CompiledGrid grid;
  SplitPlan split_plan;         // slab thicknesses and sparse slots of the split cells
  SplitDev split_geo{};         // store geometry (base pointers set when prepared)
  size_t split_buf_pairs = 0;   // split pairs per time buffer (all stores)
  DevBuf<float> fields;        // 2 x 6 field arrays
  DevBuf<float> splits;        // 2 x 12 split arrays (only when split cells exist)
  DevBuf<uint16_t> mat;
  DevBuf<float4> rows;
  DevBuf<int2> cell_probes;
  DevBuf<float> src, rec;
  DevBuf<int> is_src;
  DevBuf<int> d_series_start, d_term_probe;
  DevBuf<double> d_term_weight, d_omega;
  DevBuf<double2> dft_X;
  DevBuf<MonDev> d_mons;
  std::vector<std::unique_ptr<DevBuf<char>>> mon_out;
  std::vector<std::unique_ptr<DevBuf<float2>>> mon_phase;
  SimDev dev{};
  DevBuf<SimDev> d_dev;  // this simulation's descriptor alone (monitor kernel)

  std::unique_ptr<Engine> engine;  // batch of one for fdtd_run
  KernelConfig cfg = default_config();
  cudaStream_t ext_stream = nullptr;
  uint32_t dbg_wait_limit = kStreamWaitLimit;  // fdtd_set_debug
  int dbg_withhold = -1;
  std::string err;
  fdtd_stats stats{};
  int64_t h2d_bytes = 0, d2h_bytes = 0;  // bytes copied over PCIe/C2C by this simulation
  // What the last run kept for a gradient (fdtd_adjoint): adj_mode 1 = state
  // snapshots (fdtd_run_checkpointed), one per segment of ckpt_every steps:
  // the 6 field arrays of the time buffer the segment starts from, then (when
  // allocated) its 12 split arrays; adj_mode 2 = the forward history of the
  // gradient box at every step (fdtd_run_recorded), [nt][9][box cells].
  int adj_mode = 0;
  int ckpt_every = 0;
  int ckpt_nt = -1;
  DevBuf<float> ckpt;
  int adj_box[6] = {0, 0, 0, 0, 0, 0};
  DevBuf<float> hist;
  bool adj_in_batch = false;  // the recorded run was a batch run
  bool use_graph = true;      // fdtd_set_graph
  // table rows given to the cells of one box by fdtd_set_box_coefficients
  // (one per cell, after the compiled rows)
  int base_rows = 0;
  int box_rows_from = -1;
  int box_rows_box[6] = {0, 0, 0, 0, 0, 0};
  bool uploaded = false;  // host arrays were copied since the last wait for uploads
  int generation = 0;  // bumped whenever device buffers are reallocated
  int engine_gen = -1;  // generation the simulation's own engine was built on
};

int64_t box_cells(const int* b) { return int64_t(b[1] - b[0]) * (b[3] - b[2]) * (b[5] - b[4]); }

// dJ/d(record of probe p at step n), [P][nt], from dJ/dX of the device DFT
// (X_sf = sum over the series' terms (p, w) of w sum_n rec_p[n] e^{-i w_f n};
// with the gradient convention G = dJ/dRe X + i dJ/dIm X this is
// sum over the terms (series, p, w) of w sum_f (Re G_sf cos(w_f n) - Im G_sf sin(w_f n))).
std::vector<float> record_adjoints(const fdtd_sim* s, const double* dJdX, int nt) {
  const int P = int(s->probes.size());
  std::vector<float> radj(size_t(std::max(P, 1)) * nt, 0.f);
  std::vector<double> acc(static_cast<size_t>(nt));
  for (int se = 0; se < s->n_series; ++se) {
    std::fill(acc.begin(), acc.end(), 0.0);
    for (int f = 0; f < s->n_freq; ++f) {
      const double gr = dJdX[(size_t(se) * s->n_freq + f) * 2], gi = dJdX[(size_t(se) * s->n_freq + f) * 2 + 1];
      if (gr == 0.0 && gi == 0.0) continue;
      const double om = s->omega[size_t(f)];
      for (int n = 0; n < nt; ++n) acc[size_t(n)] += gr * std::cos(om * n) - gi * std::sin(om * n);
    }
    for (int t = s->series_start[size_t(se)]; t < s->series_start[size_t(se) + 1]; ++t) {
      const int p = s->term_probe[size_t(t)];
      const double w = s->term_weight[size_t(t)];
      for (int n = 0; n < nt; ++n) radj[size_t(p) * nt + n] += float(w * acc[size_t(n)]);
    }
  }
  return radj;
}

// Host-to-device copy that counts its bytes on the simulation.
void h2d(fdtd_sim* s, void* dst, const void* src, size_t bytes) {
  CK(cudaMemcpy(dst, src, bytes, cudaMemcpyHostToDevice));
  s->h2d_bytes += int64_t(bytes);
  s->uploaded = true;
}

void d2h(fdtd_sim* s, void* dst, const void* src, size_t bytes) {
  CK(cudaMemcpy(dst, src, bytes, cudaMemcpyDeviceToHost));
  s->d2h_bytes += int64_t(bytes);
}

// Waits for the uploads issued so far. A copy from pageable memory returns when
// the host buffer may be reused, before its last bytes are on the device, and
// the engine's streams don't wait for the legacy stream by themselves: this
// comes between the uploads and the first kernel on another stream.
void uploads_done() { CK(cudaStreamSynchronize(0)); }

// Lets a kernel be launched with as much dynamic shared memory as a block can have.
// The limit belongs to the function, not to a launch: set to what one engine uses,
// it made the launches of another engine that uses more fail.
void allow_shared(const void* fn) {
  int dev = 0, most = 0;
  CK(cudaGetDevice(&dev));
  CK(cudaDeviceGetAttribute(&most, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev));
  cudaFuncAttributes a{};
  CK(cudaFuncGetAttributes(&a, fn));
  CK(cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, most - int(a.sharedSizeBytes)));
}

using StreamKernelFn = void (*)(const SimDev, const SimDev*, const StreamTile*, int, int, unsigned*, unsigned, int*, int, int,
                                uint32_t, int);

// One tile height of the streaming step kernel: the general and the
// plain-tile instantiation, and the bytes of its exchange buffers, plane
// slots and split regions.
struct StreamVariant {
  int ty, threads, min_blocks, plain_blocks;
  uint32_t xch_bytes, main_bytes, split_bytes;
  StreamKernelFn fn, plain_of[2], plain_most;  // plain_of: several simulations, one
};

template <int TY>
StreamVariant stream_variant() {
  using G = StreamGeom<TY>;
  return StreamVariant{TY, G::THREADS, G::MIN_BLOCKS, G::PLAIN_BLOCKS, uint32_t(2 * G::XCH), G::MAIN, G::REGION,
                       &fdtd_step_stream_kernel<TY, kTilesAny, false>,
                       {&fdtd_step_stream_kernel<TY, kTilesPlain, false>, &fdtd_step_stream_kernel<TY, kTilesPlain, true>},
                       &fdtd_step_stream_kernel<TY, kTilesPlainMost, true>};
}

const std::vector<StreamVariant>& stream_variants() {
  static const std::vector<StreamVariant> v = {stream_variant<4>(), stream_variant<6>(), stream_variant<8>(),
                                               stream_variant<12>()};
  return v;
}

// The streaming kernel with tile height ty and `stages` plane slots (3..8).
const StreamVariant* find_stream_variant(int ty, int stages) {
  if (stages < 3 || stages > kSlotsMax) return nullptr;
  for (auto& v : stream_variants())
    if (v.ty == ty) return &v;
  return nullptr;
}

// Dynamic shared bytes of a streaming block with (at most) `want` plane
// slots and, when a simulation has split cells, four to six split regions,
// sized for the kernel's resident blocks per SM (or fewer blocks, when three
// plane slots and four regions do not fit beside that many); the slot and
// region counts it fits go to n_main / n_reg.
uint32_t stream_slots(const StreamVariant& v, int want, int resident, bool splits, int* n_main, int* n_reg) {
  constexpr uint32_t kSmemPerSm = 233472, kPerBlockReserve = 1024 + 512, kMaxPerBlock = 232448 - 512;
  const uint32_t split_min = splits ? kRegionsMin * v.split_bytes : 0;
  uint32_t budget = 0;
  for (int blocks = resident; blocks >= 1; --blocks) {
    budget = std::min(kSmemPerSm / blocks - kPerBlockReserve, kMaxPerBlock) - v.xch_bytes;
    if (budget >= 3 * v.main_bytes + split_min) break;
  }
  if (budget < 3 * v.main_bytes + split_min)
    throw ArgError{FDTD_ERR_LIMIT, "Streaming kernel's plane slots do not fit in shared memory."};
  const uint32_t m = std::min<uint32_t>(uint32_t(std::min(want, kSlotsMax)), (budget - split_min) / v.main_bytes);
  const uint32_t rg = splits ? std::min<uint32_t>(kRegionsMax, (budget - m * v.main_bytes) / v.split_bytes) : 0;
  *n_main = int(std::max<uint32_t>(m, 3));
  *n_reg = int(rg);
  return v.xch_bytes + uint32_t(*n_main) * v.main_bytes + rg * v.split_bytes;
}

// Whether a (variant, tile height, stages) triple names an instantiated kernel.
bool kernel_exists(int variant, int ty, int stages) {
  if (variant == 0) return true;
  if (variant == 1) return ty == 0 || find_stream_variant(ty, stages) != nullptr;
  return false;
}

PFN_cuTensorMapEncodeTiled_v12000 get_encode_fn() {
  static PFN_cuTensorMapEncodeTiled_v12000 fn = nullptr;
  if (!fn) {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    CK(cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q));
    if (q != cudaDriverEntryPointSuccess || !p) throw ArgError{FDTD_ERR_CUDA, "cuTensorMapEncodeTiled unavailable"};
    fn = reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(p);
  }
  return fn;
}

// Tiled tensor map over a field group of simulation s: dims (x, y, z) and,
// for rank 5, (component, buffer) with the given element strides.
// xmul = 2 for the split pairs, whose x rows hold 2 floats per cell.
void encode_map(CUtensorMap* m, const void* base, CUtensorMapDataType type, int elem, const fdtd_sim* s, int rank,
                int box_x, int box_y, int ncomp, size_t comp_stride, size_t buf_stride, int xmul = 1) {
  const cuuint64_t row = cuuint64_t(s->pitch) * xmul;
  const cuuint64_t dims[5] = {row, cuuint64_t(s->ny), cuuint64_t(s->nz), cuuint64_t(ncomp), 2};
  const cuuint64_t strides[4] = {row * elem, row * s->ny * elem,
                                 cuuint64_t(comp_stride) * elem, cuuint64_t(buf_stride) * elem};
  const cuuint32_t box[5] = {cuuint32_t(box_x), cuuint32_t(box_y), 1, cuuint32_t(ncomp), 1};
  const cuuint32_t estr[5] = {1, 1, 1, 1, 1};
  CUresult r = get_encode_fn()(m, type, cuuint32_t(rank), const_cast<void*>(base), dims, strides, box, estr,
                               CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE,
                               CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) throw ArgError{FDTD_ERR_CUDA, "cuTensorMapEncodeTiled failed: " + std::to_string(int(r))};
}

// Tensor maps of the streaming kernel (box widths of StreamGeom).
void encode_stream_maps(StreamMaps& m, const fdtd_sim* s, int ty) {
  std::memset(&m, 0, sizeof(m));
  const auto F = CU_TENSOR_MAP_DATA_TYPE_FLOAT32;
  const size_t N = s->cells_padded;
  encode_map(&m.E, s->fields.p, F, 4, s, 5, 36, ty + 1, 3, N, 6 * N);
  encode_map(&m.H, s->fields.p + 3 * N, F, 4, s, 5, 40, ty + 2, 3, N, 6 * N);
  if (s->splits.n) {
    // each slab store: x rows of 2 w floats (pairs interleaved), h rows, its
    // depth in planes, 6 pair components, 2 time buffers; boxes of 36 pairs
    // and the E (ty + 1) or H (ty) rows, 3 components
    const SplitDev& g = s->split_geo;
    for (int st = 0; st < 6; ++st) {
      if (!g.comp[st]) continue;
      const cuuint64_t w2 = cuuint64_t(2 * g.w[st]);
      const cuuint64_t dims[5] = {w2, cuuint64_t(g.h[st]), cuuint64_t(g.comp[st] / (int64_t(g.w[st]) * g.h[st])), 6,
                                  2};
      const cuuint64_t strides[4] = {w2 * 4, w2 * g.h[st] * 4, cuuint64_t(g.comp[st]) * 8,
                                     cuuint64_t(s->split_buf_pairs) * 8};
      const cuuint32_t estr[5] = {1, 1, 1, 1, 1};
      for (int k = 0; k < 2; ++k) {
        const cuuint32_t box[5] = {72, cuuint32_t(k == 0 ? ty + 1 : ty), 1, 3, 1};
        CUresult r = get_encode_fn()(k == 0 ? &m.Es[st] : &m.Hs[st], F, 5,
                                     reinterpret_cast<float2*>(s->splits.p) + g.off[st], dims, strides, box, estr,
                                     CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE,
                                     CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
        if (r != CUDA_SUCCESS)
          throw ArgError{FDTD_ERR_CUDA, "cuTensorMapEncodeTiled failed for a split store: " + std::to_string(int(r))};
      }
    }
  }
  encode_map(&m.ids, s->mat.p, CU_TENSOR_MAP_DATA_TYPE_UINT16, 2, s, 3, 40, ty + 1, 1, 0, 0);
}

// Everything one launch of the streaming kernel needs.
struct StreamClass {
  const StreamVariant* v = nullptr;
  StreamKernelFn fn = nullptr, fn_plain = nullptr;  // its kernels for one or several simulations
  SimDev one{};                      // the only simulation, a kernel parameter
  uint32_t ring = 0;                 // dynamic shared bytes: exchange buffers, plane slots, split slots
  int n_main = 0, n_reg = 0;
  std::vector<StreamTile> host_tiles;     // tiles with split-field or probe cells (general kernel)
  std::vector<StreamTile> host_tiles_p;   // plain tiles (plain-tile kernel, beside the general one)
  std::vector<StreamMaps> host_maps;
  DevBuf<StreamMaps> d_maps;
  DevBuf<SimDev> d_sims;
  DevBuf<StreamTile> d_tiles, d_tiles_p;
  DevBuf<unsigned> d_counter;        // tile counters: general list, plain list
  int n_tiles = 0, grid = 0;
  int n_tiles_p = 0, grid_p = 0, n_main_p = 0;
  uint32_t ring_p = 0;
  void reset() {
    v = nullptr;
    ring = ring_p = 0;
    host_tiles.clear();
    host_tiles_p.clear();
    d_tiles_p.free();
    n_tiles_p = grid_p = n_main_p = 0;
    host_maps.clear();
    d_maps.free();
    d_sims.free();
    d_tiles.free();
    d_counter.free();
    n_tiles = grid = 0;
  }
};

// Everything one launch of the resident kernel needs.
struct ResidentClass {
  ResGrid g{};
  int threads = 0, faces = 0, blocks = 0;
  uint32_t smem = 0;
  DevBuf<uint2> lists;               // E lists, H lists, E face words, H face words
  DevBuf<int4> count;                // per brick, and again for a test's launch that withholds faces
  DevBuf<uint16_t> stride, row_ids;
  DevBuf<unsigned long long> face;   // E faces, then H faces
  DevBuf<float2> far;                // pairs that do not fit in shared memory
  DevBuf<uint2> mon_list;
  DevBuf<int> mon_count;
  void reset() {
    blocks = 0;
    lists.free();
    count.free();
    stride.free();
    row_ids.free();
    face.free();
    far.free();
    mon_list.free();
    mon_count.free();
  }
};

// Launch shape of the half-step kernels.
struct HalfClass {
  int want = 0;             // threads per block asked for, within the kernels' bounds
  int threads = 0, seg = 0, rows = 0;
  dim3 grid;
  DevBuf<SimDev> d_sims;    // several simulations
  DevBuf<int4> d_blocks;
  DevBuf<CapSim> d_caps;    // per simulation, while a launch records histories
  DevBuf<int> d_boxes;      // per simulation, of segment replays
  void reset() {
    threads = 0;
    d_sims.free();
    d_blocks.free();
    d_caps.free();
    d_boxes.free();
  }
};

// A batch's members below so many cells step together in a plain run when there are
// at least so many of them; in a gradient any number; the most cells of such a part.
// Members of a gradient of so many cells and more share launches again.
struct BatchRule { size_t members; int64_t cells; };
constexpr BatchRule kBatchTogether[] = {{6, 90'000}, {5, 70'000}, {3, 50'000}};
constexpr int64_t kBatchSmallGradient = 256'000, kBatchLargeGradient = 3'500'000,
                  kBatchCells = 1'200'000;

// grids whose steps fork are launched from the host below so many cells, or when a
// monitor samples more often than every so many steps
constexpr int64_t kDirectCells = 2'000'000;
constexpr int kDirectSamples = 16;
constexpr int kDirectLaunches = 1000;  // of a run that the caller does not wait for

constexpr int kResFarRows = 128;  // table rows kept in shared memory before the last pairs
constexpr uint32_t kResSmemMax = 232448 - 4096;  // dynamic shared bytes beside the kernel's static arrays

struct Engine {
  std::vector<fdtd_sim*> sims;
  KernelConfig asked;      // as set by the caller (may leave the choice to the autotuner)
  KernelConfig cfg;        // the kernel in use
  StreamClass scls;        // streaming kernel
  // split cells of each simulation's boxes, while tiles are built (the same for every shape timed)
  std::vector<std::unique_ptr<GradedIndex>> split_index;
  ResidentClass res;       // resident kernel
  HalfClass half;          // half-step kernels
  DevBuf<SimDev> d_sims;   // plain kernel
  DevBuf<int4> d_tiles;    // plain kernel
  DevBuf<int> d_err;
  int n_tiles = 0;
  int grid = 0;
  int zchunk_used = 0;
  cudaStream_t own_stream = nullptr;
  cudaStream_t ext_stream = nullptr;
  Graph graph;
  int graph_nt = -1;
  cudaEvent_t ev0 = nullptr, ev1 = nullptr;
  cudaStream_t cap_stream = nullptr;                   // box-history captures beside the steps
  cudaEvent_t cap_fork = nullptr, cap_join = nullptr;
  cudaStream_t step_side = nullptr;                    // the plain-tile kernel beside the general one
  cudaEvent_t step_fork = nullptr, step_join = nullptr;
  cudaStream_t mon_stream = nullptr;                   // plane monitors beside the next step
  cudaEvent_t mon_fork = nullptr, mon_join = nullptr;
  cudaStream_t rep_stream = nullptr;                   // checkpointed adjoint: segment replays
  cudaEvent_t seg_done[2] = {nullptr, nullptr};        // replay of a segment into history half k & 1 done
  cudaEvent_t seg_free[2] = {nullptr, nullptr};        // its reversal done: the half may be refilled
  int64_t step_launches = 0, dft_launches = 0, adj_launches = 0;
  double adj_ms = 0;
  uint32_t wait_limit = kStreamWaitLimit;  // polls per mbarrier wait of the streaming kernel
  // test hook: plane the TMA kernels' producers never issue, or step in which the
  // resident kernel's first brick sends no E faces
  int withhold = -1;
  bool use_graph = true;  // replay the time loop as a captured CUDA graph
  int direct_nt = -1;     // steps of the last run whose launches came from the host
  bool uploaded = true;   // tables were copied since the last wait for uploads
  double last_ms = 0;
  double tune_ms = 0;      // host time of the autotuner's trial runs in the last tiling (0: cached choice)
  int tune_trials = 0;     // candidate shapes it timed
  bool timing_pending = false;

  cudaStream_t stream() const { return ext_stream ? ext_stream : own_stream; }

  void init() {
    if (!own_stream && !ext_stream) CK(cudaStreamCreateWithFlags(&own_stream, cudaStreamNonBlocking));
    if (!ev0) CK(cudaEventCreate(&ev0));
    if (!ev1) CK(cudaEventCreate(&ev1));
    if (!cap_stream) CK(cudaStreamCreateWithFlags(&cap_stream, cudaStreamNonBlocking));
    if (!cap_fork) CK(cudaEventCreateWithFlags(&cap_fork, cudaEventDisableTiming));
    if (!cap_join) CK(cudaEventCreateWithFlags(&cap_join, cudaEventDisableTiming));
    if (!rep_stream) {
      // the replays take SMs first as blocks retire; the reversal fills the rest
      int lo = 0, hi = 0;
      CK(cudaDeviceGetStreamPriorityRange(&lo, &hi));
      CK(cudaStreamCreateWithPriority(&rep_stream, cudaStreamNonBlocking, hi));
    }
    if (!mon_stream) CK(cudaStreamCreateWithFlags(&mon_stream, cudaStreamNonBlocking));
    if (!mon_fork) CK(cudaEventCreateWithFlags(&mon_fork, cudaEventDisableTiming));
    if (!mon_join) CK(cudaEventCreateWithFlags(&mon_join, cudaEventDisableTiming));
    if (!step_side) CK(cudaStreamCreateWithFlags(&step_side, cudaStreamNonBlocking));
    if (!step_fork) CK(cudaEventCreateWithFlags(&step_fork, cudaEventDisableTiming));
    if (!step_join) CK(cudaEventCreateWithFlags(&step_join, cudaEventDisableTiming));
    for (int h = 0; h < 2; ++h) {
      if (!seg_done[h]) CK(cudaEventCreateWithFlags(&seg_done[h], cudaEventDisableTiming));
      if (!seg_free[h]) CK(cudaEventCreateWithFlags(&seg_free[h], cudaEventDisableTiming));
    }
  }
  ~Engine() {
    if (ev0) cudaEventDestroy(ev0);
    if (ev1) cudaEventDestroy(ev1);
    if (cap_fork) cudaEventDestroy(cap_fork);
    if (cap_join) cudaEventDestroy(cap_join);
    if (cap_stream) cudaStreamDestroy(cap_stream);
    for (int h = 0; h < 2; ++h) {
      if (seg_done[h]) cudaEventDestroy(seg_done[h]);
      if (seg_free[h]) cudaEventDestroy(seg_free[h]);
    }
    if (rep_stream) cudaStreamDestroy(rep_stream);
    if (mon_fork) cudaEventDestroy(mon_fork);
    if (mon_join) cudaEventDestroy(mon_join);
    if (mon_stream) cudaStreamDestroy(mon_stream);
    if (step_fork) cudaEventDestroy(step_fork);
    if (step_join) cudaEventDestroy(step_join);
    if (step_side) cudaStreamDestroy(step_side);
    if (own_stream) cudaStreamDestroy(own_stream);
  }

  void reset_graph() {
    graph = Graph();
    graph_nt = direct_nt = -1;
  }

  // Waits for what this engine and its simulations uploaded, if anything.
  void wait_uploads() {
    bool any = uploaded;
    for (auto* s : sims) any = any || s->uploaded;
    if (!any) return;
    uploads_done();
    uploaded = false;
    for (auto* s : sims) s->uploaded = false;
  }

  void build_tiles() {
    reset_graph();
    uploaded = true;
    n_caps = 0;  // (a kept engine's last run may have recorded)
    cfg = asked;
    int dev = 0, n_sm = 148;
    CK(cudaGetDevice(&dev));
    CK(cudaDeviceGetAttribute(&n_sm, cudaDevAttrMultiProcessorCount, dev));
    if (!d_err.n) {
      d_err.alloc(1);
      CK(cudaMemset(d_err.p, 0, sizeof(int)));
    }
    if (cfg.variant != 0) {
      split_index.clear();
      if (cfg.variant == 1 && cfg.ty == 0)
        autotune(n_sm);
      else
        build_shape(n_sm);
      split_index.clear();
      return;
    }
    // plain kernel: 31 x 7 tiles, z cut into chunks
    std::vector<SimDev> devs;
    for (auto* s : sims) devs.push_back(s->dev);
    const std::vector<int4> tiles = plain_tiles(n_sm, cfg.zchunk, &zchunk_used);
    grid = int(tiles.size());
    d_sims.alloc(devs.size());
    CK(cudaMemcpy(d_sims.p, devs.data(), devs.size() * sizeof(SimDev), cudaMemcpyHostToDevice));
    d_tiles.alloc(tiles.size());
    CK(cudaMemcpy(d_tiles.p, tiles.data(), tiles.size() * sizeof(int4), cudaMemcpyHostToDevice));
    n_tiles = int(tiles.size());
  }

  // Tiles of the plain kernel and of the adjoint step kernel: 31 x kTileY
  // columns cut in z chunks, (simulation, x0 | y0 << 16, z0 | z1 << 16, 0),
  // about eight per SM over the whole set of simulations.
  std::vector<int4> plain_tiles(int n_sm, int zchunk, int* zlen_out = nullptr, int tx = kTileX, int ty = kTileY,
                                int per_sm = 8) {
    std::vector<int4> tiles;
    int64_t xy_tiles = 0;
    for (auto* s : sims) xy_tiles += int64_t((s->nx + tx - 1) / tx) * ((s->ny + ty - 1) / ty);
    const int64_t want = int64_t(n_sm) * per_sm;
    for (size_t i = 0; i < sims.size(); ++i) {
      fdtd_sim* s = sims[i];
      int chunks = int(std::max<int64_t>(1, (want + xy_tiles - 1) / std::max<int64_t>(xy_tiles, 1)));
      chunks = std::min(chunks, std::max(1, s->nz / 8));
      const int zlen = zchunk > 0 ? zchunk : (s->nz + chunks - 1) / chunks;
      if (zlen_out) *zlen_out = zlen;
      for (int z0 = 0; z0 < s->nz; z0 += zlen)
        for (int y0 = 0; y0 < s->ny; y0 += ty)
          for (int x0 = 0; x0 < s->nx; x0 += tx) {
            const int z1 = std::min(s->nz, z0 + zlen);
            tiles.push_back(make_int4(int(i), x0 | (y0 << 16), z0 | (z1 << 16), 0));
          }
    }
    return tiles;
  }

  // Tiles of the streaming kernel, bricks of the resident one or blocks of the
  // half-step kernels.
  void build_shape(int n_sm) {
    res.reset();
    scls.reset();
    half.reset();
    if (cfg.variant == 2)
      build_resident(n_sm);
    else if (cfg.variant == 3)
      build_half();
    else
      build_stream_tiles(n_sm);
  }

  // Whether the resident kernel may step these simulations at all: one grid,
  // nothing to do between two of its steps.
  bool resident_allowed() const {
    return sims.size() == 1 && sims[0]->adj_mode == 0;
  }

  // The cuts of a simulation into px x py x pz bricks, a cell plane of a layer
  // weighing `weight` percent of another; false when a brick would be empty.
  static bool resident_cuts(const fdtd_sim* s, int px, int py, int pz, int weight, ResPart& P) {
    const int n[3] = {s->nx, s->ny, s->nz}, parts[3] = {px, py, pz};
    P.px = px; P.py = py; P.pz = pz;
    for (int a = 0; a < 3; ++a) {
      if (parts[a] >= kResCuts || parts[a] > n[a]) return false;
      const int64_t lo = s->split_plan.t[2 * a], hi = s->split_plan.t[2 * a + 1], mid = n[a] - lo - hi;
      const int64_t wl = lo * weight, wm = mid * 100, all = wl + wm + hi * weight;
      P.most[a] = 0;
      for (int i = 0; i <= parts[a]; ++i) {
        // the first cell whose planes below weigh i / parts of all (the layers' weights cancel at 100)
        const int64_t w = all * i / parts[a];
        const int64_t c = w <= wl ? w / weight : w <= wl + wm ? lo + (w - wl) / 100 : lo + mid + (w - wl - wm) / weight;
        P.cut[a][i] = uint16_t(i == parts[a] ? n[a] : c);
        if (i > 0) {
          if (P.cut[a][i] <= P.cut[a][i - 1]) return false;
          P.most[a] = std::max(P.most[a], int(P.cut[a][i]) - int(P.cut[a][i - 1]));
        }
      }
    }
    return true;
  }

  // Partitions worth timing, (bricks along x, y, z, weight): per number of blocks
  // the one whose costliest brick costs least, with even cuts and with thinner
  // bricks in the layers. A brick's cost: its cells, 0.7 more per layer cell,
  // 0.75 per face cell; its memory from the layers the split plan found. Where
  // no partition fits, some pairs may stay in global memory. None when the fields
  // alone do not fit. Thinner bricks take grids that even cuts do not (125x46x86
  // cells with 8-cell layers: half steps 14.0, here 10.7 us per step; 133x44x88
  // 15.5 -> 11.4) and even out the time (55x140x47 8.6 -> 8.0 us).
  std::vector<std::array<int, 4>> resident_partitions(int n_sm, bool* far_used) const {
    std::vector<std::array<int, 4>> out;
    const fdtd_sim* s = sims[0];
    const int n[3] = {s->nx, s->ny, s->nz};
    const int* t = s->split_plan.t;
    struct Part { int len, layer; };  // cells of a brick along an axis, of these in a layer
    auto cost_of = [&](const ResPart& P, bool far) -> double {
      std::vector<Part> kinds[3];
      const int parts[3] = {P.px, P.py, P.pz};
      for (int a = 0; a < 3; ++a)
        for (int i = 0; i < parts[a]; ++i) {
          const int c0 = P.cut[a][i], c1 = P.cut[a][i + 1];
          const int layer = std::max(0, std::min(c1, t[2 * a]) - c0) + std::max(0, c1 - std::max(c0, n[a] - t[2 * a + 1]));
          bool seen = false;
          for (const auto& k : kinds[a]) seen = seen || (k.len >= c1 - c0 && k.layer >= layer);
          if (!seen) kinds[a].push_back({c1 - c0, layer});
        }
      double worst = 0;
      for (const auto& x : kinds[0])
        for (const auto& y : kinds[1])
          for (const auto& z : kinds[2]) {
            const int v = x.len * y.len * z.len;
            auto either = [](const Part& p, const Part& q) { return p.len * q.len - (p.len - p.layer) * (q.len - q.layer); };
            const int pairs = 2 * (x.len * either(y, z) + y.len * either(x, z) + z.len * either(x, y));
            double over = 0;  // pairs outside shared memory
            if (far) {
              const uint32_t fields = res_smem(x.len, y.len, z.len, 0) + kResFarRows * kResRowBytes;
              if (fields > kResSmemMax) return 1e300;
              over = std::max(0.0, pairs - double(kResSmemMax - fields) / 8);
            } else if (res_smem(x.len, y.len, z.len, pairs) > kResSmemMax) {
              return 1e300;
            }
            const int core = (x.len - x.layer) * (y.len - y.layer) * (z.len - z.layer);
            worst = std::max(worst, v + 0.7 * (v - core) + 0.25 * over + 0.75 * (x.len * y.len + x.len * z.len + y.len * z.len));
          }
      return worst;
    };
    const bool layers = t[0] + t[1] + t[2] + t[3] + t[4] + t[5] > 0;
    ResPart P;
    if (24 * int64_t(n[0]) * n[1] * n[2] > int64_t(n_sm) * kResSmemMax) return out;
    const int sizes[] = {n_sm, n_sm / 2, 32, 8, n_sm};
    for (int k = 0; k < 5; ++k)
      for (const int thin : {0, 1}) {
        const int most = sizes[k];
        const bool far = k == 4;  // only where no other fits
        if ((far && ((!out.empty() && !*far_used) || !layers)) || (thin && (!layers || most != n_sm))) continue;
        double best = 1e300;
        std::array<int, 4> pick{0, 0, 0, 0};
        for (int px = 1; px <= std::min(most, s->nx); ++px)
          for (int py = 1; px * py <= most && py <= s->ny; ++py)
            for (int pz = 1; px * py * pz <= most && pz <= s->nz; ++pz) {
              // (with fewer than three quarters of the blocks the next smaller `most` is at hand)
              if (4 * px * py * pz < 3 * most && most <= s->nx * s->ny * s->nz / 64) continue;
              for (const int w : {100, 125, 150}) {
                if ((w == 100) == (thin == 1) || !resident_cuts(s, px, py, pz, w, P)) continue;
                const double cost = cost_of(P, far);
                if (cost < best) {
                  best = cost;
                  pick = {px, py, pz, w};
                }
              }
            }
        if (pick[0] && std::find(out.begin(), out.end(), pick) == out.end()) {
          out.push_back(pick);
          *far_used = far;
        }
      }
    return out;
  }

  // The resident kernel's lists and launch shape for cfg's partition; a size
  // limit error when the bricks do not fit.
  void build_resident(int n_sm) {
    ResidentClass& c = res;
    fdtd_sim* s = sims[0];
    const int px = cfg.ty, py = cfg.stages, pz = cfg.zchunk, nb = px * py * pz;
    ResPart& P = c.g.part;
    if (nb > n_sm) throw ArgError{FDTD_ERR_LIMIT, "More bricks than SMs."};
    if (!resident_cuts(s, px, py, pz, cfg.one_list, P)) throw ArgError{FDTD_ERR_LIMIT, "More bricks than cells."};
    const int bx = P.most[0], by = P.most[1], bz = P.most[2];
    const int cells = bx * by * bz, nf = 2 * (by * bz + bx * bz + bx * by);
    if (ResBox{0, 0, 0, bx, by, bz, 0, 0, 0}.size() * int64_t(3) >= kResNone || res_smem(bx, by, bz, 0) > kResSmemMax)
      throw ArgError{FDTD_ERR_LIMIT, "Bricks do not fit in shared memory."};
    const int n_rows = int(s->grid.rows.size());
    c.count.alloc(2 * size_t(nb));
    DevBuf<int> map, nums, n_nums;
    map.alloc(size_t(nb) * n_rows);
    nums.alloc(size_t(nb) * kResScratch * cells);
    n_nums.alloc(size_t(nb));
    const ResScratch scratch{map.p, nums.p, n_rows, cells};
    CK(cudaMemset(map.p, 0xff, map.n * sizeof(int)));
    res_count_kernel<<<nb, 32>>>(s->dev, P, scratch, c.count.p, n_nums.p);
    CK(cudaGetLastError());
    std::vector<int4> cnt(static_cast<size_t>(nb));
    CK(cudaMemcpy(cnt.data(), c.count.p, cnt.size() * sizeof(int4), cudaMemcpyDeviceToHost));
    const int e_faces = std::exchange(cnt[0].x, 0);
    CK(cudaMemcpy(c.count.p + nb, cnt.data(), cnt.size() * sizeof(int4), cudaMemcpyHostToDevice));
    cnt[0].x = e_faces;
    int local = 0;
    uint32_t state = 0;
    for (int b = 0; b < nb; ++b) {
      const ResBox r = res_box(P, b);
      state = std::max(state, res_smem(r.bx, r.by, r.bz, cnt[size_t(b)].z));
      local = std::max(local, cnt[size_t(b)].w);
    }
    // the pairs that do not fit beside the fields and the first rows stay in global memory
    c.g.far = nullptr;
    c.g.far_cap = 0;
    if (state > kResSmemMax) {
      state = kResSmemMax - uint32_t(std::min(local, kResFarRows)) * kResRowBytes;
      for (int b = 0; b < nb; ++b) {
        const ResBox r = res_box(P, b);
        if (res_smem(r.bx, r.by, r.bz, 0) > state) throw ArgError{FDTD_ERR_LIMIT, "Bricks do not fit in shared memory."};
        c.g.far_cap = std::max(c.g.far_cap, cnt[size_t(b)].z - res_pair_cap(r, state));
      }
      c.far.alloc(size_t(nb) * c.g.far_cap);
      c.g.far = c.far.p;
    }
    c.g.state = state;
    const int row_cap = std::min<int>(local, int((kResSmemMax - state) / kResRowBytes));
    c.smem = state + uint32_t(row_cap) * kResRowBytes;
    const size_t nl = size_t(nb) * cells;
    c.lists.alloc(4 * nl);
    c.row_ids.alloc(std::max<size_t>(1, size_t(nb) * row_cap));
    c.stride.alloc(size_t(nb) * 64);
    c.face.alloc(size_t(2) * nb * nf);
    ResGrid& g = c.g;
    g.s = s->dev;
    g.cap = cells;
    g.row_cap = row_cap;
    g.e_list = c.lists.p;
    g.h_list = c.lists.p + nl;
    g.e_words = c.lists.p + 2 * nl;
    g.h_words = c.lists.p + 3 * nl;
    g.row_ids = c.row_ids.p;
    g.stride = c.stride.p;
    g.e_face = c.face.p;
    g.h_face = c.face.p + size_t(nb) * nf;
    g.face_cap = nf;
    g.err = d_err.p;
    g.mons = s->d_mons.p;
    g.n_mon = int(s->monitors.size());
    g.acc_f = g.acc_cap = 0;
    if (g.n_mon > 0) {
      std::vector<MonDev> mons;
      for (const auto& m : s->monitors)
        mons.push_back(MonDev{m.field, m.axis, m.position, m.n_step, m.n_freq, m.n1, m.n2, nullptr, nullptr});
      int most_el = 1;
      for (int b = 0; b < nb; ++b) {
        int el = 0;
        for (const auto& m : mons) el += res_mon_elements(m, res_box(P, b));
        most_el = std::max(most_el, el);
      }
      c.mon_list.alloc(size_t(nb) * most_el);
      c.mon_count.alloc(size_t(nb));
      g.mon_cap = most_el;
      g.mon_list = c.mon_list.p;
      // sums in shared memory when every monitor is a phasor monitor of the same
      // number of frequencies
      bool uniform = mons[0].n_freq > 0;
      for (const auto& m : mons) uniform = uniform && m.n_freq == mons[0].n_freq;
      if (uniform) {
        g.acc_f = mons[0].n_freq;
        g.acc_cap = std::min<int>(most_el, int((kResSmemMax - c.smem) / (8u * uint32_t(g.acc_f))));
        c.smem += uint32_t(g.acc_cap) * 8u * uint32_t(g.acc_f);
      }
      g.mon_count = c.mon_count.p;
      res_monitor_kernel<<<nb, 128>>>(P, s->d_mons.p, g.n_mon, most_el, c.mon_list.p, c.mon_count.p);
      CK(cudaGetLastError());
    }
    res_build_kernel<<<nb, 32>>>(s->dev, P, scratch, n_nums.p, cells, row_cap, c.lists.p, c.lists.p + nl,
                                 c.lists.p + 2 * nl, c.lists.p + 3 * nl, c.row_ids.p, c.stride.p);
    CK(cudaGetLastError());
    CK(cudaStreamSynchronize(0));
    // every thread the same number of cells, and room for the face values
    const int rounds = (cells + kResThreads - 1) / kResThreads;
    c.threads = std::max({64, ((cells + rounds - 1) / rounds + 31) / 32 * 32, ((nf + 3) / 4 + 31) / 32 * 32});
    if (c.threads > kResThreads) throw ArgError{FDTD_ERR_LIMIT, "Bricks have too many faces."};
    c.faces = (nf + c.threads - 1) / c.threads;
    c.blocks = nb;
    const void* fn = resident_fn();
    allow_shared(fn);
    int per_sm = 0;
    CK(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, fn, c.threads, c.smem));
    if (per_sm < 1) throw ArgError{FDTD_ERR_LIMIT, "Resident kernel does not fit on an SM."};
    n_tiles = grid = nb;
    zchunk_used = pz;
  }

  template <bool MON>
  const void* resident_variant() const {
    if (res.g.far) return reinterpret_cast<const void*>(&res_step_kernel<4, 1024, MON, true>);
    const bool small = res.threads <= 640;  // (more registers per thread)
    return res.faces <= 1   ? small ? reinterpret_cast<const void*>(&res_step_kernel<1, 640, MON, false>)
                                    : reinterpret_cast<const void*>(&res_step_kernel<1, 1024, MON, false>)
           : res.faces <= 2 ? small ? reinterpret_cast<const void*>(&res_step_kernel<2, 640, MON, false>)
                                    : reinterpret_cast<const void*>(&res_step_kernel<2, 1024, MON, false>)
           : small          ? reinterpret_cast<const void*>(&res_step_kernel<4, 640, MON, false>)
                            : reinterpret_cast<const void*>(&res_step_kernel<4, 1024, MON, false>);
  }
  const void* resident_fn() const { return res.g.n_mon > 0 ? resident_variant<true>() : resident_variant<false>(); }

  // Steps n0 .. n1-1 by the resident kernel; the face words are cleared before
  // a run's first launch (their tags are step numbers).
  void launch_resident(cudaStream_t st, int n0, int n1) {
    if (n0 == 0) CK(cudaMemsetAsync(res.face.p, 0, res.face.n * sizeof(unsigned long long), st));
    res.g.s = sims[0]->dev;
    // (its polls do not sleep and take a quarter of a microsecond: eight for one of
    // the TMA waits', so that a limit bounds both to about the same time)
    res.g.wait_limit = uint32_t(std::min<uint64_t>(uint64_t(wait_limit) * 8, UINT32_MAX));
    auto launch = [&](int a, int b, const int4* count) {
      if (a >= b) return;
      res.g.count = count;
      void* args[] = {&res.g, &a, &b};
      CK(cudaLaunchCooperativeKernel(resident_fn(), dim3(unsigned(res.blocks)), dim3(unsigned(res.threads)), args,
                                     res.smem, st));
    };
    const int4* const c = res.count.p;
    if (withhold < n0 || withhold >= n1) {
      launch(n0, n1, c);
      return;
    }
    launch(n0, withhold, c);
    launch(withhold, withhold + 1, c + res.blocks);  // (the counts with which brick 0 sends no E faces)
    launch(withhold + 1, n1, c);
  }

  // Threads per row piece and rows per block of half-step blocks of at most t
  // threads over rows of nx cells.
  static void half_shape(int nx, int ny, int t, int* seg, int* rows) {
    if (nx > t) {
      const int pieces = (nx + t - 1) / t;
      *seg = std::min(t, ((nx + pieces - 1) / pieces + 31) / 32 * 32);
      *rows = 1;
    } else {
      *seg = nx;
      *rows = std::min(std::max(1, t / nx), ny);
    }
  }

  // Blocks over every cell of every simulation, of the size around `want`
  // threads that leaves the fewest idle over all grids; returns that size.
  int half_blocks(int want, std::vector<int4>& blocks, int deep = 1) const {
    double best = -1.0;
    int threads = want;
    for (int t = std::max(64, want / 2); t <= kHalfThreads; t += 32) {
      double used = 0, all = 0;
      for (auto* s : sims) {
        int seg, rows;
        half_shape(s->nx, s->ny, t, &seg, &rows);
        used += double(s->nx) * s->ny * s->nz;
        all += double((s->nx + seg - 1) / seg) * ((s->ny + rows - 1) / rows) * s->nz * t;
      }
      if (used / all > best) {
        best = used / all;
        threads = t;
      }
    }
    for (size_t i = 0; i < sims.size(); ++i) {
      const fdtd_sim* s = sims[i];
      int seg, rows;
      half_shape(s->nx, s->ny, threads, &seg, &rows);
      for (int z = 0; z < s->nz; z += deep)
        for (int y0 = 0; y0 < s->ny; y0 += rows)
          for (int x0 = 0; x0 < s->nx; x0 += seg)
            blocks.push_back(make_int4(int(i), x0 | (rows << 16), y0, z | (seg << 16)));
    }
    if (blocks.size() > size_t(INT_MAX)) throw ArgError{FDTD_ERR_LIMIT, "Too many half-step blocks."};
    return threads;
  }

  void build_half() {
    HalfClass& c = half;
    const int want = c.want = std::min(std::max(cfg.ty, 64), kHalfThreads) / 32 * 32;
    if (sims.size() == 1) {
      const fdtd_sim* s = sims[0];
      half_shape(s->nx, s->ny, want, &c.seg, &c.rows);
      c.threads = (c.seg * c.rows + 31) / 32 * 32;
      c.grid = dim3(unsigned((s->nx + c.seg - 1) / c.seg), unsigned((s->ny + c.rows - 1) / c.rows), unsigned(s->nz));
      n_tiles = grid = int(std::min<int64_t>(int64_t(c.grid.x) * c.grid.y * c.grid.z, INT_MAX));
    } else {
      std::vector<int4> blocks;
      std::vector<SimDev> devs;
      for (auto* s : sims) devs.push_back(s->dev);
      c.threads = half_blocks(want, blocks);
      c.grid = dim3(unsigned(blocks.size()));
      c.d_sims.alloc(devs.size());
      CK(cudaMemcpy(c.d_sims.p, devs.data(), devs.size() * sizeof(SimDev), cudaMemcpyHostToDevice));
      c.d_blocks.alloc(blocks.size());
      CK(cudaMemcpy(c.d_blocks.p, blocks.data(), blocks.size() * sizeof(int4), cudaMemcpyHostToDevice));
      n_tiles = grid = int(blocks.size());
    }
    zchunk_used = 1;
  }

  // Per simulation of the engine: what the E launches record (all-zero: nothing).
  void half_captures(const std::vector<CapSim>& caps) {
    if (caps.empty()) return;
    half.d_caps.reserve(caps.size());
    CK(cudaMemcpy(half.d_caps.p, caps.data(), caps.size() * sizeof(CapSim), cudaMemcpyHostToDevice));
  }

  template <typename... A>
  static void launch_dependent(void (*fn)(A...), dim3 grid, int threads, cudaStream_t st, A... args) {
    cudaLaunchConfig_t lc{};
    lc.gridDim = grid;
    lc.blockDim = dim3(unsigned(threads));
    lc.stream = st;
    cudaLaunchAttribute at{};
    at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at.val.programmaticStreamSerializationAllowed = 1;
    lc.attrs = &at;
    lc.numAttrs = 1;
    CK(cudaLaunchKernelEx(&lc, fn, args...));
  }

  // One half of step n (E, or H) on st. cap: the E launch writes the box
  // histories of half.d_caps at slot n - n0. reach >= 0: only the cells that
  // half.d_boxes' boxes need when `reach` more cells around them have to be right.
  void launch_half(cudaStream_t st, int n, bool h_side, bool cap, int n0 = 0, int reach = -1) {
    HalfClass& c = half;
    const bool one = sims.size() == 1;
    HalfLaunch L{};
    L.n = n;
    dim3 grid = c.grid;
    int threads = c.threads;
    L.lo = reach + (h_side ? 0 : 1);  // H needs E of the -1 neighbours
    L.hi = reach;
    int w[3] = {1, 1, 1};  // the largest region along each axis
    for (size_t i = 0; i < sims.size() && reach >= 0; ++i) {
      const int* b = &rep_boxes[6 * i];
      const int nn[3] = {sims[i]->nx, sims[i]->ny, sims[i]->nz};
      for (int a = 0; a < 3; ++a)
        w[a] = std::max(w[a], std::min(nn[a], b[2 * a + 1] + L.hi) - std::max(0, b[2 * a] - L.lo));
    }
    if (reach >= 0 && int64_t(w[2]) * int64_t(sims.size()) <= 65535) {
      L.boxes = c.d_boxes.p;
      half_shape(w[0], w[1], c.want, &L.seg, &L.rows);
      L.planes = w[2];
      threads = (L.seg * L.rows + 31) / 32 * 32;
      grid = dim3(unsigned((w[0] + L.seg - 1) / L.seg), unsigned((w[1] + L.rows - 1) / L.rows),
                  unsigned(w[2]) * unsigned(sims.size()));
    } else {
      L.blocks = one ? nullptr : c.d_blocks.p;
      L.seg = c.seg;
      L.rows = c.rows;
    }
    const SimDev* ds = c.d_sims.p;
    const CapSim* dc = c.d_caps.p;
    auto fn = h_side ? (one ? &half_step_kernel<true, true, false> : &half_step_kernel<true, false, false>)
              : cap  ? (one ? &half_step_kernel<false, true, true> : &half_step_kernel<false, false, true>)
                     : (one ? &half_step_kernel<false, true, false> : &half_step_kernel<false, false, false>);
    launch_dependent(fn, grid, threads, st, sims[0]->dev, L, ds, dc, n0);
  }

  // Time buffer that holds the state before step n.
  int state_buf(int n) const { return cfg.variant >= 2 ? 0 : n & 1; }

  // Picks the step kernel and its shape for this set of grids: each candidate
  // runs a few time steps on the simulations themselves, with the monitors and the
  // box histories that these keep (all is cleared or written again by the next
  // run), the fastest is kept and remembered for the same grid sizes and the same
  // work beside the steps. A grid whose state fits in shared memory takes the
  // resident kernel, whose partitions are timed (from 24x20x16 to 120x110x80
  // cells it takes a third to three quarters of the streaming kernels' time per
  // step, the least gain at the largest that fits); the others the streaming
  // one.
  void autotune(int n_sm) {
    tune_ms = 0;
    tune_trials = 0;
    if (resident_allowed()) {
      if (tune(n_sm, {}, 2)) return;
    }
    std::vector<TuneChoice> cand;
    for (const auto& c : kTuneCandidates) cand.push_back({c[0], c[1], c[2], c[3], c[4]});
    tune(n_sm, cand, 1);
  }

  // Times the candidates (given, or the resident kernel's partitions) and builds
  // the best one; false when none fits.
  bool tune(int n_sm, const std::vector<TuneChoice>& given, int variant) {
    std::vector<int> key{variant};
    int nt_min = 1 << 30;
    for (auto* s : sims) {
      key.insert(key.end(), {s->nx, s->ny, s->nz});
      nt_min = std::min(nt_min, s->prepared_nt);
    }
    // box histories, and the monitors' elements per step and cell in octaves: kernels
    // differ in what these cost them (the resident kernel samples inside, the half
    // steps write the histories themselves and wait for the samples)
    double sampled = 0, cells = 0;
    bool recorded = false;
    for (auto* s : sims) {
      recorded = recorded || s->adj_mode == 2;
      cells += double(s->nx) * s->ny * s->nz;
      for (const auto& m : s->monitors) sampled += double(m.n1) * m.n2 * std::max(1, m.n_freq) / m.n_step;
    }
    key.push_back(recorded);
    key.push_back(sampled > 0 ? int(std::floor(std::log2(sampled / cells))) : INT_MIN);
    // (what fits in shared memory depends on the layers)
    if (variant == 2) key.insert(key.end(), sims[0]->split_plan.t, sims[0]->split_plan.t + 6);
    const KernelConfig auto_cfg = cfg;
    std::vector<TuneChoice> cand = given;
    auto build = [&](const TuneChoice& c) -> bool {
      cfg.variant = c[0];
      cfg.ty = c[1];
      cfg.stages = c[2];
      cfg.zchunk = c[3];
      cfg.one_list = c[4];
      try {
        build_shape(n_sm);
        build_caps();
      } catch (const ArgError& e) {
        cfg = auto_cfg;
        if (e.code != FDTD_ERR_LIMIT) throw;
        return false;  // this shape does not fit these grids
      }
      return true;
    };
    bool cached = false;
    TuneChoice best{};
    {
      std::lock_guard<std::mutex> lock(g_tune_mutex);
      auto it = g_tune_cache.find(key);
      if (it != g_tune_cache.end()) {
        cached = true;
        best = it->second;
      }
    }
    if (cached && best[0] < 0) return false;  // nothing fitted
    if (cached && build(best)) return true;  // (a model of the same size may hold more split cells)
    if (variant == 2)
    {
      bool far = false;
      for (const auto& p : resident_partitions(n_sm, &far)) cand.push_back({2, p[0], p[1], p[2], p[3]});
      // where pairs stay in global memory the other kernels may be faster
      if (far && !cand.empty()) cand.insert(cand.end(), {{3, 128, 0, 0, 0}, {1, 8, 6, 0, 0}, {1, 12, 4, 0, 0}});
    }
    // (a launch of the resident kernel also loads and stores the state)
    const int warm = 2, timed = std::min(variant == 2 ? 64 : 8, nt_min - warm);
    bool found = false;
    if (timed < 2) {
      for (const auto& c : cand)
        if (build(c)) return true;
      return false;
    }
    const auto t0 = std::chrono::steady_clock::now();
    init();
    cudaStream_t st = stream();
    // time per step of one candidate over `steps` steps, < 0 when it does not fit:
    // the resident kernel's launches as they are, the others' steps over a replayed
    // graph, as repeated runs launch them (from the host the two kernels of a step
    // start in either order, up to 40 % apart)
    auto trial = [&](const TuneChoice& c, int steps) -> float {
      if (!build(c)) return -1.f;
      uploads_done();
      float ms = 0;
      ++tune_trials;
      if (cfg.variant == 2) {
        launch_steps(st, 0, warm);
        CK(cudaEventRecord(ev0, st));
        launch_steps(st, warm, warm + steps);
        CK(cudaEventRecord(ev1, st));
        CK(cudaStreamSynchronize(st));
        CK(cudaEventElapsedTime(&ms, ev0, ev1));
        return ms / float(steps);
      }
      auto steps_from_zero = [&](cudaStream_t on) {
        if (scls.d_counter.n) CK(cudaMemsetAsync(scls.d_counter.p, 0, scls.d_counter.n * sizeof(unsigned), on));
        launch_steps(on, 0, steps);
      };
      const Graph g = capture(steps_from_zero);
      auto once = [&] { 
        if (g.exec)
          CK(cudaGraphLaunch(g.exec, st));
        else
          steps_from_zero(st);
      };
      once();
      CK(cudaEventRecord(ev0, st));
      once();
      CK(cudaEventRecord(ev1, st));
      CK(cudaStreamSynchronize(st));
      CK(cudaEventElapsedTime(&ms, ev0, ev1));
      return ms / float(steps);
    };
    std::vector<std::pair<float, TuneChoice>> timing;
    float least = 0;  // of the steps timed so far
    // a look takes about so many ms of steps once a step's time is known (many short
    // ones, so that a graph's own start of some microseconds counts little)
    auto steps_in = [&](float ms, int fewest, int most) {
      return least > 0 ? std::max(fewest, std::min(most, int(ms / least))) : 8;
    };
    // the half steps with half as many threads are at most a sixth faster
    auto hopeless = [&](const TuneChoice& c) {
      return c[0] == 3 && !timing.empty() && timing.back().second[0] == 3 && timing.back().first > 1.2f * least;
    };
    for (const auto& c : cand) {
      if (hopeless(c)) continue;
      const float ms = trial(c, c[0] == 2 ? timed : std::min(steps_in(0.3f, 4, 32), nt_min));
      if (ms < 0.f) continue;
      timing.emplace_back(ms, c);
      least = least > 0 ? std::min(least, ms) : ms;
    }
    std::stable_sort(timing.begin(), timing.end(), [](const auto& a, const auto& b) { return a.first < b.first; });
    found = !timing.empty();
    if (found) best = timing[0].second;
    // few steps tell shapes apart to a percent or two: the best three of those within
    // 2 % are timed again over more. (150x130x90 cells without layers, 400 steps, over
    // models and processes: 10.4 to 13.5 ms with a first look's choice from launched
    // steps.)
    if (variant != 2 && timing.size() > 1 && timing[1].first < 1.02f * timing[0].first) {
      const int steps = std::min(steps_in(0.6f, 6, 48), nt_min);
      float best_ms = 1e30f;
      for (size_t k = 0; k < std::min<size_t>(3, timing.size()); ++k) {
        if (timing[k].first >= 1.02f * timing[0].first) break;
        const float ms = trial(timing[k].second, steps);
        if (ms >= 0.f && ms < best_ms) {
          best_ms = ms;
          best = timing[k].second;
        }
      }
    }
    check_error();
    tune_ms += std::chrono::duration<double, std::milli>(std::chrono::steady_clock::now() - t0).count();
    if (variant == 2 && best[0] != 2) found = false;  // the others' shapes are timed next
    if (!found) best[0] = -1;
    {
      std::lock_guard<std::mutex> lock(g_tune_mutex);
      g_tune_cache[key] = best;
    }
    return found && build(best);
  }

  // Streaming kernel: 31 x TY column tiles cut in z chunks of at most 62
  // planes (cut at the z slabs' inner faces), each with the mask of its
  // planes that hold split-field cells.
  void build_stream_tiles(int n_sm) {
    StreamClass& c = scls;
    const void* fn = nullptr;
    int threads = 0, smem = 0, ty = 0;
    {
      c.v = find_stream_variant(cfg.ty, cfg.stages);
      if (!c.v) throw ArgError{FDTD_ERR_ARG, "No streaming kernel instantiated for this tile height / stage count."};
      c.fn = c.v->fn;
      fn = reinterpret_cast<const void*>(c.fn);
      threads = c.v->threads;
      bool splits = false;
      for (auto* s : sims) splits = splits || s->splits.n > 0;
      c.ring = stream_slots(*c.v, cfg.stages, c.v->min_blocks, splits, &c.n_main, &c.n_reg);
      smem = int(c.ring);
      ty = c.v->ty;
    }
    allow_shared(fn);
    int per_sm = 0;
    CK(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, fn, threads, smem));
    if (per_sm < 1) throw ArgError{FDTD_ERR_LIMIT, "Step kernel does not fit on an SM."};
    int64_t cols = 0;
    for (auto* s : sims) cols += int64_t((s->nx + kStreamOwnX - 1) / kStreamOwnX) * ((s->ny + ty - 1) / ty);
    const int64_t slots = int64_t(per_sm) * n_sm;
    zchunk_used = 1 << 30;
    for (size_t i = 0; i < sims.size(); ++i) {
      fdtd_sim* s = sims[i];
      int zc = cfg.zchunk;
      if (zc <= 0) {
        // about four tiles per resident block
        const int64_t chunks = std::max<int64_t>(1, (slots * 4 + cols - 1) / std::max<int64_t>(cols, 1));
        zc = int((s->nz + chunks - 1) / chunks);
      }
      zc = std::max(1, std::min(zc, 62));
      zchunk_used = std::min(zchunk_used, zc);
      c.host_maps.emplace_back();
      encode_stream_maps(c.host_maps.back(), s, ty);
      if (split_index.size() <= i) split_index.push_back(std::make_unique<GradedIndex>(s->grid, kFlagESplit | kFlagHSplit));
      const GradedIndex& split_idx = *split_index[i];
      // z chunks of at most zc planes that do not straddle a z slab's inner
      // face: the first core chunk starts one plane past the low slab (its
      // halo plane is then a core plane), so interior columns of core chunks
      // are plain tiles
      std::vector<std::pair<int, int>> zr;
      std::vector<int> chunk_of(size_t(s->nz), 0);
      {
        const int* pt = s->split_plan.t;
        const int zlo = pt[4] > 0 ? std::min(s->nz, pt[4] + 1) : 0;
        const int zhi = pt[5] > 0 ? std::max(zlo, s->nz - pt[5]) : s->nz;
        auto cut = [&](int a, int b) {
          for (int z = a; z < b; z += zc) zr.push_back({z, std::min(b, z + zc)});
        };
        cut(0, zlo);
        cut(zlo, zhi);
        cut(zhi, s->nz);
        for (size_t k = 0; k < zr.size(); ++k)
          for (int z = zr[k].first; z < zr[k].second; ++z) chunk_of[size_t(z)] = int(k);
      }
      // tiles (x / 31, y / TY, z chunk) that own a probe cell
      std::unordered_set<int64_t> probe_tiles;
      const int ntx = (s->nx + kStreamOwnX - 1) / kStreamOwnX, nty = (s->ny + ty - 1) / ty;
      for (const int64_t cell : s->grid.probe_cell) {
        const int z = int(cell % s->nz), y = int((cell / s->nz) % s->ny), x = int(cell / (int64_t(s->nz) * s->ny));
        probe_tiles.insert((int64_t(chunk_of[size_t(z)]) * nty + y / ty) * ntx + x / kStreamOwnX);
      }
      for (size_t zk = 0; zk < zr.size(); ++zk)
        for (int y0 = 0; y0 < s->ny; y0 += ty)
          for (int x0 = 0; x0 < s->nx; x0 += kStreamOwnX) {
            const int z0 = zr[zk].first, z1 = zr[zk].second;
            // planes holding split cells in the E region (columns x0-1 .. x0+30, rows y0-1 .. y0+ty-1)
            uint64_t mask = 0;
            for (int j = 0; j < z1 - z0 + 1; ++j) {
              const int z = z0 - 1 + j;
              if (z >= 0 && split_idx.count(x0 - 1, x0 + kStreamOwnX, y0 - 1, y0 + ty, z, z + 1) > 0)
                mask |= uint64_t(1) << j;
            }
            // slab stores the tile's rows and columns reach on planes outside the z slabs
            const int* pt = s->split_plan.t;
            const int zc0 = pt[4], zc1 = s->nz - pt[5];
            int ys = -1, xs = -1;
            if (zc1 > zc0) {
              if (pt[2] > 0 && y0 - 1 < pt[2]) ys = kStYlo;
              else if (pt[3] > 0 && y0 + ty - 1 >= s->ny - pt[3]) ys = kStYhi;
              if (pt[0] > 0 && x0 - 1 < pt[0]) xs = kStXlo;
              else if (pt[1] > 0 && x0 + kStreamOwnX - 1 >= s->nx - pt[1]) xs = kStXhi;
            }
            StreamTile t{};
            t.sim = int(i);
            t.x0 = x0;
            t.y0 = y0;
            t.z0 = z0;
            t.z1 = z1;
            t.ys = ys;
            t.xs = xs;
            t.plain = mask == 0 && !probe_tiles.count((int64_t(zk) * nty + y0 / ty) * ntx + x0 / kStreamOwnX);
            t.split_lo = uint32_t(mask);
            t.split_hi = uint32_t(mask >> 32);
            c.host_tiles.push_back(t);
          }
    }
    // Plain tiles go to the plain-tile kernel, the others to the general one.
    // Persistent blocks take tiles in list order, so the costliest go first
    // and the last tiles taken are short ones: a plane with split-field cells
    // costs about three ordinary planes. Stable, so tiles of equal cost keep
    // their z-chunk-major order and neighbours still share halos in L2.
    {
      std::vector<StreamTile> all;
      all.swap(c.host_tiles);
      for (const auto& t : all) (t.plain && !cfg.one_list ? c.host_tiles_p : c.host_tiles).push_back(t);
    }
    auto cost = [](const StreamTile& t) {
      return (t.z1 - t.z0 + 1) + 2 * (__builtin_popcount(t.split_lo) + __builtin_popcount(t.split_hi));
    };
    for (auto* list : {&c.host_tiles, &c.host_tiles_p})
      std::stable_sort(list->begin(), list->end(),
                       [&](const StreamTile& a, const StreamTile& b) { return cost(a) > cost(b); });
    c.n_tiles = int(c.host_tiles.size());
    c.n_tiles_p = int(c.host_tiles_p.size());
    // the plain-tile instantiation: plane slots only. It takes three to five blocks
    // per SM where it has nearly all tiles (150x130x90 cells without layers, 8-row
    // tiles: 29.8 -> 26.9 us per step); beside many general tiles more of its blocks
    // only displace theirs (256x256x128 with 8-cell layers 170 -> 178 us).
    const bool most = sims.size() == 1 && c.n_tiles_p > 9 * c.n_tiles;
    const int plain_blocks = most ? c.v->plain_blocks : c.v->min_blocks;
    c.fn_plain = most ? c.v->plain_most : c.v->plain_of[sims.size() == 1];
    int per_sm_p = 0;
    {
      int no_regions = 0;
      c.ring_p = stream_slots(*c.v, cfg.stages, plain_blocks, false, &c.n_main_p, &no_regions);
      const void* fp = reinterpret_cast<const void*>(c.fn_plain);
      allow_shared(fp);
      CK(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm_p, fp, threads, int(c.ring_p)));
      if (per_sm_p < 1) throw ArgError{FDTD_ERR_LIMIT, "Step kernel does not fit on an SM."};
      per_sm_p = std::min(per_sm_p, plain_blocks);
    }
    c.d_maps.alloc(c.host_maps.size());
    CK(cudaMemcpy(c.d_maps.p, c.host_maps.data(), c.host_maps.size() * sizeof(StreamMaps), cudaMemcpyHostToDevice));
    std::vector<SimDev> devs;
    for (size_t i = 0; i < sims.size(); ++i) {
      devs.push_back(sims[i]->dev);
      devs.back().maps = c.d_maps.p + i;
    }
    c.one = devs[0];
    c.d_sims.alloc(devs.size());
    CK(cudaMemcpy(c.d_sims.p, devs.data(), devs.size() * sizeof(SimDev), cudaMemcpyHostToDevice));
    c.d_tiles.alloc(std::max<size_t>(1, c.host_tiles.size()));
    if (c.n_tiles)
      CK(cudaMemcpy(c.d_tiles.p, c.host_tiles.data(), c.host_tiles.size() * sizeof(StreamTile), cudaMemcpyHostToDevice));
    c.d_tiles_p.alloc(std::max<size_t>(1, c.host_tiles_p.size()));
    if (c.n_tiles_p)
      CK(cudaMemcpy(c.d_tiles_p.p, c.host_tiles_p.data(), c.host_tiles_p.size() * sizeof(StreamTile),
                    cudaMemcpyHostToDevice));
    c.d_counter.alloc(2);
    c.grid = int(std::min<int64_t>(c.n_tiles, slots));
    c.grid_p = int(std::min<int64_t>(c.n_tiles_p, int64_t(per_sm_p) * n_sm));
    n_tiles = c.n_tiles + c.n_tiles_p;
    grid = c.grid + c.grid_p;
  }

  // The streaming kernels of step n (counters counted from step n0, with at
  // most `cap` blocks each): the general kernel on st and the plain-tile
  // kernel beside it on a forked stream, or on st after it when `side` is
  // false.
  int launch_stream_step(cudaStream_t st, int n, int n0, int cap, bool side) {
    StreamClass& c = scls;
    const int g = std::min(c.grid, cap), gp = std::min(c.grid_p, cap);
    const bool fork = side && c.n_tiles > 0 && c.n_tiles_p > 0;
    if (fork) {
      CK(cudaEventRecord(step_fork, st));
      CK(cudaStreamWaitEvent(step_side, step_fork, 0));
    }
    if (c.n_tiles > 0) {
      const unsigned base = unsigned(n - n0) * unsigned(c.n_tiles + g);
      c.fn<<<g, c.v->threads, c.ring, st>>>(c.one, c.d_sims.p, c.d_tiles.p, c.n_tiles, n, c.d_counter.p, base, d_err.p,
                                                  c.n_main, c.n_reg, wait_limit, withhold);
      CK(cudaGetLastError());
    }
    if (c.n_tiles_p > 0) {
      const unsigned base = unsigned(n - n0) * unsigned(c.n_tiles_p + gp);
      c.fn_plain<<<gp, c.v->threads, c.ring_p, fork ? step_side : st>>>(
          c.one, c.d_sims.p, c.d_tiles_p.p, c.n_tiles_p, n, c.d_counter.p + 1, base, d_err.p, c.n_main_p, 0, wait_limit,
          withhold);
      CK(cudaGetLastError());
    }
    if (fork) {
      CK(cudaEventRecord(step_join, step_side));
      CK(cudaStreamWaitEvent(st, step_join, 0));
    }
    return int(c.n_tiles > 0) + int(c.n_tiles_p > 0);
  }

  // Time steps n0 .. n1-1 on st as a run has them; returns how many launches that
  // took, a launch of the resident kernel counted once per step.
  int launch_steps(cudaStream_t st, int n0, int n1) {
    if (cfg.variant == 2) {
      launch_resident(st, n0, n1);
      return n1 - n0;
    }
    int k = 0;
    bool mon_pending = false;
    for (int n = n0; n < n1; ++n) k += step_and_samples(st, n, mon_pending);
    if (mon_pending) CK(cudaStreamWaitEvent(st, mon_join, 0));
    return k;
  }

  // The kernels of time step n on st; returns how many were launched.
  int launch_step(cudaStream_t st, int n) {
    if (cfg.variant == 1) {
      return launch_stream_step(st, n, 0, 1 << 30, true);
    } else if (cfg.variant == 2) {
      launch_resident(st, n, n + 1);
      return 1;
    } else if (cfg.variant == 3) {
      launch_half(st, n, false, false);
      launch_half(st, n, true, false);
      return 1;
    } else {
      fdtd_step_kernel<kTileY><<<n_tiles, dim3(32, kBlockY), 0, st>>>(d_sims.p, d_tiles.p, n);
      CK(cudaGetLastError());
      return 1;
    }
  }

  // Step n of a checkpointed adjoint's segment replay (segment from step n0),
  // with the streaming kernels on at most `per_sm` blocks per SM each, one
  // after the other, so that the reversal of the next segment, running at the
  // same time on another stream, finds room on every SM. The tile counters
  // were cleared before n0.
  void launch_replay_step(cudaStream_t st, int n, int n0, int n_sm, int per_sm) {
    if (cfg.variant == 1) {
      launch_stream_step(st, n, n0, n_sm * per_sm, false);
    } else {
      launch_step(st, n);
    }
  }

  // Orders the streaming kernels' tile lists for segment replays by the
  // Chebyshev distance (cells) of each tile's owned cells from the gradient
  // box of its simulation (boxes[i] for sims[i]; null: never needed).
  void build_replay_tiles(const std::vector<const int*>& boxes) {
    StreamClass& c = scls;
    auto order = [&](const std::vector<StreamTile>& src, DevBuf<StreamTile>& dst, std::vector<int>& dist) {
      std::vector<std::pair<int, StreamTile>> v;
      v.reserve(src.size());
      for (const auto& t : src) {
        const fdtd_sim* s = sims[size_t(t.sim)];
        const int* b = boxes[size_t(t.sim)];
        if (!b) continue;
        auto gap = [](int a0, int a1, int b0, int b1) { return std::max(0, std::max(a0 - (b1 - 1), b0 - (a1 - 1))); };
        const int x1 = std::min(s->nx, t.x0 + kStreamOwnX), y1 = std::min(s->ny, t.y0 + c.v->ty);
        const int d = std::max(gap(t.x0, x1, b[0], b[1]), std::max(gap(t.y0, y1, b[2], b[3]), gap(t.z0, t.z1, b[4], b[5])));
        v.emplace_back(d, t);
      }
      std::stable_sort(v.begin(), v.end(), [](const auto& a, const auto& b) { return a.first < b.first; });
      dist.resize(v.size());
      std::vector<StreamTile> h(v.size());
      for (size_t i = 0; i < v.size(); ++i) {
        dist[i] = v[i].first;
        h[i] = v[i].second;
      }
      dst.reserve(std::max<size_t>(1, h.size()));
      if (!h.empty()) CK(cudaMemcpy(dst.p, h.data(), h.size() * sizeof(StreamTile), cudaMemcpyHostToDevice));
    };
    order(c.host_tiles, rep_tiles, rep_dist);
    order(c.host_tiles_p, rep_tiles_p, rep_dist_p);
  }

  // Step n of a segment replay restricted to the tiles within `reach` cells of
  // the gradient boxes (lists from build_replay_tiles), the general kernel
  // then the plain-tile kernel on st, at most `cap` blocks each; base_g /
  // base_p carry the tile counters' bases from step to step of the segment.
  void launch_replay_subset(cudaStream_t st, int n, int reach, int cap, unsigned& base_g, unsigned& base_p) {
    StreamClass& c = scls;
    const int ng = int(std::upper_bound(rep_dist.begin(), rep_dist.end(), reach) - rep_dist.begin());
    const int np = int(std::upper_bound(rep_dist_p.begin(), rep_dist_p.end(), reach) - rep_dist_p.begin());
    if (ng > 0) {
      const int g = std::min(std::min(c.grid, cap), ng);
      c.fn<<<g, c.v->threads, c.ring, st>>>(c.one, c.d_sims.p, rep_tiles.p, ng, n, c.d_counter.p, base_g, d_err.p,
                                                  c.n_main, c.n_reg, wait_limit, withhold);
      CK(cudaGetLastError());
      base_g += unsigned(ng + g);
    }
    if (np > 0) {
      const int g = std::min(std::min(c.grid_p, cap), np);
      c.fn_plain<<<g, c.v->threads, c.ring_p, st>>>(c.one, c.d_sims.p, rep_tiles_p.p, np, n, c.d_counter.p + 1, base_p,
                                                        d_err.p, c.n_main_p, 0, wait_limit, withhold);
      CK(cudaGetLastError());
      base_p += unsigned(np + g);
    }
  }

  // Box-history capture of the simulations in recorded mode (adj_mode 2):
  // one adj_capture_kernel launch per time step, before the step, inside the
  // captured time loop.
  DevBuf<CapSim> d_caps;
  int n_caps = 0, cap_blocks = 1;

  void build_caps() {
    uploaded = true;
    std::vector<CapSim> v;
    int64_t nb_max = 0;
    for (auto* s : sims)
      if (s->adj_mode == 2) {
        CapSim c{};
        c.s = s->dev;
        c.bx0 = s->adj_box[0]; c.bx1 = s->adj_box[1]; c.by0 = s->adj_box[2];
        c.by1 = s->adj_box[3]; c.bz0 = s->adj_box[4]; c.bz1 = s->adj_box[5];
        c.nb = box_cells(s->adj_box);
        c.hist = s->hist.p;
        nb_max = std::max(nb_max, c.nb);
        v.push_back(c);
      }
    if (cfg.variant == 3 && !v.empty()) {
      std::vector<CapSim> hc(sims.size(), CapSim{});
      for (size_t i = 0, k = 0; i < sims.size(); ++i)
        if (sims[i]->adj_mode == 2) hc[i] = v[k++];
      half_captures(hc);
    }
    n_caps = int(v.size());
    d_caps.alloc(v.size());
    if (!v.empty()) CK(cudaMemcpy(d_caps.p, v.data(), v.size() * sizeof(CapSim), cudaMemcpyHostToDevice));
    cap_blocks = int(std::min<int64_t>(1024, std::max<int64_t>(1, (nb_max + 255) / 256)));
  }

  // Adjoint work buffers of each request slot, kept between sweeps.
  struct AdjBufs {
    DevBuf<float> lam, lams, radj, seg;
    DevBuf<float> rec_save;  // the forward's probe records, kept while segment replays rewrite them
    DevBuf<int> pidx, pfld;
    DevBuf<double> grad;
  };
  // Segment replays of a checkpointed adjoint (streaming kernels): the general
  // and plain tile lists ordered by each tile's distance from its simulation's
  // gradient box, nearest first, with those distances (cells).
  DevBuf<StreamTile> rep_tiles, rep_tiles_p;
  std::vector<int> rep_dist, rep_dist_p;
  std::vector<int> rep_boxes;      // gradient box of each simulation of the engine (empty: none)
  std::vector<std::unique_ptr<AdjBufs>> adj_bufs;
  DevBuf<AdjSim> adj_d_as;
  DevBuf<int4> adj_d_t;
  DevBuf<CapSim> adj_d_c;
  DevBuf<AdjMaps> adj_d_maps;     // streaming reverse step: tensor maps of each simulation's adjoint state
  DevBuf<int4> adj_d_ts;          // its tiles (w: the tile's boxes hold split cells)
  DevBuf<unsigned> adj_counter;   // its tile counter
  DevBuf<int4> adj_d_blocks;      // half-step reverse: blocks over several simulations
  static constexpr int kAdjHalfWant = 128;                // its threads per block (64 and 256: up to 10 % slower)
  static constexpr int64_t kAdjHalfBytes = 160'000'000;
  static int adj_tiles_per_sm() {
    const char* v = std::getenv("RFN_ADJ_TILES_PER_SM");
    return v ? std::max(1, std::atoi(v)) : 4;
  }
  // planes per tile along z (0: picked by adj_pick_zchunk)
  static int adj_zchunk() {
    const char* v = std::getenv("RFN_ADJ_ZCHUNK");
    return v ? std::max(0, std::atoi(v)) : 0;
  }
  // Planes per reverse-step tile along z when `slots` blocks of tx x ty tiles
  // are resident at once: the tiles should fill whole waves of blocks (a short
  // last wave leaves SMs idle) and load few halo planes (two per tile). Picks
  // the largest (tiles / (waves * slots)) * (owned planes / loaded planes)
  // over chunks of 4 planes or more that give at least two waves; 4 planes
  // when even those give fewer.
  // Planes per tile for the persistent reverse step on `slots` blocks: the
  // longest even chunks (nz_max / c planes, c = 1, 2, ...) that still give
  // at least 15/16 of the blocks a tile; 4 planes when none do.
  int adj_pick_zchunk_persistent(int64_t slots, int tx, int ty) const {
    int nz_max = 0;
    for (auto* s : sims) nz_max = std::max(nz_max, s->nz);
    for (int c = 1; c <= nz_max / 4; ++c) {
      const int zl = (nz_max + c - 1) / c;
      int64_t tiles = 0;
      for (auto* s : sims) tiles += int64_t((s->nx + tx - 1) / tx) * ((s->ny + ty - 1) / ty) * ((s->nz + zl - 1) / zl);
      if (16 * tiles >= 15 * slots) return zl;
    }
    return 4;
  }
  int adj_pick_zchunk(int64_t slots, int tx, int ty) const {
    int nz_max = 0;
    int64_t owned = 0;  // tile columns x planes
    for (auto* s : sims) {
      nz_max = std::max(nz_max, s->nz);
      owned += int64_t((s->nx + tx - 1) / tx) * ((s->ny + ty - 1) / ty) * s->nz;
    }
    double best = -1.0;
    int pick = 4;
    for (int zl = 4; zl <= nz_max; ++zl) {
      int64_t tiles = 0;
      for (auto* s : sims) tiles += int64_t((s->nx + tx - 1) / tx) * ((s->ny + ty - 1) / ty) * ((s->nz + zl - 1) / zl);
      const int64_t waves = (tiles + slots - 1) / slots;
      if (waves < 2) break;  // the tile count only falls as the chunks grow
      const double score = double(tiles) / double(waves * slots) * double(owned) / double(owned + 2 * tiles);
      if (score > best + 1e-12) {
        best = score;
        pick = zl;
      }
    }
    return pick;
  }

  // One simulation's part of an adjoint sweep: dJ/dX of its device DFT, the
  // gradient box, and where the [9][box cells] gradient goes.
  struct AdjRequest {
    fdtd_sim* s;
    const double* dJdX;
    const int* box;
    double* grad_out;
  };

  // Discrete adjoint of the last run of the simulations of this engine, all
  // made for a gradient in the same mode (adj_mode of the first): gradient of
  // J with respect to (Ca, Cb1, Cb2) of each E component on each box. The
  // adjoint state runs backwards from step nt-1 with one adj_step_kernel
  // launch per step over the tiles of all simulations. In recorded mode the
  // box history of every step is already on the device. With checkpoints the
  // run is replayed segment by segment, last segment first, capturing each
  // segment's box history into one half of a two-segment buffer; the replay
  // of segment k-1 (its own stream) runs while segment k is reversed.
  void adjoint(const std::vector<AdjRequest>& req) {
    init();
    cudaStream_t st = stream();
    const int mode = req[0].s->adj_mode;
    const int nt = req[0].s->ckpt_nt, K = mode == 1 ? req[0].s->ckpt_every : nt;
    int dev = 0, n_sm = 148;
    CK(cudaGetDevice(&dev));
    CK(cudaDeviceGetAttribute(&n_sm, cudaDevAttrMultiProcessorCount, dev));
    const char* sv = std::getenv("RFN_ADJ_STREAM");
    const bool stream_adj = sv && std::atoi(sv) != 0;
    // The half-step reverse where its state (six totals per cell, six halves more
    // per cell with split E or H) fits in L2, which then serves it twice per step;
    // beyond that one launch per step, which reads it once. Per step, one launch
    // against two halves: 52x44x33 cells with 6-cell layers 22.6 against 9.4 us,
    // 96x96x64 with 10 39.6 against 29.8, 128x128x96 with 10 (75 MB) 88.8 against
    // 64.7, 160x150x120 with 6 (101 MB) 148.6 against 136.2, 190x170x120 with 6 (133
    // MB) 181 against 167; 224x200x128 with 8 (207 MB) 248 against 251. RFN_ADJ_HALF=0 / 1 decides.
    int64_t adj_state = 0;
    for (const auto& rq : req)
      adj_state += 24 * (int64_t(rq.s->nx) * rq.s->ny * rq.s->nz + rq.s->grid.e_split_cells + rq.s->grid.h_split_cells);
    const char* hv = std::getenv("RFN_ADJ_HALF");
    const bool half_adj = !stream_adj && (hv ? std::atoi(hv) != 0 : adj_state <= kAdjHalfBytes);
    // work buffers are kept on the engine between sweeps (allocation and
    // release of ~36 floats per cell would otherwise come with every gradient)
    if (adj_bufs.size() < req.size()) adj_bufs.resize(req.size());
    std::vector<AdjSim> as(req.size());
    std::vector<CapSim> caps;
    int64_t nb_max = 0;
    int p_max = 0;
    for (size_t i = 0; i < req.size(); ++i) {
      fdtd_sim* s = req[i].s;
      const int* box = req[i].box;
      if (!adj_bufs[i]) adj_bufs[i] = std::make_unique<AdjBufs>();
      AdjBufs* B = adj_bufs[i].get();
      const size_t N = s->cells_padded;
      const int64_t nb = box_cells(box);
      nb_max = std::max(nb_max, nb);
      const int P = int(s->probes.size());
      p_max = std::max(p_max, P);
      const std::vector<float> radj = record_adjoints(s, req[i].dJdX, nt);
      std::vector<int> pidx(size_t(std::max(P, 1)), 0), pfld(size_t(std::max(P, 1)), 0);
      for (int pr = 0; pr < P; ++pr) {
        const int64_t cell = s->grid.probe_cell[size_t(pr)];
        const int z = int(cell % s->nz), y = int((cell / s->nz) % s->ny), x = int(cell / (int64_t(s->nz) * s->ny));
        pidx[size_t(pr)] = z * s->ny * s->pitch + y * s->pitch + x;
        pfld[size_t(pr)] = s->probes[size_t(pr)].field;
      }
      // (the half-step reverse works in place, in the first of the two buffers)
      B->lam.reserve((half_adj ? 6 : 12) * N);
      CK(cudaMemsetAsync(B->lam.p, 0, B->lam.n * sizeof(float), st));
      if (s->splits.n) {
        B->lams.reserve((half_adj ? 12 : 24) * N);
        CK(cudaMemsetAsync(B->lams.p, 0, B->lams.n * sizeof(float), st));
      }
      B->radj.reserve(radj.size());
      CK(cudaMemcpy(B->radj.p, radj.data(), radj.size() * sizeof(float), cudaMemcpyHostToDevice));
      B->pidx.reserve(pidx.size());
      CK(cudaMemcpy(B->pidx.p, pidx.data(), pidx.size() * sizeof(int), cudaMemcpyHostToDevice));
      B->pfld.reserve(pfld.size());
      CK(cudaMemcpy(B->pfld.p, pfld.data(), pfld.size() * sizeof(int), cudaMemcpyHostToDevice));
      B->grad.reserve(9 * size_t(nb));
      CK(cudaMemsetAsync(B->grad.p, 0, 9 * size_t(nb) * sizeof(double), st));
      AdjSim& a = as[i];
      a = AdjSim{};
      a.nx = s->nx; a.ny = s->ny; a.nz = s->nz; a.pitch = s->pitch; a.plane = s->ny * s->pitch; a.nt = nt;
      a.mat = s->mat.p;
      a.rows = s->rows.p;
      a.cell_probes = s->cell_probes.p;
      a.N = int64_t(N);
      a.lam = B->lam.p;
      a.lams = B->lams.p;
      a.radj = B->radj.p;
      a.probe_idx = B->pidx.p;
      a.probe_field = B->pfld.p;
      a.n_probes = P;
      a.bx0 = box[0]; a.bx1 = box[1]; a.by0 = box[2]; a.by1 = box[3]; a.bz0 = box[4]; a.bz1 = box[5];
      a.nb = nb;
      a.grad = B->grad.p;
      if (mode == 2) {
        a.hist = s->hist.p;
      } else {
        B->seg.reserve(2 * size_t(K) * 9 * size_t(nb));
        a.hist = B->seg.p;
        CapSim c{};
        c.s = s->dev;
        c.bx0 = box[0]; c.bx1 = box[1]; c.by0 = box[2]; c.by1 = box[3]; c.bz0 = box[4]; c.bz1 = box[5];
        c.nb = nb;
        c.hist = B->seg.p;
        caps.push_back(c);
      }
    }
    int plain_per_sm = 2;
    CK(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&plain_per_sm, &adj_step_kernel<kAdjTileY, 2>,
                                                     32 * (kAdjTileY + 2), 0));
    const int zc = adj_zchunk() ? adj_zchunk()
                   : std::getenv("RFN_ADJ_TILES_PER_SM")
                       ? 0
                       : adj_pick_zchunk(int64_t(std::max(plain_per_sm, 1)) * n_sm, kAdjTileX, kAdjTileY);
    const std::vector<int4> tiles = plain_tiles(n_sm, zc, nullptr, kAdjTileX, kAdjTileY, adj_tiles_per_sm());
    // The streaming reverse step, on request (RFN_ADJ_STREAM=1; the plain one
    // is the default): tiles (split tiles first), tensor maps of each
    // simulation's adjoint state and material index, plane slots sized for
    // two blocks per SM.
    using AG = AdjGeom<kAdjStreamTileY>;
    int n_ts = 0, adj_grid = 0, adj_slots = 0;
    uint32_t adj_smem = 0;
    unsigned adj_base = 0;
    if (stream_adj) {
      constexpr uint32_t kBudget = 233472 / 2 - 1024 - 512 - 9600;  // two blocks per SM, beside the static arrays
      adj_slots = int(std::min<uint32_t>(kAdjStreamSlotsMax, kBudget / AG::SLOT));
      if (adj_slots < 3) throw ArgError{FDTD_ERR_LIMIT, "Streaming reverse step's plane slots do not fit."};
      adj_smem = uint32_t(adj_slots) * AG::SLOT;
      const void* fn = reinterpret_cast<const void*>(&adj_stream_kernel<kAdjStreamTileY>);
      allow_shared(fn);
      int per_sm = 0;
      CK(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, fn, AG::THREADS, int(adj_smem)));
      if (per_sm < 1) throw ArgError{FDTD_ERR_LIMIT, "Streaming reverse step does not fit on an SM."};
      const int zcs = adj_zchunk() ? adj_zchunk()
                      : std::getenv("RFN_ADJ_TILES_PER_SM")
                          ? 0
                          : adj_pick_zchunk_persistent(int64_t(per_sm) * n_sm, kAdjTileX, kAdjStreamTileY);
      std::vector<int4> ts = plain_tiles(n_sm, zcs, nullptr, kAdjTileX, kAdjStreamTileY, adj_tiles_per_sm());
      std::vector<GradedIndex> gis;
      for (const auto& rq : req) gis.emplace_back(rq.s->grid, kFlagESplit | kFlagHSplit);
      for (auto& t : ts) {
        // the boxes of every plane of the tile: columns x0-1 .. x0+30, rows y0-1 .. y0+TY, planes z0-1 .. z1
        const int x0 = t.y & 0xffff, y0 = int(unsigned(t.y) >> 16), z0 = t.z & 0xffff, z1 = int(unsigned(t.z) >> 16);
        t.w = gis[size_t(t.x)].count(x0 - 1, x0 + kAdjTileX + 1, y0 - 1, y0 + kAdjStreamTileY + 1, z0 - 1, z1 + 1) > 0;
      }
      std::stable_sort(ts.begin(), ts.end(), [](const int4& a, const int4& b) { return a.w > b.w; });
      n_ts = int(ts.size());
      std::vector<AdjMaps> hm(req.size());
      for (size_t i = 0; i < req.size(); ++i) {
        fdtd_sim* s = req[i].s;
        const size_t N = s->cells_padded;
        std::memset(&hm[i], 0, sizeof(AdjMaps));
        const auto F = CU_TENSOR_MAP_DATA_TYPE_FLOAT32;
        float* lam = adj_bufs[i]->lam.p;
        encode_map(&hm[i].lam_e, lam, F, 4, s, 5, AG::EW, AG::ER, 3, N, 6 * N);
        encode_map(&hm[i].lam_h, lam + 3 * N, F, 4, s, 5, AG::HW, AG::HR, 3, N, 6 * N);
        if (s->splits.n) encode_map(&hm[i].halves, adj_bufs[i]->lams.p, F, 4, s, 5, AG::SW, AG::HR, 12, N, 12 * N);
        encode_map(&hm[i].ids, s->mat.p, CU_TENSOR_MAP_DATA_TYPE_UINT16, 2, s, 3, AG::IW, AG::HR, 1, 0, 0);
      }
      adj_d_maps.reserve(hm.size());
      CK(cudaMemcpy(adj_d_maps.p, hm.data(), hm.size() * sizeof(AdjMaps), cudaMemcpyHostToDevice));
      adj_d_ts.reserve(ts.size());
      CK(cudaMemcpy(adj_d_ts.p, ts.data(), ts.size() * sizeof(int4), cudaMemcpyHostToDevice));
      adj_grid = int(std::min<int64_t>(n_ts, int64_t(per_sm) * n_sm));
      adj_counter.reserve(1);
      CK(cudaMemsetAsync(adj_counter.p, 0, sizeof(unsigned), st));
    }
    // The half-step reverse: blocks of about 128 threads over every simulation.
    HalfLaunch hl{};
    dim3 half_grid;
    int half_threads = 0;
    if (half_adj) {
      // Cells per thread along z: rows are read less often, but a small grid runs
      // out of threads. 200 steps forward and back with 1 / 2 / 4 cells: 52x44x33
      // 4.55 / 5.82 / 7.95 ms, 80x72x60 8.05 / 8.21 / 9.67, 96x96x64 11.71 / 11.16 /
      // 12.09, 128x128x96 25.85 / 23.42 / 22.68, 160x150x120 49.92 / 46.83 / 45.81.
      int64_t cells = 0;
      for (const auto& a : as) cells += int64_t(a.nx) * a.ny * a.nz;
      hl.deep = cells < 400'000 ? 1 : cells < 1'000'000 ? 2 : 4;
      if (as.size() == 1) {
        half_shape(as[0].nx, as[0].ny, kAdjHalfWant, &hl.seg, &hl.rows);
        half_threads = (hl.seg * hl.rows + 31) / 32 * 32;
        half_grid = dim3(unsigned((as[0].nx + hl.seg - 1) / hl.seg), unsigned((as[0].ny + hl.rows - 1) / hl.rows),
                         unsigned((as[0].nz + hl.deep - 1) / hl.deep));
      } else {
        std::vector<int4> blocks;
        half_threads = half_blocks(kAdjHalfWant, blocks, hl.deep);
        half_grid = dim3(unsigned(blocks.size()));
        adj_d_blocks.reserve(blocks.size());
        CK(cudaMemcpy(adj_d_blocks.p, blocks.data(), blocks.size() * sizeof(int4), cudaMemcpyHostToDevice));
        hl.blocks = adj_d_blocks.p;
      }
    }
    auto reverse_step = [&](int n, int hist_n0) {
      if (half_adj) {
        const bool one = as.size() == 1;
        hl.n = n;
        const AdjSim* ds = adj_d_as.p;
        launch_dependent(one ? &adj_half_kernel<false, true> : &adj_half_kernel<false, false>, half_grid, half_threads,
                         st, as[0], hl, ds, hist_n0);
        launch_dependent(one ? &adj_half_kernel<true, true> : &adj_half_kernel<true, false>, half_grid, half_threads,
                         st, as[0], hl, ds, hist_n0);
      } else if (stream_adj) {
        adj_stream_kernel<kAdjStreamTileY><<<adj_grid, AG::THREADS, adj_smem, st>>>(
            adj_d_as.p, adj_d_maps.p, adj_d_ts.p, n_ts, n, hist_n0, adj_counter.p, adj_base, d_err.p, adj_slots,
            wait_limit);
        adj_base += unsigned(n_ts + adj_grid);
      } else {
        // register cap: two resident blocks per SM (default) or three
        const char* mb = std::getenv("RFN_ADJ_MINB");
        auto adj_fn = (mb && std::atoi(mb) == 3) ? &adj_step_kernel<kAdjTileY, 3> : &adj_step_kernel<kAdjTileY, 2>;
        adj_fn<<<int(tiles.size()), dim3(32, kAdjTileY + 2), 0, st>>>(adj_d_as.p, adj_d_t.p, n, hist_n0);
      }
      CK(cudaGetLastError());
      ++adj_launches;
    };
    DevBuf<AdjSim>& d_as = adj_d_as;
    DevBuf<int4>& d_t = adj_d_t;
    DevBuf<CapSim>& d_c = adj_d_c;
    d_as.reserve(as.size());
    CK(cudaMemcpy(d_as.p, as.data(), as.size() * sizeof(AdjSim), cudaMemcpyHostToDevice));
    d_t.reserve(tiles.size());
    CK(cudaMemcpy(d_t.p, tiles.data(), tiles.size() * sizeof(int4), cudaMemcpyHostToDevice));
    if (!caps.empty()) {
      d_c.reserve(caps.size());
      CK(cudaMemcpy(d_c.p, caps.data(), caps.size() * sizeof(CapSim), cudaMemcpyHostToDevice));
    }
    const int cap_grid = int(std::min<int64_t>(1024, std::max<int64_t>(1, (nb_max + 255) / 256)));
    uploads_done();
    if (p_max > 0) {
      adj_inject_kernel<<<dim3((p_max + 127) / 128, unsigned(as.size())), 128, 0, st>>>(
          d_as.p, nt - 1, half_adj ? 0 : (nt - 1) & 1, half_adj ? 3 : 0);
      CK(cudaGetLastError());
    }
    adj_launches = 0;
    CK(cudaEventRecord(ev0, st));
    if (mode == 2) {
      for (int n = nt - 1; n >= 0; --n) reverse_step(n, 0);
    } else {
      const int nseg = (nt + K - 1) / K;
      const char* rb = std::getenv("RFN_REPLAY_BLOCKS_PER_SM");
      const int per_sm = rb ? std::max(1, std::atoi(rb)) : 1;
      cudaStream_t rs = rep_stream;
      // The history of step n is the state before step n, so a segment
      // [n0, n1) replays steps n0 .. n1-2 only. The history reads the box and
      // the H values one cell beyond it (the +1 neighbours of the E update's
      // differences), and a step moves information by at most one cell along
      // each axis, so step n needs to be right only within n1-1-n cells of the
      // box: with the streaming kernels each replay step runs the tiles within
      // that reach (nearest first). Tiles outside it keep stale values, which
      // never reach what the history reads before the segment ends.
      const bool full = std::getenv("RFN_REPLAY_FULL") != nullptr;
      const bool cone = cfg.variant == 1 && !full, half_cone = cfg.variant == 3 && !full;
      if (cfg.variant == 3) {
        std::vector<CapSim> hc(sims.size(), CapSim{});
        rep_boxes.assign(6 * sims.size(), 0);
        for (size_t q = 0; q < req.size(); ++q)
          for (size_t i = 0; i < sims.size(); ++i)
            if (sims[i] == req[q].s) {
              hc[i] = caps[q];
              std::copy(req[q].box, req[q].box + 6, rep_boxes.begin() + 6 * std::ptrdiff_t(i));
            }
        half_captures(hc);
        half.d_boxes.reserve(rep_boxes.size());
        CK(cudaMemcpy(half.d_boxes.p, rep_boxes.data(), rep_boxes.size() * sizeof(int), cudaMemcpyHostToDevice));
      }
      if (cone) {
        std::vector<const int*> boxes(sims.size(), nullptr);
        for (const auto& r : req)
          for (size_t i = 0; i < sims.size(); ++i)
            if (sims[i] == r.s) boxes[i] = r.box;
        build_replay_tiles(boxes);
      }
      uploads_done();
      // the replays rewrite probe records (outside the reach, with stale
      // values): the forward's records are kept aside and put back at the end
      for (size_t i = 0; i < req.size(); ++i) {
        fdtd_sim* s = req[i].s;
        adj_bufs[i]->rec_save.reserve(s->rec.n);
        CK(cudaMemcpyAsync(adj_bufs[i]->rec_save.p, s->rec.p, s->rec.n * sizeof(float), cudaMemcpyDeviceToDevice, st));
      }
      // segment k replayed on rs from its snapshot into history half k & 1,
      // each step's box capture beside it (as in a recorded run)
      auto replay = [&](int k) {
        const int n0 = k * K, n1 = std::min(nt, n0 + K), h0 = n0 - (k & 1) * K;
        const size_t b = size_t(state_buf(n0));
        for (const auto& r : req) {
          fdtd_sim* s = r.s;
          const size_t N = s->cells_padded;
          const size_t sb = s->splits.n ? 2 * s->split_buf_pairs : 0;  // split floats per time buffer
          const size_t stride = 6 * N + sb;
          const float* src = s->ckpt.p + size_t(k) * stride;
          CK(cudaMemcpyAsync(s->fields.p + b * 6 * N, src, 6 * N * sizeof(float), cudaMemcpyDeviceToDevice, rs));
          if (sb)
            CK(cudaMemcpyAsync(s->splits.p + b * sb, src + 6 * N, sb * sizeof(float), cudaMemcpyDeviceToDevice, rs));
        }
        if (cfg.variant == 1) CK(cudaMemsetAsync(scls.d_counter.p, 0, scls.d_counter.n * sizeof(unsigned), rs));
        unsigned base_g = 0, base_p = 0;
        for (int n = n0; n < n1; ++n) {
          if (cfg.variant == 3) {
            // E of the segment's last step is advanced only for its history
            const int reach = half_cone ? n1 - 1 - n : -1;
            launch_half(rs, n, false, true, h0, reach);
            if (n + 1 < n1) launch_half(rs, n, true, false, 0, reach);
            continue;
          }
          CK(cudaEventRecord(cap_fork, rs));
          CK(cudaStreamWaitEvent(cap_stream, cap_fork, 0));
          adj_capture_kernel<<<dim3(cap_grid, unsigned(caps.size())), 256, 0, cap_stream>>>(d_c.p, n, h0);
          CK(cudaGetLastError());
          CK(cudaEventRecord(cap_join, cap_stream));
          if (n + 1 < n1) {
            if (cone)
              launch_replay_subset(rs, n, n1 - 1 - n, n_sm * per_sm, base_g, base_p);
            else
              launch_replay_step(rs, n, n0, n_sm, per_sm);
          }
          CK(cudaStreamWaitEvent(rs, cap_join, 0));
        }
        CK(cudaEventRecord(seg_done[k & 1], rs));
      };
      CK(cudaEventRecord(cap_fork, st));  // the replays start after this sweep's set-up on st
      CK(cudaStreamWaitEvent(rs, cap_fork, 0));
      replay(nseg - 1);
      for (int k = nseg - 1; k >= 0; --k) {
        if (k >= 1) {
          // history half (k-1) & 1 was last read by the reversal of segment k+1
          if (k + 1 < nseg) CK(cudaStreamWaitEvent(rs, seg_free[(k + 1) & 1], 0));
          replay(k - 1);
        }
        const int n0 = k * K, n1 = std::min(nt, n0 + K);
        CK(cudaStreamWaitEvent(st, seg_done[k & 1], 0));
        for (int n = n1 - 1; n >= n0; --n) reverse_step(n, n0 - (k & 1) * K);
        CK(cudaEventRecord(seg_free[k & 1], st));
      }
      for (size_t i = 0; i < req.size(); ++i) {
        fdtd_sim* s = req[i].s;
        CK(cudaMemcpyAsync(s->rec.p, adj_bufs[i]->rec_save.p, s->rec.n * sizeof(float), cudaMemcpyDeviceToDevice, st));
      }
    }
    CK(cudaEventRecord(ev1, st));
    CK(cudaStreamSynchronize(st));
    float ms = 0;
    CK(cudaEventElapsedTime(&ms, ev0, ev1));
    adj_ms = ms;
    check_error();
    // the device's box arrays run x fastest, the caller's z fastest; they are turned
    // into the adjoint state's place (24 bytes per cell), three at a time when the box
    // is larger than a third of the grid
    for (size_t i = 0; i < req.size(); ++i) {
      const int* b = req[i].box;
      const int bx = b[1] - b[0], by = b[3] - b[2], bz = b[5] - b[4];
      const size_t nb = size_t(box_cells(b));
      double* const turned = reinterpret_cast<double*>(adj_bufs[i]->lam.p);
      const int per = 9 * nb * sizeof(double) <= adj_bufs[i]->lam.n * sizeof(float) ? 9 : 3;
      for (size_t k = 0; k < 9; k += size_t(per)) {
        const dim3 grid(unsigned((bx + kBoxTile - 1) / kBoxTile), unsigned((bz + kBoxTile - 1) / kBoxTile),
                        unsigned(std::min(per * by, 65535)));
        adj_turn_kernel<<<grid, dim3(kBoxTile, 8), 0, st>>>(adj_bufs[i]->grad.p + k * nb, turned, bx, by, bz, per);
        CK(cudaGetLastError());
        CK(cudaMemcpyAsync(req[i].grad_out + k * nb, turned, per * nb * sizeof(double), cudaMemcpyDeviceToHost, st));
      }
    }
    CK(cudaStreamSynchronize(st));
  }

  // Step n with what a run takes from it: the box histories and the monitors'
  // samples. mon_pending: the samples are not waited for yet. Returns the step
  // kernels launched.
  int step_and_samples(cudaStream_t st, int n, bool& mon_pending) {
    int k = 0;
    if (cfg.variant == 3) {  // the E launch writes the box history of its step
      launch_half(st, n, false, n_caps > 0);
      launch_half(st, n, true, false);
      k = 1;
    } else if (n_caps) {
      // the box history of step n reads buffer n & 1, which step n only
      // reads and step n+1 overwrites: it runs on a side stream beside step n
      CK(cudaEventRecord(cap_fork, st));
      CK(cudaStreamWaitEvent(cap_stream, cap_fork, 0));
      adj_capture_kernel<<<dim3(cap_blocks, unsigned(n_caps)), 256, 0, cap_stream>>>(d_caps.p, n, 0);
      CK(cudaGetLastError());
      CK(cudaEventRecord(cap_join, cap_stream));
    }
    if (cfg.variant != 3) k = launch_step(st, n);
    if (n_caps && cfg.variant != 3) CK(cudaStreamWaitEvent(st, cap_join, 0));
    // The monitors of step n read the buffer that step n + 1 only reads: they
    // run on a side stream beside it, and step n + 2, which overwrites that
    // buffer, waits for them. (The half steps work in place: there the next
    // step waits.)
    if (mon_pending) {
      CK(cudaStreamWaitEvent(st, mon_join, 0));
      mon_pending = false;
    }
    bool sample = false;
    for (auto* s : sims)
      for (const auto& m : s->monitors) sample = sample || monitor_samples(n, m.n_step);
    if (sample) {
      CK(cudaEventRecord(mon_fork, st));
      CK(cudaStreamWaitEvent(mon_stream, mon_fork, 0));
      for (auto* s : sims)
        if (!s->monitors.empty()) {
          int most = 1;
          for (const auto& m : s->monitors) most = std::max(most, m.n1 * m.n2);
          monitor_kernel<<<dim3(unsigned(std::min(64, (most + 127) / 128)), unsigned(s->monitors.size())), 128, 0,
                           mon_stream>>>(s->d_dev.p, s->d_mons.p, n, state_buf(n + 1));
          CK(cudaGetLastError());
        }
      CK(cudaEventRecord(mon_join, mon_stream));
      mon_pending = cfg.variant != 3;
      if (!mon_pending) CK(cudaStreamWaitEvent(st, mon_join, 0));
    }
    return k;
  }

  // Enqueue one full run of nt steps on stream st (used for capture and for
  // direct launches alike).
  void enqueue(cudaStream_t st, int nt) {
    step_launches = dft_launches = 0;
    for (auto* s : sims) {
      CK(cudaMemsetAsync(s->fields.p, 0, s->fields.n * sizeof(float), st));
      if (s->splits.n) CK(cudaMemsetAsync(s->splits.p, 0, s->splits.n * sizeof(float), st));
      if (s->dft_X.n) CK(cudaMemsetAsync(s->dft_X.p, 0, s->dft_X.n * sizeof(double2), st));
      for (size_t m = 0; m < s->monitors.size(); ++m)
        CK(cudaMemsetAsync(s->mon_out[m]->p, 0, s->mon_out[m]->n, st));
    }
    if (scls.d_counter.n) CK(cudaMemsetAsync(scls.d_counter.p, 0, scls.d_counter.n * sizeof(unsigned), st));
    int dft_from = 0;
    bool mon_pending = false;
    auto dft_upto = [&](int n) {  // the DFT of steps dft_from .. n-1, in chunks
      while (dft_from < n) {
        const int to = std::min(n, dft_from / kDftChunk * kDftChunk + kDftChunk);
        for (auto* s : sims)
          if (s->n_series > 0 && s->n_freq > 0) {
            DftDev d{s->n_series, s->n_freq, nt, s->d_series_start.p, s->d_term_probe.p, s->d_term_weight.p,
                     s->d_omega.p, s->rec.p, s->dft_X.p};
            dft_accumulate_kernel<<<dim3(s->n_freq, s->n_series), 256, 0, st>>>(d, dft_from, to);
            CK(cudaGetLastError());
            ++dft_launches;
          }
        dft_from = to;
      }
    };
    if (cfg.variant == 2) {
      // nothing to do between the steps of a launch (also where every launch is asked
      // to come from the host: with one step per launch, which loads and stores the
      // whole state, 120x100x64 cells took 68 us per step, with the streaming
      // kernels 35, so 14)
      for (int n = 0; n < nt;) {
        const int to = std::min(nt, n + kResidentSteps);
        step_launches += launch_steps(st, n, to);
        n = to;
        if (n % kDftChunk == 0 || n == nt) dft_upto(n);
      }
    }
    for (int n = 0; n < nt && cfg.variant != 2; ++n) {
      for (auto* s : sims)
        if (s->ckpt_every > 0 && n % s->ckpt_every == 0 && s->ckpt.n) {
          const size_t N = s->cells_padded, b = size_t(state_buf(n));
          const size_t sb = s->splits.n ? 2 * s->split_buf_pairs : 0;  // split floats per time buffer
          const size_t stride = 6 * N + sb;
          float* dst = s->ckpt.p + size_t(n / s->ckpt_every) * stride;
          CK(cudaMemcpyAsync(dst, s->fields.p + b * 6 * N, 6 * N * sizeof(float), cudaMemcpyDeviceToDevice, st));
          if (sb)
            CK(cudaMemcpyAsync(dst + 6 * N, s->splits.p + b * sb, sb * sizeof(float), cudaMemcpyDeviceToDevice, st));
        }
      step_launches += step_and_samples(st, n, mon_pending);
      if ((n + 1) % kDftChunk == 0 || n + 1 == nt) dft_upto(n + 1);
    }
    if (mon_pending) CK(cudaStreamWaitEvent(st, mon_join, 0));
    // sentinel: a diverged run ends with non-finite records or fields
    for (auto* s : sims) {
      const int64_t nrec = int64_t(s->probes.size()) * nt;
      if (nrec > 0) {
        nonfinite_check_kernel<<<int(std::min<int64_t>(256, (nrec + 255) / 256)), 256, 0, st>>>(s->rec.p, nrec,
                                                                                              d_err.p);
        CK(cudaGetLastError());
      }
      const size_t b = size_t(state_buf(nt)) * 6 * s->cells_padded;  // buffer the last step wrote
      nonfinite_check_kernel<<<296, 256, 0, st>>>(s->fields.p + b, int64_t(6 * s->cells_padded), d_err.p);
      CK(cudaGetLastError());
    }
  }

  // Whether a first run is faster launched from the host. The two tile lists of a
  // streaming step, released together by the step before, start in either order
  // when they come from the host, and where the plain tiles come first the general
  // ones run on alone afterwards; in a graph the general ones go first. Per step
  // and call (a graph's making included), host against graph: 256x256x128 cells with
  // 8-cell layers 197 against 175 us, without 125 against 111; 200x180x128 without
  // 82 against 68; 165x140x100 with 81 against 77, without 39 to 54 against 43; but
  // 150x130x90 without 31 against 35, with 61 against 66; 130x120x80 without 27 to 38
  // against 33. A third branch makes the graph dear (about 70 us for a step with a box
  // history or sampled monitors beside it): 256x256x128 with monitors at every step
  // 235 against 284 us, at every fifth 193 against 219, with a box history 182 against
  // 250.
  // A caller that does not wait for the run gets a graph where the launches would
  // not fit the launch queue (1024): the call would return when most of the run is
  // over (1500 half steps of 128x128x96 cells: after 38 of 57 ms).
  bool direct_first(int nt, bool waits) const {
    if (!waits && cfg.variant != 2 && int64_t(nt) * (sims[0]->monitors.empty() ? 2 : 3) > kDirectLaunches) return false;
    if (cfg.variant != 1 || scls.n_tiles == 0 || scls.n_tiles_p == 0) return true;
    int64_t cells = 0;
    for (auto* s : sims) {
      cells += int64_t(s->nx) * s->ny * s->nz;
      if (s->adj_mode == 2) return true;
      for (const auto& m : s->monitors)
        if (m.n_step < kDirectSamples) return true;
    }
    return cells < kDirectCells;
  }

  // Enqueues a run of nt steps. waits: the caller waits for it at once.
  void run_async(int nt, bool waits) {
    init();
    cudaStream_t st = stream();
    // A time loop's first run is mostly launched from the host, its repetitions
    // replay a graph. Making a graph, launching it the first time and destroying it
    // costs about 5.5 us of host time per node and the GPU waits for it; a launch
    // costs 2 us beside the steps before it (1500 half steps of 120x100x64 cells: 14
    // ms before the first step and 3 ms at the end, then 27 ms of steps).
    bool direct = !use_graph || (graph_nt != nt && direct_nt != nt && direct_first(nt, waits));
    if (direct || graph_nt != nt) {
      reset_graph();
      build_caps();
    }
    if (!direct && graph_nt != nt) {
      graph = capture([&](cudaStream_t cap) { enqueue(cap, nt); });
      direct = !graph.exec;
      if (!direct) graph_nt = nt;
    }
    wait_uploads();
    if (direct && use_graph) direct_nt = nt;
    CK(cudaEventRecord(ev0, st));
    if (direct)
      enqueue(st, nt);
    else
      CK(cudaGraphLaunch(graph.exec, st));
    CK(cudaEventRecord(ev1, st));
    timing_pending = true;
  }

  void sync() {
    CK(cudaStreamSynchronize(stream()));
    if (timing_pending) {
      float ms = 0;
      CK(cudaEventElapsedTime(&ms, ev0, ev1));
      last_ms = ms;
      timing_pending = false;
    }
    check_error();
  }

  // Reads (and clears) the error code the kernels record: a bounded wait that
  // expired, or the end-of-run sentinel's non-finite value.
  void check_error() {
    if (!d_err.n) return;
    int e = 0;
    CK(cudaMemcpy(&e, d_err.p, sizeof(int), cudaMemcpyDeviceToHost));
    if (e) {
      CK(cudaMemset(d_err.p, 0, sizeof(int)));
      if (e == kErrNonFinite)
        throw ArgError{FDTD_ERR_NONFINITE, "the run diverged: a probe record or a field value is not finite"};
      if (e == kErrFaceExpired)
        throw ArgError{FDTD_ERR_DEVICE, "resident step kernel gave up waiting for a neighbouring brick's faces"};
      throw ArgError{FDTD_ERR_DEVICE, "step kernel gave up waiting for a TMA plane load (code " +
                                          std::to_string(e) + ")"};
    }
  }
};

namespace {

// Geometry of the split stores of a plan (SplitDev without base pointers);
// returns the pairs one time buffer holds. z and y stores span whole x rows
// (pitch); x stores span the core y rows and an even number of pairs from an
// even origin, so their rows and TMA boxes start on 16 bytes.
size_t split_layout(const SplitPlan& plan, int nx, int ny, int nz, int pitch, SplitDev& g) {
  g = SplitDev{};
  const int* t = plan.t;
  for (int k = 0; k < 6; ++k) g.t[k] = t[k];
  const int zc0 = t[4], zc = std::max(0, nz - t[4] - t[5]);
  auto set = [&](int st, int ox, int oy, int oz, int w, int h, int d) {
    g.ox[st] = ox; g.oy[st] = oy; g.oz[st] = oz; g.w[st] = w; g.h[st] = h;
    g.comp[st] = int64_t(w) * h * d;
  };
  set(kStZlo, 0, 0, 0, pitch, ny, t[4]);
  set(kStZhi, 0, 0, nz - t[5], pitch, ny, t[5]);
  set(kStYlo, 0, 0, zc0, pitch, t[2], zc);
  set(kStYhi, 0, ny - t[3], zc0, pitch, t[3], zc);
  const int yc = std::max(0, ny - t[2] - t[3]);
  const int wxl = t[0] ? (t[0] + 1) & ~1 : 0;
  const int oxh = (nx - t[1]) & ~1;
  const int wxh = t[1] ? (nx - oxh + 1) & ~1 : 0;
  set(kStXlo, 0, t[2], zc0, wxl, yc, zc);
  set(kStXhi, oxh, t[2], zc0, wxh, yc, zc);
  int64_t off = 0;
  for (int st = 0; st < 6; ++st) {
    g.off[st] = off;
    off += 6 * g.comp[st];
  }
  g.off[kStSparse] = off;
  off += 6 * plan.n_sparse;
  return size_t(off);
}

void compile_host(fdtd_sim* s) {
  if (s->compiled) return;
  for (int i = 0; i < kNumCoef; ++i)
    if (!s->have_coef[i]) throw ArgError{FDTD_ERR_STATE, std::string("Coefficient not set: ") + kCoefNames[i]};
  const float* cp[kNumCoef];
  for (int i = 0; i < kNumCoef; ++i) cp[i] = s->coef_view[i] ? s->coef_view[i] : s->coef[i].data();
  std::string err;
  if (!compile_grid(s->nx, s->ny, s->nz, cp, s->probes, threads_for_host(), s->grid, err))
    throw ArgError{FDTD_ERR_LIMIT, err};
  if (!plan_split_storage(s->grid, s->split_plan, err)) throw ArgError{FDTD_ERR_LIMIT, err};
  s->compiled = true;
  s->base_rows = int(s->grid.rows.size());
  s->box_rows_from = -1;
}

void prepare(fdtd_sim* s, int nt) {
  if (s->prepared && s->prepared_nt == nt) return;
  for (size_t p = 0; p < s->probe_values.size(); ++p)
    if (s->probes[p].is_source && int(s->probe_values[p].size()) < nt)
      throw ArgError{FDTD_ERR_ARG, "Invalid data source array shape. Expected shape greater or equal to " +
                                       std::to_string(nt)};
  const int nx = s->nx, ny = s->ny, nz = s->nz;
  if (!s->prepared) {
    compile_host(s);
    ++s->generation;
    s->prepared_nt = -1;
    s->pitch = ((nx + 31) / 32) * 32;
    s->cells_padded = size_t(nz) * ny * s->pitch;
    if (s->cells_padded >= (size_t(1) << 31) - size_t(2) * ny * s->pitch)
      throw ArgError{FDTD_ERR_LIMIT, "Grid too large for 32-bit cell offsets."};
    const size_t N = s->cells_padded;
    s->fields.alloc(12 * N);
    // split pairs only in the slab stores and the sparse store
    s->split_buf_pairs = split_layout(s->split_plan, nx, ny, nz, s->pitch, s->split_geo);
    for (int st = 0; st < 6; ++st)  // the kernels step between a store's components with 32-bit strides
      if (6 * s->split_geo.comp[st] >= (int64_t(1) << 31))
        throw ArgError{FDTD_ERR_LIMIT, "PML slab too large for 32-bit split-pair offsets."};
    const bool any_split = s->grid.e_split_cells > 0 || s->grid.h_split_cells > 0;
    s->splits.alloc(any_split ? 2 * 2 * s->split_buf_pairs : 0);
    // material index: upload in reference order, transpose on the device
    {
      DevBuf<uint16_t> tmp;
      tmp.alloc(s->grid.ids.size());
      h2d(s, tmp.p, s->grid.ids.data(), s->grid.ids.size() * 2);
      s->mat.alloc(N);
      CK(cudaMemset(s->mat.p, 0, N * 2));
      transpose_ids_kernel<<<1024, 256>>>(tmp.p, s->mat.p, nx, ny, nz, s->pitch);
      CK(cudaGetLastError());
      CK(device_wait());
    }
    s->rows.alloc(s->grid.rows.size() * 8);
    h2d(s, s->rows.p, s->grid.rows.data(), s->grid.rows.size() * sizeof(Row));
    s->cell_probes.alloc(std::max<size_t>(1, s->grid.cell_probes.size()));
    if (!s->grid.cell_probes.empty())
      h2d(s, s->cell_probes.p, s->grid.cell_probes.data(), s->grid.cell_probes.size() * sizeof(int2));
    std::vector<int> srcflag(std::max<size_t>(1, s->probes.size()), 0);
    for (size_t p = 0; p < s->probes.size(); ++p) srcflag[p] = s->probes[p].is_source;
    s->is_src.alloc(srcflag.size());
    h2d(s, s->is_src.p, srcflag.data(), srcflag.size() * sizeof(int));
    s->prepared = true;
  }
  for (const auto& m : s->monitors)
    if (m.n_freq && m.n_phase_rows < nt / m.n_step + 1)
      throw ArgError{FDTD_ERR_ARG, "Monitor phase table has fewer rows than nt/n_step + 1."};
  // per-nt buffers: source amplitudes, records, DFT, monitors
  ++s->generation;
  s->prepared_nt = -1;  // until all of them are in place
  const size_t P = s->probes.size();
  s->src.alloc(std::max<size_t>(1, P * size_t(nt)));
  s->rec.alloc(std::max<size_t>(1, P * size_t(nt)));
  {
    std::vector<float> host(std::max<size_t>(1, P * size_t(nt)), 0.f);
    for (size_t p = 0; p < P; ++p)
      if (s->probes[p].is_source)
        std::memcpy(&host[p * nt], s->probe_values[p].data(), size_t(nt) * sizeof(float));
    h2d(s, s->src.p, host.data(), host.size() * sizeof(float));
  }
  if (s->n_series > 0) {
    s->d_series_start.alloc(s->series_start.size());
    h2d(s, s->d_series_start.p, s->series_start.data(), s->series_start.size() * 4);
    s->d_term_probe.alloc(std::max<size_t>(1, s->term_probe.size()));
    if (!s->term_probe.empty())
      h2d(s, s->d_term_probe.p, s->term_probe.data(), s->term_probe.size() * 4);
    s->d_term_weight.alloc(std::max<size_t>(1, s->term_weight.size()));
    if (!s->term_weight.empty())
      h2d(s, s->d_term_weight.p, s->term_weight.data(), s->term_weight.size() * 8);
    s->d_omega.alloc(s->omega.size());
    h2d(s, s->d_omega.p, s->omega.data(), s->omega.size() * 8);
    s->dft_X.alloc(size_t(s->n_series) * s->n_freq);
  }
  std::vector<MonDev> mdev;
  s->mon_out.clear();
  s->mon_phase.clear();
  for (auto& m : s->monitors) {
    auto out = std::make_unique<DevBuf<char>>();
    out->alloc(m.out_bytes(nt));
    auto ph = std::make_unique<DevBuf<float2>>();
    if (m.n_freq) {
      ph->alloc(m.phase.size() / 2);
      h2d(s, ph->p, m.phase.data(), m.phase.size() * 4);
    }
    mdev.push_back(MonDev{m.field, m.axis, m.position, m.n_step, m.n_freq, m.n1, m.n2, out->p, ph->p});
    s->mon_out.push_back(std::move(out));
    s->mon_phase.push_back(std::move(ph));
  }
  s->d_mons.alloc(mdev.size());
  if (!mdev.empty())
    h2d(s, s->d_mons.p, mdev.data(), mdev.size() * sizeof(MonDev));

  // descriptor
  SimDev& d = s->dev;
  const size_t N = s->cells_padded;
  d.nx = nx; d.ny = ny; d.nz = nz; d.pitch = s->pitch; d.plane = ny * s->pitch; d.nt = nt;
  for (int b = 0; b < 2; ++b) {
    for (int c = 0; c < 3; ++c) {
      d.E[b][c] = s->fields.p + (size_t(b) * 6 + c) * N;
      d.H[b][c] = s->fields.p + (size_t(b) * 6 + 3 + c) * N;
    }
    // split pairs of time buffer b: the stores back to back
    d.sp = s->split_geo;
    for (int bb = 0; bb < 2; ++bb)
      d.sp.base[bb] = s->splits.n ? reinterpret_cast<float2*>(s->splits.p) + size_t(bb) * s->split_buf_pairs : nullptr;
  }
  d.mat = s->mat.p;
  d.rows = s->rows.p;
  d.cell_probes = s->cell_probes.p;
  d.src = s->src.p;
  d.rec = s->rec.p;
  d.is_src = s->is_src.p;
  d.cells = int64_t(N);
  s->d_dev.alloc(1);
  h2d(s, s->d_dev.p, &d, sizeof(SimDev));
  s->prepared_nt = nt;
}

void fill_stats(fdtd_sim* s, const Engine* e) {
  fdtd_stats& st = s->stats;
  st.nx = s->nx; st.ny = s->ny; st.nz = s->nz; st.nt = s->prepared_nt;
  st.n_rows = int(s->grid.rows.size());
  st.id_bytes = 2;
  st.e_split_cells = s->grid.e_split_cells;
  st.h_split_cells = s->grid.h_split_cells;
  st.compile_ms = s->grid.compile_ms;
  st.h2d_bytes = s->h2d_bytes;
  st.d2h_bytes = s->d2h_bytes;
  if (e) {
    st.variant = e->cfg.variant;
    st.tile_y = e->cfg.variant != 0 ? e->cfg.ty : kTileY;
    st.stages = e->cfg.variant != 0 ? e->cfg.stages : 0;
    st.zchunk = e->zchunk_used;
    st.grid = e->grid;
    st.n_tiles = e->n_tiles;
    st.step_launches = e->step_launches;
    st.dft_launches = e->dft_launches;
    st.last_run_ms = e->last_ms;
    st.tune_ms = e->tune_ms;
    st.tune_trials = e->tune_trials;
  }
}

template <typename F>
int guarded(std::string* err, F&& f) {
  try {
    f();
    return FDTD_OK;
  } catch (const ArgError& a) {
    if (err) *err = a.msg;
    return a.code;
  } catch (const CudaError& c) {
    if (err) *err = c.where + ": " + cudaGetErrorString(c.code);
    return FDTD_ERR_CUDA;
  } catch (const std::bad_alloc&) {
    if (err) *err = "host allocation failed";
    return FDTD_ERR_LIMIT;
  } catch (const std::exception& e) {
    if (err) *err = e.what();
    return FDTD_ERR_ARG;
  }
}

int coef_index(const char* name) {
  for (int i = 0; i < kNumCoef; ++i)
    if (std::strcmp(name, kCoefNames[i]) == 0) return i;
  return -1;
}

}  // namespace

// Drops what the last run kept for a gradient (snapshots or box history); the
// engines whose graphs write there, or whose kernel suited the old mode, are
// rebuilt.
void leave_adjoint_mode(fdtd_sim* s) {
  ++s->generation;
  s->adj_mode = 0;
  s->adj_in_batch = false;
  s->ckpt_every = 0;
  s->ckpt_nt = -1;
  s->ckpt.free();
  s->hist.free();
  std::fill(s->adj_box, s->adj_box + 6, 0);
}

// A fresh single-simulation engine for s (descriptors, tiles, graph).
void new_engine(fdtd_sim* s) {
  s->engine.reset();
  s->engine = std::make_unique<Engine>();
  s->engine->sims = {s};
  s->engine->asked = s->cfg;
  s->engine->ext_stream = s->ext_stream;
  s->engine->use_graph = s->use_graph;
  s->engine->wait_limit = s->dbg_wait_limit;
  s->engine->withhold = s->dbg_withhold;
  s->engine->build_tiles();
  s->engine_gen = s->generation;
}

// Whether s's own engine was built on the device buffers as they are: a batch
// run of s with another number of steps moves them too.
bool engine_current(const fdtd_sim* s) { return s->engine && s->engine_gen == s->generation; }

// A gradient box must be non-empty, inside the grid and free of cells with
// split E storage (PML slabs, source cells): the gradient treats the box
// cells' E pairs as one total with one Ca.
void check_gradient_box(const fdtd_sim* s, const int* box) {
  if (box[0] < 0 || box[2] < 0 || box[4] < 0 || box[1] > s->nx || box[3] > s->ny || box[5] > s->nz ||
      box[0] >= box[1] || box[2] >= box[3] || box[4] >= box[5])
    throw ArgError{FDTD_ERR_ARG, "gradient box must be a non-empty box inside the grid."};
  for (int x = box[0]; x < box[1]; ++x)
    for (int y = box[2]; y < box[3]; ++y)
      for (int z = box[4]; z < box[5]; ++z) {
        const uint32_t f = s->grid.rows[s->grid.ids[(size_t(x) * s->ny + y) * s->nz + z]].w[R_FLAGS];
        if (f & kFlagESplit) throw ArgError{FDTD_ERR_ARG, "gradient box holds split-field (PML or source) cells."};
      }
}

// The members of a batch run in parts, one part after the other on one stream,
// the members of a part in the same launches.
struct fdtd_batch {
  std::vector<fdtd_sim*> sims;
  KernelConfig asked;
  cudaStream_t ext_stream = nullptr;
  std::vector<std::unique_ptr<Engine>> parts;
  std::vector<std::vector<size_t>> members;  // of each part
  int run_nt = -1;        // steps the parts' graphs were made for
  bool dirty = true;
  std::vector<int> gens;  // members' device-buffer generations the parts were built on
  std::string err;
  fdtd_stats stats{};
};

// Which members step together. Members are independent, so one that fills the
// GPU alone is best stepped alone: it takes the kernel that suits it (the
// resident one holds up to a million cells) and its state stays in L2,
// while all states together do not. Eight members of 0.12 to 1.1 M cells: 151 us
// per step together, 102 one after the other. Small members share launches,
// whose latency is then paid once, the more the cheaper. Per member and step, in
// parts of up to 1.2 M cells, together against alone: 22k cells 3.2 (two members),
// 2.0 (four), 1.2 (32) against 3.2 us; 47k 3.0 (three), 2.6 (eight), 2.8 (32)
// against 3.3; 60k 3.9 (three), 3.3 (five), 3.0 (eight), 2.9 (32) against 3.6; 85k
// 4.9 (three), 4.2 (five), 3.9 (six), 3.7 (32) against 4.0; 110k 5.0 (three), 4.8
// (six to 32) against 4.3; 200k 8.5 against 5.1. For a gradient, whose steps are two or four launches: four members of 75k cells 14.9
// against 21.8 ms, 192k cells 24.8 against 28.9 ms, 346k cells 39.9 against 35.3
// ms; six of 590k cells 96 against 78 ms; two of 2.3 M 36 against 34 ms. From where
// the reverse step no longer works in L2 the members' shared launches only save
// their ends: two of 3.5 M cells 50 against 50 ms, of 4.6 M 62 against 66 (without
// layers 48 against 55), of 8.4 M 100 against 104.
std::vector<std::vector<size_t>> batch_parts(const fdtd_batch* b) {
  std::vector<std::vector<size_t>> out;
  std::vector<size_t> small;  // members that step together
  auto cells = [&](size_t i) { return int64_t(b->sims[i]->nx) * b->sims[i]->ny * b->sims[i]->nz; };
  const bool automatic = b->asked.variant == 1 && b->asked.ty == 0, run = b->sims[0]->adj_mode == 0;
  auto below = [&](int64_t limit) {
    std::vector<size_t> v;
    for (size_t i = 0; i < b->sims.size(); ++i)
      if (!automatic || cells(i) < limit) v.push_back(i);
    return v;
  };
  if (!automatic || !run) {
    small = below(kBatchSmallGradient);
  } else {
    for (const auto& r : kBatchTogether)
      if (small.empty() && below(r.cells).size() >= r.members) small = below(r.cells);
  }
  int large = -1;  // the part of a gradient's largest members
  for (size_t i = 0; i < b->sims.size(); ++i) {
    if (std::binary_search(small.begin(), small.end(), i)) continue;
    const bool shares = !run && cells(i) >= kBatchLargeGradient;
    if (shares && large >= 0) {
      out[size_t(large)].push_back(i);
    } else {
      if (shares) large = int(out.size());
      out.push_back({i});
    }
  }
  int64_t room = 0;
  for (size_t i : small) {
    if ((automatic && room < cells(i)) || room == 0) {
      out.emplace_back();
      room = kBatchCells;
    }
    out.back().push_back(i);
    room -= automatic ? cells(i) : 0;
  }
  return out;
}

// All parts use one stream: the caller's, or the first part's own.
void set_batch_streams(fdtd_batch* b) {
  for (auto& e : b->parts) {
    e->ext_stream = e == b->parts[0] ? b->ext_stream : b->parts[0]->stream();
    e->init();
  }
}

// (Re)builds the parts for the members as prepared.
void build_batch(fdtd_batch* b, int nt) {
  auto members = batch_parts(b);
  if (members != b->members) {
    for (auto& e : b->parts) cudaStreamSynchronize(e->stream());
    b->parts.clear();
    b->members = std::move(members);
    for (const auto& m : b->members) {
      b->parts.push_back(std::make_unique<Engine>());
      for (size_t i : m) b->parts.back()->sims.push_back(b->sims[i]);
    }
  }
  b->run_nt = -1;
  set_batch_streams(b);
  for (auto& e : b->parts) {
    e->asked = b->asked;
    e->graph_nt = -1;
    e->build_tiles();
  }
  b->run_nt = nt;
  b->dirty = false;  // (a call refused before this leaves a chosen kernel for the next)
}

// Runs nt steps of every part and reports the first error after all have ended.
void run_batch(fdtd_batch* b, int nt) {
  std::exception_ptr first;
  set_batch_streams(b);
  for (auto& e : b->parts) e->run_async(nt, true);
  for (auto& e : b->parts) {
    try {
      e->sync();
    } catch (...) {
      if (!first) first = std::current_exception();
    }
  }
  if (first) std::rethrow_exception(first);
  for (size_t k = 0; k < b->parts.size(); ++k)
    for (size_t i : b->members[k]) fill_stats(b->sims[i], b->parts[k].get());
}

// Times and trials summed over the parts; a launch of every part counts once.
void batch_run_stats(fdtd_batch* b, int nt) {
  fdtd_stats& st = b->stats;
  st.nt = nt;
  st.last_run_ms = st.tune_ms = 0;
  st.step_launches = st.tune_trials = 0;
  for (const auto& e : b->parts) {
    st.last_run_ms += e->last_ms;
    st.tune_ms += e->tune_ms;
    st.tune_trials += e->tune_trials;
    st.step_launches = std::max<int64_t>(st.step_launches, e->step_launches);
  }
}

// Whether a member's device buffers moved since the batch engine was built.
bool batch_moved(const fdtd_batch* b) {
  if (b->gens.size() != b->sims.size()) return true;
  for (size_t i = 0; i < b->sims.size(); ++i)
    if (b->gens[i] != b->sims[i]->generation) return true;
  return false;
}

void note_generations(fdtd_batch* b) {
  b->gens.clear();
  for (auto* s : b->sims) b->gens.push_back(s->generation);
}

// Material index of the box cells on the device: ids [x][y][z] of the box.
__global__ void set_box_ids_kernel(uint16_t* mat, int ny, int pitch, int x0, int y0, int z0, int bnx, int bny,
                                   int bnz, const uint16_t* ids) {
  const int64_t nb = int64_t(bnx) * bny * bnz;
  for (int64_t i = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; i < nb; i += int64_t(gridDim.x) * blockDim.x) {
    const int zz = int(i % bnz), yy = int((i / bnz) % bny), xx = int(i / (int64_t(bnz) * bny));
    mat[size_t(z0 + zz) * ny * pitch + size_t(y0 + yy) * pitch + (x0 + xx)] = ids[i];
  }
}

// E-update coefficients of a box: host arrays, and the compiled table when
// there is one (one dedicated row per box cell after the compiled rows).
void set_box_coefficients(fdtd_sim* s, const int* box, const float* coefs) {
  static const char* const names[3][4] = {{"Ca_ex_y", "Ca_ex_z", "Cb_ex_y", "Cb_ex_z"},
                                           {"Ca_ey_z", "Ca_ey_x", "Cb_ey_z", "Cb_ey_x"},
                                           {"Ca_ez_x", "Ca_ez_y", "Cb_ez_x", "Cb_ez_y"}};
  if (box[0] < 0 || box[2] < 0 || box[4] < 0 || box[1] > s->nx || box[3] > s->ny || box[5] > s->nz ||
      box[0] >= box[1] || box[2] >= box[3] || box[4] >= box[5])
    throw ArgError{FDTD_ERR_ARG, "box must be a non-empty box inside the grid."};
  int ci[3][4];
  for (int c = 0; c < 3; ++c)
    for (int k = 0; k < 4; ++k) {
      ci[c][k] = coef_index(names[c][k]);
      if (!s->have_coef[ci[c][k]])
        throw ArgError{FDTD_ERR_STATE, std::string("Coefficient not set: ") + names[c][k]};
    }
  if (s->compiled) check_gradient_box(s, box);
  for (int c = 0; c < 3; ++c)  // the patch writes the host arrays: copy borrowed ones first
    for (int k = 0; k < 4; ++k) {
      const int i = ci[c][k];
      if (s->coef_view[i]) {
        s->coef[i].assign(s->coef_view[i], s->coef_view[i] + size_t(s->nx) * s->ny * s->nz);
        s->coef_view[i] = nullptr;
      }
    }
  const int bny = box[3] - box[2], bnz = box[5] - box[4];
  const int64_t nb = box_cells(box);
  auto cell_of = [&](int64_t bi) {
    const int zz = int(bi % bnz), yy = int((bi / bnz) % bny), xx = int(bi / (int64_t(bnz) * bny));
    return (size_t(box[0] + xx) * s->ny + (box[2] + yy)) * s->nz + (box[4] + zz);
  };
  for (int64_t bi = 0; bi < nb; ++bi) {
    const size_t cell = cell_of(bi);
    for (int c = 0; c < 3; ++c) {
      const float ca = coefs[(3 * c + 0) * nb + bi], cb1 = coefs[(3 * c + 1) * nb + bi],
                  cb2 = coefs[(3 * c + 2) * nb + bi];
      s->coef[ci[c][0]][cell] = ca;
      s->coef[ci[c][1]][cell] = ca;
      s->coef[ci[c][2]][cell] = cb1;
      s->coef[ci[c][3]][cell] = cb2;
    }
  }
  if (!s->compiled) return;  // the next run compiles the arrays
  if (s->engine) CK(cudaStreamSynchronize(s->engine->stream()));
  std::vector<uint16_t>& ids = s->grid.ids;
  std::vector<Row>& rows = s->grid.rows;
  bool new_ids = false;
  if (s->box_rows_from >= 0 && !std::equal(box, box + 6, s->box_rows_box)) {
    // another box: the next run compiles the patched arrays afresh
    s->compiled = false;
    s->prepared = false;
    return;
  }
  if (s->box_rows_from < 0) {
    if (int64_t(s->base_rows) + nb > 65536)
      throw ArgError{FDTD_ERR_LIMIT, "box needs more rows than the 16-bit material index can address."};
    s->box_rows_from = s->base_rows;
    std::copy(box, box + 6, s->box_rows_box);
    rows.resize(size_t(s->base_rows) + size_t(nb));
    for (int64_t bi = 0; bi < nb; ++bi) {
      const size_t cell = cell_of(bi);
      rows[size_t(s->base_rows + bi)] = rows[ids[cell]];
      ids[cell] = uint16_t(s->base_rows + bi);
    }
    new_ids = true;
  }
  for (int64_t bi = 0; bi < nb; ++bi) {
    Row& r = rows[size_t(s->box_rows_from + bi)];
    for (int c = 0; c < 3; ++c) {
      const float ca = coefs[(3 * c + 0) * nb + bi], cb1 = coefs[(3 * c + 1) * nb + bi],
                  cb2 = coefs[(3 * c + 2) * nb + bi];
      std::memcpy(&r.w[4 * c + 0], &ca, 4);
      std::memcpy(&r.w[4 * c + 1], &cb1, 4);
      std::memcpy(&r.w[4 * c + 2], &ca, 4);
      std::memcpy(&r.w[4 * c + 3], &cb2, 4);
    }
  }
  if (!s->prepared) return;  // the next run uploads the table
  if (s->rows.n < rows.size() * 8) {
    // a larger table: every descriptor holding the old pointer is rebuilt
    s->rows.alloc(rows.size() * 8);
    h2d(s, s->rows.p, rows.data(), rows.size() * sizeof(Row));
    s->dev.rows = s->rows.p;
    h2d(s, s->d_dev.p, &s->dev, sizeof(SimDev));
    ++s->generation;
    s->engine.reset();
  } else {
    h2d(s, s->rows.p + size_t(s->box_rows_from) * 8, rows.data() + s->box_rows_from, size_t(nb) * sizeof(Row));
  }
  if (new_ids) {
    std::vector<uint16_t> bids(static_cast<size_t>(nb));
    for (int64_t bi = 0; bi < nb; ++bi) bids[size_t(bi)] = uint16_t(s->box_rows_from + bi);
    DevBuf<uint16_t> tmp;
    tmp.alloc(bids.size());
    h2d(s, tmp.p, bids.data(), bids.size() * 2);
    set_box_ids_kernel<<<256, 256>>>(s->mat.p, s->ny, s->pitch, box[0], box[2], box[4], box[1] - box[0], bny, bnz,
                                     tmp.p);
    CK(cudaGetLastError());
    CK(device_wait());
  }
}

extern "C" {

int fdtd_set_box_coefficients(fdtd_sim* s, const int* box, const float* coefs) {
  if (!s) return FDTD_ERR_ARG;
  return guarded(&s->err, [&] {
    if (!box || !coefs) throw ArgError{FDTD_ERR_ARG, "null argument"};
    set_box_coefficients(s, box, coefs);
  });
}

int fdtd_create(int nx, int ny, int nz, fdtd_sim** out) {
  if (!out) {
    g_error = "fdtd_create: null output pointer";
    return FDTD_ERR_ARG;
  }
  *out = nullptr;
  if (nx < 2 || ny < 2 || nz < 2 || nx > 65535 || ny > 65535 || nz > 65535) {
    g_error = "Grid dimensions must be between 2 and 65535 cells.";
    return FDTD_ERR_ARG;
  }
  auto* s = new (std::nothrow) fdtd_sim();
  if (!s) {
    g_error = "host allocation failed";
    return FDTD_ERR_LIMIT;
  }
  s->nx = nx;
  s->ny = ny;
  s->nz = nz;
  *out = s;
  return FDTD_OK;
}

int fdtd_set_coefficient(fdtd_sim* s, const char* name, const float* data, int nx, int ny, int nz) {
  if (!s) return FDTD_ERR_ARG;
  return guarded(&s->err, [&] {
    const int i = name ? coef_index(name) : -1;
    if (i < 0) throw ArgError{FDTD_ERR_ARG, std::string("Unknown coefficient array ") + (name ? name : "(null)")};
    const int expect[3] = {s->nx, s->ny, s->nz}, got[3] = {nx, ny, nz};
    for (int a = 0; a < 3; ++a)
      if (expect[a] != got[a])
        throw ArgError{FDTD_ERR_ARG, std::string("Invalid data array ") + name + ". Expected shape on axis " +
                                         std::to_string(a) + " of " + std::to_string(expect[a])};
    if (!data) throw ArgError{FDTD_ERR_ARG, "null coefficient data"};
    s->coef[i].assign(data, data + size_t(nx) * ny * nz);
    s->coef_view[i] = nullptr;
    s->have_coef[i] = true;
    s->prepared = false;
    s->compiled = false;
  });
}

int fdtd_set_coefficient_view(fdtd_sim* s, const char* name, const float* data, int nx, int ny, int nz) {
  if (!s) return FDTD_ERR_ARG;
  return guarded(&s->err, [&] {
    const int i = name ? coef_index(name) : -1;
    if (i < 0) throw ArgError{FDTD_ERR_ARG, std::string("Unknown coefficient array ") + (name ? name : "(null)")};
    const int expect[3] = {s->nx, s->ny, s->nz}, got[3] = {nx, ny, nz};
    for (int a = 0; a < 3; ++a)
      if (expect[a] != got[a])
        throw ArgError{FDTD_ERR_ARG, std::string("Invalid data array ") + name + ". Expected shape on axis " +
                                         std::to_string(a) + " of " + std::to_string(expect[a])};
    if (!data) throw ArgError{FDTD_ERR_ARG, "null coefficient data"};
    std::vector<float>().swap(s->coef[i]);
    s->coef_view[i] = data;
    s->have_coef[i] = true;
    s->prepared = false;
    s->compiled = false;
  });
}

int fdtd_add_probe(fdtd_sim* s, int field, int i, int j, int k, int is_source, const float* values, int n_values,
                   int* index) {
  if (!s) return FDTD_ERR_ARG;
  return guarded(&s->err, [&] {
    if (field < 0 || field > 5) throw ArgError{FDTD_ERR_ARG, "Invalid probe field type."};
    if (int(s->probes.size()) >= kMaxProbes) throw ArgError{FDTD_ERR_LIMIT, "Exceeded maximum number of probes."};
    if (is_source && (!values || n_values < 0)) throw ArgError{FDTD_ERR_ARG, "Source probe needs values."};
    s->probes.push_back(ProbeSpec{field, i, j, k, is_source ? 1 : 0});
    s->probe_values.emplace_back();
    if (values && n_values > 0) s->probe_values.back().assign(values, values + n_values);
    if (index) *index = int(s->probes.size()) - 1;
    s->prepared = false;
    s->compiled = false;
  });
}

int fdtd_add_monitor(fdtd_sim* s, int field, int axis, int position, int n_step, int n_freq, const float* phase,
                     int n_phase_rows, int* index) {
  if (!s) return FDTD_ERR_ARG;
  return guarded(&s->err, [&] {
    if (int(s->monitors.size()) >= kMaxMonitors)
      throw ArgError{FDTD_ERR_LIMIT, "Exceeded maximum number of monitors."};
    if (field < 0 || field > 5 || axis < 0 || axis > 2 || n_step < 1 || n_freq < 0)
      throw ArgError{FDTD_ERR_ARG, "Invalid monitor field, axis, n_step or n_frequencies."};
    Monitor m{};
    m.field = field;
    m.axis = axis;
    m.n_step = n_step;
    m.n_freq = n_freq;
    // GPU-layout position shift of solver_init_monitors (solver.cpp:394-441, gpu = 1)
    int pos = position;
    if (axis == 0 && (field == 3 || field == 1 || field == 2)) pos -= 1;
    if (axis == 1 && (field == 4 || field == 0 || field == 2)) pos -= 1;
    if (axis == 2 && (field == 5 || field == 0 || field == 1)) pos -= 1;
    m.position = pos;
    m.n1 = axis == 0 ? s->ny : s->nx;
    m.n2 = axis == 2 ? s->ny : s->nz;
    if (n_freq) {
      if (!phase || n_phase_rows < 1) throw ArgError{FDTD_ERR_ARG, "Phasor monitor needs a dtft_phase table."};
      m.phase.assign(phase, phase + size_t(n_phase_rows) * n_freq * 2);
      m.n_phase_rows = n_phase_rows;
    }
    s->monitors.push_back(std::move(m));
    if (index) *index = int(s->monitors.size()) - 1;
    s->prepared_nt = -1;
  });
}

int fdtd_set_dft(fdtd_sim* s, int n_series, int n_terms, const int* term_series, const int* term_probe,
                 const double* term_weight, int n_freq, const double* omega) {
  if (!s) return FDTD_ERR_ARG;
  return guarded(&s->err, [&] {
    if (n_series < 0 || n_terms < 0 || n_freq < 0) throw ArgError{FDTD_ERR_ARG, "Negative DFT size."};
    if (n_series > 0 && n_freq > 0 && (!omega || (n_terms > 0 && (!term_series || !term_probe || !term_weight))))
      throw ArgError{FDTD_ERR_ARG, "null DFT array"};
    std::vector<std::vector<std::pair<int, double>>> per(n_series);
    for (int t = 0; t < n_terms; ++t) {
      if (term_series[t] < 0 || term_series[t] >= n_series)
        throw ArgError{FDTD_ERR_ARG, "DFT term refers to a series out of range."};
      if (term_probe[t] < 0 || term_probe[t] >= int(s->probes.size()))
        throw ArgError{FDTD_ERR_ARG, "DFT term refers to a probe out of range (add probes first)."};
      per[term_series[t]].emplace_back(term_probe[t], term_weight[t]);
    }
    s->n_series = n_series;
    s->n_freq = n_freq;
    s->series_start.assign(1, 0);
    s->term_probe.clear();
    s->term_weight.clear();
    for (auto& v : per) {
      for (auto& pw : v) {
        s->term_probe.push_back(pw.first);
        s->term_weight.push_back(pw.second);
      }
      s->series_start.push_back(int(s->term_probe.size()));
    }
    s->omega.assign(omega, omega + n_freq);
    s->prepared_nt = -1;
  });
}

int fdtd_compile(fdtd_sim* s, int* n_rows, int64_t* e_split_cells, int64_t* h_split_cells) {
  if (!s) return FDTD_ERR_ARG;
  return guarded(&s->err, [&] {
    compile_host(s);
    if (n_rows) *n_rows = int(s->grid.rows.size());
    if (e_split_cells) *e_split_cells = s->grid.e_split_cells;
    if (h_split_cells) *h_split_cells = s->grid.h_split_cells;
  });
}

int fdtd_get_material_table(fdtd_sim* s, uint16_t* ids, int64_t n_ids, uint32_t* rows, int n_rows) {
  if (!s) return FDTD_ERR_ARG;
  return guarded(&s->err, [&] {
    if (!s->compiled) throw ArgError{FDTD_ERR_STATE, "Material table not compiled."};
    if (ids) {
      if (size_t(n_ids) != s->grid.ids.size()) throw ArgError{FDTD_ERR_ARG, "ids size mismatch."};
      std::memcpy(ids, s->grid.ids.data(), s->grid.ids.size() * 2);
    }
    if (rows) {
      if (size_t(n_rows) != s->grid.rows.size()) throw ArgError{FDTD_ERR_ARG, "rows size mismatch."};
      std::memcpy(rows, s->grid.rows.data(), s->grid.rows.size() * sizeof(Row));
    }
  });
}

int fdtd_set_kernel(fdtd_sim* s, int variant, int tile_y, int stages, int zchunk) {
  if (!s) return FDTD_ERR_ARG;
  return guarded(&s->err, [&] {
    if (variant < 0 || variant > 1)
      throw ArgError{FDTD_ERR_ARG, "variant must be 0 (plain) or 1 (stream)"};
    if (!kernel_exists(variant, tile_y, stages))
      throw ArgError{FDTD_ERR_ARG, "No kernel instantiated for this variant / tile height / stage count."};
    KernelConfig c;
    c.variant = variant;
    c.ty = tile_y;
    c.stages = stages;
    c.zchunk = zchunk;
    c.one_list = one_list_env();
    s->cfg = c;
    s->engine.reset();
  });
}

int fdtd_set_graph(fdtd_sim* s, int enabled) {
  if (!s) return FDTD_ERR_ARG;
  s->use_graph = enabled != 0;
  if (s->engine) {
    s->engine->use_graph = s->use_graph;
    s->engine->reset_graph();
  }
  return FDTD_OK;
}

int fdtd_set_debug(fdtd_sim* s, unsigned wait_limit, int withhold_plane) {
  if (!s) return FDTD_ERR_ARG;
  s->dbg_wait_limit = wait_limit ? wait_limit : kStreamWaitLimit;
  s->dbg_withhold = withhold_plane < 0 ? -1 : withhold_plane;
  if (s->engine) {
    s->engine->wait_limit = s->dbg_wait_limit;
    s->engine->withhold = s->dbg_withhold;
    s->engine->reset_graph();
  }
  return FDTD_OK;
}

int fdtd_set_stream(fdtd_sim* s, void* stream) {
  if (!s) return FDTD_ERR_ARG;
  s->ext_stream = static_cast<cudaStream_t>(stream);
  if (s->engine) s->engine->ext_stream = s->ext_stream;
  return FDTD_OK;
}

static int start_run(fdtd_sim* s, int nt, bool waits) {
  if (!s) return FDTD_ERR_ARG;
  return guarded(&s->err, [&] {
    if (nt < 1) throw ArgError{FDTD_ERR_ARG, "nt must be positive."};
    if (s->adj_mode) leave_adjoint_mode(s);  // the time loop is captured without snapshots or history again
    prepare(s, nt);
    if (!engine_current(s)) new_engine(s);
    s->engine->run_async(nt, waits);
    fill_stats(s, s->engine.get());
  });
}

int fdtd_run_async(fdtd_sim* s, int nt) { return start_run(s, nt, false); }

int fdtd_run_checkpointed(fdtd_sim* s, int nt, int every) {
  if (!s) return FDTD_ERR_ARG;
  const int rc = guarded(&s->err, [&] {
    if (nt < 1 || every < 1) throw ArgError{FDTD_ERR_ARG, "nt and the checkpoint interval must be positive."};
    // a re-prepared simulation has new device buffers: the engine (descriptors,
    // tensor maps, graph) must be rebuilt with it
    prepare(s, nt);
    const bool rebuild = !engine_current(s) || s->adj_mode != 1 || s->adj_in_batch || s->ckpt_every != every ||
                         s->ckpt_nt != nt;
    const size_t N = s->cells_padded;
    const size_t stride = 6 * N + (s->splits.n ? 2 * s->split_buf_pairs : 0);
    const size_t nseg = size_t((nt + every - 1) / every);
    if (rebuild) {
      leave_adjoint_mode(s);
      s->adj_mode = 1;
      s->ckpt_every = every;
      s->ckpt_nt = nt;
      s->ckpt.alloc(nseg * stride);
      new_engine(s);
    }
    s->engine->run_async(nt, true);
    fill_stats(s, s->engine.get());
  });
  if (rc) return rc;
  return fdtd_synchronize(s);
}

int fdtd_run_recorded(fdtd_sim* s, int nt, const int* box) {
  if (!s) return FDTD_ERR_ARG;
  const int rc = guarded(&s->err, [&] {
    if (nt < 1 || !box) throw ArgError{FDTD_ERR_ARG, "nt must be positive and the box given."};
    prepare(s, nt);
    check_gradient_box(s, box);
    const bool rebuild = !engine_current(s) || s->adj_mode != 2 || s->adj_in_batch || s->ckpt_nt != nt ||
                         !std::equal(box, box + 6, s->adj_box);
    if (rebuild) {
      leave_adjoint_mode(s);
      s->hist.alloc(size_t(nt) * 9 * size_t(box_cells(box)));
      s->adj_mode = 2;
      s->ckpt_nt = nt;
      std::copy(box, box + 6, s->adj_box);
      new_engine(s);
    }
    s->engine->run_async(nt, true);
    fill_stats(s, s->engine.get());
  });
  if (rc) return rc;
  return fdtd_synchronize(s);
}

int fdtd_adjoint(fdtd_sim* s, const double* dJ_dX, int n_series, int n_freq, const int* box, double* grad) {
  if (!s) return FDTD_ERR_ARG;
  return guarded(&s->err, [&] {
    if (!dJ_dX || !box || !grad) throw ArgError{FDTD_ERR_ARG, "null argument"};
    if (!s->engine || s->adj_mode == 0 || s->ckpt_nt < 1)
      throw ArgError{FDTD_ERR_STATE, "fdtd_adjoint needs a preceding fdtd_run_checkpointed or fdtd_run_recorded."};
    if (n_series != s->n_series || n_freq != s->n_freq || n_series < 1 || n_freq < 1)
      throw ArgError{FDTD_ERR_ARG, "dJ/dX size does not match the DFT of the run."};
    if (s->engine->sims.size() != 1) throw ArgError{FDTD_ERR_STATE, "adjoint runs need a single simulation."};
    check_gradient_box(s, box);
    if (s->adj_mode == 2 && !std::equal(box, box + 6, s->adj_box))
      throw ArgError{FDTD_ERR_ARG, "gradient box differs from the box recorded by fdtd_run_recorded."};
    if (s->adj_in_batch) throw ArgError{FDTD_ERR_STATE, "the recorded run was a batch run: use fdtd_batch_adjoint."};
    s->engine->adjoint({Engine::AdjRequest{s, dJ_dX, box, grad}});
    s->stats.adjoint_launches = s->engine->adj_launches;
    s->stats.adjoint_ms = s->engine->adj_ms;
  });
}

int fdtd_synchronize(fdtd_sim* s) {
  if (!s) return FDTD_ERR_ARG;
  return guarded(&s->err, [&] {
    if (!s->engine) throw ArgError{FDTD_ERR_STATE, "No run in flight."};
    s->engine->sync();
    fill_stats(s, s->engine.get());
  });
}

int fdtd_run(fdtd_sim* s, int nt) {
  int rc = start_run(s, nt, true);
  if (rc) return rc;
  return fdtd_synchronize(s);
}

int fdtd_get_probe_values(fdtd_sim* s, float* out, int n_probes, int nt) {
  if (!s) return FDTD_ERR_ARG;
  return guarded(&s->err, [&] {
    if (!s->prepared || s->prepared_nt < 0) throw ArgError{FDTD_ERR_STATE, "No completed run."};
    if (n_probes != int(s->probes.size()) || nt != s->prepared_nt)
      throw ArgError{FDTD_ERR_ARG, "Probe output size does not match the last run."};
    if (n_probes == 0) return;
    d2h(s, out, s->rec.p, size_t(n_probes) * nt * sizeof(float));
  });
}

int fdtd_get_dft(fdtd_sim* s, double* out, int n_series, int n_freq) {
  if (!s) return FDTD_ERR_ARG;
  return guarded(&s->err, [&] {
    if (n_series != s->n_series || n_freq != s->n_freq) throw ArgError{FDTD_ERR_ARG, "DFT size mismatch."};
    if (!s->dft_X.n) throw ArgError{FDTD_ERR_STATE, "No DFT configured."};
    d2h(s, out, s->dft_X.p, s->dft_X.n * sizeof(double2));
  });
}

int fdtd_get_monitor(fdtd_sim* s, int m, void* out, int64_t n_bytes) {
  if (!s) return FDTD_ERR_ARG;
  return guarded(&s->err, [&] {
    if (m < 0 || m >= int(s->mon_out.size())) throw ArgError{FDTD_ERR_ARG, "Monitor index out of range."};
    if (size_t(n_bytes) != s->mon_out[m]->n) throw ArgError{FDTD_ERR_ARG, "Monitor output size mismatch."};
    d2h(s, out, s->mon_out[m]->p, size_t(n_bytes));
  });
}

int fdtd_get_stats(const fdtd_sim* s, fdtd_stats* out) {
  if (!s || !out) return FDTD_ERR_ARG;
  *out = s->stats;
  out->h2d_bytes = s->h2d_bytes;
  out->d2h_bytes = s->d2h_bytes;
  if (s->compiled) {
    for (int k = 0; k < 6; ++k) out->split_slab[k] = s->split_plan.t[k];
    out->slab_cells = s->split_plan.slab_cells;
    out->sparse_split_cells = s->split_plan.sparse_cells;
    out->split_bytes = int64_t(s->splits.n * sizeof(float));
  }
  return FDTD_OK;
}

const char* fdtd_last_error(const fdtd_sim* s) { return s ? s->err.c_str() : g_error.c_str(); }

void fdtd_destroy(fdtd_sim* s) {
  if (!s) return;
  if (s->engine) {
    cudaStreamSynchronize(s->engine->stream());
    s->engine.reset();
  }
  delete s;
}

int fdtd_batch_create(fdtd_sim* const* sims, int n_sims, fdtd_batch** out) {
  if (!out || !sims || n_sims < 1) {
    g_error = "fdtd_batch_create: invalid arguments";
    return FDTD_ERR_ARG;
  }
  *out = nullptr;
  auto* b = new (std::nothrow) fdtd_batch();
  if (!b) {
    g_error = "host allocation failed";
    return FDTD_ERR_LIMIT;
  }
  for (int i = 0; i < n_sims; ++i) {
    if (!sims[i]) {
      delete b;
      g_error = "fdtd_batch_create: null simulation";
      return FDTD_ERR_ARG;
    }
    b->sims.push_back(sims[i]);
  }
  b->asked = default_config();
  *out = b;
  return FDTD_OK;
}

int fdtd_batch_set_kernel(fdtd_batch* b, int variant, int tile_y, int stages, int zchunk) {
  if (!b) return FDTD_ERR_ARG;
  return guarded(&b->err, [&] {
    if (variant < 0 || variant > 1)
      throw ArgError{FDTD_ERR_ARG, "variant must be 0 (plain) or 1 (stream)"};
    if (!kernel_exists(variant, tile_y, stages))
      throw ArgError{FDTD_ERR_ARG, "No kernel instantiated for this variant / tile height / stage count."};
    b->asked.variant = variant;
    b->asked.ty = tile_y;
    b->asked.stages = stages;
    b->asked.zchunk = zchunk;
    b->asked.one_list = one_list_env();
    b->dirty = true;
  });
}

int fdtd_batch_set_stream(fdtd_batch* b, void* stream) {
  if (!b) return FDTD_ERR_ARG;
  b->ext_stream = static_cast<cudaStream_t>(stream);
  return FDTD_OK;
}

int fdtd_batch_run(fdtd_batch* b, int nt) {
  if (!b) return FDTD_ERR_ARG;
  return guarded(&b->err, [&] {
    if (nt < 1) throw ArgError{FDTD_ERR_ARG, "nt must be positive."};
    bool rebuild = b->run_nt != nt || b->parts.empty() || b->dirty;
    for (auto* s : b->sims) {
      if (!s->prepared || s->prepared_nt != nt) rebuild = true;
      if (s->adj_mode) {
        leave_adjoint_mode(s);
        rebuild = true;
      }
      try {
        prepare(s, nt);
      } catch (ArgError& a) {
        a.msg = "batch member: " + a.msg;
        throw;
      }
    }
    if (batch_moved(b)) rebuild = true;
    if (rebuild) {
      build_batch(b, nt);
      note_generations(b);
    }
    run_batch(b, nt);
    fdtd_stats& st = b->stats;
    st = fdtd_stats{};
    batch_run_stats(b, nt);
    // the first part's kernel
    const Engine& e = *b->parts[0];
    st.variant = e.cfg.variant;
    st.tile_y = e.cfg.variant != 0 ? e.cfg.ty : kTileY;
    st.stages = e.cfg.variant != 0 ? e.cfg.stages : 0;
    st.zchunk = e.zchunk_used;
    for (const auto& p : b->parts) {
      st.grid += p->grid;
      st.n_tiles += p->n_tiles;
      st.dft_launches += p->dft_launches;
    }
    for (auto* s : b->sims) {
      st.e_split_cells += s->grid.e_split_cells;
      st.h_split_cells += s->grid.h_split_cells;
      st.n_rows += int(s->grid.rows.size());
      st.compile_ms += s->grid.compile_ms;
    }
    st.id_bytes = 2;
  });
}

int fdtd_batch_run_recorded(fdtd_batch* b, int nt, const int* boxes) {
  if (!b) return FDTD_ERR_ARG;
  return guarded(&b->err, [&] {
    if (nt < 1 || !boxes) throw ArgError{FDTD_ERR_ARG, "nt must be positive and the boxes given."};
    bool rebuild = b->run_nt != nt || b->parts.empty() || b->dirty;
    for (size_t i = 0; i < b->sims.size(); ++i) {
      fdtd_sim* s = b->sims[i];
      const int* box = boxes + 6 * i;
      if (!s->prepared || s->prepared_nt != nt) rebuild = true;
      try {
        prepare(s, nt);
        check_gradient_box(s, box);
      } catch (ArgError& a) {
        a.msg = "batch member " + std::to_string(i) + ": " + a.msg;
        throw;
      }
      if (s->adj_mode != 2 || !s->adj_in_batch || s->ckpt_nt != nt || !std::equal(box, box + 6, s->adj_box)) {
        leave_adjoint_mode(s);
        s->hist.alloc(size_t(nt) * 9 * size_t(box_cells(box)));
        s->adj_mode = 2;
        s->adj_in_batch = true;
        s->ckpt_nt = nt;
        std::copy(box, box + 6, s->adj_box);
        rebuild = true;
      }
    }
    if (batch_moved(b)) rebuild = true;
    if (rebuild) {
      build_batch(b, nt);
      note_generations(b);
    }
    run_batch(b, nt);
    batch_run_stats(b, nt);
  });
}

int fdtd_batch_run_checkpointed(fdtd_batch* b, int nt, int every, const int* boxes) {
  if (!b) return FDTD_ERR_ARG;
  return guarded(&b->err, [&] {
    if (nt < 1 || every < 1 || !boxes)
      throw ArgError{FDTD_ERR_ARG, "nt and the checkpoint interval must be positive and the boxes given."};
    bool rebuild = b->run_nt != nt || b->parts.empty() || b->dirty;
    const size_t nseg = size_t((nt + every - 1) / every);
    for (size_t i = 0; i < b->sims.size(); ++i) {
      fdtd_sim* s = b->sims[i];
      const int* box = boxes + 6 * i;
      if (!s->prepared || s->prepared_nt != nt) rebuild = true;
      try {
        prepare(s, nt);
        check_gradient_box(s, box);
      } catch (ArgError& a) {
        a.msg = "batch member " + std::to_string(i) + ": " + a.msg;
        throw;
      }
      if (s->adj_mode != 1 || !s->adj_in_batch || s->ckpt_nt != nt || s->ckpt_every != every ||
          !std::equal(box, box + 6, s->adj_box)) {
        leave_adjoint_mode(s);
        const size_t stride = 6 * s->cells_padded + (s->splits.n ? 2 * s->split_buf_pairs : 0);
        s->ckpt.alloc(nseg * stride);
        s->adj_mode = 1;
        s->adj_in_batch = true;
        s->ckpt_every = every;
        s->ckpt_nt = nt;
        std::copy(box, box + 6, s->adj_box);
        rebuild = true;
      }
    }
    if (batch_moved(b)) rebuild = true;
    if (rebuild) {
      build_batch(b, nt);
      note_generations(b);
    }
    run_batch(b, nt);
    batch_run_stats(b, nt);
  });
}

int fdtd_batch_adjoint(fdtd_batch* b, const double* const* dJ_dX, double* const* grad) {
  if (!b) return FDTD_ERR_ARG;
  return guarded(&b->err, [&] {
    if (!dJ_dX || !grad) throw ArgError{FDTD_ERR_ARG, "null argument"};
    std::vector<Engine::AdjRequest> req;
    const int mode = b->sims.empty() ? 0 : b->sims[0]->adj_mode;
    for (size_t i = 0; i < b->sims.size(); ++i) {
      fdtd_sim* s = b->sims[i];
      if (s->adj_mode == 0 || s->adj_mode != mode || !s->adj_in_batch || b->run_nt != s->ckpt_nt)
        throw ArgError{FDTD_ERR_STATE,
                       "fdtd_batch_adjoint needs a preceding fdtd_batch_run_recorded or fdtd_batch_run_checkpointed."};
      if (s->n_series < 1 || s->n_freq < 1) throw ArgError{FDTD_ERR_STATE, "batch member without a DFT."};
      if (!dJ_dX[i] || !grad[i]) throw ArgError{FDTD_ERR_ARG, "null member array"};
      req.push_back(Engine::AdjRequest{s, dJ_dX[i], s->adj_box, grad[i]});
    }
    b->stats.adjoint_launches = 0;
    b->stats.adjoint_ms = 0;
    set_batch_streams(b);
    for (size_t k = 0; k < b->parts.size(); ++k) {
      std::vector<Engine::AdjRequest> part;
      for (size_t i : b->members[k]) part.push_back(req[i]);
      Engine& e = *b->parts[k];
      e.adjoint(part);
      b->stats.adjoint_launches = std::max<int64_t>(b->stats.adjoint_launches, e.adj_launches);
      b->stats.adjoint_ms += e.adj_ms;
    }
  });
}

int fdtd_batch_get_stats(const fdtd_batch* b, fdtd_stats* out) {
  if (!b || !out) return FDTD_ERR_ARG;
  *out = b->stats;
  return FDTD_OK;
}

const char* fdtd_batch_last_error(const fdtd_batch* b) { return b ? b->err.c_str() : g_error.c_str(); }

void fdtd_batch_destroy(fdtd_batch* b) {
  if (!b) return;
  for (auto& e : b->parts) cudaStreamSynchronize(e->stream());
  delete b;
}

const char* fdtd_global_error(void) { return g_error.c_str(); }

int fdtd_trim_memory(int64_t keep_bytes, int64_t* reserved, int64_t* used) {
  return guarded(&g_error, [&] {
    if (keep_bytes < 0) throw ArgError{FDTD_ERR_ARG, "fdtd_trim_memory: keep_bytes must be >= 0"};
    cudaMemPool_t pool = engine_pool();
    // blocks freed by destroyed simulations are returned once every stream is past their last use
    CK(device_wait());
    CK(cudaMemPoolTrimTo(pool, size_t(keep_bytes)));
    uint64_t r = 0, u = 0;
    CK(cudaMemPoolGetAttribute(pool, cudaMemPoolAttrReservedMemCurrent, &r));
    CK(cudaMemPoolGetAttribute(pool, cudaMemPoolAttrUsedMemCurrent, &u));
    if (reserved) *reserved = int64_t(r);
    if (used) *used = int64_t(u);
  });
}

int fdtd_nf2ff(const fdtd_nf2ff_face* faces, int n_faces, int n_freq, const float* beta, int n_theta,
               const float* theta, int n_phi, const float* phi, float* out) {
  return guarded(&g_error, [&] {
    if (!faces || n_faces < 0 || n_freq < 1 || n_theta < 1 || n_phi < 1 || !beta || !theta || !phi || !out)
      throw ArgError{FDTD_ERR_ARG, "fdtd_nf2ff: invalid arguments"};
    if (int64_t(n_theta) * n_phi > (int64_t(1) << 30) || n_freq > 65535)
      throw ArgError{FDTD_ERR_LIMIT, "fdtd_nf2ff: too many directions or frequencies"};
    int64_t n_cells = 0;
    for (int i = 0; i < n_faces; ++i) {
      const fdtd_nf2ff_face& fc = faces[i];
      if (fc.axis < 0 || fc.axis > 2 || fc.n0 < 0 || fc.n1 < 0)
        throw ArgError{FDTD_ERR_ARG, "fdtd_nf2ff: invalid face"};
      if (int64_t(fc.n0) * fc.n1 > 0 && (!fc.r0 || !fc.r1 || !fc.ds || !fc.J || !fc.M))
        throw ArgError{FDTD_ERR_ARG, "fdtd_nf2ff: null face array"};
      n_cells += int64_t(fc.n0) * fc.n1;
    }
    if (n_cells * n_freq > (int64_t(1) << 31)) throw ArgError{FDTD_ERR_LIMIT, "fdtd_nf2ff: surface too large"};
    // one block of device memory: the faces, then beta, theta, phi and the
    // faces' arrays as they come, then the parts' sums and the result
    const size_t n_dir = size_t(n_theta) * n_phi;
    size_t at = (size_t(std::max(1, n_faces)) * sizeof(Nf2ffFaceDev) + 3) / 4;  // floats
    const size_t o_beta = at, o_theta = o_beta + n_freq, o_phi = o_theta + n_theta;
    at = o_phi + n_phi;
    std::vector<Nf2ffFaceDev> fd(size_t(std::max(1, n_faces)), Nf2ffFaceDev{});
    int64_t first = 0;
    for (int i = 0; i < n_faces; ++i) {
      const fdtd_nf2ff_face& fc = faces[i];
      const size_t nc = size_t(fc.n0) * fc.n1;
      Nf2ffFaceDev& d = fd[size_t(i)];
      d.axis = fc.axis;
      d.cells = int(nc);
      d.first = int(first);
      d.pos = fc.pos;
      d.r0 = int64_t(at);
      d.r1 = int64_t(at + nc);
      d.ds = int64_t(at + 2 * nc);
      d.J = int64_t(at + 3 * nc);
      d.M = d.J + int64_t(6 * n_freq * nc);
      at = size_t(d.M) + 6 * n_freq * nc;
      first += int64_t(nc);
    }
    const std::unique_ptr<float[]> host(new float[at]);  // every word is written below
    std::memcpy(host.get(), fd.data(), fd.size() * sizeof(Nf2ffFaceDev));
    std::memcpy(&host[o_beta], beta, size_t(n_freq) * 4);
    std::memcpy(&host[o_theta], theta, size_t(n_theta) * 4);
    std::memcpy(&host[o_phi], phi, size_t(n_phi) * 4);
    for (int i = 0; i < n_faces; ++i) {
      const fdtd_nf2ff_face& fc = faces[i];
      const Nf2ffFaceDev& d = fd[size_t(i)];
      const size_t nc = size_t(d.cells);
      if (!nc) continue;
      std::memcpy(&host[size_t(d.r0)], fc.r0, nc * 4);
      std::memcpy(&host[size_t(d.r1)], fc.r1, nc * 4);
      std::memcpy(&host[size_t(d.ds)], fc.ds, nc * 4);
      std::memcpy(&host[size_t(d.J)], fc.J, 6 * n_freq * nc * 4);
      std::memcpy(&host[size_t(d.M)], fc.M, 6 * n_freq * nc * 4);
    }
    // parts: about eight blocks per SM in all (148 SMs), at least one chunk of
    // cells each, and at most 256 MB of sums
    const int64_t dir_blocks = int64_t((n_dir + kNf2ffThreads - 1) / kNf2ffThreads);
    int64_t parts = (int64_t(148) * 8 + dir_blocks * n_freq - 1) / (dir_blocks * n_freq);
    parts = std::min(parts, (n_cells + kNf2ffThreads - 1) / kNf2ffThreads);
    parts = std::min<int64_t>(parts, (int64_t(256) << 20) / int64_t(96 * n_dir * size_t(n_freq)));
    parts = std::max<int64_t>(1, std::min<int64_t>(parts, 65535));
    const int64_t per = std::max<int64_t>(1, (n_cells + parts - 1) / parts);
    const size_t n_out = 2 * size_t(n_freq) * n_dir;
    const size_t o_sums = (at + 3) / 4 * 4, o_out = o_sums + (parts > 1 ? size_t(parts) * n_freq * 12 * n_dir * 2 : 0);
    DevBuf<float> buf;
    buf.alloc(o_out + 2 * n_out);
    CK(cudaMemcpy(buf.p, host.get(), at * 4, cudaMemcpyHostToDevice));
    const float *d_beta = buf.p + o_beta, *d_theta = buf.p + o_theta, *d_phi = buf.p + o_phi;
    double* const d_sums = reinterpret_cast<double*>(buf.p + o_sums);
    float2* const d_out = reinterpret_cast<float2*>(buf.p + o_out);
    nf2ff_kernel<<<dim3(unsigned(dir_blocks), unsigned(n_freq), unsigned(parts)), kNf2ffThreads>>>(
        buf.p, reinterpret_cast<const Nf2ffFaceDev*>(buf.p), n_faces, int(n_cells), int(per), d_beta, d_theta, n_theta,
        d_phi, n_phi, d_sums, d_out);
    CK(cudaGetLastError());
    if (parts > 1) {
      nf2ff_field_kernel<<<dim3(unsigned((n_dir + kNf2ffThreads / kNf2ffGroups - 1) / (kNf2ffThreads / kNf2ffGroups)),
                                unsigned(n_freq)),
                           kNf2ffThreads>>>(
          d_sums, int(parts), d_beta, d_theta, n_theta, d_phi, n_phi, d_out);
      CK(cudaGetLastError());
    }
    CK(cudaMemcpy(out, d_out, n_out * sizeof(float2), cudaMemcpyDeviceToHost));
  });
}

}  // extern "C"

// ------------------------------------------------ stepping without allocation
//
// fdtd_step_noalloc advances a grid whose device buffers the caller owns, with
// the plain step kernel (fdtd_step_kernel). That kernel reads two small
// engine-built arrays besides the caller's data: the grid descriptor (SimDev)
// and the tile list. The other entry points cudaMalloc them per simulation;
// here they live in one file-scope device array of fixed size, so the call
// allocates nothing on the device. A set-up kernel writes both into the array
// on the caller's stream from its launch parameters (the descriptor by value,
// the tiles from the grid sizes), so the call leaves no host memory behind
// that the GPU still has to read after it returns.
namespace {

constexpr int kNoallocMaxTiles = 65536;          // tile-list capacity (16 B per tile)
constexpr size_t kNoallocDescBytes = 1024;       // room for the SimDev descriptor
constexpr size_t kNoallocScratchBytes = kNoallocDescBytes + size_t(kNoallocMaxTiles) * sizeof(int4);  // 1 MiB + 1 KiB
static_assert(sizeof(SimDev) <= kNoallocDescBytes, "descriptor does not fit its scratch slot");

// Shared by every call on a device, for the life of the process.
static __device__ __align__(256) unsigned char g_noalloc_scratch[kNoallocScratchBytes];

constexpr int kNoallocMaxDevices = 64;
std::mutex g_noalloc_mutex;
unsigned char* g_noalloc_ptr[kNoallocMaxDevices] = {};   // device address of the array, per device

// Writes the descriptor and the tile list of one call into the scratch array:
// tiles of 31 x 7 columns in z chunks of zlen planes, x fastest, then y, then
// the chunk (the plain kernel's tile order), as (0, x0 | y0 << 16, z0 | z1 << 16, 0).
__global__ void noalloc_setup_kernel(SimDev d, int zlen, int n_tiles, unsigned char* scratch) {
  if (blockIdx.x == 0 && threadIdx.x == 0) *reinterpret_cast<SimDev*>(scratch) = d;
  int4* tiles = reinterpret_cast<int4*>(scratch + kNoallocDescBytes);
  const int ntx = (d.nx + kTileX - 1) / kTileX, nty = (d.ny + kTileY - 1) / kTileY;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n_tiles; i += gridDim.x * blockDim.x) {
    const int xt = i % ntx, yt = (i / ntx) % nty, zc = i / (ntx * nty);
    const int x0 = xt * kTileX, y0 = yt * kTileY, z0 = zc * zlen, z1 = min(d.nz, z0 + zlen);
    tiles[i] = make_int4(0, x0 | (y0 << 16), z0 | (z1 << 16), 0);
  }
}

}  // namespace

extern "C" int fdtd_step_noalloc(const fdtd_device_grid* g, int n0, int n_steps, void* stream) {
  if (!g) {
    g_error = "fdtd_step_noalloc: null grid";
    return FDTD_ERR_ARG;
  }
  const int nx = g->nx, ny = g->ny, nz = g->nz, pitch = g->pitch;
  if (nx < 2 || ny < 2 || nz < 2 || nx > 65535 || ny > 65535 || nz > 65535 || pitch < nx) {
    g_error = "fdtd_step_noalloc: dimensions must be 2..65535 cells with pitch >= nx";
    return FDTD_ERR_ARG;
  }
  if (g->nt < 1 || n0 < 0 || n_steps < 0 || int64_t(n0) + n_steps > g->nt) {
    g_error = "fdtd_step_noalloc: steps n0 .. n0+n_steps-1 must lie in [0, nt)";
    return FDTD_ERR_ARG;
  }
  if (g->n_rows < 1 || g->n_rows > 65536 || g->n_probes < 0) {
    g_error = "fdtd_step_noalloc: n_rows must be 1..65536 (a 16-bit index) and n_probes >= 0";
    return FDTD_ERR_ARG;
  }
  const size_t N = size_t(nz) * ny * pitch;
  if (N >= (size_t(1) << 31) - size_t(2) * ny * pitch) {
    g_error = "fdtd_step_noalloc: grid too large for 32-bit cell offsets";
    return FDTD_ERR_LIMIT;
  }
  // the engine's tiling of the plain kernel: 31 x 7 columns, z cut so that
  // about 8 blocks per SM exist (at least 8 planes per chunk)
  const int64_t xy_tiles = int64_t((nx + kTileX - 1) / kTileX) * ((ny + kTileY - 1) / kTileY);
  if (xy_tiles > kNoallocMaxTiles) {
    g_error = "fdtd_step_noalloc: the grid needs " + std::to_string(xy_tiles) +
              " tiles per z chunk; the static tile list holds " + std::to_string(kNoallocMaxTiles);
    return FDTD_ERR_LIMIT;
  }
  if (!g->fields || !g->splits || !g->mat || !g->rows || !g->cell_probes || !g->src || !g->rec || !g->is_src) {
    g_error = "fdtd_step_noalloc: every buffer pointer must be a device address";
    return FDTD_ERR_ARG;
  }
  if (reinterpret_cast<uintptr_t>(g->splits) % 8 != 0 || reinterpret_cast<uintptr_t>(g->rows) % 16 != 0 ||
      reinterpret_cast<uintptr_t>(g->cell_probes) % 8 != 0) {
    g_error = "fdtd_step_noalloc: splits and cell_probes must be 8-byte aligned, rows 16-byte aligned";
    return FDTD_ERR_ARG;
  }
  if (n_steps == 0) return FDTD_OK;
  try {
    int dev = 0;
    CK(cudaGetDevice(&dev));
    if (dev < 0 || dev >= kNoallocMaxDevices) throw ArgError{FDTD_ERR_LIMIT, "device ordinal out of range"};
    unsigned char* scratch = nullptr;
    {
      std::lock_guard<std::mutex> lock(g_noalloc_mutex);
      if (!g_noalloc_ptr[dev]) {
        // once per device: host code cannot name the array's device address directly
        void* p = nullptr;
        CK(cudaGetSymbolAddress(&p, g_noalloc_scratch));
        g_noalloc_ptr[dev] = static_cast<unsigned char*>(p);
      }
      scratch = g_noalloc_ptr[dev];
    }
    int n_sm = 148;
    CK(cudaDeviceGetAttribute(&n_sm, cudaDevAttrMultiProcessorCount, dev));
    const int64_t want = int64_t(n_sm) * 8;
    int chunks = int(std::max<int64_t>(1, (want + xy_tiles - 1) / xy_tiles));
    chunks = std::min(chunks, std::max(1, nz / 8));
    chunks = int(std::min<int64_t>(chunks, kNoallocMaxTiles / xy_tiles));
    const int zlen = (nz + chunks - 1) / chunks;
    const int n_tiles = int(xy_tiles) * ((nz + zlen - 1) / zlen);
    SimDev d{};
    d.nx = nx; d.ny = ny; d.nz = nz; d.pitch = pitch; d.plane = ny * pitch; d.nt = g->nt;
    for (int b = 0; b < 2; ++b) {
      for (int c = 0; c < 3; ++c) {
        d.E[b][c] = g->fields + (size_t(b) * 6 + c) * N;
        d.H[b][c] = g->fields + (size_t(b) * 6 + 3 + c) * N;
      }
    }
    // the caller's splits cover the whole grid: one z-face store holding every
    // cell, component m of time buffer b at pairs (6 b + m) N
    d.sp.t[4] = nz;
    d.sp.w[kStZlo] = pitch;
    d.sp.h[kStZlo] = ny;
    d.sp.comp[kStZlo] = int64_t(N);
    for (int b = 0; b < 2; ++b) d.sp.base[b] = reinterpret_cast<float2*>(g->splits) + size_t(b) * 6 * N;
    d.mat = g->mat;
    d.rows = reinterpret_cast<const float4*>(g->rows);
    d.cell_probes = reinterpret_cast<const int2*>(g->cell_probes);
    d.src = g->src;
    d.rec = g->rec;
    d.is_src = g->is_src;
    d.cells = int64_t(N);
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    noalloc_setup_kernel<<<std::min(1024, (n_tiles + 255) / 256), 256, 0, st>>>(d, zlen, n_tiles, scratch);
    CK(cudaGetLastError());
    const SimDev* d_desc = reinterpret_cast<const SimDev*>(scratch);
    const int4* d_tiles = reinterpret_cast<const int4*>(scratch + kNoallocDescBytes);
    for (int n = n0; n < n0 + n_steps; ++n) {
      fdtd_step_kernel<kTileY><<<n_tiles, dim3(32, kBlockY), 0, st>>>(d_desc, d_tiles, n);
      CK(cudaGetLastError());
    }
    return FDTD_OK;
  } catch (const ArgError& a) {
    g_error = "fdtd_step_noalloc: " + a.msg;
    return a.code;
  } catch (const CudaError& c) {
    g_error = "fdtd_step_noalloc: " + c.where + ": " + cudaGetErrorString(c.code);
    return FDTD_ERR_CUDA;
  }
}

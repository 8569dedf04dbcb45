// fake_cuda.cpp -- the CUDA runtime calls and the kernel launchers that the
// library's host code uses, over host memory: every copy and fill is checked
// against the allocations, freed ones stay known, and a launch looks at the
// pointers it is given and computes nothing.  Linked with the pn_*.cpp sources
// by tests/test_device_memory_cpu.py, which drives it through the C ABI.
#include <cuda_runtime.h>

#include <cstdlib>
#include <cstring>
#include <map>
#include <mutex>
#include <string>

#include "pn_noalloc.hpp"
#include "pn_solver.hpp"
#include "rsg_energy.cuh"
#include "rsg_state.cuh"

namespace {

struct Block {
  size_t bytes;
  bool live;
};
std::map<uintptr_t, Block> g_blocks;
int64_t g_held = 0, g_room = -1;  // bytes held; most that may be (-1: any)
int g_faults = 0;
bool g_capturing = false;
std::string g_first;
int64_t g_launches = 0, g_null_reciprocals = 0, g_chunk_choices = 0;

void fault(const std::string &what) {
  if (g_faults++ == 0) g_first = what;
}

const Block *block_of(const void *p, uintptr_t *base = nullptr) {
  auto it = g_blocks.upper_bound((uintptr_t)p);
  if (it == g_blocks.begin()) return nullptr;
  --it;
  if ((uintptr_t)p >= it->first + it->second.bytes) return nullptr;
  if (base) *base = it->first;
  return &it->second;
}

bool device(const void *p, size_t n, const char *what) {
  uintptr_t base = 0;
  const Block *b = block_of(p, &base);
  const char *wrong = !b ? "not device memory" : !b->live ? "freed memory"
                    : (uintptr_t)p + n > base + b->bytes ? "past the end of its allocation" : nullptr;
  if (wrong) fault(std::string(what) + ": " + wrong);
  return !wrong;
}

void table(const void *p, const char *what) {  // a table a launch reads: none, or in a live allocation
  if (p) device(p, 1, what);
}

template <typename T>
void velocity(const pn::VelLaunch<T> &a) {
  g_launches++;
  for (const void *p : {(const void *)a.V0, (const void *)a.S0, (const void *)a.S5, (const void *)a.coef,
                        (const void *)a.gnode, (const void *)a.tile_src, (const void *)a.tile_sens})
    table(p, "velocity launch");
  if (a.sigval) device(a.sigval, (size_t)a.n_sig * sizeof(T), "velocity launch's signal row");
}

template <typename T>
void stress(const pn::StressLaunch<T> &a) {
  g_launches++;
  for (const void *p : {(const void *)a.V0, (const void *)a.S0, (const void *)a.S5, (const void *)a.mat,
                        (const void *)a.gcell, (const void *)a.tile_src})
    table(p, "stress launch");
  if (a.sigval) device(a.sigval, (size_t)a.n_sig * sizeof(T), "stress launch's signal row");
}

}  // namespace

extern "C" {

int fake_faults() { return g_faults; }
const char *fake_first_fault() { return g_first.c_str(); }
int64_t fake_launches() { return g_launches; }
int64_t fake_launches_without_reciprocals() { return g_null_reciprocals; }
int64_t fake_chunk_choices() { return g_chunk_choices; }
int64_t fake_held() { return g_held; }
void fake_set_room(int64_t bytes) { g_room = bytes; }
void fake_set_capturing(int on) { g_capturing = on != 0; }
void fake_reset() {
  g_capturing = false;
  g_faults = 0;
  g_first.clear();
  g_launches = g_null_reciprocals = g_chunk_choices = 0;
  g_room = -1;
}

cudaError_t cudaMalloc(void **p, size_t n) {
  if (g_room >= 0 && g_held + (int64_t)n > g_room) return cudaErrorMemoryAllocation;
  *p = std::aligned_alloc(256, (n + 255) / 256 * 256);
  std::memset(*p, 0xa5, n);
  g_blocks[(uintptr_t)*p] = Block{n, true};
  g_held += (int64_t)n;
  return cudaSuccess;
}
cudaError_t cudaFree(void *p) {
  if (!p) return cudaSuccess;
  auto it = g_blocks.find((uintptr_t)p);
  if (it == g_blocks.end() || !it->second.live) {
    fault("cudaFree: not a live allocation");
    return cudaErrorInvalidValue;
  }
  it->second.live = false;  // (the memory stays, so that a stale pointer is known)
  std::memset(p, 0x5a, it->second.bytes);
  g_held -= (int64_t)it->second.bytes;
  return cudaSuccess;
}
cudaError_t cudaHostAlloc(void **p, size_t n, unsigned) {  // (a device may read it)
  *p = std::aligned_alloc(256, (n + 255) / 256 * 256);
  g_blocks[(uintptr_t)*p] = Block{n, true};
  return cudaSuccess;
}
cudaError_t cudaHostGetDevicePointer(void **d, void *h, unsigned) { return *d = h, cudaSuccess; }
cudaError_t cudaFreeHost(void *p) {
  g_held += (int64_t)g_blocks[(uintptr_t)p].bytes;
  return cudaFree(p);
}
cudaError_t cudaMemcpy(void *d, const void *s, size_t n, cudaMemcpyKind k) {
  bool ok = true;
  if (k != cudaMemcpyDeviceToHost) ok = device(d, n, "copy to the device") && ok;
  if (k != cudaMemcpyHostToDevice) ok = device(s, n, "copy from the device") && ok;
  if (ok) std::memcpy(d, s, n);
  return cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void *d, const void *s, size_t n, cudaMemcpyKind k, cudaStream_t) {
  return cudaMemcpy(d, s, n, k);
}
cudaError_t cudaMemset(void *d, int v, size_t n) {
  if (device(d, n, "fill")) std::memset(d, v, n);
  return cudaSuccess;
}
cudaError_t cudaMemsetAsync(void *d, int v, size_t n, cudaStream_t) { return cudaMemset(d, v, n); }
cudaError_t cudaGetDevice(int *d) { return *d = 0, cudaSuccess; }
cudaError_t cudaDeviceGetAttribute(int *v, cudaDeviceAttr, int) { return *v = 152, cudaSuccess; }
cudaError_t cudaGetLastError() { return cudaSuccess; }
const char *cudaGetErrorString(cudaError_t) { return "fake"; }
cudaError_t cudaMemGetInfo(size_t *f, size_t *t) {
  *t = (size_t)1 << 38;
  *f = g_room >= 0 ? (size_t)(g_room - g_held) : *t;
  return cudaSuccess;
}
cudaError_t cudaDeviceSynchronize() { return cudaSuccess; }
cudaError_t cudaStreamIsCapturing(cudaStream_t, cudaStreamCaptureStatus *st) {
  return *st = g_capturing ? cudaStreamCaptureStatusActive : cudaStreamCaptureStatusNone, cudaSuccess;
}
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaPointerGetAttributes(cudaPointerAttributes *, const void *) { return cudaErrorInvalidValue; }
cudaError_t cudaEventCreate(cudaEvent_t *e) { return *e = nullptr, cudaSuccess; }
cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float *ms, cudaEvent_t, cudaEvent_t) { return *ms = 1.f, cudaSuccess; }
cudaError_t cudaStreamBeginCapture(cudaStream_t, cudaStreamCaptureMode) { return cudaErrorNotSupported; }
cudaError_t cudaStreamEndCapture(cudaStream_t, cudaGraph_t *) { return cudaErrorNotSupported; }
cudaError_t cudaGraphDestroy(cudaGraph_t) { return cudaSuccess; }
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t) { return cudaSuccess; }
cudaError_t cudaGraphInstantiate(cudaGraphExec_t *, cudaGraph_t, unsigned long long) { return cudaErrorNotSupported; }
cudaError_t cudaGraphLaunch(cudaGraphExec_t, cudaStream_t) { return cudaErrorNotSupported; }

}  // extern "C"

namespace pn {

cudaError_t launch_velocity_exact(const VelLaunch<double> &a, int, cudaStream_t) {
  velocity(a);
  table(a.recips, "velocity launch's reciprocals");
  if (!a.recips) g_null_reciprocals++;
  return cudaSuccess;
}
cudaError_t launch_stress_exact(const StressLaunch<double> &a, int, cudaStream_t) {
  stress(a);
  table(a.recips, "stress launch's reciprocals");
  if (!a.recips) g_null_reciprocals++;
  return cudaSuccess;
}
cudaError_t launch_velocity_f64(const VelLaunch<double> &a, int, bool, cudaStream_t) { return velocity(a), cudaSuccess; }
cudaError_t launch_velocity_f32(const VelLaunch<float> &a, int, bool, cudaStream_t) { return velocity(a), cudaSuccess; }
cudaError_t launch_velocity_df64(const VelLaunch<float2> &a, int, bool, cudaStream_t) { return velocity(a), cudaSuccess; }
cudaError_t launch_stress_f64(const StressLaunch<double> &a, int, bool, cudaStream_t) { return stress(a), cudaSuccess; }
cudaError_t launch_stress_f32(const StressLaunch<float> &a, int, bool, cudaStream_t) { return stress(a), cudaSuccess; }
cudaError_t launch_stress_df64(const StressLaunch<float2> &a, int, bool, cudaStream_t) { return stress(a), cudaSuccess; }
cudaError_t launch_exact_reciprocals(const double *d, int64_t n, double *rec, cudaStream_t) {
  device(d, (size_t)n * 8, "spacings");
  device(rec, (size_t)n * 16, "reciprocals");
  return cudaSuccess;
}
cudaError_t launch_table_batch(const BatchLaunch &, int, int, cudaStream_t) { return g_launches++, cudaSuccess; }
cudaError_t launch_table_batch_halves(const BatchLaunch &, int, int, int, cudaStream_t) { return cudaSuccess; }
cudaError_t launch_halo_exchange(int, const int4 *, int64_t, void *const *, cudaStream_t) { return cudaSuccess; }

template <typename A>
cudaError_t grid_step(const A &a) {
  g_launches++;
  for (const void *p : {(const void *)a.V_in[0], (const void *)a.V_out[2], (const void *)a.S_in[0],
                        (const void *)a.S_out[5], (const void *)a.coef, (const void *)a.mat, (const void *)a.f_rng,
                        (const void *)a.m_rng, (const void *)a.s_rng, (const void *)a.places.f,
                        (const void *)a.places.m, (const void *)a.places.s, (const void *)a.f_key})
    table(p, "grid launch");
  return cudaSuccess;
}
cudaError_t launch_grid_f32(const GridLaunch<float> &a, int, cudaStream_t) { return grid_step(a); }
cudaError_t launch_grid_f64(const GridLaunch<double> &a, int, cudaStream_t) { return grid_step(a); }
cudaError_t launch_grid_df64(const GridLaunch<float2> &a, int, cudaStream_t) { return grid_step(a); }
cudaError_t launch_grid_tma(const void *a, int precision, int, cudaStream_t) {
  return precision == PN_PREC_F32 ? grid_step(*(const GridLaunch<float> *)a)
       : precision == PN_PREC_DF64 ? grid_step(*(const GridLaunch<float2> *)a)
                                   : grid_step(*(const GridLaunch<double> *)a);
}
cudaError_t launch_grid_batch(const GridBatchLaunch &, int, int, cudaStream_t) { return g_launches++, cudaSuccess; }
cudaError_t launch_grid_tma_batch(const GridBatchLaunch &, int, int, cudaStream_t) { return g_launches++, cudaSuccess; }
cudaError_t launch_grid_split(const void *, int, cudaStream_t) { return cudaSuccess; }
cudaError_t launch_grid_split_batch(const GridSplitBatch &, int, int, cudaStream_t) { return cudaSuccess; }
size_t grid_tma_maps_bytes() { return 1408; }
bool grid_tma_rows_supported(int precision, int rows) { return rows == 8 || (rows == 16 && precision == PN_PREC_F32); }
bool grid_tma_encode(int, int, int, int, int, int, int, const void *const[3], const void *const[6], const void *,
                     const uint8_t *, void *) {
  return true;
}
int grid_chunk_layers(int, const std::map<int, long long> &tops, bool, int) {
  g_chunk_choices++;
  return tops.empty() ? 1 : tops.rbegin()->first;
}
cudaError_t launch_state_store(int, const double *, int64_t, const int64_t *, void *, cudaStream_t, int32_t *,
                               const StateRangeFlags *) {
  return cudaSuccess;
}
cudaError_t launch_state_load(int, const void *, int64_t, const int64_t *, double *, cudaStream_t) {
  return cudaSuccess;
}
cudaError_t launch_mark_tiles(uint8_t *flags, int64_t tiles, int p0, int p1, cudaStream_t) {
  device(flags + (p0 > p1 ? p0 : p1) * tiles, (size_t)tiles, "tile marks");
  return cudaSuccess;
}
int energy_blocks(int64_t) { return 1; }
cudaError_t launch_energy_nodes(int, const void *const[3], const double *, int64_t, double *, int, cudaStream_t) {
  return cudaSuccess;
}
cudaError_t launch_energy_cells(int, const void *const[6], const void *, bool, const double *, const double *, double,
                                int64_t, double *, int, cudaStream_t) {
  return cudaSuccess;
}
cudaError_t measure_pipe_rates(double *, int) { return cudaErrorNotSupported; }
static unsigned char *scratch() {
  static void *p = nullptr;
  if (!p) cudaMalloc(&p, kNoAllocScratchBytes);
  return (unsigned char *)p;
}
cudaError_t noalloc_scratch(void **p) { return *p = scratch(), cudaSuccess; }
std::mutex &noalloc_call_lock() {
  static std::mutex m;
  return m;
}

}  // namespace pn

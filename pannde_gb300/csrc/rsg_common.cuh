// rsg_common.cuh -- argument blocks shared by the host setup and the RSG
// leapfrog kernels (velocity update at nodes, stress update at cells).
//
// Device layout (structure of arrays, one array per component):
//   V[3]     node velocities Vx,Vy,Vz                 [n_nodes]      T
//   S[6]     cell stresses Sxx,Syy,Szz,Syz,Sxz,Sxy     [n_cells]      T
//   hex      cell -> 8 corner nodes                    [n_cells] int4x2
//   ncc      node -> 8 incident cell slots (-1 none)   [n_nodes] int4x2
//   coef     dt / rho_node (0 = node not owned)        [n_nodes]      T
//   mat      cell -> material row                      [n_cells]  int32
//   ctab     per material: 36 stiffness entries         [n_mat][36]    T
//            (fast forms: dt*C; exact form: C)
// The state is never read through the read-only path (__ldg, const
// __restrict__): a launch overlaps the kernel that writes it.
// Sources and sensors are sparse lists sorted by element, with one [begin,end)
// range per tile of kTile consecutive elements, so tiles without sources or
// sensors pay nothing.
#pragma once
#include <cstdint>
#include <cuda_runtime.h>

namespace pn {

constexpr int kTile = 256;  // elements per tile == threads per block

// signal values a launch carries in its own arguments (sig_here; at most so
// many sources): a caller's values of one step need no table on the device, and
// so neither a copy nor a wait for the steps in flight
constexpr int kSignalsHere = 8;

// What only a solver's own launches take (VelLaunch, StressLaunch, GridLaunch).
// The blocks that a batch's kernels read (VelArgs, StressArgs, GridArgs) are
// staged on the device, one per member, in the allocation-free call in a scratch
// of fixed size, and hold nothing that a batch does not use.
template <typename T, bool OWN>
struct OwnLaunch {};
template <typename T>
struct OwnLaunch<T, true> {
  int32_t sig_here;    // 1: this step's values are sig_vals
  T sig_vals[kSignalsHere];
  const T *recips;     // exact form: the reciprocals of the spacings in two words (k_reciprocals), or null
};

// Connectivity as patterns (fast forms): an element's eight neighbours are its
// base plus the offsets of its pattern.  Meshes numbered along lattice lines,
// graded, holed or cracked ones too, have a few dozen patterns (interior, faces,
// edges, rims), so an element takes 5 bytes instead of 32; a mesh with more than
// 256 keeps the tables.  A missing cell's offset is INT32_MIN (base + it < 0).
// In one allocation: the patterns' offsets (two int4 each), the elements' bases
// (int32), their pattern numbers (uint8); n_patterns 0: the table, two int4 an
// element.

template <typename T, bool OWN = false>
struct VelArgs : OwnLaunch<T, OWN> {
  int32_t n_nodes;
  int32_t n_patterns;
  const int4 *__restrict__ ncc;  // the nodes' cells: table or patterns
  T *V0;
  T *V1;
  T *V2;
  const T *S0;
  const T *S1;
  const T *S2;
  const T *S3;
  const T *S4;
  const T *S5;
  const T *__restrict__ coef;
  // spacing factors: uniform (gx,gy,gz = 0.25/h) or per node [3][n_nodes]
  // (fast forms: 0.25/d; exact form: d)
  T gx, gy, gz;
  const T *__restrict__ gnode;
  // force sources
  const int2 *__restrict__ tile_src;  // [n_tiles] or null
  const int32_t *__restrict__ src_elem;
  const int32_t *__restrict__ src_code;  // dir | (signal << 2)
  const T *__restrict__ src_w;
  const T *__restrict__ sigval;  // signal values: row min(step, sig_rows-1) at stride sig_stride
  int32_t n_sig;
  int32_t sig_stride;            // 0 when sigval already points at this step's row
  int32_t sig_rows;
  // sensors
  const int2 *__restrict__ tile_sens;  // [n_tiles] or null
  const int32_t *__restrict__ sens_node;
  const int32_t *__restrict__ sens_idx;
  double *__restrict__ traces;  // [rec_cap][n_sens][3]
  int32_t n_sens;
  int64_t rec_base;
  int64_t rec_cap;
};

template <typename T, bool OWN = false>
struct StressArgs : OwnLaunch<T, OWN> {
  int32_t n_cells;
  int32_t n_patterns;
  const T *V0;
  const T *V1;
  const T *V2;
  T *S0;
  T *S1;
  T *S2;
  T *S3;
  T *S4;
  T *S5;
  // the cells' nodes: table or patterns (ahead of V0 it leaves the pointers on 16
  // bytes, and FP32 k_stress spills: graded plate 200 x 200 x 40 1.19 instead of 1.15 ms)
  const int4 *__restrict__ hex;
  const int32_t *__restrict__ mat;
  const T *__restrict__ ctab;
  T gx, gy, gz;
  const T *__restrict__ gcell;  // per cell [3][n_cells] or null
  T dt;                          // exact form only (fast forms fold dt into ctab)
  // moment sources
  const int2 *__restrict__ tile_src;
  const int32_t *__restrict__ src_elem;
  const int32_t *__restrict__ src_code;  // comp | (signal << 3)
  const T *__restrict__ src_w;
  const T *__restrict__ sigval;
  int32_t n_sig;
  int32_t sig_stride;
  int32_t sig_rows;
  int32_t has_moments;
  int32_t sym;  // symmetry class of the whole stiffness table (symmetry_class): 0 general, 1 monoclinic
                // about z, 2 orthotropic
};

template <typename T> using VelLaunch = VelArgs<T, true>;
template <typename T> using StressLaunch = StressArgs<T, true>;

// whether an argument block is a solver's own launch's
template <typename A, typename = void>
struct is_launch : std::false_type {};
template <typename A>
struct is_launch<A, std::void_t<decltype(A::sig_here)>> : std::true_type {};

// Entries (k, j) of the stiffness product by symmetry class (symmetry_class): 0
// general, 1 monoclinic about z, 2 orthotropic in the axes; the others are zero, so
// 36 / 20 / 12 terms remain
#ifdef __CUDACC__
__host__ __device__
#endif
constexpr bool c_used(int sym, int k, int j) {
  return sym == 0 ? true
       : sym == 2 ? ((k < 3 && j < 3) || k == j)
                  : ((k < 3 && j < 3) || k == j || (k == 5 && j < 3) || (j == 5 && k < 3) ||
                     (k == 3 && j == 4) || (k == 4 && j == 3));
}

#ifdef __CUDACC__
// Programmatic dependent launch between the kernels of consecutive half
// steps: launch_overlapped marks a launch that may start while the kernel
// before it ends; such a kernel reads only tables that no step writes until
// wait_previous, which waits for that kernel's end and its memory.
// let_next_start: the next one may start once every block has come here.
__device__ __forceinline__ void wait_previous() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void let_next_start() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

// The half-step kernels of the table form let the next one start when a thread
// has formed its results, a launch of many blocks already when it begins: blocks of
// the next kernel that start beside the first wave of a small one gather on the SMs
// that it leaves free, and run there one after the other.  Us per step, at the
// beginning / when formed (no overlap, older kernels): plate 64 x 64 x 8 (149 blocks)
// FP64 35.3 / 17.8 (25.8), exact 64.6 / 41.0 (53.5); 96 x 96 x 16 (625 blocks) in
// random numbering FP32 63.7 / 42.1 (49.5), FP64 41.8 / 40.3; 131 x 97 x 21 (1112) FP64
// 64.2 / 64.6; 200 x 200 x 40 (6471) FP32 54.7 / 55.4, FP64 345 / 346.
constexpr unsigned kManyBlocks = 1024;
__device__ __forceinline__ void let_next_start_if_many() {
  if (gridDim.x >= kManyBlocks) let_next_start();
}

template <typename F, typename... A>
inline cudaError_t launch_overlapped(F f, dim3 grid, unsigned threads, size_t smem, cudaStream_t st, A... args) {
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = grid;
  cfg.blockDim = dim3(threads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute at{};
  at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at.val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = &at;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, f, args...);
}

// or bits into a byte of an array of flags, or clear it (the array's words are
// only ever written by atomics while a kernel runs)
__device__ __forceinline__ void flag_or(uint8_t *flags, int64_t i, uint32_t bits) {
  atomicOr(reinterpret_cast<uint32_t *>(flags + (i & ~(int64_t)3)), bits << (8 * (int)(i & 3)));
}
__device__ __forceinline__ void flag_clear(uint8_t *flags, int64_t i) {
  atomicAnd(reinterpret_cast<uint32_t *>(flags + (i & ~(int64_t)3)), ~(0xffu << (8 * (int)(i & 3))));
}

// the eight neighbours of element i of n: by its pattern, or from the table
__device__ __forceinline__ void neighbours(const int4 *__restrict__ table, int n_patterns, int n, int i, int s[8]) {
  int4 lo, hi;
  int b = 0;
  if (n_patterns > 0) {
    const int32_t *__restrict__ base = reinterpret_cast<const int32_t *>(table + 2 * n_patterns);
    const int p = (reinterpret_cast<const uint8_t *>(base + n))[i];
    b = base[i];
    lo = __ldg(table + 2 * p);
    hi = __ldg(table + 2 * p + 1);
  } else {
    lo = table[2 * i];
    hi = table[2 * i + 1];
  }
  s[0] = b + lo.x; s[1] = b + lo.y; s[2] = b + lo.z; s[3] = b + lo.w;
  s[4] = b + hi.x; s[5] = b + hi.y; s[6] = b + hi.z; s[7] = b + hi.w;
}

// signal values of a step: the launch's own, or row min(step, sig_rows-1) of
// the table (null: no sources)
template <typename A>
__device__ __forceinline__ auto signal_row(const A &a, int step) -> decltype(a.sigval) {
  if constexpr (is_launch<A>::value) {
    if (a.sig_here) return a.sig_vals;
  }
  return a.sigval ? a.sigval + (int64_t)min(step, a.sig_rows - 1) * a.sig_stride : nullptr;
}
#endif

// Launchers (defined in rsg_fast.cu / rsg_exact.cu).  step = index of this
// step inside the current solve() call (selects the signal row).
cudaError_t launch_velocity_f64(const VelLaunch<double> &a, int step, bool uniform, cudaStream_t st);
cudaError_t launch_stress_f64(const StressLaunch<double> &a, int step, bool uniform, cudaStream_t st);
cudaError_t launch_velocity_f32(const VelLaunch<float> &a, int step, bool uniform, cudaStream_t st);
cudaError_t launch_stress_f32(const StressLaunch<float> &a, int step, bool uniform, cudaStream_t st);
cudaError_t launch_velocity_df64(const VelLaunch<float2> &a, int step, bool uniform, cudaStream_t st);
cudaError_t launch_stress_df64(const StressLaunch<float2> &a, int step, bool uniform, cudaStream_t st);
// a batch of table-form members: device arrays of their argument blocks and
// the prefix sums of their tile counts (members own consecutive tiles)
struct BatchLaunch {
  int n_members;
  const void *vel_args;   // VelArgs<S>[n_members]
  const void *str_args;   // StressArgs<S>[n_members]
  const int *vel_start;   // [n_members + 1]
  const int *str_start;   // [n_members + 1]
  int vel_tiles, str_tiles;
  int blocks_vel, blocks_str;  // grid sizes (blocks walk the tiles)
};
// precision: PN_PREC_F64 (1), PN_PREC_F32 (2), PN_PREC_DF64 (3)
cudaError_t launch_table_batch(const BatchLaunch &b, int precision, int step, cudaStream_t st);
// one or both half steps of a batch step: halves bit 0 velocity, bit 1 stress
cudaError_t launch_table_batch_halves(const BatchLaunch &b, int precision, int step, int halves, cudaStream_t st);

// rec[i], rec[i + n]: the two words of the reciprocal of spacing d[i] as the
// exact kernels take it (rsg_exact.cu)
cudaError_t launch_exact_reciprocals(const double *d, int64_t n, double *rec, cudaStream_t st);
cudaError_t launch_velocity_exact(const VelLaunch<double> &a, int step, cudaStream_t st);
cudaError_t launch_stress_exact(const StressLaunch<double> &a, int step, cudaStream_t st);

}  // namespace pn

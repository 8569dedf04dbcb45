// rsg_exact.cu -- RSG leapfrog kernels in the reference's exact FP64
// operation order.  This translation unit is compiled with -fmad=false, so
// every product and sum is rounded separately, as the reference's C++ is;
// divisions are IEEE round-to-nearest (nvcc's default -prec-div=true).  The
// results are bit-identical to HostSolver on the same inputs.
//
//   DD*_nc (RightHex.hpp:151-192, ncDifferencer 225-231):
//     value = 0; value += (f[fwd_k] or 0) - (f[bwd_k] or 0), k = 0..3;
//     return (value*0.25)/d_node
//   DD*_cc (RightHex.hpp:100-141, ccDifferencer 241-247): the same over corners
//     with the cell spacing.
//   velocity (HostRSGTDUT.hpp:343-360):
//     V_d += coef * (((DDx + DDy) + DDz) + evalXds)
//   stress (HostRSGTDUT.hpp:284-291, HostUTModel.hpp:276-284):
//     S_k += dt * (C_k0*d00 + C_k1*d11 + C_k2*d22 + C_k3*(d12+d21)
//                  + C_k4*(d02+d20) + C_k5*(d01+d10) [+ evalMoments])
//   evalXds / evalMoments: 0.125*signal summed over the in-window
//     (element, source) pairs in the reference's loop order (kept in the
//     source list order; the weight of every entry is 0.125).
//
// Both kernels are bound by the FP64 pipe (85% busy; GB300 issues about two
// FP64 operations per SM per clock), so what counts is the FP64 operations per
// element.  Three groups of them are left out where the bits allow it, and the
// integer and FP32 pipes, idle otherwise, check that they do:
//   divisions   (value*0.25)/d = value/(4d): two operations with the stored
//               reciprocal of 4d instead of about nine (div_spacing)
//   zeros       0 + x and x + 0 only turn -0 into +0: done on the bits
//   products    with entries that are zero by the material's symmetry class:
//               each adds +0 or -0, which changes a sum only when it is -0
//               (then, and for strains that are not finite, the cell takes the
//               full sum)
// 168 -> 118 and 210 -> 135 FP64-pipe instructions per node and cell
// (orthotropic rows).  Measured on an aluminium plate of 128 x 128 x 16 cells: velocity
// step 105.5 -> 76.5 us, stress step 123.2 -> 78.6 us (FP64 pipe 80% busy; with
// Markstein's three or four operations per quotient throughout 82.4 and 83.4).
#include "rsg_common.cuh"

namespace pn {
namespace {

// forward / backward corner (or slot) sets per axis, RightHex.hpp:103-104,
// 118-119, 133-134 (the same sets index the node slots, 154-186)
__host__ __device__ constexpr int fwd_of(int a, int k) {
  return a == 0 ? (k == 0 ? 1 : k == 1 ? 2 : k == 2 ? 5 : 6)
       : a == 1 ? (k == 0 ? 2 : k == 1 ? 3 : k == 2 ? 6 : 7)
                : 4 + k;
}
__host__ __device__ constexpr int bwd_of(int a, int k) {
  return a == 0 ? (k == 0 ? 0 : k == 1 ? 3 : k == 2 ? 4 : 7)
       : a == 1 ? (k == 0 ? 0 : k == 1 ? 1 : k == 2 ? 4 : 5)
                : k;
}

// Sum of the four differences along axis A.  The reference starts from 0, and
// 0 + x is x except for x = -0: the sum of four differences is -0 only when
// all four are, and div_spacing returns +0 for it.
template <int A>
__device__ __forceinline__ double sum_nc(const double *f, const int s[8]) {
  double v[4];
#pragma unroll
  for (int k = 0; k < 4; k++) {
    const int a = s[fwd_of(A, k)], b = s[bwd_of(A, k)];
    const double fa = (a == -1) ? 0. : f[a];
    const double fb = (b == -1) ? 0. : f[b];
    v[k] = fa - fb;
  }
  return ((v[0] + v[1]) + v[2]) + v[3];
}

template <int A>
__device__ __forceinline__ double sum_cc(const double *f, const int s[8]) {
  double v[4];
#pragma unroll
  for (int k = 0; k < 4; k++) v[k] = f[s[fwd_of(A, k)]] - f[s[bwd_of(A, k)]];
  return ((v[0] + v[1]) + v[2]) + v[3];
}

__device__ __forceinline__ double no_negative_zero(double x) {  // x + 0.0
  return __double_as_longlong(x) == (long long)0x8000000000000000ull ? 0. : x;
}

// sign and zero tests on the bits: a comparison of doubles is an FP64-pipe operation
__device__ __forceinline__ bool is_zero(double x) { return (__double_as_longlong(x) & 0x7fffffffffffffffll) == 0; }

// One axis' divisor c = 4d with its reciprocal in two words, r = RN(1/c) and
// rl = RN(1/c - r) (k_reciprocals; element i's at rec[i] and
// rec[i + n3], n3 = 3 elements' count): r is stored negated when the divisor
// needs the longer quotient, 0 when it is outside the range below.  Without
// stored reciprocals (rec null: no memory for them) they are formed here, at
// one division per axis, for the longer quotient.
struct Divisor {
  double d, c, r, rl;
  bool lng;
  __device__ __forceinline__ Divisor(double dd, const double *__restrict__ rec, int64_t i, int64_t n3) : d(dd) {
    c = __hiloint2double(__double2hiint(d) + (2 << 20), __double2loint(d));
    if (rec) {
      r = rec[i];
      rl = rec[i + n3];
    } else {
      r = rl = 0.;
      if (d >= 0x1p-102 && d <= 0x1p98) {
        r = -1. / c;
        rl = fma(c, r, 1.) * -r;
      }
    }
    lng = __double2hiint(r) < 0;
    r = fabs(r);
  }
};

// RN(v / c) for a divisor known in advance.  q = v r + RN(v rl), rounded once by
// the FMA, is RN(v / c) unless v / c lies within 2^-105 of itself of a rounding
// boundary (Brisebarre, Muller and Raina, "Accelerating correctly rounded
// floating-point division when the divisor is known in advance", 2004);
// k_reciprocals has tried every v for which it does, and marks the divisors one
// of them fails for (LONG).  For those the exact remainder v - q c (one FMA) times r is
// added (Markstein, "Computation of elementary functions on the IBM RISC
// System/6000 processor", 1990): q is within half an ulp and a term of 2^-52
// ulp, so the value before the last rounding is off by less than 2^-53 times
// that, below the least distance ulp/2 * ulp(c)/c of v / c from a boundary.  Both
// need quotients and remainders to be normal numbers: |v| in [2^-850, 2^850] and c in
// [2^-100, 2^100] (or r = 0); ok says so.  (v rl may be subnormal, rl lies down to
// about 2^-205: its rounding is then off by 2^-1075 at most, 2^-125 of the quotient.)  A zero v gives +0 whatever its sign,
// as (0 + v) * 0.25 / d does.
template <bool LONG>
__device__ __forceinline__ double div_spacing(double v, const Divisor &d, bool &ok) {
  const uint32_t e = ((uint32_t)__double2hiint(v) >> 20) & 0x7ffu;
  const bool zero = is_zero(v);
  ok = ok && (zero || (e - 173u) <= 1700u);
  double q = fma(v, d.r, v * d.rl);
  if (LONG) q = fma(fma(-q, d.c, v), d.r, q);
  return zero ? 0. : q;
}

// Whether fma(v, r, v * rl) is RN(v / c) for every v.  With V, C the 53-bit
// integer significands of v and c, and M the odd 54-bit one of a midpoint of two
// doubles, v / c lies within 2^-105 of itself of that midpoint only for
// |V 2^s - M C| < 4, s = 53 for V >= C and 54 below; the difference k is not 0 (a
// quotient is never a midpoint), and for each k M = -k / C modulo 2^s leaves a few
// values of M to try.  (Of 200,000 random divisors 1% failed, all at |k| = 1, and
// none at 5 <= |k| <= 200.)
__device__ bool short_quotient(double c, double r, double rl) {
  int ec = 0;
  const double f = frexp(c, &ec);  // c = f 2^ec, f in [1/2, 1)
  const uint64_t C = (uint64_t)ldexp(f, 53);
  const double cd = (double)C, rd = ldexp(r, ec - 53), rld = ldexp(rl, ec - 53);
  const int z = __ffsll((long long)C) - 1;
  if (z > 2) return true;  // k would have to be a multiple of 2^z
  const uint64_t Co = C >> z;
  uint64_t inv = Co;  // Co^-1 modulo 2^64, by Newton's iteration
  for (int i = 0; i < 6; i++) inv *= 2 - Co * inv;
  for (int s = 53; s <= 54; s++)
    for (int k = -4; k <= 4; k++) {
      if (k == 0 || (k & ((1 << z) - 1)) != 0) continue;
      const uint64_t step = 1ull << (s - z);  // M Co = -(k / 2^z) modulo 2^(s - z)
      uint64_t M = (0 - (uint64_t)(int64_t)(k / (1 << z))) * inv & (step - 1);
      for (; M < (1ull << 54); M += step) {
        if (M < (1ull << 53) || !(M & 1)) continue;
        const __int128 n = (__int128)M * (__int128)C + k;
        if ((n & (((__int128)1 << s) - 1)) != 0) continue;
        const uint64_t V = (uint64_t)(n >> s);
        if (V < (1ull << 52) || V >= (1ull << 53)) continue;
        const double v = (double)V;
        if (fma(v, rd, v * rld) != v / cd) return false;
      }
    }
  return true;
}

__global__ void __launch_bounds__(256) k_reciprocals(const double *__restrict__ d, int64_t n, double *__restrict__ rec) {
  const int64_t i = (int64_t)blockIdx.x * 256 + threadIdx.x;
  if (i >= n) return;
  const double c = 4. * d[i];
  double r = 0., rl = 0.;
  if (c >= 0x1p-100 && c <= 0x1p100) {
    r = 1. / c;
    rl = fma(-c, r, 1.) / c;  // (the remainder is exact)
    if (!short_quotient(c, r, rl)) r = -r;
  }
  rec[i] = r;
  rec[i + n] = rl;
}

// q[i][a] = RN(v[i][a] / (4 d_a)): by the short quotient when every divisor of
// the warp allows it, by the reference's own operations where a value is out of
// its range
__device__ __forceinline__ void divide9(const double v[3][3], Divisor &dx, Divisor &dy, Divisor &dz, double q[3][3]) {
  bool ok = !is_zero(dx.r) && !is_zero(dy.r) && !is_zero(dz.r);
  if (__any_sync(__activemask(), dx.lng || dy.lng || dz.lng)) {
#pragma unroll
    for (int i = 0; i < 3; i++) {
      q[i][0] = div_spacing<true>(v[i][0], dx, ok);
      q[i][1] = div_spacing<true>(v[i][1], dy, ok);
      q[i][2] = div_spacing<true>(v[i][2], dz, ok);
    }
  } else {
#pragma unroll
    for (int i = 0; i < 3; i++) {
      q[i][0] = div_spacing<false>(v[i][0], dx, ok);
      q[i][1] = div_spacing<false>(v[i][1], dy, ok);
      q[i][2] = div_spacing<false>(v[i][2], dz, ok);
    }
  }
  if (!ok) {
#pragma unroll 1
    for (int i = 0; i < 9; i++) {  // (a loop: one copy of the division)
      const int a = i % 3;
      const double d = a == 0 ? dx.d : a == 1 ? dy.d : dz.d;
      double w = v[0][0];
#pragma unroll
      for (int j = 1; j < 9; j++) w = i == j ? v[j / 3][j % 3] : w;
      w = ((0. + w) * 0.25) / d;
#pragma unroll
      for (int j = 0; j < 9; j++) q[j / 3][j % 3] = i == j ? w : q[j / 3][j % 3];
    }
  }
}

// sensor traces: V after this step at the sensors of this tile
__device__ __forceinline__ void record(const VelLaunch<double> &a, int n, int step, double v0,
                                       double v1, double v2) {
  if (!a.tile_sens) return;
  const int2 r = a.tile_sens[blockIdx.x];
  const int64_t rec = a.rec_base + step;
  if (rec >= a.rec_cap) return;
  for (int i = r.x; i < r.y; i++) {
    if (a.sens_node[i] != n) continue;
    double *t = a.traces + (rec * a.n_sens + a.sens_idx[i]) * 3;
    t[0] = v0;
    t[1] = v1;
    t[2] = v2;
  }
}

__global__ void __launch_bounds__(kTile) k_velocity_exact(const __grid_constant__ VelLaunch<double> a, int step) {
  let_next_start_if_many();
  const int n = blockIdx.x * kTile + threadIdx.x;
  if (n >= a.n_nodes) return;
  const double cf = a.coef[n];
  const int4 lo = a.ncc[2 * n], hi = a.ncc[2 * n + 1];
  wait_previous();  // (tables only so far)
  if (cf == 0.) {  // node owned by another partition: not updated, still recorded
    record(a, n, step, a.V0[n], a.V1[n], a.V2[n]);
    return;
  }
  const int s[8] = {lo.x, lo.y, lo.z, lo.w, hi.x, hi.y, hi.z, hi.w};
  const int64_t ny = (int64_t)a.n_nodes + n, nz = 2 * (int64_t)a.n_nodes + n, n3 = 3 * (int64_t)a.n_nodes;
  Divisor dx(a.gnode[n], a.recips, n, n3), dy(a.gnode[ny], a.recips, ny, n3), dz(a.gnode[nz], a.recips, nz, n3);
  double xd[3] = {0., 0., 0.};
  bool sourced = false;
  if (a.tile_src) {
    const int2 r = a.tile_src[blockIdx.x];
    const double *sig = signal_row(a, 0);  // (the table's pointer is already at the step's row)
    for (int i = r.x; i < r.y; i++) {
      if (a.src_elem[i] != n) continue;
      const int code = a.src_code[i];
      const double v = a.src_w[i] * sig[code >> 2];
      const int d = code & 3;
      if (d == 0) xd[0] = xd[0] + v;
      else if (d == 1) xd[1] = xd[1] + v;
      else xd[2] = xd[2] + v;
      sourced = true;
    }
  }
  // x: S0 S5 S4  y: S5 S1 S3  z: S4 S3 S2, each along x, y, z
  const double v[3][3] = {{sum_nc<0>(a.S0, s), sum_nc<1>(a.S5, s), sum_nc<2>(a.S4, s)},
                          {sum_nc<0>(a.S5, s), sum_nc<1>(a.S1, s), sum_nc<2>(a.S3, s)},
                          {sum_nc<0>(a.S4, s), sum_nc<1>(a.S3, s), sum_nc<2>(a.S2, s)}};
  double q[3][3];
  divide9(v, dx, dy, dz, q);
  double vn[3] = {a.V0[n], a.V1[n], a.V2[n]}, v0[3];
#pragma unroll
  for (int d = 0; d < 3; d++) {
    v0[d] = no_negative_zero((q[d][0] + q[d][1]) + q[d][2]);
  }
  if (sourced) {
#pragma unroll 1
    for (int d = 0; d < 3; d++) {  // (rolled: a branch, as in k_stress_exact)
      const double w = (d == 0 ? v0[0] : d == 1 ? v0[1] : v0[2]) + (d == 0 ? xd[0] : d == 1 ? xd[1] : xd[2]);
#pragma unroll
      for (int q = 0; q < 3; q++) v0[q] = q == d ? w : v0[q];
    }
  }
  let_next_start();
#pragma unroll
  for (int d = 0; d < 3; d++) vn[d] = vn[d] + cf * v0[d];
  a.V0[n] = vn[0];
  a.V1[n] = vn[1];
  a.V2[n] = vn[2];
  record(a, n, step, vn[0], vn[1], vn[2]);
}

template <int SYM, bool MOMENTS>
__global__ void __launch_bounds__(kTile) k_stress_exact(const __grid_constant__ StressLaunch<double> a, int step) {
  let_next_start_if_many();
  const int c = blockIdx.x * kTile + threadIdx.x;
  if (c >= a.n_cells) return;
  const int4 lo = a.hex[2 * c], hi = a.hex[2 * c + 1];
  const int s[8] = {lo.x, lo.y, lo.z, lo.w, hi.x, hi.y, hi.z, hi.w};
  const int64_t cy = (int64_t)a.n_cells + c, cz = 2 * (int64_t)a.n_cells + c, n3 = 3 * (int64_t)a.n_cells;
  Divisor dx(a.gcell[c], a.recips, c, n3), dy(a.gcell[cy], a.recips, cy, n3), dz(a.gcell[cz], a.recips, cz, n3);
  const double *V[3] = {a.V0, a.V1, a.V2};
  wait_previous();  // (tables only so far)
  // v[j][i], d[j][i]: velocity component j along axis i
  double v[3][3], d[3][3];
#pragma unroll
  for (int j = 0; j < 3; j++) {
    v[j][0] = sum_cc<0>(V[j], s);
    v[j][1] = sum_cc<1>(V[j], s);
    v[j][2] = sum_cc<2>(V[j], s);
  }
  divide9(v, dx, dy, dz, d);
  const double e[6] = {d[0][0], d[1][1], d[2][2], d[2][1] + d[1][2], d[2][0] + d[0][2], d[1][0] + d[0][1]};
  double mom[6] = {0., 0., 0., 0., 0., 0.};
  if (MOMENTS && a.tile_src) {
    const int2 r = a.tile_src[blockIdx.x];
    const double *sig = signal_row(a, 0);
    for (int i = r.x; i < r.y; i++) {
      if (a.src_elem[i] != c) continue;
      const int code = a.src_code[i];
      const double w = a.src_w[i] * sig[code >> 3];
      const int k = code & 7;
#pragma unroll
      for (int q = 0; q < 6; q++) if (q == k) mom[q] = mom[q] + w;
    }
  }
  const double *C = a.ctab + 36 * a.mat[c];
  double *S[6] = {a.S0, a.S1, a.S2, a.S3, a.S4, a.S5};
  // the products with zero entries add +0 or -0 when every strain is finite:
  // the sum without them is the same unless it is -0
  double acc[6];
  bool full = false;
#pragma unroll
  for (int j = 0; j < 6; j++) full = full || (__double2hiint(e[j]) & 0x7ff00000) == 0x7ff00000;
#pragma unroll
  for (int ks = 0; ks < 6; ks++) {
    bool first = true;
#pragma unroll
    for (int j = 0; j < 6; j++) {
      if (!c_used(SYM, ks, j)) continue;
      const double p = C[6 * ks + j] * e[j];
      acc[ks] = first ? p : acc[ks] + p;
      first = false;
    }
    full = full || __double_as_longlong(acc[ks]) == (long long)0x8000000000000000ull;
  }
  if (SYM != 0 && full) {
    // a rolled loop, so that this stays a branch: predicated-off FP64
    // instructions still take their turn on the pipe (stress step 105 us with
    // them, 86 us without)
#pragma unroll 1
    for (int ks = 0; ks < 6; ks++) {
      const double *Ck = C + 6 * ks;
      const double w = Ck[0] * e[0] + Ck[1] * e[1] + Ck[2] * e[2] + Ck[3] * e[3] + Ck[4] * e[4] + Ck[5] * e[5];
#pragma unroll
      for (int q = 0; q < 6; q++) acc[q] = q == ks ? w : acc[q];
    }
  }
  if (MOMENTS) {
#pragma unroll
    for (int ks = 0; ks < 6; ks++) acc[ks] = acc[ks] + mom[ks];
  }
  let_next_start();
#pragma unroll
  for (int ks = 0; ks < 6; ks++) S[ks][c] = S[ks][c] + a.dt * acc[ks];
}

}  // namespace

cudaError_t launch_exact_reciprocals(const double *d, int64_t n, double *rec, cudaStream_t st) {
  if (n <= 0) return cudaSuccess;
  k_reciprocals<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(d, n, rec);
  return cudaGetLastError();
}

cudaError_t launch_velocity_exact(const VelLaunch<double> &a, int step, cudaStream_t st) {
  if (a.n_nodes <= 0) return cudaSuccess;
  const unsigned grid = (unsigned)((a.n_nodes + kTile - 1) / kTile);
  return launch_overlapped(k_velocity_exact, dim3(grid), kTile, 0, st, a, step);
}

cudaError_t launch_stress_exact(const StressLaunch<double> &a, int step, cudaStream_t st) {
  if (a.n_cells <= 0) return cudaSuccess;
  const unsigned grid = (unsigned)((a.n_cells + kTile - 1) / kTile);
  auto run = [&](auto kernel) { return launch_overlapped(kernel, dim3(grid), kTile, 0, st, a, step); };
  if (a.has_moments)
    return a.sym == 2 ? run(k_stress_exact<2, true>) : a.sym == 1 ? run(k_stress_exact<1, true>) : run(k_stress_exact<0, true>);
  return a.sym == 2 ? run(k_stress_exact<2, false>) : a.sym == 1 ? run(k_stress_exact<1, false>) : run(k_stress_exact<0, false>);
}

}  // namespace pn

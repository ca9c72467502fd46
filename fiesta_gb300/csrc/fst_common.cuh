// fst_common.cuh — shared device-side definitions of libfst.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>
#include <string.h>

#include "../../include/fst.h"
#include "fst_fp64.cuh"

#define FST_MAXV (4 + FST_MAX_SPECIES + 5)

// Grid geometry and strides of one field in HBM.  Fields are stored like the
// reference's CUDA build, LayoutLeft with i fastest:
//   a[i + sy*j + sz*k + sv*v],  sy = ngi, sz = ngi*ngj, sv = ngi*ngj*ngk.
struct Geo {
  int ndim, ng, nci, ncj, nck, ngi, ngj, ngk;
  int ns, nv, nvt;
  long long sy, sz, sv;
};

// Division by a run-time constant d, on the integer pipes (fst_fp64.cuh).
// When d is a power of two, a/d equals a*(1/d) exactly for every a (both are
// the correctly rounded a*2^k) and the exponent is shifted; otherwise the
// integer division with d's reciprocal prepared on the host.  Results are
// bit-identical to a/d either way.
struct DivC {
  double d, inv;  // inv = 1/d if d is a power of two, else 0
  int k;          // inv = 2^k, or NONE: tested in place of inv, whose compare would take the
                  // FP64 unit as long as a sum (k_cell3d at 256^3: 10.1 ms against 8.2)
  fst64::Recip r;
  static constexpr int NONE = 1 << 20;
  __device__ __forceinline__ double operator()(double a) const {
    return k != NONE ? fst64::scale2(a, k, inv) : fst64::div_by(a, r);
  }
  // the same with the division as a call (fst64::div_call)
  __device__ __forceinline__ double call(double a) const {
    return k != NONE ? fst64::scale2(a, k, inv) : fst64::div_call(a, r.hi, r.lo, r.R);
  }
};

// a/x, b/y, c/z with one call
__device__ __forceinline__ fst64::Quot3 div3(const DivC& x, double a, const DivC& y, double b, const DivC& z,
                                             double c) {
  if (x.k == DivC::NONE && y.k == DivC::NONE && z.k == DivC::NONE) return fst64::div3_call(a, b, c, x.r, y.r, z.r);
  return {x.call(a), y.call(b), z.call(c)};
}

// Physics constants of one run, passed by value to the kernels.
struct Phys {
  int ns, nv, nvt, visc, ceq, buoyancy;
  int scheme;  // 2D flux: 1 WENO5, 2 centered4, 3 QUICK (src/cart2d.cpp:165-172)
  // species constants of calculateRhoPT (src/secondary.hpp:127-135):
  //   cp_s = gammas*Rs/(gammas-1), cv_s = Rs/(gammas-1), Rs = cd(7+3s)
  double cp_s[FST_MAX_SPECIES], cv_s[FST_MAX_SPECIES], mu_s[FST_MAX_SPECIES];
  double rm_s[FST_MAX_SPECIES];  // cp_s - cv_s = Rs (mixed path)
  // the same with the stride-2 species table read by maxWaveSpeed2D
  // (src/ceq.hpp:61-66): gammas = cd(6+2s), Rs = cd(7+2s)
  double cp2_s[FST_MAX_SPECIES], cv2_s[FST_MAX_SPECIES];
  double dx, dy, dz;
  DivC dd[3];             // a/dx, a/dy, a/dz
  DivC d4[3];             // a/(4*dx) ... (viscous and C-equation tangential terms)
  DivC d12[3];            // a/(12.0*dx) ... (4th-order derivatives)
  DivC d12pz;             // a/(12.0*cd(2)): the reference's dz = cd(2) in presgrad3D
  double r12x, r12y, r12pz;  // their reciprocals (mixed path)
  double dt, hdt;         // dt and 0.5f*dt
  double kap, eps, alpha, g, rho_ref;
  double dxmag2;          // dx^2+dy^2(+dz^2): alpha numerator
  double dxmag;           // sqrt(dx^2+dy^2(+dz^2)): updateCeq cell size
  double mu2d;            // constant 2D viscosity 2.928e-5 (src/viscosity.hpp:62-63)
  double kheat2d;         // 2D heat conductivity 0.026 (src/viscosity.hpp:117)
  // FP32 copies for the mixed path: cv_s, R_s = cp_s - cv_s, mu_s, and the
  // stride-2 table constants
  float cv_f[FST_MAX_SPECIES], rm_f[FST_MAX_SPECIES], mu_f[FST_MAX_SPECIES];
  // low parts of cv_s and R_s as FP32 pairs (cv_f + cv_lf, rm_f + rm_lf)
  float cv_lf[FST_MAX_SPECIES], rm_lf[FST_MAX_SPECIES];
  float cv2_f[FST_MAX_SPECIES], cp2_f[FST_MAX_SPECIES];
  // FP32 copies of the grid constants (mixed path)
  float rd_f[3];    // 1/dx, 1/dy, 1/dz
  float r12_f[3];   // 1/(12 dx), 1/(12 dy), 1/(12 dz)
  float dxmag_f, dxmag2_f, eps_f, kap_f, alpha_f, mu2d_f, kheat_f;
};

// The bit pattern of x through an opaque register move.  Integer tests on
// the bits then stay integer tests: an optimiser may otherwise rewrite a
// masked compare such as (bits & 0x7FF..F) >= c as an ordered FP compare
// |x| >= c', which is false for NaN where the integer test is true.
__device__ __forceinline__ unsigned long long fst_bits(double x) {
  unsigned long long b;
  asm("mov.b64 %0, %1;" : "=l"(b) : "d"(x));
  return b;
}

// --- order-preserving encoding of doubles for atomicMax -------------------
__device__ __forceinline__ unsigned long long fst_key(double x) {
  unsigned long long b = (unsigned long long)__double_as_longlong(x);
  return (b >> 63) ? ~b : (b | 0x8000000000000000ull);
}
__host__ __device__ __forceinline__ double fst_unkey(unsigned long long k) {
  unsigned long long b = (k >> 63) ? (k & 0x7FFFFFFFFFFFFFFFull) : ~k;
#ifdef __CUDA_ARCH__
  return __longlong_as_double((long long)b);
#else
  double d;
  memcpy(&d, &b, 8);
  return d;
#endif
}
// Kokkos::Max starts from -DBL_MAX and `if (s > lmax)` never takes a NaN.
#define FST_KEY_LOWEST 0x0010000000000000ull /* fst_key(-DBL_MAX) */

// Running maximum on the order-preserving key, NaN skipped: integer work, where
// FP64 compares would each take the FP64 unit's time.
__device__ __forceinline__ void fst_key_max(unsigned long long& k, double x) {
  const unsigned long long b = fst64::bits_of(x);
  if ((b & 0x7FFFFFFFFFFFFFFFull) > 0x7FF0000000000000ull) return;
  const unsigned long long q = (b >> 63) ? ~b : (b | 0x8000000000000000ull);
  k = q > k ? q : k;
}
// The maxima of two keys over a block of 32 W threads (every thread calls it) into
// word[0] and word[1]: one atomic per block and word.
template <int W>
__device__ __forceinline__ void fst_key_max_block(unsigned long long* word, unsigned long long a,
                                                  unsigned long long b) {
  __shared__ unsigned long long sa[W], sb[W];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const unsigned long long x = __shfl_xor_sync(0xffffffffu, a, o);
    const unsigned long long y = __shfl_xor_sync(0xffffffffu, b, o);
    a = x > a ? x : a;
    b = y > b ? y : b;
  }
  if ((threadIdx.x & 31) == 0) {
    sa[threadIdx.x >> 5] = a;
    sb[threadIdx.x >> 5] = b;
  }
  __syncthreads();
  if (threadIdx.x < 2) {
    const unsigned long long* s = threadIdx.x ? sb : sa;
    unsigned long long m = s[0];
    for (int w = 1; w < W; ++w) m = s[w] > m ? s[w] : m;
    atomicMax(&word[threadIdx.x], m);
  }
}

// Warp-wide max of per-thread maxima that already skipped NaN.
__device__ __forceinline__ double fst_warp_max(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    double w = __shfl_xor_sync(0xffffffffu, v, o);
    v = (w > v) ? w : v;  // NaN never wins, as in the reference reducer
  }
  return v;
}

// finiteness from the exponent bits (integer ops, not the FP64 pipe)
__device__ __forceinline__ bool fst_finite(double x) {
  return (fst_bits(x) & 0x7FF0000000000000ull) != 0x7FF0000000000000ull;
}

// Linear index helpers
__device__ __forceinline__ long long fst_idx(const Geo& g, int i, int j, int k) {
  return (long long)i + g.sy * j + g.sz * k;
}

// The ghost cells of a grid in a flat order: the ghost planes in k (3D), the
// ghost rows in j of the interior planes, the ghost columns in i of the
// interior rows (each part contiguous along i).  fst_shell_count gives their
// number; fst_shell_cell maps t in [0, count) to (i, j, k).
__host__ __device__ __forceinline__ long long fst_shell_count(const Geo& g) {
  const int ngz = g.ndim == 3 ? g.ng : 0;
  const long long nk = g.ngk - 2 * ngz, nj = g.ngj - 2 * g.ng;
  return 2LL * ngz * g.ngi * g.ngj + nk * 2 * g.ng * g.ngi + nk * nj * 2 * g.ng;
}
template <class T>
__device__ __forceinline__ void fst_shell_cell_of(const Geo& g, T t, int& i, int& j, int& k) {
  const int ng = g.ng, ngz = g.ndim == 3 ? g.ng : 0;
  const int nj = g.ngj - 2 * ng, nk = g.ngk - 2 * ngz;
  const T ni = (T)g.ngi, pl = ni * (T)g.ngj, w = (T)(2 * ng);
  const T nA = 2 * (T)ngz * pl, nB = (T)nk * w * ni;
  if (t < nA) {
    const T p = t / pl, r = t - p * pl;
    k = (int)p < ngz ? (int)p : g.ngk - 2 * ngz + (int)p;
    j = (int)(r / ni);
    i = (int)(r - (T)j * ni);
  } else if (t < nA + nB) {
    const T u = t - nA, row = u / ni;
    i = (int)(u - row * ni);
    const int kk = (int)(row / w), jj = (int)(row - (T)kk * w);
    k = ngz + kk;
    j = jj < ng ? jj : g.ngj - 2 * ng + jj;
  } else {
    const T u = t - nA - nB, row = u / w;
    const int ii = (int)(u - row * w);
    const int kk = (int)(row / (T)nj), jj = (int)(row - (T)kk * (T)nj);
    k = ngz + kk;
    j = ng + jj;
    i = ii < ng ? ii : g.ngi - 2 * ng + ii;
  }
}
// (64-bit divisions are most of the instructions of a ghost cell: only where needed)
__device__ __forceinline__ void fst_shell_cell(const Geo& g, long long t, int& i, int& j, int& k) {
  if (g.sv <= 0x7FFFFFFFLL) fst_shell_cell_of(g, (unsigned)t, i, j, k);
  else fst_shell_cell_of(g, t, i, j, k);
}

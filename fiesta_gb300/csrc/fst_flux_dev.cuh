// fst_flux_dev.cuh — the WENO5 advection fluxes of the plain FP64 path
// (calculateFluxesG, src/flux.hpp:223-310; computeFluxWeno2D, :23-106), shared by
// the 3D and 2D modules.  Built with --fmad=false: every value is the
// reference's, bit for bit; the fused operations written out below round what
// the reference's two operations round.
//
// The FP64 unit is the bound (fst_fp64.cuh), so a face's value is arranged to
// use it as little as exactness allows:
//  - the first difference term of a smoothness indicator, T = (13/12 a1) a1 with
//    a1 = (f- - 2f) + f+, belongs to a cell: the three faces that read it share
//    it (a thread marches along its line), once per upwind direction in use;
//  - so do f/3 and 5f/6; -f/6 is -1/2 of f/3, exactly;
//  - x - 2y, x - 4y, T + S/4 and t/2 terms are fused (2y, 4y, S/4 and t/2 are exact);
//  - divisions and products run on the integer pipes, sums as DFMA.
// The forms hold for stencil values that are 0 or in [2^-200, 2^150): then every
// difference is 0 or at least 2^-253, every product normal or 0, and weights lie
// in [2^-621, 2^40].  Any other stencil (NaN and infinity among them) takes
// weno_any, the reference's expression as written.
//
// Measured at 256^3, 9 variables, dx a power of two (per stage): 93.5 ms as one
// thread per face index with the operators, 49.5 with shared cell terms, fused
// forms and integer divisions, 24.3 with the products on the integer pipes, 23.7 with
// the sums as DFMA, 23.1 with no compare or predicated-off operation left on the FP64
// unit (either takes as long as a sum): unit 82 % busy, integer unit 55 %, 44
// instructions per FP64 one.
// A value outside the range sends the six faces of its line that read it to weno_any,
// and a warp with such a lane runs both forms.  At 128^3, 9 variables, 3.12 ms: 3.7 with
// one species falling from 1 to 1e-120 across the box, 3.9 with one at 1e-100 all over,
// 6.4 with four, 12.0 with every variable in blocks of 16 cells of either kind (both forms
// on nearly every face); the operators take 13.2 on any of them.
#pragma once
#include "fst_internal.h"

namespace fstflux {

using fst64::div_rn;

// weno's constants: float literals in the 3D module, double ones in 2D
#define FST_WENO_CONST(name, num, den)                                              \
  struct name {                                                                      \
    static constexpr double value = F32 ? (double)((float)(num) / (float)(den))      \
                                        : (double)(num) / (double)(den);             \
  };
template <bool F32>
struct K {
  FST_WENO_CONST(c1312, 13.0, 12.0)
  FST_WENO_CONST(c13, 1.0, 3.0)
  FST_WENO_CONST(c76, 7.0, 6.0)
  FST_WENO_CONST(c116, 11.0, 6.0)
  FST_WENO_CONST(c16, 1.0, 6.0)
  FST_WENO_CONST(c56, 5.0, 6.0)
  FST_WENO_CONST(three, 3.0, 1.0)
  FST_WENO_CONST(w1, 0.1, 1.0)
  FST_WENO_CONST(w2, 0.6, 1.0)
  FST_WENO_CONST(w3, 0.3, 1.0)
  static constexpr double eps = 0.000001;
};
#undef FST_WENO_CONST

// calculateFluxesG::weno (src/flux.hpp:241-266) / computeFluxWeno2D::weno
// (:37-63) as written; out of line, for stencils weno_core excludes
template <bool F32>
__device__ __noinline__ double weno_any(double f1, double f2, double f3, double f4, double f5) {
  using C = K<F32>;
  const double k = C::c1312::value, o = C::c13::value, s = -C::c16::value, e = C::c56::value;
  double b1, b2, b3, w1, w2, w3, p1, p2, p3, a1, a2;
  a1 = f1 - 2.0 * f2 + f3;
  a2 = f1 - 4.0 * f2 + 3.0 * f3;
  b1 = k * a1 * a1 + (0.25) * a2 * a2;
  a1 = f2 - 2.0 * f3 + f4;
  a2 = f2 - f4;
  b2 = k * a1 * a1 + (0.25) * a2 * a2;
  a1 = f3 - 2.0 * f4 + f5;
  a2 = 3.0 * f3 - 4.0 * f4 + f5;
  b3 = k * a1 * a1 + (0.25) * a2 * a2;
  a1 = C::eps + b1;
  w1 = C::w1::value / (a1 * a1);
  a1 = C::eps + b2;
  w2 = C::w2::value / (a1 * a1);
  a1 = C::eps + b3;
  w3 = C::w3::value / (a1 * a1);
  p1 = o * f1 + -C::c76::value * f2 + C::c116::value * f3;
  p2 = s * f2 + e * f3 + o * f4;
  p3 = o * f3 + e * f4 + s * f5;
  return (w1 * p1 + w2 * p2 + w3 * p3) / (w1 + w2 + w3);
}

// the constants of the fused operations below, in thread registers
struct FK : fst64::Fused {
  double two, four, half, quarter, eps;
  __device__ __forceinline__ explicit FK(int n)
      : Fused(n), two(fst64::lane_const(2.0, n)), four(fst64::lane_const(4.0, n)),
        half(fst64::lane_const(0.5, n)), quarter(fst64::lane_const(0.25, n)),
        eps(fst64::lane_const(0.000001, n)) {}
};
template <class C>
__device__ __forceinline__ double mc(double x) {
  return fst64::mul_const<C>(x);
}
// (13/12 a1) a1 of the cell with value f, lower neighbour (upwind order) a and
// upper neighbour b
template <bool F32>
__device__ __forceinline__ double cell_term(const FK& k, double a, double f, double b) {
  const double a1 = k.add(__fma_rn(-k.two, f, a), b);
  return fst64::mul_int<true>(mc<typename K<F32>::c1312>(a1), a1);
}
__device__ __forceinline__ double sq(double x) { return fst64::sq_int<true>(x); }

// c / (x x) for x = eps + beta and a weight constant c
template <class C>
__device__ __forceinline__ double weight(double x) {
  return fst64::div_const<C>(fst64::sq_int<false>(x));
}
// a weight times a candidate value
__device__ __forceinline__ double wp(double w, double p) { return fst64::mul_int<true>(p, w); }

// weno of f1..f5 with t = f/3 and e = 5f/6 (rounded) of the cells that need them
// and the cell terms T of f2, f3 and f4
template <bool F32>
__device__ __forceinline__ double weno_core(const FK& k, double f1, double f2, double f3, double f4, double f5,
                                            double t1, double t2, double t3, double t4, double t5,
                                            double e3, double e4, double T2, double T3, double T4) {
  using C = K<F32>;
  const double f33 = mc<typename C::three>(f3);
  double a2 = k.add(__fma_rn(-k.four, f2, f1), f33);
  const double b1 = __fma_rn(k.quarter, sq(a2), T2);
  a2 = k.sub(f2, f4);
  const double b2 = __fma_rn(k.quarter, sq(a2), T3);
  a2 = k.add(__fma_rn(-k.four, f4, f33), f5);
  const double b3 = __fma_rn(k.quarter, sq(a2), T4);
  const double w1 = weight<typename C::w1>(k.add(b1, k.eps));
  const double w2 = weight<typename C::w2>(k.add(b2, k.eps));
  const double w3 = weight<typename C::w3>(k.add(b3, k.eps));
  // -f/6 is -t/2 exactly
  const double p1 = k.add(k.sub(t1, mc<typename C::c76>(f2)), mc<typename C::c116>(f3));
  const double p2 = k.add(__fma_rn(-k.half, t2, e3), t4);
  const double p3 = __fma_rn(-k.half, t5, k.add(t3, e4));
  return div_rn(k.add(k.add(wp(w1, p1), wp(w2, p2)), wp(w3, p3)), k.add(k.add(w1, w2), w3));
}

// x + p of the energy's stencil values, out of line: one warp in nv needs it, and
// inlined it would be predicated and take the FP64 unit's time for the others too
__device__ __noinline__ static double add_apart(double x, double p) { return x + p; }

// One direction's share of the flux launch: lines of `n` interior cells along
// the direction, `lines` of them (na x nb interior transverse cells), cut into
// `nseg` segments of at most LSEG faces.
constexpr int LSEG = 32;
struct Dir {
  long long st, sa, sb;  // strides along the line and the two transverse axes
  long long base;        // first interior cell
  int n, na;             // cells along the line, transverse extent a
  int lines, nseg, seg;  // na * nb, segments per line, faces per segment
  int first;             // first block of this direction
  DivC dd;               // division by the spacing
};
struct Plan {
  Dir d[3];
  int ndim, blocks;
};

// A block takes 32 lines of one direction and one segment of them; its threads
// first form the face velocities, then each warp marches one variable after
// another along the 32 lines.  Lanes run along the first transverse axis, so loads
// and stores of the y and z directions are coalesced; along x a warp walks 32 rows
// side by side and reuses each memory line it fetched for 16 steps.  gridDim.y
// blocks share the variables.  More warps in
// flight than the 16 to 20 of this split gain nothing (18 to 28: 2 %).
// Face values go to F[(dir*nv + v)*sv + cell] for the faces of interior cells.
constexpr int WMAX = 5;  // warps per block, at most
template <bool F32>
__global__ void __launch_bounds__(32 * WMAX, 4)
    k_weno_flux(const __grid_constant__ Plan plan, long long sv, int nv, int ve,
                const double* __restrict__ U, const double* __restrict__ pr,
                const double* __restrict__ vel, double* __restrict__ F) {
  __shared__ double s_uf[LSEG][32];
  __shared__ unsigned s_neg[LSEG];           // lanes with uf < 0
  __shared__ unsigned char s_any[LSEG + 2];  // 1: a face with uf >= 0 (or NaN), 2: one with uf < 0
  const int dir = plan.ndim == 3 && (int)blockIdx.x >= plan.d[2].first ? 2
                  : (int)blockIdx.x >= plan.d[1].first                 ? 1
                                                                       : 0;
  const Dir& D = plan.d[dir];
  const int b = blockIdx.x - D.first;
  const int seg = b % D.nseg, chunk = b / D.nseg;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarp = blockDim.x >> 5;
  const int l0 = chunk * 32 + lane;
  const bool live = l0 < D.lines;
  const int l = live ? l0 : D.lines - 1;  // a spare lane repeats the last line and stores nothing
  const int lb = l / D.na, la = l - lb * D.na;
  // faces [c0, c1) of the line, face c between cells c and c + 1; cell 0 is the first interior
  const int c0 = -1 + seg * D.seg, c1 = min(c0 + D.seg, D.n);
  const long long line = D.base + D.sa * la + D.sb * lb;
  const long long st = D.st;
  const double* vd = vel + sv * dir + line;
  const FK k(nv);
  for (int m = warp; m < c1 - c0; m += nwarp) {
    const long long o = st * (c0 + m);
    const double uf =
        div_rn(k.sub(k.add(k.sub(7.0 * vd[o + st], vd[o + 2 * st]), 7.0 * vd[o]), vd[o - st]), 12.0);
    s_uf[m][lane] = uf;
    const unsigned ng = __ballot_sync(0xffffffffu, uf < 0.0);
    if (lane == 0) s_neg[m] = ng;
    if (lane == 0) s_any[m] = (unsigned char)((ng != 0xffffffffu ? 1 : 0) | (ng ? 2 : 0));
  }
  if (threadIdx.x < 2) s_any[c1 - c0 + threadIdx.x] = 0;
  __syncthreads();

  const double* pq = pr + line;
  for (int v = warp + nwarp * blockIdx.y; v < nv; v += nwarp * gridDim.y) {
    const double* q = U + sv * v + line;
    double* Fd = F + sv * ((long long)dir * nv + v) + line;
    // stencil value of a cell: var + (v==energy)*p.  For the others that is
    // var + 0*p: var itself where p is finite (the sign of a zero aside), NaN
    // where it is not.
    auto value = [&](long long o) {
      const double x = q[o], p = pq[o];
      if (v == ve) return add_apart(x, p);
      return fst_finite(p) ? x : fst64::of_bits(0x7FF8000000000000ull);
    };
    // outside weno_core's range: not 0 and not in [2^-200, 2^150)
    auto wide = [](double x) {
      const uint64_t b = fst64::bits_of(x);
      const unsigned h = (unsigned)(b >> 32) & 0x7FFFFFFFu;
      return h - (823u << 20) >= (350u << 20) && (b << 1) != 0;
    };
    using C = K<F32>;
    long long o = st * c0;
    double f0 = value(o - 2 * st), f1 = value(o - st), f2 = value(o), f3 = value(o + st),
           f4 = value(o + 2 * st), f5;
    double nxt = value(o + 3 * st);
    // faces left whose six cells hold one out of range
    int bad = wide(f4) ? 6 : wide(f3) ? 5 : wide(f2) ? 4 : wide(f1) ? 3 : wide(f0) ? 2 : 0;
    double t0 = mc<typename C::c13>(f0), t1 = mc<typename C::c13>(f1), t2 = mc<typename C::c13>(f2),
           t3 = mc<typename C::c13>(f3), t4 = mc<typename C::c13>(f4), t5;
    double e2, e3 = mc<typename C::c56>(f2);
    double tp0 = 0, tp1 = 0, tp2 = 0, tn0 = 0, tn1 = 0, tn2 = 0;
    {
      const int any = s_any[0] | s_any[1];
      if (any & 1) {
        tp1 = cell_term<F32>(k, f0, f1, f2);
        tp2 = cell_term<F32>(k, f1, f2, f3);
      }
      if (any & 2) {
        tn1 = cell_term<F32>(k, f3, f2, f1);
        tn2 = cell_term<F32>(k, f4, f3, f2);
      }
    }
    for (int m = 0; m < c1 - c0; ++m, o += st) {
      f5 = nxt;
      if (m + 1 < c1 - c0) nxt = value(o + 4 * st);
      const double uf = s_uf[m][lane];
      const bool neg = (s_neg[m] >> lane) & 1;
      bad = wide(f5) ? 6 : bad > 0 ? bad - 1 : 0;
      t5 = mc<typename C::c13>(f5);
      e2 = e3;
      e3 = mc<typename C::c56>(f3);
      // the cell terms that face m newly needs, if it or the two after it use them
      const int any = s_any[m] | s_any[m + 1] | s_any[m + 2];
      tp0 = tp1;
      tp1 = tp2;
      tn0 = tn1;
      tn1 = tn2;
      if (any & 1) tp2 = cell_term<F32>(k, f2, f3, f4);
      if (any & 2) tn2 = cell_term<F32>(k, f5, f4, f3);
      const double g1 = neg ? f5 : f0, g2 = neg ? f4 : f1, g3 = neg ? f3 : f2, g4 = neg ? f2 : f3,
                   g5 = neg ? f1 : f4;
      double wv;
      if (bad)
        wv = weno_any<F32>(g1, g2, g3, g4, g5);
      else
        wv = weno_core<F32>(k, g1, g2, g3, g4, g5, neg ? t5 : t0, neg ? t4 : t1, neg ? t3 : t2,
                            neg ? t2 : t3, neg ? t1 : t4, neg ? e3 : e2, neg ? e2 : e3,
                            neg ? tn2 : tp0, neg ? tn1 : tp1, neg ? tn0 : tp2);
      const double r = D.dd(k.mul(uf, wv));
      if (live) Fd[o] = r;
      f0 = f1;
      f1 = f2;
      f2 = f3;
      f3 = f4;
      f4 = f5;
      t0 = t1;
      t1 = t2;
      t2 = t3;
      t3 = t4;
      t4 = t5;
    }
  }
}

inline Plan make_plan(const Geo& g, const Phys& P) {
  Plan p{};
  p.ndim = g.ndim;
  const int n[3] = {g.nci, g.ncj, g.nck};
  const long long s[3] = {1, g.sy, g.sz};
  const DivC dd[3] = {P.dd[0], P.dd[1], P.dd[2]};
  const long long base = g.ng + g.sy * g.ng + (g.ndim == 3 ? g.sz * g.ng : 0);
  long long chunks = 0;  // 32-line chunks per face layer, all directions
  for (int d = 0; d < g.ndim; ++d) {
    Dir& D = p.d[d];
    const int a = d == 0 ? 1 : 0, b = d == 2 ? 1 : 2;  // transverse axes
    D.st = s[d];
    D.sa = s[a];
    D.sb = g.ndim == 3 ? s[b] : 0;
    D.base = base;
    D.n = n[d];
    D.na = n[a];
    D.lines = n[a] * (g.ndim == 3 ? n[b] : 1);
    D.dd = dd[d];
    chunks += (long long)((D.lines + 31) / 32) * (D.n + 1);
  }
  // faces per segment: as many as leave the launch 16 warps per sub-partition, 2 at
  // least (a segment starts with the work of about three faces).  Measured against
  // 8 warps and 4 faces at least, per launch: 24x20x16 33 -> 21 us, 64x48 18 -> 13,
  // 64^3 487 -> 428 (with the split below), 800x700 491 -> 407; 32 warps: 449, 406.
  const long long want = 16LL * 4 * 152;
  int len = LSEG;
  while (len > 2 && chunks * g.nv / len < want) len >>= 1;
  int first = 0;
  for (int d = 0; d < g.ndim; ++d) {
    Dir& D = p.d[d];
    D.nseg = (D.n + len) / len;  // ceil((n + 1) / len)
    D.seg = (D.n + D.nseg) / D.nseg;
    D.first = first;
    first += (D.lines + 31) / 32 * D.nseg;
  }
  p.blocks = first;
  return p;
}

template <bool F32>
inline void launch(const Geo& g, const Phys& P, int ve, const double* U, const double* pr,
                   const double* vel, double* F, cudaStream_t st) {
  const Plan p = make_plan(g, P);
  // warps per block: 3 to 5, whichever leaves the fewest idle in the last round
  int w = WMAX;
  for (int q = WMAX - 1; q >= 3; --q)
    if ((g.nv + q - 1) / q * q < (g.nv + w - 1) / w * w) w = q;
  // The rounds of a block's warps over the variables become blocks of their own
  // below 16 waves of blocks, where the last wave counts (64^3 487 -> 445 us); above,
  // forming the face velocities once per round costs more (192^3 10.43 -> 10.85 ms).
  const int rounds = (g.nv + w - 1) / w;
  const int split = p.blocks <= 16 * 4 * 152 ? rounds : 1;
  k_weno_flux<F32><<<dim3(p.blocks, split), 32 * w, 0, st>>>(p, g.sv, g.nv, ve, U, pr, vel, F);
}

}  // namespace fstflux

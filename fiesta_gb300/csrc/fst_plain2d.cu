// fst_plain2d.cu — plain FP64 right-hand side of cart2d_func::compute
// (src/cart2d.cpp:151-237) and gen2d_func::compute (src/gen2d.cpp:103-130),
// and the stage combine of rkAdvance for sm_103a.  The flux pass carries the
// three 2D schemes of both modules (WENO5, centered4, QUICK); on generalized
// grids the primitive pass writes the contravariant velocity and the cell
// pass applies the metric pressure gradient.
//
// Same structure as the 3D path: one pass for primitives and the three
// C-equation maxima, one pass for WENO fluxes, one pass for the viscous and
// C-equation face terms, one pass for the cell update fused with the RK stage.
// The 2D reference differs from 3D in ways kept here on purpose: double
// WENO constants (src/flux.hpp:41-59), constant mu = 2.928e-5 and the
// vel(i,j-1,1) operand in the x-face du/dy (src/viscosity.hpp:62-68), a heat
// flux with k = 0.026 (src/viscosity.hpp:111-136), buoyancy only where
// |rho - rho_ref| >= 1e-6 with |m_y/rho_1| (src/buoyancy.hpp:49-73), the wave
// speed read from a stride-2 species table without /rho (src/ceq.hpp:42-78),
// four C-equation variables with the fifth left unchanged, and no delta term
// in the C-equation face tensor (src/ceq.hpp:200-245).  Built with
// --fmad=false.
#include "fst_flux_dev.cuh"

namespace {
using fst64::div_by;
using fst64::div_rn;
using fst64::eight;
using fst64::half;
using fst64::mul_call;
using fst64::mul_rn;
using fst64::twice;

// calculateRhoPT2D (src/secondary.hpp:60-107), computeVelocity2D
// (src/velocity.hpp:85-99); maxWaveSpeed2D and maxCvar2D(var, 1)
// (src/ceq.hpp:23-78) over the interior.
__global__ void __launch_bounds__(256) k_prim2d(Geo g, Phys P, const double* __restrict__ U,
                                                double* __restrict__ rho, double* __restrict__ pr,
                                                double* __restrict__ vel, double* __restrict__ T,
                                                double* __restrict__ nrg,
                                                unsigned long long* __restrict__ red,
                                                const double* __restrict__ met) {
  const long long c = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const long long sv = g.sv;
  const fst64::Fused k(P.ns);
  unsigned long long kS = FST_KEY_LOWEST, kC = FST_KEY_LOWEST;
  if (c < sv) {
    double r = 0.0;
    for (int s = 0; s < P.ns; ++s) r = k.add(r, U[c + sv * (3 + s)]);
    const fst64::Recip rr = fst64::recip_of(r);
    double Cp = 0, Cv = 0, Cp2 = 0, Cv2 = 0;
    for (int s = 0; s < P.ns; ++s) {
      double ys = div_by(U[c + sv * (3 + s)], rr);
      Cp = k.add(Cp, mul_rn(ys, P.cp_s[s]));
      Cv = k.add(Cv, mul_rn(ys, P.cv_s[s]));
      if (red) {
        Cp2 = k.add(Cp2, mul_rn(ys, P.cp2_s[s]));
        Cv2 = k.add(Cv2, mul_rn(ys, P.cv2_s[s]));
      }
    }
    const double gam = div_rn(Cp, Cv);
    const double m0 = U[c], m1 = U[c + sv], E = U[c + 2 * sv];
    const double mm = k.add(mul_rn(m0, m0), mul_rn(m1, m1));
    const double p = mul_rn(k.sub(gam, 1.0), k.sub(E, mul_rn(div_by(0.5, rr), mm)));
    const double u = div_by(m0, rr), v = div_by(m1, rr);
    rho[c] = r;
    pr[c] = p;
    if (met) {
      // computeGenVelocity2D (src/velocity.hpp:49-66), metric (a,b) at
      // met[c + sv*(a + 2b)]
      vel[c] = k.add(div_by(mul_rn(met[c], m0), rr), div_by(mul_rn(met[c + 2 * sv], m1), rr));
      vel[c + sv] =
          k.add(div_by(mul_rn(met[c + sv], m0), rr), div_by(mul_rn(met[c + 3 * sv], m1), rr));
    } else {
      vel[c] = u;
      vel[c + sv] = v;
    }
    if (T) T[c] = div_rn(p, mul_rn(k.sub(Cp, Cv), r));
    if (nrg) nrg[c] = k.sub(div_by(E, rr),
                           mul_rn(half(r), k.add(mul_rn(u, u), mul_rn(v, v))));
    if (red) {
      int i = (int)(c % g.sy), j = (int)(c / g.sy);
      bool in = i >= g.ng && i < g.ngi - g.ng && j >= g.ng && j < g.ngj - g.ng;
      if (in) {
        const double gam2 = div_rn(Cp2, Cv2);
        double a = sqrt(div_by(mul_rn(gam2, p), rr));
        double s = k.add(a, sqrt(mm));
        fst_key_max(kS, s);
        fst_key_max(kC, fabs(U[c + sv * (P.nv + 1)]));
      }
    }
  }
  if (red) fst_key_max_block<8>(red, kS, kC);
}

// The centred and QUICK schemes (computeFluxCentered2D / computeFluxQuick2D,
// src/flux.hpp:108-221) for all v < nv, face box [ng-1, ngi-ng) x [ng-1,
// ngj-ng).  F[(dir*nv + v)*sv + cell].  (WENO5: fst_flux_dev.cuh.)
__global__ void __launch_bounds__(128) k_flux2d(Geo g, Phys P, const double* __restrict__ U,
                                                const double* __restrict__ rho,
                                                const double* __restrict__ pr,
                                                const double* __restrict__ vel,
                                                double* __restrict__ F) {
  const int i = g.ng - 1 + blockIdx.x * blockDim.x + threadIdx.x;
  const int j = g.ng - 1 + blockIdx.y * blockDim.y + threadIdx.y;
  if (i >= g.ngi - g.ng || j >= g.ngj - g.ng) return;
  const long long c = fst_idx(g, i, j, 0);
  const long long sv = g.sv;
  if (P.scheme == FST_SCHEME_CENTERED4) {
    // computeFluxCentered2D (src/flux.hpp:108-167): fourth-order centred
    // face values; face velocity from var(., dir) / rho, p added for the
    // energy only
#pragma unroll 1
    for (int dir = 0; dir < 2; ++dir) {
      const long long s = dir == 0 ? 1 : g.sy;
      const double* m = U + sv * dir;
      const double uf =
          div_rn(0.0 - div_rn(m[c + 2 * s], rho[c + 2 * s]) + div_rn(7.0 * m[c + s], rho[c + s]) +
                     div_rn(7.0 * m[c], rho[c]) - div_rn(m[c - s], rho[c - s]),
                 12.0);
      const double pf =
          div_rn(0.0 - pr[c + 2 * s] + 7.0 * pr[c + s] + 7.0 * pr[c] - pr[c - s], 12.0);
      const DivC dd = dir == 0 ? P.dd[0] : P.dd[1];
      double* Fd = F + (long long)dir * P.nv * sv;
#pragma unroll 1
      for (int v = 0; v < P.nv; ++v) {
        const double* q = U + sv * v;
        double x1 = div_rn(0.0 - q[c + 2 * s] + 7.0 * q[c + s] + 7.0 * q[c] - q[c - s], 12.0);
        if (v == 2) x1 = x1 + pf;
        Fd[sv * v + c] = dd(uf * x1);
      }
    }
    return;
  }
#pragma unroll 1
  for (int dir = 0; dir < 2; ++dir) {
    const long long s = dir == 0 ? 1 : g.sy;
    const double* vd = vel + sv * dir;
    const double uf =
        div_rn(-vd[c + 2 * s] + 7.0 * vd[c + s] + 7.0 * vd[c] - vd[c - s], 12.0);
    const DivC dd = dir == 0 ? P.dd[0] : P.dd[1];
    double* Fd = F + (long long)dir * P.nv * sv;
#pragma unroll 1
    for (int v = 0; v < P.nv; ++v) {
      const double* q = U + sv * v;
      const long long o = uf < 0.0 ? -s : s;  // stencil runs upwind
      const long long c0 = uf < 0.0 ? c + 2 * s : c - s;
      double f1 = q[c0], f2 = q[c0 + o], f3 = q[c0 + 2 * o];
      const double p1 = pr[c0], p2 = pr[c0 + o], p3 = pr[c0 + 2 * o];
      if (v == 2) {
        f1 = f1 + p1; f2 = f2 + p2; f3 = f3 + p3;
      } else if (!(fst_finite(p1) && fst_finite(p2) && fst_finite(p3))) {
        // var + 0*p of the reference: NaN where a pressure is not finite
        f1 = f1 + 0.0 * p1; f2 = f2 + 0.0 * p2; f3 = f3 + 0.0 * p3;
      }
      Fd[sv * v + c] = dd(uf * (0.75 * f2 + 0.375 * f3 - 0.125 * f1));
    }
  }
}

// calculateStressTensor2dv + calculateHeatFlux2dv (src/viscosity.hpp:25-136)
// and computeCeqFlux2D * computeCeqFaces2D (src/ceq.hpp:200-267) on the faces
// with normal F of each face index (blockIdx.z = F).  Only the stress components
// the momenta take on that face are formed.
// S[(F*3 + {0:xx,1:xy,2:yy})*sv + cell], Q[F*sv + cell],
// MF[((F*2+d)*2+w)*sv + cell].
template <int F>
__device__ __forceinline__ void face_terms2d(const Geo& g, const Phys& P, const fst64::Fused& k,
                                             long long c, const double* __restrict__ U,
                                             const double* __restrict__ rho,
                                             const double* __restrict__ vel,
                                             const double* __restrict__ T,
                                             const unsigned long long* __restrict__ red,
                                             double* __restrict__ S, double* __restrict__ Q,
                                             double* __restrict__ MF) {
  constexpr int A = 1 - F;
  const long long sv = g.sv;
  const long long sf = F == 0 ? 1 : g.sy, st = F == 0 ? g.sy : 1;
  double G[2][2], tm[2];  // G[d][w]; tm[w]: the lower pair's sum of the tangential difference
#pragma unroll
  for (int w = 0; w < 2; ++w) {
    const double* u = vel + sv * w;
    G[F][w] = P.dd[F](k.sub(u[c + sf], u[c]));
    tm[w] = k.add(u[c - st], u[c + sf - st]);
    G[A][w] = P.d4[A](k.sub(k.add(u[c + st], u[c + sf + st]), tm[w]));
  }
  if (P.visc) {
    const double mu = P.mu2d;
    double dudy = G[1][0];
    // the reference's vel(i,j-1,1) in du/dy on the x faces (src/viscosity.hpp:68)
    if (F == 0)
      dudy = P.d4[1](k.sub(k.add(vel[c + st], vel[c + sf + st]),
                           k.add(vel[c + sv - st], vel[c + sf - st])));
    const double n = F == 0 ? k.sub(twice(G[0][0]), G[1][1]) : k.sub(twice(G[1][1]), G[0][0]);
    S[(long long)(F * 3 + 2 * F) * sv + c] = mul_call((2.0 / 3.0) * mu, n);
    S[(long long)(F * 3 + 1) * sv + c] = mul_call(mu, k.add(dudy, G[0][1]));
    Q[F * sv + c] = P.dd[F](mul_call(-P.kheat2d, k.sub(T[c + sf], T[c])));
  }
  if (P.ceq) {
    const double* C = U + sv * P.nv;
    const double maxCh = fst_unkey(red[1]);
    const double alpha = mul_call(div_rn(P.dxmag2, k.add(maxCh, 1.0e-6)), P.alpha);  // src/cart2d.cpp:227
    auto mean = [&](const double* a) { return half(k.add(a[c], a[c + sf])); };
    const double ar = mul_call(mul_call(alpha, mean(rho)), mean(C + sv));
    const double ct[2] = {mean(C + 2 * sv), mean(C + 3 * sv)};
    const double own = mul_call(ct[F], ct[F]), other = mul_call(ct[A], ct[A]);
    const double ctmag = k.add(F == 0 ? k.add(own, other) : k.add(other, own), 1.0e-6);
    const fst64::Recip rmag = fst64::recip_of(ctmag);
#pragma unroll
    for (int d = 0; d < 2; ++d) {
      const double cc = d == F ? own : mul_call(ct[F], ct[d]);
      const double m = fst64::div_call(mul_call(ar, cc), rmag.hi, rmag.lo, rmag.R);
#pragma unroll
      for (int w = 0; w < 2; ++w)
        MF[(long long)((F * 2 + d) * 2 + w) * sv + c] = k.mul(m, G[d][w]);
    }
  }
}

__global__ void __launch_bounds__(128) k_faces2d(Geo g, Phys P, const double* __restrict__ U,
                                                 const double* __restrict__ rho,
                                                 const double* __restrict__ vel,
                                                 const double* __restrict__ T,
                                                 const unsigned long long* __restrict__ red,
                                                 double* __restrict__ S, double* __restrict__ Q,
                                                 double* __restrict__ MF) {
  const int i = g.ng - 1 + blockIdx.x * blockDim.x + threadIdx.x;
  const int j = g.ng - 1 + blockIdx.y * blockDim.y + threadIdx.y;
  if (i >= g.ngi - g.ng || j >= g.ngj - g.ng) return;
  const long long c = fst_idx(g, i, j, 0);
  const fst64::Fused k(P.nv);
  if (blockIdx.z == 0) face_terms2d<0>(g, P, k, c, U, rho, vel, T, red, S, Q, MF);
  else face_terms2d<1>(g, P, k, c, U, rho, vel, T, red, S, Q, MF);
}

// Per interior cell: advect2D, applyPressureGradient2D, computeBuoyancy,
// applyViscousTerm2dv, calculateRhoGrad2D, updateCeq2D, applyCeq2D, then the
// stage combine (src/rk.cpp:42-69).  blockIdx.z: 0 the momenta and energy, 1 the
// species, 2 the C variables, which share nothing.
template <int PER_SM>
__global__ void __launch_bounds__(128, PER_SM) k_cell2d(Geo g, Phys P, const double* __restrict__ U,
                                                const double* __restrict__ rho,
                                                const double* __restrict__ pr,
                                                const double* __restrict__ vel,
                                                const double* __restrict__ nrg,
                                                const double* __restrict__ F,
                                                const double* __restrict__ S,
                                                const double* __restrict__ Q,
                                                const double* __restrict__ MF,
                                                const unsigned long long* __restrict__ red,
                                                const double* Uold, double* Unew, double coef,
                                                double* __restrict__ Rout,
                                                const double* __restrict__ met) {
  const int i = g.ng + blockIdx.x * blockDim.x + threadIdx.x;
  const int j = g.ng + blockIdx.y * blockDim.y + threadIdx.y;
  if (i >= g.ngi - g.ng || j >= g.ngj - g.ng) return;
  const long long c = fst_idx(g, i, j, 0);
  const long long sv = g.sv, sx = 1, sy = g.sy;
  const int nv = P.nv;
  const fst64::Fused k(nv);
  auto emit = [&](int v, double R) {
    if (Rout) Rout[c + sv * v] = R;
    else Unew[c + sv * v] = k.add(Uold[c + sv * v], mul_call(coef, R));
  };
  auto divF = [&](int v) {
    const double* Fx = F + sv * v;
    const double* Fy = F + sv * (nv + v);
    return -k.add(k.sub(Fx[c], Fx[c - sx]), k.sub(Fy[c], Fy[c - sy]));
  };
  // ((a- - 8 b-) + 8 b+) - a+ of the four neighbours along a direction
  auto d4sum = [&](double am, double bm, double bp, double ap) {
    return k.sub(k.add(k.sub(am, eight(bm)), eight(bp)), ap);
  };
  if (blockIdx.z == 1) {
    for (int v = 3; v < nv; ++v) emit(v, divF(v));
    // C-equation variables carried without a right-hand side (the generalized
    // module evolves none): U + coef*0, as the reference's zero dvar gives
    if (!P.ceq)
      for (int v = nv; v < g.nvt; ++v) emit(v, 0.0);
    return;
  }
  if (blockIdx.z == 2) {
    auto d4 = [&](const double* a, int f) {
      const long long s = f == 0 ? sx : sy;
      return P.d12[f].call(d4sum(a[c - 2 * s], a[c - s], a[c + s], a[c + 2 * s]));
    };
    const double dxr = d4(rho, 0), dyr = d4(rho, 1);
    const double dxe = d4(nrg, 0), dye = d4(nrg, 1);
    const double dxu = d4(vel, 0), dyv = d4(vel + sv, 1);
    const double g2 = k.add(mul_call(dxr, dxr), mul_call(dyr, dyr));
    const double rgrad = sqrt(g2);
    const double divu = k.add(dxu, dyv);
    const double dnednr = mul_call(k.add(mul_call(dxr, dxe), mul_call(dyr, dye)), g2);
    // (1 - i1) i2 rgrad and i1 rgrad of the reference: the factors are 0 or 1
    const bool i1 = dnednr < 0.0, i2 = divu < 0.0;
    const double maxS = fst_unkey(red[0]);
    const double src = div_rn(maxS, P.eps * P.dxmag);
    const double dif = P.kap * maxS * P.dxmag;
#pragma unroll 1
    for (int n = 0; n < 4; ++n) {
      const double Gn = n == 0   ? mul_call(!i1 && i2 ? 1.0 : 0.0, rgrad)
                        : n == 1 ? mul_call(i1 ? 1.0 : 0.0, rgrad)
                        : n == 2 ? -dyr
                                 : dxr;
      const double* Cn = U + sv * (nv + n);
      const double cc = Cn[c];
      const double dx_right = P.dd[0].call(k.sub(Cn[c + sx], cc));
      const double dx_left = P.dd[0].call(k.sub(cc, Cn[c - sx]));
      const double dy_top = P.dd[1].call(k.sub(Cn[c + sy], cc));
      const double dy_bot = P.dd[1].call(k.sub(cc, Cn[c - sy]));
      const double lap = k.sub(k.add(k.sub(dx_right, dx_left), dy_top), dy_bot);
      emit(nv + n, k.add(mul_call(src, k.sub(Gn, cc)), mul_call(dif, lap)));
    }
    emit(nv + 4, 0.0);  // the fifth C variable has no right-hand side
    return;
  }
  double R0 = divF(0), R1 = divF(1), R2 = divF(2);
  if (met) {
    // applyGenPressureGradient2D (src/presgrad.hpp:148-190)
    auto d4m = [&](long long s, int a, int w) {
      const double* m = met + sv * (a + 2 * w);
      // 8.0 * p * m: the product with 8 first, exact
      return div_rn(k.sub(k.add(k.sub(mul_call(pr[c - 2 * s], m[c - 2 * s]),
                                      mul_call(eight(pr[c - s]), m[c - s])),
                                mul_call(eight(pr[c + s]), m[c + s])),
                          mul_call(pr[c + 2 * s], m[c + 2 * s])),
                    12.0);
    };
    R0 = k.sub(R0, k.add(d4m(sx, 0, 0), d4m(sy, 1, 0)));
    R1 = k.sub(R1, k.add(d4m(sx, 0, 1), d4m(sy, 1, 1)));
  } else {
    R0 = k.sub(R0, P.d12[0].call(d4sum(pr[c - 2 * sx], pr[c - sx], pr[c + sx], pr[c + 2 * sx])));
    R1 = k.sub(R1, P.d12[1].call(d4sum(pr[c - 2 * sy], pr[c - sy], pr[c + sy], pr[c + 2 * sy])));
  }
  if (P.buoyancy) {
    const double vb = div_rn(U[c + sv], U[c + 3 * sv]);
    const double rhop = k.sub(rho[c], P.rho_ref);
    const double eps = 1e-6;
    if (rhop >= eps || rhop <= -eps) {
      const double f = mul_call(-P.g, rhop);
      R1 = k.add(R1, f);
      R2 = k.add(R2, mul_call(fabs(vb), f));
    }
  }
  if (P.visc) {
    const double* u = vel;
    const double* v = vel + sv;
    auto mean = [&](const double* a, long long s) { return half(k.add(a[c + s], a[c])); };
    const double* sxx = S;
    const double* sxy = S + sv;
    const double* syx = S + 4 * sv;  // stressy(1,0) == stressy(0,1)
    const double* syy = S + 5 * sv;
    auto diff = [&](const double* s, int f) {
      return P.dd[f].call(k.sub(s[c], s[c - (f == 0 ? sx : sy)]));
    };
    // (a b)(face) - (a b)(face before) over the spacing
    auto work = [&](const double* a, const double* s, int f) {
      const long long st = f == 0 ? sx : sy;
      return P.dd[f].call(
          k.sub(mul_call(mean(a, st), s[c]), mul_call(mean(a, -st), s[c - st])));
    };
    const double a = k.add(diff(sxx, 0), diff(syx, 1));
    const double b = k.add(diff(sxy, 0), diff(syy, 1));
    const double c1 = k.add(k.add(k.add(work(u, sxx, 0), work(v, sxy, 0)), work(u, syx, 1)),
                            work(v, syy, 1));
    const double c2 = k.add(diff(Q, 0), diff(Q + sv, 1));
    R0 = k.add(R0, a);
    R1 = k.add(R1, b);
    R2 = k.sub(k.add(R2, c1), c2);
  }
  if (P.ceq) {
#pragma unroll 1
    for (int w = 0; w < 2; ++w) {
      double diffu = 0;
#pragma unroll 1
      for (int q = 0; q < 4; ++q) {  // (face, derivative) = (0,0), (0,1), (1,0), (1,1)
        const double* m = MF + (long long)(2 * q + w) * sv;
        const int f = q >> 1;
        diffu = k.add(diffu, P.dd[f].call(k.sub(m[c], m[c - (f == 0 ? sx : sy)])));
      }
      if (w == 0) R0 = k.add(R0, diffu);
      else R1 = k.add(R1, diffu);
    }
  }
  emit(0, R0);
  emit(1, R1);
  emit(2, R2);
}

// Stage-1 ghost cells: U1 = U + (0.5*dt)*0 over ghosts (dvar is zero there;
// src/rk.cpp:42-50 runs over every cell).  2D BCs are applied once per step,
// so stage 2 reads these.
__global__ void k_ghost2d(Geo g, const double* __restrict__ Uold, double* __restrict__ Unew,
                          double coef) {
  const long long c = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= g.sv) return;
  int i = (int)(c % g.sy), j = (int)(c / g.sy);
  bool in = i >= g.ng && i < g.ngi - g.ng && j >= g.ng && j < g.ngj - g.ng;
  if (in) return;
  for (int v = 0; v < g.nvt; ++v) Unew[c + g.sv * v] = Uold[c + g.sv * v] + coef * 0.0;
}

inline unsigned cdiv(long long a, int b) { return (unsigned)((a + b - 1) / b); }

}  // namespace

int fst_plain2d_stage(const Geo& g, const Phys& P, const Plain2DBufs& b, const double* Uin,
                      const double* Uold, double* Unew, double coef, double* Rout, bool ghosts,
                      cudaStream_t st, Prof* prof) {
  int n = 0;
  if (P.ceq) {
    fst_fill_keys(b.red, 2, FST_KEY_LOWEST, st);
  }
  FST_LAUNCH(prof, "prim2d", st, n,
             k_prim2d<<<cdiv(g.sv, 256), 256, 0, st>>>(g, P, Uin, b.rho, b.pr, b.vel,
                                                       P.visc ? b.T : nullptr,
                                                       P.ceq ? b.nrg : nullptr,
                                                       P.ceq ? b.red : nullptr, b.met));
  const dim3 bf(32, 4, 1);
  const dim3 gf(cdiv(g.nci + 1, 32), cdiv(g.ncj + 1, 4), 1);
  FST_LAUNCH(prof, "flux2d", st, n,
             if (P.scheme == FST_SCHEME_WENO5)
               fstflux::launch<false>(g, P, 2, Uin, b.pr, b.vel, b.F, st);
             else
               k_flux2d<<<gf, bf, 0, st>>>(g, P, Uin, b.rho, b.pr, b.vel, b.F));
  if (P.visc || P.ceq) {
    FST_LAUNCH(prof, "faces2d", st, n,
               k_faces2d<<<dim3(gf.x, gf.y, 2), bf, 0, st>>>(g, P, Uin, b.rho, b.vel, b.T, b.red, b.S, b.Q, b.MF));
  }
  const dim3 gc(cdiv(g.nci, 32), cdiv(g.ncj, 4), P.ceq ? 3 : 2);
  // Blocks per SM: what 72 registers a thread give (7; no bound set) while the launch is
  // a few waves long and a thread's chain counts, 10 (48 registers, some spilled) where
  // the FP64 unit's share does.  72 registers against 48: 200x100 15.4 and 16.2 us,
  // 400x300 (2925 blocks) 49.9 and 50.8, 600x500 (7125) 126 and 116, 999^2 369 and 328;
  // 12 blocks: 320 there, but 53 at 400x300.
  auto cell = gc.x * gc.y * gc.z > 4 * 7 * 152 ? k_cell2d<10> : k_cell2d<0>;
  FST_LAUNCH(prof, "cell2d", st, n,
             cell<<<gc, bf, 0, st>>>(g, P, Uin, b.rho, b.pr, b.vel, b.nrg, b.F, b.S, b.Q,
                                     b.MF, b.red, Uold, Unew, coef, Rout, b.met));
  if (ghosts && !Rout) {
    FST_LAUNCH(prof, "ghost2d", st, n,
               k_ghost2d<<<cdiv(g.sv, 256), 256, 0, st>>>(g, Uold, Unew, coef));
  }
  return n;
}

int fst_plain2d_secondary(const Geo& g, const Phys& P, const Plain2DBufs& b, const double* U,
                          cudaStream_t st) {
  k_prim2d<<<cdiv(g.sv, 256), 256, 0, st>>>(g, P, U, b.rho, b.pr, b.vel, b.T, nullptr, nullptr,
                                            nullptr);
  return 1;
}

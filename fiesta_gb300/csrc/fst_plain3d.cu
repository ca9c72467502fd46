// fst_plain3d.cu — plain FP64 right-hand side of cart3d_func::compute
// (src/cart3d.cpp:220-298) and gen3d_func::compute (src/gen3d.cpp:338-370),
// and the rkAdvance stage combine (src/rk.cpp:28-70) for sm_103a.  On
// generalized grids the primitive pass writes the contravariant velocity and
// the cell pass applies the metric pressure gradient; the flux pass is the
// same WENO5 with the reference's dz = cf.dx (src/gen3d.cpp:359).
//
// The reference runs ~41 Kokkos launches per stage with every intermediate in
// HBM.  Here a stage is four kernels:
//   k_prim3d        rho, p, velocity, mass fractions, internal energy, and the
//                   two global maxima of the C-equation (maxS, maxCh) folded
//                   into the same pass (block max + one atomicMax per block)
//   k_weno_flux     WENO5 fluxes of all nv variables (fst_flux_dev.cuh)
//   k_faces3d       the 27 face velocity gradients, shared by the viscous
//                   stress and the C-equation face terms, which are the same
//                   expressions in the reference
//   k_cell3d        flux divergence, pressure gradient, buoyancy, viscous
//                   divergence x/y/z, C-equation source + diffusion, then the
//                   RK stage combine straight into the next state buffer
// On GB300 the FP64 pipe, not HBM, bounds this path, so the design removes
// repeated FP64 work (species constants hoisted, Y_s and e computed once per
// cell, shared gradients) and moves divisions and products to the integer pipes
// (fst_fp64.cuh) while keeping the result of every operation the reference
// performs on every value it stores, in the same order.  Built with
// --fmad=false so no a*b+c is contracted: results match the reference's FP64
// run bit for bit.
#include "fst_flux_dev.cuh"

namespace {
using fst64::div_by;
using fst64::div_rn;
using fst64::eight;
using fst64::half;
using fst64::mul_call;
using fst64::mul_rn;
using fst64::twice;

// ---------------------------------------------------------------------------
// k_prim3d: calculateRhoPT3D (src/secondary.hpp:109-151), computeVelocity3D
// (src/velocity.hpp:68-83) over all cells; maxWaveSpeed (src/ceq3d.hpp:25-63)
// and maxGradFunctor(var, nv+1) (src/ceq3d.hpp:82-93) over the interior.
// Sums on the FP64 unit, the rest on the integer pipes; both about half busy, so
// warps in flight matter: 5 blocks per SM (48 registers) 0.72 ms at 192^3 and 5
// species, 4 blocks 0.77, 3 blocks 0.84 (operators throughout: 1.08 after the
// integer division, 2.4 before it).
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(256, 5) k_prim3d(Geo g, Phys P, const double* __restrict__ U,
                                                double* __restrict__ rho, double* __restrict__ pr,
                                                double* __restrict__ vel, double* __restrict__ Y,
                                                double* __restrict__ nrg, double* __restrict__ T,
                                                unsigned long long* __restrict__ red,
                                                const double* __restrict__ met) {
  const long long c = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const long long sv = g.sv;
  const fst64::Fused k(P.ns);
  unsigned long long kS = FST_KEY_LOWEST, kC = FST_KEY_LOWEST;
  if (c < sv) {
    double r = 0.0;
    for (int s = 0; s < P.ns; ++s) r = k.add(r, U[c + sv * (4 + s)]);
    const fst64::Recip rr = fst64::recip_of(r);
    double Cp = 0, Cv = 0;
    for (int s = 0; s < P.ns; ++s) {
      double ys = div_by(U[c + sv * (4 + s)], rr);
      Cp = k.add(Cp, mul_rn(ys, P.cp_s[s]));
      Cv = k.add(Cv, mul_rn(ys, P.cv_s[s]));
      if (Y) Y[c + sv * s] = ys;
    }
    const double gam = div_rn(Cp, Cv);
    const double m0 = U[c], m1 = U[c + sv], m2 = U[c + 2 * sv], E = U[c + 3 * sv];
    const double mm = k.add(k.add(mul_rn(m0, m0), mul_rn(m1, m1)), mul_rn(m2, m2));
    const double p = mul_rn(k.sub(gam, 1.0), k.sub(E, mul_rn(div_by(0.5, rr), mm)));
    const double u = div_by(m0, rr), v = div_by(m1, rr), w = div_by(m2, rr);
    rho[c] = r;
    pr[c] = p;
    if (met) {
      // computeGenVelocity3D (src/velocity.hpp:23-48): contravariant velocity
      // sum_b m(a,b) * var(b) / rho, metric (a,b) at met[c + sv*(a + 3b)]
#pragma unroll
      for (int a = 0; a < 3; ++a) {
        const double* M = met + c + sv * a;
        vel[c + sv * a] =
            k.add(k.add(div_by(mul_rn(M[0], m0), rr), div_by(mul_rn(M[3 * sv], m1), rr)),
                  div_by(mul_rn(M[6 * sv], m2), rr));
      }
    } else {
      vel[c] = u;
      vel[c + sv] = v;
      vel[c + 2 * sv] = w;
    }
    if (T) T[c] = div_rn(p, mul_rn(k.sub(Cp, Cv), r));
    // specific internal energy of calculateRhoGrad::nrg (src/ceq3d.hpp:137-141)
    if (nrg) nrg[c] = k.sub(div_by(E, rr), mul_rn(half(r), k.add(k.add(mul_rn(u, u), mul_rn(v, v)),
                                                                 mul_rn(w, w))));
    if (red) {
      int i = (int)(c % g.sy), j = (int)((c / g.sy) % g.ngj), kk = (int)(c / g.sz);
      bool in = i >= g.ng && i < g.ngi - g.ng && j >= g.ng && j < g.ngj - g.ng &&
                kk >= g.ng && kk < g.ngk - g.ng;
      if (in) {
        double a = sqrt(div_by(mul_rn(gam, p), rr));
        double s = k.add(a, div_by(sqrt(mm), rr));
        fst_key_max(kS, s);
        fst_key_max(kC, fabs(U[c + sv * (P.nv + 1)]));
      }
    }
  }
  if (red) fst_key_max_block<8>(red, kS, kC);
}

// ---------------------------------------------------------------------------
// k_faces3d: the faces with normal F of the interior cells, the 9 velocity
// gradients G[d][w] (derivative along d of velocity w) of each, then
//  - the viscous stress components that the momenta take on that face
//    (calculateStressTensor{x,y,z}3dv, src/viscosity.hpp:416-459, 499-541,
//    581-624), S[(F*6 + w)*sv + cell], and the products of each with the face's
//    mean velocity for the energy (applyViscousTerm*, :460-663), S[(F*6+3+w)*sv + cell]
//  - C-equation face terms: calculateCeqFaces * calculateCeqGrads
//    (src/ceq3d.hpp:226-332), MF[((F*3+d)*3+w)*sv + cell]
// The reference evaluates each gradient twice (stress and C-equation) with
// the same operations up to operand order of a commutative add, so the
// values are identical and are computed once here.
// One launch covers the three normals (blockIdx.x % 3): a block runs one of them.
// Sums and the last products run on the FP64 unit, all else on the integer pipes
// (fst_fp64.cuh), products and divisions as calls.  Measured at 192^3, 5 species,
// per launch: 6.4 ms with all of it inlined (the warps wait for instructions),
// 4.34 with calls, 3.74 at 7 blocks per SM instead of 5, 3.49 with 12 of a face's
// products on the FP64 unit, which then is as busy as the integer one.  A plane's
// faces are numbered row after row, so that warps are full for any row length (rows
// cut into warps of 32 left a fifth of the unit idle at 100 or 129 faces a row): step
// at 100^3, 3 species, 3683 -> 3467 us with this pass and k_cell3d so numbered, at
// 64^3 1516 -> 1485; where rows are multiples of 32 the cell pass loses 0.8 % (rows
// above and below no longer share a block), the step nothing.
// ---------------------------------------------------------------------------
template <int F>
__device__ __forceinline__ void face_terms3d(const Geo& g, const Phys& P, const fst64::Fused& k,
                                             long long c, const double* __restrict__ U,
                                             const double* __restrict__ rho,
                                             const double* __restrict__ vel,
                                             const double* __restrict__ Y,
                                             const unsigned long long* __restrict__ red,
                                             double* __restrict__ S, double* __restrict__ MF) {
  constexpr int A = F == 0 ? 1 : 0, B = F == 2 ? 1 : 2;  // the tangential axes
  const long long sv = g.sv;
  const long long st[3] = {1, g.sy, g.sz};
  const long long sf = st[F];  // outward normal step
  double G[3][3], um[3];
#pragma unroll
  for (int w = 0; w < 3; ++w) {
    const double* u = vel + sv * w;
    const double u0 = u[c], u1 = u[c + sf];
    G[F][w] = P.dd[F].call(k.sub(u1, u0));
    um[w] = half(k.add(u1, u0));
    auto tangential = [&](int d) {
      const long long t = st[d];
      return P.d4[d].call(k.sub(k.add(u[c + sf + t], u[c + t]), k.add(u[c + sf - t], u[c - t])));
    };
    G[A][w] = tangential(A);
    G[B][w] = tangential(B);
  }
  if (P.visc) {
    double mu = 0.0;
    for (int s = 0; s < P.ns; ++s)
      mu = k.add(mu, mul_call(half(k.add(Y[c + sf + sv * s], Y[c + sv * s])), P.mu_s[s]));
    const double m23 = mul_call(2.0 / 3.0, mu);
    double* Sf = S + (long long)F * 6 * sv + c;
#pragma unroll
    for (int w = 0; w < 3; ++w) {
      const double T = w == F ? mul_call(m23, k.sub(k.sub(twice(G[F][F]), G[A][A]), G[B][B]))
                              : mul_call(mu, k.add(G[w][F], G[F][w]));
      Sf[w * sv] = T;
      Sf[(3 + w) * sv] = k.mul(um[w], T);
    }
  }
  if (P.ceq) {
    const double maxCh = fst_unkey(red[1]);
    const double alpha = mul_call(div_rn(P.dxmag2, k.add(maxCh, 1.0e-6)), P.alpha);  // src/cart3d.cpp:285
    const double* C = U + sv * P.nv;
    auto mean = [&](const double* a) { return half(k.add(a[c], a[c + sf])); };
    const double ar = mul_call(mul_call(alpha, mean(rho)), mean(C + sv));
    const double cn[3] = {mean(C + 2 * sv), mean(C + 3 * sv), mean(C + 4 * sv)};
    double cc[3];  // cn[F] cn[d]
#pragma unroll
    for (int d = 0; d < 3; ++d) cc[d] = mul_call(cn[F], cn[d]);
    double cmag = 1.0e-6;
#pragma unroll
    for (int d = 0; d < 3; ++d) cmag = k.add(cmag, d == F ? cc[F] : mul_call(cn[d], cn[d]));
    const fst64::Recip rmag = fst64::recip_of(cmag);
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      const double M = k.sub(F == d ? 1.0 : 0.0, fst64::div_call(cc[d], rmag.hi, rmag.lo, rmag.R));
      const double base = mul_call(ar, M);
      double* MFd = MF + (long long)((F * 3 + d) * 3) * sv + c;
#pragma unroll
      for (int w = 0; w < 3; ++w) MFd[w * sv] = k.mul(base, G[d][w]);
    }
  }
}

__global__ void __launch_bounds__(128, 7) k_faces3d(Geo g, Phys P, const double* __restrict__ U,
                                                 const double* __restrict__ rho,
                                                 const double* __restrict__ vel,
                                                 const double* __restrict__ Y,
                                                 const unsigned long long* __restrict__ red,
                                                 double* __restrict__ S, double* __restrict__ MF) {
  const int f = blockIdx.x % 3;
  // faces c + 1/2 along f for c from the last ghost, interior cells across, row after row
  const int t = blockIdx.x / 3 * 128 + threadIdx.x, nx = g.nci + (f == 0), r = t / nx;
  const int i = g.ng - (f == 0) + t - r * nx;
  const int j = g.ng - (f == 1) + r;
  const int kk = g.ng - (f == 2) + blockIdx.z;
  if (j >= g.ngj - g.ng || kk >= g.ngk - g.ng) return;
  const long long c = fst_idx(g, i, j, kk);
  const fst64::Fused k(P.nv);
  if (f == 0) face_terms3d<0>(g, P, k, c, U, rho, vel, Y, red, S, MF);
  else if (f == 1) face_terms3d<1>(g, P, k, c, U, rho, vel, Y, red, S, MF);
  else face_terms3d<2>(g, P, k, c, U, rho, vel, Y, red, S, MF);
}

// ---------------------------------------------------------------------------
// k_cell3d: per interior cell, the rest of compute() in the reference's
// accumulation order, then the stage combine of rkAdvance:
//   mode 0: R -> Rout (fst_compute_rhs);  mode 1/2: Unew = Uold + coef*R
// advect3D (src/advect.hpp:39-61), applyPressureGradient3D (src/presgrad.hpp:44-71),
// computeBuoyancy3D (src/buoyancy.hpp:22-47), applyViscousTerm{x,y,z}3dv
// (src/viscosity.hpp:460-663), calculateRhoGrad (src/ceq3d.hpp:95-187),
// updateCeq (:189-224), applyCeq (:334-366), Loop1/Loop2 (src/rk.cpp:42-69).
// The variables that share nothing run in different blocks (blockIdx.x % roles):
// the momenta and energy, the species (advection only), the C variables; loops
// over the directions stay rolled.  Both keep the code of a block small and give
// a small grid three times the warps.  Quotients go three to a call (div3), which
// shortens the chain that bounds small grids and the calls of all: 256^3, 5 species,
// 8.31 -> 7.85 ms, 64^3 157 -> 143 us, 21x19x23, 2 species, 33 -> 25 us.  (The same in
// k_faces3d and k_cell2d costs registers: 6.70 -> 7.22 ms at 256^3, 50 -> 55 us at
// 400x300.  A block per variable: 27 us at 21x19x23, but 8.97 ms at 256^3.)
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(128, 8) k_cell3d(Geo g, Phys P, const double* __restrict__ U,
                                                const double* __restrict__ rho,
                                                const double* __restrict__ pr,
                                                const double* __restrict__ vel,
                                                const double* __restrict__ nrg,
                                                const double* __restrict__ F,
                                                const double* __restrict__ S,
                                                const double* __restrict__ MF,
                                                const unsigned long long* __restrict__ red,
                                                const double* Uold, double* Unew, double coef,
                                                double* __restrict__ Rout,
                                                const double* __restrict__ met, int roles) {
  const int role = blockIdx.x % roles;
  const int t = blockIdx.x / roles * 128 + threadIdx.x, r = t / g.nci;  // row after row
  const int i = g.ng + t - r * g.nci;
  const int j = g.ng + r;
  const int kk = g.ng + blockIdx.z;
  if (j >= g.ngj - g.ng) return;
  const long long c = fst_idx(g, i, j, kk);
  const long long sv = g.sv, sx = 1, sy = g.sy, sz = g.sz;
  const int nv = P.nv;
  const fst64::Fused k(nv);

  auto emit = [&](int v, double R) {
    if (Rout) Rout[c + sv * v] = R;
    else Unew[c + sv * v] = k.add(Uold[c + sv * v], mul_call(coef, R));
  };
  // -((Fx - Fx-) + (Fy - Fy-) + (Fz - Fz-))
  auto divF = [&](int v) {
    const double* Fx = F + sv * v;
    const double* Fy = F + sv * (nv + v);
    const double* Fz = F + sv * (2 * nv + v);
    return -k.add(k.add(k.sub(Fx[c], Fx[c - sx]), k.sub(Fy[c], Fy[c - sy])),
                  k.sub(Fz[c], Fz[c - sz]));
  };
  // ((a- - 8 b-) + 8 b+) - a+ of the four neighbours along a direction
  auto d4sum = [&](double am, double bm, double bp, double ap) {
    return k.sub(k.add(k.sub(am, eight(bm)), eight(bp)), ap);
  };
  auto stride = [&](int f) { return f == 0 ? sx : f == 1 ? sy : sz; };

  if (role == 1) {  // species: only the advective term
#pragma unroll 1
    for (int v = 4; v < nv; ++v) emit(v, divF(v));
    // C-equation variables carried without a right-hand side (the generalized
    // module evolves none): U + coef*0, as the reference's zero dvar gives
    if (!P.ceq)
      for (int v = nv; v < g.nvt; ++v) emit(v, 0.0);
    return;
  }
  if (role == 2) {  // C variables: calculateRhoGrad, updateCeq
    double gr[3], ge[3], divu = 0.0;
#pragma unroll 1
    for (int f = 0; f < 3; ++f) {
      const long long s = stride(f);
      const DivC& d12 = P.d12[f];
      auto d4 = [&](const double* a) { return d4sum(a[c - 2 * s], a[c - s], a[c + s], a[c + 2 * s]); };
      const fst64::Quot3 d = div3(d12, d4(rho), d12, d4(nrg), d12, d4(vel + sv * f));
      const double r = d.x, e = d.y, u = d.z;
      divu = f == 0 ? u : k.add(divu, u);
      if (f == 0) { gr[0] = r; ge[0] = e; }
      else if (f == 1) { gr[1] = r; ge[1] = e; }
      else { gr[2] = r; ge[2] = e; }
    }
    const double g2 = k.add(k.add(mul_call(gr[0], gr[0]), mul_call(gr[1], gr[1])), mul_call(gr[2], gr[2]));
    const double rgrad = sqrt(g2);
    const double dnednr = mul_call(
        k.add(k.add(mul_call(gr[0], ge[0]), mul_call(gr[1], ge[1])), mul_call(gr[2], ge[2])), g2);
    const bool ind = dnednr < 0.0;
    const double maxS = fst_unkey(red[0]);
    const double src = div_rn(maxS, P.eps * P.dxmag);
    const double dif = P.kap * maxS * P.dxmag;
#pragma unroll 1
    for (int n = 0; n < 5; ++n) {
      // (1 - ind) rgrad, ind rgrad of the reference: the factors are 0 or 1
      double Gn;
      if (n == 0) Gn = divu < 0 ? mul_call(ind ? 0.0 : 1.0, rgrad) : 0.0;
      else if (n == 1) Gn = mul_call(ind ? 1.0 : 0.0, rgrad);
      else Gn = n == 2 ? gr[0] : n == 3 ? gr[1] : gr[2];
      const double* Cn = U + sv * (nv + n);
      const double cc = Cn[c], c2 = twice(cc);
      const fst64::Quot3 l = div3(P.dd[0], k.add(k.sub(Cn[c - sx], c2), Cn[c + sx]),  //
                                  P.dd[1], k.add(k.sub(Cn[c - sy], c2), Cn[c + sy]),
                                  P.dd[2], k.add(k.sub(Cn[c - sz], c2), Cn[c + sz]));
      const double lap = k.add(k.add(l.x, l.y), l.z);
      emit(nv + n, k.add(mul_call(src, k.sub(Gn, cc)), mul_call(dif, lap)));
    }
    return;
  }

  double R0 = divF(0), R1 = divF(1), R2 = divF(2), R3 = divF(3);
  if (met) {
    // applyGenPressureGradient3D (src/presgrad.hpp:72-146): fourth-order
    // differences of p * m(a, w) along each computational direction a
#pragma unroll 1
    for (int w = 0; w < 3; ++w) {
      auto d4m = [&](long long s, int a) {
        const double* m = met + sv * (a + 3 * w);
        // 8.0 * p * m: the product with 8 first, exact
        return div_rn(k.sub(k.add(k.sub(mul_call(pr[c - 2 * s], m[c - 2 * s]),
                                        mul_call(eight(pr[c - s]), m[c - s])),
                                  mul_call(eight(pr[c + s]), m[c + s])),
                            mul_call(pr[c + 2 * s], m[c + 2 * s])),
                      12.0);
      };
      const double d = k.add(k.add(d4m(sx, 0), d4m(sy, 1)), d4m(sz, 2));
      const double R = k.sub(w == 0 ? R0 : w == 1 ? R1 : R2, d);  // one operation, not three predicated
      if (w == 0) R0 = R;
      else if (w == 1) R1 = R;
      else R2 = R;
    }
  } else {  // pressure gradient; the reference uses dz = cd(2) for the z term
#pragma unroll 1
    for (int f = 0; f < 3; ++f) {
      const long long s = stride(f);
      const DivC& d12 = f == 2 ? P.d12pz : P.d12[f];
      const double d = d12.call(d4sum(pr[c - 2 * s], pr[c - s], pr[c + s], pr[c + 2 * s]));
      const double R = k.sub(f == 0 ? R0 : f == 1 ? R1 : R2, d);  // one operation, not three predicated
      if (f == 0) R0 = R;
      else if (f == 1) R1 = R;
      else R2 = R;
    }
  }
  if (P.buoyancy) {
    const double vb = div_rn(U[c + sv], rho[c]);
    const double f = mul_call(-P.g, k.sub(rho[c], P.rho_ref));
    R1 = k.add(R1, f);
    R3 = k.add(R3, mul_call(vb, f));
  }
  if (P.visc) {
#pragma unroll 1
    for (int f = 0; f < 3; ++f) {
      const long long s = stride(f);
      const DivC& dd = P.dd[f];
      const double* Sf = S + (long long)f * 6 * sv + c;
      auto diff = [&](int q) { return k.sub(Sf[q * sv], Sf[q * sv - s]); };
      const fst64::Quot3 m = div3(dd, diff(0), dd, diff(1), dd, diff(2));
      R0 = k.add(R0, m.x);
      R1 = k.add(R1, m.y);
      R2 = k.add(R2, m.z);
      const fst64::Quot3 e = div3(dd, diff(3), dd, diff(4), dd, diff(5));
      R3 = k.add(R3, k.add(k.add(e.x, e.y), e.z));
    }
  }
  if (P.ceq) {  // applyCeq
    double diffu[3] = {0.0, 0.0, 0.0};
#pragma unroll 1
    for (int f = 0; f < 3; ++f) {
      const long long s = stride(f);
      const DivC& dd = P.dd[f];
#pragma unroll 1
      for (int d = 0; d < 3; ++d) {
        const double* m = MF + (long long)((f * 3 + d) * 3) * sv + c;
        auto diff = [&](int w) { return k.sub(m[w * sv], m[w * sv - s]); };
        const fst64::Quot3 q = div3(dd, diff(0), dd, diff(1), dd, diff(2));
        diffu[0] = k.add(diffu[0], q.x);
        diffu[1] = k.add(diffu[1], q.y);
        diffu[2] = k.add(diffu[2], q.z);
      }
    }
    R0 = k.add(R0, diffu[0]);
    R1 = k.add(R1, diffu[1]);
    R2 = k.add(R2, diffu[2]);
  }
  emit(0, R0);
  emit(1, R1);
  emit(2, R2);
  emit(3, R3);
}

// Stage-1 ghost cells: U1 = U + (0.5*dt)*0 over ghosts (dvar is zero there;
// src/rk.cpp:42-50 runs over every cell).  In 3D the next ghost fill
// rewrites them, except where a periodic copy with fewer interior cells than
// ghost layers reads ghosts; this keeps that case exact too.
__global__ void k_ghost3d(Geo g, const double* __restrict__ Uold, double* __restrict__ Unew,
                          double coef) {
  const long long c = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= g.sv) return;
  int i = (int)(c % g.sy), j = (int)((c / g.sy) % g.ngj), k = (int)(c / g.sz);
  bool in = i >= g.ng && i < g.ngi - g.ng && j >= g.ng && j < g.ngj - g.ng && k >= g.ng &&
            k < g.ngk - g.ng;
  if (in) return;
  for (int v = 0; v < g.nvt; ++v) Unew[c + g.sv * v] = Uold[c + g.sv * v] + coef * 0.0;
}

inline unsigned cdiv(long long a, int b) { return (unsigned)((a + b - 1) / b); }

}  // namespace

// One right-hand-side evaluation of Uin (ghosts already filled) followed by
// the chosen output; returns the number of launches.
int fst_plain3d_stage(const Geo& g, const Phys& P, const Plain3DBufs& b, const double* Uin,
                      const double* Uold, double* Unew, double coef, double* Rout, bool ghosts,
                      cudaStream_t st, Prof* prof) {
  int n = 0;
  if (P.ceq) {
    fst_fill_keys(b.red, 2, FST_KEY_LOWEST, st);
  }
  FST_LAUNCH(prof, "prim3d", st, n,
             k_prim3d<<<cdiv(g.sv, 256), 256, 0, st>>>(g, P, Uin, b.rho, b.pr, b.vel,
                                                       P.visc ? b.Y : nullptr,
                                                       P.ceq ? b.nrg : nullptr, nullptr,
                                                       P.ceq ? b.red : nullptr, b.met));
  FST_LAUNCH(prof, "flux3d", st, n, fstflux::launch<true>(g, P, 3, Uin, b.pr, b.vel, b.F, st));
  if (P.visc || P.ceq) {
    const dim3 gf(3 * cdiv((long long)(g.nci + 1) * (g.ncj + 1), 128), 1, g.nck + 1);
    FST_LAUNCH(prof, "faces3d", st, n,
               k_faces3d<<<gf, 128, 0, st>>>(g, P, Uin, b.rho, b.vel, b.Y, b.red, b.S, b.MF));
  }
  const int roles = P.ceq ? 3 : 2;
  const dim3 gc(roles * cdiv((long long)g.nci * g.ncj, 128), 1, g.nck);
  FST_LAUNCH(prof, "cell3d", st, n,
             k_cell3d<<<gc, 128, 0, st>>>(g, P, Uin, b.rho, b.pr, b.vel, b.nrg, b.F, b.S, b.MF,
                                         b.red, Uold, Unew, coef, Rout, b.met, roles));
  if (ghosts && !Rout)
    FST_LAUNCH(prof, "ghost3d", st, n,
               k_ghost3d<<<cdiv(g.sv, 256), 256, 0, st>>>(g, Uold, Unew, coef));
  return n;
}

// Secondary variables (postStep path): u, v, w, p, T, rho over all cells.
int fst_plain3d_secondary(const Geo& g, const Phys& P, const Plain3DBufs& b, const double* U,
                          cudaStream_t st) {
  k_prim3d<<<cdiv(g.sv, 256), 256, 0, st>>>(g, P, U, b.rho, b.pr, b.vel, nullptr, nullptr, b.T,
                                            nullptr, nullptr);
  return 1;
}

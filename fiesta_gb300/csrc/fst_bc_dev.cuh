// fst_bc_dev.cuh — per-line ghost-fill logic of applyBCs (src/bc.cpp:33-176),
// shared by the single-case launches (fst_bc.cu) and the batched 2D
// ensemble (fst_batch.cu).
#pragma once
#include "fst_common.cuh"

namespace fstbc {

// bc_xPer / bc_yPer / bc_zPer for one (transverse a, transverse b, v) line.
__device__ __forceinline__ void periodic_line(const Geo& g, double* __restrict__ U, int axis,
                                              int a, int b, int v) {
  long long base, st;
  int nc;
  if (axis == 0) {  // a=j, b=k
    base = g.sy * a + g.sz * b + g.sv * v; st = 1; nc = g.nci;
  } else if (axis == 1) {  // a=i, b=k
    base = a + g.sz * b + g.sv * v; st = g.sy; nc = g.ncj;
  } else {  // a=i, b=j
    base = a + g.sy * b + g.sv * v; st = g.sz; nc = g.nck;
  }
  for (int q = 0; q < g.ng; ++q) {
    U[base + st * q] = U[base + st * (nc + q)];
    U[base + st * (nc + g.ng + q)] = U[base + st * (g.ng + q)];
  }
}

// bc_gen::operator() (src/bc.cpp:42-130) for the ghost line through
// transverse (a, b) of one face.
__device__ __forceinline__ void face_line(const Geo& g, double* __restrict__ U, int axis, int side,
                                          int type, int a, int b) {
  const int h = side ? 1 : -1;
  int i, j, k, ih = 0, jh = 0, kh = 0;
  if (axis == 0) { i = side ? g.ng + g.nci - 1 : g.ng; j = a; k = b; ih = h; }
  else if (axis == 1) { i = a; j = side ? g.ng + g.ncj - 1 : g.ng; k = b; jh = h; }
  else { i = a; j = b; k = side ? g.ng + g.nck - 1 : g.ng; kh = h; }
  const long long c0 = fst_idx(g, i, j, k);
  const long long step = ih + g.sy * jh + g.sz * kh;  // one cell outward
  const int ng = g.ng;

  // The copies read only interior cells and write only ghosts, so a chunk of
  // variables is loaded before any of it is stored: the loads are then in
  // flight together (a store through U could alias the next load, which
  // would otherwise serialise them).  Same values as the reference's loop.
  constexpr int CH = 4;  // variables per chunk (with ng = 3: 12 values)
  double x[CH][3];
  for (int v0 = 0; v0 < g.nvt; v0 += CH) {
#pragma unroll
    for (int q = 0; q < CH; ++q)
#pragma unroll
      for (int n = 0; n < 3; ++n)
        if (v0 + q < g.nvt && n < ng) x[q][n] = U[c0 - step * n + g.sv * (v0 + q)];
#pragma unroll
    for (int q = 0; q < CH; ++q) {
      const int v = v0 + q;
      if (v >= g.nvt) break;
      // reflective, hydrostatic (reflect normal momentum) and noslip (all momenta)
      double reflect = 1.0;
      if (type == FST_BC_NOSLIP) {
        if (v == 0 || v == 1 || v == 2) reflect = -1.0;
      } else if (type != FST_BC_OUTFLOW) {
        if (ih != 0 && v == 0) reflect = -1.0;
        if (jh != 0 && v == 1) reflect = -1.0;
        if (kh != 0 && v == 2) reflect = -1.0;
      }
#pragma unroll
      for (int n = 0; n < 3; ++n)
        if (n < ng)
          U[c0 + step * (n + 1) + g.sv * v] =
              type == FST_BC_OUTFLOW ? x[q][n] : reflect * x[q][n];
    }
  }
  for (int n = 3; n < ng; ++n)  // more than 3 ghost layers: the plain loop
    for (int v = 0; v < g.nvt; ++v) {
      double reflect = 1.0;
      if (type == FST_BC_NOSLIP) {
        if (v == 0 || v == 1 || v == 2) reflect = -1.0;
      } else if (type != FST_BC_OUTFLOW) {
        if (ih != 0 && v == 0) reflect = -1.0;
        if (jh != 0 && v == 1) reflect = -1.0;
        if (kh != 0 && v == 2) reflect = -1.0;
      }
      U[c0 + step * (n + 1) + g.sv * v] = reflect * U[c0 - step * n + g.sv * v];
    }
  if (type == FST_BC_OUTFLOW) return;
  if (type != FST_BC_HYDROSTATIC) return;
  // linear extrapolation of internal energy (src/bc.cpp:92-123); density is
  // var(ndim+1), the first species
  const int edx = g.ndim, rdx = g.ndim + 1;
  for (int n = 0; n < ng; ++n) {
    long long cg = c0 + step * (n + 1), c1 = cg - step, c2 = cg - 2 * step;
    double ke = 0, ke1 = 0, ke2 = 0;
    for (int d = 0; d < g.ndim; ++d) {
      double ug = U[cg + g.sv * d], u1 = U[c1 + g.sv * d], u2 = U[c2 + g.sv * d];
      ke += 0.5 * (ug * ug);
      ke1 += 0.5 * (u1 * u1);
      ke2 += 0.5 * (u2 * u2);
    }
    ke = ke / U[cg + g.sv * rdx];
    ke1 = ke1 / U[c1 + g.sv * rdx];
    ke2 = ke2 / U[c2 + g.sv * rdx];
    U[cg + g.sv * edx] = 2 * (U[c1 + g.sv * edx] - ke1) - (U[c2 + g.sv * edx] - ke2) + ke;
  }
}

// ---------------------------------------------------------------------------
// Every ghost cell at once.  With at least ng cells on every axis the sequence of
// fills leaves in a ghost cell the value of one interior cell, found axis by axis
// (each fill runs over the full transverse extent, so a later one copies what an
// earlier one wrote), with the signs of the axes' reflections multiplied.  The
// energy beyond a hydrostatic face is the exception: an extrapolation along the
// face's normal.  On the axis filled last (the last non-periodic one) it reads, on
// its line, copies of interior cells only, so a ghost cell's energy still follows
// from up to three interior cells.  A hydrostatic face on an axis filled earlier
// takes the fills one after another.
// ---------------------------------------------------------------------------
struct GhostRule {
  int direct;       // 0: the fills have to run one after another
  int per[3];       // periodic axis
  int type[3][2];   // FST_BC_* of the low / high face
};

inline GhostRule ghost_rule(const Geo& g, const fst_config& cf) {
  GhostRule r{};
  const int n[3] = {g.nci, g.ncj, g.nck};
  const int per[3] = {cf.xper != 0, cf.yper != 0, cf.zper != 0};
  const int t[3][2] = {{cf.bc_xmin, cf.bc_xmax}, {cf.bc_ymin, cf.bc_ymax}, {cf.bc_zmin, cf.bc_zmax}};
  int last = -1;
  for (int a = 0; a < g.ndim; ++a)
    if (!per[a]) last = a;
  r.direct = g.ng == 3;
  for (int a = 0; a < g.ndim; ++a) {
    r.per[a] = per[a];
    for (int s = 0; s < 2; ++s) {
      r.type[a][s] = t[a][s];
      if (!per[a] && a != last && t[a][s] == FST_BC_HYDROSTATIC) r.direct = 0;
    }
    if (n[a] < g.ng) r.direct = 0;
  }
  return r;
}

// Where a ghost cell's values come from: the interior cell `src`, the variables
// 0..2 whose sign is flipped (bit v), and for a ghost cell beyond a hydrostatic
// face its layer (0 nearest, else -1) and the stride from a cell of its line to the
// next one inward.
struct GhostSource {
  long long src, inward;
  unsigned flip;
  int layer;
};
__device__ __forceinline__ GhostSource ghost_source(const Geo& g, const GhostRule& r, int i, int j,
                                                    int k) {
  GhostSource q{0, 0, 0u, -1};
  auto axis = [&](int a, int& x, int n, long long stride) {
    const int side = x < g.ng ? 0 : x >= g.ng + n ? 1 : -1;
    if (side < 0) return;
    if (r.per[a]) {
      x += side ? -n : n;
      return;
    }
    const int layer = side ? x - (g.ng + n) : g.ng - 1 - x;
    x = side ? g.ng + n - 1 - layer : g.ng + layer;
    const int t = side ? r.type[a][1] : r.type[a][0];  // (indexed, the rule is copied to local memory)
    q.flip ^= t == FST_BC_NOSLIP ? 7u : t == FST_BC_OUTFLOW ? 0u : 1u << a;
    if (t == FST_BC_HYDROSTATIC) {
      q.layer = layer;
      q.inward = side ? -stride : stride;
    }
  };
  axis(0, i, g.nci, 1);
  axis(1, j, g.ncj, g.sy);
  if (g.ndim == 3) axis(2, k, g.nck, g.sz);
  q.src = fst_idx(g, i, j, k);
  return q;
}
// x, its sign flipped when bit v of flip is set (what multiplying by -1 gives)
__device__ __forceinline__ double ghost_value(double x, unsigned flip, int v) {
  const unsigned long long b = fst64::bits_of(x);
  return fst64::of_bits(v < 3 && ((flip >> v) & 1) ? b ^ 0x8000000000000000ull : b);
}
// The energy of a ghost cell beyond a hydrostatic face (q.layer >= 0): the linear
// extrapolation of face_line above, layer after layer outward; the ghost layers'
// kinetic energies are those of the interior layers they mirror.
__device__ __forceinline__ double ghost_energy(const Geo& g, const double* U, const GhostSource& q) {
  const long long c0 = q.src - q.inward * q.layer;  // the line's first interior cell
  const int edx = g.ndim, rdx = g.ndim + 1;
  auto kinetic = [&](int n) {
    const long long c = c0 + q.inward * n;
    double ke = 0;
    for (int d = 0; d < g.ndim; ++d) {
      const double u = U[c + g.sv * d];
      ke += 0.5 * (u * u);
    }
    return ke / U[c + g.sv * rdx];
  };
  const double ke0 = kinetic(0), ke1 = kinetic(1);
  // (in 2D a no-slip face on the other axis has flipped the energy)
  const double E0 = ghost_value(U[c0 + g.sv * edx], q.flip, edx);
  const double E1 = ghost_value(U[c0 + q.inward + g.sv * edx], q.flip, edx);
  const double g0 = 2 * (E0 - ke0) - (E1 - ke1) + ke0;
  if (q.layer == 0) return g0;
  const double g1 = 2 * (g0 - ke0) - (E0 - ke0) + ke1;
  if (q.layer == 1) return g1;
  return 2 * (g1 - ke1) - (g0 - ke0) + kinetic(2);
}

}  // namespace fstbc

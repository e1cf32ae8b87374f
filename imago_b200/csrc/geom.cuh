// geom.cuh -- per-shell-pair geometry shared by the primitive kernels.
#pragma once

#include "intg.cuh"

namespace imago {

// True when a point at least d - pm from every lattice point of interest
// is certainly outside the screening radius^2 t: the float lower bound of
// d - pm (pmf >= pm, rounded down) squared, rounded down, exceeds tf >= t.
__device__ __forceinline__ bool beyond(float d, float pmf, float tf) {
  const float a = __fsub_rd(d, pmf);
  return a > 0.f && __fmul_rd(a, a) > tf;
}

// The images of one potential type that a unit's shell pairs are tested
// against: entry r in [beg, end) is image idx(r), at least d1(r) from the
// unit's midpoint, d1 ascending.
struct UnitWalk {
  int beg, end;
  const ImageRef *list;
  __device__ __forceinline__ ImageRef at(int r) const {
    return list ? list[r] : ImageRef{r, 0.f};
  }
};

__device__ __forceinline__ UnitWalk unit_walk(const DevSys &s, const DevWork &w, int unit,
                                              int pt) {
  if (w.ulist) {
    const int2 o = w.uoff[(long long)unit * s.npt + pt];
    return {o.x, o.y, w.ulist};
  }
  return {w.img_off[pt], w.img_off[pt + 1], nullptr};
}

// v = Ps - C for image position C; returns |v|^2.
__device__ __forceinline__ double image_d2(const double Ps[3], const double4 &C) {
  const double x = Ps[0] - C.x, y = Ps[1] - C.y, z = Ps[2] - C.z;
  return x * x + y * y + z * z;
}

// A bounded system's d2 = |Ps - C|^2 of an image: the least screening radius^2
// at which the reference's walk around Ps (integrals.F90:2632-2660, 2791-2819)
// comes to image C.  The site's image closest to Ps has to pass the screen
// too, and the lattice vector from there to C has to be in the cell list (else
// infinity).  The closest image (findLatticeVector, lattice.f90:784-888) is
// the one that rounding the fractional coordinates gives or one of its 26
// neighbours: with residual r, |r - d|^2 = |r|^2 + d.G d - 2 d.G r, G the
// lattice's Gram matrix, so a pair of neighbours +-d costs one comparison.
__device__ __forceinline__ double listed_d2(const DevSys &s, const double Ps[3], const double4 &C,
                                            double d2) {
  const double v[3] = {Ps[0] - C.x, Ps[1] - C.y, Ps[2] - C.z};
  double r[3], g[3];
  int n[3];
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    const double f = v[0] * s.inv[3 * i] + v[1] * s.inv[3 * i + 1] + v[2] * s.inv[3 * i + 2];
    n[i] = __double2int_rn(f);
    r[i] = f - n[i];
  }
#pragma unroll
  for (int i = 0; i < 3; ++i)
    g[i] = s.gram[3 * i] * r[0] + s.gram[3 * i + 1] * r[1] + s.gram[3 * i + 2] * r[2];
  const double r2 = r[0] * g[0] + r[1] * g[1] + r[2] * g[2];
  double best = -1e-12 * r2;
  int step = 0;  // code of the neighbour taken: 13 itself, less 13
#pragma unroll
  for (int m = 1; m <= 13; ++m) {
    const int d0 = (13 + m) / 9 - 1, d1 = (13 + m) / 3 % 3 - 1, d2_ = (13 + m) % 3 - 1;
    const double dg = d0 * g[0] + d1 * g[1] + d2_ * g[2];
    const double x = s.neighbour[m - 1] - 2.0 * fabs(dg);
    if (x < best) {
      best = x;
      step = dg > 0.0 ? m : -m;
    }
  }
  n[0] += (13 + step) / 9 - 1;
  n[1] += (13 + step) / 3 % 3 - 1;
  n[2] += (13 + step) % 3 - 1;
  // C lies at -n from the closest image
  if (abs(n[0]) > s.span[0] || abs(n[1]) > s.span[1] || abs(n[2]) > s.span[2]) return INFINITY;
  const long long at = ((long long)(s.span[0] - n[0]) * (2 * s.span[1] + 1) + s.span[1] - n[1]) *
                           (2 * s.span[2] + 1) + s.span[2] - n[2];
  if (!s.listed[at]) return INFINITY;
  const double c0 = r2 + (step ? best : 0.0);
  return c0 > d2 * (1.0 + 1e-9) ? c0 : d2;
}

struct SpGeom {
  double A[3], B[3];   // atom 1, shifted atom 2
  double a1, a2;       // primitive exponents
  double a1s, a2s;     // exponents of the element's first type (screening)
  double r2;
  int ti, tj;
};

__device__ __forceinline__ SpGeom sp_geom(const DevSys &s, const DevWork &w,
                                          const DSp &sp) {
  SpGeom g;
  const DUnit u = w.units[sp.unit];
  const DPair p = w.pairs[u.pair];
#pragma unroll
  for (int x = 0; x < 3; ++x) {
    g.A[x] = s.site_pos[3 * p.i + x];
    g.B[x] = s.site_pos[3 * p.j + x] + p.L0[x] + s.cell[3 * u.cell + x];
  }
  g.ti = p.ti;
  g.tj = p.tj;
  g.a1 = s.alpha[s.type_alpha_off[p.ti] + sp.a];
  g.a2 = s.alpha[s.type_alpha_off[p.tj] + sp.b];
  g.a1s = s.alpha[s.type_alpha_off[s.type_screen[p.ti]] + sp.a];
  g.a2s = s.alpha[s.type_alpha_off[s.type_screen[p.tj]] + sp.b];
  g.r2 = u.r2;
  return g;
}

// What the three-centre screens need of a shell pair (alphaDist and
// alphaCenter, gaussRelations.f90:112-131, from the element's first-type
// exponents, as the reference tables are built), and its product Gaussian.
struct SpScreen {
  double Ps[3], Pt[3];   // screening centre, centre of the product
  double zs, frac;       // a1s + a2s, 1 - r2 / alphaDist
  double zeta, xi;
  float pmf;             // at least |Ps - midpoint|
  // alphaPotDist / alphaNucDist (gaussRelations.f90:187-196, 262-270) for a
  // third screening exponent a3s: the radius^2 about Ps
  __device__ __forceinline__ double reach2(double T, double a3s) const {
    return frac * (T * (zs + a3s) / zs / a3s);
  }
};

__device__ __forceinline__ SpScreen sp_screen(const SpGeom &q, double T) {
  SpScreen r;
  const double cen = q.a1s / (q.a1s + q.a2s);
  const double adist = T / q.a2s / cen;
  r.frac = 1 - q.r2 / adist;
  r.zs = q.a1s + q.a2s;
  r.zeta = q.a1 + q.a2;
  r.xi = q.a1 * q.a2 / r.zeta;
  double pm = 0.0;
#pragma unroll
  for (int x = 0; x < 3; ++x) {
    r.Ps[x] = cen * (q.A[x] - q.B[x]) + q.B[x];
    r.Pt[x] = (q.a1 * q.A[x] + q.a2 * q.B[x]) / r.zeta;
    const double e = r.Ps[x] - 0.5 * (q.A[x] + q.B[x]);
    pm += e * e;
  }
  r.pmf = __double2float_ru(sqrt(pm));
  return r;
}

// The Hermite accumulators of the T adjacent lanes that share a shell pair,
// added by warp shuffles (every lane of the warp calls it).
template <int L, int T>
__device__ __forceinline__ void team_sum(double Q[nherm(L)]) {
#pragma unroll
  for (int off = T / 2; off > 0; off /= 2)
#pragma unroll
    for (int i = 0; i < nherm(L); ++i) Q[i] += __shfl_xor_sync(0xffffffffu, Q[i], off);
}

#define IMAGO_FOR_SPD_CLASSES(M) \
  M(0, 0) M(0, 1) M(0, 2) M(1, 0) M(1, 1) M(1, 2) M(2, 0) M(2, 1) M(2, 2)

}  // namespace imago

// k_ham.cu -- the summed potential terms of the PSCF Hamiltonian.
#include <algorithm>

#include "geom.cuh"
#include "prim.cuh"

namespace imago {

// The potential terms of the PSCF Hamiltonian (gaussOverlapHamPSCF,
// integrals.F90:3240-3442): H = sum_t coef[t] EP_t per spin, summed before
// the Hermite-to-spherical transform.  The terms of a type differ
// in a radial function only,
//   sum_j w_j exp(-mu_j |X|^2), w_j = coef_j (pi / z3_j)^1.5,
// over the terms that reach the image, so an image costs one exponential
// and L + 1 products per term, G_n = sum_j w_j (-2 mu_j)^n exp(-mu_j |X|^2),
// and one set of derivatives (accumulate_radial_q), where a term at a time
// costs a full Hermite product each.  Two spins share the walk and the
// exponentials (with the kinetic and nuclear blocks on a stream of their own:
// Si32, two spins, 3.90 -> 3.00 ms; Si8, one spin, 0.90 -> 0.85).  The team's
// mu_j, radii and weights stay in shared memory, kHamTerms terms at a time
// (32 KB at most).
template <int T>
constexpr int kHamTerms = T >= 4 ? 32 : 8;

template <int LA, int LB, int T, int SPIN, bool BND>
__global__ void __launch_bounds__(128, LA + LB >= 4 ? (SPIN == 2 ? 2 : 3) : (SPIN == 2 ? 3 : 4))
    k_prim3c_ham(DevSys s, DevWork w, int beg, int n, const Term3c *terms, int nterm,
                 const double *coef, double *H) {
  constexpr int L = LA + LB, TEAMS = 128 / T;
  __shared__ double sh[2 + SPIN][kHamTerms<T>][TEAMS];
  const long long g = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const int pair = (int)(g / T), sub = (int)(g % T), team = threadIdx.x / T;
  const bool live = pair < n;
  const DSp sp = w.sps[w.sp_by_cls[beg + (live ? pair : 0)]];
  const SpGeom q = sp_geom(s, w, sp);
  const SpScreen c = sp_screen(q, s.T);
  double Q[SPIN][nherm(L)];
#pragma unroll
  for (int h = 0; h < SPIN; ++h)
#pragma unroll
    for (int i = 0; i < nherm(L); ++i) Q[h][i] = 0.0;
  for (int t0 = 0; t0 < nterm;) {
    const int pt = terms[t0].ptype;
    int cnt = 1;
    while (cnt < kHamTerms<T> && t0 + cnt < nterm && terms[t0 + cnt].ptype == pt) ++cnt;
    const double *al = s.palpha + s.ptype_alpha_off[pt];
    const double *als = s.palpha + s.ptype_alpha_off[s.ptype_screen[pt]];
    const bool ascends = s.ptype_ascends[pt];
    double tmax = -1.0;
    __syncwarp();
    for (int j = sub; j < cnt; j += T) {
      const int ja = terms[t0 + j].j;
      const double a3 = al[ja], pz = kPi / (c.zeta + a3);
      const double t = live ? c.reach2(s.T, als[ja]) : -1.0;
      sh[0][j][team] = c.zeta * a3 / (c.zeta + a3);
      sh[1][j][team] = t;
#pragma unroll
      for (int h = 0; h < SPIN; ++h)
        sh[2 + h][j][team] = coef[h * nterm + t0 + j] * (pz * sqrt(pz));
      tmax = fmax(tmax, t);
    }
#pragma unroll
    for (int off = T / 2; off > 0; off /= 2)
      tmax = fmax(tmax, __shfl_xor_sync(0xffffffffu, tmax, off));
    __syncwarp();
    const float tf = __double2float_ru(tmax);
    const UnitWalk uw = unit_walk(s, w, sp.unit, pt);
    ImageRef en = uw.beg + sub < uw.end ? uw.at(uw.beg + sub) : ImageRef{0, 0.f};
    double4 Cn = w.ipos[en.idx];
    for (int r = uw.beg + sub; r < uw.end; r += T) {
      const ImageRef e = en;
      if (beyond(e.d1, c.pmf, tf)) break;
      const double4 C = Cn;
      if (r + T < uw.end) {  // one image ahead
        en = uw.at(r + T);
        Cn = w.ipos[en.idx];
      }
      double d2 = image_d2(c.Ps, C);
      if (d2 > tmax) continue;
      if constexpr (BND) {
        d2 = listed_d2(s, c.Ps, C, d2);
        if (d2 > tmax) continue;
      }
      const double X[3] = {c.Pt[0] - C.x, c.Pt[1] - C.y, c.Pt[2] - C.z};
      const double x2 = X[0] * X[0] + X[1] * X[1] + X[2] * X[2];
      double G[SPIN][L + 1];
#pragma unroll
      for (int h = 0; h < SPIN; ++h)
#pragma unroll
        for (int i = 0; i <= L; ++i) G[h][i] = 0.0;
      for (int j = 0; j < cnt; ++j) {
        if (d2 > sh[1][j][team]) {
          if (ascends) break;  // no later term reaches it
          continue;
        }
        const double mu = sh[0][j][team];
        const double g = exp(-mu * x2);
#pragma unroll
        for (int h = 0; h < SPIN; ++h) {
          double v = sh[2 + h][j][team] * g;
#pragma unroll
          for (int i = 0; i <= L; ++i) {
            G[h][i] += v;
            v *= -2.0 * mu;
          }
        }
      }
#pragma unroll
      for (int h = 0; h < SPIN; ++h) accumulate_radial_q<L>(X, G[h], Q[h]);
    }
    t0 += cnt;
  }
#pragma unroll
  for (int h = 0; h < SPIN; ++h) {
    team_sum<L, T>(Q[h]);
    if (live && sub == 0)
      hermite_to_sh<LA, LB, true>(q.A, q.B, q.a1, q.a2, exp(-c.xi * q.r2), Q[h],
                                  H + h * w.blk_total + sp.boff);
  }
}

template <int LA, int LB, int SPIN>
static int ham_one(const DevSys &s, const DevWork &w, int beg, int n, const Term3c *terms, int nterm,
                   const double *coef, int lanes, double *H,
                   cudaStream_t st) {
  if (n <= 0) return IMAGO_OK;
  if (s.bounded) lanes = 4;
  const unsigned grid = (unsigned)(((long long)n * lanes + 127) / 128);
  if (s.bounded)
    k_prim3c_ham<LA, LB, 4, SPIN, true><<<grid, 128, 0, st>>>(s, w, beg, n, terms, nterm, coef, H);
  else if (lanes == 8)
    k_prim3c_ham<LA, LB, 8, SPIN, false><<<grid, 128, 0, st>>>(s, w, beg, n, terms, nterm, coef, H);
  else if (lanes == 4)
    k_prim3c_ham<LA, LB, 4, SPIN, false><<<grid, 128, 0, st>>>(s, w, beg, n, terms, nterm, coef, H);
  else
    k_prim3c_ham<LA, LB, 1, SPIN, false><<<grid, 128, 0, st>>>(s, w, beg, n, terms, nterm, coef, H);
  IMAGO_LAUNCHED();
  return IMAGO_OK;
}

int launch_prim3c_ham(const DevSys &s, const DevWork &w, const int *cls_beg,
                      const Term3c *terms_dev, int nterm, const double *coef, int spin,
                      int lanes, double *H, cudaStream_t st) {
  if (nterm <= 0) return IMAGO_OK;
  if ((lanes != 1 && lanes != 4 && lanes != 8) || spin < 1 || spin > 2) return IMAGO_ERR_INVALID;
  int rc = IMAGO_OK;
#define IMAGO_PH(a, b)                                                                     \
  {                                                                                       \
    const int beg = cls_beg[a * 4 + b], n = cls_beg[a * 4 + b + 1] - beg;                 \
    if (!rc)                                                                              \
      rc = spin == 2                                                                      \
               ? ham_one<a, b, 2>(s, w, beg, n, terms_dev, nterm, coef, lanes, H, st) \
               : ham_one<a, b, 1>(s, w, beg, n, terms_dev, nterm, coef, lanes, H, st); \
  }
  IMAGO_FOR_SPD_CLASSES(IMAGO_PH)
#undef IMAGO_PH
  return rc ? rc : launch_prim3c_ham_rt(s, w, cls_beg, terms_dev, nterm, coef, spin, H, st);
}

}  // namespace imago

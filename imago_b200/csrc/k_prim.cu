// k_prim.cu -- primitive shell-pair blocks per class.
//
// Shell pairs are sorted by class; each s/p/d class runs a fully unrolled
// kernel, the f classes share runtime-class kernels.
#include <algorithm>

#include "geom.cuh"
#include "prim.cuh"

namespace imago {

// ------------------------------------------------------------ prim2c --
template <int LA, int LB, bool KIN>
__global__ void __launch_bounds__(128)
    k_prim2c(DevSys s, DevWork w, int beg, int end, double *blk) {
  const int g = beg + blockIdx.x * blockDim.x + threadIdx.x;
  if (g >= end) return;
  const DSp sp = w.sps[w.sp_by_cls[g]];
  const SpGeom q = sp_geom(s, w, sp);
  prim2c<LA, LB, KIN, true>(q.a1, q.a2, q.A, q.B, blk + sp.boff);
}

// Mass velocity (built once per SCF run, rel = 1): s/p/d classes unrolled,
// the f classes through one runtime-class kernel.
template <int LA, int LB>
__global__ void __launch_bounds__(128)
    k_prim_mv(DevSys s, DevWork w, int beg, int end, double *blk, bool add) {
  const int g = beg + blockIdx.x * blockDim.x + threadIdx.x;
  if (g >= end) return;
  const DSp sp = w.sps[w.sp_by_cls[g]];
  const SpGeom q = sp_geom(s, w, sp);
  prim_mv<LA, LB, true>(q.a1, q.a2, q.A, q.B, -kMassVelPref, blk + sp.boff,
                        add ? blk + sp.boff : nullptr);
}

__global__ void __launch_bounds__(128)
    k_prim_mv_rt(DevSys s, DevWork w, int beg, int end, int la, int lb,
                 double *blk, bool add) {
  const int g = beg + blockIdx.x * blockDim.x + threadIdx.x;
  if (g >= end) return;
  const DSp sp = w.sps[w.sp_by_cls[g]];
  const SpGeom q = sp_geom(s, w, sp);
  prim_mv_rt(la, lb, q.a1, q.a2, q.A, q.B, -kMassVelPref, blk + sp.boff,
             add ? blk + sp.boff : nullptr);
}

// Momentum / dipole: three component blocks per shell pair, component c at
// blk + c * blk_total.
template <int LA, int LB, bool DIP>
__global__ void __launch_bounds__(128)
    k_prim_vec(DevSys s, DevWork w, int beg, int end, double3 center, double *blk) {
  const int g = beg + blockIdx.x * blockDim.x + threadIdx.x;
  if (g >= end) return;
  const DSp sp = w.sps[w.sp_by_cls[g]];
  const SpGeom q = sp_geom(s, w, sp);
  const double C[3] = {center.x, center.y, center.z};
  prim_vec<LA, LB, DIP, true>(q.a1, q.a2, q.A, q.B, C, blk + sp.boff, w.blk_total);
}

template <bool DIP>
__global__ void __launch_bounds__(128)
    k_prim_vec_rt(DevSys s, DevWork w, int beg, int end, int la, int lb,
                  double3 center, double *blk) {
  const int g = beg + blockIdx.x * blockDim.x + threadIdx.x;
  if (g >= end) return;
  const DSp sp = w.sps[w.sp_by_cls[g]];
  const SpGeom q = sp_geom(s, w, sp);
  const double C[3] = {center.x, center.y, center.z};
  prim_vec_rt<DIP>(la, lb, q.a1, q.a2, q.A, q.B, C, blk + sp.boff, w.blk_total);
}

// ------------------------------------------------------------ prim3c --
// One thread per (shell pair, term).  The site and lattice-image loops are
// those of nuclearPE (integrals.F90:2533-2698) and electronicPE
// (2700-2858): the images of the type's sites within threeAlphaDist of the
// overlap centre, from the unit's image list.
// One item g < n * nterm of class (LA, LB): term g / n, shell pair g % n of
// the class's list.  Shared by the per-class launches and the work queue.
// CNT: the same walk, of EP terms or (NUC) of the nuclear term, counting
// the screened (site, image) triples into *ntrip instead of integrating
// (nothing is written).  BND: a bounded system (DevSys).
template <int LA, int LB, bool NUC, bool CNT = false, bool BND = false>
__device__ __forceinline__ void prim3c_item(const DevSys &s, const DevWork &w, int beg,
                                            int n, const Term3c *terms, double *blk,
                                            long long g, unsigned *ntrip = nullptr) {
  static_assert(CNT || !NUC, "the nuclear term is k_prim3c_nuc's");
  constexpr int L = LA + LB;
  const int tl = (int)(g / n);
  const DSp sp = w.sps[w.sp_by_cls[beg + (int)(g % n)]];
  const SpGeom q = sp_geom(s, w, sp);
  const SpScreen c = sp_screen(q, s.T);
  double Q[nherm(L)];
#pragma unroll
  for (int i = 0; i < nherm(L); ++i) Q[i] = 0.0;
  // NP runs over every potential type, EP over the term's type
  const Term3c tm = NUC ? Term3c{} : terms[tl];
  const double a3 = NUC ? 1.0 : s.palpha[s.ptype_alpha_off[tm.ptype] + tm.j];
  const double z3 = c.zeta + a3, mu = c.zeta * a3 / z3;
  for (int pt = NUC ? 0 : tm.ptype; pt < (NUC ? s.npt : tm.ptype + 1); ++pt) {
    if (NUC && s.ptype_z[pt] < kSmallThresh) continue;
    const int ps = s.ptype_screen[pt];
    const double t =
        c.reach2(s.T, NUC ? s.ptype_nucalpha[ps] : s.palpha[s.ptype_alpha_off[ps] + tm.j]);
    const float tf = __double2float_ru(t);
    const UnitWalk uw = unit_walk(s, w, sp.unit, pt);
    ImageRef en = uw.beg < uw.end ? uw.at(uw.beg) : ImageRef{0, 0.f};
    double4 Cn = w.ipos[en.idx];
    for (int r = uw.beg; r < uw.end; ++r) {
      const ImageRef e = en;
      if (beyond(e.d1, c.pmf, tf)) break;
      const double4 C = Cn;
      if (r + 1 < uw.end) {  // one image ahead
        en = uw.at(r + 1);
        Cn = w.ipos[en.idx];
      }
      const double d2 = image_d2(c.Ps, C);
      if (d2 > t) continue;
      if constexpr (BND) {
        if (listed_d2(s, c.Ps, C, d2) > t) continue;
      }
      if constexpr (CNT) {
        ++*ntrip;
      } else {
        const double X[3] = {c.Pt[0] - C.x, c.Pt[1] - C.y, c.Pt[2] - C.z};
        accumulate_overlap_q<L>(X, mu, 1.0, Q);
      }
    }
  }
  if constexpr (!CNT) {
    const double pz = kPi / z3;
    hermite_to_sh<LA, LB, true>(q.A, q.B, q.a1, q.a2, pz * sqrt(pz) * exp(-c.xi * q.r2), Q,
                                blk + (long long)tl * w.blk_total + sp.boff);
  }
}

// Screened primitive triples (shell pair, potential site, lattice image) of
// one class's items: what the reference's nuclearPE / electronicPE loops
// evaluate (integrals.F90:2533-2698, 2700-2858), summed into *count.
template <int LA, int LB, bool NUC>
__global__ void __launch_bounds__(128)
    k_prim3c_count(DevSys s, DevWork w, int beg, int n, const Term3c *terms, int nterm,
                   unsigned long long *count) {
  const long long g = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  unsigned c = 0;
  if (g < (long long)n * nterm) {
    if (s.bounded)
      prim3c_item<LA, LB, NUC, true, true>(s, w, beg, n, terms, nullptr, g, &c);
    else
      prim3c_item<LA, LB, NUC, true>(s, w, beg, n, terms, nullptr, g, &c);
  }
  c = __reduce_add_sync(0xffffffffu, c);
  if ((threadIdx.x & 31) == 0 && c) atomicAdd(count, (unsigned long long)c);
}

template <int LA, int LB, bool BND>
__global__ void __launch_bounds__(128, LA + LB >= 4 ? 3 : (LA + LB >= 3 ? 4 : (LA + LB == 2 ? 5 : 6)))
    k_prim3c(DevSys s, DevWork w, int beg, int n, const Term3c *terms,
             int nterm, double *blk) {
  const long long g = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (g >= (long long)n * nterm) return;
  prim3c_item<LA, LB, false, false, BND>(s, w, beg, n, terms, blk, g);
}

// f classes of k_prim3c_ham, runtime loops.
__global__ void __launch_bounds__(128)
    k_prim3c_ham_rt(DevSys s, DevWork w, int beg, int n, const Term3c *terms,
                    int nterm, const double *coef, int la, int lb, double *H) {
  const int L = la + lb;
  const int g = blockIdx.x * blockDim.x + threadIdx.x;
  if (g >= n) return;
  const DSp sp = w.sps[w.sp_by_cls[beg + g]];
  const SpGeom q = sp_geom(s, w, sp);
  const SpScreen c = sp_screen(q, s.T);
  double Q[kMaxHerm];
  for (int i = 0; i < kMaxHerm; ++i) Q[i] = 0.0;
  for (int tl = 0; tl < nterm; ++tl) {
    const Term3c tm = terms[tl];
    const int pt = tm.ptype;
    const double a3 = s.palpha[s.ptype_alpha_off[pt] + tm.j];
    const double t = c.reach2(s.T, s.palpha[s.ptype_alpha_off[s.ptype_screen[pt]] + tm.j]);
    const double z3 = c.zeta + a3, mu = c.zeta * a3 / z3;
    const double wt = coef[tl] * pow(kPi / z3, 1.5);
    const float tf = __double2float_ru(t);
    const UnitWalk uw = unit_walk(s, w, sp.unit, pt);
    for (int r = uw.beg; r < uw.end; ++r) {
      const ImageRef e = uw.at(r);
      if (beyond(e.d1, c.pmf, tf)) break;
      const double4 C = w.ipos[e.idx];
      const double d2 = image_d2(c.Ps, C);
      if (d2 > t || (s.bounded && listed_d2(s, c.Ps, C, d2) > t)) continue;
      const double X[3] = {c.Pt[0] - C.x, c.Pt[1] - C.y, c.Pt[2] - C.z};
      accumulate_overlap_q_rt(L, X, mu, wt, Q);
    }
  }
  hermite_to_sh_rt(la, lb, q.A, q.B, q.a1, q.a2, exp(-c.xi * q.r2), Q, H + sp.boff);
}

// f classes: one runtime-class kernel each for 2C and 3C.
template <bool KIN>
__global__ void __launch_bounds__(128)
    k_prim2c_rt(DevSys s, DevWork w, int beg, int end, int la, int lb,
                double *blk) {
  const int g = beg + blockIdx.x * blockDim.x + threadIdx.x;
  if (g >= end) return;
  const DSp sp = w.sps[w.sp_by_cls[g]];
  const SpGeom q = sp_geom(s, w, sp);
  prim2c_rt(la, lb, KIN, q.a1, q.a2, q.A, q.B, blk + sp.boff);
}

template <bool NUC>
__device__ __noinline__ void prim3c_item_rt(const DevSys &s, const DevWork &w, int beg,
                                            int n, const Term3c *terms, int la, int lb,
                                            double *blk, long long g, bool add) {
  const int L = la + lb;
  const int tl = (int)(g / n);
  const DSp sp = w.sps[w.sp_by_cls[beg + (int)(g % n)]];
  const SpGeom q = sp_geom(s, w, sp);
  const SpScreen c = sp_screen(q, s.T);
  double Q[kMaxHerm];
  for (int i = 0; i < kMaxHerm; ++i) Q[i] = 0.0;
  // NP runs over every potential type, EP over the term's type
  const Term3c tm = NUC ? Term3c{} : terms[tl];
  const double a3e = NUC ? 1.0 : s.palpha[s.ptype_alpha_off[tm.ptype] + tm.j];
  for (int pt = NUC ? 0 : tm.ptype; pt < (NUC ? s.npt : tm.ptype + 1); ++pt) {
    const double Z = NUC ? s.ptype_z[pt] : 0.0;
    if (NUC && Z < kSmallThresh) continue;
    const int ps = s.ptype_screen[pt];
    const double a3 = NUC ? s.ptype_nucalpha[pt] : a3e;
    const double t =
        c.reach2(s.T, NUC ? s.ptype_nucalpha[ps] : s.palpha[s.ptype_alpha_off[ps] + tm.j]);
    const double z3 = c.zeta + a3, mu = c.zeta * a3 / z3, nu = c.zeta * c.zeta / z3;
    const double w0 = -Z * (2.0 * kPi / z3);
    const float tf = __double2float_ru(t);
    const UnitWalk uw = unit_walk(s, w, sp.unit, pt);
    for (int r = uw.beg; r < uw.end; ++r) {
      const ImageRef e = uw.at(r);
      if (beyond(e.d1, c.pmf, tf)) break;
      const double4 C = w.ipos[e.idx];
      const double d2 = image_d2(c.Ps, C);
      if (d2 > t || (s.bounded && listed_d2(s, c.Ps, C, d2) > t)) continue;
      const double X[3] = {c.Pt[0] - C.x, c.Pt[1] - C.y, c.Pt[2] - C.z};
      if (NUC)
        accumulate_nuclear_q_rt(L, X, mu, nu, w0, Q);
      else
        accumulate_overlap_q_rt(L, X, mu, 1.0, Q);
    }
  }
  const double ex = exp(-c.xi * q.r2);
  const double pref = NUC ? ex : pow(kPi / (c.zeta + a3e), 1.5) * ex;
  double *out = blk + (long long)tl * w.blk_total + sp.boff;
  hermite_to_sh_rt(la, lb, q.A, q.B, q.a1, q.a2, pref, Q, out, add ? out : nullptr);
}

// Every f class in one launch, costliest first: cta[c] is the first CTA of
// the c-th class.  A cell's f classes are a few CTAs each and last as long as
// their longest thread, so in turn their times add up (two atoms with f
// functions, nuclear term: 6.3 ms one class after another, 3.7 together).
struct RtClasses {
  int ncls;
  int la[7], lb[7], beg[7], n[7], cta[8];
};

template <bool NUC>
__global__ void __launch_bounds__(128)
    k_prim3c_rt(DevSys s, DevWork w, RtClasses rc, const Term3c *terms, int nterm, double *blk,
                bool add) {
  int c = 0;
  while ((int)blockIdx.x >= rc.cta[c + 1]) ++c;
  const long long g = (long long)((int)blockIdx.x - rc.cta[c]) * blockDim.x + threadIdx.x;
  if (g >= (long long)rc.n[c] * nterm) return;
  prim3c_item_rt<NUC>(s, w, rc.beg[c], rc.n[c], terms, rc.la[c], rc.lb[c], blk, g, add);
}

// ------------------------------------------------------- work queue --
// Every class of a three-centre build in one persistent launch: the items
// of all classes are numbered one after another, the classes ordered by
// their per-item cost (highest angular momentum first) so that the cheap
// classes fill in behind the expensive ones, and each warp takes the next
// 32 items with one atomicAdd on a counter the host zeroes before the
// launch.  A warp's 32 items are consecutive items of one class (or of two
// at a class boundary), the same groups the per-class launches form, and
// every item writes only its own output block, so the results equal the
// per-class launches bit for bit.  No warp waits on another: a warp leaves
// as soon as the counter has passed the last item.
template <int LA, int LB>
__device__ __noinline__ void prim3c_item_q(const DevSys &s, const DevWork &w, int beg, int n,
                                           const Term3c *terms, double *blk, long long g) {
  prim3c_item<LA, LB, false>(s, w, beg, n, terms, blk, g);
}

__global__ void __launch_bounds__(128, 3)
    k_prim3c_queue(DevSys s, DevWork w, Prim3cQueue qc, const Term3c *terms, double *blk,
                   unsigned long long *counter) {
  const int lane = threadIdx.x & 31;
  const long long total = qc.off[qc.ncls];
  while (true) {
    unsigned long long base = 0;
    if (lane == 0) base = atomicAdd(counter, 32ULL);
    base = __shfl_sync(0xffffffffu, base, 0);
    if ((long long)base >= total) return;
    const long long item = (long long)base + lane;
    if (item >= total) continue;
    int c = 0;
    while (item >= qc.off[c + 1]) ++c;
    const long long g = item - qc.off[c];
    const int beg = qc.beg[c], n = qc.n[c];
    switch (qc.cls[c]) {
#define IMAGO_QC(a, b)                                                 \
  case a * 4 + b:                                                      \
    prim3c_item_q<a, b>(s, w, beg, n, terms, blk, g);             \
    break;
      IMAGO_QC(0, 0) IMAGO_QC(0, 1) IMAGO_QC(0, 2) IMAGO_QC(1, 0) IMAGO_QC(1, 1)
      IMAGO_QC(1, 2) IMAGO_QC(2, 0) IMAGO_QC(2, 1) IMAGO_QC(2, 2)
#undef IMAGO_QC
      default:
        prim3c_item_rt<false>(s, w, beg, n, terms, qc.cls[c] / 4, qc.cls[c] % 4, blk, g, false);
    }
  }
}

template <int LA, int LB>
static int prim2c_one(const DevSys &s, const DevWork &w, int beg, int end,
                      bool kin, double *blk, cudaStream_t st) {
  const int n = end - beg, tb = 128;
  if (n <= 0) return IMAGO_OK;
  if (kin)
    k_prim2c<LA, LB, true><<<(n + tb - 1) / tb, tb, 0, st>>>(s, w, beg, end, blk);
  else
    k_prim2c<LA, LB, false><<<(n + tb - 1) / tb, tb, 0, st>>>(s, w, beg, end, blk);
  IMAGO_LAUNCHED();
  return IMAGO_OK;
}

int launch_prim3c_count(const DevSys &s, const DevWork &w, const int *cls_beg,
                        const Term3c *terms_dev, int nterm, bool nuclear,
                        unsigned long long *count16, cudaStream_t st) {
#define IMAGO_PC(a, b)                                                               \
  {                                                                                 \
    const int beg = cls_beg[a * 4 + b], n = cls_beg[a * 4 + b + 1] - beg;           \
    if (n > 0 && nterm > 0) {                                                       \
      const unsigned grid = (unsigned)(((long long)n * nterm + 127) / 128);         \
      if (nuclear)                                                                  \
        k_prim3c_count<a, b, true><<<grid, 128, 0, st>>>(s, w, beg, n, terms_dev,   \
                                                         nterm, count16 + a * 4 + b); \
      else                                                                          \
        k_prim3c_count<a, b, false><<<grid, 128, 0, st>>>(s, w, beg, n, terms_dev,  \
                                                          nterm, count16 + a * 4 + b); \
      IMAGO_LAUNCHED();                                                             \
    }                                                                               \
  }
  IMAGO_FOR_SPD_CLASSES(IMAGO_PC)
#undef IMAGO_PC
  return IMAGO_OK;
}

int launch_prim2c(const DevSys &s, const DevWork &w, const int *cls_beg,
                  int op, double *blk, cudaStream_t st, bool add) {
  int rc = IMAGO_OK;
  if (add && op != kPrim2cMassVel) return IMAGO_ERR_INVALID;
  if (op == kPrim2cMassVel) {
#define IMAGO_MV(a, b)                                                        \
  {                                                                          \
    const int beg = cls_beg[a * 4 + b], n = cls_beg[a * 4 + b + 1] - beg;    \
    if (n > 0) {                                                             \
      k_prim_mv<a, b><<<(n + 127) / 128, 128, 0, st>>>(s, w, beg, beg + n, blk, add); \
      IMAGO_LAUNCHED();                                                      \
    }                                                                        \
  }
    IMAGO_FOR_SPD_CLASSES(IMAGO_MV)
#undef IMAGO_MV
    for (int c = 0; c < 16; ++c) {
      const int la = c / 4, lb = c % 4;
      if (la < 3 && lb < 3) continue;
      const int beg = cls_beg[c], n = cls_beg[c + 1] - beg;
      if (n <= 0) continue;
      k_prim_mv_rt<<<(n + 127) / 128, 128, 0, st>>>(s, w, beg, beg + n, la, lb, blk, add);
      IMAGO_LAUNCHED();
    }
    return IMAGO_OK;
  }
  const bool kinetic = op == kPrim2cKinetic;
#define IMAGO_P2(a, b)                                                       \
  if (rc == IMAGO_OK)                                                       \
    rc = prim2c_one<a, b>(s, w, cls_beg[a * 4 + b], cls_beg[a * 4 + b + 1], \
                          kinetic, blk, st);
  IMAGO_FOR_SPD_CLASSES(IMAGO_P2)
#undef IMAGO_P2
  for (int c = 0; c < 16 && rc == IMAGO_OK; ++c) {
    const int la = c / 4, lb = c % 4;
    if (la < 3 && lb < 3) continue;
    const int beg = cls_beg[c], end = cls_beg[c + 1], n = end - beg;
    if (n <= 0) continue;
    if (kinetic)
      k_prim2c_rt<true><<<(n + 127) / 128, 128, 0, st>>>(s, w, beg, end, la, lb, blk);
    else
      k_prim2c_rt<false><<<(n + 127) / 128, 128, 0, st>>>(s, w, beg, end, la, lb, blk);
    IMAGO_LAUNCHED();
  }
  return rc;
}

int launch_prim2c_vec(const DevSys &s, const DevWork &w, const int *cls_beg,
                      bool dipole, const double center[3], double *blk,
                      cudaStream_t st) {
  const double3 c3 = make_double3(center ? center[0] : 0.0, center ? center[1] : 0.0,
                                  center ? center[2] : 0.0);
#define IMAGO_PV(a, b)                                                         \
  {                                                                           \
    const int beg = cls_beg[a * 4 + b], n = cls_beg[a * 4 + b + 1] - beg;     \
    if (n > 0) {                                                              \
      const unsigned grid = (n + 127) / 128;                                  \
      if (dipole)                                                             \
        k_prim_vec<a, b, true><<<grid, 128, 0, st>>>(s, w, beg, beg + n, c3, blk);  \
      else                                                                    \
        k_prim_vec<a, b, false><<<grid, 128, 0, st>>>(s, w, beg, beg + n, c3, blk); \
      IMAGO_LAUNCHED();                                                       \
    }                                                                         \
  }
  IMAGO_FOR_SPD_CLASSES(IMAGO_PV)
#undef IMAGO_PV
  for (int c = 0; c < 16; ++c) {
    const int la = c / 4, lb = c % 4;
    if (la < 3 && lb < 3) continue;
    const int beg = cls_beg[c], n = cls_beg[c + 1] - beg;
    if (n <= 0) continue;
    const unsigned grid = (n + 127) / 128;
    if (dipole)
      k_prim_vec_rt<true><<<grid, 128, 0, st>>>(s, w, beg, beg + n, la, lb, c3, blk);
    else
      k_prim_vec_rt<false><<<grid, 128, 0, st>>>(s, w, beg, beg + n, la, lb, c3, blk);
    IMAGO_LAUNCHED();
  }
  return IMAGO_OK;
}

int launch_prim3c_ham_rt(const DevSys &s, const DevWork &w, const int *cls_beg,
                         const Term3c *terms_dev, int nterm, const double *coef, int spin,
                         double *H, cudaStream_t st) {
  for (int c = 0; c < 16; ++c) {
    const int la = c / 4, lb = c % 4;
    if (la < 3 && lb < 3) continue;
    const int beg = cls_beg[c], n = cls_beg[c + 1] - beg;
    if (n <= 0) continue;
    for (int h = 0; h < spin; ++h) {
      k_prim3c_ham_rt<<<(n + 127) / 128, 128, 0, st>>>(s, w, beg, n, terms_dev, nterm,
                                                       coef + (size_t)h * nterm, la, lb,
                                                       H + h * w.blk_total);
      IMAGO_LAUNCHED();
    }
  }
  return IMAGO_OK;
}

// K-overlap: for the three wave vectors, the real and imaginary blocks of
// each shell pair as terms 2 axis and 2 axis + 1.
__global__ void __launch_bounds__(128)
    k_prim_kov(DevSys s, DevWork w, int beg, int end, int la, int lb, KovWaves dk,
               double *blk) {
  const int g = beg + blockIdx.x * blockDim.x + threadIdx.x, ax = blockIdx.y;
  if (g >= end) return;
  const DSp sp = w.sps[w.sp_by_cls[g]];
  const SpGeom q = sp_geom(s, w, sp);
  prim_kov(la, lb, q.a1, q.a2, q.A, q.B, dk.q + 3 * ax,
           blk + (long long)(2 * ax) * w.blk_total + sp.boff,
           blk + (long long)(2 * ax + 1) * w.blk_total + sp.boff);
}

template <int LA, int LB>
__global__ void __launch_bounds__(128)
    k_prim_kov_t(DevSys s, DevWork w, int beg, int end, KovWaves dk, double *blk) {
  const int g = beg + blockIdx.x * blockDim.x + threadIdx.x, ax = blockIdx.y;
  if (g >= end) return;
  const DSp sp = w.sps[w.sp_by_cls[g]];
  const SpGeom q = sp_geom(s, w, sp);
  prim_kov_t<LA, LB>(q.a1, q.a2, q.A, q.B, dk.q + 3 * ax,
                     blk + (long long)(2 * ax) * w.blk_total + sp.boff,
                     blk + (long long)(2 * ax + 1) * w.blk_total + sp.boff);
}

// One thread per (shell pair, wave vector): s, p and d classes unrolled,
// f classes through the runtime routine.
int launch_prim_kov(const DevSys &s, const DevWork &w, const int *cls_beg,
                    const KovWaves &dk, double *blk, cudaStream_t st) {
  for (int c = 0; c < 16; ++c) {
    const int beg = cls_beg[c], n = cls_beg[c + 1] - beg;
    if (n <= 0) continue;
    const dim3 grid((n + 127) / 128, 3);
    switch (c) {
#define IMAGO_KOV(a, b)                                                                 \
  case a * 4 + b:                                                                       \
    k_prim_kov_t<a, b><<<grid, 128, 0, st>>>(s, w, beg, beg + n, dk, blk);              \
    break;
      IMAGO_FOR_SPD_CLASSES(IMAGO_KOV)
#undef IMAGO_KOV
      default:
        k_prim_kov<<<grid, 128, 0, st>>>(s, w, beg, beg + n, c / 4, c % 4, dk, blk);
    }
    IMAGO_LAUNCHED();
  }
  return IMAGO_OK;
}

int launch_prim3c_queue(const DevSys &s, const DevWork &w, const int *cls_beg,
                        const Term3c *terms_dev, int nterm, double *blk,
                        unsigned long long *counter, int ctas, cudaStream_t st) {
  if (nterm <= 0) return IMAGO_OK;
  if (s.bounded) return launch_prim3c(s, w, cls_beg, terms_dev, nterm, blk, st);
  Prim3cQueue qc{};
  // highest l_a + l_b first, then the larger l_a
  int order[16], m = 0;
  for (int L = 6; L >= 0; --L)
    for (int la = 3; la >= 0; --la) {
      const int lb = L - la;
      if (lb < 0 || lb > 3) continue;
      order[m++] = la * 4 + lb;
    }
  long long off = 0;
  for (int i = 0; i < m; ++i) {
    const int c = order[i];
    const int n = cls_beg[c + 1] - cls_beg[c];
    if (n <= 0) continue;
    qc.cls[qc.ncls] = c;
    qc.beg[qc.ncls] = cls_beg[c];
    qc.n[qc.ncls] = n;
    qc.off[qc.ncls] = off;
    off += (long long)n * nterm;
    ++qc.ncls;
  }
  qc.off[qc.ncls] = off;
  if (off == 0) return IMAGO_OK;
  IMAGO_CUDA(cudaMemsetAsync(counter, 0, sizeof(unsigned long long), st));
  const long long need = (off + 127) / 128;
  const unsigned grid = (unsigned)std::max<long long>(1, std::min<long long>(ctas, need));
  k_prim3c_queue<<<grid, 128, 0, st>>>(s, w, qc, terms_dev, blk, counter);
  IMAGO_LAUNCHED();
  return IMAGO_OK;
}

int prim3c_queue_ctas_per_sm() {
  int n = 0;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, k_prim3c_queue, 128, 0) !=
      cudaSuccess) {
    cudaGetLastError();
    return 1;
  }
  return std::max(1, n);
}

int launch_prim3c(const DevSys &s, const DevWork &w, const int *cls_beg,
                  const Term3c *terms_dev, int nterm, double *blk, cudaStream_t st) {
  if (nterm <= 0) return IMAGO_OK;
#define IMAGO_P3(a, b)                                                               \
  {                                                                                 \
    const int beg = cls_beg[a * 4 + b], n = cls_beg[a * 4 + b + 1] - beg;           \
    if (n > 0) {                                                                    \
      const unsigned grid = (unsigned)(((long long)n * nterm + 127) / 128);         \
      if (s.bounded)                                                                \
        k_prim3c<a, b, true><<<grid, 128, 0, st>>>(s, w, beg, n, terms_dev, nterm,  \
                                                   blk);                            \
      else                                                                          \
        k_prim3c<a, b, false><<<grid, 128, 0, st>>>(s, w, beg, n, terms_dev, nterm, \
                                                    blk);                           \
      IMAGO_LAUNCHED();                                                             \
    }                                                                               \
  }
  IMAGO_FOR_SPD_CLASSES(IMAGO_P3)
#undef IMAGO_P3
  return launch_prim3c_rt(s, w, cls_beg, terms_dev, nterm, false, blk, st);
}

int launch_prim3c_rt(const DevSys &s, const DevWork &w, const int *cls_beg,
                     const Term3c *terms_dev, int nterm, bool nuclear, double *blk,
                     cudaStream_t st, bool add) {
  if (nterm <= 0) return IMAGO_OK;
  RtClasses rc{};
  for (int c : {15, 11, 14, 7, 13, 3, 12}) {  // la * 4 + lb, la or lb = 3
    const int n = cls_beg[c + 1] - cls_beg[c];
    if (n <= 0) continue;
    const int i = rc.ncls++;
    rc.la[i] = c / 4;
    rc.lb[i] = c % 4;
    rc.beg[i] = cls_beg[c];
    rc.n[i] = n;
    rc.cta[i + 1] = rc.cta[i] + (int)(((long long)n * nterm + 127) / 128);
  }
  if (rc.ncls == 0) return IMAGO_OK;
  const unsigned grid = (unsigned)rc.cta[rc.ncls];
  if (nuclear)
    k_prim3c_rt<true><<<grid, 128, 0, st>>>(s, w, rc, terms_dev, nterm, blk, add);
  else
    k_prim3c_rt<false><<<grid, 128, 0, st>>>(s, w, rc, terms_dev, nterm, blk, false);
  IMAGO_LAUNCHED();
  return IMAGO_OK;
}

}  // namespace imago

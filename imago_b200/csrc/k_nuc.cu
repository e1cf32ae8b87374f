// k_nuc.cu -- the nuclear-attraction term of the three-centre primitive stage.
#include <algorithm>

#include "geom.cuh"
#include "prim.cuh"

namespace imago {

// T adjacent lanes share a shell pair: lane h takes entries h, h + T, ... of
// the unit's list, the Hermite accumulators are added by warp shuffles and
// the first lane transforms.  A shell pair of two diffuse primitives has
// hundreds of images, at some 300 FP64 operations each for the nuclear
// term: one lane per pair left the GPU waiting for the longest of them
// (0.7 of the 0.75 ms of the two-atom diamond cell's nuclear term).
template <int LA, int LB, int T, bool BND>
__global__ void __launch_bounds__(128, LA + LB >= 4 ? 3 : 4)
    k_prim3c_nuc(DevSys s, DevWork w, int beg, int n, double *blk, bool add) {
  constexpr int L = LA + LB;
  static_assert(32 % T == 0, "a shell pair's lanes stay in one warp");
  const long long g = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const int pair = (int)(g / T), sub = (int)(g % T);
  // lanes past the last pair stay for the shuffles
  const bool live = pair < n;
  const DSp sp = w.sps[w.sp_by_cls[beg + (live ? pair : 0)]];
  const SpGeom q = sp_geom(s, w, sp);
  const SpScreen c = sp_screen(q, s.T);
  double Q[nherm(L)];
#pragma unroll
  for (int i = 0; i < nherm(L); ++i) Q[i] = 0.0;
  for (int pt = 0; pt < s.npt; ++pt) {
    const double Z = s.ptype_z[pt];
    if (Z < kSmallThresh) continue;
    const double an = s.ptype_nucalpha[pt];
    const double t = live ? c.reach2(s.T, s.ptype_nucalpha[s.ptype_screen[pt]]) : -1.0;
    const double z3 = c.zeta + an;
    const double mu = c.zeta * an / z3, nu = c.zeta * c.zeta / z3, w0 = -Z * (2.0 * kPi / z3);
    const float tf = __double2float_ru(t);
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
      const double d2 = image_d2(c.Ps, C);
      if (d2 > t) continue;
      if constexpr (BND) {
        if (listed_d2(s, c.Ps, C, d2) > t) continue;
      }
      const double X[3] = {c.Pt[0] - C.x, c.Pt[1] - C.y, c.Pt[2] - C.z};
      accumulate_nuclear_q<L>(X, mu, nu, w0, Q);
    }
  }
  team_sum<L, T>(Q);
  if (live && sub == 0)
    hermite_to_sh<LA, LB, true>(q.A, q.B, q.a1, q.a2, exp(-c.xi * q.r2), Q, blk + sp.boff,
                                add ? blk + sp.boff : nullptr);
}

// Lanes per shell pair: enough threads to fill the GPU, no more, since each
// doubling adds a shuffle round and idles lanes in the transform.  One B200,
// ms at 1 / 2 / 4 / 8 / 16 lanes: two-atom diamond (40k shell pairs) 0.271 /
// 0.146 / 0.084 / 0.054 / 0.074, Si8 (62k) 0.299 / 0.200 / 0.168 / 0.220 /
// 0.333, Si16 (118k) 0.316 / 0.227 / 0.260 / 0.401 / 0.594, 162-atom quartz
// (1.36M) 1.15 / 1.23 / 1.63 / 2.39 / 3.88.  One lane with a nearest-image
// search per site took 0.73, 0.69, 0.75 and 2.42 ms.
constexpr long long kNucThreadsWanted = 320000;

template <int LA, int LB>
static int nuc_one(const DevSys &s, const DevWork &w, int beg, int n, int lanes, double *blk,
                   cudaStream_t st, bool add) {
  if (n <= 0) return IMAGO_OK;
  if (s.bounded) lanes = 4;
  const unsigned grid = (unsigned)(((long long)n * lanes + 127) / 128);
  switch (lanes) {
    case 8: k_prim3c_nuc<LA, LB, 8, false><<<grid, 128, 0, st>>>(s, w, beg, n, blk, add); break;
    case 4:
      if (s.bounded)
        k_prim3c_nuc<LA, LB, 4, true><<<grid, 128, 0, st>>>(s, w, beg, n, blk, add);
      else
        k_prim3c_nuc<LA, LB, 4, false><<<grid, 128, 0, st>>>(s, w, beg, n, blk, add);
      break;
    case 2: k_prim3c_nuc<LA, LB, 2, false><<<grid, 128, 0, st>>>(s, w, beg, n, blk, add); break;
    default: k_prim3c_nuc<LA, LB, 1, false><<<grid, 128, 0, st>>>(s, w, beg, n, blk, add);
  }
  IMAGO_LAUNCHED();
  return IMAGO_OK;
}

int launch_prim3c_nuc(const DevSys &s, const DevWork &w, const int *cls_beg, double *blk,
                      cudaStream_t st, bool add) {
  int lanes = 1, rc = IMAGO_OK;
  while (lanes < 8 && 2LL * lanes * w.nsp <= kNucThreadsWanted) lanes *= 2;
#define IMAGO_PN(a, b) \
  if (!rc) rc = nuc_one<a, b>(s, w, cls_beg[a * 4 + b], \
                              cls_beg[a * 4 + b + 1] - cls_beg[a * 4 + b], lanes, blk, st, add);
  IMAGO_FOR_SPD_CLASSES(IMAGO_PN)
#undef IMAGO_PN
  return rc ? rc : launch_prim3c_rt(s, w, cls_beg, nullptr, 1, true, blk, st, add);
}

}  // namespace imago

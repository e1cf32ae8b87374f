// k_terms.cu -- the three-centre primitive stage: the image lists of its
// screens and the electronic-potential terms of a shell pair walked
// together.
#include <algorithm>

#include "geom.cuh"
#include "prim.cuh"

namespace imago {

// ------------------------------------------------------- image lists --
// One warp per unit.  The unit's reach is the largest |Ps - M| + sqrt(t)
// over its shell pairs (t for the smallest third exponent), M the midpoint
// of its A-B segment; an image belongs to the unit's list when its float
// distance from M, less the margin that bounds the float error, is within
// that reach.  Images come in chunks of 32 neighbours, most of which their
// bounding spheres rule out (162-atom quartz: staging 17.5 ms with every
// image tested, 12.0 without lists).  Entries are placed in kListBins steps of
// the reach and carry the lower edge of their step: a walk may stop at the
// first entry whose edge is beyond its own reach.  The list
// replaces a nearest-image search per (shell pair, term, site) and the loop
// over lattice cells behind it (the walk alone was 15 of the 35 ms of the
// 162-atom quartz EP primitives).
constexpr int kListBins = 64;
constexpr int kListWarps = 8;

__device__ __forceinline__ float3 unit_mid(const DevSys &s, const DevWork &w, const DUnit &u) {
  const DPair p = w.pairs[u.pair];
  float m[3];
#pragma unroll
  for (int x = 0; x < 3; ++x)
    m[x] = (float)(0.5 * (s.site_pos[3 * p.i + x] + s.site_pos[3 * p.j + x] + p.L0[x] +
                          s.cell[3 * u.cell + x]));
  return make_float3(m[0], m[1], m[2]);
}

// Squared float distance, the same operations wherever it is formed: the
// count and the fill must agree on what belongs to a list.
__device__ __forceinline__ float list_d2(const float4 &c, const float3 &m) {
  const float x = __fsub_rn(c.x, m.x), y = __fsub_rn(c.y, m.y), z = __fsub_rn(c.z, m.z);
  return __fmaf_rn(z, z, __fmaf_rn(y, y, __fmul_rn(x, x)));
}

// f(first image) for every chunk of 32 images of type pt that may hold one
// within `lim` of m, by the chunks' bounding spheres; every lane of the warp
// calls it.
template <class F>
__device__ __forceinline__ void near_chunks(const DevWork &w, int pt, const float3 &m, float lim,
                                            int lane, F f) {
  const int c0 = w.chunk_off[pt], c1 = w.chunk_off[pt + 1];
  for (int cb = c0; cb < c1; cb += 32) {
    bool near = false;
    if (cb + lane < c1) {
      const float4 s = w.chunk[cb + lane];
      const float r = lim + s.w;
      near = list_d2(s, m) <= r * r;
    }
    for (unsigned mask = __ballot_sync(0xffffffffu, near); mask; mask &= mask - 1)
      f(w.img_off[pt] + 32 * (cb + __ffs(mask) - 1 - c0));
  }
}

__global__ void __launch_bounds__(32 * kListWarps)
    k_list_count(DevSys s, DevWork w, float margin, int2 *uoff, float *rad,
                 unsigned long long *cursor) {
  const int lane = threadIdx.x & 31;
  const int nw = gridDim.x * kListWarps;
  for (int ui = blockIdx.x * kListWarps + (threadIdx.x >> 5); ui < w.nunits; ui += nw) {
    const DUnit u = w.units[ui];
    const DPair p = w.pairs[u.pair];
    const double *as1 = s.alpha + s.type_alpha_off[s.type_screen[p.ti]];
    const double *as2 = s.alpha + s.type_alpha_off[s.type_screen[p.tj]];
    const double r = sqrt(u.r2);
    double reach = 0.0;
    for (int q = u.spbeg + lane; q < u.spend; q += 32) {
      const DSp sp = w.sps[q];
      const double a = as1[sp.a], b = as2[sp.b], z = a + b;
      const double frac = fmax(0.0, 1.0 - u.r2 * (a * b / z) / s.T);
      const double t = frac * s.T * (z + s.a3_min) / (z * s.a3_min);
      reach = fmax(reach, fabs(a / z - 0.5) * r + fmin(sqrt(t), s.reach_cap));
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) reach = fmax(reach, __shfl_xor_sync(0xffffffffu, reach, o));
    // rounding of the formulas above against the screens' own
    const float R = __double2float_ru(reach * (1.0 + 1e-9) + 1e-6);
    const float3 m = unit_mid(s, w, u);
    const float lim = R + margin, lim2 = lim * lim;
    int2 *out = uoff + (long long)ui * s.npt;
    int run = 0;
    for (int pt = 0; pt < s.npt; ++pt) {
      int n = 0;
      const int i1 = w.img_off[pt + 1];
      near_chunks(w, pt, m, lim, lane, [&](int ib) {
        const int i = ib + lane;
        n += __popc(__ballot_sync(0xffffffffu, i < i1 && list_d2(w.ftab[i], m) <= lim2));
      });
      if (lane == 0) out[pt] = make_int2(run, run + n);
      run += n;
    }
    // the units' ranges in the order they come by; their contents do not
    // depend on it
    unsigned long long base = 0;
    if (lane == 0) base = atomicAdd(cursor, (unsigned long long)run);
    base = __shfl_sync(0xffffffffu, base, 0);
    __syncwarp();
    for (int pt = lane; pt < s.npt; pt += 32) {
      const int2 o = out[pt];
      out[pt] = make_int2((int)(base + o.x), (int)(base + o.y));
    }
    if (lane == 0) rad[ui] = R;
  }
}

// Lane-private counters per step (row b, column lane, a column over for the
// step's first entry): counting and placing need neither atomics nor a match
// across the warp, whose latency bound the form with both (64-atom graphite
// 0.93 ms, short scoreboard; staging 6.43 -> 6.10 ms, 162-atom quartz 14.6 ->
// 13.8), and the order of a list is always the same: by step, lane, chunk.
// Lists of up to a warp's lanes, as where every site has its own type, are
// ranked by that order directly: clearing and adding up 64 x 32 counters for
// each took much of the staging (216 diamond atoms with their own types: 59.9 ->
// 42.2 ms, 162 quartz atoms 23.0 -> 18.0).
constexpr int kFillWarps = 4, kFillRow = 33;

__global__ void __launch_bounds__(32 * kFillWarps)
    k_list_fill(DevSys s, DevWork w, float margin, const float *rad, ImageRef *list) {
  __shared__ int bins[kFillWarps][kListBins * kFillRow];
  static_assert(kListBins == 64, "two steps per lane");
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int nw = gridDim.x * kFillWarps;
  int *bin = bins[warp];
  for (int ui = blockIdx.x * kFillWarps + warp; ui < w.nunits; ui += nw) {
    const DUnit u = w.units[ui];
    const float3 m = unit_mid(s, w, u);
    const float R = rad[ui], step = R / kListBins, inv = kListBins / R;
    const float lim = R + margin, lim2 = lim * lim;
    for (int pt = 0; pt < s.npt; ++pt) {
      const int2 range = w.uoff[(long long)ui * s.npt + pt];
      if (range.x == range.y) continue;
      const int i1 = w.img_off[pt + 1];
      // the step of an image, its distance less the margin; -1 outside
      auto place = [&](int i) {
        const float d2 = i < i1 ? list_d2(w.ftab[i], m) : 0.f;
        return i < i1 && d2 <= lim2
                   ? min(kListBins - 1, (int)(fmaxf(0.f, sqrtf(d2) - margin) * inv))
                   : -1;
      };
      ImageRef *out = list + range.x;
      // the step's lower edge, rounded to stay below the distance
      auto ref = [&](int i, int b) { return ImageRef{i, b * step * (1.f - 1e-5f)}; };
      const int len = range.y - range.x;
      if (len <= 32) {
        int n = 0;  // bin: the images found, their places in the list's order
        near_chunks(w, pt, m, lim, lane, [&](int ib) {
          const int b = place(ib + lane);
          const unsigned mask = __ballot_sync(0xffffffffu, b >= 0);
          if (b >= 0) {
            const int at = n + __popc(mask & ((1u << lane) - 1u));
            bin[at] = ib + lane;
            bin[32 + at] = (b << 10) + (lane << 5) + at;
          }
          n += __popc(mask);
        });
        __syncwarp();
        const int key = lane < len ? bin[32 + lane] : 0;
        int rank = 0;
        for (int l = 0; l < len; ++l) rank += __shfl_sync(0xffffffffu, key, l) < key;
        if (lane < len) out[rank] = ref(bin[lane], key >> 10);
        __syncwarp();
        continue;
      }
      for (int i = lane; i < kListBins * kFillRow; i += 32) bin[i] = 0;
      __syncwarp();
      near_chunks(w, pt, m, lim, lane, [&](int ib) {
        const int b = place(ib + lane);
        if (b >= 0) ++bin[b * kFillRow + lane];
      });
      __syncwarp();
      // exclusive prefix over the lanes of steps `lane` and `lane + 32`, then
      // over the steps
      int sum[2] = {0, 0};
#pragma unroll
      for (int q = 0; q < 2; ++q) {
        int *row = bin + (lane + 32 * q) * kFillRow;
#pragma unroll 8
        for (int l = 0; l < 32; ++l) {
          const int n = row[l];
          row[l] = sum[q];
          sum[q] += n;
        }
      }
      int end[2] = {sum[0], sum[1]};
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int x0 = __shfl_up_sync(0xffffffffu, end[0], o);
        const int x1 = __shfl_up_sync(0xffffffffu, end[1], o);
        if (lane >= o) {
          end[0] += x0;
          end[1] += x1;
        }
      }
      const int half = __shfl_sync(0xffffffffu, end[0], 31);
      bin[lane * kFillRow + 32] = end[0] - sum[0];
      bin[(lane + 32) * kFillRow + 32] = half + end[1] - sum[1];
      __syncwarp();
      near_chunks(w, pt, m, lim, lane, [&](int ib) {
        const int b = place(ib + lane);
        if (b >= 0) out[bin[b * kFillRow + 32] + bin[b * kFillRow + lane]++] = ref(ib + lane, b);
      });
      __syncwarp();
    }
  }
}

int launch_list_count(const DevSys &s, const DevWork &w, float margin, int2 *uoff, float *rad,
                      unsigned long long *cursor, cudaStream_t st) {
  IMAGO_CUDA(cudaMemsetAsync(cursor, 0, sizeof(unsigned long long), st));
  if (w.nunits == 0) return IMAGO_OK;
  const int grid = std::min((w.nunits + kListWarps - 1) / kListWarps, 148 * 8);
  k_list_count<<<grid, 32 * kListWarps, 0, st>>>(s, w, margin, uoff, rad, cursor);
  IMAGO_LAUNCHED();
  return IMAGO_OK;
}

int launch_list_fill(const DevSys &s, const DevWork &w, float margin, const float *rad,
                     ImageRef *list, cudaStream_t st) {
  if (w.nunits == 0) return IMAGO_OK;
  const int grid = std::min((w.nunits + kFillWarps - 1) / kFillWarps, 148 * 12);
  k_list_fill<<<grid, 32 * kFillWarps, 0, st>>>(s, w, margin, rad, list);
  IMAGO_LAUNCHED();
  return IMAGO_OK;
}

// ---------------------------------------------------------- EP terms --
// One thread per (shell pair, group of terms of one potential type).  The
// geometry, the screening quantities and the product Gaussian are formed
// once for the group.  The first terms, the most diffuse, walk the unit's
// image list; while doing so a thread notes the images that the next term
// still reaches, and as soon as every lane of the warp could note all of
// its own (kTermCap), the following terms run over the notes, each term
// striking out what it no longer reaches.  Either loop loads one image ahead,
// since a reference and then a position are waited for (162-atom quartz EP
// 8.80 -> 8.35 ms, 64-atom graphite 2.70 -> 2.41).  Every lane then works on an
// image of its own at each step, where a walk has the warp wait at images
// that only some lanes reach.  The triples of a term are exactly those of
// its own walk.
constexpr int kTermThreads = 128;
constexpr int kTermCap = 64;

template <int LA, int LB>
__device__ __forceinline__ void terms_item(const DevSys &s, const DevWork &w, int beg, int n,
                                           const Term3c *terms, const TermGroups &tg, double *blk,
                                           long long g, int (*note)[kTermThreads]) {
  constexpr int L = LA + LB;
  const int tid = threadIdx.x;
  const bool live = g < (long long)n * tg.n;
  const int gi = live ? (int)(g / n) : 0;
  const int t0 = tg.first[gi], cnt = live ? tg.count[gi] : 0;
  const DSp sp = w.sps[w.sp_by_cls[beg + (live ? (int)(g % n) : 0)]];
  const SpGeom q = sp_geom(s, w, sp);
  const SpScreen c = sp_screen(q, s.T);
  const int pt = terms[t0].ptype;
  const double *al = s.palpha + s.ptype_alpha_off[pt];
  const double *als = s.palpha + s.ptype_alpha_off[s.ptype_screen[pt]];
  const bool ascends = s.ptype_ascends[pt];
  const UnitWalk uw = unit_walk(s, w, sp.unit, pt);
  const double ex = exp(-c.xi * q.r2), inv2p = 1.0 / (2.0 * c.zeta);
  double PA[3], PB[3];
#pragma unroll
  for (int x = 0; x < 3; ++x) {
    PA[x] = c.Pt[x] - q.A[x];
    PB[x] = c.Pt[x] - q.B[x];
  }
  bool have = false;  // the notes hold every image of this and later terms
  int nn = 0;
  double t = cnt > 0 ? c.reach2(s.T, als[terms[t0].j]) : -1.0;
  for (int it = 0; __any_sync(0xffffffffu, it < cnt); ++it) {
    const bool on = it < cnt;
    const double a3 = on ? al[terms[t0 + it * tg.stride].j] : 1.0;
    const double tn = it + 1 < cnt ? c.reach2(s.T, als[terms[t0 + (it + 1) * tg.stride].j]) : -1.0;
    const double z3 = c.zeta + a3, mu = c.zeta * a3 / z3;
    double Q[nherm(L)];
#pragma unroll
    for (int i = 0; i < nherm(L); ++i) Q[i] = 0.0;
    if (__all_sync(0xffffffffu, have || !on)) {
      int keep = 0;
      int idn = nn > 0 ? note[0][tid] : 0;
      double4 Cn = w.ipos[idn];
      for (int i = 0; i < nn; ++i) {
        const int id = idn;
        const double4 C = Cn;
        if (i + 1 < nn) {
          idn = note[i + 1][tid];
          Cn = w.ipos[idn];
        }
        if (image_d2(c.Ps, C) > t) continue;
        note[keep++][tid] = id;
        const double X[3] = {c.Pt[0] - C.x, c.Pt[1] - C.y, c.Pt[2] - C.z};
        accumulate_overlap_q<L>(X, mu, 1.0, Q);
      }
      nn = keep;
    } else if (on) {
      const float tf = __double2float_ru(t);
      nn = 0;
      ImageRef en = uw.beg < uw.end ? uw.at(uw.beg) : ImageRef{0, 0.f};
      double4 Cn = w.ipos[en.idx];
      for (int r = uw.beg; r < uw.end; ++r) {
        const ImageRef e = en;
        if (beyond(e.d1, c.pmf, tf)) break;
        const double4 C = Cn;
        if (r + 1 < uw.end) {
          en = uw.at(r + 1);
          Cn = w.ipos[en.idx];
        }
        const double d2 = image_d2(c.Ps, C);
        if (d2 > t) continue;
        if (d2 <= tn) {
          if (nn < kTermCap) note[nn][tid] = e.idx;
          ++nn;
        }
        const double X[3] = {c.Pt[0] - C.x, c.Pt[1] - C.y, c.Pt[2] - C.z};
        accumulate_overlap_q<L>(X, mu, 1.0, Q);
      }
      have = ascends && nn <= kTermCap;
    }
    if (on) {
      const double pz = kPi / z3;
      hermite_to_sh<LA, LB, true>(
          PA, PB, inv2p, pz * sqrt(pz) * ex, Q,
          blk + (long long)(t0 + it * tg.stride) * w.blk_total + sp.boff);
    }
    t = tn;
  }
}

template <int LA, int LB>
__global__ void __launch_bounds__(kTermThreads, LA + LB >= 4 ? 3 : (LA + LB >= 3 ? 4 : 5))
    k_prim3c_terms(DevSys s, DevWork w, int beg, int n, const Term3c *terms, TermGroups tg,
                   double *blk) {
  __shared__ int note[kTermCap][kTermThreads];
  terms_item<LA, LB>(s, w, beg, n, terms, tg, blk,
                     (long long)blockIdx.x * kTermThreads + threadIdx.x, note);
}

// Every class in one launch, costliest first: cta[c] is the first CTA of the
// c-th class.  A small system's classes are a few CTAs each (Si8: 16 for
// p-p) and last as long as their longest thread; in turn they leave the GPU
// nearly empty, together they fill in behind the largest.
struct ClassCtas {
  int ncls;
  int cls[9], beg[9], n[9], cta[10];
};

__global__ void __launch_bounds__(kTermThreads, 3)
    k_prim3c_terms_all(DevSys s, DevWork w, ClassCtas cc, const Term3c *terms, TermGroups tg,
                       double *blk) {
  __shared__ int note[kTermCap][kTermThreads];
  int c = 0;
  while ((int)blockIdx.x >= cc.cta[c + 1]) ++c;
  const long long g = (long long)((int)blockIdx.x - cc.cta[c]) * kTermThreads + threadIdx.x;
  switch (cc.cls[c]) {
#define IMAGO_TA(a, b)                                                              \
  case a * 4 + b:                                                                   \
    terms_item<a, b>(s, w, cc.beg[c], cc.n[c], terms, tg, blk, g, note);            \
    break;
    IMAGO_FOR_SPD_CLASSES(IMAGO_TA)
#undef IMAGO_TA
  }
}

// Term groups of one launch: the terms from `from` on, split into runs of
// one potential type and each run into `split` interleaved groups, at most
// kMaxTermGroups of them.  Returns the first term not covered.
static int group_terms(const Term3c *terms, int nterm, int from, int split, TermGroups &tg) {
  tg.n = 0;
  tg.stride = split;
  int i = from;
  while (i < nterm) {
    int e = i + 1;
    while (e < nterm && terms[e].ptype == terms[i].ptype && e - i < 65535) ++e;
    const int k = std::min(split, e - i);
    if (tg.n + k > kMaxTermGroups) break;
    for (int h = 0; h < k; ++h) {
      tg.first[tg.n] = (unsigned short)(i - from + h);
      tg.count[tg.n] = (unsigned short)((e - i - h + split - 1) / split);
      ++tg.n;
    }
    i = e;
  }
  return i;
}

// Several classes and at most kTermsMergedPairs (shell pair, run of terms of
// one type): all classes in one launch.  Else a launch per class, with the
// class's own occupancy: one class gains nothing, and a large system's
// classes fill the GPU each.  Terms are split into interleaved groups until
// a launch has about the threads wanted.  One B200, EP primitives in ms, per
// class / merged, each at its best split: Si8 (62k pairs) 0.89 / 0.55, Si16
// (118k) 1.26 / 0.95, Si32 (230k) 2.03 / 1.67, 18-atom quartz (158k x 2)
// 1.58 / 1.26, 36-atom quartz (307k x 2) 2.64 / 2.32, 162-atom quartz (1.36M
// x 2) 8.79 / 8.92; one class: 16-atom diamond (226k) 2.02 / 2.29, 64-atom
// graphite (534k) 2.69 / 3.34.  Split, Si8 merged: 1.28, 0.77, 0.55, 0.57,
// 0.59, 0.69 with 1, 2, 4, 7, 10, 20 groups.
constexpr long long kTermsMergedPairs = 1000000;
constexpr long long kTermThreadsMerged = 400000, kTermThreadsWanted = 800000;

int launch_prim3c_terms(const DevSys &s, const DevWork &w, const int *cls_beg,
                        const Term3c *terms_dev, const Term3c *terms_host, int nterm,
                        double *blk, cudaStream_t st) {
  if (s.bounded) return launch_prim3c(s, w, cls_beg, terms_dev, nterm, blk, st);
  int runs = 0;
  for (int i = 0; i < nterm; ++i) runs += i == 0 || terms_host[i].ptype != terms_host[i - 1].ptype;
  const long long base = std::max(1LL, (long long)w.nsp * std::max(1, runs));
  int classes = 0;
  for (int c : {0, 1, 2, 4, 5, 6, 8, 9, 10}) classes += cls_beg[c + 1] > cls_beg[c];
  const bool merged = classes > 1 && base <= kTermsMergedPairs;
  const long long wanted = merged ? kTermThreadsMerged : kTermThreadsWanted;
  const int split = (int)std::min<long long>(32, (wanted + base - 1) / base);
  for (int from = 0; from < nterm;) {
    TermGroups tg;
    const int next = group_terms(terms_host + from, nterm - from, 0, split, tg) + from;
    double *b = blk + (long long)from * w.blk_total;
    if (merged) {
      static const int order[9] = {10, 6, 9, 5, 2, 8, 1, 4, 0};  // la * 4 + lb
      ClassCtas cc{};
      for (int c : order) {
        const int n = cls_beg[c + 1] - cls_beg[c];
        if (n <= 0) continue;
        cc.cls[cc.ncls] = c;
        cc.beg[cc.ncls] = cls_beg[c];
        cc.n[cc.ncls] = n;
        cc.cta[cc.ncls + 1] =
            cc.cta[cc.ncls] + (int)(((long long)n * tg.n + kTermThreads - 1) / kTermThreads);
        ++cc.ncls;
      }
      if (cc.ncls) {
        k_prim3c_terms_all<<<cc.cta[cc.ncls], kTermThreads, 0, st>>>(s, w, cc, terms_dev + from,
                                                                    tg, b);
        IMAGO_LAUNCHED();
      }
      from = next;
      continue;
    }
#define IMAGO_PT(a, c)                                                                     \
  {                                                                                       \
    const int beg = cls_beg[a * 4 + c], n = cls_beg[a * 4 + c + 1] - beg;                 \
    if (n > 0) {                                                                          \
      const unsigned grid = (unsigned)(((long long)n * tg.n + kTermThreads - 1) / kTermThreads); \
      k_prim3c_terms<a, c><<<grid, kTermThreads, 0, st>>>(s, w, beg, n, terms_dev + from, tg, b); \
      IMAGO_LAUNCHED();                                                                   \
    }                                                                                     \
  }
    IMAGO_PT(2, 2) IMAGO_PT(1, 2) IMAGO_PT(2, 1) IMAGO_PT(1, 1) IMAGO_PT(0, 2) IMAGO_PT(2, 0)
    IMAGO_PT(0, 1) IMAGO_PT(1, 0) IMAGO_PT(0, 0)
#undef IMAGO_PT
    from = next;
  }
  return launch_prim3c_rt(s, w, cls_beg, terms_dev, nterm, false, blk, st);
}

}  // namespace imago

// k_contract.cu -- contraction of a unit's primitive blocks with the radial
// coefficients of its two atoms.
#include <algorithm>

#include "intg.cuh"

namespace imago {

// M_t(m1, m2) = sum_{(a,b) in unit} C1(a, m1) C2(b, m2) sh_t,ab(lm1, lm2),
// the pairXBasisFn2 / multWithBasisFn1 contraction (integrals.F90:555-563,
// intgSaving.F90:56-89).  Entries whose lm lies beyond a primitive's class
// carry a zero coefficient in the reference and are skipped.  Blocks are
// stored column-major, e = m2 * ni + m1.
//
// One CTA per unit (or per part of its terms), threads over the block
// elements.  What a unit needs besides its blocks (the shell-pair list, both
// coefficient tables, the chunk bounds) is staged once; its terms then go by
// in groups of T, a unit's blocks of one term being contiguous, in chunks of
// whole shell pairs copied asynchronously one chunk ahead: the coefficient
// product of an (element, shell pair) serves the T terms of a group, and the
// next group's first chunk arrives during this one's last.  With a CTA per
// (unit, group) every group paid for the staging and waited for its own first
// chunk, 15 us a CTA.  T = 4 or 8, picked by measurement; 1 for builds of one
// matrix.  One B200, before / now: Si8 one matrix 0.18 / 0.09 ms, EP 0.53 /
// 0.38, 162-atom quartz 1.02 / 0.72 and 8.78 / 6.76, Si16 momentum 0.29 / 0.21.
constexpr int kContractThreads = 128;
constexpr int kElemsPerThread = 3;  // n_i n_j <= 384 per pass
constexpr int kSpList = 512;        // shell pairs listed at a time
constexpr int kCoefMax = 512;       // alphas x states per atom kept in shared memory
constexpr long long kContractCtas = 20000;  // below, a unit's groups are shared out

// Staged doubles per term: two of the largest blocks at least, so that the
// chunks' windows (the buffer less one block) hold whole shell pairs.
template <int T>
__host__ __device__ constexpr int contract_buf(int blk_max) {
  return blk_max > 84 ? 512 : T == 8 ? 384 : 512;
}

template <int T>
static size_t contract_smem(int blk_max) {
  return sizeof(double) * (2 * T * contract_buf<T>(blk_max) + 2 * kCoefMax) +
         sizeof(int) * (3 * kSpList + kSpList + 2);
}

template <int T>
__global__ void __launch_bounds__(kContractThreads, T == 8 ? 3 : 4)
    k_contract(DevSys s, DevWork w, int nterm, int gsplit, const double *blk, double *M) {
  extern __shared__ __align__(16) double csm[];
  const int buf = contract_buf<T>(w.blk_max), window = buf - w.blk_max;
  double *bs = csm, *c1s = bs + 2 * T * buf, *c2s = c1s + kCoefMax;
  int *sp_ab = reinterpret_cast<int *>(c2s + kCoefMax);  // a | b << 16
  int *sp_cls = sp_ab + kSpList;                          // nsh(la) | nsh(lb) << 8
  int *sp_rel = sp_cls + kSpList;                         // block offset from the list's first
  int *cb = sp_rel + kSpList;                             // first shell pair of each chunk
  const int ui = blockIdx.x / gsplit, part = blockIdx.x % gsplit;
  const int ntg = (nterm + T - 1) / T;
  const int g0 = (int)((long long)ntg * part / gsplit), g1 = (int)((long long)ntg * (part + 1) / gsplit);
  const int tid = threadIdx.x;
  const DUnit u = w.units[ui];
  const DPair p = w.pairs[u.pair];
  const int ni = p.ni, nj = p.nj, ne = ni * nj;
  const int na1 = s.type_nalpha[p.ti], na2 = s.type_nalpha[p.tj];
  const long long base = p.moff + (long long)(ui - p.ubeg) * ne;
  const int so1 = s.type_state_off[p.ti], so2 = s.type_state_off[p.tj];
  const double *c1 = s.basis + s.type_basis_off[p.ti];
  const double *c2 = s.basis + s.type_basis_off[p.tj];
  const bool stage_coef = na1 * ni <= kCoefMax && na2 * nj <= kCoefMax;
  if (stage_coef) {
    for (int i = tid; i < na1 * ni; i += kContractThreads) c1s[i] = c1[i];
    for (int i = tid; i < na2 * nj; i += kContractThreads) c2s[i] = c2[i];
  }
  const double *cf1 = stage_coef ? c1s : c1;
  const double *cf2 = stage_coef ? c2s : c2;
  const int nlist = max(1, (u.spend - u.spbeg + kSpList - 1) / kSpList);
  int nsp = 0, nch = 0;
  long long boff0 = 0;
  // the list `li` of the unit's shell pairs, and its chunks: shell pair q
  // belongs to chunk sp_rel[q] / window
  auto load_list = [&](int li) {
    const int q0 = u.spbeg + li * kSpList;
    nsp = min(kSpList, u.spend - q0);
    nch = 0;
    __syncthreads();
    if (nsp <= 0) return;
    boff0 = w.sps[q0].boff;
    for (int i = tid; i < nsp; i += kContractThreads) {
      const DSp sp = w.sps[q0 + i];
      sp_ab[i] = sp.a | (sp.b << 16);
      sp_cls[i] = nsh(sp.la) | (nsh(sp.lb) << 8);
      sp_rel[i] = (int)(sp.boff - boff0);
    }
    __syncthreads();
    nch = sp_rel[nsp - 1] / window + 1;
    for (int i = tid; i < nsp; i += kContractThreads) {
      const int ch = sp_rel[i] / window;
      if (i == 0 || sp_rel[i - 1] / window != ch) cb[ch] = i;
    }
    if (tid == 0) cb[nch] = nsp;
    __syncthreads();
  };
  for (int e0 = 0; e0 < ne; e0 += kContractThreads * kElemsPerThread) {
    int lm1[kElemsPerThread], lm2[kElemsPerThread], m1[kElemsPerThread],
        m2[kElemsPerThread];
    double acc[kElemsPerThread][T];
#pragma unroll
    for (int j = 0; j < kElemsPerThread; ++j) {
      const int e = e0 + tid + j * kContractThreads;
      m2[j] = e < ne ? e / ni : 0;
      m1[j] = e < ne ? e - m2[j] * ni : 0;
      lm1[j] = e < ne ? s.state_lm[so1 + m1[j]] : 1 << 20;
      lm2[j] = e < ne ? s.state_lm[so2 + m2[j]] : 1 << 20;
    }
    auto zero = [&]() {
#pragma unroll
      for (int j = 0; j < kElemsPerThread; ++j)
#pragma unroll
        for (int t = 0; t < T; ++t) acc[j][t] = 0.0;
    };
    auto write = [&](int g) {
      const int t0 = g * T, tn = min(T, nterm - t0);
#pragma unroll
      for (int j = 0; j < kElemsPerThread; ++j) {
        const int e = e0 + tid + j * kContractThreads;
        if (e >= ne) continue;
#pragma unroll
        for (int t = 0; t < T; ++t)
          if (t < tn) M[(long long)(t0 + t) * w.m_total + base + e] = acc[j][t];
      }
    };
    // chunk ch of group g into buffer b: 16-byte copies (the blocks start on
    // 32 bytes and are padded), 128 / T threads to a term so that a thread
    // forms one address
    auto issue = [&](int g, int ch, int b) {
      constexpr int per = kContractThreads / T;
      const int t = tid / per;
      if (t < nterm - g * T) {
        const int q = cb[ch + 1] - 1, r0 = sp_rel[cb[ch]];
        const int len = (sp_rel[q] + (sp_cls[q] & 0xff) * (sp_cls[q] >> 8) - r0 + 1) / 2;
        const double *src = blk + (long long)(g * T + t) * w.blk_total + boff0 + r0;
        const unsigned dst = (unsigned)__cvta_generic_to_shared(bs + (b * T + t) * buf);
        for (int i = tid % per; i < len; i += per)
          asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(dst + 16 * i),
                       "l"(src + 2 * i)
                       : "memory");
      }
      asm volatile("cp.async.commit_group;\n" ::: "memory");
    };
    // groups [ga, gb) over the current list
    auto run = [&](int ga, int gb, bool first, bool last) {
      if (nch == 0) {
        for (int g = ga; g < gb; ++g) {
          if (first) zero();
          if (last) write(g);
        }
        return;
      }
      issue(ga, 0, 0);
      int b = 0;
      for (int g = ga; g < gb; ++g) {
        if (first) zero();
        for (int ch = 0; ch < nch; ++ch, b ^= 1) {
          const bool more = ch + 1 < nch || g + 1 < gb;
          if (more) {
            issue(ch + 1 < nch ? g : g + 1, ch + 1 < nch ? ch + 1 : 0, b ^ 1);
            asm volatile("cp.async.wait_group 1;\n" ::: "memory");
          } else {
            asm volatile("cp.async.wait_group 0;\n" ::: "memory");
          }
          __syncthreads();
          const double *bt = bs + b * T * buf - sp_rel[cb[ch]];
          for (int q = cb[ch]; q < cb[ch + 1]; ++q) {
            const int ab = sp_ab[q], cl = sp_cls[q];
            const int ia = ab & 0xffff, ib = ab >> 16, na = cl & 0xff, nb = cl >> 8;
            const int rel = sp_rel[q];
#pragma unroll
            for (int j = 0; j < kElemsPerThread; ++j) {
              if (lm1[j] >= na || lm2[j] >= nb) continue;
              const double cw = cf1[ia * ni + m1[j]] * cf2[ib * nj + m2[j]];
              const int o = rel + lm1[j] * nb + lm2[j];
              // rows of terms beyond the last hold leftovers; never written
#pragma unroll
              for (int t = 0; t < T; ++t) acc[j][t] += cw * bt[t * buf + o];
            }
          }
          __syncthreads();  // this chunk's buffer is refilled next
        }
        if (last) write(g);
      }
    };
    if (nlist == 1) {
      if (e0 == 0) load_list(0);
      run(g0, g1, true, true);
    } else {
      for (int g = g0; g < g1; ++g)
        for (int li = 0; li < nlist; ++li) {
          load_list(li);
          run(g, g + 1, li == 0, li == nlist - 1);
        }
    }
  }
}

template <int T>
static int contract_one(const DevSys &s, const DevWork &w, int nterm, const double *blk, double *M,
                        cudaStream_t st) {
  static bool done[64] = {};
  const size_t bytes = contract_smem<T>(w.blk_max);
  int dev = 0;
  IMAGO_CUDA(cudaGetDevice(&dev));
  if (dev < 0 || dev >= 64 || !done[dev]) {
    IMAGO_CUDA(cudaFuncSetAttribute(k_contract<T>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                    (int)contract_smem<T>(256)));
    if (dev >= 0 && dev < 64) done[dev] = true;
  }
  const int ntg = (nterm + T - 1) / T;
  const int gsplit = (int)std::max<long long>(
      1, std::min<long long>(ntg, (kContractCtas + w.nunits - 1) / w.nunits));
  k_contract<T><<<(unsigned)((long long)w.nunits * gsplit), kContractThreads, bytes, st>>>(
      s, w, nterm, gsplit, blk, M);
  IMAGO_LAUNCHED();
  return IMAGO_OK;
}

int launch_contract(const DevSys &s, const DevWork &w, int nterm,
                    const double *blk, double *M, cudaStream_t st, int terms_per_cta) {
  if (w.nunits == 0 || nterm == 0) return IMAGO_OK;
  if (nterm == 1) return contract_one<1>(s, w, nterm, blk, M, st);
  if (terms_per_cta >= 8 && nterm > 4) return contract_one<8>(s, w, nterm, blk, M, st);
  return contract_one<4>(s, w, nterm, blk, M, st);
}

}  // namespace imago

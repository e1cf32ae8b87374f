// prim.cuh -- FP64 primitive integrals per shell-pair class on the device.
//
// A "class" (LA, LB) is the pair of lmAlphaIndex classes of the two
// primitives (basis.f90:138-146): all real solid harmonics up to l on each
// side, nsh = 1, 4, 9, 16.  Results are the reference's sh(16,16) blocks
// (gaussIntegrals.f90) restricted to nsh(LA) x nsh(LB), row-major.
//
//  * two-centre overlap and kinetic (overlap2CIntg, kinetic2CIntg): the
//    Obara-Saika recursions in separable 1D form;
//  * mass velocity (massvel2CIntg): <nabla^2 a|nabla^2 b> from the same
//    1D overlap tables, two orders higher;
//  * momentum and dipole (momentum2CIntg, dipole3CIntg): three Cartesian
//    components, the operator moved into one 1D factor;
//  * three-centre overlap and nuclear (electron3CIntg, nuclear3CIntg):
//    McMurchie-Davidson.  The product of the two orbital primitives is
//    expanded in Hermite Gaussians about P with coefficients E_t (they
//    depend only on the shell pair), so the lattice sum over potential
//    sites C accumulates only Hermite integrals Q_tuv(P - C), t+u+v <= LA+LB
//    (35 values for d-d), and the E transform runs once per shell pair and
//    term after the sum.
//  * The Boys function follows the reference's own branches
//    (gaussIntegrals.f90:16080-16221) so nuclear integrals agree with it.
#pragma once

#include "common.cuh"

namespace imago {

// ---------------------------------------------------------------- Boys --
// For T <= 0.1f the reference sums seven series terms with Gamma(n+1/2)
// written as default-REAL (single precision) literals; above it the closed
// forms in erf(sqrt T) and exp(-T).  Integer powers are formed as gfortran
// forms them (T^3 = T^2 T, T^4 = T^2 T^2, T^5 = T^3 T^2, T^6 = T^3 T^3).
__device__ __forceinline__ float gamma_half_f(int n) {
  const float g[14] = {1.7724538509055161f, 0.88622692545275805f,
                       1.3293403881791370f, 3.3233509704478426f,
                       11.631728396567450f, 52.342777784553533f,
                       287.88527781504416f, 1871.2543057977896f,
                       14034.407293483402f, 119292.46199460901f,
                       1133278.3889487833f, 11899423.083962219f,
                       136843365.46556622f, 1710542068.3195722f};
  return g[n];
}

template <int NMAX>
__device__ __forceinline__ void boys_ref(double T, double F[NMAX + 1]) {
  const double exp_T = exp(-T);
  const double sqrt_pi = sqrt(kPi);
  if (T <= (double)0.1f) {
    const double T2 = T * T, T3 = T2 * T, T4 = T2 * T2;
    const double T5 = T3 * T2, T6 = T3 * T3;
#pragma unroll
    for (int N = 0; N <= NMAX; ++N) {
      double a[8];
#pragma unroll
      for (int k = 0; k < 8; ++k) a[k] = (double)gamma_half_f(N + k);
      F[N] = 0.5 * exp_T * a[0] *
             ((1 / a[1]) + (T / a[2]) + (T2 / a[3]) + (T3 / a[4]) +
              (T4 / a[5]) + (T5 / a[6]) + (T6 / a[7]));
    }
    return;
  }
  // T^(m + 1/2) as sqrt(T) times the product form of T^m: a pow costs as
  // much as the rest of an order
  const double root_T = sqrt(T);
  const double erf_T = erf(root_T);
  F[0] = 0.5 * ((sqrt_pi / root_T) * erf_T);
  const double T2 = T * T, T3 = T2 * T;
  const double Tp[7] = {1.0, T, T2, T3, T2 * T2, T3 * T2, T3 * T3};
  const double fact[13] = {1, 1, 2, 6, 24, 120, 720, 5040, 40320, 362880,
                           3628800, 39916800, 479001600};
  double c = 1.0, p4m = 1.0;
#pragma unroll
  for (int m = 1; m <= NMAX; ++m) {
    if (m > 1) c *= (double)(4 * m - 2);
    p4m *= 4.0;
    double erfterm = (sqrt_pi / (p4m * (root_T * Tp[m]))) * erf_T;
    double s = 0.0, p4k = 1.0;
#pragma unroll
    for (int k = 1; k <= m; ++k) {
      const int r = m - k + 1;
      double den = (k == 1) ? fact[2 * r] * T : (p4k * fact[2 * r]) * Tp[k];
      double term = fact[r] / den;
      s = (k == 1) ? term : s + term;
      p4k *= 4.0;
    }
    double v = erfterm - exp_T * s;
    F[m] = (m == 1) ? v : c * v;
  }
}

// ------------------------------------------------------ 1D Obara-Saika --
// S[i][j] for a Gaussian product with exponent p, relative to the centres:
// S00 = 1, S_{i+1,j} = PA S_ij + (i S_{i-1,j} + j S_{i,j-1})/(2p), and the
// same with PB for j.
template <int IA, int JB>
__device__ __forceinline__ void os1d(double PA, double PB, double inv2p,
                                     double S[IA + 1][JB + 1]) {
  S[0][0] = 1.0;
#pragma unroll
  for (int i = 0; i < IA; ++i)
    S[i + 1][0] = PA * S[i][0] + (i > 0 ? i * inv2p * S[i - 1][0] : 0.0);
#pragma unroll
  for (int j = 0; j < JB; ++j)
#pragma unroll
    for (int i = 0; i <= IA; ++i) {
      double v = PB * S[i][j];
      if (i > 0) v += i * inv2p * S[i - 1][j];
      if (j > 0) v += j * inv2p * S[i][j - 1];
      S[i][j + 1] = v;
    }
}

// v += four doubles from 32-byte aligned p.
__device__ __forceinline__ void add4(const double *p, double v[4]) {
  double x[4];
  asm volatile("ld.global.v4.f64 {%0, %1, %2, %3}, [%4];"
               : "=d"(x[0]), "=d"(x[1]), "=d"(x[2]), "=d"(x[3])
               : "l"(p)
               : "memory");
#pragma unroll
  for (int i = 0; i < 4; ++i) v[i] += x[i];
}

// f(0), f(1), ... f(N - 1) with the index as a type, so that everything
// derived from it is a constant and small arrays stay in registers.
template <int I>
struct Idx {
  static constexpr int value = I;
};
template <int N, int I = 0, class F>
__device__ __forceinline__ void static_for(F &&f) {
  if constexpr (I < N) {
    f(Idx<I>{});
    static_for<N, I + 1>(f);
  }
}

// Four doubles in one 32-byte store (one whole sector; 32-byte aligned).
__device__ __forceinline__ void store4(double *p, const double v[4]) {
  asm volatile("st.global.v4.f64 [%0], {%1, %2, %3, %4};" ::"l"(p), "d"(v[0]), "d"(v[1]),
               "d"(v[2]), "d"(v[3])
               : "memory");
}

// A block's rows as they are finished: to `out`, or (PAD) to a build's
// block buffer, where every block starts on 32 bytes and has blk_len
// doubles: each thread writes its own block, so single 8-byte stores would
// send one partial sector each (162-atom quartz EP: 2.0 G of them; whole
// sectors are a quarter; overlap and kinetic blocks of that cell 0.43 and
// 0.33 ms with 8-byte stores and the Cartesian block in local memory, 0.11
// and 0.12 so).  With `base`, base's block is added (base may be out).
template <int N, bool PAD>
struct BlockWriter {
  double *out;
  const double *base;
  double quad[4];
  template <int R, int M>
  __device__ __forceinline__ void row(const double (&v)[M]) {
    static_for<M>([&](auto im) {
      constexpr int m = decltype(im)::value, o = R * M + m;
      if constexpr (!PAD) {
        out[o] = v[m];
      } else {
        quad[o & 3] = v[m];
        if constexpr (o == N - 1)
          for (int i = (o & 3) + 1; i < 4; ++i) quad[i] = 0.0;
        if constexpr (o == N - 1 || (o & 3) == 3) {
          if (base) add4(base + (o & ~3), quad);
          store4(out + (o & ~3), quad);
        }
      }
    });
  }
};

// A block from its Cartesian products cart(p, q), each formed where a
// harmonic needs it.
template <int LA, int LB, bool PAD, class F>
__device__ __forceinline__ void write_sh_block(F &&cart, double *out,
                                               const double *base = nullptr) {
  BlockWriter<nsh(LA) * nsh(LB), PAD> w{out, base, {}};
  static_for<nsh(LA)>([&](auto i1) {
    constexpr int s1 = decltype(i1)::value;
    double row[nsh(LB)];
    static_for<nsh(LB)>([&](auto i2) {
      constexpr int s2 = decltype(i2)::value;
      double v = 0.0;
      static_for<sh_nterm(s1)>([&](auto j1) {
        static_for<sh_nterm(s2)>([&](auto j2) {
          constexpr int k1 = decltype(j1)::value, k2 = decltype(j2)::value;
          constexpr int p = sh_cart(s1, k1), q = sh_cart(s2, k2);
          constexpr double f = sh_coef(s1, k1) * sh_coef(s2, k2);
          v += f * cart(p, q);
        });
      });
      row[s2] = v;
    });
    w.template row<s1>(row);
  });
}

// Two-centre overlap (KIN = false) or kinetic energy (KIN = true) between
// primitives a1 at A and a2 at B, written to out[nsh(LA) * nsh(LB)].
// Kinetic: the Obara-Saika kinetic recursion in separable form,
//   T00 = xi (1 - 2 xi X^2),
//   T_{i+1,j} = PA T_ij + (i T_{i-1,j} + j T_{i,j-1})/(2p)
//               + 2 xi (S_{i+1,j} - i/(2 a1) S_{i-1,j})   (and j likewise),
//   KE = pref (Tx Sy Sz + Sx Ty Sz + Sx Sy Tz).
template <int LA, int LB, bool KIN, bool PAD = false>
__device__ __forceinline__ void prim2c(double a1, double a2, const double *A, const double *B,
                       double *out) {
  const double zeta = a1 + a2, xi = a1 * a2 / zeta, inv2p = 1.0 / (2.0 * zeta);
  double S[3][LA + 1][LB + 1];
  double T[3][LA + 1][LB + 1];
  double d2 = 0.0;
#pragma unroll
  for (int x = 0; x < 3; ++x) {
    const double P = (a1 * A[x] + a2 * B[x]) / zeta;
    const double PA = P - A[x], PB = P - B[x], X = A[x] - B[x];
    d2 += X * X;
    os1d<LA, LB>(PA, PB, inv2p, S[x]);
    if (KIN) {
      T[x][0][0] = xi * (1.0 - 2.0 * xi * X * X);
#pragma unroll
      for (int i = 0; i < LA; ++i) {
        double v = PA * T[x][i][0] + 2.0 * xi * S[x][i + 1][0];
        if (i > 0)
          v += i * inv2p * T[x][i - 1][0] -
               2.0 * xi * (i / (2.0 * a1)) * S[x][i - 1][0];
        T[x][i + 1][0] = v;
      }
#pragma unroll
      for (int j = 0; j < LB; ++j)
#pragma unroll
        for (int i = 0; i <= LA; ++i) {
          double v = PB * T[x][i][j] + 2.0 * xi * S[x][i][j + 1];
          if (i > 0) v += i * inv2p * T[x][i - 1][j];
          if (j > 0)
            v += j * inv2p * T[x][i][j - 1] -
                 2.0 * xi * (j / (2.0 * a2)) * S[x][i][j - 1];
          T[x][i][j + 1] = v;
        }
    }
  }
  const double pref = pow(kPi / zeta, 1.5) * exp(-xi * d2);
  write_sh_block<LA, LB, PAD>(
      [&](int p, int q) {
        const int ax = cart_exp(p, 0), ay = cart_exp(p, 1), az = cart_exp(p, 2);
        const int bx = cart_exp(q, 0), by = cart_exp(q, 1), bz = cart_exp(q, 2);
        double v;
        if (KIN)
          v = T[0][ax][bx] * S[1][ay][by] * S[2][az][bz] +
              S[0][ax][bx] * T[1][ay][by] * S[2][az][bz] +
              S[0][ax][bx] * S[1][ay][by] * T[2][az][bz];
        else
          v = S[0][ax][bx] * S[1][ay][by] * S[2][az][bz];
        return pref * v;
      },
      out);
}

// (alpha^2 / 8) with alpha the fine structure constant 7.2973525693e-3,
// the prefactor (fineStructure * 0.001)^2 / 8 of gaussIntegrals.f90:39118.
constexpr double kFineStructure = 7.2973525693 * 0.001;
constexpr double kMassVelPref = kFineStructure * kFineStructure / 8.0;

// One axis of the second derivative d^2/dx^2 x^i e^{-a x^2}
//   = i(i-1) x^{i-2} - 2a(2i+1) x^i + 4a^2 x^{i+2}
// taken on the left (atom 1), the right (atom 2) or both sides of the
// overlap table S (which runs two orders past the class on each side).
template <int IA, int JB>
__device__ __forceinline__ double d2_left(const double S[IA + 1][JB + 1],
                                          int i, int j, double a) {
  double v = -2.0 * a * (2 * i + 1) * S[i][j] + 4.0 * a * a * S[i + 2][j];
  if (i >= 2) v += i * (i - 1.0) * S[i - 2][j];
  return v;
}

template <int IA, int JB>
__device__ __forceinline__ double d2_right(const double S[IA + 1][JB + 1],
                                           int i, int j, double b) {
  double v = -2.0 * b * (2 * j + 1) * S[i][j] + 4.0 * b * b * S[i][j + 2];
  if (j >= 2) v += j * (j - 1.0) * S[i][j - 2];
  return v;
}

template <int IA, int JB>
__device__ __forceinline__ double d2_both(const double S[IA + 1][JB + 1],
                                          int i, int j, double a, double b) {
  double v = -2.0 * a * (2 * i + 1) * d2_right<IA, JB>(S, i, j, b) +
             4.0 * a * a * d2_right<IA, JB>(S, i + 2, j, b);
  if (i >= 2) v += i * (i - 1.0) * d2_right<IA, JB>(S, i - 2, j, b);
  return v;
}

// Mass-velocity block scale * <a|nabla^4|b> between primitives a1 at A and
// a2 at B (scale = kMassVelPref gives massvel2CIntg's sh; the build passes
// its negative, the sign the reference accumulates it with,
// integrals.F90:1440-1447).  nabla^4 is taken as <nabla^2 a|nabla^2 b>,
//   sum_x U_x S_y S_z + sum_{x != y} L_x R_y S_z,
// whose terms carry the size of the result; the reference's recursion seeds
// on 16 a2^4 <r_B^4> - 80 a2^3 <r_B^2> + 60 a2^2, which cancels to a value
// of order a1 a2 when a1 << a2.  s, p and d classes only (registers).
template <int LA, int LB, bool PAD = false>
__device__ __forceinline__ void prim_mv(double a1, double a2, const double *A, const double *B,
                                        double scale, double *out,
                                        const double *base = nullptr) {
  const double zeta = a1 + a2, xi = a1 * a2 / zeta, inv2p = 1.0 / (2.0 * zeta);
  // per axis: S, L (left d^2), R (right d^2), U (both) for i <= LA, j <= LB;
  // the extended overlap table lives only while its axis is formed
  double t[4][3][LA + 1][LB + 1];
  double d2 = 0.0;
#pragma unroll
  for (int x = 0; x < 3; ++x) {
    const double P = (a1 * A[x] + a2 * B[x]) / zeta;
    const double X = A[x] - B[x];
    d2 += X * X;
    double S[LA + 3][LB + 3];
    os1d<LA + 2, LB + 2>(P - A[x], P - B[x], inv2p, S);
#pragma unroll
    for (int i = 0; i <= LA; ++i)
#pragma unroll
      for (int j = 0; j <= LB; ++j) {
        t[0][x][i][j] = S[i][j];
        t[1][x][i][j] = d2_left<LA + 2, LB + 2>(S, i, j, a1);
        t[2][x][i][j] = d2_right<LA + 2, LB + 2>(S, i, j, a2);
        t[3][x][i][j] = d2_both<LA + 2, LB + 2>(S, i, j, a1, a2);
      }
  }
  const double pref = scale * pow(kPi / zeta, 1.5) * exp(-xi * d2);
  // one Cartesian pair, evaluated where a harmonic component needs it
  auto cart = [&](int p, int q) {
    const int i0 = cart_exp(p, 0), i1 = cart_exp(p, 1), i2 = cart_exp(p, 2);
    const int j0 = cart_exp(q, 0), j1 = cart_exp(q, 1), j2 = cart_exp(q, 2);
    const double s0 = t[0][0][i0][j0], s1 = t[0][1][i1][j1], s2 = t[0][2][i2][j2];
    const double l0 = t[1][0][i0][j0], l1 = t[1][1][i1][j1], l2 = t[1][2][i2][j2];
    const double r0 = t[2][0][i0][j0], r1 = t[2][1][i1][j1], r2 = t[2][2][i2][j2];
    const double u0 = t[3][0][i0][j0], u1 = t[3][1][i1][j1], u2 = t[3][2][i2][j2];
    double v = u0 * s1 * s2 + s0 * u1 * s2 + s0 * s1 * u2;
    v += (l0 * r1 + r0 * l1) * s2 + (l0 * r2 + r0 * l2) * s1 + (l1 * r2 + r1 * l2) * s0;
    return pref * v;
  };
  write_sh_block<LA, LB, PAD>(cart, out, base);
}

// Momentum <a|d/dx_c|b> (DIP = false) or dipole <a|(r - C)_c|b> (DIP =
// true) blocks for the three components c, written to out + c * cstride.
// The operator goes into the component's 1D factor of the overlap table:
//   dipole: (x - C_x) = x_B + (B_x - C_x) on atom 2's side;
//   momentum: d/dx x^j e^{-a x^2} = j x^{j-1} - 2 a x^{j+1} on atom 2's
//   side, or minus the same on atom 1's side (integration by parts), on the
//   side of the smaller exponent, so that the seed is formed from whichever
//   of PA = P - A and PB = P - B has not cancelled (the reference seeds
//   with 2 a1 PA S, gaussIntegrals.f90:23080-23082).
template <bool DIP, int IA, int JB>
__device__ __forceinline__ double vec_factor(const double S[IA + 1][JB + 1],
                                             int i, int j, bool left, double a1,
                                             double a2, double BC) {
  if (DIP) return S[i][j + 1] + BC * S[i][j];
  if (left) return 2.0 * a1 * S[i + 1][j] - (i > 0 ? i * S[i - 1][j] : 0.0);
  return -2.0 * a2 * S[i][j + 1] + (j > 0 ? j * S[i][j - 1] : 0.0);
}

// s, p and d classes: bounds known at compile time, tables in registers.
template <int LA, int LB, bool DIP, bool PAD = false>
__device__ __forceinline__ void prim_vec(double a1, double a2, const double *A, const double *B,
                         const double *C, double *out, long long cstride) {
  const double zeta = a1 + a2, xi = a1 * a2 / zeta, inv2p = 1.0 / (2.0 * zeta);
  const bool left = a1 <= a2;
  double S[3][LA + 1][LB + 1], D[3][LA + 1][LB + 1];
  double d2 = 0.0;
#pragma unroll
  for (int x = 0; x < 3; ++x) {
    const double P = (a1 * A[x] + a2 * B[x]) / zeta;
    const double X = A[x] - B[x];
    d2 += X * X;
    double T[LA + 2][LB + 2];
    os1d<LA + 1, LB + 1>(P - A[x], P - B[x], inv2p, T);
    const double BC = DIP ? B[x] - C[x] : 0.0;
#pragma unroll
    for (int i = 0; i <= LA; ++i)
#pragma unroll
      for (int j = 0; j <= LB; ++j) {
        S[x][i][j] = T[i][j];
        D[x][i][j] = vec_factor<DIP, LA + 1, LB + 1>(T, i, j, left, a1, a2, BC);
      }
  }
  const double pref = pow(kPi / zeta, 1.5) * exp(-xi * d2);
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    auto cart = [&](int p, int q) {
      double v = pref;
#pragma unroll
      for (int x = 0; x < 3; ++x) {
        const int i = cart_exp(p, x), j = cart_exp(q, x);
        v *= (x == c) ? D[x][i][j] : S[x][i][j];
      }
      return v;
    };
    write_sh_block<LA, LB, PAD>(cart, out + c * cstride);
  }
}

// ---------------------------------------------- McMurchie-Davidson 3C --
// Hermite expansion coefficients of one axis (hermite_e_row):
// E^{00}_0 = 1, E^{i+1,j}_t = E^{ij}_{t-1}/(2p) + PA E^{ij}_t + (t+1) E^{ij}_{t+1}
// and likewise for j with PB.

// Accumulate one three-centre overlap term into Q: w * exp(-mu |X|^2)
// h_t(X) h_u(Y) h_v(Z), h_t = (d/dX)^t exp(-mu X^2) / exp(-mu X^2),
// h_{t+1} = -2 mu (X h_t + t h_{t-1}).
template <int L>
__device__ __forceinline__ void accumulate_overlap_q(const double X[3],
                                                     double mu, double w,
                                                     double Q[nherm(L)]) {
  double h[3][L + 1];
#pragma unroll
  for (int x = 0; x < 3; ++x) {
    h[x][0] = 1.0;
#pragma unroll
    for (int t = 0; t < L; ++t)
      h[x][t + 1] = -2.0 * mu * (X[x] * h[x][t] + (t > 0 ? t * h[x][t - 1] : 0.0));
  }
  const double g = w * exp(-mu * (X[0] * X[0] + X[1] * X[1] + X[2] * X[2]));
#pragma unroll
  for (int t = 0; t <= L; ++t)
#pragma unroll
    for (int u = 0; u <= L - t; ++u) {
      const double gtu = g * h[0][t] * h[1][u];
#pragma unroll
      for (int v = 0; v <= L - t - u; ++v)
        Q[herm_index(t, u, v)] += gtu * h[2][v];
    }
}

// Add d^{tuv}/dX^{tuv} of a radial function f(|X|^2) to Q, t + u + v <= L <=
// 4, from G_n = (2 d/d|X|^2)^n f: with the one-axis coefficients
//   c(t, i) = t! / (2^i i! (t - 2i)!),
//   d^{tuv} f = sum_ijk c(t, i) c(u, j) c(v, k) X^{t-2i} Y^{u-2j} Z^{v-2k}
//               G_{t+u+v-i-j-k},
// which needs no intermediate orders in registers.
__host__ __device__ constexpr double radial_coef(int t, int i) {
  constexpr double c[5][3] = {{1, 0, 0}, {1, 0, 0}, {1, 1, 0}, {1, 3, 0}, {1, 6, 3}};
  return c[t][i];
}

template <int L>
__device__ __forceinline__ void accumulate_radial_q(const double X[3], const double G[L + 1],
                                                    double Q[nherm(L)]) {
  double p[3][L + 1];
#pragma unroll
  for (int x = 0; x < 3; ++x) {
    p[x][0] = 1.0;
#pragma unroll
    for (int t = 0; t < L; ++t) p[x][t + 1] = p[x][t] * X[x];
  }
#pragma unroll
  for (int t = 0; t <= L; ++t)
#pragma unroll
    for (int u = 0; u <= L - t; ++u)
#pragma unroll
      for (int v = 0; v <= L - t - u; ++v) {
        double sum = 0.0;
#pragma unroll
        for (int i = 0; 2 * i <= t; ++i)
#pragma unroll
          for (int j = 0; 2 * j <= u; ++j)
#pragma unroll
            for (int k = 0; 2 * k <= v; ++k)
              sum += radial_coef(t, i) * radial_coef(u, j) * radial_coef(v, k) *
                     (p[0][t - 2 * i] * p[1][u - 2 * j] * p[2][v - 2 * k]) *
                     G[t + u + v - i - j - k];
        Q[herm_index(t, u, v)] += sum;
      }
}

// Accumulate one nuclear term: w * d^{tuv}/dX^{tuv} of
// f(X) = exp(-mu |X|^2) F_0(nu |X|^2), the Gaussian-damped Coulomb
// potential integrated against the Hermite Gaussian of exponent p about P.
// With f = int_0^1 exp(-(mu + nu s^2)|X|^2) ds,
//   G_n = (-2)^n exp(-mu|X|^2) sum_k C(n,k) mu^{n-k} nu^k F_k.
template <int L>
__device__ __forceinline__ void accumulate_nuclear_q(const double X[3],
                                                     double mu, double nu,
                                                     double w,
                                                     double Q[nherm(L)]) {
  const double r2 = X[0] * X[0] + X[1] * X[1] + X[2] * X[2];
  double F[L + 1];
  boys_ref<L>(nu * r2, F);
  const double g = w * exp(-mu * r2);
  double G[L + 1];
  double mpow[L + 1], npow[L + 1];
  mpow[0] = 1.0;
  npow[0] = 1.0;
#pragma unroll
  for (int n = 1; n <= L; ++n) {
    mpow[n] = mpow[n - 1] * mu;
    npow[n] = npow[n - 1] * nu;
  }
  double sgn = 1.0;
#pragma unroll
  for (int n = 0; n <= L; ++n) {
    double v = 0.0, binom = 1.0;
#pragma unroll
    for (int k = 0; k <= n; ++k) {
      v += binom * mpow[n - k] * npow[k] * F[k];
      binom = binom * (n - k) / (k + 1);
    }
    G[n] = sgn * g * v;
    sgn *= -2.0;
  }
  accumulate_radial_q<L>(X, G, Q);
}

// Cartesian component of an exponent triple, x + y + z <= 2 (cart_exp's
// inverse).
__host__ __device__ constexpr int cart_index(int x, int y, int z) {
  constexpr int t[27] = {0, 3, 6, 2, 9, -1, 5, -1, -1, 1, 8, -1, 7, -1,
                         -1, -1, -1, -1, 4, -1, -1, -1, -1, -1, -1, -1, -1};
  return t[9 * x + 3 * y + z];
}

// One axis's Hermite coefficients E^{ij}_t for one i and every j <= LB:
// E[j][t], t <= i + j.
template <int I, int LB>
__device__ __forceinline__ void hermite_e_row(double PA, double PB, double inv2p,
                                              double (&E)[LB + 1][I + LB + 1]) {
  double e[I + LB + 1];
  e[0] = 1.0;
  static_for<I + LB>([&](auto iq) {
    // raise from order q to q + 1: with PA up to I, then with PB
    constexpr int q = decltype(iq)::value;
    if constexpr (q >= I) static_for<q + 1>([&](auto it) {
        E[q - I][decltype(it)::value] = e[decltype(it)::value];
      });
    const double X = q < I ? PA : PB;
    double f[I + LB + 1];
    static_for<q + 2>([&](auto it) {
      constexpr int t = decltype(it)::value;
      double v = 0.0;
      if constexpr (t <= q) v = X * e[t];
      if constexpr (t > 0) v += inv2p * e[t - 1];
      if constexpr (t + 1 <= q) v += (t + 1) * e[t + 1];
      f[t] = v;
    });
    static_for<q + 2>([&](auto it) { e[decltype(it)::value] = f[decltype(it)::value]; });
  });
  static_for<I + LB + 1>([&](auto it) { E[LB][decltype(it)::value] = e[decltype(it)::value]; });
}

// Row P (a Cartesian component of atom 1) of the block, as atom 2's real
// solid harmonics: pc(P, b) = sum_tuv Ex[ax][bx][t] Ey[ay][by][u]
// Ez[az][bz][v] Q_tuv, one axis after another.
// The coefficients are formed anew for every row: the empty asm keeps the
// compiler from holding all rows' (81 for d-d) in registers it has to spill.
template <int LA, int LB, int P>
__device__ __forceinline__ void hermite_row(const double (&PA0)[3], const double (&PB0)[3],
                                            double inv2p, const double (&Q)[nherm(LA + LB)],
                                            double (&row)[nsh(LB)]) {
  constexpr int AX = cart_exp(P, 0), AY = cart_exp(P, 1), AZ = cart_exp(P, 2);
  double PA[3] = {PA0[0], PA0[1], PA0[2]}, PB[3] = {PB0[0], PB0[1], PB0[2]};
  if constexpr (LA + LB >= 3)
    asm volatile("" : "+d"(PA[0]), "+d"(PA[1]), "+d"(PA[2]), "+d"(PB[0]), "+d"(PB[1]),
                 "+d"(PB[2]));
  double ex[LB + 1][AX + LB + 1], ey[LB + 1][AY + LB + 1], ez[LB + 1][AZ + LB + 1];
  hermite_e_row<AX, LB>(PA[0], PB[0], inv2p, ex);
  hermite_e_row<AY, LB>(PA[1], PB[1], inv2p, ey);
  hermite_e_row<AZ, LB>(PA[2], PB[2], inv2p, ez);
  double pc[ncart(LB)];
  static_for<LB + 1>([&](auto ibx) {
    constexpr int bx = decltype(ibx)::value;
    double T[AY + LB - bx + 1][AZ + LB - bx + 1];
    static_for<AY + LB - bx + 1>([&](auto iu) {
      static_for<AZ + LB - bx + 1>([&](auto iv) {
        constexpr int u = decltype(iu)::value, v = decltype(iv)::value;
        if constexpr (u + v <= AY + AZ + LB - bx) {
          double q = 0.0;
          static_for<AX + bx + 1>([&](auto it) {
            constexpr int t = decltype(it)::value, h = herm_index(t, u, v);
            q += ex[bx][t] * Q[h];
          });
          T[u][v] = q;
        }
      });
    });
    static_for<LB - bx + 1>([&](auto iby) {
      constexpr int by = decltype(iby)::value;
      double U[AZ + LB - bx - by + 1];
      static_for<AZ + LB - bx - by + 1>([&](auto iv) {
        constexpr int v = decltype(iv)::value;
        double q = 0.0;
        static_for<AY + by + 1>([&](auto iu) {
          constexpr int u = decltype(iu)::value;
          q += ey[by][u] * T[u][v];
        });
        U[v] = q;
      });
      static_for<LB - bx - by + 1>([&](auto ibz) {
        constexpr int bz = decltype(ibz)::value, c = cart_index(bx, by, bz);
        double q = 0.0;
        static_for<AZ + bz + 1>([&](auto iv) {
          constexpr int v = decltype(iv)::value;
          q += ez[bz][v] * U[v];
        });
        pc[c] = q;
      });
    });
  });
  static_for<nsh(LB)>([&](auto im) {
    constexpr int m = decltype(im)::value;
    double v = 0.0;
    static_for<sh_nterm(m)>([&](auto ik) {
      constexpr int k = decltype(ik)::value, c = sh_cart(m, k);
      constexpr double f = sh_coef(m, k);
      v += f * pc[c];
    });
    row[m] = v;
  });
}

// Turn accumulated Hermite integrals Q into the sh block, one Cartesian row
// of atom 1 at a time: a d-d block as a whole (100 Cartesian values beside
// 81 E coefficients) does not fit the registers, and its spills (1.6 KB a
// thread, now 0.3) were half of that class's memory traffic (1.2 GB written
// for 0.6 GB of Si8 blocks).  162-atom quartz EP primitives 10.5 -> 8.9 ms,
// Si8 0.78 -> 0.65 ms.
template <int LA, int LB, bool PAD = false>
__device__ __forceinline__ void hermite_to_sh(const double (&PA)[3], const double (&PB)[3],
                                              double inv2p, double pref,
                                              const double Q[nherm(LA + LB)], double *out,
                                              const double *base = nullptr) {
  double H[nherm(LA + LB)];
#pragma unroll
  for (int i = 0; i < nherm(LA + LB); ++i) H[i] = pref * Q[i];
  BlockWriter<nsh(LA) * nsh(LB), PAD> w{out, base, {}};
  double row[nsh(LB)];
  hermite_row<LA, LB, 0>(PA, PB, inv2p, H, row);
  w.template row<0>(row);
  if constexpr (LA >= 1) {
    hermite_row<LA, LB, 1>(PA, PB, inv2p, H, row);
    w.template row<1>(row);
    hermite_row<LA, LB, 2>(PA, PB, inv2p, H, row);
    w.template row<2>(row);
    hermite_row<LA, LB, 3>(PA, PB, inv2p, H, row);
    w.template row<3>(row);
  }
  if constexpr (LA >= 2) {
    // xy, xz, yz, xx - yy, 2 zz - xx - yy
    hermite_row<LA, LB, 7>(PA, PB, inv2p, H, row);
    w.template row<4>(row);
    hermite_row<LA, LB, 8>(PA, PB, inv2p, H, row);
    w.template row<5>(row);
    hermite_row<LA, LB, 9>(PA, PB, inv2p, H, row);
    w.template row<6>(row);
    double yy[nsh(LB)], sum[nsh(LB)];
    hermite_row<LA, LB, 4>(PA, PB, inv2p, H, row);
    hermite_row<LA, LB, 5>(PA, PB, inv2p, H, yy);
#pragma unroll
    for (int m = 0; m < nsh(LB); ++m) {
      sum[m] = row[m] + yy[m];
      row[m] -= yy[m];
    }
    w.template row<7>(row);
    hermite_row<LA, LB, 6>(PA, PB, inv2p, H, row);
#pragma unroll
    for (int m = 0; m < nsh(LB); ++m) row[m] = 2.0 * row[m] - sum[m];
    w.template row<8>(row);
  }
  static_assert(LA <= 2 && LB <= 2, "f classes: hermite_to_sh_rt");
}

// The same from the centres and exponents.
template <int LA, int LB, bool PAD = false>
__device__ __forceinline__ void hermite_to_sh(const double *A, const double *B, double a1,
                                              double a2, double pref,
                                              const double Q[nherm(LA + LB)], double *out,
                                              const double *base = nullptr) {
  const double zeta = a1 + a2;
  double PA[3], PB[3];
#pragma unroll
  for (int x = 0; x < 3; ++x) {
    const double P = (a1 * A[x] + a2 * B[x]) / zeta;
    PA[x] = P - A[x];
    PB[x] = P - B[x];
  }
  hermite_to_sh<LA, LB, PAD>(PA, PB, 1.0 / (2.0 * zeta), pref, Q, out, base);
}

// ------------------------------------------------ f classes, runtime loops --
// Classes with an f side are rare (no f functions in the measured
// workloads) and their fully unrolled forms are very large, so they share
// one implementation with runtime class arguments and small local arrays.
constexpr int kMaxL = 6;
constexpr int kMaxHerm = nherm(kMaxL);  // 84

static __device__ __forceinline__ void cart_to_sh_rt(int la, int lb, const double *pc,
                                              double *out, const double *base = nullptr) {
  const int ncb = ncart(lb), nsa = nsh(la), nsb = nsh(lb);
#pragma unroll 1
  for (int s1 = 0; s1 < nsa; ++s1)
#pragma unroll 1
    for (int s2 = 0; s2 < nsb; ++s2) {
      double v = 0.0;
      for (int k1 = 0; k1 < sh_nterm(s1); ++k1)
        for (int k2 = 0; k2 < sh_nterm(s2); ++k2)
          v += sh_coef(s1, k1) * sh_coef(s2, k2) *
               pc[sh_cart(s1, k1) * ncb + sh_cart(s2, k2)];
      out[s1 * nsb + s2] = base ? v + base[s1 * nsb + s2] : v;
    }
}

static __device__ __noinline__ void prim2c_rt(int la, int lb, bool kin, double a1,
                                       double a2, const double *A,
                                       const double *B, double *out) {
  const double zeta = a1 + a2, xi = a1 * a2 / zeta, inv2p = 1.0 / (2.0 * zeta);
  double S[3][4][4], T[3][4][4];
  double d2 = 0.0;
#pragma unroll 1
  for (int x = 0; x < 3; ++x) {
    const double P = (a1 * A[x] + a2 * B[x]) / zeta;
    const double PA = P - A[x], PB = P - B[x], X = A[x] - B[x];
    d2 += X * X;
    S[x][0][0] = 1.0;
    for (int i = 0; i < la; ++i)
      S[x][i + 1][0] = PA * S[x][i][0] + (i > 0 ? i * inv2p * S[x][i - 1][0] : 0.0);
    for (int j = 0; j < lb; ++j)
      for (int i = 0; i <= la; ++i) {
        double v = PB * S[x][i][j];
        if (i > 0) v += i * inv2p * S[x][i - 1][j];
        if (j > 0) v += j * inv2p * S[x][i][j - 1];
        S[x][i][j + 1] = v;
      }
    if (kin) {
      T[x][0][0] = xi * (1.0 - 2.0 * xi * X * X);
      for (int i = 0; i < la; ++i) {
        double v = PA * T[x][i][0] + 2.0 * xi * S[x][i + 1][0];
        if (i > 0)
          v += i * inv2p * T[x][i - 1][0] -
               2.0 * xi * (i / (2.0 * a1)) * S[x][i - 1][0];
        T[x][i + 1][0] = v;
      }
      for (int j = 0; j < lb; ++j)
        for (int i = 0; i <= la; ++i) {
          double v = PB * T[x][i][j] + 2.0 * xi * S[x][i][j + 1];
          if (i > 0) v += i * inv2p * T[x][i - 1][j];
          if (j > 0)
            v += j * inv2p * T[x][i][j - 1] -
                 2.0 * xi * (j / (2.0 * a2)) * S[x][i][j - 1];
          T[x][i][j + 1] = v;
        }
    }
  }
  const double pref = pow(kPi / zeta, 1.5) * exp(-xi * d2);
  double pc[400];
  const int nca = ncart(la), ncb = ncart(lb);
  for (int p = 0; p < nca; ++p)
    for (int q = 0; q < ncb; ++q) {
      const int ax = cart_exp(p, 0), ay = cart_exp(p, 1), az = cart_exp(p, 2);
      const int bx = cart_exp(q, 0), by = cart_exp(q, 1), bz = cart_exp(q, 2);
      double v;
      if (kin)
        v = T[0][ax][bx] * S[1][ay][by] * S[2][az][bz] +
            S[0][ax][bx] * T[1][ay][by] * S[2][az][bz] +
            S[0][ax][bx] * S[1][ay][by] * T[2][az][bz];
      else
        v = S[0][ax][bx] * S[1][ay][by] * S[2][az][bz];
      pc[p * ncb + q] = pref * v;
    }
  cart_to_sh_rt(la, lb, pc, out);
}

// prim_mv for the f classes, with runtime loops over tables in local
// memory (a fully unrolled f-d or f-f block does not fit the registers).
static __device__ __noinline__ void prim_mv_rt(int la, int lb, double a1,
                                               double a2, const double *A,
                                               const double *B, double scale,
                                               double *out, const double *base = nullptr) {
  const double zeta = a1 + a2, xi = a1 * a2 / zeta, inv2p = 1.0 / (2.0 * zeta);
  double t[4][3][4][4];
  double d2 = 0.0;
#pragma unroll 1
  for (int x = 0; x < 3; ++x) {
    const double P = (a1 * A[x] + a2 * B[x]) / zeta;
    const double X = A[x] - B[x];
    d2 += X * X;
    double S[6][6];
    os1d<5, 5>(P - A[x], P - B[x], inv2p, S);
#pragma unroll 1
    for (int i = 0; i <= la; ++i)
#pragma unroll 1
      for (int j = 0; j <= lb; ++j) {
        t[0][x][i][j] = S[i][j];
        t[1][x][i][j] = d2_left<5, 5>(S, i, j, a1);
        t[2][x][i][j] = d2_right<5, 5>(S, i, j, a2);
        t[3][x][i][j] = d2_both<5, 5>(S, i, j, a1, a2);
      }
  }
  const double pref = scale * pow(kPi / zeta, 1.5) * exp(-xi * d2);
  double pc[ncart(3) * ncart(3)];
  const int nca = ncart(la), ncb = ncart(lb);
#pragma unroll 1
  for (int p = 0; p < nca; ++p)
#pragma unroll 1
    for (int q = 0; q < ncb; ++q) {
      double s[3], l[3], r[3], u[3];
      for (int x = 0; x < 3; ++x) {
        const int i = cart_exp(p, x), j = cart_exp(q, x);
        s[x] = t[0][x][i][j];
        l[x] = t[1][x][i][j];
        r[x] = t[2][x][i][j];
        u[x] = t[3][x][i][j];
      }
      double v = u[0] * s[1] * s[2] + s[0] * u[1] * s[2] + s[0] * s[1] * u[2];
      v += (l[0] * r[1] + r[0] * l[1]) * s[2] + (l[0] * r[2] + r[0] * l[2]) * s[1] +
           (l[1] * r[2] + r[1] * l[2]) * s[0];
      pc[p * ncb + q] = pref * v;
    }
  cart_to_sh_rt(la, lb, pc, out, base);
}

// prim_vec for the f classes: runtime loops, tables in local memory.
template <bool DIP>
__device__ __noinline__ void prim_vec_rt(int la, int lb, double a1, double a2,
                                         const double *A, const double *B,
                                         const double *C, double *out,
                                         long long cstride) {
  const double zeta = a1 + a2, xi = a1 * a2 / zeta, inv2p = 1.0 / (2.0 * zeta);
  const bool left = a1 <= a2;
  double S[3][4][4], D[3][4][4];
  double d2 = 0.0;
#pragma unroll 1
  for (int x = 0; x < 3; ++x) {
    const double P = (a1 * A[x] + a2 * B[x]) / zeta;
    const double X = A[x] - B[x];
    d2 += X * X;
    double T[5][5];
    os1d<4, 4>(P - A[x], P - B[x], inv2p, T);
    const double BC = DIP ? B[x] - C[x] : 0.0;
#pragma unroll 1
    for (int i = 0; i <= la; ++i)
#pragma unroll 1
      for (int j = 0; j <= lb; ++j) {
        S[x][i][j] = T[i][j];
        D[x][i][j] = vec_factor<DIP, 4, 4>(T, i, j, left, a1, a2, BC);
      }
  }
  const double pref = pow(kPi / zeta, 1.5) * exp(-xi * d2);
  const int nca = ncart(la), ncb = ncart(lb), nsa = nsh(la), nsb = nsh(lb);
  double pc[ncart(3) * ncart(3)];
#pragma unroll 1
  for (int c = 0; c < 3; ++c) {
#pragma unroll 1
    for (int p = 0; p < nca; ++p)
#pragma unroll 1
      for (int q = 0; q < ncb; ++q) {
        double v = pref;
        for (int x = 0; x < 3; ++x) {
          const int i = cart_exp(p, x), j = cart_exp(q, x);
          v *= (x == c) ? D[x][i][j] : S[x][i][j];
        }
        pc[p * ncb + q] = v;
      }
    double blk[256];
    cart_to_sh_rt(la, lb, pc, blk);
#pragma unroll 1
    for (int e = 0; e < nsa * nsb; ++e) out[c * cstride + e] = blk[e];
  }
}

// The plane-wave overlap for one wave vector q with compile-time classes
// (s, p, d): the same complex-shifted recursion as prim_kov below, its
// tables and the Cartesian products unrolled into registers.
template <int LA, int LB>
__device__ void prim_kov_t(double a1, double a2, const double *A, const double *B,
                           const double *q, double *out_re, double *out_im) {
  const double zeta = a1 + a2, xi = a1 * a2 / zeta, inv2p = 1.0 / (2.0 * zeta);
  double Sr[3][LA + 1][LB + 1], Si[3][LA + 1][LB + 1], fr[3], fi[3];
#pragma unroll
  for (int x = 0; x < 3; ++x) {
    const double P = (a1 * A[x] + a2 * B[x]) / zeta, X = A[x] - B[x];
    const double ar = P - A[x], br = P - B[x], sh = -q[x] * inv2p;
    Sr[x][0][0] = 1.0;
    Si[x][0][0] = 0.0;
#pragma unroll
    for (int i = 0; i < LA; ++i) {
      double vr = ar * Sr[x][i][0] - sh * Si[x][i][0];
      double vi = ar * Si[x][i][0] + sh * Sr[x][i][0];
      if (i > 0) {
        vr += i * inv2p * Sr[x][i - 1][0];
        vi += i * inv2p * Si[x][i - 1][0];
      }
      Sr[x][i + 1][0] = vr;
      Si[x][i + 1][0] = vi;
    }
#pragma unroll
    for (int j = 0; j < LB; ++j)
#pragma unroll
      for (int i = 0; i <= LA; ++i) {
        double vr = br * Sr[x][i][j] - sh * Si[x][i][j];
        double vi = br * Si[x][i][j] + sh * Sr[x][i][j];
        if (i > 0) {
          vr += i * inv2p * Sr[x][i - 1][j];
          vi += i * inv2p * Si[x][i - 1][j];
        }
        if (j > 0) {
          vr += j * inv2p * Sr[x][i][j - 1];
          vi += j * inv2p * Si[x][i][j - 1];
        }
        Sr[x][i][j + 1] = vr;
        Si[x][i][j + 1] = vi;
      }
    const double mag = sqrt(kPi / zeta) * exp(-xi * X * X) * exp(-q[x] * q[x] / (4.0 * zeta));
    double sn, cs;
    sincos(q[x] * P, &sn, &cs);
    fr[x] = mag * cs;
    fi[x] = -mag * sn;
  }
  // the phases into the tables, then a pass for each part
#pragma unroll
  for (int x = 0; x < 3; ++x)
#pragma unroll
    for (int i = 0; i <= LA; ++i)
#pragma unroll
      for (int j = 0; j <= LB; ++j) {
        const double r = Sr[x][i][j];
        Sr[x][i][j] = r * fr[x] - Si[x][i][j] * fi[x];
        Si[x][i][j] = r * fi[x] + Si[x][i][j] * fr[x];
      }
  auto part = [&](int p, int c, bool imag) {
    double vr = 1.0, vi = 0.0;
#pragma unroll
    for (int x = 0; x < 3; ++x) {
      const int i = cart_exp(p, x), j = cart_exp(c, x);
      const double nr = vr * Sr[x][i][j] - vi * Si[x][i][j];
      vi = vr * Si[x][i][j] + vi * Sr[x][i][j];
      vr = nr;
    }
    return imag ? vi : vr;
  };
  write_sh_block<LA, LB, true>([&](int p, int c) { return part(p, c, false); }, out_re);
  write_sh_block<LA, LB, true>([&](int p, int c) { return part(p, c, true); }, out_im);
}


// Overlap with a plane wave, <a|exp(-i q.r)|b> (KOverlap2CIntg), complex,
// as two real blocks.  The product Gaussian times exp(-i q x) is
// exp(-i q P - q^2/(4p)) times a Gaussian about P' = P - i q/(2p): the 1D
// recursion runs with the complex PA' = PA - i q/(2p), PB' = PB - i q/(2p)
// and each axis carries sqrt(pi/p) exp(-xi X^2) exp(-q^2/(4p)) exp(-i q P).
// Runtime loops (every class; the build runs once per optical run).
static __device__ __noinline__ void prim_kov(int la, int lb, double a1, double a2,
                                             const double *A, const double *B,
                                             const double *q, double *out_re,
                                             double *out_im) {
  const double zeta = a1 + a2, xi = a1 * a2 / zeta, inv2p = 1.0 / (2.0 * zeta);
  double Sr[3][4][4], Si[3][4][4], fr[3], fi[3];
#pragma unroll 1
  for (int x = 0; x < 3; ++x) {
    const double P = (a1 * A[x] + a2 * B[x]) / zeta, X = A[x] - B[x];
    const double ar = P - A[x], br = P - B[x], sh = -q[x] * inv2p;
    Sr[x][0][0] = 1.0;
    Si[x][0][0] = 0.0;
    for (int i = 0; i < la; ++i) {
      double vr = ar * Sr[x][i][0] - sh * Si[x][i][0];
      double vi = ar * Si[x][i][0] + sh * Sr[x][i][0];
      if (i > 0) {
        vr += i * inv2p * Sr[x][i - 1][0];
        vi += i * inv2p * Si[x][i - 1][0];
      }
      Sr[x][i + 1][0] = vr;
      Si[x][i + 1][0] = vi;
    }
    for (int j = 0; j < lb; ++j)
      for (int i = 0; i <= la; ++i) {
        double vr = br * Sr[x][i][j] - sh * Si[x][i][j];
        double vi = br * Si[x][i][j] + sh * Sr[x][i][j];
        if (i > 0) {
          vr += i * inv2p * Sr[x][i - 1][j];
          vi += i * inv2p * Si[x][i - 1][j];
        }
        if (j > 0) {
          vr += j * inv2p * Sr[x][i][j - 1];
          vi += j * inv2p * Si[x][i][j - 1];
        }
        Sr[x][i][j + 1] = vr;
        Si[x][i][j + 1] = vi;
      }
    const double mag = sqrt(kPi / zeta) * exp(-xi * X * X) * exp(-q[x] * q[x] / (4.0 * zeta));
    double sn, cs;
    sincos(q[x] * P, &sn, &cs);
    fr[x] = mag * cs;
    fi[x] = -mag * sn;
  }
  double pcr[ncart(3) * ncart(3)], pci[ncart(3) * ncart(3)];
  const int nca = ncart(la), ncb = ncart(lb);
#pragma unroll 1
  for (int p = 0; p < nca; ++p)
#pragma unroll 1
    for (int c = 0; c < ncb; ++c) {
      double vr = 1.0, vi = 0.0;
      for (int x = 0; x < 3; ++x) {
        const int i = cart_exp(p, x), j = cart_exp(c, x);
        const double gr = Sr[x][i][j] * fr[x] - Si[x][i][j] * fi[x];
        const double gi = Sr[x][i][j] * fi[x] + Si[x][i][j] * fr[x];
        const double nr = vr * gr - vi * gi, ni = vr * gi + vi * gr;
        vr = nr;
        vi = ni;
      }
      pcr[p * ncb + c] = vr;
      pci[p * ncb + c] = vi;
    }
  cart_to_sh_rt(la, lb, pcr, out_re);
  cart_to_sh_rt(la, lb, pci, out_im);
}

static __device__ __noinline__ void accumulate_overlap_q_rt(int L, const double *X,
                                                     double mu, double w,
                                                     double *Q) {
  double h[3][kMaxL + 1];
  for (int x = 0; x < 3; ++x) {
    h[x][0] = 1.0;
    for (int t = 0; t < L; ++t)
      h[x][t + 1] = -2.0 * mu * (X[x] * h[x][t] + (t > 0 ? t * h[x][t - 1] : 0.0));
  }
  const double g = w * exp(-mu * (X[0] * X[0] + X[1] * X[1] + X[2] * X[2]));
  for (int t = 0; t <= L; ++t)
    for (int u = 0; u <= L - t; ++u) {
      const double gtu = g * h[0][t] * h[1][u];
      for (int v = 0; v <= L - t - u; ++v) Q[herm_index(t, u, v)] += gtu * h[2][v];
    }
}

static __device__ __noinline__ void accumulate_nuclear_q_rt(int L, const double *X,
                                                     double mu, double nu,
                                                     double w, double *Q) {
  const double r2 = X[0] * X[0] + X[1] * X[1] + X[2] * X[2];
  double F[kMaxL + 1];
  boys_ref<kMaxL>(nu * r2, F);
  const double g = w * exp(-mu * r2);
  double R[kMaxL + 1][kMaxHerm];
  double mpow[kMaxL + 1], npow[kMaxL + 1];
  mpow[0] = npow[0] = 1.0;
  for (int n = 1; n <= L; ++n) {
    mpow[n] = mpow[n - 1] * mu;
    npow[n] = npow[n - 1] * nu;
  }
  double sgn = 1.0;
  for (int n = 0; n <= L; ++n) {
    double s = 0.0, binom = 1.0;
    for (int k = 0; k <= n; ++k) {
      s += binom * mpow[n - k] * npow[k] * F[k];
      binom = binom * (n - k) / (k + 1);
    }
    R[n][0] = sgn * g * s;
    sgn *= -2.0;
  }
  for (int tot = 1; tot <= L; ++tot)
    for (int t = tot; t >= 0; --t)
      for (int u = tot - t; u >= 0; --u) {
        const int v = tot - t - u, id = herm_index(t, u, v);
        for (int n = 0; n <= L - tot; ++n) {
          double val;
          if (t > 0) {
            val = X[0] * R[n + 1][herm_index(t - 1, u, v)];
            if (t > 1) val += (t - 1) * R[n + 1][herm_index(t - 2, u, v)];
          } else if (u > 0) {
            val = X[1] * R[n + 1][herm_index(t, u - 1, v)];
            if (u > 1) val += (u - 1) * R[n + 1][herm_index(t, u - 2, v)];
          } else {
            val = X[2] * R[n + 1][herm_index(t, u, v - 1)];
            if (v > 1) val += (v - 1) * R[n + 1][herm_index(t, u, v - 2)];
          }
          R[n][id] = val;
        }
      }
  for (int i = 0; i < nherm(L); ++i) Q[i] += R[0][i];
}

static __device__ __noinline__ void hermite_to_sh_rt(int la, int lb, const double *A,
                                              const double *B, double a1,
                                              double a2, double pref,
                                              const double *Q, double *out,
                                              const double *base = nullptr) {
  const int L = la + lb;
  const double zeta = a1 + a2, inv2p = 1.0 / (2.0 * zeta);
  double E[3][4][4][kMaxL + 1];
  for (int x = 0; x < 3; ++x) {
    const double P = (a1 * A[x] + a2 * B[x]) / zeta;
    const double PA = P - A[x], PB = P - B[x];
    for (int i = 0; i <= la; ++i)
      for (int j = 0; j <= lb; ++j)
        for (int t = 0; t <= L; ++t) {
          double v;
          if (t > i + j) v = 0.0;
          else if (i == 0 && j == 0) v = 1.0;
          else if (i > 0) {
            v = PA * E[x][i - 1][j][t];
            if (t > 0) v += inv2p * E[x][i - 1][j][t - 1];
            if (t + 1 <= i - 1 + j) v += (t + 1) * E[x][i - 1][j][t + 1];
          } else {
            v = PB * E[x][i][j - 1][t];
            if (t > 0) v += inv2p * E[x][i][j - 1][t - 1];
            if (t + 1 <= i + j - 1) v += (t + 1) * E[x][i][j - 1][t + 1];
          }
          E[x][i][j][t] = v;
        }
  }
  double pc[400];
  const int nca = ncart(la), ncb = ncart(lb);
  for (int p = 0; p < nca; ++p)
    for (int q = 0; q < ncb; ++q) {
      const int ax = cart_exp(p, 0), ay = cart_exp(p, 1), az = cart_exp(p, 2);
      const int bx = cart_exp(q, 0), by = cart_exp(q, 1), bz = cart_exp(q, 2);
      double s = 0.0;
      for (int t = 0; t <= ax + bx; ++t)
        for (int u = 0; u <= ay + by; ++u) {
          const double etu = E[0][ax][bx][t] * E[1][ay][by][u];
          for (int v = 0; v <= az + bz; ++v)
            s += etu * E[2][az][bz][v] * Q[herm_index(t, u, v)];
        }
      pc[p * ncb + q] = pref * s;
    }
  cart_to_sh_rt(la, lb, pc, out, base);
}

}  // namespace imago

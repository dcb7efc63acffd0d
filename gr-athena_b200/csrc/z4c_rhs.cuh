// Pointwise Z4c right-hand side: Z4c::Z4cRHS (z4c/calculate_z4c_rhs.cpp:29-916)
// with the derivative precompute of Z4c::PrepareZ4cDerivatives
// (z4c/adm_z4c.cpp:972-1037) evaluated in place from the state, constant-eta
// branch, vacuum (matter terms vanish), Kreiss-Oliger dissipation included.
//
// The derivatives come from a source: the scratch that the derivative pass
// leaves (DerivSrc; the mixed second derivatives are D_a of D_b, a < b, formed
// as the reference forms them from its stored first derivatives), or, for the
// adjoint's Ricci sums, the state and its stored first derivatives
// (StencilSrc).
//   ricci_point  the Ricci tensor of the conformal metric and its
//                conformal-factor part, as Rsum_ab = R_ab + Rphi_ab
//                (the reference only ever uses the sum, :603, :745);
//   rhs_point    everything, without the Kreiss-Oliger terms.
// The operation order of every quantity follows the reference line by line;
// line numbers in the comments refer to calculate_z4c_rhs.cpp.
#pragma once

#include "z4c_common.cuh"
#include "z4c_deriv.cuh"

namespace z4c {

#define GUU(a, b) g_uu[sidx(a, b)]

// (a,b) of the symmetric pair q in xx,xy,xz,yy,yz,zz order
__device__ __forceinline__ int pair_a(int q) { return q < 3 ? 0 : (q < 5 ? 1 : 2); }
__device__ __forceinline__ int pair_b(int q) { return q < 3 ? q : (q < 5 ? q - 2 : 2); }

// Slots of the fields with stored first derivatives; component
// slot*3 + direction of the sd scratch ([block][33][vertex]).
constexpr int kSdChi = 0, kSdG = 1, kSdAlpha = 7, kSdBeta = 8, kSdFields = 11;
__host__ __device__ __forceinline__ constexpr int sd_field_var(int slot) {
  return slot == 0 ? Z4C_CHI : (slot <= 6 ? Z4C_GXX + slot - 1 : (slot == 7 ? Z4C_ALPHA
                                                                        : Z4C_BETAX + slot - 8));
}

// Second derivative of f along the pair q: Dxx on the diagonal, otherwise Dx
// along the first index of the stored Dx along the second (a < b); sdf points
// at the three stored first derivatives of f (stride nvol).
__device__ __forceinline__ double fd_d2(const double* __restrict__ f,
                                        const double* __restrict__ sdf, int64_t nvol, int q,
                                        const int64_t s[3], const FdScale& F) {
  const int a = pair_a(q), b = pair_b(q);
  if (a == b) return fd_dxx(f, s[a], F.cidx2[a]);
  return fd_dx(sdf + b * nvol, s[a], F.cidx1[a]);
}
// Load and store at a block-wide array's address, uniform over the CTA, plus
// the thread's own 32-bit byte offset: the address of an operand is one
// uniform addition and the thread keeps one offset register.
__device__ __forceinline__ double ldo(const double* base, unsigned pb) {
  return __ldg(reinterpret_cast<const double*>(reinterpret_cast<const char*>(base) + pb));
}
__device__ __forceinline__ void sto(double* base, unsigned pb, double v) {
  *reinterpret_cast<double*>(reinterpret_cast<char*>(base) + pb) = v;
}

// Operands of the pointwise algebra at one interior vertex.  StencilSrc
// evaluates the second derivatives of chi and g~ and the first ones of
// Gamma~ from the state and its stored first derivatives (the linearisation
// point of the adjoint); DerivSrc reads every derivative from the scratch of
// the derivative pass (z4c_deriv.cuh).
struct StencilSrc {
  const double *U, *SD;
  int64_t nvol;
  const int64_t* s;
  const FdScale* F;
  unsigned pb;  // byte offset of the vertex in a variable
  __device__ __forceinline__ double v(int n) const { return ldo(U + n * nvol, pb); }
  __device__ __forceinline__ double d1(int slot, int dir) const {
    return ldo(SD + (slot * 3 + dir) * nvol, pb);
  }
  __device__ __forceinline__ double dx(const double* f, int a) const {
    double out = 0.;
    out += -1. * (ldo(f - 3 * s[a], pb) - ldo(f + 3 * s[a], pb));
    out += 9. * (ldo(f - 2 * s[a], pb) - ldo(f + 2 * s[a], pb));
    out += -45. * (ldo(f - s[a], pb) - ldo(f + s[a], pb));
    return out * F->cidx1[a];
  }
  __device__ __forceinline__ double d2(int slot, int q) const {
    const int a = pair_a(q), b = pair_b(q);
    if (a != b) return dx(SD + (slot * 3 + b) * nvol, a);
    const double* f = U + sd_field_var(slot) * nvol;
    double out = 0.;
    out += 2. * (ldo(f - 3 * s[a], pb) + ldo(f + 3 * s[a], pb));
    out += -27. * (ldo(f - 2 * s[a], pb) + ldo(f + 2 * s[a], pb));
    out += 270. * (ldo(f - s[a], pb) + ldo(f + s[a], pb));
    out += -490. * ldo(f, pb);
    return out * F->cidx2[a];
  }
  __device__ __forceinline__ double dgam(int c, int b) const {
    return dx(U + (Z4C_GAMX + c) * nvol, b);
  }
  __device__ __forceinline__ double dkhat(int b) const { return dx(U + Z4C_KHAT * nvol, b); }
  __device__ __forceinline__ double dtheta(int b) const { return dx(U + Z4C_THETA * nvol, b); }
};
// A warp's 32 vertices: every derivative and the state's 22 variables staged
// in shared memory, [component][vertex] and [variable][vertex].
struct DerivSrc {
  const double *U, *D;  // this lane's entry of the first row of each
  __device__ __forceinline__ double v(int n) const { return U[n * kDvGroup]; }
  __device__ __forceinline__ double c(int q) const { return D[q * kDvGroup]; }
  __device__ __forceinline__ double d1(int slot, int dir) const { return c(9 * slot + dir); }
  __device__ __forceinline__ double d2(int slot, int q) const { return c(9 * slot + 3 + q); }
  __device__ __forceinline__ double dkhat(int b) const { return c(kDvKhat + b); }
  __device__ __forceinline__ double dtheta(int b) const { return c(kDvTheta + b); }
  __device__ __forceinline__ double dgam(int k, int b) const { return c(kDvGam + 3 * k + b); }
  __device__ __forceinline__ double adv(int n) const { return c(kDvAdv + n); }
};
constexpr int kStageDoubles = (kDvComponents + NVAR) * kDvGroup;  // of one warp
constexpr int kStageBytes = kStageDoubles * (int)sizeof(double);

// Copies the first NC components of the warp's group (contiguous at D, 16-byte
// aligned) into sm, asynchronously and all at once, so that the whole piece is
// in flight however few warps the registers admit.
template <int NC>
__device__ __forceinline__ void stage_components(double* sm, const double* __restrict__ D) {
  constexpr int pieces = NC * kDvGroup / 2;
  const int lane = (int)threadIdx.x % kDvGroup;
  const unsigned s = (unsigned)__cvta_generic_to_shared(sm);
#pragma unroll 17
  for (int q = lane; q < pieces; q += 32)
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(s + 16u * q), "l"(D + 2 * q)
                 : "memory");
}
// All of them and this lane's 22 variables (at u + n nvol, if the lane holds a
// vertex) behind them.
__device__ __forceinline__ DerivSrc stage_group(double* sm, const double* __restrict__ D,
                                                const double* __restrict__ u, int64_t nvol,
                                                bool active) {
  const int lane = (int)threadIdx.x % kDvGroup;
  stage_components<kDvComponents>(sm, D);
  double* su = sm + kDvComponents * kDvGroup + lane;
  if (active) {
    const unsigned t = (unsigned)__cvta_generic_to_shared(su);
#pragma unroll
    for (int n = 0; n < NVAR; ++n)
      asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(t + 8u * kDvGroup * n),
                   "l"(u + n * nvol)
                   : "memory");
  }
  asm volatile("cp.async.commit_group;\ncp.async.wait_group 0;\n" ::: "memory");
  __syncwarp();
  return DerivSrc{su, sm + lane};
}

// The heavy derivative gathers below run as rolled loops (GATHER_LOOP)
// writing small per-thread arrays; the tensor algebra that consumes them is
// fully unrolled.  Unrolled gathers let the compiler hoist hundreds of
// stencil loads at once and spill.
#ifndef Z4C_ROLLED_GATHERS
#define Z4C_ROLLED_GATHERS 0
#endif
#if Z4C_ROLLED_GATHERS
#define GATHER_LOOP _Pragma("unroll 1")
#else
#define GATHER_LOOP _Pragma("unroll")
#endif
#define GDD(a, b) g_dd[sidx(a, b)]
#define ADD(a, b) A_dd[sidx(a, b)]

// Inverse conformal metric (:295-311) and Christoffel symbols (:317-352).
// Gamma_ddd is written only when the caller passes storage for it.
template <class Src>
__device__ __forceinline__ void christoffel(const Src& src, const double g_dd[6], double g_uu[6],
                                            double Gamma_ddd[3][6], double Gamma_udd[3][6],
                                            double Gamma_u[3]) {
  {
    const double detg = det3(g_dd[0], g_dd[1], g_dd[2], g_dd[3], g_dd[4], g_dd[5]);
    inv3(1.0 / detg, g_dd, g_uu);
  }
  double Gd[3][6];
  {
    double dg[3][6];  // [c][ab] = d_c g_ab (stored dg_ddd_3d)
#pragma unroll
    for (int q = 0; q < 6; ++q)
#pragma unroll
      for (int c = 0; c < 3; ++c) dg[c][q] = src.d1(kSdG + q, c);
#pragma unroll
    for (int c = 0; c < 3; ++c)
#pragma unroll
      for (int a = 0; a < 3; ++a)
#pragma unroll
        for (int b = a; b < 3; ++b)
          Gd[c][sidx(a, b)] = 0.5 * (dg[a][sidx(b, c)] + dg[b][sidx(a, c)] - dg[c][sidx(a, b)]);
  }
#pragma unroll
  for (int c = 0; c < 3; ++c)
#pragma unroll
    for (int a = 0; a < 3; ++a)
#pragma unroll
      for (int b = a; b < 3; ++b) {
        double sacc = 0;
#pragma unroll
        for (int d = 0; d < 3; ++d) sacc += GUU(c, d) * Gd[d][sidx(a, b)];
        Gamma_udd[c][sidx(a, b)] = sacc;
      }
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    double sacc = 0;
#pragma unroll
    for (int b = 0; b < 3; ++b)
#pragma unroll
      for (int c = b; c < 3; ++c)
        sacc += ((b == c) ? 1.0 : 2.0) * GUU(b, c) * Gamma_udd[a][sidx(b, c)];
    Gamma_u[a] = sacc;
  }
  if (Gamma_ddd) {
#pragma unroll
    for (int c = 0; c < 3; ++c)
#pragma unroll
      for (int q = 0; q < 6; ++q) Gamma_ddd[c][q] = Gd[c][q];
  }
}

// Rsum_ab = R_ab + Rphi_ab at one interior vertex (:357-458), with the
// metric's algebra (inverse, Gamma^c_ab, Gamma^c) it forms on the way.
template <class Src>
__device__ __forceinline__ void ricci_point(const Src& src, const z4c_params_t& opt,
                                            double g_dd[6], double g_uu[6],
                                            double Gamma_udd[3][6], double Gamma_u[3],
                                            double Rsum[6]) {
#pragma unroll
  for (int c = 0; c < 6; ++c) g_dd[c] = src.v(Z4C_GXX + c);
  double Gamma_ddd[3][6];
  christoffel(src, g_dd, g_uu, Gamma_ddd, Gamma_udd, Gamma_u);
#define GDDD(c, a, b) Gamma_ddd[c][sidx(a, b)]
#define GUDD(c, a, b) Gamma_udd[c][sidx(a, b)]

  // Ricci tensor of the conformal metric, :357-396; each R_ab accumulates
  // its three groups of terms in the reference's order
  double dGam[3][3];  // [b][c] = d_b Gamma^c
GATHER_LOOP
  for (int c = 0; c < 3; ++c) {
#pragma unroll
    for (int b = 0; b < 3; ++b) dGam[b][c] = src.dgam(c, b);
  }
  double R_dd[6];
#pragma unroll
  for (int a = 0; a < 3; ++a)
#pragma unroll
    for (int b = a; b < 3; ++b) {
      double sacc = 0;
#pragma unroll
      for (int c = 0; c < 3; ++c)
        sacc += 0.5 * (GDD(c, a) * dGam[b][c] + GDD(c, b) * dGam[a][c] +
                       Gamma_u[c] * (GDDD(a, b, c) + GDDD(b, a, c)));
      R_dd[sidx(a, b)] = sacc;
    }
  // ddg_dddd(c,d,a,b): second derivative along c,d of g_ab, :158-178
GATHER_LOOP
  for (int q = 0; q < 6; ++q) {
    double sacc = R_dd[q];
#pragma unroll
    for (int c = 0; c < 3; ++c)
#pragma unroll
      for (int d = c; d < 3; ++d)
        sacc -= ((c == d) ? 0.5 : 1.0) * GUU(c, d) * src.d2(kSdG + q, sidx(c, d));
    R_dd[q] = sacc;
  }
#pragma unroll
  for (int a = 0; a < 3; ++a)
#pragma unroll
    for (int b = a; b < 3; ++b) {
      double sacc = R_dd[sidx(a, b)];
#pragma unroll
      for (int c = 0; c < 3; ++c)
#pragma unroll
        for (int d = 0; d < 3; ++d)
#pragma unroll
          for (int e = 0; e < 3; ++e)
            sacc += GUU(c, d) * (GUDD(e, c, a) * GDDD(b, e, d) + GUDD(e, c, b) * GDDD(a, e, d) +
                                 GUDD(e, a, d) * GDDD(e, c, b));
      R_dd[sidx(a, b)] = sacc;
    }

  // conformal-factor part, :241-245, :402-458
  const double chi = src.v(Z4C_CHI);
  const double chi_guarded = dmax(chi, opt.chi_div_floor);
  const double oochi = 1.0 / chi_guarded;
  const double oochi_psi_power = 1.0 / opt.chi_psi_power;
  double dphi_d[3];
#pragma unroll
  for (int a = 0; a < 3; ++a) dphi_d[a] = src.d1(kSdChi, a) * oochi * oochi_psi_power;
  double ddchi[6];  // stored ddchi_dd_3d
GATHER_LOOP
  for (int q = 0; q < 6; ++q) ddchi[q] = src.d2(kSdChi, q);
  double Ddphi_dd[6];
#pragma unroll
  for (int a = 0; a < 3; ++a)
#pragma unroll
    for (int b = a; b < 3; ++b) {
      double v = ddchi[sidx(a, b)] * oochi * oochi_psi_power -
                 opt.chi_psi_power * dphi_d[a] * dphi_d[b];
#pragma unroll
      for (int c = 0; c < 3; ++c) v -= GUDD(c, a, b) * dphi_d[c];
      Ddphi_dd[sidx(a, b)] = v;
    }
  double Stmp = 0.0;
#pragma unroll
  for (int c = 0; c < 3; ++c)
#pragma unroll
    for (int d = c; d < 3; ++d)
      Stmp += ((c == d) ? 1.0 : 2.0) * GUU(c, d) *
              (Ddphi_dd[sidx(c, d)] + 2. * dphi_d[c] * dphi_d[d]);
#pragma unroll
  for (int a = 0; a < 3; ++a)
#pragma unroll
    for (int b = a; b < 3; ++b) {
      const double rphi = 4. * dphi_d[a] * dphi_d[b] - 2. * Ddphi_dd[sidx(a, b)] -
                          2. * GDD(a, b) * Stmp;
      Rsum[sidx(a, b)] = R_dd[sidx(a, b)] + rphi;
    }
#undef GDDD
#undef GUDD
}

// The 22 right-hand-side values at one interior vertex without the
// Kreiss-Oliger terms.  With LV = false the advection sums are left out: the
// contracted path adds them, scaled, with the Kreiss-Oliger terms afterwards.
template <bool LV, class Src>
__device__ __forceinline__ void rhs_point(const Src& src, const z4c_params_t& opt,
                                          double out[NVAR]) {
  double g_dd[6], g_uu[6], Gamma_udd[3][6], Gamma_u[3], Rsum[6];
  ricci_point(src, opt, g_dd, g_uu, Gamma_udd, Gamma_u, Rsum);
  double A_dd[6];
#pragma unroll
  for (int c = 0; c < 6; ++c) A_dd[c] = src.v(Z4C_AXX + c);
  const double chi = src.v(Z4C_CHI), Khat = src.v(Z4C_KHAT);
  const double Theta = src.v(Z4C_THETA), alpha = src.v(Z4C_ALPHA);
#define GUDD(c, a, b) Gamma_udd[c][sidx(a, b)]

  // :231-274
  const double K = Khat + 2. * Theta;
  const double chi_guarded = dmax(chi, opt.chi_div_floor);
  const double oochi = 1.0 / chi_guarded;
  double oopsi4;
  if (opt.chi_psi_power == -4.) oopsi4 = chi_guarded;
  else oopsi4 = pow(chi_guarded, -4. / opt.chi_psi_power);
  const double oochi_psi_power = 1.0 / opt.chi_psi_power;
  double dchi_d[3], dphi_d[3], dalpha_d[3];
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    dchi_d[a] = src.d1(kSdChi, a);
    dphi_d[a] = dchi_d[a] * oochi * oochi_psi_power;
    dalpha_d[a] = src.d1(kSdAlpha, a);
  }

  // D D alpha, :482-521
  double Ddalpha = 0;
#pragma unroll
  for (int c = 0; c < 3; ++c)
#pragma unroll
    for (int d = 0; d < 3; ++d) Ddalpha += GUU(c, d) * dphi_d[c] * dalpha_d[d];
  double ddalpha[6];
GATHER_LOOP
  for (int q = 0; q < 6; ++q) ddalpha[q] = src.d2(kSdAlpha, q);
  double Ddalpha_dd[6];
#pragma unroll
  for (int a = 0; a < 3; ++a)
#pragma unroll
    for (int b = a; b < 3; ++b) {
      const double ddal = ddalpha[sidx(a, b)];
      double v = ddal - 2. * (dphi_d[a] * dalpha_d[b] + dphi_d[b] * dalpha_d[a]) +
                 2. * GDD(a, b) * Ddalpha;
#pragma unroll
      for (int c = 0; c < 3; ++c) v -= GUDD(c, a, b) * dalpha_d[c];
      Ddalpha_dd[sidx(a, b)] = v;
    }
  Ddalpha = 0;
#pragma unroll
  for (int a = 0; a < 3; ++a)
#pragma unroll
    for (int b = a; b < 3; ++b)
      Ddalpha += ((a == b) ? 1.0 : 2.0) * oopsi4 * GUU(a, b) * Ddalpha_dd[sidx(a, b)];

  // A contractions, :525-589
  double A_ud[3][3];
#pragma unroll
  for (int c = 0; c < 3; ++c)
#pragma unroll
    for (int b = 0; b < 3; ++b) {
      double sacc = 0;
#pragma unroll
      for (int d = 0; d < 3; ++d) sacc += GUU(c, d) * ADD(d, b);
      A_ud[c][b] = sacc;
    }
  double AA_dd[6];
#pragma unroll
  for (int a = 0; a < 3; ++a)
#pragma unroll
    for (int b = a; b < 3; ++b) {
      double sacc = 0;
#pragma unroll
      for (int c = 0; c < 3; ++c) sacc += ADD(a, c) * A_ud[c][b];
      AA_dd[sidx(a, b)] = sacc;
    }
  double trAA = 0;
#pragma unroll
  for (int a = 0; a < 3; ++a)
#pragma unroll
    for (int b = a; b < 3; ++b) trAA += ((a == b) ? 1.0 : 2.0) * GUU(a, b) * AA_dd[sidx(a, b)];
  double A_uu[6];
#pragma unroll
  for (int a = 0; a < 3; ++a)
#pragma unroll
    for (int b = a; b < 3; ++b) {
      double sacc = 0;
#pragma unroll
      for (int c = 0; c < 3; ++c) sacc += GUU(b, c) * A_ud[a][c];
      A_uu[sidx(a, b)] = sacc;
    }
  const double chi_pow_DA_u = -6.0 / opt.chi_psi_power;
  double DA_u[3];
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    double sacc = 0;
#pragma unroll
    for (int b = 0; b < 3; ++b) {
      const double dKhat_b = src.dkhat(b);
      const double dTheta_b = src.dtheta(b);
      sacc -= chi_pow_DA_u * A_uu[sidx(a, b)] * dchi_d[b] * oochi;
      sacc -= (1. / 3.) * GUU(a, b) * (2. * dKhat_b + dTheta_b);
    }
#pragma unroll
    for (int b = 0; b < 3; ++b)
#pragma unroll
      for (int c = b; c < 3; ++c)
        sacc += ((b == c) ? 1.0 : 2.0) * GUDD(a, b, c) * A_uu[sidx(b, c)];
    DA_u[a] = sacc;
  }
#undef GUDD

  // Ricci scalar, Ht, :596-613
  double R = 0;
#pragma unroll
  for (int a = 0; a < 3; ++a)
#pragma unroll
    for (int b = a; b < 3; ++b)
      R += ((a == b) ? 1.0 : 2.0) * oopsi4 * GUU(a, b) * Rsum[sidx(a, b)];
  const double Ht = R + (2. / 3.) * (K * K) - trAA;

  // advective derivatives, :184-226
  double beta_u[3];
#pragma unroll
  for (int a = 0; a < 3; ++a) beta_u[a] = src.v(Z4C_BETAX + a);
  // the advection sums, each read where it enters (lv[n * stride])
  auto Lv = [&](int n) {
    if constexpr (LV) return src.adv(n);
    else return 0.0;
  };
  double LGam_u[3], Lg_dd[6], LA_dd[6];

  // finalize Lie derivatives, :619-687
  double dbeta_du[3][3];  // [b][a] = d_b beta^a
#pragma unroll
  for (int a = 0; a < 3; ++a)
#pragma unroll
    for (int b = 0; b < 3; ++b) dbeta_du[b][a] = src.d1(kSdBeta + a, b);
  double dbeta = 0;
#pragma unroll
  for (int a = 0; a < 3; ++a) dbeta += dbeta_du[a][a];
  // ddbeta_ddu(a,b,c): second derivative along a,b of beta^c, :138-156
  double ddbeta[3][6];  // [c][pair(a,b)]
GATHER_LOOP
  for (int i = 0; i < 18; ++i) {
    const int c = i / 6, q = i % 6;
    ddbeta[c][q] = src.d2(kSdBeta + c, q);
  }
  double ddbeta_d[3] = {0, 0, 0};
#pragma unroll
  for (int a = 0; a < 3; ++a)
#pragma unroll
    for (int b = 0; b < 3; ++b) ddbeta_d[a] += (1. / 3.) * ddbeta[b][sidx(a, b)];
  const double Lchi = Lv(Z4C_CHI) + (1. / 6.) * opt.chi_psi_power * chi_guarded * dbeta;
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    LGam_u[a] = Lv(Z4C_GAMX + a);
    LGam_u[a] += (2. / 3.) * Gamma_u[a] * dbeta;
#pragma unroll
    for (int b = 0; b < 3; ++b) {
      LGam_u[a] += GUU(a, b) * ddbeta_d[b] - Gamma_u[b] * dbeta_du[b][a];
#pragma unroll
      for (int c = b; c < 3; ++c)
        LGam_u[a] += ((b == c) ? 1.0 : 2.0) * GUU(b, c) * ddbeta[a][sidx(b, c)];
    }
  }
#pragma unroll
  for (int a = 0; a < 3; ++a)
#pragma unroll
    for (int b = a; b < 3; ++b) {
      double lg = Lv(Z4C_GXX + sidx(a, b)), la = Lv(Z4C_AXX + sidx(a, b));
      lg -= (2. / 3.) * GDD(a, b) * dbeta;
      la -= (2. / 3.) * ADD(a, b) * dbeta;
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        lg += dbeta_du[a][c] * GDD(b, c);
        la += dbeta_du[b][c] * ADD(a, c);
        lg += dbeta_du[b][c] * GDD(a, c);
        la += dbeta_du[a][c] * ADD(b, c);
      }
      Lg_dd[sidx(a, b)] = lg;
      LA_dd[sidx(a, b)] = la;
    }

  // assemble, :694-902 (matter fields are zero, so their terms vanish exactly)
  out[Z4C_KHAT] = -Ddalpha + alpha * (trAA + (1. / 3.) * (K * K)) + Lv(Z4C_KHAT) +
                  opt.damp_kappa1 * (1 - opt.damp_kappa2) * alpha * Theta;
  out[Z4C_CHI] = Lchi - (1. / 6.) * opt.chi_psi_power * chi_guarded * alpha * K;
  out[Z4C_THETA] = Lv(Z4C_THETA) + alpha * (0.5 * Ht - (2. + opt.damp_kappa2) * opt.damp_kappa1 * Theta);
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    double v = 2. * alpha * DA_u[a] + LGam_u[a];
    v -= 2. * alpha * opt.damp_kappa1 * (src.v(Z4C_GAMX + a) - Gamma_u[a]);
#pragma unroll
    for (int b = 0; b < 3; ++b) v -= 2. * A_uu[sidx(a, b)] * dalpha_d[b];
    out[Z4C_GAMX + a] = v;
  }
#pragma unroll
  for (int a = 0; a < 3; ++a)
#pragma unroll
    for (int b = a; b < 3; ++b) {
      const int q = sidx(a, b);
      out[Z4C_GXX + q] = -2. * alpha * A_dd[q] + Lg_dd[q];
      double v = oopsi4 * (-Ddalpha_dd[q] + alpha * Rsum[q]);
      v -= (1. / 3.) * g_dd[q] * (-Ddalpha + alpha * R);
      v += alpha * (K * A_dd[q] - 2. * AA_dd[q]);
      v += LA_dd[q];
      out[Z4C_AXX + q] = v;
    }
  {
    const double fl = opt.lapse_oplog * opt.lapse_harmonicf + opt.lapse_harmonic * alpha;
    out[Z4C_ALPHA] = (opt.lapse_advect * Lv(Z4C_ALPHA) - fl * alpha * (Khat + 2 * opt.lapse_K * Theta));
  }
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    const double gam_a = src.v(Z4C_GAMX + a);
    double v = opt.shift_Gamma * gam_a + opt.shift_advect * Lv(Z4C_BETAX + a);
    if (fabs(opt.shift_alpha2Gamma) > 0.0) v += opt.shift_alpha2Gamma * (alpha * alpha) * gam_a;
    if (fabs(opt.shift_H) > 0.0) {
#pragma unroll
      for (int b = 0; b < 3; ++b)
        v += opt.shift_H * alpha * chi_guarded * (0.5 * alpha * dchi_d[b] - dalpha_d[b]) * GUU(a, b);
    }
    v -= opt.shift_eta * beta_u[a];
    out[Z4C_BETAX + a] = v;
  }
}

#undef GUU
#undef GDD
#undef ADD

}  // namespace z4c

// Stencil and stage helpers shared by the translation units that build the
// right-hand side: the exact one (z4c_kernels.cu, compiled without
// floating-point contraction) and the contracted one (z4c_fast.cu).  Each
// unit compiles its own inline copy under its own flags.
#pragma once

#include "z4c_common.cuh"
#include "z4c_kernels.cuh"

namespace z4c {

// ---- per-variable pass: Kreiss-Oliger -------------------
// One thread per (block, variable, interior (i, j)) column and chunk of
// interior planes, looping over the chunk's k.  Stencils along x and y read
// their lines directly; along z the nine-vertex window slides in registers.
// Index arithmetic is 32-bit (the launcher checks that the thread count fits).
struct ColChunks {
  int kc;  // interior planes per thread
  int n;   // chunks per column; 1: whole columns
};
struct Column {
  int b, n, i, j, k0, k1;
};
template <bool WHOLE>
__device__ __forceinline__ bool column_index(const Grid& g, const ColChunks& T, int block0,
                                             int nblk, Column& c) {
  const int n0 = g.nx[0] + 1, per = n0 * (g.nx[1] + 1);
  const int t = (int)(blockIdx.x * blockDim.x + threadIdx.x);
  const int nc = WHOLE ? 1 : T.n;
  if (t >= per * NVAR * nblk * nc) return false;
  const int ij = t % per;
  int rest = t / per;
  c.k0 = NG;
  c.k1 = NG + g.nx[2];
  if constexpr (!WHOLE) {
    c.k0 = NG + (rest % nc) * T.kc;
    c.k1 = min(c.k0 + T.kc - 1, c.k1);
    rest /= nc;
  }
  c.n = rest % NVAR;
  c.b = block0 + rest / NVAR;
  c.i = NG + ij % n0;
  c.j = NG + ij / n0;
  return true;
}
// Columns are cut into chunks where there are too few of them to give every
// SM 48 warps: the z loop of a column is a serial chain of loads (a 48^3 block,
// low-storage stage: 331 us whole, 234 us in chunks; 16^3: 64 and 37).
struct ColLaunch {
  ColChunks T;
  int grid;
};
inline ColLaunch column_launch(const Grid& g, int nblk, int threads) {
  const int nk = g.nx[2] + 1;
  const long long cols = (long long)(g.nx[0] + 1) * (g.nx[1] + 1) * NVAR * nblk;
  long long chunks = (148LL * 48 * 32 + cols - 1) / cols;
  if (chunks > nk) chunks = nk;
  ColLaunch L;
  L.T.kc = (int)((nk + chunks - 1) / chunks);
  L.T.n = (nk + L.T.kc - 1) / L.T.kc;
  L.grid = (int)((cols * L.T.n + threads - 1) / threads);
  return L;
}

// Loads for the stencil helpers below: read-only cache path for global
// memory (GL = true), plain loads for shared memory.
template <bool GL>
__device__ __forceinline__ double ld(const double* p) {
  if (GL) return __ldg(p);
  return *p;
}

// w[0..8] = f(-4..4) along stride st, the centre c given.
__device__ __forceinline__ void load_line(const double* __restrict__ f, int st, double c,
                                          double w[9]) {
#pragma unroll
  for (int q = 0; q < 9; ++q) w[q] = q == 4 ? c : __ldg(f + (q - 4) * st);
}
// Advection factor of variable n in the right-hand side (:860-902).
__device__ __forceinline__ double adv_factor(const z4c_params_t& p, int n) {
  if (n == Z4C_ALPHA) return p.lapse_advect;
  if (n >= Z4C_BETAX && n <= Z4C_BETAZ) return p.shift_advect;
  return 1.0;
}

// Advection and Kreiss-Oliger along one line w[0..8] = f(-4..4).  Half the
// difference of the two lop-sided stencils is the Kreiss-Oliger stencil K and
// half their sum the centred C below, so the side the sign of v selects is
// (v C - |v| K) / 2: one pass over the taps gives both terms, without a
// branch.  al = advection factor / (2 * 60 dx), kd the dissipation's factor.
__device__ __forceinline__ double adv_ko_line(const double w[9], double v, double al, double kd) {
  const double K = (w[0] + w[8]) - 8. * (w[1] + w[7]) + 28. * (w[2] + w[6]) -
                   56. * (w[3] + w[5]) + 70. * w[4];
  const double C = (w[0] - w[8]) - 8. * (w[1] - w[7]) + 32. * (w[2] - w[6]) -
                   104. * (w[3] - w[5]);
  return al * v * C + (kd - al * fabs(v)) * K;
}

// Kreiss-Oliger along one direction (FDStencilCenteredDegreeEven<8,4>,
// finite_differencing.tpp:335-368) from a line pointer or from the window.
template <bool GL = true>
__device__ __forceinline__ double fd_diss_line(const double* __restrict__ u, int st, double cidxd,
                                               double diss) {
  double out = 0.;
  out += 1. * (ld<GL>(u - 4 * st) + ld<GL>(u + 4 * st));
  out += -8. * (ld<GL>(u - 3 * st) + ld<GL>(u + 3 * st));
  out += 28. * (ld<GL>(u - 2 * st) + ld<GL>(u + 2 * st));
  out += -56. * (ld<GL>(u - st) + ld<GL>(u + st));
  out += 70. * ld<GL>(u);
  return out * cidxd * diss;
}
__device__ __forceinline__ double fd_diss_window(const double w[9], double cidxd, double diss) {
  double out = 0.;
  out += 1. * (w[0] + w[8]);
  out += -8. * (w[1] + w[7]);
  out += 28. * (w[2] + w[6]);
  out += -56. * (w[3] + w[5]);
  out += 70. * w[4];
  return out * cidxd * diss;
}

// Fills the z window of column c at the first interior k.
__device__ __forceinline__ void window_init(const double* __restrict__ f, int sk, int k0,
                                            double w[9]) {
#pragma unroll
  for (int q = 0; q < 8; ++q) w[q] = __ldg(f + (k0 - 4 + q) * sk);
}
__device__ __forceinline__ void window_advance(const double* __restrict__ f, int sk, int k,
                                               double w[9]) {
  w[8] = __ldg(f + (k + 4) * sk);
}
__device__ __forceinline__ void window_shift(double w[9]) {
#pragma unroll
  for (int q = 0; q < 8; ++q) w[q] = w[q + 1];
}

// Kreiss-Oliger added to one right-hand-side value in the reference's
// order, rhs += Diss_x; rhs += Diss_y; rhs += Diss_z (:908-915).
__device__ __forceinline__ double add_ko_column(double r, const double* __restrict__ fo, int nn0,
                                                const double w[9], const FdScale& F,
                                                double diss) {
  r += fd_diss_line(fo, 1, F.cidxd[0], diss);
  r += fd_diss_line(fo, nn0, F.cidxd[1], diss);
  r += fd_diss_window(w, F.cidxd[2], diss);
  return r;
}


// The 2S stage algebra of IntegrateZ4c (task_list_gr_z4c.cpp:176-195):
//   u1 <- u1 + delta u;  u <- gamma1 u + gamma2 u1 (+ gamma3 u2 = 0);
//   u <- u + beta dt rhs
// in the reference's WeightedAve / AddZ4cRHS branch order
// (mesh/weighted_ave.cpp:20-150): un = u, u1_in = u1 (0 at stage 1), r the
// right-hand side; v1 and v are the new u1 and u.
__device__ __forceinline__ void ls_update(const LsStage& w, double un, double u1_in, double r,
                                          double& v1, double& v) {
  v1 = u1_in;
  if (w.delta != 0.0) v1 += w.delta * un;  // w0 == 1, w2 == 0 branch
  if (w.gamma1 == 1.0) {  // gamma3 == 0 for every 2S integrator accepted
    v = un;
    if (w.gamma2 != 0.0) v += w.gamma2 * v1;
  } else if (w.gamma1 == 0.0) {
    if (w.gamma2 == 1.0) v = v1;
    else v = w.gamma2 * v1;
  } else {
    if (w.gamma2 != 0.0) v = w.gamma1 * un + w.gamma2 * v1;
    else v = un * w.gamma1;
  }
  v += w.beta_dt * r;
}

}  // namespace z4c

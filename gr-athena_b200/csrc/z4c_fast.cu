// The contracted right-hand side and low-storage stage (LaunchShape::contract).
// Compiled with -fmad=true: the pointwise algebra of z4c_rhs.cuh contracts
// into fused multiply-adds, and the order of the additions that close the
// right-hand side changes, so the values agree with the exact path (and the
// reference) to round-off rather than bit for bit.
//
// Two launches per stage:
//   k_deriv<true>  every derivative of every variable and, per variable, the
//                  advection and Kreiss-Oliger sums scaled as they enter
//                  (calculate_z4c_rhs.cpp:184-226, :908-915)
//   k_point_fast   the right-hand side at each vertex (rhs_point<false>), the
//                  sums added, then the 2S stage update (ls_update) into u1
//                  and the output register, or the right-hand side into rhs
#include <cuda_runtime.h>

#include "z4c_common.cuh"
#include "z4c_kernels.cuh"
#include "z4c_rhs.cuh"
#include "z4c_stencil.cuh"

namespace z4c {

namespace {

inline int div_up(int64_t a, int64_t b) { return (int)((a + b - 1) / b); }

// One warp per 32 interior vertices, their operands staged in shared memory
// (stage_group).  512 blocks of 16^3 with the stage update: 0.89 ms, 5.2 GB.
template <bool STAGE>
__global__ void __launch_bounds__(kDvGroup)
k_point_fast(Grid g, DevParams P, const double* __restrict__ u, const double* __restrict__ D,
             double* __restrict__ rhs, double* __restrict__ u1, double* __restrict__ u_out,
             LsStage ws, int block0, int ks, int nk) {
  extern __shared__ double sm[];
  const int n0 = g.nx[0] + 1, n1 = g.nx[1] + 1, np = nk * n1 * n0;
  const int l = (int)(blockIdx.x * kDvGroup + threadIdx.x);
  const int64_t b = block0 + (int)blockIdx.y;
  const int i = NG + l % n0, j = NG + (l / n0) % n1, k = NG + ks + l / (n0 * n1);
  const int64_t at = b * NVAR * g.nvol;
  const int64_t p = ((int64_t)k * g.nn[1] + j) * g.nn[0] + i;
  const DerivSrc src = stage_group(
      sm, D + blockIdx.y * dv_doubles(np) + (int64_t)blockIdx.x * (kDvComponents * kDvGroup),
      u + at + p, g.nvol, l < np);
  if (l >= np) return;
  double out[NVAR];
  rhs_point<false>(src, P.p, out);
  // every load of u1 before the first store: the compiler cannot tell their
  // addresses apart
  double v1[NVAR];
  if constexpr (STAGE) {
#pragma unroll
    for (int n = 0; n < NVAR; ++n) v1[n] = ws.u1_zero ? 0.0 : u1[at + n * g.nvol + p];
  }
#pragma unroll
  for (int n = 0; n < NVAR; ++n) {
    const double r = out[n] + src.adv(n);
    const int64_t q = at + n * g.nvol + p;
    if constexpr (STAGE) {
      double a, v;
      ls_update(ws, src.v(n), v1[n], r, a, v);
      u1[q] = a;
      u_out[q] = v;
    } else {
      rhs[q] = r;
    }
  }
}

// ---- the 128^3 merged grid --------------------------------------------------
// One block whose strides are compile-time constants: the whole right-hand
// side of a vertex from stencils in place (k_stencil_point, on the stored
// first derivatives of k_prep; no spills at 254 registers), then one column
// pass with the advection and Kreiss-Oliger sums and the stage update.  A
// stage takes 1.55 ms against 1.86 with the derivative pass (1.81 with the
// Ricci sums in a pass of their own and a branch on the shift's sign around the
// column pass's loads).  With strides from the Grid it spills (316 B), and the
// derivative pass is the faster one (64^3: 0.26 ms against 0.44).  Instances of
// other sizes, measured against the derivative pass, us a stage: 64^3 261 and
// 260, 96^3 705 and 774, 112^3 1068 and 1323, 144^3 2216 and 2860, 160^3 3017
// and 3548, 192^3 5900 and 6270.  So the instance pays for cubes from 96^3 on;
// only the size that Z4C_MERGED_NX names (128 by default) is built.
template <int THREADS, int NX>
__global__ void __launch_bounds__(THREADS)
k_stencil_point(Grid gin, DevParams P, const double* __restrict__ u,
                const double* __restrict__ sd, double* __restrict__ rhs, int block0) {
  const Grid g = fixed_geometry<NX>(gin);
  const int npts = (int)interior_count(g);
  const int l = (int)(blockIdx.x * THREADS + threadIdx.x);
  if (l >= npts) return;
  const int64_t b = block0 + (int)blockIdx.y;
  int i, j, k;
  interior_ijk(g, l, i, j, k);
  const unsigned pb = 8u * (unsigned)((k * g.nn[1] + j) * g.nn[0] + i);
  const StencilSrc src{u + b * NVAR * g.nvol, sd + b * kSdComponents * g.nvol, g.nvol, g.s,
                       &P.fd[b], pb};
  double out[NVAR];
  rhs_point<false>(src, P.p, out);
#pragma unroll
  for (int n = 0; n < NVAR; ++n) sto(rhs + (b * NVAR + n) * g.nvol, pb, out[n]);
}

template <int NX, bool STAGE>
__global__ void __launch_bounds__(512)
k_col_fast(Grid gin, DevParams P, const double* __restrict__ u, double* __restrict__ rhs,
           double* __restrict__ u1, double* __restrict__ u_out, LsStage ws, int block0,
           int nblk) {
  const Grid g = fixed_geometry<NX>(gin);
  Column c;
  if (!column_index<true>(g, ColChunks{}, block0, nblk, c)) return;
  const int nn0 = g.nn[0], sk = nn0 * g.nn[1];
  const double* U = u + (int64_t)c.b * NVAR * g.nvol + c.j * nn0 + c.i;
  const double* f = U + (int64_t)c.n * g.nvol;
  const double* bx = U + (int64_t)Z4C_BETAX * g.nvol;
  const int64_t base = ((int64_t)c.b * NVAR + c.n) * g.nvol + c.j * nn0 + c.i;
  const FdScale& F = P.fd[c.b];
  double al[3], kd[3];
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    al[a] = 0.5 * adv_factor(P.p, c.n) * F.lidx[a];
    kd[a] = P.p.diss * F.cidxd[a];
  }
  double w[9];
  window_init(f, sk, NG, w);
#pragma unroll 1
  for (int k = NG; k <= NG + g.nx[2]; ++k) {
    window_advance(f, sk, k, w);
    const int o = k * sk;
    const int64_t q = base + o;
    double x[9], y[9];
    load_line(f + o, 1, w[4], x);
    load_line(f + o, nn0, w[4], y);
    double r = rhs[q];
    r += adv_ko_line(x, __ldg(bx + o), al[0], kd[0]);
    r += adv_ko_line(y, __ldg(bx + g.nvol + o), al[1], kd[1]);
    r += adv_ko_line(w, __ldg(bx + 2 * g.nvol + o), al[2], kd[2]);
    if constexpr (STAGE) {
      double v1, v;
      ls_update(ws, w[4], ws.u1_zero ? 0.0 : u1[q], r, v1, v);
      u1[q] = v1;
      u_out[q] = v;
    } else {
      rhs[q] = r;
    }
    window_shift(w);
  }
}

template <bool STAGE>
void launch_merged(const Grid& g, const DevParams& P, const double* u, const RhsScratch& sc,
                   double* rhs, double* u1, double* u_out, const LsStage& w, int block0, int nblk,
                   cudaStream_t st) {
  constexpr int M = kMergedNX, T = 64, C = 128;
  launch_prep(g, P, u, sc.sd, block0, nblk, st);
  k_stencil_point<T, M><<<dim3(div_up(interior_count(g), T), nblk), T, 0, st>>>(g, P, u, sc.sd,
                                                                               rhs, block0);
  const int64_t cols = (int64_t)(g.nx[0] + 1) * (g.nx[1] + 1) * NVAR * nblk;
  k_col_fast<M, STAGE><<<div_up(cols, C), C, 0, st>>>(g, P, u, rhs, u1, u_out, w, block0, nblk);
  add_kernel_launches(2);
}

template <bool STAGE>
void launch_fast(const Grid& g, const DevParams& P, const double* u, const RhsScratch& sc,
                 double* rhs, double* u1, double* u_out, const LsStage& w, int block0, int nblk,
                 cudaStream_t st) {
  if (has_merged_geometry(g)) {
    launch_merged<STAGE>(g, P, u, sc, rhs, u1, u_out, w, block0, nblk, st);
    return;
  }
  for_deriv_chunks(g, block0, nblk, sc, [&](int b, int nb, int ks, int nk, double* D) {
    const DerivLaunch L = deriv_launch(g, nb, ks, nk);
    (L.narrow ? k_deriv<true, 18, 17> : k_deriv<true, 34, 9>)<<<L.grid, L.threads, L.smem, st>>>(
        g, P, u, D, L.T, b);
    const int64_t np = (int64_t)nk * (g.nx[1] + 1) * (g.nx[0] + 1);
    k_point_fast<STAGE><<<dim3(div_up(np, kDvGroup), nb), kDvGroup, kStageBytes, st>>>(
        g, P, u, D, rhs, u1, u_out, w, b, ks, nk);
    add_kernel_launches(2);
  });
}

}  // namespace

int allow_deriv_smem_fast() {
  cudaError_t e = cudaSuccess;
  auto set = [&](const void* k, int bytes) {
    const cudaError_t r =
        cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
    if (e == cudaSuccess) e = r;
  };
  set((const void*)k_deriv<true, 18, 17>, kDvMaxSmem);
  set((const void*)k_deriv<true, 34, 9>, kDvMaxSmem);
  set((const void*)k_point_fast<false>, kStageBytes);
  set((const void*)k_point_fast<true>, kStageBytes);
  return (int)e;
}

void launch_stage_ls_fast(const Grid& g, const DevParams& P, const double* u,
                          const RhsScratch& sc, double* rhs, double* u1, double* u_out,
                          const LsStage& w, int block0, int nblk, cudaStream_t st) {
  launch_fast<true>(g, P, u, sc, rhs, u1, u_out, w, block0, nblk, st);
}

void launch_rhs_fast(const Grid& g, const DevParams& P, const double* u, const RhsScratch& sc,
                     double* rhs, int block0, int nblk, cudaStream_t st) {
  launch_fast<false>(g, P, u, sc, rhs, nullptr, nullptr, LsStage{}, block0, nblk, st);
}

}  // namespace z4c

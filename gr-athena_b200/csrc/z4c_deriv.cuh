// The derivative pass of the right-hand side: every finite difference of one
// variable in one sweep, from shared memory, into a scratch of interior
// vertices that the pointwise passes read (z4c_rhs.cuh).  Included by the
// exact translation unit (no contraction: the reference's values bit for bit)
// and by the contracted one; each compiles its own instances.
#pragma once

#include <cuda_runtime.h>

#include "z4c_common.cuh"
#include "z4c_kernels.cuh"
#include "z4c_pieces.h"
#include "z4c_stencil.cuh"

namespace z4c {

// Components of a vertex in the scratch (its layout: z4c_pieces.h).
// The variables with second derivatives (chi, g~, alpha, beta: slot s) take
// nine components each, D_x D_y D_z and D_xx D_xy D_xz D_yy D_yz D_zz; Khat,
// Gamma~ and Theta three; every variable one advection sum (contracted path:
// advection and Kreiss-Oliger together, scaled as they enter).
constexpr int kDvHess = 11;                     // variables with second derivatives
constexpr int kDvGrad = 5;                      // with first derivatives only
constexpr int kDvFirst = 9 * kDvHess;           // first component of the latter
constexpr int kDvAdv = kDvFirst + 3 * kDvGrad;  // first advection sum
constexpr int kDvComponents = kDvAdv + NVAR;
constexpr int kDvCon = 9 * 7;  // the constraints' components: chi and g~
__host__ __device__ __forceinline__ constexpr int64_t dv_doubles(int64_t vertices) {
  return dv_doubles(vertices, kDvComponents);
}

// Variable of the f-th CTA row: the slots with second derivatives first (the
// longest CTAs), then those with first derivatives, then A~.
__host__ __device__ __forceinline__ constexpr int dv_var(int f) {
  return f == 0 ? Z4C_CHI
         : f <= 6 ? Z4C_GXX + f - 1
         : f == 7 ? Z4C_ALPHA
         : f <= 10 ? Z4C_BETAX + f - 8
         : f == 11 ? Z4C_KHAT
         : f == 12 ? Z4C_THETA
         : f <= 15 ? Z4C_GAMX + f - 13
                   : Z4C_AXX + f - 16;
}
// First component of the first derivatives of Khat, Theta, Gamma~^c.
constexpr int kDvKhat = kDvFirst, kDvTheta = kDvFirst + 3, kDvGam = kDvFirst + 6;

// A CTA takes w x h columns of one variable (w even) and the planes of one
// chunk; a thread two columns beside each other.
struct DerivTile {
  int w, h;    // columns along i and j
  int nx, n;   // tiles along i, tiles of the plane
  int kc;      // planes per CTA
  int ks, nk;  // interior planes of the launch: ks .. ks + nk - 1, from 0
};
constexpr int kDvMaxThreads = 160;
constexpr int kDvRing = 8;   // planes k-2 .. k+4 and the one in flight
constexpr int kDvMaxSmem = 76 * 1024;  // three CTAs per SM

__device__ __forceinline__ double fd7(double m3, double m2, double m1, double p1, double p2,
                                      double p3, double c) {
  double out = 0.;
  out += -1. * (m3 - p3);
  out += 9. * (m2 - p2);
  out += -45. * (m1 - p1);
  return out * c;
}
__device__ __forceinline__ double fd7xx(double m3, double m2, double m1, double c0, double p1,
                                        double p2, double p3, double c) {
  double out = 0.;
  out += 2. * (m3 + p3);
  out += -27. * (m2 + p2);
  out += 270. * (m1 + p1);
  out += -490. * c0;
  return out * c;
}
__device__ __forceinline__ double2 ld2(const double* s) {
  return *reinterpret_cast<const double2*>(s);
}
// The centred first derivative of two neighbours from pairs along stride st.
__device__ __forceinline__ double2 fd7p(const double* s, int st, double c) {
  const double2 a = ld2(s - 3 * st), b = ld2(s - 2 * st), d = ld2(s - st), e = ld2(s + st),
                f = ld2(s + 2 * st), g = ld2(s + 3 * st);
  return make_double2(fd7(a.x, b.x, d.x, e.x, f.x, g.x, c), fd7(a.y, b.y, d.y, e.y, f.y, g.y, c));
}
// f(-4 .. 5) of the row around the pair at s.
__device__ __forceinline__ void row10(const double* s, double r[10]) {
#pragma unroll
  for (int q = 0; q < 5; ++q) {
    const double2 v = ld2(s - 4 + 2 * q);
    r[2 * q] = v.x;
    r[2 * q + 1] = v.y;
  }
}
// Lop-sided advection from f(-4 .. 4) in registers; the shift's sign is the
// same over most warps.
__device__ __forceinline__ double fd_lx_reg(const double* w, double vx, double lidx) {
  double d = 0.;
  if (vx < 0) {
    d += 1. * w[0];
    d += -8. * w[1];
    d += 30. * w[2];
    d += -80. * w[3];
    d += 35. * w[4];
    d += 24. * w[5];
    d += -2. * w[6];
  } else {
    d += -1. * w[8];
    d += 8. * w[7];
    d += -30. * w[6];
    d += 80. * w[5];
    d += -35. * w[4];
    d += -24. * w[3];
    d += 2. * w[2];
  }
  return (vx * d) * lidx;
}

// One CTA per (tile, chunk of planes, variable, block), marching along z: the
// planes of the variable arrive in a ring in shared memory by asynchronous
// copies, the own column's nine values slide in registers, and D_y and D_z of
// the next plane, with their halo, go through shared memory to the mixed
// derivatives D_x D_y, D_x D_z, D_y D_z (the reference's order).  A thread
// takes two columns so that its rows are 16-byte shared-memory reads (one
// column per thread: 455 instructions per vertex and variable against 307).
// The cost does not depend on the block's size, as the strides of the tile
// are constants whatever those of the array.
// Bound by shared-memory reads (its data pipe at 73% of its peak) at 14 warps
// per SM: 512 blocks of 16^3, 1.19 ms, 4.05 GB of DRAM traffic (3.4 TB/s).
// Together with the pointwise pass (0.78 ms, 5.2 TB/s) it replaces stored first
// derivatives (0.50 ms), Ricci (0.64), advection (0.59) and main (0.72) passes
// whose stencils went to L1 and L2 at eight warps per SM.  Measured and slower:
// a column per thread (1.45 ms), separate launches for the variables with and
// without second derivatives (0.87 + 0.41), the y stencils moved into the
// pass that fills D_y (0.87 against 0.79 for the former), and on the
// contracted path D_z of D_x and D_y from register windows (1.79).
// W, H: the largest tile of the instance (18 x 17 or 34 x 9).  The row pitch
// W + 16 puts consecutive pairs of a W-wide tile in consecutive banks across
// a row's end.  NC: components of a vertex in out; kDvCon stores the
// derivatives of chi and g~ (grid y: these 7 variables) and no advection sums.
template <bool CONTRACT, int W, int H, int NC = kDvComponents>
__global__ void __launch_bounds__(kDvMaxThreads, 3)
k_deriv(Grid g, DevParams P, const double* __restrict__ u, double* __restrict__ out, DerivTile T,
        int block0) {
  extern __shared__ __align__(16) double sm[];
  constexpr int pitch = W + 16, plane = pitch * (H + 8), ring = kDvRing;
  double* const fs = sm;                            // ring of planes of the variable
  double* const dzs = fs + ring * plane;         // D_z, two planes, halo of 3 rows and 4 columns
  double* const dys = dzs + 2 * pitch * (H + 6);    // D_y, two planes, halo of 4 columns
  double* const cs = dys + 2 * pitch * H;           // the block's scalings
  constexpr int dzp = pitch * (H + 6), dyp = pitch * H;

  const int f = (int)blockIdx.y, n = dv_var(f);
  const int b = block0 + (int)blockIdx.z;
  const int tile = (int)blockIdx.x % T.n, chunk = (int)blockIdx.x / T.n;
  const int i0 = NG + (tile % T.nx) * T.w, j0 = NG + (tile / T.nx) * T.h;
  const int k0 = NG + T.ks + chunk * T.kc;
  const int k1 = min(k0 + T.kc, NG + T.ks + T.nk) - 1;
  const int tid = (int)threadIdx.x, wp = T.w / 2;
  const int tx = tid % wp * 2, ty = tid / wp;
  const int nn0 = g.nn[0], sk = nn0 * g.nn[1];
  const int n0 = g.nx[0] + 1, n1 = g.nx[1] + 1;
  constexpr int np = kDvGroup;  // stride of the components of a vertex
  constexpr bool sums = NC == kDvComponents;
  const bool hess = f < kDvHess, grad = f < kDvHess + kDvGrad;

  const double* U = u + (int64_t)b * NVAR * g.nvol;
  const double* F = U + (int64_t)n * g.nvol;
  // 1/(60 dx), 1/(180 dx^2) and the advection and dissipation factors: shared
  // memory keeps them out of the loop's registers
  if ((int)threadIdx.x < 12) {
    const int a = (int)threadIdx.x % 3, kind = (int)threadIdx.x / 3;
    const FdScale& S = P.fd[b];
    double v = kind == 0 ? S.cidx1[a] : kind == 1 ? S.cidx2[a] : kind == 2 ? S.lidx[a] : S.cidxd[a];
    if (CONTRACT && kind == 2) v *= 0.5 * adv_factor(P.p, n);
    if (CONTRACT && kind == 3) v *= P.p.diss;
    cs[threadIdx.x] = v;
  }

  // this thread's columns: in the array (they feed their neighbours), on the interior
  const bool in = ty < T.h;
  const bool row = in && j0 + ty < g.nn[1];
  const bool col0 = row && i0 + tx < nn0, col1 = row && i0 + tx + 1 < nn0;
  const bool ain = in && j0 + ty <= NG + g.nx[1];
  const bool act0 = ain && i0 + tx <= NG + g.nx[0], act1 = ain && i0 + tx < NG + g.nx[0];
  const int own = (ty + 4) * pitch + tx + 4;
  const int gp = (j0 + ty) * nn0 + i0 + tx;

  // A plane's copy: each warp takes rows of the tile with its halo, a lane a
  // column (and, in the wide instance, the one 32 further on).
  const int cw = (int)blockDim.x / 32, cc = tid % 32, cr = tid / 32;
  const int w8 = min(T.w + 8, nn0 - i0 + 4), h8 = min(T.h + 8, g.nn[1] - j0 + 4);
  const int co = (j0 - 4 + cr) * nn0 + i0 - 4 + cc;
  auto fetch = [&](int k) {  // plane k into its ring slot
    unsigned s = (unsigned)__cvta_generic_to_shared(fs + (unsigned)k % ring * plane +
                                                    cr * pitch + cc);
    const double* src = F + (int64_t)k * sk + co;
    for (int r = cr; r < h8; r += cw) {
      if (cc < w8)
        asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(s), "l"(src) : "memory");
      if (W + 8 > 32 && cc + 32 < w8)
        asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(s + 256u), "l"(src + 32)
                     : "memory");
      s += 8u * pitch * cw;
      src += cw * nn0;
    }
  };
  // this thread's halo pair of the D_z (and, beside the tile, D_y) planes:
  // two pairs on either side of each row, three rows above and below
  int hx = 0, hy = 0;
  const bool halo_x = tid < 4 * T.h, halo = tid < 4 * T.h + 6 * wp;
  if (halo_x) {
    const int q = tid % 4;
    hy = tid / 4;
    hx = q < 2 ? 2 * q - 4 : T.w + 2 * q - 4;
  } else if (halo) {
    const int q = tid - 4 * T.h, r = q / wp;
    hx = q % wp * 2;
    hy = r < 3 ? r - 3 : T.h + r - 3;
  }
  const int hs = (hy + 4) * pitch + hx + 4;   // in a plane of the variable
  const int hz = (hy + 3) * pitch + hx + 4;   // in a plane of D_z
  const int hyo = hy * pitch + hx + 4;        // in a plane of D_y
  const int oz = (ty + 3) * pitch + tx + 4, oy = ty * pitch + tx + 4;

  for (int k = hess ? k0 - 3 : k0; k <= k0 + 3; ++k) fetch(k);
  asm volatile("cp.async.commit_group;\n" ::: "memory");
  fetch(k0 + 4);
  asm volatile("cp.async.commit_group;\n" ::: "memory");
  double w0[9], w1[9];
#pragma unroll
  for (int q = 0; q < 8; ++q) {
    const double* z = F + (int64_t)(k0 - 4 + q) * sk + gp;
    w0[q] = col0 ? __ldg(z) : 0.0;
    w1[q] = col1 ? __ldg(z + 1) : 0.0;
  }
  const double* bp = U + (int64_t)Z4C_BETAX * g.nvol + gp;
  double* const ob0 = out + blockIdx.z * dv_doubles((int64_t)T.nk * n1 * n0, NC);
  int l = ((k0 - NG - T.ks) * n1 + j0 + ty - NG) * n0 + i0 + tx - NG;
  const int kd0 = grad ? (hess ? 9 * f : kDvFirst + 3 * (f - kDvHess)) : 0;
  auto advect = [&](const double* line, double v, int a) {
    if constexpr (CONTRACT) return adv_ko_line(line, v, cs[6 + a], cs[9 + a]);
    else return fd_lx_reg(line, v, cs[6 + a]);
  };
  // the first derivatives D_y, D_z of plane k that the mixed second
  // derivatives read, into the buffers of k's parity
  auto inner = [&](int k, double dz0, double dz1) {
    double* z = dzs + (k & 1) * dzp;
    double* y = dys + (k & 1) * dyp;
    const double* c = fs + (unsigned)k % ring * plane;
    if (in) {
      *reinterpret_cast<double2*>(z + oz) = make_double2(dz0, dz1);
      *reinterpret_cast<double2*>(y + oy) = fd7p(c + own, pitch, cs[1]);
    }
    if (halo) {
      auto at = [&](int d) { return ld2(fs + (unsigned)(k + d) % ring * plane + hs); };
      const double2 a = at(-3), b2 = at(-2), d = at(-1), e = at(1), ff = at(2), h = at(3);
      *reinterpret_cast<double2*>(z + hz) =
          make_double2(fd7(a.x, b2.x, d.x, e.x, ff.x, h.x, cs[2]),
                       fd7(a.y, b2.y, d.y, e.y, ff.y, h.y, cs[2]));
      if (halo_x) *reinterpret_cast<double2*>(y + hyo) = fd7p(c + hs, pitch, cs[1]);
    }
  };
  asm volatile("cp.async.wait_group 1;\n" ::: "memory");
  __syncthreads();
  if (hess)
    inner(k0, fd7(w0[1], w0[2], w0[3], w0[5], w0[6], w0[7], cs[2]),
          fd7(w1[1], w1[2], w1[3], w1[5], w1[6], w1[7], cs[2]));

  for (int k = k0; k <= k1; ++k) {
    // the shift, its latency behind the barrier and the inner pass
    double be0[3], be1[3];
    if constexpr (sums) {
#pragma unroll
      for (int a = 0; a < 3; ++a) {
        const double* p = bp + a * g.nvol + (int64_t)k * sk;
        be0[a] = act0 ? __ldg(p) : 0.0;
        be1[a] = act1 ? __ldg(p + 1) : 0.0;
      }
    }
    asm volatile("cp.async.wait_group 0;\n" ::: "memory");
    __syncthreads();
    if (k < k1) fetch(k + 5);
    asm volatile("cp.async.commit_group;\n" ::: "memory");
    if (in) {
      const double2 v = ld2(fs + (unsigned)(k + 4) % ring * plane + own);
      w0[8] = v.x;
      w1[8] = v.y;
    }
    if (hess && k < k1)
      inner(k + 1, fd7(w0[2], w0[3], w0[4], w0[6], w0[7], w0[8], cs[2]),
            fd7(w1[2], w1[3], w1[4], w1[6], w1[7], w1[8], cs[2]));
    if (act0) {
      // component q of the two vertices
      double* const o0 = ob0 + (int64_t)(l / kDvGroup) * (NC * kDvGroup) + l % kDvGroup;
      const int l1 = l + 1;
      double* const o1 = ob0 + (int64_t)(l1 / kDvGroup) * (NC * kDvGroup) + l1 % kDvGroup;
      auto put = [&](int q, double v0, double v1) {
        o0[q * np] = v0;
        if (act1) o1[q * np] = v1;
      };
      const double* c = fs + (unsigned)k % ring * plane + own;
      double x[10], acc0 = 0., acc1 = 0.;
      row10(c, x);
      if (grad) {
        put(kd0, fd7(x[1], x[2], x[3], x[5], x[6], x[7], cs[0]),
            fd7(x[2], x[3], x[4], x[6], x[7], x[8], cs[0]));
        if (hess)
          put(kd0 + 3, fd7xx(x[1], x[2], x[3], x[4], x[5], x[6], x[7], cs[3]),
              fd7xx(x[2], x[3], x[4], x[5], x[6], x[7], x[8], cs[3]));
      }
      if constexpr (sums) {
        acc0 += advect(x, be0[0], 0);
        acc1 += advect(x + 1, be1[0], 0);
      }
      double y0[9], y1[9];
#pragma unroll
      for (int q = 0; q < 9; ++q) {
        const double2 v = q == 4 ? make_double2(w0[4], w1[4]) : ld2(c + (q - 4) * pitch);
        y0[q] = v.x;
        y1[q] = v.y;
      }
      if constexpr (sums) {
        acc0 += advect(y0, be0[1], 1);
        acc1 += advect(y1, be1[1], 1);
        acc0 += advect(w0, be0[2], 2);
        acc1 += advect(w1, be1[2], 2);
        put(kDvAdv + n, acc0, acc1);
      }
      if (hess) {
        put(kd0 + 6, fd7xx(y0[1], y0[2], y0[3], y0[4], y0[5], y0[6], y0[7], cs[4]),
            fd7xx(y1[1], y1[2], y1[3], y1[4], y1[5], y1[6], y1[7], cs[4]));
        put(kd0 + 8, fd7xx(w0[1], w0[2], w0[3], w0[4], w0[5], w0[6], w0[7], cs[5]),
            fd7xx(w1[1], w1[2], w1[3], w1[4], w1[5], w1[6], w1[7], cs[5]));
        const double* z = dzs + (k & 1) * dzp + oz;
        double r[10];
        row10(z, r);
        put(kd0 + 2, r[4], r[5]);
        put(kd0 + 5, fd7(r[1], r[2], r[3], r[5], r[6], r[7], cs[0]),
            fd7(r[2], r[3], r[4], r[6], r[7], r[8], cs[0]));
        const double2 yz = fd7p(z, pitch, cs[1]);
        put(kd0 + 7, yz.x, yz.y);
        row10(dys + (k & 1) * dyp + oy, r);
        put(kd0 + 1, r[4], r[5]);
        put(kd0 + 4, fd7(r[1], r[2], r[3], r[5], r[6], r[7], cs[0]),
            fd7(r[2], r[3], r[4], r[6], r[7], r[8], cs[0]));
      } else if (grad) {
        put(kd0 + 1, fd7(y0[1], y0[2], y0[3], y0[5], y0[6], y0[7], cs[1]),
            fd7(y1[1], y1[2], y1[3], y1[5], y1[6], y1[7], cs[1]));
        put(kd0 + 2, fd7(w0[1], w0[2], w0[3], w0[5], w0[6], w0[7], cs[2]),
            fd7(w1[1], w1[2], w1[3], w1[5], w1[6], w1[7], cs[2]));
      }
    }
    l += n1 * n0;
    window_shift(w0);
    window_shift(w1);
  }
}

// Tile of the derivative pass on nblk blocks: rows of up to 34 columns, as
// many as the instance holds, the plane cut evenly.  The columns are cut into
// chunks of at least four planes where the tiles alone are fewer than six per
// SM (one 16^3 block: 27 us for its right-hand side against 64 with whole
// columns), and of at most 33 so that the last wave is short.
struct DerivLaunch {
  DerivTile T;
  dim3 grid;
  int threads;
  size_t smem;
  bool narrow;  // the 18 x 17 instance
};
inline DerivLaunch deriv_launch(const Grid& g, int nblk, int ks, int nk) {
  DerivLaunch L;
  DerivTile& T = L.T;
  const int n0 = g.nx[0] + 1, n1 = g.nx[1] + 1;
  // the instance whose tiles copy and compute less, halo and padding included;
  // the narrow one by at least a sixteenth, since it makes more tiles with
  // threads to spare (49 x 49 columns: narrow, a 48^3 block's four steps 2.80
  // ms against 2.91; 23 x 14: wide, right-hand side of 12 blocks 66 us against
  // 79)
  int64_t best = 0;
  int hm = 0;
  for (int narrow = 0; narrow < 2; ++narrow) {
    const int wt = narrow ? 18 : 34, ht = narrow ? 17 : 9;
    const int nx = (n0 + wt - 1) / wt, w = ((n0 + nx - 1) / nx + 1) / 2 * 2;
    const int ny = (n1 + ht - 1) / ht, h = (n1 + ny - 1) / ny;
    const int64_t cost = (int64_t)nx * ny * ((w + 8) * (h + 8) + 2 * w * h);
    if (narrow && 16 * cost > 15 * best) continue;
    best = cost;
    L.narrow = narrow != 0;
    hm = ht;
    T.nx = nx;
    T.w = w;
    T.h = h;
  }
  const int wm = L.narrow ? 18 : 34, ny = (n1 + hm - 1) / hm;
  T.n = T.nx * ny;
  T.ks = ks;
  T.nk = nk;
  int t = T.w / 2 * T.h;
  if (t < 4 * T.h + 3 * T.w) t = 4 * T.h + 3 * T.w;
  L.threads = (t + 31) / 32 * 32;
  const int64_t ctas = (int64_t)T.n * NVAR * nblk;
  int chunks = (int)((148 * 6 + ctas - 1) / ctas);
  if (chunks > (nk + 3) / 4) chunks = (nk + 3) / 4;
  if (chunks < (nk + 32) / 33) chunks = (nk + 32) / 33;
  T.kc = (nk + chunks - 1) / chunks;
  chunks = (nk + T.kc - 1) / T.kc;
  L.grid = dim3((unsigned)(T.n * chunks), NVAR, (unsigned)nblk);
  L.smem = sizeof(double) * (wm + 16) * (kDvRing * (hm + 8) + 2 * (hm + 6) + 2 * hm) + 96;
  return L;
}

// for_deriv_chunks on the right-hand side's scratch: launch(b, nb, ks, nk,
// scratch).
template <class Launch>
inline void for_deriv_chunks(const Grid& g, int block0, int nblk, const RhsScratch& sc,
                             Launch launch) {
  for_deriv_chunks(g.nx, block0, nblk, kDvComponents, sc.share,
                   [&](int b, int nb, int ks, int nk, int64_t at) {
                     launch(b, nb, ks, nk, sc.base + at);
                   });
}

}  // namespace z4c

// How the derivative pass's scratch is laid out and cut into pieces.  Plain
// C++: the host tests compile it without CUDA.
#pragma once

#include <cstdint>
#include <initializer_list>

#ifdef __CUDACC__
#define Z4C_PIECES_HD __host__ __device__ __forceinline__
#else
#define Z4C_PIECES_HD inline
#endif

namespace z4c {

// Layout of the scratch: [block][group of 32 interior vertices of the slab]
// [component][vertex of the group], so that a warp of the pointwise pass finds
// all of its operands in one contiguous piece.
constexpr int kDvGroup = 32;
// Scratch doubles of one block's (or slab's) vertices.
Z4C_PIECES_HD constexpr int64_t dv_doubles(int64_t vertices, int components) {
  return (vertices + kDvGroup - 1) / kDvGroup * kDvGroup * components;
}

// Every block of the mesh has its share of the scratch, and a call uses the
// shares of its own blocks only, so that calls on different blocks may run at
// the same time on different streams.  Shares are whole groups: they start on
// 256-byte boundaries.
inline int64_t dv_share(int64_t cap, int nblocks) {
  return cap / nblocks / kDvGroup * kDvGroup;
}
// A block's shares of a context's scratch.
struct DvShares {
  int64_t rhs;  // right-hand side, diagnostics and adjoint
  int64_t con;  // constraints
};
// The least a context runs with: what the diagnostics and the adjoint need
// (parts), and a plane of the constraints' nc components.
inline DvShares dv_least_shares(int64_t parts, int64_t plane, int nc) {
  return {(parts + kDvGroup - 1) / kDvGroup * kDvGroup, dv_doubles(plane + kDvGroup, nc)};
}
// What serves the passes best: every component of the right-hand side (whole)
// where that is at most a little more, or small on the mesh (512 Mi doubles),
// and every one of the constraints' (an eighth of a 16^3 block's memory; with a
// seventh of it, two planes, the constraints of one block take 182 us instead
// of 30).  The passes run in pieces that fit.
inline DvShares dv_best_shares(const DvShares& least, int64_t whole, int64_t npts, int nc,
                               int nblocks) {
  DvShares s = least;
  if (whole > s.rhs &&
      (whole <= s.rhs + s.rhs / 16 || whole * nblocks <= (int64_t)1 << 29))
    s.rhs = whole;
  s.con = dv_doubles(npts, nc);
  return s;
}
// Allocates the scratch of nblocks blocks: the best shares, or, where the
// device does not hold those, the least.  alloc(doubles) says whether it could;
// returns whether one of them did, its shares in *got.
template <class Alloc>
inline bool dv_reserve(const DvShares& best, const DvShares& least, int nblocks, Alloc alloc,
                       DvShares* got) {
  for (const DvShares* s : {&best, &least}) {
    *got = *s;
    if (alloc((s->rhs + s->con) * nblocks)) return true;
  }
  return false;
}

// Runs the derivative and pointwise passes on blocks block0 .. block0 + nblk - 1
// of nx cells in pieces whose scratch fits these blocks' shares: all at once,
// by equal groups of blocks, or, where one block does not fit, by slabs of
// planes of each block.  launch(b, nb, ks, nk, at) takes blocks b .. b + nb - 1
// and interior planes ks .. ks + nk - 1, with its scratch at double `at`.
template <class Launch>
inline void for_deriv_chunks(const int nx[3], int block0, int nblk, int components, int64_t share,
                             Launch launch) {
  const int64_t at = block0 * share, cap = nblk * share;
  const int nk = nx[2] + 1;
  const int64_t plane = (int64_t)(nx[0] + 1) * (nx[1] + 1);
  const int64_t per = dv_doubles(plane * nk, components);
  if (per <= cap) {
    const int64_t room = cap / per;  // blocks that fit
    const int64_t pieces = (nblk + room - 1) / room;
    const int nb = (int)((nblk + pieces - 1) / pieces);
    for (int b = 0; b < nblk; b += nb)
      launch(block0 + b, nblk - b < nb ? nblk - b : nb, 0, nk, at);
    return;
  }
  const int64_t most = (cap / components - kDvGroup) / plane;  // planes that fit
  const int64_t slabs = (nk + most - 1) / most;
  const int h = (int)((nk + slabs - 1) / slabs);
  for (int b = 0; b < nblk; ++b)
    for (int k = 0; k < nk; k += h) launch(block0 + b, 1, k, nk - k < h ? nk - k : h, at);
}

}  // namespace z4c

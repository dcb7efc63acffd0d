// How the derivative pass's scratch is laid out and cut into pieces.  Plain
// C++: the host tests compile it without CUDA.
#pragma once

#include <cstdint>

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

// Runs the derivative and pointwise passes on nblk blocks of nx cells in pieces
// whose scratch fits cap doubles: all at once, by equal groups of blocks, or,
// where one block does not fit, by slabs of planes of each block.
// launch(b, nb, ks, nk) takes blocks b .. b + nb - 1 and interior planes ks ..
// ks + nk - 1.
template <class Launch>
inline void for_deriv_chunks(const int nx[3], int nblk, int components, int64_t cap,
                             Launch launch) {
  const int nk = nx[2] + 1;
  const int64_t plane = (int64_t)(nx[0] + 1) * (nx[1] + 1);
  const int64_t per = dv_doubles(plane * nk, components);
  if (per <= cap) {
    const int64_t room = cap / per;  // blocks that fit
    const int64_t pieces = (nblk + room - 1) / room;
    const int nb = (int)((nblk + pieces - 1) / pieces);
    for (int b = 0; b < nblk; b += nb) launch(b, nblk - b < nb ? nblk - b : nb, 0, nk);
    return;
  }
  const int64_t most = (cap / components - kDvGroup) / plane;  // planes that fit
  const int64_t slabs = (nk + most - 1) / most;
  const int h = (int)((nk + slabs - 1) / slabs);
  for (int b = 0; b < nblk; ++b)
    for (int k = 0; k < nk; k += h) launch(b, 1, k, nk - k < h ? nk - k : h);
}

}  // namespace z4c

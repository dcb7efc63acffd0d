// The host-side cutting of the derivative pass's scratch as a small C library.
#include "../../gr-athena_b200/csrc/z4c_pieces.h"

extern "C" long long pc_doubles(long long vertices, int components) {
  return z4c::dv_doubles(vertices, components);
}

// The pieces of for_deriv_chunks as rows {block, blocks, plane, planes};
// returns their number (room: rows that fit in out).
extern "C" int pc_chunks(const int nx[3], int nblk, int components, long long cap, int* out,
                         int room) {
  int n = 0;
  z4c::for_deriv_chunks(nx, nblk, components, cap, [&](int b, int nb, int ks, int nk) {
    if (n < room) {
      const int row[4] = {b, nb, ks, nk};
      for (int q = 0; q < 4; ++q) out[4 * n + q] = row[q];
    }
    ++n;
  });
  return n;
}

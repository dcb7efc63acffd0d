// The host-side cutting of the derivative pass's scratch as a small C library.
#include "../../gr-athena_b200/csrc/z4c_pieces.h"

extern "C" long long pc_doubles(long long vertices, int components) {
  return z4c::dv_doubles(vertices, components);
}

extern "C" long long pc_share(long long cap, int nblocks) { return z4c::dv_share(cap, nblocks); }

// The pieces of for_deriv_chunks as rows {block, blocks, plane, planes,
// scratch}; returns their number (room: rows that fit in out).
extern "C" int pc_chunks(const int nx[3], int block0, int nblk, int components, long long share,
                         long long* out, int room) {
  int n = 0;
  z4c::for_deriv_chunks(nx, block0, nblk, components, share,
                        [&](int b, int nb, int ks, int nk, int64_t at) {
                          if (n < room) {
                            const long long row[5] = {b, nb, ks, nk, at};
                            for (int q = 0; q < 5; ++q) out[5 * n + q] = row[q];
                          }
                          ++n;
                        });
  return n;
}

extern "C" long long pc_context_share(long long parts, long long whole, int nblocks) {
  return z4c::dv_context_share(parts, whole, nblocks);
}

extern "C" long long pc_con_share(long long npts, long long plane, int nc, int nblocks) {
  return z4c::dv_con_share(npts, plane, nc, nblocks);
}

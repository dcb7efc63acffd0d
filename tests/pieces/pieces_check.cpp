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

// {rhs, con} of the least and of the best shares.
extern "C" void pc_shares(long long parts, long long whole, long long npts, long long plane,
                          int nc, int nblocks, long long least[2], long long best[2]) {
  const z4c::DvShares a = z4c::dv_least_shares(parts, plane, nc);
  const z4c::DvShares b = z4c::dv_best_shares(a, whole, npts, nc, nblocks);
  least[0] = a.rhs;
  least[1] = a.con;
  best[0] = b.rhs;
  best[1] = b.con;
}

// dv_reserve on a device with so many doubles free: whether it succeeded, the
// shares and what was allocated.
extern "C" int pc_reserve(const long long least[2], const long long best[2], int nblocks,
                          long long room, long long got[2], long long* allocated) {
  z4c::DvShares s{};
  *allocated = 0;
  const bool ok = z4c::dv_reserve(
      z4c::DvShares{best[0], best[1]}, z4c::DvShares{least[0], least[1]}, nblocks,
      [&](int64_t n) {
        if (n > room) return false;
        *allocated += n;
        return true;
      },
      &s);
  got[0] = s.rhs;
  got[1] = s.con;
  return ok;
}

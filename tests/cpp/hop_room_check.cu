// Host check of the sizes a spin-resolved product runs with (edgpu_kernels.h): every item of every split that
// edgpu_spmv may cut a sector into holds at most as many up hops as its shared memory has room for.  All sectors of
// impurities with one orbital (star) and three orbitals of 5 to 20 sites, 1 to 64 vectors; hops counted from the basis.
// Prints the first item that does not fit and exits non-zero.  Built and run by tests/test_hop_room_cpu.py (host only).
#include <algorithm>
#include <cstdio>
#include <vector>
#include "../../edlib_gb300/csrc/edgpu_kernels.h"

using namespace edgpu;

int main() {
  long long items = 0, straddling = 0;
  for (int norb : {1, 3})
    for (int ns = 5; ns <= 20; ++ns) {
      for (int nup = 0; nup <= ns; ++nup) {
        // prefix sums of the hops per up row, rows by ascending positions of their occupied bits
        std::vector<int> rp{0}, pos(nup);
        for (int q = 0; q < nup; ++q) pos[q] = q;
        int kmax = 0;
        for (bool more = true; more;) {
          unsigned mask = 0;
          for (int p : pos) mask |= 1u << p;
          int n = 0;
          for (int b = norb; b < ns; ++b) {  // bath b belongs to orbital (b - norb) mod norb; orbital m is bit ns - 1 - m
            const unsigned o = mask >> (ns - 1 - (b - norb) % norb) & 1, k = mask >> (ns - 1 - b) & 1;
            n += o != k;
          }
          rp.push_back(rp.back() + n);
          kmax = std::max(kmax, n);
          int q = nup - 1;
          while (q >= 0 && pos[q] == ns - nup + q) --q;
          more = q >= 0;
          if (more)
            for (++pos[q]; ++q < nup;) pos[q] = pos[q - 1] + 1;
        }
        const int up_rows = (int)rp.size() - 1;
        if (up_rows != binom_at_host(ns, nup)) return 2;
        for (int ndn = 0; ndn <= ns; ++ndn) {
          const int dn_rows = (int)binom_at_host(ns, ndn);
          if (dn_rows < kSrsLongRow || dn_rows >= kSrsVeryLong) continue;  // tiles only
          const int rows = srs_item_rows(up_rows, dn_rows), n = (up_rows + rows - 1) / rows;
          const int room = item_hop_room(rows, dn_rows, kmax);
          for (int nvec : {1, 2, 3, 4, 5, 7, 8, 12, 16, 24, 32, 64}) {
            const int r = vec_item_rows(rows, up_rows, dn_rows, n, nvec);
            straddling += r < rows && rows % r != 0;
            for (int u0 = 0; u0 < up_rows; u0 += r, ++items) {
              const int hops = rp[std::min(up_rows, u0 + r)] - rp[u0];
              if (r < 1 || r > rows || hops > room) {
                std::printf("%d orbitals, %d sites, sector (%d,%d), %d vectors: rows %d..%d of %d (items of %d, the sector's of %d) "
                            "hold %d hops, room for %d\n", norb, ns, nup, ndn, nvec, u0, u0 + r, up_rows, r, rows, hops, room);
                return 1;
              }
            }
          }
        }
      }
    }
  std::printf("%lld items; %lld splits across the sector's own items\n", items, straddling);
  return straddling > 0 ? 0 : 3;
}

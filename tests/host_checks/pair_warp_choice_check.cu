// Host-side check of the warp-per-unit pair form's choice of column orbitals
// (pw::column_orbitals), compiled by nvcc and run on the CPU: every (L, N) from
// 10 orbitals on has a tiling, whose row starts take at most 4 MiB and whose
// unit list is that of the tiling; a space too large for a neighbour table (2^23
// hops) gets the tiling that the units per tile row ask for alone.
#include <cstdio>

#include "../../doci_gb300/csrc/pair_warp_index.cuh"

constexpr int BC = 35;
static unsigned long long binom(unsigned n, unsigned k) {
  if (k > n) return 0;
  unsigned long long r = 1;
  for (unsigned d = 1; d <= k; ++d) r = r * (n - k + d) / d;
  return r;
}

int main() {
  std::vector<uint32_t> B(33 * BC, 0);
  for (int n = 0; n <= 32; ++n)
    for (int k = 0; k < BC; ++k) B[n * BC + k] = static_cast<uint32_t>(binom(n, k));
  const uint32_t slots = 4 * 152;
  int bad = 0, shapes = 0;
  for (int L = 10; L <= 32; ++L)
    for (int N = 1; N <= L; ++N, ++shapes) {
      doci::pw::Groups g;
      const int P = doci::pw::column_orbitals(L, N, slots, B.data(), BC, &g);
      bool ok = (P == 8 || P == 10 || P == 12) && L - P >= 2 && (4u << (L - P)) <= (4u << 20);
      const doci::pw::Groups want = doci::pw::groups(P, L - P, N, B.data(), BC);
      ok = ok && g.n == want.n && g.first[g.n] == want.first[want.n];
      if (binom(L, N) * N * (L - N) > (1u << 23)) {
        int units = 0;
        for (int p : {12, 10, 8}) {
          if (L - p < 2) continue;
          units = p;
          const doci::pw::Groups h = doci::pw::groups(p, L - p, N, B.data(), BC);
          if (h.first[h.n] / 4.0 >= (p == 12 ? 4.0 : 1.5) * slots) break;
        }
        ok = ok && P == units;
      }
      if (!ok) {
        ++bad;
        std::printf("L=%d N=%d P=%d\n", L, N, P);
      }
    }
  std::printf("shapes=%d bad=%d\n", shapes, bad);
  return bad ? 1 : 0;
}

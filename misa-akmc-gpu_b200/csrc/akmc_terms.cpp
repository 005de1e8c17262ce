// akmc_terms.cpp -- which lanes form the dE terms that a vacancy's 8 jumps share.
#include <algorithm>
#include <vector>

#include "akmc_model.h"

namespace akmc {

// The lanes that form the dE terms of a vacancy's 8 jumps (Geometry::foot_*), in half lattice
// constants around the vacancy: the same for both x parities but for the site ids' own offsets.
void build_terms(Geometry& g, int nsh) {
  struct Site {
    int h[3], hs;
    int ht[8], n;   // the terms: shells around a target
    int first;      // index of the first one
  };
  auto shell = [&](const int* a, const int* b) {
    const int d[3] = {a[0] - b[0], a[1] - b[1], a[2] - b[2]};
    const int d2 = d[0] * d[0] + d[1] * d[1] + d[2] * d[2];
    return d2 == 0 ? kSelf : shell_code(d2, nsh);
  };
  const int origin[3] = {0, 0, 0};
  int dir[8][3];
  for (int b = 0; b < 8; ++b) {
    dir[b][0] = (b & 4) ? 1 : -1;
    dir[b][1] = (b & 2) ? 1 : -1;
    dir[b][2] = (b & 1) ? 1 : -1;
  }
  std::vector<Site> sites;
  int16_t at_h[11][11][11] = {};  // position -> site
  int terms = 0;
  for (int x = -5; x <= 5; ++x)
    for (int y = -5; y <= 5; ++y)
      for (int z = -5; z <= 5; ++z) {
        if (((x ^ y) & 1) || ((x ^ z) & 1) || (!x && !y && !z)) continue;  // a BCC site, not the vacancy
        Site s{{x, y, z}, 0, {}, 0, 0};
        s.hs = shell(s.h, origin);
        for (int b = 0; b < 8; ++b) {
          const int ht = shell(s.h, dir[b]);
          if (ht == kSelf || ht == s.hs) continue;
          bool seen = false;
          for (int i = 0; i < s.n; ++i) seen = seen || s.ht[i] == ht;
          if (!seen) s.ht[s.n++] = ht;
        }
        if (s.n == 0) continue;
        at_h[x + 5][y + 5][z + 5] = static_cast<int16_t>(sites.size());
        s.first = terms;
        terms += s.n;
        sites.push_back(s);
      }
  // groups of lanes, widest first, each inside one warp
  std::vector<size_t> order(sites.size());
  for (size_t i = 0; i < order.size(); ++i) order[i] = i;
  std::stable_sort(order.begin(), order.end(), [&](size_t a, size_t b) { return sites[a].n / 2 > sites[b].n / 2; });
  int used[kFootSlots / 32] = {};
  for (int i = 0; i < kFootSlots; ++i) {
    g.foot_out[i] = kFootNone | kFootNone << 10 | (i & 31) << 20;
    g.foot_site[0][i] = g.foot_site[1][i] = pack_entry(0, 0, 0, 0, 0);
  }
  auto place = [&](int lanes) {
    for (int w = 0; w < kFootSlots / 32; ++w)
      if (used[w] + lanes <= 32) {
        used[w] += lanes;
        return 32 * w + used[w] - lanes;
      }
    return -1;
  };
  auto put_site = [&](int slot, const int* h) {
    for (int p = 0; p < 2; ++p) {
      const int odd = (h[0] & 1) ? (p ? -1 : 1) : 0;  // x parity of the site minus the vacancy's
      g.foot_site[p][slot] = pack_entry(h[0], (h[1] - odd) / 2, (h[2] - odd) / 2, 0, 0);
    }
    for (int b = 0; b < 8; ++b) {  // jump b brought the vacancy here from -dir[b]
      const int from[3] = {-dir[b][0], -dir[b][1], -dir[b][2]};
      const int ss = shell(h, from), st = shell(h, origin);
      g.foot_refresh[b][slot] = ss == st ? 0 : static_cast<uint8_t>(ss * 8 + st);
    }
  };
  for (size_t k : order) {
    const Site& s = sites[k];
    const int lanes = s.n / 2 + 1, at = place(lanes);
    for (int i = 0; i < lanes; ++i) {
      const int slot = at + i;
      put_site(slot, s.h);
      // evaluation e of the group (0: F(rho_j); 1..n: the terms), two to a lane
      int out[2] = {kFootNone, kFootNone}, sh[2] = {0, 0};
      for (int q = 0; q < 2; ++q) {
        const int e = 2 * i + q;
        if (e == 0 || e > s.n) continue;
        out[q] = s.first + e - 1;
        sh[q] = s.hs * 8 + s.ht[e - 1];
      }
      int raw = 0;
      if (i == 0)
        for (int b = 0; b < 8; ++b)
          if (s.h[0] == dir[b][0] && s.h[1] == dir[b][1] && s.h[2] == dir[b][2]) raw = 2 + b;
      g.foot_out[slot] = out[0] | out[1] << 10 | (at & 31) << 20 | raw << 25;
      g.foot_shells[slot] = sh[0] | sh[1] << 8;
    }
  }
  {  // the vacancy's own site: F(rho_s - f_X(1)), shells (0, 1)
    const int slot = place(1);
    put_site(slot, origin);
    g.foot_out[slot] = kFootNone | kFootNone << 10 | (slot & 31) << 20 | 1 << 25;
    g.foot_shells[slot] = 1;
  }
  for (int p = 0; p < 2; ++p)
    for (int b = 0; b < 8; ++b)
      for (int i = 0; i < kJumpN; ++i) {
        const int32_t w = g.jump[p][b][i];
        const int odd = (unpack_dx(w) & 1) ? (p ? -1 : 1) : 0;
        const int h[3] = {unpack_dx(w), 2 * unpack_dy(w) + odd, 2 * unpack_dz(w) + odd};
        const Site& s = sites[static_cast<size_t>(at_h[h[0] + 5][h[1] + 5][h[2] + 5])];
        for (int t = 0; t < s.n; ++t)
          if (s.ht[t] == unpack_sh_t(w)) g.term[p][b][i] = static_cast<uint16_t>(s.first + t);
      }
}

}  // namespace akmc

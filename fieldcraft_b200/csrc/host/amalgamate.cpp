#include "amalgamate.hpp"

#include <algorithm>

namespace fc {

bool merge_pays(int64_t w_child, int64_t w_parent, double zeros, double entries) {
  const int64_t w = w_child + w_parent;
  const double share = zeros / entries;
  return w <= 4 || (w <= 16 && share < 0.8) || (w <= 48 && share < 0.1) || share < 0.05 || zeros < MERGE_ZEROS;
}

Amalgamated amalgamate(const Symbolic &sym, bool merge) {
  Amalgamated out;
  const int64_t n = sym.n, ns = sym.ns;
  std::vector<int64_t> w(ns), m(ns), into(ns, NONE);
  std::vector<double> zeros(ns, 0.0);
  std::vector<int64_t> head(ns, NONE), next(ns, NONE);  // the children left, as lists
  for (int64_t s = 0; s < ns; ++s) w[s] = sym.width(s), m[s] = sym.height(s);
  if (merge) {
    std::vector<int64_t> kids;
    for (int64_t p = 0; p < ns; ++p) {
      // every supernode before p is as it will stay but for being merged upwards; p's children by
      // falling height (the ones whose rows are most of p's first), lowest index first
      kids.clear();
      for (int64_t c = head[p]; c != NONE; c = next[c]) kids.push_back(c);
      std::sort(kids.begin(), kids.end(), [&](int64_t a, int64_t b) { return m[a] != m[b] ? m[a] > m[b] : a < b; });
      head[p] = NONE;
      auto keep = [&](int64_t c) { next[c] = head[p], head[p] = c; };
      for (int64_t c : kids) {
        const int64_t wm = w[c] + w[p], mm = m[p] + w[c];
        // the child's columns take the parent's rows that they lack
        const double z = zeros[c] + zeros[p] + (double)w[c] * (double)(m[p] - (m[c] - w[c]));
        const double entries = (double)wm * (double)mm - 0.5 * (double)wm * (double)(wm - 1);
        if (wm * mm <= INT32_MAX && merge_pays(w[c], w[p], z, entries)) {
          w[p] = wm, m[p] = mm, zeros[p] = z, into[c] = p;
          for (int64_t g = head[c], after; g != NONE; g = after) {
            after = next[g];
            keep(g);
          }
        } else {
          keep(c);
        }
      }
      if (sym.sparent[p] != NONE) {
        const int64_t q = sym.sparent[p];
        next[p] = head[q], head[q] = p;
      }
    }
  }
  // each supernode's last ancestor it was merged into names its group; groups in that order
  std::vector<int64_t> top(ns), id(ns, NONE);
  for (int64_t s = ns - 1; s >= 0; --s) top[s] = into[s] == NONE ? s : top[into[s]];
  for (int64_t s = 0; s < ns; ++s)
    if (top[s] == s) id[s] = out.ns++;
  out.first.assign(out.ns + 1, 0);
  for (int64_t s = 0; s < ns; ++s) out.first[id[top[s]] + 1] += sym.width(s);
  for (int64_t g = 0; g < out.ns; ++g) out.first[g + 1] += out.first[g];
  out.place.resize(n);
  out.column.resize(n);
  {
    std::vector<int64_t> at(out.first.begin(), out.first.end() - (out.ns ? 1 : 0));
    for (int64_t s = 0; s < ns; ++s)  // a group's members in order: descendants before ancestors
      for (int64_t j = sym.first[s]; j < sym.first[s + 1]; ++j) {
        const int64_t to = at[id[top[s]]]++;
        out.place[j] = (int32_t)to;
        out.column[to] = (int32_t)j;
      }
  }
  // a group's rows: its columns, then its last member's rows below
  out.rptr.assign(out.ns + 1, 0);
  out.sparent.assign(out.ns, NONE);
  for (int64_t s = 0; s < ns; ++s)
    if (top[s] == s) out.rptr[id[s] + 1] = out.width(id[s]) + sym.height(s) - sym.width(s);
  for (int64_t g = 0; g < out.ns; ++g) out.rptr[g + 1] += out.rptr[g];
  out.rows.resize(out.ns ? out.rptr[out.ns] : 0);
  for (int64_t s = 0; s < ns; ++s) {
    if (top[s] != s) continue;
    const int64_t g = id[s], f = out.first[g], wg = out.width(g);
    int32_t *r = out.rows.data() + out.rptr[g];
    for (int64_t c = 0; c < wg; ++c) r[c] = (int32_t)(f + c);
    const int32_t *below = sym.rows.data() + sym.rptr[s] + sym.width(s);
    const int64_t u = sym.height(s) - sym.width(s);
    for (int64_t i = 0; i < u; ++i) r[wg + i] = out.place[below[i]];
    std::sort(r + wg, r + wg + u);
    if (sym.sparent[s] != NONE) out.sparent[g] = id[top[sym.sparent[s]]];
  }
  return out;
}

}  // namespace fc

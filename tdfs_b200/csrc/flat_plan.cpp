// flat_plan.cpp -- how the flat kernel (flat.cu) runs a compiled plan.
//
// The count is a sum over the plan's DFS leaves (src/gpu_match.cu:951-1080).
// The last t vertices need no enumeration when every backward neighbour of
// each lies at or above some level s = k-1-t: below a node at level s their
// candidate sets are fixed, and the leaves are tuples of distinct vertices
// drawn one from each set.  Their number follows from the sizes of the sets
// and of their intersections, each of which is again a candidate set: the
// union of the backward neighbours under the union of the conditions.
#include <cstring>

#include "common.h"

namespace tdfs {

namespace {

FlatStep step_of(const DevPlan &d, int i, int limit) {
  FlatStep st;
  std::memset(&st, 0, sizeof st);
  st.nbn = (uint8_t)d.nbn[i];
  for (int t = 0; t < d.nbn[i]; ++t) st.bn[t] = (uint8_t)d.bn[i][t];
  st.label = (uint8_t)d.label[i];
  const unsigned mask = (2u << limit) - 1;  // conditions on phi(0..limit)
  st.larger = (uint8_t)(d.larger[i] & mask);
  st.less = (uint8_t)(d.less[i] & mask);
  st.neq = (uint8_t)(d.neq[i] & mask);
  if (d.labeled) {
    // vertices of different labels never coincide
    for (int j = 0; j <= limit; ++j)
      if (d.label[j] != d.label[i]) st.neq &= (uint8_t)~(1u << j);
  }
  return st;
}

bool same_set(const FlatStep &a, const FlatStep &b) { return std::memcmp(&a, &b, sizeof a) == 0; }

FlatStep both(const FlatStep &a, const FlatStep &b) {
  FlatStep c = a;
  for (int t = 0; t < b.nbn; ++t) {
    bool have = false;
    for (int u = 0; u < c.nbn; ++u) have |= c.bn[u] == b.bn[t];
    if (!have) c.bn[c.nbn++] = b.bn[t];
  }
  // backward neighbours in increasing order, so equal sets compare equal
  for (int x = 1; x < c.nbn; ++x)
    for (int y = x; y > 0 && c.bn[y - 1] > c.bn[y]; --y) {
      const uint8_t v = c.bn[y];
      c.bn[y] = c.bn[y - 1];
      c.bn[y - 1] = v;
    }
  c.larger |= b.larger;
  c.less |= b.less;
  c.neq |= b.neq;
  return c;
}

// The tail of t vertices: 0 = none, else 1 + form.
int tail_form(const DevPlan &d, int t) {
  const int k = d.k, s = k - 1 - t;
  bool ordered = false, unordered = false;
  for (int j = s + 1; j < k; ++j) {
    for (int u = 0; u < d.nbn[j]; ++u)
      if (d.bn[j][u] > s) return 0;
    for (int i = s + 1; i < j; ++i) {
      if ((d.larger[j] | d.less[j]) >> i & 1) ordered = true;
      else unordered = true;
    }
  }
  if (!ordered) return 1;
  if (unordered) return 0;
  // all pairs ordered: a total order (any tournament of conditions that a
  // compiled plan carries is acyclic); the t-subsets of one set
  const FlatStep a = step_of(d, s + 1, s);
  for (int j = s + 2; j < k; ++j)
    if (!same_set(a, step_of(d, j, s))) return 0;
  return 2;
}

}  // namespace

bool flat_plan(const DevPlan &d, FlatPlan *out) {
  FlatPlan f;
  std::memset(&f, 0, sizeof f);
  const int k = d.k;
  f.k = k;
  f.orient = d.orient;
  for (int i = 0; i < 3; ++i) f.deg[i] = d.deg[i];
  f.label[0] = d.label[0];
  f.label[1] = d.label[1];
  int t = 1, form = 0;
  for (int c = 3; c >= 2; --c) {
    if (k - 1 - c < 1) continue;
    const int r = tail_form(d, c);
    if (r) {
      t = c;
      form = r - 1;
      break;
    }
  }
  const int s = k - 1 - t;
  // A last vertex that does not hang on its parent has one set for all its
  // siblings, which the tail form counts without visiting them; without that
  // form enumerating them would cost a level, so such plans stay with the DFS
  // kernel.
  if (t == 1 && k >= 4) {
    bool parent = false;
    for (int u = 0; u < d.nbn[k - 1]; ++u) parent |= d.bn[k - 1][u] == k - 2;
    if (!parent) return false;
  }
  f.s = (uint8_t)s;
  f.t = (uint8_t)t;
  f.form = (uint8_t)form;
  auto with_reuse = [&](FlatStep st, int i) {
    const int dep = d.dep[i];
    if (dep >= 2 && dep < i && d.nsh[i] <= 3) {
      st.dep = (uint8_t)dep;
      st.nsh = (uint8_t)d.nsh[i];
      for (int u = 0; u < d.nsh[i]; ++u) st.bnsh[u] = (uint8_t)d.bnsh[i][u];
    }
    return st;
  };
  for (int i = 2; i <= s; ++i) f.step[i - 2] = with_reuse(step_of(d, i, i - 1), i);
  std::memset(f.term_of, kNoTerm, sizeof f.term_of);
  auto add = [&](const FlatStep &st) {
    for (int u = 0; u < f.nterm; ++u)
      if (same_set(f.term[u], st)) return (uint8_t)u;
    f.term[f.nterm] = st;
    return f.nterm++;
  };
  if (t == 1) {
    f.term_of[1] = add(with_reuse(step_of(d, k - 1, s), k - 1));
  } else if (form == 1) {
    f.term_of[1] = add(step_of(d, s + 1, s));
  } else {
    for (int m = 1; m < 1 << t; ++m) {
      FlatStep st;
      bool first = true, meet = true;
      for (int u = 0; u < t; ++u) {
        if (!(m >> u & 1)) continue;
        const FlatStep a = step_of(d, s + 1 + u, s);
        if (!first && d.labeled && a.label != st.label) meet = false;  // different labels: empty
        st = first ? a : both(st, a);
        first = false;
      }
      if (meet) f.term_of[m] = add(st);
    }
  }
  for (int i = 0; i < s - 1; ++i) f.reuse2 |= f.step[i].dep == 2;
  for (int u = 0; u < f.nterm; ++u) f.reuse2 |= f.term[u].dep == 2;
  *out = f;
  return true;
}

}  // namespace tdfs

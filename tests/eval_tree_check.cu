// Host check of the evaluation schedule: for random trees and options, the
// value along the schedule (centre, axis orders, absorbed kids) equals the
// contraction from the stored root, and the schedule keeps its own rules.
#include <cstdlib>
#include <random>

#include "eval_tree.cuh"

using namespace tnfa;
static std::mt19937_64 rng(7);
static int ri(int a, int b) { return a + (int)(rng() % (uint64_t)(b - a + 1)); }
#define REQUIRE(c)                                             \
  do {                                                         \
    if (!(c)) {                                                \
      std::printf("failed: %s (line %d)\n", #c, __LINE__);     \
      std::exit(1);                                            \
    }                                                          \
  } while (0)

struct Net {
  Topo T;
  std::vector<std::vector<double>> t;  // [site][parent][children]
  std::vector<int> s;                  // a site value per vertex
};

static std::vector<double> up_message(const Net& n, int v) {  // toward the stored parent
  const auto& ch = n.T.children[v];
  std::vector<double> cur(n.t[v].begin() + (size_t)n.s[v] * (n.t[v].size() / n.T.site_dim[v]),
                          n.t[v].begin() + (size_t)(n.s[v] + 1) * (n.t[v].size() / n.T.site_dim[v]));
  for (size_t i = ch.size(); i-- > 0;) {  // the last child is the fastest axis
    const std::vector<double> m = up_message(n, ch[i]);
    std::vector<double> next(cur.size() / m.size(), 0.0);
    for (size_t k = 0; k < cur.size(); ++k) next[k / m.size()] += cur[k] * m[k % m.size()];
    cur = next;
  }
  return cur;
}

static std::vector<double> message(const Net& n, const EvalTree& E, int v) {  // along the schedule
  const EvalVertex& e = E.v[v];
  std::vector<int> shape{n.T.site_dim[v], n.T.link[v]};
  for (int c : n.T.children[v]) shape.push_back(n.T.link[c]);
  std::vector<int64_t> str(shape.size(), 1);
  for (size_t a = shape.size() - 1; a-- > 0;) str[a] = str[a + 1] * shape[a + 1];
  REQUIRE(e.axes.size() == shape.size() && e.axes[0] == 0);
  // the slice of this site value in the order used
  std::vector<double> cur;
  std::vector<int> ix(shape.size(), 0);
  for (;;) {
    int64_t o = (int64_t)n.s[v] * str[0];
    for (size_t a = 1; a < e.axes.size(); ++a) o += ix[a] * str[e.axes[a]];
    cur.push_back(n.t[v][o]);
    size_t a = e.axes.size() - 1;
    while (a > 0 && ++ix[a] == shape[e.axes[a]]) ix[a--] = 0;
    if (a == 0) break;
  }
  for (size_t i = e.kids.size(); i-- > 0;) {
    const std::vector<double> m = message(n, E, e.kids[i]);
    std::vector<double> next(cur.size() / m.size(), 0.0);
    for (size_t k = 0; k < cur.size(); ++k) next[k / m.size()] += cur[k] * m[k % m.size()];
    cur = next;
  }
  REQUIRE((int)cur.size() == e.chi);
  return cur;
}

static double combos(const Net& n, const EvalTree& E, int v) {
  double c = n.T.site_dim[v];
  for (int k : E.v[v].kids) c *= combos(n, E, k);
  return c;
}

int main() {
  int moved = 0, tabled = 0, absorbed = 0, tensor = 0, other_centre = 0;
  for (int trial = 0; trial < 4000; ++trial) {
    Net n;
    Topo& T = n.T;
    const int V = T.V = ri(1, 12), shape = ri(0, 3);
    T.children.resize(V);
    for (int v = 0; v < V; ++v) {
      const int p = v == 0 ? -1 : shape == 0 ? v - 1 : shape == 1 ? (v - 1) / 2 : ri(0, 9) == 0 ? -1 : ri(std::max(0, v - 4), v - 1);
      T.parent.push_back(p);
      T.link.push_back(p < 0 ? 1 : ri(1, 3));
      T.site_dim.push_back(ri(0, 6) == 0 ? 1 : ri(2, 3));
      if (p >= 0) T.children[p].push_back(v);
    }
    for (int v = 0; v < V; ++v) {
      n.t.emplace_back(T.size(v));
      for (double& x : n.t.back()) x = (double)ri(-8, 8) / 4;
      n.s.push_back(ri(0, T.site_dim[v] - 1));
    }
    EvalTreeOptions o;
    o.rule = ri(0, 1) ? CentreRule::ANY_EDGE : ri(0, 1) ? CentreRule::ROOT_EDGE : CentreRule::ROOT;
    o.points = std::pow(10.0, ri(0, 7));
    o.table_rows = ri(0, 3) ? o.points : ri(0, 50);
    if (ri(0, 3) == 0) o.table_elems = ri(1, 400);
    o.absorb = ri(0, 4) != 0;
    o.absorb_points = ri(0, 1);
    o.balance = ri(0, 1);
    if (ri(0, 3) == 0) o.table_kids = ri(1, 2);
    if (ri(0, 2) == 0)
      for (int v = 0; v < V; ++v) o.tensor_ok.push_back(T.children[v].size() == 2 && ri(0, 1));
    const EvalTree E = EvalTreeBuilder(T, o).build();
    REQUIRE((int)E.order.size() == V && E.comps.size() == T.roots().size());
    std::vector<int> at(V, -1);
    for (int i = 0; i < V; ++i) {
      REQUIRE(at[E.order[i]] < 0);
      at[E.order[i]] = i;
    }
    for (int v = 0; v < V; ++v) {
      const EvalVertex& e = E.v[v];
      for (int k : e.kids) REQUIRE(at[k] < at[v] && E.v[k].up == v);
      const double c = combos(n, E, v);
      if (e.tabled) {
        REQUIRE((double)e.N == c && (e.leaf || c <= o.table_rows));
        if (o.table_kids < (1 << 30)) REQUIRE((int)e.kids.size() <= o.table_kids);
      }
      if (e.absorb) {
        REQUIRE(e.kids.size() >= 2 && E.v[e.kids.back()].tabled && !e.tensor);
        ++absorbed;
      }
      if (e.tensor) REQUIRE(!e.moved && e.up == T.parent[v]);
      moved += e.moved;
      tabled += e.tabled && !e.leaf;
      tensor += e.tensor;
    }
    double ref = 1.0, got = 1.0;
    for (int r : T.roots()) ref *= up_message(n, r)[0];
    for (const auto& c : E.comps) {
      if (o.rule == CentreRule::ROOT) REQUIRE(c.b < 0 && T.parent[c.a] < 0);
      if (o.rule == CentreRule::ROOT_EDGE && c.b >= 0) REQUIRE(T.parent[c.a] < 0);
      other_centre += c.b >= 0 && T.parent[c.a] >= 0;
      const std::vector<double> a = message(n, E, c.a);
      double x = 0.0;
      if (c.b < 0) {
        x = a[0];
      } else {
        const std::vector<double> b = message(n, E, c.b);
        REQUIRE(a.size() == b.size());
        for (size_t k = 0; k < a.size(); ++k) x += a[k] * b[k];
      }
      got *= x;
    }
    REQUIRE(std::fabs(got - ref) <= 1e-9 * std::max(1.0, std::fabs(ref)));
  }
  REQUIRE(moved && tabled && absorbed && tensor && other_centre);
  std::printf("ok\n");
}

// Host-side schedule of a batched evaluation: which messages are formed once
// per combination of digits, and toward which centre they run.
//
// The message of a vertex toward the centre depends on the digits below it
// only, so it takes at most N = prod(site dims below) different values.  When
// N is no more than the number of points, the message is a table with one row
// per digit combination (the points gather from it by an integer code);
// otherwise it is one row per point.  The centre may be any edge (a, b): the
// value is the dot product of the two messages that meet there, so a path or
// a comb evaluated at many points splits into two tables of about half the
// digits each.
#pragma once
#include <algorithm>
#include <cmath>
#include <vector>

#include "common.cuh"

namespace tnfa {

// Which centres are allowed: every edge; the edges of the stored root (its
// tensor alone is read in another axis order); the stored root itself.
enum class CentreRule { ANY_EDGE, ROOT_EDGE, ROOT };

struct EvalVertex {
  int up = -1;              // neighbour toward the centre, -1 at a vertex centre
  int chi = 1;              // bond to it
  std::vector<int> kids;    // the other neighbours, in the axis order used; the absorbed one last
  std::vector<int> axes;    // stored axes in the order used: sites, up, kids
  bool moved = false;       // that order is not the stored one
  bool leaf = false;        // no kids: the message is the tensor slice itself
  bool tabled = false;      // one row per digit combination
  bool absorb = false;      // the last kid's table is contracted into the tensor first
  bool tensor = false;      // goes to the tensor-core kernel of this precision
  double W = 1.0;           // product of all bonds of the vertex
  int64_t N = 1;            // rows when tabled
};

struct EvalTree {
  struct Comp {
    int a = -1, b = -1;  // the centre edge, or the centre vertex with b = -1
  };
  std::vector<EvalVertex> v;
  std::vector<int> order;  // kids before the vertices that read them
  std::vector<Comp> comps;
};

struct EvalTreeOptions {
  CentreRule rule = CentreRule::ANY_EDGE;
  double points = 1;
  double table_rows = 1;        // a message with at most this many combinations is a table
  double table_elems = 1e18;    // bound on the elements of one absorbed tensor
  bool absorb = true;
  bool absorb_points = true;    // also into the tensors of vertices without a table
  int table_kids = 1 << 30;     // a vertex with more kids has no table; with two, one is always absorbed
  bool balance = false;         // choose the centre by the costlier side, not the sum
  std::vector<char> tensor_ok;  // vertices the tensor-core kernel takes in the stored axis order
  double tensor_speed = 40.0;   // its rate over the CUDA cores' (measured: 46 for MIXED)
};

class EvalTreeBuilder {
 public:
  EvalTreeBuilder(const Topo& T, const EvalTreeOptions& o) : T_(T), o_(o) {}

  EvalTree build() {
    const int V = T_.V;
    tree_.v.resize(V);
    nb_.assign(V, {});
    W_.assign(V, 1.0);
    for (int v = 0; v < V; ++v) {
      if (T_.parent[v] >= 0) nb_[v].push_back(T_.parent[v]);
      W_[v] = T_.link[v];
      for (int c : T_.children[v]) {
        nb_[v].push_back(c);
        W_[v] *= T_.link[c];
      }
    }
    // combinations of the digits below (down) and above (up) every parent edge
    down_.assign(V, 1.0);
    up_.assign(V, 1.0);
    for (int v = V - 1; v >= 0; --v) {
      down_[v] = cap(down_[v] * T_.site_dim[v]);
      if (T_.parent[v] >= 0) down_[T_.parent[v]] = cap(down_[T_.parent[v]] * down_[v]);
    }
    for (int v = 0; v < V; ++v)
      for (int c : T_.children[v]) {
        double n = T_.site_dim[v] * (T_.parent[v] >= 0 ? up_[v] : 1.0);
        for (int d : T_.children[v])
          if (d != c) n = cap(n * down_[d]);
        up_[c] = n;
      }
    // cost of all messages of the subtree below v toward its parent, and of
    // everything else toward v
    std::vector<double> D(V, 0.0), U(V, 0.0);
    for (int v = V - 1; v >= 0; --v) {
      D[v] += cost(v, T_.parent[v], nullptr);
      if (T_.parent[v] >= 0) D[T_.parent[v]] += D[v];
    }
    std::vector<int> root(V), a(V, -1), b(V, -1);
    std::vector<double> best(V, INFINITY);
    for (int v = 0; v < V; ++v) root[v] = T_.parent[v] < 0 ? v : root[T_.parent[v]];
    for (int v = 0; v < V; ++v) {
      const int r = root[v], p = T_.parent[v];
      if (p < 0) {
        if (o_.rule == CentreRule::ROOT || nb_[v].empty()) best[r] = D[v], a[r] = v, b[r] = -1;
        continue;
      }
      double all = T_.parent[p] >= 0 ? U[p] : 0.0;
      for (int c : T_.children[p])
        if (c != v) all += D[c];
      U[v] = all + cost(p, v, nullptr);
      if (o_.rule == CentreRule::ROOT || (o_.rule == CentreRule::ROOT_EDGE && p != r)) continue;
      const double c = (o_.balance ? std::max(D[v], U[v]) : D[v] + U[v]) + o_.points * T_.link[v];
      if (c < best[r]) best[r] = c, a[r] = p, b[r] = v;
    }
    for (int v = 0; v < V; ++v)
      if (T_.parent[v] < 0) {
        tree_.comps.push_back({a[v], b[v]});
        orient(a[v], b[v]);
        if (b[v] >= 0) orient(b[v], a[v]);
      }
    return std::move(tree_);
  }

 private:
  static double cap(double x) { return std::min(x, 1e18); }
  double below(int v, int u) const {  // digit combinations behind the message v -> u
    if (u < 0) return down_[v];
    return u == T_.parent[v] ? down_[v] : up_[u];
  }
  int bond(int v, int u) const { return u < 0 ? 1 : u == T_.parent[v] ? T_.link[v] : T_.link[u]; }

  // Multiply-adds of the message v -> u; *absorb receives the kid whose table
  // is contracted into the tensor first (-1: none).
  double cost(int v, int u, int* absorb) const {
    if (absorb) *absorb = -1;
    int nk = 0;
    for (int w : nb_[v]) nk += w != u;
    if (nk == 0) return 0.0;
    const bool tab = is_table(v, u);
    const double rows = tab ? below(v, u) : o_.points;
    if (is_tensor(v, u)) return rows * W_[v] / o_.tensor_speed;
    const double direct = rows * W_[v];
    double best = direct;
    if (nk < 2 || !o_.absorb || (!tab && !o_.absorb_points)) return best;
    if (tab && o_.table_kids < nk + 1) best = INFINITY;
    for (int w : nb_[v]) {
      if (w == u) continue;
      if (!is_table(w, v)) continue;
      const double nw = below(w, v);
      if (nw > o_.table_rows) continue;
      const double groups = T_.site_dim[v] * nw, made = groups * W_[v];
      if (made > o_.table_elems && best < INFINITY) continue;
      // a group's last tile is padded to a few rows
      const double c = made + (rows + 4.0 * groups) * W_[v] / bond(w, v);
      if (c < best) {
        best = c;
        if (absorb) *absorb = w;
      }
    }
    return best;
  }
  // The message v -> u has a row per digit combination (a leaf always does).
  bool is_table(int v, int u) const {
    int nk = 0;
    for (int w : nb_[v]) nk += w != u;
    if (nk == 0) return true;
    if (below(v, u) > o_.table_rows || nk > o_.table_kids) return false;
    if (o_.table_kids < (1 << 30))
      for (int w : nb_[v])
        if (w != u && !is_table(w, v)) return false;
    return true;
  }
  bool is_tensor(int v, int u) const {
    return !o_.tensor_ok.empty() && o_.tensor_ok[v] && u == T_.parent[v];
  }

  // Orients the component part behind `v` toward `u` (depth first).
  void orient(int v0, int u0) {
    std::vector<std::pair<int, int>> todo{{v0, u0}}, seen;
    while (!todo.empty()) {
      const auto [v, u] = todo.back();
      todo.pop_back();
      seen.push_back({v, u});
      for (int w : nb_[v])
        if (w != u) todo.push_back({w, v});
    }
    for (size_t i = seen.size(); i-- > 0;) set(seen[i].first, seen[i].second);
  }

  void set(int v, int u) {
    EvalVertex& e = tree_.v[v];
    e.up = u;
    e.chi = bond(v, u);
    e.W = W_[v];
    int ab = -1;
    cost(v, u, &ab);
    for (int w : nb_[v])
      if (w != u && w != ab) e.kids.push_back(w);
    if (ab >= 0) e.kids.push_back(ab);
    e.absorb = ab >= 0;
    e.leaf = e.kids.empty();
    e.tensor = !e.leaf && is_tensor(v, u);
    const double n = below(v, u);
    e.tabled = is_table(v, u);
    e.N = e.tabled ? (int64_t)n : 0;
    auto axis = [&](int w) {  // stored axis of the bond to w
      if (w == T_.parent[v]) return 1;
      int k = 0;
      while (T_.children[v][k] != w) ++k;
      return 2 + k;
    };
    // a root's parent axis has dimension 1: it stays next to the sites
    e.axes.push_back(0);
    if (T_.parent[v] < 0) e.axes.push_back(1);
    if (u >= 0) e.axes.push_back(axis(u));
    for (int w : e.kids) e.axes.push_back(axis(w));
    for (size_t i = 0; i < e.axes.size(); ++i) e.moved |= e.axes[i] != (int)i;
    tree_.order.push_back(v);
  }

  const Topo& T_;
  const EvalTreeOptions& o_;
  EvalTree tree_;
  std::vector<std::vector<int>> nb_;
  std::vector<double> W_, down_, up_;
};

}  // namespace tnfa

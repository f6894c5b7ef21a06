// Host builder of the member-row tables (see mpsw_rows.h).
#include "mpsw_rows.h"

#include "mpsw_internal.h"
#include "mpsw_parts.h"

namespace mpsw {

// one(i) for 0 <= i < n over a few threads: null, or what the mesh lacks
template <class One>
static std::string side_by_side(int n, One &&one) {
  constexpr int kParts = 16;
  const char *bad[kParts] = {};
  in_turns(kParts, [&](int p) {
    const int end = (int)((long long)n * (p + 1) / kParts);
    for (int i = (int)((long long)n * p / kParts); i < end && !bad[p]; i++) bad[p] = one(i);
  });
  for (const char *b : bad)
    if (b) return b;
  return "";
}

std::string build_rows(const BuiltMesh &m, RowTabHost *t) {
  const int nC = m.nC, nE = m.nE, nV = m.nV;
  auto C = [&](int c, int k) { return (size_t)k * nC + c; };
  auto E = [&](int e, int k) { return (size_t)k * nE + e; };
  auto V = [&](int v, int k) { return (size_t)k * nV + v; };
  for (int c = 0; c < nC; c++)
    if (m.c_n[c] > 6) return "more than 6 edges on a cell";
  for (int e = 0; e < nE; e++)
    if (m.e_n[e] > 10) return "more than 10 edgesOnEdge";
  auto sign_v = [&](int v, int e) { return m.e_v2[e] == v ? 1.0 : -1.0; };  // circulation
  auto sign_c = [&](int c, int e) { return m.e_c1[e] == c ? 1.0 : -1.0; };  // divergence
  auto kite = [&](int v, int c, double *k) {  // false: c is not a cell of v
    for (int i = 0; i < VDEG; i++)
      if (m.v_c[V(v, i)] == c) {
        *k = m.v_k[V(v, i)];
        return true;
      }
    return false;
  };
  auto of_vertex = [&](int v, int e) {  // e is an edge of v, and v an end of e
    if (m.e_v1[e] != v && m.e_v2[e] != v) return false;
    for (int i = 0; i < VDEG; i++)
      if (m.v_es[V(v, i)] == e) return true;
    return false;
  };
  auto of_cell = [&](int c, int e) { return m.e_c1[e] == c || m.e_c2[e] == c; };
  const size_t S = (size_t)6 * nC;
  for (auto *x : {&t->c_nb, &t->c_sp, &t->c_va, &t->c_vb}) x->assign(S, 0);
  for (auto *x : {&t->c_g1, &t->c_g2, &t->c_g3, &t->c_n1, &t->c_n2, &t->c_m, &t->c_t, &t->c_q, &t->c_r, &t->c_ka,
                  &t->c_kb, &t->c_kk, &t->c_r2, &t->c_r3})
    x->assign(S, 0.0);
  t->c_ra.resize(nC);
  std::string bad = side_by_side(nC, [&](int c) -> const char * {
    const double area = m.c_area[c];
    t->c_ra[c] = 1.0 / area;
    for (int k = 0; k < m.c_n[c]; k++) {
      const size_t s = C(c, k);
      const int e = m.c_es[s];
      if (!of_cell(c, e) || m.e_c1[e] == m.e_c2[e]) return "an edge of a cell that does not list the cell";
      const int nb = m.e_c1[e] == c ? m.e_c2[e] : m.e_c1[e], a = m.e_v1[e], b = m.e_v2[e];
      double ka, kb, kan, kbn;
      if (!of_vertex(a, e) || !of_vertex(b, e) || !kite(a, c, &ka) || !kite(b, c, &kb) || !kite(a, nb, &kan) ||
          !kite(b, nb, &kbn))
        return "an edge whose ends do not touch its cells";
      t->c_nb[s] = nb;
      t->c_va[s] = a;
      t->c_vb[s] = b;
      const double ta = m.v_area[a], tb = m.v_area[b], dc = m.e_dc[e], dv = m.e_dv[e], sc = sign_c(c, e);
      t->c_g1[s] = ka / area * sign_v(a, e) * dc / ta;
      t->c_g2[s] = kb / area * sign_v(b, e) * dc / tb;
      t->c_n1[s] = ka * kan / (area * ta);
      t->c_n2[s] = kb * kbn / (area * tb);
      t->c_t[s] = -sc * dv / area;
      t->c_q[s] = 0.5 * dc * dv / area;
      t->c_r[s] = sc / dc;
      t->c_ka[s] = ka / ta;
      t->c_kb[s] = kb / tb;
      t->c_r2[s] = sign_v(a, e) / dv;
      const int v = m.c_vs[s];
      int sp = -1, in = 0;
      for (int i = 0; i < VDEG; i++) {
        const int x = m.v_es[V(v, i)];
        if (!of_vertex(v, x)) return "an edge of a vertex that does not end there";
        if (of_cell(c, x)) in++;
        else sp = x;
      }
      double kk;
      if (in != 2 || sp < 0 || !kite(v, c, &kk)) return "a vertex without one spoke to a cell around it";
      // the vertices of the cell's edges are the cell's vertices: each is the end of two of them,
      // so the per-edge halves below add up to the per-vertex terms
      t->c_sp[s] = sp;
      const double tv = m.v_area[v];
      t->c_g3[s] = kk / area * sign_v(v, sp) * m.e_dc[sp] / tv;
      t->c_m[s] = kk * kk / (area * tv);
      t->c_kk[s] = kk / tv;
      t->c_r3[s] = sign_v(v, sp) / m.e_dv[sp];
    }
    for (int k = 0; k < m.c_n[c]; k++) {  // every end of the cell's edges is one of its vertices
      int found = 0;
      for (int j = 0; j < m.c_n[c]; j++) found += m.c_vs[C(c, j)] == t->c_va[C(c, k)] || m.c_vs[C(c, j)] == t->c_vb[C(c, k)];
      if (found != 2) return "a cell whose edges and vertices do not alternate";
    }
    return nullptr;
  });
  if (!bad.empty()) return bad;
  for (auto *x : {&t->e_q, &t->e_o1, &t->e_o2}) x->assign(nE, 0);
  for (auto *x : {&t->e_d, &t->e_r4}) x->assign((size_t)4 * nE, 0.0);
  t->e_k.assign((size_t)6 * nE, 0.0);
  t->e_kr.assign((size_t)6 * nE, 0.0);
  t->e_t.assign((size_t)4 * nE, 0);
  for (auto *x : {&t->e_i1, &t->e_i2, &t->e_lap0}) x->assign(nE, 0.0);
  for (auto *x : {&t->e_ke, &t->e_lap}) x->assign((size_t)10 * nE, 0.0);
  return side_by_side(nE, [&](int e) -> const char * {
    const int c1 = m.e_c1[e], c2 = m.e_c2[e];
    const double dc = m.e_dc[e], dv = m.e_dv[e];
    t->e_lap0[e] = (sign_c(c2, e) * dv / m.c_area[c2] - sign_c(c1, e) * dv / m.c_area[c1]) / dc -
                   (sign_v(m.e_v2[e], e) * dc / m.v_area[m.e_v2[e]] - sign_v(m.e_v1[e], e) * dc / m.v_area[m.e_v1[e]]) / dv;
    if (m.e_n[e] != m.c_n[c1] + m.c_n[c2] - 2) return "edgesOnEdge is not the edges of the two cells";
    for (int j = 0; j < m.e_n[e]; j++) {
      const int x = m.e_eoe[E(e, j)];
      const bool in1 = of_cell(c1, x), in2 = of_cell(c2, x);
      if (x == e || in1 == in2) return "edgesOnEdge is not the edges of the two cells";
      for (int i = 0; i < j; i++)
        if (m.e_eoe[E(e, i)] == x) return "an edge twice in edgesOnEdge";
      const int c = in1 ? c1 : c2;
      const double to = in1 ? -1.0 : 1.0;  // the side c takes in the edge's gradients
      t->e_ke[E(e, j)] = sign_c(c, x) / (m.e_dc[x] * m.c_area[c]);
      double lap = to * sign_c(c, x) * m.e_dv[x] / m.c_area[c] / dc;
      for (int k = 0; k < 2; k++) {
        const int v = k ? m.e_v2[e] : m.e_v1[e];
        if (!of_vertex(v, x)) continue;
        lap -= (k ? 1.0 : -1.0) * sign_v(v, x) * m.e_dc[x] / m.v_area[v] / dv;
      }
      t->e_lap[E(e, j)] = lap;
    }
    unsigned q = 0;
    for (int k = 0; k < 2; k++) {
      const int v = k ? m.e_v2[e] : m.e_v1[e];
      int got = 0;
      for (int i = 0; i < VDEG; i++) {
        const int x = m.v_es[V(v, i)];
        if (x == e) continue;
        int slot = -1;
        for (int j = 0; j < m.e_n[e]; j++)
          if (m.e_eoe[E(e, j)] == x) slot = j;
        if (slot < 0 || got > 1) return "an edge of a vertex that is not in edgesOnEdge";
        q |= (unsigned)slot << (8 * (2 * k + got));
        t->e_t[E(e, 2 * k + got)] = x;
        t->e_d[E(e, 2 * k + got)] = sign_v(v, x) * m.e_dc[x] / m.v_area[v];
        t->e_r4[E(e, 2 * k + got)] = sign_v(v, x) / m.e_dv[x];
        got++;
      }
      int o = -1;
      for (int i = 0; i < VDEG; i++) {
        const int c = m.v_c[V(v, i)];
        if (c != c1 && c != c2) o = c;
      }
      double k1, k2, ko;
      if (got != 2 || o < 0 || !kite(v, c1, &k1) || !kite(v, c2, &k2) || !kite(v, o, &ko))
        return "a vertex of an edge without a third cell";
      (k ? t->e_o2 : t->e_o1)[e] = o;
      const double ta = m.v_area[v];
      t->e_k[E(e, 3 * k)] = k1 / ta;
      t->e_k[E(e, 3 * k + 1)] = k2 / ta;
      t->e_k[E(e, 3 * k + 2)] = ko / ta;
      t->e_kr[E(e, 3 * k)] = k1 / ta / m.c_area[c1];
      t->e_kr[E(e, 3 * k + 1)] = k2 / ta / m.c_area[c2];
      t->e_kr[E(e, 3 * k + 2)] = ko / ta / m.c_area[o];
      (k ? t->e_i2 : t->e_i1)[e] = 1.0 / ta;
    }
    for (int i = 0; i < 4; i++)  // a pass adds the four terms to their slots side by side
      for (int j = 0; j < i; j++)
        if (((q >> (8 * i)) & 0xFF) == ((q >> (8 * j)) & 0xFF)) return "two edges between the same vertices";
    t->e_q[e] = (int)q;
    return nullptr;
  });
}

}  // namespace mpsw

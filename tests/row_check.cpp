// Host run of the member-row passes (compiled by tests/test_rows.py with g++ from the package's own
// sources): one tangent-linear stage and one adjoint stage in FP64 through the coefficients of
// csrc/mpsw_rows.h, and the same stages written term by term through the intermediate fields.
#include <algorithm>
#include <cmath>
#include <cstring>
#include <random>
#include <vector>

#include "mpsw_rows.h"
#include "mpsw_setup.h"

using namespace mpsw;
using Vec = std::vector<double>;

namespace {

struct Point {  // a linearisation point
  Vec u, he, v, gpt, gpn, pe, vort, hv;
};

double worst(const Vec &a, const Vec &b) {
  double d = 0, s = 0;
  for (size_t i = 0; i < a.size(); i++) {
    d = std::max(d, std::fabs(a[i] - b[i]));
    s = std::max(s, std::fabs(b[i]));
  }
  return d / (s > 0 ? s : 1);
}

}  // namespace

// met: weightsOnEdge kites dcEdge dvEdge areaCell areaTriangle xyz of cells, edges, vertices [9] (as
// the reference holds them, lengths of the Earth's size); out: largest relative differences of
// tend_u', tend_h', u_ad, h_ad, then of delsq_u' and its transpose.
extern "C" int row_check(const int *ints, const int *const *conn, const double *const *met, double *out, char *err,
                         int errlen) {
  RefMesh r;
  r.nC = ints[0]; r.nE = ints[1]; r.nV = ints[2]; r.maxEdges = ints[3]; r.maxEdges2 = ints[4]; r.vd = 3;
  r.cellsOnEdge = conn[0]; r.verticesOnEdge = conn[1]; r.edgesOnEdge = conn[2]; r.nEdgesOnEdge = conn[3];
  r.edgesOnCell = conn[4]; r.nEdgesOnCell = conn[5]; r.cellsOnVertex = conn[6]; r.edgesOnVertex = conn[7];
  r.weightsOnEdge = met[0]; r.kiteAreasOnVertex = met[1]; r.dcEdge = met[2]; r.dvEdge = met[3];
  r.areaCell = met[4]; r.areaTriangle = met[5];
  r.xCell = met[6]; r.yCell = met[7]; r.zCell = met[8]; r.xEdge = met[9]; r.yEdge = met[10]; r.zEdge = met[11];
  r.xVertex = met[12]; r.yVertex = met[13]; r.zVertex = met[14];
  RefGeometry g;
  g.coeffs_reconstruct.assign((size_t)3 * r.maxEdges * r.nC, 0.0);
  BuiltMesh m;
  RowTabHost t;
  std::string e = build_mesh(r, g, 1, &m);
  if (e.empty()) e = build_rows(m, &t);
  if (!e.empty()) {
    std::strncpy(err, e.c_str(), errlen - 1);
    return 1;
  }
  const int nC = m.nC, nE = m.nE, nV = m.nV;
  std::mt19937_64 rng(ints[5]);
  auto rnd = [&](int n, double mean, double dev) {
    std::normal_distribution<double> d(mean, dev);
    Vec x(n);
    for (double &y : x) y = d(rng);
    return x;
  };
  m.v_f = rnd(nV, 0, 1e-4);
  Point bs{rnd(nE, 0, 20), rnd(nE, 5000, 300), rnd(nE, 0, 20), rnd(nE, 0, 1e-14), rnd(nE, 0, 1e-14), rnd(nE, 0, 2e-8),
           rnd(nV, 0, 1e-5), rnd(nV, 5000, 300)};
  const double apt = 0.5 * 300.0, G = GRAVITY;
  auto C = [&](int c, int k) { return (size_t)k * nC + c; };
  auto E = [&](int x, int j) { return (size_t)j * nE + x; };
  auto V = [&](int v, int k) { return (size_t)k * nV + v; };
  auto vsg = [&](int v, int x) { return m.e_v2[x] == v ? 1.0 : -1.0; };
  auto csg = [&](int c, int x) { return m.e_c1[x] == c ? 1.0 : -1.0; };
  // ---- tangent linear, term by term
  const Vec u = rnd(nE, 0, 0.1), h = rnd(nC, 0, 1.0);
  Vec pvv(nV), vort(nV), pc(nC, 0), ke(nC, 0), th(nC, 0), div(nC, 0), pe(nE), fl(nE), tu(nE), lap(nE);
  for (int v = 0; v < nV; v++) {
    double ci = 0, hh = 0;
    for (int k = 0; k < 3; k++) {
      const int x = m.v_es[V(v, k)];
      ci += vsg(v, x) * m.e_dc[x] * u[x];
      hh += m.v_k[V(v, k)] * h[m.v_c[V(v, k)]];
    }
    vort[v] = ci / m.v_area[v];
    pvv[v] = vort[v] / bs.hv[v] - hh / m.v_area[v] * (m.v_f[v] + bs.vort[v]) / (bs.hv[v] * bs.hv[v]);
  }
  for (int x = 0; x < nE; x++) fl[x] = u[x] * bs.he[x] + bs.u[x] * 0.5 * (h[m.e_c1[x]] + h[m.e_c2[x]]);
  for (int c = 0; c < nC; c++)
    for (int k = 0; k < m.c_n[c]; k++) {
      const int x = m.c_es[C(c, k)];
      pc[c] += m.c_vk[C(c, k)] * pvv[m.c_vs[C(c, k)]] / m.c_area[c];
      ke[c] += 0.25 * m.e_dc[x] * m.e_dv[x] * 2 * bs.u[x] * u[x] / m.c_area[c];
      th[c] -= csg(c, x) * m.e_dv[x] * fl[x] / m.c_area[c];
      div[c] += csg(c, x) * m.e_dv[x] * u[x] / m.c_area[c];
    }
  for (int x = 0; x < nE; x++) {
    double vt = 0;
    for (int j = 0; j < m.e_n[x]; j++) vt += m.e_w[E(x, j)] * u[m.e_eoe[E(x, j)]];
    const double gt = (pvv[m.e_v2[x]] - pvv[m.e_v1[x]]) / m.e_dv[x], gn = (pc[m.e_c2[x]] - pc[m.e_c1[x]]) / m.e_dc[x];
    pe[x] = 0.5 * (pvv[m.e_v1[x]] + pvv[m.e_v2[x]]) - apt * (vt * bs.gpt[x] + bs.v[x] * gt + u[x] * bs.gpn[x] + bs.u[x] * gn);
    lap[x] = (div[m.e_c2[x]] - div[m.e_c1[x]]) / m.e_dc[x] - (vort[m.e_v2[x]] - vort[m.e_v1[x]]) / m.e_dv[x];
  }
  for (int x = 0; x < nE; x++) {
    double q = 0;
    for (int j = 0; j < m.e_n[x]; j++) {
      const int y = m.e_eoe[E(x, j)];
      q += m.e_w[E(x, j)] * (fl[y] * 0.5 * (bs.pe[x] + bs.pe[y]) + bs.u[y] * bs.he[y] * 0.5 * (pe[x] + pe[y]));
    }
    tu[x] = q - ((ke[m.e_c2[x]] - ke[m.e_c1[x]]) + G * (h[m.e_c2[x]] - h[m.e_c1[x]])) / m.e_dc[x];
  }
  // ---- tangent linear, by rows
  Vec rpc(nC, 0), rke(nC, 0), rth(nC, 0), rpe(nE), rfl(nE), rtu(nE), rlap(nE);
  for (int c = 0; c < nC; c++)
    for (int k = 0; k < m.c_n[c]; k++) {
      const RowTlCell<double> q = row_tl_cell<double>(t, m, bs, c, k);
      rpc[c] += q.pe * u[q.e] + q.ps * u[q.sp] + q.pn * h[q.nb] + q.pc * h[c];
      rth[c] += q.te * u[q.e] + q.tn * h[q.nb] + q.tn * h[c];
      rke[c] += q.ke * u[q.e];
    }
  for (int x = 0; x < nE; x++) {
    const RowTlEdge<double> q = row_tl_edge<double>(t, m, bs, apt, x);
    const int c1 = m.e_c1[x], c2 = m.e_c2[x];
    rpe[x] = q.p0 * u[x] + q.h1 * h[c1] + q.h2 * h[c2] + q.o1 * h[t.e_o1[x]] + q.o2 * h[t.e_o2[x]] + q.pc * (rpc[c2] - rpc[c1]);
    rfl[x] = q.he * u[x] + q.uh * (h[c1] + h[c2]);
    rlap[x] = t.e_lap0[x] * u[x];
    for (int j = 0; j < m.e_n[x]; j++) {
      rpe[x] += row_tl_edge_slot(m.e_w[E(x, j)], apt * bs.gpt[x]) * u[m.e_eoe[E(x, j)]];
      rlap[x] += t.e_lap[E(x, j)] * u[m.e_eoe[E(x, j)]];
    }
    for (int i = 0; i < 4; i++)
      rpe[x] += row_tl_edge_tag(t, nE, x, i, q) * u[m.e_eoe[E(x, ((unsigned)t.e_q[x] >> (8 * i)) & 0xFF)]];
  }
  for (int x = 0; x < nE; x++) {
    double q = 0, own = 0;
    for (int j = 0; j < m.e_n[x]; j++) {
      const int y = m.e_eoe[E(x, j)];
      const RowTlTend<double> s = row_tl_tend<double>(bs, y, m.e_w[E(x, j)], bs.pe[x]);
      q += s.f * rfl[y] + s.p * rpe[y];
      own += s.p;
    }
    rtu[x] = q + own * rpe[x] - ((rke[m.e_c2[x]] - rke[m.e_c1[x]]) + G * (h[m.e_c2[x]] - h[m.e_c1[x]])) / m.e_dc[x];
  }
  out[0] = worst(rtu, tu);
  out[1] = worst(rth, th);
  out[4] = worst(rlap, lap);
  // ---- adjoint by rows, against the transpose of the tangent linear above: <L x, y> = <x, L^T y>
  // entry by entry is the full transpose; probed here with the term-by-term adjoint
  const Vec T = rnd(nE, 0, 1.0), H = rnd(nC, 0, 1e-12);  // tend_u_ad, tend_h_ad / areaCell
  Vec pead(nE), heada(nE), uad(nE, 0.0), had(nC, 0.0), pcad(nC, 0), keada(nC, 0), pvvad(nV, 0), x2(nE, 0.0);
  for (int x = 0; x < nE; x++) {
    double p = 0, hh = 0, uu = 0;
    for (int j = 0; j < m.e_n[x]; j++) {
      const int y = m.e_eoe[E(x, j)];
      const double w = m.e_w[E(x, j)], wr = m.e_wrev[E(x, j)], wpv = 0.5 * (bs.pe[x] + bs.pe[y]);
      p += 0.5 * w * bs.u[y] * bs.he[y] * T[x] + 0.5 * wr * bs.u[x] * bs.he[x] * T[y];
      hh += wr * bs.u[x] * wpv * T[y];
      uu += wr * wpv * bs.he[x] * T[y];
    }
    const double fa = H[m.e_c2[x]] - H[m.e_c1[x]];
    pead[x] = p;
    heada[x] = hh + bs.u[x] * m.e_dv[x] * fa;
    uad[x] = uu + m.e_dv[x] * bs.he[x] * fa - apt * bs.gpn[x] * p;
  }
  for (int c = 0; c < nC; c++)
    for (int k = 0; k < m.c_n[c]; k++) {
      const int x = m.c_es[C(c, k)];
      pcad[c] += csg(c, x) / m.e_dc[x] * apt * bs.u[x] * pead[x];
      keada[c] += csg(c, x) / m.e_dc[x] * T[x] / m.c_area[c];
      had[c] += csg(c, x) * G / m.e_dc[x] * T[x] + 0.5 * heada[x];
    }
  for (int v = 0; v < nV; v++) {
    for (int k = 0; k < 3; k++) {
      const int c = m.v_c[V(v, k)], x = m.v_es[V(v, k)];
      pvvad[v] += m.v_k[V(v, k)] / m.c_area[c] * pcad[c] + 0.5 * pead[x] - vsg(v, x) / m.e_dv[x] * apt * bs.v[x] * pead[x];
    }
    for (int k = 0; k < 3; k++)
      had[m.v_c[V(v, k)]] -= m.v_k[V(v, k)] / m.v_area[v] * (m.v_f[v] + bs.vort[v]) / (bs.hv[v] * bs.hv[v]) * pvvad[v];
  }
  for (int x = 0; x < nE; x++) {
    for (int j = 0; j < m.e_n[x]; j++) {
      const int y = m.e_eoe[E(x, j)];
      uad[x] -= m.e_wrev[E(x, j)] * apt * bs.gpt[y] * pead[y];
    }
    uad[x] += 0.5 * m.e_dc[x] * m.e_dv[x] * bs.u[x] * (keada[m.e_c1[x]] + keada[m.e_c2[x]]);
    const int a = m.e_v1[x], b = m.e_v2[x];
    uad[x] += m.e_dc[x] * (pvvad[b] / (bs.hv[b] * m.v_area[b]) - pvvad[a] / (bs.hv[a] * m.v_area[a]));
  }
  Vec qpe(nE), qhe(nE), qu(nE), qpc(nC, 0), qh(nC, 0);
  for (int x = 0; x < nE; x++) {
    double S = 0, P = 0, K = 0, sq = 0;
    const double kc = 0.5 * m.e_dc[x] * m.e_dv[x] * bs.u[x];
    for (int j = 0; j < m.e_n[x]; j++) {
      const int y = m.e_eoe[E(x, j)];
      const RowAdEdge<double> q = row_ad_edge<double>(t, bs, nE, x, j, y, m.e_w[E(x, j)], m.e_wrev[E(x, j)]);
      S += q.w * T[y];
      P += q.wp * T[y];
      K += q.ke * T[y];
      sq += q.sq;
    }
    const int c1 = m.e_c1[x], c2 = m.e_c2[x];
    const double fa = H[c2] - H[c1];
    P += 0.5 * bs.pe[x] * S;
    qpe[x] = 0.5 * bs.u[x] * bs.he[x] * S + sq * T[x];
    qhe[x] = bs.u[x] * P + bs.u[x] * m.e_dv[x] * fa;
    qu[x] = bs.he[x] * P + m.e_dv[x] * bs.he[x] * fa - apt * bs.gpn[x] * qpe[x] +
            kc * (K + (csg(c1, x) * t.c_ra[c1] + csg(c2, x) * t.c_ra[c2]) / m.e_dc[x] * T[x]);
  }
  for (int c = 0; c < nC; c++)
    for (int k = 0; k < m.c_n[c]; k++) {
      const RowAdCell<double> q = row_ad_cell<double>(t, m, bs, apt, c, k);
      qpc[c] += q.pc * qpe[q.e];
      qh[c] += q.g * T[q.e] + q.half * qhe[q.e] + q.hv * qpe[q.e] + q.hs * qpe[q.sp];
    }
  Vec qh2(qh);
  for (int c = 0; c < nC; c++)
    for (int k = 0; k < m.c_n[c]; k++) {
      const RowAdLast<double> q = row_ad_last<double>(t, m, bs, c, k);
      qh2[c] += q.n * qpc[q.nb] + q.c * qpc[c];
    }
  for (int x = 0; x < nE; x++) {
    const RowAdFinal<double> q = row_ad_final<double>(t, m, bs, apt, x);
    qu[x] += q.p0 * qpe[x] + q.k1 * qpc[m.e_c1[x]] + q.k2 * qpc[m.e_c2[x]] + q.o1 * qpc[t.e_o1[x]] + q.o2 * qpc[t.e_o2[x]];
    for (int j = 0; j < m.e_n[x]; j++) {
      const int y = m.e_eoe[E(x, j)];
      qu[x] += row_ad_final_slot(bs, apt, y, m.e_wrev[E(x, j)]) * qpe[y];
    }
    for (int i = 0; i < 4; i++) {
      const int y = m.e_eoe[E(x, ((unsigned)t.e_q[x] >> (8 * i)) & 0xFF)];
      qu[x] += row_ad_final_tag(t, bs, nE, apt, x, i, y, q) * qpe[y];
    }
  }
  out[2] = worst(qu, uad);
  out[3] = worst(qh2, had);
  // the adjoint against the tangent linear: <tu, T> + <th area, H> = <u, u_ad> + <h, h_ad>
  double a1 = 0, a2 = 0;
  for (int x = 0; x < nE; x++) {
    a1 += tu[x] * T[x];
    a2 += u[x] * qu[x];
  }
  for (int c = 0; c < nC; c++) {
    a1 += th[c] * m.c_area[c] * H[c];
    a2 += h[c] * qh2[c];
  }
  out[6] = std::fabs(a1 - a2) / std::fabs(a1);
  return 0;
}

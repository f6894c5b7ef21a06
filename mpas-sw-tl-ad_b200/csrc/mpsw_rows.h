// Tables of the FP32 member-row kernels (mpsw_rows.cuh): for every cell and edge the entities a
// tangent-linear or adjoint pass gathers directly from the pass's inputs, with the geometric part
// of each term's coefficient.  A term that the reference forms through an intermediate field
// (pv_vertex between u, h and pv_cell or pv_edge; ke, pv_vertex and vorticity adjoints) is folded
// into one coefficient per gathered row, so those fields are never stored for the members.
#pragma once

#include <string>
#include <vector>

#include "mpsw_internal.h"
#include "mpsw_setup.h"

namespace mpsw {

struct RowTab {
  bool ok = false;
  // cells [6][nC], slot k: edge k = c_es[k] of the cell, the cell nb across it, its vertices a, b;
  // vertex k = c_vs[k] and its spoke, the edge of that vertex which is not the cell's
  const int *c_nb, *c_sp, *c_va, *c_vb;
  const float *c_g1, *c_g2;  // kite(a,c) / area(c) * sign(a,e) dc(e) / areaT(a), the same at b
  const float *c_g3;         // kite(k,c) / area(c) * sign(k,spoke) dc(spoke) / areaT(k)
  const float *c_n1, *c_n2;  // kite(a,c) kite(a,nb) / (area(c) areaT(a)), the same at b
  const float *c_m;          // kite(k,c)^2 / (area(c) areaT(k))
  const float *c_t;          // -sign(c,e) dv(e) / area(c)
  const float *c_q;          // dc(e) dv(e) / (2 area(c))
  const float *c_r;          // sign(c,e) / dc(e)
  const float *c_ka, *c_kb;  // kite(a,c) / areaT(a), kite(b,c) / areaT(b)
  const float *c_kk;         // kite(k,c) / areaT(k)
  const float *c_r2;         // sign(a,e) / dv(e)
  const float *c_r3;         // sign(k,spoke) / dv(spoke)
  const float *c_ra;         // [nC] 1 / area
  // edges [nE]: slots in edgesOnEdge of the two other edges of v1 (bytes 0, 1) and v2 (bytes 2, 3);
  // the third cell of v1 and of v2
  const int *e_q, *e_o1, *e_o2;
  const int *e_t;     // [4][nE] those four edges
  const float *e_kr;  // [6][nE] e_k, each / area of its cell
  const float *e_d;   // [4][nE] sign(v,j) dc(j) / areaT(v) of those four edges
  const float *e_r4;  // [4][nE] sign(v,j) / dv(j)
  const float *e_k;   // [6][nE] kite(v1,c1) kite(v1,c2) kite(v1,o1) kite(v2,c1) kite(v2,c2) kite(v2,o2), each / areaT(v)
  const float *e_i1, *e_i2;  // 1 / areaT(v1), 1 / areaT(v2)
  const float *e_ke;         // [10][nE] sign(c,j) / (dc(j) area(c)), c the cell that edge j shares
  const float *e_lap;        // [10][nE] weight of edge j in delsq_u of the edge, e_lap0 its own
  const float *e_lap0;
};

// The same on the host.
struct RowTabHost {
  std::vector<int> c_nb, c_sp, c_va, c_vb, e_q, e_o1, e_o2, e_t;
  std::vector<double> c_g1, c_g2, c_g3, c_n1, c_n2, c_m, c_t, c_q, c_r, c_ka, c_kb, c_kk, c_r2, c_r3, c_ra;
  std::vector<double> e_d, e_r4, e_k, e_kr, e_i1, e_i2, e_ke, e_lap, e_lap0;
};

// Empty string, or what the mesh lacks (a vertex whose edges or cells are not those around it, an
// edgesOnEdge list that is not the edges of the two cells): the members then take the passes that
// go through the intermediate fields.
std::string build_rows(const BuiltMesh &m, RowTabHost *t);

// ---- coefficients of the rows an entity gathers --------------------------------------------------
// T: RowTab or RowTabHost; M: the mesh (MeshDev or BuiltMesh); BS: the linearisation point; apt: the
// APVM factor times the time step.  Slots past a list keep index 0 and zero coefficients.

// Tangent-linear cell pass, slot k (src/mpas_sw_dyncore_tlm.f90:255-316, 344-421, 541-561): rows u' at
// edge e and at the spoke, h' at the cell across;
//   pv_cell' = sum (pe u'_e + ps u'_spoke + pn h'_nb) + (sum pc) h'
//   tend_h'  = sum (te u'_e + tn h'_nb) + (sum tn) h'
//   ke'      = sum ke u'_e
// te is th he.  The passes multiply by the two in turn: the rounding of their product, the same in every
// stage of a window, would add up in h' (level 5, smooth perturbations, 24 stages: 1.2 times the general
// passes' error, 0.85 in turn).
template <typename R>
struct RowTlCell {
  int e, nb, sp;
  R pe, ps, pn, pc, te, tn, ke, th, he;
};
template <typename R, class T, class M, class BS>
MPSW_HD inline RowTlCell<R> row_tl_cell(const T &t, const M &m, const BS &bs, int c, int k) {
  const size_t s = (size_t)k * m.nC + c;
  RowTlCell<R> r;
  r.e = m.c_es[s];
  r.nb = t.c_nb[s];
  r.sp = t.c_sp[s];
  const int a = t.c_va[s], b = t.c_vb[s], v = m.c_vs[s];
  const R ra = R(1) / bs.hv[a], rb = R(1) / bs.hv[b], rv = R(1) / bs.hv[v];
  const R za = ((m.v_f[a] + bs.vort[a]) * ra) * ra, zb = ((m.v_f[b] + bs.vort[b]) * rb) * rb,
          zv = ((m.v_f[v] + bs.vort[v]) * rv) * rv;
  const R u = bs.u[r.e];
  r.th = t.c_t[s];
  r.he = bs.he[r.e];
  r.pe = t.c_g1[s] * ra + t.c_g2[s] * rb;
  r.ps = t.c_g3[s] * rv;
  r.pn = -(t.c_n1[s] * za + t.c_n2[s] * zb);
  r.pc = -(t.c_m[s] * zv);
  r.te = r.th * r.he;
  r.tn = R(0.5) * (r.th * u);
  r.ke = t.c_q[s] * u;
  return r;
}

// Tangent-linear edge pass (:117-126, 319-393, 425-445, 638-652):
//   pv_edge' = sum_j p_j u'_j + p0 u' + h1 h'_c1 + h2 h'_c2 + o1 h'_o1 + o2 h'_o2 + pc (pc'_c2 - pc'_c1)
//   (u h_edge)' = he u' + uh (h'_c1 + h'_c2);  delsq_u' = sum_j lap_j u'_j + lap0 u'
template <typename R>
struct RowTlEdge {
  R p0, h1, h2, o1, o2, pc, he, uh;
  R y1, y2, ag;  // weights of pv at the two ends, apt gradPVt: what the slots share
};
template <typename R, class T, class M, class BS>
MPSW_HD inline RowTlEdge<R> row_tl_edge(const T &t, const M &m, const BS &bs, R apt, int e) {
  const int nE = m.nE, a = m.e_v1[e], b = m.e_v2[e];
  RowTlEdge<R> r;
  const R ra = R(1) / bs.hv[a], rb = R(1) / bs.hv[b];
  const R u = bs.u[e], dc = m.e_dc[e], av = (apt * bs.v[e]) / m.e_dv[e];
  r.y1 = (R(0.5) + av) * ra;
  r.y2 = (R(0.5) - av) * rb;
  r.ag = apt * bs.gpt[e];
  const R z1 = ((m.v_f[a] + bs.vort[a]) * ra) * r.y1, z2 = ((m.v_f[b] + bs.vort[b]) * rb) * r.y2;
  r.p0 = (t.e_i2[e] * r.y2 - t.e_i1[e] * r.y1) * dc - apt * bs.gpn[e];
  r.h1 = -(t.e_k[e] * z1 + t.e_k[(size_t)3 * nE + e] * z2);
  r.h2 = -(t.e_k[(size_t)nE + e] * z1 + t.e_k[(size_t)4 * nE + e] * z2);
  r.o1 = -(t.e_k[(size_t)2 * nE + e] * z1);
  r.o2 = -(t.e_k[(size_t)5 * nE + e] * z2);
  r.pc = -(apt * u) / dc;
  r.he = bs.he[e];
  r.uh = R(0.5) * u;
  return r;
}
// p_j: the tangential velocity's part of slot j (w: weightsOnEdge there), and what slot tag i (byte i
// of e_q) adds to it through the vertex it shares with the edge
template <typename R>
MPSW_HD inline R row_tl_edge_slot(R w, R ag) {
  return -(ag * w);
}
template <typename R, class T>
MPSW_HD inline R row_tl_edge_tag(const T &t, int nE, int e, int i, const RowTlEdge<R> &r) {
  return t.e_d[(size_t)i * nE + e] * (i < 2 ? r.y1 : r.y2);
}

// Tangent-linear tendency pass, slot j (:564-600): q' = sum_j (f_j (u h_edge)'_j + p_j pv_edge'_j) +
// (sum p_j) pv_edge'
template <typename R>
struct RowTlTend {
  R f, p;
};
template <typename R, class BS>
MPSW_HD inline RowTlTend<R> row_tl_tend(const BS &bs, int nb, R w, R pe) {
  return {(R(0.5) * w) * (pe + bs.pe[nb]), ((R(0.5) * w) * bs.u[nb]) * bs.he[nb]};
}

// Adjoint edge pass, slot j (src/mpas_sw_dyncore_adj.f90:689-736, 193-200, 235-242; the ke adjoint
// of both cells, :306-317, folded into u): weights of the row T = tend_u_ad at edge j in
//   S = sum w T, P = sum wp T, K = sum ke T, and with them
//   pv_edge_ad = (u h_edge / 2) S + (sum sq) T;  h_edge_ad = u (P + pv_edge S / 2) + ..;
//   u_ad = h_edge (P + pv_edge S / 2) + (dc dv u / 2) (K + ..) + ..
// w, wr: weightsOnEdge there and back
template <typename R>
struct RowAdEdge {
  R w, wp, ke, sq;
};
template <typename R, class T, class BS>
MPSW_HD inline RowAdEdge<R> row_ad_edge(const T &t, const BS &bs, int nE, int e, int j, int nb, R w, R wr) {
  RowAdEdge<R> r;
  r.w = wr;
  r.wp = (R(0.5) * wr) * bs.pe[nb];
  r.ke = t.e_ke[(size_t)j * nE + e];
  r.sq = R(0.5) * ((w * bs.u[nb]) * bs.he[nb]);
  return r;
}

// Adjoint cell pass, slot k (:202-213, 306-326, 358-369, and pv_edge_ad's share of the h_vertex
// adjoint, :244-289): of the rows at edge e
//   pv_cell_ad = sum pc pv_edge_ad;  h_ad = sum (g T + h_edge_ad / 2 + hv pv_edge_ad) + hs pv_edge_ad_spoke
template <typename R>
struct RowAdCell {
  int e, sp;
  R pc, g, hv, hs, half;
};
template <typename R, class T, class M, class BS>
MPSW_HD inline RowAdCell<R> row_ad_cell(const T &t, const M &m, const BS &bs, R apt, int c, int k) {
  const size_t s = (size_t)k * m.nC + c;
  RowAdCell<R> r;
  r.e = m.c_es[s];
  r.sp = t.c_sp[s];
  const int a = t.c_va[s], b = t.c_vb[s], v = m.c_vs[s];
  const R ra = R(1) / bs.hv[a], rb = R(1) / bs.hv[b], rv = R(1) / bs.hv[v];
  const R za = ((m.v_f[a] + bs.vort[a]) * ra) * ra, zb = ((m.v_f[b] + bs.vort[b]) * rb) * rb,
          zv = ((m.v_f[v] + bs.vort[v]) * rv) * rv;
  const R av = (apt * bs.v[r.e]) * t.c_r2[s], avs = (apt * bs.v[r.sp]) * t.c_r3[s];
  r.pc = (apt * bs.u[r.e]) * t.c_r[s];
  r.g = R(GRAVITY) * t.c_r[s];
  r.hv = -((t.c_ka[s] * za) * (R(0.5) - av) + (t.c_kb[s] * zb) * (R(0.5) + av));
  r.hs = -((t.c_kk[s] * zv) * (R(0.5) - avs));
  r.half = R(0.5);
  return r;
}

// Adjoint final pass of a cell, slot k: h_ad += sum n pv_cell_ad_nb + (sum c) pv_cell_ad
template <typename R>
struct RowAdLast {
  int nb;
  R n, c;
};
template <typename R, class T, class M, class BS>
MPSW_HD inline RowAdLast<R> row_ad_last(const T &t, const M &m, const BS &bs, int c, int k) {
  const size_t s = (size_t)k * m.nC + c;
  RowAdLast<R> r;
  r.nb = t.c_nb[s];
  const int a = t.c_va[s], b = t.c_vb[s], v = m.c_vs[s];
  const R ra = R(1) / bs.hv[a], rb = R(1) / bs.hv[b], rv = R(1) / bs.hv[v];
  const R za = ((m.v_f[a] + bs.vort[a]) * ra) * ra, zb = ((m.v_f[b] + bs.vort[b]) * rb) * rb,
          zv = ((m.v_f[v] + bs.vort[v]) * rv) * rv;
  r.n = -(t.c_n1[s] * za + t.c_n2[s] * zb) * (m.c_area[c] * t.c_ra[r.nb]);
  r.c = -(t.c_m[s] * zv);
  return r;
}
// Adjoint final pass of an edge (:215-284, 296-303, 350-355):
//   u_ad += sum_j p_j pv_edge_ad_j + p0 pv_edge_ad + k1 pc_ad_c1 + k2 pc_ad_c2 + o1 pc_ad_o1 + o2 pc_ad_o2
template <typename R>
struct RowAdFinal {
  R p0, k1, k2, o1, o2;
  R x1, x2;  // -dc / (hv areaT) at v1, dc / (hv areaT) at v2
};
template <typename R, class T, class M, class BS>
MPSW_HD inline RowAdFinal<R> row_ad_final(const T &t, const M &m, const BS &bs, R apt, int e) {
  const int nE = m.nE;
  RowAdFinal<R> r;
  const R dc = m.e_dc[e], av = (apt * bs.v[e]) / m.e_dv[e];
  const R d1 = -dc / bs.hv[m.e_v1[e]], d2 = dc / bs.hv[m.e_v2[e]];
  r.x1 = d1 * t.e_i1[e];
  r.x2 = d2 * t.e_i2[e];
  r.p0 = r.x1 * (R(0.5) + av) + r.x2 * (R(0.5) - av);
  r.k1 = d1 * t.e_kr[e] + d2 * t.e_kr[(size_t)3 * nE + e];
  r.k2 = d1 * t.e_kr[(size_t)nE + e] + d2 * t.e_kr[(size_t)4 * nE + e];
  r.o1 = d1 * t.e_kr[(size_t)2 * nE + e];
  r.o2 = d2 * t.e_kr[(size_t)5 * nE + e];
  return r;
}
// p_j: the tangential velocity's part (wr: the edge's weight in the list of edge j), and what slot
// tag i (byte i of e_q, the edge nb) adds to it through the vertex it shares with the edge
template <typename R, class BS>
MPSW_HD inline R row_ad_final_slot(const BS &bs, R apt, int nb, R wr) {
  return -((apt * bs.gpt[nb]) * wr);
}
template <typename R, class T, class BS>
MPSW_HD inline R row_ad_final_tag(const T &t, const BS &bs, int nE, R apt, int e, int i, int nb, const RowAdFinal<R> &r) {
  return (i < 2 ? r.x1 : r.x2) * (R(0.5) - (apt * bs.v[nb]) * t.e_r4[(size_t)i * nE + e]);
}

}  // namespace mpsw

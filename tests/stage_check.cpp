// Host run of the nonlinear stage on halo tiles (compiled by tests/test_stage_tiles.py with g++ from
// the package's own sources): the phases of csrc/mpsw_stage.h, tile after tile, entity after entity.
#include <algorithm>
#include <cstring>
#include <vector>

#include "mpsw_setup.h"
#include "mpsw_tiles.h"

using namespace mpsw;

// ints: nC nE nV maxEdges maxEdges2 K.  cfg: dt apvm visc2 visc4 drag wind.  Arrays in the
// reference layout and numbering.  out: tend_u tend_h, then u h_edge v gradPVt gradPVn pv_edge
// vorticity h_vertex ke (what the stage hands to the linearised sweeps).  counts: tiles, -,
// tiles beyond the layers' caps, entities owned by no or several tiles, non-finite tendencies.
extern "C" int stage_check(const int *ints, const double *cfg, const int *const *conn, const double *const *met,
                           const double *u, const double *h, double *const *out, long long *counts, char *err,
                           int errlen) {
  RefMesh r;
  r.nC = ints[0]; r.nE = ints[1]; r.nV = ints[2]; r.maxEdges = ints[3]; r.maxEdges2 = ints[4]; r.vd = 3;
  r.cellsOnEdge = conn[0]; r.verticesOnEdge = conn[1]; r.edgesOnEdge = conn[2]; r.nEdgesOnEdge = conn[3];
  r.edgesOnCell = conn[4]; r.nEdgesOnCell = conn[5]; r.cellsOnVertex = conn[6]; r.edgesOnVertex = conn[7];
  r.weightsOnEdge = met[0]; r.kiteAreasOnVertex = met[1]; r.dcEdge = met[2]; r.dvEdge = met[3];
  r.areaCell = met[4]; r.areaTriangle = met[5]; r.fVertex = met[6]; r.h_s = met[7]; r.u_src = met[8];
  r.xCell = met[9]; r.yCell = met[10]; r.zCell = met[11]; r.xEdge = met[12]; r.yEdge = met[13]; r.zEdge = met[14];
  r.xVertex = met[15]; r.yVertex = met[16]; r.zVertex = met[17];
  RefGeometry g;
  g.coeffs_reconstruct.assign((size_t)3 * r.maxEdges * r.nC, 0.0);
  g.meshScalingDel2.assign(r.nE, 1.0);
  g.meshScalingDel4.assign(r.nE, 1.0);
  BuiltMesh m;
  StageSetHost ts;
  std::string e = build_mesh(r, g, 1, &m);
  if (e.empty()) e = build_stage_tiles(m, ints[5], &ts);
  if (!e.empty()) {
    std::strncpy(err, e.c_str(), errlen - 1);
    return 1;
  }
  auto inward = [](const std::vector<int> &p, const double *x) {
    std::vector<double> y(p.size());
    for (size_t i = 0; i < p.size(); i++) y[p[i]] = x[i];
    return y;
  };
  const std::vector<double> ui = inward(m.perm_e, u), hi = inward(m.perm_c, h);
  const std::vector<int> *perm[11] = {&m.perm_e, &m.perm_c, &m.perm_e, &m.perm_e, &m.perm_e, &m.perm_e,
                                      &m.perm_e, &m.perm_e, &m.perm_v, &m.perm_v, &m.perm_c};
  std::vector<std::vector<double>> res(11);
  for (int k = 0; k < 11; k++) res[k].assign(perm[k]->size(), 1e300);
  StageArgs<double, double> a{};
  a.u = ui.data(); a.h = hi.data();
  a.ph.dt = cfg[0]; a.ph.apvm = cfg[1]; a.ph.visc2 = cfg[2]; a.ph.visc4 = cfg[3];
  a.ph.drag = cfg[4] != 0; a.ph.wind = cfg[5] != 0;
  a.tend_u = res[0].data(); a.tend_h = res[1].data();
  for (int k = 0; k < 9; k++) a.out.d[k] = res[2 + k].data();
  a.out.on = 1;
  a.sc2 = m.e_sc2.data(); a.sc4 = m.e_sc4.data(); a.usrc = m.e_usrc.data();
  const bool del4 = cfg[3] > 0, visc = del4 || cfg[2] > 0;
  std::vector<int> oc(m.nC, 0), oe(m.nE, 0), ov(m.nV, 0);
  int bad = 0;
  a.ph.bad = &bad;
  for (int i = 0; i < ts.ntiles; i++) {
    const int *n = &ts.cnt[(size_t)i * kStageCounts];
    int off[kStageSections];
    stage_layout(n, 8, off);
    const unsigned char *b = ts.blob64.data() + ts.off64[i];
    std::vector<double> work(stage_work(8, visc, del4) / 8, 1e300);
    unsigned char *w = (unsigned char *)work.data();
    auto sec = [&](int s) { return (const StageChunk *)(b + off[s]); };
    const int *ge = (const int *)(b + off[SB_GE]), *gc = (const int *)(b + off[SB_GC]), *gv = (const int *)(b + off[SB_GV]);
    for (int x = 0; x < n[S_EA]; x++) work[W_U + x] = a.u[ge[x]];
    for (int x = 0; x < n[S_CA]; x++) work[W_H + x] = a.h[gc[x]];
    for (int x = 0; x < n[S_VA]; x++) {
      VertexRec<double> q;
      stage_rec(sec(SB_V), n[S_VA], x, &q);
      stage_vertex(q, w, a, x, x < n[S_VO] ? gv[x] : -1, visc);
    }
    for (int x = 0; x < (visc ? n[S_CM] : n[S_CK]); x++) {
      CellMRec<double> q;
      CellKRec<double> k;
      CellXRec<double> y;
      stage_rec(sec(SB_CM), n[S_CM], x, &q);
      if (x < n[S_CK]) {
        stage_rec(sec(SB_CK), n[S_CK], x, &k);
        stage_ke(k, q.v[6], w, a, x, x < n[S_CO] ? gc[x] : -1);
      }
      stage_rec(sec(SB_CX), n[S_CM], x, &y);
      if (visc) stage_div(y, q.v[6], w, x);
    }
    std::vector<EdgeRec<double>> er(n[S_EM]);
    std::vector<double> perp(n[S_EM]);
    for (int x = 0; x < n[S_EM]; x++) {
      stage_rec(sec(SB_E), n[S_EM], x, &er[x]);
      perp[x] = stage_perp(er[x], w);
    }
    for (int x = 0; x < n[S_CM]; x++) {
      CellMRec<double> q;
      stage_rec(sec(SB_CM), n[S_CM], x, &q);
      stage_pvcell(q, w, x);
    }
    for (int x = 0; x < n[S_EM]; x++) stage_edge(er[x], w, a, x, x < n[S_EO] ? ge[x] : -1, perp[x], del4);
    for (int x = 0; x < n[S_CO]; x++) {
      CellMRec<double> q;
      CellXRec<double> y;
      stage_rec(sec(SB_CM), n[S_CM], x, &q);
      stage_rec(sec(SB_CX), n[S_CM], x, &y);
      stage_thick(y, sec(SB_CO)[x], q.v[6], w, a, x, gc[x], 0.0, 0.0);
    }
    if (del4) {
      for (int x = 0; x < n[S_VA]; x++) {
        VertexRec<double> q;
        stage_rec(sec(SB_V), n[S_VA], x, &q);
        stage_del4_vertex(q, w, x, n[S_EM]);
      }
      for (int x = 0; x < n[S_CK]; x++) {
        CellMRec<double> q;
        CellXRec<double> y;
        stage_rec(sec(SB_CM), n[S_CM], x, &q);
        stage_rec(sec(SB_CX), n[S_CM], x, &y);
        stage_del4_cell(y, q.v[6], w, x, n[S_EM]);
      }
    }
    for (int x = 0; x < n[S_EO]; x++) stage_tend(er[x], w, a, x, ge[x], 0.0, 0.0);
    for (int x = 0; x < n[S_CO]; x++) oc[gc[x]]++;
    for (int x = 0; x < n[S_EO]; x++) oe[ge[x]]++;
    for (int x = 0; x < n[S_VO]; x++) ov[gv[x]]++;
  }
  for (int k = 0; k < 11; k++)
    for (size_t i = 0; i < perm[k]->size(); i++) out[k][i] = res[k][(*perm[k])[i]];
  auto wrong = [](const std::vector<int> &x) { return (long long)std::count_if(x.begin(), x.end(), [](int y) { return y != 1; }); };
  counts[0] = ts.ntiles;
  counts[2] = 0;
  for (int i = 0; i < ts.ntiles; i++) counts[2] += !stage_fits(&ts.cnt[(size_t)i * kStageCounts]);
  counts[3] = wrong(oc) + wrong(oe) + wrong(ov);
  counts[4] = bad;
  for (int k = 0; k < kStageCounts; k++) {
    counts[5 + k] = 0;
    for (int i = 0; i < ts.ntiles; i++) counts[5 + k] += ts.cnt[(size_t)i * kStageCounts + k];
  }
  return 0;
}

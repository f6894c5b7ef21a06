// Host check of the FP64 adjoint stage's tiles (compiled by tests/test_stage_ad_tiles.py with g++ from the
// package's own sources): the tables alone, every index against the layer that a phase has formed.
#include <algorithm>
#include <cstring>
#include <vector>

#include "mpsw_setup.h"
#include "mpsw_tiles.h"

using namespace mpsw;

// ints: nC nE nV maxEdges maxEdges2 K.  counts: tiles, indices outside their layer, entities not owned
// exactly once, tiles beyond the caps, blobs out of place.
extern "C" int stage_ad_check(const int *ints, const int *const *conn, const double *const *met, long long *counts,
                              char *err, int errlen) {
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
  StageSetHost t;
  std::string e = build_mesh(r, g, 1, &m);
  if (e.empty()) e = build_stage_ad_tiles(m, ints[5], &t);
  if (!e.empty()) {
    std::strncpy(err, e.c_str(), errlen - 1);
    return 1;
  }
  counts[0] = t.ntiles;
  std::vector<int> oe(m.nE, 0), oc(m.nC, 0);
  auto in = [&](int at, int n) { counts[1] += at < 0 || at >= 8 * n; };
  for (int i = 0; i < t.ntiles; i++) {
    const int *n = &t.cnt[(size_t)i * kTileCounts];
    int off[kStageAdSections];
    const long long end = t.off64[i] + stage_ad_layout(n, off);
    counts[3] += !stage_ad_fits(n);
    counts[4] += t.off64[i] % 16 != 0 || end != (i + 1 < t.ntiles ? t.off64[i + 1] : (long long)t.blob64.size());
    const unsigned char *b = t.blob64.data() + t.off64[i];
    auto sec = [&](int s) { return (const StageChunk *)(b + off[s]); };
    for (int x = 0; x < n[V_ALL]; x++) {
      AdVertexRec q;
      stage_rec(sec(YB_V), n[V_ALL], x, &q);
      for (int k = 0; k < 3; k++) { in(q.at(k), n[E_MID]); in(q.at(3 + k), n[C_MID]); in(q.at(6 + k), n[E_MID]); }
    }
    for (int x = 0; x < n[C_MID]; x++) {
      AdCellRec q;
      stage_rec(sec(YB_C), n[C_MID], x, &q);
      for (int k = 0; k < 6; k++) in(q.at(k), n[E_MID]);
    }
    for (int x = 0; x < n[C_OWN]; x++) {
      AdCellRec q;
      stage_rec(sec(YB_O), n[C_OWN], x, &q);
      for (int k = 0; k < 6; k++) in(q.at(k), n[V_ALL]);
    }
    for (int x = 0; x < n[E_MID]; x++) {
      AdEdgeRec q;
      stage_rec(sec(YB_E), n[E_MID], x, &q);
      const bool own = x < n[E_OWN];
      for (int k = 0; k < 2; k++) { in(q.at(k), n[own ? C_MID : C_ALL]); in(q.at(2 + k), n[V_ALL]); }
      for (int j = 0; j < 10; j++) in(q.at(4 + j), n[own ? E_MID : E_ALL]);
    }
    const int *ge = (const int *)(b + off[YB_GE]), *gc = (const int *)(b + off[YB_GC]), *gv = (const int *)(b + off[YB_GV]);
    for (int x = 0; x < n[E_ALL]; x++) counts[1] += ge[x] < 0 || ge[x] >= m.nE;
    for (int x = 0; x < n[C_ALL]; x++) counts[1] += gc[x] < 0 || gc[x] >= m.nC;
    for (int x = 0; x < n[V_ALL]; x++) counts[1] += gv[x] < 0 || gv[x] >= m.nV;
    for (int x = 0; x < n[E_OWN]; x++) oe[ge[x]]++;
    for (int x = 0; x < n[C_OWN]; x++) oc[gc[x]]++;
  }
  for (int x : oe) counts[2] += x != 1;
  for (int x : oc) counts[2] += x != 1;
  return 0;
}

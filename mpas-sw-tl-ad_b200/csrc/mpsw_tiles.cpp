// Host builder of the halo tiles of the fused member-stage kernels (see mpsw_tiles.h).
#include "mpsw_tiles.h"

#include <algorithm>
#include <cstring>
#include <sstream>

#include "mpsw_parts.h"

namespace mpsw {
namespace {

constexpr int kCellSlots = 6, kEoeSlots = 10;

// One local index space of a tile: entities join in layers; each layer is sorted by internal
// index before it is numbered, so the gathers of a layer walk memory in order.
struct Space {
  std::vector<int> &stamp, &loc;
  int tile;
  std::vector<int> list, pending;
  Space(std::vector<int> &s, std::vector<int> &l, int t) : stamp(s), loc(l), tile(t) {}
  void add(int g) {
    if (stamp[g] != tile) {
      stamp[g] = tile;
      loc[g] = -1;
      pending.push_back(g);
    }
  }
  int close() {
    std::sort(pending.begin(), pending.end());
    for (int g : pending) {
      loc[g] = (int)list.size();
      list.push_back(g);
    }
    pending.clear();
    return (int)list.size();
  }
  int local(int g) const { return stamp[g] == tile && loc[g] >= 0 ? loc[g] : -1; }
};

struct Builder {
  const BuiltMesh &m;
  std::vector<int> se, le, sc, lc, sv, lv;
  explicit Builder(const BuiltMesh &mesh)
      : m(mesh), se(mesh.nE, -1), le(mesh.nE, -1), sc(mesh.nC, -1), lc(mesh.nC, -1), sv(mesh.nV, -1),
        lv(mesh.nV, -1) {}
  int cn(int c) const { return m.c_n[c]; }
  int ces(int c, int k) const { return m.c_es[(size_t)k * m.nC + c]; }
  int cvs(int c, int k) const { return m.c_vs[(size_t)k * m.nC + c]; }
  int cnb(int c, int k) const {
    const int e = ces(c, k);
    return m.e_c1[e] == c ? m.e_c2[e] : m.e_c1[e];
  }
  int eoe(int e, int j) const { return m.e_eoe[(size_t)j * m.nE + e]; }
  int ves(int v, int k) const { return m.v_es[(size_t)k * m.nV + v]; }
  int vc(int v, int k) const { return m.v_c[(size_t)k * m.nV + v]; }
};

std::string fail(int tile, const char *what) {
  std::ostringstream s;
  s << "tile " << tile << ": " << what;
  return s.str();
}

// Every neighbour a phase of the stage reads must be in the tile, in the layer the phase needs
// (local index below that layer's count).
bool validate(const Builder &b, const BuiltMesh &m, const Space &E, const Space &C, const Space &V, const int *cnt,
              bool adjoint) {
  auto below = [](int x, int n) { return x >= 0 && x < n; };
  auto cells_ok = [&](int hi, int edges_below, bool verts, bool nbs) {
    for (int i = 0; i < hi; i++) {
      const int c = C.list[i];
      for (int k = 0; k < b.cn(c); k++) {
        if (!below(E.local(b.ces(c, k)), edges_below)) return false;
        if (verts && V.local(b.cvs(c, k)) < 0) return false;
        if (nbs && C.local(b.cnb(c, k)) < 0) return false;
      }
    }
    return true;
  };
  auto edges_ok = [&](int hi, int eoe_below, int cells_below, bool verts) {
    for (int i = 0; i < hi; i++) {
      const int e = E.list[i];
      if (!below(C.local(m.e_c1[e]), cells_below) || !below(C.local(m.e_c2[e]), cells_below)) return false;
      if (verts && (V.local(m.e_v1[e]) < 0 || V.local(m.e_v2[e]) < 0)) return false;
      for (int j = 0; j < m.e_n[e]; j++)
        if (!below(E.local(b.eoe(e, j)), eoe_below)) return false;
    }
    return true;
  };
  auto verts_ok = [&](int edges_below, int cells_below) {
    for (int v : V.list)
      for (int k = 0; k < VDEG; k++)
        if (!below(E.local(b.ves(v, k)), edges_below) || !below(C.local(b.vc(v, k)), cells_below)) return false;
    return true;
  };
  if (!adjoint)
    return verts_ok(cnt[E_ALL], cnt[C_ALL]) &&                  // pv_vertex'
           cells_ok(cnt[C_KE], cnt[E_ALL], false, false) &&     // ke'
           cells_ok(cnt[C_OWN], cnt[E_ALL], false, true) &&     // thickness tendency
           cells_ok(cnt[C_MID], cnt[E_ALL], true, false) &&     // pv_cell'
           edges_ok(cnt[E_MID], cnt[E_ALL], cnt[C_MID], true) &&  // pv_edge', fluxes
           edges_ok(cnt[E_OWN], cnt[E_MID], cnt[C_KE], true);     // normal-velocity tendency
  return edges_ok(cnt[E_MID], cnt[E_ALL], cnt[C_ALL], false) &&   // edge adjoints
         cells_ok(cnt[C_MID], cnt[E_MID], false, false) &&        // pv_cell / ke adjoints
         verts_ok(cnt[E_MID], cnt[C_MID]) &&                      // vertex adjoints
         edges_ok(cnt[E_OWN], cnt[E_MID], cnt[C_KE], true) &&     // owned edges
         cells_ok(cnt[C_OWN], cnt[E_MID], true, false);           // owned cells
}

// Append one tile's blob (BlobSection layout of blob_layout).  Local indices of neighbours
// outside the tile are kNoLocal (validate() has checked no phase reads them); slots past an
// entity's list length hold local index 0 with zero coefficients, so a phase may run all slots.
void pack_blob(const Builder &b, const BuiltMesh &m, const Space &E, const Space &C, const Space &V,
               const int *cnt, bool adjoint, std::vector<unsigned char> *blob) {
  int off[kBlobSections];
  const int size = blob_layout(cnt, adjoint, off);
  const size_t base = blob->size();
  blob->resize(base + size, 0);
  unsigned char *p = blob->data() + base;
  auto ints = [&](int sec) { return reinterpret_cast<int *>(p + off[sec]); };
  auto u16s = [&](int sec) { return reinterpret_cast<uint16_t *>(p + off[sec]); };
  auto flts = [&](int sec) { return reinterpret_cast<float *>(p + off[sec]); };
  auto L = [](int x) { return x < 0 ? kNoLocal : (uint16_t)x; };
  std::memcpy(ints(B_GE), E.list.data(), 4 * E.list.size());
  std::memcpy(ints(B_GC), C.list.data(), 4 * C.list.size());
  std::memcpy(ints(B_GV), V.list.data(), 4 * V.list.size());
  // records: vertex es[3] cs[3]; cell es[6] vs[6] nb[6]; edge c1 c2 v1 v2 eoe[10]
  for (int i = 0; i < cnt[V_ALL]; i++) {
    const int v = V.list[i];
    uint16_t *r = u16s(B_VREC) + (size_t)kVRec * i;
    for (int k = 0; k < VDEG; k++) {
      r[k] = L(E.local(b.ves(v, k)));
      r[3 + k] = L(C.local(b.vc(v, k)));
    }
  }
  for (int i = 0; i < cnt[C_MID]; i++) {
    const int c = C.list[i];
    uint16_t *r = u16s(B_CREC) + (size_t)kCRec * i;
    for (int k = 0; k < kCellSlots; k++) {
      const bool in = k < b.cn(c);
      r[k] = in ? L(E.local(b.ces(c, k))) : 0;
      r[6 + k] = in ? L(V.local(b.cvs(c, k))) : 0;
      r[12 + k] = in ? L(C.local(b.cnb(c, k))) : 0;
    }
  }
  for (int i = 0; i < cnt[E_MID]; i++) {
    const int e = E.list[i];
    uint16_t *r = u16s(B_EREC) + (size_t)kERec * i;
    r[0] = L(C.local(m.e_c1[e]));
    r[1] = L(C.local(m.e_c2[e]));
    r[2] = L(V.local(m.e_v1[e]));
    r[3] = L(V.local(m.e_v2[e]));
    for (int j = 0; j < kEoeSlots; j++) r[4 + j] = j < m.e_n[e] ? L(E.local(b.eoe(e, j))) : 0;
  }
  // coefficients, formed in FP64 and rounded once
  auto vslot = [&](int v, int k) { return (size_t)k * m.nV + v; };
  auto cslot = [&](int c, int k) { return (size_t)k * m.nC + c; };
  for (int i = 0; i < cnt[V_ALL]; i++) {
    const int v = V.list[i];
    float *q = flts(B_VCOEF) + 8 * (size_t)i;
    for (int k = 0; k < VDEG; k++) {
      const size_t s = vslot(v, k);
      const int e = m.v_es[s], c = m.v_c[s];
      if (!adjoint) {
        q[k] = (float)((double)m.v_esg[s] * m.e_dc[e] / m.v_area[v]);  // circulation -> vorticity'
        q[3 + k] = (float)(m.v_k[s] / m.v_area[v]);                       // h' -> h_vertex'
      } else {
        q[k] = (float)(m.v_k[s] / m.c_area[c]);                           // pv_cell_ad -> pv_vertex_ad
        q[3 + k] = (float)((double)m.v_esg[s] / m.e_dv[e]);               // gradPVt_ad -> pv_vertex_ad
      }
    }
    q[6] = (float)(adjoint ? 1.0 / m.v_area[v] : m.v_f[v]);
    q[7] = (float)(adjoint ? m.v_f[v] : 0.0);
  }
  for (int i = 0; i < cnt[C_MID]; i++) {
    const int c = C.list[i];
    float *q = flts(B_C1) + 8 * (size_t)i;
    for (int k = 0; k < b.cn(c); k++) {
      const size_t s = cslot(c, k);
      q[k] = adjoint ? (float)((double)m.c_esg[s] / m.e_dc[m.c_es[s]])  // gradPVn / ke / gravity adjoints
                     : (float)(m.c_vk[s] / m.c_area[c]);                // pv_vertex' -> pv_cell'
    }
    if (adjoint) {
      q[6] = (float)(1.0 / m.c_area[c]);
      q[7] = (float)m.c_area[c];
    }
  }
  if (!adjoint) {
    for (int i = 0; i < cnt[C_KE]; i++) {  // ke' coefficients 0.25 dcEdge dvEdge / areaCell
      const int c = C.list[i];
      float *q = flts(B_C2) + 8 * (size_t)i;
      for (int k = 0; k < b.cn(c); k++) {
        const int e = m.c_es[cslot(c, k)];
        q[k] = (float)(0.25 * m.e_dc[e] * m.e_dv[e] / m.c_area[c]);
      }
    }
    for (int i = 0; i < cnt[C_OWN]; i++) {  // thickness flux: sign dvEdge / areaCell
      const int c = C.list[i];
      float *q = flts(B_C3) + 8 * (size_t)i;
      for (int k = 0; k < b.cn(c); k++) {
        const size_t s = cslot(c, k);
        q[k] = (float)((double)m.c_esg[s] * m.e_dv[m.c_es[s]] / m.c_area[c]);
      }
    }
  } else {
    for (int i = 0; i < cnt[C_OWN]; i++) {  // owned cells: h_edge adjoint halves, kites
      const int c = C.list[i];
      float *q = flts(B_C2) + 16 * (size_t)i;
      for (int k = 0; k < b.cn(c); k++) {
        q[k] = 0.5f;
        q[6 + k] = (float)m.c_vk[cslot(c, k)];
      }
    }
  }
  for (int i = 0; i < cnt[E_MID]; i++) {
    const int e = E.list[i];
    float *q = flts(B_ECOEF) + (adjoint ? 24 : 12) * (size_t)i;
    for (int j = 0; j < kEoeSlots; j++) {
      q[j] = (float)m.e_w[(size_t)j * m.nE + e];  // zero past nEdgesOnEdge
      if (adjoint) q[10 + j] = (float)m.e_wrev[(size_t)j * m.nE + e];
    }
    if (!adjoint) {
      q[10] = (float)(1.0 / m.e_dv[e]);
      q[11] = (float)(1.0 / m.e_dc[e]);
    } else {
      q[20] = (float)m.e_dv[e];
      q[21] = (float)m.e_dc[e];
    }
  }
}

}  // namespace

// The local spaces of the tile that owns cells [c0, c1) and the edges whose lower-numbered cell
// is among them, layer by layer (TileLayer), into E, C, V; counts into cnt.
static void tile_spaces(const Builder &b, const BuiltMesh &m, int c0, int c1, bool adjoint, Space &E, Space &C,
                        Space &V, int *cnt) {
  for (int c = c0; c < c1; c++) C.add(c);
  cnt[C_OWN] = C.close();
  for (int c = c0; c < c1; c++)
    for (int k = 0; k < b.cn(c); k++) {
      const int e = b.ces(c, k), lo = std::min(m.e_c1[e], m.e_c2[e]);
      if (lo >= c0 && lo < c1) E.add(e);
    }
  cnt[E_OWN] = E.close();
  const std::vector<int> OE(E.list), OC(C.list);
  for (int e : OE) {
    C.add(m.e_c1[e]);
    C.add(m.e_c2[e]);
  }
  cnt[C_KE] = C.close();
  if (!adjoint) {
    for (int e : OE)
      for (int j = 0; j < m.e_n[e]; j++) E.add(b.eoe(e, j));
    cnt[E_MID] = E.close();
    for (int e : E.list) {
      C.add(m.e_c1[e]);
      C.add(m.e_c2[e]);
    }
    cnt[C_MID] = C.close();
    for (int c : C.list)
      for (int k = 0; k < b.cn(c); k++) V.add(b.cvs(c, k));
    for (int i = 0; i < cnt[E_MID]; i++) {
      V.add(m.e_v1[E.list[i]]);
      V.add(m.e_v2[E.list[i]]);
    }
    cnt[V_ALL] = V.close();
    for (int i = 0; i < cnt[E_MID]; i++)
      for (int j = 0; j < m.e_n[E.list[i]]; j++) E.add(b.eoe(E.list[i], j));
    for (int v : V.list)
      for (int k = 0; k < VDEG; k++) E.add(b.ves(v, k));
    for (int i = 0; i < cnt[C_KE]; i++)
      for (int k = 0; k < b.cn(C.list[i]); k++) E.add(b.ces(C.list[i], k));
    cnt[E_ALL] = E.close();
    for (int v : V.list)
      for (int k = 0; k < VDEG; k++) C.add(b.vc(v, k));
    for (int c : OC)
      for (int k = 0; k < b.cn(c); k++) C.add(b.cnb(c, k));
    cnt[C_ALL] = C.close();
  } else {
    for (int e : OE) {
      V.add(m.e_v1[e]);
      V.add(m.e_v2[e]);
    }
    for (int c : OC)
      for (int k = 0; k < b.cn(c); k++) V.add(b.cvs(c, k));
    cnt[V_ALL] = V.close();
    for (int v : V.list)
      for (int k = 0; k < VDEG; k++) C.add(b.vc(v, k));
    cnt[C_MID] = C.close();
    for (int e : OE)
      for (int j = 0; j < m.e_n[e]; j++) E.add(b.eoe(e, j));
    for (int c : C.list)
      for (int k = 0; k < b.cn(c); k++) E.add(b.ces(c, k));
    for (int v : V.list)
      for (int k = 0; k < VDEG; k++) E.add(b.ves(v, k));
    cnt[E_MID] = E.close();
    for (int i = 0; i < cnt[E_MID]; i++)
      for (int j = 0; j < m.e_n[E.list[i]]; j++) E.add(b.eoe(E.list[i], j));
    cnt[E_ALL] = E.close();
    for (int i = 0; i < cnt[E_MID]; i++) {
      C.add(m.e_c1[E.list[i]]);
      C.add(m.e_c2[E.list[i]]);
    }
    cnt[C_ALL] = C.close();
  }
}

// Shared memory of a tile's block with M members per chunk: blob, base values, member rows.
static size_t tile_smem(const int *cnt, bool adjoint, int M) {
  int off[kBlobSections];
  return (size_t)blob_layout(cnt, adjoint, off) + 4 * (size_t)base_floats(cnt, adjoint) +
         (size_t)member_rows(cnt, adjoint) * M * sizeof(float);
}

std::string build_tiles(const BuiltMesh &m, size_t budget, int kmax, int M, bool adjoint, TileSetHost *o) {
  if (kmax < 1) return "tile size must be positive";
  for (int c = 0; c < m.nC; c++)
    if (m.c_n[c] > kCellSlots) return "fused tiles need at most 6 edges per cell";
  for (int e = 0; e < m.nE; e++)
    if (m.e_n[e] > kEoeSlots) return "fused tiles need at most 10 edgesOnEdge";
  Builder b(m);
  const int nC = m.nC;
  int stamp = 0;  // a fresh id for each trial build of the spaces
  int cnt[kTileCounts];
  // shared memory of the tile [c0, c1) with M members per chunk
  auto fits = [&](int c0, int c1) {
    Space E(b.se, b.le, stamp), C(b.sc, b.lc, stamp), V(b.sv, b.lv, stamp);
    stamp++;
    tile_spaces(b, m, c0, c1, adjoint, E, C, V, cnt);
    return tile_smem(cnt, adjoint, M) <= budget && E.list.size() < kNoLocal && C.list.size() < kNoLocal &&
           V.list.size() < kNoLocal;
  };
  // partition the cells into runs of the internal order: each run as long as its tile's shared
  // memory stays within the budget (and at most kmax cells), so tiles near a jump of the
  // Hilbert curve, whose halo is larger, own fewer cells
  std::vector<int> bounds{0};
  while (bounds.back() < nC) {
    const int c0 = bounds.back(), hi = std::min(nC, c0 + kmax);
    if (!fits(c0, c0 + 1)) return fail((int)bounds.size() - 1, "one cell's halo exceeds the shared-memory budget");
    int ok = c0 + 1, step = 1;
    while (ok < hi) {  // grow geometrically, then bisect
      const int t = std::min(hi, ok + step);
      if (!fits(c0, t)) {
        int lo = ok, bad = t;
        while (bad - lo > 1) {
          const int mid = (lo + bad) / 2;
          (fits(c0, mid) ? lo : bad) = mid;
        }
        ok = lo;
        break;
      }
      ok = t;
      step *= 2;
    }
    bounds.push_back(ok);
  }
  const int ntiles = (int)bounds.size() - 1;
  *o = TileSetHost();
  o->K = kmax;
  o->ntiles = ntiles;
  o->cnt.assign((size_t)ntiles * kTileCounts, 0);
  o->off.assign((size_t)ntiles * 3, 0);
  o->blob_off.assign(ntiles, 0);
  for (int t = 0; t < ntiles; t++) {
    Space E(b.se, b.le, stamp), C(b.sc, b.lc, stamp), V(b.sv, b.lv, stamp);
    stamp++;
    int *tc = &o->cnt[(size_t)t * kTileCounts];
    tile_spaces(b, m, bounds[t], bounds[t + 1], adjoint, E, C, V, tc);
    if (!validate(b, m, E, C, V, tc, adjoint)) return fail(t, "a phase of the fused stage would read outside its tile");
    for (int k = 0; k < kTileCounts; k++) o->max_cnt[k] = std::max(o->max_cnt[k], tc[k]);
    int *off = &o->off[(size_t)t * 3];
    off[0] = (int)o->ge.size();
    off[1] = (int)o->gc.size();
    off[2] = (int)o->gv.size();
    o->ge.insert(o->ge.end(), E.list.begin(), E.list.end());
    o->gc.insert(o->gc.end(), C.list.begin(), C.list.end());
    o->gv.insert(o->gv.end(), V.list.begin(), V.list.end());
    o->blob_off[t] = (long long)o->blob.size();
    pack_blob(b, m, E, C, V, tc, adjoint, &o->blob);
    for (int i = 0; i < 4; i++) o->smem[i] = std::max(o->smem[i], tile_smem(tc, adjoint, 4 << i));
  }
  return "";
}

// ---- tiles of the nonlinear stage (mpsw_stage.h) ------------------------------------------------
namespace {

// Layers of the tile owning cells [c0, c1): the tangent-linear layers, with the owned vertices
// first among the vertices.
void stage_spaces(const Builder &b, const BuiltMesh &m, int c0, int c1, Space &E, Space &C, Space &V, int *n) {
  for (int c = c0; c < c1; c++)
    for (int k = 0; k < b.cn(c); k++) {
      const int v = b.cvs(c, k);
      if (std::min(b.vc(v, 0), std::min(b.vc(v, 1), b.vc(v, 2))) == c) V.add(v);
    }
  n[S_VO] = V.close();
  int cnt[kTileCounts];
  tile_spaces(b, m, c0, c1, false, E, C, V, cnt);
  n[S_EO] = cnt[E_OWN]; n[S_EM] = cnt[E_MID]; n[S_EA] = cnt[E_ALL];
  n[S_CO] = cnt[C_OWN]; n[S_CK] = cnt[C_KE]; n[S_CM] = cnt[C_MID]; n[S_CA] = cnt[C_ALL];
  n[S_VA] = cnt[V_ALL];
}

// Every neighbour a phase reads is in the layer it is formed on.
bool stage_valid(const Builder &b, const BuiltMesh &m, const Space &E, const Space &C, const Space &V, const int *n) {
  auto in = [](int x, int hi) { return x >= 0 && x < hi; };
  for (int v : V.list)
    for (int k = 0; k < VDEG; k++)
      if (!in(E.local(b.ves(v, k)), n[S_EA]) || !in(C.local(b.vc(v, k)), n[S_CA])) return false;
  for (int i = 0; i < n[S_CM]; i++) {
    const int c = C.list[i];
    for (int k = 0; k < b.cn(c); k++) {
      if (!in(E.local(b.ces(c, k)), n[S_EA]) || !in(V.local(b.cvs(c, k)), n[S_VA])) return false;
      if (i < n[S_CK] && !in(E.local(m.c_eoc[(size_t)k * m.nC + c]), n[S_EA])) return false;
      if (i < n[S_CO] && !in(C.local(b.cnb(c, k)), n[S_CA])) return false;
    }
  }
  for (int i = 0; i < n[S_EM]; i++) {
    const int e = E.list[i];
    const bool own = i < n[S_EO];
    for (int c : {m.e_c1[e], m.e_c2[e]}) {
      if (!in(C.local(c), own ? n[S_CK] : n[S_CM])) return false;
      if (own)  // del4: delsq_u on every edge of the cell
        for (int k = 0; k < b.cn(c); k++)
          if (!in(E.local(b.ces(c, k)), n[S_EM])) return false;
    }
    for (int v : {m.e_v1[e], m.e_v2[e]}) {
      if (!in(V.local(v), n[S_VA])) return false;
      if (own)
        for (int k = 0; k < VDEG; k++)
          if (!in(E.local(b.ves(v, k)), n[S_EM])) return false;
    }
    for (int j = 0; j < m.e_n[e]; j++)
      if (!in(E.local(b.eoe(e, j)), own ? n[S_EM] : n[S_EA])) return false;
  }
  return true;
}

// One tile's blob with values of type R (stage_layout).
template <typename R>
void stage_pack(const Builder &b, const BuiltMesh &m, const Space &E, const Space &C, const Space &V, const int *n,
                std::vector<unsigned char> *blob) {
  int off[kStageSections];
  const int size = stage_layout(n, (int)sizeof(R), off);
  const size_t base = blob->size();
  blob->resize(base + (size_t)size, 0);
  unsigned char *p = blob->data() + base;
  // entry k of entity i's list, and value k after `lists` list chunks, in a section of cnt records
  auto list = [&](int sec, int cnt, int i, int k, int x) {
    reinterpret_cast<uint16_t *>(p + off[sec] + 16 * ((k >> 3) * cnt + i))[k & 7] = (uint16_t)(x * (int)sizeof(R));
  };
  constexpr int per = 16 / (int)sizeof(R);
  auto divisor = [](double x) { return sizeof(R) == 4 ? R(1) / R(x) : R(x); };
  auto val = [&](int sec, int cnt, int lists, int i, int k, R x) {
    reinterpret_cast<R *>(p + off[sec] + 16 * ((lists + k / per) * cnt + i))[k % per] = x;
  };
  const int nv = n[S_VA], ncm = n[S_CM], nck = n[S_CK], nco = n[S_CO], nem = n[S_EM];
  for (int i = 0; i < nv; i++) {
    const int v = V.list[i];
    for (int k = 0; k < VDEG; k++) {
      const size_t s = (size_t)k * m.nV + v;
      list(SB_V, nv, i, k, E.local(m.v_es[s]));
      list(SB_V, nv, i, 3 + k, C.local(m.v_c[s]));
      val(SB_V, nv, 1, i, k, R(m.v_esg[s]) * R(m.e_dc[m.v_es[s]]));
      val(SB_V, nv, 1, i, 3 + k, R(m.v_k[s]));
    }
    val(SB_V, nv, 1, i, 6, divisor(m.v_area[v]));
    val(SB_V, nv, 1, i, 7, R(m.v_f[v]));
  }
  for (int i = 0; i < ncm; i++) {
    const int c = C.list[i];
    for (int k = 0; k < kCellSlots; k++) {
      const bool has = k < b.cn(c);  // a padded slot: the first slot's neighbours, weight 0
      const size_t s = (size_t)(has ? k : 0) * m.nC + c;
      if (i < nco) list(SB_CO, nco, i, k, C.local(b.cnb(c, has ? k : 0)));
      list(SB_CM, ncm, i, k, V.local(m.c_vs[s]));
      list(SB_CX, ncm, i, k, E.local(m.c_es[s]));
      if (i < nck) list(SB_CK, nck, i, k, E.local(m.c_eoc[s]));
      if (!has) continue;
      val(SB_CM, ncm, 1, i, k, R(m.c_vk[s]));
      val(SB_CX, ncm, 1, i, k, R(m.c_esg[s]) * R(m.e_dv[m.c_es[s]]));
      if (i < nck) {
        const int e = m.c_eoc[s];
        val(SB_CK, nck, 1, i, k, (R(0.25) * R(m.e_dc[e])) * R(m.e_dv[e]));
      }
    }
    val(SB_CM, ncm, 1, i, 6, divisor(m.c_area[c]));
    if (i < nck) val(SB_CK, nck, 1, i, 6, R(m.c_hs[c]));
  }
  for (int i = 0; i < nem; i++) {
    const int e = E.list[i];
    list(SB_E, nem, i, 0, C.local(m.e_c1[e]));
    list(SB_E, nem, i, 1, C.local(m.e_c2[e]));
    list(SB_E, nem, i, 2, V.local(m.e_v1[e]));
    list(SB_E, nem, i, 3, V.local(m.e_v2[e]));
    for (int j = 0; j < kEoeSlots; j++) {
      const bool has = j < m.e_n[e];  // a padded slot weighs nothing
      list(SB_E, nem, i, 4 + j, m.e_n[e] ? E.local(b.eoe(e, has ? j : 0)) : i);
      val(SB_E, nem, 2, i, j, has ? R(m.e_w[(size_t)j * m.nE + e]) : R(0));
    }
    val(SB_E, nem, 2, i, 10, divisor(m.e_dc[e]));
    val(SB_E, nem, 2, i, 11, divisor(m.e_dv[e]));
  }
  std::memcpy(p + off[SB_GE], E.list.data(), 4 * E.list.size());
  std::memcpy(p + off[SB_GC], C.list.data(), 4 * C.list.size());
  std::memcpy(p + off[SB_GV], V.list.data(), 4 * (size_t)nv);
}

// Cut the cells into runs and append one tile a run: one(b, stamp, c0, K, out) appends the tile of cells
// [c0, c0 + K) and returns null, or kTooLarge, or what keeps the mesh from being tiled.  A run that is
// too large is cut by 1 / shrink until it fits; neighbouring runs fit at like sizes, so the next one starts
// three sizes above the last.  Four parts of the cells, whole multiples of kmax, are cut side by side (level 6,
// both sets of tiles, eight cores: 865 -> 350 ms).
const char *const kTooLarge = "one cell's halo exceeds a tile";

template <class One>
std::string build_runs(const BuiltMesh &m, int kmax, int shrink, StageSetHost *o, One &&one) {
  std::vector<int> sizes(1, kmax);
  while (sizes.back() > 1) {
    const int K = sizes.back();
    sizes.push_back(std::max(1, K - (K + shrink - 1) / shrink));
  }
  const int tiles = (m.nC + kmax - 1) / kmax, parts = std::min(tiles, 4), len = (tiles + parts - 1) / parts * kmax;
  std::vector<StageSetHost> set(parts);
  std::vector<std::string> err(parts);
  auto cut = [&](int p) {
    Builder b(m);
    StageSetHost &out = set[p];
    const int end = (int)std::min<long long>(m.nC, (long long)(p + 1) * len);
    size_t at = 0;
    int stamp = 0;
    for (int c0 = p * len; c0 < end;) {
      const int left = end - c0;
      at -= std::min<size_t>(at, 3);
      while (at + 1 < sizes.size() && sizes[at + 1] >= left) at++;  // (sizes beyond what is left are one)
      const char *why;
      while ((why = one(b, stamp++, c0, std::min(sizes[at], left), &out)) == kTooLarge && at + 1 < sizes.size()) at++;
      if (why) {
        err[p] = why == kTooLarge ? why : fail(out.ntiles, why);
        return;
      }
      out.ntiles++;
      c0 += std::min(sizes[at], left);
    }
  };
  in_turns(parts, cut);
  *o = StageSetHost();
  for (const std::string &e : err)
    if (!e.empty()) return e;
  size_t n64 = 0, n32 = 0;
  for (const StageSetHost &t : set) {
    n64 += t.blob64.size();
    n32 += t.blob32.size();
  }
  o->blob64.reserve(n64);
  o->blob32.reserve(n32);
  for (StageSetHost &t : set) {
    for (long long x : t.off64) o->off64.push_back(x + (long long)o->blob64.size());
    for (long long x : t.off32) o->off32.push_back(x + (long long)o->blob32.size());
    o->cnt.insert(o->cnt.end(), t.cnt.begin(), t.cnt.end());
    o->blob64.insert(o->blob64.end(), t.blob64.begin(), t.blob64.end());
    o->blob32.insert(o->blob32.end(), t.blob32.begin(), t.blob32.end());
    o->ntiles += t.ntiles;
    t = StageSetHost();
  }
  return "";
}

std::string narrow_lists(const BuiltMesh &m) {
  for (int c = 0; c < m.nC; c++)
    if (m.c_n[c] > kCellSlots) return "stage tiles need at most 6 edges per cell";
  for (int e = 0; e < m.nE; e++)
    if (m.e_n[e] > kEoeSlots) return "stage tiles need at most 10 edgesOnEdge";
  return "";
}

}  // namespace

std::string build_stage_tiles(const BuiltMesh &m, int kmax, StageSetHost *o) {
  if (kmax < 1) return "tile size must be positive";
  const std::string wide = narrow_lists(m);
  if (!wide.empty()) return wide;
  return build_runs(m, kmax, 5, o, [&](Builder &b, int stamp, int c0, int K, StageSetHost *out) -> const char * {
    int n[kStageCounts];
    Space E(b.se, b.le, stamp), C(b.sc, b.lc, stamp), V(b.sv, b.lv, stamp);
    stage_spaces(b, m, c0, c0 + K, E, C, V, n);
    if (!stage_fits(n)) return kTooLarge;
    if (!stage_valid(b, m, E, C, V, n)) return "a phase of the stage would read outside its tile";
    out->cnt.insert(out->cnt.end(), n, n + kStageCounts);
    out->off64.push_back((long long)out->blob64.size());
    out->off32.push_back((long long)out->blob32.size());
    stage_pack<double>(b, m, E, C, V, n, &out->blob64);
    stage_pack<float>(b, m, E, C, V, n, &out->blob32);
    return nullptr;
  });
}

// ---- tiles of the FP64 adjoint stage (mpsw_stage.h) -----------------------------------------------
namespace {

void stage_ad_pack(const Builder &b, const BuiltMesh &m, const Space &E, const Space &C, const Space &V, const int *n,
                   std::vector<unsigned char> *blob) {
  int off[kStageAdSections];
  const int size = stage_ad_layout(n, off);
  const size_t base = blob->size();
  blob->resize(base + (size_t)size, 0);
  unsigned char *p = blob->data() + base;
  auto list = [&](int sec, int cnt, int i, int k, int x) {
    reinterpret_cast<uint16_t *>(p + off[sec] + 16 * ((k >> 3) * cnt + i))[k & 7] = (uint16_t)(8 * std::max(x, 0));
  };
  auto val = [&](int sec, int cnt, int lists, int i, int k, double x) {
    reinterpret_cast<double *>(p + off[sec] + 16 * ((lists + k / 2) * cnt + i))[k % 2] = x;
  };
  const int nv = n[V_ALL], ncm = n[C_MID], nco = n[C_OWN], nem = n[E_MID];
  for (int i = 0; i < nv; i++) {
    const int v = V.list[i];
    for (int k = 0; k < VDEG; k++) {
      const size_t s = (size_t)k * m.nV + v;
      list(YB_V, nv, i, k, E.local(m.v_es[s]));
      list(YB_V, nv, i, 3 + k, C.local(m.v_c[s]));
      list(YB_V, nv, i, 6 + k, E.local(m.v_e[s]));
      val(YB_V, nv, 2, i, k, m.v_esg[s]);
      val(YB_V, nv, 2, i, 3 + k, m.v_k[s] / m.c_area[m.v_c[s]]);
    }
    val(YB_V, nv, 2, i, 6, m.v_area[v]);
    val(YB_V, nv, 2, i, 7, m.v_f[v]);
  }
  for (int i = 0; i < ncm; i++) {
    const int c = C.list[i];
    for (int k = 0; k < kCellSlots; k++) {
      const bool has = k < b.cn(c);  // (as above)
      const size_t s = (size_t)(has ? k : 0) * m.nC + c;
      list(YB_C, ncm, i, k, E.local(m.c_es[s]));
      if (i < nco) list(YB_O, nco, i, k, V.local(m.c_vs[s]));
      if (!has) continue;
      val(YB_C, ncm, 1, i, k, m.c_esg[s]);
      if (i < nco) val(YB_O, nco, 1, i, k, m.c_vk[s]);
    }
    val(YB_C, ncm, 1, i, 6, m.c_area[c]);
    if (i < nco) val(YB_O, nco, 1, i, 6, m.c_area[c]);
  }
  for (int i = 0; i < nem; i++) {
    const int e = E.list[i];
    list(YB_E, nem, i, 0, C.local(m.e_c1[e]));
    list(YB_E, nem, i, 1, C.local(m.e_c2[e]));
    list(YB_E, nem, i, 2, V.local(m.e_v1[e]));  // (read for owned edges only)
    list(YB_E, nem, i, 3, V.local(m.e_v2[e]));
    for (int j = 0; j < kEoeSlots; j++) {
      const bool has = j < m.e_n[e];  // a padded slot weighs nothing
      list(YB_E, nem, i, 4 + j, m.e_n[e] ? E.local(b.eoe(e, has ? j : 0)) : i);
      val(YB_E, nem, 2, i, j, has ? m.e_w[(size_t)j * m.nE + e] : 0.0);
      val(YB_E, nem, 2, i, 10 + j, has ? m.e_wrev[(size_t)j * m.nE + e] : 0.0);
    }
    val(YB_E, nem, 2, i, 20, m.e_dc[e]);
    val(YB_E, nem, 2, i, 21, m.e_dv[e]);
  }
  std::memcpy(p + off[YB_GE], E.list.data(), 4 * E.list.size());
  std::memcpy(p + off[YB_GC], C.list.data(), 4 * C.list.size());
  std::memcpy(p + off[YB_GV], V.list.data(), 4 * V.list.size());
}

}  // namespace

std::string build_stage_ad_tiles(const BuiltMesh &m, int kmax, StageSetHost *o) {
  if (kmax < 1) return "tile size must be positive";
  const std::string wide = narrow_lists(m);
  if (!wide.empty()) return wide;
  return build_runs(m, kmax, 8, o, [&](Builder &b, int stamp, int c0, int K, StageSetHost *out) -> const char * {
    int n[kTileCounts];
    Space E(b.se, b.le, stamp), C(b.sc, b.lc, stamp), V(b.sv, b.lv, stamp);
    tile_spaces(b, m, c0, c0 + K, true, E, C, V, n);
    if (!stage_ad_fits(n)) return kTooLarge;
    if (!validate(b, m, E, C, V, n, true)) return "a phase of the stage would read outside its tile";
    out->cnt.insert(out->cnt.end(), n, n + kTileCounts);
    out->off64.push_back((long long)out->blob64.size());
    stage_ad_pack(b, m, E, C, V, n, &out->blob64);
    return nullptr;
  });
}

}  // namespace mpsw

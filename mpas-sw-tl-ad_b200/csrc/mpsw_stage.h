// Nonlinear RK stage on halo tiles: the tile's data layout and the per-entity arithmetic of each
// phase (mpsw_stage.cuh runs the phases in a thread block, one kernel per stage; a host loop can
// run the same functions).
//
// A tile owns a run of cells of the internal order, the edges whose lower-numbered cell it owns
// and the vertices whose lowest-numbered cell it owns.  Its local spaces are numbered in nested
// layers (owned first, then what the owned tendencies need), so that every phase works on a
// prefix.  All of the mesh a stage reads for the tile is packed into one blob of records, one per
// entity.  Values are combined in the reference's order, entity by entity
// (src/mpas_sw_dyncore.f90:95-361, 468-637), so FP64 results do not depend on the tiling.
#pragma once

#include <cmath>
#include <cstddef>

#include "mpsw_internal.h"

namespace mpsw {

// Prefix sizes of a tile's local spaces: owned edges | edges whose pv_edge is formed (owned and
// their edgesOnEdge) | edges whose u is read; owned cells | cells of owned edges (and owned) |
// cells whose pv_cell is formed | cells whose h is read; owned vertices | all vertices.
enum StageCount { S_EO, S_EM, S_EA, S_CO, S_CK, S_CM, S_CA, S_VO, S_VA, kStageCounts };

// Most entities of each layer (the builder shortens a tile until it fits): the values that the
// phases exchange then have fixed places in shared memory, and neighbour lists hold byte offsets
// into them, so a gather is one unpack and one load.  The pv_edge layer is also at most the
// threads of a block, which keep one edge's record in registers through the phases.
constexpr int kStageThreads = 448;
constexpr int kCapEM = 384, kCapEA = 672, kCapCO = 96, kCapCK = 128, kCapCM = 192, kCapCA = 256, kCapVA = 400;

// A tile fits when its layers do, and when the kinds of entities a phase forms side by side get
// threads of their own, in whole warps: vertices and ke cells, edges and pv_cell cells, edges and
// owned cells.
MPSW_HD inline int stage_up32(int x) { return (x + 31) & ~31; }
MPSW_HD inline bool stage_fits(const int *n) {
  return n[S_EM] <= kCapEM && n[S_EA] <= kCapEA && n[S_CO] <= kCapCO && n[S_CK] <= kCapCK && n[S_CM] <= kCapCM &&
         n[S_CA] <= kCapCA && n[S_VA] <= kCapVA && stage_up32(n[S_VA]) + n[S_CK] <= kStageThreads &&
         stage_up32(n[S_EM]) + stage_up32(n[S_CM]) <= kStageThreads &&
         stage_up32(n[S_EM]) + stage_up32(n[S_CO]) <= kStageThreads;
}

// Values exchanged between the phases: offsets in values from the start of the work area.
enum StageWork {
  W_U = 0,
  W_H = W_U + kCapEA,
  W_PVV = W_H + kCapCA,
  W_PC = W_PVV + kCapVA,
  W_KE = W_PC + kCapCM,
  W_HS = W_KE + kCapCK,
  W_PE = W_HS + kCapCK,
  W_HE = W_PE + kCapEM,
  W_VORT = W_HE + kCapEM,  // from here: with viscosity
  W_DIV = W_VORT + kCapVA,
  W_DSQ = W_DIV + kCapCM,  // from here: with del4
  W_V4 = W_DSQ + kCapEM,
  W_C4 = W_V4 + kCapVA,
  W_END = W_C4 + kCapCK
};
MPSW_HD inline int stage_work(int r, bool visc, bool del4) { return r * (del4 ? W_END : visc ? W_DSQ : W_VORT); }

// A tangent-linear stage exchanges the same values of the member, after the linearisation point's
// u, h_edge (all edges) and pv_edge (pv_edge layer): negative offsets from the work area.
enum StageTlWork { T_UB = -(2 * kCapEA + kCapEM), T_HB = T_UB + kCapEA, T_PB = T_HB + kCapEA, kTlBase = -T_UB };
static_assert(kTlBase % 2 == 0, "the records behind start on 16 bytes");

// A blob: per entity a record of 16-byte chunks, stored chunk by chunk ([chunk][n]), first chunk(s)
// the neighbour list as byte offsets into the work arrays, then values in the stencils' precision.
//   vertices:       edges[3] cells[3]; sign dcEdge [3], kites [3], area, f
//   pv_cell cells:  vertices[6]; kites [6], area
//   the same cells: edges[6] in the scatter order; sign dvEdge [6]
//   ke cells:       edges[6] in the cell's order; (dcEdge / 4) dvEdge [6], h_s
//   owned cells:    cells across [6]
//   pv_edge edges:  c1 c2 v1 v2 as local indices, edgesOnEdge[10]; weights [10], dc, dv
// Areas and lengths are divisors: FP64 records hold them, FP32 ones their reciprocals (stage_over).
// The edge records come last and go to registers; what is before them goes to shared memory.
// Slots past a list weigh zero and repeat its first entry, so that a NaN there spreads no further.
enum StageSection { SB_V, SB_CM, SB_CX, SB_CK, SB_CO, SB_E, SB_GE, SB_GC, SB_GV, kStageSections };

MPSW_HD inline int stage_chunks(int vals, int r) { return (vals * r + 15) / 16; }
constexpr int kValsV = 8, kValsCM = 7, kValsCX = 6, kValsCK = 7, kValsE = 12;

// Byte offsets of a blob's sections for values of `r` bytes; returns the blob's size.
MPSW_HD inline int stage_layout(const int *n, int r, int *off) {
  int o = 0;
  off[SB_V] = o; o += 16 * n[S_VA] * (1 + stage_chunks(kValsV, r));
  off[SB_CM] = o; o += 16 * n[S_CM] * (1 + stage_chunks(kValsCM, r));
  off[SB_CX] = o; o += 16 * n[S_CM] * (1 + stage_chunks(kValsCX, r));
  off[SB_CK] = o; o += 16 * n[S_CK] * (1 + stage_chunks(kValsCK, r));
  off[SB_CO] = o; o += 16 * n[S_CO];
  off[SB_E] = o; o += 16 * n[S_EM] * (2 + stage_chunks(kValsE, r));
  off[SB_GE] = o; o += (4 * n[S_EA] + 15) / 16 * 16;
  off[SB_GC] = o; o += (4 * n[S_CA] + 15) / 16 * 16;
  off[SB_GV] = o; o += (4 * n[S_VA] + 15) / 16 * 16;
  return o;
}

// 16 bytes of a record
struct alignas(16) StageChunk {
  unsigned w[4];
};
// entry k of a neighbour list held in chunks
MPSW_HD inline int stage_at(const StageChunk *c, int k) {
  const unsigned w = c[k >> 3].w[(k & 7) >> 1];
  return (int)((k & 1) ? w >> 16 : w & 0xFFFFu);
}
// A record in registers: L chunks of lists and NV values.
template <typename R, int L, int NV>
struct StageRec {
  static constexpr int kChunks = (NV * (int)sizeof(R) + 15) / 16;
  StageChunk list[L];
  union {
    StageChunk raw[kChunks > 0 ? kChunks : 1];
    R v[(kChunks > 0 ? kChunks : 1) * 16 / sizeof(R)];
  };
  MPSW_HD StageRec() {}
  MPSW_HD int at(int k) const { return stage_at(list, k); }
};
// the record of entity i, from a section's first chunk; n: records a chunk row holds
template <typename R, int L, int NV>
MPSW_HD inline void stage_rec(const StageChunk *p, int n, int i, StageRec<R, L, NV> *r) {
#pragma unroll
  for (int k = 0; k < L; k++) r->list[k] = p[k * n + i];
#pragma unroll
  for (int k = 0; k < StageRec<R, L, NV>::kChunks; k++) r->raw[k] = p[(L + k) * n + i];
}
template <typename R>
using VertexRec = StageRec<R, 1, kValsV>;
template <typename R>
using CellMRec = StageRec<R, 1, kValsCM>;
template <typename R>
using CellXRec = StageRec<R, 1, kValsCX>;
template <typename R>
using CellKRec = StageRec<R, 1, kValsCK>;
template <typename R>
using EdgeRec = StageRec<R, 2, kValsE>;

// a over a divisor of a record.  (FP64 divides: multiplying by a stored reciprocal and correcting
// to the rounded quotient measured slower here, 7.4 against 6.8 us a level-5 stage.)
template <typename R>
MPSW_HD inline R stage_over(R a, R d) {
  return sizeof(R) == 4 ? a * d : a / d;
}

// value at byte offset b of the work array that starts at value `first`
template <typename R>
MPSW_HD inline R &stage_val(unsigned char *w, int first, int b) {
  return *reinterpret_cast<R *>(w + first * (int)sizeof(R) + b);
}

// Where a stage's linearisation point goes (any may be null): u, h_edge, v, gradPVt, gradPVn,
// pv_edge on edges, vorticity, h_vertex on vertices, ke on cells, in FP64 and / or rounded to FP32.
struct StageBaseOut {
  double *d[9];
  float *f[9];
  int on;  // any of them
};
enum StageBaseField { SO_U, SO_HE, SO_V, SO_GPT, SO_GPN, SO_PE, SO_VORT, SO_HV, SO_KE };

// One stage: input state, RK bookkeeping, optional tendencies and linearisation point.
template <typename R, typename A>
struct StageArgs {
  const R *u, *h;  // h is stored relative to off
  R off;
  Phys<R> ph;
  RK<R, A> rku, rkh;
  R *tend_u, *tend_h;
  StageBaseOut out;
  const R *sc2, *sc4, *usrc;  // edge scalings of del2 / del4, wind source
};

MPSW_HD inline void stage_put(const StageBaseOut &o, int f, int g, double x) {
  if (o.d[f]) o.d[f][g] = x;
  if (o.f[f]) o.f[f][g] = (float)x;
}

// The functions below form entity i of a tile from its record; w: the work area; g: the internal
// index where the tile owns the entity, else -1.

// ---- phase 1: vertices (:208-219, :282-292) ----------------------------------------------------
template <typename R, typename A>
MPSW_HD inline void stage_vertex(const VertexRec<R> &r, unsigned char *w, const StageArgs<R, A> &a, int i, int g,
                                 bool visc) {
  R circ = R(0), hv = R(0);
#pragma unroll
  for (int k = 0; k < VDEG; k++) circ = circ + r.v[k] * stage_val<R>(w, W_U, r.at(k));
  const R area = r.v[6];
  const R vort = stage_over(circ, area);
#pragma unroll
  for (int k = 0; k < VDEG; k++) hv = hv + (stage_val<R>(w, W_H, r.at(3 + k)) + a.off) * r.v[3 + k];
  hv = stage_over(hv, area);
  stage_val<R>(w, W_PVV + i, 0) = (r.v[7] + vort) / hv;
  if (visc) stage_val<R>(w, W_VORT + i, 0) = vort;
  if (g >= 0) {
    stage_put(a.out, SO_VORT, g, vort);
    stage_put(a.out, SO_HV, g, hv);
  }
}

// RK bookkeeping of one value (src/mpas_sw_module.f90:590-611); x0 / acc: rk.x0 and rk.acc_in there
template <typename R, typename A>
MPSW_HD inline void stage_rk(const RK<R, A> &rk, int g, R t, A x0, A acc) {
  if (rk.next) rk.next[g] = rk.frozen ? R(x0) : R((x0 - A(rk.off)) + rk.c * A(t));
  if (rk.acc_out && !rk.frozen) rk.acc_out[g] = acc + rk.w * A(t);
}

// ---- phase 1: kinetic energy (:245-256) ----------------------------------------------------------
template <typename R, typename A>
MPSW_HD inline void stage_ke(const CellKRec<R> &r, R area, unsigned char *w, const StageArgs<R, A> &a, int i, int g) {
  R ke = R(0);
#pragma unroll
  for (int k = 0; k < 6; k++) {
    const R u = stage_val<R>(w, W_U, r.at(k));
    ke = ke + r.v[k] * (u * u);
  }
  ke = stage_over(ke, area);
  stage_val<R>(w, W_KE + i, 0) = ke;
  stage_val<R>(w, W_HS + i, 0) = r.v[6];
  if (g >= 0) stage_put(a.out, SO_KE, g, ke);
}
// divergence, where viscosity needs it (:222-242)
template <typename R>
MPSW_HD inline void stage_div(const CellXRec<R> &r, R area, unsigned char *w, int i) {
  R div = R(0);
#pragma unroll
  for (int k = 0; k < 6; k++) div = div + r.v[k] * stage_val<R>(w, W_U, r.at(k));
  stage_val<R>(w, W_DIV + i, 0) = div * stage_over(R(1), area);
}
// ---- phase 3: thickness tendency of an owned cell and its RK update (:468-482) ---------------------
template <typename R, typename A>
MPSW_HD inline void stage_thick(const CellXRec<R> &r, const StageChunk &across, R area, unsigned char *w, const StageArgs<R, A> &a,
                                int i, int g, A x0, A acc) {
  const R hc = stage_val<R>(w, W_H + i, 0) + a.off;
  R th = R(0);
#pragma unroll
  for (int k = 0; k < 6; k++) {
    const R he = R(0.5) * (hc + (stage_val<R>(w, W_H, stage_at(&across, k)) + a.off));
    th = th - (stage_val<R>(w, W_U, r.at(k)) * r.v[k]) * he;
  }
  th = stage_over(th, area);
  if (a.tend_h) a.tend_h[g] = th;
  stage_rk(a.rkh, g, th, x0, acc);
}

// ---- phase 2: tangential velocity (:259-267), pv_cell (:324-340) -----------------------------------
template <typename R>
MPSW_HD inline R stage_perp(const EdgeRec<R> &r, unsigned char *w) {
  R v = R(0);
#pragma unroll
  for (int j = 0; j < 10; j++) v = v + r.v[j] * stage_val<R>(w, W_U, r.at(4 + j));
  return v;
}
template <typename R>
MPSW_HD inline void stage_pvcell(const CellMRec<R> &r, unsigned char *w, int i) {
  R pc = R(0);
#pragma unroll
  for (int k = 0; k < 6; k++) {
    const R pv = stage_val<R>(w, W_PVV, r.at(k));
    if constexpr (sizeof(R) == 4) pc = pc + (r.v[k] * r.v[6]) * pv;
    else pc = pc + (r.v[k] * pv) / r.v[6];
  }
  stage_val<R>(w, W_PC + i, 0) = pc;
}

// ---- phase 3: gradients of pv (:296-301), pv_edge (:305-320, :344-359), h_edge (:95-105) and
// delsq_u (:539-551); v: the tangential velocity of phase 2 --------------------------------------------
template <typename R, typename A>
MPSW_HD inline void stage_edge(const EdgeRec<R> &r, unsigned char *w, const StageArgs<R, A> &a, int i, int g, R v,
                               bool del4) {
  const int c1 = r.at(0), c2 = r.at(1), v1 = r.at(2), v2 = r.at(3);
  const R dc = r.v[10], dv = r.v[11], u = stage_val<R>(w, W_U + i, 0);
  const R pv1 = stage_val<R>(w, W_PVV, v1), pv2 = stage_val<R>(w, W_PVV, v2);
  const R gpt = stage_over(pv2 - pv1, dv);
  R pe = R(0);
  pe = pe + R(0.5) * pv1;
  pe = pe + R(0.5) * pv2;
  pe = pe - ((a.ph.apvm * v) * a.ph.dt) * gpt;
  const R gpn = stage_over(stage_val<R>(w, W_PC, c2) - stage_val<R>(w, W_PC, c1), dc);
  pe = pe - ((a.ph.apvm * u) * a.ph.dt) * gpn;
  const R he = R(0.5) * ((stage_val<R>(w, W_H, c1) + a.off) + (stage_val<R>(w, W_H, c2) + a.off));
  stage_val<R>(w, W_PE + i, 0) = pe;
  stage_val<R>(w, W_HE + i, 0) = sizeof(R) == 4 ? u * he : he;  // FP32 stencils keep the thickness flux
  if (del4)
    stage_val<R>(w, W_DSQ + i, 0) = stage_over(stage_val<R>(w, W_DIV, c2) - stage_val<R>(w, W_DIV, c1), dc) -
                                    stage_over(stage_val<R>(w, W_VORT, v2) - stage_val<R>(w, W_VORT, v1), dv);
  if (g >= 0) {
    stage_put(a.out, SO_U, g, u);
    stage_put(a.out, SO_HE, g, he);
    stage_put(a.out, SO_V, g, v);
    stage_put(a.out, SO_GPT, g, gpt);
    stage_put(a.out, SO_GPN, g, gpn);
    stage_put(a.out, SO_PE, g, pe);
  }
}

// ---- del4 (:554-589): delsq_vorticity on the vertices, delsq_divergence on the cells of owned
// edges; entities whose neighbours lie outside the pv_edge layer are read by no owned edge -------
template <typename R>
MPSW_HD inline void stage_del4_vertex(const VertexRec<R> &r, unsigned char *w, int i, int nem) {
  R circ = R(0);
#pragma unroll
  for (int k = 0; k < VDEG; k++) {
    if (r.at(k) >= nem * (int)sizeof(R)) return;
    circ = circ + r.v[k] * stage_val<R>(w, W_DSQ, r.at(k));
  }
  stage_val<R>(w, W_V4 + i, 0) = circ * stage_over(R(1), r.v[6]);
}
template <typename R>
MPSW_HD inline void stage_del4_cell(const CellXRec<R> &r, R area, unsigned char *w, int i, int nem) {
  R div = R(0);
#pragma unroll
  for (int k = 0; k < 6; k++) {
    if (r.at(k) >= nem * (int)sizeof(R)) return;
    div = div + r.v[k] * stage_val<R>(w, W_DSQ, r.at(k));
  }
  stage_val<R>(w, W_C4 + i, 0) = div * stage_over(R(1), area);
}

// ---- phase 4: normal-velocity tendency of an owned edge (:485-637) and its RK update -----------
template <typename R, typename A>
MPSW_HD inline void stage_tend(const EdgeRec<R> &r, unsigned char *w, const StageArgs<R, A> &a, int i, int g, A x0,
                               A acc) {
  const R pee = stage_val<R>(w, W_PE + i, 0);
  R q = R(0);
#pragma unroll
  for (int j = 0; j < 10; j++) {
    const int e = r.at(4 + j);
    const R wpv = R(0.5) * (pee + stage_val<R>(w, W_PE, e));
    if constexpr (sizeof(R) == 4) q = q + (r.v[j] * stage_val<R>(w, W_HE, e)) * wpv;
    else q = q + ((r.v[j] * stage_val<R>(w, W_U, e)) * wpv) * stage_val<R>(w, W_HE, e);
  }
  const int c1 = r.at(0), c2 = r.at(1), v1 = r.at(2), v2 = r.at(3);
  const R dc = r.v[10], dv = r.v[11];
  const R h1 = stage_val<R>(w, W_H, c1), h2 = stage_val<R>(w, W_H, c2);
  const R s1 = stage_val<R>(w, W_HS, c1), s2 = stage_val<R>(w, W_HS, c2);
  R grav;
  if constexpr (sizeof(R) == 8) grav = R(GRAVITY) * ((((h2 + a.off) + s2) - (h1 + a.off)) - s1);
  else grav = R(GRAVITY) * ((h2 - h1) + (s2 - s1));  // difference the offset-free values first
  const R ke1 = stage_val<R>(w, W_KE, c1), ke2 = stage_val<R>(w, W_KE, c2);
  R tu = q - stage_over((ke2 - ke1) + grav, dc);
  if (a.ph.visc2 > R(0)) {
    R ud = stage_over(stage_val<R>(w, W_DIV, c2) - stage_val<R>(w, W_DIV, c1), dc) -
           stage_over(stage_val<R>(w, W_VORT, v2) - stage_val<R>(w, W_VORT, v1), dv);
    ud = (a.sc2[g] * a.ph.visc2) * ud;
    tu = tu + ud;
  }
  if (a.ph.visc4 > R(0)) {
    R ud = stage_over(stage_val<R>(w, W_C4, c2) - stage_val<R>(w, W_C4, c1), dc) -
           stage_over(stage_val<R>(w, W_V4, v2) - stage_val<R>(w, W_V4, v1), dv);
    ud = (a.sc4[g] * a.ph.visc4) * ud;
    tu = tu - ud;
  }
  const R hee = R(0.5) * ((h1 + a.off) + (h2 + a.off));
  if (a.ph.wind) tu = tu + (a.usrc[g] / R(RHO_REF)) / hee;
  if (a.ph.drag) {
    const R kee = R(0.5) * (ke1 + ke2);
    tu = tu - ((R(1.0e-3) * stage_val<R>(w, W_U + i, 0)) * sqrt(R(2) * kee)) / hee;
  }
  if (a.ph.bad && !(tu - tu == R(0))) *a.ph.bad = 1;  // NaN or infinite
  if (a.tend_u) a.tend_u[g] = tu;
  stage_rk(a.rku, g, tu, x0, acc);
}

// ---- tangent-linear stage of one FP64 member (src/mpas_sw_dyncore_tlm.f90), in the operation order
// of the member kernels: the same phases on the same tiles -----------------------------------------
struct StageTlArgs {
  const double *u, *h;  // the member's stage input, rows of B members
  int B;
  Base<double> bs;
  Phys<double> ph;
  RK<double, double> rku, rkh;
  double *tend_u, *tend_h;
  const double *sc2, *sc4, *usrc;
};

// :255-271, :344-360; hv, vort: the linearisation point's
MPSW_HD inline void stage_tl_vertex(const VertexRec<double> &r, unsigned char *w, int i, double hv, double vort_b,
                                    bool visc) {
  double circ = 0.0, hvt = 0.0;
#pragma unroll
  for (int k = 0; k < VDEG; k++) circ = circ + r.v[k] * stage_val<double>(w, W_U, r.at(k));
  const double vort = circ / r.v[6];
#pragma unroll
  for (int k = 0; k < VDEG; k++) hvt = hvt + stage_val<double>(w, W_H, r.at(3 + k)) * r.v[3 + k];
  hvt = hvt / r.v[6];
  stage_val<double>(w, W_PVV + i, 0) = vort / hv - (hvt * (r.v[7] + vort_b)) / (hv * hv);
  if (visc) stage_val<double>(w, W_VORT + i, 0) = vort;
}
// ke' (:274-316)
MPSW_HD inline void stage_tl_ke(const CellKRec<double> &r, double area, unsigned char *w, int i) {
  double ke = 0.0;
#pragma unroll
  for (int k = 0; k < 6; k++)
    ke = ke + r.v[k] * ((2.0 * stage_val<double>(w, T_UB, r.at(k))) * stage_val<double>(w, W_U, r.at(k)));
  stage_val<double>(w, W_KE + i, 0) = ke / area;
}
// tend_h' of an owned cell (:541-561)
MPSW_HD inline double stage_tl_thick(const CellXRec<double> &r, const StageChunk &across, double area, unsigned char *w,
                                     int i) {
  const double hc = stage_val<double>(w, W_H + i, 0);
  double th = 0.0;
#pragma unroll
  for (int k = 0; k < 6; k++) {
    const double het = 0.5 * (hc + stage_val<double>(w, W_H, stage_at(&across, k)));
    th = th - ((stage_val<double>(w, W_U, r.at(k)) * r.v[k]) * stage_val<double>(w, T_HB, r.at(k)) +
               (stage_val<double>(w, T_UB, r.at(k)) * r.v[k]) * het);
  }
  return th / area;
}
// pv_edge', h_edge' and delsq_u' (:364-393, 425-445, 117-126, 638-652); vt: the tangential velocity;
// vb, gpt, gpn: the linearisation point's at the edge
MPSW_HD inline void stage_tl_edge(const EdgeRec<double> &r, unsigned char *w, const Phys<double> &ph, int i, double vt,
                                  double vb, double gpt, double gpn, bool del4) {
  const int c1 = r.at(0), c2 = r.at(1), v1 = r.at(2), v2 = r.at(3);
  const double dc = r.v[10], dv = r.v[11], u = stage_val<double>(w, W_U + i, 0), ub = stage_val<double>(w, T_UB + i, 0);
  const double pv1 = stage_val<double>(w, W_PVV, v1), pv2 = stage_val<double>(w, W_PVV, v2);
  const double gptt = (pv2 - pv1) / dv;
  double pet = 0.0;
  pet = pet + 0.5 * pv1;
  pet = pet + 0.5 * pv2;
  pet = pet - ((ph.apvm * vt) * ph.dt) * gpt - ((ph.apvm * vb) * ph.dt) * gptt;
  const double gpnt = (stage_val<double>(w, W_PC, c2) - stage_val<double>(w, W_PC, c1)) / dc;
  pet = pet - ((ph.apvm * u) * ph.dt) * gpn - ((ph.apvm * ub) * ph.dt) * gpnt;
  stage_val<double>(w, W_PE + i, 0) = pet;
  stage_val<double>(w, W_HE + i, 0) = 0.5 * (stage_val<double>(w, W_H, c1) + stage_val<double>(w, W_H, c2));
  if (del4)
    stage_val<double>(w, W_DSQ + i, 0) = (stage_val<double>(w, W_DIV, c2) - stage_val<double>(w, W_DIV, c1)) / dc -
                                         (stage_val<double>(w, W_VORT, v2) - stage_val<double>(w, W_VORT, v1)) / dv;
}
// tend_u' of an owned edge (:564-768); gc: internal indices of the tile's cells
MPSW_HD inline double stage_tl_tend(const EdgeRec<double> &r, unsigned char *w, const StageTlArgs &a, const int *gc,
                                    int i, int g) {
  const double pet = stage_val<double>(w, W_PE + i, 0), pe = stage_val<double>(w, T_PB + i, 0);
  double qt = 0.0;
#pragma unroll
  for (int j = 0; j < 10; j++) {
    const int e = r.at(4 + j);
    const double wt = r.v[j];
    const double wpvt = 0.5 * (pet + stage_val<double>(w, W_PE, e)), wpv = 0.5 * (pe + stage_val<double>(w, T_PB, e));
    const double ub = stage_val<double>(w, T_UB, e), heb = stage_val<double>(w, T_HB, e);
    qt = qt + ((wt * stage_val<double>(w, W_U, e)) * wpv) * heb + ((wt * ub) * wpvt) * heb +
         ((wt * ub) * wpv) * stage_val<double>(w, W_HE, e);
  }
  const int c1 = r.at(0), c2 = r.at(1), v1 = r.at(2), v2 = r.at(3);
  const double dc = r.v[10], dv = r.v[11], h1 = stage_val<double>(w, W_H, c1), h2 = stage_val<double>(w, W_H, c2);
  const double ke1 = stage_val<double>(w, W_KE, c1), ke2 = stage_val<double>(w, W_KE, c2);
  const double grad = (ke2 - ke1) + GRAVITY * (h2 - h1);
  double tut = qt - grad / dc;
  if (a.ph.visc2 > 0.0) {
    double ud = (stage_val<double>(w, W_DIV, c2) - stage_val<double>(w, W_DIV, c1)) / dc -
                (stage_val<double>(w, W_VORT, v2) - stage_val<double>(w, W_VORT, v1)) / dv;
    ud = (a.sc2[g] * a.ph.visc2) * ud;
    tut = tut + ud;
  }
  if (a.ph.visc4 > 0.0) {
    double ud = (stage_val<double>(w, W_C4, c2) - stage_val<double>(w, W_C4, c1)) / dc -
                (stage_val<double>(w, W_V4, v2) - stage_val<double>(w, W_V4, v1)) / dv;
    ud = (a.sc4[g] * a.ph.visc4) * ud;
    tut = tut - ud;
  }
  const double hh = stage_val<double>(w, T_HB + i, 0), het = 0.5 * (h1 + h2);
  if (a.ph.wind) tut = tut - ((het * a.usrc[g]) / RHO_REF) / (hh * hh);
  if (a.ph.drag) {
    const double ket = 0.5 * (ke1 + ke2), ke = 0.5 * (a.bs.ke[gc[c1 / 8]] + a.bs.ke[gc[c2 / 8]]);
    const double uu = stage_val<double>(w, T_UB + i, 0), sq = sqrt(2.0 * ke);
    tut = tut - ((1.0e-3 * stage_val<double>(w, W_U + i, 0)) * sq) / hh -
          ((((0.5 * 1.0e-3) * uu) * (2.0 * ket)) / sq) / hh + (((1.0e-3 * uu) * sq) * het) / (hh * hh);
  }
  return tut;
}

// ---- adjoint stage of one FP64 member (src/mpas_sw_dyncore_adj.f90), no viscosity and no drag ------
// Tiles of their own, with the fused adjoint stage's layers (TileLayer): each phase gathers what the phase
// before formed, edges (E_MID) -> cells (C_MID) -> vertices (V_ALL) -> owned edges and cells.
constexpr int kAdThreads = 384;  // one a pv_edge layer edge
constexpr int kAdEM = 384, kAdEA = 672, kAdCO = 96, kAdCM = 160, kAdCA = 256, kAdVA = 256;
MPSW_HD inline bool stage_ad_fits(const int *n) {
  return n[E_MID] <= kAdEM && n[E_ALL] <= kAdEA && n[C_OWN] <= kAdCO && n[C_MID] <= kAdCM && n[C_ALL] <= kAdCA &&
         n[V_ALL] <= kAdVA && stage_up32(n[E_OWN]) + stage_up32(n[C_OWN]) <= kAdThreads;
}

// Values in shared memory: u, h_edge, pv_edge of the linearisation point and the tendency adjoints; per
// edge the adjoints of pv_edge and h_edge, gradPVn_ad / dc, tu / dc, g / dc tu, gradPVt_ad / dv, v_ad;
// pv_cell_ad, ke_ad / area, h_ad on cells; h_vertex_ad and circulation_ad on vertices.
enum StageAdWork {
  Y_UB = 0,
  Y_HB = Y_UB + kAdEA,
  Y_PB = Y_HB + kAdEA,
  Y_TU = Y_PB + kAdEA,
  Y_TH = Y_TU + kAdEA,
  Y_PE = Y_TH + kAdCA,
  Y_HE = Y_PE + kAdEM,
  Y_GN = Y_HE + kAdEM,
  Y_TD = Y_GN + kAdEM,
  Y_TG = Y_TD + kAdEM,
  Y_GT = Y_TG + kAdEM,
  Y_VA = Y_GT + kAdEM,
  Y_PC = Y_VA + kAdEM,
  Y_KE = Y_PC + kAdCM,
  Y_HD = Y_KE + kAdCM,
  Y_HV = Y_HD + kAdCM,
  Y_CI = Y_HV + kAdVA,
  Y_END = Y_CI + kAdVA
};
static_assert(Y_END % 2 == 0, "the records behind start on 16 bytes");

// A blob, records as above:
//   vertices:     edges[3] cells[3] edgesOnVertex[3]; sign [3], kite / areaCell [3], area, f
//   C_MID cells:  edges[6]; sign [6] (0 past the list), area
//   owned cells:  vertices[6]; kite / areaTriangle [6], area
//   E_MID edges:  c1 c2 v1 v2 edgesOnEdge[10]; weights [10], transposed weights [10], dc, dv
enum StageAdSection { YB_V, YB_C, YB_O, YB_E, YB_GE, YB_GC, YB_GV, kStageAdSections };
constexpr int kAdValsV = 8, kAdValsC = 7, kAdValsO = 7, kAdValsE = 22;
constexpr int kAdRowsV = 6, kAdRowsC = 5, kAdRowsO = 5;  // chunk rows
MPSW_HD inline int stage_ad_layout(const int *n, int *off) {
  int o = 0;
  off[YB_V] = o; o += 16 * n[V_ALL] * kAdRowsV;
  off[YB_C] = o; o += 16 * n[C_MID] * kAdRowsC;
  off[YB_O] = o; o += 16 * n[C_OWN] * kAdRowsO;
  off[YB_E] = o; o += 16 * n[E_MID] * (2 + stage_chunks(kAdValsE, 8));
  off[YB_GE] = o; o += (4 * n[E_ALL] + 15) / 16 * 16;
  off[YB_GC] = o; o += (4 * n[C_ALL] + 15) / 16 * 16;
  off[YB_GV] = o; o += (4 * n[V_ALL] + 15) / 16 * 16;
  return o;
}
using AdVertexRec = StageRec<double, 2, kAdValsV>;
using AdCellRec = StageRec<double, 1, kAdValsC>;
using AdEdgeRec = StageRec<double, 2, kAdValsE>;

struct StageAdArgs {
  AdIn<double> in;  // rows of B members
  int B;
  Base<double> bs;
  Phys<double> ph;
  AdOut<double, double> out;
  const double *usrc;
};

// (:689-736, :567-572, :193-200, :235-242); returns the edge's direct share of u_ad
MPSW_HD inline double stage_ad_edge(const AdEdgeRec &r, unsigned char *w, const StageAdArgs &a, int i, double vb,
                                    double gpt, double gpn, double usrc) {
  const double Te = stage_val<double>(w, Y_TU + i, 0), ue = stage_val<double>(w, Y_UB + i, 0);
  const double hee = stage_val<double>(w, Y_HB + i, 0), pee = stage_val<double>(w, Y_PB + i, 0);
  const double dc = r.v[20], dv = r.v[21];
  double pe = 0.0, he = 0.0, ud = 0.0;
#pragma unroll
  for (int j = 0; j < 10; j++) {
    const int e = r.at(4 + j);
    const double wt = r.v[j], wr = r.v[10 + j], Tn = stage_val<double>(w, Y_TU, e);
    pe = pe + 0.5 * (((wt * stage_val<double>(w, Y_UB, e)) * stage_val<double>(w, Y_HB, e)) * Te);
    const double wpv = 0.5 * (stage_val<double>(w, Y_PB, e) + pee);
    he = he + ((wr * ue) * wpv) * Tn;
    pe = pe + 0.5 * (((wr * ue) * hee) * Tn);
    ud = ud + ((wr * wpv) * hee) * Tn;
  }
  const double fa = stage_val<double>(w, Y_TH, r.at(1)) - stage_val<double>(w, Y_TH, r.at(0));
  he = he + (ue * dv) * fa;
  ud = ud + (dv * hee) * fa;
  if (a.ph.wind) he = he - ((usrc / RHO_REF) / (hee * hee)) * Te;
  const double gn = 0.0 - ((a.ph.apvm * ue) * a.ph.dt) * pe;
  ud = ud - ((a.ph.apvm * a.ph.dt) * gpn) * pe;
  const double gt = 0.0 - ((a.ph.apvm * vb) * a.ph.dt) * pe;
  stage_val<double>(w, Y_PE + i, 0) = pe;
  stage_val<double>(w, Y_HE + i, 0) = he;
  stage_val<double>(w, Y_GN + i, 0) = gn / dc;
  stage_val<double>(w, Y_TD + i, 0) = Te / dc;
  stage_val<double>(w, Y_TG + i, 0) = (GRAVITY / dc) * Te;
  stage_val<double>(w, Y_GT + i, 0) = gt / dv;
  stage_val<double>(w, Y_VA + i, 0) = 0.0 - ((a.ph.apvm * a.ph.dt) * gpt) * pe;
  return ud;
}
// (:202-213, :696-699, :358-369, :306-317)
MPSW_HD inline void stage_ad_cell(const AdCellRec &r, unsigned char *w, int i) {
  double pc = 0.0, ke = 0.0, hd = 0.0;
#pragma unroll
  for (int k = 0; k < 6; k++) {
    const int e = r.at(k);
    const double sg = r.v[k];
    pc = pc + (-sg) * stage_val<double>(w, Y_GN, e);
    ke = ke + sg * stage_val<double>(w, Y_TD, e);
    hd = hd + sg * stage_val<double>(w, Y_TG, e);
    hd = hd + (0.5 * fabs(sg)) * stage_val<double>(w, Y_HE, e);
  }
  stage_val<double>(w, Y_PC + i, 0) = pc;
  stage_val<double>(w, Y_KE + i, 0) = ke / r.v[6];
  stage_val<double>(w, Y_HD + i, 0) = hd;
}
// (:215-229, :244-262, :268-284, :343-349); hv, vort: the linearisation point's
MPSW_HD inline void stage_ad_vertex(const AdVertexRec &r, unsigned char *w, int i, double hv, double vort) {
  double pv = 0.0, vo = 0.0, hva = 0.0;
#pragma unroll
  for (int k = 0; k < VDEG; k++) pv = pv + r.v[3 + k] * stage_val<double>(w, Y_PC, r.at(3 + k));
#pragma unroll
  for (int k = 0; k < VDEG; k++) pv = pv + 0.5 * stage_val<double>(w, Y_PE, r.at(6 + k));
#pragma unroll
  for (int k = 0; k < VDEG; k++) pv = pv + r.v[k] * stage_val<double>(w, Y_GT, r.at(k));
  hva = hva - ((r.v[7] + vort) / (hv * hv)) * pv;
  vo = vo + pv / hv;
  stage_val<double>(w, Y_HV + i, 0) = hva / r.v[6];
  stage_val<double>(w, Y_CI + i, 0) = 0.0 + vo / r.v[6];
}
// (:296-317, :350-355); ud: stage_ad_edge's, ub: the linearisation point's u
MPSW_HD inline double stage_ad_final(const AdEdgeRec &r, unsigned char *w, double ud, double ub) {
  double pu = ud;
#pragma unroll
  for (int j = 0; j < 10; j++) pu = pu + r.v[10 + j] * stage_val<double>(w, Y_VA, r.at(4 + j));
  const double dc = r.v[20], dv = r.v[21], kc = (((0.25 * dc) * dv) * 2.0) * ub;
  pu = pu + kc * stage_val<double>(w, Y_KE, r.at(0));
  pu = pu + kc * stage_val<double>(w, Y_KE, r.at(1));
  pu = pu + dc * stage_val<double>(w, Y_CI, r.at(3));
  pu = pu - dc * stage_val<double>(w, Y_CI, r.at(2));
  return pu;
}
// (:286-289)
MPSW_HD inline double stage_ad_thick(const AdCellRec &r, unsigned char *w, int i) {
  double h = stage_val<double>(w, Y_HD + i, 0);
#pragma unroll
  for (int k = 0; k < 6; k++) h = h + r.v[k] * stage_val<double>(w, Y_HV, r.at(k));
  return h;
}

}  // namespace mpsw

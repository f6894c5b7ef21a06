// One nonlinear RK stage as one kernel over halo tiles (layout and arithmetic: mpsw_stage.h).
//
// A single trajectory is bound by latency: run as four grid-wide passes (vertices, cells, edge
// diagnostics, edge tendencies) a stage cost 4.5 us a pass on the level-5 mesh whatever the
// pass computed, launch, ramp-up and a chain of index -> value loads from L2.  Here a block
// computes the whole stage for its tile: the passes become phases separated by block barriers,
// their indirect loads go to shared memory, and the halo is recomputed (about 1.7 times the owned
// edges) instead of exchanged through another launch.  The blob is mesh data, which no kernel
// writes, so fetching it runs before the wait for the previous stage and overlaps that stage; the
// next stage's blocks are let in at once for the same reason.
#pragma once

#include "mpsw_fused.cuh"
#include "mpsw_stage.h"

namespace mpsw {

// Records of a tile in shared memory, after the work values: rows of a section's capacity, so that
// every address but the entity's is a constant.
template <typename R>
struct StageShared {
  static constexpr int row(int cap, int vals) { return 16 * cap * (1 + (vals * (int)sizeof(R) + 15) / 16); }
  static constexpr int V = 0, CM = V + row(kCapVA, kValsV), CX = CM + row(kCapCM, kValsCM),
                       CK = CX + row(kCapCM, kValsCX), CO = CK + row(kCapCK, kValsCK), END = CO + row(kCapCO, 0);
  // chunk rows of the sections, in the order V CM CX CK CO
  static constexpr int rows(int vals) { return 1 + (vals * (int)sizeof(R) + 15) / 16; }
  static constexpr int RV = rows(kValsV), RCM = RV + rows(kValsCM), RCX = RCM + rows(kValsCX),
                       RCK = RCX + rows(kValsCK), RCO = RCK + 1;
  static_assert(RCO <= 32, "one lane of a warp copies each chunk row");
};
template <typename R>
inline size_t stage_smem(bool visc, bool del4) {
  return (size_t)stage_work((int)sizeof(R), visc, del4) + StageShared<R>::END;
}
inline size_t stage_tl_smem(bool visc, bool del4) { return 8 * kTlBase + stage_smem<double>(visc, del4); }

__device__ __forceinline__ unsigned smem_addr(const void *p) { return (unsigned)__cvta_generic_to_shared(p); }

// Start the copies of a tile's records (blob g) into shared memory, one bulk copy per chunk row.
template <typename R>
__device__ __forceinline__ void stage_fetch(unsigned char *rec, const unsigned char *g, const int *n, const int *off,
                                            bool visc, unsigned long long *arrived) {
  using S = StageShared<R>;
  const int tid = threadIdx.x;
  if (tid < 32) {  // one bulk copy per chunk row of the records
    const int ncx = visc ? n[S_CM] : n[S_CO];
    if (tid == 0) {
      asm volatile("mbarrier.init.shared.b64 [%0], 1;" ::"r"(smem_addr(arrived)) : "memory");
      asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
      const int bytes = 16 * (S::RV * n[S_VA] + (S::RCM - S::RV) * n[S_CM] + (S::RCX - S::RCM) * ncx +
                              (S::RCK - S::RCX) * n[S_CK] + n[S_CO]);
      asm volatile("mbarrier.arrive.expect_tx.shared.b64 _, [%0], %1;" ::"r"(smem_addr(arrived)), "r"(bytes)
                   : "memory");
    }
    __syncwarp();
    if (tid < S::RCO) {
      const int k = tid < S::RV ? 0 : tid < S::RCM ? 1 : tid < S::RCX ? 2 : tid < S::RCK ? 3 : 4;
      const int first = k == 0 ? 0 : k == 1 ? S::RV : k == 2 ? S::RCM : k == 3 ? S::RCX : S::RCK;
      const int cnt = k == 0 ? n[S_VA] : k == 1 || k == 2 ? n[S_CM] : k == 3 ? n[S_CK] : n[S_CO];
      const int cap = k == 0 ? kCapVA : k == 1 || k == 2 ? kCapCM : k == 3 ? kCapCK : kCapCO;
      const int dst = k == 0 ? S::V : k == 1 ? S::CM : k == 2 ? S::CX : k == 3 ? S::CK : S::CO;
      const int src = k == 0 ? off[SB_V] : k == 1 ? off[SB_CM] : k == 2 ? off[SB_CX] : k == 3 ? off[SB_CK] : off[SB_CO];
      asm volatile(
          "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
              smem_addr(rec + dst + 16 * cap * (tid - first))),
          "l"(g + src + 16 * cnt * (tid - first)), "r"(16 * (k == 2 ? ncx : cnt)), "r"(smem_addr(arrived))
          : "memory");
    }
  }
}

// Wait for them (they were issued a stage ago; a bound all the same).  The same answer for every
// thread; false: they did not arrive.
__device__ __forceinline__ bool stage_arrived(unsigned long long *arrived) {
  unsigned ok = 0;
  for (int i = 0; i < (1 << 20) && !ok; i++)
    asm volatile("{\n.reg .pred p;\nmbarrier.try_wait.parity.shared.b64 p, [%1], 0;\nselp.u32 %0, 1, 0, p;\n}"
                 : "=r"(ok)
                 : "r"(smem_addr(arrived))
                 : "memory");
  return !__syncthreads_or(!ok);
}

template <typename R, typename A>
__global__ void __launch_bounds__(kStageThreads, 2) k_stage(StageDev ts, StageArgs<R, A> a) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ __align__(8) unsigned long long arrived;
  using S = StageShared<R>;
  constexpr int NT = kStageThreads;
  const int tid = threadIdx.x;
  const bool del4 = a.ph.visc4 > R(0), visc = del4 || a.ph.visc2 > R(0);
  unsigned char *const w = smem_raw, *const rec = smem_raw + stage_work((int)sizeof(R), visc, del4);
  int n[kStageCounts], off[kStageSections];
#pragma unroll
  for (int k = 0; k < kStageCounts; k++) n[k] = __ldg(ts.cnt + (size_t)blockIdx.x * kStageCounts + k);
  stage_layout(n, (int)sizeof(R), off);
  const unsigned char *g = ts.blob + __ldg(ts.blob_off + blockIdx.x);
  stage_fetch<R>(rec, g, n, off, visc, &arrived);
  auto sec = [&](int o) { return reinterpret_cast<const StageChunk *>(rec + o); };
  EdgeRec<R> er;
  if (tid < n[S_EM]) stage_rec(reinterpret_cast<const StageChunk *>(g + off[SB_E]), n[S_EM], tid, &er);
  const int *ids = reinterpret_cast<const int *>(g + off[SB_GE]), *idc = reinterpret_cast<const int *>(g + off[SB_GC]);
  int ge[2] = {0, 0}, gc = 0;
  if (tid < n[S_EA]) ge[0] = __ldg(ids + tid);
  if (tid + NT < n[S_EA]) ge[1] = __ldg(ids + tid + NT);
  if (tid < n[S_CA]) gc = __ldg(idc + tid);
  // owned edges belong to the first threads, owned cells to the last (top counts from the end)
  const int top = NT - 1 - tid;
  const bool edge = tid < n[S_EO], cell = top < n[S_CO];
  const int own = edge ? ge[0] : cell ? __ldg(idc + top) : -1;
  asm volatile("griddepcontrol.wait;" ::: "memory");
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  // the state on the tile (each value once: past L1) and what the thread's owned entity adds to
  A x0 = A(0), acc = A(0);
  {
    R u0 = R(0), u1 = R(0), h = R(0);  // in flight together
    if (tid < n[S_EA]) u0 = __ldcg(a.u + ge[0]);
    if (tid + NT < n[S_EA]) u1 = __ldcg(a.u + ge[1]);
    if (tid < n[S_CA]) h = __ldcg(a.h + gc);
    if (edge || cell) {
      const RK<R, A> &rk = edge ? a.rku : a.rkh;
      if (rk.next) x0 = __ldcg(rk.x0 + own);
      if (rk.acc_out) acc = __ldcg(rk.acc_in + own);
    }
    if (tid < n[S_EA]) stage_val<R>(w, W_U + tid, 0) = u0;
    if (tid + NT < n[S_EA]) stage_val<R>(w, W_U + tid + NT, 0) = u1;
    if (tid < n[S_CA]) stage_val<R>(w, W_H + tid, 0) = h;
  }
  __syncthreads();  // (also: the barrier's initialisation is visible)
  if (!stage_arrived(&arrived)) {
    if (a.ph.bad) *a.ph.bad = 1;
    return;
  }
  // phase 1: vertices; from the next warp on, ke cells (with viscosity also the other divergences)
  const int nv32 = stage_up32(n[S_VA]);
  if (tid < n[S_VA]) {
    VertexRec<R> r;
    stage_rec(sec(S::V), kCapVA, tid, &r);
    const int gv = a.out.on && tid < n[S_VO] ? __ldg(reinterpret_cast<const int *>(g + off[SB_GV]) + tid) : -1;
    stage_vertex(r, w, a, tid, gv, visc);
  } else if (tid >= nv32) {
    for (int i = tid - nv32; i < (visc ? n[S_CM] : n[S_CK]); i += NT - nv32) {
      CellMRec<R> m;
      stage_rec(sec(S::CM), kCapCM, i, &m);
      if (i < n[S_CK]) {
        CellKRec<R> r;
        stage_rec(sec(S::CK), kCapCK, i, &r);
        stage_ke(r, m.v[6], w, a, i, a.out.on && i < n[S_CO] ? __ldg(idc + i) : -1);
      }
      if (visc) {
        CellXRec<R> r;
        stage_rec(sec(S::CX), kCapCM, i, &r);
        stage_div(r, m.v[6], w, i);
      }
    }
  }
  __syncthreads();
  // phase 2: tangential velocity of the pv_edge layer; pv_cell on the last threads
  R v = R(0);
  if (tid < n[S_EM]) {
    v = stage_perp(er, w);
  } else if (top < n[S_CM]) {
    CellMRec<R> r;
    stage_rec(sec(S::CM), kCapCM, top, &r);
    stage_pvcell(r, w, top);
  }
  __syncthreads();
  // phase 3: pv_edge; thickness of the owned cells on the last threads
  if (tid < n[S_EM]) {
    stage_edge(er, w, a, tid, a.out.on && edge ? own : -1, v, del4);
  } else if (cell) {
    CellMRec<R> m;
    CellXRec<R> r;
    stage_rec(sec(S::CM), kCapCM, top, &m);
    stage_rec(sec(S::CX), kCapCM, top, &r);
    stage_thick(r, sec(S::CO)[top], m.v[6], w, a, top, own, x0, acc);
  }
  __syncthreads();
  if (del4) {
    if (tid < n[S_VA]) {
      VertexRec<R> r;
      stage_rec(sec(S::V), kCapVA, tid, &r);
      stage_del4_vertex(r, w, tid, n[S_EM]);
    } else if (tid - nv32 >= 0 && tid - nv32 < n[S_CK]) {
      const int i = tid - nv32;
      CellXRec<R> r;
      CellMRec<R> m;
      stage_rec(sec(S::CX), kCapCM, i, &r);
      stage_rec(sec(S::CM), kCapCM, i, &m);
      stage_del4_cell(r, m.v[6], w, i, n[S_EM]);
    }
    __syncthreads();
  }
  // phase 4
  if (edge) stage_tend(er, w, a, tid, own, x0, acc);
}

// RK bookkeeping of one value of a member sweep (rk_members with one member)
struct StageTlRk {
  double x0 = 0.0, t[3] = {0.0, 0.0, 0.0}, acc = 0.0;
  __device__ __forceinline__ void fetch(const RK<double, double> &rk, size_t o) {
    const bool last = rk.t_in[0] != nullptr;
    if ((rk.next && !last) || last) x0 = __ldcg(rk.x0 + o);
    if (last) {
#pragma unroll
      for (int j = 0; j < 3; j++) t[j] = __ldcg(rk.t_in[j] + o);
    } else if (!rk.t_out && rk.acc_out) {
      acc = __ldcg(rk.acc_in + o);
    }
  }
  __device__ __forceinline__ void put(const RK<double, double> &rk, size_t o, double x) const {
    const bool last = rk.t_in[0] != nullptr;
    if (rk.next && !last) rk.next[o] = rk.frozen ? x0 : x0 + rk.c * x;
    if (rk.frozen) return;
    if (rk.t_out) {
      rk.t_out[o] = x;
    } else if (last) {
      double a = x0;
#pragma unroll
      for (int j = 0; j < 3; j++) a = a + rk.wt[j] * t[j];
      a = a + rk.w * x;
      rk.acc_out[o] = a;
      if (rk.next) rk.next[o] = a;
    } else if (rk.acc_out) {
      rk.acc_out[o] = acc + rk.w * x;
    }
  }
};

// A tangent-linear stage of FP64 members, one a block (blockIdx.y), phase by phase as k_stage and, like
// it, bound by the chain of phases rather than by bytes or arithmetic.  early: the linearisation point is
// stored, so its values, like the mesh, are fetched before the wait for the stage before; two blocks
// stay on an SM (106 KB each, 110 with del2 viscosity), so that the next stage's fetch overlaps this one;
// del4 takes 118 KB and leaves one.  At one block an SM without viscosity: 13.4 instead of 10.0 us a level-5
// stage; the four passes took 24.5 (stages of a window sweep of one member).
template <typename R>  // double
__global__ void __launch_bounds__(kStageThreads, 2) k_stage_tl(StageDev ts, StageTlArgs a, int early) {
  static_assert(sizeof(R) == 8);
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ __align__(8) unsigned long long arrived;
  using S = StageShared<double>;
  constexpr int NT = kStageThreads;
  const int tid = threadIdx.x, B = a.B, mb = blockIdx.y;
  const bool del4 = a.ph.visc4 > 0.0, visc = del4 || a.ph.visc2 > 0.0;
  unsigned char *const w = smem_raw + 8 * kTlBase, *const rec = w + stage_work(8, visc, del4);
  int n[kStageCounts], off[kStageSections];
#pragma unroll
  for (int k = 0; k < kStageCounts; k++) n[k] = __ldg(ts.cnt + (size_t)blockIdx.x * kStageCounts + k);
  stage_layout(n, 8, off);
  const unsigned char *g = ts.blob + __ldg(ts.blob_off + blockIdx.x);
  stage_fetch<double>(rec, g, n, off, visc, &arrived);
  auto sec = [&](int o) { return reinterpret_cast<const StageChunk *>(rec + o); };
  EdgeRec<double> er;
  if (tid < n[S_EM]) stage_rec(reinterpret_cast<const StageChunk *>(g + off[SB_E]), n[S_EM], tid, &er);
  const int *ids = reinterpret_cast<const int *>(g + off[SB_GE]), *idc = reinterpret_cast<const int *>(g + off[SB_GC]);
  int ge[2] = {0, 0}, gc = 0, gv = 0;
  if (tid < n[S_EA]) ge[0] = __ldg(ids + tid);
  if (tid + NT < n[S_EA]) ge[1] = __ldg(ids + tid + NT);
  if (tid < n[S_CA]) gc = __ldg(idc + tid);
  if (tid < n[S_VA]) gv = __ldg(reinterpret_cast<const int *>(g + off[SB_GV]) + tid);
  const int top = NT - 1 - tid;
  const bool edge = tid < n[S_EO], cell = top < n[S_CO];
  const int own = edge ? ge[0] : cell ? __ldg(idc + top) : 0;
  double hv = 0.0, vo = 0.0, vb = 0.0, gpt = 0.0, gpn = 0.0;
  auto base = [&]() {
    double u0 = 0.0, u1 = 0.0, h0 = 0.0, h1 = 0.0, p0 = 0.0;
    if (tid < n[S_EA]) {
      u0 = __ldcg(a.bs.u + ge[0]);
      h0 = __ldcg(a.bs.he + ge[0]);
    }
    if (tid + NT < n[S_EA]) {
      u1 = __ldcg(a.bs.u + ge[1]);
      h1 = __ldcg(a.bs.he + ge[1]);
    }
    if (tid < n[S_EM]) {
      p0 = __ldcg(a.bs.pe + ge[0]);
      vb = __ldcg(a.bs.v + ge[0]);
      gpt = __ldcg(a.bs.gpt + ge[0]);
      gpn = __ldcg(a.bs.gpn + ge[0]);
    }
    if (tid < n[S_VA]) {
      hv = __ldcg(a.bs.hv + gv);
      vo = __ldcg(a.bs.vort + gv);
    }
    if (tid < n[S_EA]) {
      stage_val<double>(w, T_UB + tid, 0) = u0;
      stage_val<double>(w, T_HB + tid, 0) = h0;
    }
    if (tid + NT < n[S_EA]) {
      stage_val<double>(w, T_UB + tid + NT, 0) = u1;
      stage_val<double>(w, T_HB + tid + NT, 0) = h1;
    }
    if (tid < n[S_EM]) stage_val<double>(w, T_PB + tid, 0) = p0;
  };
  if (early) base();
  pdl_begin();
  if (!early) base();
  StageTlRk rk;
  {
    double u0 = 0.0, u1 = 0.0, h = 0.0;  // in flight together
    if (tid < n[S_EA]) u0 = __ldcg(a.u + (size_t)ge[0] * B + mb);
    if (tid + NT < n[S_EA]) u1 = __ldcg(a.u + (size_t)ge[1] * B + mb);
    if (tid < n[S_CA]) h = __ldcg(a.h + (size_t)gc * B + mb);
    if (edge || cell) rk.fetch(edge ? a.rku : a.rkh, (size_t)own * B + mb);
    if (tid < n[S_EA]) stage_val<double>(w, W_U + tid, 0) = u0;
    if (tid + NT < n[S_EA]) stage_val<double>(w, W_U + tid + NT, 0) = u1;
    if (tid < n[S_CA]) stage_val<double>(w, W_H + tid, 0) = h;
  }
  __syncthreads();
  if (!stage_arrived(&arrived)) {
    if (a.ph.bad) *a.ph.bad = 1;
    return;
  }
  // phase 1: vertices; from the next warp on, ke cells (with viscosity also the divergences)
  const int nv32 = stage_up32(n[S_VA]);
  if (tid < n[S_VA]) {
    VertexRec<double> r;
    stage_rec(sec(S::V), kCapVA, tid, &r);
    stage_tl_vertex(r, w, tid, hv, vo, visc);
  } else if (tid >= nv32) {
    for (int i = tid - nv32; i < (visc ? n[S_CM] : n[S_CK]); i += NT - nv32) {
      CellMRec<double> m;
      stage_rec(sec(S::CM), kCapCM, i, &m);
      if (i < n[S_CK]) {
        CellKRec<double> r;
        stage_rec(sec(S::CK), kCapCK, i, &r);
        stage_tl_ke(r, m.v[6], w, i);
      }
      if (visc) {
        CellXRec<double> r;
        stage_rec(sec(S::CX), kCapCM, i, &r);
        stage_div(r, m.v[6], w, i);
      }
    }
  }
  __syncthreads();
  // phase 2: tangential velocity of the pv_edge layer; pv_cell on the last threads
  double v = 0.0;
  if (tid < n[S_EM]) {
    v = stage_perp(er, w);
  } else if (top < n[S_CM]) {
    CellMRec<double> r;
    stage_rec(sec(S::CM), kCapCM, top, &r);
    stage_pvcell(r, w, top);
  }
  __syncthreads();
  // phase 3: pv_edge; thickness of the owned cells on the last threads
  if (tid < n[S_EM]) {
    stage_tl_edge(er, w, a.ph, tid, v, vb, gpt, gpn, del4);
  } else if (cell) {
    CellMRec<double> m;
    CellXRec<double> r;
    stage_rec(sec(S::CM), kCapCM, top, &m);
    stage_rec(sec(S::CX), kCapCM, top, &r);
    const double t = stage_tl_thick(r, sec(S::CO)[top], m.v[6], w, top);
    if (a.tend_h) a.tend_h[(size_t)own * B + mb] = t;
    rk.put(a.rkh, (size_t)own * B + mb, t);
  }
  __syncthreads();
  if (del4) {
    if (tid < n[S_VA]) {
      VertexRec<double> r;
      stage_rec(sec(S::V), kCapVA, tid, &r);
      stage_del4_vertex(r, w, tid, n[S_EM]);
    } else if (tid - nv32 >= 0 && tid - nv32 < n[S_CK]) {
      const int i = tid - nv32;
      CellXRec<double> r;
      CellMRec<double> m;
      stage_rec(sec(S::CX), kCapCM, i, &r);
      stage_rec(sec(S::CM), kCapCM, i, &m);
      stage_del4_cell(r, m.v[6], w, i, n[S_EM]);
    }
    __syncthreads();
  }
  // phase 4
  if (edge) {
    const double t = stage_tl_tend(er, w, a, idc, tid, own);
    flag_nonfinite(a.ph.bad, t);
    if (a.tend_u) a.tend_u[(size_t)own * B + mb] = t;
    rk.put(a.rku, (size_t)own * B + mb, t);
  }
}

// Destination bookkeeping of one value of an adjoint member sweep (ad_emit with one member)
struct StageAdOut {
  double x = 0.0, p[3] = {0.0, 0.0, 0.0};
  __device__ __forceinline__ void fetch(const AdOut<double, double> &out, bool edge, size_t o) {
    const double *x2 = edge ? out.x2u : out.x2h, *acc = edge ? out.acc_u : out.acc_h;
    const double *const *pin = edge ? out.pad_in_u : out.pad_in_h;
    if (x2) x = __ldcg(x2 + o);
    if (out.mode == AD_FINAL && pin[0]) {
#pragma unroll
      for (int j = 0; j < 3; j++) p[j] = __ldcg(pin[j] + o);
    } else if (out.mode == AD_FINAL || (out.mode == AD_ADD && !(edge ? out.pad_out_u : out.pad_out_h))) {
      p[0] = __ldcg(acc + o);
    }
  }
  __device__ __forceinline__ void put(const AdOut<double, double> &out, bool edge, size_t o, double pad, double area) const {
    double *tn = edge ? out.tu_next : out.th_next;
    const double wn = edge ? out.wu : out.wh, cn = edge ? out.cu : out.ch;
    double next;
    if (out.mode == AD_FINAL) {
      double a = p[0];
      if (out.pad_in_u[0]) a = (a + p[1]) + p[2];
      const double d = (a + x) + pad;
      (edge ? out.dst_u : out.dst_h)[o] = d;
      next = wn * d;
    } else {
      double *pout = edge ? out.pad_out_u : out.pad_out_h;
      if (pout) pout[o] = pad;
      else (edge ? out.acc_u : out.acc_h)[o] = out.mode == AD_SET ? pad : p[0] + pad;
      next = ((edge ? out.x2u : out.x2h) ? wn * x : 0.0) + cn * pad;
    }
    if (tn) tn[o] = edge ? next : next / area;
  }
};

// An adjoint stage of FP64 members, one a block (blockIdx.y), on the adjoint's tiles; bound by the chain of
// its phases, like k_stage_tl, and fetching as that does.  The divisions by dc and dv that the cells and
// vertices each need are formed once an edge.  384 threads leave 80 registers for the edge records (two
// weights a slot) with two blocks an SM (97 KB each).  9.5 us a level-5 stage of one member, 24.4 as four
// passes.
template <typename R>  // double
__global__ void __launch_bounds__(kAdThreads, 2) k_stage_ad(StageDev ts, StageAdArgs a, int early) {
  static_assert(sizeof(R) == 8);
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ __align__(8) unsigned long long arrived;
  constexpr int NT = kAdThreads;
  constexpr int RV = 0, RC = RV + 16 * kAdVA * kAdRowsV, RO = RC + 16 * kAdCM * kAdRowsC;
  const int tid = threadIdx.x, B = a.B, mb = blockIdx.y;
  unsigned char *const w = smem_raw, *const rec = w + 8 * Y_END;
  int n[kTileCounts], off[kStageAdSections];
#pragma unroll
  for (int k = 0; k < kTileCounts; k++) n[k] = __ldg(ts.cnt + (size_t)blockIdx.x * kTileCounts + k);
  stage_ad_layout(n, off);
  const unsigned char *g = ts.blob + __ldg(ts.blob_off + blockIdx.x);
  if (tid < 32) {  // one bulk copy per chunk row of the records
    if (tid == 0) {
      asm volatile("mbarrier.init.shared.b64 [%0], 1;" ::"r"(smem_addr(&arrived)) : "memory");
      asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
      const int bytes = 16 * (kAdRowsV * n[V_ALL] + kAdRowsC * n[C_MID] + kAdRowsO * n[C_OWN]);
      asm volatile("mbarrier.arrive.expect_tx.shared.b64 _, [%0], %1;" ::"r"(smem_addr(&arrived)), "r"(bytes)
                   : "memory");
    }
    __syncwarp();
    if (tid < kAdRowsV + kAdRowsC + kAdRowsO) {
      const int k = tid < kAdRowsV ? 0 : tid < kAdRowsV + kAdRowsC ? 1 : 2;
      const int row = tid - (k == 0 ? 0 : k == 1 ? kAdRowsV : kAdRowsV + kAdRowsC);
      const int cnt = k == 0 ? n[V_ALL] : k == 1 ? n[C_MID] : n[C_OWN], cap = k == 0 ? kAdVA : k == 1 ? kAdCM : kAdCO;
      asm volatile(
          "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
              smem_addr(rec + (k == 0 ? RV : k == 1 ? RC : RO) + 16 * cap * row)),
          "l"(g + off[k == 0 ? YB_V : k == 1 ? YB_C : YB_O] + 16 * cnt * row), "r"(16 * cnt), "r"(smem_addr(&arrived))
          : "memory");
    }
  }
  auto sec = [&](int o) { return reinterpret_cast<const StageChunk *>(rec + o); };
  AdEdgeRec er;
  if (tid < n[E_MID]) stage_rec(reinterpret_cast<const StageChunk *>(g + off[YB_E]), n[E_MID], tid, &er);
  const int *ids = reinterpret_cast<const int *>(g + off[YB_GE]), *idc = reinterpret_cast<const int *>(g + off[YB_GC]);
  int ge[2] = {0, 0}, gc = 0, gv = 0;
  if (tid < n[E_ALL]) ge[0] = __ldg(ids + tid);
  if (tid + NT < n[E_ALL]) ge[1] = __ldg(ids + tid + NT);
  if (tid < n[C_ALL]) gc = __ldg(idc + tid);
  if (tid < n[V_ALL]) gv = __ldg(reinterpret_cast<const int *>(g + off[YB_GV]) + tid);
  const int top = NT - 1 - tid;
  const bool edge = tid < n[E_OWN], cell = top < n[C_OWN];
  const int own = edge ? ge[0] : cell ? __ldg(idc + top) : 0;
  double vb = 0.0, gpt = 0.0, gpn = 0.0, src = 0.0, hv = 1.0, vort = 0.0;
  auto base = [&]() {
    double b[2][3] = {};
#pragma unroll
    for (int k = 0; k < 2; k++)
      if (tid + k * NT < n[E_ALL]) {
        b[k][0] = __ldcg(a.bs.u + ge[k]);
        b[k][1] = __ldcg(a.bs.he + ge[k]);
        b[k][2] = __ldcg(a.bs.pe + ge[k]);
      }
    if (tid < n[E_MID]) {
      vb = __ldcg(a.bs.v + ge[0]);
      gpt = __ldcg(a.bs.gpt + ge[0]);
      gpn = __ldcg(a.bs.gpn + ge[0]);
    }
    if (tid < n[V_ALL]) {
      hv = __ldcg(a.bs.hv + gv);
      vort = __ldcg(a.bs.vort + gv);
    }
#pragma unroll
    for (int k = 0; k < 2; k++)
      if (tid + k * NT < n[E_ALL]) {
        stage_val<double>(w, Y_UB + tid + k * NT, 0) = b[k][0];
        stage_val<double>(w, Y_HB + tid + k * NT, 0) = b[k][1];
        stage_val<double>(w, Y_PB + tid + k * NT, 0) = b[k][2];
      }
  };
  if (a.ph.wind && tid < n[E_MID]) src = __ldg(a.usrc + ge[0]);
  if (early) base();
  pdl_begin();
  if (!early) base();
  StageAdOut out;
  {
    double u0 = 0.0, u1 = 0.0, h = 0.0;  // in flight together
    if (tid < n[E_ALL]) u0 = __ldcg(a.in.tu + (size_t)ge[0] * B + mb);
    if (tid + NT < n[E_ALL]) u1 = __ldcg(a.in.tu + (size_t)ge[1] * B + mb);
    if (tid < n[C_ALL]) h = __ldcg(a.in.th + (size_t)gc * B + mb);
    if (edge || cell) out.fetch(a.out, edge, (size_t)own * B + mb);
    if (tid < n[E_ALL]) stage_val<double>(w, Y_TU + tid, 0) = u0;
    if (tid + NT < n[E_ALL]) stage_val<double>(w, Y_TU + tid + NT, 0) = u1;
    if (tid < n[C_ALL]) stage_val<double>(w, Y_TH + tid, 0) = h;
  }
  __syncthreads();
  if (!stage_arrived(&arrived)) {
    if (a.ph.bad) *a.ph.bad = 1;
    return;
  }
  double ud = 0.0;
  if (tid < n[E_MID]) ud = stage_ad_edge(er, w, a, tid, vb, gpt, gpn, src);
  __syncthreads();
  if (tid < n[C_MID]) {
    AdCellRec r;
    stage_rec(sec(RC), kAdCM, tid, &r);
    stage_ad_cell(r, w, tid);
  }
  __syncthreads();
  if (tid < n[V_ALL]) {
    AdVertexRec r;
    stage_rec(sec(RV), kAdVA, tid, &r);
    stage_ad_vertex(r, w, tid, hv, vort);
  }
  __syncthreads();
  if (edge) {
    const double pu = stage_ad_final(er, w, ud, stage_val<double>(w, Y_UB + tid, 0));
    flag_nonfinite(a.ph.bad, pu);
    out.put(a.out, true, (size_t)own * B + mb, pu, 1.0);
  } else if (cell) {
    AdCellRec r;
    stage_rec(sec(RO), kAdCO, top, &r);
    out.put(a.out, false, (size_t)own * B + mb, stage_ad_thick(r, w, top), r.v[6]);
  }
}
inline constexpr size_t kStageAdSmem = 8 * Y_END + 16 * (kAdVA * kAdRowsV + kAdCM * kAdRowsC + kAdCO * kAdRowsO);

}  // namespace mpsw

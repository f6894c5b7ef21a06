// FP32 member passes over gathered rows: a tangent-linear or an adjoint RK stage of B members as
// three kernels (cells, edges, tendencies / edges, cells, final) whose every term is one
// coefficient times one row (mpsw_rows.h).
//
// A stage is bound by the member rows it moves: through the intermediate fields (mpsw_members.cuh) a
// level-7 stage of 64 members moves 2.2 GB of rows, 53 rows a cell tangent linear and 57 adjoint;
// folding pv_vertex, the PV flux and the vertex adjoints into coefficients leaves 37 and 44, and
// three kernels instead of four.  Coefficients are formed once a block in shared memory, before the
// wait for the previous kernel where the linearisation point is a stored one, and shared by the
// B / V threads of an entity; a thread holds V members.  The edge passes give a block two
// neighbouring tiles of edges (the second finds rows of the first in L1: the tendency pass, measured
// without its two h' rows, 236 -> 214 us), and each kernel is held to the registers at which occupancy and
// the rows a thread keeps in flight balance.  Level 7, 64 members, cold, us: cells 107, edges 211, tendencies
// 223 (a tangent-linear stage 524, through the fields 634); edges 189, cells 109, final 248 (adjoint 524, through
// the fields 671).
#pragma once

#include "mpsw_members.cuh"
#include "mpsw_rows.h"

namespace mpsw {

// Words of a block's staged coefficients per entity.
constexpr int kRowTlCellW = 6 * 12, kRowTlEdgeW = 10 * 2 + 18, kRowTlTendW = 10 * 3, kRowAdEdgeW = 10 * 5,
              kRowAdCellW = 6 * 8, kRowAdFinalW = 10 * 2 + 14;

__device__ __forceinline__ float4 *row_smem() {
  extern __shared__ __align__(16) float4 row_smem_raw[];
  return row_smem_raw;
}
__device__ __forceinline__ float as_f(int x) { return __int_as_float(x); }
__device__ __forceinline__ int as_i(float x) { return __float_as_int(x); }

// r += c * row
template <int V>
__device__ __forceinline__ void row_add(Mv<float, V> &r, float c, const Mv<float, V> &x) {
#pragma unroll
  for (int i = 0; i < V; i++) r.x[i] = fmaf(c, x.x[i], r.x[i]);
}

// The block's entities and the thread's own: entities a tile, the thread's within it, its members;
// the block's run of consecutive tiles out of `n` entities.
struct RowThread {
  int tpe, epb, le, b;
  __device__ RowThread(int B, int V) {
    tpe = B / V;
    epb = blockDim.x / tpe;
    le = threadIdx.x / tpe;
    b = (threadIdx.x - le * tpe) * V;
  }
  __device__ void run(int n, int block, int blocks, int *first, int *last) const {
    const int tiles = (n + epb - 1) / epb, q = tiles / blocks, r = tiles - q * blocks;
    *first = block * q + min(block, r);
    *last = *first + q + (block < r);
  }
};

// ---- tangent linear ------------------------------------------------------------------------------

// pv_cell', ke', tend_h' and its RK update
template <int V>
__global__ void __maxnreg__(72) k_row_tl_cell(MeshDev<float> m, RowTab t, int B, Base<float> bs,
                                                     const float *__restrict__ ut, const float *__restrict__ ht,
                                                     float *pc, float *ke, RK<float, double> rk, int early) {
  using M = Mv<float, V>;
  float4 *s = row_smem();
  if (!early) pdl_begin();
  const RowThread th(B, V);
  const int nC = m.nC, b = th.b, c0 = blockIdx.x * th.epb;
  for (int i = threadIdx.x; i < 6 * th.epb; i += blockDim.x) {
    const int k = i / th.epb, lc = i - k * th.epb, c = c0 + lc;
    RowTlCell<float> r{};
    if (c < nC && k < m.c_n[c]) r = row_tl_cell<float>(t, m, bs, c, k);
    float4 *d = s + (size_t)(lc * 6 + k) * 3;
    d[0] = make_float4(as_f(r.e), as_f(r.nb), as_f(r.sp), r.pe);
    d[1] = make_float4(r.th, r.ke, r.ps, r.pn);
    d[2] = make_float4(r.tn, r.pc, r.he, 0.f);
  }
  __syncthreads();
  if (early) pdl_begin();
  const int c = c0 + th.le;
  if (c >= nC) return;
  const size_t o = (size_t)c * B + b;
  const M hc = ldv<V>(ht + o);
  M p = mv_fill<float, V>(0.f), q = p, k2 = p;
  float cp = 0.f, ct = 0.f;
#pragma unroll
  for (int k = 0; k < 6; k++) {
    const float4 *d = s + (size_t)(th.le * 6 + k) * 3;
    const float4 x = d[0], y = d[1], z = d[2];
    const M u = ldv<V>(ut + (size_t)as_i(x.x) * B + b);
    const M hn = ldv<V>(ht + (size_t)as_i(x.y) * B + b);
    const M us = ldv<V>(ut + (size_t)as_i(x.z) * B + b);
    row_add(p, x.w, u);
    row_add(q, z.z, y.x * u);
    row_add(k2, y.y, u);
    row_add(p, y.z, us);
    row_add(p, y.w, hn);
    row_add(q, z.x, hn);
    cp += z.y;
    ct += z.x;
  }
  row_add(p, cp, hc);
  row_add(q, ct, hc);
  stv<V>(pc + o, p);
  stv<V>(ke + o, k2);
  rk_members<float, double, V>(rk, o, q);
}

// pv_edge', the thickness flux (u h_edge)' and, with viscosity, delsq_u'
template <int V, int VISC>
__global__ void __maxnreg__(VISC ? 72 : 48) k_row_tl_edge(MeshDev<float> m, RowTab t, int B, Base<float> bs,
                                                     const float *__restrict__ ut, const float *__restrict__ ht,
                                                     const float *__restrict__ pc, float *pe, float *flux, float *dsq,
                                                     float apt, int early) {
  using M = Mv<float, V>;
  float4 *s = row_smem();
  if (!early) pdl_begin();
  const RowThread th(B, V);
  const int nE = m.nE, b = th.b;
  float4 *own = s;                                           // [epb][3]
  float2 *slot = reinterpret_cast<float2 *>(s + 3 * th.epb);  // [epb][10]
  float *tag = reinterpret_cast<float *>(slot + 10 * th.epb);  // [4][epb]
  int *eq = reinterpret_cast<int *>(tag + 4 * th.epb);         // [epb]: the tags' slots
  int tile, last;
  th.run(nE, blockIdx.x, gridDim.x, &tile, &last);
  for (; tile < last; tile++) {
    const int e0 = tile * th.epb;
    // ten slots, the edge's own terms, the four slots that end at one of its vertices
    for (int i = threadIdx.x; i < 15 * th.epb; i += blockDim.x) {
      const int j = i / th.epb, le = i - j * th.epb, e = e0 + le;
      if (j < 10) {
        int nb = 0;
        float p = 0.f;
        if (e < nE && j < m.e_n[e]) {
          nb = m.e_eoe[(size_t)j * nE + e];
          p = row_tl_edge_slot(m.e_w[(size_t)j * nE + e], apt * bs.gpt[e]);
        }
        slot[le * 10 + j] = make_float2(as_f(nb), p);
      } else if (e < nE) {
        const RowTlEdge<float> r = row_tl_edge<float>(t, m, bs, apt, e);
        if (j == 10) {
          own[3 * le] = make_float4(as_f(m.e_c1[e]), as_f(m.e_c2[e]), as_f(t.e_o1[e]), as_f(t.e_o2[e]));
          own[3 * le + 1] = make_float4(r.p0, r.h1, r.h2, r.o1);
          own[3 * le + 2] = make_float4(r.o2, r.pc, r.he, r.uh);
          eq[le] = t.e_q[e];
        } else {
          tag[(j - 11) * th.epb + le] = row_tl_edge_tag(t, nE, e, j - 11, r);
        }
      }
    }
    __syncthreads();
    for (int i = threadIdx.x; i < 4 * th.epb; i += blockDim.x) {
      const int j = i / th.epb, le = i - j * th.epb, e = e0 + le;
      if (e < nE) slot[le * 10 + (((unsigned)eq[le] >> (8 * j)) & 0xFF)].y += tag[i];
    }
    __syncthreads();
    if (early) {
      pdl_begin();
      early = 0;
    }
    const int e = e0 + th.le;
    if (e < nE) {
      const size_t o = (size_t)e * B + b;
      const M u = ldv<V>(ut + o);
      const float4 x = own[3 * th.le], y = own[3 * th.le + 1], z = own[3 * th.le + 2];
      const M h1 = ldv<V>(ht + (size_t)as_i(x.x) * B + b), h2 = ldv<V>(ht + (size_t)as_i(x.y) * B + b);
      M p = y.x * u, f = z.z * u;
      row_add(p, y.y, h1);
      row_add(p, y.z, h2);
      row_add(f, z.w, h1);
      row_add(f, z.w, h2);
      row_add(p, y.w, ldv<V>(ht + (size_t)as_i(x.z) * B + b));
      row_add(p, z.x, ldv<V>(ht + (size_t)as_i(x.w) * B + b));
      row_add(p, z.y, ldv<V>(pc + (size_t)as_i(x.y) * B + b) - ldv<V>(pc + (size_t)as_i(x.x) * B + b));
      M d = mv_fill<float, V>(0.f);
      if (VISC) d = t.e_lap0[e] * u;
#pragma unroll
      for (int j = 0; j < 10; j++) {
        const float2 c = slot[th.le * 10 + j];
        const M un = ldv<V>(ut + (size_t)as_i(c.x) * B + b);
        row_add(p, c.y, un);
        if (VISC) row_add(d, t.e_lap[(size_t)j * nE + e], un);
      }
      stv<V>(pe + o, p);
      stv<V>(flux + o, f);
      if (VISC) stv<V>(dsq + o, d);
    }
    __syncthreads();
  }
}

// tend_u' and its RK update; GEN: any of viscosity, wind and drag.  The sums run so that they round no more
// than the general pass does: a slot's two terms meet before they join the other slots', and the gradient,
// most of the tendency, is formed from differences of rows and comes last.  Adding gravity to the ke row
// and the gradient's halves to the sum first, without the two h' rows, took 215 instead of 223 us (level 7,
// 64 members) but left twice the error of a white-noise tendency and 4-12 times that of a smooth one.
// 40 registers spill and still lead: us at 40 / 48 / 56 / 64, level 6 70 / 76 / 80 / 76, level 7 223 / 226 / 218 / 233,
// a level-6 sweep of 12 steps 7.4 / 7.6 / 7.8 / 7.7 ms.
template <int V, int GEN>
__global__ void __maxnreg__(GEN ? 72 : 40) k_row_tl_tend(MeshDev<float> m, int B, Base<float> bs,
                                                     const float *__restrict__ ut, const float *__restrict__ ht,
                                                     Diag<float> d, const float *__restrict__ flux, Phys<float> ph,
                                                     RK<float, double> rk, int early) {
  using M = Mv<float, V>;
  float *s = reinterpret_cast<float *>(row_smem());
  if (!early) pdl_begin();
  const RowThread th(B, V);
  const int nE = m.nE, b = th.b;
  const int n = 10 * th.epb;
  int *nbs = reinterpret_cast<int *>(s);
  float2 *co = reinterpret_cast<float2 *>(s + n);
  int tile, last;
  th.run(nE, blockIdx.x, gridDim.x, &tile, &last);
  for (; tile < last; tile++) {
    const int e0 = tile * th.epb;
    for (int i = threadIdx.x; i < n; i += blockDim.x) {
      const int j = i / th.epb, le = i - j * th.epb, e = e0 + le;
      int nb = 0;
      RowTlTend<float> r{0.f, 0.f};
      if (e < nE && j < m.e_n[e]) {
        nb = m.e_eoe[(size_t)j * nE + e];
        r = row_tl_tend<float>(bs, nb, m.e_w[(size_t)j * nE + e], bs.pe[e]);
      }
      nbs[i] = nb;
      co[i] = make_float2(r.f, r.p);
    }
    __syncthreads();
    if (early) {
      pdl_begin();
      early = 0;
    }
    const int e = e0 + th.le;
    if (e < nE) {
      const size_t o = (size_t)e * B + b;
      const int c1 = m.e_c1[e], c2 = m.e_c2[e];
      const float rdc = 1.f / m.e_dc[e];
      M q = mv_fill<float, V>(0.f);
      float own = 0.f;
#pragma unroll
      for (int j = 0; j < 10; j++) {
        const int i = j * th.epb + th.le;
        const size_t on = (size_t)nbs[i] * B + b;
        const float2 c = co[i];
        M x = c.x * ldv<V>(flux + on);
        row_add(x, c.y, ldv<V>(d.pe + on));
        q = q + x;
        own += c.y;
      }
      row_add(q, own, ldv<V>(d.pe + o));
      const M h1 = ldv<V>(ht + (size_t)c1 * B + b), h2 = ldv<V>(ht + (size_t)c2 * B + b);
      M grad = ldv<V>(d.ke + (size_t)c2 * B + b) - ldv<V>(d.ke + (size_t)c1 * B + b);
      row_add(grad, float(GRAVITY), h2 - h1);
      row_add(q, -rdc, grad);
      if (GEN) {
        if (ph.visc2 > 0.f) row_add(q, m.e_sc2[e] * ph.visc2, ldv<V>(d.dsq_u + o));
        if (ph.visc4 > 0.f) {
          const int v1 = m.e_v1[e], v2 = m.e_v2[e];
          const float k = m.e_sc4[e] * ph.visc4, kv = k / m.e_dv[e], kc = k * rdc;
          row_add(q, -kc, ldv<V>(d.dsq_div + (size_t)c2 * B + b) - ldv<V>(d.dsq_div + (size_t)c1 * B + b));
          row_add(q, kv, ldv<V>(d.dsq_vort + (size_t)v2 * B + b) - ldv<V>(d.dsq_vort + (size_t)v1 * B + b));
        }
        if (ph.wind || ph.drag) {
          const float hh = bs.he[e];
          float k = ph.wind ? -(m.e_usrc[e] / float(RHO_REF)) / (hh * hh) : 0.f;
          if (ph.drag) {
            const float uu = bs.u[e], sq = sqrtf(bs.ke[c1] + bs.ke[c2]);
            k += ((1.0e-3f * uu) * sq) / (hh * hh);
            row_add(q, -(1.0e-3f * sq) / hh, ldv<V>(ut + o));
            const float kk = -(((0.5f * 1.0e-3f) * uu) / sq) / hh;
            row_add(q, kk, ldv<V>(d.ke + (size_t)c1 * B + b));
            row_add(q, kk, ldv<V>(d.ke + (size_t)c2 * B + b));
          }
          row_add(q, 0.5f * k, h1);
          row_add(q, 0.5f * k, h2);
        }
      }
      if (ph.bad) {
#pragma unroll
        for (int i = 0; i < V; i++) flag_nonfinite(ph.bad, q.x[i]);
      }
      rk_members<float, double, V>(rk, o, q);
    }
    __syncthreads();
  }
}

// ---- adjoint ---------------------------------------------------------------------------------------

// (The adjoint passes add the small terms of a value first and its largest last, so that a sum of many
// rows rounds no more than the general passes' shorter ones: error of one level-5 stage against 64 bits,
// general passes = 1: u_ad 0.7, h_ad 0.9; largest first 1.1 and 1.2.)

// pv_edge_ad, h_edge_ad and the edge's own part of u_ad (with the ke adjoint of both cells): three
// sums over the slots, of the weight back, the weight times pv_edge there, and the ke weight
template <int V>
__global__ void __maxnreg__(72) k_row_ad_edge(MeshDev<float> m, RowTab t, int B, Base<float> bs, float apt,
                                                     AdIn<float> in, AdWork<float> w, int early) {
  using M = Mv<float, V>;
  float *s = reinterpret_cast<float *>(row_smem());
  if (!early) pdl_begin();
  const RowThread th(B, V);
  const int nE = m.nE, b = th.b;
  const int n = 10 * th.epb;
  float4 *co = reinterpret_cast<float4 *>(s);  // [n]: neighbour and the three weights
  float *sq = s + 4 * n;                       // [n]
  int tile, last;
  th.run(nE, blockIdx.x, gridDim.x, &tile, &last);
  for (; tile < last; tile++) {
    const int e0 = tile * th.epb;
    for (int i = threadIdx.x; i < n; i += blockDim.x) {
      const int j = i / th.epb, le = i - j * th.epb, e = e0 + le;
      int nb = 0;
      RowAdEdge<float> r{0.f, 0.f, 0.f, 0.f};
      if (e < nE && j < m.e_n[e]) {
        nb = m.e_eoe[(size_t)j * nE + e];
        r = row_ad_edge<float>(t, bs, nE, e, j, nb, m.e_w[(size_t)j * nE + e], m.e_wrev[(size_t)j * nE + e]);
      }
      co[i] = make_float4(as_f(nb), r.w, r.wp, r.ke);
      sq[i] = r.sq;
    }
    __syncthreads();
    if (early) {
      pdl_begin();
      early = 0;
    }
    const int e = e0 + th.le;
    if (e < nE) {
      const size_t o = (size_t)e * B + b;
      const M T = ldv<V>(in.tu + o);
      const int c1 = m.e_c1[e], c2 = m.e_c2[e];
      const M fa = ldv<V>(in.th + (size_t)c2 * B + b) - ldv<V>(in.th + (size_t)c1 * B + b);
      M p = mv_fill<float, V>(0.f), h = p, k = p;
      float own = 0.f;
#pragma unroll
      for (int j = 0; j < 10; j++) {
        const int i = j * th.epb + th.le;
        const float4 c = co[i];
        const M Tn = ldv<V>(in.tu + (size_t)as_i(c.x) * B + b);
        row_add(p, c.y, Tn);
        row_add(h, c.z, Tn);
        row_add(k, c.w, Tn);
        own += sq[i];
      }
      const float ue = bs.u[e], he = bs.he[e], dv = m.e_dv[e], kc = ((0.5f * m.e_dc[e]) * dv) * ue;
      row_add(h, 0.5f * bs.pe[e], p);  // sum w (pv_edge there + here) / 2
      row_add(k, (t.c_ra[c1] - t.c_ra[c2]) / m.e_dc[e], T);  // cell 1 has sign +1, cell 2 -1
      M u = kc * k;
      p = (0.5f * (ue * he)) * p;
      row_add(p, own, T);
      row_add(u, -(apt * bs.gpn[e]), p);
      row_add(u, he, h);
      row_add(u, dv * he, fa);
      h = ue * h;
      row_add(h, ue * dv, fa);
      stv<V>(w.pe_ad + o, p);
      stv<V>(w.he_ad + o, h);
      stv<V>(w.ud + o, u);
    }
    __syncthreads();
  }
}

// pv_cell_ad and h_ad but for the pv_cell_ad terms of the vertex adjoints
template <int V>
__global__ void __maxnreg__(64) k_row_ad_cell(MeshDev<float> m, RowTab t, int B, Base<float> bs, float apt,
                                                     AdIn<float> in, AdWork<float> w, int early) {
  using M = Mv<float, V>;
  float4 *s = row_smem();
  if (!early) pdl_begin();
  const RowThread th(B, V);
  const int nC = m.nC, b = th.b, c0 = blockIdx.x * th.epb;
  for (int i = threadIdx.x; i < 6 * th.epb; i += blockDim.x) {
    const int k = i / th.epb, lc = i - k * th.epb, c = c0 + lc;
    RowAdCell<float> r{};
    if (c < nC && k < m.c_n[c]) r = row_ad_cell<float>(t, m, bs, apt, c, k);
    float4 *d = s + (size_t)(lc * 6 + k) * 2;
    d[0] = make_float4(as_f(r.e), as_f(r.sp), r.pc, r.g);
    d[1] = make_float4(r.hv, r.hs, r.half, 0.f);
  }
  __syncthreads();
  if (early) pdl_begin();
  const int c = c0 + th.le;
  if (c >= nC) return;
  M p = mv_fill<float, V>(0.f), h = p;
#pragma unroll
  for (int k = 0; k < 6; k++) {
    const float4 *d = s + (size_t)(th.le * 6 + k) * 2;
    const float4 x = d[0], y = d[1];
    const size_t oe = (size_t)as_i(x.x) * B + b;
    const M pe = ldv<V>(w.pe_ad + oe);
    row_add(p, x.z, pe);
    M q = y.x * pe;
    row_add(q, y.y, ldv<V>(w.pe_ad + (size_t)as_i(x.y) * B + b));
    row_add(q, y.z, ldv<V>(w.he_ad + oe));
    row_add(q, x.w, ldv<V>(in.tu + oe));
    h = h + q;
  }
  const size_t o = (size_t)c * B + b;
  stv<V>(w.pc_ad + o, p);
  stv<V>(w.hd + o, h);
}

// u_ad and h_ad of the stage with their RK bookkeeping: the first cell_blocks blocks take the cells
template <int V>
__global__ void __maxnreg__(40) k_row_ad_final(MeshDev<float> m, RowTab t, int B, Base<float> bs, float apt,
                                                      AdWork<float> w, AdOut<float, double> out, int *bad,
                                                      int cell_blocks, int early) {
  using M = Mv<float, V>;
  float4 *s = row_smem();
  if (!early) pdl_begin();
  const RowThread th(B, V);
  const int b = th.b;
  if ((int)blockIdx.x < cell_blocks) {
    const int nC = m.nC;
    int tile, last;
    th.run(nC, blockIdx.x, cell_blocks, &tile, &last);
    for (; tile < last; tile++) {
      const int c0 = tile * th.epb;
      for (int i = threadIdx.x; i < 6 * th.epb; i += blockDim.x) {
        const int k = i / th.epb, lc = i - k * th.epb, c = c0 + lc;
        RowAdLast<float> r{};
        if (c < nC && k < m.c_n[c]) r = row_ad_last<float>(t, m, bs, c, k);
        s[lc * 6 + k] = make_float4(as_f(r.nb), r.n, r.c, 0.f);
      }
      __syncthreads();
      if (early) {
        pdl_begin();
        early = 0;
      }
      const int c = c0 + th.le;
      if (c < nC) {
        const size_t o = (size_t)c * B + b;
        M h = mv_fill<float, V>(0.f);
        float own = 0.f;
#pragma unroll
        for (int k = 0; k < 6; k++) {
          const float4 x = s[th.le * 6 + k];
          row_add(h, x.y, ldv<V>(w.pc_ad + (size_t)as_i(x.x) * B + b));
          own += x.z;
        }
        row_add(h, own, ldv<V>(w.pc_ad + o));
        h = h + ldv<V>(w.hd + o);
        ad_emit<float, double, V>(out, 0, o, h, m.c_area[c]);
      }
      __syncthreads();
    }
    return;
  }
  const int nE = m.nE;
  float4 *own = s;                                           // [epb][2]
  float *o2 = reinterpret_cast<float *>(s + 2 * th.epb);      // [epb]: the edge's own coefficient
  float *tag = o2 + th.epb;                                   // [4][epb]
  int *eq = reinterpret_cast<int *>(tag + 4 * th.epb);         // [epb]: the tags' slots
  float2 *slot = reinterpret_cast<float2 *>(o2 + 6 * th.epb);  // [epb][10]
  int tile, last;
  th.run(nE, (int)blockIdx.x - cell_blocks, (int)gridDim.x - cell_blocks, &tile, &last);
  for (; tile < last; tile++) {
    const int e0 = tile * th.epb;
    // ten slots, the edge's own terms, the four slots that end at one of its vertices
    for (int i = threadIdx.x; i < 15 * th.epb; i += blockDim.x) {
      const int j = i / th.epb, le = i - j * th.epb, e = e0 + le;
      if (j < 10) {
        int nb = 0;
        float p = 0.f;
        if (e < nE && j < m.e_n[e]) {
          nb = m.e_eoe[(size_t)j * nE + e];
          p = row_ad_final_slot(bs, apt, nb, m.e_wrev[(size_t)j * nE + e]);
        }
        slot[le * 10 + j] = make_float2(as_f(nb), p);
      } else if (e < nE) {
        const RowAdFinal<float> r = row_ad_final<float>(t, m, bs, apt, e);
        if (j == 10) {
          own[2 * le] = make_float4(as_f(m.e_c1[e]), as_f(m.e_c2[e]), as_f(t.e_o1[e]), as_f(t.e_o2[e]));
          own[2 * le + 1] = make_float4(r.k1, r.k2, r.o1, r.o2);
          o2[le] = r.p0;
          eq[le] = t.e_q[e];
        } else {
          tag[(j - 11) * th.epb + le] = row_ad_final_tag(t, bs, nE, apt, e, j - 11, t.e_t[(size_t)(j - 11) * nE + e], r);
        }
      }
    }
    __syncthreads();
    for (int i = threadIdx.x; i < 4 * th.epb; i += blockDim.x) {
      const int j = i / th.epb, le = i - j * th.epb, e = e0 + le;
      if (e < nE) slot[le * 10 + (((unsigned)eq[le] >> (8 * j)) & 0xFF)].y += tag[i];
    }
    __syncthreads();
    if (early) {
      pdl_begin();
      early = 0;
    }
    const int e = e0 + th.le;
    if (e < nE) {
      const size_t o = (size_t)e * B + b;
      const float4 x = own[2 * th.le], y = own[2 * th.le + 1];
      M u = o2[th.le] * ldv<V>(w.pe_ad + o);
      row_add(u, y.x, ldv<V>(w.pc_ad + (size_t)as_i(x.x) * B + b));
      row_add(u, y.y, ldv<V>(w.pc_ad + (size_t)as_i(x.y) * B + b));
      row_add(u, y.z, ldv<V>(w.pc_ad + (size_t)as_i(x.z) * B + b));
      row_add(u, y.w, ldv<V>(w.pc_ad + (size_t)as_i(x.w) * B + b));
#pragma unroll
      for (int j = 0; j < 10; j++) {
        const float2 c = slot[th.le * 10 + j];
        row_add(u, c.y, ldv<V>(w.pe_ad + (size_t)as_i(c.x) * B + b));
      }
      u = u + ldv<V>(w.ud + o);
      if (bad) {
#pragma unroll
        for (int i = 0; i < V; i++) flag_nonfinite(bad, u.x[i]);
      }
      ad_emit<float, double, V>(out, 1, o, u, 1.f);
    }
    __syncthreads();
  }
}

}  // namespace mpsw

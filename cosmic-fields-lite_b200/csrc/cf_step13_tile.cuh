// cf_step13_tile.cuh -- one whole RK4 step in one pass over a (b, c) tile,
// marching along a, for the 4th-order 13-point Laplacian.
//
// The whole-step pass of cf_step_tile.cuh with every distance doubled.  The
// 13-point stencil reaches 2 sites, so a step depends on x within 4 (stage 3 takes
// the Laplacian of yb_phi = x_phi + dt/2 ya_pi, and ya_pi needs lap x_phi):
//
//   phase 1 (plane q, its tile and a 2-site ring), from x_phi and ya_phi of planes
//   q-2..q+2 with a 4-site ring:  k1, ya, k2, yb = x + dt/2 (ya_pi, k2), yc_phi = x_phi + dt yb_pi
//   phase 2 (plane r = q - 2, its tile), from yb_phi, yc_phi of planes r-2..r+2 with
//   a 2-site ring: k3, yc_pi = x_pi + dt k3, k4, x += dt/6 (k1 + 2 k2 + 2 k3 + k4)
//
// HBM moves the state once, like the 7-point pass: 4 words per site-update in FP64 and 8
// in FP32_COMP (+6 with Psi) against 14 and 18 (+8) for the paired passes.  Every value is
// formed and rounded as the paired (cf_pair_tile.cuh) and the single-stage
// (cf_stage_tile.cuh) 13-point passes form it, so all three routes give the same bits.
//
// As in the 7-point pass ya_phi replaces x_pi in place when a plane lands, a thread's
// own a-neighbours come from registers or from its own cells, and the warps have roles with
// loops of their own: own rows, the 2-site ring's rows, and its columns (one thread per
// row and side, two sites).  Shared memory: x_phi and x_pi / ya_phi of four planes with a
// 4-site ring (p + 1 landing, p, q + 1, q), yb_phi and yc_phi of three with a 2-site ring (q,
// r + 1, r), what phase 1 hands to phase 2 two planes later at the own sites, and x_pi of
// the own sites for five planes.  One barrier per plane.
#pragma once

#include "cf_pair_tile.cuh"
#include "cf_step_tile.cuh"

namespace cfb {

template <typename S, int TXv, int TYv>
struct Step13Smem {
  static constexpr int V = VecT<S>::n;
  static constexpr int TW = TXv * V;
  static constexpr int O = 4;                  // first interior column: 4 ring columns before it
  static constexpr int SP = TW + 2 * O;        // row pitch of every plane array
  static constexpr int R4 = TYv + 8, P4 = R4 * SP;  // 4-ring planes (x_phi, x_pi / ya_phi)
  static constexpr int R2 = TYv + 4, P2 = R2 * SP;  // 2-ring planes (yb_phi, yc_phi)
  static constexpr int PD = TYv * TW;               // own sites
  static constexpr int count = 4 * 2 * P4 + 3 * 2 * P2 + 3 * 4 * PD + 5 * PD;
};

// Thread rows beside the TYv rows of own sites: four that form the 2-ring's rows, and as
// many as its columns need threads (one per row and side of the 4-ring), in whole warps.
constexpr int step13_ring_rows(int TXv, int TYv) {
  int r = 4;
  while ((r - 4) * TXv < 2 * (TYv + 8) || ((TYv + r) * TXv) % 32 != 0) ++r;
  return r;
}

// The stencil of the V sites of a row: the row itself, the rows 1 and 2 beside it, the
// planes 1 and 2 before and behind, and the vectors left and right of it.
template <typename S, int V>
struct RowStar13 {
  Pack<S, V> c, n1, n2, s1, s2, a1, a2, b1, b2;
  Pack<S, V> l, r;
  template <int SP>
  __device__ __forceinline__ void load(const S *p0, int o) {  // the neighbours in the plane
    n1 = lds<S, V>(p0 + o + SP);
    n2 = lds<S, V>(p0 + o + 2 * SP);
    s1 = lds<S, V>(p0 + o - SP);
    s2 = lds<S, V>(p0 + o - 2 * SP);
    l = lds<S, V>(p0 + o - V);
    r = lds<S, V>(p0 + o + V);
  }
  __device__ __forceinline__ S at(int i) const {  // site i of the row, -V <= i < 2V
    return i < 0 ? l.v[i + V] : (i < V ? c.v[i] : r.v[i - V]);
  }
  // the Laplacian sum (times 12) in the order of lap_at: first neighbours a+, a-, b+, b-, c+,
  // c-, then the second ones
  __device__ __forceinline__ S lap(int v) const {
    const S u1 = a1.v[v] + b1.v[v] + n1.v[v] + s1.v[v] + at(v + 1) + at(v - 1);
    const S u2 = a2.v[v] + b2.v[v] + n2.v[v] + s2.v[v] + at(v + 2) + at(v - 2);
    return (S)16 * u1 - u2 - (S)90 * c.v[v];
  }
  __device__ __forceinline__ float2 lap2(int k) const {  // FP32: sites 2k, 2k + 1
    const int v = 2 * k;
    float2 u1 = p_add(lane2(a1, k), lane2(b1, k));
    u1 = p_add(u1, lane2(n1, k));
    u1 = p_add(u1, lane2(s1, k));
    u1 = p_add(u1, make_float2(at(v + 1), at(v + 2)));
    u1 = p_add(u1, make_float2(at(v - 1), at(v)));
    float2 u2 = p_add(lane2(a2, k), lane2(b2, k));
    u2 = p_add(u2, lane2(n2, k));
    u2 = p_add(u2, lane2(s2, k));
    u2 = p_add(u2, make_float2(at(v + 2), at(v + 3)));
    u2 = p_add(u2, make_float2(at(v - 2), at(v - 1)));
    return lap13_f32<float2>(lane2(c, k), u1, u2);
  }
};

template <typename S, int EQ, int TXv, int TYv, bool FULL = false>
__device__ __forceinline__ void step13_tile(const StepArgs<S> &A, int c0, int b0, int a_begin, int a_end, S *smem) {
  using SM = Step13Smem<S, TXv, TYv>;
  using T = typename Arith<S>::T;
  constexpr int V = SM::V, TW = SM::TW, O = SM::O, SP = SM::SP, PD = SM::PD, P2 = SM::P2, P4 = SM::P4;
  constexpr int NT = TXv * (TYv + step13_ring_rows(TXv, TYv));
  static_assert((TXv * TYv) % 32 == 0 && (4 * TXv) % 32 == 0 && NT % 32 == 0, "warps of one role each");
  S *XF = smem;           // x_phi, 4 planes of P4
  S *XW = XF + 4 * P4;    // x_pi as it lands, then ya_phi; 4 planes of P4
  S *YB = XW + 4 * P4;    // yb_phi, 3 planes of P2
  S *YC = YB + 3 * P2;    // yc_phi, 3 planes of P2
  S *DL = YC + 3 * P2;    // 3 planes x (yb_pi, acc_phi, acc_pi, x_phi) of PD
  S *PK = DL + 12 * PD;   // x_pi of the own sites, 5 planes of PD
  const int N = A.N;
  const long long N3 = A.N3, NN = (long long)N * N;
  const int tx = threadIdx.x, ty = threadIdx.y;
  const int twe = FULL ? TW : min(TW, N - c0);
  const int tye = FULL ? TYv : min(TYv, N - b0);
  const bool colact = FULL || (tx * V) < twe;
  const int c = c0 + tx * V;
  const StepK<S> K(A);

  // ya_phi = x_phi + dt/2 x_pi over the x_pi of sites a thread copied itself
  auto to_w = [&](S *xf, S *xp, auto &f, auto &q, auto &w) {
    constexpr int VV = sizeof(f.v) / sizeof(S);
    f = lds<S, VV>(xf);
    q = lds<S, VV>(xp);
    if constexpr (sizeof(S) == 4) {
#pragma unroll
      for (int l = 0; l < VV / 2; ++l) set2(w, l, c_fma(A.dt2f, lane2(q, l), lane2(f, l)));
    } else {
#pragma unroll
      for (int v = 0; v < VV; ++v) w.v[v] = w_of(f.v[v], q.v[v], K.ch);
    }
    sts<S, VV>(xp, w);
  };
  // stages 1-2 at the sites of a row of plane q
  auto phase1 = [&](const auto &F, const auto &W, const auto &Pq, const auto &ct, const auto &ch2, auto &vb, auto &vc,
                    auto &vbp, auto &vap, auto &vpp) {
    constexpr int VV = sizeof(Pq.v) / sizeof(S);
    if constexpr (sizeof(S) == 4) {  // two sites per paired FP32 instruction, same bits
      const StageCoefL<float2> K1{A.m2f, A.invf[0], A.hubf[0], A.q1f, A.q2f}, K2{A.m2f, A.invf[1], A.hubf[1], A.q1f, A.q2f};
#pragma unroll
      for (int l = 0; l < VV / 2; ++l) {
        const float2 f0 = lane2(F.c, l), p0 = lane2(Pq, l);
        float2 c_ps, c_dps, c_ps4;
        coupling2<EQ>(ct, l, c_ps, c_dps, c_ps4);
        const float2 k1 = kpi_f32<EQ, float2>(p0, f0, F.lap2(l), c_ps, c_dps, c_ps4, K1);
        const float2 yapi = c_fma(A.dt2f, k1, p0);
        coupling2<EQ>(ch2, l, c_ps, c_dps, c_ps4);
        const float2 k2 = kpi_f32<EQ, float2>(yapi, lane2(W.c, l), W.lap2(l), c_ps, c_dps, c_ps4, K2);
        const float2 bpi = c_fma(A.dt2f, k2, p0);
        set2(vb, l, c_fma(A.dt2f, yapi, f0));
        set2(vc, l, c_fma(A.dtf, bpi, f0));
        set2(vbp, l, bpi);
        set2(vap, l, p_fma(p_splat<float2>(2.0f), yapi, p0));
        set2(vpp, l, p_fma(p_splat<float2>(2.0f), k2, k1));
      }
    } else {
#pragma unroll
      for (int v = 0; v < VV; ++v) {
        const T f0 = F.c.v[v], p0 = Pq.v[v];
        const T k1 = kpi_of<EQ, S, VV>(p0, f0, F.lap(v), ct, v, K.k1);
        const S yapi = (S)K.ch.fma(k1, p0);
        const T k2 = kpi_of<EQ, S, VV>((T)yapi, (T)W.c.v[v], W.lap(v), ch2, v, K.k2);
        const S bpi = (S)K.ch.fma(k2, p0);
        vb.v[v] = (S)K.ch.fma((T)yapi, f0);
        vc.v[v] = (S)K.cf.fma((T)bpi, f0);
        vbp.v[v] = bpi;
        vap.v[v] = (S)((T)(S)p0 + (T)2 * (T)yapi);
        vpp.v[v] = (S)((T)(S)k1 + (T)2 * k2);
      }
    }
  };
  // the curvature of two stages at the sites of a row
  auto couple = [&](auto &ca, auto &cb, int ka, int kb, long long site, int ai, const auto &cc) {
    if constexpr (EqOf<EQ>::coupled) {
      constexpr int VV = sizeof(ca.ps.v) / sizeof(S);
      const int row = EqOf<EQ>::coarse ? __ldg(A.cmap + ai) : 0;
      load_coupling<EQ, S, VV>(ca, A.psi[ka], A.dpsi[ka], site, A.M, row, cc);
      if constexpr (EQ == EQ_FIXED)
        cb = ca;
      else
        load_coupling<EQ, S, VV>(cb, A.psi[kb], A.dpsi[kb], site, A.M, row, cc);
    }
  };

  const int first = wrap_n(a_begin - 4, N);
  int i0 = 0, i1 = 1, i2 = 2, i3 = 3;  // slots of planes q, q + 1, p, p + 1
  int y0 = 0, y1 = 1, y2 = 2;          // slots of planes r, r + 1, q
  int an = first, ap = 0, ap1 = 0, aq = 0, aq1 = 0, ar = 0;
  long long on = NN * first, opp = 0, op1 = 0, oq = 0, oq1 = 0, orr = 0;  // plane offsets p + 1, p, p - 1, q, q - 1, r
  auto advance = [&] {
    orr = oq1, oq1 = oq, oq = op1, op1 = opp, opp = on, on += NN;
    if constexpr (EqOf<EQ>::coarse) ar = aq1, aq1 = aq, aq = ap1, ap1 = ap, ap = an;
    if (++an == N) an = 0, on -= N3;
  };
  auto rotate = [&] {
    const int i = i0, y = y0;
    i0 = i1, i1 = i2, i2 = i3, i3 = i;
    y0 = y1, y1 = y2, y2 = y;
  };
  if (ty < TYv) {  // ---------------- own rows
    const bool act = colact && (FULL || ty < tye);
    const int o4 = (ty + 4) * SP + O + tx * V, o2 = o4 - 2 * SP, od = ty * TW + tx * V;
    const long long rowoff = (long long)N * (b0 + ty) + c;
    CoarseCols<V> cc{};
    if constexpr (EqOf<EQ>::coarse) cc = coarse_cols<EQ, V>(A.cmap, act, b0 + ty, c);
    Pack<S, V> Fm1{}, Fm2{}, Wm1{}, Wm2{};  // x_phi, ya_phi of q - 1, q - 2
    Pack<S, V> Bm1{}, Cm1{};                // yb_phi, yc_phi of r - 1
    int kp = 0;                             // slot of x_pi of plane p
    auto issue = [&](int s) {
      if (act) {
        cp_async_16(XF + s * P4 + o4, A.xphi + on + rowoff);
        cp_async_16(XW + s * P4 + o4, A.xpi + on + rowoff);
      }
      cp_async_commit();
    };
    issue(i2);
    for (int p = a_begin - 4; p <= a_end + 3; ++p) {
      advance();
      cp_async_wait_all();  // this thread's copies of plane p have landed
      Pack<S, V> Fp{}, Pp{}, Wp{};
      if (act) {
        to_w(XF + i2 * P4 + o4, XW + i2 * P4 + o4, Fp, Pp, Wp);
        sts<S, V>(PK + kp * PD + od, Pp);
      }
      step_barrier(NT);  // plane p in full; phase 2 of the last plane is done
      if (p <= a_end + 2) issue(i3);
      // L2 prefetch one plane ahead of what phases 1 (plane q + 1) and 2 (r + 1) load directly
      if (tx == 0 && act) {
        const unsigned bytes = (unsigned)(twe * sizeof(S));
        if (p >= a_begin - 1 && p <= a_end + 2) {
          if constexpr (EqOf<EQ>::psi_plane) {
            prefetch_l2(A.psi[0] + op1 + rowoff, bytes);
            if constexpr (EQ != EQ_FIXED) prefetch_l2(A.psi[1] + op1 + rowoff, bytes);
          }
          if constexpr (EqOf<EQ>::dpsi_plane) {
            prefetch_l2(A.dpsi[0] + op1 + rowoff, bytes);
            prefetch_l2(A.dpsi[1] + op1 + rowoff, bytes);
          }
        }
        if (p >= a_begin + 3 && p <= a_end + 2) {
          if constexpr (EqOf<EQ>::psi_plane && EQ != EQ_FIXED) prefetch_l2(A.psi[2] + oq1 + rowoff, bytes);
          if constexpr (EqOf<EQ>::dpsi_plane) prefetch_l2(A.dpsi[2] + oq1 + rowoff, bytes);
          if constexpr (sizeof(S) == 4) {
            prefetch_l2(A.xlo + oq1 + rowoff, bytes);
            prefetch_l2(A.xlo + N3 + oq1 + rowoff, bytes);
          }
        }
      }
      if (act) {
        Pack<S, V> vb{}, vc{};
        const Pack<S, V> Fq = lds<S, V>(XF + i0 * P4 + o4), Wq = lds<S, V>(XW + i0 * P4 + o4);
        if (p >= a_begin) {  // phase 1 on plane q = p - 2
          Coupling<S, V> ct, ch2;
          couple(ct, ch2, 0, 1, oq + rowoff, aq, cc);
          RowStar13<S, V> F, W;
          F.template load<SP>(XF + i0 * P4, o4);
          F.c = Fq, F.b1 = Fm1, F.b2 = Fm2, F.a1 = lds<S, V>(XF + i1 * P4 + o4), F.a2 = Fp;
          W.template load<SP>(XW + i0 * P4, o4);
          W.c = Wq, W.b1 = Wm1, W.b2 = Wm2, W.a1 = lds<S, V>(XW + i1 * P4 + o4), W.a2 = Wp;
          const Pack<S, V> Pq = lds<S, V>(PK + (kp >= 2 ? kp - 2 : kp + 3) * PD + od);
          Pack<S, V> vbp, vap, vpp;
          phase1(F, W, Pq, ct, ch2, vb, vc, vbp, vap, vpp);
          S *dl = DL + y2 * 4 * PD;
          sts<S, V>(dl + od, vbp);
          sts<S, V>(dl + PD + od, vap);
          sts<S, V>(dl + 2 * PD + od, vpp);
          sts<S, V>(dl + 3 * PD + od, Fq);
        }
        const Pack<S, V> Bm2 = Bm1, Cm2 = Cm1;
        Bm1 = lds<S, V>(YB + y2 * P2 + o2);  // plane r - 1, whose slot plane q takes
        Cm1 = lds<S, V>(YC + y2 * P2 + o2);
        if (p >= a_begin) {
          sts<S, V>(YB + y2 * P2 + o2, vb);
          sts<S, V>(YC + y2 * P2 + o2, vc);
        }
        if (p >= a_begin + 4) {  // phase 2 on plane r = p - 4
          Coupling<S, V> cth, cd;
          couple(cth, cd, 1, 2, orr + rowoff, ar, cc);
          Pack<S, V> lp{}, lq{};
          if constexpr (sizeof(S) == 4) {
            lp = ldv_rw<S, V>(A.xlo + orr + rowoff);
            lq = ldv_rw<S, V>(A.xlo + N3 + orr + rowoff);
          }
          const S *dl = DL + y0 * 4 * PD;
          const Pack<S, V> ybpi = lds<S, V>(dl + od), aphi = lds<S, V>(dl + PD + od), api = lds<S, V>(dl + 2 * PD + od);
          const Pack<S, V> Fr = lds<S, V>(dl + 3 * PD + od), Pr = lds<S, V>(PK + (kp >= 4 ? kp - 4 : kp + 1) * PD + od);
          RowStar13<S, V> B, C;
          B.template load<SP>(YB + y0 * P2, o2);
          B.c = lds<S, V>(YB + y0 * P2 + o2), B.a1 = lds<S, V>(YB + y1 * P2 + o2), B.a2 = vb, B.b1 = Bm1, B.b2 = Bm2;
          C.template load<SP>(YC + y0 * P2, o2);
          C.c = lds<S, V>(YC + y0 * P2 + o2), C.a1 = lds<S, V>(YC + y1 * P2 + o2), C.a2 = vc, C.b1 = Cm1, C.b2 = Cm2;
          Pack<S, V> o1v, o2v, o3v, o4v;
          if constexpr (sizeof(S) == 4) {
            const StageCoefL<float2> K2{A.m2f, A.invf[1], A.hubf[1], A.q1f, A.q2f}, K4{A.m2f, A.invf[2], A.hubf[2], A.q1f, A.q2f};
#pragma unroll
            for (int l = 0; l < V / 2; ++l) {
              const float2 p0 = lane2(ybpi, l);
              float2 c_ps, c_dps, c_ps4;
              coupling2<EQ>(cth, l, c_ps, c_dps, c_ps4);
              const float2 k3 = kpi_f32<EQ, float2>(p0, lane2(B.c, l), B.lap2(l), c_ps, c_dps, c_ps4, K2);
              const float2 c1phi = p_fma(p_splat<float2>(2.0f), p0, lane2(aphi, l));
              const float2 c1pi = p_fma(p_splat<float2>(2.0f), k3, lane2(api, l));
              const float2 ycpi = c_fma(A.dtf, k3, lane2(Pr, l));
              coupling2<EQ>(cd, l, c_ps, c_dps, c_ps4);
              const float2 k4 = kpi_f32<EQ, float2>(ycpi, lane2(C.c, l), C.lap2(l), c_ps, c_dps, c_ps4, K4);
              float2 h1, l1, h2, l2;
              comp_update_f32<float2>(lane2(Fr, l), lane2(lp, l), p_add(c1phi, ycpi), A.dt6f, h1, l1);
              comp_update_f32<float2>(lane2(Pr, l), lane2(lq, l), p_add(c1pi, k4), A.dt6f, h2, l2);
              set2(o1v, l, h1);
              set2(o3v, l, l1);
              set2(o2v, l, h2);
              set2(o4v, l, l2);
            }
          } else {
#pragma unroll
            for (int v = 0; v < V; ++v) {
              const T p0 = (T)ybpi.v[v];
              const T k3 = kpi_of<EQ, S, V>(p0, (T)B.c.v[v], B.lap(v), cth, v, K.k2);
              const S c1phi = (S)((T)aphi.v[v] + (T)2 * p0);
              const S c1pi = (S)((T)api.v[v] + (T)2 * k3);
              const S ycpi = (S)K.cf.fma(k3, (T)Pr.v[v]);
              const T k4 = kpi_of<EQ, S, V>((T)ycpi, (T)C.c.v[v], C.lap(v), cd, v, K.k4);
              state_update(Fr.v[v], lp.v[v], (T)c1phi + (T)ycpi, K.c6, o1v.v[v], o3v.v[v]);
              state_update(Pr.v[v], lq.v[v], (T)c1pi + k4, K.c6, o2v.v[v], o4v.v[v]);
            }
          }
          stv(A.ophi + orr + rowoff, o1v);
          stv(A.opi + orr + rowoff, o2v);
          if constexpr (sizeof(S) == 4) {
            stv(A.olo + orr + rowoff, o3v);
            stv(A.olo + N3 + orr + rowoff, o4v);
          }
        }
        Fm2 = Fm1, Fm1 = Fq, Wm2 = Wm1, Wm1 = Wq;
      }
      if (++kp == 5) kp = 0;
      rotate();
    }
  } else if (ty < TYv + 4) {  // ---------------- the 2-ring's rows
    const int k = ty - TYv;
    const int r4 = k < 2 ? 2 + k : tye + 2 + k, r4o = k < 2 ? k : tye + 4 + k;  // its row, and one of the outer ones
    const int b = wrap_n(b0 - 4 + r4, N);
    const int o4 = r4 * SP + O + tx * V, o2 = o4 - 2 * SP, oo = r4o * SP + O + tx * V;
    const long long rowoff = (long long)N * b + c, outoff = (long long)N * wrap_n(b0 - 4 + r4o, N) + c;
    CoarseCols<V> cc{};
    if constexpr (EqOf<EQ>::coarse) cc = coarse_cols<EQ, V>(A.cmap, colact, b, c);
    Pack<S, V> Fm1{}, Fm2{}, Wm1{}, Wm2{}, P1{}, Pq{};
    auto issue = [&](int s) {
      if (colact) {
        cp_async_16(XF + s * P4 + o4, A.xphi + on + rowoff);
        cp_async_16(XW + s * P4 + o4, A.xpi + on + rowoff);
        cp_async_16(XF + s * P4 + oo, A.xphi + on + outoff);
        cp_async_16(XW + s * P4 + oo, A.xpi + on + outoff);
      }
      cp_async_commit();
    };
    issue(i2);
    for (int p = a_begin - 4; p <= a_end + 3; ++p) {
      advance();
      cp_async_wait_all();
      Pack<S, V> Fp{}, Pp{}, Wp{};
      if (colact) {
        to_w(XF + i2 * P4 + oo, XW + i2 * P4 + oo, Fp, Pp, Wp);
        to_w(XF + i2 * P4 + o4, XW + i2 * P4 + o4, Fp, Pp, Wp);
      }
      step_barrier(NT);
      if (p <= a_end + 2) issue(i3);
      if (tx == 0 && p >= a_begin - 1 && p <= a_end + 2) {
        const unsigned bytes = (unsigned)(twe * sizeof(S));
        if constexpr (EqOf<EQ>::psi_plane) {
          prefetch_l2(A.psi[0] + op1 + rowoff, bytes);
          if constexpr (EQ != EQ_FIXED) prefetch_l2(A.psi[1] + op1 + rowoff, bytes);
        }
        if constexpr (EqOf<EQ>::dpsi_plane) {
          prefetch_l2(A.dpsi[0] + op1 + rowoff, bytes);
          prefetch_l2(A.dpsi[1] + op1 + rowoff, bytes);
        }
      }
      if (colact) {
        RowStar13<S, V> F, W;
        F.c = lds<S, V>(XF + i0 * P4 + o4);
        W.c = lds<S, V>(XW + i0 * P4 + o4);
        if (p >= a_begin) {
          Coupling<S, V> ct, ch2;
          couple(ct, ch2, 0, 1, oq + rowoff, aq, cc);
          F.template load<SP>(XF + i0 * P4, o4);
          F.b1 = Fm1, F.b2 = Fm2, F.a1 = lds<S, V>(XF + i1 * P4 + o4), F.a2 = Fp;
          W.template load<SP>(XW + i0 * P4, o4);
          W.b1 = Wm1, W.b2 = Wm2, W.a1 = lds<S, V>(XW + i1 * P4 + o4), W.a2 = Wp;
          Pack<S, V> vb, vc, vbp, vap, vpp;
          phase1(F, W, Pq, ct, ch2, vb, vc, vbp, vap, vpp);
          sts<S, V>(YB + y2 * P2 + o2, vb);
          sts<S, V>(YC + y2 * P2 + o2, vc);
        }
        Fm2 = Fm1, Fm1 = F.c, Wm2 = Wm1, Wm1 = W.c, Pq = P1, P1 = Pp;
      }
      rotate();
    }
  } else {  // ---------------- the 2-ring's columns: two sites of a row on one side
    const int ci = (ty - TYv - 4) * TXv + tx;
    const bool rc = ci < 2 * (tye + 8);
    const int rr = ci >> 1, side = ci & 1;
    const int oc = rr * SP + (side ? O + twe : O - 4), oi = oc + (side ? 0 : 2);  // four columns, the inner two
    const int b = wrap_n(b0 - 4 + (rc ? rr : 0), N), gc = wrap_n(side ? c0 + twe : c0 - 4, N), gi = gc + (side ? 0 : 2);
    const long long coff = (long long)N * b + gc, ioff = (long long)N * b + gi;
    const bool rc1 = rc && rr >= 2 && rr < tye + 6;  // rows of the 2-ring
    using P2v = Pack<S, 2>;
    CoarseCols<2> cc{};
    if constexpr (EqOf<EQ>::coarse) cc = coarse_cols<EQ, 2>(A.cmap, rc1, b, gi);
    P2v Fm1{}, Fm2{}, Wm1{}, Wm2{}, P1{}, Pq{};
    auto issue = [&](int s) {
      if (rc) {
#pragma unroll
        for (int h = 0; h < (int)sizeof(S) / 4; ++h) {  // four columns: one 16-byte piece in FP32, two in FP64
          constexpr int W16 = 16 / sizeof(S);
          cp_async_16(XF + s * P4 + oc + h * W16, A.xphi + on + coff + h * W16);
          cp_async_16(XW + s * P4 + oc + h * W16, A.xpi + on + coff + h * W16);
        }
      }
      cp_async_commit();
    };
    issue(i2);
    for (int p = a_begin - 4; p <= a_end + 3; ++p) {
      advance();
      cp_async_wait_all();
      P2v Fp{}, Pp{}, Wp{};
      if (rc) {
        const int ou = oc + (side ? 2 : 0);  // the outer two
        to_w(XF + i2 * P4 + ou, XW + i2 * P4 + ou, Fp, Pp, Wp);
        to_w(XF + i2 * P4 + oi, XW + i2 * P4 + oi, Fp, Pp, Wp);
      }
      step_barrier(NT);
      if (p <= a_end + 2) issue(i3);
      if (rc1) {
        RowStar13<S, 2> F, W;
        F.c = lds<S, 2>(XF + i0 * P4 + oi);
        W.c = lds<S, 2>(XW + i0 * P4 + oi);
        if (p >= a_begin) {
          Coupling<S, 2> ct, ch2;
          couple(ct, ch2, 0, 1, oq + ioff, aq, cc);
          F.template load<SP>(XF + i0 * P4, oi);
          F.b1 = Fm1, F.b2 = Fm2, F.a1 = lds<S, 2>(XF + i1 * P4 + oi), F.a2 = Fp;
          W.template load<SP>(XW + i0 * P4, oi);
          W.b1 = Wm1, W.b2 = Wm2, W.a1 = lds<S, 2>(XW + i1 * P4 + oi), W.a2 = Wp;
          P2v vb, vc, vbp, vap, vpp;
          phase1(F, W, Pq, ct, ch2, vb, vc, vbp, vap, vpp);
          sts<S, 2>(YB + y2 * P2 + oi - 2 * SP, vb);
          sts<S, 2>(YC + y2 * P2 + oi - 2 * SP, vc);
        }
        Fm2 = Fm1, Fm1 = F.c, Wm2 = Wm1, Wm1 = W.c, Pq = P1, P1 = Pp;
      }
      rotate();
    }
  }
  cp_async_wait_all();
}

}  // namespace cfb

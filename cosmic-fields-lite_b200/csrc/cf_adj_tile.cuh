// cf_adj_tile.cuh -- the exact reverse of one whole RK4 step in one pass over a (b, c)
// tile, marching along a (7-point Laplacian, Klein-Gordon operator; cf_adjoint.cu).
//
// With l' = (u, v) the adjoint of the new state and the reverse stages kb_i = (U_i, V_i),
// yb_i = ((-m^2 + inv lap) V_i, U_i - 3H V_i), only the phi part of yb_i has a spatial
// derivative, so chained over the four stages a step depends on l' within a distance
// of 2, as the forward step does on x (cf_step_tile.cuh):
//
//   pointwise      V_3 = dt/3 v + dt (dt/6 u - 3H dt/6 v)                       [t + dt]
//   phase 1 (plane q, tile and 1-ring): from lap v, lap V_3 -> yb_4, U_3, yb_3, U_2,
//     V_2 = dt/3 v + dt/2 yb_3.pi,  yb_2.pi,  V_1 = dt/6 v + dt/2 yb_2.pi
//   phase 2 (plane r, tile): from lap V_2, lap V_1 -> yb_2.phi, U_1, yb_1,
//     l = l' + yb_4 + yb_3 + yb_2 + yb_1
//
// dL/dm takes sum V_i y_i.phi, pointwise in phase 1 at the own sites, with the forward
// stage inputs y_i formed there from x (a 1-site ring) as phase 1 of the forward pass
// forms them (same kpi_of, same roundings, the context's storage type).
//
// HBM moves l' in, l out and x in once: 6 words per site-step.  The four reverse-stage
// passes and three forward-stage passes it replaces moved 65 (and took 212 us per step
// at N = 128 FP64).  What bounds it: FP64 latency and shared-memory traffic, as in the
// forward pass, with about twice its arithmetic; the tile (32 x 8 sites, 2 per thread)
// and the warp roles are those of the forward FP64 pass, at 3 CTAs per SM.
#pragma once

#include "cf_pair_tile.cuh"
#include "cf_stage_tile.cuh"
#include "cf_step_tile.cuh"

namespace cfb {

template <typename S>
struct AdjStepArgs {
  const double *lam;  // l' (2 N^3)
  double *out;        // l (another buffer)
  const S *x;         // the step's start state [phi | pi] (hi words in FP32_COMP)
  double *dm_partial; // per-CTA partial sums of dL/dm (accumulated across launches)
  int N, a_chunk;
  long long N3;
  double m2, inv[3], hub3[3];  // h^-2 a^-2 and 3H at t, t + dt/2, t + dt
  double dt, dt2, dt3, dt6, two_m;
};

template <typename S, int TXv, int TYv>
struct AdjSmem {
  static constexpr int V = 2, TW = TXv * V;
  static constexpr int O = 2, SP = TW + 2 * O;                  // FP64 planes
  static constexpr int OS = VecT<S>::n, SPS = TW + 2 * OS;      // x planes
  static constexpr int P2 = (TYv + 4) * SP, P1 = (TYv + 2) * SP, PX = (TYv + 2) * SPS, PD = TYv * TW;
  static constexpr size_t bytes = sizeof(double) * (6 * P2 + 4 * P1 + 8 * PD) + sizeof(S) * 6 * PX;
};

template <typename S, int TXv, int TYv, bool FULL>
__device__ __forceinline__ double adj_tile(const AdjStepArgs<S> &A, int c0, int b0, int a_begin, int a_end,
                                           unsigned char *smem) {
  using SM = AdjSmem<S, TXv, TYv>;
  using T = typename Arith<S>::T;
  constexpr int V = 2, TW = SM::TW, O = SM::O, SP = SM::SP, OS = SM::OS, SPS = SM::SPS;
  constexpr int P1 = SM::P1, P2 = SM::P2, PX = SM::PX, PD = SM::PD;
  constexpr int NT = TXv * (TYv + step_ring_rows(TXv, TYv));
  using PV = Pack<double, V>;
  using PS = Pack<S, V>;
  double *XV = reinterpret_cast<double *>(smem);  // v, 3 planes of P2
  double *XT = XV + 3 * P2;                       // u as it lands, then V_3; 3 planes of P2
  double *YB = XT + 3 * P2;                       // V_2, 2 planes of P1
  double *YC = YB + 2 * P1;                       // V_1, 2 planes of P1
  double *DL = YC + 2 * P1;                       // 2 planes x (acc.phi, acc.pi, u, v) of PD
  S *XF = reinterpret_cast<S *>(DL + 8 * PD);     // x_phi, 3 planes of PX
  S *XW = XF + 3 * PX;                            // x_pi as it lands, then ya_phi; 3 planes of PX
  const int N = A.N;
  const long long N3 = A.N3, NN = (long long)N * N;
  const int tx = threadIdx.x, ty = threadIdx.y;
  const int twe = FULL ? TW : min(TW, N - c0);
  const int tye = FULL ? TYv : min(TYv, N - b0);
  const bool colact = FULL || (tx * V) < twe;
  const int c = c0 + tx * V;
  const Coef<T> ch(A.dt2), cf(A.dt);
  const StageCoef<T> k1c{Coef<T>(A.m2), Coef<T>(A.inv[0]), Coef<T>(A.hub3[0]), Coef<T>(0.0), Coef<T>(0.0)};
  const StageCoef<T> k2c{Coef<T>(A.m2), Coef<T>(A.inv[1]), Coef<T>(A.hub3[1]), Coef<T>(0.0), Coef<T>(0.0)};
  const double *lu = A.lam, *lv = A.lam + N3;

  auto cpx = [](S *d, const S *g) {
    if constexpr (sizeof(S) == 8) cp_async_16(d, g);
    else cp_async_8(d, g);
  };
  auto v3_of = [&](double u, double v) {
    const double kv = A.dt6 * v, ku = A.dt6 * u;
    return A.dt3 * v + A.dt * (ku - A.hub3[2] * kv);
  };
  // V_3 over the u, ya_phi over the x_pi, of V sites a thread copied itself
  auto to_v3 = [&](double *pv, double *pu, PV &v, PV &u, PV &t) {
    v = lds<double, V>(pv);
    u = lds<double, V>(pu);
#pragma unroll
    for (int k = 0; k < V; ++k) t.v[k] = v3_of(u.v[k], v.v[k]);
    sts<double, V>(pu, t);
  };
  auto to_w = [&](S *pf, S *pp, PS &f, PS &p, PS &w) {
    f = lds<S, V>(pf);
    p = lds<S, V>(pp);
#pragma unroll
    for (int k = 0; k < V; ++k) w.v[k] = w_of(f.v[k], p.v[k], ch);
    sts<S, V>(pp, w);
  };
  struct P1Out {
    double v2, v1, accp, accq, v4;
  };
  // reverse stages 4 and 3 and the pointwise parts of 2 and 1 at one site
  auto phase1 = [&](double u, double v, double lapv, double v3, double lap3) {
    P1Out o;
    const double kv = A.dt6 * v, ku = A.dt6 * u;
    const double y4p = -A.m2 * kv + A.inv[2] * (A.dt6 * lapv), y4q = ku - A.hub3[2] * kv;
    const double u3 = A.dt3 * u + A.dt * y4p;
    const double y3p = -A.m2 * v3 + A.inv[1] * lap3, y3q = u3 - A.hub3[1] * v3;
    const double u2 = A.dt3 * u + A.dt2 * y3p;
    o.v2 = A.dt3 * v + A.dt2 * y3q;
    const double y2q = u2 - A.hub3[1] * o.v2;
    o.v1 = A.dt6 * v + A.dt2 * y2q;
    o.accp = y4p + y3p;
    o.accq = (y4q + y3q) + y2q;
    o.v4 = kv;
    return o;
  };

  double dm = 0.0;
  const int first = wrap_n(a_begin - 2, N);  // plane index of p = a_begin - 2
  if (ty < TYv) {  // ---------------- own rows
    const bool act = colact && (FULL || ty < tye);
    const int o2 = (ty + 2) * SP + O + tx * V, o1 = o2 - SP, od = ty * TW + tx * V;
    const int ox = (ty + 1) * SPS + OS + tx * V;
    const long long rowoff = (long long)N * (b0 + ty) + c;
    PV Vm{}, Tm{}, Uq{};  // v, V_3 of q - 1; u of q
    PS Fm{}, Wm{}, Pq{};  // x_phi, ya_phi of q - 1; x_pi of q
    int sq = 2, sp = 0, sn = 1, yq = 0;
    int an = first;
    long long on = NN * first + rowoff, opp = 0, oq = 0, orr = 0;
    auto issue = [&](int s) {
      if (act) {
        cp_async_16(XV + s * P2 + o2, lv + on);
        cp_async_16(XT + s * P2 + o2, lu + on);
        cpx(XF + s * PX + ox, A.x + on);
        cpx(XW + s * PX + ox, A.x + N3 + on);
      }
      cp_async_commit();
    };
    issue(0);
    for (int p = a_begin - 2; p <= a_end + 1; ++p) {
      orr = oq, oq = opp, opp = on, on += NN;
      if (++an == N) an = 0, on -= N3;
      cp_async_wait_all();  // this thread's copies of plane p have landed
      PV Vp{}, Up{}, Tp{};
      PS Fp{}, Pp{}, Wp{};
      if (act) {
        to_v3(XV + sp * P2 + o2, XT + sp * P2 + o2, Vp, Up, Tp);
        to_w(XF + sp * PX + ox, XW + sp * PX + ox, Fp, Pp, Wp);
      }
      step_barrier(NT);  // plane p in full; phase 2 of the last plane is done
      if (p <= a_end) issue(sn);
      if (act) {
        PV v2{}, v1{};
        const PV Vq = lds<double, V>(XV + sq * P2 + o2), Tq = lds<double, V>(XT + sq * P2 + o2);
        const PS Fq = lds<S, V>(XF + sq * PX + ox), Wq = lds<S, V>(XW + sq * PX + ox);
        PV v2m{}, v1m{};
        if (p >= a_begin) {  // phase 1 on plane q = p - 1
          RowStar<double, V, SP> D, E;
          D.load(XV + sq * P2, o2);
          D.c = Vq, D.a = Vp, D.b = Vm;
          E.load(XT + sq * P2, o2);
          E.c = Tq, E.a = Tp, E.b = Tm;
          double *dl = DL + yq * 4 * PD;
          PV ap, aq, v4;
#pragma unroll
          for (int k = 0; k < V; ++k) {
            const P1Out o = phase1(Uq.v[k], Vq.v[k], lap_of(D.template at<double>(k)), Tq.v[k],
                                   lap_of(E.template at<double>(k)));
            v2.v[k] = o.v2, v1.v[k] = o.v1, ap.v[k] = o.accp, aq.v[k] = o.accq, v4.v[k] = o.v4;
          }
          sts<double, V>(dl + od, ap);
          sts<double, V>(dl + PD + od, aq);
          sts<double, V>(dl + 2 * PD + od, Uq);
          sts<double, V>(dl + 3 * PD + od, Vq);
          double *yb = YB + yq * P1, *yc = YC + yq * P1;
          v2m = lds<double, V>(yb + o1);  // plane r - 1, whose slot plane q takes
          v1m = lds<double, V>(yc + o1);
          sts<double, V>(yb + o1, v2);
          sts<double, V>(yc + o1, v1);
          if (p >= a_begin + 1 && p <= a_end) {  // dL/dm, planes of this chunk
            RowStar<S, V, SPS> F, W;
            F.load(XF + sq * PX, ox);
            F.c = Fq, F.a = Fp, F.b = Fm;
            W.load(XW + sq * PX, ox);
            W.c = Wq, W.a = Wp, W.b = Wm;
            Coupling<S, V> none;
#pragma unroll
            for (int k = 0; k < V; ++k) {
              const T f0 = (T)Fq.v[k], p0 = (T)Pq.v[k], w0 = (T)Wq.v[k];
              const T k1 = kpi_of<EQ_FRW, S, V>(p0, f0, lap_of(F.template at<T>(k)), none, k, k1c);
              const S yapi = (S)ch.fma(k1, p0);
              const T k2 = kpi_of<EQ_FRW, S, V>((T)yapi, w0, lap_of(W.template at<T>(k)), none, k, k2c);
              const S bpi = (S)ch.fma(k2, p0);
              const S y3 = (S)ch.fma((T)yapi, f0), y4 = (S)cf.fma((T)bpi, f0);
              dm += v4.v[k] * (double)y4;
              dm += Tq.v[k] * (double)y3;
              dm += v2.v[k] * (double)w0;
              dm += v1.v[k] * (double)f0;
            }
          }
        }
        if (p >= a_begin + 2) {  // phase 2 on plane r = p - 2
          const int yr = yq ^ 1;
          const double *dl = DL + yr * 4 * PD;
          const PV ap = lds<double, V>(dl + od), aq = lds<double, V>(dl + PD + od);
          const PV u = lds<double, V>(dl + 2 * PD + od), v = lds<double, V>(dl + 3 * PD + od);
          RowStar<double, V, SP> B, C;
          B.load(YB + yr * P1, o1);
          C.load(YC + yr * P1, o1);
          B.c = lds<double, V>(YB + yr * P1 + o1), B.a = v2, B.b = v2m;
          C.c = lds<double, V>(YC + yr * P1 + o1), C.a = v1, C.b = v1m;
          PV op, oq2;
#pragma unroll
          for (int k = 0; k < V; ++k) {
            const double y2p = -A.m2 * B.c.v[k] + A.inv[1] * lap_of(B.template at<double>(k));
            const double u1 = A.dt6 * u.v[k] + A.dt2 * y2p;
            const double y1p = -A.m2 * C.c.v[k] + A.inv[0] * lap_of(C.template at<double>(k));
            const double y1q = u1 - A.hub3[0] * C.c.v[k];
            op.v[k] = u.v[k] + ((ap.v[k] + y2p) + y1p);
            oq2.v[k] = v.v[k] + (aq.v[k] + y1q);
          }
          stv(A.out + orr, op);
          stv(A.out + N3 + orr, oq2);
        }
        Vm = Vq, Tm = Tq, Fm = Fq, Wm = Wq, Uq = Up, Pq = Pp;
      }
      const int s0 = sq;
      sq = sp, sp = sn, sn = s0;
      yq ^= 1;
    }
  } else {  // ---------------- ring rows and columns
    const bool row = ty < TYv + 2 && colact;
    const int r2 = ty == TYv ? 1 : tye + 2;  // the 1-ring row, and the outer one
    const int r2o = ty == TYv ? 0 : tye + 3;
    const int o2 = r2 * SP + O + tx * V, o1 = o2 - SP, oo = r2o * SP + O + tx * V;
    const int ox = (r2 - 1) * SPS + OS + tx * V;
    const long long rowoff = (long long)N * wrap_n(b0 - 2 + r2, N) + c;
    const long long outoff = (long long)N * wrap_n(b0 - 2 + r2o, N) + c;
    // ring columns: the last 2 (tye + 4) threads take one row and side each (two columns)
    const int ci = NT - 1 - (ty * TXv + tx);
    const bool rc = ci < 2 * (tye + 4);
    const int rr = ci >> 1, side = ci & 1;
    const int oc = rr * SP + (side ? O + twe : O - 2), oi = oc + (side ? 0 : 1);  // the pair, its inner column
    const int gcc = wrap_n(side ? c0 + twe : c0 - 2, N);
    const long long coff = (long long)N * wrap_n(b0 - 2 + rr, N) + gcc;
    const bool rc1 = rc && rr >= 1 && rr <= tye + 2;  // ... of the 1-ring (and of x's)
    const int ocx = (rr - 1) * SPS + (side ? OS + twe : OS - 2);
    PV Vm{}, Tm{}, Uq{};
    double vm_c = 0, tm_c = 0, uq_c = 0;
    int sq = 2, sp = 0, sn = 1, yq = 0;
    int an = first;
    long long on = NN * first;
    auto issue = [&](int s) {
      double *xv = XV + s * P2, *xt = XT + s * P2;
      if (row) {
        cp_async_16(xv + o2, lv + on + rowoff);
        cp_async_16(xt + o2, lu + on + rowoff);
        cp_async_16(xv + oo, lv + on + outoff);
        cp_async_16(xt + oo, lu + on + outoff);
        cpx(XF + s * PX + ox, A.x + on + rowoff);
        cpx(XW + s * PX + ox, A.x + N3 + on + rowoff);
      }
      if (rc) {
        cp_async_16(xv + oc, lv + on + coff);
        cp_async_16(xt + oc, lu + on + coff);
      }
      if (rc1) {
        cpx(XF + s * PX + ocx, A.x + on + coff);
        cpx(XW + s * PX + ocx, A.x + N3 + on + coff);
      }
      cp_async_commit();
    };
    issue(0);
    for (int p = a_begin - 2; p <= a_end + 1; ++p) {
      on += NN;
      if (++an == N) an = 0, on -= N3;
      cp_async_wait_all();
      PV Vp{}, Up{}, Tp{};
      double up_c = 0;
      if (row) {
        to_v3(XV + sp * P2 + oo, XT + sp * P2 + oo, Vp, Up, Tp);
        to_v3(XV + sp * P2 + o2, XT + sp * P2 + o2, Vp, Up, Tp);
        PS f, q, w;
        to_w(XF + sp * PX + ox, XW + sp * PX + ox, f, q, w);
      }
      if (rc) {
        PV v, u, t;
        to_v3(XV + sp * P2 + oc, XT + sp * P2 + oc, v, u, t);
        up_c = side ? u.v[0] : u.v[1];
      }
      if (rc1) {
        PS f, q, w;
        to_w(XF + sp * PX + ocx, XW + sp * PX + ocx, f, q, w);
      }
      step_barrier(NT);
      if (p <= a_end) issue(sn);
      const double *xv = XV + sq * P2, *xt = XT + sq * P2;
      double *yb = YB + yq * P1, *yc = YC + yq * P1;
      if (row) {
        RowStar<double, V, SP> D, E;
        D.c = lds<double, V>(xv + o2);
        E.c = lds<double, V>(xt + o2);
        if (p >= a_begin) {
          D.load(xv, o2);
          D.a = Vp, D.b = Vm;
          E.load(xt, o2);
          E.a = Tp, E.b = Tm;
          PV v2, v1;
#pragma unroll
          for (int k = 0; k < V; ++k) {
            const P1Out o = phase1(Uq.v[k], D.c.v[k], lap_of(D.template at<double>(k)), E.c.v[k],
                                   lap_of(E.template at<double>(k)));
            v2.v[k] = o.v2, v1.v[k] = o.v1;
          }
          sts<double, V>(yb + o1, v2);
          sts<double, V>(yc + o1, v1);
        }
        Vm = D.c, Tm = E.c, Uq = Up;
      }
      if (rc1) {
        const double vc = xv[oi], tc = xt[oi];
        if (p >= a_begin) {
          const Star<double> ds{vc, XV[sp * P2 + oi], vm_c, xv[oi + SP], xv[oi - SP], xv[oi + 1], xv[oi - 1]};
          const Star<double> es{tc, XT[sp * P2 + oi], tm_c, xt[oi + SP], xt[oi - SP], xt[oi + 1], xt[oi - 1]};
          const P1Out o = phase1(uq_c, vc, lap_of(ds), tc, lap_of(es));
          yb[oi - SP] = o.v2;
          yc[oi - SP] = o.v1;
        }
        vm_c = vc, tm_c = tc, uq_c = up_c;
      }
      const int s0 = sq;
      sq = sp, sp = sn, sn = s0;
      yq ^= 1;
    }
  }
  return dm;
}

}  // namespace cfb

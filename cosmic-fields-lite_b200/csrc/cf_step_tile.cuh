// cf_step_tile.cuh -- one whole RK4 step in one pass over a (b, c) tile,
// marching along a (7-point Laplacian).
//
// In f(phi, pi) = (pi, F(phi, pi, lap phi)) only pi has a spatial derivative, so
// every stage input's phi is pointwise in the previous input (cf_pair_tile.cuh).
// Chained over the four stages that makes the whole step depend on x within a
// distance of 2 (stage 3 takes the Laplacian of yb_phi = x_phi + dt/2 ya_pi,
// ya_pi = x_pi + dt/2 k1_pi, k1_pi needs lap x_phi):
//
//   phase 1 (plane q, its tile and a 1-site ring):  from x (planes q-1..q+1, ring 2)
//     k1 = F(x_pi, x_phi, lap x_phi)                    [t]
//     ya_phi = x_phi + dt/2 x_pi,  ya_pi = x_pi + dt/2 k1
//     k2 = F(ya_pi, ya_phi, lap ya_phi)                 [t + dt/2]
//     yb = x + dt/2 (ya_pi, k2),  yc_phi = x_phi + dt yb_pi
//   phase 2 (plane r, its tile):  from yb_phi, yc_phi of planes r-1..r+1 (ring 1)
//     k3 = F(yb_pi, yb_phi, lap yb_phi)                 [t + dt/2]
//     yc_pi = x_pi + dt k3
//     k4 = F(yc_pi, yc_phi, lap yc_phi)                 [t + dt]
//     x += dt/6 (k1 + 2 k2 + 2 k3 + k4)
//
// While plane p = q + 1 streams in, phase 1 runs on plane q = p - 1 and phase 2 on
// plane r = p - 2.  HBM moves the state once (x hi in, x hi out to a second buffer,
// x lo in place) plus the curvature at three times: 8 (+6) words per site-update
// against 18 (+8) for the paired passes.  Every value is formed and rounded where
// the paired-stage kernels form and round it (same lap order, same kpi_of, the same
// storage-type roundings of the stage inputs and the accumulator), so the states are
// bit-identical.
//
// The new phi and pi go to a buffer other than x: ring sites of a plane belong to
// neighbouring tiles, and planes a_begin-2 .. a_end+1 to neighbouring a-chunks, which
// may have moved on already.  The lo words are touched only at a thread's own sites.
//
// ya_phi is formed once per site: when a thread's copies of plane p have landed it
// replaces x_pi by ya_phi in place (own sites, ring rows, ring columns; the x_pi that
// stages 1-4 still take stay with the thread), so phase 1 reads two finished planes
// instead of forming ya_phi at all seven points of every stencil (36 of 347 FP32
// instructions per 128 sites) -- the same value, rounded once, wherever it is read.
//
// A thread's own a-neighbours come from registers, not from shared memory: it marches
// along a, so the value it read as plane p is the next plane's centre and the one
// after's a - 1.  Shared memory per CTA: x_phi and x_pi / ya_phi with a 2-site ring in
// three planes each (p + 1 landing, p, q), yb_phi and yc_phi with a 1-site ring in two
// (q and r), and, in a ring of two, what phase 1 hands to phase 2 at the own sites (yb_pi
// and the accumulator).  The plane a thread copies next (p + 1) takes the slot of plane p
// - 2, last read before the barrier of plane p, so the copies are issued right after it:
// the one barrier per plane.  Rows have the interior at a 16-byte boundary, so a thread
// reads its sites and the rows next to them as 16-byte vectors (no bank conflicts), and
// only the two c-neighbours beyond its vector as single words.
//
// Warp roles: the own rows' warps run phases 1 and 2; the warps behind them (ring warps)
// form the 1-ring's rows and columns of phase 1.  Each role has a loop of its own, so a
// thread holds the registers of one role only (this, and keeping what one plane leaves for
// the next in registers or in shared memory by equation, StepKeep, is what fits the
// register budget: no spills but 4 to 8 bytes for the FP64 lambda phi^4 form and 4 to 24 for the
// FP64 approximate comoving one), and both meet at one named barrier per plane.
//
// What bounds it: latency and shared-memory bandwidth, not HBM -- at N = 256 the FP32 FRW
// pass issues in 51% of the cycles and the shared-memory pipe is busy in 69% (FP64: 82%).
// Measured against the form that read every stencil point from shared memory and formed
// ya_phi per point (N = 512, ms per step, FP32: FRW 1.18 -> 1.06, fixed Psi 1.40 -> 1.21,
// comoving with its Psi refreshes 2.34 -> 2.09; FP64 at N = 256: FRW 0.233 -> 0.192, sqrt
// potential 0.276 -> 0.266).  Measured and not taken: 2 floats or 1 double per thread
// (twice the warps: 10 to 20% slower), c-neighbours by warp shuffles (spills), 128 x 16 tiles
// at 1 CTA per SM.
#pragma once

#include "cf_stage_tile.cuh"

namespace cfb {

// FP32: the coefficients of StepArgs as lane pairs, formed once per launch (from the
// kernel's parameters they need no registers; N = 512 fixed Psi 1.43 -> 1.34 ms per step).
template <typename S>
struct StepCoefs {};
template <>
struct StepCoefs<float> {
  C2 m2f, q1f, q2f, invf[3], hubf[3], dt2f, dtf, dt6f;
};

template <typename S>
struct StepArgs : StepCoefs<S> {
  const S *xphi;  // state phi, pi (hi words in FP32_COMP), read only
  const S *xpi;
  S *ophi;        // the new phi, pi (another buffer)
  S *opi;
  const S *xlo;   // FP32_COMP lo words [phi | pi]
  S *olo;         // the new ones (may be xlo)
  const S *psi[3];   // curvature at t, t + dt/2, t + dt (StageArgs::psi / dpsi)
  const S *dpsi[3];
  const int *cmap;
  int M;
  int N;
  int a_chunk;
  long long N3;
  double q1, q2;
  double m2;
  double inv[3], hub3[3];  // h^-2 a^-2 and 3H at t, t + dt/2, t + dt
  double dt2, dt, dt6;
};
inline __host__ __device__ void step_coefs_f32(StepArgs<double> &) {}
inline __host__ __device__ void step_coefs_f32(StepArgs<float> &A) {
  A.m2f = coef_f32x2(A.m2);
  A.q1f = coef_f32x2(A.q1);
  A.q2f = coef_f32x2(A.q2);
  A.dt2f = coef_f32x2(A.dt2);
  A.dtf = coef_f32x2(A.dt);
  A.dt6f = coef_f32x2(A.dt6);
  for (int k = 0; k < 3; ++k) {
    A.invf[k] = coef_f32x2(A.inv[k]);
    A.hubf[k] = coef_f32x2(A.hub3[k]);
  }
}

// Sites per thread: 16-byte vectors, but 2 floats for the FP32 approximate comoving
// equation, whose coarse gathers hold 3 words per site and stage (N = 512: 1.84 -> 1.75 ms).
template <typename S, int EQ>
constexpr int step_vec() {
  return sizeof(S) == 4 && EQ == EQ_APPROX ? 2 : VecT<S>::n;
}

// What a thread of the own rows keeps in registers from plane to plane beyond x_phi and
// ya_phi of q - 1; the rest it reads back from shared memory:
//   x  x_phi, ya_phi of q as well       y  yb_phi, yc_phi of r and r - 1
//   p  x_pi of q and r (else in shared memory, 3 planes of own sites)
// FP64 is bound by shared memory, so the uncoupled equations keep all that fits the 96
// registers of 4 CTAs per SM (N = 256 FRW: x 0.202 -> 0.201, x and y 0.192 ms; on ragged tiles x and y spill: N = 200
// 0.118 -> 0.155).  The coupled equations hold the curvature of two stages in registers
// and need the room: FP32 comoving with x_pi in registers 2.70, in shared memory 2.36 ms
// (N = 512).
template <typename S, int EQ, bool FULL>
struct StepKeep {
  static constexpr bool wide = sizeof(S) == 8 && !EqOf<EQ>::coupled && EQ != EQ_SQRT;
  static constexpr bool x = wide, y = wide && FULL, p = !EqOf<EQ>::coupled || EQ == EQ_FIXED;
};

template <typename S, int EQ, int TXv, int TYv>
struct StepSmem {
  static constexpr int V = step_vec<S, EQ>();
  static constexpr int TW = TXv * V;
  static constexpr int O = VecT<S>::n;     // column of the first interior site (16-byte aligned)
  static constexpr int SP = TW + 2 * O;    // row pitch of every plane array
  static constexpr int R2 = TYv + 4, P2 = R2 * SP;  // 2-ring planes (x_phi, x_pi / ya_phi)
  static constexpr int R1 = TYv + 2, P1 = R1 * SP;  // 1-ring planes (yb_phi, yc_phi)
  static constexpr int PD = TYv * TW;               // own sites
  static constexpr int count = 3 * 2 * P2 + 2 * 2 * P1 + 2 * 3 * PD + (EqOf<EQ>::coupled && EQ != EQ_FIXED ? 3 * PD : 0);
};

// 7-point Laplacian sum in the order of lap_at: (-6 f0 + a+ + a- + b+ + b-) + (c+ + c-)
template <typename T>
__device__ __forceinline__ T lap7(T f0, T ap, T am, T bp, T bm, T cp, T cm) {
  if constexpr (sizeof(T) == 4) {
    return lap7_f32<float>(f0, ap, am, bp, bm, cp, cm);
  } else {
    const T s = (T)-6 * f0 + ap + am + bp + bm;
    return s + (cp + cm);
  }
}

// Curvature values of one site (a ring site of phase 1).
template <int EQ, typename S>
__device__ __forceinline__ void coupling_at(Coupling<S, 1> &cp, const S *psi, const S *dpsi, long long site,
                                            const int *cmap, int M, int a, int b, int c) {
  if constexpr (EqOf<EQ>::psi_plane) cp.ps.v[0] = __ldg(psi + site);
  if constexpr (EqOf<EQ>::dpsi_plane) cp.dps.v[0] = __ldg(dpsi + site);
  if constexpr (EqOf<EQ>::coarse) {
    const int idx = (__ldg(cmap + a) * M + __ldg(cmap + b)) * M + __ldg(cmap + c);
    cp.ps.v[0] = __ldg(psi + 4 * (long long)idx);
    cp.ps4.v[0] = __ldg(psi + 4 * (long long)idx + 1);
    cp.dps.v[0] = __ldg(psi + 4 * (long long)idx + 2);
  }
}

// Asynchronous global -> shared copies (cp.async; completion per commit group).
__device__ __forceinline__ void cp_async_16(void *smem, const void *gmem) {
  const unsigned s = (unsigned)__cvta_generic_to_shared(smem);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(s), "l"(gmem) : "memory");
}
__device__ __forceinline__ void cp_async_8(void *smem, const void *gmem) {
  const unsigned s = (unsigned)__cvta_generic_to_shared(smem);
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(s), "l"(gmem) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
// A hint that brings `bytes` (a multiple of 16, 16-byte aligned, inside an allocation)
// from global memory into L2 without occupying registers or shared memory.
__device__ __forceinline__ void prefetch_l2(const void *p, unsigned bytes) {
  asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;\n" ::"l"(p), "r"(bytes) : "memory");
}
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_group 0;\n" ::: "memory"); }

// A thread's V sites of a row, 16 bytes from shared memory.
template <typename S, int V>
__device__ __forceinline__ Pack<S, V> lds(const S *p) {
  return unpack<S, V>(*reinterpret_cast<const typename VecOf<S, V>::T *>(p));
}
template <typename S, int V>
__device__ __forceinline__ void sts(S *p, const Pack<S, V> &r) {
  stv<S, V>(p, r);
}

// One site's 7-point stencil values: centre, a+-, b+-, c+-.
template <typename T>
struct Star {
  T f0, ap, am, bp, bm, cp, cm;
};

// The stencil of the V sites of a row at `o` in planes (pm, p0, pp) of pitch SP, as vectors.
template <typename S, int V, int SP>
struct RowStar {
  Pack<S, V> c, n, s, a, b;
  S l, r;
  __device__ __forceinline__ void load(const S *p0, int o) {  // the neighbours in the plane
    n = lds<S, V>(p0 + o + SP);
    s = lds<S, V>(p0 + o - SP);
    l = p0[o - 1];
    r = p0[o + V];
  }
  template <typename T>
  __device__ __forceinline__ Star<T> at(int v) const {
    return Star<T>{(T)c.v[v], (T)a.v[v], (T)b.v[v], (T)n.v[v], (T)s.v[v], (T)(v + 1 < V ? c.v[v + 1] : r),
                   (T)(v > 0 ? c.v[v - 1] : l)};
  }
};

template <typename T>
__device__ __forceinline__ T lap_of(const Star<T> &s) {
  return lap7<T>(s.f0, s.ap, s.am, s.bp, s.bm, s.cp, s.cm);
}

// FP32: the stencil of sites (2l, 2l+1) of a row's four as lane pairs (cf_f32x2.cuh).
// The c-neighbours pair across the vector: lane 0 takes (c1, c2) and (l, c0), lane 1
// (c3, r) and (c1, c2).
template <int V, int SP>
__device__ __forceinline__ Star<float2> star2(const RowStar<float, V, SP> &R, int l) {
  const int v = 2 * l;
  if constexpr (V == 2)
    return Star<float2>{make_float2(R.c.v[0], R.c.v[1]), make_float2(R.a.v[0], R.a.v[1]),
                        make_float2(R.b.v[0], R.b.v[1]), make_float2(R.n.v[0], R.n.v[1]),
                        make_float2(R.s.v[0], R.s.v[1]), make_float2(R.c.v[1], R.r), make_float2(R.l, R.c.v[0])};
  else
  return Star<float2>{make_float2(R.c.v[v], R.c.v[v + 1]), make_float2(R.a.v[v], R.a.v[v + 1]),
                      make_float2(R.b.v[v], R.b.v[v + 1]), make_float2(R.n.v[v], R.n.v[v + 1]),
                      make_float2(R.s.v[v], R.s.v[v + 1]),
                      make_float2(R.c.v[v + 1], l == 0 ? R.c.v[2] : R.r),
                      make_float2(l == 0 ? R.l : R.c.v[1], R.c.v[v])};
}
__device__ __forceinline__ float2 lap_of2(const Star<float2> &s) {
  return lap7_f32<float2>(s.f0, s.ap, s.am, s.bp, s.bm, s.cp, s.cm);
}
template <int V>
__device__ __forceinline__ float2 lane2(const Pack<float, V> &p, int l) {
  return make_float2(p.v[2 * l], p.v[2 * l + 1]);
}
template <int V>
__device__ __forceinline__ void set2(Pack<float, V> &p, int l, float2 x) {
  p.v[2 * l] = x.x;
  p.v[2 * l + 1] = x.y;
}
// The curvature lanes of a stage (ps, dps, ps4 of kpi_f32; zero where the equation has none).
template <int EQ, int V>
__device__ __forceinline__ void coupling2(const Coupling<float, V> &c, int l, float2 &ps, float2 &dps, float2 &ps4) {
  ps = dps = ps4 = make_float2(0.0f, 0.0f);
  if constexpr (EqOf<EQ>::coupled) ps = lane2(c.ps, l);
  if constexpr (EQ == EQ_COMOV || EQ == EQ_APPROX) dps = lane2(c.dps, l);
  if constexpr (EQ == EQ_APPROX) ps4 = lane2(c.ps4, l);
}

// The coefficients of one site's arithmetic (T) at t, t + dt/2, t + dt.
template <typename S>
struct StepK {
  using T = typename Arith<S>::T;
  StageCoef<T> k1, k2, k4;
  Coef<T> ch, cf, c6;
  __device__ __forceinline__ explicit StepK(const StepArgs<double> &A)
      : k1(stage(A, 0)), k2(stage(A, 1)), k4(stage(A, 2)), ch(A.dt2), cf(A.dt), c6(A.dt6) {}
  __device__ __forceinline__ explicit StepK(const StepArgs<float> &A)
      : k1(stage(A, 0)), k2(stage(A, 1)), k4(stage(A, 2)), ch(A.dt2f.lane()), cf(A.dtf.lane()), c6(A.dt6f.lane()) {}
  __device__ __forceinline__ static StageCoef<double> stage(const StepArgs<double> &A, int k) {
    return {A.m2, A.inv[k], A.hub3[k], A.q1, A.q2};
  }
  __device__ __forceinline__ static StageCoef<float> stage(const StepArgs<float> &A, int k) {
    return {A.m2f.lane(), A.invf[k].lane(), A.hubf[k].lane(), A.q1f.lane(), A.q2f.lane()};
  }
};

// Thread rows beside the TYv rows of own sites: two that form the 1-ring's rows, and as
// many more as its columns need threads (one per row and side of the 2-ring) in whole warps.
constexpr int step_ring_rows(int TXv, int TYv) {
  int r = 2;
  while (r * TXv < 2 * (TYv + 4) || ((TYv + r) * TXv) % 32 != 0) ++r;
  return r;
}

// The least time of a plane, in the units of step_a_chunk (1.27 on a full SM): a lone CTA's chain of
// dependent steps.  Measured per plane with one CTA per SM against a full one: FP64 0.76 / 1.66
// us (5 of 20 warps), FP32 1.19 / 1.59 us, comoving 2.16 / 2.56 us (10 of 20 warps).  These are of the
// 7-point pass at 4 (FP64) or 2 CTAs per SM; at fewer a lone CTA has a larger share of a full SM's time
// (its callers' 4 / CTAs per SM).  In the 13-point pass's 2 or 1 CTAs per SM only the uncoupled FP32
// value exceeds 0.27 + c / per_sm at c = 1 and acts.
constexpr double step_latency(size_t word, bool coupled) { return word == 8 ? 0.62 : (coupled ? 1.05 : 0.95); }

__device__ __forceinline__ void step_barrier(int threads) { asm volatile("bar.sync 1, %0;\n" ::"r"(threads) : "memory"); }

template <typename S, int EQ, int TXv, int TYv, bool FULL = false>
__device__ __forceinline__ void step_tile(const StepArgs<S> &A, int c0, int b0, int a_begin, int a_end, S *smem) {
  using SM = StepSmem<S, EQ, TXv, TYv>;
  using T = typename Arith<S>::T;
  using KP = StepKeep<S, EQ, FULL>;
  constexpr int V = SM::V, TW = SM::TW, O = SM::O, SP = SM::SP, PD = SM::PD;
  constexpr int NT = TXv * (TYv + step_ring_rows(TXv, TYv));
  constexpr int P1 = SM::P1, P2 = SM::P2;
  static_assert((TXv * TYv) % 32 == 0 && NT % 32 == 0, "own rows and ring rows in warps of their own");
  S *XF = smem;           // x_phi, 3 planes of P2
  S *XW = XF + 3 * P2;    // x_pi as it lands, then ya_phi; 3 planes of P2
  S *YB = XW + 3 * P2;    // yb_phi, 2 planes of P1
  S *YC = YB + 2 * P1;    // yc_phi, 2 planes of P1
  S *DL = YC + 2 * P1;    // 2 planes x (yb_pi, acc_phi, acc_pi) of PD
  S *PK = DL + 6 * PD;    // x_pi of the own sites, 3 planes (not KP::p)
  const int N = A.N;
  const long long N3 = A.N3, NN = (long long)N * N;
  const int tx = threadIdx.x, ty = threadIdx.y;
  const int twe = FULL ? TW : min(TW, N - c0);
  const int tye = FULL ? TYv : min(TYv, N - b0);
  const bool colact = FULL || (tx * V) < twe;
  const int c = c0 + tx * V;

  const StepK<S> K(A);
  const StageCoef<T> &k1c = K.k1, &k2c = K.k2, &k4c = K.k4;
  const Coef<T> &ch = K.ch, &cf = K.cf, &c6 = K.c6;

  // ya_phi = x_phi + dt/2 x_pi over the x_pi of V sites a thread copied itself
  auto to_w = [&](S *xf, S *xp, Pack<S, V> &f, Pack<S, V> &q, Pack<S, V> &w) {
    f = lds<S, V>(xf);
    q = lds<S, V>(xp);
    if constexpr (sizeof(S) == 4) {
#pragma unroll
      for (int l = 0; l < V / 2; ++l) set2(w, l, c_fma(A.dt2f, lane2(q, l), lane2(f, l)));
    } else {
#pragma unroll
      for (int v = 0; v < V; ++v) w.v[v] = w_of(f.v[v], q.v[v], ch);
    }
    sts<S, V>(xp, w);
  };
  auto cpv = [](S *d, const S *g) {
    if constexpr (V * sizeof(S) == 16) cp_async_16(d, g);
    else cp_async_8(d, g);
  };
  // stages 1-2 at V sites of a row of plane q
  auto phase1 = [&](const RowStar<S, V, SP> &F, const RowStar<S, V, SP> &W, const Pack<S, V> &Pq, const Coupling<S, V> &ct,
                    const Coupling<S, V> &ch2, Pack<S, V> &vb, Pack<S, V> &vc, Pack<S, V> &vbp, Pack<S, V> &vap,
                    Pack<S, V> &vpp) {
    if constexpr (sizeof(S) == 4) {  // two sites per paired FP32 instruction, same bits
      const StageCoefL<float2> K1{A.m2f, A.invf[0], A.hubf[0], A.q1f, A.q2f}, K2{A.m2f, A.invf[1], A.hubf[1], A.q1f, A.q2f};
#pragma unroll
      for (int l = 0; l < V / 2; ++l) {
        const Star<float2> fs = star2(F, l), ws = star2(W, l);
        const float2 f0 = fs.f0, p0 = lane2(Pq, l);
        float2 c_ps, c_dps, c_ps4;
        coupling2<EQ>(ct, l, c_ps, c_dps, c_ps4);
        const float2 k1 = kpi_f32<EQ, float2>(p0, f0, lap_of2(fs), c_ps, c_dps, c_ps4, K1);
        const float2 yapi = c_fma(A.dt2f, k1, p0);
        coupling2<EQ>(ch2, l, c_ps, c_dps, c_ps4);
        const float2 k2 = kpi_f32<EQ, float2>(yapi, ws.f0, lap_of2(ws), c_ps, c_dps, c_ps4, K2);
        const float2 bpi = c_fma(A.dt2f, k2, p0);
        set2(vb, l, c_fma(A.dt2f, yapi, f0));
        set2(vc, l, c_fma(A.dtf, bpi, f0));
        set2(vbp, l, bpi);
        set2(vap, l, p_fma(p_splat<float2>(2.0f), yapi, p0));
        set2(vpp, l, p_fma(p_splat<float2>(2.0f), k2, k1));
      }
    } else {
#pragma unroll
      for (int v = 0; v < V; ++v) {
        const Star<T> fs = F.template at<T>(v), ws = W.template at<T>(v);
        const T f0 = fs.f0, p0 = (T)Pq.v[v];
        const T k1 = kpi_of<EQ, S, V>(p0, f0, lap_of(fs), ct, v, k1c);
        const S yapi = (S)ch.fma(k1, p0);
        const T k2 = kpi_of<EQ, S, V>((T)yapi, ws.f0, lap_of(ws), ch2, v, k2c);
        const S bpi = (S)ch.fma(k2, p0);
        vb.v[v] = (S)ch.fma((T)yapi, f0);
        vc.v[v] = (S)cf.fma((T)bpi, f0);
        vbp.v[v] = bpi;
        vap.v[v] = (S)((T)(S)p0 + (T)2 * (T)yapi);
        vpp.v[v] = (S)((T)(S)k1 + (T)2 * k2);
      }
    }
  };

  const int first = wrap_n(a_begin - 2, N);  // plane index of p = a_begin - 2
  if (ty < TYv) {  // ---------------- own rows
    const int b = b0 + ty;
    const bool act = colact && (FULL || ty < tye);
    const int o2 = (ty + 2) * SP + O + tx * V, o1 = o2 - SP, od = ty * TW + tx * V;
    const long long rowoff = (long long)N * b + c;
    CoarseCols<V> cc{};
    if constexpr (EqOf<EQ>::coarse) cc = coarse_cols<EQ, V>(A.cmap, act, b, c);
    // kept from plane to plane at the thread's sites: x_phi, ya_phi of q and q - 1, x_pi of q and r
    Pack<S, V> Fq{}, Wq{}, Pq{}, Fm{}, Wm{}, Pr{};
    Pack<S, V> Br{}, Cr{}, Bm{}, Cm{};  // yb_phi, yc_phi of r, r - 1 (KP::y)
    int sq = 2, sp = 0, sn = 1, yq = 0;
    int an = first;                      // plane index of p + 1
    long long on = NN * first + rowoff;  // its offset, and those of p, q, r
    long long opp = 0, oq = 0, orr = 0;
    int ap = 0, aq = 0, ar = 0;
    auto issue = [&](int s) {
      if (act) {
        cpv(XF + s * P2 + o2, A.xphi + on);
        cpv(XW + s * P2 + o2, A.xpi + on);
      }
      cp_async_commit();
    };
    issue(0);
    for (int p = a_begin - 2; p <= a_end + 1; ++p) {
      orr = oq, oq = opp, opp = on, on += NN;
      if constexpr (EqOf<EQ>::coarse) ar = aq, aq = ap, ap = an;
      if (++an == N) an = 0, on -= N3;
      cp_async_wait_all();  // this thread's copies of plane p have landed
      Pack<S, V> Fp{}, Pp{}, Wp{};
      if (act) {
        to_w(XF + sp * P2 + o2, XW + sp * P2 + o2, Fp, Pp, Wp);
        if constexpr (!KP::p) sts<S, V>(PK + sp * PD + od, Pp);
      }
      step_barrier(NT);  // plane p in full; phase 2 of the last plane is done
      if (p <= a_end) issue(sn);
      // L2 prefetch one plane ahead (phase 1 takes plane p next, phase 2 plane q)
      if (tx == 0 && act) {
        const unsigned bytes = (unsigned)(twe * sizeof(S));
        if (p >= a_begin - 1 && p <= a_end) {
          if constexpr (EqOf<EQ>::psi_plane) {
            prefetch_l2(A.psi[0] + opp, bytes);
            if constexpr (EQ != EQ_FIXED) prefetch_l2(A.psi[1] + opp, bytes);
          }
          if constexpr (EqOf<EQ>::dpsi_plane) {
            prefetch_l2(A.dpsi[0] + opp, bytes);
            prefetch_l2(A.dpsi[1] + opp, bytes);
          }
        }
        if (p - 1 >= a_begin && p <= a_end) {
          if constexpr (EqOf<EQ>::psi_plane && EQ != EQ_FIXED) prefetch_l2(A.psi[2] + oq, bytes);
          if constexpr (EqOf<EQ>::dpsi_plane) prefetch_l2(A.dpsi[2] + oq, bytes);
          if constexpr (sizeof(S) == 4) {
            prefetch_l2(A.xlo + oq, bytes);
            prefetch_l2(A.xlo + N3 + oq, bytes);
          }
        }
      }
      if (act) {
        const S *xf = XF + sq * P2, *xw = XW + sq * P2;
        Pack<S, V> vb{}, vc{}, vbp{}, vap{}, vpp{};
        if constexpr (!KP::x) {
          Fq = lds<S, V>(xf + o2);
          Wq = lds<S, V>(xw + o2);
        }
        if (p >= a_begin) {  // phase 1 on plane q = p - 1
          S *yb = YB + yq * P1, *yc = YC + yq * P1;
          Coupling<S, V> ct, ch2;
          if constexpr (EqOf<EQ>::coupled) {
            const int ca = EqOf<EQ>::coarse ? __ldg(A.cmap + aq) : 0;
            load_coupling<EQ, S, V>(ct, A.psi[0], A.dpsi[0], oq, A.M, ca, cc);
            if constexpr (EQ == EQ_FIXED)
              ch2 = ct;
            else
              load_coupling<EQ, S, V>(ch2, A.psi[1], A.dpsi[1], oq, A.M, ca, cc);
          }
          RowStar<S, V, SP> F, W;
          F.load(xf, o2);
          W.load(xw, o2);
          if constexpr (!KP::p) Pq = lds<S, V>(PK + sq * PD + od);
          F.c = Fq, F.a = Fp, F.b = Fm;
          W.c = Wq, W.a = Wp, W.b = Wm;
          phase1(F, W, Pq, ct, ch2, vb, vc, vbp, vap, vpp);
          if constexpr (!KP::y) {  // plane r - 1, whose slot plane q takes
            Bm = lds<S, V>(yb + o1);
            Cm = lds<S, V>(yc + o1);
          }
          sts<S, V>(yb + o1, vb);
          sts<S, V>(yc + o1, vc);
          S *dl = DL + yq * 3 * PD;
          sts<S, V>(dl + od, vbp);
          sts<S, V>(dl + PD + od, vap);
          sts<S, V>(dl + 2 * PD + od, vpp);
        }
        // phase 2: stages 3 and 4 and the update on plane r = p - 2
        if (p >= a_begin + 2) {
          const int yr = yq ^ 1;
          if constexpr (!KP::p) Pr = lds<S, V>(PK + sn * PD + od);
          Coupling<S, V> cth, cd;
          if constexpr (EqOf<EQ>::coupled) {
            const int ca = EqOf<EQ>::coarse ? __ldg(A.cmap + ar) : 0;
            load_coupling<EQ, S, V>(cth, A.psi[1], A.dpsi[1], orr, A.M, ca, cc);
            if constexpr (EQ == EQ_FIXED)
              cd = cth;
            else
              load_coupling<EQ, S, V>(cd, A.psi[2], A.dpsi[2], orr, A.M, ca, cc);
          }
          Pack<S, V> lp{}, lq{};
          if constexpr (sizeof(S) == 4) {
            lp = ldv_rw<S, V>(A.xlo + orr);
            lq = ldv_rw<S, V>(A.xlo + N3 + orr);
          }
          const S *dl = DL + yr * 3 * PD;
          const Pack<S, V> ybpi = lds<S, V>(dl + od), aphi = lds<S, V>(dl + PD + od), api = lds<S, V>(dl + 2 * PD + od);
          RowStar<S, V, SP> B, C;
          if constexpr (!KP::y) {
            Br = lds<S, V>(YB + yr * P1 + o1);
            Cr = lds<S, V>(YC + yr * P1 + o1);
          }
          B.load(YB + yr * P1, o1);
          C.load(YC + yr * P1, o1);
          B.c = Br, B.a = vb, B.b = Bm;
          C.c = Cr, C.a = vc, C.b = Cm;
          Pack<S, V> o1v, o2v, o3v, o4v;
          if constexpr (sizeof(S) == 4) {
            const StageCoefL<float2> K2{A.m2f, A.invf[1], A.hubf[1], A.q1f, A.q2f}, K4{A.m2f, A.invf[2], A.hubf[2], A.q1f, A.q2f};
#pragma unroll
            for (int l = 0; l < V / 2; ++l) {
              const Star<float2> bs = star2(B, l);
              const float2 p0 = lane2(ybpi, l);
              float2 c_ps, c_dps, c_ps4;
              coupling2<EQ>(cth, l, c_ps, c_dps, c_ps4);
              const float2 k3 = kpi_f32<EQ, float2>(p0, bs.f0, lap_of2(bs), c_ps, c_dps, c_ps4, K2);
              const float2 c1phi = p_fma(p_splat<float2>(2.0f), p0, lane2(aphi, l));
              const float2 c1pi = p_fma(p_splat<float2>(2.0f), k3, lane2(api, l));
              const float2 ycpi = c_fma(A.dtf, k3, lane2(Pr, l));
              const Star<float2> cs = star2(C, l);
              coupling2<EQ>(cd, l, c_ps, c_dps, c_ps4);
              const float2 k4 = kpi_f32<EQ, float2>(ycpi, cs.f0, lap_of2(cs), c_ps, c_dps, c_ps4, K4);
              float2 h1, l1, h2, l2;
              comp_update_f32<float2>(lane2(Fm, l), lane2(lp, l), p_add(c1phi, ycpi), A.dt6f, h1, l1);
              comp_update_f32<float2>(lane2(Pr, l), lane2(lq, l), p_add(c1pi, k4), A.dt6f, h2, l2);
              set2(o1v, l, h1);
              set2(o3v, l, l1);
              set2(o2v, l, h2);
              set2(o4v, l, l2);
            }
          } else {
#pragma unroll
            for (int v = 0; v < V; ++v) {
              const Star<T> bs = B.template at<T>(v);
              const T p0 = (T)ybpi.v[v];
              const T k3 = kpi_of<EQ, S, V>(p0, bs.f0, lap_of(bs), cth, v, k2c);
              const S c1phi = (S)((T)aphi.v[v] + (T)2 * p0);
              const S c1pi = (S)((T)api.v[v] + (T)2 * k3);
              const S ycpi = (S)cf.fma(k3, (T)Pr.v[v]);
              const Star<T> cs = C.template at<T>(v);
              const T k4 = kpi_of<EQ, S, V>((T)ycpi, cs.f0, lap_of(cs), cd, v, k4c);
              state_update(Fm.v[v], lp.v[v], (T)c1phi + (T)ycpi, c6, o1v.v[v], o3v.v[v]);
              state_update(Pr.v[v], lq.v[v], (T)c1pi + k4, c6, o2v.v[v], o4v.v[v]);
            }
          }
          stv(A.ophi + orr, o1v);
          stv(A.opi + orr, o2v);
          if constexpr (sizeof(S) == 4) {
            stv(A.olo + orr, o3v);
            stv(A.olo + N3 + orr, o4v);
          }
        }
        Fm = Fq, Wm = Wq;
        if constexpr (KP::p) Pr = Pq, Pq = Pp;
        if constexpr (KP::x) Fq = Fp, Wq = Wp;
        if constexpr (KP::y) Bm = Br, Cm = Cr, Br = vb, Cr = vc;
      }
      const int s0 = sq;
      sq = sp, sp = sn, sn = s0;
      yq ^= 1;
    }
  } else {  // ---------------- ring rows and columns
    const bool row = ty < TYv + 2 && colact;
    const int r2 = ty == TYv ? 1 : tye + 2;  // the 1-ring row, and the outer one
    const int r2o = ty == TYv ? 0 : tye + 3;
    const int b = wrap_n(b0 - 2 + r2, N);
    const int o2 = r2 * SP + O + tx * V, o1 = o2 - SP, oo = r2o * SP + O + tx * V;
    const long long rowoff = (long long)N * b + c;
    const long long outoff = (long long)N * wrap_n(b0 - 2 + r2o, N) + c - rowoff;
    // ring columns: the last 2 (tye + 4) threads take one row and side each (two columns)
    const int ci = NT - 1 - (ty * TXv + tx);
    const bool rc = ci < 2 * (tye + 4);
    const int rr = ci >> 1, side = ci & 1;
    const int oc = rr * SP + (side ? O + twe : O - 2), oi = oc + (side ? 0 : 1);  // the pair, its inner column
    const int gbc = wrap_n(b0 - 2 + rr, N), gcc = wrap_n(side ? c0 + twe : c0 - 2, N);
    const long long coff = (long long)N * gbc + gcc;
    const bool rc1 = rc && rr >= 1 && rr <= tye + 2;  // ... of the 1-ring
    const int gci = side ? gcc : gcc + 1;
    CoarseCols<V> cc{};
    if constexpr (EqOf<EQ>::coarse) cc = coarse_cols<EQ, V>(A.cmap, row, b, c);
    Pack<S, V> Fm{}, Wm{}, Pq{};
    S fm_c = 0, wm_c = 0, pq_c = 0;
    int sq = 2, sp = 0, sn = 1, yq = 0;
    int an = first, ap = 0, aq = 0;
    long long on = NN * first, opp = 0, oq = 0;
    auto issue = [&](int s) {
      S *xf = XF + s * P2, *xp = XW + s * P2;
      if (row) {
        cpv(xf + o2, A.xphi + on + rowoff);
        cpv(xp + o2, A.xpi + on + rowoff);
        cpv(xf + oo, A.xphi + on + rowoff + outoff);
        cpv(xp + oo, A.xpi + on + rowoff + outoff);
      }
      if (rc) {
        if constexpr (sizeof(S) == 8) {
          cp_async_16(xf + oc, A.xphi + on + coff);
          cp_async_16(xp + oc, A.xpi + on + coff);
        } else {
          cp_async_8(xf + oc, A.xphi + on + coff);
          cp_async_8(xp + oc, A.xpi + on + coff);
        }
      }
      cp_async_commit();
    };
    issue(0);
    for (int p = a_begin - 2; p <= a_end + 1; ++p) {
      oq = opp, opp = on, on += NN;
      aq = ap, ap = an;
      if (++an == N) an = 0, on -= N3;
      cp_async_wait_all();
      Pack<S, V> Fp{}, Pp{}, Wp{};
      S pp_c = 0;
      if (row) {
        to_w(XF + sp * P2 + oo, XW + sp * P2 + oo, Fp, Pp, Wp);
        to_w(XF + sp * P2 + o2, XW + sp * P2 + o2, Fp, Pp, Wp);
      }
      if (rc) {
        using V2 = typename VecOf<S, 2>::T;
        const V2 f = *reinterpret_cast<const V2 *>(XF + sp * P2 + oc);
        const V2 q = *reinterpret_cast<const V2 *>(XW + sp * P2 + oc);
        V2 w;
        w.x = w_of(f.x, q.x, ch);
        w.y = w_of(f.y, q.y, ch);
        *reinterpret_cast<V2 *>(XW + sp * P2 + oc) = w;
        pp_c = side ? q.x : q.y;
      }
      step_barrier(NT);
      if (p <= a_end) issue(sn);
      if (tx == 0 && row && p >= a_begin - 1 && p <= a_end) {
        const unsigned bytes = (unsigned)(twe * sizeof(S));
        if constexpr (EqOf<EQ>::psi_plane) {
          prefetch_l2(A.psi[0] + opp + rowoff, bytes);
          if constexpr (EQ != EQ_FIXED) prefetch_l2(A.psi[1] + opp + rowoff, bytes);
        }
        if constexpr (EqOf<EQ>::dpsi_plane) {
          prefetch_l2(A.dpsi[0] + opp + rowoff, bytes);
          prefetch_l2(A.dpsi[1] + opp + rowoff, bytes);
        }
      }
      const S *xf = XF + sq * P2, *xw = XW + sq * P2;
      S *yb = YB + yq * P1, *yc = YC + yq * P1;
      if (row) {
        RowStar<S, V, SP> F, W;
        F.c = lds<S, V>(xf + o2);
        W.c = lds<S, V>(xw + o2);
        if (p >= a_begin) {
          Coupling<S, V> ct, ch2;
          if constexpr (EqOf<EQ>::coupled) {
            const int ca = EqOf<EQ>::coarse ? __ldg(A.cmap + aq) : 0;
            load_coupling<EQ, S, V>(ct, A.psi[0], A.dpsi[0], oq + rowoff, A.M, ca, cc);
            if constexpr (EQ == EQ_FIXED)
              ch2 = ct;
            else
              load_coupling<EQ, S, V>(ch2, A.psi[1], A.dpsi[1], oq + rowoff, A.M, ca, cc);
          }
          F.load(xf, o2);
          W.load(xw, o2);
          F.a = Fp, F.b = Fm;
          W.a = Wp, W.b = Wm;
          Pack<S, V> vb, vc, vbp, vap, vpp;
          phase1(F, W, Pq, ct, ch2, vb, vc, vbp, vap, vpp);
          sts<S, V>(yb + o1, vb);
          sts<S, V>(yc + o1, vc);
        }
        Fm = F.c, Wm = W.c, Pq = Pp;
      }
      if (rc1) {
        const S fc = xf[oi], wc = xw[oi];
        if (p >= a_begin) {
          const long long site = oq + (long long)N * gbc + gci;
          Coupling<S, 1> ct, ch2;
          if constexpr (EqOf<EQ>::coupled) {
            coupling_at<EQ, S>(ct, A.psi[0], A.dpsi[0], site, A.cmap, A.M, aq, gbc, gci);
            if constexpr (EQ == EQ_FIXED)
              ch2 = ct;
            else
              coupling_at<EQ, S>(ch2, A.psi[1], A.dpsi[1], site, A.cmap, A.M, aq, gbc, gci);
          }
          const Star<T> fs{(T)fc, (T)XF[sp * P2 + oi], (T)fm_c, (T)xf[oi + SP], (T)xf[oi - SP], (T)xf[oi + 1], (T)xf[oi - 1]};
          const Star<T> ws{(T)wc, (T)XW[sp * P2 + oi], (T)wm_c, (T)xw[oi + SP], (T)xw[oi - SP], (T)xw[oi + 1], (T)xw[oi - 1]};
          const T p0 = (T)pq_c;
          const T k1 = kpi_of<EQ, S, 1>(p0, fs.f0, lap_of(fs), ct, 0, k1c);
          const S yapi = (S)ch.fma(k1, p0);
          const T k2 = kpi_of<EQ, S, 1>((T)yapi, ws.f0, lap_of(ws), ch2, 0, k2c);
          const S bpi = (S)ch.fma(k2, p0);
          yb[oi - SP] = (S)ch.fma((T)yapi, fs.f0);
          yc[oi - SP] = (S)cf.fma((T)bpi, fs.f0);
        }
        fm_c = fc, wm_c = wc, pq_c = pp_c;
      }
      const int s0 = sq;
      sq = sp, sp = sn, sn = s0;
      yq ^= 1;
    }
  }
  cp_async_wait_all();
  __syncthreads();
}

}  // namespace cfb

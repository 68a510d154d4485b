// cf_energy.cuh -- the energy density of a state, one warp per 64 sites of a row (shared by the
// single-lattice observers and the ensembles).
#pragma once

#include "cf_stage_tile.cuh"

namespace cfb {

// ---- energy density -----------------------------------------------------
// Potential term of the energy density by equation (ED_*):
//   ED_QUAD    1/2 m^2 phi^2                                (src/equations_cuda.cu:332-369, lambda = 0)
//   ED_LAMBDA  1/2 m^2 phi^2 + 1/4 lambda phi^4              (:332-369)
//   ED_SQRT    m^2 f_a^2 (sqrt(1 + phi^2/f_a^2) - 1)         (:431-449)
//   ED_CURV    1/2 m^2 phi^2 with e^{-2Psi} kinetic and e^{2Psi} gradient weights (:451-473)
// and rho = 1/2 pi^2 w_k + 1/8 inv w_g sum_axes (phi_{+1} - phi_{-1})^2 + V
// (src/equations.cpp:38-69, :106-138, :265-322 for the CPU twins).  `psi` holds
// e^{2 Psi} - 1.  The sqrt potential is formed as m^2 phi^2 / (sqrt(1 + phi^2/f_a^2) + 1),
// the same value without the cancellation of sqrt(1 + u) - 1 at small u.
enum EdKind : int { ED_QUAD = 0, ED_LAMBDA = 1, ED_SQRT = 2, ED_CURV = 3 };

// A warp takes 64 sites of a row (two per lane, moved as one vector) and marches along a:
// phi of planes a - 1, a, a + 1 is read and widened once per plane and kept in registers, the
// c-neighbours come from the lanes beside, the rows b +- 1 from L1 (a CTA's 8 warps take
// consecutive b).  No barrier: a warp's loads of a plane are independent of each other and
// of the other warps.  With a row per block and every stencil point loaded and widened on
// its own the pass waited on memory at a third of the bandwidth: N = 512 FP32_COMP comoving
// 1.14 -> 0.84 ms (28 bytes per site: 0.58 at the copy rate).
// SQUARES: returns the lane's sum of rho^2 over its sites (in increasing a): the
// lattice's sum, by Parseval N^-3 times that of the spectrum, scales the binning (cf_spectrum.cu).
// MEAN: instead of rho, its mean over a (summed in increasing a, then divided by N; one chunk of
// all planes) and its slice at a = 0, each optional.
template <typename S>
struct EnergyArgs {
  const S *x, *xlo, *psi;
  double *rho;
  double *slice, *mean;
  int N, a_chunk;
  double m2, inv, q;
};
constexpr int ED_TILE = 64;

template <typename S, int ED, bool MEAN, bool SQUARES = false>
__device__ __forceinline__ double energy_march(const EnergyArgs<S> &A, long long task, int a0, int a1) {
  using V2 = typename VecOf<S, 2>::T;
  // Two planes a turn, whose loads the compiler interleaves only for the mean: for rho that takes 78
  // registers and a CTA of the SM (N = 512 559 -> 646 us), with the squares also where it may not.
  constexpr int U = SQUARES ? 1 : 2;
  const int N = A.N, lane = threadIdx.x & 31;
  const long long NN = (long long)N * N, N3 = NN * N;
  const int b = (int)(task % N), c0 = (int)(task / N) * ED_TILE;
  const int c = c0 + 2 * lane;
  const bool act = c < N;
  const int last = min(ED_TILE, N - c0) / 2 - 1;  // the last active lane (N % 8 == 0: not lane 0)
  const long long row = (long long)N * b + (act ? c : c0);
  const long long up = (long long)N * (b + 1 == N ? 1 - N : 1), down = (long long)N * (b == 0 ? N - 1 : -1);
  // the c-neighbour beyond the tile: of lane 0 to the left, of the last lane to the right
  const long long edge = (long long)N * b + (lane == 0 ? (c0 == 0 ? N - 1 : c0 - 1) : (c + 2 >= N ? 0 : c + 2));
  const bool at_edge = act && (lane == 0 || lane == last);
  auto pair = [&](const S *p, const S *lo, long long i) -> double2 {
    const V2 h = *reinterpret_cast<const V2 *>(p + i);
    double2 v = make_double2((double)h.x, (double)h.y);
    if constexpr (sizeof(S) == 4) {
      const V2 l = *reinterpret_cast<const V2 *>(lo + i);
      v.x += (double)l.x;
      v.y += (double)l.y;
    }
    return v;
  };
  auto one = [&](long long i) -> double {
    double v = (double)A.x[i];
    if constexpr (sizeof(S) == 4) v += (double)A.xlo[i];
    return v;
  };
  double2 prev = pair(A.x, A.xlo, NN * (a0 == 0 ? N - 1 : a0 - 1) + row), cur = pair(A.x, A.xlo, NN * a0 + row);
  const bool vec = (reinterpret_cast<unsigned long long>(A.rho) & 15) == 0;  // a caller's rho may be 8-byte aligned
  double ss = 0.0;
  double2 sum = make_double2(0.0, 0.0);
#pragma unroll U
  for (int a = a0; a < a1; ++a) {
    const long long pl = NN * a;
    const double2 next = pair(A.x, A.xlo, NN * (a + 1 == N ? 0 : a + 1) + row);
    const double2 n = pair(A.x, A.xlo, pl + row + up), s = pair(A.x, A.xlo, pl + row + down);
    const double2 p = pair(A.x + N3, A.xlo + N3, pl + row);
    double e = 0.0;
    if (at_edge) e = one(pl + edge);
    double2 g = make_double2(0.0, 0.0);
    if constexpr (ED == ED_CURV) {
      const V2 t = *reinterpret_cast<const V2 *>(A.psi + pl + row);
      g = make_double2((double)t.x, (double)t.y);
    }
    double left = __shfl_up_sync(0xffffffffu, cur.y, 1), right = __shfl_down_sync(0xffffffffu, cur.x, 1);
    if (lane == 0) left = e;
    if (lane == last) right = e;
    auto site = [&](double f, double fp, double fm, double fn, double fs, double fr, double fl, double pi, double e2m1) {
      const double dx = fp - fm, dy = fn - fs, dz = fr - fl;
      const double grad = dx * dx + dy * dy + dz * dz;
      if constexpr (ED == ED_CURV) {
        const double w = 1.0 + e2m1;
        return 0.5 * (pi * pi / w + A.m2 * f * f + w * 0.25 * A.inv * grad);
      } else if constexpr (ED == ED_LAMBDA) {
        return 0.5 * (pi * pi + A.m2 * f * f + 0.25 * A.inv * grad) + 0.25 * A.q * f * f * f * f;
      } else if constexpr (ED == ED_SQRT) {  // q = 1 / f_a^2
        return 0.5 * (pi * pi + 0.25 * A.inv * grad) + A.m2 * f * f / (sqrt(1.0 + f * f * A.q) + 1.0);
      } else {
        return 0.5 * (pi * pi + A.m2 * f * f + 0.25 * A.inv * grad);
      }
    };
    const double2 r = make_double2(site(cur.x, next.x, prev.x, n.x, s.x, cur.y, left, p.x, g.x),
                                   site(cur.y, next.y, prev.y, n.y, s.y, right, cur.x, p.y, g.y));
    if constexpr (MEAN) {
      if (act && A.slice && a == 0) A.slice[row] = r.x, A.slice[row + 1] = r.y;  // 8-byte aligned
      sum.x += r.x;
      sum.y += r.y;
    } else {
      if (act) {
        double *o = A.rho + pl + row;
        if (vec)
          *reinterpret_cast<double2 *>(o) = r;
        else
          o[0] = r.x, o[1] = r.y;
      }
      if (SQUARES && act) ss += r.x * r.x + r.y * r.y;
    }
    if constexpr (!MEAN && !SQUARES) asm volatile("" ::: "memory");
    prev = cur, cur = next;
  }
  if constexpr (MEAN) {
    if (act && A.mean) A.mean[row] = sum.x / (double)N, A.mean[row + 1] = sum.y / (double)N;
  }
  return ss;
}

// Warp tasks of a lattice (8 a CTA).
inline long long energy_tasks(int N) { return (long long)N * ((N + ED_TILE - 1) / ED_TILE); }

// CTAs per SM: 64 registers for the forms with a polynomial potential and, by its launch bound, the
// FP64 sqrt potential; up to 80 for the others.
constexpr int energy_per_sm(int ed, size_t word) { return ed <= ED_LAMBDA || (ed == ED_SQRT && word == 8) ? 4 : 3; }

// Planes per warp: chunks of at most 32 (two planes more are read per chunk), shorter while
// `lattices` of them give fewer than 16 warps per SM.  Where the CTAs of such chunks make at most
// two waves, the chunk whose planes (and two more) times waves are least: us, FP64, N = 160 FRW
// 28.6 -> 23.0, N = 200 FRW 55.6 -> 43.2, comoving 70.1 -> 59.3, N = 224 FRW 64.0 -> 55.6.
inline int energy_chunk(int N, int lattices, int per_sm) {
  int ch = 32;
  while (ch > 2 && lattices * energy_tasks(N) * ((N + ch - 1) / ch) < 148LL * 16) ch /= 2;
  const long long row = lattices * ((energy_tasks(N) + 7) / 8), slots = 148LL * per_sm;
  auto waves = [&](int c) { return (row * ((N + c - 1) / c) + slots - 1) / slots; };
  if (ch < 32 || waves(32) > 2) return ch;
  for (int c : {24, 16, 12, 8})
    if (waves(c) * (c + 2) < waves(ch) * (ch + 2)) ch = c;
  return ch;
}

}  // namespace cfb

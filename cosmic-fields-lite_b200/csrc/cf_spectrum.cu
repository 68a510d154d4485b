// cf_spectrum.cu -- energy density, deterministic spectrum binning, spectra.
//
// The reference bins |f_k|^2 into s^2 bins with FP64 atomicAdd, whose result
// depends on the order the atomics land in (src/fdm3d_cuda.cu:3-27, comment at
// :25).  Here every mode value is converted to a 128-bit fixed-point integer
// whose scale is a power of two chosen from an order-independent upper bound on
// any bin -- the largest mode value times the entry count (a max pass over the
// modes), or by Parseval a sum over the lattice that an earlier pass forms in a fixed order: of
// rho^2 in the energy pass for the density spectrum, of the state in the widening of an FP32_COMP
// state for the mode spectrum -- and the bins accumulate those
// integers with 64-bit integer atomics (carry propagated to the high word).
// Integer addition is associative, so the bins are bit-reproducible, and the
// sums are exact up to the fixed-point resolution (2^-126 of the bound).
// Unit-width |k| shells are then exact integer regroupings of the s^2 bins.

#include <cuda_runtime.h>
#include <cufft.h>

#include <algorithm>
#include <cmath>

#include "cf_energy.cuh"
#include "cf_internal.cuh"

namespace cfb {

// The sum over a CTA of 256 threads, in a fixed order; thread 0 has it.
__device__ __forceinline__ double cta_sum(double v) {
  __shared__ double w[8];
  for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
  if ((threadIdx.x & 31) == 0) w[threadIdx.x >> 5] = v;
  __syncthreads();
  double t = w[0];
  for (int k = 1; k < 8; ++k) t += w[k];
  return t;
}

// The sum of v over a grid of CTAs of 256 threads, in a fixed order, as a bit pattern in B.total: each
// CTA leaves its sum, and the one that arrives last adds them (the count wraps to 0 by itself).
struct GridSum {
  double *part;               // a word per CTA
  unsigned *arrived;          // 0 between grids
  unsigned long long *total;
};
__device__ __forceinline__ void grid_sum(const GridSum &B, double v, unsigned cta, unsigned ctas) {
  __shared__ bool last;
  const double t = cta_sum(v);
  if (threadIdx.x == 0) {
    B.part[cta] = t;
    __threadfence();
    last = atomicInc(B.arrived, ctas - 1) == ctas - 1;
  }
  __syncthreads();
  if (!last) return;
  __threadfence();
  double s = 0.0;
  for (unsigned i = threadIdx.x; i < ctas; i += 256) s += __ldcg(B.part + i);
  s = cta_sum(s);
  if (threadIdx.x == 0) *B.total = (unsigned long long)__double_as_longlong(s);
}

// The FP64 sqrt potential is held to 64 registers (4 CTAs per SM, 8 bytes spilled): N = 256 111 -> 89
// us, N = 512 751 -> 651.
template <typename S, int ED, bool SQUARES>
__global__ void __launch_bounds__(256, energy_per_sm(ED, sizeof(S)))
    k_energy(const EnergyArgs<S> A, const GridSum B) {
  const long long task = (long long)blockIdx.x * 8 + (threadIdx.x >> 5);
  const int a0 = blockIdx.y * A.a_chunk;
  double ss = 0.0;
  if (task < (long long)A.N * ((A.N + ED_TILE - 1) / ED_TILE))  // whole warps
    ss = energy_march<S, ED, false, SQUARES>(A, task, a0, min(a0 + A.a_chunk, A.N));
  if constexpr (SQUARES) grid_sum(B, ss, blockIdx.y * gridDim.x + blockIdx.x, gridDim.x * gridDim.y);
}

// The mean over a (and the slice at a = 0): one warp sums a column of 64 sites, so there are few
// warps, each with more loads in flight at 3 CTAs per SM (72 to 80 registers) than at 4.
template <typename S, int ED, int PER_SM>
__global__ void __launch_bounds__(256, PER_SM) k_energy_mean(const EnergyArgs<S> A) {
  const long long task = (long long)blockIdx.x * 8 + (threadIdx.x >> 5);
  if (task >= (long long)A.N * ((A.N + ED_TILE - 1) / ED_TILE)) return;
  const int a0 = blockIdx.y * A.a_chunk;  // 0
  energy_march<S, ED, true>(A, task, a0, min(a0 + A.a_chunk, A.N));
}
// 4 CTAs per SM where that makes one wave of what 3 would need two for (N = 512, FP32 comoving 0.95
// -> 0.72 ms).
static int mean_per_sm(int N) {
  const long long n = (energy_tasks(N) + 7) / 8;
  return n > 148 * 3 && n <= 148 * 4 ? 4 : 3;
}

// d rho / dt of the FRW Klein-Gordon equation (src/equations_cuda.cu:372-424):
//   pi lap_inv + 1/4 inv sum_axes (dpi_e)(dphi_e) - 3H (rho + p),
//   rho = 1/2 pi^2 + 1/8 inv G + 1/2 m^2 phi^2,  p = 1/2 pi^2 - 1/2 m^2 phi^2 - 1/24 inv G,
// with dphi_e, dpi_e the central differences (phi_{+e} - phi_{-e}) along each axis,
// G = sum_e dphi_e^2 and lap_inv = inv times the 7-point Laplacian sum.
template <typename S>
__global__ void k_dot_energy(const S *__restrict__ x, const S *__restrict__ xlo, double *__restrict__ out, int N,
                             double m2, double inv, double H_t) {
  const long long N3 = (long long)N * N * N;
  const long long NN = (long long)N * N;
  const long long stride = (long long)gridDim.x * blockDim.x;
  auto val = [&](long long i) -> double {
    double v = (double)x[i];
    if (xlo) v += (double)xlo[i];
    return v;
  };
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < N3; i += stride) {
    const int c = (int)(i % N);
    const int b = (int)((i / N) % N);
    const int a = (int)(i / NN);
    const long long nb[6] = {NN * ((a + 1) % N) + (long long)N * b + c, NN * ((a + N - 1) % N) + (long long)N * b + c,
                             NN * a + (long long)N * ((b + 1) % N) + c, NN * a + (long long)N * ((b + N - 1) % N) + c,
                             NN * a + (long long)N * b + (c + 1) % N, NN * a + (long long)N * b + (c + N - 1) % N};
    const double f = val(i), p = val(N3 + i);
    double G = 0.0, cross = 0.0, lap = -6.0 * f;
#pragma unroll
    for (int e = 0; e < 3; ++e) {
      const double fp = val(nb[2 * e]), fm = val(nb[2 * e + 1]);
      const double df = fp - fm;
      const double dp = val(N3 + nb[2 * e]) - val(N3 + nb[2 * e + 1]);
      G += df * df;
      cross += dp * df;
      lap += fp + fm;
    }
    const double rho = 0.5 * p * p + (0.5 / 4.0) * inv * G + 0.5 * m2 * f * f;
    const double pr = 0.5 * p * p - 0.5 * m2 * f * f - (1.0 / 4.0 / 6.0) * inv * G;
    out[i] = p * (inv * lap) + 0.25 * inv * cross - 3.0 * H_t * (rho + pr);
  }
}

// FP32_COMP state -> FP64 [phi | pi] (hi + lo).
__global__ void k_export_f32(const float *__restrict__ s, double *__restrict__ out, long long n2) {
  const long long stride = (long long)gridDim.x * blockDim.x;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n2; i += stride)
    out[i] = (double)s[i] + (double)s[n2 + i];
}

// The same for the mode spectrum, with the sum of phi^2 + pi^2 / m^2: by Parseval N^3 times
// it bounds the sum of the weighted mode values |phi_k|^2 + |pi_k|^2 / (m^2 + k^2 / a^2),
// so the binning needs no pass over the modes to find their maximum.
__global__ void __launch_bounds__(256) k_export_bound_f32(const float *__restrict__ s, double *__restrict__ out,
                                                          long long n2, double inv_m2, const GridSum B) {
  const long long stride = 2LL * gridDim.x * blockDim.x;
  double ss = 0.0;
  for (long long i = 2 * ((long long)blockIdx.x * blockDim.x + threadIdx.x); i < n2; i += stride) {
    const float2 h = *reinterpret_cast<const float2 *>(s + i), l = *reinterpret_cast<const float2 *>(s + n2 + i);
    const double2 v = make_double2((double)h.x + (double)l.x, (double)h.y + (double)l.y);
    *reinterpret_cast<double2 *>(out + i) = v;
    const double q = v.x * v.x + v.y * v.y;
    ss += 2 * i < n2 ? q : q * inv_m2;
  }
  grid_sum(B, ss, blockIdx.x, gridDim.x);
}

// FP64 [phi | pi] -> FP32_COMP state.
__global__ void k_import_f32(const double *__restrict__ in, float *__restrict__ s, long long n2) {
  const long long stride = (long long)gridDim.x * blockDim.x;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n2; i += stride) {
    const double v = in[i];
    const float h = (float)v;
    s[i] = h;
    s[n2 + i] = (float)(v - (double)h);
  }
}

__global__ void k_count_nonfinite(const void *__restrict__ s, long long n, int is_f32,
                                  unsigned long long *__restrict__ bad) {
  const long long stride = (long long)gridDim.x * blockDim.x;
  unsigned long long local = 0;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride) {
    double v = is_f32 ? (double)((const float *)s)[i] : ((const double *)s)[i];
    if (!isfinite(v)) ++local;
  }
  for (int o = 16; o > 0; o >>= 1) local += __shfl_down_sync(0xffffffffu, local, o);
  if ((threadIdx.x & 31) == 0 && local) atomicAdd(bad, local);
}

// ---- binning --------------------------------------------------------------
struct SpecIn {
  const double *f;  // HC of the field (or phi)
  const double *g;  // HC of dphi (mode spectrum) or nullptr
  int N;
  double k2;   // (2 pi / L)^2
  double m2;   // m^2
  double a2;   // a_t^2
};

// weighted mode value of HC entry (a, b, c): weight 2 for 0 < c < N/2 (the
// entry stands for the conjugate pair c and N - c of the full grid).
__device__ __forceinline__ double mode_value(const SpecIn &A, long long i, int c, long long s2) {
  const double fr = A.f[2 * i], fi = A.f[2 * i + 1];
  double v = fr * fr + fi * fi;
  if (A.g) {
    const double gr = A.g[2 * i], gi = A.g[2 * i + 1];
    v += (gr * gr + gi * gi) / (A.m2 + A.k2 * (double)s2 / A.a2);
  }
  return (c == 0 || 2 * c == A.N) ? v : 2.0 * v;
}

__device__ __forceinline__ void decode_mode(int N, long long i, int &c, long long &s2) {
  const int nh = N / 2 + 1;
  c = (int)(i % nh);
  const long long ab = i / nh;
  const int b = (int)(ab % N);
  const int a = (int)(ab / N);
  const long long as = (a <= N / 2) ? a : N - a;
  const long long bs = (b <= N / 2) ? b : N - b;
  s2 = as * as + bs * bs + (long long)c * c;
}

// ---- orbits of the binning ---------------------------------------------------
// The HC rows (a, b) whose modes share s^2 at every c: a in {as, N - as}, b in
// {bs, N - bs} and, for as != bs, the same with a and b swapped, 0 <= as <= bs <=
// N/2 -- up to 8 rows, and every row lies in exactly one orbit.  A warp takes one
// orbit and its lanes the c values, so the reads are coalesced along c; a lane sums
// the 128-bit fixed-point words of its modes in registers and adds the sum to the
// bin with one pair of 64-bit atomics.  Integer addition is associative, so a bin
// is the same integer as with one atomic pair per mode, at an eighth of the atomics
// (a quarter on the axes).
struct Orbit {
  int as, bs, na, nb, n;  // na, nb: 1 on an axis (0 or N/2), else 2; n rows
  long long ab2;          // as^2 + bs^2
};

__device__ __forceinline__ long long orbit_count(int N) { return (long long)(N / 2 + 1) * (N / 2 + 2) / 2; }

// Orbit o = bs (bs + 1) / 2 + as (0 <= as <= bs <= N/2).
__device__ __forceinline__ bool orbit_of(int N, long long o, Orbit &ob) {
  const int h = N / 2;
  if (o >= orbit_count(N)) return false;
  int bs = (int)((sqrt(8.0 * (double)o + 1.0) - 1.0) * 0.5);
  while ((long long)(bs + 1) * (bs + 2) / 2 <= o) ++bs;
  while ((long long)bs * (bs + 1) / 2 > o) --bs;
  ob.as = (int)(o - (long long)bs * (bs + 1) / 2);
  ob.bs = bs;
  ob.na = (ob.as == 0 || ob.as == h) ? 1 : 2;
  ob.nb = (bs == 0 || bs == h) ? 1 : 2;
  ob.n = ob.na * ob.nb * (ob.as != bs ? 2 : 1);
  ob.ab2 = (long long)ob.as * ob.as + (long long)bs * bs;
  return true;
}

// Row a N + b of the orbit's r-th row (r < n): first a in {as, N - as} with b in {bs,
// N - bs}, then (as != bs) a in {bs, N - bs} with b in {as, N - as}.
__device__ __forceinline__ long long orbit_row(const Orbit &ob, int r, int N) {
  const int m = ob.na * ob.nb;
  int a, b;
  if (r < m) {
    const int i = ob.nb == 2 ? r >> 1 : r, j = ob.nb == 2 ? r & 1 : 0;
    a = i ? N - ob.as : ob.as;
    b = j ? N - ob.bs : ob.bs;
  } else {
    const int q = r - m;
    const int i = ob.na == 2 ? q >> 1 : q, j = ob.na == 2 ? q & 1 : 0;
    a = i ? N - ob.bs : ob.bs;
    b = j ? N - ob.as : ob.as;
  }
  return (long long)a * N + b;
}

// Largest weighted mode value (blockIdx.y: batch entry, HC arrays hc_count apart).
__global__ void __launch_bounds__(256) k_spec_max(SpecIn A, long long hc_count, unsigned long long *maxbits) {
  A.f += (long long)blockIdx.y * hc_count;
  Orbit ob;
  if (!orbit_of(A.N, (long long)blockIdx.x * 8 + (threadIdx.x >> 5), ob)) return;  // whole warps
  const int nh = A.N / 2 + 1;
  long long rows[8];
#pragma unroll
  for (int r = 0; r < 8; ++r) rows[r] = r < ob.n ? orbit_row(ob, r, A.N) * nh : 0;
  double m = 0.0;
  for (int c = threadIdx.x & 31; c < nh; c += 32) {
    const long long s2 = ob.ab2 + (long long)c * c;
#pragma unroll
    for (int r = 0; r < 8; ++r)
      if (r < ob.n) m = fmax(m, mode_value(A, rows[r] + c, c, s2));
  }
  for (int o = 16; o > 0; o >>= 1) m = fmax(m, __shfl_down_sync(0xffffffffu, m, o));
  // non-negative doubles order like their bit patterns
  if ((threadIdx.x & 31) == 0) atomicMax(maxbits + blockIdx.y, (unsigned long long)__double_as_longlong(m));
}

// Power-of-two exponent e with (m * pairs) * 2^e <= 2^126, m the largest mode value or a sum that
// bounds them (a rounded one: the two bits above leave room); 0 without a finite one.
__device__ __forceinline__ int fixed_exponent(unsigned long long maxbits, long long pairs) {
  const double m = __longlong_as_double((long long)maxbits);
  if (!(m > 0.0) || isinf(m)) return 0;
  int ex;
  frexp(m * (double)pairs, &ex);  // m*pairs < 2^ex
  return 126 - ex;
}

// One mode value as a 128-bit fixed-point word (lo, hi) at scale 2^e, truncated.
__device__ __forceinline__ void to_fixed(double v, int e, unsigned long long &lo, unsigned long long &hi) {
  const double y = ldexp(v, e);
  hi = __double2ull_rz(ldexp(y, -64));
  lo = __double2ull_rz(y - ldexp((double)hi, 64));
}

// (lo, hi) += (l, h), 128-bit.
__device__ __forceinline__ void add128(unsigned long long &lo, unsigned long long &hi, unsigned long long l,
                                       unsigned long long h) {
  const unsigned long long nl = lo + l;
  hi += h + (nl < lo ? 1ull : 0ull);
  lo = nl;
}

__device__ __forceinline__ void atomic_add128(unsigned long long *bin, unsigned long long lo, unsigned long long hi) {
  unsigned long long carry = 0;
  if (lo) {
    const unsigned long long old = atomicAdd(bin, lo);
    carry = (old + lo < old) ? 1ull : 0ull;
  }
  if (hi + carry) atomicAdd(bin + 1, hi + carry);
}

// Bins of the weighted mode values (blockIdx.y: batch entry; bins 2 nb words apart).
__global__ void __launch_bounds__(256) k_spec_bin(SpecIn A, long long hc_count, long long pairs,
                                                  const unsigned long long *maxbits, unsigned long long *bins,
                                                  long long nb) {
  A.f += (long long)blockIdx.y * hc_count;
  bins += 2 * nb * (long long)blockIdx.y;
  Orbit ob;
  if (!orbit_of(A.N, (long long)blockIdx.x * 8 + (threadIdx.x >> 5), ob)) return;
  const int e = fixed_exponent(maxbits[blockIdx.y], pairs);
  const int nh = A.N / 2 + 1;
  long long rows[8];
#pragma unroll
  for (int r = 0; r < 8; ++r) rows[r] = r < ob.n ? orbit_row(ob, r, A.N) * nh : 0;
  // two c values per iteration: twice the loads in flight (the pass waits on memory;
  // 3.05 -> 2.97 ms per density spectrum at N = 512)
#pragma unroll 2
  for (int c = threadIdx.x & 31; c < nh; c += 32) {
    const long long s2 = ob.ab2 + (long long)c * c;
    unsigned long long lo = 0, hi = 0;
#pragma unroll
    for (int r = 0; r < 8; ++r)
      if (r < ob.n) {
        unsigned long long l, h;
        to_fixed(mode_value(A, rows[r] + c, c, s2), e, l, h);
        add128(lo, hi, l, h);
      }
    atomic_add128(bins + 2 * s2, lo, hi);
  }
}

// (lo, hi) 2^-e, rounded once: the top 64 bits with what is below them in the last one.  (Rounding the
// two words and their sum, a bin whose high word passes 53 bits carried up to two roundings more.)
__device__ __forceinline__ double fixed_to_double(unsigned long long lo, unsigned long long hi, int e) {
  if (hi == 0) return ldexp(__ull2double_rn(lo), -e);
  const int s = __clzll((long long)hi);
  unsigned long long top = s ? (hi << s) | (lo >> (64 - s)) : hi;
  if (lo << s) top |= 1;
  return ldexp(__ull2double_rn(top), 64 - s - e);
}

__global__ void k_spec_final(const unsigned long long *bins, const unsigned long long *maxbits, long long pairs,
                             double *out, long long nb) {
  const int e = fixed_exponent(*maxbits, pairs);
  const long long stride = (long long)gridDim.x * blockDim.x;
  for (long long s = (long long)blockIdx.x * blockDim.x + threadIdx.x; s < nb; s += stride)
    out[s] = fixed_to_double(bins[2 * s], bins[2 * s + 1], e);
}

// A warp per shell, its lanes the shell's s^2 bins (shell i holds 2i + 1 of them): the
// 128-bit integer sums do not depend on the order.  (A thread per shell walked them in turn:
// 276 us at N = 512, 47 us at N = 128.)
__global__ void __launch_bounds__(256) k_shells(const unsigned long long *bins, const unsigned long long *maxbits,
                                                long long pairs, const long long *s2counts, double *shells,
                                                long long *counts, long long nb, long long ns) {
  const long long i = (long long)blockIdx.x * 8 + (threadIdx.x >> 5);
  if (i >= ns) return;
  const int lane = threadIdx.x & 31;
  unsigned long long lo = 0, hi = 0;
  long long cnt = 0;
  const long long s_end = min((i + 1) * (i + 1), nb);
  for (long long s = i * i + lane; s < s_end; s += 32) {
    add128(lo, hi, bins[2 * s], bins[2 * s + 1]);
    cnt += s2counts[s];
  }
  for (int o = 16; o > 0; o >>= 1) {
    const unsigned long long l = __shfl_down_sync(0xffffffffu, lo, o), h = __shfl_down_sync(0xffffffffu, hi, o);
    add128(lo, hi, l, h);
    cnt += __shfl_down_sync(0xffffffffu, cnt, o);
  }
  if (lane == 0) {
    if (shells) shells[i] = fixed_to_double(lo, hi, fixed_exponent(*maxbits, pairs));
    if (counts) counts[i] = cnt;
  }
}

__global__ void __launch_bounds__(256) k_s2_counts(int N, unsigned long long *counts) {
  Orbit ob;
  if (!orbit_of(N, (long long)blockIdx.x * 8 + (threadIdx.x >> 5), ob)) return;
  for (int c = threadIdx.x & 31; c <= N / 2; c += 32)
    atomicAdd(&counts[ob.ab2 + (long long)c * c], (unsigned long long)ob.n * ((c == 0 || 2 * c == N) ? 1ull : 2ull));
}

// ---- batched binning (blockIdx.y = batch entry; used by ensembles) ----------
__global__ void k_specb_final(const unsigned long long *bins, const unsigned long long *maxbits, long long pairs,
                              double *out, long long nb) {
  const int e = fixed_exponent(maxbits[blockIdx.y], pairs);
  const unsigned long long *bb = bins + 2 * nb * blockIdx.y;
  double *o = out + nb * blockIdx.y;
  const long long stride = (long long)gridDim.x * blockDim.x;
  for (long long s = (long long)blockIdx.x * blockDim.x + threadIdx.x; s < nb; s += stride)
    o[s] = fixed_to_double(bb[2 * s], bb[2 * s + 1], e);
}

// Blocks of 8 warps, one orbit per warp.
static unsigned orbit_blocks(int N) {
  const long long norb = (long long)(N / 2 + 1) * (N / 2 + 2) / 2;
  return (unsigned)((norb + 7) / 8);
}

int bin_batched(const double *hc, int N, int batch, unsigned long long *maxbits, unsigned long long *bins, double *out,
                long long nb, cudaStream_t st, cf_ctx *) {
  const long long hc_count = 2LL * N * N * (N / 2 + 1), pairs = hc_count / 2;
  CF_TRY_CUDA(cudaMemsetAsync(maxbits, 0, sizeof(unsigned long long) * batch, st));
  CF_TRY_CUDA(cudaMemsetAsync(bins, 0, sizeof(unsigned long long) * 2 * nb * batch, st));
  SpecIn A{};
  A.f = hc;
  A.N = N;
  const unsigned gx = orbit_blocks(N);
  k_spec_max<<<dim3(gx, batch), 256, 0, st>>>(A, hc_count, maxbits);
  CF_TRY_CUDA(cudaGetLastError());
  k_spec_bin<<<dim3(gx, batch), 256, 0, st>>>(A, hc_count, pairs, maxbits, bins, nb);
  CF_TRY_CUDA(cudaGetLastError());
  const unsigned gf = (unsigned)std::min<long long>((nb + 255) / 256, 148LL * 8);
  k_specb_final<<<dim3(gf, batch), 256, 0, st>>>(bins, maxbits, pairs, out, nb);
  CF_TRY_CUDA(cudaGetLastError());
  return CF_OK;
}

static unsigned grid_for(long long n, int per = 256) {
  long long b = (n + per - 1) / per;
  if (b > 148LL * 32) b = 148LL * 32;
  if (b < 1) b = 1;
  return (unsigned)b;
}

// The scratch of the spectra, all of it or none: a later call takes spec_hc for the sign that it is there.
static int alloc_spectrum_scratch(cf_ctx *ctx) {
  const size_t hc = (size_t)ctx->hc_count, nb = (size_t)ctx->s2_bins;
  void *p[5] = {};
  const size_t bytes[5] = {2 * hc * sizeof(double), 2 * (size_t)ctx->N3 * sizeof(double),
                           2 * nb * sizeof(unsigned long long), 2 * sizeof(unsigned long long), nb * sizeof(int64_t)};
  cudaError_t e = cudaSuccess;
  for (int k = 0; k < 5 && e == cudaSuccess; ++k) e = cudaMalloc(&p[k], bytes[k]);
  const bool nomem = e != cudaSuccess;
  for (int k = 2; k < 5 && e == cudaSuccess; ++k) e = cudaMemset(p[k], 0, bytes[k]);
  if (e == cudaSuccess) {
    k_s2_counts<<<orbit_blocks((int)ctx->N), 256>>>((int)ctx->N, (unsigned long long *)p[4]);
    ctx->launches++;
    e = cudaGetLastError();
  }
  if (e == cudaSuccess) e = cudaDeviceSynchronize();
  if (e != cudaSuccess) {
    cudaGetLastError();
    for (void *q : p) cudaFree(q);
    set_error("spectrum scratch (%zu bytes): %s", bytes[0] + bytes[1] + bytes[2] + bytes[3] + bytes[4], cudaGetErrorString(e));
    return nomem ? CF_ERR_NOMEM : CF_ERR_CUDA;
  }
  ctx->spec_hc = (double *)p[0];
  ctx->spec_field = (double *)p[1];
  ctx->bins = (unsigned long long *)p[2];
  ctx->maxbits = (unsigned long long *)p[3];
  ctx->s2_counts = (int64_t *)p[4];
  return CF_OK;
}

int ensure_spectrum_scratch(cf_ctx *ctx, int nfields) {
  if (!ctx->spec_hc) CF_TRY(alloc_spectrum_scratch(ctx));
  const int N = (int)ctx->N;
  if (nfields >= 1 && !ctx->have_d2z1) {
    CF_TRY_CUFFT(cufftPlan3d(&ctx->plan_d2z1, N, N, N, CUFFT_D2Z));
    ctx->have_d2z1 = true;
  }
  if (nfields >= 2 && !ctx->have_d2z2) {
    long long n[3] = {N, N, N};
    long long inembed[3] = {N, N, N};
    long long onembed[3] = {N, N, N / 2 + 1};
    size_t work = 0;
    CF_TRY_CUFFT(cufftCreate(&ctx->plan_d2z2));
    CF_TRY_CUFFT(cufftMakePlanMany64(ctx->plan_d2z2, 3, n, inembed, 1, ctx->N3, onembed, 1, ctx->hc_count / 2,
                                     CUFFT_D2Z, 2, &work));
    ctx->have_d2z2 = true;
  }
  return CF_OK;
}

// Bins the HC data already in ctx->spec_hc (1 field, or phi/dphi for the mode spectrum).
// bound_mult = 0: a max pass finds the largest weighted mode value and the scale bounds
// it times the HC entry count.  bound_mult > 0: ctx->maxbits already holds a value m
// with m * bound_mult >= the sum of all weighted mode values.
static int bin_spectrum(cf_ctx *ctx, bool mode, double a_t, double *d_out, cudaStream_t st,
                        long long bound_mult = 0) {
  const long long pairs = bound_mult > 0 ? bound_mult : ctx->hc_count / 2;
  ctx->spec_mult = pairs;
  SpecIn A{};
  A.f = ctx->spec_hc;
  A.g = mode ? ctx->spec_hc + ctx->hc_count : nullptr;
  A.N = (int)ctx->N;
  const double kir = 2 * 3.14159265358979323846 / ctx->p.L;
  A.k2 = kir * kir;
  A.m2 = ctx->p.m * ctx->p.m;
  A.a2 = a_t * a_t;
  ProfScope ps(ctx, CF_PROF_SPECTRUM, st);
  CF_TRY_CUDA(cudaMemsetAsync(ctx->bins, 0, 2 * (size_t)ctx->s2_bins * sizeof(unsigned long long), st));
  if (bound_mult <= 0) {
    CF_TRY_CUDA(cudaMemsetAsync(ctx->maxbits, 0, sizeof(unsigned long long), st));
    k_spec_max<<<orbit_blocks(A.N), 256, 0, st>>>(A, 0, ctx->maxbits);
    CF_LAUNCHED(ctx);
  }
  k_spec_bin<<<orbit_blocks(A.N), 256, 0, st>>>(A, 0, pairs, ctx->maxbits, ctx->bins, ctx->s2_bins);
  CF_LAUNCHED(ctx);
  if (d_out) {
    k_spec_final<<<grid_for(ctx->s2_bins), 256, 0, st>>>(ctx->bins, ctx->maxbits, pairs, d_out, ctx->s2_bins);
    CF_LAUNCHED(ctx);
  }
  return CF_OK;
}

int power_spectrum_s2(cf_ctx *ctx, const double *d_f, double *d_out, cudaStream_t st) {
  CF_TRY(ensure_spectrum_scratch(ctx, 1));
  CF_TRY_CUFFT(cufftSetStream(ctx->plan_d2z1, st));
  {
    ProfScope ps(ctx, CF_PROF_SPECTRUM, st);
    CF_TRY_CUFFT(cufftExecD2Z(ctx->plan_d2z1, (cufftDoubleReal *)d_f, (cufftDoubleComplex *)ctx->spec_hc));
  }
  return bin_spectrum(ctx, false, 1.0, d_out, st);
}

// The sum a bound comes from, into ctx->maxbits.  The CTAs' words are the bins, which the binning clears
// afterwards (2 s2_bins = 1.5 N^2 + 2 words; k_energy makes at most N^2 / 8 CTAs for N <= 64, max(4736,
// N^3 / 2048) beyond, the widening at most min(592, N^3 / 256)).
static GridSum grid_sum_of(cf_ctx *ctx) {
  return GridSum{(double *)ctx->bins, (unsigned *)(ctx->maxbits + 1), ctx->maxbits};
}

int mode_power_spectrum_s2(cf_ctx *ctx, const void *d_state, double a_t, double *d_out, cudaStream_t st) {
  CF_TRY(ensure_spectrum_scratch(ctx, 2));
  const double *x = (const double *)d_state;
  long long bound = 0;
  if (ctx->p.precision != CF_FP64) {
    // The state is widened for the transform anyway, so its sums come along and bound the bins
    // (N = 512: the 0.49 ms of the max pass) unless the bound could be more than 2^20 above the
    // sum of the mode values (k_max^2 against a^2 m^2).  The fixed point then keeps 2^-106 of that sum
    // at least, the max pass (largest value times entry count) 2^-100 at N = 512.  An FP64 state
    // would need a pass of its own.
    const long long n2 = 2 * ctx->N3;
    const double m2 = ctx->p.m * ctx->p.m, k = 3.14159265358979323846 * ctx->N / ctx->p.L;
    if (3.0 * k * k < 1048576.0 * m2 * a_t * a_t) {
      bound = ctx->N3;
      // 4 CTAs per SM: more of them queue for the count (N = 128, us per spectrum 107 with 4736, 102 with 592)
      k_export_bound_f32<<<std::min(grid_for(n2 / 2), 148u * 4), 256, 0, st>>>((const float *)d_state, ctx->spec_field, n2,
                                                                              1.0 / m2, grid_sum_of(ctx));
    } else {
      k_export_f32<<<grid_for(n2), 256, 0, st>>>((const float *)d_state, ctx->spec_field, n2);
    }
    CF_LAUNCHED(ctx);
    x = ctx->spec_field;
  }
  CF_TRY_CUFFT(cufftSetStream(ctx->plan_d2z2, st));
  {
    ProfScope ps(ctx, CF_PROF_SPECTRUM, st);
    CF_TRY_CUFFT(cufftExecD2Z(ctx->plan_d2z2, (cufftDoubleReal *)x, (cufftDoubleComplex *)ctx->spec_hc));
  }
  return bin_spectrum(ctx, true, a_t, d_out, st, bound);
}

// What the energy passes write: rho (and, optional, the sum of its squares), or its mean over a and
// its slice.
struct EnergyOut {
  double *rho = nullptr;
  bool squares = false;  // the sum of rho^2 as well (grid_sum_of)
  double *slice = nullptr, *mean = nullptr;
};

template <typename S, int ED>
static int launch_energy(cf_ctx *ctx, const void *d_state, const void *psi, const EnergyOut &o, double m2, double inv,
                         double q, cudaStream_t st) {
  const long long N3 = ctx->N3;
  const int N = (int)ctx->N;
  const S *x = (const S *)d_state;
  EnergyArgs<S> A{x, sizeof(S) == 4 ? x + 2 * N3 : x, (const S *)psi, o.rho, o.slice, o.mean, N, N, m2, inv, q};
  const unsigned gx = (unsigned)((energy_tasks(N) + 7) / 8);
  if (o.rho) {
    A.a_chunk = energy_chunk(N, 1, energy_per_sm(ED, sizeof(S)));
    const unsigned chunks = (unsigned)((N + A.a_chunk - 1) / A.a_chunk);
    if (o.squares)
      k_energy<S, ED, true><<<dim3(gx, chunks), 256, 0, st>>>(A, grid_sum_of(ctx));
    else
      k_energy<S, ED, false><<<dim3(gx, chunks), 256, 0, st>>>(A, GridSum{});
    CF_LAUNCHED(ctx);
    return CF_OK;
  }
  A.a_chunk = o.mean ? N : 1;  // the slice alone takes the first plane
  if (mean_per_sm(N) == 4)
    k_energy_mean<S, ED, 4><<<gx, 256, 0, st>>>(A);
  else
    k_energy_mean<S, ED, 3><<<gx, 256, 0, st>>>(A);
  CF_LAUNCHED(ctx);
  return CF_OK;
}

template <int ED>
static int launch_energy_p(cf_ctx *ctx, const void *d_state, const void *psi, const EnergyOut &o, double m2, double inv,
                           double q, cudaStream_t st) {
  if (ctx->p.precision == CF_FP32_COMP) return launch_energy<float, ED>(ctx, d_state, psi, o, m2, inv, q, st);
  return launch_energy<double, ED>(ctx, d_state, psi, o, m2, inv, q, st);
}

static int energy_density_b(cf_ctx *ctx, const void *d_state, double t, const EnergyOut &o, cudaStream_t st) {
  double inv, H;
  stage_coeffs(ctx->p, t, &inv, &H);
  const double m2 = ctx->p.m * ctx->p.m;
  const int eq = ctx->p.equation;
  const void *ps = nullptr, *dps = nullptr;
  // the approximate comoving equation reports the full comoving energy density
  // (src/equations_cuda.cu:812-815)
  if (eq == CF_EQ_COMOVING_FRW || eq == CF_EQ_APPROX_COMOVING_FRW) CF_TRY(psi_at(ctx, t, st, &ps, &dps));
  if (eq == CF_EQ_FIXED_CURVATURE_FRW) ps = ctx->fixed_e2m1;
  ProfScope prof(ctx, CF_PROF_SPECTRUM, st);
  if (ps) return launch_energy_p<ED_CURV>(ctx, d_state, ps, o, m2, inv, 0.0, st);
  if (eq == CF_EQ_LAMBDA_FRW) return launch_energy_p<ED_LAMBDA>(ctx, d_state, nullptr, o, m2, inv, ctx->p.lambda, st);
  if (eq == CF_EQ_SQRT_FRW)
    return launch_energy_p<ED_SQRT>(ctx, d_state, nullptr, o, m2, inv, 1.0 / (ctx->p.f_a * ctx->p.f_a), st);
  return launch_energy_p<ED_QUAD>(ctx, d_state, nullptr, o, m2, inv, 0.0, st);
}

int energy_density(cf_ctx *ctx, const void *d_state, double t, double *d_rho, cudaStream_t st) {
  EnergyOut o;
  o.rho = d_rho;
  return energy_density_b(ctx, d_state, t, o, st);
}

int dot_energy_density(cf_ctx *ctx, const void *d_state, double t, double *d_out, cudaStream_t st) {
  double inv, H;
  stage_coeffs(ctx->p, t, &inv, &H);
  const double m2 = ctx->p.m * ctx->p.m;
  const long long N3 = ctx->N3;
  ProfScope prof(ctx, CF_PROF_SPECTRUM, st);
  if (ctx->p.precision == CF_FP32_COMP) {
    const float *x = (const float *)d_state;
    k_dot_energy<float><<<grid_for(N3), 256, 0, st>>>(x, x + 2 * N3, d_out, (int)ctx->N, m2, inv, H);
  } else {
    k_dot_energy<double><<<grid_for(N3), 256, 0, st>>>((const double *)d_state, nullptr, d_out, (int)ctx->N, m2,
                                                       inv, H);
  }
  CF_LAUNCHED(ctx);
  return CF_OK;
}

// Mean over a of an N^3 field, per (b, c): out[i] = sum_a f[i + a N^2] / N (coalesced in i).
__global__ void k_axis_mean(const double *__restrict__ f, double *__restrict__ out, long long NN, int N) {
  const long long stride = (long long)gridDim.x * blockDim.x;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < NN; i += stride) {
    double acc = 0.0;
    for (int a = 0; a < N; ++a) acc += f[i + (long long)a * NN];
    out[i] = acc / (double)N;
  }
}

// Whether the mean over a is summed by the energy pass itself, each warp marching over all planes
// (the sum's order is fixed, so a column is one warp's), and no density is written: where its
// CTAs fill enough of the waves they make.  us, one march / the density and a pass over it: FP64 FRW N
// = 288 (41% of a wave) 180 / 165, 320 (45%) 194 / 203, 384 (65%) 240 / 317, 448 (88%) 297 / 488,
// 576 (73% of two) 761 / 1081; FP32 comoving 320 289 / 270, 336 (57%) 309 / 325, 384 356 / 427; FP32 sqrt 336
// 342 / 342.
static bool slices_in_one_march(const cf_ctx *ctx) {
  const long long n = (energy_tasks((int)ctx->N) + 7) / 8, slots = 148LL * mean_per_sm((int)ctx->N);
  const double filled = (double)n / (double)((n + slots - 1) / slots * slots);
  return filled >= (ctx->word == 8 ? 0.45 : 0.56);
}

int density_slices(cf_ctx *ctx, const void *d_state, double t, double *d_slice, double *d_avg, cudaStream_t st) {
  EnergyOut o;
  o.slice = d_slice;
  o.mean = d_avg;
  if (!d_slice && !d_avg) return CF_OK;
  const bool march = !d_avg || slices_in_one_march(ctx);
  const int scratch = march ? CF_OK : ensure_spectrum_scratch(ctx, 0);
  // without room for the density the march, which needs none, serves every lattice
  if (march || scratch == CF_ERR_NOMEM) return energy_density_b(ctx, d_state, t, o, st);
  CF_TRY(scratch);
  const long long NN = ctx->N * ctx->N;
  CF_TRY(energy_density(ctx, d_state, t, ctx->spec_field, st));
  if (d_slice)
    CF_TRY_CUDA(cudaMemcpyAsync(d_slice, ctx->spec_field, NN * sizeof(double), cudaMemcpyDeviceToDevice, st));
  ProfScope ps(ctx, CF_PROF_SPECTRUM, st);
  k_axis_mean<<<grid_for(NN), 256, 0, st>>>(ctx->spec_field, d_avg, NN, (int)ctx->N);
  CF_LAUNCHED(ctx);
  return CF_OK;
}

// The fixed-point scale comes from the energy pass: by Parseval the weighted HC
// values of rho sum to N^3 sum_x rho^2, so no bin can exceed that, and the binning needs no
// pass of its own to find a maximum.
int density_spectrum_s2(cf_ctx *ctx, const void *d_state, double t, double *d_out, cudaStream_t st) {
  CF_TRY(ensure_spectrum_scratch(ctx, 1));
  EnergyOut o;
  o.rho = ctx->spec_field;
  o.squares = true;
  CF_TRY(energy_density_b(ctx, d_state, t, o, st));
  CF_TRY_CUFFT(cufftSetStream(ctx->plan_d2z1, st));
  {
    ProfScope ps(ctx, CF_PROF_SPECTRUM, st);
    CF_TRY_CUFFT(cufftExecD2Z(ctx->plan_d2z1, (cufftDoubleReal *)ctx->spec_field, (cufftDoubleComplex *)ctx->spec_hc));
  }
  return bin_spectrum(ctx, false, 1.0, d_out, st, ctx->N3);
}

int s2_to_shells(cf_ctx *ctx, double *d_shells, int64_t *d_counts, cudaStream_t st) {
  CF_TRY(ensure_spectrum_scratch(ctx, 0));
  k_shells<<<(unsigned)((ctx->shells + 7) / 8), 256, 0, st>>>(ctx->bins, ctx->maxbits, ctx->spec_mult,
                                                       (const long long *)ctx->s2_counts, d_shells,
                                                       (long long *)d_counts, ctx->s2_bins, ctx->shells);
  CF_LAUNCHED(ctx);
  return CF_OK;
}

int s2_counts(cf_ctx *ctx, int64_t *d_counts, cudaStream_t st) {
  CF_TRY(ensure_spectrum_scratch(ctx, 0));
  CF_TRY_CUDA(cudaMemcpyAsync(d_counts, ctx->s2_counts, (size_t)ctx->s2_bins * sizeof(int64_t),
                              cudaMemcpyDeviceToDevice, st));
  return CF_OK;
}

int state_export(cf_ctx *ctx, double *d_xy, const void *d_state, cudaStream_t st) {
  const long long n2 = 2 * ctx->N3;
  if (ctx->p.precision == CF_FP64) {
    CF_TRY_CUDA(cudaMemcpyAsync(d_xy, d_state, n2 * sizeof(double), cudaMemcpyDeviceToDevice, st));
    return CF_OK;
  }
  k_export_f32<<<grid_for(n2), 256, 0, st>>>((const float *)d_state, d_xy, n2);
  CF_LAUNCHED(ctx);
  return CF_OK;
}

int state_import(cf_ctx *ctx, void *d_state, const double *d_xy, cudaStream_t st) {
  const long long n2 = 2 * ctx->N3;
  if (ctx->p.precision == CF_FP64) {
    CF_TRY_CUDA(cudaMemcpyAsync(d_state, d_xy, n2 * sizeof(double), cudaMemcpyDeviceToDevice, st));
    return CF_OK;
  }
  k_import_f32<<<grid_for(n2), 256, 0, st>>>(d_xy, (float *)d_state, n2);
  CF_LAUNCHED(ctx);
  return CF_OK;
}

// ---- host <-> device state transfer of the FP32_COMP layout ------------------
// The FP64 [phi | pi] host array goes through two device chunks of the context
// (allocated once, kStageChunk doubles each) in turn: a chunk's copy and its
// conversion are ordered on the caller's stream, and chunk i + 2 reuses chunk i's
// buffer after its conversion.  An event recorded after the last chunk orders the
// next transfer, on whatever stream it runs, behind this one.
__global__ void k_import_f32_part(const double *__restrict__ in, float *__restrict__ s, long long n2, long long off,
                                  long long len) {
  const long long stride = (long long)gridDim.x * blockDim.x;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < len; i += stride) {
    const double v = in[i];
    const float h = (float)v;
    s[off + i] = h;
    s[n2 + off + i] = (float)(v - (double)h);
  }
}

__global__ void k_export_f32_part(const float *__restrict__ s, double *__restrict__ out, long long n2, long long off,
                                  long long len) {
  const long long stride = (long long)gridDim.x * blockDim.x;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < len; i += stride)
    out[i] = (double)s[off + i] + (double)s[n2 + off + i];
}

static constexpr long long kStageChunk = 16LL << 20;  // doubles per chunk (128 MB)

static int stage_begin(cf_ctx *ctx, cudaStream_t st) {
  if (!ctx->stage) {
    if (cudaMalloc(&ctx->stage, 2 * kStageChunk * sizeof(double)) != cudaSuccess) {
      ctx->stage = nullptr;
      set_error("cudaMalloc state staging chunks failed");
      return CF_ERR_NOMEM;
    }
    CF_TRY_CUDA(cudaEventCreateWithFlags(&ctx->stage_ev, cudaEventDisableTiming));
  }
  if (ctx->stage_used) CF_TRY_CUDA(cudaStreamWaitEvent(st, ctx->stage_ev, 0));
  return CF_OK;
}

static int stage_end(cf_ctx *ctx, cudaStream_t st) {
  CF_TRY_CUDA(cudaEventRecord(ctx->stage_ev, st));
  ctx->stage_used = true;
  return CF_OK;
}

int state_upload_host(cf_ctx *ctx, void *d_state, const double *h_xy, cudaStream_t st) {
  CF_TRY(stage_begin(ctx, st));
  const long long n2 = 2 * ctx->N3;
  for (long long off = 0, i = 0; off < n2; off += kStageChunk, ++i) {
    const long long len = std::min(kStageChunk, n2 - off);
    double *buf = ctx->stage + (i & 1) * kStageChunk;
    CF_TRY_CUDA(cudaMemcpyAsync(buf, h_xy + off, len * sizeof(double), cudaMemcpyHostToDevice, st));
    k_import_f32_part<<<grid_for(len), 256, 0, st>>>(buf, (float *)d_state, n2, off, len);
    CF_LAUNCHED(ctx);
  }
  return stage_end(ctx, st);
}

int state_download_host(cf_ctx *ctx, double *h_xy, const void *d_state, cudaStream_t st) {
  CF_TRY(stage_begin(ctx, st));
  const long long n2 = 2 * ctx->N3;
  for (long long off = 0, i = 0; off < n2; off += kStageChunk, ++i) {
    const long long len = std::min(kStageChunk, n2 - off);
    double *buf = ctx->stage + (i & 1) * kStageChunk;
    k_export_f32_part<<<grid_for(len), 256, 0, st>>>((const float *)d_state, buf, n2, off, len);
    CF_LAUNCHED(ctx);
    CF_TRY_CUDA(cudaMemcpyAsync(h_xy + off, buf, len * sizeof(double), cudaMemcpyDeviceToHost, st));
  }
  return stage_end(ctx, st);
}

int check_finite(cf_ctx *ctx, const void *d_state, int64_t *h_bad, cudaStream_t st) {
  unsigned long long *d_bad = nullptr;
  if (cudaMallocAsync((void **)&d_bad, sizeof(unsigned long long), st) != cudaSuccess) {
    set_error("cudaMallocAsync failed");
    return CF_ERR_NOMEM;
  }
  CF_TRY_CUDA(cudaMemsetAsync(d_bad, 0, sizeof(unsigned long long), st));
  const bool f32 = ctx->p.precision == CF_FP32_COMP;
  const long long n = (f32 ? 4 : 2) * ctx->N3;
  k_count_nonfinite<<<grid_for(n), 256, 0, st>>>(d_state, n, f32 ? 1 : 0, d_bad);
  CF_LAUNCHED(ctx);
  unsigned long long h = 0;
  CF_TRY_CUDA(cudaMemcpyAsync(&h, d_bad, sizeof(h), cudaMemcpyDeviceToHost, st));
  CF_TRY_CUDA(cudaFreeAsync(d_bad, st));
  CF_TRY_CUDA(cudaStreamSynchronize(st));
  if (h_bad) *h_bad = (int64_t)h;
  if (h) {
    set_error("state holds %llu non-finite values", h);
    return CF_ERR_NONFINITE;
  }
  return CF_OK;
}

}  // namespace cfb

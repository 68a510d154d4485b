// cf_fft3.cuh -- FP64 1-D transform passes of the 3-D real transforms, with what comes
// before and after them in the same pass.
//
// A 3-D transform of a half-complex array is three passes over HBM (along a, b and c); what
// a cuFFT call has around it -- the transfer factors before a C2R, the exponential
// after it, the conversion of a state before an R2C -- is then another read and write of the
// whole array each.  These kernels do one dimension each and take those steps along.
//
// Each line of length N = R1 R2 R3 is a Stockham transform (self-sorting radix passes:
// butterfly i of a pass with stride s reads x[i + j N/R], j < R, and writes b_k w_n^{pk} to
// y[q + s (R p + k)], i = q + s p, n = N/s), radix 3, 4, 6 or 8 butterflies in registers, the
// first reading and the last writing global memory, the others through two buffers of
// shared memory in turn.  Twiddles come from a table of e^{2 pi i j / N} (j < N, formed in
// long double), so each carries one rounding.  The kernels form inverse (e^{+}) sums; a forward
// sum is the same with real and imaginary parts exchanged on the way in and out.
#pragma once

#include <cuda_runtime.h>

#include <type_traits>

namespace cfb {

using C64 = double2;
__device__ __forceinline__ C64 z_add(C64 a, C64 b) { return C64{a.x + b.x, a.y + b.y}; }
__device__ __forceinline__ C64 z_sub(C64 a, C64 b) { return C64{a.x - b.x, a.y - b.y}; }
__device__ __forceinline__ C64 z_mul(C64 a, C64 b) { return C64{a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x}; }
__device__ __forceinline__ C64 z_i(C64 a) { return C64{-a.y, a.x}; }  // i a

// v_k = sum_j v_j e^{2 pi i j k / R}, natural order
__device__ __forceinline__ void bfly(C64 (&v)[3]) {
  constexpr double h = 0.86602540378443864676;  // sqrt(3)/2
  const C64 t = z_add(v[1], v[2]), d = z_sub(v[1], v[2]);
  const C64 u{fma(-0.5, t.x, v[0].x), fma(-0.5, t.y, v[0].y)};
  v[0] = z_add(v[0], t);
  v[1] = C64{fma(-h, d.y, u.x), fma(h, d.x, u.y)};
  v[2] = C64{fma(h, d.y, u.x), fma(-h, d.x, u.y)};
}
__device__ __forceinline__ void bfly(C64 (&v)[4]) {
  const C64 a = z_add(v[0], v[2]), b = z_sub(v[0], v[2]), c = z_add(v[1], v[3]), d = z_i(z_sub(v[1], v[3]));
  v[0] = z_add(a, c);
  v[1] = z_add(b, d);
  v[2] = z_sub(a, c);
  v[3] = z_sub(b, d);
}
__device__ __forceinline__ void bfly(C64 (&v)[6]) {
  constexpr double h = 0.86602540378443864676;
  C64 e[3] = {v[0], v[2], v[4]}, o[3] = {v[1], v[3], v[5]};
  bfly(e);
  bfly(o);
  o[1] = C64{0.5 * o[1].x - h * o[1].y, h * o[1].x + 0.5 * o[1].y};   // e^{i pi / 3}
  o[2] = C64{-0.5 * o[2].x - h * o[2].y, h * o[2].x - 0.5 * o[2].y};  // e^{2 i pi / 3}
#pragma unroll
  for (int k = 0; k < 3; ++k) v[k] = z_add(e[k], o[k]), v[k + 3] = z_sub(e[k], o[k]);
}
__device__ __forceinline__ void bfly(C64 (&v)[8]) {
  constexpr double h = 0.70710678118654752440;
  C64 e[4] = {v[0], v[2], v[4], v[6]}, o[4] = {v[1], v[3], v[5], v[7]};
  bfly(e);
  bfly(o);
  o[1] = C64{h * (o[1].x - o[1].y), h * (o[1].x + o[1].y)};
  o[2] = z_i(o[2]);
  o[3] = C64{-h * (o[3].x + o[3].y), h * (o[3].x - o[3].y)};
#pragma unroll
  for (int k = 0; k < 4; ++k) v[k] = z_add(e[k], o[k]), v[k + 4] = z_sub(e[k], o[k]);
}

// Radices of the lengths the passes are built for (R3 = 1: two passes): the column lines N and
// the packed rows N/2 of the lattices N = 64 ... 512 of the form 2^k and 3 2^k (fft3_has); others take
// the transfer kernel, the cuFFT transform and the exponential.
template <int N>
struct FftRadix;
template <> struct FftRadix<32> { static constexpr int R1 = 8, R2 = 4, R3 = 1; };
template <> struct FftRadix<48> { static constexpr int R1 = 8, R2 = 6, R3 = 1; };
template <> struct FftRadix<64> { static constexpr int R1 = 8, R2 = 8, R3 = 1; };
template <> struct FftRadix<96> { static constexpr int R1 = 8, R2 = 4, R3 = 3; };
template <> struct FftRadix<128> { static constexpr int R1 = 8, R2 = 4, R3 = 4; };
template <> struct FftRadix<192> { static constexpr int R1 = 8, R2 = 8, R3 = 3; };
template <> struct FftRadix<256> { static constexpr int R1 = 8, R2 = 8, R3 = 4; };
template <> struct FftRadix<384> { static constexpr int R1 = 8, R2 = 8, R3 = 6; };
template <> struct FftRadix<512> { static constexpr int R1 = 8, R2 = 8, R3 = 8; };

// The twiddles of a pass at a thread's butterflies g, g + G, ...: when it has one, they do not
// change from tile to tile and stay in registers (REG); else each is loaded where it is used.
template <int N, int R, int s, bool REG>
struct Twiddles {
  C64 w[REG && s * R < N ? R - 1 : 1];
  const C64 *tw;
  __device__ __forceinline__ Twiddles(const C64 *t, int g) : tw(t) {
    if constexpr (REG && s * R < N) {
#pragma unroll
      for (int k = 1; k < R; ++k) w[k - 1] = __ldg(t + (g / s) * k * s);
    }
  }
  __device__ __forceinline__ C64 at(int p, int k) const {
    if constexpr (REG) return w[k - 1];
    else return __ldg(tw + p * k * s);
  }
};

// One radix pass at butterflies i = g, g + G, ... of a line: ld(j) the input x[j], st(j, v) the
// output y[j]; s the product of the radices before this one.
template <int N, int R, int s, bool REG, typename Ld, typename St>
__device__ __forceinline__ void radix_pass(const Twiddles<N, R, s, REG> &tw, int g, int G, Ld ld, St st) {
  constexpr int B = N / R;
  auto one = [&](int i) {
    const int p = i / s, q = i - p * s;
    C64 v[R];
#pragma unroll
    for (int j = 0; j < R; ++j) v[j] = ld(i + j * B);
    bfly(v);
#pragma unroll
    for (int k = 0; k < R; ++k) {
      C64 y = v[k];
      if (k > 0 && s * R < N) y = z_mul(y, tw.at(p, k));  // the last pass has p = 0
      st(q + s * (R * p + k), y);
    }
  };
  if constexpr (REG) {
    one(g);
  } else {
    for (int i = g; i < B; i += G) one(i);
  }
}

// Asynchronous 16-byte global -> shared copy; `in` false writes zeros and reads nothing.
__device__ __forceinline__ void z_copy(C64 *dst, const C64 *src, bool in) {
  const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(d), "l"(src), "r"(in ? 16 : 0) : "memory");
}

// ---- along a or b: L neighbouring lines per tile ---------------------------------
// The tile's lines are consecutive in memory, so each of the N rows of the tile is one
// contiguous piece of 16 L bytes; threads run over the lines first, so global pieces
// are whole sectors and the shared-memory accesses of a quarter warp are consecutive.
// The kernels are persistent (a grid of resident CTAs walks the tiles): the next tile's
// rows come in by cp.async while this one is transformed, and a thread that has one butterfly
// of a pass keeps its twiddles in registers.  What bounds the passes: shared-memory
// traffic and the latency of three dependent radix passes at 15 to 18 warps per SM.  N = 384 along b:
// 0.386 ms (0.28 at the copy rate; 0.474 with the twiddles loaded per tile, 0.48 - 0.53 with
// one tile per CTA; a cuFFT pass of the same traffic 0.458); tiles of 2 lines 0.565, of 8 the
// same with half the tiles in flight.
template <int N, int NF>
struct ColShape {  // NF outputs per tile
  static constexpr int L = N >= 192 ? 4 : 8;
  static constexpr int T = N * L / 8;  // one radix-8 butterfly a thread
  static constexpr int tile = N * L;
  static constexpr bool three = FftRadix<N>::R3 > 1;
  // the landing and the current tile, the first exchange buffer, and the second one (with one
  // output the current tile's buffer, free after the first pass)
  static constexpr int bufs = 3 + (three && NF > 1 ? 1 : 0);
  static constexpr size_t bytes = bufs * (size_t)tile * sizeof(C64);
};

// Tile: open(t) -> tile with src(j, l) (the address of entry j of line l), in(l) (whether line
// l exists), load(f, j, l, x) (what enters output f's transform for the entry read into *x, which
// the thread may overwrite for the next output) and store(f, j, l, v).
template <int N, int NF, typename Open>
__device__ __forceinline__ void fft_columns(C64 *sm, const C64 *__restrict__ tw, int ntiles, Open open) {
  using F = FftRadix<N>;
  using CS = ColShape<N, NF>;
  constexpr int L = CS::L, T = CS::T, G = T / L;
  const int l = threadIdx.x % L, g = threadIdx.x / L;
  constexpr int S2 = F::R1, S3 = F::R1 * F::R2;
  constexpr bool reg1 = N / F::R1 == G, reg2 = N / F::R2 == G;
  const Twiddles<N, F::R1, 1, reg1> t1(tw, g);
  const Twiddles<N, F::R2, S2, reg2> t2(tw, g);
  const Twiddles<N, F::R3, S3, false> t3(tw, g);  // the last pass takes none
  C64 *x0 = sm, *x1 = sm + CS::tile, *b0 = sm + 2 * CS::tile;
  auto issue = [&](int t, C64 *x) {
    if (t < ntiles) {
      const auto q = open(t);
      const bool in = q.in(l);
      for (int j = g; j < N; j += G) z_copy(x + j * L + l, q.src(j, in ? l : 0), in);
    }
    asm volatile("cp.async.commit_group;\n" ::: "memory");
  };
  issue(blockIdx.x, x0);
  for (int t = blockIdx.x; t < ntiles; t += gridDim.x) {
    const auto q = open(t);
    const bool in = q.in(l);
    __syncthreads();  // the last tile is done with x1 (and with b0)
    issue(t + gridDim.x, x1);
    asm volatile("cp.async.wait_group 1;\n" ::: "memory");
    __syncthreads();  // this tile's rows have landed
#pragma unroll
    for (int f = 0; f < NF; ++f) {
      C64 *b1 = NF > 1 ? sm + 3 * CS::tile : x0;
      auto first = [&](int j) { return q.load(f, j, l, x0 + j * L + l); };
      auto get0 = [&](int j) { return b0[j * L + l]; };
      auto out = [&](int j, C64 v) {
        if (in) q.store(f, j, l, v);
      };
      if (f) __syncthreads();  // the first output's last pass is done with the exchange buffers
      radix_pass<N, F::R1, 1, reg1>(t1, g, G, first, [&](int j, C64 v) { b0[j * L + l] = v; });
      __syncthreads();
      if constexpr (F::R3 == 1) {
        radix_pass<N, F::R2, S2, reg2>(t2, g, G, get0, out);
      } else {
        radix_pass<N, F::R2, S2, reg2>(t2, g, G, get0, [&](int j, C64 v) { b1[j * L + l] = v; });
        __syncthreads();
        radix_pass<N, F::R3, S3, false>(t3, g, G, [&](int j) { return b1[j * L + l]; }, out);
      }
    }
    C64 *x = x0;
    x0 = x1, x1 = x;
  }
}

// ---- along c: packed rows of M = N/2 complex -----------------------------------
// ROWS rows per tile, threads over a row's butterflies first.  Rows sit in shared memory with
// a pad after every 8 entries: the first pass writes a butterfly's R = 8 outputs next to each
// other, which without it would put a quarter warp on one bank.  Persistent, the next
// tile's rows coming in by cp.async, as above.
template <int M>
struct RowShape {
  static constexpr int ROWS = M >= 192 ? 4 : (M >= 96 ? 8 : 16);
  static constexpr int T = M * ROWS / 8;
  static constexpr int P = M + M / 8;             // a padded row
  static constexpr int tile = ROWS * (P > M + 1 ? P : M + 2);  // holds M + 1 entries a row too
  static constexpr size_t bytes = 3 * (size_t)tile * sizeof(C64);
};
__device__ __forceinline__ int row_pad(int j) { return j + (j >> 3); }

// Tile: open(t) -> tile with src() (its first entry), load(j, r, x) (entry j of row r of what
// is transformed, from the tile's entries x, rows of IN), store(j, r, v).
// tw: e^{2 pi i j / M}.
template <int M, int IN, typename Open>
__device__ __forceinline__ void fft_rows(C64 *sm, const C64 *__restrict__ tw, int ntiles, Open open) {
  using F = FftRadix<M>;
  using RS = RowShape<M>;
  constexpr int ROWS = RS::ROWS, P = RS::P, T = RS::T;
  static_assert(ROWS * IN <= RS::tile && ROWS * P <= RS::tile, "a tile's rows fit its buffer");
  C64 *x0 = sm, *x1 = sm + RS::tile, *b0 = sm + 2 * RS::tile;
  auto issue = [&](int t, C64 *x) {
    if (t < ntiles) {
      const C64 *s = open(t).src();
      for (int i = threadIdx.x; i < ROWS * IN; i += T) z_copy(x + i, s + i, true);
    }
    asm volatile("cp.async.commit_group;\n" ::: "memory");
  };
  // butterflies t = threadIdx.x, + T, ... of the tile: t / B its row, t % B the row's butterfly
  auto pass = [&](auto &w, auto radix, auto stride, auto in, auto out) {
    constexpr int R = decltype(radix)::value, s = decltype(stride)::value, B = M / R;
    constexpr bool reg = B * ROWS == T;
    auto one = [&](int t) {
      const int r = t / B, i = t - r * B;
      radix_pass<M, R, s, reg>(w, i, B, [&](int j) { return in(j, r); }, [&](int j, C64 v) { out(j, r, v); });
    };
    if constexpr (reg) {
      one(threadIdx.x);
    } else {
      for (int t = threadIdx.x; t < B * ROWS; t += T) one(t);
    }
  };
  constexpr int S2 = F::R1, S3 = F::R1 * F::R2;
  const Twiddles<M, F::R1, 1, M / F::R1 * ROWS == T> t1(tw, threadIdx.x % (M / F::R1));
  const Twiddles<M, F::R2, S2, M / F::R2 * ROWS == T> t2(tw, threadIdx.x % (M / F::R2));
  const Twiddles<M, F::R3, S3, M / F::R3 * ROWS == T> t3(tw, 0);
  using std::integral_constant;
  issue(blockIdx.x, x0);
  for (int t = blockIdx.x; t < ntiles; t += gridDim.x) {
    const auto q = open(t);
    __syncthreads();  // the last tile is done with x1 (and with b0)
    issue(t + gridDim.x, x1);
    asm volatile("cp.async.wait_group 1;\n" ::: "memory");
    __syncthreads();  // this tile's rows have landed
    auto get0 = [&](int j, int r) { return b0[r * P + row_pad(j)]; };
    auto out = [&](int j, int r, C64 v) { q.store(j, r, v); };
    pass(t1, integral_constant<int, F::R1>{}, integral_constant<int, 1>{}, [&](int j, int r) { return q.load(j, r, x0); },
         [&](int j, int r, C64 v) { b0[r * P + row_pad(j)] = v; });
    __syncthreads();
    if constexpr (F::R3 == 1) {
      pass(t2, integral_constant<int, F::R2>{}, integral_constant<int, S2>{}, get0, out);
    } else {
      pass(t2, integral_constant<int, F::R2>{}, integral_constant<int, S2>{}, get0,
           [&](int j, int r, C64 v) { x0[r * P + row_pad(j)] = v; });
      __syncthreads();
      pass(t3, integral_constant<int, F::R3>{}, integral_constant<int, S3>{},
           [&](int j, int r) { return x0[r * P + row_pad(j)]; }, out);
    }
    C64 *x = x0;
    x0 = x1, x1 = x;
  }
}

// CTAs of a persistent pass: as many as are resident, no more than there are tiles.
template <typename K>
inline cudaError_t fft_grid(K kern, int threads, size_t smem, int device, long long ntiles, int *grid) {
  if (smem > 48 * 1024) {
    const cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
  }
  int sms = 0, per = 0;
  cudaError_t e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
  if (e == cudaSuccess) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, kern, threads, smem);
  if (e != cudaSuccess) return e;
  const long long most = (long long)sms * (per > 0 ? per : 1);
  *grid = (int)(ntiles < most ? ntiles : most);
  return cudaSuccess;
}

// Lattices the passes are built for.
inline bool fft3_has(long long N) {
  return N == 64 || N == 96 || N == 128 || N == 192 || N == 256 || N == 384 || N == 512;
}

}  // namespace cfb

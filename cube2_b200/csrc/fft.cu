// Transforms of the PM3 meshes: density to potential (kick.f90:472-491).
#include <algorithm>

#include "common.cuh"

namespace cube {

// ---------------------------------------------------------------------------------------------
// The potential's transforms on 19 mesh sides of 64 to 1024 points (CUBE_FFT_SIDES), five passes over the mesh:
//   k_fft_rows      real rows along x to half spectra, [z][ky][kx], rows padded to whole 32-byte sectors;
//   k_fft_columns   along y;
//   k_fft_columns   along z, times the Green table (real), and back along z;
//   k_fft_columns   back along y;
//   k_ifft_rows     back along x, into the padded potential, ghost points included.
// Every pass is one read and one write of the spectrum and is bound by that: no pass does more than about 4
// operations a byte.  At 512^3 points (us): 226, 256, 425, 255, 221 against 313, 226, 439, 226, 344 + 34 for the ghost
// points with cuFFT's plane transforms; at 1024^3 (ms) 1.91, 2.38, 4.30, 2.38, 1.98 against 1.57, 2.21, 6.07, 2.21,
// 2.67 + 0.13; 64 meshes of 64^3: 166 against 255 us.  (Rows of a power of two were at 210 us and 1.78 ms before the
// passes of radix 5 and 3 came into the same source: 32 bytes of spills at 512 points.)  4 to 5 TB/s where a pass follows the rows; along z the
// 64-byte pieces of a column lie a plane apart and it is 2.6 to 3.2 TB/s.
// Sides with factors 3 and 5, where cuFFT transformed whole meshes around a separate Green multiply: the kick of a
// 120^3 box (240^3 points) 1090 -> 990 us, of the subtile meshes of a 128^3 box (80^3 points) 2724 -> 2605 us.
//
// All transforms are Stockham FFTs (Govindaraju et al., "High performance discrete Fourier transforms on
// graphics processors", SC 2008): a radix-8 pass, passes of radix 5 and 3, then radix 8 and a last one of
// radix 8, 4 or 2.  A thread holds eight points of one transform in registers, j + r N/8 before the first pass and again
// after the last (its butterflies in the passes of radix 5 and 3 are j + u N/8); in between they change
// hands through shared memory, in two buffers taken in turn, so that an exchange needs one barrier (a
// buffer is written again two exchanges later, and the barrier in between follows every read of it).
// Twiddles exp(-2 pi i k/N) are rounded from double precision.  Inverse transforms run as the
// forward transform of the complex conjugate.  Unnormalised.
constexpr int kXThreads = 128;
constexpr int spec_stride(int n) { return (n / 2 + 1 + 3) / 4 * 4; }  // row stride of the half spectrum

__device__ __forceinline__ float2 cmul(float2 a, float2 b) {
  return make_float2(fmaf(a.x, b.x, -a.y * b.y), fmaf(a.x, b.y, a.y * b.x));
}
__device__ __forceinline__ float2 cadd(float2 a, float2 b) { return make_float2(a.x + b.x, a.y + b.y); }
__device__ __forceinline__ float2 csub(float2 a, float2 b) { return make_float2(a.x - b.x, a.y - b.y); }
__device__ __forceinline__ float2 mul_mi(float2 a) { return make_float2(a.y, -a.x); }  // a * (-i)
__device__ __forceinline__ float2 conj2(float2 a) { return make_float2(a.x, -a.y); }

// 8-point DFT in place (decimation in frequency: radix-2 passes, outputs put back in order)
__device__ __forceinline__ void dft8(float2 v[8]) {
  constexpr float h = 0.70710678118654752f;  // sqrt(2) / 2
  float2 a[8];
#pragma unroll
  for (int k = 0; k < 4; k++) {
    a[k] = cadd(v[k], v[k + 4]);
    a[k + 4] = csub(v[k], v[k + 4]);
  }
  a[5] = make_float2(h * (a[5].x + a[5].y), h * (a[5].y - a[5].x));    // * exp(-i pi/4)
  a[6] = mul_mi(a[6]);                                                 // * exp(-i pi/2)
  a[7] = make_float2(h * (a[7].y - a[7].x), -h * (a[7].x + a[7].y));   // * exp(-3i pi/4)
  float2 b[8];
#pragma unroll
  for (int q = 0; q < 8; q += 4) {
    b[q] = cadd(a[q], a[q + 2]);
    b[q + 2] = csub(a[q], a[q + 2]);
    b[q + 1] = cadd(a[q + 1], a[q + 3]);
    b[q + 3] = mul_mi(csub(a[q + 1], a[q + 3]));
  }
  v[0] = cadd(b[0], b[1]);
  v[4] = csub(b[0], b[1]);
  v[2] = cadd(b[2], b[3]);
  v[6] = csub(b[2], b[3]);
  v[1] = cadd(b[4], b[5]);
  v[5] = csub(b[4], b[5]);
  v[3] = cadd(b[6], b[7]);
  v[7] = csub(b[6], b[7]);
}

__device__ __forceinline__ float2 mad2(float a, float2 x, float2 y) { return make_float2(fmaf(a, x.x, y.x), fmaf(a, x.y, y.y)); }
template <int R>
__device__ __forceinline__ void dft_odd(float2 *v) {
  if constexpr (R == 3) {
    const float2 t = cadd(v[1], v[2]), d = csub(v[1], v[2]), m = mad2(-0.5f, t, v[0]);
    const float2 s = mul_mi(make_float2(0.86602540378443865f * d.x, 0.86602540378443865f * d.y));  // sin(2 pi/3)
    v[0] = cadd(v[0], t);
    v[1] = cadd(m, s);
    v[2] = csub(m, s);
  } else {
    constexpr float c1 = 0.30901699437494745f, c2 = -0.80901699437494745f, s1 = 0.95105651629515353f,
                    s2 = 0.58778525229247314f;  // cosines and sines of 2 pi/5 and 4 pi/5
    const float2 t1 = cadd(v[1], v[4]), t2 = cadd(v[2], v[3]), d1 = csub(v[1], v[4]), d2 = csub(v[2], v[3]);
    const float2 a1 = mad2(c1, t1, mad2(c2, t2, v[0])), a2 = mad2(c2, t1, mad2(c1, t2, v[0]));
    const float2 b1 = mul_mi(mad2(s1, d1, make_float2(s2 * d2.x, s2 * d2.y))),
                 b2 = mul_mi(mad2(s2, d1, make_float2(-s1 * d2.x, -s1 * d2.y)));
    v[0] = cadd(v[0], cadd(t1, t2));
    v[1] = cadd(a1, b1);
    v[4] = csub(a1, b1);
    v[2] = cadd(a2, b2);
    v[3] = csub(a2, b2);
  }
}

// Place of point z of column c of a buffer of TX columns.  The rows are permuted so that the 16 accesses of a
// half warp hit all banks both where its rows are eight apart (the first pass's stores) and where
// they follow one another.  A buffer of one column (TX = 1): c is a multiple of the column's threads instead, which
// does the same for the columns that share a half warp.
template <int TX>
__device__ __forceinline__ int zpos(int z, int c) {
  constexpr int kMask = TX < 16 ? 16 / TX - 1 : 0;
  if constexpr (TX == 1) return z ^ ((z >> 3) & kMask) ^ c;
  else return (z ^ ((z >> 3) & kMask)) * TX + c;
}

template <bool WARP>
__device__ __forceinline__ void fft_sync() {
  if constexpr (WARP) __syncwarp();
  else __syncthreads();
}

// radix of the pass that follows passes of product Ns of an n-point transform (1: none)
__host__ __device__ constexpr int fft_radix(int n, int Ns) {
  const int rem = n / Ns;
  return Ns == 1 || (rem % 5 && rem % 3 && rem % 8 == 0) ? 8 : (rem % 5 == 0 ? 5 : (rem % 3 == 0 ? 3 : rem));
}

template <int C>
__device__ __forceinline__ void fft_put(float2 *p, const float2 *a, const float2 *b) {
  if constexpr (C == 2) *reinterpret_cast<float4 *>(p) = make_float4(a->x, a->y, b->x, b->y);
  else *p = *a;
}
template <int C>
__device__ __forceinline__ void fft_get(const float2 *p, float2 *a, float2 *b) {
  if constexpr (C == 2) {
    const float4 x = *reinterpret_cast<const float4 *>(p);
    *a = make_float2(x.x, x.y);
    *b = make_float2(x.z, x.w);
  } else {
    *a = *p;
  }
}

// The passes from product Ns on, on points in buf; v[q][r] = point j + r N/8 of column c + q after the last
template <int N, int TX, bool WARP, int Ns, int C>
__device__ __forceinline__ void fft_rest(float2 (&v)[C][8], float2 *&buf, float2 *&alt, const float2 *tw, int j, int c) {
  constexpr int R = fft_radix(N, Ns), Q = C - 1;
  auto swap = [&]() {
    float2 *t = buf;
    buf = alt;
    alt = t;
  };
  if constexpr (R == 3 || R == 5) {
    constexpr int kButterflies = N / R, U = (8 + R - 1) / R;
#pragma unroll
    for (int u = 0; u < U; u++) {
      const int b = j + u * (N / 8);
      if (u * R + R <= 8 || b < kButterflies) {
        float2 x[C][R];
        const int k = b % Ns, d = (b / Ns) * Ns * R + k;
#pragma unroll
        for (int r = 0; r < R; r++) fft_get<C>(buf + zpos<TX>(b + r * kButterflies, c), &x[0][r], &x[Q][r]);
#pragma unroll
        for (int r = 1; r < R; r++) {
          const float2 t = tw[(r - 1) * Ns + k];
#pragma unroll
          for (int q = 0; q < C; q++) x[q][r] = cmul(x[q][r], t);
        }
#pragma unroll
        for (int q = 0; q < C; q++) dft_odd<R>(x[q]);
#pragma unroll
        for (int r = 0; r < R; r++) fft_put<C>(alt + zpos<TX>(d + r * Ns, c), &x[0][r], &x[Q][r]);
      }
    }
    swap();
    fft_sync<WARP>();
    fft_rest<N, TX, WARP, Ns * R>(v, buf, alt, tw + (R - 1) * Ns, j, c);
  } else {
#pragma unroll
    for (int r = 0; r < 8; r++) fft_get<C>(buf + zpos<TX>(j + r * (N / 8), c), &v[0][r], &v[Q][r]);
    swap();
    if constexpr (R == 8) {
      const int k = j % Ns;
#pragma unroll
      for (int r = 1; r < 8; r++) {
        const float2 t = tw[(r - 1) * Ns + k];
#pragma unroll
        for (int q = 0; q < C; q++) v[q][r] = cmul(v[q][r], t);
      }
#pragma unroll
      for (int q = 0; q < C; q++) dft8(v[q]);
      if constexpr (Ns * 8 < N) {
        const int d = (j / Ns) * Ns * 8 + k;
#pragma unroll
        for (int r = 0; r < 8; r++) fft_put<C>(buf + zpos<TX>(d + r * Ns, c), &v[0][r], &v[Q][r]);
        fft_sync<WARP>();
        fft_rest<N, TX, WARP, Ns * 8>(v, buf, alt, tw + 7 * Ns, j, c);
      }
    } else if constexpr (R > 1) {
      // the last pass: butterfly j + u N/8 has points j + (u + r 8/R) N/8, all of this thread's
      constexpr int U = 8 / R;
      static_assert(R == 2 || R == 4, "a power of two");
#pragma unroll
      for (int u = 0; u < U; u++) {
#pragma unroll
        for (int r = 1; r < R; r++) {
          const float2 t = tw[(r - 1) * Ns + j + u * (N / 8)];
#pragma unroll
          for (int q = 0; q < C; q++) v[q][u + r * U] = cmul(v[q][u + r * U], t);
        }
#pragma unroll
        for (int q = 0; q < C; q++) {
          float2 *const x = v[q];
          if constexpr (R == 4) {
            const float2 a0 = cadd(x[u], x[u + 4]), a2 = csub(x[u], x[u + 4]), a1 = cadd(x[u + 2], x[u + 6]),
                         a3 = mul_mi(csub(x[u + 2], x[u + 6]));
            x[u] = cadd(a0, a1);
            x[u + 4] = csub(a0, a1);
            x[u + 2] = cadd(a2, a3);
            x[u + 6] = csub(a2, a3);
          } else {
            const float2 t = x[u + 4];
            x[u + 4] = csub(x[u], t);
            x[u] = cadd(x[u], t);
          }
        }
      }
    }
  }
}
// The N-point transforms of C (1 or 2) neighbouring columns from c on, v[q][r] = point j + r N/8 of column c + q before
// and after.  buf, alt: the exchange buffers, swapped by every exchange.  WARP: all threads of a column are in
// one warp.  tw: the twiddles in the order of use (fft_twiddles), those of a pass and radix index next
// to each other, so that lanes hit different banks.
template <int N, int TX, bool WARP, int C>
__device__ __forceinline__ void fft_regs(float2 (&v)[C][8], float2 *&buf, float2 *&alt, const float2 *tw, int j, int c) {
  static_assert(N % 8 == 0 && N > 8, "the first pass is of radix 8");
#pragma unroll
  for (int q = 0; q < C; q++) dft8(v[q]);
#pragma unroll
  for (int r = 0; r < 8; r++) fft_put<C>(buf + zpos<TX>(8 * j + r, c), &v[0][r], &v[C - 1][r]);
  fft_sync<WARP>();
  fft_rest<N, TX, WARP, 8>(v, buf, alt, tw, j, c);
}

__device__ __forceinline__ float2 fft_root(int k, int n) {  // exp(-2 pi i k/n)
  double sn, cs;
  sincospi(-2.0 * (double)k / (double)n, &sn, &cs);
  return make_float2((float)cs, (float)sn);
}
// the n - 8 twiddles of an n-point transform: pass by pass from the second on, radix index r by radix index
__device__ __forceinline__ void fft_twiddles(float2 *tw, int n) {
  for (int e = threadIdx.x; e < n - 8; e += blockDim.x) {
    int Ns = 8, q = e, R = fft_radix(n, 8);
    while (q >= (R - 1) * Ns) {
      q -= (R - 1) * Ns;
      Ns *= R;
      R = fft_radix(n, Ns);
    }
    tw[e] = fft_root((q / Ns + 1) * (q % Ns), R * Ns);
  }
}

// Rows of N real points as N/2 complex ones (two neighbours each), a row by N/16 threads; the half spectra of the even and
// the odd points are separated by their symmetry.  A block takes `per` groups of rows and loads the
// next one's points before it transforms the current one's.
template <int N>
struct RowFft {
  static constexpr int M = N / 2, kThr = M / 8, kRows = kXThreads / kThr;  // threads a row, rows a block
  static constexpr int kT = kRows * kThr;
  static constexpr int B = (M + 15) / 16 * 16;  // points of a row's buffer (zpos permutes 16 of them)
  static constexpr bool kWarp = 32 % kThr == 0;
  static constexpr size_t kSmem = sizeof(float2) * (2 * (size_t)kRows * B + 2 * M);
  static constexpr bool kWhole = N * N % kRows == 0;       // whole groups of rows
  static constexpr int kBlocks = (N & (N - 1)) ? 6 : 8;    // resident a multiprocessor (registers)
  static_assert(kBlocks * (kSmem + 1024) <= 227 * 1024, "shared memory of the resident blocks");
  static_assert(N % 16 == 0 && kThr <= kXThreads, "eight points a thread");
};
template <int N>
__global__ void __launch_bounds__(RowFft<N>::kT, RowFft<N>::kBlocks) k_fft_rows(const float *in, float2 *out, int nrows, int per) {
  using F = RowFft<N>;
  constexpr int M = F::M, S = spec_stride(N);
  __shared__ float2 b0[F::kRows * F::B], b1[F::kRows * F::B], tw[M], w[M];
  fft_twiddles(tw, M);
  for (int k = threadIdx.x; k < M; k += F::kT) w[k] = fft_root(k, N);
  __syncthreads();
  const int rr = threadIdx.x / F::kThr, j = threadIdx.x % F::kThr, f = rr * F::kThr & 15;
  float2 *buf = b0 + rr * F::B, *alt = b1 + rr * F::B;
  float2 nx[8];
  auto fetch = [&](int g) {
    const int q = F::kWhole ? g * F::kRows + rr : min(g * F::kRows + rr, nrows - 1);
    const float2 *row = reinterpret_cast<const float2 *>(in) + (int64_t)q * M;
#pragma unroll
    for (int r = 0; r < 8; r++) nx[r] = row[j + r * (M / 8)];
  };
  const int g0 = blockIdx.x * per, g1 = min(g0 + per, (nrows + F::kRows - 1) / F::kRows);
  fetch(g0);
  for (int g = g0; g < g1; g++) {
    const bool live = F::kWhole || g * F::kRows + rr < nrows;
    float2 w1[1][8];
    float2(&v)[8] = w1[0];
#pragma unroll
    for (int r = 0; r < 8; r++) v[r] = nx[r];
    if (g + 1 < g1) fetch(g + 1);
    fft_regs<M, 1, F::kWarp>(w1, buf, alt, tw, j, f);
#pragma unroll
    for (int r = 0; r < 8; r++) buf[zpos<1>(j + r * (M / 8), f)] = v[r];
    fft_sync<F::kWarp>();
    float2 *row = out + ((int64_t)g * F::kRows + rr) * S;
#pragma unroll
    for (int r = 0; r < 8; r++) {
      // X[k] = (Z[k] + Z*[M-k]) / 2 - i exp(-2 pi i k/N) (Z[k] - Z*[M-k]) / 2
      const int k = j + r * (M / 8);
      const float2 z = v[r], y = conj2(buf[zpos<1>(k ? M - k : 0, f)]);
      const float2 t = cmul(w[k], make_float2(0.5f * (z.x - y.x), 0.5f * (z.y - y.y)));
      if (live) row[k] = make_float2(fmaf(0.5f, z.x + y.x, t.y), fmaf(0.5f, z.y + y.y, -t.x));
    }
    if (j == 0 && live) row[M] = make_float2(v[0].x - v[0].y, 0.f);
    float2 *t = buf;
    buf = alt;
    alt = t;
  }
}

// and back: rows into an array of (N + 2 pad)^3 points a slot, each also where it and its ends are ghost points
template <int N>
__global__ void __launch_bounds__(RowFft<N>::kT, RowFft<N>::kBlocks) k_ifft_rows(const float2 *in, float *out, int pad, int nrows, int per) {
  using F = RowFft<N>;
  constexpr int M = F::M, S = spec_stride(N);
  __shared__ float2 b0[F::kRows * F::B], b1[F::kRows * F::B], tw[M], w[M];
  fft_twiddles(tw, M);
  for (int k = threadIdx.x; k < M; k += F::kT) w[k] = fft_root(k, N);
  __syncthreads();
  const int rr = threadIdx.x / F::kThr, j = threadIdx.x % F::kThr, f = rr * F::kThr & 15;
  float2 *buf = b0 + rr * F::B, *alt = b1 + rr * F::B;
  const int m = N + 2 * pad;
  float2 nx[8];
  float nyq = 0.f;
  auto fetch = [&](int g) {
    const float2 *row = in + (int64_t)(F::kWhole ? g * F::kRows + rr : min(g * F::kRows + rr, nrows - 1)) * S;
#pragma unroll
    for (int r = 0; r < 8; r++) nx[r] = row[j + r * (M / 8)];
    if (j == 0) nyq = row[M].x;
  };
  const int g0 = blockIdx.x * per, g1 = min(g0 + per, (nrows + F::kRows - 1) / F::kRows);
  fetch(g0);
  for (int g = g0; g < g1; g++) {
    const bool live = F::kWhole || g * F::kRows + rr < nrows;
    float2 w1[1][8];
    float2(&v)[8] = w1[0];
    const float last = nyq;
#pragma unroll
    for (int r = 0; r < 8; r++) v[r] = nx[r];
    if (j == 0) v[0].y = 0.f;  // real, as the last one is
    if (g + 1 < g1) fetch(g + 1);
#pragma unroll
    for (int r = 0; r < 8; r++) buf[zpos<1>(j + r * (M / 8), f)] = v[r];
    fft_sync<F::kWarp>();
#pragma unroll
    for (int r = 0; r < 8; r++) {
      // Z[k] = X[k] + X*[M-k] + i exp(2 pi i k/N) (X[k] - X*[M-k]), conjugated
      const int k = j + r * (M / 8);
      float2 y = buf[zpos<1>(k ? M - k : 0, f)];
      if (k == 0) y = make_float2(last, 0.f);
      y.y = -y.y;
      const float2 t = cmul(conj2(w[k]), csub(v[r], y)), s = cadd(v[r], y);
      v[r] = make_float2(s.x - t.y, -(s.y + t.x));
    }
    float2 *t = buf;
    buf = alt;
    alt = t;
    fft_regs<M, 1, F::kWarp>(w1, buf, alt, tw, j, f);
    const int64_t q = (int64_t)g * F::kRows + rr;
    const int y = (int)(q % N), z = (int)(q / N % N);
    float *slot = out + q / ((int64_t)N * N) * m * m * m;
    // copies of the row: in the interior, and past the other end of y and z (pad <= N / 2: one each at most)
    const int iy = y < pad ? N : (y >= N - pad ? -N : 0), iz = z < pad ? N : (z >= N - pad ? -N : 0);
    for (int e = 0; e < (live ? 4 : 0); e++) {
      if (((e & 1) && !iy) || ((e & 2) && !iz)) continue;
      const int yy = y + pad + (e & 1 ? iy : 0), zz = z + pad + (e & 2 ? iz : 0);
      float2 *o = reinterpret_cast<float2 *>(slot + ((int64_t)zz * m + yy) * m + pad);
#pragma unroll
      for (int r = 0; r < 8; r++) {
        const int k = j + r * (M / 8);
        const float2 x = conj2(v[r]);
        o[k] = x;
        if (r == 0 && 2 * k < pad) o[k + M] = x;
        if (r == 7 && 2 * k >= N - pad) o[k - M] = x;
      }
    }
  }
}

// Columns of the spectrum, groups of TX neighbours along kx, two of them a thread (16-byte accesses: with 8-byte ones
// the load/store unit was the bound).  kColZ: along z and back around the Green multiply; kColFwd, kColInv: along y.
// A block takes `per` groups one after the other and loads the next one's points before it transforms the
// current one's.  The column past the last one of a row (their number is odd) is transformed too, in the padding.
// sym: the Green table is even along y and z, and only its quarter is read.
enum { kColZ, kColFwd, kColInv };
template <int N>
struct ColFft {
  static constexpr int TX = N > 256 ? 8 : (N > 128 ? 16 : (N > 64 ? 32 : 64)), T = N * TX / 16;  // columns of at least 64 bytes
  static constexpr int kBlocks = 512 / T;                               // resident a multiprocessor
  static constexpr int kGroups = (N * spec_stride(N) + TX - 1) / TX;    // of a slot
  static constexpr size_t kSmem = sizeof(float2) * (2 * (size_t)N * TX + N);
};
template <int N, int MODE>
__global__ void __launch_bounds__(ColFft<N>::T, ColFft<N>::kBlocks)
    k_fft_columns(float2 *C, const float *G, float gscale, int sym, int ngroups, int per) {
  constexpr int H = N / 2 + 1, S = spec_stride(N), TX = ColFft<N>::TX;
  constexpr int64_t kPoint = MODE == kColZ ? (int64_t)N * S : S;  // stride along a column
  constexpr int64_t kRow = MODE == kColZ ? S : (int64_t)N * S;    // stride of the other axis
  extern __shared__ float4 zs4[];
  float2 *const zs = reinterpret_cast<float2 *>(zs4);
  float2 *buf = zs, *alt = zs + N * TX, *const tw = zs + 2 * N * TX;
  fft_twiddles(tw, N);
  __syncthreads();
  const int c = threadIdx.x % (TX / 2) * 2, j = threadIdx.x / (TX / 2);
  int a = 0, kx = 0;  // the columns: their place along the other axis, and the first along kx
  float4 *col = nullptr, nx[8];
  auto fetch = [&](int gr) {
    const int sl = gr / ColFft<N>::kGroups, q = (gr - sl * ColFft<N>::kGroups) * TX + c;
    a = q / S;
    kx = q - a * S;
    col = a < N && kx < H ? reinterpret_cast<float4 *>(C + (int64_t)sl * N * N * S + a * kRow + kx + j * kPoint) : nullptr;
#pragma unroll
    for (int r = 0; r < 8; r++) nx[r] = col ? col[r * (N / 16) * kPoint] : make_float4(0.f, 0.f, 0.f, 0.f);
  };
  const int g0 = blockIdx.x * per, g1 = min(g0 + per, ngroups);
  fetch(g0);
  for (int gr = g0; gr < g1; gr++) {
    float2 v[2][8];
    float gs[2][8];
    float4 *const out = col;
#pragma unroll
    for (int r = 0; r < 8; r++) {
      v[0][r] = make_float2(nx[r].x, MODE == kColInv ? -nx[r].y : nx[r].y);
      v[1][r] = make_float2(nx[r].z, MODE == kColInv ? -nx[r].w : nx[r].w);
    }
    if constexpr (MODE == kColZ) {
      const float *const g = G + (sym ? min(a, N - a) : a) * H + kx;
#pragma unroll
      for (int r = 0; r < 8; r++) {
        const int z = j + r * (N / 8);
        const int64_t at = (int64_t)(sym ? min(z, N - z) : z) * (N * H);
        gs[0][r] = col ? __ldg(g + at) : 0.f;
        gs[1][r] = col && kx + 1 < H ? __ldg(g + at + 1) : 0.f;
      }
    }
    if (gr + 1 < g1) fetch(gr + 1);
    fft_regs<N, TX, false>(v, buf, alt, tw, j, c);
    if constexpr (MODE == kColZ) {
#pragma unroll
      for (int q = 0; q < 2; q++)
#pragma unroll
        for (int r = 0; r < 8; r++) {  // conj(X) G
          const float f = gs[q][r] * gscale;
          v[q][r] = make_float2(v[q][r].x * f, -v[q][r].y * f);
        }
      fft_regs<N, TX, false>(v, buf, alt, tw, j, c);
    }
    if (out) {
#pragma unroll
      for (int r = 0; r < 8; r++)
        out[r * (N / 16) * kPoint] = MODE == kColFwd ? make_float4(v[0][r].x, v[0][r].y, v[1][r].x, v[1][r].y)
                                                     : make_float4(v[0][r].x, -v[0][r].y, v[1][r].x, -v[1][r].y);
    }
  }
}

// Mesh sides of the own transforms: multiples of 16 (eight points of a row's half transform a thread) with factors 2, 3
// and 5, those of the workloads, of the tests and between them.  It is a selection: the passes could be
// instantiated for 400, 432, 720, 800 and 864 points too, which are neither built nor measured.  cuFFT's
// three-dimensional transforms serve these and all other sides, those below 64 points among them.
#define CUBE_FFT_SIDES(X) \
  X(64) X(80) X(96) X(128) X(144) X(160) X(192) X(240) X(256) X(288) X(320) X(384) X(480) X(512) X(576) X(640) X(768) X(960) X(1024)
bool pm3_fft_ok(int n, int nslots) {
  switch (n) {
#define X(N) case N:
    CUBE_FFT_SIDES(X)
#undef X
    return (int64_t)n * n * nslots < (1 << 30);  // rows and groups are numbered in 32 bits
    default: return false;
  }
}
int64_t pm3_spec_elems(int n, int nslots) {
  return (int64_t)n * n * (pm3_fft_ok(n, nslots) ? spec_stride(n) : n / 2 + 1);
}

// Groups a block takes: up to 8, which share its twiddles, while that leaves four blocks for each place on the
// device.  (Resident blocks with equal shares were 4 % of the kick slower at 512^3: the binning runs beside these,
// and places differ in how much of it they have.)
static int fft_per(int groups, int places) { return std::max(1, std::min(8, groups / (4 * places))); }

template <int N, int MODE>
static void launch_columns(const PM3Args &a, float2 *spec, float gscale, cudaStream_t s) {
  using F = ColFft<N>;
  const int groups = F::kGroups * a.nslots, per = fft_per(groups, a.num_sms * F::kBlocks);
  set_smem_attr_once((const void *)k_fft_columns<N, MODE>, F::kSmem);
  k_fft_columns<N, MODE><<<(groups + per - 1) / per, F::T, F::kSmem, s>>>(spec, a.green, gscale, a.green_sym, groups, per);
}

template <int N>
static void launch_fft(const PM3Args &a, cudaStream_t s) {
  using F = RowFft<N>;
  float2 *const spec = reinterpret_cast<float2 *>(a.rhok);
  const float gscale = (float)((double)a.mass / ((double)N * N * N));
  const int rows = N * N * a.nslots, groups = (rows + F::kRows - 1) / F::kRows;
  const int per = fft_per(groups, F::kBlocks * a.num_sms), grid = (groups + per - 1) / per;
  k_fft_rows<N><<<grid, F::kT, 0, s>>>(a.rho, spec, rows, per);
  launch_columns<N, kColFwd>(a, spec, gscale, s);
  launch_columns<N, kColZ>(a, spec, gscale, s);
  launch_columns<N, kColInv>(a, spec, gscale, s);
  k_ifft_rows<N><<<grid, F::kT, 0, s>>>(spec, a.phi ? a.phi : a.rho, a.phi ? a.phi_pad : 0, rows, per);
}

int launch_pm3_fft(const PM3Args &a, cudaStream_t s) {
  switch (a.n) {
#define X(N) case N: launch_fft<N>(a, s); break;
    CUBE_FFT_SIDES(X)
#undef X
    default: return 0;
  }
  return 5;
}

}  // namespace cube

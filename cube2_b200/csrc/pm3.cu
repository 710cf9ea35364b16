// PM3 fine-mesh force (kick.f90:403-568, pm3_fft_cuda.cu:276-391).
//
// Pipeline per batch of meshes:
//   deposit  TSC weights of every particle of the job's coarse cells into the
//            mesh (kick.f90:420-468); one warp per coarse cell, float atomics
//            (the cost follows the particles, not the mesh, which matters for
//            clustered boxes where most mesh bricks are nearly empty);
//   R2C      along x, then y (k_fft_rows, k_fft_columns; cuFFT where the mesh side is not theirs);
//   k-space  the potential spectrum: rho(k) * G(k) * mass / n^3, in place, between the
//            transforms along z (kick.f90:472-491 and the 1/nwork^3 of kick.f90:552);
//   C2R      along y, then x;
//   force    the 4-point difference of potential_to_force (kick.f90:545-568)
//            on the periodic FFT mesh, four x points per thread, writing the
//            three force arrays and the max |F|^2 over the physical mesh
//            points (kick.f90:494) in the same pass;
//   gather   TSC gather of the force at each active particle and the kick
//            vp += dv * a_mid*dt/(6 pi) (kick.f90:497-540).
#include <cuda.h>
#include <cudaTypedefs.h>

#include <algorithm>
#include <cmath>

#include "common.cuh"

namespace cube {

struct PM3K {
  int n, nt, nte, ncb;
  int64_t n3, nk;  // mesh points, half-spectrum points per slot
  int rdep[3], ract[3];
  int wrap, shift;
  double scale;
  const MeshJob *jobs;
  int njobs;
  const int16_t *xp;
  const int32_t *rhoc;
  const int64_t *cell_base;
  float *rho;           // density, then potential [slot][n^3]
  cufftComplex *rhok;
  float *force;  // [slot][3][n^3]
  const float *green;
  int green_sym;
  float gscale;  // mass / n^3
  float kick;
  float *vp;
  float *out;
  int want_vmax;
  int fphys_lo, fphys_n;
  int nslots;
  int32_t *err;
  int32_t *brick_ctr;
};

// a + d into [0, n) for |d| < n
__device__ __forceinline__ int64_t wrap_near(int64_t a, int64_t n) { return a < 0 ? a + n : (a >= n ? a - n : a); }

// TSC weights in real(4) from a real(8) coordinate (kick.f90:439-445)
__device__ __forceinline__ int64_t tsc(double m, float w[3]) {
  const double f = floor(m);
  const float l3 = (float)(m - f);
  w[0] = __fmul_rn(1.0f - l3, 1.0f - l3) * 0.5f;
  w[2] = __fmul_rn(l3, l3) * 0.5f;
  w[1] = 1.0f - w[0] - w[2];
  return (int64_t)f;
}

// The same for the brick kernels, whose mesh has a whole number mc <= 16 of points per coarse cell: offset xp of
// a cell that lies d cells into the brick is the mesh coordinate d mc + (2u + 1) mc / 2^17 from the
// brick's first owned point.  Its floor and its fraction (17 bits) are exact in integers, so both are
// those of the real(8) coordinate.
__device__ __forceinline__ int tsc_brick(int d, int16_t xp, int mc, float w[3]) {
  const unsigned q = (2u * (uint16_t)xp + 1u) * (unsigned)mc;
  const float l3 = (float)(q & 0x1ffffu) * (1.0f / 131072.0f);
  w[0] = __fmul_rn(1.0f - l3, 1.0f - l3) * 0.5f;
  w[2] = __fmul_rn(l3, l3) * 0.5f;
  w[1] = 1.0f - w[0] - w[2];
  return d * mc + (int)(q >> 17);
}

// the same for CIC on cell-centred points: floor(x - 1/2) and its fraction
__device__ __forceinline__ int cic_brick(int d, int16_t xp, int mc, float &f) {
  const int q = (int)((2u * (uint16_t)xp + 1u) * (unsigned)mc) - 65536;
  f = (float)(q & 0x1ffff) * (1.0f / 131072.0f);
  return d * mc + (q >> 17);
}

__global__ void __launch_bounds__(kWarps * 32) k_deposit(PM3K p) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int64_t cells = (int64_t)p.rdep[0] * p.rdep[1] * p.rdep[2];
  const int64_t wid = (int64_t)blockIdx.x * kWarps + warp;
  if (wid >= cells * p.njobs) return;
  const int j = (int)(wid / cells);
  const int64_t r = wid - (int64_t)j * cells;
  const MeshJob J = p.jobs[j];
  const int ci = J.lo[0] + (int)(r % p.rdep[0]);
  const int cj = J.lo[1] + (int)((r / p.rdep[0]) % p.rdep[1]);
  const int ck = J.lo[2] + (int)(r / ((int64_t)p.rdep[0] * p.rdep[1]));
  const int64_t cidx = (((int64_t)J.t * p.nte + ck) * p.nte + cj) * p.nte + ci;
  const int np = p.rhoc[cidx];
  const int64_t base = p.cell_base[cidx];
  float *R = p.rho + (int64_t)J.slot * p.n3;
  const int64_t n = p.n;
  for (int l = lane; l < np; l += 32) {
    const int16_t *q = p.xp + 3 * (base + l);
    float wx[3], wy[3], wz[3];
    const int64_t ix = tsc(decode_pos(ci - p.ncb, q[0]) * p.scale - J.off[0], wx) + p.shift;
    const int64_t iy = tsc(decode_pos(cj - p.ncb, q[1]) * p.scale - J.off[1], wy) + p.shift;
    const int64_t iz = tsc(decode_pos(ck - p.ncb, q[2]) * p.scale - J.off[2], wz) + p.shift;
    // the three x points of a row are one vector reduction when they lie in a 16-byte
    // window, else a pair and a single (rows are 16-byte aligned when n % 4 == 0)
    const bool vec = (n % 4 == 0) && ix >= 1 && ix + 1 < n;
#pragma unroll
    for (int c = 0; c < 3; c++) {
      int64_t Z = iz + c - 1;
      if (p.wrap) Z = wrap_near(Z, n); else if (Z < 0 || Z >= n) continue;
#pragma unroll
      for (int b = 0; b < 3; b++) {
        int64_t Y = iy + b - 1;
        if (p.wrap) Y = wrap_near(Y, n); else if (Y < 0 || Y >= n) continue;
        float *row = R + (Z * n + Y) * n;
        const float w0 = (wx[0] * wy[b]) * wz[c], w1 = (wx[1] * wy[b]) * wz[c], w2 = (wx[2] * wy[b]) * wz[c];
        if (vec) {
          const int64_t x0 = ix - 1, o = x0 & 3, b4 = x0 - o;
          if (o == 0) {
            atomicAdd(reinterpret_cast<float4 *>(row + b4), make_float4(w0, w1, w2, 0.f));
          } else if (o == 1) {
            atomicAdd(reinterpret_cast<float4 *>(row + b4), make_float4(0.f, w0, w1, w2));
          } else if (o == 2) {
            atomicAdd(reinterpret_cast<float2 *>(row + b4 + 2), make_float2(w0, w1));
            atomicAdd(row + b4 + 4, w2);
          } else {
            atomicAdd(row + b4 + 3, w0);
            atomicAdd(reinterpret_cast<float2 *>(row + b4 + 4), make_float2(w1, w2));
          }
          continue;
        }
        const float wr[3] = {w0, w1, w2};
#pragma unroll
        for (int a = 0; a < 3; a++) {
          int64_t X = ix + a - 1;
          if (p.wrap) X = wrap_near(X, n); else if (X < 0 || X >= n) continue;
          atomicAdd(row + X, wr[a]);
        }
      }
    }
  }
}

// potential spectrum in place: rhok[slot] *= G(k) * mass / n^3
__global__ void k_kspace(PM3K p) {
  const int64_t total = p.nk * p.nslots;
  for (int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; e < total;
       e += (int64_t)gridDim.x * blockDim.x) {
    const int64_t k = e % p.nk;
    const float g = p.green[k] * p.gscale;
    const cufftComplex c = p.rhok[e];
    p.rhok[e] = make_float2(c.x * g, c.y * g);
  }
}

// weights of potential_to_force at offsets -2, -1, +1, +2 (parameters.f90:49-50, a = real(4) 4/3)
struct FDW {
  float m2, m1, p1, p2;
  __device__ __forceinline__ FDW() {
    const float a = 4.0f / 3.0f;
    m2 = (a - 1.0f) / 4.0f;
    m1 = -a / 2.0f;
    p1 = a / 2.0f;
    p2 = (1.0f - a) / 4.0f;
  }
  __device__ __forceinline__ float operator()(float fm2, float fm1, float fp1, float fp2) const {
    return fm2 * m2 + fm1 * m1 + fp1 * p1 + fp2 * p2;  // sum(phi(i_n) * weight), kick.f90:562-564
  }
};

__device__ __forceinline__ bool in_phys(const PM3K &p, int64_t x, int64_t y, int64_t z) {
  return x >= p.fphys_lo && x < p.fphys_lo + p.fphys_n && y >= p.fphys_lo && y < p.fphys_lo + p.fphys_n &&
         z >= p.fphys_lo && z < p.fphys_lo + p.fphys_n;
}

// Force from the potential on the periodic mesh (n % 4 == 0).  A block owns 32 float4 columns
// (128 x points) of kFzRows rows and marches through kFzChunk planes: each thread keeps the
// five planes z-2 .. z+2 of its own column in registers and loads one new float4 per plane;
// x neighbours come from the adjacent lanes (the edge lanes load theirs), y neighbours from a
// shared tile of the block's rows plus two halo rows on each side.  Each potential value is
// thus read about once from DRAM.  Stores go to the three force arrays (an interleaved
// (fx, fy, fz, 0) layout measured twice as slow in the gather); |F|^2 of the physical points is
// reduced into out[0].
constexpr int kFzRows = 8;
constexpr int kFzChunk = 32;

__device__ __forceinline__ float4 shfl_f4(float4 v, int delta, bool up) {
  float4 r;
  r.x = up ? __shfl_up_sync(0xffffffffu, v.x, delta) : __shfl_down_sync(0xffffffffu, v.x, delta);
  r.y = up ? __shfl_up_sync(0xffffffffu, v.y, delta) : __shfl_down_sync(0xffffffffu, v.y, delta);
  r.z = up ? __shfl_up_sync(0xffffffffu, v.z, delta) : __shfl_down_sync(0xffffffffu, v.z, delta);
  r.w = up ? __shfl_up_sync(0xffffffffu, v.w, delta) : __shfl_down_sync(0xffffffffu, v.w, delta);
  return r;
}

__global__ void __launch_bounds__(kFzRows * 32) k_force_zm(PM3K p) {
  __shared__ float4 tile[kFzRows + 4][32];
  const FDW w;
  const int lane = threadIdx.x & 31, wy = threadIdx.x >> 5;
  const int64_t n = p.n, n4 = p.n / 4;
  const int nzc = (p.n + kFzChunk - 1) / kFzChunk;
  const int64_t slot = blockIdx.z / nzc;
  const int64_t z0 = (int64_t)(blockIdx.z % nzc) * kFzChunk, z1 = min(z0 + kFzChunk, n);
  const int64_t x4 = (int64_t)blockIdx.x * 32 + lane, y0 = (int64_t)blockIdx.y * kFzRows, y = y0 + wy;
  const bool act = x4 < n4 && y < n;
  // idle lanes read a valid column; rows past n march the periodic image row, which the
  // rows below them read as their y neighbours
  const int64_t xs = min(x4, n4 - 1), ys = wrap_near(y, n);
  const float4 *phi = reinterpret_cast<const float4 *>(p.rho + slot * p.n3);
  auto at = [&](int64_t xx4, int64_t yy, int64_t zz) {
    return __ldg(phi + (wrap_near(zz, n) * n + wrap_near(yy, n)) * n4 + wrap_near(xx4, n4));
  };
  float4 cm2 = at(xs, ys, z0 - 2), cm1 = at(xs, ys, z0 - 1), c0 = at(xs, ys, z0), cp1 = at(xs, ys, z0 + 1);
  float4 *F = reinterpret_cast<float4 *>(p.force + slot * 3 * p.n3) + ys * n4 + xs;
  const int64_t plane4 = n * n4;
  float m = 0.f;
  for (int64_t z = z0; z < z1; z++) {
    const float4 cp2 = at(xs, ys, z + 2);
    tile[wy + 2][lane] = c0;
    if (wy < 4) {  // halo rows y0-2, y0-1 (warps 0, 1) and y0+kFzRows, y0+kFzRows+1 (warps 2, 3)
      const int64_t hy = wy < 2 ? y0 - 2 + wy : y0 + kFzRows + wy - 2;
      tile[wy < 2 ? wy : kFzRows + wy][lane] = at(xs, hy, z);
    }
    float4 l = shfl_f4(c0, 1, true), r = shfl_f4(c0, 1, false);
    if (lane == 0) l = at(xs - 1, ys, z);
    if (lane == 31 || x4 + 1 >= n4) r = at(xs + 1, ys, z);
    __syncthreads();
    const float4 ym2 = tile[wy][lane], ym1 = tile[wy + 1][lane], yp1 = tile[wy + 3][lane],
                 yp2 = tile[wy + 4][lane];
    const float4 fx = make_float4(w(l.z, l.w, c0.y, c0.z), w(l.w, c0.x, c0.z, c0.w), w(c0.x, c0.y, c0.w, r.x),
                                  w(c0.y, c0.z, r.x, r.y));
    const float4 fy = make_float4(w(ym2.x, ym1.x, yp1.x, yp2.x), w(ym2.y, ym1.y, yp1.y, yp2.y),
                                  w(ym2.z, ym1.z, yp1.z, yp2.z), w(ym2.w, ym1.w, yp1.w, yp2.w));
    const float4 fz = make_float4(w(cm2.x, cm1.x, cp1.x, cp2.x), w(cm2.y, cm1.y, cp1.y, cp2.y),
                                  w(cm2.z, cm1.z, cp1.z, cp2.z), w(cm2.w, cm1.w, cp1.w, cp2.w));
    if (act) {
      float4 *Fz = F + z * plane4;
      Fz[0] = fx;
      Fz[n * plane4] = fy;
      Fz[2 * n * plane4] = fz;
      const int64_t x = 4 * x4;
      if (in_phys(p, x, y, z)) m = fmaxf(m, fx.x * fx.x + fy.x * fy.x + fz.x * fz.x);
      if (in_phys(p, x + 1, y, z)) m = fmaxf(m, fx.y * fx.y + fy.y * fy.y + fz.y * fz.y);
      if (in_phys(p, x + 2, y, z)) m = fmaxf(m, fx.z * fx.z + fy.z * fy.z + fz.z * fz.z);
      if (in_phys(p, x + 3, y, z)) m = fmaxf(m, fx.w * fx.w + fy.w * fy.w + fz.w * fz.w);
    }
    __syncthreads();  // the next plane overwrites the tile
    cm2 = cm1;
    cm1 = c0;
    c0 = cp1;
    cp1 = cp2;
  }
  // one update of f2max per block
  __shared__ float mb[kFzRows];
  m = warp_max(m);
  if (lane == 0) mb[wy] = m;
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int w = 1; w < kFzRows; w++) m = fmaxf(m, mb[w]);
    atomic_max_nonneg(&p.out[0], m);
  }
}

// the same, one point per thread, for any n
__global__ void k_force(PM3K p) {
  const FDW w;
  const int64_t n = p.n;
  const int64_t total = p.n3 * p.nslots;
  float m = 0.f;
  for (int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; e < total;
       e += (int64_t)gridDim.x * blockDim.x) {
    const int64_t slot = e / p.n3, r = e - slot * p.n3;
    const int64_t x = r % n, y = (r / n) % n, z = r / (n * n);
    const float *phi = p.rho + slot * p.n3;
    auto at = [&](int64_t xx, int64_t yy, int64_t zz) {
      return __ldg(phi + (wrap_near(zz, n) * n + wrap_near(yy, n)) * n + wrap_near(xx, n));
    };
    const float fx = w(at(x - 2, y, z), at(x - 1, y, z), at(x + 1, y, z), at(x + 2, y, z));
    const float fy = w(at(x, y - 2, z), at(x, y - 1, z), at(x, y + 1, z), at(x, y + 2, z));
    const float fz = w(at(x, y, z - 2), at(x, y, z - 1), at(x, y, z + 1), at(x, y, z + 2));
    float *F = p.force + slot * 3 * p.n3 + r;
    F[0] = fx;
    F[p.n3] = fy;
    F[2 * p.n3] = fz;
    if (in_phys(p, x, y, z)) m = fmaxf(m, fx * fx + fy * fy + fz * fz);
  }
  m = warp_max(m);
  if ((threadIdx.x & 31) == 0) atomic_max_nonneg(&p.out[0], m);
}

__global__ void __launch_bounds__(kWarps * 32, 4) k_gather(PM3K p) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int64_t cells = (int64_t)p.ract[0] * p.ract[1] * p.ract[2];
  const int64_t wid = (int64_t)blockIdx.x * kWarps + warp;
  float vm0 = 0.f, vm1 = 0.f, vm2 = 0.f;
  if (wid < cells * p.njobs) {
    const int j = (int)(wid / cells);
    const int64_t r = wid - (int64_t)j * cells;
    const MeshJob J = p.jobs[j];
    const int ci = J.alo[0] + (int)(r % p.ract[0]);
    const int cj = J.alo[1] + (int)((r / p.ract[0]) % p.ract[1]);
    const int ck = J.alo[2] + (int)(r / ((int64_t)p.ract[0] * p.ract[1]));
    const int64_t cidx = (((int64_t)J.t * p.nte + ck) * p.nte + cj) * p.nte + ci;
    const int np = p.rhoc[cidx];
    const int64_t base = p.cell_base[cidx];
    const float *F = p.force + (int64_t)J.slot * 3 * p.n3;
    const int64_t n = p.n, n3 = p.n3;
    for (int l = lane; l < np; l += 32) {
      const int64_t ip = base + l;
      const int16_t *q = p.xp + 3 * ip;
      float wx[3], wy[3], wz[3];
      const int64_t ix = tsc(decode_pos(ci - p.ncb, q[0]) * p.scale - J.off[0], wx) + p.shift;
      const int64_t iy = tsc(decode_pos(cj - p.ncb, q[1]) * p.scale - J.off[1], wy) + p.shift;
      const int64_t iz = tsc(decode_pos(ck - p.ncb, q[2]) * p.scale - J.off[2], wz) + p.shift;
      float d0 = 0.f, d1 = 0.f, d2 = 0.f;
#pragma unroll
      for (int c = 0; c < 3; c++) {
        const int64_t Z = p.wrap ? wrap_near(iz + c - 1, n) : iz + c - 1;
#pragma unroll
        for (int b = 0; b < 3; b++) {
          const int64_t Y = p.wrap ? wrap_near(iy + b - 1, n) : iy + b - 1;
#pragma unroll
          for (int a = 0; a < 3; a++) {
            const int64_t X = p.wrap ? wrap_near(ix + a - 1, n) : ix + a - 1;
            const int64_t m = (Z * n + Y) * n + X;
            const float w = (wx[a] * wy[b]) * wz[c];
            d0 += F[m] * w;
            d1 += F[n3 + m] * w;
            d2 += F[2 * n3 + m] * w;
          }
        }
      }
      float *v = p.vp + 3 * ip;
      const float v0 = v[0] + d0 * p.kick, v1 = v[1] + d1 * p.kick, v2 = v[2] + d2 * p.kick;
      v[0] = v0;
      v[1] = v1;
      v[2] = v2;
      vm0 = fmaxf(vm0, fabsf(v0));
      vm1 = fmaxf(vm1, fabsf(v1));
      vm2 = fmaxf(vm2, fabsf(v2));
    }
  }
  if (p.want_vmax) {
    // one update of each maximum per block: a warp per coarse cell would put hundreds of
    // thousands of atomics on the same three words
    __shared__ float vmb[3][kWarps];
    vm0 = warp_max(vm0);
    vm1 = warp_max(vm1);
    vm2 = warp_max(vm2);
    if (lane == 0) {
      vmb[0][warp] = vm0;
      vmb[1][warp] = vm1;
      vmb[2][warp] = vm2;
    }
    __syncthreads();
    if (threadIdx.x < 3) {
      float m = 0.f;
      for (int w = 0; w < kWarps; w++) m = fmaxf(m, vmb[threadIdx.x][w]);
      atomic_max_nonneg(&p.out[2 + threadIdx.x], m);
    }
  }
}

// ---------------------------------------------------------------------------------------------
// Brick kernels: a brick is kBrick^3 mesh points, i.e. (kBrick / mc)^3 coarse cells of one job, mc =
// mesh points per coarse cell (4, 8 or 16).  The bricks of a job tile its deposited or active
// cells; where those are no whole number of bricks, the last brick of an axis holds fewer cells.  A
// brick's particles lie in (kBrick / mc)^2 rows of (kBrick / mc) coarse cells, and every row is one
// contiguous run of storage, so a block walks them as one flat list.
constexpr int kBrick = 16;               // owned mesh points per brick side
constexpr int kMaxCb = 4;                // coarse cells per brick side (mc >= 4)
constexpr int kMaxRowsPerBrick = kMaxCb * kMaxCb;

// brick b of the launch -> job, first coarse cell, coarse cells a side (fewer than a brick's at the end of
// a range that is no whole number of bricks), first owned mesh point (exact: the jobs' offsets are
// whole mesh points, and on buffered meshes the index is in range without wrapping)
struct BrickPos {
  int j, ci0, cj0, ck0;
  int n[3];
  int64_t X0, Y0, Z0;
};
__host__ __device__ __forceinline__ int bricks_of(int ext, int cb) { return (ext + cb - 1) / cb; }
__device__ __forceinline__ BrickPos brick_pos(const PM3K &p, int64_t b, int cb, const int *ext, const int *lo_of) {
  const int nbx = bricks_of(ext[0], cb), nby = bricks_of(ext[1], cb), nbz = bricks_of(ext[2], cb);
  const int64_t per_job = (int64_t)nbx * nby * nbz;
  BrickPos q;
  q.j = (int)(b / per_job);
  const int64_t r = b - (int64_t)q.j * per_job;
  const MeshJob &J = p.jobs[q.j];
  const int lo[3] = {lo_of == nullptr ? J.alo[0] : J.lo[0], lo_of == nullptr ? J.alo[1] : J.lo[1],
                     lo_of == nullptr ? J.alo[2] : J.lo[2]};
  const int i[3] = {(int)(r % nbx) * cb, (int)((r / nbx) % nby) * cb, (int)(r / ((int64_t)nbx * nby)) * cb};
  for (int d = 0; d < 3; d++) q.n[d] = min(cb, ext[d] - i[d]);
  q.ci0 = lo[0] + i[0];
  q.cj0 = lo[1] + i[1];
  q.ck0 = lo[2] + i[2];
  const int64_t n = p.n;
  q.X0 = wrapi(llrint((double)(q.ci0 - p.ncb) * p.scale - J.off[0]) + p.shift, n);
  q.Y0 = wrapi(llrint((double)(q.cj0 - p.ncb) * p.scale - J.off[1]) + p.shift, n);
  q.Z0 = wrapi(llrint((double)(q.ck0 - p.ncb) * p.scale - J.off[2]) + p.shift, n);
  return q;
}

struct BrickRows {
  int nrows, total;
  int cx, cy;  // coarse cells of the brick along x and y
};

// The brick's rows of coarse cells: first particle, count and the coarse cells' first particles
// (relative to the row), in shared memory.  Contains two block barriers.
__device__ __forceinline__ void brick_rows(const PM3K &p, const MeshJob &J, const BrickPos &q, int64_t *rbase, int *rstart,
                                          int *rcell, BrickRows &br) {
  const int nrows = q.n[1] * q.n[2];
  for (int r = threadIdx.x; r < nrows; r += blockDim.x) {
    const int cj = q.cj0 + r % q.n[1], ck = q.ck0 + r / q.n[1];
    const int64_t c0 = (((int64_t)J.t * p.nte + ck) * p.nte + cj) * p.nte + q.ci0;
    int acc = 0;
    for (int i = 0; i < q.n[0]; i++) {
      rcell[r * (kMaxCb + 1) + i] = acc;
      acc += p.rhoc[c0 + i];
    }
    rbase[r] = p.cell_base[c0];
    rstart[r] = acc;  // count for now
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    int acc = 0;
    for (int r = 0; r < nrows; r++) {
      const int c = rstart[r];
      rstart[r] = acc;
      acc += c;
    }
    rstart[nrows] = acc;
  }
  __syncthreads();
  br.nrows = nrows;
  br.total = rstart[nrows];
  br.cx = q.n[0];
  br.cy = q.n[1];
}

// Flat particle index k of the brick -> (storage index, coarse cell offsets within the brick).
__device__ __forceinline__ int64_t brick_particle(int k, const BrickRows &br, const int64_t *rbase, const int *rstart,
                                                  const int *rcell, int &di, int &dj, int &dk) {
  int lo = 0, hi = br.nrows - 1;  // last row with rstart <= k
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (rstart[mid] <= k) lo = mid; else hi = mid - 1;
  }
  const int l = k - rstart[lo];
  int i = 0;
  while (i + 1 < br.cx && rcell[lo * (kMaxCb + 1) + i + 1] <= l) i++;
  di = i;
  dk = 0;  // lo = dk cy + dj, with at most kMaxCb rows a side
  while (lo - dk * br.cy >= br.cy) dk++;
  dj = lo - dk * br.cy;
  return rbase[lo] + l;
}

// Force and gather in one pass, persistent and warp-specialised: one 1024-thread block per SM
// claims bricks from a work counter.
//   scheduler (one warp): claims the next brick, writes its row table into a ring of kFgRing, and requests its
//     potential window as soon as the producers have read the last one: the brick plus three points
//     on every side (along x widened to whole 16-byte groups) by one 4-d tensor copy
//     (cp.async.bulk.tensor; a periodic potential has ghost points with the periodic images, so the box
//     never wraps; what lies past the array's end is filled with zeros and used by no owned point).
//   producers: the 4-point difference of potential_to_force (kick.f90:545-568) gives the
//     three force components on the brick and one point on every side, in one of two force
//     buffers, and max |F|^2 of the owned points (kick.f90:494).
//   consumers: every active particle of the brick gathers its 27 TSC points from the force
//     buffer and is kicked (kick.f90:497-540).  A thread's next particle, of this brick or the next, is
//     loaded (offset and velocity) before the current one is worked on.
// The buffers change hands through mbarriers, every wait bounded and decided by whole warps (the roles are whole
// warps): one that gives up leaves for the block's last barrier, the others' next waits run out and they follow.  The arithmetic (weights, products,
// summation order) is the one of k_force_zm followed by k_gather, and the force arrays never reach HBM.
//
// Before the scheduler and the prefetch (the producers claimed the bricks, the consumers met each brick's
// particles behind its barrier) the kernel issued on 26 % of the cycles at 14 stall cycles an issue for
// global loads: a brick has one particle or less per consumer, so each brick exposed the latency of its
// offsets and then of its velocities.  Now it is bound by shared memory (82 % of the wavefronts it could
// issue: the 81 values a particle reads and the windows' passes): 576 -> 419 us at 192^3 fine cells.
constexpr int kFgThreads = 1024;
constexpr int kFgProd = 384;                        // producer threads (the first warps of the block)
constexpr int kFgCons = kFgThreads - kFgProd - 32;  // consumer threads (the last warps; the scheduler lies between)
static_assert(kFgProd % 32 == 0 && kFgProd >= 128 && kFgCons >= 128, "whole warps in both groups");
constexpr int kPotX = kBrick + 8, kPotW = kBrick + 6;  // potential window: x 24, y and z 22
// force window: y, z the brick and one point on every side, x two (so that pairs of points are aligned)
constexpr int kForW = kBrick + 2, kForX = kBrick + 4;
constexpr int kPotElems = kPotW * kPotW * kPotX;
constexpr uint32_t kPotBytes = sizeof(float) * kPotElems;
constexpr int kForElems = kForW * kForW * kForX;
static_assert(kForElems % 2 == 0 && kPotElems % 4 == 0 && (kForElems + kForElems / 2) % 2 == 0, "16-byte aligned buffers");
constexpr int kFgMarch = kForW / 2;                        // planes a producer thread marches through
constexpr int kFgCols = 2 * kForW * (kForX / 2);           // producer threads with work
static_assert(kFgCols <= kFgProd && kFgMarch * 2 == kForW, "one pass of the producers per brick");
constexpr size_t kFgSmem = (size_t)kPotBytes + 2 * sizeof(float) * 3 * (size_t)kForElems + 128;  // + alignment slack
constexpr int kFgRing = 4;

struct BrickMeta {
  int total;  // particles of the brick; -1: no more bricks
  int n[3];   // coarse cells a side
  int64_t rbase[kMaxRowsPerBrick];
  int rstart[kMaxRowsPerBrick + 1];
  int rcell[kMaxRowsPerBrick * (kMaxCb + 1)];
};

// a consumer thread's particle: storage index (-1: none), cell offsets in the brick, offset, velocity
struct FgItem {
  int ip, cell;
  int16_t x[3];
  float v[3];
};
__device__ __forceinline__ FgItem fg_load(const PM3K &p, const BrickMeta &mt, int k) {
  FgItem it;
  it.ip = -1;
  if (k < mt.total) {
    BrickRows br;
    br.nrows = mt.n[1] * mt.n[2];
    br.total = mt.total;
    br.cx = mt.n[0];
    br.cy = mt.n[1];
    int di, dj, dk;
    it.ip = (int)brick_particle(k, br, mt.rbase, mt.rstart, mt.rcell, di, dj, dk);
    it.cell = di | dj << 8 | dk << 16;
    const int16_t *q = p.xp + 3 * (int64_t)it.ip;
    const float *v = p.vp + 3 * (int64_t)it.ip;
#pragma unroll
    for (int d = 0; d < 3; d++) {
      it.x[d] = q[d];
      it.v[d] = v[d];
    }
  }
  return it;
}

__global__ void __launch_bounds__(kFgThreads, 1) k_force_gather(PM3K p, int mc, int64_t nbricks, int pad,
                                                                const __grid_constant__ CUtensorMap tmap) {
  extern __shared__ __align__(128) float fg_smem[];
  // the tensor copies land on a 128-byte aligned shared address
  float *pot = fg_smem + ((128u - (smem_addr(fg_smem) & 127u)) & 127u) / 4;  // [z 22][y 22][x 24]
  float2 *fwb = reinterpret_cast<float2 *>(pot + kPotElems);  // [2]: (fx, fy) pairs [z 18][y 18][x 20], then fz
  // pot: window arrived; potfree: window read; full / empty: force buffers; meta / mfree: row tables of the ring
  __shared__ __align__(8) uint64_t bar_pot, bar_potfree, bar_full[2], bar_empty[2], bar_meta[kFgRing], bar_mfree[kFgRing];
  __shared__ BrickMeta meta[kFgRing];
  __shared__ float red[4][kFgThreads / 32];
  __shared__ int s_fail;
  const int tid = threadIdx.x, lane = tid & 31;
  if (blockIdx.x >= nbricks) return;
  if (tid == 0) {
    mbar_init(&bar_pot, 1);
    mbar_init(&bar_potfree, kFgProd / 32);
    for (int b = 0; b < 2; b++) {
      mbar_init(&bar_full[b], kFgProd / 32);
      mbar_init(&bar_empty[b], kFgCons / 32);
    }
    for (int b = 0; b < kFgRing; b++) {
      mbar_init(&bar_meta[b], 1);
      mbar_init(&bar_mfree[b], kFgCons / 32);
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    s_fail = 0;
  }
  __syncthreads();
  float m = 0.f, vm0 = 0.f, vm1 = 0.f, vm2 = 0.f;
  bool ok = true;
  if (tid < kFgProd) {
    const FDW w;
    for (int k = 0;; k++) {
      const int b = k & 1;
      const BrickMeta &mt = meta[k % kFgRing];
      ok = mbar_wait_bounded(&bar_meta[k % kFgRing], (uint32_t)(k / kFgRing) & 1u);
      if (!ok || mt.total < 0) break;
      const int ox = mt.n[0] * mc, oy = mt.n[1] * mc, oz = mt.n[2] * mc;  // owned points a side
      // the consumers are done with buffer b (brick k - 2), and this brick's window is there
      ok = (k < 2 || mbar_wait_bounded(&bar_empty[b], (uint32_t)((k - 2) >> 1) & 1u)) &&
           mbar_wait_bounded(&bar_pot, (uint32_t)k & 1u);
      if (!ok) break;
      float2 *fxy = fwb + b * (kForElems + kForElems / 2);
      float *fz = reinterpret_cast<float *>(fxy + kForElems);
      // Thread (x pair, y, half of the planes) marches along z: the five planes of its two points stay in
      // registers, x and y neighbours are 8-byte reads (7 per two points).
      if (tid < kFgCols) {
        const int x2 = tid % (kForX / 2), y = (tid / (kForX / 2)) % kForW, z0 = tid / (kForX / 2 * kForW) * kFgMarch;
        constexpr int PY = kPotX / 2, PZ = kPotX * kPotW / 2;  // strides of the window in pairs
        const float2 *c = reinterpret_cast<const float2 *>(pot) + (z0 + 2) * PZ + (y + 2) * PY + (x2 + 1);
        float2 zm2 = c[-2 * PZ], zm1 = c[-PZ], z0v = c[0], zp1 = c[PZ];
        // owned points (the x window starts two points before the brick's, y and z windows one)
        const bool own = y >= 1 && y <= oy && x2 >= 1 && 2 * x2 <= ox;
        int e = (z0 * kForW + y) * kForX + 2 * x2;
#pragma unroll
        for (int s = 0; s < kFgMarch; s++, c += PZ, e += kForW * kForX) {
          const float2 zp2 = c[2 * PZ], xl = c[-1], xr = c[1];
          const float2 f0 = make_float2(w(xl.x, xl.y, z0v.y, xr.x), w(xl.y, z0v.x, xr.x, xr.y));
          const float2 a2 = c[-2 * PY], a1 = c[-PY], b1 = c[PY], b2 = c[2 * PY];
          const float2 f1 = make_float2(w(a2.x, a1.x, b1.x, b2.x), w(a2.y, a1.y, b1.y, b2.y));
          const float2 f2 = make_float2(w(zm2.x, zm1.x, zp1.x, zp2.x), w(zm2.y, zm1.y, zp1.y, zp2.y));
          *reinterpret_cast<float4 *>(fxy + e) = make_float4(f0.x, f1.x, f0.y, f1.y);
          *reinterpret_cast<float2 *>(fz + e) = f2;
          const int z = z0 + s;
          if (own && z >= 1 && z <= oz)
            m = fmaxf(m, fmaxf(f0.x * f0.x + f1.x * f1.x + f2.x * f2.x, f0.y * f0.y + f1.y * f1.y + f2.y * f2.y));
          zm2 = zm1;
          zm1 = z0v;
          z0v = zp1;
          zp1 = zp2;
        }
      }
      __syncwarp();
      if (lane == 0) {
        mbar_arrive(&bar_potfree);
        mbar_arrive(&bar_full[b]);
      }
    }
  } else if (tid < kFgProd + 32) {
    const int cb = kBrick / mc;
    int issued = 0;
    for (int k = 0;; k++) {
      BrickMeta &mt = meta[k % kFgRing];
      // the ring slot is free (brick k - kFgRing consumed)
      ok = k < kFgRing || mbar_wait_bounded(&bar_mfree[k % kFgRing], (uint32_t)(k / kFgRing - 1) & 1u);
      if (!ok) break;
      int nid = 0;
      if (lane == 0) nid = k ? (int)gridDim.x + atomicAdd(p.brick_ctr, 1) : (int)blockIdx.x;
      const int64_t id = __shfl_sync(0xffffffffu, nid, 0);
      if (id >= nbricks) {
        if (lane == 0) {
          mt.total = -1;
          mbar_arrive(&bar_meta[k % kFgRing]);
        }
        break;
      }
      const BrickPos q = brick_pos(p, id, cb, p.ract, nullptr);
      const int nrows = q.n[1] * q.n[2];
      int cnt = 0;
      if (lane < nrows) {
        const int cj = q.cj0 + lane % q.n[1], ck = q.ck0 + lane / q.n[1];
        const int64_t c0 = (((int64_t)p.jobs[q.j].t * p.nte + ck) * p.nte + cj) * p.nte + q.ci0;
        for (int i = 0; i < q.n[0]; i++) {
          mt.rcell[lane * (kMaxCb + 1) + i] = cnt;
          cnt += p.rhoc[c0 + i];
        }
        mt.rbase[lane] = p.cell_base[c0];
      }
      int incl = cnt;
      for (int o = 1; o < 32; o <<= 1) {
        const int v = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += v;
      }
      if (lane <= nrows) mt.rstart[lane] = incl - cnt;  // nrows <= 16
      if (lane == nrows) {
        mt.total = incl;
        for (int d = 0; d < 3; d++) mt.n[d] = q.n[d];
      }
      __syncwarp();
      if (lane == 0) mbar_arrive(&bar_meta[k % kFgRing]);
      ok = k == 0 || mbar_wait_bounded(&bar_potfree, (uint32_t)(k - 1) & 1u);
      if (!ok) break;
      if (lane == 0) {
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        mbar_arrive_expect_tx(&bar_pot, kPotBytes);  // the phase completes when the bytes have landed
        const int cx = (int)q.X0 - 4 + pad, cy = (int)q.Y0 - 3 + pad, cz = (int)q.Z0 - 3 + pad;
        const int cs = p.jobs[q.j].slot;
        asm volatile(
            "cp.async.bulk.tensor.4d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4, "
            "%5}], [%6];" ::"r"(smem_addr(pot)),
            "l"(reinterpret_cast<uint64_t>(&tmap)), "r"(cx), "r"(cy), "r"(cz), "r"(cs), "r"(smem_addr(&bar_pot))
            : "memory");
      }
      issued++;
    }
    // a tensor copy still in flight (a wait gave up) lands before the block's memory is released
    if (issued) ok = mbar_wait_bounded(&bar_pot, (uint32_t)(issued - 1) & 1u) && ok;
  } else {
    const int gt = tid - kFgProd - 32;
    ok = mbar_wait_bounded(&bar_meta[0], 0u);
    FgItem cur;
    cur.ip = -1;
    if (ok) cur = fg_load(p, meta[0], gt);
    for (int k = 0; ok; k++) {
      const int b = k & 1, slot = k % kFgRing, next = (k + 1) % kFgRing;
      const BrickMeta &mt = meta[slot];
      const int total = mt.total;
      if (total < 0) break;
      const float2 *fxy = fwb + b * (kForElems + kForElems / 2);
      const float *fz = reinterpret_cast<const float *>(fxy + kForElems);
      ok = mbar_wait_bounded(&bar_full[b], (uint32_t)(k >> 1) & 1u);
      if (!ok) break;
      for (int k0 = gt - lane;; k0 += kFgCons) {  // the warp's first particle of this round
        const bool last = k0 + kFgCons >= total;
        FgItem nxt;
        if (last) {
          ok = mbar_wait_bounded(&bar_meta[next], (uint32_t)((k + 1) / kFgRing) & 1u);
          nxt.ip = -1;
          if (ok) nxt = fg_load(p, meta[next], gt);
        } else {
          nxt = fg_load(p, mt, k0 + lane + kFgCons);
        }
        if (cur.ip >= 0) {
          float wx[3], wy[3], wz[3];
          // the stencil's first point ix - 1 lies at force-window index (ix - X0) + 1 along x, iy - Y0 along y
          const int lx = tsc_brick(cur.cell & 0xff, cur.x[0], mc, wx) + 1,
                    ly = tsc_brick((cur.cell >> 8) & 0xff, cur.x[1], mc, wy),
                    lz = tsc_brick(cur.cell >> 16, cur.x[2], mc, wz);
          float d0 = 0.f, d1 = 0.f, d2 = 0.f;
#pragma unroll
          for (int c = 0; c < 3; c++) {
#pragma unroll
            for (int bb = 0; bb < 3; bb++) {
              const int row = ((lz + c) * kForW + (ly + bb)) * kForX + lx;
#pragma unroll
              for (int a = 0; a < 3; a++) {
                const float wt = (wx[a] * wy[bb]) * wz[c];
                const float2 f = fxy[row + a];
                d0 += f.x * wt;
                d1 += f.y * wt;
                d2 += fz[row + a] * wt;
              }
            }
          }
          float *v = p.vp + 3 * (int64_t)cur.ip;
          const float v0 = cur.v[0] + d0 * p.kick, v1 = cur.v[1] + d1 * p.kick, v2 = cur.v[2] + d2 * p.kick;
          v[0] = v0;
          v[1] = v1;
          v[2] = v2;
          vm0 = fmaxf(vm0, fabsf(v0));
          vm1 = fmaxf(vm1, fabsf(v1));
          vm2 = fmaxf(vm2, fabsf(v2));
        }
        cur = nxt;
        if (last) break;
      }
      __syncwarp();
      if (lane == 0) {
        mbar_arrive(&bar_empty[b]);
        mbar_arrive(&bar_mfree[slot]);
      }
    }
  }
  if (!ok) s_fail = 1;
  __syncthreads();
  if (tid == 0 && s_fail && p.err) atomicOr(p.err, 1 << CUBE_ERR_TIMEOUT);
  // one update of each maximum per block
  const int warp = tid >> 5;
  m = warp_max(m);
  vm0 = warp_max(vm0);
  vm1 = warp_max(vm1);
  vm2 = warp_max(vm2);
  if (lane == 0) {
    red[0][warp] = m;
    red[1][warp] = vm0;
    red[2][warp] = vm1;
    red[3][warp] = vm2;
  }
  __syncthreads();
  if (tid < 4) {
    float r = 0.f;
    for (int qq = 0; qq < kFgThreads / 32; qq++) r = fmaxf(r, red[tid][qq]);
    if (tid == 0) atomic_max_nonneg(&p.out[0], r);
    else if (p.want_vmax) atomic_max_nonneg(&p.out[1 + tid], r);
  }
}

static PM3K make_k(const PM3Args &a) {
  const Lay &L = *a.L;
  PM3K p;
  p.n = a.n;
  p.nt = L.nt;
  p.nte = L.nte;
  p.ncb = L.ncb;
  p.n3 = (int64_t)a.n * a.n * a.n;
  p.nk = (int64_t)a.n * a.n * (a.n / 2 + 1);
  for (int d = 0; d < 3; d++) {
    p.rdep[d] = a.rdep[d];
    p.ract[d] = a.ract[d];
  }
  p.wrap = a.wrap;
  p.shift = a.shift;
  p.scale = a.scale;
  p.jobs = a.jobs;
  p.njobs = a.njobs;
  p.xp = a.xp;
  p.rhoc = a.rhoc;
  p.cell_base = a.cell_base;
  p.rho = a.rho;
  p.rhok = a.rhok;
  p.force = a.force;
  p.green = a.green;
  p.green_sym = a.green_sym;
  p.gscale = (float)((double)a.mass / ((double)a.n * a.n * a.n));
  p.kick = a.kick;
  p.vp = a.vp;
  p.out = a.out;
  p.want_vmax = a.want_vmax;
  p.fphys_lo = a.fphys_lo;
  p.fphys_n = a.fphys_n;
  p.nslots = a.nslots;
  p.err = a.err;
  p.brick_ctr = a.brick_ctr;
  return p;
}


void launch_pm3_kspace(const PM3Args &a, cudaStream_t s) {
  PM3K p = make_k(a);
  k_kspace<<<148 * 8, 256, 0, s>>>(p);
}

void launch_pm3_force(const PM3Args &a, cudaStream_t s) {
  PM3K p = make_k(a);
  if (a.n % 4 == 0) {
    const int nzc = (a.n + kFzChunk - 1) / kFzChunk;
    const dim3 grid((unsigned)((a.n / 4 + 31) / 32), (unsigned)((a.n + kFzRows - 1) / kFzRows),
                    (unsigned)(nzc * a.nslots));
    k_force_zm<<<grid, kFzRows * 32, 0, s>>>(p);
  } else
    k_force<<<148 * 8, 256, 0, s>>>(p);
}

// Deposit brick by brick: the TSC weights of the brick's particles accumulate in a shared-memory
// window (the brick plus one point on every side, widened to whole 16-byte groups along x) with
// native 32-bit integer shared atomics on fixed-point weights, w * 2^e rounded to an integer; e
// is chosen per brick from its particle count so that no window point can overflow 2^32
// (a point takes at most 0.75^3 of each particle).  The window then goes to the mesh as floats,
// one 16-byte vector reduction per group of four points that received anything: every mesh point
// takes at most one global reduction per brick that reaches it, instead of one per particle.
// kick.f90:420-468 sums the same weights; the integer sums make the brick's part exact and
// independent of the order of the atomics.  An item has at most kDepChunk particles (unless its brick has 6e7), so
// TSC weights are rounded to 2^-22 or finer.  The learned shell's CIC density, up to 4096 particles a uniform brick,
// starts at the scale of its mean density instead, 2^-26 in a uniform box.  At 2^-20, from the number alone, ten times as
// many of the network's BF16 inputs differed from the exact density's as with sums in FP32.
constexpr int kDepThreads = 256;
constexpr int kDepBlocks = 5;  // resident blocks per SM (48 registers a thread)
constexpr int kAccX = kBrick + 8;  // x window owned - 4 .. owned + kBrick + 3: whole float4 groups
constexpr int kAccW = kBrick + 2;  // y, z window owned - 1 .. owned + kBrick

constexpr int kDepChunk = 2048;  // particles of one deposit work item (a crowded brick makes several)

// The deposit's work list: brick b's item (brick, chunk, chunks) at items[b], no chunks where it has no particles.  A
// brick of more than `chunk` particles makes ceil(particles / chunk) items, the others behind the nbricks first ones in
// any order, so a crowded brick is spread over several blocks whose windows add up in the mesh.  One thread
// per brick; *count counts the items behind.  They fit unless the cells hold more particles than the list was
// sized for (the counts or the particle number are wrong): then an error and no item where a status word is given,
// else one item.
__global__ void k_dep_items(PM3K p, int mc, int64_t nbricks, int chunk, int2 *items, int *count, int64_t cap) {
  const int cb = kBrick / mc;
  for (int64_t b = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; b < nbricks;
       b += (int64_t)gridDim.x * blockDim.x) {
    const BrickPos q = brick_pos(p, b, cb, p.rdep, p.rdep);
    const int64_t t = p.jobs[q.j].t;
    int total = 0;
    for (int k = 0; k < q.n[2]; k++)
      for (int j = 0; j < q.n[1]; j++) {
        const int32_t *r = p.rhoc + ((t * p.nte + q.ck0 + k) * p.nte + q.cj0 + j) * p.nte + q.ci0;
        for (int i = 0; i < q.n[0]; i++) total += r[i];
      }
    int nch = min((total + chunk - 1) / chunk, 0x7fff);
    if (nch > 1) {
      const int64_t at = nbricks + atomicAdd(count, nch - 1);
      if (at + nch - 1 > cap) {
        if (p.err) atomicOr(p.err, 1 << CUBE_ERR_CAPACITY);
        for (int64_t i = at; i < cap; i++) items[i] = make_int2(0, 0);
        nch = p.err ? 0 : 1;
      }
      for (int c = 1; c < nch; c++) items[at + c - 1] = make_int2((int)b, c | (nch << 16));
    }
    items[b] = make_int2((int)b, nch << 16);
  }
}

template <bool CIC>
__global__ void __launch_bounds__(kDepThreads, kDepBlocks) k_deposit_brick(PM3K p, int mc, int64_t nbricks, const int2 *items,
                                                                               const int *count) {
  __shared__ __align__(16) unsigned acc[kAccW * kAccW * kAccX];
  __shared__ int64_t rbase[kMaxRowsPerBrick];
  __shared__ int rstart[kMaxRowsPerBrick + 1];
  __shared__ int rcell[kMaxRowsPerBrick * (kMaxCb + 1)];
  __shared__ unsigned long long s_sum;
  if (CIC && threadIdx.x == 0) s_sum = 0;
  int2 item = make_int2((int)blockIdx.x, 1 << 16);  // without a work list: a whole brick
  if (items) {
    if (blockIdx.x >= nbricks && blockIdx.x - nbricks >= *count) return;
    item = items[blockIdx.x];
  }
  const int chunk = item.y & 0xffff, nch = item.y >> 16;
  if (nch == 0) return;
  const int cb = kBrick / mc;
  const BrickPos q = brick_pos(p, item.x, cb, p.rdep, p.rdep);
  const MeshJob &J = p.jobs[q.j];
  for (int e4 = threadIdx.x; e4 < kAccW * kAccW * kAccX / 4; e4 += kDepThreads)
    reinterpret_cast<uint4 *>(acc)[e4] = make_uint4(0u, 0u, 0u, 0u);
  BrickRows br;
  brick_rows(p, J, q, rbase, rstart, rcell, br);  // its barriers cover the zeroing
  // this item's particles of the brick
  const int k0 = (int)((int64_t)br.total * chunk / nch), k1 = (int)((int64_t)br.total * (chunk + 1) / nch);
  if (k1 <= k0) return;
  // Fixed-point scale 2^e: particles * (largest weight) * 2^e < 2^32.  For CIC a point may get 31 times the mean density
  // plus 31, and if one then gets more, the item is done again with a coarser scale: the sums are exact, so
  // those of the window tell (each point that has wrapped is 2^32 short)
  auto fits = [](double most, int e) { return most * (double)(1u << e) < 4294967040.0; };
  const double most = (double)(k1 - k0) * (CIC ? 1.0 : 0.421875);
  int e = CIC ? 28 : 24;
  if constexpr (CIC) {
    const double points = (double)(q.n[0] * q.n[1] * q.n[2]) * (mc * mc * mc);
    while (e > 1 && !fits(fmin(most, 31.0 * (1.0 + (double)br.total / points)), e)) e--;
  } else {
    while (e > 1 && !fits(most, e)) e--;
  }
  const auto deposit = [&](const float fs) {
    for (int k = k0 + threadIdx.x; k < k1; k += kDepThreads) {
      int di, dj, dk;
      const int64_t ip = brick_particle(k, br, rbase, rstart, rcell, di, dj, dk);
      const int16_t *qp = p.xp + 3 * ip;
      if constexpr (CIC) {  // points at cell centres: the first is floor(x - 1/2), from -1 of the brick on
        float fx, fy, fz;
        const int lx = cic_brick(di, qp[0], mc, fx) + 4, ly = cic_brick(dj, qp[1], mc, fy) + 1,
                  lz = cic_brick(dk, qp[2], mc, fz) + 1;
        const float sx[2] = {(1.0f - fx) * fs, fx * fs}, sy[2] = {1.0f - fy, fy}, sz[2] = {1.0f - fz, fz};
#pragma unroll
        for (int c = 0; c < 2; c++)
#pragma unroll
          for (int bb = 0; bb < 2; bb++) {
            unsigned *row = acc + ((lz + c) * kAccW + (ly + bb)) * kAccX + lx;
            atomicAdd(row + 0, __float2uint_rn(sx[0] * sy[bb] * sz[c]));
            atomicAdd(row + 1, __float2uint_rn(sx[1] * sy[bb] * sz[c]));
          }
        continue;
      }
      float wx[3], wy[3], wz[3];
      // window indices of the stencil's first point: x (ix - 1) - (X0 - 4), y (iy - 1) - (Y0 - 1)
      const int lx = tsc_brick(di, qp[0], mc, wx) + 3, ly = tsc_brick(dj, qp[1], mc, wy), lz = tsc_brick(dk, qp[2], mc, wz);
      const float sx0 = wx[0] * fs, sx1 = wx[1] * fs, sx2 = wx[2] * fs;
#pragma unroll
      for (int c = 0; c < 3; c++) {
#pragma unroll
        for (int bb = 0; bb < 3; bb++) {
          unsigned *row = acc + ((lz + c) * kAccW + (ly + bb)) * kAccX + lx;
          const float yz = wy[bb] * wz[c];
          atomicAdd(row + 0, __float2uint_rn(sx0 * yz));
          atomicAdd(row + 1, __float2uint_rn(sx1 * yz));
          atomicAdd(row + 2, __float2uint_rn(sx2 * yz));
        }
      }
    }
  };
  deposit((float)(1u << e));
  __syncthreads();
  if constexpr (CIC) {
    while (e > 1 && !fits(most, e)) {  // the same for the whole block
      unsigned long long sum = 0;
      for (int e4 = threadIdx.x; e4 < kAccW * kAccW * kAccX / 4; e4 += kDepThreads) {
        const uint4 u = reinterpret_cast<const uint4 *>(acc)[e4];
        sum += (unsigned long long)u.x + u.y + u.z + u.w;
      }
      for (int o = 16; o; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
      if ((threadIdx.x & 31) == 0) atomicAdd(&s_sum, sum);
      __syncthreads();
      if (((unsigned long long)(k1 - k0) << e) <= s_sum + 0x80000000ull) break;
      for (int e4 = threadIdx.x; e4 < kAccW * kAccW * kAccX / 4; e4 += kDepThreads)
        reinterpret_cast<uint4 *>(acc)[e4] = make_uint4(0u, 0u, 0u, 0u);
      __syncthreads();
      if (threadIdx.x == 0) s_sum = 0;  // added to again only behind the next barrier
      e = max(e - 2, 1);
      deposit((float)(1u << e));
      __syncthreads();
    }
  }
  const float inv = 1.0f / (float)(1u << e);
  // Flush: lane (w, xg) of a warp takes x group xg (lane % 6) of window rows 5 pass + w (w < 5), so
  // the group's mesh x index is worked out once and each row's once per pass.
  float *R = p.rho + (int64_t)J.slot * p.n3;
  constexpr int G4 = kAccX / 4, kRowsPerWarp = 32 / G4, kRows = kAccW * kAccW;
  const int lane = threadIdx.x & 31, w = lane / G4, xg = lane - w * G4;
  if (w < kRowsPerWarp) {
    // periodic meshes wrap; buffered ones drop what lies outside (-1), as kick.f90:448-466 does
    const int ni = p.n, wrapped = p.wrap ? ni : 0;
    auto place = [ni, wrapped](int a) {
      a += a < 0 ? wrapped : (a >= ni ? -wrapped : 0);
      return a >= ni ? -1 : a;
    };
    const int gx = place((int)q.X0 - 4 + 4 * xg);
    for (int row = (threadIdx.x >> 5) * kRowsPerWarp + w; row < kRows; row += (kDepThreads / 32) * kRowsPerWarp) {
      const uint4 u = reinterpret_cast<const uint4 *>(acc)[row * G4 + xg];
      if ((u.x | u.y | u.z | u.w) == 0u) continue;
      const int gy = place((int)q.Y0 - 1 + row % kAccW), gz = place((int)q.Z0 - 1 + row / kAccW);
      if ((gx | gy | gz) < 0) continue;
      atomicAdd(reinterpret_cast<float4 *>(R + ((int64_t)gz * ni + gy) * ni + gx),
                make_float4((float)u.x * inv, (float)u.y * inv, (float)u.z * inv, (float)u.w * inv));
    }
  }
}

// mesh points per coarse cell when the brick kernels apply (4, 8 or 16 exactly, on rows of whole 16-byte
// groups), else 0
int pm3_brick_mc(const PM3Args &a) {
  const int mc = (int)llrint(a.scale);
  if ((double)mc != a.scale || (mc != 4 && mc != 8 && mc != 16)) return 0;
  static_assert(kBrick / 4 <= kMaxCb && kBrick % 16 == 0, "whole coarse cells per brick");
  return a.n >= 16 && a.n % 4 == 0 && a.shift % 4 == 0 ? mc : 0;
}

// the dynamic shared-memory limit of a kernel, raised once per device (the attribute is per device).  Like the other
// tables of this kind (tensor_map_encoder, the attributes in mlp.cu) it relies on the lock that every entry point holds
void set_smem_attr_once(const void *fn, size_t bytes) {
  constexpr int kDev = 64, kFn = 96;
  static const void *fns[kFn] = {};
  static bool done[kFn][kDev] = {};
  int dev = 0;
  cudaGetDevice(&dev);
  int f = 0;
  while (f < kFn && fns[f] && fns[f] != fn) f++;
  if (f == kFn) {
    cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
    return;
  }
  fns[f] = fn;
  if (dev >= 0 && dev < kDev && done[f][dev]) return;
  cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
  if (dev >= 0 && dev < kDev) done[f][dev] = true;
}

size_t pm3_dep_items_bytes(int64_t cells_per_job, int njobs, int64_t n_used) {
  // bricks hold at least one coarse cell: one item per cell at most, plus one per kDepChunk particles, plus the count
  return sizeof(int2) * ((size_t)cells_per_job * njobs + (size_t)(n_used / kDepChunk) + 2);
}

int64_t pm3_deposit_bricks(const PM3Args &a) {
  const int mc = pm3_brick_mc(a);
  if (!mc) return 0;
  const int cb = kBrick / mc;
  return (int64_t)bricks_of(a.rdep[0], cb) * bricks_of(a.rdep[1], cb) * bricks_of(a.rdep[2], cb) * a.njobs;
}

// the brick deposit (TSC or CIC), with its work list where the caller gives the scratch for one
template <bool CIC>
static int launch_deposit_bricks(const PM3Args &a, int mc, cudaStream_t s) {
  const PM3K p = make_k(a);
  const int64_t nbricks = pm3_deposit_bricks(a);
  if (nbricks <= 0) return 0;
  if (!a.dep_items) {
    k_deposit_brick<CIC><<<(unsigned)nbricks, kDepThreads, 0, s>>>(p, mc, nbricks, nullptr, nullptr);
    return 1;
  }
  // one item per brick, and behind them at most one per kDepChunk particles
  const int64_t cap = nbricks + a.n_particles_hint / kDepChunk + 1;
  int *count = a.dep_count ? a.dep_count : reinterpret_cast<int *>(a.dep_items + cap);
  if (!a.dep_count || !a.zeroed) cudaMemsetAsync(count, 0, sizeof(int), s);
  k_dep_items<<<(unsigned)std::min<int64_t>((nbricks + 255) / 256, 4096), 256, 0, s>>>(p, mc, nbricks, kDepChunk,
                                                                                     a.dep_items, count, cap);
  // one block per possible item: resident blocks that loop over the list took 6 % longer (barriers, fixed shares)
  k_deposit_brick<CIC><<<(unsigned)cap, kDepThreads, 0, s>>>(p, mc, nbricks, a.dep_items, count);
  return 2;
}

int launch_pm3_deposit(const PM3Args &a, cudaStream_t s) {
  // Buffered meshes of fewer bricks than multiprocessors go by coarse cell, a warp each: the tile mesh of PM2 on a 32^3
  // box (27 bricks of a 40^3 mesh) takes 113 us a call so, 121 by bricks; eight of them (216 bricks) 176 and 146
  const int mc = pm3_brick_mc(a);
  if (mc && (a.wrap || pm3_deposit_bricks(a) >= a.num_sms)) return launch_deposit_bricks<false>(a, mc, s);
  const PM3K p = make_k(a);
  const int64_t warps = (int64_t)a.rdep[0] * a.rdep[1] * a.rdep[2] * a.njobs;
  k_deposit<<<(unsigned)((warps + kWarps - 1) / kWarps), kWarps * 32, 0, s>>>(p);
  return 1;
}

int launch_cic_bricks(const PM3Args &a, cudaStream_t s) {
  const int mc = pm3_brick_mc(a);
  return mc ? launch_deposit_bricks<true>(a, mc, s) : 0;
}

// cuTensorMapEncodeTiled through the runtime's driver entry point (no link to libcuda)
static PFN_cuTensorMapEncodeTiled_v12000 tensor_map_encoder() {
  static PFN_cuTensorMapEncodeTiled_v12000 fn = nullptr;
  static bool tried = false;
  if (!tried) {
    tried = true;
    void *f = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &f, cudaEnableDefault, &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      fn = (PFN_cuTensorMapEncodeTiled_v12000)f;
  }
  return fn;
}

bool launch_pm3_force_gather(const PM3Args &a, cudaStream_t s) {
  const int mc = pm3_brick_mc(a);
  if (!mc || !a.phi) return false;
  PFN_cuTensorMapEncodeTiled_v12000 encode = tensor_map_encoder();
  if (!encode) return false;
  // the potential as a 4-d tensor [slot][z][y][x], boxes of the potential window
  const cuuint64_t m = (cuuint64_t)a.n + 2 * a.phi_pad;
  const cuuint64_t dims[4] = {m, m, m, (cuuint64_t)a.nslots};
  const cuuint64_t strides[3] = {m * 4, m * m * 4, m * m * m * 4};
  const cuuint32_t box[4] = {kPotX, kPotW, kPotW, 1};
  const cuuint32_t estr[4] = {1, 1, 1, 1};
  CUtensorMap tmap;
  if (encode(&tmap, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 4, a.phi, dims, strides, box, estr,
             CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
             CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
    return false;
  PM3K p = make_k(a);
  const int cb = kBrick / mc;
  const int64_t nbricks = (int64_t)bricks_of(a.ract[0], cb) * bricks_of(a.ract[1], cb) * bricks_of(a.ract[2], cb) * a.njobs;
  set_smem_attr_once((const void *)k_force_gather, kFgSmem);
  const int64_t grid = std::min<int64_t>(nbricks, a.num_sms > 0 ? a.num_sms : 148);
  if (!a.brick_ctr) return false;
  if (!a.zeroed) cudaMemsetAsync(a.brick_ctr, 0, sizeof(int32_t), s);
  if (grid > 0) k_force_gather<<<(unsigned)grid, kFgThreads, kFgSmem, s>>>(p, mc, nbricks, a.phi_pad, tmap);
  return true;
}

// ghost points of the padded potential: each takes the interior point it is a periodic image of.
// The z slabs (all y, x), the y slabs (interior z, all x) and the x slabs (interior z, y) are
// disjoint and together cover every ghost point once.
__global__ void k_pm3_ghosts(float *phi, int n, int nslots) {
  const int P = kPotPad;
  const int m = n + 2 * P;
  const int nz = 2 * P * m * m, ny = n * 2 * P * m, nx = n * n * 2 * P;
  const int per = nz + ny + nx;
  const int sl = blockIdx.y;
  float *base = phi + (int64_t)sl * m * m * m;
  for (int e = blockIdx.x * blockDim.x + threadIdx.x; e < per; e += gridDim.x * blockDim.x) {
    int r = e, x, y, z;
    if (r < nz) {
      x = r % m;
      y = (r / m) % m;
      const int g = r / (m * m);  // 0 .. 2P-1
      z = g < P ? g : n + g;
    } else if ((r -= nz) < ny) {
      x = r % m;
      const int g = (r / m) % (2 * P);
      y = g < P ? g : n + g;
      z = P + r / (m * 2 * P);
    } else {
      r -= ny;
      const int g = r % (2 * P);
      x = g < P ? g : n + g;
      y = P + (r / (2 * P)) % n;
      z = P + r / (2 * P * n);
    }
    const int sx = x < P ? x + n : (x >= n + P ? x - n : x);
    const int sy = y < P ? y + n : (y >= n + P ? y - n : y);
    const int sz = z < P ? z + n : (z >= n + P ? z - n : z);
    base[((int64_t)z * m + y) * m + x] = base[((int64_t)sz * m + sy) * m + sx];
  }
}

void launch_pm3_ghosts(const PM3Args &a, cudaStream_t s) {
  const int m = a.n + 2 * kPotPad;
  const int64_t per = (int64_t)2 * kPotPad * m * m + (int64_t)a.n * 2 * kPotPad * m + (int64_t)a.n * a.n * 2 * kPotPad;
  const unsigned gx = (unsigned)std::min<int64_t>((per + 255) / 256, 4096);
  k_pm3_ghosts<<<dim3(gx, (unsigned)a.nslots), 256, 0, s>>>(a.phi, a.n, a.nslots);
}

void launch_pm3_gather(const PM3Args &a, cudaStream_t s) {
  PM3K p = make_k(a);
  const int64_t warps = (int64_t)a.ract[0] * a.ract[1] * a.ract[2] * a.njobs;
  k_gather<<<(unsigned)((warps + kWarps - 1) / kWarps), kWarps * 32, 0, s>>>(p);
}

// ---------------------------------------------------------------------------------------------
// Green_3D (Green/Green.f90:1-80) in FP64 on the device.  G depends on |k_d|
// per axis only, so one thread evaluates an octant point and writes its (up
// to) four mirror images in the stored half spectrum [k3][k2][k1].

struct GreenK {
  int n;
  double apm_soft, apm_range, gpow, alpha, c215;
  int p2;  // 2p+2
  const double *fs;
  float *G;
};

__global__ void k_green(GreenK p) {
  const int h = p.n / 2;
  const int64_t tot = (int64_t)(h + 1) * (h + 1) * (h + 1);
  const double twopi = 6.283185307179586476925286766559;
  for (int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; e < tot; e += (int64_t)gridDim.x * blockDim.x) {
    const int a = (int)(e % (h + 1)), b = (int)((e / (h + 1)) % (h + 1)), c = (int)(e / ((int64_t)(h + 1) * (h + 1)));
    const double kv[3] = {p.fs[a], p.fs[b], p.fs[c]};
    double D[3], u2n = 1.0, ur[3] = {0, 0, 0};
    for (int d = 0; d < 3; d++) {
      D[d] = p.alpha * sin(kv[d]) + (1 - p.alpha) * sin(2 * kv[d]) / 2;
      const double s = sin(kv[d] / 2);
      u2n *= 1 - s * s + p.c215 * s * s * s * s;
    }
    for (int i3 = -2; i3 <= 2; i3++)
      for (int i2 = -2; i2 <= 2; i2++)
        for (int i1 = -2; i1 <= 2; i1++) {
          const double kn[3] = {kv[0] + twopi * i1, kv[1] + twopi * i2, kv[2] + twopi * i3};
          const double kmag = sqrt(kn[0] * kn[0] + kn[1] * kn[1] + kn[2] * kn[2]);
          double U = 1.0;
          for (int d = 0; d < 3; d++) U *= (kn[d] == 0.0) ? 1.0 : sin(kn[d] / 2) / (kn[d] / 2);
          double Up = 1.0;
          for (int q = 0; q < p.p2; q++) Up *= U;
          double Ss, Sr;
          if (kmag == 0.0) {
            Ss = 1.0;
          } else {
            const double y = p.apm_soft * kmag / 2;
            double sy, cy;
            sincos(y, &sy, &cy);
            const double y2 = y * y;
            Ss = 12.0 / (y2 * y2) * (2 - 2 * cy - y * sy);
          }
          if (p.apm_range == 0.0) {
            Sr = 0.0;
          } else if (kmag == 0.0) {
            Sr = 1.0;
          } else {
            const double y = p.apm_range * kmag / 2;
            double sy, cy;
            sincos(y, &sy, &cy);
            const double y2 = y * y;
            Sr = 12.0 / (y2 * y2) * (2 - 2 * cy - y * sy);
          }
          const double f = (Ss * Ss - Sr * Sr) / (kmag * kmag);
          for (int d = 0; d < 3; d++) ur[d] += Up * kn[d] * f;
        }
    const double num = D[0] * ur[0] + D[1] * ur[1] + D[2] * ur[2];
    const double den = D[0] * D[0] + D[1] * D[1] + D[2] * D[2];
    const double pi4 = 12.566370614359172953850573533118;
    float g = (float)(pi4 * num / den / (u2n * u2n) / p.gpow);
    // Gk(::n/2,::n/2,::n/2) = 0 (Green.f90:71)
    if ((a == 0 || a == h) && (b == 0 || b == h) && (c == 0 || c == h)) g = 0.0f;
    const int n = p.n, nh = h + 1;
    const int bs[2] = {b, (n - b) % n}, cs[2] = {c, (n - c) % n};
    for (int u = 0; u < 2; u++) {
      if (u == 1 && cs[1] == cs[0]) continue;
      for (int v = 0; v < 2; v++) {
        if (v == 1 && bs[1] == bs[0]) continue;
        p.G[((int64_t)cs[u] * n + bs[v]) * nh + a] = g;
      }
    }
  }
}

void launch_green_fp64(int n, double apm_soft, double apm_range, double gridsize, int p_order, float *G,
                       cudaStream_t s) {
  // Fortran literals 4./3, 2./15 and 1./nglobal are single precision, gridsize is real(4)
  double *h_fs = new double[n];
  const double pi = 3.14159265358979323846;
  const double inv_n = (double)(1.0f / (float)n);
  for (int k = 1; k <= n; k++) {
    const int m = (k + n / 2 - 1) % n - n / 2;
    h_fs[k - 1] = 2.0 * pi * inv_n * (double)m;
  }
  double *d_fs = nullptr;
  cudaMallocAsync(&d_fs, sizeof(double) * n, s);
  cudaMemcpyAsync(d_fs, h_fs, sizeof(double) * n, cudaMemcpyHostToDevice, s);
  GreenK p;
  p.n = n;
  p.apm_soft = apm_soft;
  p.apm_range = apm_range;
  const float gs = (float)gridsize;
  p.gpow = (double)(gs * gs);
  p.alpha = (double)(4.0f / 3.0f);
  p.c215 = (double)(2.0f / 15.0f);
  p.p2 = 2 * p_order + 2;
  p.fs = d_fs;
  p.G = G;
  k_green<<<148 * 8, 128, 0, s>>>(p);
  cudaFreeAsync(d_fs, s);
  cudaStreamSynchronize(s);
  delete[] h_fs;
}

}  // namespace cube

// PP short-range pair force over the neighbouring PP cells
// (pp_force_kernel.c:282-325, pp_force_kernel.cu:192-250) and the kick of the
// interior particles (pp_force_kernel.c:339-364).
//
// Work decomposition.  An item is one interior PP cell, or a C-particle
// chunk of a crowded one (the kick's binning orders a cell's particles by
// Morton sub-cell, so a chunk occupies a compact sub-volume).  A particle of
// range rc needs the cells within R = ceil(rc * rcp / ratio_cs) of its own
// (pp_force_kernel.cu:205); the rows (dy, dz) of that stencil whose nearest
// point is farther than rc are skipped, and the cells of a row are one
// contiguous range of the cell-sorted array.  Items are bucketed by cost
// (log2 of candidates per lane group) and a persistent kernel hands them out
// heaviest first through an atomic queue head, so the lognormal occupancy of
// clustered boxes does not leave a tail.
//
// The kick runs k_pp_pairs: per item, the stencil's rows arrive in shared memory by bulk copies, candidates
// beyond rc of the bounding box of the item's particles are dropped, a TF32 tensor-core product
// lists for every particle the candidates that can lie within rc, and only the listed pairs are
// evaluated, in FP32 on f32x2 arithmetic (FFMA2, FMUL2, FADD2: two pairs per lane and
// instruction; every operation rounds as its scalar form).  Sums are Kahan-compensated over the
// batches of an item and merged with TwoSum shuffles, and the owning lane applies af*mass^2, the
// kick, f2max and vmax.
//
// k_pp_force is the scalar form (the pair count and the comparison shapes): lane (group g,
// particle i) of floor(32/ni) groups evaluates every ngrp-th candidate that passes the box test.
//
// Both kernels are issue-bound, so the per-lane state that is touched once per batch or item (Kahan sums,
// maxima, the owned particle's velocity, which a cp.async brings in while the item runs) lives in
// shared memory, and a warp pops its work items up to four at a time, each carrying its first
// particle, count, stencil radius and pair-law constants (k_pp_items computes them once per kick).
#include <type_traits>
#include <utility>

#include "common.cuh"

namespace cube {

constexpr int kPPThreads = 256;
constexpr int kPPWarps = kPPThreads / 32;
constexpr int kMaxRows = 96;  // stencil rows per row table of the scalar kernel (a multiple of 32)
constexpr int kBuckets = 32;
constexpr float kFar = 1e7f;  // coordinate of a padding candidate: beyond every range, and its law stays finite

// Kernel shapes the autotuner picks from (the host times each on the kick's own particles):
// chunk = i-particles per work item, so a crowded PP cell of n particles gets ceil(n / chunk)
// warps; jtile = candidates a warp stages in shared memory between two flushes; unroll = unroll
// factor of the filter loop (packed) or the pair loop (scalar); blocks = resident blocks per SM
// the registers are budgeted for (4: 64 registers a thread, 3: 80), packed = the pair-list kernel
// k_pp_pairs with the law on f32x2 arithmetic.  Shape 0 is the default; the scalar shapes
// (k_pp_force) are kept for comparison.
constexpr PPShapeDesc kShapes[] = {
    {16, 224, 4, 4, 1}, {16, 256, 4, 4, 1}, {16, 224, 2, 4, 1}, {16, 128, 4, 4, 1}, {16, 256, 4, 3, 1},
    {8, 224, 4, 4, 1},  {8, 128, 4, 4, 1},  {16, 64, 2, 4, 0},  {32, 64, 2, 4, 0}};
// the pair-count kernel (scalar loop, the work list of shape 0)
constexpr PPShapeDesc kCountShape = {kShapes[0].chunk, 64, 2, 4, 0};
constexpr int kNumShapes = (int)(sizeof(kShapes) / sizeof(kShapes[0]));
static_assert(kNumShapes <= kMaxPPShapes, "shape table");
constexpr int min_shape_chunk() {
  int c = kShapes[0].chunk;
  for (int i = 1; i < kNumShapes; i++) c = kShapes[i].chunk < c ? kShapes[i].chunk : c;
  return c;
}
constexpr int kMinChunk = min_shape_chunk();  // the work list capacity is sized for it
static_assert(kShapes[0].chunk == kPPChunk, "shape 0 is the default shape");
// Per-warp shared memory: the staged candidates (float4 [jtile + 32]), then the per-lane state kept in
// shared memory rather than registers (it is touched once per flush or item): f2 and |v| maxima, the
// owned particle's velocity (copied in asynchronously while the item runs), Kahan sums and
// compensations; then the batch of work items the warp popped, and the mbarrier of its copies.  The
// scalar kernel adds its row table, the item's bounding box and the row-table cache.
constexpr int kLaneFieldsScalar = 13, kLaneFieldsPairs = 19;
constexpr int kPop = 4;  // most work items a warp takes from the queue at a time
constexpr int kRefill = 96;  // pair kernel: a batch of candidates is evaluated once less room than this is left
constexpr size_t pp_stage_bytes(int jtile) { return sizeof(float4) * (jtile + 32); }
constexpr size_t pp_smem_warp(int jtile, bool pairs) {
  return pp_stage_bytes(jtile) + sizeof(PPItem) * kPop +
         (pairs ? sizeof(float) * 32 * kLaneFieldsPairs + 16
                : sizeof(float) * (32 * kLaneFieldsScalar + 8) + sizeof(int2) * kMaxRows);
}
constexpr size_t pp_smem_block(int jtile, bool pairs) { return pp_smem_warp(jtile, pairs) * kPPWarps; }
static_assert(pp_smem_warp(64, false) % 16 == 0 && pp_smem_warp(224, true) % 16 == 0 &&
                  (sizeof(int2) * kMaxRows) % 16 == 0,
              "16-byte aligned warp areas, bounding box and item batch");

// F_ra(r, apm) of basic_functions.f08:95-109 / pp_force_kernel.c:45-74 in FP32 without
// divisions or branches: with ep = 2r/apm = r * ce and k = (1/35) / apm^2,
//   ep <= 1: k (224ep - 224ep^3 + 70ep^4 + 48ep^5 - 21ep^6)
//   ep > 1:  k (12/ep^2 - 224 + 896ep - 840ep^2 + 224ep^3 + 70ep^4 - 48ep^5 + 7ep^6)
//            = (3/35)/r^2 + k (-224 + 896ep - ... + 7ep^6)      (k 12/ep^2 = (3/35)/r^2)
//   ep > 2:  1/r^2
__device__ __forceinline__ float F_ra_soft(float r, float ir2, float ce, float k) {
  const float ep = r * ce;
  float qo = fmaf(7.0f, ep, -48.0f);
  qo = fmaf(qo, ep, 70.0f);
  qo = fmaf(qo, ep, 224.0f);
  qo = fmaf(qo, ep, -840.0f);
  qo = fmaf(qo, ep, 896.0f);
  qo = fmaf(qo, ep, -224.0f);
  float qi = fmaf(-21.0f, ep, 48.0f);
  qi = fmaf(qi, ep, 70.0f);
  qi = fmaf(qi, ep, -224.0f);
  qi = qi * ep;
  qi = fmaf(qi, ep, 224.0f);
  qi = qi * ep;
  return ep > 2.0f ? ir2 : (ep > 1.0f ? fmaf(k, qo, (3.0f / 35.0f) * ir2) : k * qi);
}

// 1/sqrt(x) on the special-function unit with subnormal inputs flushed (rsqrt.approx.ftz):
// squared pair distances are either 0 (masked), at least (2^-16 fine cell)^2 or a far sentinel,
// never subnormal, so only rsqrtf's handling of subnormal inputs is left out
__device__ __forceinline__ float rsqrt_ftz(float x) {
  float y;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

// packed f32x2 arithmetic (sm_100: one instruction updates both halves, each rounded as the
// scalar operation)
__device__ __forceinline__ float2 dup(float v) { return make_float2(v, v); }
__device__ __forceinline__ float2 add2(float2 a, float2 b) { return __fadd2_rn(a, b); }
__device__ __forceinline__ float2 mul2(float2 a, float2 b) { return __fmul2_rn(a, b); }
__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) { return __ffma2_rn(a, b, c); }

// s(r^2) = (F_ra(r,app) - F_ra(r,rc)) / r, so that the pair force is s * (dx, dy, dz).  With
// ep = 2r/rc and k = 1/(35 rc^2), for app < r:
//   outer (1 < ep < 2): 1/r^2 - F_ra(r,rc) = k/ep^2 (128 + 224ep^2 - 896ep^3 + 840ep^4 - 224ep^5 - 70ep^6
//                       + 48ep^7 - 7ep^8) = k/ep^2 (2-ep)^5 (4 + 10ep + 22ep^2 + 7ep^3)
//   inner (ep <= 1): the outer form plus k/ep^2 (1-ep)^6 (12 + 72ep + 28ep^2)
// (the octic has a fivefold root at ep = 2, the difference of the two pieces a sixfold root at ep = 1), and
// k/ep^2 / r = (1/140) / r^3.  With h = r/rc = ep/2:
//   s = r^-3 [ (1-h)^5 (32/140) (4 + 20h + 88h^2 + 56h^3) + max(1-2h, 0)^6 (1/140) (12 + 144h + 112h^2) ].
// Every term is positive, so the law keeps its relative accuracy up to r = rc (the expanded octic
// cancels there: terms of 100 leave an absolute error of 6e-6); both factors lie in [0, 1], so the
// saturating FMA gives them without a compare, and 1-h saturated makes the law exactly zero beyond rc.
// The coefficients are literals, so a law costs one register per item (1/rc).  Inside the softening
// length (soft()) both F_ra terms are evaluated directly.
struct PairLaw {
  float cep, k35;
  // the constants of range rc, as k_pp_items stores them in the work item
  __device__ __forceinline__ static float k35_of(float rc_) { return 1.0f / (35.0f * rc_ * rc_); }
  __device__ __forceinline__ static float cep_of(float rc_) { return 2.0f / rc_; }
  __device__ __forceinline__ void init(const PPItem &it) {
    k35 = it.k35;
    cep = it.cep;
  }
  __device__ __forceinline__ float scale(float r2) const {
    const float invr = rsqrt_ftz(r2);
    const float h = r2 * invr * (0.5f * cep);
    const float v = __saturatef(1.0f - h), u = __saturatef(fmaf(-2.0f, h, 1.0f));
    const float c = fmaf(fmaf(fmaf(1792.0f / 140.0f, h, 2816.0f / 140.0f), h, 640.0f / 140.0f), h, 128.0f / 140.0f);
    const float w = fmaf(fmaf(112.0f / 140.0f, h, 144.0f / 140.0f), h, 12.0f / 140.0f);
    const float v2 = v * v, u2 = u * u, u3 = u2 * u;
    const float a = (v2 * v2) * (v * c);
    return fmaf(u3 * u3, w, a) * (invr * invr * invr);
  }
  // scale() of two squared distances on packed f32x2 arithmetic: every operation is the scalar
  // one, rounded the same way, so each half equals scale() of that half bit for bit
  __device__ __forceinline__ float2 scale2(float2 r2) const {
    const float2 invr = make_float2(rsqrt_ftz(r2.x), rsqrt_ftz(r2.y));
    const float2 h = mul2(mul2(r2, invr), dup(0.5f * cep));
    const float2 v = make_float2(__saturatef(1.0f - h.x), __saturatef(1.0f - h.y)),
                 u = make_float2(__saturatef(fmaf(-2.0f, h.x, 1.0f)), __saturatef(fmaf(-2.0f, h.y, 1.0f)));
    float2 c = fma2(dup(1792.0f / 140.0f), h, dup(2816.0f / 140.0f));
    c = fma2(c, h, dup(640.0f / 140.0f));
    c = fma2(c, h, dup(128.0f / 140.0f));
    const float2 w = fma2(fma2(dup(112.0f / 140.0f), h, dup(144.0f / 140.0f)), h, dup(12.0f / 140.0f));
    const float2 v2 = mul2(v, v), u2 = mul2(u, u), u3 = mul2(u2, u);
    const float2 a = mul2(mul2(v2, v2), mul2(v, c));
    return mul2(fma2(mul2(u3, u3), w, a), mul2(mul2(invr, invr), invr));
  }
  // 0 < r <= app: (F_ra(r, app) - F_ra(r, rc)) / r; cea = 2/app, ka = (1/35)/app^2
  __device__ __forceinline__ float soft(float r2, float cea, float ka) const {
    const float invr = rsqrt_ftz(r2);
    const float r = r2 * invr, ir2 = invr * invr;
    return (F_ra_soft(r, ir2, cea, ka) - F_ra_soft(r, ir2, cep, k35)) * invr;
  }
};

// warp minimum / maximum of a float in one instruction (sm_100a)
__device__ __forceinline__ float warp_min_redux(float v) {
  float r;
  asm volatile("redux.sync.min.f32 %0, %1, 0xffffffff;" : "=f"(r) : "f"(v));
  return r;
}
__device__ __forceinline__ float warp_max_redux(float v) {
  float r;
  asm volatile("redux.sync.max.f32 %0, %1, 0xffffffff;" : "=f"(r) : "f"(v));
  return r;
}

// n / d for 0 <= n < 2^11 and 1 <= d <= 64 by a multiply with ceil(2^20 / d): the error
// n * (ceil(2^20/d) - 2^20/d) / 2^20 < 2^-9 stays below the 1/d gap to the next integer
struct DivTable {
  int m[65];
  constexpr DivTable() : m() {
    for (int d = 1; d <= 64; d++) m[d] = ((1 << 20) + d - 1) / d;
  }
};
__constant__ DivTable c_div = DivTable();
__device__ __forceinline__ int div_small(int n, int d) { return (n * c_div.m[d]) >> 20; }

__device__ __forceinline__ int lowest_bit(unsigned m) { return __ffs(m) - 1; }
__device__ __forceinline__ int lowest_bit(unsigned long long m) { return __ffsll(m) - 1; }

// 4-byte asynchronous global -> shared copy (cp.async, sm_80+), its commit and wait
__device__ __forceinline__ void cp_async4(float *smem, const float *gmem) {
  const unsigned sa = (unsigned)__cvta_generic_to_shared(smem);
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(sa), "l"(gmem) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;" ::: "memory"); }

__device__ __forceinline__ void kahan_add(float &s, float &c, float x) {
  float y = x - c;
  float t = s + y;
  c = (t - s) - y;
  s = t;
}

// (hi, lo) + (hi2, lo2) with an error-free TwoSum of the high parts
__device__ __forceinline__ void two_sum_merge(float &hi, float &lo, float hi2, float lo2) {
  float s = hi + hi2;
  float bp = s - hi;
  float err = (hi - (s - bp)) + (hi2 - bp);
  hi = s;
  lo = lo + lo2 + err;
}

struct PPK {
  int nt, ntt, nns, nnt, ntile, rcs;
  const TilePP *tiles;
  const int32_t *cs;
  const float4 *spos;
  const float *range_loc;
  PPItem *items;    // tile-major, heaviest bucket first
  int32_t *sched;   // schedule words, layout in sched_ints()
  int64_t item_cap;
  int t_lo, t_hi;   // tiles of this force launch; its queue head is sched_head(t_lo, t_hi)
  float *vp;
  float mass2, kick, app, app2;
  float cea, ka;  // softening-law constants 2/app and (1/35)/app^2 (0 without softening)
  float *out;
  int want_vmax;
  int32_t *err;
  int64_t max_cells;          // max interior PP cells per tile (grid sizing)
  unsigned long long *pairs;  // COUNT mode: accepted ordered pairs
};

// PP range of the particles of interior cell (x, y, z) of tile t (per subtile, pp_force_kernel.cu:776-790)
__device__ __forceinline__ float cell_range(const PPK &p, int t, int x, int y, int z, int rcp) {
  const int tx = t % p.nnt, ty = (t / p.nnt) % p.nnt, tz = t / (p.nnt * p.nnt);
  const int sx = (x / rcp - 1) / p.ntt, sy = (y / rcp - 1) / p.ntt, sz = (z / rcp - 1) / p.ntt;
  return p.range_loc[(((tz * p.nnt + ty) * p.nnt + tx) * p.nns + sz) * p.nns * p.nns + sy * p.nns + sx];
}

// stencil radius in cells and the row test: row (dy, dz) can hold a particle within rc
__device__ __forceinline__ int stencil_radius(float rc, int rcp, int rcs) {
  return (int)ceilf(rc * (float)rcp / (float)rcs);
}
__device__ __forceinline__ bool row_needed(int dy, int dz, float h, float rc2) {
  const float ay = (float)max(abs(dy) - 1, 0) * h, az = (float)max(abs(dz) - 1, 0) * h;
  return ay * ay + az * az < rc2;
}

// Schedule words (int32), for ntile tiles: [0, 32 ntile) item counts per (tile, bucket), turned
// into the first item slot of each (tile, bucket) by k_pp_offsets; [32 ntile, 64 ntile) cursors;
// then ntile + 1 tile bases (first item of each tile, and the total); then ntile + 1 queue
// heads: a launch over tiles [t_lo, t_hi) uses head t_lo, one over all tiles head ntile, so
// launches over disjoint tile ranges never share a head.
__host__ __device__ inline int64_t sched_base(int ntile) { return 2 * (int64_t)kBuckets * ntile; }
__host__ __device__ inline int64_t sched_head(int ntile, int t_lo, int t_hi) {
  return sched_base(ntile) + ntile + 1 + (t_hi - t_lo == ntile ? ntile : t_lo);
}

// cost bucket of a chunk with ni i-particles and nj candidates, heavy = high index:
// the warp walks the candidates in floor(32/ni) lane groups
__device__ __forceinline__ int cost_bucket(int ni, int64_t nj) {
  int64_t c = nj / (32 / max(ni, 1));
  if (c < 1) c = 1;
  int b = 63 - __clzll(c);
  return b > kBuckets - 1 ? kBuckets - 1 : b;
}

// Enumerate the chunks of the interior PP cells; pass 0 counts items per (tile, bucket),
// pass 1 writes them tile by tile, heaviest bucket first inside a tile.  A cell's full chunks
// share one bucket and its remainder chunk has another, so a thread reserves its slots with at
// most two shared-memory atomics.
template <int PASS, int C>
__global__ void __launch_bounds__(256) k_pp_items(PPK p) {
  __shared__ int sc[kBuckets], sbase[kBuckets];
  const int t = blockIdx.y;
  int32_t *cnt = p.sched + (int64_t)kBuckets * t;                     // counts, then first slots
  int32_t *cur = p.sched + (int64_t)kBuckets * (p.ntile + t);         // cursors
  if (threadIdx.x < kBuckets) sc[threadIdx.x] = 0;
  __syncthreads();
  const TilePP tp = p.tiles[t];
  const int rcp = tp.rcp, S = tp.S, npg = p.nt * rcp;
  const int64_t ncell = (int64_t)npg * npg * npg;
  const int64_t c = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  int nfull = 0, bfull = 0, brem = -1, ni = 0, i0 = 0;
  int64_t g = 0;
  PPItem it{};
  if (c < ncell) {
    // cell coordinates in 32-bit arithmetic when the tile's cells fit (64-bit division is a long
    // software sequence)
    int x, y, z;
    if (ncell <= 0xffffffffLL) {
      const unsigned u = (unsigned)c, n = (unsigned)npg, q = u / n, qq = q / n;
      x = (int)(u - q * n) + rcp;
      y = (int)(q - qq * n) + rcp;
      z = (int)qq + rcp;
    } else {
      x = (int)(c % npg) + rcp;
      y = (int)((c / npg) % npg) + rcp;
      z = (int)(c / ((int64_t)npg * npg)) + rcp;
    }
    g = tp.cell0 + ((int64_t)z * S + y) * S + x;
    i0 = p.cs[g];
    ni = p.cs[g + 1] - i0;
    // Sparse neighbouring cells along x share an item when their particles fit one chunk and
    // they lie in one subtile: an aligned group of four cells (at least three occupied), else
    // an aligned pair (both occupied).  The item's stencil rows are `span` cells longer, which
    // walks fewer candidates than separate items and saves their per-item work; the other
    // cells of the group make no item.  Every cell of a group decides the same way.
    int span = 0;
    const int lxi = x - rcp;
    {
      auto count_at = [&](int lx) {
        const int64_t gg = g + (lx - lxi);
        return p.cs[gg + 1] - p.cs[gg];
      };
      // the PP range is set per subtile: a group inside one subtile shares it (groups across a
      // subtile boundary are not formed)
      auto same_range = [&](int lx0, int n) { return lx0 / (rcp * p.ntt) == (lx0 + n - 1) / (rcp * p.ntt); };
      const int h4 = lxi & ~3, h2 = lxi & ~1;
      int tot4 = 0, occ4 = 0;
      if (h4 + 3 < npg)
        for (int k = 0; k < 4; k++) {
          const int cnt = count_at(h4 + k);
          tot4 += cnt;
          occ4 += cnt > 0 ? 1 : 0;
        }
      if (h4 + 3 < npg && tot4 <= C && occ4 >= 3 && same_range(h4, 4)) {
        if (lxi == h4) {
          ni = tot4;
          span = 3;
        } else {
          ni = 0;
        }
      } else if (h2 + 1 < npg) {
        const int n0 = count_at(h2), n1 = count_at(h2 + 1);
        if (n0 > 0 && n1 > 0 && n0 + n1 <= C && same_range(h2, 2)) {
          if (lxi == h2) {
            ni = n0 + n1;
            span = 1;
          } else {
            ni = 0;
          }
        }
      }
    }
    if (ni > 0) {
      const float rc = cell_range(p, t, x, y, z, rcp);
      const int R = stencil_radius(rc, rcp, p.rcs);
      if (R > rcp) atomicOr(p.err, 1 << CUBE_ERR_INVALID);  // beyond the one coarse-cell halo
      const float h = (float)p.rcs / (float)rcp;
      const int Rc = min(R, rcp);
      it.cell = (uint32_t)g;
      it.dims = (rcp << 8) | (Rc << 16) | (span << 24);
      it.rc = rc;
      it.cep = PairLaw::cep_of(rc);
      it.k35 = PairLaw::k35_of(rc);
      it.h = h;
      it.rc2 = rc * rc;
      int64_t nj = 0;
      for (int dz = -Rc; dz <= Rc; dz++)
        for (int dy = -Rc; dy <= Rc; dy++) {
          if (!row_needed(dy, dz, h, rc * rc)) continue;
          const int64_t b = g + ((int64_t)dz * S + dy) * S;
          nj += p.cs[b + Rc + 1 + span] - p.cs[b - Rc];
        }
      nfull = ni / C;
      bfull = cost_bucket(C, nj);
      if (ni % C) brem = cost_bucket(ni % C, nj);
    }
  }
  int rfull = 0, rrem = 0;
  if (nfull) rfull = atomicAdd(&sc[bfull], nfull);
  if (brem >= 0) rrem = atomicAdd(&sc[brem], 1);
  __syncthreads();
  if (threadIdx.x < kBuckets) {
    const int n = sc[threadIdx.x];
    if (PASS == 0) {
      if (n) atomicAdd(&cnt[threadIdx.x], n);
    } else {
      sbase[threadIdx.x] = cnt[threadIdx.x] + (n ? atomicAdd(&cur[threadIdx.x], n) : 0);
    }
  }
  if (PASS == 1) {
    __syncthreads();
    const int64_t f0 = (int64_t)sbase[bfull] + rfull;
    const int dims = it.dims;
    for (int k = 0; k < nfull; k++) {
      it.i0 = i0 + k * C;
      it.dims = dims | C;
      if (f0 + k < p.item_cap) p.items[f0 + k] = it;
      else atomicOr(p.err, 1 << CUBE_ERR_CAPACITY);
    }
    if (brem >= 0) {
      const int64_t slot = (int64_t)sbase[brem] + rrem;
      it.i0 = i0 + nfull * C;
      it.dims = dims | (ni - nfull * C);
      if (slot < p.item_cap) p.items[slot] = it;
      else atomicOr(p.err, 1 << CUBE_ERR_CAPACITY);
    }
  }
}

// Between the two item passes: turn the (tile, bucket) counts into first slots, tiles in
// order and buckets heaviest first inside a tile, and record the tile bases.  One warp.
__global__ void k_pp_offsets(int32_t *sched, int ntile) {
  const int lane = threadIdx.x;
  int32_t *base = sched + sched_base(ntile);
  int acc = 0;
  for (int t = 0; t < ntile; t++) {
    const int c = sched[kBuckets * t + lane];
    int incl = c;  // inclusive sum over the heavier buckets b' >= lane
    for (int o = 1; o < 32; o <<= 1) {
      const int v = __shfl_down_sync(0xffffffffu, incl, o);
      if (lane + o < 32) incl += v;
    }
    if (lane == 0) base[t] = acc;
    sched[kBuckets * t + lane] = acc + incl - c;
    acc += __shfl_sync(0xffffffffu, incl, 0);
  }
  if (lane == 0) base[ntile] = acc;
}

// COUNT = false: forces and kick.  COUNT = true: only count the accepted ordered
// pairs 0 < r^2 < rc^2 (the algorithmic work of the kick, for the roofline).
// Shape: C i-particles per item, J staged candidates per flush, pair loop unrolled U times,
// registers budgeted for B resident blocks per SM.
template <bool COUNT, int C, int J, int U, int B>
__global__ void __launch_bounds__(kPPThreads, B) k_pp_force(PPK p) {
  // a flush has at most ceil(J / floor(32 / C)) rounds, one bit per round and lane in the
  // soft-pair mask
  constexpr int kBits = (J + 32 / C - 1) / (32 / C);
  static_assert(kBits <= 64, "at most 64 soft-pair bits per flush");
  using Mask = typename std::conditional<(kBits > 32), unsigned long long, unsigned>::type;
  extern __shared__ float4 pp_smem[];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  char *wbase = reinterpret_cast<char *>(pp_smem) + warp * pp_smem_warp(J, false);
  float4 *buf = reinterpret_cast<float4 *>(wbase);  // staging: float4 [J + 32]
  // (end of the row in the walk, start - walk offset)
  int2 *rows = reinterpret_cast<int2 *>(wbase + pp_stage_bytes(J));
  float *const ks = reinterpret_cast<float *>(rows + kMaxRows) + lane;  // field f at ks[32 f]
  float *const bbox = reinterpret_cast<float *>(rows + kMaxRows) + 32 * kLaneFieldsScalar;
  PPItem *const batch = reinterpret_cast<PPItem *>(bbox + 8);
  int *const tcache = reinterpret_cast<int *>(bbox + 6);  // cell and walk of the row table
  if (lane == 0) tcache[0] = -1;
  __syncwarp();
  for (int f = 6; f < 10; f++) ks[32 * f] = 0.f;  // f2, |v| maxima
  unsigned long long npairs = 0;
  // The warp takes kPop consecutive items per queue pop (one atomic and one load for all of
  // them); the items of a bucket cost about the same, and the lightest come last.
  for (int nb = 0, b = 0;; b++) {
    if (b == nb) {
      // items [first, last) of tiles [t_lo, t_hi), popped through this launch's own queue head
      const int32_t *tbase = p.sched + sched_base(p.ntile);
      const int first = tbase[p.t_lo];
      const int last = (int)min((int64_t)tbase[p.t_hi], p.item_cap);
      int it = 0;
      if (lane == 0) it = first + atomicAdd(p.sched + sched_head(p.ntile, p.t_lo, p.t_hi), kPop);
      it = __shfl_sync(0xffffffffu, it, 0);
      if (it >= last) break;
      nb = min(kPop, last - it);
      b = 0;
      __syncwarp();
      if (lane < 2 * nb) reinterpret_cast<int4 *>(batch)[lane] = reinterpret_cast<const int4 *>(p.items + it)[lane];
      __syncwarp();
    }
    const PPItem &item = batch[b];  // read from shared memory where used
    const int64_t g = (int64_t)item.cell;
    const int ni = item.dims & 0xff, R = (item.dims >> 16) & 0xff, span = item.dims >> 24;
    const int S = ((item.dims >> 8) & 0xff) * (p.nt + 2);
    const float rc2 = item.rc2;
    PairLaw law;
    law.init(item);
    // lanes = ngrp groups of ni lanes; group `grp` walks every ngrp-th candidate
    const int ngrp = 32 / ni;
    const int grp = div_small(lane, ni), il = lane - grp * ni;
    const bool has_i = grp < ngrp;  // the 32 mod ni leftover lanes idle
    const float4 pi = p.spos[item.i0 + il];
    bool boxed = false;  // the bounding box is taken once pi has arrived (after the first row table)
    for (int f = 0; f < 6; f++) ks[32 * f] = 0.f;  // Kahan sums of this item
    int nbuf = 0;  // staged candidates (warp-uniform)
    // Evaluate the staged candidates: group grp takes buf[grp + k*ngrp] in round k.  The loop
    // bound is the same for every lane (no divergent loop exits): the slots past nbuf hold a
    // far-away sentinel that the r < rc mask drops, and the lanes of an incomplete last group
    // (grp == ngrp) compute values that the group merge below never reads.  The main loop has
    // no branch: pairs inside the softening length (r <= app, common only in dense clumps) are
    // masked out of it and their rounds recorded in a bit mask (at most 32 rounds per flush);
    // a second loop then evaluates exactly those pairs, one per lane per step.
    auto flush = [&]() {
      buf[nbuf + lane] = make_float4(kFar, kFar, kFar, 0.f);
      __syncwarp();
      float px = 0.f, py = 0.f, pz = 0.f;
      const int nround = div_small(nbuf + ngrp - 1, ngrp);
      Mask softmask = 0u, bit = 1u;
      const float4 *bp = buf + grp;
#pragma unroll U
      for (int k = 0; k < nround; k++, bp += ngrp, bit <<= 1) {
        const float4 pj = *bp;
        const float dx = pj.x - pi.x, dy_ = pj.y - pi.y, dz_ = pj.z - pi.z;
        const float r2 = fmaf(dx, dx, fmaf(dy_, dy_, dz_ * dz_));
        if (COUNT) {
          npairs += (r2 < rc2) & (r2 > 0.0f) & has_i ? 1ull : 0ull;  // r = 0: the particle itself
        } else {
          // evaluated for every candidate and masked: a divergent accept branch would
          // run on nearly every round of a 32-lane warp anyway
          float s = law.scale(r2);
          s = (r2 < rc2) & (r2 > p.app2) ? s : 0.0f;
          softmask |= (r2 <= p.app2) & (r2 > 0.0f) & has_i ? bit : 0u;
          px = fmaf(s, dx, px);
          py = fmaf(s, dy_, py);
          pz = fmaf(s, dz_, pz);
        }
      }
      if (!COUNT) {
        while (__any_sync(0xffffffffu, softmask != 0u)) {
          if (softmask) {
            const int k = lowest_bit(softmask);
            softmask &= softmask - 1u;
            const float4 pj = buf[grp + k * ngrp];
            const float dx = pj.x - pi.x, dy_ = pj.y - pi.y, dz_ = pj.z - pi.z;
            const float s = law.soft(fmaf(dx, dx, fmaf(dy_, dy_, dz_ * dz_)), p.cea, p.ka);
            px = fmaf(s, dx, px);
            py = fmaf(s, dy_, py);
            pz = fmaf(s, dz_, pz);
          }
        }
        kahan_add(ks[0], ks[32], px);
        kahan_add(ks[64], ks[96], py);
        kahan_add(ks[128], ks[160], pz);
      }
      nbuf = 0;
      __syncwarp();
    };
    // The needed stencil rows are laid end to end in a table of up to kMaxRows rows: row k
    // covers walk positions [rows[k-1].x, rows[k].x), and walk position v is particle
    // v + rows[k].y.  Stencils with more rows (large R) are walked in several tables.
    // Consecutive items of one cell share their stencil: a table that holds the whole stencil is
    // kept for the next item (tcache: its cell, or -1, and its walk length).
    const int side = 2 * R + 1, nr = side * side;
    for (int r0 = 0; r0 < nr;) {
      int nrows = 0, walk = 0;
      const bool reuse = r0 == 0 && tcache[0] == (int)item.cell;
      if (reuse) {
        walk = tcache[1];
        r0 = nr;
      }
      const int rstart = r0;
      for (; r0 < nr && nrows <= kMaxRows - 32; r0 += 32) {
        const int ri = r0 + lane;
        int js = 0, len = 0;
        bool need = false;
        if (ri < nr) {
          const int q = div_small(ri, side);
          const int dz = q - R, dy = ri - q * side - R;
          need = row_needed(dy, dz, item.h, rc2);
          if (need) {
            const int64_t b = g + ((int64_t)dz * S + dy) * S;
            js = p.cs[b - R];
            len = p.cs[b + R + 1 + span] - js;
          }
        }
        const unsigned m = __ballot_sync(0xffffffffu, need);
        int incl = len;  // inclusive scan of the lengths (0 for rows not needed)
        for (int o = 1; o < 32; o <<= 1) {
          const int v = __shfl_up_sync(0xffffffffu, incl, o);
          if (lane >= o) incl += v;
        }
        if (need) rows[nrows + __popc(m & ((1u << lane) - 1u))] = make_int2(walk + incl, js - (walk + incl - len));
        nrows += __popc(m);
        walk += __shfl_sync(0xffffffffu, incl, 31);
      }
      if (!reuse && lane == 0) {
        tcache[0] = rstart == 0 && r0 >= nr ? (int)item.cell : -1;
        tcache[1] = walk;
      }
      __syncwarp();
      if (!boxed) {
        // bounding box of the item's particles: candidates farther than rc from it are dropped
        // while staging, so the pair loop below only sees possibly-interacting candidates
        boxed = true;
        const float blx = warp_min_redux(pi.x), bhx = warp_max_redux(pi.x), bly = warp_min_redux(pi.y),
                    bhy = warp_max_redux(pi.y), blz = warp_min_redux(pi.z), bhz = warp_max_redux(pi.z);
        if (lane == 0) {
          *reinterpret_cast<float4 *>(bbox) = make_float4(blx, bly, blz, bhx);
          *reinterpret_cast<float2 *>(bbox + 4) = make_float2(bhy, bhz);
        }
        // the owned particle's velocity is copied in while the item runs
        if (!COUNT && grp == 0 && has_i) {
          const float *v = p.vp + 3 * (int64_t)__float_as_int(pi.w);
          cp_async4(ks + 320, v);
          cp_async4(ks + 352, v + 1);
          cp_async4(ks + 384, v + 2);
        }
        cp_async_commit();
        __syncwarp();
      }
      if (walk == 0) continue;
      // Walk position -> particle.  Each lane's row index only moves forward and stops at the
      // last row (rows[nrows-1].x = walk > v), and the lanes past the end load the last
      // candidate again and drop it, so the loop below has no divergent branch or load.
      int kr = 0;
      auto locate = [&](int v) {
        v = min(v, walk - 1);
        while (__any_sync(0xffffffffu, v >= rows[kr].x)) kr += v >= rows[kr].x ? 1 : 0;
        return v + rows[kr].y;
      };
      float4 nxt = p.spos[locate(lane)];
      for (int vb = 0; vb < walk; vb += 32) {
        const float4 pj = nxt;
        nxt = p.spos[locate(vb + 32 + lane)];  // one step ahead
        const float4 bl = *reinterpret_cast<const float4 *>(bbox);  // (lo x, y, z, hi x)
        const float2 bh = *reinterpret_cast<const float2 *>(bbox + 4);  // (hi y, z)
        const float ex = fmaxf(fmaxf(bl.x - pj.x, pj.x - bl.w), 0.f);
        const float ey = fmaxf(fmaxf(bl.y - pj.y, pj.y - bh.x), 0.f);
        const float ez = fmaxf(fmaxf(bl.z - pj.z, pj.z - bh.y), 0.f);
        const bool keep = (vb + lane < walk) & (ex * ex + ey * ey + ez * ez < rc2);
        const unsigned m = __ballot_sync(0xffffffffu, keep);
        if (keep) {
          const int q = nbuf + __popc(m & ((1u << lane) - 1u));
          buf[q] = pj;
        }
        nbuf += __popc(m);
        if (nbuf > J - 32) flush();
      }
      __syncwarp();  // the next table overwrites this one
    }
    if (nbuf) flush();
    // merge the lane groups of each i-particle (tree over groups, stride s*ni lanes);
    // Kahan c is the negated low part
    float hx = ks[0], lx = -ks[32], hy = ks[64], ly = -ks[96], hz = ks[128], lz = -ks[160];
    for (int s = 1; s < ngrp; s <<= 1) {
      const int delta = s * ni;
      const float ohx = __shfl_down_sync(0xffffffffu, hx, delta), olx = __shfl_down_sync(0xffffffffu, lx, delta);
      const float ohy = __shfl_down_sync(0xffffffffu, hy, delta), oly = __shfl_down_sync(0xffffffffu, ly, delta);
      const float ohz = __shfl_down_sync(0xffffffffu, hz, delta), olz = __shfl_down_sync(0xffffffffu, lz, delta);
      if ((grp % (2 * s)) == 0 && grp + s < ngrp) {
        two_sum_merge(hx, lx, ohx, olx);
        two_sum_merge(hy, ly, ohy, oly);
        two_sum_merge(hz, lz, ohz, olz);
      }
    }
    if (!COUNT && grp == 0 && has_i) {
      const float ax = (hx + lx) * p.mass2, ay = (hy + ly) * p.mass2, az = (hz + lz) * p.mass2;
      ks[192] = fmaxf(ks[192], ax * ax + ay * ay + az * az);
      const int64_t ip = (int64_t)__float_as_int(pi.w);
      float *v = p.vp + 3 * ip;
      cp_async_wait_all();
      const float v0 = ks[320] + ax * p.kick, v1 = ks[352] + ay * p.kick, v2 = ks[384] + az * p.kick;
      v[0] = v0;
      v[1] = v1;
      v[2] = v2;
      ks[224] = fmaxf(ks[224], fabsf(v0));
      ks[256] = fmaxf(ks[256], fabsf(v1));
      ks[288] = fmaxf(ks[288], fabsf(v2));
    }
  }
  if (COUNT) {
    for (int o = 16; o; o >>= 1) npairs += __shfl_xor_sync(0xffffffffu, npairs, o);
    if (lane == 0) atomicAdd(p.pairs, npairs);
    return;
  }
  const float f2w = warp_max(ks[192]);
  if (lane == 0) atomic_max_nonneg(&p.out[1], f2w);
  if (p.want_vmax) {
    const float vm0 = warp_max(ks[224]), vm1 = warp_max(ks[256]), vm2 = warp_max(ks[288]);
    if (lane == 0) {
      atomic_max_nonneg(&p.out[2], vm0);
      atomic_max_nonneg(&p.out[3], vm1);
      atomic_max_nonneg(&p.out[4], vm2);
    }
  }
}

// ---- the pair-list kernel ----
//
// One warp per work item, in three phases per batch of up to J candidates:
//   stage: one bulk copy per stencil row brings its particles to shared memory; those beyond rc of the
//     item's box are dropped in place.  (Walking the rows with one load per lane and step cost
//     about 120 instructions per 32 candidates in finding each lane's row; this costs 40.)
//   filter: the squared distances of the item's 16 rows (its i-particles, replicated when there are
//     fewer than 9) to 8 candidates come from one TF32 tensor-core product (mma.m16n8k8, the
//     contraction  -2 xi . xj + |xj|^2 + (|xi|^2 - T)  over positions relative to the box
//     centre); the sign of each result goes into a bit list of its lane.  T is rc^2 plus the largest
//     error that TF32 operands can make in the item's box, so no pair within rc is missed.
//   pairs: each lane takes the candidates of its two rows' lists one after the other (two rows = the two
//     halves of f32x2 arithmetic) and evaluates the law in FP32 from the exact positions; the few listed
//     pairs beyond rc get exactly zero from it.
// Lane (g, t) = (lane / 4, lane % 4) owns rows g and g + 8 against every fourth candidate (the layout of the
// accumulator fragment; neighbouring candidates go to different lanes, which keeps the four lists of a
// row alike in length: contiguous quarters needed 1.6 times the rounds).
//
// What it does instead of the law on every candidate: only one in 3 (clustered) to 5 (uniform) of the
// pairs that pass the box test is within rc, and evaluating them all took 29 (uniform) and 39 (clustered)
// rounds of 64 per item, against 11 and 21 rounds of the listed ones (75 instructions each, 2300
// instead of 2950 and 3180 instead of 3610 instructions per item together with the staging).
// It issues on 82 % of the cycles; the lists of a batch differ in length, which idles a third of the
// pair slots.  192^3 boxes under ncu, before and after: uniform 1.67 to 1.18 ms, lognormal
// (sigma 1.5) 3.09 to 3.00 ms with 224 candidates a batch and 4 blocks per SM, 2.9 ms with 256 and 3.
__device__ __forceinline__ unsigned tf32_floor(float x) { return __float_as_uint(x) & 0xffffe000u; }
__device__ __forceinline__ unsigned tf32_rna(float x) {
  unsigned r;
  asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(r) : "f"(x));
  return r;
}
__device__ __forceinline__ void mma_tf32(float d[4], const unsigned a[4], unsigned b0, unsigned b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k8.row.col.f32.tf32.tf32.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};"
      : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1), "f"(0.f));
}
// index of the highest set bit (-1: none), and 1 << b (0 for b = -1)
__device__ __forceinline__ int high_bit(unsigned m) {
  int b;
  asm("bfind.u32 %0, %1;" : "=r"(b) : "r"(m));
  return b;
}
__device__ __forceinline__ unsigned bit_at(int b) {
  unsigned r;
  asm("shl.b32 %0, 1, %1;" : "=r"(r) : "r"(b));
  return r;
}
__device__ __forceinline__ float4 lds128(unsigned a) {
  float4 v;
  asm volatile("ld.shared.v4.f32 {%0,%1,%2,%3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(a));
  return v;
}
__device__ __forceinline__ float lds32(unsigned a) {
  float v;
  asm volatile("ld.shared.f32 %0, [%1];" : "=f"(v) : "r"(a));
  return v;
}

template <int C, int J, int U, int B>
__global__ void __launch_bounds__(kPPThreads, B) k_pp_pairs(PPK p) {
  static_assert(C <= 16 && J % 32 == 0 && J <= 256, "16 rows, two 32-bit lists a row and lane");
  extern __shared__ float4 pp_smem[];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  char *wbase = reinterpret_cast<char *>(pp_smem) + warp * pp_smem_warp(J, true);
  // staged candidates, relative to the box centre: x, y, z, |x|^2
  float4 *const buf = reinterpret_cast<float4 *>(wbase);
  const unsigned buf_s = (unsigned)__cvta_generic_to_shared(buf);
  float *const ks = reinterpret_cast<float *>(wbase + pp_stage_bytes(J)) + lane;  // field f at ks[32 f]
  PPItem *const batch = reinterpret_cast<PPItem *>(wbase + pp_stage_bytes(J) + sizeof(float) * 32 * kLaneFieldsPairs);
  uint64_t *const bar = reinterpret_cast<uint64_t *>(batch + kPop);
  uint32_t phase = 0u;
  bool ok = true;
  if (lane == 0) {
    mbar_init(bar, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  // ks fields: 0 f2, 1-3 |v| maxima, 4-6 velocity of the owned particle, 7-18 Kahan sums and compensations
  for (int q = lane; q < J + 32; q += 32) buf[q] = make_float4(0.f, 0.f, 0.f, 0.f);  // always finite
  for (int f = 0; f < 4; f++) ks[32 * f] = 0.f;
  __syncwarp();
  for (int nb = 0, b = 0;; b++) {
    if (b == nb) {
      // items [first, last) of tiles [t_lo, t_hi), popped through this launch's own queue head; one at
      // a time where the items are too few to keep every warp busy otherwise
      const int32_t *tbase = p.sched + sched_base(p.ntile);
      const int first = tbase[p.t_lo];
      const int last = (int)min((int64_t)tbase[p.t_hi], p.item_cap);
      const int pop = last - first >= 16 * (int)gridDim.x * kPPWarps ? kPop : 1;
      int it = 0;
      if (lane == 0) it = first + atomicAdd(p.sched + sched_head(p.ntile, p.t_lo, p.t_hi), pop);
      it = __shfl_sync(0xffffffffu, it, 0);
      if (it >= last) break;
      nb = min(pop, last - it);
      b = 0;
      __syncwarp();
      if (lane < 2 * nb) reinterpret_cast<int4 *>(batch)[lane] = reinterpret_cast<const int4 *>(p.items + it)[lane];
      __syncwarp();
    }
    const PPItem &item = batch[b];  // read from shared memory where used
    const int ni = item.dims & 0xff;
    // row r holds particle r mod n2, n2 the power of two from ni up; the 16 / n2 replicas of a particle
    // take every (16 / n2)-th bit of its lists
    const int n2 = ni > 8 ? 16 : (ni > 4 ? 8 : (ni > 2 ? 4 : ni));
    const int iA = g & (n2 - 1), iB = (g + 8) & (n2 - 1);
    const float4 pA = p.spos[item.i0 + min(iA, ni - 1)], pB = p.spos[item.i0 + min(iB, ni - 1)];
    // The stencil's rows (dy, dz), one lane each and 32 at a time: every row is a contiguous range of the
    // cell-sorted particles, and the rows laid end to end are the candidates of the pass.
    int js = 0, off = 0, walk = 0, r0 = 0;  // this lane's row: first particle, place in the pass; candidates of the pass
    const int R = (item.dims >> 16) & 0xff, side = 2 * R + 1, nr = side * side;
    auto load_rows = [&]() {
      const int ri = r0 + lane;
      int len = 0;
      if (ri < nr) {
        const int q = div_small(ri, side), dz = q - R, dy = ri - q * side - R;
        if (row_needed(dy, dz, item.h, item.rc2)) {
          const int S = ((item.dims >> 8) & 0xff) * (p.nt + 2);
          const int32_t *c = p.cs + ((int)item.cell + (dz * S + dy) * S);
          js = c[-R];
          len = c[R + 1 + (item.dims >> 24)] - js;
        }
      }
      int incl = len;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int v = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += v;
      }
      off = incl - len;
      walk = __shfl_sync(0xffffffffu, incl, 31);
      r0 += 32;
    };
    // Candidates [w, w + n) of the pass into buf[at ..): one bulk copy per row that has some of them
    // (16-byte entries, so every address and size is a multiple of 16).
    auto fetch = [&](int w, int n, int at) {
      const int next = __shfl_down_sync(0xffffffffu, off, 1), end = lane == 31 ? walk : next;
      const int lo = max(off, w), hi = min(end, w + n);
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");  // the warp's own accesses to buf come first
      __syncwarp();
      if (lane == 0) mbar_arrive_expect_tx(bar, (uint32_t)n * 16u);
      __syncwarp();
      if (hi > lo) bulk_g2s(buf + at + (lo - w), p.spos + js + (lo - off), (uint32_t)(hi - lo) * 16u, bar);
    };
    int w = 0, got = 0;  // candidates of the pass taken so far; those on their way
    auto request = [&](int room, int at) {  // the next candidates, at most `room` of them; got = 0: the item has no more
      while (w >= walk) {
        if (r0 >= nr) {
          got = 0;
          return;
        }
        load_rows();
        w = 0;
      }
      got = min(walk - w, room);
      fetch(w, got, at);
      w += got;
    };
    request(J, 0);
    // the lane that owns a particle: t = 0 the one of row g, t = 1 the one of row g + 8 (when they differ)
    const bool owner = (t == 0 && g < min(n2, ni)) || (t == 1 && n2 == 16 && g + 8 < ni);
    const int ip = __float_as_int(t == 1 ? pB.w : pA.w);
    if (owner) {  // the owned particle's velocity is copied in while the item runs
      const float *v = p.vp + 3 * (int64_t)ip;
      cp_async4(ks + 32 * 4, v);
      cp_async4(ks + 32 * 5, v + 1);
      cp_async4(ks + 32 * 6, v + 2);
    }
    cp_async_commit();
    // The box of the item's particles: centre and half sides.  Positions are multiples of 2^-17 fine cells
    // or coarser, so differences to the centre are exact, and so are the differences of two of them.
    const float lx = warp_min_redux(fminf(pA.x, pB.x)), hx = warp_max_redux(fmaxf(pA.x, pB.x)),
                ly = warp_min_redux(fminf(pA.y, pB.y)), hy = warp_max_redux(fmaxf(pA.y, pB.y)),
                lz = warp_min_redux(fminf(pA.z, pB.z)), hz = warp_max_redux(fmaxf(pA.z, pB.z));
    const float cx = 0.5f * (lx + hx), cy = 0.5f * (ly + hy), cz = 0.5f * (lz + hz);
    const float ax = fmaxf(hx - cx, cx - lx), ay = fmaxf(hy - cy, cy - ly), az = fmaxf(hz - cz, cz - lz);
    const float xA = pA.x - cx, yA = pA.y - cy, zA = pA.z - cz;
    const float xB = pB.x - cx, yB = pB.y - cy, zB = pB.z - cz;
    // The rows' operand of the filter.  T: rc^2 and the error bound of the product for |x| <= a, |x'| <= m =
    // a + rc per axis: the rows' values are rounded to 2^-11, the candidates' cut at 2^-10, so at most
    // 1.5 2^-10 of 2 a m per axis, and 2^-10 of |x'|^2; 5 % and 2e-5 rc^2 cover the FP32 accumulation and
    // the split of |x|^2 - T.
    unsigned fa[4];
    {
      const float rc = item.rc, mx = ax + rc, my = ay + rc, mz = az + rc;
      const float T = item.rc2 * 1.00002f +
                      1.025e-3f * (3.0f * (ax * mx + ay * my + az * mz) + mx * mx + my * my + mz * mz);
      const float nA = iA < ni ? fmaf(xA, xA, fmaf(yA, yA, zA * zA)) - T : 1e30f;
      const float nB = iB < ni ? fmaf(xB, xB, fmaf(yB, yB, zB * zB)) - T : 1e30f;
      const unsigned hA = tf32_floor(nA), hB = tf32_floor(nB);
      fa[0] = tf32_rna(t == 0 ? -2.0f * xA : (t == 1 ? -2.0f * yA : (t == 2 ? -2.0f * zA : 1.0f)));
      fa[1] = tf32_rna(t == 0 ? -2.0f * xB : (t == 1 ? -2.0f * yB : (t == 2 ? -2.0f * zB : 1.0f)));
      fa[2] = t == 0 ? hA : (t == 1 ? tf32_floor(nA - __uint_as_float(hA)) : 0u);
      fa[3] = t == 0 ? hB : (t == 1 ? tf32_floor(nB - __uint_as_float(hB)) : 0u);
    }
    int nflush = 0;
    float2 px = dup(0.f), py = dup(0.f), pz = dup(0.f);
    while (got) {
      int nbuf = 0;  // staged candidates
      // Candidates farther than rc from the item's box are dropped, in place: what is kept never passes what
      // has been read.  More are fetched while there is room for a good part of a buffer.
      do {
        if (!mbar_wait_bounded(bar, phase)) {
          ok = false;
          break;
        }
        phase ^= 1u;
        const int first = nbuf;
        for (int v = lane; v - lane < got; v += 32) {
          const float4 pj = buf[first + v];
          const float qx = pj.x - cx, qy = pj.y - cy, qz = pj.z - cz;
          const float ex = fmaxf(fabsf(qx) - ax, 0.f), ey = fmaxf(fabsf(qy) - ay, 0.f), ez = fmaxf(fabsf(qz) - az, 0.f);
          const bool in = (v < got) & (fmaf(ex, ex, fmaf(ey, ey, ez * ez)) <= item.rc2);
          const unsigned m = __ballot_sync(0xffffffffu, in);
          if (in) buf[nbuf + __popc(m & ((1u << lane) - 1u))] = make_float4(qx, qy, qz, fmaf(qx, qx, fmaf(qy, qy, qz * qz)));
          nbuf += __popc(m);
        }
        const bool full = nbuf > J - kRefill;
        if (full && (w < walk || r0 < nr)) break;
        request(J - nbuf, nbuf);
      } while (got);
      if (!ok) break;
      // ---- filter: candidate 4 o + t is bit o (from the top) of lane (g, t)'s lists; a step of 8
      // candidates adds two bits to each list
      // padding that no row lists; the four candidates after the last step are what an empty list reads
      if (lane < 16) buf[nbuf + lane] = make_float4(kFar, kFar, kFar, 1e30f);
      __syncwarp();
      const int ns = (nbuf + 7) >> 3, c0 = min(ns, 16);
      unsigned mA0 = 0u, mB0 = 0u, mA1 = 0u, mB1 = 0u;
      {
        unsigned sb = buf_s + (unsigned)((4 * (g & 1) + (g >> 1)) * 16 + t * 4);
        auto filter = [&](int n, unsigned &mA, unsigned &mB) {
#pragma unroll U
          for (int s = 0; s < n; s++, sb += 128) {
            float d[4];
            mma_tf32(d, fa, tf32_floor(lds32(sb)), __float_as_uint(1.0f));
            mA = __funnelshift_l(__float_as_uint(d[0]), mA, 1);
            mA = __funnelshift_l(__float_as_uint(d[1]), mA, 1);
            mB = __funnelshift_l(__float_as_uint(d[2]), mB, 1);
            mB = __funnelshift_l(__float_as_uint(d[3]), mB, 1);
          }
        };
        filter(c0, mA0, mB0);
        filter(ns - c0, mA1, mB1);
      }
      if (n2 < 16) {
        const unsigned every = n2 == 8 ? 0x55555555u : (n2 == 4 ? 0x11111111u : (n2 == 2 ? 0x01010101u : 0x00010001u));
        const unsigned patA = every << (g / n2), patB = every << ((g + 8) / n2);
        mA0 &= patA;
        mA1 &= patA;
        mB0 &= patB;
        mB1 &= patB;
      }
      const int rounds = __reduce_max_sync(0xffffffffu, max(__popc(mA0) + __popc(mA1), __popc(mB0) + __popc(mB1)));
      // ---- pairs: bit b of the first list is o = 2 c0 - 1 - b, of the second o = 2 ns - 1 - b
      unsigned offA = buf_s + (unsigned)(4 * (2 * c0 - 1) + t) * 16u, offB = offA;
      const unsigned off1 = buf_s + (unsigned)(4 * (2 * ns - 1) + t) * 16u;
      px = py = pz = dup(0.f);
      PairLaw law;
      law.init(item);
      for (int r = 0; r < rounds; r++) {
        if (mA0 == 0u) {
          mA0 = mA1;
          mA1 = 0u;
          offA = off1;
        }
        if (mB0 == 0u) {
          mB0 = mB1;
          mB1 = 0u;
          offB = off1;
        }
        const int bA = high_bit(mA0), bB = high_bit(mB0);
        const float4 cA = lds128(offA - (unsigned)(bA * 64)), cB = lds128(offB - (unsigned)(bB * 64));
        mA0 ^= bit_at(bA);
        mB0 ^= bit_at(bB);
        const float2 dx = make_float2(cA.x - xA, cB.x - xB), dy = make_float2(cA.y - yA, cB.y - yB),
                     dz = make_float2(cA.z - zA, cB.z - zB);
        const float2 r2 = fma2(dx, dx, fma2(dy, dy, mul2(dz, dz)));
        float2 s = law.scale2(r2);
        const bool fA = r2.x > p.app2, fB = r2.y > p.app2;
        s.x = fA ? s.x : 0.0f;
        s.y = fB ? s.y : 0.0f;
        // inside the softening length (rare): both terms directly; r = 0 is the particle itself
        const bool sA = !fA & (r2.x > 0.0f), sB = !fB & (r2.y > 0.0f);
        if (sA | sB) {
          if (sA) s.x = law.soft(r2.x, p.cea, p.ka);
          if (sB) s.y = law.soft(r2.y, p.cea, p.ka);
        }
        px = fma2(s, dx, px);
        py = fma2(s, dy, py);
        pz = fma2(s, dz, pz);
      }
      nflush++;
      __syncwarp();
      const bool more = w < walk || r0 < nr;
      // compensated sums over the flushes of an item that needs several
      if (nflush > 1 || more) {
        const float v[6] = {px.x, py.x, pz.x, px.y, py.y, pz.y};
#pragma unroll
        for (int f = 0; f < 6; f++) {
          if (nflush == 1) {
            ks[32 * (7 + 2 * f)] = v[f];
            ks[32 * (8 + 2 * f)] = 0.f;
          } else {
            kahan_add(ks[32 * (7 + 2 * f)], ks[32 * (8 + 2 * f)], v[f]);
          }
        }
      }
      if (more) request(J, 0);
      else got = 0;
    }
    if (!ok) break;
    // (hi, lo) per half; Kahan c is the negated low part
    float hi[6] = {px.x, py.x, pz.x, px.y, py.y, pz.y}, lo[6] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
    if (nflush > 1) {
#pragma unroll
      for (int f = 0; f < 6; f++) {
        hi[f] = ks[32 * (7 + 2 * f)];
        lo[f] = -ks[32 * (8 + 2 * f)];
      }
    }
    // Sum over the four lanes of a row: lanes of even t keep row g, those of odd t row g + 8, then the
    // two of a row are joined
    float H[3], Lo[3];
#pragma unroll
    for (int f = 0; f < 3; f++) {
      const bool odd = t & 1;
      const float sh = __shfl_xor_sync(0xffffffffu, odd ? hi[f] : hi[3 + f], 1),
                  sl = __shfl_xor_sync(0xffffffffu, odd ? lo[f] : lo[3 + f], 1);
      H[f] = odd ? hi[3 + f] : hi[f];
      Lo[f] = odd ? lo[3 + f] : lo[f];
      two_sum_merge(H[f], Lo[f], sh, sl);
    }
    auto join = [&](int d) {
#pragma unroll
      for (int f = 0; f < 3; f++) {
        const float sh = __shfl_xor_sync(0xffffffffu, H[f], d), sl = __shfl_xor_sync(0xffffffffu, Lo[f], d);
        two_sum_merge(H[f], Lo[f], sh, sl);
      }
    };
    join(2);
    if (n2 < 16) {  // the replicas of a particle: row g + 8, and every n2-th row
      join(1);
      for (int d = 4 * n2; d < 32; d <<= 1) join(d);
    }
    if (owner) {
      const float fx = (H[0] + Lo[0]) * p.mass2, fy = (H[1] + Lo[1]) * p.mass2, fz = (H[2] + Lo[2]) * p.mass2;
      ks[0] = fmaxf(ks[0], fx * fx + fy * fy + fz * fz);
      float *v = p.vp + 3 * (int64_t)ip;
      cp_async_wait_all();
      const float v0 = ks[32 * 4] + fx * p.kick, v1 = ks[32 * 5] + fy * p.kick, v2 = ks[32 * 6] + fz * p.kick;
      v[0] = v0;
      v[1] = v1;
      v[2] = v2;
      ks[32] = fmaxf(ks[32], fabsf(v0));
      ks[64] = fmaxf(ks[64], fabsf(v1));
      ks[96] = fmaxf(ks[96], fabsf(v2));
    }
    __syncwarp();
  }
  if (!ok) {  // a copy did not arrive in time: once more (also bounded), so that none is left behind
    if (lane == 0) atomicOr(p.err, 1 << CUBE_ERR_TIMEOUT);
    (void)mbar_wait_bounded(bar, phase);
    cp_async_wait_all();
  }
  const float f2w = warp_max(ks[0]);
  if (lane == 0) atomic_max_nonneg(&p.out[1], f2w);
  if (p.want_vmax) {
    const float vm0 = warp_max(ks[32]), vm1 = warp_max(ks[64]), vm2 = warp_max(ks[96]);
    if (lane == 0) {
      atomic_max_nonneg(&p.out[2], vm0);
      atomic_max_nonneg(&p.out[3], vm1);
      atomic_max_nonneg(&p.out[4], vm2);
    }
  }
}

static PPK make_ppk(const PPArgs &a) {
  const Lay &L = *a.L;
  PPK p;
  p.nt = L.nt;
  p.ntt = L.ntt;
  p.nns = L.nns;
  p.nnt = L.nnt;
  p.ntile = L.ntile;
  p.rcs = L.rcs;
  p.tiles = a.d_tiles;
  p.cs = a.cell_start;
  p.spos = a.spos;
  p.range_loc = a.range_loc;
  p.items = a.items;
  p.sched = a.sched;
  p.item_cap = a.item_cap;
  p.t_lo = 0;
  p.t_hi = L.ntile;
  p.vp = a.vp;
  p.mass2 = a.mass2;
  p.kick = a.kick;
  p.app = L.app;
  p.app2 = L.app * L.app;
  p.cea = L.app > 0.f ? 2.0f / L.app : 0.f;
  p.ka = L.app > 0.f ? (1.0f / 35.0f) / (L.app * L.app) : 0.f;
  p.out = a.out;
  p.want_vmax = a.want_vmax;
  p.err = a.err;
  p.pairs = a.pairs;
  int max_rcp = 1;
  for (int t = 0; t < L.ntile; t++) max_rcp = a.h_tiles[t].rcp > max_rcp ? a.h_tiles[t].rcp : max_rcp;
  const int64_t npg = (int64_t)L.nt * max_rcp;
  p.max_cells = npg * npg * npg;
  return p;
}

size_t sched_ints(int ntile) { return (size_t)sched_base(ntile) + 2 * ((size_t)ntile + 1); }
int64_t sched_total_index(int ntile) { return sched_base(ntile) + ntile; }

int pp_num_shapes() { return kNumShapes; }
PPShapeDesc pp_shape_desc(int i) { return kShapes[i >= 0 && i < kNumShapes ? i : 0]; }
int pp_min_chunk() { return kMinChunk; }

template <int C>
static void launch_items_c(const PPK &p, dim3 grid, cudaStream_t s, int32_t *sched, int ntile) {
  k_pp_items<0, C><<<grid, 256, 0, s>>>(p);
  k_pp_offsets<<<1, 32, 0, s>>>(sched, ntile);
  k_pp_items<1, C><<<grid, 256, 0, s>>>(p);
}

void launch_pp_items(const PPArgs &a, cudaStream_t s, bool zeroed) {
  PPK p = make_ppk(a);
  if (!zeroed) cudaMemsetAsync(a.sched, 0, sizeof(int32_t) * sched_ints(a.L->ntile), s);
  dim3 grid((unsigned)((p.max_cells + 255) / 256), (unsigned)a.L->ntile);
  switch (pp_shape_desc(a.pairs ? 0 : a.shape).chunk) {
    case 16: launch_items_c<16>(p, grid, s, a.sched, a.L->ntile); break;
    case 32: launch_items_c<32>(p, grid, s, a.sched, a.L->ntile); break;
    default: launch_items_c<8>(p, grid, s, a.sched, a.L->ntile); break;
  }
}

// One persistent block per resident slot: blocks beyond the resident count would only start
// once the queue is empty.  The shared-memory attribute is set and the count looked up once per
// kernel (slot = shape, or the pair-count kernel) and device: the attribute is per device.
constexpr int kMaxDevices = 64;
template <bool COUNT, int S>
static auto force_kernel() {
  constexpr PPShapeDesc d = COUNT ? kCountShape : kShapes[S];
  if constexpr (d.packed != 0) return k_pp_pairs<d.chunk, d.jtile, d.unroll, d.blocks>;
  else return k_pp_force<COUNT, d.chunk, d.jtile, d.unroll, d.blocks>;
}

template <bool COUNT, int S>
static void launch_force_shape(const PPK &p, int num_sms, cudaStream_t s) {
  constexpr PPShapeDesc d = COUNT ? kCountShape : kShapes[S];
  constexpr size_t smem = pp_smem_block(d.jtile, d.packed != 0);
  auto fn = force_kernel<COUNT, S>();
  static int per_sm[kMaxDevices] = {};
  int dev = 0;
  cudaGetDevice(&dev);
  int n = 0;
  if (dev < 0 || dev >= kMaxDevices || !per_sm[dev]) {
    cudaFuncSetAttribute((const void *)fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, (const void *)fn, kPPThreads, smem);
    n = n > 0 ? n : 1;
    if (dev >= 0 && dev < kMaxDevices) per_sm[dev] = n;
  } else {
    n = per_sm[dev];
  }
  fn<<<n * num_sms, kPPThreads, smem, s>>>(p);
}

template <int... I>
static void launch_force_any(int shape, const PPK &p, int num_sms, cudaStream_t s, std::integer_sequence<int, I...>) {
  ((shape == I ? launch_force_shape<false, I>(p, num_sms, s) : void()), ...);
}

void launch_pp_force(const PPArgs &a, cudaStream_t s, int t_lo, int t_hi) {
  PPK p = make_ppk(a);
  if (t_hi < 0) t_hi = a.L->ntile;
  p.t_lo = t_lo;
  p.t_hi = t_hi;
  if (a.pairs) {
    launch_force_shape<true, 0>(p, a.num_sms, s);  // kCountShape: the work list of shape 0
  } else {
    const int shape = a.shape >= 0 && a.shape < kNumShapes ? a.shape : 0;
    launch_force_any(shape, p, a.num_sms, s, std::make_integer_sequence<int, kNumShapes>{});
  }
}

}  // namespace cube

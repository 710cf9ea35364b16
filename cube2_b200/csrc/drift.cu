// Drift of one periodic image and the rebuild of its buffers on the device:
// drift.f90:1-161 (fixed-point drift, re-binning by coarse cell, compaction) followed by
// buffer_grid.f90:13-155 and buffer_particle.f90:23-345 (periodic buffer cells, which
// hold copies of the particles of the physical cells they mirror).
//
// The reference visits each tile's stored copies (physical and buffer) layer by layer
// (source row k modulo nlayer), then in storage order, and appends every copy that lands
// in the tile's physical region to its destination cell (drift.f90:94-118).  The order
// inside a destination cell is thus by (ilayer of the source row, storage index), and
// every destination's particles come from a few nearby source cells of one tile.  Here:
//
//   k_drift_runs   warp per source cell: the destination of each copy; the copies of the
//                  cell that share a destination form a run (at most 64 per source cell),
//                  and each copy gets its rank inside its run (warp ballots, in storage
//                  order); runs go to a flat table with the reference's visiting key.
//   k_ext_counts   new counts of every extended cell (buffer cells mirror physical ones),
//   k_row_sums,
//   k_scan_rows    and the new spine idx_b_r (one inclusive scan over the rows).
//   k_runs_fill    runs grouped by destination cell (counting sort on the destination),
//   k_runs_order   and each run's first slot: the destination cell's start plus the
//                  particles of the runs with a smaller key (runs per cell are few).
//   k_drift_write  warp per source cell again: every kept copy writes its new offset
//                  (xp + nint(dt vp / (x_res ratio_cs)), int16 wrap), vp and pid to its slot.
//   k_halo_fill    warp per buffer cell: copy of the mirrored physical cell.
//
// Everything is linear in the particles and deterministic (no order depends on atomics).
#include "common.cuh"

namespace cube {

struct DriftRun {
  int32_t dest;   // physical coarse cell of the image, (z * nc + y) * nc + x
  int32_t count;  // copies of the source cell that land there
  uint64_t key;   // ilayer(source row) << 32 | source cell: the reference's visiting order
};

constexpr int kDriftMaxRuns = 64;    // destination cells of one source cell
constexpr int kRankBits = 26;        // run slot word: entry << 26 | rank inside the run
constexpr uint32_t kDropped = 0xffffffffu;
constexpr int kDriftWarps = 8;
// Run-table slots are reserved per warp kRunChunk at a time (one atomic per chunk instead of
// one per source cell on a single counter); the unused end of a chunk holds dest = -1.
constexpr int kRunChunk = 64;
static_assert(kRunChunk >= kDriftMaxRuns, "a cell's runs fit one chunk");
constexpr int kDriftGridPerSM = 16;  // blocks per SM of the warp-per-cell kernels (at most)

struct DriftK {
  int nt, ncb, nte, nnt, nc, nlayer, tile_periodic;
  int64_t ncells_src;  // ntile * nte^3 extended cells
  int64_t n_used, n_used_new;  // stored copies of the current / new image (bounds of the spines)
  float dt_mid, rcs_f;
  double xres_rcs;     // x_resolution * ratio_cs
  float inv_rcs;       // 1 / ratio_cs where that is a power of two (then a product is the quotient bit for bit), else 0
  double inv_xres_rcs;
  const int32_t *rhoc;
  const int64_t *cell_base;
  const int16_t *xp;
  const float *vp;
  const int64_t *pid;
  uint32_t *runrank;     // [n_used] run slot word of each stored copy
  int32_t *run_base;     // [ncells_src] first run of each source cell
  DriftRun *runs;
  int32_t run_cap;
  int32_t *ctr;          // [0] runs, [1] kept copies
  int32_t *dest_runs;    // [nc^3] runs per destination
  int32_t *phys_count;   // [nc^3] particles per destination
  int32_t *err;
  // second half
  const int32_t *dest_start;  // [nc^3 + 1]
  int32_t *cursor;            // [nc^3]
  int32_t *run_list;          // [runs] grouped by destination
  int64_t *run_off;           // [runs] first slot of each run
  const int64_t *cell_base_new;
  int16_t *xp_new;
  float *vp_new;
  int64_t *pid_new;
};

// 32-bit arithmetic: the images have fewer than 2^31 extended cells, and a 64-bit division is a long software
// sequence that every warp would run for each of its cells (k_halo_fill took 73 us on 256^3, most of it this)
__device__ __forceinline__ void cell_of(const DriftK &p, int64_t S, int &t, int &cx, int &cy, int &cz) {
  const unsigned n = (unsigned)p.nte, q = (unsigned)S / n, qq = q / n;
  cx = (int)((unsigned)S - q * n);
  cy = (int)(q - qq * n);
  t = (int)(qq / n);
  cz = (int)(qq - (unsigned)t * n);
}

// drift.f90:57-66: destination of a stored copy, or -1 when it leaves the tile's physical
// region.  xq = (i-1) + (u+0.5) 2^-16 is exact in double; deltax = (dt_mid*vp)/ratio_cs
// in float; ig = ceiling(xq + deltax) in [1, nt] <=> 0 < xq + deltax <= nt.
struct DriftCell {
  int c[3];  // coarse coordinates in the tile, -ncb .. nt + ncb - 1
  int o[3];  // image coordinates of the tile's first physical cell
};
__device__ __forceinline__ DriftCell drift_cell(const DriftK &p, int64_t S, int &cz) {
  DriftCell q;
  int t, cx, cy;
  cell_of(p, S, t, cx, cy, cz);
  const int ty = t / p.nnt, tz = ty / p.nnt;
  q.c[0] = cx - p.ncb;
  q.c[1] = cy - p.ncb;
  q.c[2] = cz - p.ncb;
  q.o[0] = (t - ty * p.nnt) * p.nt;
  q.o[1] = (ty - tz * p.nnt) * p.nt;
  q.o[2] = tz * p.nt;
  return q;
}
__device__ __forceinline__ int32_t drift_dest(const DriftK &p, int64_t ip, const DriftCell &q) {
  int g[3];
  float v[3];
  uint16_t u[3];
#pragma unroll
  for (int d = 0; d < 3; d++) {
    v[d] = p.vp[3 * ip + d];
    u[d] = (uint16_t)p.xp[3 * ip + d];
  }
  bool in = true;
#pragma unroll
  for (int d = 0; d < 3; d++) {
    const double xq = (double)q.c[d] + ((double)u[d] + 0.5) * (1.0 / 65536.0);
    const float dv = __fmul_rn(p.dt_mid, v[d]);
    const float dl = p.inv_rcs != 0.f ? __fmul_rn(dv, p.inv_rcs) : __fdiv_rn(dv, p.rcs_f);
    const double s = __dadd_rn(xq, (double)dl);
    in = in && s > 0.0 && s <= (double)p.nt;
    g[d] = q.o[d] + (in ? __double2int_ru(s) - 1 : 0);
  }
  return in ? (g[2] * p.nc + g[1]) * p.nc + g[0] : -1;
}

__global__ void __launch_bounds__(kDriftWarps * 32) k_drift_runs(DriftK p) {
  __shared__ int32_t s_dest[kDriftWarps][kDriftMaxRuns];
  __shared__ int32_t s_cnt[kDriftWarps][kDriftMaxRuns];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  int32_t *td = s_dest[warp], *tc = s_cnt[warp];
  const unsigned lt = (1u << lane) - 1u;
  const int64_t stride = (int64_t)gridDim.x * kDriftWarps;
  int64_t S = (int64_t)blockIdx.x * kDriftWarps + warp;
  // the count and first slot of the next cell are loaded one cell ahead
  int n_next = S < p.ncells_src ? p.rhoc[S] : 0;
  int64_t base_next = S < p.ncells_src ? p.cell_base[S] : 0;
  int cur = 0, end = 0;  // this warp's reserved run slots [cur, end)
  int kept_w = 0;        // kept copies counted by this lane
  auto close_chunk = [&]() {
    for (int e = cur + lane; e < end; e += 32)
      if (e < p.run_cap) p.runs[e].dest = -1;
  };
  for (; S < p.ncells_src; S += stride) {
    const int n = n_next;
    const int64_t base = base_next;
    if (S + stride < p.ncells_src) {
      n_next = p.rhoc[S + stride];
      base_next = p.cell_base[S + stride];
    }
    if (n <= 0) continue;
    if (n >= (1 << kRankBits) - 1) {  // the rank field holds ranks below 2^26 - 1
      if (lane == 0) atomicOr(p.err, 1 << CUBE_ERR_CAPACITY);
      continue;
    }
    if (base < 0 || base + n > p.n_used) {  // the spine does not match the counts
      if (lane == 0) atomicOr(p.err, 1 << CUBE_ERR_INVALID);
      continue;
    }
    int cz;
    const DriftCell cell = drift_cell(p, S, cz);
    int nent = 0;  // warp-uniform
    // most copies stay in their own cell: its run is counted in registers, without the search
    const bool phys = cell.c[0] >= 0 && cell.c[0] < p.nt && cell.c[1] >= 0 && cell.c[1] < p.nt && cell.c[2] >= 0 &&
                      cell.c[2] < p.nt;
    const int32_t home =
        phys ? ((cell.o[2] + cell.c[2]) * p.nc + cell.o[1] + cell.c[1]) * p.nc + cell.o[0] + cell.c[0] : -2;
    int ehome = -1, nhome = 0;  // entry and copies of that run
    // 64 copies per step: the loads of both halves are in flight together
    for (int c64 = 0; c64 < n; c64 += 64) {
    const int32_t D2[2] = {c64 + lane < n ? drift_dest(p, base + c64 + lane, cell) : -1,
                           c64 + 32 + lane < n ? drift_dest(p, base + c64 + 32 + lane, cell) : -1};
    for (int h = 0; h < 2 && c64 + 32 * h < n; h++) {
      const int c0 = c64 + 32 * h;
      const int l = c0 + lane;
      const int32_t D = D2[h];
      uint32_t word = kDropped;
      const unsigned hm = __ballot_sync(0xffffffffu, D == home);
      if (hm && ehome < 0) {
        if (nent < kDriftMaxRuns) {
          ehome = nent++;
          if (lane == 0) td[ehome] = home;
          __syncwarp();
        } else if (lane == 0) {
          atomicOr(p.err, 1 << CUBE_ERR_CAPACITY);
        }
      }
      if (ehome >= 0 && D == home) word = ((uint32_t)ehome << kRankBits) | (uint32_t)(nhome + __popc(hm & lt));
      nhome += __popc(hm);
      unsigned pending = __ballot_sync(0xffffffffu, D >= 0) & ~hm;
      while (pending) {
        const int32_t Dl = __shfl_sync(0xffffffffu, D, __ffs(pending) - 1);
        const unsigned grp = __ballot_sync(0xffffffffu, D == Dl);
        const unsigned h0 = __ballot_sync(0xffffffffu, lane < nent && td[lane] == Dl);
        const unsigned h1 = __ballot_sync(0xffffffffu, lane + 32 < nent && td[lane + 32] == Dl);
        int e = h0 ? __ffs(h0) - 1 : (h1 ? 31 + __ffs(h1) : -1);
        if (e < 0 && nent < kDriftMaxRuns) {
          e = nent++;
          if (lane == 0) {
            td[e] = Dl;
            tc[e] = 0;
          }
          __syncwarp();
        }
        if (e >= 0) {
          const int prior = tc[e];
          if ((grp >> lane) & 1u) word = ((uint32_t)e << kRankBits) | (uint32_t)(prior + __popc(grp & lt));
          __syncwarp();
          if (lane == 0) tc[e] = prior + __popc(grp);
          __syncwarp();
        } else if (lane == 0) {
          atomicOr(p.err, 1 << CUBE_ERR_CAPACITY);  // more than kDriftMaxRuns destinations
        }
        pending &= ~grp;
      }
      if (l < n) p.runrank[base + l] = word;
    }
    }
    if (ehome >= 0) {
      if (lane == 0) tc[ehome] = nhome;
      __syncwarp();
    }
    if (nent) {
      if (cur + nent > end) {  // a new chunk of run slots
        close_chunk();
        int c = 0;
        if (lane == 0) c = atomicAdd(&p.ctr[0], kRunChunk);
        cur = __shfl_sync(0xffffffffu, c, 0);
        end = cur + kRunChunk;
      }
      const int rb = cur;
      cur += nent;
      if (lane == 0) p.run_base[S] = rb;
      const uint64_t key = ((uint64_t)(cz % p.nlayer) << 32) | (uint64_t)S;
      int kept = 0;
      for (int e = lane; e < nent; e += 32) {
        if (rb + e < p.run_cap) {
          DriftRun r;
          r.dest = td[e];
          r.count = tc[e];
          r.key = key;
          p.runs[rb + e] = r;
          atomicAdd(&p.dest_runs[r.dest], 1);
          atomicAdd(&p.phys_count[r.dest], r.count);
          kept += r.count;
        } else {
          atomicOr(p.err, 1 << CUBE_ERR_CAPACITY);
        }
      }
      kept_w += kept;
      __syncwarp();  // the table is reused by the next cell
    }
  }
  close_chunk();
  kept_w = __reduce_add_sync(0xffffffffu, kept_w);
  if (lane == 0 && kept_w) atomicAdd(&p.ctr[1], kept_w);
}

// physical cell mirrored by extended cell (t, cx, cy, cz): the image's periodic neighbour
// (buffer_grid.f90:22-40), or the tile's own periodic image for independent periodic tiles; as tile
// and local coordinates
__device__ __forceinline__ void mirrored_cell(const DriftK &p, int t, int cx, int cy, int cz, int tt[3], int l[3]) {
  const int ty = t / p.nnt, tz = ty / p.nnt;
  tt[0] = t - ty * p.nnt;
  tt[1] = ty - tz * p.nnt;
  tt[2] = tz;
  l[0] = cx - p.ncb;
  l[1] = cy - p.ncb;
  l[2] = cz - p.ncb;
#pragma unroll
  for (int d = 0; d < 3; d++) {
    int w = 0;
    while (l[d] < 0) l[d] += p.nt, w--;
    while (l[d] >= p.nt) l[d] -= p.nt, w++;
    if (!p.tile_periodic) {
      tt[d] += w;
      while (tt[d] < 0) tt[d] += p.nnt;
      while (tt[d] >= p.nnt) tt[d] -= p.nnt;
    }
  }
}

// extended cell index of a physical cell in the tile that owns it
__device__ __forceinline__ int64_t ext_cell(const DriftK &p, const int tt[3], const int l[3]) {
  const int t = (tt[2] * p.nnt + tt[1]) * p.nnt + tt[0];
  return (((int64_t)t * p.nte + l[2] + p.ncb) * p.nte + l[1] + p.ncb) * p.nte + l[0] + p.ncb;
}
__device__ __forceinline__ int64_t owner_ext_cell(const DriftK &p, int32_t G) {
  const int gy = G / p.nc, gz = gy / p.nc, g[3] = {G - gy * p.nc, gy - gz * p.nc, gz};
  int tt[3], l[3];
#pragma unroll
  for (int d = 0; d < 3; d++) {
    tt[d] = g[d] / p.nt;
    l[d] = g[d] - tt[d] * p.nt;
  }
  return ext_cell(p, tt, l);
}

__global__ void k_ext_counts(DriftK p, const int32_t *phys_count, int32_t *rhoc_new) {
  const int64_t E = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (E >= p.ncells_src) return;
  int t, cx, cy, cz, tt[3], l[3];
  cell_of(p, E, t, cx, cy, cz);
  mirrored_cell(p, t, cx, cy, cz, tt, l);
  rhoc_new[E] = phys_count[((tt[2] * p.nt + l[2]) * p.nc + tt[1] * p.nt + l[1]) * p.nc + tt[0] * p.nt + l[0]];
}

__global__ void k_row_sums(const int32_t *rhoc, int64_t nrows, int nte, int64_t *rows) {
  const int64_t r = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (r >= nrows) return;
  int64_t s = 0;
  for (int i = 0; i < nte; i++) s += rhoc[r * nte + i];
  rows[r] = s;
}

// inclusive scan of the row sums (one block): the spine idx_b_r (variables.f90:184-195)
__global__ void __launch_bounds__(1024) k_scan_rows(const int64_t *rows, int64_t nrows, int64_t *idx_b_r,
                                                    int64_t *total) {
  __shared__ int64_t ws[32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  int64_t carry = 0;
  for (int64_t r0 = 0; r0 < nrows; r0 += 1024) {
    const int64_t r = r0 + threadIdx.x;
    int64_t x = r < nrows ? rows[r] : 0;
    for (int o = 1; o < 32; o <<= 1) {
      const int64_t y = __shfl_up_sync(0xffffffffu, x, o);
      if (lane >= o) x += y;
    }
    if (lane == 31) ws[warp] = x;
    __syncthreads();
    if (warp == 0) {
      int64_t w = ws[lane];
      for (int o = 1; o < 32; o <<= 1) {
        const int64_t y = __shfl_up_sync(0xffffffffu, w, o);
        if (lane >= o) w += y;
      }
      ws[lane] = w;
    }
    __syncthreads();
    const int64_t incl = x + (warp ? ws[warp - 1] : 0) + carry;
    if (r < nrows) idx_b_r[r] = incl;
    carry += ws[31];
    __syncthreads();
  }
  if (threadIdx.x == 0) *total = carry;
}

__global__ void k_runs_fill(DriftK p, int32_t nruns) {
  const int32_t r = blockIdx.x * blockDim.x + threadIdx.x;
  if (r >= nruns) return;
  const int32_t D = p.runs[r].dest;
  if (D < 0) return;  // an unused slot at the end of a warp's chunk
  const int32_t slot = atomicAdd(&p.cursor[D], 1);
  p.run_list[p.dest_start[D] + slot] = r;
}

// eight lanes per destination cell (it has few runs: its own and those of the neighbours that send copies): first
// slot of each of its runs = the cell's start plus the particles of its runs with a smaller visiting key
__global__ void __launch_bounds__(kDriftWarps * 32) k_runs_order(DriftK p) {
  constexpr int kSub = 8;
  const int sub = threadIdx.x % kSub;
  const int64_t ndest = (int64_t)p.nc * p.nc * p.nc, stride = (int64_t)gridDim.x * blockDim.x / kSub;
  const int64_t d0 = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) / kSub;
  for (int64_t it = 0; it < (ndest + stride - 1) / stride; it++) {  // the same for all lanes: the shuffles need the warp
    const int64_t D = d0 + it * stride;
    int s0 = 0, m = 0;
    int64_t start = 0;
    if (D < ndest) {
      s0 = p.dest_start[D];
      m = p.dest_start[D + 1] - s0;
      if (m) start = p.cell_base_new[owner_ext_cell(p, (int32_t)D)];
    }
    const int r = sub < m ? p.run_list[s0 + sub] : 0;
    DriftRun o;
    o.key = ~0ull;
    o.count = 0;
    if (sub < m) o = p.runs[r];
    int off = 0;
#pragma unroll
    for (int j = 0; j < kSub; j++) {
      const uint64_t kj = __shfl_sync(0xffffffffu, o.key, j, kSub);
      const int cj = __shfl_sync(0xffffffffu, o.count, j, kSub);
      off += kj < o.key ? cj : 0;
    }
    if (m <= kSub) {
      if (sub < m) p.run_off[r] = start + off;
      continue;
    }
    for (int i = sub; i < m; i += kSub) {
      const int32_t ri = p.run_list[s0 + i];
      const uint64_t key = p.runs[ri].key;
      int64_t sum = 0;
      for (int j = 0; j < m; j++) {
        const DriftRun q = p.runs[p.run_list[s0 + j]];
        sum += q.key < key ? q.count : 0;
      }
      p.run_off[ri] = start + sum;
    }
  }
}

// drift.f90:111: xp + nint(dt_mid*vp / (x_resolution*ratio_cs)), stored in int16 (wraps)
__device__ __forceinline__ int16_t drift_offset(const DriftK &p, int16_t x, float v, int32_t *err) {
  const double dv = (double)__fmul_rn(p.dt_mid, v);
  const double q = p.inv_rcs != 0.f ? __dmul_rn(dv, p.inv_xres_rcs) : __ddiv_rn(dv, p.xres_rcs);
  if (!(fabs(q) < 2147483647.0)) {  // nint beyond the default integer: undefined in the reference
    atomicOr(err, 1 << CUBE_ERR_INVALID);
    return x;
  }
  // nint: half away from zero.  The product form has at most 24 bits, so q +- 0.5 is exact
  const int n = p.inv_rcs != 0.f ? __double2int_rz(q + copysign(0.5, q)) : (int)llround(q);
  return (int16_t)(uint16_t)((uint32_t)(int32_t)x + (uint32_t)n);
}

__global__ void __launch_bounds__(kDriftWarps * 32) k_drift_write(DriftK p) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int64_t stride = (int64_t)gridDim.x * kDriftWarps;
  int64_t S = (int64_t)blockIdx.x * kDriftWarps + warp;
  int n_next = S < p.ncells_src ? p.rhoc[S] : 0;
  int64_t base_next = S < p.ncells_src ? p.cell_base[S] : 0;
  for (; S < p.ncells_src; S += stride) {
    const int n = n_next;
    const int64_t base = base_next;
    if (S + stride < p.ncells_src) {
      n_next = p.rhoc[S + stride];
      base_next = p.cell_base[S + stride];
    }
    if (n <= 0 || n >= (1 << kRankBits) - 1) continue;
    if (base < 0 || base + n > p.n_used) continue;
    const int rb = p.run_base[S];
    for (int c0 = 0; c0 < n; c0 += 32) {
      // the copy's slot (-1: dropped) ...
      const int64_t ip = base + c0 + lane;
      const uint32_t w = c0 + lane < n ? p.runrank[ip] : kDropped;
      const int64_t id = p.pid && c0 + lane < n ? p.pid[ip] : 0;
      // ... while the values of the 32 copies arrive one by one: value e = 3 copy + axis, three a lane, so that
      // loads and (runs being contiguous) stores are coalesced
      const int ne = 3 * min(32, n - c0);
      const int64_t e0 = 3 * (base + c0);
      float v[3];
      int16_t x[3];
#pragma unroll
      for (int k = 0; k < 3; k++) {
        const int e = min(lane + 32 * k, ne - 1);
        v[k] = p.vp[e0 + e];
        x[k] = p.xp[e0 + e];
      }
      int pos = -1;
      if (w != kDropped) pos = (int)(p.run_off[rb + (int)(w >> kRankBits)] + (int64_t)(w & ((1u << kRankBits) - 1u)));
#pragma unroll
      for (int k = 0; k < 3; k++) {
        const int e = lane + 32 * k, c = e / 3, d = e - 3 * c;
        const int pc = __shfl_sync(0xffffffffu, pos, c);
        if (e < ne && pc >= 0) {
          p.xp_new[3 * (int64_t)pc + d] = drift_offset(p, x[k], v[k], p.err);
          p.vp_new[3 * (int64_t)pc + d] = v[k];
        }
      }
      if (p.pid && pos >= 0) p.pid_new[pos] = id;
    }
  }
}

// warp per buffer cell: the particles of the physical cell it mirrors, in order
// (buffer_particle.f90:44-345); xp/pid may be null (velocity-only refresh, buffer_v)
__global__ void __launch_bounds__(kDriftWarps * 32) k_halo_fill(DriftK p, const int32_t *rhoc,
                                                                  const int64_t *cell_base, int16_t *xp, float *vp,
                                                                  int64_t *pid) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  for (int64_t E = (int64_t)blockIdx.x * kDriftWarps + warp; E < p.ncells_src; E += (int64_t)gridDim.x * kDriftWarps) {
    int t, cx, cy, cz;
    cell_of(p, E, t, cx, cy, cz);
    const int lo = p.ncb, hi = p.ncb + p.nt;
    if (cx >= lo && cx < hi && cy >= lo && cy < hi && cz >= lo && cz < hi) continue;  // physical
    const int n = rhoc[E];
    if (n <= 0) continue;
    const int64_t dst = cell_base[E];
    int tt[3], l[3];
    mirrored_cell(p, t, cx, cy, cz, tt, l);
    const int64_t src = cell_base[ext_cell(p, tt, l)];
    if (dst < 0 || src < 0 || dst + n > p.n_used_new || src + n > p.n_used_new) continue;  // inconsistent spine
    // The cell's arrays are contiguous on both sides: copied value by value, coalesced, 64 copies a step with
    // all its loads under way before the first store
    for (int i0 = 0; i0 < 3 * n; i0 += 192) {
      float v[6];
      int16_t x[6];
      int64_t id[2];
#pragma unroll
      for (int k = 0; k < 6; k++) {
        const int i = i0 + lane + 32 * k;
        if (i < 3 * n) {
          v[k] = vp[3 * src + i];
          if (xp) x[k] = xp[3 * src + i];
        }
      }
#pragma unroll
      for (int k = 0; k < 2; k++) {
        const int i = i0 / 3 + lane + 32 * k;
        if (pid && i < n) id[k] = pid[src + i];
      }
#pragma unroll
      for (int k = 0; k < 6; k++) {
        const int i = i0 + lane + 32 * k;
        if (i < 3 * n) {
          vp[3 * dst + i] = v[k];
          if (xp) xp[3 * dst + i] = x[k];
        }
      }
#pragma unroll
      for (int k = 0; k < 2; k++) {
        const int i = i0 / 3 + lane + 32 * k;
        if (pid && i < n) pid[dst + i] = id[k];
      }
    }
  }
}

static DriftK make_driftk(const DriftArgs &a) {
  const Lay &L = *a.L;
  DriftK p{};
  p.nt = L.nt;
  p.ncb = L.ncb;
  p.nte = L.nte;
  p.nnt = L.nnt;
  p.nc = L.nc;
  p.nlayer = a.nlayer;
  p.tile_periodic = L.pm3_mode == CUBE_PM3_TILE_PERIODIC;
  p.ncells_src = (int64_t)L.ntile * L.nte * L.nte * L.nte;
  p.n_used = a.n_used;
  p.n_used_new = a.n_used_new;
  p.dt_mid = a.dt_mid;
  p.rcs_f = (float)L.rcs;
  p.xres_rcs = (1.0 / 65536.0) * (double)L.rcs;
  p.inv_rcs = (L.rcs & (L.rcs - 1)) ? 0.f : 1.0f / (float)L.rcs;
  p.inv_xres_rcs = 1.0 / p.xres_rcs;
  p.rhoc = a.rhoc;
  p.cell_base = a.cell_base;
  p.xp = a.xp;
  p.vp = a.vp;
  p.pid = a.pid;
  p.runrank = a.runrank;
  p.run_base = a.run_base;
  p.runs = (DriftRun *)a.runs;
  p.run_cap = a.run_cap;
  p.ctr = a.ctr;
  p.dest_runs = a.dest_runs;
  p.phys_count = a.phys_count;
  p.err = a.err;
  p.dest_start = a.dest_start;
  p.cursor = a.cursor;
  p.run_list = a.run_list;
  p.run_off = a.run_off;
  p.cell_base_new = a.cell_base_new;
  p.xp_new = a.xp_new;
  p.vp_new = a.vp_new;
  p.pid_new = a.pid_new;
  return p;
}

size_t drift_run_bytes() { return sizeof(DriftRun); }
int64_t drift_run_slack(int num_sms) { return (int64_t)num_sms * kDriftGridPerSM * kDriftWarps * kRunChunk; }

static unsigned warp_grid(int64_t items, int num_sms) {
  const int64_t blocks = (items + kDriftWarps - 1) / kDriftWarps;
  const int64_t cap = (int64_t)num_sms * kDriftGridPerSM;
  return (unsigned)(blocks < cap ? (blocks > 0 ? blocks : 1) : cap);
}

void launch_drift_runs(const DriftArgs &a, cudaStream_t s) {
  const DriftK p = make_driftk(a);
  k_drift_runs<<<warp_grid(p.ncells_src, a.num_sms), kDriftWarps * 32, 0, s>>>(p);
}

void launch_drift_spine(const DriftArgs &a, int32_t *rhoc_new, int64_t *rows, int64_t *idx_b_r_new,
                        int64_t *total, cudaStream_t s) {
  const DriftK p = make_driftk(a);
  const Lay &L = *a.L;
  k_ext_counts<<<(unsigned)((p.ncells_src + 255) / 256), 256, 0, s>>>(p, a.phys_count, rhoc_new);
  const int64_t nrows = (int64_t)L.ntile * L.nte * L.nte;
  k_row_sums<<<(unsigned)((nrows + 255) / 256), 256, 0, s>>>(rhoc_new, nrows, L.nte, rows);
  k_scan_rows<<<1, 1024, 0, s>>>(rows, nrows, idx_b_r_new, total);
}

void launch_drift_place(const DriftArgs &a, int32_t nruns, int32_t *scan_tmp, cudaStream_t s) {
  const DriftK p = make_driftk(a);
  const int64_t ndest = (int64_t)a.L->nc * a.L->nc * a.L->nc;
  scan_exclusive_i32(a.dest_runs, ndest, (int32_t *)a.dest_start, scan_tmp, s);
  if (nruns > 0) k_runs_fill<<<(unsigned)((nruns + 255) / 256), 256, 0, s>>>(p, nruns);
  k_runs_order<<<warp_grid((ndest + 3) / 4, a.num_sms), kDriftWarps * 32, 0, s>>>(p);  // four cells a warp
  k_drift_write<<<warp_grid(p.ncells_src, a.num_sms), kDriftWarps * 32, 0, s>>>(p);
  k_halo_fill<<<warp_grid(p.ncells_src, a.num_sms), kDriftWarps * 32, 0, s>>>(p, a.rhoc_new, a.cell_base_new,
                                                                                 a.xp_new, a.vp_new, a.pid_new);
}

void launch_halo_velocities(const Lay &L, const int32_t *rhoc, const int64_t *cell_base, float *vp, int64_t n_used,
                            int num_sms, cudaStream_t s) {
  DriftArgs a{};
  a.L = &L;
  a.nlayer = 1;
  a.n_used = a.n_used_new = n_used;
  const DriftK p = make_driftk(a);
  k_halo_fill<<<warp_grid(p.ncells_src, num_sms), kDriftWarps * 32, 0, s>>>(p, rhoc, cell_base, nullptr, vp,
                                                                              nullptr);
}

}  // namespace cube

// The hierarchical selector without the full surface. AFNI's power-of-two
// descent (fastfuncstuff/glm/arma.py:2224-2322) reads at most 9 pairs of each
// level around the voxel's best pair so far, a tenth of a 33 x 33 grid's 561
// pairs, so only those are formed:
//   top     the levels whose pairs, over all voxels, are few enough to evaluate
//           for every voxel (48 pairs of a 33 x 33 grid: levels 4, 3 and 2):
//           one projection launch, one kernel for the recurrences, the
//           criterion and the descent through those levels;
//   rounds  one per level left: the voxels sorted by their pair (the cell), and
//           each tile of a cell's rows evaluated at the cell's <= 8 neighbours.
//
// Each criterion is the full surface's bit for bit (surface_kernel), so the
// answers are too: the same fp32 recurrence in blocks of 16 steps, each pair's
// block summed the way its chunk of the full grid sums it ("steady" blocks
// sum v^2 and scale once). One formula serves both, per step the factor e and
// per block the factor f: sq += (v e) v, st += sq f with (e, f) = (1, 1/D) in a
// steady block and (1/D, 1) otherwise; products with 1 are exact.
//
// Bound: FP32 FMAs of the recurrences (2 packed instructions per couple of
// pairs and step, 8 pairs per thread in registers). Rows reach shared memory
// 16 samples at a time by asynchronous copies three blocks deep, read by 16-byte
// loads (any T), with the coefficients of the block, laid out in couples once
// per fit (descent_tables_kernel), copied beside them.
#include <algorithm>

#include "common.cuh"
#include "project_tc.cuh"

namespace ffsk {
namespace {

constexpr int DB = 16;              // steps per block
constexpr int D_LD = DB + 4;        // row stride of a staged block: LDS.128 of 8 rows in distinct banks
constexpr int D_BUF = 3;            // blocks in flight
constexpr int D_SLOTS = 8;          // pair slots per group (one group per thread): 4 couples
constexpr int D_C = D_SLOTS / 2;
constexpr int TOP_ROWS = 64;        // rows per CTA of the top kernel
constexpr int TOP_GROUPS = 8;       // most groups (64 slots)
constexpr int ROUND_ROWS = 128;     // rows per tile of a round
constexpr int CHUNK_SLOTS = 16;     // slots per chunk of the full surface

static_assert(D_SLOTS == PAIR_SLOTS, "a cell's neighbours fill one group");

// steady[p][blk]: every filled slot of p's chunk keeps its coefficients over
// the 16 steps of the block (surface_kernel's rule). One CTA per chunk.
__global__ void __launch_bounds__(256) descent_steady_kernel(int T, const float4* __restrict__ coef,
                                                             const int* __restrict__ chunk_start,
                                                             const int* __restrict__ chunk_pairs,
                                                             uint8_t* __restrict__ steady) {
  extern __shared__ int moved[];  // [nblk] some slot's coefficients change in the block
  const int nblk = (T + DB - 1) / DB;
  const int c0 = chunk_start[blockIdx.x], ng = chunk_start[blockIdx.x + 1] - c0;
  for (int b = threadIdx.x; b < nblk; b += blockDim.x) moved[b] = b == 0 || b * DB + DB > T;
  __syncthreads();
  for (int e = threadIdx.x; e < ng * T; e += blockDim.x) {
    const int s = e / T, t = e % T;
    const int p = chunk_pairs[c0 + s];
    if (p < 0 || t == 0) continue;
    const float4 x = coef[(size_t)p * T + t], y = coef[(size_t)p * T + t - 1];
    if (!(x.x == y.x && x.y == y.y && x.z == y.z)) moved[t / DB] = 1;
  }
  __syncthreads();
  for (int e = threadIdx.x; e < ng * nblk; e += blockDim.x) {
    const int p = chunk_pairs[c0 + e / nblk];
    if (p >= 0) steady[(size_t)p * nblk + e % nblk] = !moved[e % nblk];
  }
}

// The coefficients of groups of 8 pair slots (-1: empty, all zero) as couples:
// ct[g][t][4] = (-m, -m', e, e'), nc[g][t][NZ] = (-c, -c'), fb[g][blk][4] =
// (f, f'), fast[g][blk] = every slot's block is steady. NZ = 4: a filter per
// couple; NZ = 2: one per quarter of 4 slots, which share one a.
struct Tables {
  float4* ct;
  float2* nc;
  float2* fb;
  uint8_t* fast;
};

template <int NZ>
__global__ void __launch_bounds__(128) descent_tables_kernel(int T, const float4* __restrict__ coef,
                                                             const uint8_t* __restrict__ steady,
                                                             const int* __restrict__ slots, Tables o) {
  const int g = blockIdx.x, t = blockIdx.y * blockDim.x + threadIdx.x;
  const int nblk = (T + DB - 1) / DB;
  if (t >= T) return;
  const int blk = t / DB;
  bool all = true;
  float cq[2] = {0.f, 0.f};
#pragma unroll
  for (int k = 0; k < D_C; ++k) {
    float m[2], e[2], f[2], c[2];
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int p = slots[g * D_SLOTS + 2 * k + h];
      m[h] = e[h] = f[h] = c[h] = 0.f;
      if (p >= 0) {
        const float4 q = coef[(size_t)p * T + t];
        const bool st = steady[(size_t)p * nblk + blk] != 0;
        m[h] = -q.y;
        e[h] = st ? 1.f : q.z;
        f[h] = st ? q.z : 1.f;
        c[h] = -q.x;
        all = all && st;
        cq[k >> 1] = c[h];
      }
    }
    o.ct[((size_t)g * T + t) * D_C + k] = make_float4(m[0], m[1], e[0], e[1]);
    if (NZ == D_C) o.nc[((size_t)g * T + t) * NZ + k] = make_float2(c[0], c[1]);
    if (t % DB == 0) o.fb[((size_t)g * nblk + blk) * D_C + k] = make_float2(f[0], f[1]);
  }
  if (NZ == 2) {
    o.nc[((size_t)g * T + t) * NZ] = make_float2(cq[0], cq[0]);
    o.nc[((size_t)g * T + t) * NZ + 1] = make_float2(cq[1], cq[1]);
  }
  if (t % DB == 0) o.fast[g * nblk + blk] = all;
}

__device__ __forceinline__ void cp16(void* dst, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src)
               : "memory");
}
__device__ __forceinline__ void cp4(void* dst, const void* src, bool on) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src),
               "r"(on ? 4 : 0)
               : "memory");
}

// Shared memory of one block of a group: the couples' coefficients, filters
// and factors.
template <int NZ>
struct Stage {
  float4 ct[DB][D_C];
  float2 nc[DB][NZ];
  float2 fb[D_C];
};

// y'R^-1 y of this thread's row at its group's 8 pairs, and y'y when YY.
// rows[l] (shared): the row of Y each of the CTA's R rows reads. G groups share
// the rows; a warp's threads share their group. The CTA's blockDim is R * G.
template <int NZ, int R, bool YY>
__device__ __forceinline__ void run_groups(int T, const float* __restrict__ Y, const int* rows, float* ys,
                                           Stage<NZ>* stg, int G, int g0, Tables tb, float (&ss)[D_SLOTS], float& yy) {
  const int tid = threadIdx.x, nth = blockDim.x;
  const int r = tid % R, g = tid / R;
  const int nblk = (T + DB - 1) / DB;
  const bool vec = (T & 3) == 0;
  auto issue = [&](int blk) {
    const int t0 = blk * DB, n = min(DB, T - t0);
    float* yb = ys + (size_t)(blk % D_BUF) * R * D_LD;
    if (vec) {
      const int nq = n >> 2;
      for (int i = tid; i < R * (DB / 4); i += nth) {
        const int l = i / (DB / 4), q = i % (DB / 4);
        if (q < nq) cp16(yb + l * D_LD + 4 * q, Y + (size_t)rows[l] * T + t0 + 4 * q);
      }
    } else {
      for (int i = tid; i < R * DB; i += nth) {
        const int l = i / DB, k = i % DB;
        cp4(yb + l * D_LD + k, Y + (size_t)rows[l] * T + t0 + (k < n ? k : 0), k < n);
      }
    }
    Stage<NZ>* st = stg + (blk % D_BUF) * G;
    const int per = n * D_C + n * NZ / 2 + D_C / 2;  // 16-byte words per group
    for (int i = tid; i < G * per; i += nth) {
      const int gg = i / per, w = i % per;
      const size_t gt = (size_t)(g0 + gg) * T + t0;
      if (w < n * D_C)
        cp16(reinterpret_cast<float4*>(st[gg].ct) + w, tb.ct + gt * D_C + w);
      else if (w < n * D_C + n * NZ / 2)
        cp16(reinterpret_cast<float4*>(st[gg].nc) + (w - n * D_C),
             reinterpret_cast<const float4*>(tb.nc + gt * NZ) + (w - n * D_C));
      else
        cp16(reinterpret_cast<float4*>(st[gg].fb) + (w - n * D_C - n * NZ / 2),
             reinterpret_cast<const float4*>(tb.fb + ((size_t)(g0 + gg) * nblk + blk) * D_C) +
                 (w - n * D_C - n * NZ / 2));
    }
  };
  const uint64_t zero2 = pack2(0.f, 0.f);
  uint64_t vv[D_C], st2[D_C];
#pragma unroll
  for (int c = 0; c < D_C; ++c) vv[c] = st2[c] = zero2;
  uint64_t yp = zero2;
  yy = 0.f;
  issue(0);
  asm volatile("cp.async.commit_group;" ::: "memory");
  if (nblk > 1) issue(1);
  asm volatile("cp.async.commit_group;" ::: "memory");
  for (int blk = 0; blk < nblk; ++blk) {
    asm volatile("cp.async.wait_group 1;" ::: "memory");
    __syncthreads();  // block blk has landed, and every thread is past block blk - 1
    if (blk + 2 < nblk) issue(blk + 2);
    asm volatile("cp.async.commit_group;" ::: "memory");
    const float4* y4 = reinterpret_cast<const float4*>(ys + ((size_t)(blk % D_BUF) * R + r) * D_LD);
    const Stage<NZ>& s = stg[(blk % D_BUF) * G + g];
    const int n = min(DB, T - blk * DB);
    uint64_t sq[D_C];
#pragma unroll
    for (int c = 0; c < D_C; ++c) sq[c] = zero2;
    float yb[DB];
#pragma unroll
    for (int q = 0; q < DB / 4; ++q) {
      float4 y = make_float4(0.f, 0.f, 0.f, 0.f);
      if (4 * q < n) y = y4[q];
      yb[4 * q] = y.x;
      yb[4 * q + 1] = y.y;
      yb[4 * q + 2] = y.z;
      yb[4 * q + 3] = y.w;
    }
    if (YY) {
      float b = 0.f;
#pragma unroll
      for (int k = 0; k < DB; ++k)
        if (k < n) b = fmaf(yb[k], yb[k], b);
      yy += b;
    }
    if (tb.fast[(g0 + g) * nblk + blk]) {
      uint64_t nm[D_C], nz[NZ];
#pragma unroll
      for (int c = 0; c < D_C; ++c) {
        const float4 q = s.ct[0][c];
        nm[c] = pack2(q.x, q.y);
      }
#pragma unroll
      for (int z = 0; z < NZ; ++z) nz[z] = pack2(s.nc[0][z].x, s.nc[0][z].y);
#pragma unroll
      for (int k = 0; k < DB; ++k) {
        const uint64_t y = pack2(yb[k], yb[k]);
        uint64_t z[NZ];
#pragma unroll
        for (int i = 0; i < NZ; ++i) z[i] = fma2(nz[i], yp, y);
#pragma unroll
        for (int c = 0; c < D_C; ++c) {
          vv[c] = fma2(nm[c], vv[c], z[c * NZ / D_C]);
          sq[c] = fma2(vv[c], vv[c], sq[c]);
        }
        yp = y;
      }
    } else {
#pragma unroll
      for (int k = 0; k < DB; ++k) {
        if (k < n) {
          const uint64_t y = pack2(yb[k], yb[k]);
          uint64_t z[NZ];
#pragma unroll
          for (int i = 0; i < NZ; ++i) {
            const float2 q = s.nc[k][i];
            z[i] = fma2(pack2(q.x, q.y), yp, y);
          }
#pragma unroll
          for (int c = 0; c < D_C; ++c) {
            const float4 q = s.ct[k][c];
            vv[c] = fma2(pack2(q.x, q.y), vv[c], z[c * NZ / D_C]);
            sq[c] = fma2(mul2(vv[c], pack2(q.z, q.w)), vv[c], sq[c]);
          }
          yp = y;
        }
      }
    }
#pragma unroll
    for (int c = 0; c < D_C; ++c) st2[c] = fma2(sq[c], pack2(s.fb[c].x, s.fb[c].y), st2[c]);
  }
#pragma unroll
  for (int c = 0; c < D_C; ++c) unpack2(st2[c], ss[2 * c], ss[2 * c + 1]);
}

// The criterion of a pair relative to (0, 0), as the surface kernel forms it.
__device__ __forceinline__ float crit_of(float ss, float proj, float dc, float rss0, float den, int Tk) {
  const float rss = fmaxf(ss - proj, 0.f);
  return dc + (float)Tk * log1pf((rss - rss0) / den);
}

struct TopArgs {
  int V, T, Tk, P, p0, n_groups, n_a, n_b, za, zb, ltop, lev_stop;
  const float* rows;         // [V][T]
  Tables tb;
  const int* slots;          // [n_groups * 8] pair of each slot (-1: empty)
  const int* lat_slot;       // [n_a * n_b] slot, -1: no pair, -2: an identity pair
  const int* lattice;        // [n_a * n_b] pair
  const float* proj;         // [n_groups * 8 + 1][V], the last row (0, 0)'s
  const double* logdet_R;
  const double* logdet_XtX;  // [n_designs][P]
  const int* tile_design;    // [V / 256] or NULL
  int* key;                  // [V] design * P + pair
  float* low;                // [V] criterion there
  float* rss0;               // [V]
  double* crit0;             // [V]
  int* best;                 // outputs of the last level
  float* best_crit;
  const int* flag;           // set: a projection gave up, and the criterion is a NaN
};

// At most 80 registers: with the 118 that the compiler takes by itself one CTA
// of 384 threads fills an SM, and its 12 warps waited at each block's barrier
// (ncu: 46% of the issue slots); two run at 80, without spills. 200,000 voxels of T
// = 400: 871 -> 626 us, 100,000 of T = 855: 1284 -> 950 (64 registers: 654, 1001).
__global__ void __maxnreg__(80) descent_top_kernel(TopArgs a) {
  extern __shared__ float4 dsm4[];
  __shared__ int rows[TOP_ROWS];
  __shared__ float dc[TOP_GROUPS * D_SLOTS], rss0_s[TOP_ROWS];
  const int G = a.n_groups, tid = threadIdx.x, r = tid % TOP_ROWS, g = tid / TOP_ROWS;
  Stage<2>* stg = reinterpret_cast<Stage<2>*>(dsm4);
  float* ys = reinterpret_cast<float*>(stg + D_BUF * G);   // [D_BUF][TOP_ROWS][D_LD]
  float* ds = ys + D_BUF * TOP_ROWS * D_LD;                // [G * 8][TOP_ROWS] criteria
  const int v0 = blockIdx.x * TOP_ROWS, v = min(v0 + r, a.V - 1);
  const int dsg = a.tile_design ? a.tile_design[v0 >> 8] : 0;
  const double* ldx = a.logdet_XtX + (size_t)dsg * a.P;
  const double c_p0 = a.logdet_R[a.p0] + ldx[a.p0];
  if (g == 0) rows[r] = v;
  for (int s = tid; s < G * D_SLOTS; s += blockDim.x) {
    const int p = a.slots[s];
    dc[s] = p >= 0 ? (float)((a.logdet_R[p] + ldx[p]) - c_p0) : 0.f;
  }
  __syncthreads();
  float ss[D_SLOTS], yy;
  run_groups<2, TOP_ROWS, true>(a.T, a.rows, rows, ys, stg, G, 0, a.tb, ss, yy);
  const float rss0 = fmaxf(yy - a.proj[(size_t)G * D_SLOTS * a.V + v], 0.f);
  const float den = rss0 + 1e-10f;
#pragma unroll
  for (int s = 0; s < D_SLOTS; ++s) {
    const int sl = g * D_SLOTS + s;
    if (a.slots[sl] >= 0) ds[sl * TOP_ROWS + r] = crit_of(ss[s], a.proj[(size_t)sl * a.V + v], dc[sl], rss0, den, a.Tk);
  }
  if (g == 0) rss0_s[r] = rss0;
  __syncthreads();
  if (tid >= TOP_ROWS || v0 + tid >= a.V) return;
  const float r0 = rss0_s[tid];
  const float d_id = (float)a.Tk * log1pf((r0 - r0) / (r0 + 1e-10f));  // an identity pair: 0, or NaN of an infinite row
  auto at = [&](int ai, int bi) -> float {
    const int s = a.lat_slot[ai * a.n_b + bi];
    return s >= 0 ? ds[s * TOP_ROWS + tid] : s == -2 ? d_id : INFINITY;
  };
  int ba = a.za, bb = a.zb;
  float bl = at(ba, bb);
  for (int lev = a.ltop; lev >= a.lev_stop; --lev) {
    const int step = 1 << lev;
    float mn = INFINITY;
    int sa = -1, sb = -1;
    auto take = [&](int ai, int bi) {
      const float d = at(ai, bi);
      if (sa < 0 || d < mn) {
        mn = d;
        sa = ai;
        sb = bi;
      }
    };
    if (lev == a.ltop) {
      for (int bi = 0; bi < a.n_b; bi += step)
        for (int ai = 0; ai < a.n_a; ai += step) take(ai, bi);
    } else {
      for (int ob = -1; ob <= 1; ++ob)
        for (int oa = -1; oa <= 1; ++oa)
          take(min(max(ba + oa * step, 0), a.n_a - 1), min(max(bb + ob * step, 0), a.n_b - 1));
    }
    if (mn < bl) {
      bl = mn;
      ba = sa;
      bb = sb;
    }
  }
  const int p = a.lattice[ba * a.n_b + bb], vo = v0 + tid;
  const double cr0 = c_p0 + (double)a.Tk * log((double)r0 + 1e-10);
  a.key[vo] = dsg * a.P + p;
  a.low[vo] = bl;
  a.rss0[vo] = r0;
  a.crit0[vo] = cr0;
  if (a.lev_stop == 0) {
    a.best[vo] = p;
    a.best_crit[vo] = *a.flag ? NAN : (float)(cr0 + (double)bl);
  }
}

// Row tiles of at most ROUND_ROWS rows of one key (rows sorted by key, key k's
// ending at end[k]), in no particular order.
__global__ void descent_tiles_kernel(int n_keys, const int* __restrict__ end, int4* __restrict__ tiles, int* n_tiles) {
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= n_keys) return;
  const int s0 = k ? end[k - 1] : 0, n = end[k] - s0;
  const int nt = (n + ROUND_ROWS - 1) / ROUND_ROWS;
  if (nt == 0) return;
  const int at = atomicAdd(n_tiles, nt);
  for (int t = 0; t < nt; ++t) tiles[at + t] = make_int4(s0 + t * ROUND_ROWS, min(ROUND_ROWS, n - t * ROUND_ROWS), k, 0);
}

// The fp16 operand rows and exponents in the order idx, 16 bytes per thread.
__global__ void __launch_bounds__(256) descent_gather_kernel(int n, int nw, const int* __restrict__ idx,
                                                             const uint4* __restrict__ hi, const uint4* __restrict__ lo,
                                                             const int* __restrict__ yexp, uint4* __restrict__ out_hi,
                                                             uint4* __restrict__ out_lo, int* __restrict__ out_exp) {
  const long long total = (long long)n * nw;
  for (long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x; e < total;
       e += (long long)gridDim.x * blockDim.x) {
    const int i = (int)(e / nw), k = (int)(e % nw), v = idx[i];
    out_hi[(size_t)i * nw + k] = hi[(size_t)v * nw + k];
    out_lo[(size_t)i * nw + k] = lo[(size_t)v * nw + k];
    if (k == 0) out_exp[i] = yexp[v];
  }
}

struct RoundArgs {
  int T, Tk, P, p0;
  const float* rows;
  const int* idx;            // [n] row of Y of each sorted row
  const int4* tiles;
  const int* n_tiles;
  Tables tb;
  const int* cell_group;     // [P] group of each cell
  const int* cell_pairs;     // [P][8] neighbours in the selector's order: pair, -1 none, -2 - p identity
  const float* proj;         // [n][8] by sorted row and position
  const double* logdet_R;
  const double* logdet_XtX;
  const float* rss0;
  const double* crit0;
  int* key;
  float* low;
  int* best;                 // last round only
  float* best_crit;
  const int* flag;
};

// A thread per row of the tile, its cell's 8 neighbours in registers; the
// first strictly least of them replaces the cell where it is below it.
__global__ void __launch_bounds__(ROUND_ROWS, 5) descent_round_kernel(RoundArgs a) {
  extern __shared__ float4 dsm4[];
  __shared__ int rows[ROUND_ROWS], pr[D_SLOTS];
  __shared__ float dc[D_SLOTS];
  if ((int)blockIdx.x >= *a.n_tiles) return;
  const int4 tl = a.tiles[blockIdx.x];
  const int tid = threadIdx.x, i = tl.x + min(tid, tl.y - 1), v = a.idx[i];
  const int cell = tl.z % a.P, dsg = tl.z / a.P;
  const double* ldx = a.logdet_XtX + (size_t)dsg * a.P;
  Stage<4>* stg = reinterpret_cast<Stage<4>*>(dsm4);
  float* ys = reinterpret_cast<float*>(stg + D_BUF);
  rows[tid] = v;
  if (tid < D_SLOTS) {
    const int p = a.cell_pairs[cell * D_SLOTS + tid];
    pr[tid] = p;
    dc[tid] = p >= 0 ? (float)((a.logdet_R[p] + ldx[p]) - (a.logdet_R[a.p0] + ldx[a.p0])) : 0.f;
  }
  __syncthreads();
  float ss[D_SLOTS], yy;
  run_groups<4, ROUND_ROWS, false>(a.T, a.rows, rows, ys, stg, 1, a.cell_group[cell], a.tb, ss, yy);
  if (tid >= tl.y) return;
  const float r0 = a.rss0[v], den = r0 + 1e-10f;
  float mn = INFINITY;
  int at = -1;
#pragma unroll
  for (int s = 0; s < D_SLOTS; ++s) {
    const int p = pr[s];
    const float d = p >= 0 ? crit_of(ss[s], a.proj[(size_t)i * D_SLOTS + s], dc[s], r0, den, a.Tk)
                    : p == -1 ? INFINITY
                              : (float)a.Tk * log1pf((r0 - r0) / den);
    if (s == 0 || d < mn) {
      mn = d;
      at = p >= 0 ? p : -2 - p;
    }
  }
  int p = cell;
  float bl = a.low[v];
  if (mn < bl) {
    bl = mn;
    p = at;
  }
  if (a.best) {
    a.best[v] = p;
    a.best_crit[v] = *a.flag ? NAN : (float)(a.crit0[v] + (double)bl);
  } else {
    a.key[v] = dsg * a.P + p;
    a.low[v] = bl;
  }
}

// Carves the workspace; with base NULL only the size.
struct Work {
  uint8_t* steady;
  Tables top, cells;
  float *proj, *low, *rss0;
  double* crit0;
  int *key, *end, *order, *counts, *yexp;
  int4* tiles;
  uint16_t *hi, *lo;
  size_t bytes;
};

Work carve(const ffs_descent_args& a, char* base) {
  Work w{};
  size_t at = 0;
  auto take = [&](size_t n) {
    char* p = base ? base + at : nullptr;
    at += (n + 255) & ~(size_t)255;
    return p;
  };
  const size_t V = a.V, T = a.T, nblk = (T + DB - 1) / DB, keys = (size_t)a.P * a.n_designs;
  auto tables = [&](size_t n, int nz) {
    Tables t;
    t.ct = reinterpret_cast<float4*>(take(n * T * D_C * sizeof(float4)));
    t.nc = reinterpret_cast<float2*>(take(n * T * nz * sizeof(float2)));
    t.fb = reinterpret_cast<float2*>(take(n * nblk * D_C * sizeof(float2)));
    t.fast = reinterpret_cast<uint8_t*>(take(n * nblk));
    return t;
  };
  w.steady = reinterpret_cast<uint8_t*>(take((size_t)a.P * nblk));
  w.top = tables(a.n_groups, 2);
  w.cells = tables(a.n_cell_groups, 4);
  const size_t rows = std::max<size_t>((size_t)a.n_groups * D_SLOTS + 1, D_SLOTS);
  w.proj = reinterpret_cast<float*>(take(rows * V * sizeof(float)));
  w.low = reinterpret_cast<float*>(take(V * sizeof(float)));
  w.rss0 = reinterpret_cast<float*>(take(V * sizeof(float)));
  w.crit0 = reinterpret_cast<double*>(take(V * sizeof(double)));
  w.key = reinterpret_cast<int*>(take(V * sizeof(int)));
  if (a.n_rounds > 0) {
    w.end = reinterpret_cast<int*>(take((keys + 1) * sizeof(int)));
    w.order = reinterpret_cast<int*>(take(V * sizeof(int)));
    w.counts = reinterpret_cast<int*>(take(sizeof(int)));
    w.yexp = reinterpret_cast<int*>(take(V * sizeof(int)));
    w.tiles = reinterpret_cast<int4*>(take((ceil_div(V, ROUND_ROWS) + std::min(V, keys)) * sizeof(int4)));
    w.hi = reinterpret_cast<uint16_t*>(take(V * a.ld * 2));
    w.lo = reinterpret_cast<uint16_t*>(take(V * a.ld * 2));
  }
  w.bytes = at;
  return w;
}

int check_descent(const ffs_descent_args* a) {
  FFS_REQUIRE(a && a->V > 0 && a->T > a->K && a->K > 0 && a->K <= 256 && a->P > 0 && a->n_designs > 0 &&
                  a->ld >= a->T && a->ld % 64 == 0,
              "ffs_reml_descent: bad sizes");
  FFS_REQUIRE(surface_smem(a->T) <= SURFACE_SMEM_MAX, "ffs_reml_descent: T=%d too long", a->T);
  FFS_REQUIRE((long long)a->P * a->n_designs < (1 << 24), "ffs_reml_descent: too many pairs");
  FFS_REQUIRE(a->p0 >= 0 && a->p0 < a->P && a->za >= 0 && a->za < a->n_a && a->zb >= 0 && a->zb < a->n_b,
              "ffs_reml_descent: (0, 0) outside the lattice");
  FFS_REQUIRE(a->n_groups > 0 && a->n_groups <= TOP_GROUPS && a->n_rounds >= 0 && a->n_rounds <= a->ltop &&
                  a->n_chunks > 0 && a->n_list > 0 && a->n_list <= a->n_groups * D_SLOTS + 1 &&
                  (a->n_rounds == 0 || a->n_cell_groups > 0),
              "ffs_reml_descent: bad plan (%d groups, %d rounds)", a->n_groups, a->n_rounds);
  return FFS_OK;
}

}  // namespace
}  // namespace ffsk

using namespace ffsk;

extern "C" size_t ffs_reml_descent_work_bytes(const ffs_descent_args* a) {
  clear_error();
  if (check_descent(a) != FFS_OK) return 0;
  return carve(*a, nullptr).bytes;
}

extern "C" int ffs_reml_descent(const ffs_descent_args* a, void* stream) {
  clear_error();
  if (const int rc = check_descent(a)) return rc;
  FFS_REQUIRE(a->rows && a->yr_hi && a->yr_lo && a->yexp && a->u_hi && a->u_lo && a->uexp && a->coef && a->logdet_R &&
                  a->logdet_XtX && a->chunk_start && a->chunk_pairs && a->slots && a->list && a->lat_slot &&
                  a->lattice && a->best && a->best_crit && a->flag && a->work,
              "ffs_reml_descent: null buffer");
  FFS_REQUIRE(a->n_rounds == 0 || (a->cell_slots && a->cell_group && a->cell_pairs && a->cell_list),
              "ffs_reml_descent: null cell tables");
  for (const void* p : {(const void*)a->yr_hi, (const void*)a->yr_lo, (const void*)a->u_hi, (const void*)a->u_lo,
                        (const void*)a->rows, (const void*)a->coef})
    FFS_REQUIRE(((uintptr_t)p & 15) == 0, "ffs_reml_descent: operands must be 16-byte aligned");
  FFS_REQUIRE(((uintptr_t)a->work & 255) == 0, "ffs_reml_descent: the workspace must be 256-byte aligned");
  const Work w = carve(*a, static_cast<char*>(a->work));
  if (a->work_bytes < w.bytes) {
    set_error("ffs_reml_descent: workspace of %zu bytes, %zu needed", a->work_bytes, w.bytes);
    return FFS_ERR_WORKSPACE;
  }
  cudaStream_t st = (cudaStream_t)stream;
  const int T = a->T, nblk = ceil_div(T, DB), tb = ceil_div(T, 128);
  const float4* coef = reinterpret_cast<const float4*>(a->coef);
  descent_steady_kernel<<<a->n_chunks, 256, sizeof(int) * nblk, st>>>(T, coef, a->chunk_start, a->chunk_pairs, w.steady);
  descent_tables_kernel<2><<<dim3(a->n_groups, tb), 128, 0, st>>>(T, coef, w.steady, a->slots, w.top);
  if (a->n_rounds > 0)
    descent_tables_kernel<4><<<dim3(a->n_cell_groups, tb), 128, 0, st>>>(T, coef, w.steady, a->cell_slots, w.cells);

  PairProject pp{};
  pp.V = a->V;
  pp.T = T;
  pp.K = a->K;
  pp.P = a->P;
  pp.n_designs = a->n_designs;
  pp.ld = a->ld;
  pp.hi = a->yr_hi;
  pp.lo = a->yr_lo;
  pp.yexp = a->yexp;
  pp.u_hi = a->u_hi;
  pp.u_lo = a->u_lo;
  pp.uexp = a->uexp;
  pp.list = a->list;
  pp.n_list = a->n_list;
  pp.tile_design = a->tile_design;
  pp.proj = w.proj;
  pp.flag = a->flag;
  if (const int rc = project_pairs(pp, st)) return rc;

  TopArgs ta{a->V, T, T - a->K, a->P, a->p0, a->n_groups, a->n_a, a->n_b, a->za, a->zb, a->ltop, a->n_rounds,
             a->rows, w.top, a->slots, a->lat_slot, a->lattice, w.proj, a->logdet_R, a->logdet_XtX, a->tile_design,
             w.key, w.low, w.rss0, w.crit0, a->best, a->best_crit, a->flag};
  const size_t top_smem = sizeof(Stage<2>) * D_BUF * a->n_groups +
                          sizeof(float) * TOP_ROWS * (D_BUF * D_LD + a->n_groups * D_SLOTS);
  FFS_CUDA(ensure_dyn_smem(reinterpret_cast<const void*>(descent_top_kernel), top_smem));
  descent_top_kernel<<<ceil_div(a->V, TOP_ROWS), TOP_ROWS * a->n_groups, top_smem, st>>>(ta);

  const int keys = a->P * a->n_designs;
  const int max_tiles = ceil_div(a->V, ROUND_ROWS) + std::min(a->V, keys);
  const size_t round_smem = sizeof(Stage<4>) * D_BUF + sizeof(float) * ROUND_ROWS * D_BUF * D_LD;
  int sms = 0;
  FFS_CUDA(sm_count(&sms));
  for (int r = 0; r < a->n_rounds; ++r) {
    if (const int rc = ffs_reml_group(a->V, keys, w.key, w.end, w.order, stream)) return rc;
    FFS_CUDA(cudaMemsetAsync(w.counts, 0, sizeof(int), st));
    descent_tiles_kernel<<<ceil_div(keys, 256), 256, 0, st>>>(keys, w.end, w.tiles, w.counts);
    const int nw = a->ld / 8;
    const int blocks = (int)std::min<long long>(ceil_div((long long)a->V * nw, 256), (long long)sms * 8);
    descent_gather_kernel<<<blocks, 256, 0, st>>>(a->V, nw, w.order, reinterpret_cast<const uint4*>(a->yr_hi),
                                                  reinterpret_cast<const uint4*>(a->yr_lo), a->yexp,
                                                  reinterpret_cast<uint4*>(w.hi), reinterpret_cast<uint4*>(w.lo), w.yexp);
    pp.hi = w.hi;
    pp.lo = w.lo;
    pp.yexp = w.yexp;
    pp.list = a->cell_list + (size_t)r * a->P * D_SLOTS;
    pp.tile_design = nullptr;
    pp.tiles = w.tiles;
    pp.n_tiles = w.counts;
    pp.max_tiles = max_tiles;
    if (const int rc = project_pairs(pp, st)) return rc;
    const bool last = r + 1 == a->n_rounds;
    RoundArgs ra{T, T - a->K, a->P, a->p0, a->rows, w.order, w.tiles, w.counts, w.cells,
                 a->cell_group + (size_t)r * a->P, a->cell_pairs + (size_t)r * a->P * D_SLOTS, w.proj, a->logdet_R,
                 a->logdet_XtX, w.rss0, w.crit0, w.key, w.low, last ? a->best : nullptr, a->best_crit,
                 a->flag};
    FFS_CUDA(ensure_dyn_smem(reinterpret_cast<const void*>(descent_round_kernel), round_smem));
    descent_round_kernel<<<max_tiles, ROUND_ROWS, round_smem, st>>>(ra);
  }
  return check_launch("descent kernels");
}

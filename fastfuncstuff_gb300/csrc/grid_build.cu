// K1: FP64 factorisation of the REML grid, one CTA per (a, b) pair.
//
// The ARMA(1,1) correlation of a run, R_ij = rho(|tau_i - tau_j|) with
// rho(0) = 1, rho(k) = lambda a^(k-1), becomes tridiagonal after the AR filter
// z_t = y_t - c_t y_{t-1}, c_t = a^(tau_t - tau_{t-1}) (c = 0 at a run start):
//   T_tt      = 1 + c_t^2 - 2 c_t rho(g_t)      (1 at a run start)
//   T_t,t-1   = rho(g_t) - c_t                  (g_t = tau_t - tau_{t-1})
// and every other entry is zero, censoring gaps included. Its LDL' factor
// (unit bidiagonal L~ with sub-diagonal m_t, diagonal D_t) gives the Cholesky
// factor of R exactly: chol(R) = A^-1 L~ D^1/2, A the unit bidiagonal AR filter.
// So diag(chol(R)) = sqrt(D_t) and log|R| = 2 sum log(sqrt(D_t) + 1e-10), the
// same quantity fastfuncstuff/glm/whiten.py:219-223 takes from a dense
// Cholesky, at O(T) cost instead of O(T^3).
//
// The design-dependent part follows fastfuncstuff/glm/arma.py:1459-1506:
// X_w = L^-1 X, Cholesky of X_w'X_w (QR when it is not positive definite),
// Q = X_w L_xtx^-T, logdet = 2 sum log(|diag| + 1e-10). On top of that the
// kernel emits U = L^-T Q (the projection that lets the search skip the
// whitening GEMM) and G = U L_xtx^-1 (the GLS solve), and the per-pair GLS
// constants of fastfuncstuff/glm/arma.py:4853-4905.
#include <algorithm>
#include <mutex>

#include "common.cuh"

namespace ffsk {

namespace {

constexpr int GB_PF = 4;  // samples loaded ahead in the sequential recursions
// Threads per CTA (one (design, pair) item at a time); 128 measured no faster
// at K = 20 and slower at K = 130, where the Gram matrix and the O(K^3)
// phases use every thread.
constexpr int GB_THREADS = 256;

struct PairScratch {
  double* cm;  // [T][4]  c, m, D, 1/sqrt(D)
  double* Xw;  // [K][T]  whitened design, later U = L^-T Q
  double* Qm;  // [K][T]  Q
  double* Lx;  // [K][K]  Cholesky factor of X_w'X_w (lower, row-major)
  double* Li;  // [K][K]  its inverse
  double* A;   // [K][K]  (X_w'X_w)^-1
  double* S;   // [K][K]  scratch for the task block
};

__host__ __device__ inline size_t pair_doubles(int T, int K) {
  return (size_t)4 * T + (size_t)2 * K * T + (size_t)4 * K * K;
}

__device__ PairScratch scratch_of(double* work, int p, int T, int K) {
  PairScratch s;
  double* w = work + (size_t)p * pair_doubles(T, K);
  s.cm = w;
  s.Xw = s.cm + 4 * T;
  s.Qm = s.Xw + (size_t)K * T;
  s.Lx = s.Qm + (size_t)K * T;
  s.Li = s.Lx + (size_t)K * K;
  s.A = s.Li + (size_t)K * K;
  s.S = s.A + (size_t)K * K;
  return s;
}

__device__ double block_sum(double v, double* red) {
  v = warp_sum_d(v);
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  __syncthreads();
  if (lane == 0) red[wid] = v;
  __syncthreads();
  double t = 0.0;
  if (threadIdx.x < 32) {
    t = (threadIdx.x < (blockDim.x >> 5)) ? red[threadIdx.x] : 0.0;
    t = warp_sum_d(t);
    if (threadIdx.x == 0) red[0] = t;
  }
  __syncthreads();
  return red[0];
}

// sum_t f(t), t < n, as block_sum adds it over 256 threads (f(t) in the thread t mod
// 256) whatever the CTA's width: a pair's factor does not depend on the kernel that
// forms it. Starts and ends with a barrier.
template <typename F>
__device__ __forceinline__ double block_sum256(int n, F f, double* red) {
  const int lane = threadIdx.x & 31;
  __syncthreads();
  for (int w = threadIdx.x >> 5; w < 8; w += blockDim.x >> 5) {
    double v = 0.0;
    for (int t = 32 * w + lane; t < n; t += 256) v += f(t);
    v = warp_sum_d(v);
    if (lane == 0) red[w] = v;
  }
  __syncthreads();
  if (threadIdx.x < 32) {
    const double v = warp_sum_d(lane < 8 ? red[lane] : 0.0);
    if (lane == 0) red[0] = v;
  }
  __syncthreads();
  return red[0];
}

// 1/sqrt(d) by the Newton-Raphson iteration r <- r + r (1 - d r^2) / 2 from
// the fp32 estimate (relative error about 2^-22; each step squares it, so two
// steps reach FP64 rounding). On this GPU an FP64 square root or division
// takes about ten dependent FMAs' time; the factorisations below have one of
// each per column on their critical path. Outside the range where the fp32
// estimate is a normal number, the plain expression.
__device__ __forceinline__ double rsqrt_newton(double d) {
  if (!(d > 1e-30 && d < 1e30)) return 1.0 / sqrt(d);
  double r = (double)rsqrtf((float)d);
#pragma unroll
  for (int k = 0; k < 2; ++k) {
    const double h = d * r;
    r = fma(0.5 * r, fma(-h, r, 1.0), r);
  }
  return r;
}

// Exact float -> double by its bit fields (sign, exponent rebiased by
// 1023 - 127 = 896, mantissa shifted into place), on the integer pipe;
// zeros, subnormals, infinities and NaNs take the hardware conversion.
__device__ __forceinline__ double f2d_exact(float x) {
  const uint32_t u = __float_as_uint(x);
  const uint32_t ax = u & 0x7fffffffu;
  if (ax - 0x00800000u >= 0x7f000000u) return (double)x;
  const uint32_t hi = (u & 0x80000000u) | ((ax >> 3) + (896u << 20));
  return __hiloint2double((int)hi, (int)(ax << 29));
}

// (i, j), j <= i, of the packed lower-triangle index e = i (i + 1) / 2 + j
__device__ __forceinline__ void tri_index(int e, int& i, int& j) {
  int r = (int)((sqrtf(8.f * (float)e + 1.f) - 1.f) * 0.5f);
  while (r > 0 && r * (r + 1) / 2 > e) --r;
  while ((r + 1) * (r + 2) / 2 <= e) ++r;
  i = r;
  j = e - r * (r + 1) / 2;
}

// A Gram entry sum_t x_i[t] x_j[t] as four interleaved FP64 chains (t mod 4),
// added pairwise at the end: a quarter of the dependent-FMA latency of one
// chain, and a fixed operation order, so every kernel that forms a Gram entry
// through Dot4 gets the same bits. run() continues the chains over n further
// samples; every run but the last must cover a multiple of 4 samples.
struct Dot4 {
  double s0 = 0.0, s1 = 0.0, s2 = 0.0, s3 = 0.0;
  __device__ __forceinline__ void run(const double* xi, const double* xj, int n) {
    int t = 0;
    for (; t + 4 <= n; t += 4) {
      s0 = fma(xi[t], xj[t], s0);
      s1 = fma(xi[t + 1], xj[t + 1], s1);
      s2 = fma(xi[t + 2], xj[t + 2], s2);
      s3 = fma(xi[t + 3], xj[t + 3], s3);
    }
    if (t < n) s0 = fma(xi[t], xj[t], s0);
    if (t + 1 < n) s1 = fma(xi[t + 1], xj[t + 1], s1);
    if (t + 2 < n) s2 = fma(xi[t + 2], xj[t + 2], s2);
  }
  __device__ __forceinline__ double sum() const { return (s0 + s1) + (s2 + s3); }
};

// In-place right-looking Cholesky of the leading n x n block of M (row stride
// ld, lower triangle used): the pivot's reciprocal square root by
// rsqrt_newton, the column scaled by it, L_kk = d / sqrt(d). rdiag (optional)
// receives 1 / L_kk. Returns false if a pivot is not positive (LAPACK potrf's
// failure test).
__device__ bool block_cholesky(double* M, int n, int ld, int* flag, double* rdiag = nullptr) {
  __shared__ double rk;
  if (threadIdx.x == 0) *flag = 0;
  __syncthreads();
  for (int k = 0; k < n; ++k) {
    if (threadIdx.x == 0) {
      const double d = M[k * ld + k];
      const bool pos = d > 0.0;
      if (!pos) *flag = 1;
      const double r = pos ? rsqrt_newton(d) : 1.0;
      M[k * ld + k] = pos ? d * r : 1.0;
      rk = r;
      if (rdiag) rdiag[k] = r;
    }
    __syncthreads();
    if (*flag) return false;
    const double r = rk;
    for (int i = k + 1 + threadIdx.x; i < n; i += blockDim.x) M[i * ld + k] *= r;
    __syncthreads();
    const int m = n - k - 1;
    for (int idx = threadIdx.x; idx < m * m; idx += blockDim.x) {
      const int i = k + 1 + idx / m, j = k + 1 + idx % m;
      if (j <= i) M[i * ld + j] -= M[i * ld + k] * M[j * ld + k];
    }
    __syncthreads();
  }
  return true;
}

// Li = L^-1 for lower-triangular L (n x n, row stride ld); column-parallel.
// With rdiag (1 / L_ii from block_cholesky) the diagonal divisions of the
// column recursions become products.
__device__ void block_tri_inverse(const double* L, double* Li, int n, int ld, const double* rdiag = nullptr) {
  for (int c = threadIdx.x; c < n; c += blockDim.x) {
    for (int i = 0; i < c; ++i) Li[i * ld + c] = 0.0;
    for (int i = c; i < n; ++i) {
      double s = (i == c) ? 1.0 : 0.0;
      for (int k = c; k < i; ++k) s -= L[i * ld + k] * Li[k * ld + c];
      const double d = L[i * ld + i];
      Li[i * ld + c] = rdiag ? s * rdiag[i] : (d != 0.0 ? s / d : 0.0);
    }
  }
  __syncthreads();
}

// out[n][n] = inv(A_SS + 1e-8 I) for the columns idx[0 .. n) of A = Li' Li
// = (X_w'X_w)^-1: S = A_SS + 1e-8 I (the S slot), its Cholesky factor, that
// factor's inverse (the A slot) and out = inverse' inverse, in FP64. Ends
// with a barrier.
__device__ __forceinline__ void sub_block_inverse(const PairScratch& s, int K, const int* idx, int n, int* flag, float* out) {
  for (int e = threadIdx.x; e < n * n; e += blockDim.x) {
    const int i = e / n, j = e % n;
    const int ti = idx[i], tj = idx[j];
    double acc = 0.0;
    for (int k = max(ti, tj); k < K; ++k) acc += s.Li[k * K + ti] * s.Li[k * K + tj];
    s.S[i * n + j] = acc + (i == j ? 1e-8 : 0.0);
  }
  __syncthreads();
  block_cholesky(s.S, n, n, flag);
  block_tri_inverse(s.S, s.A, n, n);
  for (int e = threadIdx.x; e < n * n; e += blockDim.x) {
    const int i = e / n, j = e % n;
    double acc = 0.0;
    for (int k = max(i, j); k < n; ++k) acc += s.A[k * n + i] * s.A[k * n + j];
    out[e] = (float)acc;
  }
  __syncthreads();
}

struct BuildArgs {
  ffs_grid_desc d;
  ffs_grid_out o;
  // the centring test (ffs_grid_build_centred), or NULL
  int p0;
  int* const_flag;
  float* const_coef;
};

// Reciprocal of n by Newton's iteration r <- r (2 - n r) from the fp32 one
// (error ~2^-24 -> 2^-48 -> below 2^-53), a quarter of the dependent FP64
// operations of a correctly rounded division.
__device__ __forceinline__ double rcp_newton(double n) {
  if (!(n > 1e-30 && n < 1e30)) return 1.0 / n;
  double r = (double)__frcp_rn((float)n);
  r = r * fma(-n, r, 2.0);
  return r * fma(-n, r, 2.0);
}

// Phase 1 of an item: the LDL' of pair p's AR-filtered tridiagonal correlation,
// m_t = T_t,t-1 / D_t-1, D_t = T_tt - m_t T_t,t-1 within each run. D_t is the
// ratio N_t / N_t-1 of the leading minors, which follow the three-term
// recurrence N_t = T_tt N_t-1 - T_t,t-1^2 N_t-2: one dependent FMA per step (64
// cycles of this GPU's FP64 pipe) where the recurrence of D takes a division
// (about 480 cycles with Newton steps), and which a warp can scan in parallel.
// The filter's entries before it and the reciprocals, square roots and outputs
// after it are formed for every sample in parallel, and log|R| = 2 sum log(sqrt(D_t) + 1e-10) telescopes to the
// log of each run's last minor + 2e-10 sum 1/sqrt(D_t) (the next term is 1e-20).
// A minor is a product of the pivots, down to 1e-4 each for (a, b) near 1, so the
// products and the walks over them carry a power of two beside them.
// cc[t], cm[t], cr[t] = c, m, 1/sqrt(D); coef[p], logdet_R[p] written; tmp holds
// 4 T doubles. A run with a pivot D_t that is not positive goes through the
// recurrence of D instead, which replaces it by 1 and sets *bad_r. Ends with a barrier.
__device__ void ldl_of_pair(const ffs_grid_desc& d, const ffs_grid_out& o, int p, double* cc, double* cm, double* cr,
                            double* tmp, double* red, int* bad_r) {
  const int T = d.T;
  const float af = d.a[p], bf = d.b[p];
  const double a = (double)af;
  double *diag = tmp, *off2 = tmp + T, *num = tmp + 2 * T, *prev = tmp + 3 * T;
  if (threadIdx.x == 0) {
    *bad_r = 0;
    red[0] = d.lambda_fp32 ? (double)lambda_f32(af, bf) : lambda_f64(a, (double)bf);
  }
  __syncthreads();
  const double lam = red[0];
  // lambda == 0: every lag correlation is zero, R = I exactly
  const bool ident = lam == 0.0;
  for (int t = threadIdx.x; t < T; t += blockDim.x) {
    double c = 0.0, off = 0.0, dg = 1.0;
    bool start = t == 0;
    for (int r = 1; r < d.n_runs && !start; ++r) start = d.run_start[r] == t;
    if (!start && !ident) {
      const int gap = d.tau[t] - d.tau[t - 1];
      // a^gap and a^(gap - 1) of small integer gaps by products (a^1 = a and
      // a^0 = 1 exactly)
      double ag1 = 1.0;
      if (gap <= 16) {
        for (int k = 1; k < gap; ++k) ag1 *= a;
      } else {
        ag1 = pow(a, (double)(gap - 1));
      }
      const double rho = lam * ag1;
      c = ag1 * a;
      dg = 1.0 + c * c - 2.0 * c * rho;
      off = rho - c;
    }
    cc[t] = c;
    cm[t] = off;
    diag[t] = dg;
    off2[t] = off * off;
  }
  __syncthreads();
  // a warp per run: N_t, N_t-1 = A_t ... A_t0 (1, 1) with A_t = [T_tt, -off2; 1, 0].
  // Each lane multiplies the matrices of its stretch, a scan over the lanes
  // gives the minors before each stretch, and the lane walks it from there.
  // (A warp has one FP64 instruction in flight, 64 cycles each: about 80 of
  // them for a run of 200, where a walk by one lane takes 400.) A run's log goes to
  // off2 of its first sample, which its warp has read by then.
  const int lane = threadIdx.x & 31;
  for (int r = threadIdx.x >> 5; r < d.n_runs && !ident; r += blockDim.x >> 5) {
    const int t0 = d.run_start[r], t1 = d.run_start[r + 1];
    const int seg = (t1 - t0 + 31) >> 5;
    const int s0 = min(t1, t0 + lane * seg), s1 = min(t1, s0 + seg);
    double a0 = 1.0, a1 = 0.0, b0 = 0.0, b1 = 1.0;  // columns (a0, b0) and (a1, b1) of the product
    int ex = 0;                                     // its scale, 2^ex
    auto rescale = [&](double lead) {
      const int e = ((__double2hiint(lead) >> 20) & 0x7ff) - 1023;
      if (e > 64 || e < -64) {
        const double sc = __hiloint2double((1023 - e) << 20, 0);
        a0 *= sc;
        a1 *= sc;
        b0 *= sc;
        b1 *= sc;
        ex += e;
      }
    };
    for (int t = s0; t < s1; ++t) {
      const double dg = diag[t], of = off2[t];
      const double na = fma(dg, a0, -(of * b0)), nb = fma(dg, a1, -(of * b1));
      b0 = a0;
      b1 = a1;
      a0 = na;
      a1 = nb;
      if (((t - s0) & 7) == 7) rescale(a0);
    }
    for (int o2 = 1; o2 < 32; o2 <<= 1) {  // inclusive: this lane's product times those before it
      const double p0 = __shfl_up_sync(0xffffffffu, a0, o2), p1 = __shfl_up_sync(0xffffffffu, a1, o2);
      const double q0 = __shfl_up_sync(0xffffffffu, b0, o2), q1 = __shfl_up_sync(0xffffffffu, b1, o2);
      const int pe = __shfl_up_sync(0xffffffffu, ex, o2);
      if (lane >= o2) {
        const double c0 = fma(a0, p0, a1 * q0), c1 = fma(a0, p1, a1 * q1);
        const double e0 = fma(b0, p0, b1 * q0), e1 = fma(b0, p1, b1 * q1);
        a0 = c0;
        a1 = c1;
        b0 = e0;
        b1 = e1;
        ex += pe;
        rescale(a0);
      }
    }
    // (N, N of the step before) entering this lane's stretch; off2 = 0 at the
    // run's start, so the second entry of the start vector is not read
    double n1 = __shfl_up_sync(0xffffffffu, a0 + a1, 1), n0 = __shfl_up_sync(0xffffffffu, b0 + b1, 1);
    int e2 = __shfl_up_sync(0xffffffffu, ex, 1);
    if (lane == 0) {
      n1 = n0 = 1.0;
      e2 = 0;
    }
    bool bad = false;
    for (int t = s0; t < s1; ++t) {
      const double n = fma(diag[t], n1, -(off2[t] * n0));
      num[t] = n;
      prev[t] = n1;
      const int hi = __double2hiint(n);
      bad = bad || hi <= 0 || hi >= 0x7ff00000;  // not positive, or not finite
      n0 = n1;
      n1 = n;
      const int e = (hi >> 20) - 1023;
      if (((t - s0) & 7) == 7 && !bad && (e > 64 || e < -64)) {
        const double sc = __hiloint2double((1023 - e) << 20, 0);
        n0 *= sc;
        n1 *= sc;
        e2 += e;
      }
    }
    __syncwarp();  // a walk by lane 0 rewrites num and prev
    if (!__any_sync(0xffffffffu, bad)) {
      if (s1 == t1 && s0 < s1) off2[t0] = log(n1) + (double)e2 * 0.693147180559945309417;
    } else if (lane == 0) {  // R is singular or not a correlation
      double D = 1.0, ld = 0.0;
      for (int t = t0; t < t1; ++t) {
        D = diag[t] - off2[t] / D;
        if (!(D > 0.0)) {
          *bad_r = 1;
          D = 1.0;
        }
        num[t] = D;
        prev[t] = 1.0;
        ld += log(D);
      }
      off2[t0] = ld;
    }
  }
  __syncthreads();
  for (int t = threadIdx.x; t < T; t += blockDim.x) {
    double id = 1.0, rs = 1.0;
    if (!ident && num[t] != prev[t]) {  // else D_t = 1
      id = prev[t] * rcp_newton(num[t]);  // 1 / D_t
      rs = id * rsqrt_newton(id);
    }
    diag[t] = id;
    cr[t] = rs;
  }
  const double rsum = block_sum256(T, [&](int t) { return cr[t]; }, red);  // its barriers order diag
  for (int t = threadIdx.x; t < T; t += blockDim.x) {
    const double m = t > 0 ? cm[t] * diag[t - 1] : 0.0;
    cm[t] = m;
    reinterpret_cast<float4*>(o.coef)[(size_t)p * T + t] =
        make_float4((float)cc[t], (float)m, (float)diag[t], (float)cr[t]);
  }
  if (threadIdx.x == 0) {
    double ld = 2e-10 * rsum;
    for (int r = 0; r < d.n_runs && !ident; ++r)
      if (d.run_start[r] < d.run_start[r + 1]) ld += off2[d.run_start[r]];
    o.logdet_R[p] = ld;
  }
  __syncthreads();
}

__device__ __forceinline__ void bar_sync(int id, int n) {
  asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(n) : "memory");
}

// Rows or columns of the band staged at a time by phases 2 and 6.
constexpr int BD_STEPS = 32;

__host__ __device__ inline int band_pitch(int W) { return W | 1; }
// Runs factored side by side, each by half the block's warps: the chain of a
// column's steps, not their work, takes the time. Two windows of W > 96 would
// not leave room for the rest.
__host__ __device__ inline int band_groups(int W, int n_runs) { return n_runs > 1 && W <= 96 ? 2 : 1; }
// Shared doubles: the staged rows or columns of phases 2 and 6, and phase 1's
// powers of a, index table, and per group a window and two columns (each raw and scaled).
__host__ __device__ inline size_t band_stage_doubles(int W) { return (size_t)BD_STEPS * band_pitch(W); }
__host__ __device__ inline size_t band_chol_doubles(int W, int n_runs) {
  const size_t n = (size_t)(W + 1) + band_groups(W, n_runs) * ((size_t)W * W + 4 * (size_t)W) +
                   ((size_t)W * (W + 1) / 2 + 3) / 4;
  return n > band_stage_doubles(W) ? n : band_stage_doubles(W);
}

// d > 0, by the words (a compare on the FP64 pipe takes as long as a product)
__device__ __forceinline__ bool positive(double d) {
  const int hi = __double2hiint(d);
  return hi > 0 ? hi < 0x7ff00000 || (hi == 0x7ff00000 && __double2loint(d) == 0) : hi == 0 && __double2loint(d) != 0;
}

// The factors of v / n = u + u p, u = v r: r the fp32 reciprocal of n and p = e + e^2,
// e = 1 - n r, the cubic form of the reciprocal's Newton iteration (Householder's; error
// e^3 ~ 2^-72). Positive n.
__device__ __forceinline__ void rcp_factors(double n, double& r, double& p) {
  const unsigned x = (unsigned)__double2hiint(n) >> 20;
  r = x - (1023u - 100u) <= 200u ? f2d_exact(__frcp_rn((float)n)) : 1.0 / n;  // 2^-100 < n < 2^100
  const double e = fma(-n, r, 1.0);
  p = fma(e, e, e);
}

// Phase 1 of an item with AFNI's banded R (d.band): the Cholesky factor of
// each run's block of R, where R(t, k) = lam a^(g-1) for 1 <= g = tau_t -
// tau_k <= band[p] and 0 beyond. The rows of run r that column k reaches are
// contiguous, k+1 .. end-1, and the fill stays inside the band, so the column
// goes rightwards over a window of the last W rows in shared memory (row t in
// slot t mod W, entry (t, t - j) at j): A(i, j) -= A(i, k) A(j, k) / D_k.
// Warps 1.. update the window's triangle, one entry per lane through a table
// of triangle indices (full warps: this GPU's FP64 pipe takes 19 cycles per
// warp instruction whatever its lanes), and set up the rows that enter;
// meanwhile warp 0 forms the next column with its pivot's reciprocal, so a
// step costs one barrier and a chain of pivot, fp32 reciprocal, its two
// correction terms and the scaling. The columns leave unscaled; the square roots,
// L(t, t - j) = A(t, t - j) / sqrt(D_{t-j}), the fp32 whitening coefficients
// and the logs follow for all entries in parallel. A pivot that is not
// positive flags the pair (bad_r) and is replaced by 1.
// FP64 throughout; band_L keeps the factor (zero outside a row's band),
// band_coef its fp32 whitening coefficients, invdiag [T] (global scratch) the
// reciprocal diagonal for phases 2 and 6. logdet_R = 2 sum log(L(t, t) +
// 1e-10) as the reference takes it from its dense factor; coef is the
// identity. The row-by-row form it replaces (a warp per run, every entry of a row
// waiting for the one before through global memory) took most of the banded
// build's 3110 us at T = 240, K = 11, 117 pairs of up to 42 lags; with phases 2
// and 6 below the build takes 398 (this phase 150, phase 2 85, phase 6 105).
// sm: band_chol_doubles shared doubles; invdiag: 1.5 T doubles
// (each column's reach behind the diagonal). Ends with a barrier.
__device__ __noinline__ void band_chol_of_pair(const ffs_grid_desc& d, const ffs_grid_out& o, int p, double* invdiag,
                                               double* sm, double* red, int* bad_r) {
  __builtin_assume(__isShared(sm));
  const int T = d.T, W = d.band_w, bw = d.band[p];
  const float af = d.a[p], bf = d.b[p];
  const double a = (double)af;
  const double lam = d.lambda_fp32 ? (double)lambda_f32(af, bf) : lambda_f64(a, (double)bf);
  const bool zero = lam == 0.0;
  const int* __restrict__ tau = d.tau;
  double* Lb = o.band_L + (size_t)p * T * W;
  float* Cb = o.band_coef + (size_t)p * T * W;
  const int ng = band_groups(W, d.n_runs), gw = (int)(blockDim.x >> 5) / ng;  // groups, warps of a group
  const int grp = (int)(threadIdx.x >> 5) / gw, gtid = threadIdx.x - grp * gw * 32, gwarp = gtid >> 5;
  double *apow = sm, *win = apow + W + 1 + grp * (W * W + 4 * W), *colA = win + (size_t)W * W, *colW = colA + 2 * W;
  uint16_t* tri = reinterpret_cast<uint16_t*>(apow + W + 1 + ng * (W * W + 4 * W));
  int* reach = reinterpret_cast<int*>(invdiag + T);  // first row past column t's band
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nw = blockDim.x >> 5;
  if (tid == 0) {
    *bad_r = 0;
    double x = 1.0;
    for (int k = 0; k <= W; ++k) {  // lam a^k: corr(g) = lam a^(g - 1), 1 <= g < W
      apow[k] = zero ? 0.0 : lam * x;
      x *= a;
    }
  }
  for (int i = warp; i < W; i += nw)
    for (int j = lane; j <= i; j += 32) tri[i * (i + 1) / 2 + j] = (uint16_t)(i << 8 | j);
  for (int r = 0; r < d.n_runs; ++r)
    for (int t = d.run_start[r] + tid; t < d.run_start[r + 1]; t += blockDim.x) {
      int lo = t + 1, hi = min(t + bw + 1, d.run_start[r + 1]);
      while (lo < hi) {
        const int mid = (lo + hi) >> 1;
        if (tau[mid] - tau[t] <= bw)
          lo = mid + 1;
        else
          hi = mid;
      }
      reach[t] = lo;
    }
  __syncthreads();

  for (int r = grp; r < d.n_runs; r += ng) {
    const int t0 = d.run_start[r], t1 = d.run_start[r + 1];
    int end = t0, cur = 0, slot1 = t0 % W;  // "column t0 - 1" reaches nothing: the first turn sets up column t0
    int nend = t0 < t1 ? reach[t0] : t0;
    for (int k = t0 - 1; k < t1 - 1; ++k) {
      const double *cA = colA + cur * W, *cW = colW + cur * W;
      const int C = end - 1 - k;  // rows k+1 .. k+C; row k + 1 in slot1
      const int nnend = k + 2 < t1 ? reach[k + 2] : 0;
      auto slot = [&](int i) { return slot1 + i >= W ? slot1 + i - W : slot1 + i; };  // of row k + 1 + i
      if (gwarp == 0) {  // column k + 1: its entries less column k's share
        double *nA = colA + (cur ^ 1) * W, *nW = colW + (cur ^ 1) * W;
        const bool seen = C >= 1;  // row k + 1 is in the window
        const double a1 = seen ? cA[1] : 0.0;
        double dk = 1.0;
        if (seen) dk = fma(-cW[1], a1, win[slot1 * W]);
        if (!positive(dk)) {
          if (lane == 0) *bad_r = 1;
          dk = 1.0;
        }
        double rk, pk;
        rcp_factors(dk, rk, pk);
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          if (k + 2 + 32 * q >= nend) break;
          const int i = 1 + lane + 32 * q, t = k + 1 + i;
          if (t < nend) {
            const double v = t < end ? fma(-cW[i + 1], a1, win[slot(i) * W + i]) : apow[tau[t] - tau[k + 1] - 1];
            nA[i] = v;
            const double u = v * rk;
            nW[i] = fma(u, pk, u);
            Lb[(size_t)t * W + i] = v;
          }
        }
        if (lane == 0) invdiag[k + 1] = dk;
      } else {
        const int m = max(C - 1, 0);
        for (int e = gtid - 32; e < m * (m + 1) / 2; e += 32 * (gw - 1)) {
          const int ij = tri[e], i = ij >> 8, j = ij & 255;  // row k+2+i, column k+2+j
          double* w = win + slot(i + 1) * W + (i - j);
          *w = fma(-cW[i + 2], cA[j + 2], *w);
        }
        for (int t = max(end, k + 2) + gwarp - 1; t < nend; t += gw - 1) {  // rows that enter, from column k + 2
          const int tt = tau[t];
          for (int j = lane; j <= t - (k + 2); j += 32) {
            const int g = tt - tau[t - j];
            if (g <= bw) win[slot(t - k - 1) * W + j] = j == 0 ? 1.0 : apow[g - 1];
          }
        }
      }
      end = nend;
      nend = nnend;
      cur ^= 1;
      slot1 = slot1 + 1 == W ? 0 : slot1 + 1;
      bar_sync(1 + grp, 32 * gw);
    }
  }
  __syncthreads();

  double ld = 0.0;
  for (int t = tid; t < T; t += blockDim.x) {
    const double ltt = sqrt(invdiag[t]);
    ld += 2.0 * log(ltt + 1e-10);
    invdiag[t] = 1.0 / ltt;
    Lb[(size_t)t * W] = ltt;
    reinterpret_cast<float4*>(o.coef)[(size_t)p * T + t] = make_float4(0.f, 0.f, 1.f, 1.f);
  }
  ld = block_sum(ld, red);
  if (tid == 0) o.logdet_R[p] = ld;
  __syncthreads();
  constexpr int ROWS = 4;  // rows in flight per warp
  for (int r = 0; r < d.n_runs; ++r) {
    const int t0 = d.run_start[r], t1 = d.run_start[r + 1];
    for (int tb = t0 + warp; tb < t1; tb += ROWS * nw)
      for (int j = lane; j < W; j += 32) {
        double l[ROWS], it[ROWS];
#pragma unroll
        for (int q = 0; q < ROWS; ++q) {
          const int t = tb + q * nw;
          const bool in = t < t1 && j >= 1 && t - j >= t0 && reach[t - j] > t;
          it[q] = t < t1 ? invdiag[t] : 0.0;
          l[q] = in ? Lb[(size_t)t * W + j] * invdiag[t - j] : 0.0;
        }
#pragma unroll
        for (int q = 0; q < ROWS; ++q) {
          const int t = tb + q * nw;
          if (t < t1) {
            if (j >= 1) Lb[(size_t)t * W + j] = l[q];
            Cb[(size_t)t * W + j] = (float)(j == 0 ? it[q] : l[q] * it[q]);
          }
        }
      }
  }
  __syncthreads();
}

// Phase 2 with the band: X_w = L^-1 X, half a warp per column of X, rightwards.
// Lane l of the half holds the column's rows k0 + l + 16 q of the running 16
// steps; step k broadcasts row k and takes L(t, k) / L(k, k) times it off the
// rows below, so the dependent chain of a step is one shuffle and one fma (the
// leftward form, a dot product per row, waits for a whole row). Half warps
// because the FP64 pipe's time goes by warp instructions: a band of 42 fills 42
// of the 50 lanes a column then takes. The columns of BD_STEPS steps are staged
// in shared memory for all the block's warps. NQ >= bw / 16 + 2. Whole blocks
// only; ends with a barrier.
template <int NQ>
__device__ __noinline__ void band_whiten_cols(const double* Lb, const double* invd, const float* __restrict__ Xd,
                                              double* Xw, double* st, int T, int K, int W, int bw) {
  __builtin_assume(__isShared(st));
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5, pitch = band_pitch(W);
  const int l16 = lane & 15;
  for (int c0 = 0; c0 < K; c0 += 2 * nw) {
    const int c = c0 + 2 * warp + (lane >> 4);
    const bool live = c < K;
    double x[NQ];
#pragma unroll
    for (int q = 0; q < NQ; ++q) {
      const int t = l16 + 16 * q;
      x[q] = live && t < T ? f2d_exact(__ldg(Xd + (size_t)t * K + c)) : 0.0;
    }
    for (int k0 = 0; k0 < T; k0 += 16) {
      if (k0 % BD_STEPS == 0) {
        __syncthreads();
        for (int tb = k0 + 1 + warp; tb < k0 + BD_STEPS + bw; tb += 4 * nw)
          for (int j = lane + 1; j <= bw; j += 32) {
            double l[4];
#pragma unroll
            for (int q = 0; q < 4; ++q) {
              const int t = tb + q * nw, k = t - j;
              l[q] = t < T && k >= k0 && k < k0 + BD_STEPS ? Lb[(size_t)t * W + j] * invd[k] : 0.0;
            }
#pragma unroll
            for (int q = 0; q < 4; ++q) {
              const int k = tb + q * nw - j;
              if (k >= k0 && k < k0 + BD_STEPS) st[(k - k0) * pitch + j] = l[q];
            }
          }
        __syncthreads();
      }
      if (c0 + 2 * warp < K) {
        const int n = min(16, T - k0);
        const double* row = st + (k0 % BD_STEPS) * pitch + l16;
#pragma unroll 4
        for (int kk = 0; kk < n; ++kk, row += pitch - 1) {  // row[16 q] = step kk's entry i = l16 + 16 q - kk
          const double xk = __shfl_sync(0xffffffffu, x[0], kk, 16);
#pragma unroll
          for (int q = 0; q < NQ; ++q) {
            if (16 * q - kk > bw) break;  // no lane's row is in reach
            const int i = l16 + 16 * q - kk;
            if (i >= 1 && i <= bw) x[q] = fma(-row[16 * q], xk, x[q]);
          }
        }
        const int t = k0 + l16, tn = t + 16 * NQ;
        if (live && t < T) Xw[(size_t)c * T + t] = x[0] * invd[t];
#pragma unroll
        for (int q = 0; q < NQ - 1; ++q) x[q] = x[q + 1];
        x[NQ - 1] = live && tn < T ? f2d_exact(__ldg(Xd + (size_t)tn * K + c)) : 0.0;
      }
    }
  }
  __syncthreads();
}

// Phase 6 with the band: U = L^-T Q by back substitution, u_t = (q_t - sum_i
// L(t + i, t) u_{t+i}) / L(t, t) with the u of fp32, leftwards as phase 2 goes
// rightwards (lane l holds rows k0 + l - 16 q; rows of L staged). Returns max
// |u| of the thread's entries. Whole blocks only; ends with a barrier.
template <int NQ>
__device__ __noinline__ float band_back_cols(const double* Lb, const double* invd, const float* qf, float* uf, float* U,
                                             double* st, int T, int LT, int K, int W, int bw) {
  __builtin_assume(__isShared(st));
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5, pitch = band_pitch(W);
  const int l16 = lane & 15;
  float umax = 0.f;
  for (int c0 = 0; c0 < K; c0 += 2 * nw) {
    const int c = c0 + 2 * warp + (lane >> 4);
    const bool live = c < K;
    const int top = (T - 1) / 16 * 16;
    double x[NQ];
#pragma unroll
    for (int q = 0; q < NQ; ++q) {
      const int t = top + l16 - 16 * q;
      x[q] = live && t >= 0 && t < T ? f2d_exact(qf[(size_t)c * T + t]) : 0.0;
    }
    for (int k0 = top; k0 >= 0; k0 -= 16) {
      if (k0 == top || (k0 + 16) % BD_STEPS == 0) {
        const int s0 = k0 / BD_STEPS * BD_STEPS;
        __syncthreads();
        for (int kb = warp; kb < BD_STEPS; kb += 4 * nw)
          for (int j = lane + 1; j <= bw; j += 32) {
            double l[4];
#pragma unroll
            for (int q = 0; q < 4; ++q) {
              const int kk = kb + q * nw;
              l[q] = kk < BD_STEPS && s0 + kk < T ? Lb[(size_t)(s0 + kk) * W + j] : 0.0;
            }
#pragma unroll
            for (int q = 0; q < 4; ++q)
              if (kb + q * nw < BD_STEPS) st[(kb + q * nw) * pitch + j] = l[q];
          }
        __syncthreads();
      }
      if (c0 + 2 * warp < K) {
        const int t = k0 + l16, n = min(16, T - k0);
        const double iv = t < T ? invd[t] : 0.0;
        const double* row = st + (k0 % BD_STEPS + n - 1) * pitch + (n - 1) - l16;
#pragma unroll 4
        for (int kk = n - 1; kk >= 0; --kk, row -= pitch + 1) {  // row[16 q] = step kk's entry i = kk - l16 + 16 q
          const double ut = f2d_exact(__shfl_sync(0xffffffffu, (float)(x[0] * iv), kk, 16));
#pragma unroll
          for (int q = 0; q < NQ; ++q) {
            if (kk - 15 + 16 * q > bw) break;
            const int i = kk - l16 + 16 * q;
            if (i >= 1 && i <= bw) x[q] = fma(-row[16 * q], ut, x[q]);
          }
        }
        if (live && t < T) {
          const float ut = (float)(x[0] * iv);
          uf[(size_t)c * T + t] = ut;
          U[(size_t)c * LT + t] = ut;
          umax = fmaxf(umax, fabsf(ut));
        }
        const int tn = t - 16 * NQ;
#pragma unroll
        for (int q = 0; q < NQ - 1; ++q) x[q] = x[q + 1];
        x[NQ - 1] = live && tn >= 0 ? f2d_exact(qf[(size_t)c * T + tn]) : 0.0;
      }
    }
    if (live)
      for (int t = T + l16; t < LT; t += 16) U[(size_t)c * LT + t] = 0.f;
  }
  __syncthreads();
  return umax;
}

// Phase 1 of every pair once, for the items of all designs (coef and
// logdet_R depend on the pair only): c, m and 1/sqrt(D) ([P][3][T], stride 4 T
// per pair) and bad [P] in the workspace, read back by the item kernels. With
// the banded R the pair's band_L, band_coef, coef and logdet_R are written here,
// and the workspace keeps the reciprocal diagonal (the first T doubles).
__global__ void __launch_bounds__(GB_THREADS) pair_ldl_kernel(BuildArgs args, double* cm, int* bad) {
  __shared__ double red[32];
  __shared__ int bad_r;
  extern __shared__ double cms[];  // 4 T doubles, or with the band as band_chol_of_pair lays it out
  const int T = args.d.T;
  double* dst = cm + (size_t)blockIdx.x * 4 * T;
  if (args.d.band)
    band_chol_of_pair(args.d, args.o, blockIdx.x, dst, cms, red, &bad_r);
  else
    ldl_of_pair(args.d, args.o, blockIdx.x, dst, dst + T, dst + 2 * T, cms, red, &bad_r);
  if (threadIdx.x == 0) bad[blockIdx.x] = bad_r;
}

// The centring test of a design at its identity pair, where X_w = X: c =
// (X'X)^-1 X'1 from the inverse factor Li (row stride ldi), accepted when
// ||X c - 1||^2 <= 1e-12 T; *const_flag stays 1 only if every design passes.
// w: 2 K doubles of scratch (a slot's A, whose K x K doubles the S of the same
// size follows: S alone is too short at K = 1). Ends with a barrier.
__device__ void const_of_design(const BuildArgs& args, int dsg, const float* Xd, const double* Li, int ldi, bool chol,
                                double* w, double* red) {
  const int T = args.d.T, K = args.d.K;
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = blockDim.x >> 5;
  __syncthreads();
  for (int j = wid; j < K; j += nw) {  // X'1
    double x = 0.0;
    for (int t = lane; t < T; t += 32) x += f2d_exact(Xd[(size_t)t * K + j]);
    x = warp_sum_d(x);
    if (lane == 0) w[K + j] = x;
  }
  __syncthreads();
  for (int k = threadIdx.x; k < K; k += blockDim.x) {  // Lx^-1 X'1
    double x = 0.0;
    for (int j = 0; j <= k; ++j) x = fma(Li[k * ldi + j], w[K + j], x);
    w[k] = x;
  }
  __syncthreads();
  for (int j = threadIdx.x; j < K; j += blockDim.x) {
    double x = 0.0;
    for (int k = j; k < K; ++k) x = fma(Li[k * ldi + j], w[k], x);
    w[K + j] = x;
  }
  __syncthreads();
  double part = 0.0;
  for (int t = threadIdx.x; t < T; t += blockDim.x) {
    double r = -1.0;
    for (int j = 0; j < K; ++j) r = fma(f2d_exact(Xd[(size_t)t * K + j]), w[K + j], r);
    part = fma(r, r, part);
  }
  const double ss = block_sum(part, red);
  const bool ok = chol && ss <= 1e-12 * (double)T;
  for (int j = threadIdx.x; j < K; j += blockDim.x) args.const_coef[(size_t)dsg * K + j] = ok ? (float)w[K + j] : 0.f;
  if (threadIdx.x == 0 && !ok) atomicAnd(args.const_flag, 0);
  __syncthreads();
}

// The end of an item: Gsum = G' 1 accumulated in FP64, the task-column F
// matrix inv(A_task + 1e-8 I), the column sets' and the GLT variances c A c',
// from s.Li with the scratch s.S and s.A. Starts and ends with a barrier.
__device__ void item_tail(const ffs_grid_desc& d, const ffs_grid_out& o, const PairScratch& s, int pd, double* red,
                          int* flag_s) {
  const int T = d.T, K = d.K, LT = ld_t(T);
  int& flag = *flag_s;
  __syncthreads();
  if (o.Gsum) {
    for (int j = threadIdx.x; j < K; j += blockDim.x) {
      double acc = 0.0;
      for (int t = 0; t < T; ++t) acc += (double)o.G[((size_t)pd * K + j) * LT + t];
      o.Gsum[(size_t)pd * K + j] = (float)acc;
    }
  }

  // ---- 9. task-column F matrix inv(A_task + 1e-8 I) and GLT variances c A c'
  const int nt = d.n_task;
  if (d.n_glt > 0 && o.glt_var) {  // c A c' = ||Lx^-1 c||^2
    for (int c = 0; c < d.n_glt; ++c) {
      const float* gc = d.glt + (size_t)c * K;
      double part = 0.0;
      for (int k = threadIdx.x; k < K; k += blockDim.x) {
        double w = 0.0;
        for (int j = 0; j <= k; ++j) w += s.Li[k * K + j] * (double)gc[j];
        part += w * w;
      }
      const double v = block_sum(part, red);
      if (threadIdx.x == 0) o.glt_var[(size_t)pd * d.n_glt + c] = (float)v;
    }
  }
  // the task block, then the column sets' blocks one after another
  const int has_task = nt > 0 && o.Ftask ? 1 : 0;
  const int nsets = o.Fsets ? d.n_sets : 0;
  size_t msum = 0, off = 0;
  for (int g = 0; g < nsets; ++g) {
    const size_t q = (size_t)(d.set_ptr[g + 1] - d.set_ptr[g]);
    msum += q * q;
  }
  for (int bk = 0; bk < has_task + nsets; ++bk) {
    const bool task = bk < has_task;
    const int g = bk - has_task;
    const int n = task ? nt : d.set_ptr[g + 1] - d.set_ptr[g];
    const int* idx = task ? d.task_idx : d.set_idx + d.set_ptr[g];
    float* out = task ? o.Ftask + (size_t)pd * nt * nt : o.Fsets + (size_t)pd * msum + off;
    sub_block_inverse(s, K, idx, n, &flag, out);
    if (!task) off += (size_t)n * n;
  }
  __syncthreads();
}

// Phases 2 to 9 of one item with its matrices in the global scratch slot s,
// after phase 1: cc, cm, cr as ldl_of_pair leaves them, or with the banded R cc
// = the reciprocal diagonal and stage = band_stage_doubles shared doubles. Any K and T.
template <bool BAND>
__device__ __noinline__ void item_global(const BuildArgs& args, const PairScratch& s, int p, int pd, const float* Xd,
                                         const double* cc, const double* cm, const double* cr, double* stage,
                                         int bad_r, double* red, int* flag_s) {
  const ffs_grid_desc& d = args.d;
  const ffs_grid_out& o = args.o;
  const int T = d.T, K = d.K, LT = ld_t(T);
  int& flag = *flag_s;

  // ---- 2. X_w = L^-1 X, one column per thread; the design samples of
  // GB_PF steps are loaded ahead of the recursion that needs them
  if constexpr (BAND) {
    const int bw = d.band[p];
    const double* Lb = o.band_L + (size_t)p * T * d.band_w;
    if (bw <= 16)
      band_whiten_cols<3>(Lb, cc, Xd, s.Xw, stage, T, K, d.band_w, bw);
    else if (bw <= 48)
      band_whiten_cols<5>(Lb, cc, Xd, s.Xw, stage, T, K, d.band_w, bw);
    else
      band_whiten_cols<10>(Lb, cc, Xd, s.Xw, stage, T, K, d.band_w, bw);
  }
  for (int j = threadIdx.x; j < K && !BAND; j += blockDim.x) {
    double xp = 0.0, vp = 0.0;
    for (int t0 = 0; t0 < T; t0 += GB_PF) {
      float xb[GB_PF];
#pragma unroll
      for (int k = 0; k < GB_PF; ++k) xb[k] = t0 + k < T ? __ldg(Xd + (size_t)(t0 + k) * K + j) : 0.f;
#pragma unroll
      for (int k = 0; k < GB_PF; ++k) {
        const int t = t0 + k;
        if (t < T) {
          const double x = f2d_exact(xb[k]);
          const double z = x - cc[t] * xp;
          const double v = z - cm[t] * vp;
          s.Xw[(size_t)j * T + t] = v * cr[t];
          xp = x;
          vp = v;
        }
      }
    }
  }
  __syncthreads();

  // ---- 3. X_w'X_w (full symmetric) into Lx, and the fp32 copy: one thread
  // per lower-triangle entry (full warps), four chains each
  for (int e = threadIdx.x; e < K * (K + 1) / 2; e += blockDim.x) {
    int i, j;
    tri_index(e, i, j);
    Dot4 acc;
    acc.run(s.Xw + (size_t)i * T, s.Xw + (size_t)j * T, T);
    const double v = acc.sum();
    s.Lx[i * K + j] = v;
    s.Lx[j * K + i] = v;
    o.XtX[(size_t)pd * K * K + i * K + j] = (float)v;
    o.XtX[(size_t)pd * K * K + j * K + i] = (float)v;
  }
  __syncthreads();

  // ---- 4. Cholesky of X_w'X_w, QR (modified Gram-Schmidt, twice) otherwise
  // 1 / diag(Lx) goes to the A slot, free until phase 9
  int info = 0;
  const bool chol = block_cholesky(s.Lx, K, K, &flag, s.A);
  if (!chol) {
    info = 1;
    // Q and R from X_w; Lx := R' (lower), so that X_w'X_w = Lx Lx'.
    for (int idx = threadIdx.x; idx < K * K; idx += blockDim.x) s.Lx[idx] = 0.0;
    __syncthreads();
    for (int j = 0; j < K; ++j) {
      double* q = s.Qm + (size_t)j * T;
      for (int t = threadIdx.x; t < T; t += blockDim.x) q[t] = s.Xw[(size_t)j * T + t];
      __syncthreads();
      for (int pass = 0; pass < 2; ++pass) {
        for (int i = 0; i < j; ++i) {
          const double* qi = s.Qm + (size_t)i * T;
          const double rij = block_sum256(T, [&](int t) { return qi[t] * q[t]; }, red);
          for (int t = threadIdx.x; t < T; t += blockDim.x) q[t] -= rij * qi[t];
          if (threadIdx.x == 0) s.Lx[j * K + i] += rij;
          __syncthreads();
        }
      }
      const double nrm = sqrt(block_sum256(T, [&](int t) { return q[t] * q[t]; }, red));
      const double inv = nrm > 0.0 ? 1.0 / nrm : 0.0;
      for (int t = threadIdx.x; t < T; t += blockDim.x) q[t] *= inv;
      if (threadIdx.x == 0) s.Lx[j * K + j] = nrm;
      __syncthreads();
    }
  }
  if (bad_r) info = 2;
  __syncthreads();

  if (threadIdx.x == 0) {
    double ld = 0.0;
    for (int j = 0; j < K; ++j) ld += 2.0 * log(fabs(s.Lx[j * K + j]) + 1e-10);
    o.logdet_XtX[pd] = ld;
    o.info[pd] = info;
  }

  // ---- 5. Q = X_w Lx^-T in fp32 (Q, U and G only leave as fp32 or fp16
  // splits; the factorisation and the logdets above stay FP64). The two [K][T]
  // FP64 slots are reused as fp32 arrays; the QR fallback converts its Q.
  float* const xw_f = reinterpret_cast<float*>(s.Xw);
  float* const qm_f = reinterpret_cast<float*>(s.Qm);
  float* const lx_f = reinterpret_cast<float*>(s.S);  // [K][K] Lx, then Li in lx_f + K*K
  float* qf;
  float* uf;
  for (int idx = threadIdx.x; idx < K * K; idx += blockDim.x) lx_f[idx] = (float)s.Lx[idx];
  __syncthreads();
  if (info != 1) {
    for (int t = threadIdx.x; t < T; t += blockDim.x) {
      for (int j = 0; j < K; ++j) {
        float acc = (float)s.Xw[(size_t)j * T + t];
        for (int i = 0; i < j; ++i) acc = fmaf(-lx_f[j * K + i], qm_f[(size_t)i * T + t], acc);
        qm_f[(size_t)j * T + t] = acc / lx_f[j * K + j];
      }
    }
    qf = qm_f;
    uf = xw_f;
  } else {
    for (int idx = threadIdx.x; idx < K * T; idx += blockDim.x) xw_f[idx] = (float)s.Qm[idx];
    qf = xw_f;
    uf = qm_f;
  }
  __syncthreads();

  // ---- 6. U = L^-T Q = A' L~^-T D^-1/2 Q (backward recursions) in fp32, with
  // the fp32 coefficients of phase 1
  const float4* cf = reinterpret_cast<const float4*>(o.coef) + (size_t)p * T;
  float umax_local = 0.f;
  if constexpr (BAND) {
    const int bw = d.band[p];
    const double* Lb = o.band_L + (size_t)p * T * d.band_w;
    float* U = o.U + (size_t)pd * K * LT;
    if (bw <= 16)
      umax_local = band_back_cols<3>(Lb, cc, qf, uf, U, stage, T, LT, K, d.band_w, bw);
    else if (bw <= 48)
      umax_local = band_back_cols<5>(Lb, cc, qf, uf, U, stage, T, LT, K, d.band_w, bw);
    else
      umax_local = band_back_cols<10>(Lb, cc, qf, uf, U, stage, T, LT, K, d.band_w, bw);
  }
  for (int j = threadIdx.x; j < K && !BAND; j += blockDim.x) {
    const float* q = qf + (size_t)j * T;
    float* u = uf + (size_t)j * T;
    float xn = 0.f, mn = 0.f, cn = 0.f;  // x_{t+1}, m_{t+1}, c_{t+1}
    for (int t1 = T - 1; t1 >= 0; t1 -= GB_PF) {  // GB_PF steps of q and coef loaded ahead
      float qb[GB_PF];
      float4 cb[GB_PF];
#pragma unroll
      for (int k = 0; k < GB_PF; ++k) {
        const int t = t1 - k;
        qb[k] = t >= 0 ? q[t] : 0.f;
        cb[k] = t >= 0 ? cf[t] : make_float4(0.f, 0.f, 0.f, 0.f);
      }
#pragma unroll
      for (int k = 0; k < GB_PF; ++k) {
        const int t = t1 - k;
        if (t >= 0) {
          const float4 c4 = cb[k];  // (c, m, 1/D, 1/sqrt(D))
          const float x = fmaf(-mn, xn, qb[k] * c4.w);
          const float ut = fmaf(-cn, xn, x);
          u[t] = ut;
          o.U[((size_t)pd * K + j) * LT + t] = ut;
          umax_local = fmaxf(umax_local, fabsf(ut));
          xn = x;
          mn = c4.y;
          cn = c4.x;
        }
      }
    }
    for (int t = T; t < LT; ++t) o.U[((size_t)pd * K + j) * LT + t] = 0.f;
  }
  __syncthreads();
  if (o.U_hi) {
    // fp16 hi/lo split of U * 2^e, e placing max|U| in [128, 256)
    double um = umax_local;
    for (int off = 16; off > 0; off >>= 1) um = fmax(um, __shfl_xor_sync(0xffffffffu, um, off));
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = um;
    __syncthreads();
    if (threadIdx.x == 0) {
      double mx = 0.0;
      for (int w = 0; w < (int)(blockDim.x >> 5); ++w) mx = fmax(mx, red[w]);
      red[0] = mx;
    }
    __syncthreads();
    const int e = scale_exp((float)red[0]);
    if (threadIdx.x == 0) o.uexp[pd] = e;
    for (int idx = threadIdx.x; idx < K * d.ld_u; idx += blockDim.x) {
      const int j = idx / d.ld_u, t = idx % d.ld_u;
      uint16_t hi = 0, lo = 0;
      if (t < T) split_fp16(ldexpf(uf[(size_t)j * T + t], e), hi, lo);
      const size_t at = ((size_t)pd * K + j) * d.ld_u + t;
      o.U_hi[at] = hi;
      o.U_lo[at] = lo;
    }
  }
  __syncthreads();

  // ---- 7. Lx^-1 and diag(A), A = Lx^-T Lx^-1 = (X_w'X_w)^-1 (only the
  // entries the statistics read are formed: the diagonal here, the task
  // block and c A c' in phase 9)
  block_tri_inverse(s.Lx, s.Li, K, K, chol ? s.A : nullptr);
  for (int j = threadIdx.x; j < K; j += blockDim.x) {
    double acc = 0.0;
    for (int k = j; k < K; ++k) acc += s.Li[k * K + j] * s.Li[k * K + j];
    o.Adiag[(size_t)pd * K + j] = (float)acc;
  }
  if (o.Afull) {  // all of A, for the per-voxel blocks of the -dsort fit
    for (int e = threadIdx.x; e < K * K; e += blockDim.x) {
      const int i = e / K, j = e % K;
      double acc = 0.0;
      for (int k = max(i, j); k < K; ++k) acc += s.Li[k * K + i] * s.Li[k * K + j];
      o.Afull[(size_t)pd * K * K + e] = (float)acc;
    }
  }
  __syncthreads();

  if (args.const_flag && p == args.p0) const_of_design(args, pd / d.P, Xd, s.Li, K, chol, s.A, red);

  // ---- 8. G = U Lx^-1 in fp32 (row t of G solves g Lx = u_t); Gsum = G' 1
  // accumulated in FP64
  float* const li_f = lx_f + (size_t)K * K;
  for (int idx = threadIdx.x; idx < K * K; idx += blockDim.x) li_f[idx] = (float)s.Li[idx];
  __syncthreads();
  for (int t = threadIdx.x; t < LT; t += blockDim.x) {
    for (int j = 0; j < K; ++j) {
      float acc = 0.f;
      if (t < T)
        for (int i = j; i < K; ++i) acc = fmaf(uf[(size_t)i * T + t], li_f[i * K + j], acc);
      o.G[((size_t)pd * K + j) * LT + t] = acc;
    }
  }
  item_tail(d, o, s, pd, red, flag_s);
}

// Items are (design, pair) = (item / P, item % P); a CTA takes items
// blockIdx.x, blockIdx.x + gridDim.x, ... with scratch slot blockIdx.x.
// Design-dependent outputs sit at pd = design * P + pair. With SHARED_LDL
// (more than one design) phase 1 comes from pair_ldl_kernel (pair_cm,
// pair_bad), which also wrote coef and logdet_R; without it every item
// factors its pair's R itself. This kernel takes the items that
// grid_item_kernel and grid_wide_kernel do not (long designs, the banded R). Capped at
// 64 registers (4 CTAs per SM): left free, the compiler takes 80 to 126 of them.
template <bool SHARED_LDL, bool BAND>
__global__ void __launch_bounds__(GB_THREADS, BAND ? 2 : 4) grid_build_kernel(BuildArgs args, int n_designs,
                                                                                  const double* pair_cm,
                                                                                  const int* pair_bad, int tmp_smem) {
  const ffs_grid_desc& d = args.d;
  const ffs_grid_out& o = args.o;
  const int T = d.T, K = d.K;
  PairScratch s = scratch_of(o.work, blockIdx.x, T, K);
  __shared__ double red[32];
  __shared__ int flag, bad_r;
  // c, m, 1/sqrt(D) of the current pair [3][T], then [4][T] with tmp_smem; or the band's scratch
  extern __shared__ double cms[];
  for (int item = blockIdx.x; item < d.P * n_designs; item += gridDim.x) {
    const int p = item % d.P;
    const double* cc = cms;
    if constexpr (SHARED_LDL) {
      // the pre-pass factored R for every pair once: copy this pair's rows
      const double* src = pair_cm + (size_t)p * 4 * T;
      if constexpr (BAND)
        cc = src;
      else
        for (int i = threadIdx.x; i < 3 * T; i += blockDim.x) cms[i] = src[i];
      if (threadIdx.x == 0) bad_r = pair_bad[p];
      __syncthreads();
    } else if constexpr (BAND) {
      band_chol_of_pair(d, o, p, s.cm, cms, red, &bad_r);
      cc = s.cm;
    } else {
      ldl_of_pair(d, o, p, cms, cms + T, cms + 2 * T, tmp_smem ? cms + 3 * T : s.cm, red, &bad_r);
    }
    item_global<BAND>(args, s, p, item, d.X + (size_t)(item / d.P) * T * K, cc, cms + T, cms + 2 * T, cms, bad_r, red, &flag);
  }
}

// --------------------------------------------------------- Gram entries in integers
// This GPU's FP64 pipe takes one warp instruction per 19 cycles and SM, its
// integer multiply-add with a 64-bit sum one per cycle or better. A Gram entry
// sum_t x_i[t] x_j[t] of FP64 series is therefore formed from fixed-point values
// x = q 2^-s, s per column, q = hi 2^27 + lo with |lo| <= 2^26, and the sums of hi hi',
// hi lo' + lo hi' and lo lo' in 64-bit integers: exact for up to 1024 samples,
// whatever the order. What remains is the rounding of x to the fixed point, where a
// chain of FP64 FMAs rounds every partial sum. s comes from the column's largest
// magnitude (|q| < 2^53, |hi| <= 2^26: the design basis, which forms all three sums) or
// from its norm (|hi| up to 2^31: the grid build, which leaves lo lo' out).
constexpr int FX_TMAX = 1024;

// s for a column of largest magnitude mx: mx (1 + 1/32) < 2^(53 - s), the margin
// for an mx found in fp32
__device__ __forceinline__ int fixed_scale(float mx) {
  int e = 0;
  frexpf(mx * 1.03125f, &e);
  return mx > 0.f ? 53 - e : 0;
}

// (hi, lo) of w 2^s rounded to an integer; over = true when that is 2^(53 + SHIFT)
// or more in magnitude (with SHIFT = 5, |hi| may be 2^31, for the caller to refuse)
template <int SHIFT>
__device__ __forceinline__ int2 fixed_of(double w, int s, bool& over) {
  const unsigned long long b = (unsigned long long)__double_as_longlong(w);
  const int ex = (int)(b >> 52) & 0x7ff;
  const int r = 1075 + SHIFT - ex - s;  // |w| 2^s = mantissa 2^(SHIFT - r)
  over = over || (r < 0 && ex != 0);
  unsigned long long m = ((b << 1) & 0x1ffffffffffffeull) | 0x20000000000000ull;
  m = (ex == 0 || r > 54 + SHIFT) ? 0ull : (((m << SHIFT) >> max(r, 0)) + 1) >> 1;
  const long long q = (long long)b < 0 ? -(long long)m : (long long)m;
  const int hi = (int)((q + (1 << 26)) >> 27);
  return make_int2(hi, (int)(q - ((long long)hi << 27)));
}

// The sums of a Gram entry, for columns scaled by fixed_scale.
struct FixedDot {
  long long hh = 0, x = 0, ll = 0;
  __device__ __forceinline__ void add(int2 a, int2 b) {
    hh += (long long)a.x * b.x;
    x += (long long)a.x * b.y;
    x += (long long)a.y * b.x;
    ll += (long long)a.y * b.y;
  }
  // the entry, for columns scaled by 2^si and 2^sj
  __device__ __forceinline__ double value(int si, int sj) const {
    const double v = fma((double)hh, 0x1p54, fma((double)x, 0x1p27, (double)ll));
    return v * __hiloint2double((1023 - si - sj) << 20, 0);
  }
};

// The columns' scales of FixedDot2, from their norms: s with B 4^(s - 27) < 2^61, B
// (at least the column's sum of squares, found in fp32: + 1/16) in 1e-30 .. 1e30;
// false otherwise. A dense column then has |hi| of about 2^26, a sample that stands
// out up to 2^31, and every column's hi a norm below 2^30.8 (norm_fits holds the
// samples as they come out to it), so that whatever the columns
//   |hh| <= 2^61.6, |x| <= 2 * 2^30.8 * 2^26 sqrt(1024) = 2^62.8 in 64 bits, and
//   |ll| <= 2^52 T, 2^-51 of the product of the norms at worst and 2^-60 at random,
// which FixedDot2 leaves out. Measured against 64 bits (largest error of an entry
// over |x_i| |x_j|, whitened designs of the ranges in use, peaked and graded columns):
// FP64 FMA chains 1.2e-16 to 7e-15, this 7e-18 to 3.1e-16.
__device__ __forceinline__ bool norm_scale(float b, int& s) {
  int e = 0;
  frexpf(b * 1.0625f, &e);
  const bool ok = b > 1e-30f && b < 1e30f;
  s = ok ? 27 + ((61 - e) >> 1) : 0;
  return ok;
}
__device__ __forceinline__ bool norm_fits(float b, int s) { return ldexpf(b, 2 * (s - 27)) <= 0x1.8p61f; }

// hh and x of FixedDot
struct FixedDot2 {
  long long hh = 0, x = 0;
  __device__ __forceinline__ void add(int ax, int ay, int bx, int by) {
    hh += (long long)ax * bx;
    x += (long long)ax * by;
    x += (long long)ay * bx;
  }
  __device__ __forceinline__ double value(int si, int sj) const {
    return fma((double)hh, 0x1p54, (double)x * 0x1p27) * __hiloint2double((1023 - si - sj) << 20, 0);
  }
};

// float of a double, rounded to nearest even, by its bit fields (integer pipe);
// anything but zeros and normal results takes the hardware conversion.
__device__ __forceinline__ float d2f_exact(double w) {
  const unsigned long long b = (unsigned long long)__double_as_longlong(w);
  const unsigned long long m = b & 0x7fffffffffffffffull;
  const uint32_t sg = (uint32_t)(b >> 32) & 0x80000000u;
  if (m == 0) return __uint_as_float(sg);
  const unsigned ex = (unsigned)(m >> 52);
  if (ex - 897u >= 253u) return (float)w;
  const unsigned long long r = m + 0x0fffffffull + ((m >> 29) & 1);
  return __uint_as_float(sg | ((uint32_t)(r >> 29) - (896u << 23)));
}

// The factor of X_w'X_w = Lu D Lu' and Lu^-1 in one pass over its packed lower
// triangle A, for the kernels below: step k takes w_r f_c off every entry (r, c) of
// the rows below k + 1, w_r = A_rk / D_k, f = (row k of Lu^-1, 1, column k of A): left
// of column k the inverse grows where the factor's columns are no longer read.
// Some warps form the next step's f and w ahead of the others (fold_ahead, lane
// by lane i < K); one barrier a step, for k = -1 .. K - 2. fw: f and w, double-
// buffered [2][2][K]; column k of A, before its division by sqrt(D_k), goes to row k of
// Lx [K][K], right of its diagonal; dk [K] receives D.
struct Fold {
  double *A, *fw, *dk, *Lx;
  int K;
};

// Returns true when pivot k + 1 is not positive.
__device__ __forceinline__ bool fold_ahead(const Fold& m, int k, int i) {
  const double *f = m.fw + (k & 1) * 2 * m.K, *w = f + m.K;
  double *fn = m.fw + ((k + 1) & 1) * 2 * m.K, *wn = fn + m.K;
  const int k1 = k + 1, row1 = k1 * (k1 + 1) / 2;
  const double w1 = k >= 0 ? w[k1] : 0.0, f1 = k >= 0 ? f[k1] : 0.0;
  double dn = m.A[row1 + k1];
  if (k >= 0) dn = fma(-w1, f1, dn);
  const bool bad = !positive(dn);
  if (bad) dn = 1.0;
  double v = 1.0, r, pc;
  if (i < k1) {  // row k + 1 of the inverse
    v = fma(-w1, f[i], i == k ? 0.0 : m.A[row1 + i]);
    m.A[row1 + i] = v;
  } else if (i > k1 && i < m.K) {
    v = m.A[i * (i + 1) / 2 + k1];
    if (k >= 0) v = fma(-w[i], f1, v);
    m.Lx[k1 * m.K + i] = v;
  }
  rcp_factors(dn, r, pc);
  if (i < m.K) {
    const double u = v * r;
    fn[i] = v;
    wn[i] = fma(u, pc, u);
  }
  if (i == k1) m.dk[k1] = dn;
  return bad;
}

// Step k >= 0 at entry e = (r, c), r > k + 1.
__device__ __forceinline__ void fold_entry(const Fold& m, int k, int e, int r, int c) {
  const double *f = m.fw + (k & 1) * 2 * m.K, *w = f + m.K;
  if (c != k + 1) m.A[e] = fma(-w[r], f[c], c == k ? 0.0 : m.A[e]);
}

// ------------------------------------------------------------- items in shared memory
// Items of up to GI_KMAX columns and FX_TMAX samples whose matrices fit in
// shared memory: the phases of item_global, arranged around the FP64 pipe,
// which a warp fills with one instruction per 64 cycles whatever its lanes do.
//   - X_w = L^-1 X in a pipeline over chunks of 8 to 32 samples of each time segment
//     (segments start at run starts, where the recursion does), a chunk in each
//     stage: z = x - c x' by all entry warps (full warps); v = z - m v' by the
//     producer warps, a lane per column and segment, one FP64 instruction a
//     step; w = v / sqrt(D) by the entry warps, in fixed point for the Gram
//     matrix and as the fp32 copy that the later phases read; the Gram matrix in
//     integers (above), blocks of 2 x 2 entries per thread, the samples split over
//     SL threads of a block.
//   - The factor and its inverse (Fold), an entry per thread; then Q, U and the fp16
//     splits in place in shared memory.
// The sums, the factor and the fp32 phases are grid_wide_kernel's to the bit, so a
// design's factors do not depend on how many others are built beside it.
// A rank-deficient item (a pivot that is not positive) or one whose series
// leave the fixed point goes through item_global.
// P = 117, T = 200, K = 8: 238 -> 107 us against item_global's phases with FP64 Gram
// chains; P = 561, T = 400, K = 20: 584 -> 307. Bound by latency: two or three CTAs
// an SM (their series fill the shared memory), a barrier per chunk.
constexpr int GI_KMAX = 22;       // 253 entries, one per entry thread
constexpr int GI_BUF = 4;         // chunks in the pipeline
constexpr int GI_PROD = 96;       // most producer lanes (3 warps)
constexpr int GI_VAL = 3;         // most values of a chunk per thread
constexpr int GI_ENTRY = 256;     // entry threads
constexpr int GI_CTAS = 3;        // CTAs an SM, by registers

struct ItemPlan {
  // entries, rows (even), 2 x 2 blocks, slices, row stride, time
  // segments, producer warps, log2 of a segment's samples per chunk
  int E, KR, NB, SL, rs, RP, PW, cs2;
  int cm, xf, ring, L, Li, rd, lxf, lif, total;  // byte offsets
};

__host__ __device__ inline ItemPlan item_plan(int T, int K, int n_runs) {
  ItemPlan m;
  m.E = K * (K + 1) / 2;
  constexpr int GT = GI_ENTRY;
  const int kb = (K + 1) / 2;
  m.KR = 2 * kb;
  m.NB = kb * (kb + 1) / 2;
  m.SL = 1;
  m.RP = 1;  // time segments: the fewest whose longest has the fewest runs
  for (int rp = 2; rp <= n_runs && rp * K <= GI_PROD; ++rp)
    if ((n_runs + rp - 1) / rp < (n_runs + m.RP - 1) / m.RP) m.RP = rp;
  m.cs2 = 3;  // 8 samples, or 16 or 32 while a chunk is at most two values per thread
  while (m.cs2 < 5 && (K * m.RP << (m.cs2 + 1)) <= 2 * GT) ++m.cs2;
  const int cs = 1 << m.cs2;
  while (2 * m.SL * m.NB <= GT && m.SL < 16 && m.SL < cs) m.SL *= 2;
  m.rs = cs + (m.SL == 4 ? 2 : m.SL == 8 ? 4 : 1);  // a half-warp's blocks and slices in distinct banks
  m.PW = (K * m.RP + 31) / 32;
  const int K4 = (K + 3) & ~3;
  int at = 0;
  auto take = [&](size_t n) {
    const int o = at;
    at += (int)((n + 15) & ~(size_t)15);
    return o;
  };
  m.cm = take(sizeof(double) * 3 * T);  // c, m, 1/sqrt(D); later the fp32 coefficients
  // the fp32 series, whose region also holds phase 1's 4 T doubles
  const size_t xf = sizeof(float) * (size_t)K * (T | 1), tmp = sizeof(double) * 4 * T;
  m.xf = take(xf > tmp ? xf : tmp);
  // [GI_BUF][RP][KR][rs] samples (FP64, then fixed point); afterwards 2 K^2 doubles of scratch
  size_t ring = sizeof(int2) * GI_BUF * m.RP * m.KR * m.rs;
  // before it, the fp32 coefficients; first the packed triangle, f and w
  const size_t fold = (size_t)m.E + 4 * K, kk = (size_t)2 * K * K;
  const size_t scr = sizeof(double) * (fold > kk ? fold : kk), cf = sizeof(float4) * T;
  ring = ring > scr ? ring : scr;
  m.ring = take(ring > cf ? ring : cf);
  m.L = take(sizeof(double) * K * K);     // [k][i]: column k of the factor, times sqrt(D_k)
  m.Li = take(sizeof(double) * K * K);
  m.rd = take(sizeof(double) * 2 * K);    // D, 1 / sqrt(D)
  m.lxf = take(sizeof(float) * K * K4);   // Lx transposed: [i][j], j contiguous
  m.lif = take(sizeof(float) * K * K4);
  m.total = at;
  return m;
}

template <bool SHARED_LDL>
__global__ void __launch_bounds__(GI_ENTRY + GI_PROD, GI_CTAS) grid_item_kernel(BuildArgs args, int n_designs,
                                                                                const double* pair_cm,
                                                                                const int* pair_bad) {
  const ffs_grid_desc& d = args.d;
  const ffs_grid_out& o = args.o;
  const int T = d.T, K = d.K, LT = ld_t(T), K4 = (K + 3) & ~3, ldx = T | 1;
  const int tid = threadIdx.x, nth = blockDim.x, lane = tid & 31, wid = tid >> 5;
  extern __shared__ double2 gi_smem[];
  char* sm = reinterpret_cast<char*>(gi_smem);
  const ItemPlan pl = item_plan(T, K, d.n_runs);
  constexpr int GT = GI_ENTRY;
  const int RP = pl.RP, rs = pl.rs;
  double* cc = reinterpret_cast<double*>(sm + pl.cm);
  double *cm = cc + T, *cr = cc + 2 * T;
  float4* cfs = reinterpret_cast<float4*>(sm + pl.cm);     // after phase 4: (c, m, 1/D, 1/sqrt(D)) in fp32
  float* xf = reinterpret_cast<float*>(sm + pl.xf);        // [K][ldx] X_w, then Q, then U
  int2* ring = reinterpret_cast<int2*>(sm + pl.ring);      // [GI_BUF][RP][KR][rs]
  const int bufw = RP * pl.KR * rs, cs2 = pl.cs2, CS = 1 << cs2;
  double* scr = reinterpret_cast<double*>(sm + pl.ring);
  double* L = reinterpret_cast<double*>(sm + pl.L);
  double* Li = reinterpret_cast<double*>(sm + pl.Li);
  double *dk = reinterpret_cast<double*>(sm + pl.rd), *rsd = dk + K;
  const Fold fold{scr, scr + pl.E, dk, L, K};              // X_w'X_w, then the inverse, packed
  float* lxf = reinterpret_cast<float*>(sm + pl.lxf);
  float* lif = reinterpret_cast<float*>(sm + pl.lif);
  __shared__ double red[32];
  __shared__ float fred[32];
  __shared__ int colss[GI_KMAX], scale[GI_KMAX + 1];
  __shared__ float colsum[GI_KMAX];
  __shared__ int seg[GI_PROD + 1];  // first sample of each time segment
  __shared__ int flag, bad_r;
  for (int q = tid; q <= RP; q += nth) seg[q] = d.run_start[q * d.n_runs / RP];
  const bool entry = tid < pl.E;
  int ei = 0, ej = 0;
  if (entry) tri_index(tid, ei, ej);
  int bi = 0, bj = 0;  // this thread's 2 x 2 block of the Gram matrix, and its slice of the samples
  const bool gram = tid < pl.NB * pl.SL;
  const int sl = tid % pl.SL;
  if (gram) tri_index(tid / pl.SL, bi, bj);
  const bool producer = tid >= GT && tid - GT < K * RP;
  const int pj = producer ? (tid - GT) % K : 0, pq = producer ? (tid - GT) / K : 0;
  __syncthreads();

  for (int item = blockIdx.x; item < d.P * n_designs; item += gridDim.x) {
    const int p = item % d.P, pd = item;
    const float* Xd = d.X + (size_t)(item / d.P) * T * K;
    if constexpr (SHARED_LDL) {
      const double* src = pair_cm + (size_t)p * 4 * T;
      for (int i = tid; i < 3 * T; i += nth) cc[i] = src[i];
      if (tid == 0) bad_r = pair_bad[p];
    } else {
      ldl_of_pair(d, o, p, cc, cm, cr, reinterpret_cast<double*>(xf), red, &bad_r);
    }
    if (tid == 0) flag = 0;
    for (int j = tid; j < K; j += nth) {
      colss[j] = 0;
      colsum[j] = 0.f;
    }
    // the design into xf, where X_w replaces it, and the fp32 coefficients into
    // the ring's region
    const float4* cf = reinterpret_cast<const float4*>(o.coef) + (size_t)p * T;
    float4* cfr = reinterpret_cast<float4*>(ring);
    if (!SHARED_LDL) __syncthreads();  // phase 1's scratch is read no more
    for (int t = tid; t < T; t += nth) cfr[t] = cf[t];
#pragma unroll 4
    for (int e = tid; e < K * T; e += nth) xf[(size_t)(e % K) * ldx + e / K] = __ldg(Xd + e);
    __syncthreads();

    // ---- 2, 3. X_w and X_w'X_w
    const int ps = producer ? seg[pq] : 0;
    if (producer) {
      // the columns' scales, from the recursion in fp32 (the largest sum of squares
      // of a run times their number)
      const float* xs = xf + (size_t)pj * ldx;
      for (int r = pq * d.n_runs / RP; r < (pq + 1) * d.n_runs / RP; ++r) {
        const int t1 = d.run_start[r + 1];
        float xp = 0.f, vp = 0.f, ss = 0.f;
#pragma unroll 8
        for (int t = d.run_start[r]; t < t1; ++t) {
          const float x = xs[t];
          const float4 q = cfr[t];
          vp = fmaf(-q.y, vp, fmaf(-q.x, xp, x));
          xp = x;
          const float w = vp * q.w;
          ss = fmaf(w, w, ss);
        }
        atomicMax(colss + pj, __float_as_int(ss));
      }
    }
    __syncthreads();
    if (pl.KR > K)  // the row past an odd K is zero
      for (int e = tid; e < GI_BUF * RP * rs; e += nth) ring[(e / rs * pl.KR + K) * rs + e % rs] = make_int2(0, 0);
    bool over = tid < K && !norm_scale(__int_as_float(colss[tid]) * (float)d.n_runs, scale[tid]);
    __syncthreads();
    int longest = 0;
    for (int q = 0; q < RP; ++q) longest = max(longest, seg[q + 1] - seg[q]);
    const int nch = (longest + CS - 1) >> cs2;
    FixedDot2 acc[2][2];
    {
      // the values of a chunk this thread forms (z) and converts (w): slot in a
      // ring buffer, sample of chunk 0 and its segment's end
      int vs[GI_VAL], vt[GI_VAL], ve[GI_VAL], vj[GI_VAL];
      float ss[GI_VAL];
#pragma unroll
      for (int i = 0; i < GI_VAL; ++i) {
        const int e = tid + i * GT;  // sample fastest: consecutive lanes, consecutive words
        const bool on = tid < GT && e < K * RP << cs2;
        const int k = e & (CS - 1), j = (e >> cs2) % K, q = on ? (e >> cs2) / K : 0;
        vj[i] = j;
        vs[i] = on ? (q * pl.KR + j) * rs + k : -1;
        vt[i] = seg[q] + k;
        ve[i] = seg[q + 1];
        ss[i] = 0.f;
      }
      double vp = 0.0;
      for (int c = 0; c < nch + GI_BUF - 1; ++c) {
        if (tid < GT) {
          double* za = reinterpret_cast<double*>(ring) + (c % GI_BUF) * bufw;
          if (c < nch) {
#pragma unroll
            for (int i = 0; i < GI_VAL; ++i) {
              const int t = vt[i] + (c << cs2);
              if (vs[i] >= 0 && t < ve[i]) {
                const float* x = xf + (size_t)vj[i] * ldx + t;
                za[vs[i]] = f2d_exact(x[0]) - cc[t] * f2d_exact(t > 0 ? x[-1] : 0.f);
              }
            }
          }
          if (c >= 2 && c < nch + 2) {
            int2* wb = ring + ((c - 2) % GI_BUF) * bufw;
#pragma unroll
            for (int i = 0; i < GI_VAL; ++i) {
              const int t = vt[i] + ((c - 2) << cs2);
              if (vs[i] >= 0) {
                int2 f = make_int2(0, 0);
                if (t < ve[i]) {
                  const double w = reinterpret_cast<double*>(wb)[vs[i]] * cr[t];
                  f = fixed_of<5>(w, scale[vj[i]], over);
                  const float wf = d2f_exact(w);
                  ss[i] = fmaf(wf, wf, ss[i]);
                  xf[(size_t)vj[i] * ldx + t] = wf;
                }
                wb[vs[i]] = f;
              }
            }
          }
          if (gram && c >= 3) {
            const int2* rg = ring + ((c - 3) % GI_BUF) * bufw;
            for (int u = sl; u < RP << cs2; u += pl.SL) {
              const int2* r0 = rg + (u >> cs2) * pl.KR * rs + (u & (CS - 1));
              const int2 *ai = r0 + 2 * bi * rs, *aj = r0 + 2 * bj * rs;
              const int2 i0 = ai[0], i1 = ai[rs], j0 = aj[0], j1 = aj[rs];
              acc[0][0].add(i0.x, i0.y, j0.x, j0.y);
              acc[0][1].add(i0.x, i0.y, j1.x, j1.y);
              acc[1][0].add(i1.x, i1.y, j0.x, j0.y);
              acc[1][1].add(i1.x, i1.y, j1.x, j1.y);
            }
          }
        } else if (producer && c >= 1 && c <= nch) {
          double* v = reinterpret_cast<double*>(ring) + ((c - 1) % GI_BUF) * bufw + (pq * pl.KR + pj) * rs;
          for (int k0 = 0; k0 < CS; k0 += 8, v += 8) {
            const int t0 = ps + ((c - 1) << cs2) + k0;
            double z[8], m[8];
#pragma unroll
            for (int k = 0; k < 8; ++k) {
              z[k] = v[k];
              m[k] = cm[min(t0 + k, T - 1)];
            }
#pragma unroll
            for (int k = 0; k < 8; ++k) z[k] = vp = z[k] - m[k] * vp;  // past the segment: not read
#pragma unroll
            for (int k = 0; k < 8; ++k) v[k] = z[k];
          }
        }
        __syncthreads();
      }
      if (tid < GT) {
#pragma unroll
        for (int i = 0; i < GI_VAL; ++i) {  // CS lanes a column
          for (int m = 1; m < CS; m <<= 1) ss[i] += __shfl_xor_sync(0xffffffffu, ss[i], m);
          if (vs[i] >= 0 && (lane & (CS - 1)) == 0) atomicAdd(colsum + vj[i], ss[i]);
        }
      }
    }
    if (wid * 32 < pl.NB * pl.SL) {  // whole warps: the slices of a block lie in one
#pragma unroll
      for (int u = 0; u < 2; ++u)
#pragma unroll
        for (int v = 0; v < 2; ++v) {
          FixedDot2& f = acc[u][v];
          for (int m = 1; m < pl.SL; m <<= 1) {
            f.hh += __shfl_xor_sync(0xffffffffu, f.hh, m);
            f.x += __shfl_xor_sync(0xffffffffu, f.x, m);
          }
          const int i = 2 * bi + u, j = 2 * bj + v;
          if (gram && sl == 0 && i < K && j <= i) {
            const double x = f.value(scale[i], scale[j]);
            fold.A[i * (i + 1) / 2 + j] = x;
            o.XtX[(size_t)pd * K * K + i * K + j] = (float)x;
            o.XtX[(size_t)pd * K * K + j * K + i] = (float)x;
          }
        }
    }
    __syncthreads();
    over = over || (tid < K && !norm_fits(colsum[tid], scale[tid]));
    bool left = __syncthreads_or(over);  // a series left the fixed point

    // ---- 4. the factor and its inverse, an entry per thread
    for (int k = -1; k < K - 1 && !left; ++k) {
      const bool bad = wid == 0 && fold_ahead(fold, k, lane);
      if (k >= 0 && entry && ei > k + 1) fold_entry(fold, k, tid, ei, ej);
      left = __syncthreads_or(bad);
    }
    if (left) {
      const PairScratch s = scratch_of(o.work, blockIdx.x, T, K);
      item_global<false>(args, s, p, pd, Xd, cc, cm, cr, nullptr, bad_r, red, &flag);
      continue;
    }
    for (int k = tid; k < K; k += nth) {
      const double r = rsqrt_newton(dk[k]);
      rsd[k] = r;
      fold.fw[k] = 2.0 * log(fabs(dk[k] * r) + 1e-10);
    }
    __syncthreads();
    if (entry) Li[ei * K + ej] = ei == ej ? rsd[ei] : fold.A[tid] * rsd[ei];  // Li = D^-1/2 Lu^-1
    for (int e = tid; e < K * K4; e += nth) {
      const int i = e / K4, j = e % K4;
      lxf[e] = j < K && j >= i ? (float)(j == i ? dk[i] * rsd[i] : L[i * K + j] * rsd[i]) : 0.f;
    }
    for (int t = tid; t < T; t += nth) cfs[t] = cf[t];  // c, m and 1/sqrt(D) in FP64 are done with
    __syncthreads();

    if (tid < GT) {
      // ---- 5. Q = X_w Lx^-T in fp32, two samples per thread, four columns at a
      // time: each earlier column is read once for them
      for (int t = tid; t < T; t += 2 * GT) {
        float* q = xf + t;
        const int u1 = t + GT < T ? GT : 0;  // the second sample, or the first again
        for (int j0 = 0; j0 < K; j0 += 4) {
          float a4[4], b4[4];
#pragma unroll
          for (int c = 0; c < 4; ++c) {
            a4[c] = j0 + c < K ? q[(size_t)(j0 + c) * ldx] : 0.f;
            b4[c] = j0 + c < K ? q[(size_t)(j0 + c) * ldx + u1] : 0.f;
          }
#pragma unroll 4
          for (int i = 0; i < j0; ++i) {
            const float qa = q[(size_t)i * ldx], qb = q[(size_t)i * ldx + u1];
            const float4 l = *reinterpret_cast<const float4*>(lxf + i * K4 + j0);
            a4[0] = fmaf(-l.x, qa, a4[0]);
            b4[0] = fmaf(-l.x, qb, b4[0]);
            a4[1] = fmaf(-l.y, qa, a4[1]);
            b4[1] = fmaf(-l.y, qb, b4[1]);
            a4[2] = fmaf(-l.z, qa, a4[2]);
            b4[2] = fmaf(-l.z, qb, b4[2]);
            a4[3] = fmaf(-l.w, qa, a4[3]);
            b4[3] = fmaf(-l.w, qb, b4[3]);
          }
#pragma unroll
          for (int c = 0; c < 4; ++c) {
            if (j0 + c < K) {
              const float* l = lxf + (j0 + c) * K4 + j0;
              a4[c] = a4[c] / l[c];
              b4[c] = b4[c] / l[c];
#pragma unroll
              for (int e = c + 1; e < 4; ++e) {
                a4[e] = fmaf(-l[e], a4[c], a4[e]);
                b4[e] = fmaf(-l[e], b4[c], b4[e]);
              }
            }
          }
#pragma unroll
          for (int c = 0; c < 4; ++c) {
            if (j0 + c < K) {
              q[(size_t)(j0 + c) * ldx] = a4[c];
              q[(size_t)(j0 + c) * ldx + u1] = b4[c];
            }
          }
        }
      }
      bar_sync(1, GT);
      // ---- 6. U = L^-T Q, the backward recursions of each column and run
      float umax = 0.f;
      for (int e = tid; e < K * d.n_runs; e += GT) {
        const int j = e % K, r = e / K;
        float* u = xf + (size_t)j * ldx;
        const int t0 = d.run_start[r];
        float xn = 0.f, mn = 0.f, cn = 0.f;  // x_{t+1}, m_{t+1}, c_{t+1} (0 past a run's end)
        constexpr int UB = 8;
        float qn[UB];
        float4 cb[UB];
        auto load_c = [&](int t1) {
#pragma unroll
          for (int k = 0; k < UB; ++k) {
            const int t = max(t1 - k, t0);
            cb[k] = cfs[t];
            qn[k] = u[t];
          }
        };
        const int te = d.run_start[r + 1] - 1;
        load_c(te);
        for (int t1 = te; t1 >= t0; t1 -= UB) {
          float qw[UB], mm[UB], ccv[UB];
#pragma unroll
          for (int k = 0; k < UB; ++k) {
            qw[k] = qn[k] * cb[k].w;
            mm[k] = cb[k].y;
            ccv[k] = cb[k].x;
          }
          load_c(t1 - UB);  // the next batch's, before this one's stores
#pragma unroll
          for (int k = 0; k < UB; ++k) {
            const float x = fmaf(-mn, xn, qw[k]);
            qw[k] = fmaf(-cn, xn, x);
            xn = x;
            mn = mm[k];
            cn = ccv[k];
          }
#pragma unroll
          for (int k = 0; k < UB; ++k) {
            if (t1 - k >= t0) {
              u[t1 - k] = qw[k];
              umax = fmaxf(umax, fabsf(qw[k]));
            }
          }
        }
      }
      for (int off = 16; off > 0; off >>= 1) umax = fmaxf(umax, __shfl_xor_sync(0xffffffffu, umax, off));
      if (lane == 0) fred[wid] = umax;
      bar_sync(1, GT);
      float mx = 0.f;
      for (int w = 0; w < GT / 32; ++w) mx = fmaxf(mx, fred[w]);
      // fp16 hi/lo split of U * 2^e, e placing max|U| in [128, 256); x * 2^e as
      // one product when 2^e is a normal float (ldexpf's value)
      const int ex = scale_exp(mx);
      if (o.U_hi && tid == 0) o.uexp[pd] = ex;
      const bool pw = ex >= -126 && ex <= 127;
      const float p2 = pw ? __int_as_float((ex + 127) << 23) : 0.f;
      for (int j = wid; j < K; j += GT / 32) {  // a warp per column
        const float* u = xf + (size_t)j * ldx;
        float* uo = o.U + ((size_t)pd * K + j) * LT;
#pragma unroll 4
        for (int t = lane; t < LT; t += 32) uo[t] = t < T ? u[t] : 0.f;
        if (o.U_hi) {
          uint32_t* ho = reinterpret_cast<uint32_t*>(o.U_hi + ((size_t)pd * K + j) * d.ld_u);
          uint32_t* lo = reinterpret_cast<uint32_t*>(o.U_lo + ((size_t)pd * K + j) * d.ld_u);
#pragma unroll 4
          for (int h = lane; h < (d.ld_u >> 1); h += 32) {
            const int t = 2 * h;
            uint16_t h0 = 0, l0 = 0, h1 = 0, l1 = 0;
            if (t < T) split_fp16(pw ? __fmul_rn(u[t], p2) : ldexpf(u[t], ex), h0, l0);
            if (t + 1 < T) split_fp16(pw ? __fmul_rn(u[t + 1], p2) : ldexpf(u[t + 1], ex), h1, l1);
            ho[h] = (uint32_t)h0 | ((uint32_t)h1 << 16);
            lo[h] = (uint32_t)l0 | ((uint32_t)l1 << 16);
          }
        }
      }
    } else {
      // ---- 7. logdet, diag(A) and the fp32 copy of Li beside them
      if (tid == GT) {
        double ld = 0.0;
        for (int j = 0; j < K; ++j) ld += fold.fw[j];
        o.logdet_XtX[pd] = ld;
        o.info[pd] = bad_r ? 2 : 0;
      }
      for (int e = tid - GT; e < K * K4; e += nth - GT) {
        const int i = e / K4, j = e % K4;
        lif[e] = j <= i ? (float)Li[i * K + j] : 0.f;
      }
      for (int j = tid - GT; j < K; j += nth - GT) {
        double a = 0.0;
        for (int k = j; k < K; ++k) a = fma(Li[k * K + j], Li[k * K + j], a);
        o.Adiag[(size_t)pd * K + j] = (float)a;
      }
    }
    __syncthreads();

    if (o.Afull) {  // all of A, for the per-voxel blocks of the -dsort fit
      for (int e = tid; e < K * K; e += nth) {
        const int i = e / K, j = e % K;
        double a = 0.0;
        for (int k = max(i, j); k < K; ++k) a = fma(Li[k * K + i], Li[k * K + j], a);
        o.Afull[(size_t)pd * K * K + e] = (float)a;
      }
    }
    if (args.const_flag && p == args.p0) const_of_design(args, pd / d.P, Xd, Li, K, true, scr, red);
    __syncthreads();

    // ---- 8. G = U Lx^-1 in fp32, two samples per thread, four columns per pass over U
    for (int t = tid; t < LT; t += 2 * nth) {
      const float* u = xf + min(t, T - 1);
      const bool two = t + nth < LT;
      const int u1 = two ? min(t + nth, T - 1) - min(t, T - 1) : 0;
      for (int j0 = 0; j0 < K; j0 += 4) {
        float a4[4] = {0.f, 0.f, 0.f, 0.f}, b4[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll 4
        for (int i = j0; i < K; ++i) {  // Li is zero above its diagonal
          const float ua = u[(size_t)i * ldx], ub = u[(size_t)i * ldx + u1];
          const float4 l = *reinterpret_cast<const float4*>(lif + i * K4 + j0);
          a4[0] = fmaf(ua, l.x, a4[0]);
          b4[0] = fmaf(ub, l.x, b4[0]);
          a4[1] = fmaf(ua, l.y, a4[1]);
          b4[1] = fmaf(ub, l.y, b4[1]);
          a4[2] = fmaf(ua, l.z, a4[2]);
          b4[2] = fmaf(ub, l.z, b4[2]);
          a4[3] = fmaf(ua, l.w, a4[3]);
          b4[3] = fmaf(ub, l.w, b4[3]);
        }
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          if (j0 + c < K) {
            float* g = o.G + ((size_t)pd * K + j0 + c) * LT;
            g[t] = t < T ? a4[c] : 0.f;
            if (two) g[t + nth] = t + nth < T ? b4[c] : 0.f;
          }
        }
      }
    }
    PairScratch s{};
    s.Li = Li;
    s.S = scr;
    s.A = scr + (size_t)K * K;
    item_tail(d, o, s, pd, red, &flag);
  }
}

// ------------------------------------------------------------- many or wide items
// The series stay in the item's scratch slot (L2), and shared memory holds what
// the CTA works on: staged samples of the Gram matrix, then the packed K x K
// factor in FP64, then the fp32 factors that Q and G read. So several CTAs share
// an SM, and one's integer Gram matrix runs beside another's FP64 recursions.
//   - X_w = L^-1 X, a lane per column and run, to fixed point (scaled by the columns'
//     norms, without the lo lo' sums: norm_scale) and to fp32; the Gram matrix in
//     blocks of 4 x 4 or 2 x 2 entries per thread (rows b,
//     b + kb, ..., so that a warp's blocks read consecutive rows) from
//     double-buffered chunks of WI_CS samples.
//   - X_w'X_w = Lu D Lu' and Lu^-1 in one pass (Fold).
//   - Q = X_w Lx^-T and G = U Lx^-1 in fp32, 8 columns x 2 samples per thread.
// A rank-deficient item or one whose series leave the fixed point goes through
// item_global, whose general phases these replace: P = 561, T = 600, K = 130 in 3
// runs: 13.7 -> 3.87 ms; 20 designs of T = 855, K = 18: 13.6 -> 4.55 (in shared
// memory with three CTAs an SM: 8.0). What bounds an item at K = 130: 0.73 M cycles of
// integer multiply-adds (Gram) beside 0.57 M cycles of the FP64 pipe (X_w, factor
// and inverse); narrow ones the latency of their phases.
constexpr int WI_WIDE = 320;     // threads: 2 CTAs an SM, blocks of 4 x 4
constexpr int WI_NARROW = 128;   // 5 (many designs: 8), blocks of 2 x 2
constexpr int WI_NARROW_K = 56;
constexpr int WI_CS = 32;        // samples per chunk
constexpr int WI_RS = WI_CS + 2; // row stride of a chunk (16-byte words of consecutive rows in distinct banks)
constexpr int WI_KMAX = 255;     // 8-bit indices of the triangle's table

struct WidePlan {
  int KP, kb, NB, SL;           // K to a multiple of 8; blocks a side, blocks, slices of the samples
  int tri, fw, dk, scale, total;  // byte offsets (the work area is at 0)
};

__host__ __device__ inline WidePlan wide_plan(int T, int K, bool shared_ldl, int threads) {
  WidePlan m;
  m.KP = (K + 7) & ~7;
  const int tb = threads == WI_WIDE ? 4 : 2;  // rows of a block
  m.kb = (K + tb - 1) / tb;
  m.NB = m.kb * (m.kb + 1) / 2;
  m.SL = 1;
  while (2 * m.SL * m.NB <= threads && m.SL < 8) m.SL *= 2;
  size_t area = sizeof(double) * (shared_ldl ? 3 : 7) * T;  // phase 1
  const size_t stage = sizeof(int2) * 2 * (size_t)(tb * m.kb) * WI_RS, pack = sizeof(double) * K * (K + 1) / 2,
               f32 = sizeof(float) * (size_t)K * m.KP;
  area = area > stage ? area : stage;
  area = area > pack ? area : pack;
  area = area > f32 ? area : f32;
  size_t at = (area + 15) & ~(size_t)15;
  auto take = [&](size_t n) {
    const size_t o = at;
    at += (n + 15) & ~(size_t)15;
    return (int)o;
  };
  m.tri = take(sizeof(uint16_t) * (size_t)K * (K + 1) / 2);
  m.fw = take(sizeof(double) * 4 * K);  // f and w, double-buffered
  m.dk = take(sizeof(double) * 2 * K);  // D, 1 / sqrt(D)
  m.scale = take(sizeof(int) * 2 * K);  // the columns' sums of squares (fp32 bits), their scales
  m.total = (int)at;
  return m;
}

// The series of an item, rows of LT samples in fixed point (8 bytes) and fp32 (4)
// from a 16-byte boundary, lie in the slot's X_w and Q (16 bytes a sample in rows
// of T, 8-byte aligned): too long for them at T = 1, 2, 3, 5, 6 and 9, which the
// item kernel takes.
__host__ __device__ inline bool wide_slot_fits(int T) { return 3 * ld_t(T) + 2 <= 4 * T; }

template <bool SHARED_LDL, int THREADS>
__global__ void __launch_bounds__(THREADS, THREADS == WI_WIDE ? 2 : SHARED_LDL ? 8 : 5)
    grid_wide_kernel(BuildArgs args, int n_designs, const double* pair_cm, const int* pair_bad) {
  const ffs_grid_desc& d = args.d;
  const ffs_grid_out& o = args.o;
  const int T = d.T, K = d.K, LT = ld_t(T);
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  constexpr int nth = THREADS, NW = THREADS / 32, TB = THREADS == WI_WIDE ? 4 : 2;
  extern __shared__ double2 gi_smem[];
  char* sm = reinterpret_cast<char*>(gi_smem);
  const WidePlan pl = wide_plan(T, K, SHARED_LDL, THREADS);
  const int KP = pl.KP, kb = pl.kb, SL = pl.SL;
  double* area = reinterpret_cast<double*>(sm);
  uint16_t* tri = reinterpret_cast<uint16_t*>(sm + pl.tri);
  double* fw = reinterpret_cast<double*>(sm + pl.fw);
  double *dk = reinterpret_cast<double*>(sm + pl.dk), *rs = dk + K;
  int *colss = reinterpret_cast<int*>(sm + pl.scale), *scale = colss + K;
  __shared__ double red[32];
  __shared__ float fred[NW];
  __shared__ int flag, bad_r;
  for (int i = wid; i < K; i += NW)
    for (int j = lane; j <= i; j += 32) tri[i * (i + 1) / 2 + j] = (uint16_t)(i << 8 | j);

  for (int item = blockIdx.x; item < d.P * n_designs; item += gridDim.x) {
    const int p = item % d.P, pd = item;
    const float* Xd = d.X + (size_t)(item / d.P) * T * K;
    const PairScratch s = scratch_of(o.work, blockIdx.x, T, K);
    // the slot: X_w in fixed point and in fp32 (then Q), rows of LT samples
    int2* fx = reinterpret_cast<int2*>(((uintptr_t)s.Xw + 15) & ~(uintptr_t)15);
    float* xf = reinterpret_cast<float*>(fx + (size_t)K * LT);
    const double *cc = area, *cm = area + T, *cr = area + 2 * T;
    __syncthreads();  // the area's last use
    if constexpr (SHARED_LDL) {
      const double* src = pair_cm + (size_t)p * 4 * T;
      for (int i = tid; i < 3 * T; i += nth) area[i] = src[i];
      if (tid == 0) bad_r = pair_bad[p];
    } else {
      ldl_of_pair(d, o, p, area, area + T, area + 2 * T, area + 3 * T, red, &bad_r);
    }
    if (tid == 0) flag = 0;
    for (int j = tid; j < K; j += nth) colss[j] = 0;
    __syncthreads();

    // ---- 2. the columns' scales, from the recursion in fp32 (the largest sum of
    // squares of a run times their number), then X_w
    const float4* cf = reinterpret_cast<const float4*>(o.coef) + (size_t)p * T;
    for (int e = tid; e < K * d.n_runs; e += nth) {
      const int j = e % K, t0 = d.run_start[e / K], t1 = d.run_start[e / K + 1];
      float xp = 0.f, vp = 0.f, ss = 0.f;
#pragma unroll 8
      for (int t = t0; t < t1; ++t) {
        const float x = __ldg(Xd + (size_t)t * K + j);
        const float4 q = cf[t];
        vp = fmaf(-q.y, vp, fmaf(-q.x, xp, x));
        xp = x;
        const float w = vp * q.w;
        ss = fmaf(w, w, ss);
      }
      atomicMax(colss + j, __float_as_int(ss));
    }
    __syncthreads();
    bool over = false;
    for (int j = tid; j < K; j += nth)
      over = !norm_scale(__int_as_float(colss[j]) * (float)d.n_runs, scale[j]) || over;
    __syncthreads();
    for (int e = tid; e < K * d.n_runs; e += nth) {
      const int j = e % K, t0 = d.run_start[e / K], t1 = d.run_start[e / K + 1], sc = scale[j];
      int2* fr = fx + (size_t)j * LT;
      float* xr = xf + (size_t)j * LT;
      double xp = 0.0, vp = 0.0;  // c = m = 0 at the run's start
      float ss = 0.f;
      float xn[4];
      auto load = [&](int tq) {
#pragma unroll
        for (int k = 0; k < 4; ++k) xn[k] = tq + k >= t0 && tq + k < t1 ? __ldg(Xd + (size_t)(tq + k) * K + j) : 0.f;
      };
      load(t0 & ~3);
      for (int tq = t0 & ~3; tq < t1; tq += 4) {
        const float xb[4] = {xn[0], xn[1], xn[2], xn[3]};
        load(tq + 4);
        int2 f[4];
        float w4[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          const int t = tq + k;
          f[k] = make_int2(0, 0);
          w4[k] = 0.f;
          if (t >= t0 && t < t1) {
            const double x = f2d_exact(xb[k]);
            const double z = x - cc[t] * xp;
            vp = z - cm[t] * vp;
            xp = x;
            const double w = vp * cr[t];
            f[k] = fixed_of<5>(w, sc, over);
            w4[k] = d2f_exact(w);
            ss = fmaf(w4[k], w4[k], ss);
          }
        }
        if (tq >= t0 && (tq + 4 <= t1 || t1 == T)) {  // whole, or the last of the row with its padding
          *reinterpret_cast<int4*>(fr + tq) = make_int4(f[0].x, f[0].y, f[1].x, f[1].y);
          *reinterpret_cast<int4*>(fr + tq + 2) = make_int4(f[2].x, f[2].y, f[3].x, f[3].y);
          *reinterpret_cast<float4*>(xr + tq) = make_float4(w4[0], w4[1], w4[2], w4[3]);
        } else {
#pragma unroll
          for (int k = 0; k < 4; ++k) {
            const int t = tq + k;
            if (t >= t0 && (t < t1 || t1 == T)) {
              fr[t] = f[k];
              xr[t] = w4[k];
            }
          }
        }
      }
      over = over || !norm_fits(ss * (float)d.n_runs, sc);
    }
    if (over) flag = 1;
    __syncthreads();
    bool left = flag != 0;

    // ---- 3. X_w'X_w, into XtX and (FP64) the slot's Lx
    if (!left) {
      int2* buf = reinterpret_cast<int2*>(area);
      const int rows = TB * kb, nch = (T + WI_CS - 1) / WI_CS;
      auto stage = [&](int c) {
        int2* b = buf + (c & 1) * rows * WI_RS;
        for (int e = tid; e < rows * (WI_CS / 2); e += nth) {
          const int j = e / (WI_CS / 2), h = e % (WI_CS / 2), t = c * WI_CS + 2 * h;
          const bool in = j < K && t < LT;
          const int2* src = in ? fx + (size_t)j * LT + t : fx;
          const uint32_t dst = static_cast<uint32_t>(__cvta_generic_to_shared(b + j * WI_RS + 2 * h));
          asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(in ? 16 : 0)
                       : "memory");
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
      };
      for (int b0 = 0; b0 < pl.NB * SL; b0 += nth) {
        const int b = b0 + tid, sl = b % SL;
        const bool on = b < pl.NB * SL;
        int bi = 0, bj = 0;
        if (on) tri_index(b / SL, bi, bj);
        FixedDot2 acc[TB][TB];
        stage(0);
        for (int c = 0; c < nch; ++c) {
          if (c + 1 < nch) {
            stage(c + 1);
            asm volatile("cp.async.wait_group 1;" ::: "memory");
          } else {
            asm volatile("cp.async.wait_group 0;" ::: "memory");
          }
          __syncthreads();
          if (on) {
            const int4* r0 = reinterpret_cast<const int4*>(buf + (c & 1) * rows * WI_RS);
            const int4 *ri = r0 + bi * (WI_RS / 2), *rj = r0 + bj * (WI_RS / 2);
            for (int h = sl; h < WI_CS / 2; h += SL) {
              int4 x[TB];
#pragma unroll
              for (int u = 0; u < TB; ++u) x[u] = ri[u * kb * (WI_RS / 2) + h];
#pragma unroll
              for (int v = 0; v < TB; ++v) {
                const int4 y = rj[v * kb * (WI_RS / 2) + h];
#pragma unroll
                for (int u = 0; u < TB; ++u) {
                  acc[u][v].add(x[u].x, x[u].y, y.x, y.y);
                  acc[u][v].add(x[u].z, x[u].w, y.z, y.w);
                }
              }
            }
          }
          __syncthreads();
        }
#pragma unroll
        for (int u = 0; u < TB; ++u)
#pragma unroll
          for (int v = 0; v < TB; ++v) {
            FixedDot2& f = acc[u][v];
            for (int m = 1; m < SL; m <<= 1) {
              f.hh += __shfl_xor_sync(0xffffffffu, f.hh, m);
              f.x += __shfl_xor_sync(0xffffffffu, f.x, m);
            }
            const int i = bi + u * kb, j = bj + v * kb;
            if (on && sl == 0 && i < K && j < K) {
              const double x = f.value(scale[i], scale[j]);
              s.Lx[i * K + j] = x;
              s.Lx[j * K + i] = x;
              o.XtX[(size_t)pd * K * K + i * K + j] = (float)x;
              o.XtX[(size_t)pd * K * K + j * K + i] = (float)x;
            }
          }
      }
      __syncthreads();

      // ---- 4. the factor and its inverse. A holds the packed triangle; column
      // k of A (before its division by sqrt(D_k)) goes to row k of s.Lx
      double* A = area;
      for (int e = tid; e < K * (K + 1) / 2; e += nth) {
        const int rc = tri[e];
        A[e] = s.Lx[(rc >> 8) * K + (rc & 255)];
      }
      __syncthreads();
      constexpr int LA = 32;  // entries of f per warp of the look-ahead
      const int nla = (K + LA - 1) / LA;
      const Fold fold{A, fw, dk, s.Lx, K};
      for (int k = -1; k < K - 1; ++k) {
        const bool bad = wid < nla && fold_ahead(fold, k, wid * LA + lane);
        if (k >= 0) {
          const int E = K * (K + 1) / 2;
#pragma unroll 2
          for (int e = (k + 2) * (k + 3) / 2 + tid; e < E; e += nth) fold_entry(fold, k, e, tri[e] >> 8, tri[e] & 255);
        }
        left = __syncthreads_or(bad);
        if (left) break;
      }
    }
    __syncthreads();
    if (left) {
      if constexpr (SHARED_LDL) {
        const double* src = pair_cm + (size_t)p * 4 * T;
        for (int i = tid; i < 3 * T; i += nth) area[i] = src[i];
        __syncthreads();
      } else {
        ldl_of_pair(d, o, p, area, area + T, area + 2 * T, area + 3 * T, red, &bad_r);
      }
      item_global<false>(args, s, p, pd, Xd, cc, cm, cr, nullptr, bad_r, red, &flag);
      continue;
    }
    double* A = area;
    // the last row's rank-1 share went no further than f; Li = D^-1/2 Lu^-1
    for (int k = tid; k < K; k += nth) {
      const double r = rsqrt_newton(dk[k]);
      rs[k] = r;
      fw[k] = 2.0 * log(fabs(dk[k] * r) + 1e-10);
    }
    __syncthreads();
    if (tid == 0) {
      double ld = 0.0;
      for (int j = 0; j < K; ++j) ld += fw[j];
      o.logdet_XtX[pd] = ld;
      o.info[pd] = bad_r ? 2 : 0;
    }
    for (int e = tid; e < K * (K + 1) / 2; e += nth) {
      const int rc = tri[e], i = rc >> 8, j = rc & 255;
      const double v = i == j ? rs[i] : A[e] * rs[i];
      A[e] = v;
      s.Li[i * K + j] = v;
    }
    __syncthreads();
    for (int j = tid; j < K; j += nth) {
      double acc = 0.0;
      for (int k = j; k < K; ++k) {
        const double v = A[k * (k + 1) / 2 + j];
        acc = fma(v, v, acc);
      }
      o.Adiag[(size_t)pd * K + j] = (float)acc;
    }
    if (o.Afull) {  // all of A, for the per-voxel blocks of the -dsort fit
      for (int e = tid; e < K * (K + 1) / 2; e += nth) {
        const int rc = tri[e], i = rc >> 8, j = rc & 255;
        double acc = 0.0;
        for (int k = i; k < K; ++k) acc = fma(A[k * (k + 1) / 2 + i], A[k * (k + 1) / 2 + j], acc);
        o.Afull[(size_t)pd * K * K + i * K + j] = (float)acc;
        o.Afull[(size_t)pd * K * K + j * K + i] = (float)acc;
      }
    }
    __syncthreads();

    // ---- 5. Q = X_w Lx^-T in fp32; lx[i][j], j contiguous
    float* lx = reinterpret_cast<float*>(area);
    for (int e = tid; e < K * KP; e += nth) {
      const int i = e / KP, j = e % KP;
      lx[e] = j < K && j >= i ? (float)(j == i ? dk[i] * rs[i] : s.Lx[i * K + j] * rs[i]) : 0.f;
    }
    __syncthreads();
    for (int t2 = tid; t2 < LT / 2; t2 += nth) {
      float2* q = reinterpret_cast<float2*>(xf) + t2;
      for (int j0 = 0; j0 < K; j0 += 8) {
        float2 a[8];
#pragma unroll
        for (int c = 0; c < 8; ++c) a[c] = j0 + c < K ? q[(size_t)(j0 + c) * (LT / 2)] : make_float2(0.f, 0.f);
#pragma unroll 4
        for (int i = 0; i < j0; ++i) {
          const float2 qi = q[(size_t)i * (LT / 2)];
          const float4 l0 = *reinterpret_cast<const float4*>(lx + i * KP + j0);
          const float4 l1 = *reinterpret_cast<const float4*>(lx + i * KP + j0 + 4);
          const float l[8] = {l0.x, l0.y, l0.z, l0.w, l1.x, l1.y, l1.z, l1.w};
#pragma unroll
          for (int c = 0; c < 8; ++c) {
            a[c].x = fmaf(-l[c], qi.x, a[c].x);
            a[c].y = fmaf(-l[c], qi.y, a[c].y);
          }
        }
#pragma unroll
        for (int c = 0; c < 8; ++c) {
          if (j0 + c < K) {
            const float* l = lx + (j0 + c) * KP + j0;
            a[c].x /= l[c];
            a[c].y /= l[c];
#pragma unroll
            for (int e = c + 1; e < 8; ++e) {
              a[e].x = fmaf(-l[e], a[c].x, a[e].x);
              a[e].y = fmaf(-l[e], a[c].y, a[e].y);
            }
          }
        }
#pragma unroll
        for (int c = 0; c < 8; ++c)
          if (j0 + c < K) q[(size_t)(j0 + c) * (LT / 2)] = a[c];
      }
    }
    __syncthreads();

    // ---- 6. U = L^-T Q, the backward recursions of each column and run
    float* const U = o.U + (size_t)pd * K * LT;
    float umax = 0.f;
    for (int e = tid; e < K * d.n_runs; e += nth) {
      const int j = e % K, t0 = d.run_start[e / K], t1 = d.run_start[e / K + 1];
      const float* q = xf + (size_t)j * LT;
      float* u = U + (size_t)j * LT;
      if (t1 == T)
        for (int t = T; t < LT; ++t) u[t] = 0.f;
      float xn = 0.f, mn = 0.f, cn = 0.f;  // x_{t+1}, m_{t+1}, c_{t+1} (0 past a run's end)
      auto step = [&](float qt, float4 c4) {
        const float x = fmaf(-mn, xn, qt * c4.w);
        const float ut = fmaf(-cn, xn, x);
        xn = x;
        mn = c4.y;
        cn = c4.x;
        umax = fmaxf(umax, fabsf(ut));
        return ut;
      };
      int t = t1 - 1;
      for (; t >= t0 && (t & 3) != 3; --t) u[t] = step(q[t], cf[t]);
#pragma unroll 2
      for (; t - 3 >= t0; t -= 4) {
        const float4 q4 = *reinterpret_cast<const float4*>(q + t - 3);
        const float4 c3 = cf[t], c2 = cf[t - 1], c1 = cf[t - 2], c0 = cf[t - 3];
        float4 r;
        r.w = step(q4.w, c3);
        r.z = step(q4.z, c2);
        r.y = step(q4.y, c1);
        r.x = step(q4.x, c0);
        *reinterpret_cast<float4*>(u + t - 3) = r;
      }
      for (; t >= t0; --t) u[t] = step(q[t], cf[t]);
    }
    for (int off = 16; off > 0; off >>= 1) umax = fmaxf(umax, __shfl_xor_sync(0xffffffffu, umax, off));
    if (lane == 0) fred[wid] = umax;
    // Lx^-1 for G, beside
    float* li = reinterpret_cast<float*>(area);
    for (int e = tid; e < K * KP; e += nth) {
      const int i = e / KP, j = e % KP;
      li[e] = j <= i ? (float)s.Li[i * K + j] : 0.f;
    }
    __syncthreads();
    if (o.U_hi) {
      // fp16 hi/lo split of U * 2^e, e placing max|U| in [128, 256)
      float mx = 0.f;
      for (int w = 0; w < NW; ++w) mx = fmaxf(mx, fred[w]);
      const int ex = scale_exp(mx);
      if (tid == 0) o.uexp[pd] = ex;
      const bool pw = ex >= -126 && ex <= 127;
      const float p2 = pw ? __int_as_float((ex + 127) << 23) : 0.f;
      for (int j = wid; j < K; j += NW) {  // a warp per column
        const float2* u = reinterpret_cast<const float2*>(U + (size_t)j * LT);
        uint32_t* ho = reinterpret_cast<uint32_t*>(o.U_hi + ((size_t)pd * K + j) * d.ld_u);
        uint32_t* lo = reinterpret_cast<uint32_t*>(o.U_lo + ((size_t)pd * K + j) * d.ld_u);
#pragma unroll 4
        for (int h = lane; h < (d.ld_u >> 1); h += 32) {
          const float2 y = 2 * h < LT ? u[h] : make_float2(0.f, 0.f);
          uint16_t h0, l0, h1, l1;
          split_fp16(pw ? __fmul_rn(y.x, p2) : ldexpf(y.x, ex), h0, l0);
          split_fp16(pw ? __fmul_rn(y.y, p2) : ldexpf(y.y, ex), h1, l1);
          ho[h] = (uint32_t)h0 | ((uint32_t)h1 << 16);
          lo[h] = (uint32_t)l0 | ((uint32_t)l1 << 16);
        }
      }
    }
    if (args.const_flag && p == args.p0) const_of_design(args, pd / d.P, Xd, s.Li, K, true, s.A, red);

    // ---- 8. G = U Lx^-1 in fp32
    for (int t2 = tid; t2 < LT / 2; t2 += nth) {
      const float2* u = reinterpret_cast<const float2*>(U) + t2;
      float2* g = reinterpret_cast<float2*>(o.G + (size_t)pd * K * LT) + t2;
      for (int j0 = 0; j0 < K; j0 += 8) {
        float2 a[8];
#pragma unroll
        for (int c = 0; c < 8; ++c) a[c] = make_float2(0.f, 0.f);
#pragma unroll 4
        for (int i = j0; i < K; ++i) {  // li is zero above its diagonal
          const float2 ui = u[(size_t)i * (LT / 2)];
          const float4 l0 = *reinterpret_cast<const float4*>(li + i * KP + j0);
          const float4 l1 = *reinterpret_cast<const float4*>(li + i * KP + j0 + 4);
          const float l[8] = {l0.x, l0.y, l0.z, l0.w, l1.x, l1.y, l1.z, l1.w};
#pragma unroll
          for (int c = 0; c < 8; ++c) {
            a[c].x = fmaf(ui.x, l[c], a[c].x);
            a[c].y = fmaf(ui.y, l[c], a[c].y);
          }
        }
#pragma unroll
        for (int c = 0; c < 8; ++c)
          if (j0 + c < K) g[(size_t)(j0 + c) * (LT / 2)] = a[c];
      }
    }
    item_tail(d, o, s, pd, red, &flag);
  }
}

// ---- Design basis: Q0 = X Lx^-T, Lx the FP64 Cholesky factor of X'X (Q0 is
// U of the pair (0, 0), where R = I and X_w = X: the grid build's to the rounding
// of FP64, so of its fp32 form almost always the same bits), and the centring
// test c = (X'X)^-1 X'1. Two launches: the Gram entries of [X | 1] spread over
// CTAs (in fixed point up to DB_FIXED_K columns, else each a chain of FP64 FMAs
// whose latency bounds it), then one CTA for the factor, Q0 and c. work: [NE] Gram entries of [X | 1] (packed lower triangle), [K][T]
// doubles (QR fallback), then K x K doubles when K > DB_SMEM_K.

constexpr int DB_ENTRIES = 32;   // Gram entries per CTA: one warp's lanes
constexpr int DB_FIXED_K = 40;   // Gram entries in fixed point up to this K (wider: too few of them per staged column)
constexpr int DB_SMEM_K = 64;    // the factor stays in shared memory up to this K
constexpr int DB_THREADS = 256;  // the finishing CTA (its MGS fallback's sums depend on it)

__host__ __device__ inline int db_entries(int K) { return (K + 1) * (K + 2) / 2; }

// Samples of the design staged per pass: a multiple of 4 (the Dot4 chains
// continue across passes), with (K + 1) columns of (chunk + 1) doubles within
// 96 KB of shared memory.
inline int db_chunk(int T, int K) {
  const int fit = (96 * 1024 / (8 * (K + 1)) - 1) & ~3;
  const int t4 = (T + 3) & ~3;
  return fit < t4 ? fit : t4;
}

__global__ void __launch_bounds__(256) design_gram_kernel(int T, int K, int chunk, int fixed,
                                                          const float* __restrict__ Xg, double* __restrict__ gram) {
  extern __shared__ double xt[];  // [ncol][chunk + 1]: the columns this CTA reads (FP64 or fixed point), odd row stride
  __shared__ int cmax[DB_FIXED_K + 1];
  const int ne = db_entries(K);
  const int e0 = blockIdx.x * DB_ENTRIES;
  const int e1 = min(e0 + DB_ENTRIES, ne);
  int ihi, jhi;
  tri_index(e1 - 1, ihi, jhi);
  const int ncol = ihi + 1;  // the entries' rows i <= ihi read columns 0..ihi (column K is the constant)
  const int ld = chunk + 1;
  const int e = e0 + (int)threadIdx.x;
  const bool mine = threadIdx.x < 32 && e < e1;
  int i = 0, j = 0;
  if (mine) tri_index(e, i, j);
  if (fixed) {  // the columns' scales
    for (int c = threadIdx.x; c < ncol; c += blockDim.x) cmax[c] = c < K ? 0 : __float_as_int(1.f);
    __syncthreads();
    for (int idx = threadIdx.x; idx < T * min(ncol, K); idx += blockDim.x) {
      const int t = idx / min(ncol, K), c = idx % min(ncol, K);
      atomicMax(cmax + c, __float_as_int(fabsf(Xg[(size_t)t * K + c])));
    }
  }
  int2* xi = reinterpret_cast<int2*>(xt);
  Dot4 acc;
  FixedDot fx;
  bool over = false;
  for (int t0 = 0; t0 < T; t0 += chunk) {
    const int n = min(chunk, T - t0);
    __syncthreads();
    for (int idx = threadIdx.x; idx < n * ncol; idx += blockDim.x) {
      const int t = idx / ncol, c = idx % ncol;
      const double x = c < K ? f2d_exact(Xg[(size_t)(t0 + t) * K + c]) : 1.0;
      if (fixed)
        xi[c * ld + t] = fixed_of<0>(x, fixed_scale(__int_as_float(cmax[c])), over);
      else
        xt[c * ld + t] = x;
    }
    __syncthreads();
    if (mine && fixed)
      for (int t = 0; t < n; ++t) fx.add(xi[i * ld + t], xi[j * ld + t]);
    else if (mine)
      acc.run(xt + i * ld, xt + j * ld, n);
  }
  // a sample that is not finite leaves the fixed point: no factor, as its FP64 sums give none
  if (fixed) over = __syncthreads_or(over);
  if (mine)
    gram[e] = over ? (double)NAN : fixed ? fx.value(fixed_scale(__int_as_float(cmax[i])), fixed_scale(__int_as_float(cmax[j]))) : acc.sum();
}

__global__ void __launch_bounds__(DB_THREADS) design_basis_kernel(int T, int K, const float* __restrict__ X,
                                                                  const double* __restrict__ gram, double* work,
                                                                  float* Q0, int* info, int* const_flag,
                                                                  float* const_coef) {
  __shared__ double red[32];
  __shared__ int flag;
  extern __shared__ double sm[];  // rd [K], cv [K]; K <= DB_SMEM_K: M [K][K], mf [K][K] fp32, q [K][DB_THREADS] fp32
  const int LT = ld_t(T);
  const bool small = K <= DB_SMEM_K;
  double* rd = sm;
  double* cv = rd + K;
  double* Qd = work + db_entries(K);  // [K][T] (QR fallback)
  double* M = small ? cv + K : Qd + (size_t)K * T;
  // the fp32 factor: in shared memory, else in the QR slot (unused once the
  // Cholesky factor exists)
  float* mf = small ? reinterpret_cast<float*>(M + (size_t)K * K) : reinterpret_cast<float*>(Qd);
  float* qs = small ? mf + (size_t)K * K : nullptr;
  for (int idx = threadIdx.x; idx < K * (LT - T); idx += blockDim.x)
    Q0[(size_t)(idx / (LT - T)) * LT + T + idx % (LT - T)] = 0.f;
  for (int e = threadIdx.x; e < K * (K + 1) / 2; e += blockDim.x) {
    int i, j;
    tri_index(e, i, j);
    M[i * K + j] = gram[e];
    M[j * K + i] = gram[e];
  }
  for (int j = threadIdx.x; j < K; j += blockDim.x) cv[j] = gram[K * (K + 1) / 2 + j];  // row K: X'1
  __syncthreads();
  if (block_cholesky(M, K, K, &flag, rd)) {
    for (int idx = threadIdx.x; idx < K * K; idx += blockDim.x) mf[idx] = (float)M[idx];
    __syncthreads();
    // Q0 row by row, the grid build's fp32 recursion; a row's earlier entries
    // are read back from shared memory (from Q0 itself when K is large)
    for (int t = threadIdx.x; t < T; t += blockDim.x) {
      float* q = small ? qs + threadIdx.x : Q0 + t;
      const size_t qst = small ? DB_THREADS : LT;
      for (int j = 0; j < K; ++j) {
        float acc = X[(size_t)t * K + j];
        for (int i = 0; i < j; ++i) acc = fmaf(-mf[j * K + i], q[i * qst], acc);
        const float v = acc / mf[j * K + j];
        q[j * qst] = v;
        if (small) Q0[(size_t)j * LT + t] = v;
      }
    }
    if (const_flag) {
      // c = (X'X)^-1 X'1 from the same factor (one warp: forward and back
      // substitution, a column of updates per step), accepted when
      // ||X c - 1||^2 <= 1e-12 T
      if (threadIdx.x < 32) {
        const int lane = threadIdx.x;
        for (int j = 0; j < K; ++j) {
          const double yj = cv[j] * rd[j];
          __syncwarp();
          for (int i = j + 1 + lane; i < K; i += 32) cv[i] = fma(-M[i * K + j], yj, cv[i]);
          if (lane == 0) cv[j] = yj;
          __syncwarp();
        }
        for (int j = K - 1; j >= 0; --j) {
          const double cj = cv[j] * rd[j];
          __syncwarp();
          for (int i = lane; i < j; i += 32) cv[i] = fma(-M[j * K + i], cj, cv[i]);
          if (lane == 0) cv[j] = cj;
          __syncwarp();
        }
      }
      __syncthreads();
      double part = 0.0;
      for (int t = threadIdx.x; t < T; t += blockDim.x) {
        double r = -1.0;
        for (int j = 0; j < K; ++j) r = fma(f2d_exact(X[(size_t)t * K + j]), cv[j], r);
        part = fma(r, r, part);
      }
      const double ss = block_sum(part, red);
      const bool ok = ss <= 1e-12 * (double)T;
      for (int j = threadIdx.x; j < K; j += blockDim.x) const_coef[j] = ok ? (float)cv[j] : 0.f;
      if (threadIdx.x == 0) *const_flag = ok ? 1 : 0;
    }
    if (threadIdx.x == 0) *info = 0;
    return;
  }
  if (const_flag) {  // X'X not positive definite: no centring
    for (int j = threadIdx.x; j < K; j += blockDim.x) const_coef[j] = 0.f;
    if (threadIdx.x == 0) *const_flag = 0;
  }
  // QR of X by modified Gram-Schmidt (twice) in FP64, the grid build's
  // fallback on X_w = X
  for (int j = 0; j < K; ++j) {
    double* q = Qd + (size_t)j * T;
    for (int t = threadIdx.x; t < T; t += blockDim.x) q[t] = (double)X[(size_t)t * K + j];
    __syncthreads();
    for (int pass = 0; pass < 2; ++pass) {
      for (int i = 0; i < j; ++i) {
        const double* qi = Qd + (size_t)i * T;
        double part = 0.0;
        for (int t = threadIdx.x; t < T; t += blockDim.x) part += qi[t] * q[t];
        const double rij = block_sum(part, red);
        for (int t = threadIdx.x; t < T; t += blockDim.x) q[t] -= rij * qi[t];
        __syncthreads();
      }
    }
    double part = 0.0;
    for (int t = threadIdx.x; t < T; t += blockDim.x) part += q[t] * q[t];
    const double nrm = sqrt(block_sum(part, red));
    const double inv = nrm > 0.0 ? 1.0 / nrm : 0.0;
    for (int t = threadIdx.x; t < T; t += blockDim.x) {
      q[t] *= inv;
      Q0[(size_t)j * LT + t] = (float)q[t];
    }
    __syncthreads();
  }
  if (threadIdx.x == 0) *info = 1;
}

}  // namespace

}  // namespace ffsk

extern "C" size_t ffs_design_basis_work_bytes(int T, int K) {
  const size_t kk = K > ffsk::DB_SMEM_K ? (size_t)K * K : 0;
  return sizeof(double) * ((size_t)ffsk::db_entries(K) + (size_t)K * T + kk);
}

extern "C" int ffs_design_basis(int T, int K, const float* X, void* work, float* Q0, int* info, int* const_flag,
                                float* const_coef, void* stream) {
  using namespace ffsk;
  clear_error();
  FFS_REQUIRE(T > 0 && K > 0 && K <= T, "ffs_design_basis: T=%d K=%d", T, K);
  FFS_REQUIRE(X && work && Q0 && info, "ffs_design_basis: null buffer");
  FFS_REQUIRE(!const_flag == !const_coef, "ffs_design_basis: const_flag and const_coef go together");
  double* gram = static_cast<double*>(work);
  const int chunk = db_chunk(T, K);
  FFS_REQUIRE(chunk >= 4, "ffs_design_basis: K=%d too wide", K);
  const size_t gsm = sizeof(double) * (size_t)(K + 1) * (chunk + 1);
  FFS_CUDA(ensure_dyn_smem(reinterpret_cast<const void*>(design_gram_kernel), gsm));
  const int nb = ceil_div(db_entries(K), DB_ENTRIES);
  const int fixed = K <= DB_FIXED_K && T <= FX_TMAX;
  design_gram_kernel<<<nb, 256, gsm, (cudaStream_t)stream>>>(T, K, chunk, fixed, X, gram);
  if (const int rc = check_launch("design_gram_kernel")) return rc;
  const size_t fsm = K <= DB_SMEM_K ? sizeof(double) * 2 * K + sizeof(double) * (size_t)K * K +
                                          sizeof(float) * (size_t)K * K + sizeof(float) * (size_t)K * DB_THREADS
                                    : sizeof(double) * 2 * K;
  FFS_CUDA(ensure_dyn_smem(reinterpret_cast<const void*>(design_basis_kernel), fsm));
  design_basis_kernel<<<1, DB_THREADS, fsm, (cudaStream_t)stream>>>(T, K, X, gram, gram, Q0, info, const_flag,
                                                                   const_coef);
  return check_launch("design_basis_kernel");
}

extern "C" size_t ffs_grid_work_bytes(int T, int K, int P) {
  return sizeof(double) * ffsk::pair_doubles(T, K) * (size_t)P;
}

// Per-slot scratch of the CTAs, then (more than one design) the pre-pass's
// factors of R: cm [P][T][4] doubles and bad [P] ints.
static size_t designs_slot_doubles(int T, int K, int P, int n_designs, int max_ctas) {
  const long long items = (long long)P * (n_designs > 0 ? n_designs : 1);
  const long long cap = max_ctas > 0 && max_ctas < FFS_GRID_MAX_SLOTS ? max_ctas : FFS_GRID_MAX_SLOTS;
  return (ffsk::pair_doubles(T, K) * (size_t)(items < cap ? items : cap) + 1) & ~(size_t)1;  // 16-byte aligned end
}

extern "C" size_t ffs_grid_work_bytes_designs(int T, int K, int P, int n_designs, int max_ctas) {
  size_t n = designs_slot_doubles(T, K, P, n_designs, max_ctas);
  if (n_designs > 1) n += (size_t)P * 4 * T + ((size_t)P + 1) / 2;
  return sizeof(double) * n;
}

// Shared memory of phase 1: 4 T doubles, or with the band its window and tables.
static size_t phase1_smem(const ffs_grid_desc& d) {
  return sizeof(double) * (d.band ? ffsk::band_chol_doubles(d.band_w, d.n_runs) : 4 * (size_t)d.T);
}

// A T past 200 KB of 4 T doubles is refused (with the band, past 200 KB of 1.5 T doubles and the powers of a too).
static bool too_long(const ffs_grid_desc& d) {
  size_t n = 4 * (size_t)d.T;
  if (d.band) n = std::max(n, (size_t)d.T + (d.T + 1) / 2 + (size_t)d.band_w + 1);
  return sizeof(double) * n > 200 * 1024;
}

// The item kernel of a build; the two kernels and their widths give the same bits.
// grid_item_kernel has the shorter latency and
// takes the builds of up to GI_KMAX columns whose items run in one wave of its
// CTAs (two up to 16 columns); grid_wide_kernel does less work on more CTAs and
// takes the others whose factor fits: with 128 threads while the items
// outnumber two CTAs an SM and the columns are at most WI_NARROW_K, else with 320.
// us, grid_item_kernel / 128 / 320 threads: P = 117, T = 331, K = 13: 106 / 120 /
// 128; P = 231, T = 600, K = 20: 197 / 262 / 239; P = 561, T = 331, K = 13: 140 / 165 /
// 277; T = 400, K = 20: 307 / 248 / 344; P = 231, K = 32: - / 242 / 215; P = 561,
// K = 44: - / 502 / 639, K = 64: - / 1300 / 1184; 20 designs of T = 855, K = 18: 8006 /
// 4545 / 8732. grid_build_kernel takes the rest (more than FX_TMAX samples, whose
// sums leave the integers' range, and the banded R).
static int launch_items(const ffsk::BuildArgs& args, int n_designs, int grid, const double* pair_cm,
                        const int* pair_bad, cudaStream_t st, const char* who) {
  using namespace ffsk;
  const ffs_grid_desc& d = args.d;
  const ffs_grid_out& o = args.o;
  FFS_REQUIRE(!too_long(d), "%s: T=%d too long", who, d.T);
  int sms = 0;
  FFS_CUDA(sm_count(&sms));
  const long long items = (long long)d.P * n_designs;
  const bool fixed = d.T <= FX_TMAX && !d.band && (((uintptr_t)o.U_hi | (uintptr_t)o.U_lo) & 3) == 0;
  const bool narrow = d.K <= WI_NARROW_K && items > 2 * sms;
  const WidePlan wp = wide_plan(d.T, d.K, pair_cm != nullptr, narrow ? WI_NARROW : WI_WIDE);
  const bool wide = fixed && d.K <= WI_KMAX && wide_slot_fits(d.T) && wp.total <= 200 * 1024 &&
                    (((uintptr_t)o.U | (uintptr_t)o.G) & 15) == 0;
  const ItemPlan pl = item_plan(d.T, d.K, d.n_runs);
  if (fixed && d.K <= GI_KMAX && pl.total <= 200 * 1024) {
    const long long wave = sms * std::min<long long>(GI_CTAS, 225 * 1024 / (pl.total + 2048));
    if (!wide || items <= (d.K <= 16 ? 2 : 1) * wave) {
      auto kern = pair_cm ? grid_item_kernel<true> : grid_item_kernel<false>;
      FFS_CUDA(ensure_dyn_smem(reinterpret_cast<const void*>(kern), pl.total));
      kern<<<grid, GI_ENTRY + 32 * pl.PW, pl.total, st>>>(args, n_designs, pair_cm, pair_bad);
      return check_launch("grid_item_kernel");
    }
  }
  if (wide) {
    auto kern = pair_cm ? (narrow ? grid_wide_kernel<true, WI_NARROW> : grid_wide_kernel<true, WI_WIDE>)
                        : (narrow ? grid_wide_kernel<false, WI_NARROW> : grid_wide_kernel<false, WI_WIDE>);
    FFS_CUDA(ensure_dyn_smem(reinterpret_cast<const void*>(kern), wp.total));
    // no more CTAs than run at once: a slot's series are then still in L2 when its
    // next item overwrites them (20 designs: 4767 -> 4545 us)
    if (narrow) grid = std::min(grid, 8 * sms);
    kern<<<grid, narrow ? WI_NARROW : WI_WIDE, wp.total, st>>>(args, n_designs, pair_cm, pair_bad);
    return check_launch("grid_wide_kernel");
  }
  // phase 1's scratch beside the coefficients while that leaves room for four CTAs an SM
  const int tmp_smem = !pair_cm && sizeof(double) * 7 * d.T <= 50 * 1024;
  size_t smem = sizeof(double) * (tmp_smem ? 7 : 3) * d.T;
  if (d.band) smem = pair_cm ? sizeof(double) * band_stage_doubles(d.band_w) : phase1_smem(d);
  auto kern = d.band ? (pair_cm ? grid_build_kernel<true, true> : grid_build_kernel<false, true>)
                     : (pair_cm ? grid_build_kernel<true, false> : grid_build_kernel<false, false>);
  FFS_CUDA(ensure_dyn_smem(reinterpret_cast<const void*>(kern), smem));
  kern<<<grid, GB_THREADS, smem, st>>>(args, n_designs, pair_cm, pair_bad, tmp_smem);
  return check_launch("grid_build_kernel");
}

// n_sets needs its index arrays and the Fsets output
static int check_sets(const ffs_grid_desc* d, const ffs_grid_out* o, const char* who) {
  FFS_REQUIRE(d->n_sets >= 0, "%s: n_sets=%d", who, d->n_sets);
  FFS_REQUIRE(d->n_sets == 0 || (d->set_ptr && d->set_idx && o->Fsets), "%s: column sets need set_ptr, set_idx and Fsets",
              who);
  return FFS_OK;
}

// The centring test of a build (ffs_grid_build_centred).
struct Centring {
  int p0;
  int* flag;
  float* coef;
};

static int build_single(const ffs_grid_desc* d, const ffs_grid_out* o, const Centring& c, void* stream) {
  using namespace ffsk;
  clear_error();
  FFS_REQUIRE(d && o, "ffs_grid_build: null descriptor");
  FFS_REQUIRE(d->T > 0 && d->K > 0 && d->P > 0 && d->n_runs > 0,
              "ffs_grid_build: T=%d K=%d P=%d n_runs=%d must be positive", d->T, d->K, d->P,
              d->n_runs);
  FFS_REQUIRE(d->K <= d->T, "ffs_grid_build: K=%d exceeds T=%d", d->K, d->T);
  FFS_REQUIRE(d->n_task >= 0 && d->n_task <= d->K, "ffs_grid_build: bad n_task=%d", d->n_task);
  if (const int rc = check_sets(d, o, "ffs_grid_build")) return rc;
  FFS_REQUIRE(!o->U_hi || (o->U_lo && o->uexp), "ffs_grid_build: U_hi needs U_lo and uexp");
  FFS_REQUIRE(!o->U_hi || (d->ld_u >= d->T && d->ld_u % 8 == 0),
              "ffs_grid_build: ld_u=%d must be >= T and a multiple of 8", d->ld_u);
  FFS_REQUIRE(d->run_start && d->tau && d->a && d->b && d->X, "ffs_grid_build: null input");
  FFS_REQUIRE(o->coef && o->logdet_R && o->logdet_XtX && o->U && o->G && o->Adiag && o->XtX &&
                  o->info && o->work,
              "ffs_grid_build: null output");
  FFS_REQUIRE(!d->band || (d->band_w >= 1 && d->band_w <= FFS_BAND_MAX_W && o->band_L && o->band_coef),
              "ffs_grid_build: the banded R needs 1 <= band_w=%d <= %d, band_L and band_coef", d->band_w,
              FFS_BAND_MAX_W);
  return launch_items(BuildArgs{*d, *o, c.p0, c.flag, c.coef}, 1, d->P, nullptr, nullptr, (cudaStream_t)stream,
                      "ffs_grid_build");
}

extern "C" int ffs_grid_build(const ffs_grid_desc* d, const ffs_grid_out* o, void* stream) {
  return build_single(d, o, Centring{}, stream);
}

static int build_designs(const ffs_grid_desc* d, int n_designs, int max_ctas, const ffs_grid_out* o, const Centring& c,
                         void* stream) {
  using namespace ffsk;
  clear_error();
  FFS_REQUIRE(d && o, "ffs_grid_build_designs: null descriptor");
  FFS_REQUIRE(n_designs > 0, "ffs_grid_build_designs: n_designs=%d must be positive", n_designs);
  FFS_REQUIRE(d->T > 0 && d->K > 0 && d->P > 0 && d->n_runs > 0,
              "ffs_grid_build_designs: T=%d K=%d P=%d n_runs=%d must be positive", d->T, d->K, d->P, d->n_runs);
  FFS_REQUIRE((long long)d->P * n_designs < (1LL << 31), "ffs_grid_build_designs: too many items");
  FFS_REQUIRE(!d->band || (d->band_w >= 1 && d->band_w <= FFS_BAND_MAX_W && o->band_L && o->band_coef),
              "ffs_grid_build_designs: the banded R needs 1 <= band_w=%d <= %d, band_L and band_coef", d->band_w,
              FFS_BAND_MAX_W);
  FFS_REQUIRE(d->K <= d->T, "ffs_grid_build_designs: K=%d exceeds T=%d", d->K, d->T);
  FFS_REQUIRE(d->n_task >= 0 && d->n_task <= d->K, "ffs_grid_build_designs: bad n_task=%d", d->n_task);
  if (const int rc = check_sets(d, o, "ffs_grid_build_designs")) return rc;
  FFS_REQUIRE(!o->U_hi || (o->U_lo && o->uexp), "ffs_grid_build_designs: U_hi needs U_lo and uexp");
  FFS_REQUIRE(!o->U_hi || (d->ld_u >= d->T && d->ld_u % 8 == 0),
              "ffs_grid_build_designs: ld_u=%d must be >= T and a multiple of 8", d->ld_u);
  FFS_REQUIRE(d->run_start && d->tau && d->a && d->b && d->X, "ffs_grid_build_designs: null input");
  FFS_REQUIRE(o->coef && o->logdet_R && o->logdet_XtX && o->U && o->G && o->Adiag && o->XtX && o->info && o->work,
              "ffs_grid_build_designs: null output");
  const long long items = (long long)d->P * n_designs;
  const long long cap = max_ctas > 0 && max_ctas < FFS_GRID_MAX_SLOTS ? max_ctas : FFS_GRID_MAX_SLOTS;
  const int grid = (int)(items < cap ? items : cap);
  BuildArgs args{*d, *o, c.p0, c.flag, c.coef};
  double* pair_cm = nullptr;
  int* pair_bad = nullptr;
  if (n_designs > 1) {
    const size_t smem = phase1_smem(*d);
    FFS_REQUIRE(!too_long(*d), "ffs_grid_build_designs: T=%d too long", d->T);
    FFS_CUDA(ensure_dyn_smem(reinterpret_cast<const void*>(pair_ldl_kernel), smem));
    pair_cm = o->work + designs_slot_doubles(d->T, d->K, d->P, n_designs, max_ctas);
    pair_bad = reinterpret_cast<int*>(pair_cm + (size_t)d->P * 4 * d->T);
    pair_ldl_kernel<<<d->P, GB_THREADS, smem, (cudaStream_t)stream>>>(args, pair_cm, pair_bad);
    if (const int rc = check_launch("pair_ldl_kernel")) return rc;
  }
  return launch_items(args, n_designs, grid, pair_cm, pair_bad, (cudaStream_t)stream, "ffs_grid_build_designs");
}

extern "C" int ffs_grid_build_designs(const ffs_grid_desc* d, int n_designs, int max_ctas, const ffs_grid_out* o,
                                      void* stream) {
  return build_designs(d, n_designs, max_ctas, o, Centring{}, stream);
}

extern "C" int ffs_grid_build_centred(const ffs_grid_desc* d, int n_designs, int max_ctas, const ffs_grid_out* o, int p0,
                                      int* const_flag, float* const_coef, void* stream) {
  ffsk::clear_error();
  FFS_REQUIRE(d && const_flag && const_coef, "ffs_grid_build_centred: null argument");
  FFS_REQUIRE(p0 >= 0 && p0 < d->P, "ffs_grid_build_centred: p0=%d outside [0, P)", p0);
  const Centring c{p0, const_flag, const_coef};
  return n_designs == 1 && max_ctas <= 0 ? build_single(d, o, c, stream)
                                         : build_designs(d, n_designs, max_ctas, o, c, stream);
}

// ---------------------------------------------------------------------------
// Allocation-free variant of ffs_grid_build.
//
// Some callers cannot allocate device memory at the point where they build the
// grid factors: code running under a framework allocator that already owns
// the device's memory, or an embedding (for example a foreign-language binding
// driving the library from inside a larger pipeline) that is handed only its
// input and output buffers and has no allocator of its own. For them the FP64
// scratch lives in this file-scope device array instead of a caller-provided
// workspace. Every GPU that loads the library holds the array until the
// process exits.
namespace ffsk {
namespace {

constexpr size_t kStaticGridScratchBytes = (size_t)16 << 20;  // 16 MiB
static __device__ __align__(256) double g_grid_scratch[kStaticGridScratchBytes / sizeof(double)];

// Device address of g_grid_scratch, resolved once per device with that device
// current (host code may only pass this address to kernels, never the symbol).
// The cache lives as long as the process; a cudaDeviceReset would leave it
// stale (documented in the header).
double* static_grid_scratch(int* status) {
  static std::mutex mu;
  static double* addr[256] = {nullptr};
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess || dev < 0 || dev >= 256) {
    set_error("ffs_grid_build_noalloc: cudaGetDevice failed (%s)", cudaGetErrorString(e));
    *status = FFS_ERR_CUDA;
    return nullptr;
  }
  std::lock_guard<std::mutex> lock(mu);
  if (!addr[dev]) {
    double* ptr = nullptr;
    e = cudaGetSymbolAddress((void**)&ptr, g_grid_scratch);
    if (e != cudaSuccess || !ptr) {
      set_error("ffs_grid_build_noalloc: cudaGetSymbolAddress failed on device %d (%s)", dev,
                cudaGetErrorString(e));
      *status = FFS_ERR_CUDA;
      return nullptr;
    }
    addr[dev] = ptr;
  }
  *status = FFS_OK;
  return addr[dev];
}

}  // namespace
}  // namespace ffsk

extern "C" int ffs_grid_build_noalloc(const ffs_grid_desc* d, const ffs_grid_out* o, void* stream) {
  using namespace ffsk;
  clear_error();
  FFS_REQUIRE(d && o, "ffs_grid_build_noalloc: null descriptor");
  FFS_REQUIRE(d->T > 0 && d->K > 0 && d->P > 0 && d->n_runs > 0,
              "ffs_grid_build_noalloc: T=%d K=%d P=%d n_runs=%d must be positive", d->T, d->K, d->P, d->n_runs);
  FFS_REQUIRE(d->K <= d->T, "ffs_grid_build_noalloc: K=%d exceeds T=%d", d->K, d->T);
  FFS_REQUIRE(d->n_task >= 0 && d->n_task <= d->K, "ffs_grid_build_noalloc: bad n_task=%d", d->n_task);
  if (const int rc = check_sets(d, o, "ffs_grid_build_noalloc")) return rc;
  FFS_REQUIRE(!o->U_hi || (o->U_lo && o->uexp), "ffs_grid_build_noalloc: U_hi needs U_lo and uexp");
  FFS_REQUIRE(!o->U_hi || (d->ld_u >= d->T && d->ld_u % 8 == 0),
              "ffs_grid_build_noalloc: ld_u=%d must be >= T and a multiple of 8", d->ld_u);
  FFS_REQUIRE(d->run_start && d->tau && d->a && d->b && d->X, "ffs_grid_build_noalloc: null input");
  FFS_REQUIRE(o->coef && o->logdet_R && o->logdet_XtX && o->U && o->G && o->Adiag && o->XtX && o->info,
              "ffs_grid_build_noalloc: null output");
  FFS_REQUIRE(!d->band || (d->band_w >= 1 && d->band_w <= FFS_BAND_MAX_W && o->band_L && o->band_coef),
              "ffs_grid_build_noalloc: the banded R needs 1 <= band_w=%d <= %d, band_L and band_coef", d->band_w,
              FFS_BAND_MAX_W);
  const size_t need = sizeof(double) * pair_doubles(d->T, d->K) * (size_t)d->P;
  if (need > kStaticGridScratchBytes) {
    set_error("ffs_grid_build_noalloc: T=%d K=%d P=%d needs %zu bytes of scratch, above the %zu-byte static "
              "scratch; use ffs_grid_build with a caller-provided workspace",
              d->T, d->K, d->P, need, kStaticGridScratchBytes);
    return FFS_ERR_WORKSPACE;
  }
  int st = FFS_OK;
  double* scratch = static_grid_scratch(&st);
  if (!scratch) return st;
  // every scratch entry the kernel reads it writes first in the same launch, so
  // the previous call's contents need no clearing
  BuildArgs args{*d, *o, 0, nullptr, nullptr};
  args.o.work = scratch;
  return launch_items(args, 1, d->P, nullptr, nullptr, (cudaStream_t)stream, "ffs_grid_build_noalloc");
}

// The learned (a, b) proposal: simulation of training voxels and a
// 9 -> 64 -> 64 -> 2 GELU MLP with hand-written forward, backward and Adam
// kernels (the features come from the prep kernel, search.cu).
//
//   simulate  y_t = a y_{t-1} + e_t + b e_{t-1} per run (200 burn-in samples,
//             standardised per run), Y = X beta + sigma * noise, beta ~ N(0,1),
//             sigma ~ U(0.5, 2); normals from Philox4x32-10 (Salmon et al.,
//             SC'11) through Box-Muller.
//   MLP       exact-erf GELU; loss sum (out - y)^2 / (2 B); Adam.
#include <algorithm>

#include "common.cuh"

namespace ffsk {
namespace {

// ------------------------------------------------------------------ Philox
struct Philox {
  uint32_t c0, c1, c2, c3, k0, k1;
  float cache[4];
  int left;

  __device__ Philox(uint64_t seed, uint32_t stream) {
    c0 = 0; c1 = 0; c2 = stream; c3 = 0;
    k0 = (uint32_t)seed;
    k1 = (uint32_t)(seed >> 32);
    left = 0;
  }

  __device__ void block(uint32_t r[4]) {
    uint32_t x0 = c0, x1 = c1, x2 = c2, x3 = c3, a = k0, b = k1;
#pragma unroll
    for (int i = 0; i < 10; ++i) {
      const uint32_t hi0 = __umulhi(0xD2511F53u, x0), lo0 = 0xD2511F53u * x0;
      const uint32_t hi1 = __umulhi(0xCD9E8D57u, x2), lo1 = 0xCD9E8D57u * x2;
      x0 = hi1 ^ x1 ^ a;
      x1 = lo1;
      x2 = hi0 ^ x3 ^ b;
      x3 = lo0;
      a += 0x9E3779B9u;
      b += 0xBB67AE85u;
    }
    r[0] = x0; r[1] = x1; r[2] = x2; r[3] = x3;
    if (++c0 == 0) ++c1;
  }

  // uniform in (0, 1]
  __device__ static float u01(uint32_t x) { return ((float)(x >> 8) + 1.0f) * (1.0f / 16777216.0f); }

  __device__ float normal() {
    if (left == 0) {
      uint32_t r[4];
      block(r);
      float rad0 = sqrtf(-2.0f * logf(u01(r[0])));
      float th0 = 6.28318530717958647692f * u01(r[1]);
      float rad1 = sqrtf(-2.0f * logf(u01(r[2])));
      float th1 = 6.28318530717958647692f * u01(r[3]);
      cache[0] = rad0 * cosf(th0);
      cache[1] = rad0 * sinf(th0);
      cache[2] = rad1 * cosf(th1);
      cache[3] = rad1 * sinf(th1);
      left = 4;
    }
    return cache[--left];
  }

  __device__ float uniform() {
    uint32_t r[4];
    block(r);
    return u01(r[0]);
  }
};

struct SimArgs {
  int V, T, K, n_runs;
  const int* run_start;
  const float* X;       // [T][K]
  const float* a;       // [V]
  const float* b;       // [V]
  uint64_t seed;
  float* Y;             // [V][T]
};

__global__ void simulate_kernel(SimArgs s) {
  const int v = blockIdx.x * blockDim.x + threadIdx.x;
  if (v >= s.V) return;
  Philox rng(s.seed, (uint32_t)v);
  const float a = s.a[v], b = s.b[v];
  float* y = s.Y + (size_t)v * s.T;
  for (int r = 0; r < s.n_runs; ++r) {
    const int t0 = s.run_start[r], t1 = s.run_start[r + 1];
    float e_prev = rng.normal();
    float yt = e_prev;
    for (int i = 1; i < 200 + (t1 - t0); ++i) {
      const float e = rng.normal();
      yt = a * yt + e + b * e_prev;
      e_prev = e;
      if (i >= 200) y[t0 + i - 200] = yt;
    }
    double m = 0.0, q = 0.0;
    for (int t = t0; t < t1; ++t) m += y[t];
    m /= (double)(t1 - t0);
    for (int t = t0; t < t1; ++t) q += ((double)y[t] - m) * ((double)y[t] - m);
    const double sd = (t1 - t0 > 1) ? sqrt(q / (double)(t1 - t0 - 1)) : 1.0;
    const float inv = sd > 0.0 ? (float)(1.0 / sd) : 0.f;
    for (int t = t0; t < t1; ++t) y[t] = (float)(((double)y[t] - m) * inv);
  }
  const float sigma = 0.5f + 1.5f * rng.uniform();
  float beta[64];
  const int K = s.K;
  for (int j0 = 0; j0 < K; j0 += 64) {
    const int nj = min(64, K - j0);
    for (int j = 0; j < nj; ++j) beta[j] = rng.normal();
    for (int t = 0; t < s.T; ++t) {
      float acc = (j0 == 0) ? sigma * y[t] : y[t];
      for (int j = 0; j < nj; ++j) acc = fmaf(s.X[(size_t)t * K + j0 + j], beta[j], acc);
      y[t] = acc;
    }
  }
}

// --------------------------------------------------------------------- MLP
constexpr int NI = 9, NH = 64, NO = 2;
constexpr int OFF_W1 = 0, OFF_B1 = OFF_W1 + NH * NI, OFF_W2 = OFF_B1 + NH, OFF_B2 = OFF_W2 + NH * NH,
              OFF_W3 = OFF_B2 + NH, OFF_B3 = OFF_W3 + NO * NH, N_PARAMS = OFF_B3 + NO;

__device__ __forceinline__ float gelu(float z) { return 0.5f * z * (1.0f + erff(z * 0.70710678118654752f)); }

// gelu and its derivative, one erf for both
__device__ __forceinline__ void gelu_both(float z, float& g, float& d) {
  const float h = 0.5f * (1.0f + erff(z * 0.70710678118654752f));
  g = 0.5f * z * (1.0f + erff(z * 0.70710678118654752f));
  d = h + z * expf(-0.5f * z * z) * 0.3989422804014327f;
}

// A CTA of 256 threads works on tiles of MT samples held in shared memory with
// the sample fastest (rows of MS floats: 16-byte loads of 8 rows fall in
// distinct banks). A 64 x 64 layer over a tile is a small matrix product: each
// thread forms 4 samples x 4 units, so a 16-byte load serves 16 FMAs, with the
// units' sums in the order of a plain loop over the inputs (bias first). With
// one or two samples per thread, every weight was read from shared memory for
// one or two FMAs, and 8,192 samples gave 32 CTAs (forward 25 us, now 14; 200,000
// samples 86 us, now 84).
constexpr int MT = 64;
constexpr int MS = MT + 4;

struct MlpSmem {
  float w1[NH * NI], b1[NH], w2t[NH][NH], b2[NH], w3[NO * NH], b3[NO + 2];
  float x[NI + 1][MS];       // inputs
  float h1[NH][MS], h2[NH][MS];
};

// Parameters, W2 transposed (input-major).
__device__ __forceinline__ void mlp_load(const float* __restrict__ prm, MlpSmem& m) {
  const int tid = threadIdx.x, nt = blockDim.x;
  for (int i = tid; i < NH * NI; i += nt) m.w1[i] = prm[OFF_W1 + i];
  for (int i = tid; i < NH; i += nt) {
    m.b1[i] = prm[OFF_B1 + i];
    m.b2[i] = prm[OFF_B2 + i];
  }
  for (int i = tid; i < NH * NH; i += nt) m.w2t[i % NH][i / NH] = prm[OFF_W2 + i];
  for (int i = tid; i < NO * NH; i += nt) m.w3[i] = prm[OFF_W3 + i];
  if (tid < NO) m.b3[tid] = prm[OFF_B3 + tid];
}

// The tile's inputs (rows idx[s0 + s], or s0 + s), zero past ns.
__device__ __forceinline__ void mlp_inputs(const float* __restrict__ x, const int* __restrict__ idx, int s0, int ns,
                                           MlpSmem& m) {
  for (int i = threadIdx.x; i < MT * NI; i += blockDim.x) {
    const int s = i / NI, k = i % NI;
    m.x[k][s] = s < ns ? x[(size_t)(idx ? idx[s0 + s] : s0 + s) * NI + k] : 0.f;
  }
}

// The two hidden layers of the tile; D1 and D2 (NULL for the forward pass
// alone) receive the derivatives at their inputs. Starts and ends with a barrier.
template <bool GRAD>
__device__ __forceinline__ void mlp_hidden(MlpSmem& m, float (*d1)[MS], float (*d2)[MS]) {
  const int tid = threadIdx.x;
  __syncthreads();
  for (int i = tid; i < NH * MT; i += 256) {
    const int u = i / MT, s = i % MT;
    float z = m.b1[u];
#pragma unroll
    for (int k = 0; k < NI; ++k) z = fmaf(m.w1[u * NI + k], m.x[k][s], z);
    if (GRAD)
      gelu_both(z, m.h1[u][s], d1[u][s]);
    else
      m.h1[u][s] = gelu(z);
  }
  __syncthreads();
  const int s4 = 4 * (tid >> 4), u4 = 4 * (tid & 15);
  float z[4][4];  // [unit][sample]
#pragma unroll
  for (int j = 0; j < 4; ++j)
#pragma unroll
    for (int i = 0; i < 4; ++i) z[j][i] = m.b2[u4 + j];
#pragma unroll 8
  for (int k = 0; k < NH; ++k) {
    const float4 h = *reinterpret_cast<const float4*>(&m.h1[k][s4]);
    const float4 w = *reinterpret_cast<const float4*>(&m.w2t[k][u4]);
    const float hv[4] = {h.x, h.y, h.z, h.w}, wv[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
    for (int j = 0; j < 4; ++j)
#pragma unroll
      for (int i = 0; i < 4; ++i) z[j][i] = fmaf(wv[j], hv[i], z[j][i]);
  }
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    float g[4], d[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      if (GRAD)
        gelu_both(z[j][i], g[i], d[i]);
      else
        g[i] = gelu(z[j][i]);
    }
    *reinterpret_cast<float4*>(&m.h2[u4 + j][s4]) = make_float4(g[0], g[1], g[2], g[3]);
    if (GRAD) *reinterpret_cast<float4*>(&d2[u4 + j][s4]) = make_float4(d[0], d[1], d[2], d[3]);
  }
  __syncthreads();
}

__global__ void __launch_bounds__(256) mlp_forward_kernel(const float* __restrict__ prm, const float* __restrict__ x,
                                                          int B, float* __restrict__ out) {
  extern __shared__ float4 mlp_smem[];
  MlpSmem& m = *reinterpret_cast<MlpSmem*>(mlp_smem);
  mlp_load(prm, m);
  for (int s0 = blockIdx.x * MT; s0 < B; s0 += gridDim.x * MT) {
    const int ns = min(MT, B - s0);
    mlp_inputs(x, nullptr, s0, ns, m);
    mlp_hidden<false>(m, nullptr, nullptr);
    if (threadIdx.x < NO * MT) {
      const int s = threadIdx.x >> 1, o = threadIdx.x & 1;
      float z = m.b3[o];
#pragma unroll 16
      for (int u = 0; u < NH; ++u) z = fmaf(m.w3[o * NH + u], m.h2[u][s], z);
      if (s < ns) out[(size_t)(s0 + s) * NO + o] = z;
    }
    __syncthreads();  // the tile's arrays are free
  }
}

// Forward, loss and backward of a CTA's tiles; the parameter gradients stay in
// registers over them (16 entries of W2 per thread as 4 x 4 products summed over
// the samples, the others 1 to 3) and are added to grad once per CTA. With 16
// samples per CTA, 8,192 samples made 2.5 million global atomics: 160 us, now 21
// (65,536 samples: 1024 us, now 98).
struct MlpGradSmem {
  MlpSmem m;
  float w2[NH][NH];                  // unit-major
  float d1[NH][MS], d2[NH][MS];      // derivatives, then the deltas
  float dout[NO][MS];
  float part[8];
};

__global__ void __launch_bounds__(256) mlp_grad_kernel(const float* __restrict__ prm, const float* __restrict__ x,
                                                       const float* __restrict__ y, const int* __restrict__ idx,
                                                       int B, float inv_n, float* __restrict__ grad,
                                                       float* __restrict__ loss) {
  extern __shared__ float4 mlp_smem[];
  MlpGradSmem& g = *reinterpret_cast<MlpGradSmem*>(mlp_smem);
  MlpSmem& m = g.m;
  const int tid = threadIdx.x, lane = tid & 31;
  mlp_load(prm, m);
  for (int i = tid; i < NH * NH; i += 256) g.w2[i / NH][i % NH] = prm[OFF_W2 + i];
  const int tu = tid >> 4, tk = tid & 15;  // W2 entries (tu + 16 i, tk + 16 j)
  float g2[4][4] = {}, g1[3] = {}, gb = 0.f, g3 = 0.f, lsum = 0.f;
  auto row_dot = [&](const float* a, const float* b) {  // sum over the tile's samples
    float r = 0.f;
#pragma unroll 4
    for (int s = 0; s < MT; s += 4) {
      const float4 p = *reinterpret_cast<const float4*>(a + s), q = *reinterpret_cast<const float4*>(b + s);
      r = fmaf(p.x, q.x, r);
      r = fmaf(p.y, q.y, r);
      r = fmaf(p.z, q.z, r);
      r = fmaf(p.w, q.w, r);
    }
    return r;
  };
  for (int s0 = blockIdx.x * MT; s0 < B; s0 += gridDim.x * MT) {
    const int ns = min(MT, B - s0);
    mlp_inputs(x, idx, s0, ns, m);
    for (int s = tid; s < MT; s += 256) m.x[NI][s] = 1.f;  // the biases' input
    mlp_hidden<true>(m, g.d1, g.d2);
    if (tid < NO * MT) {
      const int s = tid >> 1, o = tid & 1;
      float z = m.b3[o];
#pragma unroll 16
      for (int u = 0; u < NH; ++u) z = fmaf(m.w3[o * NH + u], m.h2[u][s], z);
      const float e = s < ns ? z - y[(size_t)(idx ? idx[s0 + s] : s0 + s) * NO + o] : 0.f;
      g.dout[o][s] = e * inv_n;
      lsum = fmaf(0.5f * e * e, inv_n, lsum);
    }
    __syncthreads();
    for (int i = tid; i < NH * MT; i += 256) {
      const int u = i / MT, s = i % MT;
      g.d2[u][s] *= m.w3[u] * g.dout[0][s] + m.w3[NH + u] * g.dout[1][s];
    }
    __syncthreads();
    {
      const int s4 = 4 * (tid >> 4), k4 = 4 * (tid & 15);
      float d[4][4] = {};  // [input][sample]
#pragma unroll 8
      for (int u = 0; u < NH; ++u) {
        const float4 e = *reinterpret_cast<const float4*>(&g.d2[u][s4]);
        const float4 w = *reinterpret_cast<const float4*>(&g.w2[u][k4]);
        const float ev[4] = {e.x, e.y, e.z, e.w}, wv[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
        for (int j = 0; j < 4; ++j)
#pragma unroll
          for (int i = 0; i < 4; ++i) d[j][i] = fmaf(wv[j], ev[i], d[j][i]);
      }
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        float4 f = *reinterpret_cast<float4*>(&g.d1[k4 + j][s4]);
        f = make_float4(f.x * d[j][0], f.y * d[j][1], f.z * d[j][2], f.w * d[j][3]);
        *reinterpret_cast<float4*>(&g.d1[k4 + j][s4]) = f;
      }
    }
    __syncthreads();
#pragma unroll 2
    for (int s = 0; s < MT; s += 4) {
      float4 a[4], b[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        a[i] = *reinterpret_cast<const float4*>(&g.d2[tu + 16 * i][s]);
        b[i] = *reinterpret_cast<const float4*>(&m.h1[tk + 16 * i][s]);
      }
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          float r = g2[i][j];
          r = fmaf(a[i].x, b[j].x, r);
          r = fmaf(a[i].y, b[j].y, r);
          r = fmaf(a[i].z, b[j].z, r);
          g2[i][j] = fmaf(a[i].w, b[j].w, r);
        }
    }
#pragma unroll
    for (int i = 0; i < 3; ++i) {
      const int e = tid + 256 * i;
      if (e < NH * NI) g1[i] += row_dot(g.d1[e / NI], m.x[e % NI]);
    }
    if (tid < 2 * NH) {
      gb += row_dot(tid < NH ? g.d1[tid] : g.d2[tid - NH], m.x[NI]);
      if (tid < NO) g3 += row_dot(g.dout[tid], m.x[NI]);
    } else {
      const int e = tid - 2 * NH;
      g3 += row_dot(g.dout[e / NH], m.h2[e % NH]);
    }
    __syncthreads();  // the tile's arrays are free
  }
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) atomicAdd(grad + OFF_W2 + (tu + 16 * i) * NH + tk + 16 * j, g2[i][j]);
#pragma unroll
  for (int i = 0; i < 3; ++i)
    if (tid + 256 * i < NH * NI) atomicAdd(grad + OFF_W1 + tid + 256 * i, g1[i]);
  if (tid < 2 * NH) atomicAdd(grad + (tid < NH ? OFF_B1 + tid : OFF_B2 + tid - NH), gb);
  if (tid < NO) atomicAdd(grad + OFF_B3 + tid, g3);
  if (tid >= 2 * NH) atomicAdd(grad + OFF_W3 + tid - 2 * NH, g3);
  if (loss) {
    lsum = warp_sum(lsum);
    if (lane == 0) g.part[tid >> 5] = lsum;
    __syncthreads();
    if (tid == 0) {
      float r = 0.f;
      for (int w = 0; w < 8; ++w) r += g.part[w];
      atomicAdd(loss, r);
    }
  }
}

// Adam with bias correction; consumes and zeroes the gradient.
__global__ void adam_kernel(float* prm, float* grad, float* m, float* v, int n, float lr, float b1, float b2,
                            float eps, float c1, float c2) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const float g = grad[i];
  const float mi = b1 * m[i] + (1.f - b1) * g;
  const float vi = b2 * v[i] + (1.f - b2) * g * g;
  m[i] = mi;
  v[i] = vi;
  prm[i] -= lr * (mi / c1) / (sqrtf(vi / c2) + eps);
  grad[i] = 0.f;
}

}  // namespace
}  // namespace ffsk

using namespace ffsk;

extern "C" int ffs_mlp_param_count(void) { return N_PARAMS; }

extern "C" int ffs_arma_simulate(int V, int T, int K, int n_runs, const int* run_start, const float* X,
                                 const float* a, const float* b, uint64_t seed, float* Y, void* stream) {
  clear_error();
  FFS_REQUIRE(V > 0 && T > 0 && K >= 0 && n_runs > 0, "ffs_arma_simulate: bad sizes");
  FFS_REQUIRE(run_start && a && b && Y && (K == 0 || X), "ffs_arma_simulate: null buffer");
  SimArgs s{V, T, K, n_runs, run_start, X, a, b, seed, Y};
  simulate_kernel<<<ceil_div(V, 128), 128, 0, (cudaStream_t)stream>>>(s);
  return check_launch("simulate_kernel");
}

extern "C" int ffs_mlp_forward(const float* params, const float* x, int B, float* out, void* stream) {
  clear_error();
  FFS_REQUIRE(params && x && out && B > 0, "ffs_mlp_forward: bad arguments");
  // four CTAs an SM, each over its share of the tiles
  int sms = 0;
  FFS_CUDA(sm_count(&sms));
  FFS_CUDA(ensure_dyn_smem(reinterpret_cast<const void*>(mlp_forward_kernel), sizeof(MlpSmem)));
  mlp_forward_kernel<<<std::min(ceil_div(B, MT), 4 * sms), 256, sizeof(MlpSmem), (cudaStream_t)stream>>>(params, x, B,
                                                                                                        out);
  return check_launch("mlp_forward_kernel");
}

extern "C" int ffs_mlp_grad(const float* params, const float* x, const float* y, const int* idx, int B, int n_total,
                            float* grad, float* loss, void* stream) {
  clear_error();
  FFS_REQUIRE(params && x && y && grad && B > 0 && n_total > 0, "ffs_mlp_grad: bad arguments");
  int sms = 0;
  FFS_CUDA(sm_count(&sms));
  FFS_CUDA(ensure_dyn_smem(reinterpret_cast<const void*>(mlp_grad_kernel), sizeof(MlpGradSmem)));
  mlp_grad_kernel<<<std::min(ceil_div(B, MT), sms), 256, sizeof(MlpGradSmem), (cudaStream_t)stream>>>(
      params, x, y, idx, B, 1.0f / (float)n_total, grad, loss);
  return check_launch("mlp_grad_kernel");
}

extern "C" int ffs_mlp_adam(float* params, float* grad, float* m, float* v, int n, float lr, float beta1, float beta2,
                            float eps, int step, void* stream) {
  clear_error();
  FFS_REQUIRE(params && grad && m && v && n > 0 && step > 0, "ffs_mlp_adam: bad arguments");
  const float c1 = 1.0f - powf(beta1, (float)step), c2 = 1.0f - powf(beta2, (float)step);
  adam_kernel<<<ceil_div(n, 256), 256, 0, (cudaStream_t)stream>>>(params, grad, m, v, n, lr, beta1, beta2, eps, c1,
                                                                  c2);
  return check_launch("adam_kernel");
}

// Statistics of series and the distinct (a, b) of saved parameters, for fits
// that start from given (a, b) or carry voxelwise regressors.
#include "common.cuh"

namespace ffsk {

namespace {

// A value as an unevaluated sum hi + lo of two floats (about 48 bits): the
// error-free sums and products of Dekker (1971) and Knuth. The FP64 pipe takes
// one warp instruction per 19 cycles and SM; the dozen fp32 instructions of a
// compensated step take three.
struct Two {
  float hi, lo;
};

__device__ __forceinline__ Two two_sum(float a, float b) {
  const float s = __fadd_rn(a, b), z = __fsub_rn(s, a);
  return {s, __fadd_rn(__fsub_rn(a, __fsub_rn(s, z)), __fsub_rn(b, z))};
}

__device__ __forceinline__ Two add(Two a, Two b) {
  const Two s = two_sum(a.hi, b.hi);
  const float e = __fadd_rn(s.lo, __fadd_rn(a.lo, b.lo));
  const float h = __fadd_rn(s.hi, e);
  return {h, __fsub_rn(e, __fsub_rn(h, s.hi))};
}

__device__ __forceinline__ Two warp_add(Two v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1)
    v = add(v, Two{__shfl_xor_sync(0xffffffffu, v.hi, o), __shfl_xor_sync(0xffffffffu, v.lo, o)});
  return v;
}

// v / n for a whole number n
__device__ __forceinline__ Two div_int(Two v, float n) {
  const float h = __fdiv_rn(v.hi, n);
  const float r = __fadd_rn(__fmaf_rn(-h, n, v.hi), v.lo);
  const Two q = two_sum(h, __fdiv_rn(r, n));
  return q;
}

// One warp per series of T samples: its standard deviation (N - 1 divisor, two
// passes; NaN for T = 1) as the float nearest the compensated value, into
// scale[row] (at least 1e-8); and, with n_const, a count of the rows that are
// constant and nonzero (sd < 1e-8, mean |x| > 1e-8, to one part in 10^4 on the
// safe side). Bound by the read of the
// rows: 50,000 x 400 samples 51 us, against 960 us for conversions and a
// Welford pass in FP64.
__global__ void __launch_bounds__(256) series_sd_kernel(int rows, int T, const float* __restrict__ Y,
                                                        float* __restrict__ scale, int* n_const) {
  const int lane = threadIdx.x & 31;
  const int row = (int)((blockIdx.x * (size_t)blockDim.x + threadIdx.x) >> 5);
  if (row >= rows) return;  // warp-uniform
  const float* y = Y + (size_t)row * T;
  // the samples times the power of two that brings the largest near 1, exactly:
  // no square over- or underflows
  float amax = 0.f;
#pragma unroll 4
  for (int t = lane; t < T; t += 32) amax = fmaxf(amax, fabsf(y[t]));
  for (int o = 16; o > 0; o >>= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, o));
  const int e = amax > 0.f && isfinite(amax) ? max(-126, min(126, ilogbf(amax))) : 0;
  const float p2 = __int_as_float((127 - e) << 23), back = __int_as_float((127 + e) << 23);
  Two s{0.f, 0.f};
  float ab = 0.f;
#pragma unroll 4
  for (int t = lane; t < T; t += 32) {
    const float x = y[t] * p2;
    const Two u = two_sum(s.hi, x);
    s = {u.hi, __fadd_rn(s.lo, u.lo)};
    ab += fabsf(x);
  }
  const Two m = div_int(warp_add(s), (float)T);
  Two q{0.f, 0.f};
#pragma unroll 4
  for (int t = lane; t < T; t += 32) {
    const Two d0 = two_sum(y[t] * p2, -m.hi);
    const Two dd = two_sum(d0.hi, __fsub_rn(d0.lo, m.lo));  // m.lo need not be small beside d0.hi
    const float d = dd.hi, dl = dd.lo;
    const float p = __fmul_rn(d, d);
    const float e = __fmaf_rn(2.f * d, dl, __fmaf_rn(d, d, -p));
    const Two u = two_sum(q.hi, p);
    q = {u.hi, __fadd_rn(q.lo, __fadd_rn(u.lo, e))};
  }
  const Two v = div_int(warp_add(q), (float)(T - 1));
  // sqrt(v) by one Newton step from sqrt(hi): one rounding of the result
  const float s0 = __fsqrt_rn(v.hi);
  const float r = __fadd_rn(__fmaf_rn(-s0, s0, v.hi), v.lo);
  const float sd = ((s0 > 0.f && isfinite(s0)) ? __fadd_rn(s0, __fdiv_rn(r, 2.f * s0)) : s0) * back;
  if (n_const) {
    ab = warp_sum(ab) / (float)T * back;
    if (lane == 0 && sd < 1.0001e-8f && ab > 0.9999e-8f) atomicAdd(n_const, 1);
  }
  if (lane == 0 && scale) scale[row] = sd < 1e-8f ? 1e-8f : sd;  // a NaN stays
}

constexpr unsigned long long EMPTY = ~0ull;  // no pair's key: its first half is a NaN

__device__ __forceinline__ unsigned hash_of(unsigned long long k) {
  k ^= k >> 33;
  k *= 0xff51afd7ed558ccdull;  // the finaliser of MurmurHash3 (public domain)
  k ^= k >> 33;
  k *= 0xc4ceb9fe1a85ec53ull;
  return (unsigned)(k >> 32);
}

// Each voxel's (a, b) into an open-addressing table of 2^bits >= 2 V entries:
// slot[v], and at a pair's first insertion its number from *count, in pairs.
// A probe sequence ends at the latest after 2^bits entries, half of them empty.
// -0 counts as 0; *nan = 1 if some value is a NaN (that voxel gets slot 0).
__global__ void __launch_bounds__(256) distinct_insert_kernel(int V, const float2* __restrict__ ab, int bits,
                                                              unsigned long long* __restrict__ table,
                                                              int* __restrict__ number, int* __restrict__ slot,
                                                              float2* __restrict__ pairs, int* count, int* nan) {
  const int v = blockIdx.x * blockDim.x + threadIdx.x;
  if (v >= V) return;
  float2 p = ab[v];
  p.x = __fadd_rn(p.x, 0.f);
  p.y = __fadd_rn(p.y, 0.f);
  slot[v] = 0;
  if (isnan(p.x) || isnan(p.y)) {
    *nan = 1;
    return;
  }
  const unsigned long long key = ((unsigned long long)__float_as_uint(p.x) << 32) | __float_as_uint(p.y);
  const unsigned mask = (1u << bits) - 1;
  unsigned h = hash_of(key) & mask;
  for (unsigned i = 0; i <= mask; ++i, h = (h + 1) & mask) {
    unsigned long long cur = *reinterpret_cast<volatile unsigned long long*>(table + h);
    if (cur == EMPTY) {
      cur = atomicCAS(table + h, EMPTY, key);
      if (cur == EMPTY) {
        const int n = atomicAdd(count, 1);
        number[h] = n;
        pairs[n] = p;
        cur = key;
      }
    }
    if (cur == key) {
      slot[v] = (int)h;
      return;
    }
  }
}

__global__ void __launch_bounds__(256) distinct_number_kernel(int V, const int* __restrict__ number,
                                                              const int* __restrict__ slot, int* __restrict__ index) {
  const int v = blockIdx.x * blockDim.x + threadIdx.x;
  if (v < V) index[v] = number[slot[v]];
}

int table_bits(int V) {
  int b = 6;
  while ((1ll << b) < 2ll * V) ++b;
  return b;
}

}  // namespace
}  // namespace ffsk

using namespace ffsk;

extern "C" int ffs_series_sd(int rows, int T, const float* Y, float* scale, int* n_const, void* stream) {
  clear_error();
  FFS_REQUIRE(rows > 0 && T > 0 && Y && (scale || n_const), "ffs_series_sd: bad arguments (rows=%d T=%d)", rows, T);
  cudaStream_t st = (cudaStream_t)stream;
  if (n_const) FFS_CUDA(cudaMemsetAsync(n_const, 0, sizeof(int), st));
  series_sd_kernel<<<ceil_div(rows, 8), 256, 0, st>>>(rows, T, Y, scale, n_const);
  return check_launch("series_sd_kernel");
}

extern "C" size_t ffs_distinct_pairs_work_bytes(int V) {
  const size_t n = V > 0 ? (size_t)1 << table_bits(V) : 0;
  return n * (sizeof(unsigned long long) + sizeof(int)) + sizeof(int) * (size_t)(V > 0 ? V : 0);
}

extern "C" int ffs_distinct_pairs(int V, const float* ab, void* work, float* pairs, int* index, int* counts,
                                  void* stream) {
  clear_error();
  FFS_REQUIRE(V > 0 && V <= (1 << 29) && ab && work && pairs && index && counts,
              "ffs_distinct_pairs: bad arguments (V=%d)", V);
  FFS_REQUIRE((((uintptr_t)ab | (uintptr_t)work | (uintptr_t)pairs) & 7) == 0,
              "ffs_distinct_pairs: ab, work and pairs must be 8-byte aligned");
  cudaStream_t st = (cudaStream_t)stream;
  const int bits = table_bits(V);
  const size_t n = (size_t)1 << bits;
  auto* table = static_cast<unsigned long long*>(work);
  int* number = reinterpret_cast<int*>(table + n);
  int* slot = number + n;
  FFS_CUDA(cudaMemsetAsync(table, 0xff, n * sizeof(unsigned long long), st));
  FFS_CUDA(cudaMemsetAsync(number, 0, sizeof(int), st));  // read at slot 0 for a NaN voxel
  FFS_CUDA(cudaMemsetAsync(counts, 0, 2 * sizeof(int), st));
  distinct_insert_kernel<<<ceil_div(V, 256), 256, 0, st>>>(V, reinterpret_cast<const float2*>(ab), bits, table, number,
                                                           slot, reinterpret_cast<float2*>(pairs), counts, counts + 1);
  distinct_number_kernel<<<ceil_div(V, 256), 256, 0, st>>>(V, number, slot, index);
  return check_launch("distinct kernels");
}

// Flexible preconditioned conjugate gradients: operator application, exact
// dot products and vector updates, templated on the vector precision.  The
// FP64 form's dot products are exact and order free: each product a_i*b_i is
// scaled by 2^(96-E), 2^E > max|a|*max|b|,
// truncated to a 128-bit integer and summed with two 64-bit atomics.
#pragma once
#include "mmh_launch.cuh"

namespace mmh {

__device__ __forceinline__ double bits_d(const unsigned long long* b) { return __longlong_as_double((long long)*b); }

// value of a dot product's 128-bit fixed-point accumulator
__device__ __forceinline__ double fx_unscale(const unsigned long long* acc, int E) {
  __int128 s = (__int128)(((unsigned __int128)acc[1] << 64) | (unsigned __int128)acc[0]);
  bool neg = s < 0;
  unsigned __int128 a = neg ? (unsigned __int128)(-s) : (unsigned __int128)s;
  double r = __dadd_rn(scalbn(__ull2double_rn((unsigned long long)(a >> 64)), E - 32),
                       scalbn(__ull2double_rn((unsigned long long)a), E - 96));
  return neg ? -r : r;
}

// q = L[p] = (t1 + t2 + tdiag*p) * di2, max|q| into qbits
template <class T>
__global__ void k_apply(const T* __restrict__ p, const T* __restrict__ coef, int n, T di2, T* __restrict__ q,
                        unsigned long long* qbits) {
  i64 n3 = (i64)n * n * n;
  i64 t = (i64)blockIdx.x * blockDim.x + threadIdx.x;
  T m = T(0);
  if (t < n3) {
    int i, j, k;
    cell_of(t, n, i, j, k);
    T tdiag, t1, t2;
    op_terms(p, coef, n, n3, i, j, k, tdiag, t1, t2);
    T v = (t1 + t2 + tdiag * p[t]) * di2;
    q[t] = v;
    m = fabs(v);
  }
  block_max_commit(m, qbits);
}

// the FP64 form's dot product
static __global__ void k_dot(const double* __restrict__ a, const double* __restrict__ b, i64 count,
                             const unsigned long long* abits, const unsigned long long* bbits,
                             unsigned long long* acc) {
  double ma = bits_d(abits), mb = bits_d(bbits);
  __int128 s = 0;
  if (ma > 0.0 && mb > 0.0) {
    int E = ilogb(ma) + ilogb(mb) + 2;
    for (i64 t = (i64)blockIdx.x * blockDim.x + threadIdx.x; t < count; t += (i64)gridDim.x * blockDim.x)
      s += fx_bits(a[t] * b[t], 96 - E);
  }
  fx_block_commit(s, acc);
}

// x = x + alpha*p ; r = r - alpha*q ; max|r|
template <class T>
__global__ void k_pcg_update(T* __restrict__ x, T* __restrict__ r, const T* __restrict__ p, const T* __restrict__ q,
                             i64 count, const double* __restrict__ alpha, unsigned long long* rbits) {
  i64 t = (i64)blockIdx.x * blockDim.x + threadIdx.x;
  T a = (T)*alpha;
  T m = T(0);
  if (t < count) {
    x[t] = x[t] + a * p[t];
    T v = r[t] - a * q[t];
    r[t] = v;
    m = fabs(v);
  }
  block_max_commit(m, rbits);
}

// p = z + beta*p ; max|p|
template <class T>
__global__ void k_pcg_pupdate(T* __restrict__ p, const T* __restrict__ z, i64 count, const double* __restrict__ beta,
                              unsigned long long* pbits) {
  i64 t = (i64)blockIdx.x * blockDim.x + threadIdx.x;
  T b = (T)*beta;
  T m = T(0);
  if (t < count) {
    T v = z[t] + b * p[t];
    p[t] = v;
    m = fabs(v);
  }
  block_max_commit(m, pbits);
}

template <class T>
void launch_apply(const T* p, const T* coef, int n, T dx, T* q, unsigned long long* qbits, cudaStream_t s) {
  i64 n3 = (i64)n * n * n;
  prof_begin(kk<T>(KK_APPLY), s, n3, n);
  // (the FP64 form's grids of 32^3 and up take launch_apply64)
  bool done = false;
  if constexpr (std::is_same<T, float>::value) {
    done = n >= 32;
    if (use_march(n))
      launch_stencil_march<1>(p, nullptr, coef, n, T(1) / (dx * dx), q, qbits, s);
    else if (done)
      k_stencil_plane<T, 1><<<dim3(n / 32, n / 16, n), 256, 0, s>>>(p, nullptr, coef, n, T(1) / (dx * dx), q, nullptr,
                                                                   qbits);
  }
  if (!done) k_apply<T><<<grid_of(n3, kBlock), kBlock, 0, s>>>(p, coef, n, T(1) / (dx * dx), q, qbits);
  prof_end(kk<T>(KK_APPLY), s, n);
  count_launch();
}

// The FP32 updates of the mixed form's inner solve over whole vectors of four:
// a fixed grid of at most 8 blocks per SM walks the vectors with 16-byte
// loads and commits one maximum per block (the elementwise results and the
// maximum are those of k_pcg_update / k_pcg_pupdate).  count % 4 == 0.
static __global__ void __launch_bounds__(256) k_pcg_update_v4(float4* __restrict__ x, float4* __restrict__ r,
                                                       const float4* __restrict__ p, const float4* __restrict__ q,
                                                       i64 count4, const double* __restrict__ alpha,
                                                       unsigned long long* rbits) {
  const float a = (float)*alpha;
  unsigned m = 0;
  for (i64 t = (i64)blockIdx.x * blockDim.x + threadIdx.x; t < count4; t += (i64)gridDim.x * blockDim.x) {
    float4 xv = x[t], rv = r[t];
    const float4 pv = p[t], qv = q[t];
    xv.x = xv.x + a * pv.x; xv.y = xv.y + a * pv.y; xv.z = xv.z + a * pv.z; xv.w = xv.w + a * pv.w;
    rv.x = rv.x - a * qv.x; rv.y = rv.y - a * qv.y; rv.z = rv.z - a * qv.z; rv.w = rv.w - a * qv.w;
    x[t] = xv;
    r[t] = rv;
    const unsigned b0 = __float_as_uint(fabsf(rv.x)), b1 = __float_as_uint(fabsf(rv.y));
    const unsigned b2 = __float_as_uint(fabsf(rv.z)), b3 = __float_as_uint(fabsf(rv.w));
    m = max(m, max(max(b0, b1), max(b2, b3)));
  }
  block_max_commit(__uint_as_float(m), rbits);
}
static __global__ void __launch_bounds__(256) k_pcg_pupdate_v4(float4* __restrict__ p, const float4* __restrict__ z,
                                                        i64 count4, const double* __restrict__ beta,
                                                        unsigned long long* pbits) {
  const float b = (float)*beta;
  unsigned m = 0;
  for (i64 t = (i64)blockIdx.x * blockDim.x + threadIdx.x; t < count4; t += (i64)gridDim.x * blockDim.x) {
    float4 pv = p[t];
    const float4 zv = z[t];
    pv.x = zv.x + b * pv.x; pv.y = zv.y + b * pv.y; pv.z = zv.z + b * pv.z; pv.w = zv.w + b * pv.w;
    p[t] = pv;
    const unsigned b0 = __float_as_uint(fabsf(pv.x)), b1 = __float_as_uint(fabsf(pv.y));
    const unsigned b2 = __float_as_uint(fabsf(pv.z)), b3 = __float_as_uint(fabsf(pv.w));
    m = max(m, max(max(b0, b1), max(b2, b3)));
  }
  block_max_commit(__uint_as_float(m), pbits);
}

inline unsigned vec_blocks(i64 count4) {
  i64 b = (count4 + kBlock - 1) / kBlock;
  const i64 cap = 152 * 8;
  return (unsigned)(b < 1 ? 1 : (b > cap ? cap : b));
}

template <class T>
void launch_pcg_update(T* x, T* r, const T* p, const T* q, i64 count, const double* alpha, unsigned long long* rbits,
                       cudaStream_t s) {
  if constexpr (std::is_same<T, float>::value) {
    if (count % 4 == 0) {
      k_pcg_update_v4<<<vec_blocks(count / 4), kBlock, 0, s>>>(
          reinterpret_cast<float4*>(x), reinterpret_cast<float4*>(r), reinterpret_cast<const float4*>(p),
          reinterpret_cast<const float4*>(q), count / 4, alpha, rbits);
      count_launch();
      return;
    }
  }
  k_pcg_update<T><<<grid_of(count, kBlock), kBlock, 0, s>>>(x, r, p, q, count, alpha, rbits);
  count_launch();
}

template <class T>
void launch_pcg_pupdate(T* p, const T* z, i64 count, const double* beta, unsigned long long* pbits, cudaStream_t s) {
  if constexpr (std::is_same<T, float>::value) {
    if (count % 4 == 0) {
      k_pcg_pupdate_v4<<<vec_blocks(count / 4), kBlock, 0, s>>>(
          reinterpret_cast<float4*>(p), reinterpret_cast<const float4*>(z), count / 4, beta, pbits);
      count_launch();
      return;
    }
  }
  k_pcg_pupdate<T><<<grid_of(count, kBlock), kBlock, 0, s>>>(p, z, count, beta, pbits);
  count_launch();
}

#define MMH_INSTANTIATE_PCG(T)                                                                                   \
  template void launch_apply<T>(const T*, const T*, int, T, T*, unsigned long long*, cudaStream_t);             \
  template void launch_pcg_update<T>(T*, T*, const T*, const T*, i64, const double*, unsigned long long*,        \
                                     cudaStream_t);                                                              \
  template void launch_pcg_pupdate<T>(T*, const T*, i64, const double*, unsigned long long*, cudaStream_t);

}  // namespace mmh

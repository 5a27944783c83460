// FP32 kernels of the mixed-precision inner V-cycle (smoother, residual,
// restriction, prolongation, zero-mean).  FMA contraction stays enabled here.
#include <mutex>

#include "mmh_launch.cuh"
#include "mmh_pcg.cuh"

namespace mmh {

// Tile autotuning of the FP32 plane kernel (see gs_tile_choice), per device
// (up to 64) and grid size (2^0 .. 2^15).
static std::mutex g_tile_mu;
static signed char g_tile[64][16];
static bool g_tile_init = false;
std::atomic<int> gs_tile_override{-1};
std::atomic<int> stencil_march_pin{-1};

int gs_tile_choice(int n, const float* phi, const float* rhs, const float* coef, float dx2, float* scratch,
                   cudaStream_t s) {
  const int pin = gs_tile_override.load();
  if (pin >= 0 && pin < kGsShapes && gs_shape_fits(pin, n)) return pin;
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return 0;
  int lg = 0;
  while ((1 << lg) < n && lg < 15) ++lg;
  {
    std::lock_guard<std::mutex> lock(g_tile_mu);
    if (!g_tile_init) {
      for (auto& row : g_tile)
        for (auto& x : row) x = -1;
      g_tile_init = true;
    }
    if (g_tile[dev][lg] >= 0) return g_tile[dev][lg];
  }
  cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
  if (cudaStreamIsCapturing(s, &cap) != cudaSuccess || cap != cudaStreamCaptureStatusNone) return 0;
  cudaEvent_t e0, e1;
  if (cudaEventCreate(&e0) != cudaSuccess) return 0;
  if (cudaEventCreate(&e1) != cudaSuccess) {
    cudaEventDestroy(e0);
    return 0;
  }
  int best = 0;
  float best_ms = 0.f;
  for (int v = 0; v < kGsShapes; ++v) {
    if (!gs_shape_fits(v, n)) continue;
    gs_plane_half<float>(v, phi, phi, scratch, rhs, coef, n, dx2, 0, s);  // warm-up (attribute, caches)
    cudaEventRecord(e0, s);
    for (int r = 0; r < 3; ++r) gs_plane_half<float>(v, phi, phi, scratch, rhs, coef, n, dx2, 0, s);
    cudaEventRecord(e1, s);
    count_launch(4);
    float ms = 0.f;
    if (cudaEventSynchronize(e1) != cudaSuccess || cudaEventElapsedTime(&ms, e0, e1) != cudaSuccess) continue;
    if (v == 0 || ms < best_ms) {
      best = v;
      best_ms = ms;
    }
  }
  cudaEventDestroy(e0);
  cudaEventDestroy(e1);
  std::lock_guard<std::mutex> lock(g_tile_mu);
  g_tile[dev][lg] = (signed char)best;
  return best;
}

int gs_tile_chosen(int n, int* tx, int* ty) {
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return -1;
  int lg = 0;
  while ((1 << lg) < n && lg < 15) ++lg;
  std::lock_guard<std::mutex> lock(g_tile_mu);
  if (!g_tile_init || g_tile[dev][lg] < 0) return -1;
  const int v = g_tile[dev][lg];
  *tx = kGsShape[v].tx;
  *ty = kGsShape[v].ty;
  return v;
}

MMH_INSTANTIATE(float)
template float* launch_gs_sweeps<float>(float*, const float*, const float*, int, float, int, float*, cudaStream_t,
                                        bool);
MMH_INSTANTIATE_PCG(float)

// Dot products of FP32 vectors for the mixed form's inner solve, whose
// results are not bit-matched to the oracle: a fixed grid of kDotBlocks
// blocks, each thread summing its strided products in FP32 with four
// accumulators, each block reducing in a fixed pattern, and one block adding
// the block sums in FP64 in a fixed order -- deterministic, and bound by
// memory.  z.q and r.z share the read of z and its maximum (three passes over
// the vectors instead of five), and the block that ends last forms the
// solver's scalar: below 128^3 an iteration is bound by its launches, and this
// takes twelve of the seventeen between two cycles away.
__device__ __forceinline__ float block_sum_f32(float v, float* buf) {
  for (int d = 16; d > 0; d >>= 1) v += __shfl_down_sync(0xffffffffu, v, d);
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  if (lane == 0) buf[w] = v;
  __syncthreads();
  float t = 0.f;
  if (threadIdx.x == 0)
    for (int q = 0; q < (int)(blockDim.x >> 5); ++q) t += buf[q];
  return t;
}

// The value of one dot product from the sum v of its block sums, rounded as
// its fixed-point form (2^(E-96), 2^E > max|a| max|b|) holds it.
__device__ __forceinline__ double dot_rounded(double v, unsigned long long abits, unsigned long long bbits) {
  const unsigned long long inf_bits = 0x7FF0000000000000ull;
  if (abits == 0 || bbits == 0 || abits > inf_bits || bbits > inf_bits || abs_bits(v) >= inf_bits) return 0.0;
  // the maxima are widened FP32 values: normal, so ilogb is the exponent field
  const int E = (int)(abits >> 52) + (int)(bbits >> 52) - 2 * 1023 + 2;
  const __int128 fx = fx_bits(v, 96 - E);
  const unsigned long long acc[2] = {(unsigned long long)fx, (unsigned long long)((unsigned __int128)fx >> 64)};
  return fx_unscale(acc, E);
}
// The part of a thread in the sum of a product's block sums.  The sums are
// other blocks': read past L1.
__device__ __forceinline__ double dot_share(const double* part) {
  double s = 0.0;
#pragma unroll
  for (int q = 0; q < (kDotBlocks + 255) / 256; ++q) {
    const int e = threadIdx.x + 256 * q;
    if (e < kDotBlocks) s += __ldcg(part + e);
  }
  return s;
}
// The sum of 256 shares by halving (t + 128, t + 64, ...), by one warp; valid
// in lane 0.
__device__ __forceinline__ double dot_halve(const double* buf) {
  const int l = threadIdx.x & 31;
  double v = ((buf[l] + buf[l + 128]) + (buf[l + 64] + buf[l + 192])) +
             ((buf[l + 32] + buf[l + 160]) + (buf[l + 96] + buf[l + 224]));
  for (int d = 16; d > 0; d >>= 1) v += __shfl_down_sync(0xffffffffu, v, d);
  return v;
}

// One pass over the vectors and the scalar they give, by the block that ends
// last.  STAGE 0, after the first cycle: p = z, rz = r.z; 1: alpha = rz / p.q
// (a = p, b = q); 2: beta = -(alpha z.q) / rz, rz = r.z (a = z, b = q, c = r).
// 0 and 2 also take max|z|.  Clears the maxima that are read here and reduced
// into next.  The last block is what a small grid waits for: its two totals go
// to a warp each, with FP64 instructions in one warp where 256 threads halving
// in steps issued them in eight (64^3: 11 and 22 us for stages 1 and 2 so,
// 9 and 16 now).
template <int STAGE>
__global__ void __launch_bounds__(256) k_pcg_dot(const float* __restrict__ a, const float* __restrict__ b,
                                                 const float* __restrict__ c, float* __restrict__ p, i64 count,
                                                 double* part, PcgDev* P) {
  __shared__ float buf[32], buf2[32];
  __shared__ double dbuf[2][256], total[2];
  __shared__ int last;
  const i64 stride = (i64)gridDim.x * blockDim.x;
  i64 t = (i64)blockIdx.x * blockDim.x + threadIdx.x;
  float s[4] = {0.f, 0.f, 0.f, 0.f}, u[4] = {0.f, 0.f, 0.f, 0.f};
  unsigned m = 0;
  auto take = [&](i64 at, int k) {
    const float av = a[at];
    if (STAGE != 0) s[k] += av * b[at];
    if (STAGE != 1) {
      u[k] += c[at] * av;
      const unsigned ab = abs_bits(av);
      m = ab > m ? ab : m;
    }
    if (STAGE == 0) p[at] = av;
  };
  for (; t + 3 * stride < count; t += 4 * stride) {
    take(t, 0);
    take(t + stride, 1);
    take(t + 2 * stride, 2);
    take(t + 3 * stride, 3);
  }
  for (; t < count; t += stride) take(t, 0);
  if (STAGE != 0) {
    const float blk = block_sum_f32((s[0] + s[1]) + (s[2] + s[3]), buf);
    if (threadIdx.x == 0) part[blockIdx.x] = (double)blk;
  }
  if (STAGE != 1) {
    const float blk = block_sum_f32((u[0] + u[1]) + (u[2] + u[3]), buf2);
    if (threadIdx.x == 0) part[kDotBlocks + blockIdx.x] = (double)blk;
    block_max_commit(from_bits(m), &P->zbits);
  }
  if (threadIdx.x == 0) {
    __threadfence();
    last = atomicAdd(&P->arrived, 1u) == gridDim.x - 1;
  }
  __syncthreads();
  if (!last) return;
  __threadfence();
  const unsigned long long rb = __ldcg(&P->rbits), zb = __ldcg(&P->zbits), qb = __ldcg(&P->qbits),
                           pb = __ldcg(&P->pbits);
  if (STAGE != 0) dbuf[0][threadIdx.x] = dot_share(part);
  if (STAGE != 1) dbuf[1][threadIdx.x] = dot_share(part + kDotBlocks);
  __syncthreads();
  if (threadIdx.x < 64) {
    const int w = threadIdx.x >> 5;
    if (w == 0 ? STAGE != 0 : STAGE != 1) {
      const double v = dot_halve(dbuf[w]);
      if ((threadIdx.x & 31) == 0)
        total[w] = w == 0 ? dot_rounded(v, STAGE == 1 ? pb : zb, qb) : dot_rounded(v, rb, zb);
    }
  }
  __syncthreads();
  const double first = STAGE == 0 ? 0.0 : total[0], rz = STAGE == 1 ? 0.0 : total[1];
  if (threadIdx.x == 0) {
    P->arrived = 0;
    if constexpr (STAGE == 1) {
      P->pq = first;
      P->alpha = P->rz / first;
      P->rbits = 0;
    } else {
      if (STAGE == 2) P->beta = __ddiv_rn(-__dmul_rn(P->alpha, first), P->rz);
      P->rz = rz;
      P->pbits = STAGE == 0 ? zb : 0;
      P->zbits = 0;
      P->qbits = 0;
    }
  }
}

__global__ void k_pcg_start(PcgDev* P, double bmax) {
  PcgDev z{};
  z.rbits = (unsigned long long)__double_as_longlong(bmax);
  *P = z;
}

void launch_pcg_start(PcgDev* P, double bmax, cudaStream_t s) {
  k_pcg_start<<<1, 1, 0, s>>>(P, bmax);
  count_launch();
}
void launch_pcg_first32(float* p, const float* z, const float* r, i64 count, PcgDev* P, double* part,
                        cudaStream_t s) {
  k_pcg_dot<0><<<kDotBlocks, 256, 0, s>>>(z, nullptr, r, p, count, part, P);
  count_launch();
}
void launch_pcg_alpha32(const float* p, const float* q, i64 count, PcgDev* P, double* part, cudaStream_t s) {
  k_pcg_dot<1><<<kDotBlocks, 256, 0, s>>>(p, q, nullptr, nullptr, count, part, P);
  count_launch();
}
void launch_pcg_beta32(const float* z, const float* q, const float* r, i64 count, PcgDev* P, double* part,
                       cudaStream_t s) {
  k_pcg_dot<2><<<kDotBlocks, 256, 0, s>>>(z, q, r, nullptr, count, part, P);
  count_launch();
}

// FP64 residual with fused multiply-adds, for the outer loop of the mixed
// form (fewer FP64 operations; that form is not bit-matched to the oracle).
void launch_residual_fma(const double* phi, const double* rhs, const double* coef, int n, double dx, float* r32,
                         unsigned long long* maxbits, cudaStream_t s) {
  i64 n3 = (i64)n * n * n;
  double di2 = 1.0 / (dx * dx);
  prof_begin(KK_RESIDUAL, s, n3, n);
  if (n >= 32)
    k_stencil_plane<double, 0, true><<<dim3(n / 32, n / 16, n), 256, 0, s>>>(phi, rhs, coef, n, di2, nullptr, r32,
                                                                             maxbits);
  else
    k_residual<double, true><<<grid_of(n3, kBlock), kBlock, 0, s>>>(phi, rhs, coef, n, di2, nullptr, r32, maxbits);
  prof_end(KK_RESIDUAL, s, n);
  count_launch();
}
}  // namespace mmh

// Spectral outputs (scalar2gradient, mmh/gradient.f90; defp2delta,
// mmh/reconstruct.f90) as transforms along single lines.
//
// The displacement component a is F^-1[i k_a F[def]] and the density F^-1[|k|^2
// F[def]], so every output is a sum of operators that act along one axis:
// three passes, each transforming the lines of one axis forward, multiplying
// by i k and by k^2 and transforming back, replace one forward and four
// inverse three-dimensional transforms.  These are bound by the FP64 pipe
// (0.5e12 instructions/s against 5.6 TB/s of them), so the count of FP64
// instructions is what matters: about 125 per cell here, 370 before.
// Two real lines go through one complex transform (the operators are real).
//
// The reference's packed inverse transform (rlft3, recipes12.f90:77-135) pairs
// kx with n/2 - kx and so, where i k is not Hermitian (the Nyquist planes),
// spreads the planes kx = 0 and n/2 over alternating samples.  Worked through,
// with e^{+2 pi i k x / n} forward and C_k a line's transform:
//   x: C_{n/2} counts as the mean -pi C_{n/2} of the line's derivative;
//   y: the ky = n/2 term is pi w(x, z) with w along x the operator below on
//      T(x, z) = sum_y (-1)^y def, in place of 0; z alike with T(x, y);
//   w: T^_k -> i sgn(k) T^_k, its k = 0 term -T^_{n/2}, its k = n/2 term -T^_0.
//
// One CTA transforms LC pairs of lines in shared memory with Stockham stages
// of radix 4, 8 and 16 in registers.  Along y and z a CTA takes 2 LC
// consecutive x, so global accesses are runs of 64 to 256 bytes.
// Measured: the four outputs 3.7 ms at 256^3 (12.0 ms with the
// three-dimensional transforms, cuFFT and two packing kernels each).
#include <cmath>

#include "mmh_kernels.cuh"
#include "mmh_launch.cuh"

namespace mmh {
namespace {

template <int N> struct Fft;
template <> struct Fft<8> { static constexpr int LC = 4, NT = 32, S = 1, R0 = 8, R1 = 1, R2 = 1; };
template <> struct Fft<16> { static constexpr int LC = 8, NT = 32, S = 1, R0 = 16, R1 = 1, R2 = 1; };
template <> struct Fft<32> { static constexpr int LC = 16, NT = 64, S = 2, R0 = 4, R1 = 8, R2 = 1; };
template <> struct Fft<64> { static constexpr int LC = 16, NT = 128, S = 2, R0 = 8, R1 = 8, R2 = 1; };
template <> struct Fft<128> { static constexpr int LC = 16, NT = 128, S = 2, R0 = 8, R1 = 16, R2 = 1; };
template <> struct Fft<256> { static constexpr int LC = 8, NT = 128, S = 2, R0 = 16, R1 = 16, R2 = 1; };
template <> struct Fft<512> { static constexpr int LC = 4, NT = 256, S = 3, R0 = 8, R1 = 8, R2 = 8; };
template <> struct Fft<1024> { static constexpr int LC = 4, NT = 256, S = 3, R0 = 4, R1 = 16, R2 = 16; };

__device__ __forceinline__ double2 operator+(double2 a, double2 b) { return make_double2(a.x + b.x, a.y + b.y); }
__device__ __forceinline__ double2 operator-(double2 a, double2 b) { return make_double2(a.x - b.x, a.y - b.y); }
__device__ __forceinline__ double2 times_i(double2 a) { return make_double2(-a.y, a.x); }
__device__ __forceinline__ double2 cmul(double2 a, double wx, double wy) {
  return make_double2(fma(a.x, wx, -(a.y * wy)), fma(a.x, wy, a.y * wx));
}
// a times e^{i pi/4} and e^{3 i pi/4}
__device__ __forceinline__ double2 mul_w8(double2 a) {
  const double c = 0.70710678118654752440;
  return make_double2((a.x - a.y) * c, (a.x + a.y) * c);
}
__device__ __forceinline__ double2 mul_w83(double2 a) {
  const double c = 0.70710678118654752440;
  return make_double2((a.x + a.y) * -c, (a.x - a.y) * c);
}

// DFT of R values with e^{+2 pi i jk / R}, in place, natural order
__device__ __forceinline__ void dft4(double2& a, double2& b, double2& c, double2& d) {
  const double2 s = a + c, t = a - c, u = b + d, v = times_i(b - d);
  a = s + u;
  b = t + v;
  c = s - u;
  d = t - v;
}
template <int R>
__device__ __forceinline__ void dft(double2* v) {
  if constexpr (R == 4) {
    dft4(v[0], v[1], v[2], v[3]);
  } else if constexpr (R == 8) {
    dft4(v[0], v[2], v[4], v[6]);
    dft4(v[1], v[3], v[5], v[7]);
    const double2 o0 = v[1], o1 = mul_w8(v[3]), o2 = times_i(v[5]), o3 = mul_w83(v[7]);
    const double2 e0 = v[0], e1 = v[2], e2 = v[4], e3 = v[6];
    v[0] = e0 + o0; v[4] = e0 - o0;
    v[1] = e1 + o1; v[5] = e1 - o1;
    v[2] = e2 + o2; v[6] = e2 - o2;
    v[3] = e3 + o3; v[7] = e3 - o3;
  } else {
    const double c1 = 0.92387953251128675613, s1 = 0.38268343236508977173;  // cos, sin of pi/8
#pragma unroll
    for (int j = 0; j < 4; ++j) dft4(v[j], v[j + 4], v[j + 8], v[j + 12]);
    v[5] = cmul(v[5], c1, s1);     // j1 = 1: k2 = 1, 2, 3
    v[9] = mul_w8(v[9]);
    v[13] = cmul(v[13], s1, c1);
    v[6] = mul_w8(v[6]);           // j1 = 2
    v[10] = times_i(v[10]);
    v[14] = mul_w83(v[14]);
    v[7] = cmul(v[7], s1, c1);     // j1 = 3
    v[11] = mul_w83(v[11]);
    v[15] = cmul(v[15], -c1, -s1);
#pragma unroll
    for (int k = 0; k < 16; k += 4) dft4(v[k], v[k + 1], v[k + 2], v[k + 3]);
    // value k1 of group k2 (k = 4 k2 + k1 in v) is output k2 + 4 k1
    double2 t;
#define SWAP_(a, b) t = v[a]; v[a] = v[b]; v[b] = t
    SWAP_(1, 4); SWAP_(2, 8); SWAP_(3, 12); SWAP_(6, 9); SWAP_(7, 13); SWAP_(11, 14);
#undef SWAP_
  }
}

// tables of one size: twiddles e^{2 pi i k / n}, then 2 pi k / n^2 and (2 pi
// k / n)^2 / n for the signed k (0 at n/2 in the first)
__global__ void k_fft_tables(double* tab, int n) {
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= n) return;
  double s, c;
  sincospi(2.0 * k / n, &s, &c);
  tab[2 * k] = c;
  tab[2 * k + 1] = s;
  const double kap = 2.0 * 3.14159265358979323846 * (k <= n / 2 ? k : k - n) / n;
  tab[2 * n + k] = 2 * k == n ? 0.0 : kap / n;
  tab[3 * n + k] = kap * kap / n;
}

// T(x, z) = sum_y (-1)^y d (blockIdx.y = 0), T(x, y) = sum_z (-1)^z d (1):
// n x n each, x fastest.  Clears the x pass's word (see LineArgs).
__global__ void k_altsum(const double* __restrict__ d, int n, double* __restrict__ T, unsigned* bad) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= n * n) return;
  if (t == 0 && blockIdx.y == 0) *bad = 0;
  const int x = t & (n - 1), o = t / n;
  const i64 n2 = (i64)n * n;
  const double* p = d + x + (blockIdx.y == 0 ? n2 * o : (i64)n * o);
  const i64 st = blockIdx.y == 0 ? n : n2;
  double s = 0.0;
  for (int j = 0; j < n; j += 2) s += p[j * st] - p[(j + 1) * st];
  T[blockIdx.y * n2 + t] = s;
}

enum { kAxisX = 0, kAxisY = 1, kAxisZ = 2, kHilbert = 3 };
struct LineArgs {
  const double* src;
  double *grad, *delta;  // outputs of this axis (null: not wanted); delta is added to unless axis x
  const double* w;       // y, z: pi / n times the ky (kz) = n/2 operator's result
  const double* tab;
  int axis;
  // A cell that is not finite would reach its own lines only, where the
  // three-dimensional transform carries it into every value: the x pass sets
  // *bad when a line's sum is not finite, the z pass then leaves NaN everywhere.
  unsigned* bad;
  double* all;  // z: the displacement's three planes (null: not wanted)
};

template <int N>
__global__ void __launch_bounds__(Fft<N>::NT) k_lines(LineArgs a) {
  typedef Fft<N> F;
  constexpr int LC = F::LC, NT = F::NT, P = N + 1, RL = F::S == 3 ? F::R2 : F::S == 2 ? F::R1 : F::R0;
  static_assert(F::R0 * F::R1 * F::R2 == N && LC * (N / RL) <= NT && (F::S < 3 || LC * (N / F::R1) <= NT), "one task");
  extern __shared__ double2 sm[];
  double2* A = sm;
  double2* B = sm + LC * P;
  const int tid = threadIdx.x;
  const bool along_x = a.axis == kAxisX || a.axis == kHilbert;
  const i64 n2 = (i64)N * N;
  // line `l` of the CTA, element j: base + l ls + j js, its partner line io further
  const i64 js = a.axis == kAxisY ? N : a.axis == kAxisZ ? n2 : 1;
  const i64 ls = along_x ? 2 * N : 2, io = along_x ? N : 1;
  const i64 base = (i64)blockIdx.x * LC * ls + (a.axis == kAxisZ ? (i64)N * blockIdx.y : n2 * blockIdx.y);
  if (a.axis == kAxisZ && *a.bad) {
    const double nan = __hiloint2double(0x7ff80000, 0);
    for (int t = tid; t < 2 * LC * N; t += NT) {
      const i64 c = base + t % (2 * LC) + t / (2 * LC) * n2;
      for (int ax = 0; ax < 3 && a.all; ++ax) a.all[ax * n2 * N + c] = nan;
      if (a.delta) a.delta[c] = nan;
    }
    return;
  }
  const double2* tw = reinterpret_cast<const double2*>(a.tab);
  const double* kd = a.tab + 2 * N;
  const double* ks = a.tab + 3 * N;
  // (line, j) of task t: neighbouring threads along the line for x, across lines for y and z
  auto split = [&](int t, int per, int& l, int& j) {
    if (along_x) { j = t % per; l = t / per; }
    else { l = t % LC; j = t / LC; }
  };
  // stage with radix R after stages of total size Ns, on a buffer, in place
  auto in_place = [&](double2* buf, auto radix, int Ns) {
    constexpr int R = decltype(radix)::value;
    int l = 0, j = 0;
    double2 v[R];
    const bool on = tid < LC * (N / R);
    if (on) {
      split(tid, N / R, l, j);
      const int k = j % Ns, tq = N / (Ns * R);
#pragma unroll
      for (int r = 0; r < R; ++r) {
        v[r] = buf[l * P + j + r * (N / R)];
        if (r) {
          const double2 w = __ldg(tw + k * r * tq);
          v[r] = cmul(v[r], w.x, w.y);
        }
      }
      dft<R>(v);
    }
    __syncthreads();
    if (on) {
      const int o = (j / Ns) * Ns * R + j % Ns;
#pragma unroll
      for (int r = 0; r < R; ++r) buf[l * P + o + r * Ns] = v[r];
    }
    __syncthreads();
  };
  // forward: two real lines as one complex line
  for (int t = tid; t < LC * (N / F::R0); t += NT) {
    constexpr int R = F::R0;
    int l, j;
    split(t, N / R, l, j);
    double2 v[R];
    const double* p = a.src + base + l * ls;
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const i64 o = (j + r * (N / R)) * js;
      v[r] = make_double2(p[o], p[o + io]);
    }
    dft<R>(v);
#pragma unroll
    for (int r = 0; r < R; ++r) A[l * P + j * R + r] = v[r];
  }
  __syncthreads();
  if constexpr (F::S >= 2) in_place(A, std::integral_constant<int, F::R1>(), F::R0);
  if constexpr (F::S >= 3) in_place(A, std::integral_constant<int, F::R2>(), F::R0 * F::R1);
  // a line's sum is its k = 0 value
  if (a.axis == kAxisX && tid < LC && max(bexp(A[tid * P].x), bexp(A[tid * P].y)) == 2047) *a.bad = 1;

  // inverse of m(l, k) (a multiplied spectrum with real and imaginary parts
  // exchanged, which turns the forward transform into the inverse), emitted
  // with the parts exchanged back
  auto inverse = [&](auto&& m, auto&& emit) {
    for (int t = tid; t < LC * (N / F::R0); t += NT) {
      constexpr int R = F::R0;
      int l, j;
      split(t, N / R, l, j);
      double2 v[R];
#pragma unroll
      for (int r = 0; r < R; ++r) v[r] = m(l, j + r * (N / R));
      dft<R>(v);
#pragma unroll
      for (int r = 0; r < R; ++r) {
        if (F::S == 1) emit(l, j + r, v[r]);
        else B[l * P + j * R + r] = v[r];
      }
    }
    if constexpr (F::S >= 2) {
      __syncthreads();
      if constexpr (F::S >= 3) in_place(B, std::integral_constant<int, F::R1>(), F::R0);
      constexpr int R = RL, Ns = N / RL;
      for (int t = tid; t < LC * (N / R); t += NT) {
        int l, j;
        split(t, N / R, l, j);
        double2 v[R];
#pragma unroll
        for (int r = 0; r < R; ++r) {
          v[r] = B[l * P + j + r * Ns];
          if (r) {
            const double2 w = __ldg(tw + j * r);
            v[r] = cmul(v[r], w.x, w.y);
          }
        }
        dft<R>(v);
#pragma unroll
        for (int r = 0; r < R; ++r) emit(l, j + r * Ns, v[r]);
      }
      __syncthreads();
    }
  };
  const double pi_n = 3.14159265358979323846 / N;
  if (a.grad) {
    double* g = a.grad + base;
    auto emit = [&](int l, int k, double2 v) {
      double* p = g + l * ls + k * js;
      p[0] = v.y;
      p[io] = v.x;
    };
    if (a.axis == kHilbert) {
      const double q = pi_n / N;
      inverse(
          [&](int l, int k) {
            const double2 c = A[l * P + (k == 0 ? N / 2 : k == N / 2 ? 0 : k)];
            if (2 * k == N || k == 0) return make_double2(c.y * -q, c.x * -q);
            return 2 * k < N ? make_double2(c.x * q, c.y * -q) : make_double2(c.x * -q, c.y * q);
          },
          emit);
    } else {
      const double* w = a.w ? a.w + (i64)N * blockIdx.y + (i64)blockIdx.x * LC * 2 : nullptr;
      inverse(
          [&](int l, int k) {
            const double2 c = A[l * P + k];
            const double f = kd[k];
            if (along_x && k == 0) {
              const double2 h = A[l * P + N / 2];
              return make_double2(h.y * -pi_n, h.x * -pi_n);
            }
            if (!along_x && 2 * k == N) return make_double2(w[2 * l + 1], w[2 * l]);
            return make_double2(c.x * f, c.y * -f);
          },
          emit);
    }
  }
  if (a.delta) {
    double* g = a.delta + base;
    const bool add = !along_x;
    inverse(
        [&](int l, int k) {
          const double2 c = A[l * P + k];
          const double f = ks[k];
          return make_double2(c.y * f, c.x * f);
        },
        [&](int l, int k, double2 v) {
          double* p = g + l * ls + k * js;
          p[0] = add ? p[0] + v.y : v.y;
          p[io] = add ? p[io] + v.x : v.x;
        });
  }
}

template <int N>
void lines_run(const double* src, double* grad, double* delta, const double* tab, double* T, unsigned* bad,
               cudaStream_t s) {
  typedef Fft<N> F;
  constexpr int smem = 2 * F::LC * (N + 1) * (int)sizeof(double2);
  static std::atomic<unsigned long long> done{0};
  smem_attr_once(k_lines<N>, smem, done);
  const i64 n2 = (i64)N * N, n3 = n2 * N;
  const dim3 grid(N / 2 / F::LC, N);
  if (grad) {
    k_altsum<<<dim3((unsigned)((n2 + 127) / 128), 2), 128, 0, s>>>(src, N, T, bad);
    // both T fields, in place: a CTA has read its lines before it writes them
    k_lines<N><<<dim3(N / F::LC, 1), F::NT, smem, s>>>(LineArgs{T, T, nullptr, nullptr, tab, kHilbert, nullptr, nullptr});
    count_launch(2);
  } else {
    cudaMemsetAsync(bad, 0, sizeof(unsigned), s);
  }
  for (int ax = 0; ax < 3; ++ax) {
    const LineArgs a{src, grad ? grad + ax * n3 : nullptr, delta, ax == 0 ? nullptr : T + (ax - 1) * n2, tab, ax, bad,
                     grad};
    k_lines<N><<<grid, F::NT, smem, s>>>(a);
    count_launch();
  }
}

}  // namespace

void launch_fft_tables(double* tab, int n, cudaStream_t s) {
  k_fft_tables<<<(n + 127) / 128, 128, 0, s>>>(tab, n);
  count_launch();
}

void launch_spectral_lines(const double* src, int n, double* grad, double* delta, const double* tab, double* T,
                           unsigned* bad, cudaStream_t s) {
  switch (n) {
    case 8: lines_run<8>(src, grad, delta, tab, T, bad, s); break;
    case 16: lines_run<16>(src, grad, delta, tab, T, bad, s); break;
    case 32: lines_run<32>(src, grad, delta, tab, T, bad, s); break;
    case 64: lines_run<64>(src, grad, delta, tab, T, bad, s); break;
    case 128: lines_run<128>(src, grad, delta, tab, T, bad, s); break;
    case 256: lines_run<256>(src, grad, delta, tab, T, bad, s); break;
    case 512: lines_run<512>(src, grad, delta, tab, T, bad, s); break;
    default: lines_run<1024>(src, grad, delta, tab, T, bad, s); break;
  }
}

}  // namespace mmh

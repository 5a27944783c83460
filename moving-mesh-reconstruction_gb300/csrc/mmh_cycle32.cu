// The mixed form's preconditioner cycle on the levels of 32^3 and below, and
// its whole inner conjugate-gradient solve on grids of 16^3 and 32^3, each in
// one launch (FP32, contraction allowed; not bit-matched).
//
// These levels hold 1 MB of fields and 32 thousand cells: what they cost is
// not work but launches and barriers (one launch per colour and transfer, 60
// to 100 a cycle).  Here a cluster of 16 CTAs keeps every level in shared
// memory.  Planes are dealt out along z: at 32^3 a CTA owns two planes, at
// 16^3 one, and the 8^3 and 4^3 levels run on the first CTA.  The four
// in-plane colours of a plane only need a CTA barrier; a plane's neighbours
// change once per half sweep, when each updated cell is also stored into the
// neighbour CTA's copy of the plane (distributed shared memory) and a cluster
// barrier (370 cycles) follows.  Every operation and every sum has the order
// of the per-level launches, so the bits are theirs: the relaxing step rounds
// its FP32 fluxes from def, and a def that differs in its last bits moves
// single cells of the density by 1e-7.
//
// What bounds it now is shared-memory latency per colour phase and, on the
// 4^3 level, the FP64 pipe (2048 cycles for the 4096 products; summed one by one
// per row they were a chain of 4096).  Measured: a 32^3 inner solve of
// five iterations 194 us (250 us an iteration as launches).
#include <cooperative_groups.h>

#include "mmh_kernels.cuh"
#include "mmh_launch.cuh"

namespace cg = cooperative_groups;

namespace mmh {
namespace {

constexpr int kCta = 16, kThreads = 256;

// word offsets of one level's fields in shared memory: fields read at the
// neighbour planes have a plane below and above the own ones
template <int N>
struct Slab {
  static constexpr int PP = N / kCta, PL = N * N;
  static constexpr int PHI = 0, F3 = (PP + 2) * PL, F5 = 2 * (PP + 2) * PL, F6 = 3 * (PP + 2) * PL,
                       R = 4 * (PP + 2) * PL, F1 = 5 * (PP + 2) * PL, F2 = F1 + PP * PL, F4 = F2 + PP * PL,
                       RHS = F4 + PP * PL, WORDS = RHS + PP * PL;
};
// the 8^3 level, whole: phi, r, rhs, f1..f6
struct Cube8 {
  static constexpr int PHI = 0, R = 512, RHS = 1024, F = 1536, WORDS = F + 6 * 512;
};
// conjugate-gradient vectors of the entry level: p with its neighbour planes, x, q
template <int N>
struct Vecs {
  static constexpr int P = 0, X = (Slab<N>::PP + 2) * Slab<N>::PL, Q = X + Slab<N>::PP * Slab<N>::PL,
                       WORDS = Q + Slab<N>::PP * Slab<N>::PL;
};
struct CycleArgs {
  const float* coef[3];  // 32^3, 16^3, 8^3
  const double* M;
  float dx2;
  int nu1, nu2;
  int special[3];  // k_restrict_resid's special plane on the 32^3, 16^3, 8^3 levels
};
struct Shared {
  double M[64 * 64];      // inverse of the 4^3 operator, transposed (first CTA)
  double b4[64], wsum[2];
  double part[4][64];     // quarters of the rows' sums
  double slot[3][128];     // block sums of the dot products p.q, z.q, r.z
  double smax[kCta];
  float warp[64];
  float z4[64];
  float alpha, beta;
  int go;
};

// barrier of the first two warps
__device__ __forceinline__ void bar_pair() { asm volatile("bar.sync 1, 64;" ::: "memory"); }

// word of cell (x, y) in a plane: even-x half, then odd-x half, so the cells
// of a colour are consecutive words
template <int N>
__device__ __forceinline__ int at(int x, int y) {
  return y * N + (x & 1) * (N / 2) + (x >> 1);
}

// the planes one update reads
struct Planes {
  const float *P, *Pm, *Pp, *f1, *f2, *f4, *f3, *f3m, *f3p, *f5, *f5m, *f5p, *f6, *f6m, *f6p;
};
template <int N>
__device__ __forceinline__ void terms(const Planes& s, int x, int y, float& tdiag, float& t1, float& t2) {
  const int xp = (x + 1) & (N - 1), xm = (x - 1) & (N - 1), yp = (y + 1) & (N - 1), ym = (y - 1) & (N - 1);
  const int c = at<N>(x, y), ip = at<N>(xp, y), im = at<N>(xm, y), jp = at<N>(x, yp), jm = at<N>(x, ym);
  Stencil<float> st;
  st.c = 0.f; st.ip = s.P[ip]; st.im = s.P[im]; st.jp = s.P[jp]; st.jm = s.P[jm]; st.kp = s.Pp[c]; st.km = s.Pm[c];
  st.ppk = s.P[at<N>(xp, yp)]; st.mpk = s.P[at<N>(xm, yp)]; st.pmk = s.P[at<N>(xp, ym)]; st.mmk = s.P[at<N>(xm, ym)];
  st.jpkp = s.Pp[jp]; st.jmkp = s.Pp[jm]; st.jpkm = s.Pm[jp]; st.jmkm = s.Pm[jm];
  st.ipkp = s.Pp[ip]; st.imkp = s.Pp[im]; st.ipkm = s.Pm[ip]; st.imkm = s.Pm[im];
  st.f1c = s.f1[c]; st.f1ip = s.f1[ip]; st.f1im = s.f1[im];
  st.f4c = s.f4[c]; st.f4jp = s.f4[jp]; st.f4jm = s.f4[jm];
  st.f6c = s.f6[c]; st.f6kp = s.f6p[c]; st.f6km = s.f6m[c];
  st.f2jp = s.f2[jp]; st.f2jm = s.f2[jm]; st.f2ip = s.f2[ip]; st.f2im = s.f2[im];
  st.f5kp = s.f5p[c]; st.f5km = s.f5m[c]; st.f5jp = s.f5[jp]; st.f5jm = s.f5[jm];
  st.f3kp = s.f3p[c]; st.f3km = s.f3m[c]; st.f3ip = s.f3[ip]; st.f3im = s.f3[im];
  op_eval(st, tdiag, t1, t2);
}
template <int N>
__device__ __forceinline__ Planes slab_planes(const float* w, int q, const float* phi) {
  typedef Slab<N> S;
  const int o = (q + 1) * S::PL;
  Planes s;
  s.P = phi + o; s.Pm = s.P - S::PL; s.Pp = s.P + S::PL;
  s.f3 = w + S::F3 + o; s.f3m = s.f3 - S::PL; s.f3p = s.f3 + S::PL;
  s.f5 = w + S::F5 + o; s.f5m = s.f5 - S::PL; s.f5p = s.f5 + S::PL;
  s.f6 = w + S::F6 + o; s.f6m = s.f6 - S::PL; s.f6p = s.f6 + S::PL;
  s.f1 = w + S::F1 + q * S::PL; s.f2 = w + S::F2 + q * S::PL; s.f4 = w + S::F4 + q * S::PL;
  return s;
}
__device__ __forceinline__ Planes cube_planes(const float* w, int k) {
  typedef Cube8 C;
  const int o = k * 64, om = ((k + 7) & 7) * 64, op = ((k + 1) & 7) * 64;
  const float* f = w + C::F;
  Planes s;
  s.P = w + C::PHI + o; s.Pm = w + C::PHI + om; s.Pp = w + C::PHI + op;
  s.f1 = f + o; s.f2 = f + 512 + o; s.f4 = f + 3 * 512 + o;
  s.f3 = f + 1024 + o; s.f3m = f + 1024 + om; s.f3p = f + 1024 + op;
  s.f5 = f + 2048 + o; s.f5m = f + 2048 + om; s.f5p = f + 2048 + op;
  s.f6 = f + 2560 + o; s.f6m = f + 2560 + om; s.f6p = f + 2560 + op;
  return s;
}

// one CTA of the cluster: its own words and its neighbours' along z
struct Me {
  cg::cluster_group cl;
  float *w, *up, *dn;  // the level fields here, one CTA up, one down (z periodic)
  int rank;
};

// nsweeps 8-colour sweeps of a slab level; ends with the neighbours' copies
// complete (cluster barrier after every half sweep)
template <int N>
__device__ void sweeps(const Me& me, int base, float dx2, int nsweeps) {
  typedef Slab<N> S;
  float* w = me.w + base;
  for (int h = 0; h < 2 * nsweeps; ++h) {
    const int kpar = h & 1;
    // N = 32: own plane kpar; N = 16: the own plane where its parity matches
    const int q = S::PP == 2 ? kpar : 0;
    if (S::PP == 2 || (me.rank & 1) == kpar) {
      const Planes s = slab_planes<N>(w, q, w + S::PHI);
      float* P = w + S::PHI + (q + 1) * S::PL;
      // the neighbours' copies: below the lowest own plane, above the highest
      float* to_dn = q == 0 ? me.dn + base + S::PHI + (S::PP + 1) * S::PL : nullptr;
      float* to_up = q == S::PP - 1 ? me.up + base + S::PHI : nullptr;
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        for (int e = threadIdx.x; e < S::PL / 4; e += kThreads) {
          const int x = 2 * (e % (N / 2)) + (c >> 1), y = 2 * (e / (N / 2)) + (c & 1);
          const int o = at<N>(x, y);
          float td, t1, t2;
          terms<N>(s, x, y, td, t1, t2);
          const float v = gs_div(w[S::RHS + q * S::PL + o] * dx2 - t1 - t2, td);
          P[o] = v;
          if (to_dn) to_dn[o] = v;
          if (to_up) to_up[o] = v;
        }
        if (c < 3) __syncthreads();
      }
    }
    me.cl.sync();
  }
}

// r = rhs - L[phi] of the own planes, stored into the neighbours' copies too
template <int N>
__device__ void residual(const Me& me, int base, float di2) {
  typedef Slab<N> S;
  float* w = me.w + base;
#pragma unroll
  for (int q = 0; q < S::PP; ++q) {
    const Planes s = slab_planes<N>(w, q, w + S::PHI);
    for (int e = threadIdx.x; e < S::PL; e += kThreads) {
      const int o = at<N>(e % N, e / N);
      float td, t1, t2;
      terms<N>(s, e % N, e / N, td, t1, t2);
      const float v = w[S::RHS + q * S::PL + o] - (t1 + t2 + td * s.P[o]) * di2;
      w[S::R + (q + 1) * S::PL + o] = v;
      if (q == 0) me.dn[base + S::R + (S::PP + 1) * S::PL + o] = v;
      if (q == S::PP - 1) me.up[base + S::R + o] = v;
    }
  }
  me.cl.sync();
}

// full weighting of a plane triple at coarse cell (X, Y) in the order of
// k_restrict_resid (own_first: the coarse plane `special` there)
template <int N>
__device__ __forceinline__ float weight(const float* lo, const float* mid, const float* hi, int X, int Y,
                                        bool own_first) {
  const int x = 2 * X, y = 2 * Y, xp = x + 1, xm = (x - 1) & (N - 1), yp = y + 1, ym = (y - 1) & (N - 1);
  const int c = at<N>(x, y), e0 = at<N>(xp, y), e1 = at<N>(xm, y), e2 = at<N>(x, yp), e3 = at<N>(x, ym);
  const int d0 = at<N>(xp, yp), d1 = at<N>(xp, ym), d2 = at<N>(xm, yp), d3 = at<N>(xm, ym);
  const float la = lo[c] * 0.0625f;
  const float lb = (lo[e0] + lo[e1] + lo[e2] + lo[e3]) * 0.03125f;
  const float lc = (lo[d0] + lo[d1] + lo[d2] + lo[d3]) * 0.015625f;
  const float ma = mid[c] * 0.125f;
  const float mb = (mid[e0] + mid[e1] + mid[e2] + mid[e3] + hi[c]) * 0.0625f;
  const float mc = (mid[d0] + mid[d1] + mid[d2] + mid[d3] + hi[e0] + hi[e1] + hi[e2] + hi[e3]) * 0.03125f;
  const float md = (hi[d0] + hi[d1] + hi[d2] + hi[d3]) * 0.015625f;
  float acc = 0.f;
  if (own_first) {
    acc = acc + ma + mb + mc + md;
    acc = acc + la + lb + lc;
  } else {
    acc = acc + la + lb + lc;
    acc = acc + ma + mb + mc + md;
  }
  return acc;
}

// trilinear value of the coarse planes A (below or at the fine plane) and B
// (above or the same) at fine cell (x, y); N the coarse size
template <int N>
__device__ __forceinline__ float trilinear(const float* A, const float* B, int x, int y) {
  const int xl = x >> 1, xh = ((x + 1) >> 1) & (N - 1), yl = y >> 1, yh = ((y + 1) >> 1) & (N - 1);
  const int ll = at<N>(xl, yl), lh = at<N>(xl, yh), hh = at<N>(xh, yh), hl = at<N>(xh, yl);
  return (A[ll] + B[ll] + A[lh] + B[lh] + A[hh] + B[hh] + A[hl] + B[hl]) * 0.125f;
}

// The 8^3 and 4^3 levels on the first CTA: rhs in the cube; nu1 sweeps from
// zero, residual, exact 4^3 solve, correction, nu2 sweeps.
__device__ void cube_sweeps(float* w, float dx2, int nsweeps) {
  typedef Cube8 C;
  for (int h = 0; h < 8 * nsweeps; ++h) {
    const int c = h & 7;
    if (threadIdx.x < 64) {
      const int e = threadIdx.x, k = 2 * (e >> 4) + (c >> 2);
      const int x = 2 * (e & 3) + ((c >> 1) & 1), y = 2 * ((e >> 2) & 3) + (c & 1);
      const Planes s = cube_planes(w, k);
      float td, t1, t2;
      terms<8>(s, x, y, td, t1, t2);
      w[C::PHI + k * 64 + at<8>(x, y)] = gs_div(w[C::RHS + k * 64 + at<8>(x, y)] * dx2 - t1 - t2, td);
    }
    __syncthreads();
  }
}
__device__ void cube_cycle(float* w, Shared* sh, float dx2, int nu1, int nu2, int special) {
  typedef Cube8 C;
  const int tid = threadIdx.x;
  for (int e = tid; e < 512; e += kThreads) w[C::PHI + e] = 0.f;
  __syncthreads();
  cube_sweeps(w, dx2, nu1);
  for (int e = tid; e < 512; e += kThreads) {
    const int k = e >> 6, x = e & 7, y = (e >> 3) & 7, o = k * 64 + at<8>(x, y);
    const Planes s = cube_planes(w, k);
    float td, t1, t2;
    terms<8>(s, x, y, td, t1, t2);
    w[C::R + o] = w[C::RHS + o] - (t1 + t2 + td * w[C::PHI + o]) * (1.f / dx2);
  }
  __syncthreads();
  // z = M (r - mean r) on the 4^3 cells, FP64, with the operations of
  // k_coarse_apply: four threads share a row, 16 fused multiply-adds each.
  if (tid < 64) {
    const int X = tid & 3, Y = (tid >> 2) & 3, K = tid >> 4;
    const float* r = w + C::R;
    const double v =
        (double)weight<8>(r + ((2 * K + 7) & 7) * 64, r + 2 * K * 64, r + (2 * K + 1) * 64, X, Y, K == special);
    double sv = v;
    for (int d = 16; d > 0; d >>= 1) sv = __dadd_rn(sv, __shfl_down_sync(0xffffffffu, sv, d));
    if ((tid & 31) == 0) sh->wsum[tid >> 5] = sv;
    bar_pair();
    sh->b4[tid] = __dsub_rn(v, __dadd_rn(sh->wsum[0], sh->wsum[1]) / 64);
  }
  __syncthreads();
  {
    const int row = tid & 63, q = tid >> 6;
    double acc = 0.0;
#pragma unroll
    for (int j = 16 * q; j < 16 * q + 16; ++j) acc = __fma_rn(sh->M[j * 64 + row], sh->b4[j], acc);
    sh->part[q][row] = acc;
  }
  __syncthreads();
  if (tid < 64)
    sh->z4[(tid >> 4) * 16 + at<4>(tid & 3, (tid >> 2) & 3)] =
        (float)__dadd_rn(__dadd_rn(sh->part[0][tid], sh->part[1][tid]), __dadd_rn(sh->part[2][tid], sh->part[3][tid]));
  __syncthreads();
  for (int e = tid; e < 512; e += kThreads) {
    const int k = e >> 6, x = e & 7, y = (e >> 3) & 7;
    w[C::PHI + k * 64 + at<8>(x, y)] +=
        trilinear<4>(sh->z4 + (k >> 1) * 16, sh->z4 + (((k + 1) >> 1) & 3) * 16, x, y);
  }
  __syncthreads();
  cube_sweeps(w, dx2, nu2);
}

// phi = 0 on a slab level, own planes and copies
template <int N>
__device__ void zero_phi(float* w) {
  for (int e = threadIdx.x; e < (Slab<N>::PP + 2) * Slab<N>::PL; e += kThreads) w[Slab<N>::PHI + e] = 0.f;
}

// One V(nu1, nu2) cycle from level N (32 or 16) on its rhs in shared memory;
// the result and its neighbour copies in phi.  Words: [level N | (16^3) | 8^3].
template <int N>
__device__ void cycle(const Me& me, int base, int cube, Shared* sh, float dx2, const CycleArgs& a) {
  typedef Slab<N> S;
  float* w = me.w + base;
  zero_phi<N>(w);
  me.cl.sync();  // no neighbour stores into phi before it is zero
  sweeps<N>(me, base, dx2, a.nu1);
  residual<N>(me, base, 1.f / dx2);
  if constexpr (N == 32) {
    // coarse plane `rank` from the fine planes 2 rank - 1, 2 rank, 2 rank + 1
    const int b16 = base + S::WORDS;
    float* w16 = me.w + b16;
    const float* r = w + S::R;
    for (int e = threadIdx.x; e < 256; e += kThreads)
      w16[Slab<16>::RHS + at<16>(e & 15, e >> 4)] =
          weight<32>(r, r + S::PL, r + 2 * S::PL, e & 15, e >> 4, me.rank == a.special[0]);
    cycle<16>(me, b16, cube, sh, 4.f * dx2, a);
    // the own planes and the neighbours' copies (their coarse planes are
    // here too): fine plane 2 rank + d - 1 lies at coarse plane rank - 1 + ((d + 1) >> 1)
    const float* u = w16 + Slab<16>::PHI;
    for (int e = threadIdx.x; e < 4 * S::PL; e += kThreads) {
      const int d = e / S::PL, x = e % 32, y = (e / 32) % 32;
      const float* A = u + ((d + 1) >> 1) * 256;
      const float* B = u + ((d + 2) >> 1) * 256;
      w[S::PHI + d * S::PL + at<32>(x, y)] += trilinear<16>(A, B, x, y);
    }
  } else {
    float* c0 = me.cl.map_shared_rank(me.w, 0) + cube;
    if (!(me.rank & 1) && threadIdx.x < 64) {
      const float* r = w + S::R;
      const int X = threadIdx.x & 7, Y = threadIdx.x >> 3;
      c0[Cube8::RHS + (me.rank >> 1) * 64 + at<8>(X, Y)] =
          weight<16>(r, r + S::PL, r + 2 * S::PL, X, Y, (me.rank >> 1) == a.special[1]);
    }
    me.cl.sync();
    if (me.rank == 0) cube_cycle(me.w + cube, sh, 4.f * dx2, a.nu1, a.nu2, a.special[2]);
    me.cl.sync();
    // coarse planes of the fine planes rank - 1, rank, rank + 1, into the own cube
    float* u = me.w + cube + Cube8::PHI;
    if (me.rank != 0)
      for (int e = threadIdx.x; e < 512; e += kThreads) u[e] = c0[Cube8::PHI + e];
    __syncthreads();
    for (int e = threadIdx.x; e < 3 * S::PL; e += kThreads) {
      const int d = e / S::PL, x = e % 16, y = (e / 16) % 16, k = (me.rank + d + 15) & 15;
      w[S::PHI + d * S::PL + at<16>(x, y)] += trilinear<8>(u + (k >> 1) * 64, u + (((k + 1) >> 1) & 7) * 64, x, y);
    }
  }
  me.cl.sync();  // the neighbours' copies are corrected before the sweeps store into them
  sweeps<N>(me, base, dx2, a.nu2);
}

// Asynchronous copies of single words into shared memory.  A cycle on its own
// (below a 64^3 level) reads 100 words per thread before it starts; through
// registers they came a few at a time and took as long as half the cycle, so
// all are in flight at once.
__device__ __forceinline__ void cp_word(float* dst, const float* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"((unsigned)__cvta_generic_to_shared(dst)),
               "l"(__cvta_generic_to_global(src))
               : "memory");
}
__device__ __forceinline__ void cp_word(double* dst, const double* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"((unsigned)__cvta_generic_to_shared(dst)),
               "l"(__cvta_generic_to_global(src))
               : "memory");
}
__device__ __forceinline__ void cp_wait() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// fields of a slab level from global memory
template <int N>
__device__ void load_coef(float* w, int rank, const float* coef) {
  typedef Slab<N> S;
  constexpr int n3 = N * N * N;
  for (int e = threadIdx.x; e < (S::PP + 2) * S::PL; e += kThreads) {
    const int d = e / S::PL, x = e % N, y = (e / N) % N, k = (rank * S::PP + d - 1) & (N - 1);
    const int g = k * S::PL + y * N + x, o = d * S::PL + at<N>(x, y);
    cp_word(w + S::F3 + o, coef + 2 * n3 + g);
    cp_word(w + S::F5 + o, coef + 4 * n3 + g);
    cp_word(w + S::F6 + o, coef + 5 * n3 + g);
    if (d >= 1 && d <= S::PP) {
      cp_word(w + S::F1 + o - S::PL, coef + g);
      cp_word(w + S::F2 + o - S::PL, coef + n3 + g);
      cp_word(w + S::F4 + o - S::PL, coef + 3 * n3 + g);
    }
  }
}
template <int N>
__device__ void load_rhs(float* w, int rank, const float* rhs) {
  typedef Slab<N> S;
  for (int e = threadIdx.x; e < S::PP * S::PL; e += kThreads) {
    const int q = e / S::PL, x = e % N, y = (e / N) % N;
    cp_word(w + S::RHS + q * S::PL + at<N>(x, y), rhs + (rank * S::PP + q) * S::PL + y * N + x);
  }
}


template <int N>
struct Layout {
  static constexpr int CUBE = Slab<N>::WORDS + (N == 32 ? Slab<16>::WORDS : 0);
  static constexpr int VECS = CUBE + Cube8::WORDS;
  static constexpr int BYTES_CYCLE = (int)sizeof(Shared) + 4 * VECS;
  static constexpr int BYTES_SOLVE = BYTES_CYCLE + 4 * Vecs<N>::WORDS;
  static_assert(BYTES_SOLVE <= 227 * 1024, "shared memory of one CTA");
};

template <int N>
__device__ __forceinline__ Me setup(Shared*& sh, const CycleArgs& a, unsigned char* raw) {
  sh = reinterpret_cast<Shared*>(raw);
  Me me{cg::this_cluster(), reinterpret_cast<float*>(raw + sizeof(Shared)), nullptr, nullptr, 0};
  me.rank = (int)me.cl.block_rank();
  me.up = me.cl.map_shared_rank(me.w, (me.rank + 1) % kCta);
  me.dn = me.cl.map_shared_rank(me.w, (me.rank + kCta - 1) % kCta);
  load_coef<N>(me.w, me.rank, a.coef[N == 32 ? 0 : 1]);
  if constexpr (N == 32) load_coef<16>(me.w + Slab<32>::WORDS, me.rank, a.coef[1]);
  if (me.rank == 0) {
    float* f = me.w + Layout<N>::CUBE + Cube8::F;
    for (int e = threadIdx.x; e < 6 * 512; e += kThreads) {
      const int x = e & 7, y = (e >> 3) & 7;
      cp_word(f + (e & ~63) + at<8>(x, y), a.coef[2] + e);
    }
    for (int e = threadIdx.x; e < 64 * 64; e += kThreads) cp_word(sh->M + (e & 63) * 64 + (e >> 6), a.M + e);
  }
  return me;
}

// one cycle: rhs in, u out (entry level N)
template <int N>
__global__ void __launch_bounds__(kThreads) k_cycle32(CycleArgs a, const float* __restrict__ rhs,
                                                      float* __restrict__ u) {
  extern __shared__ __align__(16) unsigned char raw[];
  typedef Slab<N> S;
  Shared* sh;
  Me me = setup<N>(sh, a, raw);
  load_rhs<N>(me.w, me.rank, rhs);
  cp_wait();  // visible to the CTA at the cycle's first barrier
  cycle<N>(me, 0, Layout<N>::CUBE, sh, a.dx2, a);
  for (int e = threadIdx.x; e < S::PP * S::PL; e += kThreads) {
    const int q = e / S::PL, x = e % N, y = (e / N) % N;
    u[(me.rank * S::PP + q) * S::PL + y * N + x] = me.w[S::PHI + (q + 1) * S::PL + at<N>(x, y)];
  }
}

// Dot product over the cluster with the sums of k_pcg_dot on such a grid (one
// product per thread there, its halving over empty blocks as well): products
// rounded to FP32, blocks of 256 consecutive cells (a warp's 32 by shuffles,
// the 8 warps in order), the block sums in FP64 by halving.  dot_post leaves
// every CTA the block sums in slot[which]; after a cluster barrier dot_sum
// (one warp) adds them.  Two uses of the same slots have a cluster barrier
// between the reads of one and the writes of the next.  The total is not
// rounded to a fixed point as dot_rounded does: with E of the maxima that is 2^(E
// - 96), which changes no total above 2^(E - 44).
template <int N>
__device__ __forceinline__ void dot_post(const Me& me, Shared* sh, int which, const float* a, const float* b) {
  typedef Slab<N> S;
  constexpr int NB = S::PP * S::PL / 256;  // blocks of this CTA: 8 or 1
  __syncthreads();
#pragma unroll
  for (int j = 0; j < NB; ++j) {
    const int g = j * 256 + threadIdx.x, x = g % N, y = (g / N) % N, o = g / S::PL * S::PL + at<N>(x, y);
    float v = __fmul_rn(a[o], b[o]);
    for (int d = 16; d > 0; d >>= 1) v = __fadd_rn(v, __shfl_down_sync(0xffffffffu, v, d));
    if ((threadIdx.x & 31) == 0) sh->warp[j * 8 + (threadIdx.x >> 5)] = v;
  }
  __syncthreads();
  if (threadIdx.x < kCta * NB) {
    const int j = threadIdx.x % NB, rank = threadIdx.x / NB;
    float t = 0.f;
#pragma unroll
    for (int q = 0; q < 8; ++q) t = __fadd_rn(t, sh->warp[j * 8 + q]);
    me.cl.map_shared_rank(sh, rank)->slot[which][me.rank * NB + j] = (double)t;
  }
}
template <int N>
__device__ __forceinline__ double dot_sum(const Shared* sh, int which) {
  const double* v = sh->slot[which];
  const int lane = threadIdx.x & 31;
  double t;
  if (N == 32)
    t = __dadd_rn(__dadd_rn(v[lane], v[lane + 64]), __dadd_rn(v[lane + 32], v[lane + 96]));
  else
    t = lane < 16 ? v[lane] : 0.0;
  for (int d = 16; d > 0; d >>= 1) t = __dadd_rn(t, __shfl_down_sync(0xffffffffu, t, d));
  t = __shfl_sync(0xffffffffu, t, 0);
  return fabs(t) < INFINITY ? t : 0.0;  // as dot_rounded
}

// The inner solve of the mixed form (pcg_core32's): x = 0,
// r = b in rhs; flexible conjugate gradients preconditioned by one cycle until
// max|r| <= tol * bn or maxit iterations.  x out; out[0] = iterations, out[1]
// = max|r| (as double bits), the residual left in rhs.
template <int N>
__global__ void __launch_bounds__(kThreads) k_solve32(CycleArgs a, float* __restrict__ rhs, float* __restrict__ x,
                                                      double bn, double tol, int maxit,
                                                      unsigned long long* __restrict__ out) {
  extern __shared__ __align__(16) unsigned char raw[];
  typedef Slab<N> S;
  typedef Vecs<N> V;
  constexpr int L = Layout<N>::VECS, OWN = S::PP * S::PL;
  Shared* sh;
  Me me = setup<N>(sh, a, raw);
  load_rhs<N>(me.w, me.rank, rhs);
  cp_wait();  // visible to the CTA at the cycle's first barrier
  float* w = me.w;
  float* r = w + S::RHS;
  const float* z = w + S::PHI + S::PL;
  float* p = w + L + V::P;  // plane q at (q + 1) PL
  float* xv = w + L + V::X;
  float* qv = w + L + V::Q;
  const float di2 = 1.f / a.dx2;
  for (int e = threadIdx.x; e < OWN; e += kThreads) xv[e] = 0.f;
  double rz = 0.0, alpha = 0.0, rmax = 0.0;
  int it = 0;
  for (;;) {
    __syncthreads();
    cycle<N>(me, 0, Layout<N>::CUBE, sh, a.dx2, a);
    // r.z, and after the first iteration z.q; then p = z + beta p
    if (it > 0) dot_post<N>(me, sh, 1, z, qv);
    dot_post<N>(me, sh, 2, r, z);
    me.cl.sync();
    if (threadIdx.x < 32) {
      const double rz_new = dot_sum<N>(sh, 2);
      float beta = 0.f;
      if (it > 0) beta = (float)(-(alpha * dot_sum<N>(sh, 1)) / rz);
      rz = rz_new;
      if (threadIdx.x == 0) sh->beta = beta;
    }
    __syncthreads();
    const float beta = sh->beta;
    for (int e = threadIdx.x; e < OWN; e += kThreads) {
      const float v = it > 0 ? z[e] + beta * p[S::PL + e] : z[e];
      p[S::PL + e] = v;
      if (e < S::PL) me.dn[L + V::P + (S::PP + 1) * S::PL + e] = v;
      if (e >= OWN - S::PL) me.up[L + V::P + e - (OWN - S::PL)] = v;
    }
    me.cl.sync();
    // q = L p, p.q
#pragma unroll
    for (int q = 0; q < S::PP; ++q) {
      const Planes s = slab_planes<N>(w, q, p);
      for (int e = threadIdx.x; e < S::PL; e += kThreads) {
        const int o = at<N>(e % N, e / N);
        float td, t1, t2;
        terms<N>(s, e % N, e / N, td, t1, t2);
        const float v = (t1 + t2 + td * s.P[o]) * di2;
        qv[q * S::PL + o] = v;
      }
    }
    dot_post<N>(me, sh, 0, p + S::PL, qv);
    me.cl.sync();
    if (threadIdx.x < 32) {
      alpha = rz / dot_sum<N>(sh, 0);
      if (threadIdx.x == 0) sh->alpha = (float)alpha;
    }
    __syncthreads();
    const float al = sh->alpha;
    float m = 0.f;
    for (int e = threadIdx.x; e < OWN; e += kThreads) {
      xv[e] = xv[e] + al * p[S::PL + e];
      const float v = r[e] - al * qv[e];
      r[e] = v;
      m = __uint_as_float(max(__float_as_uint(m), __float_as_uint(fabsf(v))));
    }
    for (int d = 16; d > 0; d >>= 1)
      m = __uint_as_float(max(__float_as_uint(m), __float_as_uint(__shfl_xor_sync(0xffffffffu, m, d))));
    if ((threadIdx.x & 31) == 0) sh->warp[threadIdx.x >> 5] = m;
    __syncthreads();
    if (threadIdx.x < kCta) {
      unsigned t = 0;
      for (int q = 0; q < kThreads / 32; ++q) t = max(t, __float_as_uint(sh->warp[q]));
      me.cl.map_shared_rank(sh, threadIdx.x)->smax[me.rank] = (double)__uint_as_float(t);
    }
    me.cl.sync();
    if (threadIdx.x < 32) {
      unsigned long long b = (unsigned long long)__double_as_longlong(sh->smax[threadIdx.x & (kCta - 1)]);
      for (int d = kCta / 2; d > 0; d >>= 1) {
        const unsigned long long o = __shfl_xor_sync(0xffffffffu, b, d);
        b = o > b ? o : b;
      }
      rmax = __longlong_as_double((long long)b);
      const double rel = rmax / bn;
      // NaN: stop; the host reports it
      if (threadIdx.x == 0) sh->go = rel > tol && it + 1 < maxit ? 1 : 0;
    }
    ++it;
    __syncthreads();
    if (!sh->go) break;
  }
  for (int e = threadIdx.x; e < OWN; e += kThreads) {
    const int q = e / S::PL, xx = e % N, y = (e / N) % N;
    const int g = (me.rank * S::PP + q) * S::PL + y * N + xx, o = q * S::PL + at<N>(xx, y);
    x[g] = xv[o];
    rhs[g] = r[o];
  }
  if (me.rank == 0 && threadIdx.x == 0) {
    out[0] = (unsigned long long)it;
    out[1] = (unsigned long long)__double_as_longlong(rmax);
  }
  me.cl.sync();  // neighbours' stores into this CTA's shared memory have landed
}

template <class K, class... A>
void cluster_launch(K* kernel, int smem, cudaStream_t s, A... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(kCta);
  cfg.blockDim = dim3(kThreads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = kCta;
  at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  cudaLaunchKernelEx(&cfg, kernel, args...);
}

CycleArgs cycle_args(int n, const float* c0, const float* c1, const float* c2, const double* M, double dx, int nu1,
                     int nu2, const int* special) {
  CycleArgs a;
  a.coef[0] = n == 32 ? c0 : nullptr;
  a.coef[1] = n == 32 ? c1 : c0;
  a.coef[2] = n == 32 ? c2 : c1;
  a.M = M;
  a.dx2 = (float)(dx * dx);
  a.nu1 = nu1;
  a.nu2 = nu2;
  a.special[0] = n == 32 ? special[0] : 0;
  a.special[1] = n == 32 ? special[1] : special[0];
  a.special[2] = n == 32 ? special[2] : special[1];
  return a;
}

}  // namespace

// the inner solve at 32^3 has the most shared memory of the four
bool cycle32_fits(cudaStream_t s) {
  static std::atomic<unsigned long long> d0{0}, d1{0};
  smem_attr_once(k_solve32<32>, Layout<32>::BYTES_SOLVE, d0);
  func_attr_once(k_solve32<32>, cudaFuncAttributeNonPortableClusterSizeAllowed, 1, d1);
  return cluster_fits(k_solve32<32>, kCta, kThreads, Layout<32>::BYTES_SOLVE, s);
}

void launch_cycle32(int n, const float* c0, const float* c1, const float* c2, const double* M, double dx, int nu1,
                    int nu2, const int* special, const float* rhs, float* u, cudaStream_t s) {
  const CycleArgs a = cycle_args(n, c0, c1, c2, M, dx, nu1, nu2, special);
  static std::atomic<unsigned long long> d0{0}, d1{0}, d2{0}, d3{0};
  if (n == 32) {
    smem_attr_once(k_cycle32<32>, Layout<32>::BYTES_CYCLE, d0);
    func_attr_once(k_cycle32<32>, cudaFuncAttributeNonPortableClusterSizeAllowed, 1, d1);
    cluster_launch(k_cycle32<32>, Layout<32>::BYTES_CYCLE, s, a, rhs, u);
  } else {
    smem_attr_once(k_cycle32<16>, Layout<16>::BYTES_CYCLE, d2);
    func_attr_once(k_cycle32<16>, cudaFuncAttributeNonPortableClusterSizeAllowed, 1, d3);
    cluster_launch(k_cycle32<16>, Layout<16>::BYTES_CYCLE, s, a, rhs, u);
  }
  count_launch();
}

void launch_solve32(int n, const float* c0, const float* c1, const float* c2, const double* M, double dx, int nu1,
                    int nu2, const int* special, float* rhs, float* x, double bn, double tol, int maxit, unsigned long long* out,
                    cudaStream_t s) {
  const CycleArgs a = cycle_args(n, c0, c1, c2, M, dx, nu1, nu2, special);
  static std::atomic<unsigned long long> d0{0}, d1{0}, d2{0}, d3{0};
  if (n == 32) {
    smem_attr_once(k_solve32<32>, Layout<32>::BYTES_SOLVE, d0);
    func_attr_once(k_solve32<32>, cudaFuncAttributeNonPortableClusterSizeAllowed, 1, d1);
    cluster_launch(k_solve32<32>, Layout<32>::BYTES_SOLVE, s, a, rhs, x, bn, tol, maxit, out);
  } else {
    smem_attr_once(k_solve32<16>, Layout<16>::BYTES_SOLVE, d2);
    func_attr_once(k_solve32<16>, cudaFuncAttributeNonPortableClusterSizeAllowed, 1, d3);
    cluster_launch(k_solve32<16>, Layout<16>::BYTES_SOLVE, s, a, rhs, x, bn, tol, maxit, out);
  }
  count_launch();
}

}  // namespace mmh

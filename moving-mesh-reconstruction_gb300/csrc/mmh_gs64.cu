// FP64 Gauss-Seidel sweeps (relax / relaxplane, mmh/gauss1.f90:64-499 and
// :866-991), bit for bit the reference's operations.  Compiled with
// --fmad=false; the fused operations below are written out and exact where
// they replace a product by a power of two.
//
// What bounds these kernels is the FP64 pipe: on GB300 one FP64 instruction
// of one warp occupies its SM quarter for 64 cycles (77 with all four
// quarters busy), however many of its lanes are active, and a dependent
// instruction can issue right after it.  A kernel therefore costs its number
// of FP64 warp instructions, lanes filled or not, and one or two warps per
// quarter keep the pipe busy.  So:
//   - a plane is cut into whole rows, not into tiles: there is no halo in x
//     and every warp instruction has 32 (16 at n = 32) useful lanes;
//   - powers of two are folded (scaling is exact and commutes with rounding):
//     with S1 = 2 t1, S2 = 4 t2, D = -2 tdiag formed from unhalved face sums,
//     phi = (rhs dx2 - t1 - t2) / tdiag = -(((rhs 2dx2) - S1) - S2/2) / D;
//   - the small grids split one update over many lanes and warps and compute
//     what does not depend on the running colour ahead of it.
#include <cooperative_groups.h>

#include "mmh_kernels.cuh"
#include "mmh_launch.cuh"

namespace cg = cooperative_groups;

namespace mmh {
namespace {

// ---------------------------------------------------------------------------
// n >= 32: one half sweep (the four in-plane colours of every plane of one
// parity).  A CTA owns TY full rows of one plane.  phi of the plane (rows -3
// .. TY+3) sits in shared memory, each row split into its even-x and odd-x
// half, so the lanes of a colour read consecutive words; everything else is
// read once per update from global memory (L1/L2), which costs a tenth of the
// FP64 time.  Colour q is updated on the rows q-2, q, ... that the later
// colours read (TY/2 + 3 - q of them): the only recomputed cells.  Reads the
// plane's own old values from src, the other parity's planes from nbr, writes
// dst != src.
//
// TY: 32 from 128^3 up (1.09 updates per cell), 16 where 39 rows would not
// fit shared memory (1024^3) or would leave SMs without a CTA (64^3), 8 at
// 32^3.  Per half sweep, against the form it replaces (from 64^3 up a 32 x 8
// tile with 1.75 updates per cell counting idle lanes, at 32^3 four
// one-colour launches): 256^3 1.26 ms (2.25), 128^3 0.187 ms (0.30), 64^3
// 33.5 us (48), 32^3 14.4 us (38).
// ---------------------------------------------------------------------------
constexpr int kRowThreads = 256;

__global__ void __launch_bounds__(kRowThreads, 2) k_gs_rows(const double* __restrict__ src,
                                                            const double* __restrict__ nbr, double* __restrict__ dst,
                                                            const double* __restrict__ rhs,
                                                            const double* __restrict__ coef, int lgn, int ty,
                                                            double dx2x2, int kpar) {
  extern __shared__ double sp[];
  const int n = 1 << lgn, h = n >> 1, lgh = lgn - 1;
  const i64 n2 = (i64)n << lgn, n3 = n2 << lgn;
  const int y0 = blockIdx.x * ty, k = 2 * blockIdx.y + kpar;
  const int kp = wp(k, n), km = wm(k, n);
  const double* own = src + n2 * k;
  for (int e = threadIdx.x; e < (ty + 7) << lgn; e += kRowThreads) {
    const int r = e >> lgn, x = e & (n - 1);
    const int y = (y0 + r - 3) & (n - 1);
    sp[(r << lgn) + (x & 1) * h + (x >> 1)] = own[((i64)y << lgn) + x];
  }
  __syncthreads();
  const double* Kp = nbr + n2 * kp;
  const double* Km = nbr + n2 * km;
  const double* f1 = coef + n2 * k;
  const double* f2 = f1 + n3;
  const double* f4 = f1 + 3 * n3;
  const double* f3 = f1 + 2 * n3;
  const double* f5 = f1 + 4 * n3;
  const double* f6 = f1 + 5 * n3;
  const i64 dkp = n2 * (kp - k), dkm = n2 * (km - k);
#pragma unroll 1
  for (int q = 0; q < 4; ++q) {
    const int io = q >> 1;
    const int cells = (ty / 2 + 3 - q) << lgh;
#pragma unroll 1
    for (int e = threadIdx.x; e < cells; e += kRowThreads) {
      const int m = e & (h - 1), yl = q - 2 + 2 * (e >> lgh);  // row relative to y0
      const int x = 2 * m + io, xp = (x + 1) & (n - 1), xm = (x - 1) & (n - 1);
      const int y = (y0 + yl) & (n - 1), yp = (y + 1) & (n - 1), ym = (y - 1) & (n - 1);
      const i64 r0 = (i64)y << lgn, rp = (i64)yp << lgn, rm = (i64)ym << lgn;
      const i64 c = r0 + x, cxp = r0 + xp, cxm = r0 + xm, cyp = rp + x, cym = rm + x;
      // face sums (twice the face coefficients) and the diagonal
      const double f1c = f1[c], f4c = f4[c], f6c = f6[c];
      const double b11p = f1[cxp] + f1c, b11m = f1[cxm] + f1c;
      const double b22p = f4[cyp] + f4c, b22m = f4[cym] + f4c;
      const double b33p = f6[c + dkp] + f6c, b33m = f6[c + dkm] + f6c;
      const double d = b11p + b11m + b22p + b22m + b33p + b33m;
      // phi of the plane: rows yl+2 .. yl+4 of the tile, x+-1 in the other half
      const double* s0 = sp + ((yl + 3) << lgn);
      const double* sP = s0 + n;
      const double* sM = s0 - n;
      const int oc = io * h + m, op = (xp & 1) * h + (xp >> 1), om = (xm & 1) * h + (xm >> 1);
      const double s1 = b11p * s0[op] + b11m * s0[om] + b22p * sP[oc] + b22m * sM[oc] + b33p * Kp[c] + b33m * Km[c];
      const double ppk = sP[op], mpk = sP[om], pmk = sM[op], mmk = sM[om];
      const double jpkp = Kp[cyp], jmkp = Kp[cym], jpkm = Km[cyp], jmkm = Km[cym];
      const double ipkp = Kp[cxp], imkp = Kp[cxm], ipkm = Km[cxp], imkm = Km[cxm];
      const double s2 = (ppk - mpk) * f2[cyp] - (pmk - mmk) * f2[cym] + (ppk - pmk) * f2[cxp] - (mpk - mmk) * f2[cxm] +
                        (jpkp - jmkp) * f5[c + dkp] - (jpkm - jmkm) * f5[c + dkm] + (jpkp - jpkm) * f5[cyp] -
                        (jmkp - jmkm) * f5[cym] + (ipkp - imkp) * f3[c + dkp] - (ipkm - imkm) * f3[c + dkm] +
                        (ipkp - ipkm) * f3[cxp] - (imkp - imkm) * f3[cxm];
      const double num = __fma_rn(-0.5, s2, rhs[n2 * k + c] * dx2x2 - s1);
      sp[((yl + 3) << lgn) + oc] = -(num / d);
    }
    __syncthreads();
  }
  double* out = dst + n2 * k;
  for (int e = threadIdx.x; e < ty << lgn; e += kRowThreads) {
    const int r = e >> lgn, x = e & (n - 1);
    out[((i64)(y0 + r) << lgn) + x] = sp[((r + 3) << lgn) + (x & 1) * h + (x >> 1)];
  }
}

int rows_ty(int n) { return n == 32 ? 8 : (n == 64 || n > 512 ? 16 : 32); }

// ---------------------------------------------------------------------------
// n = 4, 8, 16: nsweeps whole 8-colour sweeps in one launch.  A cluster of CL
// CTAs holds the grid, each CTA a box of BX x BY x BZ cells (CC cells per
// colour) with a halo of one; an updated cell on a box's surface is stored
// into its neighbours' halos through distributed shared memory, and a
// cluster barrier ends the colour phase.
//
// One update is 60 FP64 operations and a division, a chain of about 50 for
// one thread; a colour has only 8, 64 or 512 cells, so splitting the chain is
// what counts.  The products of an update (12 cross terms, 6 faces) each have
// a lane of their own, and only the two sums, in the reference's order, are
// serial.  The division uses the correctly rounded reciprocal of the diagonal
// (formed once per launch): two corrected steps give the correctly rounded
// quotient (Markstein 1990; the second step starts from a faithful quotient).
// Colour p = 4k + 2i + j reads, among the cells updated one phase before it,
//   p = 1, 3, 5, 7: its y neighbours (two face products);
//   p = 2, 6: its xy diagonals (the first four cross terms);
//   p = 0, 4: nothing.
// So while phase p runs its serial part (warp F), the others form the
// products of phase p + 1 that do not depend on p and sum its cross terms
// (warp S): a phase costs 13, 13, 20, 13 dependent FP64 instructions instead
// of some 75 (64 cycles each).
// A whole sweep that leaves every bit of the 4^3 grid unchanged ends the
// sweeps: the remaining ones would repeat it.
// Against one CTA with a thread per cell: 32 sweeps at 4^3 197 us (747), at
// 8^3 323 us (771); 16 sweeps at 16^3 185 us (1508).
// ---------------------------------------------------------------------------
template <int N>
struct BoxGeom {
  static constexpr int BX = N == 16 ? 8 : 4, BY = BX, BZ = 4;
  static constexpr int GX = N / BX, GY = N / BY, GZ = N / BZ, CL = GX * GY * GZ;
  static constexpr int CC = BX * BY * BZ / 8;             // cells per colour: 8 or 32
  static constexpr int SX = BX + 2, SY = BY + 2, SZ = BZ + 2;
  static constexpr int PHI = SX * SY * SZ;
  static constexpr int NT = CC == 8 ? 128 : 512;
  static constexpr int NXT = CC == 8 ? 96 : 384;          // threads with a cross product
};

__device__ __forceinline__ void bar_sync(int id, int count) {
  asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(count) : "memory");
}
__device__ __forceinline__ void bar_arrive(int id, int count) {
  asm volatile("bar.arrive %0, %1;" ::"r"(id), "r"(count) : "memory");
}
__device__ __forceinline__ bool mid_exp(double x) {
  const int e = (int)((__double_as_longlong(x) >> 52) & 0x7ff);
  return e > 623 && e < 1423;
}

template <int N>
__global__ void __launch_bounds__(BoxGeom<N>::NT) k_gs_box(double* __restrict__ phi, const double* __restrict__ rhs,
                                                           const double* __restrict__ coef, double dx2x2,
                                                           int nsweeps) {
  typedef BoxGeom<N> G;
  constexpr int CC = G::CC, SX = G::SX, SXY = G::SX * G::SY, NN = N * N, N3 = N * N * N;
  __shared__ double sp[G::PHI];
  __shared__ double cross[2][12][CC];  // signed cross products of a phase, by phase parity
  __shared__ double face[2][6][CC];    // face products x+ x- y+ y- z+ z-
  __shared__ double sum2[2][CC];       // S2 of a phase (of S1 for p = 2, 6), by phase parity
  __shared__ int stop;
  cg::cluster_group cl = cg::this_cluster();
  const int rank = G::CL == 1 ? 0 : (int)cl.block_rank();
  const int bx = rank % G::GX, by = (rank / G::GX) % G::GY, bz = rank / (G::GX * G::GY);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  // The warp's part.  CC = 8: F = warp 0; cross terms 4 per warp on warps
  // 1-3; faces x, z on warp 2 and y on warp 3; S = warp 1.  CC = 32: F = warp
  // 0, S = warp 1; one cross term per warp on the warps below (8 of them on
  // the two SM quarters without F and S), six faces on the first six of those.
  const int cell = CC == 8 ? (lane & 7) : lane;
  int xterm = -1, fterm = -1;
  if (CC == 8) {
    if (warp >= 1) xterm = (warp - 1) * 4 + (lane >> 3);
    if (warp == 2) fterm = (lane >> 3) < 2 ? (lane >> 3) : (lane >> 3) + 2;
    if (warp == 3 && (lane >> 3) < 2) fterm = 2 + (lane >> 3);
  } else {
    const int slot = (warp & 2) ? ((warp >> 2) * 2 + (warp & 1)) : (warp == 4 ? 8 : warp == 5 ? 9 : warp == 8 ? 10
                     : warp == 9 ? 11 : -1);
    xterm = slot;
    if (slot >= 0 && slot < 6) fterm = slot;
  }
  const int a = cell % (G::BX / 2), b = (cell / (G::BX / 2)) % (G::BY / 2), d = cell / (G::BX / 2 * (G::BY / 2));
  // box origin, and global cell (x, y, z) + offset with periodic wrap
  const int x0 = bx * G::BX, y0 = by * G::BY, z0 = bz * G::BZ;
  auto gidx = [&](int x, int y, int z) {
    return ((x + N) & (N - 1)) + N * ((y + N) & (N - 1)) + NN * ((z + N) & (N - 1));
  };
  for (int e = tid; e < G::PHI; e += G::NT)
    sp[e] = phi[gidx(x0 + e % SX - 1, y0 + (e / SX) % G::SY - 1, z0 + e / SXY - 1)];
  const int base = (2 * a + 1) + SX * (2 * b + 1) + SXY * (2 * d + 1);
  auto off = [](int p) { return ((p >> 1) & 1) + SX * (p & 1) + SXY * (p >> 2); };
  // cross term t: coefficient plane and its cell, the two phi operands
  // (offsets from the cell), sign folded into the coefficient
  int xo1 = 0, xo2 = 0, fo = 0;
  // per colour: a producer's cross coefficient and face sum; warp F's
  // right-hand side and upper y face sum in the same registers
  double xc[8], fc[8];
#pragma unroll
  for (int p = 0; p < 8; ++p) xc[p] = fc[p] = 0.0;
  if (xterm >= 0) {
    const int grp = xterm >> 2, u = xterm & 3;  // xy, yz, xz; u: +-along the second axis, then the first
    // axes (A, B): xy -> (x, y), yz -> (y, z), xz -> (x, z)
    const int dA = grp == 1 ? SX : 1, dB = grp == 0 ? SX : SXY;
    const int sg = (u & 1) ? -1 : 1;
    // u = 0, 1: (difference along A at B+-1) f(B+-1); u = 2, 3: (difference along B at A+-1) f(A+-1)
    xo1 = u < 2 ? dA + sg * dB : sg * dA + dB;
    xo2 = u < 2 ? -dA + sg * dB : sg * dA - dB;
    const int ax = u < 2 ? (grp == 0 ? 1 : 2) : (grp == 1 ? 1 : 0);  // axis of the coefficient's cell
    const double* f = coef + (grp == 0 ? 1 : grp == 1 ? 4 : 2) * N3;
#pragma unroll
    for (int p = 0; p < 8; ++p) {
      const int x = x0 + 2 * a + ((p >> 1) & 1), y = y0 + 2 * b + (p & 1), z = z0 + 2 * d + (p >> 2);
      const double v = f[gidx(x + (ax == 0 ? sg : 0), y + (ax == 1 ? sg : 0), z + (ax == 2 ? sg : 0))];
      xc[p] = sg < 0 ? -v : v;
    }
  }
  auto face_coef = [&](int t, int p) {
    const int ax = t >> 1, sg = (t & 1) ? -1 : 1;
    const int x = x0 + 2 * a + ((p >> 1) & 1), y = y0 + 2 * b + (p & 1), z = z0 + 2 * d + (p >> 2);
    const double* f = coef + (ax == 0 ? 0 : ax == 1 ? 3 : 5) * N3;
    return f[gidx(x + (ax == 0 ? sg : 0), y + (ax == 1 ? sg : 0), z + (ax == 2 ? sg : 0))] + f[gidx(x, y, z)];
  };
  if (fterm >= 0) {
    const int ax = fterm >> 1, sg = (fterm & 1) ? -1 : 1;
    fo = sg * (ax == 0 ? 1 : ax == 1 ? SX : SXY);
#pragma unroll
    for (int p = 0; p < 8; ++p) fc[p] = face_coef(fterm, p);
  }
  // warp F: diagonal, its reciprocal and the lower y face sum per colour
  double(&X2)[8] = xc;
  double(&yp)[8] = fc;
  double D[8], Y[8], ym[8];
  unsigned ok = 0;
  if (warp == 0) {
#pragma unroll
    for (int p = 0; p < 8; ++p) {
      const int x = x0 + 2 * a + ((p >> 1) & 1), y = y0 + 2 * b + (p & 1), z = z0 + 2 * d + (p >> 2);
      X2[p] = rhs[gidx(x, y, z)] * dx2x2;
      yp[p] = face_coef(2, p);
      ym[p] = face_coef(3, p);
      D[p] = face_coef(0, p) + face_coef(1, p) + yp[p] + ym[p] + face_coef(4, p) + face_coef(5, p);
      Y[p] = 1.0 / D[p];
      if (mid_exp(D[p])) ok |= 1u << p;
    }
  }
  if (tid == 0) stop = 0;
  // every CTA of the cluster runs and has its halo before the first store into it
  if (G::CL == 1) __syncthreads();
  else cl.sync();

  // products of phase p for the cross terms [t0, 12) and the faces, y faces
  // only where they do not depend on the phase before
  auto cross_products = [&](int p, bool first4, bool rest) {
    if (xterm >= 0 && (xterm < 4 ? first4 : rest)) {
      const int c = base + off(p);
      cross[p & 1][xterm][cell] = (sp[c + xo1] - sp[c + xo2]) * xc[p];
    }
  };
  auto face_products = [&](int p) {
    if (fterm >= 0 && (!(p & 1) || (fterm >> 1) != 1)) face[p & 1][fterm][cell] = fc[p] * sp[base + off(p) + fo];
  };
  auto cross_sum = [&](int p) {
    const double(*cr)[CC] = cross[p & 1];
    double s = cr[0][cell];
#pragma unroll
    for (int t = 1; t < 12; ++t) s = s + cr[t][cell];
    return s;
  };
  auto face_sum = [&](int p) {
    const double(*f)[CC] = face[p & 1];
    double s = f[0][cell];
#pragma unroll
    for (int t = 1; t < 6; ++t) s = s + f[t][cell];
    return s;
  };
  // everything of phase p + 1 that phase p does not touch; barrier 1 hands
  // the products to S
  constexpr int kProd = G::NXT + (CC == 8 ? 0 : 32);
  auto ahead = [&](int p) {
    const int t = p & 3;
    const bool producer = xterm >= 0;
    const bool summer = warp == 1;
    if (producer) {
      cross_products(p, t != 2, true);
      face_products(p);
    }
    if (summer) {
      bar_sync(1, kProd);
      if (CC == 32 || lane < 8) sum2[p & 1][cell] = t == 2 ? face_sum(p) : cross_sum(p);
    } else if (producer) {
      bar_arrive(1, kProd);
    }
  };
  ahead(0);
  __syncthreads();
  bool changed = false;
  for (int sw = 0; sw < nsweeps; ++sw) {
#pragma unroll
    for (int p = 0; p < 8; ++p) {
      const int t = p & 3;
      const int c = base + off(p);
      // p = 2, 6: the four terms that read the phase before (their warps'
      // lanes, then warp F through barrier 2)
      if (t == 2) {
        constexpr int k4 = (CC == 8 ? 32 : 128) + 32;
        if (xterm >= 0 && xterm < 4) {
          cross_products(p, true, false);
          bar_arrive(2, k4);
        } else if (warp == 0) {
          bar_sync(2, k4);
        }
      }
      if (warp != 0) {
        ahead((p + 1) & 7);
      } else {
        double s1, s2;
        if (t == 2) {
          s1 = sum2[p & 1][cell];
          s2 = cross_sum(p);
        } else if (t == 0) {
          s1 = face_sum(p);
          s2 = sum2[p & 1][cell];
        } else {
          const double fp = yp[p] * sp[c + SX], fm = ym[p] * sp[c - SX];
          const double(*f)[CC] = face[p & 1];
          s1 = f[0][cell] + f[1][cell];
          s1 = s1 + fp;
          s1 = s1 + fm;
          s1 = s1 + f[4][cell];
          s1 = s1 + f[5][cell];
          s2 = sum2[p & 1][cell];
        }
        const double num = __fma_rn(-0.5, s2, X2[p] - s1);
        double v;
        if ((ok >> p & 1u) && mid_exp(num)) {
          const double y = Y[p], dd = D[p];
          double q = num * y;
          q = __fma_rn(__fma_rn(-dd, q, num), y, q);
          q = __fma_rn(__fma_rn(-dd, q, num), y, q);
          v = -q;
        } else {
          v = -(num / D[p]);
        }
        if (N == 4) changed = changed || __double_as_longlong(v) != __double_as_longlong(sp[c]);
        // the cell, and its copies in the neighbours' halos: faces and edges
        const int i = (p >> 1) & 1, j = p & 1, kz = p >> 2;
        const int sx = i == 0 ? (a == 0 ? -1 : 0) : (a == G::BX / 2 - 1 ? 1 : 0);
        const int sy = j == 0 ? (b == 0 ? -1 : 0) : (b == G::BY / 2 - 1 ? 1 : 0);
        const int sz = kz == 0 ? (d == 0 ? -1 : 0) : (d == G::BZ / 2 - 1 ? 1 : 0);
        auto push = [&](int ux, int uy, int uz) {
          const int r = (bx + ux + G::GX) % G::GX +
                        G::GX * ((by + uy + G::GY) % G::GY + G::GY * ((bz + uz + G::GZ) % G::GZ));
          double* w = (G::CL == 1 || r == rank) ? sp : cl.map_shared_rank(sp, r);
          w[c - ux * G::BX - uy * G::BY * SX - uz * G::BZ * SXY] = v;
        };
        if (CC == 32 || lane < 8) {
          sp[c] = v;
          if (sx) push(sx, 0, 0);
          if (sy) push(0, sy, 0);
          if (sz) push(0, 0, sz);
          if (sx && sy) push(sx, sy, 0);
          if (sy && sz) push(0, sy, sz);
          if (sx && sz) push(sx, 0, sz);
        }
        if (N == 4 && p == 7) {
          const bool any = __any_sync(0xffffffffu, changed);
          changed = false;
          if (lane == 0) stop = any ? 0 : 1;
        }
      }
      if (G::CL == 1) __syncthreads();
      else cl.sync();
    }
    if (N == 4 && stop) break;
  }
  for (int e = tid; e < G::BX * G::BY * G::BZ; e += G::NT) {
    const int x = e % G::BX, y = (e / G::BX) % G::BY, z = e / (G::BX * G::BY);
    phi[gidx(x0 + x, y0 + y, z0 + z)] = sp[(x + 1) + SX * (y + 1) + SXY * (z + 1)];
  }
}

template <int N>
void box_launch(double* phi, const double* rhs, const double* coef, double dx2, int nsweeps, cudaStream_t s) {
  typedef BoxGeom<N> G;
  if (G::CL == 1) {
    k_gs_box<N><<<1, G::NT, 0, s>>>(phi, rhs, coef, 2.0 * dx2, nsweeps);
    return;
  }
  if (G::CL > 8) {
    static std::atomic<unsigned long long> attr_done{0};
    func_attr_once(k_gs_box<N>, cudaFuncAttributeNonPortableClusterSizeAllowed, 1, attr_done);
  }
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(G::CL);
  cfg.blockDim = dim3(G::NT);
  cfg.stream = s;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = G::CL;
  at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  cudaLaunchKernelEx(&cfg, k_gs_box<N>, phi, rhs, coef, 2.0 * dx2, nsweeps);
}

}  // namespace

// nsweeps FP64 8-colour sweeps of phi on an n^3 grid; scratch: n^3 doubles
// (n >= 32).  Returns the buffer that holds the swept field.
double* launch_gs64_sweeps(double* phi, const double* rhs, const double* coef, int n, double dx, int nsweeps,
                           double* scratch, cudaStream_t s) {
  if (nsweeps <= 0) return phi;
  const i64 h3 = (i64)(n / 2) * (n / 2) * (n / 2);
  const double dx2 = dx * dx;
  if (n <= 16) {
    prof_begin(KK_GS, s, h3 * 8 * nsweeps, n);
    if (n == 4) box_launch<4>(phi, rhs, coef, dx2, nsweeps, s);
    else if (n == 8) box_launch<8>(phi, rhs, coef, dx2, nsweeps, s);
    else box_launch<16>(phi, rhs, coef, dx2, nsweeps, s);
    prof_end(KK_GS, s, n);
    count_launch();
    return phi;
  }
  int lgn = 0;
  while ((1 << lgn) < n) ++lgn;
  const int ty = rows_ty(n), smem = (int)(sizeof(double) * (ty + 7) * n);
  static std::atomic<unsigned long long> attr_done{0};
  smem_attr_once(k_gs_rows, 8 * 23 * 1024, attr_done);  // the largest of any size
  // double buffer: a sweep reads a and leaves the swept field in b
  double *a = phi, *b = scratch;
  for (int sw = 0; sw < nsweeps; ++sw) {
    for (int kpar = 0; kpar < 2; ++kpar) {
      prof_begin(KK_GS, s, 4 * h3, n);
      k_gs_rows<<<dim3(n / ty, n / 2), kRowThreads, smem, s>>>(a, kpar == 0 ? a : b, b, rhs, coef, lgn, ty, 2.0 * dx2,
                                                               kpar);
      prof_end(KK_GS, s, n);
      count_launch();
    }
    std::swap(a, b);
  }
  return a;
}

}  // namespace mmh

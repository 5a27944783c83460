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
//   - the FP64 form's solver keeps, with each metric, the face sums, the
//     diagonal and its reciprocal (Face64) in place of three coefficient
//     planes: 53 FP64 instructions per update instead of 69, 52 per residual;
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
// n >= 32 (and 16 where the box kernel's cluster does not fit): one half sweep
// (the four in-plane colours of every plane of one parity).  A CTA owns TY full
// rows of one plane.  phi of the plane (rows -3 .. TY+3) sits in shared memory, each row split into its even-x and odd-x
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
// one-colour launches): 256^3 0.99 ms (2.25), 128^3 0.137 ms (0.30), 64^3
// 24.4 us (48), 32^3 14.3 us (38).
// ---------------------------------------------------------------------------
constexpr int kRowThreads = 256;

// Offsets of a cell's neighbours from its plane's first element
struct Nbr {
  i64 c, xp, xm, yp, ym;
};
// S1 = 2 t1, S2 = 4 t2 and D = -2 tdiag of one cell; fields as in Face64 (PRE)
// or the coefficient planes (else), at the cell's plane; phi: in-plane values
// through P(dx, dy), neighbour planes Kp, Km.
struct Fields {
  const double *bx, *by, *bz, *f2, *f3, *f5, *d;  // !PRE: bx, by, bz = f1, f4, f6
  i64 dkp, dkm;                                   // to the planes above and below
};
template <bool PRE, class P>
__device__ __forceinline__ void sums64(const Fields& f, const Nbr& o, P&& p, const double* __restrict__ Kp,
                                       const double* __restrict__ Km, double& s1, double& s2, double& d) {
  double b11p, b11m, b22p, b22m, b33p, b33m;
  if (PRE) {
    b11p = f.bx[o.c]; b11m = f.bx[o.xm];
    b22p = f.by[o.c]; b22m = f.by[o.ym];
    b33p = f.bz[o.c]; b33m = f.bz[o.c + f.dkm];
    d = f.d[o.c];
  } else {
    const double f1c = f.bx[o.c], f4c = f.by[o.c], f6c = f.bz[o.c];
    b11p = f.bx[o.xp] + f1c; b11m = f.bx[o.xm] + f1c;
    b22p = f.by[o.yp] + f4c; b22m = f.by[o.ym] + f4c;
    b33p = f.bz[o.c + f.dkp] + f6c; b33m = f.bz[o.c + f.dkm] + f6c;
    d = b11p + b11m + b22p + b22m + b33p + b33m;
  }
  s1 = b11p * p(1, 0) + b11m * p(-1, 0) + b22p * p(0, 1) + b22m * p(0, -1) + b33p * Kp[o.c] + b33m * Km[o.c];
  const double ppk = p(1, 1), mpk = p(-1, 1), pmk = p(1, -1), mmk = p(-1, -1);
  const double jpkp = Kp[o.yp], jmkp = Kp[o.ym], jpkm = Km[o.yp], jmkm = Km[o.ym];
  const double ipkp = Kp[o.xp], imkp = Kp[o.xm], ipkm = Km[o.xp], imkm = Km[o.xm];
  s2 = (ppk - mpk) * f.f2[o.yp] - (pmk - mmk) * f.f2[o.ym] + (ppk - pmk) * f.f2[o.xp] - (mpk - mmk) * f.f2[o.xm] +
       (jpkp - jmkp) * f.f5[o.c + f.dkp] - (jpkm - jmkm) * f.f5[o.c + f.dkm] + (jpkp - jpkm) * f.f5[o.yp] -
       (jmkp - jmkm) * f.f5[o.ym] + (ipkp - imkp) * f.f3[o.c + f.dkp] - (ipkm - imkm) * f.f3[o.c + f.dkm] +
       (ipkp - ipkm) * f.f3[o.xp] - (imkp - imkm) * f.f3[o.xm];
}
template <bool PRE>
__device__ __forceinline__ Fields fields64(const Face64& a, i64 n2, i64 plane, i64 dkp, i64 dkm) {
  const i64 o = n2 * plane;
  Fields f;
  f.bx = a.bx + o; f.by = a.by + o; f.bz = a.bz + o;
  f.f2 = a.f2 + o; f.f3 = a.f3 + o; f.f5 = a.f5 + o;
  f.d = PRE ? a.d + o : nullptr;
  f.dkp = dkp; f.dkm = dkm;
  return f;
}
// the coefficient planes themselves
Face64 raw64(const double* coef, i64 n3) {
  return Face64{coef, coef + 3 * n3, coef + 5 * n3, coef + n3, coef + 2 * n3, coef + 4 * n3, nullptr, nullptr};
}

// CL (64^3 and 128^3): the CTAs of a plane are a cluster of four, and the one
// boundary row that the next colour reads is stored into the neighbour's halo, so
// no cell is updated twice (19% at 16 rows, 9% at 32) and the rows of a colour
// divide evenly over the warps: 64^3 29.3 -> 24.4 us, 128^3 148 -> 137 us.  At
// 256^3 the cluster's barriers cost more than the 9% (1.06 ms for 0.99), at 32^3 a
// colour is one warp per SM quarter either way.
template <bool PRE, bool CL>
__global__ void __launch_bounds__(kRowThreads, 2) k_gs_rows(const double* __restrict__ src,
                                                            const double* __restrict__ nbr, double* __restrict__ dst,
                                                            const double* __restrict__ rhs, Face64 co, int lgn, int ty,
                                                            double dx2x2, int kpar) {
  extern __shared__ double sp[];
  constexpr int LO = CL ? 1 : 3, HALO = CL ? 2 : 7;  // rows held below the own ones, and in all
  const int n = 1 << lgn, h = n >> 1, lgh = lgn - 1;
  const i64 n2 = (i64)n << lgn;
  const int y0 = blockIdx.x * ty, k = 2 * blockIdx.y + kpar;
  const int kp = wp(k, n), km = wm(k, n);
  const double* own = src + n2 * k;
  for (int e = threadIdx.x; e < (ty + HALO) << lgn; e += kRowThreads) {
    const int r = e >> lgn, x = e & (n - 1);
    const int y = (y0 + r - LO) & (n - 1);
    sp[(r << lgn) + (x & 1) * h + (x >> 1)] = own[((i64)y << lgn) + x];
  }
  double *below = nullptr, *above = nullptr;  // the row above the last of the CTA below, below the first of the one above
  if constexpr (CL) {
    cg::cluster_group cl = cg::this_cluster();
    const unsigned rank = cl.block_rank(), size = cl.num_blocks();
    below = cl.map_shared_rank(sp, (rank + size - 1) % size) + ((ty + LO) << lgn);
    above = cl.map_shared_rank(sp, (rank + 1) % size);
    cl.sync();  // every CTA has its halo before the first store into it
  } else {
    __syncthreads();
  }
  const double* Kp = nbr + n2 * kp;
  const double* Km = nbr + n2 * km;
  const Fields f = fields64<PRE>(co, n2, k, n2 * (kp - k), n2 * (km - k));
  const double* rk = rhs + n2 * k;
  const double* yk = PRE ? co.y + n2 * k : nullptr;
#pragma unroll 1
  for (int q = 0; q < 4; ++q) {
    const int io = q >> 1;
    const int cells = (CL ? ty / 2 : ty / 2 + 3 - q) << lgh;
#pragma unroll 1
    for (int e = threadIdx.x; e < cells; e += kRowThreads) {
      const int m = e & (h - 1), yl = (CL ? q & 1 : q - 2) + 2 * (e >> lgh);  // row relative to y0
      const int x = 2 * m + io, xp = (x + 1) & (n - 1), xm = (x - 1) & (n - 1);
      const int y = (y0 + yl) & (n - 1), yp = (y + 1) & (n - 1), ym = (y - 1) & (n - 1);
      const i64 r0 = (i64)y << lgn;
      const Nbr o{r0 + x, r0 + xp, r0 + xm, ((i64)yp << lgn) + x, ((i64)ym << lgn) + x};
      // phi of the plane: rows yl+2 .. yl+4 of the tile, x+-1 in the other half
      double* s0 = sp + ((yl + LO) << lgn);
      const int oc = io * h + m, op = (xp & 1) * h + (xp >> 1), om = (xm & 1) * h + (xm >> 1);
      double s1, s2, d;
      sums64<PRE>(
          f, o, [&](int dx, int dy) { return s0[dy * n + (dx > 0 ? op : dx < 0 ? om : oc)]; }, Kp, Km, s1, s2, d);
      // Face64 comes with the levels' own spacings, powers of two: rhs 2dx2 is exact
      const double lead = PRE ? __fma_rn(rk[o.c], dx2x2, -s1) : rk[o.c] * dx2x2 - s1;
      const double num = __fma_rn(-0.5, s2, lead);
      const double v = neg_of(PRE ? div_by(num, d, yk[o.c]) : num / d);
      s0[oc] = v;
      if (CL && q < 3) {
        if (yl == 0) below[oc] = v;
        if (yl == ty - 1) above[oc] = v;
      }
    }
    if (CL && q < 3) cg::this_cluster().sync();
    else __syncthreads();
  }
  double* out = dst + n2 * k;
  for (int e = threadIdx.x; e < ty << lgn; e += kRowThreads) {
    const int r = e >> lgn, x = e & (n - 1);
    out[((i64)(y0 + r) << lgn) + x] = sp[((r + LO) << lgn) + (x & 1) * h + (x >> 1)];
  }
}

// MODE 0: r = rhs - L[phi] (r may be null), max|r|; 1: r = L[phi], max|r| --
// calcresid's operations (gauss1.f90:683-709) from the face sums.  One cell per
// thread straight from global memory: the FP64 pipe takes ten times as long as
// the loads.
template <int MODE>
__global__ void __launch_bounds__(256) k_op64(const double* __restrict__ phi, const double* __restrict__ rhs,
                                              Face64 co, int lgn, double hdi2, double* __restrict__ r,
                                              unsigned long long* maxbits) {
  const int n = 1 << lgn;
  const i64 n2 = (i64)n << lgn, t = (i64)blockIdx.x * blockDim.x + threadIdx.x;
  double v = 0.0;
  if (t < n2 << lgn) {
    const int x = (int)t & (n - 1), y = (int)(t >> lgn) & (n - 1), k = (int)(t >> (2 * lgn));
    const int kp = wp(k, n), km = wm(k, n), xp = wp(x, n), xm = wm(x, n);
    const i64 r0 = (i64)y << lgn, rp = (i64)wp(y, n) << lgn, rm = (i64)wm(y, n) << lgn;
    const Nbr o{r0 + x, r0 + xp, r0 + xm, rp + x, rm + x};
    const double* P = phi + n2 * k;
    const double* rows[3] = {P + rm, P + r0, P + rp};
    double s1, s2, d;
    sums64<true>(
        fields64<true>(co, n2, k, n2 * (kp - k), n2 * (km - k)), o,
        [&](int dx, int dy) { return rows[dy + 1][dx > 0 ? xp : dx < 0 ? xm : x]; }, phi + n2 * kp, phi + n2 * km, s1,
        s2, d);
    // t1 + t2 + tdiag phi = half of (S1 + S2/2) - D phi
    v = (__fma_rn(0.5, s2, s1) - d * P[o.c]) * hdi2;
    if (MODE == 0) v = rhs[t] - v;
    if (r) r[t] = v;
    v = fabs(v);
  }
  if (maxbits) block_max_commit(v, maxbits);
}

// out = f + f one cell up along the axis
__global__ void k_face_sum(const double* __restrict__ f, int n, int axis, double* __restrict__ out) {
  const i64 t = (i64)blockIdx.x * blockDim.x + threadIdx.x, n3 = (i64)n * n * n;
  if (t >= n3) return;
  int c[3];
  cell_of(t, n, c[0], c[1], c[2]);
  const i64 st = axis == 0 ? 1 : (axis == 1 ? (i64)n : (i64)n * n);
  out[t] = f[c[axis] == n - 1 ? t - (n - 1) * st : t + st] + f[t];
}
// d = sum of the six face sums in relaxplane's order, y = 1 / d
__global__ void k_face_diag(const double* __restrict__ bx, const double* __restrict__ by,
                            const double* __restrict__ bz, int n, double* __restrict__ d, double* __restrict__ y) {
  const i64 t = (i64)blockIdx.x * blockDim.x + threadIdx.x, n3 = (i64)n * n * n;
  if (t >= n3) return;
  int i, j, k;
  cell_of(t, n, i, j, k);
  const double v = bx[t] + bx[IDX(wm(i, n), j, k, n)] + by[t] + by[IDX(i, wm(j, n), k, n)] + bz[t] +
                   bz[IDX(i, j, wm(k, n), n)];
  d[t] = v;
  y[t] = 1.0 / v;
}

int lg(int n) {
  int l = 0;
  while ((1 << l) < n) ++l;
  return l;
}
int rows_ty(int n) { return n <= 32 ? 8 : (n == 64 || n > 512 ? 16 : 32); }

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
// (formed once per launch, div_by).
// Colour p = 4k + 2i + j reads, among the cells updated one phase before it,
//   p = 1, 3, 5, 7: its y neighbours (two face products);
//   p = 2, 6: its xy diagonals (the first four cross terms);
//   p = 0, 4: nothing.
// So while phase p runs its serial part (warp F), the others form the
// products of phase p + 1 that do not depend on p and sum its cross terms
// (warp S): a phase costs 13, 13, 20, 13 dependent FP64 instructions instead
// of some 75 (64 cycles each).
// Against one CTA with a thread per cell: 32 sweeps at 4^3 183 us (747), at
// 8^3 244 us (771); 16 sweeps at 16^3 162 us (1508).
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
// address of a shared variable in CTA `rank` of the cluster, and a store to it
__device__ __forceinline__ unsigned mapa(unsigned addr, int rank) {
  unsigned r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
  return r;
}
__device__ __forceinline__ void st_cluster(unsigned addr, double v) {
  asm volatile("st.shared::cluster.f64 [%0], %1;" ::"r"(addr), "d"(v) : "memory");
}
__device__ __forceinline__ void bar_arrive(int id, int count) {
  asm volatile("bar.arrive %0, %1;" ::"r"(id), "r"(count) : "memory");
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
  // Warp F's stores of an updated cell: itself and, when it lies on the box's
  // surface, its copies in the neighbours' halos (faces and edges).  A colour
  // lies on the lower side of an axis where its parity is 0, on the upper one
  // where it is 1; ok[s] has a bit per colour for set s of axes.  CC = 8: the
  // four groups of 8 lanes hold the same cells and share the seven stores (two
  // at most per lane); CC = 32: a lane makes all of its own.
  constexpr int NS = CC == 8 ? 2 : 6;
  unsigned ok_[NS], base_[NS][G::GZ > 2 ? 2 : 1];
  int shift_[CC == 8 ? 2 : 1][3];
  const unsigned here = (unsigned)__cvta_generic_to_shared(sp);
  auto axes_ok = [&](int set) {
    unsigned m = 0;
    for (int p = 0; p < 8; ++p) {
      const bool sx = ((p >> 1) & 1) ? a == G::BX / 2 - 1 : a == 0;
      const bool sy = (p & 1) ? b == G::BY / 2 - 1 : b == 0;
      const bool sz = (p >> 2) ? d == G::BZ / 2 - 1 : d == 0;
      if ((!(set & 1) || sx) && (!(set & 2) || sy) && (!(set & 4) || sz)) m |= 1u << p;
    }
    return m;
  };
  auto target = [&](int set, int uz) {  // the neighbour along the axes of the set (z: uz = -1 or 1)
    const int r = (bx + (set & 1)) % G::GX + G::GX * ((by + ((set >> 1) & 1)) % G::GY +
                                                     G::GY * ((bz + ((set >> 2) & 1) * (uz + G::GZ)) % G::GZ));
    return mapa(here, r);
  };
  if (CC == 8) {
    // sets by lane group: {own, xy}, {x, yz}, {y, xz}, {z, -}
    const int g = lane >> 3;
    const int set[2] = {g == 0 ? 0 : g == 1 ? 1 : g == 2 ? 2 : 4, g == 0 ? 3 : g == 1 ? 6 : 5};
#pragma unroll
    for (int s = 0; s < 2; ++s) {
      ok_[s] = (s == 1 && g == 3) ? 0u : axes_ok(set[s]);
      base_[s][0] = target(set[s], 1);  // GX = GY = GZ = 1 or 2: either sign is the same box
      shift_[s][0] = (set[s] & 1) ? G::BX : 0;
      shift_[s][1] = (set[s] & 2) ? G::BY * SX : 0;
      shift_[s][2] = (set[s] & 4) ? G::BZ * SXY : 0;
    }
  } else {
    constexpr int sets[6] = {1, 2, 3, 4, 5, 6};
#pragma unroll
    for (int s = 0; s < NS; ++s) {
      ok_[s] = axes_ok(sets[s]);
      base_[s][0] = target(sets[s], -1);
      if (G::GZ > 2) base_[s][G::GZ > 2 ? 1 : 0] = target(sets[s], 1);
    }
  }
  // warp F: diagonal, its reciprocal and the lower y face sum per colour
  double(&X2)[8] = xc;
  double(&yp)[8] = fc;
  double D[8], Y[8], ym[8];
  if (warp == 0) {
#pragma unroll
    for (int p = 0; p < 8; ++p) {
      const int x = x0 + 2 * a + ((p >> 1) & 1), y = y0 + 2 * b + (p & 1), z = z0 + 2 * d + (p >> 2);
      X2[p] = rhs[gidx(x, y, z)] * dx2x2;
      yp[p] = face_coef(2, p);
      ym[p] = face_coef(3, p);
      D[p] = face_coef(0, p) + face_coef(1, p) + yp[p] + ym[p] + face_coef(4, p) + face_coef(5, p);
      Y[p] = 1.0 / D[p];
    }
  }
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
        const double v = neg_of(div_by(__fma_rn(-0.5, s2, X2[p] - s1), D[p], Y[p]));
        const int i = (p >> 1) & 1, j = p & 1, kz = p >> 2;
        if (CC == 8) {
          // the box itself (and, alone, its own neighbour) by a plain store: a
          // cluster store to the own CTA takes the way between SMs too
#pragma unroll
          for (int s = 0; s < 2; ++s)
            if (ok_[s] >> p & 1u) {
              const int e = c + (i ? -shift_[s][0] : shift_[s][0]) + (j ? -shift_[s][1] : shift_[s][1]) +
                            (kz ? -shift_[s][2] : shift_[s][2]);
              if (G::CL == 1 || (s == 0 && lane < 8)) sp[e] = v;
              else st_cluster(base_[s][0] + 8u * e, v);
            }
        } else {
          constexpr int sets[6] = {1, 2, 3, 4, 5, 6};
          sp[c] = v;
#pragma unroll
          for (int s = 0; s < NS; ++s) {
            const int off = ((sets[s] & 1) ? (i ? -G::BX : G::BX) : 0) + ((sets[s] & 2) ? (j ? -1 : 1) * G::BY * SX : 0) +
                            ((sets[s] & 4) ? (kz ? -1 : 1) * G::BZ * SXY : 0);
            if (ok_[s] >> p & 1u) st_cluster(base_[s][(sets[s] & 4) && G::GZ > 2 ? kz : 0] + 8u * (c + off), v);
          }
        }
      }
      if (G::CL == 1) __syncthreads();
      else cl.sync();
    }
  }
  for (int e = tid; e < G::BX * G::BY * G::BZ; e += G::NT) {
    const int x = e % G::BX, y = (e / G::BX) % G::BY, z = e / (G::BX * G::BY);
    phi[gidx(x0 + x, y0 + y, z0 + z)] = sp[(x + 1) + SX * (y + 1) + SXY * (z + 1)];
  }
}

// whether the box kernel of n = 16 has its cluster of 16 CTAs
bool box16_fits(cudaStream_t s) {
  typedef BoxGeom<16> G;
  static std::atomic<unsigned long long> attr_done{0};
  func_attr_once(k_gs_box<16>, cudaFuncAttributeNonPortableClusterSizeAllowed, 1, attr_done);
  return cluster_fits(k_gs_box<16>, G::CL, G::NT, 0, s);
}
template <int N>
void box_launch(double* phi, const double* rhs, const double* coef, double dx2, int nsweeps, cudaStream_t s) {
  typedef BoxGeom<N> G;
  if (G::CL == 1) {
    k_gs_box<N><<<1, G::NT, 0, s>>>(phi, rhs, coef, 2.0 * dx2, nsweeps);
    return;
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

namespace {
template <bool PRE, bool CL>
void rows_launch(const double* src, const double* nbr, double* dst, const double* rhs, const Face64& f, int lgn, int ty,
                 double dx2x2, int kpar, cudaStream_t s) {
  static std::atomic<unsigned long long> done{0};
  smem_attr_once(k_gs_rows<PRE, CL>, 8 * 23 * 1024, done);  // the largest of any size
  const int n = 1 << lgn;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(n / ty, n / 2);
  cfg.blockDim = dim3(kRowThreads);
  cfg.dynamicSmemBytes = sizeof(double) * (ty + (CL ? 2 : 7)) * n;
  cfg.stream = s;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = n / ty;
  at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
  cfg.attrs = at;
  cfg.numAttrs = CL ? 1 : 0;
  cudaLaunchKernelEx(&cfg, k_gs_rows<PRE, CL>, src, nbr, dst, rhs, f, lgn, ty, dx2x2, kpar);
}
// faces: the coefficients' face sums (null: the coefficient planes themselves).
// A 16^3 grid goes by rows where its box kernel's cluster does not fit.
double* gs64_sweeps(double* phi, const double* rhs, const double* coef, const Face64* faces, int n, double dx,
                    int nsweeps, double* scratch, cudaStream_t s, int max_cluster) {
  if (nsweeps <= 0) return phi;
  const i64 h3 = (i64)(n / 2) * (n / 2) * (n / 2);
  const double dx2 = dx * dx;
  if (n <= 8 || (n == 16 && max_cluster >= 16 && box16_fits(s))) {
    prof_begin(KK_GS, s, h3 * 8 * nsweeps, n);
    if (n == 4) box_launch<4>(phi, rhs, coef, dx2, nsweeps, s);
    else if (n == 8) box_launch<8>(phi, rhs, coef, dx2, nsweeps, s);
    else box_launch<16>(phi, rhs, coef, dx2, nsweeps, s);
    prof_end(KK_GS, s, n);
    count_launch();
    return phi;
  }
  const int lgn = lg(n), ty = rows_ty(n);
  const bool cl = n == 64 || n == 128;
  const Face64 f = faces ? *faces : raw64(coef, 8 * h3);
  // double buffer: a sweep reads a and leaves the swept field in b
  double *a = phi, *b = scratch;
  for (int sw = 0; sw < nsweeps; ++sw) {
    for (int kpar = 0; kpar < 2; ++kpar) {
      prof_begin(KK_GS, s, 4 * h3, n);
      const double* nbr = kpar == 0 ? a : b;
      if (faces && cl) rows_launch<true, true>(a, nbr, b, rhs, f, lgn, ty, 2.0 * dx2, kpar, s);
      else if (faces) rows_launch<true, false>(a, nbr, b, rhs, f, lgn, ty, 2.0 * dx2, kpar, s);
      else if (cl) rows_launch<false, true>(a, nbr, b, rhs, f, lgn, ty, 2.0 * dx2, kpar, s);
      else rows_launch<false, false>(a, nbr, b, rhs, f, lgn, ty, 2.0 * dx2, kpar, s);
      prof_end(KK_GS, s, n);
      count_launch();
    }
    std::swap(a, b);
  }
  return a;
}
}  // namespace

// nsweeps FP64 8-colour sweeps of phi on an n^3 grid; scratch: n^3 doubles
// (n >= 16).  Returns the buffer that holds the swept field.
double* launch_gs64_sweeps(double* phi, const double* rhs, const double* coef, int n, double dx, int nsweeps,
                           double* scratch, cudaStream_t s, int max_cluster) {
  return gs64_sweeps(phi, rhs, coef, nullptr, n, dx, nsweeps, scratch, s, max_cluster);
}
double* launch_gs64_sweeps(double* phi, const double* rhs, const Face64& f, int n, double dx, int nsweeps,
                           double* scratch, cudaStream_t s) {
  return gs64_sweeps(phi, rhs, nullptr, &f, n, dx, nsweeps, scratch, s, 16);
}

Face64 launch_faces64(double* coef, int n, double* s0, double* s1, cudaStream_t s) {
  const i64 n3 = (i64)n * n * n;
  const unsigned g = (unsigned)((n3 + 255) / 256);
  // each pass frees the plane the next one writes
  k_face_sum<<<g, 256, 0, s>>>(coef, n, 0, s0);
  k_face_sum<<<g, 256, 0, s>>>(coef + 3 * n3, n, 1, coef);
  k_face_sum<<<g, 256, 0, s>>>(coef + 5 * n3, n, 2, coef + 3 * n3);
  k_face_diag<<<g, 256, 0, s>>>(s0, coef, coef + 3 * n3, n, coef + 5 * n3, s1);
  count_launch(4);
  return Face64{s0, coef, coef + 3 * n3, coef + n3, coef + 2 * n3, coef + 4 * n3, coef + 5 * n3, s1};
}

void launch_residual64(const double* phi, const double* rhs, const Face64& f, int n, double dx, double* r,
                       unsigned long long* maxbits, cudaStream_t s) {
  const i64 n3 = (i64)n * n * n;
  prof_begin(KK_RESIDUAL, s, n3, n);
  k_op64<0><<<(unsigned)((n3 + 255) / 256), 256, 0, s>>>(phi, rhs, f, lg(n), 0.5 * (1.0 / (dx * dx)), r, maxbits);
  prof_end(KK_RESIDUAL, s, n);
  count_launch();
}
void launch_apply64(const double* p, const Face64& f, int n, double dx, double* q, unsigned long long* qbits,
                    cudaStream_t s) {
  const i64 n3 = (i64)n * n * n;
  prof_begin(KK_APPLY, s, n3, n);
  k_op64<1><<<(unsigned)((n3 + 255) / 256), 256, 0, s>>>(p, nullptr, f, lg(n), 0.5 * (1.0 / (dx * dx)), q, qbits);
  prof_end(KK_APPLY, s, n);
  count_launch();
}

}  // namespace mmh

// Dynamic Smagorinsky eddy viscosity for sm_100a: Compute_Smagorinsky_Constant_1
// (les.c:67-1133) and Compute_eddy_viscosity_LES (les.c:1135-1252), default options
// (3-D box test filter, testfilter_ik = 0, clark = 0, no homogeneous-direction averaging).
//
// FP64 throughout:
//   k_les_prep    every DA point: contravariant centre velocity U,V,W and test-filter
//                 weight of the point itself;
//   k_les_image   interior cells: the strain products S_ab*|S| and the test-filtered
//                 velocity (les.c:191-298); k_les_ghosts gives ghost points their image's;
//   k_les_lm      interior cells: the Germano identity contractions L_ij M_ij G and
//                 M_ij M_ij G (les.c:300-661);
//   k_les_cs      interior cells: filtered LM/MM, Cs = max(0, LM/(2(MM+eps))), wall floor
//                 and [0, max_cs] clipping (les.c:708-1048), ghosts as above;
//   k_les_refilter  second test filtering of Cs over fluid cells (les.c:1051-1120);
//   k_les_nut     nu_t = Cs * Delta^2 * |S| and its periodic ghosts (les.c:1174-1243).
// The 3x3x3 test filter is integrate_testfilter (rhs2.c:412-455): the weighted sums of eight
// overlapping 2x2x2 sub-cubes over the sums of their weights.  A cell's own point lies in
// all eight, a face neighbour in four, an edge neighbour in two, a corner in one, so the
// sum is the (1 2 1) x (1 2 1) x (1 2 1) sum of value x weight: three one-dimensional
// passes instead of 64 products (the same sum in another order).
#include <cmath>

#include "vfs_internal.cuh"

namespace vfs {

constexpr double kLesEps = 1.e-4;  // les_eps, les.c:20
constexpr double kWallCs = 0.001;  // wall_cs, les.c:21

__device__ __forceinline__ bool les_interior(const Grid &g, int i, int j, int k) {
  return i >= 1 && i <= g.mx - 2 && j >= 1 && j <= g.my - 2 && k >= 1 && k <= g.mz - 2;
}

// Compute_du_center (k-omega.c:305-420): centre derivatives of a vector field along the
// three grid directions, one-sided next to cells with nvert > 0.1 and at non-periodic
// boundaries.  d = {du/dc, dv/dc, dw/dc, du/de, dv/de, dw/de, du/dz, dv/dz, dw/dz}.
// The k test uses k == 0 where the i and j tests use 1 (k-omega.c:395), as the reference.
__device__ __forceinline__ void du_center(const Grid &g, CV3 u, const uint8_t *__restrict__ nv, long long p,
                                          int i, int j, int k, double d[9]) {
  const long long sy = g.mx, sz = (long long)g.mx * g.my;
  long long a, b;
  double f;
  if (nv[p + 1] > 0 || (!g.iper && i == g.mx - 2)) { a = p; b = p - 1; f = 1.0; }
  else if (nv[p - 1] > 0 || (!g.iper && i == 1)) { a = p + 1; b = p; f = 1.0; }
  else { a = p + 1; b = p - 1; f = 0.5; }
  d[0] = (u.x[a] - u.x[b]) * f; d[1] = (u.y[a] - u.y[b]) * f; d[2] = (u.z[a] - u.z[b]) * f;
  if (nv[p + sy] > 0 || (!g.jper && j == g.my - 2)) { a = p; b = p - sy; f = 1.0; }
  else if (nv[p - sy] > 0 || (!g.jper && j == 1)) { a = p + sy; b = p; f = 1.0; }
  else { a = p + sy; b = p - sy; f = 0.5; }
  d[3] = (u.x[a] - u.x[b]) * f; d[4] = (u.y[a] - u.y[b]) * f; d[5] = (u.z[a] - u.z[b]) * f;
  if (nv[p + sz] > 0 || (!g.kper && k == g.mz - 2)) { a = p; b = p - sz; f = 1.0; }
  else if (nv[p - sz] > 0 || (!g.kper && k == 0)) { a = p + sz; b = p; f = 1.0; }
  else { a = p + sz; b = p - sz; f = 0.5; }
  d[6] = (u.x[a] - u.x[b]) * f; d[7] = (u.y[a] - u.y[b]) * f; d[8] = (u.z[a] - u.z[b]) * f;
}

// Compute_du_dxyz (k-omega.c:597-610): Cartesian gradient by the chain rule.
// o = {du/dx, du/dy, du/dz, dv/dx, dv/dy, dv/dz, dw/dx, dw/dy, dw/dz}.
__device__ __forceinline__ void du_dxyz(const double c[3], const double e[3], const double z[3], double ajc,
                                        const double d[9], double o[9]) {
#pragma unroll
  for (int v = 0; v < 3; v++) {
    o[3 * v + 0] = (d[v] * c[0] + d[3 + v] * e[0] + d[6 + v] * z[0]) * ajc;
    o[3 * v + 1] = (d[v] * c[1] + d[3 + v] * e[1] + d[6 + v] * z[1]) * ajc;
    o[3 * v + 2] = (d[v] * c[2] + d[3 + v] * e[2] + d[6 + v] * z[2]) * ajc;
  }
}

// Strain tensor {Sxx, Sxy, Sxz, Syy, Syz, Szz} and |S| (les.c:209-213).
__device__ __forceinline__ double strain(const double o[9], double s[6]) {
  s[0] = 0.5 * (o[0] + o[0]);
  s[1] = 0.5 * (o[1] + o[3]);
  s[2] = 0.5 * (o[2] + o[6]);
  s[3] = 0.5 * (o[4] + o[4]);
  s[4] = 0.5 * (o[5] + o[7]);
  s[5] = 0.5 * (o[8] + o[8]);
  return sqrt(2.0 * (s[0] * s[0] + s[1] * s[1] + s[2] * s[2] + s[1] * s[1] + s[3] * s[3] + s[4] * s[4] +
                     s[2] * s[2] + s[4] * s[4] + s[5] * s[5]));
}

// ------------------------------------------------------------------ test filter
// A block of FTX x FTY interior cells marches through `kz` planes along k.  Every plane of
// the tile and its one-cell rim is formed once (load: value x weight of NQ quantities at a
// point), filtered along i and j through shared memory and along k in two running sums per
// quantity and cell; emit gets the filtered sums of each cell.  15 quantities from 13
// fields: bound by shared-memory traffic (six 8-byte accesses per quantity and cell, where
// summing the sub-cubes as written took about ninety).
constexpr int FTX = 32, FTY = 8, FRX = FTX + 2, FRY = FTY + 2;
constexpr int kFilterThreads = FTX * FTY;
template <int NQ>
constexpr size_t filter_smem() { return sizeof(double) * NQ * (FRX * FRY + FTX * FRY); }

template <int NQ, class Load, class Emit>
__device__ __forceinline__ void box_filter(const Grid &g, int kz, const Load &load, const Emit &emit) {
  extern __shared__ __align__(16) double les_sm[];
  double *raw = les_sm, *fi = les_sm + NQ * FRX * FRY;  // the plane, and the plane filtered along i
  const int i0 = 1 + blockIdx.x * FTX, j0 = 1 + blockIdx.y * FTY;
  const int k0 = 1 + blockIdx.z * kz, k1 = min(k0 + kz, g.mz - 1);  // cells k0 .. k1-1
  const int tx = threadIdx.x % FTX, ty = threadIdx.x / FTX;
  const int i = i0 + tx, j = j0 + ty;
  const bool cell = i <= g.mx - 2 && j <= g.my - 2;
  double a[NQ], b[NQ];
#pragma unroll
  for (int q = 0; q < NQ; q++) a[q] = b[q] = 0;
  for (int k = k0 - 1; k <= k1; k++) {
    for (int t = threadIdx.x; t < FRX * FRY; t += kFilterThreads) {
      const int pi = i0 - 1 + t % FRX, pj = j0 - 1 + t / FRX;
      double v[NQ];
#pragma unroll
      for (int q = 0; q < NQ; q++) v[q] = 0;
      if (pi < g.mx && pj < g.my) load(pi, pj, k, lidx(g, pi, pj, k), v);
#pragma unroll
      for (int q = 0; q < NQ; q++) raw[q * (FRX * FRY) + t] = v[q];
    }
    __syncthreads();
    for (int t = threadIdx.x; t < FTX * FRY; t += kFilterThreads) {
      const int c = (t / FTX) * FRX + t % FTX + 1;
#pragma unroll
      for (int q = 0; q < NQ; q++) {
        const double *r = raw + q * (FRX * FRY) + c;
        fi[q * (FTX * FRY) + t] = r[-1] + 2.0 * r[0] + r[1];
      }
    }
    __syncthreads();  // also orders the next plane's writes of raw after this plane's reads
    double f[NQ];
#pragma unroll
    for (int q = 0; q < NQ; q++) {
      const double *r = fi + q * (FTX * FRY) + (ty + 1) * FTX + tx;
      const double v = r[-FTX] + 2.0 * r[0] + r[FTX];
      f[q] = a[q] + v;
      a[q] = b[q] + 2.0 * v;
      b[q] = v;
    }
    if (k > k0 && cell) emit(i, j, k - 1, lidx(g, i, j, k - 1), f);
  }
}
// Planes a block marches through: as many as leave two blocks per SM, at most 16.
static dim3 filter_grid(const Grid &g, int &kz) {
  const unsigned bx = (g.mx - 2 + FTX - 1) / FTX, by = (g.my - 2 + FTY - 1) / FTY;
  kz = 16;
  while (kz > 2 && (unsigned long long)bx * by * ((g.mz - 2 + kz - 1) / kz) < 2 * 148) kz /= 2;
  return dim3(bx, by, (g.mz - 2 + kz - 1) / kz);
}

// Ghost points of n arrays: the value of the periodic image where that is an interior cell,
// 0 elsewhere.
struct LesArrays {
  int n;
  double *a[9];
};
__global__ void __launch_bounds__(256) k_les_ghosts(Grid g, LesArrays o) {
  long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  const long long ni = 2LL * g.my * g.mz, nj = 2LL * g.mx * g.mz, nk = 2LL * g.mx * g.my;
  int i, j, k;
  if (t < ni) {
    const long long r = t >> 1;
    i = (t & 1) ? g.mx - 1 : 0; j = (int)(r % g.my); k = (int)(r / g.my);
  } else if ((t -= ni) < nj) {
    const long long r = t >> 1;
    j = (t & 1) ? g.my - 1 : 0; i = (int)(r % g.mx); k = (int)(r / g.mx);
  } else if ((t -= nj) < nk) {
    const long long r = t >> 1;
    k = (t & 1) ? g.mz - 1 : 0; i = (int)(r % g.mx); j = (int)(r / g.mx);
  } else {
    return;
  }
  const int ii = wrapi(g, i), jj = wrapj(g, j), kk = wrapk(g, k);
  const long long p = lidx(g, i, j, k), s = lidx(g, ii, jj, kk);
  const bool in = les_interior(g, ii, jj, kk);
  for (int q = 0; q < o.n; q++) o.a[q][p] = in ? o.a[q][s] : 0.0;
}
static int les_ghosts(Ctx *c, const LesArrays &o) {
  const Grid &g = c->g;
  const long long n = 2LL * g.my * g.mz + 2LL * g.mx * g.mz + 2LL * g.mx * g.my;
  c->launches++, k_les_ghosts<<<nblocks(n, 256), 256, 0, c->stream>>>(g, o);
  return check_launch(c, "k_les_ghosts");
}

struct LesPrep {
  double *U, *V, *W;   // contravariant centre velocity (own point)
  double *wgt;         // 0 where nvert > 1.1, else 1/aj (own point)
  double *ss[6];       // S_ab*|S| of the interior cells (zero at solid ones); ghosts by k_les_ghosts
  double *uf[3];       // test-filtered velocity, the same way
};

// ------------------------------------------------------------------ k_les_prep
// Own-point quantities of every DA point: U, V, W and the test-filter weight.
__global__ void k_les_prep(Grid g, CV3 u, CV3 csi, CV3 eta, CV3 zet, const double *__restrict__ aj,
                           const uint8_t *__restrict__ nv, LesPrep o) {
  const long long p = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (p >= g.N) return;
  const double ux = u.x[p], uy = u.y[p], uz = u.z[p];
  o.U[p] = ux * csi.x[p] + uy * csi.y[p] + uz * csi.z[p];
  o.V[p] = ux * eta.x[p] + uy * eta.y[p] + uz * eta.z[p];
  o.W[p] = ux * zet.x[p] + uy * zet.y[p] + uz * zet.z[p];
  o.wgt[p] = (nv[p] > 1) ? 0.0 : 1. / aj[p];  // get_weight, les.c:31-32
}

// Strain products S_ab |S| and the test-filtered velocity of the interior cells (les.c:191-238);
// zero at solid cells.
__global__ void __launch_bounds__(kFilterThreads, 2) k_les_image(Grid g, int kz, CV3 u, CV3 csi, CV3 eta, CV3 zet,
                                                                 const double *__restrict__ aj,
                                                                 const uint8_t *__restrict__ nv, LesPrep o) {
  box_filter<4>(
      g, kz,
      [&](int, int, int, long long p, double *v) {
        const double w = o.wgt[p];
        v[0] = w; v[1] = u.x[p] * w; v[2] = u.y[p] * w; v[3] = u.z[p] * w;
      },
      [&](int i, int j, int k, long long p, const double *f) {
        double ss[6] = {0, 0, 0, 0, 0, 0}, uf[3] = {0, 0, 0};
        if (nv[p] <= 1) {
          double d[9], gr[9], st[6];
          du_center(g, u, nv, p, i, j, k, d);
          const double cc[3] = {csi.x[p], csi.y[p], csi.z[p]};
          const double ee[3] = {eta.x[p], eta.y[p], eta.z[p]};
          const double zz[3] = {zet.x[p], zet.y[p], zet.z[p]};
          du_dxyz(cc, ee, zz, aj[p], d, gr);
          const double sabs = strain(gr, st);
#pragma unroll
          for (int t = 0; t < 6; t++) ss[t] = st[t] * sabs;
          uf[0] = f[1] / f[0]; uf[1] = f[2] / f[0]; uf[2] = f[3] / f[0];
        }
#pragma unroll
        for (int t = 0; t < 6; t++) o.ss[t][p] = ss[t];
        o.uf[0][p] = uf[0]; o.uf[1][p] = uf[1]; o.uf[2][p] = uf[2];
      });
}

// ------------------------------------------------------------------ k_les_lm
struct LesLmIn {
  CV3 u;
  const double *U, *V, *W, *wgt, *ss[6];
  CV3 uf;
};

// Calculate_Covariant_metrics (rhs2.c:538-554): inverse of the centre metric matrix.
__device__ __forceinline__ void covariant(const double a[3][3], double G[3][3]) {
  const double a11 = a[0][0], a12 = a[0][1], a13 = a[0][2];
  const double a21 = a[1][0], a22 = a[1][1], a23 = a[1][2];
  const double a31 = a[2][0], a32 = a[2][1], a33 = a[2][2];
  const double det = a11 * (a33 * a22 - a32 * a23) - a21 * (a33 * a12 - a32 * a13) + a31 * (a23 * a12 - a22 * a13);
  G[0][0] = (a33 * a22 - a32 * a23) / det; G[0][1] = -(a33 * a12 - a32 * a13) / det; G[0][2] = (a23 * a12 - a22 * a13) / det;
  G[1][0] = -(a33 * a21 - a31 * a23) / det; G[1][1] = (a33 * a11 - a31 * a13) / det; G[1][2] = -(a23 * a11 - a21 * a13) / det;
  G[2][0] = (a32 * a21 - a31 * a22) / det; G[2][1] = -(a32 * a11 - a31 * a12) / det; G[2][2] = (a22 * a11 - a21 * a12) / det;
}

// The contractions at one cell from its 15 test-filtered quantities F: U u, U v, ..., W w
// (les.c:381-391), then the six S_ab |S| (les.c:428-430); wsum is the filter's weight sum.
__device__ __forceinline__ void lm_cell(const Grid &g, const LesLmIn &in, CV3 csi, CV3 eta, CV3 zet,
                                        const double *__restrict__ aj, const uint8_t *__restrict__ nv, long long p,
                                        int i, int j, int k, const double *F, double wsum, double &lm, double &mm) {
  const double cc[3] = {csi.x[p], csi.y[p], csi.z[p]};
  const double ee[3] = {eta.x[p], eta.y[p], eta.z[p]};
  const double zz[3] = {zet.x[p], zet.y[p], zet.z[p]};
  const double ajc = aj[p];
  const double filter = cbrt(1. / ajc);
  const double test_filter = cbrt(0.125 * wsum);  // the (1/2 1 1/2)^3 sum of the weights (les.c:433-452)
  // filtered velocity at the cell and its contravariant components (les.c:470-475)
  const double fu = in.uf.x[p], fv = in.uf.y[p], fw = in.uf.z[p];
  const double fU = fu * cc[0] + fv * cc[1] + fw * cc[2];
  const double fV = fu * ee[0] + fv * ee[1] + fw * ee[2];
  const double fW = fu * zz[0] + fv * zz[1] + fw * zz[2];
  double d[9], gr[9], sh[6];
  du_center(g, in.uf, nv, p, i, j, k, d);
  du_dxyz(cc, ee, zz, ajc, d, gr);
  const double S_hat = strain(gr, sh);
  const double Sij[3][3] = {{sh[0], sh[1], sh[2]}, {sh[1], sh[3], sh[4]}, {sh[2], sh[4], sh[5]}};
  const double Lij[3][3] = {{F[0] - fU * fu, F[1] - fU * fv, F[2] - fU * fw},
                            {F[3] - fV * fu, F[4] - fV * fv, F[5] - fV * fw},
                            {F[6] - fW * fu, F[7] - fW * fv, F[8] - fW * fw}};
  const double SSij[3][3] = {{F[9], F[10], F[11]}, {F[10], F[12], F[13]}, {F[11], F[13], F[14]}};
  const double gg[3][3] = {{cc[0], cc[1], cc[2]}, {ee[0], ee[1], ee[2]}, {zz[0], zz[1], zz[2]}};
  double ggc[3][3];
  covariant(gg, ggc);
  const double xcsi = ggc[0][0], xeta = ggc[0][1], xzet = ggc[0][2];
  const double ycsi = ggc[1][0], yeta = ggc[1][1], yzet = ggc[1][2];
  const double zcsi = ggc[2][0], zeta = ggc[2][1], zzet = ggc[2][2];
  double G[3][3];
  G[0][0] = xcsi * xcsi + ycsi * ycsi + zcsi * zcsi;
  G[1][1] = xeta * xeta + yeta * yeta + zeta * zeta;
  G[2][2] = xzet * xzet + yzet * yzet + zzet * zzet;
  G[0][1] = G[1][0] = xeta * xcsi + yeta * ycsi + zeta * zcsi;
  G[0][2] = G[2][0] = xzet * xcsi + yzet * ycsi + zzet * zcsi;
  G[1][2] = G[2][1] = xeta * xzet + yeta * yzet + zeta * zzet;
  // Mij (les.c:616-633)
  const double tA = -(test_filter * test_filter) * S_hat;
  const double fB = filter * filter;
  double Mc[3][3], M[3][3];
#pragma unroll
  for (int a = 0; a < 3; a++)
#pragma unroll
    for (int b = 0; b < 3; b++) Mc[a][b] = tA * Sij[a][b] + fB * SSij[a][b];
#pragma unroll
  for (int a = 0; a < 3; a++) {
    M[a][0] = Mc[a][0] * cc[0] + Mc[a][1] * cc[1] + Mc[a][2] * cc[2];
    M[a][1] = Mc[a][0] * ee[0] + Mc[a][1] * ee[1] + Mc[a][2] * ee[2];
    M[a][2] = Mc[a][0] * zz[0] + Mc[a][1] * zz[1] + Mc[a][2] * zz[2];
  }
  double num = 0, denom = 0;
#pragma unroll
  for (int q = 0; q < 3; q++)
#pragma unroll
    for (int a = 0; a < 3; a++)
#pragma unroll
      for (int b = 0; b < 3; b++) num += Lij[b][a] * M[a][q] * G[b][q];
#pragma unroll
  for (int m = 0; m < 3; m++)
#pragma unroll
    for (int n = 0; n < 3; n++)
#pragma unroll
      for (int l = 0; l < 3; l++) denom += M[n][m] * M[n][l] * G[m][l];
  lm = num;
  mm = denom;
}


__global__ void __launch_bounds__(kFilterThreads, 2)
    k_les_lm(Grid g, int kz, LesLmIn in, CV3 csi, CV3 eta, CV3 zet, const double *__restrict__ aj,
             const uint8_t *__restrict__ nv, double *LM, double *MM) {
  box_filter<16>(
      g, kz,
      [&](int, int, int, long long p, double *v) {
        const double w = in.wgt[p];
        const double u = in.u.x[p] * w, vv = in.u.y[p] * w, ww = in.u.z[p] * w;
        const double U = in.U[p], V = in.V[p], W = in.W[p];
        v[0] = U * u; v[1] = U * vv; v[2] = U * ww;
        v[3] = V * u; v[4] = V * vv; v[5] = V * ww;
        v[6] = W * u; v[7] = W * vv; v[8] = W * ww;
#pragma unroll
        for (int q = 0; q < 6; q++) v[9 + q] = in.ss[q][p] * w;
        v[15] = w;
      },
      [&](int i, int j, int k, long long p, double *f) {
        double lm = 0, mm = 0;
        if (nv[p] <= 1) {
          const double wsum = f[15];
#pragma unroll
          for (int q = 0; q < 15; q++) f[q] = f[q] / wsum;
          lm_cell(g, in, csi, eta, zet, aj, nv, p, i, j, k, f, wsum, lm, mm);
        }
        LM[p] = lm;
        MM[p] = mm;
      });
}

// Test-filter weight of a point in the Cs averaging and re-filtering loops (les.c:720-762,
// les.c:1069-1110): 1/aj (0 where nvert > 1.1), zero at non-periodic boundary points; the
// value of a periodic ghost point is its image's, which the ghosts of the filtered fields
// hold.  In the j direction the reference tests the cell's own j against my-1 (les.c:748,
// les.c:1097), so only J == 0 is zeroed; that test is kept.
__device__ __forceinline__ double wrap_weight(const Grid &g, const double *__restrict__ wgt, long long p, int i,
                                              int j, int k) {
  if (!g.iper && (i == 0 || i == g.mx - 1)) return 0.0;
  if (!g.jper && j == 0) return 0.0;
  if (!g.kper && (k == 0 || k == g.mz - 1)) return 0.0;
  return wgt[p];
}

// Clipped Cs of the interior cells (les.c:708-788 with les = 2, then les.c:959-972).
__global__ void __launch_bounds__(kFilterThreads, 3) k_les_cs(Grid g, int kz, const double *__restrict__ wgt,
                                                              const uint8_t *__restrict__ nv,
                                                              const double *__restrict__ LM,
                                                              const double *__restrict__ MM, double max_cs, double *out) {
  box_filter<3>(
      g, kz,
      [&](int i, int j, int k, long long p, double *v) {
        const double w = wrap_weight(g, wgt, p, i, j, k);
        v[0] = w; v[1] = LM[p] * w; v[2] = MM[p] * w;
      },
      [&](int, int, int, long long p, const double *f) {
        double cs = 0;
        if (nv[p] <= 1) {
          const double LM_avg = f[1] / f[0], MM_avg = f[2] / f[0];
          const double C = 0.5 * LM_avg / (MM_avg + kLesEps);
          cs = (C < 0) ? 0 : C;                                // PetscMax(C, 0)
          if (nv[p] == 1) cs = (kWallCs < cs) ? cs : kWallCs;  // PetscMax(wall_cs, Cs) at IB nodes
          cs = (cs < 0) ? 0 : cs;
          cs = (cs < max_cs) ? cs : max_cs;                    // PetscMin(PetscMax(Cs, 0), max_cs)
        }
        out[p] = cs;
      });
}

// Second filtering of Cs over fluid cells (nvert < 0.1); every other interior cell keeps its
// value (k_les_keep: the ghost points).
__global__ void __launch_bounds__(kFilterThreads, 3) k_les_refilter(Grid g, int kz, const double *__restrict__ wgt,
                                                                    const uint8_t *__restrict__ nv,
                                                                    const double *__restrict__ cs_tmp, double *cs) {
  box_filter<2>(
      g, kz,
      [&](int i, int j, int k, long long p, double *v) {
        const double w = wrap_weight(g, wgt, p, i, j, k);
        v[0] = w; v[1] = cs_tmp[p] * w;
      },
      [&](int, int, int, long long p, const double *f) { cs[p] = nv[p] != 0 ? cs_tmp[p] : f[1] / f[0]; });
}
__global__ void __launch_bounds__(256) k_les_keep(Grid g, const double *__restrict__ from, double *to) {
  long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  const long long ni = 2LL * g.my * g.mz, nj = 2LL * g.mx * g.mz, nk = 2LL * g.mx * g.my;
  int i, j, k;
  if (t < ni) {
    const long long r = t >> 1;
    i = (t & 1) ? g.mx - 1 : 0; j = (int)(r % g.my); k = (int)(r / g.my);
  } else if ((t -= ni) < nj) {
    const long long r = t >> 1;
    j = (t & 1) ? g.my - 1 : 0; i = (int)(r % g.mx); k = (int)(r / g.mx);
  } else if ((t -= nj) < nk) {
    const long long r = t >> 1;
    k = (t & 1) ? g.mz - 1 : 0; i = (int)(r % g.mx); j = (int)(r / g.mx);
  } else {
    return;
  }
  const long long p = lidx(g, i, j, k);
  to[p] = from[p];
}

// nu_t of one interior cell (les.c:1177-1198).
__device__ __forceinline__ double nut_cell(const Grid &g, CV3 u, CV3 csi, CV3 eta, CV3 zet,
                                           const double *__restrict__ aj, const uint8_t *__restrict__ nv,
                                           const double *__restrict__ cs, int i, int j, int k) {
  const long long p = lidx(g, i, j, k);
  if (nv[p] > 1) return 0.0;
  double d[9], gr[9], s[6];
  du_center(g, u, nv, p, i, j, k, d);
  const double cc[3] = {csi.x[p], csi.y[p], csi.z[p]};
  const double ee[3] = {eta.x[p], eta.y[p], eta.z[p]};
  const double zz[3] = {zet.x[p], zet.y[p], zet.z[p]};
  du_dxyz(cc, ee, zz, aj[p], d, gr);
  const double sabs = strain(gr, s);
  const double filter = cbrt(1. / aj[p]);
  return cs[p] * (filter * filter) * sabs;
}

// Interior cells and periodic ghosts (value of the image; the old value of the image when
// the image is a non-periodic boundary point); other ghosts keep their value.
__global__ void k_les_nut(Grid g, CV3 u, CV3 csi, CV3 eta, CV3 zet, const double *__restrict__ aj,
                          const uint8_t *__restrict__ nv, const double *__restrict__ cs, double *nut) {
  const long long p = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (p >= g.N) return;
  int i, j, k;
  dijk(g, p, i, j, k);
  const int a = wrapi(g, i), b = wrapj(g, j), c = wrapk(g, k);
  if (les_interior(g, a, b, c)) nut[p] = nut_cell(g, u, csi, eta, zet, aj, nv, cs, a, b, c);
  else if (a != i || b != j || c != k) nut[p] = nut[lidx(g, a, b, c)];
}

__global__ void k_fill(long long n, double v, double *a) {
  const long long p = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (p < n) a[p] = v;
}

// ------------------------------------------------------------------ host side
// Scratch: the Formfunction_2 face-flux arrays, idle while the eddy viscosity is formed
// (Flow_Solver computes it before the momentum step, solvers.c:648-654).
static LesPrep les_scratch(Ctx *c, double **LM, double **MM, double **cs_tmp) {
  LesPrep o;
  o.U = c->div[0][0]; o.V = c->div[0][1]; o.W = c->div[0][2];
  o.wgt = c->div[1][0];
  o.ss[0] = c->div[1][1]; o.ss[1] = c->div[1][2]; o.ss[2] = c->div[2][0];
  o.ss[3] = c->div[2][1]; o.ss[4] = c->div[2][2]; o.ss[5] = c->visc[0][0];
  o.uf[0] = c->visc[0][1]; o.uf[1] = c->visc[0][2]; o.uf[2] = c->visc[1][0];
  *LM = c->visc[1][1]; *MM = c->visc[1][2]; *cs_tmp = c->visc[2][0];
  return o;
}

int smagorinsky_constant(Ctx *c) {
  const Grid &g = c->g;
  double *cs = c->f[VFS_CS][0];
  int rc;
  if (c->ti < 2 && c->tistart == 0 && !c->rstart) {  // les.c:69-72
    cudaMemsetAsync(cs, 0, sizeof(double) * (size_t)g.N, c->stream);
    return VFS_OK;
  }
  if (g.les == 1) {  // les.c:74-77
    c->launches++, k_fill<<<nblocks(g.N, 256), 256, 0, c->stream>>>(g.N, 0.01, cs);
    return check_launch(c, "k_fill");
  }
  Metrics m = metrics(c);
  double *LM, *MM, *cs_tmp;
  LesPrep o = les_scratch(c, &LM, &MM, &cs_tmp);
  CV3 u = cv(field3(c, VFS_UCAT));
  c->launches++, k_les_prep<<<nblocks(g.N, 256), 256, 0, c->stream>>>(g, u, m.csi, m.eta, m.zet, m.aj, c->nv, o);
  if ((rc = check_launch(c, "k_les_prep"))) return rc;
  // the shared-memory limit is an attribute of the kernel on a device
  if (cudaFuncSetAttribute(k_les_lm, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)filter_smem<16>()) != cudaSuccess)
    return set_err(c, VFS_ERR_CUDA, "k_les_lm: shared-memory limit");
  int kz;
  const dim3 grid = filter_grid(g, kz);
  c->launches++, k_les_image<<<grid, kFilterThreads, filter_smem<4>(), c->stream>>>(g, kz, u, m.csi, m.eta, m.zet, m.aj, c->nv, o);
  if ((rc = check_launch(c, "k_les_image"))) return rc;
  if ((rc = les_ghosts(c, LesArrays{9, {o.ss[0], o.ss[1], o.ss[2], o.ss[3], o.ss[4], o.ss[5], o.uf[0], o.uf[1], o.uf[2]}}))) return rc;
  LesLmIn in;
  in.u = u;
  in.U = o.U; in.V = o.V; in.W = o.W; in.wgt = o.wgt;
  for (int q = 0; q < 6; q++) in.ss[q] = o.ss[q];
  in.uf = CV3{o.uf[0], o.uf[1], o.uf[2]};
  c->launches++, k_les_lm<<<grid, kFilterThreads, filter_smem<16>(), c->stream>>>(g, kz, in, m.csi, m.eta, m.zet, m.aj, c->nv, LM, MM);
  if ((rc = check_launch(c, "k_les_lm"))) return rc;
  if ((rc = les_ghosts(c, LesArrays{2, {LM, MM}}))) return rc;
  c->launches++, k_les_cs<<<grid, kFilterThreads, filter_smem<3>(), c->stream>>>(g, kz, o.wgt, c->nv, LM, MM, c->max_cs, cs_tmp);
  if ((rc = check_launch(c, "k_les_cs"))) return rc;
  if ((rc = les_ghosts(c, LesArrays{1, {cs_tmp}}))) return rc;
  c->launches++, k_les_refilter<<<grid, kFilterThreads, filter_smem<2>(), c->stream>>>(g, kz, o.wgt, c->nv, cs_tmp, cs);
  const long long ng = 2LL * g.my * g.mz + 2LL * g.mx * g.mz + 2LL * g.mx * g.my;
  c->launches++, k_les_keep<<<nblocks(ng, 256), 256, 0, c->stream>>>(g, cs_tmp, cs);
  return check_launch(c, "k_les_refilter");
}

int eddy_viscosity(Ctx *c) {
  const Grid &g = c->g;
  Metrics m = metrics(c);
  c->launches++, k_les_nut<<<nblocks(g.N, 256), 256, 0, c->stream>>>(g, cv(field3(c, VFS_UCAT)), m.csi, m.eta, m.zet, m.aj, c->nv,
                                                     c->f[VFS_CS][0], c->f[VFS_NU_T][0]);
  return check_launch(c, "k_les_nut");
}

}  // namespace vfs

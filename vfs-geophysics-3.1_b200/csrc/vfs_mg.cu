// Geometric multigrid preconditioner of the pressure-Poisson solve (one V-cycle per
// FGMRES iteration), FP32 or FP64.
//
// The reference preconditions its Krylov solve with HYPRE BoomerAMG
// (poisson_hypre.c:26-88); this is a B200-first geometric replacement, not a port:
//
//   * Levels are cell-centred and coarsened by 2 in every direction while all interior
//     dimensions are even and at least 4 (256x192x256 -> ... -> 4x3x4: seven levels).
//   * Every level, the finest included, smooths with the 7-point conductance form of the
//     operator: the coupling of two unknowns across a face is the symmetrised, clipped
//     main-term coefficient of the reference's 19-point row (exactly the operator on
//     orthogonal grids, where the reference's filter drops every cross term).  A coarse
//     face conducts 0.5 x the sum of the four fine faces it covers; diagonals are minus
//     the sum of a cell's couplings, so every level is a consistent Neumann operator.
//   * Smoother: line Gauss-Seidel along j (the wall-normal, most strongly coupled
//     direction of the channel grids) in zebra order: the columns with (i+k) even are
//     solved first, then the odd ones, so each column's i/k neighbours are fixed while it
//     is solved and the update is in place and deterministic.  The tridiagonal factors
//     (Thomas forward coefficients and pivots) are precomputed once per operator.
//   * Restriction sums the residuals of the 8 children; prolongation is cell-centred
//     trilinear (weights 27/64, 9/64, 3/64, 1/64), a missing or inactive coarse
//     neighbour giving its weight to the parent.  With these transfers the FGMRES
//     iteration count stays flat as the grid is refined.
//
// Layout: every level stores its cells column by column (struct ZL): the ny rows of an (i, k)
// column are contiguous and lane-interleaved, the columns of one colour of a k plane are
// neighbours.  A group of lw lanes solves a column on its own, every lane seg consecutive
// rows in registers: all loads of a column are coalesced and in flight together, the two
// recurrences are a warp scan each, and there is neither shared memory nor a block barrier.
// The i/k neighbours of a row sit at the same slot of the neighbour column.  The finest level's
// right-hand side and solution are transposed from and to the solver's grid vectors once per
// V-cycle through shared memory.
//
// The FP32 V-cycle's rounding reaches the solution: a mixed solve stops at its tolerance, and
// where the operator is nearly singular (channels without bodies) the last digits it leaves
// (1e-8 of the pressure at rtol 1e-10) follow that rounding.  So the order of the operations
// of a level is fixed: 32 lanes of ceil(ny/32) rows, levels of at most kSerialCells cells (and
// coarse line Jacobi) by Thomas' recurrence row by row, no fused multiply-adds.
//
// One V-cycle on the B200, the tiled line sweeps with block barriers of before against the
// columns (us, FP32 / FP64): 256 x 192 x 256 cells 1409 / 2214 -> 830 / 1481 (a colour pass of
// the finest level 68 -> 42 FP32), 128 x 96 x 128 392 / 486 -> 197 / 297, 64^3 256 / 249 -> 119 / 127.
//
// A level with an odd number of cells along a periodic i or k direction cannot be two-
// coloured; it is smoothed by damped (0.8) line Jacobi instead.
#include <algorithm>
#include <cmath>

#include "vfs_internal.cuh"

namespace vfs {

enum { OP_CE = 0, OP_CN, OP_CT, OP_DG, OP_CPR, OP_IDEN, NOP };

// Cell (i, j, k) of slot q of a level; false for a slot that holds no cell.
__device__ __forceinline__ bool zcell(const ZL &L, unsigned q, int &i, int &j, int &k) {
  const unsigned col = q / (unsigned)L.S, pos = q - col * (unsigned)L.S;
  j = zrow_of(L, pos);
  const unsigned ck = col / (unsigned)L.hx, h = col - ck * (unsigned)L.hx;
  k = (int)(ck >> 1);
  i = (int)(2 * h + ((ck & 1) ^ (unsigned)(k & 1)));
  return j < L.ny && i < L.nx;
}

// ------------------------------------------------------------------ set-up (FP64)
// Fine-level couplings from the reference operator (19 slots on the DA layout): the coupling of
// cell (i, j, k) to its +i (q = 0), +j (1) or +k (2) neighbour.
__device__ __forceinline__ double fine_coupling(const Grid &g, const ZL &L, const double *__restrict__ coef,
                                                const uint8_t *__restrict__ fluid, int q, int i, int j, int k) {
  const long long N = vec_ld(g.N), p = lidx(g, i + 1, j + 1, k + 1);
  // every load is issued before the first is tested
  const long long e = q == 0 ? lidx(g, wrapi(g, i + 2), j + 1, k + 1)
                             : (q == 1 ? lidx(g, i + 1, wrapj(g, j + 2), k + 1) : lidx(g, i + 1, j + 1, wrapk(g, k + 2)));
  const double c = coef[(q == 0 ? EP : (q == 1 ? NP : TP)) * N + p], d = coef[(q == 0 ? WP : (q == 1 ? SP : BP)) * N + e];
  const bool f = fluid[p] && fluid[e];
  const bool has = q == 0 ? i + 1 < L.nx || L.ip : (q == 1 ? j + 1 < L.ny || L.jp : k + 1 < L.nz || L.kp);
  return f && has ? fmax(0.0, 0.5 * (c + d)) : 0.0;
}

// A block moves kTileI consecutive i of one k plane and all rows through shared memory, so that
// both the grid arrays and the columns are accessed in runs.  Columns too long for that go directly.
constexpr int kTileI = 16;
constexpr size_t kTileSmem = 200 * 1024;
template <typename T>
__host__ __device__ inline size_t tile_bytes(const ZL &L) { return sizeof(T) * kTileI * ((size_t)L.S | 1); }
__host__ __device__ inline unsigned tiles_i(const ZL &L) { return (unsigned)(L.nx + kTileI - 1) / kTileI; }

// One direction after the other through the same tile.  Bound by the latency of the loads between the
// barriers.  (A thread per slot, in column order, read the coefficients a grid row apart: 444 us at
// 256 x 192 x 256 cells against 286, 55 at 128 x 96 x 128 against 34; tiles of 32 i 361 and 50.)
__global__ void __launch_bounds__(256) k_mg_fine_couplings(Grid g, ZL L, const double *__restrict__ coef,
                                                           const uint8_t *__restrict__ fluid, double *__restrict__ op) {
  extern __shared__ __align__(16) unsigned char fine_raw[];
  double *sm = reinterpret_cast<double *>(fine_raw);
  const unsigned ib = tiles_i(L);
  const int k = (int)(blockIdx.x / ib), i0 = (int)(blockIdx.x % ib) * kTileI, ld = L.S | 1;
  const int a = threadIdx.x % kTileI;
#pragma unroll
  for (int q = 0; q < 3; q++) {
#pragma unroll 2
    for (int j = threadIdx.x / kTileI; j < L.S; j += 256 / kTileI)  // rows past ny: the empty slots
      sm[a * ld + (int)zrow(L, j)] =
          j < L.ny && i0 + a < L.nx ? fine_coupling(g, L, coef, fluid, q, i0 + a, j, k) : 0.0;
    __syncthreads();
    for (int c = threadIdx.x >> 5; c < kTileI && i0 + c < L.nx; c += 8) {  // a warp a column
      const unsigned p0 = zcol(L, i0 + c, k);
      for (int s = threadIdx.x & 31; s < L.S; s += 32) op[(OP_CE + q) * L.n + p0 + s] = sm[c * ld + s];
    }
    __syncthreads();
  }
}
__global__ void k_mg_fine_couplings_direct(Grid g, ZL L, const double *__restrict__ coef,
                                           const uint8_t *__restrict__ fluid, double *__restrict__ op) {
  const long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  int i, j, k;
  if (t >= L.n || !zcell(L, (unsigned)t, i, j, k)) return;
  for (int q = 0; q < 3; q++) op[(OP_CE + q) * L.n + t] = fine_coupling(g, L, coef, fluid, q, i, j, k);
}

// Coarse couplings: 0.5 x the sum of the four fine couplings across each coarse face.
__global__ void k_mg_coarse_couplings(ZL F, ZL C, const double *__restrict__ opF, double *__restrict__ opC) {
  const long long q = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  int I, J, K;
  if (q >= C.n || !zcell(C, (unsigned)q, I, J, K)) return;
  double sx = 0, sy = 0, sz = 0;
  for (int u = 0; u < 2; u++)
    for (int v = 0; v < 2; v++) {
      sx += opF[OP_CE * F.n + zidx(F, 2 * I + 1, 2 * J + u, 2 * K + v)];
      sy += opF[OP_CN * F.n + zidx(F, 2 * I + u, 2 * J + 1, 2 * K + v)];
      sz += opF[OP_CT * F.n + zidx(F, 2 * I + u, 2 * J + v, 2 * K + 1)];
    }
  opC[OP_CE * C.n + q] = 0.5 * sx;
  opC[OP_CN * C.n + q] = 0.5 * sy;
  opC[OP_CT * C.n + q] = 0.5 * sz;
}

// Neighbour cells of (i,j,k) with the level's periodic wrap; -1 where there is none.
struct ZNb {
  int ie, iw, jn, js, kt, kb;
};
__device__ __forceinline__ ZNb znb(const ZL &L, int i, int j, int k) {
  ZNb r;
  r.ie = i + 1 < L.nx ? i + 1 : (L.ip ? 0 : -1);
  r.iw = i > 0 ? i - 1 : (L.ip ? L.nx - 1 : -1);
  r.jn = j + 1 < L.ny ? j + 1 : (L.jp ? 0 : -1);
  r.js = j > 0 ? j - 1 : (L.jp ? L.ny - 1 : -1);
  r.kt = k + 1 < L.nz ? k + 1 : (L.kp ? 0 : -1);
  r.kb = k > 0 ? k - 1 : (L.kp ? L.nz - 1 : -1);
  return r;
}

// The diagonal, and act[q] = 1 where it is non-zero (an active unknown).
__global__ void k_mg_diag(ZL L, double *__restrict__ op, uint8_t *__restrict__ act) {
  const long long q = blockIdx.x * (long long)blockDim.x + threadIdx.x, n = L.n;
  int i, j, k;
  if (q >= n) return;
  if (!zcell(L, (unsigned)q, i, j, k)) { act[q] = 0; return; }
  const ZNb b = znb(L, i, j, k);
  const unsigned p0 = zcol(L, i, k), pos = (unsigned)q - p0;  // a column neighbour's cell has the same slot
  double s = op[OP_CE * n + q] + op[OP_CN * n + q] + op[OP_CT * n + q];
  if (b.iw >= 0) s += op[OP_CE * n + zcol(L, b.iw, k) + pos];
  if (b.js >= 0) s += op[OP_CN * n + p0 + zrow(L, b.js)];
  if (b.kb >= 0) s += op[OP_CT * n + zcol(L, i, b.kb) + pos];
  op[OP_DG * n + q] = -s;
  act[q] = s != 0.0 ? 1 : 0;
}

// Thomas factors of every j-line (the in-line couplings only; a periodic j wrap is left
// to the right-hand side): cpr_j = upper_j / den_j, iden_j = 1 / den_j,
// den_j = dg_j - lower_j * cpr_{j-1}.  Inactive or degenerate rows get zero factors, so
// the smoother leaves their unknown at zero.
struct Thomas {
  double cprev = 0, lower = 0;
  // dg and upper of the row in, iden and cpr out
  __device__ __forceinline__ void row(double &dg, double &upper) {
    const double up = upper;
    double cpr = 0, iden = 0;
    if (dg != 0) {
      const double den = dg - lower * cprev;
      if (fabs(den) > 1e-12 * fabs(dg)) {
        iden = 1.0 / den;
        cpr = up * iden;
      }
    }
    dg = iden;
    upper = cpr;
    cprev = cpr;
    lower = up;
  }
};
// A block stages `cols` columns in shared memory (dg and upper, replaced by iden and cpr), one
// thread a column runs the recurrence there: its rows are not neighbours in the column's slots, and
// straight from global memory every load was a sector of its own.  Bound by the chain of divisions of a
// row.  All levels of 256 x 192 x 256 cells 1410 -> 271 us (32 columns a block 329), 64 x 48 x 64 37 -> 22.
constexpr int kThomasThreads = 256;
constexpr size_t kThomasSmem = 200 * 1024;
static size_t thomas_smem(const ZL &L, int cols) { return sizeof(double) * 2 * cols * ((size_t)L.ny | 1); }
// Columns a block: 16, fewer where they are long (0: one does not fit).
static int thomas_cols(const ZL &L) {
  int cols = 16;
  while (cols > 0 && thomas_smem(L, cols) > kThomasSmem) cols /= 2;
  return cols;
}
__global__ void __launch_bounds__(kThomasThreads) k_mg_thomas(ZL L, int cols, double *__restrict__ op) {
  extern __shared__ __align__(16) unsigned char tho_raw[];
  const int ld = L.ny | 1, ny = L.ny;
  double *sd = reinterpret_cast<double *>(tho_raw), *su = sd + cols * ld;
  const unsigned c0 = blockIdx.x * (unsigned)cols, ncol = (unsigned)L.nz * 2u * (unsigned)L.hx, S = (unsigned)L.S;
  const int nc = (int)min((unsigned)cols, ncol - c0);
  const long long n = L.n;
  const unsigned p0 = c0 * S;
  for (unsigned t = threadIdx.x; t < (unsigned)nc * S; t += kThomasThreads) {
    const unsigned c = t / S;
    const int j = zrow_of(L, t - c * S);
    if (j >= ny) continue;
    sd[c * ld + j] = op[OP_DG * n + p0 + t];
    su[c * ld + j] = j + 1 < ny ? op[OP_CN * n + p0 + t] : 0.0;
  }
  __syncthreads();
  if ((int)threadIdx.x < nc) {
    Thomas T;
    for (int j = 0; j < ny; j++) T.row(sd[threadIdx.x * ld + j], su[threadIdx.x * ld + j]);
  }
  __syncthreads();
  for (unsigned t = threadIdx.x; t < (unsigned)nc * S; t += kThomasThreads) {
    const unsigned c = t / S;
    const int j = zrow_of(L, t - c * S);
    if (j >= ny) continue;
    op[OP_IDEN * n + p0 + t] = sd[c * ld + j];
    op[OP_CPR * n + p0 + t] = su[c * ld + j];
  }
}
__global__ void k_mg_thomas_direct(ZL L, double *__restrict__ op) {
  const unsigned col = blockIdx.x * blockDim.x + threadIdx.x;
  if (col >= (unsigned)L.nz * 2u * (unsigned)L.hx) return;
  const long long n = L.n;
  Thomas T;
  for (int j = 0; j < L.ny; j++) {
    const long long q = (long long)col * L.S + zrow(L, j);
    double a = op[OP_DG * n + q], b = j + 1 < L.ny ? op[OP_CN * n + q] : 0.0;
    T.row(a, b);
    op[OP_IDEN * n + q] = a;
    op[OP_CPR * n + q] = b;
  }
}

// ------------------------------------------------------------------ packed operator
// The smoother and the transfers read the operator as a 4-vector, a 2-vector and two scalars per cell:
// cpl = {ce, cw, ct, cb} (couplings to i+1, i-1, k+1, k-1) and tri = {cs, iden} (coupling to
// j-1, Thomas pivot inverse), and the Thomas factor cpr and the diagonal dg apart: a smoothing
// row reads 28 bytes of operator in FP32, and only the restriction reads the diagonal.  A missing neighbour has a zero coupling; cs at j = 0
// is the periodic wrap coupling when j is periodic, else 0.
template <typename T>
struct __align__(4 * sizeof(T)) Q4 {
  T a, b, c, d;
};
template <typename T>
struct __align__(2 * sizeof(T)) Q2 {
  T a, b;
};

template <typename T>
__global__ void k_mg_pack(ZL L, const double *__restrict__ op, Q4<T> *__restrict__ cpl, Q2<T> *__restrict__ tri,
                          T *__restrict__ cpr, T *__restrict__ dg) {
  const long long q = blockIdx.x * (long long)blockDim.x + threadIdx.x, n = L.n;
  int i, j, k;
  if (q >= n || !zcell(L, (unsigned)q, i, j, k)) return;
  const ZNb nb = znb(L, i, j, k);
  Q4<T> a;
  Q2<T> b;
  a.a = (T)op[OP_CE * n + q];
  const unsigned p0 = zcol(L, i, k), pos = (unsigned)q - p0;
  a.b = nb.iw >= 0 ? (T)op[OP_CE * n + zcol(L, nb.iw, k) + pos] : T(0);
  a.c = (T)op[OP_CT * n + q];
  a.d = nb.kb >= 0 ? (T)op[OP_CT * n + zcol(L, i, nb.kb) + pos] : T(0);
  b.a = nb.js >= 0 ? (T)op[OP_CN * n + p0 + zrow(L, nb.js)] : T(0);
  b.b = (T)op[OP_IDEN * n + q];
  cpl[q] = a;
  tri[q] = b;
  cpr[q] = (T)op[OP_CPR * n + q];
  dg[q] = (T)op[OP_DG * n + q];
}

// Coarse cell q: bit e (0..26) set where the cell of its 3 x 3 x 3 neighbourhood at
// (e%3-1, e/3%3-1, e/9-1) exists and is active, bit 27 + ch where its child ch (bits i, j, k) is.
__device__ __forceinline__ int wrap_or_none(int v, int n, int per) { return (v >= 0 && v < n) ? v : (per ? (v + n) % n : -1); }
__global__ void k_mg_pmask(ZL F, ZL C, const uint8_t *__restrict__ actF, const uint8_t *__restrict__ actC,
                           unsigned long long *__restrict__ mask) {
  const long long q = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  int I, J, K;
  if (q >= C.n || !zcell(C, (unsigned)q, I, J, K)) return;
  // every byte is loaded (the cell's own where there is no neighbour) before the first is used
  int Iv[3], Jv[3], Kv[3];
  bool Io[3], Jo[3], Ko[3];
#pragma unroll
  for (int d = 0; d < 3; d++) {
    const int i = wrap_or_none(I + d - 1, C.nx, C.ip), j = wrap_or_none(J + d - 1, C.ny, C.jp);
    const int k = wrap_or_none(K + d - 1, C.nz, C.kp);
    Io[d] = i >= 0; Jo[d] = j >= 0; Ko[d] = k >= 0;
    Iv[d] = Io[d] ? i : I; Jv[d] = (int)zrow(C, Jo[d] ? j : J); Kv[d] = Ko[d] ? k : K;
  }
  uint8_t a[27], b[8];
#pragma unroll
  for (int e = 0; e < 27; e++) a[e] = actC[zcol(C, Iv[e % 3], Kv[e / 9]) + (unsigned)Jv[e / 3 % 3]];
  const unsigned r[2] = {zrow(F, 2 * J), zrow(F, 2 * J + 1)};
#pragma unroll
  for (int ch = 0; ch < 8; ch++) b[ch] = actF[zcol(F, 2 * I + (ch & 1), 2 * K + (ch >> 2)) + r[(ch >> 1) & 1]];
  unsigned long long m = 0;
#pragma unroll
  for (int e = 0; e < 27; e++)
    if (Io[e % 3] && Jo[e / 3 % 3] && Ko[e / 9] && a[e]) m |= 1ull << e;
#pragma unroll
  for (int ch = 0; ch < 8; ch++)
    if (b[ch]) m |= 1ull << (27 + ch);
  mask[q] = m;
}

// ------------------------------------------------------------------ smoother
template <typename T>
__device__ __forceinline__ void scan_compose_up(T &A, T &B, int l, int lw) {
  // inclusive scan over lanes 0..l of a group of x -> A x + B maps (later lanes applied last)
#pragma unroll
  for (int off = 1; off < lw; off <<= 1) {
    const T pa = __shfl_up_sync(0xffffffffu, A, off, lw), pb = __shfl_up_sync(0xffffffffu, B, off, lw);
    if (l >= off) { B = A * pb + B; A = A * pa; }
  }
}
template <typename T>
__device__ __forceinline__ void scan_compose_down(T &A, T &B, int l, int lw) {
  // inclusive scan over lanes l..lw-1 (higher lanes applied first)
#pragma unroll
  for (int off = 1; off < lw; off <<= 1) {
    const T pa = __shfl_down_sync(0xffffffffu, A, off, lw), pb = __shfl_down_sync(0xffffffffu, B, off, lw);
    if (l + off < lw) { B = A * pb + B; A = A * pa; }
  }
}

// What a pass over the columns of one colour (or, line Jacobi, of both) may assume of x:
enum { Z_NB_ZERO = 1, Z_OWN_ZERO = 2 };  // the neighbour columns / the own column are zero

// Column t of a pass (colour 0/1: the columns of that colour; < 0: all): its first slot and
// the slot offsets of its four neighbour columns.  A missing neighbour (domain edge, zero
// coupling) borrows the opposite one's column, so every x read is of the other colour
// (every level has at least 2 cells along i and k).
struct ZCol {
  unsigned p0;
  int oe, ow, ot, ob;
  bool valid;
};
__device__ __forceinline__ unsigned zpass_columns(const ZL &L, int colour) {
  return (unsigned)L.nz * (unsigned)L.hx * (colour >= 0 ? 1u : 2u);
}
__device__ __forceinline__ ZCol zcolumn(const ZL &L, int colour, unsigned t) {
  ZCol r;
  const unsigned hx = (unsigned)L.hx;
  r.valid = t < zpass_columns(L, colour);
  if (!r.valid) t = 0;  // a real column for the addresses; nothing is stored
  unsigned k = t / hx;
  const unsigned h = t - k * hx;
  unsigned c = (unsigned)colour;
  if (colour < 0) { c = k & 1; k >>= 1; }
  int i = (int)(2 * h + (c ^ (k & 1)));
  if (i >= L.nx) { r.valid = false; i -= 2; }
  const int kk = (int)k;
  r.p0 = zcol(L, i, kk);
  int ie = i + 1 < L.nx ? i + 1 : (L.ip ? 0 : -1), iw = i > 0 ? i - 1 : (L.ip ? L.nx - 1 : -1);
  int kt = kk + 1 < L.nz ? kk + 1 : (L.kp ? 0 : -1), kb = kk > 0 ? kk - 1 : (L.kp ? L.nz - 1 : -1);
  if (ie < 0) ie = iw;
  if (iw < 0) iw = ie;
  if (kt < 0) kt = kb;
  if (kb < 0) kb = kt;
  r.oe = (int)(zcol(L, ie, kk) - r.p0);
  r.ow = (int)(zcol(L, iw, kk) - r.p0);
  r.ot = (int)(zcol(L, i, kt) - r.p0);
  r.ob = (int)(zcol(L, i, kb) - r.p0);
  return r;
}

// The operator rows of a lane: SEG rows from slot q0, ls apart; none (zeros) for a lane past ls.
template <typename T, int SEG>
struct ZRows {
  Q4<T> cp[SEG];
  Q2<T> tr[SEG];
  T cx[SEG];
};
template <typename T, int SEG, bool kFull>
__device__ __forceinline__ void zload(const ZL &L, const Q4<T> *__restrict__ cpl, const Q2<T> *__restrict__ tri,
                                      const T *__restrict__ cpr, unsigned p0, int l, int flags, ZRows<T, SEG> &R) {
  const int ls = kFull ? 32 : L.ls;
  if (!kFull && l >= ls) {
#pragma unroll
    for (int s = 0; s < SEG; s++) {
      R.tr[s] = Q2<T>{T(0), T(0)};
      R.cx[s] = T(0);
    }
    return;
  }
#pragma unroll
  for (int s = 0; s < SEG; s++) {
    const unsigned q = p0 + (unsigned)(l + s * ls);
    R.tr[s] = tri[q];
    R.cx[s] = cpr[q];
    if (!(flags & Z_NB_ZERO)) R.cp[s] = cpl[q];
  }
}

// Solves one column (SEG rows in each of the ls lanes of a group of lw): right-hand side b
// minus the couplings to the neighbour columns in xr, the forward elimination
// d_j = r_j / pivot - (cs_j / pivot) d_{j-1} and the back substitution
// x_j = d_j - cpr_j x_{j+1} as first-order linear recurrences: each lane composes its rows,
// a shuffle scan combines the lanes, each lane then replays its rows.  Every lane of the
// warp takes part.  kFull: all 32 lanes hold rows (ls = 32).
template <typename T, int SEG, bool kFull>
__device__ __forceinline__ void zsolve(const ZL &L, const ZCol &z, int l, const ZRows<T, SEG> &R, const T *b,
                                       const T *xr, T *xw, int flags) {
  const unsigned q0 = z.p0 + (unsigned)l;
  const int ls = kFull ? 32 : L.ls, lw = kFull ? 32 : L.lw;
  const bool own = kFull || l < ls;
  T r[SEG], m[SEG];
#pragma unroll
  for (int s = 0; s < SEG; s++) r[s] = own ? b[q0 + (unsigned)(s * ls)] : T(0);
  if (!(flags & Z_NB_ZERO) && own) {
    T xe[SEG], xv[SEG], xt[SEG], xb[SEG];
#pragma unroll
    for (int s = 0; s < SEG; s++) {
      const int q = (int)(q0 + (unsigned)(s * ls));
      xe[s] = xr[(unsigned)(q + z.oe)];
      xv[s] = xr[(unsigned)(q + z.ow)];
      xt[s] = xr[(unsigned)(q + z.ot)];
      xb[s] = xr[(unsigned)(q + z.ob)];
    }
#pragma unroll
    for (int s = 0; s < SEG; s++) {
      r[s] -= R.cp[s].a * xe[s];
      r[s] -= R.cp[s].b * xv[s];
      r[s] -= R.cp[s].c * xt[s];
      r[s] -= R.cp[s].d * xb[s];
    }
  }
  if (L.jp && !(flags & Z_OWN_ZERO)) {
    // periodic j: the wrap coupling (cs of row 0) and the far end of the own column (old values)
    const T wrap = __shfl_sync(0xffffffffu, R.tr[0].a, 0, lw);
    const T first = xr[z.p0], last = xr[z.p0 + zrow(L, L.ny - 1)];
#pragma unroll
    for (int s = 0; s < SEG; s++) {
      const int j = l * SEG + s;
      if (j == 0) r[s] -= wrap * last;
      if (j == L.ny - 1) r[s] -= wrap * first;
    }
  }
#pragma unroll
  for (int s = 0; s < SEG; s++) {
    r[s] *= R.tr[s].b;
    m[s] = R.tr[s].a * R.tr[s].b;
  }
  if (l == 0) m[0] = 0;
  T A = 1, B = 0;
#pragma unroll
  for (int s = 0; s < SEG; s++) { B = -m[s] * B + r[s]; A = -m[s] * A; }
  scan_compose_up<T>(A, B, l, lw);
  T d = __shfl_up_sync(0xffffffffu, B, 1, lw);
  if (l == 0) d = 0;
#pragma unroll
  for (int s = 0; s < SEG; s++) { d = -m[s] * d + r[s]; r[s] = d; }
  A = 1; B = 0;
#pragma unroll
  for (int s = SEG - 1; s >= 0; s--) { B = -R.cx[s] * B + r[s]; A = -R.cx[s] * A; }
  scan_compose_down<T>(A, B, l, lw);
  T x = __shfl_down_sync(0xffffffffu, B, 1, lw);
  if (l == lw - 1) x = 0;
#pragma unroll
  for (int s = SEG - 1; s >= 0; s--) { x = -R.cx[s] * x + r[s]; r[s] = x; }
  if (!z.valid || !own) return;
#pragma unroll
  for (int s = 0; s < SEG; s++) xw[q0 + (unsigned)(s * ls)] = r[s];
}

// The same for columns of more rows per lane than the register forms take: the rows are
// replayed through the column's own slots of xw, which no other column of the pass reads.
// kJac: damped by omega against the previous iterate xr.
template <typename T, bool kJac>
__device__ void zsolve_long(const ZL &L, const ZCol &z, int l, const Q4<T> *__restrict__ cpl,
                            const Q2<T> *__restrict__ tri, const T *__restrict__ cpr, const T *b, const T *xr, T *xw,
                            int flags, T omega) {
  const unsigned q0 = z.p0 + (unsigned)l;
  const int seg = l < L.ls ? L.seg : 0;
  const bool st = z.valid;
  T wrap = 0, first = 0, last = 0;
  if (L.jp && !(flags & Z_OWN_ZERO)) {
    wrap = tri[z.p0].a;
    first = xr[z.p0];
    last = xr[z.p0 + zrow(L, L.ny - 1)];
  }
  __syncwarp();
  T A = 1, B = 0;
  for (int s = 0; s < seg; s++) {
    const unsigned q = q0 + (unsigned)(s * L.ls);
    const Q2<T> t = tri[q];
    T r = b[q];
    if (!(flags & Z_NB_ZERO)) {
      const Q4<T> c = cpl[q];
      r -= c.a * xr[(unsigned)((int)q + z.oe)];
      r -= c.b * xr[(unsigned)((int)q + z.ow)];
      r -= c.c * xr[(unsigned)((int)q + z.ot)];
      r -= c.d * xr[(unsigned)((int)q + z.ob)];
    }
    const int j = l * seg + s;
    if (j == 0) r -= wrap * last;
    if (j == L.ny - 1) r -= wrap * first;
    r *= t.b;
    const T m = j > 0 ? t.a * t.b : T(0);
    if (st) xw[q] = r;
    B = -m * B + r;
    A = -m * A;
  }
  scan_compose_up<T>(A, B, l, L.lw);
  T d = __shfl_up_sync(0xffffffffu, B, 1, L.lw);
  if (l == 0) d = 0;
  for (int s = 0; s < seg; s++) {
    const unsigned q = q0 + (unsigned)(s * L.ls);
    const Q2<T> t = tri[q];
    const T m = l * seg + s > 0 ? t.a * t.b : T(0);
    d = -m * d + xw[q];
    if (st) xw[q] = d;
  }
  A = 1; B = 0;
  for (int s = seg - 1; s >= 0; s--) {
    const unsigned q = q0 + (unsigned)(s * L.ls);
    const T c = cpr[q];
    B = -c * B + xw[q];
    A = -c * A;
  }
  scan_compose_down<T>(A, B, l, L.lw);
  T x = __shfl_down_sync(0xffffffffu, B, 1, L.lw);
  if (l == L.lw - 1) x = 0;
  for (int s = seg - 1; s >= 0; s--) {
    const unsigned q = q0 + (unsigned)(s * L.ls);
    x = -cpr[q] * x + xw[q];
    if (st) {
      if (kJac) {
        const T xo = (flags & Z_OWN_ZERO) ? T(0) : xr[q];
        xw[q] = xo + omega * (x - xo);
      } else {
        xw[q] = x;
      }
    }
  }
}

// Thomas' recurrence of one column by one thread, row by row: r the right-hand sides on entry
// and the solution on exit, lo the lower couplings (0 at row 0), id the pivots' inverses, cx
// the forward factors.  Four rows' loads are in flight at a time.
template <typename T>
__device__ __forceinline__ void thomas_rows(T *r, const T *lo, const T *id, const T *cx, int ny) {
  constexpr int CH = 4;
  T d = 0;
  for (int j0 = 0; j0 < ny; j0 += CH) {
    T rr[CH], ll[CH], ii[CH];
#pragma unroll
    for (int u = 0; u < CH; u++) {
      const int j = min(j0 + u, ny - 1);
      rr[u] = r[j]; ll[u] = lo[j]; ii[u] = id[j];
    }
#pragma unroll
    for (int u = 0; u < CH; u++) {
      if (j0 + u >= ny) break;
      d = (rr[u] - ll[u] * d) * ii[u];
      r[j0 + u] = d;
    }
  }
  T x = 0;
  for (int j1 = ny - 1; j1 >= 0; j1 -= CH) {
    T dd[CH], cc[CH];
#pragma unroll
    for (int u = 0; u < CH; u++) {
      const int j = max(j1 - u, 0);
      dd[u] = r[j]; cc[u] = cx[j];
    }
#pragma unroll
    for (int u = 0; u < CH; u++) {
      if (j1 - u < 0) break;
      x = dd[u] - cc[u] * x;
      r[j1 - u] = x;
    }
  }
}

// One pass over the columns of one colour.  Bound by the bytes of a row (FP32:
// operator 28, b 4, the other colour's x 4, x 4); registers set the occupancy.  SEG = 0: columns
// of more than eight rows a lane.
template <typename T> struct ZBounds;
template <> struct ZBounds<float> { static constexpr int v = 5; };
template <> struct ZBounds<double> { static constexpr int v = 3; };
constexpr int kColThreads = 128;
template <typename T>
struct ZOp {
  const Q4<T> *cpl;
  const Q2<T> *tri;
  const T *cpr;
};
template <typename T, int SEG, bool kFull>
__global__ void __launch_bounds__(kColThreads, ZBounds<T>::v) k_zcol(ZL L, ZOp<T> op, const T *b, T *x, int colour,
                                                                     int flags) {
  const unsigned tid = blockIdx.x * blockDim.x + threadIdx.x;
  const int lw = kFull ? 32 : L.lw, l = (int)(tid & (unsigned)(lw - 1));
  const ZCol z = zcolumn(L, colour, kFull ? tid >> 5 : tid >> L.lwl);
  if constexpr (SEG > 0) {
    ZRows<T, SEG> R;
    zload<T, SEG, kFull>(L, op.cpl, op.tri, op.cpr, z.p0, l, flags, R);
    pdl_wait();
    zsolve<T, SEG, kFull>(L, z, l, R, b, x, x, flags);
  } else {
    pdl_wait();
    zsolve_long<T, false>(L, z, l, op.cpl, op.tri, op.cpr, b, x, x, flags, T(1));
  }
}

// A line Jacobi sweep over columns too long for the kernel below (the finest level only), by lane
// groups.
template <typename T>
__global__ void __launch_bounds__(kColThreads) k_zlong(ZL L, ZOp<T> op, const T *b, const T *xr, T *xw, int flags,
                                                       T omega) {
  const unsigned tid = blockIdx.x * blockDim.x + threadIdx.x;
  pdl_wait();
  zsolve_long<T, true>(L, zcolumn(L, -1, tid >> L.lwl), (int)(tid & (unsigned)(L.lw - 1)), op.cpl, op.tri, op.cpr, b, xr,
                       xw, flags, omega);
}

// One pass by Thomas' recurrence row by row (small levels, and every line Jacobi sweep: kJac,
// colour < 0, xr the previous iterate): a block stages the rows of kSerialCols columns in
// shared memory with coalesced loads, one thread a column solves there, and all write back.
// (One thread a column straight from global memory took 22 us a pass on 45 x 37 x 53 cells.)
constexpr int kSerialCols = 16, kSerialThreads = 32 * kSerialCols;
template <typename T>
static size_t serial_smem(int ny) { return sizeof(T) * 4 * kSerialCols * ((size_t)ny | 1); }
constexpr size_t kSerialSmem = 200 * 1024;
template <typename T, bool kJac>
__global__ void __launch_bounds__(kSerialThreads) k_zserial(ZL L, ZOp<T> op, const T *b, const T *xr, T *xw, int colour,
                                                            int flags, T omega) {
  extern __shared__ __align__(16) unsigned char ser_raw[];
  const int ny = L.ny, ld = ny | 1;
  T *sr = reinterpret_cast<T *>(ser_raw), *slo = sr + kSerialCols * ld, *sid = slo + kSerialCols * ld,
    *scx = sid + kSerialCols * ld;
  const unsigned t0 = blockIdx.x * kSerialCols;
  const int lane = threadIdx.x & 31, c = threadIdx.x >> 5;  // a warp loads and stores a column
  const ZCol z = zcolumn(L, colour, t0 + (unsigned)c);
  pdl_wait();
  if (z.valid) {
    T wrap = 0, first = 0, last = 0;
    if (L.jp && !(flags & Z_OWN_ZERO)) {
      wrap = op.tri[z.p0].a;
      first = xr[z.p0];
      last = xr[z.p0 + zrow(L, ny - 1)];
    }
#pragma unroll 2
    for (int s = lane; s < L.S; s += 32) {
      const int j = zrow_of(L, (unsigned)s);
      if (j >= ny) continue;
      const unsigned q = z.p0 + (unsigned)s;
      T r = b[q];
      const Q2<T> t = op.tri[q];
      if (!(flags & Z_NB_ZERO)) {
        const Q4<T> cp = op.cpl[q];
        r -= cp.a * xr[(unsigned)((int)q + z.oe)];
        r -= cp.b * xr[(unsigned)((int)q + z.ow)];
        r -= cp.c * xr[(unsigned)((int)q + z.ot)];
        r -= cp.d * xr[(unsigned)((int)q + z.ob)];
      }
      if (j == 0) r -= wrap * last;
      if (j == ny - 1) r -= wrap * first;
      sr[c * ld + j] = r;
      slo[c * ld + j] = j > 0 ? t.a : T(0);
      sid[c * ld + j] = t.b;
      scx[c * ld + j] = op.cpr[q];
    }
  }
  __syncthreads();
  if (threadIdx.x < kSerialCols && zcolumn(L, colour, t0 + threadIdx.x).valid) {
    T *r = sr + threadIdx.x * ld;
    const T *lo = slo + threadIdx.x * ld, *id = sid + threadIdx.x * ld, *cx = scx + threadIdx.x * ld;
    thomas_rows<T>(r, lo, id, cx, ny);
  }
  __syncthreads();
  if (!z.valid) return;
  for (int s = lane; s < L.S; s += 32) {
    const int j = zrow_of(L, (unsigned)s);
    if (j >= ny) continue;
    const unsigned q = z.p0 + (unsigned)s;
    const T v = sr[c * ld + j];
    if (kJac) {
      const T xo = (flags & Z_OWN_ZERO) ? T(0) : xr[q];
      xw[q] = (flags & Z_OWN_ZERO) ? omega * v : xo + omega * (v - xo);
    } else {
      xw[q] = v;
    }
  }
}

// ------------------------------------------------------------------ transfers
// Coarse right-hand side at slot q of the coarse level: the sum of the residuals b - A x of
// the cell's active children.  With kColour0 the children of colour 1 ((i xor k) odd) are left
// out: after a zebra sweep that ends with the colour-1 pass their line equations hold
// exactly (the j-line solve is exact when j is not periodic), so their residuals are
// rounding only.  Two rows of a fine column share their loads.
// Levels of at most this many cells are solved row by row and restricted from all children.
constexpr long long kSerialCells = 512;
__host__ __device__ inline bool colour0_restriction(const ZL &F, int zebra) {
  return zebra && !F.jp && (long long)F.nx * F.ny * F.nz > kSerialCells;
}
template <typename T, bool kColour0>
__device__ __forceinline__ void zrestrict_cell(const ZL &F, const ZL &C, const Q4<T> *__restrict__ cpl,
                                               const Q2<T> *__restrict__ tri, const T *__restrict__ dg, const T *x,
                                               const T *b, T *bc, unsigned q) {
  int I, J, K;
  if (q >= (unsigned)C.n || !zcell(C, q, I, J, K)) return;
  const int j0 = 2 * J, j1 = j0 + 1;
  const unsigned r0 = zrow(F, j0), r1 = zrow(F, j1);
  const bool lo = j0 > 0, hi = j1 + 1 < F.ny;
  const unsigned rm = lo ? zrow(F, j0 - 1) : (F.jp ? zrow(F, F.ny - 1) : r0);
  const unsigned rp = hi ? zrow(F, j1 + 1) : 0u;  // row 0 (its cs is the wrap coupling, or 0)
  T res[8];  // of child a + 2 (j & 1) + 4 c
#pragma unroll
  for (int c = 0; c < 2; c++)
#pragma unroll
    for (int a = 0; a < 2; a++) {
      if (kColour0 && a != c) continue;
      const int i = 2 * I + a, k = 2 * K + c;
      const unsigned p = zcol(F, i, k);
      const int ie = i + 1 < F.nx ? i + 1 : (F.ip ? 0 : i), iw = i > 0 ? i - 1 : (F.ip ? F.nx - 1 : i);
      const int kt = k + 1 < F.nz ? k + 1 : (F.kp ? 0 : k), kb = k > 0 ? k - 1 : (F.kp ? F.nz - 1 : k);
      const unsigned pe = zcol(F, ie, k), pw = zcol(F, iw, k), pt = zcol(F, i, kt), pb = zcol(F, i, kb);
      const Q4<T> c0 = cpl[p + r0], c1 = cpl[p + r1];
      const T s0 = tri[p + r0].a, s1 = tri[p + r1].a, s2 = (hi || F.jp) ? tri[p + rp].a : T(0);
      const T x0 = *(x + p + r0), x1 = *(x + p + r1), xm = *(x + p + rm), xp = *(x + p + rp);
      const T e0 = *(x + pe + r0), e1 = *(x + pe + r1), w0 = *(x + pw + r0), w1 = *(x + pw + r1);
      const T t0 = *(x + pt + r0), t1 = *(x + pt + r1), d0 = *(x + pb + r0), d1 = *(x + pb + r1);
      const T b0 = *(b + p + r0), b1 = *(b + p + r1);
      const T g0 = dg[p + r0], g1 = dg[p + r1];
      T a0 = g0 * x0, a1 = g1 * x1;
      a0 += c0.a * e0; a1 += c1.a * e1;
      a0 += c0.b * w0; a1 += c1.b * w1;
      a0 += s0 * xm; a1 += s1 * x0;
      a0 += s1 * x1; a1 += s2 * xp;
      a0 += c0.c * t0; a1 += c1.c * t1;
      a0 += c0.d * d0; a1 += c1.d * d1;
      res[a + 4 * c] = g0 != T(0) ? b0 - a0 : T(0);
      res[a + 2 + 4 * c] = g1 != T(0) ? b1 - a1 : T(0);
    }
  T sum = 0;
#pragma unroll
  for (int ch = 0; ch < 8; ch++)
    if (!kColour0 || (ch & 1) == ch >> 2) sum += res[ch];
  bc[q] = sum;
}

template <typename T, bool kColour0>
__global__ void __launch_bounds__(128) k_zrestrict(ZL F, ZL C, const Q4<T> *__restrict__ cpl,
                                                   const Q2<T> *__restrict__ tri, const T *__restrict__ dg, const T *x,
                                                   const T *b, T *bc) {
  pdl_wait();
  zrestrict_cell<T, kColour0>(F, C, cpl, tri, dg, x, b, bc, blockIdx.x * blockDim.x + threadIdx.x);
}

// x_fine += P x_coarse (cell-centred trilinear) for the children of the coarse cell at slot q:
// its 3 x 3 x 3 neighbourhood is loaded once.  kColour1 leaves out the children of colour 0:
// the zebra sweep that follows solves their columns from the colour-1 columns alone (when j
// is not periodic) and never reads their value.
template <typename T, bool kColour1>
__device__ __forceinline__ void zprolong_cell(const ZL &F, const ZL &C, const unsigned long long *__restrict__ mask,
                                              T *x, const T *xc, unsigned q) {
  int I, J, K;
  if (q >= (unsigned)C.n || !zcell(C, q, I, J, K)) return;
  const unsigned long long ok = mask[q];
  // a neighbour that does not exist is read from the cell itself and masked out
  auto nb = [](int v, int n, int per, int own) { const int w = wrap_or_none(v, n, per); return w < 0 ? own : w; };
  const int Ii[3] = {nb(I - 1, C.nx, C.ip, I), I, nb(I + 1, C.nx, C.ip, I)};
  const int Kk[3] = {nb(K - 1, C.nz, C.kp, K), K, nb(K + 1, C.nz, C.kp, K)};
  const unsigned rr[3] = {zrow(C, nb(J - 1, C.ny, C.jp, J)), zrow(C, J), zrow(C, nb(J + 1, C.ny, C.jp, J))};
  T v[27];
#pragma unroll
  for (int e = 0; e < 27; e++) v[e] = *(xc + zcol(C, Ii[e % 3], Kk[e / 9]) + rr[e / 3 % 3]);
  const T xo = v[13];
  const unsigned f0 = zrow(F, 2 * J), f1 = zrow(F, 2 * J + 1);
  unsigned qf[8];
  T xq[8];
#pragma unroll
  for (int ch = 0; ch < 8; ch++) {
    const int ai = ch & 1, aj = (ch >> 1) & 1, ak = ch >> 2;
    if (kColour1 && ai == ak) continue;
    qf[ch] = zcol(F, 2 * I + ai, 2 * K + ak) + (aj ? f1 : f0);
    xq[ch] = *(x + qf[ch]);
  }
#pragma unroll
  for (int ch = 0; ch < 8; ch++) {
    const int ai = ch & 1, aj = (ch >> 1) & 1, ak = ch >> 2;
    if (kColour1 && ai == ak) continue;
    // the other nearest coarse cell: the next one for an odd child index, the previous one for an even one
    const int di = ai ? 2 : 0, dj = aj ? 2 : 0, dk = ak ? 2 : 0;
    T wown = T(27) / T(64);
    T s = 0;
#pragma unroll
    for (int c = 0; c < 2; c++)
#pragma unroll
      for (int bb = 0; bb < 2; bb++)
#pragma unroll
        for (int a = 0; a < 2; a++) {
          if (a + bb + c == 0) continue;
          const T w = (a ? T(1) : T(3)) * (bb ? T(1) : T(3)) * (c ? T(1) : T(3)) / T(64);
          const int e = (a ? di : 1) + 3 * (bb ? dj : 1) + 9 * (c ? dk : 1);
          if (!((ok >> e) & 1ull)) { wown += w; continue; }
          s += w * v[e];
        }
    if ((ok >> (27 + ch)) & 1ull) x[qf[ch]] = xq[ch] + (s + wown * xo);
  }
}

template <typename T, bool kColour1>
__global__ void __launch_bounds__(128) k_zprolong(ZL F, ZL C, const unsigned long long *__restrict__ mask,
                                                  T *x, const T *xc) {
  pdl_wait();
  zprolong_cell<T, kColour1>(F, C, mask, x, xc, blockIdx.x * blockDim.x + threadIdx.x);
}

// The same prolongation, one colour-1 fine cell per thread: eight coarse values in flight instead
// of 27 and four times the threads.  The coarse-centric form loads less, this one waits less:
// it serves the levels too small to fill the GPU (kFineProlong: up to 64^3 cells; a whole step of
// 64^3 cells 1572 -> 1528 us, while on every level of 256 x 192 x 256 it costs a V-cycle 35 us).
template <typename T>
__global__ void __launch_bounds__(128) k_zprolong_fine(ZL F, ZL C, const unsigned long long *__restrict__ mask, T *x,
                                                       const T *xc) {
  const unsigned t = blockIdx.x * blockDim.x + threadIdx.x;
  const unsigned col = t / (unsigned)F.S, pos = t - col * (unsigned)F.S;
  const unsigned k = col / (unsigned)F.hx, h = col - k * (unsigned)F.hx;
  const int j = zrow_of(F, pos), i = (int)(2 * h + (1 ^ (k & 1)));
  const bool cell = k < (unsigned)F.nz && j < F.ny && i < F.nx;
  if (!cell) { pdl_wait(); return; }
  const int I = i >> 1, J = j >> 1, K = (int)k >> 1, ai = i & 1, aj = j & 1, ak = (int)k & 1;
  // the other nearest coarse cell along each direction (the cell itself where there is none: masked out)
  auto other = [](int v, int up, int n, int per) {
    const int w = up ? v + 1 : v - 1;
    return w < 0 ? (per ? n - 1 : v) : (w >= n ? (per ? 0 : v) : w);
  };
  const int In = other(I, ai, C.nx, C.ip), Jn = other(J, aj, C.ny, C.jp), Kn = other(K, ak, C.nz, C.kp);
  const unsigned c00 = zcol(C, I, K), c10 = zcol(C, In, K), c01 = zcol(C, I, Kn), c11 = zcol(C, In, Kn);
  const unsigned r0 = zrow(C, J), r1 = zrow(C, Jn);
  const unsigned q = ((k * 2 + 1) * (unsigned)F.hx + h) * (unsigned)F.S + pos;
  const unsigned long long ok = mask[c00 + r0];
  pdl_wait();
  const T xo = xc[c00 + r0];
  const T v[8] = {xo, xc[c10 + r0], xc[c00 + r1], xc[c10 + r1], xc[c01 + r0], xc[c11 + r0], xc[c01 + r1], xc[c11 + r1]};
  const T xq = x[q];
  const int di = ai ? 2 : 0, dj = aj ? 2 : 0, dk = ak ? 2 : 0;
  T wown = T(27) / T(64);
  T s = 0;
#pragma unroll
  for (int n = 1; n < 8; n++) {
    const int a = n & 1, bb = (n >> 1) & 1, c = n >> 2;
    const T w = (a ? T(1) : T(3)) * (bb ? T(1) : T(3)) * (c ? T(1) : T(3)) / T(64);
    const int e = (a ? di : 1) + 3 * (bb ? dj : 1) + 9 * (c ? dk : 1);
    if (!((ok >> e) & 1ull)) { wown += w; continue; }
    s += w * v[n];
  }
  if ((ok >> (27 + ai + 2 * aj + 4 * ak)) & 1ull) x[q] = xq + (s + wown * xo);
}
constexpr long long kFineProlong = 64 * 64 * 64;  // cells of the fine level

// ------------------------------------------------------------------ bottom of the V-cycle
// The coarse levels are too small to fill the GPU, and a launch per colour pass costs more
// than the work.  From the first level of at most kSerialCells cells down, one thread block
// runs the rest of the V-cycle (smoothing, restriction, coarsest sweeps, prolongation), one
// thread a column, with the vectors and the smoother's operator of all its levels in shared
// memory and block barriers between the phases: a phase is a chain of shared-memory loads and a barrier, with no trip
// to L2.  Starting at 4096 cells (lane groups in the same block) took 156 us a V-cycle of
// 64^3 cells against 133 (FP32); a cluster of eight blocks exchanging through L2 186.
constexpr int kBottomMaxLevels = 12;
constexpr int kBottomThreads = 512;
constexpr size_t kBottomSmem = 200 * 1024;

template <typename T>
struct BLevel {
  ZL z;
  const unsigned long long *pmask;  // of the cells of this level, for the prolongation to the finer one
  const Q4<T> *cpl;
  const Q2<T> *tri;
  const T *cpr, *dg;
  unsigned sm;  // the level's arrays in shared memory, n slots each: x, b, previous x, ce, cw, ct, cb, cs, iden, cpr
  int zebra;
};
template <typename T>
struct Bottom {
  int nl;
  int pre, post, coarse;
  T omega;
  T *x;        // the top level's vectors
  const T *b;
  BLevel<T> lv[kBottomMaxLevels];
};

// One column of a bottom level by one thread, everything in shared memory (sm: the level's
// arrays); the right-hand sides are eliminated in the column's slots of xw.
template <typename T, bool kJac>
__device__ __forceinline__ void bot_column(const ZL &L, const ZCol &z, const T *sm, const T *xr, T *xw, int flags, T omega) {
  if (!z.valid) return;
  const unsigned n = (unsigned)L.n;
  const T *b = sm + n + z.p0, *ce = sm + 3 * n + z.p0, *cw = ce + n, *ct = cw + n, *cb = ct + n, *cs = cb + n,
          *id = cs + n, *cx = id + n;
  const T *xo = xr + z.p0;
  T *xv = xw + z.p0;
  const int ny = L.ny;
  T wrap = 0, first = 0, last = 0;
  if (L.jp && !(flags & Z_OWN_ZERO)) { wrap = cs[0]; first = xo[0]; last = xo[ny - 1]; }
  constexpr int CH = 4;
  T d = 0;
  for (int j0 = 0; j0 < ny; j0 += CH) {
    T r[CH], lo[CH], ii[CH];
#pragma unroll
    for (int u = 0; u < CH; u++) {
      const int j = min(j0 + u, ny - 1);
      r[u] = b[j]; lo[u] = cs[j]; ii[u] = id[j];
      if (!(flags & Z_NB_ZERO)) {
        r[u] -= ce[j] * xo[j + z.oe];
        r[u] -= cw[j] * xo[j + z.ow];
        r[u] -= ct[j] * xo[j + z.ot];
        r[u] -= cb[j] * xo[j + z.ob];
      }
      if (j == 0) { r[u] -= wrap * last; lo[u] = 0; }
      if (j == ny - 1) r[u] -= wrap * first;
    }
#pragma unroll
    for (int u = 0; u < CH; u++) {
      if (j0 + u >= ny) break;
      d = (r[u] - lo[u] * d) * ii[u];
      xv[j0 + u] = d;
    }
  }
  T x = 0;
  for (int j1 = ny - 1; j1 >= 0; j1 -= CH) {
    T dd[CH], cc[CH], old[CH];
#pragma unroll
    for (int u = 0; u < CH; u++) {
      const int j = max(j1 - u, 0);
      dd[u] = xv[j]; cc[u] = cx[j];
      old[u] = kJac && !(flags & Z_OWN_ZERO) ? xo[j] : T(0);
    }
#pragma unroll
    for (int u = 0; u < CH; u++) {
      if (j1 - u < 0) break;
      x = dd[u] - cc[u] * x;
      xv[j1 - u] = kJac ? ((flags & Z_OWN_ZERO) ? omega * x : old[u] + omega * (x - old[u])) : x;
    }
  }
}

// `sweeps` smoothing sweeps of a bottom level; x ends in x.  At most kSerialCells columns, so
// every thread has at most one of each colour.
template <typename T>
__device__ void bot_smooth(const BLevel<T> &L, T *sm, int sweeps, bool x_zero, T omega) {
  T *x = sm;
  if (L.zebra) {
    const ZCol z[2] = {zcolumn(L.z, 0, threadIdx.x), zcolumn(L.z, 1, threadIdx.x)};
    for (int s = 0; s < sweeps; s++)
#pragma unroll
      for (int c = 0; c < 2; c++) {
        const bool zero = x_zero && s == 0;
        bot_column<T, false>(L.z, z[c], sm, x, x, (zero ? Z_OWN_ZERO : 0) | (zero && c == 0 ? Z_NB_ZERO : 0), T(1));
        __syncthreads();
      }
    return;
  }
  // line Jacobi
  T *xo = sm + 2 * L.z.n;
  T *from = x_zero ? xo : x, *to = x_zero ? x : xo;
  const ZCol z = zcolumn(L.z, -1, threadIdx.x);
  for (int s = 0; s < sweeps; s++) {
    bot_column<T, true>(L.z, z, sm, from, to, x_zero && s == 0 ? Z_NB_ZERO | Z_OWN_ZERO : 0, omega);
    __syncthreads();
    T *const t = from; from = to; to = t;
  }
  if (from != x) {
    for (unsigned q = threadIdx.x; q < (unsigned)L.z.n; q += kBottomThreads) x[q] = from[q];
    __syncthreads();
  }
}

template <typename T>
__global__ void __launch_bounds__(kBottomThreads) k_mg_bottom(const __grid_constant__ Bottom<T> B) {
  extern __shared__ __align__(16) unsigned char bot_raw[];
  T *sm = reinterpret_cast<T *>(bot_raw);
  // the operators, and zero vectors (slots that hold no cell are read and never written)
  for (int l = 0; l < B.nl; l++) {
    const BLevel<T> &L = B.lv[l];
    const unsigned n = (unsigned)L.z.n;
    T *s = sm + L.sm;
    for (unsigned q = threadIdx.x; q < n; q += kBottomThreads) {
      const Q4<T> c = L.cpl[q];
      const Q2<T> t = L.tri[q];
      s[q] = s[n + q] = s[2 * n + q] = T(0);
      s[3 * n + q] = c.a; s[4 * n + q] = c.b; s[5 * n + q] = c.c; s[6 * n + q] = c.d;
      s[7 * n + q] = t.a; s[8 * n + q] = t.b; s[9 * n + q] = L.cpr[q];
    }
  }
  __syncthreads();
  pdl_wait();
  {
    const ZL &z = B.lv[0].z;
    const T *b = B.b;
    for (unsigned q = threadIdx.x; q < (unsigned)z.n; q += kBottomThreads) sm[z.n + q] = b[q];
    __syncthreads();
  }
  for (int l = 0; l < B.nl - 1; l++) {
    const BLevel<T> &F = B.lv[l], &C = B.lv[l + 1];
    T *x = sm + F.sm, *bc = sm + C.sm + C.z.n;
    bot_smooth<T>(F, x, B.pre, true, B.omega);
    for (unsigned q = threadIdx.x; q < (unsigned)C.z.n; q += kBottomThreads)
      zrestrict_cell<T, false>(F.z, C.z, F.cpl, F.tri, F.dg, x, x + F.z.n, bc, q);
    __syncthreads();
  }
  bot_smooth<T>(B.lv[B.nl - 1], sm + B.lv[B.nl - 1].sm, B.coarse, true, B.omega);
  for (int l = B.nl - 2; l >= 0; l--) {
    const BLevel<T> &F = B.lv[l], &C = B.lv[l + 1];
    T *x = sm + F.sm;
    const bool half = F.zebra && !F.z.jp && B.post > 0;
    for (unsigned q = threadIdx.x; q < (unsigned)C.z.n; q += kBottomThreads) {
      if (half) zprolong_cell<T, true>(F.z, C.z, C.pmask, x, sm + C.sm, q);
      else zprolong_cell<T, false>(F.z, C.z, C.pmask, x, sm + C.sm, q);
    }
    __syncthreads();
    bot_smooth<T>(F, x, B.post, false, B.omega);
  }
  T *out = B.x;
  for (unsigned q = threadIdx.x; q < (unsigned)B.lv[0].z.n; q += kBottomThreads) out[q] = sm[q];
}

// ------------------------------------------------------------------ grid layout <-> columns
template <typename T, typename VT>
__global__ void __launch_bounds__(256) k_to_columns(Grid g, ZL L, DynPtrT<const VT> vv, T *b) {
  extern __shared__ __align__(16) unsigned char tile_raw[];
  T *sm = reinterpret_cast<T *>(tile_raw);
  pdl_wait();
  const VT *v = vv.get();
  const unsigned ib = tiles_i(L);
  const int k = (int)(blockIdx.x / ib), i0 = (int)(blockIdx.x % ib) * kTileI, ld = L.S | 1;
  const int a = threadIdx.x % kTileI;
  for (int j = threadIdx.x / kTileI; j < L.S; j += 256 / kTileI) {  // rows past ny: the empty slots
    T t = 0;
    if (j < L.ny && i0 + a < L.nx) t = (T)v[lidx(g, i0 + a + 1, j + 1, k + 1)];
    sm[a * ld + (int)zrow(L, j)] = t;
  }
  __syncthreads();
  for (int c = threadIdx.x >> 5; c < kTileI && i0 + c < L.nx; c += 8) {  // a warp a column
    const unsigned p0 = zcol(L, i0 + c, k);
    for (int s = threadIdx.x & 31; s < L.S; s += 32) b[p0 + s] = sm[c * ld + s];
  }
}
template <typename T, typename VT>
__global__ void __launch_bounds__(256) k_to_columns_direct(Grid g, ZL L, DynPtrT<const VT> vv, T *b) {
  pdl_wait();
  const unsigned q = blockIdx.x * blockDim.x + threadIdx.x;
  int i, j, k;
  if (q >= (unsigned)L.n || !zcell(L, q, i, j, k)) return;
  b[q] = (T)vv.get()[lidx(g, i + 1, j + 1, k + 1)];
}
// The interior points of the grid vector (the V-cycle's solution is zero off the unknowns).
template <typename T>
__global__ void __launch_bounds__(256) k_from_columns(Grid g, ZL L, const T *x, DynPtrT<T> zv) {
  extern __shared__ __align__(16) unsigned char tile_raw[];
  T *sm = reinterpret_cast<T *>(tile_raw);
  pdl_wait();
  T *z = zv.get();
  const unsigned ib = tiles_i(L);
  const int k = (int)(blockIdx.x / ib), i0 = (int)(blockIdx.x % ib) * kTileI, ld = L.S | 1;
  for (int c = threadIdx.x >> 5; c < kTileI && i0 + c < L.nx; c += 8) {  // a warp a column
    const unsigned p0 = zcol(L, i0 + c, k);
#pragma unroll 4
    for (int s = threadIdx.x & 31; s < L.S; s += 32) sm[c * ld + s] = x[p0 + s];
  }
  __syncthreads();
  const int a = threadIdx.x % kTileI;
  if (i0 + a >= L.nx) return;
  for (int j = threadIdx.x / kTileI; j < L.ny; j += 256 / kTileI)
    z[lidx(g, i0 + a + 1, j + 1, k + 1)] = sm[a * ld + (int)zrow(L, j)];
}
template <typename T>
__global__ void __launch_bounds__(256) k_from_columns_direct(Grid g, ZL L, const T *x, DynPtrT<T> zv) {
  pdl_wait();
  const unsigned q = blockIdx.x * blockDim.x + threadIdx.x;
  int i, j, k;
  if (q >= (unsigned)L.n || !zcell(L, q, i, j, k)) return;
  zv.get()[lidx(g, i + 1, j + 1, k + 1)] = x[q];
}

// ------------------------------------------------------------------ host side
// The columns of a level: 32 lanes of ceil(ny/32) rows (fewer lanes for short columns), or one
// thread a column on small levels and on coarse levels that line Jacobi smooths; their
// columns have an odd number of slots, free of shared-memory bank conflicts.
static bool two_colours(const ZL &L) { return !((L.ip && (L.nx & 1)) || (L.kp && (L.nz & 1))); }
static ZL make_zl(int nx, int ny, int nz, const Grid &g, bool finest) {
  ZL L;
  L.nx = nx; L.ny = ny; L.nz = nz;
  L.hx = (nx + 1) / 2;
  L.ip = g.iper; L.jp = g.jper; L.kp = g.kper;
  L.serial = ((long long)nx * ny * nz <= kSerialCells || (!finest && !two_colours(L) && ny <= 256)) &&
             serial_smem<double>(ny) <= kSerialSmem;  // k_zserial is the only kernel for its layout
  L.seg = L.serial ? 1 : (ny + 31) / 32;
  L.ls = L.serial ? ny | 1 : (ny + L.seg - 1) / L.seg;
  L.S = L.seg * L.ls;
  L.lwl = 0;
  while ((1 << L.lwl) < L.ls && L.lwl < 5) L.lwl++;
  L.lw = 1 << L.lwl;
  L.n = (long long)nz * 2 * L.hx * L.S;
  return L;
}

static void level_free(MGLevel &L) {
  cudaFree(L.op64); cudaFree(L.pk64); cudaFree(L.pk32); cudaFree(L.v64); cudaFree(L.v32); cudaFree(L.act);
  cudaFree(L.pmask);
  L = MGLevel();
}
void mg_free(Poisson &P) {
  for (MGLevel &L : P.lv) level_free(L);
  P.lv.clear();
}

// Per level: raw FP64 couplings and Thomas factors (op64, used to build the next level),
// the packed FP64 and FP32 operators, and the work vectors x | b | xo.  A rebuild on the
// same grid (every first time step runs PoissonLHSNew) keeps the levels' buffers.
int mg_setup(Ctx *c) {
  Poisson &P = c->ps;
  const Grid &g = c->g;
  int rc;
  std::vector<MGLevel> old;
  old.swap(P.lv);
  int nx = g.mx - 2, ny = g.my - 2, nz = g.mz - 2;
  const int maxlev = 12;
  auto fail = [&](int code, const char *msg) {
    for (size_t l = P.lv.size(); l < old.size(); l++) P.lv.push_back(old[l]);  // freed by mg_free
    return set_err(c, code, msg);
  };
  while ((int)P.lv.size() < maxlev) {
    MGLevel L;
    L.z = make_zl(nx, ny, nz, g, P.lv.empty());
    L.zebra = two_colours(L.z);
    const long long n = L.z.n;
    if (n >= (1LL << 31)) return fail(VFS_ERR_INVALID, "poisson_lhs: grid too large for the multigrid indexing");
    const size_t l = P.lv.size();
    if (l < old.size() && old[l].z.n == n && old[l].op64) {
      L.op64 = old[l].op64; L.pk64 = old[l].pk64; L.pk32 = old[l].pk32;
      L.v64 = old[l].v64; L.v32 = old[l].v32; L.act = old[l].act; L.pmask = old[l].pmask;
      old[l] = MGLevel();  // taken
    } else {
      if (l < old.size()) level_free(old[l]);
      P.alloc_epoch++;
      bool ok = cudaMalloc(&L.op64, sizeof(double) * NOP * n) == cudaSuccess;
      ok &= cudaMalloc(&L.pk64, sizeof(double) * 8 * n) == cudaSuccess;
      ok &= cudaMalloc(&L.pk32, sizeof(float) * 8 * n) == cudaSuccess;
      ok &= cudaMalloc(&L.v64, sizeof(double) * 3 * n) == cudaSuccess;
      ok &= cudaMalloc(&L.v32, sizeof(float) * 3 * n) == cudaSuccess;
      ok &= cudaMalloc(&L.act, n) == cudaSuccess;
      if (l > 0) ok &= cudaMalloc(&L.pmask, sizeof(unsigned long long) * n) == cudaSuccess;
      if (!ok) {
        level_free(L);
        return fail(VFS_ERR_CUDA, "poisson_lhs: multigrid allocation failed");
      }
    }
    cudaMemsetAsync(L.op64, 0, sizeof(double) * NOP * n, c->stream);
    cudaMemsetAsync(L.pk64, 0, sizeof(double) * 8 * n, c->stream);
    cudaMemsetAsync(L.pk32, 0, sizeof(float) * 8 * n, c->stream);
    cudaMemsetAsync(L.v64, 0, sizeof(double) * 3 * n, c->stream);
    cudaMemsetAsync(L.v32, 0, sizeof(float) * 3 * n, c->stream);
    const unsigned nb = nblocks(n, 128);
    if (P.lv.empty()) {
      const size_t smem = tile_bytes<double>(L.z);
      // the shared-memory limits are attributes of the kernels on a device
      if (cudaFuncSetAttribute(k_mg_fine_couplings, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kTileSmem) != cudaSuccess ||
          cudaFuncSetAttribute(k_mg_thomas, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kThomasSmem) != cudaSuccess) {
        P.lv.push_back(L);
        return fail(VFS_ERR_CUDA, "poisson_lhs: shared-memory limit");
      }
      if (smem <= kTileSmem)
        c->launches++, k_mg_fine_couplings<<<tiles_i(L.z) * (unsigned)nz, 256, smem, c->stream>>>(g, L.z, P.coef, P.fluid, L.op64);
      else
        c->launches++, k_mg_fine_couplings_direct<<<nb, 128, 0, c->stream>>>(g, L.z, P.coef, P.fluid, L.op64);
    } else {
      const MGLevel &F = P.lv.back();
      c->launches++, k_mg_coarse_couplings<<<nb, 128, 0, c->stream>>>(F.z, L.z, F.op64, L.op64);
    }
    if ((rc = check_launch(c, "k_mg_couplings"))) { P.lv.push_back(L); return fail(rc, "poisson_lhs: multigrid set-up failed"); }
    c->launches++, k_mg_diag<<<nb, 128, 0, c->stream>>>(L.z, L.op64, L.act);
    const unsigned ncol = (unsigned)nz * 2u * (unsigned)L.z.hx;
    const int cols = thomas_cols(L.z);
    if (cols > 0)
      c->launches++, k_mg_thomas<<<nblocks(ncol, cols), kThomasThreads, thomas_smem(L.z, cols), c->stream>>>(L.z, cols, L.op64);
    else
      c->launches++, k_mg_thomas_direct<<<nblocks(ncol, 64), 64, 0, c->stream>>>(L.z, L.op64);
    c->launches++, k_mg_pack<double><<<nb, 128, 0, c->stream>>>(L.z, L.op64, (Q4<double> *)L.pk64, (Q2<double> *)(L.pk64 + 4 * n), L.pk64 + 6 * n,
                                                                L.pk64 + 7 * n);
    c->launches++, k_mg_pack<float><<<nb, 128, 0, c->stream>>>(L.z, L.op64, (Q4<float> *)L.pk32, (Q2<float> *)(L.pk32 + 4 * n), L.pk32 + 6 * n,
                                                               L.pk32 + 7 * n);
    if (!P.lv.empty())
      c->launches++, k_mg_pmask<<<nb, 128, 0, c->stream>>>(P.lv.back().z, L.z, P.lv.back().act, L.act, L.pmask);
    P.lv.push_back(L);
    if ((rc = check_launch(c, "k_mg_setup"))) return fail(rc, "poisson_lhs: multigrid set-up failed");
    if ((nx & 1) || (ny & 1) || (nz & 1) || nx < 4 || ny < 4 || nz < 4) break;
    nx /= 2; ny /= 2; nz /= 2;
  }
  for (size_t l = P.lv.size(); l < old.size(); l++) level_free(old[l]);  // levels the new hierarchy does not reach
  return VFS_OK;
}

// Typed views of a level's packed operator and work vectors.
template <typename T>
struct LvT {
  const Q4<T> *cpl;
  const Q2<T> *tri;
  const T *cpr, *dg;
  T *x, *b, *xo;
};
template <typename T>
struct VCycle {
  Ctx *c;
  vfs_solve_opts o;
  int nl;
  LvT<T> lvt(int l) const {
    const MGLevel &L = c->ps.lv[l];
    const long long n = L.z.n;
    T *pk = sizeof(T) == 4 ? (T *)L.pk32 : (T *)L.pk64, *v = sizeof(T) == 4 ? (T *)L.v32 : (T *)L.v64;
    LvT<T> r;
    r.cpl = (const Q4<T> *)pk;
    r.tri = (const Q2<T> *)(pk + 4 * n);
    r.cpr = pk + 6 * n;
    r.dg = pk + 7 * n;
    r.x = v;
    r.b = v + n;
    r.xo = v + 2 * n;
    return r;
  }
};

static const double kJacobiOmega = 0.8;

template <typename T>
static int launch_serial(Ctx *c, const MGLevel &L, const LvT<T> &v, const T *xr, T *xw, int colour, int flags) {
  const unsigned ncol = (unsigned)L.z.nz * L.z.hx * (colour >= 0 ? 1 : 2), nb = nblocks(ncol, kSerialCols);
  const size_t smem = serial_smem<T>(L.z.ny);
  const T om = T(kJacobiOmega);
  const ZOp<T> op{v.cpl, v.tri, v.cpr};
  // the shared-memory limit is an attribute of the kernel on a device
  if (smem > 48 * 1024 &&
      (cudaFuncSetAttribute(k_zserial<T, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSerialSmem) != cudaSuccess ||
       cudaFuncSetAttribute(k_zserial<T, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSerialSmem) != cudaSuccess))
    return set_err(c, VFS_ERR_CUDA, "multigrid: shared-memory limit");
  return colour < 0 ? launch_chain(c, "k_zserial", k_zserial<T, true>, nb, kSerialThreads, smem, L.z, op, v.b, xr, xw, colour, flags, om)
                    : launch_chain(c, "k_zserial", k_zserial<T, false>, nb, kSerialThreads, smem, L.z, op, v.b, xr, xw, colour, flags, om);
}
// One colour pass, or with colour < 0 a line Jacobi sweep from xr into xw.
template <typename T>
static int launch_pass(Ctx *c, const MGLevel &L, const LvT<T> &v, const T *xr, T *xw, int colour, int flags) {
  const unsigned ncol = (unsigned)L.z.nz * L.z.hx * (colour >= 0 ? 1 : 2);
  const ZOp<T> op{v.cpl, v.tri, v.cpr};
  if (L.z.serial || (colour < 0 && serial_smem<T>(L.z.ny) <= kSerialSmem))
    return launch_serial<T>(c, L, v, xr, xw, colour, flags);
  const unsigned nb = nblocks((long long)ncol << L.z.lwl, kColThreads);
  if (colour < 0)  // columns too long for shared memory
    return launch_chain(c, "k_zlong", k_zlong<T>, nb, kColThreads, 0, L.z, op, v.b, xr, xw, flags, T(kJacobiOmega));
#define VFS_PASS(S)                                                                                                \
  case S:                                                                                                          \
    return L.z.ls == 32 ? launch_chain(c, "k_zcol", k_zcol<T, S, true>, nb, kColThreads, 0, L.z, op, v.b, xw, colour, flags) \
                        : launch_chain(c, "k_zcol", k_zcol<T, S, false>, nb, kColThreads, 0, L.z, op, v.b, xw, colour, flags);
  switch (L.z.seg) {
    VFS_PASS(1) VFS_PASS(2) VFS_PASS(3) VFS_PASS(4) VFS_PASS(5) VFS_PASS(6) VFS_PASS(7) VFS_PASS(8)
    default: break;
  }
#undef VFS_PASS
  return launch_chain(c, "k_zcol", k_zcol<T, 0, false>, nb, kColThreads, 0, L.z, op, v.b, xw, colour, flags);
}

// `sweeps` smoothing sweeps on level l; x_zero: x is taken as zero on entry.
template <typename T>
static int mg_smooth(const VCycle<T> &V, int l, int sweeps, bool x_zero) {
  Ctx *c = V.c;
  const MGLevel &L = c->ps.lv[l];
  const LvT<T> v = V.lvt(l);
  int rc = VFS_OK;
  if (L.zebra) {
    for (int s = 0; s < sweeps; s++)
      for (int col = 0; col < 2; col++) {
        const bool z = x_zero && s == 0;
        const int flags = (z ? Z_OWN_ZERO : 0) | (z && col == 0 ? Z_NB_ZERO : 0);
        if ((rc = launch_pass<T>(c, L, v, v.x, v.x, col, flags))) return rc;
      }
    return rc;
  }
  T *from = x_zero ? v.xo : v.x, *to = x_zero ? v.x : v.xo;  // from zero nothing is read
  for (int s = 0; s < sweeps; s++) {
    if ((rc = launch_pass<T>(c, L, v, from, to, -1, x_zero && s == 0 ? Z_NB_ZERO | Z_OWN_ZERO : 0))) return rc;
    std::swap(from, to);
  }
  if (from != v.x && cudaMemcpyAsync(v.x, from, sizeof(T) * L.z.n, cudaMemcpyDeviceToDevice, c->stream) != cudaSuccess)
    return set_err(c, VFS_ERR_CUDA, "multigrid: copy failed");
  return rc;
}

// Shared memory of the bottom kernel from level l (x, b, the previous x and the operator of every level).
template <typename T>
static size_t bottom_smem(const VCycle<T> &V, int l) {
  long long n = 0;
  for (int q = l; q < V.nl; q++) n += V.c->ps.lv[q].z.n;
  return sizeof(T) * 10 * (size_t)n;
}
template <typename T>
static bool bottom_fits(const VCycle<T> &V, int l) {
  const ZL &z = V.c->ps.lv[l].z;
  return (long long)z.nx * z.ny * z.nz <= kSerialCells && V.nl - l <= kBottomMaxLevels &&
         bottom_smem<T>(V, l) <= kBottomSmem;
}
template <typename T>
static int mg_bottom(const VCycle<T> &V, int l) {
  Ctx *c = V.c;
  Bottom<T> B;
  B.nl = V.nl - l;
  B.pre = V.o.pre_smooth; B.post = V.o.post_smooth; B.coarse = V.o.coarse_iters;
  B.omega = T(kJacobiOmega);
  const LvT<T> top = V.lvt(l);
  B.x = top.x;
  B.b = top.b;
  unsigned at = 0;
  for (int q = 0; q < B.nl; q++) {
    const MGLevel &L = c->ps.lv[l + q];
    const LvT<T> v = V.lvt(l + q);
    BLevel<T> &d = B.lv[q];
    d.z = L.z;
    d.pmask = L.pmask;
    d.cpl = v.cpl; d.tri = v.tri; d.cpr = v.cpr; d.dg = v.dg;
    d.sm = at;
    at += 10u * (unsigned)L.z.n;
    d.zebra = L.zebra ? 1 : 0;
  }
  const size_t smem = bottom_smem<T>(V, l);
  // the shared-memory limit is an attribute of the kernel on a device
  if (smem > 48 * 1024 &&
      cudaFuncSetAttribute(k_mg_bottom<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kBottomSmem) != cudaSuccess)
    return set_err(c, VFS_ERR_CUDA, "k_mg_bottom: shared-memory limit");
  return launch_chain(c, "k_mg_bottom", k_mg_bottom<T>, 1, kBottomThreads, smem, B);
}

// V-cycle from level l (its right-hand side already in place); levels at or below
// kSerialCells run inside one thread block.
template <typename T>
static int mg_vcycle(const VCycle<T> &V, int l) {
  Ctx *c = V.c;
  int rc;
  if (bottom_fits<T>(V, l)) return mg_bottom<T>(V, l);
  if (l == V.nl - 1) return mg_smooth<T>(V, l, V.o.coarse_iters, true);
  if ((rc = mg_smooth<T>(V, l, V.o.pre_smooth, true))) return rc;
  const MGLevel &F = c->ps.lv[l], &C = c->ps.lv[l + 1];
  const LvT<T> f = V.lvt(l), cc = V.lvt(l + 1);
  const unsigned nb = nblocks(C.z.n, 128);
  // one colour of a zebra level without periodic j is enough for either transfer
  const bool half = F.zebra && !F.z.jp;
  rc = colour0_restriction(F.z, F.zebra) ? launch_chain(c, "k_zrestrict", k_zrestrict<T, true>, nb, 128, 0, F.z, C.z, f.cpl, f.tri, f.dg, f.x, f.b, cc.b)
            : launch_chain(c, "k_zrestrict", k_zrestrict<T, false>, nb, 128, 0, F.z, C.z, f.cpl, f.tri, f.dg, f.x, f.b, cc.b);
  if (rc) return rc;
  if ((rc = mg_vcycle<T>(V, l + 1))) return rc;
  if (half && V.o.post_smooth > 0 && (long long)F.z.nx * F.z.ny * F.z.nz <= kFineProlong)
    rc = launch_chain(c, "k_zprolong", k_zprolong_fine<T>, nblocks((long long)F.z.nz * F.z.hx * F.z.S, 128), 128, 0, F.z, C.z,
                      C.pmask, f.x, cc.x);
  else
    rc = half && V.o.post_smooth > 0
             ? launch_chain(c, "k_zprolong", k_zprolong<T, true>, nb, 128, 0, F.z, C.z, C.pmask, f.x, cc.x)
             : launch_chain(c, "k_zprolong", k_zprolong<T, false>, nb, 128, 0, F.z, C.z, C.pmask, f.x, cc.x);
  if (rc) return rc;
  return mg_smooth<T>(V, l, V.o.post_smooth, false);
}

template <typename T, typename VT>
static int mg_apply(Ctx *c, DynPtrT<const VT> b, DynPtrT<T> x, const vfs_solve_opts &o) {
  const int nl = o.levels > 0 ? std::min((int)c->ps.lv.size(), o.levels) : (int)c->ps.lv.size();
  const VCycle<T> V{c, o, nl};
  const ZL &L = c->ps.lv[0].z;
  const LvT<T> l0 = V.lvt(0);
  const size_t smem = tile_bytes<T>(L);
  const bool tiled = smem <= kTileSmem;
  const unsigned nt = tiles_i(L) * (unsigned)L.nz, nd = nblocks(L.n, 256);
  int rc;
  // the shared-memory limit is an attribute of the kernel on a device
  if (tiled && smem > 48 * 1024 &&
      (cudaFuncSetAttribute(k_to_columns<T, VT>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kTileSmem) != cudaSuccess ||
       cudaFuncSetAttribute(k_from_columns<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kTileSmem) != cudaSuccess))
    return set_err(c, VFS_ERR_CUDA, "multigrid: shared-memory limit");
  rc = tiled ? launch_chain(c, "k_to_columns", k_to_columns<T, VT>, nt, 256, smem, c->g, L, b, l0.b)
             : launch_chain(c, "k_to_columns", k_to_columns_direct<T, VT>, nd, 256, 0, c->g, L, b, l0.b);
  if (rc || (rc = mg_vcycle<T>(V, 0))) return rc;
  return tiled ? launch_chain(c, "k_from_columns", k_from_columns<T>, nt, 256, smem, c->g, L, l0.x, x)
               : launch_chain(c, "k_from_columns", k_from_columns_direct<T>, nd, 256, 0, c->g, L, l0.x, x);
}

int mg_precondition(Ctx *c, DynPtrT<const double> b, DynPtrT<float> x, const vfs_solve_opts &o) { return mg_apply<float>(c, b, x, o); }
int mg_precondition(Ctx *c, DynPtrT<const double> b, DynPtrT<double> x, const vfs_solve_opts &o) { return mg_apply<double>(c, b, x, o); }
int mg_precondition(Ctx *c, DynPtrT<const float> b, DynPtrT<float> x, const vfs_solve_opts &o) { return mg_apply<float>(c, b, x, o); }

// One smoothing sweep of the finest level (both colours), for timing.
int mg_sweep_fine(Ctx *c, int precision) {
  const vfs_solve_opts o = {};
  return precision == 0 ? mg_smooth<float>(VCycle<float>{c, o, 1}, 0, 1, false) : mg_smooth<double>(VCycle<double>{c, o, 1}, 0, 1, false);
}

}  // namespace vfs

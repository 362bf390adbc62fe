// sx_factor.cu -- GPU set-up of a DIRECT or JACPCG system (MatrixSys).
//
// DIRECT (src/matrix.cpp:175-274):
//   1. k_elem_condense: one CTA per element and system builds the elemental Helmholtz
//      matrix in edge-major order (Element::HelmholtzRow,
//      src/element.cpp:1439-1509), inverts the interior block (the reference
//      uses getrf+getri, src/element.cpp:212-216; hii is SPD here so
//      Gauss-Jordan without pivoting is used) and condenses
//      hbb -= hbi hii^-1 hib, hbi <- hbi hii^-1 (src/element.cpp:218-220).
//   2. k_band_add: direct-stiffness assembly of hbb into the banded matrix,
//      one element colour per launch so no two CTAs touch the same entry
//      (deterministic; src/matrix.cpp:236-241).  Mixed-BC diagonal terms
//      follow in boundary order (Mixed::augmentSC, src/condition.cpp:347-381).
//   3. Tiled right-looking banded Cholesky, A = U^T U (LAPACK dpbtrf "U",
//      src/matrix.cpp:259): per block column k, k_trsm forms the off-diagonal
//      tiles of block row k, k_update applies the trailing rank-nb update
//      inside the band and factors the next diagonal tile.  All systems of a
//      batch share each launch.
//      What is kept is the block LDL^T form of the same factor: the diagonal
//      tiles U_kk, their inverses D_k, and off the diagonal U_kk^-1 U(k, k+i)
//      in place of U(k, k+i), so that the sweeps' block-column chains carry
//      no diagonal solve (sx_band.cu).
// JACPCG (src/matrix.cpp:276-317): k_elem_diag + k_diag_dss.
#include <cmath>
#include <cstring>
#include <mutex>

#include "sx_internal.h"
#include "sx_kernels.cuh"
#include "sx_ptx.cuh"

namespace sx {

// ---------------------------------------------------------------------------
// Element matrix + static condensation
// ---------------------------------------------------------------------------

// One system of a batched build: every launch covers all of them (blockIdx.y).
struct BuildDesc {
  double hCon;
  double *hbi, *hii, *hbb, *tiles;
  int *status;
  int nsolve, nblk, J;
};

// Shared rows are PI doubles apart (odd: row and column walks are free of bank
// conflicts).
template <int NP>
struct Condense {
  static constexpr int NN = NP * NP, NE = 4 * (NP - 1), NI = NN - NE, PI = NI | 1;
  static constexpr int AE = (NE + 15) / 16, AI = (NI + 15) / 16;  // rows of a thread: ty, ty + 16, ...
  static constexpr int WORK = 5 * NN > NI * PI ? 5 * NN : NI * PI;
  // hbi | t | D, Q1..Q4 and later hii | pivot row and column, two buffers each
  static constexpr size_t smem = sizeof(double) * (2 * (size_t)NE * PI + WORK + 4 * 16 * AI);
  static constexpr int blocks = NP <= 8 ? 4 : NP <= 11 ? 2 : 1;  // an SM: shared memory and registers
};

// The element's matrix and its condensation, one block of 16 x 16 threads per
// (element, system).  Thread (ty, tx) keeps the entries (ty + 16 a, tx + 16 b)
// of hii and of hbb in registers: the Gauss-Jordan steps exchange the pivot row
// and column through shared memory (one barrier a step, two buffers), and the
// two products that follow reuse each value they read AE or AI times.  What
// bounded the form before this (entries in shared memory, an index division and
// four shared-memory accesses per entry and step) was instruction issue: ten
// systems of 851 elements of order 7, 1.52 ms in ten launches -> 0.56 ms in one.
template <int NP>
__global__ void __launch_bounds__(256, Condense<NP>::blocks)
    k_elem_condense(MeshView M, const BuildDesc *__restrict__ desc) {
  using C = Condense<NP>;
  constexpr int NN = C::NN, NE = C::NE, NI = C::NI, PI = C::PI, AE = C::AE, AI = C::AI;
  const BuildDesc B = desc[blockIdx.y];
  extern __shared__ double sm[];
  double *hbi = sm, *t = hbi + NE * PI, *hii = t + NE * PI, *rowb = hii + C::WORK, *colb = rowb + 2 * 16 * AI;
  double *D = hii, *Q1 = D + NN, *Q2 = Q1 + NN, *Q3 = Q2 + NN, *Q4 = Q3 + NN;  // until the inverse is there
  __shared__ int emap[NN];
  const int e = blockIdx.x, tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
  const size_t eo = (size_t)e * NN;
  for (int i = tid; i < NN; i += 256) {
    D[i] = M.D[i];
    Q1[i] = M.Q1[eo + i];
    Q2[i] = M.Q2[eo + i];
    Q3[i] = M.Q3[eo + i];
    Q4[i] = M.Q4[eo + i];
    emap[i] = M.emap[i];
  }
  __syncthreads();
  const bool q3 = M.hasQ3[e];
  // Entry H[(i,j),(m,n)] of the elemental matrix in edge-major order,
  // accumulated in the order of HelmholtzRow: Q1 term, Q2 term, the two Q3
  // terms, then Q4*hCon.
  auto entry = [&](int a, int b) {
    const int r = emap[a], c = emap[b];
    const int i = r / NP, j = r - i * NP, m = c / NP, n = c - m * NP;
    double h = 0.0;
    if (m == i) {
      double s = 0.0;
#pragma unroll
      for (int q = 0; q < NP; q++) s += Q1[i * NP + q] * (D[q * NP + j] * D[q * NP + n]);
      h = s;
    }
    if (n == j) {
      double s = 0.0;
#pragma unroll
      for (int p = 0; p < NP; p++) s += Q2[p * NP + j] * (D[p * NP + i] * D[p * NP + m]);
      h += s;
    }
    if (q3) {
      h += Q3[i * NP + n] * D[n * NP + j] * D[i * NP + m];
      h += Q3[m * NP + j] * D[j * NP + n] * D[m * NP + i];
    }
    if (m == i && n == j) h += Q4[i * NP + j] * B.hCon;
    return h;
  };
  double hb[AE][AE], v[AI][AI];
#pragma unroll
  for (int a = 0; a < AE; a++) {
    const int r = ty + 16 * a;
#pragma unroll
    for (int b = 0; b < AE; b++) hb[a][b] = r < NE && tx + 16 * b < NE ? entry(r, tx + 16 * b) : 0.0;
#pragma unroll
    for (int b = 0; b < AI; b++) {
      const int c = tx + 16 * b;
      if (r < NE && c < NI) hbi[r * PI + c] = entry(r, NE + c);
    }
  }
#pragma unroll
  for (int a = 0; a < AI; a++)
#pragma unroll
    for (int b = 0; b < AI; b++)
      v[a][b] = ty + 16 * a < NI && tx + 16 * b < NI ? entry(NE + ty + 16 * a, NE + tx + 16 * b) : 0.0;
  // In-place Gauss-Jordan inverse of the SPD interior block.
  int bad = 0;
#pragma unroll
  for (int ka = 0; ka < AI; ka++) {
    for (int kk = 0; kk < 16; kk++) {
      const int k = 16 * ka + kk;
      if (k >= NI) break;
      double *rk = rowb + (k & 1) * 16 * AI, *ck = colb + (k & 1) * 16 * AI;
      if (ty == kk)
#pragma unroll
        for (int b = 0; b < AI; b++) rk[tx + 16 * b] = v[ka][b];
      if (tx == kk)
#pragma unroll
        for (int a = 0; a < AI; a++) ck[ty + 16 * a] = v[a][ka];
      __syncthreads();
      const double p = rk[k];
      // a zero (or NaN) pivot: hii is singular (src/element.cpp:212-216); a
      // negative one: hii, a principal block of H, is not positive definite,
      // so neither is H -- the reference's getrf/getri go on with an
      // indefinite hii and its dpbtrf then fails (src/matrix.cpp:259-261)
      bad |= (p < 0.0) ? 2 : (!(p > 0.0) ? 1 : 0);
      const double rp = (p != 0.0 && p == p) ? 1.0 / p : 1.0;
      double x[AI], y[AI];
#pragma unroll
      for (int b = 0; b < AI; b++) x[b] = (tx + 16 * b == k ? 1.0 : rk[tx + 16 * b]) * rp;
#pragma unroll
      for (int a = 0; a < AI; a++) y[a] = ck[ty + 16 * a];
#pragma unroll
      for (int a = 0; a < AI; a++)
#pragma unroll
        for (int b = 0; b < AI; b++)
          v[a][b] = ty + 16 * a == k ? x[b] : (tx + 16 * b == k ? 0.0 : v[a][b]) - y[a] * x[b];
    }
  }
  // every thread is past its reads of D and Q (the barriers above; NI >= 1)
#pragma unroll
  for (int a = 0; a < AI; a++)
#pragma unroll
    for (int b = 0; b < AI; b++)
      if (ty + 16 * a < NI && tx + 16 * b < NI) hii[(ty + 16 * a) * PI + tx + 16 * b] = v[a][b];
  __syncthreads();
  // t = hbi * hii^-1
  {
    double s[AE][AI];
#pragma unroll
    for (int a = 0; a < AE; a++)
#pragma unroll
      for (int b = 0; b < AI; b++) s[a][b] = 0.0;
    for (int q = 0; q < NI; q++) {
      double x[AE], y[AI];
#pragma unroll
      for (int a = 0; a < AE; a++) x[a] = hbi[min(ty + 16 * a, NE - 1) * PI + q];
#pragma unroll
      for (int b = 0; b < AI; b++) y[b] = hii[q * PI + min(tx + 16 * b, NI - 1)];
#pragma unroll
      for (int a = 0; a < AE; a++)
#pragma unroll
        for (int b = 0; b < AI; b++) s[a][b] += x[a] * y[b];
    }
#pragma unroll
    for (int a = 0; a < AE; a++)
#pragma unroll
      for (int b = 0; b < AI; b++)
        if (ty + 16 * a < NE && tx + 16 * b < NI) t[(ty + 16 * a) * PI + tx + 16 * b] = s[a][b];
  }
  __syncthreads();
  // hbb -= t * hbi^T
  double *oh = B.hbb + (size_t)e * NE * NE;
  {
    double s[AE][AE];
#pragma unroll
    for (int a = 0; a < AE; a++)
#pragma unroll
      for (int b = 0; b < AE; b++) s[a][b] = 0.0;
    for (int q = 0; q < NI; q++) {
      double x[AE], y[AE];
#pragma unroll
      for (int a = 0; a < AE; a++) {
        x[a] = t[min(ty + 16 * a, NE - 1) * PI + q];
        y[a] = hbi[min(tx + 16 * a, NE - 1) * PI + q];
      }
#pragma unroll
      for (int a = 0; a < AE; a++)
#pragma unroll
        for (int b = 0; b < AE; b++) s[a][b] += x[a] * y[b];
    }
#pragma unroll
    for (int a = 0; a < AE; a++)
#pragma unroll
      for (int b = 0; b < AE; b++) {
        const int r = ty + 16 * a, c = tx + 16 * b;
        if (r < NE && c < NE) oh[r * NE + c] = hb[a][b] - s[a][b];
      }
  }
  double *ob = B.hbi + (size_t)e * NE * NI;
  for (int o = tid; o < NE * NI; o += 256) ob[o] = t[(o / NI) * PI + o % NI];
  double *oi = B.hii + (size_t)e * NI * NI;
  // column-major, (r, c) at c * nint + r: the back-substitution's threads
  // own rows and read a column per step
  for (int o = tid; o < NI * NI; o += 256) oi[o] = hii[(o % NI) * PI + o / NI];
  if (tid == 0 && bad)
    atomicOr(B.status, ((bad & 1) ? 1 << SX_ERR_SINGULAR_HII : 0) | ((bad & 2) ? 1 << SX_ERR_NOT_SPD : 0));
}

// ---------------------------------------------------------------------------
// Band assembly into tiles
// ---------------------------------------------------------------------------

// Identity rows past the last solve node (fewer than NB), and the status word.
__global__ void k_band_init(const BuildDesc *__restrict__ desc) {
  const BuildDesc B = desc[blockIdx.y];
  if (threadIdx.x == 0) *B.status = 0;
  const int g = B.nsolve + threadIdx.x;
  if (g >= B.nblk * NB) return;
  const int b = g / NB, r = g - b * NB;
  B.tiles[((size_t)b * (B.J + 1)) * TSZ + (size_t)r * LDT + r] = 1.0;
}

__global__ void k_band_add(MeshView M, const int *__restrict__ elems, const BuildDesc *__restrict__ desc) {
  const BuildDesc B = desc[blockIdx.y];
  const int e = elems[blockIdx.x];
  const int next = M.next, kd = M.nband - 1;
  const int *bt = M.btog + (size_t)e * next;
  const double *h = B.hbb + (size_t)e * next * next;
  for (int idx = threadIdx.x; idx < next * next; idx += blockDim.x) {
    const int i = idx / next, k = idx - i * next;
    const int m = bt[i], n = bt[k];
    if (m < B.nsolve && n < B.nsolve && n >= m) {
      if (n - m > kd) {
        atomicOr(B.status, 1 << SX_ERR_BAND);
        continue;
      }
      B.tiles[tile_addr(m, n, B.J)] += h[idx];
    }
  }
}

// Mixed::augmentSC in boundary order (one thread: tiny, order-preserving).
__global__ void k_band_mixed(MeshView M, const BuildDesc *__restrict__ desc) {
  if (threadIdx.x) return;
  const BuildDesc B = desc[blockIdx.y];
  const int np = M.np, nm = np - 1;
  for (int b = 0; b < M.nbound; b++) {
    if (M.b_kind[b] != SX_BC_MIXED) continue;
    const int *bmap = M.btog + (size_t)M.b_elmt[b] * M.next;
    const int side = M.b_side[b];
    const double K = M.b_K[b];
    const double *area = M.b_area + (size_t)b * np;
    for (int i = 0; i < nm; i++) {
      const int k = bmap[side * nm + i];
      if (k < B.nsolve) B.tiles[tile_addr(k, k, B.J)] += K * area[i];
    }
    const int i = (side == 3) ? bmap[0] : bmap[side * nm + nm];
    if (i < B.nsolve) B.tiles[tile_addr(i, i, B.J)] += K * area[nm];
  }
}

// ---------------------------------------------------------------------------
// Tiled banded Cholesky
// ---------------------------------------------------------------------------

// Tile products on the FP64 tensor cores (mma.sync m8n8k4, f64).  The two
// factor tiles of a product are staged into shared memory with rows padded
// to LDM = 68 doubles (68 = 4 mod 16: the 4 x 8 slab a fragment reads, rows
// t = 0..3 and columns g = 0..7, falls on 16 distinct bank pairs in each
// half-warp).  Warp w owns rows 16 (w / 2) .. +16 and columns 32 (w % 2) ..
// +32 of the 64 x 64 result: 2 x 4 blocks of 8 x 8, two accumulators a
// thread each, held in registers from the first product to the store.
constexpr int LDM = NB + 4;

__device__ __forceinline__ void tile_stage_mma(double *dst, const double *__restrict__ src) {
  for (int idx = threadIdx.x; idx < NB * NB / 2; idx += blockDim.x) {
    const int r = idx >> 5, c = 2 * (idx & (NB / 2 - 1));
    cp_async16_cg(dst + r * LDM + c, src + r * LDT + c);
  }
}

struct MmaAcc {
  double v[2][4][2];
};

// This thread's result elements: (row r0 + 8m + g, column c0 + 8n + 2t + q).
__device__ __forceinline__ void mma_coords(int &r0, int &c0, int &g, int &t) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  g = lane >> 2;
  t = lane & 3;
  r0 = (w >> 1) * 16;
  c0 = (w & 1) * 32;
}

__device__ __forceinline__ void mma_f64(double &d0, double &d1, double a, double b) {
  asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};"
               : "+d"(d0), "+d"(d1)
               : "d"(a), "d"(b));
}

// acc += A^T B over the staged tiles: entry (r, c) gains sum_l A[l][r] B[l][c].
__device__ __forceinline__ void mma_tile(MmaAcc &acc, const double *As, const double *Bs) {
  int r0, c0, g, t;
  mma_coords(r0, c0, g, t);
#pragma unroll 4
  for (int l0 = 0; l0 < NB; l0 += 4) {
    const double *Ar = As + (l0 + t) * LDM + r0 + g;
    const double *Br = Bs + (l0 + t) * LDM + c0 + g;
    double a[2], b[4];
#pragma unroll
    for (int m = 0; m < 2; m++) a[m] = Ar[8 * m];
#pragma unroll
    for (int n = 0; n < 4; n++) b[n] = Br[8 * n];
#pragma unroll
    for (int m = 0; m < 2; m++)
#pragma unroll
      for (int n = 0; n < 4; n++) mma_f64(acc.v[m][n][0], acc.v[m][n][1], a[m], b[n]);
  }
}

__device__ __forceinline__ void mma_zero(MmaAcc &acc) {
#pragma unroll
  for (int m = 0; m < 2; m++)
#pragma unroll
    for (int n = 0; n < 4; n++) acc.v[m][n][0] = acc.v[m][n][1] = 0.0;
}

// T -= acc at this thread's result elements (one subtraction each, after
// the whole product: the order of the reference's blocked update, C - A^T B
// with the product formed first).
__device__ __forceinline__ void mma_sub(double *T, const MmaAcc &acc) {
  int r0, c0, g, t;
  mma_coords(r0, c0, g, t);
#pragma unroll
  for (int m = 0; m < 2; m++)
#pragma unroll
    for (int n = 0; n < 4; n++) {
      double2 *q = reinterpret_cast<double2 *>(&T[(r0 + 8 * m + g) * LDT + c0 + 8 * n + 2 * t]);
      const double2 v = *q;
      *q = make_double2(v.x - acc.v[m][n][0], v.y - acc.v[m][n][1]);
    }
}

// C -= A^T A over the staged tiles, in the 8 x 8 blocks of the upper triangle:
// a block row a warp (N blocks, the last N of the row), long and short rows
// paired on a scheduler.  The same sums as mma_tile and mma_sub.
template <int N>
__device__ __forceinline__ void syrk_row(double *C, const double *A) {
  const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  constexpr int R = NB - 8 * N;  // first row, and first column
  double v[N][2];
#pragma unroll
  for (int n = 0; n < N; n++) v[n][0] = v[n][1] = 0.0;
#pragma unroll 4
  for (int l0 = 0; l0 < NB; l0 += 4) {
    const double *q = A + (l0 + t) * LDM + R + g;
    double b[N];
#pragma unroll
    for (int n = 0; n < N; n++) b[n] = q[8 * n];
#pragma unroll
    for (int n = 0; n < N; n++) mma_f64(v[n][0], v[n][1], b[0], b[n]);
  }
#pragma unroll
  for (int n = 0; n < N; n++) {
    double2 *q = reinterpret_cast<double2 *>(&C[(R + g) * LDM + R + 8 * n + 2 * t]);
    const double2 c = *q;
    *q = make_double2(c.x - v[n][0], c.y - v[n][1]);
  }
}
__device__ __forceinline__ void syrk_sub(double *C, const double *A) {
  switch (threadIdx.x >> 5) {
    case 0: return syrk_row<8>(C, A);
    case 1: return syrk_row<7>(C, A);
    case 2: return syrk_row<6>(C, A);
    case 3: return syrk_row<5>(C, A);
    case 4: return syrk_row<1>(C, A);
    case 5: return syrk_row<2>(C, A);
    case 6: return syrk_row<3>(C, A);
    case 7: return syrk_row<4>(C, A);
  }
}

// One 8 x 8 block of op(A) B over rows l of the staged tiles, l in [l0, l1)
// (multiples of 4), added to (d0, d1): row r + lane / 4, columns c +
// 2 (lane % 4) + {0, 1}.
template <bool TRANS>
__device__ __forceinline__ void mma_block8(double &d0, double &d1, const double *A, const double *B, int r, int c,
                                           int l0, int l1) {
  const int g = (threadIdx.x & 31) >> 2, t = threadIdx.x & 3;
  for (int l = l0; l < l1; l += 4)
    mma_f64(d0, d1, TRANS ? A[(l + t) * LDM + r + g] : A[(r + g) * LDM + l + t], B[(l + t) * LDM + c + g]);
}

// Factor the diagonal tile of block column k, A = U^T U (upper), staged in
// shared memory (pitch LDM), and form D_k = U^-1 in X: one CTA of eight warps
// per system, the serial link between the block columns of a factorisation.
// What bounds it is the chain of 64 pivots, so the pivots' steps stay in
// registers:
//   Cholesky by panels of 16 rows.  A warp holds the panel's 16 diagonal
//   columns in its lower lanes and 16 columns to the right in its upper ones,
//   16 rows a lane.  Pivots go by fours: every lane takes the 4 x 4 diagonal
//   block by shuffles and factors it (the same numbers), so that the chain
//   from pivot to pivot is a square root and two products, then solves its own
//   column's four rows and takes them out of the rows below, with one shuffle
//   per element of the pivot rows, all independent.  The trailing tile is then
//   updated on the FP64 tensor cores.
//   Inverse: the four 16 x 16 diagonal blocks by back-substitution, a lane a
//   column, then [A B; 0 C]^-1 = [A^-1, -A^-1 B C^-1; 0, C^-1] at 16 and 32
//   on the tensor cores.
// Cycles of a diagonal tile (10 systems, other tiles being updated beside it):
// 36,600 with one pivot a step -> 29,300; a factorisation of theirs with its
// solve 10.1 -> 9.4 ms.
__device__ __forceinline__ void factor_diag(const SysDesc &S, int k, double *A, double *X, double *rinv) {
  constexpr int PW = 16, NP4 = NB / PW, MB = 4;  // panel width, panels, pivots a step
  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5, g = lane >> 2, t = lane & 3;
  bool bad = false;
  for (int p = 0; p < NP4; p++) {
    const int c0 = p * PW, right = NP4 - 1 - p;  // 16-column groups right of the panel
    const int j = lane & (PW - 1);
    const bool busy = w < max(1, right), diag = lane < PW || right == 0;
    const int col = diag ? c0 + j : c0 + PW * (w + 1) + j;
    const bool mine = diag ? w == 0 && lane < PW : true;
    double a[PW];
    if (busy)
#pragma unroll
      for (int i = 0; i < PW; i++) a[i] = A[(c0 + i) * LDM + col];
    __syncthreads();  // every warp has the diagonal columns
    if (busy) {
#pragma unroll
      for (int c = 0; c < PW; c += MB) {
        double d[MB][MB], u[MB];  // d: the rows of U in the block, above its diagonal
#pragma unroll
        for (int k = 0; k < MB; k++)
#pragma unroll
          for (int i = 0; i <= k; i++) d[i][k] = __shfl_sync(0xffffffffu, a[c + i], c + k);
#pragma unroll
        for (int m = 0; m < MB; m++) {
          const double x = d[m][m], r = rsqrt(x);
          bad |= !(x > 0.0);  // (the NaN that follow stay in this factor)
#pragma unroll
          for (int k = m + 1; k < MB; k++) d[m][k] *= r;
#pragma unroll
          for (int i = m + 1; i < MB; i++)
#pragma unroll
            for (int k = i; k < MB; k++) d[i][k] = fma(-d[m][i], d[m][k], d[i][k]);
          double v = a[c + m];
#pragma unroll
          for (int l = 0; l < m; l++) v = fma(-d[l][m], u[l], v);
          u[m] = v * r;
          const double q = x * r;  // sqrt(x), with one Newton step
          if (mine) {
            const int row = c + m;
            A[(c0 + row) * LDM + col] = !diag || j > row ? u[m] : j == row ? fma(0.5 * r, fma(-q, q, x), q) : 0.0;
          }
          if (w == 0 && lane == 0) rinv[c0 + c + m] = r;
        }
#pragma unroll
        for (int i = c + MB; i < PW; i++)
#pragma unroll
          for (int m = 0; m < MB; m++) a[i] = fma(-__shfl_sync(0xffffffffu, u[m], i), u[m], a[i]);
      }
    }
    __syncthreads();
    // A(r, c) -= sum over the panel's rows of U(l, r) U(l, c), r <= c
    const int n8 = right * (PW / 8), base = c0 + PW;
    for (int idx = w; idx < n8 * (n8 + 1) / 2; idx += 8) {
      int bj = 0, o = idx;
      while (o > bj) o -= ++bj;  // block column bj holds block rows 0..bj
      const int r = base + 8 * o, c = base + 8 * bj;
      double d0 = 0.0, d1 = 0.0;
      mma_block8<true>(d0, d1, A, A, r, c, c0, c0 + PW);
      double *q = &A[(r + g) * LDM + c + 2 * t];
      q[0] -= d0;
      q[1] -= d1;
    }
    __syncthreads();
  }
  // inverses of the diagonal blocks: column j of block w
  if (w < NP4) {
    const int c0 = w * PW, j = lane & (PW - 1);
    double s[PW];
#pragma unroll
    for (int i = 0; i < PW; i++) s[i] = 0.0;
#pragma unroll
    for (int i = PW - 1; i >= 0; i--) {
      const double r = rinv[c0 + i], x = i == j ? r : i < j ? -s[i] * r : 0.0;
#pragma unroll
      for (int m = 0; m < i; m++) s[m] = fma(A[(c0 + m) * LDM + c0 + i], x, s[m]);
      if (lane < PW) X[(c0 + i) * LDM + c0 + j] = x;
    }
  }
  __syncthreads();
  // off-diagonal blocks of width h; the product U_12 X_22 waits in X's lower
  // triangle, which is stored as zeros
  for (int h = PW; h < NB; h *= 2) {
    const int nb = h / 8, per = nb * nb, npair = NB / (2 * h);
    for (int half = 0; half < 2; half++) {
      for (int idx = w; idx < npair * per; idx += 8) {
        const int c0 = (idx / per) * 2 * h, o = idx % per, rb = 8 * (o / nb), cb = 8 * (o % nb);
        double d0 = 0.0, d1 = 0.0;
        if (half == 0) {  // U_12 X_22, X_22 upper triangular
          mma_block8<false>(d0, d1, A, X, c0 + rb, c0 + h + cb, c0 + h, c0 + h + cb + 8);
          double *q = &X[(c0 + h + rb + g) * LDM + c0 + cb + 2 * t];
          q[0] = d0;
          q[1] = d1;
        } else {  // -X_11 (U_12 X_22), X_11 upper triangular
          mma_block8<false>(d0, d1, X, X + h * LDM, c0 + rb, c0 + cb, c0 + rb, c0 + h);
          double *q = &X[(c0 + rb + g) * LDM + c0 + h + cb + 2 * t];
          q[0] = -d0;
          q[1] = -d1;
        }
      }
      __syncthreads();
    }
  }
  double *T = S.tiles + ((size_t)k * (S.J + 1)) * TSZ, *D = S.dinv + (size_t)k * TSZ;
  for (int idx = tid; idx < NB * NB / 2; idx += 256) {
    const int i = idx / (NB / 2), j = 2 * (idx % (NB / 2));
    const double2 u = *reinterpret_cast<const double2 *>(&A[i * LDM + j]);
    const double2 x = *reinterpret_cast<const double2 *>(&X[i * LDM + j]);
    reinterpret_cast<double2 *>(T)[idx] = make_double2(j < i ? 0.0 : u.x, j + 1 < i ? 0.0 : u.y);
    reinterpret_cast<double2 *>(D)[idx] = make_double2(j < i ? 0.0 : x.x, j + 1 < i ? 0.0 : x.y);
  }
  if (bad && lane == 0) atomicOr(S.status, 1 << SX_ERR_NOT_SPD);
}

// Half a tile's product with D (X, upper triangular): columns c .. c + 15 of
// D^T B (TRANS) or D B in the 8-row strips q and 7 - q, whose ranges of nonzero
// terms add up to the same for every warp.
template <bool TRANS>
__device__ __forceinline__ void tri_mma(double (&v)[2][2][2], const double *X, const double *B, int q, int c) {
  const int g = (threadIdx.x & 31) >> 2, t = threadIdx.x & 3;
#pragma unroll
  for (int m = 0; m < 2; m++)
#pragma unroll
    for (int n = 0; n < 2; n++) v[m][n][0] = v[m][n][1] = 0.0;
  const int l1 = TRANS ? 8 * (8 - q) : NB;
#pragma unroll 2
  for (int l0 = TRANS ? 0 : 8 * q; l0 < l1; l0 += 4) {
    const double *b = B + (l0 + t) * LDM + c + g;
    const double b0 = b[0], b1 = b[8];
#pragma unroll
    for (int m = 0; m < 2; m++) {
      const int r = m == 0 ? 8 * q : 8 * (7 - q);
      if (TRANS ? m == 1 || l0 < r + 8 : m == 0 || l0 >= r) {
        const double a = TRANS ? X[(l0 + t) * LDM + r + g] : X[(r + g) * LDM + l0 + t];
        mma_f64(v[m][0][0], v[m][0][1], a, b0);
        mma_f64(v[m][1][0], v[m][1][1], a, b1);
      }
    }
  }
}

// Off-diagonal tiles of block row k inside the envelope (i <= jb[k]; the
// others stay zero): U(k, k+i) = U_kk^-T A(k, k+i) into the row buffer, which
// the trailing update reads (J tiles: they stay in L2), and U_kk^-1 U(k, k+i)
// (scaled) or U(k, k+i) into the tile itself.  Two blocks a tile, 32 columns
// each, and no products with the zeros of D: a block row has fewer tiles than
// the chip has SMs, so what counts is one tile's time.  Ten systems, 10 tiles a row:
// 8.5 -> 6.4 us.
__global__ void __launch_bounds__(256, 3) k_trsm(const SysDesc *__restrict__ sys, int k, bool scaled) {
  const SysDesc S = sys[blockIdx.y];
  const int i = (blockIdx.x >> 1) + 1, h0 = (blockIdx.x & 1) * (NB / 2);
  if (k >= S.nblk || i > S.J || k + i >= S.nblk || (S.jb && i > S.jb[k])) return;
  extern __shared__ __align__(16) double smt[];
  double *X = smt, *B = X + NB * LDM;
  double *T = S.tiles + ((size_t)(k + i) * (S.J + 1) + i) * TSZ;
  tile_stage_mma(X, S.dinv + (size_t)k * TSZ);
  for (int idx = threadIdx.x; idx < NB * NB / 4; idx += 256) {
    const int r = idx >> 4, c = h0 + 2 * (idx & (NB / 4 - 1));
    cp_async16_cg(B + r * LDM + c, T + r * LDT + c);
  }
  cp_async_commit();
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, q = w & 3, c = h0 + 16 * (w >> 2);
  const int g = lane >> 2, t = lane & 3;
  double v[2][2][2];
  auto store = [&](double *R, int ld) {
#pragma unroll
    for (int m = 0; m < 2; m++)
#pragma unroll
      for (int n = 0; n < 2; n++)
        *reinterpret_cast<double2 *>(&R[((m == 0 ? 8 * q : 8 * (7 - q)) + g) * ld + c + 8 * n + 2 * t]) =
            make_double2(v[m][n][0], v[m][n][1]);
  };
  cp_async_wait_all();
  __syncthreads();
  tri_mma<true>(v, X, B, q, c);
  store(S.row + (size_t)(i - 1) * TSZ, LDT);
  if (!scaled) {
    store(T, LDT);
    return;
  }
  __syncthreads();  // every warp has read the staged A(k, k+i)
  store(B, LDM);
  __syncthreads();
  tri_mma<false>(v, X, B, q, c);
  store(T, LDT);
}

// Trailing update inside the band: A(k+i, k+j) -= U(k,k+i)^T U(k,k+j),
// 1 <= i <= j <= jb[k] (every other product has a zero factor).  The product is formed in the accumulators from zero and
// subtracted from the target tile once: accumulating into the target
// instead moved an ill-conditioned mode's solution 170 times further from
// LAPACK's (1.3e-12 -> 2.2e-10 relative, config 5's pressure mode 1).
//
// The CTA of pair (1, 1) holds the diagonal tile of block column k + 1 when
// its update is done, and factors it on the spot (k = -1: block column 0,
// which nothing updates): the pivots' chain runs under the other pairs'
// products and the block column is a launch and a tile's way to memory and
// back shorter.  Blocks count the systems first, so that every system's chain
// starts with the launch.  Ten systems of 171 block columns built and solved:
// 11.1 -> 10.1 ms against a launch of its own for the diagonal tiles.  Two
// blocks an SM: the pivots need the registers (at three 11.9 ms for 9.4), and
// large launches lose nothing (12 systems of 1,206 block columns 258 ms, 268
// at three before).
__global__ void __launch_bounds__(256, 2) k_update(const SysDesc *__restrict__ sys, int ns, int k,
                                                   const int2 *__restrict__ pairs) {
  const SysDesc S = sys[blockIdx.x % ns];
  const int2 pr = pairs[blockIdx.x / ns];
  const int i = pr.x, j = pr.y;
  const bool prod = k >= 0 && j <= S.J && !(S.jb && j > S.jb[k]);
  if (k + j >= S.nblk || !(prod || j == 1)) return;
  extern __shared__ __align__(16) double smt[];
  double *A = smt, *B = A + NB * LDM;
  double *Ct = S.tiles + ((size_t)(k + j) * (S.J + 1) + (j - i)) * TSZ;
  if (j == 1) {
    tile_stage_mma(B, Ct);
    if (prod) tile_stage_mma(A, S.row);
    cp_async_commit();
    cp_async_wait_all();
    __syncthreads();
    if (prod) syrk_sub(B, A);
    __syncthreads();
    factor_diag(S, k + 1, B, A, B + NB * LDM);
    return;
  }
  tile_stage_mma(A, S.row + (size_t)(i - 1) * TSZ);
  if (i != j) tile_stage_mma(B, S.row + (size_t)(j - 1) * TSZ);
  cp_async_commit();
  MmaAcc acc;
  mma_zero(acc);
  cp_async_wait_all();
  __syncthreads();
  mma_tile(acc, A, i == j ? A : B);
  mma_sub(Ct, acc);
}

// ---------------------------------------------------------------------------
// Jacobi diagonal (JACPCG)
// ---------------------------------------------------------------------------

// Element::HelmholtzDiag (src/element.cpp:1512-1561), emap order.
__global__ void k_elem_diag(MeshView M, double hCon, double *__restrict__ ediag) {
  const int e = blockIdx.x, np = M.np, nn = M.npnp;
  const size_t eo = (size_t)e * nn;
  const bool q3 = M.hasQ3[e];
  for (int a = threadIdx.x; a < nn; a += blockDim.x) {
    const int ij = M.emap[a], i = ij / np, j = ij - i * np;
    double s = 0.0;
    for (int q = 0; q < np; q++) s += M.Q1[eo + i * np + q] * (M.D[q * np + j] * M.D[q * np + j]);
    double dg = s;
    s = 0.0;
    for (int p = 0; p < np; p++) s += M.Q2[eo + p * np + j] * (M.D[p * np + i] * M.D[p * np + i]);
    dg += s;
    if (q3) dg += 2.0 * M.Q3[eo + ij] * M.D[j * np + j] * M.D[i * np + i];
    dg += hCon * M.Q4[eo + ij];
    ediag[eo + a] = dg;
  }
}

// PC[g] = 1 / (mixed terms + sum of element diagonals) for boundary nodes,
// 1 / element diagonal for interior nodes (src/matrix.cpp:290-310).
__global__ void k_diag_dss(MeshView M, const double *__restrict__ ediag, double *pc, float *pcf) {
  const int npts = M.nglobal + M.nel * M.nint;
  const int g = blockIdx.x * blockDim.x + threadIdx.x;
  if (g >= npts) return;
  double s = 0.0;
  if (g < M.nglobal) {
    for (int q = M.nat_ptr[g]; q < M.nat_ptr[g + 1]; q++) {
      const int bi = M.nat_idx[q], b = bi / M.np, i = bi - b * M.np;
      if (M.b_kind[b] == SX_BC_MIXED) s += M.b_K[b] * M.b_area[bi];
    }
    for (int q = M.g2e_ptr[g]; q < M.g2e_ptr[g + 1]; q++) {
      const int ei = M.g2e_idx[q], e = ei / M.next, i = ei - e * M.next;
      s += ediag[(size_t)e * M.npnp + i];
    }
  } else {
    const int r = g - M.nglobal, e = r / M.nint, i = r - e * M.nint;
    s = ediag[(size_t)e * M.npnp + M.next + i];
  }
  pc[g] = 1.0 / s;
  pcf[g] = (float)(1.0 / s);
}

// ---------------------------------------------------------------------------
// Host drivers
// ---------------------------------------------------------------------------

static int check_status(DBuf<int> &st) {
  int h = 0;
  SX_CUDA(cudaMemcpy(&h, st.p, sizeof(int), cudaMemcpyDeviceToHost));
  if (h & (1 << SX_ERR_SINGULAR_HII)) {
    set_error("interior matrix hii is singular");
    return SX_ERR_SINGULAR_HII;
  }
  if (h & (1 << SX_ERR_BAND)) {
    set_error("btog couples nodes further apart than nband - 1");
    return SX_ERR_BAND;
  }
  if (h & (1 << SX_ERR_NOT_SPD)) {
    set_error("failed to factor Helmholtz matrix (not positive definite)");
    return SX_ERR_NOT_SPD;
  }
  return SX_OK;
}

size_t System::bytes() const {
  return (tiles.n + dinv.n + hbi.n + hii.n + pc.n) * 8 + (hbif.n + hiif.n + pcf.n) * 4;
}

int system_check_status(System &S) { return S.status.p ? check_status(S.status) : SX_OK; }

int factor_batch(std::vector<System *> &systems, cudaStream_t st, bool sync, bool scaled) {
  if (systems.empty()) return SX_OK;
  std::vector<SysDesc> hd(systems.size());
  int maxblk = 0, maxJ = 0;
  size_t rows = 0;
  for (size_t s = 0; s < systems.size(); s++) {
    System &S = *systems[s];
    const sx_mesh_s &Mh = *S.mesh;
    hd[s] = SysDesc{S.tiles.p, S.dinv.p, S.nblk, S.J, S.status.p, Mh.denv.p + Mh.env_nblk, nullptr};
    rows += S.J;
    maxblk = std::max(maxblk, S.nblk);
    maxJ = std::max(maxJ, S.J);
  }
  // tiles of block row k over the systems (the launches' extent)
  std::vector<int> rowmax(std::max(maxblk, 1), 0);
  for (System *Sp : systems) {
    const sx_mesh_s &Mh = *Sp->mesh;
    for (int k = 0; k < Sp->nblk; k++)
      rowmax[k] = std::max(rowmax[k], std::min(std::min(Sp->J, Mh.env[Mh.env_nblk + k]), Sp->nblk - 1 - k));
  }
  DBuf<double> rowbuf;
  SX_TRY(rowbuf.alloc_on(rows * TSZ, st));
  for (size_t s = 0, o = 0; s < systems.size(); o += systems[s]->J, s++) hd[s].row = rowbuf.p + o * TSZ;
  DBuf<SysDesc> dd;
  SX_TRY(dd.upload_on(hd.data(), hd.size(), st));
  std::vector<int2> pairs;
  for (int j = 1; j <= std::max(maxJ, 1); j++)
    for (int i = 1; i <= j; i++) pairs.push_back(make_int2(i, j));
  DBuf<int2> dpairs;
  SX_TRY(dpairs.upload_on(pairs.data(), pairs.size(), st));
  const size_t smm = 2 * NB * LDM * sizeof(double), sm2 = (2 * NB * LDM + NB) * sizeof(double);
  SX_CUDA(cudaFuncSetAttribute(k_trsm, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smm));
  SX_CUDA(cudaFuncSetAttribute(k_update, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm2));
  const int ns = (int)systems.size();
  for (int k = -1; k < maxblk - 1; k++) {
    const int m = k < 0 ? 0 : rowmax[k];
    if (m > 0) k_trsm<<<dim3(2 * m, ns), 256, smm, st>>>(dd.p, k, scaled);
    // pairs are listed by j, so those with j <= m come first
    k_update<<<(unsigned)(ns * std::max(1, m * (m + 1) / 2)), 256, sm2, st>>>(dd.p, ns, k, dpairs.p);
  }
  SX_CUDA(cudaGetLastError());
  if (sync) SX_CUDA(cudaStreamSynchronize(st));
  return SX_OK;
}

template <int NP>
static int launch_condense(const MeshView &M, const BuildDesc *d, int ns, cudaStream_t st) {
  // the kernel's shared-memory limit is a per-function setting, the same for
  // every caller of this order
  SX_CUDA(cudaFuncSetAttribute(k_elem_condense<NP>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                               (int)Condense<NP>::smem));
  k_elem_condense<NP><<<dim3(M.nel, ns), 256, Condense<NP>::smem, st>>>(M, d);
  SX_CUDA(cudaGetLastError());
  return SX_OK;
}

static int condense(const MeshView &M, const BuildDesc *d, int ns, cudaStream_t st) {
  switch (M.np) {
#define SX_CASE(n) \
  case n: return launch_condense<n>(M, d, ns, st);
    SX_CASE(3) SX_CASE(4) SX_CASE(5) SX_CASE(6) SX_CASE(7) SX_CASE(8) SX_CASE(9) SX_CASE(10)
    SX_CASE(11) SX_CASE(12)
#undef SX_CASE
    default: return SX_ERR_UNSUPPORTED;
  }
}

// The temporary condensed matrices of the systems built together are kept
// below this many bytes (64 systems of a large mesh would take several GB), or
// to one system's where not even that is free.
constexpr size_t BUILD_TEMP = size_t(1) << 30;

// Sizes, and the memory that stays.
static int system_reserve_direct(System &S, cudaStream_t st) {
  const sx_mesh_s &Mh = *S.mesh;
  S.singular = (S.lambda2 + S.betak2) < EPSSP && (Mh.nglobal - Mh.nsolve) == 0 && !Mh.mixed;
  S.nsolve = S.singular ? Mh.nsolve - 1 : Mh.nsolve;
  S.nblk = (S.nsolve + NB - 1) / NB;
  S.J = (Mh.nband - 1 + NB - 1) / NB;
  if (S.status.p == nullptr) SX_TRY(S.status.alloc_in(1, S.pool, st));
  SX_TRY(S.hbi.alloc_in((size_t)Mh.nel * Mh.next * Mh.nint, S.pool, st));
  SX_TRY(S.hii.alloc_in((size_t)Mh.nel * Mh.nint * Mh.nint, S.pool, st));
  const size_t nb = (size_t)std::max(S.nblk, 1);
  SX_TRY(S.tiles.alloc_in(nb * (S.J + 1) * TSZ, S.pool, st));
  SX_TRY(S.tiles.zero(st));
  return S.dinv.alloc_in(nb * TSZ, S.pool, st);  // factor_diag writes every block's tile in full
}

int systems_build_direct(const std::vector<System *> &systems, cudaStream_t st) {
  for (System *S : systems) SX_TRY(system_reserve_direct(*S, st));
  for (size_t s0 = 0, s1; s0 < systems.size(); s0 = s1) {
    sx_mesh_s &Mh = *systems[s0]->mesh;
    const MeshView M = Mh.view();
    const size_t nh = (size_t)Mh.nel * Mh.next * Mh.next;
    const size_t most = std::max<size_t>(1, BUILD_TEMP / (nh * 8));
    s1 = s0;
    while (s1 < systems.size() && s1 - s0 < most && systems[s1]->mesh == &Mh) s1++;
    DBuf<double> hbb;
    int rc = hbb.alloc_in(nh * (s1 - s0), systems[s0]->pool, st, true);
    if (rc == SX_ERR_NOMEM && s1 - s0 > 1) {
      s1 = s0 + 1;
      rc = hbb.alloc_in(nh, systems[s0]->pool, st, true);
    }
    SX_TRY(rc);
    const int ns = (int)(s1 - s0);
    std::vector<BuildDesc> hd(ns);
    bool any = false;
    for (int i = 0; i < ns; i++) {
      System &S = *systems[s0 + i];
      any |= S.nsolve > 0;
      hd[i] = BuildDesc{S.betak2 + S.lambda2, S.hbi.p, S.hii.p,  hbb.p + nh * i, S.tiles.p,
                        S.status.p,           S.nsolve, S.nblk, S.J};
    }
    DBuf<BuildDesc> dd;
    SX_TRY(dd.upload_on(hd.data(), hd.size(), st));
    k_band_init<<<dim3(1, ns), NB, 0, st>>>(dd.p);
    SX_TRY(condense(M, dd.p, ns, st));
    if (!any) continue;
    for (size_t c = 0; c + 1 < Mh.colour_ptr.size(); c++) {
      const int n = Mh.colour_ptr[c + 1] - Mh.colour_ptr[c];
      if (n > 0) k_band_add<<<dim3(n, ns), 256, 0, st>>>(M, Mh.dcolour_elmt.p + Mh.colour_ptr[c], dd.p);
    }
    if (Mh.mixed) k_band_mixed<<<dim3(1, ns), 32, 0, st>>>(M, dd.p);
    SX_CUDA(cudaGetLastError());
  }
  return SX_OK;
}

int system_build_direct(System &S, cudaStream_t st, bool sync) {
  const std::vector<System *> one(1, &S);
  SX_TRY(systems_build_direct(one, st));
  if (!sync) return SX_OK;
  SX_CUDA(cudaStreamSynchronize(st));
  SX_TRY(check_status(S.status));
  return SX_OK;
}

int system_build_jacobi(System &S, cudaStream_t st, bool sync) {
  sx_mesh_s &Mh = *S.mesh;
  S.singular = (S.lambda2 + S.betak2) < EPSSP && (Mh.nglobal - Mh.nsolve) == 0 && !Mh.mixed;
  S.nsolve = S.singular ? Mh.nsolve - 1 : Mh.nsolve;
  return system_build_jacobi_diag(S, st, sync);
}

// Inverse Jacobi diagonal only (also used by DIRECT systems for the
// mixed-precision form).
int system_build_jacobi_diag(System &S, cudaStream_t st, bool sync) {
  sx_mesh_s &Mh = *S.mesh;
  const MeshView M = Mh.view();
  const double hCon = S.betak2 + S.lambda2;
  const int npts = Mh.nglobal + Mh.nel * Mh.nint;
  DBuf<double> ediag;
  SX_TRY(ediag.alloc_in((size_t)Mh.nel * Mh.npnp, S.pool, st, true));
  SX_TRY(S.pc.alloc_in(npts, S.pool, st));
  SX_TRY(S.pcf.alloc_in(npts, S.pool, st));
  k_elem_diag<<<Mh.nel, 128, 0, st>>>(M, hCon, ediag.p);
  k_diag_dss<<<(npts + 255) / 256, 256, 0, st>>>(M, ediag.p, S.pc.p, S.pcf.p);
  SX_CUDA(cudaGetLastError());
  if (sync) SX_CUDA(cudaStreamSynchronize(st));
  return SX_OK;
}

// The factor's tiles with U itself off the diagonal.  The resident ones hold
// U_kk^-1 U(k, k+i): the system is assembled and factored once more, keeping U.
static int tiles_refactored(const System &S, std::vector<double> &t) {
  System X;
  X.mesh = S.mesh;
  X.lambda2 = S.lambda2;
  X.betak2 = S.betak2;
  X.pool = S.pool;
  SX_TRY(system_build_direct(X, 0));
  std::vector<System *> one(1, &X);
  if (X.nsolve > 0) SX_TRY(factor_batch(one, 0, true, false));
  t.resize(X.tiles.n);
  SX_CUDA(cudaMemcpy(t.data(), X.tiles.p, t.size() * 8, cudaMemcpyDeviceToHost));
  return SX_OK;
}

// The same from the resident tiles, U_kk times each on the host: U to a few
// roundings (noise where it is exactly zero inside a tile), but no device
// memory.
static int tiles_unscaled(const System &S, std::vector<double> &t) {
  t.resize(S.tiles.n);
  SX_CUDA(cudaMemcpy(t.data(), S.tiles.p, t.size() * 8, cudaMemcpyDeviceToHost));
  const sx_mesh_s &Mh = *S.mesh;
  const size_t col = (size_t)(S.J + 1) * TSZ;
  for (int k = 0; k < S.nblk; k++)
    for (int j = 1; j <= std::min(std::min(S.J, k), Mh.env[k]); j++) {
      const double *U = &t[(size_t)(k - j) * col];
      double *T = &t[(size_t)k * col + (size_t)j * TSZ];
      for (int r = 0; r < NB; r++) {  // U_kk is upper triangular: row r takes rows r and below
        double row[NB] = {};
        for (int l = r; l < NB; l++)
          for (int c = 0; c < NB; c++) row[c] += U[r * LDT + l] * T[l * LDT + c];
        std::memcpy(T + r * LDT, row, sizeof(row));
      }
    }
  return SX_OK;
}

// The factor U in LAPACK "U" band storage, ldab = nband.
int system_band_export(const System &S, double *ab) {
  const int nband = S.mesh->nband, kd = nband - 1;
  std::vector<double> t;
  int rc = tiles_refactored(S, t);
  if (rc == SX_ERR_NOMEM) rc = tiles_unscaled(S, t);  // no room for the system a second time
  SX_TRY(rc);
  std::memset(ab, 0, sizeof(double) * (size_t)S.nsolve * nband);
  for (int n = 0; n < S.nsolve; n++)
    for (int m = std::max(0, n - kd); m <= n; m++) ab[(size_t)n * nband + kd + m - n] = t[tile_addr(m, n, S.J)];
  return SX_OK;
}

}  // namespace sx

// sx_band.cu -- banded triangular solves (LAPACK dpbtrs "U" as called at
// src/field.cpp:609) on the tiled band factor.
//
// The factor is held as the block LDL^T form of U^T U (sx_factor.cu): the
// off-diagonal tiles are T(k, j) = U_bb^-1 U(rows of block b = k - j, cols of
// block k), and D_k = U_kk^-1.  Both sweeps are left-looking over block
// columns of NB rows and hold no diagonal solve on their chains:
//   forward  z_k = b_k - sum_{j>=1} T(k,j)^T   z_{k-j}
//   middle   w_k = D_k D_k^T z_k                       (independent per block)
//   backward x_k = w_k - sum_{j>=1} T(k+j,j) x_{k+j}
//
// One thread-block cluster of C CTAs works on one system (up to two
// right-hand sides at once).  The block-column chain is what bounds a system:
// nothing of step t + 1 can end before block t is known.  So the leader CTA
// (rank 0) keeps the chain on one SM: it owns the tiles j <= 2, and a step of
// its chain is the j = 1 tile's product, one reduction and one block barrier
// (two forward), the j = 2 tile of the next step following off the chain.
// Ranks 1..C-1 own the tiles j >= 3 and the D_k: what they multiply was solved
// three steps earlier or more, which covers the way to another SM and back.  A solved block goes to every rank's window of the last blocks
// by st.async (its mbarrier counts the bytes: no fence, no flag, no trip
// through L2); the ranks' partial sums return to the leader the same way.
//
// Tiles (32 KB, unpadded) stream into each CTA through a ring of 1-D TMA bulk
// copies issued by a warp of their own; the eight working warps never meet
// at a block barrier over a tile: each waits for the tile's mbarrier, reads
// its eight rows (a warp reads 512 contiguous bytes of a row) and releases
// the slot.  Forward, a lane keeps two columns and the warps' sums are added
// in warp order; backward, a warp keeps eight rows and its lanes' sums are
// added by shuffles, so the ranks run without block barriers.  Partials are
// combined in rank order, so the result does not depend on timing.
//
// A tile costs an SM some 500-800 cycles: the copy writes its 32 KB into
// shared memory, the warps read it back, and each warp reads the block it
// multiplies, all through one 128-byte-a-cycle port.  So a block is kept in the
// order in which a sweep's lanes read it without conflicts, and eight warps do
// better than sixteen (each reads the whole block backward).  The leader's
// step is two such tiles and about as long again in hand-offs.
//
// Measured (B200, 1965 MHz; both sweeps, the envelope's tiles twice), against
// the previous form (y_k = D_k^T (b_k - ...) with D_k on the chain, blocks
// fetched through L2 after a cluster-scope release, four block barriers a
// step):
//   32 systems, 236 block columns of 8.9 tiles   2.64 -> 0.78 ms, 5.99 TB/s
//   12 systems, 1206 block columns of 22.5      15.85 -> 3.97 ms, 5.50 TB/s
//   64 systems of that band                     24.9 -> 16.6 ms, 7.00 TB/s
//   one system of the first kind                 (5.6 -> 1.47 us a block column)
// With the leader owning j <= 3: 0.90 / 4.64 ms; with sixteen warps 0.82 /
// 4.27 ms.  The first two are bound by the leader's chain (1.65 us a block
// column), the third by HBM.
//
// Every wait is bounded (clock64).  When one runs out, the thread marks the
// CTA as given up and goes on without waiting or sending: the control flow
// depends on the tables alone, so every barrier is still met; the kernel
// records SX_ERR_TIMEOUT, waits (bounded) for its own bulk copies, meets the
// other CTAs at the final cluster barrier and returns.
#include <algorithm>
#include <type_traits>

#include "sx_kernels.cuh"
#include "sx_ptx.cuh"
#include "sx_solve.cuh"

namespace sx {

constexpr long long WAIT_LIMIT = SWEEP_WAIT_DEFAULT;  // ~2 s at 1.9 GHz

// Cycles a wait of the sweep loop may take before the kernel gives up
// (SX_ERR_TIMEOUT); per device, set by sx_set_wait_limit.  The drain of a
// CTA's own bulk copies on the way out always uses WAIT_LIMIT: those copies
// read valid memory and land within microseconds, and a CTA must not leave
// with copies into its shared memory still in flight.
__device__ long long g_sweep_wait = WAIT_LIMIT;

int set_sweep_wait_limit(long long cycles) {
  SX_CUDA(cudaMemcpyToSymbol(g_sweep_wait, &cycles, sizeof(cycles)));
  return SX_OK;
}

namespace {

constexpr int SWP_WARPS = 8;                       // working warps
constexpr int SWP_THREADS = (SWP_WARPS + 1) * 32;  // and the copying warp
constexpr int RPW = NB / SWP_WARPS;                // rows of a tile a warp reads
constexpr int VEC = 2 * NB;                        // a block of two right-hand sides, [row][plane]
constexpr int LPE = SWP_WARPS * 32 / VEC;          // lanes that share an element of a block
constexpr int RED = VEC + 2;                       // pitch of the warps' sums (lanes of an element on distinct banks)
constexpr int NEAR = 2;                           // the leader's tiles: j <= NEAR
constexpr int DLAG = NEAR + 1;                    // steps a D_k follows its block by, on the ranks


// Slots of the leader's buffer of partial sums: a rank runs at most this many
// steps ahead of the leader.
constexpr int DEPTH = 3;
static_assert(NEAR + 1 == DEPTH, "the ranks' one wait a step covers their youngest tile");

// Blocks in a CTA's window: every block a step multiplies (j <= J), and
// those whose arrival a rank waits for before it reuses a partial's slot.
// Bands of more than WINDOW_MAX - 2 tiles a block column do not fit beside a
// ring of tiles: the WIDE kernel keeps the most recent WIDE_WINDOW blocks and
// reads older ones from the right-hand sides' array through L2.  The D_k then
// follow the forward sweep, which still needs that array's z_k.  Two systems,
// 16 CTAs each (full window / WIDE): 103 blocks of 102 tiles 0.56 / 0.62 ms,
// 121 of 120 tiles 1.28 / 0.79 (one tile in flight beside the full window).
constexpr int WINDOW_MAX = 112, WIDE_WINDOW = 64;
__host__ __device__ __forceinline__ int full_window(int J) { return max(J, DEPTH) + 2; }
__host__ __device__ __forceinline__ int window_blocks(int J) {
  return full_window(J) > WINDOW_MAX ? WIDE_WINDOW : full_window(J);
}
static bool wide_band(int J) { return full_window(J) > WINDOW_MAX; }

// Doubles of the warps' sums and the leader's partial sums (see the kernel).
__host__ __device__ __forceinline__ int red_doubles(int C) {
  return SWP_WARPS * RED + max(SWP_WARPS * RED, DEPTH * (C - 1) * VEC);
}

// This warp's rows of a tile, two columns a lane, and the values of the block
// they meet: forward the rows' own, both planes side by side (the same in
// every lane); backward the columns', plane by plane.  The window keeps each
// sweep's blocks in the order its lanes read them.
struct TileRegs {
  double2 a[RPW], z[RPW];
};
template <bool FWD>
__device__ __forceinline__ void block_load(TileRegs &r, const double *z, int w, int lane) {
  const double2 *z2 = reinterpret_cast<const double2 *>(z) + (FWD ? w * RPW : lane);
#pragma unroll
  for (int i = 0; i < (FWD ? RPW : 2); i++) r.z[i] = z2[FWD ? i : i * (NB / 2)];
}
// The same from the right-hand sides' array (z0, z1: the planes' block; a lone
// plane stands in for both, and what it gives the second is never stored).
template <bool FWD>
__device__ __forceinline__ void block_load_l2(TileRegs &r, const double *z0, const double *z1, int w, int lane) {
  if (FWD) {
#pragma unroll
    for (int i = 0; i < RPW; i++) r.z[i] = make_double2(__ldcg(z0 + w * RPW + i), __ldcg(z1 + w * RPW + i));
  } else {
    r.z[0] = __ldcg(reinterpret_cast<const double2 *>(z0) + lane);
    r.z[1] = __ldcg(reinterpret_cast<const double2 *>(z1) + lane);
  }
}
__device__ __forceinline__ void rows_load(TileRegs &r, const double *T, int w, int lane) {
  const double2 *t2 = reinterpret_cast<const double2 *>(T) + w * RPW * (NB / 2) + lane;
#pragma unroll
  for (int i = 0; i < RPW; i++) r.a[i] = t2[i * (NB / 2)];
}
template <bool FWD>
__device__ __forceinline__ void tile_load(TileRegs &r, const double *T, const double *z, int w, int lane) {
  block_load<FWD>(r, z, w, lane);
  rows_load(r, T, w, lane);
}
// Forward: acc (two columns, two planes) += T^T z; backward: acc (the rows, two
// planes) += this lane's columns of T times z.
template <bool FWD>
__device__ __forceinline__ void tile_fma(const TileRegs &r, double *acc) {
#pragma unroll
  for (int i = 0; i < RPW; i++) {
    if (FWD) {
      acc[0] = fma(r.a[i].x, r.z[i].x, acc[0]);
      acc[1] = fma(r.a[i].x, r.z[i].y, acc[1]);
      acc[2] = fma(r.a[i].y, r.z[i].x, acc[2]);
      acc[3] = fma(r.a[i].y, r.z[i].y, acc[3]);
    } else {
      acc[2 * i] = fma(r.a[i].y, r.z[0].y, fma(r.a[i].x, r.z[0].x, acc[2 * i]));
      acc[2 * i + 1] = fma(r.a[i].y, r.z[1].y, fma(r.a[i].x, r.z[1].x, acc[2 * i + 1]));
    }
  }
}

// Sums of a warp's 2 RPW values over its lanes, halving: lane l returns its
// part of value l / LPE (the rest is with the other lanes of the LPE).
__device__ __forceinline__ double lanes_reduce(const double *acc, int lane) {
  double v[2 * RPW];
#pragma unroll
  for (int i = 0; i < 2 * RPW; i++) v[i] = acc[i];
  int o = 16;
#pragma unroll
  for (int n = RPW; n >= 1; n /= 2) {
    const bool up = lane & o;
#pragma unroll
    for (int i = 0; i < n; i++) v[i] = (up ? v[i + n] : v[i]) + __shfl_xor_sync(0xffffffffu, up ? v[i] : v[i + n], o);
    o /= 2;
  }
  return v[0];
}

// The whole of an element from its lanes' parts, in each of them.
__device__ __forceinline__ double lane_sum(double s) {
#pragma unroll
  for (int o = LPE / 2; o >= 1; o /= 2) s += __shfl_xor_sync(0xffffffffu, s, o);
  return s;
}

// Off-diagonal tiles of step t (t < nblk: forward block t, else backward
// block 2 nblk - 1 - t) inside the band and the factor's envelope.
struct StepTab {
  const int *jf, *jb;
  int nblk, J;
  // the envelope's entry of step t, and the step's tiles given it: a step
  // takes its entry from a register loaded steps earlier, off the chain
  __device__ __forceinline__ int entry(int t) const {
    if (t >= 2 * nblk) return 0;
    if (t < nblk) return jf ? __ldg(jf + t) : J;
    return jb ? __ldg(jb + 2 * nblk - 1 - t) : J;
  }
  __device__ __forceinline__ int tiles(int t, int entry) const {
    const int b = t < nblk ? t : t - nblk;
    return max(0, min(min(J, b), entry));
  }
  __device__ __forceinline__ int jmax(int t) const { return tiles(t, entry(t)); }
};

// The far tiles (j > NEAR) a CTA owns, ascending: round-robin over the ranks
// 1..C-1, except the last of every Q (Q >= 2), which are the leader's.  C = 1:
// all of them.
__device__ int own_list(unsigned short *own, int J, int C, int rank, int Q) {
  int n = 0, m = 0;  // m: position among the ranks' tiles
  for (int j = NEAR + 1; j <= J; j++) {
    const bool lead = C == 1 || (Q >= 2 && (j - NEAR - 1) % Q == Q - 1);
    if (lead ? rank == 0 : (rank > 0 && m == rank - 1)) own[n++] = (unsigned short)j;
    if (!lead && ++m == C - 1) m = 0;
  }
  return n;
}

// Tiles of the list with j <= jm, from the count at the last step.
__device__ __forceinline__ int own_count(const unsigned short *own, int len, int n, int jm) {
  while (n < len && own[n] <= jm) n++;
  while (n > 0 && own[n - 1] > jm) n--;
  return n;
}

using Fwd = std::true_type;
using Bwd = std::false_type;

}  // namespace

template <bool WIDE>
__global__ void __launch_bounds__(SWP_THREADS, 1)
    k_band_sweep(const Job *__restrict__ jobs, int C, int S, int Wmax, int Q) {
  const int rank = (int)cluster_ctarank();
  const Job Jb = jobs[blockIdx.x / C];
  const int P = Jb.P, nblk = Jb.nblk, T = 2 * nblk, J = Jb.J;
  const int W = window_blocks(J);
  constexpr int D = DEPTH;
  extern __shared__ __align__(128) unsigned char smraw[];
  double *ring = reinterpret_cast<double *>(smraw);             // S tiles
  double *zwin = ring + (size_t)S * TSZ;                        // Wmax blocks
  // the warps' sums: one buffer in the leader, whose steps end with a barrier,
  // and its D * (C - 1) partial sums after it; two buffers in a rank
  double *red = zwin + (size_t)Wmax * VEC;
  double *pbuf = red + SWP_WARPS * RED;
  double *vd = red + red_doubles(C);                            // D_k^T z_k
  double *zd = vd + VEC;                                        // WIDE: z_k of a D_k
  uint64_t *full = reinterpret_cast<uint64_t *>(zd + (WIDE ? VEC : 0));  // S
  uint64_t *empty = full + S;                                   // S
  uint64_t *zbar = empty + S;                                   // Wmax
  uint64_t *pbar = zbar + Wmax;                                 // D
  unsigned short *own = reinterpret_cast<unsigned short *>(pbar + D);  // J + 1
  __shared__ int abort_flag, own_len;

  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
  const StepTab tab{Jb.jf, Jb.jb, nblk, J};
  const long long lim = g_sweep_wait;
  if (tid == 0) {
    for (int s = 0; s < S; s++) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], SWP_WARPS);
    }
    for (int s = 0; s < W; s++) mbar_init(&zbar[s], 1);
    for (int s = 0; s < D; s++) mbar_init(&pbar[s], 1);
    fence_mbar_init_cluster();
    // each phase of these barriers ends with its bytes; the owner arms it
    if (rank != 0)
      for (int s = 0; s < min(W, T); s++) mbar_arrive_expect_tx(&zbar[s], VEC * sizeof(double));
    if (rank == 0 && C > 1)
      for (int s = 0; s < min(D, T); s++) mbar_arrive_expect_tx(&pbar[s], (C - 1) * VEC * sizeof(double));
    own_len = own_list(own, J, C, rank, Q);
    abort_flag = 0;
  }
  __syncthreads();
  cluster_sync_all();
  volatile int *const aborted = &abort_flag;
  const int len = own_len;

  if (w == SWP_WARPS) {
    // ---- the copying warp: every tile this CTA reads, in its order of use
    cluster_arrive();  // the barrier between the sweeps: nothing to wait for here
    long long n = 0;  // tiles issued
    int slot = 0;
    uint32_t use = 0;  // times the ring has gone round
    bool stop = false;
    auto issue = [&](const double *src) {
      if (stop) return;
      if (use > 0) {
        if (!mbar_wait_tx(&empty[slot], (use - 1) & 1, lim)) *aborted = 1;
        if (*aborted) {
          stop = true;
          return;
        }
      }
      mbar_arrive_expect_tx(&full[slot], (uint32_t)(TSZ * sizeof(double)));
      bulk_g2s(ring + (size_t)slot * TSZ, src, (uint32_t)(TSZ * sizeof(double)), &full[slot]);
      n++;
      if (++slot == S) {
        slot = 0;
        use++;
      }
    };
    const size_t J1 = J + 1;
    auto off = [&](int t, int j) {  // tile j of step t
      return Jb.tiles + ((size_t)(t < nblk ? t : 2 * nblk - 1 - t + j) * J1 + j) * TSZ;
    };
    auto diag = [&](int k) { issue(Jb.dinv + (size_t)k * TSZ); };
    int cnt = 0, jm = tab.jmax(0), dm = 0;  // dm: block t - DLAG modulo C - 1
    auto steps = [&](int t0, int t1) {
      if (rank == 0) {
        for (int t = t0; t < t1 && !stop; t++) {
          if (jm >= 1) issue(off(t, 1));
          if (!WIDE && C == 1 && t < nblk) diag(t);
          jm = tab.jmax(t + 1);
          cnt = own_count(own, len, cnt, jm);
          for (int i = cnt - 1; i >= 0; i--) issue(off(t + 1, own[i]));
          for (int j = min(jm, NEAR); j >= 2; j--) issue(off(t + 1, j));
        }
      } else {
        for (int t = t0; t < t1 && !stop; t++) {
          if (!WIDE && t >= DLAG && t < nblk) {
            if (dm == rank - 1) diag(t - DLAG);
            if (++dm == C - 1) dm = 0;
          }
          cnt = own_count(own, len, cnt, tab.jmax(t));
          for (int i = cnt - 1; i >= 0; i--) issue(off(t, own[i]));
          if (!WIDE && t == nblk - 1)
            for (int k = max(0, nblk - DLAG); k < nblk; k++) {
              if (dm == rank - 1) diag(k);
              if (++dm == C - 1) dm = 0;
            }
        }
      }
    };
    if (WIDE) {  // the D_k between the sweeps, each CTA its share
      if (lane == 0) steps(0, nblk);
      __syncwarp();
      cluster_wait();
      cluster_arrive();
      if (lane == 0)
        for (int k = rank; k < nblk; k += C) diag(k);
    }
    if (lane == 0) {
      steps(WIDE ? nblk : 0, T);
      // the copies still in flight (none unless the sweep was given up)
      for (int s = 0; s < S && s < n; s++) {
        const uint32_t u = s < slot ? use : use - 1;  // the slot's last use
        mbar_wait_tx(&full[s], u & 1, WAIT_LIMIT);
      }
    }
    __syncwarp();
    cluster_wait();
    cluster_sync_all();
    return;
  }

  // ---- the working warps
  bool dead = false;
  auto wait = [&](uint64_t *bar, uint32_t parity) {
    if (!dead && !mbar_wait_tx(bar, parity, lim)) {
      dead = true;
      *aborted = 1;
    }
  };
  int cs = 0;  // ring slot and phase of the next tile
  uint32_t cph = 0;
  bool here = false;  // the next tile is known to have landed
  // A wait for a phase that is already complete still takes some 120 cycles, so
  // the next tile's is probed as soon as this one is in registers, under its
  // arithmetic.
  auto await_tile = [&]() {
    if (!here) wait(&full[cs], cph);
  };
  auto release = [&]() {
    __syncwarp();
    if (lane == 0) mbar_arrive(&empty[cs]);
    if (++cs == S) {
      cs = 0;
      cph ^= 1u;
    }
    here = mbar_test_cta(&full[cs], cph);
  };
  const int e = tid / LPE, q4 = tid % LPE;  // this thread's element of a block, shared by LPE lanes
  const int ec = e >> 1, ep = e & 1;       // its row and plane
  double *const gx = Jb.rhs + (size_t)(ep < P ? ep : 0) * Jb.rhs_stride + ec;
  double acc[2 * RPW];
  auto clear = [&]() {
#pragma unroll
    for (int i = 0; i < 2 * RPW; i++) acc[i] = 0.0;
  };
  // acc += tile j of step t, whose window slot is bs, times the block solved j
  // steps before it, which the caller knows to be there.
  auto tile = [&](auto F, int j, int bs, int t) {
    const int zs = bs - j < 0 ? bs - j + W : bs - j;
    TileRegs r;
    // (block t - W's slot is the one block t is stored to, and backward the
    // leader meets no barrier between a warp's read and another's store: it
    // too is read from there)
    if (WIDE && j >= W) {
      const int so = t - j;
      const double *z0 = Jb.rhs + (size_t)(so < nblk ? so : T - 1 - so) * NB;
      block_load_l2<decltype(F)::value>(r, z0, P > 1 ? z0 + Jb.rhs_stride : z0, w, lane);
      await_tile();
      rows_load(r, ring + (size_t)cs * TSZ, w, lane);
    } else {
      await_tile();
      tile_load<decltype(F)::value>(r, ring + (size_t)cs * TSZ, zwin + (size_t)zs * VEC, w, lane);
    }
    release();
    tile_fma<decltype(F)::value>(r, acc);
  };
  const int pf = e, pb = ep * NB + ec;  // its place in a block of the forward and the backward sweep
  // this CTA's sum of element e, in parts over its lanes
  // (the leader's partial sums are read on the way to the barrier, by `also`)
  auto reduce = [&](auto F, int par, auto also) -> double {
    if (!decltype(F)::value) {
      const double o = also();
      return lanes_reduce(acc, lane) + o;
    }
    double *r = rank == 0 ? red : red + par * SWP_WARPS * RED;
    double2 *r2 = reinterpret_cast<double2 *>(r + w * RED) + 2 * lane;
    r2[0] = make_double2(acc[0], acc[1]);
    r2[1] = make_double2(acc[2], acc[3]);
    const double o = also();
    bar_sync(1, SWP_WARPS * 32);
    const double *q = r + (SWP_WARPS / LPE) * q4 * RED + e;
    static_assert(SWP_WARPS / LPE == 4, "four warps' sums a lane");
    return ((q[0] + q[RED]) + (q[2 * RED] + q[3 * RED])) + o;
  };
  auto none = []() { return 0.0; };
  // w_k = D_k D_k^T z_k, z in the order of a forward sweep, into rhs
  auto apply_d = [&](int k, const double *z, int par) {
    clear();
    TileRegs r;
    await_tile();
    const double *t = ring + (size_t)cs * TSZ;
    tile_load<true>(r, t, z, w, lane);
    tile_fma<true>(r, acc);
    const double v = lane_sum(reduce(Fwd(), par, none));
    if (q4 == 0) vd[pb] = v;
    bar_sync(1, SWP_WARPS * 32);
    clear();
    tile_load<false>(r, t, vd, w, lane);
    release();
    tile_fma<false>(r, acc);
    const double x = lane_sum(lanes_reduce(acc, lane));
    if (q4 == 0 && ep < P) gx[(size_t)k * NB] = x;
    clear();
  };
  auto between_sweeps = [&]() {
    __syncwarp();
    cluster_arrive();
    cluster_wait();
  };

  // WIDE: the D_k of this CTA's share, once every z_k is in rhs
  auto wide_diags = [&]() {
    if constexpr (WIDE) {
      for (int k = rank; k < nblk; k += C) {
        if (q4 == 0) zd[pf] = ep < P ? __ldcg(gx + (size_t)k * NB) : 0.0;
        bar_sync(1, SWP_WARPS * 32);
        apply_d(k, zd, 0);
      }
      between_sweeps();
    }
  };

  clear();
  int cnt = 0, bs = 0, ps = 0;  // bs, bp: window slot and parity of step t; ps, pp: of its partial sums
  uint32_t bp = 0, pp = 0;
  if (rank == 0) {
    int jm = tab.jmax(0), e1 = tab.entry(1);
    double b = nblk > 0 && ep < P ? __ldcg(gx) : 0.0;
    // this lane's ranks to send to: 1 + q4, 1 + q4 + LPE, ... (at most 15 ranks)
    constexpr int NTO = 16 / LPE;
    uint32_t to_z[NTO], to_bar[NTO];
#pragma unroll
    for (int i = 0; i < NTO; i++) {
      const int r = min(1 + q4 + LPE * i, C - 1);
      to_z[i] = map_rank(zwin, r);
      to_bar[i] = map_rank(zbar, r);
    }
    auto step = [&](auto F, int t) {
      const int e2 = tab.entry(t + 2);
      const bool parts = C > 1 && mbar_test_cta(&pbar[ps], pp);  // the ranks' partial sums are here
      if (jm >= 1) tile(F, 1, bs, t);
      const double s = reduce(F, t & 1, [&]() {
        double o = 0.0;
        if (C > 1) {
          if (!parts) wait(&pbar[ps], pp);
          const double *q = pbuf + (size_t)ps * (C - 1) * VEC + e;
          for (int r = q4; r < C - 1; r += LPE) o += q[(size_t)r * VEC];
        }
        return o;
      });
      const double z = b - lane_sum(s);
      const int zo = bs * VEC + (decltype(F)::value ? pf : pb);
      if (q4 == 0) zwin[zo] = z;
      if (WIDE) {  // in rhs before any rank can know the block is there, whichever lane tells it
        if (q4 == 0 && ep < P) gx[(size_t)(decltype(F)::value ? t : T - 1 - t) * NB] = z;
        __threadfence();
        __syncwarp();
      }
      if (C > 1 && !dead) {
#pragma unroll
        for (int i = 0; i < NTO; i++)
          if (1 + q4 + LPE * i < C)
            st_async_f64(to_z[i] + zo * (int)sizeof(double), z, to_bar[i] + bs * (int)sizeof(uint64_t));
      }
      if (C > 1 && tid == 0 && t + D < T && !dead)
        mbar_arrive_expect_tx(&pbar[ps], (C - 1) * VEC * sizeof(double));
      // the next step's right-hand side (the first backward one is read after the barrier)
      const int tn = t + 1;
      if (!WIDE && !decltype(F)::value && q4 == 0 && ep < P) gx[(size_t)(T - 1 - t) * NB] = z;
      if (tn < T && tn != nblk && ep < P) b = __ldcg(gx + (size_t)(tn < nblk ? tn : T - 1 - tn) * NB);
      bar_sync(1, SWP_WARPS * 32);
      clear();
      if (!WIDE && C == 1 && decltype(F)::value) apply_d(t, zwin + (size_t)bs * VEC, t & 1);
      if (++bs == W) {
        bs = 0;
        bp ^= 1u;
      }
      if (++ps == D) {
        ps = 0;
        pp ^= 1u;
      }
      jm = tab.tiles(tn, e1);
      e1 = e2;
      if (len > 0) {
        cnt = own_count(own, len, cnt, jm);
        for (int i = cnt - 1; i >= 0; i--) tile(F, own[i], bs, tn);
      }
      for (int j = min(jm, NEAR); j >= 2; j--) tile(F, j, bs, tn);
    };
    for (int t = 0; t < nblk; t++) step(Fwd(), t);
    between_sweeps();
    wide_diags();
    if (nblk > 0 && ep < P) b = __ldcg(gx + (size_t)(nblk - 1) * NB);
    for (int t = nblk; t < T; t++) step(Bwd(), t);
  } else {
    int dm = 0, ej = tab.entry(0);
    const uint32_t to_p = map_rank(pbuf + (rank - 1) * VEC + e, 0), to_pbar = map_rank(pbar, 0);
    // block t - back's slot and parity
    auto slot_back = [&](int back, uint32_t &par) {
      int s = bs - back;
      par = bp;
      if (s < 0) {
        s += W;
        par ^= 1u;
      }
      return s;
    };
    auto step = [&](auto F, int t) {
      const int jm = tab.tiles(t, ej);
      ej = tab.entry(t + 1);
      // block t's phase in this CTA's window: the leader sends it once it has
      // this step's partial sum, below
      if (tid == 0 && t >= W) {
        wait(&zbar[bs], bp ^ 1u);
        if (!dead) mbar_arrive_expect_tx(&zbar[bs], VEC * sizeof(double));
      }
      if (!WIDE && decltype(F)::value && t >= DLAG) {
        if (dm == rank - 1) {
          uint32_t par;
          const int zs = slot_back(DLAG, par);
          wait(&zbar[zs], par);
          apply_d(t - DLAG, zwin + (size_t)zs * VEC, t & 1);
        }
        if (++dm == C - 1) dm = 0;
      }
      // Each step waits for one block, t - D, once: before the tile that needs
      // it (j = NEAR + 1 = D), or before the partial sum goes out -- its slot
      // has been read once block t - D is here.  Older blocks were waited for
      // in earlier steps.
      bool waited = t < D;
      auto wait_block = [&]() {
        if (waited) return;
        uint32_t par;
        const int zs = slot_back(D, par);
        wait(&zbar[zs], par);
        waited = true;
        if (WIDE) __threadfence();  // the leader's stores to rhs before it
      };
      cnt = own_count(own, len, cnt, jm);
      for (int i = cnt - 1; i >= 0; i--) {
        const int j = own[i];
        if (j <= D) wait_block();
        tile(F, j, bs, t);
      }
      const double s = lane_sum(reduce(F, t & 1, none));
      wait_block();
      if (q4 == 0 && !dead)
          st_async_f64(to_p + ps * (C - 1) * (VEC * (int)sizeof(double)), s, to_pbar + ps * (int)sizeof(uint64_t));
      clear();
      if (++bs == W) {
        bs = 0;
        bp ^= 1u;
      }
      if (++ps == D) ps = 0;
    };
    for (int t = 0; t < nblk; t++) step(Fwd(), t);
    if (!WIDE)
      for (int k = max(0, nblk - DLAG); k < nblk; k++) {
        if (dm == rank - 1) {
          uint32_t par;
          const int zs = slot_back(nblk - k, par);
          wait(&zbar[zs], par);
          apply_d(k, zwin + (size_t)zs * VEC, nblk & 1);  // not the buffer that step nblk - 1 may still be reading
        }
        if (++dm == C - 1) dm = 0;
      }
    between_sweeps();
    wide_diags();
    for (int t = nblk; t < T; t++) step(Bwd(), t);
    // every block the leader sent has landed before this CTA leaves
    for (int back = min(W, T); back >= 1; back--) {
      uint32_t par;
      const int zs = slot_back(back, par);
      wait(&zbar[zs], par);
    }
  }
  __syncwarp();
  cluster_sync_all();
  if (*aborted) {
    if (tid == 0) atomicOr(Jb.status, 1 << SX_ERR_TIMEOUT);
    // another CTA's last stores into this one's shared memory, sent before it
    // met the barrier above, land within a microsecond or two
    const long long t0 = clock64();
    while (clock64() - t0 < 200000) {
    }
  }
}

// J: the most tiles a block column of the launch; W: its largest window.
static size_t sweep_smem(int C, int S, int J, int W) {
  return sizeof(double) * ((size_t)S * TSZ + ((size_t)W + 1 + wide_band(J)) * VEC + red_doubles(C)) +
         sizeof(uint64_t) * (2 * S + W + DEPTH) + ((sizeof(unsigned short) * (J + 1) + 15) & ~(size_t)15);
}

using SweepKernel = void (*)(const Job *, int, int, int, int);
static SweepKernel sweep_kernel(int J) { return wide_band(J) ? k_band_sweep<true> : k_band_sweep<false>; }

// Dynamic shared memory available to the sweep kernel: the opt-in limit
// minus its static shared memory.
static int smem_optin() {
  static int v = 0;
  if (!v) {
    int dev = 0, optin = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
    cudaFuncAttributes a, b;
    cudaFuncGetAttributes(&a, k_band_sweep<false>);
    cudaFuncGetAttributes(&b, k_band_sweep<true>);
    v = optin - (int)std::max(a.sharedSizeBytes, b.sharedSizeBytes);
  }
  return v;
}

// The deepest ring of at most smax tiles that fits (0: none).
static int fit_stages(int C, int smax, int J, int W) {
  int S = std::max(1, std::min(smax, BAND_STAGES_MAX));
  while (S > 0 && sweep_smem(C, S, J, W) > (size_t)smem_optin()) S--;
  return S;
}

// Launch both sweeps for every job: one cluster of sc.C CTAs per job.
int band_sweep_jobs(const Job *djobs, const std::vector<Job> &hjobs, const BandSched &sc, cudaStream_t st) {
  const int C = sc.C;
  const int nj = (int)hjobs.size();
  if (nj == 0) return SX_OK;
  // one wide band makes it the WIDE kernel for all, which takes any band, and
  // one cluster size serves all (48 systems of 11 tiles a block column 0.93 ms,
  // two of 121 tiles 0.80, all in one launch of two CTAs a system 3.55)
  int maxP = 0, J = 0, Wmax = 0;
  for (const Job &j : hjobs) {
    maxP = std::max(maxP, j.P);
    J = std::max(J, j.J);
    Wmax = std::max(Wmax, window_blocks(j.J));
  }
  if (maxP > 2) return SX_ERR_UNSUPPORTED;
  const int S = fit_stages(C, sc.S, J, Wmax);
  if (S < 1) {
    set_error("band sweep needs %zu B of shared memory (limit %d)", sweep_smem(C, 1, J, Wmax), smem_optin());
    return SX_ERR_UNSUPPORTED;
  }
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(C * nj, 1, 1);
  cfg.blockDim = dim3(SWP_THREADS, 1, 1);
  cfg.dynamicSmemBytes = sweep_smem(C, S, J, Wmax);
  cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = C;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  SX_CUDA(cudaLaunchKernelEx(&cfg, sweep_kernel(J), djobs, C, S, Wmax, std::max(sc.Q, 0)));
  return SX_OK;
}

int prepare_band_kernels() {
  const int limit = smem_optin();
  for (SweepKernel k : {(SweepKernel)k_band_sweep<false>, (SweepKernel)k_band_sweep<true>}) {
    SX_CUDA(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, limit));
    SX_CUDA(cudaFuncSetAttribute(k, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
  }
  return SX_OK;
}

int default_lead(int C, int) {
  // the leader's j <= NEAR tiles are its share in clusters of four or more;
  // in smaller ones the ranks would have most of the band to themselves (64
  // systems, C = 2: half 16.6 ms, a third 17.8, none 20.7; 12 systems of that
  // band, C = 3: a quarter 8.27, a third 8.89, a fifth 8.81, none 10.0; C = 9:
  // none 3.97, a sixth 6.0)
  return C == 2 ? 2 : C == 3 ? 4 : 0;
}

// Clusters of C CTAs (ring of S tiles) that can be resident at once.
static int resident_clusters(int C, int S, int J) {
  if (S < 1) return 0;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(C, 1, 1);
  cfg.blockDim = dim3(SWP_THREADS, 1, 1);
  cfg.dynamicSmemBytes = sweep_smem(C, S, J, window_blocks(J));
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = C;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  int n = 0;
  if (cudaOccupancyMaxActiveClusters(&n, sweep_kernel(J), &cfg) != cudaSuccess) {
    cudaGetLastError();
    return 0;
  }
  return n;
}

int band_active_clusters(int C, int J, int smax) {
  return resident_clusters(C, fit_stages(C, smax, J, window_blocks(J)), J);
}

// Cluster size C <= cmax and ring depth for nj systems of J tiles a block
// column: the deepest ring with which every system's cluster is resident,
// and the largest such cluster.  Depth comes first: a CTA alone on its SM
// with four tiles in flight keeps up with its share of HBM, and shallower
// rings are slower before they let a larger cluster in (32 systems, 4 CTAs
// each: depth 4 0.78 ms, 3 0.84, 2 0.96; 5 CTAs at depth 2, in two waves,
// 1.63).  Where not even one CTA a system is resident, which is from 149
// systems on (the registers allow one CTA an SM), C = 1 at the depth with the
// most CTAs on the chip: 148 systems of 236 block columns 3.0 ms, 149 4.7, 240
// 5.2.
// stages_forced > 0 fixes the depth.
int pick_cluster(int nj, int cmax, int J, int *stages_out, int stages_forced) {
  int bestC = 0, bestS = BAND_STAGES_MAX, mostS = BAND_STAGES_MAX, most = 0;
  for (int S = BAND_STAGES_MAX; S >= 1 && bestC == 0; S--) {
    if (stages_forced > 0 && S != stages_forced) continue;
    for (int C = cmax; C >= 1 && bestC == 0; C--) {
      const int n = band_active_clusters(C, J, S);
      if (n >= nj) {
        bestC = C;
        bestS = S;
      }
      if (C == 1 && S >= 2 && n > most) {
        most = n;
        mostS = S;
      }
    }
  }
  if (bestC == 0) {
    bestC = 1;
    bestS = stages_forced > 0 ? stages_forced : mostS;
  }
  if (stages_out) *stages_out = bestS;
  return bestC;
}

}  // namespace sx

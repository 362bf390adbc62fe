// sx_solve.cu -- GPU DIRECT solve of Helmholtz planes (Field::solve, DIRECT
// branch, src/field.cpp:588-624).
//
// A "job" is a set of P planes that share one system (the Re and Im planes
// of a Fourier mode).  Every kernel takes an array of jobs (grid.y = job), so
// the plain form launches one job per mode and the batched form all modes
// at once.  Per job:
//   k_rhs_elem    constrain  f <- -(M f + H g)  (src/field.cpp:728-768) and the
//                 element half of local2globalSumSC: edge-major gather,
//                 F_b -= (hbi hii^-1) F_i  (src/element.cpp:356-395)
//   k_rhs_dss     direct-stiffness sum of F_b into the global RHS in element
//                 order, then <h, w> natural/mixed terms in boundary order, then
//                 the essential tail zeroed (src/field.cpp:892-924)
//   band sweeps   U^T y = b, U x = y: LAPACK dpbtrs "U" (src/field.cpp:609),
//                 one thread-block cluster per job (sx_band.cu)
//   k_backsub     global2localSC: u_i = hii^-1 F_i - (hii^-1 h_ib) u_b
//                 (src/element.cpp:398-438), then setEssential
//                 (src/field.cpp:1022-1040)
#include "sx_internal.h"
#include "sx_kernels.cuh"
#include "sx_ptx.cuh"
#include "sx_solve.cuh"

namespace sx {

// ---------------------------------------------------------------------------
// Element forcing and condensation
// ---------------------------------------------------------------------------

// One block of RHS_THREADS threads per (element, job); both planes of the job
// in one pass, so the element's hbi block (hbi hii^-1, NE x NI) is read once
// per job.  It goes to shared memory by 16-byte asynchronous copies issued
// before anything else, so that it arrives while the forcing and the element
// operator are computed; four neighbouring threads then share a row, so that a
// row's sum takes two shuffles.  The geometric factors of the operator are
// read only for elements that hold essential nodes.
//   HBM bounds it: the block's bytes.  Against a warp a row, its loads held in
// registers across the operator: 32 systems of 1024 elements of order 8 218 ->
// 145 us (3.9 TB/s), 12 of 4096 of order 10 495 -> 415 us, 20 of 851 of order
// 7 110 -> 54 us.
constexpr int RHS_THREADS = 128;

template <int NP>
constexpr size_t rhs_smem() {
  return (size_t)(4 * (NP - 1)) * (NP * NP - 4 * (NP - 1)) * sizeof(double);
}

template <int NP>
__global__ void __launch_bounds__(RHS_THREADS) k_rhs_elem(MeshView M, const Job *__restrict__ jobs) {
  constexpr int NN = NP * NP, NE = 4 * (NP - 1), NI = NN - NE, NT = RHS_THREADS;
  const Job &J = jobs[blockIdx.y];
  const int e = blockIdx.x, tid = threadIdx.x;
  extern __shared__ __align__(16) double H[];  // hbi hii^-1, row-major
  {
    const double *hbi = J.hbi + (size_t)e * NE * NI;
    for (int i = tid; i < NE * NI / 2; i += NT) cp_async16_cg(H + 2 * i, hbi + 2 * i);
    cp_async_commit();
  }
  const int P = J.P;
  const size_t fs = (size_t)J.fstride;
  __shared__ double F[2][NN], Fe[2][NN];
  __shared__ double D[NN], Q[4][NN], u[NN], R[NN], S[NN], T[NN];
  __shared__ int emap[NN];
  const size_t eo = (size_t)e * NN;
  double *const f = J.f + eo;
  const bool masked = M.emask[e] != 0;
  for (int i = tid; i < NN; i += NT) {
    emap[i] = M.emap[i];
    const double q8 = M.Q8[eo + i];
    F[0][i] = q8 * f[i];
    F[1][i] = P > 1 ? q8 * f[fs + i] : 0.0;
  }
  if (masked) {
    // f <- M f + H g: the operator applied to the element's essential values
    for (int i = tid; i < NN; i += NT) {
      D[i] = M.D[i];
      Q[0][i] = M.Q1[eo + i];
      Q[1][i] = M.Q2[eo + i];
      Q[2][i] = M.Q3[eo + i];
      Q[3][i] = M.Q4[eo + i];
    }
    const bool q3 = M.hasQ3[e];
    const int *bt = M.btog + (size_t)e * NE;
    for (int p = 0; p < P; p++) {
      const double *bc = J.bc ? J.bc + (size_t)p * J.bcstride : nullptr;
      __syncthreads();
      for (int i = tid; i < NN; i += NT) u[i] = 0.0;
      __syncthreads();
      for (int i = tid; i < NE; i += NT) u[emap[i]] = ess_value(M, bc, bt[i]);
      __syncthreads();
      helm_op<NP, double>(D, Q[0], Q[1], Q[2], Q[3], q3, J.hCon, u, R, S, T, NT);
      for (int i = tid; i < NN; i += NT) F[p][i] += T[i];
    }
  }
  __syncthreads();
  // boundary-first element ordering, negated: f <- -(M f + H g)
  for (int a = tid; a < NN; a += NT) {
    const int n = emap[a];
    const double v0 = -F[0][n], v1 = -F[1][n];
    Fe[0][a] = v0;
    Fe[1][a] = v1;
    if (a >= NE) {
      f[a] = v0;
      if (P > 1) f[fs + a] = v1;
    }
  }
  cp_async_wait_all();
  __syncthreads();
  // F_b -= (hbi hii^-1) F_i: row b of the block against the interior values
  const int s = tid & 3;
  for (int b0 = 0; b0 < NE; b0 += NT / 4) {
    const int b = b0 + (tid >> 2);
    double s0 = 0.0, s1 = 0.0;
    if (b < NE) {
      const double *h = H + b * NI;
#pragma unroll 4
      for (int q = s; q < NI; q += 4) {
        s0 = fma(h[q], Fe[0][NE + q], s0);
        s1 = fma(h[q], Fe[1][NE + q], s1);
      }
    }
    s0 += __shfl_xor_sync(0xffffffffu, s0, 1);
    s1 += __shfl_xor_sync(0xffffffffu, s1, 1);
    s0 += __shfl_xor_sync(0xffffffffu, s0, 2);
    s1 += __shfl_xor_sync(0xffffffffu, s1, 2);
    if (s < P && b < NE) {  // thread 0 of the four stores plane 0, thread 1 plane 1
      const double v = Fe[s][b] - (s == 0 ? s0 : s1);
      J.Fb[((size_t)s * M.nel + e) * NE + b] = v;
      f[s * fs + b] = v;
    }
  }
}

// ---------------------------------------------------------------------------
// Direct-stiffness sum into the condensed RHS
// ---------------------------------------------------------------------------

__global__ void k_rhs_dss(MeshView M, const Job *__restrict__ jobs) {
  const Job J = jobs[blockIdx.y];
  const int g = blockIdx.x * blockDim.x + threadIdx.x;
  if (g >= J.npad) return;
  for (int p = 0; p < J.P; p++) {
    double s = 0.0;
    if (g < J.nsolve) {
      const double *fb = J.Fb + (size_t)p * M.nel * M.next;
      for (int q = M.g2e_ptr[g]; q < M.g2e_ptr[g + 1]; q++) s += fb[M.g2e_idx[q]];
      if (M.nat_ptr[g] < M.nat_ptr[g + 1]) {
        const double *bc = J.bc ? J.bc + (size_t)p * J.bcstride : nullptr;
        for (int q = M.nat_ptr[g]; q < M.nat_ptr[g + 1]; q++) {
          const int bi = M.nat_idx[q], b = bi / M.np;
          if (M.b_kind[b] == SX_BC_NATURAL)
            s += (bc ? bc[bi] : 0.0) * M.b_area[bi];
          else
            s += (M.b_K[b] * M.b_C[b]) * M.b_area[bi];
        }
      }
    }
    J.rhs[(size_t)p * J.rhs_stride + g] = s;
  }
}

// ---------------------------------------------------------------------------
// Interior back-substitution + essential values
// ---------------------------------------------------------------------------

// Threads of k_backsub: one per interior row, rounded up to whole warps.
template <int NP>
__host__ __device__ constexpr int back_threads() {
  return ((NP * NP - 4 * (NP - 1) + 31) / 32) * 32;
}

// One block per (element, job), both planes in one pass.  Thread r owns
// interior row r: u_i[r] = sum_c hii^-1[r][c] F_i[c] - sum_b (hbi hii^-1)[b][r] u_b[b].
// hii^-1 is stored column-major, so that for each c the block reads one
// contiguous column (lanes along r), as it reads the rows of hbi hii^-1:
// the element's 8 (NI + NE) NI bytes stream once from HBM, coalesced and
// evict-first, straight into the FMA chains; nothing is staged in shared
// memory but the two right-hand vectors, so many blocks share an SM and
// keep enough loads in flight.
template <int NP>
__global__ void __launch_bounds__(back_threads<NP>()) k_backsub(MeshView M, const Job *__restrict__ jobs) {
  constexpr int NN = NP * NP, NE = 4 * (NP - 1), NI = NN - NE, NT = back_threads<NP>();
  const Job J = jobs[blockIdx.y];
  const int e = blockIdx.x, tid = threadIdx.x;
  const int P = J.P;
  __shared__ double ub[2][NE], fi[2][NI];
  const size_t eo = (size_t)e * NN;
  const int *bt = M.btog + (size_t)e * NE;
  for (int b = tid; b < NE; b += NT) {
    const int g = bt[b];
    for (int p = 0; p < P; p++) ub[p][b] = (g < J.nsolve) ? J.rhs[(size_t)p * J.rhs_stride + g] : 0.0;
  }
  for (int i = tid; i < NI; i += NT)
    for (int p = 0; p < P; p++) fi[p][i] = J.f[(size_t)p * J.fstride + eo + NE + i];
  __syncthreads();
  // boundary values: the solved ones, then setEssential on masked nodes
  const bool masked = M.emask[e] != 0;
  for (int b = tid; b < NE; b += NT) {
    const int n = M.emap[b];
    const bool ess = masked && M.bmask[(size_t)e * NE + b];
    for (int p = 0; p < P; p++)
      J.u[(size_t)p * J.ustride + eo + n] =
          ess ? ess_value(M, J.bc ? J.bc + (size_t)p * J.bcstride : nullptr, bt[b]) : ub[p][b];
  }
  if (tid < NI) {
    const int r = tid;
    const double *hc = J.hii + (size_t)e * NI * NI + r;
    const double *hb = J.hbi + (size_t)e * NE * NI + r;
    double s0 = 0.0, s1 = 0.0, t0 = 0.0, t1 = 0.0;
    if (P > 1) {
#pragma unroll 9
      for (int c = 0; c < NI; c++) {
        const double v = __ldcs(hc + c * NI);
        s0 += v * fi[0][c];
        s1 += v * fi[1][c];
      }
#pragma unroll 8
      for (int b = 0; b < NE; b++) {
        const double v = __ldcs(hb + b * NI);
        t0 += v * ub[0][b];
        t1 += v * ub[1][b];
      }
    } else {
#pragma unroll 9
      for (int c = 0; c < NI; c++) s0 += __ldcs(hc + c * NI) * fi[0][c];
#pragma unroll 8
      for (int b = 0; b < NE; b++) t0 += __ldcs(hb + b * NI) * ub[0][b];
    }
    const int n = M.emap[NE + r];
    J.u[eo + n] = s0 - t0;
    if (P > 1) J.u[(size_t)J.ustride + eo + n] = s1 - t1;
  }
}

// ---------------------------------------------------------------------------
// Host launchers
// ---------------------------------------------------------------------------

template <int NP>
static void launch_elem(const MeshView &M, const Job *djobs, int njobs, bool rhs, cudaStream_t st) {
  dim3 grid(M.nel, njobs);
  if (rhs)
    k_rhs_elem<NP><<<grid, RHS_THREADS, rhs_smem<NP>(), st>>>(M, djobs);
  else
    k_backsub<NP><<<grid, back_threads<NP>(), 0, st>>>(M, djobs);
}

static void dispatch_elem(const MeshView &M, const Job *djobs, int njobs, bool rhs, cudaStream_t st) {
  switch (M.np) {
#define SX_CASE(n) \
  case n: launch_elem<n>(M, djobs, njobs, rhs, st); break;
    SX_CASE(3) SX_CASE(4) SX_CASE(5) SX_CASE(6) SX_CASE(7) SX_CASE(8) SX_CASE(9) SX_CASE(10)
    SX_CASE(11) SX_CASE(12)
#undef SX_CASE
    default: break;
  }
}

int prepare_direct_kernels(const MeshView &M) {
  if (M.np < 3 || M.np > 12) return SX_ERR_UNSUPPORTED;
  // the one order whose block and work arrays exceed 48 KB together
  if (M.np == 12)
    SX_CUDA(cudaFuncSetAttribute(k_rhs_elem<12>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)rhs_smem<12>()));
  return prepare_band_kernels();
}

int direct_rhs_jobs(const MeshView &M, const Job *djobs, const std::vector<Job> &hjobs, cudaStream_t st,
                    int *launches) {
  const int nj = (int)hjobs.size();
  int maxpad = 0;
  for (const Job &j : hjobs) {
    // the element kernels take both planes of a mode in one pass, no more
    if (j.P < 1 || j.P > 2) {
      set_error("direct solve: a job of %d planes (the element kernels take 1 or 2)", j.P);
      return SX_ERR_UNSUPPORTED;
    }
    maxpad = std::max(maxpad, j.npad);
  }
  dispatch_elem(M, djobs, nj, true, st);
  k_rhs_dss<<<dim3((maxpad + 255) / 256, nj), 256, 0, st>>>(M, djobs);
  SX_CUDA(cudaGetLastError());
  if (launches) *launches += 2;
  return SX_OK;
}

int direct_backsub_jobs(const MeshView &M, const Job *djobs, int nj, cudaStream_t st, int *launches) {
  dispatch_elem(M, djobs, nj, false, st);
  SX_CUDA(cudaGetLastError());
  if (launches) *launches += 1;
  return SX_OK;
}

int direct_solve_jobs(const MeshView &M, const Job *djobs, const std::vector<Job> &hjobs,
                      cudaStream_t st, const BandSched &sc, int *launches) {
  int nl = 0;
  SX_TRY(direct_rhs_jobs(M, djobs, hjobs, st, &nl));
  SX_TRY(band_sweep_jobs(djobs, hjobs, sc, st));
  SX_TRY(direct_backsub_jobs(M, djobs, (int)hjobs.size(), st, &nl));
  if (launches) *launches = nl + 1;
  return SX_OK;
}

}  // namespace sx

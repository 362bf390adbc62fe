// sx_fourier.cu -- z-direction (Fourier) transform of field planes.
//
// semtex's dDFTr (femlib/fourier.c:47-171) as used by AuxField::transform
// (src/auxfield.cpp:1133-1170): nz real planes of a field, point p of plane
// z at data[z * stride + p], transformed along z at every point.
//   forward (sign = +1): X_k = (1/nz) sum_j x_j exp(-2 pi i j k / nz) --
//     the sign of DMPFFT's call of DGPFA with ISIGN = -1
//     (femlib/temfftd.F:218-238) and dDFTr's 1/tlen scaling -- stored as
//     plane 0 = Re X_0, plane 1 = Re X_{nz/2} (the Nyquist datum), planes
//     2k, 2k+1 = Re X_k, Im X_k for k = 1 .. nz/2 - 1 (fourier.c:58-63);
//   inverse (sign = -1): x_j = X_0 + (-1)^j X_{nz/2} + 2 sum_{k=1}^{nz/2-1}
//     Re(X_k exp(+2 pi i j k / nz)), unscaled, so that inverse(forward(x))
//     = x.
// Lengths 2, 4, ..., 64 (config 2 uses 64): one pass, k_z_fwd / k_z_inv; the
// other lengths up to 512: one pass through shared memory, k_z_fwd_any /
// k_z_inv_any (256, and 128 on smaller fields: k_z_fwd_s / k_z_inv_s).
// A thread holds one point's whole z-line in registers: the real transform
// of length N is a complex FFT of length M = N/2 on z_m = x_2m + i x_2m+1
// (radix-2, decimation in time, every index a compile-time constant), then
// the split X_k = E_k + W^k O_k with E_k = (Z_k + conj Z_{M-k})/2, O_k =
// (Z_k - conj Z_{M-k})/2i, W = exp(-2 pi i / N); the inverse runs the same
// steps backwards.  A warp's loads and stores of one plane are 32
// consecutive doubles; the field is read once and written once.  Other
// lengths: cuFFT's batched real transform (one transform per point, element
// stride = the plane stride, loaded on first use) into a half-spectrum
// workspace [nz/2 + 1][npts], and this file's packing kernels.
#include <dlfcn.h>

#include <algorithm>
#include <cmath>
#include <vector>
#include <map>
#include <mutex>
#include <tuple>

#include <cufft.h>

#include "sx_internal.h"

namespace sx {

namespace {

// cuFFT entry points, resolved from the shared library at first use.
struct CufftApi {
  decltype(&cufftPlanMany) planMany = nullptr;
  decltype(&cufftSetStream) setStream = nullptr;
  decltype(&cufftExecD2Z) execD2Z = nullptr;
  decltype(&cufftExecZ2D) execZ2D = nullptr;
  decltype(&cufftDestroy) destroy = nullptr;
  bool ok = false;
};

const CufftApi &cufft_api() {
  static CufftApi api;
  static std::once_flag once;
  std::call_once(once, []() {
    void *h = dlopen("libcufft.so.11", RTLD_NOW | RTLD_LOCAL);
    if (!h) h = dlopen("libcufft.so", RTLD_NOW | RTLD_LOCAL);
    if (!h) return;
    api.planMany = reinterpret_cast<decltype(&cufftPlanMany)>(dlsym(h, "cufftPlanMany"));
    api.setStream = reinterpret_cast<decltype(&cufftSetStream)>(dlsym(h, "cufftSetStream"));
    api.execD2Z = reinterpret_cast<decltype(&cufftExecD2Z)>(dlsym(h, "cufftExecD2Z"));
    api.execZ2D = reinterpret_cast<decltype(&cufftExecZ2D)>(dlsym(h, "cufftExecZ2D"));
    api.destroy = reinterpret_cast<decltype(&cufftDestroy)>(dlsym(h, "cufftDestroy"));
    api.ok = api.planMany && api.setStream && api.execD2Z && api.execZ2D && api.destroy;
  });
  return api;
}

// Plans and workspaces per (device, nz, npts, stride, direction), kept for
// the life of the process (a plan is a few kB; the workspace is the
// half-spectrum).
struct ZPlan {
  cufftHandle plan = 0;
  DBuf<double2> spec;  // [nz/2 + 1][npts]
};
std::mutex g_mu;
std::map<std::tuple<int, int, int, int, int>, std::unique_ptr<ZPlan>> g_plans;

bool factors_235(int n) {
  for (int f : {2, 3, 5})
    while (n % f == 0) n /= f;
  return n == 1;
}

}  // namespace

// exp(-2 pi i t / TWN), t = 0 .. TWN/2; a length-L stage uses t = j * (TWN / L).
// Part of the module's image, so that every device and context has it and the
// first call may be a captured one.  (As a kernel parameter, which the mixed-
// radix kernels' table of any length has to be, 4 KB cost a short launch 2.5
// us.)
constexpr int TWN = 256;
// cos(2 pi t / 256), t = 0 .. 64, correctly rounded
constexpr double QUARTER[TWN / 4 + 1] = {
    1.0, 0.9996988186962042, 0.9987954562051724, 0.9972904566786902, 0.9951847266721969,
    0.99247953459871, 0.989176509964781, 0.9852776423889412, 0.9807852804032304, 0.9757021300385286,
    0.970031253194544, 0.9637760657954398, 0.9569403357322088, 0.9495281805930367, 0.9415440651830208,
    0.9329927988347388, 0.9238795325112867, 0.9142097557035307, 0.9039892931234433, 0.8932243011955153,
    0.881921264348355, 0.8700869911087115, 0.8577286100002721, 0.8448535652497071, 0.8314696123025452,
    0.8175848131515837, 0.8032075314806449, 0.7883464276266062, 0.773010453362737, 0.7572088465064846,
    0.7409511253549591, 0.7242470829514669, 0.7071067811865476, 0.6895405447370669, 0.6715589548470184,
    0.6531728429537768, 0.6343932841636455, 0.6152315905806268, 0.5956993044924334, 0.5758081914178453,
    0.5555702330196022, 0.5349976198870973, 0.5141027441932218, 0.49289819222978404, 0.47139673682599764,
    0.4496113296546066, 0.4275550934302821, 0.40524131400498986, 0.3826834323650898, 0.35989503653498817,
    0.33688985339222005, 0.31368174039889146, 0.2902846772544624, 0.26671275747489837, 0.2429801799032639,
    0.2191012401568698, 0.19509032201612828, 0.17096188876030122, 0.14673047445536175, 0.1224106751992162,
    0.0980171403295606, 0.07356456359966743, 0.049067674327418015, 0.024541228522912288, 0.0};
struct Twiddles {
  double c[TWN / 2 + 1], s[TWN / 2 + 1];
  constexpr Twiddles() : c(), s() {
    for (int t = 0; t <= TWN / 2; t++) {
      c[t] = t <= TWN / 4 ? QUARTER[t] : -QUARTER[TWN / 2 - t];
      s[t] = t <= TWN / 4 ? -QUARTER[TWN / 4 - t] : -QUARTER[t - TWN / 4];
    }
  }
};
__constant__ Twiddles c_tw;  // constant-initialised

constexpr int ilog2c(int n) { return n <= 1 ? 0 : 1 + ilog2c(n / 2); }
constexpr int bitrev(int v, int bits) {
  int r = 0;
  for (int b = 0; b < bits; b++) {
    r = (r << 1) | (v & 1);
    v >>= 1;
  }
  return r;
}

// One radix-2 stage (butterflies of span LEN) of an in-place decimation-in-
// time FFT of length M, then the next stage; INV conjugates the twiddles.
// Stages are template instances so that every register index is a
// compile-time constant.
template <int M, int LEN, bool INV>
struct FftStage {
  static __device__ __forceinline__ void run(double (&re)[M], double (&im)[M]) {
#pragma unroll
    for (int i = 0; i < M; i += LEN) {
#pragma unroll
      for (int j = 0; j < LEN / 2; j++) {
        const int t = j * (TWN / LEN);
        const double wr = c_tw.c[t], wi = INV ? -c_tw.s[t] : c_tw.s[t];
        const int a = i + j, b = i + j + LEN / 2;
        const double vr = re[b] * wr - im[b] * wi, vi = re[b] * wi + im[b] * wr;
        re[b] = re[a] - vr;
        im[b] = im[a] - vi;
        re[a] += vr;
        im[a] += vi;
      }
    }
    FftStage<M, LEN * 2, INV>::run(re, im);
  }
};
template <int M, bool INV>
struct FftStage<M, M * 2, INV> {
  static __device__ __forceinline__ void run(double (&)[M], double (&)[M]) {}
};

// In-place radix-2 FFT of length M on bit-reversed input, natural-order
// output, unscaled.
template <int M, bool INV>
__device__ __forceinline__ void cfft_reg(double (&re)[M], double (&im)[M]) {
  FftStage<M, 2, INV>::run(re, im);
}

template <int N>
__global__ void __launch_bounds__(128) k_z_fwd(double *__restrict__ data, int npts, long long stride, double scale) {
  constexpr int M = N / 2, LB = ilog2c(M);
  const int p = blockIdx.x * 128 + threadIdx.x;
  if (p >= npts) return;
  double re[M], im[M];
#pragma unroll
  for (int m = 0; m < M; m++) {
    re[bitrev(m, LB)] = data[(2 * m) * stride + p];
    im[bitrev(m, LB)] = data[(2 * m + 1) * stride + p];
  }
  cfft_reg<M, false>(re, im);
  // k = 0: E_0 = Re Z_0, O_0 = Im Z_0; X_0 = E_0 + O_0, X_M = E_0 - O_0
  data[p] = (re[0] + im[0]) * scale;
  data[stride + p] = (re[0] - im[0]) * scale;
#pragma unroll
  for (int k = 1; k < M; k++) {
    const double yr = re[M - k], yi = -im[M - k];  // conj Z_{M-k}
    const double er = 0.5 * (re[k] + yr), ei = 0.5 * (im[k] + yi);
    const double orr = 0.5 * (im[k] - yi), oi = -0.5 * (re[k] - yr);  // (Z_k - conj Z_{M-k}) / 2i
    const int t = k * (TWN / N);
    const double wr = c_tw.c[t], wi = c_tw.s[t];
    data[(2 * k) * stride + p] = (er + (orr * wr - oi * wi)) * scale;
    data[(2 * k + 1) * stride + p] = (ei + (orr * wi + oi * wr)) * scale;
  }
}

template <int N>
__global__ void __launch_bounds__(128) k_z_inv(double *__restrict__ data, int npts, long long stride) {
  constexpr int M = N / 2, LB = ilog2c(M);
  const int p = blockIdx.x * 128 + threadIdx.x;
  if (p >= npts) return;
  double re[M], im[M];
  {
    // k = 0: E_0 = (X_0 + X_M)/2, O_0 = (X_0 - X_M)/2, Z_0 = E_0 + i O_0
    const double x0 = data[p], xm = data[stride + p];
    re[0] = 0.5 * (x0 + xm);
    im[0] = 0.5 * (x0 - xm);
  }
  // E_k = (X_k + conj X_{M-k})/2, O_k = (X_k - conj X_{M-k}) conj(W^k)/2,
  // Z_k = E_k + i O_k, for k and M - k together
#pragma unroll
  for (int k = 1; k <= M / 2; k++) {
    const int kk = M - k;
    const double ar = data[(2 * k) * stride + p], ai = data[(2 * k + 1) * stride + p];
    const double br = data[(2 * kk) * stride + p], bi = data[(2 * kk + 1) * stride + p];
#pragma unroll
    for (int side = 0; side < (k == kk ? 1 : 2); side++) {
      const int q = side ? kk : k;
      const double xr = side ? br : ar, xi = side ? bi : ai;   // X_q
      const double cr = side ? ar : br, ci = side ? -ai : -bi;  // conj X_{M-q}
      const double er = 0.5 * (xr + cr), ei = 0.5 * (xi + ci);
      const double dr = 0.5 * (xr - cr), di = 0.5 * (xi - ci);
      const int t = q * (TWN / N);
      const double wr = c_tw.c[t], wi = -c_tw.s[t];  // conj W^q
      const double orr = dr * wr - di * wi, oi = dr * wi + di * wr;
      re[bitrev(q, LB)] = er - oi;  // E + i O
      im[bitrev(q, LB)] = ei + orr;
    }
  }
  cfft_reg<M, true>(re, im);
#pragma unroll
  for (int m = 0; m < M; m++) {
    data[(2 * m) * stride + p] = 2.0 * re[m];
    data[(2 * m + 1) * stride + p] = 2.0 * im[m];
  }
}

// Lengths 256 and, on smaller fields, 128: a block of eight warps takes 32
// points (lane = point); the half-length complex sequence z (length M = N/2) of
// each point lies in shared memory, Zr/Zi[m][32], in natural order.  The
// complex FFT of length M = M1 M2 runs in four steps with m = M2 m1 + m2 and
// k = k1 + M1 k2: (1) the M2 FFTs of length M1 over m1, each a warp's, in
// registers; (2) the twiddles W_M^(m2 k1); (3) the M1 FFTs of length M2
// over m2, in registers.  Two round trips through shared memory and two
// barriers, against one per radix-2 stage (log2 M).  Z_k ends at row
// M2 (k mod M1) + k / M1.  The real-to-complex steps around it are the
// register kernels'; loads and stores of a plane are 32 consecutive doubles.
constexpr size_t zsmem(int nz) { return (size_t)nz * 32 * sizeof(double); }
constexpr int ZW = 8;  // warps a block: every sub-FFT of a pass at once

template <int M>
struct FourStep {
  static constexpr int M1 = M >= 128 ? 16 : 8, M2 = M / M1;
  static __device__ __forceinline__ int row(int k) { return M2 * (k % M1) + k / M1; }
};

// W_M^e = exp(-2 pi i e / M) from the half-turn table (conjugated for the
// inverse).
template <int M>
__device__ __forceinline__ void twiddle(int e, bool inv, double &wr, double &wi) {
  e &= M - 1;
  const bool neg = e >= M / 2;
  const int t = (neg ? e - M / 2 : e) * (TWN / M);
  wr = neg ? -c_tw.c[t] : c_tw.c[t];
  wi = neg ? -c_tw.s[t] : c_tw.s[t];
  if (inv) wi = -wi;
}

template <int M, bool INV>
__device__ __forceinline__ void four_step(double *Zr, double *Zi) {
  using F = FourStep<M>;
  constexpr int M1 = F::M1, M2 = F::M2, L1 = ilog2c(M1), L2 = ilog2c(M2);
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;  // ZW warps
  for (int m2 = w; m2 < M2; m2 += ZW) {
    double re[M1], im[M1];
#pragma unroll
    for (int m1 = 0; m1 < M1; m1++) {
      re[bitrev(m1, L1)] = Zr[(M2 * m1 + m2) * 32 + lane];
      im[bitrev(m1, L1)] = Zi[(M2 * m1 + m2) * 32 + lane];
    }
    cfft_reg<M1, INV>(re, im);
#pragma unroll
    for (int k1 = 0; k1 < M1; k1++) {
      double wr, wi;
      twiddle<M>(m2 * k1, INV, wr, wi);
      const double xr = re[k1] * wr - im[k1] * wi, xi = re[k1] * wi + im[k1] * wr;
      Zr[(M2 * k1 + m2) * 32 + lane] = xr;
      Zi[(M2 * k1 + m2) * 32 + lane] = xi;
    }
  }
  __syncthreads();
  for (int k1 = w; k1 < M1; k1 += ZW) {
    double re[M2], im[M2];
#pragma unroll
    for (int m2 = 0; m2 < M2; m2++) {
      re[bitrev(m2, L2)] = Zr[(M2 * k1 + m2) * 32 + lane];
      im[bitrev(m2, L2)] = Zi[(M2 * k1 + m2) * 32 + lane];
    }
    cfft_reg<M2, INV>(re, im);
#pragma unroll
    for (int k2 = 0; k2 < M2; k2++) {
      Zr[(M2 * k1 + k2) * 32 + lane] = re[k2];
      Zi[(M2 * k1 + k2) * 32 + lane] = im[k2];
    }
  }
  __syncthreads();
}

template <int N>
__global__ void __launch_bounds__(ZW * 32, 3) k_z_fwd_s(double *__restrict__ data, int npts, long long stride,
                                                  double scale) {
  constexpr int M = N / 2;
  using F = FourStep<M>;
  extern __shared__ __align__(16) double zs[];
  double *Zr = zs, *Zi = zs + M * 32;
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;  // ZW warps
  const int p = blockIdx.x * 32 + lane;
  const bool ok = p < npts;
#pragma unroll 4
  for (int m = w; m < M; m += ZW) {
    Zr[m * 32 + lane] = ok ? data[(2 * m) * stride + p] : 0.0;
    Zi[m * 32 + lane] = ok ? data[(2 * m + 1) * stride + p] : 0.0;
  }
  __syncthreads();
  four_step<M, false>(Zr, Zi);
  if (!ok) return;  // no barrier follows
#pragma unroll 2
  for (int k = w; k <= M / 2; k += ZW) {
    if (k == 0) {
      const int r0 = F::row(0);
      data[p] = (Zr[r0 * 32 + lane] + Zi[r0 * 32 + lane]) * scale;
      data[stride + p] = (Zr[r0 * 32 + lane] - Zi[r0 * 32 + lane]) * scale;
      continue;
    }
    // X_k from Z_k and conj Z_{M-k}; and X_{M-k} from the same pair
    const int kk = M - k, rk = F::row(k), rkk = F::row(kk);
    const double zr = Zr[rk * 32 + lane], zi = Zi[rk * 32 + lane];
    const double qr = Zr[rkk * 32 + lane], qi = Zi[rkk * 32 + lane];
    for (int side = 0; side < (k == kk ? 1 : 2); side++) {
      const int q = side ? kk : k;
      const double ar = side ? qr : zr, ai = side ? qi : zi;   // Z_q
      const double yr = side ? zr : qr, yi = side ? -zi : -qi;  // conj Z_{M-q}
      const double er = 0.5 * (ar + yr), ei = 0.5 * (ai + yi);
      const double orr = 0.5 * (ai - yi), oi = -0.5 * (ar - yr);
      const int t = q * (TWN / N);
      const double wr = c_tw.c[t], wi = c_tw.s[t];
      data[(2 * q) * stride + p] = (er + (orr * wr - oi * wi)) * scale;
      data[(2 * q + 1) * stride + p] = (ei + (orr * wi + oi * wr)) * scale;
    }
  }
}

template <int N>
__global__ void __launch_bounds__(ZW * 32, 3) k_z_inv_s(double *__restrict__ data, int npts, long long stride) {
  constexpr int M = N / 2;
  using F = FourStep<M>;
  extern __shared__ __align__(16) double zs[];
  double *Zr = zs, *Zi = zs + M * 32;
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;  // ZW warps
  const int p = blockIdx.x * 32 + lane;
  const bool ok = p < npts;
#pragma unroll 2
  for (int k = w; k <= M / 2; k += ZW) {
    if (k == 0) {
      const double x0 = ok ? data[p] : 0.0, xm = ok ? data[stride + p] : 0.0;
      Zr[0 * 32 + lane] = 0.5 * (x0 + xm);
      Zi[0 * 32 + lane] = 0.5 * (x0 - xm);
      continue;
    }
    const int kk = M - k;
    const double ar = ok ? data[(2 * k) * stride + p] : 0.0, ai = ok ? data[(2 * k + 1) * stride + p] : 0.0;
    const double br = ok ? data[(2 * kk) * stride + p] : 0.0, bi = ok ? data[(2 * kk + 1) * stride + p] : 0.0;
    for (int side = 0; side < (k == kk ? 1 : 2); side++) {
      const int q = side ? kk : k;
      const double xr = side ? br : ar, xi = side ? bi : ai;
      const double cr = side ? ar : br, ci = side ? -ai : -bi;
      const double er = 0.5 * (xr + cr), ei = 0.5 * (xi + ci);
      const double dr = 0.5 * (xr - cr), di = 0.5 * (xi - ci);
      const int t = q * (TWN / N);
      const double wr = c_tw.c[t], wi = -c_tw.s[t];
      const double orr = dr * wr - di * wi, oi = dr * wi + di * wr;
      Zr[q * 32 + lane] = er - oi;
      Zi[q * 32 + lane] = ei + orr;
    }
  }
  __syncthreads();
  four_step<M, true>(Zr, Zi);
  if (!ok) return;
#pragma unroll 4
  for (int m = w; m < M; m += ZW) {
    const int r = F::row(m);
    data[(2 * m) * stride + p] = 2.0 * Zr[r * 32 + lane];
    data[(2 * m + 1) * stride + p] = 2.0 * Zi[r * 32 + lane];
  }
}

// A kernel's limit on dynamic shared memory is a setting of the current
// device's copy of it, so every launch of more than the default limit allows
// (48 KB, with up to 1 KB of tables) sets it, to the kernel's `most`: callers
// do not disturb one another.
template <typename K>
static cudaError_t dynamic_smem(K *kernel, size_t bytes, size_t most) {
  if (bytes <= 47 * 1024) return cudaSuccess;
  return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)most);
}

template <int N>
static int launch_smem(double *d, int npts, long long stride, int sign, cudaStream_t st) {
  const int grid = (npts + 31) / 32;
  if (sign == 1) {
    SX_CUDA(dynamic_smem(k_z_fwd_s<N>, zsmem(N), zsmem(N)));
    k_z_fwd_s<N><<<grid, ZW * 32, zsmem(N), st>>>(d, npts, stride, 1.0 / N);
  } else {
    SX_CUDA(dynamic_smem(k_z_inv_s<N>, zsmem(N), zsmem(N)));
    k_z_inv_s<N><<<grid, ZW * 32, zsmem(N), st>>>(d, npts, stride);
  }
  return SX_OK;
}

// ---------------------------------------------------------------------------
// every other even length up to ZN_MAX with prime factors 2, 3, 5
// ---------------------------------------------------------------------------
//
// The complex FFT of length M = N / 2 of 32 points (lane = point) in two or
// three in-place stages over shared memory, Zr/Zi[row][32] (the decimation in
// frequency of Gentleman & Sande 1966, mixed radix): a stage of radix R over
// sub-sequences of length n = R L takes rows j, j + L, ... of a sub-sequence
// into registers, a warp each, transforms them, multiplies output k by
// W_n^(j k) and puts it back at row j + k L; the next stage works on the R
// sub-sequences of length L.  X_K ends at the row whose mixed-radix digits are
// K's, reversed.
//   What bounds it is HBM (a field is read and written once), so the stages
// next to global memory skip the shared-memory trip: forward, the first stage
// reads its rows from the planes; inverse, the last one writes its outputs to
// them.  The real-to-complex split needs rows k and M - k together and stays
// on the shared-memory side.  A block holds PG groups of 32 points, so that a
// short M still gives every warp a sub-transform.
//   Measured (forward / inverse, L2 flushed; before: cuFFT's batched transform
// into a workspace and a packing pass, or for 128 and 512 one radix-2 four-step
// kernel pair with a load and a store pass of its own): 24 x 495,616 points
// 98/99 -> 50/60 us, 96 x 82,944 75/73 -> 44/46, 120 x 82,944 86/88 -> 54/58,
// 128 x 495,616 261/283 -> 241/276, 240 x 82,944 185/201 -> 110/124,
// 512 x 82,944 290/375 -> 220/321.
constexpr int ZN_MAX = 512, ZST = 5;

// exp(-2 pi i t / N), t = 0 .. N / 2, and the stages: a kernel parameter, so
// that warp-uniform reads are constant-cache broadcasts and nothing is kept
// on the device between calls.
struct ZPlan235 {
  double c[ZN_MAX / 2 + 1], s[ZN_MAX / 2 + 1];
  int N, M, PG, nst, radix[ZST];
};

// W_N^t (conjugated for the inverse), 0 <= t < N.
template <bool INV>
__device__ __forceinline__ void zw(const ZPlan235 &Z, int t, double &wr, double &wi) {
  const int h = Z.M;
  const bool neg = t >= h;
  const int i = neg ? t - h : t;
  wr = neg ? -Z.c[i] : Z.c[i];
  wi = (neg != INV) ? -Z.s[i] : Z.s[i];
}

// DFT of length R in registers, natural order in and out, unscaled.
template <int R, bool INV>
struct Dft;
template <bool INV>
struct Dft<2, INV> {
  static __device__ __forceinline__ void run(const ZPlan235 &, double (&re)[2], double (&im)[2]) {
    const double ar = re[0], ai = im[0];
    re[0] += re[1];
    im[0] += im[1];
    re[1] = ar - re[1];
    im[1] = ai - im[1];
  }
};
template <bool INV>
struct Dft<4, INV> {
  static __device__ __forceinline__ void run(const ZPlan235 &, double (&re)[4], double (&im)[4]) {
    const double ar = re[0] + re[2], ai = im[0] + im[2], br = re[0] - re[2], bi = im[0] - im[2];
    const double cr = re[1] + re[3], ci = im[1] + im[3];
    const double dr = INV ? im[3] - im[1] : im[1] - im[3];  // -+ i (x1 - x3)
    const double di = INV ? re[1] - re[3] : re[3] - re[1];
    re[0] = ar + cr;
    im[0] = ai + ci;
    re[1] = br + dr;
    im[1] = bi + di;
    re[2] = ar - cr;
    im[2] = ai - ci;
    re[3] = br - dr;
    im[3] = bi - di;
  }
};
template <bool INV>
struct Dft<8, INV> {
  static __device__ __forceinline__ void run(const ZPlan235 &Z, double (&re)[8], double (&im)[8]) {
    constexpr double H = 0.70710678118654752440;  // cos(pi / 4)
    double er[4] = {re[0], re[2], re[4], re[6]}, ei[4] = {im[0], im[2], im[4], im[6]};
    double orr[4] = {re[1], re[3], re[5], re[7]}, oi[4] = {im[1], im[3], im[5], im[7]};
    Dft<4, INV>::run(Z, er, ei);
    Dft<4, INV>::run(Z, orr, oi);
    // W_8^k O_k: (1 -+ i) / sqrt 2, -+ i, (-1 -+ i) / sqrt 2
    const double ar = INV ? H * (orr[1] - oi[1]) : H * (orr[1] + oi[1]);
    const double ai = INV ? H * (oi[1] + orr[1]) : H * (oi[1] - orr[1]);
    const double br = INV ? -oi[2] : oi[2], bi = INV ? orr[2] : -orr[2];
    const double cr = INV ? -H * (orr[3] + oi[3]) : H * (oi[3] - orr[3]);
    const double ci = INV ? H * (orr[3] - oi[3]) : -H * (orr[3] + oi[3]);
    orr[1] = ar;
    oi[1] = ai;
    orr[2] = br;
    oi[2] = bi;
    orr[3] = cr;
    oi[3] = ci;
#pragma unroll
    for (int k = 0; k < 4; k++) {
      re[k] = er[k] + orr[k];
      im[k] = ei[k] + oi[k];
      re[k + 4] = er[k] - orr[k];
      im[k + 4] = ei[k] - oi[k];
    }
  }
};
template <bool INV>
struct Dft<3, INV> {
  static __device__ __forceinline__ void run(const ZPlan235 &, double (&re)[3], double (&im)[3]) {
    constexpr double S = INV ? 0.86602540378443864676 : -0.86602540378443864676;  // -+ sin(2 pi / 3)
    const double tr = re[1] + re[2], ti = im[1] + im[2], dr = S * (re[1] - re[2]), di = S * (im[1] - im[2]);
    const double mr = re[0] - 0.5 * tr, mi = im[0] - 0.5 * ti;
    re[0] += tr;
    im[0] += ti;
    re[1] = mr - di;
    im[1] = mi + dr;
    re[2] = mr + di;
    im[2] = mi - dr;
  }
};
template <bool INV>
struct Dft<5, INV> {
  static __device__ __forceinline__ void run(const ZPlan235 &, double (&re)[5], double (&im)[5]) {
    constexpr double C1 = 0.30901699437494742410, C2 = -0.80901699437494742410;  // cos(2 pi / 5), cos(4 pi / 5)
    constexpr double S1 = INV ? 0.95105651629515357212 : -0.95105651629515357212;
    constexpr double S2 = INV ? 0.58778525229247312917 : -0.58778525229247312917;
    const double ar = re[1] + re[4], ai = im[1] + im[4], br = re[2] + re[3], bi = im[2] + im[3];
    const double cr = re[1] - re[4], ci = im[1] - im[4], dr = re[2] - re[3], di = im[2] - im[3];
    const double pr = re[0] + C1 * ar + C2 * br, pi = im[0] + C1 * ai + C2 * bi;
    const double qr = re[0] + C2 * ar + C1 * br, qi = im[0] + C2 * ai + C1 * bi;
    const double ur = S1 * cr + S2 * dr, ui = S1 * ci + S2 * di;
    const double vr = S2 * cr - S1 * dr, vi = S2 * ci - S1 * di;
    re[0] += ar + br;
    im[0] += ai + bi;
    re[1] = pr - ui;
    im[1] = pi + ur;
    re[4] = pr + ui;
    im[4] = pi - ur;
    re[2] = qr - vi;
    im[2] = qi + vr;
    re[3] = qr + vi;
    im[3] = qi - vr;
  }
};
// R = A B: A-point transforms of every B-th value, twiddles, B-point ones.
template <int A, int B, bool INV>
struct DftAB {
  static constexpr int R = A * B;
  static __device__ __forceinline__ void run(const ZPlan235 &Z, double (&re)[R], double (&im)[R]) {
    const int u = Z.N / R;
#pragma unroll
    for (int b = 0; b < B; b++) {
      double x[A], y[A];
#pragma unroll
      for (int a = 0; a < A; a++) {
        x[a] = re[a * B + b];
        y[a] = im[a * B + b];
      }
      Dft<A, INV>::run(Z, x, y);
#pragma unroll
      for (int k = 0; k < A; k++) {
        if (b * k == 0) {
          re[k * B + b] = x[k];
          im[k * B + b] = y[k];
        } else {
          double wr, wi;
          zw<INV>(Z, b * k * u, wr, wi);
          re[k * B + b] = x[k] * wr - y[k] * wi;
          im[k * B + b] = x[k] * wi + y[k] * wr;
        }
      }
    }
    double ur[R], ui[R];
#pragma unroll
    for (int k = 0; k < A; k++) {
      double x[B], y[B];
#pragma unroll
      for (int b = 0; b < B; b++) {
        x[b] = re[k * B + b];
        y[b] = im[k * B + b];
      }
      Dft<B, INV>::run(Z, x, y);
#pragma unroll
      for (int l = 0; l < B; l++) {
        ur[k + A * l] = x[l];
        ui[k + A * l] = y[l];
      }
    }
#pragma unroll
    for (int q = 0; q < R; q++) {
      re[q] = ur[q];
      im[q] = ui[q];
    }
  }
};
template <bool INV> struct Dft<6, INV> : DftAB<2, 3, INV> {};
template <bool INV> struct Dft<9, INV> : DftAB<3, 3, INV> {};
template <bool INV> struct Dft<10, INV> : DftAB<2, 5, INV> {};
template <bool INV> struct Dft<12, INV> : DftAB<4, 3, INV> {};
template <bool INV> struct Dft<15, INV> : DftAB<3, 5, INV> {};
template <bool INV> struct Dft<16, INV> : DftAB<4, 4, INV> {};
constexpr int Z_RADIX[] = {16, 15, 12, 10, 9, 8, 6, 5, 4, 3, 2};

// One stage of radix R over sub-sequences of length n: the block's tasks go
// round its warps.  FROM: the rows come from the planes (forward's first
// stage); TO: the outputs go to the planes (inverse's last).
template <int R, bool INV>
__device__ __forceinline__ void z_stage(const ZPlan235 &Z, double *Zr, double *Zi, int n, bool from, bool to,
                                        int before, double *data, int npts, long long stride) {
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31, nw = blockDim.x >> 5;
  const int L = n / R, per = Z.M / R, u = Z.N / n;
  for (int idx = w; idx < Z.PG * per; idx += nw) {
    const int g = idx / per, o = idx - g * per, sb = o / L, j = o - sb * L;
    const int p = (blockIdx.x * Z.PG + g) * 32 + lane, row = sb * n + j;
    const bool ok = p < npts;
    double *zr = Zr + (size_t)g * Z.M * 32 + lane, *zi = Zi + (size_t)g * Z.M * 32 + lane;
    double re[R], im[R];
    if (from) {
#pragma unroll
      for (int q = 0; q < R; q++) {
        const double *d = data + (long long)(2 * (row + q * L)) * stride + p;
        re[q] = ok ? d[0] : 0.0;
        im[q] = ok ? d[stride] : 0.0;
      }
    } else {
#pragma unroll
      for (int q = 0; q < R; q++) {
        re[q] = zr[(row + q * L) * 32];
        im[q] = zi[(row + q * L) * 32];
      }
    }
    Dft<R, INV>::run(Z, re, im);
    if (to) {
      // L = 1: output k is X_K with K's last digit k and the others sb's,
      // reversed; z_m = x_2m + i x_2m+1
      int K = 0, v = sb, weight = before;
      for (int st = Z.nst - 2; st >= 0; st--) {
        weight /= Z.radix[st];
        K += (v % Z.radix[st]) * weight;
        v /= Z.radix[st];
      }
      if (ok) {
#pragma unroll
        for (int k = 0; k < R; k++) {
          double *d = data + (long long)(2 * (K + k * before)) * stride + p;
          d[0] = 2.0 * re[k];
          d[stride] = 2.0 * im[k];
        }
      }
      continue;
    }
    zr[row * 32] = re[0];
    zi[row * 32] = im[0];
#pragma unroll
    for (int k = 1; k < R; k++) {
      double wr, wi;
      zw<INV>(Z, j * k * u, wr, wi);
      zr[(row + k * L) * 32] = re[k] * wr - im[k] * wi;
      zi[(row + k * L) * 32] = re[k] * wi + im[k] * wr;
    }
  }
  __syncthreads();
}

template <int RMAX, bool INV>
__device__ __forceinline__ void z_stages(const ZPlan235 &Z, double *Zr, double *Zi, double *data, int npts,
                                         long long stride) {
  int n = Z.M, before = 1;  // before: the product of the earlier stages' radices
  for (int st = 0; st < Z.nst; st++) {
    const int R = Z.radix[st];
    const bool from = !INV && st == 0, to = INV && st == Z.nst - 1;
    switch (R) {
#define SX_ZCASE(r)                                                                                  \
  case r:                                                                                            \
    if constexpr (r <= RMAX) z_stage<r, INV>(Z, Zr, Zi, n, from, to, before, data, npts, stride);     \
    break;
      SX_ZCASE(2) SX_ZCASE(3) SX_ZCASE(4) SX_ZCASE(5) SX_ZCASE(6) SX_ZCASE(8)
      SX_ZCASE(9) SX_ZCASE(10) SX_ZCASE(12) SX_ZCASE(15) SX_ZCASE(16)
#undef SX_ZCASE
    }
    n /= R;
    before *= R;
  }
}

// The row of X_K after the stages.
__device__ __forceinline__ int z_row(const ZPlan235 &Z, int K) {
  int row = 0, n = Z.M;
  for (int st = 0; st < Z.nst; st++) {
    const int R = Z.radix[st];
    n /= R;
    row += (K % R) * n;
    K /= R;
  }
  return row;
}

template <int NT, int MINB, int RMAX>
__global__ void __launch_bounds__(NT, MINB) k_z_fwd_any(const __grid_constant__ ZPlan235 Z, double *__restrict__ data,
                                                        int npts, long long stride, double scale) {
  extern __shared__ __align__(16) double zs[];
  __shared__ short rowt[ZN_MAX / 2];
  const int M = Z.M;
  double *Zr = zs, *Zi = zs + (size_t)Z.PG * M * 32;
  for (int k = threadIdx.x; k < M; k += NT) rowt[k] = (short)z_row(Z, k);
  z_stages<RMAX, false>(Z, Zr, Zi, data, npts, stride);
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int per = M / 2 + 1;
  for (int idx = w; idx < Z.PG * per; idx += NT / 32) {
    const int g = idx / per, k = idx - g * per, p = (blockIdx.x * Z.PG + g) * 32 + lane;
    if (p >= npts) continue;
    const double *zr = Zr + (size_t)g * M * 32 + lane, *zi = Zi + (size_t)g * M * 32 + lane;
    double *d = data + p;
    if (k == 0) {
      const double a = zr[0], b = zi[0];
      d[0] = (a + b) * scale;
      d[stride] = (a - b) * scale;
      continue;
    }
    // X_k from Z_k and conj Z_{M-k}; and X_{M-k} from the same pair
    const int kk = M - k, rk = rowt[k] * 32, rkk = rowt[kk] * 32;
    const double ar = zr[rk], ai = zi[rk], br = zr[rkk], bi = zi[rkk];
    const double er = 0.5 * (ar + br), ei = 0.5 * (ai - bi);    // E_k; E_{M-k} is its conjugate
    const double orr = 0.5 * (ai + bi), oi = -0.5 * (ar - br);  // O_k
    double wr, wi;
    zw<false>(Z, k, wr, wi);
    const double tr = orr * wr - oi * wi, ti = orr * wi + oi * wr;  // W^k O_k
    d[(2 * k) * stride] = (er + tr) * scale;
    d[(2 * k + 1) * stride] = (ei + ti) * scale;
    if (k != kk) {  // X_{M-k} = conj(E_k - W^k O_k)
      d[(2 * kk) * stride] = (er - tr) * scale;
      d[(2 * kk + 1) * stride] = (ti - ei) * scale;
    }
  }
}

template <int NT, int MINB, int RMAX>
__global__ void __launch_bounds__(NT, MINB) k_z_inv_any(const __grid_constant__ ZPlan235 Z, double *__restrict__ data,
                                                        int npts, long long stride) {
  extern __shared__ __align__(16) double zs[];
  const int M = Z.M;
  double *Zr = zs, *Zi = zs + (size_t)Z.PG * M * 32;
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int per = M / 2 + 1;
#pragma unroll 2
  for (int idx = w; idx < Z.PG * per; idx += NT / 32) {
    const int g = idx / per, k = idx - g * per, p = (blockIdx.x * Z.PG + g) * 32 + lane;
    const bool ok = p < npts;
    double *zr = Zr + (size_t)g * M * 32 + lane, *zi = Zi + (size_t)g * M * 32 + lane;
    const double *d = data + p;
    if (k == 0) {
      const double x0 = ok ? d[0] : 0.0, xm = ok ? d[stride] : 0.0;
      zr[0] = 0.5 * (x0 + xm);
      zi[0] = 0.5 * (x0 - xm);
      continue;
    }
    // E_k = (X_k + conj X_{M-k}) / 2, O_k = (X_k - conj X_{M-k}) conj(W^k) / 2,
    // Z_k = E_k + i O_k and Z_{M-k} = conj(E_k) + i conj(O_k)
    const int kk = M - k;
    const double ar = ok ? d[(2 * k) * stride] : 0.0, ai = ok ? d[(2 * k + 1) * stride] : 0.0;
    const double br = ok ? d[(2 * kk) * stride] : 0.0, bi = ok ? d[(2 * kk + 1) * stride] : 0.0;
    const double er = 0.5 * (ar + br), ei = 0.5 * (ai - bi), dr = 0.5 * (ar - br), di = 0.5 * (ai + bi);
    double wr, wi;
    zw<true>(Z, k, wr, wi);
    const double orr = dr * wr - di * wi, oi = dr * wi + di * wr;
    zr[k * 32] = er - oi;
    zi[k * 32] = ei + orr;
    if (k != kk) {
      zr[kk * 32] = er + oi;
      zi[kk * 32] = orr - ei;
    }
  }
  __syncthreads();
  z_stages<RMAX, true>(Z, Zr, Zi, data, npts, stride);
}

// Splits M into at most `depth` radices of Z_RADIX, none above rmax, in
// descending order; false when it cannot.
static bool z_factor(int M, int depth, int rmax, int *radix, int *nst) {
  if (M == 1) {
    *nst = 0;
    return true;
  }
  if (depth == 0) return false;
  for (int R : Z_RADIX)
    if (R <= rmax && M % R == 0 && z_factor(M / R, depth - 1, R, radix + 1, nst)) {
      radix[0] = R;
      ++*nst;
      return true;
    }
  return false;
}

// Threads, blocks an SM, the largest radix and the rows of 32 points a block
// may hold.  The blocks wait for memory in turn, so what counts is how many
// share an SM: four at 64 registers and 48 KB, which radices up to 10 allow.
// Lengths that one radix of up to 12 transforms (M <= 12) take it at three
// blocks an SM (nz = 24: 48 / 61 us for one stage, 71 / 73 for two); from M =
// 111 on shared memory allows three; from 145 on one block is taken, of 16 warps
// with radices up to 16 (nz = 512: 216 / 311 us, 257 / 322 with radices up to 8
// in 32 warps).
struct ZVariant {
  int threads, blocks, rmax, rows;
};
static const ZVariant &z_variant(int M) {
  static const ZVariant small = {256, 3, 12, 144}, mid = {256, 4, 10, 110}, large = {256, 3, 10, 144},
                        whole = {512, 1, 16, ZN_MAX / 2};
  return M <= 12 ? small : M <= mid.rows ? mid : M <= large.rows ? large : whole;
}

// The plan of a length (host data, made once per length).
static const ZPlan235 &z_plan(int nz) {
  static std::mutex mu;
  static std::map<int, ZPlan235> plans;
  std::lock_guard<std::mutex> lk(mu);
  auto it = plans.find(nz);
  if (it != plans.end()) return it->second;
  ZPlan235 &Z = plans[nz];
  Z.N = nz;
  Z.M = nz / 2;
  const long double pi = 3.14159265358979323846264338327950288L;
  for (int t = 0; t <= Z.M; t++) {
    Z.c[t] = (double)cosl(2 * pi * t / nz);
    Z.s[t] = (double)-sinl(2 * pi * t / nz);
    if (4 * t == nz) Z.c[t] = 0.0;  // exact at the quarter and half turns
    if (4 * t == nz) Z.s[t] = -1.0;
    if (2 * t == nz) Z.s[t] = 0.0;
  }
  const ZVariant &v = z_variant(Z.M);
  // the fewest stages, and of those the smallest largest radix
  Z.nst = 0;
  for (int depth = 1; depth <= ZST && Z.nst == 0; depth++)
    for (int i = (int)(sizeof(Z_RADIX) / sizeof(int)) - 1; i >= 0 && Z.nst == 0; i--)
      if (Z_RADIX[i] <= v.rmax && !z_factor(Z.M, depth, Z_RADIX[i], Z.radix, &Z.nst)) Z.nst = 0;
  // enough groups that the longest stage's sub-transforms fill eight warps
  const int per = Z.M / Z.radix[0];
  Z.PG = std::max(1, std::min((8 + per - 1) / per, v.rows / Z.M));
  return Z;
}

template <int NT, int MINB, int RMAX>
static int launch_rows(const ZPlan235 &Z, int rows, double *d, int npts, long long stride, int sign,
                       cudaStream_t st) {
  const int grid = (npts + 32 * Z.PG - 1) / (32 * Z.PG);
  const size_t smem = (size_t)Z.PG * Z.M * 512;
  if (sign == 1) {
    SX_CUDA(dynamic_smem(k_z_fwd_any<NT, MINB, RMAX>, smem, (size_t)rows * 512));
    k_z_fwd_any<NT, MINB, RMAX><<<grid, NT, smem, st>>>(Z, d, npts, stride, 1.0 / Z.N);
  } else {
    SX_CUDA(dynamic_smem(k_z_inv_any<NT, MINB, RMAX>, smem, (size_t)rows * 512));
    k_z_inv_any<NT, MINB, RMAX><<<grid, NT, smem, st>>>(Z, d, npts, stride);
  }
  SX_CUDA(cudaGetLastError());
  return SX_OK;
}

static int launch_any(double *d, int nz, int npts, long long stride, int sign, cudaStream_t st) {
  const ZPlan235 &Z = z_plan(nz);
  const ZVariant &v = z_variant(Z.M);
  if (v.blocks == 4) return launch_rows<256, 4, 10>(Z, v.rows, d, npts, stride, sign, st);
  if (v.rmax == 12) return launch_rows<256, 3, 12>(Z, v.rows, d, npts, stride, sign, st);
  if (v.blocks == 3) return launch_rows<256, 3, 10>(Z, v.rows, d, npts, stride, sign, st);
  return launch_rows<512, 1, 16>(Z, v.rows, d, npts, stride, sign, st);
}

// Where the radix-2 four-step kernels beat the mixed-radix ones.  At 256 they
// need one stage less in each direction and fit 3 blocks an SM like them.  At
// 128 both have two stages: the mixed-radix kernels' stages next to global
// memory skip a trip through shared memory, which pays once HBM bounds the
// transform; before that the four-step ones' straight loads come back sooner.
// Forward / inverse, us, four-step against mixed-radix:
//   128: 10,000 points 13.1/13.3 and 15.2/15.2, 41,472 25.6/27.5 and 27.8/28.1,
//        82,944 48.7/51.6 and 51.6/54.0, 200,000 112/124 and 106/119
//   256: 10,000 points 17.6/19.2 and 24.4/28.7, 82,944 85/98 and 114/142,
//        200,000 184/221 and 246/318
static bool four_step_faster(int nz, int npts) { return nz == 256 || (nz == 128 && npts < 100000); }

template <int N>
static void launch_reg(double *d, int npts, long long stride, int sign, cudaStream_t st) {
  const int grid = (npts + 127) / 128;
  if (sign == 1)
    k_z_fwd<N><<<grid, 128, 0, st>>>(d, npts, stride, 1.0 / N);
  else
    k_z_inv<N><<<grid, 128, 0, st>>>(d, npts, stride);
}

// spec[k][p] (k = 0 .. nz/2) -> data planes in semtex order, times 1/nz.
__global__ void k_z_pack(const double2 *__restrict__ spec, double *__restrict__ data, int nz, int npts,
                         long long stride, double scale) {
  const int nh = nz / 2;
  const long long n = (long long)(nh + 1) * npts;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
    const int k = (int)(i / npts), p = (int)(i - (long long)k * npts);
    const double2 v = spec[i];
    if (k == 0) {
      data[p] = v.x * scale;
    } else if (k == nh) {
      data[stride + p] = v.x * scale;
    } else {
      data[(2 * k) * stride + p] = v.x * scale;
      data[(2 * k + 1) * stride + p] = v.y * scale;
    }
  }
}

// data planes in semtex order -> spec[k][p] (Hermitian half spectrum, the
// imaginary parts of modes 0 and nz/2 zero).
__global__ void k_z_unpack(const double *__restrict__ data, double2 *__restrict__ spec, int nz, int npts,
                           long long stride) {
  const int nh = nz / 2;
  const long long n = (long long)(nh + 1) * npts;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
    const int k = (int)(i / npts), p = (int)(i - (long long)k * npts);
    double2 v;
    if (k == 0)
      v = make_double2(data[p], 0.0);
    else if (k == nh)
      v = make_double2(data[stride + p], 0.0);
    else
      v = make_double2(data[(2 * k) * stride + p], data[(2 * k + 1) * stride + p]);
    spec[i] = v;
  }
}

}  // namespace sx

using namespace sx;

extern "C" int sx_transform_z(double *d_data, int nz, int plane_stride, int npts, int sign, void *stream) {
  if (!d_data || nz < 1 || plane_stride <= 0 || npts < 0 || npts > plane_stride || (sign != 1 && sign != -1))
    return SX_ERR_ARG;
  if (nz == 1 || npts == 0) return SX_OK;  // a 2-D field: nothing to transform
  if (nz % 2 || !factors_235(nz)) {
    set_error("transform length %d: needs an even length with prime factors 2, 3, 5 (fourier.c:135-143)", nz);
    return SX_ERR_ARG;
  }
  if (nz <= 64 && (nz & (nz - 1)) == 0) {
    // one pass in registers, enqueued without waiting (no workspace)
    cudaStream_t st = (cudaStream_t)stream;
    switch (nz) {
      case 2: launch_reg<2>(d_data, npts, plane_stride, sign, st); break;
      case 4: launch_reg<4>(d_data, npts, plane_stride, sign, st); break;
      case 8: launch_reg<8>(d_data, npts, plane_stride, sign, st); break;
      case 16: launch_reg<16>(d_data, npts, plane_stride, sign, st); break;
      case 32: launch_reg<32>(d_data, npts, plane_stride, sign, st); break;
      default: launch_reg<64>(d_data, npts, plane_stride, sign, st); break;
    }
    SX_CUDA(cudaGetLastError());
    return SX_OK;
  }
  if (nz <= ZN_MAX) {
    // one pass through shared memory, enqueued without waiting
    if (four_step_faster(nz, npts)) {
        if (nz == 256)
        SX_TRY(launch_smem<256>(d_data, npts, plane_stride, sign, (cudaStream_t)stream));
      else
        SX_TRY(launch_smem<128>(d_data, npts, plane_stride, sign, (cudaStream_t)stream));
      SX_CUDA(cudaGetLastError());
      return SX_OK;
    }
    return launch_any(d_data, nz, npts, plane_stride, sign, (cudaStream_t)stream);
  }
  const CufftApi &api = cufft_api();
  if (!api.ok) {
    set_error("libcufft.so.11 could not be loaded");
    return SX_ERR_UNSUPPORTED;
  }
  cudaStream_t st = (cudaStream_t)stream;
  int dev = 0;
  SX_CUDA(cudaGetDevice(&dev));
  ZPlan *zp = nullptr;
  {
    std::lock_guard<std::mutex> lk(g_mu);
    auto &slot = g_plans[std::make_tuple(dev, nz, npts, plane_stride, sign)];
    if (!slot) {
      std::unique_ptr<ZPlan> np_(new ZPlan());
      SX_TRY(np_->spec.alloc((size_t)(nz / 2 + 1) * npts));
      int n[1] = {nz};
      int rembed[1] = {nz}, cembed[1] = {nz / 2 + 1};
      // real side: element stride = plane stride, transforms 1 apart;
      // complex side: [k][p], element stride npts, transforms 1 apart
      cufftResult r = sign == 1 ? api.planMany(&np_->plan, 1, n, rembed, plane_stride, 1, cembed, npts, 1,
                                               CUFFT_D2Z, npts)
                                : api.planMany(&np_->plan, 1, n, cembed, npts, 1, rembed, plane_stride, 1,
                                               CUFFT_Z2D, npts);
      if (r != CUFFT_SUCCESS) {
        set_error("cufftPlanMany(nz = %d, npts = %d): error %d", nz, npts, (int)r);
        return SX_ERR_CUDA;
      }
      slot = std::move(np_);
    }
    zp = slot.get();
  }
  // one transform at a time per plan (its workspace is shared)
  std::lock_guard<std::mutex> lk(g_mu);
  if (api.setStream(zp->plan, st) != CUFFT_SUCCESS) {
    set_error("cufftSetStream failed");
    return SX_ERR_CUDA;
  }
  const long long n = (long long)(nz / 2 + 1) * npts;
  const int grid = (int)std::min<long long>((n + 255) / 256, 8 * 148);
  if (sign == 1) {
    if (api.execD2Z(zp->plan, d_data, reinterpret_cast<cufftDoubleComplex *>(zp->spec.p)) != CUFFT_SUCCESS) {
      set_error("cufftExecD2Z failed");
      return SX_ERR_CUDA;
    }
    k_z_pack<<<grid, 256, 0, st>>>(zp->spec.p, d_data, nz, npts, plane_stride, 1.0 / nz);
  } else {
    k_z_unpack<<<grid, 256, 0, st>>>(d_data, zp->spec.p, nz, npts, plane_stride);
    if (api.execZ2D(zp->plan, reinterpret_cast<cufftDoubleComplex *>(zp->spec.p), d_data) != CUFFT_SUCCESS) {
      set_error("cufftExecZ2D failed");
      return SX_ERR_CUDA;
    }
  }
  SX_CUDA(cudaGetLastError());
  // the workspace is reused by the next call on this plan: finish here
  SX_CUDA(cudaStreamSynchronize(st));
  return SX_OK;
}

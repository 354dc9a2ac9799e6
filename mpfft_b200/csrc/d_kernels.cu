// FP64 conjugate-pair split-radix 2/4 DIT FFT kernels (sm_100a).
//
// Bit-identical to the reference's double transform d_sr24_cp_fft
// (lab/serial/double/serial_d_fft6.c:93-429): the same n=8 and n=16 base
// cases, the same 4m2a butterfly for every k (twiddle (1,0) at k=0
// included), every IEEE operation with the same operands in the same
// association.  This file is compiled with --fmad=false so no multiply-add is
// contracted into an FMA (the reference's x86-64 build has no FMA either).
//
// Schedule: the reference's recursion tree, cut at T <= 4096 points.  Chunks
// of T output positions run in shared memory (d_core.cuh): base cases of 16
// and 8 points straight from global memory, then passes of up to three levels
// whose points stay in registers, the last one written out.  Levels above T
// run three (or two) per launch in global memory, again in registers.  For
// N <= 4096 a transform is one launch that reads its input once and writes its
// output once.
//
// Layout: word (c, b, p) at base[(c*B + b)*N + p] -- each signal contiguous.
#include <algorithm>
#include <cstdint>

#include "d_core.cuh"
#include "mpfft_internal.h"

namespace mpfft {

template <int LGT, bool SINGLE>
__global__ void __launch_bounds__(256, 2) d_sub_kernel(const __grid_constant__ DSubTab S, DSubArgs A, int groups) {
  extern __shared__ __align__(16) double2 d_smem[];
  const int g = A.G;
  if (SINGLE) {
    A.b0 = blockIdx.x * g;
    A.G = min(g, A.B - A.b0);
  } else {
    A.b0 = blockIdx.x / groups;
    A.c0 = (blockIdx.x % groups) * g;
    A.G = min(g, S.nchunks - A.c0);
  }
  d_sub_transform<LGT, SINGLE>(S, A, d_smem);
}

__global__ void __launch_bounds__(256) d_tiny_kernel(const __grid_constant__ DSubTab S, DSubArgs A) {
  extern __shared__ __align__(16) double2 d_smem[];
  A.b0 = blockIdx.x * A.G;
  A.G = min(A.G, A.B - A.b0);
  d_tiny(S, A, d_smem);
}

// R levels above the sub-transforms: one thread per column (d_upper_column),
// consecutive threads consecutive k of one chunk of one signal.  Memory-bound:
// three levels cross memory once instead of three times (one 2^20-point signal
// 100 -> 39 us, four launches instead of nine).
template <int R>
__global__ void __launch_bounds__(256, 2) d_upper_kernel(double *__restrict__ y, int N, int B, int lgu, int lgnch,
                                                         const double2 *__restrict__ tw, double scale, int swap_out) {
  const long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const long long r = e >> lgu;
  const long long b = r >> lgnch;
  if (b >= B) return;
  d_upper_column<R>(y, N, B, lgu, (int)b, (int)(r & ((1 << lgnch) - 1)), (int)(e & ((1 << lgu) - 1)), tw, scale,
                    swap_out != 0);
}

__global__ void __launch_bounds__(256) d_level_tw_kernel(int N, double2 *tw) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;  // entry of a level below N
  if (i >= N / 4 - 8) return;
  const int q = 1 << (31 - __clz(i + 8));  // n/4 of its level: entries q-8 .. 2q-9
  const int k = i + 8 - q;
  tw[i] = tw[sr_level_tw(N) + (size_t)k * (N / (4 * q))];
}

cudaError_t d_build_level_tw(int N, double2 *tw, cudaStream_t s) {
  if (N > 32) d_level_tw_kernel<<<(N / 4 - 8 + 255) / 256, 256, 0, s>>>(N, tw);
  return cudaGetLastError();
}

// Split step of the FP64 real transforms (n = 2M real points; layouts [c][b][k]).
// Forward: Z = FFT_M(x_2m + i x_2m+1) (M points) -> X_0..X_M (M+1 points):
//   S = Z_k + conj Z_(M-k), D = Z_k - conj Z_(M-k), T = w^k D (w = exp(-2 pi i/n)),
//   X_k = (S_r + T_i, S_i - T_r) / 2,  X_(M-k) = (S_r - T_i, -(S_i + T_r)) / 2.
// Inverse: X (M+1 points) -> W = the planes-exchanged 2Z, with
//   S' = X_k + conj X_(M-k), D' = X_k - conj X_(M-k), T' = w^-k D',
//   2Z_k = (S'_r - T'_i, S'_i + T'_r), 2Z_(M-k) = (S'_r + T'_i, T'_r - S'_i),
// so that the forward transform of W is n * (x_2m+1 + i x_2m) (the swap
// identity); the imaginary parts of X_0 and X_M are ignored.  wc, ws: cos and
// sin of 2 pi k/n for k < M/2; scale multiplies the forward outputs.
__global__ void __launch_bounds__(256) d_r2c_post(const double *__restrict__ z, double *__restrict__ x, int M, int B,
                                                   const double *__restrict__ wc, const double *__restrict__ ws,
                                                   double scale) {
  const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= (long long)(M / 2 + 1) * B) return;
  const int k = (int)(t % (M / 2 + 1));
  const int b = (int)(t / (M / 2 + 1));
  const double *zr = z + (size_t)b * M, *zi = z + ((size_t)B + b) * M;
  double *xr = x + (size_t)b * (M + 1), *xi = x + ((size_t)B + b) * (M + 1);
  const double h = 0.5 * scale;
  if (k == 0) {
    xr[0] = (zr[0] + zi[0]) * scale;
    xi[0] = 0.0;
    xr[M] = (zr[0] - zi[0]) * scale;
    xi[M] = 0.0;
    return;
  }
  const double ar = zr[k], ai = zi[k], br = zr[M - k], bi = zi[M - k];
  const double sr = ar + br, si = ai - bi, dr = ar - br, di = ai + bi;
  const double c = 2 * k == M ? 0.0 : wc[k], s = 2 * k == M ? 1.0 : ws[k];
  const double tr = c * dr + s * di, ti = c * di - s * dr;
  xr[k] = (sr + ti) * h;
  xi[k] = (si - tr) * h;
  if (2 * k != M) {
    xr[M - k] = (sr - ti) * h;
    xi[M - k] = -(si + tr) * h;
  }
}

__global__ void __launch_bounds__(256) d_c2r_pre(const double *__restrict__ x, double *__restrict__ w, int M, int B,
                                                  const double *__restrict__ wc, const double *__restrict__ ws) {
  const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= (long long)(M / 2 + 1) * B) return;
  const int k = (int)(t % (M / 2 + 1));
  const int b = (int)(t / (M / 2 + 1));
  const double *xr = x + (size_t)b * (M + 1), *xi = x + ((size_t)B + b) * (M + 1);
  // W = (2Z_i, 2Z_r): real plane holds the imaginary parts
  double *wr = w + (size_t)b * M, *wi = w + ((size_t)B + b) * M;
  if (k == 0) {
    wi[0] = xr[0] + xr[M];
    wr[0] = xr[0] - xr[M];
    return;
  }
  const double ar = xr[k], ai = xi[k], br = xr[M - k], bi = xi[M - k];
  const double sr = ar + br, si = ai - bi, dr = ar - br, di = ai + bi;
  const double c = 2 * k == M ? 0.0 : wc[k], s = 2 * k == M ? 1.0 : ws[k];
  const double tr = c * dr - s * di, ti = c * di + s * dr;
  wi[k] = sr - ti;
  wr[k] = si + tr;
  if (2 * k != M) {
    wi[M - k] = sr + ti;
    wr[M - k] = tr - si;
  }
}

cudaError_t d_real_split(bool forward, const double *in, double *out, int M, int B, const double *wc,
                         const double *ws, double scale, cudaStream_t s) {
  const long long total = (long long)(M / 2 + 1) * B;
  const int blocks = (int)((total + 255) / 256);
  if (forward) d_r2c_post<<<blocks, 256, 0, s>>>(in, out, M, B, wc, ws, scale);
  else d_c2r_pre<<<blocks, 256, 0, s>>>(in, out, M, B, wc, ws);
  return cudaGetLastError();
}

template <int LGT, bool SINGLE>
static cudaError_t d_sub_launch(const DSubTab &S, DSubArgs A, cudaStream_t s) {
  constexpr int T = 1 << LGT;
  // Chunks per CTA: as many as fit, but no more than leave two CTAs for every
  // SM (a small batch spread over more CTAs finishes earlier).
  const long long inst = SINGLE ? A.B : (long long)S.nchunks * A.B;
  int g = kDSubMax / T;
  while (g > 1 && inst / g < 2 * 148) g /= 2;
  A.G = g;
  const size_t smem = (size_t)g * T * sizeof(double2);
  if (smem > 48 * 1024) {
    const cudaError_t e = cudaFuncSetAttribute(d_sub_kernel<LGT, SINGLE>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                               kDSubMax * (int)sizeof(double2));
    if (e != cudaSuccess) return e;
  }
  const int threads = std::min(256, std::max(32, g * T / 16));
  const int groups = SINGLE ? 1 : (S.nchunks + g - 1) / g;
  const long long ctas = SINGLE ? ((long long)A.B + g - 1) / g : (long long)groups * A.B;
  d_sub_kernel<LGT, SINGLE><<<(unsigned)ctas, threads, smem, s>>>(S, A, groups);
  return cudaGetLastError();
}

cudaError_t d_run_transform(const DDeviceTables &T, const double *in, double *out, int B, double scale,
                            cudaStream_t s, bool swap_in, bool swap_out) {
  const DSubTab &S = T.d;
  const int nl = S.N > 16 ? 31 - __builtin_clz((unsigned)S.nchunks) : 0;  // levels above the sub-transforms
  DSubArgs A{in, out, B, 0, 0, 0, scale, nl == 0, swap_in, swap_out && nl == 0};
  cudaError_t e = cudaSuccess;
  if (S.N <= 16) {
    A.G = 2048 / S.N;
    d_tiny_kernel<<<(unsigned)((B + A.G - 1) / A.G), 256, 2048 * sizeof(double2), s>>>(S, A);
    return cudaGetLastError();
  }
#define MPFFT_D_CASE(LL, SINGLE)           \
  case LL:                                 \
    e = d_sub_launch<LL, SINGLE>(S, A, s); \
    break;
  if (S.nchunks == 1) {
    switch (S.lgT) {
      MPFFT_D_CASE(5, true) MPFFT_D_CASE(6, true) MPFFT_D_CASE(7, true) MPFFT_D_CASE(8, true)
      MPFFT_D_CASE(9, true) MPFFT_D_CASE(10, true) MPFFT_D_CASE(11, true) MPFFT_D_CASE(12, true)
      default: return cudaErrorInvalidValue;
    }
  } else {
    switch (S.lgT) {
      MPFFT_D_CASE(10, false) MPFFT_D_CASE(11, false) MPFFT_D_CASE(12, false)
      default: return cudaErrorInvalidValue;
    }
  }
#undef MPFFT_D_CASE
  if (e != cudaSuccess) return e;
  // The levels above: whole batches per launch.  (Groups of signals that fit
  // L2 between the launches were slower at every size: 2^24 points, N = 8192
  // 222 us, in groups of 2^21 points 282, 2^22 249, 2^23 240.)
  const int lgN = 31 - __builtin_clz((unsigned)S.N), step = d_upper_levels(nl);
  for (int done = 0; done < nl;) {
    const int r = std::min(step, nl - done), lgu = S.lgT + done - 1, lgnch = lgN - (lgu + r + 1);
    const bool last = done + r == nl;
    const long long cols = (long long)B * (S.N >> (r + 1));
    const unsigned blocks = (unsigned)((cols + 255) / 256);
    const double sc = last ? scale : 1.0;
    const int sw = last && swap_out;
    if (r == 3) d_upper_kernel<3><<<blocks, 256, 0, s>>>(out, S.N, B, lgu, lgnch, S.tw, sc, sw);
    else if (r == 2) d_upper_kernel<2><<<blocks, 256, 0, s>>>(out, S.N, B, lgu, lgnch, S.tw, sc, sw);
    else d_upper_kernel<1><<<blocks, 256, 0, s>>>(out, S.N, B, lgu, lgnch, S.tw, sc, sw);
    done += r;
  }
  return cudaGetLastError();
}

}  // namespace mpfft

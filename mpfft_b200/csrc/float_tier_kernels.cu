// Launchers of the compensated floating-point tiers (double-double,
// quad-double, float-float): the per-launch kernels over float_tiers.cuh.
#include <algorithm>
#include <cstdint>

#include "float_tiers.cuh"
#include "mpfft_internal.h"

namespace mpfft {

// Two CTAs of 256 threads per SM, 128 registers.  Measured (4096 points x 512,
// us): double-double with two levels per pass 139, one 145, two at 85 registers
// 160; quad-double with one level per pass 582, with 192 threads 631, three CTAs
// of 192 (spilling) 686, two levels per pass (8 points, 255 registers) 896.  One
// CTA of 512 threads with a chunk twice as large, which saves a pass above:
// double-double 152, quad-double 617.  FEW (fewer chunks than SMs, one each of at
// most 2^kLgFew points): a CTA has its SM to itself and takes all the registers
// (quad-double, one signal, us, two CTAs' registers / all: 16 points 11.2 / 8.8,
// 128 points 21.9 / 16.4, 1024 points 42.4 / 37.7; double-double with base cases of
// eight / four positions: 16 points 4.6 / 4.3, 128 points 7.5 / 7.0, but 2048 points
// 22.6 / 24.2).
template <class NT, bool SINGLE, bool FEW>
__global__ void __launch_bounds__(256, FEW ? 1 : 2)
    tier_sub_kernel(const __grid_constant__ TierTab S, TierArgs<NT> A, int groups) {
  extern __shared__ __align__(16) double2 tier_smem[];
  const int g = A.G;
  if (SINGLE) {
    A.b0 = blockIdx.x * g;
    A.G = min(g, A.B - A.b0);
  } else {
    A.b0 = blockIdx.x / groups;
    A.c0 = (blockIdx.x % groups) * g;
    A.G = min(g, S.nchunks - A.c0);
  }
  tier_sub_transform<NT, SINGLE, FEW>(S, A, tier_smem);
}

template <class NT>
__global__ void __launch_bounds__(256) tier_tiny_kernel(const __grid_constant__ TierTab S, TierArgs<NT> A) {
  A.b0 = blockIdx.x * A.G;
  A.G = min(A.G, A.B - A.b0);
  tier_tiny<NT>(S, A);
}

template <class NT, int R>
__global__ void __launch_bounds__(256) tier_upper_kernel(typename NT::W *__restrict__ y,
                                                         const __grid_constant__ TierTab S, int B, int lgu, int lgnch,
                                                         double scale, int swap_out) {
  const long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const long long r = e >> lgu;
  const long long b = r >> lgnch;
  if (b >= B) return;
  tier_upper_column<NT, R>(y, S, B, lgu, (int)b, (int)(r & ((1 << lgnch) - 1)), (int)(e & ((1 << lgu) - 1)), scale,
                           swap_out != 0);
}

__global__ void __launch_bounds__(256) tier_tw_kernel(int words, int N, double2 *tw) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;  // entry of a level below N, in each plane
  if (i >= N / 4 - 2) return;
  const int q = 1 << (31 - __clz(i + 2));  // n/4 of its level: entries q-2 .. 2q-3
  const size_t kn = (size_t)(i + 2 - q) * (N / (4 * q)), len = (size_t)N / 2 - 2;
  for (int h = 0; h < words; ++h) tw[h * len + i] = tw[h * len + tier_level_tw(N) + kn];
}

cudaError_t tier_build_tw(int words, int N, double2 *tw, cudaStream_t s) {
  if (N > 8) tier_tw_kernel<<<(N / 4 - 2 + 255) / 256, 256, 0, s>>>(words, N, tw);
  return cudaGetLastError();
}

template <class NT, bool SINGLE, bool FEW>
static cudaError_t tier_sub_launch(const TierTab &S, TierArgs<NT> A, cudaStream_t s) {
  const size_t smem = ((size_t)A.G << S.lgT) * NT::kUnits * sizeof(double2) + kOrderBytes;
  if (smem > 48 * 1024) {
    const cudaError_t e =
        cudaFuncSetAttribute(tier_sub_kernel<NT, SINGLE, FEW>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (NT::kUnits << NT::kLgMax) * (int)sizeof(double2) + (int)kOrderBytes);
    if (e != cudaSuccess) return e;
  }
  const int threads = std::min(256, std::max(32, (A.G << S.lgT) >> (A.per + 1)));
  const int groups = SINGLE ? 1 : (S.nchunks + A.G - 1) / A.G;
  const long long ctas = SINGLE ? ((long long)A.B + A.G - 1) / A.G : (long long)groups * A.B;
  tier_sub_kernel<NT, SINGLE, FEW><<<(unsigned)ctas, threads, smem, s>>>(S, A, groups);
  return cudaGetLastError();
}

template <class NT, bool SINGLE>
static cudaError_t tier_sub_launch(const TierTab &S, TierArgs<NT> A, cudaStream_t s) {
  // chunks per CTA: as many as fit, but no more than leave two CTAs for every SM
  const long long inst = SINGLE ? A.B : (long long)S.nchunks * A.B;
  A.G = 1 << (NT::kLgMax - S.lgT);
  while (A.G > 1 && inst / A.G < 2 * 148) A.G /= 2;
  // few CTAs: one level per pass, so that each pass has the most threads (one
  // 1024-point float-float signal: 14.4 us with three levels per pass)
  A.per = inst / A.G < 148 ? 1 : NT::kLevels;
  if (inst < 148 && S.lgT <= NT::kLgFew) return tier_sub_launch<NT, SINGLE, true>(S, A, s);
  return tier_sub_launch<NT, SINGLE, false>(S, A, s);
}

template <class NT>
static cudaError_t tier_run(const DDeviceTables &T, const void *in, void *out, int B, double scale, cudaStream_t s,
                            bool swap_in, bool swap_out) {
  using W = typename NT::W;
  const TierTab &S = T.t;
  const int nl = 31 - __builtin_clz((unsigned)S.nchunks);  // levels above the sub-transforms
  TierArgs<NT> A{static_cast<const W *>(in), static_cast<W *>(out), B, 0, 0, 0, NT::kLevels, scale, nl == 0, swap_in,
                 swap_out && nl == 0};
  if (S.N < 8) {
    A.G = 256;
    tier_tiny_kernel<NT><<<(unsigned)((B + 255) / 256), 256, 0, s>>>(S, A);
    return cudaGetLastError();
  }
  const cudaError_t e = nl == 0 ? tier_sub_launch<NT, true>(S, A, s) : tier_sub_launch<NT, false>(S, A, s);
  if (e != cudaSuccess) return e;
  const int lgN = 31 - __builtin_clz((unsigned)S.N), step = tier_upper_levels(nl, NT::kLevels);
  for (int done = 0; done < nl;) {
    const int r = std::min(step, nl - done), lgu = S.lgT + done - 1, lgnch = lgN - (lgu + r + 1);
    const bool last = done + r == nl;
    const unsigned blocks = (unsigned)(((long long)B * (S.N >> (r + 1)) + 255) / 256);
    const double sc = last ? scale : 1.0;
    const int sw = last && swap_out;
    constexpr int R2 = NT::kLevels >= 2 ? 2 : 1, R3 = NT::kLevels >= 3 ? 3 : 1;
    if (r == 3) tier_upper_kernel<NT, R3><<<blocks, 256, 0, s>>>(A.out, S, B, lgu, lgnch, sc, sw);
    else if (r == 2) tier_upper_kernel<NT, R2><<<blocks, 256, 0, s>>>(A.out, S, B, lgu, lgnch, sc, sw);
    else tier_upper_kernel<NT, 1><<<blocks, 256, 0, s>>>(A.out, S, B, lgu, lgnch, sc, sw);
    done += r;
  }
  return cudaGetLastError();
}

int tier_words(int tier) { return tier == kTierQD ? 4 : 2; }
size_t tier_word_bytes(int tier) { return tier == kTierFF ? 4 : 8; }
int tier_sub_max(int tier) {
  return 1 << (tier == kTierQD ? QDT::kLgMax : tier == kTierFF ? FFT_::kLgMax : DDT::kLgMax);
}
int tier_tw_words(int tier) {
  return tier == kTierQD ? QDT::kTwWords : tier == kTierFF ? FFT_::kTwWords : DDT::kTwWords;
}
int tier_leaf_lg(int tier, bool few) {
  if (few) return tier == kTierQD ? QDT::kLeafLgFew : tier == kTierFF ? FFT_::kLeafLgFew : DDT::kLeafLgFew;
  return tier == kTierQD ? QDT::kLeafLg : tier == kTierFF ? FFT_::kLeafLg : DDT::kLeafLg;
}
int tier_pass_levels(int tier) {
  return tier == kTierQD ? QDT::kLevels : tier == kTierFF ? FFT_::kLevels : DDT::kLevels;
}

cudaError_t tier_run_transform(int tier, const DDeviceTables &T, const void *in, void *out, int B, double scale,
                               cudaStream_t s, bool swap_in, bool swap_out) {
  switch (tier) {
    case kTierDD:
      return tier_run<DDT>(T, in, out, B, scale, s, swap_in, swap_out);
    case kTierQD:
      return tier_run<QDT>(T, in, out, B, scale, s, swap_in, swap_out);
    case kTierFF:
      return tier_run<FFT_>(T, in, out, B, scale, s, swap_in, swap_out);
    default:
      return cudaErrorInvalidValue;
  }
}

}  // namespace mpfft

// Persistent work-queue kernels for uneven batches: signals of different
// lengths and precisions in one graph launch.
//
// The reference transforms one signal per call and parallelises inside one
// butterfly loop with an OpenMP team per recursion node
// (lab/parallel/mp/parallel_mp_fft2.c:259-326).  Here a batch of signals is
// split into queues by form (fixed-point limbs of each limb count, FP64, and
// the compensated tiers); each queue is one persistent kernel whose CTAs pop
// whole signals from a device counter (atomicAdd) and transform them end to
// end, the largest first.  A CTA runs the same device functions as the
// per-launch kernels -- leaves and L-butterflies of mp_bfly.cuh, the FP64
// sub-transforms of d_core.cuh, the tier sub-transforms of float_tiers.cuh --
// level after level with a CTA barrier between levels, so every output is
// bit-identical to a single call of the same signal.  No CTA waits for
// another: the only shared state is the queue counter.
//
// Compiled with --fmad=false (FP64 bit-identity to the reference); the
// compensated tiers call fma() explicitly and the limb forms are integer
// arithmetic, so neither depends on contraction.
#include <algorithm>
#include <cstdint>

#include "d_core.cuh"
#include "float_tiers.cuh"
#include "mp_bfly.cuh"
#include "mpfft_internal.h"

namespace mpfft {

// the next item of this CTA's queue (all threads see the same value)
__device__ __forceinline__ int queue_next(int *head, int *slot) {
  __syncthreads();  // the previous item is finished before the slot changes
  if (threadIdx.x == 0) *slot = atomicAdd(head, 1);
  __syncthreads();
  return *slot;
}

// ---------------------------------------------------------------------------
// limb forms: one signal = the leaf stage and every level, in global memory
// ---------------------------------------------------------------------------
template <int L>
__global__ void __launch_bounds__(256) mp_queue_kernel(const QueueItem *__restrict__ items, int nitems, int *head) {
  extern __shared__ uint32_t Ps[];  // L x blockDim.x words: each thread's first product of a side
  __shared__ int slot;
  for (int i; (i = queue_next(head, &slot)) < nitems;) {
    const QueueItem it = items[i];
    const QueueTables &Q = *it.tab;
    const TreeTables &T = Q.tree;
    const uint32_t *in = static_cast<const uint32_t *>(it.in);
    uint32_t *out = static_cast<uint32_t *>(it.out);
    const int N = Q.N;
    for (int e = threadIdx.x; e < T.nleaves; e += blockDim.x) mp_leaf_one<L>(in, out, N, 1, 0, T.leaves[e]);
    for (int lv = 0; lv < T.nlevels; ++lv) {
      __syncthreads();  // the previous stage's outputs are visible to the whole CTA
      const int n = T.level_n[lv], q = n >> 2;
      const int total = T.level_count[lv] * q;
      const int *nodes = T.node_off + T.level_start[lv];
      for (int t = threadIdx.x; t < total; t += blockDim.x)
        mp_bfly_one<L>(out, N, 1, 0, n, nodes[t / q], t % q, Q.twp, Q.dneg, 1, Ps + threadIdx.x, blockDim.x);
    }
  }
}

// ---------------------------------------------------------------------------
// FP64: the chunks of T points one after another in shared memory, then the
// levels above them in global memory
// ---------------------------------------------------------------------------
// one signal of N points: every chunk of T points, then the levels above
template <int LGT>
__device__ __forceinline__ void d_queue_signal(const DSubTab &S, DSubArgs A, double2 *sm) {
  if (S.nchunks == 1) {
    d_sub_transform<LGT, true>(S, A, sm);
    return;
  }
  if constexpr (LGT >= 10) {
    for (A.c0 = 0; A.c0 < S.nchunks; ++A.c0) {
      __syncthreads();  // shared memory of the previous chunk is free
      d_sub_transform<LGT, false>(S, A, sm);
    }
  }
}

template <int R>
__device__ __forceinline__ void d_queue_upper(const DSubTab &S, double *out, int lgu, int cols, double scale) {
  for (int t = threadIdx.x; t < cols; t += blockDim.x)
    d_upper_column<R>(out, S.N, 1, lgu, 0, t >> lgu, t & ((1 << lgu) - 1), S.tw, scale, false);
}

__global__ void __launch_bounds__(256, 2) d_queue_kernel(const QueueItem *__restrict__ items, int nitems, int *head,
                                                         double scale) {
  extern __shared__ __align__(16) double2 dq_smem[];
  __shared__ int slot;
  for (int i; (i = queue_next(head, &slot)) < nitems;) {
    const QueueItem it = items[i];
    const DSubTab S = it.tab->ft.d;
    double *out = static_cast<double *>(it.out);
    const int nl = S.N > 16 ? 31 - __clz(S.nchunks) : 0;
    const DSubArgs A{static_cast<const double *>(it.in), out, 1, 0, 0, 1, scale, nl == 0, false, false};
    if (S.N <= 16) {
      d_tiny(S, A, dq_smem);
      continue;
    }
    switch (S.lgT) {
      case 5: d_queue_signal<5>(S, A, dq_smem); break;
      case 6: d_queue_signal<6>(S, A, dq_smem); break;
      case 7: d_queue_signal<7>(S, A, dq_smem); break;
      case 8: d_queue_signal<8>(S, A, dq_smem); break;
      case 9: d_queue_signal<9>(S, A, dq_smem); break;
      case 10: d_queue_signal<10>(S, A, dq_smem); break;
      case 11: d_queue_signal<11>(S, A, dq_smem); break;
      case 12: d_queue_signal<12>(S, A, dq_smem); break;
      default: break;
    }
    const int step = d_upper_levels(nl);
    for (int done = 0; done < nl;) {
      __syncthreads();
      const int r = min(step, nl - done), lgu = S.lgT + done - 1, cols = S.N >> (r + 1);
      const double sc = done + r == nl ? scale : 1.0;
      if (r == 3) d_queue_upper<3>(S, out, lgu, cols, sc);
      else if (r == 2) d_queue_upper<2>(S, out, lgu, cols, sc);
      else d_queue_upper<1>(S, out, lgu, cols, sc);
      done += r;
    }
  }
}

// ---------------------------------------------------------------------------
// compensated tiers: the same pattern
// ---------------------------------------------------------------------------
template <class NT, int R>
__device__ __forceinline__ void tier_queue_upper(const TierTab &S, typename NT::W *out, int lgu, int cols,
                                                 double scale) {
  for (int t = threadIdx.x; t < cols; t += blockDim.x)
    tier_upper_column<NT, R>(out, S, 1, lgu, 0, t >> lgu, t & ((1 << lgu) - 1), scale, false);
}

// SHORT: no signal is longer than one chunk of 2^kLgFew points.  A CTA takes one
// signal at a time, so short ones leave most of 256 threads idle: they run in
// small CTAs (tier_queue_threads in host.cpp), several of which share an SM, one
// level per pass, in a kernel without the code of longer signals.  Measured (2000
// signals, us; one kernel for all lengths, 256 threads, one CTA per SM / this):
// float-float 64 points 84 / 16, 512 points 123 / 27; double-double 102 / 29, 135
// / 68; quad-double 221 / 78, 368 / 232.  The longer ones keep one CTA of all the
// registers per SM: with two, of 128 registers, uniform batches are faster (double-double
// 4096 points x 300 123 / 105 us) but the longest signals later (quad-double 8192
// points alone 386 / 452 us; 2000 signals of 16 .. 8192 points in four forms 508 /
// 806 us), and those end a mixed launch.
template <class NT, bool SHORT>
__global__ void __launch_bounds__(256, 1) tier_queue_kernel(const QueueItem *__restrict__ items, int nitems, int *head,
                                                            double scale) {
  extern __shared__ __align__(16) double2 tq_smem[];
  __shared__ int slot;
  for (int i; (i = queue_next(head, &slot)) < nitems;) {
    const QueueItem it = items[i];
    const TierTab S = it.tab->ft.t;
    auto *out = static_cast<typename NT::W *>(it.out);
    const int nl = SHORT ? 0 : 31 - __clz(S.nchunks);
    TierArgs<NT> A{static_cast<const typename NT::W *>(it.in), out, 1, 0, 0, 1, 1, scale, nl == 0, false, false};
    if (S.N < 8) {
      tier_tiny<NT>(S, A);
      continue;
    }
    if constexpr (SHORT) {
      tier_sub_transform<NT, true, true>(S, A, tq_smem);
    } else {
      // as many levels per pass as leave every thread a column
      A.per = min(NT::kLevels, max(1, S.lgT - 1 - (31 - __clz(blockDim.x))));
      if (nl == 0) {
        tier_sub_transform<NT, true, false>(S, A, tq_smem);
        continue;
      }
      for (A.c0 = 0; A.c0 < S.nchunks; ++A.c0) {
        __syncthreads();  // shared memory of the previous chunk is free
        tier_sub_transform<NT, false, false>(S, A, tq_smem);
      }
      const int step = tier_upper_levels(nl, NT::kLevels);
      for (int done = 0; done < nl;) {
        __syncthreads();
        const int r = min(step, nl - done), lgu = S.lgT + done - 1, cols = S.N >> (r + 1);
        const double sc = done + r == nl ? scale : 1.0;
        constexpr int R2 = NT::kLevels >= 2 ? 2 : 1, R3 = NT::kLevels >= 3 ? 3 : 1;
        if (r == 3) tier_queue_upper<NT, R3>(S, out, lgu, cols, sc);
        else if (r == 2) tier_queue_upper<NT, R2>(S, out, lgu, cols, sc);
        else tier_queue_upper<NT, 1>(S, out, lgu, cols, sc);
        done += r;
      }
    }
  }
}

// ---------------------------------------------------------------------------
// host side
// ---------------------------------------------------------------------------
constexpr size_t kQueueSmemBytes = 64 * 1024 + kOrderBytes;  // most: FP64 (4096 points) and every tier (64 KB planes)

template <int L>
static const void *mp_queue_fn() {
  return (const void *)mp_queue_kernel<L>;
}

template <class NT>
static const void *tier_queue_fn(const QueueShape &Q) {
  if (Q.points == Q.chunk && Q.chunk <= 1 << NT::kLgFew) return (const void *)tier_queue_kernel<NT, true>;
  return (const void *)tier_queue_kernel<NT, false>;
}

static const void *queue_fn(const QueueShape &Q) {
  switch (Q.family) {
    case kQueueDouble:
      return (const void *)d_queue_kernel;
    case kQueueTierDD:
      return tier_queue_fn<DDT>(Q);
    case kQueueTierQD:
      return tier_queue_fn<QDT>(Q);
    case kQueueTierFF:
      return tier_queue_fn<FFT_>(Q);
    default:
      break;
  }
#define MPFFT_Q_CASE(LL) \
  case LL:               \
    return mp_queue_fn<LL>();
  switch (Q.L) {
    MPFFT_Q_CASE(2) MPFFT_Q_CASE(3) MPFFT_Q_CASE(4) MPFFT_Q_CASE(5) MPFFT_Q_CASE(6) MPFFT_Q_CASE(7)
    MPFFT_Q_CASE(8) MPFFT_Q_CASE(9) MPFFT_Q_CASE(10) MPFFT_Q_CASE(11) MPFFT_Q_CASE(12) MPFFT_Q_CASE(13)
    MPFFT_Q_CASE(14) MPFFT_Q_CASE(15) MPFFT_Q_CASE(16) MPFFT_Q_CASE(17) MPFFT_Q_CASE(18) MPFFT_Q_CASE(19)
    MPFFT_Q_CASE(20) MPFFT_Q_CASE(21) MPFFT_Q_CASE(22) MPFFT_Q_CASE(23) MPFFT_Q_CASE(24) MPFFT_Q_CASE(25)
    MPFFT_Q_CASE(26) MPFFT_Q_CASE(27) MPFFT_Q_CASE(28) MPFFT_Q_CASE(29) MPFFT_Q_CASE(30) MPFFT_Q_CASE(31)
    MPFFT_Q_CASE(32) MPFFT_Q_CASE(33) MPFFT_Q_CASE(34)
    default:
      return nullptr;
  }
#undef MPFFT_Q_CASE
}

static size_t queue_smem(const QueueShape &Q) {
  if (Q.family == kQueueLimbs) return (size_t)Q.L * Q.threads * sizeof(uint32_t);
  const int units = Q.family == kQueueTierDD ? DDT::kUnits : Q.family == kQueueTierQD ? QDT::kUnits : 1;
  return (size_t)Q.chunk * units * sizeof(double2) + kOrderBytes;
}

cudaError_t queue_prepare(const QueueShape &Q) {
  const void *fn = queue_fn(Q);
  if (!fn) return cudaErrorInvalidValue;
  if (Q.family == kQueueLimbs) return cudaSuccess;
  return cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kQueueSmemBytes);
}

int queue_ctas_per_sm(const QueueShape &Q) {
  const void *fn = queue_fn(Q);
  int n = 0;
  if (!fn || cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, fn, Q.threads, queue_smem(Q)) != cudaSuccess) return 1;
  return std::max(1, n);
}

cudaError_t queue_launch(const QueueShape &Q, const QueueItem *items, int nitems, int *head, int ctas, double scale,
                         cudaStream_t s) {
  if (nitems <= 0) return cudaSuccess;
  const void *fn = queue_fn(Q);
  if (!fn) return cudaErrorInvalidValue;
  void *args_mp[] = {(void *)&items, (void *)&nitems, (void *)&head};
  void *args_fp[] = {(void *)&items, (void *)&nitems, (void *)&head, (void *)&scale};
  return cudaLaunchKernel(fn, dim3(ctas), dim3(Q.threads), Q.family == kQueueLimbs ? args_mp : args_fp, queue_smem(Q),
                          s);
}

}  // namespace mpfft

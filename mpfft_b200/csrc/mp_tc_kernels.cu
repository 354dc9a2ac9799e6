// Multiprecision butterflies whose twiddle products run on the tensor cores
// (tcgen05.mma kind::i8: unsigned 8-bit operands, exact int32 accumulation
// in tensor memory), for large limb counts kTcMinLimbs <= L <= kTcMaxLimbs
// (P from about 1050 to 8200 bits at N = 1024).
//
// Product as a matrix product.  At one level and one butterfly index k every
// signal multiplies its operands by the same three twiddle constants (cos,
// cos+sin, |cos-sin| of 2 pi k/N).  Write an operand |x| as 4L bytes x_a and a
// twiddle w as 4L bytes w_c.  The byte columns of the product are
//     D[m][j] = sum_a x_m[a] * w[j - a]      (each < 4L * 255^2 < 2^27)
// i.e. the operand matrix X (signals m x bytes a) times a Toeplitz matrix of
// twiddle bytes: a dense int8 GEMM with M = 128 signals per CTA, N = output
// byte columns in tiles of 128, K = 4L operand bytes in steps of 32.
//
// The Toeplitz operand is never materialised.  In the no-swizzle K-major
// shared-memory layout an MMA operand is made of core matrices of 8 rows x 16
// bytes with a fixed 16-byte row stride; the descriptor gives the stride
// between the two 16-byte K halves (LBO) and between 8-row groups (SBO).  Row
// n = 8g + r of a tile is assigned output column j = J + g + 16(7 - r), and
// group g reads copy g of the reversed twiddle bytes, shifted by g:
//     copy_g[t] = w[Q + g - t],   B[n][a] = copy_g[Q - J - 112 + 16r + a]
// so consecutive rows are 16 bytes apart (row r+1 is column j-16), the K
// halves are 16 bytes apart (LBO = 16) and the groups are one copy apart
// (SBO = copy length).  Sixteen copies of ~4L+320 bytes describe every
// Toeplitz tile of every K step.
//
// Truncation and rounding.  Byte columns below J0 = 4L-8 (rounded down to a
// multiple of 16) are not formed; the product is
//     r = floor((sum_{j >= J0} D[j] 2^(8j) + 2^(32L-2)) / 2^(32L-1))
// (the dropped part is below 4L * 2^-64 units of r's last place), with the
// operand's sign applied afterwards.  The epilogue reads each signal's column
// sums from its tensor-memory lane, carries them in increasing j and streams
// the result limbs into their destination, merged with the first product of
// the same side exactly as the streaming kernels do (mp_big_kernels.cu).
//
// Inside a CTA: 256 threads, two per signal (group q = thread/128 of signal
// m = thread mod 128).  The integer work around the MMAs is carry chains over
// L limbs; each is cut into two segments that run at once and exchange their
// carries through shared memory:
//   operand   each thread adds and stores its half of the limbs with carry 0
//             in, publishes the segment's carry-out and whether it is all ones
//             or all zero; after a barrier every thread knows its carry-in and
//             the operand's sign and, where needed, finishes its segment
//   columns   a stage is two 128-column tiles; each thread folds the 32 limbs
//             of one from tensor memory, publishes carry-out and ripple, then
//             adds its carry-in; the MMAs of the next stage run meanwhile
//   combine   each thread forms the four outputs of the real or of the
//             imaginary part of the twiddled values
// Signs stay beside the products and enter as coefficients of the combine.
// Every wait is bounded (about two seconds of %globaltimer); on expiry the
// kernel records an error code instead of hanging.
//
// Measured (N=1024, batch 256, us per batch, one thread per signal and
// a launch per level / this):
// 36 limbs 735 / 550, 65 limbs 1239 / 962, 129 limbs 2556 / 1711, 254 limbs
// 7200 / 4390; four threads per signal (64 registers) 1416 at 65 limbs, with a
// launch per level instead of items (below) 1166.
#include <algorithm>
#include <climits>
#include <cstdint>

#include "mp_limbs.cuh"
#include "mp_stream.cuh"
#include "mpfft_internal.h"

namespace mpfft {

constexpr int kTcRows = 128;     // signals per CTA (MMA M)
constexpr int kTcThreads = 256;  // two per signal

// Tensor memory per CTA: two 128-column accumulators (one stage).  At least
// 80 KB of shared memory per CTA keeps a third CTA off the SM, so 2 x 256 of the
// 512 columns suffice and an allocation never waits.  (Measured: four CTAs per SM with one accumulator
// each and at most 128 registers per thread was slower from 65 limbs up.)
constexpr uint32_t kTcMinSmem = 80u * 1024u;
constexpr uint32_t kTcTmemCols = 256;
// instruction descriptor: D = s32, A = B = u8, both K-major, N = 128, M = 128
constexpr uint32_t kTcIdesc = (2u << 4) | ((128u >> 3) << 17) | ((128u >> 4) << 24);

__device__ int g_tc_error = 0;  // first error code of any CTA (0 = none)
// Limit of each wait -- on this CTA's own MMAs, and on the flags of the items
// whose outputs an item reads -- in ns of %globaltimer.  Only a test changes it
// (mpfft_diag_tc_set_wait_limit), to make the waits give up.
__device__ unsigned long long g_tc_wait_ns = 2000000000ull;
// Limit of the wait that drains a CTA's MMAs before it frees tensor memory
// after another wait gave up; not affected by the test setting.
constexpr unsigned long long kTcDrainNs = 2000000000ull;

struct TcGeom {
  int L, Kpad, J0, nt, Q, CL, wzw, seg;
  uint32_t offT, offWZ, offEx, offBar, offSlot, bytes;
};

__host__ __device__ inline TcGeom tc_geom(int L) {
  TcGeom g;
  g.L = L;
  g.Kpad = (4 * L + 31) & ~31;            // operand bytes, padded to the MMA K step
  g.J0 = (4 * L - 8) & ~15;               // first output byte column formed
  g.nt = (8 * L - g.J0 + 127) / 128;      // output tiles of 128 columns
  g.Q = (4 * L + 160 + 15) & ~15;         // reversal base of the twiddle copies
  g.CL = (g.Q + 160 + 15) & ~15;          // bytes per copy (covers every tile and K step)
  g.wzw = g.CL / 4 + 8;                   // words of a zero-padded twiddle
  g.seg = ((L + 1) / 2 + 3) & ~3;         // limbs per operand segment
  g.offT = 128u * g.Kpad;                 // operand rows first, then 16 copies of one twiddle
  g.offWZ = g.offT + 16u * g.CL;
  g.offEx = (g.offWZ + 4u * g.wzw + 15) & ~15u;  // exchange words [4][2][128]
  g.offBar = g.offEx + 16u * (uint32_t)kTcThreads;        // 2 mbarriers: stages, drain
  g.offSlot = g.offBar + 32;
  g.bytes = g.offSlot + 16 > kTcMinSmem ? g.offSlot + 16 : kTcMinSmem;
  return g;
}

// ---------------------------------------------------------------------------
// PTX wrappers
// ---------------------------------------------------------------------------

__device__ __forceinline__ uint32_t smem_addr(const void *p) {
  return (uint32_t)__cvta_generic_to_shared(p);
}

// shared-memory matrix descriptor: no swizzle, version 1 (sm_100)
__device__ __forceinline__ uint64_t tc_desc(uint32_t addr, uint32_t lbo, uint32_t sbo) {
  return (uint64_t)((addr >> 4) & 0x3FFFu) | ((uint64_t)((lbo >> 4) & 0x3FFFu) << 16) |
         ((uint64_t)((sbo >> 4) & 0x3FFFu) << 32) | (1ull << 46);
}

__device__ __forceinline__ void tc_mma(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::i8 [%0], %1, %2, %3, p;\n\t}\n" ::"r"(d),
      "l"(a), "l"(b), "r"(idesc), "r"(accumulate));
}

__device__ __forceinline__ void tc_commit(uint32_t bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar)
               : "memory");
}

__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void fence_async_smem() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }

__device__ __forceinline__ uint64_t global_ns() {
  uint64_t t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

// wait for the phase with the given parity to complete; false once `limit` ns
// have passed (checked before each try, so a limit of 0 gives up at once)
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity, unsigned long long limit) {
  const uint64_t t0 = global_ns();
  for (;;) {
    if (global_ns() - t0 >= limit) return false;
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}\n"
        : "=r"(ok)
        : "r"(bar), "r"(parity)
        : "memory");
    if (ok) return true;
  }
}

__device__ __forceinline__ void tmem_ld2(uint32_t addr, uint32_t &v0, uint32_t &v1) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x2.b32 {%0,%1}, [%2];" : "=r"(v0), "=r"(v1) : "r"(addr));
}

// ---------------------------------------------------------------------------
// CTA context: shared-memory layout, tensor memory, barriers
// ---------------------------------------------------------------------------

struct TcCtx {
  TcGeom G;
  uint8_t *smem;
  uint32_t *ex;          // exchange words: ex[a*256 + q*128 + m]
  uint32_t sA, sT, bar;  // shared addresses: operand rows, twiddle copies, mbarriers (stages, drain)
  uint32_t tmem;         // tensor-memory base (lane 0, first column)
  uint32_t ph;           // parity of the next stage's completion
  int q, m;              // this thread's group and signal
  bool bad;              // a wait expired: stop waiting, results are void
  unsigned long long wait_ns;  // limit of each wait
};

// all threads; warp 0 allocates the tensor memory
__device__ void tc_setup(TcCtx &c, uint8_t *smem, int L) {
  c.G = tc_geom(L);
  c.smem = smem;
  c.sA = smem_addr(smem);
  c.sT = c.sA + c.G.offT;
  c.bar = c.sA + c.G.offBar;
  c.ex = reinterpret_cast<uint32_t *>(smem + c.G.offEx);
  c.q = threadIdx.x >> 7;
  c.m = threadIdx.x & 127;
  c.ph = 0;
  c.bad = false;
  c.wait_ns = *(volatile unsigned long long *)&g_tc_wait_ns;
  if (threadIdx.x == 0) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(c.bar) : "memory");
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(c.bar + 8) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (threadIdx.x < 32) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(c.sA + c.G.offSlot),
                 "r"(kTcTmemCols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  c.tmem = *reinterpret_cast<volatile uint32_t *>(smem + c.G.offSlot);
}

__device__ void tc_teardown(TcCtx &c, int *err) {
  // After a wait gave up, MMAs of this CTA may still be writing tensor memory:
  // thread 0 (which issued them all) commits every MMA it issued to the drain
  // barrier and waits for it, bounded, before the memory is freed.  A wait
  // gives up only at the test setting of the limit or after seconds without
  // progress, so in practice this wait ends within microseconds.
  if (__syncthreads_or(c.bad ? 1 : 0)) {
    c.bad = true;
    if (threadIdx.x == 0) {
      tc_fence_after();
      tc_commit(c.bar + 8);
      if (!mbar_wait(c.bar + 8, 0, kTcDrainNs)) atomicCAS(err, 0, 2);  // 2: the drain wait expired too
    }
  }
  tc_fence_before();
  __syncthreads();
  if (threadIdx.x < 32) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(c.tmem), "r"(kTcTmemCols) : "memory");
  }
  if (c.bad) atomicCAS(err, 0, 1);  // 1: a tensor-core wait expired
}

// A twiddle (magnitude limbs w[l * tplane]) as 16 shifted reversed byte
// copies: copy_g[t] = w_byte[Q + g - t] (zero outside 0 .. 4L-1).  Two steps,
// with a barrier in between; the MMAs that read the previous copies are done.
__device__ void tc_twiddle_words(TcCtx &c, const uint32_t *w, size_t tplane) {
  const TcGeom &G = c.G;
  uint32_t *wz = reinterpret_cast<uint32_t *>(c.smem + G.offWZ);
  const int d4 = (G.CL - G.Q) / 4;  // wz byte u holds w_byte[u - (CL - Q)]
  for (int u = threadIdx.x; u < G.wzw; u += blockDim.x) {
    const int l = u - d4;
    wz[u] = (l >= 0 && l < G.L) ? w[(size_t)l * tplane] : 0u;
  }
}

__device__ void tc_twiddle_copies(TcCtx &c) {
  const TcGeom &G = c.G;
  const uint32_t *wz = reinterpret_cast<uint32_t *>(c.smem + G.offWZ);
  uint32_t *T = reinterpret_cast<uint32_t *>(c.smem + G.offT);
  const int cw = G.CL / 4;
  for (int g = threadIdx.x >> 5; g < 16; g += kTcThreads / 32)  // one copy per warp at a time
    for (int t = threadIdx.x & 31; t < cw; t += 32) {
      const int u0 = G.CL + g - 4 * t - 3;  // bytes u0 .. u0+3 of wz, reversed
      const uint32_t x = __funnelshift_r(wz[u0 >> 2], wz[(u0 >> 2) + 1], 8 * (u0 & 3));
      T[g * cw + t] = __byte_perm(x, 0, 0x0123);
    }
}

// Operand |pa +/- pb| (pb may be null) of signal m into operand row m of the
// CTA (4L bytes, zero padded to Kpad).  Rows of signals beyond the batch read
// signal 0 (the caller clamps the pointers); their products are never stored.
//
// Step 1 (before a barrier): this thread's segment [q*seg, ..) of the sum with
// carry 0 in, and the segment's flags: bit 0 carry-out, bit 1 all ones (a
// carry in goes through), bit 2 all zero, bit 3 a carry in changes the top
// limb's sign bit (every limb below it is ones, the limb 2^31-1 or 2^32-1), bit
// 31 that sign bit without it.
template <bool TWO>
__device__ __forceinline__ void tc_prep_sum(TcCtx &c, const uint32_t *pa, const uint32_t *pb, size_t plane, bool sub) {
  const TcGeom &G = c.G;
  const int lo = c.q * G.seg, hi = min(G.L, lo + G.seg);
  uint8_t *row = c.smem + (size_t)(c.m >> 3) * (8 * G.Kpad) + (c.m & 7) * 16 + (lo >> 2) * 128;
  uint32_t flags = 0x06u;  // an empty segment: no carry-out, all ones, all zero
  if (lo < hi) {
    const uint32_t msk = sub ? 0xffffffffu : 0u;
    uint32_t cy = (sub && c.q == 0) ? 1u : 0u, ones = 0xffffffffu, any = 0;
    pa += (size_t)lo * plane;
    if (TWO) pb += (size_t)lo * plane;
    int left = hi - lo;
    // blocks of kB limbs whose loads are all in flight; the last limbs (which hold the top one) apart
    constexpr int kB = TWO ? 12 : 16;
    while (left > kB) {
      uint32_t v[kB], w[kB];
#pragma unroll
      for (int e = 0; e < kB; ++e, pa += plane) {
        v[e] = *pa;
        if (TWO) {
          w[e] = *pb;
          pb += plane;
        }
      }
      if (TWO) {
        cc_set(cy);
#pragma unroll
        for (int e = 0; e < kB; ++e) v[e] = addc_cc(v[e], w[e] ^ msk);
        cy = carry();
      }
#pragma unroll
      for (int e = 0; e < kB; e += 2) {
        ones &= v[e] & v[e + 1];
        any |= v[e] | v[e + 1];
      }
#pragma unroll
      for (int h = 0; h < kB / 4; ++h, row += 128)
        *reinterpret_cast<uint4 *>(row) = make_uint4(v[4 * h], v[4 * h + 1], v[4 * h + 2], v[4 * h + 3]);
      left -= kB;
    }
    uint32_t v[kB], w[kB], last = 0, low = ones;
#pragma unroll
    for (int e = 0; e < kB; ++e) {  // (unconditional loads: predicated ones are issued one by one)
      const size_t o = (size_t)min(e, left - 1) * plane;
      v[e] = pa[o];
      if (TWO) w[e] = pb[o];
    }
#pragma unroll
    for (int e = 0; e < kB; ++e) {
      if (e < left) {
        if (TWO) v[e] = add_c(v[e], w[e] ^ msk, cy);
        low = ones;
        ones &= v[e];
        any |= v[e];
        last = v[e];
      } else {
        v[e] = 0;
      }
    }
#pragma unroll
    for (int h = 0; h < kB / 4; ++h, row += 128)
      if (4 * h < left) *reinterpret_cast<uint4 *>(row) = make_uint4(v[4 * h], v[4 * h + 1], v[4 * h + 2], v[4 * h + 3]);
    flags = cy | (ones == 0xffffffffu ? 2u : 0u) | (any == 0 ? 4u : 0u) |
            (low == 0xffffffffu && (last | 0x80000000u) == 0xffffffffu ? 8u : 0u) | (last & 0x80000000u);
    if (hi == G.L) {  // padding beyond the last chunk
      row = c.smem + (size_t)(c.m >> 3) * (8 * G.Kpad) + (c.m & 7) * 16;
      for (int ch = (G.L + 3) >> 2; ch < G.Kpad / 16; ++ch)
        *reinterpret_cast<uint4 *>(row + ch * 128) = make_uint4(0, 0, 0, 0);
    }
  }
  c.ex[threadIdx.x] = flags;
}

// Step 2 (after the barrier): carry in, sign, magnitude.  Returns the sign (1 = negative).
__device__ __forceinline__ uint32_t tc_prep_finish(TcCtx &c) {
  const TcGeom &G = c.G;
  const int L = G.L, lo = c.q * G.seg, hi = min(L, lo + G.seg), top = (L - 1) / G.seg;
  uint32_t cin = 0, ca = 0, zero = 1, cn = 0, neg = 0;
#pragma unroll
  for (int s = 0; s < 2; ++s) {
    const uint32_t f = c.ex[s * 128 + c.m];
    if (s == c.q) {
      ca = cin;   // carry into this segment
      cn = zero;  // every limb below it is zero: the +1 of a negation gets here
    }
    if (s == top) neg = ((f >> 31) ^ (cin & (f >> 3))) & 1u;
    zero &= (cin ? f >> 1 : f >> 2) & 1u;  // the segment ends up zero
    // (all ones plus a carry is zero with a carry out)
    cin = (f | (cin & (f >> 1))) & 1u;
  }
  if (ca | neg) {
    uint8_t *row = c.smem + (size_t)(c.m >> 3) * (8 * G.Kpad) + (c.m & 7) * 16;
    const uint32_t mk = neg ? 0xffffffffu : 0u;
    cn &= neg;
    row += (lo >> 2) * 128;
    int left = hi - lo;
    for (; left >= 4; left -= 4, row += 128) {
      uint4 u = *reinterpret_cast<uint4 *>(row);
      cc_set(ca);
      u.x = addc_cc(u.x, 0);
      u.y = addc_cc(u.y, 0);
      u.z = addc_cc(u.z, 0);
      u.w = addc_cc(u.w, 0);
      ca = carry();
      cc_set(cn);
      u.x = addc_cc(u.x ^ mk, 0);
      u.y = addc_cc(u.y ^ mk, 0);
      u.z = addc_cc(u.z ^ mk, 0);
      u.w = addc_cc(u.w ^ mk, 0);
      cn = carry();
      *reinterpret_cast<uint4 *>(row) = u;
    }
    if (left > 0) {
      uint4 u = *reinterpret_cast<uint4 *>(row);
      uint32_t v[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
      for (int e = 0; e < 3; ++e)
        if (e < left) v[e] = add_c(add_c(v[e], 0, ca) ^ mk, 0, cn);
      *reinterpret_cast<uint4 *>(row) = make_uint4(v[0], v[1], v[2], v[3]);
    }
  }
  return neg;
}

// thread 0: the MMAs of stage s (tiles 2s and 2s+1) into the two accumulators
__device__ void tc_issue(const TcCtx &c, int s) {
  const TcGeom &G = c.G;
  for (int t = 2 * s; t < min(2 * s + 2, G.nt); ++t) {
    const int J = G.J0 + 128 * t;
    const int k_lo = max(0, J - 4 * G.L + 1) >> 5;  // K steps that meet nonzero Toeplitz entries
    const int k_hi = min(G.Kpad >> 5, (J + 159) >> 5);
    const uint32_t tb = c.sT + (uint32_t)(G.Q - J - 112);
    const uint32_t d = c.tmem + (uint32_t)(t & 1) * 128u;
    for (int k = k_lo; k < k_hi; ++k)
      tc_mma(d, tc_desc(c.sA + 256u * k, 128u, 8u * G.Kpad), tc_desc(tb + 32u * k, 16u, G.CL), kTcIdesc,
             k > k_lo ? 1u : 0u);
  }
  tc_commit(c.bar);
}

// One product per signal of the CTA: operand rows and twiddle copies (in
// shared memory, made visible to the async proxy) -> magnitude limbs r_i at
// dst[i * ds]; all threads.
//
// Tile column n = 8g + r holds output byte column J + g + 16(7 - r), so the
// limb columns 4(7-r) + j of a tile (j < 4) are in columns 8(4j + e) + r, e < 4.
// Group q takes the 32 limb columns of tile q of a stage, eight at a time
// (two adjacent r of every column group); ONE_TILE (nt = 1, a plan forced onto
// this path at 28 limbs or less, or 30): 16 of the only tile (17 limbs, N=256, batch
// 256, us, 32 by one group / this: 204 / 179).
template <bool ONE_TILE>
__device__ __forceinline__ void tc_product(TcCtx &c, bool valid, uint32_t *dst, size_t ds) {
  const TcGeom &G = c.G;
  const int L = G.L, q = c.q;
  constexpr int kSeg = ONE_TILE ? 16 : 32;
  const uint32_t at = c.tmem + ((uint32_t)(((threadIdx.x >> 5) & 3) * 32) << 16) + (ONE_TILE ? 0u - 4u * q : 128u * q);
  uint32_t *exL = c.ex, *exC = c.ex + 256, *exT = c.ex + 512;  // low limb, carry-out | ripple, final top limb [2]
  uint32_t carry_in = 0;  // out of the stages so far (< 2^22)
  if (threadIdx.x == 0) {
    tc_fence_after();
    tc_issue(c, 0);
  }
  __syncwarp();
  const int ns = ONE_TILE ? 1 : (G.nt + 1) / 2;
#pragma unroll 1
  for (int s = 0; s < ns; ++s) {
    if (!c.bad && !mbar_wait(c.bar, c.ph, c.wait_ns)) c.bad = true;
    c.ph ^= 1u;
    tc_fence_after();
    const int m0 = (G.J0 >> 2) + 2 * kSeg * s + kSeg * q;  // this group's first limb column
    const bool some = ONE_TILE || 2 * s + q < G.nt;
    uint32_t l[kSeg];
    uint32_t co = 0;
    if (some) {
      uint64_t cy = 0;
#pragma unroll
      for (int h = 0; h < kSeg / 8; ++h) {  // limb columns 8h .. 8h+7: rows r = 7-2h, 6-2h
        uint32_t v[2][16];
#pragma unroll
        for (int g = 0; g < 16; ++g) tmem_ld2(at + 8u * g + (6u - 2u * h), v[1][g], v[0][g]);
        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          const int i = 8 * h + j;
          const uint32_t *w = v[j >> 2] + 4 * (j & 3);
          cy += (uint64_t)w[0] + (uint64_t)w[1] * 0x100u + (uint64_t)w[2] * 0x10000u + (uint64_t)w[3] * 0x1000000u;
          // + 2^(32L-2), round to nearest: limb L-1, the second to fifth of the first stage
          if (i >= 1 && i <= 4 && m0 + i == L - 1) cy += 1ull << 30;
          l[i] = (uint32_t)cy;
          cy >>= 32;
        }
      }
      co = (uint32_t)cy;
    } else {
#pragma unroll
      for (int i = 0; i < kSeg; ++i) l[i] = 0;
    }
    uint32_t ones = 0xffffffffu;
#pragma unroll
    for (int i = 1; i < kSeg; ++i) ones &= l[i];
    exL[threadIdx.x] = l[0];
    exC[threadIdx.x] = co | (ones == 0xffffffffu ? 0x80000000u : 0u);
    tc_fence_before();
    __syncthreads();  // the accumulators are in registers
    if (threadIdx.x == 0 && s + 1 < ns) {
      tc_fence_after();
      tc_issue(c, s + 1);
    }
    __syncwarp();
    uint32_t cin = 0;
#pragma unroll
    for (int g = 0; g < 2; ++g) {
      const uint32_t a = exL[g * 128 + c.m], f = exC[g * 128 + c.m];
      if (g == q) cin = carry_in;
      const uint32_t t = a + carry_in;  // the carry goes through the segment when limb 0 overflows into ones
      carry_in = (f & 0x7fffffffu) + ((t < a) & (f >> 31));
    }
    l[0] += cin;
    if (l[0] < cin) {  // rare: cin < 2^22
      l[1] = add_cc(l[1], 1);
#pragma unroll
      for (int i = 2; i < kSeg; ++i) l[i] = addc_cc(l[i], 0);
    }
    uint32_t *T = exT + (s & 1) * 256;
    T[threadIdx.x] = l[kSeg - 1];
    __syncthreads();
    if (some && valid) {
      uint32_t prev = q > 0 ? T[c.m] : (s > 0 ? exT[((s - 1) & 1) * 256 + 128 + c.m] : 0u);
      const int i0 = m0 - L;  // result limb of l[0]
      uint32_t *p = dst + (ptrdiff_t)i0 * (ptrdiff_t)ds;
      if (i0 >= 0 && i0 + kSeg <= L) {
#pragma unroll
        for (int i = 0; i < kSeg; ++i, p += ds) {
          *p = __funnelshift_r(prev, l[i], 31);
          prev = l[i];
        }
      } else {
#pragma unroll
        for (int i = 0; i < kSeg; ++i, p += ds) {
          if (i0 + i >= 0 && i0 + i < L) *p = __funnelshift_r(prev, l[i], 31);
          prev = l[i];
        }
      }
    }
  }
}

// Operand, twiddle and product in turn: the next operand's rows (and, when w is
// set, the next twiddle's copies) replace the last ones, whose MMAs are done.
__device__ __forceinline__ uint32_t tc_operand(TcCtx &c, const uint32_t *pa, const uint32_t *pb, size_t plane, bool sub,
                                               const uint32_t *w, size_t tplane) {
  if (pb) tc_prep_sum<true>(c, pa, pb, plane, sub);
  else tc_prep_sum<false>(c, pa, pa, plane, false);
  if (w) tc_twiddle_words(c, w, tplane);
  __syncthreads();
  const uint32_t neg = tc_prep_finish(c);
  if (w) tc_twiddle_copies(c);
  fence_async_smem();
  __syncthreads();
  return neg;
}

// The 3m3a merges and the L-combine, streamed 8 limbs at a time.  Per side h
// (Z+, Z-) the twiddled value is
//     T_h = sa_h P_h + sb_h S_h      (coefficients -1, 0, 1)
// with P_h the side's first product (in s0, s1) and S_h its slot, for the real
// (group 0) or the imaginary part (group 1); the outputs of mp_kernels.cu combine():
//     group 0  u0.r, zp.r = U0.r +- (T_0.r + T_1.r),  u1.i, zm.i = U1.i -+ (T_0.r - T_1.r)
//     group 1  u0.i, zp.i = U0.i +- (T_0.i + T_1.i),  u1.r, zm.r = U1.r +- (T_0.i - T_1.i)
// Both groups of a signal read each block of limbs before either writes it (the
// outputs go where the products are).
struct TcTerm {
  uint32_t S;  // word of the slot in a limb plane
  int sa, sb;
};

// y: the planes; c0, cs, c1: the component (0 or cim) of U0 and Z+ outputs, of
// the S slots, and of U1 and Z- outputs; U0, U1, D0, D1: words in a plane.
__device__ __forceinline__ void tc_combine(uint32_t *y, const uint32_t *s0, const uint32_t *s1, uint32_t U0, uint32_t U1,
                                           uint32_t D0, uint32_t D1, uint32_t P, size_t c0, size_t cs, size_t c1,
                                           size_t plane, size_t ps, int L, const TcTerm &t0, const TcTerm &t1,
                                           bool outer_swap, bool valid) {
  auto keep = [](int v) { return v ? 0xffffffffu : 0u; };
  auto flip = [](int v) { return v < 0 ? 0xffffffffu : 0u; };
  const uint32_t ka0 = keep(t0.sa), ma0 = flip(t0.sa), kb0 = keep(t0.sb), mb0 = flip(t0.sb);
  const uint32_t ka1 = keep(t1.sa), ma1 = flip(t1.sa), kb1 = keep(t1.sb), mb1 = flip(t1.sb);
  // A negated term is ~x + 1; with two of them in one sum the second +1 is added by a chain of its own
  const int n0 = (t0.sa < 0) + (t0.sb < 0), n1 = (t1.sa < 0) + (t1.sb < 0);
  uint32_t k0 = n0 > 0, k1 = n1 > 0, e0 = n0 > 1, e1 = n1 > 1, kp = 0, km = 1, ku0 = 0, kd0 = 1;
  uint32_t ku1 = outer_swap, kd1 = !outer_swap;
  const uint32_t mo = outer_swap ? 0xffffffffu : 0u;
  const bool extra = __any_sync(0xffffffffu, e0 | e1);
  uint32_t *y0 = y + c0, *ys = y + cs, *y1 = y + c1;
  constexpr int kB = 8;
#pragma unroll 1
  for (int i0 = 0; i0 < L; i0 += kB) {
    uint32_t u0[kB], u1[kB], x[kB], xs[kB], z[kB], zs[kB];
#pragma unroll
    for (int e = 0; e < kB; ++e) {
      const size_t i = (size_t)min(i0 + e, L - 1);  // tail: re-read the top limb, not stored
      u0[e] = (y0 + i * plane)[U0];
      u1[e] = (y1 + i * plane)[U1];
      xs[e] = (ys + i * plane)[t0.S];
      zs[e] = (ys + i * plane)[t1.S];
      x[e] = (s0 + i * ps)[P];
      z[e] = (s1 + i * ps)[P];
    }
    __syncthreads();
    // chains over the block's limbs, one after another, carries kept between blocks
    auto chain = [&](uint32_t(&r)[kB], const uint32_t(&p)[kB], const uint32_t(&q)[kB], uint32_t &k, uint32_t mq) {
      cc_set(k);
#pragma unroll
      for (int e = 0; e < kB; ++e) r[e] = addc_cc(p[e], q[e] ^ mq);
      k = carry();
    };
#pragma unroll
    for (int e = 0; e < kB; ++e) {
      x[e] = (x[e] & ka0) ^ ma0;
      xs[e] = (xs[e] & kb0) ^ mb0;
      z[e] = (z[e] & ka1) ^ ma1;
      zs[e] = (zs[e] & kb1) ^ mb1;
    }
    chain(x, x, xs, k0, 0u);
    chain(z, z, zs, k1, 0u);
    if (extra) {
      cc_set(e0);
#pragma unroll
      for (int e = 0; e < kB; ++e) x[e] = addc_cc(x[e], 0);
      e0 = carry();
      cc_set(e1);
#pragma unroll
      for (int e = 0; e < kB; ++e) z[e] = addc_cc(z[e], 0);
      e1 = carry();
    }
    chain(xs, x, z, kp, 0u);            // T_0 + T_1
    chain(zs, x, z, km, 0xffffffffu);   // T_0 - T_1
    chain(x, u0, xs, ku0, 0u);
    chain(u0, u0, xs, kd0, 0xffffffffu);
    chain(z, u1, zs, ku1, mo);
    chain(u1, u1, zs, kd1, ~mo);
    if (valid) {
      const int left = L - i0;
#pragma unroll
      for (int e = 0; e < kB; ++e)
        if (e < left) {
          (y0 + (size_t)(i0 + e) * plane)[U0] = x[e];
          (y0 + (size_t)(i0 + e) * plane)[D0] = u0[e];
          (y1 + (size_t)(i0 + e) * plane)[U1] = z[e];
          (y1 + (size_t)(i0 + e) * plane)[D1] = u1[e];
        }
    }
  }
}

// ---------------------------------------------------------------------------
// level kernel
// ---------------------------------------------------------------------------

// All levels in one persistent launch.  An item is one butterfly index k of one
// node for a group of 128 signals; the CTAs (two per SM) take items from a
// counter, level after level and k by k inside a level.  Butterfly k of a node
// of size n touches positions k mod n/4, which exactly three earlier items
// wrote: its first child's butterfly k mod n/8 and its other children's
// butterflies k mod n/16.  An item waits for those three (a flag each), not for
// the level, so the GPU stays full where a launch per level ended in a nearly
// empty wave (N=1024, batch 256: 254 to 510 items a level on 296 CTAs).  An item
// only waits for items taken before it, by CTAs that are running, so the waits
// end; they are bounded all the same.
//
// Products of an item (three per side, two at k = n/8) are formed on the tensor
// cores, their magnitudes stored unmerged (the first one of each side in the
// CTA's scratch, 2L limb planes of 128 words per CTA, the others in their Z
// slots), then one streamed merge + L-combine pass.  Products with the same
// twiddle follow each other, so each is laid out once.
struct TcRun {
  uint32_t *y;
  const uint32_t *tw;
  const uint8_t *dneg;
  uint32_t *scratch;
  uint32_t *flags;  // [level][N/4][groups]: item done; word k of a node at off/4 + k
  int *head;
  int *err;
  const int *node_off;
  int N, B, L, tws, groups;
  int lv0, lv1;  // levels of this launch
  int level_n[kMaxLevels], level_start[kMaxLevels], level_count[kMaxLevels];
  long long first[kMaxLevels + 1];  // first item of each level of the launch
};

__device__ __forceinline__ uint32_t ld_acquire(const uint32_t *p) {
  uint32_t v;
  asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}

// Butterfly k of the node of size n at offset off for signals 128 bg ..
template <bool ONE_TILE>
__device__ __forceinline__ void tc_butterfly(TcCtx &c, const TcRun &A, int n, int off, int k, int bg) {
  const int N = A.N, B = A.B, L = A.L, q = n >> 2, grp = c.q;
  uint32_t *y = A.y;
  const int b = bg * kTcRows + c.m;
  const bool valid = b < B;
  const int bs = valid ? b : 0;
  const size_t plane = (size_t)N * B;
  const size_t cim = (size_t)L * plane;
  // words of this thread's points within a limb plane (N*B < 2^31)
  const uint32_t qB = (uint32_t)q * B, u0 = (uint32_t)(off + k) * B + bs, u1 = u0 + qB, z0 = u1 + qB, z1 = z0 + qB;
  const size_t c0 = grp ? cim : 0, c1 = cim - c0;  // this group's part of the twiddled values and of U0; of U1
  if (k == 0) {  // no twiddle products: T = Z
    tc_combine(y, y, y, u0, u1, z0, z1, z0, c0, c0, c1, plane, plane, L, TcTerm{z0, 0, 1}, TcTerm{z1, 0, 1}, grp == 0,
               valid);
    return;
  }
  const size_t tplane = (size_t)(N >> 2) * A.tws;
  const int kn = k * (N / n) * A.tws;
  const bool special = 2 * k == q;
  const bool dn = special ? false : (A.dneg[kn] != 0);
  // scratch planes of 128 words: first product of Z+, of Z-
  const size_t ss = kTcRows;
  uint32_t *P0 = A.scratch + (size_t)blockIdx.x * 2 * L * kTcRows, *P1 = P0 + (size_t)L * ss;
  // Products j, side j & 1:
  //   j/2 = 0  P = c (Zr +/- Zi) -> scratch
  //   j/2 = 1  R1 = |cos-sin| Zi -> zi slot;   k = n/8: R = c (Zi - Zr) resp. c (Zr + Zi) -> zr slot
  //   j/2 = 2  R2 = (cos+sin) Zr -> zr slot
  uint32_t neg = 0;  // bit j: sign of product j of this thread's signal
#pragma unroll 1
  for (int j = 0; j < (special ? 4 : 6); ++j) {
    const int side = j & 1, step = j >> 1;
    uint32_t *zr = y + (side ? z1 : z0), *zi = zr + cim;
    const uint32_t *pa = zr, *pb = nullptr, *w = nullptr;
    bool sub = false;
    uint32_t *dst = (side ? P1 : P0) + c.m;
    size_t ds = ss;
    if (step == 0) {
      pb = zi;
      sub = side;
      if (side == 0) w = A.tw + kn;
    } else if (special) {
      pa = side ? zr : zi;
      pb = side ? zi : zr;
      sub = !side;
      dst = zr;
      ds = plane;
    } else if (step == 1) {
      pa = zi;
      if (side == 0) w = A.tw + (size_t)2 * L * tplane + kn;
      dst = zi;
      ds = plane;
    } else {
      if (side == 0) w = A.tw + (size_t)L * tplane + kn;
      dst = zr;
      ds = plane;
    }
    neg |= tc_operand(c, pa, pb, plane, sub, w, tplane) << j;
    tc_product<ONE_TILE>(c, valid, dst, ds);
  }
  // merges (T.r from the zi slot, T.i from the zr slot):
  //   Z+: T.r = P + (dn ? R1 : -R1), T.i = P - R2;   Z-: T.r = P + (dn ? -R1 : R1), T.i = R2 - P
  //   k = n/8: T.r = P, T.i = R
  auto sg = [&](int s, int j) { return ((neg >> j) & 1u) ? -s : s; };
  TcTerm t[2];
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    const uint32_t S = h ? z1 : z0;
    if (special) t[h] = grp ? TcTerm{S, 0, sg(1, 2 + h)} : TcTerm{S, sg(1, h), 0};
    else if (grp) t[h] = TcTerm{S, sg(h ? -1 : 1, h), sg(h ? 1 : -1, 4 + h)};
    else t[h] = TcTerm{S, sg(1, h), sg((dn != (h != 0)) ? 1 : -1, 2 + h)};
  }
  __syncthreads();  // every product is stored
  // (the slots are swapped: T.r from the imaginary one)
  tc_combine(y, P0, P1, u0, u1, z0, z1, c.m, c0, c1, c1, plane, ss, L, t[0], t[1], grp == 0, valid);
}

template <bool ONE_TILE>
__global__ void __launch_bounds__(kTcThreads, 2) mp_tc_levels_kernel(const __grid_constant__ TcRun A) {
  extern __shared__ __align__(1024) uint8_t tc_smem[];
  __shared__ int s_item;
  TcCtx c;
  tc_setup(c, tc_smem, A.L);
  for (;;) {
    if (threadIdx.x == 0) s_item = atomicAdd(A.head, 1);
    __syncthreads();
    const long long item = s_item;
    int lv = A.lv0;
    while (lv < A.lv1 && item >= A.first[lv + 1]) ++lv;
    if (lv == A.lv1) break;
    const int n = A.level_n[lv];
    int r = (int)(item - A.first[lv]);
    const int bg = r % A.groups;
    r /= A.groups;
    const int cnt = A.level_count[lv], off = A.node_off[A.level_start[lv] + r % cnt], k = r / cnt;
    // flags of this item and of the three it needs (children of 4 points and less come from the base cases)
    const size_t row = (size_t)(A.N >> 2);
    auto flag = [&](int level, int at) { return A.flags + ((size_t)level * row + at) * A.groups + bg; };
    if (threadIdx.x < 3 && !c.bad) {
      const int lw = threadIdx.x == 0 ? lv - 1 : lv - 2;
      if (lw >= A.lv0) {
        const int at = threadIdx.x == 0 ? (off >> 2) + (k & (n / 8 - 1))
                                        : ((off + n / 2 + (threadIdx.x == 2 ? n / 4 : 0)) >> 2) + (k & (n / 16 - 1));
        const uint32_t *f = flag(lw, at);
        const uint64_t t0 = global_ns();
        while (ld_acquire(f) == 0) {
          if (global_ns() - t0 >= c.wait_ns) {
            c.bad = true;
            break;
          }
          __nanosleep(100);
        }
      }
      __threadfence();
    }
    c.bad = __syncthreads_or(c.bad ? 1 : 0) != 0;
    tc_butterfly<ONE_TILE>(c, A, n, off, k, bg);
    __syncthreads();  // the item's outputs are written (and s_item is read)
    if (threadIdx.x == 0) {
      __threadfence();
      asm volatile("st.release.gpu.global.u32 [%0], %1;" ::"l"(flag(lv, (off >> 2) + k)), "r"(1u) : "memory");
    }
  }
  tc_teardown(c, A.err);
}

// products of B operands (limb planes x[i*B + b], two's complement) with one
// twiddle magnitude w[0 .. L-1]: out[i*B + b] = sign(x) * r (diagnostics)
__global__ void __launch_bounds__(kTcThreads, 2)
    mp_tc_mul_kernel(const uint32_t *__restrict__ x, const uint32_t *__restrict__ w, uint32_t *__restrict__ out,
                     int L, int B, int *err) {
  extern __shared__ __align__(1024) uint8_t tc_smem[];
  const int b = blockIdx.x * kTcRows + (int)(threadIdx.x & 127);
  const bool valid = b < B;
  const int bs = valid ? b : 0;
  TcCtx c;
  tc_setup(c, tc_smem, L);
  const uint32_t neg = tc_operand(c, x + bs, nullptr, (size_t)B, false, w, 1);
  tc_product<false>(c, valid, out + bs, (size_t)B);
  __syncthreads();
  if (valid && neg && threadIdx.x < kTcRows) {
    uint32_t cy = 1;
    for (int i = 0; i < L; ++i) out[(size_t)i * B + b] = add_c(~out[(size_t)i * B + b], 0, cy);
  }
  tc_teardown(c, err);
}

// ---------------------------------------------------------------------------
// the int8 tensor-core rate (the roofline denominator of the products above)
// ---------------------------------------------------------------------------
//
// Thread 0 of each CTA issues `count` MMAs of M=128, N=256, K=32 unsigned
// bytes into one 256-column tensor-memory accumulator (operands: zeroed
// shared-memory tiles, no-swizzle K-major as above), commits them to an
// mbarrier and waits for it (bounded); MACs = count * 128*256*32 per CTA.
static cudaError_t tc_prepare(const void *fn, uint32_t bytes, int **err);
constexpr uint32_t kTcPeakIdesc = (2u << 4) | ((256u >> 3) << 17) | ((128u >> 4) << 24);
constexpr uint32_t kTcPeakSmem = 80u * 1024u;  // keeps a third CTA off an SM (2 x 256 columns)

__global__ void __launch_bounds__(128, 1) mp_tc_peak_kernel(int count, int *err) {
  extern __shared__ __align__(1024) uint8_t sm[];
  // A: 128 rows x 32 bytes at 0, B: 256 rows x 32 bytes at 4096; slot and barrier after
  for (int i = threadIdx.x; i < (4096 + 8192) / 16; i += blockDim.x) reinterpret_cast<uint4 *>(sm)[i] = make_uint4(0, 0, 0, 0);
  const uint32_t base = smem_addr(sm), bar = base + 12288, slot = base + 12304;
  if (threadIdx.x == 0) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(bar) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (threadIdx.x < 32) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(slot), "r"(256u) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  fence_async_smem();
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *reinterpret_cast<volatile uint32_t *>(sm + 12304);
  if (threadIdx.x == 0) {
    const uint64_t da = tc_desc(base, 128u, 256u), db = tc_desc(base + 4096u, 128u, 256u);
    for (int i = 0; i < count; ++i) tc_mma(tmem, da, db, kTcPeakIdesc, i > 0 ? 1u : 0u);
    tc_commit(bar);
    if (!mbar_wait(bar, 0, kTcDrainNs)) atomicCAS(err, 0, 2);
  }
  tc_fence_before();
  __syncthreads();
  if (threadIdx.x < 32) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(256u) : "memory");
  }
}

cudaError_t mp_tc_int8_rate(double *macs_per_s) {
  int *err = nullptr;
  cudaError_t e = tc_prepare((const void *)mp_tc_peak_kernel, kTcPeakSmem, &err);
  if (e != cudaSuccess) return e;
  int dev = 0, sms = 0;
  if ((e = cudaGetDevice(&dev)) != cudaSuccess) return e;
  if ((e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev)) != cudaSuccess) return e;
  cudaEvent_t e0, e1;
  cudaEventCreate(&e0);
  cudaEventCreate(&e1);
  const int ctas = 2 * sms, count = 16384;
  mp_tc_peak_kernel<<<ctas, 128, kTcPeakSmem>>>(256, err);  // warm-up
  cudaEventRecord(e0);
  mp_tc_peak_kernel<<<ctas, 128, kTcPeakSmem>>>(count, err);
  cudaEventRecord(e1);
  e = cudaEventSynchronize(e1);
  float ms = 0;
  if (e == cudaSuccess) e = cudaEventElapsedTime(&ms, e0, e1);
  cudaEventDestroy(e0);
  cudaEventDestroy(e1);
  if (e == cudaSuccess) e = cudaGetLastError();
  if (e == cudaSuccess) *macs_per_s = (double)ctas * count * 128.0 * 256.0 * 32.0 / (ms * 1e-3);
  return e;
}

// ---------------------------------------------------------------------------
// host side
// ---------------------------------------------------------------------------

static cudaError_t tc_prepare(const void *fn, uint32_t bytes, int **err) {
  cudaError_t e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
  if (e != cudaSuccess) return e;
  return cudaGetSymbolAddress(reinterpret_cast<void **>(err), g_tc_error);
}

// CTAs of a persistent launch: two per SM, as far as there are items
static int tc_ctas(const MpDeviceTables &T, int B) {
  int dev = 0, sms = 148;
  if (cudaGetDevice(&dev) == cudaSuccess) cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  long long items = 0;
  for (int lv = 0; lv < T.nlevels; ++lv) items += (long long)T.level_count[lv] * (T.level_n[lv] / 4);
  return (int)std::max<long long>(1, std::min<long long>(2 * sms, items * (((long long)B + kTcRows - 1) / kTcRows)));
}

// scratch of one run: each CTA's product planes, then the item flags and the counter
static size_t tc_flag_words(const MpDeviceTables &T, int B) {
  const size_t nbg = ((size_t)B + kTcRows - 1) / kTcRows;
  return (size_t)std::max(T.nlevels, 1) * (T.N / 4) * nbg + 4;
}

size_t mp_tc_scratch_words(const MpDeviceTables &T, int L, int B) {
  return (size_t)tc_ctas(T, B) * 2 * L * kTcRows + tc_flag_words(T, B);
}

cudaError_t mp_tc_run_levels(int L, const MpDeviceTables &T, uint32_t *out, int B, uint32_t *scratch,
                             cudaStream_t s, LaunchTimer &timer) {
  if (T.nlevels == 0) return cudaSuccess;
  const TcGeom G = tc_geom(L);
  int *err = nullptr;
  const auto kernel = G.nt == 1 ? mp_tc_levels_kernel<true> : mp_tc_levels_kernel<false>;
  cudaError_t e = tc_prepare((const void *)kernel, G.bytes, &err);
  if (e != cudaSuccess) return e;
  const int ctas = tc_ctas(T, B);
  TcRun A{};
  A.y = out;
  A.tw = T.tw;
  A.dneg = T.dneg;
  A.scratch = scratch;
  A.flags = scratch + (size_t)ctas * 2 * L * kTcRows;
  const size_t fw = tc_flag_words(T, B);
  A.head = reinterpret_cast<int *>(A.flags + fw - 4);
  A.err = err;
  A.node_off = T.node_off;
  A.N = T.N;
  A.B = B;
  A.L = L;
  A.tws = T.tws;
  A.groups = (B + kTcRows - 1) / kTcRows;
  for (int lv = 0; lv < T.nlevels; ++lv) {
    A.level_n[lv] = T.level_n[lv];
    A.level_start[lv] = T.level_start[lv];
    A.level_count[lv] = T.level_count[lv];
  }
  // one launch; a timed call runs each level as a launch of its own
  const int step = timer.ms ? 1 : T.nlevels;
  for (int lv = 0; lv < T.nlevels && e == cudaSuccess; lv += step) {
    A.lv0 = lv;
    A.lv1 = std::min(lv + step, T.nlevels);
    A.first[lv] = 0;
    for (int l = lv; l < A.lv1; ++l)
      A.first[l + 1] = A.first[l] + (long long)T.level_count[l] * (T.level_n[l] / 4) * A.groups;
    if (A.first[A.lv1] > INT32_MAX - 2 * ctas) return cudaErrorInvalidValue;
    timer.begin();
    e = step == 1 ? cudaMemsetAsync(A.head, 0, sizeof(int), s) : cudaMemsetAsync(A.flags, 0, fw * 4, s);
    if (e != cudaSuccess) break;
    kernel<<<(unsigned)std::min<long long>(ctas, A.first[A.lv1]), kTcThreads, G.bytes, s>>>(A);
    timer.end();
    e = cudaGetLastError();
  }
  return e;
}

cudaError_t mp_tc_mul(int L, int B, const uint32_t *x, const uint32_t *w, uint32_t *out, cudaStream_t s) {
  const TcGeom G = tc_geom(L);
  int *err = nullptr;
  cudaError_t e = tc_prepare((const void *)mp_tc_mul_kernel, G.bytes, &err);
  if (e != cudaSuccess) return e;
  mp_tc_mul_kernel<<<(B + kTcRows - 1) / kTcRows, kTcThreads, G.bytes, s>>>(x, w, out, L, B, err);
  return cudaGetLastError();
}

cudaError_t mp_tc_set_wait_limit(unsigned long long ns) {
  return cudaMemcpyToSymbol(g_tc_wait_ns, &ns, sizeof ns);
}

cudaError_t mp_tc_take_error(int *code) {
  int *err = nullptr;
  cudaError_t e = cudaGetSymbolAddress(reinterpret_cast<void **>(&err), g_tc_error);
  if (e != cudaSuccess) return e;
  const int zero = 0;
  if ((e = cudaMemcpy(code, err, sizeof(int), cudaMemcpyDeviceToHost)) != cudaSuccess) return e;
  return cudaMemcpy(err, &zero, sizeof(int), cudaMemcpyHostToDevice);
}

size_t mp_tc_smem_bytes(int L) { return tc_geom(L).bytes; }

}  // namespace mpfft

// Fixed-point multi-limb arithmetic for the multiprecision FFT kernels.
//
// Number format (device): a signal is stored in block floating point -- one
// exponent per signal, kept on the host -- and each real component is an
// L-limb two's-complement integer A (32-bit limbs, least significant first)
// with F = 32L-1-H fraction bits, H = log2(N)+2 headroom bits.  Because the
// format is fixed point, additions and subtractions are exact carry chains
// (modular, so signs need no special handling); the only rounding in the whole
// transform is the one in each twiddle product.
//
// Twiddles are unsigned L-limb magnitudes with 32L-1 fraction bits (|w| <= sqrt 2
// for cos+sin); their signs are applied by the caller when it combines products.
//
// Layout: limb i of a component lives at `ptr[i * plane]` -- limb planes, so
// that consecutive threads (consecutive signals or butterfly indices) touch
// consecutive words and every load/store is coalesced.
#pragma once

#include <cstdint>

namespace mpfft {

// L2 eviction priorities for global accesses (cache-policy operands of
// ld/st ... .L2::cache_hint): evict_last keeps a line that will be read again
// soon, evict_first marks a line that will not be read before it leaves L2.
__device__ __forceinline__ uint64_t l2_policy_evict_last() {
  uint64_t p;
  asm volatile("createpolicy.fractional.L2::evict_last.b64 %0, 1.0;" : "=l"(p));
  return p;
}
__device__ __forceinline__ uint64_t l2_policy_evict_first() {
  uint64_t p;
  asm volatile("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(p));
  return p;
}
__device__ __forceinline__ uint64_t l2_policy_evict_normal() {
  uint64_t p;
  asm volatile("createpolicy.fractional.L2::evict_normal.b64 %0, 1.0;" : "=l"(p));
  return p;
}
__device__ __forceinline__ void st_hint(uint32_t *a, uint32_t v, uint64_t pol) {
  asm volatile("st.global.L2::cache_hint.b32 [%0], %1, %2;" ::"l"(a), "r"(v), "l"(pol) : "memory");
}
// (asm volatile: the compiler keeps these loads in program order, which also
// stops it from hoisting them far ahead of their use)
__device__ __forceinline__ uint32_t ld_hint(const uint32_t *a, uint64_t pol) {
  uint32_t v;
  asm volatile("ld.global.L2::cache_hint.b32 %0, [%1], %2;" : "=r"(v) : "l"(a), "l"(pol) : "memory");
  return v;
}

// one word of global memory to shared memory, asynchronously (cp_async_wait:
// this thread's copies so far have arrived)
__device__ __forceinline__ void cp_async4(uint32_t *dst, const uint32_t *src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src)
               : "memory");
}
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// one step of a carry chain: returns a + b + c (mod 2^32), c <- carry out
__device__ __forceinline__ uint32_t addc(uint32_t a, uint32_t b, uint32_t &c) {
  const uint64_t t = (uint64_t)a + b + c;
  c = (uint32_t)(t >> 32);
  return (uint32_t)t;
}

// Carry chains through the condition code: cc_set(c) sets the carry flag to c
// (0 or 1), add_cc / addc_cc add and set it, carry() reads it.  One chain at a time, with
// nothing else between its steps; the steps are volatile, so they stay in
// program order.  (One instruction per limb; addc above takes two.)
__device__ __forceinline__ void cc_set(uint32_t c) {
  uint32_t t;
  asm volatile("add.cc.u32 %0, %1, 0xffffffff;" : "=r"(t) : "r"(c));
}
__device__ __forceinline__ uint32_t add_cc(uint32_t a, uint32_t b) {
  uint32_t r;
  asm volatile("add.cc.u32 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b));
  return r;
}
__device__ __forceinline__ uint32_t addc_cc(uint32_t a, uint32_t b) {
  uint32_t r;
  asm volatile("addc.cc.u32 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b));
  return r;
}
__device__ __forceinline__ uint32_t carry() {
  uint32_t r;
  asm volatile("addc.u32 %0, 0, 0;" : "=r"(r));
  return r;
}
// (hi:lo) += x * t, carry out (mad_cc), carry in and out (madc_cc): the two
// halves of one product side by side, which is one 32x32+64-bit multiply-add
__device__ __forceinline__ void mad_cc(uint32_t &lo, uint32_t &hi, uint32_t x, uint32_t t) {
  asm volatile("mad.lo.cc.u32 %0, %2, %3, %0;\n\tmadc.hi.cc.u32 %1, %2, %3, %1;" : "+r"(lo), "+r"(hi) : "r"(x), "r"(t));
}
__device__ __forceinline__ void madc_cc(uint32_t &lo, uint32_t &hi, uint32_t x, uint32_t t) {
  asm volatile("madc.lo.cc.u32 %0, %2, %3, %0;\n\tmadc.hi.cc.u32 %1, %2, %3, %1;" : "+r"(lo), "+r"(hi) : "r"(x), "r"(t));
}

template <int L>
__device__ __forceinline__ void ld(uint32_t (&x)[L], const uint32_t *p, size_t plane) {
#pragma unroll
  for (int i = 0; i < L; ++i, p += plane) x[i] = *p;
}

template <int L>
__device__ __forceinline__ void st(uint32_t *p, size_t plane, const uint32_t (&x)[L]) {
#pragma unroll
  for (int i = 0; i < L; ++i, p += plane) *p = x[i];
}

// x = pa + pb  or  pa - pb, streamed from memory (pb may be null: x = pa)
template <int L>
__device__ __forceinline__ void ld_addsub(uint32_t (&x)[L], const uint32_t *pa, const uint32_t *pb,
                                          size_t plane, bool subtract) {
  if (!pb) {
    ld<L>(x, pa, plane);
    return;
  }
  const uint32_t m = subtract ? 0xffffffffu : 0u;
  uint32_t y[L];
#pragma unroll
  for (int i = 0; i < L; ++i, pa += plane, pb += plane) {
    x[i] = *pa;
    y[i] = *pb ^ m;
  }
  cc_set(subtract ? 1u : 0u);
#pragma unroll
  for (int i = 0; i < L; ++i) x[i] = addc_cc(x[i], y[i]);
}

// x = sx*x + sp*p with sx in {+1,-1}, sp in {+1,-1,0}; p streamed from memory.
// At most one operand is negated: a two's complement negation is ~v + 1.
template <int L>
__device__ __forceinline__ void combine_p(uint32_t (&x)[L], const uint32_t *p, size_t stride, bool negx,
                                          int sp) {
  const uint32_t mx = negx ? 0xffffffffu : 0u;
  const uint32_t mp = sp < 0 ? 0xffffffffu : 0u;
  const uint32_t keep = sp != 0 ? 0xffffffffu : 0u;
  uint32_t y[L];
#pragma unroll
  for (int i = 0; i < L; ++i, p += stride) y[i] = (*p & keep) ^ mp;
  cc_set(negx || sp < 0 ? 1u : 0u);
#pragma unroll
  for (int i = 0; i < L; ++i) x[i] = addc_cc(x[i] ^ mx, y[i]);
}

// ---------------------------------------------------------------------------
// truncated, rounded signed fixed-point product  x <- round(x * w / 2^(32L-1))
// ---------------------------------------------------------------------------
//
// In place: x (two's complement, |x| < 2^(32L-2)) holds the operand on entry
// and the product on return.  w: unsigned magnitude, L limbs at stride tplane.
//
// The limbs of x are multiplied as an unsigned integer x_u = x + s*2^(32L)
// (s = sign bit); the signed product is x_u*w - s*w*2^(32L), so for negative
// x the twiddle is subtracted once from the columns at and above 32L.  Only
// partial products x_i*w_j with i+j >= L-2 are formed (about L^2/2 + 3L/2 of
// them); the dropped lower part is below L*2^-31 units of the result's last
// place.  Adding 2^(32L-2) before the final shift rounds to nearest.
//
// The product is formed row by row (operand scanning): for each twiddle limb
// w_j the products x_i*w_j go to columns i+j and i+j+1.  Two accumulators,
// one for products whose low half falls on an even column (counted from L-2)
// and one for the odd ones, so that the products of a row fall on disjoint
// column pairs of each and run as two carry chains of one 32x32+64-bit
// multiply-add per product (mad_cc / madc_cc); the accumulators are added once
// at the end.  A form that adds each product's halves and a carry in C takes
// three instructions per product; the products are bound by instruction issue,
// so that costs (N=1024, batch 2048, us per batch, that form / this one): 9
// limbs 470 / 432, 17 limbs 1057 / 907, 25 limbs 1810 / 1521, 33 limbs 2810 / 2330.
//
// kPacked: w holds the L limbs contiguously, 16-byte aligned
// (tplane unused); they are read four at a time with 128-bit loads.
template <int L, bool kPacked = false>
__device__ __forceinline__ void mul_tw(uint32_t (&x)[L], const uint32_t *w, size_t tplane) {
  static_assert(L >= 2, "fixed-point product needs at least two limbs");
  // limb j of the twiddle: p points at it (strided planes) or at limb 0 (packed)
  uint4 v4;  // packed: limbs 4*(j/4) .. 4*(j/4)+3
  auto limb = [&](const uint32_t *p, int j) -> uint32_t {
    if (!kPacked) return *p;
    if ((j & 3) == 0) v4 = *reinterpret_cast<const uint4 *>(p + j);
    return (j & 3) == 0 ? v4.x : (j & 3) == 1 ? v4.y : (j & 3) == 2 ? v4.z : v4.w;
  };
  const uint32_t smask = 0u - (x[L - 1] >> 31);

  // ev[a] + od[a] is column (L-2+a), a = 0 .. L+1; ev holds the products with
  // even a in the pairs (a, a+1), od those with odd a
  uint32_t ev[L + 4], od[L + 4];
#pragma unroll
  for (int a = 0; a < L + 4; ++a) ev[a] = od[a] = 0;
  ev[1] = 1u << 30;  // + 2^(32L-2): round to nearest on the final >> (32L-1)

  const uint32_t *w0 = w;
#pragma unroll
  for (int j = 0; j < L; ++j, w += kPacked ? 0 : tplane) {
    const uint32_t t = limb(w, j);
    const int i0 = (L - 2 - j) > 0 ? (L - 2 - j) : 0;
    // rows below j reach column j+1, so the chains' carries land on empty words
#pragma unroll
    for (int par = 0; par < 2; ++par) {
      uint32_t(&acc)[L + 4] = par ? od : ev;
      const int a0 = i0 + j - (L - 2);
      const int first = i0 + ((a0 & 1) != par ? 1 : 0);
      if (first < L) {
        int a = 0;
#pragma unroll
        for (int i = first; i < L; i += 2) {
          a = i + j - (L - 2);
          if (i == first) mad_cc(acc[a], acc[a + 1], x[i], t);
          else madc_cc(acc[a], acc[a + 1], x[i], t);
        }
        if (a + 2 <= L + 1) acc[a + 2] = carry();
      }
    }
  }
  // columns = ev + od, minus s * w * 2^(32L) (columns L .. 2L-1, a = 2 .. L+1)
  uint32_t acc[L + 2];
  acc[0] = add_cc(ev[0], od[0]);
#pragma unroll
  for (int a = 1; a < L + 2; ++a) acc[a] = addc_cc(ev[a], od[a]);
  uint32_t nw[L];
#pragma unroll
  for (int j = 0; j < L; ++j, w0 += kPacked ? 0 : tplane) nw[j] = ~(limb(w0, j) & smask);
  cc_set(1u);
#pragma unroll
  for (int j = 0; j < L; ++j) acc[j + 2] = addc_cc(acc[j + 2], nw[j]);
  // x = (columns L-1 .. 2L-1) >> 31
#pragma unroll
  for (int i = 0; i < L; ++i) x[i] = __funnelshift_r(acc[i + 1], acc[i + 2], 31);
}

}  // namespace mpfft

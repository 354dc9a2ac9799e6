// Compensated floating-point tiers of the conjugate-pair split-radix FFT
// (device code shared by float_tier_kernels.cu and queue_kernels.cu):
// double-double (about 106 bits), quad-double (about 212 bits) and
// float-float (about 48 bits).
//
// A tier value is an unevaluated sum of K machine numbers (the "words") of
// decreasing magnitude, each at most half an ulp of the one above:
//   double-double  K = 2 doubles    hi + lo
//   quad-double    K = 4 doubles    x0 + x1 + x2 + x3
//   float-float    K = 2 floats     hi + lo
// The arithmetic is built from the published error-free transformations --
// Knuth's TwoSum, Dekker's Fast2Sum, the FMA form of TwoProd -- combined as in
// Hida, Li and Bailey's double-double / quad-double algorithms ("Algorithms
// for quad-double precision floating point arithmetic", ARITH 15, 2001):
// terms are summed order by order (order k = magnitude about 2^(-53k) of the
// leading word), the rounding errors of each order carried into the next,
// and the result renormalised with Fast2Sum / TwoSum chains.  Float-float
// keeps its additions on the FP32 pipe but forms every twiddle product, and
// rounds it back to a float pair, in FP64 (a float pair is exact in a
// double), which keeps the products at 2^-52 before the final 2^-48 rounding.
//
// Same tree and schedule as the FP64 kernels (d_core.cuh): chunks of up to T
// output positions run in shared memory, base cases straight from global memory
// (eight positions a thread: base cases of 4 and 2 points and the 8-point
// level), then passes that keep a column of points in registers for one level
// (quad-double), two (double-double) or three (float-float), the last one
// written out; the levels above run in global memory the same way.  T is the
// largest chunk whose planes fit 64 KB: 2048 points for double-double, 1024 for
// quad-double, 4096 for float-float.  Every level is the 4m2a butterfly with
// twiddles cos and sin of 2 pi k/N rounded to the tier by MPFR (float-float:
// to double).  Layout: word (c, h, b, p) at base[((c*K + h)*B + b)*N + p] -- c
// real/imaginary, h the word, each signal contiguous.
//
// Every file that includes this is compiled with --fmad=false: an error-free
// transformation must see the rounded product, not a contracted one.
#pragma once

#include <cstdint>

#include "mpfft_internal.h"
#include "sr_chunks.cuh"

namespace mpfft {

// ---------------------------------------------------------------------------
// error-free transformations
// ---------------------------------------------------------------------------

struct dd {
  double h, l;
};

__device__ __forceinline__ dd two_sum(double a, double b) {  // Knuth: s + e = a + b exactly
  const double s = a + b;
  const double bb = s - a;
  return dd{s, (a - (s - bb)) + (b - bb)};
}

__device__ __forceinline__ dd fast_two_sum(double a, double b) {  // Dekker, |a| >= |b|
  const double s = a + b;
  return dd{s, b - (s - a)};
}

__device__ __forceinline__ dd two_prod(double a, double b) {  // p + e = a * b exactly (FMA)
  const double p = a * b;
  return dd{p, fma(a, b, -p)};
}

struct ff {
  float h, l;
};

__device__ __forceinline__ ff two_sum_f(float a, float b) {
  const float s = __fadd_rn(a, b);
  const float bb = __fsub_rn(s, a);
  return ff{s, __fadd_rn(__fsub_rn(a, __fsub_rn(s, bb)), __fsub_rn(b, bb))};
}

__device__ __forceinline__ ff fast_two_sum_f(float a, float b) {
  const float s = __fadd_rn(a, b);
  return ff{s, __fsub_rn(b, __fsub_rn(s, a))};
}

// ---------------------------------------------------------------------------
// double-double
// ---------------------------------------------------------------------------

struct DDT {
  using W = double;  // storage word
  using V = dd;      // value
  using TW = dd;     // twiddle
  static constexpr int K = 2;
  static constexpr int kLgMax = 11;   // lg of the largest chunk (64 KB)
  static constexpr int kLeafLg = 3;   // lg of the positions of a base-case slot
  static constexpr int kLeafLgFew = 2, kLgFew = 9;  // the same for one chunk alone, up to 2^kLgFew points
  static constexpr int kLevels = 2;   // levels per pass

  // accurate addition (two TwoSums, two renormalisations)
  static __device__ __forceinline__ V add(V x, V y) {
    dd s = two_sum(x.h, y.h);
    const dd t = two_sum(x.l, y.l);
    s.l += t.h;
    s = fast_two_sum(s.h, s.l);
    s.l += t.l;
    return fast_two_sum(s.h, s.l);
  }
  static __device__ __forceinline__ V neg(V x) { return V{-x.h, -x.l}; }
  static __device__ __forceinline__ V sub(V x, V y) { return add(x, neg(y)); }
  static __device__ __forceinline__ V mul(V x, V y) {
    const double p = x.h * y.h;
    double e = fma(x.h, y.h, -p);  // TwoProd: p + e = x.h * y.h exactly
    e = fma(x.h, y.l, e);
    e = fma(x.l, y.h, e);
    return fast_two_sum(p, e);
  }
  static __device__ __forceinline__ V scale(V x, double s) { return V{x.h * s, x.l * s}; }
  static __device__ __forceinline__ V load(const W *p, size_t stride) { return V{p[0], p[stride]}; }
  static __device__ __forceinline__ void store(W *p, size_t stride, V v) {
    p[0] = v.h;
    p[stride] = v.l;
  }
  // shared memory: 16-byte units (re, im) of each word, planes of pl units
  static constexpr int kUnits = 2;
  static __device__ __forceinline__ void sload(const double2 *p, int pl, V &r, V &i) {
    const double2 a = p[0], b = p[pl];
    r = V{a.x, b.x};
    i = V{a.y, b.y};
  }
  static __device__ __forceinline__ void sstore(double2 *p, int pl, V r, V i) {
    p[0] = make_double2(r.h, i.h);
    p[pl] = make_double2(r.l, i.l);
  }
  // twiddles: (cos, sin) of each word, planes of len entries
  static constexpr int kTwWords = 2;
  static __device__ __forceinline__ void twiddle(const double2 *t, size_t len, TW &c, TW &s) {
    const double2 a = __ldg(t), b = __ldg(t + len);
    c = TW{a.x, b.x};
    s = TW{a.y, b.y};
  }
};

// ---------------------------------------------------------------------------
// quad-double
// ---------------------------------------------------------------------------

struct qd {
  double x0, x1, x2, x3;
};

// Four terms of decreasing order -> four non-overlapping words: a Fast2Sum
// chain from the bottom compresses the terms, a TwoSum chain from the top
// (exact whatever the magnitudes) pushes what overlaps down again.
__device__ __forceinline__ qd qd_renorm(double c0, double c1, double c2, double c3) {
  dd t = fast_two_sum(c2, c3);
  c2 = t.h, c3 = t.l;
  t = fast_two_sum(c1, c2);
  c1 = t.h, c2 = t.l;
  t = fast_two_sum(c0, c1);
  c0 = t.h, c1 = t.l;
  t = two_sum(c1, c2);
  c1 = t.h, c2 = t.l;
  t = two_sum(c2, c3);
  return qd{c0, c1, t.h, t.l};
}

struct QDT {
  using W = double;
  using V = qd;
  using TW = qd;
  static constexpr int K = 4;
  static constexpr int kLgMax = 10;
  static constexpr int kLeafLg = 2;
  static constexpr int kLeafLgFew = 2, kLgFew = 10;
  static constexpr int kLevels = 1;

  // Sum order by order: word i of x and of y are order i; the error of an
  // order-i TwoSum is order i+1; order 3 is summed plainly (its errors are
  // below 2^-212 relative).
  static __device__ __forceinline__ V add(const V &a, const V &b) {
    const dd s0 = two_sum(a.x0, b.x0);
    const dd s1 = two_sum(a.x1, b.x1);
    const dd s2 = two_sum(a.x2, b.x2);
    const double s3 = a.x3 + b.x3;
    const dd t1 = two_sum(s1.h, s0.l);   // order 1
    const dd u = two_sum(s2.h, s1.l);    // order 2 ...
    const dd t2 = two_sum(u.h, t1.l);
    const double t3 = s3 + s2.l + u.l + t2.l;  // order 3
    return qd_renorm(s0.h, t1.h, t2.h, t3);
  }
  static __device__ __forceinline__ V neg(const V &x) { return V{-x.x0, -x.x1, -x.x2, -x.x3}; }
  static __device__ __forceinline__ V sub(const V &x, const V &y) { return add(x, neg(y)); }
  // Products of order 0..2 exactly (TwoProd), order 3 plainly, order >= 4
  // dropped (below 2^-210 relative); each order summed with TwoSums whose
  // errors go to the next order.
  static __device__ __forceinline__ V mul(const V &a, const V &b) {
    const dd p00 = two_prod(a.x0, b.x0);
    const dd p01 = two_prod(a.x0, b.x1), p10 = two_prod(a.x1, b.x0);
    const dd p02 = two_prod(a.x0, b.x2), p11 = two_prod(a.x1, b.x1), p20 = two_prod(a.x2, b.x0);
    const double o3 = fma(a.x0, b.x3, fma(a.x1, b.x2, fma(a.x2, b.x1, a.x3 * b.x0)));
    const dd t = two_sum(p01.h, p10.h);  // order 1
    const dd t1 = two_sum(t.h, p00.l);
    const dd u = two_sum(p02.h, p11.h);  // order 2
    const dd v = two_sum(u.h, p20.h);
    const dd w = two_sum(v.h, p01.l);
    const dd x = two_sum(w.h, p10.l);
    const dd y = two_sum(x.h, t.l);
    const dd t2 = two_sum(y.h, t1.l);
    const double t3 = o3 + (p02.l + p11.l + p20.l) + (u.l + v.l + w.l) + (x.l + y.l + t2.l);  // order 3
    return qd_renorm(p00.h, t1.h, t2.h, t3);
  }
  static __device__ __forceinline__ V scale(const V &x, double s) { return V{x.x0 * s, x.x1 * s, x.x2 * s, x.x3 * s}; }
  static __device__ __forceinline__ V load(const W *p, size_t stride) {
    return V{p[0], p[stride], p[2 * stride], p[3 * stride]};
  }
  static __device__ __forceinline__ void store(W *p, size_t stride, const V &v) {
    p[0] = v.x0;
    p[stride] = v.x1;
    p[2 * stride] = v.x2;
    p[3 * stride] = v.x3;
  }
  static constexpr int kUnits = 4;
  static __device__ __forceinline__ void sload(const double2 *p, int pl, V &r, V &i) {
    const double2 a = p[0], b = p[pl], c = p[2 * pl], d = p[3 * pl];
    r = V{a.x, b.x, c.x, d.x};
    i = V{a.y, b.y, c.y, d.y};
  }
  static __device__ __forceinline__ void sstore(double2 *p, int pl, const V &r, const V &i) {
    p[0] = make_double2(r.x0, i.x0);
    p[pl] = make_double2(r.x1, i.x1);
    p[2 * pl] = make_double2(r.x2, i.x2);
    p[3 * pl] = make_double2(r.x3, i.x3);
  }
  static constexpr int kTwWords = 4;
  static __device__ __forceinline__ void twiddle(const double2 *t, size_t len, TW &c, TW &s) {
    const double2 a = __ldg(t), b = __ldg(t + len), e = __ldg(t + 2 * len), d = __ldg(t + 3 * len);
    c = TW{a.x, b.x, e.x, d.x};
    s = TW{a.y, b.y, e.y, d.y};
  }
};

// ---------------------------------------------------------------------------
// float-float (additions on the FP32 pipe, twiddle products in FP64)
// ---------------------------------------------------------------------------

struct FFT_ {
  using W = float;
  using V = ff;
  using TW = double;
  static constexpr int K = 2;
  static constexpr int kLgMax = 12;
  static constexpr int kLeafLg = 3;
  static constexpr int kLeafLgFew = 3, kLgFew = 9;
  static constexpr int kLevels = 3;

  static __device__ __forceinline__ V add(V a, V b) {
    const ff s = two_sum_f(a.h, b.h);
    return fast_two_sum_f(s.h, __fadd_rn(s.l, __fadd_rn(a.l, b.l)));
  }
  static __device__ __forceinline__ V neg(V x) { return V{-x.h, -x.l}; }
  static __device__ __forceinline__ V sub(V x, V y) { return add(x, neg(y)); }
  static __device__ __forceinline__ V scale(V x, double s) { return V{x.h * (float)s, x.l * (float)s}; }
  static __device__ __forceinline__ double to_d(V a) { return (double)a.h + (double)a.l; }
  // renormalisation in FP64: the nearest float, then the nearest float to the rest
  static __device__ __forceinline__ V from_d(double v) {
    const float h = __double2float_rn(v);
    return V{h, __double2float_rn(v - (double)h)};
  }
  static __device__ __forceinline__ V load(const W *p, size_t stride) { return V{p[0], p[stride]}; }
  static __device__ __forceinline__ void store(W *p, size_t stride, V v) {
    p[0] = v.h;
    p[stride] = v.l;
  }
  // one 16-byte unit per point: (re.h, im.h, re.l, im.l)
  static constexpr int kUnits = 1;
  static __device__ __forceinline__ void sload(const double2 *p, int, V &r, V &i) {
    const float4 a = *reinterpret_cast<const float4 *>(p);
    r = V{a.x, a.z};
    i = V{a.y, a.w};
  }
  static __device__ __forceinline__ void sstore(double2 *p, int, V r, V i) {
    *reinterpret_cast<float4 *>(p) = make_float4(r.h, i.h, r.l, i.l);
  }
  static constexpr int kTwWords = 1;
  static __device__ __forceinline__ void twiddle(const double2 *t, size_t, TW &c, TW &s) {
    const double2 a = __ldg(t);
    c = a.x;
    s = a.y;
  }
};

// ---------------------------------------------------------------------------
// the butterflies
// ---------------------------------------------------------------------------

// P = Z+ (c - i s) and M = Z- (c + i s), the twiddle products of the 4m2a
// butterfly (reference butterfly: lab/serial/double/serial_d_fft6.c:392-427)
template <class NT>
struct TwProducts {
  static __device__ __forceinline__ void run(typename NT::V zpr, typename NT::V zpi, typename NT::V zmr,
                                             typename NT::V zmi, typename NT::TW c, typename NT::TW s,
                                             typename NT::V &pr, typename NT::V &pi, typename NT::V &mr,
                                             typename NT::V &mi) {
    pr = NT::add(NT::mul(c, zpr), NT::mul(s, zpi));
    pi = NT::sub(NT::mul(c, zpi), NT::mul(s, zpr));
    mr = NT::sub(NT::mul(c, zmr), NT::mul(s, zmi));
    mi = NT::add(NT::mul(c, zmi), NT::mul(s, zmr));
  }
};

template <>
struct TwProducts<FFT_> {  // each complex product formed in FP64, rounded once to a float pair
  static __device__ __forceinline__ void run(ff zpr, ff zpi, ff zmr, ff zmi, double c, double s, ff &pr, ff &pi,
                                             ff &mr, ff &mi) {
    const double a = FFT_::to_d(zpr), b = FFT_::to_d(zpi), u = FFT_::to_d(zmr), v = FFT_::to_d(zmi);
    pr = FFT_::from_d(fma(c, a, s * b));
    pi = FFT_::from_d(fma(c, b, -(s * a)));
    mr = FFT_::from_d(fma(c, u, -(s * v)));
    mi = FFT_::from_d(fma(c, v, s * u));
  }
};

template <class NT>
__device__ __forceinline__ void bfly(typename NT::V &u0r, typename NT::V &u0i, typename NT::V &u1r,
                                     typename NT::V &u1i, typename NT::V &zpr, typename NT::V &zpi,
                                     typename NT::V &zmr, typename NT::V &zmi, typename NT::TW c, typename NT::TW s) {
  using V = typename NT::V;
  V pr, pi, mr, mi;
  TwProducts<NT>::run(zpr, zpi, zmr, zmi, c, s, pr, pi, mr, mi);
  const V sr = NT::add(pr, mr), si = NT::add(pi, mi), dr = NT::sub(pr, mr), di = NT::sub(pi, mi);
  const V a0r = NT::add(u0r, sr), a0i = NT::add(u0i, si), a2r = NT::sub(u0r, sr), a2i = NT::sub(u0i, si);
  const V a1r = NT::add(u1r, di), a1i = NT::sub(u1i, dr), a3r = NT::sub(u1r, di), a3i = NT::add(u1i, dr);
  u0r = a0r, u0i = a0i, u1r = a1r, u1i = a1i, zpr = a2r, zpi = a2i, zmr = a3r, zmi = a3i;
}

// the same with the outputs in the place of the inputs' columns
template <class NT>
struct Pt {
  typename NT::V r, i;
};
template <class NT>
__device__ __forceinline__ void bfly(Pt<NT> &u0, Pt<NT> &u1, Pt<NT> &zp, Pt<NT> &zm, typename NT::TW c,
                                     typename NT::TW s) {
  bfly<NT>(u0.r, u0.i, u1.r, u1.i, zp.r, zp.i, zm.r, zm.i, c, s);
}

// DFT of 2 and of 4 points in place (the base cases, reference :108-147)
template <class NT>
__device__ __forceinline__ void leaf2(Pt<NT> &a, Pt<NT> &b) {
  const Pt<NT> x = a, y = b;
  a = Pt<NT>{NT::add(x.r, y.r), NT::add(x.i, y.i)};
  b = Pt<NT>{NT::sub(x.r, y.r), NT::sub(x.i, y.i)};
}
template <class NT>
__device__ __forceinline__ void leaf4(Pt<NT> &a, Pt<NT> &b, Pt<NT> &c, Pt<NT> &d) {
  leaf2<NT>(a, c);  // even samples: a = sum, c = difference
  leaf2<NT>(b, d);
  const Pt<NT> e = a, f = c, g = b, h = d;
  a = Pt<NT>{NT::add(e.r, g.r), NT::add(e.i, g.i)};
  b = Pt<NT>{NT::add(f.r, h.i), NT::sub(f.i, h.r)};
  c = Pt<NT>{NT::sub(e.r, g.r), NT::sub(e.i, g.i)};
  d = Pt<NT>{NT::sub(f.r, h.i), NT::add(f.i, h.r)};
}

// the butterfly of an 8-point node at k = 0 (twiddle 1)
template <class NT>
__device__ __forceinline__ void leaf8_k0(Pt<NT> &u0, Pt<NT> &u1, Pt<NT> &zp, Pt<NT> &zm) {
  const Pt<NT> a = u0, b = u1;
  const typename NT::V sr = NT::add(zp.r, zm.r), si = NT::add(zp.i, zm.i);
  const typename NT::V dr = NT::sub(zp.r, zm.r), di = NT::sub(zp.i, zm.i);
  u0 = Pt<NT>{NT::add(a.r, sr), NT::add(a.i, si)};
  zp = Pt<NT>{NT::sub(a.r, sr), NT::sub(a.i, si)};
  u1 = Pt<NT>{NT::add(b.r, di), NT::sub(b.i, dr)};
  zm = Pt<NT>{NT::sub(b.r, di), NT::add(b.i, dr)};
}

// twiddle k of node size n: entry tier_level_tw(n) + k of the table of all levels n = 8 .. N
__host__ __device__ inline int tier_level_tw(int n) { return n / 4 - 2; }

template <class NT>
__device__ __forceinline__ void tier_tw(const TierTab &S, int n, int k, typename NT::TW &c, typename NT::TW &s) {
  NT::twiddle(S.tw + tier_level_tw(n) + k, S.tw_len, c, s);
}

// R levels of one column in registers: d_levels (d_core.cuh) for a tier
template <class NT, int R>
__device__ __forceinline__ void tier_levels(Pt<NT> (&v)[2 << R], bool big, const TierTab &S, int u, int k) {
  typename NT::TW c, s;
  if constexpr (R == 1) {
    if (!big) return;
    if (NT::kLeafLg == 3 && u == 2 && k == 0) {  // as in the 8-position base case: the same bits
      leaf8_k0<NT>(v[0], v[1], v[2], v[3]);
      return;
    }
    tier_tw<NT>(S, 4 * u, k, c, s);
    bfly<NT>(v[0], v[1], v[2], v[3], c, s);
  } else if constexpr (R == 2) {
    tier_tw<NT>(S, 4 * u, k, c, s);
    bfly<NT>(v[0], v[1], v[2], v[3], c, s);
    if (big) {
      tier_tw<NT>(S, 8 * u, k, c, s);
      bfly<NT>(v[0], v[2], v[4], v[6], c, s);
      tier_tw<NT>(S, 8 * u, k + u, c, s);
      bfly<NT>(v[1], v[3], v[5], v[7], c, s);
    } else {
      bfly<NT>(v[4], v[5], v[6], v[7], c, s);
    }
  } else {
    tier_tw<NT>(S, 4 * u, k, c, s);
    bfly<NT>(v[0], v[1], v[2], v[3], c, s);
    bfly<NT>(v[8], v[9], v[10], v[11], c, s);
    if (big) bfly<NT>(v[12], v[13], v[14], v[15], c, s);
    tier_tw<NT>(S, 8 * u, k, c, s);
    bfly<NT>(v[0], v[2], v[4], v[6], c, s);
    if (!big) bfly<NT>(v[8], v[10], v[12], v[14], c, s);
    tier_tw<NT>(S, 8 * u, k + u, c, s);
    bfly<NT>(v[1], v[3], v[5], v[7], c, s);
    if (!big) bfly<NT>(v[9], v[11], v[13], v[15], c, s);
    if (big) {
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        tier_tw<NT>(S, 16 * u, k + i * u, c, s);
        bfly<NT>(v[i], v[i + 4], v[i + 8], v[i + 12], c, s);
      }
    }
  }
}

// shared-memory index of the 16-byte units (as d_swz in d_core.cuh)
__device__ __forceinline__ int tier_swz(int m) { return m ^ (((m >> 3) ^ (m >> 6) ^ (m >> 9)) & 7); }

// One CTA's sub-transforms, as in d_core.cuh: SINGLE: G whole signals b0 ..;
// otherwise G chunks (input classes c0 ..) of signal b0.
template <class NT>
struct TierArgs {
  const typename NT::W *in;
  typename NT::W *out;
  int B, b0, c0, G;
  int per;  // levels per pass, up to kLevels
  double scale;
  bool final, swap_in, swap_out;
};

// What it takes (a gather pass, base cases of 4 points and one
// level per pass, one level per launch above / this; us): double-double 4096
// points x 512 171 / 139, 65536 x 32 266 / 197 -- half of the FP64 pipe's rate at
// 376 operations a butterfly; quad-double 4096 x 512 640 / 564; float-float 4096 x
// 512 84 / 52, 2^20 x 2 210 / 115 (memory).
//
// Base cases from global memory, one thread per slot of 2^kLeafLg output
// positions; either way the slot's inputs are of one class mod N/2^kLeafLg:
//   8  a node of 8 points (a leaf of 4, two of 2, and the level above) or two leaves of 4
//   4  a leaf of 4 or two of 2 (quad-double: eight points do not fit in registers)
template <class NT, bool SINGLE, bool FEW>
__device__ __forceinline__ void tier_leaves(const TierTab &S, const TierArgs<NT> &A, double2 *sm) {
  constexpr int kLg = FEW ? NT::kLeafLgFew : NT::kLeafLg, kPts = 1 << kLg;
  const int G = FEW ? 1 : A.G;
  const int lgT = S.lgT, nslots = 1 << (lgT - kLg), pl = G << lgT, N = S.N;
  const size_t hplane = (size_t)A.B * N, cplane = (size_t)NT::K * hplane;
  const size_t in_re = A.swap_in ? cplane : 0, in_im = A.swap_in ? 0 : cplane;
  for (int e = threadIdx.x; e < G * nslots; e += blockDim.x) {
    const int g = FEW ? 0 : SINGLE ? e / nslots : e % G;
    int s = FEW ? e : SINGLE ? e % nslots : e / G;
    int half = 0, sna = 0, rs = 1, chunk = 0, lgt = lgT;
    const TierLeafSlot *tab = S.slots[0];
    if (!SINGLE) {
      const SrChunk ch = S.chunks[A.c0 + g];
      chunk = ch.chunk;
      sna = ch.sna;
      rs = N >> lgT;
      if (!sr_chunk_big(chunk)) {
        tab = S.slots[1];
        --lgt;
        rs *= 2;
        half = s >= nslots / 2;
        s -= half ? nslots / 2 : 0;
        if (half) sna = ch.snb;
      }
    }
    if (kLg != NT::kLeafLg) tab += 1 << (lgt - NT::kLeafLg);  // behind the slots of 2^kLeafLg positions
    const TierLeafSlot L = tab[s];
    const int m = half * (nslots / 2) + L.m;
    const bool big = sr_chunk_big(chunk * nslots + m);
    const int a0 = sna + L.in[0] * rs, a1 = sna + L.in[1] * rs, a2 = sna + L.in[2] * rs, st = N >> 2;
    const size_t sig = (size_t)(SINGLE ? A.b0 + g : A.b0) * N;
    Pt<NT> v[kPts];
#pragma unroll
    for (int j = 0; j < kPts; ++j) {
      int idx;
      if (kPts == 8)  // block 0: a leaf of 4; block 1: a leaf of 4, or two of 2 points with stride N/2
        idx = j < 4 ? a0 + j * st : !big ? a1 + (j - 4) * st : (j < 6 ? a1 : a2) + 2 * (j & 1) * st;
      else
        idx = big ? a0 + j * st : (j < 2 ? a0 : a1) + 2 * (j & 1) * st;
      if (idx < 0) idx += N;
      v[j].r = NT::load(A.in + in_re + sig + idx, hplane);
      v[j].i = NT::load(A.in + in_im + sig + idx, hplane);
    }
    if constexpr (kPts == 8) {
      leaf4<NT>(v[0], v[1], v[2], v[3]);
      if (big) {
        leaf2<NT>(v[4], v[5]);
        leaf2<NT>(v[6], v[7]);
        // level of 8 points: k = 0 has no products, k = 1 the twiddle of 1/8 turn
        leaf8_k0<NT>(v[0], v[2], v[4], v[6]);
        typename NT::TW c, sn;
        tier_tw<NT>(S, 8, 1, c, sn);
        bfly<NT>(v[1], v[3], v[5], v[7], c, sn);
      } else {
        leaf4<NT>(v[4], v[5], v[6], v[7]);
      }
    } else if (big) {
      leaf4<NT>(v[0], v[1], v[2], v[3]);
    } else {
      leaf2<NT>(v[0], v[1]);
      leaf2<NT>(v[2], v[3]);
    }
    const int at = tier_swz((g << lgT) + kPts * m);
#pragma unroll
    for (int j = 0; j < kPts; ++j) NT::sstore(sm + (at ^ tier_swz(j)), pl, v[j].r, v[j].i);
  }
}

// a point of the transform's output (or of the levels below the upper ones)
template <class NT>
__device__ __forceinline__ void tier_put(typename NT::W *re, typename NT::W *im, size_t hplane, const Pt<NT> &v,
                                         double scale) {
  NT::store(re, hplane, NT::scale(v.r, scale));
  NT::store(im, hplane, NT::scale(v.i, scale));
}

// The chunks of a granularity by type, so that a warp's lanes mostly take the
// same branch: chunk indexes that are one node, ascending, at order[0 ..], those
// that are pairs at order[kOrderPairs ..] (by the index inside the sub-transform:
// in one that is itself a pair, its last chunk has the other type).
constexpr int kOrder = 272, kOrderPairs = 176;  // up to 256 chunks (16 of 4096 points), 171 nodes and 85 pairs
constexpr size_t kOrderBytes = kOrder * sizeof(uint16_t);

__device__ __forceinline__ uint16_t *tier_order(double2 *sm, int units) {
  return reinterpret_cast<uint16_t *>(sm + units);
}

__device__ __forceinline__ void tier_fill_order(uint16_t *order, int chunks) {
  for (int m = threadIdx.x; m < chunks; m += blockDim.x) {
    int rank = 0;  // nodes below m
    for (int s = 0; m >> s; ++s) rank += (s & 1) ? -(m >> s) : (m >> s);
    if (sr_chunk_big(m)) order[rank] = (uint16_t)m;
    else order[kOrderPairs + m - rank] = (uint16_t)m;
  }
}

// R levels of every chunk of 2^(R+1)*u positions, u = 2^lgu; last: to global memory
template <class NT, int R, bool SINGLE, bool FEW>
__device__ __forceinline__ void tier_pass(const TierTab &S, const TierArgs<NT> &A, double2 *sm, int lgu, bool last) {
  constexpr int M = 2 << R;
  const int G = FEW ? 1 : A.G;
  const int lgT = S.lgT, pl = G << lgT, u = 1 << lgu, lgc = lgu + R + 1, lgnch = lgT - lgc;
  const size_t hplane = (size_t)A.B * S.N, cplane = (size_t)NT::K * hplane;
  int off[M];
#pragma unroll
  for (int j = 0; j < M; ++j) off[j] = tier_swz(j << lgu);
  const uint16_t *order = tier_order(sm, pl * NT::kUnits);
  const int nch = 1 << lgnch, nodes = ((2 << lgnch) + ((lgnch & 1) ? -1 : 1)) / 3;
  // one level alone only has work in the nodes (and in a pair's last chunk, see above)
  const bool only = R == 1 && !last;
  const int slots = only ? nodes + (!SINGLE && (lgnch & 1) ? 1 : 0) : nch;
  for (int e = threadIdx.x; e < (G * slots) << lgu; e += blockDim.x) {
    const int k = e & (u - 1), x = e >> lgu, g = FEW ? 0 : only ? x / slots : x >> lgnch, i = x - g * slots;
    const int ci = i < nodes ? order[i] : only ? nch - 1 : order[kOrderPairs + i - nodes], c = (g << lgnch) + ci;
    const int chunk = SINGLE ? 0 : __ldg(&S.chunks[A.c0 + g].chunk);
    const bool big = sr_chunk_big((chunk << lgnch) + ci);
    if (only && !big) continue;
    const int at = tier_swz((c << lgc) + k);
    Pt<NT> v[M];
#pragma unroll
    for (int j = 0; j < M; ++j) NT::sload(sm + (at ^ off[j]), pl, v[j].r, v[j].i);
    tier_levels<NT, R>(v, big, S, u, k);
    if (!last) {
#pragma unroll
      for (int j = 0; j < M; ++j) NT::sstore(sm + (at ^ off[j]), pl, v[j].r, v[j].i);
    } else {
      const size_t p = (size_t)(SINGLE ? A.b0 + g : A.b0) * S.N + ((size_t)chunk << lgT) + ((size_t)ci << lgc) + k;
      typename NT::W *re = A.out + (A.swap_out ? cplane : 0) + p, *im = A.out + (A.swap_out ? 0 : cplane) + p;
      const double sc = A.final ? A.scale : 1.0;
#pragma unroll
      for (int j = 0; j < M; ++j) tier_put<NT>(re + ((size_t)j << lgu), im + ((size_t)j << lgu), hplane, v[j], sc);
    }
  }
}

// T = 2^lgT >= 8.  FEW: one chunk (A.G = 1) of few points: one level per pass
// (A.per = 1) and base cases of 2^kLeafLgFew positions, so that the most threads
// have work and none has much.
template <class NT, bool SINGLE, bool FEW>
__device__ __forceinline__ void tier_sub_transform(const TierTab &S, const TierArgs<NT> &A, double2 *sm) {
  constexpr int kLg = FEW ? NT::kLeafLgFew : NT::kLeafLg;
  tier_fill_order(tier_order(sm, (A.G << S.lgT) * NT::kUnits), 1 << (S.lgT - kLg) >> 1);
  tier_leaves<NT, SINGLE, FEW>(S, A, sm);
  int done = kLg;
  if (done == S.lgT) {  // (8 points) the base cases are the transform
    __syncthreads();
    const size_t hplane = (size_t)A.B * S.N, cplane = (size_t)NT::K * hplane;
    for (int e = threadIdx.x; e < A.G * 8; e += blockDim.x) {
      Pt<NT> v;
      NT::sload(sm + tier_swz(e), A.G * 8, v.r, v.i);
      typename NT::W *o = A.out + (size_t)A.b0 * 8 + e;
      tier_put<NT>(o + (A.swap_out ? cplane : 0), o + (A.swap_out ? 0 : cplane), hplane, v, A.final ? A.scale : 1.0);
    }
    return;
  }
  while (done < S.lgT) {
    const int r = FEW ? 1 : min(A.per, S.lgT - done);
    const bool last = done + r == S.lgT;
    __syncthreads();
    if (FEW) tier_pass<NT, 1, SINGLE, true>(S, A, sm, done - 1, last);
    else if (NT::kLevels == 3 && r == 3) tier_pass<NT, NT::kLevels, SINGLE, false>(S, A, sm, done - 1, last);
    else if (NT::kLevels >= 2 && r == 2)
      tier_pass<NT, NT::kLevels >= 2 ? 2 : 1, SINGLE, false>(S, A, sm, done - 1, last);
    else tier_pass<NT, 1, SINGLE, false>(S, A, sm, done - 1, last);
    done += r;
  }
}

// transforms of N <= 4 points: signal b0 + g
template <class NT>
__device__ __forceinline__ void tier_tiny(const TierTab &S, const TierArgs<NT> &A) {
  const size_t hplane = (size_t)A.B * S.N, cplane = (size_t)NT::K * hplane;
  for (int g = threadIdx.x; g < A.G; g += blockDim.x) {
    const size_t sig = (size_t)(A.b0 + g) * S.N;
    const typename NT::W *re = A.in + (A.swap_in ? cplane : 0) + sig, *im = A.in + (A.swap_in ? 0 : cplane) + sig;
    typename NT::W *ore = A.out + (A.swap_out ? cplane : 0) + sig, *oim = A.out + (A.swap_out ? 0 : cplane) + sig;
    Pt<NT> v[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int p = min(j, S.N - 1);
      v[j] = Pt<NT>{NT::load(re + p, hplane), NT::load(im + p, hplane)};
    }
    if (S.N == 4) leaf4<NT>(v[0], v[1], v[2], v[3]);
    else if (S.N == 2) leaf2<NT>(v[0], v[1]);
#pragma unroll
    for (int j = 0; j < 4; ++j)
      if (j < S.N) tier_put<NT>(ore + j, oim + j, hplane, v[j], A.scale);
  }
}

// R levels above the sub-transforms: column k of chunk c of signal b, in place
// in global memory
template <class NT, int R>
__device__ __forceinline__ void tier_upper_column(typename NT::W *__restrict__ y, const TierTab &S, int B, int lgu, int b,
                                                  int c, int k, double scale, bool swap_out) {
  constexpr int M = 2 << R;
  const size_t hplane = (size_t)B * S.N, cplane = (size_t)NT::K * hplane;
  const bool big = sr_chunk_big(c);
  if (R == 1 && !big) return;  // (never the last level: its chunk is the root)
  typename NT::W *re = y + (size_t)b * S.N + ((size_t)c << (lgu + R + 1)) + k, *im = re + cplane;
  Pt<NT> v[M];
#pragma unroll
  for (int j = 0; j < M; ++j) {
    v[j].r = NT::load(re + ((size_t)j << lgu), hplane);
    v[j].i = NT::load(im + ((size_t)j << lgu), hplane);
  }
  tier_levels<NT, R>(v, big, S, 1 << lgu, k);
  typename NT::W *ore = swap_out ? im : re, *oim = swap_out ? re : im;
#pragma unroll
  for (int j = 0; j < M; ++j) tier_put<NT>(ore + ((size_t)j << lgu), oim + ((size_t)j << lgu), hplane, v[j], scale);
}

// levels above the sub-transforms per pass: the fewest passes of at most
// `most` levels, evenly
__host__ __device__ inline int tier_upper_levels(int nl, int most) {
  const int passes = (nl + most - 1) / most;
  return passes ? (nl + passes - 1) / passes : 0;
}

}  // namespace mpfft

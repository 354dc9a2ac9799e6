// Device functions of the FP64 conjugate-pair split-radix kernels: the
// reference's n=8 and n=16 base cases, the 4m2a butterfly, passes of up to
// three levels in registers and one CTA's shared-memory sub-transforms.
// Shared by the per-launch kernels (d_kernels.cu) and the persistent
// work-queue kernels (queue_kernels.cu); every file that includes it is compiled with --fmad=false so that no
// multiply-add is contracted and results stay bit-identical to the reference.
#pragma once

#include <cstdint>

#include "mpfft_internal.h"
#include "sr_chunks.cuh"

namespace mpfft {

// 8-point base case on one part (reference :153-191); v = b1..b8
__device__ __forceinline__ void d8_part(const DConst &K, const double *x, double *v) {
  const double s04 = x[0] + x[4], d04 = x[0] - x[4];
  const double s26 = x[2] + x[6], d26 = x[2] - x[6];
  const double s17 = x[1] + x[7], d17 = x[1] - x[7];
  const double s35 = x[3] + x[5], d35 = x[3] - x[5];
  const double p = K.c8 * (d17 + d35);
  const double q = K.c8 * (s17 - s35);
  v[0] = s17 + s35;
  v[1] = s04 + s26;
  v[2] = s04 - s26;
  v[3] = d17 - d35;
  v[4] = d04 + q;
  v[5] = d04 - q;
  v[6] = d26 + p;
  v[7] = d26 - p;
}

struct D16 {
  double b5, b6, b11, b12, c1, c2, c3, c4, c9, c10, c11, c12, c17, c18, c19, c20;
};

// 16-point base case on one part (reference :218-348); the imaginary-part
// variant has a10, b3, b12 and the products m2, m4, m5, m6, m7 with the
// opposite sign convention, exactly as the reference writes them.
__device__ __forceinline__ void d16_part(const DConst &K, const double *x, bool im, D16 &o) {
  double s[8], d[8];
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    s[j] = x[j] + x[j + 8];
    d[j] = x[j] - x[j + 8];
  }
  const double a10 = im ? (-x[4] + x[12]) : d[4];
  const double b1 = s[0] - s[4], b2 = s[0] + s[4];
  const double b3 = im ? (-s[2] + s[6]) : (s[2] - s[6]);
  const double b4 = s[2] + s[6];
  const double b7 = s[1] - s[5], b8 = s[1] + s[5];
  const double b9 = s[3] - s[7], b10 = s[3] + s[7];
  const double b13 = d[1] + d[7], b14 = d[1] - d[7];
  const double b15 = d[3] + d[5], b16 = d[5] - d[3];
  o.b5 = b2 + b4;
  o.b6 = b2 - b4;
  o.b11 = b8 + b10;
  o.b12 = im ? (-b8 + b10) : (b8 - b10);
  const double m1 = K.c8 * (d[2] - d[6]);
  const double m2 = (im ? -K.c8 : K.c8) * (d[2] + d[6]);
  const double m3 = K.c8 * (b7 - b9);
  const double m4 = (im ? -K.c8 : K.c8) * (b7 + b9);
  const double m5 = (im ? -K.c16a : K.c16a) * (b13 + b15);
  const double m6 = (im ? K.c16b : -K.c16b) * b13;
  const double m7 = (im ? -K.c16d : K.c16d) * b15;
  const double m8 = K.c16c * (b14 + b16);
  const double m9 = K.c16d * b14;
  const double m10 = -K.c16b * b16;
  o.c1 = b1 + m3;
  o.c2 = b1 - m3;
  o.c3 = b3 + m4;
  o.c4 = m4 - b3;
  const double c5 = d[0] + m1, c6 = d[0] - m1;
  const double c7 = m9 - m8, c8 = m10 - m8;
  o.c9 = c5 + c7;
  o.c10 = c5 - c7;
  o.c11 = c6 + c8;
  o.c12 = c6 - c8;
  const double c13 = a10 + m2, c14 = a10 - m2;
  const double c15 = m5 + m6, c16 = m5 - m7;
  o.c17 = c13 + c15;
  o.c18 = c13 - c15;
  o.c19 = c14 + c16;
  o.c20 = c14 - c16;
}

// 16-point base case (reference :213-385): x -> out(position, value)
template <class F>
__device__ __forceinline__ void d_leaf16(const DConst &K, const double *xr, const double *xi, F out) {
  D16 R, I;
  d16_part(K, xr, false, R);
  d16_part(K, xi, true, I);
  // output stage (reference :350-382)
  out(0, R.b5 + R.b11, I.b5 + I.b11);
  out(8, R.b5 - R.b11, I.b5 - I.b11);
  out(4, R.b6 - I.b12, I.b6 - R.b12);
  out(12, R.b6 + I.b12, I.b6 + R.b12);
  out(1, R.c9 - I.c17, I.c9 - R.c17);
  out(15, R.c9 + I.c17, I.c9 + R.c17);
  out(2, R.c1 - I.c3, I.c1 - R.c3);
  out(14, R.c1 + I.c3, I.c1 + R.c3);
  out(3, R.c12 + I.c20, I.c12 + R.c20);
  out(13, R.c12 - I.c20, I.c12 - R.c20);
  out(5, R.c11 - I.c19, I.c11 - R.c19);
  out(11, R.c11 + I.c19, I.c11 + R.c19);
  out(6, R.c2 - I.c4, I.c2 - R.c4);
  out(10, R.c2 + I.c4, I.c2 + R.c4);
  out(7, R.c10 + I.c18, I.c10 + R.c18);
  out(9, R.c10 - I.c18, I.c10 - R.c18);
}

// 8-point base case (reference :148-212)
template <class F>
__device__ __forceinline__ void d_leaf8(const DConst &K, const double *xr, const double *xi, F out) {
  double R[8], I[8];
  d8_part(K, xr, R);
  d8_part(K, xi, I);
  // output stage (reference :193-209)
  out(0, R[1] + R[0], I[1] + I[0]);
  out(4, R[1] - R[0], I[1] - I[0]);
  out(1, R[4] + I[6], I[4] - R[6]);
  out(7, R[4] - I[6], I[4] + R[6]);
  out(2, R[2] + I[3], I[2] - R[3]);
  out(6, R[2] - I[3], I[2] + R[3]);
  out(3, R[5] - I[7], I[5] + R[7]);
  out(5, R[5] + I[7], I[5] - R[7]);
}

// 4m2a butterfly (reference :392-427) on values in registers: (U0, U1, Z+, Z-)
// -> the outputs that go to the same four positions.  A complex value is a
// double2 (x real, y imaginary), a twiddle w = (cos, sin).
__device__ __forceinline__ void d_bfly(double2 &u0, double2 &u1, double2 &zp, double2 &zm, double2 w) {
  const double pr = w.x * zp.x + w.y * zp.y, pi = w.x * zp.y - w.y * zp.x;
  const double mr = w.x * zm.x - w.y * zm.y, mi = w.x * zm.y + w.y * zm.x;
  const double sr = pr + mr, si = pi + mi, dr = pr - mr, di = pi - mi;
  const double2 a = u0, b = u1;
  u0 = make_double2(a.x + sr, a.y + si);
  zp = make_double2(a.x - sr, a.y - si);
  u1 = make_double2(b.x + di, b.y - dr);
  zm = make_double2(b.x - di, b.y + dr);
}

// R levels (node sizes 4u, 8u, 16u) of one column: v[j] = y[base + k + j*u],
// j < 2^(R+1), of the chunk of 2^(R+1)*u positions at `base`.  The chunk is
// one node of its own size (big), or a pair of nodes of half of it
// (sr_chunk_big); nodes of size 2u and below are complete.  Butterfly k + i*u of
// a node of size n only touches positions k mod u, so the column is closed
// under all its levels and they run in registers: the points cross memory once
// per R levels.  tw: per-level twiddles (sr_level_tw), all k.
template <int R>
__device__ __forceinline__ void d_levels(double2 (&v)[2 << R], bool big, const double2 *__restrict__ tw, int u, int k) {
  const double2 *t4 = tw + sr_level_tw(4 * u), *t8 = tw + sr_level_tw(8 * u), *t16 = tw + sr_level_tw(16 * u);
  if constexpr (R == 1) {
    if (big) d_bfly(v[0], v[1], v[2], v[3], __ldg(t4 + k));
  } else if constexpr (R == 2) {
    const double2 w4 = __ldg(t4 + k);
    d_bfly(v[0], v[1], v[2], v[3], w4);
    if (big) {
      d_bfly(v[0], v[2], v[4], v[6], __ldg(t8 + k));
      d_bfly(v[1], v[3], v[5], v[7], __ldg(t8 + k + u));
    } else {
      d_bfly(v[4], v[5], v[6], v[7], w4);
    }
  } else {
    const double2 w4 = __ldg(t4 + k), w8a = __ldg(t8 + k), w8b = __ldg(t8 + k + u);
    d_bfly(v[0], v[1], v[2], v[3], w4);
    d_bfly(v[8], v[9], v[10], v[11], w4);
    d_bfly(v[0], v[2], v[4], v[6], w8a);
    d_bfly(v[1], v[3], v[5], v[7], w8b);
    if (big) {
      d_bfly(v[12], v[13], v[14], v[15], w4);
#pragma unroll
      for (int i = 0; i < 4; ++i) d_bfly(v[i], v[i + 4], v[i + 8], v[i + 12], __ldg(t16 + k + i * u));
    } else {
      d_bfly(v[8], v[10], v[12], v[14], w8a);
      d_bfly(v[9], v[11], v[13], v[15], w8b);
    }
  }
}

// ---------------------------------------------------------------------------
// one CTA's sub-transforms: G chunks of T = 2^lgT points in shared memory
// ---------------------------------------------------------------------------
//
// SINGLE: T = N and the chunks are whole signals b0 .. b0+G-1.  Otherwise the
// chunks are those of G consecutive input classes c0 .. of signal b0 (chunk m
// = output positions [mT, (m+1)T), whose inputs are x[c + j*(N/T)] for its
// class c, so neighbouring classes share 32-byte sectors).
//
// Base cases straight from global memory: one thread per 16 output positions
// (a leaf of 16 points or a pair of leaves of 8, either way 16 inputs x[c' + j*(N/16)]
// of one class c'), then passes of up to three levels (d_levels), the last of
// which writes its outputs to global memory.  Shared memory is crossed once
// per pass: 3.5 times (in + out) at T = 4096 against about ten for two levels
// per pass after a separate gather.  Measured, 2^24 points in and out (us, that
// form / this one): N = 64 272 / 116, 1024 268 / 113, 4096 305 / 125 (4.3 TB/s
// of the 6.5 TB/s copy rate; two CTAs of 256 threads per SM, 16 points a thread,
// 122 registers), 65536 724 / 303, 2^20 963 / 439.
//
// Shared positions m are swizzled (low 3 bits ^= bits 3-5 ^ 6-8 ^ 9-11, 16-byte
// elements): columns are 8 or more consecutive k, conflict-free; the base
// cases' stores are scattered, and the host orders the slots so that they
// average 1.0-1.4 wavefronts per ideal one (counted by simulating them).
struct DSubArgs {
  const double *in;
  double *out;
  int B, b0, c0, G;
  double scale;       // applied to the outputs when `final`
  bool final;         // these outputs are the transform's
  bool swap_in, swap_out;
};

__device__ __forceinline__ int d_swz(int m) { return m ^ (((m >> 3) ^ (m >> 6) ^ (m >> 9)) & 7); }

template <bool SINGLE>
__device__ __forceinline__ int d_chunk_of(const DSubTab &S, const DSubArgs &A, int g) {
  return SINGLE ? 0 : __ldg(&S.chunks[A.c0 + g].chunk);
}

template <int LGT, bool SINGLE>
__device__ __forceinline__ void d_sub_leaves(const DSubTab &S, const DSubArgs &A, double2 *sm) {
  constexpr int T = 1 << LGT, kSlots = T / 16;
  const int step = S.N >> 4;  // input stride of a 16-point leaf
  for (int e = threadIdx.x; e < A.G * kSlots; e += blockDim.x) {
    const int g = SINGLE ? e / kSlots : e % A.G;
    int s = SINGLE ? e % kSlots : e / A.G;
    int half = 0, sna = 0, rs = 1, chunk = 0;
    const SrLeafSlot *tab = S.slots[0];
    if (!SINGLE) {
      const SrChunk ch = S.chunks[A.c0 + g];
      chunk = ch.chunk;
      sna = ch.sna;
      rs = S.N >> LGT;
      if (!sr_chunk_big(chunk)) {  // a pair of sub-transforms of T/2 points
        tab = S.slots[1];
        rs *= 2;
        half = s >= kSlots / 2;
        s -= half ? kSlots / 2 : 0;
        if (half) sna = ch.snb;
      }
    }
    const SrLeafSlot L = tab[s];
    const int m = half * (kSlots / 2) + L.m;  // 16-point block of the chunk
    const bool big = sr_chunk_big(chunk * kSlots + m);
    // leaf input j: sn + j*stride, j = 0 wrapped when negative
    const int a0 = sna + L.sna * rs, b0 = sna + L.snb * rs;
    const size_t b = (size_t)(SINGLE ? A.b0 + g : A.b0);
    const double *pr = A.in + (A.swap_in ? (size_t)A.B + b : b) * S.N;
    const double *pi = A.in + (A.swap_in ? b : (size_t)A.B + b) * S.N;
    double xr[16], xi[16];
#pragma unroll
    for (int j = 0; j < 16; ++j) {
      int idx = big ? a0 + j * step : (j < 8 ? a0 + 2 * j * step : b0 + 2 * (j - 8) * step);
      if ((j == 0 || j == 8) && idx < 0) idx += S.N;
      xr[j] = pr[idx];
      xi[j] = pi[idx];
    }
    const int at = d_swz(g * T + 16 * m);  // position p of the block is at ^ d_swz(p)
    if (big) {
      d_leaf16(S.K, xr, xi, [&](int p, double r, double i) { sm[at ^ d_swz(p)] = make_double2(r, i); });
    } else {
      d_leaf8(S.K, xr, xi, [&](int p, double r, double i) { sm[at ^ d_swz(p)] = make_double2(r, i); });
      d_leaf8(S.K, xr + 8, xi + 8, [&](int p, double r, double i) { sm[at ^ d_swz(p + 8)] = make_double2(r, i); });
    }
  }
}

// R levels of every chunk of 2^(R+1)*u positions, u = 2^LGU; LAST: the outputs go to global memory
template <int LGT, int LGU, int R, bool LAST, bool SINGLE>
__device__ __forceinline__ void d_sub_pass(const DSubTab &S, const DSubArgs &A, double2 *sm) {
  constexpr int u = 1 << LGU, M = 2 << R, lgc = LGU + R + 1, nch = 1 << (LGT - lgc);
  __syncthreads();
  for (int e = threadIdx.x; e < A.G << (LGT - R - 1); e += blockDim.x) {
    const int k = e & (u - 1), c = e >> LGU, g = c / nch;
    const int chunk = d_chunk_of<SINGLE>(S, A, g);
    const int at = d_swz((c << lgc) + k);  // the swizzle is linear over xor: position j*u is at ^ d_swz(j*u)
    double2 v[M];
#pragma unroll
    for (int j = 0; j < M; ++j) v[j] = sm[at ^ d_swz(j << LGU)];
    d_levels<R>(v, sr_chunk_big(chunk * nch + c % nch), S.tw, u, k);
    if (!LAST) {
#pragma unroll
      for (int j = 0; j < M; ++j) sm[at ^ d_swz(j << LGU)] = v[j];
    } else {
      const size_t b = (size_t)(SINGLE ? A.b0 + g : A.b0);
      const size_t p = ((size_t)chunk << LGT) + ((c % nch) << lgc) + k;
      double *qr = A.out + (A.swap_out ? (size_t)A.B + b : b) * S.N + p;
      double *qi = A.out + (A.swap_out ? b : (size_t)A.B + b) * S.N + p;
      const double sc = A.final ? A.scale : 1.0;
#pragma unroll
      for (int j = 0; j < M; ++j) {
        qr[j << LGU] = v[j].x * sc;
        qi[j << LGU] = v[j].y * sc;
      }
    }
  }
}

template <int LGT, bool SINGLE>
__device__ __forceinline__ void d_sub_transform(const DSubTab &S, const DSubArgs &A, double2 *sm) {
  static_assert(LGT >= 5 && LGT <= 12, "sub-transforms of 32 to 4096 points");
  d_sub_leaves<LGT, SINGLE>(S, A, sm);
  constexpr int R1 = LGT - 4 < 3 ? LGT - 4 : 3;
  d_sub_pass<LGT, 3, R1, (LGT <= 7), SINGLE>(S, A, sm);
  if constexpr (LGT > 7) {
    constexpr int R2 = LGT - 7 < 3 ? LGT - 7 : 3;
    d_sub_pass<LGT, 6, R2, (LGT <= 10), SINGLE>(S, A, sm);
  }
  if constexpr (LGT > 10) d_sub_pass<LGT, 9, LGT - 10, true, SINGLE>(S, A, sm);
}

// Transforms of N <= 16 points (one base case): G signals b0 .. through
// shared memory, so that the global accesses are contiguous.
__device__ __forceinline__ void d_tiny(const DSubTab &S, const DSubArgs &A, double2 *sm) {
  const int N = S.N, total = A.G * N;
  const size_t at = (size_t)A.b0 * N, im = (size_t)A.B * N;
  if (N == 1) {  // a scaled copy (2^23 signals, us, through shared memory / this: 120 / 85)
#pragma unroll 4
    for (int e = threadIdx.x; e < total; e += blockDim.x) {
      const double r = A.in[at + e + (A.swap_in ? im : 0)], i = A.in[at + e + (A.swap_in ? 0 : im)];
      A.out[at + e + (A.swap_out ? im : 0)] = r * A.scale;
      A.out[at + e + (A.swap_out ? 0 : im)] = i * A.scale;
    }
    return;
  }
  for (int e = threadIdx.x; e < total; e += blockDim.x)
    sm[d_swz(e)] = make_double2(A.in[at + e + (A.swap_in ? im : 0)], A.in[at + e + (A.swap_in ? 0 : im)]);
  __syncthreads();
  for (int g = threadIdx.x; g < A.G; g += blockDim.x) {
    const int o = g * N;
    double xr[16], xi[16];
#pragma unroll
    for (int j = 0; j < 16; ++j)
      if (j < N) {
        const double2 v = sm[d_swz(o + j)];
        xr[j] = v.x;
        xi[j] = v.y;
      }
    auto put = [&](int p, double r, double i) { sm[d_swz(o + p)] = make_double2(r * A.scale, i * A.scale); };
    if (N == 16) {
      d_leaf16(S.K, xr, xi, put);
    } else if (N == 8) {
      d_leaf8(S.K, xr, xi, put);
    } else if (N == 4) {  // reference :121-147
      const double er = xr[0] + xr[2], fr = xr[0] - xr[2], gr = xr[1] + xr[3], hr = xr[1] - xr[3];
      const double ei = xi[0] + xi[2], fi = xi[0] - xi[2], gi = xi[1] + xi[3], hi = xi[1] - xi[3];
      put(0, er + gr, ei + gi);
      put(1, fr + hi, fi - hr);
      put(2, er - gr, ei - gi);
      put(3, fr - hi, fi + hr);
    } else {  // N = 2, reference :108-120
      put(0, xr[0] + xr[1], xi[0] + xi[1]);
      put(1, xr[0] - xr[1], xi[0] - xi[1]);
    }
  }
  __syncthreads();
  for (int e = threadIdx.x; e < total; e += blockDim.x) {
    const double2 v = sm[d_swz(e)];
    A.out[at + e + (A.swap_out ? im : 0)] = v.x;
    A.out[at + e + (A.swap_out ? 0 : im)] = v.y;
  }
}

// ---------------------------------------------------------------------------
// R levels above the sub-transforms, in place in global memory: column k of
// chunk c (of 2^(R+1)*u positions) of signal b
// ---------------------------------------------------------------------------
template <int R>
__device__ __forceinline__ void d_upper_column(double *__restrict__ y, int N, int B, int lgu, int b, int c, int k,
                                               const double2 *__restrict__ tw, double scale, bool swap_out) {
  constexpr int M = 2 << R;
  const size_t u = (size_t)1 << lgu, p = ((size_t)c << (lgu + R + 1)) + k;
  double *yr = y + (size_t)b * N + p, *yi = y + ((size_t)B + b) * N + p;
  double2 v[M];
#pragma unroll
  for (int j = 0; j < M; ++j) v[j] = make_double2(yr[j * u], yi[j * u]);
  d_levels<R>(v, sr_chunk_big(c), tw, (int)u, k);
  double *qr = swap_out ? yi : yr, *qi = swap_out ? yr : yi;
#pragma unroll
  for (int j = 0; j < M; ++j) {
    qr[j * u] = v[j].x * scale;
    qi[j * u] = v[j].y * scale;
  }
}

// levels above the sub-transforms per pass: nl levels in the fewest passes of at most three, evenly
__host__ __device__ inline int d_upper_levels(int nl) {
  const int passes = (nl + 2) / 3;
  return passes ? (nl + passes - 1) / passes : 0;
}

}  // namespace mpfft

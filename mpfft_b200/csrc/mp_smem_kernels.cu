// Multiprecision transforms with several tree levels per launch in shared
// memory (sm_100a).
//
// A CTA holds a tile of M rows x F columns of complex limb numbers and runs
// every level of the tree that lies inside it, then writes it back: the planes
// cross L2 once per launch instead of once per level, and between levels a
// thread's operands are a shared-memory load away instead of an L2 round trip.
//
// Row j of a tile is output position off + j*u, its columns are consecutive
// words of the flattened (k, signal) index f = k*B + b, k < u, b < B, so any
// batch size fills the tile's rows with contiguous memory.  The M rows are a
// chunk of the tree of M*u positions (one node or a pair of half its size,
// sr_chunks.cuh); nodes of fewer than 4 rows are complete, and every node of 4
// rows or more lies inside the chunk together with all its butterflies of the
// tile's columns: butterfly r of a node of 4*qr rows combines rows r, r+qr,
// r+2qr, r+3qr of one column and has index k + r*u.
//   first launch  u = 1 (so f = b): rows are positions, columns signals; base
//                 cases of 4 and 2 points are read from the input
//   later ones    u = the rows of all earlier tiles: tiles of M rows, in place
//
// Two threads per butterfly, one per side: the thread of Z+ (Z-) forms the
// side's three products (3m3a; two at k = n/8) and their merges in place, as
// mp_level_kernel does, keeping the side's first product in registers; then
// the Z+ thread forms the four output components that involve U0, the Z- thread
// those of U1.  The same modular sums and products of the same operands as the
// level kernels, so the results are bit-identical.  The last level writes to
// global memory directly.
#include <algorithm>
#include <cstdint>

#include "mp_limbs.cuh"
#include "mpfft_internal.h"
#include "sr_chunks.cuh"

namespace mpfft {

// Tile size (complex numbers) by limb count, threads per CTA and the CTAs per
// SM the register allocation must allow.  The tile's planes take 8L bytes per
// number, so 227 KB hold 3228 numbers at 9 limbs and 880 at 33.  One thread per
// four numbers: a level keeps between half and all of P/2 sides busy, so more
// threads idle at the barriers and take the registers that let products
// overlap.  Measured (us, N=1024, batch 2048; tile/threads): 9 limbs 512/128
// 332, 512/256 410, 1024/256 369, 1024/512 443, 256/64 359; 13 limbs 512/128
// 626, 512/256 693, 256/64 647; 17 limbs 512/128 954, 512/256 1021, 256/64 954.
template <int L>
__host__ __device__ constexpr int smem_lg_tile() {
  return L <= 18 ? 9 : 8;
}
// Threads of a CTA: P/4, or P/2 (WIDE), which takes a level's butterflies in one
// round where the other takes two, but leaves room for fewer CTAs: their
// registers, not shared memory, then limit them.  smem_min_blocks: CTAs per SM.
template <int L, bool WIDE>
__host__ __device__ constexpr int tile_threads() {
  return 1 << (smem_lg_tile<L>() - (WIDE ? 1 : 2));
}
template <int L, bool WIDE>
__host__ __device__ constexpr int smem_min_blocks() {
  return WIDE ? (L <= 18 ? 2 : L <= 21 ? 4 : L <= 27 ? 3 : 2)
              : (L <= 4 ? 8 : L <= 6 ? 6 : L <= 10 ? 5 : L <= 14 ? 4 : L <= 18 ? 3 : L <= 27 ? 4 : 3);
}
// Limb counts whose tiles are always wide: four wide CTAs per SM without spills
// (20 limbs, us, narrow / wide: 65 k points 100 / 83, 131 k 101 / 94, 410 k
// 379 / 330, 524 k 355 / 343, 2 M 1267 / 1259)
template <int L>
__host__ __device__ constexpr bool tile_always_wide() {
  return L >= 19 && L <= 21;
}

struct MpTile {
  const uint32_t *in;  // first launch: the input planes
  uint32_t *out;
  int N, B;
  int lgM, lgF, lgu;
  int groups;           // column groups: ceil(u*B / F)
  const uint32_t *twp;  // packed twiddles [k][cos, cos+sin, |cos-sin|][Lp]
  const uint8_t *dneg;
  int tws;
};

// word of (row*F + col) in a plane: bit 4 ^= parity of the bits above, so that
// the two sides of a butterfly (rows qr apart) lie in different banks
__device__ __forceinline__ int tile_word(int w) { return w ^ ((__popc(w >> 5) & 1) << 4); }

// Limb counts whose three products are written out one after another (the
// side's operands loaded once, independent products overlapping); above, one
// copy of the product in a rolled loop keeps code and registers small.
constexpr int kTileUnrollMaxLimbs = 12;

// x = (negx ? -x : x) + (negq ? -q : q), at most one of them negated
template <int L>
__device__ __forceinline__ void merge(uint32_t (&x)[L], bool negx, const uint32_t (&q)[L], bool negq) {
  const uint32_t mx = negx ? 0xffffffffu : 0u, mq = negq ? 0xffffffffu : 0u;
  cc_set(negx || negq ? 1u : 0u);
#pragma unroll
  for (int i = 0; i < L; ++i) x[i] = addc_cc(x[i] ^ mx, q[i] ^ mq);
}

// The side's products of one butterfly: z points at the tile word of the
// side's Z row (real part; limbs P apart, imaginary part L*P on).  Operand,
// twiddle row and merge with the side's first product Q:
//            step 0           step 1                      step 2
//   general  Q=(Zr+-Zi)c      m.r = Q -+ d Zi -> im slot   m.i = +-(Q - s Zr) -> re slot
//   k = n/8  Q=(Zr+-Zi)c      m.i = (Zi-Zr)c | (Zr+Zi)c    m.r = Q -> im slot
//                                   -> re slot
template <int L>
__device__ __forceinline__ void tile_products(uint32_t *z, int side, bool special, bool dn,
                                              const uint32_t *__restrict__ tw) {
  constexpr int Lp = (L + 3) & ~3, P = 1 << smem_lg_tile<L>();
  uint32_t *zi = z + L * P;
  if constexpr (L <= kTileUnrollMaxLimbs) {
    uint32_t R[L], I[L], Q[L];
    ld<L>(R, z, P);
    ld<L>(I, zi, P);
#pragma unroll
    for (int i = 0; i < L; ++i) Q[i] = R[i];
    merge<L>(Q, false, I, side);
    mul_tw<L, true>(Q, tw, 0);
    if (!special) {
      mul_tw<L, true>(I, tw + 2 * Lp, 0);
      merge<L>(I, dn ^ (side == 0), Q, false);
      st<L>(zi, P, I);
      mul_tw<L, true>(R, tw + Lp, 0);
      merge<L>(R, side == 0, Q, side);
      st<L>(z, P, R);
    } else {
      merge<L>(R, !side, I, false);
      mul_tw<L, true>(R, tw, 0);
      st<L>(z, P, R);
      st<L>(zi, P, Q);
    }
    return;
  }
  uint32_t X[L], Q[L];
#pragma unroll 1
  for (int step = 0; step < 3; ++step) {
    const uint32_t *pa = z, *pb = nullptr;
    bool sub = false;
    int row = 0;
    if (step == 0) {
      pb = zi;
      sub = side;
    } else if (special) {
      if (step == 2) {
        st<L>(zi, P, Q);
        break;
      }
      pa = side ? z : zi;
      pb = side ? zi : z;
      sub = !side;
    } else if (step == 1) {
      pa = zi;
      row = 2;
    } else {
      row = 1;
    }
    ld_addsub<L>(X, pa, pb, P, sub);
    mul_tw<L, true>(X, tw + row * Lp, 0);
    if (step == 0) {
#pragma unroll
      for (int i = 0; i < L; ++i) Q[i] = X[i];
    } else if (special) {
      st<L>(z, P, X);
    } else {
      merge<L>(X, step == 1 ? dn ^ (side == 0) : side == 0, Q, step == 2 && side);
      st<L>(step == 1 ? zi : z, P, X);
    }
  }
}

// The four output components of one side (side 0: U0 and the Z+ row; side 1:
// U1 and the Z- row).  U: the side's U row, z1 / z2: the Z+ / Z- rows; d0, d1:
// where the two outputs go (words dp apart per limb, dc from real to imaginary
// part).  swapped: the Z rows hold (imaginary, real).  Both threads of a
// butterfly are lanes of one warp; each block of limbs is read by both before
// either writes it.
template <int L, bool kShared>
__device__ __forceinline__ void tile_combine(const uint32_t *U, const uint32_t *z1, const uint32_t *z2, int side,
                                             bool swapped, bool valid, uint32_t *d0, uint32_t *d1, size_t dp, size_t dc) {
  constexpr int P = 1 << smem_lg_tile<L>(), cim = L * P;
  const int cv = (swapped ? 1 : 0) != side ? cim : 0, cw = cim - cv;
  const uint32_t ms = side ? 0xffffffffu : 0u;
  uint32_t kv = side, kw = side, k0 = 0, k1 = 1, k2 = side, k3 = !side;  // the chains' carries
  constexpr int kB = L <= 10 ? L : 5;
#pragma unroll
  for (int i0 = 0; i0 < L; i0 += kB) {
    uint32_t ur[kB], ui[kB], v1[kB], v2[kB], w1[kB], w2[kB], r1[kB], s1[kB];
#pragma unroll
    for (int e = 0; e < kB; ++e)
      if (i0 + e < L) {
        const int o = (i0 + e) * P;
        ur[e] = U[o];
        ui[e] = U[o + cim];
        v1[e] = z1[o + cv];
        v2[e] = z2[o + cv] ^ ms;
        w1[e] = z1[o + cw];
        w2[e] = z2[o + cw] ^ ms;
      }
    if (kShared) __syncwarp();
    constexpr int kLast = (L - 1) / kB * kB;
    // a = b + c over the block's limbs, carry kept in k between blocks
    auto chain = [&](auto &a, const auto &b, const auto &c, uint32_t &k, uint32_t mc) {
      cc_set(k);
#pragma unroll
      for (int e = 0; e < kB; ++e)
        if (i0 + e < L) a[e] = addc_cc(b[e], c[e] ^ mc);
      if (i0 < kLast) k = carry();
    };
    chain(v1, v1, v2, kv, 0u);
    chain(w1, w1, w2, kw, 0u);
    chain(r1, ur, v1, k1, 0xffffffffu);
    chain(ur, ur, v1, k0, 0u);
    chain(s1, ui, w1, k3, ~ms);
    chain(ui, ui, w1, k2, ms);
#pragma unroll
    for (int e = 0; e < kB; ++e)
      if (i0 + e < L && valid) {
        const size_t o = (size_t)(i0 + e) * dp;
        d0[o] = ur[e];
        d1[o] = r1[e];
        d0[o + dc] = ui[e];
        d1[o + dc] = s1[e];
      }
  }
}

// Inputs of the leaf block at output positions 4m .. 4m+3: one leaf of 4 points
// x[a + j*N/4] (sr_chunk_big(m)) or two of 2 points, x[a + j*N/2] and x[b + j*N/2];
// j = 0 wraps when negative.  The walk of the recursion (parallel_mp_fft2.c:
// 180-182) along the bits of m.
__device__ __forceinline__ int2 leaf_inputs(int m, int lgN) {
  int sn = 0, s = 1;
  for (int i = lgN - 3; i >= 0;) {
    if (!((m >> i) & 1)) {
      s <<= 1;
      --i;
    } else if (i == 0) {
      return make_int2(sn + s, sn - s);
    } else {
      sn += ((m >> (i - 1)) & 1) ? -s : s;
      s <<= 2;
      i -= 2;
    }
  }
  return make_int2(sn, 0);
}

// Base cases (u = 1): one thread per (block of 4 positions, signal).
template <int L>
__device__ __forceinline__ void tile_leaves(const MpTile &A, int chunk, int b0, uint32_t *sm, const int2 *leaves) {
  constexpr int P = 1 << smem_lg_tile<L>();
  const int F = 1 << A.lgF, nslots = 1 << (A.lgM - 2);
  const size_t plane = (size_t)A.N * A.B, cim = (size_t)L * plane;
  for (int e = threadIdx.x; e < nslots << A.lgF; e += blockDim.x) {
    const int col = e & (F - 1), b = b0 + col;
    if (b >= A.B) continue;
    const int m = e >> A.lgF;
    const bool big = sr_chunk_big(chunk * nslots + m);
    const int sa = leaves[m].x, sb = leaves[m].y, step = A.N >> 2;
    const uint32_t *x[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      int idx = big ? sa + j * step : (j < 2 ? sa + 2 * j * step : sb + 2 * (j - 2) * step);
      if ((j == 0 || j == 2) && idx < 0) idx += A.N;
      x[j] = A.in + (size_t)idx * A.B + b;
    }
    uint32_t *y[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) y[j] = sm + tile_word(((4 * m + j) << A.lgF) + col);
    // leaf of 4:  X0 = x0+x2 + (x1+x3)      X2 = x0+x2 - (x1+x3)
    //             X1 = x0-x2 - i(x1-x3)     X3 = x0-x2 + i(x1-x3)
    // two of 2:   X0 = x0+x1, X1 = x0-x1 and the same of x2, x3
    int64_t c[8] = {0, 0, 0, 0, 0, 0, 0, 0};
#pragma unroll
    for (int i = 0; i < L; ++i) {
      int64_t r[4], q[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const uint32_t vr = x[j][i * plane], vi = x[j][i * plane + cim];
        r[j] = (i == L - 1) ? (int64_t)(int32_t)vr : (int64_t)vr;
        q[j] = (i == L - 1) ? (int64_t)(int32_t)vi : (int64_t)vi;
      }
      if (big) {
        const int64_t er = r[0] + r[2], fr = r[0] - r[2], gr = r[1] + r[3], hr = r[1] - r[3];
        const int64_t ei = q[0] + q[2], fi = q[0] - q[2], gi = q[1] + q[3], hi = q[1] - q[3];
        c[0] += er + gr, c[1] += fr + hi, c[2] += er - gr, c[3] += fr - hi;
        c[4] += ei + gi, c[5] += fi - hr, c[6] += ei - gi, c[7] += fi + hr;
      } else {
        c[0] += r[0] + r[1], c[1] += r[0] - r[1], c[2] += r[2] + r[3], c[3] += r[2] - r[3];
        c[4] += q[0] + q[1], c[5] += q[0] - q[1], c[6] += q[2] + q[3], c[7] += q[2] - q[3];
      }
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        y[j][i * P] = (uint32_t)c[j];
        y[j][(L + i) * P] = (uint32_t)c[4 + j];
        c[j] >>= 32;
        c[4 + j] >>= 32;
      }
    }
  }
}

// Butterflies r0 .. r0+nr-1 of every node of one level.  t: lg of the number of
// chunks of the node size in the tile; cnt nodes, node j < listed at chunk
// nodes[j], the one after them at the last chunk.  last: outputs to global memory.
template <int L>
__device__ __forceinline__ void tile_level(const MpTile &A, uint32_t *sm, const uint16_t *nodes, int chunk, int lgq,
                                           int t, int cnt, int listed, int r0, int nr, int f0, int fmax, bool last) {
  constexpr int Lp = (L + 3) & ~3, P = 1 << smem_lg_tile<L>();
  const int qr = 1 << lgq;
  const int ls = min(4, A.lgF), colhi = A.lgF - ls;
  const size_t plane = (size_t)A.N * A.B;
  const int total = (cnt * nr) << (A.lgF + 1);
  const int lgn = A.lgu + lgq + 2;  // lg of the node size
  const int wq = qr << A.lgF, sw1 = tile_word(wq), sw2 = tile_word(2 * wq);
  // divisions by nr and B as multiplications: exact while x * divisor < 2^20
  const unsigned inv_nr = ((1u << 20) + nr - 1) / nr;
  const int k0 = A.lgu ? f0 / A.B : 0, b0 = f0 - k0 * A.B;
  const unsigned inv_B = A.B < 512 ? ((1u << 20) + A.B - 1) / A.B : 0;
  for (int e0 = threadIdx.x & ~31; e0 < total; e0 += blockDim.x) {
    const int e = e0 + (threadIdx.x & 31);
    const int side = (e >> ls) & 1;
    const int col = (e & ((1 << ls) - 1)) | (((e >> (ls + 1)) & ((1 << colhi) - 1)) << ls);
    const int xi = e >> (A.lgF + 1);
    const int f = f0 + col;
    const bool valid = e < total && f < fmax;
    const int node = (int)((xi * inv_nr) >> 20), r = r0 + xi - node * nr;
    const int m = node < listed ? nodes[node] : (1 << t) - 1;
    const int row = valid ? m * 4 * qr + r : 0;
    // tile_word is linear over xor and the row quarters are separate bits
    const int w0 = tile_word((row << A.lgF) + (valid ? col : 0));
    uint32_t *u = sm + (w0 ^ (side ? sw1 : 0)), *z1 = sm + (w0 ^ sw2), *z2 = sm + (w0 ^ sw1 ^ sw2);
    int k = r << A.lgu;
    if (A.lgu) k += k0 + (A.B < 512 ? (int)(((b0 + col) * inv_B) >> 20) : b0 + col >= A.B ? 1 : 0);
    if (valid && k != 0) {
      const bool special = 2 * k == (1 << (lgn - 2));
      const int kn = (k * A.tws) << (31 - __clz(A.N) - lgn);
      const bool dn = special ? false : A.dneg[kn] != 0;
      tile_products<L>(side ? z2 : z1, side, special, dn, A.twp + (size_t)kn * (3 * Lp));
    }
    __syncwarp();
    if (last) {
      const size_t at = (size_t)chunk << A.lgM << A.lgu;
      uint32_t *g = A.out + (at + ((size_t)(row + side * qr) << A.lgu)) * A.B + (valid ? f : 0);
      tile_combine<L, false>(u, z1, z2, side, k != 0, valid, g, g + (((size_t)2 * qr) << A.lgu) * A.B, plane,
                             (size_t)L * plane);
    } else {
      tile_combine<L, true>(u, z1, z2, side, k != 0, valid, u, side ? z2 : z1, P, (size_t)L * P);
    }
  }
}

template <int L, bool LEAF, bool WIDE>
__global__ void __launch_bounds__(tile_threads<L, WIDE>(), smem_min_blocks<L, WIDE>())
    mp_tile_kernel(const __grid_constant__ MpTile A) {
  extern __shared__ __align__(16) uint32_t tile_smem[];
  constexpr int P = 1 << smem_lg_tile<L>();
  const int M = 1 << A.lgM, F = 1 << A.lgF;
  uint32_t *sm = tile_smem;
  int2 *leaves = reinterpret_cast<int2 *>(sm + 2 * L * P);                   // M/4 (first launch)
  uint16_t *nodes = reinterpret_cast<uint16_t *>(leaves + (LEAF ? M / 4 : 0));  // M/4
  const int group = blockIdx.x % A.groups, chunk = blockIdx.x / A.groups;
  const bool big = sr_chunk_big(chunk);
  const int f0 = group << A.lgF;
  const int fmax = (int)min((long long)A.B << A.lgu, (long long)f0 + F);
  // node j of a level is chunk nodes[j]: the chunks with an even number of trailing ones, ascending
  for (int m = threadIdx.x; m < M / 4; m += blockDim.x) {
    if (sr_chunk_big(m)) {
      int rank = 0;
      for (int s = 0; m >> s; ++s) rank += (s & 1) ? -(m >> s) : (m >> s);
      nodes[rank] = (uint16_t)m;
    }
    if (LEAF) leaves[m] = leaf_inputs(chunk * (M / 4) + m, 31 - __clz(A.N));
  }
  if (LEAF) {
    __syncthreads();
    tile_leaves<L>(A, chunk, f0, sm, leaves);
  } else {
    const size_t plane = (size_t)A.N * A.B, rstep = (size_t)A.B << A.lgu;
    const uint32_t *src = A.out + ((size_t)chunk << A.lgM << A.lgu) * A.B + f0;
    for (int w = threadIdx.x; w < M << A.lgF; w += blockDim.x) {
      const int col = w & (F - 1), row = w >> A.lgF;
      if (f0 + col < fmax) {
        const uint32_t *p = src + row * rstep + col;
        uint32_t *d = sm + tile_word(w);
#pragma unroll 4
        for (int x = 0; x < 2 * L; ++x) cp_async4(d + x * P, p + x * plane);
      }
    }
    cp_async_wait();
  }
  // phase 0 of a first-launch level: the butterflies with products, r = k = 1 .. qr-1;
  // phase 1: k = 0
  int lgq = LEAF ? 1 : 0, phase = 0;
#pragma unroll 1
  for (;;) {
    const int t = A.lgM - lgq - 2;
    if (t < 0) break;
    // the nodes of a big chunk's level; in a pair chunk the last chunk (all ones) changes sides
    const int of_big = ((2 << t) + ((t & 1) ? -1 : 1)) / 3;
    const int cnt = big ? of_big : ((t & 1) ? of_big + 1 : of_big - 1);
    if (cnt <= 0) break;
    const bool last = t == (big ? 0 : 1);
    const int qr = 1 << lgq;
    const int r0 = LEAF && phase == 0 ? 1 : 0, nr = LEAF ? (phase == 0 ? qr - 1 : 1) : qr;
    if (phase == 0) __syncthreads();
    tile_level<L>(A, sm, nodes, chunk, lgq, t, cnt, min(cnt, of_big), r0, nr, f0, fmax, last);
    if (LEAF && phase == 0) {
      phase = 1;
    } else {
      if (last) break;
      phase = 0;
      ++lgq;
    }
  }
}

// ---------------------------------------------------------------------------
// host side
// ---------------------------------------------------------------------------

template <int L, bool LEAF, bool WIDE>
static cudaError_t tile_launch(const MpTile &A, long long ctas, cudaStream_t s) {
  constexpr int P = 1 << smem_lg_tile<L>();
  const size_t smem = (size_t)8 * L * P + ((size_t)(LEAF ? 10 : 2) << (A.lgM - 2)) + 8;
  const cudaError_t e = cudaFuncSetAttribute(mp_tile_kernel<L, LEAF, WIDE>,
                                             cudaFuncAttributeMaxDynamicSharedMemorySize, 8 * L * P + 10 * P / 4 + 8);
  if (e != cudaSuccess) return e;
  mp_tile_kernel<L, LEAF, WIDE><<<(unsigned)ctas, tile_threads<L, WIDE>(), smem, s>>>(A);
  return cudaGetLastError();
}

// Launches whose tiles all run at once as wide CTAs take those, to 14 limbs
// only while no SM gets two (us, narrow / wide: 4 limbs 16 k points 22.2 / 19.9;
// 9 limbs 66 k 40.7 / 37.4; 17 limbs 33 k 68.6 / 55.8, 131 k 83.3 / 75.5; 23 limbs 66 k
// 115.8 / 94.8; 33 limbs 66 k 184 / 149).  Past that the narrow ones, of which more
// fit, are the faster or the same (11 limbs 131 k 48.9 / 50.1, 205 k 58.3 / 63.2;
// 9 limbs 2 M 329 / 409; 17 limbs 410 k 267 / 284; 25 limbs 131 k 130 / 153; 33 limbs
// 524 k 849 / 901).
template <int L>
constexpr int kWideTilesPerSm = L <= 14 ? 1 : smem_min_blocks<L, true>();

template <int L, bool LEAF>
static cudaError_t tile_launch(const MpTile &A, cudaStream_t s) {
  const long long ctas = ((long long)A.N >> (A.lgM + A.lgu)) * A.groups;
  if constexpr (!tile_always_wide<L>()) {
    if (ctas > 148LL * kWideTilesPerSm<L>) return tile_launch<L, LEAF, false>(A, ctas, s);
  }
  return tile_launch<L, LEAF, true>(A, ctas, s);
}

static int lg2(long long n) { return 63 - __builtin_clzll((unsigned long long)n); }

// Signals per first-launch tile: the largest power of two up to the room that
// wastes at most an eighth of the columns.  Fewer than 16 signals: the fewest
// columns, those of one signal counted 3/2 times and of two 11/9 times (rows of
// one or two words: what they took more, geometric mean over 2 to 33 limbs, 64 to
// 2^18 points; an eighth at most / this: 3 signals 1 / 0.87, 5 1 / 0.91, 7 1 / 0.78,
// 9 1 / 0.92, 13 1 / 0.88; from 16 signals on the two differ by less than waves of
// CTAs do).
static int tile_lg_signals(int B, int most) {
  long long least = 0;
  int best = 0;
  for (int l = most; l >= 0; --l) {
    const long long S = 1LL << l, columns = (B + S - 1) / S * S;
    if (B >= 16) {
      if (columns * 8 <= 9LL * B) return l;
      continue;
    }
    const long long cost = columns * (l == 0 ? 27 : l == 1 ? 22 : 18);
    if (l == most || cost < least) least = cost, best = l;
  }
  return best;
}

template <int L>
static cudaError_t tile_run(const MpDeviceTables &T, const uint32_t *in, uint32_t *out, int B, cudaStream_t s) {
  constexpr int lgP = smem_lg_tile<L>();
  const int lgN = lg2(T.N);
  MpTile A{in, out, T.N, B, 0, 0, 0, 1, T.twp, T.dneg, T.tws};
  // eight signals a row fill 32-byte sectors; more only when the signals are short
  A.lgF = tile_lg_signals(B, std::max(3, lgP - lgN));
  A.lgM = std::min(lgN, lgP - A.lgF);
  A.groups = (B + (1 << A.lgF) - 1) >> A.lgF;
  cudaError_t e = tile_launch<L, true>(A, s);
  // the levels above in the fewest tiles of at least eight columns
  int done = A.lgM;
  const int most = lgP - 4, passes = (lgN - done + most - 1) / most;
  for (int p = 0; p < passes && e == cudaSuccess; ++p) {
    const int r = (lgN - done + passes - p - 1) / (passes - p);
    A.lgu = done - 1;
    A.lgM = r + 1;
    A.lgF = lgP - A.lgM;
    const long long cols = (long long)B << A.lgu;
    A.groups = (int)((cols + (1 << A.lgF) - 1) >> A.lgF);
    e = tile_launch<L, false>(A, s);
    done += r;
  }
  return e;
}

// Which transforms run in tiles (points N*B by limb count), measured over N = 64
// .. 16384, B = 1 .. 1536 against one launch per level or level pair:
//   from   a tile's latency is hidden by the others; long single signals, which
//          take a launch more, last (4 limbs: 4 k points 1.00x, 8 k 1.01 .. 1.15x;
//          9 limbs: 8 k 0.88 .. 1.06x, 12 k 0.93 .. 1.0x for three to seven
//          signals, 16 k 1.12 .. 1.27x; 12 limbs: 16 k 0.92 .. 1.09x, 20 k 1.16x;
//          17 limbs 25 k 0.85 .. 1.01x, 33 k 1.05 .. 1.18x; 33 limbs 25 k 0.88 ..
//          0.98x, 33 k 1.08 .. 1.41x)
//   to     large batches fill the GPU level by level too, and from 15 limbs up
//          the register-resident kernels keep more products in flight than a
//          tile's share of shared memory does (12 limbs 1.5 M points 1.11x, 14 limbs
//          1.5 M 0.99x; 17 limbs 1 M 1.04x, 1.5 M 0.93x; 20 limbs 786 k 1.08x, 1 M
//          0.90x; 25 limbs 262 k 1.16x, 328 k 0.94x; 30 limbs 205 k 1.16x, 262 k 0.96x;
//          33 limbs 131 k 1.23x, 164 k 0.98x, 262 k 0.84x)
bool mp_tile_used(const MpDeviceTables &T, int L, int B) {
  if (!T.twp || L > kMaxLimbs || T.N < 16) return false;
  const long long w = (long long)T.N * B;
  const long long from = L <= 6 ? 8192 : L <= 9 ? (B < 8 ? 13000 : 12288) : L <= 12 ? 20000 : 28672;
  const long long to = L <= 14   ? (1LL << 62)
                       : L <= 18 ? 1200000
                       : L <= 21 ? 900000
                       : L <= 27 ? 300000
                       : L <= 30 ? 250000
                                 : 150000;
  return w >= from && w <= to;
}

cudaError_t mp_tile_run(int L, const MpDeviceTables &T, const uint32_t *in, uint32_t *out, int B, cudaStream_t s) {
#define MPFFT_TILE_CASE(LL) \
  case LL:                  \
    return tile_run<LL>(T, in, out, B, s);
  switch (L) {
    MPFFT_TILE_CASE(2) MPFFT_TILE_CASE(3) MPFFT_TILE_CASE(4) MPFFT_TILE_CASE(5) MPFFT_TILE_CASE(6)
    MPFFT_TILE_CASE(7) MPFFT_TILE_CASE(8) MPFFT_TILE_CASE(9) MPFFT_TILE_CASE(10) MPFFT_TILE_CASE(11)
    MPFFT_TILE_CASE(12) MPFFT_TILE_CASE(13) MPFFT_TILE_CASE(14) MPFFT_TILE_CASE(15) MPFFT_TILE_CASE(16)
    MPFFT_TILE_CASE(17) MPFFT_TILE_CASE(18) MPFFT_TILE_CASE(19) MPFFT_TILE_CASE(20) MPFFT_TILE_CASE(21)
    MPFFT_TILE_CASE(22) MPFFT_TILE_CASE(23) MPFFT_TILE_CASE(24) MPFFT_TILE_CASE(25) MPFFT_TILE_CASE(26)
    MPFFT_TILE_CASE(27) MPFFT_TILE_CASE(28) MPFFT_TILE_CASE(29) MPFFT_TILE_CASE(30) MPFFT_TILE_CASE(31)
    MPFFT_TILE_CASE(32) MPFFT_TILE_CASE(33) MPFFT_TILE_CASE(34)
    default:
      return cudaErrorInvalidValue;
  }
#undef MPFFT_TILE_CASE
}

}  // namespace mpfft

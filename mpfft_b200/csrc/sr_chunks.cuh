// The shape of the split-radix tree by output position, shared by the kernels
// that run several levels per pass.
//
// A node of size n (offset a multiple of n) has children of n/2 at its offset
// and of n/4 at +n/2 and +3n/4 (lab/parallel/mp/parallel_mp_fft2.c:180-182).
// So every aligned chunk of g positions, from the smallest size up, is either
// one node of size g or a pair of nodes of size g/2 (the two conjugate-pair
// children of one node of size 2g).  Walking the bits of the chunk's index m =
// offset/g from the top, a 0 bit steps into the first child and a 1 bit plus
// the bit after it into one of the other two; the chunk is a pair exactly when
// the walk ends on a lone 1, i.e. when m ends in an odd number of ones.
#pragma once

namespace mpfft {

// chunk m of any granularity is one node (else a pair of nodes of half its size)
__host__ __device__ inline bool sr_chunk_big(unsigned m) {
#ifdef __CUDA_ARCH__
  return (__ffs(~m) & 1) != 0;  // trailing ones + 1
#else
  return (__builtin_ctz(~m) & 1) == 0;
#endif
}

// Offset of the twiddles of node size n (n/4 of them, k = 0 .. n/4-1) in a
// table of all levels n = 32, 64, ..., N one after another: consecutive k of a
// level are consecutive entries, whatever N.
__host__ __device__ inline int sr_level_tw(int n) { return n / 4 - 8; }

}  // namespace mpfft

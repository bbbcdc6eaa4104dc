// Keccak-f[1600] on a lane pair, for sponges on the critical path of a latency-bound stage.
//
// Threads 2i and 2i+1 of a warp hold one state in bit-interleaved form: thread p keeps bit
// 2k + p of every 64-bit lane as bit k of a 32-bit word (25 registers).  A rotation by an
// even offset 2k is a 32-bit rotation by k on both threads; an odd offset 2k + 1 swaps the
// halves (even' = rot(odd, k + 1), odd' = rot(even, k)), one shuffle with the partner.  A
// round is 90 integer operations and 17 shuffles per thread instead of 180 operations on
// one thread.  Where a stage has one warp per SM sub-partition, a warp is bound by its own
// issue rate (the 16-lane integer pipe takes a warp instruction every two cycles), so
// halving the instructions per state shortens a sponge chain: 2.51 us a permutation against 4.55
// on one thread, at the same 135 integer operations a state.
//
// Sponge bytes (msponge.cuh's Multi<2>) cross the boundary through to_slice / half_to_slice (a
// 64-bit word, or the thread's half of it, into this thread's 32 bits) and from_slice (this thread's
// 32-bit half of the natural word: p = 0 the low half, p = 1 the high half).  Both are a byte permute and three delta swaps of an
// interleave / de-interleave of 32 bits.  Every thread of the warp must execute the
// shuffles: callers keep whole warps in step and predicate only memory accesses.
#pragma once
#include <cstdint>

#include "keccak.cuh"

namespace dpkem {
namespace kpair {

// Bit k of the result = bit 2k + p of w.
__host__ __device__ constexpr uint32_t slice_of(uint64_t w, int p) {
  uint32_t s = 0;
  for (int k = 0; k < 32; k++) s |= (uint32_t)((w >> (2 * k + p)) & 1u) << k;
  return s;
}

#define DPKEM_RCS(i) slice_of(kc::rc(i), 0), slice_of(kc::rc(i), 1)
__constant__ uint32_t c_rc_slice[48] = {
    DPKEM_RCS(0),  DPKEM_RCS(1),  DPKEM_RCS(2),  DPKEM_RCS(3),  DPKEM_RCS(4),  DPKEM_RCS(5),
    DPKEM_RCS(6),  DPKEM_RCS(7),  DPKEM_RCS(8),  DPKEM_RCS(9),  DPKEM_RCS(10), DPKEM_RCS(11),
    DPKEM_RCS(12), DPKEM_RCS(13), DPKEM_RCS(14), DPKEM_RCS(15), DPKEM_RCS(16), DPKEM_RCS(17),
    DPKEM_RCS(18), DPKEM_RCS(19), DPKEM_RCS(20), DPKEM_RCS(21), DPKEM_RCS(22), DPKEM_RCS(23)};
#undef DPKEM_RCS

__device__ __forceinline__ uint32_t partner(uint32_t x) { return __shfl_xor_sync(0xffffffffu, x, 1); }

// Lane rotation by R on this thread's slice; q = 1 - p.
template <int R>
__device__ __forceinline__ uint32_t rot(uint32_t own, uint32_t q) {
  if constexpr (R == 0) {
    return own;
  } else if constexpr (R % 2 == 0) {
    return __funnelshift_l(own, own, R / 2);
  } else {
    const uint32_t x = partner(own);
    return __funnelshift_l(x, x, R / 2 + q);
  }
}

__device__ __forceinline__ void round(uint32_t (&a)[25], uint32_t rc, uint32_t q) {
  uint32_t c[5], b[25];
#pragma unroll
  for (int x = 0; x < 5; x++) c[x] = a[x] ^ a[x + 5] ^ a[x + 10] ^ a[x + 15] ^ a[x + 20];
#pragma unroll
  for (int x = 0; x < 5; x++) {
    const uint32_t r = rot<1>(c[(x + 1) % 5], q), l = c[(x + 4) % 5];
#pragma unroll
    for (int y = 0; y < 5; y++) a[x + 5 * y] = lop3_xor3(a[x + 5 * y], l, r);
  }
#define DPKEM_RHOPI(i) b[kc::pi_dst(i)] = rot<kc::rho(i)>(a[i], q);
  DPKEM_RHOPI(0) DPKEM_RHOPI(1) DPKEM_RHOPI(2) DPKEM_RHOPI(3) DPKEM_RHOPI(4)
  DPKEM_RHOPI(5) DPKEM_RHOPI(6) DPKEM_RHOPI(7) DPKEM_RHOPI(8) DPKEM_RHOPI(9)
  DPKEM_RHOPI(10) DPKEM_RHOPI(11) DPKEM_RHOPI(12) DPKEM_RHOPI(13) DPKEM_RHOPI(14)
  DPKEM_RHOPI(15) DPKEM_RHOPI(16) DPKEM_RHOPI(17) DPKEM_RHOPI(18) DPKEM_RHOPI(19)
  DPKEM_RHOPI(20) DPKEM_RHOPI(21) DPKEM_RHOPI(22) DPKEM_RHOPI(23) DPKEM_RHOPI(24)
#undef DPKEM_RHOPI
#pragma unroll
  for (int y = 0; y < 5; y++)
#pragma unroll
    for (int x = 0; x < 5; x++)
      a[x + 5 * y] = b[x + 5 * y] ^ (~b[(x + 1) % 5 + 5 * y] & b[(x + 2) % 5 + 5 * y]);
  a[0] ^= rc;
}

// Four rounds per iteration: one warp per sub-partition waits for its own shuffles, and a longer
// body lets a round's first operations start among the previous round's last.  Measured us per
// permutation of a chain (512 states; 8,192): 1 round 2.99 (3.05), 2 2.67 (2.83), 4 2.51 (2.62), 8
// 2.47 (2.56; not measured in the stages, which inline several permutations), 24 4.01 (4.13: past the
// instruction cache).
__device__ __forceinline__ void f1600(uint32_t (&a)[25], int p) {
  const uint32_t q = 1u - (uint32_t)p;
#pragma unroll 4
  for (int r = 0; r < 24; r++) {
    const uint32_t e = c_rc_slice[2 * r], o = c_rc_slice[2 * r + 1];  // warp-uniform loads
    round(a, p ? o : e, q);
  }
}

// This thread's slice of the 64-bit word w = {lo, hi}: the p-bits of lo and hi are merged
// into one word (lo's at even positions, hi's at odd) and de-interleaved.
__device__ __forceinline__ uint32_t to_slice(uint2 w, int p) {
  const uint32_t lo = w.x >> p, hi = w.y << (1 - p);
  uint32_t x = (lo & 0x55555555u) | (hi & 0xAAAAAAAAu), t;
  t = (x ^ (x >> 1)) & 0x22222222u;
  x ^= t ^ (t << 1);
  t = (x ^ (x >> 2)) & 0x0C0C0C0Cu;
  x ^= t ^ (t << 2);
  t = (x ^ (x >> 4)) & 0x00F000F0u;
  x ^= t ^ (t << 4);
  return __byte_perm(x, 0, 0x3120);
}

// The same from the 32-bit half p of the word, each thread having loaded its own: both
// de-interleave their halves and swap the 16 bits that belong to the other.
__device__ __forceinline__ uint32_t half_to_slice(uint32_t w, int p) {
  uint32_t x = w, t;
  t = (x ^ (x >> 1)) & 0x22222222u;
  x ^= t ^ (t << 1);
  t = (x ^ (x >> 2)) & 0x0C0C0C0Cu;
  x ^= t ^ (t << 2);
  t = (x ^ (x >> 4)) & 0x00F000F0u;
  x ^= t ^ (t << 4);
  x = __byte_perm(x, 0, 0x3120);
  const uint32_t y = partner(x);
  return p ? __byte_perm(y, x, 0x7632) : __byte_perm(x, y, 0x5410);
}

// This thread's 32-bit half of the natural word whose slices the pair holds (p = 0: bits
// 0-31, p = 1: bits 32-63).  Shuffles with the partner: every thread of the warp calls it.
__device__ __forceinline__ uint32_t from_slice(uint32_t own, int p) {
  const uint32_t other = partner(own);
  // bytes (even0, odd0, even1, odd1) for the low half, (even2, odd2, even3, odd3) for the high
  uint32_t x = __byte_perm(own, other, p ? 0x3726u : 0x5140u), t;
  t = (x ^ (x >> 4)) & 0x00F000F0u;
  x ^= t ^ (t << 4);
  t = (x ^ (x >> 2)) & 0x0C0C0C0Cu;
  x ^= t ^ (t << 2);
  t = (x ^ (x >> 1)) & 0x22222222u;
  x ^= t ^ (t << 1);
  return x;
}

}  // namespace kpair
}  // namespace dpkem

// Keccak-f[1600] with one state on ten lanes of a warp, three states per warp: for sponge
// chains whose batch leaves the integer pipe idle but holds more states than warps.
//
// Thread (x, p) of a state holds column x of its bit-interleaved half p: bit 2k + p of lane
// (x, y) is bit k of the 32-bit word a[y] (keccak_pair.cuh's slices).  Rotations are then 32-bit
// rotations, an odd offset also changing the half, and each move of a round is one shuffle or
// one store per word:
//   theta  own column's parity (local), C[x-1] from (x-1, p), rot(C[x+1], 1) from (x+1, 1-p):
//          two shuffles; the even half's word needs a rotation by one
//   rho    five rotations by per-thread amounts (an odd offset's two halves rotate differently)
//   pi     into rows: row thread (y', p') takes slot s from column thread (3y' + s mod 5), whose
//          half is p' or, for an odd offset, 1 - p': five shuffles, slots static
//   chi    local on the row; iota on row 0
//   back   rows -> columns through shared memory: five 4-byte stores, a 16-byte and a 4-byte load
// 20 integer instructions, 7 shuffles and 7 shared-memory accesses per thread and round.
//
// What bounds it: shuffles and shared-memory accesses share one pipe per SM (a warp access per
// cycle), so the layouts differ by those: 18 per state and round on a warp per state
// (keccak25.cuh), 24 / 6 on five lanes with 64-bit words, here 18 cycles per 3 states once no access has a bank
// conflict.  Hence the buffer's shape: slot s of all six (state, half) pairs c is one line of
// 208 bytes, rows 0..3 at 16 c, row 4 at 96 + 4 c.  The stores of a slot then hit 30 different banks,
// and the 208-byte stride (13 x 16) puts the eight 16-byte loads of every quarter warp on
// different banks too.  Measured, us per permutation of a dependent chain (dpkem_probe_keccak_chain; a warp per
// state / five lanes / pair / here): 6 states 2.02 / 3.07 / 2.50 / 1.91, 1,024 2.27 / 3.08 / 2.51 / 1.95, 2,048
// 4.11 / 3.26 / 2.51 / 2.01, 4,096 6.69 / 3.92 / 2.53 / 2.54, 8,192 13.4 / 6.28 / 2.62 / 4.87.
//
// Lanes 30 and 31 repeat lanes 0 and 1 (the same loads, stores of the same words); callers drop their
// writes to global memory.  Every lane of the warp must execute every call.
#pragma once
#include <cstdint>

#include "keccak.cuh"
#include "keccak_pair.cuh"

namespace dpkem {
namespace k10 {

constexpr int kLine = 208;
constexpr int kSmemPerWarp = 5 * kLine;

struct Lanes {
  int x, p, g;            // column, half, state of the warp
  int left, right, mate;  // lanes of (x-1, p), (x+1, 1-p) and (x, 1-p)
  int src[5];             // pi: source lane of row slot s
  uint32_t rot[5];        // this half's rotation of slot y
  uint32_t rl;            // 1 on the even half (theta's rotation of C[x+1])
  uint32_t iota;          // all-ones on row 0
  uint32_t st, ld4, ld1;  // shared-window addresses: this row's store of slot 0, this column's loads
};

__device__ __forceinline__ Lanes make_lanes(uint8_t *warp_smem) {
  Lanes k;
  const int lane = (threadIdx.x & 31) % 30;
  k.g = lane / 10;
  const int t = lane - 10 * k.g, base = 10 * k.g;
  k.p = t / 5;
  k.x = t - 5 * k.p;
  k.left = base + (k.x + 4) % 5 + 5 * k.p;
  k.right = base + (k.x + 1) % 5 + 5 * (1 - k.p);
  k.mate = base + k.x + 5 * (1 - k.p);
#pragma unroll
  for (int y = 0; y < 5; y++) {
    int r = 0, ro = 0;  // rho of this column's slot y, and of the lane pi brings to row x, slot y
    const int xs = (3 * k.x + y) % 5;
#pragma unroll
    for (int c = 0; c < 5; c++) {
      if (c == k.x) r = kc::rho(c + 5 * y);
      if (c == xs) ro = kc::rho(c + 5 * y);
    }
    k.rot[y] = (uint32_t)((r & 1) ? (k.p ? (r + 1) / 2 : r / 2) : r / 2);
    k.src[y] = base + xs + 5 * (k.p ^ (ro & 1));
  }
  k.rl = 1u - (uint32_t)k.p;
  k.iota = k.x == 0 ? 0xFFFFFFFFu : 0u;
  const uint32_t b = static_cast<uint32_t>(__cvta_generic_to_shared(warp_smem)), c = 2 * k.g + k.p;
  k.st = b + (k.x < 4 ? 16 * c + 4 * k.x : 96 + 4 * c);
  k.ld4 = b + kLine * k.x + 16 * c;
  k.ld1 = b + kLine * k.x + 96 + 4 * c;
  return k;
}

__device__ __forceinline__ void round10(uint32_t (&a)[5], const Lanes &k, uint32_t rc) {
  const uint32_t c = lop3_xor3(lop3_xor3(a[0], a[1], a[2]), a[3], a[4]);
  uint32_t cr = __shfl_sync(0xffffffffu, c, k.right);
  const uint32_t cl = __shfl_sync(0xffffffffu, c, k.left);
  cr = __funnelshift_l(cr, cr, k.rl);
  uint32_t b[5];
#pragma unroll
  for (int y = 0; y < 5; y++) {
    const uint32_t v = lop3_xor3(a[y], cl, cr);
    a[y] = __funnelshift_l(v, v, k.rot[y]);
  }
#pragma unroll
  for (int s = 0; s < 5; s++) b[s] = __shfl_sync(0xffffffffu, a[s], k.src[s]);
#pragma unroll
  for (int s = 0; s < 5; s++) {
    uint32_t v = b[s] ^ (~b[(s + 1) % 5] & b[(s + 2) % 5]);
    if (s == 0) v ^= rc & k.iota;
    asm volatile("st.shared.u32 [%0], %1;" ::"r"(k.st + kLine * s), "r"(v) : "memory");
  }
  __syncwarp();
  asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];"
               : "=r"(a[0]), "=r"(a[1]), "=r"(a[2]), "=r"(a[3])
               : "r"(k.ld4)
               : "memory");
  asm volatile("ld.shared.u32 %0, [%1];" : "=r"(a[4]) : "r"(k.ld1) : "memory");
  // The next stores follow the next round's shuffles, which no lane passes before every
  // lane's loads above have returned (the shuffled values depend on them).
}

// U rounds per iteration (us per permutation of a chain, 512 / 4,096 states: 1 round 2.26 / 3.05, 2 2.07 / 3.03,
// 4 2.06 / 2.93, 8 2.02 / 2.91, 24 1.92 / 2.55).  Eight where a stage inlines several permutations (24
// rounds of each would not stay in the instruction cache), 24 where it has one.
template <int U = 8>
__device__ __forceinline__ void f1600(uint32_t (&a)[5], const Lanes &k) {
#pragma unroll U
  for (int r = 0; r < 24; r++) {
    const uint32_t e = kpair::c_rc_slice[2 * r], o = kpair::c_rc_slice[2 * r + 1];
    round10(a, k, k.p ? o : e);
  }
}

// Bits of w: the even ones to the low 16, the odd ones to the high 16; and back.
__device__ __forceinline__ uint32_t unzip(uint32_t w) {
  uint32_t x = w, t;
  t = (x ^ (x >> 1)) & 0x22222222u;
  x ^= t ^ (t << 1);
  t = (x ^ (x >> 2)) & 0x0C0C0C0Cu;
  x ^= t ^ (t << 2);
  t = (x ^ (x >> 4)) & 0x00F000F0u;
  x ^= t ^ (t << 4);
  return __byte_perm(x, 0, 0x3120);
}
// From bytes (even, odd, even, odd) of the two halves' 16 bits.
__device__ __forceinline__ uint32_t zip_bytes(uint32_t x) {
  uint32_t t;
  t = (x ^ (x >> 4)) & 0x00F000F0u;
  x ^= t ^ (t << 4);
  t = (x ^ (x >> 2)) & 0x0C0C0C0Cu;
  x ^= t ^ (t << 2);
  t = (x ^ (x >> 1)) & 0x22222222u;
  x ^= t ^ (t << 1);
  return x;
}

// This half of a lane from its 32-bit half word w (p = 0: bits 0-31, p = 1: bits 32-63): both
// threads de-interleave their words and swap the 16 bits that belong to the other.
__device__ __forceinline__ uint32_t to_slice(uint32_t w, const Lanes &k) {
  const uint32_t x = unzip(w), y = __shfl_sync(0xffffffffu, x, k.mate);
  return k.p ? __byte_perm(y, x, 0x7632) : __byte_perm(x, y, 0x5410);
}

// The reverse: this thread's 32-bit half word of the lane whose halves the two threads hold.
__device__ __forceinline__ uint32_t from_slice(uint32_t own, const Lanes &k) {
  const uint32_t other = __shfl_sync(0xffffffffu, own, k.mate);
  return zip_bytes(__byte_perm(own, other, k.p ? 0x3726u : 0x5140u));
}

// A whole lane {lo, hi} from its halves {even, odd} on one thread, and back.
__device__ __forceinline__ uint2 lane_of(uint2 s) {
  return make_uint2(zip_bytes(__byte_perm(s.x, s.y, 0x5140)), zip_bytes(__byte_perm(s.x, s.y, 0x7362)));
}
__device__ __forceinline__ uint2 slices_of(uint2 w) {
  const uint32_t l = unzip(w.x), h = unzip(w.y);
  return make_uint2(__byte_perm(l, h, 0x5410), __byte_perm(l, h, 0x7632));
}

}  // namespace k10
}  // namespace dpkem

// FrodoKEM prologue chains on ten lanes per state: the dependent permutations of the sponges on a warp
// of their own, everything else on a helper warp.  Used by the batched kernels (frodo_ahead.cuh)
// and the planned mixed batches (mixed_dev.cuh).
#pragma once
#include "frodo_dev.cuh"

namespace dpkem {
namespace fchain {

using namespace frodo;
using fdev::Inst;

constexpr int HALF = N * NBAR;  // S' (S^T) words; E' (E) follows in the stream

// A prologue's dependent permutations on a warp of their own, three instances on ten lanes each
// (keccak10.cuh); a second warp does all else: it fetches, pads and de-interleaves the next
// message block and samples the previous squeezed one, exchanged through shared memory as
// bit-interleaved halves {even, odd}, one barrier of the two warps per step.  The chain warp's
// loop is one unrolled permutation, four loads and four stores per thread: 2.05 us a step,
// against 2.32 with conversions and sampling in line.
//
// Steps of a chain: A blocks absorbed from a zero state; then per further hash (its message needs
// the previous one's output) an idle step, in which the helper forms the message, and an
// absorbing step from a zero state; then squeezing steps.
//   encaps   A = 115 (H(pk)), G2, seed          keypair  A = 1 (seed)
//   decaps, encaps with H(pk) at hand   A = 1 (G2), seed
// Insts: src(i) is instance i of src.n.
struct Exchange {
  uint2 msg[2][3][17], raw[2][3][17];
};
enum Role : int { R_KEYPAIR, R_ENC, R_ENC_PKH, R_DEC };

template <int ROLE>
struct Steps {
  static constexpr int A = ROLE == R_ENC ? 115 : 1;
  static constexpr int K = ROLE == R_ENC ? 2 : ROLE == R_KEYPAIR ? 0 : 1;  // hashes after the first
  static constexpr int op = ROLE == R_KEYPAIR ? OP_KEYPAIR : ROLE == R_DEC ? OP_DEC : OP_ENC;
  // step after which squeezed block 0 is there
  static constexpr int FIRST = A + 2 * K - 1;
};
static_assert(PK / 136 + 1 == 115, "absorbed blocks");

// Barrier of chain warp w and its helper.  A barrier number in a register makes the kernel
// reserve all 16 (four blocks per SM); with two chain warps the numbers are constants.
template <bool TWO>
__device__ __forceinline__ void pair_sync(int w) {
  if (!TWO) asm volatile("bar.sync %0, 64;" ::"r"(1 + w) : "memory");
  else if (w) asm volatile("bar.sync 2, 64;" ::: "memory");
  else asm volatile("bar.sync 1, 64;" ::: "memory");
}

template <int ROLE, bool TWO, class Insts>
__device__ __forceinline__ void chain_warp(const Insts &src, int first, int squeezes, bool keep, Exchange &x,
                                           uint8_t *xbuf, int bar) {
  using T = Steps<ROLE>;
  using S = msp::Multi<10>;
  const S s(xbuf);
  const int g = s.state();
  uint32_t a[5];
  msp::zero<S>(a);
  const int steps = T::FIRST + 1 + squeezes;
  for (int t = 0; t < steps; t++) {
    pair_sync<TWO>(bar);
    const int u = t - T::A;
    const bool later = u >= 0 && u < 2 * T::K;
    if (later && !(u & 1)) continue;
    if (later) msp::zero<S>(a);
    if (t <= T::FIRST) {
#pragma unroll
      for (int y = 0; y < 4; y++)
        if (s.lane(y) < 17) a[y] ^= s.load(reinterpret_cast<const uint8_t *>(&x.msg[t & 1][g][s.lane(y)]));
    }
    k10::f1600<24>(a, s.k);
#pragma unroll
    for (int y = 0; y < 4; y++)
      if (s.lane(y) < 17) s.store(reinterpret_cast<uint8_t *>(&x.raw[t & 1][g][s.lane(y)]), a[y]);
  }
  pair_sync<TWO>(bar);
  if (keep) {
    const int i = first + g;
    const bool live = i < src.n;
    fdev::save_state_multi<S>(a, s, src(live ? i : src.n - 1).hs, live);
  }
}

// Lane q of block t of the first hash's message, padding included.
template <int ROLE>
__device__ __forceinline__ uint2 first_message(const Inst &v, int t, int q) {
  constexpr uint32_t kEnd = 0x80000000u;
  if (ROLE == R_ENC) {  // pk: 1,954 lanes
    const int m = 17 * t + q;
    return m < PK / 8 ? ld_lane(v.pk + 8 * m) : make_uint2(0x1Fu, kEnd);
  }
  if (ROLE == R_DEC || ROLE == R_ENC_PKH) {  // pkh || mu
    if (q < 3) return ld_lane((ROLE == R_DEC ? v.sk + SK_PKH : v.pkh) + 8 * q);
    if (q < 6) return ld_lane((ROLE == R_DEC ? v.mu : v.coins) + 8 * (q - 3));
    return make_uint2(q == 6 ? 0x1Fu : 0u, q == 16 ? kEnd : 0u);
  }
  return make_uint2(0u, 0u);  // keypair: see seed_message
}
static_assert(PK / 8 == 114 * 17 + 16, "H(pk)'s padding fills lane 16 of the last block");

// Lane q of dom || seed (25 bytes) with its padding; lane(j) yields lane j of the seed.
template <class F>
__device__ __forceinline__ uint2 seed_message(uint32_t dom, int q, F lane) {
  if (q > 3) return make_uint2(0u, q == 16 ? 0x80000000u : 0u);
  const uint2 z = make_uint2(0u, 0u), p = q > 0 ? lane(q - 1) : z, c = q < 3 ? lane(q) : z;
  uint2 w = msp::Multi<1>::shl8(p, c);
  if (q == 0) w.x |= dom;
  if (q == 3) w.x |= 0x1Fu << 8;  // byte 25
  return w;
}

template <int ROLE, bool TWO, class Insts>
__device__ __forceinline__ void helper_warp(const Insts &src, int first, int words, Exchange &x, int bar) {
  using T = Steps<ROLE>;
  const int lane = threadIdx.x & 31;
  // lanes of the block, three instances: f(instance, slot, lane q)
  auto each = [&](auto f) {
#pragma unroll 1
    for (int e = lane; e < 51; e += 32) {
      const int g = e / 17, i = first + g;
      f(src(i < src.n ? i : src.n - 1), g, e - 17 * g, i < src.n);
    }
  };
  // message of step t (t - 1 has finished when it depends on that)
  auto prepare = [&](int t) {
    each([&](const Inst &v, int g, int q, bool) {
      uint2 w;
      auto out = [&](int j) { return k10::lane_of(x.raw[t & 1][g][j]); };  // step t - 2's lanes
      if (ROLE == R_KEYPAIR) {
        w = seed_message(0x5Fu, q, [&](int j) { return ld_lane(v.coins + 24 + 8 * j); });
      } else if (t < T::A) {
        w = first_message<ROLE>(v, t, q);
      } else if (ROLE == R_ENC && t == T::A + 1) {  // G2: pkh || mu
        w = q < 3 ? out(q) : q < 6 ? ld_lane(v.coins + 8 * (q - 3)) : make_uint2(q == 6 ? 0x1Fu : 0u, q == 16 ? 0x80000000u : 0u);
      } else {  // 0x96 || seedSE
        w = seed_message(0x96u, q, out);
      }
      x.msg[t & 1][g][q] = k10::slices_of(w);
    });
  };
  // what step t left in raw[t & 1]
  auto consume = [&](int t) {
    const int blk = t - T::FIRST;
    if (blk < 0) {
      if (t != T::FIRST - 2 || ROLE == R_KEYPAIR) return;
      each([&](const Inst &v, int g, int q, bool live) {  // G2's lanes 3..5 = k
        if (q >= 3 && q < 6 && live) *reinterpret_cast<uint2 *>(v.kk + 8 * (q - 3)) = k10::lane_of(x.raw[t & 1][g][q]);
      });
      return;
    }
    each([&](const Inst &v, int g, int q, bool live) {
      const int w = 68 * blk + 4 * q;
      const uint2 r = fdev::sample_lane(k10::lane_of(x.raw[t & 1][g][q]));
      if (!live || w >= words) return;
      *reinterpret_cast<uint2 *>(v.rw + w) = r;
      if (ROLE == R_KEYPAIR && w < HALF) *reinterpret_cast<uint2 *>(v.sk + SK_S + 2 * w) = r;
    });
  };
  if (ROLE == R_KEYPAIR)
    each([&](const Inst &v, int, int q, bool live) {  // s, and seedA from pk (kp_seed_kernel)
      if (!live || q >= 5) return;
      *reinterpret_cast<uint2 *>(v.sk + 8 * q) = q < 3 ? ld_lane(v.coins + 8 * q) : ld_lane(v.pk + 8 * (q - 3));
    });
  prepare(0);
  const int steps = T::FIRST + 1 + max(0, (words + 67) / 68 - 1);
  for (int t = 0; t < steps; t++) {
    pair_sync<TWO>(bar);
    if (t > 0) consume(t - 1);
    const int u = t + 1;
    if (u < T::A || (u <= T::FIRST && ((u - T::A) & 1))) {
      __syncwarp();
      prepare(u);
    }
  }
  pair_sync<TWO>(bar);
  consume(steps - 1);
}

// seedA = SHAKE256(z, 16) into pk, which a keypair's chain and A need (one thread).
__device__ __forceinline__ void write_seed_a(const Inst &v) {
  uint2 a[25];
  keccak_zero(a);
  a[0] = ld_lane(v.coins + 48);
  a[1] = ld_lane(v.coins + 56);
  absorb_finish<136>(a, 16, 0x1Fu);
  *reinterpret_cast<uint2 *>(v.pk) = a[0];
  *reinterpret_cast<uint2 *>(v.pk + 8) = a[1];
}

}  // namespace fchain
}  // namespace dpkem

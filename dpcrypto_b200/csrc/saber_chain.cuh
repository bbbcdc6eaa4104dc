// Saber prologue and finish sponges on ten lanes per state (keccak10.cuh) with the dependent
// permutations on a warp of their own: a helper warp fetches, pads and de-interleaves the message blocks
// and stores what is squeezed (the scheme of frodo_chain.cuh).  The chain warp's code is one
// unrolled permutation for both of a prologue's sponges, which differ in their programs: which
// steps absorb a message block, which start from a zero state, which idle (the helper then
// forms a message from the previous step's output).
//
// us, prologue of encaps, a warp per state / ten lanes with conversions in line / here: l = 3, one
// instance 56 / 60 / 52, 1,024 105 / 68 / 57; l = 4, 1,536 251 / 107 / 98.
#pragma once
#include "saber_dev.cuh"

namespace dpkem {
namespace schain {

using sdev::Inst;
using sdev::Scr;
using sdev::SP;

constexpr int LANES = 21;  // SHAKE128's rate, the largest

struct Exchange {
  uint2 msg[2][3][LANES], raw[2][3][LANES], keep[3][4];
};
static_assert(sizeof(Exchange) % 16 == 0, "16-byte aligned transpose buffers");

// Bit t: step t absorbs msg / starts from zero / idles.
struct Program {
  int steps;
  uint64_t msg, reset, idle;
};

// Barrier of chain w and its helper (constant numbers: see fchain::pair_sync).
__device__ __forceinline__ void pair_sync(int w) {
  if (w) asm volatile("bar.sync 2, 64;" ::: "memory");
  else asm volatile("bar.sync 1, 64;" ::: "memory");
}

__device__ __forceinline__ void chain_warp(Program p, Exchange &x, uint8_t *xbuf, int w) {
  using S = msp::Multi<10>;
  const S s(xbuf);
  const int g = s.state();
  uint32_t a[5];
  msp::zero<S>(a);
  for (int t = 0; t < p.steps; t++) {
    pair_sync(w);
    if ((p.idle >> t) & 1) continue;
    if ((p.reset >> t) & 1) msp::zero<S>(a);
    if ((p.msg >> t) & 1) {
#pragma unroll
      for (int y = 0; y < 5; y++)
        if (s.lane(y) < LANES) a[y] ^= s.load(reinterpret_cast<const uint8_t *>(&x.msg[t & 1][g][s.lane(y)]));
    }
    k10::f1600<24>(a, s.k);
#pragma unroll
    for (int y = 0; y < 5; y++)
      if (s.lane(y) < LANES) s.store(reinterpret_cast<uint8_t *>(&x.raw[t & 1][g][s.lane(y)]), a[y]);
  }
  pair_sync(w);
}

// Lane q of a block: `lane` while q < len, then the padding of a message that ends there (dom),
// zero past the rate.
__device__ __forceinline__ uint2 padded(uint2 lane, int q, int len, int rate, uint32_t dom) {
  if (q < len) return lane;
  return make_uint2(q == len ? dom : 0u, q == rate - 1 ? 0x80000000u : 0u);
}
// Lane q of block t of SHA3-256 over n lanes at p.
__device__ __forceinline__ uint2 sha3_block(const uint8_t *p, int n, int t, int q) {
  const int m = 17 * t + q;
  if (q >= 17) return make_uint2(0u, 0u);
  return m < n ? ld_lane(p + 8 * m) : padded(make_uint2(0u, 0u), m, n, 17 * (n / 17 + 1), 0x06u);
}

// ---- what a helper does per step: message(t, v, q, out) is lane q of step t's message, out(j) lane j of
// the previous absorbing step's output; consume(t, v, q, w, live) gets lane q of step t's output.
__host__ __device__ constexpr int blocks(int bytes, int rate) { return (bytes + rate - 1) / rate; }
__host__ __device__ constexpr uint64_t ones(int n) { return n >= 64 ? ~0ull : (1ull << n) - 1; }

__device__ __forceinline__ void put(uint8_t *p, uint2 w) { *reinterpret_cast<uint2 *>(p) = w; }

// Squeezed block t of `len` bytes at dst.
__device__ __forceinline__ void put_block(uint8_t *dst, int t, int len, int q, uint2 w) {
  const int off = 168 * t + 8 * q;
  if (off < len) put(dst + off, w);
}

// GenMatrix (role 1).
template <int L, int OP>
struct Matrix {
  using P = SP<L>;
  static constexpr int NB = blocks(P::ARAW, 168), A = OP == OP_KEYPAIR ? 2 : 0;  // seed_A first: SHAKE128(coins)
  static constexpr Program prog = {A + NB, A ? 0b101ull : 1ull, A ? 0b100ull : 0ull, A ? 0b010ull : 0ull};
  template <class Out>
  __device__ __forceinline__ static uint2 message(int t, const Inst &v, int q, Out out, const uint2 *) {
    uint2 w = make_uint2(0u, 0u);
    if (q < 4) {
      if (OP == OP_KEYPAIR) w = t == 0 ? ld_lane(v.coins + 8 * q) : out(q);
      else w = ld_lane((OP == OP_ENC ? v.pk + P::POLYVECCOMP : v.sk + P::POLYVEC + P::POLYVECCOMP) + 8 * q);
    }
    return padded(w, q, 4, 21, 0x1Fu);
  }
  __device__ __forceinline__ static void consume(int t, const Inst &v, int q, uint2 w, uint2 *) {
    if (A && t == 0 && q < 4) put(v.pk + P::POLYVECCOMP + 8 * q, w);
    if (t >= A) put_block(v.scr + Scr<L>::ARAW, t - A, P::ARAW, q, w);
  }
};

// The hash chain and GenSecret (role 0).
template <int L, int OP>
struct Secret;

template <int L>
struct Secret<L, OP_KEYPAIR> {
  using P = SP<L>;
  static constexpr Program prog = {blocks(P::SRAW, 168), 1, 0, 0};
  template <class Out>
  __device__ __forceinline__ static uint2 message(int, const Inst &v, int q, Out, const uint2 *) {
    return padded(q < 4 ? ld_lane(v.coins + 32 + 8 * q) : make_uint2(0u, 0u), q, 4, 21, 0x1Fu);
  }
  __device__ __forceinline__ static void consume(int t, const Inst &v, int q, uint2 w, uint2 *) {
    put_block(v.scr + Scr<L>::SRAW, t, P::SRAW, q, w);
  }
};

// H(pk) in HP blocks, m = SHA3-256(coins), kr = SHA3-512(m || H(pk)), GenSecret from kr[32:64].
template <int L>
struct Secret<L, OP_ENC> {
  using P = SP<L>;
  static constexpr int HP = P::PK / 8 / 17 + 1, KR = HP + 2, GS = HP + 4;
  static constexpr Program prog = {GS + blocks(P::SRAW, 168), ones(HP + 1) | (1ull << KR) | (1ull << GS),
                                   (1ull << HP) | (1ull << KR) | (1ull << GS), (1ull << (HP + 1)) | (1ull << (HP + 3))};
  template <class Out>
  __device__ __forceinline__ static uint2 message(int t, const Inst &v, int q, Out out, const uint2 *keep) {
    const uint2 z = make_uint2(0u, 0u);
    if (t < HP) return sha3_block(v.pk, P::PK / 8, t, q);
    if (t == HP) return padded(q < 4 ? ld_lane(v.coins + 8 * q) : z, q, 4, 17, 0x06u);
    if (t == KR) return padded(q < 4 ? out(q) : q < 8 ? keep[q - 4] : z, q, 8, 9, 0x06u);
    return padded(q < 4 ? out(4 + q) : z, q, 4, 21, 0x1Fu);
  }
  __device__ __forceinline__ static void consume(int t, const Inst &v, int q, uint2 w, uint2 *keep) {
    if (t == HP - 1 && q < 4) keep[q] = w;
    if (t == HP && q < 4) put(v.scr + Scr<L>::MTXT + 8 * q, w);
    if (t == KR && q < 8) put(v.scr + Scr<L>::KR + 8 * q, w);
    if (t >= GS) put_block(v.scr + Scr<L>::SRAW, t - GS, P::SRAW, q, w);
  }
};

// kr = SHA3-512(m' || H(pk)), GenSecret, then H(c) of the input ciphertext.
template <int L>
struct Secret<L, OP_DEC> {
  using P = SP<L>;
  static constexpr int GS = 2, HC = GS + blocks(P::SRAW, 168), HB = P::CT / 8 / 17 + 1;
  static constexpr Program prog = {HC + HB, 1ull | (1ull << GS) | (ones(HB) << HC), (1ull << GS) | (1ull << HC), 1ull << 1};
  template <class Out>
  __device__ __forceinline__ static uint2 message(int t, const Inst &v, int q, Out out, const uint2 *) {
    const uint2 z = make_uint2(0u, 0u);
    if (t == 0)
      return padded(q < 4 ? ld_lane(v.scr + Scr<L>::MTXT + 8 * q) : q < 8 ? ld_lane(v.sk + P::SK - 64 + 8 * (q - 4)) : z,
                    q, 8, 9, 0x06u);
    if (t == GS) return padded(q < 4 ? out(4 + q) : z, q, 4, 21, 0x1Fu);
    return sha3_block(v.ct, P::CT / 8, t - HC, q);
  }
  __device__ __forceinline__ static void consume(int t, const Inst &v, int q, uint2 w, uint2 *) {
    if (t == 0 && q < 8) put(v.scr + Scr<L>::KR + 8 * q, w);
    if (t >= GS && t < HC) put_block(v.scr + Scr<L>::SRAW, t - GS, P::SRAW, q, w);
    if (t == HC + HB - 1 && q < 4) put(v.scr + Scr<L>::HC + 8 * q, w);
  }
};

// Encaps finish: k = SHA3-256(kr[0:32] || SHA3-256(c)).  Keypair finish: SHA3-256(pk) into sk.
template <int L, int OP>
struct Finish {
  using P = SP<L>;
  static constexpr bool ENC = OP == OP_ENC;
  static constexpr int N = (ENC ? P::CT : P::PK) / 8, HB = N / 17 + 1, K = HB + 1;
  static constexpr Program prog = {ENC ? K + 1 : HB, ones(HB) | (ENC ? 1ull << K : 0), ENC ? 1ull << K : 0,
                                   ENC ? 1ull << HB : 0};
  template <class Out>
  __device__ __forceinline__ static uint2 message(int t, const Inst &v, int q, Out out, const uint2 *) {
    if (t < HB) return sha3_block(ENC ? v.ct : v.pk, N, t, q);
    const uint2 z = make_uint2(0u, 0u);
    return padded(q < 4 ? ld_lane(v.scr + Scr<L>::KR + 8 * q) : q < 8 ? out(q - 4) : z, q, 8, 17, 0x06u);
  }
  __device__ __forceinline__ static void consume(int t, const Inst &v, int q, uint2 w, uint2 *) {
    if (t == (ENC ? K : HB - 1) && q < 4) put((ENC ? v.ss : v.sk + P::SK - 64) + 8 * q, w);
  }
};

// The helper of three instances from `first` on; inst(i) is instance i of n.
template <class R, class Get>
__device__ __forceinline__ void helper_warp(Get inst, int n, int first, Exchange &x, int w) {
  const int lane = threadIdx.x & 31;
  constexpr Program p = R::prog;
  auto each = [&](auto f) {
#pragma unroll 1
    for (int e = lane; e < 3 * LANES; e += 32) {
      const int g = e / LANES, i = first + g;
      if (i < n) f(inst(i), g, e - LANES * g);
    }
  };
  auto prepare = [&](int t) {
    each([&](const Inst &v, int g, int q) {
      auto out = [&](int j) { return k10::lane_of(x.raw[t & 1][g][j]); };  // step t - 2 (t - 1 idled)
      x.msg[t & 1][g][q] = k10::slices_of(R::message(t, v, q, out, x.keep[g]));
    });
  };
  auto consume = [&](int t) {
    if ((p.idle >> t) & 1) return;
    each([&](const Inst &v, int g, int q) { R::consume(t, v, q, k10::lane_of(x.raw[t & 1][g][q]), x.keep[g]); });
    __syncwarp();
  };
  prepare(0);
  for (int t = 0; t < p.steps; t++) {
    pair_sync(w);
    if (t > 0) consume(t - 1);
    if (t + 1 < p.steps && ((p.msg >> (t + 1)) & 1)) prepare(t + 1);
  }
  pair_sync(w);
  consume(p.steps - 1);
}

}  // namespace schain
}  // namespace dpkem

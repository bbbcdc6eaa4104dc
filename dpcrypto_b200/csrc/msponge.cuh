// Sponge helpers over the multi-lane Keccak layouts, so that a stage body is written once for
// a warp per state (keccak25.cuh), ten lanes per state (keccak10.cuh, three states per warp) and
// a lane pair (keccak_pair.cuh, sixteen).
//
// A layout S gives each thread S::NS slots of the state (S::W a[S::NS]); slot y holds rate
// lane S::lane(y), at least S::least(y).  Memory holds natural words: load / store move this
// thread's part of a lane (all of it, or its 32-bit half), in / out convert a part to and from
// the layout's form (bit-interleaved halves: with a shuffle, so every thread of the warp calls
// them).  Every thread of the warp runs every call (the permutation shuffles); `live`
// predicates the global-memory accesses of a state without an instance, and S::writer() drops
// the duplicate lanes a layout keeps (the 25-lane form's threads 25..31, the ten-lane form's
// 30 and 31).
#pragma once
#include <cstdint>

#include "keccak.cuh"
#include "keccak10.cuh"
#include "keccak25.cuh"
#include "keccak_pair.cuh"

namespace dpkem {
namespace msp {

template <int NS>
struct Multi;

// A bit-interleaved layout's memory side: thread p of a state's two halves moves the 32-bit half p.
struct Halves {
  using W = uint32_t;
  // (cur << 8) | (prev >> 56) of the 64-bit lanes: four bits in each half
  __device__ static W shl8(W prev, W cur) { return (cur << 4) | (prev >> 28); }
};

// Ten lanes per state: thread (x, p) holds half p of lanes x, x + 5, ..., x + 20.
template <>
struct Multi<10> : Halves {
  static constexpr int NS = 5, STATES_PER_WARP = 3, SMEM_PER_WARP = k10::kSmemPerWarp;
  static constexpr bool FIXED = false;  // slot y holds lane y on every thread
  __host__ __device__ static constexpr int least(int y) { return 5 * y; }
  k10::Lanes k;
  __device__ explicit Multi(uint8_t *warp_smem) : k(k10::make_lanes(warp_smem)) {}
  __device__ int state() const { return k.g; }
  __device__ bool writer() const { return (threadIdx.x & 31) < 30; }
  __device__ int lane(int y) const { return k.x + 5 * y; }
  __device__ void perm(W (&a)[5]) const { k10::f1600(a, k); }
  __device__ W load(const uint8_t *p) const { return reinterpret_cast<const uint32_t *>(p)[k.p]; }
  __device__ void store(uint8_t *p, W w) const { reinterpret_cast<uint32_t *>(p)[k.p] = w; }
  __device__ W part(uint2 c) const { return k.p ? c.y : c.x; }
  __device__ W in(W w) const { return k10::to_slice(w, k); }
  __device__ W out(W w) const { return k10::from_slice(w, k); }
  template <int I>
  __device__ W get(const W (&a)[5]) const {
    return __shfl_sync(0xffffffffu, a[I / 5], 10 * k.g + I % 5 + 5 * k.p);
  }
};

// A lane pair: thread p holds half p of all 25 lanes.
template <>
struct Multi<2> : Halves {
  static constexpr int NS = 25, STATES_PER_WARP = 16, SMEM_PER_WARP = 0;
  static constexpr bool FIXED = true;
  __host__ __device__ static constexpr int least(int y) { return y; }
  __device__ explicit Multi(uint8_t *) {}
  __device__ static int p() { return threadIdx.x & 1; }
  __device__ int state() const { return (threadIdx.x & 31) >> 1; }
  __device__ bool writer() const { return true; }
  __device__ int lane(int y) const { return y; }
  __device__ void perm(W (&a)[25]) const { kpair::f1600(a, p()); }
  __device__ W load(const uint8_t *q) const { return reinterpret_cast<const uint32_t *>(q)[p()]; }
  __device__ void store(uint8_t *q, W w) const { reinterpret_cast<uint32_t *>(q)[p()] = w; }
  __device__ W part(uint2 c) const { return p() ? c.y : c.x; }
  __device__ W in(W w) const { return kpair::half_to_slice(w, p()); }
  __device__ W out(W w) const { return kpair::from_slice(w, p()); }
  template <int I>
  __device__ W get(const W (&a)[25]) const {
    return a[I];
  }
};

// A warp per state: thread i holds lane i (threads 25..31 a copy of lane i - 25).
template <>
struct Multi<1> {
  using W = uint2;
  static constexpr int NS = 1, STATES_PER_WARP = 1, SMEM_PER_WARP = 0;
  static constexpr bool FIXED = false;
  __host__ __device__ static constexpr int least(int) { return 0; }
  k25::Lane k;
  __device__ explicit Multi(uint8_t *) : k(k25::make_lane()) {}
  __device__ int state() const { return 0; }
  __device__ bool writer() const { return (threadIdx.x & 31) < 25; }
  __device__ int lane(int) const { return k.i; }
  __device__ void perm(W (&a)[1]) const { k25::f1600(a[0], k); }
  __device__ W load(const uint8_t *p) const { return ld_lane(p); }
  __device__ void store(uint8_t *p, W w) const { *reinterpret_cast<uint2 *>(p) = w; }
  __device__ W part(uint2 c) const { return c; }
  __device__ W in(W w) const { return w; }
  __device__ W out(W w) const { return w; }
  __device__ static W shl8(W prev, W cur) {
    return make_uint2((cur.x << 8) | (prev.y >> 24), __funnelshift_l(cur.x, cur.y, 8));
  }
  template <int I>
  __device__ W get(const W (&a)[1]) const {
    return k5::shfl(a[0], I);
  }
};

__device__ __forceinline__ void fold(uint2 &a, uint2 w) {
  a.x ^= w.x;
  a.y ^= w.y;
}
__device__ __forceinline__ void fold(uint32_t &a, uint32_t w) { a ^= w; }
__device__ __forceinline__ void clear(uint2 &a) { a = make_uint2(0u, 0u); }
__device__ __forceinline__ void clear(uint32_t &a) { a = 0u; }
// Keeps a converted word from being computed inside the branch that stores it: a block's
// conversions then overlap instead of following one another (each is a chain of about 15
// dependent instructions).
__device__ __forceinline__ void pin(uint2 &a) { asm volatile("" : "+r"(a.x), "+r"(a.y)); }
__device__ __forceinline__ void pin(uint32_t &a) { asm volatile("" : "+r"(a)); }
template <class W>
__device__ __forceinline__ W none() {
  W w;
  clear(w);
  return w;
}

template <class S>
__device__ __forceinline__ void zero(typename S::W (&a)[S::NS]) {
#pragma unroll
  for (int y = 0; y < S::NS; y++) clear(a[y]);
}

// Keep lanes 0 .. n-1, clear the rest.
template <class S>
__device__ __forceinline__ void keep(typename S::W (&a)[S::NS], const S &s, int n) {
#pragma unroll
  for (int y = 0; y < S::NS; y++)
    if (s.lane(y) >= n) clear(a[y]);
}

// XOR w (in the layout's form) into lane I (the owner's copy of w is the one used).
template <class S, int I>
__device__ __forceinline__ void xor_lane(typename S::W (&a)[S::NS], const S &s, typename S::W w) {
#pragma unroll
  for (int y = 0; y < S::NS; y++)
    if (S::least(y) <= I && s.lane(y) == I) fold(a[y], w);
}

// Lanes 0..3 of a finished state `src` moved (XORed) into lanes D..D+3 of `dst`.
template <class S, int D>
__device__ __forceinline__ void move4(typename S::W (&dst)[S::NS], const typename S::W (&src)[S::NS], const S &s) {
  xor_lane<S, D + 0>(dst, s, s.template get<0>(src));
  xor_lane<S, D + 1>(dst, s, s.template get<1>(src));
  xor_lane<S, D + 2>(dst, s, s.template get<2>(src));
  xor_lane<S, D + 3>(dst, s, s.template get<3>(src));
}

// Absorb whole 8-byte words (len % 8 == 0, p 8-byte aligned) at fill `pos` (a multiple of
// 8); returns the new fill.
// Whole blocks at fill 0 load the next block's words before permuting the current one, so the
// global-load latency passes during the permutation.
template <class S, int RATE>
__device__ __forceinline__ int absorb_aligned(typename S::W (&a)[S::NS], const S &s, int pos, const uint8_t *p, int len,
                                              bool live) {
  using T = typename S::W;
  constexpr int W = RATE / 8;
  if (pos == 0 && len >= RATE) {
    T w[S::NS];
#pragma unroll
    for (int y = 0; y < S::NS; y++) {
      const int q = s.lane(y);
      w[y] = (q < W && live) ? s.load(p + 8 * q) : none<T>();
    }
    while (true) {
#pragma unroll
      for (int y = 0; y < S::NS; y++)
        if (S::least(y) < W) fold(a[y], s.in(w[y]));
      p += RATE;
      len -= RATE;
      const bool more = len >= RATE;
      if (more) {
#pragma unroll
        for (int y = 0; y < S::NS; y++) {
          const int q = s.lane(y);
          if (q < W && live) w[y] = s.load(p + 8 * q);
        }
      }
      s.perm(a);
      if (!more) break;
    }
  }
  while (len > 0) {
    const int take = min(len, RATE - pos);
    const int q0 = pos / 8, nq = take / 8;
#pragma unroll
    for (int y = 0; y < S::NS; y++) {
      if (S::least(y) >= W || (S::FIXED && (y < q0 || y >= q0 + nq))) continue;
      const int q = s.lane(y);
      fold(a[y], s.in((q < W && q >= q0 && q < q0 + nq && live) ? s.load(p + 8 * (q - q0)) : none<T>()));
    }
    pos += take;
    p += take;
    len -= take;
    if (pos == RATE) {
      s.perm(a);
      pos = 0;
    }
  }
  return pos;
}

// Padding (domain byte at `pos`, 0x80 in the last rate byte), then the permutation.
template <class S, int RATE>
__device__ __forceinline__ void absorb_finish(typename S::W (&a)[S::NS], const S &s, int pos, uint32_t domain) {
  const int qd = pos / 8, sh = 8 * (pos % 8), ql = RATE / 8 - 1;
  const typename S::W d = s.in(s.part(sh < 32 ? make_uint2(domain << sh, 0u) : make_uint2(0u, domain << (sh - 32))));
  const typename S::W e = s.in(s.part(make_uint2(0u, 0x80000000u)));
#pragma unroll
  for (int y = 0; y < S::NS; y++) {
    if (S::least(y) > ql) continue;
    const int q = s.lane(y);
    if (q == qd) fold(a[y], d);
    if (q == ql) fold(a[y], e);
  }
  s.perm(a);
}

// Squeeze `len` bytes (a multiple of 8) of a finished state to dst.  RAW: each 64-bit word in the
// layout's form, which a bit-interleaved layout stores as its halves {even, odd} (k10::lane_of
// restores it), sparing the chain the conversions.
template <class S, int RATE, bool RAW = false>
__device__ __forceinline__ void squeeze(typename S::W (&a)[S::NS], const S &s, uint8_t *dst, int len, bool live) {
  constexpr int W = RATE / 8;
  for (int off = 0;; off += RATE) {
    typename S::W w[S::NS];
#pragma unroll
    for (int y = 0; y < S::NS; y++)
      if (S::least(y) < W) w[y] = RAW ? a[y] : s.out(a[y]);
#pragma unroll
    for (int y = 0; y < S::NS; y++)
      if (S::least(y) < W) pin(w[y]);
    const int words = min(W, (len - off) / 8);
    if (live && s.writer()) {
#pragma unroll
      for (int y = 0; y < S::NS; y++)
        if (S::least(y) < W && s.lane(y) < words) s.store(dst + off + 8 * s.lane(y), w[y]);
    }
    if (off + RATE >= len) break;
    s.perm(a);
  }
}

// Store lanes 0 .. N-1 of a state to dst.
template <class S, int N>
__device__ __forceinline__ void store(const typename S::W (&a)[S::NS], const S &s, uint8_t *dst, bool live) {
#pragma unroll
  for (int y = 0; y < S::NS; y++) {
    if (S::least(y) >= N) continue;
    const int q = s.lane(y);
    const typename S::W w = s.out(a[y]);
    if (q < N && live && s.writer()) s.store(dst + 8 * q, w);
  }
}

}  // namespace msp
}  // namespace dpkem

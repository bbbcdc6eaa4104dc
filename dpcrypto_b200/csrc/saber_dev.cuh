// Saber (LightSaber l=2, Saber l=3, FireSaber l=4) device routines for sm_100a, written per
// instance so the batched kernels (saber.cu) and the persistent mixed-batch kernel
// (mixed.cu) run the same code.
//
// Kernel chain per operation:
//   prologue  (two sponges an instance: role 0 the hash chain and GenSecret's SHAKE128, decaps: then
//              SHA3-256 of the input ciphertext; role 1 GenMatrix's SHAKE128; XOF bytes go to the
//              scratch arena.  Lanes per state by batch size, saber.cu)
//   product   (CTA/instance: CBD sampling, 13/10-bit unpacking, the negacyclic
//              matrix-vector and inner products, rounding, packing / comparison)
//   finish    (SHA3-256(c) (encaps), final key, or H(pk) for keypair)
// Decaps runs the product kernel twice: first the inner product v = b'^T s with the
// secret from sk (-> m'), then the re-encryption in compare mode.
//
// Two product forms:
//   dp4a: thread = output coefficient; dp2a(16-bit public pair, 8-bit secret pair)
//         over a reversed, sign-extended secret window (no branch on the wrap).
//   tc:   tcgen05.mma kind::i8, D[coef][(out, limb)] = sum_K H_j[coef][K] * P[K][(out,limb)].
//         The public polynomials are written in reversed coefficient order along K,
//         which turns the negacyclic Toeplitz block of each secret into a Hankel block:
//         T'[i][k'] = s_ext[i + k' - 255].  Its core matrix (8 rows x 16 bytes) at
//         (mi, ki) depends only on t = mi + 2 ki, so the whole 256 x 256 block is 62
//         distinct 128-byte core matrices (SBO = 128, LBO = 256) instead of 64 KB.
//         Public coefficients are split into u8 limbs (lo 8 bits, hi bits) along N.
//
// Replaces the reference's per-stage launches (SABER-GPU/src/cuda_kernel.cu:19-299),
// its dp4a-shaped DoDP4Av7/_inner products over HBM rotation tables
// (SABER-GPU/src/poly.cu:26-206) and its FO helpers (pack.cu:215-255), following the
// round-3 specification order (cmov of z before the final hash).
#pragma once
#include "common.cuh"
#include "keccak.cuh"
#include "msponge.cuh"
#include "tc.cuh"

namespace dpkem {
namespace sdev {

using saber::EP;
using saber::EQ;
constexpr int SN = saber::N;

enum PMode : int { PM_KEYPAIR = 0, PM_ENC = 1, PM_DEC_CMP = 2, PM_DEC_INNER = 3 };

template <int L>
struct SP {
  static constexpr saber::Params p = saber::params(L);
  static constexpr int MU = p.mu, ET = p.et;
  static constexpr int POLYVEC = p.polyvec, POLYVECCOMP = p.polyveccomp, PK = p.pk, SK = p.sk, CT = p.ct;
  static constexpr int ARAW = L * L * EQ * SN / 8;  // GenMatrix bytes
  static constexpr int SRAW = L * MU * SN / 8;      // GenSecret bytes
  static constexpr uint32_t H1 = 1u << (EQ - EP - 1);
  static constexpr uint32_t H2 = (1u << (EP - 2)) - (1u << (EP - ET - 1)) + (1u << (EQ - EP - 1));
};

// Scratch offsets within one instance's record (all multiples of 16).
template <int L>
struct Scr {
  static constexpr int ARAW = 0;
  static constexpr int SRAW = (SP<L>::ARAW + 15) & ~15;
  static constexpr int KR = SRAW + ((SP<L>::SRAW + 15) & ~15);
  static constexpr int MTXT = KR + 64;
  static constexpr int HC = MTXT + 32;  // decaps: SHA3-256(c), hashed by the prologue
  static constexpr int BYTES = HC + 32;
};

// Pointers of one instance, already offset into the caller's arrays and the scratch arena.
struct Inst {
  const uint8_t *coins;  // keypair 96 B, enc 32 B
  uint8_t *pk, *sk, *ct, *ss;
  uint8_t *scr;          // this instance's scratch record (Scr<L>::BYTES)
  uint32_t *fail;
};

template <int L>
__device__ __forceinline__ Inst inst_of(const SaberBatch &b, int i, int op) {
  using P = SP<L>;
  Inst v;
  v.coins = b.coins ? b.coins + (size_t)i * (op == OP_KEYPAIR ? 96 : 32) : nullptr;
  v.pk = b.pk ? b.pk + (size_t)i * P::PK : nullptr;
  v.sk = b.sk ? b.sk + (size_t)i * P::SK : nullptr;
  v.ct = b.ct ? b.ct + (size_t)i * P::CT : nullptr;
  v.ss = b.ss ? b.ss + (size_t)i * 32 : nullptr;
  v.scr = b.scr + (size_t)i * Scr<L>::BYTES;
  v.fail = b.fail + i;
  return v;
}

// SHAKE128 of a 32-byte seed held in 4 lanes, squeezing `len` bytes (len % 8 == 0) to dst.
__device__ __forceinline__ void shake128_seed32(const uint2 (&seed)[4], uint8_t *dst, int len) {
  uint2 a[25];
  keccak_zero(a);
#pragma unroll
  for (int q = 0; q < 4; q++) a[q] = seed[q];
  absorb_finish<168>(a, 32, 0x1Fu);
  for (int off = 0;; off += 168) {
#pragma unroll
    for (int q = 0; q < 21; q++)
      if (off + 8 * q < len) *reinterpret_cast<uint2 *>(dst + off + 8 * q) = a[q];
    if (off + 168 >= len) break;
    keccak_f1600(a);
  }
}

// SHA3-256 of a whole byte string (length multiple of 8, 8-byte aligned).
__device__ __forceinline__ void sha3_256_msg(const uint8_t *p, int len, uint2 (&out)[4]) {
  uint2 a[25];
  keccak_zero(a);
  const int pos = absorb_aligned<136>(a, 0, p, len);
  absorb_finish<136>(a, pos, 0x06u);
#pragma unroll
  for (int q = 0; q < 4; q++) out[q] = a[q];
}

// SHA3-256 / SHA3-512 of 64 bytes held in lanes.
__device__ __forceinline__ void sha3_256_64(const uint2 (&m)[8], uint2 (&out)[4]) {
  uint2 a[25];
  keccak_zero(a);
#pragma unroll
  for (int q = 0; q < 8; q++) a[q] = m[q];
  absorb_finish<136>(a, 64, 0x06u);
#pragma unroll
  for (int q = 0; q < 4; q++) out[q] = a[q];
}
__device__ __forceinline__ void sha3_512_64(const uint2 (&m)[8], uint2 (&out)[8]) {
  uint2 a[25];
  keccak_zero(a);
#pragma unroll
  for (int q = 0; q < 8; q++) a[q] = m[q];
  absorb_finish<72>(a, 64, 0x06u);
#pragma unroll
  for (int q = 0; q < 8; q++) out[q] = a[q];
}

// ---------------------------------------------------------------- prologue
// role 0 = hash chain + GenSecret XOF, role 1 = GenMatrix XOF: the two independent sponges
// of one instance (the batched kernel runs them on different warps).
template <int L, int OP>
__device__ __forceinline__ void prologue_inst(const Inst &v, int role) {
  using P = SP<L>;
  using S = Scr<L>;
  uint8_t *scr = v.scr;
  if (role == 1) {
    uint2 seed[4];
    if (OP == OP_KEYPAIR) {
      // seed_A = SHAKE128(coins[0:32], 32), published in pk.
      uint2 a[25];
      keccak_zero(a);
#pragma unroll
      for (int q = 0; q < 4; q++) a[q] = ld_lane(v.coins + 8 * q);
      absorb_finish<168>(a, 32, 0x1Fu);
      uint8_t *pk = v.pk + P::POLYVECCOMP;
#pragma unroll
      for (int q = 0; q < 4; q++) {
        seed[q] = a[q];
        *reinterpret_cast<uint2 *>(pk + 8 * q) = a[q];
      }
    } else {
      const uint8_t *src = OP == OP_ENC ? v.pk + P::POLYVECCOMP : v.sk + P::POLYVEC + P::POLYVECCOMP;
#pragma unroll
      for (int q = 0; q < 4; q++) seed[q] = ld_lane(src + 8 * q);
    }
    shake128_seed32(seed, scr + S::ARAW, P::ARAW);
    return;
  }
  uint2 seed[4];
  if (OP == OP_KEYPAIR) {
#pragma unroll
    for (int q = 0; q < 4; q++) seed[q] = ld_lane(v.coins + 32 + 8 * q);
  } else {
    uint2 buf[8], kr[8];
    if (OP == OP_ENC) {
      // m = SHA3-256(coins), H(pk), kr = SHA3-512(m || H(pk))  (cuda_kernel.cu:68-70)
      uint2 c8[8], h[4];
#pragma unroll
      for (int q = 0; q < 4; q++) c8[q] = ld_lane(v.coins + 8 * q);
#pragma unroll
      for (int q = 4; q < 8; q++) c8[q] = make_uint2(0, 0);
      uint2 a[25];
      keccak_zero(a);
#pragma unroll
      for (int q = 0; q < 4; q++) a[q] = c8[q];
      absorb_finish<136>(a, 32, 0x06u);
#pragma unroll
      for (int q = 0; q < 4; q++) buf[q] = a[q];
      sha3_256_msg(v.pk, P::PK, h);
#pragma unroll
      for (int q = 0; q < 4; q++) buf[4 + q] = h[q];
    } else {
      // m' from the inner-product pass, H(pk) stored in sk (cuda_kernel.cu:231-232)
      const uint8_t *hpk = v.sk + P::SK - 64;
#pragma unroll
      for (int q = 0; q < 4; q++) {
        buf[q] = ld_lane(scr + S::MTXT + 8 * q);
        buf[4 + q] = ld_lane(hpk + 8 * q);
      }
    }
    sha3_512_64(buf, kr);
    uint8_t *krp = scr + S::KR;
#pragma unroll
    for (int q = 0; q < 8; q++) *reinterpret_cast<uint2 *>(krp + 8 * q) = kr[q];
    if (OP == OP_ENC) {
#pragma unroll
      for (int q = 0; q < 4; q++) *reinterpret_cast<uint2 *>(scr + S::MTXT + 8 * q) = buf[q];
    }
#pragma unroll
    for (int q = 0; q < 4; q++) seed[q] = kr[4 + q];
  }
  shake128_seed32(seed, scr + S::SRAW, P::SRAW);
  if (OP == OP_DEC) {
    // H(c) of the input ciphertext does not wait for the products: hashing it here keeps
    // this role (15 permutations at l = 3) shorter than GenMatrix's, and the finish stage
    // down to one permutation.
    uint2 hc[4];
    sha3_256_msg(v.ct, P::CT, hc);
#pragma unroll
    for (int q = 0; q < 4; q++) *reinterpret_cast<uint2 *>(scr + S::HC + 8 * q) = hc[q];
  }
}

// ---------------------------------------------------------------- several lanes per state
// The same prologue roles and encaps / keypair finish with each sponge spread over several
// lanes (msponge.cuh: S = msp::Multi<1>, a warp per state, msp::Multi<10>, ten lanes, or
// msp::Multi<2>, a pair): the bytes written are those of prologue_inst / finish_inst.  live = false keeps a
// state without an instance in step (reads stay in bounds, writes are skipped).
// RAW: the XOF bytes stay in the layout's form (msp::squeeze), the product's staging restores them.
template <class S, int L, int OP, bool RAW = false>
__device__ __forceinline__ void prologue_multi(const Inst &v, const S &s, int role, bool live) {
  using P = SP<L>;
  using Q = Scr<L>;
  uint8_t *scr = v.scr;
  typename S::W a[S::NS];
  msp::zero<S>(a);
  if (role == 1) {  // GenMatrix
    if (OP == OP_KEYPAIR) {  // seed_A = SHAKE128(coins[0:32], 32), published in pk
      msp::absorb_aligned<S, 168>(a, s, 0, v.coins, 32, live);
      msp::absorb_finish<S, 168>(a, s, 32, 0x1Fu);
      msp::store<S, 4>(a, s, v.pk + P::POLYVECCOMP, live);
      msp::keep<S>(a, s, 4);
    } else {
      const uint8_t *src = OP == OP_ENC ? v.pk + P::POLYVECCOMP : v.sk + P::POLYVEC + P::POLYVECCOMP;
      msp::absorb_aligned<S, 168>(a, s, 0, src, 32, live);
    }
    msp::absorb_finish<S, 168>(a, s, 32, 0x1Fu);
    msp::squeeze<S, 168, RAW>(a, s, scr + Q::ARAW, P::ARAW, live);
    return;
  }
  if (OP == OP_KEYPAIR) {
    msp::absorb_aligned<S, 168>(a, s, 0, v.coins + 32, 32, live);
  } else {
    typename S::W kr[S::NS];
    msp::zero<S>(kr);
    if (OP == OP_ENC) {
      // m = SHA3-256(coins), H(pk), kr = SHA3-512(m || H(pk))  (cuda_kernel.cu:68-70)
      msp::absorb_aligned<S, 136>(kr, s, 0, v.coins, 32, live);
      msp::absorb_finish<S, 136>(kr, s, 32, 0x06u);
      msp::store<S, 4>(kr, s, scr + Q::MTXT, live);
      msp::keep<S>(kr, s, 4);  // lanes 0..3 = m
      const int pos = msp::absorb_aligned<S, 136>(a, s, 0, v.pk, P::PK, live);
      msp::absorb_finish<S, 136>(a, s, pos, 0x06u);
      msp::move4<S, 4>(kr, a, s);  // lanes 4..7 = H(pk)
    } else {
      // m' from the inner-product pass, H(pk) stored in sk (cuda_kernel.cu:231-232)
      const int pos = msp::absorb_aligned<S, 72>(kr, s, 0, scr + Q::MTXT, 32, live);
      msp::absorb_aligned<S, 72>(kr, s, pos, v.sk + P::SK - 64, 32, live);
    }
    msp::absorb_finish<S, 72>(kr, s, 64, 0x06u);
    msp::store<S, 8>(kr, s, scr + Q::KR, live);
    // GenSecret seed = kr[32:64] = lanes 4..7 -> lanes 0..3
    msp::zero<S>(a);
    msp::xor_lane<S, 0>(a, s, s.template get<4>(kr));
    msp::xor_lane<S, 1>(a, s, s.template get<5>(kr));
    msp::xor_lane<S, 2>(a, s, s.template get<6>(kr));
    msp::xor_lane<S, 3>(a, s, s.template get<7>(kr));
  }
  msp::absorb_finish<S, 168>(a, s, 32, 0x1Fu);
  msp::squeeze<S, 168, RAW>(a, s, scr + Q::SRAW, P::SRAW, live);
  if (OP == OP_DEC) {  // H(c) of the input ciphertext (see prologue_inst)
    msp::zero<S>(a);
    const int pos = msp::absorb_aligned<S, 136>(a, s, 0, v.ct, P::CT, live);
    msp::absorb_finish<S, 136>(a, s, pos, 0x06u);
    msp::store<S, 4>(a, s, scr + Q::HC, live);
  }
}

// Encaps finish: k = SHA3-256(kr[0:32] || SHA3-256(c)).
template <class S, int L>
__device__ __forceinline__ void finish_enc_multi(const Inst &v, const S &s, bool live) {
  using P = SP<L>;
  using Q = Scr<L>;
  typename S::W h[S::NS], a[S::NS];
  msp::zero<S>(h);
  const int pos = msp::absorb_aligned<S, 136>(h, s, 0, v.ct, P::CT, live);
  msp::absorb_finish<S, 136>(h, s, pos, 0x06u);
  msp::zero<S>(a);
  msp::absorb_aligned<S, 136>(a, s, 0, v.scr + Q::KR, 32, live);
  msp::move4<S, 4>(a, h, s);
  msp::absorb_finish<S, 136>(a, s, 64, 0x06u);
  msp::store<S, 4>(a, s, v.ss, live);
}

// Keypair finish: sk = s || pk || H(pk) || z (the secret part was written by the product).
template <class S, int L>
__device__ __forceinline__ void finish_kp_multi(const Inst &v, const S &s, bool live) {
  using P = SP<L>;
  if (live && s.writer()) {  // pk, words t, t + T, ... on thread t of the state's T
    constexpr int T = 32 / S::STATES_PER_WARP < 25 ? 32 / S::STATES_PER_WARP : 25;
    const int t = (int)(threadIdx.x & 31) - T * s.state();
    for (int off = 8 * t; off < P::PK; off += 8 * T)
      *reinterpret_cast<uint2 *>(v.sk + P::POLYVEC + off) = ld_lane(v.pk + off);
  }
  typename S::W a[S::NS];
  msp::zero<S>(a);
  const int pos = msp::absorb_aligned<S, 136>(a, s, 0, v.pk, P::PK, live);
  msp::absorb_finish<S, 136>(a, s, pos, 0x06u);
  msp::store<S, 4>(a, s, v.sk + P::SK - 64, live);
#pragma unroll
  for (int y = 0; y < S::NS; y++)
    if (S::least(y) < 4 && live && s.writer() && s.lane(y) < 4)
      s.store(v.sk + P::SK - 32 + 8 * s.lane(y), s.load(v.coins + 64 + 8 * s.lane(y)));
}

// ---------------------------------------------------------------- finish
template <int L, int OP>
__device__ __forceinline__ void finish_inst(const Inst &v) {
  using P = SP<L>;
  using S = Scr<L>;
  if (OP == OP_KEYPAIR) {
    const uint8_t *pk = v.pk;
    uint8_t *sk = v.sk;
    for (int off = 0; off < P::PK; off += 8) *reinterpret_cast<uint2 *>(sk + P::POLYVEC + off) = ld_lane(pk + off);
    uint2 h[4];
    sha3_256_msg(pk, P::PK, h);
#pragma unroll
    for (int q = 0; q < 4; q++) {
      *reinterpret_cast<uint2 *>(sk + P::SK - 64 + 8 * q) = h[q];
      *reinterpret_cast<uint2 *>(sk + P::SK - 32 + 8 * q) = ld_lane(v.coins + 64 + 8 * q);
    }
    return;
  }
  const uint8_t *scr = v.scr;
  uint2 m[8], hc[4], k[4];
  if (OP == OP_DEC) {
#pragma unroll
    for (int q = 0; q < 4; q++) hc[q] = ld_lane(scr + S::HC + 8 * q);
  } else {
    sha3_256_msg(v.ct, P::CT, hc);
  }
  const uint32_t msk = OP == OP_DEC ? 0u - (uint32_t)(*v.fail != 0u) : 0u;
  const uint8_t *z = v.sk + P::SK - 32;
#pragma unroll
  for (int q = 0; q < 4; q++) {
    uint2 x = ld_lane(scr + S::KR + 8 * q);
    if (OP == OP_DEC) {  // cmov(kr, z, fail) before the final hash
      const uint2 y = ld_lane(z + 8 * q);
      x = make_uint2((x.x & ~msk) | (y.x & msk), (x.y & ~msk) | (y.y & msk));
    }
    m[q] = x;
    m[4 + q] = hc[q];
  }
  sha3_256_64(m, k);
#pragma unroll
  for (int q = 0; q < 4; q++) *reinterpret_cast<uint2 *>(v.ss + 8 * q) = k[q];
}

// ---------------------------------------------------------------- bit packing helpers
// Coefficient c of `bits` bits from a little-endian packed array in shared memory that is
// 4-byte aligned and readable 8 bytes past the coefficient: two aligned words, one funnel
// shift (sh <= 31 and sh + bits <= 44, so two words always suffice).
__device__ __forceinline__ uint32_t unpack_smem(const uint8_t *src, int c, int bits) {
  const int bit = c * bits, by = bit >> 3;
  const uint32_t *w = reinterpret_cast<const uint32_t *>(src + (by & ~3));
  return __funnelshift_r(w[0], w[1], (bit & 7) + 8 * (by & 3)) & ((1u << bits) - 1u);
}

// Unpacks NC little-endian BITS-bit fields from whole words (NC * BITS a multiple of 32)
// and calls f(i, value) for each; all bit offsets are compile-time after unrolling.
template <int BITS, int NC, class F>
__device__ __forceinline__ void unpack_words(const uint32_t *w, F &&f) {
  static_assert(NC * BITS % 32 == 0, "whole words");
  constexpr int NW = NC * BITS / 32;
  uint32_t r[NW + 1];
#pragma unroll
  for (int k = 0; k < NW; k++) r[k] = w[k];
  r[NW] = 0;
#pragma unroll
  for (int i = 0; i < NC; i++) {
    const int bit = i * BITS, k = bit >> 5, sh = bit & 31;
    const uint32_t v = sh + BITS <= 32 ? r[k] >> sh : __funnelshift_r(r[k], r[k + 1], sh);
    f(i, v & ((1u << BITS) - 1u));
  }
}

// Byte-wise two's-complement negation of four int8 lanes.
__device__ __forceinline__ uint32_t neg_bytes(uint32_t x) {
  return ((~x & 0x7F7F7F7Fu) + 0x01010101u) ^ (~x & 0x80808080u);
}

// Packs the G = 8 / gcd(BITS, 8) coefficients v[0..G) (each < 2^BITS) little-endian into
// G * BITS / 8 bytes at out: the smallest group that ends on a byte boundary, unrolled.
template <int BITS>
__device__ __forceinline__ constexpr int group_coefs() {
  return BITS % 8 == 0 ? 1 : BITS % 4 == 0 ? 2 : BITS % 2 == 0 ? 4 : 8;
}
template <int BITS>
__device__ __forceinline__ void pack_group(const uint16_t *v, uint8_t *out) {
  constexpr int G = group_coefs<BITS>();
  uint64_t acc = 0;
  int nb = 0, o = 0;
#pragma unroll
  for (int i = 0; i < G; i++) {
    acc |= (uint64_t)v[i] << nb;
    nb += BITS;
#pragma unroll
    for (int k = 0; k < 2; k++)
      if (nb >= 8) {
        out[o++] = (uint8_t)acc;
        acc >>= 8;
        nb -= 8;
      }
  }
}
// n coefficients (a multiple of the group size) into `out` (shared memory), CTA-wide.
// Group g on thread (off + g) mod blockDim: a second pack in the same phase starts where the
// first one's groups end.
template <int BITS>
__device__ __forceinline__ void pack_poly(const uint16_t *v, int n, uint8_t *out, int off = 0) {
  constexpr int G = group_coefs<BITS>(), NB = G * BITS / 8;
  const int nt = blockDim.x;
  for (int g = ((int)threadIdx.x + nt - off % nt) % nt; g < n / G; g += nt) pack_group<BITS>(v + g * G, out + g * NB);
}

__device__ __forceinline__ uint32_t pack_byte(const uint16_t *v, int q, int bits) {
  const int bit0 = 8 * q;
  int c = bit0 / bits;
  const int off = bit0 - c * bits;
  const uint32_t mask = (1u << bits) - 1u;
  uint32_t acc = (v[c] & mask) >> off;
  int have = bits - off;
  while (have < 8) {
    c++;
    acc |= (uint32_t)(v[c] & mask) << have;
    have += bits;
  }
  return acc & 0xFFu;
}

// ---------------------------------------------------------------- product kernel
// Shared-memory layout of the dp4a / INT32 forms.
template <int L>
struct PL {
  static constexpr int NO_MAX = L + 1;
  // Public polynomials are 264 u16 apart (528 B): polynomials read at the same offset
  // by neighbouring threads start 4 banks apart.
  static constexpr int PS = SN + 8;
  static constexpr int A16 = 0;                               // u16 [L*L][PS]
  static constexpr int B16 = A16 + L * L * PS * 2;            // u16 [L][PS] public b / b'
  static constexpr int SEC = B16 + L * PS * 2;                // s8  [L][256]
  static constexpr int RES = SEC + L * SN;                    // u16 [L+1][256]
  static constexpr int CM = RES + NO_MAX * SN * 2;            // u16 [256]
  static constexpr int SEQ = CM + SN * 2;                     // s8  [L][528] secret sequences
  static constexpr int SEQ_STRIDE = 528;
  static constexpr int COMMON = SEQ + L * SEQ_STRIDE;
  // Packed operands copied in from global memory before unpacking.  Each piece is followed by
  // 8 readable bytes (unpack_smem).
  static constexpr int STAGE = (COMMON + 127) & ~127;
  static constexpr int ST_A = STAGE;                                        // GenMatrix bytes
  static constexpr int ST_S = ST_A + SP<L>::ARAW + 8;                       // GenSecret bytes
  static constexpr int ST_P = ST_S + SP<L>::SRAW + 8;                       // packed b (pk)
  static constexpr int ST_END = ST_P + SP<L>::POLYVECCOMP + 8;
  static constexpr int ST_SK = STAGE;                                       // decaps inner: 13-bit s
  static constexpr int ST_CT = ST_SK + SP<L>::POLYVEC + 8;                  // and the ciphertext
  static constexpr int ST_END_INNER = ST_CT + SP<L>::CT + 8;
  static constexpr int DP4A_TOTAL = ST_END > ST_END_INNER ? ST_END : ST_END_INNER;
};

// Shared-memory layout of the tcgen05 form.
template <int L>
struct TL {
  static constexpr int SEQ = 0;                               // s8 [L][528]: E_j, see tc_product
  static constexpr int SEQ_STRIDE = 528;
  static constexpr int RES = L * SEQ_STRIDE;                  // u16 [L+1][256] rounded results
  static constexpr int CM = RES + (L + 1) * SN * 2;           // 32 message bytes
  static constexpr int HANK = (CM + 32 + 127) & ~127;         // [L][62][128]
  static constexpr int HANK_STRIDE = 62 * 128;
  // B operand, [NPAD/8][K/16] core matrices of 8 rows x 16 bytes, 144 bytes apart: the sixteen chunks
  // of a polynomial are stored by sixteen threads at once, 128 bytes apart all in the same banks.
  static constexpr int BOP = HANK + L * HANK_STRIDE;
  static constexpr int CHUNK = 144;
  static constexpr int NPAD = 2 * (L + 1) <= 8 ? 8 : 16;
  static constexpr int BOP_GROUP = L * SN / 16 * CHUNK;       // bytes per 8-row N group
  static constexpr int BAR = BOP + (NPAD / 8) * BOP_GROUP;
  static constexpr int TSLOT = BAR + 8;
  static constexpr int TOTAL = TSLOT + 8;
  // Packed operands: unpacked before the Hankel matrices are built, so in their place.
  static constexpr int ST_A = HANK;
  static constexpr int ST_S = ST_A + SP<L>::ARAW + 8;
  static constexpr int ST_P = ST_S + SP<L>::SRAW + 8;
  static constexpr int ST_SK = HANK;
  static constexpr int ST_CT = ST_SK + SP<L>::POLYVEC + 8;
  static_assert(ST_P + SP<L>::POLYVECCOMP + 8 <= BOP && ST_CT + SP<L>::CT + 8 <= BOP, "staging fits the Hankel area");
};

template <int L, int MODE>
__device__ __forceinline__ constexpr int n_out() {
  return MODE == PM_KEYPAIR ? L : MODE == PM_DEC_INNER ? 1 : L + 1;
}

// 8-byte copy of `bytes` (a multiple of 8, both ends 8-byte aligned) by the whole CTA.
__device__ __forceinline__ void copy8(uint8_t *dst, const uint8_t *src, int bytes) {
  for (int q = threadIdx.x; q < bytes / 8; q += blockDim.x)
    reinterpret_cast<uint2 *>(dst)[q] = reinterpret_cast<const uint2 *>(src)[q];
}

// Phase 1: secrets and public polynomials into shared memory.  The packed inputs are
// first copied in with 8-byte loads (a handful per thread), then unpacked from shared
// memory, instead of up to three byte loads from global memory per coefficient.
// The packed inputs of one instance as 8-byte words: source in global memory and
// destination in the staging area.
template <int L, int MODE, class Y>
struct Staged {
  using P = SP<L>;
  static_assert(P::ARAW % 8 == 0 && P::SRAW % 8 == 0 && P::POLYVECCOMP % 8 == 0 && P::POLYVEC % 8 == 0 &&
                    P::CT % 8 == 0,
                "8-byte staging");
  static constexpr bool INNER = MODE == PM_DEC_INNER;
  static constexpr int W0 = (INNER ? P::POLYVEC : P::ARAW) / 8;                      // words of piece 0
  static constexpr int W1 = (INNER ? P::CT : P::SRAW) / 8;                            // piece 1
  static constexpr int W2 = (INNER || MODE == PM_KEYPAIR) ? 0 : P::POLYVECCOMP / 8;  // piece 2
  // piece 3: the message bits m (32 bytes of scratch) that the epilogue encodes into v'
  // (encaps, decaps re-encryption), staged in the CM region, which only the inner pass uses
  static constexpr int W3 = (INNER || MODE == PM_KEYPAIR) ? 0 : 4;
  static constexpr int WORDS = W0 + W1 + W2 + W3;
  static constexpr int PER_THREAD = (WORDS + 255) / 256;  // with 256 threads
  // Word w of the XOF bytes, which the prologue may have left as bit-interleaved halves.
  __device__ __forceinline__ static uint2 natural(int w, uint2 x, bool sliced) {
    return !INNER && sliced && w < W0 + W1 ? k10::lane_of(x) : x;
  }
  __device__ __forceinline__ static const uint2 *src(const Inst &v, int w) {
    if (INNER)
      return w < W0 ? reinterpret_cast<const uint2 *>(v.sk) + w : reinterpret_cast<const uint2 *>(v.ct) + (w - W0);
    if (w < W0) return reinterpret_cast<const uint2 *>(v.scr + Scr<L>::ARAW) + w;
    if (w < W0 + W1) return reinterpret_cast<const uint2 *>(v.scr + Scr<L>::SRAW) + (w - W0);
    if (w < W0 + W1 + W2)
      return reinterpret_cast<const uint2 *>(MODE == PM_ENC ? v.pk : v.sk + P::POLYVEC) + (w - W0 - W1);
    return reinterpret_cast<const uint2 *>(v.scr + Scr<L>::MTXT) + (w - W0 - W1 - W2);
  }
  __device__ __forceinline__ static uint2 *dst(uint8_t *sm, int w) {
    if (INNER)
      return w < W0 ? reinterpret_cast<uint2 *>(sm + Y::ST_SK) + w : reinterpret_cast<uint2 *>(sm + Y::ST_CT) + (w - W0);
    if (w < W0) return reinterpret_cast<uint2 *>(sm + Y::ST_A) + w;
    if (w < W0 + W1) return reinterpret_cast<uint2 *>(sm + Y::ST_S) + (w - W0);
    if (w < W0 + W1 + W2) return reinterpret_cast<uint2 *>(sm + Y::ST_P) + (w - W0 - W1);
    return reinterpret_cast<uint2 *>(sm + Y::CM) + (w - W0 - W1 - W2);
  }
};

// Copy one instance's packed inputs into the staging area (CTA-wide, 8-byte accesses).
template <int L, int MODE, class Y>
__device__ __forceinline__ void stage_operands(const Inst &v, uint8_t *sm, bool sliced) {
  using T = Staged<L, MODE, Y>;
  for (int w = threadIdx.x; w < T::WORDS; w += blockDim.x) *T::dst(sm, w) = T::natural(w, *T::src(v, w), sliced);
}

// The same copy split in two for a persistent loop (256 threads): load() into registers
// early, store() into the staging area once it is free.
template <int L, int MODE>
struct OperandPrefetch {
  using T = Staged<L, MODE, TL<L>>;
  uint2 r[T::PER_THREAD];
  __device__ __forceinline__ void load(const Inst &v) {
#pragma unroll
    for (int k = 0; k < T::PER_THREAD; k++) {
      const int w = threadIdx.x + 256 * k;
      if (w < T::WORDS) r[k] = *T::src(v, w);
    }
  }
  __device__ __forceinline__ void store(uint8_t *sm, bool sliced) const {
#pragma unroll
    for (int k = 0; k < T::PER_THREAD; k++) {
      const int w = threadIdx.x + 256 * k;
      if (w < T::WORDS) *T::dst(sm, w) = T::natural(w, r[k], sliced);
    }
  }
};

template <int L, int MODE>
__device__ __forceinline__ void unpack_operands(const Inst &v, uint8_t *sm);

template <int L, int MODE>
__device__ __forceinline__ void load_operands(const Inst &v, uint8_t *sm, bool sliced) {
  stage_operands<L, MODE, PL<L>>(v, sm, sliced);
  __syncthreads();
  unpack_operands<L, MODE>(v, sm);
}

// Unpack the staged inputs (after stage_operands and a CTA barrier).
template <int L, int MODE>
__device__ __forceinline__ void unpack_operands(const Inst &v, uint8_t *sm) {
  using P = SP<L>;
  using Y = PL<L>;
  const int tid = threadIdx.x;
  uint32_t *secw = reinterpret_cast<uint32_t *>(sm + Y::SEC);  // 4 int8 coefficients per word
  uint16_t *a16 = reinterpret_cast<uint16_t *>(sm + Y::A16);
  uint16_t *b16 = reinterpret_cast<uint16_t *>(sm + Y::B16);
  uint16_t *cm = reinterpret_cast<uint16_t *>(sm + Y::CM);
  // Public polynomials with 10-bit coefficients: 16 coefficients (5 words) per thread, two
  // 16-byte stores.
  // The unpack loops of one mode start at disjoint thread ranges (job g of a loop that starts
  // at thread `off` runs on thread off + g), so no thread does two jobs while others wait at
  // the barrier that follows: l = 3 encaps has 48 + 72 + 48 jobs for 256 threads.
  auto job0 = [&](int off) { return (tid + (int)blockDim.x - off) % (int)blockDim.x; };
  auto unpack_p = [&](const uint8_t *src, int off) {
    for (int g = job0(off); g < L * SN / 16; g += blockDim.x) {
      uint32_t o[8];
      unpack_words<EP, 16>(reinterpret_cast<const uint32_t *>(src) + 5 * g, [&](int i, uint32_t x) {
        if (i & 1) o[i >> 1] |= x << 16;
        else o[i >> 1] = x;
      });
      uint4 *d = reinterpret_cast<uint4 *>(b16 + (g >> 4) * Y::PS + 16 * (g & 15));
      d[0] = make_uint4(o[0], o[1], o[2], o[3]);
      d[1] = make_uint4(o[4], o[5], o[6], o[7]);
    }
  };
  if (MODE == PM_DEC_INNER) {
    const uint8_t *ct = sm + Y::ST_CT;
    // 13-bit secret from sk, centred: 32 coefficients (13 words) per thread.
    for (int g = tid; g < L * SN / 32; g += blockDim.x) {
      uint32_t o[8];
      unpack_words<EQ, 32>(reinterpret_cast<const uint32_t *>(sm + Y::ST_SK) + 13 * g, [&](int i, uint32_t x) {
        const uint32_t b = x & 0xFFu;  // low byte of the centred value (|s| < 128)
        if ((i & 3) == 0) o[i >> 2] = b;
        else o[i >> 2] |= b << (8 * (i & 3));
      });
      uint4 *d = reinterpret_cast<uint4 *>(secw + 8 * g);
      d[0] = make_uint4(o[0], o[1], o[2], o[3]);
      d[1] = make_uint4(o[4], o[5], o[6], o[7]);
    }
    unpack_p(ct, L * SN / 32);
    for (int c = tid; c < SN; c += blockDim.x) cm[c] = (uint16_t)unpack_smem(ct + P::POLYVECCOMP, c, P::ET);
  } else {
    // CBD_mu from the GenSecret bytes: 16 coefficients (mu/2 words) per thread.
    constexpr uint32_t hm = (1u << (P::MU / 2)) - 1u;
    for (int g = job0(0); g < L * SN / 16; g += blockDim.x) {
      uint32_t o[4];
      unpack_words<P::MU, 16>(reinterpret_cast<const uint32_t *>(sm + Y::ST_S) + (P::MU / 2) * g,
                              [&](int i, uint32_t x) {
                                const uint32_t b = (uint32_t)(__popc(x & hm) - __popc((x >> (P::MU / 2)) & hm)) & 0xFFu;
                                if ((i & 3) == 0) o[i >> 2] = b;
                                else o[i >> 2] |= b << (8 * (i & 3));
                              });
      reinterpret_cast<uint4 *>(secw)[g] = make_uint4(o[0], o[1], o[2], o[3]);
    }
    // GenMatrix: 13-bit coefficients, 32 (13 words) per thread, four 16-byte stores.
    for (int g = job0(L * SN / 16); g < L * L * SN / 32; g += blockDim.x) {
      uint32_t o[16];
      unpack_words<EQ, 32>(reinterpret_cast<const uint32_t *>(sm + Y::ST_A) + 13 * g, [&](int i, uint32_t x) {
        if (i & 1) o[i >> 1] |= x << 16;
        else o[i >> 1] = x;
      });
      uint4 *d = reinterpret_cast<uint4 *>(a16 + (g >> 3) * Y::PS + 32 * (g & 7));
#pragma unroll
      for (int q = 0; q < 4; q++) d[q] = make_uint4(o[4 * q], o[4 * q + 1], o[4 * q + 2], o[4 * q + 3]);
    }
    if (MODE != PM_KEYPAIR) unpack_p(sm + Y::ST_P, L * SN / 16 + L * L * SN / 32);
  }
}

// Secret sequences of the dp4a form, one 32-bit word (4 int8) per thread step, from the secrets
// in SEC: R_j[t] = s_ext[255 - t]: s[255 - t] for t < 256, -s[511 - t] below 512, 0 above.
template <int L>
__device__ __forceinline__ void build_seq(uint8_t *sm) {
  using Y = PL<L>;
  constexpr int NW = Y::SEQ_STRIDE / 4;  // 132
  const uint32_t *secw = reinterpret_cast<const uint32_t *>(sm + Y::SEC);
  uint32_t *seqw = reinterpret_cast<uint32_t *>(sm + Y::SEQ);
  for (int x = threadIdx.x; x < L * NW; x += blockDim.x) {
    const int j = x / NW, k = x - j * NW;
    const uint32_t *sw = secw + 64 * j;
    uint32_t e = 0;
    if (k < 64) e = __byte_perm(sw[63 - k], 0, 0x0123);
    else if (k < 128) e = neg_bytes(__byte_perm(sw[127 - k], 0, 0x0123));
    seqw[x] = e;
  }
}

// Public polynomial multiplied by secret j for output o.
template <int L, int MODE>
__device__ __forceinline__ const uint16_t *pub_poly(const uint8_t *sm, int o, int j) {
  using Y = PL<L>;
  const uint16_t *a16 = reinterpret_cast<const uint16_t *>(sm + Y::A16);
  const uint16_t *b16 = reinterpret_cast<const uint16_t *>(sm + Y::B16);
  if (MODE == PM_DEC_INNER) return b16 + j * Y::PS;
  if (MODE == PM_KEYPAIR) return a16 + (j * L + o) * Y::PS;  // transposed: b = A^T s
  return o < L ? a16 + (o * L + j) * Y::PS : b16 + j * Y::PS;
}

// Rounding, packing / comparison of the dp4a / INT32 forms.  res holds the products mod 2^16.
template <int L, int MODE>
__device__ __forceinline__ void epilogue(const Inst &v, uint8_t *sm) {
  using P = SP<L>;
  using S = Scr<L>;
  using Y = PL<L>;
  const int tid = threadIdx.x, nt = blockDim.x;
  uint16_t *res = reinterpret_cast<uint16_t *>(sm + Y::RES);
  uint8_t *scr = v.scr;
  if (MODE == PM_DEC_INNER) {
    const uint16_t *cm = reinterpret_cast<const uint16_t *>(sm + Y::CM);
    for (int c = tid; c < SN; c += nt)
      res[c] = (uint16_t)(((uint32_t)res[c] + P::H2 - ((uint32_t)cm[c] << (EP - P::ET))) >> (EP - 1)) & 1u;
    __syncthreads();
    if (tid < 32) scr[S::MTXT + tid] = (uint8_t)pack_byte(res, tid, 1);
    return;
  }
  for (int c = tid; c < L * SN; c += nt) res[c] = (uint16_t)((((uint32_t)res[c] + P::H1) >> (EQ - EP)) & 0x3FFu);
  if (MODE != PM_KEYPAIR) {
    const uint8_t *mt = sm + Y::CM;  // staged with the operands
    for (int c = tid; c < SN; c += nt) {
      const uint32_t mb = (mt[c >> 3] >> (c & 7)) & 1u;
      res[L * SN + c] = (uint16_t)((((uint32_t)res[L * SN + c] - (mb << (EP - 1)) + P::H1) >> (EP - P::ET)) &
                                   ((1u << P::ET) - 1u));
    }
  }
  __syncthreads();
  // Pack into shared memory (the staging area, free again), then 8-byte stores / compares.
  uint8_t *stg = sm + Y::ST_A;
  if (MODE == PM_KEYPAIR) {
    const int8_t *sec = reinterpret_cast<const int8_t *>(sm + Y::SEC);
    pack_poly<EP>(res, L * SN, stg);  // POLYVECCOMP bytes
    uint16_t *s13 = reinterpret_cast<uint16_t *>(sm + Y::A16);  // A no longer needed
    for (int c = tid; c < L * SN; c += nt) s13[c] = (uint16_t)((int32_t)sec[c] & 0x1FFF);
    __syncthreads();
    pack_poly<EQ>(s13, L * SN, stg + P::POLYVECCOMP);  // POLYVEC bytes
    __syncthreads();
    copy8(v.pk, stg, P::POLYVECCOMP);
    copy8(v.sk, stg + P::POLYVECCOMP, P::POLYVEC);
    return;
  }
  pack_poly<EP>(res, L * SN, stg);
  pack_poly<P::ET>(res + L * SN, SN, stg + P::POLYVECCOMP, L * SN / group_coefs<EP>());
  __syncthreads();
  if (MODE == PM_ENC) {
    copy8(v.ct, stg, P::CT);
  } else {
    uint32_t diff = 0;
    for (int q = tid; q < P::CT / 8; q += nt) {
      const uint2 a = reinterpret_cast<const uint2 *>(stg)[q], b = reinterpret_cast<const uint2 *>(v.ct)[q];
      diff |= (a.x ^ b.x) | (a.y ^ b.y);
    }
    const int any = __syncthreads_or(diff != 0);
    if (tid == 0) *v.fail = (uint32_t)any;
  }
}

// ---------------------------------------------------------------- dp4a form
// Secret j's reversed sign-extended window R_j[t] = s_ext[255 - t], t in [0, 512), with
// s_ext[d] = s[d] (d >= 0), -s[d + 256] (d < 0): coefficient i of s*P is
// sum_m P[m] R_j[255 - i + m].
// I32 = true is the INT32 schoolbook form (SABER-GPU/src/poly.cu:209-358, the reference's
// mode 1): the same window, one 32-bit multiply-add per coefficient pair instead of dp2a.
template <int L, int MODE, bool I32 = false>
__device__ __forceinline__ void product_dp4a_cta(const Inst &v, uint8_t *sm, bool sliced = false) {
  using Y = PL<L>;
  constexpr int NO = n_out<L, MODE>();
  const int tid = threadIdx.x;
  load_operands<L, MODE>(v, sm, sliced);
  __syncthreads();
  build_seq<L>(sm);
  __syncthreads();
  const int base = 255 - tid, wb = base >> 2, sh = 8 * (base & 3);
  int acc[NO];
#pragma unroll
  for (int o = 0; o < NO; o++) acc[o] = 0;
  for (int j = 0; j < L; j++) {
    const uint32_t *rw = reinterpret_cast<const uint32_t *>(sm + Y::SEQ + j * Y::SEQ_STRIDE);
    const uint2 *pp[NO];
#pragma unroll
    for (int o = 0; o < NO; o++) pp[o] = reinterpret_cast<const uint2 *>(pub_poly<L, MODE>(sm, o, j));
    uint32_t w0 = rw[wb];
#pragma unroll 4
    for (int mq = 0; mq < SN / 4; mq++) {
      const uint32_t w1 = rw[wb + mq + 1];
      const int win = (int)__funnelshift_r(w0, w1, sh);
      w0 = w1;
      if (I32) {
        const int s0 = (int)(int8_t)win, s1 = (int)(int8_t)(win >> 8), s2 = (int)(int8_t)(win >> 16),
                  s3 = win >> 24;
#pragma unroll
        for (int o = 0; o < NO; o++) {
          const uint2 pw = pp[o][mq];
          acc[o] += (int)(pw.x & 0xFFFFu) * s0 + (int)(pw.x >> 16) * s1 + (int)(pw.y & 0xFFFFu) * s2 +
                    (int)(pw.y >> 16) * s3;
        }
      } else {
#pragma unroll
        for (int o = 0; o < NO; o++) {
          const uint2 pw = pp[o][mq];
          acc[o] = dp2a_hi((int)pw.y, win, dp2a_lo((int)pw.x, win, acc[o]));
        }
      }
    }
  }
  uint16_t *res = reinterpret_cast<uint16_t *>(sm + Y::RES);
#pragma unroll
  for (int o = 0; o < NO; o++) res[o * SN + tid] = (uint16_t)acc[o];
  __syncthreads();
  epilogue<L, MODE>(v, sm);
  __syncthreads();
}

// ---------------------------------------------------------------- tcgen05 form
// Four barrier-separated phases per instance (256 threads; the packed operands are staged):
//   1  operands: every thread unpacks 16 coefficients, the public ones straight into the bytes of
//      the B operand, the secret ones into the sequences E_j (their negatives and themselves)
//   2  the Hankel core matrices from E_j
//   3  one thread's MMAs; read-back, rounding (coefficient = thread), results to shared memory
//   4  packing: 16 results (5 words at 10 bits) per thread, to global memory or compared there
// What bounds it: the tensor pipe's operand reads.  An MMA step of 128 x 32 bytes of A takes about 45
// cycles whatever N is (the math itself 6 % of the pipe), 36 steps an encaps at l = 3: two thirds of the
// time at 16,384 instances, the rest exposed phases of a few hundred cycles.  The form before had 48 steps,
// eight barriers (u16 polynomials, secret sequences, rounding and byte-wise packing as passes of their
// own) and 6,470 warp instructions an encaps; this one has four barriers and 3,900.  Product stage of
// encaps at l = 2 / 3 / 4, 16,384 / 16,384 / 8,192 instances: 137 / 184 / 156 -> 93 / 123 / 111 us.
//
// E_j[e] = s_ext[e - 256], e in [0, 512): -s[e] below 256, s[e - 256] above.  T'[i][k'] = s_ext[i + k' - 255]
// = E[i + k' + 1], so core matrix t = mi + 2 ki has rows H[t][r][c] = E[8 t + r + c + 1].

// 16 fields of BITS bits starting OFF bits into w, as bytes in reversed order: lo[q] holds the low
// bytes of fields 15 - 4q (byte 0) .. 12 - 4q, hi[q] their upper bits.
template <int BITS, int OFF>
__device__ __forceinline__ void reversed_bytes(const uint32_t *w, uint4 &lo, uint4 &hi) {
  constexpr int NW = (OFF + 16 * BITS + 31) / 32;
  uint32_t r[NW + 1], l[4], h[4];
#pragma unroll
  for (int k = 0; k < NW; k++) r[k] = w[k];
  r[NW] = 0;
  auto field = [&](int i) {
    const int bit = OFF + i * BITS;
    return __funnelshift_r(r[bit >> 5], r[(bit >> 5) + 1], bit & 31);
  };
#pragma unroll
  for (int q = 0; q < 4; q++) {
    const uint32_t a = field(15 - 4 * q), b = field(14 - 4 * q), c = field(13 - 4 * q), d = field(12 - 4 * q);
    const uint32_t ab = prmt(a, b, 0x5140), cd = prmt(c, d, 0x5140);  // low bytes, then second bytes
    l[q] = prmt(ab, cd, 0x5410);
    h[q] = prmt(ab, cd, 0x7632) & (((1u << (BITS - 8)) - 1u) * 0x01010101u);
  }
  lo = make_uint4(l[0], l[1], l[2], l[3]);
  hi = make_uint4(h[0], h[1], h[2], h[3]);
}

// 16 secret coefficients (words q = 0..3 of 4 int8 each) of polynomial j, group g, into E_j.
template <int L>
__device__ __forceinline__ void store_secret(uint8_t *sm, int j, int g, uint4 s) {
  using Y = TL<L>;
  uint8_t *e = sm + Y::SEQ + j * Y::SEQ_STRIDE + 16 * g;
  *reinterpret_cast<uint4 *>(e) = make_uint4(neg_bytes(s.x), neg_bytes(s.y), neg_bytes(s.z), neg_bytes(s.w));
  *reinterpret_cast<uint4 *>(e + SN) = s;
}

// Phase 1.
template <int L, int MODE>
__device__ __forceinline__ void tc_operands(uint8_t *sm) {
  using P = SP<L>;
  using Y = TL<L>;
  constexpr int NO = n_out<L, MODE>();
  constexpr bool INNER = MODE == PM_DEC_INNER;
  constexpr int NA = INNER ? 0 : L * L * 16, NP = MODE == PM_KEYPAIR ? 0 : L * 16, NS = L * 16;
  // chunk of 16 columns K of row n: K = 256 j + 255 - c for coefficient c
  auto store_public = [&](int o, int j, int g, uint4 lo, uint4 hi) {
    uint8_t *d = sm + Y::BOP + (16 * j + 15 - g) * Y::CHUNK;
    const int nl = o, nh = o + NO;
    *reinterpret_cast<uint4 *>(d + (nl >> 3) * Y::BOP_GROUP + (nl & 7) * 16) = lo;
    *reinterpret_cast<uint4 *>(d + (nh >> 3) * Y::BOP_GROUP + (nh & 7) * 16) = hi;
  };
  for (int x = threadIdx.x; x < NA + NP + NS; x += 256) {
    if (x < NA) {  // A: 13 bits; an odd group starts in the middle of a word
      const int m = x >> 4, g = x & 15, row = m / L, col = m - row * L;
      const int o = MODE == PM_KEYPAIR ? col : row, j = MODE == PM_KEYPAIR ? row : col;  // keypair: A^T s
      const uint32_t *w = reinterpret_cast<const uint32_t *>(sm + Y::ST_A) + 104 * m + 13 * (g >> 1);
      uint4 lo, hi;
      if (g & 1) reversed_bytes<EQ, 16>(w + 6, lo, hi);
      else reversed_bytes<EQ, 0>(w, lo, hi);
      store_public(o, j, g, lo, hi);
    } else if (x < NA + NP) {  // b (b' in the inner product): 10 bits
      const int y = x - NA, j = y >> 4, g = y & 15;
      uint4 lo, hi;
      reversed_bytes<EP, 0>(reinterpret_cast<const uint32_t *>(sm + (INNER ? Y::ST_CT : Y::ST_P)) + 5 * y, lo, hi);
      store_public(NO - 1, j, g, lo, hi);
    } else {
      const int y = x - NA - NP, j = y >> 4, g = y & 15;
      uint4 s;
      if (INNER) {  // low bytes of the 13-bit fields (|s| < 128), in order
        const uint32_t *w = reinterpret_cast<const uint32_t *>(sm + Y::ST_SK) + 13 * (y >> 1);
        uint4 hi;
        if (g & 1) reversed_bytes<EQ, 16>(w + 6, s, hi);
        else reversed_bytes<EQ, 0>(w, s, hi);
        s = make_uint4(prmt(s.w, 0, 0x0123), prmt(s.z, 0, 0x0123), prmt(s.y, 0, 0x0123), prmt(s.x, 0, 0x0123));
      } else {  // CBD_mu
        const uint32_t *w = reinterpret_cast<const uint32_t *>(sm + Y::ST_S) + (P::MU / 2) * y;
        uint32_t o[4];
        if (P::MU == 8) {  // a coefficient per byte: popcounts of its nibbles side by side
#pragma unroll
          for (int q = 0; q < 4; q++) {
            uint32_t t = w[q];
            t = t - ((t >> 1) & 0x55555555u);
            t = (t & 0x33333333u) + ((t >> 2) & 0x33333333u);
            o[q] = (((t & 0x0F0F0F0Fu) | 0x80808080u) - ((t >> 4) & 0x0F0F0F0Fu)) ^ 0x80808080u;
          }
        } else {
          constexpr uint32_t hm = (1u << (P::MU / 2)) - 1u;
          unpack_words<P::MU, 16>(w, [&](int i, uint32_t t) {
            const uint32_t c = (uint32_t)(__popc(t & hm) - __popc((t >> (P::MU / 2)) & hm)) & 0xFFu;
            if ((i & 3) == 0) o[i >> 2] = c;
            else o[i >> 2] |= c << (8 * (i & 3));
          });
        }
        s = make_uint4(o[0], o[1], o[2], o[3]);
      }
      store_secret<L>(sm, j, g, s);
    }
  }
}

// Phase 2.  Thread (j, r, part): row r of core matrices t = part, part + STEP, ... of secret j.
template <int L>
__device__ __forceinline__ void tc_hankel(uint8_t *sm) {
  using Y = TL<L>;
  const int r = threadIdx.x & 7, sh = 8 * ((r + 1) & 3);
  int j = 0, t = threadIdx.x >> 3;
  while (j < L) {
    const uint32_t *sw =
        reinterpret_cast<const uint32_t *>(sm + Y::SEQ + j * Y::SEQ_STRIDE) + 2 * t + ((r + 1) >> 2);
    const uint32_t x0 = sw[0], x1 = sw[1], x2 = sw[2], x3 = sw[3], x4 = sw[4];
    *reinterpret_cast<uint4 *>(sm + Y::HANK + j * Y::HANK_STRIDE + t * 128 + r * 16) =
        make_uint4(__funnelshift_r(x0, x1, sh), __funnelshift_r(x1, x2, sh), __funnelshift_r(x2, x3, sh),
                   __funnelshift_r(x3, x4, sh));
    t += 32;
    if (t >= 62) {
      t -= 62;
      j++;
    }
  }
}

// Packs N results of BITS bits (u16 at v, 16-byte aligned) into N * BITS / 32 words.
template <int BITS, int N>
__device__ __forceinline__ void pack_words(const uint16_t *v, uint32_t (&out)[N * BITS / 32]) {
  uint32_t w[N / 2];
#pragma unroll
  for (int q = 0; q < N / 8; q++) {
    const uint4 x = reinterpret_cast<const uint4 *>(v)[q];
    w[4 * q] = x.x;
    w[4 * q + 1] = x.y;
    w[4 * q + 2] = x.z;
    w[4 * q + 3] = x.w;
  }
#pragma unroll
  for (int k = 0; k < N * BITS / 32; k++) out[k] = 0;
#pragma unroll
  for (int i = 0; i < N; i++) {
    const uint32_t x = (i & 1) ? w[i >> 1] >> 16 : w[i >> 1] & 0xFFFFu;
    const int bit = i * BITS, k = bit >> 5, sh = bit & 31;
    out[k] |= x << sh;
    if (sh + BITS > 32) out[k + 1] |= x >> (32 - sh);
  }
}

// Phases 1..4 on staged operands (a CTA barrier after the staging, by the caller); the MMAs'
// completion is on the mbarrier at TL::BAR, parity `phase`.  TMEM columns [tbase, tbase + 32) must
// be allocated.  Returns false if the bounded wait expired.  The caller may stage the next
// instance's operands at once (they go where the Hankel matrices were), not other layouts before a CTA
// barrier.
template <int L, int MODE>
__device__ __forceinline__ bool tc_product(const Inst &v, uint8_t *sm, uint32_t tbase, uint32_t *err, uint32_t phase) {
  using P = SP<L>;
  using Y = TL<L>;
  constexpr int NO = n_out<L, MODE>();
  constexpr int NPAD = 2 * NO <= 8 ? 8 : 16;
  constexpr bool INNER = MODE == PM_DEC_INNER;
  uint64_t *bar = reinterpret_cast<uint64_t *>(sm + Y::BAR);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  tc_operands<L, MODE>(sm);
  uint32_t cm = 0;  // decaps inner: this coefficient's et bits of c_m (before the Hankel matrices take the place)
  if (INNER) cm = unpack_smem(sm + Y::ST_CT + P::POLYVECCOMP, tid, P::ET);
  __syncthreads();
  tc_hankel<L>(sm);
  fence_proxy_async_smem();
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  if (tid == 0) {
    constexpr uint32_t idesc = idesc_i8(128, NPAD, true, false, false, false);
    // Base descriptors; a step moves only the start-address field (address / 16, low word).  The
    // B operand's eight-row groups are eight chunks (128 columns of K) apart for the double steps.
    const uint64_t a0 = sdesc(smem_u32(sm + Y::HANK), 256, 128),
                   b0 = sdesc(smem_u32(sm + Y::BOP), Y::CHUNK, NPAD == 8 ? 8 * Y::CHUNK : Y::BOP_GROUP);
    auto step = [&](int d, int ks, int j, int chunk, uint32_t id, uint32_t acc) {
      mma_i8(tbase + d, a0 + (uint64_t)((j * Y::HANK_STRIDE + 4 * ks * 128) >> 4),
             b0 + (uint64_t)(((16 * j + chunk) * Y::CHUNK) >> 4), id, acc);
    };
    if constexpr (NPAD == 8) {
      // Rows i + 128 of the Hankel block are rows i, 128 columns on: D[i + 128] = sum over K'' of
      // E[i + K'' + 1] P[K'' - 128].  With K'' in 0 .. 383 one A tile serves both halves of the
      // coefficients, as 16 columns where both have terms (lower half in columns 8..15): 12
      // tiles of A per secret instead of 16.  Reading A (4 KB a step) is what the MMAs cost.
      constexpr uint32_t id16 = idesc_i8(128, 16, true, false, false, false);
#pragma unroll
      for (int j = 0; j < L; j++) {
#pragma unroll
        for (int ks = 8; ks < 12; ks++) step(0, ks, j, 2 * ks - 8, idesc, (j | (ks - 8)) ? 1u : 0u);
#pragma unroll
        for (int ks = 0; ks < 4; ks++) step(8, ks, j, 2 * ks, idesc, (j | ks) ? 1u : 0u);
#pragma unroll
        for (int ks = 4; ks < 8; ks++) step(0, ks, j, 2 * ks - 8, id16, 1u);
      }
    } else {
      // Rolled: unrolled, the persistent kernel keeps the descriptors of all 64 steps across its loop,
      // in spilled registers.
#pragma unroll 1
      for (int mj = 0; mj < 2 * L; mj++) {
        const int mt = mj / L, j = mj - mt * L;
#pragma unroll
        for (int ks = 0; ks < 8; ks++) step(mt * NPAD, 4 * mt + ks, j, 2 * ks, idesc, (j | ks) ? 1u : 0u);
      }
    }
    mma_commit(bar);
  }
  // While the MMAs run: the packing jobs' ciphertext words (comparison), sk's 13-bit secret (keypair).
  constexpr int NW = EP * 16 / 32;                        // 5 words of 16 results
  constexpr int VG = P::ET == 4 ? 8 : P::ET == 3 ? 32 : 16, VW = P::ET * VG / 32, VJ = SN / VG;  // c_m: per job
  const bool pjob = tid < L * 16, vjob = MODE != PM_KEYPAIR && !INNER && tid >= L * 16 && tid < L * 16 + VJ;
  const int vx = tid - L * 16;
  uint32_t have[NW];
  if (MODE == PM_DEC_CMP) {
    const uint32_t *c = reinterpret_cast<const uint32_t *>(v.ct);
    if (pjob) {
#pragma unroll
      for (int k = 0; k < NW; k++) have[k] = c[NW * tid + k];
    } else if (vjob) {
#pragma unroll
      for (int k = 0; k < VW; k++) have[k] = c[P::POLYVECCOMP / 4 + VW * vx + k];
    }
  }
  if (MODE == PM_KEYPAIR && tid >= 128 && tid < 128 + L * 16) {  // 16 coefficients: 26 bytes
    const int y = tid - 128;
    const uint32_t *sw = reinterpret_cast<const uint32_t *>(sm + Y::SEQ + (y >> 4) * Y::SEQ_STRIDE + SN + 16 * (y & 15));
    uint32_t out[7] = {0, 0, 0, 0, 0, 0, 0};
#pragma unroll
    for (int i = 0; i < 16; i++) {
      const uint32_t x = (uint32_t)((int32_t)(sw[i >> 2] << (24 - 8 * (i & 3))) >> 24) & 0x1FFFu;
      const int bit = i * EQ, k = bit >> 5, sh = bit & 31;
      out[k] |= x << sh;
      if (sh + EQ > 32) out[k + 1] |= x >> (32 - sh);
    }
    uint16_t *d = reinterpret_cast<uint16_t *>(v.sk + 26 * y);
#pragma unroll
    for (int k = 0; k < 13; k++) d[k] = (uint16_t)(out[k >> 1] >> (16 * (k & 1)));
  }
  const bool ok = mbar_wait(bar, phase);
  if (!ok && lane == 0) atomicOr(err, DEV_ERR_TIMEOUT);
  tc_fence_after();
  // Warp w reads TMEM lanes 32 (w % 4) .. of coefficient half w / 4: coefficient = tid.
  uint32_t r[16];
  tmem_ld16(tbase + ((uint32_t)((warp & 3) * 32) << 16) + (NPAD == 8 ? 8 - 8 * (warp >> 2) : NPAD * (warp >> 2)), r);
  tmem_wait_ld();
  tc_fence_before();
  if (INNER) {
    const uint32_t x = r[0] + (r[1] << 8);
    const uint32_t m = __ballot_sync(0xffffffffu, ((x + P::H2 - (cm << (EP - P::ET))) >> (EP - 1)) & 1u);
    if (lane == 0) reinterpret_cast<uint32_t *>(v.scr + Scr<L>::MTXT)[warp] = m;
    if (tid == 0) *v.fail = 0;  // the re-encryption's comparison ORs into it
    return ok;
  }
  uint16_t *res = reinterpret_cast<uint16_t *>(sm + Y::RES);
#pragma unroll
  for (int o = 0; o < NO; o++) {
    const uint32_t x = r[o] + (r[NO + o] << 8) + P::H1;
    if (MODE == PM_KEYPAIR || o < L) {
      res[o * SN + tid] = (uint16_t)((x >> (EQ - EP)) & 0x3FFu);
    } else {
      const uint32_t mb = (sm[Y::CM + (tid >> 3)] >> (tid & 7)) & 1u;
      res[o * SN + tid] = (uint16_t)(((x - (mb << (EP - 1))) >> (EP - P::ET)) & ((1u << P::ET) - 1u));
    }
  }
  __syncthreads();
  uint8_t *dst = MODE == PM_KEYPAIR ? v.pk : v.ct;
  uint32_t diff = 0;
  if (pjob) {
    uint32_t w[NW];
    pack_words<EP, 16>(res + 16 * tid, w);
#pragma unroll
    for (int k = 0; k < NW; k++) {
      if (MODE == PM_DEC_CMP) diff |= w[k] ^ have[k];
      else reinterpret_cast<uint32_t *>(dst)[NW * tid + k] = w[k];
    }
  } else if (vjob) {
    uint32_t w[VW];
    pack_words<P::ET, VG>(res + L * SN + VG * vx, w);
#pragma unroll
    for (int k = 0; k < VW; k++) {
      if (MODE == PM_DEC_CMP) diff |= w[k] ^ have[k];
      else reinterpret_cast<uint32_t *>(dst + P::POLYVECCOMP)[VW * vx + k] = w[k];
    }
  }
  if (MODE == PM_DEC_CMP && __any_sync(0xffffffffu, diff != 0) && lane == 0) atomicOr(v.fail, 1u);
  return ok;
}

// One instance on a CTA whose TMEM columns [tbase, tbase + 32) are allocated; the mbarrier is
// initialised here.
template <int L, int MODE>
__device__ __forceinline__ bool product_tc_cta(const Inst &v, uint8_t *sm, uint32_t tbase, uint32_t *err,
                                               bool sliced = false) {
  using Y = TL<L>;
  uint64_t *bar = reinterpret_cast<uint64_t *>(sm + Y::BAR);
  if (threadIdx.x == 0) {
    mbar_init(bar, 1);
    fence_mbar_init();
  }
  stage_operands<L, MODE, Y>(v, sm, sliced);
  __syncthreads();
  const bool ok = tc_product<L, MODE>(v, sm, tbase, err, 0);
  __syncthreads();
  if (threadIdx.x == 0 && ok) mbar_inval(bar);
  return ok;
}

}  // namespace sdev
}  // namespace dpkem

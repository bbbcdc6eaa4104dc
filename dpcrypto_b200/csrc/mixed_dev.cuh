// Device side of the persistent mixed-scheme kernels (mixed.cu: one launch over a planned
// task list; serve.cu: a long-lived service fed from a host-written request ring): stage
// codes and kinds, per-request scratch records, the request record the kernels read, and
// the stage bodies (one instance per thread, a warp per instance, or a CTA per instance)
// built from the routines the batched kernels use.
#pragma once
#include <cuda_runtime.h>

#include <algorithm>

#include "coins_dev.cuh"
#include "frodo_chain.cuh"
#include "frodo_dev.cuh"
#include "saber_dev.cuh"

namespace dpkem {
namespace mixed {

// ---- stage codes: scheme * 128 + op * 32 + stage * 4 + form ----
__host__ __device__ constexpr int code_of(int scheme, int op, int stage, int form) {
  return scheme * 128 + op * 32 + stage * 4 + form;
}
__host__ __device__ constexpr int scheme_of(int code) { return code >> 7; }
__host__ __device__ constexpr int op_of(int code) { return (code >> 5) & 3; }
__host__ __device__ constexpr int stage_of(int code) { return (code >> 2) & 7; }
__host__ __device__ constexpr int form_of(int code) { return code & 3; }

// Stage kinds: 0 = thread (one instance per thread), 2 = thread with two roles (instance
// t on threads t and t + 128: Saber's two prologue sponges, Frodo decaps' prologue and
// ciphertext pre-absorb), 1 = CTA (one instance per task).
enum Kind : int { K_THREAD = 0, K_CTA = 1, K_THREAD2 = 2 };

// Task code flag (above the stage code's 10 bits, masked off before decoding): a
// thread-level stage run on a warp per instance (and role): the Keccak
// sponges spread over the warp's lanes (keccak25.cuh), 8 instances per task (4 for two-role
// stages).  The planner uses it for groups small enough that one thread per instance would
// leave the GPU idle (knob mixed_warp_max).
constexpr int kWarpTask = 1 << 10;
static_assert(code_of(4, 3, 7, 3) < kWarpTask, "stage codes must stay below the warp-task flag");

// A FrodoKEM prologue or hash stage on ten lanes per state (frodo_chain.cuh): a task is as many
// instances as one CTA's warps take at once, so a request's 232-348 dependent permutations cost 0.5-0.8 ms
// instead of the 2-3 ms of one thread beside the product CTAs.
constexpr int kChainTask = 1 << 11;
__host__ __device__ constexpr bool chain_stage(int scheme, int op, int stage) {
  return scheme <= 1 && (op == OP_DEC ? stage == 1 : stage != 1);
}
__host__ __device__ constexpr int chain_per(int op, int stage) { return op == OP_DEC ? 6 : stage == 0 ? 12 : 24; }

__host__ __device__ constexpr int nstages(int scheme, int op) { return op == OP_DEC ? 4 : 3; }

__host__ __device__ constexpr int kind_of(int scheme, int op, int stage) {
  if (scheme <= 1) {  // FrodoKEM-976, SHAKE (0) or AES (1)
    if (op == OP_DEC) return stage == 0 || stage == 2 ? K_CTA : stage == 1 ? K_THREAD2 : K_THREAD;
    return stage == 1 ? K_CTA : K_THREAD;
  }
  if (op == OP_DEC) return stage == 1 ? K_THREAD2 : stage == 3 ? K_THREAD : K_CTA;
  return stage == 0 ? K_THREAD2 : stage == 1 ? K_CTA : K_THREAD;
}

// Completed-role count an instance must show before `stage` may start.
__host__ __device__ constexpr uint32_t threshold(int scheme, int op, int stage) {
  uint32_t t = 0;
  for (int s = 0; s < stage; s++) t += kind_of(scheme, op, s) == K_THREAD2 ? 2u : 1u;
  return t;
}

// ---- per-request scratch records (256-byte multiples so no line is shared) ----
constexpr size_t kFrodoRec = 31744;  // rw 31,360 | k 24 | mu 24 | fail 4 (+12) | sponge 200
constexpr size_t kFrodoK = frodo::RW * 2, kFrodoMu = kFrodoK + 24, kFrodoFail = kFrodoMu + 24;
constexpr size_t kFrodoHs = kFrodoFail + 16;
constexpr size_t kFrodoCoins = kFrodoHs + 200;  // 64 B of device-drawn coins
static_assert(kFrodoCoins + 64 <= kFrodoRec, "Frodo record too small");

// Saber record: scratch | fail word | two 96-byte coin slots (one per prologue role).
__host__ __device__ inline size_t saber_scr_bytes(int level) {
  return level == 2 ? sdev::Scr<2>::BYTES : level == 3 ? sdev::Scr<3>::BYTES : sdev::Scr<4>::BYTES;
}
__host__ __device__ inline size_t saber_coins_off(int level) { return (saber_scr_bytes(level) + 4 + 7) & ~(size_t)7; }
__host__ __device__ inline size_t saber_rec_bytes(int level) {
  return (saber_coins_off(level) + 192 + 255) & ~(size_t)255;
}

struct DevReq {
  int32_t scheme, op;
  const uint8_t *in0, *in1;
  uint8_t *out0, *out1;
  uint8_t *scr;
  uint64_t coin_index;  // with gen: coins = SHAKE256(key || LE64(coin_index) || tag), drawn into in0
  uint32_t gen;
  uint32_t ticket;  // service requests: the ticket whose completion the last stage reports
};

// Draws a request's coins into `dst` (the first stage of a keypair / encaps whose request
// carried none): tag "kp" / "enc", length of the scheme's coins.
__device__ __forceinline__ void draw_coins(const CoinKey &key, const DevReq &r, uint8_t *dst) {
  const uint8_t kp[2] = {'k', 'p'}, enc[3] = {'e', 'n', 'c'};
  const bool is_kp = r.op == OP_KEYPAIR;
  const int len = r.scheme <= 1 ? (is_kp ? frodo::KP_COINS : frodo::ENC_COINS) : (is_kp ? 96 : 32);
  coin_generate(key, r.coin_index, is_kp ? kp : enc, is_kp ? 2 : 3, len, dst);
}

__device__ __forceinline__ fdev::Inst frodo_view(const DevReq &r) {
  fdev::Inst v{};
  const bool kp = r.op == OP_KEYPAIR, enc = r.op == OP_ENC;
  v.coins = kp || enc ? r.in0 : nullptr;
  v.pk = kp ? r.out0 : enc ? const_cast<uint8_t *>(r.in1) : nullptr;
  v.sk = kp ? r.out1 : enc ? nullptr : const_cast<uint8_t *>(r.in1);
  v.ct = enc ? r.out0 : kp ? nullptr : const_cast<uint8_t *>(r.in0);
  v.ss = enc ? r.out1 : kp ? nullptr : r.out0;
  v.rw = reinterpret_cast<uint16_t *>(r.scr);
  v.kk = r.scr + kFrodoK;
  v.mu = r.scr + kFrodoMu;
  v.fail = reinterpret_cast<uint32_t *>(r.scr + kFrodoFail);
  v.hs = reinterpret_cast<uint2 *>(r.scr + kFrodoHs);
  return v;
}

template <int L>
__device__ __forceinline__ sdev::Inst saber_view(const DevReq &r) {
  sdev::Inst v{};
  const bool kp = r.op == OP_KEYPAIR, enc = r.op == OP_ENC;
  v.coins = kp || enc ? r.in0 : nullptr;
  v.pk = kp ? r.out0 : enc ? const_cast<uint8_t *>(r.in1) : nullptr;
  v.sk = kp ? r.out1 : enc ? nullptr : const_cast<uint8_t *>(r.in1);
  v.ct = enc ? r.out0 : kp ? nullptr : const_cast<uint8_t *>(r.in0);
  v.ss = enc ? r.out1 : kp ? nullptr : r.out0;
  v.scr = r.scr;
  v.fail = reinterpret_cast<uint32_t *>(r.scr + sdev::Scr<L>::BYTES);
  return v;
}

__device__ __forceinline__ uint32_t ld_acquire(const uint32_t *p) {
  uint32_t v;
  asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}

// Spin loads: a relaxed load reads L2 (these kernels bypass L1) without the L1 invalidation
// an acquire load performs on every iteration, which would evict the register spills of the
// CTA sharing the SM; a spin that succeeds then fences once (__threadfence), which orders
// the loads after it behind the value it saw.
__device__ __forceinline__ uint32_t ld_relaxed(const uint32_t *p) {
  uint32_t v;
  asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}


// ---- stage bodies as calls ----
// Each body is a function of its own: inlined into one kernel, the compiler allocates registers for all of
// them together (8.6 KB of spill stores), and a change to one stage moved the spills of the others: the
// Saber product's new form made a mix of 4,096 requests 14 % slower (7.09 -> 8.08 ms) although that
// stage is faster; with calls the same mix takes 6.84 ms.
template <int OP>
static __device__ __noinline__ void call_frodo_prologue(const fdev::Inst &v) {
  if constexpr (OP == OP_KEYPAIR) fdev::kp_prologue_inst(v);
  else fdev::prologue_inst<OP>(v);
}
template <int OP>
static __device__ __noinline__ void call_frodo_hash(const fdev::Inst &v) {
  if constexpr (OP == OP_KEYPAIR) fdev::pk_hash_inst(v);
  else fdev::ss_inst<OP>(v);
}
static __device__ __noinline__ void call_frodo_absorb(const fdev::Inst &v) { fdev::ct_absorb_inst(v); }
template <int OP>
static __device__ __noinline__ void call_frodo_prologue_warp(const fdev::Inst &v) {
  const msp::Multi<1> s(nullptr);
  if constexpr (OP == OP_KEYPAIR) fdev::kp_prologue_multi(v, s, true);
  else fdev::prologue_multi<msp::Multi<1>, OP>(v, s, true);
}
template <int OP>
static __device__ __noinline__ void call_frodo_hash_warp(const fdev::Inst &v) {
  const msp::Multi<1> s(nullptr);
  if constexpr (OP == OP_KEYPAIR) fdev::pk_hash_multi(v, s, true);
  else fdev::ss_multi<msp::Multi<1>, OP>(v, s, true);
}
static __device__ __noinline__ void call_frodo_absorb_warp(const fdev::Inst &v) {
  fdev::ct_absorb_multi(v, msp::Multi<1>(nullptr), true);
}
template <int L, int OP>
static __device__ __noinline__ void call_saber_prologue(const sdev::Inst &v, int role) {
  sdev::prologue_inst<L, OP>(v, role);
}
template <int L, int OP>
static __device__ __noinline__ void call_saber_finish(const sdev::Inst &v) {
  sdev::finish_inst<L, OP>(v);
}
template <int L, int OP>
static __device__ __noinline__ void call_saber_prologue_warp(const sdev::Inst &v, int role) {
  sdev::prologue_multi<msp::Multi<1>, L, OP>(v, msp::Multi<1>(nullptr), role, true);
}
template <int L, int OP>
static __device__ __noinline__ void call_saber_finish_warp(const sdev::Inst &v) {
  const msp::Multi<1> s(nullptr);
  if constexpr (OP == OP_KEYPAIR) sdev::finish_kp_multi<msp::Multi<1>, L>(v, s, true);
  else sdev::finish_enc_multi<msp::Multi<1>, L>(v, s, true);
}
template <int L, int MODE, int FORM>
static __device__ __noinline__ void call_saber_product(const sdev::Inst &v, uint8_t *smem, uint32_t tbase, uint32_t *err) {
  if constexpr (FORM == FORM_TC) sdev::product_tc_cta<L, MODE>(v, smem, tbase, err);
  else sdev::product_dp4a_cta<L, MODE, FORM == FORM_INT32>(v, smem);
}
template <int OP, int FORM, int NST, class G>
static __device__ __noinline__ void call_frodo_product(const fdev::Inst &v, uint8_t *smem, uint32_t tbase, uint32_t *err) {
  if constexpr (OP == OP_KEYPAIR) {
    if constexpr (FORM == FORM_TC) fdev::kp_as_tc_cta<NST == 2 ? fdev::KPT_NST : 1, G>(v, smem, tbase, err);
    else fdev::kp_as_dp4a_cta<FORM == FORM_INT32, G>(v, smem);
  } else {
    if constexpr (FORM == FORM_TC) fdev::sa_tc_cta<OP, NST, G>(v, smem, tbase, err);
    else fdev::sa_dp4a_cta<OP, FORM == FORM_INT32, G>(v, smem);
  }
}
static __device__ __noinline__ void call_frodo_dec_w(const fdev::Inst &v, uint8_t *smem) { fdev::dec_w_cta(v, smem); }

// Requests of a chain task, copied to shared memory.
struct ReqInsts {
  const DevReq *rq;
  int n;
  __device__ __forceinline__ fdev::Inst operator()(int i) const { return frodo_view(rq[i]); }
};

template <int ROLE, int CW>
__device__ __forceinline__ void frodo_chain(const ReqInsts &src, uint8_t *smem) {
  using namespace fchain;
  const int warp = threadIdx.x >> 5;
  if (warp >= 2 * CW) return;
  const bool helper = warp >= CW;
  const int w = helper ? (warp - CW + 2) % CW : warp;
  if (3 * w >= src.n) return;
  constexpr int words = ROLE == R_KEYPAIR ? 2 * HALF : frodo::RW;
  Exchange &x = reinterpret_cast<Exchange *>(smem)[w];
  uint8_t *xbuf = smem + 4 * sizeof(Exchange) + w * k10::kSmemPerWarp;
  if (helper) helper_warp<ROLE, false>(src, 3 * w, words, x, w);
  else chain_warp<ROLE, false>(src, 3 * w, (words + 67) / 68 - 1, false, x, xbuf, w);
}

// One chain task (the whole CTA, 256 threads).
template <int OP>
static __device__ __noinline__ void call_frodo_chain(const ReqInsts &src, uint8_t *smem) {
  if constexpr (OP == OP_KEYPAIR) {
    if ((int)threadIdx.x < src.n) fchain::write_seed_a(src(threadIdx.x));
    __syncthreads();
    frodo_chain<fchain::R_KEYPAIR, 4>(src, smem);
  } else if constexpr (OP == OP_ENC) {
    frodo_chain<fchain::R_ENC, 4>(src, smem);
  } else {
    const int warp = threadIdx.x >> 5;
    frodo_chain<fchain::R_DEC, 2>(src, smem);
    if (warp >= 4 && 3 * (warp - 4) < src.n) {  // the ciphertext's part of the final hash
      using S = msp::Multi<10>;
      const S s(smem + 4 * sizeof(fchain::Exchange) + warp * S::SMEM_PER_WARP);
      const int i = 3 * (warp - 4) + s.state();
      fdev::ct_absorb_multi<S>(src(i < src.n ? i : src.n - 1), s, i < src.n);
    }
  }
}
template <int OP>
static __device__ __noinline__ void call_frodo_hash_ten(const ReqInsts &src, uint8_t *smem) {
  using S = msp::Multi<10>;
  const int warp = threadIdx.x >> 5;
  if (3 * warp >= src.n) return;
  const S s(smem + warp * S::SMEM_PER_WARP);
  const int i = 3 * warp + s.state();
  const fdev::Inst v = src(i < src.n ? i : src.n - 1);
  if constexpr (OP == OP_KEYPAIR) fdev::pk_hash_multi<S>(v, s, i < src.n);
  else fdev::ss_multi<S, OP>(v, s, i < src.n);
}
constexpr int kChainReqs = 32 << 10;  // where a chain task's requests lie in shared memory

__device__ __forceinline__ void chain_task(const CoinKey &key, int code, int count, uint8_t *smem) {
  const int op = op_of(code), stage = stage_of(code);
  const ReqInsts src{reinterpret_cast<const DevReq *>(smem + kChainReqs), count};
  if (stage == 0 && (int)threadIdx.x < count && src.rq[threadIdx.x].gen)
    draw_coins(key, src.rq[threadIdx.x], const_cast<uint8_t *>(src.rq[threadIdx.x].in0));
  __syncthreads();
  if (op == OP_KEYPAIR) {
    if (stage == 0) call_frodo_chain<OP_KEYPAIR>(src, smem);
    else call_frodo_hash_ten<OP_KEYPAIR>(src, smem);
  } else if (op == OP_ENC) {
    if (stage == 0) call_frodo_chain<OP_ENC>(src, smem);
    else call_frodo_hash_ten<OP_ENC>(src, smem);
  } else {
    call_frodo_chain<OP_DEC>(src, smem);
  }
}

template <int L>
__device__ __forceinline__ void saber_thread(const CoinKey &key, int op, int stage, const DevReq &r, int role) {
  sdev::Inst v = saber_view<L>(r);
  if (r.gen && stage == 0 && op != OP_DEC) {
    // each prologue role draws its own copy (role 1 into the second slot), so neither
    // waits for the other; later stages read the first slot through in0
    uint8_t *slot = const_cast<uint8_t *>(r.in0) + (role ? 96 : 0);
    if (role == 0 || op == OP_KEYPAIR) draw_coins(key, r, slot);
    v.coins = slot;
  }
  if (op == OP_KEYPAIR) {
    if (stage == 0) call_saber_prologue<L, OP_KEYPAIR>(v, role);
    else call_saber_finish<L, OP_KEYPAIR>(v);
  } else if (op == OP_ENC) {
    if (stage == 0) call_saber_prologue<L, OP_ENC>(v, role);
    else call_saber_finish<L, OP_ENC>(v);
  } else {
    if (stage == 1) call_saber_prologue<L, OP_DEC>(v, role);
    else call_saber_finish<L, OP_DEC>(v);
  }
}

// The same stages on a warp per instance (a warp-wide call: every lane runs it).
template <int L>
__device__ __forceinline__ void saber_warp(const CoinKey &key, int op, int stage, const DevReq &r, int role) {
  sdev::Inst v = saber_view<L>(r);
  if (r.gen && stage == 0 && op != OP_DEC) {
    uint8_t *slot = const_cast<uint8_t *>(r.in0) + (role ? 96 : 0);
    if ((role == 0 || op == OP_KEYPAIR) && (threadIdx.x & 31) == 0) draw_coins(key, r, slot);
    __syncwarp();
    v.coins = slot;
  }
  if (op == OP_KEYPAIR) {
    if (stage == 0) call_saber_prologue_warp<L, OP_KEYPAIR>(v, role);
    else call_saber_finish_warp<L, OP_KEYPAIR>(v);
  } else if (op == OP_ENC) {
    if (stage == 0) call_saber_prologue_warp<L, OP_ENC>(v, role);
    else call_saber_finish_warp<L, OP_ENC>(v);
  } else {
    if (stage == 1) call_saber_prologue_warp<L, OP_DEC>(v, role);
    else if ((threadIdx.x & 31) == 0) call_saber_finish<L, OP_DEC>(v);  // one permutation
  }
}

__device__ __forceinline__ void warp_stage(const CoinKey &key, int code, const DevReq &r, int role) {
  const int scheme = scheme_of(code), op = op_of(code), stage = stage_of(code);
  if (scheme <= 1) {
    if (r.gen && stage == 0 && op != OP_DEC) {
      if ((threadIdx.x & 31) == 0) draw_coins(key, r, const_cast<uint8_t *>(r.in0));
      __syncwarp();
    }
    const fdev::Inst v = frodo_view(r);
    if (op == OP_KEYPAIR) {
      if (stage == 0) call_frodo_prologue_warp<OP_KEYPAIR>(v);
      else call_frodo_hash_warp<OP_KEYPAIR>(v);
    } else if (op == OP_ENC) {
      if (stage == 0) call_frodo_prologue_warp<OP_ENC>(v);
      else call_frodo_hash_warp<OP_ENC>(v);
    } else {
      if (stage == 1 && role == 0) call_frodo_prologue_warp<OP_DEC>(v);
      else if (stage == 1) call_frodo_absorb_warp(v);
      else call_frodo_hash_warp<OP_DEC>(v);
    }
  } else if (scheme == 2) {
    saber_warp<2>(key, op, stage, r, role);
  } else if (scheme == 3) {
    saber_warp<3>(key, op, stage, r, role);
  } else {
    saber_warp<4>(key, op, stage, r, role);
  }
}

__device__ __forceinline__ void thread_stage(const CoinKey &key, int code, const DevReq &r, int role) {
  const int scheme = scheme_of(code), op = op_of(code), stage = stage_of(code);
  if (scheme <= 1) {
    if (r.gen && stage == 0 && op != OP_DEC) draw_coins(key, r, const_cast<uint8_t *>(r.in0));
    const fdev::Inst v = frodo_view(r);
    if (op == OP_KEYPAIR) {
      if (stage == 0) call_frodo_prologue<OP_KEYPAIR>(v);
      else call_frodo_hash<OP_KEYPAIR>(v);
    } else if (op == OP_ENC) {
      if (stage == 0) call_frodo_prologue<OP_ENC>(v);
      else call_frodo_hash<OP_ENC>(v);
    } else {
      if (stage == 1 && role == 0) call_frodo_prologue<OP_DEC>(v);
      else if (stage == 1) call_frodo_absorb(v);
      else call_frodo_hash<OP_DEC>(v);
    }
  } else if (scheme == 2) {
    saber_thread<2>(key, op, stage, r, role);
  } else if (scheme == 3) {
    saber_thread<3>(key, op, stage, r, role);
  } else {
    saber_thread<4>(key, op, stage, r, role);
  }
}

template <int L, int MODE>
__device__ __forceinline__ void saber_product(int form, const sdev::Inst &v, uint8_t *smem, uint32_t tbase,
                                              uint32_t *err) {
  if (form == FORM_TC) call_saber_product<L, MODE, FORM_TC>(v, smem, tbase, err);
  else if (form == FORM_INT32) call_saber_product<L, MODE, FORM_INT32>(v, smem, tbase, err);
  else call_saber_product<L, MODE, FORM_DP4A>(v, smem, tbase, err);
}

template <int L>
__device__ __forceinline__ void saber_cta(int op, int stage, int tc, const DevReq &r, uint8_t *smem, uint32_t tbase,
                                          uint32_t *err) {
  const sdev::Inst v = saber_view<L>(r);
  if (op == OP_KEYPAIR) saber_product<L, sdev::PM_KEYPAIR>(tc, v, smem, tbase, err);
  else if (op == OP_ENC) saber_product<L, sdev::PM_ENC>(tc, v, smem, tbase, err);
  else if (stage == 0) saber_product<L, sdev::PM_DEC_INNER>(tc, v, smem, tbase, err);
  else saber_product<L, sdev::PM_DEC_CMP>(tc, v, smem, tbase, err);
}

constexpr int kTcStages = 2;

// Frodo product of one operation with row generator GT (tcgen05 stage, NST tile stages; keypair: every
// form) / GD (the other forms).
template <int OP, class GT, class GD, int NST>
__device__ __forceinline__ void frodo_product(int form, const fdev::Inst &v, uint8_t *smem, uint32_t tbase,
                                              uint32_t *err) {
  if (form == FORM_TC) call_frodo_product<OP, FORM_TC, NST, GT>(v, smem, tbase, err);
  else if (form == FORM_INT32) call_frodo_product<OP, FORM_INT32, NST, GD>(v, smem, tbase, err);
  else call_frodo_product<OP, FORM_DP4A, NST, GD>(v, smem, tbase, err);
}

template <class GT, class GD, int NST>
__device__ __forceinline__ void frodo_cta(int op, int stage, int tc, const DevReq &r, uint8_t *smem, uint32_t tbase,
                                          uint32_t *err) {
  const fdev::Inst v = frodo_view(r);
  if (op == OP_KEYPAIR) frodo_product<OP_KEYPAIR, GT, GT, NST>(tc, v, smem, tbase, err);
  else if (op == OP_ENC) frodo_product<OP_ENC, GT, GD, NST>(tc, v, smem, tbase, err);
  else if (stage == 0) call_frodo_dec_w(v, smem);
  else frodo_product<OP_DEC, GT, GD, NST>(tc, v, smem, tbase, err);
}

__device__ __forceinline__ void cta_stage(int code, const DevReq &r, uint8_t *smem, uint32_t tbase, uint32_t *err) {
  const int scheme = scheme_of(code), op = op_of(code), stage = stage_of(code);
  const int tc = form_of(code);  // product form (FORM_DP4A / FORM_INT32 / FORM_TC)
  if (scheme == 0) {
    frodo_cta<fdev::ShakeRows, fdev::ShakeRows, kTcStages>(op, stage, tc, r, smem, tbase, err);
  } else if (scheme == 1) {  // FrodoKEM-976-AES (one tile stage: see frodo.cu)
    frodo_cta<fdev::AesRowsFull, fdev::AesRowsHalf, 1>(op, stage, tc, r, smem, tbase, err);
  } else if (scheme == 2) {
    saber_cta<2>(op, stage, tc, r, smem, tbase, err);
  } else if (scheme == 3) {
    saber_cta<3>(op, stage, tc, r, smem, tbase, err);
  } else {
    saber_cta<4>(op, stage, tc, r, smem, tbase, err);
  }
}

constexpr int kSmem = std::max({fdev::TcLayout<kTcStages>::total, fdev::DP4A_SMEM, fdev::DEC_W_SMEM,
                                fdev::KP_AS_SMEM, fdev::KptLayout::total, sdev::PL<4>::DP4A_TOTAL, sdev::PL<3>::DP4A_TOTAL,
                                sdev::PL<2>::DP4A_TOTAL, sdev::TL<4>::TOTAL, sdev::TL<3>::TOTAL, sdev::TL<2>::TOTAL,
                                // FrodoKEM-976-AES stages: layout + AES table copies
                                fdev::TcLayout<1>::total + fdev::AesRowsFull::SMEM,
                                fdev::DP4A_SMEM + fdev::AesRowsHalf::SMEM, fdev::KP_AS_SMEM + fdev::AesRowsFull::SMEM,
                                fdev::KptLayoutT<1>::total + fdev::AesRowsFull::SMEM});
static_assert(kChainReqs >= 4 * sizeof(fchain::Exchange) + 8 * k10::kSmemPerWarp && kChainReqs + 24 * sizeof(DevReq) <= kSmem,
              "a chain task's shared memory");
static_assert(kSmem == fdev::TcLayout<kTcStages>::total, "the AES stages must not raise the kernel's shared memory");


}  // namespace mixed
}  // namespace dpkem

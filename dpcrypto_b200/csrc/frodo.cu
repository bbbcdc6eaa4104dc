// FrodoKEM-976 (SHAKE and AES variants) batched keypair / encaps / decaps: one launch per
// stage over n instances.  The stage bodies live in frodo_dev.cuh (shared with the persistent
// mixed-batch kernel); these wrappers only map blockIdx/threadIdx to instances.
#include <algorithm>

#include "frodo_dev.cuh"
#include "frodo_ahead.cuh"
#include "frodo_gemm.cuh"

namespace dpkem {
namespace {

using namespace frodo;
using fdev::inst_of;

// Thread-per-instance prologues: dynamic shared memory of kParkBytes per thread parks the
// sampling stream's blocks (fdev::sample_stream).
constexpr int kParkBytes = 17 * 8;

template <int OP>
__global__ void __launch_bounds__(256) kp_prologue_kernel(FrodoBatch b) {
  extern __shared__ uint2 park[];
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < b.n) fdev::kp_prologue_inst(inst_of(b, i, OP), park + threadIdx.x, blockDim.x);
}

template <int OP>
__global__ void __launch_bounds__(256) pk_hash_kernel(FrodoBatch b) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < b.n) fdev::pk_hash_inst(inst_of(b, i, OP));
}

template <int MODE>
__global__ void __launch_bounds__(256) prologue_kernel(FrodoBatch b) {
  extern __shared__ uint2 park[];
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < b.n) fdev::prologue_inst<MODE>(inst_of(b, i, MODE), park + threadIdx.x, blockDim.x);
}

// Decaps prologue, 64 threads = 32 instances: warp 0 runs the sampling chain, warp 1 the
// ciphertext pre-absorb of the final hash.
__global__ void __launch_bounds__(64) dec_prologue_kernel(FrodoBatch b) {
  __shared__ uint2 park[17 * 32];
  const int i = blockIdx.x * 32 + (threadIdx.x & 31);
  if (i >= b.n) return;
  if (threadIdx.x < 32) fdev::prologue_inst<OP_DEC>(inst_of(b, i, OP_DEC), park + threadIdx.x, 32);
  else fdev::ct_absorb_inst(inst_of(b, i, OP_DEC));
}

// Several lanes per state (msponge.cuh; NS = 1: a warp per instance; NS = 10: ten lanes, three
// instances per warp; NS = 2: a pair, sixteen), one warp per block.  STAGE selects the stage body: 0 keypair
// prologue, 1 H(pk), 2 encaps prologue, 3 encaps final hash, 4 decaps final hash; the
// decaps prologue has its own kernels.
template <int STAGE, int NS>
__global__ void __launch_bounds__(32) stage_multi_kernel(FrodoBatch b) {
  using S = msp::Multi<NS>;
  __shared__ __align__(16) uint8_t xbuf[S::SMEM_PER_WARP > 0 ? S::SMEM_PER_WARP : 16];
  const S s(xbuf);
  const int g = s.state(), i = blockIdx.x * S::STATES_PER_WARP + g;
  const bool live = g < S::STATES_PER_WARP && i < b.n;
  constexpr int op = STAGE <= 1 ? OP_KEYPAIR : STAGE <= 3 ? OP_ENC : OP_DEC;
  const fdev::Inst v = inst_of(b, live ? i : b.n - 1, op);
  if constexpr (STAGE == 0) fdev::kp_prologue_multi<S>(v, s, live);
  else if constexpr (STAGE == 1) fdev::pk_hash_multi<S>(v, s, live);
  else if constexpr (STAGE == 2) fdev::prologue_multi<S, OP_ENC>(v, s, live);
  else if constexpr (STAGE == 3) fdev::ss_multi<S, OP_ENC>(v, s, live);
  else fdev::ss_multi<S, OP_DEC>(v, s, live);
}

template <int MODE>
__global__ void __launch_bounds__(256) ss_kernel(FrodoBatch b) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < b.n) fdev::ss_inst<MODE>(inst_of(b, i, MODE));
}

__global__ void __launch_bounds__(256) dec_w_kernel(FrodoBatch b) {
  extern __shared__ __align__(1024) uint8_t smem[];
  fdev::dec_w_cta(inst_of(b, blockIdx.x, OP_DEC), smem);
}

template <int MODE, bool I32, class G>
__global__ void __launch_bounds__(256, 2) sa_dp4a_kernel(FrodoBatch b) {
  extern __shared__ __align__(1024) uint8_t smem[];
  fdev::sa_dp4a_cta<MODE, I32, G>(inst_of(b, blockIdx.x, MODE), smem);
}

template <int MODE, int NST, class G>
__global__ void __launch_bounds__(256, 2) sa_tc_kernel(FrodoBatch b) {
  using L = fdev::TcLayout<NST>;
  extern __shared__ __align__(1024) uint8_t smem[];
  uint32_t *tslot = reinterpret_cast<uint32_t *>(smem + L::tslot);
  if (threadIdx.x < 32) {
    tmem_alloc(tslot, fdev::TC_TMEM_COLS);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tbase = *tslot;
  fdev::sa_tc_cta<MODE, NST, G>(inst_of(b, blockIdx.x, MODE), smem, tbase, b.err);
  tc_fence_before();
  __syncthreads();
  if (threadIdx.x < 32) {
    tc_fence_after();
    tmem_dealloc(tbase, fdev::TC_TMEM_COLS);
  }
}

template <bool I32, class G>
__global__ void __launch_bounds__(256, 2) kp_as_dp4a_kernel(FrodoBatch b) {
  extern __shared__ __align__(1024) uint8_t smem[];
  fdev::kp_as_dp4a_cta<I32, G>(inst_of(b, blockIdx.x, OP_KEYPAIR), smem);
}

template <int NST, class G>
__global__ void __launch_bounds__(256, 2) kp_as_tc_kernel(FrodoBatch b) {
  extern __shared__ __align__(1024) uint8_t smem[];
  __shared__ uint32_t tslot;
  if (threadIdx.x < 32) {
    tmem_alloc(&tslot, 64);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tbase = tslot;
  fdev::kp_as_tc_cta<NST, G>(inst_of(b, blockIdx.x, OP_KEYPAIR), smem, tbase, b.err);
  tc_fence_before();
  __syncthreads();
  if (threadIdx.x < 32) {
    tc_fence_after();
    tmem_dealloc(tbase, 64);
  }
}

inline int blocks_for(int n, int t) { return (n + t - 1) / t; }

// Lanes per state of a hash stage: a warp per state up to frodo_ss_warp_max, ten lanes up to frodo_ss_five_max (the
// name is from a layout of five), a pair up to frodo_pair_max, else one (false: the caller launches that).
template <int STAGE>
bool launch_multi(const FrodoBatch &b, cudaStream_t st) {
  const Tuning &t = tuning();
  if (b.n <= t.frodo_ss_warp_max) {
    stage_multi_kernel<STAGE, 1><<<b.n, 32, 0, st>>>(b);
    return true;
  }
  if (b.n <= t.frodo_ss_five_max) {
    stage_multi_kernel<STAGE, 10><<<blocks_for(b.n, 3), 32, 0, st>>>(b);
    return true;
  }
  if (b.n <= t.frodo_pair_max) {
    stage_multi_kernel<STAGE, 2><<<blocks_for(b.n, 16), 32, 0, st>>>(b);
    return true;
  }
  return false;
}

template <typename K>
cudaError_t set_smem(K kernel, int bytes) {
  return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
}

constexpr int kTcStages = 2;

// GT feeds the tcgen05 stage (with NST tile stages per warp), GD the dp4a / INT32 stage.
// FrodoKEM-976-AES runs its tensor stages with one tile stage: a warp spends thousands of
// cycles producing a tile, long after the previous tile's MMAs have finished, and the
// shared memory goes to the AES table copies instead.
template <int MODE, class GT, class GD, int NST>
cudaError_t launch_sa_g(const FrodoBatch &b, int form, cudaStream_t st) {
  cudaError_t e;
  if (form == FORM_TC) {
    constexpr int bytes = fdev::TcLayout<NST>::total + GT::SMEM;
    if ((e = set_smem(sa_tc_kernel<MODE, NST, GT>, bytes)) != cudaSuccess) return e;
    sa_tc_kernel<MODE, NST, GT><<<b.n, 256, bytes, st>>>(b);
  } else if (form == FORM_INT32) {
    constexpr int bytes = fdev::DP4A_SMEM + GD::SMEM;
    if ((e = set_smem(sa_dp4a_kernel<MODE, true, GD>, bytes)) != cudaSuccess) return e;
    sa_dp4a_kernel<MODE, true, GD><<<b.n, 256, bytes, st>>>(b);
  } else {
    constexpr int bytes = fdev::DP4A_SMEM + GD::SMEM;
    if ((e = set_smem(sa_dp4a_kernel<MODE, false, GD>, bytes)) != cudaSuccess) return e;
    sa_dp4a_kernel<MODE, false, GD><<<b.n, 256, bytes, st>>>(b);
  }
  return cudaGetLastError();
}

// Shared key, A in memory, tensor-core form: one GEMM over all instances (frodo_gemm.cuh).
template <int MODE>
cudaError_t launch_sa_gemm(const FrodoBatch &b, cudaStream_t st) {
  using namespace fgemm;
  cudaError_t e;
  const int groups = (b.n + INST - 1) / INST;
  tile_ab_kernel<<<blocks_for(MT * KSTEPS * 2 * 8 * 32, 256), 256, 0, st>>>(b.amat, MODE == OP_ENC ? b.pk : b.sk + LENS,
                                                                             b.abt);
  tile_s_kernel<<<blocks_for(groups * INST * NBAR * 62, 256), 256, 0, st>>>(b.rw, b.n, b.stile);
  if (MODE == OP_DEC && (e = cudaMemsetAsync(b.fail, 0, (size_t)b.n * 4, st)) != cudaSuccess) return e;
  if ((e = set_smem(gemm_kernel<MODE>, SMEM_LAUNCH)) != cudaSuccess) return e;
  const GemmArgs g{b.abt, b.stile, b.rw, MODE == OP_ENC ? b.coins : b.mu, b.ct, b.fail, b.err, b.n};
  gemm_kernel<MODE><<<MT * groups, THREADS, SMEM_LAUNCH, st>>>(g);
  return cudaGetLastError();
}

template <int MODE>
cudaError_t launch_sa(const FrodoBatch &b, int form, cudaStream_t st) {
  if (b.amat && b.abt && b.stile && form == FORM_TC) return launch_sa_gemm<MODE>(b, st);
  if (b.amat) return launch_sa_g<MODE, fdev::MemRows, fdev::MemRows, kTcStages>(b, form, st);
  if (b.aes) return launch_sa_g<MODE, fdev::AesRowsFull, fdev::AesRowsHalf, 1>(b, form, st);
  return launch_sa_g<MODE, fdev::ShakeRows, fdev::ShakeRows, kTcStages>(b, form, st);
}

// A (976 x 976 LE u16, row-major) of the public key pk, one row per thread, with the same
// row generators as the S'A stages (SHAKE128 or AES-128 rows).
template <class G>
__global__ void __launch_bounds__(256) expand_a_kernel(const uint8_t *pk, uint16_t *amat) {
  extern __shared__ __align__(16) uint8_t gmem[];
  G gen;
  gen.setup(pk, gmem);
  __syncthreads();
  const int j = blockIdx.x * blockDim.x + threadIdx.x;
  if (j >= N) return;
  uint2 a[25];
  gen.start(a, j);
  uint2 *row = reinterpret_cast<uint2 *>(amat + (size_t)j * N);
  for (int blk = 0; blk < 12; blk++) {
    gen.next(a);
#pragma unroll
    for (int q = 0; q < 21; q++)
      if (84 * blk + 4 * q < N) row[21 * blk + q] = a[q];
  }
}

// H(pk) = SHAKE256(pk, 24) of one public key, on a warp (a warp per state).
__global__ void __launch_bounds__(32) pk_digest_kernel(const uint8_t *pk, uint8_t *out) {
  using S = msp::Multi<1>;
  const S s(nullptr);
  uint2 a[1];
  msp::zero<S>(a);
  const int pos = msp::absorb_aligned<S, 136>(a, s, 0, pk, PK, true);
  msp::absorb_finish<S, 136>(a, s, pos, 0x1Fu);
  msp::store<S, 3>(a, s, out, true);
}

template <class G, int NST>
cudaError_t launch_kp_as(const FrodoBatch &b, int form, cudaStream_t st) {
  cudaError_t e;
  if (form == FORM_TC) {
    constexpr int bytes = fdev::KptLayoutT<NST>::total + G::SMEM;
    if ((e = set_smem(kp_as_tc_kernel<NST, G>, bytes)) != cudaSuccess) return e;
    kp_as_tc_kernel<NST, G><<<b.n, 256, bytes, st>>>(b);
  } else {
    constexpr int bytes = fdev::KP_AS_SMEM + G::SMEM;
    if (form == FORM_INT32) {
      if ((e = set_smem(kp_as_dp4a_kernel<true, G>, bytes)) != cudaSuccess) return e;
      kp_as_dp4a_kernel<true, G><<<b.n, 256, bytes, st>>>(b);
    } else {
      if ((e = set_smem(kp_as_dp4a_kernel<false, G>, bytes)) != cudaSuccess) return e;
      kp_as_dp4a_kernel<false, G><<<b.n, 256, bytes, st>>>(b);
    }
  }
  return cudaGetLastError();
}

// The prologue without A's rows: on chain and helper warps up to frodo_warp_max / frodo_five_max (decaps,
// whose ciphertext hash shares the SMs, at most to kDecChains), encaps and keypair on pairs up to
// frodo_pair_max; false above.  us of the whole call under one key, chains / pairs, encaps: n = 4,096 1,508 / 1,719,
// 6,144 1,782 / 1,832, 7,000 1,903 / 1,853; chains / one lane, decaps: 1,024 655 / 1,544, 4,096 1,121 / 1,662, 4,871 (the
// blocks that are resident at once end there) 1,327 / 1,696, 5,300 1,387 / 1,706, 5,700 1,609 / 1,721, 6,144
// 1,816 / 1,738.
constexpr int kDecChains = 5600;
template <int ROLE>
bool launch_prologue(const FrodoBatch &b, cudaStream_t st) {
  const int most = std::max(tuning().frodo_warp_max, tuning().frodo_five_max);
  if (b.n <= (ROLE == ahead::R_DEC ? std::min(most, kDecChains) : most)) {
    const int chain = blocks_for(b.n, 6), absorb = ROLE == ahead::R_DEC ? blocks_for(b.n, 16 * ahead::kAbsorbWarps) : 0;
    if (ROLE == ahead::R_KEYPAIR) ahead::kp_seed_kernel<<<blocks_for(b.n, 32), 32, 0, st>>>(b);
    ahead::chains_kernel<ROLE><<<chain + absorb, 128, ahead::chain_smem(2), st>>>(b, chain);
    return true;
  }
  if (ROLE == ahead::R_DEC || b.n > tuning().frodo_pair_max) return false;
  stage_multi_kernel<ROLE == ahead::R_KEYPAIR ? 0 : 2, 2><<<blocks_for(b.n, 16), 32, 0, st>>>(b);
  return true;
}

inline void mark(const FrodoBatch &b, cudaStream_t st) {
  if (b.timer) b.timer->mark(st);
}

// ---- A generated ahead (frodo_ahead.cuh) ----

// Instances [first, n) of a batch (a key per instance).
FrodoBatch rest_of(const FrodoBatch &b, int first, int op) {
  FrodoBatch r = b;
  const size_t i = (size_t)first;
  r.n = b.n - first;
  if (b.coins) r.coins = b.coins + i * (op == OP_KEYPAIR ? KP_COINS : ENC_COINS);
  if (b.pk) r.pk = b.pk + i * PK;
  if (b.sk) r.sk = b.sk + i * SK;
  if (b.ct) r.ct = b.ct + i * CT;
  if (b.ss) r.ss = b.ss + i * SS;
  r.rw = b.rw + i * RW;
  r.kk = b.kk + i * LENSE;
  r.mu = b.mu + i * LENMU;
  r.fail = b.fail + i;
  if (b.hs) r.hs = b.hs + i * 25;
  r.atile = nullptr;
  r.ahead = 0;
  return r;
}

// Chain warps of a front block on ten lanes: four (one per SM sub-partition, 2.05 us per
// permutation) while the chains outlast the rows, else eight (2.5 us, half the SMs): 2.8 us of the
// whole chip per instance's rows against the chain's steps.  Measured, n = 128 / 256: encaps 4
// warps 824 / 1,185 us, 8 warps 902 / 1,164 us; keypair (half the steps) 754 / 1,171 and 701 / 1,120.
int chain_warps(int ahead, int steps) { return ahead * 28 > steps * 25 ? 8 : 4; }

template <int STAGE, int NS, bool HALVE, class G>
cudaError_t launch_front_g(const FrodoBatch &b, cudaStream_t st) {
  cudaError_t e;
  constexpr int spw = NS == 10 ? 3 : 32;
  constexpr int steps = STAGE == ahead::F_KEYPAIR ? (HALVE ? 115 : 230) : STAGE == ahead::F_ENC && !HALVE ? 348 : 232;
  const int warps = blocks_for(b.n, spw), cw = NS == 10 ? chain_warps(b.ahead, steps) : 4, chain = blocks_for(warps, cw);
  const int absorb = STAGE == ahead::F_DEC ? (NS == 10 ? blocks_for(b.n, 16 * ahead::kAbsorbWarps) : blocks_for(warps, ahead::kFrontWarps)) : 0;
  const int early = std::max(0, device_sms() - chain - absorb);
  const int rows = std::min(device_sms(), std::max(1, ahead::WarpRows<G>::tasks(b.ahead)));
  if ((e = set_smem(ahead::front_kernel<STAGE, NS, HALVE, G>, ahead::kFrontSmem)) != cudaSuccess) return e;
  ahead::front_kernel<STAGE, NS, HALVE, G>
      <<<chain + absorb + rows, 32 * ahead::kFrontWarps, ahead::kFrontSmem, st>>>(b, cw, chain, absorb, std::min(early, rows));
  return cudaGetLastError();
}
template <int STAGE, int NS, bool HALVE>
cudaError_t launch_front_ns(const FrodoBatch &b, cudaStream_t st) {
  return b.aes ? launch_front_g<STAGE, NS, HALVE, fdev::AesRowsFull>(b, st)
               : launch_front_g<STAGE, NS, HALVE, fdev::ShakeRows>(b, st);
}
// Ten lanes per state up to kFrontTenMax; beyond, one: a permutation is 135 integer instructions per state there, 160 on
// ten lanes, whose chain blocks hold more SM time, while the rows fill the other SMs as long as one lane's
// chains last.  Between about 2,000 and 4,000 it depends on the rows ahead (n mod 296): few of them end before
// one lane's chains do.  ms, ten lanes / one, encaps: 1,025 3.72 / 4.30, 2,072 (0 mod 296) 7.45 / 7.77, 2,600 8.82 / 8.74, 3,700
// 12.44 / 12.26, 3,848 (0) 13.48 / 13.04, 4,096 13.64 / 13.13, 5,000 16.64 / 15.95; decaps: 1,025 3.46 / 4.08, 2,072 6.74 / 7.52,
// 3,700 11.92 / 11.95, 3,848 12.34 / 12.74, 4,096 13.15 / 12.84; keypair: 1,536 5.31 / 5.57, 2,000 6.89 / 6.73, 2,072 7.14 / 7.40,
// 4,096 13.75 / 13.39.  `halve` (encaps, keypair): stop the stream after S', tail_kernel runs the rest.
constexpr int kFrontTenMax = 4096;
template <int STAGE>
cudaError_t launch_front(const FrodoBatch &b, bool halve, cudaStream_t st) {
  if constexpr (STAGE != ahead::F_DEC)
    if (halve) return launch_front_ns<STAGE, 10, true>(b, st);
  if (b.n <= kFrontTenMax) return launch_front_ns<STAGE, 10, false>(b, st);
  return launch_front_ns<STAGE, 0, false>(b, st);
}

template <int MODE, int NB>
cudaError_t launch_product_nb(const FrodoBatch &b, cudaStream_t st) {
  cudaError_t e;
  if ((e = set_smem(ahead::product_kernel<MODE, NB>, ahead::PLayout::total)) != cudaSuccess) return e;
  ahead::product_kernel<MODE, NB><<<b.ahead * (ahead::BLKS / NB), 256, ahead::PLayout::total, st>>>(b);
  return cudaGetLastError();
}
template <int MODE>
cudaError_t launch_product(const FrodoBatch &b, cudaStream_t st) {
  return b.ahead <= ahead::kProductFew ? launch_product_nb<MODE, 2>(b, st) : launch_product_nb<MODE, 4>(b, st);
}
template <bool RAW>
cudaError_t launch_product_kp(const FrodoBatch &b, cudaStream_t st) {
  cudaError_t e;
  if ((e = set_smem(ahead::product_kp_kernel<RAW>, ahead::KLayout::total)) != cudaSuccess) return e;
  ahead::product_kp_kernel<RAW><<<b.ahead * ahead::TILES, 256, ahead::KLayout::total, st>>>(b);
  return cudaGetLastError();
}

// Whether the batch runs the halved stream and the stepped tail (ten lanes per state): every instance's
// products must come raw from product_kernel.
bool halved(const FrodoBatch &b) { return b.ahead == b.n; }
bool use_ahead(const FrodoBatch &b, int form) { return form == FORM_TC && b.atile && b.ahead > 0 && !b.amat; }

}  // namespace

cudaError_t frodo_expand_a(int aes, const uint8_t *pk, uint16_t *amat, cudaStream_t st) {
  cudaError_t e;
  if (aes) {
    if ((e = set_smem(expand_a_kernel<fdev::AesRowsFull>, fdev::AesRowsFull::SMEM)) != cudaSuccess) return e;
    expand_a_kernel<fdev::AesRowsFull><<<blocks_for(N, 256), 256, fdev::AesRowsFull::SMEM, st>>>(pk, amat);
  } else {
    expand_a_kernel<fdev::ShakeRows><<<blocks_for(N, 256), 256, 0, st>>>(pk, amat);
  }
  return cudaGetLastError();
}

// The driver loads a kernel's code at its first launch, for which it waits until the device is idle.
cudaError_t frodo_load_untiled() {
  const void *const kernels[] = {
      (const void *)ahead::kp_seed_kernel, (const void *)ahead::chains_kernel<ahead::R_KEYPAIR>,
      (const void *)ahead::chains_kernel<ahead::R_ENC>, (const void *)ahead::chains_kernel<ahead::R_DEC>,
      (const void *)stage_multi_kernel<0, 2>, (const void *)stage_multi_kernel<2, 2>,
      (const void *)kp_prologue_kernel<OP_KEYPAIR>, (const void *)prologue_kernel<OP_ENC>,
      (const void *)dec_prologue_kernel, (const void *)dec_w_kernel,
      (const void *)kp_as_tc_kernel<fdev::KPT_NST, fdev::ShakeRows>, (const void *)kp_as_tc_kernel<1, fdev::AesRowsFull>,
      (const void *)sa_tc_kernel<OP_ENC, kTcStages, fdev::ShakeRows>,
      (const void *)sa_tc_kernel<OP_DEC, kTcStages, fdev::ShakeRows>,
      (const void *)sa_tc_kernel<OP_ENC, 1, fdev::AesRowsFull>, (const void *)sa_tc_kernel<OP_DEC, 1, fdev::AesRowsFull>,
      (const void *)stage_multi_kernel<1, 1>, (const void *)stage_multi_kernel<1, 10>,
      (const void *)stage_multi_kernel<1, 2>, (const void *)stage_multi_kernel<3, 1>,
      (const void *)stage_multi_kernel<3, 10>, (const void *)stage_multi_kernel<3, 2>,
      (const void *)stage_multi_kernel<4, 1>, (const void *)stage_multi_kernel<4, 10>,
      (const void *)stage_multi_kernel<4, 2>, (const void *)pk_hash_kernel<OP_KEYPAIR>, (const void *)ss_kernel<OP_ENC>,
      (const void *)ss_kernel<OP_DEC>};
  cudaFuncAttributes a;
  for (const void *k : kernels) {
    const cudaError_t e = cudaFuncGetAttributes(&a, k);
    if (e != cudaSuccess) return e;
  }
  return cudaSuccess;
}

size_t frodo_gemm_ab_bytes() { return fgemm::AB_BYTES; }
size_t frodo_gemm_s_bytes(size_t n) { return fgemm::s_bytes((int)n); }

cudaError_t frodo_pk_digest(const uint8_t *pk, uint8_t *out, cudaStream_t st) {
  pk_digest_kernel<<<1, 32, 0, st>>>(pk, out);
  return cudaGetLastError();
}

size_t frodo_ahead_bytes() { return ahead::A_BYTES; }

// Batches up to kAheadAll are generated whole: rows are dealt evenly over the SMs, while
// sa_tc_kernel's two CTAs per SM run in waves of 296 instances (0.88 ms each, 0.5 ms for one
// instance), and errors and final hash then run in step (tail_kernel).  Above it the A stage runs for the
// others; an ahead part of 296 .. 591 instances fills the SMs that the prologue leaves free, and
// leaves whole waves.  Measured ms, encaps: n = 768 all ahead 2.80, 176 ahead 3.45; 1,024 all
// 3.65, 432 ahead 3.83, none 4.6; 8,192: none 26.99, 200 ahead 26.23, 350 25.83, 496 25.65, 560 25.87.
// With scratch for fewer, as many as leave whole waves to the A stage, or none: other numbers cost more than they
// save, and so does a part of a batch of 1,025 .. kFrontTenMax, whose chains then hold the SMs.  ms, none / that
// many / another number, encaps: n = 64 1.42 / - / 16 1.49; 768 3.61 / 176 3.03, 472 2.94 / 4 3.68, 296 3.38;
// 1,024 4.14 / 136 4.01, 432 3.72 / 64 4.20; 4,096 13.7 / 248 14.4 / 128 14.6; 8,192 27.0 / 200 26.2.
constexpr int kAheadAll = 1024;

int frodo_ahead_count(int n, size_t cap) {
  const int wave = 2 * device_sms(), rest = n % wave, most = n <= kAheadAll ? n : wave + rest;
  if (cap >= (size_t)most) return most;
  if ((int)cap < rest || (n > kAheadAll && n <= kFrontTenMax)) return 0;
  return rest + ((int)cap - rest) / wave * wave;
}

cudaError_t frodo_keypair(const FrodoBatch &b, int form, cudaStream_t st) {
  if (b.n <= 0) return cudaSuccess;
  const int tb = tuning().thread_block;
  if (use_ahead(b, form)) {
    cudaError_t e;
    const bool half = halved(b);
    mark(b, st);
    ahead::kp_seed_kernel<<<blocks_for(b.n, 32), 32, 0, st>>>(b);
    if ((e = launch_front<ahead::F_KEYPAIR>(b, half, st)) != cudaSuccess) return e;
    mark(b, st);
    if ((e = half ? launch_product_kp<true>(b, st) : launch_product_kp<false>(b, st)) != cudaSuccess) return e;
    if (b.ahead < b.n) {
      const FrodoBatch r = rest_of(b, b.ahead, OP_KEYPAIR);
      e = b.aes ? launch_kp_as<fdev::AesRowsFull, 1>(r, form, st) : launch_kp_as<fdev::ShakeRows, fdev::KPT_NST>(r, form, st);
      if (e != cudaSuccess) return e;
    }
    mark(b, st);
    if (half) ahead::tail_kernel<OP_KEYPAIR><<<blocks_for(b.n, 3), 96, 0, st>>>(b);
    else if (!launch_multi<1>(b, st))
      pk_hash_kernel<OP_KEYPAIR><<<blocks_for(b.n, tb), tb, 0, st>>>(b);
    mark(b, st);
    return cudaGetLastError();
  }
  mark(b, st);
  if (!launch_prologue<ahead::R_KEYPAIR>(b, st))
    kp_prologue_kernel<OP_KEYPAIR><<<blocks_for(b.n, tb), tb, kParkBytes * tb, st>>>(b);
  mark(b, st);
  const cudaError_t e = b.aes ? launch_kp_as<fdev::AesRowsFull, 1>(b, form, st)
                             : launch_kp_as<fdev::ShakeRows, fdev::KPT_NST>(b, form, st);
  if (e != cudaSuccess) return e;
  mark(b, st);
  if (!launch_multi<1>(b, st)) pk_hash_kernel<OP_KEYPAIR><<<blocks_for(b.n, tb), tb, 0, st>>>(b);
  mark(b, st);
  return cudaGetLastError();
}

cudaError_t frodo_enc(const FrodoBatch &b, int form, cudaStream_t st) {
  if (b.n <= 0) return cudaSuccess;
  const int tb = tuning().thread_block;
  if (use_ahead(b, form)) {
    cudaError_t e;
    const bool half = halved(b);
    mark(b, st);
    if ((e = launch_front<ahead::F_ENC>(b, half, st)) != cudaSuccess) return e;
    mark(b, st);
    if ((e = half ? launch_product<ahead::PM_RAW>(b, st) : launch_product<ahead::PM_ENC>(b, st)) != cudaSuccess) return e;
    if (b.ahead < b.n && (e = launch_sa<OP_ENC>(rest_of(b, b.ahead, OP_ENC), form, st)) != cudaSuccess) return e;
    mark(b, st);
    if (half) ahead::tail_kernel<OP_ENC><<<blocks_for(b.n, 3), 96, 0, st>>>(b);
    else if (!launch_multi<3>(b, st))
      ss_kernel<OP_ENC><<<blocks_for(b.n, tb), tb, 0, st>>>(b);
    mark(b, st);
    return cudaGetLastError();
  }
  mark(b, st);
  if (!(b.pkh ? launch_prologue<ahead::R_ENC_PKH>(b, st) : launch_prologue<ahead::R_ENC>(b, st))) prologue_kernel<OP_ENC><<<blocks_for(b.n, tb), tb, kParkBytes * tb, st>>>(b);
  mark(b, st);
  cudaError_t e = launch_sa<OP_ENC>(b, form, st);
  if (e != cudaSuccess) return e;
  mark(b, st);
  if (!launch_multi<3>(b, st)) ss_kernel<OP_ENC><<<blocks_for(b.n, tb), tb, 0, st>>>(b);
  mark(b, st);
  return cudaGetLastError();
}

cudaError_t frodo_dec(const FrodoBatch &b, int form, cudaStream_t st) {
  if (b.n <= 0) return cudaSuccess;
  const int tb = tuning().thread_block;
  mark(b, st);
  dec_w_kernel<<<b.n, 256, fdev::DEC_W_SMEM, st>>>(b);
  mark(b, st);
  if (use_ahead(b, form)) {
    cudaError_t e;
    if ((e = launch_front<ahead::F_DEC>(b, false, st)) != cudaSuccess) return e;
    mark(b, st);
    if ((e = launch_product<ahead::PM_DEC>(b, st)) != cudaSuccess) return e;
    if (b.ahead < b.n && (e = launch_sa<OP_DEC>(rest_of(b, b.ahead, OP_DEC), form, st)) != cudaSuccess) return e;
    mark(b, st);
    if (!launch_multi<4>(b, st))
      ss_kernel<OP_DEC><<<blocks_for(b.n, tb), tb, 0, st>>>(b);
    mark(b, st);
    return cudaGetLastError();
  }
  if (!launch_prologue<ahead::R_DEC>(b, st)) dec_prologue_kernel<<<blocks_for(b.n, 32), 64, 0, st>>>(b);
  mark(b, st);
  cudaError_t e = launch_sa<OP_DEC>(b, form, st);
  if (e != cudaSuccess) return e;
  mark(b, st);
  if (!launch_multi<4>(b, st)) ss_kernel<OP_DEC><<<blocks_for(b.n, tb), tb, 0, st>>>(b);
  mark(b, st);
  return cudaGetLastError();
}

}  // namespace dpkem

// Saber (LightSaber l=2, Saber l=3, FireSaber l=4) batched keypair / encaps / decaps: one
// launch per stage over n instances.  The stage bodies live in saber_dev.cuh (shared with
// the persistent mixed-batch kernel); these wrappers only map blockIdx/threadIdx to instances.
#include <algorithm>
#include <atomic>

#include "saber_chain.cuh"
#include "saber_dev.cuh"

namespace dpkem {
namespace {

using sdev::inst_of;
using sdev::PL;
using sdev::Scr;
using sdev::TL;

// The stages of a call follow one another at once: each kernel lets the next one's blocks start when
// all of its own have, and waits for its predecessor's results itself (programmatic dependent launch), so
// launch latency and a kernel's set-up pass while the predecessor drains.  The first kernel of a call is
// launched plainly and waits for the whole stream.  Only up to follow_max instances: a waiting kernel
// that fills the SMs keeps the next call's sponges, or a persistent product's CTAs, off them.  us, plain /
// following, encaps at l = 3: n = 1 80 / 74, 444 86 / 82, 600 89 / 88, 1,501 112 / 140, 4,096 149 / 202.
// FireSaber's product CTAs, started early, share SMs that the prologue leaves free instead of spreading
// over all of them, where they are long and the prologue's blocks uneven.  us, plain / following, at l = 4:
//   tensor-core  encaps 300 125 / 125, 444 128 / 126, 512 128 / 143; keypair 444 129 / 129, 512 130 / 136; decaps
//                512 117 / 115
//   dp4a         encaps 100 130 / 127, 200 136 / 140, 300 144 / 170; keypair 148 133 / 131, 256 138 / 150; decaps
//                300 126 / 122, 512 147 / 145
//   INT32        encaps 100 144 / 140, 148 144 / 158, 300 181 / 236; keypair 300 176 / 173, 512 195 / 193; decaps
//                350 190 / 183, 400 188 / 204
// (l = 3, INT32 encaps: 300 124 / 119, 512 137 / 134).
template <int L>
constexpr int follow_max(int op, int form) {
  if (L < 4) return 512;
  if (form == FORM_TC) return op == OP_DEC ? 512 : 444;
  return op == OP_ENC ? 100 : op == OP_KEYPAIR ? (form == FORM_INT32 ? 512 : 148) : form == FORM_INT32 ? 350 : 512;
}
__device__ __forceinline__ void next_may_start() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void wait_predecessor() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

template <class... P, class... A>
cudaError_t launch_next(bool follows, void (*kernel)(P...), int grid, int block, int smem, cudaStream_t st, A... args) {
  cudaLaunchAttribute attr{};
  attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(grid);
  cfg.blockDim = dim3(block);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cfg.attrs = &attr;
  cfg.numAttrs = follows ? 1 : 0;
  return cudaLaunchKernelEx(&cfg, kernel, P(args)...);
}

// Prologue kernels: role 0 is the hash chain and GenSecret, role 1 GenMatrix.  A launch runs both, a
// warp each (roles = 2, first = 0), or the one `first` names.
//
// The role (of two) of this warp: GenMatrix's chain is the longer, so the warps that share a sub-partition
// must not all run it.  us with fixed roles / exchanged: pairs at 8,192 (l = 3) 145 / 116, one lane at
// 16,384 (l = 2 / 3 / 4) 112 / 84, 229 / 192, 390 / 290.
__device__ __forceinline__ int role_warp() {
  const int w = threadIdx.x >> 5;
  return blockDim.x == 64 && exchange_roles() ? 1 - w : w;
}

// One lane per state: 32 instances per block.
template <int L, int OP>
__global__ void __launch_bounds__(64) prologue_kernel(SaberBatch b, int first) {
  next_may_start();
  wait_predecessor();
  const int i = blockIdx.x * 32 + (threadIdx.x & 31), w = role_warp();
  if (i < b.n) sdev::prologue_inst<L, OP>(inst_of<L>(b, i, OP), first + w);
}

// Several lanes per state (msponge.cuh; NS = 1: a warp per instance; NS = 2: a pair, sixteen
// instances per warp).  Pairs leave the XOF bytes in their form (b.sliced): converted there, a pair's 21 words a permutation made the l = 3 prologue of
// 4,096 85 us against 77, and ten lanes' FireSaber prologue of 1,501 120 against 107; in the product's
// staging they are two words a thread (2 us).
template <int L, int OP, int NS>
__global__ void __launch_bounds__(64) prologue_multi_kernel(SaberBatch b, int first) {
  next_may_start();
  wait_predecessor();
  using S = msp::Multi<NS>;
  __shared__ __align__(16) uint8_t xbuf[2 * (S::SMEM_PER_WARP > 0 ? S::SMEM_PER_WARP : 16)];
  const int w = role_warp();
  const S s(xbuf + w * S::SMEM_PER_WARP);
  const int g = s.state(), i = blockIdx.x * S::STATES_PER_WARP + g;
  const bool live = g < S::STATES_PER_WARP && i < b.n;
  sdev::prologue_multi<S, L, OP, NS == 2>(inst_of<L>(b, live ? i : b.n - 1, OP), s, first + w, live);
}

// Ten lanes per state on chain and helper warps (saber_chain.cuh), three instances per block: the
// chains of the roles, then their helpers, exchanged from wave to wave.
template <int L, int OP>
__global__ void __launch_bounds__(128) prologue_chain_kernel(SaberBatch b, int first_role, int roles) {
  next_may_start();
  wait_predecessor();
  using namespace schain;
  __shared__ Exchange x[2];
  __shared__ __align__(16) uint8_t xbuf[2][k10::kSmemPerWarp];
  const bool swap = exchange_roles();
  const int warps = 2 * roles, warp = ((threadIdx.x >> 5) + (swap ? roles : 0)) & (warps - 1);
  const int w = warp & (roles - 1), role = first_role + w, first = 3 * blockIdx.x;
  if (warp < roles) {
    constexpr Program m = Matrix<L, OP>::prog, s = Secret<L, OP>::prog;
    const Program p = {role ? m.steps : s.steps, role ? m.msg : s.msg, role ? m.reset : s.reset, role ? m.idle : s.idle};
    chain_warp(p, x[w], xbuf[w], w);
  } else {
    auto inst = [&](int i) { return inst_of<L>(b, i, OP); };
    if (role) helper_warp<Matrix<L, OP>>(inst, b.n, first, x[w], w);
    else helper_warp<Secret<L, OP>>(inst, b.n, first, x[w], w);
  }
}

// Encaps / keypair finish likewise, 64 threads.
template <int L, int OP>
__global__ void __launch_bounds__(64) finish_chain_kernel(SaberBatch b) {
  next_may_start();
  wait_predecessor();
  using namespace schain;
  __shared__ Exchange x;
  __shared__ __align__(16) uint8_t xbuf[k10::kSmemPerWarp];
  const int warp = (threadIdx.x >> 5) ^ (exchange_roles() ? 1 : 0), lane = threadIdx.x & 31, first = 3 * blockIdx.x;
  if (warp == 0) {
    constexpr Program p = Finish<L, OP>::prog;
    chain_warp(p, x, xbuf, 0);
    return;
  }
  auto inst = [&](int i) { return inst_of<L>(b, i, OP); };
  if (OP == OP_KEYPAIR) {  // sk = s || pk || H(pk) || z: pk and z
    using P = sdev::SP<L>;
    for (int i = first; i < first + 3 && i < b.n; i++) {
      const sdev::Inst v = inst(i);
      for (int q = lane; q < P::PK / 8; q += 32) put(v.sk + P::POLYVEC + 8 * q, ld_lane(v.pk + 8 * q));
      if (lane < 4) put(v.sk + P::SK - 32 + 8 * lane, ld_lane(v.coins + 64 + 8 * lane));
    }
  }
  helper_warp<Finish<L, OP>>(inst, b.n, first, x, 0);
}

// Lanes per state of the prologue's sponges for a batch of n: a warp per state up to
// saber_warp_max, ten lanes up to saber_five_max (the knob's name is from a layout of five), a
// pair up to saber_pair_max (LightSaber decaps, whose two chains are the shortest: half of that), else one.
// us, decaps at l = 2 on pairs / one lane: tensor-core 4,096 105 / 120, 5,000 133 / 129, 8,192 173 / 164;
// dp4a 4,096 182 / 197, 5,000 228 / 223, 8,192 325 / 315 (l = 3, 9,472 261 / 268; keypair at l = 2 136 / 157).
template <int L, int OP>
int prologue_lanes(int n) {
  const Tuning &t = tuning();
  const int pair_max = L == 2 && OP == OP_DEC ? t.saber_pair_max / 2 : t.saber_pair_max;
  return n <= t.saber_warp_max ? 25 : n <= t.saber_five_max ? 10 : n <= pair_max ? 2 : 1;
}
template <int L>
int prologue_lanes(int n, int op) {
  return op == OP_KEYPAIR ? prologue_lanes<L, OP_KEYPAIR>(n) : op == OP_ENC ? prologue_lanes<L, OP_ENC>(n)
                                                                            : prologue_lanes<L, OP_DEC>(n);
}

// Whether decaps runs GenMatrix on a second stream beside the inner product and the chain that needs
// its m'.  It pays while every chain warp finds an SM with little else on it (up to 100
// blocks), and again when the chains fill the chip several times over; between, the chains slow down
// next to the product's CTAs by more than the inner product takes, and LightSaber's chain is too short.
// us, one stream / two, l = 3: n = 1 76 / 70, 300 83 / 78, 444 84 / 93, 1,500 113 / 116, 8,192 260 / 311,
// 12,000 413 / 388, 16,384 474 / 448; l = 4: 128 115 / 109, 12,000 669 / 539; l = 2: 128 49 / 51.
template <int L>
bool matrix_beside_inner(int n) {
  const int lanes = prologue_lanes<L, OP_DEC>(n);
  return L > 2 && ((lanes == 25 && n <= 100) || (lanes == 10 && n <= 300) || (lanes == 1 && n >= 12000));
}

template <int L, int OP>
cudaError_t launch_prologue(const SaberBatch &b, cudaStream_t st, bool follows, int first = 0, int roles = 2) {
  auto blocks = [&](int per) { return (b.n + per - 1) / per; };
  const int threads = 32 * roles;
  switch (prologue_lanes<L, OP>(b.n)) {
    case 25: return launch_next(follows, prologue_multi_kernel<L, OP, 1>, b.n, threads, 0, st, b, first);
    case 10: return launch_next(follows, prologue_chain_kernel<L, OP>, blocks(3), 2 * threads, 0, st, b, first, roles);
    case 2: return launch_next(follows, prologue_multi_kernel<L, OP, 2>, blocks(16), threads, 0, st, b, first);
    default: return launch_next(follows, prologue_kernel<L, OP>, blocks(32), threads, 0, st, b, first);
  }
}

// Encaps / keypair finish on a warp (NS = 1) or a pair (2) per state, one warp per block.
template <int L, int OP, int NS>
__global__ void __launch_bounds__(32) finish_multi_kernel(SaberBatch b) {
  next_may_start();
  wait_predecessor();
  using S = msp::Multi<NS>;
  __shared__ __align__(16) uint8_t xbuf[S::SMEM_PER_WARP > 0 ? S::SMEM_PER_WARP : 16];
  const S s(xbuf);
  const int g = s.state(), i = blockIdx.x * S::STATES_PER_WARP + g;
  const bool live = g < S::STATES_PER_WARP && i < b.n;
  const sdev::Inst v = inst_of<L>(b, live ? i : b.n - 1, OP);
  if (OP == OP_ENC) sdev::finish_enc_multi<S, L>(v, s, live);
  else sdev::finish_kp_multi<S, L>(v, s, live);
}

template <int L, int OP>
__global__ void __launch_bounds__(256) finish_kernel(SaberBatch b) {
  next_may_start();
  wait_predecessor();
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < b.n) sdev::finish_inst<L, OP>(inst_of<L>(b, i, OP));
}

// The finish on a warp, ten lanes or a pair per state when n is within the thresholds (decaps: one
// permutation), else on one lane.
template <int L, int OP>
cudaError_t launch_finish(const SaberBatch &b, cudaStream_t st, bool follows) {
  const Tuning &t = tuning();
  auto blocks = [&](int per) { return (b.n + per - 1) / per; };
  if constexpr (OP != OP_DEC) {
    if (b.n <= t.saber_finish_warp_max) return launch_next(follows, finish_multi_kernel<L, OP, 1>, b.n, 32, 0, st, b);
    if (b.n <= t.saber_finish_five_max) return launch_next(follows, finish_chain_kernel<L, OP>, blocks(3), 64, 0, st, b);
    if (b.n <= t.saber_pair_max) return launch_next(follows, finish_multi_kernel<L, OP, 2>, blocks(16), 32, 0, st, b);
  }
  return launch_next(follows, finish_kernel<L, OP>, blocks(t.thread_block), t.thread_block, 0, st, b);
}

__host__ __device__ constexpr int op_of(int mode) {
  return mode == sdev::PM_KEYPAIR ? OP_KEYPAIR : mode == sdev::PM_ENC ? OP_ENC : OP_DEC;
}

template <int L, int MODE, bool I32>
__global__ void __launch_bounds__(256) product_dp4a_kernel(SaberBatch b) {
  next_may_start();
  wait_predecessor();
  extern __shared__ __align__(1024) uint8_t sm[];
  sdev::product_dp4a_cta<L, MODE, I32>(inst_of<L>(b, blockIdx.x, op_of(MODE)), sm, b.sliced != 0);
}

template <int L, int MODE>
__global__ void __launch_bounds__(256) product_tc_kernel(SaberBatch b) {
  using Y = TL<L>;
  next_may_start();
  extern __shared__ __align__(1024) uint8_t sm[];
  uint32_t *tslot = reinterpret_cast<uint32_t *>(sm + Y::TSLOT);
  if (threadIdx.x < 32) {
    tmem_alloc(tslot, 32);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tbase = *tslot;
  wait_predecessor();
  sdev::product_tc_cta<L, MODE>(inst_of<L>(b, blockIdx.x, op_of(MODE)), sm, tbase, b.err, b.sliced != 0);
  tc_fence_before();
  __syncthreads();
  if (threadIdx.x < 32) {
    tc_fence_after();
    tmem_dealloc(tbase, 32);
  }
}

// Persistent tensor-core product: each CTA keeps its TMEM columns and mbarrier across the
// instances it takes (i = blockIdx.x, + gridDim.x, ...) and loads the next instance's
// packed operands into registers while the current one is processed, so an instance's
// global-load latency hides behind the previous instance's work.  The launch bound asks for
// kProductCtas<L> resident CTAs per SM (40 registers at six; FireSaber's shared memory allows four)
// and the grid never has more: a seventh CTA waits for a whole CTA's share of the batch.  Encaps
// product, us, 4 / 5 / 6 / 7 CTAs per SM, measured before the last changes to its stores: l = 3, 16,384
// instances 143 / 142 / 134 / 162; l = 4, 8,192 170 / 242 / 209 / 186.
template <int L>
constexpr int kProductCtas = L == 4 ? 4 : 6;
template <int L, int MODE>
__global__ void __launch_bounds__(256, kProductCtas<L>) product_tc_persistent_kernel(SaberBatch b) {
  using Y = TL<L>;
  next_may_start();
  extern __shared__ __align__(1024) uint8_t sm[];
  uint32_t *tslot = reinterpret_cast<uint32_t *>(sm + Y::TSLOT);
  uint64_t *bar = reinterpret_cast<uint64_t *>(sm + Y::BAR);
  if (threadIdx.x < 32) {
    tmem_alloc(tslot, 32);
    tmem_relinquish();
  }
  if (threadIdx.x == 0) {
    mbar_init(bar, 1);
    fence_mbar_init();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tbase = *tslot;
  wait_predecessor();
  constexpr int op = op_of(MODE);
  sdev::OperandPrefetch<L, MODE> pf;
  int i = blockIdx.x;
  if (i < b.n) pf.load(inst_of<L>(b, i, op));
  uint32_t phase = 0;
  bool ok = true;
  for (; i < b.n; i += gridDim.x) {
    pf.store(sm, b.sliced != 0);  // the staging area is free: the previous instance's MMAs have read it
    __syncthreads();
    if (i + (int)gridDim.x < b.n) pf.load(inst_of<L>(b, i + gridDim.x, op));
    ok = sdev::tc_product<L, MODE>(inst_of<L>(b, i, op), sm, tbase, b.err, phase) && ok;
    phase ^= 1u;
  }
  tc_fence_before();
  __syncthreads();
  if (threadIdx.x == 0 && ok) mbar_inval(bar);
  if (threadIdx.x < 32) {
    tc_fence_after();
    tmem_dealloc(tbase, 32);
  }
}

template <typename K>
cudaError_t prep(K kernel, int bytes) {
  return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
}

template <int L, int MODE>
cudaError_t launch_product(const SaberBatch &b, int form, cudaStream_t st, bool follows) {
  using Y = PL<L>;
  cudaError_t e;
  if (form == FORM_TC) {
    constexpr int bytes = TL<L>::TOTAL;
    const int per_sm = tuning().saber_tc_ctas_per_sm;
    if (per_sm > 0) {
      // persistent: per_sm CTAs per SM, several instances each.  The CTAs never wait on one
      // another, so a grid larger than what is resident only queues; TMEM (32 columns per
      // CTA) fits 16 CTAs per SM.
      if ((e = prep(product_tc_persistent_kernel<L, MODE>, bytes)) != cudaSuccess) return e;
      static std::atomic<uint64_t> carved{0};  // per instantiation, a bit per device
      int dev = 0;
      if ((e = cudaGetDevice(&dev)) != cudaSuccess) return e;
      const uint64_t bit = 1ull << (dev & 63);
      if (!(carved.load(std::memory_order_relaxed) & bit)) {
        if ((e = cudaFuncSetAttribute(product_tc_persistent_kernel<L, MODE>,
                                      cudaFuncAttributePreferredSharedMemoryCarveout, 100)) != cudaSuccess)
          return e;
        carved.fetch_or(bit, std::memory_order_relaxed);
      }
      const int grid = std::min(b.n, device_sms() * std::min(per_sm, kProductCtas<L>));
      return launch_next(follows, product_tc_persistent_kernel<L, MODE>, grid, 256, bytes, st, b);
    } else {
      if ((e = prep(product_tc_kernel<L, MODE>, bytes)) != cudaSuccess) return e;
      return launch_next(follows, product_tc_kernel<L, MODE>, b.n, 256, bytes, st, b);
    }
  } else if (form == FORM_INT32) {
    constexpr int bytes = Y::DP4A_TOTAL;
    if ((e = prep(product_dp4a_kernel<L, MODE, true>, bytes)) != cudaSuccess) return e;
    return launch_next(follows, product_dp4a_kernel<L, MODE, true>, b.n, 256, bytes, st, b);
  } else {
    constexpr int bytes = Y::DP4A_TOTAL;
    if ((e = prep(product_dp4a_kernel<L, MODE, false>, bytes)) != cudaSuccess) return e;
    return launch_next(follows, product_dp4a_kernel<L, MODE, false>, b.n, 256, bytes, st, b);
  }
}

inline void mark(const SaberBatch &b, cudaStream_t st) {
  if (b.timer) b.timer->mark(st);
}

template <int L>
cudaError_t run(const SaberBatch &batch, int op, int form, cudaStream_t st) {
  SaberBatch b = batch;
  b.sliced = prologue_lanes<L>(b.n, op) == 2;
  const bool next = b.timer == nullptr && b.n <= follow_max<L>(op, form);  // stages are timed one after the other
  cudaError_t e;
  mark(b, st);
  switch (op) {
    case OP_KEYPAIR:
      if ((e = launch_prologue<L, OP_KEYPAIR>(b, st, false)) != cudaSuccess) return e;
      mark(b, st);
      if ((e = launch_product<L, sdev::PM_KEYPAIR>(b, form, st, next)) != cudaSuccess) return e;
      mark(b, st);
      if ((e = launch_finish<L, OP_KEYPAIR>(b, st, next)) != cudaSuccess) return e;
      break;
    case OP_ENC:
      if ((e = launch_prologue<L, OP_ENC>(b, st, false)) != cudaSuccess) return e;
      mark(b, st);
      if ((e = launch_product<L, sdev::PM_ENC>(b, form, st, next)) != cudaSuccess) return e;
      mark(b, st);
      if ((e = launch_finish<L, OP_ENC>(b, st, next)) != cudaSuccess) return e;
      break;
    default:
      if (b.aux && !b.timer && matrix_beside_inner<L>(b.n)) {
        // GenMatrix needs the seed alone, the other sponges m': it runs beside the inner product and the
        // hash chain that follows it.
        if ((e = cudaEventRecord(b.fork, st)) != cudaSuccess) return e;
        if ((e = cudaStreamWaitEvent(b.aux, b.fork, 0)) != cudaSuccess) return e;
        if ((e = launch_prologue<L, OP_DEC>(b, b.aux, false, 1, 1)) != cudaSuccess) return e;
        if ((e = cudaEventRecord(b.join, b.aux)) != cudaSuccess) return e;
        if ((e = launch_product<L, sdev::PM_DEC_INNER>(b, form, st, false)) != cudaSuccess) return e;
        if ((e = launch_prologue<L, OP_DEC>(b, st, next, 0, 1)) != cudaSuccess) return e;
        if ((e = cudaStreamWaitEvent(st, b.join, 0)) != cudaSuccess) return e;
        if ((e = launch_product<L, sdev::PM_DEC_CMP>(b, form, st, false)) != cudaSuccess) return e;
      } else {
        if ((e = launch_product<L, sdev::PM_DEC_INNER>(b, form, st, false)) != cudaSuccess) return e;
        mark(b, st);
        if ((e = launch_prologue<L, OP_DEC>(b, st, next)) != cudaSuccess) return e;
        mark(b, st);
        if ((e = launch_product<L, sdev::PM_DEC_CMP>(b, form, st, next)) != cudaSuccess) return e;
      }
      mark(b, st);
      if ((e = launch_finish<L, OP_DEC>(b, st, next)) != cudaSuccess) return e;
      break;
  }
  mark(b, st);
  return cudaGetLastError();
}

cudaError_t dispatch(const SaberBatch &b, int op, int form, cudaStream_t st) {
  if (b.n <= 0) return cudaSuccess;
  switch (b.level) {
    case 2: return run<2>(b, op, form, st);
    case 3: return run<3>(b, op, form, st);
    case 4: return run<4>(b, op, form, st);
    default: return cudaErrorInvalidValue;
  }
}

}  // namespace

size_t saber_scratch_bytes(int level) {
  switch (level) {
    case 2: return Scr<2>::BYTES;
    case 3: return Scr<3>::BYTES;
    case 4: return Scr<4>::BYTES;
    default: return 0;
  }
}

cudaError_t saber_keypair(const SaberBatch &b, int form, cudaStream_t st) { return dispatch(b, OP_KEYPAIR, form, st); }
cudaError_t saber_enc(const SaberBatch &b, int form, cudaStream_t st) { return dispatch(b, OP_ENC, form, st); }
cudaError_t saber_dec(const SaberBatch &b, int form, cudaStream_t st) { return dispatch(b, OP_DEC, form, st); }

}  // namespace dpkem

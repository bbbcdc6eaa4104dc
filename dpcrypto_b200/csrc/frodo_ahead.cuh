// FrodoKEM-976 with A generated ahead of its use (tensor-core form, a key per instance).
//
// A depends on seedA alone, not on the sampling stream, so its rows (11,712 permutations per
// instance) need not wait for the prologue (up to 348 dependent ones, one to a few warps'
// worth of issue slots).  The front kernel runs both: a few blocks the sponge chains, all others
// the rows of A, stored as operand tiles.  The product of an instance is then a pass of
// tcgen05 MMAs over its 2.1 MB of tiles, on three CTAs (few instances: six).
//
//   front    blocks [0, chain): the prologue's sponges; [chain, chain + absorb): decaps'
//            ciphertext pre-absorb; the rest: 256 rows of A each, a row per thread
//   product  S'A (encaps, decaps) per (instance, range of column blocks), or A S (keypair)
//            per (instance, 128 rows)
//   tail     encaps / keypair: the second half of the sampling stream (E', E''; E) and the
//            final hash in step, see tail_kernel
//
// A front block takes an SM to itself (kFrontSmem): a chain warp that shares its sub-partition
// with warps that keep the integer pipe full runs several times slower, and the chain is
// what the batch waits for.
//
// Tile layout: rows in groups of 128, the 84 columns of one squeeze block as their 168
// bytes in stream order (byte 2e / 2e + 1 = low / high byte of entry e).  Byte b of row r of
// a tile is at (b / 16) * 2048 + (r / 8) * 128 + (r % 8) * 16 + b % 16: 8 x 16-byte core matrices,
// which tcgen05 reads as an MN-major operand (M = bytes, K = rows: S'A) and as a K-major one
// (M = rows, K = bytes: A S).  A warp's 32 rows store 512 contiguous bytes per 16 columns.
#pragma once
#include "frodo_chain.cuh"
#include "frodo_gemm.cuh"

namespace dpkem {
namespace ahead {

using namespace frodo;
using fdev::Inst;
using fdev::inst_of;
using namespace fchain;

// A batch's instances for the chains.
template <int OP>
struct BatchInsts {
  const FrodoBatch &b;
  int n;
  __device__ __forceinline__ explicit BatchInsts(const FrodoBatch &batch) : b(batch), n(batch.n) {}
  __device__ __forceinline__ Inst operator()(int i) const { return inst_of(b, i, OP); }
};

constexpr int TROWS = 128, TILES = 8, BLKS = 12;
constexpr int CHUNKS = 11, LAST_CHUNKS = 7;              // 16-byte chunks of a block (84 entries) and of block 11 (52)
constexpr int CHUNK_BYTES = TROWS * 16;
constexpr int TILE_BYTES = CHUNKS * CHUNK_BYTES;         // 22,528
constexpr size_t A_BYTES = (size_t)TILES * BLKS * TILE_BYTES;  // 2,162,688 per instance

// More than half an SM's shared memory: one front block per SM.
constexpr int kFrontSmem = 120 * 1024;
constexpr int kFrontWarps = 16;

// ---------------------------------------------------------------- front
enum Stage : int { F_KEYPAIR = 0, F_ENC = 1, F_DEC = 2 };

// Row j of an instance from generator gen into the instance's tiles (every lane of the warp).
template <class G>
__device__ __forceinline__ void store_row(G &gen, uint8_t *tiles, int j, bool live) {
  uint2 a[25];
  gen.start(a, j);
  uint8_t *dst = tiles + (size_t)(j / TROWS) * (BLKS * TILE_BYTES) + ((j % TROWS) >> 3) * 128 + (j & 7) * 16;
  for (int blk = 0; blk < BLKS; blk++, dst += TILE_BYTES) {
    gen.next(a);
    if (live) {
#pragma unroll
      for (int c = 0; c < CHUNKS - 1; c++)
        if (c < LAST_CHUNKS || blk < BLKS - 1)
          *reinterpret_cast<uint4 *>(dst + c * CHUNK_BYTES) =
              make_uint4(a[2 * c].x, a[2 * c].y, a[2 * c + 1].x, a[2 * c + 1].y);
      if (blk < BLKS - 1) *reinterpret_cast<uint2 *>(dst + (CHUNKS - 1) * CHUNK_BYTES) = a[20];
    }
  }
}

// A warp's generator of 32 consecutive rows.  SHAKE rows: any 32 rows of the batch, numbered through
// its instances (the seed is per thread).  AES rows: rows of one instance, whose key schedule
// the warp expands; the block shares the round table.
template <class G>
struct WarpRows;

template <>
struct WarpRows<fdev::ShakeRows> {
  static constexpr int SMEM = 0;
  __host__ __device__ static int tasks(int m) { return (m * N + 31) / 32; }
  __device__ static void prepare(uint8_t *) {}
  template <class Seed>
  __device__ __forceinline__ static void run(int task, int m, uint8_t *tiles, uint8_t *, Seed seed) {
    const int g = task * 32 + (threadIdx.x & 31);
    const bool live = g < m * N;
    const int i = live ? g / N : 0, j = live ? g - i * N : 0;
    fdev::ShakeRows gen;
    gen.setup(seed(i), nullptr);
    store_row(gen, tiles + (size_t)i * A_BYTES, j, live);
  }
};

template <int C>
struct WarpRows<fdev::AesRows<C>> {
  static constexpr int TABLE = 256 * C * 4, KEY = 52 * 4, PER_INST = (N + 31) / 32;
  static constexpr int SMEM = TABLE + 16 * KEY;
  __host__ __device__ static int tasks(int m) { return m * PER_INST; }
  __device__ static void prepare(uint8_t *smem) {
    for (int i = threadIdx.x; i < 256 * C; i += blockDim.x)
      reinterpret_cast<uint32_t *>(smem)[i] = fdev::kAesTable.te[i / C];
    __syncthreads();
  }
  template <class Seed>
  __device__ __forceinline__ static void run(int task, int, uint8_t *tiles, uint8_t *smem, Seed seed) {
    const int i = task / PER_INST, lane = threadIdx.x & 31, j = 32 * (task - i * PER_INST) + lane;
    uint32_t *key = reinterpret_cast<uint32_t *>(smem + TABLE + (threadIdx.x >> 5) * KEY);
    __syncwarp();
    if (lane == 0) {
      fdev::AesRows<C>::expand(seed(i), key);
      key[48] = 4 * C;
    }
    __syncwarp();
    fdev::AesRows<C> gen;
    gen.rk = key;
    gen.base = smem_u32(smem + 4 * (lane % C));
    store_row(gen, tiles + (size_t)i * A_BYTES, j < N ? j : N - 1, j < N);
  }
};

// A block's share of the rows, 32 per warp and task.  The first tasks are dealt across the
// `early` blocks that start at once (few tasks: one warp per SM, not sixteen on some), the
// others come from the queue {head, blocks done}, which the last block leaves zeroed for the
// next launch.
template <int STAGE, class G>
__device__ __forceinline__ void rows_block(const FrodoBatch &b, int block, int blocks, int early, uint8_t *smem) {
  using R = WarpRows<G>;
  constexpr int op = STAGE == F_KEYPAIR ? OP_KEYPAIR : STAGE == F_ENC ? OP_ENC : OP_DEC;
  R::prepare(smem);
  const int lane = threadIdx.x & 31, tasks = R::tasks(b.ahead);
  auto seed = [&](int i) -> const uint8_t * {
    const Inst v = inst_of(b, i, op);
    return STAGE == F_DEC ? v.sk + LENS : v.pk;
  };
  bool dealt = block < early;
  while (true) {
    int task = (threadIdx.x >> 5) * early + block;
    if (!dealt) {
      if (lane == 0) task = kFrontWarps * early + (int)atomicAdd(b.queue, 1u);
      task = __shfl_sync(0xffffffffu, task, 0);
    }
    dealt = false;
    if (task >= tasks) break;
    R::run(task, b.ahead, b.atile, smem, seed);
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();
    if (atomicAdd(b.queue + 1, 1u) == (uint32_t)blocks - 1) {
      b.queue[0] = 0;
      b.queue[1] = 0;
    }
  }
}

// One block of chains on ten lanes: cw chain warps (three instances each, from block * cw * 3 on) and a
// helper warp for each, on another SM sub-partition.  HALVE: stop the sampling stream after S'
// (S^T) and keep its state (tail_kernel goes on).
template <int ROLE, bool HALVE, bool TWO>
__device__ __forceinline__ void chain_block(const FrodoBatch &b, int block, int cw, int warp, uint8_t *smem) {
  constexpr int words = HALVE ? HALF : ROLE == R_KEYPAIR ? 2 * HALF : RW, squeezes = (words + 67) / 68 - 1;
  const int lane = threadIdx.x & 31;
  const bool helper = warp >= cw;
  const int w = helper ? (warp - cw + 2) % cw : warp, first = (block * cw + w) * 3;
  if (warp >= 2 * cw || first >= b.n) return;
  Exchange &x = reinterpret_cast<Exchange *>(smem)[w];
  uint8_t *xbuf = smem + cw * sizeof(Exchange) + w * k10::kSmemPerWarp;
  if (helper) {
    if (ROLE == R_DEC && lane < 3 && first + lane < b.n) b.fail[first + lane] = 0;
    helper_warp<ROLE, TWO>(BatchInsts<Steps<ROLE>::op>(b), first, words, x, w);
  } else {
    chain_warp<ROLE, TWO>(BatchInsts<Steps<ROLE>::op>(b), first, squeezes, HALVE, x, xbuf, w);
  }
}
constexpr int chain_smem(int cw) { return cw * (int)(sizeof(Exchange) + k10::kSmemPerWarp); }
static_assert(sizeof(Exchange) % 16 == 0 && k10::kSmemPerWarp % 16 == 0, "16-byte aligned transpose buffers");

// Decaps: the final hash over ct's full blocks, which does not wait for k.  Half as long as the
// sampling chain, so it runs on lane pairs: 135 integer instructions per state and permutation
// against the ten lanes' 160, and two shuffles against six shared-memory pipe cycles.
constexpr int kAbsorbWarps = 4;
__device__ __forceinline__ void absorb_warp(const FrodoBatch &b, int w) {
  using S = msp::Multi<2>;
  const S s(nullptr);
  const int i = w * S::STATES_PER_WARP + s.state();
  if (w * S::STATES_PER_WARP >= b.n) return;
  const bool live = i < b.n;
  fdev::ct_absorb_multi<S>(inst_of(b, live ? i : b.n - 1, OP_DEC), s, live);
}

// NS: lanes per state of the sponges (10: ten lanes, 0: one lane, a thread per instance).
// Chain blocks run `chain_warps` chain warps each (at most 8); row blocks [0, early) find an SM
// at once.
template <int STAGE, int NS, bool HALVE, class G>
__global__ void __launch_bounds__(32 * kFrontWarps, 1) front_kernel(FrodoBatch b, int chain_warps, int chain_blocks,
                                                                    int absorb_blocks, int early) {
  extern __shared__ __align__(1024) uint8_t smem[];
  const int warp = threadIdx.x >> 5;
  constexpr int op = STAGE == F_KEYPAIR ? OP_KEYPAIR : STAGE == F_ENC ? OP_ENC : OP_DEC;
  const int first_rows = chain_blocks + absorb_blocks;
  if ((int)blockIdx.x >= first_rows) {
    rows_block<STAGE, G>(b, blockIdx.x - first_rows, gridDim.x - first_rows, early, smem);
    return;
  }
  const bool absorb = STAGE == F_DEC && (int)blockIdx.x >= chain_blocks;
  const int block = absorb ? blockIdx.x - chain_blocks : blockIdx.x;
  if constexpr (NS == 0) {
    const int cw = absorb ? kFrontWarps : chain_warps;
    const int i = (block * cw + warp) * 32 + (threadIdx.x & 31);
    if (warp >= cw || i >= b.n) return;
    const Inst v = inst_of(b, i, op);
    uint2 *park = reinterpret_cast<uint2 *>(smem) + threadIdx.x;
    if constexpr (STAGE == F_DEC) {
      if (absorb) {
        fdev::ct_absorb_inst(v);
        return;
      }
      *v.fail = 0;
      fdev::prologue_inst<OP_DEC>(v, park, 32 * kFrontWarps);
    } else if constexpr (STAGE == F_ENC) {
      fdev::prologue_inst<OP_ENC>(v, park, 32 * kFrontWarps);
    } else {
      fdev::kp_prologue_inst(v, park, 32 * kFrontWarps);
    }
  } else {
    if (absorb) {
      if constexpr (STAGE == F_DEC)
        if (warp < kAbsorbWarps) absorb_warp(b, block * kAbsorbWarps + warp);
    } else {
      chain_block<STAGE == F_KEYPAIR ? R_KEYPAIR : STAGE == F_ENC ? R_ENC : R_DEC, HALVE, false>(b, block, chain_warps,
                                                                                                 warp, smem);
    }
  }
}

// The chains alone, for batches whose A needs no generating (one key) or runs in another form: two
// chain and two helper warps a block (small blocks spread evenly over the SMs; every other wave of
// blocks holds the helpers first, so every sub-partition gets both), decaps' absorb blocks after them.
template <int ROLE>
__global__ void __launch_bounds__(128, 6) chains_kernel(FrodoBatch b, int chain_blocks) {
  extern __shared__ __align__(16) uint8_t smem[];
  const int warp = threadIdx.x >> 5, block = blockIdx.x;
  const bool swap = exchange_roles();
  if (block < chain_blocks) {
    chain_block<ROLE, false, true>(b, block, 2, (warp + (swap ? 2 : 0)) & 3, smem);
    return;
  }
  if constexpr (ROLE == R_DEC) absorb_warp(b, (block - chain_blocks) * kAbsorbWarps + warp);
}

// seedA = SHAKE256(z, 16) into pk, one thread per instance: the front kernel's rows need it.
__global__ void __launch_bounds__(32) kp_seed_kernel(FrodoBatch b) {
  const int i = blockIdx.x * 32 + threadIdx.x;
  if (i >= b.n) return;
  write_seed_a(inst_of(b, i, OP_KEYPAIR));
}

// ---------------------------------------------------------------- product S'A
// CTA (256 threads) = one instance, column blocks [b0, b0 + NB).  Warp 0 lane 0 moves the tiles
// (one bulk copy each) through an NST-stage mbarrier ring, warp 1 lane 0 issues the MMAs (per
// 32 rows: bytes 0..127 and 128..167 of the block, N = 8), the CTA of the last block also forms
// V = S'B on warps 2..7 meanwhile.  All eight warps read the accumulators back.
// PM_RAW: the products mod 2^16 replace E' / E'' in rw (V plus Encode(mu)); tail_kernel adds
// the errors.  PM_ENC: ciphertext.  PM_DEC: compare, an OR into the fail word.
enum PMode : int { PM_RAW = 0, PM_ENC = 1, PM_DEC = 2 };
constexpr int P_NST = 4;
// Column blocks of a CTA: four read S' three times an instance; up to kProductFew instances two, whose MMAs are half as
// many one after the other.  us, 1 / 2 / 4 blocks, decaps: n = 1 502 / 501 / 504, 8 528 / 527 / 530, 24 534 / 532 / 534, 32
// 554 / 547 / 548, 128 617 / 609 / 600, 1,024 3,618 / 3,536 / 3,503; encaps: 1 745 / 744 / 744, 32 783 / 781 / 778, 1,024 3,786 / 3,722 /
// 3,700.
constexpr int kProductFew = 24;
__host__ __device__ constexpr uint32_t product_cols(int nb) { return nb <= 2 ? 32 : 64; }  // TMEM columns

struct PLayout {
  static constexpr int sp = 0;                                   // S' operand, 62 * 128
  static constexpr int ring = 8192;
  // the second MMA of a stage reads M-chunks 8..15, five past the tile's eleven
  static constexpr int bars = ring + P_NST * TILE_BYTES + 5 * CHUNK_BYTES;
  static constexpr int tslot = bars + (2 * P_NST + 1) * 8;
  static constexpr int red = (tslot + 4 + 15) & ~15;             // 3 x 64 partial sums of V
  static constexpr int total = red + 3 * 64 * 4;
};

template <int MODE, int NB>
__global__ void __launch_bounds__(256, 2) product_kernel(FrodoBatch b) {
  using L = PLayout;
  extern __shared__ __align__(1024) uint8_t smem[];
  constexpr int op = MODE == PM_DEC ? OP_DEC : OP_ENC;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  constexpr int parts = BLKS / NB, nst = NB * TILES;
  const int inst = blockIdx.x / parts, b0 = (blockIdx.x % parts) * NB, b1 = b0 + NB;
  const Inst v = inst_of(b, inst, op);
  const uint8_t *tiles = b.atile + (size_t)inst * A_BYTES;
  uint8_t *sp = smem + L::sp;
  uint64_t *full = reinterpret_cast<uint64_t *>(smem + L::bars), *empty = full + P_NST, *done = full + 2 * P_NST;
  uint32_t *tslot = reinterpret_cast<uint32_t *>(smem + L::tslot);
  uint32_t(*red)[64] = reinterpret_cast<uint32_t(*)[64]>(smem + L::red);
  const uint16_t *rw = v.rw;
  if (warp == 0) {
    tmem_alloc(tslot, product_cols(NB));
    tmem_relinquish();
  }
  if (tid == 32) {
    for (int q = 0; q < 2 * P_NST + 1; q++) mbar_init(&full[q], 1);
    fence_mbar_init();
  }
  for (int q = tid; q < 62 * NBAR; q += 256) {  // S'^T, K-major s8, as in sa_tc_cta
    const int g = q >> 3, k = q & 7;
    uint4 o = make_uint4(0, 0, 0, 0);
    if (16 * g < N) {
      const uint4 x0 = *reinterpret_cast<const uint4 *>(rw + k * N + 16 * g);
      const uint4 x1 = *reinterpret_cast<const uint4 *>(rw + k * N + 16 * g + 8);
      o = make_uint4(prmt(x0.x, x0.y, 0x6420), prmt(x0.z, x0.w, 0x6420), prmt(x1.x, x1.y, 0x6420),
                     prmt(x1.z, x1.w, 0x6420));
    }
    *reinterpret_cast<uint4 *>(sp + g * 128 + k * 16) = o;
  }
  fence_proxy_async_smem();
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tbase = *tslot;
  bool ok = true;
  if (warp == 0) {
    if (lane == 0) {  // producer
      for (int u = 0; u < nst; u++) {
        const int q = u % P_NST, blk = b0 + u / TILES, t = u % TILES;
        if (u >= P_NST && !(ok = mbar_wait(&empty[q], ((u / P_NST) - 1) & 1))) break;
        const uint32_t bytes = (blk < BLKS - 1 ? CHUNKS : LAST_CHUNKS) * CHUNK_BYTES;
        fgemm::mbar_expect_tx(&full[q], bytes);
        fgemm::bulk_g2s(smem_u32(smem + L::ring + q * TILE_BYTES), tiles + (size_t)(t * BLKS + blk) * TILE_BYTES, bytes,
                        &full[q]);
      }
    }
  } else if (warp == 1) {
    if (lane == 0) {  // MMA issuer
      constexpr uint32_t idesc = idesc_i8(128, 8, false, true, true, false);
      const uint32_t sp_addr = smem_u32(sp);
      for (int u = 0; u < nst; u++) {
        const int q = u % P_NST, t = u % TILES;
        const uint32_t d = tbase + (u / TILES) * 16;
        if (!(ok = mbar_wait(&full[q], (u / P_NST) & 1))) break;
        tc_fence_after();
        const uint32_t sa = smem_u32(smem + L::ring + q * TILE_BYTES);
        const int ksteps = t < TILES - 1 ? 4 : 3;  // rows 896..991 of the last tile (S' is zero from 976 on)
        for (int ks = 0; ks < ksteps; ks++) {
          const uint64_t bd = sdesc(sp_addr + t * 1024 + ks * 256, 128, 1024);
          const uint32_t acc = (t | ks) ? 1u : 0u;
          mma_i8(d, sdesc(sa + ks * 512, 128, CHUNK_BYTES), bd, idesc, acc);
          mma_i8(d + 8, sdesc(sa + ks * 512 + 8 * CHUNK_BYTES, 128, CHUNK_BYTES), bd, idesc, acc);
        }
        mma_commit(&empty[q]);
      }
      if (ok) mma_commit(done);
    }
  } else if (b1 == BLKS) {  // V = S'B: 64 outputs, three segments of rows
    const int x = tid - 64, o = x & 63, seg = x >> 6, k = o >> 3, l = o & 7;
    const uint8_t *bsrc = (op == OP_ENC ? v.pk : v.sk + LENS) + SEEDA + 2 * l;
    uint32_t acc = 0;
    const int j1 = min(N, 326 * seg + 326);
#pragma unroll 4
    for (int j = 326 * seg; j < j1; j++) {
      const uint32_t w = *reinterpret_cast<const uint16_t *>(bsrc + 16 * j);
      const int32_t s = (int8_t)sp[(j >> 4) * 128 + k * 16 + (j & 15)];
      acc += (uint32_t)s * ((w >> 8) | ((w & 0xFFu) << 8));
    }
    red[seg][o] = acc;
  }
  __syncwarp();
  __syncthreads();
  const bool fin = mbar_wait(done, 0);
  // every stage's last commit, before the barriers' memory goes away with the CTA
  if (tid == 0 && fin)
    for (int q = 0; q < P_NST; q++) {
      const int last = nst - 1 - ((nst - 1 - q) % P_NST);
      mbar_wait(&empty[q], (last / P_NST) & 1);
    }
  if ((!fin || !ok) && lane == 0) atomicOr(b.err, DEV_ERR_TIMEOUT);
  tc_fence_after();
  uint32_t diff = 0;
  if (__all_sync(0xffffffffu, fin)) {
    // TMEM lane 2e: low-byte sum of entry e, lane 2e + 1: high-byte sum (see sa_tc_cta).
    const int qd = warp & 3, t = qd * 32 + lane;
    for (int blk = b0 + (warp >> 2); blk < b1; blk += 2) {
      uint32_t r[16];
      tmem_ld16(tbase + ((uint32_t)(qd * 32) << 16) + (blk - b0) * 16, r);
      tmem_wait_ld();
#pragma unroll
      for (int q = 0; q < 16; q++) r[q] += __shfl_down_sync(0xffffffffu, r[q], 1) << 8;
      const int valid = blk < BLKS - 1 ? 84 : 52;
#pragma unroll
      for (int h = 0; h < 2; h++) {
        const int e = 64 * h + (t >> 1);
        if ((lane & 1) == 0 && e < valid && (h == 0 || t < 40)) {
          const int col = 84 * blk + e;
#pragma unroll
          for (int k = 0; k < 8; k++) {
            uint16_t *ep = v.rw + HALF + k * N + col;
            if (MODE == PM_RAW) {
              *ep = (uint16_t)r[8 * h + k];
              continue;
            }
            const uint32_t x = (r[8 * h + k] + *ep) & 0xFFFFu, be = (x >> 8) | ((x & 0xFFu) << 8);
            uint16_t *d = reinterpret_cast<uint16_t *>(v.ct + 2 * (k * N + col));
            if (MODE == PM_ENC) *d = (uint16_t)be;
            else diff |= be ^ *d;
          }
        }
      }
    }
    if (b1 == BLKS && tid < 64) {
      uint16_t *epp = v.rw + 2 * HALF;
      const uint8_t *mu = MODE == PM_DEC ? v.mu : v.coins;
      const int kr = tid >> 3, lc = tid & 7;
      const uint32_t t3 = mu[3 * kr] | ((uint32_t)mu[3 * kr + 1] << 8) | ((uint32_t)mu[3 * kr + 2] << 16);
      const uint32_t c = red[0][tid] + red[1][tid] + red[2][tid] + (((t3 >> (3 * lc)) & 7u) << 13);
      if (MODE == PM_RAW) {
        epp[tid] = (uint16_t)c;
      } else {
        const uint32_t x = (c + epp[tid]) & 0xFFFFu, be = (x >> 8) | ((x & 0xFFu) << 8);
        uint16_t *d = reinterpret_cast<uint16_t *>(v.ct + PKB + 2 * tid);
        if (MODE == PM_ENC) *d = (uint16_t)be;
        else diff |= be ^ *d;
      }
    }
  }
  if (MODE == PM_DEC && __any_sync(0xffffffffu, diff != 0) && lane == 0) atomicOr(v.fail, 1u);
  tc_fence_before();
  __syncthreads();
  if (warp == 0) {
    tc_fence_after();
    tmem_dealloc(tbase, product_cols(NB));
  }
}

// ---------------------------------------------------------------- product A S (keypair)
// CTA (256 threads) = one instance, 128 rows: D[i][n] = sum over the row's bytes, N = 16: rows
// n < 8 of the S^T operand hold S^T[n] under the low bytes (even K) and zeros under the high
// bytes, rows n >= 8 the reverse, so B[i][k] = D[i][k] + 256 D[i][8 + k] (mod 2^16).  K runs over a
// block's 168 bytes in steps of 32, zero-padded in the S^T operand.
// RAW: the products replace E in rw (tail_kernel adds E); else pk and sk are written.
constexpr int K_NST = 3;
constexpr int KS_BLK = 12 * 256;  // S^T operand of a block: 12 chunks of 16 K bytes x 16 rows

struct KLayout {
  static constexpr int st = 0;
  static constexpr int ring = BLKS * KS_BLK;
  static constexpr int bars = ring + K_NST * TILE_BYTES + CHUNK_BYTES;  // the last K step reads a twelfth chunk
  static constexpr int tslot = bars + (2 * K_NST + 1) * 8;
  static constexpr int total = tslot + 8;
};

template <bool RAW>
__global__ void __launch_bounds__(256, 2) product_kp_kernel(FrodoBatch b) {
  using L = KLayout;
  extern __shared__ __align__(1024) uint8_t smem[];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int inst = blockIdx.x / TILES, t = blockIdx.x % TILES;
  const Inst v = inst_of(b, inst, OP_KEYPAIR);
  const uint8_t *tiles = b.atile + (size_t)inst * A_BYTES + (size_t)t * BLKS * TILE_BYTES;
  uint64_t *full = reinterpret_cast<uint64_t *>(smem + L::bars), *empty = full + K_NST, *done = full + 2 * K_NST;
  uint32_t *tslot = reinterpret_cast<uint32_t *>(smem + L::tslot);
  const uint16_t *rw = v.rw;
  if (warp == 0) {
    tmem_alloc(tslot, 32);
    tmem_relinquish();
  }
  if (tid == 32) {
    for (int q = 0; q < 2 * K_NST + 1; q++) mbar_init(&full[q], 1);
    fence_mbar_init();
  }
  // S^T operand: 16 K bytes (8 entries) of row n: byte (kk, n) of a block at
  // (kk / 16) * 256 + (n / 8) * 128 + (n % 8) * 16 + kk % 16.
  for (int x = tid; x < BLKS * 12 * 8; x += 256) {
    const int k = x & 7, c = (x >> 3) % 12, blk = x / 96, e = 8 * c, j = 84 * blk + e;
    uint2 w0 = make_uint2(0, 0), w1 = w0;  // entries e .. e + 3 and e + 4 .. e + 7 (84, and N, are multiples of 4)
    const uint16_t *src = rw + k * N + j;
    if (e < 84 && j < N) w0 = *reinterpret_cast<const uint2 *>(src);
    if (e + 4 < 84 && j + 4 < N) w1 = *reinterpret_cast<const uint2 *>(src + 4);
    const uint4 lo = make_uint4(w0.x & 0x00FF00FFu, w0.y & 0x00FF00FFu, w1.x & 0x00FF00FFu, w1.y & 0x00FF00FFu);
    uint8_t *d = smem + L::st + blk * KS_BLK + c * 256 + k * 16;
    *reinterpret_cast<uint4 *>(d) = lo;
    *reinterpret_cast<uint4 *>(d + 128) = make_uint4(lo.x << 8, lo.y << 8, lo.z << 8, lo.w << 8);
  }
  fence_proxy_async_smem();
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tbase = *tslot;
  bool ok = true;
  if (warp == 0) {
    if (lane == 0) {
      for (int blk = 0; blk < BLKS; blk++) {
        const int q = blk % K_NST;
        if (blk >= K_NST && !(ok = mbar_wait(&empty[q], ((blk / K_NST) - 1) & 1))) break;
        const uint32_t bytes = (blk < BLKS - 1 ? CHUNKS : LAST_CHUNKS) * CHUNK_BYTES;
        fgemm::mbar_expect_tx(&full[q], bytes);
        fgemm::bulk_g2s(smem_u32(smem + L::ring + q * TILE_BYTES), tiles + (size_t)blk * TILE_BYTES, bytes, &full[q]);
      }
    }
  } else if (warp == 1) {
    if (lane == 0) {
      constexpr uint32_t idesc = idesc_i8(128, 16, false, true, false, false);
      const uint32_t st_addr = smem_u32(smem + L::st);
      for (int blk = 0; blk < BLKS; blk++) {
        const int q = blk % K_NST;
        if (!(ok = mbar_wait(&full[q], (blk / K_NST) & 1))) break;
        tc_fence_after();
        const uint32_t sa = smem_u32(smem + L::ring + q * TILE_BYTES);
        const int ksteps = blk < BLKS - 1 ? 6 : 4;
        for (int ks = 0; ks < ksteps; ks++)
          mma_i8(tbase, sdesc(sa + ks * 2 * CHUNK_BYTES, CHUNK_BYTES, 128),
                 sdesc(st_addr + blk * KS_BLK + ks * 512, 256, 128), idesc, (blk | ks) ? 1u : 0u);
        mma_commit(&empty[q]);
      }
      if (ok) mma_commit(done);
    }
  }
  __syncwarp();
  __syncthreads();
  const bool fin = mbar_wait(done, 0);
  if (tid == 0 && fin)
    for (int q = 0; q < K_NST; q++) {
      const int last = BLKS - 1 - ((BLKS - 1 - q) % K_NST);
      mbar_wait(&empty[q], (last / K_NST) & 1);
    }
  if ((!fin || !ok) && lane == 0) atomicOr(b.err, DEV_ERR_TIMEOUT);
  tc_fence_after();
  if (warp < 4 && __all_sync(0xffffffffu, fin)) {
    uint32_t r[16];
    tmem_ld16(tbase + ((uint32_t)(warp * 32) << 16), r);
    tmem_wait_ld();
    const int i = TROWS * t + tid;
    if (i < N) {
      uint4 *ep = reinterpret_cast<uint4 *>(v.rw + HALF + NBAR * i);  // E[i][0..7]
      uint32_t x[8];
#pragma unroll
      for (int k = 0; k < 8; k++) x[k] = (r[k] + (r[8 + k] << 8)) & 0xFFFFu;
      if (RAW) {
        *ep = make_uint4(x[0] | (x[1] << 16), x[2] | (x[3] << 16), x[4] | (x[5] << 16), x[6] | (x[7] << 16));
      } else {
        const uint4 e = *ep;
        const uint32_t ew[4] = {e.x, e.y, e.z, e.w};
#pragma unroll
        for (int k = 0; k < 8; k++) x[k] += (ew[k >> 1] >> (16 * (k & 1))) & 0xFFFFu;
        const uint2 o0 = make_uint2(fdev::bswap16x2(x[0], x[1]), fdev::bswap16x2(x[2], x[3]));
        const uint2 o1 = make_uint2(fdev::bswap16x2(x[4], x[5]), fdev::bswap16x2(x[6], x[7]));
        *reinterpret_cast<uint2 *>(v.pk + SEEDA + 16 * i) = o0;
        *reinterpret_cast<uint2 *>(v.pk + SEEDA + 16 * i + 8) = o1;
        *reinterpret_cast<uint2 *>(v.sk + LENS + SEEDA + 16 * i) = o0;
        *reinterpret_cast<uint2 *>(v.sk + LENS + SEEDA + 16 * i + 8) = o1;
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 0) {
    tc_fence_after();
    tmem_dealloc(tbase, 32);
  }
}

// ---------------------------------------------------------------- tail
// The second half of the sampling stream yields the errors in the order in which the final
// hash absorbs the words they complete (136 bytes each per permutation), so the two sponges
// run in step: per step
//   warp 0  one permutation of the stream; its 17 rate lanes to shared memory
//   warp 1  the previous block's words: sampled errors + products (rw), big-endian, stored and
//           handed on
//   warp 2  one permutation of the hash over the block before that
// 116 permutations less on the chain of an encaps, 115 of a keypair.
//   encaps   SHAKE256(ct || k): stream word 7808 + w completes ct word w
//   keypair  H(pk) = SHAKE256(seedA || B): stream word 7808 + w completes pk word 8 + w
template <int OP>
struct Tail {
  static constexpr bool ENC = OP == OP_ENC;
  static constexpr int HASH_LANES = (ENC ? CT : PK) / 8;          // message lanes before k / the padding
  static constexpr int HASH_BLOCKS = HASH_LANES / 17 + 1;         // k and the padding fit in the last block
  static constexpr int SHIFT = ENC ? 14 : 12;                     // stream lane under hash lane 0, block 114
  static constexpr int STREAM_PERMS = ENC ? 116 : 115;            // blocks 115 .. 230 / 229
};
static_assert(HALF == 114 * 68 + 4 * 14, "E' starts at lane 14 of stream block 114");
static_assert(CT / 8 % 17 + 3 == 16 && PK / 8 % 17 == 16, "k ends, and the padding starts, at lane 16 of the last block");

// Three instances per block, ten lanes per state (keccak10.cuh).  The lanes cross between the
// warps as bit-interleaved halves {even, odd}: warp 1 converts, off the two chains.
template <int OP>
__global__ void __launch_bounds__(96) tail_kernel(FrodoBatch b) {
  using T = Tail<OP>;
  using S = msp::Multi<10>;
  __shared__ __align__(16) uint8_t xbuf[3 * S::SMEM_PER_WARP];
  __shared__ uint2 raw[3][3][17], msg[2][3][17];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const S s(xbuf + warp * S::SMEM_PER_WARP);
  const int mine = blockIdx.x * 3 + s.state();
  const bool live = mine < b.n;
  const Inst v = inst_of(b, live ? mine : b.n - 1, OP);
  uint32_t a[5];
  msp::zero<S>(a);
  auto hand_over = [&](int slot) {  // rate lanes of the stream
#pragma unroll
    for (int y = 0; y < 4; y++)
      if (s.lane(y) < 17) s.store(reinterpret_cast<uint8_t *>(&raw[slot][s.state()][s.lane(y)]), a[y]);
  };
  if (warp == 0) {
#pragma unroll
    for (int y = 0; y < 5; y++) a[y] = s.in(s.load(reinterpret_cast<const uint8_t *>(v.hs + s.lane(y))));
    hand_over(0);
  }
  __syncthreads();
  for (int t = 0; t < T::HASH_BLOCKS + 2; t++) {
    if (warp != 1) {
      if (warp == 0 ? t < T::STREAM_PERMS : t >= 2) {
        if (warp == 2) {
#pragma unroll
          for (int y = 0; y < 4; y++)
            if (s.lane(y) < 17) a[y] ^= s.load(reinterpret_cast<const uint8_t *>(&msg[t & 1][s.state()][s.lane(y)]));
        }
        k10::f1600<24>(a, s.k);
        if (warp == 0) hand_over((t + 1) % 3);
      }
    } else {
      const int h = t - 1;  // hash block
      if (h >= 0 && h < T::HASH_BLOCKS)
        for (int x = lane; x < 51; x += 32) {
          const int g = x / 17, q = x - 17 * g, i = blockIdx.x * 3 + g, m = 17 * h + q;  // message lane m
          if (i >= b.n) break;
          const Inst u = inst_of(b, i, OP);
          uint2 w;
          if (m >= T::HASH_LANES) {
            w = T::ENC && q < 16 ? ld_lane(u.kk + 8 * (m - T::HASH_LANES)) : make_uint2(0x1Fu, 0x80000000u);
          } else if (!T::ENC && m < 2) {
            w = ld_lane(u.pk + 8 * m);  // seedA
          } else {
            const int at = q + T::SHIFT, w0 = 4 * (T::ENC ? m : m - 2);  // ct word / word of B
            const uint2 p = *reinterpret_cast<const uint2 *>(u.rw + HALF + w0);
            const uint2 e = fdev::sample_lane(k10::lane_of(at < 17 ? raw[h % 3][g][at] : raw[(h + 1) % 3][g][at - 17]));
            w = make_uint2(prmt(__vadd2(e.x, p.x), 0u, 0x2301), prmt(__vadd2(e.y, p.y), 0u, 0x2301));
            if (T::ENC) {
              *reinterpret_cast<uint2 *>(u.ct + 8 * m) = w;
            } else {
              *reinterpret_cast<uint2 *>(u.pk + 8 * m) = w;
              *reinterpret_cast<uint2 *>(u.sk + LENS + 8 * m) = w;
            }
          }
          msg[h & 1][g][q] = k10::slices_of(w);
        }
    }
    __syncthreads();
  }
  if (warp == 2) msp::store<S, 3>(a, s, T::ENC ? v.ss : v.sk + SK_PKH, live);
}

}  // namespace ahead
}  // namespace dpkem

// FlashAttention-2 backward for sm_100a: dK/dV/dQ with P recomputed from the
// forward's log-sum-exp, five tcgen05 GEMMs per (key tile, query tile) pair,
// all accumulators in TMEM.
//
// Replaces precompute_D_kernel, flash_attn_bwd_volta_kernel and the fp32->fp16
// dQ cast (csrc/kernels/flash_attn_bwd.cu:76-107, :425-647 and
// csrc/flash_attn_legacy.cpp:126,184 of the reference).  Same loop nest -- a
// CTA owns one 128-key tile of one KV head and sweeps the query heads of its
// group and their (causally reachable) query tiles -- and the same math:
//   P  = exp(S*scale - L)          dV += P^T dO
//   dP = dO V^T                    dS  = P o (dP - D)      (scale applied at the end)
//   dK += dS^T Q                   dQ += dS K
// with P and dS rounded to fp16 before they feed a GEMM.
//
// S, dP, dV and dK are computed transposed (keys on the 128 TMEM lanes), 128 queries per step,
// so that every MMA is a full M=128 x N=128 instruction (an N=64 instruction costs the same
// tensor-pipe time as an N=128 one):
//   S^T  = K Q^T      (M=128 keys, N=128 queries, K=head_dim)   smem x smem
//   dP^T = V dO^T     (same shape)                              smem x smem
//   dV  += P^T dO     (M=128, N=head_dim, K=128)                TMEM x smem
//   dK  += dS^T Q     (M=128, N=head_dim, K=128)                smem x smem
//   dQ   = dS K       (M=128 queries, N=head_dim, K=128)        smem x smem (dS^T read M-contiguous)
// P^T is produced in place over S^T, a compute thread holds 16 columns of four key rows (the layout of
// stmatrix), and dS^T is written to shared memory once and serves both dK and dQ.  The dQ tile leaves TMEM through
// a swizzled shared-memory staging buffer and TMA tensor reductions (fp32 add) into the
// accumulator that the post-pass casts.
//
//   warps 0-7    compute (two per TMEM lane quarter, 64 query columns each)
//   warp  8      TMA producer
//   warp  9      tcgen05.mma issuer, TMEM owner
//   warps 10-13  dQ write-back
//   warp  14     LSE / delta staging (kept apart from the TMA producer so that neither waits
//                behind the other's global-memory latency)
//   warp  15     idle
//
// TMEM columns: S^T/P^T [0,128), dP^T/dQ [128,256) (the dQ tile of a step reuses the columns of
//               that step's consumed dP^T), dV [256,256+D), dK [256+D,256+2D).
// At head_dim 64 there is room for more, and a step is bound by the compute warps' chain (exponentials, dS, its
// stores) where nothing holds them up: S^T / P^T of odd steps have columns [384,512), so that the scores of a step are
// computed under the exponentials of the step before instead of behind its dV, Q has three buffers and dO two.  us:
// 16 x 16 384 causal 1 530 -> 1 447, 4 x 16 x 2 048 235 -> 216, 32 x 16 x 577 278 -> 260.
// Shared memory at head_dim 128: K 32K, V 32K, Q 2 x 32K, dO 32K, dS^T 32K, dQ staging 2 x 16K.
//
// head_dim 256 (SPLIT = true): two CTAs share a key tile, each owning 128 of the 256 columns of dV, dK and
// dQ.  The two score GEMMs contract over all 256 columns, so a CTA needs both halves of K, Q, V and dO:
// K and V stay in shared memory for the whole key tile (128 KB); of Q and dO the own half has a buffer and
// the other half passes through one more, X, which then takes dS^T.  A step: S^T = K Q^T (other half from X,
// own half), dP^T = V dO^T (the same), dV, dQ, dK.  128 KB a step come from L2.  Bound by the latency of a
// step's chain of loads, GEMMs and softmax, of which only the own dO's load overlaps the step before.
// 2 x 16 heads x 2 048 causal: 327 us; with K and V reloaded every step (256 KB, all eight half tiles through
// four buffers) 395.
#include <type_traits>

#include "fal_common.h"
#include "fal_launch.h"
#include "sm100_ptx.cuh"

namespace fal {

namespace {

constexpr int kBwdThreads = 512;
constexpr int kKvTile = 128;
constexpr int kQTile = 128;
constexpr float kLog2e = 1.4426950408889634f;
constexpr int kDqBoxBytes = 32 * 128;  // one dQ staging box: 32 rows of 32 fp32 columns

enum BwdBarrier : int {
  kBbKFull = 100, kBbVFull = 101, kBbQFull = 110, kBbDoFull = 120, kBbStatFull = 130,
  kBbQEmpty = 140, kBbDoEmpty = 145, kBbSReady = 150, kBbDpReady = 160, kBbPReady = 161,
  kBbDsReady = 162, kBbDqReady = 164, kBbDqFree = 165, kBbAllDone = 166, kBbAFull = 170, kBbADone = 171,
  kBbBFull = 172,
};

template <int D>
struct BwdSmem {
  static constexpr int kQStages = D == 64 ? 3 : 2;             // Q tiles and row statistics
  static constexpr int kDoStages = D == 64 ? 2 : 1;
  static constexpr int kSBuffers = D == 64 ? 2 : 1;            // S^T / P^T blocks in TMEM
  static constexpr bool kEarlyLoads = D == 64;                 // first tiles requested before the CTA-wide sync
  static constexpr int kBoxes = D / 64;
  static constexpr int kBoxBytes = 128 * 128;                  // one 128-row x 128-byte box
  static constexpr int kTileBytes = kBoxes * kBoxBytes;        // K, V, Q and dO tiles are 128 x D
  static constexpr int kKOff = 0;
  static constexpr int kVOff = kTileBytes;
  static constexpr int kQOff = 2 * kTileBytes;
  static constexpr int kDoOff = kQOff + kQStages * kTileBytes;
  static constexpr int kDsOff = kDoOff + kDoStages * kTileBytes;  // [2 boxes][128 keys][64 queries] fp16
  static constexpr int kDsBytes = 2 * kBoxBytes;
  static constexpr int kStageOff = kDsOff + kDsBytes;           // dQ staging: 2 x [128 rows][32 fp32], or per warp 2 x [32][32]
  static constexpr bool kWarpDq = D == 128;                     // the write-back warps work independently
  static constexpr int kStageBytes = 2 * kBoxBytes;
  static_assert(kStageBytes == 4 * 2 * kDqBoxBytes, "staging");
  static constexpr int kStatOff = kStageOff + kStageBytes;      // per Q stage: lse2[128], delta[128]
  static constexpr int kStatBytes = kQStages * 2 * kQTile * 4;
  static constexpr int kBarOff = kStatOff + kStatBytes;
  // k_full v_full q_full[NQ] q_empty[NQ] stat_full[NQ] do_full[ND] do_empty[ND] s_ready[NB] p_ready[NB]
  // dp_ready dq_ready dq_free ds_ready all_done ds_free a_full a_done b_full
  static constexpr int kNumBars = 2 + 3 * kQStages + 2 * kDoStages + 2 * kSBuffers + 9;
  static constexpr int kMiscOff = kBarOff + kNumBars * 8;
  static constexpr int kBytes = kMiscOff + 16;
  // No slack for re-aligning the base: at head_dim 128 the layout fills the 227 KB limit, so the
  // kernel requires the dynamic shared memory window itself to be 1024-byte aligned and reports
  // an error otherwise.
  static constexpr int kAllocBytes = kBytes;
  static_assert(kAllocBytes <= 232448, "exceeds the per-CTA shared memory limit");
};

// The layout of the head_dim 256 kernel: K and V in full (own columns, then the other CTA's), one Q and one
// dO buffer (own columns), and X = kDsOff: Q's other columns, then dO's, then dS^T.
struct BwdSplitSmem {
  static constexpr int kQStages = 1;
  static constexpr int kDoStages = 1;
  static constexpr int kSBuffers = 1;
  static constexpr bool kEarlyLoads = false;
  static constexpr int kBoxes = 2;
  static constexpr int kBoxBytes = 128 * 128;
  static constexpr int kTileBytes = kBoxes * kBoxBytes;
  static constexpr int kKOff = 0;
  static constexpr int kVOff = 2 * kTileBytes;
  static constexpr int kQOff = 4 * kTileBytes;
  static constexpr int kDoOff = 5 * kTileBytes;
  static constexpr int kDsOff = 6 * kTileBytes;
  static constexpr int kStatOff = 7 * kTileBytes;
  static constexpr int kBarOff = kStatOff + 2 * kQTile * 4;
  static constexpr int kNumBars = 2 + 3 + 2 + 2 + 9;
  static constexpr int kMiscOff = kBarOff + kNumBars * 8;
  static constexpr int kBytes = kMiscOff + 16;
  static constexpr int kAllocBytes = kBytes;
  static_assert(kAllocBytes <= 232448, "exceeds the per-CTA shared memory limit");
};

struct BwdWork {
  int batch;      // TMA batch coordinate
  int kv_head;
  int kvblk;      // 128-key block inside the sequence
  int q_row0;     // global row of the sequence's first query (packed), else 0
  int k_row0;
  int seqlen_q;
  int seqlen_k;
};

__device__ __forceinline__ bool bwd_decode_work(const BwdParams& p, int idx, BwdWork& w) {
  if (p.cu_k == nullptr) {
    // CTAs are numbered in waves of up to p.wave_groups (batch, KV head) groups; inside a wave the first key
    // blocks come first (under a causal mask they see the most queries).  The CTAs that run at the
    // same time then add into the fp32 dQ accumulators of a few groups only (8 MB per group at
    // 4 heads x 4096 rows), which stay in L2 between the 32 key tiles that touch them.
    const int bh_count = p.batch * p.heads_kv;
    const int nkvblk = (p.seqlen_k + kKvTile - 1) / kKvTile;
    // equal waves (a short last wave leaves SMs idle at the end)
    const int num_waves = (bh_count + p.wave_groups - 1) / p.wave_groups;
    const int wave_groups = (bh_count + num_waves - 1) / num_waves;
    const int wave = idx / (wave_groups * nkvblk);
    const int first_group = wave * wave_groups;
    const int groups_here = min(wave_groups, bh_count - first_group);
    const int r = idx - wave * wave_groups * nkvblk;
    w.kvblk = r / groups_here;
    const int bh = first_group + r % groups_here;
    w.batch = bh / p.heads_kv;
    w.kv_head = bh % p.heads_kv;
    w.q_row0 = 0;
    w.k_row0 = 0;
    w.seqlen_q = p.seqlen_q;
    w.seqlen_k = p.seqlen_k;
    return true;
  }
  // Packed: sequence by sequence, every key block for all KV heads in turn, or for p.wave_groups of them at a time.
  const int num_waves = (p.heads_kv + p.wave_groups - 1) / p.wave_groups;
  const int wave_groups = (p.heads_kv + num_waves - 1) / num_waves;
  const int wave = idx / (wave_groups * p.num_kvblk);
  const int first_head = wave * wave_groups;
  const int heads_here = min(wave_groups, p.heads_kv - first_head);
  const int r = idx - wave * wave_groups * p.num_kvblk;
  const int slot = r / heads_here;
  w.kv_head = first_head + r % heads_here;
  w.batch = 0;
  // Which sequence owns key block `slot`: every warp scans the lengths 32 sequences at a time (one
  // coalesced load, a prefix sum of the block counts, a vote) instead of walking them one by one.
  const int lane = threadIdx.x & 31;
  int first = 0;
  for (int base = 0; base < p.num_seqs; base += 32) {
    const int s = base + lane;
    int a = 0, e = 0;
    if (s < p.num_seqs) {
      a = p.cu_k[s];
      e = p.cu_k[s + 1];
    }
    const int nblk = (e - a + kKvTile - 1) / kKvTile;
    int incl = nblk;
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
      const int t = __shfl_up_sync(0xffffffffu, incl, off);
      if (lane >= off) incl += t;
    }
    const int excl = first + incl - nblk;
    const unsigned hit = __ballot_sync(0xffffffffu, slot >= excl && slot < excl + nblk);
    if (hit != 0u) {
      const int src = __ffs(hit) - 1;
      w.kvblk = slot - __shfl_sync(0xffffffffu, excl, src);
      w.k_row0 = __shfl_sync(0xffffffffu, a, src);
      w.seqlen_k = __shfl_sync(0xffffffffu, e, src) - w.k_row0;
      w.q_row0 = p.cu_q[base + src];
      w.seqlen_q = p.cu_q[base + src + 1] - w.q_row0;
      return true;
    }
    first += __shfl_sync(0xffffffffu, incl, 31);
  }
  return false;
}

// Where the per-query values (-lse * log2(e), -delta) of query row r of a tile stand: a compute thread reads columns
// 8 k + 2 t + {0, 1} for its t = lane % 4, two k to a 16-byte load.
__device__ __forceinline__ int stat_slot(int r) {
  const int k = r >> 3, t = (r >> 1) & 3;
  return ((k >> 1) * 4 + t) * 4 + (k & 1) * 2 + (r & 1);
}

// fp32 add-reduction of one swizzled shared-memory box into a 4-D tensor (TMA).
__device__ __forceinline__ void tma_reduce_add_4d(const CUtensorMap* map, uint32_t src_smem, int c0, int c1,
                                                  int c2, int c3) {
  asm volatile(
      "cp.reduce.async.bulk.tensor.4d.global.shared::cta.add.tile.bulk_group [%0, {%2, %3, %4, %5}], [%1];"
      ::"l"(reinterpret_cast<uint64_t>(map)), "r"(src_smem), "r"(c0), "r"(c1), "r"(c2), "r"(c3)
      : "memory");
}

__device__ __forceinline__ void red_add_v4(float* dst, const uint32_t (&v)[4]) {
  asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(dst), "f"(__uint_as_float(v[0])),
               "f"(__uint_as_float(v[1])), "f"(__uint_as_float(v[2])), "f"(__uint_as_float(v[3]))
               : "memory");
}

// Adds 16 rows of a dQ tile to the accumulator rows at `rows` (row_floats apart; the first `valid` of them).
// r[c][4 k + 0, 1]: columns 64 c + 8 k + 2 (lane % 4) + {0, 1} of row lane / 4; r[c][4 k + 2, 3]: of row
// lane / 4 + 8.  Lane pairs trade registers so that an instruction covers 64 contiguous bytes of each of 8 rows.
template <int D>
__device__ __forceinline__ void dq_reduce(float* rows, int row_floats, const uint32_t (&r)[D / 64][32], int valid) {
  const int lane = threadIdx.x & 31;
  const bool odd = (lane & 1) != 0;
  // four columns of one row per lane: lane pairs trade halves of two neighbouring 8-column blocks
  auto four_columns = [&](int c, int k, int h, uint32_t (&v)[4]) {
    const uint32_t a0 = r[c][4 * k + 2 * h], a1 = r[c][4 * k + 2 * h + 1];
    const uint32_t b0 = r[c][4 * k + 4 + 2 * h], b1 = r[c][4 * k + 4 + 2 * h + 1];
    const uint32_t x0 = __shfl_xor_sync(0xffffffffu, odd ? a0 : b0, 1);
    const uint32_t x1 = __shfl_xor_sync(0xffffffffu, odd ? a1 : b1, 1);
    v[0] = odd ? x0 : a0;
    v[1] = odd ? x1 : a1;
    v[2] = odd ? b0 : x0;
    v[3] = odd ? b1 : x1;
  };
  const int col = (odd ? 8 : 0) + ((lane & 2) << 1);
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    const int row = h * 8 + (lane >> 2);
#pragma unroll
    for (int c = 0; c < D / 64; ++c)
#pragma unroll
      for (int k = 0; k < 8; k += 2) {
        uint32_t v[4];
        four_columns(c, k, h, v);
        if (row < valid) red_add_v4(rows + row * row_floats + c * 64 + k * 8 + col, v);
      }
  }
}

// One swizzled shared-memory box into a 4-D tensor (TMA store; rows and columns past the tensor's
// extent are dropped).
__device__ __forceinline__ void tma_store_4d(const CUtensorMap* map, uint32_t src_smem, int c0, int c1, int c2,
                                             int c3) {
  asm volatile(
      "cp.async.bulk.tensor.4d.global.shared::cta.tile.bulk_group [%0, {%2, %3, %4, %5}], [%1];"
      ::"l"(reinterpret_cast<uint64_t>(map)), "r"(src_smem), "r"(c0), "r"(c1), "r"(c2), "r"(c3)
      : "memory");
}

__device__ __forceinline__ void named_barrier_sync(int id, int threads) {
  asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(threads) : "memory");
}

template <int D, bool CAUSAL, bool SPLIT>
__global__ void __launch_bounds__(kBwdThreads, 1)
fal_bwd_kernel(const __grid_constant__ CUtensorMap tm_q, const __grid_constant__ CUtensorMap tm_k,
               const __grid_constant__ CUtensorMap tm_v, const __grid_constant__ CUtensorMap tm_do,
               const __grid_constant__ CUtensorMap tm_dq, const __grid_constant__ CUtensorMap tm_dk,
               const __grid_constant__ CUtensorMap tm_dv, const BwdParams p) {
  using L = std::conditional_t<SPLIT, BwdSplitSmem, BwdSmem<D>>;
  constexpr int NS = L::kQStages, ND = L::kDoStages, NB = L::kSBuffers;
  // SPLIT: head_dim is 2 * D; CTAs 2n and 2n+1 share key tile n and own columns [0, D) and [D, 2D).
  const int col_own = SPLIT ? static_cast<int>(blockIdx.x & 1) * D : 0;
  const int col_other = SPLIT ? D - col_own : 0;

  extern __shared__ __align__(1024) uint8_t smem_raw[];
  const uint32_t sbase = smem_u32(smem_raw);
  uint8_t* sgen = smem_raw;
  if ((sbase & 1023u) != 0) {  // the 128-byte swizzle needs 1024-byte aligned tiles
    grid_dependency_wait();
    if (threadIdx.x == 0 && p.status) atomicCAS(p.status, 0, kDevWaitTimeout + 999);
    return;
  }
  const uint32_t bar0 = sbase + L::kBarOff;
  auto bar = [&](int i) { return bar0 + 8u * i; };
  constexpr int iKFull = 0, iVFull = 1, iQFull = 2, iQEmpty = iQFull + NS, iStatFull = iQEmpty + NS,
                iDoFull = iStatFull + NS, iDoEmpty = iDoFull + ND, iSReady = iDoEmpty + ND, iPReady = iSReady + NB,
                iDpReady = iPReady + NB, iDqReady = iDpReady + 1, iDqFree = iDpReady + 2, iDsReady = iDpReady + 3,
                iAllDone = iDpReady + 4, iDsFree = iDpReady + 5, iAFull = iDpReady + 6, iADone = iDpReady + 7,
                iBFull = iDpReady + 8;
  static_assert(iBFull + 1 == L::kNumBars, "barrier count");
  volatile uint32_t* tmem_slot = reinterpret_cast<volatile uint32_t*>(sgen + L::kMiscOff);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(sgen + L::kMiscOff + 4);
  const WaitCtx wctx{abort_flag, p.status};

  const int warp = warp_index();
  const int lane = threadIdx.x & 31;

  if (warp == 8 && elect_one()) {
    *abort_flag = 0;
    mbar_init(bar(iKFull), 1);
    mbar_init(bar(iVFull), 1);
    for (int s = 0; s < NS; ++s) {
      mbar_init(bar(iQFull + s), 1);
      mbar_init(bar(iQEmpty + s), 1);
      mbar_init(bar(iStatFull + s), 32);
    }
    for (int s = 0; s < ND; ++s) {
      mbar_init(bar(iDoFull + s), 1);
      mbar_init(bar(iDoEmpty + s), 1);
    }
    for (int s = 0; s < NB; ++s) {
      mbar_init(bar(iSReady + s), 1);
      mbar_init(bar(iPReady + s), 8);
    }
    mbar_init(bar(iDpReady), 1);
    mbar_init(bar(iDqReady), 1);
    mbar_init(bar(iDqFree), 128);
    mbar_init(bar(iDsReady), 8);
    mbar_init(bar(iAllDone), 1);
    mbar_init(bar(iDsFree), 1);
    mbar_init(bar(iAFull), 1);
    mbar_init(bar(iADone), 1);
    mbar_init(bar(iBFull), 1);
    fence_mbar_init();
    if (L::kEarlyLoads) {
      tma_prefetch_desc(&tm_k);
      tma_prefetch_desc(&tm_q);
      tma_prefetch_desc(&tm_v);
      tma_prefetch_desc(&tm_do);
    }
  }
  grid_dependency_wait();  // (up to here the pre-pass may still run)
  BwdWork wk;
  if (!bwd_decode_work(p, SPLIT ? static_cast<int>(blockIdx.x >> 1) : static_cast<int>(blockIdx.x), wk)) return;

  const int group = p.heads_q / p.heads_kv;
  const int kv0 = wk.kvblk * kKvTile;                       // local index of the tile's first key
  const int nqt = (wk.seqlen_q + kQTile - 1) / kQTile;
  // Keys the causal diagonal is moved by: query i sees keys <= i + cshift (0 = the reference's
  // top-left-aligned mask; seqlen_k - seqlen_q aligns it to the end of the keys).
  const int cshift = !CAUSAL ? 0
                     : (p.cu_k != nullptr ? (p.shift_per_sequence ? wk.seqlen_k - wk.seqlen_q : 0) : p.causal_shift);
  const int qt0 = CAUSAL ? min(max(kv0 - cshift, 0) / kQTile, nqt) : 0;  // first query tile that sees this key tile
  const int nq = nqt - qt0;                                  // query tiles per head
  const int n_iter = group * nq;

  // At head_dim 64 the first tiles are on their way before the TMEM allocation and the CTA-wide sync (a microsecond of
  // the 13 that a CTA of five pairs takes): us, 32 x 16 x 577 261 -> 257, 128 x 16 x 128 causal 142 -> 138, 4 x 16 x 2 048
  // causal 145 -> 143.  At head_dim 128 the same gave 16 x 16 x 577 196 -> 194 but 4 x 32 / 8 x 4 096 causal 1 355 -> 1 380.
  auto load_tile = [&](uint32_t dst, const CUtensorMap* map, int b, int row, int head) {
    mbar_arrive_expect_tx(bar(b), L::kTileBytes);
    for (int bx = 0; bx < L::kBoxes; ++bx)
      tma_load_4d(sbase + dst + bx * L::kBoxBytes, map, bar(b), bx * 64, row, head, wk.batch);
  };
  if (L::kEarlyLoads && warp == 8 && n_iter > 0 && elect_one()) {
    load_tile(L::kKOff, &tm_k, iKFull, wk.k_row0 + kv0, wk.kv_head);
    load_tile(L::kQOff, &tm_q, iQFull, wk.q_row0 + qt0 * kQTile, wk.kv_head * group);
    load_tile(L::kVOff, &tm_v, iVFull, wk.k_row0 + kv0, wk.kv_head);
    load_tile(L::kDoOff, &tm_do, iDoFull, wk.q_row0 + qt0 * kQTile, wk.kv_head * group);
  }
  if (warp == 9) {
    tmem_alloc(smem_u32(const_cast<uint32_t*>(tmem_slot)), 512);
    tmem_relinquish();
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem_base = *tmem_slot;
  constexpr uint32_t kColS = 0, kColDpq = 128, kColDv = 256, kColDk = 256 + D;
  constexpr uint32_t kColS1 = NB == 2 ? kColDk + D : kColS;  // S^T / P^T of odd steps
  static_assert(NB == 1 || kColS1 + 128 <= 512, "TMEM columns");

  if (warp == 8) {
    // ===================== producer: TMA ======================================
    if constexpr (SPLIT) {
      if (n_iter > 0 && elect_one()) {
        tma_prefetch_desc(&tm_q);
        tma_prefetch_desc(&tm_k);
        tma_prefetch_desc(&tm_v);
        tma_prefetch_desc(&tm_do);
        tma_prefetch_desc(&tm_dq);
        auto load_half = [&](uint32_t dst, const CUtensorMap* map, int b, int col, int row, int head) {
          for (int bx = 0; bx < L::kBoxes; ++bx)
            tma_load_4d(dst + bx * L::kBoxBytes, map, bar(b), col + bx * 64, row, head, wk.batch);
        };
        const int krow = wk.k_row0 + kv0;
        const uint32_t x_s = sbase + L::kDsOff;
        for (int i = 0; i < n_iter; ++i) {
          const int head = wk.kv_head * group + i / nq;
          const int row = wk.q_row0 + (qt0 + i % nq) * kQTile;
          // own dO: free once dV of the previous step has read it
          if (i >= 1) mbar_wait(bar(iDoEmpty), (i - 1) & 1, wctx, kBbDoEmpty);
          if (i >= 1) {
            mbar_arrive_expect_tx(bar(iDoFull), L::kTileBytes);
            load_half(sbase + L::kDoOff, &tm_do, iDoFull, col_own, row, head);
          }
          // X and own Q: free once the dQ tile of the previous step has left them
          if (i >= 1) mbar_wait(bar(iQEmpty), (i - 1) & 1, wctx, kBbQEmpty);
          mbar_arrive_expect_tx(bar(iAFull), L::kTileBytes);
          load_half(x_s, &tm_q, iAFull, col_other, row, head);
          if (i == 0) {
            mbar_arrive_expect_tx(bar(iKFull), 2 * L::kTileBytes);
            load_half(sbase + L::kKOff + L::kTileBytes, &tm_k, iKFull, col_other, krow, wk.kv_head);
            load_half(sbase + L::kKOff, &tm_k, iKFull, col_own, krow, wk.kv_head);
          }
          mbar_arrive_expect_tx(bar(iQFull), L::kTileBytes);
          load_half(sbase + L::kQOff, &tm_q, iQFull, col_own, row, head);
          if (i == 0) {
            mbar_arrive_expect_tx(bar(iVFull), 2 * L::kTileBytes);
            load_half(sbase + L::kVOff + L::kTileBytes, &tm_v, iVFull, col_other, krow, wk.kv_head);
            load_half(sbase + L::kVOff, &tm_v, iVFull, col_own, krow, wk.kv_head);
            mbar_arrive_expect_tx(bar(iDoFull), L::kTileBytes);
            load_half(sbase + L::kDoOff, &tm_do, iDoFull, col_own, row, head);
          }
          // the other half of dO follows Q's through X as soon as S^T has read that
          mbar_wait(bar(iADone), i & 1, wctx, kBbADone);
          mbar_arrive_expect_tx(bar(iBFull), L::kTileBytes);
          load_half(x_s, &tm_do, iBFull, col_other, row, head);
        }
      }
      __syncwarp();
    } else {
      if (n_iter > 0 && elect_one()) {
        if (!L::kEarlyLoads) {
          tma_prefetch_desc(&tm_q);
          tma_prefetch_desc(&tm_k);
          tma_prefetch_desc(&tm_v);
          tma_prefetch_desc(&tm_do);
          load_tile(L::kKOff, &tm_k, iKFull, wk.k_row0 + kv0, wk.kv_head);
          load_tile(L::kVOff, &tm_v, iVFull, wk.k_row0 + kv0, wk.kv_head);
        }
        tma_prefetch_desc(&tm_dq);
        for (int i = L::kEarlyLoads ? 1 : 0; i < n_iter; ++i) {
          // (where the tiles are is worked out before the wait for their buffer)
          const int st = i % NS, sd = i % ND;
          const int head = wk.kv_head * group + i / nq;
          const int row = wk.q_row0 + (qt0 + i % nq) * kQTile;
          if (i >= NS) mbar_wait(bar(iQEmpty + st), ((i / NS) - 1) & 1, wctx, kBbQEmpty + st);
          load_tile(L::kQOff + st * L::kTileBytes, &tm_q, iQFull + st, row, head);
          // a dO buffer is reloaded as soon as dV of its last step has read it
          if (i >= ND) mbar_wait(bar(iDoEmpty + sd), ((i / ND) - 1) & 1, wctx, kBbDoEmpty);
          load_tile(L::kDoOff + sd * L::kTileBytes, &tm_do, iDoFull + sd, row, head);
        }
      }
      __syncwarp();
    }
  } else if (warp == 14) {
    // ===================== per-row statistics: lse * log2(e) and delta ========
    // A tile's values are fetched, all at once, while the tile before is worked on.  Fetched row by row when their
    // buffer came free, they were what every step waited for at head_dim 128 (1 000 to 1 500 of 4 600 cycles; now the
    // loads of Q behind the dQ reductions set the pace there, 1 382 -> 1 362 us on 4 x 32 / 8 x 4 096 causal; at head_dim
    // 64 16 x 16 384 causal 1 660 -> 1 530).
    float lse[kQTile / 32], delta[kQTile / 32];
    int fetched = 0;
    auto fetch = [&](int i) {
      const int head = wk.kv_head * group + i / nq;
      fetched = (qt0 + i % nq) * kQTile;
      const float* lse_head = p.lse + wk.batch * p.lse_strides.batch + head * p.lse_strides.head;
      const float* delta_head = p.delta + wk.batch * p.delta_batch_stride + head * p.delta_head_stride;
#pragma unroll
      for (int rr = 0; rr < kQTile / 32; ++rr) {
        const int64_t row = static_cast<int64_t>(wk.q_row0) + min(fetched + lane + rr * 32, wk.seqlen_q - 1);
        lse[rr] = lse_head[row * p.lse_strides.row];
        delta[rr] = delta_head[row];
      }
    };
    if (n_iter > 0) fetch(0);
    for (int i = 0; i < n_iter; ++i) {
      const int st = i % NS;
      if (i >= NS) mbar_wait(bar(iQEmpty + st), ((i / NS) - 1) & 1, wctx, kBbQEmpty + st);
      float* stat = reinterpret_cast<float*>(sgen + L::kStatOff) + st * 2 * kQTile;
#pragma unroll
      for (int rr = 0; rr < kQTile / 32; ++rr) {
        const int r = lane + rr * 32;
        const bool row_ok = fetched + r < wk.seqlen_q;
        // exp2(x - inf) = 0: rows past the sequence, and rows that see no key, contribute nothing
        stat[stat_slot(r)] = row_ok && lse[rr] > -INFINITY ? -lse[rr] * kLog2e : -INFINITY;
        stat[kQTile + stat_slot(r)] = row_ok ? -delta[rr] : 0.f;
      }
      mbar_arrive(bar(iStatFull + st));
      if (i + 1 < n_iter) fetch(i + 1);
    }
  } else if (warp == 9) {
    // ===================== MMA issuer =========================================
    if (n_iter > 0 && elect_one()) {
      constexpr uint32_t idesc_st = make_idesc_f16(kKvTile, kQTile, 0, 0);   // S^T, dP^T
      constexpr uint32_t idesc_dkv = make_idesc_f16(kKvTile, D, 0, 1);       // dV, dK
      constexpr uint32_t idesc_dq = make_idesc_f16(kQTile, D, 1, 1);         // dQ = dS K (queries on lanes)
      const uint32_t k_s = sbase + L::kKOff, v_s = sbase + L::kVOff, ds_s = sbase + L::kDsOff;
      // Descriptors are stepped with 32-bit adds on their low words (address field = addr >> 4).
      constexpr uint32_t kHi = smem_desc_hi_sw128(1024);
      const uint32_t k_lo_k = smem_desc_lo(k_s, 16);                // K as K-major A of S^T
      const uint32_t v_lo_k = smem_desc_lo(v_s, 16);                // V as K-major A of dP^T
      const uint32_t k_lo_mn = smem_desc_lo(k_s, L::kBoxBytes);     // K^T, MN-major A of dQ^T
      const uint32_t ds_lo_k = smem_desc_lo(ds_s, 16);              // dS^T, K-major A of dK
      const uint32_t ds_lo_mn = smem_desc_lo(ds_s, L::kBoxBytes);   // dS^T, MN-major B of dQ^T

      // acc[128 keys x 128 queries] = X[keys x D] * Y[queries x D]^T, both head_dim-contiguous
      auto issue_xyT = [&](uint32_t d_col, uint32_t x_lo, uint32_t y_s, bool accumulate = false) {
        const uint32_t y_lo = smem_desc_lo(y_s, 16);
#pragma unroll
        for (int ks = 0; ks < D / 16; ++ks) {
          const uint32_t off = ((ks >> 2) * L::kBoxBytes + (ks & 3) * 32) >> 4;
          umma_ss(tmem_base + d_col, smem_desc_join(x_lo + off, kHi), smem_desc_join(y_lo + off, kHi),
                  idesc_st, (accumulate || ks > 0) ? 1u : 0u);
        }
      };

      if constexpr (!SPLIT) {
        mbar_wait(bar(iKFull), 0, wctx, kBbKFull);
        mbar_wait(bar(iQFull + 0), 0, wctx, kBbQFull);
        tc_fence_after_sync();
        issue_xyT(kColS, k_lo_k, sbase + L::kQOff);
        tc_commit(bar(iSReady));
        mbar_wait(bar(iVFull), 0, wctx, kBbVFull);
        mbar_wait(bar(iDoFull), 0, wctx, kBbDoFull);
        tc_fence_after_sync();
        issue_xyT(kColDpq, v_lo_k, sbase + L::kDoOff);
        tc_commit(bar(iDpReady));
      }

      for (int i = 0; i < n_iter; ++i) {
        const int st = i % NS;
        const int st1 = (i + 1) % NS;
        const uint32_t col_s = (NB == 2 && (i & 1) != 0) ? kColS1 : kColS;
        const uint32_t do_lo_mn = smem_desc_lo(sbase + L::kDoOff + (i % ND) * L::kTileBytes, L::kBoxBytes);
        // S^T(i+1) overwrites P^T(i+1-NB): issued behind dV(i+1-NB), which reads it.
        auto next_scores = [&]() {
          mbar_wait(bar(iQFull + st1), ((i + 1) / NS) & 1, wctx, kBbQFull + st1);
          tc_fence_after_sync();
          issue_xyT(NB == 2 ? kColS + kColS1 - col_s : kColS, k_lo_k, sbase + L::kQOff + st1 * L::kTileBytes);
          tc_commit(bar(iSReady + (i + 1) % NB));
        };
        if (NB == 2 && i + 1 < n_iter) next_scores();
        const uint32_t q_lo_mn = smem_desc_lo(sbase + L::kQOff + st * L::kTileBytes, L::kBoxBytes);
        if constexpr (SPLIT) {
          // S^T(i) and dP^T(i) in two parts, the other column half (from X) first.  S^T goes over P^T(i-1),
          // which dV(i-1) -- issued before -- has read; dP^T goes over dQ(i-1), which the write-back warps
          // must have read out.
          const uint32_t k_lo_other = smem_desc_lo(k_s + L::kTileBytes, 16);
          const uint32_t v_lo_other = smem_desc_lo(v_s + L::kTileBytes, 16);
          if (i == 0) mbar_wait(bar(iKFull), 0, wctx, kBbKFull);
          mbar_wait(bar(iAFull), i & 1, wctx, kBbAFull);
          tc_fence_after_sync();
          issue_xyT(kColS, k_lo_other, sbase + L::kDsOff);
          tc_commit(bar(iADone));
          mbar_wait(bar(iQFull), i & 1, wctx, kBbQFull);
          tc_fence_after_sync();
          issue_xyT(kColS, k_lo_k, sbase + L::kQOff, true);
          tc_commit(bar(iSReady));
          if (i == 0) mbar_wait(bar(iVFull), 0, wctx, kBbVFull);
          else mbar_wait(bar(iDqFree), (i - 1) & 1, wctx, kBbDqFree);
          mbar_wait(bar(iBFull), i & 1, wctx, kBbBFull);
          tc_fence_after_sync();
          issue_xyT(kColDpq, v_lo_other, sbase + L::kDsOff);
          mbar_wait(bar(iDoFull), i & 1, wctx, kBbDoFull);
          tc_fence_after_sync();
          issue_xyT(kColDpq, v_lo_k, sbase + L::kDoOff, true);
          tc_commit(bar(iDpReady));
        }
        // dV += P^T(i) dO(i): P^T as packed fp16 in TMEM; query columns [0,64) at +0, [64,128) at +64
        mbar_wait(bar(iPReady + i % NB), (i / NB) & 1, wctx, kBbPReady);
        tc_fence_after_sync();
#pragma unroll
        for (int ks = 0; ks < kQTile / 16; ++ks) {
          const uint32_t a_col = col_s + (ks >> 2) * 64 + (ks & 3) * 8;
          umma_ts(tmem_base + kColDv, tmem_base + a_col,
                  smem_desc_join(do_lo_mn + ((ks * 2048) >> 4), kHi), idesc_dkv,
                  (i > 0 || ks > 0) ? 1u : 0u);
        }
        tc_commit(bar(iDoEmpty + i % ND));  // dO(i) has no reader left once dV(i) is done
        if (!SPLIT && NB == 1 && i + 1 < n_iter) next_scores();
        mbar_wait(bar(iDsReady), i & 1, wctx, kBbDsReady);
        tc_fence_after_sync();
        // dK += dS^T(i) Q(i)
        auto issue_dk = [&]() {
#pragma unroll
          for (int ks = 0; ks < kQTile / 16; ++ks) {
            const uint32_t a_off = ((ks >> 2) * L::kBoxBytes + (ks & 3) * 32) >> 4;
            umma_ss(tmem_base + kColDk, smem_desc_join(ds_lo_k + a_off, kHi),
                    smem_desc_join(q_lo_mn + ((ks * 2048) >> 4), kHi), idesc_dkv,
                    (i > 0 || ks > 0) ? 1u : 0u);
          }
          // Q(i) has no reader left once dK(i) is done.  (SPLIT: nor has X, which holds dS^T(i): a commit
          // covers everything issued before it, so dQ(i), its other reader, must have been.)
          tc_commit(bar(iQEmpty + st));
        };
        // dQ(i) = dS(i) K: the dS^T buffer read as an M-contiguous A operand; the result (queries on
        // the lanes, head_dim on the columns) goes into the columns of the consumed dP^T(i)
        auto issue_dq = [&]() {
#pragma unroll
          for (int ks = 0; ks < kKvTile / 16; ++ks) {
            umma_ss(tmem_base + kColDpq, smem_desc_join(ds_lo_mn + ((ks * 2048) >> 4), kHi),
                    smem_desc_join(k_lo_mn + ((ks * 2048) >> 4), kHi), idesc_dq, ks > 0 ? 1u : 0u);
          }
          tc_commit(bar(iDqReady));
        };
        // dQ first: the write-back warps drain it out of TMEM -- which the next step's dP^T needs gone --
        // while dK still runs; and see the commit in issue_dk.
        issue_dq();
        issue_dk();
        tc_commit(bar(iDsFree));  // both readers of the dS^T buffer are done
        // dP^T(i+1) goes where dQ(i) is: the write-back warps must have read it out first.
        if (!SPLIT && i + 1 < n_iter) {
          const int sd1 = (i + 1) % ND;
          mbar_wait(bar(iDoFull + sd1), ((i + 1) / ND) & 1, wctx, kBbDoFull);
          mbar_wait(bar(iDqFree), i & 1, wctx, kBbDqFree);
          tc_fence_after_sync();
          issue_xyT(kColDpq, v_lo_k, sbase + L::kDoOff + sd1 * L::kTileBytes);
          tc_commit(bar(iDpReady));
        }
      }
      tc_commit(bar(iAllDone));
    }
    __syncwarp();
  } else if (warp < 8) {
    // ===================== compute ============================================
    const int quarter = warp & 3;
    const int half = warp >> 2;                       // query columns [64*half, 64*half+64)
    const int kv_row = quarter * 32 + lane;           // key row of the epilogue (= TMEM lane)
    const int kv_local = kv0 + kv_row;
    const bool kv_ok = kv_local < wk.seqlen_k;
    const uint32_t lane_addr = static_cast<uint32_t>(quarter * 32) << 16;
    const uint64_t c2p = pack_f32x2(p.scale_log2, p.scale_log2);
    // What a compute thread needs of the queries are two numbers per column it holds.  With a key row of 64 columns to a
    // thread those were 32 broadcast loads of 16 bytes a step, as many wavefronts of the shared-memory pipe -- the unit
    // that bounds head_dim 128 -- as storing dS^T and staging dQ take together.  With 16 columns of four rows they are 8, and
    // neighbouring columns sit in one register pair for the two-float instructions.  us on the GPU: 4 x 32 / 8 x 4 096 of
    // 128 causal 1 401 -> 1 382, 4 x 16 x 2 048 of 64 causal 191 -> 185; with the statistics fetched ahead (warp 14) 1 362
    // and 153.
    // In the main loop a thread holds columns 8 k + 2 (lane % 4) + {0, 1} of the four key rows lane / 4 + 8 g of
    // the warp's 32: register [g / 2][4 k + 2 (g % 2) + {0, 1}].
    const int frag_row = quarter * 32 + (lane >> 2);
    const int frag_col = half * 64 + 2 * (lane & 3);
    // this lane's row of the dS^T matrices it names to stmatrix: row lane % 8 of key rows 8 (lane / 8 % 2), 16-byte
    // chunk lane / 16 (+ k), 128-byte XOR swizzle
    const int ds_row = quarter * 32 + (lane & 15);
    const uint32_t ds_base = sbase + L::kDsOff + half * L::kBoxBytes + ds_row * 128;
    const uint32_t ds_chunk = static_cast<uint32_t>((lane >> 4) ^ (lane & 7)) << 4;

    for (int i = 0; i < n_iter; ++i) {
      const int st = i % NS;
      const int qt = qt0 + i % nq;
      // per-query values of this thread's columns: 4 (of columns 8 k and 8 k + 8) to a 16-byte load
      const float4* stat = reinterpret_cast<const float4*>(sgen + L::kStatOff) + st * (2 * kQTile / 4) + half * 16 + (lane & 3);
      const uint32_t t_s = tmem_base + lane_addr + ((NB == 2 && (i & 1) != 0) ? kColS1 : kColS) + half * 64;
      const bool tile_mask = kv0 + kKvTile > wk.seqlen_k || (CAUSAL && (kv0 + kKvTile - 1 > qt * kQTile + cshift));

      mbar_wait(bar(iStatFull + st), (i / NS) & 1, wctx, kBbStatFull + st);
      mbar_wait(bar(iSReady + i % NB), (i / NB) & 1, wctx, kBbSReady);
      tc_fence_after_sync();

      // ---- P^T = exp2(S^T * c2 - lse2), kept as packed fp16 for the dS step ----
      uint32_t pk[2][16];
      {
        uint32_t r[2][32];
#pragma unroll
        for (int h = 0; h < 2; ++h)
          tmem_ld_16x256b_x8(t_s + (static_cast<uint32_t>(h * 16) << 16), r[h]);
        tmem_wait_ld();
        if (tile_mask) {  // hidden scores become -inf before the exponential (exp2(-inf) = 0)
#pragma unroll
          for (int g = 0; g < 4; ++g) {
            const int key = kv0 + frag_row + 8 * g;
            // the first of this thread's columns (less 2 (lane % 4)) that sees the key
            int first = CAUSAL ? key - cshift - (qt * kQTile + frag_col) : 0;
            if (key >= wk.seqlen_k) first = 64;
#pragma unroll
            for (int k = 0; k < 8; ++k)
#pragma unroll
              for (int e = 0; e < 2; ++e) {
                uint32_t& x = r[g >> 1][4 * k + 2 * (g & 1) + e];
                x = 8 * k + e >= first ? x : 0xff800000u;
              }
          }
        }
#pragma unroll
        for (int k = 0; k < 8; k += 2) {
          const float4 l4 = stat[(k >> 1) * 4];
          const uint64_t nl[2] = {pack_f32x2(l4.x, l4.y), pack_f32x2(l4.z, l4.w)};
#pragma unroll
          for (int g = 0; g < 4; ++g)
#pragma unroll
            for (int kk = 0; kk < 2; ++kk) {
              const uint32_t* x = &r[g >> 1][4 * (k + kk) + 2 * (g & 1)];
              float p0, p1;
              unpack_f32x2(ffma2(pack_f32x2(__uint_as_float(x[0]), __uint_as_float(x[1])), c2p, nl[kk]), p0, p1);
              pk[g >> 1][2 * (k + kk) + (g & 1)] = pack_half2(fast_exp2(p0), fast_exp2(p1));
            }
        }
        // P^T overwrites this warp's own S^T columns: 32 packed columns at [64*half, 64*half+32)
#pragma unroll
        for (int h = 0; h < 2; ++h)
          tmem_st_16x128b_x8(t_s + (static_cast<uint32_t>(h * 16) << 16), pk[h]);
        tmem_wait_st();
      }
      tc_fence_before_sync();
      __syncwarp();
      if (lane == 0) mbar_arrive(bar(iPReady + i % NB));

      // ---- dS^T = P^T o (dP^T - delta) ------------------------------------------
      mbar_wait(bar(iDpReady), i & 1, wctx, kBbDpReady);
      tc_fence_after_sync();
      {
        uint32_t r[2][32];
#pragma unroll
        for (int h = 0; h < 2; ++h)
          tmem_ld_16x256b_x8(tmem_base + lane_addr + (static_cast<uint32_t>(h * 16) << 16) + kColDpq + half * 64, r[h]);
        tmem_wait_ld();
#pragma unroll
        for (int k = 0; k < 8; k += 2) {
          // (dP - delta) in fp32 (it cancels), rounded to fp16, then one packed multiply by the
          // fp16 P: the product is the fp16 dS the GEMMs consume.
          const float4 d4 = stat[kQTile / 4 + (k >> 1) * 4];
          const uint64_t nd[2] = {pack_f32x2(d4.x, d4.y), pack_f32x2(d4.z, d4.w)};
#pragma unroll
          for (int g = 0; g < 4; ++g)
#pragma unroll
            for (int kk = 0; kk < 2; ++kk) {
              const uint32_t* x = &r[g >> 1][4 * (k + kk) + 2 * (g & 1)];
              float e0, e1;
              unpack_f32x2(fadd2(pack_f32x2(__uint_as_float(x[0]), __uint_as_float(x[1])), nd[kk]), e0, e1);
              uint32_t& ds = pk[g >> 1][2 * (k + kk) + (g & 1)];
              ds = hmul2_bits(ds, pack_half2(e0, e1));
            }
        }
      }
      if (i > 0) mbar_wait(bar(iDsFree), (i - 1) & 1, wctx, kBbDqReady);
#pragma unroll
      for (int h = 0; h < 2; ++h)
#pragma unroll
        for (int k = 0; k < 8; k += 2)
          stmatrix_x4(ds_base + h * (16 * 128) + (ds_chunk ^ (k << 4)), pk[h][2 * k], pk[h][2 * k + 1], pk[h][2 * k + 2],
                      pk[h][2 * k + 3]);
      fence_proxy_async_smem();
      tc_fence_before_sync();
      __syncwarp();
      if (lane == 0) mbar_arrive(bar(iDsReady));
    }

    // ---- epilogue: dV (warps 0-3) and dK (warps 4-7) -------------------------
    if (n_iter > 0) {
      mbar_wait(bar(iAllDone), 0, wctx, kBbAllDone);
      tc_fence_after_sync();
    }
    const bool is_dk = half == 1;
    const RowStrides& st_o = is_dk ? p.dk_strides : p.dv_strides;
    const int64_t out_off = wk.batch * st_o.batch + wk.kv_head * st_o.head +
                            (static_cast<int64_t>(wk.k_row0) + kv_local) * st_o.row + col_own;
    __half* out_row = static_cast<__half*>(is_dk ? p.dk : p.dv) + out_off;
    float* out_row32 = p.dk_f32 != nullptr ? (is_dk ? p.dk_f32 : p.dv_f32) + out_off : nullptr;
    const float mul = is_dk ? p.scale : 1.f;
    const uint32_t t_acc = tmem_base + lane_addr + (is_dk ? kColDk : kColDv);
    // Whole tiles leave through shared memory (the K buffer for dK, the V buffer for dV: every MMA that
    // read them has completed) and TMA stores: a thread owns a key row, and 32 threads storing 16
    // bytes each into 32 different rows of global memory is what takes microseconds here otherwise.
    // A packed sequence's last, partial tile keeps the row-by-row path (the rows behind it belong to
    // the next sequence, which a tile store would overwrite), and so do the fp32 partials.
    const bool by_tma = p.store_by_tma != 0 && out_row32 == nullptr &&
                        (p.cu_k == nullptr || wk.seqlen_k - kv0 >= kKvTile);
    uint8_t* stage_row = sgen + (is_dk ? L::kKOff : L::kVOff) + kv_row * 128;
#pragma unroll
    for (int c = 0; c < D / 32; ++c) {
      uint32_t r[32];
      if (n_iter > 0) {
        tmem_ld_32x32b_x32(t_acc + c * 32, r);
        tmem_wait_ld();
      } else {
#pragma unroll
        for (int j = 0; j < 32; ++j) r[j] = 0u;
      }
      if (by_tma) {
#pragma unroll
        for (int v = 0; v < 4; ++v) {
          uint4 out;
          out.x = pack_half2(__uint_as_float(r[v * 8 + 0]) * mul, __uint_as_float(r[v * 8 + 1]) * mul);
          out.y = pack_half2(__uint_as_float(r[v * 8 + 2]) * mul, __uint_as_float(r[v * 8 + 3]) * mul);
          out.z = pack_half2(__uint_as_float(r[v * 8 + 4]) * mul, __uint_as_float(r[v * 8 + 5]) * mul);
          out.w = pack_half2(__uint_as_float(r[v * 8 + 6]) * mul, __uint_as_float(r[v * 8 + 7]) * mul);
          // box c / 2, 16-byte chunk (c % 2) * 4 + v of the row, 128-byte XOR swizzle
          *reinterpret_cast<uint4*>(stage_row + (c >> 1) * L::kBoxBytes + ((((c & 1) * 4 + v) ^ (kv_row & 7)) << 4)) = out;
        }
      } else if (kv_ok && out_row32 != nullptr) {
        // unrounded partial for a caller that sums the key shard's gradient over several calls
#pragma unroll
        for (int v = 0; v < 8; ++v)
          *reinterpret_cast<float4*>(out_row32 + c * 32 + v * 4) =
              make_float4(__uint_as_float(r[v * 4 + 0]) * mul, __uint_as_float(r[v * 4 + 1]) * mul,
                          __uint_as_float(r[v * 4 + 2]) * mul, __uint_as_float(r[v * 4 + 3]) * mul);
      } else if (kv_ok) {
#pragma unroll
        for (int v = 0; v < 4; ++v) {
          if (col_own + c * 32 + v * 8 >= p.head_dim) continue;  // head_dim 32 / 96: no such column
          uint4 out;
          out.x = pack_half2(__uint_as_float(r[v * 8 + 0]) * mul, __uint_as_float(r[v * 8 + 1]) * mul);
          out.y = pack_half2(__uint_as_float(r[v * 8 + 2]) * mul, __uint_as_float(r[v * 8 + 3]) * mul);
          out.z = pack_half2(__uint_as_float(r[v * 8 + 4]) * mul, __uint_as_float(r[v * 8 + 5]) * mul);
          out.w = pack_half2(__uint_as_float(r[v * 8 + 6]) * mul, __uint_as_float(r[v * 8 + 7]) * mul);
          *reinterpret_cast<uint4*>(out_row + c * 32 + v * 8) = out;
        }
      }
    }
    if (by_tma) {  // uniform over the CTA
      fence_proxy_async_smem();
      named_barrier_sync(2 + half, 128);
      if (quarter == 0 && elect_one()) {
        const uint32_t src = sbase + (is_dk ? L::kKOff : L::kVOff);
        for (int bx = 0; bx < L::kBoxes; ++bx)
          tma_store_4d(is_dk ? &tm_dk : &tm_dv, src + bx * L::kBoxBytes, col_own + bx * 64, wk.k_row0 + kv0,
                       wk.kv_head, wk.batch);
        bulk_commit_group();
        bulk_wait_group_read<0>();  // the boxes must have been read before the CTA's shared memory goes away
      }
    }
  } else if (warp < 14) {
    // ===================== dQ write-back ======================================
    const int quarter = warp & 3;
    if constexpr (SPLIT) {
      // At head_dim 256 there is no room for staging boxes.  The tile is read in the 16-lane x 8-column shape, in
      // which four lanes hold 8 columns of a row, and added to the accumulator from registers.  (Where the
      // boxes fit, TMA reductions from shared memory are faster: 1 410 against 1 518 us at head_dim 128 on
      // 4 x 32 / 8 x 4 096 causal.)  Staging through X and the Q buffer instead, which then wait for the
      // reductions to read them, took 360 us against 327.
      for (int i = 0; i < n_iter; ++i) {
        const int head = wk.kv_head * group + i / nq;
        const int qt = qt0 + i % nq;
        mbar_wait(bar(iDqReady), i & 1, wctx, kBbDqReady);
        tc_fence_after_sync();
        float* tile = p.dq_accum + wk.batch * p.dq_accum_batch_stride + head * p.dq_accum_head_stride +
                      (static_cast<int64_t>(wk.q_row0) + qt * kQTile) * (2 * D) + col_own;
        const int rows_here = wk.seqlen_q - qt * kQTile;  // rows behind the sequence are another's, or nobody's
#pragma unroll
        for (int hr = 0; hr < 2; ++hr) {
          uint32_t r[D / 64][32];
#pragma unroll
          for (int c = 0; c < D / 64; ++c)
            tmem_ld_16x256b_x8(tmem_base + (static_cast<uint32_t>(quarter * 32 + hr * 16) << 16) + kColDpq + c * 64, r[c]);
          tmem_wait_ld();
          if (hr == 1) {  // everything is in registers: the issuer may overwrite the columns
            tc_fence_before_sync();
            mbar_arrive(bar(iDqFree));
          }
          const int row = quarter * 32 + hr * 16;
          dq_reduce<D>(tile + static_cast<int64_t>(row) * (2 * D), 2 * D, r, rows_here - row);
        }
      }
    } else if constexpr (L::kWarpDq) {
      // dQ tile: TMEM lane = query row, column = head_dim.  Every warp takes its 32 rows by itself, 32 columns at a
      // time: a row per thread into one of its two swizzled [32 rows][128 bytes] boxes, which its first lane
      // hands to the TMA unit as an fp32 reduction while the other box fills.  Three column groups are in
      // registers before the first is staged, so that the TMEM columns go back to the issuer as soon as that
      // one has left its registers to the fourth.  The four warps in step instead, 64 columns at a time through two
      // boxes of 128 rows, wrote for 4 490 of a step's 5 170 cycles, 2 290 of them waiting for the boxes to be
      // read (an SM sends out 25 bytes of reductions a clock), and the next dP^T waited 1 120 for the columns:
      // 4 x 32 / 8 x 4 096 causal 1 438 -> 1 293 us, 4 x 16 x 2 048 374 -> 317, 1 x 32 / 8 x 2 987 causal 297 -> 240.
      const uint32_t t_dq = tmem_base + (static_cast<uint32_t>(quarter * 32) << 16) + kColDpq;
      const uint32_t box_off = L::kStageOff + quarter * 2 * kDqBoxBytes;
      uint8_t* box_row = sgen + box_off + lane * 128;
      for (int i = 0; i < n_iter; ++i) {
        const int head = wk.kv_head * group + i / nq;
        const int q_row = (qt0 + i % nq) * kQTile + quarter * 32;  // local index of the warp's first query
        const int grow = wk.q_row0 + q_row;                        // its accumulator row
        mbar_wait(bar(iDqReady), i & 1, wctx, kBbDqReady);
        tc_fence_after_sync();
        if (q_row >= wk.seqlen_q) {  // no query of the sequence among the warp's rows
          mbar_arrive(bar(iDqFree));
          continue;
        }
        constexpr int kGroups = D / 32, kAhead = 3;
        static_assert(kGroups == kAhead + 1, "one column group is fetched late");
        uint32_t r[kAhead][32];
#pragma unroll
        for (int c = 0; c < kAhead; ++c) tmem_ld_32x32b_x32(t_dq + c * 32, r[c]);
        tmem_wait_ld();
#pragma unroll
        for (int c = 0; c < kGroups; ++c) {
          const uint32_t box = (c & 1) * kDqBoxBytes;
          if (elect_one()) bulk_wait_group_read<1>();  // the box's last reduction has read it
          __syncwarp();
#pragma unroll
          for (int v = 0; v < 8; ++v)
            *reinterpret_cast<uint4*>(box_row + box + ((v ^ (lane & 7)) << 4)) =
                make_uint4(r[c % kAhead][4 * v + 0], r[c % kAhead][4 * v + 1], r[c % kAhead][4 * v + 2],
                           r[c % kAhead][4 * v + 3]);
          fence_proxy_async_smem();
          __syncwarp();
          if (elect_one()) {
            tma_reduce_add_4d(&tm_dq, sbase + box_off + box, c * 32, grow, head, wk.batch);
            bulk_commit_group();
          }
          if (c == 0) {  // everything is in registers then: the issuer may overwrite the columns
            tmem_ld_32x32b_x32(t_dq + kAhead * 32, r[0]);
            tmem_wait_ld();
            tc_fence_before_sync();
            mbar_arrive(bar(iDqFree));
          }
        }
      }
      if (elect_one()) bulk_wait_group0();
    } else {
      // head_dim 64: the tile is 64 columns wide and leaves at once, a row per thread into the two swizzled
      // [128 rows][32 floats] boxes, by two reductions.  (By warps as above 235 -> 254 us on 4 x 16 x 2 048: here
      // the write-back warps are not what a step waits for, and eight small reductions take more of the TMA
      // unit's and the issue slots' time than two.)
      const int qrow = quarter * 32 + lane;
      const uint32_t lane_addr = static_cast<uint32_t>(quarter * 32) << 16;
      uint8_t* box_row = sgen + L::kStageOff + qrow * 128;
      for (int i = 0; i < n_iter; ++i) {
        const int head = wk.kv_head * group + i / nq;
        const int qt = qt0 + i % nq;
        mbar_wait(bar(iDqReady), i & 1, wctx, kBbDqReady);
        tc_fence_after_sync();
        const int grow = wk.q_row0 + qt * kQTile;  // accumulator row of the tile's first query
#pragma unroll
        for (int hf = 0; hf < D / 64; ++hf) {
          uint32_t r[2][32];
          tmem_ld_32x32b_x32(tmem_base + lane_addr + kColDpq + hf * 64, r[0]);
          tmem_ld_32x32b_x32(tmem_base + lane_addr + kColDpq + hf * 64 + 32, r[1]);
          tmem_wait_ld();
          if (hf == D / 64 - 1) {  // everything is in registers: the issuer may overwrite the columns
            tc_fence_before_sync();
            mbar_arrive(bar(iDqFree));
          }
          // Earlier reductions must be done reading the staging boxes.
          if (warp == 10 && elect_one()) bulk_wait_group_read<0>();
          named_barrier_sync(1, 128);
#pragma unroll
          for (int c = 0; c < 2; ++c)
#pragma unroll
            for (int v = 0; v < 8; ++v)
              *reinterpret_cast<uint4*>(box_row + c * L::kBoxBytes + ((v ^ (qrow & 7)) << 4)) =
                  make_uint4(r[c][4 * v + 0], r[c][4 * v + 1], r[c][4 * v + 2], r[c][4 * v + 3]);
          fence_proxy_async_smem();
          named_barrier_sync(1, 128);
          if (warp == 10 && elect_one()) {
            tma_reduce_add_4d(&tm_dq, sbase + L::kStageOff, hf * 64, grow, head, wk.batch);
            tma_reduce_add_4d(&tm_dq, sbase + L::kStageOff + L::kBoxBytes, hf * 64 + 32, grow, head, wk.batch);
            bulk_commit_group();
          }
        }
      }
      if (warp == 10 && elect_one()) bulk_wait_group0();
    }
  }

  tc_fence_before_sync();
  __syncthreads();
  if (warp == 9) {
    tc_fence_after_sync();
    tmem_dealloc(tmem_base, 512);
  }
}

// ---------------------------------------------------------------------------
// Pre-pass: delta[row] = sum_d dO*O  (precompute_D_kernel, bwd.cu:76-107 of the reference) and
// the zeroing of the fp32 dQ accumulator (dQ_fp32 = zeros at csrc/flash_attn_legacy.cpp:126).
// ---------------------------------------------------------------------------
template <int D>
__global__ void __launch_bounds__(256) fal_bwd_prep_kernel(const BwdPrepParams p) {
  grid_dependency_launch();  // the main kernel's blocks set themselves up under this grid's last ones
  constexpr int kLanesPerRow = D / 8;
  constexpr int kRowsPerBlock = 256 / kLanesPerRow;
  const int sub = threadIdx.x % kLanesPerRow;
  const int64_t row_id = static_cast<int64_t>(blockIdx.x) * kRowsPerBlock + threadIdx.x / kLanesPerRow;
  const int64_t total = static_cast<int64_t>(p.batch) * p.heads_q * p.rows;
  float acc = 0.f;
  int b = 0, h = 0, r = 0;
  const bool ok = row_id < total;
  if (ok) {
    r = static_cast<int>(row_id % p.rows);
    const int64_t bh = row_id / p.rows;
    h = static_cast<int>(bh % p.heads_q);
    b = static_cast<int>(bh / p.heads_q);
    const __half* o = static_cast<const __half*>(p.o) + b * p.o_strides.batch + h * p.o_strides.head +
                      static_cast<int64_t>(r) * p.o_strides.row + sub * 8;
    const __half* d_o = static_cast<const __half*>(p.d_o) + b * p.do_strides.batch +
                        h * p.do_strides.head + static_cast<int64_t>(r) * p.do_strides.row + sub * 8;
    uint4 ov = make_uint4(0u, 0u, 0u, 0u), dv = ov;
    if (sub * 8 < p.head_dim_real) {  // head_dim 32 / 96: the columns beyond it do not exist
      ov = *reinterpret_cast<const uint4*>(o);
      dv = *reinterpret_cast<const uint4*>(d_o);
    }
    const __half2* oh = reinterpret_cast<const __half2*>(&ov);
    const __half2* dh = reinterpret_cast<const __half2*>(&dv);
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const float2 a = __half22float2(oh[j]);
      const float2 g = __half22float2(dh[j]);
      acc = fmaf(a.x, g.x, acc);
      acc = fmaf(a.y, g.y, acc);
    }
  }
#pragma unroll
  for (int off = kLanesPerRow / 2; off > 0; off >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, off);
  if (ok && sub == 0) p.delta[b * p.delta_batch_stride + h * p.delta_head_stride + r] = acc;
  // The fp32 dQ accumulator must start at zero (the main kernel only ever adds to it): this thread
  // clears the 8 columns of the row it has just read from O and dO.  Rows between p.rows and the
  // padded row count may be added into by partial tiles but are never read, so they stay as they are.
  if (ok && p.dq_accum != nullptr) {  // (a caller-owned accumulator that is being continued is left alone)
    float4* acc_row = reinterpret_cast<float4*>(p.dq_accum + b * p.dq_accum_batch_stride +
                                                h * p.dq_accum_head_stride + static_cast<int64_t>(r) * D + sub * 8);
    acc_row[0] = make_float4(0.f, 0.f, 0.f, 0.f);
    acc_row[1] = make_float4(0.f, 0.f, 0.f, 0.f);
  }
}

// ---------------------------------------------------------------------------
// Post-pass: dQ = fp16(scale * accumulator)  (csrc/flash_attn_legacy.cpp:184 of the reference).
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(256) fal_bwd_post_kernel(const BwdPostParams p) {
  const int chunks = p.head_dim_real / 8;  // only the columns the tensors have
  const int64_t total = static_cast<int64_t>(p.batch) * p.heads_q * p.rows * chunks;
  const int64_t idx = static_cast<int64_t>(blockIdx.x) * 256 + threadIdx.x;
  if (idx >= total) return;
  const int c = static_cast<int>(idx % chunks);
  const int64_t row_id = idx / chunks;
  const int r = static_cast<int>(row_id % p.rows);
  const int64_t bh = row_id / p.rows;
  const int h = static_cast<int>(bh % p.heads_q);
  const int b = static_cast<int>(bh / p.heads_q);
  const float* src = p.dq_accum + b * p.dq_accum_batch_stride + h * p.dq_accum_head_stride +
                     static_cast<int64_t>(r) * p.head_dim + c * 8;
  const float4 x = *reinterpret_cast<const float4*>(src);
  const float4 y = *reinterpret_cast<const float4*>(src + 4);
  uint4 out;
  out.x = pack_half2(x.x * p.scale, x.y * p.scale);
  out.y = pack_half2(x.z * p.scale, x.w * p.scale);
  out.z = pack_half2(y.x * p.scale, y.y * p.scale);
  out.w = pack_half2(y.z * p.scale, y.w * p.scale);
  __half* dst = static_cast<__half*>(p.dq) + b * p.dq_strides.batch + h * p.dq_strides.head +
                static_cast<int64_t>(r) * p.dq_strides.row + c * 8;
  *reinterpret_cast<uint4*>(dst) = out;
}

template <int D, bool CAUSAL, bool SPLIT = false>
cudaError_t launch_bwd_t(const CUtensorMap& tq, const CUtensorMap& tk, const CUtensorMap& tv,
                         const CUtensorMap& tdo, const CUtensorMap& tdq, const CUtensorMap& tdk,
                         const CUtensorMap& tdv, const BwdParams& p, int grid, cudaStream_t stream) {
  auto kern = fal_bwd_kernel<D, CAUSAL, SPLIT>;
  constexpr int kSmem = SPLIT ? BwdSplitSmem::kAllocBytes : BwdSmem<D>::kAllocBytes;
  static DeviceOnce configured;
  cudaError_t e = configured.run(
      [&] { return cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmem); });
  if (e != cudaSuccess) return e;
  if (SPLIT && grid > 0x3fffffff) return cudaErrorInvalidValue;
  // Under the pre-pass's last blocks (2 x 8 x 1 024 of 64 causal 22.8 -> 22.4 us; the pre- and the post-pass started in the
  // same way made that 23.4, and 32 / 8 x 2 987 of 128 256 -> 260).
  return launch_dependent(kern, dim3(SPLIT ? 2 * grid : grid), dim3(kBwdThreads), kSmem, stream, tq, tk, tv, tdo, tdq, tdk,
                          tdv, p);
}

}  // namespace

cudaError_t launch_bwd_prep(const BwdPrepParams& p, cudaStream_t stream) {
  const int64_t total = static_cast<int64_t>(p.batch) * p.heads_q * p.rows;
  auto launch = [&](auto kern, int rows_per_block) {
    kern<<<static_cast<unsigned>((total + rows_per_block - 1) / rows_per_block), 256, 0, stream>>>(p);
    return cudaGetLastError();
  };
  if (p.head_dim == 256) return launch(fal_bwd_prep_kernel<256>, 8);
  if (p.head_dim == 128) return launch(fal_bwd_prep_kernel<128>, 16);
  if (p.head_dim == 64) return launch(fal_bwd_prep_kernel<64>, 32);
  return cudaErrorInvalidValue;
}

cudaError_t launch_bwd(int head_dim, bool causal, const CUtensorMap& tq, const CUtensorMap& tk,
                       const CUtensorMap& tv, const CUtensorMap& tdo, const CUtensorMap& tdq,
                       const CUtensorMap& tdk, const CUtensorMap& tdv, const BwdParams& p, int grid,
                       cudaStream_t stream) {
  if (head_dim == 128) {
    return causal ? launch_bwd_t<128, true>(tq, tk, tv, tdo, tdq, tdk, tdv, p, grid, stream)
                  : launch_bwd_t<128, false>(tq, tk, tv, tdo, tdq, tdk, tdv, p, grid, stream);
  }
  if (head_dim == 64) {
    return causal ? launch_bwd_t<64, true>(tq, tk, tv, tdo, tdq, tdk, tdv, p, grid, stream)
                  : launch_bwd_t<64, false>(tq, tk, tv, tdo, tdq, tdk, tdv, p, grid, stream);
  }
  if (head_dim == 256) {  // two CTAs per key tile, 128 output columns each
    return causal ? launch_bwd_t<128, true, true>(tq, tk, tv, tdo, tdq, tdk, tdv, p, grid, stream)
                  : launch_bwd_t<128, false, true>(tq, tk, tv, tdo, tdq, tdk, tdv, p, grid, stream);
  }
  return cudaErrorInvalidValue;
}

cudaError_t launch_bwd_post(const BwdPostParams& p, cudaStream_t stream) {
  const int64_t total = static_cast<int64_t>(p.batch) * p.heads_q * p.rows * (p.head_dim_real / 8);
  const int64_t blocks = (total + 255) / 256;
  fal_bwd_post_kernel<<<static_cast<unsigned>(blocks), 256, 0, stream>>>(p);
  return cudaGetLastError();
}

}  // namespace fal

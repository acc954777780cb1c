// Single-token decode against an fp16 KV cache: a split-K streaming kernel (which
// also appends the new token's K/V row) followed by a log-sum-exp combine.
//
// Stands in for the eager matmul -> softmax -> matmul fallback that the
// reference's attention hook uses whenever q_len != kv_len
// (flash_attn_legacy/integrations.py:77-98): softmax(q K^T * scale) V over the
// valid cache positions, no causal mask, GQA by head mapping instead of
// repeat_interleave.
//
// The pass is bound by HBM bandwidth (4 flops per cache byte), so the kernel is
// organised around keeping 16-byte loads in flight:
//   - grid (kv_head x head-chunk, split, batch); each CTA streams a split (256
//     to 2 048 cache positions, by the entry's length) of one KV head exactly once for all the query heads that
//     share it (up to 16 per CTA);
//   - every warp runs its own cp.async pipeline over interleaved 16-key slices
//     (no block-level barrier inside the main loop), shared memory XOR-swizzled
//     for conflict-free ldmatrix;
//   - scores and PV use mma.sync m16n8k16 with the query heads as the M rows:
//     tensor throughput is irrelevant here, the MMA only keeps the issue slots
//     free for the loads;
//   - the CTA whose split holds the position the new token goes to writes that
//     row into the cache before it starts streaming (no separate append launch);
//   - each split writes an unnormalised fp32 partial (O, max, sum); the combine
//     kernel merges the splits that the sequence length actually reaches.  (Letting
//     the last split of an entry to finish do the merge instead -- an arrival
//     counter per entry, one launch in all -- was built and measured: every CTA then
//     ends with a fence and an atomic round trip to L2, which cost more than the
//     second launch saves, 84 against 80 us per step on an 8-entry batch replayed as
//     a CUDA graph and 0.797 against 0.787 ms at batch 64.)
// An optional first position per batch entry (cache_starts) skips a padded prefix
// of the cache: the entry's row pointers start there and its length shrinks.
#include <type_traits>

#include "fal_common.h"
#include "fal_launch.h"
#include "sm100_ptx.cuh"

namespace fal {

namespace {

constexpr int kDecWarps = 4;
constexpr int kDecThreads = kDecWarps * 32;
constexpr int kSliceKeys = 16;  // keys per warp step
constexpr int kDecStages = 3;   // per-warp pipeline depth
constexpr float kNegInfD = -INFINITY;

__device__ __forceinline__ void cp_async_16_zfill(uint32_t dst, const void* src, bool valid) {
  const uint32_t n = valid ? 16u : 0u;
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(n)
               : "memory");
}
__device__ __forceinline__ void cp_async_commit() {
  asm volatile("cp.async.commit_group;" ::: "memory");
}
template <int N>
__device__ __forceinline__ void cp_async_wait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

__device__ __forceinline__ void ldmatrix_x4(uint32_t addr, uint32_t& r0, uint32_t& r1, uint32_t& r2,
                                            uint32_t& r3) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];"
               : "=r"(r0), "=r"(r1), "=r"(r2), "=r"(r3)
               : "r"(addr));
}
__device__ __forceinline__ void ldmatrix_x4_trans(uint32_t addr, uint32_t& r0, uint32_t& r1,
                                                  uint32_t& r2, uint32_t& r3) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0, %1, %2, %3}, [%4];"
               : "=r"(r0), "=r"(r1), "=r"(r2), "=r"(r3)
               : "r"(addr));
}
// D (fp32, 16x8) += A (fp16, 16x16) * B (fp16, 16x8)
__device__ __forceinline__ void mma_16816(float (&c)[4], const uint32_t (&a)[4], uint32_t b0,
                                          uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, "
      "{%8, %9}, {%0, %1, %2, %3};"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

// ---------------------------------------------------------------------------
// Append + split-K pass + merge by the last CTA to arrive.
// ---------------------------------------------------------------------------
// The keys entry b attends to: [start, start + len) of its cache, the appended token included when
// there is one and it fits.  `can_append`: a new token is given and position len_old is inside the
// cache.  A cache that is already full (or a negative length) cannot take the token: it is then
// neither stored nor attended to, and the status word says so.
struct DecodeRange {
  int len_old;
  int start;
  int len;
  bool can_append;
};
__device__ __forceinline__ DecodeRange decode_range(const DecodeParams& p, int b) {
  DecodeRange r;
  r.len_old = p.cache_seqlens[b];
  r.can_append = p.k_new != nullptr && r.len_old >= 0 && r.len_old < p.capacity;
  int len = min(max(r.len_old + (r.can_append ? 1 : 0), 0), p.capacity);
  r.start = p.cache_starts ? min(max(p.cache_starts[b], 0), len) : 0;
  r.len = len - r.start;
  return r;
}

// log2 of the positions per split of an entry of `len`: the finest cut that leaves it with no more than fine_splits.
__device__ __forceinline__ int decode_split_shift(const DecodeParams& p, int len) {
  int shift = kDecodeFinestShift;
  while (shift < p.split_shift && ((len - 1) >> shift) + 1 > p.fine_splits) ++shift;
  return shift;
}

template <int D>
struct DecSmem {
  static constexpr int kRowBytes = D * 2;
  static constexpr int kSliceBytes = kSliceKeys * kRowBytes;            // one K or V slice
  static constexpr int kStageBytes = 2 * kSliceBytes;                   // K then V
  static constexpr int kWarpBytes = kDecStages * kStageBytes;
  static constexpr int kPipeBytes = kDecWarps * kWarpBytes;
  // After the main loop the same memory holds the per-warp partials.
  static constexpr int kMergeBytes = kDecWarps * 16 * (D + 2) * 4;
  static constexpr int kBytes = kPipeBytes > kMergeBytes ? kPipeBytes : kMergeBytes;
};

template <int D>
__global__ void __launch_bounds__(kDecThreads)
fal_decode_splitk_kernel(const DecodeParams p) {
  using L = DecSmem<D>;
  constexpr int kChunks = D / 8;       // 16-byte chunks per row
  constexpr int kKSteps = D / 16;      // k-steps of the score MMA
  constexpr int kNTiles = D / 8;       // 8-wide output tiles of the PV MMA
  constexpr int kLoadsPerLane = kSliceKeys * kChunks / 32;

  extern __shared__ __align__(128) uint8_t dec_smem[];
  grid_dependency_wait();    // the kernel before this one may still run up to here
  grid_dependency_launch();  // the combine kernel may take its place on the SMs; it waits for this grid's end

  const int group = p.heads_q / p.heads_kv;          // query heads per KV head
  const int head_chunks = (group + 15) / 16;
  const int kv_head = blockIdx.x / head_chunks;
  const int head_chunk = blockIdx.x % head_chunks;
  const int split = blockIdx.y;
  const int b = blockIdx.z;

  const DecodeRange rg = decode_range(p, b);
  const int len_old = rg.len_old, start = rg.start, len = rg.len;
  const bool can_append = rg.can_append;
  if (p.k_new != nullptr && !can_append && split == 0 && blockIdx.x == 0 && threadIdx.x == 0 && p.status)
    atomicCAS(p.status, 0, kDevAppendOverflow);
  const int split_shift = decode_split_shift(p, len);
  const int pos0 = split << split_shift;

  const int rows_valid = min(16, group - head_chunk * 16);
  const int hq0 = kv_head * group + head_chunk * 16;  // first query head of this CTA

  // ---- append: the split that holds the new position stores the row (split 0 does when the position lies before
  // `start` and nobody attends to it), and streams it from where it came from: read back through L2 it would have to
  // wait for a load, a store and a fence, at the head of the one CTA that all others then wait for.  us a step on the GPU,
  // with the statistics and rows of the combine kernel fetched together: 1 entry of 1 999 positions, 32 / 8 heads of 128,
  // 9.1 -> 7.7 (without a new row 8.2 -> 6.9), 8 of 2 049, 32 / 4 of 64, 8.5 -> 7.0, 16 of 2 000 27.4 -> 26.0.
  // Only the slice that holds the row chooses between two sources.  With the choice in all of an entry's slices: 1 entry of
  // 1 999 7.6 -> 7.2, 3 of 8 000, 16 heads of 64, 22.4 -> 20.7, 4 of 3 000 of 256 29.7 -> 25.7, 32 of 1 000, 32 / 32 of 96,
  // 87 -> 79, 64 of 5 000 220 -> 207, 64 of 1 024 to 32 512 765 -> 685: what the same steps take without a new row.  (It is
  // not the compare alone: a kernel of its own for steps without a new row, which has one form of the loads, was as slow
  // again, 207 -> 217, with 167 registers instead of 224.) ----
  const int new_local = can_append ? len_old - start : -1;
  if (can_append) {
    const int store_split = new_local >= 0 ? new_local >> split_shift : 0;
    if (split == store_split) {
      const int real_chunks = p.head_dim_real / 8;  // head_dim 32 / 96 run on the 64 / 128 kernels
      for (int c = threadIdx.x; c < 2 * real_chunks; c += kDecThreads) {
        const bool is_v = c >= real_chunks;
        const int cc = is_v ? c - real_chunks : c;
        const __half* src = static_cast<const __half*>(is_v ? p.v_new : p.k_new) +
                            (static_cast<int64_t>(b) * p.heads_kv + kv_head) * p.head_dim_real + cc * 8;
        const RowStrides& st = is_v ? p.v_strides : p.k_strides;
        __half* dst = static_cast<__half*>(is_v ? p.v_cache : p.k_cache) + b * st.batch + kv_head * st.head +
                      static_cast<int64_t>(len_old) * st.row + cc * 8;
        *reinterpret_cast<uint4*>(dst) = *reinterpret_cast<const uint4*>(src);
      }
    }
  }
  if (pos0 >= len) return;  // this split lies beyond the sequence
  const int pos_end = min(pos0 + (1 << split_shift), len);
  const int num_slices = (pos_end - pos0 + kSliceKeys - 1) / kSliceKeys;

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const int g = lane >> 2;
  const int t = lane & 3;

  // ---- query fragments (A operand: row = head, col = head_dim) ---------------
  uint32_t qa[kKSteps][4];
  {
    // (columns beyond the tensors' head_dim -- 32 and 96 run on the 64 / 128 kernels -- read as zero)
    const int dr = p.head_dim_real;
    const __half* qb = static_cast<const __half*>(p.q) + (static_cast<int64_t>(b) * p.heads_q + hq0) * dr;
#pragma unroll
    for (int ks = 0; ks < kKSteps; ++ks) {
      const int col = ks * 16 + 2 * t;
      qa[ks][0] = (g < rows_valid && col < dr) ? *reinterpret_cast<const uint32_t*>(qb + g * dr + col) : 0u;
      qa[ks][1] = (g + 8 < rows_valid && col < dr) ? *reinterpret_cast<const uint32_t*>(qb + (g + 8) * dr + col) : 0u;
      qa[ks][2] = (g < rows_valid && col + 8 < dr) ? *reinterpret_cast<const uint32_t*>(qb + g * dr + col + 8) : 0u;
      qa[ks][3] = (g + 8 < rows_valid && col + 8 < dr) ? *reinterpret_cast<const uint32_t*>(qb + (g + 8) * dr + col + 8) : 0u;
    }
  }

  const __half* kbase = static_cast<const __half*>(p.k_cache) + b * p.k_strides.batch +
                        kv_head * p.k_strides.head + static_cast<int64_t>(start) * p.k_strides.row;
  const __half* vbase = static_cast<const __half*>(p.v_cache) + b * p.v_strides.batch +
                        kv_head * p.v_strides.head + static_cast<int64_t>(start) * p.v_strides.row;
  const uint32_t wbase = smem_u32(dec_smem) + warp * L::kWarpBytes;
  const int real_chunks = p.head_dim_real / 8;
  const int64_t new_row = (static_cast<int64_t>(b) * p.heads_kv + kv_head) * p.head_dim_real;

  // Issues the loads of this warp's i-th slice (keys pos0 + (i*4 + warp)*16 ...).
  auto issue_slice = [&](int i) {
    const int slice = i * kDecWarps + warp;
    if (slice < num_slices) {
      const uint32_t sb = wbase + (i % kDecStages) * L::kStageBytes;
      const int key0 = pos0 + slice * kSliceKeys;
      auto load = [&](auto with_new) {
#pragma unroll
        for (int it = 0; it < kLoadsPerLane; ++it) {
          const int idx = it * 32 + lane;
          const int row = idx / kChunks;
          const int ch = idx % kChunks;
          const int key = key0 + row;
          const bool ok = key < pos_end && ch < real_chunks;  // chunks past the tensors' head_dim fill with zeros
          const int64_t krow = static_cast<int64_t>(key < pos_end ? key : pos0);
          const int src_ch = ch < real_chunks ? ch : 0;
          const uint32_t soff = row * L::kRowBytes + ((ch ^ (row & 7)) << 4);
          const __half* ks = kbase + krow * p.k_strides.row;
          const __half* vs = vbase + krow * p.v_strides.row;
          if (decltype(with_new)::value && krow == new_local) {
            ks = static_cast<const __half*>(p.k_new) + new_row;
            vs = static_cast<const __half*>(p.v_new) + new_row;
          }
          cp_async_16_zfill(sb + soff, ks + src_ch * 8, ok);
          cp_async_16_zfill(sb + L::kSliceBytes + soff, vs + src_ch * 8, ok);
        }
      };
      if (static_cast<unsigned>(new_local - key0) >= kSliceKeys) load(std::false_type{});
      else load(std::true_type{});  // (the slice that holds the new row)
    }
    cp_async_commit();  // always commit so that group counting stays uniform
  };

  float acc_o[kNTiles][4];
#pragma unroll
  for (int n = 0; n < kNTiles; ++n)
#pragma unroll
    for (int i = 0; i < 4; ++i) acc_o[n][i] = 0.f;
  float m_run[2] = {kNegInfD, kNegInfD};  // rows g and g+8, log2 domain
  float l_run[2] = {0.f, 0.f};
  const float c2 = p.scale * 1.4426950408889634f;

  const int my_slices = (num_slices - warp + kDecWarps - 1) / kDecWarps;  // may be <= 0
#pragma unroll
  for (int i = 0; i < kDecStages - 1; ++i) issue_slice(i);

  for (int i = 0; i < my_slices; ++i) {
    issue_slice(i + kDecStages - 1);
    cp_async_wait<kDecStages - 1>();
    __syncwarp();
    const uint32_t sb = wbase + (i % kDecStages) * L::kStageBytes;
    const int key0 = pos0 + (i * kDecWarps + warp) * kSliceKeys;

    // ---- S = Q K^T (16 heads x 16 keys) ------------------------------------
    float s[2][4] = {{0.f, 0.f, 0.f, 0.f}, {0.f, 0.f, 0.f, 0.f}};
    {
      const int mi = lane >> 3;
      const int r = lane & 7;
      const int krow = (mi >> 1) * 8 + r;
#pragma unroll
      for (int ks = 0; ks < kKSteps; ++ks) {
        const int ch = 2 * ks + (mi & 1);
        uint32_t b00, b01, b10, b11;
        ldmatrix_x4(sb + krow * L::kRowBytes + ((ch ^ (krow & 7)) << 4), b00, b01, b10, b11);
        mma_16816(s[0], qa[ks], b00, b01);
        mma_16816(s[1], qa[ks], b10, b11);
      }
    }
    // ---- online softmax (log2 domain) --------------------------------------
    const bool tail = key0 + kSliceKeys > pos_end;
#pragma unroll
    for (int nt = 0; nt < 2; ++nt)
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        float v = s[nt][e] * c2;
        if (tail && (key0 + nt * 8 + 2 * t + (e & 1) >= pos_end)) v = kNegInfD;
        s[nt][e] = v;
      }
    float alpha[2];
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      float mx = fmaxf(fmaxf(s[0][2 * h], s[0][2 * h + 1]), fmaxf(s[1][2 * h], s[1][2 * h + 1]));
      mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 1));
      mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 2));
      const float m_new = fmaxf(m_run[h], mx);
      const float m_use = (m_new == kNegInfD) ? 0.f : m_new;
      alpha[h] = fast_exp2(m_run[h] - m_use);  // exp2(-inf) = 0 on the first slice
      float sum = 0.f;
#pragma unroll
      for (int nt = 0; nt < 2; ++nt) {
        const float p0 = fast_exp2(s[nt][2 * h] - m_use);
        const float p1 = fast_exp2(s[nt][2 * h + 1] - m_use);
        s[nt][2 * h] = p0;
        s[nt][2 * h + 1] = p1;
        sum += p0 + p1;
      }
      sum += __shfl_xor_sync(0xffffffffu, sum, 1);
      sum += __shfl_xor_sync(0xffffffffu, sum, 2);
      l_run[h] = l_run[h] * alpha[h] + sum;
      m_run[h] = m_new;
    }
    uint32_t pa[4];
    pa[0] = pack_half2(s[0][0], s[0][1]);
    pa[1] = pack_half2(s[0][2], s[0][3]);
    pa[2] = pack_half2(s[1][0], s[1][1]);
    pa[3] = pack_half2(s[1][2], s[1][3]);

    // ---- O = alpha * O + P V ----------------------------------------------
    {
      const int mi = lane >> 3;
      const int r = lane & 7;
      const int vrow = (mi & 1) * 8 + r;
      const uint32_t vb = sb + L::kSliceBytes + vrow * L::kRowBytes;
#pragma unroll
      for (int n = 0; n < kNTiles; n += 2) {
        const int ch = n + (mi >> 1);
        uint32_t b00, b01, b10, b11;
        ldmatrix_x4_trans(vb + ((ch ^ (vrow & 7)) << 4), b00, b01, b10, b11);
        acc_o[n][0] *= alpha[0];
        acc_o[n][1] *= alpha[0];
        acc_o[n][2] *= alpha[1];
        acc_o[n][3] *= alpha[1];
        acc_o[n + 1][0] *= alpha[0];
        acc_o[n + 1][1] *= alpha[0];
        acc_o[n + 1][2] *= alpha[1];
        acc_o[n + 1][3] *= alpha[1];
        mma_16816(acc_o[n], pa, b00, b01);
        mma_16816(acc_o[n + 1], pa, b10, b11);
      }
    }
    __syncwarp();  // all lanes are done with this stage before it is refilled
  }
  cp_async_wait<0>();
  __syncthreads();  // the pipeline memory is reused for the merge below

  // ---- merge the four warps' partials and write the split's result ----------
  float* mo = reinterpret_cast<float*>(dec_smem);               // [warp][16][D]
  float* mml = mo + kDecWarps * 16 * D;                         // [warp][16][2]
#pragma unroll
  for (int n = 0; n < kNTiles; ++n) {
    const int col = n * 8 + 2 * t;
    *reinterpret_cast<float2*>(mo + (warp * 16 + g) * D + col) = make_float2(acc_o[n][0], acc_o[n][1]);
    *reinterpret_cast<float2*>(mo + (warp * 16 + g + 8) * D + col) = make_float2(acc_o[n][2], acc_o[n][3]);
  }
  if (t == 0) {
    mml[(warp * 16 + g) * 2 + 0] = m_run[0];
    mml[(warp * 16 + g) * 2 + 1] = l_run[0];
    mml[(warp * 16 + g + 8) * 2 + 0] = m_run[1];
    mml[(warp * 16 + g + 8) * 2 + 1] = l_run[1];
  }
  __syncthreads();
  for (int idx = threadIdx.x; idx < rows_valid * D; idx += kDecThreads) {
    const int r = idx / D;
    const int c = idx % D;
    float mmax = kNegInfD;
#pragma unroll
    for (int w = 0; w < kDecWarps; ++w) mmax = fmaxf(mmax, mml[(w * 16 + r) * 2]);
    const float muse = (mmax == kNegInfD) ? 0.f : mmax;
    float o = 0.f, lsum = 0.f;
#pragma unroll
    for (int w = 0; w < kDecWarps; ++w) {
      const float sc = fast_exp2(mml[(w * 16 + r) * 2] - muse);
      o += sc * mo[(w * 16 + r) * D + c];
      lsum += sc * mml[(w * 16 + r) * 2 + 1];
    }
    const int64_t prow = (static_cast<int64_t>(b) * p.heads_q + hq0 + r) * p.splits + split;
    p.part_o[prow * D + c] = o;
    if (c == 0) {
      p.part_ml[prow * 2 + 0] = mmax;
      p.part_ml[prow * 2 + 1] = lsum;
    }
  }

}

// ---------------------------------------------------------------------------
// Combine: merge the splits a sequence actually reaches.
// ---------------------------------------------------------------------------
// WARPS warps per (batch, head), blocks of four warps.  The statistics of all splits are reduced by all lanes at
// once and the partial rows are summed by groups of D / 4 threads (16-byte loads), a split each: with one thread
// per column walking every split three times the kernel took 4.8 us at 2 splits, most of it exposed
// load latency that grows with the number of splits.
// Four warps per row where a row's partials are many, one where they are few and the rows make the grid large.
// Whole decode step, four against one, us: 64 x 32 heads of 64, 4 splits 8.7 / 7.0 (12 positions) and 50.5 / 49.5
// (4 095); 256 x 32 of 128, 1 split 36.5 / 30.0; 8 x 32 of 64, 9 splits 8.2 / 8.0; 1 x 32 of 128, 16 splits 9.1 / 10.8;
// 4 x 32 of 128, 32 splits 93.1 / 101.3; 1 x 8 of 64, 64 splits 8.8 / 13.2.
// It is launched while the split-K grid still runs and waits here for that grid's results.
constexpr int kCombineThreads = 128;
constexpr int kCombineWarpBytes = 2048;  // of partials of a row, up to which one warp merges them;
constexpr int kCombineManyRows = 256;    // twice as many in a grid of this many rows

// (m, l) <- the merge with another running maximum and sum (log2 domain).
__device__ __forceinline__ void merge_stats(float& m, float& l, float m2, float l2) {
  const float m_new = fmaxf(m, m2);
  const float m_use = (m_new == kNegInfD) ? 0.f : m_new;
  l = l * fast_exp2(m - m_use) + l2 * fast_exp2(m2 - m_use);
  m = m_new;
}

template <int D, int WARPS>
__global__ void __launch_bounds__(kCombineThreads)
fal_decode_combine_kernel(const DecodeParams p) {
  static_assert(WARPS == 1 || WARPS * 32 == kCombineThreads, "a row per warp or per block");
  constexpr int kRows = kCombineThreads / (32 * WARPS);      // (batch, head) rows per block
  constexpr int kThreads = 32 * WARPS;                       // threads per row
  constexpr int kLanes = D / 4 < kThreads ? D / 4 : kThreads;  // threads per partial row
  constexpr int kVecs = D / (4 * kLanes);                    // 16-byte pieces of it per thread
  constexpr int kGroups = kThreads / kLanes;                 // partial rows in flight
  __shared__ float2 warp_ml[WARPS];
  __shared__ float4 part[kGroups][kLanes];
  const int tid = threadIdx.x % kThreads;
  const int bh = blockIdx.x * kRows + threadIdx.x / kThreads;
  const bool row_ok = bh < p.batch * p.heads_q;
  int n = 0;
  if (row_ok) {
    const int len = decode_range(p, bh / p.heads_q).len;
    n = ((len - 1) >> decode_split_shift(p, len)) + 1;  // (an empty entry: (-1 >> shift) + 1 = 0)
  }
  const float2* ml = reinterpret_cast<const float2*>(p.part_ml) + static_cast<int64_t>(bh) * p.splits;
  const float4* po = reinterpret_cast<const float4*>(p.part_o) + static_cast<int64_t>(bh) * p.splits * (D / 4);
  // (The lengths were not written by the split-K grid, and whatever wrote them ended before that grid let this one start.)
  grid_dependency_wait();
  if (!row_ok) return;  // (whole warps; a block of one row has that row)

  // The first partial rows of this thread are fetched with the statistics, not behind them: one round trip to L2 for three.
  constexpr int kAhead = 4;
  const int lane = tid % kLanes;
  const int grp = tid / kLanes;
  float mx[kAhead];
  float4 px[kAhead][kVecs];
#pragma unroll
  for (int k = 0; k < kAhead; ++k) {
    const int i = grp + k * kGroups;
    mx[k] = kNegInfD;
#pragma unroll
    for (int v = 0; v < kVecs; ++v) px[k][v] = make_float4(0.f, 0.f, 0.f, 0.f);
    if (i < n) {
      mx[k] = ml[i].x;
#pragma unroll
      for (int v = 0; v < kVecs; ++v) px[k][v] = po[static_cast<int64_t>(i) * (D / 4) + v * kLanes + lane];
    }
  }
  float m = kNegInfD, l = 0.f;
  for (int i = tid; i < n; i += kThreads) {
    const float2 x = ml[i];
    merge_stats(m, l, x.x, x.y);
  }
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) {
    const float m2 = __shfl_xor_sync(0xffffffffu, m, off);
    const float l2 = __shfl_xor_sync(0xffffffffu, l, off);
    merge_stats(m, l, m2, l2);
  }
  if constexpr (WARPS > 1) {
    if ((tid & 31) == 0) warp_ml[tid >> 5] = make_float2(m, l);
    __syncthreads();
    m = warp_ml[0].x;
    l = warp_ml[0].y;
#pragma unroll
    for (int w = 1; w < WARPS; ++w) merge_stats(m, l, warp_ml[w].x, warp_ml[w].y);
  }
  const float muse = (m == kNegInfD) ? 0.f : m;
  const float inv = l > 0.f ? 1.f / l : 0.f;

  float4 o[kVecs];
#pragma unroll
  for (int v = 0; v < kVecs; ++v) o[v] = make_float4(0.f, 0.f, 0.f, 0.f);
  auto add_weighted = [&](float4& a, float w, const float4& x) {
    a.x += w * x.x;
    a.y += w * x.y;
    a.z += w * x.z;
    a.w += w * x.w;
  };
#pragma unroll
  for (int k = 0; k < kAhead; ++k) {
    if (grp + k * kGroups < n) {
      const float w = fast_exp2(mx[k] - muse);
#pragma unroll
      for (int v = 0; v < kVecs; ++v) add_weighted(o[v], w, px[k][v]);
    }
  }
#pragma unroll 4
  for (int i = grp + kAhead * kGroups; i < n; i += kGroups) {
    const float w = fast_exp2(ml[i].x - muse);
#pragma unroll
    for (int v = 0; v < kVecs; ++v) add_weighted(o[v], w, po[static_cast<int64_t>(i) * (D / 4) + v * kLanes + lane]);
  }
  auto add = [&](float4& a, const float4& x) {
    a.x += x.x;
    a.y += x.y;
    a.z += x.z;
    a.w += x.w;
  };
  if constexpr (WARPS > 1) {
    static_assert(kVecs == 1, "one piece per thread");
    part[grp][lane] = o[0];
    __syncthreads();
    if (grp == 0) {
#pragma unroll
      for (int g = 1; g < kGroups; ++g) add(o[0], part[g][lane]);
    }
  } else {
#pragma unroll
    for (int off = kLanes; off < 32; off <<= 1) {  // (one piece per thread then)
      const float4 x = make_float4(__shfl_xor_sync(0xffffffffu, o[0].x, off), __shfl_xor_sync(0xffffffffu, o[0].y, off),
                                   __shfl_xor_sync(0xffffffffu, o[0].z, off), __shfl_xor_sync(0xffffffffu, o[0].w, off));
      add(o[0], x);
    }
  }
  __half* out_row = static_cast<__half*>(p.o) + static_cast<int64_t>(bh) * p.head_dim_real;
#pragma unroll
  for (int v = 0; v < kVecs; ++v) {
    const int col = (v * kLanes + lane) * 4;
    if (grp == 0 && col < p.head_dim_real) {
      uint2 out;
      out.x = pack_half2(o[v].x * inv, o[v].y * inv);
      out.y = pack_half2(o[v].z * inv, o[v].w * inv);
      *reinterpret_cast<uint2*>(out_row + col) = out;
    }
  }
  if (p.lse != nullptr && tid == 0) p.lse[bh] = (l > 0.f) ? (m + log2f(l)) * 0.6931471805599453f : kNegInfD;
}

// ---------------------------------------------------------------------------
// Append of a chunk of new rows to caches filled to a different length per entry.
// ---------------------------------------------------------------------------
// Bound by HBM (each byte read once and written once); a thread moves 16 bytes.  One launch for K and V,
// the new lengths and the room check: as tensor indexing it was ten launches, whose two scatter kernels
// took 27 us each for 4 entries x 1024 rows x 8 heads x 128.
__global__ void __launch_bounds__(256) fal_cache_append_kernel(const CacheAppendParams p) {
  const int b = blockIdx.y;
  const bool is_v = blockIdx.z != 0;
  const int len = __ldg(p.cache_seqlens + b);
  if (blockIdx.x == 0 && !is_v && threadIdx.x == 0) p.new_seqlens[b] = len + p.rows;
  if (blockIdx.x == 0 && b == 0 && is_v) {  // every position of every entry must be inside the cache
    bool fits = true;
    for (int i = threadIdx.x; i < p.batch; i += 256) {
      const int64_t l = __ldg(p.cache_seqlens + i);
      fits = fits && l >= -static_cast<int64_t>(p.capacity) && l + p.rows <= p.capacity;
    }
    fits = __syncthreads_and(fits) != 0;
    if (threadIdx.x == 0) *p.fits = fits ? 1 : 0;
  }
  const int chunks = p.head_dim / 8;
  const int64_t idx = static_cast<int64_t>(blockIdx.x) * 256 + threadIdx.x;
  if (idx >= static_cast<int64_t>(p.rows) * p.heads_kv * chunks) return;
  const int c = static_cast<int>(idx % chunks);
  const int64_t rh = idx / chunks;
  const int h = static_cast<int>(rh % p.heads_kv);
  const int r = static_cast<int>(rh / p.heads_kv);
  int64_t pos = static_cast<int64_t>(len) + r;
  if (pos < 0) pos += p.capacity;  // counts from the end, as an index does
  if (pos < 0 || pos >= p.capacity) return;
  const RowStrides& ss = is_v ? p.v_new_strides : p.k_new_strides;
  const RowStrides& ds = is_v ? p.v_strides : p.k_strides;
  const __half* src = static_cast<const __half*>(is_v ? p.v_new : p.k_new) + b * ss.batch + h * ss.head + r * ss.row;
  __half* dst = static_cast<__half*>(is_v ? p.v_cache : p.k_cache) + b * ds.batch + h * ds.head + pos * ds.row;
  *reinterpret_cast<uint4*>(dst + c * 8) = *reinterpret_cast<const uint4*>(src + c * 8);
}

template <int D>
cudaError_t launch_splitk_t(const DecodeParams& p, cudaStream_t stream) {
  auto kern = fal_decode_splitk_kernel<D>;
  static DeviceOnce configured;
  cudaError_t e = configured.run([&] {
    return cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                DecSmem<D>::kBytes);
  });
  if (e != cudaSuccess) return e;
  const int group = p.heads_q / p.heads_kv;
  const int head_chunks = (group + 15) / 16;
  dim3 grid(p.heads_kv * head_chunks, p.splits, p.batch);
  // Its launch and set-up run under the tail of the kernel before.  us a step, one after the other: one entry of 1 999
  // positions, 32 / 8 heads of 128, 10.3 -> 9.0; eight of 2 049, 32 / 4 of 64, 10.3 -> 8.4.  (The combine kernel does not let the
  // next step's grid start early: 11.4 for the eight.)
  return launch_dependent(kern, grid, dim3(kDecThreads), DecSmem<D>::kBytes, stream, p);
}

}  // namespace

// ---------------------------------------------------------------------------
// Fixed scratch for fal_decode_static: split-K partials for callers that cannot
// allocate device memory.  It lives in the library image, so every GPU that
// loads the library carries these bytes until the process exits.
// ---------------------------------------------------------------------------
namespace {
static __device__ __align__(256) float g_decode_static_scratch[kDecodeStaticScratchBytes / sizeof(float)];
}  // namespace

// In host code the array's name is only a handle for the runtime, not a device address, so the
// address is looked up once per device (with that device current) and cached.
cudaError_t decode_static_scratch(float** ptr) {
  static std::mutex mu;
  static float* cached[64] = {};
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  if (dev < 0 || dev >= 64) return cudaErrorInvalidDevice;
  std::lock_guard<std::mutex> g(mu);
  if (cached[dev] == nullptr) {
    void* p = nullptr;
    e = cudaGetSymbolAddress(&p, g_decode_static_scratch);
    if (e != cudaSuccess) return e;
    cached[dev] = static_cast<float*>(p);
  }
  *ptr = cached[dev];
  return cudaSuccess;
}

cudaError_t launch_cache_append(const CacheAppendParams& p, cudaStream_t stream) {
  const int64_t blocks = (static_cast<int64_t>(p.rows) * p.heads_kv * (p.head_dim / 8) + 255) / 256;
  if (blocks > 0x7fffffff || p.batch > 65535) return cudaErrorInvalidValue;
  fal_cache_append_kernel<<<dim3(static_cast<unsigned>(blocks), p.batch, 2), 256, 0, stream>>>(p);
  return cudaGetLastError();
}

cudaError_t launch_decode_combine(const DecodeParams& p, cudaStream_t stream) {
  const int rows = p.batch * p.heads_q;
  const dim3 block(kCombineThreads);
  auto launch = [&](auto by_warp, auto by_block) {
    const int most = rows >= kCombineManyRows ? 2 * kCombineWarpBytes : kCombineWarpBytes;
    return p.splits * p.head_dim * 4 <= most ? launch_dependent(by_warp, dim3((rows + 3) / 4), block, 0, stream, p)
                                             : launch_dependent(by_block, dim3(rows), block, 0, stream, p);
  };
  if (p.head_dim == 128) return launch(fal_decode_combine_kernel<128, 1>, fal_decode_combine_kernel<128, 4>);
  if (p.head_dim == 64) return launch(fal_decode_combine_kernel<64, 1>, fal_decode_combine_kernel<64, 4>);
  if (p.head_dim == 256) return launch(fal_decode_combine_kernel<256, 1>, fal_decode_combine_kernel<256, 4>);
  return cudaErrorInvalidValue;
}

cudaError_t launch_decode_splitk(const DecodeParams& p, cudaStream_t stream) {
  if (p.head_dim == 128) return launch_splitk_t<128>(p, stream);
  if (p.head_dim == 64) return launch_splitk_t<64>(p, stream);
  if (p.head_dim == 256) return launch_splitk_t<256>(p, stream);
  return cudaErrorInvalidValue;
}

}  // namespace fal

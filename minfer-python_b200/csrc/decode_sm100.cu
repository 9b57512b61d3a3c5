// Split-KV decode attention over a padded KV cache, HBM-bound.
//
// The reference has no decode op (its attention op requires seq_q == seq_k,
// src/minfer/kernels/torch_ext/csrc/cuda/flash_attn/op.cuh:76); the cache
// layout [batch, n_kv_heads, max_len, head_dim] is the one its model skeleton
// allocates (src/minfer/core.py:105-127).
//
// decode_kernel: grid (parts, n_kv_heads, batch).  A thread block streams a part of the keys of one (sequence, kv
// head) and serves all `group` query heads at once, so every cache byte is read once.  Each warp runs a private
// cp.async ring of 16-key tiles (128-bit loads, rows of the cache are contiguous, so a warp instruction covers
// whole 256/128-byte rows) and keeps its own online-softmax state.
//
// The products are taken transposed: S^T = K Q^T and O^T = V^T P^T, keys (dimensions) as the 16 rows of an
// m16n8k16 tile and query heads as its 8 columns, because a GQA group is rarely more than 8.  With the heads as rows
// half of every MMA, of the accumulators and of the exponentials belonged to rows that do not exist; transposed, a
// 16-key tile takes half the MMAs and 4 exponentials per lane (groups of 9-16 take two column tiles).  P^T comes
// from S^T by two 8x8 transposes (movmatrix) per tile.  A tile in which no score exceeds
// its row's maximum so far needs no reduction over lanes.  (Counted from the source, a Q8_0 tile takes some 430 warp
// instructions, 780 were measured before.)
//
// Precision: the weights are rounded to 16 bits relative to the reference maximum, so a weight of exactly 1 - the largest
// key's so far - costs nothing, and that is worth more the fewer keys share a maximum.  Therefore the maximum is exact
// within a segment (letting it lag by up to 2^8, as the prefill kernel does, gives 2.9e-4 of the output at float16 against
// 64 bits), and every chunk / 64 tiles - as many as a warp has of a chunk in the form with chunks - the reference may
// fall by 2^4, so that the next segment's largest keys set it again.  64 sequences of 512-8192, float16 / bfloat16:
// 2.57e-4 / 2.06e-3; one maximum for all keys of a warp 2.65e-4 / 2.12e-3; chunks of 512 keys 2.59e-4 / 2.07e-3.  What it
// costs (us, with / without): those 64 sequences 165.6 / 165.2, Q8_0 115 / 109.7; one of 8192 keys, 8 kv heads, Q8_0 13.6 / 13.3;
// 8 of 48-777 6.9 / 6.8.  (As a block of its own in front of the tile, which scaled O and the sums: 116, 14.0, 7.1.  A second
// product with the rounding errors of the weights gives 2.07e-4, but an infinite value times an error of 0 is NaN.)
//
// The blocks of one (sequence, kv head) form a cluster: they share the sequence's actual tiles evenly - a padded
// cache has no empty blocks - and each pushes its partial output into the shared memory of the block that finishes
// that slice of the result, so one launch does the whole call and no partial result touches memory (one
// sequence of 1024 keys, 8 kv heads: 4.6 us, with chunks and a merging kernel 6.9).  Calls with an explicit chunk, or a
// handful of heads over a very long cache (see decode_parts in attn_api.cu), write partials to the workspace
// instead, merged by decode_combine_kernel.
//
// Q8 = true: the caches hold GGML Q8_0 blocks (32 int8 + one fp16 scale, 34 bytes;
// the reference's block_q8_0, src/minfer/kernels/torch_ext/csrc/common/types.hpp:141-146).
// The raw bytes of a 16-key tile are contiguous in the cache and ride the same
// cp.async ring; every lane then builds its tensor-core fragments straight from
// the raw rows in shared memory - two int8 dropped into the mantissas of a pair of
// halves, the bias subtracted, one multiply by the block's scale - so each value
// is (16-bit type)(q * d), rounded once, exactly as the reference's
// dequant_row_q8_0<half> produces it (csrc/quants/impl.cpp:1153-1166), and no
// 16-bit copy of the tile is ever written.  A lane takes four consecutive
// dimensions at a time: for K that permutes the 16 summands of an MMA (whose sum
// does not depend on their order), for V the rows of the output inside a block (put
// back in the merge), so every result has the bits of the 16-bit path.  Cache bytes per key drop from 4 D to 2.125 D.
//
// decode_combine_kernel: grid (n_heads, batch) merges the partials of the ceil(len / chunk) chunks of a sequence.
#include "attn_internal.h"
#include "ptx.cuh"

#include <atomic>
#include <cuda_bf16.h>
#include <cuda_fp16.h>

namespace minfer_attn {

namespace {

constexpr int kWarps = 4;
constexpr int kStages = 3;
constexpr int kMaxParts = 16;    // blocks per cluster (above 8: the non-portable size, which sm_100 has)
constexpr int kMaxRanked = 256;  // sequences a block ranks by length
// Q8_0: thread blocks per SM and ring depth (raw tiles are about half the bytes of 16-bit ones)
#ifndef MINFER_ATTN_Q8_CTAS
#define MINFER_ATTN_Q8_CTAS 3
#endif
#ifndef MINFER_ATTN_Q8_STAGES
#define MINFER_ATTN_Q8_STAGES 4
#endif
constexpr int kTileKeys = 16;

// Shared memory of a decode block: the warps' rings (reused for their partial outputs), then what the merges need.
template <int D, bool Q8, int NT>
struct Layout {
  static constexpr int kStages = Q8 ? MINFER_ATTN_Q8_STAGES : minfer_attn::kStages;
  static constexpr int kTileBytes = Q8 ? kTileKeys * (D / 32) * 34 : kTileKeys * D * 2;
  static constexpr int kWarpBytes = kStages * 2 * kTileBytes;
  static constexpr int kRingBytes = kWarps * kWarpBytes;
  static constexpr int kWmlBytes = kWarps * 8 * NT * 8;
  static constexpr int kPartBytes = 8 * NT * D * 4;
  static constexpr int kMlBytes = kMaxParts * 8 * NT * 8;
  static constexpr int kBytes = kRingBytes + kWmlBytes + kPartBytes + kMlBytes + 16;  // + the arrival barrier, an abort flag
  static_assert(kWarpBytes >= 8 * NT * (D + 4) * 4, "the per-warp ring also holds the warp's partial output");
  static_assert(kRingBytes >= (kMaxRanked + 2) * 4, "the ranking by length borrows the ring");
};

// kept out of line: the error path must not cost the streaming loop registers
__device__ __noinline__ void report_bad_page(int32_t* status, int b, int slot, int page) {
  if (status != nullptr && atomicCAS(status, 0, kStatusBadPage) == 0) {
    status[1] = b;
    status[2] = slot;
    status[3] = page;
  }
}

// A block whose wait for the cluster's partial outputs ran out.  It reports that, and stays until nothing can be stored into
// its shared memory any more: the barrier waits for the threads of the cluster that have not ended, so it passes when
// every other block has sent and ended, or has given up (after sending) as well; what is then on its way completes the mbarrier.
__device__ __noinline__ void give_up(uint64_t* arrived, int32_t* status, int part) {
  if (status != nullptr && atomicCAS(status, 0, kStatusWaitTimeout) == 0) {
    status[1] = part;
    status[2] = static_cast<int32_t>(blockIdx.z);
    status[3] = 50;
  }
  cluster_sync_unaligned();
  volatile int own_flag = 0;
  mbar_wait<true>(arrived, 0, &own_flag);
}

template <int D>
__device__ __forceinline__ uint32_t swz(int row, int chunk) {
  // 16-byte chunk index -> swizzled byte offset inside a [16 x D] 16-bit tile
  if constexpr (D == 128) return row * 256 + (((chunk & 8) | ((chunk ^ row) & 7)) << 4);
  else return row * 128 + (((chunk ^ row) & 7) << 4);
}

// Two int8 of a Q8_0 block -> a pair of 16-bit values (q * d), rounded once.  `src` holds the bytes already
// XORed with 0x80 (q + 128 as an unsigned byte); I0 / I1 pick the bytes of the low / high value.
//   float16: the byte dropped into the mantissa of the half 1024.0 reads 1024 + 128 + q; subtracting 1152 leaves q
//   exactly and one half multiply by d rounds once, as (half)(q * d) does.  No conversion instruction.
//   bfloat16: the same in fp32 (2^23 + 128 + q), where q * d is exact, then one rounding to bfloat16.
template <bool BF16>
struct Q8Scale { uint32_t h2; };          // two fp16 scales (low value's, high value's)
template <>
struct Q8Scale<true> { float2 f2; };
template <bool BF16>
__device__ __forceinline__ Q8Scale<BF16> q8_scale(uint32_t d_lo, uint32_t d_hi) {  // fp16 bit patterns
  Q8Scale<BF16> r;
  if constexpr (BF16) {
    r.f2 = make_float2(__half2float(__ushort_as_half(static_cast<unsigned short>(d_lo))),
                       __half2float(__ushort_as_half(static_cast<unsigned short>(d_hi))));
  } else {
    r.h2 = d_lo | (d_hi << 16);
  }
  return r;
}
template <bool BF16>
__device__ __forceinline__ Q8Scale<BF16> q8_scale_pair(uint32_t d) {  // both bit patterns in one word
  if constexpr (BF16) return q8_scale<true>(d & 0xFFFFu, d >> 16);
  Q8Scale<BF16> r;
  if constexpr (!BF16) r.h2 = d;
  return r;
}
// four bytes of a Q8_0 row in shared memory: a block's values start 2 bytes behind a multiple of 4 in every other block
__device__ __forceinline__ uint32_t ld_q8_word(const uint8_t* p, bool aligned4) {
  if (aligned4) return *reinterpret_cast<const uint32_t*>(p);
  return static_cast<uint32_t>(*reinterpret_cast<const uint16_t*>(p)) |
         (static_cast<uint32_t>(*reinterpret_cast<const uint16_t*>(p + 2)) << 16);
}

// The sequence that is i-th when the batch is ordered by descending length (ties by index); every block finds its own.
// Blocks start in grid order, so the long sequences start first and the last wave holds the short ones.  Four lengths
// per shared-memory read, the reads of one sequence dealt out over the lanes a small batch leaves free.  Returns the
// sequence and its length.  The lengths are clamped to [0, max_len] before they are ranked: only then is every one of them
// above the padding (-1), `mine + 1` exact, and every rank taken once.
__device__ __forceinline__ int2 sequence_by_length(const int32_t* lens, int batch, int max_len, int i, int* scratch, int tid) {
  const int n4 = (batch + 3) / 4;
  for (int t = tid; t < 4 * n4; t += kWarps * 32) scratch[t] = t < batch ? max(0, min(lens[t], max_len)) : -1;
  int lanes = 1;  // per sequence
  while (lanes < 16 && 2 * lanes * batch <= kWarps * 32) lanes *= 2;
  __syncthreads();
  for (int t0 = 0; t0 < batch; t0 += kWarps * 32 / lanes) {
    const int t = t0 + tid / lanes;
    const int mine = t < batch ? scratch[t] : 0;
    int rank = 0;
    for (int u = tid % lanes; u < n4; u += lanes) {
      const int4 x = reinterpret_cast<const int4*>(scratch)[u];
      // lengths before `t` count when equal, those behind it do not
      rank += (x.x >= mine + (4 * u >= t ? 1 : 0)) + (x.y >= mine + (4 * u + 1 >= t ? 1 : 0)) +
              (x.z >= mine + (4 * u + 2 >= t ? 1 : 0)) + (x.w >= mine + (4 * u + 3 >= t ? 1 : 0));
    }
    for (int d = lanes >> 1; d > 0; d >>= 1) rank += __shfl_xor_sync(0xFFFFFFFFu, rank, d);
    if (t < batch && rank == i && tid % lanes == 0) *reinterpret_cast<int2*>(&scratch[kMaxRanked]) = make_int2(t, mine);
  }
  __syncthreads();
  return *reinterpret_cast<const int2*>(&scratch[kMaxRanked]);
}

template <bool BF16, int I0, int I1>
__device__ __forceinline__ uint32_t q8_pair(uint32_t src, const Q8Scale<BF16>& d) {
  if constexpr (BF16) {
    const float lo = __uint_as_float(__byte_perm(src, 0x4B000000u, 0x7650 | I0));
    const float hi = __uint_as_float(__byte_perm(src, 0x4B000000u, 0x7650 | I1));
    const float2 q = __fadd2_rn(make_float2(lo, hi), make_float2(-8388736.f, -8388736.f));
    const float2 v = __fmul2_rn(q, d.f2);
    return pack2<true>(v.x, v.y);
  } else {
    const uint32_t x = __byte_perm(src, 0x64646464u, 0x5040 | I0 | (I1 << 8));
    const uint32_t bias = 0x64806480u;  // 1152.0 twice
    const __half2 q = __hsub2(*reinterpret_cast<const __half2*>(&x), *reinterpret_cast<const __half2*>(&bias));
    const __half2 v = __hmul2(q, *reinterpret_cast<const __half2*>(&d.h2));
    return *reinterpret_cast<const uint32_t*>(&v);
  }
}

// Paged: the caches are pools of pages reached through a.block_table (a separate instantiation, so that the
// contiguous form keeps its registers).  NT: 8-column tiles the query heads of a kv head fill (1: group <= 8).
template <int D, bool BF16, bool Q8, bool Paged, int NT>
__global__ void __launch_bounds__(kWarps * 32, (Q8 && NT == 1) ? MINFER_ATTN_Q8_CTAS : 2) decode_kernel(const DecodeArgs a) {
  using L = Layout<D, Q8, NT>;
  constexpr int kSt = L::kStages;
  constexpr int kTileBytes = L::kTileBytes;                // one of K or V
  constexpr int kChunksPerRow = D / 8;                     // 16-byte chunks
  constexpr int kLoadsPerLane = kTileKeys * kChunksPerRow / 32;
  // Q8_0: raw rows of D/32 blocks of 34 bytes; a 16-row tile is one contiguous, 16-byte aligned span
  constexpr int kQRowBytes = (D / 32) * 34;
  constexpr int kQChunks = kTileKeys * kQRowBytes / 16;
  constexpr int kQLoadsPerLane = (kQChunks + 31) / 32;
  constexpr int kWarpBytes = L::kWarpBytes;

  extern __shared__ __align__(128) uint8_t smem[];

  const int tid = threadIdx.x;
  const int warp = tid >> 5;
  const int lane = tid & 31;
  const int kvh = blockIdx.y;
  const bool clustered = a.part_o == nullptr;
  const int part = blockIdx.x;       // which piece of the sequence
  const int n_parts = gridDim.x;

  uint64_t* arrived = reinterpret_cast<uint64_t*>(smem + L::kBytes - 16);  // completes when all blocks' partial outputs are here
  volatile int* abort_flag = reinterpret_cast<volatile int*>(arrived + 1);
  grid_launch_dependents();
  if (clustered && n_parts > 1) {
    if (tid == 0) {
      *abort_flag = 0;
      mbar_init(arrived, 1);
      mbar_fence_init();
      // D / n_parts dimensions and the (max, sum) of every head, from every block
      mbar_arrive_expect_tx(arrived, static_cast<uint32_t>(a.group * (D * 4 + n_parts * 8)));
    }
    __syncwarp();
    cluster_arrive();  // awaited before the first access to another block's shared memory
  }
  grid_dependency_wait();

  // ---- which sequence: in order, or the i-th longest (a.by_length: few enough sequences to rank them here) ----
  int b = blockIdx.z, len;
  if (a.by_length) {
    const int2 x = sequence_by_length(a.lens, a.batch, a.max_len, b, reinterpret_cast<int*>(smem), tid);
    b = x.x;
    len = x.y;
  } else {
    len = max(0, min(a.lens[b], a.max_len));
  }
  // ---- the keys of this block: an even share of the sequence's tiles, or the part-th chunk ----
  int c0, c1;
  if (clustered) {
    const int nt_seq = (len + kTileKeys - 1) / kTileKeys;
    c0 = static_cast<int>(static_cast<unsigned>(nt_seq) * static_cast<unsigned>(part) / static_cast<unsigned>(n_parts)) * kTileKeys;
    c1 = min(len, static_cast<int>(static_cast<unsigned>(nt_seq) * static_cast<unsigned>(part + 1) / static_cast<unsigned>(n_parts)) * kTileKeys);
  } else {
    c0 = part * a.chunk;
    if (c0 >= len) return;
    c1 = min(len, c0 + a.chunk);
  }
  const int nt = c1 > c0 ? (c1 - c0 + kTileKeys - 1) / kTileKeys : 0;
  const int nt_w = (nt > warp) ? (nt - warp + kWarps - 1) / kWarps : 0;

  uint8_t* wsm = smem + warp * kWarpBytes;
  const uint32_t wsm_u32 = smem_u32(wsm);
  // Byte offset of the first row of a 16-key tile inside either cache.  Paged caches: the tile lies inside one
  // page (page_size is a multiple of 16), found through the block table; strides are then those of the pool.
  // (Everything is recomputed per tile from kernel parameters, which costs no registers between tiles.)
  auto tile_offset = [&](int key0) -> size_t {
    constexpr size_t kUnit = Q8 ? 1 : 2;  // Q8_0 strides are in bytes
    const size_t row_bytes = Q8 ? static_cast<size_t>(kQRowBytes) : 2 * static_cast<size_t>(a.kv_stride[2]);
    const size_t head_off = kUnit * static_cast<size_t>(kvh) * a.kv_stride[1];
    if constexpr (Paged) {
      const int slot = key0 / a.page_size;
      // (an ordinary load: the read-only path is for memory that nobody writes while this kernel is resident, and it is
      // resident before the kernel in front, which may write the table, has ended)
      int page = a.block_table[static_cast<size_t>(b) * a.table_stride + slot];
      if (static_cast<unsigned>(page) >= static_cast<unsigned>(a.n_pages)) {
        // never follow an entry that points outside the pools: report it and read page 0 instead
        if (lane == 0) report_bad_page(a.status, b, slot, page);
        page = 0;
      }
      return kUnit * static_cast<size_t>(page) * a.kv_stride[0] + head_off + static_cast<size_t>(key0 % a.page_size) * row_bytes;
    }
    return kUnit * static_cast<size_t>(b) * a.kv_stride[0] + head_off + static_cast<size_t>(key0) * row_bytes;
  };
  const size_t row_stride_bytes = 2 * static_cast<size_t>(a.kv_stride[2]);  // 16-bit caches

  auto issue_tile = [&](int i) {  // i-th tile of this warp -> stage i % kSt
    if (i < nt_w) {
      const int key0 = c0 + (warp + i * kWarps) * kTileKeys;
      const size_t toff = tile_offset(key0);
      uint8_t* dst_k = wsm + (i % kSt) * 2 * kTileBytes;
      uint8_t* dst_v = dst_k + kTileBytes;
      if constexpr (Q8) {
        // strides of a Q8_0 cache are in bytes; rows are contiguous
        const uint8_t* kq = reinterpret_cast<const uint8_t*>(a.k) + toff;
        const uint8_t* vq = reinterpret_cast<const uint8_t*>(a.v) + toff;
        // bytes of live rows in this tile (rows beyond the sequence are neither read nor used)
        const int live = min(kTileKeys, c1 - key0) * kQRowBytes;
#pragma unroll
        for (int t = 0; t < kQLoadsPerLane; ++t) {
          const int ch = t * 32 + lane;
          if (ch < kQChunks) {
            const bool pred = ch * 16 < live;  // a chunk that starts inside a live row stays inside the cache
            cp_async_16(dst_k + ch * 16, kq + (pred ? ch * 16 : 0), pred);
            cp_async_16(dst_v + ch * 16, vq + (pred ? ch * 16 : 0), pred);
          }
        }
      } else {
#pragma unroll
        for (int t = 0; t < kLoadsPerLane; ++t) {
          const int idx = t * 32 + lane;
          const int row = idx / kChunksPerRow;
          const int chunk = idx % kChunksPerRow;
          const bool pred = key0 + row < c1;
          const size_t goff = toff + static_cast<size_t>(pred ? row : 0) * row_stride_bytes + chunk * 16;
          cp_async_16(dst_k + swz<D>(row, chunk), reinterpret_cast<const uint8_t*>(a.k) + goff, pred);
          cp_async_16(dst_v + swz<D>(row, chunk), reinterpret_cast<const uint8_t*>(a.v) + goff, pred);
        }
      }
    }
    cp_async_commit();
  };

  if (a.by_length) __syncthreads();  // the ranking's scratch is the ring's memory
#pragma unroll
  for (int s = 0; s < kSt - 1; ++s) issue_tile(s);

  // ---- Q^T fragments (B operand): columns = query heads of this kv head (zero beyond group).  Q8_0: the 16 k slots
  // of a step hold its dimensions in another order (slots 2t, 2t+1, 2t+8, 2t+9 of lane t: dimensions 4t .. 4t+3), so that a lane's
  // four K values are four consecutive bytes; an MMA's sum over its 16 slots does not depend on their order. ----
  const int g0 = lane >> 2;
  const int tq = lane & 3;
  uint32_t qf[NT][D / 16][2];
  {
    const uint8_t* qb = reinterpret_cast<const uint8_t*>(a.q) + 2 * static_cast<size_t>(b) * a.q_stride[0];
#pragma unroll
    for (int n = 0; n < NT; ++n) {
      const int g = g0 + 8 * n;
      const bool live = g < a.group;
      const uint8_t* qp = qb + 2 * static_cast<size_t>(kvh * a.group + (live ? g : 0)) * a.q_stride[1];
#pragma unroll
      for (int ks = 0; ks < D / 16; ++ks) {
        if constexpr (Q8) {
          const uint2 x = *reinterpret_cast<const uint2*>(qp + 2 * (ks * 16 + tq * 4));
          qf[n][ks][0] = live ? x.x : 0u;
          qf[n][ks][1] = live ? x.y : 0u;
        } else {
          const uint32_t x = *reinterpret_cast<const uint32_t*>(qp + 2 * (ks * 16 + tq * 2));
          const uint32_t y = *reinterpret_cast<const uint32_t*>(qp + 2 * (ks * 16 + tq * 2 + 8));
          qf[n][ks][0] = live ? x : 0u;
          qf[n][ks][1] = live ? y : 0u;
        }
      }
    }
  }

  // O^T: oacc[n][m][0..3] = (row g0, heads 2 tq, 2 tq + 1), (row g0 + 8, the same) of the m-th 16-row tile
  float oacc[NT][D / 16][4];
#pragma unroll
  for (int n = 0; n < NT; ++n)
#pragma unroll
    for (int m = 0; m < D / 16; ++m) oacc[n][m][0] = oacc[n][m][1] = oacc[n][m][2] = oacc[n][m][3] = 0.f;
  float m_ref[NT][2], l_run[NT][2];  // per head: reference maximum (log2 domain), this lane's share of the row sum
#pragma unroll
  for (int n = 0; n < NT; ++n) {
    m_ref[n][0] = m_ref[n][1] = -INFINITY;
    l_run[n][0] = l_run[n][1] = 0.f;
  }
  const float sl2 = a.scale_log2;
  const int seg_mask = clustered ? a.chunk / 64 - 1 : -1;  // tiles per segment (a power of two) - 1; a chunk is one segment

  // ldmatrix lane roles
  const int lm_mi = lane >> 3;
  const int lm_r = lane & 7;

  for (int i = 0; i < nt_w; ++i) {
    cp_async_wait<kSt - 2>();
    __syncwarp();
    issue_tile(i + kSt - 1);

    const int key0 = c0 + (warp + i * kWarps) * kTileKeys;
    // ---- S^T[16 keys x 8 heads] = K Q^T ----
    // (two accumulators: half the length of the chain of dependent MMAs)
    float s[NT][4], s2[NT][4];
#pragma unroll
    for (int n = 0; n < NT; ++n)
#pragma unroll
      for (int e = 0; e < 4; ++e) s[n][e] = s2[n][e] = 0.f;
    [[maybe_unused]] const uint8_t* raw_k = wsm + (i % kSt) * 2 * kTileBytes;  // Q8: this tile's raw K rows, then V
    [[maybe_unused]] const uint32_t sk = wsm_u32 + (i % kSt) * 2 * kTileBytes;
    if constexpr (Q8) {
      // A fragments from the raw rows: keys g0 / g0 + 8, per 16-dimension step four consecutive bytes.  Rows beyond
      // the chunk were zero-filled by the copy (their scores are masked below).
#pragma unroll
      for (int blk = 0; blk < D / 32; ++blk) {
        uint32_t kf[2][4];
#pragma unroll
        for (int kk = 0; kk < 2; ++kk) {
          const uint8_t* bp = raw_k + (g0 + 8 * kk) * kQRowBytes + blk * 34;
          const uint32_t db = *reinterpret_cast<const uint16_t*>(bp);
          const Q8Scale<BF16> d = q8_scale<BF16>(db, db);
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            const uint32_t x = ld_q8_word(bp + 2 + 16 * h + 4 * tq, (blk & 1) != 0) ^ 0x80808080u;
            kf[h][kk] = q8_pair<BF16, 0, 1>(x, d);
            kf[h][2 + kk] = q8_pair<BF16, 2, 3>(x, d);
          }
        }
#pragma unroll
        for (int h = 0; h < 2; ++h)
#pragma unroll
          for (int n = 0; n < NT; ++n) mma_16816<BF16>(h ? s2[n] : s[n], kf[h], qf[n][2 * blk + h][0], qf[n][2 * blk + h][1]);
      }
    } else {
#pragma unroll
      for (int ks = 0; ks < D / 16; ++ks) {
        uint32_t kf[4];
        ldmatrix_x4(sk + swz<D>((lm_mi & 1) * 8 + lm_r, 2 * ks + (lm_mi >> 1)), kf[0], kf[1], kf[2], kf[3]);
#pragma unroll
        for (int n = 0; n < NT; ++n) mma_16816<BF16>((ks & 1) ? s2[n] : s[n], kf, qf[n][ks][0], qf[n][ks][1]);
      }
    }

#pragma unroll
    for (int n = 0; n < NT; ++n)
#pragma unroll
      for (int e = 0; e < 4; ++e) s[n][e] += s2[n][e];

    // ---- online softmax over the keys: x = s * scale - maximum so far; a tile in which no score exceeds it needs no
    // reduction over the lanes.  The first tile of a segment lets the reference fall (by up to 2^4, to its own maximum);
    // not while a sum is large, so that a long run of falling scores cannot overflow. ----
    const bool partial = key0 + kTileKeys > c1;
    const bool dead0 = partial && key0 + g0 >= c1, dead1 = partial && key0 + g0 + 8 >= c1;
    float x[NT][4];
    const bool fresh = (i & seg_mask) == 0;
    bool move = fresh;
#pragma unroll
    for (int n = 0; n < NT; ++n) {
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        x[n][e] = fmaf(s[n][e], sl2, -m_ref[n][e & 1]);  // +inf before the first tile
        if (e < 2 ? dead0 : dead1) x[n][e] = -INFINITY;
      }
      move |= fmaxf(fmaxf(x[n][0], x[n][1]), fmaxf(x[n][2], x[n][3])) > 0.f;
    }
    if (__any_sync(0xFFFFFFFFu, move)) {
      bool room = fresh;
#pragma unroll
      for (int n = 0; n < NT; ++n) room = room && fmaxf(l_run[n][0], l_run[n][1]) < 512.f;
      const float drop = __all_sync(0xFFFFFFFFu, room) ? 4.f : 0.f;
#pragma unroll
      for (int n = 0; n < NT; ++n) {
        float alpha[2];
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          float mx = fmaxf(dead0 ? -INFINITY : s[n][h] * sl2, dead1 ? -INFINITY : s[n][2 + h] * sl2);
          mx = fmaxf(mx, __shfl_xor_sync(0xFFFFFFFFu, mx, 4));
          mx = fmaxf(mx, __shfl_xor_sync(0xFFFFFFFFu, mx, 8));
          mx = fmaxf(mx, __shfl_xor_sync(0xFFFFFFFFu, mx, 16));
          const float m_new = fmaxf(m_ref[n][h] - drop, mx);  // finite: every tile holds at least one live key
          alpha[h] = ex2_approx(m_ref[n][h] - m_new);  // first tile: exp2(-inf) = 0
          m_ref[n][h] = m_new;
          l_run[n][h] *= alpha[h];
        }
#pragma unroll
        for (int m = 0; m < D / 16; ++m) {
          oacc[n][m][0] *= alpha[0];
          oacc[n][m][1] *= alpha[1];
          oacc[n][m][2] *= alpha[0];
          oacc[n][m][3] *= alpha[1];
        }
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          x[n][e] = fmaf(s[n][e], sl2, -m_ref[n][e & 1]);
          if (e < 2 ? dead0 : dead1) x[n][e] = -INFINITY;
        }
      }
    }
    uint32_t pb[NT][2];  // P^T fragments (B operand): keys 2 tq, 2 tq + 1 (+ 8) of head g0
#pragma unroll
    for (int n = 0; n < NT; ++n) {
#pragma unroll
      for (int e = 0; e < 4; ++e) x[n][e] = ex2_approx(x[n][e]);
      l_run[n][0] += x[n][0] + x[n][2];
      l_run[n][1] += x[n][1] + x[n][3];
      pb[n][0] = movmatrix_trans(pack2<BF16>(x[n][0], x[n][1]));
      pb[n][1] = movmatrix_trans(pack2<BF16>(x[n][2], x[n][3]));
    }

    // ---- O^T[D x 8 heads] += V^T P^T ----
    if constexpr (Q8) {
      // A fragments pair two keys per register: lane (g0, tq) reads, for keys 2 tq, 2 tq + 1, 2 tq + 8, 2 tq + 9, the
      // four bytes at dimensions 4 g0 .. 4 g0 + 3 of every block, interleaves the rows pairwise and converts.  Row r of
      // 16-row tile 2 blk + j is then dimension 32 blk + 4 (r % 8) + 2 j + r / 8.
      const uint8_t* rv = raw_k + kTileBytes + (2 * tq) * kQRowBytes;
      // The copy zero-fills whole 16-byte pieces beyond the chunk, so the first row past the end can hold a few
      // real cache bytes, a scale among them: rows past the end get scale 0 (their weights are 0, and 0 * 0 = 0
      // whatever the cache holds there).
      uint32_t ok01 = 0xFFFFFFFFu, ok23 = 0xFFFFFFFFu;
      if (partial) {
        const int left = c1 - key0 - 2 * tq;
        ok01 = (left > 0 ? 0xFFFFu : 0u) | (left > 1 ? 0xFFFF0000u : 0u);
        ok23 = (left > 8 ? 0xFFFFu : 0u) | (left > 9 ? 0xFFFF0000u : 0u);
      }
#pragma unroll
      for (int blk = 0; blk < D / 32; ++blk) {
        uint32_t w[4], dsc[4];
#pragma unroll
        for (int r = 0; r < 4; ++r) {
          const uint8_t* bp = rv + ((r & 1) + 8 * (r >> 1)) * kQRowBytes + blk * 34;
          dsc[r] = *reinterpret_cast<const uint16_t*>(bp);
          w[r] = ld_q8_word(bp + 2 + 4 * g0, (blk & 1) != 0) ^ 0x80808080u;
        }
        const Q8Scale<BF16> d01 = q8_scale_pair<BF16>((dsc[0] | (dsc[1] << 16)) & ok01);
        const Q8Scale<BF16> d23 = q8_scale_pair<BF16>((dsc[2] | (dsc[3] << 16)) & ok23);
#pragma unroll
        for (int j = 0; j < 2; ++j) {
          const uint32_t e01 = __byte_perm(w[0], w[1], j ? 0x7362 : 0x5140), e23 = __byte_perm(w[2], w[3], j ? 0x7362 : 0x5140);
          const uint32_t vf[4] = {q8_pair<BF16, 0, 1>(e01, d01), q8_pair<BF16, 2, 3>(e01, d01),
                                  q8_pair<BF16, 0, 1>(e23, d23), q8_pair<BF16, 2, 3>(e23, d23)};
#pragma unroll
          for (int n = 0; n < NT; ++n) mma_16816<BF16>(oacc[n][2 * blk + j], vf, pb[n][0], pb[n][1]);
        }
      }
    } else {
      const uint32_t sv = sk + kTileBytes;
#pragma unroll
      for (int m = 0; m < D / 16; ++m) {
        uint32_t vf[4];
        ldmatrix_x4_trans(sv + swz<D>((lm_mi >> 1) * 8 + lm_r, 2 * m + (lm_mi & 1)), vf[0], vf[1], vf[2], vf[3]);
#pragma unroll
        for (int n = 0; n < NT; ++n) mma_16816<BF16>(oacc[n][m], vf, pb[n][0], pb[n][1]);
      }
    }
  }
  cp_async_wait<0>();

  // ---- merge the warps through shared memory (reusing the ring buffers) ----
  const int group = a.group;
#pragma unroll
  for (int n = 0; n < NT; ++n)
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      l_run[n][h] += __shfl_xor_sync(0xFFFFFFFFu, l_run[n][h], 4);
      l_run[n][h] += __shfl_xor_sync(0xFFFFFFFFu, l_run[n][h], 8);
      l_run[n][h] += __shfl_xor_sync(0xFFFFFFFFu, l_run[n][h], 16);
    }
  __syncthreads();
  constexpr int kRow = D + 4;  // floats per head: the four lanes of a row fall into different banks
  float* mo = reinterpret_cast<float*>(wsm);
  float2* wml = reinterpret_cast<float2*>(smem + L::kRingBytes);                       // [kWarps][8 NT] (max, sum) per warp
  float* pbuf = reinterpret_cast<float*>(smem + L::kRingBytes + L::kWmlBytes);         // [n_parts][group][dims]
  float2* pml = reinterpret_cast<float2*>(smem + L::kRingBytes + L::kWmlBytes + L::kPartBytes);  // [n_parts][group]
  static_assert(D / 4 >= kMaxParts, "a head's four-dimension pieces cover the blocks of a cluster");
  constexpr int kLogD = D == 128 ? 7 : 6;
#pragma unroll
  for (int n = 0; n < NT; ++n)
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int g = 8 * n + 2 * tq + h;
      if (g < group) {
#pragma unroll
        for (int m = 0; m < D / 16; ++m) {
          if constexpr (Q8) {
            *reinterpret_cast<float2*>(&mo[g * kRow + 32 * (m >> 1) + 4 * g0 + 2 * (m & 1)]) = make_float2(oacc[n][m][h], oacc[n][m][2 + h]);
          } else {
            mo[g * kRow + 16 * m + g0] = oacc[n][m][h];
            mo[g * kRow + 16 * m + 8 + g0] = oacc[n][m][2 + h];
          }
        }
        if (g0 == 0) wml[warp * 8 * NT + g] = make_float2(m_ref[n][h], l_run[n][h]);
      }
    }
  __syncthreads();
  // Block r of the cluster finishes dimensions [r, r + 1) * D / n_parts of every head (n_parts is a power of two of at
  // most D / 4).  All index arithmetic below is shifts: this is a chain of latencies, and a division by a runtime value is
  // a tenth of it.
  const bool exchange = clustered && n_parts > 1;
  const int log_dims = kLogD - (exchange ? __ffs(n_parts) - 1 : 0);  // dimensions per block
  const int dims = 1 << log_dims;
  if (exchange) cluster_wait();  // every block of the cluster has started and initialised its barrier
  for (int e4 = tid; e4 < group * (D / 4); e4 += kWarps * 32) {
    const int g = e4 / (D / 4), j = e4 % (D / 4), d = j * 4;
    float2 ml[kWarps];
    float M = -INFINITY;
#pragma unroll
    for (int w = 0; w < kWarps; ++w) {
      ml[w] = wml[w * 8 * NT + g];
      M = fmaxf(M, ml[w].x);
    }
    float4 o = make_float4(0.f, 0.f, 0.f, 0.f);
    float l = 0.f;
#pragma unroll
    for (int w = 0; w < kWarps; ++w) {
      const float sc = (ml[w].x == -INFINITY) ? 0.f : ex2_approx(ml[w].x - M);
      const float4 x = *reinterpret_cast<const float4*>(reinterpret_cast<const float*>(smem + w * kWarpBytes) + g * kRow + d);
      o.x += sc * x.x;
      o.y += sc * x.y;
      o.z += sc * x.z;
      o.w += sc * x.w;
      l += sc * ml[w].y;
    }
    const int h = kvh * group + g;
    if (exchange) {
      // the block that finishes these four dimensions gets them, and (from one lane each) every block the (max, sum)
      const uint32_t bar_addr = smem_u32(arrived);
      const int rank = d >> log_dims;
      st_async_v4(cluster_map(smem_u32(&pbuf[(((part * group + g) << log_dims) + d) - (rank << log_dims)]), rank), o, cluster_map(bar_addr, rank));
      if (j < n_parts) st_async_v2(cluster_map(smem_u32(&pml[part * group + g]), j), M, l, cluster_map(bar_addr, j));
    } else if (clustered) {
      const float inv = 1.f / l;
      if (!(l > 0.f)) o = make_float4(0.f, 0.f, 0.f, 0.f);  // no key, or a sum that is NaN
      else o = make_float4(o.x * inv, o.y * inv, o.z * inv, o.w * inv);
      uint8_t* op = reinterpret_cast<uint8_t*>(a.out) +
                    2 * (static_cast<size_t>(b) * a.out_stride[0] + static_cast<size_t>(h) * a.out_stride[1] + d);
      *reinterpret_cast<uint2*>(op) = make_uint2(pack2<BF16>(o.x, o.y), pack2<BF16>(o.z, o.w));
    } else {
      const size_t pidx = (static_cast<size_t>(b) * a.n_heads + h) * n_parts + part;
      *reinterpret_cast<float4*>(a.part_o + pidx * D + d) = o;
      if (d == 0) *reinterpret_cast<float2*>(a.part_ml + pidx * 2) = make_float2(M, l);
    }
  }
  if (!exchange) return;
  // ---- merge the cluster's blocks: each finishes its dimensions once every block's values have arrived (a block that
  // has sent its own and received the others' has nothing more to do with them) ----
  // (their stores are released at the scope of the cluster: the wait acquires there)
  if (!mbar_wait<true>(arrived, 0, abort_flag)) {
    give_up(arrived, a.status, part);
    return;
  }
  for (int t = 2 * tid; t < (group << log_dims); t += 2 * kWarps * 32) {
    const int g = t >> log_dims, d = (part << log_dims) + (t & (dims - 1));
    float2 ml[kMaxParts], x[kMaxParts];
    float M = -INFINITY, l = 0.f, o0 = 0.f, o1 = 0.f;
#pragma unroll
    for (int p = 0; p < kMaxParts; ++p) {
      const int q = p < n_parts ? p : 0;
      ml[p] = pml[q * group + g];
      x[p] = *reinterpret_cast<const float2*>(&pbuf[((q * group) << log_dims) + t]);
      if (p >= n_parts) {  // counts for nothing, whatever part 0 holds
        ml[p] = make_float2(-INFINITY, 0.f);
        x[p] = make_float2(0.f, 0.f);
      }
      M = fmaxf(M, ml[p].x);
    }
#pragma unroll
    for (int p = 0; p < kMaxParts; ++p) {
      const float sc = (ml[p].x == -INFINITY) ? 0.f : ex2_approx(ml[p].x - M);
      o0 += sc * x[p].x;
      o1 += sc * x[p].y;
      l += sc * ml[p].y;
    }
    const float inv = 1.f / l;
    o0 = l > 0.f ? o0 * inv : 0.f;
    o1 = l > 0.f ? o1 * inv : 0.f;
    uint8_t* op = reinterpret_cast<uint8_t*>(a.out) + 2 * (static_cast<size_t>(b) * a.out_stride[0] +
                                                           static_cast<size_t>(kvh * group + g) * a.out_stride[1] + d);
    *reinterpret_cast<uint32_t*>(op) = pack2<BF16>(o0, o1);
  }
}

// The merge is a latency problem (a few hundred bytes per thread, every load a trip to L2 or HBM), so the loads are
// issued eight at a time: the (max, sum) pairs of eight splits, then the eight partial outputs they weight.
template <int D, bool BF16>
__global__ void __launch_bounds__(D) decode_combine_kernel(const DecodeArgs a) {
  const int h = blockIdx.x;
  const int b = blockIdx.y;
  const int d = threadIdx.x;
  grid_launch_dependents();
  grid_dependency_wait();
  const int len = min(a.lens[b], a.max_len);
  const int ns = (len + a.chunk - 1) / a.chunk;
  const size_t p0 = (static_cast<size_t>(b) * a.n_heads + h) * a.n_split;
  const float2* ml = reinterpret_cast<const float2*>(a.part_ml) + p0;
  const float* po = a.part_o + p0 * D + d;
  constexpr int kBatch = 8;
  float M = -INFINITY;
  for (int s0 = 0; s0 < ns; s0 += kBatch) {
    float m[kBatch];
#pragma unroll
    for (int j = 0; j < kBatch; ++j) m[j] = (s0 + j < ns) ? ml[s0 + j].x : -INFINITY;
#pragma unroll
    for (int j = 0; j < kBatch; ++j) M = fmaxf(M, m[j]);
  }
  float o = 0.f, l = 0.f;
  for (int s0 = 0; s0 < ns; s0 += kBatch) {
    float2 w[kBatch];
    float x[kBatch];
#pragma unroll
    for (int j = 0; j < kBatch; ++j) {
      const bool live = s0 + j < ns;
      w[j] = live ? ml[s0 + j] : make_float2(-INFINITY, 0.f);
      x[j] = live ? po[static_cast<size_t>(s0 + j) * D] : 0.f;
    }
#pragma unroll
    for (int j = 0; j < kBatch; ++j) {
      const float sc = (w[j].x == -INFINITY) ? 0.f : ex2_approx(w[j].x - M);
      l += sc * w[j].y;
      o += sc * x[j];
    }
  }
  const float r = (l > 0.f) ? o / l : 0.f;
  uint8_t* op = reinterpret_cast<uint8_t*>(a.out) +
                2 * (static_cast<size_t>(b) * a.out_stride[0] + static_cast<size_t>(h) * a.out_stride[1] + d);
  if constexpr (BF16) *reinterpret_cast<__nv_bfloat16*>(op) = __float2bfloat16_rn(r);
  else *reinterpret_cast<__half*>(op) = __float2half_rn(r);
}

template <int D, bool BF16, bool Q8, bool Paged, int NT>
cudaError_t launch_heads(const DecodeArgs& a, cudaStream_t stream) {
  auto* kernel = decode_kernel<D, BF16, Q8, Paged, NT>;
  constexpr int smem = Layout<D, Q8, NT>::kBytes;
  static std::atomic<bool> attr_done[64] = {};  // set-once flags; the attribute calls themselves are idempotent
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  if (dev >= 64 || !attr_done[dev].load(std::memory_order_acquire)) {
    e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e != cudaSuccess) return e;
    e = cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
    if (e != cudaSuccess) return e;
    if (dev < 64) attr_done[dev].store(true, std::memory_order_release);
  }
  const bool clustered = a.part_o == nullptr;
  LaunchAttrs at(stream);
  at.cfg.gridDim = dim3(a.n_split, a.n_kv_heads, a.batch);
  at.cfg.blockDim = dim3(kWarps * 32);
  at.cfg.dynamicSmemBytes = smem;
  if (clustered && a.n_split > 1) at.cluster(a.n_split);
  e = cudaLaunchKernelEx(&at.cfg, kernel, a);
  if (e != cudaSuccess || clustered) return e;
  LaunchAttrs ac(stream);
  ac.cfg.gridDim = dim3(a.n_heads, a.batch);
  ac.cfg.blockDim = dim3(D);
  return cudaLaunchKernelEx(&ac.cfg, decode_combine_kernel<D, BF16>, a);
}

template <int D, bool BF16, bool Q8>
cudaError_t launch_one(const DecodeArgs& a, cudaStream_t stream) {
  if (a.group <= 8)
    return a.block_table != nullptr ? launch_heads<D, BF16, Q8, true, 1>(a, stream) : launch_heads<D, BF16, Q8, false, 1>(a, stream);
  return a.block_table != nullptr ? launch_heads<D, BF16, Q8, true, 2>(a, stream) : launch_heads<D, BF16, Q8, false, 2>(a, stream);
}

}  // namespace

cudaError_t launch_decode(const DecodeArgs& a, int head_dim, bool bf16, bool q8, cudaStream_t stream) {
  if (q8) {
    if (head_dim == 128) return bf16 ? launch_one<128, true, true>(a, stream) : launch_one<128, false, true>(a, stream);
    return bf16 ? launch_one<64, true, true>(a, stream) : launch_one<64, false, true>(a, stream);
  }
  if (head_dim == 128) return bf16 ? launch_one<128, true, false>(a, stream) : launch_one<128, false, false>(a, stream);
  return bf16 ? launch_one<64, true, false>(a, stream) : launch_one<64, false, false>(a, stream);
}

}  // namespace minfer_attn

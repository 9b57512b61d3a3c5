// One pass over a dense attention mask that lets the prefill kernel skip key
// tiles nobody can see and read mask bytes only where a tile is mixed.
//
// The reference's op takes a dense bool mask [B, 1, L, L] for every call
// (src/minfer/kernels/torch_ext/csrc/cuda/flash_attn/op.cuh:28; its callers
// build a causal or a sliding-window one, test/kernels.py:242,276-278), so a
// drop-in cannot assume causality; classifying 128 x 128 tiles recovers the
// structure at the cost of reading the mask once (HBM-bound, ~1 byte per
// score instead of the B*H re-reads a per-head kernel would do).
#include "attn_internal.h"
#include "ptx.cuh"

namespace minfer_attn {

namespace {

constexpr int kTile = 128;

// 16 columns of one mask row as words.  (Ordinary loads: the kernel starts beside the one that may write the mask, and
// the read-only path is for memory that nobody writes during the kernel's life.)
__device__ __forceinline__ void row_words16(const uint8_t* p, uint32_t (&w)[4]) {
  const uint32_t mis = static_cast<uint32_t>(reinterpret_cast<uintptr_t>(p)) & 15u;
  if (mis == 0) {
    const uint4 v = *reinterpret_cast<const uint4*>(p);
    w[0] = v.x; w[1] = v.y; w[2] = v.z; w[3] = v.w;
  } else {
    // rows of a mask whose length is no multiple of 16 start anywhere: aligned words, shifted into place (every
    // word read holds at least one byte of these 16 columns)
    const uint32_t* q = reinterpret_cast<const uint32_t*>(p - (mis & 3u));
    const uint32_t sh = (mis & 3u) * 8u;
    uint32_t a[5];
#pragma unroll
    for (int i = 0; i < 4; ++i) a[i] = q[i];
    a[4] = sh ? q[4] : 0u;
#pragma unroll
    for (int i = 0; i < 4; ++i) w[i] = __funnelshift_r(a[i], a[i + 1], sh);
  }
}

// grid (key tiles, query tiles, batch), 256 threads: 8 threads per row (16 columns each), 32 rows per pass, four
// passes whose loads are all in flight together.  The class of a tile needs no bits: an OR of its words, and an AND of
// their bytes' top bits after a carry (nonzero_bits below); computing every tile's bits first made the kernel
// instruction-bound.  Mixed tiles then leave their bits behind (128 rows of 16 bytes), so that the attention
// kernel, which needs a mixed tile once per head pair, reads 16 bytes per row instead of 128 and no row of it is
// misaligned.
__global__ void __launch_bounds__(256, 6) mask_classify_kernel(const uint8_t* mask, uint8_t* cls, uint32_t* bits,
                                                               int* counter, int seq_q, int seq_k) {
  grid_launch_dependents();  // the attention kernel sets up beside the last blocks of this pass
  grid_dependency_wait();
  // its work-item counter starts at zero
  if (threadIdx.x == 0 && blockIdx.x == 0 && blockIdx.y == 0 && blockIdx.z == 0) *counter = 0;
  const int kt = blockIdx.x, qt = blockIdx.y, b = blockIdx.z;
  const int part = threadIdx.x & 7;
  const int r0 = static_cast<int>(threadIdx.x) >> 3;
  const int n = min(16, seq_k - (kt * kTile + part * 16));  // columns of this thread that exist (may be <= 0)
  const int rows = seq_q - qt * kTile - r0;                 // pass i has a row of this thread if 32 i < rows
  const uint8_t* base = mask + (static_cast<size_t>(b) * seq_q + qt * kTile + r0) * seq_k + kt * kTile + part * 16;
  uint32_t w[4][4];
  uint32_t seen = 0u, shown = 0x80808080u;
  if (n == 16) {
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      if (32 * i < rows) {
        row_words16(base + static_cast<size_t>(32 * i) * seq_k, w[i]);
      } else {
        w[i][0] = w[i][1] = w[i][2] = w[i][3] = 0u;
      }
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      if (32 * i < rows) {
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          seen |= w[i][e];
          shown &= ((w[i][e] & 0x7F7F7F7Fu) + 0x7F7F7F7Fu) | w[i][e];
        }
      }
    }
  } else {
#pragma unroll
    for (int i = 0; i < 4; ++i) {
#pragma unroll
      for (int e = 0; e < 16; ++e) {
        uint32_t& x = w[i][e >> 2];
        if ((e & 3) == 0) x = 0u;
        if (e < n && 32 * i < rows) {
          const uint32_t byte = base[static_cast<size_t>(32 * i) * seq_k + e];
          x |= byte << (8 * (e & 3));
          seen |= byte;
          if (byte == 0u) shown = 0u;
        }
      }
    }
  }
  const int any_cta = __syncthreads_or(seen != 0u ? 1 : 0);
  const int all_cta = __syncthreads_and(shown == 0x80808080u ? 1 : 0);
  const size_t tile = (static_cast<size_t>(b) * gridDim.y + qt) * gridDim.x + kt;
  if (threadIdx.x == 0) cls[tile] = any_cta ? (all_cta ? 1 : 2) : 0;
  if (bits != nullptr && any_cta && !all_cta) {
    uint32_t* dst = bits + tile * (kTile * kTile / 32);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      uint32_t v = 0u;
#pragma unroll
      for (int e = 0; e < 4; ++e) v |= nonzero_bits(w[i][e]) << (4 * e);
      v |= __shfl_down_sync(0xFFFFFFFFu, v, 1) << 16;
      if ((part & 1) == 0) dst[(r0 + 32 * i) * 4 + (part >> 1)] = v;
    }
  }
}

}  // namespace

cudaError_t launch_mask_classify(const uint8_t* mask, uint8_t* cls, uint32_t* bits, int* counter, int batch, int seq_q,
                                 int seq_k, cudaStream_t stream) {
  LaunchAttrs at(stream);
  at.cfg.gridDim = dim3((seq_k + kTile - 1) / kTile, (seq_q + kTile - 1) / kTile, batch);
  at.cfg.blockDim = dim3(256);
  return cudaLaunchKernelEx(&at.cfg, mask_classify_kernel, mask, cls, bits, counter, seq_q, seq_k);
}

}  // namespace minfer_attn

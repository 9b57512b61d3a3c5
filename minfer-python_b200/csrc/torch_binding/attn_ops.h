// The attention ops between a tensor type and the C ABI: argument checks and parameter blocks.
//
// One definition for the two ways a call arrives: through torch's dispatcher, with tensors of LibTorch's stable ABI
// (reg_cuda.cpp), and straight from Python (direct.cpp), with at::Tensor.  The two tensor classes share the names of the
// accessors used here; Env supplies what they do not: streams, buffers, how the library is called.
//
// Counterpart of the reference's launcher src/minfer/kernels/torch_ext/csrc/cuda/flash_attn/op.cuh:21-106: the same
// checks in the same order (devices, innermost stride 1 and k/v sharing strides, dtypes, ranks, shapes), the QKVStrides
// capture (:80-83), the current stream of the current device (:98-103) - and then, where the reference stops at
// "TODO: implement", one call into the C ABI of libminfer_attn.so.  Relaxed against the reference only as the benchmark
// configurations demand: bfloat16 next to float16, head_dim 64 next to 128 (both enforced by the library, not here).
#pragma once

#include <torch/headeronly/core/ScalarType.h>
#include <torch/headeronly/macros/Macros.h>
#include <torch/headeronly/util/Exception.h>

#include <cstddef>
#include <cstdint>
#include <string>

#include "../../../include/minfer_attn.h"

namespace minfer {

struct Scratch {
  void* ptr;
  size_t bytes;
};

template <class Env>
struct AttnOps {
  using T = typename Env::Tensor;
  using ScalarType = torch::headeronly::ScalarType;
  static int device_of(const T& t) { return Env::device_of(t); }

  // Scratch of a dense-mask call: with the tiles' bits (an eighth of the mask's bytes) while that is no more than 256 MB,
  // as for masks up to 2 GB, and the device has room for it; otherwise the tile classes alone.
  static size_t mask_workspace_bytes(int32_t batch, int32_t seq_q, int32_t seq_k) {
    const size_t with_bits = minfer_attn_prefill_workspace_bytes_bits(batch, seq_q, seq_k);
    return with_bits <= (size_t{256} << 20) ? with_bits : minfer_attn_prefill_workspace_bytes(batch, seq_q, seq_k);
  }

  static int dtype_tag(const T& t) {
    const auto st = t.scalar_type();
    STD_TORCH_CHECK(st == ScalarType::Half || st == ScalarType::BFloat16, "minfer attention: float16 or bfloat16 tensors expected");
    return st == ScalarType::Half ? MINFER_ATTN_F16 : MINFER_ATTN_BF16;
  }

  static void check_rc(int rc, const char* what) {
    if (rc == MINFER_ATTN_OK) return;
    std::string msg = std::string(what) + ": " + minfer_attn_strerror(rc);
    if (rc == MINFER_ATTN_ECUDA) msg += std::string(" [") + minfer_attn_last_cuda_error() + "]";
    STD_TORCH_CHECK(false, msg);
  }

  // GGML Q8_0 cache: uint8 [B, Hkv, Lmax, head_dim / 32 * 34], rows of one head contiguous
  static void check_q8_cache(const T& cache, int64_t batch, int64_t head_dim, const char* what) {
    STD_TORCH_CHECK(cache.is_cuda() && cache.scalar_type() == ScalarType::Byte && cache.dim() == 4,
                    std::string(what) + " must be a CUDA uint8 [B, Hkv, Lmax, bytes] tensor");
    STD_TORCH_CHECK(cache.size(0) == batch && cache.size(3) == head_dim / 32 * 34,
                    std::string(what) + ": batch or row bytes do not match (row = head_dim/32 blocks of 34 bytes)");
    STD_TORCH_CHECK(cache.stride(3) == 1 && cache.stride(2) == cache.size(3), std::string(what) + ": rows of one head must be contiguous");
    // rows of one (batch, head) must end on a 16-byte boundary
    STD_TORCH_CHECK(cache.size(2) % (head_dim == 64 ? 4 : 2) == 0, std::string(what) + ": the padded length must be a multiple of 2 (4 for head_dim 64)");
  }

  static void check_qkv(const T& q, const T& k, const T& v, const T& out) {
    STD_TORCH_CHECK(q.is_cuda() && k.is_cuda() && v.is_cuda() && out.is_cuda(), "all tensors must be on CUDA");
    STD_TORCH_CHECK(device_of(q) == device_of(k) && device_of(q) == device_of(v) &&
                    device_of(q) == device_of(out), "tensors on different devices");
    STD_TORCH_CHECK(q.dim() == 4 && k.dim() == 4 && v.dim() == 4 && out.dim() == 4, "tensors must be 4-D");
    STD_TORCH_CHECK(q.stride(-1) == 1 && k.stride(-1) == 1 && v.stride(-1) == 1 && out.stride(-1) == 1 &&
                    k.stride(0) == v.stride(0) && k.stride(1) == v.stride(1) && k.stride(2) == v.stride(2),
                    "innermost stride must be 1 and k, v must share strides");
    STD_TORCH_CHECK(q.scalar_type() == k.scalar_type() && q.scalar_type() == v.scalar_type() &&
                    q.scalar_type() == out.scalar_type(), "q, k, v, out must share one dtype");
    STD_TORCH_CHECK(q.sizes().equals(out.sizes()), "q and out shapes differ");
    STD_TORCH_CHECK(k.sizes().equals(v.sizes()), "k and v shapes differ");
    STD_TORCH_CHECK(q.size(0) == k.size(0) && q.size(3) == k.size(3), "batch or head_dim mismatch");
    STD_TORCH_CHECK(q.size(1) % k.size(1) == 0, "n_heads must be a multiple of n_kv_heads");
  }

  static void prefill(const T& q, const T& k, const T& v, const T* mask, T& out, bool causal) {
    MinferAttnPrefillParams p{};
    p.q = q.const_data_ptr();
    p.k = k.const_data_ptr();
    p.v = v.const_data_ptr();
    p.out = out.mutable_data_ptr();
    p.mask = mask != nullptr ? static_cast<const uint8_t*>(mask->const_data_ptr()) : nullptr;
    p.status = Env::status(q);
    for (int i = 0; i < 3; ++i) {
      p.q_stride[i] = q.stride(i);
      p.kv_stride[i] = k.stride(i);
      p.out_stride[i] = out.stride(i);
    }
    p.batch = static_cast<int32_t>(q.size(0));
    p.n_heads = static_cast<int32_t>(q.size(1));
    p.n_kv_heads = static_cast<int32_t>(k.size(1));
    p.seq_q = static_cast<int32_t>(q.size(2));
    p.seq_k = static_cast<int32_t>(k.size(2));
    p.head_dim = static_cast<int32_t>(q.size(3));
    p.dtype = dtype_tag(q);
    p.causal = causal ? 1 : 0;
    p.max_ctas = Env::max_ctas();
    void* stream = Env::stream(q);
    const size_t least = mask != nullptr ? minfer_attn_prefill_workspace_bytes(p.batch, p.seq_q, p.seq_k) : 16;
    const size_t want = mask != nullptr ? mask_workspace_bytes(p.batch, p.seq_q, p.seq_k) : least;
    const Scratch ws = Env::scratch(q, stream, /*purpose=*/0, want, least);
    p.workspace = ws.ptr;
    p.workspace_bytes = ws.bytes;
    check_rc(Env::call(minfer_attn_prefill, &p, stream), "minfer_attn_prefill");
  }

  static void decode(const T& q, const T& kc, const T& vc, const T* table, const T& lens, T& out,
              int kv_format) {
    STD_TORCH_CHECK(lens.is_cuda() && device_of(lens) == device_of(q), "lens must be on the same CUDA device");
    STD_TORCH_CHECK(lens.scalar_type() == ScalarType::Int && lens.dim() == 1 && lens.is_contiguous(),
                    "lens must be a contiguous int32 vector");
    STD_TORCH_CHECK(lens.numel() == q.size(0), "lens must have one entry per sequence");
    STD_TORCH_CHECK(q.size(2) == 1, "decode takes one query token per sequence");
    MinferAttnDecodeParams p{};
    p.q = q.const_data_ptr();
    p.k_cache = kc.const_data_ptr();
    p.v_cache = vc.const_data_ptr();
    p.lens = static_cast<const int32_t*>(lens.const_data_ptr());
    p.out = out.mutable_data_ptr();
    p.batch = static_cast<int32_t>(q.size(0));
    p.n_heads = static_cast<int32_t>(q.size(1));
    p.n_kv_heads = static_cast<int32_t>(kc.size(1));
    p.max_len = static_cast<int32_t>(kc.size(2));
    p.head_dim = static_cast<int32_t>(q.size(3));
    if (table != nullptr) {
      p.block_table = static_cast<const int32_t*>(table->const_data_ptr());
      p.page_size = static_cast<int32_t>(kc.size(2));
      p.table_stride = static_cast<int32_t>(table->size(1));
      p.max_len = p.page_size * p.table_stride;
      p.n_pages = static_cast<int32_t>(kc.size(0));
    }
    p.status = Env::status(q);
    p.dtype = dtype_tag(q);
    p.kv_format = kv_format;
    for (int i = 0; i < 2; ++i) {
      p.q_stride[i] = q.stride(i);
      p.out_stride[i] = out.stride(i);
    }
    for (int i = 0; i < 3; ++i) p.kv_stride[i] = kc.stride(i);
    void* stream = Env::stream(q);
    const size_t need = minfer_attn_decode_workspace_bytes(p.batch, p.n_heads, p.max_len, p.head_dim, 0);
    const Scratch ws = Env::scratch(q, stream, /*purpose=*/1, need, need);
    p.workspace = ws.ptr;
    p.workspace_bytes = ws.bytes;
    check_rc(Env::call(minfer_attn_decode, &p, stream), "minfer_attn_decode");
  }

  static void flash_attn(int64_t qtype_int, int64_t qblock_size, int64_t qtype_size,
                       const T& q,  // [B, n_heads, L, head_dim]
                       const T& k,  // [B, n_kv_heads, L, head_dim]
                       const T& v,  // [B, n_kv_heads, L, head_dim]
                       T& mask,     // [B, 1, L, L] bool, contiguous
                       T& out) {    // [B, n_heads, L, head_dim]
    (void)qtype_int;
    (void)qblock_size;
    (void)qtype_size;
    check_qkv(q, k, v, out);
    STD_TORCH_CHECK(mask.is_cuda() && device_of(mask) == device_of(q), "mask must be on the same CUDA device");
    STD_TORCH_CHECK(mask.scalar_type() == ScalarType::Bool, "mask must be bool");
    STD_TORCH_CHECK(mask.dim() == 4 && mask.is_contiguous(), "mask must be a contiguous 4-D tensor");
    STD_TORCH_CHECK(q.size(2) == k.size(2), "flash_attn requires seq_q == seq_k");
    STD_TORCH_CHECK(mask.size(0) == q.size(0) && mask.size(1) == 1 && mask.size(2) == q.size(2) && mask.size(3) == k.size(2),
                    "mask must be [B, 1, L, L]");
    prefill(q, k, v, &mask, out, /*causal=*/false);
  }

  static void flash_attn_causal(const T& q, const T& k, const T& v, T& out) {
    check_qkv(q, k, v, out);
    STD_TORCH_CHECK(k.size(2) >= q.size(2), "causal attention requires seq_k >= seq_q");
    prefill(q, k, v, nullptr, out, /*causal=*/true);
  }

  static void flash_attn_decode(const T& q, const T& k_cache, const T& v_cache, const T& lens, T& out) {
    check_qkv(q, k_cache, v_cache, out);
    decode(q, k_cache, v_cache, nullptr, lens, out, MINFER_ATTN_KV_16BIT);
  }

  static void flash_attn_decode_paged(const T& q, const T& k_pages, const T& v_pages, const T& block_table,
                                    const T& lens, T& out) {
    STD_TORCH_CHECK(q.is_cuda() && out.is_cuda() && q.dim() == 4 && out.dim() == 4 && q.sizes().equals(out.sizes()),
                    "q/out must be CUDA [B, H, 1, D] tensors");
    STD_TORCH_CHECK(out.scalar_type() == q.scalar_type(), "q/out must share one dtype");
    STD_TORCH_CHECK(k_pages.is_cuda() && v_pages.is_cuda() && k_pages.dim() == 4 && v_pages.dim() == 4,
                    "the page pools must be CUDA [n_pages, n_kv_heads, page_size, D] tensors");
    STD_TORCH_CHECK(k_pages.scalar_type() == q.scalar_type() && v_pages.scalar_type() == q.scalar_type(),
                    "the page pools must have q's dtype");
    STD_TORCH_CHECK(k_pages.sizes().equals(v_pages.sizes()) && k_pages.strides().equals(v_pages.strides()),
                    "the page pools must share shape and strides");
    STD_TORCH_CHECK(k_pages.size(3) == q.size(3) && k_pages.stride(-1) == 1 && q.stride(-1) == 1 && out.stride(-1) == 1,
                    "head_dim mismatch or innermost stride not 1");
    STD_TORCH_CHECK(k_pages.size(2) % 16 == 0, "page_size must be a multiple of 16");
    STD_TORCH_CHECK(q.size(1) % k_pages.size(1) == 0, "n_heads must be a multiple of n_kv_heads");
    STD_TORCH_CHECK(block_table.is_cuda() && block_table.scalar_type() == ScalarType::Int && block_table.dim() == 2 &&
                    block_table.is_contiguous() && block_table.size(0) == q.size(0),
                    "block_table must be a contiguous CUDA int32 [B, max_pages] tensor");
    decode(q, k_pages, v_pages, &block_table, lens, out, MINFER_ATTN_KV_16BIT);
  }

  static void flash_attn_decode_q8(const T& q, const T& k_cache, const T& v_cache, const T& lens, T& out) {
    STD_TORCH_CHECK(q.is_cuda() && out.is_cuda() && q.dim() == 4 && out.dim() == 4 && q.sizes().equals(out.sizes()),
                    "q/out must be CUDA [B, H, 1, D] tensors");
    STD_TORCH_CHECK(q.scalar_type() == out.scalar_type() && q.stride(-1) == 1 && out.stride(-1) == 1, "q/out dtype or innermost stride");
    check_q8_cache(k_cache, q.size(0), q.size(3), "k_cache");
    check_q8_cache(v_cache, q.size(0), q.size(3), "v_cache");
    STD_TORCH_CHECK(k_cache.sizes().equals(v_cache.sizes()) && k_cache.strides().equals(v_cache.strides()),
                    "the caches must share shape and strides");
    STD_TORCH_CHECK(q.size(1) % k_cache.size(1) == 0, "n_heads must be a multiple of n_kv_heads");
    decode(q, k_cache, v_cache, nullptr, lens, out, MINFER_ATTN_KV_Q8_0);
  }

  // ---- rotary embedding (+ KV-cache append): minfer_attn_rope_append ----
  static void rope_in_place(int style, int64_t rotary_dim, int64_t start_pos, double freq_base, T& x) {
    // the checks of the reference's launcher (csrc/cuda/il_rope/op.cuh:27-31), bfloat16 admitted
    STD_TORCH_CHECK(x.is_cuda(), "x must be on CUDA");
    STD_TORCH_CHECK(x.is_contiguous(), "x must be contiguous");
    STD_TORCH_CHECK(x.dim() == 4, "x must be [B, L, n_heads, head_dim]");
    STD_TORCH_CHECK(rotary_dim <= x.size(3), "rotary_dim exceeds head_dim");
    MinferRopeParams p{};
    p.q = x.mutable_data_ptr();
    for (int i = 0; i < 3; ++i) p.q_stride[i] = x.stride(i);
    p.batch = static_cast<int32_t>(x.size(0));
    p.seq = static_cast<int32_t>(x.size(1));
    p.n_heads = static_cast<int32_t>(x.size(2));
    p.head_dim = static_cast<int32_t>(x.size(3));
    p.rotary_dim = static_cast<int32_t>(rotary_dim);
    p.start_pos = static_cast<int32_t>(start_pos);
    p.freq_base = static_cast<float>(freq_base);
    p.dtype = dtype_tag(x);
    p.style = style;
    check_rc(Env::call(minfer_attn_rope_append, &p, Env::stream(x)), "minfer_attn_rope_append");
  }

  static void il_rope(int64_t rotary_dim, int64_t start_pos, double freq_base, T& x) {
    rope_in_place(0, rotary_dim, start_pos, freq_base, x);
  }

  static void neox_rope(int64_t rotary_dim, int64_t start_pos, double freq_base, T& x) {
    rope_in_place(1, rotary_dim, start_pos, freq_base, x);
  }

  static void rope_append(int64_t rotary_dim, double freq_base, int64_t style, T& q, const T& k, const T& v,
                   T& k_cache, T& v_cache, const T* table, const T& start, bool q8) {
    STD_TORCH_CHECK(q.is_cuda() && k.is_cuda() && v.is_cuda() && k_cache.is_cuda() && v_cache.is_cuda() && start.is_cuda(),
                    "all tensors must be on CUDA");
    STD_TORCH_CHECK(q.dim() == 4 && k.dim() == 4 && v.dim() == 4 && k_cache.dim() == 4 && v_cache.dim() == 4,
                    "q/k/v must be [B, L, H, D] and the caches [B, Hkv, Lmax, D]");
    if (q8) {
      STD_TORCH_CHECK(q.scalar_type() == k.scalar_type() && q.scalar_type() == v.scalar_type(), "dtypes differ");
      check_q8_cache(k_cache, q.size(0), q.size(3), "k_cache");
      check_q8_cache(v_cache, q.size(0), q.size(3), "v_cache");
    } else {
      STD_TORCH_CHECK(q.scalar_type() == k.scalar_type() && q.scalar_type() == v.scalar_type() &&
                      q.scalar_type() == k_cache.scalar_type() && q.scalar_type() == v_cache.scalar_type(), "dtypes differ");
    }
    STD_TORCH_CHECK(k.sizes().equals(v.sizes()) && k.strides().equals(v.strides()), "k and v must share shape and strides");
    STD_TORCH_CHECK(k_cache.sizes().equals(v_cache.sizes()) && k_cache.strides().equals(v_cache.strides()),
                    "the caches must share shape and strides");
    STD_TORCH_CHECK(q.size(0) == k.size(0) && (table != nullptr || k.size(0) == k_cache.size(0)) && q.size(1) == k.size(1),
                    "batch / seq mismatch");
    STD_TORCH_CHECK(k.size(2) == k_cache.size(1) && q.size(3) == k.size(3), "head count / head_dim mismatch");
    STD_TORCH_CHECK(q8 || k.size(3) == k_cache.size(3), "head_dim mismatch");
    STD_TORCH_CHECK(q.stride(-1) == 1 && k.stride(-1) == 1 && k_cache.stride(-1) == 1, "innermost stride must be 1");
    STD_TORCH_CHECK(start.scalar_type() == ScalarType::Int && start.dim() == 1 && start.numel() == q.size(0) && start.is_contiguous(),
                    "start must be a contiguous int32 vector with one entry per sequence");
    MinferRopeParams p{};
    p.q = q.mutable_data_ptr();
    p.k = k.const_data_ptr();
    p.v = v.const_data_ptr();
    p.k_cache = k_cache.mutable_data_ptr();
    p.v_cache = v_cache.mutable_data_ptr();
    p.start = static_cast<const int32_t*>(start.const_data_ptr());
    for (int i = 0; i < 3; ++i) {
      p.q_stride[i] = q.stride(i);
      p.kv_stride[i] = k.stride(i);
      p.cache_stride[i] = k_cache.stride(i);
    }
    p.batch = static_cast<int32_t>(q.size(0));
    p.seq = static_cast<int32_t>(q.size(1));
    p.n_heads = static_cast<int32_t>(q.size(2));
    p.n_kv_heads = static_cast<int32_t>(k.size(2));
    p.head_dim = static_cast<int32_t>(q.size(3));
    p.rotary_dim = static_cast<int32_t>(rotary_dim);
    p.max_len = static_cast<int32_t>(k_cache.size(2));
    p.freq_base = static_cast<float>(freq_base);
    if (table != nullptr) {
      STD_TORCH_CHECK(table->is_cuda() && table->scalar_type() == ScalarType::Int && table->dim() == 2 && table->is_contiguous() &&
                      table->size(0) == q.size(0), "block_table must be a contiguous CUDA int32 [B, max_pages] tensor");
      p.block_table = static_cast<const int32_t*>(table->const_data_ptr());
      p.page_size = static_cast<int32_t>(k_cache.size(2));
      p.table_stride = static_cast<int32_t>(table->size(1));
      p.max_len = p.page_size * p.table_stride;
      p.n_pages = static_cast<int32_t>(k_cache.size(0));
    }
    p.status = Env::status(q);
    p.dtype = dtype_tag(q);
    p.style = static_cast<int32_t>(style);
    p.cache_format = q8 ? MINFER_ATTN_KV_Q8_0 : MINFER_ATTN_KV_16BIT;
    check_rc(Env::call(minfer_attn_rope_append, &p, Env::stream(q)), "minfer_attn_rope_append");
  }

  static void rope_kv_append(int64_t rotary_dim, double freq_base, int64_t style, T& q, const T& k, const T& v,
                           T& k_cache, T& v_cache, const T& start) {
    rope_append(rotary_dim, freq_base, style, q, k, v, k_cache, v_cache, nullptr, start, false);
  }

  static void rope_kv_append_q8(int64_t rotary_dim, double freq_base, int64_t style, T& q, const T& k, const T& v,
                              T& k_cache, T& v_cache, const T& start) {
    rope_append(rotary_dim, freq_base, style, q, k, v, k_cache, v_cache, nullptr, start, true);
  }

  static void rope_kv_append_paged(int64_t rotary_dim, double freq_base, int64_t style, T& q, const T& k, const T& v,
                                 T& k_pages, T& v_pages, const T& block_table, const T& start) {
    rope_append(rotary_dim, freq_base, style, q, k, v, k_pages, v_pages, &block_table, start, false);
  }
};

}  // namespace minfer

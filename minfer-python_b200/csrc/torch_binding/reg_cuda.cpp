// CUDA implementations of the attention ops, bound through LibTorch's stable ABI.
//
// Counterpart of the reference's src/minfer/kernels/torch_ext/csrc/cuda/reg.cu:16-27
// (STABLE_TORCH_LIBRARY_IMPL(minfer, CUDA, m) + TORCH_BOX(&flash_attn_cuda)).  The checks and the parameter blocks are
// in attn_ops.h; this unit supplies the current stream from the shim, the buffers this layer owns, and the registration.
//
// No device code lives in this unit; it is compiled by the host compiler.
#include <torch/csrc/stable/accelerator.h>
#include <torch/csrc/stable/library.h>
#include <torch/csrc/stable/ops.h>
#include <torch/csrc/stable/tensor.h>
#include <torch/csrc/stable/macros.h>

#include <torch/csrc/stable/c/shim.h>

#include <array>
#include <exception>
#include <map>
#include <memory>
#include <mutex>
#include <utility>

#include "attn_ops.h"
#include "buffers.h"

namespace minfer {

using torch::headeronly::DeviceType;
using torch::headeronly::ScalarType;
using torch::stable::Tensor;

namespace {

void* current_stream() {
  auto device_index = torch::stable::accelerator::getCurrentDeviceIndex();
  void* stream_ptr = nullptr;
  TORCH_ERROR_CODE_CHECK(aoti_torch_get_current_cuda_stream(device_index, &stream_ptr));
  return stream_ptr;
}

// Device buffers this layer owns (the library itself allocates nothing): one status word per
// device, one scratch buffer per (device, stream, purpose), grown on demand through torch's
// allocator and kept for the life of the process.
// g_mu guards the maps only and is never held while torch allocates: the allocator may want the interpreter's lock (it
// records Python stacks when asked to), and the direct entry points come here with that lock held.
std::mutex g_mu;
std::map<int, Tensor*> g_status;
struct ScratchSlot {
  Tensor* buffer = nullptr;
  size_t refused = 0;  // the smallest size beyond `least` that could not be had, 0: none
  int passed_over = 0;  // calls since then that did without
};
std::map<std::array<int64_t, 3>, ScratchSlot> g_scratch;
int g_max_ctas = 0;

Tensor& status_word(const Tensor& like) {
  const int dev = like.get_device_index();
  {
    std::lock_guard<std::mutex> lock(g_mu);
    auto it = g_status.find(dev);
    if (it != g_status.end()) return *it->second;
  }
  const int64_t n[1] = {4};
  auto mine = std::make_unique<Tensor>(torch::stable::new_zeros(like, {n, 1}, ScalarType::Int));
  std::lock_guard<std::mutex> lock(g_mu);
  Tensor*& kept = g_status[dev];  // another thread's, if it was quicker
  if (kept == nullptr) kept = mine.release();
  return *kept;
}

bool fits(const ScratchSlot& slot, size_t bytes) {
  return slot.buffer != nullptr && static_cast<size_t>(slot.buffer->numel()) >= bytes;
}

Tensor& grow_scratch(const Tensor& like, const std::array<int64_t, 3>& key, size_t bytes) {
  // powers of two, so that the outgrown buffers of a slowly growing series of calls add up to less than the last one
  int64_t n[1] = {1 << 20};
  while (static_cast<size_t>(n[0]) < bytes) n[0] *= 2;
  auto mine = std::make_unique<Tensor>(torch::stable::new_empty(like, {n, 1}, ScalarType::Byte));
  std::lock_guard<std::mutex> lock(g_mu);
  ScratchSlot& slot = g_scratch[key];
  if (!fits(slot, bytes)) slot.buffer = mine.release();  // an outgrown buffer stays alive: launches in flight may still use it
  return *slot.buffer;
}

// At least `least` bytes, and `want` where the device has them.  A refused allocation is costly (torch gives its cached
// blocks back and tries again), so on a full device the larger size is asked for once in 256 calls only.
Tensor& scratch(const Tensor& like, void* stream, int64_t purpose, size_t want, size_t least) {
  const std::array<int64_t, 3> key = {like.get_device_index(), reinterpret_cast<int64_t>(stream), purpose};
  {
    std::lock_guard<std::mutex> lock(g_mu);
    ScratchSlot& slot = g_scratch[key];
    if (fits(slot, want)) return *slot.buffer;
    if (least < want && slot.refused != 0 && want >= slot.refused && ++slot.passed_over % 256 != 0) {
      if (fits(slot, least)) return *slot.buffer;
      want = least;
    }
  }
  if (least < want) {
    try {
      return grow_scratch(like, key, want);
    } catch (const std::exception&) {
      std::lock_guard<std::mutex> lock(g_mu);
      ScratchSlot& slot = g_scratch[key];
      if (slot.refused == 0 || want < slot.refused) slot.refused = want;
      if (fits(slot, least)) return *slot.buffer;
    }
  }
  return grow_scratch(like, key, least);
}

struct StableEnv {
  using Tensor = torch::stable::Tensor;
  static int device_of(const Tensor& t) { return t.get_device_index(); }
  static void* stream(const Tensor&) { return current_stream(); }
  static int32_t* status(const Tensor& like) { return static_cast<int32_t*>(status_word(like).mutable_data_ptr()); }
  static Scratch scratch(const Tensor& like, void* stream, int64_t purpose, size_t want, size_t least) {
    Tensor& t = minfer::scratch(like, stream, purpose, want, least);
    return {t.mutable_data_ptr(), static_cast<size_t>(t.numel())};
  }
  static int max_ctas() { return g_max_ctas; }
  template <class P>
  static int call(int (*fn)(const P*, void*), const P* p, void* stream) { return fn(p, stream); }
};
using Ops = AttnOps<StableEnv>;

Tensor borrowed(void* at_tensor) {  // a stable tensor sharing the at::Tensor behind the pointer
  AtenTensorHandle h = nullptr;
  TORCH_ERROR_CODE_CHECK(aoti_torch_new_tensor_handle(reinterpret_cast<AtenTensorHandle>(at_tensor), &h));
  return Tensor(h);
}

}  // namespace

// the buffers, for the direct entry points (buffers.h)
int32_t* binding_status(void* like) { return StableEnv::status(borrowed(like)); }
Scratch binding_scratch(void* like, void* stream, int64_t purpose, size_t want, size_t least) {
  return StableEnv::scratch(borrowed(like), stream, purpose, want, least);
}
int binding_max_ctas() { return g_max_ctas; }

Tensor attn_status_word_cuda(const Tensor& like) { return status_word(like); }

void attn_set_prefill_cta_limit_cuda(const Tensor& like, int64_t max_ctas) {
  (void)like;
  STD_TORCH_CHECK(max_ctas >= 0, "max_ctas must be >= 0");
  g_max_ctas = static_cast<int>(max_ctas);
}

STABLE_TORCH_LIBRARY_IMPL(minfer, CUDA, m) {
  m.impl("flash_attn", TORCH_BOX(&Ops::flash_attn));
  m.impl("flash_attn_causal", TORCH_BOX(&Ops::flash_attn_causal));
  m.impl("flash_attn_decode", TORCH_BOX(&Ops::flash_attn_decode));
  m.impl("flash_attn_decode_paged", TORCH_BOX(&Ops::flash_attn_decode_paged));
  m.impl("flash_attn_decode_q8", TORCH_BOX(&Ops::flash_attn_decode_q8));
  m.impl("il_rope", TORCH_BOX(&Ops::il_rope));
  m.impl("neox_rope", TORCH_BOX(&Ops::neox_rope));
  m.impl("rope_kv_append", TORCH_BOX(&Ops::rope_kv_append));
  m.impl("rope_kv_append_q8", TORCH_BOX(&Ops::rope_kv_append_q8));
  m.impl("rope_kv_append_paged", TORCH_BOX(&Ops::rope_kv_append_paged));
  m.impl("attn_status_word", TORCH_BOX(&attn_status_word_cuda));
  m.impl("attn_set_prefill_cta_limit", TORCH_BOX(&attn_set_prefill_cta_limit_cuda));
}

}  // namespace minfer

// What the two binding libraries share: the device buffers this layer owns (the kernel library allocates nothing) live in
// _C and are handed to the direct entry points by pointer.  `like` points to an at::Tensor on the device in question.
#pragma once

#include <cstddef>
#include <cstdint>

#include "attn_ops.h"

namespace minfer {

int32_t* binding_status(void* like);                                              // the device's status word
// `want` bytes where the device has them, `least` in any case; never moves while the process lives
Scratch binding_scratch(void* like, void* stream, int64_t purpose, size_t want, size_t least);
int binding_max_ctas();

}  // namespace minfer

// Operands of kernels that read 16 bytes at a time.
#pragma once
#include <ATen/ATen.h>
#include <stdint.h>

namespace uttt {

// `t` contiguous and on a 16-byte boundary.  contiguous() by itself hands out a contiguous view as it is, also one at an
// odd offset (a narrow of a flat buffer, as the backward of a concatenation gives), and a vector load from it faults.
inline at::Tensor dense16(const at::Tensor& t) {
  at::Tensor c = t.contiguous();
  return (reinterpret_cast<uintptr_t>(c.data_ptr()) & 15) == 0 ? c : c.clone();
}

}  // namespace uttt

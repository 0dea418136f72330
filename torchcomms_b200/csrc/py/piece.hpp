// Small tensors cut from one allocation.
#pragma once

#include <ATen/ATen.h>
#include <c10/core/TensorImpl.h>

namespace b200c {

// A tensor over `sizes` elements from byte `byte` of a CUDA storage, which lives as long as one of its pieces. Not a view:
// it has a version counter of its own. Pieces of one storage are of one type (torch.save refuses to write a storage that
// is seen as two).
inline at::Tensor piece(const c10::Storage& storage, int64_t byte, at::IntArrayRef sizes, at::ScalarType type) {
  at::Tensor t = at::detail::make_tensor<c10::TensorImpl>(c10::Storage(storage), c10::DispatchKeySet(c10::DispatchKey::CUDA),
                                                          c10::scalarTypeToTypeMeta(type));
  t.unsafeGetTensorImpl()->set_storage_offset(byte / static_cast<int64_t>(c10::elementSize(type)));
  t.unsafeGetTensorImpl()->set_sizes_contiguous(sizes);
  return t;
}

} // namespace b200c

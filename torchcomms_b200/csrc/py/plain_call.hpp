// Whether a tensor-level call may go straight to a kernel: nothing that works
// through PyTorch's dispatcher (autograd, forward-mode, functorch transforms,
// dispatch and function modes, tracing, lazy conjugation) wants to see it.
#pragma once

#include <ATen/ATen.h>
#include <ATen/PythonTorchFunctionTLS.h>
#include <c10/core/DispatchKeySet.h>
#include <c10/core/GradMode.h>
#include <c10/core/impl/LocalDispatchKeySet.h>

namespace b200c {

// `grad_ok`: the caller records the operation with autograd itself.
inline bool plain_call(const at::Tensor& t, bool grad_ok = false) {
  using K = c10::DispatchKey;
  constexpr c10::DispatchKeySet watched({K::Python, K::PythonTLSSnapshot, K::FuncTorchDynamicLayerFrontMode,
                                         K::FuncTorchDynamicLayerBackMode, K::FuncTorchGradWrapper, K::FuncTorchBatched,
                                         K::FuncTorchVmapMode, K::Batched, K::VmapMode, K::Functionalize, K::Tracer,
                                         K::Conjugate, K::Negative, K::ZeroTensor});
  if (!t.defined() || !t.is_cuda() || t.layout() != at::kStrided || !t.has_storage()) return false;
  if (t.key_set().has_any(watched) || c10::impl::tls_local_dispatch_key_set().included_.has_any(watched)) return false;
  if (at::impl::torch_function_mode_enabled()) return false;
  if (t._fw_grad(/*level=*/0).defined()) return false;
  return grad_ok || !(c10::GradMode::is_enabled() && t.requires_grad());
}

} // namespace b200c

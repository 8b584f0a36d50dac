// The operators of torch.ops.matgptq_cuda and the host path of MatGPTQLinear, in C++.
//
// Same names, schemas, checks and messages as the reference's binding (csrc/bindings.cpp:43-191,197-207 and
// inference_lib/matgptq_cuda/__init__.py:5-63); the work is done by libmatgptq_b200.so through its C ABI, whose
// entry points are looked up at run time (bind()), so that this file and the kernels are built apart.
//
// What bounds a call with few rows is not the GPU but the host: registered from Python the operator took 45 us a call
// (argument parsing, two Python frames of torch.library, checks, a context manager, ctypes) in front of 4 to 12 us of
// kernel.  Here a call is parsed once, checked, allocates its result and launches; linear_forward() also leaves out the
// dispatcher when nothing that listens to it is active (no dispatch or function mode, no functorch level) and the tensors
// are ordinary CUDA tensors, which is what an eager MatGPTQLinear needs.
#include <ATen/EmptyTensor.h>
#include <ATen/cuda/EmptyTensor.h>
#include <ATen/ops/empty_like.h>
#include <ATen/record_function.h>
#include <c10/core/impl/LocalDispatchKeySet.h>
#include <c10/core/impl/PythonDispatcherTLS.h>
#include <c10/core/impl/TorchDispatchModeTLS.h>
#include <ATen/PythonTorchFunctionTLS.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <dlfcn.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/VariableTypeUtils.h>
#include <torch/csrc/autograd/functions/basic_ops.h>
#include <torch/csrc/autograd/functions/utils.h>
#include <torch/csrc/autograd/python_variable.h>
#include <torch/library.h>

#include "../../include/matgptq_b200.h"

namespace {

using at::Tensor;

struct Library {
  decltype(&matgptq_b200_strerror) strerror = nullptr;
  decltype(&matgptq_b200_matmul_ws) matmul_ws = nullptr;
  decltype(&matgptq_b200_matmul_zp) matmul_zp = nullptr;
  decltype(&matgptq_b200_matmul_grouped) matmul_grouped = nullptr;
  decltype(&matgptq_b200_matmul_workspace_bytes) workspace_bytes = nullptr;
  decltype(&matgptq_b200_pack_qweights) pack_qweights = nullptr;
  decltype(&matgptq_b200_reorder_scales) reorder_scales = nullptr;
  decltype(&matgptq_b200_dequantize) dequantize = nullptr;
};
Library lib;  // filled once by bind() when the package is imported

void check_status(int status, const char *what) {
  TORCH_CHECK(status == MATGPTQ_B200_OK, what, ": ", lib.strerror(status), " (status ", status, ")");
}

void check_common(int64_t bitwidth, int64_t group_size, int64_t n_in) {  // csrc/bindings.cpp:55-59
  TORCH_CHECK(bitwidth == 2 || bitwidth == 3 || bitwidth == 4 || bitwidth == 6 || bitwidth == 8,
              "bitwidth must be one of {2, 3, 4, 6, 8}");
  TORCH_CHECK(group_size == -1 || group_size == 32 || group_size == 128, "group_size must be one of {-1, 32, 128}");
  TORCH_CHECK(group_size == -1 || n_in % group_size == 0, "group_size must divide n_in_features. Got group_size=", group_size,
              ", n_in_features=", n_in);
}

c10::Device cuda_device_of(const Tensor &t) {
  if (t.is_cuda()) return t.device();
  TORCH_CHECK(c10::cuda::device_count() > 0,
              "matgptq_b200 needs a CUDA device: there is no CPU implementation of this operator");
  return c10::Device(c10::kCUDA, c10::cuda::current_device());
}

void *stream_of(c10::Device dev) { return c10::cuda::getCurrentCUDAStream(dev.index()).stream(); }

Tensor empty_on(at::IntArrayRef sizes, at::ScalarType dtype, c10::Device dev) {
  return at::detail::empty_cuda(sizes, dtype, dev, std::nullopt);
}

at::ScalarType type_of(int64_t flags) { return (flags & MATGPTQ_B200_FLAG_BF16) ? at::kBFloat16 : at::kHalf; }
const char *type_name(int64_t flags) { return (flags & MATGPTQ_B200_FLAG_BF16) ? "torch.bfloat16" : "torch.float16"; }

// ---- load-time operators ------------------------------------------------------------------------------------
Tensor pack_impl(const Tensor &qweights, int64_t n_out, int64_t n_in, int64_t bitwidth, int64_t group_size, int64_t master) {
  // csrc/bindings.cpp:50-59
  TORCH_CHECK(qweights.scalar_type() == at::kByte, "qweights must be uint8");
  TORCH_CHECK(qweights.is_contiguous(), "qweights must be contiguous");
  TORCH_CHECK(qweights.dim() == 2, "qweights must be 2D (n_out_features, n_in_features)");
  TORCH_CHECK(qweights.size(0) == n_out, "n_out_features does not match qweights.size(0)");
  TORCH_CHECK(qweights.size(1) == n_in, "n_in_features does not match qweights.size(1)");
  check_common(bitwidth, group_size, n_in);
  const c10::Device dev = cuda_device_of(qweights);
  const c10::cuda::CUDAGuard on_device(dev);
  const bool on_host = !qweights.is_cuda();
  const Tensor codes = on_host ? qweights.to(dev, qweights.scalar_type(), /*non_blocking=*/true) : qweights;
  Tensor packed = empty_on({bitwidth * n_out * n_in / 32}, at::kUInt32, dev);
  check_status(lib.pack_qweights(static_cast<const uint8_t *>(codes.const_data_ptr()), static_cast<uint32_t *>(packed.data_ptr()), n_out,
                                 n_in, static_cast<int>(bitwidth), static_cast<int>(master), stream_of(dev)),
               "pack_matgptq_qweights");
  if (on_host) codes.record_stream(c10::cuda::getCurrentCUDAStream(dev.index()));
  return packed;
}

Tensor pack(const Tensor &qweights, int64_t n_out, int64_t n_in, int64_t bitwidth, int64_t group_size, int64_t /*flags*/) {
  return pack_impl(qweights, n_out, n_in, bitwidth, group_size, 0);
}

Tensor slice_pack(const Tensor &qweights, int64_t n_out, int64_t n_in, int64_t master, int64_t bitwidth, int64_t group_size,
                  int64_t /*flags*/) {
  TORCH_CHECK(bitwidth <= master && master <= 8, "need bitwidth <= master_bitwidth <= 8");
  return pack_impl(qweights, n_out, n_in, bitwidth, group_size, master);
}

Tensor reorder(const Tensor &scales, int64_t m, int64_t n, int64_t group_size) {
  // csrc/bindings.cpp:92-97
  TORCH_CHECK(scales.is_contiguous(), "scales must be contiguous");
  TORCH_CHECK(scales.dim() == 2, "scales must be 2D (n_out_features, n_groups)");
  TORCH_CHECK(scales.scalar_type() == at::kHalf || scales.scalar_type() == at::kBFloat16, "scales must be float16 or bfloat16");
  check_common(8, group_size, n);
  const int64_t groups = group_size == -1 ? 1 : n / group_size;
  TORCH_CHECK(scales.size(0) == m && scales.size(1) == groups, "scales must have shape (", m, ", ", groups, ")");
  const c10::Device dev = cuda_device_of(scales);
  const c10::cuda::CUDAGuard on_device(dev);
  const bool on_host = !scales.is_cuda();
  const Tensor src = on_host ? scales.to(dev, scales.scalar_type(), /*non_blocking=*/true) : scales;
  Tensor out = at::empty_like(src);
  check_status(lib.reorder_scales(src.const_data_ptr(), out.data_ptr(), m, n, group_size, stream_of(dev)), "reorder_matgptq_scales");
  if (on_host) src.record_stream(c10::cuda::getCurrentCUDAStream(dev.index()));
  return out;
}

Tensor dequantize(const Tensor &weights, const Tensor &scales, int64_t n_out, int64_t n_in, int64_t bitwidth, int64_t group_size,
                  int64_t flags) {
  // the C ABI sees addresses only: what the kernel reads has to be on the GPU, dense and as large as the shape says
  TORCH_CHECK(weights.is_cuda(), "dequantize_matgptq: expected matgptq_weights to be a CUDA tensor");
  TORCH_CHECK(scales.is_cuda() && scales.device() == weights.device(),
              "dequantize_matgptq: expected matgptq_scales to be a CUDA tensor on the GPU of matgptq_weights");
  check_common(bitwidth, group_size, n_in);
  TORCH_CHECK(scales.scalar_type() == type_of(flags), "matgptq_scales must be ", type_name(flags), " for feature_flag=", flags);
  const int64_t groups = group_size == -1 ? 1 : n_in / group_size;
  TORCH_CHECK(weights.is_contiguous() && weights.element_size() == 4 && weights.numel() >= bitwidth * n_out * n_in / 32,
              "matgptq_weights must hold ", bitwidth * n_out * n_in / 32, " contiguous 32-bit words");
  TORCH_CHECK(scales.is_contiguous() && scales.numel() >= n_out * groups, "matgptq_scales must hold ", n_out * groups,
              " contiguous elements");
  const c10::Device dev = weights.device();
  const c10::cuda::CUDAGuard on_device(dev);
  Tensor out = empty_on({n_out, n_in}, type_of(flags), dev);
  check_status(lib.dequantize(static_cast<const uint32_t *>(weights.const_data_ptr()), scales.const_data_ptr(), nullptr, out.data_ptr(),
                              n_out, n_in, static_cast<int>(bitwidth), group_size, static_cast<uint32_t>(flags), stream_of(dev)),
               "dequantize_matgptq");
  return out;
}

// ---- products -----------------------------------------------------------------------------------------------
void check_matmul(const Tensor &input, const Tensor &weights, const Tensor &scales, int64_t n_out, int64_t n_in, int64_t bitwidth,
                  int64_t group_size) {
  // csrc/bindings.cpp:155-168
  TORCH_CHECK(input.is_cuda(), "matmul_matgptq: expected input to be a CUDA tensor");
  TORCH_CHECK(weights.is_cuda(), "matmul_matgptq: expected matgptq_weights to be a CUDA tensor");
  TORCH_CHECK(scales.is_cuda(), "matmul_matgptq: expected matgptq_scales to be a CUDA tensor");
  TORCH_CHECK(input.device() == weights.device() && input.device() == scales.device(),
              "matmul_matgptq: input, matgptq_weights and matgptq_scales must be on the same GPU");
  TORCH_CHECK(weights.scalar_type() == at::kUInt32, "matgptq_weights must be uint32");
  TORCH_CHECK(weights.is_contiguous(), "matgptq_weights must be contiguous");
  TORCH_CHECK(weights.dim() == 1, "qweights must be 1D");
  TORCH_CHECK(weights.size(0) == bitwidth * n_out * n_in / 32, "matgptq_weights has the wrong size");
  check_common(bitwidth, group_size, n_in);
  TORCH_CHECK(input.dim() >= 2 && input.size(-1) == n_in, "input must have shape [..., M, n_in_features]");
}

// the rows the operator computes: the last two dimensions (csrc/bindings.cpp:171), contiguous and 16-byte aligned
Tensor prepare_input(const Tensor &input, int64_t batch, int64_t n_in) {
  Tensor x = input;
  if (x.dim() > 2) x = x.reshape({-1, batch, n_in}).select(0, 0);
  if (!x.is_contiguous()) x = x.contiguous();
  if (reinterpret_cast<uintptr_t>(x.const_data_ptr()) % 16 != 0) x = x.clone();
  return x;
}

// One product.  Scratch is only allocated when it is used: with FLAG_SCRATCH_REDUCE, or for the second attempt on a
// device that could not place the thread-block cluster of a split K.
void launch_matmul(const char *what, c10::Device dev, int64_t bitwidth, int64_t group_size, int64_t n_out, int64_t n_in, int64_t batch,
                   const Tensor &weights, const Tensor &scales, const void *x, void *y, int64_t flags) {
  void *stream = stream_of(dev);
  const auto call = [&](const Tensor &ws) {
    return lib.matmul_ws(bitwidth, group_size, n_out, n_in, batch, weights.const_data_ptr(), scales.const_data_ptr(), x, y, stream,
                         static_cast<uint32_t>(flags), ws.defined() ? ws.data_ptr() : nullptr, ws.defined() ? ws.numel() : 0, 0, 0);
  };
  const auto scratch = [&]() {
    const int64_t need = lib.workspace_bytes(n_out, n_in, batch);
    return need > 0 ? empty_on({need}, at::kByte, dev) : Tensor();
  };
  const bool through_scratch = (flags & MATGPTQ_B200_FLAG_SCRATCH_REDUCE) != 0;
  int st = call(through_scratch ? scratch() : Tensor());
  if (st == MATGPTQ_B200_ERR_CUDA && !through_scratch) {
    const Tensor ws = scratch();
    if (ws.defined()) st = call(ws);
  }
  check_status(st, what);
}

void check_types(const Tensor &input, const Tensor &scales, int64_t flags) {
  const at::ScalarType want = type_of(flags);
  TORCH_CHECK(input.scalar_type() == want && scales.scalar_type() == want, "input and matgptq_scales must be ", type_name(flags),
              " for feature_flag=", flags);
}

Tensor matmul(const Tensor &input, const Tensor &weights, const Tensor &scales, int64_t n_out, int64_t n_in, int64_t bitwidth,
              int64_t group_size, int64_t flags) {
  check_matmul(input, weights, scales, n_out, n_in, bitwidth, group_size);
  check_types(input, scales, flags);
  const c10::Device dev = weights.device();
  const int64_t batch = input.size(-2);
  const c10::cuda::CUDAGuard on_device(dev);
  const Tensor x = prepare_input(input, batch, n_in);
  Tensor out = empty_on({batch, n_out}, type_of(flags), dev);
  launch_matmul("matmul_matgptq", dev, bitwidth, group_size, n_out, n_in, batch, weights, scales, x.const_data_ptr(), out.data_ptr(), flags);
  return out;
}

void matmul_out(const Tensor &input, const Tensor &weights, const Tensor &scales, int64_t n_out, int64_t n_in, int64_t bitwidth,
                int64_t group_size, int64_t flags, const Tensor &out) {
  check_matmul(input, weights, scales, n_out, n_in, bitwidth, group_size);
  check_types(input, scales, flags);
  const c10::Device dev = weights.device();
  const int64_t batch = input.size(-2);
  TORCH_CHECK(out.scalar_type() == type_of(flags) && out.device() == dev && out.dim() == 2 && out.size(0) == batch &&
                  out.size(1) == n_out && out.is_contiguous() && reinterpret_cast<uintptr_t>(out.const_data_ptr()) % 2 == 0,
              "out must be a contiguous ", type_name(flags), " tensor of shape (", batch, ", ", n_out, ") on ", dev);
  const c10::cuda::CUDAGuard on_device(dev);
  const Tensor x = prepare_input(input, batch, n_in);
  launch_matmul("matmul_matgptq_out", dev, bitwidth, group_size, n_out, n_in, batch, weights, scales, x.const_data_ptr(), out.data_ptr(),
                flags);
}

// The C-ABI grouped product: segment i fills its column block of out [M, sum(n_out)].
template <typename Weights, typename Ints>
Tensor grouped_unchecked(const Tensor &x, const Weights &weights, const Weights &scales, const Ints &n_out, int64_t n_in, const Ints &bits,
                         int64_t group_size, int64_t flags) {
  const c10::Device dev = x.device();
  const int64_t batch = x.size(-2);
  matgptq_b200_segment segs[8];
  int64_t total = 0, need = 0;
  const size_t n = weights.size();
  for (size_t i = 0; i < n; ++i) {
    segs[i] = matgptq_b200_segment{static_cast<const Tensor &>(weights[i]).const_data_ptr(),
                                   static_cast<const Tensor &>(scales[i]).const_data_ptr(), n_out[i], bits[i]};
    total += n_out[i];
    if (flags & MATGPTQ_B200_FLAG_SCRATCH_REDUCE) need = std::max(need, lib.workspace_bytes(n_out[i], n_in, batch));
  }
  Tensor out = empty_on({batch, total}, x.scalar_type(), dev);
  const Tensor ws = need > 0 ? empty_on({need}, at::kByte, dev) : Tensor();
  check_status(lib.matmul_grouped(segs, static_cast<int>(n), group_size, n_in, batch, x.const_data_ptr(), out.data_ptr(), stream_of(dev),
                                  static_cast<uint32_t>(flags), ws.defined() ? ws.data_ptr() : nullptr, ws.defined() ? ws.numel() : 0),
               "matgptq_b200_matmul_grouped");
  return out;
}

Tensor matmul_grouped(const Tensor &input, at::TensorList weights, at::TensorList scales, at::IntArrayRef n_out, int64_t n_in,
                      at::IntArrayRef bits, int64_t group_size, int64_t flags) {
  TORCH_CHECK(!weights.empty() && weights.size() == scales.size() && weights.size() == n_out.size() && weights.size() == bits.size(),
              "matmul_matgptq_grouped: one weight, scale, n_out_features and bitwidth per segment");
  TORCH_CHECK(weights.size() <= 8, "matmul_matgptq_grouped: at most 8 segments");
  const at::ScalarType want = type_of(flags);
  for (size_t i = 0; i < weights.size(); ++i) {
    check_matmul(input, weights[i], scales[i], n_out[i], n_in, bits[i], group_size);
    TORCH_CHECK(scales[i].scalar_type() == want, "matgptq_scales must be ", type_name(flags), " for feature_flag=", flags);
  }
  TORCH_CHECK(input.scalar_type() == want, "input must be ", type_name(flags), " for feature_flag=", flags);
  const c10::cuda::CUDAGuard on_device(input.device());
  const Tensor x = prepare_input(input, input.size(-2), n_in);
  return grouped_unchecked(x, weights, scales, n_out, n_in, bits, group_size, flags);
}

Tensor matmul_zeros(const Tensor &input, const Tensor &weights, const Tensor &scales, const Tensor &zeros, int64_t n_out, int64_t n_in,
                    int64_t bitwidth, int64_t group_size, int64_t flags) {
  check_matmul(input, weights, scales, n_out, n_in, bitwidth, group_size);
  const at::ScalarType want = type_of(flags);
  TORCH_CHECK(input.scalar_type() == want && scales.scalar_type() == want && zeros.scalar_type() == want,
              "input, matgptq_scales and matgptq_zeros must be ", type_name(flags), " for feature_flag=", flags);
  TORCH_CHECK(zeros.sizes() == scales.sizes() && zeros.device() == scales.device(),
              "matgptq_zeros must have the shape and device of matgptq_scales");
  const c10::Device dev = weights.device();
  const int64_t batch = input.size(-2);
  const c10::cuda::CUDAGuard on_device(dev);
  const Tensor x = prepare_input(input, batch, n_in);
  const Tensor z = zeros.contiguous();
  Tensor out = empty_on({batch, n_out}, want, dev);
  check_status(lib.matmul_zp(bitwidth, group_size, n_out, n_in, batch, weights.const_data_ptr(), scales.const_data_ptr(),
                             z.const_data_ptr(), x.const_data_ptr(), out.data_ptr(), stream_of(dev), static_cast<uint32_t>(flags)),
               "matmul_matgptq_zeros");
  return out;
}

}  // namespace

TORCH_LIBRARY(matgptq_cuda, m) {
  const std::vector<at::Tag> tags = {at::Tag::pt2_compliant_tag};
  m.def("pack_matgptq_qweights(Tensor qweights, SymInt n_out_features, SymInt n_in_features, SymInt bitwidth, SymInt group_size, "
        "SymInt feature_flag) -> Tensor", tags);
  m.def("slice_pack_matgptq_qweights(Tensor qweights, SymInt n_out_features, SymInt n_in_features, SymInt master_bitwidth, "
        "SymInt bitwidth, SymInt group_size, SymInt feature_flag) -> Tensor", tags);
  m.def("reorder_matgptq_scales(Tensor scales, SymInt m, SymInt n, SymInt group_size) -> Tensor", tags);
  m.def("matmul_matgptq(Tensor input, Tensor matgptq_weights, Tensor matgptq_scales, SymInt n_out_features, SymInt n_in_features, "
        "SymInt bitwidth, SymInt group_size, SymInt feature_flag) -> Tensor", tags);
  m.def("matmul_matgptq_out(Tensor input, Tensor matgptq_weights, Tensor matgptq_scales, SymInt n_out_features, "
        "SymInt n_in_features, SymInt bitwidth, SymInt group_size, SymInt feature_flag, Tensor(a8!) out) -> ()", tags);
  m.def("matmul_matgptq_grouped(Tensor input, Tensor[] matgptq_weights, Tensor[] matgptq_scales, SymInt[] n_out_features, "
        "SymInt n_in_features, SymInt[] bitwidths, SymInt group_size, SymInt feature_flag) -> Tensor", tags);
  m.def("matmul_matgptq_zeros(Tensor input, Tensor matgptq_weights, Tensor matgptq_scales, Tensor matgptq_zeros, "
        "SymInt n_out_features, SymInt n_in_features, SymInt bitwidth, SymInt group_size, SymInt feature_flag) -> Tensor", tags);
  m.def("dequantize_matgptq(Tensor matgptq_weights, Tensor matgptq_scales, SymInt n_out_features, SymInt n_in_features, "
        "SymInt bitwidth, SymInt group_size, SymInt feature_flag) -> Tensor", tags);
}

// The CPU registrations move what the packers and the reordering take from the host; the other operators refuse host
// tensors there.
#define MG_REGISTER(key)                                                    \
  TORCH_LIBRARY_IMPL(matgptq_cuda, key, m) {                                \
    m.impl("pack_matgptq_qweights", pack);                                  \
    m.impl("slice_pack_matgptq_qweights", slice_pack);                      \
    m.impl("reorder_matgptq_scales", reorder);                              \
    m.impl("matmul_matgptq", matmul);                                       \
    m.impl("matmul_matgptq_out", matmul_out);                               \
    m.impl("matmul_matgptq_grouped", matmul_grouped);                       \
    m.impl("matmul_matgptq_zeros", matmul_zeros);                           \
    m.impl("dequantize_matgptq", dequantize);                               \
  }
MG_REGISTER(CPU)
MG_REGISTER(CUDA)

// ---- autograd -------------------------------------------------------------------------------------------------
namespace {

// No operator has a derivative: a result of inputs that require one says so when backward reaches it.  Any other call goes
// on below autograd as it is; forward-mode tangents end here, and `out` may be a leaf that requires a gradient.
void without_derivative(const c10::OperatorHandle &op, c10::DispatchKeySet keys, torch::jit::Stack *stack) {
  std::vector<Tensor> inputs;  // those that require a gradient
  const auto &arguments = op.schema().arguments();
  if (at::GradMode::is_enabled()) {
    const size_t first = stack->size() - arguments.size();
    const auto add = [&](const Tensor &t) {
      if (!t.requires_grad()) return;
      TORCH_CHECK_NOT_IMPLEMENTED(!torch::autograd::isFwGradDefined(t), "forward AD through ", op.schema().name(), " is not implemented");
      inputs.push_back(t);
    };
    for (size_t i = 0; i < arguments.size(); ++i) {
      const c10::IValue &v = (*stack)[first + i];
      if (arguments[i].alias_info()) continue;  // written, not read
      if (v.isTensor()) add(v.toTensor());
      if (v.isTensorList())
        for (const Tensor &t : v.toTensorVector()) add(t);
    }
  }
  {
    const at::AutoDispatchBelowAutograd below;
    op.redispatchBoxed(keys & c10::after_autograd_keyset, stack);
  }
  if (inputs.empty() || op.schema().returns().empty()) return;
  const auto node = std::make_shared<torch::autograd::NotImplemented>(op.schema().name(), torch::autograd::collect_next_edges(inputs));
  Tensor result = stack->back().toTensor();
  torch::autograd::set_history(result, node);
}

// matmul_matgptq_out writes its last argument
void counts_as_write(const c10::OperatorHandle &op, c10::DispatchKeySet keys, torch::jit::Stack *stack) {
  const Tensor out = stack->back().toTensor();
  {
    const at::AutoDispatchBelowADInplaceOrView below;
    op.redispatchBoxed(keys & c10::after_ADInplaceOrView_keyset, stack);
  }
  if (!out.is_inference()) out.unsafeGetTensorImpl()->bump_version();
}

}  // namespace

TORCH_LIBRARY_IMPL(matgptq_cuda, Autograd, m) {
  for (const char *name : {"pack_matgptq_qweights", "slice_pack_matgptq_qweights", "reorder_matgptq_scales", "matmul_matgptq",
                           "matmul_matgptq_out", "matmul_matgptq_grouped", "matmul_matgptq_zeros", "dequantize_matgptq"})
    m.impl(name, torch::CppFunction::makeFromBoxedFunction<&without_derivative>());
}

TORCH_LIBRARY_IMPL(matgptq_cuda, ADInplaceOrView, m) {
  m.impl("matmul_matgptq_out", torch::CppFunction::makeFromBoxedFunction<&counts_as_write>());
}

// ---- Python module --------------------------------------------------------------------------------------------
namespace {

// A launch may wait for room in the stream's queue, and an allocation for the device: other Python threads (and Python
// callbacks that the stream is waiting for) go on meanwhile.
struct WithoutGil {
  PyThreadState *state = PyEval_SaveThread();
  ~WithoutGil() { PyEval_RestoreThread(state); }
};

// A tensor whose bytes are what the kernel would read.  The keys are those of an ordinary CUDA tensor and nothing else: one
// with the negative bit or without storage, or a subclass's, has a key of its own and is the dispatcher's to materialise.
bool plain_cuda(PyObject *o) {
  if (!THPVariable_CheckExact(o)) return false;
  const Tensor &t = THPVariable_Unpack(o);
  constexpr c10::DispatchKeySet ordinary({c10::DispatchKey::CUDA, c10::DispatchKey::AutogradCUDA, c10::DispatchKey::ADInplaceOrView,
                                          c10::DispatchKey::AutocastCUDA});
  return t.is_cuda() && t.layout() == at::kStrided && (t.key_set() - ordinary).highestFunctionalityKey() == c10::DispatchKey::Undefined;
}

// nothing between the caller and the kernel wants to see the call
bool dispatcher_not_needed() {
  const c10::impl::LocalDispatchKeySet tls = c10::impl::tls_local_dispatch_key_set();
  constexpr c10::DispatchKeySet listeners({c10::DispatchKey::Python, c10::DispatchKey::PythonTLSSnapshot, c10::DispatchKey::PythonDispatcher,
                                           c10::DispatchKey::Functionalize, c10::DispatchKey::FuncTorchDynamicLayerFrontMode,
                                           c10::DispatchKey::FuncTorchDynamicLayerBackMode, c10::DispatchKey::Tracer,
                                           c10::DispatchKey::PreDispatch});
  return (tls.included_ & listeners).empty() && !c10::impl::TorchDispatchModeTLS::any_modes_set() &&
         at::impl::PythonTorchFunctionTLS::stack_len() == 0 && c10::impl::PythonDispatcherTLS::get_state() == nullptr;
}

// Whole numbers, numpy's among them (anything with __index__).
bool as_ints(PyObject *const *args, Py_ssize_t n, int64_t *out) {
  for (Py_ssize_t i = 0; i < n; ++i) {
    out[i] = PyLong_AsLongLong(args[i]);
    if (out[i] == -1 && PyErr_Occurred()) {
      PyErr_Clear();
      return false;
    }
  }
  return true;
}

// linear_forward(x, weights, scales, n_out, n_in, bitwidth, group_size, flags): x [..., n_in] -> [..., n_out], every
// leading dimension counted as rows.  None when the call has to go through the dispatcher.
PyObject *py_linear_forward(PyObject *, PyObject *const *args, Py_ssize_t nargs) {
  HANDLE_TH_ERRORS
  int64_t v[5];  // n_out, n_in, bitwidth, group_size, flags
  if (nargs != 8 || !plain_cuda(args[0]) || !plain_cuda(args[1]) || !plain_cuda(args[2]) || !as_ints(args + 3, 5, v) ||
      !dispatcher_not_needed())
    Py_RETURN_NONE;
  const Tensor &input = THPVariable_Unpack(args[0]), &weights = THPVariable_Unpack(args[1]), &scales = THPVariable_Unpack(args[2]);
  if (input.dim() < 2) Py_RETURN_NONE;
  RECORD_FUNCTION("matgptq_cuda::matmul_matgptq", std::vector<c10::IValue>());
  check_matmul(input, weights, scales, v[0], v[1], v[2], v[3]);
  check_types(input, scales, v[4]);
  const c10::Device dev = weights.device();
  const c10::cuda::CUDAGuard on_device(dev);
  c10::SmallVector<int64_t, 5> sizes(input.sizes().begin(), input.sizes().end());
  int64_t rows = 1;
  for (size_t i = 0; i + 1 < sizes.size(); ++i) rows *= sizes[i];
  sizes.back() = v[0];
  Tensor out;
  {
    const WithoutGil released;
    Tensor copy;
    if (!input.is_contiguous() || reinterpret_cast<uintptr_t>(input.const_data_ptr()) % 16 != 0) {
      const at::AutoDispatchBelowADInplaceOrView below;
      copy = input.clone(at::MemoryFormat::Contiguous);
    }
    out = empty_on(sizes, type_of(v[4]), dev);
    launch_matmul("matmul_matgptq", dev, v[2], v[3], v[0], v[1], rows, weights, scales,
                  copy.defined() ? copy.const_data_ptr() : input.const_data_ptr(), out.data_ptr(), v[4]);
  }
  return THPVariable_Wrap(std::move(out));
  END_HANDLE_TH_ERRORS
}

// grouped_raw(x, weights, scales, n_out, n_in, bits, group_size, flags): no checks beyond the C ABI's own
PyObject *py_grouped_raw(PyObject *, PyObject *const *args, Py_ssize_t nargs) {
  HANDLE_TH_ERRORS
  TORCH_CHECK(nargs == 8 && THPVariable_Check(args[0]) && PyList_Check(args[1]) && PyList_Check(args[2]) && PyList_Check(args[3]) &&
                  PyList_Check(args[5]),
              "grouped_raw(x, weights, scales, n_out, n_in, bits, group_size, flags)");
  const Py_ssize_t n = PyList_GET_SIZE(args[1]);
  TORCH_CHECK(n >= 1 && n <= 8 && PyList_GET_SIZE(args[2]) == n && PyList_GET_SIZE(args[3]) == n && PyList_GET_SIZE(args[5]) == n,
              "matmul_matgptq_grouped: one weight, scale, n_out_features and bitwidth per segment, at most 8 segments");
  c10::SmallVector<Tensor, 8> w, s;
  c10::SmallVector<int64_t, 8> rows(n), bits(n);
  for (Py_ssize_t i = 0; i < n; ++i) {
    PyObject *pw = PyList_GET_ITEM(args[1], i), *ps = PyList_GET_ITEM(args[2], i);
    PyObject *ints[2] = {PyList_GET_ITEM(args[3], i), PyList_GET_ITEM(args[5], i)};
    int64_t v[2];
    TORCH_CHECK(THPVariable_Check(pw) && THPVariable_Check(ps) && as_ints(ints, 2, v), "grouped_raw: tensors and whole numbers");
    w.push_back(THPVariable_Unpack(pw));
    s.push_back(THPVariable_Unpack(ps));
    rows[i] = v[0];
    bits[i] = v[1];
  }
  int64_t n_in, gf[2];
  TORCH_CHECK(as_ints(args + 4, 1, &n_in) && as_ints(args + 6, 2, gf), "grouped_raw: whole numbers");
  const Tensor &x = THPVariable_Unpack(args[0]);
  const c10::cuda::CUDAGuard on_device(x.device());
  Tensor out;
  {
    const WithoutGil released;
    out = grouped_unchecked(x, w, s, rows, n_in, bits, gf[0], gf[1]);
  }
  return THPVariable_Wrap(std::move(out));
  END_HANDLE_TH_ERRORS
}

// matmul_raw(x, weights, scales, n_out, n_in, bitwidth, group_size, flags, out or None): no checks beyond the C ABI's own
PyObject *py_matmul_raw(PyObject *, PyObject *const *args, Py_ssize_t nargs) {
  HANDLE_TH_ERRORS
  int64_t v[5];
  TORCH_CHECK(nargs == 9 && THPVariable_Check(args[0]) && THPVariable_Check(args[1]) && THPVariable_Check(args[2]) &&
                  as_ints(args + 3, 5, v) && (args[8] == Py_None || THPVariable_Check(args[8])),
              "matmul_raw(x, weights, scales, n_out, n_in, bitwidth, group_size, flags, out)");
  const Tensor &x = THPVariable_Unpack(args[0]), &weights = THPVariable_Unpack(args[1]), &scales = THPVariable_Unpack(args[2]);
  const c10::Device dev = x.device();
  const c10::cuda::CUDAGuard on_device(dev);
  const int64_t batch = x.size(-2);
  Tensor out = args[8] == Py_None ? Tensor() : THPVariable_Unpack(args[8]);
  {
    const WithoutGil released;
    if (!out.defined()) out = empty_on({batch, v[0]}, x.scalar_type(), dev);
    launch_matmul("matgptq_b200_matmul", dev, v[2], v[3], v[0], v[1], batch, weights, scales, x.const_data_ptr(), out.data_ptr(), v[4]);
  }
  return THPVariable_Wrap(std::move(out));
  END_HANDLE_TH_ERRORS
}

// bind(path): the C-ABI library that the operators call (already loaded by the caller; its handle is kept)
PyObject *py_bind(PyObject *, PyObject *path) {
  HANDLE_TH_ERRORS
  const char *p = PyUnicode_AsUTF8(path);
  if (!p) return nullptr;
  void *handle = dlopen(p, RTLD_NOW | RTLD_LOCAL);
  TORCH_CHECK(handle, "cannot load ", p, ": ", dlerror());
  const auto find = [&](auto &fn, const char *name) {
    fn = reinterpret_cast<std::decay_t<decltype(fn)>>(dlsym(handle, name));
    TORCH_CHECK(fn, p, " does not export ", name);
  };
  find(lib.strerror, "matgptq_b200_strerror");
  find(lib.matmul_ws, "matgptq_b200_matmul_ws");
  find(lib.matmul_zp, "matgptq_b200_matmul_zp");
  find(lib.matmul_grouped, "matgptq_b200_matmul_grouped");
  find(lib.workspace_bytes, "matgptq_b200_matmul_workspace_bytes");
  find(lib.pack_qweights, "matgptq_b200_pack_qweights");
  find(lib.reorder_scales, "matgptq_b200_reorder_scales");
  find(lib.dequantize, "matgptq_b200_dequantize");
  Py_RETURN_NONE;
  END_HANDLE_TH_ERRORS
}

PyMethodDef methods[] = {
    {"bind", py_bind, METH_O, "bind(path): the C-ABI library to call"},
    {"linear_forward", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(py_linear_forward)), METH_FASTCALL, nullptr},
    {"grouped_raw", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(py_grouped_raw)), METH_FASTCALL, nullptr},
    {"matmul_raw", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(py_matmul_raw)), METH_FASTCALL, nullptr},
    {nullptr, nullptr, 0, nullptr}};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "_torch_ops", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__torch_ops() { return PyModule_Create(&module); }

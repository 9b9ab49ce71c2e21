// Python entry to the library's hot calls: allocates the outputs with torch, looks up the current stream and calls the
// C ABI, in one native function per call.
//
// A small layer is paced by the host, not by its kernels. Through ctypes one quantizer call on 16 x 4096 values cost 27 us,
// 13 of them in the library (three launches): the rest was argument conversion, three allocations and the checks in
// Python. The functions below make the same checks with the same messages and exception types (what is not a tensor is a
// RuntimeError with the argument's name, memory that runs out is torch.OutOfMemoryError), allocate through torch's
// dispatcher as torch.empty does, and release the interpreter lock while the library runs, as ctypes does. Nothing is kept
// between calls.
#include <ATen/ATen.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>
#include <torch/csrc/utils/pybind.h>

#include <stdexcept>
#include <string>
#include <tuple>

#include "../../include/bitlattice_b200.h"

namespace {

using at::Tensor;
using Arg = pybind11::handle;

[[noreturn]] void fail(const std::string& what) { throw std::runtime_error(what); }

template <typename F>
void run(F&& call) {
  int rc;
  {
    pybind11::gil_scoped_release release;
    rc = call();
  }
  if (rc != 0) fail(bl_last_error());
}

std::string type_name(at::ScalarType t) {
  switch (t) {
    case at::kByte: return "torch.uint8";
    case at::kFloat: return "torch.float32";
    case at::kBFloat16: return "torch.bfloat16";
    case at::kHalf: return "torch.float16";
    default: return std::string("torch.") + at::toString(t);
  }
}

// int(value) in its lowest 64 bits, which is what ctypes passes on
int64_t integer(Arg value) {
  PyObject* number = PyNumber_Long(value.ptr());
  if (number == nullptr) throw python_error();
  const unsigned long long bits = PyLong_AsUnsignedLongLongMask(number);
  Py_DECREF(number);
  return static_cast<int64_t>(bits);
}

const Tensor& require(const Tensor& t, const char* name) {
  if (!t.defined() || !t.is_cuda()) fail(std::string(name) + " must be a CUDA tensor (this build has no CPU path)");
  if (!t.is_contiguous()) fail(std::string(name) + " must be contiguous");
  return t;
}

const Tensor& require(const Tensor& t, const char* name, at::ScalarType type) {
  require(t, name);
  if (t.scalar_type() != type) fail(std::string(name) + " must be " + type_name(type) + ", got " + type_name(t.scalar_type()));
  return t;
}

// (the caller's reference keeps the tensor alive during the call)
const Tensor& require(Arg t, const char* name) {
  if (!THPVariable_Check(t.ptr())) fail(std::string(name) + " must be a CUDA tensor (this build has no CPU path)");
  return require(THPVariable_Unpack(t.ptr()), name);
}

const Tensor& require(Arg t, const char* name, at::ScalarType type) {
  return require(require(t, name), name, type);
}

// a per-tensor scale of any type, shape and stride
Tensor scalar(Arg t, const char* name) {
  if (!THPVariable_Check(t.ptr())) fail(std::string(name) + " must be a CUDA tensor (this build has no CPU path)");
  Tensor g = THPVariable_Unpack(t.ptr());
  if (g.scalar_type() != at::kFloat || g.numel() != 1 || !g.is_contiguous()) g = g.to(at::kFloat).reshape({1}).contiguous();
  return require(g, name);
}

int dtype_code(const Tensor& t, const char* message) {
  switch (t.scalar_type()) {
    case at::kFloat: return BL_F32;
    case at::kBFloat16: return BL_BF16;
    case at::kHalf: return BL_F16;
    default: fail(message);
  }
}
constexpr const char* kDense = "x must be bf16, fp16 or fp32";

int device_index(const Tensor& t) { return t.get_device(); }
bl_stream_t stream_of(const Tensor& t) {
  return reinterpret_cast<bl_stream_t>(c10::cuda::getCurrentCUDAStream(static_cast<c10::DeviceIndex>(t.get_device())).stream());
}

Tensor empty(at::IntArrayRef size, at::ScalarType type, const Tensor& like) {
  return at::empty(size, at::TensorOptions().dtype(type).device(like.device()));
}
Tensor scale_buffer(int64_t rows, int64_t cols16, bool blocked, const Tensor& like) {
  if (blocked) return empty({((rows + 127) / 128) * ((cols16 + 3) / 4) * 512}, at::kByte, like);
  return empty({rows, cols16}, at::kByte, like);
}

uint8_t* bytes(const Tensor& t) { return static_cast<uint8_t*>(t.data_ptr()); }
float* floats(const Tensor& t) { return static_cast<float*>(t.data_ptr()); }

int64_t last(const Tensor& x) {
  if (x.dim() == 0 || x.size(-1) == 0) fail("x: the last dimension must not be empty");
  return x.size(-1);
}

Tensor amax_global(Arg x_) {
  const Tensor& x = require(x_, "x");
  const int code = dtype_code(x, kDense);
  Tensor out = empty({4}, at::kFloat, x);
  run([&] { return bl_nvfp4_amax(x.data_ptr(), code, x.numel(), floats(out), device_index(x), stream_of(x)); });
  return out;
}

std::tuple<Tensor, Tensor, Tensor> amax_quantize(Arg x_, Arg seed_, Arg step_, Arg blocked) {
  const Tensor& x = require(x_, "x");
  const int code = dtype_code(x, kDense), layout = static_cast<int>(integer(blocked));
  const int64_t cols = last(x), rows = x.numel() / cols, seed = integer(seed_), step = integer(step_);
  Tensor am = empty({4}, at::kFloat, x), packed = empty({rows, cols / 2}, at::kByte, x);
  Tensor scales = scale_buffer(rows, cols / 16, layout != 0, x);
  run([&] {
    return bl_nvfp4_amax_quantize(x.data_ptr(), code, rows, cols, floats(am), seed, static_cast<uint32_t>(step), bytes(packed),
                                  bytes(scales), layout, device_index(x), stream_of(x));
  });
  return {packed, scales, am};
}

std::tuple<Tensor, Tensor> quantize_4over6(Arg x_, Arg global, bool mae, Arg blocked) {
  const Tensor &x = require(x_, "x"), &g = require(global, "global_scale", at::kFloat);
  const int code = dtype_code(x, kDense), layout = static_cast<int>(integer(blocked));
  const int64_t cols = last(x), rows = x.numel() / cols;
  Tensor packed = empty({rows, cols / 2}, at::kByte, x), scales = scale_buffer(rows, cols / 16, layout != 0, x);
  run([&] {
    return bl_nvfp4_quantize_4over6(x.data_ptr(), code, rows, cols, floats(g), mae ? 1 : 0, bytes(packed), bytes(scales),
                                    layout, device_index(x), stream_of(x));
  });
  return {packed, scales};
}

std::tuple<Tensor, Tensor, Tensor> quantize_t(Arg x_, Arg hadamard, Arg seed_, Arg step_, Arg bound, double bound_factor,
                                              Arg blocked, int64_t pad_rows) {
  const Tensor& x = require(x_, "x");
  if (x.dim() != 2) fail("x must be a contiguous 2-D CUDA tensor");
  if (pad_rows < 1) fail("pad_rows must be at least 1, got " + std::to_string(pad_rows));
  const int code = dtype_code(x, kDense), layout = static_cast<int>(integer(blocked));
  const int64_t rows = x.size(0), K = x.size(1), M = (rows + pad_rows - 1) / pad_rows * pad_rows;
  const int64_t seed = integer(seed_), step = integer(step_);
  const float* H = nullptr;
  if (!hadamard.is_none()) {
    const Tensor& h = require(hadamard, "hadamard", at::kFloat);
    if (h.numel() != 256) fail("hadamard must be a contiguous fp32 [16, 16] tensor");
    H = floats(h);
  }
  Tensor packed = empty({K, M / 2}, at::kByte, x), scales = scale_buffer(K, M / 16, layout != 0, x), gout = empty({1}, at::kFloat, x);
  Tensor given, amax;
  if (bound.is_none()) amax = empty({4}, at::kFloat, x);
  else given = scalar(bound, "global_scale");
  run([&] {
    return bl_nvfp4_quantize_t_rows(x.data_ptr(), code, rows, M, K, H, seed, static_cast<uint32_t>(step),
                                    given.defined() ? floats(given) : nullptr, static_cast<float>(bound_factor),
                                    amax.defined() ? floats(amax) : nullptr, bytes(packed), bytes(scales), floats(gout),
                                    layout, device_index(x), stream_of(x));
  });
  return {packed, scales, gout};
}

std::tuple<Tensor, Tensor, Tensor> requantize_t(Arg packed_, Arg scales_, Arg global, Arg blocked) {
  const Tensor &packed = require(packed_, "packed", at::kByte), &scales = require(scales_, "scales");
  const Tensor g = scalar(global, "global_scale");
  const int layout = static_cast<int>(integer(blocked));
  const int64_t N = packed.size(0), K = packed.size(1) * 2;
  Tensor out = empty({K, N / 2}, at::kByte, packed), osc = scale_buffer(K, N / 16, layout != 0, packed), gout = empty({1}, at::kFloat, packed);
  run([&] {
    return bl_nvfp4_requantize_t(bytes(packed), bytes(scales), floats(g), N, K, bytes(out), bytes(osc), floats(gout), layout,
                                 device_index(packed), stream_of(packed));
  });
  return {out, osc, gout};
}

Tensor to_blocked(Arg scales_) {
  const Tensor& scales = require(scales_, "scales");
  if (scales.dim() != 2) fail("scales must be a 2-D tensor");
  Tensor out = scale_buffer(scales.size(0), scales.size(1), true, scales);
  run([&] {
    return bl_nvfp4_scales_to_blocked(bytes(scales), scales.size(0), scales.size(1), bytes(out), device_index(scales), stream_of(scales));
  });
  return out;
}

Tensor dequantize(Arg packed_, Arg scales_, Arg global_, int64_t rows, int64_t cols, int code) {
  const Tensor &packed = require(packed_, "packed", at::kByte), &scales = require(scales_, "scales");
  const Tensor& global = require(global_, "global_scale", at::kFloat);
  Tensor out = empty({rows, cols}, code == BL_F32 ? at::kFloat : code == BL_BF16 ? at::kBFloat16 : at::kHalf, packed);
  run([&] {
    return bl_nvfp4_dequantize(bytes(packed), bytes(scales), floats(global), rows, cols, out.data_ptr(), code, device_index(packed),
                               stream_of(packed));
  });
  return out;
}

Tensor gemm(Arg a_, Arg a_sf_, Arg ga_, Arg b_, Arg b_sf_, Arg gb_, int out_code, Arg into, bool accumulate) {
  const Tensor &a = require(a_, "a_packed", at::kByte), &b = require(b_, "b_packed", at::kByte);
  const Tensor &a_sf = require(a_sf_, "a_sf"), &b_sf = require(b_sf_, "b_sf");
  const int64_t M = a.size(0), K = a.size(1) * 2, N = b.size(0);
  if (b.size(1) * 2 != K) fail("operand K mismatch: " + std::to_string(K) + " vs " + std::to_string(b.size(1) * 2));
  auto blocked = [&](int64_t rows) { return ((rows + 127) / 128) * ((K / 16 + 3) / 4) * 512; };
  if (a_sf.numel() < blocked(M) || b_sf.numel() < blocked(N)) fail("scale buffers are smaller than the blocked layout of their operands");
  const Tensor &ga = require(ga_, "a_global", at::kFloat), &gb = require(gb_, "b_global", at::kFloat);
  Tensor out;
  if (into.is_none()) {
    if (accumulate) fail("accumulate needs the tensor to add to (out=)");
    out = empty({M, N}, out_code == BL_F32 ? at::kFloat : out_code == BL_BF16 ? at::kBFloat16 : at::kHalf, a);
  } else {
    if (THPVariable_Check(into.ptr())) out = THPVariable_Unpack(into.ptr());
    if (!out.defined() || out.dim() != 2 || out.size(0) != M || out.size(1) != N || !out.is_cuda() || out.stride(1) != 1)
      fail("out must be a CUDA tensor [" + std::to_string(M) + ", " + std::to_string(N) + "] with unit column stride");
  }
  const int code = dtype_code(out, "out must be bf16, fp16 or fp32");
  run([&] {
    return (accumulate ? bl_nvfp4_gemm_accumulate : bl_nvfp4_gemm)(bytes(a), bytes(a_sf), floats(ga), bytes(b), bytes(b_sf),
                                                                    floats(gb), M, N, K, out.data_ptr(), code, out.stride(0),
                                                                    device_index(a), stream_of(a));
  });
  return out;
}

}  // namespace

// wrap_pybind_function: exceptions of torch keep their Python types (torch.OutOfMemoryError, IndexError)
PYBIND11_MODULE(_host, m) {
  m.def("amax_global", torch::wrap_pybind_function(&amax_global));
  m.def("amax_quantize", torch::wrap_pybind_function(&amax_quantize));
  m.def("quantize_4over6", torch::wrap_pybind_function(&quantize_4over6));
  m.def("quantize_t", torch::wrap_pybind_function(&quantize_t));
  m.def("requantize_t", torch::wrap_pybind_function(&requantize_t));
  m.def("to_blocked", torch::wrap_pybind_function(&to_blocked));
  m.def("dequantize", torch::wrap_pybind_function(&dequantize));
  m.def("gemm", torch::wrap_pybind_function(&gemm));
  m.attr("AMAX_QUANTIZE_SMALL") = BL_AMAX_QUANTIZE_SMALL;
}

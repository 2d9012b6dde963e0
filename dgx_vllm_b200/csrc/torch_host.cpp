// Host path of the torch-facing ops: argument checks, output allocation, workspace and the call into libb200nvfp4.so.
//
// The kernels of a decode step or of a small linear run for 5 to 20 us; the same host path in Python (checks, torch.empty,
// stream and device look-ups, a ctypes call with 15 to 30 arguments) took 20 to 35 us per call and was what such a step
// waited for.  Here it is plain C++ on the tensors' own objects behind METH_FASTCALL functions: launches included 6 us for one
// or two of them, 9 for the decode layer's three, 17 for the prefill layer's five.  The Python mirrors keep their signatures
// and hand their arguments straight over.
//
// Arguments are read with the GIL held; allocation and launches run without it (an allocation can reach cudaMalloc, a launch
// blocks while the stream's queue is full), under a lock per stream that keeps a call's steps and their scratch together.
#define PY_SSIZE_T_CLEAN
#include <Python.h>

#include <ATen/core/Tensor.h>
#include <ATen/cuda/EmptyTensor.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Dtype.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>

#include <mutex>
#include <stdexcept>
#include <string>
#include <unordered_map>

#include "../../include/b200_nvfp4.h"

namespace {

// ------------------------------------------------------------------------------------------ plumbing

struct StatusError {
  int status;
  const char* where;
};
struct PythonError {};        // a Python exception is already set

void require(bool ok, const char* msg) {
  if (!ok) throw std::runtime_error(msg);
}

void check(int status, const char* where) {
  if (status != B200FP4_STATUS_SUCCESS) throw StatusError{status, where};
}

// Runs a function body and turns what it throws into the Python exceptions the mirrors have always raised.
template <typename F>
PyObject* guarded(F&& f) {
  try {
    return f();
  } catch (const StatusError& e) {
    PyObject* mod = PyImport_ImportModule("dgx_vllm_b200._lib");
    PyObject* cls = mod ? PyObject_GetAttrString(mod, "B200Fp4Error") : nullptr;
    PyObject* err = cls ? PyObject_CallFunction(cls, "is", e.status, e.where) : nullptr;
    if (err) PyErr_SetObject(cls, err);
    Py_XDECREF(err);
    Py_XDECREF(cls);
    Py_XDECREF(mod);
  } catch (const PythonError&) {
  } catch (...) {
    torch::translate_exception_to_python(std::current_exception());     // RuntimeError, or torch's own (out of memory)
  }
  return nullptr;
}

void want_args(Py_ssize_t got, Py_ssize_t want) {
  if (got != want) {
    PyErr_Format(PyExc_TypeError, "%zd arguments expected, got %zd", want, got);
    throw PythonError{};
  }
}

const at::Tensor& tensor(PyObject* o) {
  if (!THPVariable_Check(o)) {
    PyErr_Format(PyExc_TypeError, "a torch.Tensor is expected, got %s", Py_TYPE(o)->tp_name);
    throw PythonError{};
  }
  return THPVariable_Unpack(o);
}
// None stands for "not given"
const at::Tensor* maybe_tensor(PyObject* o) { return o == Py_None ? nullptr : &tensor(o); }

int64_t integer(PyObject* o) {
  const int64_t v = PyLong_AsLongLong(o);
  if (v == -1 && PyErr_Occurred()) throw PythonError{};
  return v;
}
bool truth(PyObject* o) {
  const int v = PyObject_IsTrue(o);
  if (v < 0) throw PythonError{};
  return v != 0;
}

int require_cuda(std::initializer_list<const at::Tensor*> ts) {
  int dev = -1;
  for (const at::Tensor* t : ts) {
    if (t == nullptr) continue;
    require(t->is_cuda(), "b200 nvfp4 ops take CUDA tensors only (there is no CPU path)");
    const int d = t->get_device();
    require(dev < 0 || d == dev, "all tensors must be on the same device");
    dev = d;
  }
  return dev;
}

int dtype_code(at::ScalarType t) {
  if (t == at::kHalf) return B200FP4_DTYPE_F16;
  if (t == at::kBFloat16) return B200FP4_DTYPE_BF16;
  if (t == at::kFloat) return B200FP4_DTYPE_F32;
  throw std::runtime_error(std::string("unsupported dtype ") + c10::toString(t));
}

bool is_16bit(const at::Tensor& t) { return t.scalar_type() == at::kHalf || t.scalar_type() == at::kBFloat16; }
bool is_f32_scalar(const at::Tensor& t) { return t.scalar_type() == at::kFloat && t.numel() == 1; }
bool is_2d(const at::Tensor& t, int64_t rows, int64_t cols) { return t.dim() == 2 && t.size(0) == rows && t.size(1) == cols; }

at::Tensor empty(at::IntArrayRef shape, at::ScalarType dtype, int dev) {
  return at::Tensor(at::detail::empty_cuda(shape, dtype, c10::Device(c10::kCUDA, (c10::DeviceIndex)dev), std::nullopt));
}

template <typename T = void>
T* ptr(const at::Tensor& t) {
  return static_cast<T*>(t.data_ptr());
}

// Other Python threads run while one of these is alive: nothing under it touches a Python object.
struct WithoutGil {
  PyThreadState* state = PyEval_SaveThread();
  WithoutGil() = default;
  WithoutGil(const WithoutGil&) = delete;
  ~WithoutGil() { PyEval_RestoreThread(state); }
};

// Grow-only scratch per (device, stream): calls issued on one stream serialise on the GPU, so consecutive ops share it; its
// address is stable once large enough, which CUDA-graph capture relies on.  One slot for each family of ops with a status word of
// its own (or whose words another's would land on).  The lock is held from the look-up to the last launch of a call: another
// thread on the same stream neither replaces the scratch under it nor puts a launch between its steps.  It is never waited
// for with the GIL held.
enum Slot { kSlotShared = 0, kSlotLinear = 1, kSlotRouter = 2, kSlotGemm = 3, kSlots = 4 };        // Python names them in _torch_util.py
struct StreamScratch {
  std::mutex mu;
  at::Tensor slots[kSlots];
};
struct StreamKey {
  int dev;
  cudaStream_t stream;
  bool operator==(const StreamKey& o) const { return dev == o.dev && stream == o.stream; }
};
struct StreamHash {
  size_t operator()(const StreamKey& k) const { return reinterpret_cast<size_t>(k.stream) * 0x9E3779B97F4A7C15ull + (size_t)k.dev; }
};

class Workspace {
 public:
  Workspace(int dev, cudaStream_t stream, size_t bytes, int slot = kSlotShared) : scratch_(of(dev, stream)), lock_(scratch_.mu), t_(scratch_.slots[slot]) {
    if (t_.defined() && (size_t)t_.numel() >= bytes) return;
    t_ = empty({(int64_t)std::max(bytes, (size_t)1 << 20)}, at::kByte, dev);
    t_.narrow(0, 0, 256).zero_();                  // a status word that no op has written yet reads 0
  }
  const at::Tensor& tensor() const { return t_; }
  void* data() const { return t_.data_ptr(); }
  size_t bytes() const { return t_.nbytes(); }

 private:
  static StreamScratch& of(int dev, cudaStream_t stream) {
    // never destroyed: at interpreter exit the allocator may be gone before this table would be
    static auto* table = new std::unordered_map<StreamKey, StreamScratch, StreamHash>();
    static std::mutex mu;
    std::lock_guard<std::mutex> lock(mu);
    return (*table)[StreamKey{dev, stream}];
  }
  StreamScratch& scratch_;
  std::lock_guard<std::mutex> lock_;
  at::Tensor& t_;
};

PyObject* wrap(at::Tensor t) {
  PyObject* o = THPVariable_Wrap(std::move(t));
  if (!o) throw PythonError{};
  return o;
}
PyObject* wrap2(at::Tensor a, at::Tensor b) {
  PyObject* x = wrap(std::move(a));
  PyObject* y = THPVariable_Wrap(std::move(b));
  PyObject* r = y ? PyTuple_Pack(2, x, y) : nullptr;
  Py_XDECREF(x);
  Py_XDECREF(y);
  if (!r) throw PythonError{};
  return r;
}

int64_t round_up(int64_t v, int64_t m) { return (v + m - 1) / m * m; }

#define B200_FN(name) PyObject* name(PyObject*, PyObject* const* args, Py_ssize_t n_args)

// ------------------------------------------------------------------------------------------ dense ops

// workspace(device index, bytes, slot) -> a scratch tensor of the current stream
B200_FN(py_workspace) {
  return guarded([&] {
    want_args(n_args, 3);
    const int dev = (int)integer(args[0]), slot = (int)integer(args[2]);
    const size_t bytes = (size_t)integer(args[1]);
    require(slot >= 0 && slot < kSlots, "no such workspace slot");
    at::Tensor t;
    {
      WithoutGil nogil;
      c10::cuda::CUDAGuard guard((c10::DeviceIndex)dev);
      t = Workspace(dev, c10::cuda::getCurrentCUDAStream((c10::DeviceIndex)dev).stream(), bytes, slot).tensor();
    }
    return wrap(std::move(t));
  });
}

// scaled_fp4_quant(input, global_scale, swizzled) -> (codes, scales)
B200_FN(py_quant) {
  return guarded([&] {
    want_args(n_args, 3);
    const at::Tensor &x = tensor(args[0]), &gs = tensor(args[1]);
    const bool swizzled = truth(args[2]);
    const int dev = require_cuda({&x, &gs});
    require(x.dim() == 2, "input must be 2-D");
    require(is_16bit(x), "input must be float16 or bfloat16");
    require(x.stride(1) == 1, "input rows must be contiguous");
    require(is_f32_scalar(gs), "global scale must be one f32");
    const int64_t M = x.size(0), K = x.size(1), KB = K / 16;
    require(K % 16 == 0, "K must be a multiple of 16");
    at::Tensor codes, sf;
    {
      WithoutGil nogil;
      c10::cuda::CUDAGuard guard((c10::DeviceIndex)dev);
      codes = empty({M, K / 2}, at::kByte, dev);
      sf = swizzled ? empty({round_up(M, 128), round_up(KB, 4)}, at::kFloat8_e4m3fn, dev) : empty({M, KB}, at::kFloat8_e4m3fn, dev);
      check(b200fp4_quantize(ptr(x), dtype_code(x.scalar_type()), M, K, M > 1 ? x.stride(0) : K, ptr<float>(gs), ptr(codes), ptr(sf),
                             swizzled ? 1 : 0, c10::cuda::getCurrentCUDAStream((c10::DeviceIndex)dev).stream()),
            "scaled_fp4_quant");
    }
    return wrap2(std::move(codes), std::move(sf));
  });
}

// cutlass_scaled_fp4_mm(a, b, block_scale_a, block_scale_b, alpha, out_dtype, out or None, tile_n) -> out
B200_FN(py_mm) {
  return guarded([&] {
    want_args(n_args, 8);
    const at::Tensor &a = tensor(args[0]), &b = tensor(args[1]), &sa = tensor(args[2]), &sb = tensor(args[3]), &alpha = tensor(args[4]);
    const int dev = require_cuda({&a, &b, &sa, &sb, &alpha});
    require(a.dim() == 2 && b.dim() == 2 && a.size(1) == b.size(1), "a [M,K/2] and b [N,K/2] must share K");
    require(a.scalar_type() == at::kByte && b.scalar_type() == at::kByte, "a and b must be uint8 (packed E2M1)");
    require(a.is_contiguous() && b.is_contiguous(), "a and b must be contiguous");
    const int64_t M = a.size(0), K = a.size(1) * 2, N = b.size(0);
    require(K % 64 == 0, "K must be a multiple of 64");
    auto want_scales = [&](const at::Tensor& t, int64_t rows, const char* name) {
      const size_t need = b200fp4_sf_swizzled_bytes(rows, K / 16);
      if (!t.is_contiguous() || t.nbytes() < need)
        throw std::runtime_error(std::string(name) + " must be the swizzled scale tensor of at least " + std::to_string(need) + " bytes");
    };
    want_scales(sa, M, "block_scale_a");
    want_scales(sb, N, "block_scale_b");
    require(is_f32_scalar(alpha), "alpha must be one f32");
    require(THPDtype_Check(args[5]), "out_dtype must be bfloat16 or float16");
    const at::ScalarType dt = reinterpret_cast<THPDtype*>(args[5])->scalar_type;
    require(dt == at::kBFloat16 || dt == at::kHalf, "out_dtype must be bfloat16 or float16");
    const at::Tensor* given = maybe_tensor(args[6]);
    if (given)
      require(given->is_cuda() && given->scalar_type() == dt && is_2d(*given, M, N) && given->is_contiguous(),
              "out must be a contiguous [M,N] CUDA tensor of out_dtype");
    const int tile_n = (int)integer(args[7]);
    at::Tensor out;
    {
      WithoutGil nogil;
      c10::cuda::CUDAGuard guard((c10::DeviceIndex)dev);
      out = given ? *given : empty({M, N}, dt, dev);
      cudaStream_t st = c10::cuda::getCurrentCUDAStream((c10::DeviceIndex)dev).stream();
      const Workspace ws(dev, st, b200fp4_gemm_workspace_bytes(M, N, K), kSlotGemm);
      check(b200fp4_gemm_nvfp4(ptr(a), ptr(b), ptr(sa), ptr(sb), ptr<float>(alpha), ptr(out), dtype_code(dt), M, N, K, tile_n, ws.data(),
                               ws.bytes(), st),
            "cutlass_scaled_fp4_mm");
    }
    if (given) {
      Py_INCREF(args[6]);
      return args[6];
    }
    return wrap(std::move(out));
  });
}

// nvfp4_linear(x, x_global_scale, w_codes, w_block_scale, alpha, out or None, tile_n) -> out
B200_FN(py_linear) {
  return guarded([&] {
    want_args(n_args, 7);
    const at::Tensor &x = tensor(args[0]), &gs = tensor(args[1]), &w = tensor(args[2]), &wsf = tensor(args[3]), &alpha = tensor(args[4]);
    const int dev = require_cuda({&x, &gs, &w, &wsf, &alpha});
    require(x.dim() == 2 && is_16bit(x) && x.stride(1) == 1, "x must be [M,K] bf16/f16, unit inner stride");
    require(w.dim() == 2 && w.scalar_type() == at::kByte && w.is_contiguous() && w.size(1) * 2 == x.size(1),
            "w_codes must be contiguous [N,K/2] uint8");
    const int64_t M = x.size(0), K = x.size(1), N = w.size(0);
    require(K % 64 == 0, "K must be a multiple of 64");
    require(wsf.is_contiguous() && wsf.nbytes() >= b200fp4_sf_swizzled_bytes(N, K / 16),
            "w_block_scale must be the swizzled scale tensor of the weight");
    require(is_f32_scalar(alpha) && is_f32_scalar(gs), "alpha and x_global_scale must be one f32 each");
    const at::Tensor* given = maybe_tensor(args[5]);
    if (given)
      require(given->is_cuda() && is_16bit(*given) && is_2d(*given, M, N) && given->is_contiguous(),
              "out must be a contiguous [M,N] 16-bit CUDA tensor");
    const int tile_n = (int)integer(args[6]);
    at::Tensor out;
    {
      WithoutGil nogil;
      c10::cuda::CUDAGuard guard((c10::DeviceIndex)dev);
      out = given ? *given : empty({M, N}, x.scalar_type(), dev);
      if (M > 0) {
        cudaStream_t st = c10::cuda::getCurrentCUDAStream((c10::DeviceIndex)dev).stream();
        const Workspace ws(dev, st, b200fp4_linear_workspace_bytes(M, N, K), kSlotLinear);
        check(b200fp4_linear_nvfp4(ptr(x), dtype_code(x.scalar_type()), M > 1 ? x.stride(0) : K, ptr<float>(gs), ptr(w), ptr(wsf),
                                   ptr<float>(alpha), ptr(out), dtype_code(out.scalar_type()), M, N, K, tile_n, ws.data(), ws.bytes(), st),
              "nvfp4_linear");
      }
    }
    if (given) {
      Py_INCREF(args[5]);
      return args[5];
    }
    return wrap(std::move(out));
  });
}

// ------------------------------------------------------------------------------------------ router

// moe_router(hidden, gate_weight, topk, renormalize) -> (weights, ids)
B200_FN(py_router) {
  return guarded([&] {
    want_args(n_args, 4);
    const at::Tensor &x = tensor(args[0]), &w = tensor(args[1]);
    const int64_t topk = integer(args[2]);
    const int dev = require_cuda({&x, &w});
    require(x.dim() == 2 && w.dim() == 2 && x.size(1) == w.size(1), "hidden_states [M,H] and gate_weight [E,H] must share H");
    require(x.scalar_type() == w.scalar_type() && is_16bit(x),
            "hidden_states and gate_weight must both be bfloat16 or both float16");
    require(x.stride(1) == 1 && w.is_contiguous(), "rows must be contiguous");
    const int64_t M = x.size(0), H = x.size(1), E = w.size(0);
    const int renormalize = truth(args[3]) ? 1 : 0;
    at::Tensor tw, ids;
    {
      WithoutGil nogil;
      c10::cuda::CUDAGuard guard((c10::DeviceIndex)dev);
      tw = empty({M, topk}, at::kFloat, dev);
      ids = empty({M, topk}, at::kInt, dev);
      cudaStream_t st = c10::cuda::getCurrentCUDAStream((c10::DeviceIndex)dev).stream();
      const Workspace ws(dev, st, b200fp4_moe_router_workspace_bytes(M, E), kSlotRouter);
      check(b200fp4_moe_router(ptr(x), M > 1 ? x.stride(0) : H, dtype_code(x.scalar_type()), ptr(w), M, H, E, topk, renormalize,
                               ptr<float>(tw), ptr<int32_t>(ids), ws.data(), ws.bytes(), st),
            "moe_router");
    }
    return wrap2(std::move(tw), std::move(ids));
  });
}

// ------------------------------------------------------------------------------------------ fused decode layer

// The weight side of a layer, bound once: the tensors are kept alive here, their checks are the Python constructor's.
struct BoundMoe {
  at::Tensor w13_comp, w13_meta, w13_scale, w13_g, w2_comp, w2_meta, w2_scale, w2_g, emap;
  int64_t H, I, E;
  int dev, flags;
};
constexpr const char* kMoeCapsule = "dgx_vllm_b200.bound_moe";

// moe_bind(w13_comp, w13_meta, w13_scale, w13_g, w2_comp, w2_meta, w2_scale, w2_g, expert_map or None, H, I, E, flags)
B200_FN(py_moe_bind) {
  return guarded([&] {
    want_args(n_args, 13);
    auto b = std::make_unique<BoundMoe>();
    at::Tensor* slots[8] = {&b->w13_comp, &b->w13_meta, &b->w13_scale, &b->w13_g, &b->w2_comp, &b->w2_meta, &b->w2_scale, &b->w2_g};
    for (int i = 0; i < 8; ++i) *slots[i] = tensor(args[i]);
    if (const at::Tensor* m = maybe_tensor(args[8])) b->emap = *m;
    b->H = integer(args[9]);
    b->I = integer(args[10]);
    b->E = integer(args[11]);
    b->flags = (int)integer(args[12]);
    b->dev = b->w13_comp.get_device();
    PyObject* cap = PyCapsule_New(b.get(), kMoeCapsule, [](PyObject* c) {
      delete static_cast<BoundMoe*>(PyCapsule_GetPointer(c, kMoeCapsule));
    });
    if (!cap) throw PythonError{};
    b.release();
    return cap;
  });
}

// moe_call(bound, hidden, topk_weights, topk_ids, apply_router_weight_on_input, out or None) -> out
B200_FN(py_moe_call) {
  return guarded([&] {
    want_args(n_args, 6);
    const BoundMoe* b = static_cast<BoundMoe*>(PyCapsule_GetPointer(args[0], kMoeCapsule));
    if (!b) throw PythonError{};
    const at::Tensor& x = tensor(args[1]);
    at::Tensor tw = tensor(args[2]), ids = tensor(args[3]);
    require(x.dim() == 2 && x.is_cuda() && x.size(1) == b->H && x.is_contiguous() && is_16bit(x),
            "hidden_states must be a contiguous [M,H] 16-bit CUDA tensor");
    require(tw.is_cuda() && ids.is_cuda() && ids.dim() == 2, "topk_weights / topk_ids must be contiguous [M, topk]");
    const int64_t M = x.size(0), topk = ids.size(1);
    const int flags = b->flags | (truth(args[4]) ? B200FP4_MOE_ROUTER_WEIGHT_ON_INPUT : 0);
    const at::Tensor* given = maybe_tensor(args[5]);
    at::Tensor out;
    {
      WithoutGil nogil;
      c10::cuda::CUDAGuard guard((c10::DeviceIndex)b->dev);
      if (tw.scalar_type() != at::kFloat) tw = tw.to(at::kFloat);
      if (ids.scalar_type() != at::kInt) ids = ids.to(at::kInt);
      require(tw.is_contiguous() && ids.is_contiguous() && is_2d(tw, M, topk) && ids.size(0) == M,
              "topk_weights / topk_ids must be contiguous [M, topk]");
      out = given ? *given : empty({M, b->H}, x.scalar_type(), b->dev);
      cudaStream_t st = c10::cuda::getCurrentCUDAStream((c10::DeviceIndex)b->dev).stream();
      const Workspace ws(b->dev, st, b200fp4_fused_moe_workspace_bytes(M, topk, b->H, b->I, b->E));
      check(b200fp4_fused_sparse_moe(
                ptr(x), dtype_code(x.scalar_type()), ptr<float>(tw), ptr<int32_t>(ids), b->emap.defined() ? ptr<int32_t>(b->emap) : nullptr,
                b->emap.defined() ? b->emap.numel() : 0, ptr<uint8_t>(b->w13_comp), ptr<uint8_t>(b->w13_meta), ptr<uint8_t>(b->w13_scale),
                ptr<float>(b->w13_g), b->w13_scale.size(1), ptr<uint8_t>(b->w2_comp), ptr<uint8_t>(b->w2_meta), ptr<uint8_t>(b->w2_scale),
                ptr<float>(b->w2_g), b->w2_scale.size(1), ptr(out), dtype_code(out.scalar_type()), M, topk, b->H, b->I, b->E, flags,
                ws.data(), ws.bytes(), st),
            "fused_sparse_moe_v7");
    }
    if (given) {
      Py_INCREF(args[5]);
      return args[5];
    }
    return wrap(std::move(out));
  });
}

// ------------------------------------------------------------------------------------------ prefill layer

at::Tensor as_i32(const at::Tensor& t) { return (t.scalar_type() == at::kInt ? t : t.to(at::kInt)).contiguous(); }

// moe_prefill(hidden, topk_weights, topk_ids, w13_codes, w13_sf, w2_codes, w2_sf, a1_gs, a2_gs, alpha1, alpha2,
//             expert_map or None) -> out.  topk <= 32, intermediate size a multiple of 128.
B200_FN(py_moe_prefill) {
  return guarded([&] {
    want_args(n_args, 12);
    const at::Tensor &x = tensor(args[0]), &tw_in = tensor(args[1]), &ids_in = tensor(args[2]), &w13 = tensor(args[3]),
                     &w13_sf = tensor(args[4]), &w2 = tensor(args[5]), &w2_sf = tensor(args[6]), &a1 = tensor(args[7]),
                     &a2 = tensor(args[8]), &al1 = tensor(args[9]), &al2 = tensor(args[10]);
    const at::Tensor* emap_in = maybe_tensor(args[11]);
    if (emap_in && emap_in->numel() == 0) emap_in = nullptr;
    const int dev = require_cuda({&x, &tw_in, &ids_in, &w13, &w13_sf, &w2, &w2_sf, &a1, &a2, &al1, &al2, emap_in});
    require(x.dim() == 2 && x.is_contiguous(), "input must be a contiguous 2-D tensor");
    require(is_16bit(x), "input must be float16 or bfloat16");
    require(w13.dim() == 3 && w2.dim() == 3 && ids_in.dim() == 2, "w13_codes [E,2I,H/2], w2_codes [E,H,I/2], topk_ids [M,topk]");
    const int64_t M = x.size(0), H = x.size(1), topk = ids_in.size(1), E = w13.size(0), N1 = w13.size(1), I = N1 / 2, P = M * topk;
    require(w13.size(2) * 2 == H && w2.size(0) == E && w2.size(1) == H && w2.size(2) * 2 == I && w13.is_contiguous() &&
                w2.is_contiguous(),
            "a and b must share K and be contiguous");
    require(H % 64 == 0 && I % 128 == 0 && topk > 0 && topk <= 32, "H % 64, the intermediate size % 128 and topk <= 32 are required");
    require(ids_in.size(0) == M && is_2d(tw_in, M, topk), "topk_weights and topk_ids must be [M, topk]");
    for (const at::Tensor* g : {&a1, &a2}) require(g->scalar_type() == at::kFloat && g->numel() >= E, "one f32 global scale per expert");
    for (const at::Tensor* g : {&al1, &al2}) require(g->scalar_type() == at::kFloat && g->numel() >= E, "one f32 alpha per expert");
    require(w13_sf.nbytes() >= (size_t)E * b200fp4_sf_swizzled_bytes(N1, H / 16) &&
                w2_sf.nbytes() >= (size_t)E * b200fp4_sf_swizzled_bytes(H, I / 16),
            "b_scales must hold one swizzled scale tensor per expert");
    at::Tensor out;
    {
      WithoutGil nogil;
      c10::cuda::CUDAGuard guard((c10::DeviceIndex)dev);
      const at::Tensor ids = as_i32(ids_in), tw = (tw_in.scalar_type() == at::kFloat ? tw_in : tw_in.to(at::kFloat)).contiguous();
      at::Tensor emap;
      if (emap_in) emap = as_i32(*emap_in);
      out = empty({M, H}, x.scalar_type(), dev);
      cudaStream_t st = c10::cuda::getCurrentCUDAStream((c10::DeviceIndex)dev).stream();
      const at::Tensor scratch = empty({(int64_t)b200fp4_moe_prefill_workspace_bytes(M, topk, H, I, E)}, at::kByte, dev);
      // the GEMMs' tile list and status word lie in the stream's scratch for GEMMs, where the status is read
      const Workspace gemm_ws(dev, st, b200fp4_grouped_gemm_workspace_bytes(P, E), kSlotGemm);
      check(b200fp4_moe_prefill(ptr(x), dtype_code(x.scalar_type()), ptr<float>(tw), ptr<int32_t>(ids),
                                emap.defined() ? ptr<int32_t>(emap) : nullptr, emap.defined() ? emap.numel() : 0, ptr(w13), ptr(w13_sf),
                                ptr<float>(al1), ptr(w2), ptr(w2_sf), ptr<float>(al2), ptr<float>(a1), ptr<float>(a2), ptr(out), M, topk,
                                H, I, E, ptr(scratch), scratch.nbytes(), gemm_ws.data(), st),
            "nvfp4_moe_prefill");
    }
    return wrap(std::move(out));
  });
}

PyMethodDef kMethods[] = {
    {"workspace", (PyCFunction)(void (*)())py_workspace, METH_FASTCALL, nullptr},
    {"scaled_fp4_quant", (PyCFunction)(void (*)())py_quant, METH_FASTCALL, nullptr},
    {"cutlass_scaled_fp4_mm", (PyCFunction)(void (*)())py_mm, METH_FASTCALL, nullptr},
    {"nvfp4_linear", (PyCFunction)(void (*)())py_linear, METH_FASTCALL, nullptr},
    {"moe_router", (PyCFunction)(void (*)())py_router, METH_FASTCALL, nullptr},
    {"moe_bind", (PyCFunction)(void (*)())py_moe_bind, METH_FASTCALL, nullptr},
    {"moe_call", (PyCFunction)(void (*)())py_moe_call, METH_FASTCALL, nullptr},
    {"moe_prefill", (PyCFunction)(void (*)())py_moe_prefill, METH_FASTCALL, nullptr},
    {nullptr, nullptr, 0, nullptr}};

PyModuleDef kModule = {PyModuleDef_HEAD_INIT, "b200_host", "Host path of the torch-facing NVFP4 ops.", -1, kMethods,
                       nullptr, nullptr, nullptr, nullptr};

}  // namespace

extern "C" __attribute__((visibility("default"))) PyObject* PyInit_b200_host(void) { return PyModule_Create(&kModule); }

// Python extension `_host_calls`: the host side of one analog call (nn/functional.py) -- outputs, tensors kept for the
// backward pass, workspaces, the argument block, the library call.  What bounds a small layer is this path and not
// its kernels (a 1 x 2048 x 2048 evaluation: 11 us of kernels): a torch.empty from Python costs about 2.4 us and an
// fp32 training step made fourteen of them next to some sixty ctypes field assignments.
//
// Both functions are positional (METH_FASTCALL), take and return torch tensors and return the library's status first;
// the caller turns a status into the exception it stands for.  The library call runs without the GIL.
#include <Python.h>

#include <ATen/ATen.h>
#include <c10/core/DeviceGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>

#include <mutex>

#include "../../include/analog_b200.h"

// what the loader and the build look for in this file before they use it
__attribute__((used)) extern const char al_host_built_for[] = "built for torch " AL_TORCH_VERSION ";";

namespace {

// a positional argument: a tensor, or None
const at::Tensor* tensor_or_null(PyObject* o) {
  if (o == Py_None) return nullptr;
  TORCH_CHECK_TYPE(THPVariable_Check(o), "expected a tensor or None");
  return &THPVariable_Unpack(o);
}
const at::Tensor& tensor_of(PyObject* o) {
  TORCH_CHECK_TYPE(THPVariable_Check(o), "expected a tensor");
  return THPVariable_Unpack(o);
}
void* ptr_of(const at::Tensor* t) { return t ? t->data_ptr() : nullptr; }
void* ptr_of(const at::Tensor& t) { return t.defined() ? t.data_ptr() : nullptr; }
bool truth(PyObject* o) { return PyObject_IsTrue(o) == 1; }

PyObject* wrap(const at::Tensor& t) {
  if (t.defined()) return THPVariable_Wrap(t);
  Py_RETURN_NONE;
}

// A ctypes structure or array (borrowed while the call runs)
struct Block {
  Py_buffer view{};
  Block(PyObject* o, size_t at_least) {
    TORCH_CHECK_TYPE(PyObject_GetBuffer(o, &view, PyBUF_WRITABLE) == 0, "expected a ctypes structure");
    if ((size_t)view.len < at_least) {
      PyBuffer_Release(&view);
      TORCH_CHECK_VALUE(false, "ctypes structure too small");
    }
  }
  Block(const Block&) = delete;
  ~Block() { PyBuffer_Release(&view); }
};

int64_t round_up(int64_t v, int64_t to) { return (v + to - 1) / to * to; }

// Workspace that nothing keeps beyond the call: one allocation, carved by offset
struct Arena {
  int64_t bytes = 0;
  struct Slot {
    void** where;
    int64_t offset;
  } slots[12];
  int n = 0;
  void add(void** where, int64_t size) {
    slots[n++] = Slot{where, bytes};
    bytes += round_up(size, 256);
  }
  at::Tensor place(const at::TensorOptions& like) {
    at::Tensor t;
    if (n == 0) return t;
    t = at::empty({bytes}, like.dtype(at::kByte));
    char* base = static_cast<char*>(t.data_ptr());
    for (int i = 0; i < n; ++i) *slots[i].where = base + slots[i].offset;
    return t;
  }
};

enum ForwardArg {
  F_DESC, F_ENDS, F_X, F_W, F_BIAS, F_IR, F_IDX, F_XMIN, F_XMAX, F_LWC, F_STD, F_WNOISE, F_ONOISE, F_PRE_XQ, F_PRE_IR,
  F_PRE_CODES, F_PREQUANT, F_MODIFIES, F_NEED_STD, F_KEEP, F_CAPTURE, F_WANT_CODES, F_DRAW, F_SEED, F_OFFSET, F_BASE, F_COUNT
};

// -> (status, out, xq, ir_rows, w_amax, w_tile_max, w_mod, keep_mask, codes, codes16, w_planes)
// KEEP: a backward pass will follow.  CAPTURE: the caller also wants the statistics.  DRAW: the noise counter comes
// from torch's generator of the device (advanced as a kernel drawing four values per thread would); otherwise SEED,
// OFFSET and BASE say it.
PyObject* forward(PyObject*, PyObject* const* a, Py_ssize_t nargs) {
  HANDLE_TH_ERRORS
  TORCH_CHECK_VALUE(nargs == F_COUNT, "forward: wrong number of arguments");
  Block desc_block(a[F_DESC], sizeof(AlDesc)), ends_block(a[F_ENDS], sizeof(int32_t));
  AlDesc& d = *static_cast<AlDesc*>(desc_block.view.buf);
  const int32_t* ends = static_cast<const int32_t*>(ends_block.view.buf);
  TORCH_CHECK_VALUE(d.T >= 1 && ends_block.view.len >= (Py_ssize_t)(d.T * sizeof(int32_t)), "forward: tile ends missing");
  const at::Tensor* x = tensor_or_null(a[F_X]);
  const at::Tensor& w = tensor_of(a[F_W]);
  const bool modifies = truth(a[F_MODIFIES]), need_std = truth(a[F_NEED_STD]), keep = truth(a[F_KEEP]);
  const bool capture = truth(a[F_CAPTURE]), replay = a[F_WNOISE] != Py_None || a[F_ONOISE] != Py_None;
  const long prequant = PyLong_AsLong(a[F_PREQUANT]);
  const bool is_static = d.ir_mode == AL_IR_STATIC || d.ir_mode == AL_IR_FAST;
  const int64_t m = d.M, k = d.K, n = d.N, t = d.T, es = d.dtype == AL_BF16 ? 2 : 4;
  const auto opt = at::TensorOptions().dtype(w.scalar_type()).device(w.device());
  const c10::DeviceGuard guard(w.device());

  AlForwardArgs args{};
  args.x = prequant ? nullptr : ptr_of(x);
  args.w = w.data_ptr();
  args.bias = ptr_of(tensor_or_null(a[F_BIAS]));
  args.input_range = ptr_of(tensor_or_null(a[F_IR]));
  args.input_range_update_idx = ptr_of(tensor_or_null(a[F_IDX]));
  args.x_min = ptr_of(tensor_or_null(a[F_XMIN]));
  args.x_max = ptr_of(tensor_or_null(a[F_XMAX]));
  args.learnable_weight_clip = ptr_of(tensor_or_null(a[F_LWC]));
  args.std_override = static_cast<const float*>(ptr_of(tensor_or_null(a[F_STD])));
  args.w_noise = ptr_of(tensor_or_null(a[F_WNOISE]));
  args.out_noise = ptr_of(tensor_or_null(a[F_ONOISE]));
  args.x_prequantised = (int32_t)prequant;
  args.tile_ends = ends;
  at::Tensor out = at::empty({m, n}, opt);
  args.out = out.data_ptr();

  // sizes that are no multiples of 8: the tensor-core route takes its operands in a pitched layout (a layer whose
  // pitch equals K reads x and w themselves where nothing modifies them: those must be aligned)
  int64_t k_rows = k;
  if (d.dtype == AL_BF16 && !prequant && !capture && !replay &&
      (n % 8 || k % 8 || ends[0] % 8 || (t > 1 && (ends[t - 1] - ends[t - 2]) % 8))) {
    const int32_t pitch = al_operand_pitch(&d, ends);
    if (pitch != 0 && (pitch != k || !(((uintptr_t)args.x | (uintptr_t)args.w) % 16))) {
      d.engine = AL_ENGINE_PITCHED;
      k_rows = pitch;
    }
  }
  const bool pitched = k_rows != k;
  // fp32 layer on the tensor cores: the GEMMs read the DAC codes and the weights as bf16 planes
  const bool planes = d.dtype == AL_F32 && al_uses_tcgen05(&d, ends);

  at::Tensor xq, ir_rows, w_amax, w_tile_max, w_mod, keep_mask, codes, codes16, w_planes;
  Arena arena;
  const auto place = [&](bool kept, at::Tensor* tensor, void** where, at::IntArrayRef shape, at::ScalarType type) {
    if (!kept) {
      int64_t count = 1;
      for (int64_t s : shape) count *= s;
      arena.add(where, count * (int64_t)c10::elementSize(type));
      return;
    }
    *tensor = at::empty(shape, opt.dtype(type));
    *where = tensor->data_ptr();
  };
  const at::ScalarType type = w.scalar_type();
  // with bf16 planes the backward GEMMs read those: the fp32 copies are kept only for the CUDA-core input gradient
  // of a layer with fewer than 64 channels
  const bool keep_xq = capture || (keep && !planes), keep_wmod = capture || (keep && !(planes && n >= 64));
  // such a layer writes neither fp32 copy at all where nothing reads it (al_forward: codes_only, weight_planes)
  const bool codes_only = planes && !capture && !prequant && (uintptr_t)args.x % 16 == 0;
  const bool planes_only = planes && !capture && !replay && n >= 64 && d.quant_type == AL_QUANT_NONE &&
                           !(d.training && d.noise_type == AL_NOISE_ADD_NORMAL) &&
                           d.clip_type != AL_CLIP_LEARNABLE_PER_CHANNEL && (uintptr_t)args.w % 16 == 0;
  if (prequant) {
    args.xq = ptr_of(tensor_or_null(a[F_PRE_XQ]));
    args.ir_rows = ptr_of(tensor_or_null(a[F_PRE_IR]));
  } else if (d.ir_mode != AL_IR_OFF || pitched) {
    if (!codes_only) place(keep_xq, &xq, &args.xq, {m, k_rows}, type);
    if (is_static) place(keep || capture, &ir_rows, &args.ir_rows, {t}, type);
    else place(keep || capture, &ir_rows, &args.ir_rows, {t, m}, type);
  } else {
    args.xq = const_cast<void*>(args.x);
  }
  place(capture, &w_amax, &args.w_amax, {t, n}, type);
  place(capture, &w_tile_max, &args.w_tile_max, {2 * t}, at::kFloat);
  if (modifies && planes_only) args.w_mod = nullptr;
  else if (modifies || pitched) place(keep_wmod, &w_mod, &args.w_mod, {n, k_rows}, type);
  else args.w_mod = const_cast<void*>(args.w);
  if (d.out_bound > 0 && keep) place(true, &keep_mask, reinterpret_cast<void**>(&args.keep_mask), {t, (n + 31) / 32, m}, at::kInt);
  if (need_std) arena.add(reinterpret_cast<void**>(&args.std_scratch), al_std_scratch_floats(d.M, d.T) * 4);
  if (m <= 16 && !keep && !capture && d.dtype == AL_BF16)
    arena.add(reinterpret_cast<void**>(&args.smallm_scratch), al_smallm_scratch_floats(d.M, d.N, d.T) * 4);
  if (planes) {
    place(keep || capture, &w_planes, &args.w_planes, {al_f32_planes(), n, k}, at::kBFloat16);
    if (a[F_PRE_CODES] != Py_None) args.codes16 = ptr_of(tensor_or_null(a[F_PRE_CODES]));
    else place(keep || capture, &codes16, &args.codes16, {m, k}, at::kBFloat16);
  } else {
    args.codes16 = nullptr;
  }
  if (truth(a[F_WANT_CODES])) place(true, &codes, &args.codes, {m, k}, type);
  const at::Tensor workspace = arena.place(opt);

  if (truth(a[F_DRAW])) {
    at::Generator gen = at::globalContext().defaultGenerator(w.device());
    const std::lock_guard<std::mutex> lock(gen.mutex());
    args.seed = gen.current_seed();
    args.offset = gen.get_offset();
    gen.set_offset(args.offset + 4);
  } else {
    args.seed = PyLong_AsUnsignedLongLongMask(a[F_SEED]);
    args.offset = PyLong_AsUnsignedLongLongMask(a[F_OFFSET]);
    args.offset_base = reinterpret_cast<const uint64_t*>(PyLong_AsUnsignedLongLongMask(a[F_BASE]));
  }
  if (PyErr_Occurred()) return nullptr;
  const cudaStream_t stream = c10::cuda::getCurrentCUDAStream(w.device().index()).stream();
  int status;
  Py_BEGIN_ALLOW_THREADS
  status = al_forward(&d, &args, stream);
  Py_END_ALLOW_THREADS
  PyObject* const items[] = {PyLong_FromLong(status), wrap(out), wrap(xq), wrap(ir_rows), wrap(w_amax), wrap(w_tile_max),
                             wrap(w_mod), wrap(keep_mask), wrap(codes), wrap(codes16), wrap(w_planes)};
  constexpr int kItems = sizeof(items) / sizeof(items[0]);
  PyObject* result = PyTuple_New(kItems);
  for (int i = 0; i < kItems; ++i) PyTuple_SET_ITEM(result, i, items[i]);
  return result;
  END_HANDLE_TH_ERRORS
}

enum BackwardArg {
  B_DESC, B_ENDS, B_G, B_X, B_XQ, B_WMOD, B_IR, B_MASK, B_W, B_LWC, B_CODES, B_PLANES, B_NEED_X, B_GRAD_W, B_NEED_W, B_NEED_B,
  B_NEED_IR, B_NEED_CLIP, B_COUNT
};

// -> (status, grad_x, grad_w, grad_b, grad_ir, grad_clip); GRAD_W: where the weight gradient goes (None: a fresh tensor)
PyObject* backward(PyObject*, PyObject* const* a, Py_ssize_t nargs) {
  HANDLE_TH_ERRORS
  TORCH_CHECK_VALUE(nargs == B_COUNT, "backward: wrong number of arguments");
  Block desc_block(a[B_DESC], sizeof(AlDesc)), ends_block(a[B_ENDS], sizeof(int32_t));
  const AlDesc& d = *static_cast<const AlDesc*>(desc_block.view.buf);
  const int32_t* ends = static_cast<const int32_t*>(ends_block.view.buf);
  TORCH_CHECK_VALUE(d.T >= 1 && ends_block.view.len >= (Py_ssize_t)(d.T * sizeof(int32_t)), "backward: tile ends missing");
  const at::Tensor& g = tensor_of(a[B_G]);
  const int64_t m = d.M, k = d.K, n = d.N, t = d.T;
  const auto opt = at::TensorOptions().dtype(g.scalar_type()).device(g.device());
  const c10::DeviceGuard guard(g.device());

  AlBackwardArgs args{};
  args.tile_ends = ends;
  args.grad_out = g.data_ptr();
  args.x = ptr_of(tensor_or_null(a[B_X]));
  args.xq = ptr_of(tensor_or_null(a[B_XQ]));
  args.w_mod = ptr_of(tensor_or_null(a[B_WMOD]));
  args.ir_rows = ptr_of(tensor_or_null(a[B_IR]));
  args.keep_mask = static_cast<const uint32_t*>(ptr_of(tensor_or_null(a[B_MASK])));
  args.codes16 = ptr_of(tensor_or_null(a[B_CODES]));
  args.w_planes = ptr_of(tensor_or_null(a[B_PLANES]));
  at::Tensor grad_x, grad_w, grad_b, grad_ir, grad_clip;
  if (truth(a[B_NEED_X])) grad_x = at::empty({m, k}, opt);
  if (truth(a[B_NEED_W])) {
    if (a[B_GRAD_W] != Py_None) grad_w = tensor_of(a[B_GRAD_W]);
    else grad_w = at::empty({n, k}, opt);
  }
  if (truth(a[B_NEED_B])) grad_b = at::empty({n}, opt);
  if (truth(a[B_NEED_IR])) grad_ir = at::empty({t}, opt);
  if (truth(a[B_NEED_CLIP])) {
    grad_clip = at::empty({t, n}, opt);
    args.w = ptr_of(tensor_or_null(a[B_W]));
    args.learnable_weight_clip = ptr_of(tensor_or_null(a[B_LWC]));
  }
  args.grad_x = ptr_of(grad_x);
  args.grad_w = ptr_of(grad_w);
  args.grad_bias = ptr_of(grad_b);
  args.grad_input_range = ptr_of(grad_ir);
  args.grad_weight_clip = ptr_of(grad_clip);
  Arena arena;
  args.reduce_scratch_floats = al_backward_scratch_floats(d.M, d.K, d.N, d.T);
  arena.add(reinterpret_cast<void**>(&args.reduce_scratch), args.reduce_scratch_floats * 4);
  if (args.codes16) args.g_planes_elems = al_backward_plane_elems(&d, ends);
  else if (d.engine == AL_ENGINE_PITCHED && (n % 8 || (uintptr_t)args.grad_out % 16)) args.g_planes_elems = m * round_up(n, 8);
  if (args.g_planes_elems > 0) arena.add(&args.g_planes, args.g_planes_elems * 2);
  const at::Tensor workspace = arena.place(opt);
  const cudaStream_t stream = c10::cuda::getCurrentCUDAStream(g.device().index()).stream();
  int status;
  Py_BEGIN_ALLOW_THREADS
  status = al_backward(&d, &args, stream);
  Py_END_ALLOW_THREADS
  PyObject* const items[] = {PyLong_FromLong(status), wrap(grad_x), wrap(grad_w), wrap(grad_b), wrap(grad_ir), wrap(grad_clip)};
  constexpr int kItems = sizeof(items) / sizeof(items[0]);
  PyObject* result = PyTuple_New(kItems);
  for (int i = 0; i < kItems; ++i) PyTuple_SET_ITEM(result, i, items[i]);
  return result;
  END_HANDLE_TH_ERRORS
}

PyMethodDef methods[] = {
    {"forward", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(forward)), METH_FASTCALL, nullptr},
    {"backward", reinterpret_cast<PyCFunction>(reinterpret_cast<void (*)()>(backward)), METH_FASTCALL, nullptr},
    {nullptr, nullptr, 0, nullptr}};
PyModuleDef module_def = {PyModuleDef_HEAD_INIT, "_host_calls", nullptr, -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__host_calls(void) { return PyModule_Create(&module_def); }

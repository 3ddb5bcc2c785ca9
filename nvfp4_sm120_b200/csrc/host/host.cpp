// Host side of the quantizer and GEMM entry points: argument handling, output allocation, stream lookup and the calls
// into libnvfp4_b200.so, in C++.  quant.py and gemm.py keep the public functions, their defaults and the seed counter
// and call in here.
//
// Why native: the small calls of this path are bound by the host.  One quantization took 25 us through Python (a
// device context manager, three torch.empty, a ctypes call with sixteen arguments) for 6 us of kernel, an FP4Linear
// step of 512 tokens 484 us for 74 us of kernels.
#include <dlfcn.h>

#include <mutex>
#include <unordered_map>

#include <ATen/ATen.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/utils/pybind.h>

#include "nvfp4_b200.h"

namespace py = pybind11;

namespace {

#define NVFP4_FOR_EACH(F)                                                                                              \
  F(nvfp4_amax_bf16) F(nvfp4_amax_both_bf16) F(nvfp4_quantize_fused_bf16) F(nvfp4_quantize_shard_bf16)                 \
  F(nvfp4_quantize_weight_bf16) F(nvfp4_quantize_dual_bf16) F(nvfp4_round_amax_f32) F(nvfp4_gemm) F(nvfp4_gemm_amax) \
  F(nvfp4_gemm_bf16_as_f32)

struct Library {
#define F(name) decltype(&::name) name = nullptr;
  NVFP4_FOR_EACH(F)
#undef F
} lib;

// Python callables of _lib.py: check(code, what) and cuda_device_of(*tensors), which raise the package's exceptions
py::object* g_check = nullptr;
py::object* g_device_of = nullptr;

void init(const std::string& path, py::object check, py::object device_of) {
  void* h = dlopen(path.c_str(), RTLD_NOW | RTLD_LOCAL);
  if (h == nullptr) throw std::runtime_error(std::string("dlopen failed: ") + dlerror());
#define F(name)                                                                        \
  lib.name = reinterpret_cast<decltype(lib.name)>(dlsym(h, #name));                     \
  if (lib.name == nullptr) throw std::runtime_error(path + " does not export " #name);
  NVFP4_FOR_EACH(F)
#undef F
  g_check = new py::object(std::move(check));          // live as long as the process
  g_device_of = new py::object(std::move(device_of));
}

void check(int code, const char* what) {
  if (code != 0) (*g_check)(code, what);
}

[[noreturn]] void raise(PyObject* type, const std::string& msg) {
  PyErr_SetString(type, msg.c_str());
  throw py::error_already_set();
}

using OptTensor = c10::optional<at::Tensor>;

const at::Tensor* ptr_of(const OptTensor& t) { return t.has_value() ? &*t : nullptr; }

// The one CUDA device of all operands; anything else goes to _lib.cuda_device_of, which says what is wrong.
c10::Device device_of(std::initializer_list<const at::Tensor*> ts) {
  c10::optional<c10::Device> dev;
  bool good = true;
  for (const at::Tensor* t : ts) {
    if (t == nullptr) continue;
    if (!t->is_cuda() || (dev.has_value() && *dev != t->device())) { good = false; break; }
    dev = t->device();
  }
  if (!good || !dev.has_value()) {
    py::list l;
    for (const at::Tensor* t : ts) {
      if (t == nullptr) l.append(py::none());
      else l.append(py::cast(*t));
    }
    (*g_device_of)(*l);
    throw std::runtime_error("operands are not on one CUDA device");
  }
  return *dev;
}

void* stream_of(c10::Device dev) { return c10::cuda::getCurrentCUDAStream(dev.index()).stream(); }

// ---- scratch words ----------------------------------------------------------------------------------------------
struct Key {
  int device;
  void* stream;
  bool operator==(const Key& o) const { return device == o.device && stream == o.stream; }
};
struct KeyHash {
  size_t operator()(const Key& k) const { return std::hash<void*>()(k.stream) * 31 + (size_t)k.device; }
};
std::mutex g_mutex;
// never destroyed: tensors must not be freed after the CUDA context is gone
auto& g_workspaces = *new std::unordered_map<Key, at::Tensor, KeyHash>();
auto& g_status = *new std::unordered_map<int, at::Tensor>();
auto& g_ones = *new std::unordered_map<int, at::Tensor>();

// The entry of `key`, made by `make` if there is none.  The lock is not held while it is made: a dispatch mode may run Python
// there, which can give up the GIL or come back in here.  Of two tensors made at once the first one in stays.
template <class Map, class Make> at::Tensor find_or_make(Map& map, const typename Map::key_type& key, Make make) {
  {
    std::lock_guard<std::mutex> lock(g_mutex);
    const auto it = map.find(key);
    if (it != map.end()) return it->second;
  }
  at::Tensor made = make();
  std::lock_guard<std::mutex> lock(g_mutex);
  return map.emplace(key, std::move(made)).first->second;
}

at::TensorOptions on(c10::Device dev, at::ScalarType t) { return at::TensorOptions().device(dev).dtype(t); }

// 64-byte scratch of the single-launch quantizer, zeroed once, one per (device, stream): every launch leaves it ready
// for the next, and launches on one stream never overlap
at::Tensor workspace(int device) {
  const c10::Device dev(c10::kCUDA, (c10::DeviceIndex)device);
  const Key key{device, stream_of(dev)};
  return find_or_make(g_workspaces, key, [&] { return at::zeros({16}, on(dev, at::kInt)); });
}
// the workspace of the current stream if there is one yet
OptTensor workspace_if_any(int device) {
  const Key key{device, stream_of(c10::Device(c10::kCUDA, (c10::DeviceIndex)device))};
  std::lock_guard<std::mutex> lock(g_mutex);
  auto it = g_workspaces.find(key);
  return it == g_workspaces.end() ? OptTensor() : OptTensor(it->second);
}
at::Tensor status_word(int device) {
  return find_or_make(g_status, device,
                      [&] { return at::zeros({1}, on(c10::Device(c10::kCUDA, (c10::DeviceIndex)device), at::kInt)); });
}

at::Tensor signs_on(const OptTensor& signs, c10::Device dev) {
  if (!signs.has_value()) return find_or_make(g_ones, dev.index(), [&] { return at::ones({16}, on(dev, at::kFloat)); });
  at::Tensor s = *signs;
  if (s.device() != dev || s.scalar_type() != at::kFloat) s = s.to(dev, at::kFloat);
  s = s.contiguous();
  if (s.numel() != 16) raise(PyExc_ValueError, "signs must have 16 entries");
  return s;
}

void check_matrix(const at::Tensor& t) {
  if (t.dim() != 2) raise(PyExc_ValueError, "expected a 2-D tensor");
  if (!t.is_cuda()) device_of({&t});
}
// rows the kernels can read: unit column stride, a row pitch of 16-byte multiples, a 16-byte aligned start
bool readable_rows(const at::Tensor& x) {
  return x.stride(1) == 1 && x.stride(0) * x.element_size() % 16 == 0 && x.stride(0) >= x.size(1) &&
         reinterpret_cast<uintptr_t>(x.data_ptr()) % 16 == 0;
}
at::Tensor as_bf16_rows(const at::Tensor& t) {
  check_matrix(t);
  const at::Tensor x = t.scalar_type() == at::kBFloat16 ? t : t.to(at::kBFloat16);
  return readable_rows(x) ? x : x.contiguous();
}

// An fp32 matrix whose bf16 rounding and maximum (both maxima with signs: after the Hadamard transform along the rows
// too) one kernel finds: (bf16 copy, maxima).  For shapes that the kernel takes and memory it can read as it is: the
// cast of any other matrix makes an aligned copy, where an fp32 copy in front of this kernel would be a pass more.
bool can_round(const at::Tensor& t, bool rht) {
  return t.scalar_type() == at::kFloat && t.size(0) > 0 && t.size(1) > 0 && t.size(1) % 8 == 0 &&
         (!rht || t.size(0) % 16 == 0) && t.size(0) <= 64 * 65535LL && readable_rows(t) && !t.is_neg();
}
std::pair<at::Tensor, at::Tensor> round_amax(const at::Tensor& x, const at::Tensor* signs) {
  const c10::Device dev = device_of({&x, signs});
  at::Tensor out = at::empty({x.size(0), x.size(1)}, on(dev, at::kBFloat16));
  at::Tensor maxima = at::empty({signs != nullptr ? 2 : 1}, on(dev, at::kFloat));
  check(lib.nvfp4_round_amax_f32(static_cast<const float*>(x.data_ptr()), x.size(0), x.size(1), x.stride(0), out.data_ptr(),
                                 signs != nullptr ? static_cast<const float*>(signs->data_ptr()) : nullptr,
                                 static_cast<float*>(maxima.data_ptr()), 1, stream_of(dev)),
        "nvfp4_round_amax_f32");
  return {out, maxima};
}

struct Operand {
  at::Tensor q, s, p;
  uint8_t* qp() { return q.data_ptr<uint8_t>(); }
  uint8_t* sp() { return static_cast<uint8_t*>(s.data_ptr()); }
  float* pp() { return p.data_ptr<float>(); }
};
Operand alloc(c10::Device dev, int64_t m, int64_t k, bool scalar = true) {
  Operand o;
  o.q = at::empty({m, k / 2}, on(dev, at::kByte));
  o.s = at::empty({(m + 127) / 128 * 128, (k / 16 + 3) / 4 * 4}, on(dev, at::kFloat8_e4m3fn));
  if (scalar) o.p = at::empty({}, on(dev, at::kFloat));
  return o;
}

float* float_ptr(const at::Tensor& t) { return static_cast<float*>(t.data_ptr()); }

at::Tensor amax_rows(const at::Tensor& x, bool rht, const at::Tensor* sg, bool transpose, const OptTensor& out) {
  const at::Tensor a = out.has_value() ? *out : at::empty({1}, on(x.device(), at::kFloat));
  const c10::Device dev = device_of({&x, &a, sg});
  check(lib.nvfp4_amax_bf16(x.data_ptr(), x.size(0), x.size(1), x.stride(0), rht, transpose,
                            rht ? float_ptr(*sg) : nullptr, float_ptr(a), 1, stream_of(dev)),
        "nvfp4_amax_bf16");
  return a;
}

at::Tensor amax(const at::Tensor& t, bool rht, const OptTensor& signs, bool transpose, const OptTensor& out) {
  check_matrix(t);
  const c10::cuda::CUDAGuard guard(t.device());
  const at::Tensor x = as_bf16_rows(t);
  at::Tensor sg;
  if (rht) sg = signs_on(signs, x.device());
  return amax_rows(x, rht, rht ? &sg : nullptr, transpose, out);
}

at::Tensor amax_both_rows(const at::Tensor& x, const at::Tensor& sg) {
  const c10::Device dev = device_of({&x, &sg});
  at::Tensor m = at::empty({2}, on(dev, at::kFloat));
  check(lib.nvfp4_amax_both_bf16(x.data_ptr(), x.size(0), x.size(1), x.stride(0), float_ptr(sg), float_ptr(m), 1,
                                 stream_of(dev)),
        "nvfp4_amax_both_bf16");
  return m;
}

at::Tensor amax_both(const at::Tensor& t, const OptTensor& signs) {
  check_matrix(t);
  const c10::cuda::CUDAGuard guard(t.device());
  const at::Tensor x = as_bf16_rows(t);
  return amax_both_rows(x, signs_on(signs, x.device()));
}

// shard: pitch and base number the blocks; otherwise the tensor is whole
py::tuple quantize(const at::Tensor& t, bool stochastic, bool rht, const OptTensor& signs, uint64_t seed, bool transpose,
                   const OptTensor& amax_in, uint64_t offset, bool fused, bool shard, uint64_t pitch, uint64_t base) {
  check_matrix(t);
  const c10::cuda::CUDAGuard guard(t.device());
  // fp32 without a known maximum: the rounding finds it on the way.  Row-wise the single-launch kernel needs no pass of
  // its own for it, so there this pays only from 4M elements on (one read of the bf16 copy against one more launch).
  at::Tensor x, found;
  if (!amax_in.has_value() && !rht && fused && can_round(t, false) && (transpose || t.numel() >= (1 << 22)))
    std::tie(x, found) = round_amax(t, nullptr);
  else
    x = as_bf16_rows(t);
  const at::Tensor* known = amax_in.has_value() ? &*amax_in : (found.defined() ? &found : nullptr);
  const int64_t rows = x.size(0), cols = x.size(1), m = transpose ? cols : rows, k = transpose ? rows : cols;
  if (k % 16 != 0) raise(PyExc_AssertionError, "K=" + std::to_string(k) + " must be divisible by 16");
  at::Tensor sg;
  if (rht) sg = signs_on(signs, x.device());
  const c10::Device dev = device_of({&x, rht ? &sg : nullptr, known});
  Operand o = alloc(dev, m, k);
  void* stream = stream_of(dev);
  const float* sgp = rht ? float_ptr(sg) : nullptr;
  if (fused && known == nullptr && !transpose && rows * (cols / 16) < (1LL << 31)) {
    at::Tensor ws = workspace(dev.index());
    check(lib.nvfp4_quantize_fused_bf16(x.data_ptr(), rows, cols, x.stride(0), stochastic, rht, sgp, seed, offset, o.qp(),
                                        o.sp(), o.pp(), ws.data_ptr(), 64, stream),
          "nvfp4_quantize_fused_bf16");
    return py::make_tuple(o.q, o.s, o.p);
  }
  const at::Tensor a = known != nullptr ? *known : amax_rows(x, rht, rht ? &sg : nullptr, transpose, OptTensor());
  check(lib.nvfp4_quantize_shard_bf16(x.data_ptr(), rows, cols, x.stride(0), transpose, stochastic, rht, sgp, float_ptr(a),
                                      seed, offset, shard ? pitch : (uint64_t)(k / 16), shard ? base : 0, o.qp(),
                                      o.sp(), o.pp(), stream),
        "nvfp4_quantize_shard_bf16");
  return py::make_tuple(o.q, o.s, o.p);
}

// (q, scales) of w and of w^T and their one per-tensor scale
py::tuple quantize_weight(const at::Tensor& w, const OptTensor& amax_in, bool two_d) {
  check_matrix(w);
  const c10::cuda::CUDAGuard guard(w.device());
  at::Tensor x, a;
  if (!amax_in.has_value() && can_round(w, false)) std::tie(x, a) = round_amax(w, nullptr);
  else x = as_bf16_rows(w);
  const int64_t rows = x.size(0), cols = x.size(1);
  if (rows % 16 != 0 || cols % 16 != 0)
    raise(PyExc_AssertionError, "weight dims " + std::to_string(rows) + "x" + std::to_string(cols) + " must be divisible by 16");
  if (amax_in.has_value()) a = *amax_in;
  else if (!a.defined()) a = amax_rows(x, false, nullptr, false, OptTensor());
  const c10::Device dev = device_of({&x, &a});
  Operand r = alloc(dev, rows, cols), c = alloc(dev, cols, rows, false);
  check(lib.nvfp4_quantize_weight_bf16(x.data_ptr(), rows, cols, x.stride(0), two_d, float_ptr(a), r.qp(), r.sp(), c.qp(),
                                       c.sp(), r.pp(), stream_of(dev)),
        "nvfp4_quantize_weight_bf16");
  return py::make_tuple(r.q, r.s, c.q, c.s, r.p);
}

// counters: empty, or pitch and base of the row-wise and of the transposed layout
py::tuple quantize_dual(const at::Tensor& t, const OptTensor& signs, const OptTensor& amax_r, const OptTensor& amax_c,
                        bool sr_rows, bool sr_cols, uint64_t seed_r, uint64_t seed_c, uint64_t offset,
                        const std::vector<uint64_t>& counters) {
  check_matrix(t);
  const c10::cuda::CUDAGuard guard(t.device());
  const int64_t rows = t.size(0), cols = t.size(1);
  if (rows % 16 != 0 || cols % 16 != 0)
    raise(PyExc_AssertionError, "dims " + std::to_string(rows) + "x" + std::to_string(cols) + " must be divisible by 16");
  const at::Tensor sg = signs_on(signs, t.device());
  at::Tensor x, r, c, both;                                  // `both`: the two maxima found here
  if (amax_r.has_value()) r = *amax_r;
  if (amax_c.has_value()) c = *amax_c;
  if (!r.defined() && !c.defined() && can_round(t, true)) std::tie(x, both) = round_amax(t, &sg);
  else x = as_bf16_rows(t);
  if (both.defined()) {}
  else if (!r.defined() && !c.defined()) both = amax_both_rows(x, sg);
  else if (!c.defined()) c = amax_rows(x, true, &sg, true, OptTensor());
  else if (!r.defined()) r = amax_rows(x, false, nullptr, false, OptTensor());
  const c10::Device dev = device_of({&x, &sg, r.defined() ? &r : nullptr, c.defined() ? &c : nullptr});
  const float* rp = both.defined() ? float_ptr(both) : float_ptr(r);
  const float* cp = both.defined() ? float_ptr(both) + 1 : float_ptr(c);
  Operand a = alloc(dev, rows, cols), b = alloc(dev, cols, rows);
  check(lib.nvfp4_quantize_dual_bf16(x.data_ptr(), rows, cols, x.stride(0), sr_rows, sr_cols, float_ptr(sg), rp, cp, seed_r,
                                     seed_c, offset, counters.size() == 4 ? counters.data() : nullptr, a.qp(), a.sp(),
                                     a.pp(), b.qp(), b.sp(), b.pp(), stream_of(dev)),
        "nvfp4_quantize_dual_bf16");
  return py::make_tuple(a.q, a.s, a.p, b.q, b.s, b.p);
}

at::Tensor mm(const at::Tensor& aq, const at::Tensor& as, const at::Tensor& ap, const at::Tensor& bq, const at::Tensor& bs,
              const at::Tensor& bp, bool f32, const OptTensor& out, const OptTensor& amax_out) {
  const int64_t m = aq.size(0), k2 = aq.size(1), n = bq.size(0);
  const c10::Device dev = device_of({&aq, &as, &ap, &bq, &bs, &bp, ptr_of(out), ptr_of(amax_out)});
  const c10::cuda::CUDAGuard guard(dev);
  const at::Tensor d = out.has_value() ? *out : at::empty({m, n}, on(dev, f32 ? at::kFloat : at::kBFloat16));
  auto u8 = [](const at::Tensor& t) { return static_cast<const uint8_t*>(t.data_ptr()); };
  int32_t* status = status_word(dev.index()).data_ptr<int32_t>();
  const int type = f32 ? NVFP4_OUT_F32 : NVFP4_OUT_BF16;
  check(amax_out.has_value()
            ? lib.nvfp4_gemm_amax(u8(aq), u8(as), float_ptr(ap), u8(bq), u8(bs), float_ptr(bp), d.data_ptr(), type, m, n,
                                  k2 * 2, d.stride(0), float_ptr(*amax_out), status, stream_of(dev))
            : lib.nvfp4_gemm(u8(aq), u8(as), float_ptr(ap), u8(bq), u8(bs), float_ptr(bp), d.data_ptr(), type, m, n, k2 * 2,
                             d.stride(0), status, stream_of(dev)),
        "nvfp4_gemm");
  return d;
}

// the bf16 product in an fp32 tensor
at::Tensor mm_bf16_as_f32(const at::Tensor& aq, const at::Tensor& as, const at::Tensor& ap, const at::Tensor& bq,
                          const at::Tensor& bs, const at::Tensor& bp) {
  const int64_t m = aq.size(0), k2 = aq.size(1), n = bq.size(0);
  const c10::Device dev = device_of({&aq, &as, &ap, &bq, &bs, &bp});
  const c10::cuda::CUDAGuard guard(dev);
  const at::Tensor d = at::empty({m, n}, on(dev, at::kFloat));
  auto u8 = [](const at::Tensor& t) { return static_cast<const uint8_t*>(t.data_ptr()); };
  check(lib.nvfp4_gemm_bf16_as_f32(u8(aq), u8(as), float_ptr(ap), u8(bq), u8(bs), float_ptr(bp), float_ptr(d), m, n, k2 * 2,
                                   n, status_word(dev.index()).data_ptr<int32_t>(), stream_of(dev)),
        "nvfp4_gemm_bf16_as_f32");
  return d;
}

}  // namespace

PYBIND11_MODULE(_host, m) {
  m.def("init", &init);
  m.def("workspace", &workspace);
  m.def("workspace_if_any", &workspace_if_any);
  m.def("status_word", &status_word);
  m.def("amax", &amax);
  m.def("amax_both", &amax_both);
  m.def("quantize", &quantize);
  m.def("quantize_weight", &quantize_weight);
  m.def("quantize_dual", &quantize_dual);
  m.def("mm", &mm);
  m.def("mm_bf16_as_f32", &mm_bf16_as_f32);
}

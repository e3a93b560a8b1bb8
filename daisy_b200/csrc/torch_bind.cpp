// Python bindings over the C ABI of libdaisy_b200.so: tensors in, tensors out, one C++ call per layer or per step.
//
// The calls a decode step or a short prompt makes are a few microseconds of GPU work each; reading forty attributes per
// call from Python and converting them one by one costs more than that.  Here the checks, the allocations and the launches
// of a whole layer are native, the Python classes above only hold parameters and state.  Nothing is computed by torch on
// these paths: it supplies device memory, the stream and the tensor type.
#include <ATen/cuda/CUDAContext.h>
#include <ATen/cuda/CUDAGraphsUtils.cuh>
#include <c10/cuda/CUDAGuard.h>
#include <torch/extension.h>

#include <list>
#include <mutex>

#include "../../include/daisy_b200.h"

namespace {

using at::Tensor;
using OptTensor = std::optional<Tensor>;

// A negative status of the library; becomes daisy_b200._lib.DaisyB200Error in Python.
struct StatusError : std::runtime_error {
  int code;
  StatusError(int c, const char* what) : std::runtime_error(what), code(c) {}
};
void check(int rc, const char* what) {
  if (rc != DAISY_OK) throw StatusError(rc, what);
}

void* stream_of(const Tensor& t) { return at::cuda::getCurrentCUDAStream(t.get_device()).stream(); }

// ------------------------------------------------------------------ argument checks (same errors as the Python wrappers)
void req(const Tensor& t, const char* name, at::ScalarType dt = at::kBFloat16) {
  TORCH_CHECK_VALUE(t.is_cuda(), name, " must be a CUDA tensor (daisy_b200 has no CPU path)");
  TORCH_CHECK_TYPE(t.scalar_type() == dt, name, " must be ", dt, ", got ", t.scalar_type());
  TORCH_CHECK_VALUE(t.dim() > 0 && t.stride(-1) == 1, name, " must be contiguous in its last dimension");
}

// ------------------------------------------------------------------ per-device status word, per-stream workspaces
constexpr int MAX_DEV = 64;
std::mutex g_mutex;
Tensor g_status[MAX_DEV];

Tensor status_word(int dev) {
  std::lock_guard<std::mutex> lock(g_mutex);
  TORCH_CHECK(dev >= 0 && dev < MAX_DEV, "device index out of range");
  if (!g_status[dev].defined()) {
    c10::InferenceMode off(false);
    g_status[dev] = at::zeros({1}, at::TensorOptions().device(at::kCUDA, dev).dtype(at::kInt));
  }
  return g_status[dev];
}
int* status_ptr(const Tensor& t) { return status_word(t.get_device()).data_ptr<int>(); }

// Workspaces that only have to be zero before their first use are kept per (device, stream): calls on one stream run one after
// another, whatever thread makes them, so they can share one; calls on two streams never do.  At most POOL_MAX are kept,
// the least recently used goes first (its memory returns to torch's allocator, which keeps it on its stream).
struct PoolEntry { int dev; void* stream; int kind; Tensor ws; };
constexpr size_t POOL_MAX = 32;
std::list<PoolEntry> g_pool;

Tensor zeroed(int dev, int64_t bytes) {
  return at::zeros({bytes}, at::TensorOptions().device(at::kCUDA, dev).dtype(at::kByte));
}
Tensor stream_workspace(const Tensor& like, int kind, int64_t bytes) {
  const int dev = like.get_device();
  void* st = stream_of(like);
  // a captured call may be replayed on any stream: it gets a workspace of its own inside the graph
  if (at::cuda::currentStreamCaptureStatus() != at::cuda::CaptureStatus::None) return zeroed(dev, bytes);
  std::lock_guard<std::mutex> lock(g_mutex);
  for (auto it = g_pool.begin(); it != g_pool.end(); ++it)
    if (it->dev == dev && it->stream == st && it->kind == kind && it->ws.numel() >= bytes) {
      if (it != g_pool.begin()) g_pool.splice(g_pool.begin(), g_pool, it);
      return g_pool.front().ws;
    }
  g_pool.remove_if([&](const PoolEntry& e) { return e.dev == dev && e.stream == st && e.kind == kind; });
  g_pool.push_front(PoolEntry{dev, st, kind, zeroed(dev, bytes)});
  if (g_pool.size() > POOL_MAX) g_pool.pop_back();
  return g_pool.front().ws;
}
void release_workspaces() {
  std::lock_guard<std::mutex> lock(g_mutex);
  g_pool.clear();
}
enum { WS_TOKEN = 0 };

// ------------------------------------------------------------------ decode step
void rope_table(const Tensor& t, const char* name) {
  TORCH_CHECK_VALUE(t.is_cuda() && t.scalar_type() == at::kFloat && t.is_contiguous() && t.dim() == 2 && t.size(1) == 64, name,
                    " must be a contiguous float32 CUDA tensor [rows, 64]");
}

// Whether the single-launch step takes these sizes.
bool token_step_supported(int64_t B, int64_t H, int64_t layers) {
  return layers >= 1 && B >= 1 && daisy_b200_swa_token_workspace_bytes((int)B, (int)H, 128) != 0 &&
         B * H <= 2 * (int64_t)daisy_b200_sm_count();
}

// x [B,1,dim] through the layers over their rings k, v [L,B,H,cap,128]; position `t`, or *t_dev; `t_advance` is stepped.
// `out`, `workspace`: fixed buffers of the caller, or None.
Tensor token_step(const Tensor& x_, const std::vector<Tensor>& weights, const std::vector<Tensor>& cos, const std::vector<Tensor>& sin,
                  const Tensor& k, const Tensor& v, int64_t t, const OptTensor& t_dev, const OptTensor& t_advance, int64_t window,
                  double scale, double eps, int64_t flags, const OptTensor& ve, const OptTensor& ve_gate, const OptTensor& k_new,
                  const OptTensor& v_new, const OptTensor& out, const OptTensor& workspace) {
  const int64_t L = (int64_t)weights.size();
  TORCH_CHECK_VALUE(L >= 1 && (int64_t)cos.size() == L && (int64_t)sin.size() == L, "one weight and one RoPE table pair per layer");
  TORCH_CHECK_VALUE(k.dim() == 5 && k.size(0) == L && k.size(4) == 128 && v.sizes() == k.sizes() && v.strides() == k.strides(),
                    "rings must both be [layers, B, H, cap, 128] with equal strides");
  const int64_t B = k.size(1), H = k.size(2), cap = k.size(3), dim = H * 128;
  const bool f16 = k.scalar_type() == at::kHalf;
  req(k, "kcache", f16 ? at::kHalf : at::kBFloat16);
  req(v, "vcache", k.scalar_type());
  TORCH_CHECK_VALUE(x_.is_cuda(), "x must be a CUDA tensor (daisy_b200 has no CPU path)");
  TORCH_CHECK_VALUE(x_.numel() == B * dim && x_.size(-1) == dim, "x must be [", B, ", 1, ", dim, "]");
  c10::cuda::CUDAGuard guard(k.device());
  Tensor x = x_.scalar_type() == at::kBFloat16 ? x_ : x_.to(at::kBFloat16);
  int64_t x_sb = dim;
  if (x.dim() == 3 && x.size(1) == 1 && x.stride(2) == 1 && x.stride(0) % 8 == 0) x_sb = x.stride(0);
  else if (!x.is_contiguous()) x = x.contiguous();
  std::vector<daisy_b200_token_layer> ly(L);
  int64_t rows = INT32_MAX;
  for (int64_t l = 0; l < L; ++l) {
    const Tensor& w = weights[l];
    req(w, "qkvo_w");
    TORCH_CHECK_VALUE(w.dim() == 3 && w.size(0) == 4 && w.size(1) == dim && w.size(2) == dim && w.is_contiguous(), "qkvo_w must be a contiguous [4, ", dim, ", ", dim, "]");
    rope_table(cos[l], "cos"); rope_table(sin[l], "sin");
    rows = std::min({rows, cos[l].size(0), sin[l].size(0)});
    ly[l].qkvo_w = w.data_ptr();
    ly[l].kcache = (char*)k.data_ptr() + l * k.stride(0) * 2;
    ly[l].vcache = (char*)v.data_ptr() + l * v.stride(0) * 2;
    ly[l].cos = cos[l].data_ptr<float>(); ly[l].sin = sin[l].data_ptr<float>();
  }
  Tensor ve_c;
  if (ve.has_value()) {
    TORCH_CHECK_VALUE(L == 1 && ve_gate.has_value() && ve_gate->is_cuda() && ve_gate->scalar_type() == at::kFloat && ve_gate->numel() == 1,
                      "ve needs ve_gate_logit, a float32 scalar CUDA tensor");
    ve_c = ve->to(at::kBFloat16).reshape({B, dim});
    if (ve_c.stride(1) != 1) ve_c = ve_c.contiguous();
    ly[0].ve = ve_c.data_ptr(); ly[0].ve_gate_logit = ve_gate->data_ptr<float>();
  }
  if (k_new.has_value()) { ly[0].k_new_out = k_new->data_ptr(); ly[0].v_new_out = v_new->data_ptr(); }
  TORCH_CHECK_VALUE(!t_dev.has_value() || (t_dev->is_cuda() && t_dev->scalar_type() == at::kLong && t_dev->numel() == 1),
                    "a device-side position must be an int64 CUDA tensor with one element");
  Tensor y = out.has_value() ? *out : at::empty({B, 1, dim}, x.options());
  const int64_t need = (int64_t)daisy_b200_swa_token_workspace_bytes((int)B, (int)H, 128);
  Tensor ws = workspace.has_value() ? *workspace : stream_workspace(x, WS_TOKEN, need);
  constexpr int64_t PER_LAUNCH = 16;
  for (int64_t l0 = 0; l0 < L; l0 += PER_LAUNCH) {                       // a deeper stack takes several launches, handing x on in y
    const bool end = l0 + PER_LAUNCH >= L;
    check(daisy_b200_swa_token_step(ly.data() + l0, (int)std::min(PER_LAUNCH, L - l0), l0 ? y.data_ptr() : x.data_ptr(), l0 ? dim : x_sb, y.data_ptr(),
                                    k.stride(1), k.stride(2), k.stride(3), t, t_dev.has_value() ? t_dev->data_ptr<int64_t>() : nullptr,
                                    end && t_advance.has_value() ? t_advance->data_ptr<int64_t>() : nullptr, (int)cap, (int)window, (int)rows,
                                    ve_c.defined() ? ve_c.stride(0) : 0, (int)B, (int)H, 128, (float)scale, (float)eps,
                                    (unsigned)flags | (f16 ? DAISY_CACHE_FP16 : 0), ws.data_ptr(), (size_t)ws.numel(), status_ptr(x), stream_of(x)),
          "daisy_b200_swa_token_step");
  }
  return y;
}

}  // namespace

PYBIND11_MODULE(TORCH_EXTENSION_NAME, m) {
  py::register_exception_translator([](std::exception_ptr p) {
    try {
      if (p) std::rethrow_exception(p);
    } catch (const StatusError& e) {
      py::object cls = py::module_::import("daisy_b200._lib").attr("DaisyB200Error");
      PyErr_SetObject(cls.ptr(), cls(e.code, e.what()).ptr());
    }
  });
  m.def("status_word", &status_word);
  m.def("release_workspaces", &release_workspaces);
  m.def("token_workspace_bytes", [](int64_t B, int64_t H) { return (int64_t)daisy_b200_swa_token_workspace_bytes((int)B, (int)H, 128); });
  m.def("token_step_supported", &token_step_supported);
  m.def("token_step", &token_step);
}

// Python bindings over the C ABI of libdaisy_b200.so: tensors in, tensors out, one C++ call per layer or per step.
//
// The calls a decode step or a short prompt makes are a few microseconds of GPU work each; reading forty attributes per
// call from Python and converting them one by one costs more than that.  Here the checks, the allocations and the launches
// of a whole layer are native, the Python classes above only hold parameters and state.  Nothing is computed by torch on
// these paths: it supplies device memory, the stream and the tensor type.
//
// Python objects are read first; the calls then run without the interpreter lock, as torch's own do.  A launch waits when the
// queue is full and packed lengths on the device wait for the stream: other Python threads go on, also the one whose launch
// that stream may be waiting for.
#include <ATen/cuda/CUDAContext.h>
#include <ATen/cuda/CUDAEvent.h>
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

bool on16(const Tensor& t) { return (reinterpret_cast<uintptr_t>(t.data_ptr()) & 15) == 0; }
// the same values where 16-byte loads can fetch them
Tensor aligned(const Tensor& t) { return t.is_contiguous() && on16(t) ? t : t.clone(at::MemoryFormat::Contiguous); }

// An attention layer's weights; a layout with gaps between rows or matrices is packed.
Tensor layer_weight(const Tensor& w, int64_t dim) {
  req(w, "qkvo_w");
  TORCH_CHECK_VALUE(w.dim() == 3 && w.size(0) == 4 && w.size(1) == dim && w.size(2) == dim, "qkvo_w must be [4, ", dim, ", ", dim, "]");
  return w.contiguous();
}

// A decode step's vectors: x beside the state or ring it goes with, and the caller's buffer for the result.
void req_step(const Tensor& x, const OptTensor& out, const Tensor& state, int64_t B, int64_t dim) {
  TORCH_CHECK_VALUE(x.is_cuda(), "x must be a CUDA tensor (daisy_b200 has no CPU path)");
  TORCH_CHECK_VALUE(x.device() == state.device(), "x is on ", x.device(), ", the states are on ", state.device());
  TORCH_CHECK_VALUE(x.dim() > 0 && x.numel() == B * dim && x.size(-1) == dim, "x must be [", B, ", 1, ", dim, "]");
  if (!out.has_value()) return;
  TORCH_CHECK_VALUE(out->device() == state.device() && out->scalar_type() == at::kBFloat16 && out->is_contiguous() && out->numel() == B * dim,
                    "out must be a contiguous bf16 [", B, ", 1, ", dim, "] on ", state.device());
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
enum { WS_TOKEN = 0, WS_KDA_TOKEN = 1 };

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
  req_step(x_, out, k, B, dim);
  c10::cuda::CUDAGuard guard(k.device());
  Tensor x = x_.scalar_type() == at::kBFloat16 ? x_ : x_.to(at::kBFloat16);
  int64_t x_sb = dim;
  if (x.dim() == 3 && x.size(1) == 1 && x.stride(2) == 1 && x.stride(0) % 8 == 0) x_sb = x.stride(0);
  else if (!x.is_contiguous()) x = x.contiguous();
  std::vector<daisy_b200_token_layer> ly(L);
  std::vector<Tensor> packed;                                            // weights that had to be copied, until the launch
  int64_t rows = INT32_MAX;
  for (int64_t l = 0; l < L; ++l) {
    const Tensor w = layer_weight(weights[l], dim);
    if (!w.is_same(weights[l])) packed.push_back(w);
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


// ------------------------------------------------------------------ attention layer, whole sequences
struct Doc { Tensor t; const int32_t* ptr = nullptr; int64_t sb = 0; };
Doc doc_arg(const OptTensor& doc, int64_t B, int64_t T, const Tensor& like) {
  Doc d;
  if (!doc.has_value()) return d;
  TORCH_CHECK_VALUE(doc->is_cuda(), "doc_start must be a CUDA tensor");
  d.t = doc->to(like.device(), at::kInt).contiguous();
  d.ptr = d.t.data_ptr<int32_t>();
  if (d.t.dim() == 1 && d.t.size(0) == T) return d;
  if (d.t.dim() == 2 && d.t.size(0) == B && d.t.size(1) == T) { d.sb = T; return d; }
  TORCH_CHECK_VALUE(false, "doc_start must have shape [", T, "] or [", B, ",", T, "], got ", d.t.sizes());
  return d;
}

Tensor rows_of(const Tensor& x, int64_t K) {
  Tensor x2 = x.reshape({-1, K});
  return x2.stride(1) == 1 ? x2 : x2.contiguous();
}

Tensor gemm_nt(const Tensor& x, const Tensor& w) {
  req(x, "x"); req(w, "w");
  const int64_t K = x.size(-1), N = w.size(0);
  Tensor x2 = rows_of(x, K);
  std::vector<int64_t> shape(x.sizes().begin(), x.sizes().end());
  shape.back() = N;
  Tensor c = at::empty(shape, x.options());
  check(daisy_b200_gemm_nt(x2.data_ptr(), x2.stride(0), w.data_ptr(), w.stride(0), c.data_ptr(), N, (int)x2.size(0), (int)N, (int)K, status_ptr(x), stream_of(x)),
        "daisy_b200_gemm_nt");
  return c;
}

// merged projection with the norm / RoPE / gate epilogue -> q', k', v' [B,T,H,128]
std::vector<Tensor> qkv_gemm(const Tensor& x, const Tensor& w_qkv, const OptTensor& cos, const OptTensor& sin, int64_t H, double eps, int64_t flags,
                             const OptTensor& ve, const OptTensor& ve_gate, const OptTensor& ring_k, const OptTensor& ring_v, int64_t ring_first) {
  req(x, "x"); req(w_qkv, "w_qkv");
  TORCH_CHECK_VALUE(x.dim() == 3, "x must be [B, T, dim]");
  const int64_t B = x.size(0), T = x.size(1), dim = x.size(2);
  TORCH_CHECK_VALUE(w_qkv.dim() == 2 && w_qkv.size(0) == 3 * H * 128 && w_qkv.size(1) == dim, "w_qkv must be [", 3 * H * 128, ", ", dim, "], got ", w_qkv.sizes());
  Tensor x2 = rows_of(x, dim);
  if (flags & DAISY_ROPE)
    for (const OptTensor* t : {&cos, &sin})
      TORCH_CHECK_VALUE(t->has_value() && (*t)->is_cuda() && (*t)->scalar_type() == at::kFloat && (*t)->is_contiguous() && (*t)->size(0) >= T && (*t)->size(1) == 64,
                        "cos, sin must be contiguous float32 CUDA tensors of at least T rows");
  Tensor ve2;
  if (ve.has_value()) {
    TORCH_CHECK_VALUE(ve_gate.has_value() && ve_gate->is_cuda() && ve_gate->scalar_type() == at::kFloat && ve_gate->numel() == 1,
                      "ve needs ve_gate_logit, a float32 scalar CUDA tensor");
    ve2 = ve->reshape({B * T, H * 128});
    req(ve2, "ve");
  }
  int64_t sb = 0, sh = 0, sr = 0, cap = 0;
  unsigned f = (unsigned)flags;
  if (ring_k.has_value()) {
    const Tensor &rk = *ring_k, &rv = *ring_v;
    const bool f16 = rk.scalar_type() == at::kHalf;
    req(rk, "ring k", f16 ? at::kHalf : at::kBFloat16); req(rv, "ring v", rk.scalar_type());
    TORCH_CHECK_VALUE(rk.dim() == 4 && rk.sizes() == rv.sizes() && rk.strides() == rv.strides() && rk.size(0) == B && rk.size(1) == H && rk.size(3) == 128,
                      "ring tensors must both be [", B, ", ", H, ", cap, 128] with equal strides");
    sb = rk.stride(0); sh = rk.stride(1); sr = rk.stride(2); cap = rk.size(2);
    f |= f16 ? DAISY_CACHE_FP16 : 0;
  }
  std::vector<Tensor> out;
  for (int i = 0; i < 3; ++i) out.push_back(at::empty({B, T, H, 128}, x.options()));
  check(daisy_b200_qkv_gemm_ring(x2.data_ptr(), x2.stride(0), w_qkv.data_ptr(), w_qkv.stride(0), cos.has_value() ? cos->data_ptr<float>() : nullptr,
                                 sin.has_value() ? sin->data_ptr<float>() : nullptr, out[0].data_ptr(), out[1].data_ptr(), out[2].data_ptr(),
                                 ve2.defined() ? ve2.data_ptr() : nullptr, ve2.defined() ? ve2.stride(0) : 0, ve2.defined() ? ve_gate->data_ptr<float>() : nullptr,
                                 ring_k.has_value() ? ring_k->data_ptr() : nullptr, ring_k.has_value() ? ring_v->data_ptr() : nullptr, sb, sh, sr, (int)cap,
                                 (int)ring_first, (int)B, (int)T, (int)H, 128, (int)dim, (float)eps, f, status_ptr(x), stream_of(x)),
        "daisy_b200_qkv_gemm_ring");
  return out;
}

// windowed attention on prepared [B,T,H,128] tensors -> (out, lse2 or undefined)
std::pair<Tensor, Tensor> swa_attend(const Tensor& q, const Tensor& k, const Tensor& v, int64_t window, double scale, const OptTensor& out_, bool bounded,
                                     const OptTensor& doc_start, bool in_blocks, bool want_lse) {
  req(q, "q"); req(k, "k"); req(v, "v");
  TORCH_CHECK_VALUE(q.dim() == 4 && k.sizes() == q.sizes() && v.sizes() == q.sizes(), "q, k, v must be [B,T,H,D] of one shape");
  const int64_t B = q.size(0), T = q.size(1), H = q.size(2), D = q.size(3);
  Tensor out = out_.has_value() ? *out_ : at::empty({B, T, H, D}, q.options());
  Doc d = doc_arg(doc_start, B, T, q);
  Tensor lse;
  if (want_lse) lse = at::empty({B, H, T}, q.options().dtype(at::kFloat));
  const unsigned flags = (bounded ? DAISY_BOUNDED_QK : 0) | (in_blocks ? DAISY_WINDOW_BLOCKS : 0);
  auto call = [&](auto fn, auto... extra) {
    return fn(q.data_ptr(), k.data_ptr(), v.data_ptr(), q.stride(0), q.stride(1), q.stride(2), k.stride(0), k.stride(1), k.stride(2), v.stride(0), v.stride(1),
              v.stride(2), out.data_ptr(), out.stride(0), out.stride(1), out.stride(2), extra..., (int)B, (int)T, (int)H, (int)D, (int)window, (float)scale, d.ptr,
              d.sb, flags, status_ptr(q), stream_of(q));
  };
  if (want_lse) check(call(daisy_b200_swa_attend_lse, lse.data_ptr<float>()), "daisy_b200_swa_attend_lse");
  else check(call(daisy_b200_swa_attend), "daisy_b200_swa_attend");
  return {out, lse};
}

// The layer's output alone: q', k', v' and the attention output are scratch, one allocation.
Tensor attn_forward(const Tensor& x_, const Tensor& w_, const Tensor& cos, const Tensor& sin, int64_t H, double eps, double scale, int64_t window,
                    const OptTensor& doc_start, bool in_blocks, const OptTensor& ve, const OptTensor& ve_gate) {
  TORCH_CHECK_VALUE(x_.is_cuda(), "x must be a CUDA tensor (daisy_b200 has no CPU path)");
  const Tensor x = x_.detach().to(w_.scalar_type());
  req(x, "x");
  c10::cuda::CUDAGuard guard(x.device());
  TORCH_CHECK_VALUE(x.dim() == 3, "x must be [B, T, dim]");
  const int64_t B = x.size(0), T = x.size(1), dim = x.size(2), M = B * T;
  const Tensor qkvo_w = layer_weight(w_, H * 128);
  TORCH_CHECK_VALUE(dim == H * 128, "x must be [B, T, ", H * 128, "]");
  rope_table(cos, "cos"); rope_table(sin, "sin");
  TORCH_CHECK_VALUE(cos.size(0) >= T && sin.size(0) >= T, "cos, sin must be contiguous float32 CUDA tensors of at least T rows");
  Tensor x2 = rows_of(x, dim), ve2;
  if (ve.has_value()) {
    TORCH_CHECK_VALUE(ve_gate.has_value() && ve_gate->is_cuda() && ve_gate->scalar_type() == at::kFloat && ve_gate->numel() == 1,
                      "ve needs ve_gate_logit, a float32 scalar CUDA tensor");
    ve2 = ve->reshape({M, dim});
    req(ve2, "ve");
  }
  const int64_t n = M * dim, sb = T * dim;
  Tensor buf = at::empty({4 * n}, x.options()), y = at::empty({B, T, dim}, x.options());
  char *q = (char*)buf.data_ptr(), *k = q + 2 * n, *v = k + 2 * n, *o = v + 2 * n;
  Doc dc = doc_arg(doc_start, B, T, x);
  int* status = status_ptr(x);
  void* st = stream_of(x);
  check(daisy_b200_qkv_gemm(x2.data_ptr(), x2.stride(0), qkvo_w.data_ptr(), dim, cos.data_ptr<float>(), sin.data_ptr<float>(), q, k, v,
                            ve2.defined() ? ve2.data_ptr() : nullptr, ve2.defined() ? ve2.stride(0) : 0, ve2.defined() ? ve_gate->data_ptr<float>() : nullptr, (int)B,
                            (int)T, (int)H, 128, (int)dim, (float)eps, DAISY_QKV_DEFAULT, status, st),
        "daisy_b200_qkv_gemm");
  check(daisy_b200_swa_attend(q, k, v, sb, dim, 128, sb, dim, 128, sb, dim, 128, o, sb, dim, 128, (int)B, (int)T, (int)H, 128, (int)window, (float)scale, dc.ptr, dc.sb,
                              DAISY_BOUNDED_QK | (in_blocks ? DAISY_WINDOW_BLOCKS : 0), status, st),
        "daisy_b200_swa_attend");                                                          // q, k are RMS-normalised
  check(daisy_b200_gemm_nt(o, dim, (char*)qkvo_w.data_ptr() + 3 * dim * dim * 2, dim, y.data_ptr(), dim, (int)M, (int)dim, (int)dim, status, st), "daisy_b200_gemm_nt");
  return y;
}

// One attention layer: projection, attention, output projection -> (y, k', v', q')
std::vector<Tensor> attn_layer(const Tensor& x_, const Tensor& qkvo_w, const Tensor& cos, const Tensor& sin, int64_t H, double eps, double scale, int64_t window,
                               const OptTensor& doc_start, bool in_blocks, const OptTensor& ve, const OptTensor& ve_gate, const OptTensor& ring_k,
                               const OptTensor& ring_v, int64_t ring_first) {
  Tensor w = layer_weight(qkvo_w.detach(), H * 128), x = x_.detach().to(w.scalar_type());
  TORCH_CHECK_VALUE(x.is_cuda(), "x must be a CUDA tensor (daisy_b200 has no CPU path)");
  c10::cuda::CUDAGuard guard(x.device());
  const int64_t B = x.size(0), T = x.size(1), dim = w.size(2);
  auto p = qkv_gemm(x, w.narrow(0, 0, 3).view({3 * dim, dim}), cos, sin, H, eps, DAISY_QKV_DEFAULT, ve, ve_gate, ring_k, ring_v, ring_first);
  Tensor y = swa_attend(p[0], p[1], p[2], window, scale, std::nullopt, true, doc_start, in_blocks, false).first;   // q, k are RMS-normalised
  y = gemm_nt(y.view({B, T, dim}), w.select(0, 3));
  return {y, p[1], p[2], p[0]};
}

// A stack of plain layers over a prompt: layer l fills ring k[l], v[l] with rows t >= ring_first (none if negative).  The layers
// share their scratch (they run one after another on the stream), so a prompt costs seven allocations, not seven a layer.
Tensor attn_stack(const Tensor& x_, const std::vector<Tensor>& weights, const std::vector<Tensor>& cos, const std::vector<Tensor>& sin, int64_t H, double eps, double scale,
                  int64_t window, const Tensor& k, const Tensor& v, int64_t ring_first) {
  const size_t L = weights.size();
  TORCH_CHECK_VALUE(L >= 1 && cos.size() == L && sin.size() == L && k.dim() == 5 && (size_t)k.size(0) == L && v.sizes() == k.sizes() && v.strides() == k.strides(),
                    "one weight, one RoPE table pair and one ring per layer");
  TORCH_CHECK_VALUE(x_.is_cuda(), "x must be a CUDA tensor (daisy_b200 has no CPU path)");
  TORCH_CHECK_VALUE(x_.dim() == 3, "x must be [B, T, dim]");
  c10::cuda::CUDAGuard guard(x_.device());
  Tensor x = x_.detach().to(weights[0].scalar_type());
  const int64_t B = x.size(0), T = x.size(1), dim = x.size(2), M = B * T;
  const bool f16 = k.scalar_type() == at::kHalf, ring = ring_first >= 0;
  req(x, "x"); req(k, "ring k", f16 ? at::kHalf : at::kBFloat16); req(v, "ring v", k.scalar_type());
  TORCH_CHECK_VALUE(dim == H * 128 && k.size(1) == B && k.size(2) == H && k.size(4) == 128, "rings must be [layers, ", B, ", ", H, ", cap, 128], x [B, T, ", H * 128, "]");
  Tensor q = at::empty({B, T, H, 128}, x.options()), kp = at::empty_like(q), vp = at::empty_like(q), o = at::empty_like(q), ya = at::empty({B, T, dim}, x.options());
  Tensor yb = L > 1 ? at::empty_like(ya) : Tensor(), in = rows_of(x, dim);
  int* status = status_ptr(x);
  void* st = stream_of(x);
  for (size_t l = 0; l < L; ++l) {
    const Tensor w = layer_weight(weights[l], dim);
    rope_table(cos[l], "cos"); rope_table(sin[l], "sin");
    TORCH_CHECK_VALUE(cos[l].size(0) >= T && sin[l].size(0) >= T, "cos, sin must be contiguous float32 CUDA tensors of at least T rows");
    char *rk = ring ? (char*)k.data_ptr() + l * k.stride(0) * 2 : nullptr, *rv = ring ? (char*)v.data_ptr() + l * v.stride(0) * 2 : nullptr;
    check(daisy_b200_qkv_gemm_ring(in.data_ptr(), in.stride(0), w.data_ptr(), dim, cos[l].data_ptr<float>(), sin[l].data_ptr<float>(), q.data_ptr(), kp.data_ptr(),
                                   vp.data_ptr(), nullptr, 0, nullptr, rk, rv, k.stride(1), k.stride(2), k.stride(3), (int)k.size(3), ring ? (int)ring_first : 0, (int)B,
                                   (int)T, (int)H, 128, (int)dim, (float)eps, DAISY_QKV_DEFAULT | (f16 ? DAISY_CACHE_FP16 : 0), status, st),
          "daisy_b200_qkv_gemm_ring");
    swa_attend(q, kp, vp, window, scale, o, true, std::nullopt, false, false);             // q, k are RMS-normalised
    Tensor& y = (L - 1 - l) % 2 ? yb : ya;
    check(daisy_b200_gemm_nt(o.data_ptr(), dim, (char*)w.data_ptr() + 3 * dim * dim * 2, dim, y.data_ptr(), dim, (int)M, (int)dim, (int)dim, status, st), "daisy_b200_gemm_nt");
    in = y.view({M, dim});
  }
  return ya;
}

// Workspace of an attention backward: with room for the dZ images, up to 2 GB, where the allocator has it, else without (dQ from
// the scores).  Before the allocator refuses it gives back every block it has cached, behind waits for the device: a size it refused
// is not asked for again in the next REFUSED_CALLS calls on that device.
constexpr int REFUSED_CALLS = 256;
struct Refused { int64_t bytes = 0; int calls = 0; };
Refused g_refused[MAX_DEV];

Tensor bwd_workspace(const Tensor& like, int64_t B, int64_t T, int64_t H, int64_t window, bool in_blocks) {
  const int64_t full = (int64_t)daisy_b200_swa_attend_bwd_workspace_bytes_full((int)B, (int)T, (int)H, (int)window, in_blocks ? DAISY_WINDOW_BLOCKS : 0);
  const auto bytes = like.options().dtype(at::kByte);
  const int dev = like.get_device();
  TORCH_CHECK(dev >= 0 && dev < MAX_DEV, "device index out of range");
  bool ask = true;
  {
    std::lock_guard<std::mutex> lock(g_mutex);
    Refused& r = g_refused[dev];
    if (r.calls > 0) { --r.calls; ask = full < r.bytes; }
  }
  if (ask) {
    try {
      return at::empty({full}, bytes);
    } catch (const c10::OutOfMemoryError&) {
      std::lock_guard<std::mutex> lock(g_mutex);
      g_refused[dev] = {full, REFUSED_CALLS};
    }
  }
  return at::empty({(int64_t)daisy_b200_swa_attend_bwd_workspace_bytes((int)B, (int)T, (int)H)}, bytes);
}

// ------------------------------------------------------------------ attention layer under autograd
// Forward: the fused projection (which also leaves 1 / rms of every head row), attention with its log-sum-exp, output
// projection.  Backward: two library products for each projection, the attention backward, and one row-wise pass that undoes
// norms, RoPE and gate into the merged gradient matrix.  As F.linear calls around the attention core this took a copy of the
// merged gradient (concatenation of three), zero fills and an addition for the two slices of the weight's gradient, a separate
// norm / RoPE pass and its raw inputs.
// What the forward leaves for the backward, in one allocation (a small step costs more in allocator calls than in kernels):
// byte offsets of q', k', v', vn (gated layers), o, 1 / rms and the log-sum-exp.
struct Saved {
  int64_t q, k, v, vn, o, rstd, lse, elems;
  static int64_t up(int64_t n) { return (n + 255) / 256 * 256; }
  Saved(int64_t M, int64_t H, bool gated) {
    const int64_t rows = up(M * H * 256);
    q = 0; k = rows; v = 2 * rows; vn = 3 * rows;
    o = (gated ? 4 : 3) * rows; rstd = o + rows; lse = rstd + up(M * 3 * H * 4);
    elems = (lse + up(M * H * 4)) / 2;                                                      // of bf16
  }
};
struct AttnFunction : public torch::autograd::Function<AttnFunction> {
  static Tensor forward(torch::autograd::AutogradContext* ctx, const Tensor& x, const Tensor& w_, const OptTensor& ve, const OptTensor& logit, const Tensor& cos,
                        const Tensor& sin, int64_t H, double eps, double scale, int64_t window, const OptTensor& doc_start, bool in_blocks) {
    at::AutoDispatchBelowADInplaceOrView guard;
    req(x, "x"); req(w_, "qkvo_w");
    TORCH_CHECK_VALUE(x.dim() == 3 && w_.dim() == 3, "x must be [B, T, dim], qkvo_w [4, dim, dim]");
    const int64_t B = x.size(0), T = x.size(1), dim = H * 128, M = B * T;
    TORCH_CHECK_VALUE(w_.size(0) == 4 && w_.size(1) == dim && w_.size(2) == dim && x.size(2) == dim, "qkvo_w must be [4, dim, dim]");
    rope_table(cos, "cos"); rope_table(sin, "sin");
    const Tensor w = aligned(w_);
    Tensor x2 = rows_of(x, dim);
    if (!on16(x2) || x2.stride(0) % 8) x2 = x2.clone(at::MemoryFormat::Contiguous);
    Tensor ve2, g32;
    if (ve.has_value()) {
      req(*ve, "ve");
      TORCH_CHECK_VALUE(ve->numel() == M * dim && logit->numel() == 1, "ve must be [", B, ", ", T, ", ", dim, "], its gate one number");
      ve2 = aligned(*ve);
      g32 = logit->to(at::kFloat);
    }
    const Saved at_(M, H, ve2.defined());
    Tensor buf = at::empty({at_.elems}, x.options());
    char* p = (char*)buf.data_ptr();
    Doc dc = doc_arg(doc_start, B, T, x);
    int* status = status_ptr(x);
    void* st = stream_of(x);
    check(daisy_b200_qkv_gemm_train(x2.data_ptr(), x2.stride(0), w.data_ptr(), dim, cos.data_ptr<float>(), sin.data_ptr<float>(), p + at_.q, p + at_.k, p + at_.v,
                                    (float*)(p + at_.rstd), ve2.defined() ? p + at_.vn : nullptr, ve2.defined() ? ve2.data_ptr() : nullptr, ve2.defined() ? dim : 0,
                                    ve2.defined() ? g32.data_ptr<float>() : nullptr, (int)B, (int)T, (int)H, 128, (int)dim, (float)eps, DAISY_QKV_DEFAULT, status, st),
          "daisy_b200_qkv_gemm_train");
    const int64_t sb = T * dim, sh = 128;
    check(daisy_b200_swa_attend_lse(p + at_.q, p + at_.k, p + at_.v, sb, dim, sh, sb, dim, sh, sb, dim, sh, p + at_.o, sb, dim, sh, (float*)(p + at_.lse), (int)B, (int)T,
                                    (int)H, 128, (int)window, (float)scale, dc.ptr, dc.sb, DAISY_BOUNDED_QK | (in_blocks ? DAISY_WINDOW_BLOCKS : 0), status, st),
          "daisy_b200_swa_attend_lse");                                                    // q, k are RMS-normalised
    Tensor y = at::empty({B, T, dim}, x.options());
    check(daisy_b200_gemm_nt(p + at_.o, dim, (char*)w.data_ptr() + 3 * dim * dim * 2, dim, y.data_ptr(), dim, (int)M, (int)dim, (int)dim, status, st), "daisy_b200_gemm_nt");
    // the inputs themselves, not views of them made here: below the autograd keys a view has a version counter of its own, and
    // a change in place between forward and backward would go unnoticed
    ctx->save_for_backward({x, w_, buf, cos, sin, ve.value_or(Tensor()), ve.has_value() ? *logit : Tensor(), doc_start.value_or(Tensor())});
    ctx->saved_data["dims"] = std::vector<int64_t>{B, T, H, window, in_blocks ? 1 : 0};
    ctx->saved_data["scale"] = scale;
    if (ve.has_value()) {
      ctx->saved_data["ve_shape"] = ve->sizes().vec();
      ctx->saved_data["logit_shape"] = logit->sizes().vec();
      ctx->saved_data["logit_type"] = (int64_t)logit->scalar_type();
    }
    return y;
  }
  static torch::autograd::variable_list backward(torch::autograd::AutogradContext* ctx, torch::autograd::variable_list grads) {
    at::AutoDispatchBelowADInplaceOrView guard;
    auto s = ctx->get_saved_variables();
    const Tensor &w = s[1], &buf = s[2], &cos = s[3], &sin = s[4], &doc = s[7];
    auto d = ctx->saved_data["dims"].toIntVector();
    const int64_t B = d[0], T = d[1], H = d[2], window = d[3], dim = H * 128, M = B * T;
    Tensor ve2, g32;
    if (s[5].defined()) { ve2 = aligned(s[5]); g32 = s[6].to(at::kFloat); }
    const float scale = (float)ctx->saved_data["scale"].toDouble();
    const bool need_x = ctx->needs_input_grad(0), need_w = ctx->needs_input_grad(1);
    Tensor dy = grads[0].to(at::kBFloat16).reshape({M, dim});
    if (dy.stride(1) != 1) dy = dy.contiguous();
    const Saved at_(M, H, ve2.defined());
    char* p = (char*)buf.data_ptr();
    Tensor dw, dx;
    if (need_w) {
      dw = at::empty(w.sizes(), w.options());
      Tensor dwo = dw.select(0, 3);
      at::mm_out(dwo, dy.t(), buf.narrow(0, at_.o / 2, M * dim).view({M, dim}));
    }
    Tensor d_o = at::mm(dy, w.select(0, 3));
    const unsigned bwd_flags = d[4] ? DAISY_WINDOW_BLOCKS : 0;
    const int64_t row = Saved::up(M * dim * 2), part_at = 6 * row;
    const int64_t n_part = ve2.defined() ? daisy_b200_qkv_prep_grad_blocks((int)M, (int)H) : 0;
    Tensor tmp = at::empty({(part_at + Saved::up(4 * n_part)) / 2}, buf.options());          // dqkv, dq, dk, dv, partial sums
    char *g = (char*)tmp.data_ptr(), *dq = g + 3 * row, *dk = g + 4 * row, *dv = g + 5 * row;
    Tensor dqkv = tmp.narrow(0, 0, M * 3 * dim).view({M, 3 * dim}), d_ve, d_logit;
    Tensor ws = bwd_workspace(buf, B, T, H, window, d[4]);
    Doc dc = doc_arg(doc.defined() ? OptTensor(doc) : std::nullopt, B, T, buf);
    const int64_t sb = T * H * 128, st = H * 128, sh = 128;
    void* stream = stream_of(buf);
    check(daisy_b200_swa_attend_bwd(p + at_.q, p + at_.k, p + at_.v, p + at_.o, d_o.data_ptr(), sb, st, sh, sb, st, sh, sb, st, sh, sb, st, sh, sb, st, sh,
                                    (const float*)(p + at_.lse), dq, dk, dv, (int)B, (int)T, (int)H, 128, (int)window, scale, dc.ptr, dc.sb,
                                    bwd_flags, ws.data_ptr(), (size_t)ws.numel(), status_ptr(buf), stream),
          "daisy_b200_swa_attend_bwd");
    if (ve2.defined()) {
      d_ve = at::empty({M, dim}, buf.options());
      d_logit = at::empty({1}, buf.options().dtype(at::kFloat));
    }
    auto ptr = [](const Tensor& t) { return t.defined() ? t.data_ptr() : nullptr; };
    check(daisy_b200_qkv_prep_grad(p + at_.q, p + at_.k, p + (ve2.defined() ? at_.vn : at_.v), dq, dk, dv, (const float*)(p + at_.rstd), cos.data_ptr<float>(),
                                   sin.data_ptr<float>(), dqkv.data_ptr(), ptr(ve2), (const float*)ptr(g32), ptr(d_ve), (float*)ptr(d_logit),
                                   n_part ? (float*)(g + part_at) : nullptr, (int)M, (int)T, (int)H, 128, stream),
          "daisy_b200_qkv_prep_grad");
    const Tensor wqkv = w.narrow(0, 0, 3).reshape({3 * dim, dim});
    if (need_w) {
      Tensor dwq = dw.narrow(0, 0, 3).view({3 * dim, dim});
      at::mm_out(dwq, dqkv.t(), rows_of(s[0], dim));
    }
    if (need_x) dx = at::mm(dqkv, wqkv).view({B, T, dim});
    torch::autograd::variable_list out(12);
    out[0] = dx; out[1] = dw;
    if (ve2.defined()) {
      out[2] = d_ve.view(ctx->saved_data["ve_shape"].toIntVector());
      out[3] = d_logit.to((at::ScalarType)ctx->saved_data["logit_type"].toInt()).view(ctx->saved_data["logit_shape"].toIntVector());
    }
    return out;
  }
};

Tensor attn_train(const Tensor& x, const Tensor& w, const OptTensor& ve, const OptTensor& logit, const Tensor& cos, const Tensor& sin, int64_t H, double eps,
                  double scale, int64_t window, const OptTensor& doc_start, bool in_blocks) {
  TORCH_CHECK_VALUE(x.is_cuda(), "x must be a CUDA tensor (daisy_b200 has no CPU path)");
  c10::cuda::CUDAGuard guard(x.device());
  // an embedding made in inference mode cannot be saved for the backward: a copy can
  const OptTensor e = ve.has_value() && ve->is_inference() ? OptTensor(ve->clone()) : ve;
  return AttnFunction::apply(x.scalar_type() == w.scalar_type() ? x : x.to(w.scalar_type()), w, e, logit, cos, sin, H, eps, scale, window, doc_start, in_blocks);
}

// ------------------------------------------------------------------ Kimi layer, one token
// whether all of them are there, bf16 and contiguous
bool plain_bf16(const std::vector<OptTensor>& ts) {
  for (const OptTensor& t : ts)
    if (!t.has_value() || t->scalar_type() != at::kBFloat16 || !t->is_contiguous()) return false;
  return true;
}
bool kda_token_supported(int64_t H) { return H >= 1 && daisy_b200_kda_token_workspace_bytes(1, (int)H, 128) != 0; }
int64_t kda_token_workspace_bytes(int64_t B, int64_t H) { return (int64_t)daisy_b200_kda_token_workspace_bytes((int)B, (int)H, 128); }

// weights: q, k, v, f0, f1, g0, g1, b, o; conv: q, k, v weights (and biases); the states are updated in place
Tensor kda_token_step(const Tensor& x_, const std::vector<Tensor>& w_, const OptTensor& g1_bias, const OptTensor& norm_w, const std::vector<Tensor>& conv_w,
                      const std::vector<OptTensor>& conv_b, const Tensor& a_log, const Tensor& dt_bias, Tensor state, const std::vector<Tensor>& conv_s,
                      bool silu, double eps, const OptTensor& out, const OptTensor& workspace) {
  TORCH_CHECK_VALUE(w_.size() == 9 && conv_w.size() == 3 && conv_b.size() == 3 && conv_s.size() == 3, "nine weights, three convolutions");
  const int64_t B = state.size(0), H = state.size(1), dim = H * 128;
  req_step(x_, out, state, B, dim);
  c10::cuda::CUDAGuard guard(x_.device());
  Tensor x = aligned(x_.to(at::kBFloat16).reshape({B, dim}));
  bool as_is = true;
  for (const Tensor& t : w_) { req(t, "weight"); TORCH_CHECK_VALUE(t.is_contiguous(), "weights must be contiguous"); as_is = as_is && on16(t); }
  std::vector<Tensor> copies;
  if (!as_is) for (const Tensor& t : w_) copies.push_back(aligned(t));
  const std::vector<Tensor>& w = as_is ? w_ : copies;
  daisy_b200_kda_layer ly{};
  ly.q_w = w[0].data_ptr(); ly.k_w = w[1].data_ptr(); ly.v_w = w[2].data_ptr(); ly.f0_w = w[3].data_ptr(); ly.f1_w = w[4].data_ptr();
  ly.g0_w = w[5].data_ptr(); ly.g1_w = w[6].data_ptr(); ly.b_w = w[7].data_ptr(); ly.o_w = w[8].data_ptr();
  if (g1_bias.has_value()) { req(*g1_bias, "g_proj bias"); ly.g1_bias = g1_bias->data_ptr(); }
  if (norm_w.has_value()) { req(*norm_w, "norm weight"); ly.norm_w = norm_w->data_ptr(); }
  req(a_log, "A_log", at::kFloat); req(dt_bias, "dt_bias", at::kFloat); req(state, "state", at::kFloat);
  TORCH_CHECK_VALUE(a_log.numel() == H && dt_bias.numel() == dim && a_log.is_contiguous() && state.is_contiguous() && state.numel() == B * H * 128 * 128,
                    "state must be a contiguous [B, H, 128, 128]");
  for (int i = 0; i < 3; ++i) {
    req(conv_w[i], "conv weight"); req(conv_s[i], "conv state");
    TORCH_CHECK_VALUE(conv_w[i].numel() == dim * 4 && conv_w[i].is_contiguous() && conv_s[i].is_contiguous() && conv_s[i].numel() == B * dim * 4,
                      "four taps, states [B, dim, 4]");
    ly.conv_w[i] = conv_w[i].data_ptr();
    if (conv_b[i].has_value()) { req(*conv_b[i], "conv bias"); ly.conv_bias[i] = conv_b[i]->data_ptr(); }
  }
  ly.a_log = a_log.data_ptr<float>(); ly.dt_bias = dt_bias.data_ptr<float>();
  Tensor y = out.has_value() ? *out : at::empty({B, 1, dim}, x.options());
  const int64_t need = kda_token_workspace_bytes(B, H);                  // above 16 rows plain scratch, below words that have to be zero at first
  Tensor ws = workspace.has_value() ? *workspace : B > 16 ? at::empty({need}, x.options().dtype(at::kByte)) : stream_workspace(x, WS_KDA_TOKEN, need);
  check(daisy_b200_kda_token_step(&ly, x.data_ptr(), dim, y.data_ptr(), state.data_ptr<float>(), conv_s[0].data_ptr(), conv_s[1].data_ptr(), conv_s[2].data_ptr(),
                                  (int)B, (int)H, 128, (float)eps, silu ? DAISY_KDA_CONV_SILU : 0, ws.data_ptr(), (size_t)ws.numel(), status_ptr(x), stream_of(x)),
        "daisy_b200_kda_token_step");
  return y;
}


// ------------------------------------------------------------------ KDA
Tensor f32c(const Tensor& t, const char* name) {
  TORCH_CHECK_VALUE(t.is_cuda() && t.scalar_type() == at::kFloat && t.is_contiguous(), name, " must be a contiguous float32 CUDA tensor");
  return t;
}

// `cu_seqlens` as the caller gave it: nothing, a tensor, or any sequence of integers.
struct Lengths { bool given = false; Tensor t; std::vector<int64_t> list; };
Lengths lengths_of(const py::object& cu_seqlens) {
  Lengths r;
  r.given = !cu_seqlens.is_none();
  if (THPVariable_Check(cu_seqlens.ptr())) r.t = THPVariable_Unpack(cu_seqlens.ptr());
  else if (r.given)
    for (auto item : cu_seqlens) r.list.push_back(py::cast<int64_t>(py::int_(py::reinterpret_borrow<py::object>(item))));
  return r;
}

void check_offsets(const std::vector<int64_t>& cu) {
  bool ok = cu.size() >= 2 && cu[0] == 0;
  for (size_t i = 1; ok && i < cu.size(); ++i) ok = cu[i] >= cu[i - 1];
  TORCH_CHECK_VALUE(ok, "cu_seqlens must start at 0 and not decrease");
}
// The integers of a tensor that was copied to the host.
std::vector<int64_t> to_list(const Tensor& c) {
  if (c.scalar_type() == at::kInt) return {c.data_ptr<int32_t>(), c.data_ptr<int32_t>() + c.numel()};
  return {c.data_ptr<int64_t>(), c.data_ptr<int64_t>() + c.numel()};
}

// Tables of a packed batch on the device (see kda_varlen_tables); tok only if asked for.
struct Packed { Tensor chunks, ptr, tok, cu; int64_t n_chunks = 0, n_seq = 0, total = 0; };
Packed pack_tables(const Lengths& lengths, c10::Device dev, int64_t chunk, bool want_tok) {
  TORCH_CHECK_VALUE(chunk > 0, "chunk must be positive, got ", chunk);
  std::vector<int64_t> cu = lengths.list;
  if (const Tensor& t = lengths.t; t.defined()) {
    TORCH_CHECK_VALUE(t.dim() == 1, "cu_seqlens must have one dimension, got ", t.sizes());
    if (t.is_cuda() && t.numel() > 1 && (t.scalar_type() == at::kInt || t.scalar_type() == at::kLong)) {
      c10::cuda::CUDAGuard guard(t.device());
      Tensor c = at::empty(t.sizes(), at::TensorOptions().dtype(t.scalar_type()).pinned_memory(true));
      c.copy_(t, /*non_blocking=*/true);
      at::cuda::getCurrentCUDAStream(t.get_device()).synchronize();
      cu = to_list(c);
    } else {
      cu = to_list(t.to(at::kCPU, at::kLong).contiguous());
    }
  }
  check_offsets(cu);
  Packed p;
  p.n_seq = (int64_t)cu.size() - 1;
  p.total = cu.back();
  for (int64_t n = 0; n < p.n_seq; ++n) p.n_chunks += (cu[n + 1] - cu[n] + chunk - 1) / chunk;
  // one staging buffer, one copy: [n_chunks][2], [n_seq + 1] (padded to 8 bytes), [total][2], [n_seq + 1]
  const int64_t at_ptr = 2 * p.n_chunks, at_tok = at_ptr + (p.n_seq + 2) / 2 * 2, at_cu = at_tok + (want_tok ? 2 * p.total : 0);
  const int64_t size = at_cu + (want_tok ? p.n_seq + 1 : 0);
  Tensor host = at::empty({std::max<int64_t>(size, 1)}, at::TensorOptions().dtype(at::kInt).pinned_memory(dev.is_cuda()));
  int32_t* h = host.data_ptr<int32_t>();
  int64_t c = 0;
  for (int64_t n = 0; n < p.n_seq; ++n) {
    h[at_ptr + n] = (int32_t)c;
    for (int64_t t = cu[n]; t < cu[n + 1]; t += chunk, ++c) { h[2 * c] = (int32_t)t; h[2 * c + 1] = (int32_t)std::min(chunk, cu[n + 1] - t); }
    if (want_tok)
      for (int64_t t = cu[n]; t < cu[n + 1]; ++t) { h[at_tok + 2 * t] = (int32_t)cu[n]; h[at_tok + 2 * t + 1] = (int32_t)n; }
  }
  h[at_ptr + p.n_seq] = (int32_t)c;
  for (int64_t i = at_ptr + p.n_seq + 1; i < at_tok; ++i) h[i] = 0;
  for (int64_t n = 0; want_tok && n <= p.n_seq; ++n) h[at_cu + n] = (int32_t)cu[n];
  Tensor d = host.to(dev, /*non_blocking=*/true);
  p.chunks = d.narrow(0, 0, 2 * p.n_chunks).view({p.n_chunks, 2});
  p.ptr = d.narrow(0, at_ptr, p.n_seq + 1);
  if (want_tok) { p.tok = d.narrow(0, at_tok, 2 * p.total).view({p.total, 2}); p.cu = d.narrow(0, at_cu, p.n_seq + 1); }
  return p;
}

// chunked forward, dense ([B,T,H,K], packed == nullptr) or packed ([1,T_total,H,K])
std::pair<Tensor, OptTensor> kda_chunk(const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& g_, const Tensor& beta_, std::optional<double> scale,
                                       const OptTensor& h0_, bool want_state, bool l2norm, bool out_fp32, const Packed* pk) {
  const Tensor* in[] = {&q, &k, &v};
  const char* names[] = {"q", "k", "v"};
  for (int i = 0; i < 3; ++i) { req(*in[i], names[i]); TORCH_CHECK_VALUE(in[i]->is_contiguous(), names[i], " must be contiguous"); }
  TORCH_CHECK_VALUE(!pk || q.size(0) == 1, "packed sequences come as one row: q must be [1, T_total, H, K]");
  Tensor g = f32c(g_, "g"), beta = f32c(beta_, "beta");
  const int64_t B = q.size(0), T = q.size(1), H = q.size(2), K = q.size(3), V = v.size(3), n = pk ? pk->n_seq : B;
  TORCH_CHECK_VALUE(!pk || pk->total == T, "cu_seqlens covers ", pk ? pk->total : 0, " tokens, the inputs hold ", T);
  Tensor h0;
  if (h0_.has_value()) {
    h0 = f32c(*h0_, "initial_state");
    TORCH_CHECK_VALUE(!pk || (h0.dim() == 4 && h0.size(0) == n && h0.size(1) == H && h0.size(2) == K && h0.size(3) == V), "initial_state must be [", n, ", ", H, ", ",
                      K, ", ", V, "]");
  }
  const int64_t need = pk ? (int64_t)daisy_b200_kda_varlen_workspace_bytes((int)pk->n_chunks, (int)H, (int)K, (int)V)
                          : (int64_t)daisy_b200_kda_workspace_bytes((int)B, (int)T, (int)H, (int)K, (int)V);
  Tensor o = at::empty({B, T, H, V}, q.options().dtype(out_fp32 ? at::kFloat : at::kBFloat16)), ws = at::empty({std::max<int64_t>(need, 16)}, q.options().dtype(at::kByte));
  OptTensor hT;
  if (want_state) hT = at::empty({n, H, K, V}, q.options().dtype(at::kFloat));
  if (pk && (T == 0 || pk->n_chunks == 0)) {
    if (want_state) { if (h0.defined()) hT->copy_(h0); else hT->zero_(); }
    return {o, hT};
  }
  const unsigned flags = (l2norm ? DAISY_KDA_L2NORM_QK : 0) | (out_fp32 ? DAISY_KDA_OUT_FP32 : 0);
  const float sc = scale.has_value() ? (float)*scale : 0.f;
  const float* h0p = h0.defined() ? h0.data_ptr<float>() : nullptr;
  float* hTp = want_state ? hT->data_ptr<float>() : nullptr;
  if (pk)
    check(daisy_b200_kda_chunk_fwd_varlen(q.data_ptr(), k.data_ptr(), v.data_ptr(), g.data_ptr<float>(), beta.data_ptr<float>(), h0p, o.data_ptr(), hTp, (int)T, (int)H,
                                          (int)K, (int)V, 64, sc, flags, pk->chunks.data_ptr<int32_t>(), (int)pk->n_chunks, pk->ptr.data_ptr<int32_t>(), (int)n,
                                          ws.data_ptr(), (size_t)ws.numel(), status_ptr(q), stream_of(q)),
          "daisy_b200_kda_chunk_fwd_varlen");
  else
    check(daisy_b200_kda_chunk_fwd(q.data_ptr(), k.data_ptr(), v.data_ptr(), g.data_ptr<float>(), beta.data_ptr<float>(), h0p, o.data_ptr(), hTp, (int)B, (int)T, (int)H,
                                   (int)K, (int)V, 64, sc, flags, ws.data_ptr(), (size_t)ws.numel(), status_ptr(q), stream_of(q)),
          "daisy_b200_kda_chunk_fwd");
  return {o, hT};
}

// token by token; with in_place the state handed in is updated and returned
std::pair<Tensor, OptTensor> kda_recurrent(const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& g_, const Tensor& beta_, std::optional<double> scale,
                                           const OptTensor& h0_, bool want_state, bool l2norm, bool out_fp32, bool in_place) {
  const Tensor* in[] = {&q, &k, &v};
  const char* names[] = {"q", "k", "v"};
  for (int i = 0; i < 3; ++i) { req(*in[i], names[i]); TORCH_CHECK_VALUE(in[i]->is_contiguous(), names[i], " must be contiguous"); }
  Tensor g = f32c(g_, "g"), beta = f32c(beta_, "beta");
  const int64_t B = q.size(0), T = q.size(1), H = q.size(2), K = q.size(3), V = v.size(3);
  Tensor h0;
  if (h0_.has_value()) h0 = f32c(*h0_, in_place ? "an in-place state" : "initial_state");
  TORCH_CHECK_VALUE(!in_place || h0.defined(), "state_in_place needs an initial_state");
  Tensor o = at::empty({B, T, H, V}, q.options().dtype(out_fp32 ? at::kFloat : at::kBFloat16));
  OptTensor hT;
  if (in_place) hT = h0;
  else if (want_state) hT = at::empty({B, H, K, V}, q.options().dtype(at::kFloat));
  const unsigned flags = (l2norm ? DAISY_KDA_L2NORM_QK : 0) | (out_fp32 ? DAISY_KDA_OUT_FP32 : 0);
  check(daisy_b200_kda_recurrent_fwd(q.data_ptr(), k.data_ptr(), v.data_ptr(), g.data_ptr<float>(), beta.data_ptr<float>(), h0.defined() ? h0.data_ptr<float>() : nullptr,
                                     o.data_ptr(), hT.has_value() ? hT->data_ptr<float>() : nullptr, (int)B, (int)T, (int)H, (int)K, (int)V,
                                     scale.has_value() ? (float)*scale : 0.f, flags, stream_of(q)),
        "daisy_b200_kda_recurrent_fwd");
  return {o, hT};
}

constexpr int64_t RECURRENT_MAX_T = 4;           // up to this many tokens the state is carried token by token in registers

// the layer's chunk_kda call: any float types, dense or packed
std::pair<Tensor, OptTensor> chunk_kda(const Tensor& q_, const Tensor& k_, const Tensor& v_, const Tensor& g_, const Tensor& beta_, std::optional<double> scale,
                                       const OptTensor& h0_, bool want_state, bool l2norm, const Lengths& cu_seqlens, bool out_fp32) {
  Tensor q = q_.to(at::kBFloat16).contiguous(), k = k_.to(at::kBFloat16).contiguous(), v = v_.to(at::kBFloat16).contiguous();
  Tensor g = g_.to(at::kFloat).contiguous(), beta = beta_.to(at::kFloat).contiguous();
  OptTensor h0;
  if (h0_.has_value()) h0 = h0_->to(at::kFloat).contiguous();
  if (const Tensor& t = cu_seqlens.t; t.defined() && t.is_cuda() && t.device() == q.device() && t.dim() == 1 && t.is_contiguous() && t.numel() > 1 && t.numel() <= 1024 &&
                                      (t.scalar_type() == at::kInt || t.scalar_type() == at::kLong) && q.dim() == 4 && q.size(0) == 1 && q.size(1) > 0) {
    // Offsets on the device: the tables are made there, and the offsets are read and checked here while the kernels run.
    c10::cuda::CUDAGuard guard(q.device());
    const auto stream = at::cuda::getCurrentCUDAStream();
    Tensor c = at::empty(t.sizes(), at::TensorOptions().dtype(t.scalar_type()).pinned_memory(true));
    c.copy_(t, /*non_blocking=*/true);
    at::cuda::CUDAEvent there;
    there.record(stream);
    Packed p;
    p.n_seq = t.numel() - 1;
    p.total = q.size(1);
    p.n_chunks = p.total / 64 + p.n_seq;                                                   // every sequence may end in a short chunk
    Tensor tabs = at::empty({2 * p.n_chunks + p.n_seq + 1}, q.options().dtype(at::kInt));
    p.chunks = tabs.narrow(0, 0, 2 * p.n_chunks);
    p.ptr = tabs.narrow(0, 2 * p.n_chunks, p.n_seq + 1);
    check(daisy_b200_kda_chunk_tables(t.data_ptr(), (int)t.element_size(), (int)p.n_seq, (int)p.total, p.chunks.data_ptr<int32_t>(), (int)p.n_chunks,
                                      p.ptr.data_ptr<int32_t>(), stream.stream()),
          "daisy_b200_kda_chunk_tables");
    std::pair<Tensor, OptTensor> r = kda_chunk(q, k, v, g, beta, scale, h0, want_state, l2norm, out_fp32, &p);
    there.synchronize();
    const std::vector<int64_t> cu = to_list(c);
    check_offsets(cu);
    TORCH_CHECK_VALUE(cu.back() == p.total, "cu_seqlens covers ", cu.back(), " tokens, the inputs hold ", p.total);
    return r;
  }
  if (cu_seqlens.given) {
    Packed p = pack_tables(cu_seqlens, q.device(), 64, false);
    return kda_chunk(q, k, v, g, beta, scale, h0, want_state, l2norm, out_fp32, &p);
  }
  return q.size(1) <= RECURRENT_MAX_T ? kda_recurrent(q, k, v, g, beta, scale, h0, want_state, l2norm, out_fp32, false)
                                      : kda_chunk(q, k, v, g, beta, scale, h0, want_state, l2norm, out_fp32, nullptr);
}

// ------------------------------------------------------------------ Kimi layer, whole sequences
// F.linear on this library's GEMM where its tiles apply; the narrow ones (the per-head beta projection, few rows) go to torch's
Tensor kimi_linear(const Tensor& x, const Tensor& w) {
  const int64_t N = w.size(0), K = w.size(1);
  if (x.numel() / K >= 64 && N % 128 == 0 && K % 64 == 0 && w.scalar_type() == at::kBFloat16 && x.scalar_type() == at::kBFloat16) return gemm_nt(x, w);
  return at::linear(x, w);
}

// y[i] = x[i] w[i]^T; products of one shape go out in one launch
void kimi_linears(std::vector<Tensor> x, std::vector<Tensor> w, Tensor* y) {
  const size_t n = x.size();
  const int64_t N = w[0].size(0), K = w[0].size(1);
  bool group = x[0].numel() / K >= 64 && N % 128 == 0 && K % 64 == 0;
  for (size_t i = 0; i < n; ++i)
    group = group && x[i].scalar_type() == at::kBFloat16 && w[i].scalar_type() == at::kBFloat16 && x[i].sizes() == x[0].sizes() && w[i].sizes() == w[0].sizes() &&
            x[i].is_contiguous() && w[i].is_contiguous();
  if (!group) {
    for (size_t i = 0; i < n; ++i) y[i] = kimi_linear(x[i], w[i]);
    return;
  }
  const void *xp[3], *wp[3];
  void* cp[3];
  auto shape = x[0].sizes().vec();
  shape.back() = N;
  for (size_t i = 0; i < n; ++i) {
    y[i] = at::empty(shape, x[0].options());
    xp[i] = x[i].data_ptr(); wp[i] = w[i].data_ptr(); cp[i] = y[i].data_ptr();
  }
  check(daisy_b200_gemm_nt_group(xp, K, wp, K, cp, N, (int)n, (int)(x[0].numel() / K), (int)N, (int)K, status_ptr(x[0]), stream_of(x[0])), "daisy_b200_gemm_nt_group");
}

// weights: q, k, v, f0, f1, g0, g1, b, o.  conv_s, rec: carried states or nothing.  -> y, final state, convolution states
// With a mask [B, T] the kept tokens of all rows are one packed row, one sequence per batch row, and y is zero elsewhere; without
// any kept token there is nothing but y.
std::tuple<Tensor, OptTensor, std::vector<Tensor>> kimi_layer(const Tensor& x_, const std::vector<Tensor>& w, const OptTensor& g1_bias, const OptTensor& norm_w,
                                                              const std::vector<Tensor>& conv_w, const std::vector<OptTensor>& conv_b, const Tensor& a_log,
                                                              const Tensor& dt_bias, const std::vector<OptTensor>& conv_s, const OptTensor& rec, bool use_cache,
                                                              bool silu, double eps, int64_t H, const Lengths& cu_seqlens, const OptTensor& mask_) {
  TORCH_CHECK_VALUE(x_.is_cuda(), "x must be a CUDA tensor (daisy_b200 has no CPU path)");
  c10::cuda::CUDAGuard guard(x_.device());
  Packed p;
  const bool packed = cu_seqlens.given || mask_.has_value();
  Tensor x = x_, rank;
  if (mask_.has_value()) {
    const int64_t B0 = x.size(0), T0 = x.size(1), dim = x.size(2);
    Tensor mask = *mask_;
    TORCH_CHECK_VALUE(mask.dim() == 2 && mask.size(0) == B0 && mask.size(1) == T0 && mask.device() == x.device(), "mask must be [", B0, ", ", T0, "] beside x");
    const auto type = mask.scalar_type();
    if (type != at::kBool && type != at::kByte && type != at::kChar && type != at::kInt && type != at::kLong) mask = mask.to(at::kBool);
    if (mask.stride(1) != 1 || mask.stride(0) < 0) mask = mask.contiguous();
    const auto ints = x.options().dtype(at::kInt);
    rank = at::empty({2 * B0 * T0 + B0}, ints);                                            // rank, idx, len
    int32_t *r = rank.data_ptr<int32_t>(), *idx = r + B0 * T0, *len = idx + B0 * T0;
    check(daisy_b200_kda_mask_rows(mask.data_ptr(), (int)mask.element_size(), mask.stride(0), (int)B0, (int)T0, r, idx, len, stream_of(x)), "daisy_b200_kda_mask_rows");
    Tensor host = at::empty({B0}, ints.device(at::kCPU).pinned_memory(true));
    host.copy_(rank.narrow(0, 2 * B0 * T0, B0), /*non_blocking=*/true);
    Tensor rows = aligned(x.contiguous());                                                 // while the lengths are on their way
    at::cuda::getCurrentCUDAStream(x.get_device()).synchronize();
    Lengths lengths;
    lengths.given = true;
    lengths.list.push_back(0);
    for (int64_t b = 0; b < B0; ++b) lengths.list.push_back(lengths.list.back() + host.data_ptr<int32_t>()[b]);
    p = pack_tables(lengths, x.device(), 64, true);
    if (p.total == 0) return {at::zeros_like(x), OptTensor(), {}};
    x = at::empty({1, p.total, dim}, x.options());
    check(daisy_b200_kda_pack_rows(rows.data_ptr(), idx, p.tok.data_ptr<int32_t>(), x.data_ptr(), (int)p.total, (int)T0, (int)dim, stream_of(x)), "daisy_b200_kda_pack_rows");
  } else if (packed) {
    p = pack_tables(cu_seqlens, x.device(), 64, true);
  }
  const int64_t B = x.size(0), T = x.size(1), C = w[0].size(0), M = B * T;
  const int64_t n = packed ? p.n_seq : B;
  Tensor qkv[3], pr[3];
  std::vector<Tensor> out_s;
  kimi_linears({x, x, x}, {w[0], w[1], w[2]}, pr);
  const void *xp[3], *wp[3], *bp[3], *sp[3];
  void *op[3], *yp[3];
  int64_t W[3];
  Tensor fresh;                                                                            // states of packed sequences that begin here
  if (use_cache && packed && !conv_s[0].has_value() && conv_w[0].numel() == conv_w[1].numel() && conv_w[0].numel() == conv_w[2].numel())
    fresh = at::zeros({3, n, C, conv_w[0].numel() / C}, x.options());
  for (int i = 0; i < 3; ++i) {
    qkv[i] = at::empty_like(pr[i]);
    const bool have = conv_s[i].has_value(), in_place = have && !packed && T <= 32;
    W[i] = conv_w[i].numel() / C;
    if (have)
      TORCH_CHECK_VALUE(conv_s[i]->scalar_type() == at::kBFloat16 && conv_s[i]->is_contiguous() && conv_s[i]->numel() == n * C * W[i],
                        "state must be a contiguous bf16 [", n, ", ", C, ", ", W[i], "] tensor");
    Tensor so;
    if (in_place) so = *conv_s[i];
    else if (use_cache && packed) so = have ? conv_s[i]->clone() : fresh.defined() ? fresh.select(0, i) : at::zeros({n, C, W[i]}, x.options());   // sequences without tokens keep their state
    else if (use_cache) so = at::empty({n, C, W[i]}, x.options());
    xp[i] = pr[i].data_ptr(); wp[i] = conv_w[i].data_ptr(); bp[i] = conv_b[i].has_value() ? conv_b[i]->data_ptr() : nullptr;
    sp[i] = have ? conv_s[i]->data_ptr() : nullptr; op[i] = so.defined() ? so.data_ptr() : nullptr; yp[i] = qkv[i].data_ptr();
    qkv[i] = qkv[i].view({B, T, H, 128});
    if (so.defined()) out_s.push_back(so);
  }
  const int step = W[0] == W[1] && W[1] == W[2] && B * 3 <= 65535 ? 3 : 1;                 // one launch for the three
  for (int i = 0; i < 3; i += step)
    check(daisy_b200_kda_short_conv_group(step, xp + i, T * C, C, wp + i, bp + i, sp + i, op + i, yp + i, T * C, C, (int)B, (int)T, (int)C, (int)W[i],
                                          packed ? p.tok.data_ptr<int32_t>() : nullptr, silu ? DAISY_KDA_CONV_SILU : 0, stream_of(x)),
          "daisy_b200_kda_short_conv_group");
  Tensor g = at::empty({B, T, H, 128}, x.options().dtype(at::kFloat)), gp, beta;
  bool fused = M >= 64 && H <= 32 && x.scalar_type() == at::kBFloat16 && C == x.size(2) && x.is_contiguous() && on16(x) && on16(dt_bias);
  for (int i = 3; i < 8; ++i) fused = fused && w[i].scalar_type() == at::kBFloat16 && w[i].is_contiguous() && on16(w[i]) && w[i].size(0) == (i == 7 ? H : i % 2 ? 128 : C);
  if (fused) {                                                                             // low-rank products and write strength, then both gates
    Tensor low = at::empty({2, M, 128}, x.options());
    beta = at::empty({B, T, H}, g.options());
    gp = at::empty({B, T, C}, x.options());
    void *f0 = low.data_ptr(), *g0 = low.select(0, 1).data_ptr();
    check(daisy_b200_kda_low_rank(x.data_ptr(), C, w[3].data_ptr(), w[5].data_ptr(), w[7].data_ptr(), f0, g0, beta.data_ptr<float>(), (int)M, (int)H, (int)C,
                                  status_ptr(x), stream_of(x)),
          "daisy_b200_kda_low_rank");
    check(daisy_b200_kda_gates(f0, g0, w[4].data_ptr(), w[6].data_ptr(), a_log.data_ptr<float>(), dt_bias.data_ptr<float>(), g.data_ptr<float>(), gp.data_ptr(), (int)M,
                               (int)H, status_ptr(x), stream_of(x)),
          "daisy_b200_kda_gates");
  } else {
    Tensor low[2], up[2];                                                                    // the two low-rank projections: decay gate, output gate
    kimi_linears({x, x}, {w[3], w[5]}, low);
    kimi_linears({low[0], low[1]}, {w[4], w[6]}, up);
    const Tensor& f = up[0];
    gp = up[1];
    check(daisy_b200_kda_gate(f.data_ptr(), 1, a_log.data_ptr<float>(), dt_bias.data_ptr<float>(), g.data_ptr<float>(), M, (int)H, 128, 1.f, 20.f,
                              DAISY_KDA_GATE_ROUND_BF16, stream_of(x)),
          "daisy_b200_kda_gate");
    Tensor bx = at::linear(x, w[7]);
    if (bx.scalar_type() == at::kBFloat16) {
      beta = at::empty(bx.sizes(), bx.options().dtype(at::kFloat));
      check(daisy_b200_kda_beta(bx.data_ptr(), beta.data_ptr<float>(), beta.numel(), stream_of(x)), "daisy_b200_kda_beta");
    } else {
      beta = bx.sigmoid_().to(at::kFloat);
    }
  }
  std::pair<Tensor, OptTensor> r = packed ? kda_chunk(qkv[0], qkv[1], qkv[2], g, beta, std::nullopt, rec, use_cache, true, false, &p)
                                   : T <= RECURRENT_MAX_T ? kda_recurrent(qkv[0], qkv[1], qkv[2], g, beta, std::nullopt, rec, use_cache, true, false, rec.has_value())
                                                          : kda_chunk(qkv[0], qkv[1], qkv[2], g, beta, std::nullopt, rec, use_cache, true, false, nullptr);
  Tensor o = r.first, yn = at::empty({B, T, C}, x.options());
  check(daisy_b200_kda_out_norm(o.data_ptr(), 0, gp.data_ptr(), g1_bias.has_value() ? g1_bias->data_ptr() : nullptr, g1_bias.has_value() ? (int)H : 1,
                                norm_w.has_value() ? norm_w->data_ptr() : nullptr, yn.data_ptr(), M * H, 128, (float)eps, 2, stream_of(x)),
        "daisy_b200_kda_out_norm");
  Tensor y = kimi_linear(yn, w[8]);
  if (mask_.has_value()) {
    Tensor out = at::empty(x_.sizes(), y.options());
    check(daisy_b200_kda_unpack_rows(y.data_ptr(), rank.data_ptr<int32_t>(), p.cu.data_ptr<int32_t>(), out.data_ptr(), (int)x_.size(0), (int)x_.size(1), (int)x_.size(2),
                                     stream_of(y)),
          "daisy_b200_kda_unpack_rows");
    y = out;
  }
  return {y, r.second, out_s};
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
  using nogil = py::call_guard<py::gil_scoped_release>;
  m.def("status_word", &status_word, nogil());
  m.def("release_workspaces", &release_workspaces, nogil());
  m.def("token_workspace_bytes", [](int64_t B, int64_t H) { return (int64_t)daisy_b200_swa_token_workspace_bytes((int)B, (int)H, 128); });
  m.def("token_step_supported", &token_step_supported);
  m.def("token_step", &token_step, nogil());
  m.def("gemm_nt", &gemm_nt, nogil());
  m.def("qkv_gemm", &qkv_gemm, nogil());
  m.def("swa_attend", [](const Tensor& q, const Tensor& k, const Tensor& v, int64_t window, double scale, const OptTensor& out, bool bounded,
                         const OptTensor& doc_start, bool in_blocks) {
    return swa_attend(q, k, v, window, scale, out, bounded, doc_start, in_blocks, false).first;
  }, nogil());
  m.def("bwd_workspace", &bwd_workspace, nogil());
  m.def("swa_attend_lse", [](const Tensor& q, const Tensor& k, const Tensor& v, int64_t window, double scale, const OptTensor& out, bool bounded,
                             const OptTensor& doc_start, bool in_blocks) {
    return swa_attend(q, k, v, window, scale, out, bounded, doc_start, in_blocks, true);
  }, nogil());
  m.def("attn_stack", &attn_stack, nogil());
  m.def("attn_forward", &attn_forward, nogil());
  m.def("attn_layer", &attn_layer, nogil());
  m.def("attn_train", &attn_train, nogil());
  m.def("kda_tables", [](const py::object& cu, const py::object& device, int64_t chunk) {
    const Lengths lengths = lengths_of(cu);
    const c10::Device dev = py::cast<c10::Device>(device);
    py::gil_scoped_release released;
    Packed p = pack_tables(lengths, dev, chunk, true);
    return std::make_tuple(p.chunks, p.ptr, p.tok, p.n_chunks);
  });
  m.def("kda_chunk_fwd", [](const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& g, const Tensor& beta, std::optional<double> scale, const OptTensor& h0,
                            bool want_state, bool l2norm, bool out_fp32) {
    return kda_chunk(q, k, v, g, beta, scale, h0, want_state, l2norm, out_fp32, nullptr);
  }, nogil());
  m.def("kda_chunk_fwd_varlen", [](const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& g, const Tensor& beta, const Tensor& chunks, const Tensor& ptr,
                                   int64_t total, int64_t n_chunks, std::optional<double> scale, const OptTensor& h0, bool want_state, bool l2norm, bool out_fp32) {
    Packed p;
    p.chunks = chunks; p.ptr = ptr; p.n_chunks = n_chunks; p.n_seq = ptr.numel() - 1; p.total = total;
    return kda_chunk(q, k, v, g, beta, scale, h0, want_state, l2norm, out_fp32, &p);
  }, nogil());
  m.def("kda_recurrent_fwd", &kda_recurrent, nogil());
  m.def("chunk_kda", [](const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& g, const Tensor& beta, std::optional<double> scale, const OptTensor& h0,
                        bool want_state, bool l2norm, const py::object& cu, bool out_fp32) {
    const Lengths lengths = lengths_of(cu);
    py::gil_scoped_release released;
    return chunk_kda(q, k, v, g, beta, scale, h0, want_state, l2norm, lengths, out_fp32);
  });
  m.def("kimi_layer", [](const Tensor& x, const std::vector<Tensor>& w, const OptTensor& g1_bias, const OptTensor& norm_w, const std::vector<Tensor>& conv_w,
                         const std::vector<OptTensor>& conv_b, const Tensor& a_log, const Tensor& dt_bias, const std::vector<OptTensor>& conv_s, const OptTensor& rec,
                         bool use_cache, bool silu, double eps, int64_t H, const py::object& cu, const OptTensor& mask) {
    const Lengths lengths = lengths_of(cu);
    py::gil_scoped_release released;
    return kimi_layer(x, w, g1_bias, norm_w, conv_w, conv_b, a_log, dt_bias, conv_s, rec, use_cache, silu, eps, H, lengths, mask);
  });
  m.def("plain_bf16", &plain_bf16);
  m.def("kda_token_supported", &kda_token_supported);
  m.def("kda_token_workspace_bytes", &kda_token_workspace_bytes);
  m.def("kda_token_step", &kda_token_step, nogil());
}

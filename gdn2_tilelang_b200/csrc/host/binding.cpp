// The short calls' host path: argument checks, allocations and launches of one call without going back to Python in
// between. A one-token decode is a few microseconds of device work, and the same sequence in Python (views, shape
// comparisons, a 20-argument foreign call) took 34 us, a layer step of it 165 us.
//
// Every function takes the plain case only -- dense, aligned CUDA tensors of the expected shapes and types on the
// current device -- and returns None for anything else, so that the general path in Python handles it or raises the
// error that belongs to it. Nothing is kept between calls.
#include <ATen/ATen.h>
#include <ATen/autocast_mode.h>
#include <ATen/core/grad_mode.h>
#include <c10/core/impl/TorchDispatchModeTLS.h>
#include <c10/cuda/CUDAFunctions.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/utils/pybind.h>

#include "../../../include/gdn2_b200.h"

namespace py = pybind11;
using at::Tensor;

namespace {

// a tensor of this dtype on the current device, not wrapped by a transform or a subclass
bool unwrapped(const Tensor& t, at::ScalarType dt, c10::DeviceIndex dev) {
  return t.defined() && t.is_cuda() && t.get_device() == dev && t.scalar_type() == dt &&
         !t.is_conj() && !t.is_neg() && t.key_set().has(c10::DispatchKey::CUDA) && !t.key_set().has(c10::DispatchKey::Python) &&
         !t.key_set().has(c10::DispatchKey::FuncTorchBatched) && !t.key_set().has(c10::DispatchKey::FuncTorchGradWrapper) &&
         !t.key_set().has(c10::DispatchKey::Functionalize);
}
// dense and 16-byte aligned
bool dense(const Tensor& t) { return t.is_contiguous() && (reinterpret_cast<uintptr_t>(t.data_ptr()) & 15u) == 0; }
bool plain(const Tensor& t, at::ScalarType dt, c10::DeviceIndex dev) { return unwrapped(t, dt, dev) && dense(t); }

int dtype_code(at::ScalarType dt) {
  return dt == at::kBFloat16 ? GDN2_BF16 : dt == at::kHalf ? GDN2_F16 : dt == at::kFloat ? GDN2_F32 : -1;
}

struct Problem {
  int64_t B, S, H, HK, DK, DV;
  int dtype;
  at::ScalarType type;
  c10::DeviceIndex dev;
};

// q, k, b, g [.., HK, DK] and v, w [.., H, DV] with `lead` leading dimensions (batch, and tokens when lead == 2)
bool plain_tokens(const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& g, const Tensor& b, const Tensor& w, Problem& p,
                  int64_t lead) {
  if (q.dim() != lead + 2 || v.dim() != lead + 2 || !q.is_cuda()) return false;
  p.type = q.scalar_type();
  p.dtype = dtype_code(p.type);
  p.dev = c10::cuda::current_device();
  if (p.dtype < 0 || !plain(q, p.type, p.dev) || !plain(k, p.type, p.dev) || !plain(v, p.type, p.dev) || !plain(b, p.type, p.dev) ||
      !plain(w, p.type, p.dev) || !plain(g, at::kFloat, p.dev))
    return false;
  const auto qs = q.sizes(), vs = v.sizes();
  if (k.sizes() != qs || b.sizes() != qs || g.sizes() != qs || w.sizes() != vs) return false;
  p.B = qs[0];
  p.S = lead == 2 ? qs[1] : 1;
  if (vs[0] != p.B || (lead == 2 && vs[1] != p.S)) return false;
  p.HK = qs[lead]; p.DK = qs[lead + 1];
  p.H = vs[lead]; p.DV = vs[lead + 1];
  return p.B > 0 && p.S > 0 && p.HK > 0 && p.DK > 0 && p.DV > 0 && p.H > 0 && p.H % p.HK == 0;
}

bool plain_state(const Tensor& s, const Problem& p) {
  return plain(s, at::kFloat, p.dev) && s.dim() == 4 && s.size(0) == p.B && s.size(1) == p.H && s.size(2) == p.DK && s.size(3) == p.DV;
}

void* stream_of(const Problem& p) { return c10::cuda::getCurrentCUDAStream(p.dev).stream(); }

// gdn2_decode ([B, n, H, D] tokens) and gdn2_decode_step ([B, H, D]); the state is updated in place. Returns o or None.
std::optional<Tensor> decode(const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& g, const Tensor& b, const Tensor& w,
                  const Tensor& state, std::optional<double> scale) {
  Problem p;
  if (!plain_tokens(q, k, v, g, b, w, p, q.dim() == 3 ? 1 : 2) || !plain_state(state, p)) return std::nullopt;
  Tensor o = at::empty(v.sizes(), v.options().requires_grad(false));
  const float sc = scale ? (float)*scale : (float)(1.0 / std::sqrt((double)p.DK));
  const int rc = gdn2_decode(q.data_ptr(), k.data_ptr(), v.data_ptr(), static_cast<const float*>(g.data_ptr()), b.data_ptr(),
                             w.data_ptr(), static_cast<float*>(state.data_ptr()), o.data_ptr(), p.B, p.S, p.H, p.HK, p.DK, p.DV,
                             p.S, p.S, sc, p.dtype, stream_of(p));
  if (rc != GDN2_OK) return std::nullopt;
  return o;
}

// Whether a prefill of at least 64 tokens is one call of gdn2_prefill_ragged: resolves `path` and gives its workspace
bool ragged_plan(const Problem& p, int& path, size_t& bytes) {
  const int64_t n_full = p.S / 64 * 64;
  if (path == GDN2_PATH_AUTO) path = p.DK == 128 && p.DV == 128 && p.dtype == GDN2_BF16 ? GDN2_PATH_TCGEN05 : GDN2_PATH_SIMT;
  // the caller overlaps the stages of long, uncut problems segment by segment
  if (path != GDN2_PATH_SIMT && n_full / 64 >= 32 && gdn2_prefill_scan_segments(p.B, n_full, p.H, p.DK, p.DV, p.dtype, path) <= 1)
    return false;
  bytes = gdn2_prefill_ragged_workspace_bytes(p.B, p.S, p.H, p.HK, p.DK, p.DV, p.dtype, path);
  return bytes != 0;
}
int64_t ragged_launches(const Problem& p, int path) {
  const int64_t n_full = p.S / 64 * 64;
  const bool tc = path != GDN2_PATH_SIMT;
  const int64_t scans = gdn2_prefill_scan_launches(p.B, n_full, p.H, p.DK, p.DV, p.dtype, path);
  return (tc ? 2 : 1) + scans + (tc && p.S > n_full);
}

// gdn2_prefill_ragged. `side`: the second stream (0: none). Returns (o, final state, kernels launched) or None.
std::optional<std::tuple<Tensor, Tensor, int64_t>> prefill(const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& g, const Tensor& b, const Tensor& w,
                   std::optional<double> scale, const std::optional<Tensor>& state, int path, uint64_t side) {
  Problem p;
  if (q.dim() != 4 || !plain_tokens(q, k, v, g, b, w, p, 2)) return std::nullopt;
  if (state && !plain_state(*state, p)) return std::nullopt;
  size_t bytes = 0;
  if (p.S < 64 || !ragged_plan(p, path, bytes)) return std::nullopt;
  const auto opt = v.options().requires_grad(false);
  Tensor ws = at::empty({(int64_t)bytes}, opt.dtype(at::kByte));
  Tensor o = at::empty(v.sizes(), opt);
  Tensor fin = at::empty({p.B, p.H, p.DK, p.DV}, opt.dtype(at::kFloat));
  const float sc = scale ? (float)*scale : (float)(1.0 / std::sqrt((double)p.DK));
  const int rc = gdn2_prefill_ragged(
      q.data_ptr(), k.data_ptr(), v.data_ptr(), static_cast<const float*>(g.data_ptr()), b.data_ptr(), w.data_ptr(),
      state ? static_cast<const float*>(state->data_ptr()) : nullptr, o.data_ptr(), static_cast<float*>(fin.data_ptr()), ws.data_ptr(),
      bytes, p.B, p.S, p.H, p.HK, p.DK, p.DV, p.S, p.S, sc, p.dtype, path, p.S % 64 ? reinterpret_cast<void*>(side) : nullptr,
      stream_of(p));
  if (rc != GDN2_OK) return std::nullopt;
  return std::make_tuple(o, fin, ragged_launches(p, path));
}


// gdn2_prefill of a prompt shorter than a chunk: the decode of its tokens, `state` updated in place and returned (none: from zero).
// Returns (o, state) or None.
std::optional<std::tuple<Tensor, Tensor>> prefill_short(const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& g, const Tensor& b,
                                                        const Tensor& w, std::optional<double> scale, const std::optional<Tensor>& state) {
  Problem p;
  if (q.dim() != 4 || !plain_tokens(q, k, v, g, b, w, p, 2) || p.S >= 64 || p.DK > 256) return std::nullopt;
  if (state && !plain_state(*state, p)) return std::nullopt;
  const auto opt = v.options().requires_grad(false);
  Tensor o = at::empty(v.sizes(), opt);
  Tensor st = state ? *state : at::zeros({p.B, p.H, p.DK, p.DV}, opt.dtype(at::kFloat));
  const float sc = scale ? (float)*scale : (float)(1.0 / std::sqrt((double)p.DK));
  const int rc = gdn2_decode_tail(q.data_ptr(), k.data_ptr(), v.data_ptr(), static_cast<const float*>(g.data_ptr()), b.data_ptr(), w.data_ptr(),
                                  static_cast<float*>(st.data_ptr()), o.data_ptr(), p.B, p.S, p.H, p.HK, p.DK, p.DV, p.S, p.S, sc, p.dtype,
                                  stream_of(p));
  if (rc != GDN2_OK) return std::nullopt;
  return std::make_tuple(o, st);
}

// What the layer's calls below share: x [B, n, hidden], the cache, the layer's tensors and sizes.
struct Layer {
  const Tensor &state, &w_cat, &A_log, &dt_bias, &norm_w, &o_w;
  const std::optional<Tensor> &conv_state, &conv_w, &conv_b;
  const std::vector<int64_t>& offs;
  int64_t H, HK, DK, DV, K;
  double erase_scale, eps, scale;
  int64_t CC() const { return 2 * HK * DK + H * DV; }       // convolved channels
};

bool plain_layer(Tensor& x, const Layer& l, Problem& p) {
  p.type = x.scalar_type();
  p.dtype = dtype_code(p.type);
  if (p.dtype < 0 || x.dim() != 3 || !x.is_cuda() || x.numel() == 0 || l.DK > 256 || l.DV > 256 || l.offs.size() != 7) return false;
  p.dev = c10::cuda::current_device();
  p.B = x.size(0); p.S = x.size(1); p.H = l.H; p.HK = l.HK; p.DK = l.DK; p.DV = l.DV;
  for (const Tensor* t : {&l.w_cat, &l.A_log, &l.dt_bias, &l.norm_w, &l.o_w})
    if (!plain(*t, p.type, p.dev)) return false;
  // one token out of a prompt that lies in memory whole (x[:, t]): its rows are brought together
  if (p.S == 1 && unwrapped(x, p.type, p.dev) && !dense(x)) x = x.clone(at::MemoryFormat::Contiguous);
  if (!plain(x, p.type, p.dev) || !plain_state(l.state, p) || x.size(2) != l.w_cat.size(1)) return false;
  return l.K >= 2 && l.conv_w && plain(*l.conv_w, p.type, p.dev) && (!l.conv_b || plain(*l.conv_b, p.type, p.dev)) && l.conv_state &&
         plain(*l.conv_state, p.type, p.dev) && l.conv_state->dim() == 3 && l.conv_state->size(0) == p.B &&
         l.conv_state->size(1) == l.CC() && l.conv_state->size(2) == l.K - 1;
}

// The layer stage by stage: projections, gdn2_layer_front, `attend` on the buffers of its inputs and output (true: done),
// gdn2_layer_back, output projection. Returns (out, new convolution cache, kernels of the front and the back launched) or None
// while nothing of the cache has changed, so that the general path can still take the call over.
struct Stages { char *q, *k, *b, *v, *w, *o; float* g; };
template <typename Attend>
std::optional<std::tuple<Tensor, Tensor, int64_t>> layer_stages(const Tensor& x, const Layer& l, const Problem& p, Attend attend) {
  Tensor proj = at::linear(x, l.w_cat);
  if (proj.scalar_type() != p.type || !proj.is_contiguous()) return std::nullopt;       // an autocast region
  const auto opt = x.options().requires_grad(false);
  // one allocation for what lives between the stages, every part 256-byte aligned
  const int64_t esz = p.dtype == GDN2_F32 ? 4 : 2, tokens = p.B * p.S;
  auto part = [](int64_t bytes) { return (bytes + 255) / 256 * 256; };
  const int64_t key = part(tokens * l.HK * l.DK * esz), decay = part(tokens * l.HK * l.DK * 4), value = part(tokens * l.H * l.DV * esz);
  Tensor mid = at::empty({3 * key + decay + 3 * value}, opt.dtype(at::kByte));
  Tensor conv = at::empty({p.B, l.CC(), l.K - 1}, opt);
  char* at_ = static_cast<char*>(mid.data_ptr());
  auto take = [&](int64_t bytes) { char* r = at_; at_ += bytes; return r; };
  Stages m;
  m.q = take(key); m.k = take(key); m.b = take(key); m.g = reinterpret_cast<float*>(take(decay));
  m.v = take(value); m.w = take(value); m.o = take(value);
  void* st = stream_of(p);
  gdn2_layer_front_args a{};
  a.proj = proj.data_ptr(); a.conv_state = l.conv_state->data_ptr(); a.conv_weight = l.conv_w->data_ptr();
  a.conv_bias = l.conv_b ? l.conv_b->data_ptr() : nullptr;
  a.A_log = l.A_log.data_ptr(); a.dt_bias = l.dt_bias.data_ptr();
  a.q = m.q; a.k = m.k; a.v = m.v; a.g = m.g; a.b = m.b; a.w = m.w; a.new_conv_state = conv.data_ptr();
  a.B = p.B; a.S = p.S; a.H = l.H; a.HK = l.HK; a.DK = l.DK; a.DV = l.DV; a.K = l.K; a.NP = proj.size(2);
  a.off_q = l.offs[0]; a.off_k = l.offs[1]; a.off_v = l.offs[2]; a.off_b = l.offs[3]; a.off_w = l.offs[4]; a.off_f = l.offs[5];
  a.erase_scale = (float)l.erase_scale;
  if (gdn2_layer_front(&a, p.dtype, st) != GDN2_OK || !attend(m)) return std::nullopt;
  Tensor normed = at::empty({p.B, p.S, l.H * l.DV}, opt);   // now, where the scan's workspace was
  const int rc = gdn2_layer_back(m.o, proj.data_ptr(), l.norm_w.data_ptr(), normed.data_ptr(), p.B * p.S, l.H, l.DV,
                                 proj.size(2), l.offs[6], (float)l.eps, p.dtype, st);
  if (rc != GDN2_OK) throw std::runtime_error(std::string("gdn2_layer_back: ") + gdn2_status_string(rc));
  // the front kernel writes the new convolution cache itself in its 16-bit forms, else a second one does
  bool fused = p.dtype != GDN2_F32 && l.DK == 128 && l.DV == 128 && l.K == 4 && a.NP % 4 == 0;
  for (int i = 0; i < 6; ++i) fused = fused && l.offs[i] % 4 == 0;
  return std::make_tuple(at::linear(normed, l.o_w), conv, int64_t(fused ? 2 : 3));
}

// GatedDeltaNet2.decode on x [B, n, hidden]: gdn2_layer_step where it applies, else stage by stage. The recurrent state is updated
// in place. Returns (out [B, n, hidden], new convolution cache, kernels launched) or None. `conv_in_place`: the convolution
// cache is updated in place too, or the call is not made.
std::optional<std::tuple<Tensor, Tensor, int64_t>> layer_decode(Tensor x, const Tensor& state, const std::optional<Tensor>& conv_state, const Tensor& w_cat,
                        const std::optional<Tensor>& conv_w, const std::optional<Tensor>& conv_b, const Tensor& A_log,
                        const Tensor& dt_bias, const Tensor& norm_w, const Tensor& o_w, const std::vector<int64_t>& offs, int64_t H,
                        int64_t HK, int64_t DK, int64_t DV, int64_t K, double erase_scale, double eps, double scale, bool conv_in_place) {
  const Layer l{state, w_cat, A_log, dt_bias, norm_w, o_w, conv_state, conv_w, conv_b, offs, H, HK, DK, DV, K, erase_scale, eps, scale};
  Problem p;
  at::NoGradGuard no_grad;
  if (!plain_layer(x, l, p)) return std::nullopt;
  const int64_t hidden = x.size(2);
  // (an autocast region or a dispatch mode would have seen the two linear layers)
  const size_t step_bytes = p.S == 1 && o_w.dim() == 2 && o_w.size(0) == hidden && o_w.size(1) == H * DV &&
                                    !at::autocast::is_autocast_enabled(at::kCUDA) && !c10::impl::TorchDispatchModeTLS::any_modes_set()
                                ? gdn2_layer_step_workspace_bytes(p.B, hidden, H, HK, DK, DV, K, p.dtype)
                                : 0;
  if (step_bytes > 0) {
    const auto opt = x.options().requires_grad(false);
    Tensor ws = at::empty({(int64_t)step_bytes}, opt.dtype(at::kByte)), out = at::empty({p.B, 1, hidden}, opt);
    Tensor conv = conv_in_place ? *conv_state : at::empty({p.B, l.CC(), K - 1}, opt);
    gdn2_layer_step_args s{};
    s.x = x.data_ptr(); s.w_cat = w_cat.data_ptr(); s.conv_state = conv_state->data_ptr(); s.conv_weight = conv_w->data_ptr();
    s.conv_bias = conv_b ? conv_b->data_ptr() : nullptr;
    s.A_log = A_log.data_ptr(); s.dt_bias = dt_bias.data_ptr(); s.norm_weight = norm_w.data_ptr(); s.o_weight = o_w.data_ptr();
    s.state = static_cast<float*>(state.data_ptr()); s.new_conv_state = conv.data_ptr(); s.out = out.data_ptr();
    s.workspace = ws.data_ptr(); s.workspace_bytes = step_bytes;
    s.B = p.B; s.hidden = hidden; s.H = H; s.HK = HK; s.DK = DK; s.DV = DV; s.K = K;
    s.off_q = offs[0]; s.off_k = offs[1]; s.off_v = offs[2]; s.off_b = offs[3]; s.off_w = offs[4]; s.off_f = offs[5]; s.off_gate = offs[6];
    s.erase_scale = (float)erase_scale; s.eps = (float)eps; s.scale = (float)scale;
    const int rc = gdn2_layer_step(&s, p.dtype, stream_of(p));
    if (rc == GDN2_OK) return std::make_tuple(out, conv, int64_t(3));
    // refused before anything ran; after a launch that failed part of the cache may have been written
    if (rc == GDN2_ERR_CUDA) throw std::runtime_error(std::string("gdn2_layer_step: ") + gdn2_status_string(rc));
  }
  if (conv_in_place) return std::nullopt;
  auto res = layer_stages(x, l, p, [&](const Stages& m) {
    return gdn2_decode(m.q, m.k, m.v, m.g, m.b, m.w, static_cast<float*>(state.data_ptr()), m.o, p.B, p.S, H, HK, DK, DV, p.S, p.S,
                       (float)scale, p.dtype, stream_of(p)) == GDN2_OK;
  });
  if (res) std::get<2>(*res) += 1;
  return res;
}

// GatedDeltaNet2.prefill on x [B, S, hidden], continuing from the cache. Returns (out [B, S, hidden], final recurrent state, new
// convolution cache, kernels launched) or None. A prompt shorter than a chunk is decoded and updates the recurrent state in
// place, as gdn2_prefill does.
std::optional<std::tuple<Tensor, Tensor, Tensor, int64_t>> layer_prefill(Tensor x, const Tensor& state, const std::optional<Tensor>& conv_state, const Tensor& w_cat,
                        const std::optional<Tensor>& conv_w, const std::optional<Tensor>& conv_b, const Tensor& A_log,
                        const Tensor& dt_bias, const Tensor& norm_w, const Tensor& o_w, const std::vector<int64_t>& offs, int64_t H,
                        int64_t HK, int64_t DK, int64_t DV, int64_t K, double erase_scale, double eps, double scale, int path, uint64_t side) {
  const Layer l{state, w_cat, A_log, dt_bias, norm_w, o_w, conv_state, conv_w, conv_b, offs, H, HK, DK, DV, K, erase_scale, eps, scale};
  Problem p;
  at::NoGradGuard no_grad;
  if (!plain_layer(x, l, p)) return std::nullopt;
  size_t bytes = 0;
  if (p.S >= 64 && !ragged_plan(p, path, bytes)) return std::nullopt;
  Tensor fin = state;
  const auto opt = x.options().requires_grad(false);
  int64_t launched = 1;
  auto res = layer_stages(x, l, p, [&](const Stages& m) {
    if (p.S < 64)
      return gdn2_decode_tail(m.q, m.k, m.v, m.g, m.b, m.w, static_cast<float*>(state.data_ptr()), m.o, p.B, p.S, H, HK, DK, DV, p.S, p.S,
                              (float)scale, p.dtype, stream_of(p)) == GDN2_OK;
    Tensor ws = at::empty({(int64_t)bytes}, opt.dtype(at::kByte));
    fin = at::empty({p.B, H, DK, DV}, opt.dtype(at::kFloat));
    launched = ragged_launches(p, path);
    return gdn2_prefill_ragged(m.q, m.k, m.v, m.g, m.b, m.w, static_cast<const float*>(state.data_ptr()), m.o, static_cast<float*>(fin.data_ptr()),
                               ws.data_ptr(), bytes, p.B, p.S, H, HK, DK, DV, p.S, p.S, (float)scale, p.dtype, path,
                               p.S % 64 ? reinterpret_cast<void*>(side) : nullptr, stream_of(p)) == GDN2_OK;
  });
  if (!res) return std::nullopt;
  return std::make_tuple(std::get<0>(*res), fin, std::get<1>(*res), std::get<2>(*res) + launched);
}

// The state of a list of parameters: where each lies, its version and its type. Equal bytes = nothing was replaced,
// moved, converted or written to since.
py::bytes parameter_key(const std::vector<Tensor>& params) {
  std::string key;
  for (const Tensor& t : params) {
    const uint64_t rec[3] = {reinterpret_cast<uint64_t>(t.data_ptr()), (uint64_t)t._version(), (uint64_t)t.scalar_type()};
    key.append(reinterpret_cast<const char*>(rec), sizeof(rec));
  }
  return py::bytes(key);
}

}  // namespace

PYBIND11_MODULE(_gdn2_host, m) {
  // none of them touches Python objects: the lock is released meanwhile, as a foreign call does
  const auto unlocked = py::call_guard<py::gil_scoped_release>();
  m.def("decode", &decode, unlocked);
  m.def("prefill", &prefill, unlocked);
  m.def("prefill_short", &prefill_short, unlocked);
  m.def("layer_decode", &layer_decode, unlocked);
  m.def("layer_prefill", &layer_prefill, unlocked);
  m.def("parameter_key", &parameter_key);
}

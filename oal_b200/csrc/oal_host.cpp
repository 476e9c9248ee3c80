// Host path of the prepared call: checks, allocation, the autograd node and the status queue, on top of the C ABI.
//
// At one or two (batch row, KV head) units the kernels of a step take less time than Python needs to marshal its
// calls, so everything a repeated call does between the caller's tensors and the launches is here: one pass over
// the arguments, one allocation per result, saved buffer and workspace (six forward, up to five backward, all from the
// caching allocator), one C call.  The argument
// checks of this file only decide whether the call is the prepared one; when they say no, the Python layer goes
// through the full validation and raises what it always raised.
//
// The autograd node covers the packed factor too (oal_forward_packed / oal_backward_packed), so a step has one node
// where the expansion and the operator used to have two.
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAGraphsC10Utils.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/extension.h>

#include <atomic>
#include <deque>
#include <map>
#include <mutex>
#include <optional>

#include "../../include/oal_b200.h"

namespace {

using at::Tensor;
using torch::autograd::AutogradContext;
using torch::autograd::variable_list;

[[noreturn]] void raise_code(int64_t rc) {
  const std::string msg = oal_last_error_string();
  if (rc == OAL_ERR_DTYPE) throw py::type_error(msg);
  if (rc == OAL_ERR_ARGUMENT || rc == OAL_ERR_WORKSPACE) throw py::value_error(msg);
  throw std::runtime_error(msg);
}
inline void check_rc(int64_t rc) {
  if (rc < 0) raise_code(rc);
}

// ---- status words of calls whose result is looked at later ------------------------------------------
struct Pending {
  int64_t ticket, call_id;
  const char* what;
};
std::mutex g_pending_mutex;
std::map<int, std::deque<Pending>> g_pending;
std::atomic<int64_t> g_call_ids{1};
constexpr size_t kPendingLimit = 256;

void raise_for_bits(int bits, const std::string& where) {
  if (bits & OAL_STATUS_WAIT_TIMEOUT) {
    char word[32];
    snprintf(word, sizeof(word), "%#x", bits);
    throw std::runtime_error("oal_b200 kernel gave up on a bounded wait (device status word " + std::string(word) + ")" + where);
  }
  if (bits & OAL_STATUS_BAD_LAYOUT) throw py::value_error("a head's group layout does not fit the kernels" + where);
  if (bits & (OAL_STATUS_NONFINITE | OAL_STATUS_DENOMINATOR))
    throw std::runtime_error("HD Block-GEMM denominator must be finite and strictly positive (device status " + std::to_string(bits) +
                             ")" + where);
}

// Finished entries in order; the first that reports a problem is dropped and raised.  With `block` also unfinished ones,
// until `leave` are left.  Called without the GIL (see Unlocked).
void drain(int device, bool block, size_t leave = 0) {
  for (;;) {
    Pending e;
    bool wait;
    {
      std::lock_guard<std::mutex> lock(g_pending_mutex);
      auto it = g_pending.find(device);
      if (it == g_pending.end() || it->second.empty()) return;
      e = it->second.front();
      wait = block && it->second.size() > leave;
    }
    int32_t word = 0;
    const int rc = oal_status_poll(e.ticket, wait ? 1 : 0, &word);
    if (rc == 0) return;
    {
      std::lock_guard<std::mutex> lock(g_pending_mutex);
      auto& q = g_pending[device];
      if (q.empty() || q.front().ticket != e.ticket) continue;      // another thread took it
      q.pop_front();
    }
    check_rc(rc);
    if (word) raise_for_bits(word, std::string(" [") + e.what + ", call " + std::to_string(e.call_id) + "]");
  }
}

void enqueue(int device, int64_t ticket, const char* what) {
  bool full;
  {
    std::lock_guard<std::mutex> lock(g_pending_mutex);
    auto& q = g_pending[device];
    q.push_back(Pending{ticket, g_call_ids++, what});
    full = q.size() > kPendingLimit;
  }
  if (full) drain(device, true, kPendingLimit);
}

// Gives up the GIL where it is held (a call from Python; the autograd engine's threads come without it): this file
// waits for calls, and the work that they wait for may need another Python thread's launch.
struct Unlocked {
  std::optional<py::gil_scoped_release> release;
  Unlocked() {
    if (PyGILState_Check()) release.emplace();
  }
};

void check_pending(bool block, int device) {
  std::vector<int> devices;
  {
    std::lock_guard<std::mutex> lock(g_pending_mutex);
    for (auto& kv : g_pending)
      if (device < 0 || kv.first == device) devices.push_back(kv.first);
  }
  py::gil_scoped_release release;
  for (int d : devices) drain(d, block);
}

// words of calls recorded into a CUDA graph, handed to the Python list that keeps them
std::mutex g_captured_mutex;
std::vector<std::tuple<int, Tensor, std::string>> g_captured;

std::vector<std::tuple<int, Tensor, std::string>> take_captured() {
  std::lock_guard<std::mutex> lock(g_captured_mutex);
  return std::move(g_captured);
}

bool capturing() {
  return c10::cuda::currentStreamCaptureStatusMayInitCtx() != c10::cuda::CaptureStatus::None;
}

// ---- the prepared call --------------------------------------------------------------------------------
struct Prepared {
  OalProblem problem{};          // grad_mask of the preparation
  int64_t B, Hq, Hkv, N, D, Dv, G, P;
  at::ScalarType dtype, out_dtype, kernel_out;
  c10::Device device{c10::kCUDA, 0};
  Tensor dim_perm, group_start;
  float eps;
  int64_t forward_bytes, backward_bytes, saved_bytes, coef_floats;
  bool grad[4];                  // q, k, v, factor
  bool token_major;

  bool takes(const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& f) const {
    auto shape = [&](const Tensor& t, int64_t h, int64_t d) {
      return t.dim() == 4 && t.size(0) == B && t.size(1) == h && t.size(2) == N && t.size(3) == d && t.scalar_type() == dtype &&
             t.device() == device && t.layout() == c10::kStrided && t.is_contiguous();
    };
    if (!shape(q, Hq, D) || !shape(k, Hkv, D) || !shape(v, Hkv, Dv)) return false;
    if (f.scalar_type() != at::kFloat || f.device() != device || f.dim() < 1 || f.dim() > 2 || f.size(-1) != P) return false;
    if (f.dim() == 2 && f.size(0) != Hq) return false;
    // forward-mode tangents: the operator has none, and the Python layer says so
    const auto tangent = [](const Tensor& t) {
      const auto* meta = torch::autograd::impl::get_autograd_meta(t);
      return meta && meta->fw_grad(/*level=*/0, t).defined();
    };
    if (tangent(q) || tangent(k) || tangent(v) || tangent(f)) return false;
    const bool live = at::GradMode::is_enabled();
    return (live && q.requires_grad()) == grad[0] && (live && k.requires_grad()) == grad[1] &&
           (live && v.requires_grad()) == grad[2] && (live && f.requires_grad()) == grad[3];
  }
};

// A contiguous tensor may start anywhere in its storage; the tensor-core kernels read 16 bytes at a time.  (The exact
// fp32 kernels look at the alignment themselves.)
Tensor on_boundary(const Prepared& p, const Tensor& t) {
  const bool off = p.problem.precision == OAL_PRECISION_BF16_TENSORCORE && t.defined() && (reinterpret_cast<uintptr_t>(t.data_ptr()) & 15);
  return off ? t.clone() : t;
}
Tensor pad_last(const Prepared& p, const Tensor& t) {
  const int64_t d = t.size(-1);
  return d == OAL_HEAD_DIM ? on_boundary(p, t) : at::constant_pad_nd(t, {0, OAL_HEAD_DIM - d}).contiguous();
}
inline void* ptr(const Tensor& t) { return t.defined() ? t.data_ptr() : nullptr; }
inline float* fptr(const Tensor& t) { return static_cast<float*>(ptr(t)); }

struct Forward {
  Tensor out, num, den, saved, meta, q, k, v, factor;
};

// meta: [fwd status, fwd counter, bwd status, unused] then A, B, C
constexpr int64_t kMetaWords = 4;

Forward forward_call(const Prepared& p, const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& f, bool blocking) {
  const int dev = p.device.index();
  c10::cuda::CUDAGuard guard(p.device);
  const bool recording = capturing();
  if (!recording) drain(dev, false);
  Forward r;
  r.q = pad_last(p, q);
  r.k = pad_last(p, k);
  r.v = pad_last(p, v);
  r.factor = f.contiguous();
  const auto opt = q.options().requires_grad(false);
  r.out = at::empty(p.token_major ? at::IntArrayRef({p.B, p.N, p.Hq, OAL_HEAD_DIM}) : at::IntArrayRef({p.B, p.Hq, p.N, OAL_HEAD_DIM}),
                    opt.dtype(p.kernel_out));
  r.num = at::empty({p.B, p.Hq, p.N, OAL_HEAD_DIM}, opt.dtype(at::kFloat));
  r.den = at::empty({p.B, p.Hq, p.N, 1}, opt.dtype(at::kFloat));
  r.meta = at::empty({kMetaWords + p.coef_floats}, opt.dtype(at::kFloat));
  if (p.saved_bytes) r.saved = at::empty({p.saved_bytes}, opt.dtype(at::kByte));
  Tensor ws = at::empty({std::max<int64_t>(p.forward_bytes, 16)}, opt.dtype(at::kByte));
  int32_t* status = static_cast<int32_t*>(r.meta.data_ptr());
  int64_t ticket = 0;
  check_rc(oal_forward_packed(&p.problem, ptr(r.q), ptr(r.k), ptr(r.v), static_cast<int32_t*>(ptr(p.dim_perm)),
                              static_cast<int32_t*>(ptr(p.group_start)), fptr(r.factor), r.factor.dim() == 1 ? 1 : (int)r.factor.size(0),
                              p.eps, fptr(r.meta) + kMetaWords, ptr(r.out), fptr(r.num), fptr(r.den), ptr(r.saved), ptr(ws),
                              (size_t)ws.numel(), status, recording ? nullptr : &ticket,
                              c10::cuda::getCurrentCUDAStream(dev).stream()));
  if (recording) {
    std::lock_guard<std::mutex> lock(g_captured_mutex);
    g_captured.emplace_back(dev, r.meta.view(at::kInt).slice(0, 0, 1), "forward");
  } else if (blocking) {
    int32_t word = 0;
    check_rc(oal_status_poll(ticket, 1, &word));
    if (word) raise_for_bits(word, "");
  } else {
    enqueue(dev, ticket, "forward");
  }
  if (p.Dv != OAL_HEAD_DIM) r.out = r.out.slice(-1, 0, p.Dv).contiguous();
  if (p.out_dtype != p.kernel_out) r.out = r.out.to(p.out_dtype);
  return r;
}

// gradients of the outputs as the kernels read them
Tensor upstream(const Prepared& p, const Tensor& g, at::ScalarType dtype, bool pad) {
  if (!g.defined()) return g;
  Tensor t = g.to(dtype);
  if (pad && t.size(-1) != OAL_HEAD_DIM) t = at::constant_pad_nd(t, {0, OAL_HEAD_DIM - t.size(-1)});
  return on_boundary(p, t.contiguous());
}

struct PackedNode : torch::autograd::Function<PackedNode> {
  static variable_list forward(AutogradContext* ctx, const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& f,
                               std::shared_ptr<Prepared> p) {
    at::AutoDispatchBelowADInplaceOrView below;
    ctx->set_materialize_grads(false);
    Forward r = forward_call(*p, q, k, v, f, false);
    const bool narrow = p->Dv != OAL_HEAD_DIM;
    Tensor num = narrow ? r.num.slice(-1, 0, p->Dv).contiguous() : r.num;
    // the padded numerator of narrow heads is what the kernels read back; otherwise it is the output itself
    ctx->save_for_backward({r.q, r.k, r.v, r.factor, narrow ? r.num : num, r.den, r.saved, r.meta});
    ctx->saved_data["prepared"] = c10::IValue::make_capsule(c10::make_intrusive<Holder>(p));
    return {r.out, num, r.den};
  }

  struct Holder : torch::CustomClassHolder {
    std::shared_ptr<Prepared> p;
    explicit Holder(std::shared_ptr<Prepared> x) : p(std::move(x)) {}
  };

  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    TORCH_CHECK(!at::GradMode::is_enabled(), "HD Block-GEMM does not support double backward");
    variable_list result(5);
    if (!grads[0].defined() && !grads[1].defined() && !grads[2].defined()) return result;
    auto holder = ctx->saved_data["prepared"].toCapsule();
    const Prepared& p = *static_cast<Holder*>(holder.get())->p;
    const variable_list s = ctx->get_saved_variables();
    // saved-tensor hooks may hand back copies that start elsewhere
    const Tensor q = on_boundary(p, s[0]), k = on_boundary(p, s[1]), v = on_boundary(p, s[2]), num = on_boundary(p, s[4]),
                 saved = on_boundary(p, s[6]);
    const Tensor &factor = s[3], &den = s[5], &meta = s[7];
    const int dev = p.device.index();
    c10::cuda::CUDAGuard guard(p.device);
    const bool recording = capturing();
    if (!recording) drain(dev, false);
    const Tensor go = upstream(p, grads[0], p.kernel_out, true), gn = upstream(p, grads[1], at::kFloat, true), gd = upstream(p, grads[2], at::kFloat, false);
    Tensor d[4];
    if (p.grad[0]) d[0] = at::empty_like(q);
    if (p.grad[1]) d[1] = at::empty_like(k);
    if (p.grad[2]) d[2] = at::empty_like(v);
    if (p.grad[3]) d[3] = at::empty_like(factor);
    Tensor ws = at::empty({std::max<int64_t>(p.backward_bytes, 16)}, q.options().dtype(at::kByte));
    int32_t* status = static_cast<int32_t*>(meta.data_ptr()) + 2;
    // in the backward only a bounded wait that gave up can set the word, and only tensor-core kernels wait
    const bool report = p.problem.precision == OAL_PRECISION_BF16_TENSORCORE && !recording;
    int64_t ticket = 0;
    check_rc(oal_backward_packed(&p.problem, ptr(q), ptr(k), ptr(v), static_cast<int32_t*>(ptr(p.dim_perm)),
                                 static_cast<int32_t*>(ptr(p.group_start)), fptr(factor), factor.dim() == 1 ? 1 : (int)factor.size(0),
                                 fptr(meta) + kMetaWords, fptr(num), fptr(den), ptr(saved), ptr(go), fptr(gn), fptr(gd), ptr(d[0]),
                                 ptr(d[1]), ptr(d[2]), fptr(d[3]), ptr(ws), (size_t)ws.numel(), status, report ? &ticket : nullptr,
                                 c10::cuda::getCurrentCUDAStream(dev).stream()));
    if (recording) {
      std::lock_guard<std::mutex> lock(g_captured_mutex);
      g_captured.emplace_back(dev, meta.view(at::kInt).slice(0, 2, 3), "backward");
    } else if (report) {
      enqueue(dev, ticket, "backward");
    }
    if (p.D != OAL_HEAD_DIM)
      for (int i = 0; i < 2; ++i)
        if (d[i].defined()) d[i] = d[i].slice(-1, 0, p.D).contiguous();
    if (p.Dv != OAL_HEAD_DIM && d[2].defined()) d[2] = d[2].slice(-1, 0, p.Dv).contiguous();
    for (int i = 0; i < 4; ++i) result[i] = d[i];
    return result;
  }
};

// (out, numerator, denominator), or None when the arguments are not those of the preparation
py::object run(const std::shared_ptr<Prepared>& p, const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& f) {
  if (!p->takes(q, k, v, f)) return py::none();
  Tensor out, num, den;
  {
    Unlocked unlocked;
    if (p->grad[0] || p->grad[1] || p->grad[2] || p->grad[3]) {
      variable_list o = PackedNode::apply(q, k, v, f, p);
      out = o[0], num = o[1], den = o[2];
    } else {
      at::AutoDispatchBelowADInplaceOrView below;
      Forward r = forward_call(*p, q, k, v, f, true);
      out = r.out, den = r.den;
      num = p->Dv != OAL_HEAD_DIM ? r.num.slice(-1, 0, p->Dv).contiguous() : r.num;
    }
  }
  return py::make_tuple(out, num, den);
}

std::shared_ptr<Prepared> prepare(py::bytes problem, std::vector<int64_t> geometry, int64_t groups, at::ScalarType dtype,
                                  at::ScalarType out_dtype, int device, Tensor dim_perm, Tensor group_start, double eps,
                                  std::vector<int64_t> bytes, std::vector<bool> grad) {
  auto p = std::make_shared<Prepared>();
  const std::string raw = problem;
  TORCH_CHECK(raw.size() == sizeof(OalProblem), "problem struct size");
  memcpy(&p->problem, raw.data(), sizeof(OalProblem));
  p->B = geometry[0]; p->Hq = geometry[1]; p->Hkv = geometry[2]; p->N = geometry[3]; p->D = geometry[4]; p->Dv = geometry[5];
  p->G = groups;
  p->P = (groups + 1) * (groups + 2) / 2;
  p->dtype = dtype;
  p->out_dtype = out_dtype;
  p->kernel_out = out_dtype == at::kDouble ? at::kFloat : out_dtype;
  p->device = c10::Device(c10::kCUDA, (c10::DeviceIndex)device);
  p->dim_perm = dim_perm;
  p->group_start = group_start;
  p->eps = (float)eps;
  // at least what this library needs, whatever a preparation that was stored by another build says: a forward call has no
  // length of the saved state to check
  for (int phase = 0; phase < 3; ++phase) bytes[phase] = std::max(bytes[phase], (int64_t)oal_workspace_bytes(&p->problem, phase));
  p->forward_bytes = bytes[0]; p->backward_bytes = bytes[1]; p->saved_bytes = bytes[2];
  p->coef_floats = p->Hq * (1 + groups + groups * groups);
  for (int i = 0; i < 4; ++i) p->grad[i] = grad[i];
  p->token_major = p->problem.flags & OAL_FLAG_OUT_TOKEN_MAJOR;
  return p;
}

// ---- dimension groups ---------------------------------------------------------------------------------
// ids [rows, D] of any device -> (problem, dim_perm [hq, 64], group_start [hq, 17]) with problem 0 none, 1 an id out
// of range, 2 ids of a row not a prefix.  One copy down, the counting sort on the host, one copy up; a single row
// stands for every head.  Dimensions beyond D are padding and belong to group 0.
std::tuple<int, Tensor, Tensor> group_tables(const Tensor& ids, int64_t hq, int64_t gmax) {
  const c10::Device device = ids.device();
  Tensor host;
  {
    Unlocked unlocked;      // waits for the work that writes the ids
    host = ids.detach().to(at::kCPU, at::kLong).contiguous();
  }
  const int64_t rows = host.size(0), d = host.size(1);
  const int64_t* id = host.data_ptr<int64_t>();
  for (int64_t r = 0; r < rows; ++r) {
    std::vector<char> used((size_t)gmax, 0);
    for (int64_t x = 0; x < d; ++x) {
      const int64_t g = id[r * d + x];
      if (g < 0 || g >= gmax) return {1, Tensor(), Tensor()};
      used[(size_t)g] = 1;
    }
    for (int64_t g = 1; g < gmax; ++g)
      if (used[(size_t)g] && !used[(size_t)g - 1]) return {2, Tensor(), Tensor()};
    if (!used[0]) return {2, Tensor(), Tensor()};
  }
  if (d > OAL_HEAD_DIM || gmax > OAL_MAX_GROUPS) return {0, Tensor(), Tensor()};      // refused by the plan
  const int64_t perm_words = hq * OAL_HEAD_DIM, words = perm_words + hq * (OAL_MAX_GROUPS + 1);
  Tensor up = at::empty({words}, at::TensorOptions().dtype(at::kInt).pinned_memory(device.is_cuda()));
  int32_t* perm = up.data_ptr<int32_t>();
  int32_t* start = perm + perm_words;
  for (int64_t h = 0; h < hq; ++h) {
    const int64_t* row = id + (rows == 1 ? 0 : h) * d;
    int32_t* st = start + h * (OAL_MAX_GROUPS + 1);
    int count[OAL_MAX_GROUPS] = {0};
    for (int64_t x = 0; x < OAL_HEAD_DIM; ++x) ++count[x < d ? row[x] : 0];
    st[0] = 0;
    for (int g = 0; g < OAL_MAX_GROUPS; ++g) st[g + 1] = st[g] + count[g];
    int at_[OAL_MAX_GROUPS];
    for (int g = 0; g < OAL_MAX_GROUPS; ++g) at_[g] = st[g];
    for (int64_t x = 0; x < OAL_HEAD_DIM; ++x) perm[h * OAL_HEAD_DIM + at_[x < d ? row[x] : 0]++] = (int32_t)x;
  }
  const Tensor table = device.is_cuda() ? up.to(device, at::kInt, /*non_blocking=*/true) : up;
  return {0, table.narrow(0, 0, perm_words).view({hq, OAL_HEAD_DIM}),
          table.narrow(0, perm_words, words - perm_words).view({hq, OAL_MAX_GROUPS + 1})};
}

}  // namespace

PYBIND11_MODULE(_host, m) {
  py::class_<Prepared, std::shared_ptr<Prepared>>(m, "Prepared");
  m.def("prepare", &prepare);
  m.def("run", &run);
  m.def("group_tables", &group_tables);
  m.def("check_pending", &check_pending);
  m.def("next_call_id", [] { return g_call_ids++; });
  m.def("take_captured", &take_captured);
}

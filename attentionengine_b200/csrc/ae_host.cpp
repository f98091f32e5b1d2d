// The operators' host path as one native call each: checks, allocations, parameter blocks, launches (through the C ABI of
// include/ae_b200.h) and the autograd nodes.
//
// Why native: at the sizes of a decode step or of a small training step the kernels take 10 - 40 us, and the same path in
// Python (ctypes structures, torch.autograd.Function in both directions) took 28 us for a split-KV decode and 195 us for
// an attention forward + backward of 44 us of kernels.
//
// Convention: a call whose tensors do not fit its engine returns None without launching anything; the Python front end
// then runs its own checks, which raise the error that names the reason.
#include <Python.h>
#include <c10/cuda/CUDAGraphsC10Utils.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <cuda_runtime_api.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/function.h>
#include <torch/csrc/autograd/functions/utils.h>
#include <torch/csrc/autograd/saved_variable.h>
#include <torch/csrc/autograd/variable.h>
#include <torch/csrc/jit/frontend/tracer.h>
#include <torch/csrc/utils/pybind.h>
#include <ATen/ATen.h>

#include <algorithm>
#include <cstring>
#include <memory>
#include <mutex>
#include <optional>
#include <vector>

#include "../../include/ae_b200.h"

namespace py = pybind11;
using at::Tensor;
using torch::autograd::Node;
using torch::autograd::SavedVariable;
using torch::autograd::variable_list;

namespace {

// ---------------------------------------------------------------------------------------------------- errors
// AeError (attentionengine_b200.runtime), also out of autograd's worker threads
[[noreturn]] void throw_ae(int rc, const char* what) {
  const std::string text = std::string(what) + ": " + ae_strerror(rc) + " - " + ae_last_error();
  py::gil_scoped_acquire gil;
  py::object cls = py::module_::import("attentionengine_b200.runtime").attr("AeError");
  PyErr_SetString(cls.ptr(), text.c_str());
  python_error err;
  err.persist();
  throw err;
}
void check(int rc, const char* what) {
  if (rc != AE_OK) throw_ae(rc, what);
}

// A Python object that a node holds; released with the interpreter's lock, wherever the node dies.
std::shared_ptr<PyObject> hold(py::handle h) {
  Py_INCREF(h.ptr());
  return std::shared_ptr<PyObject>(h.ptr(), [](PyObject* p) {
    if (Py_IsInitialized()) {
      py::gil_scoped_acquire gil;
      Py_DECREF(p);
    }
  });
}

// Runs a Python call from a node; a Python exception travels on through autograd unchanged.
template <class F>
auto with_python(F&& f) {
  py::gil_scoped_acquire gil;
  try {
    return f();
  } catch (py::error_already_set& e) {
    e.restore();
    python_error err;
    err.persist();
    throw err;
  }
}

// ---------------------------------------------------------------------------------------------------- common
struct Custom {
  int slot;
  bool is16;
  std::vector<int> dim_slots;
};

struct Plan {
  at::ScalarType dtype = at::kHalf;
  Tensor status;  // one word per engine; reallocated when the engine moves to another device, under `mu`
  Tensor status_for(const Tensor& like) {
    std::lock_guard<std::mutex> lk(mu);
    if (!status.defined() || status.device() != like.device())
      status = at::zeros({1}, like.options().dtype(at::kInt));
    return status;
  }
  // the front end's side, which holds the interpreter's lock: calls in other threads do not
  Tensor status_now() {
    std::lock_guard<std::mutex> lk(mu);
    return status;
  }
  void set_status(Tensor t) {
    std::lock_guard<std::mutex> lk(mu);
    status = std::move(t);
  }
  std::mutex mu;
};

uint32_t* word(const Tensor& status) { return reinterpret_cast<uint32_t*>(status.data_ptr()); }

void* handle(uint64_t h) { return reinterpret_cast<void*>(h); }

void strides3(const Tensor& t, int64_t (&st)[3]) {
  st[0] = t.stride(0);
  st[1] = t.stride(1);
  st[2] = t.stride(2);
}

bool good4(const Tensor& t, at::ScalarType dtype) {
  return t.is_cuda() && t.scalar_type() == dtype && t.dim() == 4 && t.stride(3) == 1;
}

void* stream_of(const Tensor& t) { return c10::cuda::getCurrentCUDAStream(t.device().index()).stream(); }
bool capturing(void* stream) {
  cudaStreamCaptureStatus s = cudaStreamCaptureStatusNone;
  if (cudaStreamIsCapturing((cudaStream_t)stream, &s) == cudaSuccess) return s != cudaStreamCaptureStatusNone;
  (void)cudaGetLastError();  // the default stream while another one captures: the launch will say so
  return false;
}

bool wants_grad(std::initializer_list<const Tensor*> ts) {
  if (!at::GradMode::is_enabled()) return false;
  for (const Tensor* t : ts)
    if (t->defined() && t->requires_grad()) return true;
  return false;
}

// Calls that a native node cannot stand for: it has no forward-mode rule (the result would lose the tangent in silence), and
// torch.jit.trace would record the result's allocation and not the kernel.  The front end takes them through
// torch.autograd.Function, which PyTorch knows to refuse and to record.
bool needs_function(std::initializer_list<const Tensor*> ts) {
  if (torch::jit::tracer::isTracing()) return true;
  for (const Tensor* t : ts)
    if (torch::autograd::isFwGradDefined(*t)) return true;
  return false;
}

std::vector<Tensor> tensors_of(const py::handle& seq) {
  std::vector<Tensor> out;
  if (seq.is_none()) return out;
  for (auto h : py::reinterpret_borrow<py::sequence>(seq)) out.push_back(h.cast<Tensor>());
  return out;
}

// Pointers and strides of the custom inputs, by the slots the generated functors read; false when one does not fit.  A decode
// call takes no tile-shaped input, and of the others whatever has the dims it indexes; the rest need the dims of their spec.
bool custom_args(const std::vector<Custom>& specs, std::vector<Tensor>& ts, at::ScalarType dtype, int64_t Sq, int64_t Skv,
                 bool decode, const void* (&ptr)[AE_MAX_CUSTOM_INPUTS], int64_t (&st)[AE_MAX_CUSTOM_INPUTS][4]) {
  if (specs.size() != ts.size()) return false;
  for (size_t i = 0; i < specs.size(); ++i) {
    const Custom& sp = specs[i];
    if (!ts[i].is_cuda() || (!decode && (size_t)ts[i].dim() != sp.dim_slots.size())) return false;
    if (sp.is16 && (decode || Sq % 128 || Skv % 128)) return false;
    for (size_t d = ts[i].dim(); d < sp.dim_slots.size(); ++d)
      if (sp.dim_slots[d] >= 0) return false;
    const at::ScalarType want = sp.is16 ? dtype : at::kFloat;
    if (ts[i].scalar_type() != want) ts[i] = ts[i].to(want);
    ptr[sp.slot] = ts[i].data_ptr();
    for (size_t d = 0; d < sp.dim_slots.size(); ++d)
      if (sp.dim_slots[d] >= 0 && ts[i].size(d) > 1) st[sp.slot][sp.dim_slots[d]] = ts[i].stride(d);
  }
  return true;
}

std::vector<Custom> customs_from(const py::list& specs) {
  std::vector<Custom> out;
  for (auto h : specs) {
    auto t = h.cast<py::tuple>();
    out.push_back({t[0].cast<int>(), t[1].cast<bool>(), t[2].cast<std::vector<int>>()});
  }
  return out;
}

// ---------------------------------------------------------------------------------------------------- attention
struct AttnPlan : Plan {
  void* fwd = nullptr;
  void *prep = nullptr, *fused = nullptr, *cast = nullptr;  // one-pass backward, set when it is first needed
  int D = 0, DV = 0, n_final = 0;
  bool uses_doosum = false;
  std::vector<Custom> custom;
};

struct Dims {
  int B, Sq, Hq, Skv, Hkv;
};
bool attn_dims(const AttnPlan& p, const Tensor& q, const Tensor& k, const Tensor& v, Dims& d) {
  if (!good4(q, p.dtype) || !good4(k, p.dtype) || !good4(v, p.dtype)) return false;
  d = {(int)q.size(0), (int)q.size(1), (int)q.size(2), (int)k.size(1), (int)k.size(2)};
  return q.size(3) == p.D && k.size(3) == p.D && v.size(3) == p.DV && d.Hkv > 0 && d.Hq % d.Hkv == 0 && v.size(1) == d.Skv &&
         v.size(2) == d.Hkv && k.size(0) == d.B && v.size(0) == d.B;
}

struct AttnNode : Node {
  std::shared_ptr<AttnPlan> plan;
  std::shared_ptr<PyObject> eng;
  SavedVariable q, k, v, o;
  std::vector<SavedVariable> finals, custom;
  std::vector<Tensor> lists;
  Dims d{};
  Tensor status;

  variable_list apply(variable_list&& grads) override {
    variable_list out(3 + custom.size());
    if (!grads[0].defined()) grads[0] = input_metadata(0).zeros_like();  // as torch.autograd.Function does
    Tensor Q, K, V, O;
    std::vector<Tensor> F, C, lists;
    {
      std::lock_guard<std::mutex> lock(mutex_);
      Q = q.unpack(), K = k.unpack(), V = v.unpack(), O = o.unpack(shared_from_this());
      for (auto& f : finals) F.push_back(f.unpack());
      for (auto& c : custom) C.push_back(c.unpack());
      lists = this->lists;
    }
    at::AutoGradMode no_grad(false);
    c10::cuda::CUDAGuard guard(Q.device());
    Tensor dO = grads[0];
    const bool native = with_python([&] {
      py::handle e(eng.get());
      return e.attr("_native_bwd")(d.B, d.Hq, d.Sq, (int)Q.device().index()).cast<bool>();
    });
    if (!native) {
      return with_python([&] {
        py::handle e(eng.get());
        py::object l = py::none();
        if (!lists.empty()) l = py::make_tuple(lists[0], lists[1], lists[2], lists[3]);
        py::tuple g = e.attr("_launch_bwd")(Q, K, V, O, dO, F, py::cast(C).cast<py::tuple>(), l);
        for (int i = 0; i < 3; ++i) out[i] = g[i].cast<Tensor>();
        return out;
      });
    }
    if (dO.stride(3) != 1 || dO.stride(2) % 8 || dO.stride(1) % 8 || reinterpret_cast<uintptr_t>(dO.data_ptr()) % 16)
      dO = dO.contiguous();
    Tensor dq = at::empty_like(Q), dk = at::empty_like(K), dv = at::empty_like(V);
    AeAttnBwdParams p;
    memset(&p, 0, sizeof p);
    p.q = Q.data_ptr(); p.k = K.data_ptr(); p.v = V.data_ptr(); p.o = O.data_ptr(); p.d_o = dO.data_ptr();
    p.dq = dq.data_ptr(); p.dk = dk.data_ptr(); p.dv = dv.data_ptr();
    strides3(Q, p.q_stride); strides3(K, p.k_stride); strides3(V, p.v_stride); strides3(O, p.o_stride);
    strides3(dO, p.do_stride); strides3(dq, p.dq_stride); strides3(dk, p.dk_stride); strides3(dv, p.dv_stride);
    for (size_t i = 0; i < F.size(); ++i) p.final_rowscales[i] = (const float*)F[i].data_ptr();
    custom_args(plan->custom, C, plan->dtype, d.Sq, d.Skv, false, p.custom, p.custom_stride);
    if (!lists.empty()) {
      p.block_count = (const int32_t*)lists[0].data_ptr(); p.block_index = (const int32_t*)lists[1].data_ptr();
      p.block_count_t = (const int32_t*)lists[2].data_ptr(); p.block_index_t = (const int32_t*)lists[3].data_ptr();
    }
    p.B = d.B; p.Hq = d.Hq; p.Hkv = d.Hkv; p.Sq = d.Sq; p.Skv = d.Skv;
    p.status = word(status);
    // fp32 scratch in one allocation: dQ accumulator, then delta
    const int64_t rows = (int64_t)d.B * d.Sq * d.Hq, acc = rows * plan->D;
    Tensor scratch = at::empty({acc + (plan->uses_doosum ? rows : 0)}, Q.options().dtype(at::kFloat));
    p.dq_accum = (float*)scratch.data_ptr();
    void* st = stream_of(Q);
    if (plan->uses_doosum) {
      p.delta = p.dq_accum + acc;
      p.dq_cleared = 1;
      check(ae_launch_attn_bwd_prep(plan->prep, &p, st), "ae_launch_attn_bwd_prep");
    }
    check(ae_launch_attn_bwd_fused(plan->fused, &p, st), "ae_launch_attn_bwd_fused");
    check(ae_launch_attn_bwd_dq_cast(plan->cast, &p, st), "ae_launch_attn_bwd_dq_cast");
    out[0] = std::move(dq); out[1] = std::move(dk); out[2] = std::move(dv);
    return out;
  }
  void release_variables() override {
    std::lock_guard<std::mutex> lock(mutex_);
    q.reset_data(); k.reset_data(); v.reset_data(); o.reset_data();
    for (auto& f : finals) f.reset_data();
    for (auto& c : custom) c.reset_data();
    lists.clear();
  }
  std::string name() const override { return "AttentionEngineBackward"; }
};

// o = engine(q, k, v, *custom); None when the tensors do not fit or the call needs an autograd function.  `with_finals`:
// (o, [final row scales]) without autograd.
py::object attn(const std::shared_ptr<AttnPlan>& plan, py::handle eng, const Tensor& q, const Tensor& k, const Tensor& v,
                py::handle custom, py::handle lists, bool with_finals) {
  Dims d;
  if (!attn_dims(*plan, q, k, v, d)) return py::none();
  std::vector<Tensor> C = tensors_of(custom), L = tensors_of(lists), F(plan->n_final);
  if (!with_finals) {
    bool function = needs_function({&q, &k, &v});
    for (const Tensor& c : C) function = function || needs_function({&c});
    if (function) return py::none();
  }
  Tensor o, status;
  {
    py::gil_scoped_release nogil;
    c10::cuda::CUDAGuard guard(q.device());
    at::AutoGradMode no_grad(false);
    AeAttnParams p;
    memset(&p, 0, sizeof p);
    std::vector<Tensor> c = C;
    if (!custom_args(plan->custom, c, plan->dtype, d.Sq, d.Skv, false, p.custom, p.custom_stride)) {
      o = Tensor();
    } else {
      o = at::empty({d.B, d.Sq, d.Hq, plan->DV}, q.options());
      for (int i = 0; i < plan->n_final; ++i) {
        F[i] = at::empty({d.B, d.Hq, d.Sq}, q.options().dtype(at::kFloat));
        p.final_rowscales[i] = (float*)F[i].data_ptr();
      }
      p.q = q.data_ptr(); p.k = k.data_ptr(); p.v = v.data_ptr(); p.o = o.data_ptr();
      strides3(q, p.q_stride); strides3(k, p.k_stride); strides3(v, p.v_stride); strides3(o, p.o_stride);
      if (!L.empty()) {
        p.block_count = (const int32_t*)L[0].data_ptr();
        p.block_index = (const int32_t*)L[1].data_ptr();
      }
      p.B = d.B; p.Hq = d.Hq; p.Hkv = d.Hkv; p.Sq = d.Sq; p.Skv = d.Skv;
      status = plan->status_for(q);
      p.status = word(status);
      check(ae_launch_attn_fwd(plan->fwd, &p, stream_of(q)), "ae_launch_attn_fwd");
    }
  }
  if (!o.defined()) return py::none();
  if (with_finals) return py::make_tuple(o, F);
  bool need = wants_grad({&q, &k, &v});
  for (const Tensor& c : C) need = need || wants_grad({&c});
  if (need) {
    auto node = std::shared_ptr<AttnNode>(new AttnNode(), torch::autograd::deleteNode);
    torch::autograd::edge_list edges = torch::autograd::collect_next_edges(q, k, v, C);
    node->set_next_edges(std::move(edges));
    node->plan = plan;
    node->eng = hold(eng);
    node->q = SavedVariable(q, false); node->k = SavedVariable(k, false); node->v = SavedVariable(v, false);
    for (const Tensor& f : F) node->finals.emplace_back(f, false);
    for (const Tensor& c : C) node->custom.emplace_back(c, false);
    node->lists = std::move(L);
    node->d = d;
    node->status = status;
    torch::autograd::set_history(o, node);
    node->o = SavedVariable(o, true);
  }
  return py::cast(o);
}

// ---------------------------------------------------------------------------------------------------- split-KV decode
struct DecodePlan : Plan {
  void *kernel = nullptr, *combine = nullptr;
  void* cut = nullptr;  // intervals and merges in a cluster
  int Hq = 0, Hkv = 0, Sq = 0, D = 0, DV = 0, n_final = 0;
  std::vector<Custom> custom;
};

// `meta`: None, or (work, n_items, seqlens, part_off, n_slots, max_seqlen, B) of a schedule; `table`: None or the block table.
py::object decode(const std::shared_ptr<DecodePlan>& plan, const Tensor& q, const Tensor& k, const Tensor& v, py::handle custom,
                  int n_split, py::handle meta, const std::optional<Tensor>& table, int intervals, bool in_cluster) {
  const DecodePlan& P = *plan;
  if (!good4(q, P.dtype) || !good4(k, P.dtype) || !good4(v, P.dtype)) return py::none();
  const int B = (int)q.size(0), Skv = (int)k.size(1);
  if (q.size(1) != P.Sq || q.size(2) != P.Hq || k.size(2) != P.Hkv || q.size(3) != P.D || k.size(3) != P.D ||
      v.size(3) != P.DV || v.size(0) != k.size(0) || v.size(1) != k.size(1) || v.size(2) != k.size(2))
    return py::none();
  AeDecodeParams p;
  memset(&p, 0, sizeof p);
  int64_t n_slots = n_split > 1 ? (int64_t)B * n_split : 0;
  bool merge = n_split > 1;
  p.Skv = Skv;
  std::vector<Tensor> keep;
  if (!meta.is_none()) {
    auto m = py::reinterpret_borrow<py::tuple>(meta);
    for (int i : {0, 2, 3}) keep.push_back(m[i].cast<Tensor>());
    const int max_seqlen = m[5].cast<int>();
    if (m[6].cast<int>() != B || (!table && max_seqlen > Skv)) return py::none();
    p.work = (const AeDecodeWorkItem*)keep[0].data_ptr();
    p.n_items = m[1].cast<int>();
    p.seqlens = (const int32_t*)keep[1].data_ptr();
    p.part_off = (const int32_t*)keep[2].data_ptr();
    n_slots = m[4].cast<int64_t>();
    merge = n_slots > B || intervals;
    p.Skv = max_seqlen;
    n_split = 1;
  }
  if (table) {
    if (meta.is_none() || Skv != 128 || k.stride(0) != 128 * k.stride(1) || v.stride(0) != 128 * v.stride(1) ||
        !table->is_cuda() || table->scalar_type() != at::kInt || table->dim() != 2 || table->size(0) != B ||
        !table->is_contiguous() || table->size(1) * 128 < p.Skv)
      return py::none();
    p.block_table = (const int32_t*)table->data_ptr();
    p.max_pages = (int)table->size(1);
    p.num_pages = (int)k.size(0);
  } else if (k.size(0) != B) {
    return py::none();
  }
  if (in_cluster && capturing(stream_of(q))) in_cluster = false;  // bit for bit the same, see attn_decode.cuh
  const int64_t units = P.Hq > P.Hkv ? P.Hkv : P.Hq, rows = P.Hq > P.Hkv ? P.Hq / P.Hkv : P.Sq;
  if ((intervals || in_cluster) && !P.cut) return py::none();
  if (intervals) {
    p.n_intervals = (int)std::min<int64_t>(intervals, (int64_t)B * ((p.Skv + 127) / 128));
    if (p.n_intervals < 1) return py::none();
    n_slots = 2 * units * p.n_intervals;
  }
  if (merge && !P.combine) return py::none();
  if (in_cluster) {  // the kernel merges
    merge = false;
    n_slots = 0;
    p.in_cluster = 1;
  }
  std::vector<Tensor> C = tensors_of(custom);
  py::gil_scoped_release nogil;
  c10::cuda::CUDAGuard guard(q.device());
  at::AutoGradMode no_grad(false);
  Tensor o;
  if (custom_args(P.custom, C, P.dtype, P.Sq, p.Skv, true, p.custom, p.custom_stride)) {
    o = at::empty({B, P.Sq, P.Hq, P.DV}, q.options());
    p.q = q.data_ptr(); p.k = k.data_ptr(); p.v = v.data_ptr(); p.o = o.data_ptr();
    strides3(q, p.q_stride); strides3(k, p.k_stride); strides3(v, p.v_stride);
    if (n_slots) {  // the partial outputs, their row scales and the table of the units' rows in one allocation
      const int64_t n = n_slots * (intervals ? rows : P.Sq * P.Hq);
      keep.push_back(at::empty({n * (P.DV + P.n_final) + (intervals ? 2 * B * units : 0)}, q.options().dtype(at::kFloat)));
      p.o_partial = (float*)keep.back().data_ptr();
      for (int i = 0; i < P.n_final; ++i) p.rowscale_partial[i] = p.o_partial + n * P.DV + n * i;
      if (intervals) p.row_info = (int32_t*)(p.o_partial + n * (P.DV + P.n_final));
    }
    p.B = B; p.Hq = P.Hq; p.Hkv = P.Hkv; p.Sq = P.Sq; p.n_split = n_split;
    p.status = word(plan->status_for(q));
    void* st = stream_of(q);
    check(ae_launch_attn_decode(intervals || in_cluster ? P.cut : P.kernel, &p, st), "ae_launch_attn_decode");
    if (merge) check(ae_launch_decode_combine(P.combine, &p, st), "ae_launch_decode_combine");
  }
  py::gil_scoped_acquire gil;
  return o.defined() ? py::cast(o) : py::none();
}

// ---------------------------------------------------------------------------------------------------- MLA decode
struct MlaPlan : Plan {
  void *kernel = nullptr, *combine = nullptr;
  int n_final = 0, pairs = 1;  // CTA pairs the device holds at a time
  // intervals the rows' tiles are cut into: one per pair, two 128-key tiles at least
  int clusters(int64_t tiles) const { return (int)std::max<int64_t>(1, std::min<int64_t>(pairs, (tiles + 1) / 2)); }
};

// Partials, their row scales and the row table of a split call, in one allocation.
struct MlaScratch {
  Tensor buf;
  float *part = nullptr, *scales = nullptr;
  int32_t* rows = nullptr;
  MlaScratch(int64_t slots, int64_t H, int n_final, int64_t B, const Tensor& like) {
    const int64_t n = slots * H;
    buf = at::empty({n * (512 + n_final) + 2 * B}, like.options().dtype(at::kFloat));
    part = (float*)buf.data_ptr();
    scales = part + n * 512;
    rows = (int32_t*)(scales + n * n_final);
  }
};

// The most intervals that a row touches, cut as the kernel cuts them (ae_mla_decode): `keys(b)` of every row.
template <class Keys>
int most_shares(int64_t B, int64_t clusters, Keys&& keys) {
  auto tiles = [&](int64_t b) { return std::max<int64_t>(1, (keys(b) + 127) / 128); };
  int64_t total = 0, longest = 0, before = 0, most = 1;
  for (int64_t b = 0; b < B; ++b) {
    total += tiles(b);
    longest = std::max(longest, tiles(b));
  }
  const int64_t share = std::max((total + clusters - 1) / clusters, (longest + 30) / 31);
  for (int64_t b = 0; b < B; ++b) {
    most = std::max(most, (before % share + tiles(b) - 1) / share + 1);
    before += tiles(b);
  }
  return (int)most;
}

bool same(const Tensor& t, std::initializer_list<int64_t> shape) { return t.sizes() == at::IntArrayRef(shape.begin(), shape.size()); }

py::object mla(const std::shared_ptr<MlaPlan>& plan, const Tensor& q, const Tensor& q_pe, const Tensor& kv, const Tensor& k_pe,
               int n_split) {
  const MlaPlan& P = *plan;
  for (const Tensor* t : {&q, &q_pe, &kv, &k_pe})
    if (!t->is_cuda() || t->scalar_type() != P.dtype) return py::none();
  if (q.dim() != 4 || kv.dim() != 4) return py::none();
  const int64_t B = q.size(0), H = q.size(2), S = kv.size(1);
  if (!same(q, {B, 1, H, 512}) || !same(q_pe, {B, 1, H, 64}) || !same(kv, {B, S, 1, 512}) || !same(k_pe, {B, S, 1, 64}))
    return py::none();
  if (B == 0 || H == 0 || S == 0) return py::none();  // the cut into intervals below divides by the tiles of a row
  py::gil_scoped_release nogil;
  c10::cuda::CUDAGuard guard(q.device());
  at::AutoGradMode no_grad(false);
  const Tensor Q = q.contiguous(), QP = q_pe.contiguous(), KV = kv.contiguous(), KP = k_pe.contiguous();
  Tensor o = at::empty({B, 1, H, 512}, q.options());
  AeMlaParams p;
  memset(&p, 0, sizeof p);
  p.q = Q.data_ptr(); p.q_pe = QP.data_ptr(); p.kv = KV.data_ptr(); p.k_pe = KP.data_ptr(); p.o = o.data_ptr();
  p.B = (int)B; p.H = (int)H; p.S = (int)S; p.n_split = n_split;
  std::optional<MlaScratch> scratch;
  bool merge = n_split > 1;
  if (n_split != 1) {
    const int64_t n_t = (S + 127) / 128;
    p.n_clusters = P.clusters(B * n_t);
    scratch.emplace(n_split ? B * n_split : 2 * (int64_t)p.n_clusters, H, P.n_final, B, q);
    p.o_partial = scratch->part;
    for (int i = 0; i < P.n_final; ++i) p.rowscale_partial[i] = scratch->scales + (scratch->scales - scratch->part) / 512 * i;
    p.row_info = scratch->rows;
    if (n_split == 0) {
      const int64_t share = (B * n_t + p.n_clusters - 1) / p.n_clusters;
      merge = share % n_t != 0;  // intervals of whole rows leave nothing to merge
    }
  }
  p.status = word(plan->status_for(q));
  void* st = stream_of(q);
  check(ae_launch_mla_decode(P.kernel, &p, st), "ae_launch_mla_decode");
  if (merge) check(ae_launch_mla_combine(P.combine, &p, st), "ae_launch_mla_combine");
  const int shares = n_split ? n_split : most_shares(B, p.n_clusters, [&](int64_t) { return S; });
  py::gil_scoped_acquire gil;
  return py::make_tuple(o, shares);
}

// Pinned landing place of the row lengths, one per thread: the number of the call, then the lengths.
struct Lengths {
  int32_t* host = nullptr;
  int64_t room = 0;
  int device = -1;
  int32_t call = 0;
  void release() {
    if (host) cudaFreeHost(host);
    host = nullptr;
    room = 0;
    device = -1;
  }
  void make(int dev, int64_t n) {  // nothing is left behind that a failed allocation would make look usable
    if (device != dev || room < n) {
      release();
      C10_CUDA_CHECK(cudaHostAlloc((void**)&host, (size_t)(n + 1) * 4, cudaHostAllocPortable | cudaHostAllocMapped));
      host[0] = call;
      room = n;
      device = dev;
    }
    ++call;
  }
  ~Lengths() { release(); }
};

// What the decode kernel writes into the landing place: waited for on every way out, so that the thread's next call finds no
// older kernel that may still write.  A call that fails before its kernel is launched returns behind the stream's work.
struct Landing {
  Lengths& land;
  cudaStream_t st;
  bool launched = false, waiting = true;
  Landing(Lengths& l, cudaStream_t s) : land(l), st(s) {}
  cudaError_t wait() {
    waiting = false;
    auto arrived = [&] { return __atomic_load_n(land.host, __ATOMIC_ACQUIRE) == land.call; };
    for (int64_t i = 1; !arrived(); ++i) {
      if (i % 4096) continue;
      const cudaError_t e = cudaStreamQuery(st);  // a kernel that failed never writes
      if (e == cudaErrorNotReady) continue;
      return e != cudaSuccess ? e : arrived() ? cudaSuccess : cudaErrorUnknown;
    }
    return cudaSuccess;
  }
  ~Landing() {
    if (waiting) (void)(launched ? wait() : cudaStreamSynchronize(st));
  }
};

// (o, lse, most shares of a row) over a paged cache; n_split 0: equal intervals of all rows' tiles.  The row lengths are checked on
// the host behind the launches: the decode kernel writes them to pinned memory as it starts and clamps every length to the
// block table itself, so neither the kernels nor the stream wait for the check (a copy in front of them: 39.5 -> 33 us of a call of 8
// rows).  Returns None when the tensors do not fit, or an empty tuple for
// lengths outside their range.
py::object mla_paged(const std::shared_ptr<MlaPlan>& plan, const Tensor& q, const Tensor& pool, const Tensor& table_in,
                     const Tensor& lens_in, int n_split) {
  const MlaPlan& P = *plan;
  if (!q.is_cuda() || q.scalar_type() != P.dtype || q.dim() != 4 || q.size(1) != 1 || q.size(3) != 576 || q.size(2) > 128)
    return py::none();
  if (!pool.is_cuda() || pool.scalar_type() != P.dtype || !pool.is_contiguous()) return py::none();
  const bool d4 = pool.dim() == 4;
  if ((!d4 && pool.dim() != 3) || pool.size(1) != 64 || pool.size(-1) != 576 || (d4 && pool.size(2) != 1)) return py::none();
  const int64_t B = q.size(0), H = q.size(2);
  if (B == 0 || H == 0) return py::none();
  if (table_in.dim() < 2 || table_in.size(0) != B || table_in.numel() != B * table_in.size(1) || lens_in.dim() != 1 ||
      lens_in.size(0) != B)
    return py::none();
  py::gil_scoped_release nogil;
  c10::cuda::CUDAGuard guard(q.device());
  at::AutoGradMode no_grad(false);
  const auto ints = q.options().dtype(at::kInt);
  const Tensor table = table_in.to(ints).contiguous(), lens = lens_in.to(ints).contiguous();
  const int64_t max_pages = table.size(1);
  if (max_pages == 0) {
    py::gil_scoped_acquire gil;
    return py::tuple();
  }
  TORCH_CHECK(c10::cuda::currentStreamCaptureStatusMayInitCtx() == c10::cuda::CaptureStatus::None,
              "paged MLA decode reads the row lengths on the host: it cannot be captured into a CUDA graph");
  static thread_local Lengths land;
  cudaStream_t st = (cudaStream_t)stream_of(q);
  land.make(q.device().index(), B);
  Landing landing(land, st);
  Tensor Q = q.contiguous();
  if (reinterpret_cast<uintptr_t>(Q.data_ptr()) % 16) Q = Q.clone();  // TMA reads from 16-byte boundaries
  Tensor o = at::empty({B, 1, H, 512}, q.options());
  const auto f32 = q.options().dtype(at::kFloat);
  Tensor lse = at::empty({B, H}, f32);
  AeMlaPagedParams p;
  memset(&p, 0, sizeof p);
  p.q = Q.data_ptr();
  p.q_pe = (const char*)Q.data_ptr() + 512 * 2;
  p.q_row_stride = 576;
  p.kcache = pool.data_ptr(); p.o = o.data_ptr();
  p.block_table = (const int32_t*)table.data_ptr();
  p.cache_seqlens = (const int32_t*)lens.data_ptr();
  p.lse_out = (float*)lse.data_ptr();
  p.B = (int)B; p.H = (int)H; p.num_pages = (int)pool.size(0); p.max_pages = (int)max_pages;
  p.max_seqlen = (int)(max_pages * 64); p.n_split = n_split;
  std::optional<MlaScratch> scratch;
  if (n_split != 1) {
    p.n_clusters = P.clusters(B * ((max_pages + 1) / 2));
    scratch.emplace(n_split ? B * n_split : 2 * (int64_t)p.n_clusters, H, 1, B, q);
    p.o_partial = scratch->part;
    p.rowscale_partial[0] = scratch->scales;
    p.row_info = scratch->rows;
  }
  p.status = word(plan->status_for(q));
  p.lens_host = land.host;
  p.lens_call = land.call;
  check(ae_launch_mla_decode_paged(P.kernel, &p, st), "ae_launch_mla_decode_paged");
  landing.launched = true;
  if (n_split != 1) {
    AeMlaParams m;
    memset(&m, 0, sizeof m);
    m.o = p.o; m.o_partial = p.o_partial; m.rowscale_partial[0] = p.rowscale_partial[0];
    m.B = p.B; m.H = p.H; m.S = p.max_seqlen; m.n_split = n_split; m.row_info = p.row_info;
    m.lse_out = p.lse_out;
    check(ae_launch_mla_combine(P.combine, &m, st), "ae_launch_mla_combine");
  }
  C10_CUDA_CHECK(landing.wait());
  bool in_range = true;
  const int32_t* const len = land.host + 1;
  for (int64_t b = 0; b < B; ++b) in_range = in_range && len[b] >= 1 && len[b] <= max_pages * 64;
  const int shares = n_split || !in_range ? n_split : most_shares(B, p.n_clusters, [&](int64_t b) { return (int64_t)len[b]; });
  py::gil_scoped_acquire gil;
  if (!in_range) return py::tuple();
  return py::make_tuple(o, lse, shares);
}

// ---------------------------------------------------------------------------------------------------- scan
struct ScanPlan : Plan {
  void *fwd_mods = nullptr;  // the forward built with the Mamba2 block's mods inside (64 value dims)
  void *bwd = nullptr, *bwd_mods = nullptr, *head_sum = nullptr;  // set when first needed
  // what a sequence cut into segments takes, set when first needed: the contributions by value dims, and the scan kernel's
  // builds that start from them
  void *seg64 = nullptr, *seg128 = nullptr;
  void *fwd_cut64 = nullptr, *fwd_cut128 = nullptr, *fwd_mods_cut = nullptr;
  int segments = 0;  // segments a sequence is cut into; 0: as many as seg_chunks() finds
};

// Chunks per segment of a scan of `walks` (batch, head) walks over n chunks.  A walk is a chain, and a launch lasts as long as
// the walks on the fullest SM; segments shorten the chain and fill idle SMs, at the price of a launch that computes what
// every segment but one adds to the state (two CTAs per SM) and of summing those in front of a segment.  Microseconds as
// measured on a B200 over 1 to 16 segments: a CTA of the scan 5 + 2.95 per chunk + 0.25 per segment, one of the
// contributions (64 value dims) 3 + 1.3 per chunk, 3 for the second launch.  One walk against the cut, microseconds a call among
// others: 8 walks of 64 chunks 154 -> 30 (16 segments), 48 of 56 140 -> 90 (6), 32 of 64 with 128 value dims 224 -> 93 (4), 320 of 24
// (more walks than SMs) 227 uncut, 231 in two.
// Only without gradients: a segment's start is a sum of fp32 states in another order than the walk's, and a training step's results
// do not depend on how many heads and rows run beside, bit for bit.
int best_seg_chunks(int64_t walks, int64_t n, int64_t dv, int sms) {
  auto rounds = [](int64_t ctas, int64_t room) { return (double)((ctas + room - 1) / room); };
  const double chunk_us = 2.95;
  int64_t best = n;
  double least = rounds(walks, sms) * (n * chunk_us + 5);
  for (int64_t p = 2; p <= std::min<int64_t>(n, 16); ++p) {
    const int64_t len = (n + p - 1) / p, cut = (n + len - 1) / len;
    const double t = rounds(walks * cut, sms) * (len * chunk_us + 5 + 0.25 * cut) + rounds(walks * (dv / 64) * (cut - 1), 2 * sms) * (len * 1.3 + 3) + 3;
    if (t < least) least = t, best = len;
  }
  return (int)best;
}

int seg_chunks(const ScanPlan& plan, int64_t walks, int64_t n, int64_t dv, int device) {
  if (plan.segments) return (int)((n + plan.segments - 1) / plan.segments);
  int sms = 0;
  C10_CUDA_CHECK(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device));
  return best_seg_chunks(walks, n, dv, sms);
}

// Scratch of a cut and the launch that fills it; nothing with one segment.  `scan` is the plan's kernel for the other case.
struct Segments {
  Tensor buf;
  int chunks = 0, count = 1;
  float *state = nullptr, *decay = nullptr;
  void* scan = nullptr;
  Segments(const ScanPlan& plan, py::handle eng, const Tensor& k, const Tensor& v, const Tensor& a, const Tensor& asc, const Tensor& vscale, uint32_t* status) {
    const int64_t B = v.size(0), H = v.size(1), T = v.size(2), DV = v.size(3), n = (T + 127) / 128;
    if (n < 2) return;
    chunks = seg_chunks(plan, B * H, n, DV, v.device().index());
    count = (int)((n + chunks - 1) / chunks);
    if (count == 1) return;
    void* const& kernel = DV == 64 ? plan.seg64 : plan.seg128;
    void* const& cut = vscale.defined() ? plan.fwd_mods_cut : DV == 64 ? plan.fwd_cut64 : plan.fwd_cut128;
    if (!cut) with_python([&] { eng.attr("_load_segment_kernels")((int)DV, vscale.defined()); });
    scan = cut;
    const int64_t slots = B * H * (count - 1);
    buf = at::empty({slots * (128 * DV + 1)}, a.options());
    state = (float*)buf.data_ptr();
    decay = state + slots * 128 * DV;
    AeLinearSegParams p;
    memset(&p, 0, sizeof p);
    p.k = k.data_ptr(); p.v = v.data_ptr(); p.a = (const float*)a.data_ptr();
    p.ascale = asc.defined() ? (const float*)asc.data_ptr() : nullptr;
    p.vscale = vscale.defined() ? vscale.data_ptr() : nullptr;
    p.vscale_16bit = vscale.defined() && vscale.scalar_type() != at::kFloat;
    p.B = (int)B; p.H = (int)H; p.HK = (int)k.size(1); p.T = (int)T;
    p.seg_chunks = chunks; p.seg_state = state; p.seg_decay = decay;
    p.status = status;
    check(ae_launch_linear_segments(kernel, &p, stream_of(v)), "ae_launch_linear_segments");
  }
};

// the tensors of one scan; s / d / asc undefined without the block's mods
struct ScanSaved {
  SavedVariable q, k, v, a, x, s, d, asc, hs;
  std::vector<SavedVariable*> all() { return {&q, &k, &v, &a, &x, &s, &d, &asc, &hs}; }
};

Tensor sum_over_batch(const Tensor& t, const std::vector<int64_t>& shape, at::ScalarType dtype) {
  // [B, H] -> the operand's shape; one batch row needs no sum
  return (t.size(0) == 1 ? t : t.sum(0)).reshape(shape).to(dtype);
}

struct ScanNode : Node {
  std::shared_ptr<ScanPlan> plan;
  std::shared_ptr<PyObject> eng;
  ScanSaved saved;
  bool mods = false, has_asc = false;
  Tensor status;
  std::vector<int64_t> d_shape, asc_shape;
  at::ScalarType d_dtype = at::kFloat, asc_dtype = at::kFloat;

  variable_list apply(variable_list&& grads) override {
    variable_list out(mods ? 7 : 4);
    if (!grads[0].defined()) grads[0] = input_metadata(0).zeros_like();  // as torch.autograd.Function does
    Tensor q, k, v, a, x, s, d, asc, hs;
    {
      std::lock_guard<std::mutex> lock(mutex_);
      q = saved.q.unpack(), k = saved.k.unpack(), v = saved.v.unpack(), a = saved.a.unpack();
      if (mods) x = saved.x.unpack(), s = saved.s.unpack(), d = saved.d.unpack();
      if (has_asc) asc = saved.asc.unpack();
      hs = saved.hs.unpack();
    }
    at::AutoGradMode no_grad(false);
    c10::cuda::CUDAGuard guard(q.device());
    const Tensor g = grads[0].contiguous();
    const int B = (int)q.size(0), HQ = (int)q.size(1), T = (int)q.size(2), HK = (int)k.size(1), H = (int)v.size(1);
    const int how = with_python([&] {  // 0: through the Python path, 1: one launch from here
      return py::handle(eng.get()).attr("_native_bwd")(B, H, HQ != H || HK != H, mods, (int)q.device().index()).cast<int>();
    });
    if (how == 0) {
      return with_python([&] {
        py::handle e(eng.get());
        auto opt = [](const Tensor& t) -> py::object { return t.defined() ? py::cast(t) : py::none(); };
        py::tuple r = e.attr("_bwd_from_saved")(q, k, v, a, g, hs, opt(x), opt(s), opt(d), opt(asc));
        for (size_t i = 0; i < out.size(); ++i)
          if (!r[i].is_none()) out[i] = r[i].cast<Tensor>();
        if (mods) {
          out[5] = sum_over_batch(out[5], d_shape, d_dtype);
          if (out[6].defined()) out[6] = sum_over_batch(out[6], asc_shape, asc_dtype);
        }
        return out;
      });
    }
    const auto o16 = q.options(), f32 = q.options().dtype(at::kFloat);
    AeLinearBwdParams p;
    memset(&p, 0, sizeof p);
    void* st = stream_of(q);
    Tensor dq_h = at::empty({B, H, T, 128}, o16), dk_h = at::empty({B, H, T, 128}, o16), dv = at::empty({B, H, T, 64}, o16);
    Tensor da = at::empty({B, H, T}, f32), gs, gd, gasc;
    p.q = q.data_ptr(); p.k = k.data_ptr(); p.v = v.data_ptr(); p.a = (const float*)a.data_ptr(); p.d_o = g.data_ptr();
    p.h_states = hs.data_ptr(); p.dq = dq_h.data_ptr(); p.dk = dk_h.data_ptr(); p.dv = dv.data_ptr();
    p.da = (float*)da.data_ptr();
    p.B = B; p.H = H; p.HQ = HQ; p.HK = HK; p.T = T;
    p.status = word(status);
    if (mods) {
      gs = at::empty_like(s);
      gd = at::empty({B, H}, f32);
      p.x = x.data_ptr(); p.vscale = s.data_ptr(); p.dskip = (const float*)d.data_ptr();
      p.gs = gs.data_ptr(); p.gd = (float*)gd.data_ptr();
      p.vscale_16bit = s.scalar_type() != at::kFloat;
    }
    if (asc.defined()) {
      gasc = at::empty({B, H}, f32);
      p.ascale = (const float*)asc.data_ptr();
      p.gasc = (float*)gasc.data_ptr();
    }
    check(ae_launch_linear_bwd(mods ? plan->bwd_mods : plan->bwd, &p, st), "ae_launch_linear_bwd");
    auto head_sum = [&](const Tensor& in, int heads) {
      if (heads == H) return in;
      Tensor y = at::empty({B, heads, T, 128}, o16);
      AeRowScaleParams r;
      memset(&r, 0, sizeof r);
      r.x = in.data_ptr(); r.y = y.data_ptr();
      r.n_rows = (int64_t)B * heads * T; r.rows_per_head = T; r.n_heads = H / heads;
      check(ae_launch_rowscale(plan->head_sum, &r, st), "ae_launch_rowscale");
      return y;
    };
    out[0] = head_sum(dq_h, HQ);
    out[1] = head_sum(dk_h, HK);
    out[2] = std::move(dv);
    out[3] = std::move(da);
    if (mods) {
      out[4] = std::move(gs);
      out[5] = sum_over_batch(gd, d_shape, d_dtype);
      if (gasc.defined()) out[6] = sum_over_batch(gasc, asc_shape, asc_dtype);
    }
    return out;
  }
  void release_variables() override {
    std::lock_guard<std::mutex> lock(mutex_);
    for (SavedVariable* s : saved.all()) s->reset_data();
  }
  std::string name() const override { return mods ? "ScaleScanSkipBackward" : "LinearScanBackward"; }
};

// The scan kernel on contiguous tensors, in segments where that is faster (with `eng`, whose builds it then takes); those after `a` may be undefined: the row scale, skip weight and decay
// scale of the Mamba2 block (a kernel built with the mods inside), and what receives the scaled v and the chunk start-states.
Tensor scan_launch(ScanPlan& plan, void* kernel, const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& a, const Tensor& s,
                   const Tensor& d, const Tensor& asc, const Tensor& v_out, const Tensor& hs, py::handle eng = {}) {
  AeLinearParams p;
  memset(&p, 0, sizeof p);
  Tensor y = at::empty({q.size(0), v.size(1), q.size(2), v.size(3)}, q.options());
  auto ptr = [](const Tensor& t) { return t.defined() ? t.data_ptr() : nullptr; };
  p.q = q.data_ptr(); p.k = k.data_ptr(); p.v = v.data_ptr(); p.a = (const float*)a.data_ptr(); p.o = y.data_ptr();
  p.vscale = ptr(s);
  p.vscale_16bit = s.defined() && s.scalar_type() != at::kFloat;
  p.dskip = (const float*)ptr(d);
  p.ascale = (const float*)ptr(asc);
  p.v_out = ptr(v_out);
  p.h_states_out = ptr(hs);
  p.B = (int)q.size(0); p.H = (int)v.size(1); p.HQ = (int)q.size(1); p.HK = (int)k.size(1); p.T = (int)q.size(2);
  p.status = word(plan.status_for(q));
  std::optional<Segments> seg;
  if (eng) {
    seg.emplace(plan, eng, k, v, a, asc, s, p.status);
    p.seg_chunks = seg->chunks; p.seg_state = seg->state; p.seg_decay = seg->decay;
    if (seg->scan) kernel = seg->scan;
  }
  check(ae_launch_linear_fwd(kernel, &p, stream_of(q)), "ae_launch_linear_fwd");
  return y;
}

// y = scan(q, k, v, a), or with s, d (and asc): y = scan(q, k, v * s[..., None], a * asc[head]) + v * d[head] as one node.
// q / k have 128 dims; v has 64 dims with mods, 64 or 128 (no gradient) without.
Tensor scan_run(const std::shared_ptr<ScanPlan>& plan, void* kernel, py::handle eng, const Tensor& q_, const Tensor& k_,
                const Tensor& v_, const Tensor& a_, const Tensor& s_, const Tensor& d_, const Tensor& asc_) {
  const bool mods = s_.defined();
  const bool need = wants_grad({&q_, &k_, &v_, &a_, &s_, &d_, &asc_});
  Tensor q, k, v, a, s, d, asc, y, hs, v_out, status;
  {
    py::gil_scoped_release nogil;
    c10::cuda::CUDAGuard guard(q_.device());
    at::AutoGradMode no_grad(false);
    q = q_.contiguous(); k = k_.contiguous(); v = v_.contiguous();
    a = a_.to(at::kFloat).contiguous();
    const int64_t B = q.size(0), T = q.size(2), H = v.size(1), DV = v.size(3);
    if (mods) {
      s = s_.contiguous();
      d = d_.to(at::kFloat).reshape({-1}).contiguous();
      if (asc_.defined()) asc = asc_.to(at::kFloat).reshape({-1}).contiguous();
      if (need) v_out = at::empty_like(v);
    }
    if (need) {  // the reverse pass reads the chunk start-states the forward has at hand
      TORCH_CHECK(DV == 64, "the scan has gradients in value blocks of 64 dims");
      hs = at::empty({B, H, (T + 127) / 128, 128, DV}, q.options());
    }
    y = scan_launch(*plan, kernel, q, k, v, a, s, d, asc, v_out, hs, need ? py::handle() : eng);
    status = plan->status_for(q);
  }
  if (need) {
    auto node = std::shared_ptr<ScanNode>(new ScanNode(), torch::autograd::deleteNode);
    if (mods)
      node->set_next_edges(torch::autograd::collect_next_edges(q_, k_, v_, a_, s_, d_, asc_));
    else
      node->set_next_edges(torch::autograd::collect_next_edges(q_, k_, v_, a_));
    node->plan = plan;
    node->eng = hold(eng);
    node->mods = mods;
    node->status = status;
    auto& sv = node->saved;
    sv.q = SavedVariable(q, false);
    sv.k = SavedVariable(k, false);
    sv.v = SavedVariable(mods ? v_out : v, false);
    sv.a = SavedVariable(a, false);
    if (mods) {
      sv.x = SavedVariable(v, false);
      sv.s = SavedVariable(s, false);
      sv.d = SavedVariable(d, false);
      node->d_shape = d_.sizes().vec();
      node->d_dtype = d_.scalar_type();
      if (asc.defined()) {
        sv.asc = SavedVariable(asc, false);
        node->has_asc = true;
        node->asc_shape = asc_.sizes().vec();
        node->asc_dtype = asc_.scalar_type();
      }
    }
    sv.hs = SavedVariable(hs, false);
    torch::autograd::set_history(y, node);
  }
  return y;
}

// One launch of the scan kernel, for the front end's autograd function and for direct use: bit-equal states to ae_linear_states.
Tensor scan_forward(const std::shared_ptr<ScanPlan>& plan, uint64_t kernel, const Tensor& q, const Tensor& k, const Tensor& v,
                    const Tensor& a, const std::optional<Tensor>& s, const std::optional<Tensor>& d, const std::optional<Tensor>& asc,
                    const std::optional<Tensor>& v_out, const std::optional<Tensor>& hs) {
  py::gil_scoped_release nogil;
  c10::cuda::CUDAGuard guard(q.device());
  at::AutoGradMode no_grad(false);
  auto opt = [](const std::optional<Tensor>& t) { return t ? *t : Tensor(); };
  return scan_launch(*plan, handle(kernel), q.contiguous(), k.contiguous(), v.contiguous(), a.to(at::kFloat).contiguous(), opt(s),
                     opt(d), opt(asc), opt(v_out), opt(hs));
}

// None when the call needs an autograd function.
py::object scan(const std::shared_ptr<ScanPlan>& plan, uint64_t kernel, py::handle eng, const Tensor& q, const Tensor& k,
                const Tensor& v, const Tensor& a) {
  if (needs_function({&q, &k, &v, &a})) return py::none();
  return py::cast(scan_run(plan, handle(kernel), eng, q, k, v, a, Tensor(), Tensor(), Tensor()));
}

// The Mamba2 block: x * s[b, h, t] into the scan, + x * d[head] after it, decay * asc[head] (None: decay as passed).  None
// when the operands are not of that form at run time or the call needs an autograd function (the caller then takes the mods
// one by one).
py::object scan_block(const std::shared_ptr<ScanPlan>& plan, py::handle eng, const Tensor& q, const Tensor& k, const Tensor& x,
                      const Tensor& decay, const Tensor& s, const Tensor& d, const std::optional<Tensor>& asc) {
  for (const Tensor* t : {&q, &k, &x})
    if (!t->is_cuda() || t->scalar_type() != plan->dtype || t->dim() != 4) return py::none();
  if (!decay.is_cuda() || decay.scalar_type() != at::kFloat || !s.is_cuda() || !d.is_cuda()) return py::none();
  const int64_t B = x.size(0), H = x.size(1), T = x.size(2);
  if (q.size(3) != 128 || k.size(3) != 128 || x.size(3) != 64 || H % q.size(1) || H % k.size(1)) return py::none();
  if (s.sizes() != x.sizes().slice(0, 3) || (s.scalar_type() != at::kFloat && s.scalar_type() != plan->dtype)) return py::none();
  if (d.numel() != H || d.scalar_type() != at::kFloat) return py::none();
  if (decay.dim() != 3 || !same(decay, {B, H, T}) || q.size(0) != B || k.size(0) != B || q.size(2) != T || k.size(2) != T)
    return py::none();
  if (needs_function({&q, &k, &x, &decay, &s, &d}) || (asc && needs_function({&*asc}))) return py::none();
  if (asc && (!asc->is_cuda() || asc->numel() != H || asc->scalar_type() != at::kFloat)) return py::none();
  if (!plan->fwd_mods) eng.attr("_load_block_kernel")();
  return py::cast(scan_run(plan, plan->fwd_mods, eng, q, k, x, decay, s, d, asc ? *asc : Tensor()));
}

}  // namespace

#define AE_HANDLE(cls, name)                                                  \
  .def_property(#name, [](const cls& p) { return (uint64_t)(uintptr_t)p.name; }, \
                [](cls& p, uint64_t h) { p.name = handle(h); })
#define AE_STATUS(cls)                                                                                     \
  .def_property("status", [](cls& p) -> py::object {                                                        \
                  Tensor t = p.status_now();                                                                 \
                  return t.defined() ? py::cast(t) : py::none();                                             \
                },                                                                                           \
                [](cls& p, std::optional<Tensor> t) { p.set_status(t ? *t : Tensor()); })

PYBIND11_MODULE(_ae_host, m) {
  m.attr("built_for") = AE_HOST_BUILT_FOR;  // the build step looks for this text in the file
  py::class_<AttnPlan, std::shared_ptr<AttnPlan>>(m, "AttnPlan")
      .def(py::init([](uint64_t fwd, bool bf16, int D, int DV, int n_final, bool uses_doosum, py::list custom) {
        auto p = std::make_shared<AttnPlan>();
        p->fwd = handle(fwd);
        p->dtype = bf16 ? at::kBFloat16 : at::kHalf;
        p->D = D; p->DV = DV; p->n_final = n_final; p->uses_doosum = uses_doosum;
        p->custom = customs_from(custom);
        return p;
      })) AE_HANDLE(AttnPlan, prep) AE_HANDLE(AttnPlan, fused) AE_HANDLE(AttnPlan, cast) AE_STATUS(AttnPlan);
  py::class_<DecodePlan, std::shared_ptr<DecodePlan>>(m, "DecodePlan")
      .def(py::init([](uint64_t kernel, uint64_t combine, bool bf16, int Hq, int Hkv, int Sq, int D, int DV, int n_final,
                       py::list custom, uint64_t cut) {
        auto p = std::make_shared<DecodePlan>();
        p->kernel = handle(kernel); p->combine = handle(combine); p->cut = handle(cut);
        p->dtype = bf16 ? at::kBFloat16 : at::kHalf;
        p->Hq = Hq; p->Hkv = Hkv; p->Sq = Sq; p->D = D; p->DV = DV; p->n_final = n_final;
        p->custom = customs_from(custom);
        return p;
      })) AE_STATUS(DecodePlan);
  py::class_<MlaPlan, std::shared_ptr<MlaPlan>>(m, "MlaPlan")
      .def(py::init([](uint64_t kernel, uint64_t combine, bool bf16, int n_final, int pairs) {
        auto p = std::make_shared<MlaPlan>();
        p->kernel = handle(kernel); p->combine = handle(combine);
        p->dtype = bf16 ? at::kBFloat16 : at::kHalf;
        p->n_final = n_final;
        p->pairs = pairs;
        return p;
      })) AE_STATUS(MlaPlan);
  py::class_<ScanPlan, std::shared_ptr<ScanPlan>>(m, "ScanPlan")
      .def(py::init([](bool bf16) {
        auto p = std::make_shared<ScanPlan>();
        p->dtype = bf16 ? at::kBFloat16 : at::kHalf;
        return p;
      })) AE_HANDLE(ScanPlan, fwd_mods) AE_HANDLE(ScanPlan, bwd) AE_HANDLE(ScanPlan, bwd_mods)
          AE_HANDLE(ScanPlan, head_sum) AE_HANDLE(ScanPlan, seg64) AE_HANDLE(ScanPlan, seg128)
          AE_HANDLE(ScanPlan, fwd_cut64) AE_HANDLE(ScanPlan, fwd_cut128) AE_HANDLE(ScanPlan, fwd_mods_cut)
      .def_readwrite("segments", &ScanPlan::segments) AE_STATUS(ScanPlan);
  m.def("attn", torch::wrap_pybind_function(&attn));
  m.def("decode", torch::wrap_pybind_function(&decode));
  m.def("mla", torch::wrap_pybind_function(&mla));
  m.def("mla_paged", torch::wrap_pybind_function(&mla_paged));
  m.def("scan_forward", torch::wrap_pybind_function(&scan_forward));
  m.def("scan", torch::wrap_pybind_function(&scan));
  m.def("scan_block", torch::wrap_pybind_function(&scan_block));
  m.def("best_seg_chunks", &best_seg_chunks);
}

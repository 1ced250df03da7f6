// The host path of the training and serving calls in C++: operand preparation, allocations, the argument blocks of the C
// library (include/selective_attention_b200.h) and the autograd nodes.  The kernels of a small call take less time than the
// same steps did in Python: forward + backward of 8 heads x 200 tokens was 172 us on the host around 37 us on the GPU.
//
// A failed library call raises the package's LibraryError, from a backward too.
#include <ATen/cuda/CUDAContext.h>
#include <ATen/cuda/CUDAGraphsUtils.cuh>
#include <c10/cuda/CUDAGuard.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/functions/basic_ops.h>
#include <torch/extension.h>

#include <algorithm>

#include "../../../include/selective_attention_b200.h"

namespace {

using at::Tensor;
using torch::autograd::AutogradContext;
using torch::autograd::variable_list;

int code_of(at::ScalarType t) {
  switch (t) {
    case at::kFloat: return SA_F32;
    case at::kBFloat16: return SA_BF16;
    case at::kHalf: return SA_F16;
    default: return -1;
  }
}
int code_of(const Tensor& t) { return code_of(t.scalar_type()); }
void* stream_of(const Tensor& t) { return at::cuda::getCurrentCUDAStream(t.get_device()).stream(); }

// Raises LibraryError for a non-zero status.  `in_engine`: in a backward, on a thread of the autograd engine, which carries
// torch's own exception type to the caller.
void check(const char* fn, int status, bool in_engine = false) {
  if (status == SA_OK) return;
  pybind11::gil_scoped_acquire gil;
  try {
    pybind11::module_::import("selective_attention_b200._lib").attr("check")(fn, status);
  } catch (pybind11::error_already_set& e) {
    if (!in_engine) throw;
    e.restore();
    python_error err;
    err.persist();
    throw err;
  }
}

sa_tensor rows_of(const Tensor& t) {              // (B, H, T, D) with a contiguous last axis
  sa_tensor d{};
  d.ptr = t.data_ptr();
  d.dtype = code_of(t);
  for (int i = 0; i < 3; ++i) d.stride[i] = t.stride(i);
  return d;
}

sa_problem problem_of(const Tensor& q, const Tensor& k, const Tensor& v, int engine, int64_t exempt) {
  sa_problem p{};
  p.struct_bytes = sizeof(sa_problem);
  p.dtype = code_of(q);
  p.engine = engine;
  p.batch = (int32_t)q.size(0); p.heads = (int32_t)q.size(1); p.seq = (int32_t)q.size(2); p.head_dim = (int32_t)q.size(3);
  p.exempt = (int32_t)exempt;
  for (int i = 0; i < 3; ++i) {
    p.q_stride[i] = q.stride(i);
    p.k_stride[i] = k.stride(i);
    p.v_stride[i] = v.stride(i);
  }
  return p;
}

// The kernels take any batch / head / token strides with a contiguous last axis; the TMA path also needs 16-byte rows.
Tensor strided(const Tensor& t, bool tc) {
  bool ok = t.stride(3) == 1 || t.size(3) == 1;
  if (ok && tc) {
    const int64_t es = t.element_size();
    ok = reinterpret_cast<uintptr_t>(t.data_ptr()) % 16 == 0;
    for (int i = 0; i < 3; ++i) ok = ok && (t.stride(i) * es) % 16 == 0;
  }
  return ok ? t : t.contiguous();
}

// What the backward needs of a forward besides its operands and output, in one allocation.
struct Scratch {
  size_t lse2 = 0, carry = 0, total = 0, table = 0, table_bytes = 0, bytes = 0;
  Scratch(const sa_problem& p, bool skip) {
    auto take = [&](size_t n) {
      const size_t at = bytes;
      bytes += (n + 255) / 256 * 256;
      return at;
    };
    const size_t b = p.batch, t = p.seq;
    lse2 = take(b * p.heads * t * 4);
    carry = take(b * sa_carry_checkpoints(p.engine, p.seq) * t * 4);
    total = take(b * t * 4);
    table_bytes = skip ? sa_tile_table_bytes(&p) : 0;
    table = take(table_bytes);
  }
};

Tensor bytes_on(const Tensor& like, size_t n) {
  return at::empty({(int64_t)std::max<size_t>(n, 1)}, like.options().dtype(at::kByte));
}

// A saved scratch as it comes back: a hook on saved tensors may have put its bytes anywhere, the kernels read floats.
Tensor unpacked(const Tensor& t) {
  const Tensor c = t.contiguous();
  return reinterpret_cast<uintptr_t>(c.data_ptr()) % 256 == 0 ? c : c.clone();
}

Tensor run_forward(const sa_problem& p, const Tensor& q, const Tensor& k, const Tensor& v, const Scratch& at_, const Tensor& scratch,
                   const sa_tensor* low) {
  Tensor out = at::empty({p.batch, p.heads, p.seq, p.head_dim}, q.options().dtype(at::kFloat));
  char* s = static_cast<char*>(scratch.data_ptr());
  check("sa_forward", sa_forward_live_tiles(&p, q.data_ptr(), k.data_ptr(), v.data_ptr(), nullptr, out.data_ptr<float>(), low,
                                            reinterpret_cast<float*>(s + at_.lse2), reinterpret_cast<float*>(s + at_.carry),
                                            reinterpret_cast<float*>(s + at_.total), at_.table_bytes ? s + at_.table : nullptr,
                                            at_.table_bytes, stream_of(q)));
  return out;
}

void run_backward(const sa_problem& p, const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& out, const Scratch& at_,
                  const Tensor& scratch, const Tensor& d_out, const Tensor& dq, const Tensor& dk, const Tensor& dv) {
  const size_t need = sa_backward_workspace_bytes(&p);
  const Tensor workspace = bytes_on(q, need);
  const char* s = static_cast<const char*>(scratch.data_ptr());
  const float* lse2 = reinterpret_cast<const float*>(s + at_.lse2);
  const float* carry = reinterpret_cast<const float*>(s + at_.carry);
  int st;
  if (p.engine == SA_ENGINE_TCGEN05) {
    const sa_tensor rows[4] = {rows_of(d_out), rows_of(dq), rows_of(dk), rows_of(dv)};
    st = sa_backward_live_tiles(&p, q.data_ptr(), k.data_ptr(), v.data_ptr(), nullptr, out.data_ptr<float>(), lse2, carry, &rows[0],
                                &rows[1], &rows[2], &rows[3], nullptr, nullptr, workspace.data_ptr(), need,
                                at_.table_bytes ? s + at_.table : nullptr, stream_of(q));
  } else {
    st = sa_backward(&p, q.data_ptr(), k.data_ptr(), v.data_ptr(), out.data_ptr<float>(), lse2, carry, d_out.data_ptr(),
                     code_of(d_out), dq.data_ptr(), dk.data_ptr(), dv.data_ptr(), workspace.data_ptr(), need, stream_of(q));
  }
  check("sa_backward", st, true);
}

// The backward is written by hand: a second differentiation through it raises.  A cotangent without a graph of its own has none
// to be differentiated through.
variable_list once_differentiable(const variable_list& grad_out, variable_list grads) {
  if (!c10::GradMode::is_enabled()) return grads;
  if (std::none_of(grad_out.begin(), grad_out.end(), [](const Tensor& g) { return g.defined() && g.requires_grad(); })) return grads;
  variable_list fake;
  size_t n = 0;
  for (auto& g : grads)
    if (g.defined()) {
      fake.push_back(g.detach().set_requires_grad(true));
      ++n;
    }
  auto node = std::make_shared<torch::autograd::DelayedError>(
      "trying to differentiate twice a function that was marked with @once_differentiable", (int64_t)n);
  variable_list out = (*node)(std::move(fake));
  size_t i = 0;
  for (auto& g : grads)
    if (g.defined()) g = out[i++];
  return grads;
}

struct Attend : public torch::autograd::Function<Attend> {
  static Tensor forward(AutogradContext* ctx, const Tensor& q_in, const Tensor& k_in, const Tensor& v_in, int64_t exempt, bool lowp,
                        bool tensor_cores, bool skip, bool low) {
    const c10::cuda::CUDAGuard guard(q_in.device());
    // bf16 when the products run on bf16 operands, otherwise a common dtype (the CUDA-core engine converts as it loads)
    const auto same = q_in.scalar_type() == k_in.scalar_type() && q_in.scalar_type() == v_in.scalar_type();
    const at::ScalarType want = lowp ? at::kBFloat16 : same ? q_in.scalar_type() : at::kFloat;
    auto prepare = [&](const Tensor& t) { return strided(t.scalar_type() == want ? t : t.to(want), tensor_cores); };
    const Tensor q = prepare(q_in), k = prepare(k_in), v = prepare(v_in);
    const sa_problem p = problem_of(q, k, v, tensor_cores ? SA_ENGINE_TCGEN05 : SA_ENGINE_SIMT, exempt);
    const Scratch at_(p, skip);
    const Tensor scratch = bytes_on(q, at_.bytes);
    Tensor y;                                      // `low`: the result in the operand type; fp32 is kept for the backward's row sums
    sa_tensor rows{};
    if (low) {
      y = at::empty(q.sizes(), q.options());
      rows = rows_of(y);
    }
    const Tensor out = run_forward(p, q, k, v, at_, scratch, low ? &rows : nullptr);
    ctx->save_for_backward({q, k, v, out, scratch});
    ctx->saved_data["args"] = c10::List<int64_t>({exempt, (int64_t)p.engine, (int64_t)skip, (int64_t)q_in.scalar_type(),
                                                  (int64_t)k_in.scalar_type(), (int64_t)v_in.scalar_type()});
    return low ? y : out;
  }
  static variable_list backward(AutogradContext* ctx, variable_list grad_out) {
    const auto saved = ctx->get_saved_variables();
    const auto args = ctx->saved_data["args"].toIntVector();
    const Tensor &q = saved[0], &k = saved[1], &v = saved[2];
    variable_list grads(8);
    {
      at::AutoDispatchBelowADInplaceOrView below;
      const c10::cuda::CUDAGuard guard(q.device());
      const sa_problem p = problem_of(q, k, v, (int)args[1], args[0]);
      const Scratch at_(p, args[2] != 0);
      Tensor d_out = grad_out[0];
      if (code_of(d_out) < 0) d_out = d_out.to(at::kFloat);
      d_out = d_out.contiguous();
      if (reinterpret_cast<uintptr_t>(d_out.data_ptr()) % 16 != 0) d_out = d_out.clone();
      const Tensor dq = at::empty(q.sizes(), q.options()), dk = at::empty(q.sizes(), q.options()), dv = at::empty(q.sizes(), q.options());
      run_backward(p, q, k, v, saved[3], at_, unpacked(saved[4]), d_out, dq, dk, dv);
      const Tensor* all[3] = {&dq, &dk, &dv};
      for (int i = 0; i < 3; ++i) {
        const auto want = (at::ScalarType)args[3 + i];
        grads[i] = all[i]->scalar_type() == want ? *all[i] : all[i]->to(want);
      }
    }
    return once_differentiable(grad_out, std::move(grads));
  }
};

// The operator between a fused QKV projection and the output projection: q, k, v are read in place from the (B, T, 3, H, D)
// projection output, the result is (B, T, H * D) in its type, and dq, dk, dv go into one gradient of its shape.
struct AttendPacked : public torch::autograd::Function<AttendPacked> {
  static Tensor part(const Tensor& qkv, int64_t i) { return qkv.select(2, i).transpose(1, 2); }
  static Tensor forward(AutogradContext* ctx, const Tensor& qkv, int64_t exempt, bool skip) {
    const c10::cuda::CUDAGuard guard(qkv.device());
    const int64_t b = qkv.size(0), t = qkv.size(1), h = qkv.size(3), d = qkv.size(4);
    const Tensor q = part(qkv, 0), k = part(qkv, 1), v = part(qkv, 2);
    const sa_problem p = problem_of(q, k, v, SA_ENGINE_TCGEN05, exempt);
    const Scratch at_(p, skip);
    const Tensor scratch = bytes_on(qkv, at_.bytes);
    const Tensor merged = at::empty({b, t, h * d}, qkv.options());
    sa_tensor low{};
    low.ptr = merged.data_ptr();
    low.dtype = code_of(merged);
    low.stride[0] = t * h * d; low.stride[1] = d; low.stride[2] = h * d;
    const Tensor out = run_forward(p, q, k, v, at_, scratch, &low);       // kept for the backward's row sums
    ctx->save_for_backward({qkv, out, scratch});
    ctx->saved_data["args"] = c10::List<int64_t>({exempt, (int64_t)skip});
    return merged;
  }
  static variable_list backward(AutogradContext* ctx, variable_list grad_out) {
    const auto saved = ctx->get_saved_variables();
    const auto args = ctx->saved_data["args"].toIntVector();
    const Tensor& qkv = saved[0];
    variable_list grads(3);
    {
      at::AutoDispatchBelowADInplaceOrView below;
      const c10::cuda::CUDAGuard guard(qkv.device());
      const int64_t b = qkv.size(0), t = qkv.size(1), h = qkv.size(3), d = qkv.size(4);
      const Tensor q = part(qkv, 0), k = part(qkv, 1), v = part(qkv, 2);
      const sa_problem p = problem_of(q, k, v, SA_ENGINE_TCGEN05, args[0]);
      const Scratch at_(p, args[1] != 0);
      Tensor d_out = grad_out[0].to(qkv.scalar_type()).contiguous();
      if (reinterpret_cast<uintptr_t>(d_out.data_ptr()) % 16 != 0) d_out = d_out.clone();
      d_out = d_out.view({b, t, h, d}).transpose(1, 2);
      const Tensor d_qkv = at::empty(qkv.sizes(), qkv.options());
      run_backward(p, q, k, v, saved[1], at_, unpacked(saved[2]), d_out, part(d_qkv, 0), part(d_qkv, 1), part(d_qkv, 2));
      grads[0] = d_qkv;
    }
    return once_differentiable(grad_out, std::move(grads));
  }
};

Tensor attend(const Tensor& q, const Tensor& k, const Tensor& v, int64_t exempt, bool lowp, bool tensor_cores, bool skip, bool low) {
  return Attend::apply(q, k, v, exempt, lowp, tensor_cores, skip, low);
}
Tensor attend_packed(const Tensor& qkv, int64_t exempt, bool skip) { return AttendPacked::apply(qkv, exempt, skip); }

// Rows `cached` .. of a prompt in bf16, (B, H, Tn, D), and the totals of its keys into `selected` (B, G, capacity).  q holds the
// new queries; k, v all keys, or a cache of them.
Tensor prefill_rows(const Tensor& q_in, const Tensor& k_in, const Tensor& v_in, int64_t cached, const Tensor& selected,
                    int64_t exempt, bool skip) {
  const at::NoGradGuard no_grad;
  const c10::cuda::CUDAGuard guard(q_in.device());
  const int64_t b = q_in.size(0), h = q_in.size(1), tn = q_in.size(2), d = q_in.size(3);
  const bool per_head = selected.size(1) == h && h > 1;                   // every head is its own one-head sequence
  auto prepare = [&](const Tensor& t) { return strided(per_head ? t.reshape({b * h, 1, t.size(2), d}) : t, true); };
  const Tensor q = prepare(q_in), k = prepare(k_in), v = prepare(v_in);
  const Tensor y = at::empty({b, h, tn, d}, q.options().dtype(at::kBFloat16));
  sa_problem p = problem_of(q, k, v, SA_ENGINE_TCGEN05, exempt);
  p.seq = (int32_t)(cached + tn);
  auto round_up = [](size_t n) { return (n + 255) / 256 * 256; };
  const size_t lse = round_up((size_t)b * h * tn * 4);
  const size_t carry = round_up((size_t)p.batch * sa_carry_checkpoints(p.engine, p.seq) * p.seq * 4);
  const size_t table = skip ? sa_tile_table_bytes(&p) : 0;
  const size_t split = sa_prefill_scratch_bytes(&p, (int)cached), table_room = round_up(table);
  const Tensor scratch = bytes_on(q, lse + carry + table_room + split);
  char* s = static_cast<char*>(scratch.data_ptr());
  sa_tensor rows{};
  rows.ptr = y.data_ptr();
  rows.dtype = SA_BF16;
  rows.stride[0] = p.heads * tn * d; rows.stride[1] = tn * d; rows.stride[2] = d;
  check("sa_prefill_rows",
        sa_prefill_rows(&p, (int)cached, q.data_ptr(), k.data_ptr(), v.data_ptr(), selected.data_ptr<float>(), selected.size(2), &rows,
                        reinterpret_cast<float*>(s), reinterpret_cast<float*>(s + lse), table ? s + lse + carry : nullptr, table,
                        split ? s + lse + carry + table_room : nullptr, split, stream_of(q)));
  return y;
}

// New keys and values into the cache from position `at` on; `begin`: the first ones, with zeros behind them (and in `selected`).
// False where the rows are not of the cache's type and device with a contiguous last axis, or are a view of the cache: the
// caller copies.
bool store_rows(const Tensor& kc, const Tensor& vc, const Tensor& selected, const Tensor& k, const Tensor& v, int64_t at, bool begin) {
  const int64_t d = kc.size(3);
  if (!kc.is_cuda() || code_of(kc) < 0 || vc.scalar_type() != kc.scalar_type() || k.scalar_type() != kc.scalar_type() ||
      v.scalar_type() != kc.scalar_type() || k.device() != kc.device() || v.device() != kc.device() || k.stride(3) != 1 ||
      v.stride(3) != 1 || !kc.is_contiguous() || !vc.is_contiguous() || !selected.is_contiguous() || kc.size(0) * kc.size(1) > 65535 ||
      (d != 16 && d != 32 && d != 64 && d != 128))
    return false;
  for (const Tensor* x : {&k, &v})
    if (x->is_alias_of(kc) || x->is_alias_of(vc)) return false;
  const c10::cuda::CUDAGuard guard(kc.device());
  const sa_tensor kr = rows_of(k), vr = rows_of(v);
  check("sa_cache_store", sa_cache_store(code_of(kc), (int)kc.size(0), (int)kc.size(1), (int)selected.size(1), (int)k.size(2),
                                         (int)kc.size(2), (int)d, (int)at, begin, &kr, &vr, kc.data_ptr(), vc.data_ptr(),
                                         selected.data_ptr<float>(), stream_of(kc)));
  return true;
}

// A decode step.  Everything about the cache is looked at in every step.  What stays with it is the step's scratch: (tensor,
// address of `selected`, stream, tickets), good for steps that have all three alike, since the tickets are at zero only between
// steps of one order and a copy of a cache, or another stream, must not share them.  Returns y and the scratch to be kept,
// None where the one that was given is.  A step that is being captured uses scratch of the graph's own: what the graph
// will write to is not the cache's to replace, and what it is to clear has not been cleared yet.
pybind11::tuple decode(const Tensor& kc, const Tensor& vc, const Tensor& selected, const std::optional<Tensor>& norms,
                       const pybind11::object& kept, Tensor q1, Tensor k1, Tensor v1, int64_t length, int64_t exempt, bool y_low) {
  TORCH_CHECK_VALUE(kc.dim() == 4 && selected.dim() == 3, "the cache must be (B, H, capacity, D) with (B, G, capacity) `selected`");
  const int64_t b = kc.size(0), h = kc.size(1), capacity = kc.size(2), d = kc.size(3), groups = selected.size(1);
  TORCH_CHECK_VALUE(length < capacity, "decode step past the cache capacity (context_length)");
  TORCH_CHECK_VALUE(kc.is_cuda() && kc.is_contiguous() && vc.is_contiguous() && selected.is_contiguous() && vc.device() == kc.device() &&
                        selected.device() == kc.device() && vc.numel() >= kc.numel() && selected.numel() >= b * groups * capacity,
                    "the cache must be contiguous CUDA tensors");
  TORCH_CHECK_VALUE(code_of(kc) >= 0 && vc.scalar_type() == kc.scalar_type() && selected.scalar_type() == at::kFloat,
                    "cache dtype must be float16, bfloat16 or float32 with fp32 `selected`");
  TORCH_CHECK_VALUE(d == 16 || d == 32 || d == 64 || d == 128, "head_dim must be one of (16, 32, 64, 128); got ", d);
  TORCH_CHECK_VALUE(!norms || (norms->device() == kc.device() && norms->scalar_type() == at::kFloat && norms->is_contiguous() &&
                               norms->sizes() == kc.sizes().slice(0, 3)),
                    "cache['key_norms'] must be a contiguous fp32 CUDA tensor (B, H, capacity)");
  const at::NoGradGuard no_grad;
  const c10::cuda::CUDAGuard guard(kc.device());
  void* const stream = stream_of(kc);
  const auto selected_at = reinterpret_cast<uint64_t>(selected.data_ptr()), stream_at = reinterpret_cast<uint64_t>(stream);
  const bool captured = at::cuda::currentStreamCaptureStatusMayInitCtx() != at::cuda::CaptureStatus::None;
  const size_t need = sa_decode_workspace_bytes((int)b, (int)h, (int)groups, (int)(captured ? length : capacity - 1), (int)d);
  const uint64_t layout = ((uint64_t)(b * h) << 32) + (uint64_t)(b * groups);      // with the capacity: where the tickets are
  Tensor workspace;
  if (!captured && PyTuple_Check(kept.ptr()) && PyTuple_GET_SIZE(kept.ptr()) == 5) {
    auto number = [&](int i) { return PyLong_AsUnsignedLongLongMask(PyTuple_GET_ITEM(kept.ptr(), i)); };
    if (THPVariable_Check(PyTuple_GET_ITEM(kept.ptr(), 0)) && number(1) == selected_at && number(2) == stream_at &&
        number(3) == layout && number(4) == (uint64_t)capacity) {
      const Tensor& t = THPVariable_Unpack(PyTuple_GET_ITEM(kept.ptr(), 0));
      if (t.device() == kc.device() && t.scalar_type() == at::kByte && t.is_contiguous() && (size_t)t.numel() >= need) workspace = t;
    }
  }
  const bool fresh = !workspace.defined();
  Tensor y;
  {
    const pybind11::gil_scoped_release release;
    for (Tensor* t : {&q1, &k1, &v1})
      if (t->scalar_type() != kc.scalar_type() || t->device() != kc.device() || !t->is_contiguous() || t->numel() != b * h * d)
        *t = t->reshape({b, h, d}).to(kc.options()).contiguous();
    if (fresh) workspace = bytes_on(kc, need);
    y = at::empty({b, h, 1, d}, y_low ? kc.options() : kc.options().dtype(at::kFloat));
    sa_decode a{};
    a.struct_bytes = sizeof(sa_decode);
    a.dtype = code_of(kc);
    a.y_dtype = y_low ? a.dtype : SA_F32;
    a.batch = (int32_t)b; a.heads = (int32_t)h; a.groups = (int32_t)groups; a.capacity = (int32_t)capacity; a.head_dim = (int32_t)d;
    a.length = (int32_t)length;
    a.exempt = (int32_t)exempt;
    a.tickets_zero = captured ? 0 : fresh ? 2 : 1;
    a.q1 = q1.data_ptr(); a.k1 = k1.data_ptr(); a.v1 = v1.data_ptr();
    a.k_cache = kc.data_ptr(); a.v_cache = vc.data_ptr(); a.selected = selected.data_ptr<float>();
    a.key_norms = norms ? norms->data_ptr<float>() : nullptr;
    a.y = y.data_ptr();
    a.workspace = workspace.data_ptr();
    a.workspace_bytes = workspace.numel();
    a.stream = stream;
    check("sa_decode_step", sa_decode_run(&a));
  }
  pybind11::object keep = pybind11::none();
  if (fresh && !captured) keep = pybind11::make_tuple(workspace, selected_at, stream_at, layout, capacity);
  return pybind11::make_tuple(y, keep);
}

}  // namespace

PYBIND11_MODULE(_native, m) {
  using nogil = pybind11::call_guard<pybind11::gil_scoped_release>;
  m.def("attend", &attend, nogil());
  m.def("attend_packed", &attend_packed, nogil());
  m.def("prefill_rows", &prefill_rows, nogil());
  m.def("store_rows", &store_rows, nogil());
  m.def("decode", &decode);
}

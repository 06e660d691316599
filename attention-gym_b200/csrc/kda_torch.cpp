// CUDA implementations of the operators that stand on the path of small calls: they allocate outputs and workspace
// and make one call into the C ABI of libkda_b200.so on the current stream, as the Python implementations of
// kda_b200/ops.py do for the other operators.  The schemas and the fake implementations are declared there.
//
// A call of a few tokens is bound by the host: an implementation in Python costs the dispatcher's way through
// the interpreter, some ten allocations and a ctypes call of thirty arguments.
#include <ATen/ATen.h>
#include <ATen/record_function.h>
#include <c10/cuda/CUDAFunctions.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/library.h>

#include <atomic>
#include <optional>
#include <tuple>

#include "../../include/kda_b200.h"

namespace {

using at::Tensor;
using OptTensor = std::optional<Tensor>;

constexpr int64_t kChunk = 64, kDim = 128;
std::atomic<int64_t> g_launches{0};

void* stream() { return (void*)c10::cuda::getCurrentCUDAStream().stream(); }
void* ptr(const Tensor& t) { return t.data_ptr(); }
void* ptr(const OptTensor& t) { return t ? t->data_ptr() : nullptr; }
float* fptr(const Tensor& t) { return (float*)t.data_ptr(); }
float* fptr(const OptTensor& t) { return t ? (float*)t->data_ptr() : nullptr; }
const int32_t* iptr(const OptTensor& t) { return t ? (const int32_t*)t->data_ptr() : nullptr; }

int dtype_code(const Tensor& t) {
  switch (t.scalar_type()) {
    case at::kFloat: return KDA_F32;
    case at::kBFloat16: return KDA_BF16;
    case at::kHalf: return KDA_F16;
    default: TORCH_CHECK_TYPE(false, "unsupported dtype ", t.scalar_type());
  }
}
const char* error_text(int rc) {
  switch (rc) {
    case KDA_ERR_ARG: return "invalid argument";
    case KDA_ERR_UNSUPPORTED: return "unsupported shape";
    case KDA_ERR_LAUNCH: return "CUDA launch failed";
    case KDA_ERR_SCRATCH: return "problem exceeds the built-in scratch array";
    default: return "unknown error";
  }
}
// the entry point as a named range of an active profiler, its launches counted, its status an exception
template <typename F>
void call(const char* name, int launches, F&& entry) {
  int rc;
  {
    RECORD_USER_SCOPE(name);
    rc = entry();
  }
  TORCH_CHECK(rc == KDA_OK, name + 9, " failed: ", error_text(rc));       // (without "kda_b200/")
  g_launches.fetch_add(launches, std::memory_order_relaxed);
}

Tensor f32(const Tensor& t) { return t.to(at::kFloat).contiguous(); }
OptTensor f32(const OptTensor& t) { return t ? OptTensor(f32(*t)) : OptTensor(); }
Tensor empty(at::IntArrayRef shape, const Tensor& like, at::ScalarType dtype) {
  return at::empty(shape, like.options().dtype(dtype));
}
Tensor fresh(at::IntArrayRef shape, const Tensor& like, at::ScalarType dtype, bool zero) {
  return zero ? at::zeros(shape, like.options().dtype(dtype)) : empty(shape, like, dtype);
}
// zeroes the rows of [1, tokens, ...] results that no packed sequence covers
void zero_unused_rows(std::initializer_list<Tensor> results, int64_t tokens, const OptTensor& cu, const OptTensor& co) {
  void* buffers[8];
  int64_t row_bytes[8];
  int count = 0;
  for (const Tensor& t : results) {
    if (!t.defined()) continue;
    buffers[count] = t.data_ptr();
    row_bytes[count++] = t.numel() / std::max<int64_t>(tokens, 1) * t.element_size();
  }
  call("kda_b200/kda_zero_unused_rows", 1, [&] {
    return kda_zero_unused_rows(buffers, row_bytes, count, iptr(cu), iptr(co), (int)kChunk, (int)(cu->size(0) - 1), tokens,
                                stream());
  });
}
// the largest number of chunks that `nseq` sequences can have in `tokens` tokens
int64_t chunk_capacity(int64_t tokens, int64_t nseq) {
  TORCH_CHECK_VALUE(nseq >= 1, "num_sequences must be positive, got ", nseq);
  const int64_t nonempty = std::min(tokens, nseq);
  return nonempty == 0 ? 0 : nonempty + (tokens - nonempty) / kChunk;
}

int64_t fwd_workspace(int64_t batch, int64_t tokens, int64_t heads, int64_t packed_nseq, bool keep) {
  if (packed_nseq < 0) return kda_chunk_fwd_dense_workspace_bytes((int)batch, tokens, (int)heads, keep);
  if (keep) return kda_chunk_bwd_workspace_bytes(tokens, (int)heads, chunk_capacity(tokens, packed_nseq));
  return kda_chunk_fwd_workspace_bytes(tokens, (int)heads);
}

void check_core(const Tensor& q, const Tensor& k, const Tensor& v) {
  TORCH_CHECK_VALUE(q.is_cuda(), "the fused KDA core requires CUDA tensors");
  TORCH_CHECK_VALUE(q.dim() == 4 && q.size(3) == kDim && v.size(-1) == kDim, "the fused KDA core requires K=V=128");
  TORCH_CHECK_TYPE(q.scalar_type() == at::kBFloat16 && k.scalar_type() == at::kBFloat16 && v.scalar_type() == at::kBFloat16,
                   "the fused KDA core takes bfloat16 q, k, v");
}

struct Forward { Tensor out, state, aqk, akk, workspace, rstd_q, rstd_k; };
struct Shape {
  int64_t batch, tokens, heads, nseq, capacity;
  bool packed;
  Shape(const Tensor& x, const OptTensor& cu) {
    TORCH_CHECK_VALUE(x.dim() == 4, "expected q [B, T, H, 128], got ", x.sizes());
    batch = x.size(0); tokens = x.size(1); heads = x.size(2);
    packed = cu.has_value();
    TORCH_CHECK_VALUE(!packed || batch == 1, "packed cu_seqlens require batch size one");
    nseq = packed ? cu->size(0) - 1 : batch;
    capacity = packed ? chunk_capacity(tokens, nseq) : batch * ((tokens + kChunk - 1) / kChunk);
  }
  int64_t total() const { return batch * tokens; }
};

// q, k, v given; norm: they arrive unnormalised (eps)
Forward chunk_forward(const Tensor& q_, const Tensor& k_, const Tensor& v_, const Tensor& gate_, const Tensor& beta_,
                      const OptTensor& h0_, const OptTensor& cu, const OptTensor& co, bool want_state, bool keep, bool norm,
                      double eps) {
  check_core(q_, k_, v_);
  const Shape s(q_, cu);
  const Tensor q = q_.contiguous(), k = k_.contiguous(), v = v_.contiguous(), gate = f32(gate_), beta = f32(beta_);
  const OptTensor h0 = f32(h0_);
  Forward f;
  f.out = empty(v.sizes(), v, v.scalar_type());
  f.aqk = empty({s.batch, s.tokens, s.heads, kChunk}, q, q.scalar_type());
  f.akk = at::empty_like(f.aqk);
  if (norm) {
    f.rstd_q = empty({s.batch, s.tokens, s.heads}, q, at::kFloat);
    f.rstd_k = at::empty_like(f.rstd_q);
  }
  if (s.packed) zero_unused_rows({f.out, f.rstd_q, f.rstd_k}, s.tokens, cu, co);
  if (want_state) f.state = empty({s.nseq, s.heads, kDim, kDim}, q, at::kFloat);
  const int64_t bytes = fwd_workspace(s.batch, s.tokens, s.heads, s.packed ? s.nseq : -1, keep);
  f.workspace = empty({bytes}, q, at::kByte);
  float* ht = want_state ? fptr(f.state) : nullptr;
  const int D = (int)kDim, H = (int)s.heads;
  if (s.packed && norm) {
    call("kda_b200/kda_chunk_fwd_qknorm", 3, [&] {
      return kda_chunk_fwd_qknorm(ptr(q), ptr(k), ptr(v), fptr(gate), fptr(beta), fptr(h0), ht, ptr(f.out), ptr(f.aqk),
                                  ptr(f.akk), fptr(f.rstd_q), fptr(f.rstd_k), (float)eps, iptr(cu), iptr(co), (int)s.nseq,
                                  s.total(), H, D, D, (int)s.capacity, ptr(f.workspace), bytes, keep, stream());
    });
  } else if (norm) {
    call("kda_b200/kda_chunk_fwd_dense_qknorm", 3, [&] {
      return kda_chunk_fwd_dense_qknorm(ptr(q), ptr(k), ptr(v), fptr(gate), fptr(beta), fptr(h0), ht, ptr(f.out), ptr(f.aqk),
                                        ptr(f.akk), fptr(f.rstd_q), fptr(f.rstd_k), (float)eps, (int)s.batch, s.tokens, H, D,
                                        D, ptr(f.workspace), bytes, keep, stream());
    });
  } else if (s.packed) {
    call(keep ? "kda_b200/kda_chunk_fwd_save" : "kda_b200/kda_chunk_fwd", 3, [&] {
      return (keep ? kda_chunk_fwd_save : kda_chunk_fwd)(
          ptr(q), ptr(k), ptr(v), fptr(gate), fptr(beta), fptr(h0), ht, ptr(f.out), ptr(f.aqk), ptr(f.akk), iptr(cu), iptr(co),
          (int)s.nseq, s.total(), H, D, D, (int)s.capacity, ptr(f.workspace), bytes, stream());
    });
  } else {
    call(keep ? "kda_b200/kda_chunk_fwd_dense_save" : "kda_b200/kda_chunk_fwd_dense", 3, [&] {
      return (keep ? kda_chunk_fwd_dense_save : kda_chunk_fwd_dense)(
          ptr(q), ptr(k), ptr(v), fptr(gate), fptr(beta), fptr(h0), ht, ptr(f.out), ptr(f.aqk), ptr(f.akk), (int)s.batch,
          s.tokens, H, D, D, ptr(f.workspace), bytes, stream());
    });
  }
  return f;
}
Tensor state_or_empty(const Forward& f) { return f.state.defined() ? f.state : empty({0}, f.out, at::kFloat); }

std::tuple<Tensor, Tensor, Tensor> chunk_fwd(const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& gate,
                                             const Tensor& beta, const OptTensor& h0, bool) {
  Forward f = chunk_forward(q, k, v, gate, beta, h0, {}, {}, false, false, false, 0);
  return {f.out, f.aqk, f.akk};
}
std::tuple<Tensor, Tensor, Tensor, Tensor> chunk_fwd_with_state(const Tensor& q, const Tensor& k, const Tensor& v,
                                                                const Tensor& gate, const Tensor& beta, const OptTensor& h0,
                                                                bool) {
  Forward f = chunk_forward(q, k, v, gate, beta, h0, {}, {}, true, false, false, 0);
  return {f.out, f.state, f.aqk, f.akk};
}
std::tuple<Tensor, Tensor, Tensor> chunk_fwd_ragged(const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& gate,
                                                    const Tensor& beta, const OptTensor& h0, const Tensor& cu,
                                                    const Tensor& co, bool) {
  Forward f = chunk_forward(q, k, v, gate, beta, h0, cu, co, false, false, false, 0);
  return {f.out, f.aqk, f.akk};
}
std::tuple<Tensor, Tensor, Tensor, Tensor> chunk_fwd_ragged_with_state(const Tensor& q, const Tensor& k, const Tensor& v,
                                                                       const Tensor& gate, const Tensor& beta,
                                                                       const OptTensor& h0, const Tensor& cu,
                                                                       const Tensor& co, bool) {
  Forward f = chunk_forward(q, k, v, gate, beta, h0, cu, co, true, false, false, 0);
  return {f.out, f.state, f.aqk, f.akk};
}
std::tuple<Tensor, Tensor, Tensor, Tensor, Tensor> chunk_fwd_saved(const Tensor& q, const Tensor& k, const Tensor& v,
                                                                   const Tensor& gate, const Tensor& beta,
                                                                   const OptTensor& h0, const OptTensor& cu,
                                                                   const OptTensor& co, bool want_state) {
  Forward f = chunk_forward(q, k, v, gate, beta, h0, cu, co, want_state, true, false, 0);
  return {f.out, state_or_empty(f), f.aqk, f.akk, f.workspace};
}
std::tuple<Tensor, Tensor, Tensor, Tensor, Tensor, Tensor, Tensor> chunk_fwd_qknorm(
    const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& gate, const Tensor& beta, const OptTensor& h0,
    const OptTensor& cu, const OptTensor& co, bool want_state, bool keep, double eps) {
  Forward f = chunk_forward(q, k, v, gate, beta, h0, cu, co, want_state, keep, true, eps);
  return {f.out, state_or_empty(f), f.aqk, f.akk, f.workspace, f.rstd_q, f.rstd_k};
}

// ---- backward from kept intermediates ----------------------------------------------------------------------
struct Cotangents {
  Tensor gate, beta, d_out, offsets;
  OptTensor d_state, h0;
  const int32_t *cu, *co;
  Tensor dg, db, dh0;
  Cotangents(const Shape& s, const Tensor& like, const Tensor& gate_, const Tensor& beta_, const Tensor& saved,
             const OptTensor& cu_, const OptTensor& co_, const OptTensor& d_out_, const OptTensor& d_state_,
             const OptTensor& h0_, bool want_state_grad) {
    TORCH_CHECK_VALUE(saved.numel() >= kda_chunk_bwd_workspace_bytes(s.total(), (int)s.heads, s.capacity) &&
                          saved.scalar_type() == at::kByte && saved.is_cuda(),
                      "`saved` is not the buffer the forward operator returned for these shapes");
    gate = f32(gate_); beta = f32(beta_);
    d_out = d_out_ ? d_out_->to(at::kBFloat16).contiguous()
                   : at::zeros({s.batch, s.tokens, s.heads, kDim}, like.options().dtype(at::kBFloat16));
    d_state = f32(d_state_); h0 = f32(h0_);
    if (s.packed) {
      cu = iptr(cu_); co = iptr(co_);
    } else {
      offsets = empty({2 * (s.batch + 1)}, like, at::kInt);
      int32_t* base = (int32_t*)offsets.data_ptr();
      call("kda_b200/kda_dense_offsets", 1, [&] { return kda_dense_offsets(base, (int)s.batch, (int)s.tokens, stream()); });
      cu = base; co = base + s.batch + 1;
    }
    dg = at::empty_like(gate);
    db = at::empty_like(beta);
    if (want_state_grad) dh0 = empty({s.nseq, s.heads, kDim, kDim}, like, at::kFloat);
  }
  float* dh0_ptr() const { return dh0.defined() ? fptr(dh0) : nullptr; }
  Tensor dh0_or_empty(const Tensor& like) const { return dh0.defined() ? dh0 : empty({0}, like, at::kFloat); }
};

std::tuple<Tensor, Tensor, Tensor, Tensor, Tensor, Tensor> chunk_backward(
    const Tensor& q_, const Tensor& k_, const Tensor& v_, const Tensor& gate, const Tensor& beta, const Tensor& aqk,
    const Tensor& akk, const Tensor& saved, const OptTensor& rstd_q, const OptTensor& rstd_k, const OptTensor& cu,
    const OptTensor& co, const OptTensor& d_out, const OptTensor& d_state, const OptTensor& h0, bool want_state_grad) {
  const Shape s(q_, cu);
  const Tensor q = q_.contiguous(), k = k_.contiguous(), v = v_.contiguous();
  const Cotangents c(s, q, gate, beta, saved, cu, co, d_out, d_state, h0, want_state_grad);
  const Tensor dq = at::empty_like(q), dk = at::empty_like(k), dv = at::empty_like(v);
  if (s.packed) zero_unused_rows({dq, dk, dv, c.dg, c.db}, s.tokens, cu, co);
  const int D = (int)kDim, H = (int)s.heads;
  if (rstd_q) {
    const Tensor rq = rstd_q->contiguous(), rk = rstd_k->contiguous();
    call("kda_b200/kda_chunk_bwd_qknorm_saved", 2, [&] {
      return kda_chunk_bwd_qknorm_saved(ptr(q), ptr(k), ptr(v), fptr(c.gate), fptr(c.beta), ptr(aqk), ptr(akk), fptr(c.h0),
                                        ptr(c.d_out), fptr(c.d_state), ptr(dq), ptr(dk), ptr(dv), fptr(c.dg), fptr(c.db),
                                        c.dh0_ptr(), c.cu, c.co, (int)s.nseq, s.total(), H, D, D, (int)s.capacity, fptr(rq),
                                        fptr(rk), ptr(saved), saved.numel(), stream());
    });
  } else {
    call("kda_b200/kda_chunk_bwd_saved", 2, [&] {
      return kda_chunk_bwd_saved(ptr(q), ptr(k), ptr(v), fptr(c.gate), fptr(c.beta), ptr(aqk), ptr(akk), fptr(c.h0),
                                 ptr(c.d_out), fptr(c.d_state), ptr(dq), ptr(dk), ptr(dv), fptr(c.dg), fptr(c.db),
                                 c.dh0_ptr(), c.cu, c.co, (int)s.nseq, s.total(), H, D, D, (int)s.capacity, ptr(saved),
                                 saved.numel(), stream());
    });
  }
  return {dq, dk, dv, c.dg, c.db, c.dh0_or_empty(q)};
}
std::tuple<Tensor, Tensor, Tensor, Tensor, Tensor, Tensor> chunk_bwd_saved(
    const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& gate, const Tensor& beta, const Tensor& aqk,
    const Tensor& akk, const Tensor& saved, const OptTensor& cu, const OptTensor& co, const OptTensor& d_out,
    const OptTensor& d_state, const OptTensor& h0, bool want_state_grad) {
  return chunk_backward(q, k, v, gate, beta, aqk, akk, saved, {}, {}, cu, co, d_out, d_state, h0, want_state_grad);
}
std::tuple<Tensor, Tensor, Tensor, Tensor, Tensor, Tensor> chunk_bwd_qknorm(
    const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& gate, const Tensor& beta, const Tensor& aqk,
    const Tensor& akk, const Tensor& saved, const Tensor& rstd_q, const Tensor& rstd_k, const OptTensor& cu,
    const OptTensor& co, const OptTensor& d_out, const OptTensor& d_state, const OptTensor& h0, bool want_state_grad) {
  return chunk_backward(q, k, v, gate, beta, aqk, akk, saved, rstd_q, rstd_k, cu, co, d_out, d_state, h0, want_state_grad);
}

// ---- token scan and decode step --------------------------------------------------------------------------------
std::pair<Tensor, Tensor> recurrent(const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& gate,
                                    const Tensor& beta, const OptTensor& h0_, const OptTensor& cu, const OptTensor& slots,
                                    bool want_state) {
  TORCH_CHECK_VALUE(q.is_cuda(), "the fused recurrent scan requires CUDA tensors");
  TORCH_CHECK_VALUE(q.dim() == 4, "expected q [B, T, H, K], got ", q.sizes());
  const int64_t batch = q.size(0), tokens = q.size(1), heads = q.size(2), K = q.size(3), V = v.size(-1);
  const int64_t nseq = cu ? cu->size(0) - 1 : batch;
  const Tensor out = fresh(v.sizes(), q, q.scalar_type(), cu.has_value());
  Tensor final;
  OptTensor h0 = h0_;
  int64_t slot_stride = heads * K * V, num_slots = 0;
  if (slots) {
    slot_stride = h0->stride(0);
    num_slots = h0->size(0);
  } else {
    h0 = f32(h0_);
    if (want_state) final = empty({nseq, heads, K, V}, q, at::kFloat);
  }
  call("kda_b200/kda_recurrent_fwd", 1, [&] {
    return kda_recurrent_fwd(ptr(q), ptr(k), ptr(v), ptr(gate), ptr(beta), dtype_code(q), dtype_code(k), dtype_code(v),
                             dtype_code(gate), dtype_code(beta), fptr(h0), final.defined() ? fptr(final) : nullptr, ptr(out),
                             dtype_code(out), iptr(cu), iptr(slots), slot_stride, (int)num_slots, (int)nseq, (int)tokens,
                             (int)heads, (int)K, (int)V, (float)std::pow((double)K, -0.5), stream());
  });
  return {out, final};
}
std::tuple<Tensor, Tensor> recurrent_fwd(const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& gate,
                                         const Tensor& beta, const OptTensor& h0, const OptTensor& cu, bool) {
  auto r = recurrent(q, k, v, gate, beta, h0, cu, {}, true);
  return {r.first, r.second};
}
Tensor recurrent_fwd_no_state(const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& gate, const Tensor& beta,
                              const OptTensor& h0, const OptTensor& cu, bool) {
  return recurrent(q, k, v, gate, beta, h0, cu, {}, false).first;
}
Tensor recurrent_fwd_paged(const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& gate, const Tensor& beta,
                           const Tensor& pool, const Tensor& slots, const OptTensor& cu, bool) {
  return recurrent(q, k, v, gate, beta, pool, cu, slots, false).first;
}

int activation_code(const std::optional<std::string>& activation) {
  if (!activation) return 0;
  TORCH_CHECK_VALUE(*activation == "silu", "unknown activation '", *activation, "'; built in: None, 'silu'");
  return 1;
}
Tensor decode_step(const Tensor& x_, const Tensor& weight_, const Tensor& conv_state, const Tensor& pool,
                   const Tensor& slots, const Tensor& raw_gate_, const Tensor& A_log_, const Tensor& dt_bias_,
                   const Tensor& beta_, std::optional<std::string> activation, double lower_bound, double eps) {
  const Tensor x = x_.contiguous(), weight = weight_.contiguous(), raw_gate = raw_gate_.contiguous(),
               beta = beta_.contiguous(), A_log = f32(A_log_), dt_bias = f32(dt_bias_);
  const int nseq = (int)x.size(0), heads = (int)pool.size(1), width = (int)weight.size(1), dtype = dtype_code(x);
  const Tensor out = empty({nseq, heads, kDim}, x, x.scalar_type());
  const int64_t bits = (int64_t)ptr(x) | (int64_t)ptr(weight) | (int64_t)ptr(conv_state) | (int64_t)ptr(dt_bias) |
                       (int64_t)ptr(pool) | 4 * pool.stride(0);
  const int64_t need = kda_decode_step_scratch_bytes(bits, dtype, nseq, heads, width);      // 0: one launch
  const Tensor scratch = need ? empty({need}, x, at::kByte) : Tensor();
  const int act = activation_code(activation);
  call("kda_b200/kda_decode_step", need ? 2 : 1, [&] {
    return kda_decode_step(ptr(x), ptr(weight), ptr(conv_state), (const int32_t*)ptr(slots), ptr(raw_gate),
                           dtype_code(raw_gate), fptr(A_log), fptr(dt_bias), ptr(beta), dtype_code(beta), fptr(pool),
                           pool.stride(0), need ? ptr(scratch) : nullptr, ptr(out), dtype, nseq, heads, width,
                           (int)conv_state.size(0), (int)pool.size(0), act, (float)lower_bound, (float)eps, stream());
  });
  return out;
}

}  // namespace

// launches counted here since the library was loaded
extern "C" int64_t kda_torch_launches(void) { return g_launches.load(std::memory_order_relaxed); }

TORCH_LIBRARY_IMPL(kda_b200, CUDA, m) {
  m.impl("kda_chunk_fwd", chunk_fwd);
  m.impl("kda_chunk_fwd_with_state", chunk_fwd_with_state);
  m.impl("kda_chunk_fwd_ragged", chunk_fwd_ragged);
  m.impl("kda_chunk_fwd_ragged_with_state", chunk_fwd_ragged_with_state);
  m.impl("kda_chunk_fwd_saved", chunk_fwd_saved);
  m.impl("kda_chunk_fwd_qknorm", chunk_fwd_qknorm);
  m.impl("kda_chunk_bwd_saved", chunk_bwd_saved);
  m.impl("kda_chunk_bwd_qknorm", chunk_bwd_qknorm);
  m.impl("kda_recurrent_fwd", recurrent_fwd);
  m.impl("kda_recurrent_fwd_no_state", recurrent_fwd_no_state);
  m.impl("kda_recurrent_fwd_paged", recurrent_fwd_paged);
}
TORCH_LIBRARY_IMPL(kda_b200_fused, CUDA, m) { m.impl("decode_step", decode_step); }

// The operator classes' usual calls as native functions (Python module `iex_torch_ext`).
//
// MySpMM and MyLinear are autograd operators in Python
// (intrasm_engine/pytorch/cpp_extensions/layers_and_funcs/sputnik.py:19-149, torch.py:6-31): the keyword
// dictionaries, the saved-tensor bookkeeping and the backward pass in the interpreter cost 50 us
// forward and 130 us forward + backward, several times the kernels of an ordinary layer.  When no
// graph constructor is recording, `run` comes here instead: the same kernels in the same order,
// with the autograd node, its saved tensors and its backward pass in C++.
//
// It also holds the choice between the ways to multiply an fp16 CSR matrix (spmm_half_way).
#include "iex_torch_ops.h"

#include <c10/core/impl/TorchDispatchModeTLS.h>
#include <torch/csrc/autograd/edge.h>
#include <torch/csrc/autograd/function.h>
#include <torch/csrc/autograd/functions/basic_ops.h>
#include <torch/csrc/autograd/functions/utils.h>
#include <torch/csrc/autograd/saved_variable.h>
#include <torch/csrc/jit/frontend/tracer.h>
#include <torch/csrc/utils/pybind.h>

#include <algorithm>
#include <array>
#include <optional>

namespace iex_torch {
namespace {

using torch::autograd::Node;
using torch::autograd::SavedVariable;
using torch::autograd::variable_list;

int index_bits(const at::Tensor& ci) { return ci.scalar_type() == at::kShort ? 16 : 32; }
int64_t round8(int64_t v) { return (v + 7) / 8 * 8; }
bool aligned16(const at::Tensor& t) { return (reinterpret_cast<uintptr_t>(t.data_ptr()) & 15u) == 0; }

// Whether a call may go past the dispatcher: nobody records the operators (torch.jit.trace, a dispatch mode such as
// make_fx or FakeTensorMode), and the operands are ordinary tensors without tangents.  Otherwise the callers in Python go on to the
// autograd functions and registered operators, which a recorder sees and which refuse what they have no rule for.
bool plain(std::initializer_list<const at::Tensor*> operands) {
  if (torch::jit::tracer::isTracing() || c10::impl::TorchDispatchModeTLS::any_modes_set()) return false;
  constexpr c10::DispatchKeySet special({c10::DispatchKey::Python, c10::DispatchKey::PythonTLSSnapshot,
                                         c10::DispatchKey::Functionalize, c10::DispatchKey::Conjugate,
                                         c10::DispatchKey::Negative, c10::DispatchKey::ZeroTensor,
                                         c10::DispatchKey::FuncTorchBatched, c10::DispatchKey::BatchedNestedTensor,
                                         c10::DispatchKey::FuncTorchGradWrapper});
  for (const at::Tensor* t : operands)
    if (!t->defined() || t->key_set().has_any(special) || t->_fw_grad(/*level=*/0).defined()) return false;
  return true;
}

// First-order gradients of a backward pass that is itself recorded (create_graph): differentiating them again is an error,
// as the kernels have no second derivative.
variable_list once_differentiable(variable_list&& grads, const at::Tensor& grad, const at::Tensor& a, const at::Tensor& b,
                                  const char* what) {
  if (torch::autograd::compute_requires_grad(grad, a, b)) {
    auto error = std::make_shared<torch::autograd::Error>(std::string(what) + " cannot be differentiated twice",
                                                          torch::autograd::collect_next_edges(grad, a, b));
    for (at::Tensor& g : grads)
      if (g.defined()) torch::autograd::set_history(g, error);
  }
  return std::move(grads);
}

// ---------------------------------------------------------------------------- fp16 CSR products

// The dense fp16 copy [m, round8(k)] of a CSR matrix, as an operand of the products below that sum NaN outputs again.
at::Tensor expand(const at::Tensor& values, const at::Tensor& ro, const at::Tensor& ci, int64_t m, int64_t k) {
  const int64_t ld = round8(k);
  at::Tensor dense = empty(values, {m, ld});
  check_status(iex_csr_expand_f16(m, k, ld, ro.data_ptr<int>(), ci.data_ptr(), index_bits(ci), values.data_ptr(),
                                  dense.data_ptr(), stream_of(values)),
               "iex_csr_expand_f16");
  return dense;
}

// A row-major matrix as a TMA operand: itself, or a copy with rows padded to 16 bytes.
at::Tensor tma_rows(const at::Tensor& x) {
  if (x.size(1) % 8 == 0 && aligned16(x)) return x;
  const int64_t ld = round8(x.size(1));
  at::Tensor padded = empty(x, {x.size(0), ld});
  check_status(iex_pad_rows_f16(x.size(0), x.size(1), ld, x.data_ptr(), padded.data_ptr(), stream_of(x)),
               "iex_pad_rows_f16");
  return padded;
}

// The CSR matrix that one operand of a product is the dense copy of; `perm` (optional) gives each position's value.
struct Stored {
  int operand;  // 0: a, 1: b
  const at::Tensor &ro, &ci, &values;
  const at::Tensor* perm = nullptr;
};

// The dense product.  Outputs that come out NaN are summed again from the stored positions, so that an infinity or NaN in the
// other operand reaches only the outputs that have a position there, as in a CSR product.
void gemm(int64_t m, int64_t n, int64_t k, const at::Tensor& a, bool a_mn, const at::Tensor& b, bool b_mn,
          const at::Tensor& out, bool out_t, const Stored& s) {
  check_status(iex_gemm_f16_csr(m, n, k, a.data_ptr(), a_mn, a.size(1), b.data_ptr(), b_mn, b.size(1), out.data_ptr(), out_t,
                                out.size(1), s.operand, s.ro.data_ptr<int>(), s.ci.data_ptr(), index_bits(s.ci),
                                s.values.data_ptr(),
                                s.perm ? reinterpret_cast<const long long*>(s.perm->data_ptr<int64_t>()) : nullptr, 0, 0,
                                stream_of(a)),
               "iex_gemm_f16_csr");
}
// The same for dense operands.
void gemm(int64_t m, int64_t n, int64_t k, const at::Tensor& a, bool a_mn, const at::Tensor& b, bool b_mn,
          const at::Tensor& out, bool out_t) {
  check_status(iex_gemm_f16(m, n, k, a.data_ptr(), a_mn, a.size(1), b.data_ptr(), b_mn, b.size(1), out.data_ptr(), out_t,
                            out.size(1), 0, 0, stream_of(a)),
               "iex_gemm_f16");
}

// Estimates in microseconds, fitted to measurements on B200.
//   expand   one pass over the CSR arrays and the dense copy, at 5.5 TB/s
//   decode   the block decoder of spmm_tile.cu: a chain of blocks of 512 columns, and per row of a unit its stored
//            positions and its part of a block.  Within -16 and +23 % of 504 measurements (256 to 11008 rows, 512 to 4096
//            columns, 2 to 70 % stored, 64 to 256 tokens), where the choice of spmm_half_way takes 4 % longer than the fastest way on
//            (geometric) average, 1.7 x at worst: short rows of large matrices, whose time on CUDA cores is underestimated
double expand_us(int64_t m, int64_t k, int64_t nnz, int bits) {
  return 2.5 + (2.0 * m * round8(k) + static_cast<double>(nnz) * (2 + bits / 8)) / 5.5e6;
}
double block_decode_us(int64_t m, int64_t k, int64_t n, int64_t nnz) {
  const int64_t step = n <= 64 ? 8 : 16, rows = ((m + 147) / 148 + step - 1) / step * step;  // of an SM's unit
  const double blocks = static_cast<double>((k + 511) / 512), waves = static_cast<double>(std::max<int64_t>(1, (rows + 127) / 128));
  const double wide = std::clamp((n - 128) / 128.0, 0.0, 1.0);
  return 4.85 + 1.35 * wide + waves * blocks * (1.6 + 0.15 * wide) +
         rows * (0.155e-3 * nnz / std::max<int64_t>(m, 1) + (0.006 + 0.014 * wide) * blocks);
}
bool decode_supported(int64_t k, int64_t n, int bits) {
  return n % 64 == 0 && n > 0 && n <= 256 && k % 8 == 0 && k > 0 && (bits == 32 || k <= 65280);
}

enum Mode { kCudaCores = 0, kTensorCores = 1, kAuto = 2 };
enum Way { kRows = 0, kDecode = 1, kExpand = 2, kFewColumns = 3 };

// How an fp16 CSR product [m, k] x [k, n] runs.  On tensor cores the matrix is either decoded tile by tile inside the
// product (tc_fused.cu) or expanded once and multiplied as a dense matrix: the decoder needs no scratch and no second pass,
// the expansion costs the dense copy's traffic but then runs at the dense kernel's rate, for any n.
//   aligned   operands start on 16-byte boundaries
//   eager     scratch may be used; not in a graph constructor's recording, where it would be handed out again before the
//             graph runs, and which knows the registered operators only: there the choice is between kRows and kDecode
Way spmm_half_way(int64_t m, int64_t k, int64_t n, int64_t nnz, int bits, int mode, bool aligned, bool eager) {
  if (mode == kCudaCores || m == 0 || k == 0 || n == 0) return kRows;
  // Up to 8 columns one lane per nonzero (spmm_skinny.cu) instead of one per column: 4096 x 4096 at 10 %, 4 columns 12 us
  // against 21, at 30 % 23 against 27.  Not for rows of less than 96 nonzeros, or 2 % of the columns, which do not pay for
  // a row's start or for x in every block's shared memory (32768 x 256 at 30 %: 17 us against 13; 2048 x 14000 at 0.5 %: 11
  // against 8), and not above one half stored (2048 x 14000 at 90 %: 58 against 52).
  if (mode == kAuto && eager && n <= 8 && nnz >= 96 * m && 50 * nnz >= m * k && 2 * nnz <= m * k &&
      iex_spmm_f16_skinny_supported(k, n))
    return kFewColumns;
  const double expand = eager ? expand_us(m, k, nnz, bits) + iex_gemm_f16_estimate_us(m, n, k, 1, 0) + (n % 8 == 0 ? 0.0 : 2.0)
                              : 1e30;
  const double decode = decode_supported(k, n, bits) && aligned ? block_decode_us(m, k, n, nnz) : 1e30;
  // Tensor cores where the estimates are close: they are good to 10 %, and the walk along the longest row, which only
  // the CUDA cores pay for, is estimated from the average one.
  if (mode == kAuto && 1.15 * iex_spmm_f16_estimate_us(m, k, n, nnz, bits) <= std::min(expand, decode)) return kRows;
  return decode <= expand ? kDecode : kExpand;
}

void check_csr_half(const at::Tensor& b, const at::Tensor& values, const at::Tensor& ro, const at::Tensor& ci,
                    int64_t m) {
  TORCH_CHECK(b.dim() == 2, "b must be [k, n]");
  TORCH_CHECK(values.dim() == 1 && ci.dim() == 1 && values.size(0) == ci.size(0),
              "values and column_indices must be 1-D with nnz entries");
  TORCH_CHECK(ro.dim() == 1 && ro.size(0) == m + 1, "row_offsets must have m + 1 entries");
  check_common({{"b", &b}, {"row_offsets", &ro}, {"values", &values}, {"column_indices", &ci}});
  TORCH_CHECK(b.scalar_type() == at::kHalf && values.scalar_type() == at::kHalf, "b and values must be float16");
  TORCH_CHECK(ro.scalar_type() == at::kInt, "row_offsets must be int32");
  TORCH_CHECK(ci.scalar_type() == at::kShort || ci.scalar_type() == at::kInt, "column_indices must be int16 or int32");
}

// A_csr [m, k] @ b [k, n], fp16
at::Tensor spmm_half(const at::Tensor& b, const at::Tensor& ri, const at::Tensor& values, const at::Tensor& ro,
                     const at::Tensor& ci, int64_t m, int mode) {
  const int64_t k = b.size(0), n = b.size(1), nnz = values.numel();
  const bool aligned = aligned16(b) && aligned16(values) && aligned16(ci);
  const Way way = spmm_half_way(m, k, n, nnz, index_bits(ci), mode, aligned, true);
  if (way == kRows) return spmm_matrix(b, ri, values, ro, ci, m);
  check_csr_half(b, values, ro, ci, m);
  if (way == kDecode) return spmm_tc_half(b, ro, values, ci, m);
  c10::cuda::CUDAGuard guard(b.device());
  maybe_validate(ro, ci, m, k, nullptr, false);
  at::Tensor out = empty(b, {m, n});
  if (way == kFewColumns) {
    const int st = iex_spmm_f16_skinny(m, k, n, nnz, ro.data_ptr<int>(), ci.data_ptr(), index_bits(ci), values.data_ptr(),
                                       b.data_ptr(), n, 1, out.data_ptr(), n, 1, stream_of(b));
    if (st == 0) return out;
    // pairs of nonzeros are loaded together; a matrix that is not aligned for that is expanded
    TORCH_CHECK(st == IEX_ERR_UNSUPPORTED, "iex_spmm_f16_skinny failed with status ", st, ": ", iex_error_string(st));
  }
  gemm(m, n, k, expand(values, ro, ci, m, k), false, tma_rows(b), true, out, false, Stored{0, ro, ci, values});
  return out;
}

// ------------------------------------------------------------------------------------- MySpMM

struct SpmmArgs {
  at::Tensor ri, ro, ci;                 // the pattern
  at::Tensor ri_t, ro_t, ci_t, perm;     // the transposed pattern (undefined without transp_info)
  int64_t m = 0;
  int mode = kCudaCores;
};

at::Tensor spmm_forward(const at::Tensor& b, const at::Tensor& values, const SpmmArgs& p) {
  if (values.scalar_type() == at::kFloat)
    return spmm_matrix(b, p.ri, values, p.ro, p.ci, p.m);
  return spmm_half(b, p.ri, values, p.ro, p.ci, p.m, p.mode);
}

at::Tensor grad_of_values(const at::Tensor& grad, const at::Tensor& b, const at::Tensor& values, const SpmmArgs& p) {
  if (grad.scalar_type() != at::kHalf)
    return sddmm_matrix(grad, b, p.ri, p.ro, p.ci.scalar_type() == at::kInt ? p.ci : p.ci.to(at::kInt));
  const int64_t m = grad.size(0), n = grad.size(1), k = b.size(0), nnz = values.numel();
  if (p.mode != kCudaCores && b.scalar_type() == at::kHalf && m > 0 && n > 0 && k > 0 && nnz > 0) {
    // every product of the dense matrix, of which the stored positions are kept, against one
    // gathered row of b per stored position
    // (bytes, and a chain of L2 latencies for every 256 or, unaligned, 32 columns)
    const double dense = iex_gemm_f16_estimate_us(m, k, n, 0, 0) + 3.0 + 6.0e-6 * nnz + (n % 8 == 0 ? 0.0 : 4.0);
    const double chain = n % 8 == 0 ? 4.0 * ((n + 255) / 256) : 3.5 * ((n + 31) / 32);
    const double cores = 2.0 + 0.19e-6 * 2.0 * nnz * n + chain;
    if (dense < cores) {
      c10::cuda::CUDAGuard guard(grad.device());
      at::Tensor all = empty(grad, {m, round8(k)});
      gemm(m, k, n, tma_rows(grad), false, tma_rows(b), false, all, false);
      at::Tensor out = empty(grad, {nnz});
      check_status(iex_csr_sample_f16(m, k, all.size(1), p.ro.data_ptr<int>(), p.ci.data_ptr(), index_bits(p.ci),
                                      all.data_ptr(), out.data_ptr(), stream_of(grad)),
                   "iex_csr_sample_f16");
      return out;
    }
  }
  return sddmm_matrix(grad, b.scalar_type() == at::kHalf ? b : b.to(at::kHalf), p.ri, p.ro, p.ci);
}

at::Tensor grad_of_b(const at::Tensor& grad, const at::Tensor& b, const at::Tensor& values, const SpmmArgs& p) {
  const int64_t m = grad.size(0), n = grad.size(1), k = b.size(0), nnz = values.numel();
  const bool perm_ok = p.perm.scalar_type() == at::kLong && p.perm.is_contiguous() && values.is_contiguous() &&
                       p.perm.dim() == 1 && p.perm.numel() == nnz && p.perm.device() == values.device();
  if (p.mode != kCudaCores && grad.scalar_type() == at::kHalf && values.scalar_type() == at::kHalf && m > 0 && n > 0 &&
      k > 0 && nnz > 0 && perm_ok && p.ro_t.scalar_type() == at::kInt && p.ro_t.is_contiguous() && p.ro_t.numel() == k + 1 &&
      p.ci_t.is_contiguous() && p.ci_t.numel() == nnz && p.ro_t.device() == values.device() &&
      p.ci_t.device() == values.device() && (p.ci_t.scalar_type() == at::kShort || p.ci_t.scalar_type() == at::kInt)) {
    // the expanded matrix read with its row dimension as the contraction; the transposed pattern is for outputs that
    // have to be summed again
    const double dense = expand_us(m, k, nnz, index_bits(p.ci)) + iex_gemm_f16_estimate_us(k, n, m, 1, 0);
    const double cores = iex_spmm_f16_estimate_us(k, m, n, nnz, index_bits(p.ci)) + 5.0;
    if (dense < cores) {
      c10::cuda::CUDAGuard guard(grad.device());
      at::Tensor out = empty(grad, {k, n});
      gemm(k, n, m, expand(values, p.ro, p.ci, m, k), true, tma_rows(grad), true, out, false,
           Stored{0, p.ro_t, p.ci_t, values, &p.perm});
      return out;
    }
  }
  // transposing the pattern is bookkeeping done once (get_transpose_info); the values follow it
  at::Tensor values_t;
  if (perm_ok && (values.scalar_type() == at::kFloat || values.scalar_type() == at::kHalf)) {
    c10::cuda::CUDAGuard guard(values.device());
    values_t = empty(values, {nnz});
    check_status(iex_gather_values(nnz, values.element_size(), values.data_ptr(),
                                   reinterpret_cast<const long long*>(p.perm.data_ptr<int64_t>()), values_t.data_ptr(),
                                   stream_of(values)),
                 "iex_gather_values");
  } else {
    values_t = values.index({p.perm});
  }
  return spmm_matrix(grad, p.ri_t, values_t, p.ro_t, p.ci_t, k);
}

struct MySpMMBackward : public Node {
  // b, values and the pattern: hooks on saved tensors see all of them, and changing one in place before the backward
  // pass is an error
  std::array<SavedVariable, 9> saved_;
  int64_t m_ = 0;
  int mode_ = kCudaCores;
  std::string name() const override { return "MySpMMBackward"; }
  void release_variables() override {
    std::lock_guard<std::mutex> lock(mutex_);
    for (SavedVariable& v : saved_) v.reset_data();
  }
  variable_list apply(variable_list&& grads) override {
    std::lock_guard<std::mutex> lock(mutex_);
    variable_list out(2);
    if (!grads[0].defined()) return out;
    std::array<at::Tensor, 9> t;
    for (int i = 0; i < 9; ++i) t[i] = saved_[i].unpack();
    const SpmmArgs args{t[2], t[3], t[4], t[5], t[6], t[7], t[8], m_, mode_};
    {
      at::AutoDispatchBelowADInplaceOrView below;
      const at::Tensor grad = grads[0].contiguous();
      if (task_should_compute_output(1)) out[1] = grad_of_values(grad, t[0], t[1], args);
      if (task_should_compute_output(0)) out[0] = grad_of_b(grad, t[0], t[1], args);
    }
    return once_differentiable(std::move(out), grads[0], t[0], t[1], "MySpMM");
  }
};

// MySpMM.run without a graph constructor; nothing for calls that have to go through the dispatcher.  `transp` is
// (row_indices_t, row_offsets_t, column_indices_t, perm) or empty; without it b must not require a gradient.
std::optional<at::Tensor> myspmm(const at::Tensor& b_in, const at::Tensor& ri, const at::Tensor& values, const at::Tensor& ro,
                                 const at::Tensor& ci, int64_t m, const std::vector<at::Tensor>& transp, int mode) {
  if (!plain({&b_in, &values, &ri, &ro, &ci})) return std::nullopt;
  SpmmArgs p;
  p.ri = ri;
  p.ro = ro;
  p.ci = ci;
  p.m = m;
  p.mode = mode;
  if (transp.size() == 4) {
    p.ri_t = transp[0];
    p.ro_t = transp[1];
    p.ci_t = transp[2];
    p.perm = transp[3];
  }
  const bool needs_grad = torch::autograd::compute_requires_grad(b_in, values);
  at::Tensor b = b_in.contiguous();
  at::Tensor out;
  {
    at::AutoDispatchBelowADInplaceOrView below;
    out = spmm_forward(b, values, p);
  }
  if (needs_grad) {
    auto node = std::shared_ptr<MySpMMBackward>(new MySpMMBackward(), torch::autograd::deleteNode);
    node->set_next_edges(torch::autograd::collect_next_edges(b, values));
    const std::array<const at::Tensor*, 9> saved = {&b, &values, &p.ri, &p.ro, &p.ci, &p.ri_t, &p.ro_t, &p.ci_t, &p.perm};
    for (int i = 0; i < 9; ++i) node->saved_[i] = SavedVariable(*saved[i], false);
    node->m_ = m;
    node->mode_ = mode;
    torch::autograd::set_history(out, node);
  }
  return out;
}

// ------------------------------------------------------------------------------------ MyLinear

struct MyLinearBackward : public Node {
  SavedVariable input_, weight_;
  std::string name() const override { return "MyLinearBackward"; }
  void release_variables() override {
    std::lock_guard<std::mutex> lock(mutex_);
    input_.reset_data();
    weight_.reset_data();
  }
  variable_list apply(variable_list&& grads) override {
    std::lock_guard<std::mutex> lock(mutex_);
    variable_list out(2);
    if (!grads[0].defined()) return out;
    const at::Tensor input = input_.unpack(), weight = weight_.unpack();
    const at::Tensor& grad = grads[0];
    const bool own = grad.scalar_type() == at::kHalf && grad.is_cuda() && weight.size(0) % 8 == 0 &&
                     weight.size(1) % 8 == 0;
    if (own) {
      {
        at::AutoDispatchBelowADInplaceOrView below;
        const at::Tensor g = grad.contiguous();
        if (task_should_compute_output(0)) out[0] = linear_fp16_dgrad(g, weight);
        if (task_should_compute_output(1)) out[1] = linear_fp16_wgrad(g, input);
      }
      return once_differentiable(std::move(out), grad, input, weight, "MyLinear's tensor-core path");
    } else {  // differentiable products
      if (task_should_compute_output(0)) out[0] = grad.mm(weight);
      if (task_should_compute_output(1)) out[1] = grad.t().mm(input);
    }
    return out;
  }
};

// MyLinear.run without a graph constructor; nothing for operands the tensor-core kernel does not
// take (tc_linear_eligible in layers_and_funcs/torch.py) and for calls that have to go through the dispatcher.
std::optional<at::Tensor> mylinear(const at::Tensor& input, const at::Tensor& weight) {
  if (!plain({&input, &weight})) return std::nullopt;
  const bool eligible = input.is_cuda() && weight.is_cuda() && input.scalar_type() == at::kHalf &&
                        weight.scalar_type() == at::kHalf && input.dim() == 2 && weight.dim() == 2 &&
                        input.size(0) > 0 && input.size(1) % 8 == 0 && input.is_contiguous() &&
                        weight.is_contiguous() && aligned16(input) && aligned16(weight);
  if (!eligible) return std::nullopt;
  at::Tensor out;
  {
    at::AutoDispatchBelowADInplaceOrView below;
    out = linear_fp16(input, weight);
  }
  if (torch::autograd::compute_requires_grad(input, weight)) {
    auto node = std::shared_ptr<MyLinearBackward>(new MyLinearBackward(), torch::autograd::deleteNode);
    node->set_next_edges(torch::autograd::collect_next_edges(input, weight));
    node->input_ = SavedVariable(input, false);
    node->weight_ = SavedVariable(weight, false);
    torch::autograd::set_history(out, node);
  }
  return out;
}

// --------------------------------------------------------------------------- inference layers

// The dense fp16 copy [m, k] of a layer's CSR weight.
at::Tensor expand_weight(const at::Tensor& values, const at::Tensor& ro, const at::Tensor& ci, int64_t m, int64_t k) {
  check_common({{"row_offsets", &ro}, {"values", &values}, {"column_indices", &ci}});
  TORCH_CHECK(values.scalar_type() == at::kHalf && ro.scalar_type() == at::kInt && ro.numel() == m + 1, "not an fp16 CSR matrix");
  TORCH_CHECK(k % 8 == 0, "in_features must be a multiple of 8");
  c10::cuda::CUDAGuard guard(values.device());
  return expand(values, ro, ci, m, k);
}

// The dense copy a layer keeps of its CSR weight (pytorch/utils.py: DenseCopy, which says what it follows).  Asked for on
// every inference call, so the comparison is done here: 0.3 us, 3 us in Python.
class KeptCopy {
 public:
  KeptCopy(int64_t m, int64_t k, double density) : m_(m), k_(k), density_(density) {}
  int64_t rows() const { return m_; }
  int64_t columns() const { return k_; }
  void reset() {
    weight_.reset();
    held_ = {};
  }

  // Called with the interpreter lock held, which is what makes the members' update atomic.
  std::optional<at::Tensor> current(const at::Tensor& values, const at::Tensor& ro, const at::Tensor& ci) {
    if (!plain({&values, &ro, &ci}) || !values.is_cuda() || values.scalar_type() != at::kHalf || k_ % 8 != 0 || m_ == 0 ||
        static_cast<double>(values.numel()) < density_ * m_ * k_ || values.is_inference() || ro.is_inference() ||
        ci.is_inference() || iex_stream_is_capturing(stream_of(values)))
      return std::nullopt;
    const std::array<const at::Tensor*, 3> now = {&values, &ro, &ci};
    bool same = weight_.has_value();
    for (int i = 0; i < 3 && same; ++i) same = held_[i].is(*now[i]);
    if (same) return weight_;
    std::array<Held, 3> held = {Held(values), Held(ro), Held(ci)};
    at::Tensor weight = expand_weight(values, ro, ci, m_, k_);
    {
      pybind11::gil_scoped_release unlocked;
      at::cuda::getCurrentCUDAStream(values.get_device()).synchronize();
    }
    held_ = std::move(held);
    weight_ = std::move(weight);
    return weight_;
  }

 private:
  struct Held {
    at::Tensor tensor;      // the object itself ...
    c10::Storage storage;   // ... and what it lay in, so that its address cannot come back as something else
    const void* data = nullptr;
    int64_t count = 0, version = 0;
    Held() = default;
    explicit Held(const at::Tensor& t)
        : tensor(t), storage(t.storage()), data(t.data_ptr()), count(t.numel()), version(t._version()) {}
    bool is(const at::Tensor& t) const {
      return tensor.is_same(t) && data == t.data_ptr() && count == t.numel() && version == t._version();
    }
  };
  const int64_t m_, k_;
  const double density_;
  std::array<Held, 3> held_;
  std::optional<at::Tensor> weight_;
};

// The two branches of a sparse || dense layer with both weights dense: x [k, n] ->
// (weight0 @ x [m0, n], (weight1 @ x)^T [n, m1]) in one launch.  weight0 is the layer's dense copy of a CSR matrix, `stored`
// (values, row_offsets, column_indices) or, for two dense matrices, nothing.
std::tuple<at::Tensor, at::Tensor> linear_pair(const at::Tensor& x, const at::Tensor& weight0, const at::Tensor& weight1,
                                               const std::vector<at::Tensor>& stored) {
  check_common({{"x", &x}, {"weight0", &weight0}, {"weight1", &weight1}});
  TORCH_CHECK(stored.empty() || stored.size() == 3, "stored must be (values, row_offsets, column_indices)");
  const int64_t k = x.size(0), n = x.size(1), m0 = weight0.size(0), m1 = weight1.size(0);
  TORCH_CHECK(weight0.size(1) == k && weight1.size(1) == k, "weights must be [rows, k]");
  c10::cuda::CUDAGuard guard(x.device());
  at::Tensor out0 = empty(x, {m0, n}), out1 = empty(x, {n, m1});
  mark_stream(weight0);
  const int* ro = nullptr;
  const void *ci = nullptr, *values = nullptr;
  int bits = 16;
  if (!stored.empty()) {
    check_common({{"values", &stored[0]}, {"row_offsets", &stored[1]}, {"column_indices", &stored[2]}});
    TORCH_CHECK(stored[0].scalar_type() == at::kHalf && stored[0].device() == x.device(), "values must be float16 on x's device");
    TORCH_CHECK(stored[1].scalar_type() == at::kInt && stored[1].numel() == m0 + 1, "row_offsets must be int32 with m + 1 entries");
    TORCH_CHECK(stored[2].scalar_type() == at::kShort || stored[2].scalar_type() == at::kInt, "column_indices must be int16 or int32");
    values = stored[0].data_ptr();
    ro = stored[1].data_ptr<int>();
    ci = stored[2].data_ptr();
    bits = index_bits(stored[2]);
  }
  check_status(iex_linear_pair_f16_csr(m0, m1, k, n, weight0.data_ptr(), ro, ci, bits, values, weight1.data_ptr(), x.data_ptr(), 0,
                                       out0.data_ptr(), 0, out1.data_ptr(), 1, stream_of(x)),
               "iex_linear_pair_f16_csr");
  return {out0, out1};
}

// Whether 1 or 2 tokens take the CSR arrays (spmm_skinny.cu) although there is a dense copy, whose product is estimated at
// `copy_us`.  A call has 7.8 us of host time either way and 0.4 more with the copy (its checks), so that a kernel below that is as
// good as any.  The kernel takes 2.5 us and 1.05 ns a nonzero for one token, for two up to 4 us and 2.2 ns.  Measured (us a call with
// the CSR arrays, with the copy): 1024 x 1024, half stored, 1 token 7.8, 8.2; 4096 x 2048 30 % 7.7, 8.1; 4096 x 4096 30 % 2 tokens
// 19 (the kernel 15.8), 8.2.
bool skinny_first(int64_t tokens, int64_t nnz, double copy_us) {
  const double skinny_us = tokens == 1 ? 2.5 + 1.05e-6 * nnz : 4.0 + 2.2e-6 * nnz;
  return skinny_us <= std::max(7.8, copy_us);
}

// SparseLinear without gradients: x [tokens, k] @ W_csr^T -> [tokens, m], W_csr [m, k].
//   1 or 2 tokens    CUDA cores, the CSR arrays read once (spmm_skinny.cu), without a dense copy or where it is no slower
//   with `dense`     the layer's dense copy of W: for a handful of tokens linear_few.cu, else the dense GEMM
//   up to 256        block decoder on tensor cores (spmm_tile.cu), unless ...
//   otherwise        ... expanding W for the dense GEMM is estimated faster (many tokens)
// `settled`: the dense copy was complete before the call and nothing writes it (a KeptCopy).
// All read x as it lies and write [tokens, m]: no transposed copies of either.  Nothing for calls that have to go through the
// dispatcher.
std::optional<at::Tensor> sparse_linear(const at::Tensor& x, const at::Tensor& values, const at::Tensor& ro, const at::Tensor& ci,
                         int64_t m, int64_t k, const std::optional<at::Tensor>& dense_weight, bool settled) {
  if (!plain({&x, &values, &ro, &ci})) return std::nullopt;
  TORCH_CHECK(x.dim() == 2 && x.is_contiguous(), "x must be a contiguous [tokens, in_features] matrix");
  TORCH_CHECK(x.size(1) == k, "x has ", x.size(1), " columns, the weight ", k);
  TORCH_CHECK(values.dim() == 1 && ci.dim() == 1 && values.size(0) == ci.size(0),
              "values and column_indices must be 1-D with nnz entries");
  check_common({{"x", &x}, {"row_offsets", &ro}, {"values", &values}, {"column_indices", &ci}});
  TORCH_CHECK(x.scalar_type() == at::kHalf && values.scalar_type() == at::kHalf, "x and values must be float16");
  TORCH_CHECK(ro.scalar_type() == at::kInt && ro.numel() == m + 1, "row_offsets must be int32 with m + 1 entries");
  TORCH_CHECK(ci.scalar_type() == at::kShort || ci.scalar_type() == at::kInt, "column_indices must be int16 or int32");
  const int64_t tokens = x.size(0);
  c10::cuda::CUDAGuard guard(x.device());
  maybe_validate(ro, ci, m, k, nullptr, false);
  at::Tensor out = empty(x, {tokens, m});
  if (tokens == 0 || m == 0) return out;
  const int64_t nnz = values.numel();
  const double gemm_us = std::min(m % 8 == 0 ? iex_gemm_f16_estimate_us(m, tokens, k, 0, 1) : 1e30,
                                  iex_gemm_f16_estimate_us(tokens, m, k, 0, 0));
  const double few_us = dense_weight.has_value() ? iex_linear_f16_few_estimate_us(tokens, k, m, settled) : 1e30;
  if (tokens <= 2 && iex_spmm_f16_skinny_supported(k, tokens) &&
      (!dense_weight.has_value() || skinny_first(tokens, nnz, std::min(gemm_us, few_us)))) {
    const int st = iex_spmm_f16_skinny(m, k, tokens, nnz, ro.data_ptr<int>(), ci.data_ptr(), index_bits(ci),
                                       values.data_ptr(), x.data_ptr(), 1, k, out.data_ptr(), 1, m, stream_of(x));
    if (st == 0) return out;
    // pairs of nonzeros are loaded together; a matrix that is not aligned for that takes the ways below
    TORCH_CHECK(st == IEX_ERR_UNSUPPORTED, "iex_spmm_f16_skinny failed with status ", st, ": ", iex_error_string(st));
  }
  at::Tensor dense;
  if (dense_weight.has_value()) {
    dense = *dense_weight;
    TORCH_CHECK(dense.dim() == 2 && dense.size(0) == m && dense.size(1) == k && k % 8 == 0 && dense.scalar_type() == at::kHalf &&
                    dense.is_contiguous() && dense.device() == x.device(),
                "dense copy of another shape");
    mark_stream(dense);
  } else {
    // a launch and a buffer more than the decoder: 13 us a call from the host, 10 with the decoder, where kernels are short
    const double as_dense = std::max(13.0, expand_us(m, k, nnz, index_bits(ci)) + gemm_us);
    if (tokens <= 256 && k % 8 == 0 && block_decode_us(m, k, tokens, nnz) < as_dense) {
      const int st = iex_spmm_linear_f16_tile(m, 0, k, tokens, nnz, ro.data_ptr<int>(), ci.data_ptr(), index_bits(ci),
                                              values.data_ptr(), nullptr, x.data_ptr(), 1, nullptr, out.data_ptr(), 1,
                                              nullptr, 0, stream_of(x));
      if (st == 0) return out;
      TORCH_CHECK(st == IEX_ERR_UNSUPPORTED, "iex_spmm_linear_f16_tile failed with status ", st, ": ", iex_error_string(st));
    }
    dense = expand(values, ro, ci, m, k);
  }
  const at::Tensor xp = tma_rows(x);
  if (1.15 * few_us <= gemm_us) {
    check_status(iex_linear_f16_few(tokens, k, m, xp.data_ptr(), dense.data_ptr(), out.data_ptr(), settled ? 1 : 0,
                                    ro.data_ptr<int>(), ci.data_ptr(), index_bits(ci), values.data_ptr(), stream_of(x)),
                 "iex_linear_f16_few");
    return out;
  }
  if (m % 8 == 0 && iex_gemm_f16_estimate_us(m, tokens, k, 0, 1) <= iex_gemm_f16_estimate_us(tokens, m, k, 0, 0))
    gemm(m, tokens, k, dense, false, xp, false, out, true, Stored{0, ro, ci, values});
  else
    gemm(tokens, m, k, xp, false, dense, false, out, false, Stored{1, ro, ci, values});
  return out;
}

// Masked attention over heads (pytorch/attention.py): the mask's bits, and the chain in one launch.
at::Tensor attention_plan(const at::Tensor& ro, const at::Tensor& ci, int64_t m, int64_t n) {
  check_common({{"row_offsets", &ro}, {"column_indices", &ci}});
  TORCH_CHECK(ro.scalar_type() == at::kInt && ci.scalar_type() == at::kInt && ro.numel() == m + 1, "not an int32 CSR pattern");
  c10::cuda::CUDAGuard guard(ro.device());
  const size_t bytes = iex_attention_plan_bytes(m, n);
  at::Tensor plan = empty_bytes(ro, bytes);
  check_status(iex_attention_plan_build(m, n, ro.data_ptr<int>(), ci.data_ptr<int>(), plan.data_ptr(), bytes, stream_of(ro)),
               "iex_attention_plan_build");
  return plan;
}

// q [heads, m, d], k [heads, n, d], v [heads, n, dv] -> [heads, m, dv]; nothing for shapes the kernel does not take or is
// not the faster way for
std::optional<at::Tensor> attention(const at::Tensor& q, const at::Tensor& k, const at::Tensor& v, const at::Tensor& plan,
                                    const at::Tensor& ro, const at::Tensor& ci) {
  check_common({{"q", &q}, {"k", &k}, {"v", &v}, {"plan", &plan}, {"row_offsets", &ro}, {"column_indices", &ci}});
  TORCH_CHECK(q.dim() == 3 && k.dim() == 3 && v.dim() == 3, "q, k and v must be [heads, rows, columns]");
  TORCH_CHECK(q.scalar_type() == at::kFloat && k.scalar_type() == at::kFloat && v.scalar_type() == at::kFloat,
              "q, k and v must be float32");
  TORCH_CHECK(k.size(0) == q.size(0) && v.size(0) >= q.size(0), "k and v have fewer heads than q");
  TORCH_CHECK(k.size(2) == q.size(2) && v.size(1) == k.size(1), "q and k disagree on d, or k and v on n");
  const int64_t heads = q.size(0), m = q.size(1), d = q.size(2), n = k.size(1), dv = v.size(2);
  if (!iex_attention_f32_prefers(heads, m, n, d, dv, ci.numel()) || !aligned16(q) || !aligned16(k) || !aligned16(v)) return std::nullopt;
  TORCH_CHECK(ro.scalar_type() == at::kInt && ci.scalar_type() == at::kInt, "row_offsets and column_indices must be int32");
  TORCH_CHECK(ro.numel() == m + 1 && static_cast<size_t>(plan.nbytes()) >= iex_attention_plan_bytes(m, n), "plan of another mask");
  c10::cuda::CUDAGuard guard(q.device());
  at::Tensor out = empty(q, {heads, m, dv});
  const size_t bytes = iex_attention_workspace_bytes(heads, m, n, d, dv);
  at::Tensor workspace = empty_bytes(q, bytes);
  check_status(iex_attention_f32(heads, m, n, d, dv, plan.data_ptr(), ro.data_ptr<int>(), ci.data_ptr<int>(),
                                 q.data_ptr<float>(), k.data_ptr<float>(), v.data_ptr<float>(), out.data_ptr<float>(),
                                 workspace.data_ptr(), bytes, stream_of(q)),
               "iex_attention_f32");
  return out;
}

// ReluSparseDownProj without a gather of its own: CSR activations [tokens, k] (expanded into
// `dense`) times weight [n, k]^T into `out`.
void ffn_down(const at::Tensor& values, const at::Tensor& ro, const at::Tensor& ci, const at::Tensor& weight,
              const at::Tensor& dense, const at::Tensor& out) {
  check_common({{"values", &values}, {"row_offsets", &ro}, {"column_indices", &ci}, {"weight", &weight},
                {"dense", &dense}, {"out", &out}});
  const int64_t tokens = dense.size(0), k = dense.size(1), n = weight.size(0);
  TORCH_CHECK(ro.scalar_type() == at::kInt && ro.numel() == tokens + 1, "row_offsets must be int32 with tokens + 1 entries");
  c10::cuda::CUDAGuard guard(values.device());
  check_status(iex_csr_to_dense_f16(tokens, k, ro.data_ptr<int>(), ci.data_ptr(), index_bits(ci), values.data_ptr(),
                                    dense.data_ptr(), stream_of(values)),
               "iex_csr_to_dense_f16");
  check_status(iex_linear_f16_any(tokens, k, n, dense.data_ptr(), weight.data_ptr(), out.data_ptr(), stream_of(values)),
               "iex_linear_f16_any");
}

// relu(hidden [tokens, k]) @ weight [n, k]^T
at::Tensor relu_down_proj(const at::Tensor& hidden, const at::Tensor& weight) {
  check_common({{"hidden", &hidden}, {"weight", &weight}});
  TORCH_CHECK(hidden.scalar_type() == at::kHalf && weight.scalar_type() == at::kHalf, "hidden and weight must be float16");
  const int64_t tokens = hidden.size(0), k = hidden.size(1), n = weight.size(0);
  c10::cuda::CUDAGuard guard(hidden.device());
  at::Tensor out = empty(hidden, {tokens, n});
  if (tokens == 0 || n == 0) return out;
  at::Tensor act = empty(hidden, {tokens, k});
  check_status(iex_relu_f16(tokens * k, hidden.data_ptr(), act.data_ptr(), stream_of(hidden)), "iex_relu_f16");
  check_status(iex_linear_f16_any(tokens, k, n, act.data_ptr(), weight.data_ptr(), out.data_ptr(), stream_of(hidden)),
               "iex_linear_f16_any");
  return out;
}

}  // namespace
}  // namespace iex_torch

PYBIND11_MODULE(iex_torch_ext, mod) {
  mod.def("myspmm", &iex_torch::myspmm);
  mod.def("spmm_half_way", [](int64_t m, int64_t k, int64_t n, int64_t nnz, int bits, bool eager) {
    return static_cast<int>(iex_torch::spmm_half_way(m, k, n, nnz, bits, iex_torch::kAuto, true, eager));
  });
  mod.def("skinny_first", &iex_torch::skinny_first);
  mod.def("mylinear", &iex_torch::mylinear);
  mod.def("sparse_linear", &iex_torch::sparse_linear, pybind11::arg("x"), pybind11::arg("values"), pybind11::arg("row_offsets"),
          pybind11::arg("column_indices"), pybind11::arg("out_features"), pybind11::arg("in_features"),
          pybind11::arg("dense_weight"), pybind11::arg("settled") = false);
  mod.def("expand_weight", &iex_torch::expand_weight);
  pybind11::class_<iex_torch::KeptCopy>(mod, "KeptCopy")
      .def(pybind11::init<int64_t, int64_t, double>())
      .def_property_readonly("m", &iex_torch::KeptCopy::rows)
      .def_property_readonly("k", &iex_torch::KeptCopy::columns)
      .def("reset", &iex_torch::KeptCopy::reset)
      .def("current", &iex_torch::KeptCopy::current, pybind11::arg("values"), pybind11::arg("row_offsets"),
           pybind11::arg("column_indices"));
  mod.def("stream_capturing", [](const at::Tensor& t) { return iex_stream_is_capturing(iex_torch::stream_of(t)) != 0; });
  mod.def("plain", [](const at::Tensor& a, const at::Tensor& b, const at::Tensor& c) { return iex_torch::plain({&a, &b, &c}); });
  mod.def("linear_pair", &iex_torch::linear_pair, pybind11::arg("x"), pybind11::arg("weight0"), pybind11::arg("weight1"),
          pybind11::arg("stored") = std::vector<at::Tensor>());
  mod.def("attention_plan", &iex_torch::attention_plan);
  mod.def("attention", &iex_torch::attention);
  mod.def("ffn_down", &iex_torch::ffn_down);
  mod.def("relu_down_proj", &iex_torch::relu_down_proj);
  mod.def("fused_spmm_linear_half", &iex_torch::fused_spmm_linear_half);
}

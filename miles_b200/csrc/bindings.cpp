// PyTorch bindings for the sm_100a kernels. Only this file includes the PyTorch headers; every
// kernel lives in a plain CUDA translation unit with a C++ launcher declared in a header.
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/extension.h>

#include "binding_helpers.h"
#include "gemm.h"
#include "launchers.h"

namespace {

using namespace mb_bind;

// a: [rows, K] rows grouped in 128-row tiles; b: [G, N, K] (K-major) or [G, K, N] (MN-major).
void grouped_gemm_rows(const at::Tensor& a, const at::Tensor& b, at::Tensor& c, const at::Tensor& tile_group,
                       const at::Tensor& num_m_tiles, bool b_mn, bool accumulate, int64_t block_n,
                       const c10::optional<at::Tensor>& status, const c10::optional<at::Tensor>& row_ptrs,
                       const c10::optional<at::Tensor>& sig_ctrl, const std::vector<int64_t>& sig_flags, int64_t sig_me) {
  check_bf16_2d(a, "a");
  TORCH_CHECK(b.is_cuda() && b.scalar_type() == at::kBFloat16 && b.dim() == 3 && b.is_contiguous(),
              "b must be a contiguous 3-D bf16 tensor");
  TORCH_CHECK(tile_group.scalar_type() == at::kInt && num_m_tiles.scalar_type() == at::kInt, "tile maps must be int32");
  const c10::cuda::CUDAGuard guard(a.device());
  mb::GemmProblem p{};
  p.mode = mb::GEMM_GROUPED_ROWS;
  p.num_groups = b.size(0);
  p.M = a.size(0);
  p.K = a.size(1);
  p.N = b_mn ? b.size(2) : b.size(1);
  TORCH_CHECK((b_mn ? b.size(1) : b.size(2)) == p.K, "contraction extents differ");
  TORCH_CHECK(tile_group.dim() == 2 && tile_group.size(1) == 4 && num_m_tiles.numel() >= 1, "tile maps must be [tiles, 4] and [2]");
  p.max_tiles = tile_group.size(0);
  TORCH_CHECK(c.dim() == 2 && c.size(0) == p.M && c.size(1) == p.N, "bad output shape");
  p.a = operand(a, false);
  at::Tensor b2 = b.view({b.size(0) * b.size(1), b.size(2)});
  p.b = operand(b2, b_mn);
  fill_out(p, c);
  p.ldc = c.stride(0);
  p.accumulate = accumulate;
  p.tile_group = tile_group.data_ptr<int>();
  p.num_m_tiles = num_m_tiles.data_ptr<int>();
  p.status = status_ptr(status);
  p.block_n = static_cast<int>(block_n);
  if (row_ptrs.has_value()) {  // scattered output: the epilogue stores each row at its own (possibly remote) address
    TORCH_CHECK(row_ptrs->is_cuda() && row_ptrs->scalar_type() == at::kLong && row_ptrs->numel() >= p.M, "row_ptrs must be int64 [M]");
    p.row_ptrs = reinterpret_cast<const unsigned long long*>(row_ptrs->data_ptr<int64_t>());
    if (sig_ctrl.has_value()) {
      TORCH_CHECK(sig_ctrl->scalar_type() == at::kLong && sig_ctrl->numel() >= 6 && sig_flags.size() <= 8, "bad signal arguments");
      p.sig_ctrl = reinterpret_cast<unsigned long long*>(sig_ctrl->data_ptr<int64_t>());
      for (size_t i = 0; i < sig_flags.size(); ++i) p.sig_flags[i] = reinterpret_cast<unsigned long long*>(sig_flags[i]);
      p.sig_nranks = static_cast<int>(sig_flags.size());
      p.sig_me = static_cast<int>(sig_me);
    }
  }
  TORCH_CHECK(mb::gemm_bf16_launch(p, cur_stream()) == 0, "grouped_gemm_rows: ", mb::gemm_last_error());
}

// (log-probabilities of the targets, entropies, log-sum-exps, means) of softmax(h . w^T * inv_temp), all fp32 [T]; logits [T, V] fp32 or none.
std::vector<at::Tensor> score_rows(const at::Tensor& h, const at::Tensor& w, const at::Tensor& targets, double inv_temp,
                                   const c10::optional<at::Tensor>& logits, const c10::optional<at::Tensor>& status, int64_t pair) {
  check_bf16_2d(h, "h");
  check_bf16_2d(w, "w");
  CHECK_I32(targets);
  const int64_t T = h.size(0), V = w.size(0);
  TORCH_CHECK(h.size(1) == w.size(1) && targets.numel() == T, "shapes differ");
  const c10::cuda::CUDAGuard guard(h.device());
  auto o = h.options().dtype(at::kFloat);
  at::Tensor lp = at::empty({T}, o), ent = at::empty({T}, o), lse = at::empty({T}, o), px = at::empty({T}, o), tgt = at::empty({T}, o);
  if (T == 0) return {lp, ent, lse, px};
  at::Tensor part = at::empty({(V + 127) / 128, T, 4}, o);
  mb::GemmProblem p{};
  p.mode = mb::GEMM_DENSE;
  p.M = T;
  p.N = V;
  p.K = h.size(1);
  p.a = operand(h, false);
  p.b = operand(w, false);
  p.out_fp32 = true;
  if (logits.has_value()) {
    TORCH_CHECK(logits->scalar_type() == at::kFloat && logits->dim() == 2 && logits->size(0) == T && logits->size(1) == V, "logits must be fp32 [T, V]");
    fill_out(p, *logits);
    p.ldc = logits->stride(0);
  }
  p.score_part = part.data_ptr<float>();
  p.targets = targets.data_ptr<int>();
  p.score_target = tgt.data_ptr<float>();
  p.inv_temp = inv_temp;
  p.status = status_ptr(status);
  p.pair = static_cast<int>(pair);
  TORCH_CHECK(mb::gemm_bf16_launch(p, cur_stream()) == 0, "score_rows: ", mb::gemm_last_error());
  mb::logprob_entropy_merge(part.data_ptr<float>(), tgt.data_ptr<float>(), targets.data_ptr<int>(), lp.data_ptr<float>(), ent.data_ptr<float>(),
                            lse.data_ptr<float>(), px.data_ptr<float>(), T, V, cur_stream());
  return {lp, ent, lse, px};
}

// act [rows, I] = silu(gate) * up for gate | up = a . b[g]^T, b [G, 2I, K] (or [2I, K] without tiles: one product over all rows);
// gu [rows, 2I] or none: gate | up too.
void gated_gemm(const at::Tensor& a, const at::Tensor& b, at::Tensor& act, const c10::optional<at::Tensor>& gu,
                const c10::optional<at::Tensor>& tile_group, const c10::optional<at::Tensor>& num_m_tiles, const c10::optional<at::Tensor>& status,
                int64_t pair) {
  check_bf16_2d(a, "a");
  check_bf16_2d(act, "act");
  TORCH_CHECK(b.is_cuda() && b.scalar_type() == at::kBFloat16 && b.is_contiguous() && b.dim() == (tile_group.has_value() ? 3 : 2),
              "b must be contiguous bf16, [G, 2I, K] with tiles and [2I, K] without");
  TORCH_CHECK(tile_group.has_value() == num_m_tiles.has_value(), "tiles and their number go together");
  const c10::cuda::CUDAGuard guard(a.device());
  mb::GemmProblem p{};
  p.mode = tile_group.has_value() ? mb::GEMM_GROUPED_ROWS : mb::GEMM_DENSE;
  p.num_groups = tile_group.has_value() ? b.size(0) : 1;
  p.M = a.size(0);
  p.K = a.size(1);
  p.N = b.size(-2);
  TORCH_CHECK(b.size(-1) == p.K && act.size(0) == p.M && act.size(1) * 2 == p.N, "shapes differ");
  p.a = operand(a, false);
  p.b = operand(b.view({-1, p.K}), false);
  fill_out(p, act);
  p.ldc = act.stride(0);
  p.glu = true;
  if (gu.has_value()) {
    check_bf16_2d(*gu, "gu");
    TORCH_CHECK(gu->size(0) == p.M && gu->size(1) == p.N, "gu must be [rows, 2I]");
    p.gu = gu->data_ptr();
    p.gu_ld = gu->stride(0);
  }
  if (tile_group.has_value()) {
    TORCH_CHECK(tile_group->scalar_type() == at::kInt && num_m_tiles->scalar_type() == at::kInt && tile_group->dim() == 2 &&
                    tile_group->size(1) == 4 && num_m_tiles->numel() >= 1, "tile maps must be int32 [tiles, 4] and [2]");
    p.max_tiles = tile_group->size(0);
    p.tile_group = tile_group->data_ptr<int>();
    p.num_m_tiles = num_m_tiles->data_ptr<int>();
  }
  p.status = status_ptr(status);
  p.pair = static_cast<int>(pair);
  TORCH_CHECK(mb::gemm_bf16_launch(p, cur_stream()) == 0, "gated_gemm: ", mb::gemm_last_error());
}

// c[g] (+)= a[rows of g]^T . b[rows of g];  a: [R, M], b: [R, N], c: [G, M, N].
void grouped_gemm_contr(const at::Tensor& a, const at::Tensor& b, at::Tensor& c, const at::Tensor& group_offsets,
                        bool accumulate, int64_t block_n, const c10::optional<at::Tensor>& status) {
  check_bf16_2d(a, "a");
  check_bf16_2d(b, "b");
  TORCH_CHECK(a.size(0) == b.size(0), "a and b must have the same number of rows");
  TORCH_CHECK(c.dim() == 3 && c.is_contiguous(), "c must be a contiguous [G, M, N] tensor");
  TORCH_CHECK(group_offsets.scalar_type() == at::kInt && group_offsets.numel() == c.size(0) + 1, "group_offsets must be int32 [G+1]");
  const c10::cuda::CUDAGuard guard(a.device());
  mb::GemmProblem p{};
  p.mode = mb::GEMM_GROUPED_CONTR;
  p.num_groups = c.size(0);
  p.M = a.size(1);
  p.N = b.size(1);
  p.K = 0;
  TORCH_CHECK(c.size(1) == p.M && c.size(2) == p.N, "bad output shape");
  p.a = operand(a, true);
  p.b = operand(b, true);
  fill_out(p, c);
  p.ldc = c.stride(1);
  p.c_group_stride = c.stride(0);
  p.accumulate = accumulate;
  p.group_offsets = group_offsets.data_ptr<int>();
  p.status = status_ptr(status);
  p.block_n = static_cast<int>(block_n);
  TORCH_CHECK(mb::gemm_bf16_launch(p, cur_stream()) == 0, "grouped_gemm_contr: ", mb::gemm_last_error());
}

}  // namespace

void register_elementwise(pybind11::module_& m);  // ops_bindings.cpp
void register_serving(pybind11::module_& m);      // serve_bindings.cpp
void register_vmm(pybind11::module_& m);          // vmm_allocator.cpp

PYBIND11_MODULE(TORCH_EXTENSION_NAME, m) {
  namespace py = pybind11;
  register_serving(m);
  m.def("grouped_gemm_rows", &grouped_gemm_rows, "MoE grouped GEMM over 128-row tiles tagged with a group id", py::arg("a"),
        py::arg("b"), py::arg("c"), py::arg("tile_group"), py::arg("num_m_tiles"), py::arg("b_mn"), py::arg("accumulate"),
        py::arg("block_n"), py::arg("status"), py::arg("row_ptrs") = py::none(), py::arg("sig_ctrl") = py::none(),
        py::arg("sig_flags") = std::vector<int64_t>(), py::arg("sig_me") = 0);
  m.def("score_rows", &score_rows, py::arg("h"), py::arg("w"), py::arg("targets"), py::arg("inv_temp"), py::arg("logits"), py::arg("status"),
        py::arg("pair") = 0);
  m.def("gated_gemm", &gated_gemm, py::arg("a"), py::arg("b"), py::arg("act"), py::arg("gu"), py::arg("tile_group"), py::arg("num_m_tiles"),
        py::arg("status"), py::arg("pair") = 0);
  m.def("grouped_gemm_contr", &grouped_gemm_contr, "MoE weight-gradient GEMM (contraction over each group's rows)");
  register_elementwise(m);
  register_vmm(m);
}

// Python bindings of the local expand / aggregate operators and of the expert activation.
#include <pybind11/pybind11.h>
#include <pybind11/stl.h>

#include <chrono>
#include <stdexcept>
#include <string>

#include "kernels/expand_api.h"
#include "kernels/swiglu_api.h"
#include "rows.h"

namespace py = pybind11;
using namespace dep;

namespace {
template <class T> T* eptr(const py::dict& d, const char* key) {
  if (!d.contains(key) || d[key].is_none()) return nullptr;
  return reinterpret_cast<T*>(d[key].cast<uintptr_t>());
}
void check_launch(cudaError_t e, const char* what) {
  if (e != cudaSuccess) throw std::runtime_error(std::string(what) + ": " + cudaGetErrorString(e));
}
}  // namespace

void bind_expand(py::module_& m) {
  // `dh` null: h from gu; otherwise the gradient of gu.
  m.def("swiglu", [](uintptr_t gu, uintptr_t dh, uintptr_t out, long long rows, int inter, uintptr_t stream) {
    SwigluParams p{};
    p.gu = reinterpret_cast<const __nv_bfloat16*>(gu);
    p.dh = reinterpret_cast<const __nv_bfloat16*>(dh);
    (dh ? p.dgu : p.h) = reinterpret_cast<__nv_bfloat16*>(out);
    p.rows = rows; p.inter = inter;
    if (rows < 0 || inter < 8 || inter % 8) throw std::invalid_argument("swiglu: the width must be a positive multiple of 8");
    if (rows > 0 && (!gu || !out)) throw std::invalid_argument("swiglu: a tensor is missing");
    if ((gu | dh | out) % 16) throw std::invalid_argument("swiglu: rows must start on a 16-byte boundary");
    check_launch(launch_swiglu(p, dh != 0, reinterpret_cast<cudaStream_t>(stream)), "swiglu");
  });
  // `out` and the pair `b`, `prod` may be null, not both.
  m.def("row_scale", [](uintptr_t a, uintptr_t w, uintptr_t out, uintptr_t b, uintptr_t prod, long long rows, int width, int blocks,
                        uintptr_t stream) {
    RowScaleParams p{};
    p.a = reinterpret_cast<const __nv_bfloat16*>(a); p.w = reinterpret_cast<const float*>(w);
    p.out = reinterpret_cast<__nv_bfloat16*>(out);
    p.b = reinterpret_cast<const __nv_bfloat16*>(b); p.prod = reinterpret_cast<__nv_bfloat16*>(prod);
    p.rows = rows; p.width = width;
    if (rows < 0 || width < 8 || width % 8) throw std::invalid_argument("row_scale: the width must be a positive multiple of 8");
    if (rows > 0 && (!a || !w || (!out && !prod) || !b != !prod)) throw std::invalid_argument("row_scale: a tensor is missing");
    if ((a | out | b | prod) % 16) throw std::invalid_argument("row_scale: rows must start on a 16-byte boundary");
    check_launch(launch_row_scale(p, blocks, reinterpret_cast<cudaStream_t>(stream)), "row_scale");
  });
  // `dy` and `dw` may be null, not both.
  m.def("return_grad", [](uintptr_t g, uintptr_t y, uintptr_t w, uintptr_t slot_row, uintptr_t dy, uintptr_t dw, int tokens, int topk,
                          long long rows, int width, uintptr_t stream) {
    ReturnGradParams p{};
    p.g = reinterpret_cast<const __nv_bfloat16*>(g); p.y = reinterpret_cast<const __nv_bfloat16*>(y);
    p.w = reinterpret_cast<const float*>(w); p.slot_row = reinterpret_cast<const int*>(slot_row);
    p.dy = reinterpret_cast<__nv_bfloat16*>(dy); p.dw = reinterpret_cast<float*>(dw);
    p.rows = rows; p.tokens = tokens; p.topk = topk; p.width = width;
    if (tokens < 0 || rows < 0 || topk < 1 || topk > kMaxTopk) throw std::invalid_argument("return_grad: tokens, rows or top-k out of range");
    if (width < 8 || width % 8 || width > 8192) throw std::invalid_argument("return_grad: the width must be a multiple of 8 up to 8192");
    if (tokens > 0 && rows > 0 && (!g || !w || !slot_row || (!dy && !dw) || (dw && !y))) throw std::invalid_argument("return_grad: a tensor is missing");
    if ((g | y | dy) % 16) throw std::invalid_argument("return_grad: rows must start on a 16-byte boundary");
    check_launch(launch_return_grad(p, reinterpret_cast<cudaStream_t>(stream)), "return_grad");
  });
  // Polls a word of host memory until it is not negative; false when `microseconds` passed first.
  m.def("wait_word", [](uintptr_t word, int microseconds) {
    py::gil_scoped_release unlocked;
    const volatile int* w = reinterpret_cast<const volatile int*>(word);
    const auto end = std::chrono::steady_clock::now() + std::chrono::microseconds(microseconds);
    for (unsigned spins = 0; *w < 0; ++spins)
      if ((spins & 63u) == 63u && std::chrono::steady_clock::now() > end) return false;
    return true;
  });
  m.def("expand_scratch", &expand_scratch, py::arg("rows"), py::arg("experts"), py::arg("topk"));
  m.def("expand", [](const py::dict& d, int blocks, uintptr_t stream) {
    ExpandParams p{};
    p.x = eptr<const uint8_t>(d, "x"); p.x_sf = eptr<const float>(d, "x_sf");
    p.topk_idx = eptr<const long long>(d, "topk_idx"); p.topk_w = eptr<const float>(d, "topk_w");
    p.out = eptr<uint8_t>(d, "out"); p.out_sf = eptr<float>(d, "out_sf"); p.out_w = eptr<float>(d, "out_w");
    p.expert_offsets = eptr<int>(d, "expert_offsets"); p.actual_counts = eptr<int>(d, "actual_counts");
    p.mapping = eptr<int>(d, "mapping"); p.tile_counts = eptr<int>(d, "tile_counts"); p.error_flag = eptr<int>(d, "err");
    p.R = d["rows"].cast<int>(); p.K = d["topk"].cast<int>(); p.L = d["experts"].cast<int>(); p.N = d["expanded_rows"].cast<int>();
    p.row_bytes = d["row_bytes"].cast<int>(); p.num_sf = d["num_sf"].cast<int>(); p.cached = d["cached"].cast<int>();
    if (p.K < 1 || p.K > kMaxTopk) throw std::invalid_argument("num_topk must be in [1, 16]");
    if (p.L < 1 || p.L > kMaxExperts) throw std::invalid_argument("1..1024 local experts are supported");
    if (p.row_bytes <= 0 || p.row_bytes % 16) throw std::invalid_argument("a row must be a positive multiple of 16 bytes");
    if (p.R < 0 || p.N < 0) throw std::invalid_argument("negative row count");
    if (!p.expert_offsets || !p.actual_counts || (p.R > 0 && (!p.x || !p.mapping)) || (p.N > 0 && !p.out))
      throw std::invalid_argument("missing tensor");
    if (!p.cached) {
      if (!p.error_flag || (p.R > 0 && (!p.topk_idx || (!p.tile_counts && expand_scratch(p.R, p.L, p.K) > 0))))
        throw std::invalid_argument("expand needs topk_idx and its scratch");
      const py::list caps = d["caps"];
      if ((int)caps.size() != p.L) throw std::invalid_argument("expand needs a capacity per expert");
      for (int e = 0; e < p.L; ++e) p.caps[e] = caps[e].cast<int>();
    }
    require_rows(p.R, {p.x}, "expand"); require_rows(p.N, {p.out}, "expand");
    if ((p.x_sf == nullptr) != (p.out_sf == nullptr)) throw std::invalid_argument("scales need an input and an output");
    check_launch(launch_expand(p, blocks, reinterpret_cast<cudaStream_t>(stream)), "expand launch");
  });
  m.def("aggregate", [](const py::dict& d, uintptr_t stream) {
    AggregateParams p{};
    p.x = eptr<const uint8_t>(d, "x"); p.row_w = eptr<const float>(d, "row_w"); p.values = eptr<const float>(d, "values");
    p.mapping = eptr<const int>(d, "mapping"); p.out = eptr<uint8_t>(d, "out"); p.out_values = eptr<float>(d, "out_values");
    p.R = d["rows"].cast<int>(); p.K = d["topk"].cast<int>(); p.H = d["hidden"].cast<int>(); p.N = d["expanded_rows"].cast<int>();
    p.is_half = d["is_half"].cast<int>();
    if (p.K < 1 || p.K > kMaxTopk) throw std::invalid_argument("num_topk must be in [1, 16]");
    if (p.H <= 0 || p.H % 8) throw std::invalid_argument("hidden must be a positive multiple of 8");
    if (p.R > 0 && (!p.mapping || !p.out || (p.N > 0 && !p.x))) throw std::invalid_argument("missing tensor");
    if (p.R == 0) return;
    require_rows(p.N, {p.x}, "aggregate"); require_rows(p.R, {p.out}, "aggregate");
    check_launch(launch_aggregate(p, reinterpret_cast<cudaStream_t>(stream)), "aggregate launch");
  });
}

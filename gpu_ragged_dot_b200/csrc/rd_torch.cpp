// Host path of the torch layer in native code: argument checks, allocation of the result and the
// workspace, and the C ABI call, for the calls that need nothing else.
//
// A small ragged_dot is bound by its host: the kernels take 5 to 10 us, and the same steps in Python
// (two allocations, a device guard, a stream object, a 16-argument ctypes call) 21 us a call.
// Every function returns the result; None when the call is not of the plain form (the Python layer
// then takes its general path, which pads, converts or raises); or the C ABI's error code.
// From the first allocation on the GIL is released: cudaMalloc may wait for the device and a launch for
// room in the queue, and other Python threads run meanwhile.
#include <ATen/ATen.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/extension.h>

#include "../../include/ragged_dot_b200.h"

namespace {

using at::Tensor;

bool dense(const Tensor& t, c10::DeviceIndex device) {
  return t.is_cuda() && t.device().index() == device && t.layout() == at::kStrided && t.is_contiguous() &&
         !t.is_conj() && !t.is_neg();
}

int dtype_code(at::ScalarType t) {
  switch (t) {
    case at::kHalf: return RD_DTYPE_F16;
    case at::kBFloat16: return RD_DTYPE_BF16;
    case at::kFloat: return RD_DTYPE_F32;
    default: return -1;
  }
}

bool aligned16(const Tensor& t) { return (reinterpret_cast<uintptr_t>(t.data_ptr()) & 15u) == 0; }
bool fits_int(int64_t v) { return v >= 0 && v <= INT32_MAX; }

Tensor bytes(size_t n, const Tensor& like) {
  return at::empty({static_cast<int64_t>(n)}, like.options().dtype(at::kByte));
}

Tensor workspace(int m, int g, const Tensor& like) {
  size_t n = 0;
  rd_workspace_bytes(m, g, &n);
  return bytes(n, like);
}

py::object result(int rc, const Tensor& t) {
  if (rc != RD_OK) return py::int_(rc);
  return py::cast(t);
}

// The tile choice travels as plain integers; all zero = the library chooses.
struct Cfg {
  rd_tile_cfg cfg;
  bool set;
  Cfg(int tile_n, int cta_group, int tile_m, int max_ctas, int flags)
      : cfg{tile_n, max_ctas, cta_group, tile_m, flags, 0}, set((tile_n | cta_group | tile_m | max_ctas | flags) != 0) {}
  const rd_tile_cfg* ptr() const { return set ? &cfg : nullptr; }
};

// max_unaligned: elements up to which rows that are not multiples of 16 bytes go to rd_*_unaligned.
py::object gmm(const Tensor& x, const Tensor& A, const Tensor& gs, bool trans_rhs, int tile_n, int cta_group,
               int tile_m, int max_ctas, int flags, int64_t max_unaligned) {
  if (!x.is_cuda()) return py::none();
  const auto device = x.device().index();
  if (!dense(x, device) || !dense(A, device) || !dense(gs, device)) return py::none();
  const int dtype = dtype_code(x.scalar_type());
  if (dtype < 0 || A.scalar_type() != x.scalar_type() || gs.scalar_type() != at::kInt) return py::none();
  if (x.dim() != 2 || A.dim() != 3 || gs.dim() != 1 || A.size(0) != gs.size(0)) return py::none();
  const int64_t m = x.size(0), k = x.size(1), g = gs.size(0);
  const int64_t n = A.size(trans_rhs ? 1 : 2);
  if (A.size(trans_rhs ? 2 : 1) != k) return py::none();
  if (!fits_int(m) || !fits_int(k) || !fits_int(n) || !fits_int(g)) return py::none();
  const int mask = dtype == RD_DTYPE_F32 ? 3 : 7;
  const bool odd = (k & mask) || (n & mask);
  if (!odd && (!aligned16(x) || !aligned16(A))) return py::none();
  const Cfg cfg(tile_n, cta_group, tile_m, max_ctas, flags);
  if (odd && (dtype == RD_DTYPE_F32 || cfg.set || g > 256 || m > (1 << 20) ||
              m * k + g * k * n + m * n > max_unaligned))
    return py::none();
  const c10::cuda::OptionalCUDAGuard guard(x.device());
  void* stream = c10::cuda::getCurrentCUDAStream(device).stream();
  Tensor y;
  int rc;
  {
    const py::gil_scoped_release no_gil;
    y = at::empty({m, n}, x.options());
    Tensor ws = workspace(m, g, x);
    if (odd) {
      const int64_t a_cols = trans_rhs ? k : n, a_rows = g * (trans_rhs ? n : k);
      Tensor scratch = bytes(rd_unaligned_scratch_bytes(m, k, a_rows, a_cols), x);
      rc = rd_gmm_unaligned(x.data_ptr(), A.data_ptr(), gs.data_ptr<int>(), y.data_ptr(), ws.data_ptr(), ws.numel(),
                            scratch.data_ptr(), scratch.numel(), m, k, n, g, trans_rhs, dtype, stream);
    } else {
      rc = rd_gmm(x.data_ptr(), A.data_ptr(), gs.data_ptr<int>(), y.data_ptr(), ws.data_ptr(), ws.numel(), m, k, n, g,
                  trans_rhs, dtype, cfg.ptr(), stream);
    }
  }
  return result(rc, y);
}

py::object tgmm(const Tensor& x, const Tensor& y, const Tensor& gs, int tile_n, int cta_group, int tile_m,
                int max_ctas, int flags, int64_t max_unaligned) {
  if (!x.is_cuda()) return py::none();
  const auto device = x.device().index();
  if (!dense(x, device) || !dense(y, device) || !dense(gs, device)) return py::none();
  const int dtype = dtype_code(x.scalar_type());
  if (dtype < 0 || y.scalar_type() != x.scalar_type() || gs.scalar_type() != at::kInt) return py::none();
  if (x.dim() != 2 || y.dim() != 2 || gs.dim() != 1 || x.size(0) != y.size(0)) return py::none();
  const int64_t m = x.size(0), k = x.size(1), n = y.size(1), g = gs.size(0);
  if (!fits_int(m) || !fits_int(k) || !fits_int(n) || !fits_int(g)) return py::none();
  const int mask = dtype == RD_DTYPE_F32 ? 3 : 7;
  const bool odd = (k & mask) || (n & mask);
  if (!odd && (!aligned16(x) || !aligned16(y))) return py::none();
  const Cfg cfg(tile_n, cta_group, tile_m, max_ctas, flags);
  if (odd && (dtype == RD_DTYPE_F32 || cfg.set || g > 256 || m > (1 << 20) ||
              m * k + m * n + g * k * n > max_unaligned))
    return py::none();
  const c10::cuda::OptionalCUDAGuard guard(x.device());
  void* stream = c10::cuda::getCurrentCUDAStream(device).stream();
  Tensor out;
  int rc;
  {
    const py::gil_scoped_release no_gil;
    out = at::empty({g, k, n}, x.options());
    Tensor ws = workspace(m, g, x);
    if (odd) {
      Tensor scratch = bytes(rd_unaligned_scratch_bytes(m, k, m, n), x);
      rc = rd_tgmm_unaligned(x.data_ptr(), y.data_ptr(), gs.data_ptr<int>(), out.data_ptr(), ws.data_ptr(), ws.numel(),
                             scratch.data_ptr(), scratch.numel(), m, k, n, g, dtype, stream);
    } else {
      rc = rd_tgmm(x.data_ptr(), y.data_ptr(), gs.data_ptr<int>(), out.data_ptr(), ws.data_ptr(), ws.numel(), m, k, n, g,
                   dtype, cfg.ptr(), stream);
    }
  }
  return result(rc, out);
}

py::object gmm_fp8(const Tensor& x, const Tensor& A, const Tensor& gs, const c10::optional<Tensor>& scale) {
  if (!x.is_cuda()) return py::none();
  const auto device = x.device().index();
  if (!dense(x, device) || !dense(A, device) || !dense(gs, device)) return py::none();
  if (x.scalar_type() != at::kFloat8_e4m3fn || A.scalar_type() != at::kFloat8_e4m3fn || gs.scalar_type() != at::kInt)
    return py::none();
  if (x.dim() != 2 || A.dim() != 3 || gs.dim() != 1 || A.size(0) != gs.size(0) || A.size(2) != x.size(1))
    return py::none();
  const int64_t m = x.size(0), k = x.size(1), n = A.size(1), g = gs.size(0);
  if (!fits_int(m) || !fits_int(k) || !fits_int(n) || !fits_int(g) || (k & 15) || (n & 7)) return py::none();
  if (!aligned16(x) || !aligned16(A)) return py::none();
  const float* sc = nullptr;
  if (scale.has_value()) {
    if (!dense(*scale, device) || scale->scalar_type() != at::kFloat || scale->numel() != g) return py::none();
    sc = scale->data_ptr<float>();
  }
  const c10::cuda::OptionalCUDAGuard guard(x.device());
  void* stream = c10::cuda::getCurrentCUDAStream(device).stream();
  Tensor y;
  int rc;
  {
    const py::gil_scoped_release no_gil;
    y = at::empty({m, n}, x.options().dtype(at::kBFloat16));
    Tensor ws = workspace(m, g, x);
    rc = rd_gmm_fp8(x.data_ptr(), A.data_ptr(), g, gs.data_ptr<int>(), nullptr, sc, y.data_ptr(), ws.data_ptr(),
                    ws.numel(), m, k, n, g, nullptr, stream);
  }
  return result(rc, y);
}

}  // namespace

PYBIND11_MODULE(TORCH_EXTENSION_NAME, mod) {
  mod.def("gmm", &gmm);
  mod.def("tgmm", &tgmm);
  mod.def("gmm_fp8", &gmm_fp8);
}

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

// One product in the plain form: what its call needs, and whether the operands are of that form at all.
// max_unaligned: elements up to which rows that are not multiples of 16 bytes go to rd_*_unaligned.
struct Product {
  Tensor a, b, gs, out;  // gmm: x, A; tgmm: x, y
  int64_t m = 0, k = 0, n = 0, g = 0;
  int dtype = -1;
  bool tgmm, trans_rhs, odd = false;
  Cfg cfg;

  Product(bool tgmm_, const Tensor& a_, const Tensor& b_, const Tensor& gs_, bool trans_rhs_, const Cfg& cfg_)
      : a(a_), b(b_), gs(gs_), tgmm(tgmm_), trans_rhs(trans_rhs_), cfg(cfg_) {}

  bool plain(int64_t max_unaligned) {
    if (!a.is_cuda()) return false;
    const auto device = a.device().index();
    if (!dense(a, device) || !dense(b, device) || !dense(gs, device)) return false;
    dtype = dtype_code(a.scalar_type());
    if (dtype < 0 || b.scalar_type() != a.scalar_type() || gs.scalar_type() != at::kInt) return false;
    if (a.dim() != 2 || b.dim() != (tgmm ? 2 : 3) || gs.dim() != 1) return false;
    m = a.size(0);
    k = a.size(1);
    g = gs.size(0);
    if (tgmm) {
      if (b.size(0) != m) return false;
      n = b.size(1);
    } else {
      if (b.size(0) != g || b.size(trans_rhs ? 2 : 1) != k) return false;
      n = b.size(trans_rhs ? 1 : 2);
    }
    if (!fits_int(m) || !fits_int(k) || !fits_int(n) || !fits_int(g)) return false;
    const int mask = dtype == RD_DTYPE_F32 ? 3 : 7;
    odd = (k & mask) || (n & mask);
    if (!odd) return aligned16(a) && aligned16(b);
    return !(dtype == RD_DTYPE_F32 || cfg.set || g > 256 || m > (1 << 20) || m * k + g * k * n + m * n > max_unaligned);
  }

  // Allocates the result and launches; the caller holds the device guard, and no GIL.
  int run(void* stream) {
    out = tgmm ? at::empty({g, k, n}, a.options()) : at::empty({m, n}, a.options());
    Tensor ws = workspace(m, g, a);
    if (odd) {
      const int64_t b_cols = tgmm || !trans_rhs ? n : k, b_rows = tgmm ? m : g * (trans_rhs ? n : k);
      Tensor scratch = bytes(rd_unaligned_scratch_bytes(m, k, b_rows, b_cols), a);
      return tgmm ? rd_tgmm_unaligned(a.data_ptr(), b.data_ptr(), gs.data_ptr<int>(), out.data_ptr(), ws.data_ptr(),
                                      ws.numel(), scratch.data_ptr(), scratch.numel(), m, k, n, g, dtype, stream)
                  : rd_gmm_unaligned(a.data_ptr(), b.data_ptr(), gs.data_ptr<int>(), out.data_ptr(), ws.data_ptr(),
                                     ws.numel(), scratch.data_ptr(), scratch.numel(), m, k, n, g, trans_rhs, dtype,
                                     stream);
    }
    return tgmm ? rd_tgmm(a.data_ptr(), b.data_ptr(), gs.data_ptr<int>(), out.data_ptr(), ws.data_ptr(), ws.numel(), m, k,
                          n, g, dtype, cfg.ptr(), stream)
                : rd_gmm(a.data_ptr(), b.data_ptr(), gs.data_ptr<int>(), out.data_ptr(), ws.data_ptr(), ws.numel(), m, k,
                         n, g, trans_rhs, dtype, cfg.ptr(), stream);
  }
};

py::object run_one(Product p, int64_t max_unaligned) {
  if (!p.plain(max_unaligned)) return py::none();
  const c10::cuda::OptionalCUDAGuard guard(p.a.device());
  void* stream = c10::cuda::getCurrentCUDAStream(p.a.device().index()).stream();
  int rc;
  {
    const py::gil_scoped_release no_gil;
    rc = p.run(stream);
  }
  return result(rc, p.out);
}

py::object gmm(const Tensor& x, const Tensor& A, const Tensor& gs, bool trans_rhs, int tile_n, int cta_group,
               int tile_m, int max_ctas, int flags, int64_t max_unaligned) {
  return run_one(Product(false, x, A, gs, trans_rhs, Cfg(tile_n, cta_group, tile_m, max_ctas, flags)), max_unaligned);
}

py::object tgmm(const Tensor& x, const Tensor& y, const Tensor& gs, int tile_n, int cta_group, int tile_m,
                int max_ctas, int flags, int64_t max_unaligned) {
  return run_one(Product(true, x, y, gs, false, Cfg(tile_n, cta_group, tile_m, max_ctas, flags)), max_unaligned);
}

// Both products of gmm's backward pass in one call: (dx, dA), None or an error code.  Nothing is launched unless both are of
// the plain form.  The two calls from Python, on autograd's thread, took 31 us of the host's time.
py::object gmm_backward(const Tensor& dout, const Tensor& x, const Tensor& A, const Tensor& gs, bool trans_rhs,
                        int64_t max_unaligned) {
  const Cfg none(0, 0, 0, 0, 0);
  Product dx(false, dout, A, gs, !trans_rhs, none);
  Product dA(true, trans_rhs ? dout : x, trans_rhs ? x : dout, gs, false, none);
  if (!dx.plain(max_unaligned) || !dA.plain(max_unaligned) || dA.a.device() != dx.a.device()) return py::none();
  const c10::cuda::OptionalCUDAGuard guard(dout.device());
  void* stream = c10::cuda::getCurrentCUDAStream(dout.device().index()).stream();
  int rc;
  {
    const py::gil_scoped_release no_gil;
    rc = dx.run(stream);
    if (rc == RD_OK) rc = dA.run(stream);
  }
  if (rc != RD_OK) return py::int_(rc);
  return py::make_tuple(dx.out, dA.out);
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
  mod.def("gmm_backward", &gmm_backward);
  mod.def("gmm_fp8", &gmm_fp8);
}

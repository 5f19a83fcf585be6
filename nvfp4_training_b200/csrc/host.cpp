// Native host path of the Python operators: argument checks, output allocation, stream look-up and the calls into the
// C-ABI library, in one C++ call per operator and one per layer pass.
//
// What bounds the small and middle-sized layers is not the GPU but the interpreter: a forward and backward pass of one
// linear is seven kernels and, written in Python over ctypes, was 25 tensor allocations, 11 foreign calls of up to 20
// converted arguments and 11 walks of torch's Python stream objects -- 340 us of host work around 41 us of kernels
// at [128, 256] x [384, 256].  Here a pass is one call: scratch that dies with the call is one allocation addressed by
// offsets, what the backward pass needs is one more, and the backward is an autograd node that runs without the
// interpreter except for one look at the caller's switches (seed, gradient type, rounding mode, cached weight).  That
// pass takes 79 us now, [4096, 2048] x [3072, 2048] 126 instead of 344 (kernel time), a forward without gradients
// [256, 5632] x [2048, 5632] 15.6 instead of 79.  Calls release the interpreter lock, as ctypes does.
//
// The library itself is not linked: `bind` receives the addresses of its entry points from the ctypes binding, so both
// always use the same build.  Exceptions: AssertionError for shapes and types (as the Python asserts it replaces),
// the package's Nvfp4Error for CPU tensors and for calls the library rejects.
#include <ATen/ATen.h>
#include <ATen/cuda/EmptyTensor.h>
#include <c10/cuda/CUDAStream.h>
#include <pybind11/pybind11.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/custom_function.h>
#include <torch/csrc/autograd/function.h>
#include <torch/csrc/autograd/functions/utils.h>
#include <torch/csrc/autograd/python_variable.h>
#include <torch/csrc/autograd/saved_variable.h>
#include <torch/csrc/utils/pybind.h>

#include <atomic>
#include <mutex>

#include "../../include/nvfp4_b200.h"

namespace py = pybind11;
using at::Tensor;
using OptTensor = std::optional<Tensor>;

namespace {

// ------------------------------------------------------------------------------------------ library entry points
#define NVFP4_API(X)                                                                                                        \
  X(nvfp4_amax_bf16) X(nvfp4_amax_bf16_update) X(nvfp4_quant_rows) X(nvfp4_quant_cols_rht) X(nvfp4_quant_tile) X(nvfp4_quant_tile_amax)             \
  X(nvfp4_quant_w2d) X(nvfp4_gemm) X(nvfp4_error_string) X(nvfp4_amax_f32) X(nvfp4_amax_bf16_word) X(nvfp4_swizzle_scales) X(nvfp4_emit_rows)        \
  X(nvfp4_emit_cols) X(nvfp4_rms_emit) X(nvfp4_swiglu_emit) X(nvfp4_mom_acc)
struct Api {
#define X(name) decltype(&::name) name = nullptr;
  NVFP4_API(X)
#undef X
};
Api lib;

struct AssertionFailure : std::runtime_error { using std::runtime_error::runtime_error; };
struct LibraryError : std::runtime_error { using std::runtime_error::runtime_error; };
// Python objects the module keeps for the life of the process (never released: the interpreter may be gone by then)
py::handle error_class, lin_ctx, nvq_module, status_word_fn;

#define REQUIRE(cond, what) do { if (!(cond)) throw AssertionFailure(what); } while (0)

void check(int rc, const char* what) {
  if (rc != 0)
    throw LibraryError(std::string(what) + ": " + lib.nvfp4_error_string(rc) + " (status " + std::to_string(rc) + ")");
}
void require_cuda(const Tensor& t) {
  if (!t.is_cuda()) throw LibraryError("nvfp4_b200 kernels need CUDA tensors; there is no CPU path");
}
void require_cuda(const OptTensor& t) { if (t) require_cuda(*t); }

std::string shape_of(int64_t a, int64_t b) { return "(" + std::to_string(a) + ", " + std::to_string(b) + ")"; }

// ------------------------------------------------------------------------------------------ small pieces
void* stream() { return c10::cuda::getCurrentCUDAStream().stream(); }

Tensor empty(at::IntArrayRef size, at::ScalarType dtype, const Tensor& like) {
  return at::detail::empty_cuda(size, dtype, like.device(), std::nullopt);
}
const void* cptr(const OptTensor& t) { return t ? t->const_data_ptr() : nullptr; }

// Host seed or a device word: a CUDA int32 / uint32 tensor selects the device-side seed.  (Constructed from a Python
// object with the interpreter lock held, by the caster at the end of this file.)
struct Seed {
  unsigned host = 0;
  const unsigned* dev = nullptr;
  Tensor keep;
  Seed() = default;
  explicit Seed(unsigned h) : host(h) {}
  explicit Seed(py::handle o) {
    if (THPVariable_Check(o.ptr())) {
      keep = THPVariable_Unpack(o.ptr());
      REQUIRE(keep.is_cuda() && keep.numel() >= 1 && keep.element_size() == 4, "seed: a CUDA tensor of 32-bit words");
      dev = static_cast<const unsigned*>(keep.const_data_ptr());
    } else {
      host = (unsigned)PyLong_AsUnsignedLongLongMask(o.ptr());
      if (PyErr_Occurred()) throw py::error_already_set();
    }
  }
};

// Per-device status word of the GEMM, created and owned by the Python binding.
int* status_word(const Tensor& like) {
  constexpr int kDevices = 64;
  static std::atomic<int*> words[kDevices];
  const int dev = like.get_device();
  TORCH_CHECK(dev >= 0 && dev < kDevices);
  int* p = words[dev].load(std::memory_order_relaxed);
  if (!p) {
    py::gil_scoped_acquire gil;
    p = static_cast<int*>(py::cast<Tensor>(status_word_fn(like.device())).data_ptr());
    words[dev].store(p, std::memory_order_relaxed);
  }
  return p;
}

// Carves sub-buffers, each at a multiple of 256 bytes, out of one allocation; in a dry run it only adds up sizes.
struct Carver {
  char* base = nullptr;
  size_t used = 0;
  template <typename T = void>
  T* take(size_t bytes) {
    T* p = base ? reinterpret_cast<T*>(base + used) : nullptr;
    used += (bytes + 255) & ~size_t(255);
    return p;
  }
};

// A packed matrix [R, C]: codes, bytes from row to row of them, swizzled scales, tensor scale.
struct Packed {
  const void* d; int64_t ld; const void* s; const float* gs;
};
// One of whole rows, as the quantizers write it.
struct PackedOut {
  void* d = nullptr; void* s = nullptr; float* gs = nullptr;
  Packed in(int64_t C) const { return {d, C / 2, s, gs}; }
};
PackedOut carve_packed(Carver& c, int64_t R, int64_t C) {
  void* d = c.take(R * C / 2);
  void* s = c.take(R * C / 16);
  return {d, s, c.take<float>(4)};
}

using Packed3 = std::tuple<Tensor, Tensor, Tensor>;          // the `d`, `s`, `gs` of a Q
using OptPacked3 = std::optional<Packed3>;

// Fresh output tensors of a packed matrix (the `d`, `s`, `gs` of a Q).
struct PackedTensors {
  Tensor d, s, gs;
  PackedTensors(int64_t R, int64_t C, const Tensor& like)
      : d(empty({R, C / 2}, at::kFloat4_e2m1fn_x2, like)), s(empty({R * C / 16}, at::kFloat8_e4m3fn, like)),
        gs(empty({1}, at::kFloat, like)) {}
  PackedOut out() const { return {d.data_ptr(), s.data_ptr(), gs.data_ptr<float>()}; }
  Packed3 tuple() const { return {d, s, gs}; }
};

// ------------------------------------------------------------------------------------------ launches
void run_amax(const Tensor& x, float* out, bool clear = true) {
  check((clear ? lib.nvfp4_amax_bf16 : lib.nvfp4_amax_bf16_update)(x.const_data_ptr(), x.numel(), out, stream()), "amax");
}

// amax for consumers that this thread launches next: a word of the library, or `fallback` (null: nothing is launched)
// where it has none
const float* passing_amax(const Tensor& x, float* fallback) {
  const float* word = nullptr;
  check(lib.nvfp4_amax_bf16_word(x.const_data_ptr(), x.numel(), fallback, &word, stream()), "amax");
  return word;
}

void run_tile(const Tensor& x, const PackedOut* row, const PackedOut* col, const float* am, unsigned signs, int mode,
              const Seed& seed, const Seed& seed_cols) {
  check(lib.nvfp4_quant_tile(x.const_data_ptr(), x.stride(0), (int)x.size(0), (int)x.size(1), row ? row->d : nullptr,
                             row ? row->s : nullptr, col ? col->d : nullptr, col ? col->s : nullptr, NVFP4_SCALES_SWIZZLED, am,
                             row ? row->gs : nullptr, col ? col->gs : nullptr, signs & 0xFFFFu, mode, seed.host,
                             seed_cols.host, seed.dev, seed_cols.dev, stream()), "quant_tile");
}

// The same with the tensor's amax found on the way (into `amax_out`, unless that is null); false: not launched
bool run_tile_amax(const Tensor& x, const PackedOut* row, const PackedOut* col, float* amax_out, unsigned signs, int mode, const Seed& seed,
                   const Seed& seed_cols) {
  int launched = 0;
  check(lib.nvfp4_quant_tile_amax(x.const_data_ptr(), x.stride(0), (int)x.size(0), (int)x.size(1), row ? row->d : nullptr,
                                  row ? row->s : nullptr, col ? col->d : nullptr, col ? col->s : nullptr, NVFP4_SCALES_SWIZZLED, amax_out,
                                  &launched, row ? row->gs : nullptr, col ? col->gs : nullptr, signs & 0xFFFFu, mode, seed.host,
                                  seed_cols.host, seed.dev, seed_cols.dev, stream()), "quant_tile_amax");
  return launched != 0;
}

void run_w2d(const Tensor& w, const PackedOut* q, const PackedOut* qt, const float* am) {
  check(lib.nvfp4_quant_w2d(w.const_data_ptr(), NVFP4_DTYPE_BF16, (int)w.size(0), (int)w.size(1), q ? q->d : nullptr,
                            q ? q->s : nullptr, qt ? qt->d : nullptr, qt ? qt->s : nullptr, NVFP4_SCALES_SWIZZLED, am,
                            (q ? q : qt)->gs, stream()), "quant_w2d");
}

// packed operands a [M, K], b [N, K] -> c [M, N]
void run_mm(const Packed& a, const Packed& b, const Tensor& c, int64_t K, bool accumulate, int splitk) {
  const bool fp32 = c.scalar_type() == at::kFloat;
  check(lib.nvfp4_gemm(a.d, a.s, a.ld, b.d, b.s, b.ld, c.data_ptr(), fp32 ? NVFP4_DTYPE_FP32 : NVFP4_DTYPE_BF16,
                       c.stride(0), (int)c.size(0), (int)c.size(1), (int)K, NVFP4_ALPHA_GS, a.gs, b.gs, 1.f, 1.f, accumulate,
                       fp32 ? splitk : 1, status_word(c), stream()), "mm");
}

// ------------------------------------------------------------------------------------------ nvq operators
Tensor nvq_amax(const Tensor& x, const OptTensor& out_, bool clear) {
  require_cuda(x); require_cuda(out_);
  REQUIRE(out_ || clear, "amax: clear=False needs out");
  REQUIRE(x.numel() % 8 == 0 && x.is_contiguous() && x.scalar_type() == at::kBFloat16, "amax: contiguous bf16, a multiple of 8 values");
  Tensor out = out_ ? *out_ : empty({1}, at::kFloat, x);
  run_amax(x, static_cast<float*>(out.data_ptr()), clear);
  return out;
}

const float* word(const Tensor& am) { return static_cast<const float*>(am.const_data_ptr()); }
// amax word of `x` for the launches that follow: the caller's, or computed now.  `keep` holds the word where the
// library has none to offer.
const float* amax_or(const OptTensor& am, const Tensor& x, Tensor& keep) {
  if (am) return word(*am);
  REQUIRE(x.numel() % 8 == 0, "amax: a multiple of 8 values");
  at::NoGradGuard no_grad;
  const Tensor xc = x.contiguous();
  const float* w = xc.numel() ? passing_amax(xc, nullptr) : nullptr;
  if (w) return w;
  keep = empty({1}, at::kFloat, x);
  run_amax(xc, keep.data_ptr<float>());
  return word(keep);
}

Packed3 nvq_quant_rows(const Tensor& x, int mode, const Seed& seed, const OptTensor& am_) {
  require_cuda(x);
  REQUIRE(x.dim() == 2 && x.scalar_type() == at::kBFloat16, "quant_rows: a bf16 matrix");
  const int64_t R = x.size(0), C = x.size(1);
  REQUIRE(x.stride(1) == 1 && C % 64 == 0 && R % 128 == 0, shape_of(R, C));
  PackedTensors q(R, C, x);
  const PackedOut o = q.out();
  Tensor keep;
  const float* am = amax_or(am_, x, keep);
  check(lib.nvfp4_quant_rows(x.const_data_ptr(), x.stride(0), (int)R, (int)C, o.d, o.s, NVFP4_SCALES_SWIZZLED, am, o.gs,
                             mode, seed.host, seed.dev, stream()), "quant_rows");
  return q.tuple();
}

Packed3 nvq_quant_cols_rht(const Tensor& x_, unsigned signs, int mode, const Seed& seed, const OptTensor& am_) {
  require_cuda(x_);
  REQUIRE(x_.dim() == 2 && x_.scalar_type() == at::kBFloat16, "quant_cols_rht: a bf16 matrix");
  at::NoGradGuard no_grad;
  const Tensor x = x_.contiguous();
  const int64_t M = x.size(0), C = x.size(1);
  REQUIRE(M % 64 == 0 && C % 128 == 0, shape_of(M, C));
  PackedTensors q(C, M, x);
  const PackedOut o = q.out();
  if (!am_ && M % 128 == 0 && run_tile_amax(x, nullptr, &o, nullptr, signs, mode, Seed(), seed)) return q.tuple();
  Tensor keep;
  const float* am = amax_or(am_, x, keep);
  // the tile kernel takes whole 128-token tiles: same bits, faster than the register-tiled kernel
  if (M % 128 == 0) run_tile(x, nullptr, &o, am, signs, mode, Seed(), seed);
  else check(lib.nvfp4_quant_cols_rht(x.const_data_ptr(), (int)M, (int)C, o.d, o.s, NVFP4_SCALES_SWIZZLED, am, o.gs,
                                      signs & 0xFFFFu, mode, seed.host, seed.dev, stream()), "quant_cols_rht");
  return q.tuple();
}

std::pair<OptPacked3, OptPacked3> nvq_quant_rows_cols_rht(const Tensor& x, unsigned signs, int mode, const Seed& seed, const Seed& seed_cols,
                                                          const OptTensor& am_, bool want_rows, bool want_cols) {
  require_cuda(x);
  REQUIRE(x.dim() == 2 && x.scalar_type() == at::kBFloat16 && x.stride(1) == 1, "quant_rows_cols_rht: a bf16 matrix with contiguous rows");
  const int64_t M = x.size(0), C = x.size(1);
  REQUIRE(M % 128 == 0 && C % 128 == 0, shape_of(M, C));
  std::optional<PackedTensors> qr, qc;
  PackedOut r, c;
  if (want_rows) { qr.emplace(M, C, x); r = qr->out(); }
  if (want_cols) { qc.emplace(C, M, x); c = qc->out(); }
  if (am_ || !(want_rows || want_cols) || !run_tile_amax(x, want_rows ? &r : nullptr, want_cols ? &c : nullptr, nullptr, signs, mode, seed, seed_cols)) {
    Tensor keep;
    const float* am = amax_or(am_, x, keep);
    run_tile(x, want_rows ? &r : nullptr, want_cols ? &c : nullptr, am, signs, mode, seed, seed_cols);
  }
  return {qr ? OptPacked3(qr->tuple()) : std::nullopt, qc ? OptPacked3(qc->tuple()) : std::nullopt};
}

// Fresh outputs, the two operands sharing one tensor scale; a skipped operand is None.
std::pair<OptPacked3, OptPacked3> nvq_quant_w2d(const Tensor& w_, const OptTensor& am_, bool want, bool want_t) {
  require_cuda(w_);
  REQUIRE(w_.dim() == 2 && w_.scalar_type() == at::kBFloat16, "quant_w2d: a bf16 matrix");
  at::NoGradGuard no_grad;
  const Tensor w = w_.contiguous();
  const int64_t N = w.size(0), K = w.size(1);
  REQUIRE(N % 128 == 0 && K % 128 == 0, shape_of(N, K));
  const Tensor gs = empty({1}, at::kFloat, w);
  auto alloc = [&](int64_t R, int64_t C, Tensor& d, Tensor& s) {
    d = empty({R, C / 2}, at::kFloat4_e2m1fn_x2, w);
    s = empty({R * C / 16}, at::kFloat8_e4m3fn, w);
    return PackedOut{d.data_ptr(), s.data_ptr(), gs.data_ptr<float>()};
  };
  Tensor d, s, dt, st;
  PackedOut q, qt;
  if (want) q = alloc(N, K, d, s);
  if (want_t) qt = alloc(K, N, dt, st);
  Tensor keep;
  run_w2d(w, want ? &q : nullptr, want_t ? &qt : nullptr, amax_or(am_, w, keep));
  return {want ? OptPacked3({d, s, gs}) : std::nullopt, want_t ? OptPacked3({dt, st, gs}) : std::nullopt};
}

// In place into an earlier call's buffers.
void nvq_quant_w2d_into(const Tensor& w_, const OptTensor& am_, const OptTensor& d, const OptTensor& s, const OptTensor& dt,
                        const OptTensor& st, const Tensor& gs) {
  require_cuda(w_);
  REQUIRE(w_.dim() == 2 && w_.scalar_type() == at::kBFloat16, "quant_w2d: a bf16 matrix");
  at::NoGradGuard no_grad;
  const Tensor w = w_.contiguous();
  REQUIRE(w.size(0) % 128 == 0 && w.size(1) % 128 == 0, shape_of(w.size(0), w.size(1)));
  float* g = static_cast<float*>(gs.data_ptr());
  const PackedOut q{d ? d->data_ptr() : nullptr, s ? s->data_ptr() : nullptr, g};
  const PackedOut qt{dt ? dt->data_ptr() : nullptr, st ? st->data_ptr() : nullptr, g};
  Tensor keep;
  run_w2d(w, d ? &q : nullptr, dt ? &qt : nullptr, amax_or(am_, w, keep));
}

// A block-scaled GEMM into `out` (or a fresh tensor): alpha = product of the two words as `alpha_mode` says.  Slices asked
// for are added to `out`; a fresh tensor has nothing to add to, so there the library picks the slices and clears it first.
Tensor gemm(const Tensor& ad, const Tensor& as, const Tensor& bd, const Tensor& bs, const OptTensor& out_, bool fp32, int alpha_mode,
            const OptTensor& pa, const OptTensor& pb, float ka, float kb, bool accumulate, int splitk, const char* what) {
  require_cuda(ad); require_cuda(bd);
  const int64_t M = ad.size(0), N = bd.size(0), K = ad.size(1) * 2;
  REQUIRE(bd.size(1) * 2 == K, shape_of(M, K / 2) + ", " + shape_of(N, bd.size(1)));
  const at::ScalarType dtype = fp32 ? at::kFloat : at::kBFloat16;
  if (out_) {
    require_cuda(out_);
    REQUIRE(out_->dim() == 2 && out_->size(0) == M && out_->size(1) == N && out_->scalar_type() == dtype && out_->stride(1) == 1,
            "out: shape, type or row layout");
  } else {
    REQUIRE(!accumulate, "accumulate needs out");
  }
  Tensor out = out_ ? *out_ : empty({M, N}, dtype, ad);
  check(lib.nvfp4_gemm(ad.const_data_ptr(), as.const_data_ptr(), ad.stride(0), bd.const_data_ptr(), bs.const_data_ptr(), bd.stride(0),
                       out.data_ptr(), fp32 ? NVFP4_DTYPE_FP32 : NVFP4_DTYPE_BF16, out.stride(0), (int)M, (int)N, (int)K, alpha_mode,
                       static_cast<const float*>(cptr(pa)), static_cast<const float*>(cptr(pb)), ka, kb, accumulate,
                       !fp32 ? 1 : !out_ && splitk > 1 ? 0 : splitk, status_word(ad), stream()), what);
  return out;
}

Tensor nvq_mm(const Tensor& ad, const Tensor& as, const Tensor& ag, const Tensor& bd, const Tensor& bs, const Tensor& bg, bool fp32,
              bool scale, const OptTensor& out, bool accumulate, int splitk) {
  return gemm(ad, as, bd, bs, out, fp32, scale ? NVFP4_ALPHA_GS : NVFP4_ALPHA_ONE, scale ? OptTensor(ag) : OptTensor(),
              scale ? OptTensor(bg) : OptTensor(), 1.f, 1.f, accumulate, splitk, "mm");
}

// ------------------------------------------------------------------------------------------ the linear layer
// y = Q_rn(x) Q(W)^T with the row operand of x in scratch; `xt` (optional) receives the transposed operand.  `am`: the
// caller's amax(x); null: it is found here, into `am_out` (unless that is null too).
Tensor forward_core(const Tensor& x, const float* am, float* am_out, const Packed& w, int64_t N, const PackedOut* xt, unsigned signs) {
  const int64_t T = x.size(0), K = x.size(1);
  Carver size;
  carve_packed(size, T, K);
  const Tensor scratch = empty({(int64_t)size.used}, at::kByte, x);
  Carver c{static_cast<char*>(scratch.data_ptr())};
  const PackedOut qx = carve_packed(c, T, K);
  if (am || !run_tile_amax(x, &qx, xt, am_out, signs, NVFP4_ROUND_NEAREST, Seed(), Seed())) {
    Tensor keep;
    if (!am && am_out) {
      run_amax(x.contiguous(), am_out);
      am = am_out;
    } else if (!am) {
      am = amax_or(std::nullopt, x, keep);
    }
    run_tile(x, &qx, xt, am, signs, NVFP4_ROUND_NEAREST, Seed(), Seed());
  }
  Tensor y = empty({T, N}, at::kBFloat16, x);
  run_mm(qx.in(K), w, y, K, false, 1);
  return y;
}

struct BackwardArgs {
  int64_t K, Kw;                   // columns of gx and of gW: in-features
  unsigned signs;
  int mode;
  bool want_x = true, want_w = true;
  OptTensor gw_out;                // FP32 [N, K] to add into (or overwrite); else a new tensor of `gw_dtype`
  bool overwrite = false;
  at::ScalarType gw_dtype = at::kFloat;
  OptTensor am;                    // amax(gy) where the caller has it
  OptTensor am_out;                // else a cleared word to compute it into
};

// gx = Q_sr(gy) Q(W^T)^T and gW = Q_sr(H gy)^T Q(H x): one amax, one pass over gy for both operands, two GEMMs
std::pair<Tensor, Tensor> backward_core(const Tensor& gy, const Packed& wt, const Packed& xt, const Seed& seed,
                                        const Seed& seed_cols, const BackwardArgs& a) {
  const int64_t T = gy.size(0), N = gy.size(1);
  Tensor gx, gw;
  auto carve = [&](Carver& c, PackedOut& r, PackedOut& t, float*& am) {
    am = c.take<float>(4);
    if (a.want_x) r = carve_packed(c, T, N);
    if (a.want_w) t = carve_packed(c, N, T);
  };
  PackedOut qg, qgt;
  float* own_am;
  Carver size;
  carve(size, qg, qgt, own_am);
  const Tensor scratch = empty({(int64_t)size.used}, at::kByte, gy);
  Carver c{static_cast<char*>(scratch.data_ptr())};
  carve(c, qg, qgt, own_am);
  const PackedOut *row = a.want_x ? &qg : nullptr, *col = a.want_w ? &qgt : nullptr;
  if (a.am || a.am_out || !run_tile_amax(gy, row, col, nullptr, a.signs, a.mode, seed, seed_cols)) {
    const float* am = a.am ? word(*a.am) : a.am_out ? word(*a.am_out) : own_am;
    if (!a.am && a.am_out) run_amax(gy, const_cast<float*>(am), false);
    else if (!a.am && gy.numel()) am = passing_amax(gy, own_am);
    run_tile(gy, row, col, am, a.signs, a.mode, seed, seed_cols);
  }
  if (a.want_x) {
    gx = empty({T, a.K}, at::kBFloat16, gy);
    run_mm(qg.in(N), wt, gx, N, false, 1);
  }
  if (a.want_w) {
    gw = a.gw_out ? *a.gw_out : empty({N, a.Kw}, a.gw_dtype, gy);
    run_mm(qgt.in(T), xt, gw, T, a.gw_out && !a.overwrite, a.gw_out ? 0 : 1);
  }
  return {gx, gw};
}

// a code matrix [R, C/2] (its rows may have a stride) with its scales; R < 0: any number of rows
Packed packed_of(const Tensor& d, const Tensor& s, const Tensor& gs, int64_t R, int64_t C, const char* what) {
  require_cuda(d);
  REQUIRE(d.dim() == 2 && (R < 0 || d.size(0) == R) && d.size(1) * 2 == C && d.stride(1) == 1, what);
  return {d.const_data_ptr(), d.stride(0), s.const_data_ptr(), word(gs)};
}

std::tuple<Tensor, Tensor, Tensor, Tensor, Tensor> linear_fwd(const Tensor& x, const Tensor& wd, const Tensor& ws, const Tensor& wg, unsigned signs, const OptTensor& am_out) {
  require_cuda(x);
  at::NoGradGuard no_grad;
  REQUIRE(x.dim() == 2 && x.scalar_type() == at::kBFloat16 && x.stride(1) == 1, "linear_fwd: a bf16 matrix with contiguous rows");
  const int64_t T = x.size(0), K = x.size(1), N = wd.size(0);
  const Packed w = packed_of(wd, ws, wg, N, K, "linear_fwd: quantized weight");
  const Tensor am = am_out ? nvq_amax(x.contiguous(), am_out, false) : empty({1}, at::kFloat, x);
  PackedTensors xt(K, T, x);
  const PackedOut o = xt.out();
  Tensor y = forward_core(x, am_out ? word(am) : nullptr, am_out ? nullptr : am.data_ptr<float>(), w, N, &o, signs);
  return {y, am, xt.d, xt.s, xt.gs};
}

std::pair<Tensor, Tensor> linear_bwd(const Tensor& gy_, const Tensor& wd, const Tensor& ws, const Tensor& wg, const Tensor& xd,
                                     const Tensor& xs, const Tensor& xg, const Seed& seed, const Seed& seed_cols, unsigned signs, int mode,
                                     const OptTensor& gw_out, bool overwrite, bool gw_fp32, const OptTensor& am, const OptTensor& am_out) {
  require_cuda(gy_); require_cuda(am_out);
  at::NoGradGuard no_grad;
  const Tensor gy = gy_.contiguous();
  REQUIRE(gy.dim() == 2 && gy.scalar_type() == at::kBFloat16, "linear_bwd: bf16 output gradient");
  BackwardArgs a;
  a.K = wd.size(0);
  a.Kw = xd.size(0);
  const Packed wt = packed_of(wd, ws, wg, -1, gy.size(1), "linear_bwd: quantized transposed weight");
  const Packed xt = packed_of(xd, xs, xg, -1, gy.size(0), "linear_bwd: transposed operand of x");
  a.signs = signs; a.mode = mode; a.gw_out = gw_out; a.overwrite = overwrite; a.am = am; a.am_out = am_out;
  a.gw_dtype = gw_fp32 ? at::kFloat : at::kBFloat16;
  if (gw_out) {
    require_cuda(gw_out);
    REQUIRE(gw_out->dim() == 2 && gw_out->size(0) == gy.size(1) && gw_out->size(1) == a.Kw && gw_out->scalar_type() == at::kFloat &&
                gw_out->stride(1) == 1, "linear_bwd: gw_out is fp32 [N, K]");
  }
  return backward_core(gy, wt, xt, seed, seed_cols, a);
}

// Offsets inside the one buffer a forward pass keeps for its backward pass.
struct Kept {
  PackedOut xt, wt;
  Kept(Carver& c, int64_t T, int64_t K, int64_t N, bool keep_x, bool keep_w) {
    if (keep_x) xt = carve_packed(c, K, T);
    if (keep_w) wt = carve_packed(c, K, N);
  }
};

struct Q3 { Tensor d, s, gs; };
Q3 q_of(py::handle q) {
  return {py::cast<Tensor>(q.attr("d")), py::cast<Tensor>(q.attr("s")), py::cast<Tensor>(q.attr("gs"))};
}

struct LinearNode : torch::autograd::Node {
  torch::autograd::SavedVariable w, kept;       // the weight: only so that an in-place change of it is noticed
  int64_t T, K, N;
  unsigned lid, signs;
  bool keep_x, keep_w;
  PyObject* cache = nullptr;                    // the layer's WeightCache, or null

  ~LinearNode() override {
    if (cache && Py_IsInitialized()) {
      py::gil_scoped_acquire gil;
      Py_DECREF(cache);
    }
  }
  std::string name() const override { return "FP4LinearFnBackward"; }
  void release_variables() override {
    std::lock_guard<std::mutex> lock(mutex_);
    w.reset_data(); kept.reset_data();
  }

  // Exceptions leave through the autograd engine, not through this module: as Python errors of their types
  torch::autograd::variable_list apply(torch::autograd::variable_list&& grads) override {
    try {
      return backward(std::move(grads));
    } catch (const AssertionFailure& e) {
      throw_as(PyExc_AssertionError, e.what());
    } catch (const LibraryError& e) {
      throw_as(error_class.ptr(), e.what());
    } catch (py::error_already_set& e) {
      py::gil_scoped_acquire gil;
      e.restore();
      throw_python_error_set();
    }
  }

 private:
  [[noreturn]] static void throw_python_error_set() {
    python_error error;
    error.persist();
    throw std::move(error);
  }
  [[noreturn]] static void throw_as(PyObject* type, const char* what) {
    py::gil_scoped_acquire gil;
    PyErr_SetString(type, what);
    throw_python_error_set();
  }

  torch::autograd::variable_list backward(torch::autograd::variable_list&& grads) {
    torch::autograd::variable_list out(2);
    if (!grads[0].defined()) return out;
    at::NoGradGuard no_grad;
    Tensor buf;
    {
      std::lock_guard<std::mutex> lock(mutex_);   // another thread's backward pass may free the graph
      w.unpack(getptr());                         // raises when the graph was freed or the weight changed in place
      buf = kept.unpack(getptr());
    }
    BackwardArgs a;
    a.K = a.Kw = K; a.signs = signs;
    a.want_x = task_should_compute_output(0);
    a.want_w = task_should_compute_output(1);
    if (!a.want_x && !a.want_w) return out;
    unsigned seed;
    Q3 cached;
    {
      // the switches as they stand when the backward pass runs
      py::gil_scoped_acquire gil;
      const py::object s = lin_ctx.attr("seed");
      seed = (unsigned)PyLong_AsUnsignedLongLongMask(s.ptr()) * 1000003u + lid * 7919u;
      if (PyErr_Occurred()) throw py::error_already_set();
      const py::object dtype = lin_ctx.attr("wgrad_dtype");
      a.gw_dtype = THPDtype_Check(dtype.ptr()) ? reinterpret_cast<THPDtype*>(dtype.ptr())->scalar_type : at::kByte;
      a.mode = py::cast<int>(nvq_module.attr("SR_MODE"));
      if (cache && a.want_x) cached = q_of(py::handle(cache).attr("qt"));
    }
    REQUIRE(a.gw_dtype == at::kFloat || a.gw_dtype == at::kBFloat16, "LinCtx.wgrad_dtype: float32 or bfloat16");
    Carver c{static_cast<char*>(buf.data_ptr())};
    const Kept k(c, T, K, N, keep_x, keep_w);
    const Packed wt = cached.d.defined() ? packed_of(cached.d, cached.s, cached.gs, K, N, "cached transposed weight") : k.wt.in(N);
    const Tensor gy = grads[0].contiguous();
    std::tie(out[0], out[1]) = backward_core(gy, wt, k.xt.in(T), Seed(seed), Seed(seed ^ 0x5bd1e995u), a);
    return out;
  }
};

// The layer on x [T, K], w [N, K] -> y [T, N].  With `cache` the quantized weight is taken from it, else W is quantized
// here: both orientations in one pass when the backward pass will want W^T (one amax and one read of W instead of two
// of each).  Without gradients only the row operand of x is produced.
Tensor linear_apply(unsigned signs, const Tensor& x_, const OptTensor& w_opt, py::handle lid, py::handle cache) {
  require_cuda(x_);
  const Tensor w_ = w_opt.value_or(Tensor());
  if (torch::autograd::isFwGradDefined(x_) || torch::autograd::isFwGradDefined(w_opt)) {
    PyErr_SetString(PyExc_NotImplementedError, "the NVFP4 linear has no jvp: forward-mode AD is not supported");
    throw py::error_already_set();
  }
  const bool cached = !cache.is_none();
  const bool grad = at::GradMode::is_enabled();
  const bool need_x = grad && x_.requires_grad(), need_w = grad && w_.defined() && w_.requires_grad();
  REQUIRE(x_.dim() == 2 && x_.scalar_type() == at::kBFloat16 && x_.stride(1) == 1, "linear: x is bf16 [T, K] with contiguous rows");
  const int64_t T = x_.size(0), K = x_.size(1);
  REQUIRE(T % 128 == 0 && K % 128 == 0, shape_of(T, K));
  const unsigned layer = (unsigned)PyLong_AsUnsignedLongLongMask(lid.ptr());
  if (PyErr_Occurred()) throw py::error_already_set();
  Q3 cq;
  if (cached) cq = q_of(cache.attr("q"));
  Tensor y;
  std::shared_ptr<LinearNode> node;
  Tensor kept_buf;
  int64_t N;
  {
    py::gil_scoped_release unlocked;
    at::NoGradGuard no_grad;
    const Tensor x = x_.detach();
    Packed qw;
    Tensor w;
    if (cached) {
      N = cq.d.size(0);
      qw = packed_of(cq.d, cq.s, cq.gs, N, K, "cached weight");
    } else {
      REQUIRE(w_.defined(), "linear: no weight");
      require_cuda(w_);
      REQUIRE(w_.dim() == 2 && w_.scalar_type() == at::kBFloat16, "quant_w2d: a bf16 matrix");
      w = w_.contiguous();
      N = w.size(0);
      REQUIRE(N % 128 == 0 && w.size(1) == K, shape_of(N, w.size(1)));
    }
    const bool keep_w = !cached && need_x;
    Carver ksize;
    Kept(ksize, T, K, N, need_w, keep_w);
    if (need_x || need_w) kept_buf = empty({(int64_t)ksize.used}, at::kByte, x);
    Carver kc{kept_buf.defined() ? static_cast<char*>(kept_buf.data_ptr()) : nullptr};
    const Kept kept(kc, T, K, N, need_w, keep_w);

    PackedOut wq;
    Tensor scratch;
    if (!cached) {
      auto carve = [&](Carver& c) {
        float* am_w = c.take<float>(4);
        wq = carve_packed(c, N, K);
        return am_w;
      };
      Carver size;
      carve(size);
      scratch = empty({(int64_t)size.used}, at::kByte, x);
      Carver c{static_cast<char*>(scratch.data_ptr())};
      const float* amw = passing_amax(w, carve(c));
      if (keep_w) wq.gs = kept.wt.gs;         // both orientations share one tensor scale, which the backward pass reads
      run_w2d(w, &wq, keep_w ? &kept.wt : nullptr, amw);
      qw = wq.in(K);
    }
    y = forward_core(x, nullptr, nullptr, qw, N, need_w ? &kept.xt : nullptr, signs);
  }
  if (need_x || need_w) {
    node = std::shared_ptr<LinearNode>(new LinearNode(), torch::autograd::deleteNode);
    node->set_next_edges(torch::autograd::collect_next_edges(x_, w_));
    node->T = T; node->K = K; node->N = N;
    node->lid = layer;
    node->signs = signs; node->keep_x = need_w; node->keep_w = !cached && need_x;
    if (cached) { node->cache = cache.ptr(); Py_INCREF(node->cache); }
    node->w = torch::autograd::SavedVariable(w_, false);
    node->kept = torch::autograd::SavedVariable(kept_buf, false);
    torch::autograd::set_history(y, node);
  }
  return y;
}

// ------------------------------------------------------------------------------------------ fp4ops operators
// max|x| as FP32 [1]: one kernel for contiguous bf16 and FP32, torch's reduction for everything else
Tensor k_amax(const Tensor& x) {
  at::NoGradGuard no_grad;
  const bool bf16 = x.scalar_type() == at::kBFloat16, f32 = x.scalar_type() == at::kFloat;
  if (x.is_cuda() && (bf16 || f32) && x.is_contiguous() && x.numel() > 0 && x.numel() % (bf16 ? 8 : 4) == 0 &&
      (bf16 || (reinterpret_cast<uintptr_t>(x.const_data_ptr()) & 15u) == 0)) {
    Tensor out = empty({1}, at::kFloat, x);
    if (bf16) run_amax(x, out.data_ptr<float>());
    else check(lib.nvfp4_amax_f32(static_cast<const float*>(x.const_data_ptr()), x.numel(), out.data_ptr<float>(), stream()), "amax");
    return out;
  }
  return x.abs().amax().to(at::kFloat).reshape({1});
}
Tensor k_amax_or(const OptTensor& am, const Tensor& x) { return am ? *am : k_amax(x); }

// Row-major scales [R, C16]; where whole swizzled tiles exist the same buffer also holds the swizzled bytes, which the
// quantizers then write in the same pass (`sw`: what the tensor core reads, so that a GEMM on the result has nothing
// left to convert).
struct LinearScales {
  Tensor s;
  OptTensor sw;
  int layout;
  LinearScales(int64_t R, int64_t C, bool both, const Tensor& like) : layout(both ? NVFP4_SCALES_BOTH : NVFP4_SCALES_LINEAR) {
    const int64_t n = R * (C / 16);
    if (both) {
      const Tensor buf = empty({2 * n}, at::kByte, like);
      s = buf.as_strided({R, C / 16}, {C / 16, 1}, 0);
      sw = buf.as_strided({n}, {1}, n);
    } else {
      s = empty({R, C / 16}, at::kByte, like);
    }
  }
};
bool whole_tiles(int64_t R, int64_t C) { return R % 128 == 0 && C % 128 == 0 && R > 0 && C > 0; }

using Scaled = std::tuple<Tensor, Tensor, Tensor, OptTensor>;          // d, s, amax, swizzled s
Scaled k_quant_rows(const Tensor& x_, int mode, const Seed& seed, const OptTensor& am_) {
  require_cuda(x_);
  at::NoGradGuard no_grad;
  REQUIRE(x_.dim() == 2 && x_.scalar_type() == at::kBFloat16 && x_.size(1) % 16 == 0, "quant_rows: a bf16 matrix, columns a multiple of 16");
  const Tensor x = x_.contiguous();
  const int64_t R = x.size(0), C = x.size(1);
  const Tensor am = k_amax_or(am_, x);
  Tensor d = empty({R, C / 2}, at::kByte, x);
  LinearScales s(R, C, whole_tiles(R, C), x);
  check(lib.nvfp4_quant_rows(x.const_data_ptr(), C, (int)R, (int)C, d.data_ptr(), s.s.data_ptr(), s.layout, word(am), nullptr, mode,
                             seed.host, seed.dev, stream()), "quant_rows");
  return {d, s.s, am, s.sw};
}

Scaled k_quant_cols_rht(const Tensor& x_, unsigned signs, int mode, const Seed& seed, const OptTensor& am_) {
  require_cuda(x_);
  at::NoGradGuard no_grad;
  const Tensor x = x_.contiguous();
  REQUIRE(x.dim() == 2 && x.scalar_type() == at::kBFloat16 && x.size(0) % 16 == 0 && x.size(1) % 8 == 0,
          "quant_cols_rht: a bf16 matrix, rows a multiple of 16, columns of 8");
  const int64_t M = x.size(0), C = x.size(1);
  const Tensor am = k_amax_or(am_, x);
  Tensor d = empty({C, M / 2}, at::kByte, x);
  LinearScales s(C, M, whole_tiles(C, M), x);
  check(lib.nvfp4_quant_cols_rht(x.const_data_ptr(), (int)M, (int)C, d.data_ptr(), s.s.data_ptr(), s.layout, word(am), nullptr, signs,
                                 mode, seed.host, seed.dev, stream()), "quant_cols_rht");
  return {d, s.s, am, s.sw};
}

std::pair<Scaled, Scaled> k_quant_rows_cols_rht(const Tensor& x, unsigned signs, int mode, const Seed& seed, const Seed& seed_cols, const OptTensor& am_) {
  require_cuda(x);
  at::NoGradGuard no_grad;
  REQUIRE(x.dim() == 2 && x.scalar_type() == at::kBFloat16 && x.stride(1) == 1, "quant_rows_cols_rht: a bf16 matrix with contiguous rows");
  const int64_t M = x.size(0), C = x.size(1);
  REQUIRE(M % 128 == 0 && C % 64 == 0, shape_of(M, C));
  const bool both = whole_tiles(M, C);
  Tensor dr = empty({M, C / 2}, at::kByte, x), dc = empty({C, M / 2}, at::kByte, x);
  LinearScales sr(M, C, both, x), sc(C, M, both, x);
  Tensor am;
  int launched = 0;
  if (am_ || !x.is_contiguous()) {
    am = k_amax_or(am_, x);
  } else {
    am = empty({1}, at::kFloat, x);
    check(lib.nvfp4_quant_tile_amax(x.const_data_ptr(), x.stride(0), (int)M, (int)C, dr.data_ptr(), sr.s.data_ptr(), dc.data_ptr(),
                                    sc.s.data_ptr(), sr.layout, am.data_ptr<float>(), &launched, nullptr, nullptr, signs, mode, seed.host,
                                    seed_cols.host, seed.dev, seed_cols.dev, stream()), "quant_tile_amax");
    if (!launched) am = k_amax(x);
  }
  if (!launched)
    check(lib.nvfp4_quant_tile(x.const_data_ptr(), x.stride(0), (int)M, (int)C, dr.data_ptr(), sr.s.data_ptr(), dc.data_ptr(),
                               sc.s.data_ptr(), sr.layout, word(am), nullptr, nullptr, signs, mode, seed.host, seed_cols.host,
                               seed.dev, seed_cols.dev, stream()), "quant_tile");
  return {{dr, sr.s, am, sr.sw}, {dc, sc.s, am, sc.sw}};
}

Tensor k_swizzle(const Tensor& s, const OptTensor& out_) {
  const int64_t R = s.size(0), C16 = s.size(1);
  REQUIRE(R % 128 == 0 && C16 % 4 == 0, shape_of(R, C16));
  Tensor out = out_ ? *out_ : empty({R * C16}, at::kByte, s);
  check(lib.nvfp4_swizzle_scales(s.const_data_ptr(), s.stride(0), (int)R, (int)C16, out.data_ptr(), stream()), "swizzle_scales");
  return out;
}

// Buffers of one weight: (d, s, sw) of W and of W^T and the shared amax.
std::tuple<Tensor, Tensor, OptTensor, Tensor, Tensor, OptTensor, Tensor> k_w2d_buffers(const Tensor& w) {
  require_cuda(w);
  REQUIRE(w.dim() == 2 && w.scalar_type() == at::kFloat && w.size(0) % 16 == 0 && w.size(1) % 16 == 0, "quant_w2d: an FP32 matrix, sides multiples of 16");
  const int64_t N = w.size(0), K = w.size(1);
  const bool both = whole_tiles(N, K);
  LinearScales s(N, K, both, w), st(K, N, both, w);
  return {empty({N, K / 2}, at::kByte, w), s.s, s.sw, empty({K, N / 2}, at::kByte, w), st.s, st.sw, empty({1}, at::kFloat, w)};
}

void k_quant_w2d(const Tensor& w_, const Tensor& d, const Tensor& s, const OptTensor& sw, const Tensor& dt, const Tensor& st,
                 const OptTensor& stw, const Tensor& am) {
  require_cuda(w_);
  at::NoGradGuard no_grad;
  REQUIRE(w_.dim() == 2 && w_.scalar_type() == at::kFloat && w_.size(0) % 16 == 0 && w_.size(1) % 16 == 0, "quant_w2d: an FP32 matrix, sides multiples of 16");
  const Tensor w = w_.contiguous();
  const int64_t N = w.size(0), K = w.size(1);
  if (w.numel() > 0 && w.numel() % 4 == 0 && (reinterpret_cast<uintptr_t>(w.const_data_ptr()) & 15u) == 0)
    check(lib.nvfp4_amax_f32(static_cast<const float*>(w.const_data_ptr()), w.numel(), static_cast<float*>(am.data_ptr()), stream()), "amax");
  else
    am.copy_(k_amax(w));
  // the kernel writes both layouts where the swizzled bytes follow the row-major ones
  auto follows = [](const Tensor& a, const OptTensor& b) {
    return b && static_cast<const char*>(a.const_data_ptr()) + a.numel() == static_cast<const char*>(b->const_data_ptr());
  };
  const bool both = whole_tiles(N, K) && follows(s, sw) && follows(st, stw);
  check(lib.nvfp4_quant_w2d(w.const_data_ptr(), NVFP4_DTYPE_FP32, (int)N, (int)K, d.data_ptr(), s.data_ptr(), dt.data_ptr(),
                            st.data_ptr(), both ? NVFP4_SCALES_BOTH : NVFP4_SCALES_LINEAR, word(am), nullptr, stream()), "quant_w2d");
  if (!both) {
    if (sw) k_swizzle(s, sw);
    if (stw) k_swizzle(st, stw);
  }
}

// a [M, K], b [N, K] with row-major scales and, where they are known, swizzled ones
Tensor k_gemm(const Tensor& ad, const Tensor& as, const OptTensor& asw, const Tensor& aam, float ak, const Tensor& bd, const Tensor& bs,
              const OptTensor& bsw, const Tensor& bam, float bk, const OptTensor& out_, int splitk) {
  require_cuda(ad); require_cuda(bd);
  at::NoGradGuard no_grad;
  const int64_t M = ad.size(0), N = bd.size(0), K = as.size(1) * 16;
  REQUIRE(M % 128 == 0 && N % 128 == 0 && K % 128 == 0, shape_of(M, N) + ", " + std::to_string(K));
  const bool fp32 = splitk != 1 || out_;
  Tensor out;
  if (!fp32) {
    out = empty({M, N}, at::kBFloat16, ad);
  } else {
    out = out_ ? *out_ : empty({M, N}, at::kFloat, ad);       // a fresh result is stored, the library slices K as it sees fit
    REQUIRE(out.scalar_type() == at::kFloat && out.stride(1) == 1, "gemm: out is FP32 with contiguous rows");
  }
  // scales of the operand's rows; more may be there (a slice of the codes with the scales of the whole)
  auto swizzled = [](const Tensor& s, const OptTensor& sw, int64_t rows) {
    return sw ? *sw : k_swizzle(s.size(0) == rows ? s : s.narrow(0, 0, rows), std::nullopt);
  };
  const Tensor sa = swizzled(as, asw, M), sb = swizzled(bs, bsw, N);
  check(lib.nvfp4_gemm(ad.const_data_ptr(), sa.const_data_ptr(), ad.stride(0), bd.const_data_ptr(), sb.const_data_ptr(), bd.stride(0),
                       out.data_ptr(), fp32 ? NVFP4_DTYPE_FP32 : NVFP4_DTYPE_BF16, out.stride(0), (int)M, (int)N, (int)K,
                       NVFP4_ALPHA_AMAX, word(aam), word(bam), ak, bk, fp32 && out_, fp32 && !out_ && splitk > 1 ? 0 : splitk, status_word(ad), stream()), "gemm");
  return out;
}

// ------------------------------------------------------------------------------------------ operand emitters
const unsigned* words(const OptTensor& t) { return static_cast<const unsigned*>(cptr(t)); }

void e_rows(const Tensor& x, const Tensor& d, const Tensor& s, const Tensor& rs, const OptTensor& rng, int sr, unsigned salt) {
  require_cuda(x); require_cuda(d); require_cuda(s); require_cuda(rs);
  const int64_t T = x.size(0), C = x.size(1);
  REQUIRE(x.scalar_type() == at::kBFloat16 && x.stride(1) == 1 && C % 256 == 0, "row_emit: bf16, contiguous rows, columns a multiple of 256");
  REQUIRE(T % 128 == 0, std::to_string(T));
  if (sr) REQUIRE(rng && rng->is_cuda() && rng->element_size() == 4, "row_emit: stochastic rounding needs rng");
  check(lib.nvfp4_emit_rows(x.const_data_ptr(), x.stride(0), (int)T, (int)C, d.data_ptr(), s.data_ptr(), static_cast<float*>(rs.data_ptr()),
                            sr, words(rng), salt, stream()), "emit_rows");
}

void e_cols(const Tensor& x, const Tensor& d, const Tensor& s, const Tensor& use, const Tensor& cur, const Tensor& rng, int sr, unsigned salt) {
  require_cuda(x); require_cuda(d); require_cuda(s); require_cuda(use); require_cuda(cur); require_cuda(rng);
  const int64_t M = x.size(0), C = x.size(1);
  REQUIRE(x.scalar_type() == at::kBFloat16 && x.stride(1) == 1 && M % 256 == 0 && C % 64 == 0, "col_emit: bf16, contiguous rows, tokens a multiple of 256");
  REQUIRE(C % 128 == 0, std::to_string(C));          // swizzled scale tiles of 128 columns are written whole
  REQUIRE(rng.element_size() == 4 && rng.numel() >= 2 && cur.element_size() == 4, "col_emit: rng holds two 32-bit words, amax_cur one");
  check(lib.nvfp4_emit_cols(x.const_data_ptr(), x.stride(0), (int)M, (int)C, d.data_ptr(), s.data_ptr(), word(use),
                            static_cast<unsigned*>(cur.data_ptr()), sr, words(rng), salt, stream()), "emit_cols");
}

void e_rms(const Tensor& x, const Tensor& w, const OptTensor& d, const OptTensor& s, const OptTensor& rs, const OptTensor& h,
           const OptTensor& rstd, const OptTensor& y, const OptTensor& ys, const OptTensor& ygw, const OptTensor& xout, float eps) {
  const int64_t T = x.size(0), D = x.size(1);
  REQUIRE(x.scalar_type() == at::kBFloat16 && x.is_contiguous() && w.scalar_type() == at::kBFloat16 && w.numel() == D, "rms_emit: x, w");
  require_cuda(x); require_cuda(w);
  if (y) {
    REQUIRE(y->sizes() == x.sizes() && y->is_contiguous() && ys && ygw && xout, "rms_emit: y comes with ys, ygw and xout");
    REQUIRE(xout->sizes() == x.sizes() && xout->is_contiguous() && ys->scalar_type() == at::kFloat && ygw->scalar_type() == at::kFloat, "rms_emit: xout, ys, ygw");
  }
  if (d) REQUIRE(T % 128 == 0 && d->size(0) == T && d->size(1) == D / 2, "rms_emit: q");
  if (h) REQUIRE(h->sizes() == x.sizes() && h->is_contiguous() && h->scalar_type() == at::kBFloat16, "rms_emit: h");
  auto p = [](const OptTensor& t) { return t ? t->data_ptr() : nullptr; };
  check(lib.nvfp4_rms_emit(x.const_data_ptr(), cptr(y), static_cast<const float*>(cptr(ys)), static_cast<const float*>(cptr(ygw)), p(xout),
                           w.const_data_ptr(), p(h), p(d), p(s), static_cast<float*>(p(rs)), static_cast<float*>(p(rstd)), (int)T, (int)D,
                           eps, stream()), "rms_emit");
}

void e_swiglu(const Tensor& gu, const Tensor& rs_in, const Tensor& gw, const OptTensor& d, const OptTensor& s, const OptTensor& rs,
              const OptTensor& a, const OptTensor& a_f32) {
  const int64_t T = gu.size(0), F2 = gu.size(1), F = F2 / 2;
  REQUIRE(gu.scalar_type() == at::kBFloat16 && gu.is_contiguous() && F2 % 512 == 0, "swiglu_emit: gu");
  REQUIRE(rs_in.scalar_type() == at::kFloat && rs_in.numel() == T && gw.scalar_type() == at::kFloat, "swiglu_emit: rs_in, gw");
  require_cuda(gu); require_cuda(rs_in); require_cuda(gw);
  if (d) REQUIRE(T % 128 == 0 && d->size(0) == T && d->size(1) == F / 2, "swiglu_emit: q");
  auto p = [](const OptTensor& t) { return t ? t->data_ptr() : nullptr; };
  check(lib.nvfp4_swiglu_emit(gu.const_data_ptr(), word(rs_in), word(gw), (int)F, p(a), static_cast<float*>(p(a_f32)), p(d), p(s),
                              static_cast<float*>(p(rs)), (int)T, stream()), "swiglu_emit");
}

void e_mom(const Tensor& m, const Tensor& g, const Tensor& alpha, float scale, const Tensor& rng, unsigned salt) {
  const int64_t n = m.numel();
  REQUIRE(n % 8 == 0 && g.numel() == n && m.scalar_type() == at::kBFloat16 && g.scalar_type() == at::kBFloat16, "mom_acc: bf16 m and g of one size");
  REQUIRE(m.is_contiguous() && g.is_contiguous() && alpha.scalar_type() == at::kFloat, "mom_acc: contiguous m and g, FP32 alpha");
  require_cuda(m); require_cuda(g); require_cuda(alpha); require_cuda(rng);
  check(lib.nvfp4_mom_acc(m.data_ptr(), g.const_data_ptr(), word(alpha), scale, n, words(rng), salt, stream()), "mom_acc");
}

// raw = A B^T with block scales only (alpha_mode ONE), or times the words of `pa`, `pb`
Tensor e_mm(const Tensor& ad, const Tensor& as, const Tensor& bd, const Tensor& bs, bool fp32, int alpha_mode, const OptTensor& pa,
            const OptTensor& pb, const OptTensor& out, bool accumulate, int splitk) {
  auto bytes = [](const Tensor& t) { return t.element_size() == 1 ? t : t.view(at::kByte); };     // codes in wider words
  return gemm(bytes(ad), as, bytes(bd), bs, out, fp32, alpha_mode, pa, pb, 1.f, 1.f, accumulate, splitk, "gemm");
}

void bind(const py::dict& addresses, py::object error, py::object lin, py::object nvq, py::object status) {
#define X(name) lib.name = reinterpret_cast<decltype(lib.name)>(py::cast<uintptr_t>(addresses[#name]));
  NVFP4_API(X)
#undef X
  error_class = error.release();
  lin_ctx = lin.release();
  nvq_module = nvq.release();
  status_word_fn = status.release();
}

}  // namespace

namespace pybind11::detail {
template <> struct type_caster<Seed> {
  PYBIND11_TYPE_CASTER(Seed, const_name("Seed"));
  bool load(handle src, bool) {
    value = Seed(src);
    return true;
  }
};
}  // namespace pybind11::detail

PYBIND11_MODULE(_host, m) {
  py::register_exception_translator([](std::exception_ptr p) {
    try {
      if (p) std::rethrow_exception(p);
    } catch (const AssertionFailure& e) {
      PyErr_SetString(PyExc_AssertionError, e.what());
    } catch (const LibraryError& e) {
      PyErr_SetString(error_class.ptr(), e.what());
    }
  });
  m.attr("built_for") = NVFP4_HOST_TAG;
  m.def("bind", &bind);
  m.def("entry_points", [] {
    py::list names;
#define X(name) names.append(#name);
    NVFP4_API(X)
#undef X
    return names;
  });
  // Launches wait while the queue of the stream is full, and allocations may: other Python threads go on meanwhile.
  // (linear_apply, which reads Python objects, lets go of the interpreter lock by itself.)
  const py::call_guard<py::gil_scoped_release> unlocked;
  m.def("amax", &nvq_amax, unlocked);
  m.def("quant_rows", &nvq_quant_rows, unlocked);
  m.def("quant_cols_rht", &nvq_quant_cols_rht, unlocked);
  m.def("quant_rows_cols_rht", &nvq_quant_rows_cols_rht, unlocked);
  m.def("quant_w2d", &nvq_quant_w2d, unlocked);
  m.def("quant_w2d_into", &nvq_quant_w2d_into, unlocked);
  m.def("mm", &nvq_mm, unlocked);
  m.def("linear_fwd", &linear_fwd, unlocked);
  m.def("linear_bwd", &linear_bwd, unlocked);
  m.def("linear_apply", &linear_apply, py::arg(), py::arg(), py::arg(), py::arg(), py::arg() = py::none());
  m.def("k_amax", &k_amax, unlocked);
  m.def("k_quant_rows", &k_quant_rows, unlocked);
  m.def("k_quant_cols_rht", &k_quant_cols_rht, unlocked);
  m.def("k_quant_rows_cols_rht", &k_quant_rows_cols_rht, unlocked);
  m.def("k_swizzle", &k_swizzle, unlocked);
  m.def("k_w2d_buffers", &k_w2d_buffers, unlocked);
  m.def("k_quant_w2d", &k_quant_w2d, unlocked);
  m.def("k_gemm", &k_gemm, unlocked);
  m.def("e_rows", &e_rows, unlocked);
  m.def("e_cols", &e_cols, unlocked);
  m.def("e_rms", &e_rms, unlocked);
  m.def("e_swiglu", &e_swiglu, unlocked);
  m.def("e_mom", &e_mom, unlocked);
  m.def("e_mm", &e_mm, unlocked);
}

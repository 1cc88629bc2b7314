// Host side of an attention call in C++: argument checks, output allocation, the launches of libjvpfa.so and the
// autograd graph around them, behind one Python entry point (`attend`).
//
// What bounds the calls it serves is host time, not the GPU: up to a few hundred microseconds of kernels, the pass of a
// program was the Python layer's.  Measured on a B200 machine before and after, whole passes through the public API:
// attention() at B2 H12 L32 D64 43 -> 9 us, fwd_dual on forward-AD dual tensors at L256 96 -> 28 us, fwd_dual and the
// gradients through both outputs under torch.func.jvp (fp32, B2 H4 L256 D64) 493 -> 207 us, of which torch.func.jvp itself
// takes some 150.
//
// Graph: one node with two outputs, O and tO.  Autograd hands it both cotangents at once, so a loss on both outputs is
// one backward launch.  Under create_graph the gradient through O is a node that can be differentiated once more (the
// Hessian-vector product of upstream's missing double backward); the gradient through tO refuses a second differentiation.
// The tangent rides on O as its forward-mode gradient, set directly instead of through make_dual's view.
//
// CUDA tensors go straight to the library.  For tensors of another device the launch is handed back to the Python
// module's _launch_fwd / _launch_bwd (the CPU suite puts its oracle there), so that its tests run this graph.
// The Functions of the Python module serve what this layer declines: nested functorch transforms, cotangents that belong to
// one, JVPAttn.apply, and calls that are refused.
#include <ATen/ATen.h>
#include <ATen/cuda/EmptyTensor.h>
#include <ATen/functorch/DynamicLayer.h>
#include <ATen/functorch/TensorWrapper.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <cuda_runtime_api.h>
#include <torch/csrc/autograd/function.h>
#include <torch/csrc/autograd/functions/utils.h>
#include <torch/csrc/autograd/saved_variable.h>
#include <torch/csrc/utils/pybind.h>

#include <atomic>
#include <memory>
#include <optional>
#include <string>
#include <vector>

#include "jvpfa.h"

namespace py = pybind11;
using at::Tensor;
using torch::autograd::Node;
using torch::autograd::SavedVariable;
using torch::autograd::variable_list;

namespace {

// Process-wide switches of the Python module (its attributes of the same meaning are forwarded here when they are set).
std::atomic<int> g_impl{JVPFA_IMPL_AUTO};
std::atomic<bool> g_single_pass{true};

py::object& python_module() {
  static py::object* m = new py::object(py::module_::import("jvp_flash_attention_b200.jvp_attention"));  // lives as long as the process
  return *m;
}

// The kernel-side mask description, built once per mask.  `spec` is the Python object it was made from.
struct MaskDesc {
  jvpfa_mask c{};
  Tensor tensor, tile_live, tile_live_t;
  std::vector<int32_t> kv_len;  // JVPFA_MASK_KVLEN: the lengths on the host
  double dead;                  // with tile bitmaps: the share of tiles that verification found without a true entry
  std::shared_ptr<py::object> spec;

  MaskDesc(int kind, int bias_dtype, std::optional<Tensor> t, std::array<int64_t, 4> strides, std::optional<Tensor> live,
           std::optional<Tensor> live_t, std::vector<int32_t> kv_len_, double dead_, py::object spec_)
      : kv_len(std::move(kv_len_)),
        dead(dead_),
        spec(new py::object(std::move(spec_)), [](py::object* o) {
          py::gil_scoped_acquire gil;
          delete o;
        }) {
    c.kind = kind;
    c.bias_dtype = bias_dtype;
    for (int i = 0; i < 4; ++i) c.stride[i] = strides[i];
    if (t) tensor = *t;
    if (live) tile_live = *live;
    if (live_t) tile_live_t = *live_t;
    if (kind == JVPFA_MASK_KVLEN)
      c.kv_len = static_cast<const int32_t*>(tensor.data_ptr());
    else if (kind == JVPFA_MASK_BOOL || kind == JVPFA_MASK_BIAS)
      c.ptr = tensor.data_ptr();
  }
};
using MaskPtr = std::shared_ptr<MaskDesc>;

// What a call's backward has to know besides its tensors.
struct Call {
  MaskPtr mask;
  double scale;
  bool tf32;  // fp32 tensors: one TF32 product instead of three, recorded so that the backward recomputes what the forward saw
  // fp32: the tcgen05 kernels, which recompute the scores as the tcgen05 forward forms them.  Asked for where whatever may be asked
  // of the call's backward is theirs, and kept for that backward if the forward ran on them.  (The register-tiled kernels, whose
  // scores are off in their own way, keep the forward whose lse is off in the same.)
  bool parts = false;
  // A boolean mask as bits, by rows and transposed: the form the 16-bit tensor-core kernels read best, made by this call for
  // its forward and backward (pack_mask).
  Tensor bits, bits_t;
  Tensor tiles;  // fp32: both tile bitmaps, made by this call's forward for its register-tiled launches (make_tiles)

  void drop_tensors() { bits = bits_t = tiles = Tensor(); }
};

bool is_wrapped(const Tensor& x) {
  return x.key_set().has(c10::DispatchKey::FuncTorchGradWrapper) || x.key_set().has(c10::DispatchKey::FuncTorchBatched);
}

// The tensor under functorch's wrappers.
Tensor unwrap(Tensor x) {
  while (x.defined()) {
    auto* w = at::functorch::maybeGetTensorWrapper(x);
    if (!w) break;
    x = Tensor(w->value());
  }
  return x;
}

const void* data(const Tensor& t) { return t.defined() ? t.const_data_ptr() : nullptr; }

int dtype_of(const Tensor& t, bool tf32) {
  switch (t.scalar_type()) {
    case at::kBFloat16:
      return JVPFA_BF16;
    case at::kHalf:
      return JVPFA_FP16;
    case at::kFloat:
      return tf32 ? JVPFA_FP32_TF32 : JVPFA_FP32;
    default:
      return -1;
  }
}

void check_status(int rc, const char* what) {
  if (rc == JVPFA_OK) return;
  std::string msg = std::string(what) + " failed: [" + std::to_string(rc) + "] " + jvpfa_strerror(rc);
  const std::string cuda = jvpfa_last_cuda_error();
  if (!cuda.empty()) msg += " | " + cuda;
  throw std::runtime_error(msg);
}

// Allocation without the dispatcher: these run inside functorch levels as well, and a call makes up to nine of them.
Tensor empty(at::IntArrayRef sizes, at::ScalarType dtype, at::Device device) {
  return Tensor(at::detail::empty_cuda(sizes, dtype, device, std::nullopt));
}

// Operators on plain tensors while a functorch level may be active: without its dispatch keys.
struct NoFunctorch {
  c10::impl::ExcludeDispatchKeyGuard guard;
  NoFunctorch()
      : guard(c10::DispatchKeySet({c10::DispatchKey::FuncTorchDynamicLayerFrontMode, c10::DispatchKey::FuncTorchDynamicLayerBackMode})) {}
};

struct NoFunctorchScope {  // the same as a Python context manager
  std::optional<NoFunctorch> guard;
};

// Common (batch, head, row) strides of tensors the kernels can read in place.  True with st all zero: row-major.
bool common_layout(std::initializer_list<const Tensor*> ts, int64_t* st) {
  bool dense = true;
  for (auto* t : ts) dense = dense && (!t->defined() || t->is_contiguous());
  st[0] = st[1] = st[2] = 0;
  if (dense) return true;
  const auto ref = (*ts.begin())->strides();
  for (auto* t : ts) {
    if (!t->defined()) continue;
    if (t->strides() != ref || ref[3] != 1 || (reinterpret_cast<uintptr_t>(t->const_data_ptr()) & 15u) != 0) return false;
    for (int d = 0; d < 3; ++d)
      if (ref[d] <= 0 || (ref[d] & 7) != 0) return false;
  }
  for (int d = 0; d < 3; ++d) st[d] = ref[d];
  return true;
}

struct FwdResult {
  Tensor o, to, lse, mu;
  bool parts = false;  // fp32: there was a workspace for the tcgen05 kernels (Call::parts of a backward from this lse and mu)
};
using Grads = std::array<Tensor, 3>;

// The six inputs as plain tensors, copied to row-major only when they share no layout the kernels read in place.
struct Inputs {
  Tensor q, k, v, tq, tk, tv;
  int64_t st[3];

  Inputs(const Tensor& q_, const Tensor& k_, const Tensor& v_, const Tensor& tq_, const Tensor& tk_, const Tensor& tv_)
      : q(q_), k(k_), v(v_), tq(tq_), tk(tk_), tv(tv_) {
    if (!common_layout({&q, &k, &v, &tq, &tk, &tv}, st)) make_dense();
  }
  void make_dense() {
    NoFunctorch nf;
    at::AutoDispatchBelowADInplaceOrView below;
    for (Tensor* t : {&q, &k, &v, &tq, &tk, &tv})
      if (t->defined()) *t = t->contiguous();
    st[0] = st[1] = st[2] = 0;
  }
};

// ---- masks -----------------------------------------------------------------------------------------------------------
// The lengths of a key padding where they are known on the host.
const int32_t* host_lengths(const MaskDesc& m, int B) { return m.kv_len.size() == (size_t)B ? m.kv_len.data() : nullptr; }

// Whether the launches of a call may take the forms that only the 16-bit tensor-core kernels read.
bool takes_16_bit_forms(const Tensor& q) { return q.is_cuda() && q.scalar_type() != at::kFloat && g_impl != JVPFA_IMPL_GENERIC; }

// A bias of the tensors' type with its rows padded to whole pieces of 16 elements, where its length does not fill the pieces of `step` that the
// launch takes: 8, 16 bytes, or 16 for the single-pass backward (padding_for_one_pass; what lies beyond the row's end is not looked at);
// undefined for every other mask.  Up to one tile of keys a
// bias is read element by element, whatever its layout.  Dimensions that broadcast are not written out, and the copy lives
// for one launch: layers that share a bias do not hold a copy each until their backward.  Where there is no memory for it the
// bias is read in place, by the register-tiled kernels.
Tensor padded_bias(const MaskDesc& m, const Tensor& q, int64_t step = 8) {
  if (m.c.kind != JVPFA_MASK_BIAS || !takes_16_bit_forms(q) || m.tensor.scalar_type() != q.scalar_type() || m.c.stride[2] == 0) return {};
  const int64_t L = q.size(2), width = (L + 15) / 16 * 16;
  if (L <= 64 || L % step == 0) return {};
  const int64_t n_b = m.c.stride[0] ? m.tensor.size(0) : 1, n_h = m.c.stride[1] ? m.tensor.size(1) : 1;
  Tensor padded;
  try {
    padded = empty({n_b, n_h, L, width}, m.tensor.scalar_type(), m.tensor.device());
  } catch (const c10::OutOfMemoryError&) {
    return {};
  }
  jvpfa_pad_bias_args a{};
  a.struct_size = sizeof(a);
  a.n_b = (int)n_b, a.n_h = (int)n_h, a.L = (int)L, a.width = (int)width;
  a.mask = m.c;
  a.out = padded.data_ptr();
  check_status(jvpfa_pad_bias(&a, c10::cuda::getCurrentCUDAStream(q.get_device()).stream()), "jvpfa_pad_bias");
  return padded;
}

jvpfa_mask c_mask(const MaskDesc& m, const Tensor& padded) {
  jvpfa_mask c = m.c;
  if (padded.defined()) {
    c.ptr = padded.const_data_ptr();
    for (int d = 0; d < 4; ++d) c.stride[d] = padded.size(d) == 1 ? 0 : padded.stride(d);
  }
  return c;
}

// Whether a backward becomes one pass when its bias gets rows of whole 32-byte pieces, which those of L % 16 == 8 are not.  The library's own rule is
// asked: where it stays with two launches they would read a copy that nobody needs (bf16 through tO, backward with / without it, us: B2 H12 L4104 D64,
// 0.8 GB of bias, 1523 / 1247, B1 H64 L2056 D64 1060 / 886, D = 32 B1 H61 L2056 988 / 835).
bool padding_for_one_pass(const jvpfa_bwd_args& a) {
  if (a.mask.kind != JVPFA_MASK_BIAS || a.dtype == JVPFA_FP32 || a.L <= 64 || a.L % 16 != 8 || !g_single_pass) return false;
  if (jvpfa_bwd_workspace(&a) > 0) return false;
  jvpfa_bwd_args padded = a;
  const int64_t width = a.L + 8, n_h = a.mask.stride[1] ? a.H : 1;
  padded.mask.ptr = a.q;  // any 16-byte aligned address; nothing is read
  padded.mask.stride[0] = a.mask.stride[0] ? n_h * a.L * width : 0;
  padded.mask.stride[1] = a.mask.stride[1] ? a.L * width : 0;
  padded.mask.stride[2] = width;
  padded.mask.stride[3] = 1;
  return jvpfa_bwd_workspace(&padded) > 0;
}

// Whether the mask's own entries can be read as 16-byte pieces of its rows.
bool whole_pieces(const MaskDesc& m, int64_t L) {
  const int64_t esz = m.tensor.element_size();
  bool ok = m.c.stride[3] == 1 && (reinterpret_cast<uintptr_t>(m.c.ptr) & 15u) == 0 && L % 16 == 0;
  for (int d = 0; d < 3; ++d) ok = ok && m.c.stride[d] * esz % 16 == 0;
  return ok;
}

// Bits by rows and, if asked for, transposed; both stay undefined where there is no memory or the mask is too large.
void pack(const MaskDesc& m, const Tensor& q, Tensor& bits_out, Tensor* bits_t_out) {
  const int64_t L = q.size(2);
  const int64_t n_b = m.c.stride[0] ? m.tensor.size(0) : 1, n_h = m.c.stride[1] ? m.tensor.size(1) : 1;
  const int64_t n_rows = m.c.stride[2] ? L : 1;
  const int64_t w = (L + 63) / 64 * 2;
  jvpfa_mask_tiles_args a{};
  a.struct_size = sizeof(a);
  a.n_b = (int)n_b, a.n_h = (int)n_h, a.n_rows = (int)n_rows, a.L = (int)L;
  a.mask = m.c;
  Tensor bits, bits_t;
  try {
    bits = empty({n_b * n_h * n_rows * w}, at::kInt, q.device());
    if (bits_t_out) bits_t = empty({n_b * n_h * L * (n_rows > 1 ? w : 1)}, at::kInt, q.device());
  } catch (const c10::OutOfMemoryError&) {
    return;
  }
  a.bits = bits.data_ptr();
  if (bits_t_out) a.bits_t = bits_t.data_ptr();
  const int rc = jvpfa_mask_tiles(&a, c10::cuda::getCurrentCUDAStream(q.get_device()).stream());
  if (rc == JVPFA_ERR_TOO_LARGE) return;  // the kernels read the bytes
  check_status(rc, "jvpfa_mask_tiles");
  bits_out = bits;
  if (bits_t_out) *bits_t_out = bits_t;
}

// Packs a call's boolean mask.  Bits are made anew by every call and not kept with the mask's description: the entries that
// the kernels read are then those that the mask holds when they run, also where it was written behind torch's version
// counter (a replayed graph, a foreign kernel).  Which tiles are stepped over, and the lengths of a key-padding mask, are
// those of its verification.
//
// Packing reads the mask once (HBM bound) and saves a kernel that reads it one 16-byte piece per row and sub-tile.
// B2 H12 L2048 D64, 100 MB of mask: packing 28 to 32 us; forward with tangents 140 -> 86 us, backward through tO 221 -> 142.
// So it pays with a backward, for a mask that several heads share, and where the bytes' layout would send the call to
// the register-tiled kernels.  Where there is no memory for the bits the kernels read the bytes.
void pack_mask(Call& call, const Tensor& q, bool backward) {
  const MaskDesc& m = *call.mask;
  if (m.c.kind != JVPFA_MASK_BOOL || !takes_16_bit_forms(q)) return;
  const int64_t n_b = m.c.stride[0] ? m.tensor.size(0) : 1, n_h = m.c.stride[1] ? m.tensor.size(1) : 1;
  if (!backward && whole_pieces(m, q.size(2)) && 4 * n_b * n_h > q.size(0) * q.size(1)) return;
  c10::cuda::OptionalCUDAGuard guard;
  if (q.get_device() != c10::cuda::current_device()) guard.set_index(q.get_device());
  pack(m, q, call.bits, backward ? &call.bits_t : nullptr);
}

// The tile bitmaps of a call's fp32 launches on the register-tiled kernels, [tile_live | tile_live_t], for a boolean mask whose verification left
// tiles to step over.  These launches visited every tile before they knew of bitmaps, and their results were the mask's present entries' whatever
// had been written since; so theirs are made anew, like the bits (B1 H8 L2048, a window as one (L, L) mask: 5 us).  The 16-bit
// kernels are given those of the verification.  Left undefined where there is no memory: every tile is visited then.
// And where dead tiles are no more than the bitmaps cost: 11 us of the launch by a rough model of it, in which a key takes 0.03 us, and more where
// there are rows for every SM.  Of 550 forwards on a B200 (windows of a quarter and half the length, key padding, L 160 to 3000), with bitmaps made
// for all 148 took more than 3 % longer than without any, up to 1.79 times (TF32 B1 H7 L170 D32 7.5 / 13.5 us); by this rule 5, 1.14 at most, and
// of the 309 that gain as much 284 have them.  Of 573 backward launches that find none 349 gain, 7 more would, and 25 take longer, 1.09 at most.
Tensor make_tiles(const Call& call, const Tensor& q, bool tangents, bool backward) {
  const MaskDesc& m = *call.mask;
  if (q.scalar_type() != at::kFloat || !m.tile_live.defined() || !m.tile_live_t.defined()) return {};
  const int64_t L = q.size(2), n = m.tile_live.numel();
  const double deep = (double)(q.size(0) * q.size(1) * ((L + 15) / 16)) / 148, width = (double)q.size(3) / 32 * (tangents ? 1.8 : 1) * (call.tf32 ? 1 : 1.8);
  if (m.dead * L * (0.03 + 0.004 * width * deep) * (backward ? 1.5 : 1) < 11) return {};
  jvpfa_mask_tiles_args a{};
  a.struct_size = sizeof(a);
  a.n_b = m.c.stride[0] ? (int)m.tensor.size(0) : 1, a.n_h = m.c.stride[1] ? (int)m.tensor.size(1) : 1;
  a.n_rows = m.c.stride[2] ? (int)L : 1, a.L = (int)L;
  a.mask = m.c;
  Tensor tiles;
  try {
    NoFunctorch nf;
    at::AutoDispatchBelowADInplaceOrView below;
    tiles = at::zeros({n + m.tile_live_t.numel()}, q.options().dtype(at::kLong).requires_grad(false));
  } catch (const c10::OutOfMemoryError&) {
    return {};
  }
  a.tile_live = tiles.data_ptr();
  a.tile_live_t = static_cast<int64_t*>(tiles.data_ptr()) + n;
  check_status(jvpfa_mask_tiles(&a, c10::cuda::getCurrentCUDAStream(q.get_device()).stream()), "jvpfa_mask_tiles");
  return tiles;
}

// ---- launches ------------------------------------------------------------------------------------------------------
// The workspace of a launch, which its kernels on the call's stream are the last to use; undefined for 0 bytes, and where
// there is no memory for it (the kernels that need none serve the call then).
Tensor workspace_of(int64_t bytes, const Tensor& q) {
  if (bytes <= 0) return {};
  try {
    return empty({bytes}, at::kByte, q.device());
  } catch (const c10::OutOfMemoryError&) {
    return {};
  }
}

py::object or_none(const Tensor& t) { return t.defined() ? py::cast(t) : py::object(py::none()); }

// Gives a launch its workspace, and an fp32 launch a boolean mask whose rows cannot be read 16 bytes at a time as bits (returned: they
// live as long as the launch is being issued).
template <typename Args>
Tensor use_workspace(Args& a, const Tensor& workspace, const Call& call, const Tensor& q) {
  Tensor bits;
  if (!workspace.defined()) return bits;
  a.workspace = workspace.data_ptr(), a.workspace_bytes = workspace.numel();
  if (q.scalar_type() == at::kFloat && a.mask.kind == JVPFA_MASK_BOOL && !whole_pieces(*call.mask, q.size(2))) {
    pack(*call.mask, q, bits, nullptr);
    a.mask_bits = data(bits);
  }
  return bits;
}

// tq without tk and tv: JVPFA_ZERO_TKV.
FwdResult launch_fwd(const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& tq, const Tensor& tk, const Tensor& tv,
                     Call& call) {
  const bool dual = tq.defined();
  FwdResult r;
  if (!q.is_cuda()) {
    py::gil_scoped_acquire gil;
    NoFunctorch nf;
    at::AutoGradMode no_grad(false);
    py::tuple out = python_module().attr("_launch_fwd")(or_none(q), or_none(k), or_none(v), or_none(tq), or_none(tk), or_none(tv),
                                                        *call.mask->spec, call.scale);
    r.o = out[0].cast<Tensor>();
    if (!out[1].is_none()) r.to = out[1].cast<Tensor>();
    r.lse = out[2].cast<Tensor>();
    if (!out[3].is_none()) r.mu = out[3].cast<Tensor>();
    return r;
  }
  c10::cuda::OptionalCUDAGuard guard;
  if (q.get_device() != c10::cuda::current_device()) guard.set_index(q.get_device());
  Inputs in(q, k, v, tq, tk, tv);
  const auto sizes = q.sizes();
  r.o = empty(sizes, q.scalar_type(), q.device());
  r.lse = empty(sizes.slice(0, 3), at::kFloat, q.device());
  if (dual) {
    r.to = empty(sizes, q.scalar_type(), q.device());
    r.mu = empty(sizes.slice(0, 3), at::kFloat, q.device());
  }
  const Tensor padded = padded_bias(*call.mask, q);
  jvpfa_fwd_args a{};
  a.struct_size = sizeof(a);
  a.dtype = dtype_of(q, call.tf32);
  a.B = (int)sizes[0], a.H = (int)sizes[1], a.L = (int)sizes[2], a.D = (int)sizes[3];
  a.impl = g_impl;
  a.sm_scale = (float)call.scale;
  a.o = r.o.data_ptr();
  a.lse = static_cast<float*>(r.lse.data_ptr());
  a.to = dual ? r.to.data_ptr() : nullptr;
  a.mu = dual ? static_cast<float*>(r.mu.data_ptr()) : nullptr;
  a.mask = c_mask(*call.mask, padded);
  const bool fp32 = q.scalar_type() == at::kFloat;
  a.mask_tile_live = fp32 ? nullptr : data(call.mask->tile_live);
  a.mask_bits = data(call.bits);
  a.flags = dual && !tk.defined() ? JVPFA_ZERO_TKV : 0;
  a.q = data(in.q), a.k = data(in.k), a.v = data(in.v);
  a.tq = data(in.tq), a.tk = data(in.tk), a.tv = data(in.tv);
  for (int d = 0; d < 3; ++d) a.in_stride[d] = in.st[d];
  a.kv_len_host = host_lengths(*call.mask, a.B);
  const Tensor workspace = workspace_of(!fp32 || call.parts ? jvpfa_fwd_workspace(&a) : 0, q);
  const Tensor bits = use_workspace(a, workspace, call, q);
  r.parts = fp32 && workspace.defined();
  if (fp32 && !r.parts) {
    call.tiles = make_tiles(call, q, dual, false);
    a.mask_tile_live = data(call.tiles);
  }
  check_status(jvpfa_fwd(&a, c10::cuda::getCurrentCUDAStream(q.get_device()).stream()), "jvpfa_fwd");
  return r;
}

// Gradients of <go, O> + <gto, tO> with respect to q, k, v; those named in `skip` (JVPFA_SKIP_*) stay undefined.
Grads launch_bwd(const Tensor& q, const Tensor& k, const Tensor& v, Tensor tq, Tensor tk, Tensor tv, const Tensor& o, Tensor to,
                 const Tensor& lse, Tensor mu, Tensor go, Tensor gto, const Call& call, int skip = 0) {
  if (!q.is_cuda()) {
    py::gil_scoped_acquire gil;
    NoFunctorch nf;
    at::AutoGradMode no_grad(false);
    py::tuple out = python_module().attr("_launch_bwd")(or_none(q), or_none(k), or_none(v), or_none(tq), or_none(tk), or_none(tv),
                                                        or_none(o), or_none(to), or_none(lse), or_none(mu), or_none(go),
                                                        or_none(gto), *call.mask->spec, call.scale);
    return {out[0].cast<Tensor>(), out[1].cast<Tensor>(), out[2].cast<Tensor>()};
  }
  c10::cuda::OptionalCUDAGuard guard;
  if (q.get_device() != c10::cuda::current_device()) guard.set_index(q.get_device());
  for (Tensor* t : {&go, &gto}) {
    if (!t->defined()) continue;
    *t = unwrap(*t);
    if (!t->is_contiguous() || t->scalar_type() != q.scalar_type()) {
      NoFunctorch nf;
      at::AutoDispatchBelowADInplaceOrView below;
      *t = t->to(q.scalar_type()).contiguous();
    }
  }
  if (!gto.defined()) tq = tk = tv = to = mu = Tensor();
  Inputs in(q, k, v, tq, tk, tv);
  const auto sizes = q.sizes();
  const int64_t rows = sizes[0] * sizes[1] * sizes[2];
  const MaskDesc& m = *call.mask;
  void* stream = c10::cuda::getCurrentCUDAStream(q.get_device()).stream();

  // One scratch allocation: the three row statistics, and fp32 dQ where the single-pass kernel takes it (head dimension 64,
  // 16-bit; index masks, and as far as rows are whole 16-byte pieces a boolean mask without tile bitmaps or, through O
  // alone, a bias of the tensors' type).  Such a bias through tO, and head dimension 32, have a workspace instead, below
  // (bwd_parts_workspace; else the two launches).
  bool single = g_single_pass && !(skip & JVPFA_SKIP_DKDV) && sizes[3] == 64 && q.scalar_type() != at::kFloat;
  if (m.c.kind == JVPFA_MASK_BOOL)
    single = single && !m.tile_live.defined() && !m.tile_live_t.defined() && whole_pieces(m, sizes[2]);
  else if (m.c.kind == JVPFA_MASK_BIAS)
    single = single && !gto.defined() && m.c.bias_dtype == dtype_of(q, false) && whole_pieces(m, sizes[2]);
  const int64_t stat = (rows + 63) / 64 * 64;  // 256-byte steps
  Tensor scratch = empty({3 * stat + (single ? rows * sizes[3] : 0)}, at::kFloat, q.device());
  float* f = static_cast<float*>(scratch.data_ptr());

  jvpfa_pre_args p{};
  p.struct_size = sizeof(p);
  p.dtype = dtype_of(q, call.tf32);
  p.B = (int)sizes[0], p.H = (int)sizes[1], p.L = (int)sizes[2], p.D = (int)sizes[3];
  p.o = data(o), p.to = data(to), p.go = data(go), p.gto = data(gto);
  p.mu = static_cast<const float*>(data(mu));
  p.delta = f, p.eps = f + stat, p.cterm = f + 2 * stat;
  p.dq_accum = single ? f + 3 * stat : nullptr;
  check_status(jvpfa_bwd_preprocess(&p, stream), "jvpfa_bwd_preprocess");

  Grads g;
  if (!(skip & JVPFA_SKIP_DQ)) g[0] = empty(sizes, q.scalar_type(), q.device());
  if (!(skip & JVPFA_SKIP_DKDV))
    for (int i = 1; i < 3; ++i) g[i] = empty(sizes, q.scalar_type(), q.device());
  jvpfa_bwd_args a{};
  a.struct_size = sizeof(a);
  a.dtype = p.dtype;
  a.B = p.B, a.H = p.H, a.L = p.L, a.D = p.D;
  a.impl = g_impl;
  a.sm_scale = (float)call.scale;
  a.go = p.go, a.gto = p.gto;
  a.lse = static_cast<const float*>(data(lse));
  a.mu = p.mu;
  a.delta = p.delta, a.eps = p.eps, a.cterm = p.cterm;
  a.flags = skip | (single ? JVPFA_DQ_ACCUM_IS_ZERO : 0) | (tq.defined() && !tk.defined() ? JVPFA_ZERO_TKV : 0);
  if (g[0].defined()) a.dq = g[0].data_ptr();
  if (g[1].defined()) a.dk = g[1].data_ptr(), a.dv = g[2].data_ptr();
  a.mask = m.c;
  const bool fp32 = q.scalar_type() == at::kFloat;
  if (!fp32 && m.tile_live.defined() && m.tile_live_t.defined() && a.L <= 8192) {
    a.mask_tile_live = data(m.tile_live);
    a.mask_tile_live_t = data(m.tile_live_t);
  }
  a.dq_accum = p.dq_accum;
  a.mask_bits = data(call.bits);
  a.mask_bits_t = data(call.bits_t);
  a.q = data(in.q), a.k = data(in.k), a.v = data(in.v);
  a.tq = data(in.tq), a.tk = data(in.tk), a.tv = data(in.tv);
  for (int d = 0; d < 3; ++d) a.in_stride[d] = in.st[d];
  a.kv_len_host = host_lengths(m, a.B);
  const Tensor padded = padded_bias(m, q, padding_for_one_pass(a) ? 16 : 8);
  a.mask = c_mask(m, padded);
  const Tensor workspace = workspace_of((fp32 ? call.parts : g_single_pass.load()) ? jvpfa_bwd_workspace(&a) : 0, q);
  const Tensor bits = use_workspace(a, workspace, call, q);
  // (Bitmaps that a backward makes are its own: of one that is being captured they hold nothing before a replay, and another may come first.)
  Tensor tiles;
  if (fp32 && !workspace.defined() && a.L <= 8192) {
    tiles = call.tiles.defined() ? call.tiles : make_tiles(call, q, gto.defined(), true);
    if (tiles.defined()) a.mask_tile_live = tiles.data_ptr(), a.mask_tile_live_t = static_cast<int64_t*>(tiles.data_ptr()) + m.tile_live.numel();
  }
  check_status(jvpfa_bwd(&a, stream), "jvpfa_bwd");
  return g;
}

// What autograd will not use of a node's gradients with respect to q, k, v (its first three outputs).
int unused_gradients(bool need_q, bool need_kv) { return (need_q ? 0 : JVPFA_SKIP_DQ) | (need_kv ? 0 : JVPFA_SKIP_DKDV); }

Tensor zeros_like_input(const Tensor& q) {
  NoFunctorch nf;
  at::AutoDispatchBelowADInplaceOrView below;
  return at::zeros_like(q);
}

// ---- graph ---------------------------------------------------------------------------------------------------------
// Stands behind gradients that cannot be differentiated again, and says so when asked.
struct Refuse : public Node {
  std::string message;
  explicit Refuse(std::string m) : message(std::move(m)) {}
  variable_list apply(variable_list&&) override { throw std::runtime_error(message); }
  std::string name() const override { return "JVPAttnRefuse"; }
};

template <typename... Ts>
void attach_refusal(const char* message, std::initializer_list<Tensor*> outs, const Ts&... inputs) {
  if (!torch::autograd::compute_requires_grad(inputs...)) return;
  auto node = std::shared_ptr<Refuse>(new Refuse(message), torch::autograd::deleteNode);
  node->set_next_edges(torch::autograd::collect_next_edges(inputs...));
  for (Tensor* t : outs)
    if (t->defined()) torch::autograd::set_history(*t, node);
}

Tensor primal_of(const Tensor& x) {  // inside a forward-AD level the saved tensors are still dual
  return x.defined() && x._fw_grad(0).defined() ? x._fw_primal(0) : x;
}

// A tensor of the forward's own as the kernels read it, under functorch's wrappers.  Hooks on saved tensors may hand back
// another layout than the row-major one it was allocated with; upstream refuses such an output in its backward
// (jvp_attention.py:2858-2877).
Tensor saved_output(const Tensor& x, const char* name) {
  const Tensor t = unwrap(x);
  TORCH_CHECK_VALUE(t.is_contiguous(), "JVPAttn expected ", name, " to be contiguous; got ", name, ".is_contiguous()=False");
  return t;
}

// (dq, dk, dv) = d<do, O>/d(q, k, v), as a node that can be differentiated once more.  With u the incoming gradients of
// (dq, dk, dv):  d<(dq,dk,dv), u>/d(q,k,v) = d<tO(q,k,v; u), do>/d(q,k,v)  and  d<...>/d(do) = tO(q,k,v; u), so a
// Hessian-vector product is one primal + tangent forward with tangents u and one backward through the tangent output.
struct AttnBwdNode : public Node {
  Call call;
  SavedVariable q, k, v, go;

  variable_list apply(variable_list&& u) override {
    std::lock_guard<std::mutex> lock(mutex_);
    variable_list out(4);
    if (!u[0].defined() && !u[1].defined() && !u[2].defined()) return out;
    const Tensor q_ = q.unpack(), k_ = k.unpack(), v_ = v.unpack(), go_ = go.unpack();
    const Tensor qp = unwrap(q_), kp = unwrap(k_), vp = unwrap(v_), gop = unwrap(go_);
    Tensor t[3];
    // a product with a vector that is zero on K and V (only q is differentiated): the fp32 kernels leave their terms out
    const bool zero_tkv = u[0].defined() && !u[1].defined() && !u[2].defined() && qp.is_cuda() && qp.scalar_type() == at::kFloat &&
                          !call.tf32;
    {
      NoFunctorch nf;
      at::AutoDispatchBelowADInplaceOrView below;
      // In the layout of q, k and v where the kernels read that in place: else all six, and again the backward's, are copied to row-major
      // (bf16 B3 H10 L3392 D128, views of (B, L, H, D): 254 of the 1530 us of a Hessian-vector product).  A tensor of the layout of q with
      // gaps between its rows (slices of one packed projection) is not made anew: only tangents that come in it are read in place, and
      // else row-major ones cost the fewest copies, those of q, k and v.
      const int n = zero_tkv ? 1 : 3;
      auto aligned = [](const Tensor& x) { return (reinterpret_cast<uintptr_t>(x.const_data_ptr()) & 15u) == 0; };
      int64_t st[3];
      bool views = common_layout({&qp, &kp, &vp}, st) && st[2] != 0;
      const bool gaps = views && !qp.is_non_overlapping_and_dense();
      for (int i = 0; i < n; ++i) {
        if (u[i].defined()) t[i] = unwrap(u[i]);
        if (gaps) views = views && t[i].defined() && t[i].strides() == qp.strides() && aligned(t[i]);
      }
      for (int i = 0; i < n; ++i) {
        if (!t[i].defined())
          t[i] = views ? at::zeros_like(qp) : at::zeros_like(qp, at::MemoryFormat::Contiguous);
        else if ((views ? t[i].strides() != qp.strides() : !t[i].is_contiguous()) || !aligned(t[i]))
          t[i] = (views ? at::empty_like(qp) : at::empty_like(qp, at::MemoryFormat::Contiguous)).copy_(t[i]);
      }
    }
    const int skip = unused_gradients(task_should_compute_output(0), task_should_compute_output(1) || task_should_compute_output(2));
    const bool again = skip != (JVPFA_SKIP_DQ | JVPFA_SKIP_DKDV);
    Call c = call;
    c.parts = !again || (zero_tkv && (skip & JVPFA_SKIP_DKDV));
    FwdResult f = launch_fwd(qp, kp, vp, t[0], t[1], t[2], c);
    c.parts = f.parts;
    if (again) {
      Grads h = launch_bwd(qp, kp, vp, t[0], t[1], t[2], f.o, f.to, f.lse, f.mu, Tensor(), gop, c, skip);
      for (int i = 0; i < 3; ++i) out[i] = h[i];
    }
    if (task_should_compute_output(3)) out[3] = f.to;
    if (at::GradMode::is_enabled())
      attach_refusal("trying to differentiate twice a function that was marked with @once_differentiable",
                     {&out[0], &out[1], &out[2], &out[3]}, q_, k_, v_, go_, u[0], u[1], u[2]);
    return out;
  }
  void release_variables() override {
    std::lock_guard<std::mutex> lock(mutex_);
    for (SavedVariable* s : {&q, &k, &v, &go}) s->reset_data();
    call.drop_tensors();
  }
  std::string name() const override { return "JVPAttnBackwardBackward"; }
};

Grads backward_through_o(const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& o, const Tensor& lse, const Tensor& go,
                         const Call& call, int skip) {
  if (is_wrapped(go)) {  // the cotangent belongs to a functorch transform: a Function, which the transform differentiates or refuses
    py::gil_scoped_acquire gil;
    py::tuple g = python_module().attr("_backward_under_functorch")(q, k, v, o, lse, go, *call.mask->spec, call.scale, call.tf32, call.parts);
    return {g[0].cast<Tensor>(), g[1].cast<Tensor>(), g[2].cast<Tensor>()};
  }
  Grads g = launch_bwd(unwrap(q), unwrap(k), unwrap(v), Tensor(), Tensor(), Tensor(), o, Tensor(), lse, Tensor(), go, Tensor(), call, skip);
  if (torch::autograd::compute_requires_grad(q, k, v, go)) {  // create_graph: a second differentiation was asked for
    auto node = std::shared_ptr<AttnBwdNode>(new AttnBwdNode(), torch::autograd::deleteNode);
    node->set_next_edges(torch::autograd::collect_next_edges(q, k, v, go));
    node->call = call;
    node->q = SavedVariable(q, false);
    node->k = SavedVariable(k, false);
    node->v = SavedVariable(v, false);
    node->go = SavedVariable(go, false);
    for (Tensor& t : g) torch::autograd::set_history(t, node);
  }
  return g;
}

// The node of a call: outputs O (0) and, with tangents, tO (1); edges to q, k, v, with tangents to these, and to a mask that
// requires a gradient (which is undefined: O is part of the mask's graph, and the mask's gradient stays None).
struct AttnNode : public Node {
  Call call;
  SavedVariable q, k, v, tq, tk, tv, o, to, lse, mu;

  variable_list apply(variable_list&& grads) override {
    std::lock_guard<std::mutex> lock(mutex_);
    variable_list out(num_outputs());
    const Tensor go = primal_of(grads[0]);
    const Tensor gto = grads.size() > 1 ? primal_of(grads[1]) : Tensor();
    if (!go.defined() && !gto.defined()) return out;
    const auto self = shared_from_this();
    const Tensor q_ = primal_of(q.unpack()), k_ = primal_of(k.unpack()), v_ = primal_of(v.unpack());
    const Tensor o_ = saved_output(o.unpack(self), "o"), lse_ = saved_output(lse.unpack(), "lse");
    const int skip = unused_gradients(task_should_compute_output(0), task_should_compute_output(1) || task_should_compute_output(2));
    const bool need_primals = skip != (JVPFA_SKIP_DQ | JVPFA_SKIP_DKDV);
    if (!gto.defined()) {
      if (need_primals) {
        Grads g = backward_through_o(q_, k_, v_, o_, lse_, go, call, skip);
        for (int i = 0; i < 3; ++i) out[i] = g[i];
      }
      return out;
    }
    const Tensor tq_ = tq.unpack(), tk_ = tk.unpack(), tv_ = tv.unpack();
    const Tensor to_ = saved_output(to.unpack(self), "to"), mu_ = saved_output(mu.unpack(), "mu");
    const Tensor qp = unwrap(q_), kp = unwrap(k_), vp = unwrap(v_), tqp = unwrap(tq_), tkp = unwrap(tk_), tvp = unwrap(tv_);
    static constexpr const char* kOnce = "the gradient through the tangent output of JVPAttn cannot be differentiated a second time";
    if (need_primals) {
      const bool again = at::GradMode::is_enabled();  // a second differentiation was asked for: the part through O stays a node of its own
      Grads g = launch_bwd(qp, kp, vp, tqp, tkp, tvp, o_, to_, lse_, mu_, again ? Tensor() : go, gto, call, skip);
      if (again) {
        attach_refusal(kOnce, {&g[0], &g[1], &g[2]}, q_, k_, v_, tq_, tk_, tv_, gto);
        if (go.defined()) {
          Grads h = backward_through_o(q_, k_, v_, o_, lse_, go, call, skip);
          for (int i = 0; i < 3; ++i)
            if (h[i].defined()) g[i] = h[i] + g[i];
        }
      }
      for (int i = 0; i < 3; ++i) out[i] = g[i];
    }
    if (task_should_compute_output(3) || task_should_compute_output(4) || task_should_compute_output(5)) {
      // with respect to the tangents tO is an ordinary attention output with cotangent gto
      Grads g = launch_bwd(qp, kp, vp, Tensor(), Tensor(), Tensor(), o_, Tensor(), lse_, Tensor(), gto, Tensor(), call,
                           unused_gradients(task_should_compute_output(3), task_should_compute_output(4) || task_should_compute_output(5)));
      if (at::GradMode::is_enabled()) attach_refusal(kOnce, {&g[0], &g[1], &g[2]}, q_, k_, v_, tq_, tk_, tv_, gto);
      for (int i = 0; i < 3; ++i) out[3 + i] = g[i];
    }
    return out;
  }
  void release_variables() override {
    std::lock_guard<std::mutex> lock(mutex_);
    for (SavedVariable* s : {&q, &k, &v, &tq, &tk, &tv, &o, &to, &lse, &mu}) s->reset_data();
    call.drop_tensors();
  }
  std::string name() const override { return "JVPAttnBackward"; }
};

// ---- entry point ---------------------------------------------------------------------------------------------------
// What the kernels and the single graph node take: 4-D q, k, v of one shape, type and device, head dimension 32, 64 or
// 128, and (upstream's check, unless lifted) an even length of at least 32.  Everything else goes back to the Python
// layer, which words the errors.
bool acceptable(const Tensor& q, const Tensor& k, const Tensor& v, bool strict_length) {
  if (q.dim() != 4 || q.layout() != at::kStrided) return false;
  if (k.sizes() != q.sizes() || v.sizes() != q.sizes()) return false;
  if (k.scalar_type() != q.scalar_type() || v.scalar_type() != q.scalar_type()) return false;
  if (k.device() != q.device() || v.device() != q.device()) return false;
  const int64_t L = q.size(2), D = q.size(3);
  if (strict_length && (L % 2 != 0 || L < 32)) return false;
  if (D != 32 && D != 64 && D != 128) return false;
  return !q.is_cuda() || dtype_of(q, false) >= 0;
}

// Tangent as the kernels read it: q's type, zero where there is none.
Tensor tangent(const Tensor& t, const Tensor& q) {
  if (!t.defined()) return zeros_like_input(q);
  if (t.scalar_type() == q.scalar_type()) return t;
  NoFunctorch nf;
  return t.to(q.scalar_type());
}

struct Outputs {
  Tensor o, to;
};

// The call itself on plain tensors; tangents all undefined or all given.  nullopt: not a case for this path.
std::optional<Outputs> attend_plain(const Tensor& q, const Tensor& k, const Tensor& v, Tensor tq, Tensor tk, Tensor tv,
                                    const Tensor& mask_tensor, const MaskPtr& mask, std::optional<double> scale, bool tf32,
                                    bool strict_length) {
  for (const Tensor* t : std::initializer_list<const Tensor*>{&q, &k, &v, &tq, &tk, &tv})
    if (t->defined() && is_wrapped(*t)) return std::nullopt;
  if (!acceptable(q, k, v, strict_length)) return std::nullopt;
  const bool dual = tq.defined() || tk.defined() || tv.defined();
  if (dual) {
    for (const Tensor* t : {&tq, &tk, &tv})
      if (t->defined() && (t->sizes() != q.sizes() || t->device() != q.device())) return std::nullopt;
    tq = tangent(tq, q), tk = tangent(tk, q), tv = tangent(tv, q);
  }
  Call call{mask, scale ? *scale : 1.0 / std::sqrt((double)q.size(3)), tf32};
  const bool grad_qkv = torch::autograd::compute_requires_grad(q, k, v), grad_mask = torch::autograd::compute_requires_grad(mask_tensor);
  const bool backward = grad_qkv || torch::autograd::compute_requires_grad(tq, tk, tv);
  call.parts = !dual || !grad_qkv;  // (with respect to the tangents tO is an ordinary attention output)
  FwdResult r;
  {
    // A launch waits while the queue of launches is full: other Python threads run meanwhile.
    std::optional<py::gil_scoped_release> no_gil;
    if (q.is_cuda()) no_gil.emplace();
    pack_mask(call, q, backward);
    r = launch_fwd(q, k, v, tq, tk, tv, call);
    call.parts = r.parts;
  }
  if (backward || grad_mask) {
    auto node = std::shared_ptr<AttnNode>(new AttnNode(), torch::autograd::deleteNode);
    node->call = call;
    torch::autograd::edge_list edges =
        dual ? torch::autograd::collect_next_edges(q, k, v, tq, tk, tv) : torch::autograd::collect_next_edges(q, k, v);
    if (grad_mask) edges.push_back(torch::autograd::impl::gradient_edge(mask_tensor));
    node->set_next_edges(std::move(edges));
    node->q = SavedVariable(q, false);
    node->k = SavedVariable(k, false);
    node->v = SavedVariable(v, false);
    const bool grad_o = grad_qkv || grad_mask;
    if (grad_o)
      torch::autograd::set_history(r.o, node);
    else
      node->add_input_metadata(Node::undefined_input());
    if (dual && backward) {
      torch::autograd::set_history(r.to, node);
      node->tq = SavedVariable(tq, false);
      node->tk = SavedVariable(tk, false);
      node->tv = SavedVariable(tv, false);
      node->to = SavedVariable(r.to, true);
      node->mu = SavedVariable(r.mu, false);
    }
    node->o = SavedVariable(r.o, grad_o);
    node->lse = SavedVariable(r.lse, false);
  }
  return Outputs{r.o, r.to};
}

// attention (dual = false) or fwd_dual (true).  None: not a case for this path (bad arguments, dual inputs of a
// primal-only call, a mask's tangent alone, functorch transforms other than a lone torch.func.jvp); the caller takes its
// general route.  `mask_in`: the caller's mask tensor.
py::object attend(const Tensor& q_in, const Tensor& k_in, const Tensor& v_in, const std::optional<Tensor>& mask_in, const MaskPtr& mask,
                  std::optional<double> scale, bool tf32, bool dual, bool strict_length) {
  const auto& stack = at::functorch::getDynamicLayerStack();
  Tensor q = q_in, k = k_in, v = v_in, tq = q._fw_grad(0), tk = k._fw_grad(0), tv = v._fw_grad(0);
  const bool any_tangent = tq.defined() || tk.defined() || tv.defined();
  if (!dual && any_tangent) return py::none();
  if (mask_in && !any_tangent && mask_in->_fw_grad(0).defined()) return py::none();
  int64_t level = -1;
  if (!stack.empty()) {
    // Primals and tangents are taken off the transform's wrappers, the call runs one level down on plain tensors, and
    // the two results become a dual tensor of its level again: what torch.func.jvp does for a built-in operator.
    if (!any_tangent || stack.size() != 1 || stack.back().key() != at::functorch::TransformType::Jvp) return py::none();
    level = stack.back().layerId();
    for (Tensor* t : {&q, &k, &v, &tq, &tk, &tv}) {
      auto* w = t->defined() ? at::functorch::maybeGetTensorWrapper(*t) : nullptr;
      if (w && w->level() == level) *t = Tensor(w->value());
    }
  }
  auto out = attend_plain(q, k, v, tq, tk, tv, mask_in ? unwrap(*mask_in) : Tensor(), mask, scale, tf32, strict_length);
  if (!out) return py::none();
  if (!out->to.defined()) return py::cast(out->o);
  Tensor o = out->o, to = out->to;
  if (level >= 0) {
    o = at::functorch::makeTensorWrapper(o, level);
    to = at::functorch::makeTensorWrapper(to, level);
  }
  o._set_fw_grad(to, /*level=*/0, /*is_inplace_op=*/false);
  return py::cast(o);
}

}  // namespace

PYBIND11_MODULE(_native, m) {
  py::class_<NoFunctorchScope>(m, "NoFunctorch")
      .def(py::init<>())
      .def("__enter__", [](NoFunctorchScope& s) { s.guard.emplace(); })
      .def("__exit__", [](NoFunctorchScope& s, py::args) { s.guard.reset(); });
  py::class_<MaskDesc, MaskPtr>(m, "MaskDesc")
      .def(py::init<int, int, std::optional<Tensor>, std::array<int64_t, 4>, std::optional<Tensor>, std::optional<Tensor>,
                    std::vector<int32_t>, double, py::object>());
  m.def("attend", &attend);
  m.def("set_impl", [](int v) { g_impl = v; });
  m.def("set_single_pass", [](bool v) { g_single_pass = v; });
}

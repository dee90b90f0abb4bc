// Native host path of the layers: the forward and backward of the LatentMoE and MoE layers as sequences of the C-ABI
// entry points of liblmoe.so, with buffers from PyTorch's caching allocator and autograd nodes in C++.
//
// Why native: at small batches the layer is bound by its host.  Assembled in Python (one ctypes call per stage, about 25
// allocations per direction, a Python autograd function) a forward cost 215 us and a training step 740 us of host time
// whatever the batch, against 90 and 256 us of kernels at 1 and 1,024 tokens.  Here a direction is one call: the
// activations kept for the backward are ONE allocation cut into 256-byte-aligned pieces (saved_layout), the scratch
// another one, and the device status words live in mapped host memory, so that no step queues a fill, a copy or an
// event for them.
//
// The order of the stages is the reference's (models/moe.py:702-734 for the latent layer, 344-372 for the other one);
// the backward is the adjoint of each.
#include <ATen/ATen.h>
#include <ATen/cuda/CUDAContext.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <cuda_runtime.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/custom_function.h>
#include <torch/csrc/jit/frontend/tracer.h>
#include <torch/extension.h>

#include <atomic>
#include <cstring>
#include <map>
#include <mutex>
#include <utility>

#include "../../include/lmoe.h"

namespace py = pybind11;
using at::Tensor;
using torch::autograd::AutogradContext;
using torch::autograd::variable_list;

namespace {

// ---------------------------------------------------------------- errors
struct LmoeFailure : std::runtime_error {
  using std::runtime_error::runtime_error;
};
PyObject* g_error_class = nullptr;  // swamla_b200._cabi.LmoeError

void check(int rc, const char* what) {
  if (rc != 0)
    throw LmoeFailure(std::string(what) + " failed with code " + std::to_string(rc) + ": " + lmoe_status_string(rc));
}
#define LMOE(name, ...) check(name(__VA_ARGS__), #name)

// A failure inside the autograd engine's thread has to travel as a Python exception to keep its class.
[[noreturn]] void rethrow_as_python(const LmoeFailure& e) {
  py::gil_scoped_acquire gil;
  PyErr_SetString(g_error_class ? g_error_class : PyExc_RuntimeError, e.what());
  python_error err;
  err.persist();
  throw err;
}

// ---------------------------------------------------------------- device status words
// One int32 per device and kind of call, in mapped pinned memory: a kernel whose bounded wait gives up writes its code
// straight to the host, which reads the word at its next call.  Never freed: kernels of any stream may still hold the address.
enum Kind : int { kLatentFwd = 0, kLatentBwd = 1, kMoeFwd = 2, kMoeBwd = 3, kKinds = 4 };
const char* const kKindName[kKinds] = {"LatentMoE forward", "LatentMoE backward", "MoE forward", "MoE backward"};
constexpr int kStatusDevices = 64;
constexpr int kStatusStride = 16;  // int32 per word: a cache line each
std::atomic<bool> g_device_used[kStatusDevices];

int32_t* status_words() {
  static int32_t* words = [] {
    constexpr size_t bytes = kStatusDevices * kKinds * kStatusStride * sizeof(int32_t);
    void* p = nullptr;
    cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;  // the first call may be one that is being captured
    cudaThreadExchangeStreamCaptureMode(&mode);
    const cudaError_t e = cudaHostAlloc(&p, bytes, cudaHostAllocMapped | cudaHostAllocPortable);
    cudaThreadExchangeStreamCaptureMode(&mode);
    if (e != cudaSuccess)
      throw LmoeFailure("no pinned memory for the device status words");
    std::memset(p, 0, bytes);
    return static_cast<int32_t*>(p);
  }();
  return words;
}
int32_t* status_word(int device, Kind k) { return status_words() + (device * kKinds + k) * kStatusStride; }
// The word of a call that is about to launch on the current device.
int32_t* status_word(Kind k) {
  const int device = c10::cuda::current_device();
  TORCH_CHECK(device >= 0 && device < kStatusDevices, "device ordinal out of range");
  g_device_used[device].store(true, std::memory_order_relaxed);
  return status_word(device, k);
}
std::vector<int> devices_used() {
  std::vector<int> v;
  for (int d = 0; d < kStatusDevices; ++d)
    if (g_device_used[d].load(std::memory_order_relaxed)) v.push_back(d);
  return v;
}

// Throws for the first word that a kernel has written; the word is cleared.
void poll_status() {
  for (int d = 0; d < kStatusDevices; ++d) {
    if (!g_device_used[d].load(std::memory_order_relaxed)) continue;
    for (int k = 0; k < kKinds; ++k) {
      int32_t* w = status_word(d, static_cast<Kind>(k));
      if (__atomic_load_n(w, __ATOMIC_RELAXED) == 0) continue;
      const int32_t code = __atomic_exchange_n(w, 0, __ATOMIC_RELAXED);
      if (code != 0)
        throw LmoeFailure("device status " + std::to_string(code) + " in " + kKindName[k] + " on cuda:" + std::to_string(d) + ": " +
                          lmoe_status_string(code));
    }
  }
}

// ---------------------------------------------------------------- side stream of the backward
// HBM-bound row kernels run beside tensor-bound GEMMs of the main stream.  Every buffer belongs to the main stream and
// every side section is joined before the call returns, so the caching allocator never recycles a block in use.
struct Side {
  cudaStream_t stream = nullptr;
  cudaEvent_t ev = nullptr;
};
std::mutex g_side_mutex;
std::map<std::pair<int, cudaStream_t>, Side> g_sides;

class Fork {
 public:
  explicit Fork(const c10::cuda::CUDAStream& main) : main_(main.stream()) {
    std::lock_guard<std::mutex> lock(g_side_mutex);
    Side& s = g_sides[{main.device_index(), main_}];
    if (!s.stream) {
      // A stream of its own, not one of PyTorch's pool, which hands the same 32 out to everybody: while this one is part of a
      // capture, what another user of it queued would be recorded instead of run.
      cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;  // the first call may be one that is being captured
      C10_CUDA_CHECK(cudaThreadExchangeStreamCaptureMode(&mode));
      cudaError_t e = cudaStreamCreateWithFlags(&s.stream, cudaStreamNonBlocking);
      if (e == cudaSuccess) e = cudaEventCreateWithFlags(&s.ev, cudaEventDisableTiming);
      cudaThreadExchangeStreamCaptureMode(&mode);
      C10_CUDA_CHECK(e);
    }
    side_ = &s;
  }
  // A stage that fails between to_side and to_main: what the side stream has been given still uses the call's buffers.
  ~Fork() {
    if (!open_) return;
    std::lock_guard<std::mutex> lock(g_side_mutex);
    if (cudaEventRecord(side_->ev, side_->stream) == cudaSuccess) cudaStreamWaitEvent(main_, side_->ev, 0);
  }
  Fork(const Fork&) = delete;
  Fork& operator=(const Fork&) = delete;
  cudaStream_t side() const { return side_->stream; }
  void to_side() {
    open_ = true;
    order(main_, side_->stream);
  }
  // more: the side stream goes on with work that a later to_main joins
  void to_main(bool more = false) {
    order(side_->stream, main_);
    open_ = more;
  }

 private:
  bool open_ = false;
  void order(cudaStream_t first, cudaStream_t then) {
    std::lock_guard<std::mutex> lock(g_side_mutex);  // record and wait belong together: the event is shared
    C10_CUDA_CHECK(cudaEventRecord(side_->ev, first));
    C10_CUDA_CHECK(cudaStreamWaitEvent(then, side_->ev, 0));
  }
  cudaStream_t main_;
  Side* side_;
};

// ---------------------------------------------------------------- buffers
// Cuts one allocation into 256-byte-aligned pieces.
struct Carver {
  size_t bytes = 0;
  size_t take(int64_t n) {
    const size_t at = bytes;
    bytes += (static_cast<size_t>(n) + 255) / 256 * 256;
    return at;
  }
};

Tensor new_bytes(size_t n, const Tensor& like) {
  return at::empty({static_cast<int64_t>(n)}, like.options().dtype(at::kByte).requires_grad(false));
}
char* base_of(const Tensor& arena) { return static_cast<char*>(arena.data_ptr()); }

struct Sizes {
  int T, D, L, E, K, F, Fs;
  int64_t P;
  lmoe_shape s;
  Sizes(int64_t T_, int64_t D_, int64_t L_, int64_t E_, int64_t K_, int64_t F_, int64_t Fs_)
      : T(T_), D(D_), L(L_), E(E_), K(K_), F(F_), Fs(Fs_) {
    s = lmoe_shape{T, D, L, E, K, F, Fs, 1};
    P = (static_cast<int64_t>(T) * K + 127) / 128 * 128 + static_cast<int64_t>(E) * 128;
  }
  int64_t route_ints() const {
    const int64_t n[8] = {E, E + 1, E + 1, 1, P / 128, int64_t(T) * K, int64_t(T) * K, P};
    int64_t sum = 0;
    for (int64_t v : n) sum += (v + 3) / 4 * 4;
    return sum;
  }
  // The tables of functional.RouteTables, in its order; counts go to their own tensor (the router keeps them).
  lmoe_route route(void* storage, int32_t* counts) const {
    int32_t* p = static_cast<int32_t*>(storage);
    auto next = [&p](int64_t n) {
      int32_t* at = p;
      p += (n + 3) / 4 * 4;
      return at;
    };
    lmoe_route r;
    next(E);
    r.counts = counts;
    r.offsets = next(E + 1);
    r.pad_offsets = next(E + 1);
    r.n_tiles = next(1);
    r.tile_expert = next(P / 128);
    r.perm = next(int64_t(T) * K);
    r.pos = next(int64_t(T) * K);
    r.row_src = next(P);
    return r;
  }
};

void check_device(const Tensor& t, at::Device device) {
  if (t.device() != device) throw LmoeFailure("a tensor of the layer is on " + t.device().str() + ", its input on " + device.str());
}

// bf16, contiguous forms of the operands; everything that is fp32 is converted by one launch.
// All on one device: a pointer to another one's memory, or to the host's, would only be found out by a kernel.
struct Caster {
  explicit Caster(const Tensor& x) : device(x.device()) {}
  const at::Device device;
  const float* src[LMOE_CAST_MANY_MAX];
  void* dst[LMOE_CAST_MANY_MAX];
  int64_t n[LMOE_CAST_MANY_MAX];
  std::vector<Tensor> keep;
  int count = 0;
  Tensor operator()(const Tensor& t) {
    check_device(t, device);
    if (t.scalar_type() == at::kBFloat16) return t.is_contiguous() ? t.detach() : t.detach().contiguous();
    Tensor f = t.detach();
    if (f.scalar_type() != at::kFloat) f = f.to(at::kFloat);
    f = f.contiguous();
    Tensor out = at::empty(f.sizes(), f.options().dtype(at::kBFloat16));
    if (f.numel() > 0) {
      if (count == LMOE_CAST_MANY_MAX) throw LmoeFailure("too many operands to convert at once");
      src[count] = f.data_ptr<float>();
      dst[count] = out.data_ptr();
      n[count++] = f.numel();
      keep.push_back(f);
    }
    return out;
  }
  void run(cudaStream_t st) {
    if (count > 0) LMOE(lmoe_cast_many_f32_to_bf16, count, src, dst, n, st);
  }
};

// t in another shape, not recorded as a view: an output of a custom function that autograd takes for a view refuses to be
// changed in place (y += ..., an in-place dropout).
Tensor shaped(const Tensor& t, at::IntArrayRef sizes) { return at::_unsafe_view(t, sizes); }

// A gradient in its parameter's dtype.
Tensor as_param(const Tensor& g, at::ScalarType d) { return g.scalar_type() == d ? g : g.to(d); }

bool tma_gather_enabled() {
  static const bool on = [] {
    const char* e = getenv("LMOE_TMA_GATHER");
    return e && e[0] == '1' && e[1] == 0;
  }();
  return on;
}

Tensor f32_bias(const Tensor& b, const Tensor& x) {
  check_device(b, x.device());
  return b.scalar_type() == at::kFloat && b.is_contiguous() ? b : b.detach().to(at::kFloat).contiguous();
}

// ---------------------------------------------------------------- LatentMoE: what a forward keeps
// Byte offsets in the saved allocation.  functional.saved_bytes (shape arithmetic of the compiled operators) computes the
// same total.
struct LatentLayout {
  size_t logits, weights, lse, route, act_cat, h1_s, y_sorted, h1;
  size_t x_rows = 0, hidden = 0;                                      // bf16 experts (x_rows: x_sorted, or the latent rows)
  size_t xq = 0, hq = 0, wguq = 0, wdq = 0, scal = 0;                 // e4m3 experts
  size_t bytes = 0;
  LatentLayout(const Sizes& d, bool fp8, bool gather, bool keep = true) {  // !keep: no backward follows, no gate / up

    Carver c;
    const int64_t T = d.T, P = d.P;
    logits = c.take(T * d.E * 4);
    weights = c.take(T * d.K * 4);
    lse = c.take(T * 4);
    route = c.take(d.route_ints() * 4);
    act_cat = c.take(T * (d.L + d.Fs) * 2);
    h1_s = c.take(keep ? T * 2 * d.Fs * 2 : 0);
    y_sorted = c.take(P * d.L * 2);
    h1 = c.take(keep ? P * 2 * d.F * 2 : 0);
    if (fp8) {
      xq = c.take(P * d.L);
      hq = c.take(P * d.F);
      wguq = c.take(int64_t(d.E) * d.L * 2 * d.F);
      wdq = c.take(int64_t(d.E) * d.F * d.L);
      scal = c.take(32 * 4);
    } else {
      x_rows = c.take((gather ? T + 1 : P) * d.L * 2);
      hidden = c.take(P * d.F * 2);
    }
    bytes = c.bytes;
  }
};
// scal: [amax, amax / 448] per quantised tensor
enum Scal : int { kSx = 0, kSwgu = 1, kSwd = 2, kSh = 3, kSdy = 4, kSdh1 = 5, kScals = 6 };
float* amax_of(float* scal, Scal k) { return scal + 2 * k; }
float* deq_of(float* scal, Scal k) { return scal + 2 * k + 1; }

// Intermediates by name, for the parity tests only.
using Views = std::vector<std::pair<std::string, Tensor>>;
Tensor view_of(const Tensor& arena, size_t at, std::vector<int64_t> shape, at::ScalarType dt) {
  int64_t n = 1;
  for (int64_t v : shape) n *= v;
  return arena.narrow(0, static_cast<int64_t>(at), n * static_cast<int64_t>(c10::elementSize(dt))).view(dt).view(shape);
}

struct LatentOps {
  Tensor x, wg, wdn, wup, wgus, wds, wgu, wde;  // bf16, contiguous; x [T, D]
};

struct LatentOut {
  Tensor y, z_loss, sel, counts, saved;
};

Sizes latent_sizes(const Tensor& x2d, const Tensor& wgu, const Tensor& wds, int64_t top_k) {
  TORCH_CHECK(wgu.dim() == 3 && x2d.size(1) == wds.size(0), "activation of another width than the layer's");
  return Sizes(x2d.size(0), x2d.size(1), wgu.size(1), wgu.size(0), top_k, wgu.size(2) / 2, wds.size(1));
}

// Up to this many tokens the dense GEMMs leave SMs free: the router chain and the shared expert then run side by side.
constexpr int kForkForwardTokens = 2048;

LatentOut latent_forward(const Sizes& d, const LatentOps& o, const Tensor& bias, float z_coef, bool fp8, bool keep,
                         const c10::optional<Tensor>& forced_sel, Views* views) {
  const auto stream = at::cuda::getCurrentCUDAStream();
  void* st = stream.stream();
  int32_t* status = status_word(kLatentFwd);
  const bool gather = tma_gather_enabled() && !fp8 && d.L % 128 == 0;  // whole 128-column tiles of the weight gradient
  const LatentLayout at_(d, fp8, gather, keep);
  const int64_t T = d.T, P = d.P;

  LatentOut r;
  const auto f32 = o.x.options().dtype(at::kFloat).requires_grad(false);
  const auto i32 = f32.dtype(at::kInt);
  r.y = at::empty({T, d.D}, o.x.options().requires_grad(false));
  r.z_loss = at::empty({}, f32);
  r.sel = at::empty({T, d.K}, i32);
  r.counts = at::empty({d.E}, i32);
  r.saved = new_bytes(at_.bytes, o.x);
  char* sv = base_of(r.saved);

  // scratch that nothing keeps
  Carver c;
  const size_t ws_bytes = std::max<size_t>({16, lmoe_route_workspace_bytes(&d.s), lmoe_route_fwd_workspace_bytes(&d.s)});
  const size_t t_ws = c.take(ws_bytes), t_zp = forced_sel ? c.take((T + 7) / 8 * 4) : 0;
  const size_t t_lat = gather ? 0 : c.take(T * d.L * 2);
  const size_t t_xs = (gather && views) ? c.take(P * d.L * 2) : 0;
  const size_t t_latq = fp8 ? c.take(T * d.L) : 0;
  const size_t t_hid = fp8 ? c.take(P * d.F * 2) : 0;
  Tensor tmp = new_bytes(c.bytes, o.x);
  char* tv = base_of(tmp);

  float* logits = reinterpret_cast<float*>(sv + at_.logits);
  float* weights = reinterpret_cast<float*>(sv + at_.weights);
  float* lse = reinterpret_cast<float*>(sv + at_.lse);
  const lmoe_route route = d.route(sv + at_.route, r.counts.data_ptr<int32_t>());
  void* act_cat = sv + at_.act_cat;
  void* h1_s = keep ? sv + at_.h1_s : nullptr;
  void* y_sorted = sv + at_.y_sorted;
  void* h1 = keep ? sv + at_.h1 : nullptr;
  void* x_latent = gather ? sv + at_.x_rows : tv + t_lat;
  // what the routed GEMMs read: e4m3 rows (the latents are quantised before they are gathered: the maximum over the
  // gathered rows is theirs, every token being routed), bf16 rows, or nothing (gather in the GEMM's producer)
  void* x_sorted = fp8 ? sv + at_.xq : (gather ? (views ? tv + t_xs : nullptr) : sv + at_.x_rows);
  const void* gather_src = fp8 ? tv + t_latq : x_latent;
  const int gather_bytes = fp8 ? d.L : 2 * d.L;
  float* scal = fp8 ? reinterpret_cast<float*>(sv + at_.scal) : nullptr;
  lmoe_fp8_tensor q[3];
  if (fp8) {
    C10_CUDA_CHECK(cudaMemsetAsync(scal, 0, 32 * sizeof(float), stream.stream()));
    q[0] = {x_latent, tv + t_latq, T, d.L, nullptr, amax_of(scal, kSx), deq_of(scal, kSx)};
    q[1] = {o.wgu.data_ptr(), sv + at_.wguq, int64_t(d.E) * d.L, 2 * d.F, nullptr, amax_of(scal, kSwgu), deq_of(scal, kSwgu)};
    q[2] = {o.wde.data_ptr(), sv + at_.wdq, int64_t(d.E) * d.F, d.L, nullptr, amax_of(scal, kSwd), deq_of(scal, kSwd)};
  }
  void* hidden = fp8 ? tv + t_hid : sv + at_.hidden;
  int32_t* sel = r.sel.data_ptr<int32_t>();

  if (gather)  // the pad rows of the routed layout read a row of zeros behind the T latent rows
    C10_CUDA_CHECK(cudaMemsetAsync(static_cast<char*>(x_latent) + T * d.L * 2, 0, d.L * 2, stream.stream()));
  const bool forked = d.T <= kForkForwardTokens && !forced_sel;
  c10::optional<Fork> fork;
  if (forked) fork.emplace(stream);
  if (forced_sel) {  // parity tests: another selection, the gating weights recomputed from this pass's own logits
    LMOE(lmoe_xproj_fwd, &d.s, o.x.data_ptr(), o.wg.data_ptr(), o.wdn.data_ptr(), logits, x_latent, status, st);
    LMOE(lmoe_gate_topk_fwd, &d.s, logits, bias.data_ptr<float>(), z_coef, sel, weights, lse,
         reinterpret_cast<float*>(tv + t_zp), r.z_loss.data_ptr<float>(), st);
    r.sel.copy_(*forced_sel);
    Tensor aff = at::sigmoid(view_of(r.saved, at_.logits, {T, d.E}, at::kFloat)).gather(1, r.sel.to(at::kLong));
    view_of(r.saved, at_.weights, {T, d.K}, at::kFloat).copy_(aff / (aff.sum(-1, true) + 1e-9));
    LMOE(lmoe_route_permute, &d.s, sel, &route, tv + t_ws, ws_bytes, st);
    if (fp8) {
      LMOE(lmoe_fp8_amax, 3, q, st);
      LMOE(lmoe_fp8_cast, 3, q, st);
    }
    if (x_sorted) LMOE(lmoe_gather_rows, gather_src, route.row_src, d.K, P, gather_bytes / 2, route.n_tiles, x_sorted, st);
    LMOE(lmoe_shared_gateup_fwd, &d.s, o.x.data_ptr(), o.wgus.data_ptr(), h1_s, act_cat, status, st);
  } else {
    // Small batches: [x_latent, shared gate_up] on the side stream beside [logits, top-k].  At larger ones every GEMM
    // fills the SMs and the routing kernels' static shared memory does not fit beside a GEMM CTA: one stream.
    void* side = forked ? fork->side() : st;
    if (forked) fork->to_side();
    LMOE(lmoe_xproj_fwd, &d.s, o.x.data_ptr(), o.wg.data_ptr(), nullptr, logits, nullptr, status, st);
    LMOE(lmoe_xproj_fwd, &d.s, o.x.data_ptr(), nullptr, o.wdn.data_ptr(), nullptr, x_latent, status, side);
    LMOE(lmoe_topk_hist_fwd, &d.s, logits, bias.data_ptr<float>(), sel, weights, lse, tv + t_ws, ws_bytes, st);
    if (forked) fork->to_main(true);
    if (fp8) {  // the weights beside the latents: on the side stream, or in the same launches
      const int n = forked ? 1 : 3;
      LMOE(lmoe_fp8_amax, n, q, st);
      LMOE(lmoe_fp8_cast, n, q, st);
      if (forked) {
        LMOE(lmoe_fp8_amax, 2, q + 1, side);
        LMOE(lmoe_fp8_cast, 2, q + 1, side);
      }
    }
    LMOE(lmoe_route_gather_fwd, &d.s, sel, tv + t_ws, ws_bytes, z_coef, r.z_loss.data_ptr<float>(), &route,
         x_sorted ? gather_src : nullptr, gather_bytes, x_sorted, st);
    if (fp8 && forked) fork->to_main(true);
    LMOE(lmoe_shared_gateup_fwd, &d.s, o.x.data_ptr(), o.wgus.data_ptr(), h1_s, act_cat, status, side);
  }

  // routed experts in the padded layout
  if (fp8) {
    void *hq = sv + at_.hq, *wguq = sv + at_.wguq, *wdq = sv + at_.wdq;
    LMOE(lmoe_grouped_gateup_fp8_amax, P, d.E, d.L, d.F, x_sorted, wguq, deq_of(scal, kSx), deq_of(scal, kSwgu), route.tile_expert,
         route.n_tiles, h1, hidden, amax_of(scal, kSh), status, st);
    const lmoe_fp8_tensor h = {hidden, hq, P, d.F, route.n_tiles, amax_of(scal, kSh), deq_of(scal, kSh)};
    LMOE(lmoe_fp8_cast, 1, &h, st);
    LMOE(lmoe_grouped_rows_fp8, P, d.E, d.F, d.L, hq, wdq, 1, deq_of(scal, kSh), deq_of(scal, kSwd), route.tile_expert,
         route.n_tiles, y_sorted, status, st);
  } else if (gather) {
    LMOE(lmoe_grouped_fwd_gather, P, d.E, d.L, d.F, x_latent, T + 1, route.row_src, 1, d.K, T, o.wgu.data_ptr(),
         o.wde.data_ptr(), route.tile_expert, route.n_tiles, h1, hidden, y_sorted, status, st);
  } else {
    LMOE(lmoe_grouped_fwd, P, d.E, d.L, d.F, x_sorted, o.wgu.data_ptr(), o.wde.data_ptr(), route.tile_expert, route.n_tiles,
         route.pad_offsets, h1, hidden, y_sorted, status, st);
  }
  // weighted combine, up-projection, shared down-projection, add
  if (forked) fork->to_main();
  LMOE(lmoe_combine_out_fwd, &d.s, y_sorted, &route, weights, act_cat, o.wds.data_ptr(), o.wup.data_ptr(), r.y.data_ptr(),
       status, st);

  if (views) {
    const auto bf = at::kBFloat16;
    views->emplace_back("logits", view_of(r.saved, at_.logits, {T, d.E}, at::kFloat));
    views->emplace_back("weights", view_of(r.saved, at_.weights, {T, d.K}, at::kFloat));
    views->emplace_back("lse", view_of(r.saved, at_.lse, {T}, at::kFloat));
    views->emplace_back("route_storage", view_of(r.saved, at_.route, {d.route_ints()}, at::kInt));
    views->emplace_back("x_latent", gather ? view_of(r.saved, at_.x_rows, {T, d.L}, bf) : view_of(tmp, t_lat, {T, d.L}, bf));
    if (!fp8) views->emplace_back("x_sorted", gather ? view_of(tmp, t_xs, {P, d.L}, bf) : view_of(r.saved, at_.x_rows, {P, d.L}, bf));
    views->emplace_back("h1", view_of(r.saved, at_.h1, {P, 2 * d.F}, bf));
    views->emplace_back("hidden", fp8 ? view_of(tmp, t_hid, {P, d.F}, bf) : view_of(r.saved, at_.hidden, {P, d.F}, bf));
    views->emplace_back("y_sorted", view_of(r.saved, at_.y_sorted, {P, d.L}, bf));
    views->emplace_back("h1_s", view_of(r.saved, at_.h1_s, {T, 2 * d.Fs}, bf));
    Tensor cat = view_of(r.saved, at_.act_cat, {T, d.L + d.Fs}, bf);
    views->emplace_back("routed", cat.narrow(1, 0, d.L));
    views->emplace_back("hidden_s", cat.narrow(1, d.L, d.Fs));
    views->emplace_back("status", at::from_blob(status, {1}, at::TensorOptions().dtype(at::kInt)));
  }
  return r;
}

// ---------------------------------------------------------------- LatentMoE: backward
struct LatentGrads {
  Tensor dx, wg, wdn, wup, wgus, wds, wgu, wde;  // dx and the expert gradients bf16; the linears' in `lin_dtype`
};

LatentGrads latent_backward(const Sizes& d, const LatentOps& o, const Tensor& dy, const float* dz, const Tensor& sel_t,
                            const Tensor& saved, float z_coef, bool fp8, at::ScalarType lin_dtype, Views* views) {
  const auto stream = at::cuda::getCurrentCUDAStream();
  void* st = stream.stream();
  int32_t* status = status_word(kLatentBwd);
  const bool gather = tma_gather_enabled() && !fp8 && d.L % 128 == 0;
  const LatentLayout at_(d, fp8, gather);
  TORCH_CHECK(saved.numel() == static_cast<int64_t>(at_.bytes), "saved activations of another shape");
  const int64_t T = d.T, P = d.P, ld_cat = 2 * int64_t(d.Fs) + d.L + d.E;
  const int gtype = lin_dtype == at::kFloat ? LMOE_F32 : LMOE_BF16;
  const auto bf = o.x.options().requires_grad(false);
  const auto lin = bf.dtype(lin_dtype);

  LatentGrads g;
  g.dx = at::empty({T, d.D}, bf);
  g.wg = at::empty({d.E, d.D}, lin);
  g.wdn = at::empty({d.L, d.D}, lin);
  g.wup = at::empty({d.D, d.L}, lin);
  g.wgus = at::empty({2 * d.Fs, d.D}, lin);
  g.wds = at::empty({d.D, d.Fs}, lin);
  g.wgu = at::empty({d.E, d.L, 2 * d.F}, bf);
  g.wde = at::empty({d.E, d.F, d.L}, bf);

  Carver c;
  const size_t ws_bytes = std::max<size_t>(16, lmoe_wgrad_workspace_bytes(&d.s));
  const size_t t_ws = c.take(ws_bytes), t_dr = c.take(T * d.L * 2), t_cat = c.take(T * ld_cat * 2);
  const size_t t_dw = c.take(T * d.K * 4), t_dys = c.take(P * d.L * (fp8 ? 1 : 2)), t_dh1 = c.take(P * 2 * d.F * 2);
  const size_t t_dxs = c.take(P * d.L * 2);
  const size_t t_dh1q = fp8 ? c.take(P * 2 * d.F) : 0;
  const size_t t_scal = fp8 ? c.take(kScals * 2 * sizeof(float)) : 0;
  Tensor tmp = new_bytes(c.bytes, o.x);
  char *tv = base_of(tmp), *sv = base_of(saved);
  // the forward's scales are read; the backward's own are scratch (what is saved may be read by another backward at the time)
  float* scal = fp8 ? reinterpret_cast<float*>(sv + at_.scal) : nullptr;
  float* d_scal = fp8 ? reinterpret_cast<float*>(tv + t_scal) : nullptr;
  if (fp8) C10_CUDA_CHECK(cudaMemsetAsync(d_scal, 0, kScals * 2 * sizeof(float), stream.stream()));

  float* logits = reinterpret_cast<float*>(sv + at_.logits);
  float* weights = reinterpret_cast<float*>(sv + at_.weights);
  float* lse = reinterpret_cast<float*>(sv + at_.lse);
  const int32_t* sel = sel_t.data_ptr<int32_t>();
  const lmoe_route route = d.route(sv + at_.route, nullptr);
  void *act_cat = sv + at_.act_cat, *h1_s = sv + at_.h1_s, *y_sorted = sv + at_.y_sorted, *h1 = sv + at_.h1;
  void *ws = tv + t_ws, *d_routed = tv + t_dr, *cat = tv + t_cat, *d_ys = tv + t_dys, *d_h1 = tv + t_dh1, *d_xs = tv + t_dxs;
  float* d_w = reinterpret_cast<float*>(tv + t_dw);

  // output stage dgrads, then [adjoint of the combine] beside [output-stage weight gradients]; the shared expert's SwiGLU
  // adjoint runs in the epilogue of the d_hidden_s GEMM
  Fork fork(stream);
  void* side = fork.side();
  LMOE(lmoe_combine_out_bwd_dgrad, &d.s, dy.data_ptr(), o.wup.data_ptr(), o.wds.data_ptr(), h1_s, d_routed, nullptr, cat,
       status, st);
  fork.to_side();
  if (fp8)
    LMOE(lmoe_fp8_combine_bwd, &d.s, d_routed, y_sorted, weights, &route, amax_of(d_scal, kSdy), deq_of(d_scal, kSdy), d_ys, d_w, side);
  else
    LMOE(lmoe_combine_bwd, &d.s, d_routed, y_sorted, weights, &route, d_ys, d_w, side);
  LMOE(lmoe_combine_out_bwd_wgrad, &d.s, dy.data_ptr(), act_cat, g.wup.data_ptr(), g.wds.data_ptr(), gtype, ws, ws_bytes,
       status, st);
  fork.to_main();

  if (fp8) {
    void *xq = sv + at_.xq, *hq = sv + at_.hq, *wguq = sv + at_.wguq, *wdq = sv + at_.wdq, *dyq = d_ys, *dh1q = tv + t_dh1q;
    // d_h1 = swiglu'(h1, d_y * Wd[e]^T): the down weights [E, F, L] read as [N = F rows, K = L] (K-major operand)
    LMOE(lmoe_grouped_swiglu_bwd_fp8, P, d.E, d.L, d.F, dyq, wdq, deq_of(d_scal, kSdy), deq_of(scal, kSwd), route.tile_expert,
         route.n_tiles, h1, d_h1, amax_of(d_scal, kSdh1), status, st);
    const lmoe_fp8_tensor h = {d_h1, dh1q, P, 2 * d.F, route.n_tiles, amax_of(d_scal, kSdh1), deq_of(d_scal, kSdh1)};
    LMOE(lmoe_fp8_cast, 1, &h, st);
    // d_x_sorted = d_h1 * Wgu[e]^T: the gate_up weights [E, L, 2F] read as [N = L rows, K = 2F]
    LMOE(lmoe_grouped_rows_fp8, P, d.E, 2 * d.F, d.L, dh1q, wguq, 0, deq_of(d_scal, kSdh1), deq_of(scal, kSwgu),
         route.tile_expert, route.n_tiles, d_xs, status, st);
    fork.to_side();
    LMOE(lmoe_unpermute_sum_bwd, &d.s, d_xs, &route, cat, side);
    LMOE(lmoe_gate_topk_bwd, &d.s, logits, sel, weights, d_w, lse, dz, z_coef, cat, side);
    LMOE(lmoe_grouped_wgrad_fp8, P, d.E, d.L, 2 * d.F, xq, dh1q, deq_of(scal, kSx), deq_of(d_scal, kSdh1), route.pad_offsets,
         g.wgu.data_ptr(), status, st);
    LMOE(lmoe_grouped_wgrad_fp8, P, d.E, d.F, d.L, hq, dyq, deq_of(scal, kSh), deq_of(d_scal, kSdy), route.pad_offsets,
         g.wde.data_ptr(), status, st);
    fork.to_main();
  } else {
    void *x_rows = sv + at_.x_rows, *hidden = sv + at_.hidden;
    // d_h1 = swiglu'(h1, d_y_sorted * Wd[e]^T), d_x_sorted = d_h1 * Wgu[e]^T; d_hidden never reaches memory
    LMOE(lmoe_grouped_bwd_dgrad, P, d.E, d.L, d.F, d_ys, h1, o.wgu.data_ptr(), o.wde.data_ptr(), route.tile_expert, route.n_tiles, route.pad_offsets,
         nullptr, d_h1, d_xs, status, st);
    // [gather adjoint + router adjoint] beside [routed weight gradients]
    fork.to_side();
    LMOE(lmoe_unpermute_sum_bwd, &d.s, d_xs, &route, cat, side);
    LMOE(lmoe_gate_topk_bwd, &d.s, logits, sel, weights, d_w, lse, dz, z_coef, cat, side);
    if (gather)
      LMOE(lmoe_grouped_bwd_wgrad_gather, P, d.E, d.L, d.F, x_rows, T + 1, route.row_src, 1, d.K, T, d_h1, hidden, d_ys,
           route.pad_offsets, g.wgu.data_ptr(), g.wde.data_ptr(), status, st);
    else
      LMOE(lmoe_grouped_bwd_wgrad, P, d.E, d.L, d.F, x_rows, d_h1, hidden, d_ys, route.pad_offsets, g.wgu.data_ptr(),
           g.wde.data_ptr(), status, st);
    fork.to_main();
  }
  // x side: dx and the three weight gradients that contract with x
  LMOE(lmoe_xside_bwd, &d.s, cat, o.wgus.data_ptr(), o.wdn.data_ptr(), o.wg.data_ptr(), o.x.data_ptr(), g.dx.data_ptr(),
       g.wgus.data_ptr(), g.wdn.data_ptr(), g.wg.data_ptr(), gtype, ws, ws_bytes, status, st);

  if (views) {
    const auto b16 = at::kBFloat16;
    Tensor cv = view_of(tmp, t_cat, {T, ld_cat}, b16);
    views->emplace_back("d_routed", view_of(tmp, t_dr, {T, d.L}, b16));
    views->emplace_back("d_h1_s", cv.narrow(1, 0, 2 * d.Fs));
    views->emplace_back("d_x_latent", cv.narrow(1, 2 * d.Fs, d.L));
    views->emplace_back("d_logits", cv.narrow(1, 2 * d.Fs + d.L, d.E));
    views->emplace_back("d_weights", view_of(tmp, t_dw, {T, d.K}, at::kFloat));
    if (!fp8) views->emplace_back("d_y_sorted", view_of(tmp, t_dys, {P, d.L}, b16));
    views->emplace_back("d_h1", view_of(tmp, t_dh1, {P, 2 * d.F}, b16));
    views->emplace_back("d_x_sorted", view_of(tmp, t_dxs, {P, d.L}, b16));
  }
  return g;
}

// dz as a device scalar in fp32; `keep` owns the memory.
const float* scalar_grad(const Tensor& d_z, Tensor& keep) {
  if (!d_z.defined()) return nullptr;
  keep = d_z.detach().to(at::kFloat).contiguous();
  return keep.data_ptr<float>();
}

// ---------------------------------------------------------------- non-latent MoE layer
// The same kernels at the model width (L = D): x itself is gathered into the padded layout and the weighted sum of the
// expert outputs is added to the shared expert's output (models/moe.py:344-372).
struct MoeLayout {  // !keep: no backward follows, no gate / up
  size_t logits, weights, lse, route, x_sorted, h1, hidden, y_sorted, h1_s, hidden_s, bytes;
  explicit MoeLayout(const Sizes& d, bool keep = true) {
    Carver c;
    const int64_t T = d.T, P = d.P;
    logits = c.take(T * d.E * 4);
    weights = c.take(T * d.K * 4);
    lse = c.take(T * 4);
    route = c.take(d.route_ints() * 4);
    x_sorted = c.take(P * d.D * 2);
    h1 = c.take(keep ? P * 2 * d.F * 2 : 0);
    hidden = c.take(P * d.F * 2);
    y_sorted = c.take(P * d.D * 2);
    h1_s = c.take(keep ? T * 2 * d.Fs * 2 : 0);
    hidden_s = c.take(T * d.Fs * 2);
    bytes = c.bytes;
  }
};

struct MoeOps {
  Tensor x, wg, wgus, wds, wgu, wde;
};

Sizes moe_sizes(const Tensor& x2d, const Tensor& wgu, const Tensor& wds, int64_t top_k) {
  TORCH_CHECK(wgu.dim() == 3 && x2d.size(1) == wgu.size(1), "activation of another width than the layer's");
  return Sizes(x2d.size(0), x2d.size(1), x2d.size(1), wgu.size(0), top_k, wgu.size(2) / 2, wds.size(1));
}

LatentOut moe_forward(const Sizes& d, const MoeOps& o, const Tensor& bias, float z_coef, bool keep,
                      const c10::optional<Tensor>& forced_sel) {
  const auto stream = at::cuda::getCurrentCUDAStream();
  void* st = stream.stream();
  int32_t* status = status_word(kMoeFwd);
  const MoeLayout at_(d, keep);
  const int64_t T = d.T, P = d.P, D = d.D;
  LatentOut r;
  const auto f32 = o.x.options().dtype(at::kFloat).requires_grad(false);
  r.y = at::empty({T, D}, o.x.options().requires_grad(false));
  r.z_loss = at::empty({}, f32);
  r.sel = at::empty({T, d.K}, f32.dtype(at::kInt));
  r.counts = at::empty({d.E}, f32.dtype(at::kInt));
  r.saved = new_bytes(at_.bytes, o.x);
  char* sv = base_of(r.saved);
  Carver c;
  const size_t ws_bytes = std::max<size_t>({16, lmoe_route_workspace_bytes(&d.s), lmoe_route_fwd_workspace_bytes(&d.s)});
  const size_t t_ws = c.take(ws_bytes), t_zp = forced_sel ? c.take((T + 7) / 8 * 4) : 0, t_ysh = c.take(T * D * 2);
  Tensor tmp = new_bytes(c.bytes, o.x);
  char* tv = base_of(tmp);
  float* logits = reinterpret_cast<float*>(sv + at_.logits);
  float* weights = reinterpret_cast<float*>(sv + at_.weights);
  float* lse = reinterpret_cast<float*>(sv + at_.lse);
  const lmoe_route route = d.route(sv + at_.route, r.counts.data_ptr<int32_t>());
  int32_t* sel = r.sel.data_ptr<int32_t>();
  const void* x = o.x.data_ptr();

  // Small batches: the shared expert on the side stream beside the router and the experts, whose GEMMs leave SMs free then.
  // (335 tokens 121 -> 97 us; from kForkForwardTokens on either side fills the SMs by itself)
  const bool forked = d.T <= kForkForwardTokens && !forced_sel;
  c10::optional<Fork> fork;
  if (forked) fork.emplace(stream);
  void* side = forked ? fork->side() : st;
  void* h1 = keep ? sv + at_.h1 : nullptr;
  void* h1_s = keep ? sv + at_.h1_s : nullptr;
  auto shared_expert = [&] {                                            // (moe.py:351-354, 63-69)
    LMOE(lmoe_gemm_swiglu_bf16, d.T, d.Fs, d.D, x, D, o.wgus.data_ptr(), D, h1_s, 2 * int64_t(d.Fs), sv + at_.hidden_s,
         d.Fs, status, side);
    LMOE(lmoe_gemm_bf16, d.T, d.D, d.Fs, sv + at_.hidden_s, d.Fs, 0, o.wds.data_ptr(), d.Fs, 0, tv + t_ysh, D, LMOE_BF16, 1,
         nullptr, 0, status, side);
  };
  if (forked) {
    fork->to_side();
    shared_expert();
  }

  // router: fp32 logits, top-k, z-loss; routing tables                         (moe.py:357-358)
  LMOE(lmoe_gemm_bf16, d.T, d.E, d.D, x, D, 0, o.wg.data_ptr(), D, 0, logits, d.E, LMOE_F32, 1, nullptr, 0, status, st);
  if (forced_sel) {  // parity tests only
    LMOE(lmoe_gate_topk_fwd, &d.s, logits, bias.data_ptr<float>(), z_coef, sel, weights, lse,
         reinterpret_cast<float*>(tv + t_zp), r.z_loss.data_ptr<float>(), st);
    r.sel.copy_(*forced_sel);
    Tensor aff = at::sigmoid(view_of(r.saved, at_.logits, {T, d.E}, at::kFloat)).gather(1, r.sel.to(at::kLong));
    view_of(r.saved, at_.weights, {T, d.K}, at::kFloat).copy_(aff / (aff.sum(-1, true) + 1e-9));
    LMOE(lmoe_route_permute, &d.s, sel, &route, tv + t_ws, ws_bytes, st);
    LMOE(lmoe_gather_rows, x, route.row_src, d.K, P, d.D, route.n_tiles, sv + at_.x_sorted, st);
  } else {
    LMOE(lmoe_topk_hist_fwd, &d.s, logits, bias.data_ptr<float>(), sel, weights, lse, tv + t_ws, ws_bytes, st);
    LMOE(lmoe_route_gather_fwd, &d.s, sel, tv + t_ws, ws_bytes, z_coef, r.z_loss.data_ptr<float>(), &route, x, 2 * d.D,
         sv + at_.x_sorted, st);
  }
  // routed experts on x itself                                                 (moe.py:462-470, 509-532)
  LMOE(lmoe_grouped_fwd, P, d.E, d.D, d.F, sv + at_.x_sorted, o.wgu.data_ptr(), o.wde.data_ptr(), route.tile_expert,
       route.n_tiles, route.pad_offsets, h1, sv + at_.hidden, sv + at_.y_sorted, status, st);
  if (forked)
    fork->to_main();
  else
    shared_expert();
  // y = shared + sum_k w_k * expert_k(x)                                       (moe.py:534, 473-479, 366)
  LMOE(lmoe_combine_rows_add, sv + at_.y_sorted, route.pos, weights, tv + t_ysh, D, d.T, d.K, d.D, r.y.data_ptr(), D, st);
  return r;
}

struct MoeGrads {
  Tensor dx, wg, wgus, wds, wgu, wde;
};

MoeGrads moe_backward(const Sizes& d, const MoeOps& o, const Tensor& dy, const float* dz, const Tensor& sel_t,
                      const Tensor& saved, float z_coef, at::ScalarType lin_dtype) {
  const auto stream = at::cuda::getCurrentCUDAStream();
  void* st = stream.stream();
  int32_t* status = status_word(kMoeBwd);
  const MoeLayout at_(d);
  const int64_t T = d.T, P = d.P, D = d.D, ld_cat = 2 * int64_t(d.Fs) + d.E;
  const int gtype = lin_dtype == at::kFloat ? LMOE_F32 : LMOE_BF16;
  const auto bf = o.x.options().requires_grad(false);
  const auto lin = bf.dtype(lin_dtype);
  MoeGrads g;
  g.dx = at::empty({T, D}, bf);
  g.wg = at::empty({d.E, D}, lin);
  g.wgus = at::empty({2 * d.Fs, D}, lin);
  g.wds = at::empty({D, d.Fs}, lin);
  g.wgu = at::empty({d.E, D, 2 * d.F}, bf);
  g.wde = at::empty({d.E, d.F, D}, bf);
  Carver c;
  const size_t ws_bytes = std::max<size_t>(16, lmoe_moe_wgrad_workspace_bytes(&d.s));
  const size_t t_ws = c.take(ws_bytes), t_cat = c.take(T * ld_cat * 2), t_dw = c.take(T * d.K * 4);
  const size_t t_dys = c.take(P * D * 2), t_dh1 = c.take(P * 2 * d.F * 2), t_dxs = c.take(P * D * 2), t_dx = c.take(T * D * 2);
  Tensor tmp = new_bytes(c.bytes, o.x);
  char *tv = base_of(tmp), *sv = base_of(saved);
  float* logits = reinterpret_cast<float*>(sv + at_.logits);
  float* weights = reinterpret_cast<float*>(sv + at_.weights);
  float* lse = reinterpret_cast<float*>(sv + at_.lse);
  const lmoe_route route = d.route(sv + at_.route, nullptr);
  float* d_w = reinterpret_cast<float*>(tv + t_dw);
  void *cat = tv + t_cat, *ws = tv + t_ws, *d_ys = tv + t_dys, *d_h1 = tv + t_dh1, *d_xs = tv + t_dxs;

  // [adjoint of the weighted sum: d_y_sorted = w * dy[t], d_w = <dy[t], y_sorted>] beside
  // [shared expert: d_h1_s (SwiGLU adjoint in the epilogue) -> cat[:, :2Fs]; d_Wd_s = dy^T * hidden_s]
  // (both side sections: 924 tokens 354 -> 323 us with both directions; at 4,096 tokens, 550 us, within the 3 % between runs)
  Fork fork(stream);
  void* side = fork.side();
  fork.to_side();
  LMOE(lmoe_moe_shared_bwd, &d.s, dy.data_ptr(), o.wds.data_ptr(), sv + at_.h1_s, sv + at_.hidden_s, cat, g.wds.data_ptr(), gtype,
       ws, ws_bytes, status, st);
  LMOE(lmoe_combine_bwd, &d.s, dy.data_ptr(), sv + at_.y_sorted, weights, &route, d_ys, d_w, side);
  fork.to_main();
  // routed experts
  LMOE(lmoe_moe_experts_bwd_dgrad, P, d.E, d.D, d.F, d_ys, sv + at_.h1, o.wgu.data_ptr(), o.wde.data_ptr(), route.tile_expert,
       route.n_tiles, route.pad_offsets, d_h1, d_xs, status, st);
  // [router adjoint (+ z-loss) -> cat[:, 2Fs:]; the entry point places d_logits after 2Fs + L columns] beside
  // [routed weight gradients]
  lmoe_shape cat_shape = d.s;
  cat_shape.L = 0;
  fork.to_side();
  LMOE(lmoe_gate_topk_bwd, &cat_shape, logits, sel_t.data_ptr<int32_t>(), weights, d_w, lse, dz, z_coef, cat, side);
  LMOE(lmoe_grouped_bwd_wgrad, P, d.E, d.D, d.F, sv + at_.x_sorted, d_h1, sv + at_.hidden, d_ys, route.pad_offsets,
       g.wgu.data_ptr(), g.wde.data_ptr(), status, st);
  fork.to_main();
  // x side: dx = [d_h1_s | d_logits] * [Wgu_s ; Wg] + sum_k d_x_sorted; [d_Wgu_s ; d_Wg] = [d_h1_s | d_logits]^T * x
  LMOE(lmoe_moe_xside_bwd, &d.s, cat, o.wgus.data_ptr(), o.wg.data_ptr(), o.x.data_ptr(), tv + t_dx, g.wgus.data_ptr(),
       g.wg.data_ptr(), gtype, ws, ws_bytes, status, st);
  LMOE(lmoe_combine_rows_add, d_xs, route.pos, nullptr, tv + t_dx, D, d.T, d.K, d.D, g.dx.data_ptr(), D, st);
  return g;
}

// ---------------------------------------------------------------- a few tokens, no backward
// For a module in evaluation mode only: the sums run in another order than in the training forward, which an activation
// checkpoint recomputes bit for bit.
std::vector<Tensor> few_forward(const Sizes& d, const Tensor& x2d, const Tensor& wg, const Tensor* wdn, const Tensor* wup,
                                const Tensor& wgus, const Tensor& wds, const Tensor& wgu, const Tensor& wde, const Tensor& bias,
                                float z_coef) {
  Tensor y = at::empty({d.T, d.D}, x2d.options());
  Tensor z = at::empty({}, x2d.options().dtype(at::kFloat));
  const size_t n = lmoe_few_workspace_bytes(&d.s);
  Tensor ws = new_bytes(n, x2d);
  LMOE(lmoe_few_forward, &d.s, x2d.data_ptr(), wg.data_ptr(), wdn ? wdn->data_ptr() : nullptr, wup ? wup->data_ptr() : nullptr,
       wgus.data_ptr(), wds.data_ptr(), wgu.data_ptr(), wde.data_ptr(), bias.data_ptr<float>(), z_coef, y.data_ptr(),
       z.data_ptr<float>(), ws.data_ptr(), n, status_word(wdn ? kLatentFwd : kMoeFwd), at::cuda::getCurrentCUDAStream().stream());
  return {y, z};
}

// ---------------------------------------------------------------- autograd


// torch.jit.trace would bake the results of a native call in as constants.
void require_cuda(const Tensor& x, const char* what) {
  if (torch::jit::tracer::isTracing()) throw LmoeFailure(std::string("the ") + what + " path cannot be recorded by torch.jit.trace");
  if (!x.is_cuda()) throw LmoeFailure(std::string("the ") + what + " path runs on a CUDA device only (no CPU fallback)");
}

// The dtype of the dense linears' gradients: fp32 when any of them is fp32.
at::ScalarType lin_dtype_of(std::initializer_list<at::ScalarType> dts) {
  for (auto t : dts)
    if (t == at::kFloat) return at::kFloat;
  return at::kBFloat16;
}

LatentOps latent_ops(const Tensor& x, const Tensor& wg, const Tensor& wdn, const Tensor& wup, const Tensor& wgus,
                     const Tensor& wds, const Tensor& wgu, const Tensor& wde) {
  Caster cast(x);
  LatentOps o{cast(x).view({-1, x.size(-1)}), cast(wg), cast(wdn), cast(wup), cast(wgus), cast(wds), cast(wgu), cast(wde)};
  cast.run(at::cuda::getCurrentCUDAStream().stream());
  return o;
}

std::vector<int64_t> dtypes_of(const std::vector<Tensor>& ts) {
  std::vector<int64_t> v;
  for (const auto& t : ts) v.push_back(static_cast<int64_t>(t.scalar_type()));
  return v;
}

Tensor grad_rows(const Tensor& dy, const Tensor& like2d) {
  if (!dy.defined()) return at::zeros_like(like2d);
  Caster cast(like2d);
  Tensor d = cast(dy);
  cast.run(at::cuda::getCurrentCUDAStream().stream());
  return d.view({like2d.size(0), like2d.size(1)});
}

// y, aux_loss, sel, counts = f(x, ...); y has x's shape and dtype.
class LatentFn : public torch::autograd::Function<LatentFn> {
 public:
  static variable_list forward(AutogradContext* ctx, const Tensor& x, const Tensor& wg, const Tensor& wdn, const Tensor& wup,
                               const Tensor& wgus, const Tensor& wds, const Tensor& wgu, const Tensor& wde, const Tensor& bias,
                               int64_t top_k, double z_coef, bool fp8) {
    const LatentOps o = latent_ops(x, wg, wdn, wup, wgus, wds, wgu, wde);
    const Sizes d = latent_sizes(o.x, o.wgu, o.wds, top_k);
    LatentOut r = latent_forward(d, o, f32_bias(bias, x), static_cast<float>(z_coef), fp8, true, c10::nullopt, nullptr);
    ctx->set_materialize_grads(false);
    // e4m3: the quantised copies in `saved` replace the bf16 expert weights
    const Tensor none = fp8 ? Tensor() : o.wgu;
    ctx->save_for_backward({o.x, o.wg, o.wdn, o.wup, o.wgus, o.wds, none, fp8 ? Tensor() : o.wde, r.sel, r.saved});
    ctx->saved_data["i"] = std::vector<int64_t>{d.L, d.E, d.K, d.F, d.Fs, fp8};
    ctx->saved_data["t"] = dtypes_of({x, wg, wdn, wup, wgus, wds, wgu, wde});
    ctx->saved_data["s"] = x.sizes().vec();
    ctx->saved_data["z"] = z_coef;
    ctx->mark_non_differentiable({r.sel, r.counts});
    return {as_param(shaped(r.y, x.sizes()), x.scalar_type()), r.z_loss, r.sel, r.counts};
  }

  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    try {
      const auto sv = ctx->get_saved_variables();
      const auto i = ctx->saved_data["i"].toIntVector();
      const auto t = ctx->saved_data["t"].toIntVector();
      const c10::cuda::CUDAGuard guard(sv[0].device());
      const LatentOps o{sv[0], sv[1], sv[2], sv[3], sv[4], sv[5], sv[6], sv[7]};
      const Sizes d(o.x.size(0), o.x.size(1), i[0], i[1], i[2], i[3], i[4]);
      Tensor keep;
      const float* dz = scalar_grad(grads[1], keep);
      auto dt = [&t](int k) { return static_cast<at::ScalarType>(t[k]); };
      const auto lin = lin_dtype_of({dt(1), dt(2), dt(3), dt(4), dt(5)});
      LatentGrads g = latent_backward(d, o, grad_rows(grads[0], o.x), dz, sv[8], sv[9],
                                      static_cast<float>(ctx->saved_data["z"].toDouble()), i[5] != 0, lin, nullptr);
      Tensor dx = g.dx.view(ctx->saved_data["s"].toIntVector());
      const Tensor none;
      return {as_param(dx, dt(0)),     as_param(g.wg, dt(1)),  as_param(g.wdn, dt(2)), as_param(g.wup, dt(3)), as_param(g.wgus, dt(4)),
              as_param(g.wds, dt(5)), as_param(g.wgu, dt(6)), as_param(g.wde, dt(7)), none, none, none, none};
    } catch (const LmoeFailure& e) {
      rethrow_as_python(e);
    }
  }
};

class MoeFn : public torch::autograd::Function<MoeFn> {
 public:
  static variable_list forward(AutogradContext* ctx, const Tensor& x, const Tensor& wg, const Tensor& wgus, const Tensor& wds,
                               const Tensor& wgu, const Tensor& wde, const Tensor& bias, int64_t top_k, double z_coef,
                               const c10::optional<Tensor>& forced) {
    Caster cast(x);
    const MoeOps o{cast(x).view({-1, x.size(-1)}), cast(wg), cast(wgus), cast(wds), cast(wgu), cast(wde)};
    cast.run(at::cuda::getCurrentCUDAStream().stream());
    const Sizes d = moe_sizes(o.x, o.wgu, o.wds, top_k);
    LatentOut r = moe_forward(d, o, f32_bias(bias, x), static_cast<float>(z_coef), true, forced);
    ctx->set_materialize_grads(false);
    ctx->save_for_backward({o.x, o.wg, o.wgus, o.wds, o.wgu, o.wde, r.sel, r.saved});
    ctx->saved_data["i"] = std::vector<int64_t>{d.E, d.K, d.F, d.Fs};
    ctx->saved_data["t"] = dtypes_of({x, wg, wgus, wds, wgu, wde});
    ctx->saved_data["s"] = x.sizes().vec();
    ctx->saved_data["z"] = z_coef;
    ctx->mark_non_differentiable({r.sel, r.counts});
    return {as_param(shaped(r.y, x.sizes()), x.scalar_type()), r.z_loss, r.sel, r.counts};
  }

  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    try {
      const auto sv = ctx->get_saved_variables();
      const auto i = ctx->saved_data["i"].toIntVector();
      const auto t = ctx->saved_data["t"].toIntVector();
      const c10::cuda::CUDAGuard guard(sv[0].device());
      const MoeOps o{sv[0], sv[1], sv[2], sv[3], sv[4], sv[5]};
      const Sizes d(o.x.size(0), o.x.size(1), o.x.size(1), i[0], i[1], i[2], i[3]);
      Tensor keep;
      const float* dz = scalar_grad(grads[1], keep);
      auto dt = [&t](int k) { return static_cast<at::ScalarType>(t[k]); };
      MoeGrads g = moe_backward(d, o, grad_rows(grads[0], o.x), dz, sv[6], sv[7],
                                static_cast<float>(ctx->saved_data["z"].toDouble()), lin_dtype_of({dt(1), dt(2), dt(3)}));
      Tensor dx = g.dx.view(ctx->saved_data["s"].toIntVector());
      const Tensor none;
      return {as_param(dx, dt(0)),    as_param(g.wg, dt(1)),  as_param(g.wgus, dt(2)), as_param(g.wds, dt(3)),
              as_param(g.wgu, dt(4)), as_param(g.wde, dt(5)), none, none, none, none};
    } catch (const LmoeFailure& e) {
      rethrow_as_python(e);
    }
  }
};

// ---------------------------------------------------------------- norm and residual either side of a feed-forward layer
int lmoe_type(const Tensor& t) { return t.scalar_type() == at::kFloat ? LMOE_F32 : LMOE_BF16; }
bool aligned(const Tensor& t) { return reinterpret_cast<uintptr_t>(t.data_ptr()) % 16 == 0; }
// bf16 and fp32 pass as they are; anything else in fp32
Tensor rows_of(const Tensor& t) {
  const Tensor d = t.detach();
  return (d.scalar_type() == at::kFloat || d.scalar_type() == at::kBFloat16 ? d : d.to(at::kFloat)).contiguous();
}
// ... where the 16 bytes that the kernels read at once begin: a slice of a flat parameter or of another gradient need not
Tensor aligned_rows_of(const Tensor& t) {
  const Tensor r = rows_of(t);
  return aligned(r) ? r : r.clone();
}

// (xn, x_pass) = (rmsnorm(x) * weight, x).  x_pass is x itself, handed on to the residual add, so that the backward sees the
// gradients of both branches in one call and adds them inside the norm's adjoint.  `keep`: a backward may follow; it reads
// copies that the norm's kernel wrote (an fp32 stream's rows as the norm saw them, a bf16 weight in fp32), so that either may be
// changed in place in between.  What is bf16 rows or an fp32 weight is kept as it is, under autograd's check.
class NormFn : public torch::autograd::Function<NormFn> {
 public:
  static variable_list forward(AutogradContext* ctx, const Tensor& x, const Tensor& weight, double eps, bool bf16_out, bool keep) {
    const Tensor xr = rows_of(x), w = aligned_rows_of(weight);
    TORCH_CHECK(x.dim() > 0 && weight.numel() == x.size(-1), "the norm's weight has another width than its input");
    const int64_t D = x.size(-1), T = xr.numel() / D;
    const bool wide = !bf16_out && xr.scalar_type() == at::kFloat;
    Tensor xn = at::empty(x.sizes(), xr.options().dtype(wide ? at::kFloat : at::kBFloat16));
    Tensor rstd = at::empty({T}, xr.options().dtype(at::kFloat));
    Tensor x_keep, w_keep;
    if (keep && xr.scalar_type() == at::kFloat) x_keep = at::empty(xr.sizes(), xr.options().dtype(at::kBFloat16));
    if (keep && w.scalar_type() == at::kBFloat16) w_keep = at::empty({D}, w.options().dtype(at::kFloat));
    LMOE(lmoe_rmsnorm_fwd_keep, xr.data_ptr(), lmoe_type(xr), w.data_ptr(), lmoe_type(w), static_cast<float>(eps), T, static_cast<int>(D),
         xn.data_ptr(), lmoe_type(xn), rstd.data_ptr<float>(), x_keep.defined() ? x_keep.data_ptr() : nullptr,
         w_keep.defined() ? w_keep.data_ptr<float>() : nullptr, at::cuda::getCurrentCUDAStream().stream());
    ctx->set_materialize_grads(false);
    ctx->save_for_backward({x_keep.defined() ? x_keep : xr, w_keep.defined() ? w_keep : w, rstd});
    ctx->saved_data["t"] = dtypes_of({x, weight});
    ctx->saved_data["s"] = std::vector<int64_t>{static_cast<int64_t>(xr.scalar_type()), static_cast<int64_t>(w.scalar_type())};
    return {bf16_out ? xn : as_param(xn, x.scalar_type()), x};
  }

  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    try {
      const auto sv = ctx->get_saved_variables();
      const Tensor &x = sv[0], &w = sv[1], &rstd = sv[2];
      const c10::cuda::CUDAGuard guard(x.device());
      const auto t = ctx->saved_data["t"].toIntVector();
      const auto x_type = static_cast<at::ScalarType>(t[0]), w_type = static_cast<at::ScalarType>(t[1]);
      const auto s = ctx->saved_data["s"].toIntVector();  // the types that the forward's kernel took
      const auto stream_type = static_cast<at::ScalarType>(s[0]), dw_type = static_cast<at::ScalarType>(s[1]);
      const int64_t D = x.size(-1), T = x.numel() / D;
      const Tensor g = grads[0].defined() ? aligned_rows_of(grads[0]) : at::zeros_like(x);
      Tensor r;
      if (grads[1].defined()) r = aligned_rows_of(grads[1].to(stream_type));
      Tensor dx = at::empty(x.sizes(), x.options().dtype(stream_type));
      Tensor dw = at::empty({D}, x.options().dtype(dw_type));
      Tensor ws = new_bytes(lmoe_rmsnorm_workspace_bytes(static_cast<int>(D)), x);
      LMOE(lmoe_rmsnorm_bwd_kept, x.data_ptr(), w.data_ptr(), lmoe_type(w), rstd.data_ptr<float>(), g.data_ptr(), lmoe_type(g),
           r.defined() ? r.data_ptr() : nullptr, lmoe_type(dx), T, static_cast<int>(D), dx.data_ptr(), dw.data_ptr(), lmoe_type(dw),
           ws.data_ptr(), static_cast<size_t>(ws.numel()), at::cuda::getCurrentCUDAStream().stream());
      const Tensor none;
      return {as_param(dx, x_type), as_param(dw, w_type), none, none, none};
    } catch (const LmoeFailure& e) {
      rethrow_as_python(e);
    }
  }
};

// out = a + b in a's dtype; both inputs receive the output's gradient, in their own dtype.
class AddFn : public torch::autograd::Function<AddFn> {
 public:
  static variable_list forward(AutogradContext* ctx, const Tensor& a, const Tensor& b) {
    ctx->saved_data["t"] = dtypes_of({a, b});
    return {add(a, b)};
  }
  static Tensor add(const Tensor& a, const Tensor& b) {
    const bool bf = b.scalar_type() == at::kBFloat16;
    if (!bf || (a.scalar_type() != at::kBFloat16 && a.scalar_type() != at::kFloat)) return a.detach() + b.detach().to(a.scalar_type());
    check_device(b, a.device());
    const Tensor ac = a.detach().contiguous(), bc = b.detach().contiguous();
    if (ac.scalar_type() == at::kFloat && !(aligned(ac) && aligned(bc))) return ac + bc;
    Tensor out = at::empty_like(ac);
    void* st = at::cuda::getCurrentCUDAStream().stream();
    if (ac.scalar_type() == at::kFloat)
      LMOE(lmoe_add_f32_bf16, ac.data_ptr<float>(), bc.data_ptr(), out.data_ptr<float>(), out.numel(), st);
    else
      LMOE(lmoe_add_bf16, ac.data_ptr(), bc.data_ptr(), out.data_ptr(), out.numel(), st);
    return out;
  }
  static variable_list backward(AutogradContext* ctx, variable_list grads) {
    const auto t = ctx->saved_data["t"].toIntVector();
    auto cast = [&](int k) {
      const auto d = static_cast<at::ScalarType>(t[k]);
      if (!grads[0].defined() || grads[0].scalar_type() == d) return grads[0];
      if (d != at::kBFloat16 || grads[0].scalar_type() != at::kFloat || !aligned(grads[0])) return grads[0].to(d);
      const c10::cuda::CUDAGuard guard(grads[0].device());
      Caster narrow(grads[0]);
      Tensor g = narrow(grads[0]);
      narrow.run(at::cuda::getCurrentCUDAStream().stream());
      return g;
    };
    return {cast(0), cast(1)};
  }
};

// Whether the call needs an autograd node.  A forward-mode tangent counts whatever the grad mode is: the node refuses it
// (no jvp), the direct path would drop it without a word.
bool any_grad(std::initializer_list<const Tensor*> ts) {
  const bool grad = at::GradMode::is_enabled();
  for (const Tensor* t : ts)
    if ((grad && t->requires_grad()) || t->_fw_grad(/*level=*/0).defined()) return true;
  return false;
}

// ---------------------------------------------------------------- Python entry points
std::vector<Tensor> latent_moe(const Tensor& x, const Tensor& wg, const Tensor& wdn, const Tensor& wup, const Tensor& wgus,
                               const Tensor& wds, const Tensor& wgu, const Tensor& wde, const Tensor& bias, int64_t top_k,
                               double z_coef, bool fp8, bool evaluation) {
  require_cuda(x, "LatentMoE");
  poll_status();
  const c10::cuda::CUDAGuard guard(x.device());
  if (any_grad({&x, &wg, &wdn, &wup, &wgus, &wds, &wgu, &wde}))
    return LatentFn::apply(x, wg, wdn, wup, wgus, wds, wgu, wde, bias, top_k, z_coef, fp8);
  const LatentOps o = latent_ops(x, wg, wdn, wup, wgus, wds, wgu, wde);
  const Sizes d = latent_sizes(o.x, o.wgu, o.wds, top_k);
  if (evaluation && !fp8 && d.T <= LMOE_FEW_TOKENS && lmoe_few_applies(&d.s)) {  // (its experts are bf16)
    auto yz = few_forward(d, o.x, o.wg, &o.wdn, &o.wup, o.wgus, o.wds, o.wgu, o.wde, f32_bias(bias, x), static_cast<float>(z_coef));
    return {as_param(yz[0].view(x.sizes()), x.scalar_type()), yz[1]};
  }
  LatentOut r = latent_forward(d, o, f32_bias(bias, x), static_cast<float>(z_coef), fp8,
                               false, c10::nullopt, nullptr);
  return {as_param(r.y.view(x.sizes()), x.scalar_type()), r.z_loss, r.sel, r.counts};
}

std::vector<Tensor> moe(const Tensor& x, const Tensor& wg, const Tensor& wgus, const Tensor& wds, const Tensor& wgu,
                        const Tensor& wde, const Tensor& bias, int64_t top_k, double z_coef,
                        const c10::optional<Tensor>& forced_sel, bool evaluation) {
  require_cuda(x, "MoE");
  poll_status();
  const c10::cuda::CUDAGuard guard(x.device());
  if (any_grad({&x, &wg, &wgus, &wds, &wgu, &wde})) return MoeFn::apply(x, wg, wgus, wds, wgu, wde, bias, top_k, z_coef, forced_sel);
  Caster cast(x);
  const MoeOps o{cast(x).view({-1, x.size(-1)}), cast(wg), cast(wgus), cast(wds), cast(wgu), cast(wde)};
  cast.run(at::cuda::getCurrentCUDAStream().stream());
  const Sizes d = moe_sizes(o.x, o.wgu, o.wds, top_k);
  if (evaluation && !forced_sel && d.T <= LMOE_FEW_TOKENS && lmoe_few_applies(&d.s)) {
    auto yz = few_forward(d, o.x, o.wg, nullptr, nullptr, o.wgus, o.wds, o.wgu, o.wde, f32_bias(bias, x), static_cast<float>(z_coef));
    return {as_param(yz[0].view(x.sizes()), x.scalar_type()), yz[1]};
  }
  LatentOut r = moe_forward(d, o, f32_bias(bias, x), static_cast<float>(z_coef), false, forced_sel);
  return {as_param(r.y.view(x.sizes()), x.scalar_type()), r.z_loss, r.sel, r.counts};
}

std::vector<Tensor> norm_and_pass(const Tensor& x, const Tensor& weight, double eps, bool bf16_out) {
  require_cuda(x, "fused norm");
  check_device(weight, x.device());
  const c10::cuda::CUDAGuard guard(x.device());
  return NormFn::apply(x, weight, eps, bf16_out, any_grad({&x, &weight}));
}
Tensor residual_add(const Tensor& a, const Tensor& b_in) {
  const c10::cuda::CUDAGuard guard(a.device());
  // a feed-forward module may return its rows flattened; one whose result only broadcasts is added by PyTorch
  const Tensor b = b_in.sizes() != a.sizes() && b_in.numel() == a.numel() ? b_in.reshape(a.sizes()) : b_in;
  if (b.sizes() != a.sizes()) return a + b.to(a.scalar_type());
  return any_grad({&a, &b}) ? AddFn::apply(a, b)[0] : AddFn::add(a, b);
}

py::dict dict_of(const Views& v) {
  py::dict d;
  for (const auto& kv : v) d[py::str(kv.first)] = kv.second;
  return d;
}

// The two directions without an autograd node, for the compiled operators and the parity tests' hooks.
py::tuple latent_fwd_raw(const Tensor& x, const Tensor& wg, const Tensor& wdn, const Tensor& wup, const Tensor& wgus,
                         const Tensor& wds, const Tensor& wgu, const Tensor& wde, const Tensor& bias, int64_t top_k, double z_coef,
                         bool fp8, const c10::optional<Tensor>& forced_sel, bool capture) {
  require_cuda(x, "LatentMoE");
  poll_status();
  const c10::cuda::CUDAGuard guard(x.device());
  const LatentOps o = latent_ops(x, wg, wdn, wup, wgus, wds, wgu, wde);
  Views views;
  LatentOut r = latent_forward(latent_sizes(o.x, o.wgu, o.wds, top_k), o, f32_bias(bias, x), static_cast<float>(z_coef), fp8,
                               true, forced_sel, capture ? &views : nullptr);
  const Tensor y = as_param(r.y.view(x.sizes()), x.scalar_type());
  py::gil_scoped_acquire gil;
  return py::make_tuple(y, r.z_loss, r.sel, r.counts, r.saved, dict_of(views));
}

py::tuple latent_bwd_raw(const c10::optional<Tensor>& dy, const c10::optional<Tensor>& d_z, const Tensor& x, const Tensor& wg,
                         const Tensor& wdn, const Tensor& wup, const Tensor& wgus, const Tensor& wds, const Tensor& wgu,
                         const Tensor& wde, const Tensor& sel, const Tensor& saved, int64_t top_k, double z_coef, bool fp8,
                         bool capture) {
  const c10::cuda::CUDAGuard guard(x.device());
  const LatentOps o = latent_ops(x, wg, wdn, wup, wgus, wds, wgu, wde);
  Tensor keep;
  const float* dz = d_z ? scalar_grad(*d_z, keep) : nullptr;
  const auto lin = lin_dtype_of({wg.scalar_type(), wdn.scalar_type(), wup.scalar_type(), wgus.scalar_type(), wds.scalar_type()});
  Views views;
  LatentGrads g = latent_backward(latent_sizes(o.x, o.wgu, o.wds, top_k), o, grad_rows(dy ? *dy : Tensor(), o.x), dz, sel, saved,
                                  static_cast<float>(z_coef), fp8, lin, capture ? &views : nullptr);
  std::vector<Tensor> out{as_param(g.dx.view(x.sizes()), x.scalar_type()), as_param(g.wg, wg.scalar_type()),
                          as_param(g.wdn, wdn.scalar_type()), as_param(g.wup, wup.scalar_type()),
                          as_param(g.wgus, wgus.scalar_type()), as_param(g.wds, wds.scalar_type()),
                          as_param(g.wgu, wgu.scalar_type()), as_param(g.wde, wde.scalar_type())};
  py::gil_scoped_acquire gil;
  return py::make_tuple(out, dict_of(views));
}

// bias -= gamma * sign(load - mean load), the load history's running mean and the update counter, in one launch.
void bias_update(const Tensor& counts, double gamma, Tensor& bias, Tensor& history, Tensor& update_count) {
  poll_status();
  const c10::cuda::CUDAGuard guard(counts.device());
  LMOE(lmoe_router_bias_update_counted, static_cast<int>(counts.numel()), counts.data_ptr<int32_t>(), static_cast<float>(gamma),
       bias.data_ptr<float>(), history.data_ptr<float>(), update_count.data_ptr<int64_t>(),
       at::cuda::getCurrentCUDAStream().stream());
}

}  // namespace

PYBIND11_MODULE(TORCH_EXTENSION_NAME, m) {
  py::register_exception_translator([](std::exception_ptr p) {
    try {
      if (p) std::rethrow_exception(p);
    } catch (const LmoeFailure& e) {
      PyErr_SetString(g_error_class ? g_error_class : PyExc_RuntimeError, e.what());
    }
  });
  // Whatever launches does so without the interpreter lock, as PyTorch's own operators do: a launch blocks while the device's
  // queue is full, and what empties it may be another thread's to launch.
  using NoGil = py::call_guard<py::gil_scoped_release>;
  m.def("set_error_class", [](py::object cls) { g_error_class = cls.inc_ref().ptr(); });
  m.def("poll_status", &poll_status);
  m.def("devices_used", &devices_used);
  m.def("latent_moe", &latent_moe, NoGil());
  m.def("moe", &moe, NoGil());
  m.def("latent_fwd_raw", &latent_fwd_raw, NoGil());
  m.def("latent_bwd_raw", &latent_bwd_raw, NoGil());
  m.def("latent_saved_bytes", [](int64_t T, int64_t D, int64_t L, int64_t E, int64_t K, int64_t F, int64_t Fs) {
    return LatentLayout(Sizes(T, D, L, E, K, F, Fs), false, false).bytes;
  });
  m.def("bias_update", &bias_update, NoGil());
  m.def("norm_and_pass", &norm_and_pass, NoGil());
  m.def("residual_add", &residual_add, NoGil());
}

// Host side of the layer operators in C++ (CPython extension `_host`): argument checks, buffers from torch's caching
// allocator, the calls of the C ABI, and device-side errors through a mailbox in mapped memory.  The operator functions
// of fastlstm/lstm.py:31-146, :236-334 and :494-501 as they are seen from Python live in lstm.py; what they cost per
// call in Python (ctypes, tensor checks, allocations, a status copy with its event: 130 us a layer) is what this file is
// for.
#include <ATen/cuda/CUDAContext.h>
#include <c10/cuda/CUDAGuard.h>
#include <cuda_runtime_api.h>
#include <torch/extension.h>

#include <array>
#include <atomic>
#include <mutex>
#include <optional>
#include <string>
#include <vector>

#include "../../include/fastlstm_b200.h"

namespace {

using at::Tensor;
using OptTensor = std::optional<Tensor>;

struct DeviceError {
  int code;
  std::string where;
};

int g_flags = 0;              // BLSTM_FLAG_FORCE_GENERIC or 0
int g_wait_limit_us = 0;
bool g_sync_check = false;
PyObject* g_error_class = nullptr;

// One mailbox per device, kept for the life of the process.  [1] code, [2..3] detail.
constexpr int kMaxDevices = 64;
std::array<std::atomic<int32_t*>, kMaxDevices> g_mail{};
std::mutex g_mail_mutex;

void cuda_ok(cudaError_t e, const char* what) {
  TORCH_CHECK(e == cudaSuccess, what, ": ", cudaGetErrorString(e));
}

int32_t* mailbox(int dev) {
  TORCH_CHECK(dev >= 0 && dev < kMaxDevices, "device index out of range");
  int32_t* m = g_mail[dev].load(std::memory_order_acquire);
  if (m) return m;
  std::lock_guard<std::mutex> lock(g_mail_mutex);
  m = g_mail[dev].load(std::memory_order_acquire);
  if (!m) {
    void* p = nullptr;
    cuda_ok(cudaHostAlloc(&p, 64, cudaHostAllocMapped | cudaHostAllocPortable), "cudaHostAlloc");
    m = static_cast<int32_t*>(p);
    for (int i = 0; i < 16; ++i) m[i] = 0;
    g_mail[dev].store(m, std::memory_order_release);
  }
  return m;
}

// Throws when a finished launch of this device has left an error.
void poll(int dev) {
  volatile int32_t* m = mailbox(dev);
  if (__builtin_expect(m[1] == 0, 1)) return;
  const int code = m[1], d0 = m[2], d1 = m[3];
  m[1] = 0;
  throw DeviceError{code, "recurrence (step " + std::to_string(d0) + ", batch tile " + std::to_string(d1) + ")"};
}

void check(int rc, const char* where) {
  if (rc != BLSTM_OK) throw DeviceError{rc, where};
}

int dtype_code(at::ScalarType t) {
  if (t == at::kFloat) return BLSTM_F32;
  if (t == at::kHalf) return BLSTM_F16;
  if (t == at::kBFloat16) return BLSTM_BF16;
  throw py::value_error(std::string("unsupported dtype ") + c10::toString(t) + "; expected float32, float16 or bfloat16");
}

std::string shape_str(at::IntArrayRef s) {
  std::string r = "(";
  for (size_t i = 0; i < s.size(); ++i) r += (i ? ", " : "") + std::to_string(s[i]);
  return r + ")";
}

void require(const Tensor& t, const char* name) {
  if (!t.is_cuda()) throw py::value_error(std::string(name) + " must be a CUDA tensor (there is no CPU path)");
  if (!t.is_contiguous()) throw py::value_error(std::string(name) + " must be contiguous");
}
void require(const Tensor& t, const char* name, at::ScalarType dt, const at::Device& dev, at::IntArrayRef shape) {
  require(t, name);
  if (t.scalar_type() != dt)
    throw py::value_error(std::string(name) + " has dtype " + c10::toString(t.scalar_type()) + ", expected " + c10::toString(dt));
  if (t.device() != dev) throw py::value_error(std::string(name) + " is on " + t.device().str() + ", expected " + dev.str());
  if (t.sizes() != shape) throw py::value_error(std::string(name) + " has shape " + shape_str(t.sizes()) + ", expected " + shape_str(shape));
}
void require(const OptTensor& t, const char* name, at::ScalarType dt, const at::Device& dev, at::IntArrayRef shape) {
  if (t) require(*t, name, dt, dev, shape);
}

const void* ptr(const Tensor& t) { return t.const_data_ptr(); }
const void* ptr(const OptTensor& t) { return t ? t->const_data_ptr() : nullptr; }

blstm_desc desc(at::ScalarType dt, int64_t T, int64_t B, int64_t I, int64_t H, int flags) {
  blstm_desc d{};
  d.dtype = dtype_code(dt);
  d.seq_len = (int32_t)T; d.batch = (int32_t)B; d.input_size = (int32_t)I; d.hidden_size = (int32_t)H;
  d.flags = flags | g_flags;
  d.wait_limit_us = g_wait_limit_us;
  return d;
}

// What every call does around its launches.
struct Call {
  c10::cuda::CUDAGuard guard;
  int dev;
  void* stream;
  explicit Call(const at::Device& d) : guard(d), dev(d.index()), stream(at::cuda::getCurrentCUDAStream(d.index()).stream()) {
    poll(dev);
    blstm_set_mailbox(mailbox(dev));
  }
  ~Call() { blstm_set_mailbox(nullptr); }
  void done(const Tensor& ws, const char* where) {
    if (g_sync_check && ws.defined()) check(blstm_read_status(ws.const_data_ptr(), nullptr, stream), where);
  }
};

struct FwdOut {
  Tensor out, cell, ifgo;
};

// Two tensors of one shape in one allocation, each on a 16-byte boundary (which the kernels ask of 16-bit tensors).
std::array<Tensor, 2> empty_pair(at::IntArrayRef shape, const at::TensorOptions& opt) {
  const int64_t n = c10::multiply_integers(shape), step = (n + 7) / 8 * 8;
  const Tensor both = at::empty({2 * step}, opt);
  return {both.narrow(0, 0, n).view(shape), both.narrow(0, step, n).view(shape)};
}

// t contiguous and on a 16-byte boundary
Tensor fit(const Tensor& t) {
  const Tensor c = t.contiguous();
  return reinterpret_cast<uintptr_t>(c.const_data_ptr()) & 15 ? c.clone() : c;
}

FwdOut fwd_impl(const Tensor& x, const OptTensor& h0, const OptTensor& c0, const Tensor& Wx, const OptTensor& bx, const Tensor& Wh,
                const OptTensor& bh, bool inference, bool half_device) {
  require(x, "x");
  if (x.dim() != 3) throw py::value_error("expected x as [T,B,I]");
  const int64_t T = x.size(0), B = x.size(1), I = x.size(2), H = Wh.size(-1);
  const auto dt = x.scalar_type();
  const at::Device dev = x.device();
  const blstm_desc d = desc(dt, T, B, I, H, (inference ? BLSTM_FLAG_INFERENCE : 0) | (half_device ? BLSTM_FLAG_HALF_DEVICE : 0));
  require(Wx, "Wx", dt, dev, {4 * H, I});
  require(Wh, "Wh", dt, dev, {4 * H, H});
  require(bx, "bx", dt, dev, {4 * H});
  require(bh, "bh", dt, dev, {4 * H});
  if (h0.has_value() != c0.has_value()) throw py::value_error("h0 and c0 must both be given or both be None");
  require(h0, "h0", dt, dev, {B, H});
  require(c0, "c0", dt, dev, {B, H});
  Call call(dev);
  const auto opt = x.options().requires_grad(false);
  FwdOut r;
  auto [out, cell] = empty_pair({T + 1, B, H}, opt);
  r.out = out;
  r.cell = cell;
  const bool lone = inference && T == 1 && blstm_plan_family(&d, BLSTM_PHASE_FWD_OP) == BLSTM_FAMILY_STEP;
  Tensor ws;
  size_t ws_bytes = 0;
  if (!lone) {
    r.ifgo = at::empty({T, B, 4 * H}, opt);
    ws_bytes = blstm_workspace_bytes(&d, BLSTM_PHASE_FWD);
    ws = at::empty({(int64_t)ws_bytes}, opt.dtype(at::kByte));
  }
  check(blstm_fwd(&d, ptr(x), ptr(h0), ptr(c0), ptr(Wx), ptr(Wh), ptr(bx), ptr(bh), r.out.data_ptr(), r.cell.data_ptr(),
                  lone ? nullptr : r.ifgo.data_ptr(), lone ? nullptr : ws.data_ptr(), ws_bytes, call.stream),
        "blstm_fwd");
  call.done(ws, "forward recurrence");
  return r;
}

py::tuple fwd(const Tensor& x, const OptTensor& h0, const OptTensor& c0, const Tensor& Wx, const OptTensor& bx, const Tensor& Wh,
              const OptTensor& bh, bool inference, bool half_device) {
  FwdOut r;
  {
    py::gil_scoped_release nogil;
    r = fwd_impl(x, h0, c0, Wx, bx, Wh, bh, inference, half_device);
    if (!r.ifgo.defined()) r.ifgo = at::empty({x.size(0), x.size(1), 4 * r.out.size(2)}, r.out.options());
  }
  return py::make_tuple(r.out, r.cell, r.ifgo);
}

struct BwdOut {
  Tensor d_x, dh_0, dc_0, wgrads;
};

BwdOut bwd_impl(const Tensor& dh, const OptTensor& dc_n, const OptTensor& dh_n, const Tensor& x, const Tensor& h, const Tensor& cell,
                const Tensor& ifgo, const Tensor& Wx, const Tensor& Wh, bool need_dx, const OptTensor& wgrads_in, bool half_device) {
  const int64_t T = dh.size(0), B = dh.size(1), H = dh.size(2), I = x.size(-1);
  const auto dt = x.scalar_type();
  const at::Device dev = x.device();
  require(dh, "dh", dt, dev, {T, B, H});
  require(dh_n, "dh_n", dt, dev, {B, H});
  require(dc_n, "dc_n", dt, dev, {B, H});
  require(h, "h", dt, dev, {T + 1, B, H});
  require(cell, "cell", dt, dev, {T + 1, B, H});
  require(ifgo, "ifgo", dt, dev, {T, B, 4 * H});
  const blstm_desc d = desc(dt, T, B, I, H, half_device ? BLSTM_FLAG_HALF_DEVICE : 0);
  Call call(dev);
  const auto opt = x.options().requires_grad(false);
  const Tensor d_ifgo = at::empty({T, B, 4 * H}, opt);
  BwdOut r;
  if (need_dx) r.d_x = at::empty({T, B, I}, opt);
  auto [dh_0, dc_0] = empty_pair({B, H}, opt);
  r.dh_0 = dh_0;
  r.dc_0 = dc_0;
  const int64_t n = 4 * H * (I + H + 1);
  r.wgrads = wgrads_in ? *wgrads_in : at::empty({n}, opt.dtype(at::kFloat));
  require(r.wgrads, "wgrads", at::kFloat, dev, {n});
  float* w = static_cast<float*>(r.wgrads.data_ptr());
  const size_t ws_bytes = blstm_workspace_bytes(&d, BLSTM_PHASE_BWD);
  const Tensor ws = at::empty({(int64_t)ws_bytes}, opt.dtype(at::kByte));
  check(blstm_bwd(&d, ptr(dh), ptr(dh_n), ptr(dc_n), ptr(x), ptr(h), ptr(cell), ptr(ifgo), ptr(Wx), ptr(Wh), d_ifgo.data_ptr(),
                  need_dx ? r.d_x.data_ptr() : nullptr, r.dh_0.data_ptr(), r.dc_0.data_ptr(), w, w + 4 * H * I, w + 4 * H * (I + H),
                  ws.data_ptr(), ws_bytes, call.stream),
        "blstm_bwd");
  call.done(ws, "backward recurrence");
  return r;
}

py::tuple bwd(const Tensor& dh, const OptTensor& dc_n, const OptTensor& dh_n, const Tensor& x, const Tensor& h, const Tensor& cell,
              const Tensor& ifgo, const Tensor& Wx, const Tensor& Wh, bool need_dx, const OptTensor& wgrads, bool half_device) {
  BwdOut r;
  {
    py::gil_scoped_release nogil;
    r = bwd_impl(dh, dc_n, dh_n, x, h, cell, ifgo, Wx, Wh, need_dx, wgrads, half_device);
  }
  const int64_t H = dh.size(2), I = x.size(-1);
  const Tensor dWx = r.wgrads.narrow(0, 0, 4 * H * I).view({4 * H, I}), dWh = r.wgrads.narrow(0, 4 * H * I, 4 * H * H).view({4 * H, H});
  const Tensor db = r.wgrads.narrow(0, 4 * H * (I + H), 4 * H);
  return py::make_tuple(need_dx ? py::cast(r.d_x) : py::none(), r.dh_0, r.dc_0, dWx, db, dWh, db);
}

// Collects tensors of a layer that need another type or size and moves them in one launch.
struct Repack {
  std::vector<blstm_repack_item> items;
  std::vector<Tensor> keep;
  // t as [groups, rows, cols] -> the same groups of [rows_to, cols_to] of type `to`
  Tensor add(const Tensor& t, at::ScalarType to, int64_t groups, int64_t rows, int64_t cols, int64_t rows_to, int64_t cols_to, at::IntArrayRef shape) {
    const Tensor src = t.contiguous();
    const Tensor dst = at::empty(shape, src.options().requires_grad(false).dtype(to));
    if (src.numel() == 0) return dst;
    keep.push_back(src);
    items.push_back({src.const_data_ptr(), dst.data_ptr(), dtype_code(src.scalar_type()), dtype_code(to), groups, (int32_t)rows, (int32_t)cols,
                     (int32_t)rows_to, (int32_t)cols_to});
    return dst;
  }
  void run(const at::Device& dev) {
    if (items.empty()) return;
    c10::cuda::CUDAGuard guard(dev);
    check(blstm_repack(items.data(), (int)items.size(), at::cuda::getCurrentCUDAStream(dev.index()).stream()), "blstm_repack");
    items.clear();
    keep.clear();
  }
};

// A layer's inputs contiguous, in type `to` (or their own) and zero-padded to input size Ip and hidden size Hp (0: as they are).
py::tuple prepare(const Tensor& x, const OptTensor& h0, const OptTensor& c0, const Tensor& Wx, const OptTensor& bx, const Tensor& Wh,
                  const OptTensor& bh, std::optional<at::ScalarType> to, int64_t Ip, int64_t Hp) {
  std::array<OptTensor, 7> r{x, h0, c0, Wx, bx, Wh, bh};
  {
    py::gil_scoped_release nogil;
    at::NoGradGuard no_grad;
    if (!x.is_cuda()) throw py::value_error("x must be a CUDA tensor (there is no CPU path)");
    const int64_t I = x.size(-1), H = Wh.size(-1);
    if (!Ip) { Ip = I; Hp = H; }
    Repack m;
    auto move = [&](OptTensor& t, int64_t groups, int64_t rows, int64_t cols, int64_t rows_to, int64_t cols_to, std::vector<int64_t> shape) {
      if (!t) return;
      const auto ty = to.value_or(t->scalar_type());
      if (ty == t->scalar_type() && rows == rows_to && cols == cols_to) t = fit(*t);
      else t = m.add(*t, ty, groups, rows, cols, rows_to, cols_to, shape);
    };
    auto last = [&](const OptTensor& t, int64_t n) { std::vector<int64_t> s = t ? t->sizes().vec() : std::vector<int64_t>(); if (t) s.back() = n; return s; };
    move(r[0], 1, x.numel() / I, I, x.numel() / I, Ip, last(r[0], Ip));
    for (int k = 1; k < 3; ++k) move(r[k], 1, r[k] ? r[k]->numel() / H : 0, H, r[k] ? r[k]->numel() / H : 0, Hp, last(r[k], Hp));
    move(r[3], 4, H, I, Hp, Ip, {4 * Hp, Ip});
    move(r[4], 4, 1, H, 1, Hp, {4 * Hp});
    move(r[5], 4, H, H, Hp, Hp, {4 * Hp, Hp});
    move(r[6], 4, 1, H, 1, Hp, {4 * Hp});
    m.run(x.device());
  }
  py::tuple out(7);
  for (int k = 0; k < 7; ++k) out[k] = r[k] ? py::cast(*r[k]) : py::none();
  return out;
}

// ---------------------------------------------------------------- autograd node of one layer
// (PersistentLSTMfn of fastlstm/lstm.py:504-538.)  The forward has already run: the node hands out its results and keeps
// what backward reads, in the padded sizes and the compute type it ran in.
struct LayerState {
  Tensor x, Wx, Wh, out, cell, ifgo;
  int64_t I, H;                // the layer's own sizes
  bool stacked;                // final states as [1,B,H]
  std::optional<std::array<int64_t, 3>> main;   // planned for half of the device, another layer beside it: the stream (id, device
};                                              // index and type) that the gradients are used on, whichever one backward runs on

struct LayerFn : public torch::autograd::Function<LayerFn> {
  static torch::autograd::variable_list forward(torch::autograd::AutogradContext* ctx, const Tensor& x, const OptTensor& h0, const OptTensor& c0,
                                                const Tensor& Wx, const OptTensor& bx, const Tensor& Wh, const OptTensor& bh, LayerState s) {
    const int64_t T = s.out.size(0) - 1;
    ctx->saved_data["sizes"] = std::vector<int64_t>{s.I, s.H};
    ctx->saved_data["given"] = std::vector<int64_t>{h0.has_value(), bx.has_value(), bh.has_value(), x.requires_grad(), s.stacked, s.main.has_value(), (int64_t)x.scalar_type()};
    if (s.main) ctx->saved_data["main"] = std::vector<int64_t>(s.main->begin(), s.main->end());
    Tensor y = s.out.narrow(0, 1, T), hn = s.out.select(0, T), cn = s.cell.select(0, T);
    if (s.out.size(2) != s.H) { y = y.narrow(2, 0, s.H); hn = hn.narrow(1, 0, s.H); cn = cn.narrow(1, 0, s.H); }
    if (s.stacked) {             // tensors of their own, in one copy
      const Tensor both = at::stack({hn, cn}).unsqueeze_(1);
      hn = both.select(0, 0);
      cn = both.select(0, 1);
    }
    ctx->save_for_backward({s.x, s.out, s.cell, s.ifgo, s.Wx, s.Wh});
    return {y, hn, cn};
  }

  static torch::autograd::variable_list backward(torch::autograd::AutogradContext* ctx, torch::autograd::variable_list g) {
    const auto saved = ctx->get_saved_variables();
    const Tensor &x = saved[0], &out = saved[1], &cell = saved[2], &ifgo = saved[3], &Wx = saved[4], &Wh = saved[5];
    const auto sizes = ctx->saved_data["sizes"].toIntVector(), given = ctx->saved_data["given"].toIntVector();
    const int64_t I = sizes[0], H = sizes[1], T = out.size(0) - 1, B = out.size(1), Hp = out.size(2), Ip = x.size(2);
    const auto dt = x.scalar_type();
    const bool pad = Hp != H || Ip != I;
    Repack m;
    auto state_grad = [&](const Tensor& t) -> OptTensor {
      if (!t.defined()) return std::nullopt;
      Tensor v = given[4] ? t.squeeze(0) : t;
      if (Hp != H || v.scalar_type() != dt) return m.add(v, dt, 1, B, H, B, Hp, {B, Hp});
      return v.contiguous();
    };
    Tensor dy;
    if (!g[0].defined()) dy = at::zeros({T, B, Hp}, x.options());
    else if (Hp != H || g[0].scalar_type() != dt) dy = m.add(g[0], dt, 1, T * B, H, T * B, Hp, {T, B, Hp});
    else dy = g[0].contiguous();
    const OptTensor dhn = state_grad(g[1]), dcn = state_grad(g[2]);
    m.run(x.device());
    BwdOut r = bwd_impl(dy, dcn, dhn, x, out, cell, ifgo, Wx, Wh, given[3] != 0, std::nullopt, given[5] != 0);
    Tensor dWx = r.wgrads.narrow(0, 0, 4 * Hp * Ip).view({4 * Hp, Ip}), dWh = r.wgrads.narrow(0, 4 * Hp * Ip, 4 * Hp * Hp).view({4 * Hp, Hp});
    Tensor db = r.wgrads.narrow(0, 4 * Hp * (Ip + Hp), 4 * Hp), dh0 = r.dh_0, dc0 = r.dc_0, dx = r.d_x;
    // (the type x came in, here: autograd's own conversion took 2.7 times as long, 142 us at 256 x 256 x 768)
    const auto x_type = (at::ScalarType)given[6];
    if (dx.defined() && x_type != dt) dx = m.add(dx, x_type, 1, T * B, Ip, T * B, I, {T, B, I});
    else if (dx.defined() && pad) dx = dx.narrow(2, 0, I);
    if (pad) {
      dWx = m.add(dWx, at::kFloat, 4, Hp, Ip, H, I, {4 * H, I});
      dWh = m.add(dWh, at::kFloat, 4, Hp, Hp, H, H, {4 * H, H});
      db = m.add(db, at::kFloat, 4, 1, Hp, 1, H, {4 * H});
      dh0 = dh0.narrow(1, 0, H);
      dc0 = dc0.narrow(1, 0, H);
    }
    m.run(x.device());
    if (given[5]) {
      const auto on = ctx->saved_data["main"].toIntVector();
      const auto main = c10::Stream::unpack3(on[0], (c10::DeviceIndex)on[1], (c10::DeviceType)on[2]);
      for (Tensor* t : {&dx, &dh0, &dc0, &dWx, &dWh, &db})
        if (t->defined()) t->record_stream(main);
    }
    const Tensor none;
    return {dx, given[0] ? dh0 : none, given[0] ? dc0 : none, dWx, given[1] ? db : none, dWh, given[2] ? db : none, none};
  }
};

py::tuple attach(const Tensor& x, const OptTensor& h0, const OptTensor& c0, const Tensor& Wx, const OptTensor& bx, const Tensor& Wh,
                 const OptTensor& bh, const Tensor& xp, const Tensor& Wxp, const Tensor& Whp, const Tensor& out, const Tensor& cell,
                 const Tensor& ifgo, bool stacked, std::optional<std::array<int64_t, 3>> main) {
  const auto r = LayerFn::apply(x, h0, c0, Wx, bx, Wh, bh, LayerState{xp, Wxp, Whp, out, cell, ifgo, x.size(-1), Wh.size(-1), stacked, main});
  return py::make_tuple(r[0], r[1], r[2]);
}

py::tuple wgrad(const Tensor& d_ifgo, const Tensor& x, const Tensor& h) {
  Tensor db, dWx, dWh;
  {
    py::gil_scoped_release nogil;
    const int64_t T = d_ifgo.size(0), B = d_ifgo.size(1), G = d_ifgo.size(2), H = G / 4, I = x.size(-1);
    const blstm_desc d = desc(x.scalar_type(), T, B, I, H, 0);
    Call call(x.device());
    const auto f32 = x.options().requires_grad(false).dtype(at::kFloat);
    dWx = at::empty({G, I}, f32);
    dWh = at::empty({G, H}, f32);
    db = at::empty({G}, f32);
    const size_t ws_bytes = blstm_workspace_bytes(&d, BLSTM_PHASE_BWD);
    const Tensor ws = at::empty({(int64_t)ws_bytes}, f32.dtype(at::kByte));
    check(blstm_wgrad(&d, ptr(d_ifgo), ptr(x), ptr(h), (float*)dWx.data_ptr(), (float*)dWh.data_ptr(), ws.data_ptr(), ws_bytes, call.stream), "blstm_wgrad");
    check(blstm_bias_grad(&d, ptr(d_ifgo), (float*)db.data_ptr(), ws.data_ptr(), ws_bytes, call.stream), "blstm_bias_grad");
  }
  return py::make_tuple(db, db, dWx, dWh);
}

// A unidirectional stack without gradients (the layer loop of fastlstm/lstm.py:685-696): params = (Wx, bx, Wh, bh) per
// layer, h0 / c0 [L,B,H] or both None.  Returns (out, h_n, c_n).
py::tuple infer(const Tensor& x_in, const OptTensor& h0, const OptTensor& c0, const std::vector<OptTensor>& params, bool batch_first) {
  Tensor out, hn, cn;
  {
    py::gil_scoped_release nogil;
    at::NoGradGuard no_grad;
    const int64_t L = (int64_t)params.size() / 4;
    Tensor x = batch_first ? x_in.transpose(0, 1) : x_in;
    x = fit(x);
    std::vector<Tensor> h(L), c(L);
    for (int64_t l = 0; l < L; ++l) {
      OptTensor hl, cl;
      if (h0) hl = fit(h0->select(0, l));
      if (c0) cl = fit(c0->select(0, l));
      FwdOut r = fwd_impl(x, hl, cl, params[4 * l]->contiguous(), params[4 * l + 1], params[4 * l + 2]->contiguous(), params[4 * l + 3], true, false);
      const int64_t T = x.size(0);
      x = fit(r.out.narrow(0, 1, T));
      h[l] = r.out.select(0, T);
      c[l] = r.cell.select(0, T);
    }
    out = batch_first ? x.transpose(0, 1) : x;
    hn = at::stack(h);
    cn = at::stack(c);
  }
  return py::make_tuple(out, hn, cn);
}

// ---------------------------------------------------------------- packed sequences
Tensor gather_rows_impl(const Tensor& src_in, const Tensor& idx, at::IntArrayRef lead) {
  const Tensor src = src_in.contiguous();
  const int64_t C = src.size(-1);
  std::vector<int64_t> shape = lead.vec();
  shape.push_back(C);
  const Tensor dst = at::empty(shape, src.options().requires_grad(false));
  c10::cuda::CUDAGuard guard(src.device());
  check(blstm_gather_rows(dst.data_ptr(), src.const_data_ptr(), (const int32_t*)idx.const_data_ptr(), idx.numel(), C * src.element_size(),
                          at::cuda::getCurrentCUDAStream(src.device().index()).stream()),
        "blstm_gather_rows");
  return dst;
}

// Rows of src (its last dimension) in another order; `inv` maps every row of src to the row it went to, or -1.
struct GatherRowsFn : public torch::autograd::Function<GatherRowsFn> {
  static Tensor forward(torch::autograd::AutogradContext* ctx, const Tensor& src, const Tensor& idx, const Tensor& inv, std::vector<int64_t> lead) {
    ctx->save_for_backward({inv});
    std::vector<int64_t> s = src.sizes().vec();
    s.pop_back();
    ctx->saved_data["lead"] = s;
    return gather_rows_impl(src, idx, lead);
  }
  static torch::autograd::variable_list backward(torch::autograd::AutogradContext* ctx, torch::autograd::variable_list g) {
    const auto saved = ctx->get_saved_variables();
    return {gather_rows_impl(g[0], saved[0], ctx->saved_data["lead"].toIntVector()), Tensor(), Tensor(), Tensor()};
  }
};

Tensor gather_rows(const Tensor& src, const Tensor& idx, const Tensor& inv, std::vector<int64_t> lead) {
  py::gil_scoped_release nogil;
  return GatherRowsFn::apply(src, idx, inv, lead);
}

// The maps of blstm_packed_maps as tensors: (padded, turned, rev, inv_last, last, packed, packed_turned).
std::vector<Tensor> packed_maps(const Tensor& batch_sizes, const OptTensor& rank, const Tensor& data) {
  py::gil_scoped_release nogil;
  const int64_t T = batch_sizes.numel();
  const Tensor bs = batch_sizes.contiguous();
  const int64_t* b = static_cast<const int64_t*>(bs.const_data_ptr());
  const int64_t B = b[0];
  const Tensor host = at::empty({2 * T}, at::TensorOptions().dtype(at::kInt).pinned_memory(true));
  int32_t* h = static_cast<int32_t*>(host.data_ptr());
  int64_t n = 0;
  for (int64_t t = 0; t < T; ++t) {
    h[t] = (int32_t)b[t];
    h[T + t] = (int32_t)n;
    n += b[t];
  }
  c10::cuda::CUDAGuard guard(data.device());
  const auto i32 = data.options().requires_grad(false).dtype(at::kInt);
  const Tensor dev = host.to(data.device(), /*non_blocking=*/true);
  const Tensor maps = at::empty({4 * T * B + B + 2 * n}, i32);
  check(blstm_packed_maps((const int32_t*)dev.const_data_ptr(), (const int32_t*)dev.const_data_ptr() + T,
                          rank ? (const int64_t*)rank->const_data_ptr() : nullptr, (int)T, (int)B, (int32_t*)maps.data_ptr(),
                          at::cuda::getCurrentCUDAStream(data.device().index()).stream()),
        "blstm_packed_maps");
  std::vector<Tensor> r;
  for (int k = 0; k < 4; ++k) r.push_back(maps.narrow(0, k * T * B, T * B));
  r.push_back(maps.narrow(0, 4 * T * B, B));
  for (int k = 0; k < 2; ++k) r.push_back(maps.narrow(0, 4 * T * B + B + k * n, n));
  return r;
}

void check_status(bool wait) {
  for (int dev = 0; dev < kMaxDevices; ++dev) {
    if (!g_mail[dev].load(std::memory_order_acquire)) continue;
    if (wait) {
      py::gil_scoped_release nogil;
      c10::cuda::CUDAGuard guard((c10::DeviceIndex)dev);
      cuda_ok(cudaDeviceSynchronize(), "cudaDeviceSynchronize");
    }
    poll(dev);
  }
}

void configure(int flags, int wait_limit_us, bool sync_check, py::object error_class) {
  g_flags = flags;
  g_wait_limit_us = wait_limit_us;
  g_sync_check = sync_check;
  g_error_class = error_class.release().ptr();
}

}  // namespace

PYBIND11_MODULE(_host, m) {
  py::register_exception_translator([](std::exception_ptr p) {
    try {
      if (p) std::rethrow_exception(p);
    } catch (const DeviceError& e) {
      PyErr_SetObject(g_error_class, py::make_tuple(e.code, e.where).ptr());
    }
  });
  m.def("configure", &configure);
  m.def("fwd", &fwd);
  m.def("bwd", &bwd);
  m.def("wgrad", &wgrad);
  m.def("prepare", &prepare);
  m.def("attach", &attach);
  m.def("infer", &infer);
  m.def("gather_rows", &gather_rows);
  m.def("packed_maps", &packed_maps);
  m.def("check_status", &check_status);
}

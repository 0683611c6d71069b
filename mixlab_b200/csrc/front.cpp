// Native half of the torch front end (mixlab_b200/ops.py): checks every operand, allocates the results, keeps the
// per-device workspace and calls the C ABI.  The C ABI sees only pointers, so a wrong operand would otherwise be read
// out of bounds or as the wrong type.
//
// What bounds a small call is this host work: in Python the checks, the ctypes conversions and the allocations of one
// decode step took 17 us beside a kernel of 5 us, those of a short scan 30 us.
#include <ATen/cuda/EmptyTensor.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <cuda_runtime_api.h>
#include <dlfcn.h>
#include <torch/extension.h>

#include <algorithm>
#include <map>
#include <memory>
#include <mutex>
#include <optional>
#include <string>
#include <vector>

#include "../../include/mixlab_b200.h"

namespace py = pybind11;
using at::Tensor;
using Opt = std::optional<Tensor>;
using Shape = at::IntArrayRef;

namespace {

// ------------------------------------------------------------------ the C ABI
#define MXB_FUNCTIONS(X)                                                                                              \
  X(mxb_gdn_fwd_workspace_bytes) X(mxb_gdn_bwd_workspace_bytes) X(mxb_gdn_fwd) X(mxb_gdn_bwd) X(mxb_gdn_decode_step)  \
  X(mxb_gdn_block_workspace_bytes) X(mxb_gdn_block_pre_fwd) X(mxb_gdn_block_pre_bwd) X(mxb_gdn_block_post_fwd)        \
  X(mxb_gdn_block_post_bwd) X(mxb_mamba3_fwd_workspace_bytes) X(mxb_mamba3_bwd_workspace_bytes) X(mxb_mamba3_fwd)     \
  X(mxb_mamba3_bwd) X(mxb_mamba3_block_workspace_bytes) X(mxb_mamba3_block_conv_fwd) X(mxb_mamba3_block_conv_bwd)     \
  X(mxb_mamba3_block_bc_fwd) X(mxb_mamba3_block_bc_bwd) X(mxb_mamba3_block_post_fwd) X(mxb_mamba3_block_post_bwd)     \
  X(mxb_ir_op_workspace_bytes) X(mxb_ir_op_forward)
struct Abi {
#define X(name) decltype(&::name) name = nullptr;
  MXB_FUNCTIONS(X)
#undef X
} abi;

void open_library(const std::string& path) {
  void* h = dlopen(path.c_str(), RTLD_NOW | RTLD_LOCAL);
  if (!h) throw py::import_error(dlerror());
#define X(name)                                                     \
  abi.name = reinterpret_cast<decltype(abi.name)>(dlsym(h, #name)); \
  if (!abi.name) throw py::import_error("missing export " #name);
  MXB_FUNCTIONS(X)
#undef X
}

// ------------------------------------------------------------------ operands
[[noreturn]] void not_cuda() { throw py::value_error("mixlab_b200 operators take CUDA tensors only (no CPU fallback)"); }

int32_t io_code(const Tensor& t) {
  if (t.scalar_type() == at::kFloat) return MXB_F32;
  if (t.scalar_type() == at::kBFloat16) return MXB_BF16;
  throw py::type_error(std::string("unsupported dtype ") + c10::toString(t.scalar_type()) + " (float32 or bfloat16)");
}

std::string text(Shape s) {
  std::string r = "(";
  for (size_t i = 0; i < s.size(); ++i) r += (i ? ", " : "") + std::to_string(s[i]);
  return r + ")";
}

at::Device cuda_device(const Tensor& t) {
  if (!t.is_cuda()) not_cuda();
  return t.device();
}
void check(const Tensor& t, Shape shape, at::ScalarType dtype, at::Device dev, const char* name) {
  if (!t.is_cuda()) not_cuda();
  if (t.sizes() != shape) throw py::value_error(std::string(name) + ": shape " + text(t.sizes()) + ", expected " + text(shape));
  if (t.scalar_type() != dtype)
    throw py::type_error(std::string(name) + ": dtype " + c10::toString(t.scalar_type()) + ", expected " + c10::toString(dtype));
  if (t.device() != dev) throw py::value_error(std::string(name) + ": on " + t.device().str() + ", expected " + dev.str());
  if (!t.is_contiguous()) throw py::value_error(std::string(name) + ": tensor must be contiguous");
}
void check(const Opt& t, Shape shape, at::ScalarType dtype, at::Device dev, const char* name) {
  if (t) check(*t, shape, dtype, dev, name);
}

template <typename T = void>
T* ptr(const Tensor& t) { return static_cast<T*>(t.data_ptr()); }
template <typename T = void>
T* ptr(const Opt& t) { return t ? static_cast<T*>(t->data_ptr()) : nullptr; }

Tensor make(Shape shape, at::ScalarType dtype, at::Device dev) {
  return at::detail::empty_cuda(shape, dtype, dev, std::nullopt);
}
Tensor like(const Tensor& t) { return make(t.sizes(), t.scalar_type(), t.device()); }
constexpr at::ScalarType F = at::kFloat;

// A call on a device: that device is current, its current stream is the one to launch on.  Made when every operand has
// been checked: a refused call does not touch the device.
struct On {
  c10::cuda::CUDAGuard guard;
  at::Device dev;
  void* stream;
  explicit On(at::Device d) : guard(d), dev(d), stream(c10::cuda::getCurrentCUDAStream(d.index()).stream()) {}
};

template <typename Fn, typename... A>
mxb_status run(Fn fn, A... args) {
  py::gil_scoped_release nogil;  // a launch can block while the stream's queue is full
  return fn(args...);
}
void raise_unless_ok(mxb_status s, const char* what) {
  if (s != MXB_OK) py::module_::import("mixlab_b200._lib").attr("check")(s, what);  // raises MxbError
}
template <typename Fn, typename... A>
void call(const char* what, Fn fn, A... args) { raise_unless_ok(run(fn, args...), what); }

// ------------------------------------------------------------------ workspace
// One cached byte buffer per device and stream, grown to the largest size asked for: launches of one stream run one after
// the other and can share scratch, those of two streams cannot.  `saved` describes the forward call whose intermediates
// the buffer holds; any other use of the buffer clears it, so that a backward with use_saved=True cannot consume
// overwritten tiles.
//
// A graph keeps the addresses it was captured with.  So a buffer belongs to the capture it was allocated in (its memory
// then comes from that graph's own pool, which nobody else is given): calls outside that capture take another one, and
// a captured call never takes one that a later call may outgrow and give back.
struct Token {
  int kind = 0;  // 0: nothing saved
  int64_t extra[4] = {};
  struct Operand {
    const void* data;
    std::vector<int64_t> shape;
    at::ScalarType dtype;
    bool operator==(const Operand& o) const { return data == o.data && dtype == o.dtype && shape == o.shape; }
  };
  std::vector<Operand> operands;
  bool operator==(const Token& o) const {
    return kind == o.kind && std::equal(extra, extra + 4, o.extra) && operands == o.operands;
  }
};
struct Workspace {
  std::mutex busy;  // held by a Lease
  Tensor buf;
  Token saved;
  unsigned long long capture = 0;  // the capture `buf` was allocated in, 0: none
  uint64_t used = 0;  // for the choice of the one to give back
};
// At most this many streams of a device keep a buffer; the one unused for longest goes back to the allocator (it was
// allocated on the stream that used it, so its memory is handed on in that stream's order).
constexpr size_t kStreamsPerDevice = 8;
using Workspaces = std::map<std::pair<int, void*>, std::shared_ptr<Workspace>>;
// The workspace of a stream.  The table is only touched under the interpreter lock.
std::shared_ptr<Workspace> workspace_of(int device, void* stream) {
  static auto* all = new Workspaces;  // never destroyed: the allocator may be gone by then
  static uint64_t clock = 0;
  auto& w = (*all)[{device, stream}];
  if (!w) w = std::make_shared<Workspace>();
  w->used = ++clock;
  const std::shared_ptr<Workspace> found = w;
  size_t count = 0;
  auto oldest = all->end();
  for (auto i = all->begin(); i != all->end(); ++i) {
    if (i->first.first != device) continue;
    ++count;
    if (i->second.use_count() == 1 && (oldest == all->end() || i->second->used < oldest->second->used)) oldest = i;
  }
  if (count > kStreamsPerDevice && oldest != all->end()) all->erase(oldest);
  return found;
}
unsigned long long capture_of(void* stream) {
  cudaStreamCaptureStatus status = cudaStreamCaptureStatusNone;
  unsigned long long id = 0;
  if (cudaStreamGetCaptureInfo(static_cast<cudaStream_t>(stream), &status, &id) != cudaSuccess) {
    cudaGetLastError();  // (the legacy stream may not be asked while another one captures; it does not capture itself)
    return 0;
  }
  return status == cudaStreamCaptureStatusActive ? id : 0;
}
// The workspace of the current stream, for one call: from the look at its buffer and token until the launches are
// enqueued and the new token is set.  The interpreter lock does not cover that span - run() releases it - so the
// workspace has a lock of its own, which is waited for without the interpreter lock.  Whatever may run Python code
// (allocating results, raising) stays outside the span.
class Lease {
 public:
  explicit Lease(const On& on) : w_(workspace_of(on.dev.index(), on.stream)), dev_(on.dev), capture_(capture_of(on.stream)) {
    py::gil_scoped_release nogil;
    lock_ = std::unique_lock<std::mutex>(w_->busy);
  }
  // a buffer of at least nbytes, whatever it held
  void take(size_t nbytes) {
    w_->saved.kind = 0;
    if (!w_->buf.defined() || bytes() < nbytes || w_->capture != capture_) {
      w_->buf = Tensor();
      w_->buf = make({static_cast<int64_t>(nbytes < 256 ? 256 : nbytes)}, at::kByte, dev_);
      w_->capture = capture_;
    }
  }
  // the buffer of a use_saved backward, which still has to hold what the forward described by `want` left in it
  void take_saved(const Token& want, size_t nbytes, const char* what) {
    if (!(w_->saved == want))
      throw std::runtime_error(std::string(what) + ": use_saved=True needs the immediately preceding save_for_backward forward on "
                               "the same tensors, stream and device (the cached workspace has been reused since, or never held them)");
    if (bytes() < nbytes)
      throw std::runtime_error(std::string(what) + ": the cached workspace was reallocated after the forward saved into it");
  }
  void save(Token t) { w_->saved = std::move(t); }
  void* data() const { return ptr(w_->buf); }
  size_t bytes() const { return static_cast<size_t>(w_->buf.numel()); }
  const Tensor& buffer() const { return w_->buf; }

 private:
  std::shared_ptr<Workspace> w_;  // (released after the lock: the last owner frees it)
  std::unique_lock<std::mutex> lock_;
  at::Device dev_;
  unsigned long long capture_;
};
// The current stream's buffer itself (its contents are the caller's from then on).
Tensor workspace(size_t nbytes, int device) {
  const On on(at::Device(at::kCUDA, device));
  Lease ws(on);
  ws.take(nbytes);
  return ws.buffer();
}
Token token(int kind, std::initializer_list<const Tensor*> ts, std::initializer_list<int64_t> extra) {
  Token t;
  t.kind = kind;
  std::copy(extra.begin(), extra.end(), t.extra);
  t.operands.reserve(ts.size());
  for (const Tensor* x : ts) t.operands.push_back({x->data_ptr(), x->sizes().vec(), x->scalar_type()});
  return t;
}
// A call that needs scratch and leaves nothing in it.
template <typename Fn, typename... A>
void call_with_scratch(const On& on, size_t nbytes, const char* what, Fn fn, A... args) {
  mxb_status s;
  {
    Lease ws(on);
    ws.take(nbytes);
    s = run([&] { return fn(args..., ws.data(), ws.bytes(), on.stream); });
  }
  raise_unless_ok(s, what);
}

// ------------------------------------------------------------------ gated delta rule
mxb_gdn_desc gdn_desc(const Tensor& q, const Tensor& v, int64_t chunk, bool gate_is_log, int64_t flags) {
  if (q.dim() != 4 || v.dim() != 4) throw py::value_error("q, k must be [B,T,H,Dk] and v [B,T,H,Dv]");
  return {(int32_t)q.size(0), (int32_t)q.size(1), (int32_t)q.size(2), (int32_t)q.size(3), (int32_t)v.size(3), (int32_t)chunk,
          io_code(q), gate_is_log ? 1 : 0, (int32_t)flags};
}
void check_gdn(const mxb_gdn_desc& d, const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& beta, const Tensor& gate) {
  const auto dev = q.device();
  const auto io = q.scalar_type();
  const int64_t kd[] = {d.B, d.T, d.H, d.Dk}, vd[] = {d.B, d.T, d.H, d.Dv};
  check(q, kd, io, dev, "q");
  check(k, kd, io, dev, "k");
  check(v, vd, io, dev, "v");
  check(beta, Shape(kd, 3), F, dev, "beta");
  check(gate, Shape(kd, 3), F, dev, "gate");
}
Token gdn_token(const mxb_gdn_desc& d, const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& beta,
                const Tensor& gate) {
  // the flag bits that choose a kernel family choose the layout of what a forward saves
  return token(1, {&q, &k, &v, &beta, &gate},
               {d.chunk, d.gate_is_log, d.flags & ~(MXB_GDN_SAVE_FOR_BWD | MXB_GDN_BWD_USE_SAVED)});
}

py::object gdn_forward(const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& beta, const Tensor& gate, int64_t chunk,
                       bool gate_is_log, const Opt& h0, bool want_final, int64_t flags, bool save) {
  const at::Device dev = cuda_device(q);
  const mxb_gdn_desc d = gdn_desc(q, v, chunk, gate_is_log, save ? flags | MXB_GDN_SAVE_FOR_BWD : flags);
  check_gdn(d, q, k, v, beta, gate);
  const int64_t sd[] = {d.B, d.H, d.Dk, d.Dv};
  check(h0, sd, F, dev, "h0");
  const On on(dev);
  Tensor out = like(v), hT;
  if (want_final) hT = make(sd, F, on.dev);
  mxb_status s;
  {
    Lease ws(on);
    ws.take(abi.mxb_gdn_fwd_workspace_bytes(&d));
    s = run(abi.mxb_gdn_fwd, &d, ptr(q), ptr(k), ptr(v), ptr<float>(beta), ptr<float>(gate), ptr<float>(h0), ptr(out),
            want_final ? ptr<float>(hT) : nullptr, ws.data(), ws.bytes(), on.stream);
    if (save && s == MXB_OK) ws.save(gdn_token(d, q, k, v, beta, gate));
  }
  raise_unless_ok(s, "mxb_gdn_fwd");
  return want_final ? py::object(py::make_tuple(out, hT)) : py::cast(out);
}

py::dict gdn_backward(const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& beta, const Tensor& gate, const Tensor& d_out,
                      int64_t chunk, bool gate_is_log, const Opt& h0, const Opt& d_final, int64_t flags, bool use_saved) {
  const at::Device dev = cuda_device(q);
  const mxb_gdn_desc d = gdn_desc(q, v, chunk, gate_is_log, use_saved ? flags | MXB_GDN_BWD_USE_SAVED : flags);
  check_gdn(d, q, k, v, beta, gate);
  const int64_t sd[] = {d.B, d.H, d.Dk, d.Dv};
  check(d_out, v.sizes(), q.scalar_type(), dev, "d_out");
  check(h0, sd, F, dev, "h0");
  check(d_final, sd, F, dev, "d_final_state");
  const On on(dev);
  Tensor dq = like(q), dk = like(k), dv = like(v), db = like(beta), dg = like(gate);
  Opt dh0;
  if (h0) dh0 = like(*h0);
  const size_t nws = abi.mxb_gdn_bwd_workspace_bytes(&d);
  mxb_status s;
  {
    Lease ws(on);
    if (use_saved) ws.take_saved(gdn_token(d, q, k, v, beta, gate), nws, "gated_delta_scan_backward");
    else ws.take(nws);
    s = run(abi.mxb_gdn_bwd, &d, ptr(q), ptr(k), ptr(v), ptr<float>(beta), ptr<float>(gate), ptr<float>(h0), ptr(d_out),
            ptr<float>(d_final), ptr(dq), ptr(dk), ptr(dv), ptr<float>(db), ptr<float>(dg), ptr<float>(dh0), ws.data(), ws.bytes(),
            on.stream);
  }
  raise_unless_ok(s, "mxb_gdn_bwd");
  py::dict r;
  r["dq"] = dq; r["dk"] = dk; r["dv"] = dv; r["dbeta"] = db; r["dgate"] = dg; r["dh0"] = dh0;
  return r;
}

Tensor gdn_decode(const Tensor& state, const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& beta, const Tensor& gate,
                  bool gate_is_log, const Opt& out_, int64_t flags) {
  const at::Device dev = cuda_device(state);
  if (!q.is_cuda()) not_cuda();
  if (state.dim() != 4) throw py::value_error("state must be [N,H,Dk,Dv]");
  const int64_t N = state.size(0), H = state.size(1), K = state.size(2), V = state.size(3);
  const mxb_gdn_desc d{(int32_t)N, 1, (int32_t)H, (int32_t)K, (int32_t)V, 0, io_code(q), gate_is_log ? 1 : 0, (int32_t)flags};
  const auto io = q.scalar_type();
  const int64_t kd[] = {N, H, K}, vd[] = {N, H, V};
  check(state, state.sizes(), F, dev, "state");
  check(q, kd, io, dev, "q");
  check(k, kd, io, dev, "k");
  check(v, vd, io, dev, "v");
  check(beta, Shape(kd, 2), F, dev, "beta");
  check(gate, Shape(kd, 2), F, dev, "gate");
  check(out_, vd, io, dev, "out");
  const On on(dev);
  Tensor out = out_ ? *out_ : like(v);
  call("mxb_gdn_decode_step", abi.mxb_gdn_decode_step, &d, ptr<float>(state), ptr(q), ptr(k), ptr(v), ptr<float>(beta),
       ptr<float>(gate), ptr(out), on.stream);
  return out;
}

// ------------------------------------------------------------------ gated_deltanet block stages
struct BlockArgs {
  mxb_gdn_desc d;
  int64_t kd[3], vd[3], hd[3];
};
BlockArgs check_block_pre(at::Device dev, const Tensor& qp, const Tensor& kp, const Tensor& vp, const Tensor& cq, const Tensor& ck,
                          const Tensor& cv, const Tensor& a, const Tensor& b, const Tensor& al, const Tensor& bias, int64_t H,
                          int64_t Dk, int64_t Dv, bool gate_is_log) {
  if (qp.dim() != 3) throw py::value_error("q_proj must be [B,T,H*Dk]");
  const int64_t B = qp.size(0), T = qp.size(1);
  BlockArgs r{{(int32_t)B, (int32_t)T, (int32_t)H, (int32_t)Dk, (int32_t)Dv, 64, io_code(qp), gate_is_log ? 1 : 0, 0},
              {B, T, H * Dk}, {B, T, H * Dv}, {B, T, H}};
  const auto io = qp.scalar_type();
  const int64_t wk[] = {4, H * Dk}, wv[] = {4, H * Dv};
  check(qp, r.kd, io, dev, "q_proj");
  check(kp, r.kd, io, dev, "k_proj");
  check(vp, r.vd, io, dev, "v_proj");
  check(cq, wk, F, dev, "conv_q");
  check(ck, wk, F, dev, "conv_k");
  check(cv, wv, F, dev, "conv_v");
  check(a, r.hd, F, dev, "a_raw");
  check(b, r.hd, F, dev, "b_raw");
  check(al, Shape(&H, 1), F, dev, "a_log");
  check(bias, Shape(&H, 1), F, dev, "dt_bias");
  return r;
}
py::tuple gdn_block_pre(const Tensor& qp, const Tensor& kp, const Tensor& vp, const Tensor& cq, const Tensor& ck, const Tensor& cv,
                        const Tensor& a, const Tensor& b, const Tensor& al, const Tensor& bias, int64_t H, int64_t Dk, int64_t Dv,
                        bool gate_is_log) {
  const at::Device dev = cuda_device(qp);
  BlockArgs x = check_block_pre(dev, qp, kp, vp, cq, ck, cv, a, b, al, bias, H, Dk, Dv, gate_is_log);
  const On on(dev);
  const int64_t k4[] = {x.d.B, x.d.T, H, Dk}, v4[] = {x.d.B, x.d.T, H, Dv};
  const auto io = qp.scalar_type();
  Tensor q = make(k4, io, on.dev), k = make(k4, io, on.dev), v = make(v4, io, on.dev), beta = make(x.hd, F, on.dev), gate = make(x.hd, F, on.dev);
  call("mxb_gdn_block_pre_fwd", abi.mxb_gdn_block_pre_fwd, &x.d, ptr(qp), ptr(kp), ptr(vp), ptr<float>(cq), ptr<float>(ck), ptr<float>(cv),
       ptr<float>(a), ptr<float>(b), ptr<float>(al), ptr<float>(bias), ptr(q), ptr(k), ptr(v), ptr<float>(beta), ptr<float>(gate), on.stream);
  return py::make_tuple(q, k, v, beta, gate);
}
py::dict gdn_block_pre_backward(const Tensor& qp, const Tensor& kp, const Tensor& vp, const Tensor& cq, const Tensor& ck,
                                const Tensor& cv, const Tensor& a, const Tensor& b, const Tensor& al, const Tensor& bias, int64_t H,
                                int64_t Dk, int64_t Dv, const Tensor& dq, const Tensor& dk, const Tensor& dv, const Tensor& dbeta,
                                const Tensor& dgate, bool gate_is_log) {
  const at::Device dev = cuda_device(qp);
  BlockArgs x = check_block_pre(dev, qp, kp, vp, cq, ck, cv, a, b, al, bias, H, Dk, Dv, gate_is_log);
  const int64_t k4[] = {x.d.B, x.d.T, H, Dk}, v4[] = {x.d.B, x.d.T, H, Dv};
  const auto io = qp.scalar_type();
  check(dq, k4, io, dev, "dq");
  check(dk, k4, io, dev, "dk");
  check(dv, v4, io, dev, "dv");
  check(dbeta, x.hd, F, dev, "dbeta");
  check(dgate, x.hd, F, dev, "dgate");
  const On on(dev);
  Tensor dqp = like(qp), dkp = like(kp), dvp = like(vp), dcq = like(cq), dck = like(ck), dcv = like(cv), da = like(a), db = like(b),
         dal = like(al), dbias = like(bias);
  call_with_scratch(on, abi.mxb_gdn_block_workspace_bytes(&x.d), "mxb_gdn_block_pre_bwd", abi.mxb_gdn_block_pre_bwd,
                    &x.d, ptr(qp), ptr(kp), ptr(vp), ptr<float>(cq), ptr<float>(ck), ptr<float>(cv), ptr<float>(a),
                    ptr<float>(b), ptr<float>(al), ptr<float>(bias), ptr(dq), ptr(dk), ptr(dv), ptr<float>(dbeta),
                    ptr<float>(dgate), ptr(dqp), ptr(dkp), ptr(dvp), ptr<float>(dcq), ptr<float>(dck),
                    ptr<float>(dcv), ptr<float>(da), ptr<float>(db), ptr<float>(dal), ptr<float>(dbias));
  py::dict r;
  r["dq_proj"] = dqp; r["dk_proj"] = dkp; r["dv_proj"] = dvp; r["dconv_q"] = dcq; r["dconv_k"] = dck; r["dconv_v"] = dcv;
  r["da_raw"] = da; r["db_raw"] = db; r["da_log"] = dal; r["ddt_bias"] = dbias;
  return r;
}
mxb_gdn_desc check_block_post(at::Device dev, const Tensor& o, const Tensor& z, const Tensor& w) {
  if (o.dim() != 4) throw py::value_error("o must be [B,T,H,Dv]");
  const int64_t B = o.size(0), T = o.size(1), H = o.size(2), Dv = o.size(3), zd[] = {B, T, H * Dv};
  const mxb_gdn_desc d{(int32_t)B, (int32_t)T, (int32_t)H, 8, (int32_t)Dv, 64, io_code(o), 0, 0};
  check(o, o.sizes(), o.scalar_type(), dev, "o");
  check(z, zd, o.scalar_type(), dev, "z");
  check(w, Shape(&Dv, 1), F, dev, "o_norm");
  return d;
}
Tensor gdn_block_post(const Tensor& o, const Tensor& z, const Tensor& w) {
  const at::Device dev = cuda_device(o);
  const mxb_gdn_desc d = check_block_post(dev, o, z, w);
  const On on(dev);
  Tensor y = like(z);
  call("mxb_gdn_block_post_fwd", abi.mxb_gdn_block_post_fwd, &d, ptr(o), ptr(z), ptr<float>(w), ptr(y), on.stream);
  return y;
}
py::dict gdn_block_post_backward(const Tensor& o, const Tensor& z, const Tensor& w, const Tensor& dy) {
  const at::Device dev = cuda_device(o);
  const mxb_gdn_desc d = check_block_post(dev, o, z, w);
  check(dy, z.sizes(), o.scalar_type(), dev, "dy");
  const On on(dev);
  Tensor d_o = like(o), dz = like(z), dw = like(w);
  call_with_scratch(on, abi.mxb_gdn_block_workspace_bytes(&d), "mxb_gdn_block_post_bwd", abi.mxb_gdn_block_post_bwd,
                    &d, ptr(o), ptr(z), ptr<float>(w), ptr(dy), ptr(d_o), ptr(dz), ptr<float>(dw));
  py::dict r;
  r["do"] = d_o; r["dz"] = dz; r["do_norm"] = dw;
  return r;
}

// ------------------------------------------------------------------ Mamba-3 scan
mxb_mamba3_desc check_mamba3(at::Device dev, const Tensor& x, const Tensor& dt, const Tensor& lam, const Tensor& theta,
                             const Tensor& a_log, const Tensor& b, const Tensor& c, int64_t nheads, int64_t flags) {
  if (x.dim() != 3 || b.dim() != 4) throw py::value_error("x must be [B,T,D] and b, c [B,T,G,N]");
  const int64_t B = x.size(0), T = x.size(1), D = x.size(2), G = b.size(2), N = b.size(3);
  const mxb_mamba3_desc d{(int32_t)B, (int32_t)T, (int32_t)D, (int32_t)N, (int32_t)G, (int32_t)nheads, io_code(x), (int32_t)flags};
  const auto io = x.scalar_type();
  const int64_t per[] = {B, T, nheads > 0 ? nheads : D, N / 2}, al[] = {nheads > 0 ? nheads : D, N}, gn[] = {B, T, G, N};
  check(x, x.sizes(), io, dev, "x");
  check(dt, Shape(per, 3), F, dev, "dt");
  check(lam, Shape(per, 3), F, dev, "lambda");
  check(theta, Shape(per, nheads > 0 ? 3 : 4), F, dev, "theta");
  check(a_log, Shape(al, nheads > 0 ? 1 : 2), F, dev, "a_log");
  check(b, gn, io, dev, "b");
  check(c, gn, io, dev, "c");
  return d;
}
Token mamba3_token(const mxb_mamba3_desc& d, const Tensor& x, const Tensor& dt, const Tensor& lam, const Tensor& theta,
                   const Tensor& a_log, const Tensor& b, const Tensor& c) {
  return token(2, {&x, &dt, &lam, &theta, &a_log, &b, &c}, {d.nheads, d.flags & ~(MXB_MAMBA3_SAVE_FOR_BWD | MXB_MAMBA3_BWD_USE_SAVED)});
}
Tensor mamba3_forward(const Tensor& x, const Tensor& dt, const Tensor& lam, const Tensor& theta, const Tensor& a_log, const Tensor& b,
                      const Tensor& c, int64_t nheads, int64_t flags, bool save) {
  const at::Device dev = cuda_device(x);
  const mxb_mamba3_desc d = check_mamba3(dev, x, dt, lam, theta, a_log, b, c, nheads, save ? flags | MXB_MAMBA3_SAVE_FOR_BWD : flags);
  const On on(dev);
  Tensor y = like(x);
  mxb_status s;
  {
    Lease ws(on);
    // (a forward that saves nothing needs little or no scratch, but the backward that may follow finds its buffer here)
    const size_t fwd = abi.mxb_mamba3_fwd_workspace_bytes(&d), bwd = save ? abi.mxb_mamba3_bwd_workspace_bytes(&d) : 0;
    ws.take(std::max(fwd, bwd));
    s = run(abi.mxb_mamba3_fwd, &d, ptr(x), ptr<float>(dt), ptr<float>(lam), ptr<float>(theta), ptr<float>(a_log), ptr(b), ptr(c),
            ptr(y), ws.data(), ws.bytes(), on.stream);
    if (save && s == MXB_OK) ws.save(mamba3_token(d, x, dt, lam, theta, a_log, b, c));
  }
  raise_unless_ok(s, "mxb_mamba3_fwd");
  return y;
}
py::dict mamba3_backward(const Tensor& x, const Tensor& dt, const Tensor& lam, const Tensor& theta, const Tensor& a_log, const Tensor& b,
                         const Tensor& c, const Tensor& dy, int64_t nheads, int64_t flags, bool use_saved) {
  const at::Device dev = cuda_device(x);
  const mxb_mamba3_desc d = check_mamba3(dev, x, dt, lam, theta, a_log, b, c, nheads, use_saved ? flags | MXB_MAMBA3_BWD_USE_SAVED : flags);
  check(dy, x.sizes(), x.scalar_type(), dev, "dy");
  const On on(dev);
  Tensor dx = like(x), ddt = like(dt), dlam = like(lam), dth = like(theta), dal = like(a_log), db = like(b), dc = like(c);
  const size_t nws = abi.mxb_mamba3_bwd_workspace_bytes(&d);
  mxb_status s;
  {
    Lease ws(on);
    if (use_saved) ws.take_saved(mamba3_token(d, x, dt, lam, theta, a_log, b, c), nws, "mamba3_selective_scan_backward");
    else ws.take(nws);
    s = run(abi.mxb_mamba3_bwd, &d, ptr(x), ptr<float>(dt), ptr<float>(lam), ptr<float>(theta), ptr<float>(a_log), ptr(b), ptr(c),
            ptr(dy), ptr(dx), ptr<float>(ddt), ptr<float>(dlam), ptr<float>(dth), ptr<float>(dal), ptr(db), ptr(dc), ws.data(),
            ws.bytes(), on.stream);
  }
  raise_unless_ok(s, "mxb_mamba3_bwd");
  py::dict r;
  r["dx"] = dx; r["ddt"] = ddt; r["dlambda"] = dlam; r["dtheta"] = dth; r["da_log"] = dal; r["db"] = db; r["dc"] = dc;
  return r;
}

// ------------------------------------------------------------------ Mamba-3 block stages
mxb_mamba3_desc m3_rows(const Tensor& x) {
  if (x.dim() != 3) throw py::value_error("expected a [B,T,D] tensor");
  return {(int32_t)x.size(0), (int32_t)x.size(1), (int32_t)x.size(2), 8, 1, 0, io_code(x), 0};
}
mxb_mamba3_desc check_conv(at::Device dev, const Tensor& x, const Tensor& w) {
  const mxb_mamba3_desc d = m3_rows(x);
  const int64_t wd[] = {d.D, w.dim() ? w.size(-1) : 0};
  check(x, x.sizes(), x.scalar_type(), dev, "x");
  check(w, wd, F, dev, "w");
  return d;
}
Tensor mamba3_block_conv(const Tensor& x, const Tensor& w) {
  const at::Device dev = cuda_device(x);
  const mxb_mamba3_desc d = check_conv(dev, x, w);
  const On on(dev);
  Tensor y = like(x);
  call("mxb_mamba3_block_conv_fwd", abi.mxb_mamba3_block_conv_fwd, &d, (int32_t)w.size(1), ptr(x), ptr<float>(w), ptr(y), on.stream);
  return y;
}
py::dict mamba3_block_conv_backward(const Tensor& x, const Tensor& w, const Tensor& dy) {
  const at::Device dev = cuda_device(x);
  const mxb_mamba3_desc d = check_conv(dev, x, w);
  check(dy, x.sizes(), x.scalar_type(), dev, "dy");
  const On on(dev);
  Tensor dx = like(x), dw = like(w);
  call_with_scratch(on, abi.mxb_mamba3_block_workspace_bytes(&d), "mxb_mamba3_block_conv_bwd",
                    abi.mxb_mamba3_block_conv_bwd, &d, (int32_t)w.size(1), ptr(x), ptr<float>(w), ptr(dy), ptr(dx),
                    ptr<float>(dw));
  py::dict r;
  r["dx"] = dx; r["dw"] = dw;
  return r;
}
mxb_mamba3_desc check_bc(at::Device dev, const Tensor& bp, const Tensor& cp, const Tensor& bs, const Tensor& cs, int64_t G, int64_t N) {
  if (bp.dim() != 3) throw py::value_error("b_proj must be [B,T,G*N]");
  const int64_t gn[] = {bp.size(0), bp.size(1), G * N};
  const mxb_mamba3_desc d{(int32_t)gn[0], (int32_t)gn[1], 8, (int32_t)N, (int32_t)G, 0, io_code(bp), 0};
  check(bp, gn, bp.scalar_type(), dev, "b_proj");
  check(cp, gn, bp.scalar_type(), dev, "c_proj");
  check(bs, Shape(&N, 1), F, dev, "b_scale");
  check(cs, Shape(&N, 1), F, dev, "c_scale");
  return d;
}
py::tuple mamba3_block_bc(const Tensor& bp, const Tensor& cp, const Tensor& bs, const Tensor& cs, const Tensor& bb, const Tensor& cb,
                          int64_t G, int64_t N, double eps) {
  const at::Device dev = cuda_device(bp);
  const mxb_mamba3_desc d = check_bc(dev, bp, cp, bs, cs, G, N);
  const int64_t gn = G * N, o4[] = {d.B, d.T, G, N};
  check(bb, Shape(&gn, 1), F, dev, "b_bias");
  check(cb, Shape(&gn, 1), F, dev, "c_bias");
  const On on(dev);
  Tensor b = make(o4, bp.scalar_type(), on.dev), c = make(o4, bp.scalar_type(), on.dev);
  call("mxb_mamba3_block_bc_fwd", abi.mxb_mamba3_block_bc_fwd, &d, (float)eps, ptr(bp), ptr(cp), ptr<float>(bs), ptr<float>(cs),
       ptr<float>(bb), ptr<float>(cb), ptr(b), ptr(c), on.stream);
  return py::make_tuple(b, c);
}
py::dict mamba3_block_bc_backward(const Tensor& bp, const Tensor& cp, const Tensor& bs, const Tensor& cs, const Tensor& db,
                                  const Tensor& dc, int64_t G, int64_t N, double eps) {
  const at::Device dev = cuda_device(bp);
  const mxb_mamba3_desc d = check_bc(dev, bp, cp, bs, cs, G, N);
  const int64_t gn = G * N, o4[] = {d.B, d.T, G, N};
  check(db, o4, bp.scalar_type(), dev, "db");
  check(dc, o4, bp.scalar_type(), dev, "dc");
  const On on(dev);
  Tensor dbp = like(bp), dcp = like(cp), dbs = like(bs), dcs = like(cs), dbb = make(Shape(&gn, 1), F, on.dev), dcb = make(Shape(&gn, 1), F, on.dev);
  call_with_scratch(on, abi.mxb_mamba3_block_workspace_bytes(&d), "mxb_mamba3_block_bc_bwd",
                    abi.mxb_mamba3_block_bc_bwd, &d, (float)eps, ptr(bp), ptr(cp), ptr<float>(bs), ptr<float>(cs),
                    ptr(db), ptr(dc), ptr(dbp), ptr(dcp), ptr<float>(dbs), ptr<float>(dcs), ptr<float>(dbb),
                    ptr<float>(dcb));
  py::dict r;
  r["db_proj"] = dbp; r["dc_proj"] = dcp; r["db_scale"] = dbs; r["dc_scale"] = dcs; r["db_bias"] = dbb; r["dc_bias"] = dcb;
  return r;
}
mxb_mamba3_desc check_post(at::Device dev, const Tensor& y, const Tensor& z, const Tensor& w) {
  const mxb_mamba3_desc d = m3_rows(y);
  const int64_t D = d.D;
  check(y, y.sizes(), y.scalar_type(), dev, "y");
  check(z, y.sizes(), y.scalar_type(), dev, "z");
  check(w, Shape(&D, 1), F, dev, "post_norm");
  return d;
}
Tensor mamba3_block_post(const Tensor& y, const Tensor& z, const Tensor& w, double eps) {
  const at::Device dev = cuda_device(y);
  const mxb_mamba3_desc d = check_post(dev, y, z, w);
  const On on(dev);
  Tensor out = like(y);
  call("mxb_mamba3_block_post_fwd", abi.mxb_mamba3_block_post_fwd, &d, (float)eps, ptr(y), ptr(z), ptr<float>(w), ptr(out), on.stream);
  return out;
}
py::dict mamba3_block_post_backward(const Tensor& y, const Tensor& z, const Tensor& w, const Tensor& dout, double eps) {
  const at::Device dev = cuda_device(y);
  const mxb_mamba3_desc d = check_post(dev, y, z, w);
  check(dout, y.sizes(), y.scalar_type(), dev, "dout");
  const On on(dev);
  Tensor dy = like(y), dz = like(z), dw = like(w);
  call_with_scratch(on, abi.mxb_mamba3_block_workspace_bytes(&d), "mxb_mamba3_block_post_bwd",
                    abi.mxb_mamba3_block_post_bwd, &d, (float)eps, ptr(y), ptr(z), ptr<float>(w), ptr(dout), ptr(dy),
                    ptr(dz), ptr<float>(dw));
  py::dict r;
  r["dy"] = dy; r["dz"] = dz; r["dpost_norm"] = dw;
  return r;
}

// ------------------------------------------------------------------ IR op records
Tensor ir_op_forward(int64_t op_type, const std::vector<Tensor>& inputs, const std::vector<int64_t>& int_params,
                     const std::vector<int64_t>& out_shape, const std::vector<double>& float_params) {
  for (const Tensor& t : inputs)
    if (!t.is_cuda()) not_cuda();
  for (size_t i = 0; i < inputs.size(); ++i)
    if (!inputs[i].is_contiguous() || inputs[i].device() != inputs[0].device())
      throw py::value_error("input " + std::to_string(i) + ": contiguous tensors on one device expected");
  if (inputs.empty()) throw py::value_error("an op record has inputs");
  const at::Device dev = cuda_device(inputs[0]);
  const int32_t io = io_code(inputs[0]);
  const On on(dev);
  Tensor out = make(out_shape, inputs[0].scalar_type(), on.dev);
  std::vector<const void*> in;
  for (const Tensor& t : inputs) in.push_back(t.data_ptr());
  void* outs[] = {out.data_ptr()};
  const std::vector<int32_t> ints(int_params.begin(), int_params.end());
  const std::vector<float> floats(float_params.begin(), float_params.end());
  const mxb_ir_op op{(int32_t)op_type, in.data(), (int32_t)in.size(), outs, 1, floats.data(), (int32_t)floats.size(),
                     ints.data(), (int32_t)ints.size(), io};
  call_with_scratch(on, abi.mxb_ir_op_workspace_bytes(&op), "mxb_ir_op_forward", abi.mxb_ir_op_forward, &op);
  return out;
}

}  // namespace

PYBIND11_MODULE(_front, m) {
  m.def("open", &open_library);
  m.def("workspace", &workspace);
  m.def("ir_op_forward", &ir_op_forward);
  m.def("gdn_forward", &gdn_forward);
  m.def("gdn_backward", &gdn_backward);
  m.def("gdn_decode", &gdn_decode);
  m.def("gdn_block_pre", &gdn_block_pre);
  m.def("gdn_block_pre_backward", &gdn_block_pre_backward);
  m.def("gdn_block_post", &gdn_block_post);
  m.def("gdn_block_post_backward", &gdn_block_post_backward);
  m.def("mamba3_forward", &mamba3_forward);
  m.def("mamba3_backward", &mamba3_backward);
  m.def("mamba3_block_conv", &mamba3_block_conv);
  m.def("mamba3_block_conv_backward", &mamba3_block_conv_backward);
  m.def("mamba3_block_bc", &mamba3_block_bc);
  m.def("mamba3_block_bc_backward", &mamba3_block_bc_backward);
  m.def("mamba3_block_post", &mamba3_block_post);
  m.def("mamba3_block_post_backward", &mamba3_block_post_backward);
}

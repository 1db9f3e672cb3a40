// The host side of one fused-MoE layer call in native code: permutation (+ quantisation), gemm1,
// activation, gemm2 and the top-k reduction are launched from one function of the extension
// module, with the intermediates carved out of one workspace.  The stages are the reference's
// (vllm_xpu_kernels/fused_moe_interface.py:328-419 of vllm-xpu-kernels).
//
// A decode step is bound by the host as much as by the GPU: as seven torch ops with their Python
// wrappers, argument checks and buffer look-ups, a call took 50 to 80 us of host time; here the
// launches are what is left (about 2 us each).
#include "layer.h"

#include <c10/cuda/CUDAGraphsC10Utils.h>
#include <torch/csrc/Dtype.h>
#include <torch/csrc/Exceptions.h>
#include <torch/csrc/autograd/python_variable.h>

#include <map>
#include <memory>
#include <mutex>
#include <utility>

namespace b200shim {
namespace {

enum ActKind { kSilu = 0, kGelu, kGeluTanh, kSwigluOai, kRelu2NoMul, kSwigluStep };
enum Form { kUnfused = 0, kEpilogue = 1, kFp8 = 2 };   // what gemm1 does besides multiplying

struct Plan {
  at::Tensor w13, w2;
  std::optional<at::Tensor> s13, b13, s2, b2;
  int64_t inter = 0, experts = 0, total_experts = 0;
  int topk = 0, act = 0, inter_scale = 1, planes = 1;
  bool block_fp8 = false, mx = false;
  double clamp = 0.0;
  // Up to this many rows per expert the block-scaled int4 kernel (gemm_tc_i4.cu) takes the layer: it
  // streams the weights faster than the one that expands them to 16 bits (gemm_tc_dq.cu), until experts
  // need a second of its tiles of 32 tokens.  A layer of 8 experts of 4096 x 14336, 2 a token, with routing as it
  // comes, this / that kernel, us: bfloat16 218 / 305 at 8 rows an expert, 235 / 289 at 12, 249 / 293 at 16, 292 / 297 at
  // 20, 295 / 298 at 24 (since then the first one 207 at 8, 226 at 12, 238 at 16); float16 (three planes) 222 / 304 at 8, 236 /
  // 287 at 10, 266 / 288 at 12, 292 / 292 at 16, 365 / 295 at 20.  Half a tile leaves room for uneven routing, and the
  // planes are the more accurate: error of the layer's output against 64 bits (2-norm, 9 to
  // 16 rows an expert) 5.3e-4 / 6.1e-4, where the other kernel rounds a weight after its scale; bfloat16 4.3e-3 / 4.9e-3.
  static constexpr int64_t kI4PlaneRows = 16;
};
const char* const kPlanName = "b200moe.layer_plan";

// ------------------------------- workspace ------------------------------------
// One grow-only buffer per (device, stream), shared by all layers: the calls of a stream run one
// after the other, so the next one may overwrite what the previous one left.  A call has the buffer
// to itself while it launches and puts it back when it returns; one that launches on the same stream
// meanwhile (from another thread, or from a stage hook) finds none and takes its own.  At most
// kMaxSlabs streams keep one (the least recently used is given back), all are given back with the last
// layer object.  A call under stream capture takes its memory from the graph's pool instead: a graph
// is replayed on any stream, beside later calls on the one it was captured on and beside other graphs,
// and what it uses has to live as long as it does.
constexpr size_t kMaxSlabs = 8;
struct Slab {
  at::Tensor mem;
  uint64_t used = 0;
};
std::mutex g_mutex;
auto& g_slabs = *new std::map<std::pair<int, int64_t>, Slab>();   // (never destroyed: CUDA may be gone at exit)
uint64_t g_tick = 0;
int64_t g_plans = 0;

void clear_slabs() {
  std::map<std::pair<int, int64_t>, Slab> old;   // (freed behind the lock)
  std::lock_guard<std::mutex> lock(g_mutex);
  g_slabs.swap(old);
}

class Workspace {
 public:
  Workspace(const c10::cuda::CUDAStream& stream, size_t bytes, bool persistent)
      : key_(stream.device_index(), (int64_t)stream.id()),
        keep_(persistent && c10::cuda::currentStreamCaptureStatusMayInitCtx() == c10::cuda::CaptureStatus::None) {
    if (keep_) {
      std::lock_guard<std::mutex> lock(g_mutex);
      auto it = g_slabs.find(key_);
      if (it != g_slabs.end()) {
        mem = std::move(it->second.mem);
        g_slabs.erase(it);
      }
    }
    if (mem.defined() && (size_t)mem.numel() >= bytes) return;
    mem = at::Tensor();
    if (keep_) bytes = (bytes + ((size_t)1 << 20)) & ~(((size_t)1 << 20) - 1);
    mem = at::empty({(int64_t)bytes}, at::TensorOptions().dtype(at::kByte).device(stream.device()));
  }
  ~Workspace() {
    if (!keep_ || !mem.defined()) return;
    at::Tensor old;                       // (freed behind the lock)
    std::lock_guard<std::mutex> lock(g_mutex);
    Slab& slab = g_slabs[key_];
    if (!slab.mem.defined() || slab.mem.numel() < mem.numel()) {
      old = std::move(slab.mem);
      slab.mem = mem;
    }
    slab.used = ++g_tick;
    if (g_slabs.size() > kMaxSlabs) {
      auto oldest = g_slabs.begin();
      for (auto it = g_slabs.begin(); it != g_slabs.end(); ++it)
        if (it->second.used < oldest->second.used) oldest = it;
      old = std::move(oldest->second.mem);
      g_slabs.erase(oldest);
    }
  }
  Workspace(const Workspace&) = delete;
  at::Tensor mem;

 private:
  const std::pair<int, int64_t> key_;
  const bool keep_;
};

// Other Python threads run while a call launches (a launch waits when the stream's queue is full, and what
// it waits for may need a Python thread); back in for a hook, for Python objects and when an error leaves.
class WithoutGil {
 public:
  WithoutGil() : state_(PyEval_SaveThread()) {}
  ~WithoutGil() { end(); }
  void end() {
    if (state_ != nullptr) PyEval_RestoreThread(state_);
    state_ = nullptr;
  }
  void begin() { state_ = PyEval_SaveThread(); }

 private:
  PyThreadState* state_;
};

// Offsets into a workspace whose size is known once everything has been laid out.
struct Layout {
  size_t end = 0;
  size_t take(size_t bytes) {
    const size_t at = end;
    end += (bytes + 255) & ~(size_t)255;
    return at;
  }
};

b200moe_dtype dtype16(at::ScalarType t, const char* what) {
  if (t == at::kBFloat16) return B200MOE_BF16;
  if (t == at::kHalf) return B200MOE_F16;
  TORCH_CHECK(false, what, " must be bfloat16 or float16");
  return B200MOE_BF16;
}

// A layer's weights as the library reads them.  Checked by every call: a tensor of the plan may have got
// other contents, sizes or memory meanwhile.
struct Weights {
  WeightDesc d13, d2;
  bool i4;                    // int4 weights whose shapes the block-scaled kernel takes (gemm_tc_i4.cu)
};
Weights describe(const Plan& p, int64_t hidden, at::ScalarType out_dtype) {
  const at::ScalarType a = (p.block_fp8 || p.mx) ? at::kFloat8_e4m3fn : out_dtype;
  const int64_t k2 = p.inter * p.inter_scale;
  Weights w;
  w.d13 = describe_weights(p.w13, p.s13, 2 * p.inter, hidden, p.experts, 0, a);
  w.d2 = describe_weights(p.w2, p.s2, hidden, k2, p.experts, 0, a);
  for (const auto* b : {&p.b13, &p.b2}) {
    if (!b->has_value()) continue;
    TORCH_CHECK((*b)->dim() == 2, "ptr_bias must be 2D [num_experts, N]");
    TORCH_CHECK((*b)->is_contiguous(), "ptr_bias must be contiguous");
    TORCH_CHECK((*b)->size(0) == p.experts, "ptr_bias.size(0) must match num_experts");
    TORCH_CHECK((*b)->size(1) == (b == &p.b13 ? 2 * p.inter : hidden), "ptr_bias.size(1) must match N");
    TORCH_CHECK((*b)->scalar_type() == out_dtype, "ptr_bias must have ptr_D's dtype");
  }
  auto i4_ok = [](const WeightDesc& d, int64_t k) {
    return d.format == B200MOE_W_INT4_NK && (d.group == 128 || d.group == 256) && k % 128 == 0;
  };
  w.i4 = i4_ok(w.d13, hidden) && i4_ok(w.d2, k2);
  return w;
}

// What a call brings along besides its tensors.
struct CallOptions {
  int form = kUnfused;
  int64_t rows_hint = 0;
  int max_ctas = 0;
  PyObject* hook = nullptr;   // called with a stage's name after it has been launched
};
void mark(const CallOptions& o, WithoutGil& gil, const char* stage) {
  if (o.hook == nullptr) return;
  gil.end();
  PyObject* r = PyObject_CallFunction(o.hook, "s", stage);
  if (r == nullptr) throw python_error();
  Py_DECREF(r);
  gil.begin();
}

// gemm1 (+ activation) and gemm2 on expert-major rows.
struct Experts {
  const Plan& p;
  const Weights& weights;
  const CallOptions& o;
  WithoutGil& gil;
  b200moe_dtype out;          // 16-bit type between the stages
  at::ScalarType out_scalar;
  int64_t M, hidden;
  int segments;               // row segments (a multiple of the experts)
  int device;
  b200moe_stream stream;
  bool a_fp8;                 // gemm1's rows are e4m3 with 1x128 scales
  bool planes_in;             // ... or e4m3 planes with one scale per 32 values
  int planes;
  bool sums;                  // ... and the sums of their 128-wide blocks behind the scales (int4 weights)
  int64_t inter2() const { return p.inter * p.inter_scale; }
  // offsets
  size_t g1 = 0, act = 0, act_q = 0, act_s = 0;

  void lay_out(Layout& l) {
    if (o.form == kUnfused) g1 = l.take(M * 2 * p.inter * 2);
  }
  void lay_out_second(Layout& l) {
    const int64_t I = p.inter, I2 = o.form == kUnfused ? inter2() : I;
    const bool direct_fp8 = p.block_fp8 && (o.form == kFp8 || (p.act == kSilu && I % 128 == 0));
    if (!direct_fp8 && !gated_quant() && !planes_out()) act = l.take(M * I2 * 2);
    if (p.block_fp8) {
      act_q = l.take(M * I2);
      act_s = l.take(M * (I2 / 128) * 4);
    } else if (planes_in) {
      act_q = l.take((size_t)planes * M * I2);
      act_s = l.take((size_t)(planes + (sums ? 1 : 0)) * ((I2 + 127) / 128) * M * 4);
    }
  }
  // SiLU, multiply and the planes of gemm2's input in one pass
  bool gated_quant() const { return planes_in && o.form == kUnfused && p.act == kSilu && p.inter % 32 == 0; }

  // gemm1's SwigluOAI epilogue writes the planes of gemm2's input.  That saves a launch in the chain of a small decode
  // step; with many tiles a CTA its epilogue warps take more time from the other roles than the quantiser's launch
  // costs.  Layer calls in a row, quantiser / so, us: 128 experts of 2880 x 2880, top 4, 1 token 39.7 / 37.1, 4 tokens 69.5 /
  // 67.5, 8 tokens 106.6 / 105.7, 16 tokens 174.9 / 174.9, 2048 tokens 768 / 813 (bursts: 32 tokens 232.8 / 233.7, 64 tokens
  // 297.4 / 300.5, 512 tokens 427 / 457); 32 such experts 16 tokens 105.3 / 103.8, with very uneven routing 56.6 / 54.4; 8 of
  // 4096 x 6144, top 2, 8 and 32 tokens 83.5 / 81.9 and 89.9 / 88.6; 16 of 1024 x 512, 32 tokens 23.6 / 22.7.
  // (Only token tiles of 16 have it, which experts with 8 rows or fewer on average take.)
  static constexpr int64_t kPlanesOutRows = 64;
  bool planes_out() const {
    return planes_in && !sums && o.form == kEpilogue && p.act == kSwigluOai && p.inter % 32 == 0 &&
           M <= std::min<int64_t>(kPlanesOutRows, 8 * p.experts);
  }

  void gemm(bool first, const void* a, b200moe_dtype a_dtype, const void* a_scale, void* d, b200moe_dtype d_dtype,
            void* d_scale, const int32_t* rows, b200moe_epilogue epi) const {
    b200moe_gemm_args g = {};
    const WeightDesc& w = first ? weights.d13 : weights.d2;
    const at::Tensor& wt = first ? p.w13 : p.w2;
    const auto& sc = first ? p.s13 : p.s2;
    const auto& bias = first ? p.b13 : p.b2;
    g.a = a; g.a_dtype = a_dtype; g.a_scale = a_scale;
    g.w = wt.data_ptr(); g.w_format = w.format; g.group_size = w.group;
    g.w_scale = sc.has_value() ? sc->data_ptr() : nullptr;
    g.bias = bias.has_value() ? bias->data_ptr() : nullptr;
    g.d = d; g.d_dtype = d_dtype; g.d_scale = (float*)d_scale; g.mid_dtype = out;
    g.rows_per_expert = rows;
    g.m = M; g.n = (int)(first ? 2 * p.inter : hidden); g.k = (int)(first ? hidden : inter2());
    g.num_experts = segments;
    g.w_experts = segments != p.experts ? (int)p.experts : 0;
    g.epilogue = epi;
    g.act_alpha = 1.702f; g.act_limit = 7.0f;
    g.clamp_limit = epi != B200MOE_EPI_NONE && p.clamp > 0 ? (float)p.clamp : 0.f;
    g.status = device_status_word(device);
    g.max_ctas = o.max_ctas; g.rows_hint = o.rows_hint;
    g.rows_ready = !first;   // gemm1 has waited for them
    check_status(b200moe_grouped_gemm(&g, stream));
  }

  void run(uint8_t* ws, const void* a, const void* a_scale, const int32_t* rows, void* d) const {
    const int64_t I = p.inter, I2 = inter2();
    const b200moe_dtype mx_dtype =
        sums ? (planes == 3 ? B200MOE_FP8_E4M3_X3_EVENS_FIRST : B200MOE_FP8_E4M3_X2_EVENS_FIRST) :
        planes == 2 ? B200MOE_FP8_E4M3_X2 : B200MOE_FP8_E4M3;
    const int terms = planes + (sums ? B200MOE_PLANES_EVENS_FIRST : 0);
    const b200moe_dtype a_dtype = a_fp8 ? B200MOE_FP8_E4M3 : planes_in ? mx_dtype : out;
    bool fp8_ready = false, planes_ready = false;
    if (o.form == kFp8) {
      gemm(true, a, a_dtype, a_scale, ws + act_q, B200MOE_FP8_E4M3, ws + act_s, rows, B200MOE_EPI_SILU_MUL);
      mark(o, gil, "gemm1");
      fp8_ready = true;
    } else if (planes_out()) {
      gemm(true, a, a_dtype, a_scale, ws + act_q, mx_dtype, ws + act_s, rows, B200MOE_EPI_SWIGLUOAI);
      mark(o, gil, "gemm1");
      planes_ready = true;
    } else if (o.form == kEpilogue) {
      gemm(true, a, a_dtype, a_scale, ws + act, out, nullptr, rows,
           p.act == kSilu ? B200MOE_EPI_SILU_MUL : B200MOE_EPI_SWIGLUOAI);
      mark(o, gil, "gemm1");
    } else {
      gemm(true, a, a_dtype, a_scale, ws + g1, out, nullptr, rows, B200MOE_EPI_NONE);
      mark(o, gil, "gemm1");
      if (p.clamp > 0) {
        at::Tensor t = at::from_blob(ws + g1, {M, 2 * I},
                                     at::TensorOptions().dtype(out_scalar).device(at::kCUDA, device));
        t.narrow(1, 0, I).clamp_max_(p.clamp);
        t.narrow(1, I, I).clamp_(-p.clamp, p.clamp);
      }
      if (p.block_fp8 && p.act == kSilu && I % 128 == 0) {
        // SiLU, multiply and the 1x128 e4m3 quantisation of gemm2's input in one pass over the rows
        // that the experts' segments use (the buffers may be sized for a worst case)
        check_status(b200moe_silu_and_mul_per_block_quant_ragged(ws + act_q, (float*)(ws + act_s), ws + g1, out, M,
                                                                 (int)I, rows, segments, stream));
        fp8_ready = true;
      } else if (gated_quant()) {
        check_status(b200moe_quant_mxfp8_ex(ws + g1, out, ws + act_q, ws + act_s, M, (int)I, terms, sums, 1, stream));
        planes_ready = true;
      } else {
        void *to = ws + act, *from = ws + g1;
        switch (p.act) {
          case kSilu: check_status(b200moe_silu_and_mul(to, from, out, M, (int)I, stream)); break;
          case kGelu: check_status(b200moe_gelu_and_mul(to, from, out, M, (int)I, stream)); break;
          case kGeluTanh: check_status(b200moe_gelu_tanh_and_mul(to, from, out, M, (int)I, stream)); break;
          case kSwigluOai:
            check_status(b200moe_swigluoai_and_mul(to, from, out, M, (int)I, 1.702f, 7.0f, stream)); break;
          case kRelu2NoMul: check_status(b200moe_relu2_no_mul(to, from, out, M, (int)I2, stream)); break;
          default: check_status(b200moe_swiglustep_and_mul(to, from, out, M, (int)I, 7.0f, stream)); break;
        }
      }
    }
    mark(o, gil, "activation");
    if (p.block_fp8) {
      if (!fp8_ready)
        check_status(b200moe_per_token_group_fp8_quant(ws + act, out, ws + act_q, (float*)(ws + act_s), M, (int)I2, 128,
                                                       1e-10f, 0, I2 / 128, 1, stream));
      gemm(false, ws + act_q, B200MOE_FP8_E4M3, ws + act_s, d, out, nullptr, rows, B200MOE_EPI_NONE);
    } else if (planes_in) {
      if (!planes_ready)
        check_status(b200moe_quant_mxfp8_ex(ws + act, out, ws + act_q, ws + act_s, M, (int)I2, terms, sums, 0, stream));
      gemm(false, ws + act_q, mx_dtype, ws + act_s, d, out, nullptr, rows, B200MOE_EPI_NONE);
    } else {
      gemm(false, ws + act, out, nullptr, d, out, nullptr, rows, B200MOE_EPI_NONE);
    }
    mark(o, gil, "gemm2");
  }
};

const at::Tensor& tensor_arg(PyObject* o, const char* name) {
  TORCH_CHECK_TYPE(THPVariable_Check(o), name, " must be a tensor");
  return THPVariable_Unpack(o);
}
std::optional<at::Tensor> optional_arg(PyObject* o, const char* name) {
  if (o == Py_None) return std::nullopt;
  return tensor_arg(o, name);
}
int64_t int_arg(PyObject* o) {
  const int64_t v = PyLong_AsLongLong(o);
  if (v == -1 && PyErr_Occurred()) throw python_error();
  return v;
}
Plan* plan_arg(PyObject* o) {
  Plan* p = (Plan*)PyCapsule_GetPointer(o, kPlanName);
  if (p == nullptr) throw python_error();
  return p;
}
void need_cuda(const at::Tensor& t, const char* name) {
  TORCH_CHECK_NOT_IMPLEMENTED(t.is_cuda(), name, " must be a CUDA tensor: the layer has no CPU path");
}

void free_plan(PyObject* capsule) {
  delete (Plan*)PyCapsule_GetPointer(capsule, kPlanName);
  bool last;
  { std::lock_guard<std::mutex> lock(g_mutex); last = --g_plans == 0; }
  if (last) clear_slabs();
}

// layer_plan(w13, s13, b13, w2, s2, b2, inter, topk, experts, total_experts, act, inter_scale,
//            block_fp8, mx, planes, clamp)
PyObject* layer_plan(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  TORCH_CHECK(n == 16, "layer_plan takes 16 arguments");
  auto p = std::make_unique<Plan>();
  p->w13 = tensor_arg(a[0], "w13"); p->s13 = optional_arg(a[1], "w13_scales"); p->b13 = optional_arg(a[2], "w13_bias");
  p->w2 = tensor_arg(a[3], "w2"); p->s2 = optional_arg(a[4], "w2_scales"); p->b2 = optional_arg(a[5], "w2_bias");
  p->inter = int_arg(a[6]); p->topk = (int)int_arg(a[7]); p->experts = int_arg(a[8]); p->total_experts = int_arg(a[9]);
  p->act = (int)int_arg(a[10]); p->inter_scale = (int)int_arg(a[11]);
  p->block_fp8 = int_arg(a[12]) != 0; p->mx = int_arg(a[13]) != 0; p->planes = (int)int_arg(a[14]);
  p->clamp = PyFloat_AsDouble(a[15]);
  if (PyErr_Occurred()) throw python_error();
  PyObject* capsule = PyCapsule_New(p.get(), kPlanName, free_plan);
  if (capsule == nullptr) throw python_error();
  p.release();
  std::lock_guard<std::mutex> lock(g_mutex);
  ++g_plans;
  return capsule;
  END_HANDLE_TH_ERRORS
}

// layer_run(plan, form, output | None, hidden, topk_weights, topk_ids, expert_map | None, a1q_scale | None,
//           rows_hint, max_ctas, persistent, hook | None, out_dtype | None)
// With output None the reduction is left to the caller: returns (rows [T*K, hidden], row map [T, K]),
// valid until the next layer call on the stream.
PyObject* layer_run(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  TORCH_CHECK(n == 13, "layer_run takes 13 arguments");
  const Plan& p = *plan_arg(a[0]);
  CallOptions o;
  o.form = (int)int_arg(a[1]);
  o.rows_hint = int_arg(a[8]);
  o.max_ctas = (int)int_arg(a[9]);
  o.hook = a[11] == Py_None ? nullptr : a[11];
  const bool gather = a[2] != Py_None;
  const at::Tensor& x = tensor_arg(a[3], "hidden_states");
  const at::Tensor& ids = tensor_arg(a[5], "topk_ids");
  const std::optional<at::Tensor> map = optional_arg(a[6], "expert_map"), a1q = optional_arg(a[7], "a1q_scale");
  need_cuda(x, "hidden_states");
  TORCH_CHECK(x.dim() == 2, "hidden_states must be [num_rows, hidden_size]");
  const int64_t T = x.size(0), H = x.size(1), K = p.topk, M = T * K;
  at::ScalarType od = x.scalar_type();
  if (gather) od = tensor_arg(a[2], "output").scalar_type();
  else if (a[12] != Py_None) od = ((THPDtype*)a[12])->scalar_type;
  TORCH_CHECK_NOT_IMPLEMENTED(!(a1q.has_value() && x.scalar_type() != od && !p.block_fp8),
              // The reference forwards caller-quantised activations and their scales to gemm1 for
              // every recipe; here only the block-scaled fp8 kernels take them (1x128 fp32 scales).
              "a1q_scale with pre-quantised hidden_states is built for block-scaled fp8 weights only; "
              "pass 16-bit hidden_states instead");
  const b200moe_dtype out = dtype16(od, "ptr_D");
  if (map.has_value()) {
    TORCH_CHECK(map->scalar_type() == at::kInt, "expert_map must be int32");
    TORCH_CHECK(map->size(0) == p.total_experts, "expert_map must be [total_experts_num]");
  }
  TORCH_CHECK(ids.scalar_type() == at::kLong || ids.scalar_type() == at::kInt, "topk_ids must be int64 or int32");
  TORCH_CHECK(ids.dim() == 2 && ids.size(0) == T && ids.size(1) == K, "topk_ids must be [num_rows, TopK]");
  TORCH_CHECK(x.is_contiguous() && ids.is_contiguous(), "remap_hidden_states expects contiguous tensors");
  if (p.experts > 1024) throw std::runtime_error("local_experts_num exceeds the maximum supported number");
  if (a1q.has_value()) {
    TORCH_CHECK(a1q->is_contiguous() && a1q->dim() == 2, "remap_hidden_states expects contiguous scales");
    TORCH_CHECK(a1q->size(0) >= T, "hidden_states_scales must be [num_rows, hidden_size // block_k]");
    const bool rows_fp8 = p.block_fp8 && x.scalar_type() == at::kFloat8_e4m3fn;   // gemm1 reads the scales as they are
    TORCH_CHECK(!rows_fp8 || (a1q->scalar_type() == at::kFloat && a1q->size(1) == H / 128),
                "ptr_A_scale must be float32 [Total_M, K / 128]");
    TORCH_CHECK(rows_fp8 || x.scalar_type() == od, "ptr_A and ptr_D must have the same dtype");
  }
  if (gather) {
    const at::Tensor& y = tensor_arg(a[2], "output");
    const at::Tensor& w = tensor_arg(a[4], "topk_weights");
    TORCH_CHECK(w.scalar_type() == at::kFloat, "topk_weights must be float32");
    TORCH_CHECK(y.is_cuda() && w.is_cuda() && y.is_contiguous() && w.is_contiguous(),
                "moe_gather expects contiguous tensors");
    TORCH_CHECK(y.dim() == 2 && y.size(0) == T && y.size(1) == H && w.numel() == M,
                "output must be [num_rows, hidden_size], topk_weights [num_rows, TopK]");
  }
  const c10::cuda::CUDAGuard guard(x.device());
  const auto stream = at::cuda::getCurrentCUDAStream();
  const b200moe_stream st = (b200moe_stream)stream.stream();
  const Weights weights = describe(p, H, od);
  raise_if_timed_out(device_status_word(x.get_device()));   // an earlier call on this device gave up a wait
  if (o.rows_hint == 0 && map.has_value() && p.total_experts > p.experts)
    o.rows_hint = std::max<int64_t>(1, M * p.experts / p.total_experts);   // the other ranks' share is masked
  const bool quant_fp8 = p.block_fp8 && !a1q.has_value();
  // (the block-scaled int4 kernel has no activation in its epilogue)
  const bool i4 = weights.i4 && o.form == kUnfused &&
                  (o.rows_hint > 0 && o.rows_hint < M ? o.rows_hint : M) <= Plan::kI4PlaneRows * p.experts;
  const bool planes_in = p.mx || i4;
  const int planes = i4 ? (od == at::kHalf ? 3 : 2) : p.planes;   // exact for the 16-bit type
  if (!p.mx && !p.block_fp8)
    TORCH_CHECK(x.scalar_type() == od, "ptr_A and ptr_D must have the same dtype");
  // (16-bit rows with caller-made scales: the scales are permuted and left unused)
  const bool a_fp8 = quant_fp8 || (p.block_fp8 && x.scalar_type() == at::kFloat8_e4m3fn);
  const at::Tensor* y = gather ? &THPVariable_Unpack(a[2]) : nullptr;
  const at::Tensor* w = gather ? &THPVariable_Unpack(a[4]) : nullptr;
  WithoutGil gil;
  mark(o, gil, "routing");
  Experts e{p, weights, o, gil, out, od, M, H, (int)p.experts, (int)x.get_device(), st, a_fp8, planes_in, planes, i4};
  Layout l;
  const size_t rows_at = l.take(p.experts * 4), map_at = l.take(M * 4);
  const size_t sort_bytes = b200moe_sort_workspace_bytes(M, (int)p.experts);
  const size_t sort_at = l.take(sort_bytes);
  const size_t a_at = l.end;
  size_t as_at = a_at;
  if (quant_fp8) {
    l.take(M * H);
    as_at = l.take(M * (H / 128) * 4);
  } else if (planes_in) {
    l.take((size_t)planes * M * H);
    as_at = l.take((size_t)(planes + (i4 ? 1 : 0)) * ((H + 127) / 128) * M * 4);
  } else {
    l.take(M * H * x.element_size());
    if (a1q.has_value()) as_at = l.take(M * a1q->size(1) * a1q->element_size());
  }
  e.lay_out(l);
  // gemm2's rows take the place of gemm1's operands (and, unfused, of its output) where they fit
  size_t d_at = a_at;
  if (l.end - a_at < (size_t)M * H * 2) d_at = l.take(M * H * 2);
  e.lay_out_second(l);
  const Workspace workspace(stream, l.end, a[10] == Py_True);
  uint8_t* ws = workspace.mem.data_ptr<uint8_t>();
  int32_t *rows = (int32_t*)(ws + rows_at), *row_map = (int32_t*)(ws + map_at);
  const int32_t* emap = map.has_value() ? map->data_ptr<int32_t>() : nullptr;
  if (quant_fp8)
    check_status(b200moe_remap_quant_fp8(x.data_ptr(), float_dtype(x, "b200_remap_quant_fp8"), ws + a_at,
                                         (float*)(ws + as_at), emap, rows, row_map, ids.data_ptr(), index_dtype(ids), T,
                                         (int)H, (int)K, (int)p.total_experts, (int)p.experts, ws + sort_at, sort_bytes,
                                         st));
  else if (planes_in)
    check_status(b200moe_remap_quant_mxfp8(x.data_ptr(), float_dtype(x, "hidden_states"), ws + a_at, ws + as_at,
                                           planes + (i4 ? B200MOE_PLANES_EVENS_FIRST : 0), i4, emap, rows, row_map,
                                           ids.data_ptr(), index_dtype(ids), T, (int)H, (int)K, (int)p.total_experts,
                                           (int)p.experts, ws + sort_at, sort_bytes, st));
  else
    check_status(b200moe_remap_hidden_states(
        x.data_ptr(), a1q.has_value() ? a1q->data_ptr() : nullptr, ws + a_at, a1q.has_value() ? ws + as_at : nullptr,
        emap, rows, row_map, ids.data_ptr(), index_dtype(ids), T, (int)H, (int)x.element_size(),
        a1q.has_value() ? (int)a1q->size(1) : 0, a1q.has_value() ? (int)a1q->element_size() : 0, (int)K,
        (int)p.total_experts, (int)p.experts, ws + sort_at, sort_bytes, st));
  mark(o, gil, "permute");
  e.run(ws, ws + a_at, (a_fp8 || planes_in) ? ws + as_at : nullptr, rows, ws + d_at);
  if (gather) {
    check_status(b200moe_moe_gather(y->data_ptr(), ws + d_at, w->data_ptr<float>(), row_map, out, T, (int)H, (int)K, st));
    mark(o, gil, "gather");
    gil.end();
    Py_RETURN_NONE;
  }
  gil.end();
  auto view = [&](size_t at, int64_t r, int64_t c, at::ScalarType t) {
    return workspace.mem.narrow(0, (int64_t)at, r * c * (int64_t)c10::elementSize(t)).view(t).view({r, c});
  };
  PyObject* rows_out = THPVariable_Wrap(view(d_at, M, H, od));
  PyObject* map_out = THPVariable_Wrap(view(map_at, T, K, at::kInt));
  return Py_BuildValue("(NN)", rows_out, map_out);
  END_HANDLE_TH_ERRORS
}

// layer_experts(plan, form, output_rows, rows, rows_per_segment, a_scale | None, rows_hint, max_ctas,
//               persistent, hook | None): gemm1, activation and gemm2 on rows that are grouped already.
PyObject* layer_experts(PyObject*, PyObject* const* a, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  TORCH_CHECK(n == 10, "layer_experts takes 10 arguments");
  const Plan& p = *plan_arg(a[0]);
  CallOptions o;
  o.form = (int)int_arg(a[1]);
  o.rows_hint = int_arg(a[6]);
  o.max_ctas = (int)int_arg(a[7]);
  o.hook = a[9] == Py_None ? nullptr : a[9];
  const at::Tensor &y = tensor_arg(a[2], "output_rows"), &x = tensor_arg(a[3], "rows"),
                   &rows = tensor_arg(a[4], "rows_per_segment");
  const std::optional<at::Tensor> scale = optional_arg(a[5], "a1q_scale");
  need_cuda(x, "rows");
  const int64_t M = x.size(0), H = x.size(1), segments = rows.numel();
  TORCH_CHECK(x.dim() == 2 && y.dim() == 2 && y.size(0) == M && y.size(1) == H, "ptr_A.size(0) must match ptr_D.size(0)");
  TORCH_CHECK(x.is_contiguous() && y.is_contiguous(), "ptr_A must be contiguous");
  TORCH_CHECK(rows.scalar_type() == at::kInt && rows.is_contiguous() && segments > 0 && segments % p.experts == 0,
              "rows_per_expert must be int32 [num_experts]");
  const b200moe_dtype out = dtype16(y.scalar_type(), "ptr_D");
  if (p.block_fp8) {
    TORCH_CHECK(scale.has_value() && x.scalar_type() == at::kFloat8_e4m3fn && scale->scalar_type() == at::kFloat &&
                    scale->is_contiguous() && scale->dim() == 2 && scale->size(0) == M && scale->size(1) == H / 128,
                "ptr_A_scale must be float32 [Total_M, K / 128]");
  } else {
    TORCH_CHECK(x.scalar_type() == y.scalar_type(), "ptr_A and ptr_D must have the same dtype");
  }
  const c10::cuda::CUDAGuard guard(x.device());
  const auto stream = at::cuda::getCurrentCUDAStream();
  const Weights weights = describe(p, H, y.scalar_type());
  raise_if_timed_out(device_status_word(x.get_device()));
  WithoutGil gil;
  Experts e{p, weights, o, gil, out, y.scalar_type(), M, H, (int)segments, (int)x.get_device(),
            (b200moe_stream)stream.stream(), p.block_fp8, false, 0};
  Layout l;
  e.lay_out(l);
  e.lay_out_second(l);
  const Workspace workspace(stream, l.end, a[8] == Py_True);
  e.run(workspace.mem.data_ptr<uint8_t>(), x.data_ptr(), scale.has_value() ? scale->data_ptr() : nullptr,
        rows.data_ptr<int32_t>(), y.data_ptr());
  gil.end();
  Py_RETURN_NONE;
  END_HANDLE_TH_ERRORS
}

PyObject* workspace_clear(PyObject*, PyObject*) {
  HANDLE_TH_ERRORS
  clear_slabs();
  Py_RETURN_NONE;
  END_HANDLE_TH_ERRORS
}

}  // namespace

PyMethodDef* layer_methods() {
  static PyMethodDef methods[] = {
      {"layer_plan", (PyCFunction)(void (*)(void))layer_plan, METH_FASTCALL, nullptr},
      {"layer_run", (PyCFunction)(void (*)(void))layer_run, METH_FASTCALL, nullptr},
      {"layer_experts", (PyCFunction)(void (*)(void))layer_experts, METH_FASTCALL, nullptr},
      {"workspace_clear", workspace_clear, METH_NOARGS, nullptr},
      {nullptr, nullptr, 0, nullptr}};
  return methods;
}

}  // namespace b200shim

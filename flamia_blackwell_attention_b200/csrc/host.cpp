// Host path of the attention call in native code: the CUDA and autograd implementations of the registered ops
// lowbit_attn::fp8 / ::fp4 (+ _bwd), and the entry the Python API calls with a resolved plan. What one call launches,
// forward and backward (the launch sequence of the reference's flash_attn/cute/lowprec/_routes.py, _fp8_forward_mx :709,
// _fp8_backward_mx :911, _e4pv_forward_blk32 :308, run_documents :1388):
//
//   forward   1 quantiser launch (Q, K [rotated], V) + 1 forward kernel
//   backward  1 fused prologue (dO quantiser + D + shifted LSE + zeroed accumulator) + 1 pre-scale + 1 main kernel
//             + 1 dQ postprocess
//   also      packed documents: the work lists before the forward, with cu_seqlens the tables before the quantiser, with return_lse
//             the LSE's way back (a zero fill and a launch); per-token scales: a quantiser launch per operand and V's tables;
//             per-row pre-scale, ordered dQ: zero fills of their tables, copies of the statistics
//
// Why native: the same sequence in Python (ctypes structures, a Python autograd node, one tensor object per table) held a
// small call (b1 s512 h4 d64, forward and backward) at 600 us of host time for about 60 us of kernels. No host
// synchronisation anywhere; everything is enqueued on the current stream of the inputs' device. The functions here hold no
// state but the plan and entry registries (append-only, under a lock) and one status word per device, so calls from several
// threads and streams are independent.
#include <ATen/ATen.h>
#include <ATen/cuda/EmptyTensor.h>
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <cuda_runtime_api.h>
#include <torch/csrc/autograd/custom_function.h>
#include <torch/csrc/autograd/python_variable.h>
#include <torch/csrc/utils/pybind.h>
#include <torch/library.h>

#include <algorithm>
#include <cstdlib>
#include <cstring>
#include <deque>
#include <map>
#include <mutex>
#include <sstream>
#include <tuple>

#include "../../include/flamia_b200.h"

namespace {

using at::Tensor;
using torch::autograd::variable_list;

constexpr double kPShiftLog2 = 8.0;     // the backward recomputes P' = 2^8 P (its E4M3 P-hat then uses the normal range)
constexpr int kDevWaitTimeout = 0x100, kDevBadTable = 0x200;

// ---------------------------------------------------------------------------------------------------- plans and entries
// The numbers of one resolved plan (plan.py::AttnPlan) that the launches need.
struct Plan {
  bool fp4, token_local, hadamard, causal, need_bwd, p_group, seqused_k, varlen, aligned, ragged, return_lse, deterministic,
      rowlocal;
  int prescale;              // 0 = one per batch row, 1 = causal per query tile, 2 = causal per query row
  int window_left_p1, window_right_p1;
  double softcap, softmax_scale;
  int64_t b, s_q, s_k, h, h_kv, d, tot_q;
  int64_t d_call;            // the call's own head dim: d, or less where the kernels run it with zero columns up to d
};
struct Entry {
  int64_t plan, capacity;    // capacity < 0: the batched form
  bool aligned;
};
std::mutex g_lock;
std::deque<Plan> g_plans;    // (a deque: references stay valid while others are added)
std::deque<Entry> g_entries;
std::map<std::tuple<int64_t, int64_t, bool>, int64_t> g_entry_ids;

const Plan& plan_at(int64_t i) {
  std::lock_guard<std::mutex> g(g_lock);
  TORCH_CHECK(i >= 0 && i < (int64_t)g_plans.size(), "unknown plan handle ", i);
  return g_plans[(size_t)i];
}
Entry entry_at(int64_t i) {
  std::lock_guard<std::mutex> g(g_lock);
  TORCH_CHECK(i >= 0 && i < (int64_t)g_entries.size(), "unknown backward entry ", i);
  return g_entries[(size_t)i];
}
int64_t entry_of(int64_t plan, int64_t capacity, bool aligned) {
  std::lock_guard<std::mutex> g(g_lock);
  const auto key = std::make_tuple(plan, capacity, aligned);
  auto it = g_entry_ids.find(key);
  if (it != g_entry_ids.end()) return it->second;
  const int64_t id = (int64_t)g_entries.size();
  g_entries.push_back({plan, capacity, aligned});
  g_entry_ids.emplace(key, id);
  return id;
}

void check(int rc, const char* what) {
  if (rc == 0) return;
  static const char* names[] = {"", "bad argument", "CUDA error", "unsupported configuration", "size beyond the supported maximum"};
  char detail[256] = "";
  if (rc == 2) fl_last_cuda_error(detail, 256);
  TORCH_CHECK(false, what, " failed: ", rc >= 1 && rc <= 4 ? names[rc] : "?", " (code ", rc, ")", rc == 2 ? ": " : "", detail);
}

// ---------------------------------------------------------------------------------------------------- status words
// Every device-side wait of the kernels is bounded; one that runs out writes 0x100 | site into the call's status word and
// the kernel drains, leaving its outputs partly written. One persistent word per device, zeroed when it is made and again
// once a code has been reported (kernels only ever write it when something went wrong), so a call launches no fill kernel.
// Reading it costs a host synchronisation: only check_status() does it, and every call while FLAMIA_B200_CHECK_STATUS=1.
constexpr int kMaxDevices = 64;
std::mutex g_status_lock;
// (never destroyed: at process exit the allocator that owns them may be gone already)
Tensor* const g_status = new Tensor[kMaxDevices];
Tensor* const g_last_status = new Tensor[kMaxDevices];

Tensor new_status(at::Device dev) { return at::zeros({1}, at::TensorOptions().dtype(at::kInt).device(dev)); }

Tensor status_word(at::Device dev) {
  std::lock_guard<std::mutex> g(g_status_lock);
  TORCH_CHECK(dev.index() >= 0 && dev.index() < kMaxDevices, "device index ", (int)dev.index());
  Tensor& st = g_status[dev.index()];
  if (!st.defined()) {
    cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
    C10_CUDA_CHECK(cudaStreamIsCapturing(c10::cuda::getCurrentCUDAStream(dev.index()), &cap));
    // a first call made inside a stream capture gets a word of the capture's own
    if (cap != cudaStreamCaptureStatusNone) return g_last_status[dev.index()] = new_status(dev);
    st = new_status(dev);
  }
  return g_last_status[dev.index()] = st;
}

int64_t check_status(int64_t idx) {
  Tensor st;
  {
    std::lock_guard<std::mutex> g(g_status_lock);
    if (idx < 0 || idx >= kMaxDevices || !g_last_status[idx].defined()) return 0;
    st = g_last_status[idx];
  }
  const c10::cuda::CUDAGuard guard((c10::DeviceIndex)idx);
  int32_t code = 0;
  check(fl_read_status(st.const_data_ptr<int32_t>(), &code, c10::cuda::getCurrentCUDAStream((c10::DeviceIndex)idx).stream()),
        "fl_read_status");
  if (code == 0) return 0;
  st.zero_();
  std::ostringstream what;
  if (code & kDevWaitTimeout) what << "a bounded wait ran out at site " << (code & 0xFF);
  else if (code & kDevBadTable) what << "the document table is inconsistent (code 0x" << std::hex << code << ")";
  else what << "code 0x" << std::hex << code;
  TORCH_CHECK(false, "flamia_blackwell_attention_b200: an attention call on cuda:", idx, " did not complete: ", what.str(),
              "; its outputs are not valid");
}

void check_status_if_asked(at::Device dev) {
  const char* e = std::getenv("FLAMIA_B200_CHECK_STATUS");
  if (e && *e && std::strcmp(e, "0") != 0) check_status(dev.index());
}

// ---------------------------------------------------------------------------------------------------- tensors
Tensor empty(at::IntArrayRef sizes, at::ScalarType dt, at::Device dev) {
  return at::detail::empty_cuda(sizes, dt, dev, std::nullopt);
}
template <typename T>
T* ptr(const Tensor& t) {
  return t.defined() ? reinterpret_cast<T*>(const_cast<void*>(t.const_data_ptr())) : nullptr;
}
template <typename T>
T* ptr(void* p) {
  return reinterpret_cast<T*>(p);
}

// An operand's rows as the quantisers read them. Zero-padded head dims are served at any start address (they used to be copied for their
// zero columns); the tensor maps want 16-byte alignment, and an odd view is copied. The kernels' own head dims refuse it.
Tensor rows_of(const Plan& p, const Tensor& x) {
  const Tensor c = x.contiguous();
  return p.d_call != p.d && reinterpret_cast<uintptr_t>(c.const_data_ptr()) % 16 ? c.clone() : c;
}

// Temporaries of one call carved out of one allocation (256-byte aligned pieces): sizes first, pointers afterwards.
struct Workspace {
  size_t size = 0;
  Tensor buf;
  size_t piece(size_t bytes) {
    const size_t at = size;
    size += (bytes + 255) & ~size_t(255);
    return at;
  }
  void allocate(at::Device dev) { buf = empty({(int64_t)size}, at::kByte, dev); }
  void* at(size_t off) const { return static_cast<char*>(buf.data_ptr()) + off; }
};

// ---------------------------------------------------------------------------------------------------- documents
// Packed documents laid out at 128-aligned starts of one padded buffer of `capacity` rows (a host-known bound, so no device
// value is read). The quantisers read the packed rows in place through the slot tables (first source row and number of real
// rows of every 128-row slot), and the kernels write the caller's packed rows themselves. aligned: the caller's rows are
// the buffer's rows already.
struct Docs {
  Tensor start, len, row_map, slot_src, slot_rows, work;
  Tensor all;                // pooled: one buffer of the five tables
  int64_t capacity = 0;
  bool aligned = false;
  void split(int64_t n) {
    const auto parts = all.split_with_sizes({n, n, capacity, capacity / 128, capacity / 128});
    start = parts[0]; len = parts[1]; row_map = parts[2]; slot_src = parts[3]; slot_rows = parts[4];
  }
};

Docs docs_of(const Plan& p, const Tensor& q, at::TensorList t, bool pooled, cudaStream_t st) {
  Docs d;
  const auto dev = q.device();
  if (t.size() == 6) {                        // precomputed maps: cu, start, len, row_map, slot_src, slot_rows
    d.start = t[1]; d.len = t[2]; d.row_map = t[3]; d.slot_src = t[4]; d.slot_rows = t[5];
    d.capacity = t[3].numel();
    for (const Tensor& x : t) TORCH_CHECK(x.scalar_type() == at::kInt && x.is_contiguous(), "document maps are contiguous int32 tables");
    TORCH_CHECK(d.start.numel() == d.len.numel() && d.capacity % 128 == 0 && d.slot_src.numel() == d.capacity / 128 &&
                    d.slot_rows.numel() == d.capacity / 128,
                "document maps: start / len of one size, slot_src / slot_rows one entry per 128 rows of row_map");
    return d;
  }
  if (p.aligned) {
    TORCH_CHECK(t.size() == 4, "aligned documents: cu_seqlens_q, cu_seqlens_k, seqused_q, seqused_k");
    d.aligned = true;
    d.start = t[0].slice(0, 0, t[0].size(0) - 1).to(at::kInt).contiguous();
    d.len = t[2].to(at::kInt).contiguous();
    TORCH_CHECK(d.len.numel() == d.start.numel(), "aligned documents: one seqused entry per document");
    d.capacity = p.tot_q;
    return d;
  }
  // cu_seqlens: the tables in one launch
  TORCH_CHECK(t.size() >= 1, "packed documents: cu_seqlens");
  const int64_t n = t[0].size(0) - 1, total = p.tot_q;
  d.capacity = (total + 127 * n + 127) / 128 * 128;
  const int64_t slots = d.capacity / 128;
  if (pooled) {
    d.all = empty({2 * n + d.capacity + 2 * slots}, at::kInt, dev);
    d.split(n);
  } else {
    d.start = empty({n}, at::kInt, dev); d.len = empty({n}, at::kInt, dev); d.row_map = empty({d.capacity}, at::kInt, dev);
    d.slot_src = empty({slots}, at::kInt, dev); d.slot_rows = empty({slots}, at::kInt, dev);
  }
  const Tensor cu = t[0].to(at::kInt).contiguous();
  check(fl_doc_tables(ptr<int32_t>(cu), (int32_t)n, 0, (int32_t)total, (int32_t)d.capacity,
                      ptr<int32_t>(d.start), ptr<int32_t>(d.len), ptr<int32_t>(d.row_map), ptr<int32_t>(d.slot_src),
                      ptr<int32_t>(d.slot_rows), st),
        "fl_doc_tables");
  return d;
}

// ---------------------------------------------------------------------------------------------------- forward
struct Quantised {
  Tensor codes, fac, token_factors, x4, sf4, tile_stats;
  fl_quant_args args = {};
};

// Tensors of one call over one buffer: every tensor object of its own costs an allocator round trip of about half a microsecond, a
// view made directly a fifth of that. Two passes over the same requests: sizes first, then the tensors. Such tensors stay inside a
// call: what autograd saves is the buffer, and the registered op, whose outputs may not share memory, has tensors of their own.
class Pool {
 public:
  Pool() = default;
  Pool(Tensor buf, bool traced) : buf_(std::move(buf)), traced_(traced) {}       // a buffer made before (the same requests again)
  void add(at::IntArrayRef sizes, at::ScalarType dt) { size_ = round(size_ + bytes(sizes, dt)); }
  const Tensor& allocate(at::Device dev) { buf_ = empty({(int64_t)size_}, at::kByte, dev); size_ = 0; return buf_; }
  Tensor take(at::IntArrayRef sizes, at::ScalarType dt) {
    if (traced_) {
      Tensor t = buf_.narrow(0, (int64_t)size_, (int64_t)bytes(sizes, dt)).view(dt).view(sizes);
      size_ = round(size_ + bytes(sizes, dt));
      return t;
    }
    Tensor t = at::detail::make_tensor<c10::TensorImpl>(c10::Storage(buf_.storage()), buf_.key_set(), c10::scalarTypeToTypeMeta(dt));
    t.unsafeGetTensorImpl()->set_sizes_contiguous(sizes);
    t.unsafeGetTensorImpl()->set_storage_offset((int64_t)(size_ / c10::elementSize(dt)));
    size_ = round(size_ + bytes(sizes, dt));
    return t;
  }

 private:
  static size_t round(size_t n) { return (n + 255) & ~size_t(255); }
  static size_t bytes(at::IntArrayRef sizes, at::ScalarType dt) { return (size_t)c10::multiply_integers(sizes) * c10::elementSize(dt); }
  size_t size_ = 0;
  Tensor buf_;
  bool traced_ = false;      // through operators, for a program that records them
};

struct Shapes {            // the kernels' view of the call: one batch entry of `capacity` rows under documents, batch rows of whole tiles
  int64_t b, s_q, s_k;
};
Shapes shapes_of(const Plan& p, int64_t capacity) {
  return capacity >= 0 ? Shapes{1, capacity, capacity} : Shapes{p.b, (p.s_q + 127) / 128 * 128, (p.s_k + 127) / 128 * 128};
}

// The outputs of one operand's quantiser: `make` allocates (or sizes) a tensor.
template <typename Make>
void quantised_tensors(Quantised& o, const Plan& p, int64_t b, int64_t s, int64_t heads, bool scores, bool tile_stats, Make make) {
  const int64_t d = p.d;
  o.codes = make({b, s, heads, d}, at::kFloat8_e4m3fn);
  o.fac = make({b, heads, s / 32}, at::kFloat);
  if (p.token_local) o.token_factors = make({b, heads, s}, at::kFloat);
  if (scores && p.fp4) {
    o.x4 = make({b, s, heads, d / 2}, at::kByte);
    o.sf4 = make({b, heads, s / 128, d / 64, 32, 4, 4}, at::kByte);
  }
  if (tile_stats) o.tile_stats = make({b, heads, s / 128, 2}, at::kFloat);
}

void quantise_args(Quantised& o, const Plan& p, const Tensor& x, int64_t b, int64_t s, int64_t heads, bool scores, const Docs* docs,
                   const Tensor& row_stat, int row_stat_kind, int32_t* status) {
  fl_quant_args& a = o.args;
  a.x = ptr<void>(x);
  a.b = (int32_t)b; a.s = (int32_t)s; a.h = (int32_t)heads; a.d = (int32_t)p.d;
  a.in_f16 = x.scalar_type() == at::kHalf;
  // rotation: the 8-bit route rotates the E4M3 codes; the mixed route rotates only the NVFP4 S operands
  if (scores && p.hadamard) a.flags |= p.fp4 ? FL_Q_HADAMARD_NVFP4_ONLY : FL_Q_HADAMARD;
  if (p.token_local) a.flags |= FL_Q_TOKEN_LOCAL;
  if (p.d_call != p.d) a.flags |= FL_Q_COLS(p.d_call);
  a.codes = ptr<uint8_t>(o.codes); a.fac = ptr<float>(o.fac); a.token_factors = ptr<float>(o.token_factors);
  a.x4 = ptr<uint8_t>(o.x4); a.sf4 = ptr<uint8_t>(o.sf4); a.tile_stats = ptr<float>(o.tile_stats);
  if (docs && !docs->aligned) {
    a.slot_src = ptr<int32_t>(docs->slot_src); a.slot_rows = ptr<int32_t>(docs->slot_rows);
    a.src_rows = (int32_t)(x.numel() / (heads * p.d_call));
  } else if (p.ragged) {
    a.flags |= FL_Q_ROWS; a.src_rows = (int32_t)p.s_q;
  }
  if (row_stat.defined()) { a.row_stat = ptr<float>(row_stat); a.row_stat_kind = row_stat_kind; }
  a.status = status;
}

void attn_common(fl_attn_args& a, const Plan& p, const Shapes& sh, bool f16) {
  a.b = (int32_t)sh.b; a.s_q = (int32_t)sh.s_q; a.s_k = (int32_t)sh.s_k;
  a.h = (int32_t)p.h; a.h_kv = (int32_t)p.h_kv; a.d = (int32_t)p.d;
  a.softmax_scale = (float)p.softmax_scale;
  a.mode = p.fp4 ? FL_MODE_FP4 : FL_MODE_FP8;
  a.flags = (p.causal ? FL_A_CAUSAL : 0) | (f16 ? FL_A_OUT_F16 : 0) | (p.token_local ? FL_A_TOKEN_LOCAL : 0) |
            (p.d_call != p.d ? FL_A_COLS(p.d_call) : 0);
  a.window_left_p1 = p.window_left_p1; a.window_right_p1 = p.window_right_p1;
  a.softcap = (float)p.softcap;
  if (p.ragged) { a.flags |= FL_A_ROWS; a.out_rows = (int32_t)p.s_q; }
}

// One call's tensors: the results in the caller's layout and what the backward needs.
struct State {
  Tensor out, lse_user;
  Tensor lse;                // of the kernels: the caller's, except under documents
  Quantised q, k, v;
  Tensor buf;                // pooled: the buffer of the three operands' tensors
  Tensor status, k_rows, v_rows, seqused;
  Docs docs;
};

template <typename Make>
void operand_tensors(State& s, const Plan& p, const Shapes& sh, Make make) {
  const bool stats = p.need_bwd && p.prescale != 2;     // per tile (prescale == 2: per token instead, k_rows / v_rows)
  quantised_tensors(s.q, p, sh.b, sh.s_q, p.h, true, false, make);
  quantised_tensors(s.k, p, sh.b, sh.s_k, p.h_kv, true, stats, make);
  quantised_tensors(s.v, p, sh.b, sh.s_k, p.h_kv, false, stats, make);
}

// The tensors of a call in the order of _routes.py::state_spec, without O and the LSE.
std::vector<Tensor> state_list(const Plan& p, const State& s) {
  std::vector<Tensor> state;
  state.reserve(22);
  for (const Quantised* x : {&s.q, &s.k, &s.v}) { state.push_back(x->codes); state.push_back(x->fac); }
  state.push_back(s.status);
  const bool rows = p.prescale == 2;
  if (p.need_bwd) { state.push_back(rows ? s.k_rows : s.k.tile_stats); state.push_back(rows ? s.v_rows : s.v.tile_stats); }
  if (p.fp4) { state.push_back(s.q.x4); state.push_back(s.q.sf4); state.push_back(s.k.x4); state.push_back(s.k.sf4); }
  if (p.token_local)
    for (const Quantised* x : {&s.q, &s.k, &s.v}) state.push_back(x->token_factors);
  if (p.seqused_k) state.push_back(s.seqused);
  if (p.varlen) {
    state.push_back(s.docs.start); state.push_back(s.docs.len);
    if (!s.docs.aligned) { state.push_back(s.docs.row_map); state.push_back(s.docs.slot_src); state.push_back(s.docs.slot_rows); }
    state.push_back(s.docs.work);
  }
  return state;
}

// pooled: the operands' tensors (and document tables made here) are views of one buffer each, s.buf and s.docs.all.
State forward(int64_t handle, const Tensor& q_, const Tensor& k_, const Tensor& v_, at::TensorList docs_in, bool pooled) {
  const Plan& p = plan_at(handle);
  TORCH_CHECK(q_.is_cuda() && k_.is_cuda() && v_.is_cuda(), "q, k, v must be CUDA tensors: this library has no CPU path");
  // (the kernels take plain pointers: a host tensor's or another device's would be followed)
  TORCH_CHECK(k_.device() == q_.device() && v_.device() == q_.device(), "q, k, v must be on one device; got ", q_.device(), ", ",
              k_.device(), ", ", v_.device());
  for (const Tensor& t : docs_in)
    TORCH_CHECK(t.device() == q_.device(), "cu_seqlens / seqused / document maps must be on q's device ", q_.device(), "; got ", t.device());
  const c10::cuda::CUDAGuard guard(q_.device());
  const auto dev = q_.device();
  const cudaStream_t st = c10::cuda::getCurrentCUDAStream(dev.index()).stream();
  const Tensor q = rows_of(p, q_), k = rows_of(p, k_), v = rows_of(p, v_);
  TORCH_CHECK(!p.ragged || p.s_q == p.s_k, "batch rows that are no whole tiles: s_q must equal s_k");
  TORCH_CHECK(q.numel() == (p.varlen ? p.tot_q : p.b * p.s_q) * p.h * p.d_call &&
                  k.numel() == (p.varlen ? p.tot_q : p.b * p.s_k) * p.h_kv * p.d_call &&
                  v.numel() == k.numel() && k.scalar_type() == q.scalar_type() && v.scalar_type() == q.scalar_type(),
              "q, k, v do not have the shapes and types of their plan");
  State S;
  Tensor& seqused = S.seqused;
  if (p.seqused_k) {                          // batched form: docs = [seqused_k]
    TORCH_CHECK(docs_in.size() == 1, "docs is [seqused_k]");
    seqused = docs_in[0];
    TORCH_CHECK(seqused.scalar_type() == at::kInt && seqused.numel() == p.b && seqused.is_contiguous(),
                "seqused_k is an int32 tensor of shape (batch,)");
  }
  Docs& docs = S.docs;
  const bool has_docs = p.varlen;
  if (has_docs) docs = docs_of(p, q, docs_in, pooled, st);
  const Docs* dp = has_docs ? &docs : nullptr;
  const bool repacked = has_docs && !docs.aligned;
  const Shapes sh = shapes_of(p, has_docs ? docs.capacity : -1);
  const Tensor status = S.status = status_word(dev);
  int32_t* stp = ptr<int32_t>(status);
  const bool f16 = q.scalar_type() == at::kHalf;

  const bool rows = p.need_bwd && p.prescale == 2;      // per-token K / V statistics instead of per-tile ones
  Tensor &k_rows = S.k_rows, &v_rows = S.v_rows;
  if (rows) {
    k_rows = at::zeros({sh.b, sh.s_k}, at::TensorOptions().dtype(at::kFloat).device(dev));
    v_rows = at::zeros_like(k_rows);
  }
  using Sizes = std::initializer_list<int64_t>;
  if (pooled) {
    Pool pool;
    operand_tensors(S, p, sh, [&](Sizes sz, at::ScalarType dt) { pool.add(sz, dt); return Tensor(); });
    S.buf = pool.allocate(dev);
    operand_tensors(S, p, sh, [&](Sizes sz, at::ScalarType dt) { return pool.take(sz, dt); });
  } else {
    operand_tensors(S, p, sh, [&](Sizes sz, at::ScalarType dt) { return empty(sz, dt, dev); });
  }
  Quantised &qq = S.q, &kq = S.k, &vq = S.v;
  quantise_args(qq, p, q, sh.b, sh.s_q, p.h, true, dp, Tensor(), 0, stp);
  // max |K_j| of the codes' values; where those are rotated, the rotation-invariant 2-norm bounds it
  quantise_args(kq, p, k, sh.b, sh.s_k, p.h_kv, true, dp, k_rows, p.hadamard && !p.fp4 ? 3 : 2, stp);
  quantise_args(vq, p, v, sh.b, sh.s_k, p.h_kv, false, dp, v_rows, 1, stp);
  if (has_docs) {          // with them, which blocks exist, longest first
    docs.work = empty({FL_DOC_WORK_INTS(docs.capacity)}, at::kInt, dev);
    check(fl_quant_qkv_work(&qq.args, &kq.args, &vq.args, ptr<int32_t>(docs.start), ptr<int32_t>(docs.len), (int32_t)docs.len.numel(),
                            (int32_t)docs.capacity, p.window_left_p1, p.window_right_p1, p.causal, p.deterministic,
                            ptr<int32_t>(docs.work), st),
          "fl_quant_qkv_work");
  } else {
    check(fl_quant_qkv(&qq.args, &kq.args, &vq.args, st), "fl_quant_qkv");
  }

  // O has the caller's rows: under repacked documents the kernel writes the packed rows itself. On the aligned form the
  // kernel writes the rows of its documents only, and the padding rows read as zeros. (The LSE of repacked documents keeps
  // the aligned buffer's rows; its padding rows are never used: the backward selects zero wherever a row is no document's.)
  Tensor& out = S.out = empty(q.sizes(), q.scalar_type(), dev);
  Tensor& lse = S.lse = empty({sh.b, p.h, sh.s_q}, at::kFloat, dev);
  if (has_docs && docs.aligned) { out.zero_(); lse.zero_(); }
  fl_attn_args a = {};
  attn_common(a, p, sh, f16);
  if (p.p_group) a.flags |= FL_A_P_GROUP;
  a.q_codes = ptr<uint8_t>(qq.codes); a.k_codes = ptr<uint8_t>(kq.codes); a.v_codes = ptr<uint8_t>(vq.codes);
  a.fac_q = ptr<float>(p.token_local ? qq.token_factors : qq.fac);
  a.fac_k = ptr<float>(p.token_local ? kq.token_factors : kq.fac);
  a.fac_v = ptr<float>(p.token_local ? vq.token_factors : vq.fac);
  a.q4 = ptr<uint8_t>(qq.x4); a.k4 = ptr<uint8_t>(kq.x4); a.sfq4 = ptr<uint8_t>(qq.sf4); a.sfk4 = ptr<uint8_t>(kq.sf4);
  a.out = ptr<void>(out); a.lse = ptr<float>(lse);
  a.status = stp;
  a.seqused_k = ptr<int32_t>(seqused);
  if (has_docs) {
    a.doc_start = ptr<int32_t>(docs.start); a.doc_len = ptr<int32_t>(docs.len); a.n_docs = (int32_t)docs.len.numel();
  }
  const int64_t total = p.tot_q;
  if (repacked) {
    a.slot_src = ptr<int32_t>(docs.slot_src); a.slot_rows = ptr<int32_t>(docs.slot_rows); a.out_rows = (int32_t)total;
  }
  Tensor tok;
  if (p.token_local) {     // f_K, log2 f_V and 1 / f_V per key, which the forward applies to every score
    const int64_t n = vq.token_factors.numel();
    tok = empty({3 * n}, at::kShort, dev);
    check(fl_token_tables(ptr<float>(kq.token_factors), ptr<float>(vq.token_factors), n, ptr<uint32_t>(tok), ptr<uint16_t>(tok) + 2 * n, st),
          "fl_token_tables");
  }
  if (has_docs) {
    check(fl_fwd_work(&a, ptr<int32_t>(docs.work), st), "fl_fwd_work");
  } else if (p.token_local) {
    check(fl_fwd_tokens(&a, ptr<uint32_t>(tok), ptr<uint16_t>(tok) + 2 * vq.token_factors.numel(), st), "fl_fwd_tokens");
  } else {
    check(fl_fwd(&a, st), "fl_fwd");
  }

  Tensor& lse_user = S.lse_user = lse;
  if (has_docs) {
    if (docs.aligned) {
      lse_user = lse.select(0, 0);            // (h, total_q): the caller's rows are the kernels' rows
    } else if (p.return_lse) {
      // the kernels' LSE has the aligned buffer's rows; its live rows go to the caller's: (h, total) in packed order
      lse_user = empty({p.h, total}, at::kFloat, dev);
      lse_user.zero_();                       // (rows that no document covers read as zeros)
      check(fl_unpack_lse(ptr<float>(lse), ptr<int32_t>(docs.slot_src), ptr<int32_t>(docs.slot_rows), (int32_t)docs.capacity,
                          (int32_t)p.h, (int32_t)total, (int32_t)total, ptr<float>(lse_user), st),
            "fl_unpack_lse");
    } else {
      lse_user = empty({0}, at::kFloat, dev);
    }
  } else if (p.ragged) {                      // the kernels' LSE has whole tiles of rows: a copy (of one row and head, too, whose rows are contiguous)
    lse_user = p.return_lse ? lse.narrow(2, 0, p.s_q).clone(at::MemoryFormat::Contiguous) : empty({0}, at::kFloat, dev);
  }
  check_status_if_asked(dev);
  return S;
}

// ---------------------------------------------------------------------------------------------------- backward
// dq, dk, dv in the caller's layout. state = [O, LSE of the kernels] + what forward() saved; dk_mult / dq_mult: per-head
// factors of operands with float descales (prequant_fa3.py), or undefined tensors.
std::tuple<Tensor, Tensor, Tensor> backward(int64_t handle, int64_t capacity, bool aligned, const Tensor& dout_, at::TensorList state,
                                            const Tensor& dk_mult, const Tensor& dq_mult) {
  const Plan& p = plan_at(handle);
  const c10::cuda::CUDAGuard guard(dout_.device());
  const auto dev = dout_.device();
  const cudaStream_t st = c10::cuda::getCurrentCUDAStream(dev.index()).stream();
  const Tensor dout = rows_of(p, dout_);
  const bool has_docs = capacity >= 0, repacked = has_docs && !aligned;
  const Shapes sh = shapes_of(p, capacity);
  TORCH_CHECK(dout.numel() == (p.varlen ? p.tot_q : p.b * p.s_q) * p.h * p.d_call, "dout does not have the shape of the output");
  size_t i = 0;
  auto next = [&]() -> const Tensor& {
    TORCH_CHECK(i < state.size(), "the saved state of the forward is incomplete");
    TORCH_CHECK(state[i].device() == dev, "the saved state of the forward must be on dout's device ", dev, "; got ", state[i].device());
    return state[i++];
  };
  const Tensor &out = next(), &lse = next();
  const Tensor &qc = next(), &qf = next(), &kc = next(), &kf = next(), &vc = next(), &vf = next();
  const Tensor& status = next();
  const Tensor &kstats = next(), &vstats = next();
  fl_attn_args a = {};
  const bool f16 = out.scalar_type() == at::kHalf;
  attn_common(a, p, sh, f16);
  a.q_codes = ptr<uint8_t>(qc); a.k_codes = ptr<uint8_t>(kc); a.v_codes = ptr<uint8_t>(vc);
  a.fac_q = ptr<float>(qf); a.fac_k = ptr<float>(kf); a.fac_v = ptr<float>(vf);
  if (p.fp4) { a.q4 = ptr<uint8_t>(next()); a.sfq4 = ptr<uint8_t>(next()); a.k4 = ptr<uint8_t>(next()); a.sfk4 = ptr<uint8_t>(next()); }
  if (p.token_local) { a.fac_q = ptr<float>(next()); a.fac_k = ptr<float>(next()); a.fac_v = ptr<float>(next()); }
  if (p.seqused_k) a.seqused_k = ptr<int32_t>(next());
  const int32_t *slot_src = nullptr, *slot_rows = nullptr, *work = nullptr;
  const int64_t total = p.tot_q;
  if (has_docs) {
    a.doc_start = ptr<int32_t>(next());
    const Tensor& len = next();
    a.doc_len = ptr<int32_t>(len); a.n_docs = (int32_t)len.numel();
    if (repacked) {
      next();                                  // the row map (part of the op's state; the kernels work from the slot tables)
      slot_src = ptr<int32_t>(next()); slot_rows = ptr<int32_t>(next());
      a.slot_src = slot_src; a.slot_rows = slot_rows; a.out_rows = (int32_t)total;
    }
    work = ptr<int32_t>(next());
  }
  int32_t* stp = ptr<int32_t>(status);
  const bool rows = p.prescale == 2;
  const size_t nq = (size_t)(sh.b * p.h * sh.s_q), nbs = (size_t)(sh.b * sh.s_q);
  const int64_t nt_q = sh.s_q / 128, nt_k = sh.s_k / 128;
  Workspace ws;
  const size_t w_acc = ws.piece(nq * p.d * 2), w_codes = ws.piece(nq * p.d), w_fac = ws.piece(nq / 32 * 4),
               w_tok = p.token_local ? ws.piece(nq * 4) : 0, w_D = ws.piece(nq * 4), w_lse = ws.piece(nq * 4),
               w_stats = rows ? 0 : ws.piece((size_t)(sh.b * p.h * nt_q) * 8), w_ks = ws.piece((rows ? nbs : (size_t)(sh.b * nt_q)) * 4),
               w_ps = ws.piece((rows ? nbs : (size_t)(sh.b * nt_q)) * 4);
  // the tables that have to be zero on entry sit together at the end: one fill
  const size_t w_zero = ws.size, w_order = p.deterministic ? ws.piece((size_t)(sh.b * p.h * nt_q) * 8) : 0,
               w_rows = rows ? ws.piece(nbs * 4) : 0;
  ws.allocate(dev);
  if (ws.size > w_zero) C10_CUDA_CHECK(cudaMemsetAsync(ws.at(w_zero), 0, ws.size - w_zero, st));

  // dO quantiser + D + shifted LSE + zeroed accumulator
  fl_quant_args g = {};
  g.x = ptr<void>(dout); g.o = ptr<void>(out); g.lse = ptr<float>(lse);
  g.b = (int32_t)sh.b; g.s = (int32_t)sh.s_q; g.h = (int32_t)p.h; g.d = (int32_t)p.d;
  g.in_f16 = dout.scalar_type() == at::kHalf;
  TORCH_CHECK(dout.scalar_type() == out.scalar_type(), "dout is ", dout.scalar_type(), ", the output ", out.scalar_type());
  if (p.d_call != p.d) g.flags |= FL_Q_COLS(p.d_call);
  if (p.token_local) { g.flags |= FL_Q_TOKEN_LOCAL | FL_Q_D_PER_FACTOR; g.token_factors = ptr<float>(ws.at(w_tok)); }
  g.codes = ptr<uint8_t>(ws.at(w_codes)); g.fac = ptr<float>(ws.at(w_fac));
  g.d_out = ptr<float>(ws.at(w_D)); g.lse_log2 = ptr<float>(ws.at(w_lse)); g.zero_acc = ws.at(w_acc);
  if (!rows) g.tile_stats = ptr<float>(ws.at(w_stats));
  else { g.row_stat = ptr<float>(ws.at(w_rows)); g.row_stat_kind = 1; }
  g.lse_shift = (float)kPShiftLog2;
  g.d_multiplier = -0.00390625f;               // -2^-8: slot 6 of the reference's backward scalars (_routes.backward_scalars)
  g.status = stp;
  if (repacked) {
    g.slot_src = slot_src; g.slot_rows = slot_rows; g.src_rows = (int32_t)total;
    g.flags |= FL_Q_O_PACKED;                  // the forward output has the packed rows
  } else if (p.ragged) {
    g.flags |= FL_Q_ROWS; g.src_rows = (int32_t)p.s_q;
  }
  check(fl_quant_blocks(&g, st), "fl_quant_blocks");

  float *ks = ptr<float>(ws.at(w_ks)), *ps = ptr<float>(ws.at(w_ps));
  if (rows) {      // kstats / vstats are the per-token tables here; the prefix maxima go into copies (the state is read-only)
    const Tensor vs = vstats.clone(), kst = kstats.clone();
    check(fl_dq_prescale_rows(ptr<float>(ws.at(w_rows)), ptr<float>(vs), ptr<float>(kst), (int32_t)sh.b, (int32_t)sh.s_q, 1.0f, ks, ps, st),
          "fl_dq_prescale_rows");
    a.dq_scale_rows = ks;
  } else {
    check(fl_dq_prescale(ptr<float>(ws.at(w_stats)), ptr<float>(vstats), ptr<float>(kstats), (int32_t)sh.b, (int32_t)p.h, (int32_t)p.h_kv,
                         (int32_t)nt_q, (int32_t)nt_k, p.prescale == 1, 1.0f, ks, ps, st),
          "fl_dq_prescale");
    a.dq_scale = ks;
  }

  const bool had8 = p.hadamard && !p.fp4;      // only the 8-bit route's E4M3 codes are rotated
  // the gradients in the caller's shapes: the kernels write the caller's rows (packed ones through the slot tables)
  const std::vector<int64_t> kshape = p.varlen ? std::vector<int64_t>{p.tot_q, p.h_kv, p.d_call}
                                               : std::vector<int64_t>{p.b, p.s_k, p.h_kv, p.d_call};
  const Tensor dq = empty(dout.sizes(), out.scalar_type(), dev), dk = empty(kshape, out.scalar_type(), dev),
               dv = empty(kshape, out.scalar_type(), dev);
  a.flags |= (had8 ? FL_A_HAD_DK : 0) | (p.rowlocal ? FL_A_DQ_ROWLOCAL : 0) | (p.token_local ? FL_A_D_PER_FACTOR : 0);
  a.do_codes = g.codes; a.fac_do = p.token_local ? g.token_factors : g.fac;
  a.lse_log2 = g.lse_log2; a.d_rows = g.d_out; a.dq_acc = g.zero_acc;
  a.dk = ptr<void>(dk); a.dv = ptr<void>(dv);
  a.dk_mult = ptr<float>(dk_mult);
  if (p.deterministic) a.dq_order = ptr<int32_t>(ws.at(w_order));
  a.status = stp;
  if (work) check(fl_bwd_work(&a, work, st), "fl_bwd_work");
  else check(fl_bwd(&a, st), "fl_bwd");
  if (p.ragged)
    check(fl_dq_post_trim(g.zero_acc, ps, a.softmax_scale, ptr<void>(dq), (int32_t)sh.b, (int32_t)sh.s_q, (int32_t)p.s_q, (int32_t)p.h,
                          (int32_t)p.d, (int32_t)p.d_call, had8, f16, st),
          "fl_dq_post_trim");
  else
    check(fl_dq_post_cols(g.zero_acc, ps, rows, ptr<float>(dq_mult), a.softmax_scale, ptr<void>(dq), (int32_t)sh.b, (int32_t)sh.s_q,
                        (int32_t)p.h, (int32_t)p.d, (int32_t)p.d_call, had8, f16, slot_src, slot_rows, st),
        "fl_dq_post_cols");
  check_status_if_asked(dev);
  return {dq, dk, dv};
}

// ---------------------------------------------------------------------------------------------------- ops and autograd
using FwdSig = std::tuple<Tensor, Tensor, std::vector<Tensor>>(const Tensor&, const Tensor&, const Tensor&, at::TensorList, int64_t, int64_t);
using BwdSig = std::tuple<Tensor, Tensor, Tensor>(const Tensor&, at::TensorList, int64_t);

template <bool FP4>
const c10::TypedOperatorHandle<FwdSig>& fwd_op() {
  static const auto op = c10::Dispatcher::singleton().findSchemaOrThrow(FP4 ? "lowbit_attn::fp4" : "lowbit_attn::fp8", "").typed<FwdSig>();
  return op;
}
template <bool FP4>
const c10::TypedOperatorHandle<BwdSig>& bwd_op() {
  static const auto op = c10::Dispatcher::singleton().findSchemaOrThrow(FP4 ? "lowbit_attn::fp4_bwd" : "lowbit_attn::fp8_bwd", "").typed<BwdSig>();
  return op;
}

std::tuple<Tensor, Tensor, std::vector<Tensor>> fwd_cuda(const Tensor& q, const Tensor& k, const Tensor& v, at::TensorList docs,
                                                         int64_t plan, int64_t /*docs_id*/) {
  const Plan& p = plan_at(plan);
  State s = forward(plan, q, k, v, docs, false);
  std::vector<Tensor> state = state_list(p, s);
  for (Tensor& t : state)                     // (nor do an op's outputs share memory with its inputs: the tables it was given)
    if (std::any_of(docs.begin(), docs.end(), [&](const Tensor& d) { return t.is_alias_of(d); })) t = t.clone();
  const bool has_docs = p.varlen;
  if ((has_docs && !p.aligned) || p.ragged) state.insert(state.begin(), s.lse);       // (otherwise the kernels' LSE is the op's output)
  // the entry handle rides along as a 0-d tensor, so that the backward op needs no object beside its tensors
  Tensor entry = at::empty({}, at::TensorOptions().dtype(at::kLong));
  *entry.mutable_data_ptr<int64_t>() = entry_of(plan, has_docs ? s.docs.capacity : -1, has_docs && s.docs.aligned);
  state.push_back(entry);
  return {s.out, s.lse_user, std::move(state)};
}
std::tuple<Tensor, Tensor, Tensor> bwd_cuda(const Tensor& dout, at::TensorList state, int64_t entry) {
  const Entry e = entry_at(entry);
  return backward(e.plan, e.capacity, e.aligned, dout, state, Tensor(), Tensor());
}

// O is the node's output; the LSE (no gradient) and the state (codes, tables) are saved beside it and leave the op as plain tensors.
struct Call {
  at::TensorList docs;
  int64_t plan, docs_id;
  Tensor* lse;
  std::vector<Tensor>* state;
};
template <bool FP4>
struct AttnNode : public torch::autograd::Function<AttnNode<FP4>> {
  // compiled autograd may trace backward(): it reads nothing but its inputs, the saved tensors and two saved numbers
  static constexpr bool is_traceable = true;
  static Tensor forward(torch::autograd::AutogradContext* ctx, const Tensor& q, const Tensor& k, const Tensor& v, Call c) {
    at::AutoDispatchBelowADInplaceOrView below;
    auto [out, lse, state] = fwd_op<FP4>().call(q, k, v, c.docs, c.plan, c.docs_id);
    const Plan& p = plan_at(c.plan);
    variable_list saved;
    saved.reserve(state.size() + 2);
    saved.push_back(out);
    saved.push_back(lse);
    saved.insert(saved.end(), state.begin(), state.end() - 1);     // (the entry handle is kept as a number)
    ctx->save_for_backward(std::move(saved));
    // the capacity of the aligned buffer is in the shapes: repacked documents keep its LSE (1, h, capacity) first (as do batch rows that
    // are no whole tiles)
    const bool has_docs = p.varlen, repacked = has_docs && !p.aligned;
    ctx->saved_data["entry"] = entry_of(c.plan, !has_docs ? -1 : repacked ? state[0].sym_size(2).guard_int(__FILE__, __LINE__) : p.tot_q, has_docs && p.aligned);
    ctx->saved_data["own_lse"] = repacked || p.ragged;
    ctx->set_materialize_grads(false);
    *c.lse = std::move(lse);
    *c.state = std::move(state);
    return out;
  }
  static variable_list backward(torch::autograd::AutogradContext* ctx, variable_list grads) {
    if (!grads[0].defined()) return {Tensor(), Tensor(), Tensor(), Tensor()};
    variable_list state = ctx->get_saved_variables();
    if (ctx->saved_data["own_lse"].toBool()) state.erase(state.begin() + 1);      // the kernels' own LSE follows the caller's
    auto [dq, dk, dv] = bwd_op<FP4>().call(grads[0].contiguous(), state, ctx->saved_data["entry"].toInt());
    return {dq, dk, dv, Tensor()};
  }
};

template <bool FP4>
std::tuple<Tensor, Tensor, std::vector<Tensor>> fwd_autograd(const Tensor& q, const Tensor& k, const Tensor& v, at::TensorList docs,
                                                             int64_t plan, int64_t docs_id) {
  if (!at::GradMode::is_enabled() || !(q.requires_grad() || k.requires_grad() || v.requires_grad())) {
    at::AutoDispatchBelowADInplaceOrView below;
    return fwd_op<FP4>().call(q, k, v, docs, plan, docs_id);
  }
  std::vector<Tensor> state;
  Tensor lse, out = AttnNode<FP4>::apply(q, k, v, Call{docs, plan, docs_id, &lse, &state});
  return {std::move(out), std::move(lse), std::move(state)};
}

// Nothing between the caller and the CUDA kernels wants to see the op: no dispatch mode, fake or wrapped tensor, transform or tracer.
bool direct(std::initializer_list<const Tensor*> ts) {
  static const c10::DispatchKeySet known =
      c10::DispatchKeySet({c10::DispatchKey::CUDA, c10::DispatchKey::AutogradCUDA, c10::DispatchKey::ADInplaceOrView,
                           c10::DispatchKey::BackendSelect}) |
      c10::autocast_dispatch_keyset;
  const auto tls = c10::impl::tls_local_dispatch_key_set();
  c10::DispatchKeySet ks = tls.included_;
  for (const Tensor* t : ts) ks = ks | t->key_set();
  return ((ks - tls.excluded_).raw_repr() & ~known.raw_repr()) == 0;
}

// The node of a call that went to the kernels directly. It saves the call's buffers whole and makes the tensors in them again: a
// saved tensor can be offloaded, resized or freed without touching another.
struct DirectNode : public torch::autograd::Function<DirectNode> {
  static constexpr bool is_traceable = true;         // (as AttnNode; traced, the views and the op are recorded)
  static Tensor forward(torch::autograd::AutogradContext* ctx, const Tensor& q, const Tensor& k, const Tensor& v, Call c) {
    at::AutoDispatchBelowADInplaceOrView below;
    State s = ::forward(c.plan, q, k, v, c.docs, true);
    const Docs& d = s.docs;
    const bool made = d.all.defined();               // (then the tables are views of it)
    ctx->save_for_backward({s.out, s.lse, s.buf, s.status, s.k_rows, s.v_rows, s.seqused, made ? Tensor() : d.start,
                            made ? Tensor() : d.len, made ? Tensor() : d.row_map, made ? Tensor() : d.slot_src,
                            made ? Tensor() : d.slot_rows, d.all, d.work});
    ctx->saved_data["plan"] = c.plan;
    ctx->set_materialize_grads(false);
    *c.lse = std::move(s.lse_user);
    return s.out;
  }
  static variable_list backward(torch::autograd::AutogradContext* ctx, variable_list grads) {
    if (!grads[0].defined()) return {Tensor(), Tensor(), Tensor(), Tensor()};
    const int64_t plan = ctx->saved_data["plan"].toInt();
    const Plan& p = plan_at(plan);
    const variable_list t = ctx->get_saved_variables();
    State s;
    s.status = t[3]; s.k_rows = t[4]; s.v_rows = t[5]; s.seqused = t[6];
    Docs& d = s.docs;
    d.start = t[7]; d.len = t[8]; d.row_map = t[9]; d.slot_src = t[10]; d.slot_rows = t[11]; d.all = t[12]; d.work = t[13];
    const bool has_docs = p.varlen;
    d.aligned = has_docs && p.aligned;
    d.capacity = !has_docs ? -1 : d.aligned ? p.tot_q : t[1].sym_size(2).guard_int(__FILE__, __LINE__);   // (repacked documents: the kernels' LSE, (1, h, capacity))
    if (d.all.defined()) d.split((d.all.sym_numel().guard_int(__FILE__, __LINE__) - d.capacity - d.capacity / 128 * 2) / 2);
    // (a backward that records a graph of its own meets the op, too: it has no derivative, and says so)
    const bool plain = !at::GradMode::is_enabled() && direct({&grads[0], &t[0], &t[2]});
    Pool pool(t[2], !plain);
    operand_tensors(s, p, shapes_of(p, d.capacity), [&](std::initializer_list<int64_t> sz, at::ScalarType dt) { return pool.take(sz, dt); });
    std::vector<Tensor> state = state_list(p, s);
    state.insert(state.begin(), {t[0], t[1]});
    Tensor dq, dk, dv;
    if (plain) {
      at::AutoDispatchBelowADInplaceOrView below;
      RECORD_FUNCTION(p.fp4 ? "lowbit_attn::fp4_bwd" : "lowbit_attn::fp8_bwd", c10::ArrayRef<const c10::IValue>{});
      std::tie(dq, dk, dv) = ::backward(plan, d.capacity, d.aligned, grads[0], state, Tensor(), Tensor());
    } else {
      const auto& op = p.fp4 ? bwd_op<true>() : bwd_op<false>();
      std::tie(dq, dk, dv) = op.call(grads[0].contiguous(), state, entry_of(plan, d.capacity, d.aligned));
    }
    return {dq, dk, dv, Tensor()};
  }
};

TORCH_LIBRARY_IMPL(lowbit_attn, CUDA, m) {
  m.impl("fp8", fwd_cuda);
  m.impl("fp4", fwd_cuda);
  m.impl("fp8_bwd", bwd_cuda);
  m.impl("fp4_bwd", bwd_cuda);
}
TORCH_LIBRARY_IMPL(lowbit_attn, Autograd, m) {
  m.impl("fp8", fwd_autograd<false>);
  m.impl("fp4", fwd_autograd<true>);
}

// ---------------------------------------------------------------------------------------------------- Python
// run(fp4, plan, q, k, v, docs) -> (out, lse): the registered op on a resolved plan, without going through torch.ops (whose
// argument matching alone costs more than the C++ side of a call), and without the op where nothing would see it
PyObject* py_run(PyObject*, PyObject* const* args, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  TORCH_CHECK(n == 6 && PyTuple_Check(args[5]), "run(fp4, plan, q, k, v, docs)");
  for (int i = 2; i < 5; ++i) TORCH_CHECK_TYPE(THPVariable_Check(args[i]), "q, k, v are tensors");
  const bool fp4 = PyObject_IsTrue(args[0]) != 0;
  const int64_t plan = PyLong_AsLongLong(args[1]);
  std::vector<Tensor> docs;
  for (Py_ssize_t i = 0; i < PyTuple_GET_SIZE(args[5]); ++i) {
    PyObject* t = PyTuple_GET_ITEM(args[5], i);
    TORCH_CHECK_TYPE(THPVariable_Check(t), "docs are tensors");
    docs.push_back(THPVariable_Unpack(t));
  }
  const Tensor &q = THPVariable_Unpack(args[2]), &k = THPVariable_Unpack(args[3]), &v = THPVariable_Unpack(args[4]);
  Tensor out, lse;
  {
    pybind11::gil_scoped_release nogil;
    if (direct({&q, &k, &v})) {
      RECORD_FUNCTION(fp4 ? "lowbit_attn::fp4" : "lowbit_attn::fp8", c10::ArrayRef<const c10::IValue>{});
      if (at::GradMode::is_enabled() && (q.requires_grad() || k.requires_grad() || v.requires_grad())) {
        out = DirectNode::apply(q, k, v, Call{docs, plan, 0, &lse, nullptr});
      } else {
        at::AutoDispatchBelowADInplaceOrView below;
        State s = forward(plan, q, k, v, docs, true);
        out = std::move(s.out);
        lse = std::move(s.lse_user);
      }
    } else {
      const auto& op = fp4 ? fwd_op<true>() : fwd_op<false>();
      std::vector<Tensor> state;
      std::tie(out, lse, state) = op.call(q, k, v, docs, plan, 0);
    }
  }
  PyObject* t = PyTuple_New(2);
  PyTuple_SET_ITEM(t, 0, THPVariable_Wrap(std::move(out)));
  PyTuple_SET_ITEM(t, 1, THPVariable_Wrap(std::move(lse)));
  return t;
  END_HANDLE_TH_ERRORS
}
PyMethodDef kRun = {"run", reinterpret_cast<PyCFunction>(reinterpret_cast<void*>(py_run)), METH_FASTCALL,
                    "run(fp4, plan, q, k, v, docs) -> (out, lse)"};

// call_key(q, k, v, *values) -> tuple: what plan resolution may look at, as a key. Tensors as their sizes, type and requires_grad, everything
// else as it is; None where q, k, v are not plain tensors of known sizes (the caller makes its key from their attributes). In Python the
// same key (thirty attributes and type tests) was half of the 5 us that a short call spends before it gets here.
PyObject* py_call_key(PyObject*, PyObject* const* args, Py_ssize_t n) {
  HANDLE_TH_ERRORS
  TORCH_CHECK(n >= 3, "call_key(q, k, v, *values)");
  PyObject* key = PyTuple_New(n + 1);
  PyTuple_SET_ITEM(key, n, PyBool_FromLong(at::GradMode::is_enabled()));
  for (Py_ssize_t i = 0; i < n; ++i) {
    PyObject* item = nullptr;
    if (PyType_IsSubtype(Py_TYPE(args[i]), reinterpret_cast<PyTypeObject*>(THPVariableClass))) {      // (an isinstance of Tensor takes its metaclass along)
      const Tensor& t = THPVariable_Unpack(args[i]);
      const c10::TensorImpl* impl = t.unsafeGetTensorImpl();
      if (!THPVariable_CheckExact(args[i]) || impl->has_symbolic_sizes_strides() || impl->is_python_dispatch() || t.dim() > 8) {
        Py_DECREF(key);
        Py_RETURN_NONE;
      }
      int64_t facts[10] = {(int64_t)t.scalar_type() * 2 + t.requires_grad(), t.dim()};
      for (int64_t d = 0; d < t.dim(); ++d) facts[2 + d] = t.size(d);
      item = PyBytes_FromStringAndSize(reinterpret_cast<const char*>(facts), (2 + t.dim()) * sizeof(int64_t));
    } else if (i < 3) {
      Py_DECREF(key);
      Py_RETURN_NONE;
    } else {
      item = args[i];
      Py_INCREF(item);
    }
    PyTuple_SET_ITEM(key, i, item);
  }
  return key;
  END_HANDLE_TH_ERRORS
}
PyMethodDef kCallKey = {"call_key", reinterpret_cast<PyCFunction>(reinterpret_cast<void*>(py_call_key)), METH_FASTCALL,
                        "call_key(q, k, v, *values) -> tuple or None"};

int64_t register_plan(const pybind11::dict& d) {
  Plan p;
  auto b = [&](const char* n) { return d[n].cast<bool>(); };
  auto i = [&](const char* n) { return d[n].cast<int64_t>(); };
  p.fp4 = b("fp4"); p.token_local = b("token_local"); p.hadamard = b("hadamard"); p.causal = b("causal"); p.need_bwd = b("need_bwd");
  p.p_group = b("p_group"); p.seqused_k = b("seqused_k"); p.varlen = b("varlen"); p.aligned = b("aligned"); p.ragged = b("ragged");
  p.return_lse = b("return_lse"); p.deterministic = b("deterministic"); p.rowlocal = b("rowlocal");
  p.prescale = (int)i("prescale"); p.window_left_p1 = (int)i("window_left_p1"); p.window_right_p1 = (int)i("window_right_p1");
  p.softcap = d["softcap"].cast<double>(); p.softmax_scale = d["softmax_scale"].cast<double>();
  p.b = i("b"); p.s_q = i("s_q"); p.s_k = i("s_k"); p.h = i("h"); p.h_kv = i("h_kv"); p.d = i("d"); p.tot_q = i("tot_q"); p.d_call = i("d_call");
  std::lock_guard<std::mutex> g(g_lock);
  g_plans.push_back(p);
  return (int64_t)g_plans.size() - 1;
}
std::tuple<int64_t, int64_t, bool> entry_facts(int64_t i) {
  const Entry e = entry_at(i);
  return {e.plan, e.capacity, e.aligned};
}
std::tuple<Tensor, Tensor, Tensor> backward_batched(int64_t plan, const Tensor& dout, const std::vector<Tensor>& state,
                                                    const Tensor& dk_mult, const Tensor& dq_mult) {
  return backward(plan, -1, false, dout, state, dk_mult, dq_mult);
}
Tensor device_status_word(int64_t idx) {
  const c10::cuda::CUDAGuard guard((c10::DeviceIndex)idx);
  return status_word(at::Device(at::kCUDA, (c10::DeviceIndex)idx));
}
void note_status(const Tensor& t) {
  TORCH_CHECK(t.is_cuda() && t.device().index() < kMaxDevices, "a status word is a CUDA tensor");
  {
    std::lock_guard<std::mutex> g(g_status_lock);
    g_last_status[t.device().index()] = t;
  }
  check_status_if_asked(t.device());
}

}  // namespace

// (every function is wrapped: PyTorch's own translation of its exceptions, which does not symbolise a C++ stack)
PYBIND11_MODULE(_host, m) {
  using torch::wrap_pybind_function;
  using torch::wrap_pybind_function_no_gil;
  m.def("register_plan", wrap_pybind_function(register_plan));
  m.def("register_entry", wrap_pybind_function(entry_of));
  m.def("entry", wrap_pybind_function(entry_facts));
  m.def("backward", wrap_pybind_function_no_gil(backward_batched));
  m.def("status_word", wrap_pybind_function_no_gil(device_status_word));
  m.def("note_status", wrap_pybind_function_no_gil(note_status));
  m.def("check_status", wrap_pybind_function_no_gil(check_status));
  m.attr("call_key") = pybind11::reinterpret_steal<pybind11::object>(PyCFunction_NewEx(&kCallKey, nullptr, nullptr));
  m.attr("run") = pybind11::reinterpret_steal<pybind11::object>(PyCFunction_NewEx(&kRun, nullptr, nullptr));
}

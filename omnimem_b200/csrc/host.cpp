// Host path of the tensor-level operators: argument checks, output and scratch allocation through torch's caching
// allocator, stream lookup and the call into the C ABI, in native code.  A call of the small kernels costs the host
// more than the kernel runs (a Python wrapper over ctypes: 20 to 40 us); here it costs a few microseconds.
// Nothing here synchronises, except the id check of selection_attention, which its contract asks for.
#include <c10/cuda/CUDAGuard.h>
#include <c10/cuda/CUDAStream.h>
#include <cuda_runtime.h>
#include <torch/extension.h>

#include <cstdlib>
#include <cstring>
#include <mutex>
#include <string>
#include <vector>

#include "../../include/omnimem_b200.h"

namespace py = pybind11;
using at::Tensor;
using torch::autograd::AutogradContext;
using torch::autograd::Variable;
using torch::autograd::variable_list;
using OptTensor = c10::optional<Tensor>;

namespace {

// ------------------------------------------------------------------------------------------ errors
PyObject* g_error = nullptr;                       // omnimem_b200._lib.NSABackendError
struct BackendError : std::runtime_error {
  using std::runtime_error::runtime_error;
};
void check(const char* name, int rc) {
  if (rc == 0) return;
  throw BackendError(std::string(name) + " failed (" + std::to_string(rc) + "): " + nsa_last_error());
}
// (the text is put together only where it is needed: a call checks some twenty conditions)
#define NEED(ok, text)                    \
  do {                                    \
    if (!(ok)) throw BackendError(text);  \
  } while (0)

// ----------------------------------------------------------------------------------------- tensors
int dtype_of(const Tensor& t) {
  switch (t.scalar_type()) {
    case at::kBFloat16: return NSA_BF16;
    case at::kHalf: return NSA_F16;
    case at::kFloat: return NSA_F32;
    default: throw BackendError(std::string("unsupported dtype torch.") + c10::toString(t.scalar_type()));
  }
}
void need_cuda(std::initializer_list<const Tensor*> ts) {
  for (const Tensor* t : ts)
    if (t->defined() && !t->is_cuda()) throw BackendError("omnimem_b200 ops need CUDA tensors (there is no CPU path)");
}
bool is_rows16(const Tensor& t) {
  const int64_t esz = t.element_size(), nd = t.dim();
  if (nd == 0 || t.stride(nd - 1) != 1 || reinterpret_cast<uintptr_t>(t.data_ptr()) % 16 != 0) return false;
  for (int64_t i = 0; i + 1 < nd; ++i)
    if (t.stride(i) * esz % 16 != 0) return false;
  return true;
}
// t or a contiguous copy whose innermost stride is 1 and whose rows are 16-byte aligned
Tensor rows16(const Tensor& t) { return is_rows16(t) ? t : t.contiguous(); }
// The one stride between the rows that t's first `dims` dimensions count, if they lie evenly.  A dimension of size 1 says
// nothing: its own stride is arbitrary.
c10::optional<int64_t> even_stride(const Tensor& t, int64_t dims) {
  bool any = false;
  int64_t stride = 0, next = 0;
  for (int64_t i = dims - 1; i >= 0; --i) {
    if (t.size(i) == 1) continue;
    if (any && t.stride(i) != next) return c10::nullopt;
    if (!any) stride = t.stride(i);
    any = true;
    next = t.stride(i) * t.size(i);
  }
  return stride;
}
// Whether two contiguous CPU tensors hold the same bytes of the same type and shape.
bool same_bytes(const Tensor& a, const Tensor& b) {
  const auto plain = [](const Tensor& t) { return t.device().is_cpu() && t.is_contiguous() && !t.is_conj() && !t.is_neg(); };
  return plain(a) && plain(b) && a.scalar_type() == b.scalar_type() && a.sizes() == b.sizes() &&
         (a.numel() == 0 || std::memcmp(a.const_data_ptr(), b.const_data_ptr(), a.nbytes()) == 0);
}
struct Strides {
  int64_t v[4];
  explicit Strides(const Tensor& t) {
    for (int64_t i = 0; i < 4; ++i) v[i] = i < t.dim() ? t.stride(i) : 0;
  }
  operator const int64_t*() const { return v; }
};
void* stream_of(const Tensor& t) { return c10::cuda::getCurrentCUDAStream(t.device().index()).stream(); }
Tensor scratch(size_t bytes, const Tensor& like) {
  return at::empty({static_cast<int64_t>(bytes > 0 ? bytes : 1)}, like.options().dtype(at::kByte));
}
const Tensor& or_none(const OptTensor& t) {
  static const Tensor none;
  return t.has_value() ? *t : none;
}
void* ptr(const Tensor& t) { return t.defined() ? t.data_ptr() : nullptr; }
int32_t i32(int64_t x, const char* what) {
  NEED(x >= INT32_MIN && x <= INT32_MAX, std::string(what) + "=" + std::to_string(x) + " does not fit in int32");
  return static_cast<int32_t>(x);
}
int64_t ceil_div(int64_t a, int64_t b) { return (a + b - 1) / b; }

std::string shape(const Tensor& t) {
  std::string s = "(";
  for (int64_t i = 0; i < t.dim(); ++i) s += (i ? ", " : "") + std::to_string(t.size(i));
  return s + ")";
}
// (the callers unpack four sizes: a fifth dimension would be dropped)
void need_4d(const Tensor& t, const char* what) {
  if (t.dim() != 4) throw py::value_error(std::string(what) + ": a tensor of four dimensions is expected, got " + shape(t));
}

// ----------------------------------------------------------------------------------------- pooling
Tensor pool_rows(const Tensor& x_, int64_t size) {
  need_4d(x_, "pool_rows x");
  need_cuda({&x_});
  const Tensor x = rows16(x_);
  const c10::cuda::CUDAGuard guard(x.device());
  const int64_t B = x.size(0), N = x.size(1), H = x.size(2), D = x.size(3);
  TORCH_CHECK(size > 0, "pool_rows: size must be > 0");
  Tensor out = at::empty({B, ceil_div(N, size), H, D}, x.options());
  check("nsa_pool_rows", nsa_pool_rows(x.data_ptr(), Strides(x), out.data_ptr(), Strides(out), B, N, H, D, i32(size, "size"),
                                       dtype_of(x), stream_of(x)));
  return out;
}

// ------------------------------------------------------------------------------------------- top-k
// (block_size, chunk_size, chunk_size_k, q_group_size, q_chunk_offset, ex_win, ex_sink, causal, tf_mask, prog_excl,
// id_base, id_stride)
using MaskArgs = std::vector<int64_t>;
nsa_topk_mask mask_of(const MaskArgs& a) {
  static const char* names[12] = {"block_size", "chunk_size", "chunk_size_k", "q_group_size", "q_chunk_offset", "ex_win", "ex_sink",
                                  "causal", "tf_mask", "prog_excl", "id_base", "id_stride"};
  NEED(a.size() == 12, "topk: 12 mask values are expected");
  int32_t v[12];
  for (int i = 0; i < 12; ++i) v[i] = i32(a[i], names[i]);
  return nsa_topk_mask{v[0], v[1], v[2], v[3], v[4], v[5], v[6], v[7] != 0, v[8] != 0, v[9] != 0, v[10], v[11]};
}
Tensor unit_inner(const Tensor& t) { return t.stride(-1) == 1 ? t : t.contiguous(); }

std::pair<Tensor, OptTensor> topk(const Tensor& q_, const Tensor& k_, int64_t T, double scale, const MaskArgs& mask, bool scores) {
  need_4d(q_, "topk q");
  need_4d(k_, "topk k");
  need_cuda({&q_, &k_});
  NEED(q_.scalar_type() == k_.scalar_type(), std::string("topk: q and k must share a dtype, got torch.") + c10::toString(q_.scalar_type()) +
                                                 " vs torch." + c10::toString(k_.scalar_type()));
  const int64_t B = q_.size(0), MG = q_.size(1), H = q_.size(2), D = q_.size(3), NC = k_.size(1);
  NEED(k_.size(0) == B && k_.size(2) == H && k_.size(3) == D, "topk: incompatible shapes q=" + shape(q_) + " k=" + shape(k_));
  const Tensor q = unit_inner(q_), k = unit_inner(k_);
  const c10::cuda::CUDAGuard guard(q.device());
  Tensor out = at::empty({B, MG, H, T}, q.options().dtype(at::kInt)), sc;
  if (scores) sc = at::empty({B, MG, H, T}, q.options().dtype(at::kFloat));
  const nsa_topk_mask m = mask_of(mask);
  const size_t wsb = nsa_topk_workspace_bytes(B, MG, H, NC);
  const Tensor ws = scratch(wsb, q);
  check("nsa_topk", nsa_topk(q.data_ptr(), Strides(q), k.data_ptr(), Strides(k), B, MG, H, D, NC, i32(T, "topk"), static_cast<float>(scale), &m,
                             out.data_ptr<int32_t>(), static_cast<float*>(ptr(sc)), ws.data_ptr(), wsb, dtype_of(q), stream_of(q)));
  return {out, scores ? OptTensor(sc) : OptTensor()};
}

std::tuple<Tensor, Tensor, Tensor, OptTensor> select_blocks(const Tensor& q_, const Tensor& k_, int64_t T, double scale, const MaskArgs& mask,
                                                            bool scores) {
  need_4d(q_, "select_blocks q");
  need_4d(k_, "select_blocks k");
  need_cuda({&q_, &k_});
  NEED(q_.scalar_type() == k_.scalar_type(), std::string("select_blocks: q and k must share a dtype, got torch.") +
                                                 c10::toString(q_.scalar_type()) + " vs torch." + c10::toString(k_.scalar_type()));
  const Tensor q = rows16(q_), k = rows16(k_);
  const c10::cuda::CUDAGuard guard(k.device());
  const nsa_topk_mask m = mask_of(mask);
  TORCH_CHECK(m.q_group_size > 0 && m.block_size > 0, "select_blocks: group and block sizes must be > 0");
  const int64_t B = q.size(0), M = q.size(1), H = q.size(2), D = q.size(3), N = k.size(1);
  const int64_t MG = ceil_div(M, m.q_group_size), NC = ceil_div(N, m.block_size);
  Tensor qp = at::empty({B, MG, H, D}, q.options()), kp = at::empty({B, NC, H, D}, k.options());
  Tensor out = at::empty({B, MG, H, T}, q.options().dtype(at::kInt)), sc;
  if (scores) sc = at::empty({B, MG, H, T}, q.options().dtype(at::kFloat));
  const size_t wsb = nsa_topk_workspace_bytes(B, MG, H, NC);
  const Tensor ws = scratch(wsb, q);
  check("nsa_select_blocks",
        nsa_select_blocks(q.data_ptr(), Strides(q), k.data_ptr(), Strides(k), B, M, H, D, N, i32(T, "topk"), static_cast<float>(scale), &m,
                          qp.data_ptr(), kp.data_ptr(), out.data_ptr<int32_t>(), static_cast<float*>(ptr(sc)), ws.data_ptr(), wsb, dtype_of(k),
                          stream_of(k)));
  return {out, qp, kp, scores ? OptTensor(sc) : OptTensor()};
}

// --------------------------------------------------------------------------------------- attention
// A K/V source: dense (k, v), paged (pools + block table) or pointers (address tables in k, v; n_tokens carries the
// element stride between tokens).
struct Source {
  int mode;
  Tensor k, v, table;
  int64_t n_tokens, page_tokens;
  nsa_kv_source c() const {
    nsa_kv_source s;
    std::memset(&s, 0, sizeof(s));
    s.mode = mode;
    if (mode == NSA_KV_PTR) {
      s.ptr_k = k.data_ptr<int64_t>();
      s.ptr_v = v.data_ptr<int64_t>();
      s.ptr_stride_n = n_tokens;
      return s;
    }
    s.k = k.data_ptr();
    s.v = v.data_ptr();
    s.n_tokens = n_tokens;
    if (mode == NSA_KV_DENSE) {
      for (int i = 0; i < 3; ++i) { s.k_stride[i] = k.stride(i); s.v_stride[i] = v.stride(i); }
    } else {
      s.block_table = table.data_ptr<int32_t>();
      s.max_blocks = static_cast<int32_t>(table.size(-1));
      s.page_tokens = static_cast<int32_t>(page_tokens);
      s.num_pages = k.size(0);
    }
    return s;
  }
};
// n_tokens < 0: as many as k has
Source dense(const Tensor& k, const Tensor& v, int64_t n_tokens = -1) {
  need_4d(k, "k");
  need_cuda({&k, &v});
  NEED(k.sizes() == v.sizes(), "k and v must have the same shape");
  return Source{NSA_KV_DENSE, rows16(k), rows16(v), Tensor(), n_tokens < 0 ? k.size(1) : n_tokens, 0};
}
Tensor output_like(const Tensor& q, const OptTensor& given, const char* what) {
  if (!given.has_value()) return at::empty(q.sizes(), q.options());
  NEED(given->sizes() == q.sizes() && given->scalar_type() == q.scalar_type() && is_rows16(*given),
       std::string(what) + ": `out` must have q's shape and dtype, unit innermost stride and 16-byte aligned rows");
  return *given;
}

std::pair<Tensor, Tensor> sel_fwd(const Tensor& q_, const Source& kv, const OptTensor& ids_, int64_t bs, int64_t chunk, double scale, bool causal,
                                  int64_t G, const OptTensor& out_) {
  need_4d(q_, "sel_fwd q");
  const Tensor& ids = or_none(ids_);
  need_cuda({&q_, &ids});
  const Tensor q = rows16(q_);
  const c10::cuda::CUDAGuard guard(q.device());
  const int64_t B = q.size(0), M = q.size(1), H = q.size(2), D = q.size(3);
  Tensor out = output_like(q, out_, "sel_fwd");
  Tensor lse = at::empty({B, H, M}, q.options().dtype(at::kFloat));
  const Tensor& layout = kv.mode == NSA_KV_PTR ? kv.k : ids;
  NEED(layout.defined() && layout.dim() == 4, "block_indices must be [B,MG,H,T]");
  NEED(!ids.defined() || ids.scalar_type() == at::kInt, "block_indices must be int32");
  const nsa_kv_source s = kv.c();
  check("nsa_sel_fwd", nsa_sel_fwd(q.data_ptr(), Strides(q), &s, static_cast<const int32_t*>(ptr(ids)), Strides(layout), out.data_ptr(),
                                   Strides(out), lse.data_ptr<float>(), B, M, H, D, layout.size(-1), i32(bs, "block_size"),
                                   i32(chunk, "chunk_size"), causal, i32(G, "group_size"), static_cast<float>(scale), dtype_of(q), stream_of(q)));
  return {out, lse};
}

// None: the shape is not one of the range kernel's (the caller lists the blocks)
c10::optional<std::pair<Tensor, Tensor>> range_fwd(const Tensor& q_, const Source& kv, int64_t first, int64_t n, int64_t bs, double scale,
                                                   const OptTensor& out_) {
  need_4d(q_, "range_fwd q");
  need_cuda({&q_});
  const char* hook = std::getenv("OMNIMEM_B200_RANGE_KERNEL");          // test hook "listed": always list the blocks
  const int64_t B = q_.size(0), M = q_.size(1), H = q_.size(2), D = q_.size(3);
  if (q_.scalar_type() != at::kBFloat16 || D != 128 || bs != 64 || H <= 1 || !(scale > 0) || kv.mode == NSA_KV_PTR || n > 1024 ||
      kv.n_tokens <= 0 || (hook != nullptr && std::strcmp(hook, "listed") == 0))
    return c10::nullopt;
  const Tensor q = rows16(q_);
  const c10::cuda::CUDAGuard guard(q.device());
  Tensor out = output_like(q, out_, "range_fwd");
  Tensor lse = at::empty({B, H, M}, q.options().dtype(at::kFloat)), ws;
  const size_t bytes = out.is_contiguous() ? nsa_range_fwd_workspace_bytes(B, M, H, D, n) : 0;
  if (bytes) ws = scratch(bytes, q);
  const nsa_kv_source s = kv.c();
  check("nsa_range_fwd", nsa_range_fwd(q.data_ptr(), Strides(q), &s, i32(first, "first_block"), i32(n, "n_blocks"), out.data_ptr(), Strides(out),
                                       lse.data_ptr<float>(), B, M, H, D, i32(bs, "block_size"), static_cast<float>(scale), ptr(ws), bytes,
                                       dtype_of(q), stream_of(q)));
  return std::make_pair(out, lse);
}

// Size of the P / dS buffer when the backward of this call can compute them once (the dQ kernel stores, the dK/dV
// kernel streams), else 0.  16 KiB per (query group, head, slot); OMNIMEM_B200_BWD_STORED_MB caps it (default 4096,
// 0 turns the path off).
int64_t stored_bytes(const Tensor& q, int mode, int64_t T, int64_t bs, int64_t G) {
  const char* cap_s = std::getenv("OMNIMEM_B200_BWD_STORED_MB");
  const int64_t cap = cap_s != nullptr ? std::atoll(cap_s) : 4096;
  if (cap <= 0 || q.scalar_type() != at::kBFloat16 || q.size(3) != 128 || bs != 64 || G < 16 || G > 64 || q.size(2) == 1 || T > 64 ||
      mode == NSA_KV_PTR)
    return 0;
  const size_t n = nsa_sel_bwd_pds_bytes(q.size(0), q.size(1), q.size(2), T, G);
  return n > 0 && static_cast<int64_t>(n) <= cap << 20 ? static_cast<int64_t>(n) : 0;
}

std::tuple<Tensor, Tensor, Tensor> sel_bwd(const Tensor& q_, const Source& kv, const Tensor& ids, const Tensor& out_, const Tensor& lse_,
                                           const Tensor& do_, int64_t bs, int64_t chunk, double scale_, bool causal, int64_t G) {
  for (const Tensor* t : {&q_, &ids, &out_, &do_}) need_4d(*t, "sel_bwd q, ids, out, d_out");
  need_cuda({&q_, &ids, &out_, &lse_, &do_});
  const Tensor q = rows16(q_), out = rows16(out_), d_out = rows16(do_), lse = lse_.contiguous();
  NEED(ids.scalar_type() == at::kInt, "block_indices must be int32");
  const c10::cuda::CUDAGuard guard(q.device());
  const int64_t B = q.size(0), M = q.size(1), H = q.size(2), D = q.size(3), N = kv.n_tokens, T = ids.size(-1), MG = ids.size(1);
  const int32_t block = i32(bs, "block_size"), chunk32 = i32(chunk, "chunk_size"), group = i32(G, "group_size");
  const float scale = static_cast<float>(scale_);
  const int dt = dtype_of(q);
  void* st = stream_of(q);
  Tensor dq = at::empty({B, M, H, D}, q.options());
  Tensor dk = at::empty({B, N, H, D}, q.options()), dv = at::empty({B, N, H, D}, q.options());
  const nsa_kv_source s = kv.c();
  const int64_t pds_bytes = stored_bytes(q, kv.mode, T, bs, G);
  if (pds_bytes == 0 || N == 0 || M == 0) {
    const size_t wsb = nsa_sel_bwd_workspace_bytes(B, M, H, N, T, block, group);
    const Tensor ws = scratch(wsb, q);
    check("nsa_sel_bwd", nsa_sel_bwd(q.data_ptr(), Strides(q), &s, ids.data_ptr<int32_t>(), Strides(ids), out.data_ptr(), Strides(out),
                                     lse.data_ptr<float>(), d_out.data_ptr(), Strides(d_out), dq.data_ptr(), Strides(dq), dk.data_ptr(),
                                     dv.data_ptr(), B, M, H, D, T, block, chunk32, causal, group, scale, ws.data_ptr(), wsb, dt, st));
    return {dq, dk, dv};
  }
  // P and dS computed once: the dQ kernel stores them, the dK/dV kernel streams them
  const int64_t NS = ceil_div(N, bs);
  const Tensor pds = scratch(pds_bytes, q);
  Tensor delta = at::empty({B, H, M}, q.options().dtype(at::kFloat));
  const size_t idx_ws = nsa_inverted_index_workspace_bytes(B, H, NS);
  // one buffer: groups, slots, offsets, the index's workspace
  const int64_t pairs = B * H * MG * T, offs = B * H * (NS + 1);
  const Tensor idx = at::empty({2 * pairs + offs + static_cast<int64_t>(idx_ws / 4) + 256 + 64}, ids.options());
  int32_t* groups = idx.data_ptr<int32_t>();
  int32_t *slots = groups + pairs, *offsets = slots + pairs;
  auto align = [](int32_t* p) { return reinterpret_cast<int32_t*>((reinterpret_cast<uintptr_t>(p) + 255) & ~static_cast<uintptr_t>(255)); };
  int32_t* iws = align(offsets + offs);
  check("nsa_inverted_index_slots", nsa_inverted_index_slots(ids.data_ptr<int32_t>(), Strides(ids), B, MG, H, T, NS, block, chunk32, causal, group,
                                                             groups, offsets, slots, iws, idx_ws, st));
  int32_t written = 0;
  check("nsa_sel_bwd_dq_pds", nsa_sel_bwd_dq_pds(q.data_ptr(), Strides(q), &s, ids.data_ptr<int32_t>(), Strides(ids), out.data_ptr(), Strides(out),
                                                 lse.data_ptr<float>(), d_out.data_ptr(), Strides(d_out), dq.data_ptr(), Strides(dq),
                                                 delta.data_ptr<float>(), B, M, H, D, T, block, chunk32, causal, group, scale, pds.data_ptr(),
                                                 pds_bytes, &written, dt, st));
  const Tensor ws = scratch(256, q);
  check("nsa_sel_bwd_dkv_pds", nsa_sel_bwd_dkv_pds(q.data_ptr(), Strides(q), &s, groups, offsets, written ? slots : nullptr,
                                                   written ? pds.data_ptr() : nullptr, written ? pds_bytes : 0, lse.data_ptr<float>(),
                                                   delta.data_ptr<float>(), d_out.data_ptr(), Strides(d_out), dk.data_ptr(), dv.data_ptr(), B, M,
                                                   H, D, T, block, chunk32, causal, group, scale, ws.data_ptr(), 256, dt, st));
  return {dq, dk, dv};
}

// ---------------------------------------------------------------------------------- id range check
// One word of mapped pinned memory and an event per check in flight, kept for the next ones (at most kFlagsKept).
struct Flag {
  int32_t* word = nullptr;
  cudaEvent_t event = nullptr;
  int device = -1;
};
std::mutex g_flags_mutex;
std::vector<Flag> g_flags;
constexpr size_t kFlagsKept = 64;

Flag take_flag(int device) {
  {
    std::lock_guard<std::mutex> lock(g_flags_mutex);
    for (size_t i = 0; i < g_flags.size(); ++i)
      if (g_flags[i].device == device) {
        const Flag f = g_flags[i];
        g_flags.erase(g_flags.begin() + static_cast<ptrdiff_t>(i));
        return f;
      }
  }
  Flag f;
  f.device = device;
  C10_CUDA_CHECK(cudaHostAlloc(reinterpret_cast<void**>(&f.word), 64, cudaHostAllocPortable | cudaHostAllocMapped));
  C10_CUDA_CHECK(cudaEventCreateWithFlags(&f.event, cudaEventDisableTiming));
  return f;
}
void give_flag(const Flag& f) {
  {
    std::lock_guard<std::mutex> lock(g_flags_mutex);
    if (g_flags.size() < kFlagsKept) { g_flags.push_back(f); return; }
  }
  cudaEventDestroy(f.event);
  cudaFreeHost(f.word);
}
// Launched before the forward and looked at after it: the host waits while the forward is already queued (ids that
// are out of range are skipped by the kernels, so a forward that was wrong to launch does no harm).
struct IdCheck {
  Flag flag;
  bool live = false, waited = false;
  IdCheck(const Tensor& ids, int64_t limit) {
    if (ids.numel() == 0) return;
    flag = take_flag(ids.device().index());
    live = true;
    *flag.word = 0;
    check("nsa_check_block_ids", nsa_check_block_ids(ids.data_ptr<int32_t>(), ids.numel(), i32(limit, "blocks"), flag.word, stream_of(ids)));
    C10_CUDA_CHECK(cudaEventRecord(flag.event, static_cast<cudaStream_t>(stream_of(ids))));
  }
  bool bad() {
    if (!live) return false;
    C10_CUDA_CHECK(cudaEventSynchronize(flag.event));
    waited = true;
    return *static_cast<volatile int32_t*>(flag.word) != 0;
  }
  ~IdCheck() {
    // a forward that threw leaves the check in flight: its word serves no other call before it has run
    if (live && (waited || cudaEventSynchronize(flag.event) == cudaSuccess)) give_flag(flag);
  }
  IdCheck(const IdCheck&) = delete;
};

// ----------------------------------------------------------------------------------------- autograd
// The autograd engine hands a C++ exception to Python as a RuntimeError: a backward raises the package's own instead.
template <typename F> auto in_backward(F&& f) -> decltype(f()) {
  try {
    return f();
  } catch (const BackendError& e) {
    py::gil_scoped_acquire gil;
    PyErr_SetString(g_error != nullptr ? g_error : PyExc_RuntimeError, e.what());
    throw py::error_already_set();
  }
}
struct SelectionFunction : torch::autograd::Function<SelectionFunction> {
  // fp32 tensors are computed on bf16 operands with fp32 accumulation (the kernels are 16-bit; the reference's
  // default for fp32 is TF32, also a reduced-precision product) and the results are returned in fp32
  static variable_list forward(AutogradContext* ctx, Tensor q, Tensor k, Tensor v, const Tensor& ids, int64_t bs, int64_t chunk, double scale,
                               bool causal, int64_t G) {
    const auto io = q.scalar_type();
    if (io == at::kFloat) {
      q = q.to(at::kBFloat16);
      k = k.to(at::kBFloat16);
      v = v.to(at::kBFloat16);
    }
    auto r = sel_fwd(q, dense(k, v), ids, bs, chunk, scale, causal, G, c10::nullopt);
    ctx->save_for_backward({q, k, v, ids, r.first, r.second});
    ctx->saved_data["bs"] = bs;
    ctx->saved_data["chunk"] = chunk;
    ctx->saved_data["scale"] = scale;
    ctx->saved_data["causal"] = causal;
    ctx->saved_data["G"] = G;
    ctx->saved_data["io"] = static_cast<int64_t>(io);
    ctx->mark_non_differentiable({r.second});
    // (the saved tensor must not be the returned variable's alias-free copy: save_for_backward tracks outputs itself)
    return {io == at::kFloat ? r.first.to(io) : r.first, r.second};
  }
  static variable_list backward(AutogradContext* ctx, const variable_list& grads) {
    const auto s = ctx->get_saved_variables();
    const Tensor &q = s[0], &k = s[1], &v = s[2], &ids = s[3], &out = s[4], &lse = s[5];
    const auto io = static_cast<at::ScalarType>(ctx->saved_data["io"].toInt());
    auto g = in_backward([&] {
      return sel_bwd(q, dense(k, v), ids, out, lse, grads[0].to(q.scalar_type()), ctx->saved_data["bs"].toInt(),
                     ctx->saved_data["chunk"].toInt(), ctx->saved_data["scale"].toDouble(), ctx->saved_data["causal"].toBool(),
                     ctx->saved_data["G"].toInt());
    });
    const Tensor none;
    return {std::get<0>(g).to(io), std::get<1>(g).to(io), std::get<2>(g).to(io), none, none, none, none, none, none};
  }
};

// (out, lse, bad): bad says that an id was >= n_blocks (the caller words the error)
std::tuple<Tensor, Tensor, bool> selection_attention(const Tensor& q, const Tensor& k, const Tensor& v, const Tensor& ids, int64_t bs, int64_t chunk,
                                                     double scale, bool causal, int64_t G, int64_t n_blocks, bool check_ids) {
  need_cuda({&q, &k, &v, &ids});
  const c10::cuda::CUDAGuard guard(q.device());
  if (!check_ids) {
    auto r = SelectionFunction::apply(q, k, v, ids, bs, chunk, scale, causal, G);
    return {r[0], r[1], false};
  }
  IdCheck c(ids, n_blocks);
  auto r = SelectionFunction::apply(q, k, v, ids, bs, chunk, scale, causal, G);
  return {r[0], r[1], c.bad()};
}

// --------------------------------------------------------------------------------------------- gates
struct Gated {
  Tensor g, o[3], ref;
};
Gated gate_args(const Tensor& g, const Tensor& a, const Tensor& b, const Tensor& c) {
  Gated r;
  const Tensor* in[3] = {&a, &b, &c};
  for (auto* t : in)
    if (t->defined() && !r.ref.defined()) r.ref = *t;
  if (!r.ref.defined()) throw py::value_error("gate_combine: at least one branch is needed");
  need_cuda({&g, &a, &b, &c});
  const int64_t nd = r.ref.dim();
  bool ok = g.dim() == nd && g.size(-1) == 3;
  for (int64_t i = 0; ok && i + 1 < nd; ++i) ok = g.size(i) == r.ref.size(i);
  if (!ok) throw py::value_error("gate_combine: gate logits " + shape(g) + " do not match branches " + shape(r.ref));
  for (int i = 0; i < 3; ++i)
    if (in[i]->defined()) {
      if (in[i]->sizes() != r.ref.sizes() || in[i]->scalar_type() != r.ref.scalar_type())
        throw py::value_error("gate_combine: branches must share shape and dtype");
      r.o[i] = in[i]->contiguous();
    }
  if (g.scalar_type() != r.ref.scalar_type()) throw py::value_error("gate_combine: gate logits must have the branches' dtype");
  r.g = g;
  return r;
}
// logits as (token, head, 3) with one stride between tokens, if they lie that way
bool token_logits(const Tensor& g, int64_t* stride, int64_t* H) {
  const int64_t nd = g.dim();
  if (nd < 3 || g.stride(-1) != 1 || g.stride(-2) != 3) return false;
  const auto tokens = even_stride(g, nd - 2);
  if (!tokens.has_value()) return false;
  *H = g.size(-2);
  *stride = *tokens;
  return true;
}
Tensor gate_combine(const Tensor& g_, const Tensor& a, const Tensor& b, const Tensor& c, bool softmax) {
  Gated x = gate_args(g_, a, b, c);
  const c10::cuda::CUDAGuard guard(x.ref.device());
  Tensor out = at::empty(x.ref.sizes(), x.ref.options());
  const int64_t D = x.ref.size(-1), rows = x.ref.numel() / (D > 0 ? D : 1);
  int64_t stride = 3, H = 1;
  Tensor g = x.g;
  if (!token_logits(g, &stride, &H)) {
    g = g.contiguous();
    stride = 3;
    H = 1;
  }
  check("nsa_gate_combine", nsa_gate_combine_strided(g.data_ptr(), stride, ptr(x.o[0]), ptr(x.o[1]), ptr(x.o[2]), out.data_ptr(), rows / (H > 0 ? H : 1),
                                                     H > 0 ? H : 1, D, softmax, dtype_of(x.ref), stream_of(x.ref)));
  return out;
}
std::vector<OptTensor> gate_combine_bwd(const Tensor& g_, const Tensor& a, const Tensor& b, const Tensor& c, const Tensor& dx_, bool softmax) {
  Gated x = gate_args(g_, a, b, c);
  need_cuda({&dx_});
  const c10::cuda::CUDAGuard guard(x.ref.device());
  const Tensor g = x.g.contiguous(), dx = dx_.contiguous();
  Tensor dg = at::empty_like(g), d[3];
  for (int i = 0; i < 3; ++i)
    if (x.o[i].defined()) d[i] = at::empty_like(x.o[i]);
  const int64_t D = x.ref.size(-1);
  check("nsa_gate_combine_bwd", nsa_gate_combine_bwd(g.data_ptr(), ptr(x.o[0]), ptr(x.o[1]), ptr(x.o[2]), dx.data_ptr(), dg.data_ptr(), ptr(d[0]),
                                                     ptr(d[1]), ptr(d[2]), x.ref.numel() / (D > 0 ? D : 1), D, softmax, dtype_of(x.ref), stream_of(x.ref)));
  auto opt = [](const Tensor& t) { return t.defined() ? OptTensor(t) : OptTensor(); };
  return {OptTensor(dg), opt(d[0]), opt(d[1]), opt(d[2])};
}
struct GateFunction : torch::autograd::Function<GateFunction> {
  // (a skipped branch is an empty optional: an undefined tensor is not a valid input of a Function)
  static Tensor forward(AutogradContext* ctx, const Tensor& g, const OptTensor& a, const OptTensor& b, const OptTensor& c, bool softmax) {
    ctx->save_for_backward({g, or_none(a), or_none(b), or_none(c)});
    ctx->saved_data["softmax"] = softmax;
    return gate_combine(g, or_none(a), or_none(b), or_none(c), softmax);
  }
  static variable_list backward(AutogradContext* ctx, const variable_list& grads) {
    const auto s = ctx->get_saved_variables();
    auto r = in_backward([&] { return gate_combine_bwd(s[0], s[1], s[2], s[3], grads[0], ctx->saved_data["softmax"].toBool()); });
    variable_list out;
    for (auto& t : r) out.push_back(or_none(t));
    out.emplace_back();
    return out;
  }
};

// ---------------------------------------------------------------------------------- rotary embedding
struct Rope {
  Tensor f, h, w;                                   // float64 [rows, pairs, 2] tables
  int64_t grid_h, grid_w, pool_f, pool_h, pool_w, start_frame;
  nsa_rope c() const {
    nsa_rope r;
    r.freqs_f = f.data_ptr();
    r.freqs_h = h.data_ptr();
    r.freqs_w = w.data_ptr();
    r.c_f = f.size(1); r.c_h = h.size(1); r.c_w = w.size(1);
    r.grid_h = grid_h; r.grid_w = grid_w;
    r.pool_f = pool_f; r.pool_h = pool_h; r.pool_w = pool_w;
    r.start_frame = start_frame;
    return r;
  }
};

Tensor rope_apply(const Tensor& x_, const Rope& rope) {
  NEED(x_.is_cuda() && x_.dim() == 3, "rope_apply: x must be a CUDA tensor [S,H,D]");
  const Tensor x = rows16(x_);
  const c10::cuda::CUDAGuard guard(x.device());
  Tensor out = at::empty(x.sizes(), x.options());
  const nsa_rope r = rope.c();
  check("nsa_rope_apply", nsa_rope_apply(x.data_ptr(), Strides(x), x.size(0), x.size(1), x.size(2), out.data_ptr(), dtype_of(x), &r, stream_of(x)));
  return out;
}

// --------------------------------------------------------------------------------------- block cache
// The device state of a BlockKVCache; sizes that change (tokens, epoch) come with each call.
struct CacheState {
  Tensor k_pool, v_pool, table, owner, stamp, k_pooled, v_pooled, stamp32, status, counters;
  int64_t H, D, page_tokens, max_blocks;
};
void cache_append(const CacheState& c, const Tensor& k, const Tensor& v, int64_t pos0, int64_t n_tokens, int64_t epoch,
                  const OptTensor& new_pages, const Rope* rope) {
  const c10::cuda::CUDAGuard guard(c.k_pool.device());
  const int64_t S = k.size(0), first = pos0 / c.page_tokens, last = (pos0 + S - 1) / c.page_tokens;
  const int64_t st[2] = {k.stride(0), k.stride(1)};
  const int32_t* pages = static_cast<const int32_t*>(ptr(or_none(new_pages)));
  int32_t* table = c.table.data_ptr<int32_t>();
  int32_t* owner = c.owner.data_ptr<int32_t>();
  int64_t* stamp = c.stamp.data_ptr<int64_t>();
  int32_t* status = c.status.data_ptr<int32_t>();
  void* s = stream_of(c.k_pool);
  const int dt = dtype_of(c.k_pool);
  if (rope == nullptr) {
    check("nsa_cache_append", nsa_cache_append(k.data_ptr(), v.data_ptr(), st, S, pos0, n_tokens, c.H, c.D, c.k_pool.data_ptr(), c.v_pool.data_ptr(),
                                               c.page_tokens, table, c.max_blocks, pages, last - first + 1, owner, stamp, epoch,
                                               c.k_pooled.data_ptr(), c.v_pooled.data_ptr(), status, dt, s));
  } else {
    const nsa_rope r = rope->c();
    check("nsa_cache_append_rope", nsa_cache_append_rope(k.data_ptr(), v.data_ptr(), st, S, pos0, n_tokens, c.H, c.D, c.k_pool.data_ptr(),
                                                         c.v_pool.data_ptr(), c.page_tokens, table, c.max_blocks, pages, last - first + 1, owner,
                                                         stamp, epoch, c.k_pooled.data_ptr(), c.v_pooled.data_ptr(), status, dt, &r, s));
  }
}
void cache_touch(const CacheState& c, const Tensor& ids, int64_t T, int64_t epoch) {
  const c10::cuda::CUDAGuard guard(c.k_pool.device());
  check("nsa_cache_touch", nsa_cache_touch(ids.data_ptr<int32_t>(), ids.numel(), c.H, T, c.max_blocks, c.stamp32.data_ptr<int32_t>(), epoch,
                                           c.table.data_ptr<int32_t>(), c.stamp.data_ptr<int64_t>(), epoch, c.counters.data_ptr<int64_t>(),
                                           stream_of(c.k_pool)));
}

// ------------------------------------------------------------------------------------------- layers
// The kernels address every operand by x's rows: an operand that is smaller than it should be would be read past its end.
void need_like(const Tensor& t, const Tensor& x, at::ScalarType type, const char* what) {
  NEED(t.scalar_type() == type, std::string(what) + ": dtype torch." + c10::toString(t.scalar_type()) + ", expected torch." + c10::toString(type));
  NEED(t.device() == x.device(), std::string(what) + ": all tensors must be on one device");
}
// a contiguous row of d values (undefined: none)
const Tensor& need_row(const Tensor& t, const Tensor& x, at::ScalarType type, int64_t d, const char* what) {
  if (!t.defined()) return t;
  need_like(t, x, type, what);
  NEED(t.is_contiguous() && t.numel() == d, std::string(what) + ": a row of shape " + shape(t) + ", expected " + std::to_string(d) + " contiguous values");
  return t;
}
int64_t row_length(const Tensor& x, const char* what) {
  NEED(x.dim() > 0 && x.size(-1) > 0, std::string(what) + ": rows of shape " + shape(x));
  return x.size(-1);
}
// (x', h): see nsa_residual_norm.  Each vector is (rows of T, rows of fp32), either missing.
using Vec = std::pair<OptTensor, OptTensor>;
std::pair<Tensor, OptTensor> residual_norm(const Tensor& x, const OptTensor& y, const Vec& gate, const Vec& scale, const Vec& shift,
                                           bool modulated, bool norm, double eps) {
  const char* what = "residual_norm";
  const int64_t d = row_length(x, what), rows = x.numel() / d;
  if (y.has_value()) {
    NEED(y->sizes() == x.sizes(), std::string(what) + ": x of shape " + shape(x) + " and y of shape " + shape(*y));
    need_like(*y, x, x.scalar_type(), what);
  }
  const auto mod = [&](const Vec& v) -> void* { return ptr(need_row(or_none(v.first), x, x.scalar_type(), d, what)); };
  const auto f32 = [&](const Vec& v) { return static_cast<const float*>(ptr(need_row(or_none(v.second), x, at::kFloat, d, what))); };
  const void *gm = mod(gate), *sm = mod(scale), *hm = mod(shift);
  const float *ge = f32(gate), *se = f32(scale), *he = f32(shift);
  need_cuda({&x});
  const c10::cuda::CUDAGuard guard(x.device());
  const Tensor xc = x.contiguous(), yc = y.has_value() ? y->contiguous() : Tensor();
  Tensor x_out = yc.defined() ? at::empty(x.sizes(), x.options()) : xc, h;
  if (norm) h = at::empty(x.sizes(), x.options());
  check("nsa_residual_norm", nsa_residual_norm(xc.data_ptr(), ptr(yc), gm, ge, sm, se, hm, he, modulated,
                                               yc.defined() ? x_out.data_ptr() : nullptr, ptr(h), rows, d, static_cast<float>(eps),
                                               dtype_of(x), stream_of(x)));
  return {x_out, norm ? OptTensor(h) : OptTensor()};
}
// rows of the last dimension; leading dimensions must lie at one stride
Tensor rms_rows(const Tensor& x, const Tensor& weight, double eps) {
  const int64_t d = row_length(x, "rms_rows"), nd = x.dim();
  need_row(weight, x, x.scalar_type(), d, "rms_rows");
  need_cuda({&x});
  const c10::cuda::CUDAGuard guard(x.device());
  const auto stride = even_stride(x, nd - 1);
  const bool as_is = stride.has_value() && is_rows16(x);
  const Tensor xr = as_is ? x : x.contiguous();
  Tensor out = at::empty(x.sizes(), x.options().memory_format(c10::nullopt));
  check("nsa_rms_rows", nsa_rms_rows(xr.data_ptr(), as_is ? *stride : d, weight.data_ptr(), out.data_ptr(), x.numel() / d, d,
                                     static_cast<float>(eps), dtype_of(x), stream_of(x)));
  return out;
}
// q, k [S, H*D] views with a common row stride -> q' [S,H,D]; k is overwritten with k'
Tensor qk_norm_rope(const Tensor& q, const Tensor& k, const Tensor& qw, const Tensor& kw, double eps, int64_t H, const Rope& rope) {
  const char* what = "qk_norm_rope";
  NEED(q.dim() == 2 && k.sizes() == q.sizes() && H > 0 && q.size(1) % H == 0,
       std::string(what) + ": q of shape " + shape(q) + " and k of shape " + shape(k) + ", expected [S, " + std::to_string(H) + " * D]");
  need_like(k, q, q.scalar_type(), what);
  need_row(qw, q, q.scalar_type(), q.size(1), what);
  need_row(kw, q, q.scalar_type(), q.size(1), what);
  NEED(q.stride(0) == k.stride(0) && q.stride(1) == 1 && k.stride(1) == 1, "qk_norm_rope: q and k must share a row stride");
  need_cuda({&q, &rope.f, &rope.h, &rope.w});
  const c10::cuda::CUDAGuard guard(q.device());
  const int64_t S = q.size(0), D = q.size(1) / H;
  Tensor qo = at::empty({S, H, D}, q.options());
  const nsa_rope r = rope.c();
  check("nsa_qk_norm_rope", nsa_qk_norm_rope(q.data_ptr(), k.data_ptr(), q.stride(0), qw.data_ptr(), kw.data_ptr(), static_cast<float>(eps), S, H, D,
                                             qo.data_ptr(), k.data_ptr(), k.stride(0), &r, dtype_of(q), stream_of(q)));
  return qo;
}

// ------------------------------------------------------------------------- what a module's call would do
// The fused rollout layers use their sub-layers' parameters without calling them.  Two questions about that, asked for some
// thirty modules per transformer block, which costs Python 80 us and this code a few.
PyObject* dict_of(PyObject* o) {
  PyObject** d = _PyObject_GetDictPtr(o);
  return d != nullptr ? *d : nullptr;
}
const Tensor* tensor_of(PyObject* o, PyObject* parameter) {            // (not of subclasses, which may keep their values elsewhere)
  return o != nullptr && (reinterpret_cast<PyObject*>(Py_TYPE(o)) == parameter || reinterpret_cast<PyObject*>(Py_TYPE(o)) == THPVariableClass)
             ? &THPVariable_Unpack(o) : nullptr;
}
bool has_entries(PyObject* dict, PyObject* name) {
  PyObject* v = PyDict_GetItem(dict, name);
  return v != nullptr && v != Py_None && (PyDict_Check(v) ? PyDict_Size(v) != 0 : PyObject_IsTrue(v) != 0);
}
struct Names {
  PyObject *forward = PyUnicode_InternFromString("forward"), *hooks = PyUnicode_InternFromString("_forward_hooks"),
           *pre_hooks = PyUnicode_InternFromString("_forward_pre_hooks"), *compiled = PyUnicode_InternFromString("_compiled_call_impl"),
           *params = PyUnicode_InternFromString("_parameters"), *weight = PyUnicode_InternFromString("weight"),
           *bias = PyUnicode_InternFromString("bias");
};
const Names& names() {
  static const Names n;
  return n;
}
// Whether every module is exactly of its kind, untouched (no hooks, no forward of its own, its class's forward is the one in
// `table`, not compiled) and has the parameters its kind is built with, of type `dtype`.  table: {class: (forward, kind of
// parameters)}: 0 none, 1 a weight and perhaps a bias, 2 a weight that the row kernels can read as it lies, 3 and a bias.
bool plain(const py::tuple& mods, const py::tuple& kinds, const py::dict& table, py::handle parameter, at::ScalarType dtype) {
  const Names& n = names();
  const auto row = [&](const Tensor* t) {
    return t != nullptr && t->scalar_type() == dtype && t->is_contiguous() && reinterpret_cast<uintptr_t>(t->const_data_ptr()) % 16 == 0;
  };
  for (size_t i = 0; i < mods.size(); ++i) {
    PyObject *m = mods[i].ptr(), *type = reinterpret_cast<PyObject*>(Py_TYPE(m)), *entry = PyDict_GetItem(table.ptr(), type);
    if (type != kinds[i].ptr() || entry == nullptr) return false;
    const py::object now = py::reinterpret_steal<py::object>(PyObject_GetAttr(type, n.forward));
    PyObject* d = dict_of(m);
    if (!now || now.ptr() != PyTuple_GET_ITEM(entry, 0) || d == nullptr || PyDict_Contains(d, n.forward) != 0) {
      PyErr_Clear();
      return false;
    }
    if (has_entries(d, n.hooks) || has_entries(d, n.pre_hooks) || has_entries(d, n.compiled)) return false;
    const long kind = PyLong_AsLong(PyTuple_GET_ITEM(entry, 1));
    if (kind == 0) continue;
    PyObject* params = PyDict_GetItem(d, n.params);
    if (params == nullptr) return false;
    PyObject *w = PyDict_GetItem(params, n.weight), *b = PyDict_GetItem(params, n.bias);
    const Tensor* weight = tensor_of(w, parameter.ptr());
    if (kind == 1) {
      const Tensor* bias = tensor_of(b, parameter.ptr());
      if (weight == nullptr || weight->scalar_type() != dtype) return false;
      if (b != nullptr && b != Py_None && (bias == nullptr || bias->scalar_type() != dtype)) return false;
    } else if (!row(weight) || (kind == 3 && !row(tensor_of(b, parameter.ptr())))) {
      return false;
    }
  }
  return true;
}
// Whether the modules' weights and biases still lie one below the other in the two tensors of `whole` (whose storage is
// kept, so that an equal address is a view of it).
bool joined(const py::tuple& mods, const py::tuple& whole, py::handle parameter) {
  for (int k = 0; k < 2; ++k) {
    const Tensor& t = THPVariable_Unpack(whole[k].ptr());
    const char* at = static_cast<const char*>(t.const_data_ptr());
    for (const py::handle m : mods) {
      PyObject* d = dict_of(m.ptr());
      PyObject* params = d != nullptr ? PyDict_GetItem(d, names().params) : nullptr;
      const Tensor* p = params != nullptr ? tensor_of(PyDict_GetItem(params, k == 0 ? names().weight : names().bias), parameter.ptr()) : nullptr;
      if (p == nullptr || p->const_data_ptr() != at || p->scalar_type() != t.scalar_type() || !p->is_contiguous()) return false;
      at += p->nbytes();
    }
  }
  return true;
}

}  // namespace

PYBIND11_MODULE(_host, m) {
  // a launch may block on a full queue, and the id check waits: other Python threads run meanwhile
  using nogil = py::call_guard<py::gil_scoped_release>;
  m.def("set_error", [](py::object e) { g_error = e.release().ptr(); });
  py::register_exception_translator([](std::exception_ptr p) {
    try {
      if (p) std::rethrow_exception(p);
    } catch (const BackendError& e) {
      PyErr_SetString(g_error != nullptr ? g_error : PyExc_RuntimeError, e.what());
    }
  });
  py::class_<Source>(m, "Source")
      .def_readonly("mode", &Source::mode)
      .def_readonly("k", &Source::k)
      .def_readonly("v", &Source::v)
      .def_readonly("n_tokens", &Source::n_tokens);
  m.def("dense", &dense, nogil(), py::arg("k"), py::arg("v"), py::arg("n_tokens") = -1);
  m.def("paged", [](const Tensor& k, const Tensor& v, const Tensor& table, int64_t n_tokens, int64_t page_tokens) {
    need_cuda({&k, &v, &table});
    return Source{NSA_KV_PAGED, k, v, table, n_tokens, page_tokens};
  });
  m.def("pointers", [](const Tensor& k, const Tensor& v, int64_t stride_bn) {
    need_cuda({&k, &v});
    return Source{NSA_KV_PTR, k, v, Tensor(), stride_bn, 0};
  });
  m.def("even_stride", &even_stride);
  m.def("same_bytes", &same_bytes, nogil());
  m.def("pool_rows", &pool_rows, nogil());
  m.def("topk", &topk, nogil());
  m.def("select_blocks", &select_blocks, nogil());
  m.def("sel_fwd", &sel_fwd, nogil(), py::arg("q"), py::arg("kv"), py::arg("ids"), py::arg("block_size"), py::arg("chunk_size"), py::arg("scale"),
        py::arg("causal"), py::arg("group_size"), py::arg("out") = py::none());
  m.def("range_fwd", &range_fwd, nogil());
  m.def("stored_bytes", &stored_bytes);
  m.def("sel_bwd", &sel_bwd, nogil());
  m.def("selection_attention", &selection_attention, nogil());
  m.def("gate_combine", [](const Tensor& g, const OptTensor& a, const OptTensor& b, const OptTensor& c, bool softmax) {
    return gate_combine(g, or_none(a), or_none(b), or_none(c), softmax);
  }, nogil());
  m.def("gate_combine_bwd", [](const Tensor& g, const OptTensor& a, const OptTensor& b, const OptTensor& c, const Tensor& dx, bool softmax) {
    return gate_combine_bwd(g, or_none(a), or_none(b), or_none(c), dx, softmax);
  }, nogil());
  m.def("gated_sum", [](const Tensor& g, const OptTensor& a, const OptTensor& b, const OptTensor& c, bool softmax) {
    return GateFunction::apply(g, a, b, c, softmax);
  }, nogil());
  py::class_<Rope>(m, "Rope").def(py::init([](const Tensor& f, const Tensor& h, const Tensor& w, int64_t gh, int64_t gw, int64_t pf, int64_t ph,
                                              int64_t pw, int64_t start) { return Rope{f, h, w, gh, gw, pf, ph, pw, start}; }));
  m.def("rope_apply", &rope_apply, nogil());
  py::class_<CacheState>(m, "CacheState").def(py::init([](std::vector<Tensor> t, int64_t H, int64_t D, int64_t page_tokens, int64_t max_blocks) {
    NEED(t.size() == 10, "CacheState: ten tensors are expected");
    return CacheState{t[0], t[1], t[2], t[3], t[4], t[5], t[6], t[7], t[8], t[9], H, D, page_tokens, max_blocks};
  }));
  m.def("cache_append", &cache_append, nogil());
  m.def("cache_touch", &cache_touch, nogil());
  m.def("plain", &plain);
  m.def("joined", &joined);
  m.def("residual_norm", &residual_norm, nogil());
  m.def("rms_rows", &rms_rows, nogil());
  m.def("qk_norm_rope", &qk_norm_rope, nogil());
}

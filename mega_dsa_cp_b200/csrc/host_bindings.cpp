// Host side of the tile runners: reads the tensors' addresses and shapes, checks them, fills the C-ABI
// parameter struct and calls the launcher in libmdc.so.
//
// The runners in tiles/*.py are called once per layer and step on buffers of a few microseconds of device
// work, and building a ctypes struct field by field took longer than that (10-24 us per call against 3-5 us
// here, launch included).  The Python functions keep the signatures; a failed check raises AssertionError.
//
// The launchers' addresses come from the library that _native.py loaded (bind), so there is one libmdc.so.
#include <ATen/cuda/CUDAContext.h>
#include <c10/cuda/CUDAStream.h>
#include <torch/csrc/autograd/python_variable.h>

#include "../../include/mdc.h"

namespace {

struct Entries {
  int (*logits)(const mdc_logits_params*, void*);
  int (*merge_topk)(const mdc_merge_topk_params*, void*);
  int (*lse_merge)(const mdc_lse_merge_params*, void*);
  int (*sparse_mla)(const mdc_sparse_mla_params*, void*);
  int (*sparse_mla_static_ws)(const mdc_sparse_mla_params*, void*);
  int (*compress_step)(const mdc_compress_params*, void*);
  int (*compress_finalize)(const mdc_compress_params*, void*);
  int (*megakernel)(const mdc_mega_params*, void*);
  int (*causal_lens)(const int64_t*, int32_t*, int32_t, int32_t, int32_t, void*);
} entries;

struct Failed {};   // a Python error has been set

[[noreturn]] void fail(PyObject* type, const char* what) {
  PyErr_SetString(type, what);
  throw Failed{};
}
void require(bool ok, const char* what) {
  if (!ok) fail(PyExc_AssertionError, what);
}

// nullptr for None
const at::Tensor* tensor(PyObject* o) {
  if (o == Py_None) return nullptr;
  if (!THPVariable_Check(o)) fail(PyExc_TypeError, "expected a tensor or None");
  return &THPVariable_Unpack(o);
}
const at::Tensor& tensor_of(PyObject* o) {
  const at::Tensor* t = tensor(o);
  if (!t) fail(PyExc_TypeError, "expected a tensor");
  return *t;
}
template <typename T = void>
T* ptr(const at::Tensor* t) {
  return t ? static_cast<T*>(t->data_ptr()) : nullptr;
}
int64_t integer(PyObject* o) {
  const int64_t v = PyLong_AsLongLong(o);
  if (v == -1 && PyErr_Occurred()) throw Failed{};
  return v;
}
double real(PyObject* o) {
  const double v = PyFloat_AsDouble(o);
  if (v == -1.0 && PyErr_Occurred()) throw Failed{};
  return v;
}
// None = the current stream; else a raw handle
void* stream_of(PyObject* o) {
  return o == Py_None ? static_cast<void*>(at::cuda::getCurrentCUDAStream().stream()) : reinterpret_cast<void*>(integer(o));
}
template <typename Fn, typename P>
PyObject* launch(Fn fn, const P& p, void* stream) {
  int rc;
  Py_BEGIN_ALLOW_THREADS;
  rc = fn(&p, stream);
  Py_END_ALLOW_THREADS;
  return PyLong_FromLong(rc);
}
// FASTCALL wrapper: argument count, and C++ exceptions -> Python errors
template <int N, PyObject* (*F)(PyObject* const*)>
PyObject* entry(PyObject*, PyObject* const* a, Py_ssize_t n) {
  if (n != N) {
    PyErr_Format(PyExc_TypeError, "expected %d arguments, got %zd", N, n);
    return nullptr;
  }
  try {
    return F(a);
  } catch (const Failed&) {
    return nullptr;
  } catch (const std::exception& e) {
    PyErr_SetString(PyExc_RuntimeError, e.what());
    return nullptr;
  }
}

int dtype_code(const at::Tensor& t) {   // fp32 / bf16 outputs and partials
  if (t.scalar_type() == at::kFloat) return MDC_DT_F32;
  if (t.scalar_type() == at::kBFloat16) return MDC_DT_BF16;
  fail(PyExc_KeyError, "dtype must be float32 or bfloat16");
}

PyObject* bind(PyObject* const* a) {
  void** slots = reinterpret_cast<void**>(&entries);
  for (size_t i = 0; i < sizeof(entries) / sizeof(void*); ++i)
    slots[i] = reinterpret_cast<void*>(integer(PyTuple_GetItem(a[0], static_cast<Py_ssize_t>(i))));
  Py_RETURN_NONE;
}

// kv, q, q_sf, w, table, logits, blocks_per_chunk, seq_lens, cand_v, cand_i, cand_c, stream, top_k, mxfp4, page_tokens,
// window_exclude, id_mul, id_add, status, row_v, row_i, row_c
PyObject* logits(PyObject* const* a) {
  const at::Tensor &kv = tensor_of(a[0]), &q = tensor_of(a[1]), &w = tensor_of(a[3]), &bt = tensor_of(a[4]);
  const at::Tensor *q_sf = tensor(a[2]), *out = tensor(a[5]), *lens = tensor(a[7]), *cv = tensor(a[8]), *ci = tensor(a[9]),
                   *cc = tensor(a[10]), *status = tensor(a[18]), *rv = tensor(a[19]), *ri = tensor(a[20]), *rc = tensor(a[21]);
  constexpr int64_t kHeads = 64;
  const int64_t B = q.size(0), rows = q.size(1), T = rows / kHeads, bpc = integer(a[6]), top_k = integer(a[12]);
  const bool mxfp4 = integer(a[13]) != 0, fused = cv != nullptr, row = rv != nullptr;
  const int64_t page = integer(a[14]), max_pages = bt.size(1);
  require(rows == T * kHeads, "query rows must be q_len * 64");
  if (row) require(rv->size(-1) == top_k && ri && ri->sizes() == rv->sizes() && rv->is_contiguous(), "row_topk tensors");
  require(bpc >= 1, "blocks_per_chunk must be positive");
  const int64_t n_chunks = max_pages / bpc + (max_pages % bpc != 0);
  for (const at::Tensor* t : {&kv, &q, &w, &bt}) require(t->is_cuda() && t->is_contiguous(), "inputs must be contiguous CUDA tensors");
  require(bt.scalar_type() == at::kInt && w.scalar_type() == at::kFloat, "block_table is int32, weights are float32");
  require(kv.size(1) == page * 64 + page * (mxfp4 ? 4 : 8), "page size does not match fmt/page_tokens");
  if (!row && fused) {
    require(ci && cc && cv->dim() == 4 && cv->size(0) == B && cv->size(1) == T && cv->size(2) == n_chunks && cv->size(3) == top_k &&
                ci->sizes() == cv->sizes() && cc->dim() == 3 && cc->size(0) == B && cc->size(1) == T && cc->size(2) == n_chunks,
            "candidate buffers");
  } else if (!row) {
    require(out && out->size(0) == B * T && out->size(1) >= max_pages * page && out->stride(1) == 1, "logits buffer");
  }
  mdc_logits_params p{};
  p.kv_pages = ptr<uint8_t>(&kv);
  p.num_pages = static_cast<int32_t>(kv.size(0));
  p.page_tokens = static_cast<int32_t>(page);
  p.fmt = mxfp4 ? MDC_FMT_MXFP4 : MDC_FMT_NVFP4;
  p.q_fmt = q.scalar_type() == at::kBFloat16 ? MDC_Q_BF16 : MDC_Q_FP4;
  p.q = q.data_ptr();
  p.q_sf = ptr<uint8_t>(q_sf);
  p.weights = ptr<float>(&w);
  p.block_table = ptr<int32_t>(&bt);
  p.max_pages = static_cast<int32_t>(max_pages);
  p.seq_lens = ptr<int32_t>(lens);
  if (!row && !fused) {
    p.logits = ptr<float>(out);
    p.logits_stride = out->stride(0);
  }
  p.cand_v = ptr<float>(cv);
  p.cand_i = ptr<int32_t>(ci);
  p.cand_c = ptr<int32_t>(cc);
  p.top_k = static_cast<int32_t>(top_k);
  p.B = static_cast<int32_t>(B);
  p.q_len = static_cast<int32_t>(T);
  p.heads = kHeads;
  p.blocks_per_chunk = static_cast<int32_t>(bpc);
  p.n_chunks = static_cast<int32_t>(n_chunks);
  p.window_exclude = a[15] == Py_None ? (mxfp4 && (fused || row) ? 128 : 0) : static_cast<int32_t>(integer(a[15]));
  p.id_mul = static_cast<int32_t>(integer(a[16]));
  p.id_add = static_cast<int32_t>(integer(a[17]));
  p.status = ptr<int32_t>(status);
  p.row_v = ptr<float>(rv);
  p.row_i = ptr<int32_t>(ri);
  p.row_c = ptr<int32_t>(rc);
  return launch(entries.logits, p, stream_of(a[11]));
}

// cand_v, cand_i, cand_c, out_v, out_i, out_c, dbg, stream, top_k
PyObject* merge_topk(PyObject* const* a) {
  const at::Tensor* t[6];
  for (int i = 0; i < 6; ++i) {
    t[i] = &tensor_of(a[i]);
    require(t[i]->is_cuda() && t[i]->is_contiguous(), "candidate and output tensors must be contiguous CUDA tensors");
  }
  require(t[0]->dim() == 4, "cand_v is (B, q_len, L, maxK)");
  mdc_merge_topk_params p{};
  p.cand_v = ptr<float>(t[0]);
  p.cand_i = ptr<int32_t>(t[1]);
  p.cand_c = ptr<int32_t>(t[2]);
  p.out_v = ptr<float>(t[3]);
  p.out_i = ptr<int32_t>(t[4]);
  p.out_c = ptr<int32_t>(t[5]);
  p.dbg = ptr<int32_t>(tensor(a[6]));
  p.B = static_cast<int32_t>(t[0]->size(0));
  p.q_len = static_cast<int32_t>(t[0]->size(1));
  p.L = static_cast<int32_t>(t[0]->size(2));
  p.maxK = static_cast<int32_t>(t[0]->size(3));
  p.top_k = static_cast<int32_t>(integer(a[8]));
  require(p.L <= 256 && t[3]->size(-1) == p.top_k, "at most 256 lists, out_v holds top_k entries");
  return launch(entries.merge_topk, p, stream_of(a[7]));
}

// acc_o, acc_lse, o, lse, cp, stream
PyObject* lse_merge(PyObject* const* a) {
  const at::Tensor &acc = tensor_of(a[0]), &acc_l = tensor_of(a[1]), &o = tensor_of(a[2]);
  const at::Tensor* lse = tensor(a[3]);
  require(acc.dim() == 5, "acc_o is (B, q_len, cp_max, H, D)");
  for (const at::Tensor* t : {&acc, &acc_l, &o}) require(t->is_cuda() && t->is_contiguous(), "partials and output must be contiguous CUDA tensors");
  const int64_t B = acc.size(0), T = acc.size(1), n = acc.size(2), heads = acc.size(3), D = acc.size(4);
  require(acc_l.scalar_type() == at::kFloat && acc_l.sizes() == at::IntArrayRef({B, T, n, heads}), "acc_lse");
  require(o.sizes() == at::IntArrayRef({B, T, heads, D}), "o");
  mdc_lse_merge_params p{};
  p.acc_o = acc.data_ptr();
  p.acc_lse = ptr<float>(&acc_l);
  p.o = o.data_ptr();
  p.lse = ptr<float>(lse);
  p.rows = static_cast<int32_t>(B * T);
  p.H = static_cast<int32_t>(heads);
  p.D = static_cast<int32_t>(D);
  p.n_slices = static_cast<int32_t>(integer(a[4]));
  p.n_slices_max = static_cast<int32_t>(n);
  p.acc_dtype = dtype_code(acc);
  p.out_dtype = dtype_code(o);
  return launch(entries.lse_merge, p, stream_of(a[5]));
}

// q, kv_win, kv_cmp, pt_win, pt_cmp, o, lse, k_valid, win_valid, attn_sink, softmax_scale, output_scale, n_splits, fp8_p,
// status, stream, ws_o, ws_lse
PyObject* sparse_mla(PyObject* const* a) {
  const at::Tensor &q = tensor_of(a[0]), &kv = tensor_of(a[2]), &pt = tensor_of(a[4]), &o = tensor_of(a[5]), &k_valid = tensor_of(a[7]);
  const at::Tensor *kv_win = tensor(a[1]), *pt_win = tensor(a[3]), *lse = tensor(a[6]), *win_valid = tensor(a[8]), *sink = tensor(a[9]),
                   *status = tensor(a[14]), *ws_o = tensor(a[16]), *ws_l = tensor(a[17]);
  constexpr int64_t kDv = 512;
  require(q.dim() == 4, "q is (B, T, H, d_qk)");
  const int64_t B = q.size(0), T = q.size(1), heads = q.size(2), rows = B * T;
  require(kv.scalar_type() == q.scalar_type() && kv.is_contiguous() && q.is_contiguous(), "q and kv_cmp: one dtype, contiguous");
  // elements between the rows of o, and from its first to behind its last
  int64_t o_stride, room;
  const int64_t dv = o.size(-1);
  if (o.dim() == 4 && o.is_contiguous()) {
    o_stride = heads * dv;
    room = o.numel();
    require(room == rows * o_stride, "o is (B, T, H, 512)");
  } else {
    const at::Tensor o2 = o.dim() == 4 ? o.view({rows, heads, dv}) : o;
    require(o2.dim() == 3 && o2.stride(2) == 1 && o2.stride(1) == o2.size(2), "the heads of a row of o must be contiguous");
    o_stride = o2.stride(0);
    room = o2.size(0) > 0 ? (o2.size(0) - 1) * o_stride + o2.size(1) * o2.size(2) : 0;
  }
  require(rows == 0 || (rows - 1) * o_stride + heads * kDv <= room, "o does not hold the output rows");
  require(!lse || lse->numel() == rows * heads, "lse is (B, T, H)");
  // KV splits so that rows * heads / 64 * splits blocks roughly fill the SMs
  int64_t n_splits;
  if (a[12] == Py_None) {
    const int64_t slots = pt.size(1) * kv.size(1) + 128, tiles = std::max<int64_t>(1, (slots + 63) / 64);
    const int64_t sms = at::cuda::getDeviceProperties(q.get_device())->multiProcessorCount;
    n_splits = std::max<int64_t>(1, std::min({int64_t{16}, tiles, sms / std::max<int64_t>(1, rows * (heads / 64))}));
  } else {
    n_splits = integer(a[12]);
  }
  if (o_stride != heads * dv || (lse && !lse->is_contiguous())) n_splits = 1;
  bool static_ws = false;
  if (n_splits > 1 && ws_o) {
    require(ws_o->scalar_type() == at::kFloat && ws_o->numel() >= rows * n_splits * heads * kDv, "split workspace: partials");
    require(ws_l && ws_l->scalar_type() == at::kFloat && ws_l->numel() >= rows * n_splits * heads, "split workspace: LSEs");
  } else if (n_splits > 1) {
    const int64_t per_split = std::max<int64_t>(1, rows * heads);   // (the launcher refuses an empty batch)
    n_splits = std::max<int64_t>(1, std::min<int64_t>(n_splits, MDC_STATIC_WS_MAX_SLOTS / per_split));
    static_ws = n_splits > 1;
  }
  mdc_sparse_mla_params p{};
  p.q = q.data_ptr();
  p.kv_win = ptr(kv_win);
  p.kv_cmp = kv.data_ptr();
  p.pt_win = ptr<int32_t>(pt_win);
  p.pt_cmp = ptr<int32_t>(&pt);
  p.k_valid = ptr<int32_t>(&k_valid);
  p.win_valid = ptr<int32_t>(win_valid);
  p.attn_sink = ptr<float>(sink);
  p.o = o.data_ptr();
  p.lse = ptr<float>(lse);
  p.o_stride = o_stride;
  p.lse_stride = !lse || lse->is_contiguous() ? heads : lse->reshape({rows, heads}).stride(0);
  p.ws_o = n_splits > 1 && !static_ws ? ptr<float>(ws_o) : nullptr;
  p.ws_lse = n_splits > 1 && !static_ws ? ptr<float>(ws_l) : nullptr;
  p.B = static_cast<int32_t>(B);
  p.q_len = static_cast<int32_t>(T);
  p.H = static_cast<int32_t>(heads);
  p.d_qk = static_cast<int32_t>(q.size(3));
  p.d_v = kDv;
  p.pages_win = kv_win ? static_cast<int32_t>(kv_win->size(0)) : 0;
  p.pages_cmp = static_cast<int32_t>(kv.size(0));
  p.page_cmp = static_cast<int32_t>(kv.size(1));
  p.pt_cols = static_cast<int32_t>(pt.size(1));
  p.kv_dtype = q.scalar_type() == at::kFloat8_e4m3fn ? MDC_DT_E4M3 : MDC_DT_BF16;
  p.out_dtype = o.scalar_type() == at::kFloat ? MDC_DT_F32 : MDC_DT_BF16;
  p.n_splits = static_cast<int32_t>(n_splits);
  p.fp8_p = integer(a[13]) != 0;
  p.softmax_scale = static_cast<float>(real(a[10]));
  p.output_scale = static_cast<float>(real(a[11]));
  p.status = ptr<int32_t>(status);
  return launch(static_ws ? entries.sparse_mla_static_ws : entries.sparse_mla, p, stream_of(a[15]));
}

// ---- compressor: the state, arena and event objects are read by attribute, each held while it is read
struct Ref {
  PyObject* o;
  explicit Ref(PyObject* x) : o(x) {
    if (!o) throw Failed{};
  }
  Ref(const Ref&) = delete;
  ~Ref() { Py_DECREF(o); }
};
Ref get(PyObject* o, const char* name) { return Ref(PyObject_GetAttrString(o, name)); }
int64_t get_int(PyObject* o, const char* name) { return integer(get(o, name).o); }
template <typename T = void>
T* get_ptr(PyObject* o, const char* name) {
  const Ref r = get(o, name);
  return ptr<T>(tensor(r.o));
}

void fill_compress(mdc_compress_params& p, PyObject* st, const at::Tensor& seq_len, PyObject* arena, PyObject* region, PyObject* events,
                   int64_t ev_base_id, int64_t phase, bool do_push, int64_t wait_budget_ns) {
  p.B = static_cast<int32_t>(get_int(st, "B"));
  p.cp = static_cast<int32_t>(get_int(st, "cp"));
  p.rank = static_cast<int32_t>(get_int(st, "rank"));
  p.q_len = static_cast<int32_t>(get_int(st, "q_len"));
  p.ratio = static_cast<int32_t>(get_int(st, "ratio"));
  p.phase = static_cast<int32_t>(phase);
  p.seq_len = ptr<int32_t>(&seq_len);
  p.ring_attn = get_ptr<float>(st, "ring_attn");
  p.ring_idx = get_ptr<float>(st, "ring_idx");
  p.state = get_ptr<float>(st, "state");
  p.arena = mdc_peer_buffer{get_ptr(arena, "tensor"), get_ptr<int64_t>(arena, "offsets"),
                            static_cast<int32_t>(get_int(arena, "rank")), static_cast<int32_t>(get_int(arena, "world_size")),
                            get_int(arena, "mc_base")};
  const Ref regions = get(arena, "regions");
  p.stats_off = integer(Ref(PyObject_GetItem(regions.o, region)).o);
  p.events = mdc_event_set{get_ptr(events, "tensor"), get_ptr<int64_t>(events, "offsets"),
                           static_cast<int32_t>(get_int(events, "rank")), static_cast<int32_t>(get_int(events, "world_size"))};
  p.ev_base_id = static_cast<int32_t>(ev_base_id);
  p.do_push = do_push;
  p.wait_budget_ns = wait_budget_ns;
  p.status = get_ptr<int32_t>(st, "status");
}

// st, seq_len, new_attn, new_idx, ape_attn, ape_idx, arena, stats_region, events, ev_base_id, do_push, stream
PyObject* compress_step(PyObject* const* a) {
  mdc_compress_params p{};
  fill_compress(p, a[0], tensor_of(a[1]), a[6], a[7], a[8], integer(a[9]), 0, integer(a[10]) != 0, 2000000000);
  p.new_attn = ptr<float>(tensor(a[2]));
  p.new_idx = ptr<float>(tensor(a[3]));
  p.ape_attn = ptr<float>(tensor(a[4]));
  p.ape_idx = ptr<float>(tensor(a[5]));
  return launch(entries.compress_step, p, stream_of(a[11]));
}

// st, seq_len, arena, stats_region, events, phase, norm_w_attn, norm_w_idx, norm_eps, freqs, fp8_scale, ev_base_id,
// wait_budget_ns, stream, mxfp4 index entries
PyObject* compress_finalize(PyObject* const* a) {
  mdc_compress_params p{};
  PyObject* st = a[0];
  fill_compress(p, st, tensor_of(a[1]), a[2], a[3], a[4], integer(a[11]), integer(a[5]), true, integer(a[12]));
  const at::Tensor& freqs = tensor_of(a[9]);
  const Ref attn_pool = get(st, "attn_pool");
  const at::Tensor& pool = tensor_of(attn_pool.o);
  p.norm_w_attn = ptr<float>(tensor(a[6]));
  p.norm_w_idx = ptr<float>(tensor(a[7]));
  p.freqs = ptr<float>(&freqs);
  p.freq_rows = static_cast<int32_t>(freqs.size(0));
  p.norm_eps = static_cast<float>(real(a[8]));
  const double fp8_scale = real(a[10]);
  if (fp8_scale == 0.0) fail(PyExc_ZeroDivisionError, "fp8_scale must not be zero");
  p.inv_fp8_scale = static_cast<float>(1.0 / fp8_scale);
  p.attn_pool_dtype = pool.scalar_type() == at::kFloat8_e4m3fn ? MDC_DT_E4M3 : MDC_DT_BF16;
  p.attn_pool = pool.data_ptr();
  p.idx_pool = get_ptr<uint8_t>(st, "idx_pool");
  p.idx_fmt = integer(a[14]) ? MDC_FMT_MXFP4 : MDC_FMT_NVFP4;
  p.idx_page_tokens = static_cast<int32_t>(get_int(st, "idx_page_tokens"));
  p.max_entries = static_cast<int32_t>(get_int(st, "max_entries"));
  p.k_valid = get_ptr<int32_t>(st, "k_valid");
  p.dbg_attn = get_ptr<float>(st, "dbg_attn");
  p.dbg_idx = get_ptr<float>(st, "dbg_idx");
  return launch(entries.compress_finalize, p, stream_of(a[13]));
}

// address of an mdc_mega_params, address of the launch's mdc_layer_params (0: the one inside), stream, address and entries
// of its trace, its wait budget (None: the one inside).  The block is read here, under the interpreter's lock: threads that
// launch share it.
PyObject* megakernel(PyObject* const* a) {
  mdc_mega_params p = *reinterpret_cast<const mdc_mega_params*>(integer(a[0]));
  if (const int64_t layer = integer(a[1])) p.layer = *reinterpret_cast<const mdc_layer_params*>(layer);
  p.trace = reinterpret_cast<unsigned long long*>(integer(a[3]));
  p.trace_cap = static_cast<int32_t>(integer(a[4]));
  if (a[5] != Py_None) p.wait_budget_ns = integer(a[5]);
  return launch(entries.megakernel, p, stream_of(a[2]));
}

// ---- chunked prefill: addresses of a chunk's tensors in the launch parameters (prefill.py)
struct Span {
  uintptr_t lo, hi;
};
Span span_of(const at::Tensor& t) {   // the memory that a tensor may touch
  if (t.is_contiguous()) {
    const uintptr_t at = reinterpret_cast<uintptr_t>(t.data_ptr());
    return {at, at + t.nbytes()};
  }
  const uintptr_t at = reinterpret_cast<uintptr_t>(t.storage().data());
  return {at, at + t.storage().nbytes()};
}
PyObject* item(PyObject* tuple, Py_ssize_t i) {   // borrowed
  PyObject* o = PyTuple_GetItem(tuple, i);
  if (!o) throw Failed{};
  return o;
}
constexpr int kResults = 4;   // out, out_lse (a row per owned query token), sel_i, sel_c (a row per query token)
int64_t tokens_per_row(int result, int64_t cp) { return result < 2 ? cp : 1; }

// positions (int64), lens (int32), cp, rank, stream
PyObject* causal_lens(PyObject* const* a) {
  const at::Tensor &pos = tensor_of(a[0]), &lens = tensor_of(a[1]);
  require(pos.scalar_type() == at::kLong && lens.scalar_type() == at::kInt && pos.is_contiguous() && lens.is_contiguous() &&
              pos.numel() == lens.numel(), "one int32 length per int64 position");
  const int64_t cp = integer(a[2]), rank = integer(a[3]);
  void* stream = stream_of(a[4]);
  int rc;
  Py_BEGIN_ALLOW_THREADS;
  rc = entries.causal_lens(ptr<int64_t>(&pos), ptr<int32_t>(&lens), static_cast<int32_t>(pos.numel()), static_cast<int32_t>(cp),
                           static_cast<int32_t>(rank), stream);
  Py_END_ALLOW_THREADS;
  return PyLong_FromLong(rc);
}

// The results that a chunk's launches can write straight into the caller's tensors, as a bit mask: rows of the shape, type
// and device of the layer's own buffers, contiguous, on the 16-byte boundary that the kernels' stores need, and clear of the
// memory of what the launches read.
// tensors read, results (None: not asked for), the layer's own buffers, query tokens, cp
PyObject* prefill_targets(PyObject* const* a) {
  const Py_ssize_t n_reads = PyTuple_Size(a[0]);
  if (n_reads < 0) throw Failed{};
  const int64_t tokens = integer(a[3]), cp = integer(a[4]);
  Span reads[8];
  require(n_reads <= 8 && cp >= 1, "prefill_targets");
  for (Py_ssize_t i = 0; i < n_reads; ++i) reads[i] = span_of(tensor_of(item(a[0], i)));
  long mask = 0;
  for (int r = 0; r < kResults; ++r) {
    const at::Tensor *t = tensor(item(a[1], r)), &like = tensor_of(item(a[2], r));
    if (!t || t->scalar_type() != like.scalar_type() || t->device() != like.device() || t->dim() != like.dim() || !t->is_contiguous()) continue;
    if (t->sizes().slice(1) != like.sizes().slice(1) || t->size(0) < tokens / tokens_per_row(r, cp)) continue;
    const Span s = span_of(*t);
    bool clear = s.lo % 16 == 0;
    for (Py_ssize_t i = 0; i < n_reads; ++i) clear = clear && (s.hi <= reads[i].lo || reads[i].hi <= s.lo);
    if (clear) mask |= 1l << r;
  }
  return PyLong_FromLong(mask);
}

// address of the mdc_layer_params to fill, address of the layer's on its caches, causal lengths, q_idx (None: the queries
// are staged), w_idx, q_mla, first query token of the launch, cp, results, mask of prefill_targets
PyObject* prefill_fill(PyObject* const* a) {
  mdc_layer_params& L = *reinterpret_cast<mdc_layer_params*>(integer(a[0]));
  L = *reinterpret_cast<const mdc_layer_params*>(integer(a[1]));
  const int64_t t0 = integer(a[6]), cp = integer(a[7]), mask = integer(a[9]);
  auto row = [](const at::Tensor& t, int64_t i) { return static_cast<char*>(t.data_ptr()) + i * t.stride(0) * t.element_size(); };
  L.logits.seq_lens = reinterpret_cast<int32_t*>(row(tensor_of(a[2]), t0));
  if (const at::Tensor* q = tensor(a[3])) {
    L.logits.q = row(*q, t0);
    L.logits.weights = reinterpret_cast<float*>(row(tensor_of(a[4]), t0));
    L.mla.q = row(tensor_of(a[5]), t0);
  }
  void* at[kResults] = {};
  for (int r = 0; r < kResults; ++r)
    if ((mask >> r) & 1) at[r] = row(tensor_of(item(a[8], r)), t0 / tokens_per_row(r, cp));
  if (at[0]) L.out = at[0];
  if (at[1]) L.out_lse = static_cast<float*>(at[1]);
  if (at[2]) L.sel_i = static_cast<int32_t*>(at[2]);
  if (at[3]) L.sel_c = static_cast<int32_t*>(at[3]);
  Py_RETURN_NONE;
}

#define MDC_METHOD(name, n) {#name, reinterpret_cast<PyCFunction>(reinterpret_cast<void*>(entry<n, name>)), METH_FASTCALL, nullptr}
PyMethodDef methods[] = {MDC_METHOD(bind, 1),          MDC_METHOD(logits, 22),        MDC_METHOD(merge_topk, 9),
                         MDC_METHOD(lse_merge, 6),     MDC_METHOD(sparse_mla, 18),    MDC_METHOD(compress_step, 12),
                         MDC_METHOD(compress_finalize, 15), MDC_METHOD(megakernel, 6),
                         MDC_METHOD(causal_lens, 5), MDC_METHOD(prefill_targets, 5), MDC_METHOD(prefill_fill, 10), {nullptr, nullptr, 0, nullptr}};
PyModuleDef module = {PyModuleDef_HEAD_INIT, "_mdc_host", "Host side of the tile runners", -1, methods, nullptr, nullptr, nullptr, nullptr};

}  // namespace

PyMODINIT_FUNC PyInit__mdc_host(void) { return PyModule_Create(&module); }

// Launch wrapper of the candidate-merge tile (see tile_merge.cuh).
#include "hist_select.cuh"
#include "tile_merge.cuh"

namespace mdc {
// Rows of up to this many positions (a multiple of 4) are staged whole and selected by their histogram: 8 queries x 4 lists
// of 1024 candidates took 20 us by the search (cold caches).  Longer rows, and ties across the threshold, which
// go by id, take the search.
constexpr int kMergeHistPos = 16384;
constexpr int kMergeHistSmem = MDC_THR_BINS * 4 + (static_cast<int>(sizeof(HistSelectSmem)) + 15) / 16 * 16;   // behind the row
__device__ inline bool merge_row_by_hist(const mdc_merge_topk_params& p, int row, MergeSmem& sm, unsigned char* stage) {
  const int tid = threadIdx.x, n_pos = p.L * p.maxK;
  MergeLists ls;
  const int64_t base = static_cast<int64_t>(row) * n_pos;
  ls.v = p.cand_v + base;
  ls.i = p.cand_i + base;
  ls.c = p.cand_c + static_cast<int64_t>(row) * p.L;
  ls.stride = p.maxK;
  ls.c_stride = 1;
  uint32_t* vb = reinterpret_cast<uint32_t*>(stage);
  int32_t* ib = reinterpret_cast<int32_t*>(vb) + n_pos;
  uint32_t* hist = reinterpret_cast<uint32_t*>(ib) + n_pos;
  HistSelectSmem& hs = *reinterpret_cast<HistSelectSmem*>(hist + MDC_THR_BINS);
  for (int i = tid; i < MDC_THR_BINS / 4; i += kBlockThreads) reinterpret_cast<uint4*>(hist)[i] = make_uint4(0u, 0u, 0u, 0u);
  merge_load_counts<kInputLists>(ls, p.L, p.maxK, sm);
  merge_stage_lists<kInputLists>(ls, p.L, p.maxK, sm, vb, ib);
  for (int i = tid; i < n_pos / 4; i += kBlockThreads) {
    const uint4 q = reinterpret_cast<const uint4*>(vb)[i];
    const uint32_t v[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
    for (int j = 0; j < 4; ++j)
      if (v[j]) atomicAdd(&hist[v[j] >> kKeyShift], 1u);
  }
  sync_workers();
  float* ov = p.out_v + static_cast<int64_t>(row) * p.top_k;
  int32_t* oi = p.out_i + static_cast<int64_t>(row) * p.top_k;
  const int n = hist_select_emit<1>(vb, n_pos, p.top_k, hist, hs, tid, [&](int pos, int slot) {
    ov[slot] = unsortable_f32(vb[pos]);
    oi[slot] = ib[pos];
  });
  if (n < 0) return false;
  if (tid == 0) {
    p.out_c[row] = n;
    int valid = 0;
    for (int l = 0; l < p.L; ++l) valid += sm.cnt[l];
    if (p.dbg && n != min(valid, p.top_k)) atomicAdd(p.dbg, 1);
  }
  return true;
}

constexpr int kMergeStageMax = 200 * 1024;  // rows of up to 25600 positions are staged in shared memory
constexpr int kMergeHistBytes = 2048 * 4;    // behind a staged row: the histogram of the threshold search
static_assert(kMergeHistSmem >= kMergeHistBytes && kMergeHistPos * 8 + kMergeHistSmem <= 220 * 1024, "the search's scratch fits too");
__global__ void __launch_bounds__(kBlockThreads) merge_topk_kernel(const __grid_constant__ mdc_merge_topk_params p) {
  __shared__ MergeSmem sm;
  extern __shared__ __align__(16) unsigned char stage[];
  wait_for_predecessor();
  const int n_pos = p.L * p.maxK;
  if (n_pos <= kMergeHistPos && (n_pos & 3) == 0) {
    if (merge_row_by_hist(p, blockIdx.x, sm, stage)) return;
    sync_workers();
  }
  const int need = n_pos * 8 <= kMergeStageMax ? n_pos * 8 + kMergeHistBytes : (n_pos * 4 <= kMergeStageMax ? n_pos * 4 : 0);
  merge_topk_tile(p, blockIdx.x, sm, need ? stage : nullptr, need);
}
}  // namespace mdc

extern "C" int mdc_merge_topk_launch(const mdc_merge_topk_params* p, void* stream) {
  using namespace mdc;
  if (!p || !p->cand_v || !p->cand_i || !p->cand_c || !p->out_v || !p->out_i || !p->out_c) return MDC_ERR_NULL;
  if (p->B < 1 || p->q_len < 1 || p->L < 1 || p->L > kMergeMaxLists || p->maxK < 1 || p->top_k < 1)
    return MDC_ERR_BAD_SHAPE;
  if (static_cast<int64_t>(p->L) * p->maxK > (1ll << 30)) return MDC_ERR_TOO_LARGE;
  const int64_t n_pos = static_cast<int64_t>(p->L) * p->maxK;
  int smem = n_pos * 8 <= kMergeStageMax ? static_cast<int>(n_pos * 8) + kMergeHistBytes
                                               : (n_pos * 4 <= kMergeStageMax ? static_cast<int>(n_pos * 4) : 0);
  if (n_pos <= kMergeHistPos && (n_pos & 3) == 0) smem = static_cast<int>(n_pos * 8) + kMergeHistSmem;   // (more than the search wants)
  if (const int rc = allow_dynamic_smem<merge_topk_kernel>(smem); rc != MDC_OK) return rc;
  return launch_behind(merge_topk_kernel, dim3(p->B * p->q_len), kBlockThreads, smem, static_cast<cudaStream_t>(stream), *p);
}

int mdc_attrs_merge_topk(cudaFuncAttributes* a) {
  return static_cast<int>(cudaFuncGetAttributes(a, mdc::merge_topk_kernel));
}

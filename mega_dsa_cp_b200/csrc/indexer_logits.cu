// Launch wrapper of the indexer-logits tile (see tile_logits.cuh).
#include "tile_logits.cuh"

#include <cudaTypedefs.h>

namespace mdc {

// The page pool as a tensor of 64-byte rows: (64 bytes, rows of a page, pages).  One box is a page; the copy swizzles its
// rows (see tile_logits.cuh).
int logits_page_map(const mdc_logits_params& p, CUtensorMap* map) {
  static std::atomic<PFN_cuTensorMapEncodeTiled_v12000> encode;
  auto fn = encode.load(std::memory_order_acquire);
  if (!fn) {
    void* f = nullptr;
    cudaDriverEntryPointQueryResult found;
    MDC_CUDA_OK(cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &f, cudaEnableDefault, &found));
    if (!f) return MDC_ERR_CUDA;
    fn = reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(f);
    encode.store(fn, std::memory_order_release);
  }
  const cuuint64_t page_bytes = static_cast<cuuint64_t>(p.page_tokens) * (p.fmt == MDC_FMT_MXFP4 ? 68 : 72);
  const cuuint64_t dims[3] = {64, page_bytes / 64, static_cast<cuuint64_t>(p.num_pages)};
  const cuuint64_t strides[2] = {64, page_bytes};
  const cuuint32_t box[3] = {64, static_cast<cuuint32_t>(page_bytes / 64), 1}, ones[3] = {1, 1, 1};
  const CUresult r = fn(map, CU_TENSOR_MAP_DATA_TYPE_UINT8, 3, const_cast<uint8_t*>(p.kv_pages), dims, strides, box, ones,
                        CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_64B, CU_TENSOR_MAP_L2_PROMOTION_NONE,
                        CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS ? MDC_OK : MDC_ERR_BAD_SHAPE;
}

template <int FMT, int PAGE, int T>
__global__ void __launch_bounds__(kLogitsThreads, 1) logits_kernel(const __grid_constant__ mdc_logits_params p,
                                                                      const __grid_constant__ CUtensorMap pages) {
  extern __shared__ unsigned char smem_raw[];
  wait_for_predecessor();
  let_successor_start();
  // the UMMA operand block wants a 1024-byte aligned base
  unsigned char* smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
  logits_tile<FMT, PAGE, T, true>(p, &pages, blockIdx.y, blockIdx.x, smem);
}

// Row mode: the blocks of one request form a cluster and select across their chunks.
template <int FMT, int PAGE, int T>
__global__ void __launch_bounds__(kLogitsThreads, 1) logits_row_kernel(const __grid_constant__ mdc_logits_params p,
                                                                          const __grid_constant__ CUtensorMap pages) {
  extern __shared__ unsigned char smem_raw[];
  wait_for_predecessor();
  unsigned char* smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
  logits_tile<FMT, PAGE, T, true, true>(p, &pages, blockIdx.y, blockIdx.x, smem);
}

template <int FMT, int PAGE, int T>
static int launch_logits_row(const mdc_logits_params& p, const CUtensorMap& pages, cudaStream_t st, int smem) {
  constexpr auto kern = logits_row_kernel<FMT, PAGE, T>;
  if (const int rc = allow_dynamic_smem<kern>(smem); rc != MDC_OK) return rc;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(p.n_chunks, p.B);
  cfg.blockDim = dim3(kLogitsThreads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = p.n_chunks;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 2;
  MDC_CUDA_OK(cudaLaunchKernelEx(&cfg, kern, p, pages));
  return MDC_OK;
}

template <int FMT, int PAGE, int T>
static int launch_logits(const mdc_logits_params& p, cudaStream_t st, int smem) {
  CUtensorMap pages;
  if (const int rc = logits_page_map(p, &pages); rc != MDC_OK) return rc;
  if (p.row_v) return launch_logits_row<FMT, PAGE, T>(p, pages, st, smem);
  constexpr auto kern = logits_kernel<FMT, PAGE, T>;
  if (const int rc = allow_dynamic_smem<kern>(smem); rc != MDC_OK) return rc;
  dim3 grid(p.n_chunks, p.B);
  return launch_behind(kern, grid, kLogitsThreads, smem, st, p, pages);
}

int logits_check(const mdc_logits_params* p) {
  if (!p) return MDC_ERR_NULL;
  if (!p->kv_pages || !p->q || !p->weights || !p->block_table) return MDC_ERR_NULL;
  if (p->fmt != MDC_FMT_MXFP4 && p->fmt != MDC_FMT_NVFP4) return MDC_ERR_BAD_FORMAT;
  if (p->q_fmt != MDC_Q_FP4 && p->q_fmt != MDC_Q_BF16) return MDC_ERR_BAD_FORMAT;
  if (p->q_fmt == MDC_Q_FP4 && !p->q_sf) return MDC_ERR_NULL;
  if (p->page_tokens != 64 && p->page_tokens != 128) return MDC_ERR_BAD_SHAPE;
  if (p->fmt == MDC_FMT_MXFP4 && p->page_tokens != 128) return MDC_ERR_BAD_SHAPE;
  if (p->heads != kIdxHeads || (p->q_len != 1 && p->q_len != 2)) return MDC_ERR_BAD_SHAPE;
  if (p->num_pages < 1 || p->B < 1 || p->n_chunks < 1 || p->blocks_per_chunk < 1 || p->max_pages < 1) return MDC_ERR_BAD_SHAPE;
  if (p->blocks_per_chunk > (1 << 20)) return MDC_ERR_TOO_LARGE;   // (far past what fits on chip; the sizes below are 32-bit)
  if (p->n_chunks > 65535 * 32 || p->B > 65535) return MDC_ERR_BAD_SHAPE;
  const bool fused = p->cand_v != nullptr && !p->row_v;
  if (p->row_v) {
    if (!p->row_i || !p->row_c) return MDC_ERR_NULL;
    if (p->top_k < 1 || p->id_mul < 1) return MDC_ERR_BAD_SHAPE;
    if (p->n_chunks != 1 && p->n_chunks != 2 && p->n_chunks != 4 && p->n_chunks != 8) return MDC_ERR_BAD_SHAPE;
    if (p->blocks_per_chunk * p->page_tokens > kBlockThreads * kFusedRegE) return MDC_ERR_TOO_LARGE;
  } else if (fused) {
    if (!p->cand_i || !p->cand_c) return MDC_ERR_NULL;
    if (p->top_k < 1) return MDC_ERR_BAD_SHAPE;
    if (p->id_mul < 1) return MDC_ERR_BAD_SHAPE;
  } else if (!p->logits) {
    return MDC_ERR_NULL;
  }
  if (reinterpret_cast<uintptr_t>(p->kv_pages) & 15) return MDC_ERR_BAD_ALIGN;
  if (reinterpret_cast<uintptr_t>(p->q) & (p->q_fmt == MDC_Q_BF16 ? 15 : 7)) return MDC_ERR_BAD_ALIGN;   // (bf16 rows are read in 16-byte pieces)
  return MDC_OK;
}

static int logits_smem(const mdc_logits_params* p) {
  const bool fused = p->cand_v != nullptr || p->row_v != nullptr;
  const int ct = p->blocks_per_chunk * p->page_tokens;
  int total;
  auto size = [&](auto layout, bool keys) { return layout(p->q_len, ct, fused, fused && keys).total; };
  if (p->fmt == MDC_FMT_MXFP4) total = size(logits_smem_layout<MDC_FMT_MXFP4, 128>, logits_as_keys<MDC_FMT_MXFP4, 128>(p->q_len, ct));
  else if (p->page_tokens == 64) total = size(logits_smem_layout<MDC_FMT_NVFP4, 64>, logits_as_keys<MDC_FMT_NVFP4, 64>(p->q_len, ct));
  else total = size(logits_smem_layout<MDC_FMT_NVFP4, 128>, logits_as_keys<MDC_FMT_NVFP4, 128>(p->q_len, ct));
  // slack for the 1024-byte alignment of the base; at least 116 KB so that one
  // block owns an SM (each block allocates all of the SM's tensor memory)
  total += 1024;
  return total < 116 * 1024 ? 116 * 1024 : total;
}

}  // namespace mdc

extern "C" int mdc_logits_fp4_smem_bytes(const mdc_logits_params* p) {
  int rc = mdc::logits_check(p);
  if (rc != MDC_OK) return rc;
  return mdc::logits_smem(p);
}

extern "C" int mdc_logits_fp4_launch(const mdc_logits_params* p, void* stream) {
  using namespace mdc;
  int rc = logits_check(p);
  if (rc != MDC_OK) return rc;
  const int smem = logits_smem(p);
  if (smem > 227 * 1024) return MDC_ERR_TOO_LARGE;  // chunk too long to keep its scores on chip
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const int key = (p->fmt == MDC_FMT_MXFP4 ? 0 : (p->page_tokens == 64 ? 1 : 2)) * 2 + (p->q_len - 1);
  switch (key) {
    case 0: return launch_logits<MDC_FMT_MXFP4, 128, 1>(*p, st, smem);
    case 1: return launch_logits<MDC_FMT_MXFP4, 128, 2>(*p, st, smem);
    case 2: return launch_logits<MDC_FMT_NVFP4, 64, 1>(*p, st, smem);
    case 3: return launch_logits<MDC_FMT_NVFP4, 64, 2>(*p, st, smem);
    case 4: return launch_logits<MDC_FMT_NVFP4, 128, 1>(*p, st, smem);
    default: return launch_logits<MDC_FMT_NVFP4, 128, 2>(*p, st, smem);
  }
}

int mdc_attrs_logits(cudaFuncAttributes* a) {
  return static_cast<int>(cudaFuncGetAttributes(a, mdc::logits_kernel<MDC_FMT_NVFP4, 64, 1>));
}

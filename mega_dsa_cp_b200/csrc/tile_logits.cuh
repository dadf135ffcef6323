// Indexer-logits tile: one thread block scores one chunk of one request's
// paged FP4 index-K cache against its 64 (x q_len) query heads and either
// writes the fp32 logits row or keeps the chunk's scores in shared memory and
// emits the exact local top-k.
//
// Groups of four warps (four stand-alone, three in the persistent kernel) take the 128-token stages in turn, each with
// tensor memory, a slot pair of the raw ring and barriers of its own:
//
//   copy     a page is contiguous in HBM (P x 64 B of packed E2M1, then the page's block scales); one tiled TMA load
//            per page fills a raw stage in shared memory and swizzles its 64-byte rows on the way (16-byte chunk j of
//            row r at j ^ (r / 2 % 4)), which is what makes the row loads below bank-conflict free.  The group that
//            has read a stage loads the stage two of its turns further on into it.
//   decode   thread i of a group owns token row i: it reads 64 B of codes (four 16-byte loads) and the row's scales,
//            converts with cvt.f16x2.e2m1x2, multiplies by the block scale (exact in fp16) and stores the row into
//            TENSOR MEMORY (tcgen05.st) as the A operand.
//   product  behind a barrier of the group's 128 threads one of them issues eight tcgen05.mma (M=128 tokens, N=64
//            heads, K=16, fp16 x fp16 -> fp32) per query token, B = the query block, staged once in shared memory in
//            the K-major 128-byte-swizzle layout.
//   gate     while it runs, the group takes the accumulator row that it has read (tcgen05.ld) before issuing it: relu,
//            head weights, sum over heads, the scores of the stage (or query token) before.
//
// Keeping A in tensor memory instead of shared memory matters: the decode
// output (32 KB per stage) and its re-read by the tensor core would otherwise
// triple the shared-memory traffic of a kernel that has to sustain one stage
// per ~400 cycles to follow HBM.
//
// What bounds the loop is latency between dependent steps, with every pipe half used (ALU, shared
// memory, issue slots and tensor core each need 250-400 cycles per stage).  So the groups share nothing: no counters or
// barriers between producer and consumer warps, no warp that only polls; a group's step waits for its raw stage and for
// its own product, both of which have had most of a step to complete.  The form before had two decode groups, two gate
// groups, two issue warps and a copy warp (one gate group and one issue warp in the persistent kernel), handing stages on
// in pairs.  32 x 32768 tokens with row top-k 38.9 -> 36.0 us, 37 sequences x 16384 tokens, logits out, 18.0 -> 15.4,
// two query tokens, 16 x 32768 MXFP4, 32.2 -> 28.8, 3 x 20032 6.4 -> 5.1, the persistent kernel's step of 8 x 131072
// 85.5 -> 76.3: with the query's loads in flight together and the page table read ahead of the length, which shortened the
// prologue from 6400 to 2570 cycles by clock stamps (1.95 us of the first figure's 2.9, 1.0 of the fourth's), and in the
// persistent kernel with what else changed there.
// Three groups with issue and copy warps between them: 43.5 for the
// first of these; the warps of a group taking turns to issue: 37.7.
//
// The persistent kernel's blocks have 14 warps: three groups there.  Four, in blocks of 16 warps, need the decode loop rolled,
// or the step's code does not stay in the instruction cache (step of 8 x 131072 84.7 us unrolled, 78.2 rolled; three
// groups 79.7 rolled, 76.3 unrolled).
//
// Exactness.  K values (E2M1 x scale) are exact in fp16.  Query rows are
// rescaled per head by a power of two so that the largest element lands in
// [2^14, 2^15) before the fp16 conversion, and the head weight absorbs the
// inverse factor; relu commutes with a positive scale, so the logit is the
// same real number, accumulated in fp32.
//
// Every wait is bounded; a wait that runs out records MDC_DEV_COPY_TIMEOUT,
// raises a block-wide flag all roles poll, and the block leaves through the
// common exit (tensor memory is freed there).
#pragma once

#include <cooperative_groups.h>

#include "common.cuh"
#include "events.cuh"
#include "fp4.cuh"
#include "hist_select.cuh"
#include "radix.cuh"
#include "radix_regs.cuh"
#include "umma.cuh"

namespace mdc {

constexpr int kIdxDim = 128;
constexpr int kIdxHeads = 64;
constexpr int kTileTok = 128;    // tokens per pipeline stage (= UMMA M)
constexpr int kLogitsGroups = 4; // groups of four warps; 512 threads leave each 128 registers
constexpr int kRawStages = 8;    // raw page ring: two slots per group
constexpr int kTmemCols = 512;   // per group 64 columns of accumulator (128 rows x 64 heads) and 64 of decoded A
constexpr int kFusedRegE = 32;   // fused top-k keeps up to 256 * 32 scores per query token in registers
constexpr int kLogitsThreads = kLogitsGroups * 128;
// The persistent kernel: three groups (see above) and six of the stages.
constexpr int kMegaGroups = 3, kMegaThreads = 448;
static_assert(kMegaGroups * 128 <= kMegaThreads && kMegaGroups <= kLogitsGroups, "the groups' warps");
static_assert(kRawStages % kLogitsGroups == 0 && kLogitsGroups * 128 <= kTmemCols, "slots and columns of the groups");

template <int FMT, int PAGE>
struct IdxPage {
  static constexpr int kData = PAGE * 64;
  static constexpr int kSf = PAGE * (FMT == MDC_FMT_MXFP4 ? 4 : 8);
  static constexpr int kBytes = kData + kSf;
  static constexpr int kTilePages = kTileTok / PAGE;
  static constexpr int kStageBytes = kTilePages * kBytes;
  static constexpr int kRows = kBytes / 64;   // a page as 64-byte rows: the tensor map's box
  static_assert(kBytes % 512 == 0 && kRows <= 256, "the 64-byte swizzle repeats every 512 bytes");
  // byte offset o of a page lies here after the copy's swizzle (a page starts on a 512-byte boundary)
  __device__ static int swizzled(int o) { return o ^ ((o >> 3) & 0x30); }
};

// Scratch of the cluster-wide row select (read by the other blocks of the cluster).
struct RowSelectScratch {
  uint32_t hist[2][256];   // digit histograms of this block, double buffered over the radix passes
  int32_t cnt_gt, cnt_eq;  // this block's counts above / at the row threshold
  int32_t digit, excl;     // result of a pass: boundary digit, number of keys in higher bins
  int32_t bin_cnt, pad0;   // keys in the boundary bin
  int32_t wsum[kWarps];
};

struct LogitsSmem {
  // byte offsets inside the tile's dynamic shared memory (base 1024 B aligned)
  int qb, ring, bars, misc, page_ok, wsc, sel, row, scores, hist, total;
};

template <int FMT, int PAGE>
__host__ __device__ constexpr LogitsSmem logits_smem_layout(int q_len, int chunk_tokens, bool fused, bool hist = false) {
  LogitsSmem L{};
  int off = 0;
  L.qb = off;  // [2 K-halves][N rows][128 B], swizzled; needs 1024 B alignment
  off += 2 * q_len * kIdxHeads * 128;
  L.ring = off;
  off += kRawStages * IdxPage<FMT, PAGE>::kStageBytes;
  off = static_cast<int>(align_up(off, 128));
  L.bars = off;
  off += (kRawStages + kLogitsGroups) * 8;
  L.misc = off;  // [0] tensor-memory base, [1] abort flag, [12..13] selected
  off += 64;
  L.wsc = off;
  off += q_len * kIdxHeads * 4;
  off = static_cast<int>(align_up(off, 16));
  L.sel = off;
  off += static_cast<int>(align_up(sizeof(SelectScratch) > sizeof(RegSelectScratch<kFusedRegE>) ? sizeof(SelectScratch)
                                                                                             : sizeof(RegSelectScratch<kFusedRegE>), 16));
  L.row = off;
  off += static_cast<int>(align_up(sizeof(RowSelectScratch), 16));
  L.page_ok = off;  // page id per page of the chunk (-1 = not usable)
  off += static_cast<int>(align_up((chunk_tokens / PAGE + 4) * 4, 16));
  L.scores = off;
  if (fused) off += q_len * chunk_tokens * 4;
  off = static_cast<int>(align_up(off, 16));
  L.hist = off;  // histograms of the chunk's keys, one per query token, filled with the scores
  if (hist) off += q_len * MDC_THR_BINS * 4;
  L.total = static_cast<int>(align_up(off, 128));
  return L;
}

// Whether a chunk's scores are kept as sortable keys with their histogram (hist_select.cuh): when that fits an SM's shared
// memory and the bitmap of positions.  (Otherwise, two query tokens on more than 8192 tokens, the scores alone.)
template <int FMT, int PAGE>
__host__ __device__ inline bool logits_as_keys(int q_len, int chunk_tokens) {
  return chunk_tokens <= kHistSelectMax && logits_smem_layout<FMT, PAGE>(q_len, chunk_tokens, true, true).total + 1024 <= 227 * 1024 &&
         2 * static_cast<int>(sizeof(HistSelectSmem)) <= kRawStages * IdxPage<FMT, PAGE>::kStageBytes;
}

// Prologue: the request's query rows as prescaled fp16 in the UMMA B layout,
// and the matching head weights (halved: the gate computes (x + |x|) * w/2).
// Row r of the request = head r % 64 of query token r / 64.  Called by warps
// 0..7; a half-warp stages one row, lane l of it the dims 8l..8l+7.
template <int T>
__device__ inline void logits_stage_query(const mdc_logits_params& p, int b, unsigned char* qb, float* wsc) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int hl = lane & 15, sub = lane >> 4;
  constexpr int N = T * kIdxHeads, kBatch = 4;   // rows of a half-warp whose loads are in flight together
  static_assert(N % (kWarps * 2 * kBatch) == 0, "whole batches");
#pragma unroll 1
  for (int row0 = warp * 2 + sub; row0 < N; row0 += kWarps * 2 * kBatch) {
    uint4 raw[kBatch];
    float w[kBatch];
#pragma unroll
    for (int k = 0; k < kBatch; ++k) {
      const int row = row0 + k * kWarps * 2;
      const int64_t at = static_cast<int64_t>(b) * N + row;
      if (p.q_fmt == MDC_Q_BF16) {
        raw[k] = *reinterpret_cast<const uint4*>(static_cast<const __nv_bfloat16*>(p.q) + at * kIdxDim + 8 * hl);
      } else {
        raw[k].x = *reinterpret_cast<const uint32_t*>(static_cast<const uint8_t*>(p.q) + at * 64 + 4 * hl);
        // atom-ordered scales: 512 B per block of 128 rows
        const uint8_t* sfb = p.q_sf + static_cast<int64_t>(b) * ceil_div(N, 128) * 512 + (row / 128) * 512;
        const int r = row % 128;
        raw[k].y = sfb[(r % 32) * 16 + (r / 32) * 4 + hl / 4];
      }
      w[k] = p.weights[at];
    }
#pragma unroll
    for (int k = 0; k < kBatch; ++k) {
      const int row = row0 + k * kWarps * 2;
      float v[8];
      if (p.q_fmt == MDC_Q_BF16) {
        const uint32_t w4[4] = {raw[k].x, raw[k].y, raw[k].z, raw[k].w};
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          v[2 * i] = __uint_as_float(w4[i] << 16);
          v[2 * i + 1] = __uint_as_float(w4[i] & 0xffff0000u);
        }
      } else {
        const float sc = __uint_as_float(raw[k].y << 23);
#pragma unroll
        for (int i = 0; i < 8; ++i) v[i] = e2m1_to_float((raw[k].x >> (4 * i)) & 0xf) * sc;
      }
      float m = 0.f;
#pragma unroll
      for (int i = 0; i < 8; ++i) m = fmaxf(m, fabsf(v[i]));
#pragma unroll
      for (int o = 8; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
      // power-of-two rescale: bring the largest magnitude to [2^14, 2^15)
      int ex = static_cast<int>((__float_as_uint(m) >> 23) & 0xff) - 127;
      int up = 14 - ex;
      up = max(-100, min(100, up));
      if (m == 0.f || !(m < 3.0e38f)) up = 0;
      const float scale = __uint_as_float(static_cast<uint32_t>(127 + up) << 23);
      const float inv = __uint_as_float(static_cast<uint32_t>(127 - up) << 23);
      uint4 out;
      {
        __half2 h0 = __floats2half2_rn(v[0] * scale, v[1] * scale);
        __half2 h1 = __floats2half2_rn(v[2] * scale, v[3] * scale);
        __half2 h2 = __floats2half2_rn(v[4] * scale, v[5] * scale);
        __half2 h3 = __floats2half2_rn(v[6] * scale, v[7] * scale);
        out.x = *reinterpret_cast<uint32_t*>(&h0);
        out.y = *reinterpret_cast<uint32_t*>(&h1);
        out.z = *reinterpret_cast<uint32_t*>(&h2);
        out.w = *reinterpret_cast<uint32_t*>(&h3);
      }
      // dims 8*hl .. 8*hl+7: K-half = hl / 8, 16-byte chunk = hl % 8
      unsigned char* dst = qb + (hl >> 3) * (N * 128) + row * 128 + (((hl & 7) ^ (row & 7)) << 4);
      *reinterpret_cast<uint4*>(dst) = out;
      // 0.5 for the (x + |x|) form of relu
      if (hl == 0) wsc[row] = 0.5f * w[k] * inv;
    }
  }
}

// Exact top-k of one chunk's scores (shared memory).  The scores become sortable keys in place
// (0 = not a candidate); search and position-ordered emit are rolled loops over them: code that a
// block executes once per task is bound by instruction fetch, so it is kept small.  Ties at the
// threshold go to the smaller position.  Returns the number of entries emitted.
template <typename Emit>
__device__ inline int fused_chunk_select(const float* sc_row, uint32_t* keys, int n_local, int base_pos, int limit, int top_k,
                                         SelectScratch& sel, Emit emit) {
  sync_workers();
  for (int pos = threadIdx.x; pos < n_local; pos += kBlockThreads)
    keys[pos] = (base_pos + pos) < limit ? max(sortable_u32(sc_row[pos]), 1u) : 0u;
  sync_workers();
  const Threshold<uint32_t> th = block_select_bits_smem(keys, n_local, top_k, sel);
  return block_emit_keys(keys, n_local, th, sel, emit);
}

// Row-threshold candidate filter (used by the persistent kernel, one query token).  The chunks of a
// request run as separate tasks on different blocks; instead of each emitting the exact top-k of its
// own chunk (a quarter of the chunk at k = 2048 of 8192: long lists, a tree of merges behind them),
// the tasks agree on a lower bound of the ROW's k-th largest score and emit only what reaches it:
//
//   1. every task adds the histogram of its scores (kThrBins bins = the top 12 bits of the sortable
//      key: sign, exponent, three mantissa bits) to the row's histogram in global memory and counts in;
//   2. it waits (bounded) until all n_chunks tasks of the row have counted in, reads the summed
//      histogram and takes the lowest bin B such that the bins >= B hold at least k scores: the
//      row's k-th largest score lies in bin B, so nothing below B can be selected;
//   3. it emits its scores in bins >= B, in position order: over the row about k plus one bin's worth.
//
// The one merge behind the tasks selects exactly.  Waiting on row mates inside a task cannot deadlock:
// tasks are dealt to the blocks in row-major order and every block runs its queue in order, so the
// lowest unfinished row always has all of its tasks running or next in line.  A wait that runs out
// is reported, and the task falls back to the exact top-k of its own chunk, which is always a valid
// candidate set; so does a chunk whose filtered set would not fit its list (heavily tied scores).
constexpr int kThrBins = MDC_THR_BINS, kThrShift = 32 - 12;   // sign, exponent, three mantissa bits
static_assert(kThrBins == 1 << (32 - kThrShift), "bins = the key's upper bits");

// Exact mode (RowThreshold::x set).  The chunk tasks of a row, on ALL ranks of a context-parallel group,
// settle the row's exact top-k between them, so that no merge has to run behind them:
//   a. the last task of a rank's row to count in stores the rank's row histogram into every rank's arena
//      and notifies the row's "histograms" cell there; every task waits for the cp histograms, sums them
//      and finds the boundary bin of the GLOBAL row (one rank: the local histogram is the global one);
//   b. every task stores a slot {scores above the bin, scores inside it, overflow flag, the keys inside
//      it} into every rank's arena and notifies the row's "keys" cell; it waits for all cp x n_chunks slots;
//   c. every task finds the exact threshold among the undecided keys of all slots (the same computation
//      on the same data everywhere), derives each slot's share (ties go to the lower rank, chunk,
//      position) and emits its own share: the gather list of this rank at its local offset, and the
//      selection list at its global offset on every rank.  Its candidate count is then -1 ("published").
// A slot that would overflow (heavily tied scores) makes every task of the row fall back to emitting
// candidates for the merge task, which always remains in the task graph.  All waits are bounded.
constexpr int kUndCap = 512;                      // boundary-bin keys one chunk contributes at most
constexpr int kUndRowCap = 4096;                  // ... and a whole row (the exact search's shared-memory list)
constexpr int kRowSlotBytes = 16 + kUndCap * 4;   // {n_above, n_und, overflow, 0} then the keys
constexpr int kRowHistBytes = MDC_THR_BINS * 4;
constexpr int kRowMaxSlots = 256;

// One rank: the row's tasks share one list of undecided keys instead of a slot each.  Entry = the key's bits below the
// boundary bin << 8 | chunk, in no particular order; `count` = entries reserved (>= kUndOverflow: a chunk gave up).
struct RowOneRank {
  uint32_t* count;        // this step's counter, zero when the step starts
  uint32_t* count_next;   // the next step's: zeroed by this step
  uint32_t* list;         // kUndRowCap entries
  uint32_t* n_above;      // per chunk: its keys in bins above the boundary bin
};
constexpr uint32_t kUndOverflow = 1u << 20;

struct RowExact {
  EventSet ev;
  int ev_hist, ev_keys;                        // the row's two cells
  unsigned long long hist_target, keys_target;  // cp and cp * n_chunks arrivals per step
  unsigned char* arena;                        // this rank's arena; rank d's is at arena + arena_offsets[d]
  const int64_t* arena_offsets;
  int64_t hist_off;                            // this step, this row: [cp][bins] u32 (unused with one rank)
  int64_t slot_off;                            // this step, this row: [cp * n_chunks] slots
  int64_t out_off;                             // several ranks: the row's candidate slices (slice 0 receives the
  int64_t slice_bytes;                         //   selection behind its 16-byte cell: [K f32][K i32]; every slice's cell: {-1, total})
  int cp, rank;                                // the ranks of the context-parallel group, and this one
  int pcp, prank;                              // the ranks that settle the row together: (cp, rank), or (1, 0): this rank's
                                               //   tasks settle the rank's own top-k and store it as the rank's candidate
                                               //   list (slice `rank` of the row, a plain count in its cell) on every rank
  float* out_v;                                // one rank: the row of the selection lists, written directly
  int32_t* out_i;
  int32_t* sel_c;
  int32_t* pt;                                 // the row of this rank's gather list (pool rows)
  int pt_cols;
  int32_t* k_valid;
  int row_base, win_slots;
  RowOneRank one;                              // (cp == 1)
};

struct RowThreshold {
  uint32_t* hist;       // (B, kThrBins) of this phase, zero when the step starts
  uint32_t* hist_next;  // the other phase's histogram: this step zeroes it for the next one
  uint32_t* done;       // (B,) tasks counted in, monotonic over the steps
  uint32_t target;      // value of done[b] when all n_chunks tasks of this step have counted in
  long long budget_ns;
  const RowExact* x;    // exact mode, or nullptr
};


// exclusive prefix sums of n <= 256 ints in shared memory, by one warp (eight consecutive per lane);
// out[n] receives the total
__device__ inline void warp_prefix256(const int* in, int* out, int n, int lane) {
  int c[8], sum = 0;
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    c[j] = lane * 8 + j < n ? in[lane * 8 + j] : 0;
    sum += c[j];
  }
  int total;
  int run = warp_excl_scan(sum, lane, &total);
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    if (lane * 8 + j <= n) out[lane * 8 + j] = run;
    run += c[j];
  }
}

struct RowExactSmem {
  int32_t na[kRowMaxSlots], nu[kRowMaxSlots];     // slot headers
  int32_t g[kRowMaxSlots], e[kRowMaxSlots];       // per slot: selected above the threshold, tied at it
  int32_t take[kRowMaxSlots];
  int32_t uo[kRowMaxSlots + 1], eo[kRowMaxSlots + 1], to[kRowMaxSlots + 1];  // prefixes of nu, e, take
  int32_t overflow, my_n, ok, pad;
};

constexpr int kSurvCap = 2048;   // scores of one chunk at or above the row's boundary bin (more: the row falls back)

// Shared-memory scratch of the exact mode with several ranks, in the raw ring, which is idle by then (its size is checked
// where the tile is instantiated).
struct RowExactScratch {
  uint32_t skey[kSurvCap];    // the chunk's survivors (keys in bins >= the boundary bin), in position order
  uint16_t spos[kSurvCap];    // ... and their positions inside the chunk
  uint32_t mylist[kUndCap];   // those inside the boundary bin: this chunk's slot
  uint32_t und[kUndRowCap];   // the undecided keys of the whole row
  RowExactSmem xs;
};

// Steps b and c of the exact mode with several ranks, after the boundary bin `bin` of the global row is known (0: the row
// holds fewer than top_k scores, everything valid is selected).  n_pass: this chunk's scores in bins >= bin.
// hist2: 2048 words of shared memory for the threshold search (the chunk histogram's space, which is no longer
// needed).  Returns true when the row was published (this task emitted its share), false when the row falls back.
static __device__ __noinline__ bool chunk_publish_row_exact(const RowThreshold& rt, int32_t* status, int b, int chunk, int n_chunks,
                                               const uint32_t* keys, int n_local, int base_pos, int top_k, int id_mul,
                                               int id_add, uint32_t bin, int n_pass, SelectScratch& sel,
                                               RowExactScratch& rs, uint32_t* hist2) {
  const RowExact& x = *rt.x;
  RowExactSmem& xs = rs.xs;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int J = x.pcp * n_chunks, me = x.prank * n_chunks + chunk;
  const bool local_only = x.pcp == 1;   // (slots, cells and counters on this rank only)
  const uint32_t floor_tau = bin ? (bin << kThrShift) - 1u : 0u;   // keys > floor_tau: the bins >= bin
  // ---- the chunk's survivors, compacted in position order: every later step works on this short list
  const bool fits = n_pass <= kSurvCap;
  int n_s = 0;
  if (fits) {
    Threshold<uint32_t> th;
    th.tau = floor_tau;
    th.need_eq = 0;
    th.n_sel = n_pass;
    n_s = block_emit_keys(keys, n_local, th, sel, [&](int pos, int slot) {
      if (slot < kSurvCap) {
        rs.skey[slot] = keys[pos];
        rs.spos[slot] = static_cast<uint16_t>(pos);
      }
    });
    n_s = min(n_s, kSurvCap);
  }
  const int n_s4 = (n_s + 3) & ~3;
  if (tid < n_s4 - n_s) rs.skey[n_s + tid] = 0u;
  if (tid == 0) xs.my_n = 0;
  sync_workers();
  // ---- b. this chunk's slot: how many above the bin, and the keys inside it
  int above = 0;
  for (int i0 = 0; i0 < n_s; i0 += kBlockThreads) {
    const int i = i0 + tid;
    const uint32_t v = i < n_s ? rs.skey[i] : 0u;
    const bool in = v != 0u && bin != 0u && (v >> kThrShift) == bin;
    above += v != 0u && !in;
    const uint32_t m = __ballot_sync(0xffffffffu, in);
    if (m != 0u) {
      int base = 0;
      if (lane == 0) base = atomicAdd(&xs.my_n, __popc(m));
      base = __shfl_sync(0xffffffffu, base, 0);
      const int slot = base + __popc(m & ((1u << lane) - 1u));
      if (in && slot < kUndCap) rs.mylist[slot] = v;
    }
  }
  above = __reduce_add_sync(0xffffffffu, above);
  if (lane == 0) sel.weq[warp] = above;
  sync_workers();
  int n_above = 0;
#pragma unroll
  for (int w = 0; w < kWarps; ++w) n_above += sel.weq[w];
  const int n_und = xs.my_n;
  const bool over = !fits || n_und > kUndCap;
  {
    const int n_keys = over ? 0 : n_und;
    const int64_t at = x.slot_off + static_cast<int64_t>(me) * kRowSlotBytes;
    for (int d = 0; d < x.pcp; ++d) {
      unsigned char* dst = x.arena + x.arena_offsets[local_only ? x.rank : d] + at;
      if (tid == 0) *reinterpret_cast<int4*>(dst) = make_int4(n_above, n_keys, over ? 1 : 0, 0);
      for (int i = tid; i < n_keys; i += kBlockThreads) reinterpret_cast<uint32_t*>(dst + 16)[i] = rs.mylist[i];
    }
    if (!local_only) __threadfence_system();
    else __threadfence();
    sync_workers();
    if (tid == 0) {
      for (int d = 0; d < x.pcp; ++d) x.ev.notify_1t(x.ev_keys, local_only ? x.rank : d);
      unsigned long long seen = 0;
      const bool ok = x.ev.poll_1t(x.ev_keys, x.keys_target, !local_only, rt.budget_ns, &seen, 64);
      if (!ok) report_failure(status, MDC_DEV_WAIT_TIMEOUT, -1000 - b, chunk, seen, x.keys_target);
      xs.ok = ok ? 1 : 0;
      xs.overflow = 0;
    }
    sync_workers();
    if (!xs.ok) return false;
  }
  // ---- c. all slots -> the exact threshold and every slot's share
  const unsigned char* slots = x.arena + x.slot_off;
  for (int j = tid; j < J; j += kBlockThreads) {
    const uint4 h = ld_sys_u4(reinterpret_cast<const uint4*>(slots + static_cast<int64_t>(j) * kRowSlotBytes));
    xs.na[j] = static_cast<int>(h.x);
    xs.nu[j] = min(max(static_cast<int>(h.y), 0), kUndCap);
    if (h.z != 0u) xs.overflow = 1;
  }
  sync_workers();
  if (warp == 0) warp_prefix256(xs.nu, xs.uo, J, lane);
  if (warp == 1) warp_prefix256(xs.na, xs.to, J, lane);   // (to: scratch here, its total is the count above the bin)
  sync_workers();
  const int U = xs.uo[J], A = xs.to[J];
  if (xs.overflow != 0 || U > kUndRowCap) return false;
  uint32_t* und = rs.und;
  for (int i0 = tid; i0 < U; i0 += 4 * kBlockThreads) {   // (independent loads: four in flight per thread)
    const float* src[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const int i = min(i0 + u * kBlockThreads, U - 1);
      int lo = 0, hi = J;   // the slot j with uo[j] <= i < uo[j + 1]
      while (hi - lo > 1) {
        const int mid = (lo + hi) >> 1;
        if (xs.uo[mid] <= i) lo = mid;
        else hi = mid;
      }
      src[u] = reinterpret_cast<const float*>(slots + static_cast<int64_t>(lo) * kRowSlotBytes + 16) + (i - xs.uo[lo]);
    }
    float v[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) v[u] = ld_sys_f32(src[u]);
#pragma unroll
    for (int u = 0; u < 4; ++u)
      if (i0 + u * kBlockThreads < U) und[i0 + u * kBlockThreads] = __float_as_uint(v[u]);
  }
  const int U4 = (U + 3) & ~3;
  if (tid < U4 - U) und[U + tid] = 0u;
  sync_workers();
  uint32_t tau = floor_tau;   // bin == 0, or the whole bin is taken: everything above the floor
  int need_eq = 0;
  if (bin != 0u) {
    const int need = top_k - A;   // 1 <= need <= U by the choice of the bin
    if (need > 0 && need < U) {
      const Threshold<uint32_t> th = block_select_hist_smem(und, U4, need, sel, hist2);
      if (th.need_eq != 0x7fffffff) {
        tau = th.tau;
        need_eq = th.need_eq;
      }
    }
  }
  // per slot: keys above the threshold and tied at it (one warp per slot in turn)
  for (int j = warp; j < J; j += kWarps) {
    int g = 0, e = 0;
    const int n = xs.nu[j], o = xs.uo[j];
    for (int i = lane; i < n; i += 32) {
      const uint32_t v = und[o + i];
      g += v > tau;
      e += v == tau;
    }
    g = __reduce_add_sync(0xffffffffu, g);
    e = __reduce_add_sync(0xffffffffu, e);
    if (lane == 0) {
      xs.g[j] = xs.na[j] + g;
      xs.e[j] = need_eq > 0 ? e : 0;
    }
  }
  sync_workers();
  if (warp == 0) warp_prefix256(xs.e, xs.eo, J, lane);
  sync_workers();
  for (int j = tid; j < J; j += kBlockThreads) xs.take[j] = xs.g[j] + min(xs.e[j], max(0, need_eq - xs.eo[j]));
  sync_workers();
  if (warp == 0) warp_prefix256(xs.take, xs.to, J, lane);
  sync_workers();
  const int my_eq = min(xs.e[me], max(0, need_eq - xs.eo[me]));
  const int off_g = xs.to[me], off_l = xs.to[me] - xs.to[x.prank * n_chunks];
  const int total = xs.to[J], local_total = xs.to[(x.prank + 1) * n_chunks] - xs.to[x.prank * n_chunks];
  const bool as_list = local_only;   // the result is this rank's candidate list, not the selection
  const int64_t out_at = x.out_off + (as_list ? static_cast<int64_t>(x.rank) * x.slice_bytes : 0);
  // ---- this chunk's share, from its survivor list (position order)
  Threshold<uint32_t> th;
  th.tau = tau;
  th.need_eq = my_eq;
  th.n_sel = xs.take[me];
  const int K = top_k;
  block_emit_keys(rs.skey, n_s4, th, sel, [&](int idx, int slot) {
    const uint32_t kv = rs.skey[idx];
    const int pos = rs.spos[idx];
    const float v = __uint_as_float((kv & 0x80000000u) ? (kv ^ 0x80000000u) : ~kv);
    const int id = (base_pos + pos) * id_mul + id_add;
    if (!as_list && off_l + slot < x.pt_cols) x.pt[off_l + slot] = x.row_base + base_pos + pos;
    const int o = off_g + slot;
    if (o < K) {
      for (int d = 0; d < x.cp; ++d) {
        unsigned char* dst = x.arena + x.arena_offsets[d] + out_at;   // slice: [cell 16 B][K f32][K i32]
        reinterpret_cast<float*>(dst + 16)[o] = v;
        reinterpret_cast<int32_t*>(dst + 16 + static_cast<int64_t>(K) * 4)[o] = id;
      }
    }
  });
  if (tid == 0) {
    if (chunk == 0 && !as_list) *x.k_valid = x.win_slots + min(local_total, x.pt_cols);
    if (as_list) {   // the rank's list on every rank: its length, by the row's first task
      if (chunk == 0)
        for (int d = 0; d < x.cp; ++d)
          *reinterpret_cast<int4*>(x.arena + x.arena_offsets[d] + out_at) = make_int4(min(total, K), 0, 0, 0);
    } else {  // this task's slice on every rank: "published", and the length of the selection
      for (int d = 0; d < x.cp; ++d)
        *reinterpret_cast<int4*>(x.arena + x.arena_offsets[d] + x.out_off + static_cast<int64_t>(me) * x.slice_bytes) =
            make_int4(-1, min(total, K), 0, 0);
    }
  }
  return true;
}

// Exclusive prefix of v over the 256 worker threads (one barrier; wsum: kWarps words nobody else uses meanwhile).
__device__ inline int workers_excl_scan(int v, int32_t* wsum, int* total) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  int t;
  int x = warp_excl_scan(v, lane, &t);
  if (lane == 0) wsum[warp] = t;
  sync_workers();
  int all = 0;
#pragma unroll
  for (int w = 0; w < kWarps; ++w) {
    if (w < warp) x += wsum[w];
    all += wsum[w];
  }
  *total = all;
  return x;
}

// Thread 0's release of everything the workers wrote before the last barrier, its count into a cell and the bounded wait
// until all of the row's tasks have counted in.  (The barrier orders the block's writes before the fence, which is
// cumulative: the other threads need none of their own.)
template <typename Arrive, typename There>
__device__ inline bool arrive_and_wait(Arrive arrive, There there, long long budget_ns) {
  fence_acq_rel_gpu();
  arrive();
  if (there()) return true;
  const unsigned long long t0 = global_timer_ns();
  while (!there()) {
    if (static_cast<long long>(global_timer_ns() - t0) > budget_ns) return false;
  }
  return true;
}

struct RowOneRankSmem {
  uint32_t skey[kSurvCap];       // the chunk's survivors (keys in bins >= the boundary bin), in no particular order
  uint16_t spos[kSurvCap];       // ... and their positions inside the chunk
  uint32_t und[kUndRowCap];      // the row's undecided entries
  uint32_t sub[1024];            // histogram of their upper ten bits
  uint32_t bits[1024];           // the chunk's selected positions (<= 32768 tokens)
  int32_t before[1024];          // selected positions in lower words
  uint32_t few[32];              // the entries of the sub-histogram's boundary bin
  int32_t wsum[2][kWarps], sums[4];
  int32_t n_s, n_above, n_mine, off, u, sub_bin, sub_above, n_few, tau, need_eq, ok;
};

// Exact row selection with one rank, after the boundary bin of the row is known (0: the row holds no more than top_k
// scores, everything valid is selected).  n_above_row: the row's scores in bins above it.
//
// Every step is a chain of latencies: the work itself is a few hundred keys.  So the exchange is one reserved range of one
// list per chunk, read by everybody with loads that do not depend on its length; the exact threshold comes from one
// histogram of ten more bits and a warp that ranks the handful of keys left; a chunk's share of the output needs only the
// sums over the lower chunks; and its position order comes from a bitmap of the selected positions.  The row's tasks were
// 22-26 us after the streaming with per-chunk slots, an adaptive search and ordered compactions; 11-15 us now (1 x 4096
// tokens: task 31.4 -> 20.5 us; 8 x 131072: 62.1 -> 51.8).
// Returns true when the row was published, false when it falls back (heavily tied scores) to the merge.
static __device__ __noinline__ bool chunk_publish_row_one_rank(const RowThreshold& rt, int32_t* status, int b, int chunk, int n_chunks,
                                                               const uint32_t* keys, int n_local, int base_pos, int top_k, int id_mul,
                                                               int id_add, uint32_t bin, int n_above_row, uint32_t n_und,
                                                               RowOneRankSmem& sm) {
  const RowExact& x = *rt.x;
  const RowOneRank& one = x.one;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const uint32_t lt = (1u << lane) - 1u;
  uint32_t off = 0u;   // (thread 0) the chunk's place in the row's list: a round trip to L2 under the search for the survivors
  if (tid == 0) {
    sm.n_s = sm.n_above = sm.n_mine = 0;
    sm.n_few = sm.need_eq = 0;
    sm.sums[0] = sm.sums[1] = sm.sums[2] = sm.sums[3] = 0;
    if (bin && n_und) off = atomicAdd(one.count, n_und);
    if (chunk == 0) *one.count_next = 0u;
  }
  sync_workers();
  // ---- the chunk's survivors
  const uint32_t floor_key = bin ? bin << kThrShift : 1u;
  const int n4 = n_local >> 2;   // (pages hold 64 or 128 tokens)
#pragma unroll 1
  for (int i0 = 0; i0 < n4; i0 += kBlockThreads) {
    const int i = i0 + tid;
    uint4 k = make_uint4(0u, 0u, 0u, 0u);
    if (i < n4) k = reinterpret_cast<const uint4*>(keys)[i];
    const uint32_t kk[4] = {k.x, k.y, k.z, k.w};
    uint32_t m[4];
    int n = 0;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      m[j] = __ballot_sync(0xffffffffu, kk[j] >= floor_key);
      n += __popc(m[j]);
    }
    if (n == 0) continue;
    int at = 0;
    if (lane == 0) at = atomicAdd(&sm.n_s, n);
    at = __shfl_sync(0xffffffffu, at, 0);
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int slot = at + __popc(m[j] & lt);
      if (kk[j] >= floor_key && slot < kSurvCap) {
        sm.skey[slot] = kk[j];
        sm.spos[slot] = static_cast<uint16_t>(4 * i + j);
      }
      at += __popc(m[j]);
    }
  }
  if (tid == 0) sm.off = static_cast<int>(off);
  sync_workers();
  const int n_s = min(sm.n_s, kSurvCap);
  // ---- those inside the boundary bin -> the row's list
  for (int i0 = 0; i0 < n_s; i0 += kBlockThreads) {
    const int i = i0 + tid;
    const uint32_t v = i < n_s ? sm.skey[i] : 0u;
    const bool in = bin != 0u && v != 0u && (v >> kThrShift) == bin;
    const uint32_t mi = __ballot_sync(0xffffffffu, in), ma = __ballot_sync(0xffffffffu, v != 0u && !in);
    int at = 0;
    if (lane == 0) {
      if (ma) atomicAdd(&sm.n_above, __popc(ma));
      if (mi) at = atomicAdd(&sm.n_mine, __popc(mi));
    }
    at = __shfl_sync(0xffffffffu, at, 0) + sm.off + __popc(mi & lt);
    if (in && at < kUndRowCap) one.list[at] = ((v & ((1u << kThrShift) - 1u)) << 8) | static_cast<uint32_t>(chunk);
  }
  for (int i = tid; i < 1024; i += kBlockThreads) sm.sub[i] = sm.bits[i] = 0u;
  sync_workers();
  if (tid == 0) {
    if (sm.n_s > kSurvCap) atomicAdd(one.count, kUndOverflow);
    one.n_above[chunk] = static_cast<uint32_t>(sm.n_above);
    const bool ok = arrive_and_wait([&] { red_relaxed_gpu_add_u64(x.ev.cell(x.ev_keys), 1ull); },
                                    [&] { return ld_acquire_gpu_u64(x.ev.cell(x.ev_keys)) >= x.keys_target; }, rt.budget_ns);
    if (!ok) report_failure(status, MDC_DEV_WAIT_TIMEOUT, -1000 - b, chunk, ld_acquire_gpu_u64(x.ev.cell(x.ev_keys)), x.keys_target);
    sm.ok = ok ? 1 : 0;
  }
  sync_workers();
  if (!sm.ok) return false;
  // ---- the row's list and the chunks' counts, all in flight together
  const uint32_t u_all = __ldcg(one.count);
  const int above_j = tid < n_chunks ? static_cast<int>(__ldcg(one.n_above + tid)) : 0;
  uint32_t e[4];
#pragma unroll
  for (int j = 0; j < 4; ++j) e[j] = __ldcg(one.list + j * kBlockThreads + tid);
  if (u_all > static_cast<uint32_t>(kUndRowCap)) return false;
  const int U = static_cast<int>(u_all);
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const int i = j * kBlockThreads + tid;
    if (i < U) {
      sm.und[i] = e[j];
      atomicAdd(&sm.sub[e[j] >> 18], 1u);
    }
  }
  for (int i = 4 * kBlockThreads + tid; i < U; i += kBlockThreads) {
    const uint32_t v = __ldcg(one.list + i);
    sm.und[i] = v;
    atomicAdd(&sm.sub[v >> 18], 1u);
  }
  sync_workers();
  // ---- the exact threshold: entries with value > tau are selected, need_eq of those equal to it
  int tau = -1, need_eq = 0;
  const int need = top_k - n_above_row;
  if (bin != 0u && need > 0 && need < U) {
    uint32_t c[4];
    const int first = 1023 - 4 * tid;   // thread t owns four bins, from the top
#pragma unroll
    for (int j = 0; j < 4; ++j) c[j] = sm.sub[first - j];
    int total;
    int cum = workers_excl_scan(static_cast<int>(c[0] + c[1] + c[2] + c[3]), sm.wsum[0], &total);
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      if (cum < need && cum + static_cast<int>(c[j]) >= need) {   // (one thread)
        sm.sub_bin = first - j;
        sm.sub_above = cum;
      }
      cum += static_cast<int>(c[j]);
    }
    sync_workers();
    const uint32_t sb = static_cast<uint32_t>(sm.sub_bin);
    const int need2 = need - sm.sub_above, m = static_cast<int>(sm.sub[sb]);
    if (m <= 32) {
      for (int i = tid; i < U; i += kBlockThreads) {
        const uint32_t v = sm.und[i];
        if ((v >> 18) == sb) sm.few[atomicAdd(&sm.n_few, 1)] = v >> 8;
      }
      sync_workers();
      if (warp == 0) {
        const uint32_t v = lane < m ? sm.few[lane] : 0u;
        int g = 0, q = 0;
        for (int j = 0; j < m; ++j) {
          const uint32_t o = __shfl_sync(0xffffffffu, v, j);
          g += o > v;
          q += o == v;
        }
        if (lane < m && g < need2 && g + q >= need2) {   // (every lane that ties writes the same)
          sm.tau = static_cast<int>(v);
          sm.need_eq = need2 - g;
        }
      }
    } else if (warp == 0) {   // many keys that agree in 22 bits: bit by bit over the list
      uint32_t t = sb << 10;
      for (int bit = 9; bit >= 0; --bit) {
        const uint32_t cand = t | (1u << bit);
        int n = 0;
        for (int i = lane; i < U; i += 32) n += (sm.und[i] >> 8) >= cand;
        if (__reduce_add_sync(0xffffffffu, n) >= need) t = cand;
      }
      int g = 0;
      for (int i = lane; i < U; i += 32) g += (sm.und[i] >> 8) > t;
      g = __reduce_add_sync(0xffffffffu, g);
      if (lane == 0) {
        sm.tau = static_cast<int>(t);
        sm.need_eq = need - g;
      }
    }
    sync_workers();
    tau = sm.tau;
    need_eq = sm.need_eq;
  }
  // ---- what the lower chunks select, and the ties of this one
  {
    int sel_before = tid < chunk ? above_j : 0, eq_before = 0, eq_mine = 0, all = above_j;
    for (int i = tid; i < U; i += kBlockThreads) {
      const int v = static_cast<int>(sm.und[i] >> 8), j = static_cast<int>(sm.und[i] & 255u);
      sel_before += j < chunk && v > tau;
      eq_before += j < chunk && v == tau;
      eq_mine += j == chunk && v == tau;
    }
    sel_before = __reduce_add_sync(0xffffffffu, sel_before);
    eq_before = __reduce_add_sync(0xffffffffu, eq_before);
    eq_mine = __reduce_add_sync(0xffffffffu, eq_mine);
    all = __reduce_add_sync(0xffffffffu, all);
    if (lane == 0) {
      atomicAdd(&sm.sums[0], sel_before);
      atomicAdd(&sm.sums[1], eq_before);
      atomicAdd(&sm.sums[2], eq_mine);
      atomicAdd(&sm.sums[3], all);
    }
  }
  sync_workers();
  const int base = sm.sums[0] + min(sm.sums[1], need_eq);
  const int my_eq = min(sm.sums[2], max(0, need_eq - sm.sums[1]));
  const bool some_ties = my_eq > 0 && my_eq < sm.sums[2];   // the lower positions win
  // ---- this chunk's share in position order
  const uint32_t tau_key = bin ? (bin << kThrShift) + static_cast<uint32_t>(max(tau, 0)) : 0u;
  auto taken = [&](int i) -> bool {
    const uint32_t k = sm.skey[i];
    if (bin == 0u || tau < 0 || k > tau_key) return true;   // (survivors all reach the boundary bin)
    if (k < tau_key || my_eq == 0) return false;
    if (!some_ties) return true;
    int lower = 0;
    for (int o = 0; o < n_s; ++o) lower += sm.skey[o] == tau_key && sm.spos[o] < sm.spos[i];
    return lower < my_eq;
  };
  for (int i = tid; i < n_s; i += kBlockThreads) {
    if (taken(i)) atomicOr(&sm.bits[sm.spos[i] >> 5], 1u << (sm.spos[i] & 31));
  }
  sync_workers();
  {
    const int per = ceil_div(ceil_div(n_local, 32), kBlockThreads);   // consecutive words of a thread
    int n = 0;
    for (int j = 0; j < per; ++j) n += __popc(sm.bits[tid * per + j]);
    int total;
    int run = workers_excl_scan(n, sm.wsum[1], &total);
    for (int j = 0; j < per; ++j) {
      sm.before[tid * per + j] = run;
      run += __popc(sm.bits[tid * per + j]);
    }
  }
  sync_workers();
  for (int i = tid; i < n_s; i += kBlockThreads) {
    const int pos = sm.spos[i];
    const uint32_t word = sm.bits[pos >> 5];
    if ((word >> (pos & 31)) & 1u) {
      const int o = base + sm.before[pos >> 5] + __popc(word & ((1u << (pos & 31)) - 1u));
      const uint32_t k = sm.skey[i];
      if (o < x.pt_cols) x.pt[o] = x.row_base + base_pos + pos;
      if (o < top_k) {
        x.out_v[o] = __uint_as_float((k & 0x80000000u) ? (k ^ 0x80000000u) : ~k);
        x.out_i[o] = (base_pos + pos) * id_mul + id_add;
      }
    }
  }
  if (tid == 0 && chunk == 0) {
    const int n = bin ? top_k : min(sm.sums[3], top_k);
    *x.k_valid = x.win_slots + min(n, x.pt_cols);
    *x.sel_c = n;
  }
  return true;
}

// hs: the chunk's histogram, already filled, keys: the chunk's keys.  scratch: the
// raw ring, idle by now.
template <typename Emit>
__device__ inline int chunk_emit_above_row_threshold(const RowThreshold& rt, int32_t* status, int b, int chunk, int n_chunks,
                                                     const uint32_t* keys, int n_local, int base_pos, int top_k, SelectScratch& sel,
                                                     uint32_t* hs, unsigned char* scratch, Emit emit, int id_mul = 1,
                                                     int id_add = 0) {
  constexpr int PER = kThrBins / kBlockThreads;   // bins a thread owns in the scan from the top
  static_assert(kThrBins % (4 * kBlockThreads) == 0, "the bin scan reads whole 16-byte pieces");
  const int tid = threadIdx.x, lane = tid & 31;
  uint32_t* gh = rt.hist + static_cast<int64_t>(b) * kThrBins;
#pragma unroll
  for (int q = 0; q < PER / 4; ++q) {
    const int i = q * kBlockThreads + tid;
    const uint4 h = reinterpret_cast<const uint4*>(hs)[i];
    const uint32_t v[4] = {h.x, h.y, h.z, h.w};
#pragma unroll
    for (int j = 0; j < 4; ++j)
      if (v[j]) atomicAdd(&gh[4 * i + j], v[j]);
  }
  sync_workers();
  const RowExact* x = rt.x;
  const bool many = x != nullptr && x->pcp > 1;   // the ranks settle the row together: the histograms are exchanged
  if (tid == 0) {
    bool ok = true;
    if (!many) {
      ok = arrive_and_wait([&] { atomicAdd(&rt.done[b], 1u); },
                           [&] { return static_cast<int32_t>(ld_acquire_gpu_u32(&rt.done[b]) - rt.target) >= 0; }, rt.budget_ns);
      if (!ok) report_failure(status, MDC_DEV_WAIT_TIMEOUT, -1 - b, chunk, ld_acquire_gpu_u32(&rt.done[b]), rt.target);
    } else {
      fence_acq_rel_gpu();
      const uint32_t before = atomicAdd(&rt.done[b], 1u);
      sel.hist_bnd = (before + 1u == rt.target) ? 1 : 0;   // the last task of this rank's row to count in
    }
    sel.bnd = ok ? 0 : -1;
    sel.c_gt = 0;
  }
  sync_workers();
  if (many) {
    if (sel.hist_bnd) {  // this rank's row histogram is complete: it goes to every rank, then one notify each
      __threadfence();
      const int64_t at = x->hist_off + static_cast<int64_t>(x->rank) * kRowHistBytes;
      for (int i = tid; i < kThrBins / 4; i += kBlockThreads) {
        const uint4 v = __ldcg(reinterpret_cast<const uint4*>(gh) + i);
        for (int d = 0; d < x->cp; ++d) reinterpret_cast<uint4*>(x->arena + x->arena_offsets[d] + at)[i] = v;
      }
      __threadfence_system();
      sync_workers();
      if (tid == 0)
        for (int d = 0; d < x->cp; ++d) x->ev.notify_1t(x->ev_hist, d);
    }
    if (tid == 0) {
      unsigned long long seen = 0;
      const bool ok = x->ev.poll_1t(x->ev_hist, x->hist_target, true, rt.budget_ns, &seen, 64);
      if (!ok) report_failure(status, MDC_DEV_WAIT_TIMEOUT, -500 - b, chunk, seen, x->hist_target);
      sel.bnd = ok ? 0 : -1;
    }
    sync_workers();
  }
  if (sel.bnd >= 0) {   // (uniform: written before the last barrier)
    // thread t owns the bins kThrBins-1-PER*t .. kThrBins-PER-PER*t, scanned from the top
    uint32_t c[PER];
    int local = 0;
#pragma unroll
    for (int j = 0; j < PER; ++j) c[j] = 0u;
    const int first = kThrBins - PER - PER * tid;   // lowest bin of this thread, a multiple of 4
    for (int r = 0; r < (many ? x->cp : 1); ++r) {
      const uint4* src = many ? reinterpret_cast<const uint4*>(x->arena + x->hist_off + static_cast<int64_t>(r) * kRowHistBytes)
                              : reinterpret_cast<const uint4*>(gh);
      src += first / 4;
#pragma unroll
      for (int q = 0; q < PER / 4; ++q) {
        const uint4 v = many ? ld_sys_u4(src + q) : __ldcg(src + q);   // bins first + 4q .. first + 4q + 3, ascending
        c[PER - 1 - 4 * q] += v.x;
        c[PER - 2 - 4 * q] += v.y;
        c[PER - 3 - 4 * q] += v.z;
        c[PER - 4 - 4 * q] += v.w;
      }
    }
#pragma unroll
    for (int j = 0; j < PER; ++j) local += static_cast<int>(c[j]);
    int total;
    int cum = workers_excl_scan(local, sel.wgt, &total);
#pragma unroll
    for (int j = 0; j < PER; ++j) {
      if (cum < top_k && cum + static_cast<int>(c[j]) >= top_k) {   // (one thread at most)
        sel.bnd = kThrBins - 1 - PER * tid - j;
        sel.c_gt = cum;
      }
      cum += static_cast<int>(c[j]);
    }
    sync_workers();
    const uint32_t bin = static_cast<uint32_t>(sel.bnd);   // 0 when the row holds fewer than k scores: everything passes
    if (x != nullptr && x->cp == 1) {
      if (chunk_publish_row_one_rank(rt, status, b, chunk, n_chunks, keys, n_local, base_pos, top_k, id_mul, id_add, bin, sel.c_gt,
                                     hs[bin], *reinterpret_cast<RowOneRankSmem*>(scratch)))
        return -1;
      sync_workers();
    }
    // this chunk's scores in the bins >= bin
    int mine = 0;
    for (int i = tid; i < kThrBins; i += kBlockThreads) mine += static_cast<uint32_t>(i) >= bin ? static_cast<int>(hs[i]) : 0;
    mine = __reduce_add_sync(0xffffffffu, mine);
    sync_workers();
    if (lane == 0) sel.weq[tid >> 5] = mine;
    sync_workers();
    int n_pass = 0;
#pragma unroll
    for (int w = 0; w < kWarps; ++w) n_pass += sel.weq[w];
    sync_workers();
    if (x != nullptr && x->cp > 1) {
      if (chunk_publish_row_exact(rt, status, b, chunk, n_chunks, keys, n_local, base_pos, top_k, id_mul, id_add, bin, n_pass,
                                  sel, *reinterpret_cast<RowExactScratch*>(scratch), hs))
        return -1;
      sync_workers();
    }
    if (n_pass <= top_k) {   // the chunk's share fits its list
      Threshold<uint32_t> th;
      th.tau = bin ? (bin << kThrShift) - 1u : 0u;
      th.need_eq = 0;
      th.n_sel = n_pass;
      return block_emit_keys(keys, n_local, th, sel, emit);
    }
  }
  const Threshold<uint32_t> th = block_select_bits_smem(keys, n_local, top_k, sel);
  return block_emit_keys(keys, n_local, th, sel, emit);
}

// Exact top-k of a whole request row across the blocks of a thread-block
// cluster (block rank = chunk), every block's keys and their histogram in its shared memory.
//
// First by histograms, like hist_select.cuh for one block: the row's boundary bin from the sum of the blocks' histograms
// over distributed shared memory, ten more bits the same way, then the few keys that share 22 bits, from all blocks.
// Every block computes the same sums, so no result has to be sent back.  Rows whose ties straddle the threshold (all
// blocks see that alike) go through the search below.
//
// The search: a 4-pass byte radix search for the row's k-th largest key with summed histograms, then
// each block emits its selected entries in position order at
// the offset given by the lower ranks' counts.  Ties at the threshold go to the
// smaller position.  Called by the 256 worker threads of
// every block of the cluster; n_local = 0 for a block that has nothing to offer.
template <int T>
__device__ void logits_row_select(const mdc_logits_params& p, int b, int chunk, int n_local, int base_pos, int chunk_tokens,
                                  const uint32_t* keys0, const uint32_t* hist0, HistSelectSmem& hsm, RegSelectScratch<kFusedRegE>& rsel,
                                  RowSelectScratch& rs) {
  namespace cg = cooperative_groups;
  cg::cluster_group cluster = cg::this_cluster();
  const int nr = static_cast<int>(cluster.num_blocks());
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  constexpr int E = kFusedRegE;
  for (int t = 0; t < T; ++t) {
    const uint32_t* keys = keys0 + t * chunk_tokens;
    const uint32_t* hist = hist0 + t * kThrBins;
    const int64_t out0 = (static_cast<int64_t>(b) * T + t) * p.top_k;
    auto put = [&](int pos, int o) {
      if (o < p.top_k) {
        const uint32_t kv = keys[pos];
        p.row_v[out0 + o] = __uint_as_float((kv & 0x80000000u) ? (kv ^ 0x80000000u) : ~kv);
        p.row_i[out0 + o] = (base_pos + pos) * p.id_mul + p.id_add;
      }
    };
    bool done = false;
    {
      if (tid == 0) {
        hsm.n_few = 0;
        hsm.bin = hsm.above = hsm.sub_bin = hsm.sub_above = 0;
      }
      // The whole histogram of every block would be 64 KB of remote loads (8100 cycles for four blocks): the sums of 16
      // bins each first, then the 16 bins of the group that holds the boundary.
      uint32_t c[16];
      load_top_bins(hist, tid, c);
      int local = 0;
#pragma unroll
      for (int j = 0; j < 16; ++j) local += static_cast<int>(c[j]);
      hsm.sup[tid] = local;
#pragma unroll
      for (int j = 0; j < 4; ++j) hsm.sub[4 * tid + j] = 0u;
      cluster.sync();
      int group = 0, total;
      for (int r = 0; r < nr; ++r) group += cluster.map_shared_rank(&hsm, r)->sup[tid];
      const int cum = group_excl_scan<1>(group, tid, hsm.wsum[0], &total);
      uint32_t tau = 1u;
      bool ties = false;
      if (total > p.top_k) {
        if (cum < p.top_k && cum + group >= p.top_k) {   // (one thread)
          hsm.bin = kThrBins - 1 - 16 * tid;
          hsm.above = cum;
        }
        sync_workers();
        const int top = hsm.bin, above0 = hsm.above;
        sync_workers();
        if (warp == 0) {
          uint32_t one[1] = {0u};
          if (lane < 16)
            for (int r = 0; r < nr; ++r) one[0] += cluster.map_shared_rank(hist, r)[top - lane];
          int all;
          const int below = above0 + warp_excl_scan(static_cast<int>(one[0]), lane, &all);
          write_boundary(one, below, top - lane, p.top_k, &hsm.bin, &hsm.above);
        }
        sync_workers();
        const uint32_t bin = static_cast<uint32_t>(hsm.bin);
        const int need = p.top_k - hsm.above;
        count_sub_bins(keys, n_local, bin, hsm.sub, tid);
        cluster.sync();
        uint32_t d[4] = {0u, 0u, 0u, 0u};   // bins 1023 - 4 * tid - j
        for (int r = 0; r < nr; ++r) {
          const uint4 v = *reinterpret_cast<const uint4*>(cluster.map_shared_rank(hsm.sub, r) + 1020 - 4 * tid);
          d[0] += v.w; d[1] += v.z; d[2] += v.y; d[3] += v.x;
        }
        int n_bin;
        const int dcum = group_excl_scan<1>(static_cast<int>(d[0] + d[1] + d[2] + d[3]), tid, hsm.wsum[1], &n_bin);
        write_boundary(d, dcum, 1023 - 4 * tid, need, &hsm.sub_bin, &hsm.sub_above);
        sync_workers();
        const uint32_t top22 = (bin << 10) | static_cast<uint32_t>(hsm.sub_bin);
        collect_few(keys, n_local, top22, hsm.few, &hsm.n_few, tid);
        cluster.sync();
        if (warp == 0) {   // lane l takes the l-th of the blocks' keys
          int m = 0;
          uint32_t mine = 0u;
          for (int r = 0; r < nr; ++r) {
            const HistSelectSmem* o = cluster.map_shared_rank(&hsm, r);
            const int n = o->n_few, at = lane - m;
            if (at >= 0 && at < min(n, 32)) mine = o->few[at];
            m += n;
          }
          if (lane == 0) {
            hsm.need_eq = -1;   // (differs from n_eq: the search)
            hsm.n_eq = 0;
          }
          __syncwarp();
          if (m <= 32) rank_few(mine, m, need - hsm.sub_above, lane, &hsm.tau, &hsm.need_eq, &hsm.n_eq);
        }
        sync_workers();
        tau = hsm.tau;
        ties = hsm.need_eq != hsm.n_eq;
      }
      if (!ties) {
        int n;
        const int before = mark_selected<1>(keys, n_local, tau, hsm, tid, &n);
        if (tid == 0) rs.cnt_gt = n;
        cluster.sync();
        int lower = 0, all = 0;
        for (int r = 0; r < nr; ++r) {
          const int g = cluster.map_shared_rank(&rs, r)->cnt_gt;
          lower += r < chunk ? g : 0;
          all += g;
        }
        emit_marked<1>(n_local, hsm, tid, before, n, [&](int pos, int slot) { put(pos, lower + slot); });
        if (chunk == 0 && tid == 0) p.row_c[static_cast<int64_t>(b) * T + t] = min(p.top_k, all);
        cluster.sync();   // nobody reuses or leaves its shared memory while a peer may read it
        done = true;
      }
    }
    if (done) continue;
    uint32_t key[E];
#pragma unroll
    for (int it = 0; it < E; ++it) {
      const int pos = it * kBlockThreads + tid;
      key[it] = pos < n_local ? keys[pos] : 0u;
    }
    uint32_t prefix = 0u;
    int kk = p.top_k;
    bool all = false;
    int low_bits = 0;  // undecided low bits when the search stopped early (the boundary bin is taken whole)
#pragma unroll 1
    for (int pass = 0; pass < 4; ++pass) {
      const int shift = 24 - 8 * pass, buf = pass & 1;
      rs.hist[buf][tid] = 0u;
      sync_workers();
      // run-length over this thread's keys: equal digits in a row cost one atomic
      uint32_t run_d = 0xffffffffu, run_n = 0u;
#pragma unroll
      for (int it = 0; it < E; ++it) {
        const bool in = key[it] != 0u && (pass == 0 || (key[it] >> (shift + 8)) == prefix);
        const uint32_t d = in ? (key[it] >> shift) & 255u : 0xffffffffu;
        if (d != run_d) {
          if (run_n) atomicAdd(&rs.hist[buf][run_d], run_n);
          run_d = d;
          run_n = 0u;
        }
        run_n += in;
      }
      if (run_n) atomicAdd(&rs.hist[buf][run_d], run_n);
      cluster.sync();
      // thread tid owns bin 255 - tid, summed over the cluster
      const int bin = 255 - tid;
      uint32_t g = 0u;
      for (int r = 0; r < nr; ++r) g += cluster.map_shared_rank(&rs.hist[buf][0], r)[bin];
      // inclusive scan over tid = number of keys in bins >= bin
      uint32_t inc = g;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, inc, o);
        if (lane >= o) inc += y;
      }
      if (lane == 31) rs.wsum[warp] = static_cast<int32_t>(inc);
      if (tid == 0) rs.digit = -1;
      sync_workers();
      uint32_t before = 0u, total = 0u;
#pragma unroll
      for (int w = 0; w < kWarps; ++w) {
        if (w < warp) before += static_cast<uint32_t>(rs.wsum[w]);
        total += static_cast<uint32_t>(rs.wsum[w]);
      }
      inc += before;
      const uint32_t exc = inc - g;
      if (!all && static_cast<int>(exc) < kk && kk <= static_cast<int>(inc)) {
        rs.digit = bin;
        rs.excl = static_cast<int32_t>(exc);
        rs.bin_cnt = static_cast<int32_t>(g);
      }
      sync_workers();
      if (pass == 0 && static_cast<int>(total) <= kk) all = true;  // fewer valid entries than k: take all
      if (all) break;  // (every block of the cluster sees the same sums and takes the same exit)
      prefix = (prefix << 8) | static_cast<uint32_t>(rs.digit);
      kk -= rs.excl;
      if (rs.bin_cnt == kk && shift > 0) {  // the whole boundary bin is selected: no finer digit needed
        low_bits = shift;
        break;
      }
    }
    // Threshold key: entries above it are selected outright, kk of those equal to it in position
    // order.  After an early stop everything at or above prefix << low_bits is selected.
    uint32_t tau = all ? 0u : prefix;
    if (low_bits > 0) {
      tau = (prefix << low_bits) - 1u;
      kk = 0;
      if ((prefix << low_bits) == 0u) all = true;
    }
    int c_gt = 0, c_eq = 0;
#pragma unroll
    for (int it = 0; it < E; ++it) {
      c_gt += all ? key[it] != 0u : key[it] > tau;
      c_eq += !all && key[it] == tau;
    }
    c_gt = __reduce_add_sync(0xffffffffu, c_gt);
    c_eq = __reduce_add_sync(0xffffffffu, c_eq);
    if (tid == 0) rs.cnt_gt = rs.cnt_eq = 0;
    sync_workers();
    if (lane == 0) {
      atomicAdd(&rs.cnt_gt, c_gt);
      atomicAdd(&rs.cnt_eq, c_eq);
    }
    cluster.sync();
    int gt_before = 0, eq_before = 0, gt_all = 0, eq_all = 0, eq_mine = 0;
    for (int r = 0; r < nr; ++r) {
      const RowSelectScratch* o = cluster.map_shared_rank(&rs, r);
      const int g1 = o->cnt_gt, e1 = o->cnt_eq;
      if (r < chunk) {
        gt_before += g1;
        eq_before += e1;
      }
      if (r == chunk) eq_mine = e1;
      gt_all += g1;
      eq_all += e1;
    }
    const int need_row = all ? 0 : kk;
    const int need = max(0, min(need_row - eq_before, eq_mine));   // ties this block contributes
    const int base = gt_before + min(eq_before, need_row);         // entries selected in lower chunks
    // position-ordered emit as a rolled loop over the scores (compact code: it runs once per block)
    Threshold<uint32_t> th;
    th.tau = tau;
    th.need_eq = need;
    th.n_sel = 0;
    block_emit_selected<uint32_t>(
        [&](int pos, bool& valid) {
          valid = keys[pos] != 0u;
          return keys[pos];
        },
        n_local, th, *reinterpret_cast<SelectScratch*>(&rsel), [&](int pos, int slot) { put(pos, base + slot); });
    if (chunk == 0 && tid == 0) p.row_c[static_cast<int64_t>(b) * T + t] = min(p.top_k, gt_all + min(eq_all, need_row));
    cluster.sync();  // counts and histograms are reused by the next query token; nobody leaves while a peer may read
  }
}

// Whether the chunk's scores are kept as sortable keys and counted: for a row threshold, and in the stand-alone kernels where
// they fit.
template <int FMT, int PAGE, int T, bool ALONE, bool THR>
__device__ __forceinline__ bool logits_keeps_keys(bool fused, int chunk_tokens) {
  return ALONE ? fused && logits_as_keys<FMT, PAGE>(T, chunk_tokens) : THR;
}

// The stages whose copies a group may have on their way when it gives up in front of the product of `tile` and query token
// t: first, first + groups, ... below end.  (A group's stages are first loaded two at a time; its stage `tile` is handed the
// copy of tile + 2 * groups once it is decoded, with t = 0.  A stage that has been waited for is not in the range: its
// barrier may be two phases on, which a wait by parity takes for not complete.)
struct StageRange {
  int first, end;
};
__host__ __device__ inline StageRange stages_on_their_way(int tile, int t, int groups, int n_tiles) {
  const int first = t > 0 ? tile + groups : tile;
  return {first, first + 2 * groups < n_tiles ? first + 2 * groups : n_tiles};
}

// Scores the chunk.  smem: dynamic shared memory base (1024 B aligned), laid out by logits_smem_layout.  All threads of the
// block call it.  ALONE: the stand-alone kernels; THR: the persistent kernel with a row threshold, `hist_next`: the row's
// histogram of the next step, of which this task zeroes its slice.  Returns the chunk's pages, or their complement (< 0) when
// a wait ran out.
template <int FMT, int PAGE, int T, bool ALONE, bool ROWK, bool THR>
__device__ __forceinline__ int logits_stream(const mdc_logits_params& p, const CUtensorMap* pages, int b, int chunk, unsigned char* smem,
                                             uint32_t* hist_next) {
  using PG = IdxPage<FMT, PAGE>;
  constexpr int N = T * kIdxHeads;
  constexpr int G = ALONE ? kLogitsGroups : kMegaGroups, NS = 2 * G;   // groups, raw stages in use
  constexpr int kThreads = ALONE ? kLogitsThreads : kMegaThreads;
  constexpr int kCopyWarp = kWarps, kTmemWarp = kWarps + 1;   // set-up: the first ring fill and the barriers; tensor memory
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const bool fused = p.cand_v != nullptr || (ROWK && p.row_v != nullptr);
  const int chunk_tokens = p.blocks_per_chunk * PAGE;
  const bool as_keys = logits_keeps_keys<FMT, PAGE, T, ALONE, THR>(fused, chunk_tokens);
  const LogitsSmem L = logits_smem_layout<FMT, PAGE>(T, chunk_tokens, fused, as_keys);
  uint32_t* hs = reinterpret_cast<uint32_t*>(smem + L.hist);

  unsigned char* qb = smem + L.qb;
  unsigned char* ring = smem + L.ring;
  uint64_t* raw_full = reinterpret_cast<uint64_t*>(smem + L.bars);
  uint64_t* mma_done = raw_full + NS;   // [G]: the group's product is complete
  uint32_t* misc = reinterpret_cast<uint32_t*>(smem + L.misc);
  volatile uint32_t* abort_flag = misc + 1;
  int32_t* page_id = reinterpret_cast<int32_t*>(smem + L.page_ok);
  float* wsc = reinterpret_cast<float*>(smem + L.wsc);
  float* scores = reinterpret_cast<float*>(smem + L.scores);

  const int blk0 = chunk * p.blocks_per_chunk;
  const int seq_len = p.seq_lens ? p.seq_lens[b] : p.max_pages * PAGE;
  const int limit = max(0, seq_len - p.window_exclude);
  // pages this block actually streams: the whole chunk when logits are
  // written out, only pages below the selection limit when fused
  int blk_end = min(blk0 + p.blocks_per_chunk, p.max_pages);
  if (fused) blk_end = min(blk_end, ceil_div(limit, PAGE));
  const int n_pages = max(0, blk_end - blk0);
  const int n_tiles = ceil_div(n_pages, PG::kTilePages);  // pipeline stages of this block
  const int32_t* bt = p.block_table + static_cast<int64_t>(b) * p.max_pages;
  const int table_end = min(p.blocks_per_chunk, p.max_pages - blk0);   // the chunk's entries of the page table
  int bad_page = 0;
  constexpr long long kBudget = 1ll << 31, kDrain = 1ll << 24;  // clock cycles a role waits before it gives up, and after

  // ---------------- prologue.  One warp fills the ring at once; the query, the page table and tensor memory are
  // set up meanwhile.
  const uint64_t stream_policy = l2_policy_evict_first();  // the index cache is read once per step
  // Loads page `id` (-1 = none) into page slot cp of raw stage cs; one lane per page, the lanes of a stage next to each other
  // (cp = lane % pages of a stage).  `go`: alike in the lanes of a stage.
  auto refill = [&](bool go, int cs, int cp, int id) {
    const uint32_t there = __ballot_sync(0xffffffffu, id >= 0);
    const int n = __popc((there >> (lane - cp)) & ((1u << PG::kTilePages) - 1u));
    if (go && cp == 0) {
      if (n == 0) mbar_arrive(&raw_full[cs]);
      else mbar_expect_tx(&raw_full[cs], static_cast<uint32_t>(n) * PG::kBytes);
    }
    __syncwarp();
    if (go && id >= 0)
      tma_load_3d_hint(ring + cs * PG::kStageBytes + cp * PG::kBytes, pages, 0, 0, id, &raw_full[cs], stream_policy);
  };
  if (warp == kCopyWarp) {
    if (lane == 0) {
      for (int s = 0; s < NS + G; ++s) mbar_init(&raw_full[s], 1);
      for (int i = 1; i < 16; ++i) misc[i] = 0;
      mbar_fence_init();
    }
    fence_proxy_async_smem();   // (the ring may have been the previous task's scratch)
    __syncwarp();
    // (read up to the chunk's end: the load does not wait for the sequence's length)
    int id = lane < table_end ? bt[blk0 + lane] : -1;
    if (lane >= n_pages || id >= p.num_pages) id = -1;
    refill(lane < min(NS, n_tiles) * PG::kTilePages, lane / PG::kTilePages, lane % PG::kTilePages, id);
  } else if (warp < kWarps) {
    logits_stage_query<T>(p, b, qb, wsc);
    fence_proxy_async_smem();  // the tensor core reads the query block through the async proxy
  } else {
    if (warp == kTmemWarp) umma::tmem_alloc(misc, kTmemCols);
    if (as_keys) {
      const int t = tid - kBlockThreads - (warp > kCopyWarp ? 32 : 0), nt = kThreads - kBlockThreads - 32;
      for (int i = t; i < T * kThrBins / 4; i += nt) reinterpret_cast<uint4*>(hs)[i] = make_uint4(0u, 0u, 0u, 0u);
      if (THR) {  // this task's slice of the next step's histogram
        const int per = ceil_div(kThrBins, p.n_chunks), end = min(kThrBins, (chunk + 1) * per);
        for (int i = chunk * per + t; i < end; i += nt) hist_next[i] = 0u;
      }
    }
    const int t = tid - kBlockThreads - (warp > kCopyWarp ? 32 : 0);
    for (int i = t; i < table_end + 4; i += kThreads - kBlockThreads - 32) {  // (+4: the slots behind the last page)
      int32_t id = i < table_end ? bt[blk0 + i] : -1;
      if (i >= n_pages) {
        id = -1;
      } else if (id < 0 || id >= p.num_pages) {
        report_failure(p.status, MDC_DEV_BAD_INDEX, id, blk0 + i, 0, 0);
        id = -1;
        bad_page = 1;
      }
      page_id[i] = id;
    }
  }
  umma::fence_before_sync();
  const bool any_bad = __syncthreads_or(bad_page) != 0;
  umma::fence_after_sync();
  const uint32_t tmem = misc[0];
  const float neg_inf = __int_as_float(0xff800000);

  auto give_up = [&](int what, int idx) {
    report_failure(p.status, MDC_DEV_COPY_TIMEOUT, what, idx, 0, 0);
    *abort_flag = 1;
  };
  {
    // ---------------- the groups: thread = token row; group g (warps 4g..4g+3) takes the stages g, g + G, ...
    const int quad = warp & 3, grp = warp >> 2;  // TMEM lane quadrant, group
    const int row = quad * 32 + lane;
    const int pp = row / PAGE, tok = row % PAGE;
    const uint32_t t_acc = tmem + grp * 64, t_a = tmem + (G + grp) * 64;
    const uint32_t t_lane = static_cast<uint32_t>(quad * 32) << 16;
    const int row_at = pp * PG::kBytes + tok * 64, turn = (tok * 8) & 0x30;   // the row in its stage: chunk j at (16 j) ^ turn
    const int sf_at = PG::swizzled(PG::kData + (FMT == MDC_FMT_NVFP4 ? tok * 8 : (tok % 32) * 16 + (tok / 32) * 4)) - tok * 64;   // from there
    const int n_here = n_pages * PAGE, n_cand = limit - blk0 * PAGE;   // positions that exist; that can be selected
    auto emit = [&](int local, int t, float score) {   // local: position inside the chunk
      if (local < n_here) {
        float val = score;
        if (any_bad && page_id[local / PAGE] < 0) val = neg_inf;
        if (as_keys) {   // 0 = not a candidate
          const uint32_t key = local < n_cand ? max(sortable_u32(val), 1u) : 0u;
          reinterpret_cast<uint32_t*>(scores)[t * chunk_tokens + local] = key;
          if (key) atomicAdd(&hs[t * kThrBins + (key >> kThrShift)], 1u);
        } else if (fused) scores[t * chunk_tokens + local] = val;
        else p.logits[(static_cast<int64_t>(b) * T + t) * p.logits_stride + static_cast<int64_t>(blk0) * PAGE + local] = val;
      }
    };
    constexpr uint32_t idesc = umma::idesc_f16(kTileTok, kIdxHeads, 0);
    const uint32_t qb_u = smem_u32(qb);
    // Step n of the group: the product of stage grp + G * (n / T) and query token n % T is issued, the scores of step n - 1
    // are computed.  A wait that runs out in any lane ends its warp's steps: it issues and writes nothing more, walks the
    // barriers that are left (the group's other warps go on until the block's flag ends a wait of theirs, or to the end) and
    // waits for what it has put on its way.
    // (The tensor-memory loads stand outside the conditions, the first step's read nothing of use: inside the persistent
    // kernel conditional ones made every function of it spill.)
    const int steps = grp < G && n_tiles > grp ? ceil_div(n_tiles - grp, G) * T : 0;
    int n = 0, tile = grp, t = 0;
#pragma unroll 1
    for (; n <= steps && steps > 0; ++n) {
      const bool issue = n < steps, decode = issue && t == 0, gate = n > 0;
      const int slot = tile % NS;
      const unsigned char* st = ring + slot * PG::kStageBytes + row_at;
      uint4 d = make_uint4(0u, 0u, 0u, 0u);
      uint2 sf = make_uint2(0u, 0u);  // the row's block scales
      bool there = true, done = true;   // the raw stage; the product
      if (decode) {
        there = mbar_wait(&raw_full[slot], (tile / NS) & 1, kBudget, abort_flag);
        // (a page that is not there leaves what the stage held: its rows' scores are replaced)
        d = *reinterpret_cast<const uint4*>(st + turn);
        if (FMT == MDC_FMT_NVFP4) sf = *reinterpret_cast<const uint2*>(st + sf_at);
        else sf.x = *reinterpret_cast<const uint32_t*>(st + sf_at);
      }
      float x[4][16], s4[4] = {0.f, 0.f, 0.f, 0.f};
      // Heads 16c .. 16c + 15 of the row: x + |x| is exactly 0 or 2x; the weighted sums run as packed fp32 pairs.
      const int done_tile = t == 0 ? tile - G : tile, done_t = t == 0 ? T - 1 : t - 1;   // of step n - 1
      auto gate_heads = [&](int c, const float (&v)[16]) {
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const float4 w = reinterpret_cast<const float4*>(wsc + done_t * kIdxHeads)[4 * c + i];
          ffma2(s4[0], s4[1], v[4 * i] + fabsf(v[4 * i]), v[4 * i + 1] + fabsf(v[4 * i + 1]), w.x, w.y);
          ffma2(s4[2], s4[3], v[4 * i + 2] + fabsf(v[4 * i + 2]), v[4 * i + 3] + fabsf(v[4 * i + 3]), w.z, w.w);
        }
      };
      if (gate && there) done = mbar_wait(&mma_done[grp], (n - 1) & 1, kBudget, abort_flag);
      const bool go = __all_sync(0xffffffffu, there && done);   // (the lanes may have seen the last poll differently)
      umma::fence_after_sync();
      umma::tmem_ld16_f(t_acc + t_lane, x[0]);   // on its way while the new stage is decoded
      umma::tmem_ld16_f(t_acc + t_lane + 16, x[1]);
      if (decode) {
#pragma unroll
        for (int j = 0; j < 4; ++j) {  // 16-byte chunk j = 32 dims = 16 columns
          const uint4 following = *reinterpret_cast<const uint4*>(st + (((16 * j + 16) & 48) ^ turn));
          uint32_t s_lo, s_hi;  // fp16x2 block scale of dims 0-15 and 16-31 of the chunk
          if (FMT == MDC_FMT_NVFP4) {   // scale bytes 2j, 2j + 1
            const uint32_t two = e4m3x2_to_f16x2(static_cast<uint16_t>(sf.x & 0xffff));
            s_lo = bcast_lo(two);
            s_hi = bcast_hi(two);
            sf.x = __funnelshift_r(sf.x, sf.y, 16);
            sf.y >>= 16;
          } else {
            s_lo = s_hi = ue8m0_to_f16x2(sf.x & 0xff);
            sf.x >>= 8;
          }
          const uint32_t w4[4] = {d.x, d.y, d.z, d.w};
          uint32_t out[16];
#pragma unroll
          for (int q4 = 0; q4 < 4; ++q4) {
            uint32_t e[4];
            e2m1x8_to_f16x2(w4[q4], e);  // e[i] = elements (2i, 2i+1) of the word
#pragma unroll
            for (int i = 0; i < 4; ++i) out[4 * q4 + i] = hmul2_u32(e[i], q4 < 2 ? s_lo : s_hi);
          }
          umma::tmem_st16(t_a + t_lane + 16 * j, out);
          d = following;
        }
      }
      // half of the heads while the stores land and the other half is on its way
      umma::wait_ld();
      if (!go) {
        const bool all_there = __all_sync(0xffffffffu, there);
        if (lane == 0) give_up(all_there ? 5 : 3, tile);
        break;
      }
      umma::tmem_ld16_f(t_acc + t_lane + 32, x[2]);
      umma::tmem_ld16_f(t_acc + t_lane + 48, x[3]);
      if (gate) {
        gate_heads(0, x[0]);
        gate_heads(1, x[1]);
      }
      umma::wait_ld();
      if (issue) {
        umma::wait_st();
        umma::fence_before_sync();
        asm volatile("bar.sync %0, 128;" ::"r"(4 + grp) : "memory");   // A is complete, the accumulator and the raw stage are read
        if (quad == 0) {
          umma::fence_after_sync();
          if (umma::elect_one()) {
            umma::mma_f16_ts_x8(t_acc, t_a, umma::smem_desc_sw128(qb_u + t * (kIdxHeads * 128)), N * 128, idesc);
            umma::commit(&mma_done[grp]);
          }
          __syncwarp();
        } else if (quad == 1 && decode) {
          const int next = tile + NS, i = next * PG::kTilePages + lane;
          refill(next < n_tiles && lane < PG::kTilePages, slot, lane < PG::kTilePages ? lane : 0,
                 next < n_tiles && lane < PG::kTilePages ? page_id[i] : -1);
        }
        if (++t == T) {
          t = 0;
          tile += G;
        }
      }
      if (!gate) continue;
      gate_heads(2, x[2]);
      gate_heads(3, x[3]);
      emit(done_tile * kTileTok + row, done_t, (s4[0] + s4[1]) + (s4[2] + s4[3]));
    }
    if (steps > 0 && n <= steps) {   // gave up in step n (alike in the warp's lanes)
      umma::wait_st();
      for (int i = n; i < steps; ++i) asm volatile("bar.sync %0, 128;" ::"r"(4 + grp) : "memory");
      // (bounded, without the block's flag)
      if (quad == 0 && n > 0) mbar_wait(&mma_done[grp], (n - 1) & 1, kDrain);
      const StageRange on_way = stages_on_their_way(tile, t, G, n_tiles);
      if (quad == 1)
        for (int i = on_way.first; i < on_way.end; i += G) mbar_wait(&raw_full[i % NS], (i / NS) & 1, kDrain);
    }
  }

  // ---------------- common exit of the pipeline
  umma::fence_before_sync();
  __syncthreads();
  umma::fence_after_sync();
  const bool failed = *abort_flag != 0;
  if (warp == kTmemWarp) umma::tmem_dealloc(tmem, kTmemCols);
  if (warp == kCopyWarp && lane < NS + G) mbar_inval(raw_full + lane);   // the memory is reused by the block's next task
  return failed ? ~n_pages : n_pages;
}
// The tile: the scores, then what becomes of them.  All threads of the block call it.
// Returns, to the worker threads alike, the entries of the (last) candidate list, or -1 when the row has been published or
// nothing was written.
template <int FMT, int PAGE, int T, bool ALONE, bool ROWK = false, bool THR = false>
__device__ __forceinline__ int logits_tile(const mdc_logits_params& p, const CUtensorMap* pages, int b, int chunk, unsigned char* smem,
                                           const RowThreshold* rt = nullptr) {
  using PG = IdxPage<FMT, PAGE>;
  const int tid = threadIdx.x, warp = tid >> 5;
  const int streamed = logits_stream<FMT, PAGE, T, ALONE, ROWK, THR>(p, pages, b, chunk, smem,
                                                                     THR ? rt->hist_next + static_cast<int64_t>(b) * kThrBins : nullptr);
  const bool failed = streamed < 0, row_mode = ROWK && p.row_v != nullptr, fused = p.cand_v != nullptr || row_mode;
  const int n_pages = failed ? ~streamed : streamed, chunk_tokens = p.blocks_per_chunk * PAGE;
  const bool as_keys = logits_keeps_keys<FMT, PAGE, T, ALONE, THR>(fused, chunk_tokens);
  const LogitsSmem L = logits_smem_layout<FMT, PAGE>(T, chunk_tokens, fused, as_keys);
  uint32_t* hs = reinterpret_cast<uint32_t*>(smem + L.hist);
  unsigned char* ring = smem + L.ring;
  SelectScratch& sel = *reinterpret_cast<SelectScratch*>(smem + L.sel);
  float* scores = reinterpret_cast<float*>(smem + L.scores);
  const int n_local = n_pages * PAGE, base_pos = chunk * chunk_tokens;
  uint32_t* keys0 = reinterpret_cast<uint32_t*>(scores);
  auto put = [&](int t, int pos, int slot) {   // entry `slot` of query token t's list (keys kept as keys)
    const int64_t at = ((static_cast<int64_t>(b) * T + t) * p.n_chunks + chunk) * p.top_k + slot;
    const uint32_t kv = keys0[t * chunk_tokens + pos];
    p.cand_v[at] = __uint_as_float((kv & 0x80000000u) ? (kv ^ 0x80000000u) : ~kv);
    p.cand_i[at] = (base_pos + pos) * p.id_mul + p.id_add;
  };
  int32_t* selected = reinterpret_cast<int32_t*>(smem + L.misc) + 12;       // [T] entries of a token's list, -1: to be selected by a search
  const bool by_hist = ALONE && as_keys && !(ROWK && row_mode) && !failed;
  if constexpr (ALONE) {
    if (by_hist) {
      // one query token per group of eight warps
      static_assert(T == 1 || kLogitsThreads >= 2 * kBlockThreads, "a second group of eight warps");
      HistSelectSmem* hsm = reinterpret_cast<HistSelectSmem*>(ring);   // (the raw ring is idle by now)
      if (warp < kWarps) {
        const int n = hist_select_emit<1>(keys0, n_local, p.top_k, hs, hsm[0], tid, [&](int pos, int slot) { put(0, pos, slot); });
        if (tid == 0) selected[0] = n;
      } else if (T == 2 && warp < 2 * kWarps) {
        const int n = hist_select_emit<2>(keys0 + chunk_tokens, n_local, p.top_k, hs + kThrBins, hsm[1], tid - kBlockThreads,
                                          [&](int pos, int slot) { put(1, pos, slot); });
        if (tid == kBlockThreads) selected[1] = n;
      }
      __syncthreads();
    }
  }
  if (warp >= kWarps) return -1;
  if (ROWK && row_mode) {
    // every block of the cluster walks the same barriers, also one whose pipeline gave up
    logits_row_select<T>(p, b, chunk, failed ? 0 : n_local, base_pos, chunk_tokens, keys0, hs, *reinterpret_cast<HistSelectSmem*>(ring),
                         *reinterpret_cast<RegSelectScratch<kFusedRegE>*>(smem + L.sel),
                         *reinterpret_cast<RowSelectScratch*>(smem + L.row));
    return -1;
  }
  int n = -1;
  if (failed) return n;

  if (fused) {
    for (int t = 0; t < T; ++t) {
      uint32_t* keys = keys0 + t * chunk_tokens;
      auto emit = [&](int pos, int slot) { put(t, pos, slot); };
      if constexpr (THR) {
        n = chunk_emit_above_row_threshold(*rt, p.status, b, chunk, p.n_chunks, keys, n_local, base_pos, p.top_k, sel, hs, ring, emit,
                                           p.id_mul, p.id_add);
      } else if (!by_hist) {
        const int limit = max(0, (p.seq_lens ? p.seq_lens[b] : p.max_pages * PAGE) - p.window_exclude);
        n = fused_chunk_select(scores + t * chunk_tokens, keys, n_local, base_pos, limit, p.top_k, sel, emit);
      } else {
        n = selected[t];
        if (n < 0) {   // ties at the threshold
          const Threshold<uint32_t> th = block_select_bits_smem(keys, n_local, p.top_k, sel);
          n = block_emit_keys(keys, n_local, th, sel, emit);
        }
      }
      if (tid == 0) p.cand_c[(static_cast<int64_t>(b) * T + t) * p.n_chunks + chunk] = n;
    }
  }
  return n;
}

}  // namespace mdc

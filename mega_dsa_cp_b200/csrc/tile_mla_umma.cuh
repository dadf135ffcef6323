// Sparse MLA decode-attention tile on the 5th-generation tensor cores: 128
// query heads of one (b, t) row against a range of KV slots, 128 of the 512
// output columns per block (four blocks cover a row's output; each repeats the
// cheap-to-issue Q.K^T so that the output accumulator fits tensor memory).
//
// Operands are bf16 (DQK 576 or 512) or e4m3 (DQK 512, probabilities rounded
// to e4m3).  A K step of one MMA is 32 bytes of either type and every panel
// below is 128 bytes wide, so both types share all address arithmetic.
//
// Tensor memory (512 columns x 128 lanes, lane = head):
//   Q   row bytes / 4 columns   the A operand of S = Q K^T, loaded once
//   O   128 columns             fp32 output accumulator
//   S   64 columns              fp32 logits of one 64-slot tile
//   P   at most 32 columns      its probabilities, the A operand of O += P V
// Shared memory: a ring of KV tiles, each 64 slots stored as panels of 64
// rows x 128 bytes with the 128-byte swizzle.  One image serves both products:
// a panel is a K-major B operand for Q K^T (row = slot, 128 bytes of dims per
// row) and, read "MN-major", the B operand of P V (for a fixed slot the output
// columns are contiguous), so V needs no transposed copy.
//
// Order of a tile's phases.  As soon as the softmax warps hold S of tile i in
// registers, Q K^T of tile i + 1 overwrites it, so the tensor core works while they
// compute P of tile i; P V of tile i follows.  The two products are issued by a warp each: one
// issuing both spent 500 cycles per tile on waits and issue slots with the tensor core idle (2500
// cycles per tile, of which the MMAs are 1540).
//
// Measured, 32 rows x 2048 selected slots: 65.4 us with one warp issuing both products -> 50.7 to 57.9 now, by the box (a box
// gives the same time call after call, the boxes differ); e4m3, 16 rows x 512 slots and the window: 59.4 us on the mma.sync
// tile, 17.2 here.
//
// Roles (448 threads): warps 0-3 softmax (thread = head: no cross-thread
// reductions; reads S with tcgen05.ld, writes P with tcgen05.st, rescales O
// only when the running maximum grew by more than 2^8; e4m3 probabilities follow
// the running maximum exactly), warps 4-11 gather KV rows with 16-byte cp.async (a
// warp instruction reads 512 contiguous bytes of one row), warp 12 issues
// the MMAs of Q K^T and warp 13 those of P V.  All waits are bounded.
#pragma once

#include "common.cuh"
#include "tile_mla.cuh"
#include "umma.cuh"

namespace mdc {

constexpr int kMuHeads = 128;   // heads per block (= UMMA M)
constexpr int kMuTile = 64;     // slots per tile
constexpr int kMuDv = 128;      // output columns per block
constexpr int kMuThreads = 448;   // 14 warps
constexpr int kMuGatherWarp0 = 4, kMuGatherWarps = 8, kMuIssueWarp = 12, kMuPvWarp = 13;

template <int DQK, bool FP8 = false>
struct MlaUmmaSmem {
  static constexpr int kRowBytes = DQK * (FP8 ? 1 : 2);
  static constexpr int kPanels = kRowBytes / 128;
  static constexpr int kStageBytes = kPanels * kMuTile * 128;
  static constexpr int kStages = FP8 ? 6 : 3;           // what fits beside ~3 KB of bookkeeping in 226 KB
  static constexpr int kK = 0;
  static constexpr int kBars = kStages * kStageBytes;   // full[S], free[S], s_ready, s_taken, p_ready, q_ready, o_final, qs_ready
  static constexpr int kNumBars = 2 * kStages + 6;
  static constexpr int kMisc = kBars + kNumBars * 8;    // [0] tmem base, [1] abort flag
  static constexpr int kValid = kMisc + 64;             // [S][8] bytes: validity bits of 8 slots per gather warp
  static constexpr int kTotal = kValid + kStages * 8 + 56;
};

namespace umma {
// Shared-memory B operand read MN-major with the 128-byte swizzle: for one K index (row of 128
// bytes) 64 consecutive N elements; 8 K rows form a 1024-byte atom.  lbo = bytes between
// consecutive 64-element N blocks, sbo = bytes between consecutive groups of 8 K rows.
__device__ inline uint64_t smem_desc_mn_sw128(uint32_t addr, uint32_t lbo, uint32_t sbo) {
  uint64_t d = 0;
  d |= static_cast<uint64_t>((addr & 0x3ffff) >> 4);
  d |= static_cast<uint64_t>((lbo >> 4) & 0x3fff) << 16;
  d |= static_cast<uint64_t>((sbo >> 4) & 0x3fff) << 32;
  d |= static_cast<uint64_t>(1) << 46;
  d |= static_cast<uint64_t>(2) << 61;
  return d;
}
// instruction descriptor, fp32 accumulator: bf16 operands of kind::f16, or e4m3 operands of
// kind::f8f6f4; b_mn = B operand MN-major
__host__ __device__ constexpr uint32_t idesc_mla(bool fp8, int M, int N, bool b_mn) {
  return (1u << 4) | (fp8 ? 0u : (1u << 7) | (1u << 10)) | (b_mn ? (1u << 16) : 0u) | (static_cast<uint32_t>(N >> 3) << 17) |
         (static_cast<uint32_t>(M >> 4) << 24);
}
}  // namespace umma

__device__ inline float ex2_approx(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

// The four bytes of e4m3 probabilities of one tensor-memory column.  The sum takes the rounded values, so
// they come back as fp32.
__device__ inline uint32_t pack_e4m3x4(float (&x)[4]) {
  uint16_t a, b;
  asm("cvt.rn.satfinite.e4m3x2.f32 %0, %1, %2;" : "=h"(a) : "f"(x[1]), "f"(x[0]));
  asm("cvt.rn.satfinite.e4m3x2.f32 %0, %1, %2;" : "=h"(b) : "f"(x[3]), "f"(x[2]));
  uint32_t h0, h1;
  asm("cvt.rn.f16x2.e4m3x2 %0, %1;" : "=r"(h0) : "h"(a));
  asm("cvt.rn.f16x2.e4m3x2 %0, %1;" : "=r"(h1) : "h"(b));
  const float2 f0 = __half22float2(*reinterpret_cast<__half2*>(&h0)), f1 = __half22float2(*reinterpret_cast<__half2*>(&h1));
  x[0] = f0.x; x[1] = f0.y; x[2] = f1.x; x[3] = f1.y;
  return static_cast<uint32_t>(a) | (static_cast<uint32_t>(b) << 16);
}

constexpr int kMuRows = kMuTile / kMuGatherWarps;   // rows a gather warp fetches of every tile
constexpr int kMuBatch = 32 / kMuRows;              // tiles whose row pointers are looked up together

// Row pointers of this warp's slots of the tiles [tile, end): lane l looks up row l % 8 of the tile l / 8
// further on, so the page-table reads of four tiles are one instruction (nullptr = masked slot).  The
// first `win` slots of the tiles are the window's, the gathered pool's follow.
template <int DQK, int ESZ>
__device__ inline const unsigned char* mla_umma_row_ptrs(const mdc_sparse_mla_params& p, int r, int tile, int end, int win,
                                                         int k_valid, int win_valid, int gw, int lane) {
  const int t = tile + lane / kMuRows;
  if (t >= end) return nullptr;
  const int x = t * kMuTile + gw * kMuRows + lane % kMuRows;
  return mla_slot_ptr<DQK, ESZ>(p, r, x < win ? x : x - win + kWinSlots, k_valid, win_valid);
}

// Gathers this warp's 8 rows of one tile; their pointers sit in lanes 8j .. of `ptrs`.  Returns the
// validity bits of its rows.
template <int ROWB>
__device__ inline uint32_t mla_umma_gather_rows(const mdc_sparse_mla_params& p, const unsigned char* ptrs, int j,
                                                unsigned char* stage, int gw, int lane) {
  constexpr int kFull = ROWB / 512, kTail = ROWB % 512 / 16;   // 512-byte pieces of a row, chunks behind them
  static_assert(kTail == 0 || kTail == 8, "the chunks behind the whole pieces are eight per row");
  const uint32_t bits = (__ballot_sync(0xffffffffu, ptrs != nullptr) >> (j * kMuRows)) & ((1u << kMuRows) - 1u);
  const unsigned long long mine = reinterpret_cast<unsigned long long>(ptrs);
  const unsigned char* pool = static_cast<const unsigned char*>(p.kv_cmp);
  auto put = [&](const unsigned char* src, int rr, int ch) {
    const int s = gw * kMuRows + rr;
    unsigned char* dst = stage + (ch >> 3) * (kMuTile * 128) + s * 128 + (((ch & 7) ^ (s & 7)) << 4);
    cp_async16_zfill(dst, (src ? src : pool) + ch * 16, src != nullptr);
  };
#pragma unroll
  for (int rr = 0; rr < kMuRows; ++rr) {
    const unsigned char* src = reinterpret_cast<const unsigned char*>(__shfl_sync(0xffffffffu, mine, j * kMuRows + rr));
#pragma unroll
    for (int k = 0; k < kFull; ++k) put(src, rr, k * 32 + lane);
  }
  if (kTail) {   // four rows per instruction
#pragma unroll
    for (int r0 = 0; r0 < kMuRows; r0 += 4) {
      const int rr = r0 + (lane >> 3);
      const unsigned char* src = reinterpret_cast<const unsigned char*>(__shfl_sync(0xffffffffu, mine, j * kMuRows + rr));
      put(src, rr, kFull * 32 + (lane & 7));
    }
  }
  cp_async_commit();
  return bits;
}

// r = b*q_len + t, hb = block of 128 heads, dq = block of 128 output columns,
// split / n_splits = slice of the slot range.  o_row / lse_row, when given,
// replace p.o / p.lse for this row (they point at the row's (H, d_v) block and
// (H,) vector, possibly in a peer GPU's memory); with to_row a split's partial goes there too
// instead of the split workspace.  All threads of the block call it.
// ALONE: the stand-alone kernel.
template <int DQK, bool FP8, bool ALONE>
__device__ __forceinline__ void mla_umma_tile(const mdc_sparse_mla_params& p, int r, int hb, int dq, int split, int n_splits,
                              unsigned char* smem, void* o_row = nullptr, float* lse_row = nullptr, bool to_row = false,
                              bool remote = false) {
  using SM = MlaUmmaSmem<DQK, FP8>;
  constexpr int S = SM::kStages, ESZ = FP8 ? 1 : 2, ROWB = SM::kRowBytes;
  constexpr uint32_t kQCols = ROWB / 4, kOCol = kQCols, kSCol = kOCol + kMuDv, kPCol = kSCol + kMuTile;
  static_assert(kPCol + kMuTile * ESZ / 4 <= 512, "tensor memory over-subscribed");
  static_assert(S >= 3 && SM::kPanels * kMuHeads * 128 <= (S - 1) * SM::kStageBytes,
                "two tiles are held while the next is gathered, and the staged query must fit the KV ring behind its first stage");
  constexpr long long kBudget = 1ll << 31, kDrain = 1ll << 24;   // clock cycles a role waits before it gives up, and after
  // Warps of a lane quadrant that move the query into tensor memory: the softmax warp and, stand-alone, two gather warps (3 rows x
  // 700 slots with window 16.6 -> 16.4 us, 32 x 2048 56.2 -> 55.7, e4m3 16 x 640 17.25 -> 17.1 on one box; on another the last two
  // are inside the spread.  Inside the persistent kernel the three of them gained nothing).
  constexpr int kMovers = ALONE ? 3 : 1;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  unsigned char* kst = smem + SM::kK;
  unsigned char* qst = kst + SM::kStageBytes;   // the query rows are staged in stages 1.. while tile 0 lands in stage 0
  uint64_t* full = reinterpret_cast<uint64_t*>(smem + SM::kBars);
  uint64_t* free_ = full + S;         // P V of the stage's tile has completed
  uint64_t* s_ready = free_ + S;
  uint64_t* s_taken = s_ready + 1;    // the softmax warps hold S in registers
  uint64_t* p_ready = s_taken + 1;
  uint64_t* q_ready = p_ready + 1;
  uint64_t* o_final = q_ready + 1;
  uint64_t* qs_ready = o_final + 1;  // the query rows are staged in shared memory
  uint32_t* misc = reinterpret_cast<uint32_t*>(smem + SM::kMisc);
  volatile uint32_t* abort_flag = misc + 1;
  unsigned char* validb = smem + SM::kValid;
  const float neg_inf = __int_as_float(0xff800000);
  const float c2 = p.softmax_scale * kLog2e;

  const int k_valid = min(max(p.k_valid[r], 0), kWinSlots + p.pt_cols * p.page_cmp);
  const int win_valid = p.win_valid ? min(max(p.win_valid[r], 0), kWinSlots) : 0;
  // Window slots in the tiles: the valid ones, no slots for the masked ones behind them.  e4m3 probabilities
  // keep the masked slots: which slots share a tile decides how they round.  (k_valid counts the window's 128 slots: a row
  // that ends before them has the window slots of its own tiles.)
  const int win = (win_valid > 0 && p.kv_win) ? min(FP8 ? kWinSlots : win_valid, ceil_div(k_valid, kMuTile) * kMuTile) : 0;
  const int n_tiles_all = ceil_div(win + max(k_valid - kWinSlots, 0), kMuTile);
  const int per = ceil_div(n_tiles_all, n_splits);
  const int t_begin = split * per;
  const int n_my = max(0, min(n_tiles_all, t_begin + per) - t_begin);

  __syncthreads();  // shared memory may be in use by the previous task of this block
  if (tid == 0) {
    for (int s = 0; s < S; ++s) {
      mbar_init(&full[s], kMuGatherWarps);
      mbar_init(&free_[s], 1);
    }
    mbar_init(s_ready, 1);
    mbar_init(s_taken, 4);
    mbar_init(p_ready, 4);
    mbar_init(q_ready, 4 * kMovers);
    mbar_init(o_final, 1);
    mbar_init(qs_ready, kMuGatherWarps);
    misc[1] = 0;
    mbar_fence_init();
  }
  if (warp == kMuIssueWarp) umma::tmem_alloc(misc, 512);
  umma::fence_before_sync();
  __syncthreads();
  umma::fence_after_sync();
  const uint32_t tmem = misc[0];
  auto give_up = [&](int what, int idx) {
    report_failure(p.status, MDC_DEV_COPY_TIMEOUT, 16 + what, idx, 0, 0);
    *abort_flag = 1;
  };
  // The lanes of a warp may have seen the last poll of a wait that ran out differently, and what follows takes whole warps.  So no
  // lane leaves its role alone: the issue warps vote on every wait, the others go on to the end (once the flag is set no
  // wait lasts) and write no result.

  // Query rows -> tensor memory (16 columns per store), from the copy the gather warps staged
  // in the (still empty) stages 1.. of the KV ring as panels of 128 rows x 128 bytes, 128-byte swizzle.  Mover
  // `m` of its lane quadrant (a warp's number % 4) takes every kMovers-th 16 columns.
  auto query_to_tmem = [&](int m) {
    if (!mbar_wait(qs_ready, 0, kBudget, abort_flag)) give_up(7, 0);
    const int row = (warp & 3) * 32 + lane;
    const uint32_t t_row = tmem + (static_cast<uint32_t>((warp & 3) * 32) << 16);
#pragma unroll 2
    for (int j = m; j < static_cast<int>(kQCols) / 16; j += kMovers) {
      uint32_t v[16];
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const int ch = 4 * j + u;
        const uint4 x = *reinterpret_cast<const uint4*>(qst + (ch >> 3) * (kMuHeads * 128) + row * 128 +
                                                        (((ch & 7) ^ (row & 7)) << 4));
        v[4 * u] = x.x; v[4 * u + 1] = x.y; v[4 * u + 2] = x.z; v[4 * u + 3] = x.w;
      }
      umma::tmem_st16(t_row + 16 * j, v);
    }
    umma::wait_st();
    umma::fence_before_sync();
    __syncwarp();
    mbar_arrive_if(q_ready, lane == 0);
  };

  if (warp < 4) {
    // ---------------- softmax warps: thread = head
    const int h = hb * kMuHeads + warp * 32 + lane;
    const uint32_t t_lane = tmem + (static_cast<uint32_t>(warp * 32) << 16);
    query_to_tmem(0);
    float m_used = neg_inf, l = 0.f;
    if (p.attn_sink && split == 0) {
      const float sk = p.attn_sink[h];
      if (sk != neg_inf) {
        m_used = sk;
        l = 1.f;
      }
    }
    bool ok = true;
    for (int i = 0; i < n_my; ++i) {
      if (!mbar_wait(s_ready, i & 1, kBudget, abort_flag)) {
        if (ok) give_up(0, i);
        ok = false;
      }
      umma::fence_after_sync();
      float sv[kMuTile];
      {
        float a[32], b[32];
        umma::tmem_ld32_f(t_lane + kSCol, a);
        umma::tmem_ld32_f(t_lane + kSCol + 32, b);
        umma::wait_ld();
#pragma unroll
        for (int j = 0; j < 32; ++j) {
          sv[j] = a[j];
          sv[32 + j] = b[j];
        }
      }
      const uint2 vb = *reinterpret_cast<const uint2*>(validb + (i % S) * 8);
      umma::fence_before_sync();
      __syncwarp();
      mbar_arrive_if(s_taken, lane == 0);
      // (one warp per scheduler: dependent chains are what costs here, so the maximum and the sum
      // run on four independent accumulators and a full tile skips the masking)
      if ((vb.x & vb.y) != 0xffffffffu) {
#pragma unroll
        for (int j = 0; j < kMuTile; ++j) {
          const bool valid = ((j < 32 ? vb.x >> j : vb.y >> (j - 32)) & 1u) != 0;
          sv[j] = valid ? sv[j] : neg_inf;
        }
      }
      float tm[4] = {neg_inf, neg_inf, neg_inf, neg_inf};
#pragma unroll
      for (int j = 0; j < kMuTile; j += 4) {
        tm[0] = fmaxf(tm[0], sv[j]);
        tm[1] = fmaxf(tm[1], sv[j + 1]);
        tm[2] = fmaxf(tm[2], sv[j + 2]);
        tm[3] = fmaxf(tm[3], sv[j + 3]);
      }
      const float tmax = fmaxf(fmaxf(tm[0], tm[1]), fmaxf(tm[2], tm[3]));
      // bf16 probabilities: the reference maximum moves only when the tile maximum exceeds it by more than 2^8.
      // e4m3 ones follow the running maximum: their rounding depends on it.
      const bool grow = tmax > m_used && (FP8 || m_used == neg_inf || (tmax - m_used) * c2 > 8.f);
      const float corr = !grow ? 1.f : (m_used == neg_inf) ? 0.f : exp2f((m_used - tmax) * c2);
      if (grow) m_used = tmax;
      uint32_t pk[kMuTile * ESZ / 4];
      float ps4[4] = {0.f, 0.f, 0.f, 0.f};
      {
        // p = 2^((s - m) * c2) as one fused multiply-add and one ex2.approx; a masked slot (-inf)
        // gives 0, and with m = -inf (nothing valid so far) the whole tile is 0
        const bool dead = m_used == neg_inf;
        const float off = dead ? 0.f : -m_used * c2;
        auto prob = [&](int j) { return dead ? 0.f : ex2_approx(fmaf(sv[j], c2, off)); };
        if constexpr (FP8) {
#pragma unroll
          for (int j = 0; j < kMuTile / 4; ++j) {
            float x[4] = {prob(4 * j), prob(4 * j + 1), prob(4 * j + 2), prob(4 * j + 3)};
            pk[j] = pack_e4m3x4(x);
            ps4[j & 3] += (x[0] + x[1]) + (x[2] + x[3]);
          }
        } else {
#pragma unroll
          for (int j = 0; j < kMuTile / 2; ++j) {
            const float p0 = prob(2 * j), p1 = prob(2 * j + 1);
            ps4[j & 3] += p0 + p1;
            pk[j] = pack_bf16x2(p0, p1);
          }
        }
      }
      l = l * corr + ((ps4[0] + ps4[1]) + (ps4[2] + ps4[3]));
      if (i > 0) {
        // P V of tile i - 1 has read P, and the accumulator holds the tiles up to it, once it has freed its stage
        if (!mbar_wait(&free_[(i - 1) % S], ((i - 1) / S) & 1, kBudget, abort_flag)) {
          if (ok) give_up(9, i);
          ok = false;
        }
        umma::fence_after_sync();
        if (__any_sync(0xffffffffu, grow)) {
#pragma unroll 1
          for (int cb = 0; cb < kMuDv / 32; ++cb) {
            uint32_t o[32];
            umma::tmem_ld32(t_lane + kOCol + 32 * cb, o);
            umma::wait_ld();
            uint32_t lo[16], hi[16];
#pragma unroll
            for (int j = 0; j < 16; ++j) {
              lo[j] = __float_as_uint(__uint_as_float(o[j]) * corr);
              hi[j] = __float_as_uint(__uint_as_float(o[16 + j]) * corr);
            }
            umma::tmem_st16(t_lane + kOCol + 32 * cb, lo);
            umma::tmem_st16(t_lane + kOCol + 32 * cb + 16, hi);
          }
        }
      }
#pragma unroll
      for (int c = 0; c < kMuTile * ESZ / 4; c += 16) {
        uint32_t v[16];
#pragma unroll
        for (int j = 0; j < 16; ++j) v[j] = pk[c + j];
        umma::tmem_st16(t_lane + kPCol + c, v);
      }
      umma::wait_st();
      umma::fence_before_sync();
      __syncwarp();
      mbar_arrive_if(p_ready, lane == 0);
    }
    if (n_my > 0 && !mbar_wait(o_final, 0, kBudget, abort_flag)) {
      if (ok) give_up(1, n_my);
      ok = false;
    }
    umma::fence_after_sync();
    if (__all_sync(0xffffffffu, ok)) {
      const bool live = l > 0.f;
      const float inv = live ? p.output_scale / l : 0.f;
      const float lse = live ? log2f(l) + c2 * m_used : neg_inf;
      const bool direct = n_splits == 1 || to_row;  // a split partial may also go to o_row / lse_row
      if (dq == 0) {
        if (direct) {
          if (lse_row) lse_row[h] = lse;
          else if (p.lse) p.lse[static_cast<int64_t>(r) * p.lse_stride + h] = lse;
        } else {
          p.ws_lse[(static_cast<int64_t>(r) * n_splits + split) * p.H + h] = lse;
        }
      }
      const int col0 = dq * kMuDv;
      // A bf16 row that goes to o_row (the owner's inbox) is staged in shared memory (the KV ring is idle now).  To a peer GPU
      // it leaves as ONE 256-byte bulk copy per head: sixteen 16-byte stores per thread over NVLink take an order of magnitude
      // longer.  On this GPU the warp stores its 32 rows, two per instruction (step of 1 x 4096 tokens 42.9 -> 41.7 us,
      // 8 x 131072 79.2 -> 78.1: the copies' completion had to be waited for before the notify).
      const bool stage_out = direct && o_row != nullptr && p.out_dtype != MDC_DT_F32;
      constexpr int kPitch = kMuDv * 2 + 16;   // (the 16 bytes keep a warp's stores off one bank)
      unsigned char* stage_row = kst + (warp * 32 + lane) * kPitch;
#pragma unroll 1
      for (int cb = 0; cb < kMuDv / 32; ++cb) {
        float o[32];
        if (n_my > 0) {
          umma::tmem_ld32_f(t_lane + kOCol + 32 * cb, o);
          umma::wait_ld();
        } else {
#pragma unroll
          for (int j = 0; j < 32; ++j) o[j] = 0.f;
        }
#pragma unroll
        for (int j = 0; j < 32; ++j) o[j] *= inv;
        const int col = col0 + 32 * cb;
        if (stage_out) {
          uint4* dst = reinterpret_cast<uint4*>(stage_row + 64 * cb);
#pragma unroll
          for (int j = 0; j < 4; ++j)
            dst[j] = make_uint4(pack_bf16x2(o[8 * j], o[8 * j + 1]), pack_bf16x2(o[8 * j + 2], o[8 * j + 3]),
                                pack_bf16x2(o[8 * j + 4], o[8 * j + 5]), pack_bf16x2(o[8 * j + 6], o[8 * j + 7]));
        } else if (!direct) {
          float4* dst = reinterpret_cast<float4*>(p.ws_o + ((static_cast<int64_t>(r) * n_splits + split) * p.H + h) * kMlaDv + col);
#pragma unroll
          for (int j = 0; j < 8; ++j) dst[j] = make_float4(o[4 * j], o[4 * j + 1], o[4 * j + 2], o[4 * j + 3]);
        } else if (p.out_dtype == MDC_DT_F32) {
          float* base = (o_row ? static_cast<float*>(o_row) : static_cast<float*>(p.o) + static_cast<int64_t>(r) * p.o_stride) +
                        static_cast<int64_t>(h) * kMlaDv + col;
          float4* dst = reinterpret_cast<float4*>(base);
#pragma unroll
          for (int j = 0; j < 8; ++j) dst[j] = make_float4(o[4 * j], o[4 * j + 1], o[4 * j + 2], o[4 * j + 3]);
        } else {
          __nv_bfloat16* base = (o_row ? static_cast<__nv_bfloat16*>(o_row)
                                       : static_cast<__nv_bfloat16*>(p.o) + static_cast<int64_t>(r) * p.o_stride) +
                                static_cast<int64_t>(h) * kMlaDv + col;
          uint4* dst = reinterpret_cast<uint4*>(base);
#pragma unroll
          for (int j = 0; j < 4; ++j)
            dst[j] = make_uint4(pack_bf16x2(o[8 * j], o[8 * j + 1]), pack_bf16x2(o[8 * j + 2], o[8 * j + 3]),
                                pack_bf16x2(o[8 * j + 4], o[8 * j + 5]), pack_bf16x2(o[8 * j + 6], o[8 * j + 7]));
        }
      }
      if (stage_out && !remote) {
        __syncwarp();
        unsigned char* to = static_cast<unsigned char*>(o_row) + (static_cast<int64_t>(h - lane) * kMlaDv + col0) * 2;
        const unsigned char* from = kst + warp * 32 * kPitch;
#pragma unroll 4
        for (int i = lane; i < 32 * (kMuDv / 8); i += 32) {   // row i / 16, 16 bytes each
          const int rr = i / (kMuDv / 8), ch = i % (kMuDv / 8);
          *reinterpret_cast<uint4*>(to + rr * (kMlaDv * 2) + ch * 16) = *reinterpret_cast<const uint4*>(from + rr * kPitch + ch * 16);
        }
      } else if (stage_out) {
        fence_proxy_async_smem();  // the copy engine reads the staged row through the async proxy
        bulk_s2g(static_cast<__nv_bfloat16*>(o_row) + static_cast<int64_t>(h) * kMlaDv + col0, stage_row, kMuDv * 2);
        bulk_commit();
        bulk_wait_all();           // the row has been written before this thread reaches the block's notify
        fence_proxy_async_global();
      }
    }
  } else if (warp >= kMuGatherWarp0 && warp < kMuGatherWarp0 + kMuGatherWarps) {
    // ---------------- gather warps: 8 rows of every tile each, up to two tiles in flight per warp
    const int gw = warp - kMuGatherWarp0;
    // Row pointers are looked up four tiles at a time and a batch ahead: a page-table read takes about as
    // long as a whole tile, and one tile of lead left it on the path (42 against 83 GB/s per SM in a copy of
    // this loop with 8 warps and rows that four blocks share).
    auto lookup = [&](int tile) {
      return mla_umma_row_ptrs<DQK, ESZ>(p, r, t_begin + tile, t_begin + n_my, win, k_valid, win_valid, gw, lane);
    };
    const unsigned char* cur = lookup(0);
    {  // stage the 128 query rows (coalesced: a warp instruction copies 512 contiguous bytes of a row)
      constexpr int kChunks = ROWB / 16;
      const unsigned char* q0 = static_cast<const unsigned char*>(p.q) +
                                (static_cast<int64_t>(r) * p.H + hb * kMuHeads) * ROWB;
#pragma unroll 4
      for (int rr = 0; rr < kMuHeads / kMuGatherWarps; ++rr) {
        const int row = gw * (kMuHeads / kMuGatherWarps) + rr;
#pragma unroll
        for (int ch = lane; ch < kChunks; ch += 32) {
          cp_async16_zfill(qst + (ch >> 3) * (kMuHeads * 128) + row * 128 + (((ch & 7) ^ (row & 7)) << 4),
                           q0 + static_cast<int64_t>(row) * ROWB + ch * 16, true);
        }
      }
      cp_async_commit();
    }
    const unsigned char* nxt = lookup(kMuBatch);
    int i0 = 0;
    if (n_my > 0) {  // tile 0 goes into stage 0 behind the query copies: its latency hides under the query's
      const uint32_t bits = mla_umma_gather_rows<ROWB>(p, cur, 0, kst, gw, lane);
      if (lane == 0) validb[gw] = static_cast<unsigned char>(bits);
      i0 = 1;
      cp_async_wait<1>();   // the query rows (the older group) have landed
    } else {
      cp_async_wait<0>();
    }
    {
      __syncwarp();
      mbar_arrive_if(qs_ready, lane == 0);
      if constexpr (ALONE) query_to_tmem(warp / 4);
      // stages 1.. are free for KV tiles once all of them have moved their share
      if (!mbar_wait(q_ready, 0, kBudget, abort_flag)) give_up(8, 0);
    }
    // Tiles [done, i) have been issued but not yet published.  A tile is published as soon as
    // its copies have landed -- never held back until the NEXT tile could be issued: when the
    // stage of the next tile is still in use, this warp first drains and publishes what it has
    // in flight (the tensor core is waiting for exactly that), then waits for the stage.
    int done = 0;
    auto publish = [&](int upto) {
      fence_proxy_async_smem();  // the tensor core reads the tiles through the async proxy
      __syncwarp();
      for (int t = done; t < upto; ++t) mbar_arrive_if(&full[t % S], lane == 0);
      done = upto;
    };
    if (i0 == 1) {  // tile 0 was issued before the query hand-over: it has had time to land, publish it now
      cp_async_wait<0>();
      publish(1);
    }
    for (int i = i0; i < n_my; ++i) {
      const int j = i % kMuBatch;   // tile i's place in the batch of row pointers
      if (j == 0) {
        cur = nxt;
        nxt = lookup(i + kMuBatch);
      }
      const int st = i % S;
      if (i >= S) {
        const uint32_t par = ((i / S) - 1) & 1;
        if (!__all_sync(0xffffffffu, mbar_test(&free_[st], par))) {
          if (done < i) {
            cp_async_wait<0>();
            publish(i);
          }
          if (!mbar_wait(&free_[st], par, kBudget, abort_flag)) give_up(2, i);
        }
      }
      const uint32_t bits = mla_umma_gather_rows<ROWB>(p, cur, j, kst + st * SM::kStageBytes, gw, lane);
      if (lane == 0) validb[st * 8 + gw] = static_cast<unsigned char>(bits);
      if (i - done >= 1) {  // at most two tiles in flight per warp
        cp_async_wait<1>();
        publish(i);
      }
    }
    cp_async_wait<0>();
    if (n_my > 0) publish(n_my);
  } else if (warp == kMuIssueWarp) {
    // ---------------- S = Q K^T of tile i, once it is gathered and the softmax warps have taken tile i - 1
    constexpr uint32_t idesc_qk = umma::idesc_mla(FP8, kMuHeads, kMuTile, false);
    const uint32_t kst_u = smem_u32(kst);
    bool ok = mbar_wait(q_ready, 0, kBudget, abort_flag);
    if (!ok) give_up(3, 0);
    for (int i = 0; i < n_my; ++i) {
      ok = ok && mbar_wait(&full[i % S], (i / S) & 1, kBudget, abort_flag) &&
           (i == 0 || mbar_wait(s_taken, (i - 1) & 1, kBudget, abort_flag));
      if (!__all_sync(0xffffffffu, ok)) {
        if (lane == 0) give_up(4, i);
        if (i > 0) mbar_wait(s_ready, (i - 1) & 1, kDrain);   // the last product (without the block's flag)
        break;
      }
      umma::fence_after_sync();
      if (umma::elect_one()) {
        const uint32_t base = kst_u + (i % S) * SM::kStageBytes;
#pragma unroll 4
        for (int k = 0; k < ROWB / 32; ++k) {
          const uint64_t bdesc = umma::smem_desc_sw128(base + (k >> 2) * (kMuTile * 128) + (k & 3) * 32);
          umma::mma_ts<FP8>(tmem + kSCol, tmem + 8 * k, bdesc, idesc_qk, k > 0);
        }
        umma::commit(s_ready);
      }
      __syncwarp();
    }
  } else if (warp == kMuPvWarp) {
    // ---------------- O (+)= P V of tile i: K steps of 32 bytes of probabilities, i.e. 32 / ESZ slots
    constexpr uint32_t idesc_pv = umma::idesc_mla(FP8, kMuHeads, kMuDv, true);
    const uint32_t v_u = smem_u32(kst) + (dq * kMuDv * ESZ / 128) * (kMuTile * 128);
    bool ok = true;
    for (int i = 0; i < n_my; ++i) {
      ok = __all_sync(0xffffffffu, mbar_wait(p_ready, i & 1, kBudget, abort_flag));
      if (!ok) {
        if (lane == 0) give_up(5, i);
        for (int j = max(0, i - S); j < i; ++j) mbar_wait(&free_[j % S], (j / S) & 1, kDrain);   // the last products
        break;
      }
      umma::fence_after_sync();
      if (umma::elect_one()) {
        const uint32_t base = v_u + (i % S) * SM::kStageBytes;
#pragma unroll
        for (int kk = 0; kk < kMuTile * ESZ / 32; ++kk) {
          const uint64_t bdesc = umma::smem_desc_mn_sw128(base + kk * (32 / ESZ) * 128, kMuTile * 128, 1024);
          umma::mma_ts<FP8>(tmem + kOCol, tmem + kPCol + 8 * kk, bdesc, idesc_pv, i > 0 || kk > 0);
        }
        umma::commit(&free_[i % S]);
        if (i == n_my - 1) umma::commit(o_final);
      }
      __syncwarp();
    }
    if (ok) {
      // The "free" arrivals of the last tiles have no consumer.  They are asynchronous: wait for
      // them here, or one could land after the barriers are invalidated below, on shared memory
      // that the block's next task already uses for something else.
      for (int i = max(0, n_my - S); i < n_my; ++i) {
        if (!mbar_wait(&free_[i % S], (i / S) & 1, kBudget)) {   // (also when another role has given up)
          give_up(6, i);
          break;
        }
      }
    }
  }

  umma::fence_before_sync();
  __syncthreads();
  umma::fence_after_sync();
  if (warp == kMuIssueWarp) umma::tmem_dealloc(tmem, 512);
  if (tid == 0) {
    for (int i = 0; i < SM::kNumBars; ++i) mbar_inval(full + i);
  }
}

}  // namespace mdc

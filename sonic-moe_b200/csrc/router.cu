// Fused routing front end: router GEMM (tokens x H x E on tcgen05, the accumulator row of a token never leaves the
// SM) -> logits rounded to bf16 and written out -> top-K and softmax over the K winners straight from the
// accumulator row -> per-expert token counts and the column sums of the full softmax (what the load-balancing loss
// needs), all in one pass over x.  The layer otherwise spends a library GEMM, a top-k kernel, a (T, E) fp32
// softmax and its column sum on the same 8 MiB of logits.
//
// One persistent CTA per SM, 128 tokens per tile, N = E (<= 256) accumulator columns:
//   warp 0      TMA producer: x tile 128 x 64 and router-weight tile E x 64 per stage (128-byte swizzle)
//   warp 1      MMA issuer: tcgen05.mma M 128 x N E x K 16 into one of two tensor-memory accumulators
//   warps 2-5   thread = token: the accumulator's row, rounded to bf16, goes to shared memory
//   warps 6-15  warp = token (finish_tokens): logits out, the K best, their softmax, the full softmax's column sums, which
//               a warp keeps for all its tokens; the warps' and then the CTAs' sums are added up in a fixed order, so the
//               column sums are bit-reproducible.
// With a thread per token that kept its K best in a sorted list, the 128 threads took 28 us a tile (E 128, K 8), more than its
// loads and multiplications, and nothing of it was hidden.  Event time of the two launches, before and now: T 24576, H 1536,
// E 128, K 8 77 -> 52 us, T 32768, H 4096, E 128, K 8 101 -> 83, T 65536, H 768, E 256, K 16 322 -> 122.  What is left depends on
// the layer: with K 1 in the place of K the first two take 37 of 44 us and 66 of 71 (launches in a row, inputs partly in the L2), so
// there it is the walk over H, loads and multiplications; the third takes 68 of 115, so there it is the search for 16 winners, by
// ten warps, beside a walk of 12 k-blocks a tile.
// The routing decision is taken on the bf16-rounded logits the kernel writes, so it can be checked bit for bit
// against a stable sort of that output.  Every wait is bounded (ptx.cuh).
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <math.h>
#include <stdint.h>

#include <mutex>
#include <type_traits>

#include "../../include/sonicmoe_b200.h"
#include "internal.h"
#include "launch.cuh"
#include "ptx.cuh"

namespace smoe {
namespace router {

constexpr int BM = 128;
constexpr int BK = 64;
constexpr int UMMA_K = 16;
constexpr int A_STAGE_BYTES = BM * BK * 2;  // 16 KiB
constexpr int MAX_E = kMaxRouterExperts;
constexpr int THREADS = 512;
constexpr int FIRST_DRAIN_WARP = 2;   // 4 warps, one per quarter of the tensor-memory lanes
constexpr int FIRST_TOKEN_WARP = 6;   // the large kernel's warps that work on tokens
constexpr int TOKEN_WARPS = THREADS / 32 - FIRST_TOKEN_WARP;
constexpr int MAX_STAGES = 16;

struct Shared {
  uint64_t full[MAX_STAGES];
  uint64_t empty[MAX_STAGES];
  uint64_t acc_full[2];
  uint64_t acc_empty[2];
  uint64_t rows_full, rows_empty;  // large kernel: the tile's rows in shared memory
  uint32_t tmem_base;
  int abort_flag;
  int hist[MAX_E];
};

struct Params {
  int T, H, E, K;
  int tile_rows, split;  // router_forward_small_kernel: tokens per tile, CTAs that share its experts
  int stages;
  int acc_cols;  // tensor-memory columns per accumulator (power of two >= E)
  __nv_bfloat16* logits;  // (T, E)
  float* scores;          // (T, K)
  int* indices;           // (T, K)
  float* colsum_partial;  // (grid, E)
  int* hist_partial;      // (grid, E)
  int* status;
};

__device__ __forceinline__ uint32_t order_key(float v) {  // larger key = better; NaN first, -0 == +0
  if (v != v) return 0xFFFFFFFFu;
  v = v + 0.0f;
  const uint32_t b = __float_as_uint(v);
  return (b & 0x80000000u) ? ~b : (b | 0x80000000u);
}

// Shared memory (offsets from its 1024-byte aligned start).  router_forward_kernel: tile_rows = BM, split = 1.  The warps'
// column sums take the stages' place once these are done with.
struct Layout {
  int stage, logits, pitch, shared, total;
  __host__ __device__ Layout(int tile_rows, int split, int E, int stages) {
    stage = (tile_rows + E / split) * BK * 2;  // E / split is a multiple of 16: 1024-byte aligned
    // the MMA reads 128 rows of A from the last stage on, whatever is behind its tile_rows
    logits = stages * stage + (BM - tile_rows) * BK * 2;
    pitch = 2 * E + 16;                        // bf16 rows; the pad spreads 16-byte writes of eight rows over the banks
    shared = logits + tile_rows / split * pitch;  // a multiple of 16
    total = 1024 + shared + static_cast<int>(sizeof(Shared));
  }
};

// value of a key whose upper half holds a bf16's order key
__device__ __forceinline__ float half_key_value(uint32_t k) {
  const uint32_t b = (k & 0x80000000u) ? (k & 0x7FFF0000u) : (~k & 0xFFFF0000u);
  return __uint_as_float(b);
}

// PER_LANE consecutive bf16 values, in the widest accesses that their alignment allows.
template <int PER_LANE>
struct LaneRow {
  using Word = std::conditional_t<PER_LANE % 4 == 0, uint2, std::conditional_t<PER_LANE % 2 == 0, uint32_t, uint16_t>>;
  static constexpr int WORDS = PER_LANE * 2 / static_cast<int>(sizeof(Word));
  union {
    Word words[WORDS];
    __nv_bfloat16_raw values[PER_LANE];
  };
};

// Tokens by one warp, from their bf16 logits in shared memory (`count` rows of `pitch` bytes, the first of them token
// `token0`): the warp takes first, first + step, ..., two at a time, because a token is a chain of warp-wide steps.  A lane
// holds PER_LANE = E / 32 neighbouring columns and sorts them; then the K best are K warp-wide maxima of the lanes' best
// (value, lower column first), each followed by one pop.  Adds the tokens' full softmax to colsum and counts the winners in
// hist.
template <int PER_LANE>
__device__ __forceinline__ void finish_tokens(const Params& p, const uint8_t* rows, int pitch, int token0, int count,
                                              int first, int step, int lane, float (&colsum)[PER_LANE], int* hist) {
  constexpr int N = 2, E = 32 * PER_LANE;
  for (int i = first; i < count; i += N * step) {
    bool valid[N];
    long long row[N];
    uint32_t key[N][PER_LANE];
    float f[N][PER_LANE];
#pragma unroll
    for (int n = 0; n < N; ++n) {
      valid[n] = i + n * step < count;
      const int at = valid[n] ? i + n * step : i;
      row[n] = token0 + at;
      LaneRow<PER_LANE> v;
      const auto* src = reinterpret_cast<const typename LaneRow<PER_LANE>::Word*>(rows + at * pitch + lane * PER_LANE * 2);
      auto* dst = reinterpret_cast<typename LaneRow<PER_LANE>::Word*>(p.logits + row[n] * E + lane * PER_LANE);
#pragma unroll
      for (int w = 0; w < LaneRow<PER_LANE>::WORDS; ++w) {
        v.words[w] = src[w];
        dst[w] = v.words[w];  // a token that the warp takes twice is written twice
      }
#pragma unroll
      for (int j = 0; j < PER_LANE; ++j) {
        f[n][j] = __bfloat162float(__nv_bfloat16(v.values[j]));
        // a bf16 value's order key is exact in its upper half; the lower half prefers the lower column
        key[n][j] = (order_key(f[n][j]) & 0xFFFF0000u) | static_cast<uint32_t>(0xFFFF - (lane * PER_LANE + j));
      }
      // odd-even transposition, largest first
#pragma unroll
      for (int r = 0; r < PER_LANE; ++r) {
#pragma unroll
        for (int j = r & 1; j + 1 < PER_LANE; j += 2) {
          const uint32_t a = max(key[n][j], key[n][j + 1]), b = min(key[n][j], key[n][j + 1]);
          key[n][j] = a;
          key[n][j + 1] = b;
        }
      }
    }
    // lane k keeps the k-th best
    uint32_t mine[N];
    float vmax[N];
#pragma unroll 1
    for (int k = 0; k < p.K; ++k) {
#pragma unroll
      for (int n = 0; n < N; ++n) {
        const uint32_t best = __reduce_max_sync(0xffffffffu, key[n][0]);
        if (k == 0) vmax[n] = half_key_value(best);
        if (k == 0 || lane == k) mine[n] = best;
        const bool pop = key[n][0] == best;
#pragma unroll
        for (int j = 0; j < PER_LANE; ++j) key[n][j] = pop ? (j + 1 < PER_LANE ? key[n][j + 1] : 0u) : key[n][j];
      }
    }
    // full softmax of the rows
    float s[N];
#pragma unroll
    for (int n = 0; n < N; ++n) {
      s[n] = 0.f;
#pragma unroll
      for (int j = 0; j < PER_LANE; ++j) {
        f[n][j] = __expf(f[n][j] - vmax[n]);
        s[n] += f[n][j];
      }
    }
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) {
#pragma unroll
      for (int n = 0; n < N; ++n) s[n] += __shfl_xor_sync(0xffffffffu, s[n], d);
    }
    float ex[N], sum[N];
#pragma unroll
    for (int n = 0; n < N; ++n) {
      const float inv_s = 1.f / s[n];
#pragma unroll
      for (int j = 0; j < PER_LANE; ++j)
        if (valid[n]) colsum[j] += f[n][j] * inv_s;
      ex[n] = lane < p.K ? expf(half_key_value(mine[n]) - vmax[n]) : 0.f;
      sum[n] = 0.f;
    }
#pragma unroll 4
    for (int k = 0; k < p.K; ++k) {
#pragma unroll
      for (int n = 0; n < N; ++n) sum[n] += __shfl_sync(0xffffffffu, ex[n], k);
    }
#pragma unroll
    for (int n = 0; n < N; ++n) {
      if (valid[n] && lane < p.K) {
        const int col = 0xFFFF - static_cast<int>(mine[n] & 0xFFFFu);
        p.scores[row[n] * p.K + lane] = ex[n] / sum[n];
        p.indices[row[n] * p.K + lane] = col;
        atomicAdd(&hist[col], 1);
      }
    }
  }
}

// The warps' column sums and the token counts as this CTA's partial results (by all threads).
template <int PER_LANE>
__device__ __forceinline__ void write_partials(const Params& p, float* sums, const float (&colsum)[PER_LANE], int warp,
                                               int lane, const int* hist) {
#pragma unroll
  for (int j = 0; j < PER_LANE; ++j) sums[warp * p.E + lane * PER_LANE + j] = colsum[j];
  __syncthreads();
  for (int col = threadIdx.x; col < p.E; col += THREADS) {
    float s = 0.f;
#pragma unroll
    for (int w = 0; w < THREADS / 32; ++w) s += sums[w * p.E + col];
    p.colsum_partial[static_cast<long long>(blockIdx.x) * p.E + col] = s;
    p.hist_partial[static_cast<long long>(blockIdx.x) * p.E + col] = hist[col];
  }
}

template <int PER_LANE>
__global__ void __launch_bounds__(THREADS, 1)
router_forward_kernel(const __grid_constant__ CUtensorMap tmX, const __grid_constant__ CUtensorMap tmW, const Params p) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  const Layout lay(BM, 1, p.E, p.stages);
  const int stage_bytes = lay.stage;
  Shared& ss = *reinterpret_cast<Shared*>(smem + lay.shared);
  const int warp = warp_index();
  const int lane = threadIdx.x & 31;
  volatile int* abort_flag = &ss.abort_flag;
  const int num_tiles = (p.T + BM - 1) / BM;
  const int num_kb = p.H / BK;

  if (threadIdx.x == 0) {
    for (int s = 0; s < p.stages; ++s) {
      mbar_init(smem_u32(&ss.full[s]), 1);
      mbar_init(smem_u32(&ss.empty[s]), 1);
    }
    for (int a = 0; a < 2; ++a) {
      mbar_init(smem_u32(&ss.acc_full[a]), 1);
      mbar_init(smem_u32(&ss.acc_empty[a]), 4);
    }
    mbar_init(smem_u32(&ss.rows_full), 4);
    mbar_init(smem_u32(&ss.rows_empty), TOKEN_WARPS);
    ss.abort_flag = 0;
    fence_mbar_init();
    tma_prefetch_desc(&tmX);
    tma_prefetch_desc(&tmW);
  }
  for (int e = threadIdx.x; e < MAX_E; e += THREADS) ss.hist[e] = 0;
  if (warp == 1) {
    tmem_alloc(smem_u32(&ss.tmem_base), 2 * p.acc_cols);
    tmem_relinquish();
  }
  wait_for_previous();
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = ss.tmem_base;
  float colsum[PER_LANE];
#pragma unroll
  for (int j = 0; j < PER_LANE; ++j) colsum[j] = 0.f;

  if (warp == 0) {
    // ---- TMA producer -------------------------------------------------------------------------------------
    if (elect_one()) {  // one thread, as in the MMA issuer: nothing in these loops is warp-wide
      int stage = 0;
      uint32_t phase = 0;
      bool ok = true;
      for (int tile = blockIdx.x; ok && tile < num_tiles; tile += gridDim.x) {
        for (int kb = 0; kb < num_kb; ++kb) {
          if (!mbar_wait(smem_u32(&ss.empty[stage]), phase ^ 1u, abort_flag)) { ok = false; break; }
          const uint32_t bar = smem_u32(&ss.full[stage]);
          const uint32_t a_dst = smem_u32(smem + stage * stage_bytes);
          mbar_arrive_expect_tx(bar, stage_bytes);
          tma_load_2d(&tmX, bar, a_dst, kb * BK, tile * BM);
          tma_load_2d(&tmW, bar, a_dst + A_STAGE_BYTES, kb * BK, 0);
          if (++stage == p.stages) { stage = 0; phase ^= 1u; }
        }
      }
      if (!ok && p.status) atomicCAS(p.status, SMOE_ST_OK, SMOE_ST_TIMEOUT_PRODUCER);
    }
  } else if (warp == 1) {
    // ---- MMA issuer ---------------------------------------------------------------------------------------
    if (elect_one()) {
      const uint32_t idesc = make_idesc_bf16(BM, p.E, false, false);
      int stage = 0;
      uint32_t phase = 0;
      int acc = 0;
      uint32_t acc_phase = 0;
      bool ok = true;
      for (int tile = blockIdx.x; ok && tile < num_tiles; tile += gridDim.x) {
        if (!mbar_wait(smem_u32(&ss.acc_empty[acc]), acc_phase ^ 1u, abort_flag)) { ok = false; break; }
        tc_fence_after();
        const uint32_t d_tmem = tmem_base + acc * p.acc_cols;
        for (int kb = 0; kb < num_kb; ++kb) {
          if (!mbar_wait(smem_u32(&ss.full[stage]), phase, abort_flag)) { ok = false; break; }
          tc_fence_after();
          const uint32_t a_addr = smem_u32(smem + stage * stage_bytes);
          const uint64_t a_desc = make_smem_desc(a_addr, 16, 1024);
          const uint64_t b_desc = make_smem_desc(a_addr + A_STAGE_BYTES, 16, 1024);
#pragma unroll
          for (int k4 = 0; k4 < BK / UMMA_K; ++k4)
            umma_bf16(d_tmem, a_desc + ((k4 * UMMA_K * 2) >> 4), b_desc + ((k4 * UMMA_K * 2) >> 4), idesc,
                      (kb > 0 || k4 > 0) ? 1u : 0u);
          umma_commit(smem_u32(&ss.empty[stage]));
          if (++stage == p.stages) { stage = 0; phase ^= 1u; }
        }
        if (!ok) break;
        umma_commit(smem_u32(&ss.acc_full[acc]));
        if (++acc == 2) { acc = 0; acc_phase ^= 1u; }
      }
      if (!ok && p.status) atomicCAS(p.status, SMOE_ST_OK, SMOE_ST_TIMEOUT_MMA);
    }
  } else if (warp < FIRST_TOKEN_WARP) {
    // ---- accumulator rows to shared memory: thread = token --------------------------------------------------
    const int quad = warp & 3;  // the 32 tensor-memory lanes this warp may read
    const uint32_t dst = smem_u32(smem + lay.logits + (quad * 32 + lane) * lay.pitch);
    int acc = 0;
    uint32_t acc_phase = 0, rows_phase = 0;
    bool ok = true;
    for (int tile = blockIdx.x; ok && tile < num_tiles; tile += gridDim.x) {
      if (!mbar_wait_warp(smem_u32(&ss.acc_full[acc]), acc_phase, abort_flag) ||
          !mbar_wait_warp(smem_u32(&ss.rows_empty), rows_phase ^ 1u, abort_flag)) {
        ok = false;
        break;
      }
      tc_fence_after();
      const uint32_t t_addr = tmem_base + acc * p.acc_cols + (static_cast<uint32_t>(quad * 32) << 16);
      for (int c = 0; c < p.E; c += 32) {
        uint32_t v[32];
        tmem_ld32(t_addr + c, v);
        tmem_ld_wait();
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          uint32_t w[4];
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            const __nv_bfloat162 h =
                __floats2bfloat162_rn(__uint_as_float(v[8 * q + 2 * j]), __uint_as_float(v[8 * q + 2 * j + 1]));
            w[j] = *reinterpret_cast<const uint32_t*>(&h);
          }
          st_shared_v4(dst + 2 * c + 16 * q, w[0], w[1], w[2], w[3]);
        }
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) {
        mbar_arrive(smem_u32(&ss.acc_empty[acc]));
        mbar_arrive(smem_u32(&ss.rows_full));
      }
      if (++acc == 2) { acc = 0; acc_phase ^= 1u; }
      rows_phase ^= 1u;
    }
    if (!ok && lane == 0 && p.status) atomicCAS(p.status, SMOE_ST_OK, SMOE_ST_TIMEOUT_EPILOGUE);
  } else {
    // ---- tokens: warp = token -------------------------------------------------------------------------------
    uint32_t rows_phase = 0;
    bool ok = true;
    for (int tile = blockIdx.x; ok && tile < num_tiles; tile += gridDim.x) {
      if (!mbar_wait_warp(smem_u32(&ss.rows_full), rows_phase, abort_flag)) { ok = false; break; }
      finish_tokens<PER_LANE>(p, smem + lay.logits, lay.pitch, tile * BM, min(BM, p.T - tile * BM), warp - FIRST_TOKEN_WARP,
                              TOKEN_WARPS, lane, colsum, ss.hist);
      __syncwarp();
      if (lane == 0) mbar_arrive(smem_u32(&ss.rows_empty));
      rows_phase ^= 1u;
    }
    if (!ok && lane == 0 && p.status) atomicCAS(p.status, SMOE_ST_OK, SMOE_ST_TIMEOUT_EPILOGUE);
  }

  if (*abort_flag != 0) {
    const uint64_t t0 = global_timer_ns();
    while (global_timer_ns() - t0 < 200000ull) __nanosleep(1000);
  }
  tc_fence_before();
  block_sync_diverged();
  __syncwarp();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base, 2 * p.acc_cols);
  }
  write_partials<PER_LANE>(p, reinterpret_cast<float*>(smem), colsum, warp, lane, ss.hist);
}

// Few tokens: smaller tiles, so that the chip is not left idle.  With one CTA per 128 tokens the walk over H is all of the time.
// Here a cluster of S CTAs takes R = 32, 64 or 128 tokens and CTA r multiplies them with its E / S experts over all of H: every
// logit is the same sum in the same order as in the kernel above, so the two agree bit for bit (a split of H would flip the
// rounding of a logit now and then, and with it near ties).  The rows, rounded to bf16, go to the CTAs that own the tokens (CTA
// d takes R / S of them) over distributed shared memory; then all 16 warps work on tokens (6 warps took 14 us for 64 tokens of
// 128 experts, more than their loads and multiplications).  What is left is the chain of H / 64 loads and multiplications, 180
// ns each.  Event time with the finishing kernel, before and now: T 1, H 2048, E 64 23.5 -> 15.4 us, T 64, H 4096, E 128 31.7 ->
// 21.5, T 1027, H 4096, E 256 39.7 -> 27.4, T 8192, H 4096, E 128 52 -> 38 (of which elect_one, the MMAs' issue: 8, 10, 12 and 8).
// The MMA has 128 rows whatever R is: rows from R on multiply whatever is in shared memory there, and are not read back.
template <int PER_LANE>
__global__ void __launch_bounds__(THREADS, 1)
router_forward_small_kernel(const __grid_constant__ CUtensorMap tmX, const __grid_constant__ CUtensorMap tmW,
                            const Params p) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  const Layout lay(p.tile_rows, p.split, p.E, p.stages);
  Shared& ss = *reinterpret_cast<Shared*>(smem + lay.shared);
  const int warp = warp_index();
  const int lane = threadIdx.x & 31;
  volatile int* abort_flag = &ss.abort_flag;
  const int rank = static_cast<int>(cluster_ctarank());
  const int tile = blockIdx.x / p.split;
  const int num_kb = p.H / BK;
  const int cols = p.E / p.split;           // experts of this CTA
  const int owned = p.tile_rows / p.split;  // tokens that each CTA of the cluster finishes

  if (threadIdx.x == 0) {
    for (int s = 0; s < p.stages; ++s) {
      mbar_init(smem_u32(&ss.full[s]), 1);
      mbar_init(smem_u32(&ss.empty[s]), 1);
    }
    mbar_init(smem_u32(&ss.acc_full[0]), 1);
    ss.abort_flag = 0;
    fence_mbar_init();
    tma_prefetch_desc(&tmX);
    tma_prefetch_desc(&tmW);
  }
  for (int e = threadIdx.x; e < MAX_E; e += THREADS) ss.hist[e] = 0;
  if (warp == 1) {
    tmem_alloc(smem_u32(&ss.tmem_base), p.acc_cols);
    tmem_relinquish();
  }
  wait_for_previous();
  tc_fence_before();
  __syncthreads();
  cluster_sync_all();  // every CTA of the cluster runs before anything is written to its shared memory
  tc_fence_after();
  const uint32_t tmem_base = ss.tmem_base;

  bool ok = true;
  if (warp == 0) {
    if (elect_one()) {
      int stage = 0;
      uint32_t phase = 0;
      for (int kb = 0; kb < num_kb; ++kb) {
        if (!mbar_wait(smem_u32(&ss.empty[stage]), phase ^ 1u, abort_flag)) { ok = false; break; }
        const uint32_t bar = smem_u32(&ss.full[stage]);
        const uint32_t a_dst = smem_u32(smem + stage * lay.stage);
        mbar_arrive_expect_tx(bar, lay.stage);
        tma_load_2d(&tmX, bar, a_dst, kb * BK, tile * p.tile_rows);
        tma_load_2d(&tmW, bar, a_dst + p.tile_rows * BK * 2, kb * BK, rank * cols);
        if (++stage == p.stages) { stage = 0; phase ^= 1u; }
      }
      if (!ok && p.status) atomicCAS(p.status, SMOE_ST_OK, SMOE_ST_TIMEOUT_PRODUCER);
    }
  } else if (warp == 1) {
    if (elect_one()) {
      const uint32_t idesc = make_idesc_bf16(BM, cols, false, false);
      int stage = 0;
      uint32_t phase = 0;
      for (int kb = 0; kb < num_kb; ++kb) {
        if (!mbar_wait(smem_u32(&ss.full[stage]), phase, abort_flag)) { ok = false; break; }
        tc_fence_after();
        const uint32_t a_addr = smem_u32(smem + stage * lay.stage);
        const uint64_t a_desc = make_smem_desc(a_addr, 16, 1024);
        const uint64_t b_desc = make_smem_desc(a_addr + p.tile_rows * BK * 2, 16, 1024);
#pragma unroll
        for (int k4 = 0; k4 < BK / UMMA_K; ++k4)
          umma_bf16(tmem_base, a_desc + ((k4 * UMMA_K * 2) >> 4), b_desc + ((k4 * UMMA_K * 2) >> 4), idesc,
                    (kb > 0 || k4 > 0) ? 1u : 0u);
        umma_commit(smem_u32(&ss.empty[stage]));
        if (++stage == p.stages) { stage = 0; phase ^= 1u; }
      }
      if (ok) umma_commit(smem_u32(&ss.acc_full[0]));
      else if (p.status) atomicCAS(p.status, SMOE_ST_OK, SMOE_ST_TIMEOUT_MMA);
    }
  } else if (warp < FIRST_TOKEN_WARP) {
    ok = mbar_wait_warp(smem_u32(&ss.acc_full[0]), 0, abort_flag);
    tc_fence_after();
    const int row = (warp & 3) * 32 + lane;
    if (!ok) {
      if (lane == 0 && p.status) atomicCAS(p.status, SMOE_ST_OK, SMOE_ST_TIMEOUT_EPILOGUE);
    } else if ((warp & 3) * 32 < p.tile_rows) {
      const uint32_t t_addr = tmem_base + (static_cast<uint32_t>((warp & 3) * 32) << 16);
      const uint32_t dst =
          map_to_cta(smem_u32(smem + lay.logits + (row % owned) * lay.pitch + rank * cols * 2), row / owned);
      for (int c = 0; c < cols; c += 16) {
        uint32_t v[16];
        tmem_ld16(t_addr + c, v);
        tmem_ld_wait();
        uint32_t w[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          const __nv_bfloat162 h = __floats2bfloat162_rn(__uint_as_float(v[2 * j]), __uint_as_float(v[2 * j + 1]));
          w[j] = *reinterpret_cast<const uint32_t*>(&h);
        }
        st_cluster_v4(dst + 2 * c, w[0], w[1], w[2], w[3]);
        st_cluster_v4(dst + 2 * c + 16, w[4], w[5], w[6], w[7]);
      }
      tc_fence_before();
    }
  }
  __syncwarp();
  if (*abort_flag != 0) {  // let this CTA's loads in flight land
    const uint64_t t0 = global_timer_ns();
    while (global_timer_ns() - t0 < 200000ull) __nanosleep(1000);
  }
  __syncwarp();
  cluster_sync_all();  // all rows of the owned tokens are here; after this no CTA touches another's shared memory
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base, p.acc_cols);
  }

  float colsum[PER_LANE];
#pragma unroll
  for (int j = 0; j < PER_LANE; ++j) colsum[j] = 0.f;
  const int token0 = tile * p.tile_rows + rank * owned;
  finish_tokens<PER_LANE>(p, smem + lay.logits, lay.pitch, token0, min(owned, p.T - token0), warp, THREADS / 32, lane, colsum,
                          ss.hist);
  write_partials<PER_LANE>(p, reinterpret_cast<float*>(smem), colsum, warp, lane, ss.hist);
}

// count[e] and colsum[e]: the CTAs' partials added up in a fixed order (each column by 1024 / 256 groups of threads, each
// over its share of the CTAs); without hist_partial, count is an input.  With `aux` also the load-balancing loss E <mean, share>, mean = colsum / sum(colsum) and
// share = count / sum(count) (denominators at least 1e-12), and its gradient by colsum, E (share - <mean, share>) /
// sum(colsum): two norms, divisions and a product over E values that took ten launches forward and fifteen backward.
__global__ void __launch_bounds__(1024) router_finish_kernel(const float* colsum_partial, const int* hist_partial,
                                                             int blocks, int E, float* colsum, int* count, float* aux,
                                                             float* aux_grad) {
  release_next();
  wait_for_previous();
  __shared__ float part_s[4][MAX_E];
  __shared__ int part_c[4][MAX_E];
  __shared__ float red[3][8];
  const int e = threadIdx.x & (MAX_E - 1), group = threadIdx.x / MAX_E;
  float s = 0.f;
  int c = 0;
  if (e < E) {
    const int begin = blocks * group / 4, end = blocks * (group + 1) / 4;
#pragma unroll 8
    for (int b = begin; b < end; ++b) {
      s += colsum_partial[static_cast<long long>(b) * E + e];
      if (hist_partial != nullptr) c += hist_partial[static_cast<long long>(b) * E + e];
    }
    if (hist_partial == nullptr && group == 0) c = count[e];
  }
  part_s[group][e] = s;
  part_c[group][e] = c;
  __syncthreads();
  s = ((part_s[0][e] + part_s[1][e]) + part_s[2][e]) + part_s[3][e];
  c = part_c[0][e] + part_c[1][e] + part_c[2][e] + part_c[3][e];
  if (group == 0 && e < E) {
    if (colsum != nullptr) colsum[e] = s;
    if (hist_partial != nullptr) count[e] = c;
  }
  if (aux == nullptr) return;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  float sums = fabsf(s), counts = static_cast<float>(c);
#pragma unroll
  for (int d = 16; d > 0; d >>= 1) {
    sums += __shfl_xor_sync(0xffffffffu, sums, d);
    counts += __shfl_xor_sync(0xffffffffu, counts, d);
  }
  if (group == 0 && lane == 0) {
    red[0][warp] = sums;
    red[1][warp] = counts;
  }
  __syncthreads();
  sums = counts = 0.f;
#pragma unroll
  for (int w = 0; w < MAX_E / 32; ++w) {
    sums += red[0][w];
    counts += red[1][w];
  }
  sums = fmaxf(sums, 1e-12f);
  const float share = static_cast<float>(c) / fmaxf(counts, 1e-12f);
  float dot = s / sums * share;
#pragma unroll
  for (int d = 16; d > 0; d >>= 1) dot += __shfl_xor_sync(0xffffffffu, dot, d);
  if (group == 0 && lane == 0) red[2][warp] = dot;
  __syncthreads();
  dot = 0.f;
#pragma unroll
  for (int w = 0; w < MAX_E / 32; ++w) dot += red[2][w];
  if (threadIdx.x == 0) *aux = static_cast<float>(E) * dot;
  if (group == 0 && e < E) aux_grad[e] = static_cast<float>(E) * (share - dot) / sums;
}

// Column sums of softmax(logits) for logits that another kernel made: one warp per row, partial sums per CTA.  The
// accurate exponential and division: the fast ones are off by |x| 2^-24 of a probability, which shows in the loss when the
// tokens go to experts of small probability.
template <int PER_LANE>
__global__ void __launch_bounds__(256) softmax_colsum_kernel(const __nv_bfloat16* logits, int rows, int E,
                                                             float* colsum_partial) {
  wait_for_previous();
  __shared__ float sums[8][MAX_E];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  float colsum[PER_LANE];
#pragma unroll
  for (int j = 0; j < PER_LANE; ++j) colsum[j] = 0.f;
  for (long long row = blockIdx.x * 8ll + warp; row < rows; row += gridDim.x * 8ll) {
    float l[PER_LANE], m = -INFINITY, s = 0.f;
#pragma unroll
    for (int j = 0; j < PER_LANE; ++j) {
      const int col = lane + 32 * j;
      l[j] = col < E ? __bfloat162float(logits[row * E + col]) : -INFINITY;
      m = fmaxf(m, l[j]);
    }
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, d));
#pragma unroll
    for (int j = 0; j < PER_LANE; ++j) {
      l[j] = lane + 32 * j < E ? expf(l[j] - m) : 0.f;
      s += l[j];
    }
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) s += __shfl_xor_sync(0xffffffffu, s, d);
#pragma unroll
    for (int j = 0; j < PER_LANE; ++j) colsum[j] += l[j] / s;
  }
#pragma unroll
  for (int j = 0; j < PER_LANE; ++j) sums[warp][lane + 32 * j] = colsum[j];
  __syncthreads();
  for (int col = threadIdx.x; col < E; col += 256) {
    float s = 0.f;
#pragma unroll
    for (int w = 0; w < 8; ++w) s += sums[w][col];
    colsum_partial[static_cast<long long>(blockIdx.x) * E + col] = s;
  }
}

// dlogits[t, e] = g_logits[t, e]                                      (optional)
//              + s_k (g_k - sum_j g_j s_j) for e = idx[t, k]           (gradient through the K winners' softmax)
//              + p[t, e] (c_e - sum_j p[t, j] c_j)                     (optional: gradient c of the column sums of
//                                                                       the full softmax p of the row);
//                                                                       c = g_colsum + *g_aux * aux_grad
// One warp per row; the row's probabilities are recomputed from the saved bf16 logits, with the exponential that the forward
// pass used: the fast one behind the router kernels, the accurate one (EXACT) behind softmax_colsum_kernel.
template <int PER_LANE, bool EXACT>
__global__ void __launch_bounds__(256) router_backward_kernel(__nv_bfloat16* dlogits, const __nv_bfloat16* logits,
                                                              const float* dscore, const float* score,
                                                              const int* indices, const float* g_colsum,
                                                              const __nv_bfloat16* g_logits, const float* g_aux,
                                                              const float* aux_grad, int rows, int E, int K) {
  release_next();
  wait_for_previous();
  const int lane = threadIdx.x & 31;
  const long long row = static_cast<long long>(blockIdx.x) * (blockDim.x >> 5) + (threadIdx.x >> 5);
  if (row >= rows) return;
  float out[PER_LANE];
#pragma unroll
  for (int j = 0; j < PER_LANE; ++j) {
    const int col = lane + 32 * j;
    out[j] = (g_logits != nullptr && col < E) ? __bfloat162float(g_logits[row * E + col]) : 0.f;
  }
  if (g_colsum != nullptr || g_aux != nullptr) {
    float l[PER_LANE], c[PER_LANE];
    float m = -INFINITY;
    const float scale = g_aux != nullptr ? *g_aux : 0.f;
#pragma unroll
    for (int j = 0; j < PER_LANE; ++j) {
      const int col = lane + 32 * j;
      c[j] = (g_colsum != nullptr && col < E) ? g_colsum[col] : 0.f;
      if (g_aux != nullptr && col < E) c[j] += scale * aux_grad[col];
      l[j] = col < E ? __bfloat162float(logits[row * E + col]) : -INFINITY;
      m = fmaxf(m, l[j]);
    }
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, d));
    float s = 0.f, dot = 0.f;
#pragma unroll
    for (int j = 0; j < PER_LANE; ++j) {
      const int col = lane + 32 * j;
      l[j] = col < E ? (EXACT ? expf(l[j] - m) : __expf(l[j] - m)) : 0.f;
      s += l[j];
      dot += l[j] * c[j];
    }
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) {
      s += __shfl_xor_sync(0xffffffffu, s, d);
      dot += __shfl_xor_sync(0xffffffffu, dot, d);
    }
    const float inv = 1.f / s;
    dot *= inv;
#pragma unroll
    for (int j = 0; j < PER_LANE; ++j) {
      const int col = lane + 32 * j;
      if (col < E) out[j] += l[j] * inv * (c[j] - dot);
    }
  }
  if (dscore != nullptr) {
    float dot = 0.f;
    for (int k = lane; k < K; k += 32) dot += dscore[row * K + k] * score[row * K + k];
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) dot += __shfl_xor_sync(0xffffffffu, dot, d);
    for (int k = 0; k < K; ++k) {  // every lane walks the K winners; the owner of the column adds the term
      const int col = indices[row * K + k];
      const float term = score[row * K + k] * (dscore[row * K + k] - dot);
#pragma unroll
      for (int j = 0; j < PER_LANE; ++j)
        if (col == lane + 32 * j) out[j] += term;
    }
  }
#pragma unroll
  for (int j = 0; j < PER_LANE; ++j) {
    const int col = lane + 32 * j;
    if (col < E) dlogits[row * E + col] = __float2bfloat16_rn(out[j]);
  }
}

using EncodeTiledFn = CUresult (*)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                   const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                   CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

static EncodeTiledFn encode_fn() {
  static EncodeTiledFn fn = nullptr;
  static std::once_flag once;
  std::call_once(once, [] {
    void* ptr = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &ptr, cudaEnableDefault, &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      fn = reinterpret_cast<EncodeTiledFn>(ptr);
  });
  return fn;
}

static int encode_rows(CUtensorMap* map, const void* base, uint64_t rows, uint64_t cols, uint32_t box_rows) {
  EncodeTiledFn fn = encode_fn();
  if (fn == nullptr) return SMOE_ERR_DRIVER;
  static thread_local bool context_bound = false;
  if (!context_bound) {
    if (cudaFree(nullptr) != cudaSuccess) return SMOE_ERR_DRIVER;
    context_bound = true;
  }
  if ((reinterpret_cast<uintptr_t>(base) & 15u) != 0) return SMOE_ERR_ALIGNMENT;
  const cuuint64_t dims[2] = {cols, rows};
  const cuuint64_t strides[1] = {cols * 2};
  const cuuint32_t box[2] = {BK, box_rows};
  const cuuint32_t estr[2] = {1, 1};
  const CUresult r = fn(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(base), dims, strides, box, estr,
                        CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                        CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS ? SMOE_OK : SMOE_ERR_TENSORMAP;
}

// Tile of router_forward_small_kernel: what a CTA loads per k-block is (rows + E / split) lines, so the smallest such tile
// whose CTAs all fit on the chip at once; one with the large kernel's 128 rows and all experts means that kernel (from
// 9473 tokens on at 148 SMs, where tiles of half its traffic would take a second wave).  At that line, H 4096, E 128, K 8:
// 9400 tokens 40 us by small tiles, 9600 by large ones 48.
static void small_tile(int T, int E, int sms, int& rows, int& split) {
  rows = BM;
  split = 1;
  int best = BM + E;
  for (int r = 32; r <= BM; r *= 2) {
    for (int s = 1; s <= 8 && s <= r; s *= 2) {
      if (E % (16 * s) != 0 || (T + r - 1) / r * s > sms) continue;
      if (r + E / s < best) {
        best = r + E / s;
        rows = r;
        split = s;
      }
    }
  }
}

static bool unsupported(int T, int H, int E, int K) {
  return T < 0 || H <= 0 || (H % BK) != 0 || E < 32 || E > MAX_E || (E % 32) != 0 || K <= 0 || K > 16 || K > E;
}

}  // namespace router
}  // namespace smoe

using namespace smoe;
using namespace smoe::router;

extern "C" {

int smoe_router_forward_supported(int H, int E, int K) { return unsupported(1, H, E, K) ? 0 : 1; }

size_t smoe_router_forward_workspace_bytes(int E) {
  const int sms = num_sms();
  return static_cast<size_t>(sms > 0 ? sms : 256) * static_cast<size_t>(E > 0 ? E : 1) * 8;
}

int smoe_router_forward(const void* x, const void* router_w, void* logits, float* scores, int* indices,
                        int* expert_count, float* prob_colsum, void* workspace, int T, int H, int E, int K,
                        int* status, void* stream) {
  return smoe_router_forward_aux(x, router_w, logits, scores, indices, expert_count, prob_colsum, nullptr, nullptr,
                                 workspace, T, H, E, K, status, stream);
}

int smoe_router_forward_aux(const void* x, const void* router_w, void* logits, float* scores, int* indices,
                            int* expert_count, float* prob_colsum, float* aux, float* aux_grad, void* workspace, int T,
                            int H, int E, int K, int* status, void* stream) {
  if ((aux == nullptr) != (aux_grad == nullptr)) return SMOE_ERR_SHAPE;
  if (unsupported(T, H, E, K)) return SMOE_ERR_SHAPE;
  if (workspace == nullptr) return SMOE_ERR_WORKSPACE;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const int sms = num_sms();
  if (sms <= 0) return SMOE_ERR_DRIVER;
  const int tiles = (T + BM - 1) / BM;
  int grid = tiles < sms ? tiles : sms;
  float* colsum_partial = static_cast<float*>(workspace);
  int* hist_partial = reinterpret_cast<int*>(colsum_partial + static_cast<size_t>(sms) * E);
  if (T > 0) {
    Params p = {};
    p.T = T; p.H = H; p.E = E; p.K = K;
    small_tile(T, E, sms, p.tile_rows, p.split);
    const bool small = p.tile_rows < BM || p.split > 1;
    CUtensorMap tmX, tmW;
    int rc = encode_rows(&tmX, x, T, H, p.tile_rows);
    if (rc != SMOE_OK) return rc;
    rc = encode_rows(&tmW, router_w, E, H, E / p.split);
    if (rc != SMOE_OK) return rc;
    const int cols = E / p.split;
    // as many stages as fit, and no more than 128 KiB where the tiles are small
    const int stage = Layout(p.tile_rows, p.split, E, 0).stage;
    p.stages = ((small ? 128 : 226) * 1024 - (small ? 0 : Layout(p.tile_rows, p.split, E, 0).total)) / stage;
    p.stages = p.stages > MAX_STAGES ? MAX_STAGES : p.stages;
    p.acc_cols = cols <= 32 ? 32 : cols <= 64 ? 64 : cols <= 128 ? 128 : 256;
    p.logits = static_cast<__nv_bfloat16*>(logits);
    p.scores = scores; p.indices = indices;
    p.colsum_partial = colsum_partial; p.hist_partial = hist_partial;
    p.status = status;
    const int dev = current_device();
    if (dev < 0) return SMOE_ERR_DRIVER;
    using Kernel = void (*)(CUtensorMap, CUtensorMap, Params);
    static constexpr Kernel kernels[2][8] = {
        {router_forward_kernel<1>, router_forward_kernel<2>, router_forward_kernel<3>, router_forward_kernel<4>,
         router_forward_kernel<5>, router_forward_kernel<6>, router_forward_kernel<7>, router_forward_kernel<8>},
        {router_forward_small_kernel<1>, router_forward_small_kernel<2>, router_forward_small_kernel<3>,
         router_forward_small_kernel<4>, router_forward_small_kernel<5>, router_forward_small_kernel<6>,
         router_forward_small_kernel<7>, router_forward_small_kernel<8>}};
    static PerDeviceFlag configured[2][8];
    const int per_lane = E / 32;
    const Kernel kernel = kernels[small][per_lane - 1];
    if (!configured[small][per_lane - 1].test(dev)) {
      if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024) != cudaSuccess)
        return SMOE_ERR_LAUNCH;
      configured[small][per_lane - 1].set(dev);
    }
    if (small) grid = (T + p.tile_rows - 1) / p.tile_rows * p.split;
    launch_chained(kernel, grid, THREADS, Layout(p.tile_rows, p.split, E, p.stages).total, st, p.split, tmX, tmW, p);
    if (cudaGetLastError() != cudaSuccess) return SMOE_ERR_LAUNCH;
  }
  launch_chained(router_finish_kernel, 1, 1024, 0, st, 1, colsum_partial, hist_partial,
                 T > 0 ? grid : 0, E, prob_colsum, expert_count, aux, aux_grad);
  return launch_rc(T > 0 ? 2 : 1);
}

int smoe_switch_loss(const void* logits, const int* expert_count, float* aux, float* aux_grad, void* workspace, int T,
                     int E, void* stream) {
  if (T < 0 || E <= 0 || E > MAX_E) return SMOE_ERR_SHAPE;
  if (workspace == nullptr) return SMOE_ERR_WORKSPACE;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const int sms = num_sms();
  if (sms <= 0) return SMOE_ERR_DRIVER;
  const int blocks = T == 0 ? 0 : (T + 7) / 8 < sms ? (T + 7) / 8 : sms;
  float* colsum_partial = static_cast<float*>(workspace);
  const __nv_bfloat16* l = static_cast<const __nv_bfloat16*>(logits);
  if (blocks > 0) {
    const int per_lane = (E + 31) / 32;
    if (per_lane <= 1)
      launch_chained(softmax_colsum_kernel<1>, blocks, 256, 0, st, 1, l, T, E, colsum_partial);
    else if (per_lane <= 4)
      launch_chained(softmax_colsum_kernel<4>, blocks, 256, 0, st, 1, l, T, E, colsum_partial);
    else
      launch_chained(softmax_colsum_kernel<8>, blocks, 256, 0, st, 1, l, T, E, colsum_partial);
    if (cudaGetLastError() != cudaSuccess) return SMOE_ERR_LAUNCH;
  }
  launch_chained(router_finish_kernel, 1, 1024, 0, st, 1, colsum_partial, nullptr, blocks, E, nullptr,
                 const_cast<int*>(expert_count), aux, aux_grad);
  return launch_rc(blocks > 0 ? 2 : 1);
}

int smoe_router_backward(void* dlogits, const void* logits, const float* dscores, const float* scores,
                         const int* indices, const float* g_colsum, const void* g_logits, int T, int E, int K,
                         void* stream) {
  return smoe_router_backward_aux(dlogits, logits, dscores, scores, indices, g_colsum, g_logits, nullptr, nullptr, T, E,
                                  K, stream);
}

int smoe_router_backward_aux(void* dlogits, const void* logits, const float* dscores, const float* scores,
                             const int* indices, const float* g_colsum, const void* g_logits, const float* g_aux,
                             const float* aux_grad, int T, int E, int K, void* stream) {
  if (T < 0 || E <= 0 || E > MAX_E || K <= 0 || K > E) return SMOE_ERR_SHAPE;
  if (g_aux != nullptr && (aux_grad == nullptr || (T > 0 && logits == nullptr))) return SMOE_ERR_SHAPE;
  if (dscores != nullptr && (scores == nullptr || indices == nullptr)) return SMOE_ERR_SHAPE;
  if (g_colsum != nullptr && logits == nullptr) return SMOE_ERR_SHAPE;
  if (T == 0) return SMOE_OK;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const unsigned grid = (T + 7) / 8;
  __nv_bfloat16* d = static_cast<__nv_bfloat16*>(dlogits);
  const __nv_bfloat16* l = static_cast<const __nv_bfloat16*>(logits);
  const __nv_bfloat16* g = static_cast<const __nv_bfloat16*>(g_logits);
  // the gradient of smoe_switch_loss alone
  const bool exact = dscores == nullptr && g_colsum == nullptr && g_logits == nullptr;
  const int per_lane = (E + 31) / 32;
  const auto kernel = per_lane <= 2   ? (exact ? router_backward_kernel<2, true> : router_backward_kernel<2, false>)
                      : per_lane <= 4 ? (exact ? router_backward_kernel<4, true> : router_backward_kernel<4, false>)
                                      : (exact ? router_backward_kernel<8, true> : router_backward_kernel<8, false>);
  launch_chained(kernel, grid, 256, 0, st, 1, d, l, dscores, scores, indices, g_colsum, g, g_aux, aux_grad, T, E, K);
  return launch_rc();
}

}  // extern "C"

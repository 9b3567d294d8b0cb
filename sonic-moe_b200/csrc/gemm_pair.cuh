// Grouped GEMM on CTA pairs: a cluster of two CTAs (one SM pair) computes a 256 x 256 output tile with
// tcgen05.mma.cta_group::2.  Each CTA stages its own 128 rows of A and its own 128 of the tile's 256 B rows,
// so a stage costs 32 KiB of shared-memory fill per CTA instead of 48 KiB and six stages fit; the
// accumulator (this CTA's 128 rows x all 256 columns, fp32) lives in the CTA's own tensor memory, two
// of them so the epilogue of one tile overlaps the main loop of the next.
//
// DUAL mode (kernels with a gathered operand): one work unit is two tiles that share the gathered operand's
// stage -- 256 x 512 (DUAL_N: two B tiles) or 512 x 256 (DUAL_M: two A tiles) -- one per accumulator.  A stage
// is then 48 KiB (gathered tile + two plain tiles), four stages deep, and every gathered row feeds twice the
// MMA work, which is what bounds these kernels (row gathers are many small TMA operations); the price is that
// the two accumulators no longer alternate between consecutive units.
//
// Roles per CTA (warp index):
//   0        TMA producer for the operands that are not gathered (both CTAs; completion bytes are counted
//            on the leader CTA's "full" barrier)
//   1        leader CTA: MMA issuer.  other CTA: idle
//   2..      8 epilogue warps (each 32 rows x 128 columns)
//   10..     GW gather warps (0, 4 or 8): the routed rows of the gathered operand by TMA tile::gather4, issued by one
//            thread of each
//
// Barriers.  full[s]: leader only; one arrival (the leader's expect_tx), tx = TMA bytes of both CTAs,
// gathered rows included.  empty[s], acc_full[a]: per CTA, signalled by the leader's multicast
// tcgen05.commit.  acc_empty[a]: leader only, one arrival per epilogue warp of both CTAs.  Every wait is
// bounded (ptx.cuh).
#pragma once
#include "epilogue.cuh"
#include "launch.cuh"
#include "ptx.cuh"

namespace smoe {
namespace pair {

constexpr int BM = 128;          // rows per CTA (TMEM lanes); the pair's tile has 2 * BM rows
constexpr int BN = 256;          // tile columns = accumulator columns
constexpr int BN_CTA = 128;      // B rows each CTA stages
constexpr int BK = 64;
constexpr int STAGES = 6;
constexpr int UMMA_K = 16;
constexpr int A_STAGE_BYTES = BM * BK * 2;       // 16 KiB
constexpr int B_STAGE_BYTES = BN_CTA * BK * 2;   // 16 KiB
constexpr int CHUNK_BYTES = BK * 128;            // 64-element MN chunk: BK rows x 128 B
constexpr int MAX_EXPERTS = 1024;
constexpr int EPI_WARPS = 8;

// Kernels whose epilogue warps need more than 128 registers (a whole accumulator piece held by each thread, or z of two
// chunks beside the activation's arithmetic) move registers to them with setmaxnreg.  That is a warpgroup-wide
// instruction, so these keep warps 2 and 3 idle: warps 0-3 producer / MMA, 4-11 epilogue, 12-15 gather.
__host__ __device__ constexpr bool splits_registers(int epi, int dual) {
  return dual != 0 || epi_base(epi) == EPI_DSWIGLU || epi_base(epi) == EPI_DACT || epi_base(epi) == EPI_ACT;
}
__host__ __device__ constexpr int threads(int gather_warps, bool split) {
  return 32 * ((split ? 4 : 2) + EPI_WARPS + gather_warps);
}

struct SharedStorage {
  uint64_t full[STAGES];
  uint64_t empty[STAGES];
  uint64_t acc_full[2];
  uint64_t acc_empty[2];
  uint32_t tmem_base;
  int abort_flag;
  int off[MAX_EXPERTS + 1];            // first grouped row of every expert
  int m_tile_prefix[MAX_EXPERTS + 1];  // ragged-M: exclusive prefix of the experts' row tiles; ragged-K: counts
  int expert_order[MAX_EXPERTS];       // ragged-K with a skewed load: experts by descending count
  int most_rows;                       // ragged-K: the largest count
};

// Output staging of the epilogues: each epilogue warp has 32 rows of 64 bytes (epilogue.cuh), through which a tile leaves
// in whole 64-byte row segments: 8 requests to L2 per store instruction instead of 32 (with one row per lane the epilogue
// sent about as many requests to L2 as the main loop's operand fetches and competed with them).
constexpr int STAGE_OUT_BYTES = EPI_WARPS * STAGE_ROWS_BYTES;
constexpr int SMEM_BYTES =
    1024 + STAGES * (A_STAGE_BYTES + B_STAGE_BYTES) + ((sizeof(SharedStorage) + 127) & ~127) + STAGE_OUT_BYTES;
static_assert(SMEM_BYTES <= 227 * 1024, "shared memory per CTA");

struct Tile {
  int e;
  int row0;     // ragged-M: first grouped row of THIS CTA's 128 rows; ragged-K: first output row of this CTA
  int row_end;  // ragged-M: off[e+1]; ragged-K: M
  int n0;       // first column of the pair's 256-column tile
  int k_begin, k_end;
  int num_kb;
};

enum { DUAL_NONE = 0, DUAL_N = 1, DUAL_M = 2 };

// Ragged-K: whether one expert has more than twice the mean number of rows.  Ordering is quadratic in the experts, so it
// stops at 512 (1 us per 128).
__device__ __forceinline__ bool is_skewed(const GemmParams& p, const SharedStorage& ss) {
  return p.E <= 512 && static_cast<long long>(ss.most_rows) * p.E > 2ll * p.total_rows;
}

// Ragged-K: fills expert_order if the load is skewed (ties: lower expert first).  Called by the whole block; most_rows was
// zeroed before an earlier barrier, and the arrays are complete after the caller's next one.
__device__ __forceinline__ void order_experts(const GemmParams& p, SharedStorage& ss) {
  int* count = ss.m_tile_prefix;
  for (int e = threadIdx.x; e < p.E; e += blockDim.x) {
    count[e] = p.off[e + 1] - p.off[e];
    atomicMax(&ss.most_rows, count[e]);
  }
  __syncthreads();
  if (!is_skewed(p, ss)) return;
  for (int e = threadIdx.x; e < p.E; e += blockDim.x) {
    const int mine = count[e];
    int rank = 0;
#pragma unroll 8
    for (int f = 0; f < p.E; ++f) {
      const int c = count[f];
      rank += (c > mine || (c == mine && f < e)) ? 1 : 0;
    }
    ss.expert_order[rank] = e;
  }
}

// The work units of one cluster, in the order in which every role of its CTAs walks them.  Each warp keeps its own
// walker; all lanes must call next().  All state is in registers and shared memory: with 64-bit divisions, a binary
// search and two dependent global loads per unit, finding a unit took longer than the MMAs of a short reduction.
// Units go expert by expert, row tiles outermost, and are dealt out round-robin.
// Ragged-K with a skewed load: a unit is as long as its expert's token count, so the experts go in descending order of
// their counts and every other round is dealt out in reverse, which evens out the clusters' sums: at 65536 tokens, top-4 of
// 64 experts, loads falling with the square of the rank, the longest cluster has 1379 k-blocks (dW2) where the mean is
// 1336 and plain round-robin gave 2356; dW2 1342 -> 922 us, dW1 1642 -> 1199 us (alternating; the eight-warp epilogue is in
// it).  Even loads keep the plain order, which is 3 % faster there (dW1 of the 128-expert benchmark layer 3560 against
// 3666 us): the line is a largest count of twice the mean, below which round-robin is at most one such unit off.
template <bool RAGGED_K, int DUAL>
struct UnitWalker {
  static constexpr int UNIT_N = DUAL == DUAL_N ? 2 * BN : BN;
  static constexpr int UNIT_M = DUAL == DUAL_M ? 4 * BM : 2 * BM;
  const GemmParams& p;
  const SharedStorage& ss;
  const int cluster, clusters, lane, num_n;
  int total;         // units of the whole grid
  int per_expert;    // ragged-K: units per expert
  bool skewed;       // ragged-K: dealt out by descending count
  int round = 0;
  int mi, ni, e = 0;  // ragged-M: row tile, unit along N and expert of the next unit
  int step_m, step_n;

  __device__ __forceinline__ UnitWalker(const GemmParams& p_, const SharedStorage& ss_, int lane_)
      : p(p_), ss(ss_), cluster(blockIdx.x >> 1), clusters(gridDim.x >> 1), lane(lane_),
        num_n((p_.N + UNIT_N - 1) / UNIT_N) {
    if constexpr (RAGGED_K) {
      per_expert = (p.M + UNIT_M - 1) / UNIT_M * num_n;
      total = per_expert * p.E;
      skewed = is_skewed(p, ss);
    } else {
      total = ss.m_tile_prefix[p.E] * num_n;
      mi = cluster / num_n;
      ni = cluster % num_n;
      step_m = clusters / num_n;
      step_n = clusters % num_n;
    }
  }
  __device__ __forceinline__ int unit_of_round() const {
    return round * clusters + (RAGGED_K && skewed && (round & 1) ? clusters - 1 - cluster : cluster);
  }
  // Number of k-blocks of the next unit, or -1 when there is none (all that the MMA issuer wants to know).
  __device__ __forceinline__ int next_num_kb() {
    const int t = unit_of_round();
    if (t >= total) return -1;
    ++round;
    if constexpr (!RAGGED_K) {
      return p.K / BK;
    } else {
      const int i = t / per_expert, ex = skewed ? ss.expert_order[i] : i;
      return (ss.off[ex + 1] - ss.off[ex] + BK - 1) / BK;
    }
  }
  __device__ __forceinline__ bool next(uint32_t rank, Tile& tile) {
    const int t = unit_of_round();
    if (t >= total) return false;
    ++round;
    if constexpr (!RAGGED_K) {
      while (true) {  // the first expert whose tiles end beyond mi, 32 experts at a time
        const int i = e + 1 + lane;
        const unsigned before = __ballot_sync(0xffffffffu, i <= p.E && ss.m_tile_prefix[i] <= mi);
        e += __popc(before);
        if (before != 0xffffffffu) break;
      }
      tile.e = e;
      tile.row0 = ss.off[e] + (mi - ss.m_tile_prefix[e]) * (2 * BM) + static_cast<int>(rank) * BM;
      tile.row_end = ss.off[e + 1];
      tile.n0 = ni * UNIT_N;
      tile.k_begin = 0;
      tile.k_end = p.K;
      tile.num_kb = p.K / BK;
      mi += step_m;
      ni += step_n;
      if (ni >= num_n) {
        ni -= num_n;
        ++mi;
      }
    } else {
      const int i = t / per_expert, rem = t - i * per_expert, m = rem / num_n;
      tile.e = skewed ? ss.expert_order[i] : i;
      tile.row0 = m * UNIT_M + static_cast<int>(rank) * BM;
      tile.row_end = p.M;
      tile.n0 = (rem - m * num_n) * UNIT_N;
      tile.k_begin = ss.off[tile.e];
      tile.k_end = ss.off[tile.e + 1];
      tile.num_kb = (tile.k_end - tile.k_begin + BK - 1) / BK;
    }
    return true;
  }
};

// An MN-major operand tile of one stage: 64-column chunks of BK rows.
__device__ __forceinline__ void load_mn_tile(const CUtensorMap* tm, uint32_t bar, uint32_t dst, int col, int row) {
#pragma unroll
  for (int c = 0; c < BM / 64; ++c) tma_load_2d_pair(tm, bar, dst + c * CHUNK_BYTES, col + 64 * c, row);
}

template <bool RAGGED_K, bool A_GATHER, bool A_MN, bool B_GATHER, bool B_MN, int EPI_CODE, int GW,
          int DUAL = DUAL_NONE>
__global__ void __launch_bounds__(threads(GW, splits_registers(EPI_CODE, DUAL)), 1)
grouped_gemm_pair_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB,
                         const GemmParams p) {
  constexpr int EPI = epi_base(EPI_CODE);
  constexpr int ACT = EPI_CODE / 16;  // general epilogues: the Activation
  // DUAL: four stages of three 16 KiB tiles (A, B and the second plain tile X) instead of six stages of two
  constexpr int NSTAGES = DUAL != DUAL_NONE ? 4 : STAGES;
  constexpr int X_STAGE_BYTES = DUAL != DUAL_NONE ? A_STAGE_BYTES : 0;
  static_assert(DUAL != DUAL_N || !B_GATHER, "DUAL_N doubles the plain B tile");
  static_assert(DUAL != DUAL_M || (!A_GATHER && A_MN && RAGGED_K), "DUAL_M doubles the plain MN-major A tile of a ragged-K kernel");
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* sA = smem;
  uint8_t* sB = smem + NSTAGES * A_STAGE_BYTES;
  uint8_t* sX = sB + NSTAGES * B_STAGE_BYTES;
  SharedStorage& ss = *reinterpret_cast<SharedStorage*>(smem + NSTAGES * (A_STAGE_BYTES + B_STAGE_BYTES + X_STAGE_BYTES));
  uint8_t* stage_out = reinterpret_cast<uint8_t*>(&ss) + ((sizeof(SharedStorage) + 127) & ~127);

  const int warp = warp_index();
  const int lane = threadIdx.x & 31;
  const uint32_t rank = cluster_ctarank();  // 0 = leader
  const bool leader = rank == 0;
  volatile int* abort_flag = &ss.abort_flag;

  constexpr bool kGather = A_GATHER || B_GATHER;
  static_assert(!(A_GATHER && B_GATHER), "at most one operand is gathered");
  static_assert(!kGather || GW > 0, "a gathered operand needs gather warps");
  static_assert(GW == 0 || GW == 4 || GW == 8, "0, 4 or 8 gather warps");
  constexpr bool SPLIT_REGS = splits_registers(EPI, DUAL);
  constexpr int FIRST_EPI_WARP = SPLIT_REGS ? 4 : 2;
  constexpr int FIRST_GATHER_WARP = FIRST_EPI_WARP + EPI_WARPS;
  static_assert(!SPLIT_REGS || GW == 4, "4 gather warps (512 threads)");
  constexpr uint32_t kTmaBytesPerCta = A_STAGE_BYTES + B_STAGE_BYTES + X_STAGE_BYTES;  // gathered rows included

  // ---- set-up -------------------------------------------------------------------------------
  if (threadIdx.x == 0) {
    for (int s = 0; s < NSTAGES; ++s) {
      mbar_init(smem_u32(&ss.full[s]), 1);
      mbar_init(smem_u32(&ss.empty[s]), 1);
    }
    for (int a = 0; a < 2; ++a) {
      mbar_init(smem_u32(&ss.acc_full[a]), 1);
      mbar_init(smem_u32(&ss.acc_empty[a]), 2 * EPI_WARPS);
    }
    ss.abort_flag = 0;
    fence_mbar_init();
  }
  if (warp == 0 && lane == 0) {
    tma_prefetch_desc(&tmA);
    tma_prefetch_desc(&tmB);
  }
  if (warp == 1) {
    tmem_alloc(smem_u32(&ss.tmem_base), 2 * BN);  // all 512 columns: both CTAs get the same base
    tmem_relinquish();
  }
  wait_for_previous();
  for (int e = threadIdx.x; e <= p.E; e += blockDim.x) ss.off[e] = p.off[e];
  if constexpr (RAGGED_K) {
    if (threadIdx.x == 0) ss.most_rows = 0;
    __syncthreads();
    order_experts(p, ss);
  } else {
    if (warp == 2) {
      const int min_rows = p.min_rows > 0 && !tiles_take_all(p, p.min_rows, lane) ? p.min_rows : 0;
      int running = 0;
      for (int base = 0; base < p.E; base += 32) {
        const int e = base + lane;
        int v = 0;
        if (e < p.E) {
          const int rows = p.off[e + 1] - p.off[e];
          v = rows > min_rows ? (rows + 2 * BM - 1) / (2 * BM) : 0;
        }
        int incl = v;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
          const int o = __shfl_up_sync(0xffffffffu, incl, d);
          if (lane >= d) incl += o;
        }
        if (e < p.E) ss.m_tile_prefix[e] = running + incl - v;
        running += __shfl_sync(0xffffffffu, incl, 31);
      }
      if (lane == 0) ss.m_tile_prefix[p.E] = running;
    }
  }
  tc_fence_before();
  __syncthreads();
  cluster_sync_all();  // the other CTA's barriers are initialised before anything can arrive on them
  tc_fence_after();
  const uint32_t tmem_base = ss.tmem_base;

  // SPLIT_REGS: registers move to the epilogue warps from the other roles
  // (512 threads x 128 registers at launch; two warpgroups give up 72 registers per thread, two take 72).  Each
  // role branch starts with its own setmaxnreg so that the register limit is known along the whole branch.
  if (warp < FIRST_EPI_WARP) {
  if constexpr (SPLIT_REGS) asm volatile("setmaxnreg.dec.sync.aligned.u32 56;");
  // ---- TMA producer -------------------------------------------------------------------------
  if (warp == 0) {
    if constexpr (kTmaBytesPerCta > 0) {
      const bool elected = elect_one();
      int stage = 0;
      uint32_t phase = 0;
      bool ok = true;
      Tile tile;
      UnitWalker<RAGGED_K, DUAL> walk(p, ss, lane);
      while (ok && walk.next(rank, tile)) {
        for (int kb = 0; kb < tile.num_kb; ++kb) {
          if (!mbar_wait_warp(smem_u32(&ss.empty[stage]), phase ^ 1u, abort_flag)) { ok = false; break; }
          const uint32_t bar = map_to_cta(smem_u32(&ss.full[stage]), 0);  // the leader's barrier
          const uint32_t a_dst = smem_u32(sA + stage * A_STAGE_BYTES);
          const uint32_t b_dst = smem_u32(sB + stage * B_STAGE_BYTES);
          [[maybe_unused]] const uint32_t x_dst = smem_u32(sX + stage * X_STAGE_BYTES);
          if (elected) {
            if (leader) mbar_arrive_expect_tx(smem_u32(&ss.full[stage]), 2 * kTmaBytesPerCta);
            const int k0 = RAGGED_K ? (tile.k_begin + kb * BK) : kb * BK;
            if constexpr (!A_GATHER && !A_MN) {
              // no rows at all in this CTA's half of the tile: read past the tensor's end, which delivers zeros
              tma_load_2d_pair(&tmA, bar, a_dst, k0, tile.row0 < tile.row_end ? tile.row0 : p.total_rows);
            }
            if constexpr (!A_GATHER && A_MN) load_mn_tile(&tmA, bar, a_dst, tile.row0, k0);
            if constexpr (!B_GATHER) {
              const int nb = tile.n0 + static_cast<int>(rank) * BN_CTA;  // this CTA's half of the B rows
              const int krow = RAGGED_K ? k0 : (tile.e * p.b_rows_per_expert + k0);
              if constexpr (!B_MN) tma_load_2d_pair(&tmB, bar, b_dst, k0, tile.e * p.b_rows_per_expert + nb);
              else load_mn_tile(&tmB, bar, b_dst, nb, krow);
              if constexpr (DUAL == DUAL_N) {  // the unit's second B tile: columns n0 + 256 ...
                if constexpr (!B_MN) tma_load_2d_pair(&tmB, bar, x_dst, k0, tile.e * p.b_rows_per_expert + nb + BN);
                else load_mn_tile(&tmB, bar, x_dst, nb + BN, krow);
              }
            }
            // the unit's second A tile: rows row0 + 256 ...
            if constexpr (DUAL == DUAL_M) load_mn_tile(&tmA, bar, x_dst, tile.row0 + 2 * BM, k0);
          }
          __syncwarp();
          if (++stage == NSTAGES) { stage = 0; phase ^= 1u; }
        }
      }
      if (!ok && lane == 0 && p.status) atomicCAS(p.status, ST_OK, ST_TIMEOUT_PRODUCER);
    }
  }
  // ---- MMA issuer (leader) / gather relay (other CTA) ----------------------------------------
  else if (warp == 1) {
    if (leader && elect_one()) {  // one thread: nothing in this loop is warp-wide
      constexpr uint32_t idesc = make_idesc_bf16(2 * BM, BN, A_MN, B_MN);
      constexpr uint32_t a_lbo = A_MN ? CHUNK_BYTES : 16;
      constexpr uint32_t b_lbo = B_MN ? CHUNK_BYTES : 16;
      constexpr uint32_t a_kstep = A_MN ? (UMMA_K * 128) : (UMMA_K * 2);
      constexpr uint32_t b_kstep = B_MN ? (UMMA_K * 128) : (UMMA_K * 2);
      int stage = 0;
      uint32_t phase = 0;
      int acc = 0;
      uint32_t acc_phase = 0;
      bool ok = true;
      UnitWalker<RAGGED_K, DUAL> walk(p, ss, lane);
      for (int num_kb = walk.next_num_kb(); ok && num_kb >= 0; num_kb = walk.next_num_kb()) {
        if (num_kb == 0) continue;
        if constexpr (DUAL == DUAL_NONE) {
          if (!mbar_wait(smem_u32(&ss.acc_empty[acc]), acc_phase ^ 1u, abort_flag)) { ok = false; break; }
        } else {
          // both accumulators belong to this unit; the first group may start as soon as the epilogue has copied the
          // previous unit's first accumulator out, the second group waits for the second one (below)
          if (!mbar_wait(smem_u32(&ss.acc_empty[0]), acc_phase ^ 1u, abort_flag)) { ok = false; break; }
        }
        tc_fence_after();
        const uint32_t d_tmem = tmem_base + (DUAL == DUAL_NONE ? acc * BN : 0);
        for (int kb = 0; kb < num_kb; ++kb) {
          if (!mbar_wait(smem_u32(&ss.full[stage]), phase, abort_flag)) { ok = false; break; }
          tc_fence_after();
          const uint64_t a_desc = make_smem_desc(smem_u32(sA + stage * A_STAGE_BYTES), a_lbo, 1024);
          const uint64_t b_desc = make_smem_desc(smem_u32(sB + stage * B_STAGE_BYTES), b_lbo, 1024);
#pragma unroll
          for (int k4 = 0; k4 < BK / UMMA_K; ++k4) {
            umma_bf16_pair(d_tmem, a_desc + ((k4 * a_kstep) >> 4), b_desc + ((k4 * b_kstep) >> 4), idesc,
                           (kb > 0 || k4 > 0) ? 1u : 0u);
          }
          if constexpr (DUAL != DUAL_NONE) {
            if (kb == 0) {  // the second accumulator of the previous unit has been copied out
              if (!mbar_wait(smem_u32(&ss.acc_empty[1]), acc_phase ^ 1u, abort_flag)) { ok = false; break; }
              tc_fence_after();
            }
          }
          if constexpr (DUAL == DUAL_N) {
            const uint64_t x_desc = make_smem_desc(smem_u32(sX + stage * X_STAGE_BYTES), b_lbo, 1024);
#pragma unroll
            for (int k4 = 0; k4 < BK / UMMA_K; ++k4) {
              umma_bf16_pair(d_tmem + BN, a_desc + ((k4 * a_kstep) >> 4), x_desc + ((k4 * b_kstep) >> 4), idesc,
                             (kb > 0 || k4 > 0) ? 1u : 0u);
            }
          }
          if constexpr (DUAL == DUAL_M) {
            const uint64_t x_desc = make_smem_desc(smem_u32(sX + stage * X_STAGE_BYTES), a_lbo, 1024);
#pragma unroll
            for (int k4 = 0; k4 < BK / UMMA_K; ++k4) {
              umma_bf16_pair(d_tmem + BN, x_desc + ((k4 * a_kstep) >> 4), b_desc + ((k4 * b_kstep) >> 4), idesc,
                             (kb > 0 || k4 > 0) ? 1u : 0u);
            }
          }
          umma_commit_pair(smem_u32(&ss.empty[stage]), 3);  // frees the stage in both CTAs
          if (++stage == NSTAGES) { stage = 0; phase ^= 1u; }
        }
        if (!ok) break;
        if constexpr (DUAL == DUAL_NONE) {
          umma_commit_pair(smem_u32(&ss.acc_full[acc]), 3);
          if (++acc == 2) { acc = 0; acc_phase ^= 1u; }
        } else {
          umma_commit_pair(smem_u32(&ss.acc_full[0]), 3);
          umma_commit_pair(smem_u32(&ss.acc_full[1]), 3);
          acc_phase ^= 1u;
        }
      }
      if (!ok && p.status) atomicCAS(p.status, ST_OK, ST_TIMEOUT_MMA);
    }
  }
  }  // warps below FIRST_EPI_WARP (SPLIT_REGS: warps 2 and 3 idle)
  // ---- gather producers ----------------------------------------------------------------------
  else if (warp >= FIRST_GATHER_WARP) {
    if constexpr (SPLIT_REGS) asm volatile("setmaxnreg.dec.sync.aligned.u32 56;");
    if constexpr (kGather) {
      // One thread of each gather warp issues its share of a stage's 32 gather4 operations (4 rows x 128 B each).  With eight
      // issuing threads a warp the compiler's loop over active lanes (elect_one) took about 75 cycles an operation, which
      // with eight of them a stage is more than the 512 cycles of a single tile's MMAs: a training step of T 24576, H 1536, I 256,
      // E 128, K 8 2051 -> 2013 us (alternating, repeated runs within 0.4 %; in power-capped steps no more than their spread).
      constexpr int OPS = 32 / GW;
      const int gw = warp - FIRST_GATHER_WARP;
      const bool elected = elect_one();
      const CUtensorMap* tm = A_GATHER ? &tmA : &tmB;
      uint8_t* stage_base = A_GATHER ? sA : sB;
      constexpr int STAGE_BYTES = A_GATHER ? A_STAGE_BYTES : B_STAGE_BYTES;
      int stage = 0;
      uint32_t phase = 0;
      bool ok = true;
      Tile tile;
      UnitWalker<RAGGED_K, DUAL> walk(p, ss, lane);
      while (ok && walk.next(rank, tile)) {
        if constexpr (!RAGGED_K) {
          // lane l fetches the index of the warp's row l; then every lane has them all, for the whole unit
          const int r = tile.row0 + 4 * OPS * gw + lane;
          const int mine = lane < 4 * OPS && r < tile.row_end ? p.gather[r] : p.gather_rows;  // rows that do not exist: zeros
          // (they cost no traffic and next to no power; multiplying other rows in their place took 2.5 % longer where a
          // fifth of the tiles' rows do not exist, up projection of 512 rows per expert 980 -> 959 us)
          int rows[4 * OPS];
#pragma unroll
          for (int i = 0; i < 4 * OPS; ++i) rows[i] = __shfl_sync(0xffffffffu, mine, i);
          if (elected) {
            for (int kb = 0; kb < tile.num_kb; ++kb) {
              if (!mbar_wait(smem_u32(&ss.empty[stage]), phase ^ 1u, abort_flag)) { ok = false; break; }
              const uint32_t bar = map_to_cta(smem_u32(&ss.full[stage]), 0);
              const uint32_t dst = smem_u32(stage_base + stage * STAGE_BYTES) + gw * OPS * 512;
#pragma unroll
              for (int q = 0; q < OPS; ++q)
                tma_gather4_pair(tm, bar, dst + q * 512, kb * BK, rows[4 * q], rows[4 * q + 1], rows[4 * q + 2],
                                 rows[4 * q + 3]);
              if (++stage == NSTAGES) { stage = 0; phase ^= 1u; }
            }
          }
          ok = __all_sync(0xffffffffu, ok);
        } else {
          // 2 chunks of 64 columns x 16 groups of 4 tokens; a warp has OPS / 2 groups of both chunks.  Lane l fetches the
          // index of its warp's token l, two k-blocks ahead.
          constexpr int TOKENS = 2 * OPS;
          const int col0 = A_GATHER ? tile.row0 : tile.n0 + static_cast<int>(rank) * BN_CTA;
          const auto load_idx = [&](int kb) {
            const int tok = tile.k_begin + kb * BK + TOKENS * gw + lane;
            return lane < TOKENS && kb < tile.num_kb && tok < tile.k_end ? p.gather[tok] : p.gather_rows;  // beyond: zeros
          };
          int cur = load_idx(0), nxt = load_idx(1);
          for (int kb = 0; kb < tile.num_kb; ++kb) {
            if (!mbar_wait_warp(smem_u32(&ss.empty[stage]), phase ^ 1u, abort_flag)) { ok = false; break; }
            int tokens[TOKENS];
#pragma unroll
            for (int i = 0; i < TOKENS; ++i) tokens[i] = __shfl_sync(0xffffffffu, cur, i);
            if (elected) {
              const uint32_t bar = map_to_cta(smem_u32(&ss.full[stage]), 0);
              const uint32_t dst = smem_u32(stage_base + stage * STAGE_BYTES) + gw * (OPS / 2) * 512;
#pragma unroll
              for (int q = 0; q < OPS; ++q) {
                const int g = q % (OPS / 2), chunk = q / (OPS / 2);
                tma_gather4_pair(tm, bar, dst + chunk * CHUNK_BYTES + g * 512, col0 + 64 * chunk, tokens[4 * g],
                                 tokens[4 * g + 1], tokens[4 * g + 2], tokens[4 * g + 3]);
              }
            }
            __syncwarp();
            cur = nxt;
            nxt = load_idx(kb + 2);
            if (++stage == NSTAGES) { stage = 0; phase ^= 1u; }
          }
        }
      }
      if (!ok && lane == 0 && p.status) atomicCAS(p.status, ST_OK, ST_TIMEOUT_PRODUCER);
    }
  }
  // ---- epilogue -----------------------------------------------------------------------------
  else {
    if constexpr (SPLIT_REGS) asm volatile("setmaxnreg.inc.sync.aligned.u32 200;");
    const int quad = warp & 3;
    constexpr int COLS_PER_WARP = BN * 4 / EPI_WARPS;
    const int col_half = (warp - FIRST_EPI_WARP) >> 2;
    const int row_in_tile = quad * 32 + lane;
    int acc = 0;
    uint32_t acc_phase = 0;
    bool ok = true;
    Tile tile;
    UnitWalker<RAGGED_K, DUAL> walk(p, ss, lane);
    while (ok && walk.next(rank, tile)) {
      const bool have_acc = tile.num_kb > 0;
      constexpr int SUBTILES = DUAL == DUAL_NONE ? 1 : 2;
      if constexpr (DUAL != DUAL_NONE && EPI == EPI_STORE) {
        // Plain stores: both accumulators are copied out, rounded to bf16 (two values per register, 64 registers
        // per accumulator) and handed back before anything is stored, so the next unit's MMAs wait for two
        // tensor-memory reads and not for this unit's stores.
        constexpr int CHUNKS = COLS_PER_WARP / 32;  // 4
        static_assert(COLS_PER_WARP == 128, "dual tiles use 8 epilogue warps");
        uint32_t packed[2][CHUNKS * 16];
#pragma unroll
        for (int sub = 0; sub < 2; ++sub) {
          if (have_acc) {
            if (!mbar_wait_warp(smem_u32(&ss.acc_full[sub]), acc_phase, abort_flag)) { ok = false; break; }
            tc_fence_after();
            const uint32_t t_addr = tmem_base + sub * BN + (static_cast<uint32_t>(quad * 32) << 16);
#pragma unroll
            for (int h = 0; h < CHUNKS / 2; ++h) {
              uint32_t v0[32], v1[32];
              tmem_ld32(t_addr + (col_half * CHUNKS + 2 * h) * 32, v0);
              tmem_ld32(t_addr + (col_half * CHUNKS + 2 * h + 1) * 32, v1);
              tmem_ld_wait();
              if (h == CHUNKS / 2 - 1) {  // last read of this accumulator: give it back before converting
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive_cluster_relaxed(map_to_cta(smem_u32(&ss.acc_empty[sub]), 0));
              }
#pragma unroll
              for (int j = 0; j < 16; ++j) {
                packed[sub][(2 * h) * 16 + j] = pack_bf16(__uint_as_float(v0[2 * j]), __uint_as_float(v0[2 * j + 1]));
                packed[sub][(2 * h + 1) * 16 + j] = pack_bf16(__uint_as_float(v1[2 * j]), __uint_as_float(v1[2 * j + 1]));
              }
            }
          } else {
#pragma unroll
            for (int j = 0; j < CHUNKS * 16; ++j) packed[sub][j] = 0u;
          }
        }
        if (!ok) break;
        {
          // stores: 64-byte row segments through this warp's staging rows (8 rows per store instruction)
          const uint32_t my_stage = smem_u32(stage_out) + (warp - FIRST_EPI_WARP) * STAGE_ROWS_BYTES;
#pragma unroll
          for (int sub = 0; sub < 2; ++sub) {
            const int row_base = tile.row0 + (DUAL == DUAL_M ? sub * 2 * BM : 0) + quad * 32;
            const int n0 = tile.n0 + (DUAL == DUAL_N ? sub * BN : 0);
            __nv_bfloat16* out = p.out0 + (RAGGED_K ? tile.e * p.out0_expert_stride : 0ll);
#pragma unroll
            for (int c = 0; c < CHUNKS; ++c) {
              const int n = n0 + (col_half * CHUNKS + c) * 32;
              if (n >= p.N) break;
              uint32_t w[16];
#pragma unroll
              for (int j = 0; j < 16; ++j) w[j] = packed[sub][c * 16 + j];
              warp_store_rows64(my_stage, lane, w, out, p.ld0, row_base, tile.row_end, n, p.accumulate);
            }
          }
        }
        if (have_acc) acc_phase ^= 1u;
        continue;
      }
#pragma unroll 1
      for (int sub = 0; sub < SUBTILES && ok; ++sub) {
        if constexpr (DUAL != DUAL_NONE) acc = sub;
        const int r = tile.row0 + (DUAL == DUAL_M ? sub * 2 * BM : 0) + row_in_tile;
        const int n0 = tile.n0 + (DUAL == DUAL_N ? sub * BN : 0);
        const bool row_ok = r < tile.row_end;
        float score = 0.f;
        if constexpr (EPI == EPI_DSWIGLU || EPI == EPI_DACT || EPI == EPI_SCATTER || EPI == EPI_STORE_ROWS) {
          if (row_ok && (EPI != EPI_STORE_ROWS || p.scores != nullptr))
            score = load_score(p.scores, p.scores_are_bf16, p.s_scatter[r]);
        }
        const auto wait_acc = [&] {
          if (have_acc) {
            if (!mbar_wait_warp(smem_u32(&ss.acc_full[acc]), acc_phase, abort_flag)) return false;
            tc_fence_after();
          }
          return true;
        };
        // Hands the accumulator back as soon as the last of it is in registers.  Relaxed: what has to be ordered before
        // it, the tensor-memory reads, is (tcgen05.wait::ld and the fence); a release would also wait for the tile's
        // global stores, 1800 to 2500 cycles of the 6000 that a plain-store tile took.
        const auto release_acc = [&] {
          if (have_acc) {
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive_cluster_relaxed(map_to_cta(smem_u32(&ss.acc_empty[acc]), 0));
          }
        };
        if constexpr (EPI != EPI_DSWIGLU && EPI != EPI_DACT) {  // those wait once their first loads are in flight
          if (!wait_acc()) { ok = false; break; }
        }
        float ds_acc = 0.f;
        const uint32_t t_addr = tmem_base + acc * BN + (static_cast<uint32_t>(quad * 32) << 16);
        if constexpr (DUAL != DUAL_NONE) {
          // Copy this warp's columns of the accumulator into registers and hand the accumulator back at once: the
          // next unit's MMAs need both accumulators, so the epilogue arithmetic and stores must not hold them.
          static_assert(EPI == EPI_SWIGLU || EPI == EPI_STORE, "dual tiles: SwiGLU, and plain stores (done above)");
          constexpr int CHUNKS = COLS_PER_WARP / 32;
          uint32_t v[CHUNKS][32];
          if (have_acc) {
#pragma unroll
            for (int c = 0; c < CHUNKS; ++c) tmem_ld32(t_addr + (col_half * CHUNKS + c) * 32, v[c]);
            tmem_ld_wait();
            release_acc();
          } else {
#pragma unroll
            for (int c = 0; c < CHUNKS; ++c)
#pragma unroll
              for (int j = 0; j < 32; ++j) v[c][j] = 0u;
          }
          if constexpr (EPI == EPI_SWIGLU) {
            // z (unless not wanted) and y1 = silu(gate) * up leave through the warp's staging rows as 64-byte row
            // segments: one per 32 accumulator columns for z, one per 64 for y1 (N = 2I is a multiple of 128, so
            // chunks come in pairs)
            const uint32_t my_stage = smem_u32(stage_out) + (warp - FIRST_EPI_WARP) * STAGE_ROWS_BYTES;
            const int row_base = r - lane;
            uint32_t yp[16];
#pragma unroll
            for (int c = 0; c < CHUNKS; ++c) {
              const int n = n0 + (col_half * CHUNKS + c) * 32;
              if (n >= p.N) break;
              uint32_t zp[16];
#pragma unroll
              for (int j = 0; j < 16; ++j) {
                const float g = __uint_as_float(v[c][2 * j]);
                const float u = __uint_as_float(v[c][2 * j + 1]);
                zp[j] = pack_bf16(g, u);
                v[c][j] = __float_as_uint(g * sigmoid_f(g) * u);  // the chunk's 16 products, kept in place
              }
#pragma unroll
              for (int j = 0; j < 8; ++j)
                yp[(c & 1) * 8 + j] = pack_bf16(__uint_as_float(v[c][2 * j]), __uint_as_float(v[c][2 * j + 1]));
              if (p.out0 != nullptr)
                warp_store_rows64(my_stage, lane, zp, p.out0, p.ld0, row_base, tile.row_end, n);
              if (c & 1)
                warp_store_rows64(my_stage, lane, yp, p.out1, p.ld1, row_base, tile.row_end,
                                                          (n - 32) >> 1);
            }
          }
        } else {
          // Single tiles: each warp's 128 columns 32 at a time, row traffic in whole 64-byte segments through its staging
          // rows.  Eight warps, not four: with a short reduction the epilogue of a tile is longer than its main loop, and
          // it is latency (tensor memory, shared memory, the stores) that its warps wait for.  Four warps took 4.1 us per
          // plain-store tile and 25 us per dSwiGLU tile: down projection, dX and dH at T 24576, H 1536, I 256, E 128,
          // K 8 278, 327 and 284 us against 1.1, 2.2 and 6.5 us of MMAs per tile.
          const uint32_t my_stage = smem_u32(stage_out) + (warp - FIRST_EPI_WARP) * STAGE_ROWS_BYTES;
          const int row_base = r - lane;
          const int n_first = n0 + col_half * COLS_PER_WARP;
          constexpr int CHUNKS = COLS_PER_WARP / 32;
          const uint32_t t_cols = t_addr + col_half * COLS_PER_WARP;
          if constexpr (EPI == EPI_DSWIGLU) {
            ok = dact_columns<FN_SILU, true, CHUNKS>(p, my_stage, lane, row_base, tile.row_end, n_first,
                                                                      t_cols, score, ds_acc, wait_acc, release_acc);
          } else if constexpr (EPI == EPI_DACT) {
            ok = dact_columns<act_fn(ACT), act_is_gated(ACT), CHUNKS>(p, my_stage, lane, row_base, tile.row_end, n_first,
                                                                      t_cols, score, ds_acc, wait_acc, release_acc);
          } else if constexpr (EPI == EPI_SWIGLU) {
            act_columns<FN_SILU, true, CHUNKS>(p, tile.e, my_stage, lane, row_base, tile.row_end, n_first,
                                                                t_cols, release_acc);
          } else if constexpr (EPI == EPI_ACT) {
            act_columns<act_fn(ACT), act_is_gated(ACT), CHUNKS>(p, tile.e, my_stage, lane, row_base, tile.row_end, n_first,
                                                                t_cols, release_acc);
          } else {
            int dst_row = 0;
            if constexpr (EPI == EPI_STORE_ROWS || EPI == EPI_SCATTER) {
              if (row_ok) dst_row = p.gather[r];
            }
            if (n_first >= p.N) release_acc();
#pragma unroll 1
            for (int c = 0; c < CHUNKS; ++c) {
              const int n = n_first + 32 * c;
              if (n >= p.N) break;
              uint32_t v[32];
              if (have_acc) {
                tmem_ld32(t_cols + 32 * c, v);
                tmem_ld_wait();
                if (c + 1 == CHUNKS || n + 32 >= p.N) release_acc();
              } else {
#pragma unroll
                for (int j = 0; j < 32; ++j) v[j] = 0u;
              }
              store_chunk<EPI, RAGGED_K>(p, tile.e, my_stage, lane, row_base, tile.row_end, n, v, score,
                                                          dst_row);
            }
          }
          if (!ok) break;
        }
        if constexpr (EPI == EPI_DSWIGLU || EPI == EPI_DACT) {
          if (row_ok && n0 < p.N) {
            p.ds_partial[static_cast<long long>(2 * (n0 / BN) + col_half) * p.total_rows + r] = ds_acc;
          }
        }
        if constexpr (DUAL == DUAL_NONE) {
          if (have_acc && ++acc == 2) { acc = 0; acc_phase ^= 1u; }
        }
      }
      if constexpr (DUAL != DUAL_NONE) {
        if (have_acc) acc_phase ^= 1u;
      }
    }
    if (!ok && lane == 0 && p.status) atomicCAS(p.status, ST_OK, ST_TIMEOUT_EPILOGUE);
  }

  // ---- tear-down ----------------------------------------------------------------------------
  if (*abort_flag != 0) {
    const uint64_t t0 = global_timer_ns();
    while (global_timer_ns() - t0 < 200000ull) __nanosleep(1000);
  }
  // The MMA role is one lane's, and the other 31 of its warp come here at once.  They wait in barriers that allow for that;
  // a warp barrier before aligned ones would do as well, but slowed the whole loop of the lane (T 32768, H 4096, I 1024,
  // E 128, K 8: dX 3665 -> 3823 us, dH 2571 -> 2776).
  tc_fence_before();
  block_sync_diverged();
  cluster_sync_diverged();  // neither CTA leaves while the other may still signal its barriers or read its smem
  if (warp == 1) {
    __syncwarp();
    tc_fence_after();
    tmem_dealloc(tmem_base, 2 * BN);
  }
}

}  // namespace pair
}  // namespace smoe

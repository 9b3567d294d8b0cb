// Grouped GEMM for experts with few rows each (decode steps, short prompts): the weights are read once and that is the
// work, so the roles of the operands are exchanged.  A CTA computes 128 output features (the 128 rows of the MMA) x up to
// NT routed rows (its columns, as many as there are, rounded up to 16), instead of 256 x 256 tiles in which the rows that
// an expert does not have are loaded and multiplied like the others: with 256 rows a k-block's MMAs take as long as its
// weights take to arrive from memory, here they take an eighth of it at 32 rows, and the stages hold weights.
//
// Persistent, one CTA per SM; a unit is (expert, 128 features, NT rows), rows innermost.  Warps:
//   0        TMA producer: the weight tile 128 x 64, and the row tile when rows are not gathered (boxes of 32 rows)
//   1        MMA issuer (one thread)
//   2..9     epilogue: warp = 32 features (tensor-memory lanes) x every other 32 rows
//   10..13   row gather with TMA tile::gather4 (GATHER)
// Every wait is bounded (ptx.cuh).
//
// A thread of the epilogue holds one feature of 32 rows, and memory wants 32 features of a row: neighbouring lanes
// exchange half of their values, so that each has two features (gate and up of SwiGLU) of every other row, and the warp's
// staging rows turn these words into 64-byte row segments.
#pragma once
#include "epilogue.cuh"
#include "launch.cuh"
#include "ptx.cuh"

namespace smoe {
namespace skinny {

constexpr int BM = 128;  // features per unit
constexpr int BK = 64;
constexpr int UMMA_K = 16;
constexpr int W_STAGE_BYTES = BM * BK * 2;
constexpr int MAX_NT = 128;
constexpr int MAX_STAGES = 10;
constexpr int MAX_EXPERTS = 1024;
constexpr int EPI_WARPS = 8;
constexpr int FIRST_EPI_WARP = 2;
constexpr int FIRST_GATHER_WARP = FIRST_EPI_WARP + EPI_WARPS;
constexpr int GATHER_WARPS = 4;
constexpr int BOX_ROWS = 32;  // rows per TMA box of a row tile that is not gathered
__host__ __device__ constexpr int threads(bool gather) { return 32 * (FIRST_GATHER_WARP + (gather ? GATHER_WARPS : 0)); }

struct Shared {
  uint64_t full[MAX_STAGES];
  uint64_t empty[MAX_STAGES];
  uint64_t acc_full[2];
  uint64_t acc_empty[2];
  uint32_t tmem_base;
  int abort_flag;
  int off[MAX_EXPERTS + 1];
  int tile_prefix[MAX_EXPERTS + 1];  // exclusive prefix of the experts' row tiles: ceil(count / NT), 0 above max_rows
};

__host__ __device__ constexpr int stage_bytes(int nt) { return W_STAGE_BYTES + nt * BK * 2; }
__host__ __device__ constexpr int smem_bytes(int nt, int stages) {
  return 1024 + stages * stage_bytes(nt) + EPI_WARPS * STAGE_ROWS_BYTES + static_cast<int>(sizeof(Shared));
}
// as many stages as fit beside the rest (227 KiB per CTA)
__host__ __device__ constexpr int num_stages(int nt) {
  const int fit = (227 * 1024 - smem_bytes(nt, 0)) / stage_bytes(nt);
  return fit < MAX_STAGES ? fit : MAX_STAGES;
}
static_assert(num_stages(MAX_NT) >= 4 && smem_bytes(MAX_NT, num_stages(MAX_NT)) <= 227 * 1024, "shared memory");

struct Unit {
  int e, row0, rows, f0;  // expert, first grouped row, rows (1..NT), first feature
};

// The units of this CTA: every role's warps walk them with a walker of their own (all lanes call next()).
struct Walker {
  const GemmParams& p;
  const Shared& ss;
  const int lane, nt, blocks;
  int tile = 0, block = 0, e = 0, total, unit;  // expert-major: (feature block of expert e) x (its row tiles)

  __device__ __forceinline__ Walker(const GemmParams& p_, const Shared& ss_, int lane_, int nt_)
      : p(p_), ss(ss_), lane(lane_), nt(nt_), blocks((p_.N + BM - 1) / BM) {
    total = ss.tile_prefix[p.E] * blocks;
    unit = blockIdx.x;
  }
  __device__ __forceinline__ bool next(Unit& u) {
    if (unit >= total) return false;
    while (true) {  // the expert whose units contain this one, 32 experts at a time
      const int i = e + 1 + lane;
      const unsigned before = __ballot_sync(0xffffffffu, i <= p.E && ss.tile_prefix[i] * blocks <= unit);
      e += __popc(before);
      if (before != 0xffffffffu) break;
    }
    const int tiles = ss.tile_prefix[e + 1] - ss.tile_prefix[e];
    const int in_expert = unit - ss.tile_prefix[e] * blocks;
    const int b = in_expert / tiles;
    u.e = e;
    u.f0 = b * BM;
    u.row0 = ss.off[e] + (in_expert - b * tiles) * nt;
    u.rows = min(nt, ss.off[e + 1] - u.row0);
    unit += gridDim.x;
    return true;
  }
};

// Lane l holds feature l of 32 rows in v.  Afterwards word j of an even lane has the features (l, l + 1) of row 2j, and
// word j of an odd lane the features (l - 1, l) of row 2j + 1, as (lo, hi).
__device__ __forceinline__ void pair_features(const uint32_t (&v)[32], int lane, float (&lo)[16], float (&hi)[16]) {
  const bool odd = lane & 1;
#pragma unroll
  for (int j = 0; j < 16; ++j) {
    const uint32_t other = __shfl_xor_sync(0xffffffffu, odd ? v[2 * j] : v[2 * j + 1], 1);
    lo[j] = __uint_as_float(odd ? other : v[2 * j]);
    hi[j] = __uint_as_float(odd ? v[2 * j + 1] : other);
  }
}

__device__ __forceinline__ void st_shared_b32(uint32_t addr, uint32_t v) {
  asm volatile("st.shared.b32 [%0], %1;" ::"r"(addr), "r"(v) : "memory");
}
__device__ __forceinline__ void st_shared_b16(uint32_t addr, __nv_bfloat16 v) {
  asm volatile("st.shared.b16 [%0], %1;" ::"r"(addr), "h"(__bfloat16_as_ushort(v)) : "memory");
}

// 32 rows x BYTES (64 or 32) that lie row by row in the staging area go out in 16-byte pieces.
template <int BYTES>
__device__ __forceinline__ void store_staged(uint32_t stage, int lane, __nv_bfloat16* out, long long ld, int row0,
                                             int rows, int col) {
  constexpr int PIECES = BYTES / 16, ROWS = 32 / PIECES;
#pragma unroll
  for (int i = 0; i < PIECES; ++i) {
    const int rr = ROWS * i + lane / PIECES;
    const uint4 v = ld_shared_v4(stage + rr * BYTES + 16 * (lane % PIECES));
    if (rr < rows) *reinterpret_cast<uint4*>(out + (row0 + rr) * ld + col + 8 * (lane % PIECES)) = v;
  }
}

template <bool GATHER, bool SWIGLU>
__global__ void __launch_bounds__(threads(GATHER), 1)
skinny_gemm_kernel(const __grid_constant__ CUtensorMap tmW, const __grid_constant__ CUtensorMap tmX, const GemmParams p,
                   const int nt, const int stages) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  const int stage_size = stage_bytes(nt);
  uint8_t* stage_out = smem + stages * stage_size;
  Shared& ss = *reinterpret_cast<Shared*>(stage_out + EPI_WARPS * STAGE_ROWS_BYTES);
  const int warp = warp_index();
  const int lane = threadIdx.x & 31;
  volatile int* abort_flag = &ss.abort_flag;
  const int num_kb = p.K / BK;

  if (threadIdx.x == 0) {
    for (int s = 0; s < stages; ++s) {
      mbar_init(smem_u32(&ss.full[s]), 1 + (GATHER ? GATHER_WARPS : 0));
      mbar_init(smem_u32(&ss.empty[s]), 1);
    }
    for (int a = 0; a < 2; ++a) {
      mbar_init(smem_u32(&ss.acc_full[a]), 1);
      mbar_init(smem_u32(&ss.acc_empty[a]), EPI_WARPS);
    }
    ss.abort_flag = 0;
    fence_mbar_init();
    tma_prefetch_desc(&tmW);
    tma_prefetch_desc(&tmX);
  }
  if (warp == 1) {
    tmem_alloc(smem_u32(&ss.tmem_base), 2 * MAX_NT);
    tmem_relinquish();
  }
  wait_for_previous();
  for (int e = threadIdx.x; e <= p.E; e += blockDim.x) ss.off[e] = p.off[e];
  if (warp == 2) {
    const int max_rows = p.max_rows < p.total_rows && tiles_take_all(p, p.max_rows, lane) ? 0 : p.max_rows;
    int running = 0;
    for (int base = 0; base < p.E; base += 32) {
      const int e = base + lane;
      const int rows = e < p.E ? p.off[e + 1] - p.off[e] : 0;
      const int v = rows <= max_rows ? (rows + nt - 1) / nt : 0;
      int incl = v;
#pragma unroll
      for (int d = 1; d < 32; d <<= 1) {
        const int o = __shfl_up_sync(0xffffffffu, incl, d);
        if (lane >= d) incl += o;
      }
      if (e < p.E) ss.tile_prefix[e] = running + incl - v;
      running += __shfl_sync(0xffffffffu, incl, 31);
    }
    if (lane == 0) ss.tile_prefix[p.E] = running;
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = ss.tmem_base;
  bool ok = true;
  Unit u;
  Walker walk(p, ss, lane, nt);

  if (warp == 0) {
    // ---- TMA producer -------------------------------------------------------------------------
    const bool elected = elect_one();
    int stage = 0;
    uint32_t phase = 0;
    while (ok && walk.next(u)) {
      const int boxes = (u.rows + BOX_ROWS - 1) / BOX_ROWS;
      const uint32_t bytes = W_STAGE_BYTES + (GATHER ? (u.rows + 3) / 4 * 512 : boxes * (BOX_ROWS * BK * 2));
      for (int kb = 0; kb < num_kb; ++kb) {
        if (!mbar_wait_warp(smem_u32(&ss.empty[stage]), phase ^ 1u, abort_flag)) { ok = false; break; }
        const uint32_t bar = smem_u32(&ss.full[stage]);
        const uint32_t dst = smem_u32(smem + stage * stage_size);
        if (elected) {
          mbar_arrive_expect_tx(bar, bytes);
          tma_load_2d(&tmW, bar, dst, kb * BK, u.e * p.b_rows_per_expert + u.f0);
          if constexpr (!GATHER) {
            for (int b = 0; b < boxes; ++b)
              tma_load_2d(&tmX, bar, dst + W_STAGE_BYTES + b * (BOX_ROWS * BK * 2), kb * BK, u.row0 + b * BOX_ROWS);
          }
        }
        __syncwarp();
        if (++stage == stages) { stage = 0; phase ^= 1u; }
      }
    }
    if (!ok && lane == 0 && p.status) atomicCAS(p.status, ST_OK, ST_TIMEOUT_PRODUCER);
  } else if (warp == 1) {
    // ---- MMA issuer ---------------------------------------------------------------------------
    const bool elected = elect_one();
    int stage = 0, acc = 0;
    uint32_t phase = 0, acc_phase = 0;
    while (ok && walk.next(u)) {
      if (elected) {
        const uint32_t idesc = make_idesc_bf16(BM, (u.rows + 15) & ~15, false, false);
        ok = mbar_wait(smem_u32(&ss.acc_empty[acc]), acc_phase ^ 1u, abort_flag);
        tc_fence_after();
        for (int kb = 0; ok && kb < num_kb; ++kb) {
          if (!mbar_wait(smem_u32(&ss.full[stage]), phase, abort_flag)) { ok = false; break; }
          tc_fence_after();
          const uint32_t w_addr = smem_u32(smem + stage * stage_size);
          const uint64_t a_desc = make_smem_desc(w_addr, 16, 1024);
          const uint64_t b_desc = make_smem_desc(w_addr + W_STAGE_BYTES, 16, 1024);
#pragma unroll
          for (int k4 = 0; k4 < BK / UMMA_K; ++k4)
            umma_bf16(tmem_base + acc * MAX_NT, a_desc + ((k4 * UMMA_K * 2) >> 4), b_desc + ((k4 * UMMA_K * 2) >> 4),
                      idesc, (kb > 0 || k4 > 0) ? 1u : 0u);
          umma_commit(smem_u32(&ss.empty[stage]));
          if (++stage == stages) { stage = 0; phase ^= 1u; }
        }
        if (ok) umma_commit(smem_u32(&ss.acc_full[acc]));
      }
      ok = __all_sync(0xffffffffu, ok);
      if (++acc == 2) { acc = 0; acc_phase ^= 1u; }
    }
    if (!ok && lane == 0 && p.status) atomicCAS(p.status, ST_OK, ST_TIMEOUT_MMA);
  } else if (warp >= FIRST_GATHER_WARP) {
    // ---- row gather ---------------------------------------------------------------------------
    if constexpr (GATHER) {
      const int gt = threadIdx.x - 32 * FIRST_GATHER_WARP;
      const bool issuer = (gt & 3) == 0;  // every fourth thread: a warp issues for 32 rows, so units of 128 rows take all four
      const int j = gt >> 2;              // rows 4j .. 4j+3 of the unit
      int stage = 0;
      uint32_t phase = 0;
      while (ok && walk.next(u)) {
        const bool mine = issuer && 4 * j < u.rows;
        int r4[4];
#pragma unroll
        for (int i = 0; i < 4; ++i)  // an index out of range delivers zeros
          r4[i] = mine && 4 * j + i < u.rows ? p.gather[u.row0 + 4 * j + i] : p.gather_rows;
        for (int kb = 0; kb < num_kb; ++kb) {
          if (!mbar_wait_warp(smem_u32(&ss.empty[stage]), phase ^ 1u, abort_flag)) { ok = false; break; }
          if (mine)
            tma_gather4(&tmX, smem_u32(&ss.full[stage]), smem_u32(smem + stage * stage_size) + W_STAGE_BYTES + j * 512,
                        kb * BK, r4[0], r4[1], r4[2], r4[3]);
          __syncwarp();
          // A stage is not full without this warp, also where the warp has no rows: it waits by parity, and a warp that the
          // ring could overtake twice would take an old phase for the one it waits for.
          if (lane == 0) mbar_arrive(smem_u32(&ss.full[stage]));
          if (++stage == stages) { stage = 0; phase ^= 1u; }
        }
      }
      if (!ok && lane == 0 && p.status) atomicCAS(p.status, ST_OK, ST_TIMEOUT_PRODUCER);
    }
  } else {
    // ---- epilogue -----------------------------------------------------------------------------
    const int quad = warp & 3;
    const int half = (warp - FIRST_EPI_WARP) >> 2;
    const uint32_t my_stage = smem_u32(stage_out) + (warp - FIRST_EPI_WARP) * STAGE_ROWS_BYTES;
    int acc = 0;
    uint32_t acc_phase = 0;
    while (ok && walk.next(u)) {
      if (!mbar_wait_warp(smem_u32(&ss.acc_full[acc]), acc_phase, abort_flag)) { ok = false; break; }
      tc_fence_after();
      const uint32_t t_addr = tmem_base + acc * MAX_NT + (static_cast<uint32_t>(quad * 32) << 16);
      const int f = u.f0 + quad * 32;
      const auto release = [&] {
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(smem_u32(&ss.acc_empty[acc]));
      };
      const bool works = 32 * half < u.rows && f < p.N;  // N is a multiple of 64
      if (!works) release();
      for (int c = half; works && 32 * c < u.rows; c += 2) {
        uint32_t v[32];
        tmem_ld32(t_addr + 32 * c, v);
        tmem_ld_wait();
        if (32 * (c + 2) >= u.rows) release();
        float lo[16], hi[16];
        pair_features(v, lane, lo, hi);
        const int row0 = u.row0 + 32 * c, rows = u.rows - 32 * c;
        if (!SWIGLU || p.out0 != nullptr) {
#pragma unroll
          for (int j = 0; j < 16; ++j)
            st_shared_b32(my_stage + (2 * j + (lane & 1)) * 64 + 4 * (lane >> 1), pack_bf16(lo[j], hi[j]));
          __syncwarp();
          store_staged<64>(my_stage, lane, p.out0, p.ld0, row0, rows, f);
          __syncwarp();
        }
        if constexpr (SWIGLU) {
#pragma unroll
          for (int j = 0; j < 16; ++j)
            st_shared_b16(my_stage + (2 * j + (lane & 1)) * 32 + 2 * (lane >> 1),
                          __float2bfloat16_rn(lo[j] * sigmoid_f(lo[j]) * hi[j]));
          __syncwarp();
          store_staged<32>(my_stage, lane, p.out1, p.ld1, row0, rows, f >> 1);
          __syncwarp();
        }
      }
      if (++acc == 2) { acc = 0; acc_phase ^= 1u; }
    }
    if (!ok && lane == 0 && p.status) atomicCAS(p.status, ST_OK, ST_TIMEOUT_EPILOGUE);
  }

  // ---- tear-down ----------------------------------------------------------------------------
  __syncwarp();
  if (*abort_flag != 0) {
    const uint64_t t0 = global_timer_ns();
    while (global_timer_ns() - t0 < 200000ull) __nanosleep(1000);
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base, 2 * MAX_NT);
  }
}

}  // namespace skinny
}  // namespace smoe

// Parameter block, status codes and the fused epilogues shared by the grouped GEMM kernels.
#pragma once
#include "ptx.cuh"

namespace smoe {


enum Epilogue : int {
  EPI_STORE = 0,    // out0[r, n] = bf16(acc)
  EPI_SWIGLU = 1,   // out0[r, n] = bf16(acc) (unless out0 == nullptr); out1[r, n/2] = silu(acc[2j]) * acc[2j+1]
  EPI_DSWIGLU = 2,  // acc = dy1; reads z, score; writes dz (out0), y1*s (out1), per-row partial of ds
  EPI_SCATTER = 3,  // red.add fp32: acc_out[token(r), n] += score(r) * acc
  // general forms: any activation of the layer, optional per-expert bias (EPI + 16 * Activation, GemmParams::bias)
  EPI_ACT = 4,         // z = acc + b1 -> out0 (unless nullptr); y1 = act(z) (gated: act(z_even) * z_odd) -> out1
  EPI_DACT = 5,        // acc = dy1; reads z, score; writes dz (out0), y1*s (out1), per-row partial of ds
  EPI_STORE_BIAS = 6,  // out0[r, n] = bf16(acc + bias[e, n])
  EPI_STORE_ROWS = 7,  // out0[gather[r], n] = bf16(score(r) * bf16(acc)) (score 1 when scores == nullptr): grouped rows
                       // written straight back to their source rows -- the combine of a layer whose tokens have one
                       // routed row each, with the rounding points of the store + gather_sum pair it replaces
};

// Activation codes.  The first three are gated: the pre-activation has 2I columns,
// gate = even column, up = odd column.
enum Activation : int { ACT_SWIGLU = 0, ACT_GEGLU = 1, ACT_REGLU = 2, ACT_RELU_SQ = 3, ACT_RELU = 4, ACT_GELU = 5,
                        ACT_SILU = 6 };
__host__ __device__ constexpr bool act_is_gated(int act) { return act <= ACT_REGLU; }

// Status codes written to GemmParams::status (first failure wins).
enum Status : int { ST_OK = 0, ST_TIMEOUT_PRODUCER = 1, ST_TIMEOUT_MMA = 2, ST_TIMEOUT_EPILOGUE = 3 };

struct GemmParams {
  int E;            // experts
  int M;            // ragged-K: rows of each expert's output; ragged-M: unused
  int N;            // output columns (per expert)
  int K;            // ragged-M: reduction length; ragged-K: unused
  int total_rows;   // rows of the grouped (expert-sorted) layout
  int gather_rows;  // rows of the tensor a gather reads from (an index >= gather_rows reads zeros)
  int b_rows_per_expert;  // ragged-M: rows one expert occupies in B's flattened 2D tensor map
  const int* off;         // (E+1) first grouped row of every expert
  const int* gather;      // (total_rows) source row of every grouped row, or nullptr
  __nv_bfloat16* out0;
  long long ld0;
  long long out0_expert_stride;  // ragged-K only
  __nv_bfloat16* out1;
  long long ld1;
  // EPI_DSWIGLU / EPI_SCATTER
  const __nv_bfloat16* z;   // (total_rows, 2N) pre-activation saved by the forward pass
  const void* scores;       // flat routing scores, fp32 or bf16
  int scores_are_bf16;
  const int* s_scatter;     // (total_rows) flat score slot of every grouped row
  float* ds_partial;        // (2 * ceil(N/BN), total_rows) fp32: one row of partials per 128 accumulator columns
  float* acc_out;           // EPI_SCATTER: (gather_rows, N) fp32
  int* status;              // device word, 0 = ok
  int accumulate;           // plain-store epilogues: add to what out0 holds (bf16, fp32 sum, one rounding) instead of
                            // overwriting it -- weight gradients summed over several chunks of tokens, rows of dx that
                            // hold the router's part already
  int min_rows;             // ragged-M tiles: experts with at most this many rows are left to another launch
  int max_rows;             // kernel for experts with few rows: those with more are left to another launch
  // general epilogues
  const __nv_bfloat16* bias;  // (E, N) added to the accumulator, or nullptr
  // EPI_DSWIGLU of the hardware-scaled FP8 kernel: dz also leaves the epilogue quantised (E4M3, one UE8M0 scale
  // byte per row and 128 columns), nullptr = not wanted
  uint8_t* q_out;             // (total_rows, 2N)
  uint8_t* q_scale;           // (total_rows, q_scale_ld)
  long long q_scale_ld;
};

// Whether the experts with more than `limit` rows hold at least half of all rows.  Then the 256 x 256 tiles take all experts
// and the kernel for experts with few rows finds nothing to do: most of the others have next to none, and a wave of each
// kernel would cost more than tiles for all of them (H 4096, I 1024, 5120 rows in 128 experts, loads falling with the square
// of the rank: up projection 208 us divided, 170 by tiles).  One warp, all lanes; both kernels come to the same answer.
__device__ __forceinline__ bool tiles_take_all(const GemmParams& p, int limit, int lane) {
  int above = 0;
  for (int e = lane; e < p.E; e += 32) {
    const int rows = p.off[e + 1] - p.off[e];
    if (rows > limit) above += rows;
  }
  above = __reduce_add_sync(0xffffffffu, above);
  return 2ll * above >= p.total_rows;
}

__device__ __forceinline__ float load_score(const void* scores, int is_bf16, int slot) {
  return is_bf16 ? __bfloat162float(reinterpret_cast<const __nv_bfloat16*>(scores)[slot])
                 : reinterpret_cast<const float*>(scores)[slot];
}

__device__ __forceinline__ uint32_t pack_bf16(float lo, float hi) {
  __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
  return *reinterpret_cast<uint32_t*>(&v);
}

// sigmoid(x) = 0.5 tanh(x / 2) + 0.5 with the hardware tanh: one special-function operation per value instead of
// an exponential and a reciprocal (the epilogues are bound by those), the form the reference's epilogue uses too
// (sonicmoe/functional/grouped_gemm.py:413-421).  Absolute error about 2.5e-4, far below one bf16 step of the outputs.
__device__ __forceinline__ float sigmoid_f(float x) {
  float t;
  asm("tanh.approx.f32 %0, %1;" : "=f"(t) : "f"(0.5f * x));
  return fmaf(0.5f, t, 0.5f);
}

// Ask the L2 for `lines` consecutive 128-byte lines starting at p (no register, no wait).
__device__ __forceinline__ void prefetch_l2_lines(const void* p, int lines) {
  const char* c = static_cast<const char*>(p);
  for (int i = 0; i < lines; ++i) asm volatile("prefetch.global.L2 [%0];" ::"l"(c + 128 * i));
}

// The elementwise functions behind the layer's activations: value a and derivative da at x.
enum ActFn : int { FN_SILU = 0, FN_GELU = 1, FN_RELU_SQ = 2, FN_RELU = 3 };

template <int FN>
__device__ __forceinline__ void act_value_grad(float x, float& a, float& da) {
  if constexpr (FN == FN_SILU) {
    const float sig = sigmoid_f(x);
    a = x * sig;
    da = sig * (1.f + x * (1.f - sig));
  } else if constexpr (FN == FN_GELU) {  // exact (erf) GELU
    const float cdf = 0.5f * (1.f + erff(x * 0.70710678118654752f));
    a = x * cdf;
    da = cdf + x * 0.3989422804014327f * __expf(-0.5f * x * x);
  } else if constexpr (FN == FN_RELU_SQ) {
    const float r = fmaxf(x, 0.f);
    a = r * r;
    da = 2.f * r;
  } else {
    a = fmaxf(x, 0.f);
    da = x > 0.f ? 1.f : 0.f;
  }
}

// The general epilogues are compiled once per activation (GEMM template argument EPI + 16 * Activation): with a switch
// inside the element loop the values of a row formed one serial chain of branches and function latencies, and with one
// around the tile's loop the widest variant's spills slowed all of them (dH of T 8191, H 1024, I 512, E 32, K 4 with GELU:
// 196 us, 119 us, and 64 as it is).
__host__ __device__ constexpr int epi_base(int epi_code) { return epi_code % 16; }
__host__ __device__ constexpr int act_fn(int act) {
  return act == ACT_GEGLU || act == ACT_GELU ? FN_GELU
         : act == ACT_RELU_SQ                ? FN_RELU_SQ
         : act == ACT_REGLU || act == ACT_RELU ? FN_RELU : FN_SILU;
}

__device__ __forceinline__ void store_bf16x32(__nv_bfloat16* dst, const float (&f)[32]) {
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    uint4 w;
    w.x = pack_bf16(f[8 * j + 0], f[8 * j + 1]);
    w.y = pack_bf16(f[8 * j + 2], f[8 * j + 3]);
    w.z = pack_bf16(f[8 * j + 4], f[8 * j + 5]);
    w.w = pack_bf16(f[8 * j + 6], f[8 * j + 7]);
    reinterpret_cast<uint4*>(dst)[j] = w;
  }
}

// eight packed bf16 values plus the eight at dst (fp32 sums, rounded once)
__device__ __forceinline__ uint4 add_bf16x8(uint4 a, const uint4* dst) {
  const uint4 b = *dst;
  const uint32_t aw[4] = {a.x, a.y, a.z, a.w}, bw[4] = {b.x, b.y, b.z, b.w};
  uint32_t o[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const float2 x = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&aw[i]));
    const float2 y = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&bw[i]));
    o[i] = pack_bf16(x.x + y.x, x.y + y.y);
  }
  return make_uint4(o[0], o[1], o[2], o[3]);
}

// Warp-cooperative row I/O through a warp's staging rows (32 rows of 64 bytes, 2 KiB).  Lane l owns row l of a 32-row
// block; global memory is touched with consecutive lanes on consecutive 16-byte pieces of one row, so an instruction
// moves whole 64-byte segments.  Rows at or beyond row_end are skipped.  Every lane must call.
// The four pieces of a row are permuted by its row pair, so that both directions are free of bank conflicts (eight lanes
// write the same piece of eight rows, or read two whole rows): with 80-byte rows the reads took twice the shared-memory
// cycles, of which the tensor cores' operands leave few.
constexpr int STAGE_ROWS_BYTES = 32 * 64;
__device__ __forceinline__ uint32_t stage_piece(uint32_t stage, int row, int piece) {
  return stage + row * 64 + 16 * (piece ^ ((row >> 1) & 3));
}

// dst(rr) gives the address of the 64-byte segment of the block's row rr, or nullptr (called by every lane).
template <class Dst>
__device__ __forceinline__ void warp_store_segments64(uint32_t stage, int lane, const uint32_t (&w)[16], bool accumulate,
                                                      Dst&& dst) {
#pragma unroll
  for (int q = 0; q < 4; ++q) st_shared_v4(stage_piece(stage, lane, q), w[4 * q], w[4 * q + 1], w[4 * q + 2], w[4 * q + 3]);
  __syncwarp();
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int rr = 8 * i + (lane >> 2);
    const uint4 v = ld_shared_v4(stage_piece(stage, rr, lane & 3));
    __nv_bfloat16* d = dst(rr);
    if (d != nullptr) {
      uint4* d4 = reinterpret_cast<uint4*>(d + 8 * (lane & 3));
      *d4 = accumulate ? add_bf16x8(v, d4) : v;
    }
  }
  __syncwarp();
}

__device__ __forceinline__ void warp_store_rows64(uint32_t stage, int lane, const uint32_t (&w)[16], __nv_bfloat16* out,
                                                  long long ld, int row_base, int row_end, int col,
                                                  bool accumulate = false) {
  warp_store_segments64(stage, lane, w, accumulate, [&](int rr) {
    return row_base + rr < row_end ? out + (row_base + rr) * ld + col : nullptr;
  });
}

// acc (+ bias) as 32 floats
__device__ __forceinline__ void load_biased(const GemmParams& p, int expert, int n, const uint32_t (&v)[32],
                                            float (&f)[32]) {
#pragma unroll
  for (int j = 0; j < 32; ++j) f[j] = __uint_as_float(v[j]);
  if (p.bias != nullptr) {
    const uint4* b = reinterpret_cast<const uint4*>(p.bias + static_cast<long long>(expert) * p.N + n);
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const uint4 w = b[j];
      const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&w);
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const float2 t = __bfloat1622float2(h[i]);
        f[8 * j + 2 * i] += t.x;
        f[8 * j + 2 * i + 1] += t.y;
      }
    }
  }
}

// dSwiGLU on 32 accumulator columns (= 64 columns of dz).  acc[., i] = dy1[r, i]; z[r, 2i] = gate, z[r, 2i+1] = up.
// Writes dz (bf16), y1 * score, accumulates ds.
__device__ __forceinline__ void dswiglu_chunk(const GemmParams& p, int r, int n, const uint32_t (&v)[32], float score,
                                              float& ds_acc) {
  const uint4* zsrc = reinterpret_cast<const uint4*>(p.z + static_cast<long long>(r) * (2ll * p.N) + 2 * n);
  __nv_bfloat16* dz_dst = p.out0 + r * p.ld0 + 2 * n;
  __nv_bfloat16* ys_dst = p.out1 + r * p.ld1 + n;
#pragma unroll
  for (int j = 0; j < 4; ++j) {  // 8 accumulator columns per step
    const uint4 za = zsrc[2 * j], zb = zsrc[2 * j + 1];
    const uint32_t zw[8] = {za.x, za.y, za.z, za.w, zb.x, zb.y, zb.z, zb.w};
    uint32_t dzw[8];
    float ys[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const __nv_bfloat162 gu = *reinterpret_cast<const __nv_bfloat162*>(&zw[i]);
      const float g = __low2float(gu), u = __high2float(gu);
      const float dy = __uint_as_float(v[8 * j + i]);
      const float sig = sigmoid_f(g);
      const float silu = g * sig;
      const float y1 = silu * u;
      ds_acc += dy * y1;
      const float dg = dy * u * (sig * (1.f + g * (1.f - sig))) * score;
      const float du = dy * silu * score;
      dzw[i] = pack_bf16(dg, du);
      ys[i] = y1 * score;
    }
    reinterpret_cast<uint4*>(dz_dst)[2 * j] = make_uint4(dzw[0], dzw[1], dzw[2], dzw[3]);
    reinterpret_cast<uint4*>(dz_dst)[2 * j + 1] = make_uint4(dzw[4], dzw[5], dzw[6], dzw[7]);
    reinterpret_cast<uint4*>(ys_dst)[j] = make_uint4(pack_bf16(ys[0], ys[1]), pack_bf16(ys[2], ys[3]),
                                                     pack_bf16(ys[4], ys[5]), pack_bf16(ys[6], ys[7]));
  }
}

// The inverse: 32 rows x 64 bytes read with whole-row-segment loads; lane l ends with row l (zeros past row_end).
__device__ __forceinline__ void warp_load_rows64(uint32_t stage, int lane, uint32_t (&w)[16], const __nv_bfloat16* src,
                                                 long long ld, int row_base, int row_end, int col) {
  uint4 v[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int rr = 8 * i + (lane >> 2);
    v[i] = make_uint4(0u, 0u, 0u, 0u);
    if (row_base + rr < row_end)
      v[i] = *reinterpret_cast<const uint4*>(src + (row_base + rr) * ld + col + 8 * (lane & 3));
  }
#pragma unroll
  for (int i = 0; i < 4; ++i)
    st_shared_v4(stage_piece(stage, 8 * i + (lane >> 2), lane & 3), v[i].x, v[i].y, v[i].z, v[i].w);
  __syncwarp();
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    const uint4 t = ld_shared_v4(stage_piece(stage, lane, q));
    w[4 * q] = t.x; w[4 * q + 1] = t.y; w[4 * q + 2] = t.z; w[4 * q + 3] = t.w;
  }
  __syncwarp();
}

// dswiglu_chunk with the row traffic (z in, dz and y1 * score out) going through the warp's staging rows as 64-byte
// row segments.  Every lane of the warp must call (lane l owns row row_base + l; rows at or past row_end read zeros
// and store nothing).  Same arithmetic, same results.  KEEP: the 32 packed bf16x2 words of dz replace v and amax collects
// max |dz| over the bf16 values (for a caller that also quantises dz).
template <bool KEEP>
__device__ __forceinline__ void dswiglu_chunk_staged(const GemmParams& p, uint32_t stage, int lane, int row_base,
                                                     int row_end, int n, uint32_t (&v)[32], float score, float& ds_acc,
                                                     float& amax) {
  uint32_t za[16], zb[16], ys[16];
  warp_load_rows64(stage, lane, za, p.z, 2ll * p.N, row_base, row_end, 2 * n);
  warp_load_rows64(stage, lane, zb, p.z, 2ll * p.N, row_base, row_end, 2 * n + 32);
#pragma unroll
  for (int i = 0; i < 32; ++i) {
    uint32_t& zw = i < 16 ? za[i] : zb[i - 16];
    const __nv_bfloat162 gu = *reinterpret_cast<const __nv_bfloat162*>(&zw);
    const float g = __low2float(gu), u = __high2float(gu);
    const float dy = __uint_as_float(v[i]);
    const float sig = sigmoid_f(g);
    const float silu = g * sig;
    const float y1 = silu * u;
    ds_acc += dy * y1;
    const float dg = dy * u * (sig * (1.f + g * (1.f - sig))) * score;
    const float du = dy * silu * score;
    zw = pack_bf16(dg, du);
    v[i] = __float_as_uint(y1 * score);
  }
#pragma unroll
  for (int j = 0; j < 16; ++j) ys[j] = pack_bf16(__uint_as_float(v[2 * j]), __uint_as_float(v[2 * j + 1]));
  warp_store_rows64(stage, lane, za, p.out0, p.ld0, row_base, row_end, 2 * n);
  warp_store_rows64(stage, lane, zb, p.out0, p.ld0, row_base, row_end, 2 * n + 32);
  warp_store_rows64(stage, lane, ys, p.out1, p.ld1, row_base, row_end, n);
  if constexpr (KEEP) {
#pragma unroll
    for (int i = 0; i < 32; ++i) {
      const uint32_t w = i < 16 ? za[i] : zb[i - 16];
      v[i] = w;
      amax = fmaxf(amax, fmaxf(fabsf(__uint_as_float(w << 16)), fabsf(__uint_as_float(w & 0xFFFF0000u))));
    }
  }
}

// One 32-column piece of one accumulator row, stored by the lane that holds it: v[j] = acc[r, n + j].  FP8 kernels.
template <int EPI>
__device__ __forceinline__ void epilogue_chunk(const GemmParams& p, int r, int n, uint32_t (&v)[32], float score,
                                               float& ds_acc) {
  if constexpr (EPI == EPI_STORE) {
    __nv_bfloat16* dst = p.out0 + r * p.ld0 + n;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      uint4 w;
      w.x = pack_bf16(__uint_as_float(v[8 * j + 0]), __uint_as_float(v[8 * j + 1]));
      w.y = pack_bf16(__uint_as_float(v[8 * j + 2]), __uint_as_float(v[8 * j + 3]));
      w.z = pack_bf16(__uint_as_float(v[8 * j + 4]), __uint_as_float(v[8 * j + 5]));
      w.w = pack_bf16(__uint_as_float(v[8 * j + 6]), __uint_as_float(v[8 * j + 7]));
      reinterpret_cast<uint4*>(dst)[j] = w;
    }
  } else if constexpr (EPI == EPI_SWIGLU) {
    if (p.out0 != nullptr) {
      __nv_bfloat16* dst = p.out0 + r * p.ld0 + n;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        uint4 w;
        w.x = pack_bf16(__uint_as_float(v[8 * j + 0]), __uint_as_float(v[8 * j + 1]));
        w.y = pack_bf16(__uint_as_float(v[8 * j + 2]), __uint_as_float(v[8 * j + 3]));
        w.z = pack_bf16(__uint_as_float(v[8 * j + 4]), __uint_as_float(v[8 * j + 5]));
        w.w = pack_bf16(__uint_as_float(v[8 * j + 6]), __uint_as_float(v[8 * j + 7]));
        reinterpret_cast<uint4*>(dst)[j] = w;
      }
    }
    // gate = even column, up = odd column
    float y[16];
#pragma unroll
    for (int j = 0; j < 16; ++j) {
      const float g = __uint_as_float(v[2 * j]);
      const float u = __uint_as_float(v[2 * j + 1]);
      y[j] = g * sigmoid_f(g) * u;
    }
    __nv_bfloat16* dst1 = p.out1 + r * p.ld1 + (n >> 1);
#pragma unroll
    for (int j = 0; j < 2; ++j) {
      uint4 w;
      w.x = pack_bf16(y[8 * j + 0], y[8 * j + 1]);
      w.y = pack_bf16(y[8 * j + 2], y[8 * j + 3]);
      w.z = pack_bf16(y[8 * j + 4], y[8 * j + 5]);
      w.w = pack_bf16(y[8 * j + 6], y[8 * j + 7]);
      reinterpret_cast<uint4*>(dst1)[j] = w;
    }
  } else if constexpr (EPI == EPI_DSWIGLU) {
    dswiglu_chunk(p, r, n, v, score, ds_acc);
  } else if constexpr (EPI == EPI_STORE_ROWS) {
    __nv_bfloat16* dst = p.out0 + static_cast<long long>(p.gather[r]) * p.ld0 + n;
    float f[32];
#pragma unroll
    for (int j = 0; j < 32; ++j) f[j] = __uint_as_float(v[j]);
    if (p.scores != nullptr) {
#pragma unroll
      for (int j = 0; j < 32; ++j) f[j] = score * __bfloat162float(__float2bfloat16_rn(f[j]));
    }
    store_bf16x32(dst, f);
  }
}

// The backward activation epilogue of one warp: CHUNKS x 32 accumulator columns (dy1) of its 32 rows.  Reads the saved
// pre-activation z, writes dz and y1 * score, adds to the row's partial of ds.  acc[., i] = dy1[r, i]; gated: z[r, 2i] =
// gate, z[r, 2i+1] = up.  All row traffic goes through the warp's staging rows in whole 64-byte segments, and the next
// chunk's z is in flight while this one is worked on: the first one's before the accumulator is waited for.  Lane l owns
// row row_base + l; rows at or past row_end read zeros and store nothing.
// Bound by latency, not by arithmetic: four warps without the z pipeline needed 25 us for a 256 x 256 tile (dH of
// T 24576, H 1536, I 256, E 128, K 8: 284 us), more than the MMAs of a reduction of 4096.
template <int FN, bool GATED, int CHUNKS, class Wait, class Release>
__device__ __forceinline__ bool dact_columns(const GemmParams& p, uint32_t stage, int lane, int row_base, int row_end,
                                             int n_first, uint32_t t_addr, float score, float& ds_acc, Wait&& wait_acc,
                                             Release&& release_acc) {
  constexpr int ZW = GATED ? 2 : 1;          // z columns per accumulator column
  constexpr int ROWS = GATED ? 4 : 8;        // rows that one load instruction of the warp covers
  constexpr int PIECES = 32 / ROWS;          // 16-byte pieces per row and chunk
  const __nv_bfloat16* z = p.z + 8 * (lane % PIECES);
  const long long z_ld = static_cast<long long>(ZW) * p.N;
  uint4 vz[4 * ZW];
  auto fetch_z = [&](int n) {
#pragma unroll
    for (int i = 0; i < 4 * ZW; ++i) {
      const int r = row_base + ROWS * i + lane / PIECES;
      vz[i] = make_uint4(0u, 0u, 0u, 0u);
      if (r < row_end) vz[i] = *reinterpret_cast<const uint4*>(z + r * z_ld + ZW * n);
    }
  };
  if (n_first < p.N) {
    fetch_z(n_first);
    // the other chunks' pieces of this lane's row: have the L2 fetch them meanwhile
    if (row_base + lane < row_end)
      prefetch_l2_lines(p.z + (row_base + lane) * z_ld + ZW * n_first, min(CHUNKS * 32, p.N - n_first) * ZW * 2 / 128);
  }
  if (!wait_acc()) return false;
  if (n_first >= p.N) release_acc();
#pragma unroll 1
  for (int c = 0; c < CHUNKS; ++c) {
    const int n = n_first + 32 * c;
    if (n >= p.N) break;
    uint32_t v[32], zw[16 * ZW];
    tmem_ld32(t_addr + 32 * c, v);
#pragma unroll
    for (int h = 0; h < ZW; ++h) {  // 64 bytes of every row at a time
#pragma unroll
      for (int i = 0; i < 4 * ZW; ++i)
        if (!GATED || ((lane >> 2) & 1) == h)
          st_shared_v4(stage_piece(stage, ROWS * i + lane / PIECES, lane & 3), vz[i].x, vz[i].y, vz[i].z, vz[i].w);
      __syncwarp();
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const uint4 t = ld_shared_v4(stage_piece(stage, lane, q));
        zw[16 * h + 4 * q] = t.x; zw[16 * h + 4 * q + 1] = t.y; zw[16 * h + 4 * q + 2] = t.z; zw[16 * h + 4 * q + 3] = t.w;
      }
      __syncwarp();
    }
    const bool more = c + 1 < CHUNKS && n + 32 < p.N;
    if (more) fetch_z(n + 32);
    tmem_ld_wait();
    if (!more) release_acc();
    uint32_t out[16];
    if constexpr (GATED) {
#pragma unroll
      for (int i = 0; i < 32; ++i) {
        const __nv_bfloat162 gu = *reinterpret_cast<const __nv_bfloat162*>(&zw[i]);
        const float g = __low2float(gu), u = __high2float(gu);
        const float dy = __uint_as_float(v[i]);
        float a, da;
        act_value_grad<FN>(g, a, da);
        const float y1 = a * u;
        ds_acc += dy * y1;
        zw[i] = pack_bf16(dy * u * da * score, dy * a * score);
        v[i] = __float_as_uint(y1 * score);
      }
#pragma unroll
      for (int h = 0; h < 2; ++h) {
#pragma unroll
        for (int j = 0; j < 16; ++j) out[j] = zw[16 * h + j];
        warp_store_rows64(stage, lane, out, p.out0, p.ld0, row_base, row_end, 2 * n + 32 * h);
      }
    } else {
#pragma unroll
      for (int i = 0; i < 16; ++i) {
        const __nv_bfloat162 zz = *reinterpret_cast<const __nv_bfloat162*>(&zw[i]);
        const float d0 = __uint_as_float(v[2 * i]), d1 = __uint_as_float(v[2 * i + 1]);
        float a0, da0, a1, da1;
        act_value_grad<FN>(__low2float(zz), a0, da0);
        act_value_grad<FN>(__high2float(zz), a1, da1);
        ds_acc += d0 * a0;
        ds_acc += d1 * a1;
        out[i] = pack_bf16(d0 * da0 * score, d1 * da1 * score);
        v[2 * i] = __float_as_uint(a0 * score);
        v[2 * i + 1] = __float_as_uint(a1 * score);
      }
      warp_store_rows64(stage, lane, out, p.out0, p.ld0, row_base, row_end, n);
    }
#pragma unroll
    for (int j = 0; j < 16; ++j) out[j] = pack_bf16(__uint_as_float(v[2 * j]), __uint_as_float(v[2 * j + 1]));
    warp_store_rows64(stage, lane, out, p.out1, p.ld1, row_base, row_end, n);
  }
  return true;
}

// The forward activation epilogue of one warp, laid out like dact_columns: z = acc (+ bias) unless p.out0 is null,
// y1 = act(z) (gated: act(even) * odd; two chunks make one 64-byte segment of y1, N is a multiple of 128).
template <int FN, bool GATED, int CHUNKS, class Release>
__device__ __forceinline__ void act_columns(const GemmParams& p, int expert, uint32_t stage, int lane, int row_base,
                                            int row_end, int n_first, uint32_t t_addr, Release&& release_acc) {
  if (n_first >= p.N) release_acc();
  uint32_t first_half[8];
#pragma unroll 1
  for (int c = 0; c < CHUNKS; ++c) {
    const int n = n_first + 32 * c;
    if (n >= p.N) break;
    uint32_t v[32], out[16];
    tmem_ld32(t_addr + 32 * c, v);
    tmem_ld_wait();
    if (c + 1 == CHUNKS || n + 32 >= p.N) release_acc();
    float f[32];
    load_biased(p, expert, n, v, f);
    if (p.out0 != nullptr) {
#pragma unroll
      for (int j = 0; j < 16; ++j) out[j] = pack_bf16(f[2 * j], f[2 * j + 1]);
      warp_store_rows64(stage, lane, out, p.out0, p.ld0, row_base, row_end, n);
    }
    if constexpr (GATED) {
#pragma unroll
      for (int j = 0; j < 16; ++j) {
        float a, da;
        act_value_grad<FN>(f[2 * j], a, da);
        f[j] = a * f[2 * j + 1];
      }
      if ((c & 1) == 0) {
#pragma unroll
        for (int j = 0; j < 8; ++j) first_half[j] = pack_bf16(f[2 * j], f[2 * j + 1]);
      } else {
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          out[j] = first_half[j];
          out[8 + j] = pack_bf16(f[2 * j], f[2 * j + 1]);
        }
        warp_store_rows64(stage, lane, out, p.out1, p.ld1, row_base, row_end, (n - 32) >> 1);
      }
    } else {
#pragma unroll
      for (int j = 0; j < 16; ++j) {
        float a0, a1, da;
        act_value_grad<FN>(f[2 * j], a0, da);
        act_value_grad<FN>(f[2 * j + 1], a1, da);
        out[j] = pack_bf16(a0, a1);
      }
      warp_store_rows64(stage, lane, out, p.out1, p.ld1, row_base, row_end, n);
    }
  }
}

// One 32-column piece of a warp's 32 accumulator rows for the epilogues that store it as it is: v[j] = acc[r, n + j] of
// lane l's row r = row_base + l (ragged-K: the output row inside the expert's matrix).  Every lane must call.
// `dst_row`: EPI_STORE_ROWS, the lane's source row.
template <int EPI, bool RAGGED_K>
__device__ __forceinline__ void store_chunk(const GemmParams& p, int expert, uint32_t stage, int lane, int row_base,
                                            int row_end, int n, const uint32_t (&v)[32], float score, int dst_row) {
  if constexpr (EPI == EPI_SCATTER) {
    if (row_base + lane < row_end) {
      float* dst = p.acc_out + static_cast<long long>(dst_row) * p.N + n;
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(dst + 4 * j),
                     "f"(score * __uint_as_float(v[4 * j + 0])), "f"(score * __uint_as_float(v[4 * j + 1])),
                     "f"(score * __uint_as_float(v[4 * j + 2])), "f"(score * __uint_as_float(v[4 * j + 3]))
                     : "memory");
      }
    }
    __syncwarp();  // the next piece's tensor-memory read is warp-wide
  } else {
    float f[32];
    if constexpr (EPI == EPI_STORE_BIAS) {
      load_biased(p, expert, n, v, f);
    } else {
#pragma unroll
      for (int j = 0; j < 32; ++j) f[j] = __uint_as_float(v[j]);
    }
    if constexpr (EPI == EPI_STORE_ROWS) {
      if (p.scores != nullptr) {
#pragma unroll
        for (int j = 0; j < 32; ++j) f[j] = score * __bfloat162float(__float2bfloat16_rn(f[j]));
      }
    }
    uint32_t w[16];
#pragma unroll
    for (int j = 0; j < 16; ++j) w[j] = pack_bf16(f[2 * j], f[2 * j + 1]);
    if constexpr (EPI == EPI_STORE_ROWS) {
      warp_store_segments64(stage, lane, w, p.accumulate, [&](int rr) {
        const int row = __shfl_sync(0xffffffffu, dst_row, rr);
        return row_base + rr < row_end ? p.out0 + row * p.ld0 + n : nullptr;
      });
    } else {
      warp_store_rows64(stage, lane, w, p.out0 + (RAGGED_K ? expert * p.out0_expert_stride : 0ll), p.ld0, row_base,
                               row_end, n, EPI == EPI_STORE && p.accumulate);
    }
  }
}

}  // namespace smoe

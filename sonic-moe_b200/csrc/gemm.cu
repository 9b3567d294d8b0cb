// Host side of the grouped GEMMs: tensor-map construction and the C-ABI launchers.
#include "gemm_pair.cuh"
#include "gemm_skinny.cuh"
#include "internal.h"

#include <cstdlib>
#include <mutex>

#include "../../include/sonicmoe_b200.h"

namespace smoe {

using pair::BK;
using pair::BM;
using pair::BN;
using pair::MAX_EXPERTS;
static_assert(MAX_EXPERTS == kMaxExperts, "checked by the compound entry points");

// cuTensorMapEncodeTiled is fetched through the runtime so that the library links against cudart
// only and still loads on a machine without a driver.
using EncodeTiledFn = CUresult (*)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                   const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                   CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

static EncodeTiledFn get_encode_fn() {
  static EncodeTiledFn fn = nullptr;
  static std::once_flag once;
  std::call_once(once, [] {
    void* ptr = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &ptr, cudaEnableDefault, &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess) {
      fn = reinterpret_cast<EncodeTiledFn>(ptr);
    }
  });
  return fn;
}

// bf16 row-major 2D tensor (rows, cols) with a row pitch in elements; box = (box_rows, box_cols),
// 128-byte swizzle, out-of-bounds elements read as zero.
static int encode_2d(CUtensorMap* map, const void* base, uint64_t rows, uint64_t cols, uint64_t pitch_elems,
                     uint32_t box_rows, uint32_t box_cols) {
  EncodeTiledFn fn = get_encode_fn();
  if (fn == nullptr) return SMOE_ERR_DRIVER;
  // The encoder is a driver-API call and needs the device's primary context current on the calling
  // thread; a thread that has made no runtime call yet (an autograd worker) has none.  A no-op runtime
  // call binds it.
  static thread_local bool context_bound = false;
  if (!context_bound) {
    if (cudaFree(nullptr) != cudaSuccess) return SMOE_ERR_DRIVER;
    context_bound = true;
  }
  if ((reinterpret_cast<uintptr_t>(base) & 15u) != 0 || (pitch_elems * 2) % 16 != 0) return SMOE_ERR_ALIGNMENT;
  const cuuint64_t dims[2] = {cols, rows};
  const cuuint64_t strides[1] = {pitch_elems * 2};
  const cuuint32_t box[2] = {box_cols, box_rows};
  const cuuint32_t estr[2] = {1, 1};
  const CUresult r = fn(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(base), dims, strides, box, estr,
                        CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                        CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS ? SMOE_OK : SMOE_ERR_TENSORMAP;
}

// Kernels with a gathered operand work on two tiles per gathered stage (256 x 512 or 512 x 256 units) unless
// SMOE_DUAL=0 (kept for the test that compares the two forms).
static bool use_dual_tiles() {
  static const bool v = [] {
    const char* e = getenv("SMOE_DUAL");
    return !(e != nullptr && e[0] == '0');
  }();
  return v;
}

// What two tiles per gathered tile save, the rest costs: their accumulators do not alternate between units, so each unit's
// hand-over is exposed, and there are half as many units to share out.  Both sides alternating, whole training steps (single /
// dual):
//   * up projection: reductions up to 2048 go faster as single tiles (T 24576, H 1536, I 256, E 128, K 8 1907 / 1929 us, T 8197,
//     H 2048, I 1024, E 64, K 1 780 / 793, T 8000, H 1536, I 512, E 64, K 4 665 / 677; the kernel alone, H 2048, I 1024, E 64: 128 rows
//     per expert 148 / 177 us, 512 301 / 343, 4096 1730 / 2061; H 1024 and 1536 like it at every load), longer ones do not (H
//     4096, I 1024, E 128, inference of 8192 tokens 1928 / 1883, step of 2080 2719 / 2701; H 3072 the same either way);
//   * weight gradients: their reduction is an expert's rows, and the line lies between a mean of 384 and 500 (dW1, H 1536, I
//     512, E 64, K 4: 256 rows 73 / 91 us, 384 94 / 101, 500 117 / 116; 512 rows, H 4096, I 1024, E 128: 1337 / 1101).  The kernel
//     alone is up to a tenth faster as dual tiles from 384 rows on with even loads (H 4096, I 1024, E 32, 448 rows 236 / 216) and
//     a tenth slower with skewed ones (H 1536, I 512, E 64, 448 rows 151 / 165).
// Never where the doubled dimension is so far from a multiple of 512 that the half-empty last unit wastes more than an eighth of
// the MMA work (e.g. N = 768).
static bool dual_tiles(int doubled, bool pays) {
  return use_dual_tiles() && pays && ((doubled + 511) / 512 * 512 - doubled) * 8 <= doubled;
}
static bool dual_reduction(int K) { return K > 2048; }
static bool dual_rows(long long total_rows, int E) { return total_rows >= 480ll * E; }

template <bool RAGGED_K, bool A_GATHER, bool A_MN, bool B_GATHER, bool B_MN, int EPI, int GW,
          int DUAL = pair::DUAL_NONE>
static int launch_variant(const CUtensorMap& tmA, const CUtensorMap& tmB, const GemmParams& p, cudaStream_t stream) {
  auto kernel = pair::grouped_gemm_pair_kernel<RAGGED_K, A_GATHER, A_MN, B_GATHER, B_MN, EPI, GW, DUAL>;
  constexpr bool kSplit = pair::splits_registers(EPI, DUAL);
  static PerDeviceFlag configured;
  const int dev = current_device();
  if (dev < 0) return SMOE_ERR_DRIVER;
  if (!configured.test(dev)) {
    if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, pair::SMEM_BYTES) != cudaSuccess)
      return SMOE_ERR_LAUNCH;
    if (kSplit) {
      // the kernel re-partitions registers between its warpgroups (setmaxnreg 56 / 200 around 128): that only
      // balances if it was compiled to exactly 128 registers per thread -- refuse to launch otherwise
      cudaFuncAttributes fa;
      if (cudaFuncGetAttributes(&fa, kernel) != cudaSuccess || fa.numRegs != 128) return SMOE_ERR_LAUNCH;
    }
    configured.set(dev);
  }
  const int sms = num_sms();
  if (sms < 2) return SMOE_ERR_DRIVER;
  return launched(launch_chained(kernel, dim3(static_cast<unsigned>(sms & ~1)), pair::threads(GW, kSplit),
                                 pair::SMEM_BYTES, stream, 2, tmA, tmB, p));
}

// Kernels without a gathered operand work on single tiles, kernels with one on dual tiles where they pay.
template <bool RAGGED_K, bool A_GATHER, bool A_MN, bool B_GATHER, bool B_MN, int EPI>
static int launch(const CUtensorMap& tmA, const CUtensorMap& tmB, const GemmParams& p, cudaStream_t stream) {
  constexpr bool kGather = A_GATHER || B_GATHER;
  if constexpr (!kGather) {
    return launch_variant<RAGGED_K, A_GATHER, A_MN, B_GATHER, B_MN, EPI, 0>(tmA, tmB, p, stream);
  } else {
    // The activation-gradient epilogues keep single tiles: with both accumulators belonging to one unit the next
    // unit's second MMA group waits for the first accumulator's dSwiGLU pass.  Measured with four epilogue warps in the
    // single form, T 32768, H 4096, I 1024, E 128, K 8: the kernel alone 2.26-2.69 ms dual against 2.09-2.58 single.  Eight
    // warps made the single form 3 % faster since (2.59 -> 2.51 ms, alternating).  The general forward epilogue is too long
    // to be worked off from registers, and must not hold accumulators that the next unit needs.
    if constexpr (EPI != EPI_DSWIGLU && epi_base(EPI) != EPI_DACT && epi_base(EPI) != EPI_ACT) {
      if (dual_tiles(A_GATHER ? p.N : p.M, RAGGED_K ? dual_rows(p.total_rows, p.E) : dual_reduction(p.K))) {
        constexpr int kDual = A_GATHER ? pair::DUAL_N : pair::DUAL_M;
        return launch_variant<RAGGED_K, A_GATHER, A_MN, B_GATHER, B_MN, EPI, 4, kDual>(tmA, tmB, p, stream);
      }
    }
    // plain stores leave registers for eight gather warps (four: dW2 at H 1536, I 256, 1536 rows per expert 206 us, eight 175)
    constexpr int kGatherWarps = EPI == EPI_STORE ? 8 : 4;
    return launch_variant<RAGGED_K, A_GATHER, A_MN, B_GATHER, B_MN, EPI, kGatherWarps>(tmA, tmB, p, stream);
  }
}

// The kernel of a general epilogue (gathered rows, weights K-major or MN-major) compiled for this activation.
template <bool B_MN, int EPI>
static int launch_activation(const CUtensorMap& tmA, const CUtensorMap& tmB, const GemmParams& p, int activation,
                             cudaStream_t stream) {
  switch (activation) {
    case ACT_SWIGLU: return launch<false, true, false, false, B_MN, EPI + 16 * ACT_SWIGLU>(tmA, tmB, p, stream);
    case ACT_GEGLU: return launch<false, true, false, false, B_MN, EPI + 16 * ACT_GEGLU>(tmA, tmB, p, stream);
    case ACT_REGLU: return launch<false, true, false, false, B_MN, EPI + 16 * ACT_REGLU>(tmA, tmB, p, stream);
    case ACT_RELU_SQ: return launch<false, true, false, false, B_MN, EPI + 16 * ACT_RELU_SQ>(tmA, tmB, p, stream);
    case ACT_RELU: return launch<false, true, false, false, B_MN, EPI + 16 * ACT_RELU>(tmA, tmB, p, stream);
    case ACT_GELU: return launch<false, true, false, false, B_MN, EPI + 16 * ACT_GELU>(tmA, tmB, p, stream);
    case ACT_SILU: return launch<false, true, false, false, B_MN, EPI + 16 * ACT_SILU>(tmA, tmB, p, stream);
  }
  return SMOE_ERR_SHAPE;
}

// How a forward projection is shared between the kernel for experts with few rows (gemm_skinny.cuh) and the 256 x 256 tiles.
// The host knows the mean number of rows per expert and not the load, so the choice has to hold for an even load and for one
// in which all tokens take the same experts.  Measured inside inference layers in a row, us, to the start of the next kernel.
//   * Rows per unit by the mean: an even load costs least with the smallest unit that holds most experts' rows (more stages of
//     weights in flight).  H 4096, I 1024, E 128, units of 32 / 64 / 128 rows / tiles, up projection: mean 4 318, 324, 336,
//     350; mean 16 329, 332, 343, 361; mean 24 367, 346, 354, 364; down projection at mean 4 162, 164, 171, 193.
//   * An expert with more rows than a unit has its weights streamed again by every further unit, so a load in few experts
//     costs one pass per wave of units, where the tiles need about one.  One launch therefore takes all experts only where even
//     all rows in the fewest units give no more than two per SM, if need be with units of twice the rows: 2048 rows in 8 of
//     256 experts, H 4096, I 1024, up projection 184 with units of 32 rows, 109 with 64, 64 with 128 and 54 by tiles.
//   * Beyond that experts with more than two units' rows go to the tiles in a second launch, which finds nothing to do in an
//     even load: 60 for the load above, and even 645 where units alone take 635 and tiles 714.  Layers whose weights do not
//     outweigh that launch (6 to 9 us: half a GB) take larger units still, or the tiles: H 1536, I 256, E 128, 8192 rows,
//     divided / units of 128 / tiles, up 55, 49, 51.
struct FewRows {
  int unit = 0;      // rows per unit; 0: the tiles take all experts
  int max_rows = 0;  // experts with more rows are left to the tiles
};
static FewRows few_rows(const GemmParams& p) {
  FewRows f;
  const double mean = static_cast<double>(p.total_rows) / p.E;
  if (mean > 96) return f;
  const int by_mean = mean <= 12 ? 32 : mean <= 40 ? 64 : skinny::MAX_NT;
  const bool divide = 2.0 * p.E * p.N * p.K >= 0.5e9;
  const int largest = divide && 2 * by_mean < skinny::MAX_NT ? 2 * by_mean : skinny::MAX_NT;
  const long long blocks = (p.N + skinny::BM - 1) / skinny::BM, most = 2ll * num_sms();
  for (f.unit = by_mean; f.unit <= largest; f.unit *= 2) {
    if ((p.total_rows + f.unit - 1) / f.unit * blocks <= most) {
      f.max_rows = p.total_rows;
      return f;
    }
  }
  f.unit = divide ? by_mean : 0;
  f.max_rows = 2 * by_mean;
  return f;
}

template <bool GATHER, bool SWIGLU>
static int launch_skinny(const CUtensorMap& tmW, const CUtensorMap& tmX, const GemmParams& p, int nt, cudaStream_t stream) {
  auto kernel = skinny::skinny_gemm_kernel<GATHER, SWIGLU>;
  static PerDeviceFlag configured;
  const int dev = current_device();
  if (dev < 0) return SMOE_ERR_DRIVER;
  if (!configured.test(dev)) {
    if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024) != cudaSuccess)
      return SMOE_ERR_LAUNCH;
    configured.set(dev);
  }
  const int sms = num_sms();
  if (sms <= 0) return SMOE_ERR_DRIVER;
  const int stages = skinny::num_stages(nt);
  return launched(launch_chained(kernel, dim3(static_cast<unsigned>(sms)), skinny::threads(GATHER),
                                 skinny::smem_bytes(nt, stages), stream, 1, tmW, tmX, p, nt, stages));
}

// An empty batch (T == 0, hence TK == 0) is valid: the entry points return at once (weight-gradient entry points
// after zero-filling their output).  What is refused: negative sizes, or routed rows without any token.
static bool bad_tokens(int T, int TK) { return T < 0 || TK < 0 || (T == 0 && TK > 0); }

static bool bad_shape(int H, int I, int E) {
  return H <= 0 || I <= 0 || E <= 0 || E > MAX_EXPERTS || (H % 64) != 0 || (I % 64) != 0;
}

}  // namespace smoe

using namespace smoe;

#define SMOE_TRY(expr)              \
  do {                              \
    const int _rc = (expr);         \
    if (_rc != SMOE_OK) return _rc; \
  } while (0)

extern "C" {

int smoe_up_projection_forward(const void* x, const void* w1, void* z, void* y1, const int* expert_offset,
                               const int* x_gather_idx, int T, int H, int I, int E, int TK, int* status,
                               void* stream) {
  if (bad_shape(H, I, E) || bad_tokens(T, TK)) return SMOE_ERR_SHAPE;
  if (TK == 0) return SMOE_OK;
  CUtensorMap tmA, tmB;
  SMOE_TRY(encode_2d(&tmA, x, T, H, H, 1, BK));                        // gather4 rows of x
  SMOE_TRY(encode_2d(&tmB, w1, (uint64_t)E * 2 * I, H, H, pair::BN_CTA, BK));    // W1[e] rows = output features, K-major
  static_assert(pair::BN_CTA == skinny::BM, "one weight map for both kernels");
  GemmParams p = {};
  p.E = E; p.N = 2 * I; p.K = H; p.total_rows = TK; p.gather_rows = T; p.b_rows_per_expert = 2 * I;
  p.off = expert_offset; p.gather = x_gather_idx;
  p.out0 = static_cast<__nv_bfloat16*>(z); p.ld0 = 2 * I;
  p.out1 = static_cast<__nv_bfloat16*>(y1); p.ld1 = I;
  p.status = status;
  const FewRows few = few_rows(p);
  if (few.unit > 0) {
    p.max_rows = p.min_rows = few.max_rows;
    SMOE_TRY((launch_skinny<true, true>(tmB, tmA, p, few.unit, static_cast<cudaStream_t>(stream))));
    if (few.max_rows >= TK) return SMOE_OK;
  }
  return launch<false, true, false, false, false, EPI_SWIGLU>(tmA, tmB, p, static_cast<cudaStream_t>(stream));
}

int smoe_down_projection_forward(const void* y1, const void* w2, void* y2, const int* expert_offset, int H, int I,
                                 int E, int TK, int* status, void* stream) {
  if (bad_shape(H, I, E) || TK < 0) return SMOE_ERR_SHAPE;
  if (TK == 0) return SMOE_OK;
  CUtensorMap tmA, tmB;
  SMOE_TRY(encode_2d(&tmA, y1, TK, I, I, BM, BK));
  SMOE_TRY(encode_2d(&tmB, w2, (uint64_t)E * H, I, I, pair::BN_CTA, BK));        // W2[e] is (H, I): K-major
  GemmParams p = {};
  p.E = E; p.N = H; p.K = I; p.total_rows = TK; p.b_rows_per_expert = H;
  p.off = expert_offset;
  p.out0 = static_cast<__nv_bfloat16*>(y2); p.ld0 = H;
  p.status = status;
  const FewRows few = few_rows(p);
  if (few.unit > 0) {
    CUtensorMap tmX;
    SMOE_TRY(encode_2d(&tmX, y1, TK, I, I, skinny::BOX_ROWS, BK));
    p.max_rows = p.min_rows = few.max_rows;
    SMOE_TRY((launch_skinny<false, false>(tmB, tmX, p, few.unit, static_cast<cudaStream_t>(stream))));
    if (few.max_rows >= TK) return SMOE_OK;
  }
  return launch<false, false, false, false, false, EPI_STORE>(tmA, tmB, p, static_cast<cudaStream_t>(stream));
}

int smoe_down_projection_forward_rows(const void* y1, const void* w2, void* o, const void* scores, int scores_are_bf16,
                                      const int* expert_offset, const int* x_gather_idx, const int* s_scatter_idx,
                                      int H, int I, int E, int TK, int* status, void* stream) {
  if (bad_shape(H, I, E) || TK < 0) return SMOE_ERR_SHAPE;
  if (TK == 0) return SMOE_OK;
  if (x_gather_idx == nullptr || (scores != nullptr && s_scatter_idx == nullptr)) return SMOE_ERR_SHAPE;
  CUtensorMap tmA, tmB;
  SMOE_TRY(encode_2d(&tmA, y1, TK, I, I, BM, BK));
  SMOE_TRY(encode_2d(&tmB, w2, (uint64_t)E * H, I, I, pair::BN_CTA, BK));
  GemmParams p = {};
  p.E = E; p.N = H; p.K = I; p.total_rows = TK; p.b_rows_per_expert = H;
  p.off = expert_offset; p.gather = x_gather_idx; p.s_scatter = s_scatter_idx;
  p.scores = scores; p.scores_are_bf16 = scores_are_bf16;
  p.out0 = static_cast<__nv_bfloat16*>(o); p.ld0 = H;
  p.status = status;
  return launch<false, false, false, false, false, EPI_STORE_ROWS>(tmA, tmB, p, static_cast<cudaStream_t>(stream));
}

int smoe_down_projection_forward_scatter(const void* y1, const void* w2, float* o_acc, const void* scores,
                                         int scores_are_bf16, const int* expert_offset, const int* x_gather_idx,
                                         const int* s_scatter_idx, int T, int H, int I, int E, int TK, int* status,
                                         void* stream) {
  if (bad_shape(H, I, E) || bad_tokens(T, TK)) return SMOE_ERR_SHAPE;
  if (TK == 0) return SMOE_OK;
  CUtensorMap tmA, tmB;
  SMOE_TRY(encode_2d(&tmA, y1, TK, I, I, BM, BK));
  SMOE_TRY(encode_2d(&tmB, w2, (uint64_t)E * H, I, I, pair::BN_CTA, BK));
  GemmParams p = {};
  p.E = E; p.N = H; p.K = I; p.total_rows = TK; p.gather_rows = T; p.b_rows_per_expert = H;
  p.off = expert_offset; p.gather = x_gather_idx; p.s_scatter = s_scatter_idx;
  p.scores = scores; p.scores_are_bf16 = scores_are_bf16; p.acc_out = o_acc;
  p.status = status;
  return launch<false, false, false, false, false, EPI_SCATTER>(tmA, tmB, p, static_cast<cudaStream_t>(stream));
}

int smoe_down_projection_backward_act(const void* dout, const void* w2, const void* z, const void* scores,
                                      int scores_are_bf16, void* dz, void* y1s, float* ds_partial,
                                      const int* expert_offset, const int* x_gather_idx, const int* s_scatter_idx,
                                      int T, int H, int I, int E, int TK, int* status, void* stream) {
  if (bad_shape(H, I, E) || bad_tokens(T, TK)) return SMOE_ERR_SHAPE;
  if (TK == 0) return SMOE_OK;
  CUtensorMap tmA, tmB;
  SMOE_TRY(encode_2d(&tmA, dout, T, H, H, 1, BK));                     // gather4 rows of dout
  SMOE_TRY(encode_2d(&tmB, w2, (uint64_t)E * H, I, I, BK, 64));        // W2[e] (H, I): rows are k, MN-major
  GemmParams p = {};
  p.E = E; p.N = I; p.K = H; p.total_rows = TK; p.gather_rows = T; p.b_rows_per_expert = H;
  p.off = expert_offset; p.gather = x_gather_idx; p.s_scatter = s_scatter_idx;
  p.out0 = static_cast<__nv_bfloat16*>(dz); p.ld0 = 2 * I;
  p.out1 = static_cast<__nv_bfloat16*>(y1s); p.ld1 = I;
  p.z = static_cast<const __nv_bfloat16*>(z);
  p.scores = scores; p.scores_are_bf16 = scores_are_bf16; p.ds_partial = ds_partial;
  p.status = status;
  return launch<false, true, false, false, true, EPI_DSWIGLU>(tmA, tmB, p, static_cast<cudaStream_t>(stream));
}

// ---- general activations and biases ---------------------------------------------
// Biases are read in 16-byte pieces; unlike the tensor maps' operands nothing else looks at their address.
static bool bad_bias(const void* b) { return (reinterpret_cast<uintptr_t>(b) & 15u) != 0; }

static bool bad_activation(int a) { return a < ACT_SWIGLU || a > ACT_SILU; }

int smoe_up_projection_forward_act(const void* x, const void* w1, const void* b1, void* z, void* y1,
                                   const int* expert_offset, const int* x_gather_idx, int T, int H, int N1, int E,
                                   int TK, int activation, int* status, void* stream) {
  if (bad_activation(activation) || H <= 0 || (H % 64) != 0 || N1 <= 0 || (N1 % 128) != 0 || E <= 0 ||
      E > MAX_EXPERTS || bad_tokens(T, TK))
    return SMOE_ERR_SHAPE;
  if (TK == 0) return SMOE_OK;
  if (bad_bias(b1)) return SMOE_ERR_ALIGNMENT;
  CUtensorMap tmA, tmB;
  SMOE_TRY(encode_2d(&tmA, x, T, H, H, 1, BK));
  SMOE_TRY(encode_2d(&tmB, w1, (uint64_t)E * N1, H, H, pair::BN_CTA, BK));
  GemmParams p = {};
  p.E = E; p.N = N1; p.K = H; p.total_rows = TK; p.gather_rows = T; p.b_rows_per_expert = N1;
  p.off = expert_offset; p.gather = x_gather_idx;
  p.out0 = static_cast<__nv_bfloat16*>(z); p.ld0 = N1;
  p.out1 = static_cast<__nv_bfloat16*>(y1); p.ld1 = act_is_gated(activation) ? N1 / 2 : N1;
  p.bias = static_cast<const __nv_bfloat16*>(b1);
  p.status = status;
  return launch_activation<false, EPI_ACT>(tmA, tmB, p, activation, static_cast<cudaStream_t>(stream));
}

int smoe_down_projection_forward_bias(const void* y1, const void* w2, const void* b2, void* y2,
                                      const int* expert_offset, int H, int I, int E, int TK, int* status,
                                      void* stream) {
  if (bad_shape(H, I, E) || TK < 0) return SMOE_ERR_SHAPE;
  if (TK == 0) return SMOE_OK;
  if (bad_bias(b2)) return SMOE_ERR_ALIGNMENT;
  CUtensorMap tmA, tmB;
  SMOE_TRY(encode_2d(&tmA, y1, TK, I, I, BM, BK));
  SMOE_TRY(encode_2d(&tmB, w2, (uint64_t)E * H, I, I, pair::BN_CTA, BK));
  GemmParams p = {};
  p.E = E; p.N = H; p.K = I; p.total_rows = TK; p.b_rows_per_expert = H;
  p.off = expert_offset;
  p.out0 = static_cast<__nv_bfloat16*>(y2); p.ld0 = H;
  p.bias = static_cast<const __nv_bfloat16*>(b2);
  p.status = status;
  return launch<false, false, false, false, false, EPI_STORE_BIAS>(tmA, tmB, p,
                                                                        static_cast<cudaStream_t>(stream));
}

int smoe_down_projection_backward_dact(const void* dout, const void* w2, const void* z, const void* scores,
                                       int scores_are_bf16, void* dz, void* y1s, float* ds_partial,
                                       const int* expert_offset, const int* x_gather_idx, const int* s_scatter_idx,
                                       int T, int H, int I, int E, int TK, int activation, int* status,
                                       void* stream) {
  if (bad_activation(activation) || bad_shape(H, I, E) || bad_tokens(T, TK)) return SMOE_ERR_SHAPE;
  if (TK == 0) return SMOE_OK;
  CUtensorMap tmA, tmB;
  SMOE_TRY(encode_2d(&tmA, dout, T, H, H, 1, BK));
  SMOE_TRY(encode_2d(&tmB, w2, (uint64_t)E * H, I, I, BK, 64));
  const int n1 = act_is_gated(activation) ? 2 * I : I;
  GemmParams p = {};
  p.E = E; p.N = I; p.K = H; p.total_rows = TK; p.gather_rows = T; p.b_rows_per_expert = H;
  p.off = expert_offset; p.gather = x_gather_idx; p.s_scatter = s_scatter_idx;
  p.out0 = static_cast<__nv_bfloat16*>(dz); p.ld0 = n1;
  p.out1 = static_cast<__nv_bfloat16*>(y1s); p.ld1 = I;
  p.z = static_cast<const __nv_bfloat16*>(z);
  p.scores = scores; p.scores_are_bf16 = scores_are_bf16; p.ds_partial = ds_partial;
  p.status = status;
  return launch_activation<true, EPI_DACT>(tmA, tmB, p, activation, static_cast<cudaStream_t>(stream));
}

int smoe_ds_partial_columns(int I) { return 2 * ((I + BN - 1) / BN); }

int smoe_up_projection_backward_dx(const void* dz, const void* w1, void* dx_expanded, const int* expert_offset, int H,
                                   int I, int E, int TK, int* status, void* stream) {
  if (bad_shape(H, I, E) || TK < 0) return SMOE_ERR_SHAPE;
  if (TK == 0) return SMOE_OK;
  CUtensorMap tmA, tmB;
  SMOE_TRY(encode_2d(&tmA, dz, TK, 2 * I, 2 * I, BM, BK));
  SMOE_TRY(encode_2d(&tmB, w1, (uint64_t)E * 2 * I, H, H, BK, 64));    // W1[e] (2I, H): rows are k, MN-major
  GemmParams p = {};
  p.E = E; p.N = H; p.K = 2 * I; p.total_rows = TK; p.b_rows_per_expert = 2 * I;
  p.off = expert_offset;
  p.out0 = static_cast<__nv_bfloat16*>(dx_expanded); p.ld0 = H;
  p.status = status;
  return launch<false, false, false, false, true, EPI_STORE>(tmA, tmB, p, static_cast<cudaStream_t>(stream));
}

static int backward_dx_rows(const void* dz, const void* w1, void* dx, const int* expert_offset, const int* x_gather_idx,
                            int H, int I, int E, int TK, int* status, void* stream, int accumulate) {
  if (bad_shape(H, I, E) || TK < 0) return SMOE_ERR_SHAPE;
  if (TK == 0) return SMOE_OK;
  if (x_gather_idx == nullptr) return SMOE_ERR_SHAPE;
  CUtensorMap tmA, tmB;
  SMOE_TRY(encode_2d(&tmA, dz, TK, 2 * I, 2 * I, BM, BK));
  SMOE_TRY(encode_2d(&tmB, w1, (uint64_t)E * 2 * I, H, H, BK, 64));    // W1[e] (2I, H): rows are k, MN-major
  GemmParams p = {};
  p.E = E; p.N = H; p.K = 2 * I; p.total_rows = TK; p.b_rows_per_expert = 2 * I;
  p.off = expert_offset; p.gather = x_gather_idx;
  p.out0 = static_cast<__nv_bfloat16*>(dx); p.ld0 = H;
  p.status = status; p.accumulate = accumulate;
  return launch<false, false, false, false, true, EPI_STORE_ROWS>(tmA, tmB, p, static_cast<cudaStream_t>(stream));
}

int smoe_up_projection_backward_dx_rows(const void* dz, const void* w1, void* dx, const int* expert_offset,
                                        const int* x_gather_idx, int H, int I, int E, int TK, int* status,
                                        void* stream) {
  return backward_dx_rows(dz, w1, dx, expert_offset, x_gather_idx, H, I, E, TK, status, stream, 0);
}

static int down_weight_grad(const void* dout, const void* y1s, void* dw2, const int* expert_offset,
                            const int* x_gather_idx, int T, int H, int I, int E, int TK, int* status, void* stream,
                            int accumulate) {
  if (bad_shape(H, I, E) || bad_tokens(T, TK)) return SMOE_ERR_SHAPE;
  if (TK == 0) {
    if (accumulate) return SMOE_OK;
    return cudaMemsetAsync(dw2, 0, (size_t)E * H * I * 2, static_cast<cudaStream_t>(stream)) == cudaSuccess
               ? SMOE_OK : SMOE_ERR_LAUNCH;
  }
  CUtensorMap tmA, tmB;
  SMOE_TRY(encode_2d(&tmA, dout, T, H, H, 1, 64));                     // A[h, t] = dout[gather[t], h]
  SMOE_TRY(encode_2d(&tmB, y1s, TK, I, I, BK, 64));                    // B[i, t] = y1s[t, i]
  GemmParams p = {};
  p.E = E; p.M = H; p.N = I; p.total_rows = TK; p.gather_rows = T;
  p.off = expert_offset; p.gather = x_gather_idx;
  p.out0 = static_cast<__nv_bfloat16*>(dw2); p.ld0 = I; p.out0_expert_stride = (long long)H * I;
  p.status = status; p.accumulate = accumulate;
  return launch<true, true, true, false, true, EPI_STORE>(tmA, tmB, p, static_cast<cudaStream_t>(stream));
}

static int up_weight_grad(const void* x, const void* dz, void* dw1, const int* expert_offset, const int* x_gather_idx,
                          int T, int H, int I, int E, int TK, int* status, void* stream, int accumulate) {
  if (bad_shape(H, I, E) || bad_tokens(T, TK)) return SMOE_ERR_SHAPE;
  if (TK == 0) {
    if (accumulate) return SMOE_OK;
    return cudaMemsetAsync(dw1, 0, (size_t)E * 2 * I * H * 2, static_cast<cudaStream_t>(stream)) == cudaSuccess
               ? SMOE_OK : SMOE_ERR_LAUNCH;
  }
  CUtensorMap tmA, tmB;
  SMOE_TRY(encode_2d(&tmA, dz, TK, 2 * I, 2 * I, BK, 64));             // A[j, t] = dz[t, j]
  SMOE_TRY(encode_2d(&tmB, x, T, H, H, 1, 64));                        // B[h, t] = x[gather[t], h]
  GemmParams p = {};
  p.E = E; p.M = 2 * I; p.N = H; p.total_rows = TK; p.gather_rows = T;
  p.off = expert_offset; p.gather = x_gather_idx;
  p.out0 = static_cast<__nv_bfloat16*>(dw1); p.ld0 = H; p.out0_expert_stride = (long long)2 * I * H;
  p.status = status; p.accumulate = accumulate;
  return launch<true, false, true, true, true, EPI_STORE>(tmA, tmB, p, static_cast<cudaStream_t>(stream));
}

int smoe_dual_tiles(int gemm, int H, int I, int E, int TK) {
  switch (gemm) {
    case SMOE_GEMM_UP: return dual_tiles(2 * I, dual_reduction(H));
    case SMOE_GEMM_DW1: return dual_tiles(2 * I, dual_rows(TK, E));
    case SMOE_GEMM_DW2: return dual_tiles(I, dual_rows(TK, E));
    default: return 0;
  }
}

int smoe_down_projection_weight_grad(const void* dout, const void* y1s, void* dw2, const int* expert_offset,
                                     const int* x_gather_idx, int T, int H, int I, int E, int TK, int* status,
                                     void* stream) {
  return down_weight_grad(dout, y1s, dw2, expert_offset, x_gather_idx, T, H, I, E, TK, status, stream, 0);
}

int smoe_down_projection_weight_grad_accumulate(const void* dout, const void* y1s, void* dw2,
                                                const int* expert_offset, const int* x_gather_idx, int T, int H, int I,
                                                int E, int TK, int* status, void* stream) {
  return down_weight_grad(dout, y1s, dw2, expert_offset, x_gather_idx, T, H, I, E, TK, status, stream, 1);
}

int smoe_up_projection_weight_grad(const void* x, const void* dz, void* dw1, const int* expert_offset,
                                   const int* x_gather_idx, int T, int H, int I, int E, int TK, int* status,
                                   void* stream) {
  return up_weight_grad(x, dz, dw1, expert_offset, x_gather_idx, T, H, I, E, TK, status, stream, 0);
}

int smoe_up_projection_weight_grad_accumulate(const void* x, const void* dz, void* dw1, const int* expert_offset,
                                              const int* x_gather_idx, int T, int H, int I, int E, int TK, int* status,
                                              void* stream) {
  return up_weight_grad(x, dz, dw1, expert_offset, x_gather_idx, T, H, I, E, TK, status, stream, 1);
}

}  // extern "C"

int smoe::up_projection_backward_dx_rows_add(const void* dz, const void* w1, void* dx, const int* expert_offset,
                                             const int* x_gather_idx, int H, int I, int E, int TK, int* status,
                                             void* stream) {
  return backward_dx_rows(dz, w1, dx, expert_offset, x_gather_idx, H, I, E, TK, status, stream, 1);
}

// The layer's passes as a few entry points each: the same launches as the separate ones, without a trip through the
// caller's language for each.  A layer call of a few tokens is shorter on the device (60 us for one token of a 64-expert
// layer) than eight launches with their allocations and argument conversions take from Python, and so is a training step of
// 2048 tokens of a small layer (140 us of kernels, 600 us of host work in four autograd nodes and 17 calls).
#include <cuda_runtime.h>
#include <stddef.h>
#include <stdint.h>

#include <initializer_list>

#include "../../include/sonicmoe_b200.h"
#include "epilogue.cuh"
#include "internal.h"

namespace {

// Scratch of a call, in 256-byte aligned pieces.
struct Scratch {
  size_t scores, indices, aux_grad, off, idx3, y1, y2, route_ws, router_ws, total;
  Scratch(int T, int H, int I, int E, int K) {
    const size_t tk = static_cast<size_t>(T) * K;
    size_t at = 0;
    const auto take = [&at](size_t bytes) {
      const size_t here = at;
      at += (bytes + 255) & ~static_cast<size_t>(255);
      return here;
    };
    scores = take(tk * 4);
    indices = take(tk * 4);
    aux_grad = take(static_cast<size_t>(E) * 4);
    off = take((static_cast<size_t>(E) + 1) * 4);
    idx3 = take(3 * tk * 4);
    y1 = take(tk * I * 2);
    y2 = take(K == 1 ? 0 : tk * H * 2);
    route_ws = take(smoe_route_metadata_workspace_bytes(E));
    router_ws = take(smoe_router_forward_workspace_bytes(E));
    total = at;
  }
};

// What a training forward pass leaves for the backward pass, in 4-byte words.
struct Meta {
  float* scores;   // (T, K)
  int* indices;    // (T, K)
  int* s_scatter;  // (TK)
  int* s_reverse;  // (TK)
  int* x_gather;   // (TK)
  int* off;        // (E + 1)
  float* aux_grad; // (E)
  Meta(void* meta, size_t tk, int E) {
    int* at = static_cast<int*>(meta);
    scores = reinterpret_cast<float*>(at);
    indices = at + tk;
    s_scatter = at + 2 * tk;
    s_reverse = at + 3 * tk;
    x_gather = at + 4 * tk;
    off = at + 5 * tk;
    aux_grad = reinterpret_cast<float*>(off + E + 1);
  }
};

size_t round256(size_t bytes) { return (bytes + 255) & ~static_cast<size_t>(255); }

// Scratch of the training forward pass.  y2 comes last: the plain kernels' combine of one row per token has none.
struct ForwardScratch {
  size_t y1, route_ws, router_ws, y2, total;
  ForwardScratch(int T, int H, int I, int E, int K) {
    const size_t tk = static_cast<size_t>(T) * K;
    y1 = 0;
    route_ws = y1 + round256(tk * I * 2);
    router_ws = route_ws + round256(smoe_route_metadata_workspace_bytes(E));
    y2 = router_ws + round256(smoe_router_forward_workspace_bytes(E));
    total = y2 + round256(tk * H * 2);
  }
};

// Scratch of the backward pass, shared by its entry points.
struct BackwardScratch {
  size_t dz, y1s, ds_partial, ds, total;
  BackwardScratch(int T, int I, int N1, int K) {
    const size_t tk = static_cast<size_t>(T) * K;
    dz = 0;
    y1s = dz + round256(tk * N1 * 2);
    ds_partial = y1s + round256(tk * I * 2);
    ds = ds_partial + round256(tk * smoe_ds_partial_columns(I) * 4);
    total = ds + round256(tk * 4);
  }
};

// What the calls below would refuse is refused before the first of them launches something: sizes, pointers and alignment are
// checked by the compound entry points themselves.
bool bad_layer(int T, int H, int I, int N1, int E, int K) {
  return T <= 0 || H <= 0 || H % 64 != 0 || I <= 0 || I % 64 != 0 || (N1 != I && N1 != 2 * static_cast<long long>(I)) ||
         N1 % 128 != 0 || E <= 0 || E > smoe::kMaxExperts || K <= 0 || K > E || static_cast<long long>(T) * K > 0x7fffffffll;
}

// Scratch and metadata are laid out for N1 rows, and the activation's kernels write as many as it has.
bool bad_activation_rows(int activation, int I, int N1) {
  return activation < smoe::ACT_SWIGLU || activation > smoe::ACT_SILU ||
         N1 != (smoe::act_is_gated(activation) ? 2 : 1) * static_cast<long long>(I);
}

bool aligned(const void* p, uintptr_t bytes) { return reinterpret_cast<uintptr_t>(p) % bytes == 0; }

int check_given(std::initializer_list<const void*> pointers, uintptr_t bytes) {
  for (const void* p : pointers) {
    if (p == nullptr) return SMOE_ERR_SHAPE;
    if (!aligned(p, bytes)) return SMOE_ERR_ALIGNMENT;
  }
  return SMOE_OK;
}

int check_optional(std::initializer_list<const void*> pointers, uintptr_t bytes) {
  for (const void* p : pointers)
    if (!aligned(p, bytes)) return SMOE_ERR_ALIGNMENT;
  return SMOE_OK;
}

int check_workspace(const void* p, uintptr_t bytes) {
  return p == nullptr ? SMOE_ERR_WORKSPACE : aligned(p, bytes) ? SMOE_OK : SMOE_ERR_ALIGNMENT;
}

// The router's logits (T,E): bytes per value, or 0 for an unknown type.
int logit_bytes(int dtype) { return dtype == SMOE_F32 ? 4 : dtype == SMOE_BF16 ? 2 : 0; }

}  // namespace

#define SMOE_TRY(expr)              \
  do {                              \
    const int _rc = (expr);         \
    if (_rc != SMOE_OK) return _rc; \
  } while (0)

extern "C" {

size_t smoe_layer_forward_scratch_bytes(int T, int H, int I, int E, int K) {
  if (T < 0 || H <= 0 || I <= 0 || E <= 0 || K <= 0) return 0;
  return Scratch(T, H, I, E, K).total;
}

int smoe_layer_forward(const void* x, const void* router_w, const void* w1, const void* w2, void* o, void* logits,
                       int* expert_count, float* prob_colsum, float* aux, void* scratch, int T, int H, int I, int E,
                       int K, int* status, void* stream) {
  if (T <= 0 || !smoe_router_forward_supported(H, E, K) || I <= 0 || I % 64 != 0 ||
      static_cast<long long>(T) * K > 0x7fffffffll)
    return SMOE_ERR_SHAPE;
  SMOE_TRY(check_given({x, router_w, w1, w2, o, logits}, 16));  // TMA sources, and rows stored in 16-byte pieces
  SMOE_TRY(check_given({expert_count, prob_colsum, aux}, 4));
  SMOE_TRY(check_workspace(scratch, 256));
  const Scratch at(T, H, I, E, K);
  char* base = static_cast<char*>(scratch);
  const auto ints = [base](size_t o_) { return reinterpret_cast<int*>(base + o_); };
  const auto floats = [base](size_t o_) { return reinterpret_cast<float*>(base + o_); };
  const int tk = T * K;
  int* s_scatter = ints(at.idx3);
  int* s_reverse = s_scatter + tk;
  int* x_gather = s_reverse + tk;
  SMOE_TRY(smoe_router_forward_aux(x, router_w, logits, floats(at.scores), ints(at.indices), expert_count, prob_colsum,
                                   aux, floats(at.aux_grad), base + at.router_ws, T, H, E, K, status, stream));
  SMOE_TRY(smoe_route_metadata(ints(at.indices), nullptr, tk, E, K, expert_count, ints(at.off), s_scatter, s_reverse,
                               x_gather, ints(at.route_ws), stream));
  SMOE_TRY(smoe_up_projection_forward(x, w1, nullptr, base + at.y1, ints(at.off), x_gather, T, H, I, E, tk, status,
                                      stream));
  if (K == 1)
    return smoe_down_projection_forward_rows(base + at.y1, w2, o, floats(at.scores), 0, ints(at.off), x_gather, s_scatter,
                                             H, I, E, tk, status, stream);
  SMOE_TRY(smoe_down_projection_forward(base + at.y1, w2, base + at.y2, ints(at.off), H, I, E, tk, status, stream));
  return smoe_gather_sum(base + at.y2, o, floats(at.scores), SMOE_F32, s_reverse, nullptr, T, H, K, stream);
}

size_t smoe_layer_meta_words(int T, int E, int K) {
  if (T <= 0 || E <= 0 || K <= 0) return 0;
  return 5 * static_cast<size_t>(T) * K + 2 * static_cast<size_t>(E) + 1;
}

size_t smoe_layer_train_forward_scratch_bytes(int T, int H, int I, int E, int K) {
  if (T <= 0 || H <= 0 || I <= 0 || E <= 0 || K <= 0) return 0;
  return ForwardScratch(T, H, I, E, K).total;
}

size_t smoe_layer_train_forward_plain_scratch_bytes(int T, int H, int I, int E, int K) {
  if (T <= 0 || H <= 0 || I <= 0 || E <= 0 || K <= 0) return 0;
  const ForwardScratch at(T, H, I, E, K);
  return K == 1 ? at.y2 : at.total;
}

int smoe_layer_train_forward(const void* x, const void* router_w, void* logits, int logits_dtype, const void* w1,
                             const void* b1, const void* w2, const void* b2, void* o, void* z, void* meta,
                             int* expert_count, float* prob_colsum, float* aux, void* scratch, int T, int H, int I, int N1,
                             int E, int K, int activation, int* status, void* stream) {
  if (bad_layer(T, H, I, N1, E, K) || bad_activation_rows(activation, I, N1)) return SMOE_ERR_SHAPE;
  if (router_w != nullptr) {
    if (!smoe_router_forward_supported(H, E, K)) return SMOE_ERR_SHAPE;
    SMOE_TRY(check_given({router_w, logits}, 16));
    SMOE_TRY(check_given({expert_count, aux}, 4));
  } else {
    if (logit_bytes(logits_dtype) == 0) return SMOE_ERR_DTYPE;
    SMOE_TRY(check_given({logits}, logit_bytes(logits_dtype)));
  }
  SMOE_TRY(check_given({x, w1, w2, o}, 16));
  SMOE_TRY(check_optional({b1, b2, z}, 16));
  SMOE_TRY(check_optional({expert_count, prob_colsum}, 4));
  SMOE_TRY(check_workspace(meta, 4));
  SMOE_TRY(check_workspace(scratch, 256));
  const int tk = T * K;
  const Meta m(meta, tk, E);
  const ForwardScratch at(T, H, I, E, K);
  char* base = static_cast<char*>(scratch);
  if (router_w != nullptr)
    SMOE_TRY(smoe_router_forward_aux(x, router_w, logits, m.scores, m.indices, expert_count, prob_colsum, aux, m.aux_grad,
                                     base + at.router_ws, T, H, E, K, status, stream));
  else
    SMOE_TRY(smoe_topk_softmax(logits, logits_dtype, m.scores, m.indices, T, E, K, stream));
  SMOE_TRY(smoe_route_metadata(m.indices, nullptr, tk, E, K, expert_count, m.off, m.s_scatter, m.s_reverse, m.x_gather,
                               base + at.route_ws, stream));
  const bool plain = activation == smoe::ACT_SWIGLU && b1 == nullptr && b2 == nullptr;
  if (plain)
    SMOE_TRY(smoe_up_projection_forward(x, w1, z, base + at.y1, m.off, m.x_gather, T, H, I, E, tk, status, stream));
  else
    SMOE_TRY(smoe_up_projection_forward_act(x, w1, b1, z, base + at.y1, m.off, m.x_gather, T, H, N1, E, tk, activation,
                                            status, stream));
  if (plain && K == 1)
    return smoe_down_projection_forward_rows(base + at.y1, w2, o, m.scores, 0, m.off, m.x_gather, m.s_scatter, H, I, E, tk,
                                             status, stream);
  if (plain)
    SMOE_TRY(smoe_down_projection_forward(base + at.y1, w2, base + at.y2, m.off, H, I, E, tk, status, stream));
  else
    SMOE_TRY(smoe_down_projection_forward_bias(base + at.y1, w2, b2, base + at.y2, m.off, H, I, E, tk, status, stream));
  return smoe_gather_sum(base + at.y2, o, m.scores, SMOE_F32, m.s_reverse, nullptr, T, H, K, stream);
}

size_t smoe_layer_backward_scratch_bytes(int T, int I, int N1, int K) {
  if (T <= 0 || I <= 0 || N1 <= 0 || K <= 0) return 0;
  return BackwardScratch(T, I, N1, K).total;
}

int smoe_layer_backward_act(const void* dout, const void* w2, const void* b2, const void* z, void* meta,
                            const void* logits, int logits_dtype, int fused_router, const void* g_logits,
                            const float* g_colsum, const float* g_aux, void* dlogits, void* db1, void* db2, void* scratch,
                            int T, int H, int I, int N1, int E, int K, int activation, int* status, void* stream) {
  if (bad_layer(T, H, I, N1, E, K) || bad_activation_rows(activation, I, N1)) return SMOE_ERR_SHAPE;
  SMOE_TRY(check_workspace(meta, 4));
  if (dout != nullptr) {
    SMOE_TRY(check_given({dout, w2, z}, 16));
    SMOE_TRY(check_optional({b2}, 16));
    if (b2 != nullptr) SMOE_TRY(check_given({db1, db2}, 16));
    SMOE_TRY(check_workspace(scratch, 256));
  }
  if (dlogits != nullptr) {
    if (fused_router) {
      if (E > smoe::kMaxRouterExperts) return SMOE_ERR_SHAPE;
      if (g_colsum != nullptr || g_aux != nullptr) SMOE_TRY(check_given({logits}, 2));
      SMOE_TRY(check_optional({dlogits, g_logits}, 2));
      SMOE_TRY(check_optional({g_colsum, g_aux}, 4));
    } else {
      if (dout == nullptr) return SMOE_ERR_SHAPE;  // nothing else has a gradient by the scores
      if (logit_bytes(logits_dtype) == 0) return SMOE_ERR_DTYPE;
      SMOE_TRY(check_optional({dlogits}, logit_bytes(logits_dtype)));
    }
  }
  const int tk = T * K;
  const Meta m(meta, tk, E);
  const BackwardScratch at(T, I, N1, K);
  char* base = static_cast<char*>(scratch);
  float* ds = dout != nullptr ? reinterpret_cast<float*>(base + at.ds) : nullptr;
  if (dout != nullptr) {
    float* partial = reinterpret_cast<float*>(base + at.ds_partial);
    if (activation == smoe::ACT_SWIGLU && b2 == nullptr)
      SMOE_TRY(smoe_down_projection_backward_act(dout, w2, z, m.scores, 0, base + at.dz, base + at.y1s, partial, m.off,
                                                 m.x_gather, m.s_scatter, T, H, I, E, tk, status, stream));
    else
      SMOE_TRY(smoe_down_projection_backward_dact(dout, w2, z, m.scores, 0, base + at.dz, base + at.y1s, partial, m.off,
                                                  m.x_gather, m.s_scatter, T, H, I, E, tk, activation, status, stream));
    SMOE_TRY(smoe_ds_reduce(partial, m.s_scatter, ds, SMOE_F32, tk, smoe_ds_partial_columns(I), stream));
    if (b2 != nullptr) {
      SMOE_TRY(smoe_ds_add_bias_term(dout, b2, m.off, m.x_gather, m.s_scatter, ds, SMOE_F32, E, H, tk, stream));
      SMOE_TRY(smoe_expert_column_sum(dout, H, m.x_gather, m.scores, SMOE_F32, m.s_scatter, m.off, db2, E, H, stream));
      SMOE_TRY(smoe_expert_column_sum(base + at.dz, N1, nullptr, nullptr, 0, nullptr, m.off, db1, E, N1, stream));
    }
  }
  if (dlogits == nullptr) return SMOE_OK;
  if (fused_router)
    return smoe_router_backward_aux(dlogits, logits, ds, m.scores, m.indices, g_colsum, g_logits, g_aux, m.aux_grad, T, E,
                                    K, stream);
  return smoe_softmax_topk_backward(dlogits, logits_dtype, ds, m.scores, m.indices, T, E, K, stream);
}

int smoe_layer_backward_dx(const void* w1, void* meta, const void* scratch, void* dx_expanded, void* dx, int add, int T,
                           int H, int I, int N1, int E, int K, int* status, void* stream) {
  if (bad_layer(T, H, I, N1, E, K)) return SMOE_ERR_SHAPE;
  SMOE_TRY(check_given({w1, dx}, 16));
  SMOE_TRY(check_workspace(meta, 4));
  SMOE_TRY(check_workspace(scratch, 256));
  if (K > 1) SMOE_TRY(check_workspace(dx_expanded, 16));
  const int tk = T * K;
  const Meta m(meta, tk, E);
  const char* dz = static_cast<const char*>(scratch) + BackwardScratch(T, I, N1, K).dz;
  // the kernels take the up projection's output rows as 2 * (their I argument)
  if (K == 1)
    return add ? smoe::up_projection_backward_dx_rows_add(dz, w1, dx, m.off, m.x_gather, H, N1 / 2, E, tk, status, stream)
               : smoe_up_projection_backward_dx_rows(dz, w1, dx, m.off, m.x_gather, H, N1 / 2, E, tk, status, stream);
  SMOE_TRY(smoe_up_projection_backward_dx(dz, w1, dx_expanded, m.off, H, N1 / 2, E, tk, status, stream));
  return add ? smoe::gather_sum_add(dx_expanded, dx, nullptr, m.s_reverse, T, H, K, stream)
             : smoe_gather_sum(dx_expanded, dx, nullptr, SMOE_F32, m.s_reverse, nullptr, T, H, K, stream);
}

int smoe_layer_backward_weights(const void* x, const void* dout, void* meta, const void* scratch, void* dw1, void* dw2,
                                int T, int H, int I, int N1, int E, int K, int* status, void* stream) {
  if (bad_layer(T, H, I, N1, E, K)) return SMOE_ERR_SHAPE;
  SMOE_TRY(check_given({x, dout, dw1, dw2}, 16));
  SMOE_TRY(check_workspace(meta, 4));
  SMOE_TRY(check_workspace(scratch, 256));
  const int tk = T * K;
  const Meta m(meta, tk, E);
  const BackwardScratch at(T, I, N1, K);
  const char* base = static_cast<const char*>(scratch);
  SMOE_TRY(smoe_down_projection_weight_grad(dout, base + at.y1s, dw2, m.off, m.x_gather, T, H, I, E, tk, status, stream));
  return smoe_up_projection_weight_grad(x, base + at.dz, dw1, m.off, m.x_gather, T, H, N1 / 2, E, tk, status, stream);
}

}  // extern "C"

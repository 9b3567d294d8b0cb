// The inference forward pass as one entry point: the same launches as the separate ones, without a trip through the
// caller's language for each.  A layer call of a few tokens is shorter on the device (60 us for one token of a 64-expert
// layer) than eight launches with their allocations and argument conversions take from Python.
#include <cuda_runtime.h>
#include <stddef.h>
#include <stdint.h>

#include "../../include/sonicmoe_b200.h"

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

bool aligned(const void* p, uintptr_t bytes) { return reinterpret_cast<uintptr_t>(p) % bytes == 0; }

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
  // what any of the calls below would refuse is refused before the first of them launches something
  if (T <= 0 || !smoe_router_forward_supported(H, E, K) || I <= 0 || I % 64 != 0 ||
      static_cast<long long>(T) * K > 0x7fffffffll)
    return SMOE_ERR_SHAPE;
  const void* const wide[] = {x, router_w, w1, w2, o, logits};  // TMA sources, and rows stored in 16-byte pieces
  for (const void* ptr : wide) {
    if (ptr == nullptr) return SMOE_ERR_SHAPE;
    if (!aligned(ptr, 16)) return SMOE_ERR_ALIGNMENT;
  }
  const void* const words[] = {expert_count, prob_colsum, aux};
  for (const void* ptr : words) {
    if (ptr == nullptr) return SMOE_ERR_SHAPE;
    if (!aligned(ptr, 4)) return SMOE_ERR_ALIGNMENT;
  }
  if (scratch == nullptr) return SMOE_ERR_WORKSPACE;
  if (!aligned(scratch, 256)) return SMOE_ERR_ALIGNMENT;
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

}  // extern "C"

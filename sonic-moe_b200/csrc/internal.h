// What the library's own compound entry points (layer.cu) need beyond the exported ones.
#pragma once

namespace smoe {

constexpr int kMaxExperts = 1024;  // experts whose offsets the grouped GEMMs keep in shared memory
constexpr int kMaxRouterExperts = 256;  // experts of the router kernels

// smoe_gather_sum with fp32 weights or none whose result is added to `out` (bf16) instead of replacing it: one rounding of the sum.
int gather_sum_add(const void* src, void* out, const float* weights, const int* reverse_idx, int T, int H, int K,
                   void* stream);
// smoe_up_projection_backward_dx_rows whose rows (rounded to bf16) are added to those of dx.
int up_projection_backward_dx_rows_add(const void* dz, const void* w1, void* dx, const int* expert_offset,
                                       const int* x_gather_idx, int H, int I, int E, int TK, int* status, void* stream);

}  // namespace smoe

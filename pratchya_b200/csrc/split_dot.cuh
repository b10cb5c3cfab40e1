// The form of the literal f32 dots whose operands are made ready for the tensor core once (split_dot.cu), for dense_dot.cu.
#pragma once

#include <cstddef>
#include <cstdint>

#include <cuda_runtime.h>

namespace pb {

constexpr size_t kSplitAlign = 32;    // of the workspace: the terms are stored 32 bytes at a time

struct SplitDotPlan {
  int n, tiles, row_tiles, splits, units, units_per_split, variants, nbc, log2_K;
  int64_t slab;                       // rows of the three-term operand at a time
  bool exact;                         // that operand is one term: the fp8 values times their block's power of two
  size_t off_other, off_parts, bytes; // of the workspace, which starts with the terms
};
// False where dense_dot_kernel takes the call: shapes this form does not take, and those it is not faster for.
bool split_dot_plan(int tokens, int64_t rows, int64_t cols, int a, int b, int64_t g_free, bool g_bf16, SplitDotPlan* d);
int split_dot_run(const SplitDotPlan& d, int tokens, const uint8_t* q, const uint8_t* sc8, const float* sc32, int64_t rows, int64_t cols, int a, int b,
                  const void* g, bool g_bf16, int64_t g_free, float* out, void* workspace, cudaStream_t st);
// dense_dot.cu: out = the sum of `splits` parts of n elements (a multiple of 4), in their order
int add_parts(const float* parts, float* out, int64_t n, int splits, cudaStream_t st);
int split_dot_status_fetch(unsigned int* out);
#ifdef PB_DIAGNOSTICS
void split_dot_control(uint32_t polls, int withhold);
#endif

}  // namespace pb

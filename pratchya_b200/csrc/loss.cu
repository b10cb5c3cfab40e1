// The training loss of the reference, compute_loss (pratchya/_nnx_impl/_utils.py:7-13): softmax cross entropy against
// one-hot labels smoothed by alpha (optax.smooth_labels), mean over the positions that count.  Per row of logits z with
// target t:   loss_row = lse(z) - (1 - alpha) * z_t - alpha * mean_j(z_j)
// (the cross entropy against (1 - alpha) * onehot + alpha / V, written out), and its cotangent
//             dz_j = g_row * (exp(z_j - lse) - (1 - alpha) * [j == t] - alpha / V).
// As framework operations this is a log-softmax, a gather, a mean and their backward passes over an array of
// [tokens, vocabulary] f32 (8.6 GB at 32768 x 65536): six passes and three arrays of that size.  Here the forward kernel
// reads the logits once (one CTA per row, every thread with a running maximum of its own) and the backward kernel reads them
// once more and writes dz: HBM-bound, 4 + 8 bytes per logit.
#include "common.cuh"

namespace pb {
namespace {

// Threads per row: 256, or 1024 where there are few long rows (wide_forward, wide_backward).
constexpr int kLossThreads = 256, kWideThreads = 1024;
constexpr int kLoads = 4;             // 16-byte loads that a thread has in flight

// A thread's maximum, sum of exp(z - maximum) and sum of z.  While the maximum is -inf (nothing but -inf seen) the
// exponentials are taken from 0, so that -inf - -inf does not make a NaN of a logit that only weighs nothing.
struct RowTerms {
  float m = -INFINITY, s = 0.0f, zs = 0.0f;
  __device__ __forceinline__ void raise(float top) {
    const float m2 = fmaxf(m, top);
    if (m2 > m) {
      if (s != 0.0f) s *= expf(m - m2);      // the first logits have nothing to rescale
      m = m2;
    }
  }
  __device__ __forceinline__ void add(const float4& v) {
    const float base = m == -INFINITY ? 0.0f : m;
    s += (expf(v.x - base) + expf(v.y - base)) + (expf(v.z - base) + expf(v.w - base));
    zs += (v.x + v.y) + (v.z + v.w);
  }
  // the terms of LANES lanes of a warp together, in each of them
  template <int LANES>
  __device__ __forceinline__ void over_lanes() {
    float top = m;
#pragma unroll
    for (int o = LANES / 2; o > 0; o >>= 1) top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, o));
    s *= expf(m - (top == -INFINITY ? 0.0f : top));      // m = -inf: 0 * 0
    m = top;
#pragma unroll
    for (int o = LANES / 2; o > 0; o >>= 1) {
      s += __shfl_xor_sync(0xffffffffu, s, o);
      zs += __shfl_xor_sync(0xffffffffu, zs, o);
    }
  }
};
__device__ __forceinline__ float top4(const float4& v) { return fmaxf(fmaxf(v.x, v.y), fmaxf(v.z, v.w)); }

// row_loss[r] = weight[r] * loss_row, lse[r] kept for the backward pass.  One CTA per row, one read of it: a thread keeps a
// running maximum and rescales its sum of exponentials where the maximum rises; the threads' terms meet at the end, in their
// warps and then in the first one, behind one barrier.
// Bound by the 4 bytes per logit.  The form before read the row twice, maximum and sum of z first and the exponentials on
// a second read from L2, with one 16-byte load of a thread in flight:
// 4096 x 65536 logits 0.316 ms, now 0.17 ms (6.3 TB/s; the loss and its gradient 0.684 -> 0.537 ms).
template <int THREADS, int PER_SM>
__global__ void __launch_bounds__(THREADS, PER_SM) smoothed_xent_fwd_kernel(const float* logits, const int64_t* target, const float* weight,
                                                                   float* row_loss, float* lse, int64_t vocab, float alpha) {
  grid_wait();
  __shared__ float red[3][THREADS / 32];
  const int64_t row = blockIdx.x;
  const float4* z4 = reinterpret_cast<const float4*>(logits + row * vocab);
  const int64_t quads = vocab / 4, whole = quads - quads % (THREADS * kLoads);
  RowTerms t;
  for (int64_t j = threadIdx.x; j < whole; j += THREADS * kLoads) {
    float4 v[kLoads];
#pragma unroll
    for (int k = 0; k < kLoads; ++k) v[k] = __ldg(z4 + j + k * THREADS);
    float top = top4(v[0]);
#pragma unroll
    for (int k = 1; k < kLoads; ++k) top = fmaxf(top, top4(v[k]));
    t.raise(top);
#pragma unroll
    for (int k = 0; k < kLoads; ++k) t.add(v[k]);
  }
  for (int64_t j = whole + threadIdx.x; j < quads; j += THREADS) {
    const float4 v = __ldg(z4 + j);
    t.raise(top4(v));
    t.add(v);
  }
  t.over_lanes<32>();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (lane == 0) { red[0][warp] = t.m; red[1][warp] = t.s; red[2][warp] = t.zs; }
  __syncthreads();
  if (warp != 0) return;
  RowTerms r;
  if (lane < THREADS / 32) { r.m = red[0][lane]; r.s = red[1][lane]; r.zs = red[2][lane]; }
  r.over_lanes<THREADS / 32>();
  if (lane == 0) {
    const float l = r.m + logf(r.s * expf(r.m - r.m));      // a row of -inf only: NaN, as its softmax is
    lse[row] = l;
    row_loss[row] = weight[row] * (l - (1.0f - alpha) * logits[row * vocab + target[row]] - alpha * (r.zs / (float)vocab));
  }
}

// dz[r][j] = g[r] * (exp(z - lse) - (1 - alpha) * [j == t] - alpha / V), g[r] = upstream * weight[r] / denominator
template <int THREADS>
__global__ void __launch_bounds__(THREADS) smoothed_xent_bwd_kernel(const float* logits, const int64_t* target, const float* weight,
                                                                   const float* lse, const float* upstream, float inv_denominator,
                                                                   float* dlogits, int64_t vocab, float alpha) {
  grid_wait();
  const int64_t row = blockIdx.x;
  const float* z = logits + row * vocab;
  float* dz = dlogits + row * vocab;
  const float g = upstream[0] * weight[row] * inv_denominator, l = lse[row];
  const int64_t t = target[row];
  const float smooth = alpha / (float)vocab;
  for (int64_t j = (int64_t)threadIdx.x * 4; j < vocab; j += THREADS * 4) {
    const float4 v = *reinterpret_cast<const float4*>(z + j);
    float4 d = make_float4(expf(v.x - l) - smooth, expf(v.y - l) - smooth, expf(v.z - l) - smooth, expf(v.w - l) - smooth);
    if (t >= j && t < j + 4) {
      const float hit = 1.0f - alpha;
      if (t == j) d.x -= hit; else if (t == j + 1) d.y -= hit; else if (t == j + 2) d.z -= hit; else d.w -= hit;
    }
    *reinterpret_cast<float4*>(dz + j) = make_float4(g * d.x, g * d.y, g * d.z, g * d.w);
  }
}

// Where 1024 threads a row are faster than 256.  A CTA of 1024 has an SM to itself in the forward pass, and a thread's few
// loads do not pay for meeting at the end.  Forward, us, 256 | 1024 threads: 65536 logits 10.3 | 7.5 with 148 rows, 12.2 | 13.1
// with 222; 16384 logits 4.4 | 4.2 with 148 rows; 8192 3.6 | 3.8; 4096 logits 4.3 | 11.6 with 740 rows.
bool wide_forward(int64_t rows, int64_t vocab) { return rows <= sm_count() && vocab >= 16384; }
// Backward: 4096 logits 3.0 | 2.6 with 148 rows, 3.4 | 3.4 with 296, 3.6 | 4.2 with 444; 16384 logits 7.3 | 5.9 with 296 rows,
// 14.6 | 15.7 with 740; 32768 logits 38 | 35 with 740 rows; 65536 18.9 | 9.1 with 148 rows, 73 | 66 with 740.
bool wide_backward(int64_t rows, int64_t vocab) {
  return (vocab >= 4096 && rows <= 2 * (int64_t)sm_count()) || (vocab >= 32768 && rows < 6 * (int64_t)sm_count());
}

}  // namespace
}  // namespace pb

using namespace pb;

extern "C" int pb_smoothed_xent(const float* logits, const int64_t* target, const float* weight, int64_t rows, int64_t vocab, float alpha,
                                float* row_loss, float* lse, void* stream) {
  if (!logits || !target || !weight || !row_loss || !lse) return fail(PB_ERR_NULL_POINTER, "pb_smoothed_xent: null argument");
  if (rows <= 0 || vocab <= 0 || vocab % 4 != 0 || rows > 0x7fffffffll)
    return fail(PB_ERR_BAD_SHAPE, "pb_smoothed_xent: rows=%lld vocab=%lld (vocab must be a multiple of 4)", (long long)rows, (long long)vocab);
  if (reinterpret_cast<uintptr_t>(logits) & 15) return fail(PB_ERR_MISALIGNED, "pb_smoothed_xent: logits must be 16-byte aligned");
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  // eight CTAs on an SM (32 registers) where no thread has a whole round of loads, six otherwise: 4096 rows, 2048 logits 12.1 us with
  // six and 11.5 with eight, 65536 logits 157 and 161
  if (wide_forward(rows, vocab))
    launch_behind(smoothed_xent_fwd_kernel<kWideThreads, 1>, (unsigned)rows, kWideThreads, 0, st, logits, target, weight, row_loss, lse, vocab, alpha);
  else if (vocab < kLossThreads * kLoads * 4)
    launch_behind(smoothed_xent_fwd_kernel<kLossThreads, 8>, (unsigned)rows, kLossThreads, 0, st, logits, target, weight, row_loss, lse, vocab, alpha);
  else
    launch_behind(smoothed_xent_fwd_kernel<kLossThreads, 6>, (unsigned)rows, kLossThreads, 0, st, logits, target, weight, row_loss, lse, vocab, alpha);
  PB_LAUNCH_CHECK("smoothed_xent_fwd_kernel");
  return PB_OK;
}

extern "C" int pb_smoothed_xent_bwd(const float* logits, const int64_t* target, const float* weight, const float* lse, const float* upstream,
                                    float denominator, int64_t rows, int64_t vocab, float alpha, float* dlogits, void* stream) {
  if (!logits || !target || !weight || !lse || !upstream || !dlogits) return fail(PB_ERR_NULL_POINTER, "pb_smoothed_xent_bwd: null argument");
  if (rows <= 0 || vocab <= 0 || vocab % 4 != 0 || rows > 0x7fffffffll || !(denominator > 0.0f))
    return fail(PB_ERR_BAD_SHAPE, "pb_smoothed_xent_bwd: rows=%lld vocab=%lld denominator=%g", (long long)rows, (long long)vocab, (double)denominator);
  if ((reinterpret_cast<uintptr_t>(logits) & 15) || (reinterpret_cast<uintptr_t>(dlogits) & 15))
    return fail(PB_ERR_MISALIGNED, "pb_smoothed_xent_bwd: logits and dlogits must be 16-byte aligned");
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  if (wide_backward(rows, vocab))
    launch_behind(smoothed_xent_bwd_kernel<kWideThreads>, (unsigned)rows, kWideThreads, 0, st, logits, target, weight, lse, upstream, 1.0f / denominator, dlogits, vocab, alpha);
  else
    launch_behind(smoothed_xent_bwd_kernel<kLossThreads>, (unsigned)rows, kLossThreads, 0, st, logits, target, weight, lse, upstream, 1.0f / denominator, dlogits, vocab, alpha);
  PB_LAUNCH_CHECK("smoothed_xent_bwd_kernel");
  return PB_OK;
}

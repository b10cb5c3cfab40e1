// WKV-7 state scan of the modified RWKV-7 TimeMix block (sm_100a): the per-timestep recurrence of
// pratchya/_nnx_impl/_module.py:187-207 as one kernel instead of a scan of T small matmuls, and its
// cotangents (what jax.grad derives from that scan) as a second kernel.
//
// Per (batch b, head n) the state S is an H x H fp32 matrix (rows: value channel i, columns: key
// channel j).  With, at timestep t, w = decay, a = iclr, kap = removal_k, kt = replacement_k, v and r
// (each a vector of H channels of that head):
//     sa_i  = sum_j S[i][j] * kap_j                         (wkv_state @ removal_k_t, :197)
//     S[i][j] = S[i][j] * w_j - sa_i * (a_j * kap_j)        (:197)
//     S[i][j] += v_i * kt_j                                 (:198)
//     y_i   = sum_j S[i][j] * r_j                           (:199)
// All arithmetic is fp32, as in the reference (its inputs are cast to f32 before the scan).
//
// Both kernels keep the state in 2-D register tiles (H = 64), so that a lane reads a part of each vector per timestep: what
// those reads return to the registers, 128 bytes per clock and SM, is what a whole row per thread was bound by.  Sums along a
// row stay inside a warp (shuffles); sums along a column, which only the backward pass has and which are outputs, not part of
// the recurrence, meet in shared memory.
// The input vectors of a timestep arrive by cp.async ahead of time.  HBM traffic is near the algorithmic minimum: every
// input read once (where several CTAs share a head each reads its vectors, at about the same time: all but one from L2), every
// output written once, the state once per sequence, plus what the backward pass needs when one follows (below).
#include "common.cuh"

namespace pb {
namespace {

constexpr int kH = 64;            // head size
constexpr int kWarps = 4;         // of the backward kernel: a warp owns 16 rows
constexpr int kThreads = 32 * kWarps;      // per head
constexpr int kVecs = 6;          // decay, iclr, removal_k, replacement_k, v, r
constexpr int kCk = 8;            // spacing of the state checkpoints the backward pass restarts from
constexpr int kSub = 4;           // timesteps whose recomputed states the backward pass keeps at once
constexpr int kBwdVecs = kVecs + 2;      // the six inputs, dy and sa
constexpr int kNegB = kBwdVecs;          // and -b = -(a o kap), made from them
constexpr int kBwdSlots = kBwdVecs + 1;
constexpr int kTileQuads = kH * kH / 4;  // float4 per state

__device__ __forceinline__ void cp_async16(uint32_t dst, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N> __device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

__device__ __forceinline__ float2 dup(float x) { return make_float2(x, x); }

// A state in the kernels' own layout (checkpoints in global memory, kept states in shared memory): 1024 quads, a quad the
// rows 2P, 2P + 1 of the columns 2Q, 2Q + 1 as ((2P, 2Q), (2P+1, 2Q), (2P, 2Q+1), (2P+1, 2Q+1)).  Backward thread
// 16 * (P >> 2) + (Q >> 1) keeps it as its quad 2 * (P & 3) + (Q & 1): consecutive threads, consecutive 16 bytes.
__device__ __forceinline__ int ckpt_quad(int P, int Q) { return (2 * (P & 3) + (Q & 1)) * kThreads + 16 * (P >> 2) + (Q >> 1); }

// ---- forward ---------------------------------------------------------------------------------------------------
// The rows of a head's state are independent of one another given the timestep's vectors, so a head's 64 rows are cut over
// warps, and where there are few heads over CTAs as well.  A warp's lanes are a grid of 2 x 16 or 4 x 8; a lane keeps ROWS rows x 4
// or 8 columns, and a row's dot products end in shuffles.
//
// The chain.  sa_t = S_{t-1} kap_t waits for the timestep before, and everything else hangs on it: a dot product, a sum over lanes, the
// update.  sa is taken of the state as it is stored, at every timestep: what rounding left in it is then read and erased with it, and a scan cut after
// any timestep and continued from its state gives the bits of the whole one.  (Written with S_{t-1} in terms of S_{t-2}, whose sum could start a timestep
// earlier, 16 heads take 101 us instead of 125, but a timestep behind one that has erased something large is off by 2^-24 of what was erased: one
// key repeated, a value of 64 among others of size one, that timestep's y 4e-6 instead of 5e-8.)  b = a o kap is made a chunk ahead, once per CTA, by warps
// of their own, from the chunk's vectors as they arrive by cp.async; one barrier per chunk.
//
// Sums.  sa of a timestep and y of the one before, both of the same state, are summed together: of two lanes half a row apart one keeps sa's part
// and hands over its part of y, the other the reverse (each reads its two vectors in that order); a lane's rows are in an order
// of its own (register a holds row a ^ its lane bits), so that every further halving hands over the upper registers and no value
// is selected.  A row's sa ends on lanes that broadcast it; its y on as many, which store it.  A sum's levels
// have the same order in every form, so the bits do not depend on the number of heads.
//
// The update is (S o w - sa b^T) + v kt^T with the erasure's product rounded and the other two fused: v kt^T comes last (added
// to a state that is about to be erased, its low bits would go with it), and of the three roundings one is of the erased part's
// size instead of the state's: 2-norm errors against 64 bits 9.8e-8 -> 9.1e-8 of y, 7.1e-8 -> 6.0e-8 of the state (500 timesteps).
//
// What bounds it: with few heads the chain (235 cycles a timestep: five shuffles behind one another, the dot product and the update; sums that every
// lane of a row makes, four shuffles but twice as many of them, 125 -> 129 us; vectors read in front of the shuffles, or between them, the same), with many
// the f32x2 products, three cycles each where their operands are three different registers, on top of the reads.  Two CTAs of a whole head
// an SM: four preparing warps, one a scheduler (one alone makes its scheduler the slowest), which hand their registers over.
// 1024 timesteps, us, against each lane's own b and sums of sa and y one after the other: 16 heads 122 -> 125 (with saves 159 -> 131), 32 heads 144 -> 125
// (160 -> 131), 60 heads 162 -> 145 (183 -> 157), 128 heads 218 -> 198 (254 -> 235), 160 heads 326 -> 327 (356 -> 360), 222 heads 354 -> 327 (424 -> 360),
// 256 heads 353 -> 335 (423 -> 389); 32 heads x 4096 571 -> 492.
constexpr int kFwdChunk = 8;      // timesteps between barriers
constexpr int kFwdBufs = 5;       // chunks in shared memory: the one before, the one computed with, the one prepared, two under way

struct WkvParams {
  const float* in[kVecs];
  const float* state_in;          // [B, N, H, H] or null (zeros)
  float* y;                       // [B, T, C]
  float* state_out;               // [B, N, H, H] or null
  float4* ckpt;                   // [B, N, ceil(T / kCk)][kTileQuads] float4 or null: the state before timesteps 0, kCk, 2*kCk, ... (tile layout)
  float* sa;                      // [B, T, C] or null: sa of every timestep, for the backward pass
  int T, N;                       // timesteps, heads
};

// the preparing warps and the others arrive from different places
__device__ __forceinline__ void cta_meet() { asm volatile("bar.sync 0;" ::: "memory"); }

struct WkvFwdChunk {
  float vec[kFwdChunk][kVecs][kH];      // decay, b (iclr as it arrives), removal_k, replacement_k, v, r
};

// a lane's share of one timestep's vectors
template <int ROWS, int PAIRS>
struct StepVecs {
  float2 w[PAIRS], b[PAIRS], kt[PAIRS];
  float v[ROWS];                  // register 0 is the row whose sums the lane ends with
};
// a lane's columns of a shared-memory vector: four, or four and four 32 further on
template <int PAIRS>
__device__ __forceinline__ void ld_cols(const float* p, float2 (&out)[PAIRS]) {
  const float4 t = *reinterpret_cast<const float4*>(p);
  out[0] = make_float2(t.x, t.y); out[1] = make_float2(t.z, t.w);
  if constexpr (PAIRS == 4) {
    const float4 u = *reinterpret_cast<const float4*>(p + 32);
    out[2] = make_float2(u.x, u.y); out[3] = make_float2(u.z, u.w);
  }
}

// sum over a lane's columns of S * x, row by row: four columns' sum, or two of those added as two lanes' are
template <int ROWS, int PAIRS>
__device__ __forceinline__ void row_dots(const float2 (&S)[ROWS][PAIRS], const float2 (&x)[PAIRS], float (&out)[ROWS]) {
  float2 p[ROWS], q[ROWS];
#pragma unroll
  for (int a = 0; a < ROWS; ++a) p[a] = __fmul2_rn(S[a][0], x[0]);
#pragma unroll
  for (int a = 0; a < ROWS; ++a) p[a] = __ffma2_rn(S[a][1], x[1], p[a]);
  if constexpr (PAIRS == 4) {
#pragma unroll
    for (int a = 0; a < ROWS; ++a) q[a] = __fmul2_rn(S[a][2], x[2]);
#pragma unroll
    for (int a = 0; a < ROWS; ++a) q[a] = __ffma2_rn(S[a][3], x[3], q[a]);
#pragma unroll
    for (int a = 0; a < ROWS; ++a) out[a] = (p[a].x + p[a].y) + (q[a].x + q[a].y);
  } else {
#pragma unroll
    for (int a = 0; a < ROWS; ++a) out[a] = p[a].x + p[a].y;
  }
}

// A warp's lanes are a grid of 32 / LANES x LANES.  SAVE: checkpoints and sa are wanted (a backward pass follows).  PREP warps prepare the
// chunks.
template <int ROWS, int LANES, int WARPS, int PREP, int PER_SM, bool SAVE>
__global__ void __launch_bounds__(32 * (WARPS + PREP), PER_SM)
wkv7_forward_kernel(const __grid_constant__ WkvParams p) {
  grid_wait();
  constexpr int kWarpRows = ROWS * (32 / LANES), kCtaRows = kWarpRows * WARPS, kCtasPerHead = kH / kCtaRows;
  constexpr int kPairs = kH / LANES / 2;        // float2 of a lane's row
  constexpr int kPrepSteps = kFwdChunk / PREP;
  constexpr int kSame = LANES / 2 / ROWS;       // lanes that end with the same row's sum
  constexpr int kSameBits = kSame == 1 ? 0 : (kSame == 2 ? 1 : 2);
  static_assert(kH % kCtaRows == 0 && kFwdChunk % PREP == 0 && (LANES == 8 || LANES == 16) && (ROWS << kSameBits) * 2 == LANES, "whole CTAs of rows, whole timesteps");
  extern __shared__ __align__(16) unsigned char wkv_fwd_smem[];
  WkvFwdChunk* const ring = reinterpret_cast<WkvFwdChunk*>(wkv_fwd_smem);
  const int head = blockIdx.x / kCtasPerHead;
  const int n = head % p.N, b = head / p.N;
  const int C = p.N * kH;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const size_t head_base = (size_t)b * p.T * C + (size_t)n * kH;      // element (b, t = 0, channel n*H)
  const int full = p.T / kFwdChunk, n_chunks = (p.T + kFwdChunk - 1) / kFwdChunk;

  constexpr bool kMoveRegs = WARPS == 4 && PREP == 4 && PER_SM == 2 && ROWS * LANES == 32;      // two CTAs of 256 threads: 128 registers each at launch
  if (warp >= WARPS) {
    if constexpr (kMoveRegs) asm volatile("setmaxnreg.dec.sync.aligned.u32 56;");
    // every thread commits one (possibly empty) group per chunk: its warp's timesteps, 6 vectors of 16 quarters of 16 bytes each
    const int s0 = (warp - WARPS) * kPrepSteps;
    auto issue = [&](int chunk) {
      WkvFwdChunk& to = ring[chunk % kFwdBufs];
#pragma unroll
      for (int i = 0; i < kPrepSteps * 3; ++i) {
        const int s = s0 + i / 3, v = 2 * (i % 3) + (lane >> 4), t = chunk * kFwdChunk + s;
        if (t < p.T) {
          const float* src = i % 3 == 0 ? (lane < 16 ? p.in[0] : p.in[1]) : (i % 3 == 1 ? (lane < 16 ? p.in[2] : p.in[3]) : (lane < 16 ? p.in[4] : p.in[5]));
          cp_async16((uint32_t)__cvta_generic_to_shared(&to.vec[s][v][(lane & 15) * 4]), src + head_base + (size_t)t * C + (lane & 15) * 4);
        }
      }
      cp_async_commit();
    };
    // b of the warp's own timesteps; a lane two columns.  (Timesteps past the sequence's end: what the buffer holds, which nothing reads.)
    auto prepare = [&](int chunk) {
      WkvFwdChunk& at = ring[chunk % kFwdBufs];
#pragma unroll
      for (int s = s0; s < s0 + kPrepSteps; ++s) {
        const float2 a = *reinterpret_cast<const float2*>(&at.vec[s][1][2 * lane]), kap = *reinterpret_cast<const float2*>(&at.vec[s][2][2 * lane]);
        *reinterpret_cast<float2*>(&at.vec[s][1][2 * lane]) = make_float2(a.x * kap.x, a.y * kap.y);
      }
    };
#pragma unroll
    for (int c = 0; c < kFwdBufs - 1; ++c) issue(c);
    cp_async_wait<kFwdBufs - 2>();
    __syncwarp();                               // the warp's vectors of chunk 0
    prepare(0);
    cta_meet();
    for (int c = 0; c < full; ++c) {
      cp_async_wait<kFwdBufs - 3>();
      __syncwarp();                             // the warp's vectors of chunk c + 1
      if (c + 1 < n_chunks) prepare(c + 1);
      cta_meet();                               // chunk c + 1 is ready, chunk c - 1 has been read
      issue(c + kFwdBufs - 1);
    }
    cp_async_wait<0>();
    return;
  }

  if constexpr (kMoveRegs) asm volatile("setmaxnreg.inc.sync.aligned.u32 200;");      // 128 * (56 + 200) = 256 * 128
  const int tj = lane & (LANES - 1), own_row = (tj & (LANES / 2 - 1)) >> kSameBits, part = tj & (kSame - 1);
  const bool for_y = tj & (LANES / 2);
  const int row0 = (blockIdx.x % kCtasPerHead) * kCtaRows + kWarpRows * warp + ROWS * (lane / LANES), col0 = 4 * tj;
  float2 S[ROWS][kPairs];
  const size_t shead = (size_t)head * kH * kH;
#pragma unroll
  for (int a = 0; a < ROWS; ++a) {
    if (p.state_in) {
#pragma unroll
      for (int k = 0; k < kPairs; k += 2) {
        const float4 t = __ldg(reinterpret_cast<const float4*>(p.state_in + shead + (row0 + (a ^ own_row)) * kH + col0 + 16 * k));
        S[a][k] = make_float2(t.x, t.y); S[a][k + 1] = make_float2(t.z, t.w);
      }
    } else {
#pragma unroll
      for (int k = 0; k < kPairs; ++k) S[a][k] = make_float2(0.0f, 0.0f);
    }
  }
  // A row's kSame lanes keep one timestep each of kSame and store together: y, and with a backward pass to follow sa
  const bool stores = for_y || (SAVE && p.sa);
  const long out_step = (long)kSame * C;
  float* out = (SAVE && stores && !for_y ? p.sa : p.y) + head_base + row0 + own_row + (long)part * C;      // of the next kSame timesteps the one that this lane keeps
  float keep = 0.0f;
  int from[ROWS];                               // the lane that makes sa of register a's row
#pragma unroll
  for (int a = 0; a < ROWS; ++a) from[a] = (lane & ~(LANES - 1)) | ((tj & (LANES / 2 - 1)) ^ (a << kSameBits));

  using Vecs = StepVecs<ROWS, kPairs>;
  auto load = [&](Vecs& x, const WkvFwdChunk& at, int s) {
    ld_cols(at.vec[s][0] + col0, x.w); ld_cols(at.vec[s][1] + col0, x.b); ld_cols(at.vec[s][3] + col0, x.kt);
#pragma unroll
    for (int a = 0; a < ROWS; ++a) x.v[a] = at.vec[s][4][row0 + (a ^ own_row)];
  };
  // A state's parts of sa of the next timestep and of y of its own, not yet summed over lanes: pa the lane's kept one, pb the other.
  float pa[ROWS], pb[ROWS];
  const int kept_at = (for_y ? kVecs - 1 : kVecs + 2) * kH + col0, other_at = (for_y ? kVecs + 2 : kVecs - 1) * kH + col0;      // from r's or the next timestep's kap
  // A row's sum over lanes: y's part goes to the lanes that keep y and sa's to the others, then the upper half of the registers left to
  // the lane that keeps those rows; the last one is added.
  auto sum_over_lanes = [&] {
    float got[ROWS];
#pragma unroll
    for (int a = 0; a < ROWS; ++a) got[a] = __shfl_xor_sync(0xffffffffu, pb[a], LANES / 2);
#pragma unroll
    for (int a = 0; a < ROWS; ++a) pa[a] += got[a];
    int left = ROWS;
#pragma unroll
    for (int m = LANES / 4; m >= 1; m /= 2) {
      const int gives = left > 1 ? left / 2 : 0;          // the first register that goes
      left = left > 1 ? left / 2 : 1;
#pragma unroll
      for (int a = 0; a < ROWS; ++a)
        if (a < left) got[a] = __shfl_xor_sync(0xffffffffu, pa[(a + gives) % ROWS], m);
#pragma unroll
      for (int a = 0; a < ROWS; ++a)
        if (a < left) pa[a] += got[a];
    }
    return pa[0];
  };

  float own = 0.0f;                             // -sa of the timestep before, of the row whose sums the lane ends with
  auto put = [&](int u, float val) {            // val: of a timestep, u = t % kSame
    if (part == u) keep = val;
    if (u == kSame - 1) {
      if (stores) *out = keep;
      out += out_step;
    }
  };
  Vecs cur, next;
  // Timestep s of chunk c: the sums over lanes of the last state's parts, sa to all lanes, the update, the new state's parts.  The
  // vectors that these want are read behind the shuffles (in front of them the shuffles queue behind the reads).
  auto step = [&](int c, int s) {
    const WkvFwdChunk& at = ring[c % kFwdBufs];
    const WkvFwdChunk& after = ring[(c + 1) % kFwdBufs];
    const float* const rec = &at.vec[s][0][0];
    const float sum = sum_over_lanes();         // y of the timestep before, or sa
    const float done = SAVE && !for_y ? -own : sum;
    own = -sum;
    float nsa[ROWS];                            // -sa of the lane's rows
#pragma unroll
    for (int a = 0; a < ROWS; ++a) nsa[a] = __shfl_sync(0xffffffffu, own, from[a]);
    float2 kept[kPairs], other[kPairs];
    if (s + 1 == kFwdChunk) {
      cta_meet();
      const float *kap = after.vec[0][2] + col0, *r = rec + (kVecs - 1) * kH + col0;
      ld_cols(for_y ? r : kap, kept);
      ld_cols(for_y ? kap : r, other);
      load(next, after, 0);
    } else {
      ld_cols(rec + kept_at, kept);
      ld_cols(rec + other_at, other);
      load(next, at, s + 1);
    }
    if (s > 0 || c > 0) put((s + kFwdChunk - 1) % kSame, done);
    float2 m[ROWS][kPairs];
#pragma unroll
    for (int a = 0; a < ROWS; ++a)
#pragma unroll
      for (int j = 0; j < kPairs; ++j) m[a][j] = __fmul2_rn(dup(nsa[a]), cur.b[j]);
#pragma unroll
    for (int j = 0; j < kPairs; ++j)
#pragma unroll
      for (int a = 0; a < ROWS; ++a) S[a][j] = __ffma2_rn(S[a][j], cur.w[j], m[a][j]);
#pragma unroll
    for (int a = 0; a < ROWS; ++a)
#pragma unroll
      for (int j = 0; j < kPairs; ++j) S[a][j] = __ffma2_rn(dup(cur.v[a]), cur.kt[j], S[a][j]);
    row_dots(S, other, pb);
    row_dots(S, kept, pa);
    cur = next;
  };
  auto checkpoint = [&](int c) {                // the state before the chunk (kCk == kFwdChunk), in the backward kernel's layout
    if constexpr (SAVE) {
      if (p.ckpt) {
        float4* ck = p.ckpt + ((size_t)head * n_chunks + c) * kTileQuads;
#pragma unroll
        for (int a = 0; a < ROWS; a += 2)
#pragma unroll
          for (int k = 0; k < kPairs; ++k) {
            const float2 e = own_row & 1 ? S[a + 1][k] : S[a][k], o = own_row & 1 ? S[a][k] : S[a + 1][k];
            ck[ckpt_quad((row0 + (a ^ own_row)) >> 1, (col0 >> 1) + (k & 1) + 16 * (k >> 1))] = make_float4(e.x, o.x, e.y, o.y);
          }
      }
    }
  };

  cta_meet();
  load(cur, ring[0], 0);
  {
    float2 kap[kPairs];
    ld_cols(ring[0].vec[0][2] + col0, kap);
    row_dots(S, kap, pa);
#pragma unroll
    for (int a = 0; a < ROWS; ++a) pb[a] = pa[a];         // y of no timestep: not stored
  }
  for (int c = 0; c < full; ++c) {
    checkpoint(c);
#pragma unroll
    for (int s = 0; s < kFwdChunk; ++s) step(c, s);
  }
  const int tail = p.T - full * kFwdChunk;
  if (tail) {
    checkpoint(full);
#pragma unroll 1
    for (int s = 0; s < tail; ++s) step(full, s);
  }
  // the last timestep's outputs are still open
  const float y_last = sum_over_lanes();
  const int u = (p.T - 1) % kSame;
  if (part == u) keep = SAVE && !for_y ? -own : y_last;
  if (part <= u && stores) *out = keep;
  if (p.state_out) {
#pragma unroll
    for (int a = 0; a < ROWS; ++a)
#pragma unroll
      for (int k = 0; k < kPairs; k += 2)
        *reinterpret_cast<float4*>(p.state_out + shead + (row0 + (a ^ own_row)) * kH + col0 + 16 * k) = make_float4(S[a][k].x, S[a][k].y, S[a][k + 1].x, S[a][k + 1].y);
  }
}

template <int ROWS, int LANES, int WARPS, int PREP, int PER_SM>
int launch_forward(const WkvParams& p, int64_t heads, cudaStream_t st) {
  const unsigned grid = (unsigned)(heads * (kH / (ROWS * (32 / LANES) * WARPS)));
  const int smem = kFwdBufs * (int)sizeof(WkvFwdChunk);
  auto go = [&](auto kernel) {
    PB_CUDA_TRY(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));   // per device
    launch_behind(kernel, grid, 32 * (WARPS + PREP), smem, st, p);
    PB_LAUNCH_CHECK("wkv7_forward_kernel");
    return (int)PB_OK;
  };
  if (p.ckpt || p.sa) return go(wkv7_forward_kernel<ROWS, LANES, WARPS, PREP, PER_SM, true>);
  return go(wkv7_forward_kernel<ROWS, LANES, WARPS, PREP, PER_SM, false>);
}

// ---- backward of the scan ------------------------------------------------------------------------------------
// With G_t = dS_t + dy_t r_t^T the gradient of the loss with respect to S_t (dS_t arriving from timestep t+1):
//     dr_t   = S_t^T dy_t                    dv_t  = G_t kt_t                 dkt_t = G_t^T v_t
//     dsa_t  = -G_t b_t   (b = a * kap)      db_t  = -G_t^T sa_t              dw_t  = sum_i G_t[i][:] * S_{t-1}[i][:]
//     dkap_t = S_{t-1}^T dsa_t + db_t * a_t  da_t  = db_t * kap_t             dS_{t-1} = G_t diag(w_t) + dsa_t kap_t^T
// Warp q owns rows 16q .. 16q+15; its lanes form a 2 x 16 grid and a lane keeps 8 rows (as float2 row pairs) x 4 columns of dS
// and of S_{t-1}: per timestep it reads 4 elements of five vectors and 8 of three, and a column's sum needs one shuffle.  dsa,
// the only sum that the recurrence waits for, goes first, and dv with it: the upper eight of a row's sixteen lanes hand over
// their parts of dsa for those of dv, four levels of shuffles instead of twice four, between the products of the sums that only
// leave the kernel, whose own shuffles go out together.  dr_t = S_t^T dy_t is formed a timestep later
// in the walk, where S_t is the state at hand: put together from S_{t-1} instead, w o (S_{t-1}^T dy) - b (sa . dy) + kt (v . dy),
// it loses what a timestep writes where it has just erased something larger.
//
// S_{t-1} is needed for every t and is not stored by the forward pass; inverting the recurrence would divide by the
// decay, which the reference lets go to zero.  The forward pass writes a checkpoint every kCk = 8 timesteps and
// sa_t for every t; with sa_t known the recurrence is element-wise, so every lane recomputes its own tile of the
// states from the checkpoint with no sums and no exchange: first to the state before timestep 4, from where the
// chunk's last four timesteps run backwards with three of their states in registers, then again for the first four.  The
// column sums of four timesteps wait in shared memory for one block barrier.  The chunk's eight vectors per timestep
// arrive by cp.async one chunk ahead, and the next checkpoint into the slot that the upper half has emptied.
//
// Bound by its f32x2 products, three cycles each where their operands are three different registers (some 1450 of the 1850
// cycles a timestep takes with two heads on an SM), and by what shuffles and shared memory return (half of their rate).
// 8 x 32 heads x 1024 timesteps 1577 -> 1030 us, 32 heads 1035 -> 698 us, against 4 x 8 tiles with every state in shared memory
// and a barrier per timestep; 256 heads 1016 -> 994, 32 heads 685 -> 663 by the sums' shuffles as above, 988 and 661 by stores of
// column sums to all banks, 979 and 650 by -b made once per chunk, 965 and 635 by the erasure's products (below).
struct WkvBwdParams {
  const float* in[kVecs];
  const float* dy;                // [B, T, C]
  const float* sa;                // [B, T, C]: S_{t-1} kap_t, from the forward pass
  const float4* ckpt;             // as the forward pass wrote it
  const float* dstate_out;        // [B, N, H, H] or null: gradient with respect to the final state
  float* din[kVecs];              // gradients of the six inputs, [B, T, C] each
  float* dstate_in;               // [B, N, H, H] or null: gradient with respect to the initial state
  int T, N;
};

struct WkvBwdSmem {
  float4 slot[2][kTileQuads];               // every thread its own quads: the chunk's checkpoint, and the state before its timestep 4
  float vec[2][kCk][kBwdSlots][kH];         // the chunk's vectors and -b, two chunks
  float col_part[2][kSub][kWarps][5][kH];   // two halves of a chunk: [timestep][warp][S^T dy of the timestep before, dkt, sum G sa, dw, S^T dsa][column]
  float dy_before[2][kH];                   // dy of the timestep before the chunk, two chunks (the first has none: what it reads is dropped)
  float last_part[kWarps][kH];              // S^T dy of the last timestep, a warp's rows each
};

// A lane's tile: the row pairs rp of rows row0 + 2 rp, + 1 by the columns col0 + c.
using BwdTile = float2[4][4];

__device__ __forceinline__ void load_quads(const float4* base, int tid, BwdTile& S) {
#pragma unroll
  for (int q = 0; q < 8; ++q) {
    const float4 t = base[q * kThreads + tid];
    S[q >> 1][2 * (q & 1)] = make_float2(t.x, t.y); S[q >> 1][2 * (q & 1) + 1] = make_float2(t.z, t.w);
  }
}
__device__ __forceinline__ void store_quads(float4* base, int tid, const BwdTile& S) {
#pragma unroll
  for (int q = 0; q < 8; ++q) {
    const float2 l = S[q >> 1][2 * (q & 1)], r = S[q >> 1][2 * (q & 1) + 1];
    base[q * kThreads + tid] = make_float4(l.x, l.y, r.x, r.y);
  }
}
// eight rows' values as row pairs
__device__ __forceinline__ void ld_rows(const float* p, float2 (&out)[4]) {
  const float4 lo = *reinterpret_cast<const float4*>(p), hi = *reinterpret_cast<const float4*>(p + 4);
  out[0] = make_float2(lo.x, lo.y); out[1] = make_float2(lo.z, lo.w); out[2] = make_float2(hi.x, hi.y); out[3] = make_float2(hi.z, hi.w);
}
// sum over a lane's rows of M * x, column by column, each still as a row pair
__device__ __forceinline__ void column_sums(const BwdTile& M, const float2 (&x)[4], float2 (&sum)[4]) {
#pragma unroll
  for (int c = 0; c < 4; ++c) sum[c] = __fmul2_rn(M[0][c], x[0]);
#pragma unroll
  for (int rp = 1; rp < 4; ++rp)
#pragma unroll
    for (int c = 0; c < 4; ++c) sum[c] = __ffma2_rn(M[rp][c], x[rp], sum[c]);
}
// sum over a lane's columns of M * x, row by row
__device__ __forceinline__ void row_sums(const BwdTile& M, float4 x, float2 (&sum)[4]) {
  const float2 x2[4] = {dup(x.x), dup(x.y), dup(x.z), dup(x.w)};
#pragma unroll
  for (int rp = 0; rp < 4; ++rp) sum[rp] = __fmul2_rn(M[rp][0], x2[0]);
#pragma unroll
  for (int c = 1; c < 4; ++c)
#pragma unroll
    for (int rp = 0; rp < 4; ++rp) sum[rp] = __ffma2_rn(M[rp][c], x2[c], sum[rp]);
}
__device__ __forceinline__ float2 from_lane_xor(float2 v, int mask) {
  return make_float2(__shfl_xor_sync(0xffffffffu, v.x, mask), __shfl_xor_sync(0xffffffffu, v.y, mask));
}
__device__ __forceinline__ float2 plus(float2 a, float2 b) { return make_float2(a.x + b.x, a.y + b.y); }
// Four column sums over the two lanes of a tile column: a lane ends with columns 2 tc, 2 tc + 1, and gives the other two away.
struct ColumnPair { float2 keep, give; };
__device__ __forceinline__ ColumnPair split_columns(const float2 (&v)[4], int tc) {
  const float2 lo = make_float2(v[0].x + v[0].y, v[1].x + v[1].y), hi = make_float2(v[2].x + v[2].y, v[3].x + v[3].y);
  return tc ? ColumnPair{hi, lo} : ColumnPair{lo, hi};
}

__global__ void __launch_bounds__(kThreads, 2)
wkv7_backward_kernel(const __grid_constant__ WkvBwdParams p) {
  grid_wait();
  extern __shared__ __align__(16) unsigned char wkv_bwd_smem[];
  WkvBwdSmem& sm = *reinterpret_cast<WkvBwdSmem*>(wkv_bwd_smem);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int ti = lane >> 4, tj = lane & 15, row0 = 16 * warp + 8 * ti, col0 = 4 * tj;
  const int tc = ti ^ (tj >> 3);  // which two of its four columns a lane's sums end with: sixteen lanes then store to all banks
  const int n = blockIdx.x % p.N, b = blockIdx.x / p.N;
  const int C = p.N * kH;
  const size_t head_base = (size_t)b * p.T * C + (size_t)n * kH;
  const size_t head = (size_t)b * p.N + n;
  const int n_ck = (p.T + kCk - 1) / kCk;

  BwdTile dS;
#pragma unroll
  for (int rp = 0; rp < 4; ++rp) {
    float4 e = make_float4(0.f, 0.f, 0.f, 0.f), o = e;
    if (p.dstate_out) {
      e = __ldg(reinterpret_cast<const float4*>(p.dstate_out + head * kH * kH + (row0 + 2 * rp) * kH + col0));
      o = __ldg(reinterpret_cast<const float4*>(p.dstate_out + head * kH * kH + (row0 + 2 * rp + 1) * kH + col0));
    }
    dS[rp][0] = make_float2(e.x, o.x); dS[rp][1] = make_float2(e.y, o.y); dS[rp][2] = make_float2(e.z, o.z); dS[rp][3] = make_float2(e.w, o.w);
  }

  // the eight vectors of every timestep of chunk ck -> vec[ck & 1]; every thread commits one group per call
  auto issue_vec = [&](int ck) {
    if (ck >= 0) {
      const int s = tid >> 4, t = ck * kCk + s;              // a timestep per sixteen threads
      if (t < p.T) {
        const size_t at = head_base + (size_t)t * C + (tid & 15) * 4;
#pragma unroll
        for (int v = 0; v < kBwdVecs; ++v)
          cp_async16((uint32_t)__cvta_generic_to_shared(&sm.vec[ck & 1][s][v][(tid & 15) * 4]), (v < kVecs ? p.in[v] : (v == kVecs ? p.dy : p.sa)) + at);
        if (s == 0 && t > 0) cp_async16((uint32_t)__cvta_generic_to_shared(&sm.dy_before[ck & 1][(tid & 15) * 4]), p.dy + at - C);
      }
    }
    cp_async_commit();
  };
  // checkpoint ck -> slot; the thread that copies is the thread that reads, so its own cp.async wait is all the ordering this needs
  auto prefetch_ckpt = [&](int ck, int slot) {
    if (ck >= 0) {
      const float4* src = p.ckpt + (head * n_ck + ck) * kTileQuads;
#pragma unroll
      for (int q = 0; q < 8; ++q)
        cp_async16((uint32_t)__cvta_generic_to_shared(&sm.slot[slot][q * kThreads + tid]), src + q * kThreads + tid);
    }
    cp_async_commit();
  };
  // to = from * w - sa b^T + v kt^T on the tile, rounded as the forward pass rounds it.  The erasure's products one at a time: a
  // packed one wants its column twice, and 256 heads x 1024 timesteps were then 976 us against 957 (other products
  // one at a time as well: 956 to 1011).
  auto update = [&](const float (*buf)[kH], const BwdTile& from, BwdTile& to) {
    const float4 w4 = *reinterpret_cast<const float4*>(buf[0] + col0), b4 = *reinterpret_cast<const float4*>(buf[kNegB] + col0);
    const float4 t4 = *reinterpret_cast<const float4*>(buf[3] + col0);
    const float2 w[4] = {dup(w4.x), dup(w4.y), dup(w4.z), dup(w4.w)}, kt[4] = {dup(t4.x), dup(t4.y), dup(t4.z), dup(t4.w)};
    const float nb[4] = {b4.x, b4.y, b4.z, b4.w};
    float2 v[4], sa[4];
    ld_rows(buf[4] + row0, v); ld_rows(buf[kVecs + 1] + row0, sa);
#pragma unroll
    for (int c = 0; c < 4; ++c)
#pragma unroll
      for (int rp = 0; rp < 4; ++rp) to[rp][c] = __ffma2_rn(from[rp][c], w[c], make_float2(sa[rp].x * nb[c], sa[rp].y * nb[c]));
#pragma unroll
    for (int rp = 0; rp < 4; ++rp)
#pragma unroll
      for (int c = 0; c < 4; ++c) to[rp][c] = __ffma2_rn(v[rp], kt[c], to[rp][c]);
  };
  const bool upper = tj & 8;        // of the sixteen lanes of a tile row
  const int mine_at = (upper ? 3 : kNegB) * kH + col0, theirs_at = (upper ? kNegB : 3) * kH + col0, col = col0 + 2 * tc;
  float2 dy[4];                     // of the timestep that goes backwards next
  // One timestep backwards, S the state before it, which is also the one after the timestep before: dr of that one, whose dy
  // is at `dy_below`
  auto back = [&](const float (*buf)[kH], const float* dy_below, const BwdTile& S, float (*part)[kH], size_t out) {
    const float4 k4 = *reinterpret_cast<const float4*>(buf[2] + col0), r4 = *reinterpret_cast<const float4*>(buf[5] + col0);
    const float2 kap[4] = {dup(k4.x), dup(k4.y), dup(k4.z), dup(k4.w)}, r[4] = {dup(r4.x), dup(r4.y), dup(r4.z), dup(r4.w)};
    // G = dS + dy r^T
#pragma unroll
    for (int rp = 0; rp < 4; ++rp)
#pragma unroll
      for (int c = 0; c < 4; ++c) dS[rp][c] = __ffma2_rn(dy[rp], r[c], dS[rp][c]);
    // dsa = -G b and dv = G kt, summed over the sixteen lanes of a tile row together: the lower eight lanes keep dsa, the upper ones dv,
    // and every further level halves the rows.  The levels wait for shuffles between the products of the sums that only leave.
    float2 rows[4], away[4];
    row_sums(dS, *reinterpret_cast<const float4*>(buf[0] + theirs_at), away);
#pragma unroll
    for (int rp = 0; rp < 4; ++rp) away[rp] = from_lane_xor(away[rp], 8);
    row_sums(dS, *reinterpret_cast<const float4*>(buf[0] + mine_at), rows);
#pragma unroll
    for (int rp = 0; rp < 4; ++rp) rows[rp] = plus(rows[rp], away[rp]);
    const bool b2 = tj & 4, b1 = tj & 2, b0 = tj & 1;
    const float2 away0 = from_lane_xor(b2 ? rows[0] : rows[2], 4), away1 = from_lane_xor(b2 ? rows[1] : rows[3], 4);
    float2 x[4], dkt[4], db[4], dr[4], dw[4];
    ld_rows(buf[4] + row0, x);
    column_sums(dS, x, dkt);
    const float2 four0 = plus(b2 ? rows[2] : rows[0], away0), four1 = plus(b2 ? rows[3] : rows[1], away1);
    const float2 away2 = from_lane_xor(b1 ? four0 : four1, 2);
    ld_rows(buf[kVecs + 1] + row0, x);
    column_sums(dS, x, db);
    const float2 two = plus(b1 ? four1 : four0, away2);
    const float row_sum = (b0 ? two.y : two.x) + __shfl_xor_sync(0xffffffffu, b0 ? two.x : two.y, 1);       // of row tj & 7
#pragma unroll
    for (int c = 0; c < 4; ++c) dw[c] = __fmul2_rn(S[0][c], dS[0][c]);
#pragma unroll
    for (int rp = 1; rp < 4; ++rp)
#pragma unroll
      for (int c = 0; c < 4; ++c) dw[c] = __ffma2_rn(S[rp][c], dS[rp][c], dw[c]);
    float2 dsa[4];
#pragma unroll
    for (int rp = 0; rp < 4; ++rp) {
      dsa[rp].x = __shfl_sync(0xffffffffu, row_sum, (lane & 16) + 2 * rp);
      dsa[rp].y = __shfl_sync(0xffffffffu, row_sum, (lane & 16) + 2 * rp + 1);
    }
    if (upper) p.din[4][out + row0 + (tj & 7)] = row_sum;
    ld_rows(dy_below + row0, dy);
    column_sums(S, dy, dr);
    const ColumnPair left[4] = {split_columns(dr, tc), split_columns(dkt, tc), split_columns(db, tc), split_columns(dw, tc)};
    float2 got[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) got[q] = from_lane_xor(left[q].give, 16);
    const float4 w4 = *reinterpret_cast<const float4*>(buf[0] + col0);
    const float2 w[4] = {dup(w4.x), dup(w4.y), dup(w4.z), dup(w4.w)};
    float2 dkap[4];
#pragma unroll
    for (int rp = 0; rp < 4; ++rp)
#pragma unroll
      for (int c = 0; c < 4; ++c) dS[rp][c] = __fmul2_rn(dS[rp][c], w[c]);
    column_sums(S, dsa, dkap);
    const ColumnPair last = split_columns(dkap, tc);
    *reinterpret_cast<float2*>(part[4] + col) = plus(last.keep, from_lane_xor(last.give, 16));
#pragma unroll
    for (int rp = 0; rp < 4; ++rp)
#pragma unroll
      for (int c = 0; c < 4; ++c) dS[rp][c] = __ffma2_rn(dsa[rp], kap[c], dS[rp][c]);
#pragma unroll
    for (int q = 0; q < 4; ++q) *reinterpret_cast<float2*>(part[q] + col) = plus(left[q].keep, got[q]);
  };
  // The column sums of the half chunk's timesteps [lo, hi): every warp's part is in shared memory behind the barrier.  (The
  // other buffer is written by the next half, and this one again only behind that half's barrier.)
  auto finish_columns = [&](const float (*V)[kBwdSlots][kH], const float (*part)[kWarps][5][kH], int t0, int lo, int hi) {
    __syncthreads();
    const int j = tid & (kH - 1);
    for (int s = lo + (tid >> 6); s < hi; s += 2) {
      float sum[5];
#pragma unroll
      for (int q = 0; q < 5; ++q) {
        sum[q] = part[s - lo][0][q][j];
#pragma unroll
        for (int w = 1; w < kWarps; ++w) sum[q] += part[s - lo][w][q][j];
      }
      const size_t out = head_base + (size_t)(t0 + s) * C + j;
      const float a = V[s][1][j], kap = V[s][2][j];
      if (t0 + s > 0) p.din[5][out - C] = sum[0];
      p.din[3][out] = sum[1];
      p.din[0][out] = sum[3];
      p.din[1][out] = -sum[2] * kap;
      p.din[2][out] = sum[4] - sum[2] * a;
    }
  };
  // Timesteps lo .. lo + count - 1 backwards, `first` holding the state before lo; the later ones' states stay in registers.
  auto run_half = [&](const float (*V)[kBwdSlots][kH], const float* dy_below, const float4* first, int t0, int lo, int count, int half, BwdTile& S1) {
    float (*part)[kWarps][5][kH] = sm.col_part[half];
    const size_t out = head_base + (size_t)(t0 + lo) * C;
    BwdTile S2, S3;                   // S1 comes as the state before lo
    if (count > 1) update(V[lo], S1, S1);
    if (count > 2) update(V[lo + 1], S1, S2);
    if (count > 3) {
      update(V[lo + 2], S2, S3);
      back(V[lo + 3], V[lo + 2][kVecs], S3, part[3][warp], out + 3 * (size_t)C);
    }
    if (count > 2) back(V[lo + 2], V[lo + 1][kVecs], S2, part[2][warp], out + 2 * (size_t)C);
    if (count > 1) back(V[lo + 1], V[lo][kVecs], S1, part[1][warp], out + (size_t)C);
    load_quads(first, tid, S1);
    back(V[lo], dy_below, S1, part[0][warp], out);
  };

  issue_vec(n_ck - 1);
  int ck_slot = 0;                // the slot of the current chunk's checkpoint; the other takes the state before timestep 4
  prefetch_ckpt(n_ck - 1, ck_slot);
  for (int ck = n_ck - 1; ck >= 0; --ck) {
    const int t0 = ck * kCk, steps = min(kCk, p.T - t0);
    __syncthreads();              // everyone is done with the vectors of the chunk after this one
    issue_vec(ck - 1);            // into the buffer that chunk used
    cp_async_wait<1>();           // this thread's copies of chunk ck, and of its checkpoint, have landed
    if (t0 + (tid >> 4) < p.T) {  // a thread's own copies: -b of those columns
      float (*mine)[kH] = sm.vec[ck & 1][tid >> 4];
      const float4 a4 = *reinterpret_cast<const float4*>(&mine[1][(tid & 15) * 4]), k4 = *reinterpret_cast<const float4*>(&mine[2][(tid & 15) * 4]);
      *reinterpret_cast<float4*>(&mine[kNegB][(tid & 15) * 4]) = make_float4(-(a4.x * k4.x), -(a4.y * k4.y), -(a4.z * k4.z), -(a4.w * k4.w));
    }
    __syncthreads();              // ... and everyone's vectors
    const float (*V)[kBwdSlots][kH] = sm.vec[ck & 1];
    if (ck == n_ck - 1) {         // the last timestep's dr takes the final state
      BwdTile S;
      load_quads(sm.slot[ck_slot], tid, S);
#pragma unroll 1
      for (int s = 0; s < steps; ++s) update(V[s], S, S);
      ld_rows(V[steps - 1][kVecs] + row0, dy);
      float2 sum[4];
      column_sums(S, dy, sum);
      const ColumnPair pair = split_columns(sum, tc);
      *reinterpret_cast<float2*>(sm.last_part[warp] + col) = plus(pair.keep, from_lane_xor(pair.give, 16));
      __syncthreads();
      if (tid < kH) {
        float r = sm.last_part[0][tid];
#pragma unroll
        for (int w = 1; w < kWarps; ++w) r += sm.last_part[w][tid];
        p.din[5][head_base + (size_t)(p.T - 1) * C + tid] = r;
      }
    }
    // The upper half chunk, then the lower one, through the same instructions: written out for each, they are twice what the
    // instruction cache holds (a tenth of the warps' stalls were for instructions): 256 heads x
    // 1024 timesteps 1121 -> 1045 us, 128 heads 799 -> 716; 32 heads, whose four warps an SM hide less, 646 -> 675.
#pragma unroll 1
    for (int half = steps > kSub; half >= 0; --half) {
      BwdTile S;
      load_quads(sm.slot[ck_slot], tid, S);
      if (half) {
#pragma unroll 1
        for (int s = 0; s < kSub; ++s) update(V[s], S, S);
        store_quads(sm.slot[ck_slot ^ 1], tid, S);
      } else {
        prefetch_ckpt(ck - 1, ck_slot ^ 1);    // the state in that slot has been read
      }
      const int lo = half * kSub, hi = min(steps, lo + kSub);
      run_half(V, half ? V[kSub - 1][kVecs] : sm.dy_before[ck & 1], sm.slot[half ? ck_slot ^ 1 : ck_slot], t0, lo, hi - lo, half, S);
      finish_columns(V, sm.col_part[half], t0, lo, hi);
    }
    ck_slot ^= 1;
  }
  cp_async_wait<0>();
  if (p.dstate_in) {
#pragma unroll
    for (int rp = 0; rp < 4; ++rp) {
      float* m = p.dstate_in + head * kH * kH + (row0 + 2 * rp) * kH + col0;
      *reinterpret_cast<float4*>(m) = make_float4(dS[rp][0].x, dS[rp][1].x, dS[rp][2].x, dS[rp][3].x);
      *reinterpret_cast<float4*>(m + kH) = make_float4(dS[rp][0].y, dS[rp][1].y, dS[rp][2].y, dS[rp][3].y);
    }
  }
}

}  // namespace
}  // namespace pb

using namespace pb;

extern "C" int pb_wkv7_forward(const float* decay, const float* iclr, const float* removal_k, const float* replacement_k,
                               const float* v, const float* r, const float* state_in,
                               int64_t batch, int64_t steps, int64_t heads, int head_dim,
                               float* y, float* state_out, float* checkpoints, float* sa, void* stream) {
  if (!decay || !iclr || !removal_k || !replacement_k || !v || !r || !y)
    return fail(PB_ERR_NULL_POINTER, "pb_wkv7_forward: the six inputs and y must be non-null");
  if (head_dim != kH) return fail(PB_ERR_UNSUPPORTED, "pb_wkv7_forward: head size %d (this kernel is built for %d)", head_dim, kH);
  if (batch <= 0 || steps <= 0 || heads <= 0 || batch * heads > 0x7fffffffll || steps > 0x7fffffffll)
    return fail(PB_ERR_BAD_SHAPE, "pb_wkv7_forward: batch=%lld steps=%lld heads=%lld", (long long)batch, (long long)steps, (long long)heads);
  const void* ptrs[] = {decay, iclr, removal_k, replacement_k, v, r, state_in, state_out, checkpoints, sa};
  for (const void* ptr : ptrs)
    if (reinterpret_cast<uintptr_t>(ptr) & 15) return fail(PB_ERR_MISALIGNED, "pb_wkv7_forward: every array must be 16-byte aligned");
  WkvParams p{{decay, iclr, removal_k, replacement_k, v, r}, state_in, y, state_out, reinterpret_cast<float4*>(checkpoints), sa, (int)steps, (int)heads};
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const int64_t n = batch * heads;
  // Rows of a head per CTA: 16, 32 or 64, as many CTAs as there are SMs and no more of them on one (each reads the head's vectors);
  // from a wave of whole heads to one and a half, three halves on an SM instead of two heads.  1024 timesteps, us, of the forms 16 |
  // 32 | halves | 64: 37 heads 125 | 144 | 177 | 199, 74 heads 171 | 145 | 177 | 198, 96 heads 289 | 217 | 302 | 198, 160 heads 451 | 346 |
  // 327 | 338 (with saves 479 | 378 | 359 | 391), 222 heads 507 | 345 | 327 | 336 (537 | 378 | 360 | 389), 256 heads 616 | 428 | 434 | 335.
  if (4 * n <= sm_count()) return launch_forward<2, 16, 4, 4, 1>(p, n, st);
  if (2 * n <= sm_count()) return launch_forward<4, 16, 4, 4, 1>(p, n, st);
  if (n > sm_count() && 2 * n <= 3 * sm_count()) return launch_forward<4, 8, 2, 2, 3>(p, n, st);
  return launch_forward<4, 8, 4, 4, 2>(p, n, st);
}

extern "C" size_t pb_wkv7_checkpoint_floats(int64_t batch, int64_t steps, int64_t heads, int head_dim) {
  if (batch <= 0 || steps <= 0 || heads <= 0 || head_dim != kH) return 0;
  return (size_t)batch * heads * ((steps + kCk - 1) / kCk) * kH * kH;
}

extern "C" int pb_wkv7_backward(const float* decay, const float* iclr, const float* removal_k, const float* replacement_k,
                                const float* v, const float* r, const float* checkpoints, const float* sa, const float* dy, const float* dstate_out,
                                int64_t batch, int64_t steps, int64_t heads, int head_dim,
                                float* d_decay, float* d_iclr, float* d_removal_k, float* d_replacement_k, float* d_v, float* d_r,
                                float* dstate_in, void* stream) {
  if (!decay || !iclr || !removal_k || !replacement_k || !v || !r || !checkpoints || !sa || !dy || !d_decay || !d_iclr || !d_removal_k ||
      !d_replacement_k || !d_v || !d_r)
    return fail(PB_ERR_NULL_POINTER, "pb_wkv7_backward: the six inputs, the checkpoints, sa, dy and the six gradients must be non-null");
  if (head_dim != kH) return fail(PB_ERR_UNSUPPORTED, "pb_wkv7_backward: head size %d (this kernel is built for %d)", head_dim, kH);
  if (batch <= 0 || steps <= 0 || heads <= 0 || batch * heads > 0x7fffffffll || steps > 0x7fffffffll)
    return fail(PB_ERR_BAD_SHAPE, "pb_wkv7_backward: batch=%lld steps=%lld heads=%lld", (long long)batch, (long long)steps, (long long)heads);
  const void* ptrs[] = {decay, iclr, removal_k, replacement_k, v, r, checkpoints, sa, dy, dstate_out, dstate_in};
  for (const void* ptr : ptrs)
    if (reinterpret_cast<uintptr_t>(ptr) & 15) return fail(PB_ERR_MISALIGNED, "pb_wkv7_backward: every array must be 16-byte aligned");
  WkvBwdParams p{{decay, iclr, removal_k, replacement_k, v, r}, dy, sa, reinterpret_cast<const float4*>(checkpoints), dstate_out,
                 {d_decay, d_iclr, d_removal_k, d_replacement_k, d_v, d_r}, dstate_in, (int)steps, (int)heads};
  PB_CUDA_TRY(cudaFuncSetAttribute(wkv7_backward_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(WkvBwdSmem)));   // per device
  launch_behind(wkv7_backward_kernel, (unsigned)(batch * heads), kThreads, sizeof(WkvBwdSmem), static_cast<cudaStream_t>(stream), p);
  PB_LAUNCH_CHECK("wkv7_backward_kernel");
  return PB_OK;
}

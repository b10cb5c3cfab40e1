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
constexpr int kTileQuads = kH * kH / 4;  // float4 per state

__device__ __forceinline__ void cp_async16(uint32_t dst, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N> __device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

__device__ __forceinline__ float2 dup(float x) { return make_float2(x, x); }

// a lane's eight columns of a shared-memory vector (four at p, four at p + 32) as four float2
__device__ __forceinline__ void ld8(const float* p, float2 (&out)[4]) {
  const float4 lo = *reinterpret_cast<const float4*>(p), hi = *reinterpret_cast<const float4*>(p + 32);
  out[0] = make_float2(lo.x, lo.y); out[1] = make_float2(lo.z, lo.w); out[2] = make_float2(hi.x, hi.y); out[3] = make_float2(hi.z, hi.w);
}
// A state in the kernels' own layout (checkpoints in global memory, kept states in shared memory): 1024 quads, a quad the
// rows 2P, 2P + 1 of the columns 2Q, 2Q + 1 as ((2P, 2Q), (2P+1, 2Q), (2P, 2Q+1), (2P+1, 2Q+1)).  Backward thread
// 16 * (P >> 2) + (Q >> 1) keeps it as its quad 2 * (P & 3) + (Q & 1): consecutive threads, consecutive 16 bytes.
__device__ __forceinline__ int ckpt_quad(int P, int Q) { return (2 * (P & 3) + (Q & 1)) * kThreads + 16 * (P >> 2) + (Q >> 1); }

// ---- forward ---------------------------------------------------------------------------------------------------
// The rows of a head's state are independent of one another given the timestep's vectors, so a head's 64 rows are cut over
// warps, and where there are few heads over CTAs as well.  A warp owns 4 * ROWS rows on the backward pass's 4 x 8 lane grid:
// a lane keeps ROWS rows x 8 columns, a row's two dot products end in three xor-shuffles (the state's one only delays the
// warp, the output's one nothing).  No barrier inside a chunk of eight timesteps: the chunk's vectors arrive by cp.async two
// chunks ahead, a step's are in registers one step ahead, and S * w is formed while sa's shuffles are under way.  v kt^T comes
// last: added to a state that is about to be erased, its low bits would go with it.
// What bounds it: with few heads the latency of a timestep (dot product, three shuffles, update: 250 cycles); with many the
// f32x2 products, three cycles each where their operands are three different registers, and the 4 * (40 + ROWS) bytes per lane
// and timestep that the vector reads return, which more rows per lane spread over more of them.
// The order within a timestep keeps everything but that chain off it: sa of the next timestep is formed from the new state before
// y of this one, the vectors of the next are read behind sa's shuffles (in front of them the shuffles queue behind the reads), y's
// shuffles come a timestep late and behind the state's update, a lane stores a row's outputs once in 8 / ROWS timesteps, and the
// next chunk's first vectors are read before this one's last update, so that no chunk starts with an empty pipeline.
// 1024 timesteps, against y's dot product and the reads in front of sa's and a pipeline emptied every chunk: 16 heads 172 -> 125 us,
// 32 heads 173 -> 139 (with sa and checkpoints 197 -> 160), 60 heads 188 -> 165, 128 heads 247 -> 214, 256 heads 387 -> 347
// (474 -> 422) in graphs of repeated calls; 32 heads x 4096, called with L2 flushed in between, 685 -> 571.
constexpr int kFwdChunk = 8;      // timesteps between barriers
constexpr int kFwdBufs = 3;       // chunks in shared memory

struct WkvParams {
  const float* in[kVecs];
  const float* state_in;          // [B, N, H, H] or null (zeros)
  float* y;                       // [B, T, C]
  float* state_out;               // [B, N, H, H] or null
  float4* ckpt;                   // [B, N, ceil(T / kCk)][kTileQuads] float4 or null: the state before timesteps 0, kCk, 2*kCk, ... (tile layout)
  float* sa;                      // [B, T, C] or null: sa of every timestep, for the backward pass
  int T, N;                       // timesteps, heads
};

// a lane's share of one timestep's vectors
template <int ROWS>
struct StepVecs {
  float2 w[4], b[4], kap[4], kt[4], r[4];
  float v[ROWS];
  __device__ __forceinline__ void load(const float (*buf)[kH], int col0, int row0) {
    ld8(buf[2] + col0, kap);
    ld8(buf[0] + col0, w);
    ld8(buf[3] + col0, kt);
    ld8(buf[1] + col0, b);
    ld8(buf[5] + col0, r);
    if constexpr (ROWS == 4) {
      const float4 t = *reinterpret_cast<const float4*>(buf[4] + row0);
      v[0] = t.x; v[1] = t.y; v[2] = t.z; v[3] = t.w;
    } else if constexpr (ROWS == 1) {
      v[0] = buf[4][row0];
    } else {
      const float2 t = *reinterpret_cast<const float2*>(buf[4] + row0);
      v[0] = t.x; v[1] = t.y;
    }
  }
};

// The sums over the eight lanes of a tile row that a timestep ends with: sa for every lane (the state's update waits for it),
// y for the lanes that keep it, each lane ending with row own of its ROWS
template <int ROWS>
__device__ __forceinline__ void reduce_sa(float (&sa)[ROWS]) {
#pragma unroll
  for (int m = 1; m <= 4; m *= 2)
#pragma unroll
    for (int a = 0; a < ROWS; ++a) sa[a] += __shfl_xor_sync(0xffffffffu, sa[a], m);
}
template <int ROWS>
__device__ __forceinline__ float reduce_y(const float (&y)[ROWS], int tj) {
  const bool hi = tj & 4, mid = tj & 2;
  float k0;
  if constexpr (ROWS == 1) {
    k0 = y[0] + __shfl_xor_sync(0xffffffffu, y[0], 4);
    k0 += __shfl_xor_sync(0xffffffffu, k0, 2);
  } else if constexpr (ROWS == 2) {
    k0 = (hi ? y[1] : y[0]) + __shfl_xor_sync(0xffffffffu, hi ? y[0] : y[1], 4);
    k0 += __shfl_xor_sync(0xffffffffu, k0, 2);
  } else {
    const float s0 = hi ? y[0] : y[2], s1 = hi ? y[1] : y[3];
    k0 = hi ? y[2] : y[0];
    float k1 = hi ? y[3] : y[1];
    k0 += __shfl_xor_sync(0xffffffffu, s0, 4);
    k1 += __shfl_xor_sync(0xffffffffu, s1, 4);
    k0 = (mid ? k1 : k0) + __shfl_xor_sync(0xffffffffu, mid ? k0 : k1, 2);
  }
  return k0 + __shfl_xor_sync(0xffffffffu, k0, 1);
}
template <int ROWS>
__device__ __forceinline__ float pick_row(const float (&v)[ROWS], int a) {
  float r = v[0];
#pragma unroll
  for (int k = 1; k < ROWS; ++k) r = a == k ? v[k] : r;
  return r;
}
// sum over a lane's columns of S * x, row by row.  Loops over columns outside, rows inside: consecutive products share x.
template <int ROWS>
__device__ __forceinline__ void row_dots(const float2 (&S)[ROWS][4], const float2 (&x)[4], float (&out)[ROWS]) {
  float2 p[ROWS], q[ROWS];
#pragma unroll
  for (int a = 0; a < ROWS; ++a) p[a] = __fmul2_rn(S[a][0], x[0]);
#pragma unroll
  for (int a = 0; a < ROWS; ++a) q[a] = __fmul2_rn(S[a][2], x[2]);
#pragma unroll
  for (int a = 0; a < ROWS; ++a) p[a] = __ffma2_rn(S[a][1], x[1], p[a]);
#pragma unroll
  for (int a = 0; a < ROWS; ++a) q[a] = __ffma2_rn(S[a][3], x[3], q[a]);
#pragma unroll
  for (int a = 0; a < ROWS; ++a) out[a] = (p[a].x + p[a].y) + (q[a].x + q[a].y);
}


// S_t from S_{t-1} and sa
template <int ROWS>
__device__ __forceinline__ void update_state(float2 (&S)[ROWS][4], StepVecs<ROWS>& x, const float (&sa)[ROWS]) {
#pragma unroll
  for (int k = 0; k < 4; ++k) x.b[k] = __fmul2_rn(x.b[k], x.kap[k]);
#pragma unroll
  for (int k = 0; k < 4; ++k)
#pragma unroll
    for (int a = 0; a < ROWS; ++a) S[a][k] = __fmul2_rn(S[a][k], x.w[k]);
#pragma unroll
  for (int a = 0; a < ROWS; ++a) {
    const float2 nsa = dup(-sa[a]);
#pragma unroll
    for (int k = 0; k < 4; ++k) S[a][k] = __ffma2_rn(nsa, x.b[k], S[a][k]);
  }
#pragma unroll
  for (int a = 0; a < ROWS; ++a)
#pragma unroll
    for (int k = 0; k < 4; ++k) S[a][k] = __ffma2_rn(dup(x.v[a]), x.kt[k], S[a][k]);
}

// SAVE: checkpoints and sa are wanted (a backward pass follows).
template <int ROWS, int WARPS, bool SAVE>
__global__ void __launch_bounds__(32 * WARPS)
wkv7_forward_kernel(const __grid_constant__ WkvParams p) {
  constexpr int kFwdThreads = 32 * WARPS;
  constexpr int kCtaRows = 4 * ROWS * WARPS, kCtasPerHead = kH / kCtaRows;
  static_assert(kFwdThreads <= 16 * kFwdChunk && kH % kCtaRows == 0, "sixteen threads a timestep of a chunk; a head's rows in whole CTAs");
  __shared__ __align__(16) float ring[kFwdBufs][kFwdChunk][kVecs][kH];
  const int head = blockIdx.x / kCtasPerHead;
  const int n = head % p.N, b = head / p.N;
  const int C = p.N * kH;
  const int tid = threadIdx.x, lane = tid & 31, ti = lane >> 3, tj = lane & 7;
  const int row0 = (blockIdx.x % kCtasPerHead) * kCtaRows + 4 * ROWS * (tid >> 5) + ROWS * ti, col0 = 4 * tj;
  const size_t head_base = (size_t)b * p.T * C + (size_t)n * kH;      // element (b, t = 0, channel n*H)
  const int n_chunks = (p.T + kFwdChunk - 1) / kFwdChunk;

  // a chunk is 8 x 6 vectors of 16 quarters of 16 bytes; every thread commits one (possibly empty) group per call
  auto issue = [&](int chunk) {
    constexpr int kStepsAtOnce = kFwdThreads / 16;
#pragma unroll
    for (int s0 = 0; s0 < kFwdChunk; s0 += kStepsAtOnce) {
      const int s = s0 + (tid >> 4), t = chunk * kFwdChunk + s;
      if (t < p.T) {
        const size_t at = head_base + (size_t)t * C + (tid & 15) * 4;
#pragma unroll
        for (int v = 0; v < kVecs; ++v)
          cp_async16((uint32_t)__cvta_generic_to_shared(&ring[chunk % kFwdBufs][s][v][(tid & 15) * 4]), p.in[v] + at);
      }
    }
    cp_async_commit();
  };

  float2 S[ROWS][4];
  const size_t shead = (size_t)head * kH * kH;
#pragma unroll
  for (int a = 0; a < ROWS; ++a) {
    if (p.state_in) {
      const float4 lo = __ldg(reinterpret_cast<const float4*>(p.state_in + shead + (row0 + a) * kH + col0));
      const float4 hi = __ldg(reinterpret_cast<const float4*>(p.state_in + shead + (row0 + a) * kH + col0 + 32));
      S[a][0] = make_float2(lo.x, lo.y); S[a][1] = make_float2(lo.z, lo.w); S[a][2] = make_float2(hi.x, hi.y); S[a][3] = make_float2(hi.z, hi.w);
    } else {
#pragma unroll
      for (int k = 0; k < 4; ++k) S[a][k] = make_float2(0.0f, 0.0f);
    }
  }
  // four rows a lane: of the two lanes that end up with a row's y one stores it, and its neighbour sa, both a timestep late
  constexpr int kSame = 8 / ROWS;              // lanes with the same row
  const int own = tj / kSame, part = tj % kSame;
  float* const out = part == 0 ? p.y : (SAVE && part == 1 ? p.sa : nullptr);
  float* dst = out ? out + head_base + row0 + own : nullptr;
  float y[ROWS], sa[ROWS], sa_before = 0.0f, y_keep = 0.0f, sa_keep = 0.0f;
  constexpr bool kKeep = ROWS < 4;     // eight timesteps' stores of a lane become ROWS (two arrays: no fewer with four rows)
  // with kKeep: a row's kSame lanes keep one timestep each of kSame and store together
  float* const yp = p.y + head_base + row0 + own;
  float* const sp = SAVE && p.sa ? p.sa + head_base + row0 + own : nullptr;
#pragma unroll
  for (int a = 0; a < ROWS; ++a) y[a] = 0.0f;

  issue(0);
  issue(1);
  issue(2);
  cp_async_wait<2>();
  __syncthreads();
  StepVecs<ROWS> cur;
  cur.load(ring[0][0], col0, row0);
  row_dots<ROWS>(S, cur.kap, sa);
  for (int c = 0; c < n_chunks; ++c) {
    const float (*buf)[kVecs][kH] = ring[c % kFwdBufs];
    const float (*buf_next)[kVecs][kH] = ring[(c + 1) % kFwdBufs];
    if constexpr (SAVE && ROWS > 1) {
      if (p.ckpt) {                   // the state before the chunk (kCk == kFwdChunk), in the backward kernel's layout
        float4* ck = p.ckpt + ((size_t)head * n_chunks + c) * kTileQuads;
#pragma unroll
        for (int a = 0; a < ROWS; a += 2)
#pragma unroll
          for (int k = 0; k < 4; ++k)
            ck[ckpt_quad((row0 + a) >> 1, (col0 >> 1) + (k & 1) + 16 * (k >> 1))] = make_float4(S[a][k].x, S[a + 1][k].x, S[a][k].y, S[a + 1][k].y);
      }
    }
    const int steps = min(kFwdChunk, p.T - c * kFwdChunk);
#pragma unroll
    for (int s = 0; s < kFwdChunk; ++s) {
      if (s >= steps) break;
      StepVecs<ROWS> next;
      const bool last_step = s + 1 == kFwdChunk;
      if (last_step) {
        cp_async_wait<1>();
        __syncthreads();
      }
      const float (*from)[kH] = last_step ? buf_next[0] : buf[(s + 1) % kFwdChunk];
      if (last_step) issue(c + 3);
      reduce_sa<ROWS>(sa);
      next.load(from, col0, row0);
      float y_old[ROWS];
#pragma unroll
      for (int a = 0; a < ROWS; ++a) y_old[a] = y[a];
      update_state<ROWS>(S, cur, sa);
      float sa_next[ROWS];
      row_dots<ROWS>(S, next.kap, sa_next);
      row_dots<ROWS>(S, cur.r, y);
      const float y_before = reduce_y<ROWS>(y_old, tj);
      if constexpr (kKeep) {
        constexpr int kLast = kSame - 1;
        const int u = (s + kFwdChunk - 1) % kSame;           // of timestep c * 8 + s - 1
        if (part == u) { y_keep = y_before; if (SAVE) sa_keep = sa_before; }
        if (u == kLast && (s > 0 || c > 0)) {
          const long at = (long)(c * kFwdChunk + s - kSame + part) * C;
          yp[at] = y_keep;
          if (SAVE) if (sp) sp[at] = sa_keep;
        }
      } else if (dst && (s > 0 || c > 0)) {
        *dst = SAVE && part != 0 ? sa_before : y_before;
        dst += C;
      }
      if (SAVE) sa_before = pick_row<ROWS>(sa, own);
      cur = next;
#pragma unroll
      for (int a = 0; a < ROWS; ++a) sa[a] = sa_next[a];
    }
  }
  const float y_last = reduce_y<ROWS>(y, tj);
  if constexpr (kKeep) {
    const int last = (p.T - 1) % kSame;
    if (part == last) { y_keep = y_last; if (SAVE) sa_keep = sa_before; }
    if (part <= last) {
      const long at = (long)(p.T - 1 - last + part) * C;
      yp[at] = y_keep;
      if (SAVE) if (sp) sp[at] = sa_keep;
    }
  } else if (dst) *dst = SAVE && part != 0 ? sa_before : y_last;
  cp_async_wait<0>();
  if (p.state_out) {
#pragma unroll
    for (int a = 0; a < ROWS; ++a) {
      *reinterpret_cast<float4*>(p.state_out + shead + (row0 + a) * kH + col0) = make_float4(S[a][0].x, S[a][0].y, S[a][1].x, S[a][1].y);
      *reinterpret_cast<float4*>(p.state_out + shead + (row0 + a) * kH + col0 + 32) = make_float4(S[a][2].x, S[a][2].y, S[a][3].x, S[a][3].y);
    }
  }
}

template <int ROWS, int WARPS>
int launch_forward(const WkvParams& p, int64_t heads, cudaStream_t st) {
  const unsigned grid = (unsigned)(heads * (kH / (4 * ROWS * WARPS)));
  if constexpr (ROWS > 1) {       // a lane of one row has no row pair to put into a checkpoint
    if (p.ckpt || p.sa) {
      wkv7_forward_kernel<ROWS, WARPS, true><<<grid, 32 * WARPS, 0, st>>>(p);
      PB_LAUNCH_CHECK("wkv7_forward_kernel");
      return PB_OK;
    }
  }
  wkv7_forward_kernel<ROWS, WARPS, false><<<grid, 32 * WARPS, 0, st>>>(p);
  PB_LAUNCH_CHECK("wkv7_forward_kernel");
  return PB_OK;
}

// ---- backward of the scan ------------------------------------------------------------------------------------
// With G_t = dS_t + dy_t r_t^T the gradient of the loss with respect to S_t (dS_t arriving from timestep t+1):
//     dr_t   = S_t^T dy_t                    dv_t  = G_t kt_t                 dkt_t = G_t^T v_t
//     dsa_t  = -G_t b_t   (b = a * kap)      db_t  = -G_t^T sa_t              dw_t  = sum_i G_t[i][:] * S_{t-1}[i][:]
//     dkap_t = S_{t-1}^T dsa_t + db_t * a_t  da_t  = db_t * kap_t             dS_{t-1} = G_t diag(w_t) + dsa_t kap_t^T
// Warp q owns rows 16q .. 16q+15; its lanes form a 2 x 16 grid and a lane keeps 8 rows (as float2 row pairs) x 4 columns of dS
// and of S_{t-1}: per timestep it reads 4 elements of five vectors and 8 of three, and a column's sum needs one shuffle.  dsa,
// the only sum that the recurrence waits for, is reduced first (a reduce-scatter over the sixteen lanes and eight
// broadcasts), and everything that only leaves the kernel is formed behind it.  dr_t = S_t^T dy_t is formed a timestep later
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
// Bound by the bytes its shared-memory reads and shuffles return and by its f32x2 products, both near 1300 of the 1950 cycles
// a timestep takes with two heads on an SM.  8 x 32 heads x 1024 timesteps 1577 -> 1030 us, 32 heads 1035 -> 698 us, against
// 4 x 8 tiles with every state in shared memory and a barrier per timestep.
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
  float vec[2][kCk][kBwdVecs][kH];          // the chunk's vectors, two chunks
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
// Eight row values over the sixteen lanes of a tile row: lane tj ends with the sum of row tj >> 1.
__device__ __forceinline__ float rows_reduce_scatter(const float2 (&v)[4], int tj) {
  const bool b3 = tj & 8, b2 = tj & 4, b1 = tj & 2;
  float2 k0 = b3 ? v[2] : v[0], k1 = b3 ? v[3] : v[1];
  const float2 s0 = b3 ? v[0] : v[2], s1 = b3 ? v[1] : v[3];
  k0.x += __shfl_xor_sync(0xffffffffu, s0.x, 8); k0.y += __shfl_xor_sync(0xffffffffu, s0.y, 8);
  k1.x += __shfl_xor_sync(0xffffffffu, s1.x, 8); k1.y += __shfl_xor_sync(0xffffffffu, s1.y, 8);
  float2 k = b2 ? k1 : k0;
  const float2 s = b2 ? k0 : k1;
  k.x += __shfl_xor_sync(0xffffffffu, s.x, 4); k.y += __shfl_xor_sync(0xffffffffu, s.y, 4);
  float r = (b1 ? k.y : k.x) + __shfl_xor_sync(0xffffffffu, b1 ? k.x : k.y, 2);
  return r + __shfl_xor_sync(0xffffffffu, r, 1);
}
// Four column sums (each still as a row pair) over the two lanes of a tile column: lane ti ends with columns 2 ti, 2 ti + 1.
__device__ __forceinline__ float2 cols_reduce_scatter(const float2 (&v)[4], int ti) {
  const float c0 = v[0].x + v[0].y, c1 = v[1].x + v[1].y, c2 = v[2].x + v[2].y, c3 = v[3].x + v[3].y;
  return make_float2((ti ? c2 : c0) + __shfl_xor_sync(0xffffffffu, ti ? c0 : c2, 16), (ti ? c3 : c1) + __shfl_xor_sync(0xffffffffu, ti ? c1 : c3, 16));
}

__global__ void __launch_bounds__(kThreads, 2)
wkv7_backward_kernel(const __grid_constant__ WkvBwdParams p) {
  extern __shared__ __align__(16) unsigned char wkv_bwd_smem[];
  WkvBwdSmem& sm = *reinterpret_cast<WkvBwdSmem*>(wkv_bwd_smem);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int ti = lane >> 4, tj = lane & 15, row0 = 16 * warp + 8 * ti, col0 = 4 * tj;
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
  // to = from * w - sa b^T + v kt^T on the tile
  auto update = [&](const float (*buf)[kH], const BwdTile& from, BwdTile& to) {
    const float4 w4 = *reinterpret_cast<const float4*>(buf[0] + col0), a4 = *reinterpret_cast<const float4*>(buf[1] + col0);
    const float4 k4 = *reinterpret_cast<const float4*>(buf[2] + col0), t4 = *reinterpret_cast<const float4*>(buf[3] + col0);
    const float2 w[4] = {dup(w4.x), dup(w4.y), dup(w4.z), dup(w4.w)}, kt[4] = {dup(t4.x), dup(t4.y), dup(t4.z), dup(t4.w)};
    const float2 nb[4] = {dup(-(a4.x * k4.x)), dup(-(a4.y * k4.y)), dup(-(a4.z * k4.z)), dup(-(a4.w * k4.w))};
    float2 v[4], sa[4];
    ld_rows(buf[4] + row0, v); ld_rows(buf[kVecs + 1] + row0, sa);
#pragma unroll
    for (int c = 0; c < 4; ++c)
#pragma unroll
      for (int rp = 0; rp < 4; ++rp) to[rp][c] = __fmul2_rn(from[rp][c], w[c]);
#pragma unroll
    for (int rp = 0; rp < 4; ++rp)
#pragma unroll
      for (int c = 0; c < 4; ++c) to[rp][c] = __ffma2_rn(sa[rp], nb[c], to[rp][c]);
#pragma unroll
    for (int rp = 0; rp < 4; ++rp)
#pragma unroll
      for (int c = 0; c < 4; ++c) to[rp][c] = __ffma2_rn(v[rp], kt[c], to[rp][c]);
  };
  float2 dy[4];                     // of the timestep that goes backwards next
  // one timestep backwards, S the state before it, which is also the one after the timestep before: dr of that one, whose dy
  // is at `dy_below`
  auto back = [&](const float (*buf)[kH], const float* dy_below, const BwdTile& S, float (*part)[kH], size_t out) {
    float2 nb[4], kap[4], rds[4];
    {
      const float4 a4 = *reinterpret_cast<const float4*>(buf[1] + col0), k4 = *reinterpret_cast<const float4*>(buf[2] + col0);
      const float4 r4 = *reinterpret_cast<const float4*>(buf[5] + col0);
      kap[0] = dup(k4.x); kap[1] = dup(k4.y); kap[2] = dup(k4.z); kap[3] = dup(k4.w);
      nb[0] = dup(-(a4.x * k4.x)); nb[1] = dup(-(a4.y * k4.y)); nb[2] = dup(-(a4.z * k4.z)); nb[3] = dup(-(a4.w * k4.w));
      const float2 r[4] = {dup(r4.x), dup(r4.y), dup(r4.z), dup(r4.w)};
      // G = dS + dy r^T, and dsa = -G b: the only sum the recurrence waits for, so it goes first
#pragma unroll
      for (int rp = 0; rp < 4; ++rp)
#pragma unroll
        for (int c = 0; c < 4; ++c) dS[rp][c] = __ffma2_rn(dy[rp], r[c], dS[rp][c]);
#pragma unroll
      for (int rp = 0; rp < 4; ++rp) rds[rp] = __fmul2_rn(dS[rp][0], nb[0]);
#pragma unroll
      for (int c = 1; c < 4; ++c)
#pragma unroll
        for (int rp = 0; rp < 4; ++rp) rds[rp] = __ffma2_rn(dS[rp][c], nb[c], rds[rp]);
    }
    const float dsa_row = rows_reduce_scatter(rds, tj);
    float2 dsa[4];
#pragma unroll
    for (int rp = 0; rp < 4; ++rp) {
      dsa[rp].x = __shfl_sync(0xffffffffu, dsa_row, (lane & 16) + 4 * rp);
      dsa[rp].y = __shfl_sync(0xffffffffu, dsa_row, (lane & 16) + 4 * rp + 2);
    }
    const int col = col0 + 2 * ti;
    // the sums that only leave: dv along the rows, the others along the columns
    {
      float2 v[4], sum[4], dvp[4];
      ld_rows(buf[4] + row0, v);
      const float4 t4 = *reinterpret_cast<const float4*>(buf[3] + col0);
      const float2 kt[4] = {dup(t4.x), dup(t4.y), dup(t4.z), dup(t4.w)};
#pragma unroll
      for (int rp = 0; rp < 4; ++rp) dvp[rp] = __fmul2_rn(dS[rp][0], kt[0]);
#pragma unroll
      for (int c = 1; c < 4; ++c)
#pragma unroll
        for (int rp = 0; rp < 4; ++rp) dvp[rp] = __ffma2_rn(dS[rp][c], kt[c], dvp[rp]);
      const float dv = rows_reduce_scatter(dvp, tj);
      if (!(tj & 1)) p.din[4][out + row0 + (tj >> 1)] = dv;
#pragma unroll
      for (int c = 0; c < 4; ++c) sum[c] = __fmul2_rn(dS[0][c], v[0]);
#pragma unroll
      for (int rp = 1; rp < 4; ++rp)
#pragma unroll
        for (int c = 0; c < 4; ++c) sum[c] = __ffma2_rn(dS[rp][c], v[rp], sum[c]);
      *reinterpret_cast<float2*>(part[1] + col) = cols_reduce_scatter(sum, ti);
    }
    {
      float2 sa[4], sum[4];
      ld_rows(buf[kVecs + 1] + row0, sa);
#pragma unroll
      for (int c = 0; c < 4; ++c) sum[c] = __fmul2_rn(dS[0][c], sa[0]);
#pragma unroll
      for (int rp = 1; rp < 4; ++rp)
#pragma unroll
        for (int c = 0; c < 4; ++c) sum[c] = __ffma2_rn(dS[rp][c], sa[rp], sum[c]);
      *reinterpret_cast<float2*>(part[2] + col) = cols_reduce_scatter(sum, ti);
    }
    {
      float2 sum[4], dw[4];
      ld_rows(dy_below + row0, dy);
#pragma unroll
      for (int c = 0; c < 4; ++c) sum[c] = __fmul2_rn(S[0][c], dy[0]);
#pragma unroll
      for (int c = 0; c < 4; ++c) dw[c] = __fmul2_rn(S[0][c], dS[0][c]);
#pragma unroll
      for (int rp = 1; rp < 4; ++rp) {
#pragma unroll
        for (int c = 0; c < 4; ++c) sum[c] = __ffma2_rn(S[rp][c], dy[rp], sum[c]);
#pragma unroll
        for (int c = 0; c < 4; ++c) dw[c] = __ffma2_rn(S[rp][c], dS[rp][c], dw[c]);
      }
      *reinterpret_cast<float2*>(part[0] + col) = cols_reduce_scatter(sum, ti);
      *reinterpret_cast<float2*>(part[3] + col) = cols_reduce_scatter(dw, ti);
    }
    {
      const float4 w4 = *reinterpret_cast<const float4*>(buf[0] + col0);
      const float2 w[4] = {dup(w4.x), dup(w4.y), dup(w4.z), dup(w4.w)};
      float2 sum[4];
#pragma unroll
      for (int c = 0; c < 4; ++c)
#pragma unroll
        for (int rp = 0; rp < 4; ++rp) dS[rp][c] = __fmul2_rn(dS[rp][c], w[c]);
#pragma unroll
      for (int c = 0; c < 4; ++c) sum[c] = __fmul2_rn(S[0][c], dsa[0]);
#pragma unroll
      for (int rp = 0; rp < 4; ++rp) {
#pragma unroll
        for (int c = 0; c < 4; ++c) dS[rp][c] = __ffma2_rn(dsa[rp], kap[c], dS[rp][c]);
        if (rp > 0) {
#pragma unroll
          for (int c = 0; c < 4; ++c) sum[c] = __ffma2_rn(S[rp][c], dsa[rp], sum[c]);
        }
      }
      *reinterpret_cast<float2*>(part[4] + col) = cols_reduce_scatter(sum, ti);
    }
  };
  // The column sums of the half chunk's timesteps [lo, hi): every warp's part is in shared memory behind the barrier.  (The
  // other buffer is written by the next half, and this one again only behind that half's barrier.)
  auto finish_columns = [&](const float (*V)[kBwdVecs][kH], const float (*part)[kWarps][5][kH], int t0, int lo, int hi) {
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
  auto run_half = [&](const float (*V)[kBwdVecs][kH], const float* dy_below, const float4* first, int t0, int lo, int count, int half, BwdTile& S1) {
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
    __syncthreads();              // ... and everyone's vectors
    const float (*V)[kBwdVecs][kH] = sm.vec[ck & 1];
    if (ck == n_ck - 1) {         // the last timestep's dr takes the final state
      BwdTile S;
      load_quads(sm.slot[ck_slot], tid, S);
#pragma unroll 1
      for (int s = 0; s < steps; ++s) update(V[s], S, S);
      ld_rows(V[steps - 1][kVecs] + row0, dy);
      float2 sum[4];
#pragma unroll
      for (int c = 0; c < 4; ++c) sum[c] = __fmul2_rn(S[0][c], dy[0]);
#pragma unroll
      for (int rp = 1; rp < 4; ++rp)
#pragma unroll
        for (int c = 0; c < 4; ++c) sum[c] = __ffma2_rn(S[rp][c], dy[rp], sum[c]);
      *reinterpret_cast<float2*>(sm.last_part[warp] + col0 + 2 * ti) = cols_reduce_scatter(sum, ti);
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
  // 8 (one row a lane: no pair of rows for a checkpoint), 16, 32 or 64 rows of a head per CTA: as many CTAs as there are SMs, and no
  // more of them on one (each reads the head's vectors); 16 heads x 1024: 125 us with 8 rows, 139 with 16
  const int64_t n = batch * heads;
  if (8 * n <= sm_count() && !checkpoints && !sa) return launch_forward<1, 2>(p, n, st);
  if (4 * n <= sm_count()) return launch_forward<2, 2>(p, n, st);
  if (2 * n <= sm_count()) return launch_forward<2, 4>(p, n, st);
  // just over a wave of whole heads: quarters of them fill SMs more evenly (160 heads x 1024: 326 us for 350, with saves 358 for 425)
  if (n > sm_count() && 4 * n <= 5 * sm_count()) return launch_forward<2, 2>(p, n, st);
  return launch_forward<4, 4>(p, n, st);
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
  wkv7_backward_kernel<<<(unsigned)(batch * heads), kThreads, sizeof(WkvBwdSmem), static_cast<cudaStream_t>(stream)>>>(p);
  PB_LAUNCH_CHECK("wkv7_backward_kernel");
  return PB_OK;
}

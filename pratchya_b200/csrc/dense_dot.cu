// The f32 dots of a Linear's backward pass where no 128-deep scale block can carry the cotangent (a (128,1) weight, or a
// token count that is no multiple of 1024): one operand is an fp8 triple, the other a dense f32 cotangent g,
//     tokens == 0:  out[j, i] = sum_c g[j, c] * dq(Q)[i, c]      (dX = g W^T,  pratchya/_qualia/_qarr.py:620)
//     tokens == 1:  out[i, j] = sum_c dq(Q)[c, i] * g[c, j]      (dW = X^T g,  :621)
// which the reference computes as f32 dots on dequantized arrays (pratchya/_qualia/_qarr.py:616-640).
//
// The fp8 values are exact in bf16, and over a tile of 128 i their block scale depends on c alone (blocks are 128 wide in i):
// so the scale goes to the other operand, f = g * scale(c) in f32 (one rounding, where dequantizing rounds q * scale), and f
// is split into three bf16 terms, hi + mid + lo, which keep all 24 bits of it.  Every product of the contraction is then exact in
// three bf16 tensor-core products.  Their accumulator is emptied into f32 registers with an ordinary add every 32 of c (the
// tensor core's own additions do not round to nearest), so the sums are no worse than an f32 dot's: 2-norm
// errors of 1.0e-7 to 3.1e-7 against 64 bits for contractions of 37 to 8192, where the library's SGEMM has 1.1e-7 to 1.6e-6.
//
// The ends of the f32 range.  bf16's exponents are f32's, so below 2^-110 the three terms of an f would run into its subnormals,
// and scaling the cotangent before it meets a small fp8 value can pass f32's largest number where their product does not.  So
// f carries an exact factor of 2^40, which moves the first below anything that f32 holds, and the second to |g scale| near
// 2^87, where it shows: an f without a finite bf16 makes every sum that it enters infinite or NaN.  A thread whose sums
// are not all finite makes them again with f32 products of dequantized values, one after the other (infinite cotangents among them:
// their infinities and NaNs are then an f32 dot's).  The look at the sums is free, behind their stores; ranges kept by
// the converting warps instead cost 5 % (3000 tokens, 2048 x 2048, f32: dW 173 -> 182 us).
//
// A CTA makes 128 x 128 tiles of out, one after the other: eight warps convert (global loads into registers, scale, split, 128-byte
// swizzled tiles in shared memory: K-major for dX, with c outermost, as the operands lie in memory, for dW), four warps empty one pair of
// accumulators while the other fills and store finished tiles, and a lane of a warp of its own issues tcgen05.mma: as a lane of an
// emptying warp it was what a stage waited for (1200 cycles to issue a stage's twelve, 700 to empty one).  Where the tiles do not
// fill the SMs the contraction is cut, and the parts are added in order by a second kernel.
//
// What bounds it: shared memory's data path.  A stage takes 2400 cycles, of which the converting warps' stores, loads and shuffles hold
// it for 1000 and the tensor core's reads of both operands (three terms against the same fp8 tile) for 770; their shuffles
// queue behind the stores.  Prefetching g into L2 gained 2 us where g streams from HBM and lost one where it does not; two stages' loads
// under way, other orders of the conversions: nothing.  Against the first form (emptying warps that issued, an address computed for every store
// of a tile: 15000 cycles of a 58000-cycle CTA), us in a CUDA graph: 8192 tokens, f32, 2048 x 128 dX 62 -> 28, dW 40 -> 30, 128 x 2048 38 -> 35 and 41 -> 31; 704 tokens, 128 x 1024 15.0 -> 12.0, 19.0 -> 13.4; 64 tokens, 2048 x 128 9.6 -> 7.6, 8.5 -> 7.0;
// the same bits.
//
// Every tile converts what it reads, so an operand that many tiles share is converted many times: where 512 columns or more share
// it and there is enough to do, split_dot.cu makes it ready once (split_dot_pays: 3000 tokens, 2048 x 2048, bf16 cotangent, dX 141 -> 38 us,
// dW 178 -> 68).  Left to this form are few tokens, the low-rank layers' f32 cotangents and callers without the workspace.
#include <algorithm>
#include <atomic>
#include <type_traits>

#include "common.cuh"
#include "split_dot.cuh"

namespace pb {
namespace {

constexpr int kTile = 128;            // i and j per CTA
constexpr int kDepth = 64;            // c per stage; an accumulator takes 32 of them
constexpr int kStages = 2;
constexpr int kMinSplitDepth = 256;   // c per part: below this a part is mostly prologue
constexpr int kConvWarps = 8, kDrainWarps = 4, kIssueWarp = kConvWarps + kDrainWarps;
constexpr int kDotThreads = 512;      // 128 registers each at launch; the emptying warpgroup takes 216, the issuing one's three other warps have nothing to do
constexpr int kOpBytes = kTile * kDepth * 2;            // one bf16 operand tile: 128 rows of 128 bytes
constexpr int kStageBytes = 4 * kOpBytes;               // q, then f's lo, mid and hi
constexpr int kOutPitch = 4 * kTile + 16;                // bytes of a finished tile's row in shared memory
constexpr int kDotSmem = kStages * kStageBytes + kTile * kOutPitch + 1024;      // 1024: the tiles start on a swizzle atom
constexpr uint32_t kAccCols = 4 * kTile;                // tensor memory: two stages of two accumulators, each of half a stage's c
constexpr float kScaleUp = 0x1p40f, kScaleDown = 0x1p-40f;      // of f, and of its sums (see above)
constexpr uint32_t kWaitPolls = 1u << 21;               // a poll parks for up to 2 us: about four seconds at most

__device__ unsigned int g_dot_status; // 0, or PB_ERR_DEVICE_TIMEOUT once a bounded wait ran out

struct DotParams {
  const uint8_t* q; const uint8_t* sc8; const float* sc32;
  const void* g;                      // f32 or bf16
  float* out;                         // or the parts, [splits][out]
  int64_t ldq, ldg, ldo, part;        // row strides in elements; elements of out
  int I, J, C;                        // extents: i and j of out, and the contraction
  uint32_t nbc, log2_K;               // blocks per block row of the triple; blocks per super-group, a power of two
  int per_column;                     // tokens == 0: the blocks are (128,1), not (128,128)
  int i_tiles, tiles, items, split_depth;
#ifdef PB_DIAGNOSTICS
  uint32_t polls;                     // poll budget of every wait
  int withhold;                       // the first stage is filled and never announced: every role runs out of patience
#endif
};
#ifdef PB_DIAGNOSTICS
__device__ __forceinline__ uint32_t wait_polls(const DotParams& p) { return p.polls; }
#else
__device__ __forceinline__ uint32_t wait_polls(const DotParams&) { return kWaitPolls; }
#endif

__device__ __forceinline__ uint32_t dot_smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void bar_init(uint32_t bar, uint32_t count) { asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count)); }
__device__ __forceinline__ void bar_arrive(uint32_t bar) { asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory"); }
// Bounded: false, and the status word set, when the poll budget ran out.
__device__ __forceinline__ bool bar_wait(uint32_t bar, uint32_t parity, uint32_t polls) {
  for (uint32_t n = 0; n < polls; ++n) {
    uint32_t ok;
    asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, 2000;\n\tselp.u32 %0, 1, 0, p;\n\t}"
                 : "=r"(ok) : "r"(bar), "r"(parity) : "memory");
    if (ok) return true;
  }
  atomicExch(&g_dot_status, (unsigned int)PB_ERR_DEVICE_TIMEOUT);
  return false;
}
__device__ __forceinline__ void tc_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void commit_to(uint32_t bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}
// Operand tiles, 128-byte swizzle (descriptor version 1, layout 2).  TOKENS == false, K-major: rows of 128 bytes (64 of c), 8-row groups
// 1024 bytes apart.  TOKENS, c outermost, as the operands lie in memory: 64 rows of 128 bytes (64 of i or j), eight c 1024 bytes apart,
// the next 64 of i or j 8192.
template <bool TOKENS>
__device__ __forceinline__ uint64_t tile_desc(uint32_t smem_addr) {
  return (uint64_t)((smem_addr & 0x3ffffu) >> 4) | ((uint64_t)(TOKENS ? 8192 >> 4 : 1) << 16) | ((uint64_t)(1024 >> 4) << 32) | (1ull << 46) | (2ull << 61);
}
template <bool TOKENS> constexpr uint32_t kStep16 = TOKENS ? 16 * 128 / 16 : 32 / 16;      // 16 of c further, in descriptor units
// kind::f16: f32 accumulator, both operands bf16, both K-major or both not, N = M = 128
template <bool TOKENS>
constexpr uint32_t kDotInstr = (1u << 4) | (1u << 7) | (1u << 10) | (TOKENS ? 3u << 15 : 0u) | ((uint32_t)(kTile >> 3) << 17) | ((uint32_t)(kTile >> 4) << 24);
template <bool TOKENS>
__device__ __forceinline__ void mma_f16(uint32_t d, uint64_t a, uint64_t b, uint32_t accumulate) {
  asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\ttcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
               ::"r"(d), "l"(a), "l"(b), "r"(kDotInstr<TOKENS>), "r"(accumulate) : "memory");
}
__device__ __forceinline__ void ld_acc32(uint32_t taddr, uint32_t (&r)[32]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
      "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
        "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]),
        "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]),
        "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
      : "r"(taddr) : "memory");
}

// two fp8 bytes -> two bf16 (exact)
__device__ __forceinline__ uint32_t fp8x2_to_bf16x2(uint32_t v) {
  const float2 f = fp8x2_to_f32x2<PB_E4M3>((uint16_t)v);
  return pack_bf16x2(f.x, f.y);
}
// f = hi + mid + lo, two elements at a time.  An f that is no finite bf16 leaves NaN rests, and its sums are made again.
__device__ __forceinline__ void split3(float2 f, uint32_t& hi, uint32_t& mid, uint32_t& lo) {
  hi = pack_bf16x2(f.x, f.y);
  const float2 minus = make_float2(-1.0f, -1.0f);
  const float2 r = __ffma2_rn(make_float2(__uint_as_float(hi << 16), __uint_as_float(hi & 0xffff0000u)), minus, f);
  mid = pack_bf16x2(r.x, r.y);
  const float2 t = __ffma2_rn(make_float2(__uint_as_float(mid << 16), __uint_as_float(mid & 0xffff0000u)), minus, r);
  lo = pack_bf16x2(t.x, t.y);
}
// eight f of one chunk
__device__ __forceinline__ void split_chunk(const float (&g)[8], const float (&s)[8], uint32_t (&hi)[4], uint32_t (&mid)[4], uint32_t (&lo)[4]) {
#pragma unroll
  for (int e = 0; e < 4; ++e) split3(__fmul2_rn(make_float2(g[2 * e], g[2 * e + 1]), make_float2(s[2 * e], s[2 * e + 1])), hi[e], mid[e], lo[e]);
}
// byte offset of a 16-byte chunk of a swizzled tile: eight c of row i or j, or eight i or j of row c
template <bool TOKENS>
__device__ __forceinline__ uint32_t chunk_at(int row, int chunk) {
  if (TOKENS) return (uint32_t)(chunk >> 3) * 8192u + (uint32_t)row * 128u + (uint32_t)(((chunk & 7) ^ (row & 7)) << 4);
  return (uint32_t)row * 128u + (uint32_t)((chunk ^ (row & 7)) << 4);
}
__device__ __forceinline__ void st_chunk(uint32_t addr, uint32_t a, uint32_t b, uint32_t c, uint32_t d) {
  asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(addr), "r"(a), "r"(b), "r"(c), "r"(d));      // ordered by the fence at the stage's end
}

// What a converting thread holds of a stage: four chunks of g, two pairs of chunks of q, the scales of their c.
template <bool TOKENS, typename G>
struct StageRegs {
  static constexpr int kWords = sizeof(G) == 4 ? 8 : 4;
  static constexpr int kScales = TOKENS ? 4 : 8;      // it uses: TOKENS, of the rows of its chunks of g; else of the eight c of all of them
  uint32_t g[4][kWords];              // as loaded: f32, or two bf16
  __device__ __forceinline__ void chunk(int k, float (&f)[8]) const {
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      if constexpr (sizeof(G) == 4) f[e] = __uint_as_float(g[k][e]);
      else f[e] = __uint_as_float(e & 1 ? g[k][e / 2] & 0xffff0000u : g[k][e / 2] << 16);
    }
  }
  uint32_t q[8];                      // TOKENS: sixteen i of two c; else 32 c of a row
  uint32_t e8[2];                     // of the two c of a stage whose scales this lane makes for its warp
  float e32[2];
};

// what dequantizing multiplies a block's values by, before the exact 1/128
__device__ __forceinline__ float block_multiplier(uint32_t e8, float e32) { return __fmul_rn(e8m0_to_f32(e8), e32); }

// One emptying thread's 64 sums (row i, columns from jb) made and stored one f32 product after the other: the rare ones whose
// scaled cotangent has no finite bf16.  A call of its own, sixteen sums at a time, to leave the kernel's registers alone; the
// cotangents of a c are the same for a whole warp.
template <bool TOKENS, typename G>
__device__ __noinline__ void plain_dots(const DotParams& p, float* out, int i, int jb, int it, int c_begin, int c_end) {
  const G* g = static_cast<const G*>(p.g);
#pragma unroll 1
  for (int j0 = jb; j0 < jb + 64 && j0 < p.J; j0 += 16) {
    float acc[16];
#pragma unroll
    for (int n = 0; n < 16; ++n) acc[n] = 0.0f;
#pragma unroll 1
    for (int c = c_begin; c < c_end; ++c) {
      const uint8_t q = __ldg(p.q + (TOKENS ? (int64_t)c * p.ldq + i : (int64_t)i * p.ldq + c));
      const uint32_t id = TOKENS ? (uint32_t)c * p.nbc + it : (uint32_t)it * p.nbc + (p.per_column ? c : c / 128);
      const float x_sc = block_multiplier(__ldg(p.sc8 + id), __ldg(p.sc32 + (id >> p.log2_K)));
      const float x = __fmul_rn(__fmul_rn(fp8x2_to_f32x2<PB_E4M3>((uint16_t)q).x, x_sc), 0.0078125f);
      const G* at = g + (TOKENS ? (int64_t)c * p.ldg + j0 : (int64_t)j0 * p.ldg + c);
#pragma unroll
      for (int n = 0; n < 16; ++n) {
        const int k = min(n, p.J - 1 - j0);
        acc[n] = fmaf(Elem<G>::to_f32(at[TOKENS ? (int64_t)k : k * p.ldg]), x, acc[n]);
      }
    }
#pragma unroll
    for (int n = 0; n < 16; ++n)
      if (j0 + n < p.J) out[TOKENS ? (int64_t)i * p.ldo + j0 + n : (int64_t)(j0 + n) * p.ldo + i] = acc[n];
  }
}

// Where an item of the grid's work lies: a tile, and a part of the contraction.
struct DotItem {
  int it, i0, j0, c_begin, c_end, n_stages, split;
  __device__ __forceinline__ DotItem(const DotParams& p, int w) {
    split = w / p.tiles;
    const int tile = w - split * p.tiles;
    it = tile % p.i_tiles; i0 = it * kTile; j0 = (tile / p.i_tiles) * kTile;
    c_begin = split * p.split_depth; c_end = min(p.C, c_begin + p.split_depth);
    n_stages = (c_end - c_begin + kDepth - 1) / kDepth;
  }
};

template <bool TOKENS, typename G>
__global__ void __launch_bounds__(kDotThreads, 1) dense_dot_kernel(const __grid_constant__ DotParams p) {
  extern __shared__ unsigned char dot_smem[];
  __shared__ __align__(8) uint64_t bars[2 * kStages + 4];
  __shared__ uint32_t tmem_slot;
  const uint32_t tiles_base = (dot_smem_u32(dot_smem) + 1023u) & ~1023u, out_base = tiles_base + kStages * kStageBytes;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  auto full = [&](int s) { return dot_smem_u32(&bars[s]); };
  auto empty = [&](int s) { return dot_smem_u32(&bars[kStages + s]); };
  auto acc_full = [&](int a) { return dot_smem_u32(&bars[2 * kStages + a]); };
  auto acc_empty = [&](int a) { return dot_smem_u32(&bars[2 * kStages + 2 + a]); };

  if (tid == 0) {
    for (int s = 0; s < kStages; ++s) { bar_init(full(s), kConvWarps); bar_init(empty(s), 1); }
    for (int a = 0; a < 2; ++a) { bar_init(acc_full(a), 1); bar_init(acc_empty(a), kDrainWarps); }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == kIssueWarp) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(dot_smem_u32(&tmem_slot)), "r"(kAccCols) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tc_before();
  __syncthreads();
  tc_after();
  const uint32_t tmem = *(volatile uint32_t*)&tmem_slot;
  grid_wait();

  if (warp < kConvWarps) {
    // a thread's chunks: TOKENS, eight j of rows c = (tid >> 4) + 16 k; else eight c of rows j = (tid >> 3) + 32 k
    const int chunk = TOKENS ? tid & 15 : tid & 7, row = TOKENS ? tid >> 4 : tid >> 3;
    constexpr int kRows = TOKENS ? 16 : 32, kScales = StageRegs<TOKENS, G>::kScales;
    StageRegs<TOKENS, G> r;
    const bool whole_chunks = p.J % 8 == 0;       // TOKENS: else the last chunk of a row of g ends in its middle
    // Offsets from a stage's first element, the same for every stage of an item.  Rows past J are read again from the last one:
    // what they make is never stored.  c past the end, and j past J where those are what is contiguous, are zeros.
    uint32_t g_row[4];
    const uint32_t ldg = (uint32_t)p.ldg, q_step = TOKENS ? 32u * (uint32_t)p.ldq : 16u;
    const uint32_t q_at = TOKENS ? (uint32_t)(tid >> 3) * (uint32_t)p.ldq + 16u * (tid & 7) : (uint32_t)(tid >> 1) * (uint32_t)p.ldq + (tid & 1) * 32;
    auto set_rows = [&](const DotItem& w) {
#pragma unroll
      for (int k = 0; k < 4; ++k)
        g_row[k] = TOKENS ? (uint32_t)(row + kRows * k) * ldg + 8u * chunk : (uint32_t)min(row + kRows * k, p.J - 1 - w.j0) * ldg + 8u * chunk;
    };
    auto load_g = [&](const DotItem& w, int c0, int k) {
      if constexpr (TOKENS) {
        const G* src = static_cast<const G*>(p.g) + (int64_t)c0 * p.ldg + w.j0 + g_row[k];
        const bool lo = c0 + row + kRows * k < w.c_end && w.j0 + 8 * chunk < p.J, hi = c0 + row + kRows * k < w.c_end && w.j0 + 8 * chunk + 4 < p.J;
        if constexpr (sizeof(G) == 4) {
          const uint4 zero = make_uint4(0, 0, 0, 0);
          const uint4 a = lo ? __ldg(reinterpret_cast<const uint4*>(src)) : zero, b = hi ? __ldg(reinterpret_cast<const uint4*>(src) + 1) : zero;
          r.g[k][0] = a.x; r.g[k][1] = a.y; r.g[k][2] = a.z; r.g[k][3] = a.w;
          r.g[k][4] = b.x; r.g[k][5] = b.y; r.g[k][6] = b.z; r.g[k][7] = b.w;
        } else if (whole_chunks) {
          const uint4 a = lo ? __ldg(reinterpret_cast<const uint4*>(src)) : make_uint4(0, 0, 0, 0);
          r.g[k][0] = a.x; r.g[k][1] = a.y; r.g[k][2] = a.z; r.g[k][3] = a.w;
        } else {                                  // rows of whole 8-byte units
          const uint2 zero = make_uint2(0, 0);
          const uint2 a = lo ? __ldg(reinterpret_cast<const uint2*>(src)) : zero, b = hi ? __ldg(reinterpret_cast<const uint2*>(src) + 1) : zero;
          r.g[k][0] = a.x; r.g[k][1] = a.y; r.g[k][2] = b.x; r.g[k][3] = b.y;
        }
      } else {
        const bool in = c0 + 8 * chunk < w.c_end;           // C is a multiple of 16: a chunk is in or out together
        const uint4* src = reinterpret_cast<const uint4*>(static_cast<const G*>(p.g) + (int64_t)w.j0 * p.ldg + c0 + g_row[k]);
#pragma unroll
        for (int h = 0; h < StageRegs<TOKENS, G>::kWords / 4; ++h) {
          const uint4 v = in ? __ldg(src + h) : make_uint4(0, 0, 0, 0);
          r.g[k][4 * h] = v.x; r.g[k][4 * h + 1] = v.y; r.g[k][4 * h + 2] = v.z; r.g[k][4 * h + 3] = v.w;
        }
      }
    };
    auto load_q = [&](const DotItem& w, int c0) {
      const uint8_t* src = (TOKENS ? p.q + (int64_t)c0 * p.ldq + w.i0 : p.q + (int64_t)w.i0 * p.ldq + c0) + q_at;
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int c = TOKENS ? (tid >> 3) + 32 * h : (tid & 1) * 32 + 16 * h;
        const uint4 v = c0 + c < w.c_end ? __ldg(reinterpret_cast<const uint4*>(src + h * q_step)) : make_uint4(0, 0, 0, 0);
        r.q[4 * h] = v.x; r.q[4 * h + 1] = v.y; r.q[4 * h + 2] = v.z; r.q[4 * h + 3] = v.w;
      }
    };
    // A lane makes the scales of two of a stage's c and the warp hands them round: which register a thread takes one from is fixed.
    auto load_scales = [&](const DotItem& w, int c0) {
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int c = c0 + (TOKENS ? lane + 32 * h : 2 * lane + h);
        r.e8[h] = 0u; r.e32[h] = 0.0f;
        if (c < w.c_end) {
          const uint32_t id = TOKENS ? (uint32_t)c * p.nbc + w.it : (uint32_t)w.it * p.nbc + (p.per_column ? c : c / 128);
          r.e8[h] = __ldg(p.sc8 + id); r.e32[h] = __ldg(p.sc32 + (id >> p.log2_K));
        }
      }
    };
    int at = blockIdx.x, st = 0;
    DotItem w(p, at);
    int c0 = w.c_begin;
    set_rows(w);
    load_scales(w, c0);
    load_q(w, c0);
#pragma unroll
    for (int k = 0; k < 4; ++k) load_g(w, c0, k);
    // The next stage's loads are asked for as their registers become free.  The fence that makes the stores visible to the tensor core
    // is the issuing lane's: a thread's own waits for all that it has under way, loads too.
    for (uint32_t n = 0;; ++n) {
      if (++st == w.n_stages) {
        at += gridDim.x;
        st = 0;
        if (at < p.items) {
          w = DotItem(p, at);
          set_rows(w);
        }
      }
      const bool more = at < p.items;
      c0 = w.c_begin + st * kDepth;
      const int buf = n % kStages;
      if (!bar_wait(empty(buf), ((n / kStages) & 1) ^ 1, wait_polls(p))) break;
      const uint32_t base = tiles_base + buf * kStageBytes;
      float s[kScales];
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const float own = __fmul_rn(block_multiplier(r.e8[h], r.e32[h]), kScaleUp * 0.0078125f);
#pragma unroll
        for (int e = 0; e < kScales / 2; ++e) {
          if constexpr (TOKENS) s[2 * h + e] = __shfl_sync(0xffffffffu, own, row + kRows * e);
          else s[2 * e + h] = __shfl_sync(0xffffffffu, own, 4 * chunk + e);
        }
      }
      if (more) load_scales(w, c0);
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        uint32_t o[2][4];
#pragma unroll
        for (int e = 0; e < 4; ++e) { o[e >> 1][2 * (e & 1)] = fp8x2_to_bf16x2(r.q[4 * h + e]); o[e >> 1][2 * (e & 1) + 1] = fp8x2_to_bf16x2(r.q[4 * h + e] >> 16); }
#pragma unroll
        for (int b = 0; b < 2; ++b) {
          if constexpr (TOKENS) {       // the lanes of the second 64 of i store their second chunk first: else two lanes meet in every bank
            const int x = tid & 7, which = b ^ (x >> 2);
            st_chunk(base + chunk_at<TOKENS>((tid >> 3) + 32 * h, 2 * x + which), which ? o[1][0] : o[0][0], which ? o[1][1] : o[0][1], which ? o[1][2] : o[0][2], which ? o[1][3] : o[0][3]);
          } else {
            st_chunk(base + chunk_at<TOKENS>(tid >> 1, 4 * (tid & 1) + 2 * h + b), o[b][0], o[b][1], o[b][2], o[b][3]);
          }
        }
      }
      if (more) load_q(w, c0);
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        uint32_t hi[4], mid[4], lo[4];
        float g[8], f[8];
        r.chunk(k, g);
#pragma unroll
        for (int e = 0; e < 8; ++e) f[e] = TOKENS ? s[k % kScales] : s[e % kScales];
        split_chunk(g, f, hi, mid, lo);
        const uint32_t to = base + chunk_at<TOKENS>(row, chunk) + (uint32_t)(kRows * k) * 128u;      // eight rows further the same swizzle
        st_chunk(to + kOpBytes, lo[0], lo[1], lo[2], lo[3]);
        st_chunk(to + 2 * kOpBytes, mid[0], mid[1], mid[2], mid[3]);
        st_chunk(to + 3 * kOpBytes, hi[0], hi[1], hi[2], hi[3]);
        if (more) load_g(w, c0, k);
      }
      __syncwarp();
#ifdef PB_DIAGNOSTICS
      if (lane == 0 && !(p.withhold && n == 0)) bar_arrive(full(buf));
#else
      if (lane == 0) bar_arrive(full(buf));
#endif
      if (!more) break;
    }
  } else if (warp >= kIssueWarp) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 40;");
    if (warp == kIssueWarp && lane == 0) {
      bool ok = true;
      uint32_t n = 0;
      for (int at = blockIdx.x; at < p.items && ok; at += gridDim.x)
        for (int left = DotItem(p, at).n_stages; left > 0 && ok; --left, ++n) {
          const int buf = n % kStages, ab = n & 1;
          ok = bar_wait(full(buf), (n / kStages) & 1, wait_polls(p)) && bar_wait(acc_empty(ab), ((n >> 1) & 1) ^ 1, wait_polls(p));
          if (!ok) break;
          asm volatile("fence.proxy.async.shared::cta;" ::: "memory");      // the tensor core reads what the converting threads stored
          tc_after();
          const uint64_t a = tile_desc<TOKENS>(tiles_base + buf * kStageBytes);
#pragma unroll
          for (int kk = 0; kk < kDepth / 16; ++kk)            // smallest terms first
#pragma unroll
            for (int t = 1; t <= 3; ++t)
              mma_f16<TOKENS>(tmem + (2 * ab + (kk >> 1)) * kTile, a + kk * kStep16<TOKENS>, a + (uint64_t)(t * (kOpBytes >> 4)) + kk * kStep16<TOKENS>, (kk & 1) || t > 1);
          commit_to(empty(buf));
          commit_to(acc_full(ab));
        }
    }
  } else {
    asm volatile("setmaxnreg.inc.sync.aligned.u32 216;");      // 128 * (2 * 128 + 216 + 40) = 512 * 128
    const int quad = warp & 3, r = quad * 32 + lane;         // the thread's row of the tile, an i
    bool ok = true, odd = false;        // odd: some sum of this thread is not finite
    uint32_t n = 0;
    for (int at = blockIdx.x; at < p.items && ok; at += gridDim.x) {
      const DotItem w(p, at);
      float acc[kTile];
#pragma unroll
      for (int e = 0; e < kTile; ++e) acc[e] = 0.0f;
      for (int st = 0; st < w.n_stages; ++st, ++n) {
        const int ab = n & 1;
        ok = __all_sync(0xffffffffu, bar_wait(acc_full(ab), (n >> 1) & 1, wait_polls(p)));
        if (!ok) break;
        tc_after();
        const uint32_t from = tmem + ((uint32_t)(quad * 32) << 16) + 2 * ab * kTile;
        uint32_t v[2][32];
        ld_acc32(from, v[0]);
#pragma unroll
        for (int k = 0; k < 8; ++k) {   // 32 columns of one accumulator, then of the other
          asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
          if (k + 1 < 8) {
            ld_acc32(from + (k + 1) * 32, v[(k + 1) & 1]);
          } else {
            tc_before();
            __syncwarp();
            if (lane == 0) bar_arrive(acc_empty(ab));
          }
#pragma unroll
          for (int e = 0; e < 32; e += 2) {
            float* to = acc + 32 * (k & 3) + e;
            const float2 t = __fadd2_rn(make_float2(to[0], to[1]), make_float2(__uint_as_float(v[k & 1][e]), __uint_as_float(v[k & 1][e + 1])));
            to[0] = t.x; to[1] = t.y;
          }
        }
      }
      if (!ok) break;
      float2 zero = make_float2(0.0f, 0.0f);            // times 0: NaN where a sum is not finite
#pragma unroll
      for (int e = 0; e < kTile; e += 2) {
        zero = __ffma2_rn(make_float2(acc[e], acc[e + 1]), make_float2(0.0f, 0.0f), zero);
        const float2 t = __fmul2_rn(make_float2(acc[e], acc[e + 1]), make_float2(kScaleDown, kScaleDown));
        acc[e] = t.x; acc[e + 1] = t.y;
      }
      odd |= !(zero.x + zero.y == 0.0f);
      float* out = p.out + (int64_t)w.split * p.part;
      if constexpr (TOKENS) {           // a thread's row of out, by way of shared memory: whole lines (of 16 bytes a lane: 1 us more)
        asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");    // the tile before has left
#pragma unroll
        for (int e = 0; e < kTile; e += 4)
          asm volatile("st.shared.v4.f32 [%0], {%1, %2, %3, %4};" ::"r"(out_base + r * kOutPitch + e * 4), "f"(acc[e]), "f"(acc[e + 1]), "f"(acc[e + 2]), "f"(acc[e + 3]) : "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;"
                     ::"l"(out + (int64_t)(w.i0 + r) * p.ldo + w.j0), "r"(out_base + r * kOutPitch), "r"(4 * min(kTile, p.J - w.j0)) : "memory");      // J is a multiple of 4
        asm volatile("cp.async.bulk.commit_group;" ::: "memory");
      } else {                          // one address, moved on: with an address per store the code took 15000 cycles to fetch for one use
        float* to = out + (int64_t)w.j0 * p.ldo + w.i0 + r;
        if (w.j0 + kTile <= p.J) {
#pragma unroll
          for (int e = 0; e < kTile; ++e, to += p.ldo) *to = acc[e];
        } else {
#pragma unroll
          for (int e = 0; e < kTile; ++e, to += p.ldo)
            if (w.j0 + e < p.J) *to = acc[e];
        }
      }
    }
    // Sums that are not finite are made again when the CTA's tiles are done: nothing waits for these warps any more, however long it takes.
    if (odd && ok) {
      asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");           // what the thread makes again lies in out already
#pragma unroll 1
      for (int at = blockIdx.x; at < p.items; at += gridDim.x) {
        const DotItem w(p, at);
        float* out = p.out + (int64_t)w.split * p.part;
        const int i = w.i0 + r;
#pragma unroll 1
        for (int jb = w.j0; jb < w.j0 + kTile; jb += 64) {
          bool again = false;
#pragma unroll 1
          for (int j = jb; j < min(jb + 64, p.J); ++j) again |= __float_as_uint(out[TOKENS ? (int64_t)i * p.ldo + j : (int64_t)j * p.ldo + i]) << 1 >= 2 * 0x7f800000u;
          if (again) plain_dots<TOKENS, G>(p, out, i, jb, w.it, w.c_begin, w.c_end);
        }
      }
    }
    asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");        // shared memory is the CTA's until the last tile has left it
  }
  tc_before();
  __syncthreads();
  if (warp == kIssueWarp) {
    tc_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(kAccCols) : "memory");
  }
}

__global__ void __launch_bounds__(256) add_parts_kernel(const float4* parts, float4* out, int64_t n4, int splits) {
  grid_wait();
  const int64_t i = (int64_t)blockIdx.x * 256 + threadIdx.x;
  if (i >= n4) return;
  float4 s = parts[i];
  for (int k = 1; k < splits; ++k) {
    const float4 v = parts[(int64_t)k * n4 + i];
    s.x += v.x; s.y += v.y; s.z += v.z; s.w += v.w;
  }
  out[i] = s;
}

struct DotPlan { int I, J, C, i_tiles, tiles, splits, split_depth; };

// Parts so that the tiles times the parts come near the SM count, none of them shorter than kMinSplitDepth.
DotPlan make_plan(int tokens, int64_t rows, int64_t cols, int64_t g_free) {
  DotPlan d;
  d.I = (int)(tokens ? cols : rows); d.C = (int)(tokens ? rows : cols); d.J = (int)g_free;
  d.i_tiles = d.I / kTile;
  const int64_t tiles = (int64_t)d.i_tiles * ((d.J + kTile - 1) / kTile);
  d.tiles = (int)tiles;
  int64_t splits = sm_count() / (tiles > 0 ? tiles : 1);
  splits = std::min<int64_t>(splits, d.C / kMinSplitDepth);
  if (splits < 1) splits = 1;
  const int64_t stages = (d.C + kDepth - 1) / kDepth, per = (stages + splits - 1) / splits;
  d.split_depth = (int)(per * kDepth);
  d.splits = (int)((stages + per - 1) / per);
  return d;
}

#ifdef PB_DIAGNOSTICS
std::atomic<uint32_t> g_dot_polls{kWaitPolls};
std::atomic<int> g_dot_withhold{0};
#endif

template <bool TOKENS, typename G>
int launch_dot(const DotParams& p, unsigned grid, cudaStream_t st) {
  PB_CUDA_TRY(cudaFuncSetAttribute(dense_dot_kernel<TOKENS, G>, cudaFuncAttributeMaxDynamicSharedMemorySize, kDotSmem));      // per device
  launch_behind(dense_dot_kernel<TOKENS, G>, grid, kDotThreads, kDotSmem, st, p);
  PB_LAUNCH_CHECK("dense_dot_kernel");
  return PB_OK;
}

bool dot_shape_ok(int tokens, int64_t rows, int64_t cols, int a, int b, int64_t g_free) {
  if (rows <= 0 || cols <= 0 || g_free <= 0 || rows > 0x7fffff00ll || cols > 0x7fffff00ll || g_free > 0x7fffff00ll) return false;
  if (tokens) return a == 1 && b == 128 && cols % 128 == 0 && g_free % 4 == 0;
  return a == 128 && (b == 128 || b == 1) && rows % 128 == 0 && cols % 16 == 0 && cols % b == 0;
}

}  // namespace

int add_parts(const float* parts, float* out, int64_t n, int splits, cudaStream_t st) {
  const int64_t n4 = n / 4;
  launch_behind(add_parts_kernel, (unsigned)((n4 + 255) / 256), 256, 0, st, reinterpret_cast<const float4*>(parts), reinterpret_cast<float4*>(out), n4, splits);
  PB_LAUNCH_CHECK("add_parts_kernel");
  return PB_OK;
}

// Reads and clears this file's device status word (see pb_gemm_check).
int dense_dot_status_fetch(unsigned int* out) {
  const unsigned int zero = 0;
  PB_CUDA_TRY(cudaMemcpyFromSymbol(out, g_dot_status, sizeof(*out)));
  if (*out != 0) PB_CUDA_TRY(cudaMemcpyToSymbol(g_dot_status, &zero, sizeof(zero)));
  unsigned int split = 0;
  if (int s = split_dot_status_fetch(&split)) return s;
  if (split != 0) *out = split;
  return PB_OK;
}
}  // namespace pb

using namespace pb;

extern "C" size_t pb_dense_dot_workspace_size(int tokens, int64_t rows, int64_t cols, int a, int b, int64_t g_free) {
  if (!dot_shape_ok(tokens, rows, cols, a, b, g_free)) return 0;
  const DotPlan d = make_plan(tokens, rows, cols, g_free);
  return d.splits > 1 ? (size_t)d.splits * d.I * d.J * sizeof(float) : 0;
}

extern "C" size_t pb_dense_dot_workspace_best(int tokens, int64_t rows, int64_t cols, int a, int b, int64_t g_free, int g_dtype) {
  const size_t least = pb_dense_dot_workspace_size(tokens, rows, cols, a, b, g_free);
  SplitDotPlan split;
  if ((g_dtype != PB_F32 && g_dtype != PB_BF16) || !dot_shape_ok(tokens, rows, cols, a, b, g_free) ||
      !split_dot_plan(tokens, rows, cols, a, b, g_free, g_dtype == PB_BF16, &split))
    return least;
  return std::max(least, split.bytes + kSplitAlign - 16);
}

extern "C" int pb_dense_dot(int tokens, const uint8_t* q, const uint8_t* sc8, const float* sc32, int64_t rows, int64_t cols, int a, int b,
                            const void* g, int g_dtype, int64_t g_free, float* out, void* workspace, size_t workspace_bytes, void* stream) {
  if (!q || !sc8 || !sc32 || !g || !out) return fail(PB_ERR_NULL_POINTER, "pb_dense_dot: q, sc8, sc32, g and out must be non-null");
  if (!dot_shape_ok(tokens, rows, cols, a, b, g_free))
    return fail(PB_ERR_UNSUPPORTED, "pb_dense_dot: a [%lld, %lld] triple on (%d,%d) against %lld (see the header for what it takes)",
                (long long)rows, (long long)cols, a, b, (long long)g_free);
  if (g_dtype != PB_F32 && g_dtype != PB_BF16) return fail(PB_ERR_BAD_DTYPE, "pb_dense_dot: g_dtype %d is neither PB_F32 nor PB_BF16", g_dtype);
  Geometry geo;
  if (int s = make_geometry(rows, cols, a, b, &geo)) return s;
  const DotPlan d = make_plan(tokens, rows, cols, g_free);
  if ((int64_t)kTile * std::max(cols, g_free) > kMaxIndexed || geo.Nb > kMaxIndexed || (int64_t)d.tiles * d.splits > kMaxIndexed || (int64_t)d.i_tiles * ((d.J + kTile - 1) / kTile) > kMaxIndexed)
    return fail(PB_ERR_UNSUPPORTED, "pb_dense_dot: [%lld, %lld] against %lld is too large", (long long)rows, (long long)cols, (long long)g_free);
  if ((reinterpret_cast<uintptr_t>(q) | reinterpret_cast<uintptr_t>(g) | reinterpret_cast<uintptr_t>(out)) & 15)
    return fail(PB_ERR_MISALIGNED, "pb_dense_dot: q, g and out must be 16-byte aligned");
  const int64_t out_elems = (int64_t)d.I * d.J;
  const size_t need = d.splits > 1 ? (size_t)d.splits * out_elems * sizeof(float) : 0;
  if (need && (!workspace || workspace_bytes < need))
    return fail(PB_ERR_WORKSPACE_TOO_SMALL, "pb_dense_dot: needs %zu bytes of workspace, got %zu", need, workspace_bytes);
  if (reinterpret_cast<uintptr_t>(workspace) & 15) return fail(PB_ERR_MISALIGNED, "pb_dense_dot: workspace must be 16-byte aligned");
  SplitDotPlan split;
  const size_t skip = (size_t)(-reinterpret_cast<uintptr_t>(workspace)) & (kSplitAlign - 1);
  if (workspace && split_dot_plan(tokens, rows, cols, a, b, g_free, g_dtype == PB_BF16, &split) && workspace_bytes >= split.bytes + skip)
    return split_dot_run(split, tokens, q, sc8, sc32, rows, cols, a, b, g, g_dtype == PB_BF16, g_free, out, static_cast<unsigned char*>(workspace) + skip,
                         static_cast<cudaStream_t>(stream));
  uint32_t log2_K = 0;                  // K divides 8, or 1024 for (128,128)
  while ((1ll << log2_K) < geo.K) ++log2_K;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  float* dst = d.splits > 1 ? static_cast<float*>(workspace) : out;
  DotParams p{q, sc8, sc32, g, dst, cols, tokens ? g_free : cols, tokens ? g_free : (int64_t)d.I, out_elems, d.I, d.J, d.C,
              (uint32_t)geo.nbc, log2_K, b == 1, d.i_tiles, d.tiles, d.tiles * d.splits, d.split_depth};
#ifdef PB_DIAGNOSTICS
  p.polls = g_dot_polls.load();
  p.withhold = g_dot_withhold.load();
#endif
  const unsigned grid = (unsigned)std::min(p.items, sm_count());
  const int status = tokens ? (g_dtype == PB_F32 ? launch_dot<true, float>(p, grid, st) : launch_dot<true, __nv_bfloat16>(p, grid, st))
                            : (g_dtype == PB_F32 ? launch_dot<false, float>(p, grid, st) : launch_dot<false, __nv_bfloat16>(p, grid, st));
  if (status) return status;
  return d.splits > 1 ? add_parts(dst, out, out_elems, d.splits, st) : PB_OK;      // I is a multiple of 128
}

#ifdef PB_DIAGNOSTICS
// Diagnostics build only (not part of the reference's surface, not in the product library).  Sets the poll budget of the
// waits (0 restores the default) and whether the first stage of the launches that follow is withheld.
extern "C" PB_API int pb_debug_dot_control(unsigned int polls, int withhold) {
  g_dot_polls.store(polls ? polls : kWaitPolls);
  g_dot_withhold.store(withhold);
  split_dot_control(polls, withhold);
  return PB_OK;
}
#endif

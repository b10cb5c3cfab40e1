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
// A CTA makes a 128 x 128 tile of out: eight warps convert (global loads into registers, scale, split, 128-byte
// swizzled K-major tiles in shared memory; where i and j are the contiguous dimensions the eight c of a 16-byte chunk come from
// eight rows, so the transpose is in the loads), eight warps empty one pair of accumulators
// while the other fills, and one lane of theirs issues tcgen05.mma.  Where the tiles do not fill the SMs the contraction is
// cut, and the parts are added in order by a second kernel.
//
// What bounds it: no one part.  A stage of dX takes 2800 cycles (of dW 3500), of which the tensor core works 768; before the loads moved behind the
// fence, dX took 17 % less with the split left out, 14 with the loads, 13 with the emptying, 8 with eleven of the twelve
// products (dW: 28, 40, 11, 5), and sixteen converting warps were no faster than eight.  Against dequantizing and the library's
// SGEMM (inside a CUDA graph): 3000 tokens, 2048 x 2048, dX 491 -> 143 us, dW 432 -> 175 (bf16 g, read as it is: 507 -> 142 and
// 448 -> 179); 8192 tokens, 2048 x 128, 100 -> 62 and 139 -> 37; 64 tokens, 1024 x 1024, 22 -> 14 and 9 -> 8.5.  Where there is less
// than that to do the library's kernels are shorter (64 tokens, 2048 x 128, 8 | 10 and 7 | 8), but a call of it is not: one after
// the other the two dots take 48 us there and these 24, for the host's part of four library calls.
//
// Every tile converts what it reads, so an operand that many tiles share is converted many times: where 512 columns or more share
// it and there is enough to do, split_dot.cu makes it ready once (split_dot_pays: 3000 tokens, 2048 x 2048, bf16 cotangent, dX 141 -> 75 us,
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
constexpr int kStages = 3;
constexpr int kMinSplitDepth = 256;   // c per part: below this a part is mostly prologue
constexpr int kConvWarps = 8, kDrainWarps = 8;
constexpr int kDotThreads = 32 * (kConvWarps + kDrainWarps);       // 128 registers each: a seventeenth warp for the MMAs leaves 96, and spills
constexpr int kOpBytes = kTile * kDepth * 2;            // one bf16 operand tile: 128 rows of 128 bytes
constexpr int kStageBytes = 4 * kOpBytes;               // q, then f's lo, mid and hi
constexpr int kDotSmem = kStages * kStageBytes + 1024 + 128;      // 1024: the tiles start on a swizzle atom
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
  int i_tiles, tiles, split_depth;
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
// K-major tile, 128-byte swizzle: rows of 128 bytes, 8-row groups 1024 bytes apart (descriptor version 1, layout 2)
__device__ __forceinline__ uint64_t tile_desc(uint32_t smem_addr) {
  return (uint64_t)((smem_addr & 0x3ffffu) >> 4) | (1ull << 16) | ((uint64_t)(1024 >> 4) << 32) | (1ull << 46) | (2ull << 61);
}
// kind::f16: f32 accumulator, both operands bf16 and K-major, N = M = 128
constexpr uint32_t kDotInstr = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(kTile >> 3) << 17) | ((uint32_t)(kTile >> 4) << 24);
__device__ __forceinline__ void mma_f16(uint32_t d, uint64_t a, uint64_t b, uint32_t accumulate) {
  asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\ttcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
               ::"r"(d), "l"(a), "l"(b), "r"(kDotInstr), "r"(accumulate) : "memory");
}
__device__ __forceinline__ void ld_acc16(uint32_t taddr, uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
        "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
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
// byte offset of the 16-byte chunk (eight c) of a row in a swizzled tile
__device__ __forceinline__ uint32_t chunk_at(int row, int chunk) { return (uint32_t)row * 128u + (uint32_t)((chunk ^ (row & 7)) << 4); }
__device__ __forceinline__ void st_chunk(uint32_t addr, uint32_t a, uint32_t b, uint32_t c, uint32_t d) {
  asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(addr), "r"(a), "r"(b), "r"(c), "r"(d));      // ordered by the fence at the stage's end
}

// What a converting thread holds of a stage: four chunks (eight c each) of g for rows j, its share of q, the scales of its c.
template <bool TOKENS, typename G>
struct StageRegs {
  static constexpr int kWords = sizeof(G) == 4 || TOKENS ? 8 : 4;
  uint32_t g[4][kWords];              // as loaded: f32, or a bf16 in the low half, or two bf16
  __device__ __forceinline__ void chunk(int k, float (&f)[8]) const {
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      if constexpr (sizeof(G) == 4) f[e] = __uint_as_float(g[k][e]);
      else if constexpr (TOKENS) f[e] = __uint_as_float(g[k][e] << 16);
      else f[e] = __uint_as_float(e & 1 ? g[k][e / 2] & 0xffff0000u : g[k][e / 2] << 16);
    }
  }
  uint32_t q[TOKENS ? 16 : 8];        // TOKENS: [half][c] two i each; else 32 bytes of a row
  uint32_t e8[TOKENS ? 1 : 8];        // TOKENS: lanes 0-7 a c each, handed round; else this thread's
  float e32[TOKENS ? 1 : 8];
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

template <bool TOKENS, typename G>
__global__ void __launch_bounds__(kDotThreads, 1) dense_dot_kernel(const __grid_constant__ DotParams p) {
  extern __shared__ unsigned char dot_smem[];
  __shared__ __align__(8) uint64_t bars[2 * kStages + 4];
  __shared__ uint32_t tmem_slot;
  const uint32_t tiles_base = (dot_smem_u32(dot_smem) + 1023u) & ~1023u;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int split = blockIdx.x / p.tiles, tile = blockIdx.x - split * p.tiles;
  const int it = tile % p.i_tiles, i0 = it * kTile, j0 = (tile / p.i_tiles) * kTile;
  const int c_begin = split * p.split_depth, c_end = min(p.C, c_begin + p.split_depth);
  const int n_stages = (c_end - c_begin + kDepth - 1) / kDepth;
  auto full = [&](int s) { return dot_smem_u32(&bars[s]); };
  auto empty = [&](int s) { return dot_smem_u32(&bars[kStages + s]); };
  auto acc_full = [&](int a) { return dot_smem_u32(&bars[2 * kStages + a]); };
  auto acc_empty = [&](int a) { return dot_smem_u32(&bars[2 * kStages + 2 + a]); };

  if (tid == 0) {
    for (int s = 0; s < kStages; ++s) { bar_init(full(s), kConvWarps); bar_init(empty(s), 1); }
    for (int a = 0; a < 2; ++a) { bar_init(acc_full(a), 1); bar_init(acc_empty(a), kDrainWarps); }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == kConvWarps) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(dot_smem_u32(&tmem_slot)), "r"(kAccCols) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tc_before();
  __syncthreads();
  tc_after();
  const uint32_t tmem = *(volatile uint32_t*)&tmem_slot;

  if (warp < kConvWarps) {
    const int chunk = TOKENS ? warp : tid & 7;              // this thread's eight c of a stage
    StageRegs<TOKENS, G> r;
    auto row_of = [&](int k) { return TOKENS ? 32 * k + lane : 32 * k + (tid >> 3); };
    // Offsets from a stage's first element, the same for every stage: one add per load.  Rows past J are read again from the
    // last one: what they make is never stored.  c past the end are zeros (only a last stage has them: `whole`).
    uint32_t g_row[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const uint32_t j = (uint32_t)min(row_of(k), p.J - 1 - j0);
      g_row[k] = TOKENS ? j : j * (uint32_t)p.ldg + 8 * chunk;
    }
    const uint32_t ldg = (uint32_t)p.ldg, ldq = (uint32_t)p.ldq;
    const uint32_t q_at = TOKENS ? 8 * chunk * ldq + 2 * lane : (uint32_t)(tid >> 1) * ldq + (tid & 1) * 32;
    auto load_g = [&](int st, int k) {
      const int c0 = c_begin + st * kDepth;
      const bool whole = c0 + kDepth <= c_end;
      if constexpr (TOKENS) {
        const G* src = static_cast<const G*>(p.g) + (int64_t)c0 * p.ldg + j0;
        using Word = typename std::conditional<sizeof(G) == 4, uint32_t, uint16_t>::type;
#pragma unroll
        for (int e = 0; e < 8; ++e)
          r.g[k][e] = (whole || c0 + 8 * chunk + e < c_end) ? (uint32_t)__ldg(reinterpret_cast<const Word*>(src) + (8 * chunk + e) * ldg + g_row[k]) : 0u;
      } else {
        const bool in = whole || c0 + 8 * chunk < c_end;    // C is a multiple of 16: a chunk is in or out together
        const uint4* src = reinterpret_cast<const uint4*>(static_cast<const G*>(p.g) + (int64_t)j0 * p.ldg + c0 + g_row[k]);
#pragma unroll
        for (int h = 0; h < StageRegs<TOKENS, G>::kWords / 4; ++h) {
          const uint4 v = in ? __ldg(src + h) : make_uint4(0, 0, 0, 0);
          r.g[k][4 * h] = v.x; r.g[k][4 * h + 1] = v.y; r.g[k][4 * h + 2] = v.z; r.g[k][4 * h + 3] = v.w;
        }
      }
    };
    auto load_q = [&](int st) {
      const int c0 = c_begin + st * kDepth;
      const bool whole = c0 + kDepth <= c_end;
      if constexpr (TOKENS) {
        const uint8_t* src = p.q + (int64_t)c0 * p.ldq + i0;
#pragma unroll
        for (int e = 0; e < 8; ++e) {
          const bool in = whole || c0 + 8 * chunk + e < c_end;
          r.q[e] = in ? (uint32_t)__ldg(reinterpret_cast<const uint16_t*>(src + q_at + e * ldq)) : 0u;
          r.q[8 + e] = in ? (uint32_t)__ldg(reinterpret_cast<const uint16_t*>(src + q_at + e * ldq + 64)) : 0u;
        }
      } else {
        const uint8_t* src = p.q + (int64_t)i0 * p.ldq + c0;
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const uint4 v = whole || c0 + (tid & 1) * 32 + 16 * h < c_end ? __ldg(reinterpret_cast<const uint4*>(src + q_at) + h) : make_uint4(0, 0, 0, 0);
          r.q[4 * h] = v.x; r.q[4 * h + 1] = v.y; r.q[4 * h + 2] = v.z; r.q[4 * h + 3] = v.w;
        }
      }
    };
    auto load_scales = [&](int st) {
      const int c = c_begin + st * kDepth + 8 * chunk;
#pragma unroll
      for (int e = 0; e < (TOKENS ? 1 : 8); ++e) { r.e8[e] = 0u; r.e32[e] = 0.0f; }
      if constexpr (TOKENS) {
        const int own = c + (lane & 7);
        if (own < c_end) {
          const uint32_t id = (uint32_t)own * p.nbc + it;
          r.e8[0] = __ldg(p.sc8 + id); r.e32[0] = __ldg(p.sc32 + (id >> p.log2_K));
        }
      } else if (c < c_end) {
        const uint32_t id = (uint32_t)it * p.nbc + (p.per_column ? c : c / 128);
        r.e8[0] = __ldg(p.sc8 + id); r.e32[0] = __ldg(p.sc32 + (id >> p.log2_K));
        if (p.per_column) {           // else 64 of c lie in one block
#pragma unroll
          for (int e = 1; e < 8; ++e) { r.e8[e] = __ldg(p.sc8 + id + e); r.e32[e] = __ldg(p.sc32 + ((id + e) >> p.log2_K)); }
        }
      }
    };
    auto load_stage = [&](int st) {
      load_scales(st);
      load_q(st);
#pragma unroll
      for (int k = 0; k < 4; ++k) load_g(st, k);
    };
    load_stage(0);
    for (int st = 0; st < n_stages; ++st) {
      const int buf = st % kStages;
      if (!bar_wait(empty(buf), ((st / kStages) & 1) ^ 1, wait_polls(p))) break;
      const uint32_t base = tiles_base + buf * kStageBytes;
      const bool more = st + 1 < n_stages;
      if constexpr (TOKENS) {
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          uint32_t lo[4], hi[4];      // the chunks of i = 64 h + 2 lane and the next
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            const uint32_t a = r.q[8 * h + 2 * e], b = r.q[8 * h + 2 * e + 1];
            lo[e] = fp8x2_to_bf16x2(__byte_perm(a, b, 0x0040)); hi[e] = fp8x2_to_bf16x2(__byte_perm(a, b, 0x0051));
          }
          st_chunk(base + chunk_at(64 * h + 2 * lane, chunk), lo[0], lo[1], lo[2], lo[3]);
          st_chunk(base + chunk_at(64 * h + 2 * lane + 1, chunk), hi[0], hi[1], hi[2], hi[3]);
        }
      } else {
#pragma unroll
        for (int h = 0; h < 4; ++h) {
          uint32_t o[4];
#pragma unroll
          for (int e = 0; e < 2; ++e) { o[2 * e] = fp8x2_to_bf16x2(r.q[2 * h + e]); o[2 * e + 1] = fp8x2_to_bf16x2(r.q[2 * h + e] >> 16); }
          st_chunk(base + chunk_at(tid >> 1, 4 * (tid & 1) + h), o[0], o[1], o[2], o[3]);
        }
      }
      float s[8];
      auto scale = [](uint32_t e8, float e32) { return __fmul_rn(block_multiplier(e8, e32), kScaleUp * 0.0078125f); };
      if constexpr (TOKENS) {
        const float own = scale(r.e8[0], r.e32[0]);
#pragma unroll
        for (int e = 0; e < 8; ++e) s[e] = __shfl_sync(0xffffffffu, own, e);
      } else {
        s[0] = scale(r.e8[0], r.e32[0]);
#pragma unroll
        for (int e = 1; e < 8; ++e) s[e] = p.per_column ? scale(r.e8[e], r.e32[e]) : s[0];
      }
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        uint32_t hi[4], mid[4], lo[4];
        float g[8];
        r.chunk(k, g);
        split_chunk(g, s, hi, mid, lo);
        const uint32_t at = base + chunk_at(row_of(k), chunk);
        st_chunk(at + kOpBytes, lo[0], lo[1], lo[2], lo[3]);
        st_chunk(at + 2 * kOpBytes, mid[0], mid[1], mid[2], mid[3]);
        st_chunk(at + 3 * kOpBytes, hi[0], hi[1], hi[2], hi[3]);
      }
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");      // the tensor core reads what was stored
      __syncwarp();
#ifdef PB_DIAGNOSTICS
      if (lane == 0 && !(p.withhold && st == 0)) bar_arrive(full(buf));
#else
      if (lane == 0) bar_arrive(full(buf));
#endif
      // The next stage's loads go behind the fence, which waits for the thread's accesses that are under way: asked for as
      // their registers became free, they held every stage up at its fence (dX 155 -> 150 us, dW 174 -> 160, 2368 tokens).
      if (more) load_stage(st + 1);
    }
  } else {
    const int quad = warp & 3, half = (warp - kConvWarps) >> 2;      // rows 32 quad .., columns 64 half ..
    // The first of these warps has one lane issue a stage's products, always a stage ahead of the one the warp empties.
    auto issue = [&](int st) {
      const int buf = st % kStages, ab = st & 1;
      if (!bar_wait(full(buf), (st / kStages) & 1, wait_polls(p)) || !bar_wait(acc_empty(ab), ((st >> 1) & 1) ^ 1, wait_polls(p))) return false;
      tc_after();
      const uint64_t a = tile_desc(tiles_base + buf * kStageBytes);
#pragma unroll
      for (int kk = 0; kk < kDepth / 16; ++kk)              // smallest terms first; 16 of c are 32 bytes of a row
#pragma unroll
        for (int t = 1; t <= 3; ++t)
          mma_f16(tmem + (2 * ab + (kk >> 1)) * kTile, a + 2 * kk, a + (uint64_t)(t * (kOpBytes >> 4)) + 2 * kk, (kk & 1) || t > 1);
      commit_to(empty(buf));
      commit_to(acc_full(ab));
      return true;
    };
    bool issuing = warp == kConvWarps && lane == 0;
    if (issuing) issuing = issue(0);
    __syncwarp();
    float acc[64];
#pragma unroll
    for (int n = 0; n < 64; ++n) acc[n] = 0.0f;
    for (int st = 0; st < n_stages; ++st) {
      const int ab = st & 1;
      if (issuing && st + 1 < n_stages) issuing = issue(st + 1);
      __syncwarp();
      if (!bar_wait(acc_full(ab), (st >> 1) & 1, wait_polls(p))) break;
      tc_after();
      const uint32_t at = tmem + ((uint32_t)(quad * 32) << 16) + 2 * ab * kTile + half * 64;
      uint32_t v[2][16];
      ld_acc16(at, v[0]);
#pragma unroll
      for (int k = 0; k < 8; ++k) {   // 16 columns of one accumulator, then of the other
        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
        if (k + 1 < 8) {
          ld_acc16(at + ((k + 1) & 3) * 16 + ((k + 1) >> 2) * kTile, v[(k + 1) & 1]);
        } else {
          tc_before();
          __syncwarp();
          if (lane == 0) bar_arrive(acc_empty(ab));
        }
#pragma unroll
        for (int n = 0; n < 16; ++n) acc[16 * (k & 3) + n] += __uint_as_float(v[k & 1][n]);
      }
    }
    float* out = p.out + (int64_t)split * p.part;
    const int i = i0 + quad * 32 + lane, jb = j0 + half * 64;
    if constexpr (TOKENS) {
#pragma unroll
      for (int n = 0; n < 64; n += 4)
        if (jb + n < p.J)             // J is a multiple of 4
          *reinterpret_cast<float4*>(out + (int64_t)i * p.ldo + jb + n) =
              make_float4(acc[n] * kScaleDown, acc[n + 1] * kScaleDown, acc[n + 2] * kScaleDown, acc[n + 3] * kScaleDown);
    } else {
#pragma unroll
      for (int n = 0; n < 64; ++n)
        if (jb + n < p.J) out[(int64_t)(jb + n) * p.ldo + i] = acc[n] * kScaleDown;
    }
    uint32_t most = 0;                // twice the largest magnitude's bits
#pragma unroll
    for (int n = 0; n < 64; ++n) most = max(most, __float_as_uint(acc[n]) << 1);
    if (most >= 2 * 0x7f800000u) plain_dots<TOKENS, G>(p, out, i, jb, it, c_begin, c_end);
  }
  tc_before();
  __syncthreads();
  if (warp == kConvWarps) {
    tc_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(kAccCols) : "memory");
  }
}

__global__ void __launch_bounds__(256) add_parts_kernel(const float4* parts, float4* out, int64_t n4, int splits) {
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
  dense_dot_kernel<TOKENS, G><<<grid, kDotThreads, kDotSmem, st>>>(p);
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
  add_parts_kernel<<<(unsigned)((n4 + 255) / 256), 256, 0, st>>>(reinterpret_cast<const float4*>(parts), reinterpret_cast<float4*>(out), n4, splits);
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
              (uint32_t)geo.nbc, log2_K, b == 1, d.i_tiles, d.tiles, d.split_depth};
#ifdef PB_DIAGNOSTICS
  p.polls = g_dot_polls.load();
  p.withhold = g_dot_withhold.load();
#endif
  const unsigned grid = (unsigned)(d.tiles * d.splits);
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

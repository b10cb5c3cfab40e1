// The f32 dots of dense_dot.cu for the shapes whose operands many tiles share: the same products, with the operands made
// ready for the tensor core once, by an element-wise kernel, instead of by every tile that reads them.
//
//   tokens == 0:  out[j, i] = sum_c g[j, c] * dq(Q)[i, c]      (dX = g W^T,  pratchya/_qualia/_qarr.py:620)
//   tokens == 1:  out[i, j] = sum_c dq(Q)[c, i] * g[c, j]      (dW = X^T g,  :621)
//
// One operand is exact in bf16 as it is, the other is kept as three bf16 terms, hi + mid + lo, which hold all 24 bits of an f32:
//   g in bf16:  g as it is; the dequantized values (the one f32 rounding that dequantizing makes) as three terms.  Any grid.  For dX with
//               a super-group's factor that belongs to rows of Q (out's columns) the fp8 values times their block's power of two and the factor's,
//               one term: the rest of that factor, a number in [1, 2), goes to the finished sum, and every product is one tensor-core product.
//   g in f32:   the fp8 values times their block's power of two (exact; where it is not, a NaN, see below); g as three terms, times
//               the super-group's f32 factor where that varies along c (tokens == 1, one set of terms per 1024 columns of
//               Q; one f32 rounding), while of a factor that belongs to a column of dX the power of two goes to Q's values and the rest to the finished sum
//               (all of it there, and rows 2^-60 and less of a large super-group leave f32's range before the sum is scaled back).
// Every f32 product is then exact in its tensor-core products, and the accumulator is emptied into f32 registers every 64 of c
// (the tensor core's own additions do not round to nearest; dense_dot.cu empties every 32): the low terms of all 64 go first, so that
// four additions meet a sum of full size, as many as there, and half as many f32 additions follow.  Contractions of a few hundred have
// few of those to save, and where the low terms are the fp8 operand's the four are all that is left: bf16 g over fewer than
// 384 of c empties every 32.  2-norm errors against 64 bits, dense_dot_kernel | every 64 | every 32, dW of 2048 x 2048, bf16 g: operands of
// one sign, 128 of c 8.4e-8 | 8.7e-8 | 6.3e-8, 256 8.7e-8 | 8.8e-8 | 6.7e-8, 384 9.5e-8 | 9.1e-8 | 7.6e-8, 2048 13.8e-8 | 11.4e-8 | 12.6e-8; of mixed signs, 128
// 11.3e-8 | 8.3e-8 | 7.0e-8, 2048 18.1e-8 | 13.1e-8 | 15.8e-8.  f32 g, one sign, 128: 8.5e-8 | 5.6e-8 | 5.6e-8, 2048 13.8e-8 | 9.4e-8 | 12.3e-8.
// The terms carry an exact 2^40, which keeps
// them above bf16's subnormals.  A sum that is not finite, for an infinity or a NaN in the operands, an overflow of a scaled
// term or a power of two that bf16 does not hold, is made again with f32 products of dequantized values, behind the last tile.
//
// One term for three, us in a CUDA graph: 3000 tokens, 2048 x 2048 79 -> 39, 1000 tokens 40 -> 23; 2-norm errors 1.31e-7 -> 1.06e-7.  What it is bound
// by then is waits and issuing, so its stages hold 64 of c, not 32 (53 -> 44 us), and the stores of a finished tile: one address that
// moves on, where sixteen columns a time through shared memory and bulk copies took 44 -> 39, and an address and a look at every sum more
// (f32 dW of 300 tokens, 2048 x 4096: 30.5 -> 26.6).
//
// Element-wise kernel: bound by its bytes.  Main kernel: persistent, one CTA per SM; a tile is 128 rows of the three-term operand
// by N of the other; a stage is 32 of c of both (64 with one term), by TMA, K-major (64-byte swizzle, 128 with one term) for tokens == 0 and with c
// outermost, as it lies in memory, for tokens == 1 (128-byte swizzle): no transpose anywhere.  Warp 0 loads, warp 1 issues six (four)
// tcgen05.mma a stage, eight warps empty one accumulator while the other fills.  N is 256, 192 or 128, whichever fills whole waves of SMs best.
#include <cuda.h>

#include <algorithm>
#include <atomic>

#include "common.cuh"
#include "split_dot.cuh"

namespace pb {
namespace {

constexpr int kTermRows = 128;        // of the three-term operand, per tile
constexpr int kDepth = 32;            // c per stage
constexpr int kGroup = 2;             // stages per accumulator, at most
constexpr int kShortDepth = 384;      // of c, from which bf16 g takes that many
constexpr int kDrainWarps = 8;
constexpr int kThreads = 64 + 32 * kDrainWarps;
constexpr uint32_t kWaitPolls = 1u << 21;               // a poll parks for up to 2 us: about four seconds at most
constexpr float kScaleUp = 0x1p40f, kScaleDown = 0x1p-40f;
constexpr float kQScaleUp = 0x1p10f;  // of it, Q's share where g is f32 and Q's values hold their super-group's power of two
constexpr size_t kMaxTerms = (size_t)512 << 20;         // bytes of three-term operand at a time: more of it takes several rounds (1024 of its rows at least)

constexpr int kOutCols = 16;           // of a finished tile that a thread stores at a time

template <int N, bool TOKENS, bool G32, int TERMS>
struct Cfg {
  static constexpr int kUnits = TERMS == 1 ? 2 : 1;    // of kDepth, per stage: one term's stages are otherwise more waiting and issuing than products
  static constexpr int kTermBytes = kTermRows * kDepth * 2 * kUnits;
  static constexpr int kStageBytes = TERMS * kTermBytes + N * kDepth * 2 * kUnits;
  static constexpr int kStages = TERMS == 1 ? (N == 256 ? 4 : (N == 192 ? 5 : 6)) : (N == 256 ? 5 : 6);
  static constexpr int kSmem = kStages * kStageBytes + 1024;      // 1024: the tiles start on a swizzle atom
  static_assert(kSmem + 512 <= 232448, "an SM's shared memory");
};

__device__ unsigned int g_split_status; // 0, or PB_ERR_DEVICE_TIMEOUT once a bounded wait ran out

// What a finished sum that is not finite is made again from, and where it goes.
struct DotSource {
  const uint8_t* q; const uint8_t* sc8; const float* sc32;
  const void* g;
  int64_t ldq, ldg;
  uint32_t nbc, log2_K, log2_a, log2_b;      // blocks per block row, of log2 sizes
  int C;
};

struct SplitParams {
  DotSource src;
  float* out;                         // or the parts, [splits][out]
  const float* factor;                // tokens == 0, one factor per 128 of i (sc32), whose rest the finished sums take: of the tile's columns with f32 g, of its rows with one term
  int64_t ld, part;                   // row stride of out, elements of a part
  int rows, cols;                     // extents of the three-term operand and of the other
  int row_first;                      // the first of these rows, for the sums that are made again
  int row_tiles, tiles, splits, units, units_per_split;
  int cols_per_variant;               // columns of Q that share a set of terms
  int group;                          // stages per accumulator: 1 or kGroup
  uint32_t polls;
  int withhold;                       // diagnostics build: the first stage is never filled
};

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void bar_init(uint32_t bar, uint32_t count) { asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count)); }
__device__ __forceinline__ void bar_arrive(uint32_t bar) { asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory"); }
__device__ __forceinline__ void bar_expect(uint32_t bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
// Bounded: false, and the status word set, when the poll budget ran out.
__device__ __forceinline__ bool bar_wait(uint32_t bar, uint32_t parity, uint32_t polls) {
  for (uint32_t n = 0; n < polls; ++n) {
    uint32_t ok;
    asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, 2000;\n\tselp.u32 %0, 1, 0, p;\n\t}"
                 : "=r"(ok) : "r"(bar), "r"(parity) : "memory");
    if (ok) return true;
  }
  atomicExch(&g_split_status, (unsigned int)PB_ERR_DEVICE_TIMEOUT);
  return false;
}
__device__ __forceinline__ void load_box(uint32_t dst, const CUtensorMap* map, int x, int y, int z, uint32_t bar) {
  asm volatile("cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];"
               ::"r"(dst), "l"(map), "r"(x), "r"(y), "r"(z), "r"(bar) : "memory");
}
__device__ __forceinline__ void tc_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void commit_to(uint32_t bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}
// Operand tiles (descriptor version 1).  K-major: rows of 64 bytes (32 of c), 8-row groups 512 bytes apart, 64-byte swizzle; with 64 of c
// (UNITS == 2) twice of each.  c outermost: 32 rows of 128 bytes (64 of the operand's rows), eight c 1024 bytes apart, the next 64 rows 4096,
// 128-byte swizzle.
template <bool TOKENS, int UNITS>
__device__ __forceinline__ uint64_t tile_desc(uint32_t addr) {
  const uint64_t start = (uint64_t)((addr & 0x3ffffu) >> 4) | (1ull << 46);
  if (TOKENS) return start | ((uint64_t)(4096 >> 4) << 16) | ((uint64_t)(1024 >> 4) << 32) | (2ull << 61);
  return start | (1ull << 16) | ((uint64_t)(512 * UNITS >> 4) << 32) | ((UNITS == 2 ? 2ull : 4ull) << 61);
}
template <bool TOKENS> constexpr uint32_t kStep16 = TOKENS ? 16 * 128 / 16 : 32 / 16;      // 16 of c further, in descriptor units
// kind::f16: f32 accumulator, both operands bf16, both K-major or both not
template <int N, bool TOKENS>
constexpr uint32_t kInstr = (1u << 4) | (1u << 7) | (1u << 10) | (TOKENS ? 3u << 15 : 0u) | ((uint32_t)(N >> 3) << 17) | ((uint32_t)(kTermRows >> 4) << 24);
template <int N, bool TOKENS>
__device__ __forceinline__ void mma_f16(uint32_t d, uint64_t a, uint64_t b, uint32_t accumulate) {
  asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\ttcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
               ::"r"(d), "l"(a), "l"(b), "r"(kInstr<N, TOKENS>), "r"(accumulate) : "memory");
}
__device__ __forceinline__ void ld_acc16(uint32_t taddr, uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
        "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr) : "memory");
}

__device__ __forceinline__ void st_32bytes(void* at, const uint32_t (&v)[8]) {
  asm volatile("st.global.v8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};"
               ::"l"(at), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]) : "memory");
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

// ---- making the operands ready ------------------------------------------------------------------------------------
struct PrepareParams {
  const uint8_t* q; const uint8_t* sc8; const float* sc32;      // null: this round's q is there already
  const float* g;                     // f32 g, at the round's first element; null where g is used as it is
  __nv_bfloat16* q_out;               // exact values, or [3] terms, of the round's rows and columns of Q
  __nv_bfloat16* g_out;               // [variants][3][g_rows, g_cols]
  int64_t q_plane, g_plane, ldq, ldg;
  uint32_t q_row0, q_col0;
  FastDiv q_vecs, g_vecs;             // vectors of 16 (q) and 8 (g) elements per row
  uint32_t n_q, n_g, q_blocks;        // vectors in all; thread blocks that work on q
  uint32_t nbc, log2_a, log2_b, log2_K;
  int variants;                       // tokens == 1: sets of terms of g, K blocks of a row of Q each
};

// A super-group's factor as a power of two and what is left of it, in [1, 2) (below for a subnormal one).  An infinite one is left to the
// power, and the sums that meet it are made again.
__device__ __forceinline__ float power_of(float f) { return __uint_as_float(max(__float_as_uint(f) & 0x7f800000u, 0x00800000u)); }
__device__ __forceinline__ float rest_of(float f) {
  const uint32_t bits = __float_as_uint(f);
  return bits & 0x7f800000u ? __uint_as_float((bits & 0x807fffffu) | 0x3f800000u) : f * 0x1p126f;
}

// sixteen values of Q from their bytes: terms of the dequantized values (TERMS), or value times its block's power of two, and with POWER
// (the finished sums take the rest of the super-group's factor) times that one's and `up`
template <bool TERMS, bool POWER>
__device__ __forceinline__ void prepare_q(const PrepareParams& p, uint32_t v, float up) {
  const uint32_t in_row = p.q_vecs.div(v), row = p.q_row0 + in_row, col = p.q_col0 + (v - in_row * p.q_vecs.d) * 16;
  const uint4 bytes = __ldg(reinterpret_cast<const uint4*>(p.q + (int64_t)row * p.ldq + col));
  const uint32_t words[4] = {bytes.x, bytes.y, bytes.z, bytes.w};
  const uint32_t id0 = (row >> p.log2_a) * p.nbc + (col >> p.log2_b);
  auto multiplier = [&](uint32_t id) {
    const float two = e8m0_to_f32(__ldg(p.sc8 + id));
    if (!TERMS && !POWER) return two;
    const float group = __ldg(p.sc32 + (id >> p.log2_K));
    return TERMS ? __fmul_rn(__fmul_rn(two, group), kScaleUp * 0.0078125f) : two * (up * 0.0078125f) * power_of(group);
  };
  const float m0 = multiplier(id0);
  uint32_t hi[8], mid[8], lo[8];
#pragma unroll
  for (int e = 0; e < 8; ++e) {
    const float2 x = fp8x2_to_f32x2<PB_E4M3>((uint16_t)(words[e >> 1] >> (16 * (e & 1))));
    const float2 m = p.log2_b == 0 ? make_float2(2 * e ? multiplier(id0 + 2 * e) : m0, multiplier(id0 + 2 * e + 1)) : make_float2(m0, m0);
    const float2 f = make_float2(__fmul_rn(x.x, m.x), __fmul_rn(x.y, m.y));
    if (TERMS) {
      split3(f, hi[e], mid[e], lo[e]);
    } else {        // four bits times a power of two: exact in bf16 unless it is subnormal
      auto exact = [](float a) { return a != 0.0f && fabsf(a) < 0x1p-126f ? __uint_as_float(0x7fffffffu) : a; };
      hi[e] = pack_bf16x2(exact(f.x), exact(f.y));
    }
  }
  __nv_bfloat16* out = p.q_out + (size_t)v * 16;
  st_32bytes(out, hi);
  if (TERMS) {
    st_32bytes(out + p.q_plane, mid);
    st_32bytes(out + 2 * p.q_plane, lo);
  }
}

// eight values of g as terms, once per set
template <bool TOKENS>
__device__ __forceinline__ void prepare_g(const PrepareParams& p, uint32_t v) {
  const uint32_t row = p.g_vecs.div(v), col = (v - row * p.g_vecs.d) * 8;
  const float4* src = reinterpret_cast<const float4*>(p.g + (size_t)row * p.ldg + col);
  const float4 a = __ldg(src), b = __ldg(src + 1);
  const float2 x[4] = {make_float2(a.x, a.y), make_float2(a.z, a.w), make_float2(b.x, b.y), make_float2(b.z, b.w)};
  for (int set = 0; set < (TOKENS ? p.variants : 1); ++set) {
    const float m = TOKENS ? __fmul_rn(__ldg(p.sc32 + ((row * p.nbc) >> p.log2_K) + set), kScaleUp * 0.0078125f) : kScaleUp / kQScaleUp;
    uint32_t hi[4], mid[4], lo[4];
#pragma unroll
    for (int e = 0; e < 4; ++e) split3(__fmul2_rn(x[e], make_float2(m, m)), hi[e], mid[e], lo[e]);
    uint4* out = reinterpret_cast<uint4*>(p.g_out) + (size_t)set * 3 * (p.g_plane / 8) + v;
    out[0] = make_uint4(hi[0], hi[1], hi[2], hi[3]);
    out[p.g_plane / 8] = make_uint4(mid[0], mid[1], mid[2], mid[3]);
    out[2 * (p.g_plane / 8)] = make_uint4(lo[0], lo[1], lo[2], lo[3]);
  }
}

// G32: f32 g.  TERMS: of Q, where g is used as it is.  Blocks [0, q_blocks) work on Q, the others on g.
template <bool TOKENS, bool G32, int TERMS>
__global__ void __launch_bounds__(256) split_prepare_kernel(const __grid_constant__ PrepareParams p) {
  grid_wait();
  if (blockIdx.x < p.q_blocks) {
    const uint32_t v = blockIdx.x * 256 + threadIdx.x;
    if (v < p.n_q) prepare_q<!G32 && TERMS == 3, !TOKENS>(p, v, G32 ? kQScaleUp : kScaleUp);
  } else if (G32) {
    const uint32_t v = (blockIdx.x - p.q_blocks) * 256 + threadIdx.x;
    if (v < p.n_g) prepare_g<TOKENS>(p, v);
  }
}

// ---- the products -------------------------------------------------------------------------------------------------
// The sums of this warp's part of a tile (rows p.row_first + 32 quad .., columns cb .. cb + kCols) that are not finite, made again with f32
// products of dequantized values, one after the other in c: sixteen columns a pass over c.  A lane holds its row's value of a c
// and one column's, which goes round by shuffles.  All of 2048 x 2048 sums: 4.2 ms over 3000 of c,
// 32 to 40 over 16384 (dense_dot_kernel 7.4 to 8.4 and 58 to 61).
template <int N, bool TOKENS, bool G32>
__device__ __noinline__ void remake_sums(const SplitParams& p, float* out, int row0, int cb, int c_begin, int c_end) {
  constexpr bool kLanes = TOKENS == G32;
  const DotSource& s = p.src;
  const int lane = threadIdx.x & 31, row = row0 + lane, at_row = min(row, p.rows - 1);
  auto q_value = [&](int i, int c) {
    const uint32_t r = TOKENS ? c : i, col = TOKENS ? i : c;
    const uint32_t id = (r >> s.log2_a) * s.nbc + (col >> s.log2_b);
    const float x_sc = __fmul_rn(e8m0_to_f32(__ldg(s.sc8 + id)), __ldg(s.sc32 + (id >> s.log2_K)));
    return __fmul_rn(__fmul_rn(fp8x2_to_f32x2<PB_E4M3>((uint16_t)__ldg(s.q + (int64_t)r * s.ldq + col)).x, x_sc), 0.0078125f);
  };
  auto g_value = [&](int j, int c) {
    const int64_t at = TOKENS ? (int64_t)c * s.ldg + j : (int64_t)j * s.ldg + c;
    return G32 ? __ldg(static_cast<const float*>(s.g) + at) : __bfloat162float(static_cast<const __nv_bfloat16*>(s.g)[at]);
  };
#pragma unroll 1
  for (int c0 = cb; c0 < cb + N / 2 && c0 < p.cols; c0 += 16) {
    auto place = [&](int n) { return out + (kLanes ? (int64_t)(c0 + n) * p.ld + row : (int64_t)row * p.ld + c0 + n); };
    uint32_t odd = 0;
#pragma unroll 1
    for (int n = 0; n < 16; ++n)
      if (row < p.rows && c0 + n < p.cols) odd |= (__float_as_uint(*place(n)) << 1 >= 2 * 0x7f800000u ? 1u : 0u) << n;
    if (!__any_sync(0xffffffffu, odd != 0)) continue;
    const int at_col = min(c0 + (lane & 15), p.cols - 1);
    float acc[16];
#pragma unroll
    for (int n = 0; n < 16; ++n) acc[n] = 0.0f;
#pragma unroll 4
    for (int c = c_begin; c < c_end; ++c) {
      const float mine = G32 ? g_value(p.row_first + at_row, c) : q_value(p.row_first + at_row, c);
      const float theirs = G32 ? q_value(at_col, c) : g_value(at_col, c);
#pragma unroll
      for (int n = 0; n < 16; ++n) acc[n] = fmaf(mine, __shfl_sync(0xffffffffu, theirs, n), acc[n]);
    }
#pragma unroll
    for (int n = 0; n < 16; ++n)
      if (odd >> n & 1) *place(n) = acc[n];
  }
}

// N columns per tile; TOKENS: c is the operands' outer dimension; G32: the terms are g's (rows are j, columns i), else Q's (rows i, columns j);
// TERMS: 3, or 1 where Q's exact values are multiplied and the rest of their super-group's factor goes to the finished sums.
template <int N, bool TOKENS, bool G32, int TERMS>
__global__ void __launch_bounds__(kThreads, 1)
split_dot_kernel(const __grid_constant__ CUtensorMap map_terms, const __grid_constant__ CUtensorMap map_other, const __grid_constant__ SplitParams p) {
  using C = Cfg<N, TOKENS, G32, TERMS>;
  constexpr bool kLanes = TOKENS == G32;        // out is contiguous along the tile's rows, that is across the lanes of a warp
  constexpr int kCols = N / 2;                  // of an emptying thread
  extern __shared__ unsigned char split_smem[];
  __shared__ __align__(8) uint64_t bars[2 * C::kStages + 4];
  __shared__ uint32_t tmem_slot;
  const uint32_t base = (smem_u32(split_smem) + 1023u) & ~1023u;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  auto full = [&](int s) { return smem_u32(&bars[s]); };
  auto empty = [&](int s) { return smem_u32(&bars[C::kStages + s]); };
  auto acc_full = [&](int a) { return smem_u32(&bars[2 * C::kStages + a]); };
  auto acc_empty = [&](int a) { return smem_u32(&bars[2 * C::kStages + 2 + a]); };
  if (tid == 0) {
    for (int s = 0; s < C::kStages; ++s) { bar_init(full(s), 1); bar_init(empty(s), 1); }
    for (int a = 0; a < 2; ++a) { bar_init(acc_full(a), 1); bar_init(acc_empty(a), kDrainWarps); }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_slot)), "r"(512u) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tc_before();
  __syncthreads();
  tc_after();
  const uint32_t tmem = *(volatile uint32_t*)&tmem_slot;
  grid_wait();
  const int items = p.tiles * p.splits;
  auto item_of = [&](int w, int& row0, int& col0, int& u_begin, int& u_end) {
    const int split = w / p.tiles, tile = w - split * p.tiles;
    row0 = tile % p.row_tiles * kTermRows; col0 = tile / p.row_tiles * N;
    u_begin = split * p.units_per_split; u_end = min(p.units, u_begin + p.units_per_split);
    return split;
  };

  if (warp == 0) {
    if (lane == 0) {
      uint32_t it = 0;
      bool ok = true;
      for (int w = blockIdx.x; w < items && ok; w += gridDim.x) {
        int row0, col0, u, u_end;
        item_of(w, row0, col0, u, u_end);
        const int set = TOKENS && G32 ? 3 * (col0 / p.cols_per_variant) : 0;
        for (; u < u_end; u += C::kUnits, ++it) {      // a last stage that ends behind c is filled with zeros
          const int s = it % C::kStages;
          if (!bar_wait(empty(s), ((it / C::kStages) & 1) ^ 1, p.polls)) { ok = false; break; }
          if (p.withhold && it == 0) continue;
          const uint32_t bar = full(s), at = base + s * C::kStageBytes, other = at + TERMS * C::kTermBytes;
          bar_expect(bar, C::kStageBytes);
#pragma unroll
          for (int t = 0; t < TERMS; ++t) {
            if (TOKENS) {
              load_box(at + t * C::kTermBytes, &map_terms, row0, u * kDepth, set + t, bar);
              load_box(at + t * C::kTermBytes + 4096, &map_terms, row0 + 64, u * kDepth, set + t, bar);
            } else {
              load_box(at + t * C::kTermBytes, &map_terms, u * kDepth, row0, t, bar);
            }
          }
          if (TOKENS) {
#pragma unroll
            for (int b = 0; b < N / 64; ++b) load_box(other + b * 4096, &map_other, col0 + 64 * b, u * kDepth, 0, bar);
          } else {
            load_box(other, &map_other, u * kDepth, col0, 0, bar);
          }
        }
      }
      // leave only when every copy this thread started has landed (bounded)
      for (uint32_t k = it > (uint32_t)C::kStages ? it - C::kStages : 0; k < it; ++k)
        if (!(p.withhold && k == 0)) (void)bar_wait(full(k % C::kStages), (k / C::kStages) & 1, p.polls);
    }
  } else if (warp == 1) {
    if (lane == 0) {
      uint32_t it = 0, group = 0;
      bool ok = true;
      for (int w = blockIdx.x; w < items && ok; w += gridDim.x) {
        int row0, col0, u, u_end;
        item_of(w, row0, col0, u, u_end);
        for (; u < u_end; u += p.group, ++group) {
          const int ab = group & 1, depth = C::kUnits == 2 ? 1 : min(p.group, u_end - u);      // stages
          if (!bar_wait(acc_empty(ab), ((group >> 1) & 1) ^ 1, p.polls)) { ok = false; break; }
          constexpr int kMost = kGroup / C::kUnits;
          uint32_t at[kMost], freed[kMost];
#pragma unroll
          for (int h = 0; h < kMost; ++h) {
            if (h >= depth) break;
            const int s = it % C::kStages;
            if (!bar_wait(full(s), (it / C::kStages) & 1, p.polls)) { ok = false; break; }
            at[h] = base + s * C::kStageBytes; freed[h] = empty(s);
            ++it;
          }
          if (!ok) break;
          tc_after();
          // Smallest terms first, over all of the group: only the last few additions meet a sum of full size.
#pragma unroll
          for (int t = TERMS - 1; t >= 0; --t)
#pragma unroll
            for (int h = 0; h < kMost; ++h) {
              if (h >= depth) break;
              const uint64_t a = tile_desc<TOKENS, C::kUnits>(at[h]), b = tile_desc<TOKENS, C::kUnits>(at[h] + TERMS * C::kTermBytes);
#pragma unroll
              for (int k = 0; k < C::kUnits * kDepth / 16; ++k)
                mma_f16<N, TOKENS>(tmem + ab * N, a + (uint64_t)(t * (C::kTermBytes >> 4) + k * kStep16<TOKENS>), b + (uint64_t)(k * kStep16<TOKENS>), h > 0 || k > 0 || t < TERMS - 1);
            }
#pragma unroll
          for (int h = 0; h < kMost; ++h)
            if (h < depth) commit_to(freed[h]);
          commit_to(acc_full(ab));
        }
      }
    }
  } else {
    const int quad = warp & 3, half = (warp - 2) >> 2;      // rows 32 quad .., columns kCols half ..
    const int r = quad * 32 + lane;             // the thread's row of the tile
    uint32_t group = 0;
    bool ok = true, odd = false;        // odd: some sum of this thread is not finite
    for (int w = blockIdx.x; w < items && ok; w += gridDim.x) {
      int row0, col0, u, u_end;
      const int split = item_of(w, row0, col0, u, u_end);
      float acc[kCols];
#pragma unroll
      for (int n = 0; n < kCols; ++n) acc[n] = 0.0f;
      for (; u < u_end; u += p.group, ++group) {
        const int ab = group & 1;
        ok = __all_sync(0xffffffffu, bar_wait(acc_full(ab), (group >> 1) & 1, p.polls));
        if (!ok) break;
        tc_after();
        const uint32_t at = tmem + ((uint32_t)(quad * 32) << 16) + ab * N + half * kCols;
        uint32_t v[2][16];
        ld_acc16(at, v[0]);
#pragma unroll
        for (int k = 0; k < kCols / 16; ++k) {
          asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
          if (k + 1 < kCols / 16) {
            ld_acc16(at + (k + 1) * 16, v[(k + 1) & 1]);
          } else {
            tc_before();
            __syncwarp();
            if (lane == 0) bar_arrive(acc_empty(ab));
          }
#pragma unroll
          for (int n = 0; n < 16; n += 2) {
            const float2 s = __fadd2_rn(make_float2(acc[16 * k + n], acc[16 * k + n + 1]), make_float2(__uint_as_float(v[k & 1][n]), __uint_as_float(v[k & 1][n + 1])));
            acc[16 * k + n] = s.x; acc[16 * k + n + 1] = s.y;
          }
        }
      }
      if (!ok) break;
      const int cb = col0 + half * kCols;
      float* out = p.out + (int64_t)split * p.part;
      constexpr bool kFactor = TERMS == 1 || (!TOKENS && G32);
      float row_factor = 1.0f;
      if (TERMS == 1) row_factor = rest_of(__ldg(p.factor + (((uint32_t)(p.row_first + row0) / 128 * p.src.nbc) >> p.src.log2_K)));
      float2 zero = make_float2(0.0f, 0.0f);    // times 0: NaN where a sum is not finite
#pragma unroll
      for (int k = 0; k < kCols / kOutCols; ++k) {
        const int c0 = cb + k * kOutCols;
        if (c0 >= p.cols) break;
        const float down = kScaleDown * (TERMS == 1 ? row_factor : (kFactor ? rest_of(__ldg(p.factor + (((uint32_t)c0 / 128 * p.src.nbc) >> p.src.log2_K))) : 1.0f));
#pragma unroll
        for (int n = kOutCols * k; n < kOutCols * (k + 1); n += 2) {
          zero = __ffma2_rn(make_float2(acc[n], acc[n + 1]), make_float2(0.0f, 0.0f), zero);
          const float2 v = __fmul2_rn(make_float2(acc[n], acc[n + 1]), make_float2(down, down));
          acc[n] = v.x; acc[n + 1] = v.y;
        }
        const float* v = acc + kOutCols * k;
        if (row0 + r >= p.rows) continue;
        if constexpr (kLanes) {
          float* to = out + (int64_t)c0 * p.ld + row0 + r;
          if (c0 + kOutCols <= p.cols) {
#pragma unroll
            for (int n = 0; n < kOutCols; ++n, to += p.ld) *to = v[n];
          } else {
#pragma unroll
            for (int n = 0; n < kOutCols; ++n, to += p.ld)
              if (c0 + n < p.cols) *to = v[n];
          }
        } else {
          float* to = out + (int64_t)(row0 + r) * p.ld + c0;
#pragma unroll
          for (int n = 0; n < kOutCols; n += 4)
            if (c0 + n < p.cols) *reinterpret_cast<float4*>(to + n) = make_float4(v[n], v[n + 1], v[n + 2], v[n + 3]);
        }
      }
      odd |= row0 + r < p.rows && !(zero.x + zero.y == 0.0f);
    }
    // Sums that are not finite are made again when the CTA's tiles are done: nothing waits for these warps any more, however long it takes
    // (with all of a long contraction's sums to make, longer than a bounded wait lasts).
    if (__any_sync(0xffffffffu, ok && odd)) {
#pragma unroll 1
      for (int w = blockIdx.x; w < items; w += gridDim.x) {
        int row0, col0, u, u_end;
        const int split = item_of(w, row0, col0, u, u_end);
        remake_sums<N, TOKENS, G32>(p, p.out + (int64_t)split * p.part, row0 + quad * 32, col0 + half * kCols, u * kDepth, min(p.src.C, u_end * kDepth));
      }
    }
  }
  tc_before();
  __syncthreads();
  if (warp == 1) {
    tc_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512u) : "memory");
  }
}

// ---- host side ----------------------------------------------------------------------------------------------------
using EncodeFn = CUresult (*)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*,
                              const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                              CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

// planes of [outer, inner] bf16
int make_map(CUtensorMap* map, const void* base, int64_t inner, int64_t outer, int64_t ld, int64_t planes, int64_t plane, int box_inner, int box_outer) {
  EncodeFn encode = reinterpret_cast<EncodeFn>(tensor_map_encoder());
  if (!encode) return fail(PB_ERR_CUDA, "cuTensorMapEncodeTiled is not available from this driver");
  const cuuint64_t dims[3] = {(cuuint64_t)inner, (cuuint64_t)outer, (cuuint64_t)planes};
  const cuuint64_t strides[2] = {(cuuint64_t)(ld * 2), (cuuint64_t)(plane * 2)};
  const cuuint32_t box[3] = {(cuuint32_t)box_inner, (cuuint32_t)box_outer, 1}, step[3] = {1, 1, 1};
  const CUresult r = encode(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, const_cast<void*>(base), dims, strides, box, step, CU_TENSOR_MAP_INTERLEAVE_NONE,
                            box_inner == 64 ? CU_TENSOR_MAP_SWIZZLE_128B : CU_TENSOR_MAP_SWIZZLE_64B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) return fail(PB_ERR_CUDA, "cuTensorMapEncodeTiled (split dot) failed with CUresult %d", (int)r);
  return PB_OK;
}

#ifdef PB_DIAGNOSTICS
std::atomic<uint32_t> g_split_polls{kWaitPolls};
std::atomic<int> g_split_withhold{0};
#endif

template <int N, bool TOKENS, bool G32, int TERMS>
int launch(const CUtensorMap& terms, const CUtensorMap& other, const SplitParams& p, cudaStream_t st) {
  PB_CUDA_TRY(cudaFuncSetAttribute(split_dot_kernel<N, TOKENS, G32, TERMS>, cudaFuncAttributeMaxDynamicSharedMemorySize, Cfg<N, TOKENS, G32, TERMS>::kSmem));      // per device
  const int items = p.tiles * p.splits;
  launch_behind(split_dot_kernel<N, TOKENS, G32, TERMS>, items < sm_count() ? items : sm_count(), kThreads, Cfg<N, TOKENS, G32, TERMS>::kSmem, st, terms, other, p);
  PB_LAUNCH_CHECK("split_dot_kernel");
  return PB_OK;
}
template <bool TOKENS, bool G32, int TERMS>
int launch_n(int n, const CUtensorMap& terms, const CUtensorMap& other, const SplitParams& p, cudaStream_t st) {
  if (n == 256) return launch<256, TOKENS, G32, TERMS>(terms, other, p, st);
  return n == 192 ? launch<192, TOKENS, G32, TERMS>(terms, other, p, st) : launch<128, TOKENS, G32, TERMS>(terms, other, p, st);
}
template <bool TOKENS, bool G32, int TERMS>
int launch_prepare(const PrepareParams& p, cudaStream_t st) {
  launch_behind(split_prepare_kernel<TOKENS, G32, TERMS>, p.q_blocks + (G32 ? (p.n_g + 255) / 256 : 0), 256, 0, st, p);
  PB_LAUNCH_CHECK("split_prepare_kernel");
  return PB_OK;
}

// Where this form is taken.  What it makes ready has to be shared, and its two launches and the passes over the operands want something to do.
// us, dense_dot_kernel | this form, inside a graph:
// One term (a bf16 cotangent's dX), everywhere: 128 x 128 8 rows 7.1 | 5.3, 8000 6.9 | 7.0; 512 x 128 500 rows 6.8 | 6.9; 2048 x 2048 8 rows 11.6 | 10.3,
// 64 11.4 | 10.5, 128 11.3 | 11.3, 1000 37.5 | 19.8, 3000 104 | 34; 1024 x 4096 128 rows 11.8 | 12.2; 8192 x 2048 8 rows 22.5 | 20.4, 64 22.9 | 20.4, 2000 274 | 80.
// f32 dX, 2048 x 2048: 100 rows 12.0 | 14.2, 200 16.3 | 17.6, 500 25.1 | 24.6, 1000 39.6 | 35.6, 3000 110 | 83; 1024 x 1024: 500 rows 11.9 | 13.7, 3000 41 | 28;
// 2048 x 128: 2000 rows 10.6 | 15.7, 8000 25.4 | 34.0; 128 x 2048: 8000 rows 26 | 48.
// dW, 2048 x 2048, f32: 64 rows 8.9 | 9.8, 200 15.0 | 13.4, 3000 100 | 77, bf16: 64 rows 9.0 | 13.5, 200 14.9 | 16.3, 300 17.2 | 18.0, 500 23.4 | 21.7,
// 3000 110 | 67; 1024 x 1024, bf16: 200 rows 9.3 | 11.0, 500 13.9 | 13.1, 8000 77 | 67; 4096 x 512, f32: 500 rows 13.6 | 15.1, 16000 323 | 267; 2048 x 128,
// f32: 8000 rows 21.6 | 29.6.
// The lines of the last two have sizes on this form's side that take it up to half as long again, next to them: it is the more precise of the
// two (the errors above), and no size's sums are to become less precise for it.
bool split_dot_pays(int tokens, bool exact, int64_t I, int64_t J, int64_t C) {
  const double products = (double)I * (double)J * (double)C;
  if (exact) return true;
  if (I < 512 || J < 512) return false;
  if (tokens) return C >= 192 || products >= 0x1p28;
  return products >= 0x1p29 && J >= 192;
}

int log2_of(int64_t v) { int l = 0; while ((1ll << l) < v) ++l; return l; }

}  // namespace

// I x J outputs, C the contraction.  False: dense_dot.cu's kernel.
bool split_dot_plan(int tokens, int64_t rows, int64_t cols, int a, int b, int64_t g_free, bool g_bf16, SplitDotPlan* d) {
  Geometry geo;
  if (make_geometry(rows, cols, a, b, &geo)) return false;
  const int64_t I = tokens ? cols : rows, C = tokens ? rows : cols, J = g_free;
  if (J % 8 != 0 && tokens) return false;             // rows of g are whole 16-byte units of bf16
  if (C % 8 != 0 && !tokens) return false;
  if ((geo.K & (geo.K - 1)) || I > (1ll << 30) || J > (1ll << 30) || C > (1ll << 30) || rows * cols / 8 > kMaxIndexed || J * C / 8 > kMaxIndexed || geo.Nb > kMaxIndexed) return false;
  d->variants = 1;
  if (!g_bf16) {
    if (b != 128) return false;                       // a factor per c for every 128 of i
    if (tokens) {
      if (geo.nbc % geo.K == 0 && (geo.K >= 4 || geo.nbc == geo.K)) d->variants = (int)(geo.nbc / geo.K);      // 512 columns share a set at least
      else if (geo.K % geo.nbc != 0) return false;    // super-groups that end inside a row of Q
    } else if (geo.K % geo.nbc != 0) {
      return false;                                   // ... a factor that varies along c
    }
  }
  d->log2_K = log2_of(geo.K); d->nbc = (int)geo.nbc;
  d->units = (int)((C + kDepth - 1) / kDepth);
  // The three-term operand's rows are the tile's 128, the other's columns its N.
  d->exact = g_bf16 && !tokens && b == 128 && geo.K % geo.nbc == 0;      // a factor per 128 of i
  const int64_t R = g_bf16 ? I : J, S = g_bf16 ? J : I, row_bytes = (d->exact ? 2 : 6) * (int64_t)d->variants * C;
  d->slab = std::min(R, std::max<int64_t>(1024, (int64_t)kMaxTerms / row_bytes / 1024 * 1024));
  d->row_tiles = (int)((d->slab + kTermRows - 1) / kTermRows);
  const int sms = sm_count();
  int64_t best = -1;
  for (int n : {256, 192, 128}) {
    if (d->variants > 1 && I / d->variants % n != 0) continue;      // a tile's columns share their set of terms
    const int64_t tiles = d->row_tiles * ((S + n - 1) / n), waves = (tiles + sms - 1) / sms, cost = waves * (d->exact ? n + kTermRows : n);
    if (best < 0 || cost < best) { best = cost; d->n = n; d->tiles = (int)tiles; }
    if (tiles > kMaxIndexed / 64) return false;
  }
  d->splits = 1;
  if (d->tiles < sms) d->splits = (int)std::min<int64_t>(sms / d->tiles, d->units / 8);
  if (d->splits < 1 || d->slab < R) d->splits = 1;
  d->units_per_split = ((d->units + d->splits - 1) / d->splits + kGroup - 1) / kGroup * kGroup;
  d->splits = (d->units + d->units_per_split - 1) / d->units_per_split;
  auto align = [](size_t v) { return (v + 255) & ~(size_t)255; };
  d->off_other = align((size_t)row_bytes * d->slab);
  d->off_parts = d->off_other + (g_bf16 ? 0 : align((size_t)rows * cols * 2));
  d->bytes = d->off_parts + (d->splits > 1 ? (size_t)d->splits * I * J * 4 : 0);
  return split_dot_pays(tokens, d->exact, I, J, C);
}

int split_dot_run(const SplitDotPlan& d, int tokens, const uint8_t* q, const uint8_t* sc8, const float* sc32, int64_t rows, int64_t cols, int a, int b,
                  const void* g, bool g_bf16, int64_t g_free, float* out, void* workspace, cudaStream_t st) {
  const int64_t I = tokens ? cols : rows, C = tokens ? rows : cols, J = g_free;
  unsigned char* ws = static_cast<unsigned char*>(workspace);
  __nv_bfloat16* terms_at = reinterpret_cast<__nv_bfloat16*>(ws);
  __nv_bfloat16* q_exact = reinterpret_cast<__nv_bfloat16*>(ws + d.off_other);
  float* parts = reinterpret_cast<float*>(ws + d.off_parts);
  const int64_t R = g_bf16 ? I : J, oc = g_bf16 ? J : I;      // rows of the terms, columns of the other operand
  for (int64_t r0 = 0; r0 < R; r0 += d.slab) {
    const int64_t tr = std::min(d.slab, R - r0);
    PrepareParams pp{};
    pp.q = q; pp.sc8 = sc8; pp.sc32 = sc32; pp.ldq = cols; pp.ldg = tokens ? J : C;
    pp.nbc = (uint32_t)d.nbc; pp.log2_a = (uint32_t)log2_of(a); pp.log2_b = (uint32_t)log2_of(b); pp.log2_K = (uint32_t)d.log2_K;
    pp.variants = d.variants;
    int64_t q_rows = rows, q_cols = cols;
    if (g_bf16) {                       // this round's i
      (tokens ? q_cols : q_rows) = tr;
      (tokens ? pp.q_col0 : pp.q_row0) = (uint32_t)r0;
      pp.q_out = terms_at; pp.q_plane = tr * C;
    } else {
      const int64_t g_rows = tokens ? C : tr, g_cols = tokens ? tr : C;
      pp.q_out = q_exact;
      pp.g = static_cast<const float*>(g) + (tokens ? r0 : r0 * C);
      pp.g_out = terms_at; pp.g_plane = tr * C;
      pp.g_vecs = FastDiv((uint32_t)(g_cols / 8)); pp.n_g = (uint32_t)(g_rows * g_cols / 8);
    }
    pp.q_vecs = FastDiv((uint32_t)(q_cols / 16));
    pp.n_q = g_bf16 || r0 == 0 ? (uint32_t)(q_rows * q_cols / 16) : 0u;      // the exact values serve all rounds
    pp.q_blocks = (pp.n_q + 255) / 256;
    if (int s = d.exact ? launch_prepare<false, false, 1>(pp, st) : g_bf16 ? launch_prepare<false, false, 3>(pp, st) : (tokens ? launch_prepare<true, true, 3>(pp, st) : launch_prepare<false, true, 3>(pp, st))) return s;

    CUtensorMap terms, other;
    const void* other_at = g_bf16 ? g : static_cast<const void*>(q_exact);
    const int64_t planes = (d.exact ? 1 : 3) * (int64_t)d.variants, plane = tr * C;
    const int deep = d.exact ? 2 * kDepth : kDepth;       // c per stage
    if (tokens) {
      if (int s = make_map(&terms, terms_at, tr, C, tr, planes, plane, 64, kDepth)) return s;
      if (int s = make_map(&other, other_at, oc, C, oc, 1, oc * C, 64, kDepth)) return s;
    } else {
      if (int s = make_map(&terms, terms_at, C, tr, C, planes, plane, deep, kTermRows)) return s;
      if (int s = make_map(&other, other_at, C, oc, C, 1, oc * C, deep, d.n)) return s;
    }
    SplitParams p{};
    p.src = DotSource{q, sc8, sc32, g, cols, tokens ? J : C, (uint32_t)d.nbc, (uint32_t)d.log2_K, (uint32_t)log2_of(a), (uint32_t)log2_of(b), (int)C};
    p.ld = tokens ? J : I;
    p.out = d.splits > 1 ? parts : out + (g_bf16 ? (tokens ? r0 * J : r0) : (tokens ? r0 : r0 * I));
    p.part = I * J;
    p.factor = sc32;
    p.rows = (int)tr; p.cols = (int)oc;
    p.row_first = (int)r0;
    p.row_tiles = (int)((tr + kTermRows - 1) / kTermRows);
    p.tiles = p.row_tiles * (int)((oc + d.n - 1) / d.n);
    p.splits = d.splits; p.units = d.units; p.units_per_split = d.units_per_split;
    p.cols_per_variant = (int)(I / d.variants);
    p.group = g_bf16 && !d.exact && C < kShortDepth ? 1 : kGroup;
    p.polls = kWaitPolls;
#ifdef PB_DIAGNOSTICS
    p.polls = g_split_polls.load(); p.withhold = g_split_withhold.load();
#endif
    const int status = d.exact ? launch_n<false, false, 1>(d.n, terms, other, p, st)
                     : tokens ? (g_bf16 ? launch_n<true, false, 3>(d.n, terms, other, p, st) : launch_n<true, true, 3>(d.n, terms, other, p, st))
                              : (g_bf16 ? launch_n<false, false, 3>(d.n, terms, other, p, st) : launch_n<false, true, 3>(d.n, terms, other, p, st));
    if (status) return status;
    if (d.splits > 1)         // there is one round then
      if (int s = add_parts(parts, out, I * J, d.splits, st)) return s;
  }
  return PB_OK;
}

// Reads and clears this file's device status word (see pb_gemm_check).
int split_dot_status_fetch(unsigned int* out) {
  const unsigned int zero = 0;
  PB_CUDA_TRY(cudaMemcpyFromSymbol(out, g_split_status, sizeof(*out)));
  if (*out != 0) PB_CUDA_TRY(cudaMemcpyToSymbol(g_split_status, &zero, sizeof(zero)));
  return PB_OK;
}

#ifdef PB_DIAGNOSTICS
void split_dot_control(uint32_t polls, int withhold) {
  g_split_polls.store(polls ? polls : kWaitPolls);
  g_split_withhold.store(withhold);
}
#endif
}  // namespace pb

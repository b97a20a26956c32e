// fp32 matrix products on the tensor cores: every operand is written as the sum of three bf16 pieces.
//
// A float has 24 significant bits, a bf16 has 8: x rounded to bf16, what is left rounded to bf16, and what is left then are three
// bf16 whose sum is x: exactly from 2^-110 on; below, the last piece is a multiple of 2^-133 and x is off by half of that at most (2^-19 of itself at
// 2^-115, 2^-9 at 2^-125).  Of the nine products of pieces the six that reach 2^-24 of the result are
// taken and accumulated in fp32 in TMEM, the small ones first, over one tile only (64 terms of the contraction for probabilities, D for
// scores): the tensor cores truncate where they accumulate, so the sums over tiles are made in registers, by rounded additions.  What the
// truncations take is not given back: on average it is 0.75e-7 of a sum of 64 products of mixed signs, but other data lose other shares, sums of
// few or of few bits none, and dP - delta makes much of little (operands of [0.5, 1.5], D = 128: dK 2.8e-7 off as it is, 15.5e-7 with that
// average added).  Relative error against 64 bits (2-norm), 4 x 8 heads x 500, and that of fp32 FMAs, 1e-7:
//                   D = 64: O, dQ, dK, dV                                D = 128
//   N(0, 1)           1.9 (3.5)  3.2 (3.8)  3.2 (4.5)  2.9 (4.3)           2.5 (4.7)  3.8 (4.2)  3.8 (5.6)  3.2 (5.4)
//   ... 3 Q, 3 K      3.8 (7.0)  11.3 (17)  11.3 (17)  10.5 (13.5)         5.6 (9.2)  18 (21)    18 (21)    16.1 (14.6)
//   [0.5, 1.5]        0.8 (1.7)  dQ is 0 but for errors  1.1 (2.2)  0.6 (1.8)      0.9 (3.3)             2.8 (4.9)  2.7 (4.5)
//   Q, K in -2 .. 2   1.6 (3.2)  4.8 (6.9)  4.7 (6.8)  4.6 (5.7)           1.5 (3.4)  8.3 (10.7) 8.3 (10.8) 8.1 (9.2)
// Six bf16 products at 1.63 PFLOP/s are 271 TFLOP/s of fp32, 3.7 times the FMA pipes' 74.
//
// Infinities: where a piece is zero its product with an infinite piece of the other operand would be NaN where x * inf is inf, and
// pieces of other signs than x would subtract infinities.  Kernels therefore walk their tiles again with the CAREFUL split once they
// have met a value that is not finite (or too large for a bf16): truncated pieces, which all have the sign of x, none of them zero
// (2^-40 of the value in its place, or the smallest bf16, 2^-133, where that is less) unless x is, and all infinite where x is.
#pragma once
#include "common.cuh"
#include "ptx.cuh"

namespace ttattn {
namespace pieces {

constexpr int kPieces = 3;
constexpr int kProducts = 6;
// the products taken, small ones first: piece of A and piece of B (0: leading), a nibble each
constexpr uint32_t kPieceA = 0x001012, kPieceB = 0x010210;
__host__ __device__ constexpr uint32_t piece_a(int p) { return kPieceA >> (4 * p) & 3; }
__host__ __device__ constexpr uint32_t piece_b(int p) { return kPieceB >> (4 * p) & 3; }
static_assert(piece_a(0) == 2 && piece_b(0) == 0 && piece_a(1) == 1 && piece_b(1) == 1 && piece_a(2) == 0 && piece_b(2) == 2 &&
                  piece_a(3) == 1 && piece_b(3) == 0 && piece_a(4) == 0 && piece_b(4) == 1 && piece_a(5) == 0 && piece_b(5) == 0,
              "every pair of pieces that reaches 2^-24, the small ones first");

// How the products of a tile are summed.  kOneSum: in one accumulator.  The others have a second one beside it, and an MMA whose second
// operand is the two first planes as one of twice the rows fills both.  kTwoSums: (l, h), (m, h), (h, h) in the first, the rest in the second.
// kLeadApart: (h, h) alone in the first.  Its truncations are those of a sum of the leading pieces alone then, none where these are few or
// fit 24 bits, and the same whichever operand comes first, in the forward and in the backward.  D = 64, for scores, dP and the forward's O.  Two MMAs of
// 64 columns in the place of one of 128: forward 18.1 -> 18.4 us (4 x 8 heads x 500), backward 58.8 -> 59.1; relative error of dV against 64 bits, scores of standard
// deviation 9, 18.6e-7 -> 13.0e-7 (fp32 FMAs 13.5e-7), of dK, operands of [0.5, 1.5], 2.8e-7 -> 1.1e-7 (2.2e-7; scores alone so, and dP not: 12.7e-7).  dV, dK and dQ
// are as exact with either.
enum Sums { kOneSum, kTwoSums, kLeadApart };
struct Step {
  uint32_t a, b;  // pieces
  bool second;    // into the second sum
  bool two;       // pieces b and b + 1, into both
  bool onto;      // what there is
};
__host__ __device__ constexpr int steps_of(Sums s) { return s == kOneSum ? kProducts : (s == kTwoSums ? 4 : 5); }
__host__ __device__ constexpr Step step_of(Sums s, int p) {
  return s == kOneSum    ? Step{piece_a(p), piece_b(p), false, false, p > 0}
         : s == kTwoSums ? Step{p == 0 ? 2u : (p == 2 ? 1u : 0u), p == 1 ? 2u : 0u, p == 1, p >= 2, p >= 2}
                         : Step{p == 1 ? 2u : (p >= 3 ? 1u : 0u), p == 2 ? 2u : (p == 4 ? 1u : 0u), p > 0, p == 0, p > 0};
}

__device__ __forceinline__ float lead(float x) { return __uint_as_float(__float_as_uint(x) & 0xffff0000u); }
__device__ __forceinline__ uint32_t pack_lead(float x0, float x1) {  // leading halves of two floats, x0 below
  return __byte_perm(__float_as_uint(x0), __float_as_uint(x1), 0x7632);
}
// The float that a piece of x is the lead of, where it must not be zero unless x is: `rest`, or 2^-40 of x, or the smallest bf16 there is.
__device__ __forceinline__ float never_zero(float rest, float x) {
  float least = fabsf(x) * 0x1p-40f;
  if (least < 0x1p-133f && x != 0.f) least = 0x1p-133f;
  return copysignf(fmaxf(fabsf(rest), least), x);  // (fmaxf(NaN, inf) = inf: inf - inf is not taken)
}

// the second pass: its code out of the way (the kernels' loops are long for the instruction caches)
__device__ __forceinline__ bool rare(bool careful) { return __builtin_expect(careful, 0); }

// Pieces of two neighbouring elements.  `odd` turns NaN where the first pieces are not both finite.
template <bool CAREFUL>
__device__ __forceinline__ void split2(float x0, float x1, uint32_t& h, uint32_t& m, uint32_t& l, float2& odd) {
  if constexpr (CAREFUL) {
    h = pack_lead(never_zero(x0, x0), never_zero(x1, x1));
    const float2 r = make_float2(x0 - lead(x0), x1 - lead(x1)), q = make_float2(r.x - lead(r.x), r.y - lead(r.y));
    m = pack_lead(never_zero(r.x, x0), never_zero(r.y, x1));
    l = pack_lead(never_zero(q.x, x0), never_zero(q.y, x1));
  } else {
    const float2 minus = make_float2(-1.f, -1.f);
    auto floats = [](uint32_t two) { return make_float2(__uint_as_float(two << 16), __uint_as_float(two & 0xffff0000u)); };
    h = pack2<true>(x0, x1);
    const float2 r = ptx::fma2(floats(h), minus, make_float2(x0, x1));
    m = pack2<true>(r.x, r.y);
    const float2 q = ptx::fma2(floats(m), minus, r);
    l = pack2<true>(q.x, q.y);
    odd = ptx::fma2(r, make_float2(0.f, 0.f), odd);
  }
}
// ... of probabilities, which are finite where the others are
template <bool CAREFUL>
__device__ __forceinline__ void split2(float x0, float x1, uint32_t& h, uint32_t& m, uint32_t& l) {
  float2 unused = make_float2(0.f, 0.f);
  split2<CAREFUL>(x0, x1, h, m, l, unused);
}

// Eight consecutive floats as 16 bytes of each piece, `plane` bytes apart, at shared-memory addresses; N times, side by side.
template <bool CAREFUL, int N>
__device__ __forceinline__ void store8(const uint32_t (&dst)[N], uint32_t plane, const float4 (&x)[N][2], float2& odd) {
  uint32_t p[N][kPieces][4];
#pragma unroll
  for (int i = 0; i < N; ++i)
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      split2<CAREFUL>(x[i][e].x, x[i][e].y, p[i][0][2 * e], p[i][1][2 * e], p[i][2][2 * e], odd);
      split2<CAREFUL>(x[i][e].z, x[i][e].w, p[i][0][2 * e + 1], p[i][1][2 * e + 1], p[i][2][2 * e + 1], odd);
    }
#pragma unroll
  for (int i = 0; i < N; ++i)
#pragma unroll
    for (int e = 0; e < kPieces; ++e)
      asm volatile("st.shared.v4.u32 [%0], {%1, %2, %3, %4};" ::"r"(dst[i] + e * plane), "r"(p[i][e][0]), "r"(p[i][e][1]), "r"(p[i][e][2]),
                   "r"(p[i][e][3])
                   : "memory");
}
__device__ __forceinline__ bool was_odd(const float2& odd) { return !(odd.x + odd.y == 0.f); }

// A tile of ROWS x D floats on its way from global memory into three planes of bf16 in shared memory, in the layout that both
// K-major and MN-major descriptors read: rows of 128 bytes with the 128-byte swizzle; the planes of 64 columns one after the other, so that
// two of them serve as one operand of twice the rows (K-major) or columns (MN-major), then those of the next 64.  NT threads
// take chunks of eight floats, neighbouring threads neighbouring chunks.
template <int ROWS, int D, int NT>
struct Tile {
  static constexpr int kPlane = ROWS * 128;
  static constexpr int kBlock = kPlane * kPieces;      // 64 columns
  static constexpr int kBytes = kBlock * (D / 64);
  static constexpr int kChunks = ROWS * (D / 8) / NT;  // of a thread
  static_assert(ROWS * (D / 8) % NT == 0 && NT % (D / 8) == 0, "chunks");

  static __device__ __forceinline__ int row(int tid, int i) { return tid / (D / 8) + i * (NT / (D / 8)); }
  static __device__ __forceinline__ int col(int tid) { return tid % (D / 8) * 8; }
  static __device__ __forceinline__ uint32_t at(int tid, int i) {  // of chunk i in the first plane
    const int r = row(tid, i), c = tid % (D / 8);
    return (c / 8) * kBlock + r * 128 + (((c % 8) ^ (r & 7)) << 4);
  }
  // chunks i .. i + N - 1
  template <int N>
  static __device__ __forceinline__ void put(uint32_t base, int tid, int i, const float4 (&x)[N][2], bool careful, float2& odd) {
    uint32_t dst[N];
#pragma unroll
    for (int e = 0; e < N; ++e) dst[e] = base + at(tid, i + e);
    if (rare(careful))
      store8<true, N>(dst, kPlane, x, odd);
    else
      store8<false, N>(dst, kPlane, x, odd);
  }
};

// Rows of a group's queries: query by query, the heads of the group together.
struct Group {
  int n;            // heads
  uint32_t magic;   // row / n is the upper word of row * magic; 0: by a division
  __device__ __forceinline__ Group(int heads, int rows)
      : n(heads), magic(heads > 1 && static_cast<uint64_t>(rows + 256u) * heads < (1ull << 32) ? 0xffffffffu / heads + 1 : 0) {}
  // (magic = (2^32 + e) / n with e < n: exact while row * e < 2^32)
  __device__ __forceinline__ int query(int row) const { return n == 1 ? row : (magic ? static_cast<int>(__umulhi(row, magic)) : row / n); }
  __device__ __forceinline__ int head(int row) const { return row - query(row) * n; }  // of the group
};

// A row's log-sum-exp in units of the exponents without an integer of 0 .. log2(n), n: how many keys the row may see; negated.  2 to minus that
// integer is the factor that the row's exponentials still want (x: the first, y: the second).  What a key of average probability has for an exponent is near 0 then, and so is its rounding, where it would be
// near -log2(n): relative error of dQ against 64 bits, 4 x 8 heads x 500, 3.8e-7 -> 3.2e-7 (D = 64; fp32 FMAs 3.8e-7), 4.4e-7 -> 3.8e-7 (D = 128; 4.2e-7).
__device__ __forceinline__ float2 exponent_base(float lse, int n) {
  const float x = lse * kLog2e, whole = fminf(fmaxf(rintf(x), 0.f), static_cast<float>(31 - __clz(max(n, 1))));
  // (a row without any participating key: P is 0)
  return make_float2(lse == -INFINITY ? -INFINITY : whole - x, __int_as_float((127 - static_cast<int>(whole)) << 23));
}

// Four bytes of a boolean mask, from byte `mis` of two words on, as bits: whether they are not zero.
__device__ __forceinline__ uint32_t mask_bits(uint32_t lo, uint32_t hi, int mis) {
  uint32_t v = __funnelshift_r(lo, hi, 8 * mis);
  v |= v >> 4, v |= v >> 2, v = (v | v >> 1) & 0x01010101u;
  return v * 0x01020408u >> 24 & 15;
}

// Every `step`-th of a group's rows (`rows` of them) from row r on, whose head is g and whose mask begins at `at`, `count` times and without a division for each:
// f(which of them, whether there is such a row, where its mask begins).
template <int UNROLL, typename F>
__device__ __forceinline__ void each_mask_row(const MaskArgs& m, int group, int rows, int r, int g, int64_t at, int step, int count, F f) {
  const int dg = step % group;
  const int64_t d = step / group * m.sl + dg * m.sh, wrap = m.sl - group * m.sh;
#pragma unroll UNROLL
  for (int e = 0; e < count; ++e) {
    f(e * step, r < rows, at);
    r += step, g += dg, at += d;
    if (g >= group) g -= group, at += wrap;
  }
}

// Two floats of a mask's row, 32 apart, global -> shared by asynchronous copies, where the key (a, b) takes part; zeros where there is no such row.  By predicates:
// as zero-filling copies (two selects more each) 2 x 8/4 heads x 99 on 131 keys took 11.7 us forward, by branches 12.5, so 11.0; 8 x 8 x 127 12.7, 14.0, 11.0.
__device__ __forceinline__ void copies4(uint32_t dst, const float* src, bool row, bool a, bool b) {
  asm volatile(
      "{\n.reg .pred p, q;\nsetp.ne.b32 p, %3, 0;\nsetp.ne.b32 q, %4, 0;\n"
      "@p cp.async.ca.shared.global [%0], [%1], 4, %2;\n@q cp.async.ca.shared.global [%0 + 128], [%1 + 128], 4, %2;\n}" ::"r"(dst),
      "l"(src), "r"(row ? 4 : 0), "r"(static_cast<int>(a)), "r"(static_cast<int>(b))
      : "memory");
}

__device__ __forceinline__ float4 load4_or_zero(const float* p, bool in) {
  float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
  if (in) v = __ldg(reinterpret_cast<const float4*>(p));
  return v;
}

}  // namespace pieces
}  // namespace ttattn

// FP64 contractions on the FP16 tensor cores.
//
// GB300 retires 1.7 FP64 FMAs per cycle and SM (measured: one warp instruction
// per 19 cycles and SM, per 64 cycles and sub-partition, whatever its active
// lanes), and 1026 FP16 multiply-adds per cycle and SM through mma.sync.  So an
// FP64 contraction is done on integer slices of its operands (Ozaki, Ogita,
// Oishi, Rump, Numer. Algorithms 59, 2012):
//
//   * A row of an operand (its elements along the contraction) is put on one
//     fixed-point scale: x = q 2^(er - 1084), er the largest exponent field of
//     the row, |q| <= 2^62: at most 2^-62 of the row's maximum off, so elements
//     down to 2^-9 of it keep all their bits.  Basis matrices are put on it once,
//     when the plan is made.
//   * q is written in 8 balanced base-256 digits, each in [-128, 127] (the top
//     one in [-65, 65]), which FP16 holds exactly.
//   * Products of digits u and v (0 = top) go to level u + v.  Levels 0..7 are
//     kept (36 digit products); what is dropped is about 2^-60 of the rows'
//     maxima.  A level's sum over K = 32 stays below 2^22 and is therefore exact
//     in the FP32 accumulator, which starts at 1.5 * 2^23, so that its bit
//     pattern is the integer.
//   * The levels are added up in 64-bit integers (hi: levels 0..3, lo: 4..7),
//     over any number of K = 32 blocks, and converted once, also in integers: no
//     FP64 instruction is left of a contraction.
//
// The result's error is that of the inputs on the row's scale and one final
// rounding; a chain of FP64 FMAs rounds K times.  (With 7 digits, 2^-54 of the
// maximum, rows that fall by orders of magnitude lost bits: meridional winds were
// up to 9 times further off the oracle than with FMAs.)  So the error is a part, K
// 2^-59 at most, of the product of the two rows' maxima, as an FFT's is of its row's,
// and not of each sum's own terms: rows that meet only where both are faint need more.
// The Legendre bases are levelled over the latitudes for that (spectral_f64.cu), the
// emission projection takes such sums again with FMAs (emission.cu).
// A row that holds an infinity or a NaN gives NaN, against a zero row too.  A row
// below 2^-959 counts as zero; rows whose maxima's product is below 2^-1006 give zero,
// beyond 2^1006 NaN.
#pragma once
#include <cuda_fp16.h>
#include <stdint.h>

namespace swp {
namespace slices {

constexpr int ND = 8;                       // digits
constexpr int NL = 8;                       // levels kept
constexpr uint64_t BIAS = 0x8080808080808080ull;  // 128 in each digit
constexpr float ACC0 = 12582912.0f;         // 1.5 * 2^23
constexpr int ACC0_BITS = 0x4B400000;
constexpr int ER_ZERO = -8000;              // row exponent of a zero row
constexpr int ER_BAD = 20000;               // of a row with an infinity or a NaN: NaN times a zero row too
constexpr int KFLUSH = 2;                   // mma k-steps (of 16) per flush of the accumulators

__device__ __forceinline__ int expo(double x) { return (__double2hiint(x) >> 20) & 0x7ff; }
// A row's exponent from the maximum of expo over it; a row below 2^-959 counts as zero.
__device__ __forceinline__ int row_exponent(int emax) { return emax >= 0x7ff ? ER_BAD : emax < 64 ? ER_ZERO : emax; }

// Biased fixed point of x on its row's scale, rounded: byte 7 - u is digit u plus
// 128.  Elements below half the scale's unit, and all of a zero or bad row, give 0.
__device__ __forceinline__ uint64_t fixed(double x, int er) {
  const uint32_t h = (uint32_t)__double2hiint(x), l = (uint32_t)__double2loint(x);
  const uint32_t sh = min((uint32_t)(er - (int)((h >> 20) & 0x7ff)), 63u);
  const uint32_t m1 = __funnelshift_l(l, (h & 0xfffffu) | 0x100000u, 10), m0 = l << 10;  // significand, one bit too many
  const uint32_t a1 = __funnelshift_rc(m1, 0u, sh), a0 = __funnelshift_rc(m0, m1, sh);
  const uint32_t b0 = __funnelshift_rc(m1, 0u, sh - 32u);
  const uint64_t q = ((sh < 32u ? ((uint64_t)a1 << 32) | a0 : (uint64_t)b0) + 1) >> 1;
  return (h >> 31) ? BIAS - q : BIAS + q;
}

// Digit u of two elements as an FP16 pair.
template <int U>
__device__ __forceinline__ uint32_t digit_pair(uint64_t a, uint64_t b) {
  constexpr int i = 7 - U;
  const uint32_t wa = i < 4 ? (uint32_t)a : (uint32_t)(a >> 32), wb = i < 4 ? (uint32_t)b : (uint32_t)(b >> 32);
  // bytes (a, any, b, any), then the upper byte of each half set to 0x64: 1024 + byte, exact in FP16
  const uint32_t p = __byte_perm(wa, wb, (uint32_t)((i & 3) | ((4 + (i & 3)) << 8)));
  const uint32_t h = (p & 0x00ff00ffu) | 0x64006400u;
  const __half2 v = __hsub2(*reinterpret_cast<const __half2*>(&h), __floats2half2_rn(1152.0f, 1152.0f));
  return *reinterpret_cast<const uint32_t*>(&v);
}
// Digits of two elements adjacent along K: out[u * stride], u = 0..7.
__device__ __forceinline__ void store_digits(uint32_t* out, int stride, uint64_t a, uint64_t b) {
  out[0] = digit_pair<0>(a, b);
  out[stride] = digit_pair<1>(a, b);
  out[2 * stride] = digit_pair<2>(a, b);
  out[3 * stride] = digit_pair<3>(a, b);
  out[4 * stride] = digit_pair<4>(a, b);
  out[5 * stride] = digit_pair<5>(a, b);
  out[6 * stride] = digit_pair<6>(a, b);
  out[7 * stride] = digit_pair<7>(a, b);
}

// Exchange between the lanes of a pair (l, l ^ 1): each lane holds elements of
// two rows at its own position; the even lane leaves with row a's pair, the odd
// lane with row b's.
__device__ __forceinline__ void pair_exchange(uint64_t& a, uint64_t& b) {
  const bool odd = threadIdx.x & 1;
  const uint64_t mine = odd ? b : a, give = odd ? a : b;
  const uint64_t got = __shfl_xor_sync(0xffffffffu, give, 1);
  a = odd ? got : mine;  // element at the even position
  b = odd ? mine : got;
}

__device__ __forceinline__ void mma(float (&d)[4], const uint32_t (&a)[4], const uint32_t (&b)[2]) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b[0]), "r"(b[1]));
}

// A 16 x 8 output tile of a warp.  Lane l holds rows l / 4 and l / 4 + 8,
// columns 2 (l % 4) and + 1: element 2 r + c is (row r, column c).
struct Tile {
  float acc[NL][4];
  long long hi[4], lo[4];

  __device__ __forceinline__ void reset() {
#pragma unroll
    for (int e = 0; e < 4; ++e) hi[e] = lo[e] = 0;
    restart();
  }
  __device__ __forceinline__ void restart() {
#pragma unroll
    for (int l = 0; l < NL; ++l)
#pragma unroll
      for (int e = 0; e < 4; ++e) acc[l][e] = ACC0;
  }
  // one k-step: a[u] the A fragment of digit u, b[v] the B fragment of digit v
  __device__ __forceinline__ void step(const uint32_t (&a)[ND][4], const uint32_t (&b)[ND][2]) {
#pragma unroll
    for (int u = 0; u < ND; ++u)
#pragma unroll
      for (int v = 0; v < ND; ++v)
        if (u + v < NL) mma(acc[u + v], a[u], b[v]);
  }
  // add the accumulated levels (at most KFLUSH k-steps) to the integer sums
  __device__ __forceinline__ void flush() {
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      int i[NL];
#pragma unroll
      for (int l = 0; l < NL; ++l) i[l] = __float_as_int(acc[l][e]) - ACC0_BITS;
      hi[e] += (long long)(i[0] * 256 + i[1]) * 65536 + (i[2] * 256 + i[3]);
      lo[e] += (long long)(i[4] * 256 + i[5]) * 65536 + (i[6] * 256 + i[7]);
    }
    restart();
  }
};

// The FP64 value of integer sums over at most 2^14 elements on the scales of an
// A row and a B row: (hi 2^32 + lo) 2^(era + erb - 2112), rounded to nearest.  In
// integers: about 35 instructions, where the three FP64 additions of two
// magic-number conversions would cost the SM 57 cycles a warp against 9.
__device__ __forceinline__ double value(long long hi, long long lo, int era, int erb) {
  const int s = era + erb;
  hi += lo >> 32;  // a unit of hi is 2^32 units of lo
  // magnitude as three words, most significant first
  const uint32_t neg = (uint32_t)(hi >> 63);
  uint32_t w0 = (uint32_t)lo ^ neg;
  uint64_t h = (uint64_t)hi ^ (((uint64_t)neg << 32) | neg);
  w0 += neg & 1u;
  h += (neg && w0 == 0) ? 1u : 0u;
  uint32_t w2 = (uint32_t)(h >> 32), w1 = (uint32_t)h;
  // normalise: leading one to bit 31 of w2
  int p = s - 1089 + 95;
  if (w2 == 0) {
    w2 = w1;
    w1 = w0;
    w0 = 0;
    p -= 32;
  }
  if (w2 == 0) {
    w2 = w1;
    w1 = 0;
    p -= 32;
  }
  const int z = __clz(w2);
  const uint32_t a2 = __funnelshift_lc(w1, w2, z), a1 = __funnelshift_lc(w0, w1, z);
  p -= z;
  // 53 significant bits, rounded; the leading one adds 1 to the exponent field
  uint64_t m = (((uint64_t)a2 << 32) | a1) >> 11;
  m += (a1 >> 10) & 1u;
  const uint64_t bits = ((uint64_t)(uint32_t)(p - 1) << 52) + m;
  const bool zero = p < 1 || w2 == 0 || s < 1038;  // zero sum or row, or below 2^-1000
  const uint64_t r = s > 3051 ? 0x7ff8000000000000ull : zero ? 0ull : bits | ((uint64_t)neg << 63);
  return __longlong_as_double((long long)r);
}

// The B fragment of one k-step from digit planes in shared memory (words of two
// elements): p0 and p1 point at this lane's words of digit 0, k = 2 t and 2 t + 8
// of its column's row.
__device__ __forceinline__ void load_b(uint32_t (&b)[ND][2], const uint32_t* p0, const uint32_t* p1, int plane) {
#pragma unroll
  for (int v = 0; v < ND; ++v) {
    b[v][0] = p0[v * plane];
    b[v][1] = p1[v * plane];
  }
}
// Bring a packed static operand (bytes, 128-byte lines) towards the SM while the
// data that it multiplies are still being formed.
__device__ __forceinline__ void prefetch_lines(const void* p, int bytes) {
  for (int o = threadIdx.x * 128; o < bytes; o += blockDim.x * 128)
    asm volatile("prefetch.global.L1 [%0];" ::"l"((const char*)p + o));
}
// The A fragment of one k-step from a packed static operand (pack_a):
// [k-step][digit][lane] of 16 bytes.
__device__ __forceinline__ void load_a(uint32_t (&a)[ND][4], const uint4* __restrict__ p) {
#pragma unroll
  for (int u = 0; u < ND; ++u) {
    const uint4 w = __ldg(p + u * 32);
    a[u][0] = w.x;
    a[u][1] = w.y;
    a[u][2] = w.z;
    a[u][3] = w.w;
  }
}

}  // namespace slices
}  // namespace swp

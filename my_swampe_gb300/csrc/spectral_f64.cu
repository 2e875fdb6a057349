// The FP64 Legendre sandwich of a step and its adjoint on the FP16 tensor cores
// (slices.cuh).  The chain per zonal wavenumber m is k_spectral's (spectral.cu):
// combined inputs, forward Legendre, spectral epilogue, inverse Legendre,
// write-out; here both contractions run on integer slices of their operands.
//
// What bounds it: on the FMA kernel the contractions were two thirds of the FP64
// instructions and ran at the FP64 pipe's rate (0.88 ms a step at M = 42, B = 256;
// 98 us for one member, whose contraction filled one warp of one sub-partition).
// Left on the FP64 pipe now are the pointwise parts.  One unit is one m and MT members; 8 warps:
//
//   1. a thread per (member, latitude) forms the combined inputs (FP64) into
//      shared memory, rows (slot, member component) x J latitudes;
//   2. a warp per row finds its scale and slices its equatorially symmetric and
//      antisymmetric parts (lanes over latitudes);
//   3. warps take 16 x 8 output tiles (degrees x rows) over J/2 latitudes, the
//      basis slices coming from global memory in fragment order (packed once
//      per plan, L2 resident), and convert them to FP64;
//   4. a thread per (member, degree) applies the spectral epilogue;
//   5. a warp per row slices the spectra, 6. warps take tiles (latitudes x rows),
//      even and odd degrees added and subtracted in integers: north and south;
//   7. a thread per (member, latitude) writes the point out.
//
// No result depends on MT: sums are exact, scales are per row.
#include <algorithm>
#include "slices.cuh"
#include "swp_internal.h"
#include "spec_common.cuh"

namespace swp {
namespace {

using namespace slices;

// Tile counts of a truncation.
template <int M_>
struct Sh {
  static constexpr int J = trunc_J(M_), Jh = J / 2, CNT = M_ + 1;
  static constexpr int C0 = (CNT + 1) / 2;           // degrees of the even parity at m = 0
  static constexpr int MTF = (C0 + 15) / 16;         // degree tiles of a parity
  static constexpr int KSF = Jh / 16;                // k-steps over latitudes
  static constexpr int LT = Jh / 16;                 // latitude tiles
  static constexpr int KSI = MTF;                    // k-steps over degrees
  static constexpr int PC = 16 * KSI;                // degrees of a parity, padded
  // Words of a sliced latitude row.  The 8 columns g of a B fragment are rows of
  // one symmetry of 8 consecutive n: padded so that they start on different
  // banks, or, at J / 2 = 32 (where the padding would cost the second CTA per
  // SM), swizzled: bits 2, 3 of the word with n mod 4, the two symmetries of a
  // row in the order of bit 2 of n.
  static constexpr bool SWZ = Jh == 32;
  static constexpr int XW = SWZ ? 16 : Jh / 2 + 2;
  __device__ static __forceinline__ int xrow(int n, int sym) { return (2 * n + (SWZ ? sym ^ ((n >> 2) & 1) : sym)) * XW; }
  __device__ static __forceinline__ int xword(int n, int w) { return SWZ ? w ^ ((n & 3) << 2) : w; }
  static constexpr int KW = PC + 4;                  // words of a sliced spectral row, both parities (padded)
  static_assert(Jh % 16 == 0 && J % 32 == 0, "latitude tiles");
};

// Packed basis of one plan group: per m, for the contraction over latitudes
// (F) [P, H][parity][degree tile][k-step][digit][lane] and over degrees (I)
// [P, H][parity][latitude tile][k-step][digit][lane], 16 bytes each, and the
// rows' exponents: F [P, H][parity][PC], I [P, H][Jh] (common to both parities,
// whose sums are added in integers).  Last, for the contraction over latitudes,
// the powers of two EP [Jh] (exponents, at most 0) that the data are multiplied
// and the basis divided by: the basis falls towards the poles as cos^m, where
// the data rise (their factor 1 / (1 - mu^2)); with the basis level over the
// latitudes the data's scale follows what enters the sums.  (Without them the
// explicit scheme's winds were 1.5e-9 off the oracle, with them as before.)
template <class S>
struct Pack {
  static constexpr size_t F = (size_t)2 * 2 * S::MTF * S::KSF * ND * 32;  // uint4 per m
  static constexpr size_t I = (size_t)2 * 2 * S::LT * S::KSI * ND * 32;
  static constexpr size_t EF = 2 * 2 * S::PC, EI = 2 * S::Jh, EP = S::Jh;  // ints per m
  static constexpr size_t bytes = (size_t)S::CNT * ((F + I) * 16 + (EF + EI + EP) * 4);
};
template <class S>
struct PackView {
  const uint4 *f, *i;
  const int *ef, *ei, *ep;
  __device__ PackView(const void* base, int m) {
    const uint4* p = (const uint4*)base;
    f = p + (size_t)m * Pack<S>::F;
    i = p + (size_t)S::CNT * Pack<S>::F + (size_t)m * Pack<S>::I;
    const int* e = (const int*)(p + (size_t)S::CNT * (Pack<S>::F + Pack<S>::I));
    ef = e + (size_t)m * Pack<S>::EF;
    ei = e + (size_t)S::CNT * Pack<S>::EF + (size_t)m * Pack<S>::EI;
    ep = e + (size_t)S::CNT * (Pack<S>::EF + Pack<S>::EI) + (size_t)m * Pack<S>::EP;
  }
};

// One CTA per m.  fp, fh: the forward-layout bases [parity][j'][c] of the
// latitude contraction; ip, ih: those of the degree contraction (same layout).
template <class S>
__global__ void k_pack_slices(const double* fp, const double* fh, const double* ip, const double* ih, const int* boff,
                              void* out) {
  const int m = blockIdx.x, cnt = S::CNT - m, C0 = (cnt + 1) / 2, C1 = cnt / 2;
  const PackView<S> v(out, m);
  int* ef = const_cast<int*>(v.ef);
  int* ei = const_cast<int*>(v.ei);
  int* ep = const_cast<int*>(v.ep);
  __shared__ int top;
  if (threadIdx.x == 0) top = 0;
  __syncthreads();
  auto elem = [&](const double* P, const double* H, int mat, int par, int c, int j) {
    const int Cp = par ? C1 : C0;
    return c < Cp ? (mat ? H : P)[boff[m] + (par ? S::Jh * C0 : 0) + j * Cp + c] : 0.0;
  };
  // the basis' largest exponent at each latitude (P; H follows it), relative to the largest of all
  for (int j = threadIdx.x; j < S::Jh; j += blockDim.x) {
    int e = 0;
    for (int par = 0; par < 2; ++par)
      for (int c = 0; c < (par ? C1 : C0); ++c) e = max(e, expo(elem(fp, fh, 0, par, c, j)));
    ep[j] = e;
    atomicMax(&top, e);
  }
  __syncthreads();
  for (int j = threadIdx.x; j < S::Jh; j += blockDim.x) ep[j] -= top;
  __syncthreads();
  for (int t = threadIdx.x; t < (int)(Pack<S>::EF + Pack<S>::EI); t += blockDim.x) {
    int e = 0;
    if (t < (int)Pack<S>::EF) {
      const int c = t % S::PC, par = (t / S::PC) & 1, mat = t / (2 * S::PC);
      for (int j = 0; j < S::Jh; ++j) e = max(e, expo(elem(fp, fh, mat, par, c, j)) - ep[j]);
      ef[t] = row_exponent(e);
    } else {
      const int u = t - (int)Pack<S>::EF, j = u % S::Jh, mat = u / S::Jh;
      for (int par = 0; par < 2; ++par)
        for (int c = 0; c < (par ? C1 : C0); ++c) e = max(e, expo(elem(ip, ih, mat, par, c, j)));
      ei[u] = row_exponent(e);
    }
  }
  __syncthreads();
  // a thread per (tile, k-step, lane): fragment register q holds (row g + 8 (q & 1), k 2 t + 8 (q >> 1) and + 1)
  for (int inv = 0; inv < 2; ++inv) {
    const int ntile = 2 * 2 * (inv ? S::LT : S::MTF), ks = inv ? S::KSI : S::KSF;
    for (int u = threadIdx.x; u < ntile * ks * 32; u += blockDim.x) {
      const int lane = u & 31, k0 = 16 * ((u / 32) % ks), tile = u / (32 * ks);
      const int nt = inv ? S::LT : S::MTF, r0 = 16 * (tile % nt), par = (tile / nt) & 1, mat = tile / (2 * nt);
      uint32_t w[4][ND];
      for (int q = 0; q < 4; ++q) {
        const int row = r0 + (lane >> 2) + 8 * (q & 1), k = k0 + 2 * (lane & 3) + 8 * (q >> 1);
        const double a = inv ? elem(ip, ih, mat, par, k, row) : elem(fp, fh, mat, par, row, k);
        const double b = inv ? elem(ip, ih, mat, par, k + 1, row) : elem(fp, fh, mat, par, row, k + 1);
        const int e = inv ? ei[mat * S::Jh + row] : ef[(mat * 2 + par) * S::PC + row];
        store_digits(w[q], 1, fixed(a, e + (inv ? 0 : ep[k])), fixed(b, e + (inv ? 0 : ep[k + 1])));
      }
      uint4* dst = const_cast<uint4*>(inv ? v.i : v.f) + (size_t)(u / 32) * ND * 32 + lane;
      for (int d = 0; d < ND; ++d) dst[d * 32] = make_uint4(w[0][d], w[1][d], w[2][d], w[3][d]);
    }
  }
}

// Shared memory of a unit.  Two regions, each used in turn:
//   A: raw rows [NIN R][J]  ->  spectra [NF R][CNT]  ->  inverse inputs [NK R][2 PC]  ->  outputs [NO R][J]
//   B: latitude slices [ND][NIN R][2][XW]  ->  spectral slices [ND][NK R][KW]
// NIN raw rows, NF forward outputs, NK inverse inputs, NO inverse outputs per
// member component.
template <class S, int MT, int NIN, int NF, int NK, int NO>
struct Mem {
  static constexpr int R = 2 * MT;
  static constexpr size_t raw = (size_t)NIN * R * S::J, spec = (size_t)NF * R * S::CNT;
  static constexpr size_t kin = (size_t)NK * R * 2 * S::PC, out = (size_t)NO * R * S::J;
  static constexpr size_t cmax(size_t a, size_t b) { return a > b ? a : b; }
  static constexpr size_t A = cmax(cmax(raw, spec), cmax(kin, out)) * 8;
  static constexpr size_t B = cmax((size_t)ND * NIN * R * 2 * S::XW, (size_t)ND * NK * R * S::KW) * 4;
  static constexpr size_t E = (size_t)(NIN * R + NK * R) * 4;
  static constexpr size_t total = A + B + E;
};

// Symmetric (s = 0) and antisymmetric (s = 1) parts of the raw rows over the
// southern latitudes j' (plus / minus their mirror), times 2^ep[j'], sliced.  Both
// are formed in integers, on the scale of the row's largest element with one bit of
// headroom.
__device__ __forceinline__ int expo_scaled(double x, int ep) {
  const int e = expo(x);
  return e == 0x7ff ? ER_BAD : max(e + ep, 0);
}
template <class S>
__device__ __forceinline__ void slice_latitudes(const double* raw, int rows, const int* ep, uint32_t* dig, int plane,
                                                int* er) {
  constexpr int KI = (S::Jh + 31) / 32;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  int p[KI];
#pragma unroll
  for (int i = 0; i < KI; ++i) p[i] = S::Jh % 32 == 0 || lane + 32 * i < S::Jh ? __ldg(ep + lane + 32 * i) : 0;
  for (int r = warp; r < rows; r += 8) {
    const double* x = raw + (size_t)r * S::J;
    double xn[KI], xs[KI];
    int e = 0;
#pragma unroll
    for (int i = 0; i < KI; ++i) {
      const int k = lane + 32 * i;
      const bool on = S::Jh % 32 == 0 || k < S::Jh;
      xn[i] = on ? x[k] : 0.0;
      xs[i] = on ? x[S::J - 1 - k] : 0.0;
      e = max(e, max(expo_scaled(xn[i], p[i]), expo_scaled(xs[i], p[i])));
    }
    e = (int)__reduce_max_sync(0xffffffffu, (unsigned)e);
    e = row_exponent(e >= 0x7ff ? e : e + 1);
    if (lane == 0) er[r] = e;
#pragma unroll
    for (int i = 0; i < KI; ++i) {
      const uint64_t fn = fixed(xn[i], e - p[i]), fs = fixed(xs[i], e - p[i]);
      uint64_t a = fn + fs - BIAS, b = fn - fs + BIAS;
      pair_exchange(a, b);
      if (S::Jh % 32 == 0 || lane + 32 * i < S::Jh)
        store_digits(dig + S::xrow(r, lane & 1) + S::xword(r, (lane >> 1) + 16 * i), plane, a, b);
    }
  }
}

// Forward contraction: tiles of 16 degrees x 8 rows.  P outputs are rows 0 ..
// nP - 1 of the raw rows, read with the parity's own symmetry; H outputs are raw
// rows h0 .. h0 + nH - 1 with the other one.  out: [nP + nH][CNT].
template <class S>
__device__ __forceinline__ void contract_latitudes(const PackView<S>& pk, int C0, int C1, const uint32_t* dig,
                                                   int plane, const int* er, int nP, int h0, int nH, double* out) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  const int tP = (nP + 7) / 8, NT = tP + (nH + 7) / 8;
  const int m0 = (C0 + 15) / 16, m1 = (C1 + 15) / 16;
  for (int job = warp; job < (m0 + m1) * NT; job += 8) {
    const int nt = job % NT, mj = job / NT;
    const int par = mj >= m0, mt = par ? mj - m0 : mj, mat = nt >= tP;
    const int n0 = 8 * (mat ? nt - tP : nt), nrow = mat ? nH : nP, rbase = mat ? h0 : 0;
    const int sym = par ^ mat;
    const uint4* a = pk.f + (size_t)(((mat * 2 + par) * S::MTF + mt) * S::KSF) * ND * 32 + lane;
    const int bn = rbase + min(n0 + g, nrow - 1);
    const uint32_t* b = dig + S::xrow(bn, sym);
    Tile tile;
    tile.reset();
#pragma unroll
    for (int ks = 0; ks < S::KSF; ++ks) {
      uint32_t af[ND][4], bf[ND][2];
      load_a(af, a + (size_t)ks * ND * 32);
      load_b(bf, b + S::xword(bn, 8 * ks + t), b + S::xword(bn, 8 * ks + 4 + t), plane);
      tile.step(af, bf);
      if (ks % KFLUSH == KFLUSH - 1 || ks == S::KSF - 1) tile.flush();
    }
    const int Cp = par ? C1 : C0;
    const int* ef = pk.ef + (mat * 2 + par) * S::PC + 16 * mt;
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const int c = 16 * mt + g + 8 * (e >> 1), n = n0 + 2 * t + (e & 1);
      if (c < Cp && n < nrow)
        out[(size_t)((mat ? nP : 0) + n) * S::CNT + (par ? C0 + c : c)] =
            value(tile.hi[e], tile.lo[e], ef[g + 8 * (e >> 1)], er[rbase + n]);
    }
  }
}

// Slices of the inverse inputs: row r holds degrees [parity][PC], zero beyond
// the parity's count, on one scale for both parities.
template <class S>
__device__ __forceinline__ void slice_degrees(const double* kin, int rows, int C0, int C1, uint32_t* dig, int plane,
                                              int* er) {
  constexpr int KI = (S::PC + 31) / 32;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  for (int r = warp; r < rows; r += 8) {
    const double* x = kin + (size_t)r * 2 * S::PC;
    double x0[KI], x1[KI];
    int e = 0;
#pragma unroll
    for (int i = 0; i < KI; ++i) {
      const int c = lane + 32 * i;
      x0[i] = c < C0 ? x[c] : 0.0;
      x1[i] = c < C1 ? x[S::PC + c] : 0.0;
      e = max(e, max(expo(x0[i]), expo(x1[i])));
    }
    e = row_exponent((int)__reduce_max_sync(0xffffffffu, (unsigned)e));
    if (lane == 0) er[r] = e;
#pragma unroll
    for (int i = 0; i < KI; ++i) {
      uint64_t a = fixed(x0[i], e), b = fixed(x1[i], e);
      pair_exchange(a, b);
      store_digits(dig + (size_t)r * S::KW + (lane & 1) * (S::PC / 2) + (lane >> 1) + 16 * i, plane, a, b);
    }
  }
}

// Inverse contraction: tiles of 16 latitudes x 8 rows.  P outputs are rows 0 ..
// nP - 1; H outputs take rows hrow(0 .. nH - 1) and change sign in the south.
// out: [nP + nH][J].
template <class S, typename HR>
__device__ __forceinline__ void contract_degrees(const PackView<S>& pk, int C0, int C1, const uint32_t* dig,
                                                 int plane, const int* er, int nP, int nH, HR hrow, double* out) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  const int tP = (nP + 7) / 8, NT = tP + (nH + 7) / 8;
  for (int job = warp; job < S::LT * NT; job += 8) {
    const int nt = job % NT, lt = job / NT, mat = nt >= tP;
    const int n0 = 8 * (mat ? nt - tP : nt), nrow = mat ? nH : nP;
    const int bn = min(n0 + g, nrow - 1);
    const uint32_t* b = dig + (size_t)(mat ? hrow(bn) : bn) * S::KW + t;
    long long eh[4], el[4];
    Tile tile;
#pragma unroll
    for (int par = 0; par < 2; ++par) {
      const uint4* a = pk.i + (size_t)(((mat * 2 + par) * S::LT + lt) * S::KSI) * ND * 32 + lane;
      const int nk = ((par ? C1 : C0) + 15) / 16;
      tile.reset();
#pragma unroll
      for (int ks = 0; ks < S::KSI; ++ks) {
        if (ks >= nk) break;
        uint32_t af[ND][4], bf[ND][2];
        load_a(af, a + (size_t)ks * ND * 32);
        load_b(bf, b + par * (S::PC / 2) + 8 * ks, b + par * (S::PC / 2) + 8 * ks + 4, plane);
        tile.step(af, bf);
        if (ks % KFLUSH == KFLUSH - 1 || ks == nk - 1) tile.flush();
      }
      if (par == 0) {
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          eh[e] = tile.hi[e];
          el[e] = tile.lo[e];
        }
      }
    }
    const int* ei = pk.ei + mat * S::Jh + 16 * lt;
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const int j = 16 * lt + g + 8 * (e >> 1), n = n0 + 2 * t + (e & 1);
      if (n >= nrow) continue;
      const int sa = ei[g + 8 * (e >> 1)], sb = er[mat ? hrow(n) : n];
      double* o = out + (size_t)((mat ? nP : 0) + n) * S::J;
      o[j] = value(eh[e] + tile.hi[e], el[e] + tile.lo[e], sa, sb);
      // south: even minus odd degrees for P, the negative of it for H
      o[S::J - 1 - j] = mat ? value(tile.hi[e] - eh[e], tile.lo[e] - el[e], sa, sb)
                            : value(eh[e] - tile.hi[e], el[e] - tile.lo[e], sa, sb);
    }
  }
}

constexpr int NIN = NSP + NSH;  // combined inputs of a step: 5 on Pw, 4 on Hw

// --------------------------------------------------------------------- step
template <int M_, int MT>
__global__ void __launch_bounds__(256, 2) k_spectral_f64(const __grid_constant__ SpecLaunch<double> L,
                                                         const __grid_constant__ SliceBasis basis) {
  typedef Sh<M_> S;
  typedef Mem<S, MT, NIN, NIN, 7, 7> Mm;
  constexpr int R = 2 * MT, J = S::J;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  double* A = (double*)smem_raw;
  uint32_t* D = (uint32_t*)(smem_raw + Mm::A);
  int* erx = (int*)(smem_raw + Mm::A + Mm::B);  // [NIN R]
  int* erk = erx + NIN * R;                     // [7 R]
  __shared__ int sdead[MT];
  int idx;
  const SpecGroup<double>& G = pick_group(L, idx);
  const StepCfg& cfg = L.cfg;
  const int m = idx / G.ntb, b0 = (idx % G.ntb) * MT, mt = min(MT, G.B - b0);
  const int cnt = S::CNT - m, C0 = (cnt + 1) / 2, C1 = cnt / 2;
  const size_t FS = (size_t)S::CNT * G.B * J;
  const PackView<S> pk(basis.p[&G - L.grp], m);
  if (MT == 1) {  // few units: their basis is not in L1 yet
    prefetch_lines(pk.f, (int)(Pack<S>::F * 16));
    prefetch_lines(pk.i, (int)(Pack<S>::I * 16));
  }

  // blow-up gate (model.py:838-864)
  if (threadIdx.x < MT) {
    const int bt = threadIdx.x;
    int dead = 0;
    if (bt < mt && cfg.diagnostics) {
      const int b = b0 + bt;
      const double ms = G.diag[((size_t)cfg.step * NDIAG + D_RMS2) * G.B + b];
      dead = (G.member[MS_DEAD * G.B + b] != 0.0) || blown_up(cfg, ms);
      if (m == 0) {
        G.member[MS_DEAD * G.B + b] = dead ? 1.0 : 0.0;
        G.diag[((size_t)cfg.step * NDIAG + D_DEAD) * G.B + b] = dead ? 1.0 : 0.0;
      }
    }
    sdead[bt] = dead;
  }
  // 1. combined inputs.  One member: two threads per latitude, real and imaginary
  // parts (each form drops the other's arithmetic), since two warps alone would use
  // half of the SM's FP64 sub-partitions
  for (int t = threadIdx.x; t < (MT == 1 ? 2 : MT) * J; t += 256) {
    const int bt = MT == 1 ? 0 : t / J, j = t % J;
    auto combos = [&](double2* c) {
      if (bt < mt) {
        step_combos<double>(G, cfg, 0, false, m, b0 + bt, j, FS, c);
      } else {
#pragma unroll
        for (int q = 0; q < NIN; ++q) c[q] = make_double2(0.0, 0.0);
      }
    };
    double2 c[NIN];
    if (MT == 1 && t >= J) {
      combos(c);
#pragma unroll
      for (int q = 0; q < NIN; ++q) A[(size_t)(q * R + 1) * J + j] = c[q].y;
    } else if (MT == 1) {
      combos(c);
#pragma unroll
      for (int q = 0; q < NIN; ++q) A[(size_t)(q * R) * J + j] = c[q].x;
    } else {
      combos(c);
#pragma unroll
      for (int q = 0; q < NIN; ++q) {
        A[(size_t)(q * R + 2 * bt) * J + j] = c[q].x;
        A[(size_t)(q * R + 2 * bt + 1) * J + j] = c[q].y;
      }
    }
  }
  __syncthreads();
  // 2., 3. forward Legendre
  constexpr int planeX = NIN * R * 2 * S::XW, planeK = 7 * R * S::KW;
  slice_latitudes<S>(A, NIN * R, pk.ep, D, planeX, erx);
  __syncthreads();
  contract_latitudes<S>(pk, C0, C1, D, planeX, erx, NSP * R, NSP * R, NSH * R, A);
  __syncthreads();
  // 4. spectral epilogue: a thread per (member, degree) and, where the CTA has the
  // threads, component
  constexpr int NC = 2 * MT * S::CNT <= 256 ? 1 : 2;  // components per thread
  static_assert(MT * S::CNT <= 256, "one spectral point per thread");
  {
    const int comp0 = NC == 1 ? (int)threadIdx.x / (MT * cnt) : 0, t = (int)threadIdx.x - comp0 * MT * cnt;
    const int bt = t / cnt, kk = t % cnt;
    const bool on = comp0 < 2 && bt < mt;
    const int par = kk & 1, c = kk >> 1, pc = par ? C0 + c : c, n = m + kk, b = b0 + bt;
    double e[NC], d[NC], p[NC];  // new spectral eta, delta, Phi
    double tc = 0.0, om = 0.0;
    if (on) {
      const size_t qs = (size_t)G.B * S::CNT, qo = (size_t)b * S::CNT + n;
      const bool expo_sig = cfg.scheme == 2;
      const double s = cfg.diffflag ? G.nco[(expo_sig ? NC_SIGX : NC_SIG) * qs + qo] : 1.0;
      const double sp = cfg.diffflag ? G.nco[(expo_sig ? NC_SIGPX : NC_SIGP) * qs + qo] : 1.0;
      tc = G.nco[NC_TC * qs + qo];
      const double nn1 = (double)(n * (n + 1));
      const double* mc = G.mco;
      om = (m == 0 && n == 1) ? mc[MC_OM * G.B + b] : 0.0;
      // semi-implicit solve (semi_implicit_tdiff.py): shares and rates as in k_spectral
      double xi = 0.0, kd = 0.0, kr = 0.0, gd = 0.0, bq = 0.0, cq = 0.0, ikr = 1.0, ed = 1.0, Dn = 1.0;
      if (cfg.scheme == 2) {
        xi = mc[MC_SIXI * G.B + b];
        if (cfg.si_relax) {
          const double itd = mc[MC_SIITD * G.B + b];
          kd = xi * itd;
          kr = xi * mc[MC_SIITR * G.B + b];
          gd = mc[MC_SIEX * G.B + b] * itd;
        }
        bq = xi * (nn1 * mc[MC_IA2 * G.B + b]);
        cq = xi * mc[MC_PB * G.B + b];
        ikr = 1.0 / (1.0 + kr);
        ed = 1.0 + kd;
        Dn = (1.0 + kd) + bq * cq * ikr;
      }
#pragma unroll
      for (int k = 0; k < NC; ++k) {
        const int comp = comp0 + k;
        auto a = [&](int q) { return A[(size_t)(q * R + 2 * bt + comp) * S::CNT + pc]; };
        const double sphi = a(SP_PHI1) + a(NSP + SH_PHI1), seta = a(SP_E1) + a(NSP + SH_E1);
        if (cfg.scheme == 2) {
          const double sdel = a(SP_D1) + a(NSP + SH_D1) + nn1 * a(SP_D2);
          const double se = comp == 0 ? seta + (gd * om + kd * om) : seta;
          const double dn = (sdel + bq * sphi * ikr) / Dn;
          p[k] = sp * ((sphi - cq * dn) * ikr);
          d[k] = s * dn;
          e[k] = s * (se / ed);
        } else {
          p[k] = sp * (sphi + nn1 * a(SP_PHI2));
          d[k] = s * (a(SP_D1) + a(NSP + SH_D1) + nn1 * (a(SP_D2) + a(NSP + SH_D2)));
          e[k] = s * seta;
        }
      }
      if (n == 0) tc = 0.0;
    }
    __syncthreads();  // the spectra are read: their place takes the inverse inputs
    if (on) {
      constexpr size_t RS = 2 * S::PC, QS = (size_t)R * 2 * S::PC;
      const double xm = (double)m;
#pragma unroll
      for (int k = 0; k < NC; ++k) {
        const int comp = comp0 + k;
        double* K = A + (size_t)(2 * bt + comp) * RS + par * S::PC + c;
        // planetary vorticity: a real constant of the wind inversion
        const double es = (comp == 0 ? e[k] - om : e[k]) * tc, ds = d[k] * tc;
        K[0] = e[k];
        K[QS] = d[k];
        K[2 * QS] = p[k];
        // wind inversion inputs (spectral_transform.py:577-594): on P -i m delta_s,
        // -i m eta_s (into the other component's row); on H eta_s, -delta_s
        double* Ko = comp == 0 ? K + RS : K - RS;
        const double xs = comp == 0 ? -xm : xm;
        Ko[3 * QS] = xs * ds;
        Ko[4 * QS] = xs * es;
        K[5 * QS] = es;
        K[6 * QS] = -ds;
      }
    }
    // rows of absent members of the last tile
    for (int i = threadIdx.x; i < 7 * (R - 2 * mt) * 2 * S::PC; i += 256) {
      const int k = i % (2 * S::PC), r = 2 * mt + (i / (2 * S::PC)) % (R - 2 * mt), q = i / (2 * S::PC * (R - 2 * mt));
      A[(size_t)(q * R + r) * 2 * S::PC + k] = 0.0;
    }
  }
  __syncthreads();
  // 5., 6. inverse Legendre
  slice_degrees<S>(A, 7 * R, C0, C1, D, planeK, erk);
  __syncthreads();
  contract_degrees<S>(pk, C0, C1, D, planeK, erk, 5 * R, 2 * R, [](int n) { return 5 * R + n; }, A);
  __syncthreads();
  // 7. write-out and carries (coalesced along j): a thread per (field, member,
  // latitude), the winds and the semi-implicit scheme's lagged remainders fourth.
  // All loads of a thread precede its stores (input and output may be one buffer),
  // and no two threads share a field.  Filters as write_step_point.
  for (int t = threadIdx.x; t < 4 * MT * J; t += 256) {
    const int j = t % J, bt = (t / J) % MT, q = t / (J * MT);
    if (bt >= mt || sdead[bt]) continue;
    const int b = b0 + bt;
    const size_t o = ((size_t)m * G.B + b) * J + j;
    auto get = [&](int f) {
      return make_double2(A[(size_t)(f * R + 2 * bt) * J + j], A[(size_t)(f * R + 2 * bt + 1) * J + j]);
    };
    const double2* Fi = G.four;
    double2* Fo = G.four_out;
    if (q < 3) {
      const int cf = q == 0 ? F_ETA : q == 1 ? F_DELTA : F_PHI;
      const int pf = q == 0 ? F_ETA_PREV : q == 1 ? F_DELTA_PREV : F_PHI_PREV;
      const int rf = q == 0 ? F_ETA_MID : q == 1 ? F_DELTA_MID : F_PHI_MID;
      double2 nw = get(q), old = make_double2(0.0, 0.0), mid = old;
      if (cfg.write_prev || cfg.ra_mode) old = Fi[cf * FS + o];
      if (cfg.ra_mode == 2) mid = Fi[rf * FS + o];
      if (cfg.write_prev) Fo[pf * FS + o] = old;
      if (cfg.ra_mode == 1) {
        Fo[rf * FS + o] = old;
      } else if (cfg.ra_mode == 2) {
        const double2 d = cadd(csub(mid, cscale(old, 2.0)), nw);
        Fo[rf * FS + o] = cadd(old, cscale(d, G.mco[(cfg.raw ? MC_RAWM : MC_ALPHA) * G.B + b]));
        if (cfg.raw) nw = csub(nw, cscale(d, G.mco[MC_RAWN * G.B + b]));
      }
      Fo[cf * FS + o] = nw;
    } else {
      if (cfg.scheme == 2) {
        const double itd = G.mco[MC_SIITD * G.B + b];
        const double2 l0 = cadd(Fi[F_F * FS + o], cscale(Fi[F_U * FS + o], itd));
        const double2 l1 = cadd(Fi[F_G * FS + o], cscale(Fi[F_V * FS + o], itd));
        Fo[F_RU_LAG * FS + o] = l0;
        Fo[F_RV_LAG * FS + o] = l1;
      }
      if (cfg.test != 1) {
        Fo[F_U * FS + o] = cadd(get(3), get(5));
        Fo[F_V * FS + o] = cadd(get(4), get(6));
      }
    }
  }
  // residual weights of the initial condition in the physical curr / prev fields
  if (m == 0 && threadIdx.x < mt && !sdead[threadIdx.x]) {
    const int b = b0 + threadIdx.x;
    double wc = G.member[MS_WCURR * G.B + b], wm = G.member[MS_WMID * G.B + b];
    step_residual_weights(cfg, G.par[P_ALPHA * G.B + b], G.par[P_WALPHA * G.B + b], wc, wm);
    G.member[MS_WMID * G.B + b] = wm;
    G.member[MS_WCURR * G.B + b] = wc;
    G.member[MS_UPDATED * G.B + b] = 1.0;
  }
}

// ------------------------------------------------------------------ adjoint
// The transpose (k_spectral_adj): lambda of the five outputs -> transposed
// inverse Legendre (5 rows on P, U and V on H) -> transposed epilogue ->
// transposed forward Legendre (5 on Pw, 4 on Hw) -> lambda of the state.
template <int M_, int MT>
__global__ void __launch_bounds__(256, 2) k_spectral_adj_f64(const __grid_constant__ SpecLaunch<double> L,
                                                             const __grid_constant__ SliceBasis basis) {
  typedef Sh<M_> S;
  typedef Mem<S, MT, 5, 7, 5, 9> Mm;
  constexpr int R = 2 * MT, J = S::J, NWS = J / 32;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  double* A = (double*)smem_raw;
  uint32_t* D = (uint32_t*)(smem_raw + Mm::A);
  int* erx = (int*)(smem_raw + Mm::A + Mm::B);
  int* erk = erx + 5 * R;
  __shared__ double sgrad[2][MT][NWS];
  int idx;
  const SpecGroup<double>& G = pick_group(L, idx);
  const StepCfg& cfg = L.cfg;
  const int m = idx / G.ntb, b0 = (idx % G.ntb) * MT, mt = min(MT, G.B - b0);
  const int cnt = S::CNT - m, C0 = (cnt + 1) / 2, C1 = cnt / 2;
  const size_t FS = (size_t)S::CNT * G.B * J;
  const PackView<S> pk(basis.p[&G - L.grp], m);
  if (MT == 1) {  // few units: their basis is not in L1 yet
    prefetch_lines(pk.f, (int)(Pack<S>::F * 16));
    prefetch_lines(pk.i, (int)(Pack<S>::I * 16));
  }
  for (int t = threadIdx.x; t < 2 * MT * NWS; t += 256) (&sgrad[0][0][0])[t] = 0.0;

  // 1. lambda of the outputs; the semi-implicit step's new level also enters its
  // filtered mid carry with weight alpha
  const bool si_ra = cfg.scheme == 2 && cfg.ra_mode == 2;
  for (int t = threadIdx.x; t < MT * J; t += 256) {
    const int bt = t / J, j = t % J, b = b0 + bt;
    const size_t o = ((size_t)m * G.B + b) * J + j;
#pragma unroll
    for (int f = 0; f < 5; ++f) {
      double2 u = make_double2(0.0, 0.0);
      if (bt < mt) {
        u = G.lamY[f * FS + o];
        if (si_ra && f < 3)
          u = cadd(u, cscale(G.lam[(f == 0 ? F_ETA_MID : f == 1 ? F_DELTA_MID : F_PHI_MID) * FS + o],
                             G.mco[MC_ALPHA * G.B + b]));
      }
      A[(size_t)(f * R + 2 * bt) * J + j] = u.x;
      A[(size_t)(f * R + 2 * bt + 1) * J + j] = u.y;
    }
  }
  __syncthreads();
  // 2., 3. transposed inverse Legendre: 5 rows on P, U and V again on H
  constexpr int planeX = 5 * R * 2 * S::XW, planeK = 5 * R * S::KW;
  slice_latitudes<S>(A, 5 * R, pk.ep, D, planeX, erx);
  __syncthreads();
  contract_latitudes<S>(pk, C0, C1, D, planeX, erx, 5 * R, 3 * R, 2 * R, A);
  __syncthreads();
  // 4. transposed wind inversion, n(n+1) and hyperdiffusion (solve per degree in scheme 2)
  constexpr int NC = 2 * MT * S::CNT <= 256 ? 1 : 2;  // components per thread
  static_assert(MT * S::CNT <= 256, "one spectral point per thread");
  {
    const int comp0 = NC == 1 ? (int)threadIdx.x / (MT * cnt) : 0, t = (int)threadIdx.x - comp0 * MT * cnt;
    const int bt = t / cnt, kk = t % cnt;
    const bool on = comp0 < 2 && bt < mt;
    const int par = kk & 1, c = kk >> 1, pc = par ? C0 + c : c, n = m + kk, b = b0 + bt;
    double k[5][NC];
    if (on) {
      auto S_ = [&](int q, int comp) { return A[(size_t)(q * R + 2 * bt + comp) * S::CNT + pc]; };
      const size_t qs = (size_t)G.B * S::CNT, qo = (size_t)b * S::CNT + n;
      const bool expo_sig = cfg.scheme == 2;
      const double s = cfg.diffflag ? G.nco[(expo_sig ? NC_SIGX : NC_SIG) * qs + qo] : 1.0;
      const double sp = cfg.diffflag ? G.nco[(expo_sig ? NC_SIGPX : NC_SIGP) * qs + qo] : 1.0;
      const double w = n == 0 ? 0.0 : G.nco[NC_TC * qs + qo];
      const double nn1 = (double)(n * (n + 1)), xm = (double)m;
      // lambda delta_s = (i m) lambda Uprep - lambda Hin_V ; lambda eta_s = (i m) lambda Vprep + lambda Hin_U
      auto lds = [&](int comp) { return (comp == 0 ? -xm * S_(3, 1) : xm * S_(3, 0)) - S_(6, comp); };
      auto les = [&](int comp) { return (comp == 0 ? -xm * S_(4, 1) : xm * S_(4, 0)) + S_(5, comp); };
      double bq = 0.0, cq = 0.0, ikr = 1.0, ikd = 1.0, Dn = 1.0;
      if (cfg.scheme == 2) {
        const double* mc = G.mco;
        const double xi = mc[MC_SIXI * G.B + b];
        double kd = 0.0, kr = 0.0;
        if (cfg.si_relax) {
          kd = xi * mc[MC_SIITD * G.B + b];
          kr = xi * mc[MC_SIITR * G.B + b];
        }
        bq = xi * (nn1 * mc[MC_IA2 * G.B + b]);
        cq = xi * mc[MC_PB * G.B + b];
        ikr = 1.0 / (1.0 + kr);
        ikd = 1.0 / (1.0 + kd);
        Dn = (1.0 + kd) + bq * cq * ikr;
      }
#pragma unroll
      for (int i = 0; i < NC; ++i) {
        const int comp = comp0 + i;
        const double lce = S_(0, comp) + w * les(comp), lcd = S_(1, comp) + w * lds(comp), lcp = S_(2, comp);
        if (cfg.scheme == 2) {
          const double lpn = sp * lcp, ldn = s * lcd - cq * ikr * lpn, lsd = ldn / Dn;
          k[0][i] = ikr * lpn + bq * ikr * lsd;
          k[1][i] = 0.0;
          k[2][i] = lsd;
          k[3][i] = nn1 * lsd;
          k[4][i] = ikd * s * lce;
        } else {
          k[0][i] = sp * lcp;
          k[1][i] = nn1 * sp * lcp;
          k[2][i] = s * lcd;
          k[3][i] = nn1 * s * lcd;
          k[4][i] = s * lce;
        }
      }
    }
    __syncthreads();
    if (on) {
      double* K = A + (size_t)(2 * bt + comp0) * 2 * S::PC + par * S::PC + c;
#pragma unroll
      for (int q = 0; q < 5; ++q)
#pragma unroll
        for (int i = 0; i < NC; ++i) K[(size_t)(q * R + i) * 2 * S::PC] = k[q][i];
    }
    for (int i = threadIdx.x; i < 5 * (R - 2 * mt) * 2 * S::PC; i += 256) {
      const int kx = i % (2 * S::PC), r = 2 * mt + (i / (2 * S::PC)) % (R - 2 * mt), q = i / (2 * S::PC * (R - 2 * mt));
      A[(size_t)(q * R + r) * 2 * S::PC + kx] = 0.0;
    }
  }
  __syncthreads();
  // 5., 6. transposed forward Legendre: K0..K4 on Pw; K0, K2, K3, K4 on Hw
  slice_degrees<S>(A, 5 * R, C0, C1, D, planeK, erk);
  __syncthreads();
  contract_degrees<S>(pk, C0, C1, D, planeK, erk, 5 * R, 4 * R, [](int n) { return n < R ? n : n + R; }, A);
  __syncthreads();
  // 7. transposed combination; Phibar (and explicit-scheme drag) gradient
  for (int t = threadIdx.x; t < MT * J; t += 256) {
    const int bt = t / J, j = t % J;
    if (bt >= mt) continue;
    const int b = b0 + bt;
    const size_t o = ((size_t)m * G.B + b) * J + j;
    auto ld = [&](int q) {
      return make_double2(A[(size_t)(q * R + 2 * bt) * J + j], A[(size_t)(q * R + 2 * bt + 1) * J + j]);
    };
    AdjPointIn<double> in;
    adj_load_point<double>(G, cfg, false, FS, o, in);
    double gtd = 0.0;
    double gp = adj_store_point<double, 5>(G, cfg, false, FS, o, m, b, j, ld, in, gtd);
    if (G.grad) {  // J is a multiple of 32: a warp holds one member
#pragma unroll
      for (int off = 16; off > 0; off >>= 1) {
        gp += __shfl_xor_sync(0xffffffffu, gp, off);
        if (cfg.scheme == 1) gtd += __shfl_xor_sync(0xffffffffu, gtd, off);
      }
      if ((threadIdx.x & 31) == 0) {
        sgrad[0][bt][j / 32] = gp;
        sgrad[1][bt][j / 32] = gtd;
      }
    }
  }
  __syncthreads();
  if (G.grad && threadIdx.x < mt) {
    double acc = 0.0, acd = 0.0;
    for (int w = 0; w < NWS; ++w) {
      acc += sgrad[0][threadIdx.x][w];
      acd += sgrad[1][threadIdx.x][w];
    }
    atomicAdd(&G.grad[G_PHIBAR * G.B + b0 + threadIdx.x], acc);
    if (cfg.scheme == 1) atomicAdd(&G.grad[G_TAUDRAG * G.B + b0 + threadIdx.x], acd);
  }
}

// Members per unit.  One round of CTAs (two per SM) at one member each, then two;
// four (M = 42 only: the unit's shared memory has to fit twice in an SM) once
// those are most of a round themselves.  Step (transpose), M = 42, us with 1 / 2 / 4
// members: 7 members 21 / 25 / 32 (21 / 27 / 32), 8 members 28 / 25 / 32 (31 / 27 /
// 32), 16 members 43 / 34 / 40 (47 / 41 / 42), 20 members 45 / 40 / 40 (49 / 44 / 43),
// 24 members 53 / 42 / 40 (61 / 46 / 43), 32 members 67 / 54 / 55 (76 / 63 / 56), 256
// members 459 / 317 / 296 (544 / 381 / 292); M = 63 with 1 / 2: 4 members 28 / 29 (28 /
// 27), 5 members 44 / 35 (41 / 35), 32 members 153 / 119 (158 / 115).  The FMA kernels
// took 880 / 840 us for 256 members and 98 / 80 us for one, now 17 / 18.
template <int M_>
int tile_for(const SpecLaunch<double>& L) {
  auto units = [&](int mt) {
    int n = 0;
    for (int g = 0; g < L.ng; ++g)
      if (L.grp[g].g.M == M_) n += (M_ + 1) * ((L.grp[g].B + mt - 1) / mt);
    return n;
  };
  if (M_ == 42 && units(4) >= 256) return 4;
  return M_ <= 63 && units(1) > 2 * 152 ? 2 : 1;
}

template <int M_, int MT, bool ADJ>
cudaError_t launch_one(SpecLaunch<double> L, const SliceBasis& basis, cudaStream_t s) {
  int acc = 0;
  for (int g = 0; g < L.ng; ++g) {
    if (L.grp[g].g.M != M_) L.grp[g].B = 0;
    L.grp[g].MT = MT;
    L.grp[g].ntb = (L.grp[g].B + MT - 1) / MT;
    L.prefix[g] = acc;
    acc += (M_ + 1) * L.grp[g].ntb;
  }
  L.prefix[L.ng] = acc;
  if (acc == 0) return cudaSuccess;
  typedef Sh<M_> S;
  if constexpr (ADJ) {
    constexpr size_t smem = Mem<S, MT, 5, 7, 5, 9>::total;
    k_spectral_adj_f64<M_, MT><<<acc, 256, smem, s>>>(L, basis);
  } else {
    constexpr size_t smem = Mem<S, MT, NIN, NIN, 7, 7>::total;
    k_spectral_f64<M_, MT><<<acc, 256, smem, s>>>(L, basis);
  }
  return cudaGetLastError();
}

template <int M_, bool ADJ>
cudaError_t launch_trunc(const SpecLaunch<double>& L, const SliceBasis& basis, cudaStream_t s) {
  const int mt = tile_for<M_>(L);
  if constexpr (M_ == 42)
    if (mt == 4) return launch_one<M_, 4, ADJ>(L, basis, s);
  if constexpr (M_ <= 63)
    if (mt == 2) return launch_one<M_, 2, ADJ>(L, basis, s);
  return launch_one<M_, 1, ADJ>(L, basis, s);
}

template <int M_, int MT>
void set_attr() {
  typedef Sh<M_> S;
  static_assert(Mem<S, MT, NIN, NIN, 7, 7>::total <= 112 * 1024 && Mem<S, MT, 5, 7, 5, 9>::total <= 112 * 1024,
                "two CTAs per SM");
  cudaFuncSetAttribute(k_spectral_f64<M_, MT>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                       (int)Mem<S, MT, NIN, NIN, 7, 7>::total);
  cudaFuncSetAttribute(k_spectral_adj_f64<M_, MT>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                       (int)Mem<S, MT, 5, 7, 5, 9>::total);
}

}  // namespace

size_t spec_f64_basis_bytes(int M) {
  return M == 42 ? Pack<Sh<42>>::bytes : M == 63 ? Pack<Sh<63>>::bytes : Pack<Sh<106>>::bytes;
}

// The packed basis of the step (adjoint = false: weighted basis over latitudes,
// unweighted over degrees) or of its transpose.
cudaError_t pack_spec_f64(const GroupGeom& gg, bool adjoint, void* out, cudaStream_t s) {
  const double *fp = gg.b64[adjoint ? B_P_F : B_PW_F], *fh = gg.b64[adjoint ? B_H_F : B_HW_F];
  const double *ip = gg.b64[adjoint ? B_PW_F : B_P_F], *ih = gg.b64[adjoint ? B_HW_F : B_H_F];
  if (gg.M == 42) k_pack_slices<Sh<42>><<<43, 256, 0, s>>>(fp, fh, ip, ih, gg.boff, out);
  else if (gg.M == 63) k_pack_slices<Sh<63>><<<64, 256, 0, s>>>(fp, fh, ip, ih, gg.boff, out);
  else k_pack_slices<Sh<106>><<<107, 256, 0, s>>>(fp, fh, ip, ih, gg.boff, out);
  return cudaGetLastError();
}

void spec_f64_set_attributes() {
  set_attr<42, 1>(); set_attr<42, 2>(); set_attr<42, 4>();
  set_attr<63, 1>(); set_attr<63, 2>();
  set_attr<106, 1>();
}

cudaError_t launch_spec_f64(const SpecLaunch<double>& L, const SliceBasis& basis, bool adjoint, cudaStream_t s) {
  cudaError_t e = adjoint ? launch_trunc<106, true>(L, basis, s) : launch_trunc<106, false>(L, basis, s);
  if (e == cudaSuccess) e = adjoint ? launch_trunc<63, true>(L, basis, s) : launch_trunc<63, false>(L, basis, s);
  if (e == cudaSuccess) e = adjoint ? launch_trunc<42, true>(L, basis, s) : launch_trunc<42, false>(L, basis, s);
  return e;
}

}  // namespace swp

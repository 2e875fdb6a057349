// The FP64 grid half of a step (GM_STEP) and its adjoint (GM_ADJ_STEP) with the
// longitude transforms as matrix products on the FP16 tensor cores (slices.cuh).
// The other modes, and FP32, are grid.cu's FFTs; the physics is shared.
//
// What bounded the FFT kernels was the FP64 pipe (1.7 instructions per cycle and
// SM): of about 32,000 FP64 instructions per latitude row of a step at M = 42,
// 24,000 were the 12 transforms.  A transform of truncated Fourier rows is a
// product with a static cosine and sine matrix of M + 1 by I / 2; on slices it
// costs no FP64 instruction, and the physics' 4,000 remain.  M = 42, step / adjoint:
// 256 members 806 / 1174 -> 371 / 622 us, one member 39 / 55 -> 14 / 18 us.  FP64
// pipe, tensor cores and integer issue each account for about a third of that; the
// phases between barriers overlap only across the two CTAs of an SM (128 registers).
//
// One CTA: one member, JB latitude rows.
//   1. cp.async of the rows' truncated Fourier coefficients;
//   2. a warp per (field, row) slices real and imaginary parts, lanes over m;
//   3. tiles of 16 longitudes x 8 rows: even part e_i = sum_m w_m Re Y_m cos,
//      odd part o_i = sum_m w_m Im Y_m sin, i < I/2, w_0 = 1, w_m = 2; added and
//      subtracted in integers: x_i = e - o, x_{I-i} = e + o.  The longitude I/2,
//      an alternating sum, is taken while slicing;
//   4. physics, a thread per point, in place;
//   5. a warp per (field, row) folds x_i +- x_{I-i} in integers and slices;
//   6. tiles of 16 wavenumbers x 8 rows over i < I/2, real and imaginary parts
//      apart; the term of longitude I/2, folded into i = 0 with the sign of even
//      m, is corrected in the integers for odd m.
#include "grid_common.cuh"
#include "slices.cuh"

namespace swp {
namespace {

using namespace slices;

template <int M_>
struct Sh {
  static constexpr int M = M_, J = trunc_J(M_), I = trunc_I(M_), L = I / 2, N1 = M_ + 1;
  static constexpr int KM = (N1 + 15) / 16;  // k-steps, or tiles, over wavenumbers
  static constexpr int KL = L / 16;          // tiles, or k-steps, over longitudes
  static constexpr int KP = 16 * KM;         // padded wavenumbers
  static constexpr int YW = KP + 4;          // words of a sliced Fourier row: Re [KP/2], Im [KP/2], padded
  static constexpr int ZW = L + 4;           // words of a sliced longitude row: sums [L/2], differences [L/2], padded
  // 1/I as a power of two (I = 128) goes into the scale of the result; else a factor
  static constexpr bool POW2 = (I & (I - 1)) == 0;
  static constexpr int LOG2I = 7;
  static_assert(L % 32 == 0 && (!POW2 || I == 128), "grid sizes");
};
// Scales of the static matrices: entries up to 2 (C2R weights) and up to 1.
constexpr int ER_C2R = 1024, ER_R2C = 1023;

// Packed matrices [C2R cos, sin][KL tiles][KM k-steps], [R2C cos, -sin][KM tiles][KL k-steps], each [digit][lane].
template <class S>
struct Pack {
  static constexpr size_t part = (size_t)S::KL * S::KM * ND * 32;  // uint4 of one matrix
  static constexpr size_t bytes = 4 * part * 16;
};

// cos(2 pi k / I) by folding k into [0, I/8] with exact values at the axes.
__device__ double cos_grid(int k, int I) {
  k %= I;
  if (k > I / 2) k = I - k;
  double s = 1.0;
  if (k > I / 4) {
    k = I / 2 - k;
    s = -1.0;
  }
  return s * (4 * k == I ? 0.0 : 8 * k <= I ? cospi(2.0 * k / I) : sinpi(0.5 - 2.0 * k / I));
}
__device__ double sin_grid(int k, int I) { return cos_grid(k + 3 * I / 4, I); }

template <class S>
__global__ void k_pack_grid(uint4* out) {
  const int total = 4 * S::KL * S::KM * 32;
  for (int u = blockIdx.x * blockDim.x + threadIdx.x; u < total; u += gridDim.x * blockDim.x) {
    const int lane = u & 31, mat = u / (S::KL * S::KM * 32);
    const int ks = mat < 2 ? S::KM : S::KL, q0 = (u / 32) % (S::KL * S::KM), tile = q0 / ks, k0 = 16 * (q0 % ks);
    auto elem = [&](int row, int k) {
      const int m = mat < 2 ? k : row, i = mat < 2 ? row : k;
      if (m > S::M) return 0.0;
      const double w = mat < 2 ? (m ? 2.0 : 1.0) : 1.0;
      return w * (mat == 0 || mat == 2 ? cos_grid(i * m, S::I) : mat == 1 ? sin_grid(i * m, S::I) : -sin_grid(i * m, S::I));
    };
    const int er = mat < 2 ? ER_C2R : ER_R2C;
    uint32_t w[4][ND];
    for (int q = 0; q < 4; ++q) {
      const int row = 16 * tile + (lane >> 2) + 8 * (q & 1), k = k0 + 2 * (lane & 3) + 8 * (q >> 1);
      store_digits(w[q], 1, fixed(elem(row, k), er), fixed(elem(row, k + 1), er));
    }
    uint4* dst = out + (size_t)(u / 32) * ND * 32 + lane;
    for (int d = 0; d < ND; ++d) dst[d * 32] = make_uint4(w[0][d], w[1][d], w[2][d], w[3][d]);
  }
}

// NF Fourier rows to the grid and NZ grid rows back, per latitude row.
template <class S, int JB, int NF, int NZ>
struct Mem {
  static constexpr int NG = NF > NZ ? NF : NZ;  // grid fields held
  static constexpr size_t raw = (size_t)NF * S::N1 * JB * 16, grid = (size_t)NG * JB * S::I * 8;
  static constexpr size_t A = raw > grid ? raw : grid;
  static constexpr size_t sy = (size_t)ND * NF * JB * S::YW * 4, sz = (size_t)ND * NZ * JB * S::ZW * 4;
  static constexpr size_t B = sy > sz ? sy : sz;
  static constexpr size_t Q = (size_t)NZ * JB * 8, E = (size_t)(NF + NZ) * JB * 4;
  static constexpr size_t total = A + B + Q + E;
};

// Slices of the raw rows [f][m][r] (complex).  Rows of fields f < nhalf have the
// coefficients of m >= 1 halved (adjoint rows: their weight is 1, the matrix'
// 2).  mid: the value at longitude I/2, sum_m w_m (-1)^m Re Y_m, summed in
// integers from every digit and rounded once; a lane converts a row of the warp's, so
// that the FP64 instructions serve them all.
template <class S, int JB>
__device__ __forceinline__ void slice_fourier(const double2* raw, int nrow, int nhalf, uint32_t* dig, int plane,
                                              int* er, double* mid) {
  constexpr int KI = (S::KP + 31) / 32;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  long long row_alt = 0;  // of row warp + 8 lane
  int row_low = 0, row_e = ER_ZERO;
  for (int row = warp; row < nrow; row += 8) {
    const int f = row / JB, r = row % JB, half = f < nhalf ? 1 : 0;
    double2 y[KI];
    int e = 0;
#pragma unroll
    for (int i = 0; i < KI; ++i) {
      const int m = lane + 32 * i;
      y[i] = m < S::N1 ? raw[((size_t)f * S::N1 + m) * JB + r] : make_double2(0.0, 0.0);
      const int h = m ? half : 0;
      const int ex = max(expo(y[i].x), expo(y[i].y));
      e = max(e, ex == 0x7ff ? ER_BAD : max(ex - h, 0));
    }
    e = row_exponent((int)__reduce_max_sync(0xffffffffu, (unsigned)e));
    if (lane == 0) er[row] = e;
    long long alt = 0;  // in units of 2^8 of the scale (a lane's m are of one parity)
    int low = 0;        // and of its unit
#pragma unroll
    for (int i = 0; i < KI; ++i) {
      const int m = lane + 32 * i, h = m ? half : 0;
      uint64_t a = fixed(y[i].x, e + h), b = fixed(y[i].y, e + h);
      const long long q = (long long)(a - BIAS);
      const long long qh = q >> 8;
      const int ql = (int)q & 0xff;
      alt += m ? 2 * qh : qh;
      low += m ? 2 * ql : ql;
      pair_exchange(a, b);
      if (S::KP % 32 == 0 || m < S::KP)
        store_digits(dig + (size_t)row * S::YW + (lane & 1) * (S::KP / 2) + (lane >> 1) + 16 * i, plane, a, b);
    }
    if (lane & 1) {
      alt = -alt;
      low = -low;
    }
    // the warp's sums, 24 bits of alt at a time: four independent reductions
    const int a0 = __reduce_add_sync(0xffffffffu, (int)(alt & 0xffffff));
    const int a1 = __reduce_add_sync(0xffffffffu, (int)((alt >> 24) & 0xffffff));
    const int a2 = __reduce_add_sync(0xffffffffu, (int)(alt >> 48));
    low = __reduce_add_sync(0xffffffffu, low);
    alt = (long long)a0 + ((long long)a1 << 24) + (long long)a2 * (1ll << 48);
    if (lane == row >> 3) {
      row_alt = alt;
      row_low = low;
      row_e = e;
    }
  }
  if (warp + 8 * lane < nrow) {
    // (alt 2^8 + low) 2^(e - 1084): alt's upper 50 bits and the rest are exact in FP64, one rounding
    const double hi = (double)(row_alt >> 12), lo = (double)(int)(((int)(row_alt & 0xfff) << 8) + row_low);
    double v = fma(hi, 1048576.0, lo) * __hiloint2double((row_e - 61) << 20, 0);
    if (row_e == ER_ZERO) v = 0.0;
    if (row_e == ER_BAD) v = __longlong_as_double(0x7ff8000000000000ll);
    mid[warp + 8 * lane] = v;
  }
}

// Grid rows [row][I] from the sliced Fourier rows.  Rows of fields f < nscaled
// are multiplied by 1/I.  mid: the values at longitude I/2.
template <class S, int JB>
__device__ __forceinline__ void c2r_tiles(const uint4* __restrict__ mats, const uint32_t* dig, int plane,
                                          const int* er, const double* mid, int nrow, int nscaled, double* grid) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  const int NT = (nrow + 7) / 8;
  for (int job = warp; job < S::KL * NT; job += 8) {
    const int nt = job % NT, tile_i = job / NT, n0 = 8 * nt;
    const uint32_t* b = dig + (size_t)min(n0 + g, nrow - 1) * S::YW + t;
    long long eh[4], el[4];
    Tile tile;
#pragma unroll
    for (int part = 0; part < 2; ++part) {
      const uint4* a = mats + part * Pack<S>::part + (size_t)tile_i * S::KM * ND * 32 + lane;
      tile.reset();
#pragma unroll
      for (int ks = 0; ks < S::KM; ++ks) {
        uint32_t af[ND][4], bf[ND][2];
        load_a(af, a + (size_t)ks * ND * 32);
        const uint32_t* p = b + part * (S::KP / 2) + 8 * ks;
        load_b(bf, p, p + 4, plane);
        tile.step(af, bf);
        if (ks % KFLUSH == KFLUSH - 1 || ks == S::KM - 1) tile.flush();
      }
      if (part == 0) {
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          eh[e] = tile.hi[e];
          el[e] = tile.lo[e];
        }
      }
    }
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const int i = 16 * tile_i + g + 8 * (e >> 1), n = n0 + 2 * t + (e & 1);
      if (n >= nrow) continue;
      const bool scaled = n < nscaled * JB;
      const int sa = ER_C2R - (S::POW2 && scaled ? S::LOG2I : 0), sb = er[n];
      double lo = value(eh[e] - tile.hi[e], el[e] - tile.lo[e], sa, sb);
      double hi = value(eh[e] + tile.hi[e], el[e] + tile.lo[e], sa, sb);
      if (!S::POW2 && scaled) {
        lo *= 1.0 / S::I;
        hi *= 1.0 / S::I;
      }
      double* x = grid + (size_t)n * S::I;
      x[i] = lo;
      if (i > 0) x[S::I - i] = hi;
      else x[S::L] = scaled ? mid[n] * (1.0 / S::I) : mid[n];
    }
  }
}

// Folded slices of the grid rows: sums x_i + x_{I-i} (i = 0: x_0 + x_{I/2}) and
// differences, formed in integers on a scale with one bit of headroom.
// qmid: the fixed-point value at longitude I/2.
template <class S>
__device__ __forceinline__ void slice_grid(const double* grid, int nrow, uint32_t* dig, int plane, int* er,
                                           long long* qmid) {
  constexpr int KI = S::L / 32;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  for (int row = warp; row < nrow; row += 8) {
    const double* x = grid + (size_t)row * S::I;
    double xa[KI], xb[KI];
    int e = 0;
#pragma unroll
    for (int i = 0; i < KI; ++i) {
      const int k = lane + 32 * i;
      xa[i] = x[k];
      xb[i] = x[k ? S::I - k : S::L];
      e = max(e, max(expo(xa[i]), expo(xb[i])));
    }
    e = (int)__reduce_max_sync(0xffffffffu, (unsigned)e);
    e = row_exponent(e == 0x7ff ? e : e + 1);
    if (lane == 0) er[row] = e;
#pragma unroll
    for (int i = 0; i < KI; ++i) {
      const int k = lane + 32 * i;
      const uint64_t fa = fixed(xa[i], e), fb = fixed(xb[i], e);
      uint64_t s = fa + fb - BIAS, d = k ? fa - fb + BIAS : BIAS;
      if (k == 0) qmid[row] = (long long)(fb - BIAS);
      pair_exchange(s, d);
      store_digits(dig + (size_t)row * S::ZW + (lane & 1) * (S::L / 2) + (lane >> 1) + 16 * i, plane, s, d);
    }
  }
}

// Fourier coefficients of the folded rows: put(row, m, component, sum) receives
// sum_i x_i cos or -sin (2 pi i m / I) times 2^shift(m).
template <class S, typename F>
__device__ __forceinline__ void r2c_tiles(const uint4* __restrict__ mats, const uint32_t* dig, int plane,
                                          const int* er, const long long* qmid, int nrow, int shift0, int shift1,
                                          F put) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  const int NT = (nrow + 7) / 8;
  for (int job = warp; job < 2 * S::KM * NT; job += 8) {
    const int nt = job % NT, comp = (job / NT) & 1, tile_m = job / (2 * NT), n0 = 8 * nt;
    const uint32_t* b = dig + (size_t)min(n0 + g, nrow - 1) * S::ZW + comp * (S::L / 2) + t;
    const uint4* a = mats + (2 + comp) * Pack<S>::part + (size_t)tile_m * S::KL * ND * 32 + lane;
    Tile tile;
    tile.reset();
#pragma unroll 2
    for (int ks = 0; ks < S::KL; ++ks) {
      uint32_t af[ND][4], bf[ND][2];
      load_a(af, a + (size_t)ks * ND * 32);
      load_b(bf, b + 8 * ks, b + 8 * ks + 4, plane);
      tile.step(af, bf);
      if (ks % KFLUSH == KFLUSH - 1) tile.flush();
    }
    static_assert(S::KL % KFLUSH == 0, "whole flushes");
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const int m = 16 * tile_m + g + 8 * (e >> 1), n = n0 + 2 * t + (e & 1);
      if (m > S::M || n >= nrow) continue;
      if (comp == 0 && (m & 1)) {
        // longitude I/2 entered with +1; odd m have -1.  q times the matrix' 1 (2^61 on
        // its scale) is q 2^5 units of lo (2^56)
        const long long q2 = 2 * qmid[n];
        tile.hi[e] -= q2 >> 27;
        tile.lo[e] -= (q2 & 0x7ffffffll) << 5;
      }
      put(n, m, comp, value(tile.hi[e], tile.lo[e], ER_R2C + (m ? shift1 : shift0), er[n]));
    }
  }
}

template <typename C>
__device__ __forceinline__ void copy_rows(const C& src, int nf, int n1, int JB, int B, int b, int J, int j0,
                                          double2* raw, int f0 = 0) {
  for (int t = threadIdx.x; t < nf * n1 * JB; t += 256) {
    const int r = t % JB, k = (t / JB) % n1, f = t / (JB * n1);
    cp_async<16>(raw + ((size_t)(f0 + f) * n1 + k) * JB + r, src(f) + ((size_t)k * B + b) * J + j0 + r);
  }
}

// --------------------------------------------------------------------- step
constexpr int STEP_NF = 6, STEP_NZ = 8;  // eta, Phi, U, V (+ delta for the history, + the diagnostic Phi) -> A .. G
template <int M_, int JB>
__global__ void __launch_bounds__(256, 2) k_grid_step_f64(const __grid_constant__ GridLaunch<double> Lc,
                                                          const __grid_constant__ SliceBasis basis) {
  typedef Sh<M_> S;
  typedef Mem<S, JB, STEP_NF, STEP_NZ> Mm;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  double* A = (double*)smem_raw;
  uint32_t* D = (uint32_t*)(smem_raw + Mm::A);
  long long* qmid = (long long*)(smem_raw + Mm::A + Mm::B);
  int* ery = (int*)(qmid + STEP_NZ * JB);
  int* erz = ery + STEP_NF * JB;
  __shared__ double s_mid[STEP_NF * JB], s_par[7];
  __shared__ StepDiag<double>::Block s_diag;
  __shared__ int s_flag[2];
  int idx;
  const GridGroup<double>& G = pick_ggroup(Lc, idx);
  const StepCfg& cfg = Lc.cfg;
  const int B = G.B, b = idx / (S::J / JB), j0 = (idx % (S::J / JB)) * JB;
  const size_t FS = (size_t)S::N1 * B * S::J, PS = (size_t)B * S::J * S::I;
  const uint4* mats = (const uint4*)basis.p[&G - Lc.grp];
  const int nfix = G.hist ? 5 : 4, nf = nfix + (cfg.diagnostics ? 1 : 0);
  double2* raw = (double2*)A;
  copy_rows([&](int f) { return G.four + (size_t)(f == 0 ? F_ETA : f == 1 ? F_PHI : f == 2 ? F_U : f == 3 ? F_V : F_DELTA) * FS; },
            nfix, S::N1, JB, B, b, S::J, j0, raw);
  // the diagnosed Phi is the filtered level's; a dead member's, the current's, replaces it below
  if (cfg.diagnostics)
    copy_rows([&](int) { return G.four + (size_t)F_PHI_MID * FS; }, 1, S::N1, JB, B, b, S::J, j0, raw, nfix);
  if (threadIdx.x == 0) {
    const double td = G.par[P_TAUDRAG * B + b];
    const bool stepped = G.member && G.member[MS_UPDATED * B + b] != 0.0;
    const double wc = G.member ? G.member[MS_WCURR * B + b] : 0.0;
    s_par[0] = G.par[P_PHIBAR * B + b];
    s_par[1] = G.mco[MC_SIITR * B + b];  // 1 / taurad and 1 / taudrag, from the call's tables
    s_par[2] = G.mco[MC_ITD * B + b];
    s_par[3] = G.par[P_DPHIEQ * B + b];
    s_par[4] = wc;
    s_par[5] = G.member ? G.member[MS_WMID * B + b] : 0.0;
    // the winds of a stepped member are band-limited; test 1 keeps its initial winds
    s_par[6] = cfg.test == 1 ? 1.0 : stepped ? 0.0 : wc;
    s_flag[0] = td == -1.0;
    s_flag[1] = (cfg.diagnostics && G.member) ? (G.member[MS_DEAD * B + b] != 0.0) : 0;
  }
  __syncthreads();
  const bool dead = s_flag[1] != 0;
  if (dead) {
    cp_async_wait_all();
    __syncthreads();
    copy_rows([&](int) { return G.four + (size_t)F_PHI * FS; }, 1, S::N1, JB, B, b, S::J, j0, raw, nfix);
  }
  Physics<double> ph;
  ph.Pb = s_par[0]; ph.itr = s_par[1]; ph.itd = s_par[2]; ph.DPe = s_par[3];
  ph.nodrag = s_flag[0] != 0; ph.forced = cfg.test == 0;
  cp_async_wait_all();
  __syncthreads();
  constexpr int planeY = STEP_NF * JB * S::YW, planeZ = STEP_NZ * JB * S::ZW;
  slice_fourier<S, JB>(raw, nf * JB, 0, D, planeY, ery, s_mid);
  __syncthreads();
  c2r_tiles<S, JB>(mats, D, planeY, ery, s_mid, nf * JB, 0, A);
  __syncthreads();
  // physics: a thread per point, outputs in place of the fields
  StepDiag<double> dg;
  const int nout = ph.forced ? 8 : 5;
  for (int t = threadIdx.x; t < JB * S::I; t += 256) {
    const int i = t % S::I, r = t / S::I, j = j0 + r;
    double v[STEP_NF];
#pragma unroll
    for (int f = 0; f < STEP_NF; ++f) {
      if (f >= nf) break;
      v[f] = A[(size_t)(f * JB + r) * S::I + i];
      // initial-condition residual (weights non-zero before a member's first step, with the RAW filter, in test 1)
      const bool mid = f >= nfix && !dead;
      const double w = (f == 2 || f == 3) ? s_par[6] : mid ? s_par[5] : s_par[4];
      if (w != 0.0 && G.resid) {
        const int rf = f == 0 ? R_ETA : f == 2 ? R_U : f == 3 ? R_V : (f == 4 && nfix == 5) ? R_DELTA : R_PHI;
        v[f] += w * G.resid[rf * PS + ((size_t)b * S::J + j) * S::I + i];
      }
    }
    double o[8];
    ph.eval(v[0], v[1], v[2], v[3], G.g.ihalf[j], G.g.dayc[i] * G.g.coslat[j], o);
#pragma unroll
    for (int q = 0; q < 8; ++q)
      if (q < nout) A[(size_t)(q * JB + r) * S::I + i] = o[q];
    if (G.hist) {  // [5][B][J][I]: eta, delta, Phi, U, V
      double* h = G.hist + ((size_t)b * S::J + j) * S::I + i;
      h[0] = v[0];
      h[PS] = v[4];
      h[2 * PS] = v[1];
      h[3 * PS] = v[2];
      h[4 * PS] = v[3];
    }
    if (cfg.diagnostics) {
      dg.speed(G.g.area[j], v[2] * v[2] + v[3] * v[3]);
      dg.phi(nfix == 5 ? v[5] : v[4]);
    }
  }
  if (cfg.diagnostics) dg.put(s_diag);
  __syncthreads();
  slice_grid<S>(A, nout * JB, D, planeZ, erz, qmid);
  __syncthreads();
  double* four = (double*)(G.four + (size_t)F_A * FS);
  r2c_tiles<S>(mats, D, planeZ, erz, qmid, nout * JB, S::POW2 ? -S::LOG2I : 0, S::POW2 ? -S::LOG2I : 0,
               [&](int n, int m, int comp, double x) {
                 if (!S::POW2) x *= 1.0 / S::I;
                 four[2 * ((size_t)(n / JB) * FS + ((size_t)m * B + b) * S::J + j0 + n % JB) + comp] = x;
               });
  // after the products, which leave the last warps without a tile for few rows
  if (cfg.diagnostics) {
    double* dc = G.diag + (size_t)cfg.step * NDIAG * B;
    StepDiag<double>::add(s_diag, dc + NDIAG * B, dc, B, b);
  }
  // unforced runs: zero forcing terms, written explicitly (model.py:601-603)
  if (!ph.forced)
    for (int t = threadIdx.x; t < 3 * S::N1 * JB; t += 256) {
      const int r = t % JB, k = (t / JB) % S::N1, q = t / (JB * S::N1);
      G.four[(F_PHIF + q) * FS + ((size_t)k * B + b) * S::J + j0 + r] = make_double2(0.0, 0.0);
    }
}

// ------------------------------------------------------------------ adjoint
constexpr int ADJ_NF = 12, ADJ_NZ = 4;  // lambda of up to 8 terms and eta, Phi, U, V -> lambda of eta, Phi, U, V
template <int M_, int JB>
__global__ void __launch_bounds__(256, 2) k_grid_adj_f64(const __grid_constant__ GridLaunch<double> Lc,
                                                         const __grid_constant__ SliceBasis basis) {
  typedef Sh<M_> S;
  typedef Mem<S, JB, ADJ_NF, ADJ_NZ> Mm;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  double* A = (double*)smem_raw;
  uint32_t* D = (uint32_t*)(smem_raw + Mm::A);
  long long* qmid = (long long*)(smem_raw + Mm::A + Mm::B);
  int* ery = (int*)(qmid + ADJ_NZ * JB);
  int* erz = ery + ADJ_NF * JB;
  __shared__ double s_mid[ADJ_NF * JB], s_par[4], s_red[8 * NGRAD];
  __shared__ int s_nodrag;
  int idx;
  const GridGroup<double>& G = pick_ggroup(Lc, idx);
  const StepCfg& cfg = Lc.cfg;
  const int B = G.B, b = idx / (S::J / JB), j0 = (idx % (S::J / JB)) * JB;
  const size_t FS = (size_t)S::N1 * B * S::J;
  const uint4* mats = (const uint4*)basis.p[&G - Lc.grp];
  const bool forced = cfg.test == 0;
  // inside an adjoint sweep lambda_F = lambda_B and lambda_G = -lambda_A: taken from them
  const bool tied = forced && cfg.lam_fg_tied != 0;
  const int nz = tied ? 6 : forced ? 8 : 5, nf = nz + 4;
  double2* raw = (double2*)A;
  copy_rows([&](int f) {
    return f < nz ? (const double2*)G.lam + (size_t)(F_A + f) * FS
                  : G.primal + (size_t)(f == nz ? F_ETA : f == nz + 1 ? F_PHI : f == nz + 2 ? F_U : F_V) * FS;
  }, nf, S::N1, JB, B, b, S::J, j0, raw);
  if (threadIdx.x == 0) {
    const double td = G.par[P_TAUDRAG * B + b];
    s_par[0] = G.par[P_PHIBAR * B + b];
    s_par[1] = G.mco[MC_SIITR * B + b];
    s_par[2] = G.mco[MC_ITD * B + b];
    s_par[3] = G.par[P_DPHIEQ * B + b];
    s_nodrag = td == -1.0;
  }
  cp_async_wait_all();
  __syncthreads();
  PhysicsAdj<double> pa;
  pa.Pb = s_par[0]; pa.itr = s_par[1]; pa.itd = s_par[2]; pa.DPe = s_par[3];
  pa.nodrag = s_nodrag != 0; pa.forced = forced;
  constexpr int planeY = ADJ_NF * JB * S::YW, planeZ = ADJ_NZ * JB * S::ZW;
  slice_fourier<S, JB>(raw, nf * JB, nz, D, planeY, ery, s_mid);
  __syncthreads();
  c2r_tiles<S, JB>(mats, D, planeY, ery, s_mid, nf * JB, nz, A);
  __syncthreads();
  double gacc[NGRAD] = {0.0, 0.0, 0.0, 0.0};
  for (int t = threadIdx.x; t < JB * S::I; t += 256) {
    const int i = t % S::I, r = t / S::I, j = j0 + r;
    auto at = [&](int f) { return A[(size_t)(f * JB + r) * S::I + i]; };
    double lz[8], lx[4];
#pragma unroll
    for (int q = 0; q < 8; ++q) lz[q] = q < nz ? at(q) : 0.0;
    if (tied) {
      lz[6] = lz[1];
      lz[7] = -lz[0];
    }
    pa.eval(at(nz), at(nz + 1), at(nz + 2), at(nz + 3), G.g.ihalf[j], G.g.dayc[i] * G.g.coslat[j], lz, lx, gacc);
#pragma unroll
    for (int q = 0; q < 4; ++q) A[(size_t)(q * JB + r) * S::I + i] = lx[q];
  }
  {
    // the warp's sums of the four gradients, halving the values a lane keeps in
    // the first two exchanges: 6 FP64 additions instead of 20
    static_assert(NGRAD == 4, "two halvings");
    const bool hi16 = threadIdx.x & 16, hi8 = threadIdx.x & 8;
    double u[2];
#pragma unroll
    for (int q = 0; q < 2; ++q)
      u[q] = (hi16 ? gacc[q + 2] : gacc[q]) + __shfl_xor_sync(0xffffffffu, hi16 ? gacc[q] : gacc[q + 2], 16);
    double v = (hi8 ? u[1] : u[0]) + __shfl_xor_sync(0xffffffffu, hi8 ? u[0] : u[1], 8);
#pragma unroll
    for (int o = 4; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    if ((threadIdx.x & 7) == 0) s_red[(threadIdx.x >> 5) * NGRAD + (hi16 ? 2 : 0) + (hi8 ? 1 : 0)] = v;
  }
  __syncthreads();
  if (threadIdx.x < NGRAD && G.grad) {
    double acc = 0.0;
    for (int w = 0; w < 8; ++w) acc += s_red[w * NGRAD + threadIdx.x];
    atomicAdd(&G.grad[threadIdx.x * B + b], acc);
  }
  slice_grid<S>(A, ADJ_NZ * JB, D, planeZ, erz, qmid);
  __syncthreads();
  // lambda_y of eta, Phi, U, V: their own lambda plus the transform; delta has no grid part
  auto own = [&](int q, size_t o) {
    const int fy = q == 0 ? F_ETA : q == 1 ? F_DELTA : q == 2 ? F_PHI : q == 3 ? F_U : F_V;
    return (const double*)(G.lam + (size_t)fy * FS + o);
  };
  r2c_tiles<S>(mats, D, planeZ, erz, qmid, ADJ_NZ * JB, 0, 1, [&](int n, int m, int comp, double x) {
    const int q4 = n / JB, q = q4 == 0 ? 0 : q4 + 1;
    const size_t o = ((size_t)m * B + b) * S::J + j0 + n % JB;
    if (!(q >= 3 && cfg.adj_zeroed)) x += own(q, o)[comp];  // lambda of U, V: zero after the sweep's first step
    ((double*)(G.lamy + (size_t)q * FS + o))[comp] = x;
  });
  for (int t = threadIdx.x; t < S::N1 * JB; t += 256) {
    const size_t o = ((size_t)(t / JB) * B + b) * S::J + j0 + t % JB;
    G.lamy[FS + o] = G.lam[(size_t)F_DELTA * FS + o];
  }
}

// ------------------------------------------------------------------- output
// GM_OUTPUT (the physical curr and prev fields of a state or its tangent) and,
// after GM_INIT / GM_TL_INIT, the residual of the initial fields beyond the
// truncation: the same transform as the step's, so that an initial state's
// output is its initial fields and a history row the output of its state, to
// the last bit.
constexpr int OUT_NF = 8;
template <int M_, int JB>
__global__ void __launch_bounds__(256, 2) k_grid_out_f64(const __grid_constant__ GridLaunch<double> Lc,
                                                         const __grid_constant__ SliceBasis basis) {
  typedef Sh<M_> S;
  typedef Mem<S, JB, OUT_NF, 0> Mm;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  double* A = (double*)smem_raw;
  uint32_t* D = (uint32_t*)(smem_raw + Mm::A);
  int* er = (int*)(smem_raw + Mm::A + Mm::B);
  __shared__ double s_mid[OUT_NF * JB];
  int idx;
  const GridGroup<double>& G = pick_ggroup(Lc, idx);
  const StepCfg& cfg = Lc.cfg;
  const int B = G.B, b = idx / (S::J / JB), j0 = (idx % (S::J / JB)) * JB;
  const size_t FS = (size_t)S::N1 * B * S::J, PS = (size_t)B * S::J * S::I;
  const bool out = Lc.mode == GM_OUTPUT;
  const int nf = out ? 8 : 5;
  // eta, delta, Phi, U, V, then the mid levels
  auto field = [](int f) {
    return f == 0 ? F_ETA : f == 1 ? F_DELTA : f == 2 ? F_PHI : f == 3 ? F_U : f == 4 ? F_V
           : f == 5 ? F_ETA_MID : f == 6 ? F_DELTA_MID : F_PHI_MID;
  };
  double2* raw = (double2*)A;
  copy_rows([&](int f) { return G.four + (size_t)field(f) * FS; }, nf, S::N1, JB, B, b, S::J, j0, raw);
  double wc = 0.0, wm = 0.0, wuv = 0.0, dwc = 0.0, dwm = 0.0;
  if (out) {
    wc = G.member ? G.member[MS_WCURR * B + b] : 0.0;
    wm = G.member ? G.member[MS_WMID * B + b] : 0.0;
    const bool stepped = G.member && G.member[MS_UPDATED * B + b] != 0.0;
    wuv = cfg.test == 1 ? 1.0 : stepped ? 0.0 : wc;
    if (G.resid_p && G.dw) {  // tangent output: the weights' own tangents times the primal residual
      dwc = G.dw[b];
      dwm = G.dw[B + b];
    }
  }
  cp_async_wait_all();
  __syncthreads();
  slice_fourier<S, JB>(raw, nf * JB, 0, D, OUT_NF * JB * S::YW, er, s_mid);
  __syncthreads();
  c2r_tiles<S, JB>((const uint4*)basis.p[&G - Lc.grp], D, OUT_NF * JB * S::YW, er, s_mid, nf * JB, 0, A);
  __syncthreads();
  for (int t = threadIdx.x; t < nf * JB * S::I; t += 256) {
    const int i = t % S::I, r = (t / S::I) % JB, f = t / (S::I * JB);
    const size_t at = ((size_t)b * S::J + j0 + r) * S::I + i;
    double v = A[t];
    if (out) {
      const int rf = f < 5 ? f : f - 5;
      const double w = f >= 5 ? wm : f >= 3 ? wuv : wc, dw = f >= 5 ? dwm : f >= 3 ? 0.0 : dwc;
      if (w != 0.0 && G.resid) v += w * G.resid[rf * PS + at];
      if (dw != 0.0 && G.resid) v += dw * G.resid_p[rf * PS + at];
      G.phys_out[f * PS + at] = v;
    } else {
      G.resid[f * PS + at] = G.phys_in[f * PS + at] - v;
    }
  }
}

// Rows per CTA: at most as many as leave two CTAs per SM their shared memory.  Few
// rows for few members: two from 1.5 CTAs of one row per SM on (the two then share
// the SM's FP64 pipe), four from 1.5 rounds of two.  Step (adjoint, at most two), M =
// 42, us with 1 / 2 / 4 rows: 1 member 15 / 17 / 25 (18 / 23), 4 members 18 / 18 / 25
// (23 / 23), 6 members 25 / 25 / 25 (35 / 31), 8 members 29 / 24 / 25 (41 / 32), 12
// members 39 / 35 / 37 (55 / 47), 14 members 39 / 35 / 37 (57 / 47), 16 members 47 / 41 /
// 37 (68 / 53), 20 members 57 / 51 / 54 (84 / 70), 24 members 66 / 55 / 54 (97 / 76), 48
// members 120 / 97 / 89 (181 / 137), 256 members 596 / 438 / 371 (934 / 622); M = 63 with
// 1 / 2: 2 members 23 / 23 (33 / 32), 5 members 39 / 35 (55 / 47), 32 members 181 / 150
// (267 / 209).  (The forms not taken: before the row sums of I/2 were reduced together.)
enum Kind { STEP, ADJ, OUT };
template <int M_, Kind K>
constexpr int max_rows() { return K == OUT ? 1 : K == ADJ ? (M_ == 106 ? 1 : 2) : M_ == 42 ? 4 : M_ == 63 ? 2 : 1; }

template <int M_, int JB, Kind K>
cudaError_t launch_one(GridLaunch<double> L, const SliceBasis& basis, cudaStream_t s) {
  typedef Sh<M_> S;
  int acc = 0;
  for (int g = 0; g < L.ng; ++g) {
    if (L.grp[g].g.M != M_) L.grp[g].B = 0;
    L.grp[g].JB = JB;
    L.grp[g].njb = S::J / JB;
    L.prefix[g] = acc;
    acc += L.grp[g].B * L.grp[g].njb;
  }
  L.prefix[L.ng] = acc;
  if (acc == 0) return cudaSuccess;
  if constexpr (K == ADJ) k_grid_adj_f64<M_, JB><<<acc, 256, Mem<S, JB, ADJ_NF, ADJ_NZ>::total, s>>>(L, basis);
  else if constexpr (K == OUT) k_grid_out_f64<M_, JB><<<acc, 256, Mem<S, JB, OUT_NF, 0>::total, s>>>(L, basis);
  else k_grid_step_f64<M_, JB><<<acc, 256, Mem<S, JB, STEP_NF, STEP_NZ>::total, s>>>(L, basis);
  return cudaGetLastError();
}
template <int M_, Kind K>
cudaError_t launch_trunc(const GridLaunch<double>& L, const SliceBasis& basis, cudaStream_t s) {
  int members = 0;
  for (int g = 0; g < L.ng; ++g)
    if (L.grp[g].g.M == M_) members += L.grp[g].B;
  if (members == 0) return cudaSuccess;
  constexpr int most = max_rows<M_, K>();
  const int rows = members * trunc_J(M_);
  if constexpr (most >= 4)
    if (rows >= 6 * 152) return launch_one<M_, 4, K>(L, basis, s);
  if constexpr (most >= 2)
    if (2 * rows >= 3 * 152) return launch_one<M_, 2, K>(L, basis, s);
  return launch_one<M_, 1, K>(L, basis, s);
}

template <int M_, int JB>
void set_attr() {
  typedef Sh<M_> S;
  if constexpr (JB <= max_rows<M_, STEP>()) {
    constexpr size_t n = Mem<S, JB, STEP_NF, STEP_NZ>::total;
    static_assert(n <= 112 * 1024, "two CTAs per SM");
    cudaFuncSetAttribute(k_grid_step_f64<M_, JB>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)n);
  }
  if constexpr (JB <= max_rows<M_, ADJ>()) {
    constexpr size_t n = Mem<S, JB, ADJ_NF, ADJ_NZ>::total;
    static_assert(n <= 112 * 1024, "two CTAs per SM");
    cudaFuncSetAttribute(k_grid_adj_f64<M_, JB>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)n);
  }
  if constexpr (JB == 1)
    cudaFuncSetAttribute(k_grid_out_f64<M_, 1>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                         (int)Mem<S, 1, OUT_NF, 0>::total);
}

}  // namespace

size_t grid_f64_basis_bytes(int M) {
  return M == 42 ? Pack<Sh<42>>::bytes : M == 63 ? Pack<Sh<63>>::bytes : Pack<Sh<106>>::bytes;
}
cudaError_t pack_grid_f64(int M, void* out, cudaStream_t s) {
  if (M == 42) k_pack_grid<Sh<42>><<<32, 256, 0, s>>>((uint4*)out);
  else if (M == 63) k_pack_grid<Sh<63>><<<32, 256, 0, s>>>((uint4*)out);
  else k_pack_grid<Sh<106>><<<64, 256, 0, s>>>((uint4*)out);
  return cudaGetLastError();
}
void grid_f64_set_attributes() {
  set_attr<42, 1>(); set_attr<42, 2>(); set_attr<42, 4>();
  set_attr<63, 1>(); set_attr<63, 2>();
  set_attr<106, 1>();
}
namespace {
template <Kind K>
cudaError_t launch_all(const GridLaunch<double>& L, const SliceBasis& basis, cudaStream_t s) {
  cudaError_t e = launch_trunc<106, K>(L, basis, s);
  if (e == cudaSuccess) e = launch_trunc<63, K>(L, basis, s);
  if (e == cudaSuccess) e = launch_trunc<42, K>(L, basis, s);
  return e;
}
}  // namespace
// L.mode: GM_STEP, GM_ADJ_STEP or GM_OUTPUT; GM_INIT and GM_TL_INIT: the residuals only
cudaError_t launch_grid_f64(const GridLaunch<double>& L, const SliceBasis& basis, cudaStream_t s) {
  return L.mode == GM_STEP ? launch_all<STEP>(L, basis, s)
         : L.mode == GM_ADJ_STEP ? launch_all<ADJ>(L, basis, s) : launch_all<OUT>(L, basis, s);
}

}  // namespace swp

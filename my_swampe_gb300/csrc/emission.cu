// Emission stage of the retrieval, batched over ensemble members, in FP64 like
// the reference (whose emission / light-curve stage stays float64 even when the
// dynamics run in float32).  It maps a member's terminal Phi to the
// spherical-harmonic coefficients of its emission map and to a phase curve:
//
//   phi_to_temperature            retrieval/scripts/pipeline.py:696-714
//   temperature_to_intensity      pipeline.py:716-754 (bolometric T^4, or the
//                                 relative Planck intensity, optionally band-averaged)
//   intensity_map_to_y_dense      pipeline.py:821-846 (weighted ridge least-squares
//                                 projection onto the Ylm basis, normalised by y0)
//   the planet's light curve      pipeline.py:983-994: linear in the map
//                                 coefficients, amplitude planet_fpfs
//   the simplified phase curve    unit_tests/test_parity_reference_regression.py:67-82
//
// The Ylm design matrix and the light-curve design matrix come from a
// third-party model (jaxoplanet 0.1.0, starry Surface.intensity and
// light_curve) that the caller evaluates once; the projector built from the
// former is an input here, as in the reference, which builds it once per
// pipeline (pipeline.py:808-819).
//
// Every kernel's reductions run in a fixed order, so results are reproducible
// run to run.  Non-finite inputs give all-NaN outputs per member, as the
// reference's lax.cond guards do.
#include <cmath>
#include <type_traits>
#include <cooperative_groups.h>
#include "slices.cuh"
#include "swp_internal.h"

namespace swp {
namespace {

namespace cg = cooperative_groups;

constexpr int EM_THREADS = 256;
constexpr int EM_WARPS = EM_THREADS / 32;
// The map and the simple phase curve run one cluster of EM_CL CTAs per member,
// whatever the ensemble's size: a member's FP64 work (two divisions, expm1 and
// a reciprocal per pixel; GB300 retires 1.7 FP64 instructions per cycle and SM)
// then spreads over 8 SMs, and its sums run in one fixed order (lanes, warps,
// ranks), so that ensembles equal single-member calls bit for bit.
constexpr int EM_CL = 8;

__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// Sums of two values and the conjunction of a flag over the cluster's threads.
// Warp sums go to this CTA's slots; each warp slot of each rank is then added
// in rank and warp order by every thread.  `slot` is 3 * EM_WARPS doubles of
// shared memory per call (a slot is not reused: no barrier after the reads).
struct ClusterSum {
  double a, b;
  bool all;
};
__device__ ClusterSum cluster_sum(double a, double b, bool ok, double* slot) {
  cg::cluster_group cl = cg::this_cluster();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  a = warp_sum(a);
  b = warp_sum(b);
  const bool wok = __all_sync(0xffffffffu, ok) != 0;
  if (lane == 0) {
    slot[warp] = a;
    slot[EM_WARPS + warp] = b;
    slot[2 * EM_WARPS + warp] = wok ? 0.0 : 1.0;
  }
  cl.sync();
  // lane l reads warp slots l and l + 32 of the 64 (8 ranks x 8 warps)
  double va = 0.0, vb = 0.0, bad = 0.0;
#pragma unroll
  for (int h = 0; h < EM_CL * EM_WARPS / 32; ++h) {
    const int s = lane + 32 * h;
    const double* r = cl.map_shared_rank(slot, s / EM_WARPS);
    va += r[s % EM_WARPS];
    vb += r[EM_WARPS + s % EM_WARPS];
    bad += r[2 * EM_WARPS + s % EM_WARPS];
  }
  ClusterSum t;
  t.a = warp_sum(va);
  t.b = warp_sum(vb);
  t.all = __all_sync(0xffffffffu, bad == 0.0) != 0;
  return t;
}

constexpr int EXP_N = 64;  // steps of 2^(j / 64) in the table of planck_rel

struct EmCfg {
  int temp_mode, model, nbands, input;  // input: 0 = Phi, 1 = T, 2 = intensity
  double R_d, T_ref, phi_to_T_scale, Tmin, x_clip;
  // Planck bands: x = pl[k] / max(p0 + v, pmin), the argument h c / (lambda kB T)
  // with the scale of T folded into pl, p0 and pmin (p0 null for Phibar); see
  // planck_bands
  double pl[SWP_EMISSION_MAX_BANDS], bw[SWP_EMISSION_MAX_BANDS];
  double p0, pmin;
  int folded;  // scale >= 1: T need not be formed
  double tm1[EXP_N];  // 2^(j / 64) - 1
};

__device__ __forceinline__ bool finite_bits(double v) { return (__double2hiint(v) & 0x7ff00000) != 0x7ff00000; }

__device__ __forceinline__ double temperature(const EmCfg& c, double phi, double Phibar) {
  const double T = c.temp_mode == 0 ? (Phibar + phi) / c.R_d : c.T_ref + phi / c.phi_to_T_scale;
  return fmax(T, c.Tmin);
}
// relative Planck intensity 1 / (expm1(x) + tiny) at x in [0, 700]
// (pipeline.py:716-735).  expm1 by table-driven reduction (Tang, ACM TOMS 15,
// 1989): x = n ln2 / 64 + r, 2^(n/64) = 2^e (1 + tm1[j]),
//   expm1(x) = 2^e (1 + tm1) p + (2^e tm1 + (2^e - 1)),  p = expm1(r), |r| <= ln2 / 128,
// with p's Taylor polynomial to r^6, whose next term is below 2^-57 p (for x below
// ln2 / 128, n = 0, p is the result itself).  The table holds tm1 and 1 + tm1, whose
// exponent is raised in integers.  12 FP64 instructions, where the library call took
// about 40 of the map's 100 a pixel.
__device__ __forceinline__ double planck_rel(double x, const double2* __restrict__ tab) {
  const double magic = 6755399441055744.0;  // 1.5 * 2^52: rounds to an integer in the low word
  const double t = fma(x, 92.332482616893656877, magic);  // 64 / ln 2
  const int n = __double2loint(t);
  const double fn = t - magic;
  // ln2 / 64 as a 33-bit head (n < 2^17: the products are exact) and a tail
  double r = fma(fn, -0x1.62e42feep-7, x);
  r = fma(fn, -0x1.a39ef35793c76p-39, r);
  const double r2 = r * r;
  double p = fma(fma(r, 1.0 / 720.0, 1.0 / 120.0), r2, fma(r, 1.0 / 24.0, 1.0 / 6.0));
  p = fma(fma(p, r, 0.5), r2, r);
  const double e2 = __hiloint2double((1023 + (n >> 6)) << 20, 0);
  const double2 t1 = tab[n & (EXP_N - 1)];
  const double q = fma(e2, t1.x, e2 - 1.0);
  const double s = __hiloint2double(__double2hiint(t1.y) + ((n >> 6) << 20), __double2loint(t1.y));
  return 1.0 / (fma(s, p, q) + 1.0e-30);
}
// v: Phi, or T (c.input 1).  ANY_X: x_clip is outside planck_rel's range
template <bool ANY_X>
__device__ __forceinline__ double planck_bands(const EmCfg& c, double v, double Phibar,
                                               const double2* __restrict__ tab) {
  const double p0 = c.input == 0 && c.temp_mode == 0 ? Phibar : c.p0;
  const double u = c.input != 0 ? v : c.folded ? fmax(p0 + v, c.pmin) : temperature(c, v, Phibar);
  double out = 0.0;
  for (int k = 0; k < c.nbands; ++k) {
    const double x = fmin(fmax(c.pl[k] / u, 0.0), c.x_clip);
    out += c.bw[k] * (ANY_X ? 1.0 / (expm1(x) + 1.0e-30) : planck_rel(x, tab));
  }
  return out;
}

// One cluster per member, a warp per latitude row.  stage 0 writes T, 1 the
// intensity map, 2 the weighted relative intensity w_sqrt I / I_mean that the
// projector multiplies (and ok[b] = the map's guards passed).  The passes
// follow the reference's guards: a non-finite Phi makes T all NaN; a non-finite
// T makes the Planck intensity all NaN; the relative map needs a finite,
// nonzero weighted mean.
//
// FP64-bound (see EM_CL).  The Planck argument takes one division (T itself is
// not formed), finiteness is tested on the exponent bits, the square root of a
// weight is taken once per row, with the quotient by the mean folded into it.
template <bool ANY_X>
__global__ void __cluster_dims__(EM_CL, 1, 1) __launch_bounds__(EM_THREADS)
    k_emission_map(const double* __restrict__ in, const double* __restrict__ Phibar, int J, int I,
                   const double* __restrict__ w_lat, const __grid_constant__ EmCfg c, int stage,
                   double* __restrict__ out, int* __restrict__ ok) {
  __shared__ double slots[2][3 * EM_WARPS];
  __shared__ double2 tab[EXP_N];
  cg::cluster_group cl = cg::this_cluster();
  const int rank = (int)cl.block_rank(), b = blockIdx.x / EM_CL;
  const int lane = threadIdx.x & 31;
  const int row0 = rank * EM_WARPS + (threadIdx.x >> 5);
  constexpr int ROWS = EM_CL * EM_WARPS;
  const size_t npix = (size_t)J * I;
  const double* x = in + (size_t)b * npix;
  double* y = out + (size_t)b * npix;
  const double pb = Phibar ? Phibar[b] : 0.0;
  const double qnan = __longlong_as_double(0x7ff8000000000000ll);
  if (threadIdx.x < EXP_N) tab[threadIdx.x] = make_double2(c.tm1[threadIdx.x], 1.0 + c.tm1[threadIdx.x]);
  // pass 1: all of the input finite (Phi -> T guard) and, with the Planck
  // model, all of T finite
  bool nan_map = false;
  if (c.input == 0 || (c.input == 1 && c.model == 1)) {
    bool fin = true;
    const double p0 = c.temp_mode == 0 ? pb : c.p0;
    for (int j = row0; j < J; j += ROWS)
      for (int i = lane; i < I; i += 32) {
        const double v = x[(size_t)j * I + i];
        fin &= finite_bits(v);
        if (c.input == 0 && c.model == 1 && stage > 0) fin &= finite_bits(c.folded ? p0 + v : temperature(c, v, pb));
      }
    nan_map = !cluster_sum(0.0, 0.0, fin, slots[0]).all;
  } else {
    cl.sync();  // the table, and every rank running before the remote reads below
  }
  // pass 2: T, or the intensity and, for stage 2, its weighted mean over the
  // finite pixels (pipeline.py:821-837)
  double sw = 0.0, swi = 0.0;
  bool fi = true;
  for (int j = row0; j < J; j += ROWS) {
    const double w = stage == 2 ? w_lat[j] : 0.0;
    for (int i = lane; i < I; i += 32) {
      const size_t p = (size_t)j * I + i;
      double v = x[p];
      if (nan_map) {
        v = qnan;
      } else if (c.input < 2) {
        if (stage > 0 && c.model == 1) {
          v = planck_bands<ANY_X>(c, v, pb, tab);
        } else {
          if (c.input == 0) v = temperature(c, v, pb);
          if (stage > 0) {
            v *= v;
            v *= v;
          }
        }
      }
      y[p] = v;
      if (stage == 2) {
        const bool f = finite_bits(v);
        fi &= f;
        if (f) {
          sw += w;
          swi += w * v;
        }
      }
    }
  }
  if (stage < 2) {
    cl.sync();  // a peer may still read this CTA's slots
    return;
  }
  const ClusterSum s = cluster_sum(sw, swi, fi, slots[1]);
  const double mean = s.a > 0.0 ? s.b / s.a : qnan;
  const bool mean_ok = isfinite(mean) && fabs(mean) > 1.0e-30;
  // pass 3: rhs = sqrt(w) * I_rel, I_rel = I / mean (NaN where the mean fails, 0 where I is not finite)
  for (int j = row0; j < J; j += ROWS) {
    const double q = mean_ok ? sqrt(w_lat[j]) / mean : qnan;
    for (int i = lane; i < I; i += 32) {
      const size_t p = (size_t)j * I + i;
      const double v = y[p];
      y[p] = finite_bits(v) ? q * v : q * 0.0;
    }
  }
  if (rank == 0 && threadIdx.x == 0 && ok) ok[b] = (s.all && mean_ok) ? 1 : 0;
  cl.sync();
}

// Y[b][c] = sum_p P[c][p] rhs[b][p] on the FP16 tensor cores (slices.cuh): a
// cluster of EM_CL CTAs takes 16 members and PR_COEF (32 or 64) coefficients, each
// CTA an eighth of the pixels, 64 at a time (cp.async, double-buffered).  A warp owns 16
// coefficients and half of a chunk: it slices its projector rows in registers,
// in the fragment layout; the members' rows are sliced into shared memory by
// all threads.  A row's scale is the largest exponent it has shown so far: a
// chunk that raises it first converts the sums on the old scale, which happens
// a few times per row, so nearly all sums stay in integers.  The partial results
// are added in a fixed order, and neither they nor the scales of a member depend
// on the other members of its tile.
//
// The slices' error is a part of the product of the rows' scales, below npix 2^-59
// of it, and not of what the products add up to: a coefficient whose row is
// non-zero only where the map is faint (a sector, the night side, a patch) could
// lose every digit.  So the products of the top digits' magnitudes are summed
// beside the result (a 37th MMA a step): each is at most four times the product of
// the elements' magnitudes, and where their sum does not reach PR_GUARD, so that
// sum |P r| is not shown to reach the product of the scales, the output is taken
// again with FP64 FMAs (a warp, lanes over pixels), as is any whose scales are near
// the ends of FP64's range, infinite or NaN.  An output of slices is then within
// npix 2^-59 sum |P r| and its roundings, one of FMAs within npix / 32 2^-53
// sum |P r|.  Of the sums over a whole disc, which the guard leaves alone, none
// comes near it.
//
// FP64 FMAs took 475 us for 256 members (M = 42, 121 coefficients), 96% of the
// FP64 pipe.  At most 64 coefficients a CTA, for two CTAs per SM.
constexpr int PR_MEMB = 16, PR_KC = 64;        // members, pixels per chunk
constexpr int PR_KMAX = 8192;                  // pixels of a CTA per forced conversion (integer range of the sums)
constexpr int PR_ROW = PR_KC / 2 + 4;          // words of a sliced member row, padded: conflict-free B fragments
constexpr int PR_LD = PR_KC + 8;               // doubles of a staged row, padded: conflict-free A fragments
constexpr float PR_GUARD = 32768.0f;  // top-digit products: 2^-2 of it in units of 2^112 reaches 2^124, a scale's square
template <int PR_COEF>
struct ProjectSmem {
  union {
    double stage[2][PR_COEF + PR_MEMB][PR_LD];  // coefficients, then members
    struct {  // the halves' results, once the last chunk is read
      double part[2][PR_COEF][PR_MEMB + 1];
      float mag[2][PR_COEF][PR_MEMB + 1];  // sums of the top digits' magnitudes
      int ec[2][PR_COEF];                  // coefficient scales
      int2 ms[PR_COEF][PR_MEMB + 1];       // both halves' magnitudes (FP32 bits) and their scale
      int again[PR_COEF * PR_MEMB / EM_CL], nagain;  // outputs below the guard (static memory for them: 2 us more)
    };
  };
  uint32_t dig[slices::ND][PR_MEMB][PR_ROW];
  int er[2][PR_MEMB];  // member scales: current, and before this chunk
};
// 2^-n, n >= 0; zero beyond FP32's normal range
__device__ __forceinline__ float pow2_down(int n) { return __int_as_float(max(127 - n, 0) << 23); }
// VEC: 16-byte copies (every row starts on 16 bytes)
template <bool VEC, int PR_COEF>
__global__ void __cluster_dims__(EM_CL, 1, 1) __launch_bounds__(EM_THREADS, 2)
    k_emission_project(const double* __restrict__ rhs, int B, int npix, const double* __restrict__ P, int ncoef,
                       double* __restrict__ yraw) {
  using namespace slices;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  constexpr int PR_ROWS = PR_COEF + PR_MEMB, NMT = PR_COEF / 16;  // staged rows; coefficient tiles
  typedef ProjectSmem<PR_COEF> Smem;
  Smem& S = *reinterpret_cast<Smem*>(smem_raw);
  cg::cluster_group cl = cg::this_cluster();
  const int rank = (int)cl.block_rank();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  const int mt = warp % NMT, half = (warp / NMT) & 1;  // warps from 2 NMT on only stage and slice members
  const int c0 = (blockIdx.x / EM_CL) * PR_COEF, b0 = blockIdx.y * PR_MEMB;
  const int nm = min(PR_MEMB, B - b0), nn = nm > 8 ? 2 : 1;
  // this CTA's pixels: a multiple of the chunk but for the last
  const int per = ((npix + EM_CL * PR_KC - 1) / (EM_CL * PR_KC)) * PR_KC;
  const int k0 = min(rank * per, npix), k1 = min(k0 + per, npix);
  const bool busy = warp < 2 * NMT && c0 + mt * 16 < ncoef;
  // rows beyond the last coefficient or member, and pixels beyond the end, are zero
  constexpr int STEP = VEC ? 2 : 1, NS = PR_KC / STEP;  // a thread copies the same pixels of every EM_THREADS / NS rows
  const int sk = (threadIdx.x % NS) * STEP;
  auto stage = [&](int buf, int kc) {
#pragma unroll 4
    for (int r = threadIdx.x / NS; r < PR_ROWS; r += EM_THREADS / NS) {
      double* dst = &S.stage[buf][r][sk];
      const int row = r < PR_COEF ? c0 + r : b0 + r - PR_COEF;
      const bool on = kc + sk < k1 && row < (r < PR_COEF ? ncoef : B);
      if (on) {
        cp_async<8 * STEP>(dst, (r < PR_COEF ? P : rhs) + (size_t)row * npix + kc + sk);
      } else {
        dst[0] = 0.0;
        if (VEC) dst[1] = 0.0;
      }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  int ea[2] = {0, 0};
  double res[2][4] = {};
  Tile tile[2];
  tile[0].reset();
  tile[1].reset();
  float mag[2][4] = {};
  if (threadIdx.x < PR_MEMB) S.er[0][threadIdx.x] = S.er[1][threadIdx.x] = 0;
  stage(0, k0);
  int buf = 0;
  for (int kc = k0; kc < k1; kc += PR_KC, buf ^= 1) {
    const bool force = (kc - k0) % PR_KMAX == 0;
    stage(buf ^ 1, kc + PR_KC);
    asm volatile("cp.async.wait_group 1;" ::: "memory");
    __syncthreads();
    // members: scale and slices, a warp per two rows, a lane per pixel pair
    for (int r = warp; r < PR_MEMB; r += EM_WARPS) {
      const double2 x = *(const double2*)&S.stage[buf][PR_COEF + r][2 * lane];
      const int e0 = S.er[0][r];
      const int e = max(e0, row_exponent((int)__reduce_max_sync(0xffffffffu, (unsigned)max(expo(x.x), expo(x.y)))));
      __syncwarp();
      if (lane == 0) {
        S.er[1][r] = e0;
        S.er[0][r] = e;
      }
      store_digits(&S.dig[0][r][lane], PR_MEMB * PR_ROW, fixed(x.x, e), fixed(x.y, e));
    }
    // projector rows g, g + 8 of the warp's 16, its half of the chunk: lanes t over pixels
    int en[2];
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int2* row = (const int2*)&S.stage[buf][mt * 16 + g + 8 * h][32 * half];
      unsigned m = 0;
#pragma unroll
      for (int i = 0; i < 8; ++i) m = max(m, (unsigned)row[t + 4 * i].y & 0x7fffffffu);
      m = max(m, __shfl_xor_sync(0xffffffffu, m, 1));
      m = max(m, __shfl_xor_sync(0xffffffffu, m, 2));
      en[h] = max(ea[h], row_exponent((int)(m >> 20)));
    }
    __syncthreads();
    // sums whose row or member scale rises (or that reach the integers' range) are converted first
    if (kc > k0) {
#pragma unroll
      for (int n = 0; n < 2; ++n)
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const int c = 8 * n + 2 * t + (e & 1), h = e >> 1;
          const int rise = en[h] - ea[h] + S.er[0][c] - S.er[1][c];
          if (force || en[h] != ea[h] || S.er[0][c] != S.er[1][c]) {
            res[n][e] += value(tile[n].hi[e], tile[n].lo[e], ea[h], S.er[1][c]);
            tile[n].hi[e] = tile[n].lo[e] = 0;
            mag[n][e] *= pow2_down(rise);  // to the new scales
          }
        }
    }
    ea[0] = en[0];
    ea[1] = en[1];
    if (busy) {
#pragma unroll
      for (int ks = 0; ks < KFLUSH; ++ks) {
        uint32_t a[ND][4], bf[ND][2];
#pragma unroll
        for (int q = 0; q < 4; ++q) {  // fragment registers: (row g + 8 (q & 1), k 2 t + 8 (q >> 1) and + 1)
          const int h = q & 1;
          const double2 x =
              *(const double2*)&S.stage[buf][mt * 16 + g + 8 * h][32 * half + 16 * ks + 2 * t + 8 * (q >> 1)];
          const uint64_t u = fixed(x.x, ea[h]), v = fixed(x.y, ea[h]);
          a[0][q] = digit_pair<0>(u, v);
          a[1][q] = digit_pair<1>(u, v);
          a[2][q] = digit_pair<2>(u, v);
          a[3][q] = digit_pair<3>(u, v);
          a[4][q] = digit_pair<4>(u, v);
          a[5][q] = digit_pair<5>(u, v);
          a[6][q] = digit_pair<6>(u, v);
          a[7][q] = digit_pair<7>(u, v);
        }
#pragma unroll
        for (int n = 0; n < 2; ++n) {
          if (n >= nn) break;
          const uint32_t* bp = &S.dig[0][8 * n + g][16 * half + 8 * ks + t];
          load_b(bf, bp, bp + 4, PR_MEMB * PR_ROW);
          tile[n].step(a, bf);
          uint32_t am[4], bm[2];
#pragma unroll
          for (int q = 0; q < 4; ++q) am[q] = a[0][q] & 0x7fff7fffu;
#pragma unroll
          for (int q = 0; q < 2; ++q) bm[q] = bf[0][q] & 0x7fff7fffu;
          mma(mag[n], am, bm);
        }
      }
      tile[0].flush();
      if (nn > 1) tile[1].flush();
    }
    __syncthreads();  // the buffer and the slices are read
  }
  asm volatile("cp.async.wait_all;" ::: "memory");
#pragma unroll
  for (int n = 0; n < 2; ++n) {
    if (warp >= 2 * NMT) break;
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const int c = 8 * n + 2 * t + (e & 1);
      if (k1 > k0) res[n][e] += value(tile[n].hi[e], tile[n].lo[e], ea[e >> 1], S.er[0][c]);
      S.part[half][mt * 16 + g + 8 * (e >> 1)][c] = res[n][e];
      S.mag[half][mt * 16 + g + 8 * (e >> 1)][c] = mag[n][e];
    }
  }
  if (t == 0 && warp < 2 * NMT) {
    S.ec[half][mt * 16 + g] = ea[0];
    S.ec[half][mt * 16 + g + 8] = ea[1];
  }
  __syncthreads();
  // the halves together: sums, and the magnitudes on the larger of their scales
  for (int i = threadIdx.x; i < PR_COEF * PR_MEMB; i += EM_THREADS) {
    const int c = i / PR_MEMB, r = i % PR_MEMB, e0 = S.ec[0][c], e1 = S.ec[1][c], e = max(e0, e1);
    S.part[0][c][r] += S.part[1][c][r];
    S.ms[c][r] = make_int2(
        __float_as_int(S.mag[0][c][r] * pow2_down(e - e0) + S.mag[1][c][r] * pow2_down(e - e1)), S.er[0][r] + e);
  }
  cl.sync();
  // every eighth coefficient per rank: the sum over ranks, in order
  static_assert(PR_COEF * PR_MEMB / EM_CL <= EM_THREADS, "an output per thread");
  bool again = false;
  const int c = rank + EM_CL * (threadIdx.x / PR_MEMB), r = threadIdx.x % PR_MEMB;
  if (threadIdx.x < PR_COEF * PR_MEMB / EM_CL) {
    double s = 0.0;
    int2 ms[EM_CL];
    int top = 0;
    float m = 0.0f;
#pragma unroll
    for (int q = 0; q < EM_CL; ++q) {
      const Smem* p = cl.map_shared_rank(&S, q);
      s += p->part[0][c][r];
      ms[q] = p->ms[c][r];
      top = max(top, ms[q].y);
    }
#pragma unroll
    for (int q = 0; q < EM_CL; ++q) m += __int_as_float(ms[q].x) * pow2_down(top - ms[q].y);
    const bool out = c0 + c < ncoef && r < nm;
    // scales within 2^1200 and 2^3000: no partial sum was cut off at either end (value())
    again = out && !(m >= PR_GUARD && top >= 1200 && top <= 3000);
    if (out && !again) yraw[(size_t)(b0 + r) * ncoef + c0 + c] = s;
  }
  // the outputs below the guard, spread over the CTA's warps
  if (threadIdx.x == 0) S.nagain = 0;
  __syncthreads();
  if (again) S.again[atomicAdd(&S.nagain, 1)] = (c0 + c) * PR_MEMB + r;
  __syncthreads();
  for (int i = warp; i < S.nagain; i += EM_WARPS) {
    const int cc = S.again[i] / PR_MEMB, bb = b0 + S.again[i] % PR_MEMB;
    const double *x = rhs + (size_t)bb * npix, *w = P + (size_t)cc * npix;
    double s = 0.0;
#pragma unroll 8
    for (int p = lane; p < npix; p += 32) s = fma(w[p], x[p], s);
    s = warp_sum(s);
    if (lane == 0) yraw[(size_t)bb * ncoef + cc] = s;
  }
  cl.sync();
}

// y / y0 with the reference's guards (pipeline.py:838-846): one warp per member.
__global__ void k_emission_normalise(const int* __restrict__ ok, int B, int ncoef, double* __restrict__ y) {
  const int b = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (b >= B) return;
  double* v = y + (size_t)b * ncoef;
  const double qnan = __longlong_as_double(0x7ff8000000000000ll);
  const double y0 = v[0];
  const bool y0_ok = isfinite(y0) && fabs(y0) > 1.0e-30;
  __syncwarp();
  bool fin = true;
  for (int c = lane; c < ncoef; c += 32) {
    const double q = y0_ok ? v[c] / y0 : qnan;
    fin &= finite_bits(q);
    v[c] = q;  // y0 is in a register of every lane
  }
  fin = __all_sync(0xffffffffu, fin);
  if (!((ok ? ok[b] != 0 : true) && y0_ok && fin))
    for (int c = lane; c < ncoef; c += 32) v[c] = qnan;
}

// lc[b][t] = amplitude[b] * sum_c A[t][c] y[b][c]
__global__ void k_phase_curve_linear(const double* __restrict__ y, const double* __restrict__ A,
                                     const double* __restrict__ amp, int B, int ncoef, int ntimes,
                                     double* __restrict__ lc) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= B * ntimes) return;
  const int b = i / ntimes, t = i % ntimes;
  const double* yv = y + (size_t)b * ncoef;
  const double* a = A + (size_t)t * ncoef;
  double s = 0.0;
  for (int c = 0; c < ncoef; ++c) s = fma(a[c], yv[c], s);
  lc[i] = (amp ? amp[b] : 1.0) * s;
}

// flux[b][k] = sum_{j,i} Phi max(cos(lambda_i - phase_k), 0) sqrt(1 - mu_j^2),
// then divided by mean_k |flux| when that is positive: one cluster per member.
// The sum over latitudes does not depend on the phase, so each rank first forms
// the columns s_i = sum_j Phi_ij sqrt(1 - mu_j^2) of its share of a block of
// PC_BLOCK longitudes, with cos and sin of those longitudes, and hands them to
// every rank; a warp then takes a phase and its lanes the longitudes, with
// cos(lambda - phase) by the addition theorem.  One cosine per longitude and
// per phase in the place of one per (pixel, phase): 8.0 ms before for one M = 42
// map and 100 phases, FP64-bound on one SM.
constexpr int PC_BLOCK = 512;
__global__ void __cluster_dims__(EM_CL, 1, 1) __launch_bounds__(EM_THREADS)
    k_phase_curve_simple(const double* __restrict__ phi, int J, int I, const double* __restrict__ mus,
                         const double* __restrict__ phases, int nph, double* __restrict__ flux) {
  __shared__ double col[3][PC_BLOCK];      // s_i, cos(lambda_i), sin(lambda_i) of the block
  __shared__ double part[EM_THREADS];      // column partial sums of each row group
  __shared__ double trig[2][32];           // cos, sin of this CTA's next 32 phases
  __shared__ double slots[3 * EM_WARPS];
  cg::cluster_group cl = cg::this_cluster();
  const int rank = (int)cl.block_rank(), b = blockIdx.x / EM_CL;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const double* x = phi + (size_t)b * J * I;
  double* f = flux + (size_t)b * nph;
  const double pi = 3.141592653589793, step = (pi - (-pi)) / I;  // numpy linspace(-pi, pi, I, endpoint=False)
  for (int i0 = 0; i0 < I; i0 += PC_BLOCK) {
    const int nb = min(PC_BLOCK, I - i0), share = (nb + EM_CL - 1) / EM_CL;
    const int c0 = rank * share, nc = max(0, min(share, nb - c0));
    const int ng = EM_THREADS / share;  // row groups (share <= 64: at least 4)
    const int g = threadIdx.x / share, cc = threadIdx.x % share;
    double s = 0.0;
    if (g < ng && cc < nc)
      for (int j = g; j < J; j += ng) {
        const double mu = mus[j];
        s = fma(x[(size_t)j * I + i0 + c0 + cc], sqrt(fmax(1.0 - mu * mu, 0.0)), s);
      }
    part[threadIdx.x] = s;
    double sl = 0.0, cs = 0.0;
    if (threadIdx.x < nc) sincos(-pi + (i0 + c0 + (int)threadIdx.x) * step, &sl, &cs);
    cl.sync();  // part is complete; every rank is done with the previous block's columns
    if (threadIdx.x < nc) {
      double t = 0.0;
      for (int q = 0; q < ng; ++q) t += part[q * share + threadIdx.x];
      for (int r = 0; r < EM_CL; ++r) {
        double* dst = cl.map_shared_rank(&col[0][0], r) + c0 + threadIdx.x;
        dst[0] = t;
        dst[PC_BLOCK] = cs;
        dst[2 * PC_BLOCK] = sl;
      }
    }
    cl.sync();
    // this rank's phases k = rank + 8 q, 32 at a time: their sines and cosines
    // by one warp, then a warp per phase
    for (int q0 = 0; rank + EM_CL * q0 < nph; q0 += 32) {
      __syncthreads();
      if (warp == 0) {
        const int k = rank + EM_CL * (q0 + lane);
        double sp = 0.0, cp = 0.0;
        if (k < nph) sincos(phases[k], &sp, &cp);
        trig[0][lane] = cp;
        trig[1][lane] = sp;
      }
      __syncthreads();
      for (int q = warp; q < 32; q += EM_WARPS) {
        const int k = rank + EM_CL * (q0 + q);
        if (k >= nph) break;
        const double cp = trig[0][q], sp = trig[1][q];
        double t = 0.0;
        for (int i = lane; i < nb; i += 32)
          t = fma(col[0][i], fmax(fma(col[1][i], cp, col[2][i] * sp), 0.0), t);
        t = warp_sum(t);
        if (lane == 0) f[k] = i0 == 0 ? t : f[k] + t;
      }
    }
  }
  // the mean of |flux| and the division, by the thread that wrote each value
  double asum = 0.0;
  for (int q = warp; rank + EM_CL * q < nph; q += EM_WARPS)
    if (lane == 0) asum += fabs(f[rank + EM_CL * q]);
  const double norm = cluster_sum(asum, 0.0, true, slots).a / nph;
  if (norm > 0.0 && lane == 0)
    for (int q = warp; rank + EM_CL * q < nph; q += EM_WARPS) f[rank + EM_CL * q] /= norm;
  cl.sync();  // a peer may still read this CTA's slots
}

int em_check(cudaError_t e) { return e == cudaSuccess ? SWP_OK : SWP_ERR_CUDA; }

}  // namespace
}  // namespace swp

using namespace swp;

extern "C" int swp_emission_map(const double* in, const double* Phibar, int B, int J, int I, const double* w_lat,
                                const swp_emission_cfg* cfg, int input, int stage, double* out, int* ok,
                                void* stream) {
  if (!in || !cfg || !out || B < 1 || J < 1 || I < 1 || stage < 0 || stage > 2 || input < 0 || input > 2)
    return SWP_ERR_ARG;
  if (input > stage) return SWP_ERR_ARG;                 // the stage is computed from an earlier one
  if (input == 0 && !Phibar && cfg->temp_mode == 0) return SWP_ERR_ARG;
  if (stage == 2 && !w_lat) return SWP_ERR_ARG;
  if (cfg->temp_mode < 0 || cfg->temp_mode > 1 || cfg->model < 0 || cfg->model > 1) return SWP_ERR_ARG;
  if (cfg->model == 1 && (cfg->nbands < 1 || cfg->nbands > SWP_EMISSION_MAX_BANDS)) return SWP_ERR_ARG;
  EmCfg c;
  c.temp_mode = cfg->temp_mode;
  c.model = cfg->model;
  c.nbands = cfg->model == 1 ? cfg->nbands : 0;
  c.input = input;
  c.R_d = cfg->R_d;
  c.T_ref = cfg->T_ref;
  c.phi_to_T_scale = cfg->phi_to_T_scale;
  c.Tmin = cfg->Tmin;
  // T = (p0 + Phi) / scale: with scale >= 1 (so that T is finite where p0 + Phi
  // is) the Planck argument needs no T of its own.  Formed in long double and
  // rounded once.
  const long double hck = 6.62607015e-34L * 299792458.0L / 1.380649e-23L;
  const double div = cfg->temp_mode == 0 ? cfg->R_d : cfg->phi_to_T_scale;
  c.folded = input == 0 && div >= 1.0;
  const long double scale = c.folded ? div : 1.0L;
  c.x_clip = cfg->x_clip;
  c.p0 = c.folded && cfg->temp_mode == 1 ? (double)(cfg->T_ref * scale) : 0.0;
  c.pmin = (double)(cfg->Tmin * scale);
  for (int k = 0; k < SWP_EMISSION_MAX_BANDS; ++k) {
    c.pl[k] = k < c.nbands ? (double)(hck * scale / cfg->wavelengths[k]) : 1.0;
    c.bw[k] = k < c.nbands ? cfg->band_weights[k] : 0.0;
  }
  for (int j = 0; j < EXP_N; ++j) c.tm1[j] = (double)(exp2l((long double)j / EXP_N) - 1.0L);
  auto kernel = cfg->x_clip >= 0.0 && cfg->x_clip <= 700.0 ? k_emission_map<false> : k_emission_map<true>;
  kernel<<<EM_CL * B, EM_THREADS, 0, (cudaStream_t)stream>>>(in, Phibar, J, I, w_lat, c, stage, out, ok);
  return em_check(cudaGetLastError());
}

extern "C" int swp_emission_project(const double* rhs, const int* ok, int B, int npix, const double* projector,
                                    int ncoef, double* y, void* stream) {
  if (!rhs || !projector || !y || B < 1 || npix < 1 || ncoef < 1 || B > 65535) return SWP_ERR_ARG;
  cudaStream_t s = (cudaStream_t)stream;
  const bool vec = npix % 2 == 0 && ((uintptr_t)rhs | (uintptr_t)projector) % 16 == 0;
  auto run = [&](auto vk, auto ck) {
    constexpr int COEF = decltype(ck)::value;
    auto kernel = k_emission_project<decltype(vk)::value, COEF>;
    const dim3 grid(EM_CL * ((ncoef + COEF - 1) / COEF), (B + PR_MEMB - 1) / PR_MEMB);
    cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(ProjectSmem<COEF>));
    if (e != cudaSuccess) return e;
    kernel<<<grid, EM_THREADS, sizeof(ProjectSmem<COEF>), s>>>(rhs, B, npix, projector, ncoef, y);
    return cudaGetLastError();
  };
  // 32 coefficients per CTA while those CTAs fit two per SM at once: a small ensemble's
  // chain per chunk is shorter by half the MMAs and the slicing.  121 coefficients, M = 42,
  // us with 64 / 32: 1 member 90 / 59, 16 members 105 / 71 (FP64 FMAs 82 and 86), 48
  // members 105 / 72, 64 members 106 / 98, 128 members 150 / 102, 256 members 148 / 194;
  // 36 coefficients, 256 members 141 / 98.
  const long long small = (long long)EM_CL * ((ncoef + 31) / 32) * ((B + PR_MEMB - 1) / PR_MEMB);
  auto by_coef = [&](auto vk) {
    return small <= 2 * 152 ? run(vk, std::integral_constant<int, 32>()) : run(vk, std::integral_constant<int, 64>());
  };
  const cudaError_t e = vec ? by_coef(std::true_type()) : by_coef(std::false_type());
  if (e != cudaSuccess) return em_check(e);
  k_emission_normalise<<<(B + 7) / 8, 256, 0, s>>>(ok, B, ncoef, y);
  return em_check(cudaGetLastError());
}

extern "C" int swp_phase_curve_linear(const double* y, const double* design, const double* amplitude, int B,
                                      int ncoef, int ntimes, double* lc, void* stream) {
  if (!y || !design || !lc || B < 1 || ncoef < 1 || ntimes < 1) return SWP_ERR_ARG;
  const long long n = (long long)B * ntimes;
  if (n > (1ll << 31) - 1) return SWP_ERR_ARG;
  k_phase_curve_linear<<<(int)((n + 255) / 256), 256, 0, (cudaStream_t)stream>>>(y, design, amplitude, B, ncoef,
                                                                                 ntimes, lc);
  return em_check(cudaGetLastError());
}

extern "C" int swp_phase_curve_simple(const double* phi, int B, int J, int I, const double* mus,
                                      const double* phases, int nphase, double* flux, void* stream) {
  if (!phi || !mus || !phases || !flux || B < 1 || J < 1 || I < 1 || nphase < 1) return SWP_ERR_ARG;
  k_phase_curve_simple<<<EM_CL * B, EM_THREADS, 0, (cudaStream_t)stream>>>(phi, J, I, mus, phases, nphase, flux);
  return em_check(cudaGetLastError());
}

// K1: the per-zonal-wavenumber "Legendre sandwich" of one time step.
//
// For a fixed m, everything between the Fourier inputs and the Fourier
// outputs of a step is independent of the other wavenumbers:
//   Fourier inputs (J values per field)  --forward Legendre-->  spectral (n = m..N)
//   --tendency combine, n(n+1), hyperdiffusion, wind inversion-->
//   --inverse Legendre-->  Fourier outputs (J values per field).
// One CTA owns one m and a tile of ensemble members and does the whole chain
// in shared memory.  Reference functions covered:
//   modEuler_tdiff.py:30-268      phi/delta/eta_timestep (quirks: /4, forced A,B in delta, eta asymmetry)
//   explicit_tdiff.py:20-233      phi/delta/eta_timestep (delta carry-only, extra drag terms)
//   spectral_transform.py:370-481 fwd_leg_w / invrs_leg  (negative-m half is conj, never formed)
//   spectral_transform.py:535-596 invrsUV_with_coeffs
//   filters.py:11-27,95-151       diffusion, sigma6, sigma6Phi
//   time_stepping.py:491-534      tstepcoeff, tstepcoeff2, tstepcoeffmn, narray, mJarray, marray
//   semi_implicit_tdiff.py        si_timestep (implicit gravity waves, relaxation and drag)
//   model.py:988-1110             Robert-Asselin / RAW filters of the prev carry; spectral prev carry
// The 19 distinct forward transforms of the reference collapse, by linearity,
// into 9 combined inputs per member (5 on Pw, 4 on Hw), and both contractions
// use the equatorial symmetry of the Gauss grid, Pbar(-mu) = (-1)^(n-m) Pbar(mu),
// so each contraction runs over J/2 latitudes.
#include <algorithm>
#include "swp_internal.h"
#include "spec_common.cuh"

namespace swp {

constexpr int NKIN_P = 5;  // inverse inputs on P: eta, delta, Phi, Uprep, Vprep
constexpr int NKIN_H = 2;  // inverse inputs on H: eta_s (U), -delta_s (V)
constexpr int NKIN = NKIN_P + NKIN_H;
// Register tiles of the contractions: n-columns per thread in the forward one,
// latitudes in the inverse one.  The small tiles are for units of one or two
// members, whose few rows would leave most of a CTA's threads without work (FP32,
// M = 42, 8 members: 25 us with units of 8 members and the large tiles, 18 us with
// units of 2 and the small ones).  A result is one thread's sum over the latitudes
// (degrees) in order, whatever the tile.
template <bool SMALL> struct Reg { static constexpr int FWD_TC = SMALL ? 1 : 4, INV_TJ = SMALL ? 1 : 2; };
constexpr int SMALL_MT = 2;

template <typename T>
size_t spec_smem_bytes(int M, int J, int MT) {
  int Jh = J / 2, R = 2 * MT, cnt = M + 1;
  size_t x = (size_t)(SlotCount<T>::NP + NSH) * 2 * Jh * R;  // symmetrised inputs (reused for outputs)
  size_t bf = (size_t)2 * cnt * Jh;                  // two basis blocks
  size_t kin = (size_t)NKIN * cnt * R;               // inverse inputs
  size_t coef = (size_t)5 * MT * cnt;                // sigma, sigmaPhi, their -1's, a/(n(n+1))
  return (x + bf + kin + coef) * sizeof(T) + 64 * sizeof(int);
}
template size_t spec_smem_bytes<double>(int, int, int);
template size_t spec_smem_bytes<float>(int, int, int);

// The two basis matrices of one m (nb elements each, a multiple of 16 bytes) to
// shared memory; completed by cp_async_wait_all and a block barrier.  Issued at
// the start of a unit -- both blocks where L.early_inv has room for the second
// one -- so that their latency runs beside the combined inputs and not, as loads
// and stores of each thread, between the phases (FP32, one member, M = 106: 36 ->
// 28 us a step).
template <typename T>
__device__ __forceinline__ void copy_basis(T* dst, int ld, const T* srcP, const T* srcH, int nb) {
  constexpr int E = 16 / (int)sizeof(T);
  for (int t = threadIdx.x * E; t < nb; t += blockDim.x * E) {
    cp_async<16>(dst + t, srcP + t);
    cp_async<16>(dst + ld + t, srcH + t);
  }
}
template <typename T>
__host__ __device__ __forceinline__ size_t basis_bytes(int M, int J) { return (size_t)2 * (M + 1) * (J / 2) * sizeof(T); }

// Run body(group, unit index) for every unit of the launch: one unit per CTA,
// or -- persistent launches (L.sched set) -- units taken in turn from the
// launch's counter by resident CTAs, largest truncation first (its units cost
// the most), m ascending within a group.  No CTA waits on another: the last
// CTA to finish resets the counter for the next launch on the stream.
template <typename T, typename F>
__device__ __forceinline__ void for_each_unit(const SpecLaunch<T>& L, F body) {
  if (!L.sched) {
    int idx;
    const SpecGroup<T>& G = pick_group(L, idx);
    body(G, idx);
    return;
  }
  __shared__ int s_unit;
  const int total = L.prefix[L.ng];
  for (;;) {
    if (threadIdx.x == 0) s_unit = atomicAdd(&L.sched->next, 1);
    __syncthreads();
    const int u = s_unit;
    __syncthreads();
    if (u >= total) break;
    int k = 0;
    while (k + 1 < L.ng && u >= L.sprefix[k + 1]) ++k;
    body(L.grp[L.sorder[k]], u - L.sprefix[k]);
    __syncthreads();  // the next unit reuses the shared memory
  }
  if (threadIdx.x == 0) {
    __threadfence();
    if (atomicAdd(&L.sched->done, 1) == (int)gridDim.x - 1) {
      L.sched->next = 0;
      L.sched->done = 0;
      __threadfence();
    }
  }
}

template <typename T, bool SMALL>
__device__ __forceinline__ void spectral_unit(const SpecLaunch<T>& L, const SpecGroup<T>& G, const int idx) {
  typedef typename cplx<T>::type T2;
  constexpr int NSPX = SlotCount<T>::NP;
  constexpr int NSLOT = NSPX + NSH;
  constexpr int FWD_TC = Reg<SMALL>::FWD_TC, INV_TJ = Reg<SMALL>::INV_TJ;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const StepCfg& cfg = L.cfg;
  const int mode = L.mode;
  const Geom<T>& g = G.g;
  const int M = g.M, N = M, J = g.J, Jh = J / 2;
  const int m = idx / G.ntb;
  const int b0 = (idx % G.ntb) * G.MT;
  const int MT = G.MT;
  const int mt = min(MT, G.B - b0);
  const int R = 2 * MT;
  const int cnt = N + 1 - m, C0 = (cnt + 1) / 2, C1 = cnt / 2;
  const int cntmax = N + 1;
  const size_t FS = (size_t)(M + 1) * G.B * J;  // field stride (complex elements)

  T* X = (T*)smem_raw;                                  // [NSLOT][2][Jh][R]
  T* Bf = X + (size_t)NSLOT * 2 * Jh * R;                // [2][cnt*Jh]
  T* Kin = Bf + (size_t)2 * cntmax * Jh;                 // [NKIN][cnt][R]
  T* sig = Kin + (size_t)NKIN * cntmax * R;              // [MT][cnt]
  T* sigP = sig + MT * cntmax;
  T* sigm1 = sigP + MT * cntmax;                         // sigma - 1, formed without cancellation
  T* sigPm1 = sigm1 + MT * cntmax;
  T* tcmn = sigPm1 + MT * cntmax;
  int* sdead = (int*)(((uintptr_t)(tcmn + MT * cntmax) + 15) & ~(uintptr_t)15);  // [MT]
  T* Bi = L.early_inv ? (T*)(((uintptr_t)(sdead + 64) + 15) & ~(uintptr_t)15) : Bf;
  copy_basis<T>(Bf, cntmax * Jh, g.Pw_f + g.boff[m], g.Hw_f + g.boff[m], cnt * Jh);
  if (L.early_inv) copy_basis<T>(Bi, cntmax * Jh, g.P_i + g.boff[m], g.H_i + g.boff[m], cnt * Jh);
  const bool step_mode = mode == 0 || mode == 3;  // 3: tangent-linear step on the tangent state
  const bool incr = SlotCount<T>::INCR && cfg.incremental && step_mode && cfg.scheme == 0;

  // ---- phase 0: per-member spectral coefficients and the blow-up gate
  load_spec_coefs<T>(G, cfg.diffflag && step_mode, m, b0, mt, MT, cnt, cntmax, sig, sigP, sigm1, sigPm1, tcmn,
                     cfg.scheme == 2);
  if (threadIdx.x < MT) {
    int bt = threadIdx.x, dead = 0;
    if (bt < mt && cfg.diagnostics && mode == 0) {
      int b = b0 + bt;
      const double ms = G.diag[((size_t)cfg.step * NDIAG + D_RMS2) * G.B + b];
      dead = (G.member[MS_DEAD * G.B + b] != 0.0) || blown_up(cfg, ms);
      if (m == 0) {
        G.member[MS_DEAD * G.B + b] = dead ? 1.0 : 0.0;
        G.diag[((size_t)cfg.step * NDIAG + D_DEAD) * G.B + b] = dead ? 1.0 : 0.0;
      }
    }
    sdead[bt] = dead;
  }

  // Tangent-linear step with coefficient tangents (a, dt, K6, K6Phi, omega): a
  // first pass transforms the primal combined inputs of the pre-step state; the
  // tangent's hyperdiffusion and wind-inversion terms multiply those spectra
  // (kept per (n, member component) in Kin slots 0-2, which only their owner
  // thread writes).
  const bool tl_coef = mode == 3 && cfg.tl_coef;
  for (int pass = tl_coef ? 0 : 1; pass < 2; ++pass) {
  const bool prim = pass == 0;
  // ---- phase 1: combined, symmetrised inputs
  const T2* F = G.four;
  for (int t = threadIdx.x; t < MT * Jh; t += blockDim.x) {
    int bt = t / Jh, jp = t % Jh;
    T2 xs[NSLOT], xa[NSLOT];
    if (bt < mt) {
      int b = b0 + bt;
#pragma unroll
      for (int side = 0; side < 2; ++side) {
        int j = side ? (J - 1 - jp) : jp;
        T2 c[NSLOT];
        if (prim) {
          const T2* Fq = G.four_p;
          const size_t o = ((size_t)m * G.B + b) * J + j;
          step_combos_ld<T>(G, cfg, 0, incr, m, b, j, [&](int f) { return Fq[f * FS + o]; }, c);
        } else {
          step_combos<T>(G, cfg, mode == 3 ? 0 : mode, incr, m, b, j, FS, c);
          if (mode == 3) tangent_coef_terms<T>(G, cfg, m, b, j, FS, c);
        }
        if (side == 0) {
#pragma unroll
          for (int q = 0; q < NSLOT; ++q) { xs[q] = c[q]; xa[q] = c[q]; }
        } else {
#pragma unroll
          for (int q = 0; q < NSLOT; ++q) { xs[q] = cadd(xs[q], c[q]); xa[q] = csub(xa[q], c[q]); }
        }
      }
    } else {
#pragma unroll
      for (int q = 0; q < NSLOT; ++q) { xs[q] = mk<T2>(0, 0); xa[q] = xs[q]; }
    }
#pragma unroll
    for (int q = 0; q < NSLOT; ++q) {
      T* base = X + (size_t)q * 2 * Jh * R;
      base[(0 * Jh + jp) * R + 2 * bt] = xs[q].x;
      base[(0 * Jh + jp) * R + 2 * bt + 1] = xs[q].y;
      base[(1 * Jh + jp) * R + 2 * bt] = xa[q].x;
      base[(1 * Jh + jp) * R + 2 * bt + 1] = xa[q].y;
    }
  }
  // ---- phase 2: the basis blocks have arrived
  cp_async_wait_all();
  __syncthreads();

  // ---- phase 3: forward contraction over J/2 latitudes + spectral epilogue
  {
    const int nt0 = (C0 + FWD_TC - 1) / FWD_TC, nt1 = (C1 + FWD_TC - 1) / FWD_TC;
    const int tasks = R * (nt0 + nt1);
    const T* BP = Bf;
    const T* BH = Bf + cntmax * Jh;
    for (int task = threadIdx.x; task < tasks; task += blockDim.x) {
      int r = task % R;
      int ct = task / R;
      int par = ct < nt0 ? 0 : 1;
      if (par) ct -= nt0;
      int Cp = par ? C1 : C0;
      int c0 = ct * FWD_TC;
      const T* bp = BP + (par ? Jh * C0 : 0);
      const T* bh = BH + (par ? Jh * C0 : 0);
      // P slots read the symmetric sum for even (n-m), the antisymmetric for odd; H the reverse.
      const int sP = par, sH = 1 - par;
      T acc[NSLOT][FWD_TC];
#pragma unroll
      for (int q = 0; q < NSLOT; ++q)
#pragma unroll
        for (int k = 0; k < FWD_TC; ++k) acc[q][k] = (T)0;
      for (int jp = 0; jp < Jh; ++jp) {
        T xp[NSPX], xh[NSH];
#pragma unroll
        for (int q = 0; q < NSPX; ++q) xp[q] = X[((size_t)q * 2 * Jh + sP * Jh + jp) * R + r];
#pragma unroll
        for (int q = 0; q < NSH; ++q) xh[q] = X[((size_t)(NSPX + q) * 2 * Jh + sH * Jh + jp) * R + r];
        T vp[FWD_TC], vh[FWD_TC];
#pragma unroll
        for (int k = 0; k < FWD_TC; ++k) {
          int c = c0 + k;
          vp[k] = c < Cp ? bp[jp * Cp + c] : (T)0;
          vh[k] = c < Cp ? bh[jp * Cp + c] : (T)0;
        }
#pragma unroll
        for (int k = 0; k < FWD_TC; ++k) {
#pragma unroll
          for (int q = 0; q < NSPX; ++q) acc[q][k] = fma(xp[q], vp[k], acc[q][k]);
#pragma unroll
          for (int q = 0; q < NSH; ++q) acc[NSPX + q][k] = fma(xh[q], vh[k], acc[NSPX + q][k]);
        }
      }
      const int bt = r >> 1, comp = r & 1;
      // planetary vorticity f_{0,1}: a constant of the wind inversion; its
      // tangent is the omega tangent's
      const T om = bt < mt ? G.mco[(mode == 3 ? MC_DOM : MC_OM) * G.B + b0 + bt] : (T)0;
      const T om_p = (tl_coef && bt < mt) ? G.mco[MC_OM * G.B + b0 + bt] : (T)0;
      // semi-implicit solve constants (semi_implicit_tdiff.py): implicit share
      // xi, implicit drag / relaxation kd, kr, explicit drag gd, Phibar, 1/a^2
      T si_xi = (T)0, si_kd = (T)0, si_kr = (T)0, si_gd = (T)0, si_pb = (T)0, si_ia2 = (T)0;
      // and, for the tangent step, their tangents
      T si_dxi = (T)0, si_dkd = (T)0, si_dkr = (T)0, si_dgd = (T)0, si_dpb = (T)0, si_dia2 = (T)0;
      if ((mode == 0 || mode == 3) && cfg.scheme == 2 && bt < mt) {
        const T* mc = G.mco;
        const int b = b0 + bt, B = G.B;
        si_xi = mc[MC_SIXI * B + b];
        si_pb = mc[MC_PB * B + b];
        si_ia2 = mc[MC_IA2 * B + b];
        if (mode == 3) {
          si_dxi = mc[MC_DSIXI * B + b];
          si_dpb = (T)2 * mc[MC_DHPB * B + b];
          si_dia2 = mc[MC_DIA2 * B + b];
        }
        if (cfg.si_relax) {
          const T itd = mc[MC_SIITD * B + b], itr = mc[MC_SIITR * B + b], ex = mc[MC_SIEX * B + b];
          si_kd = si_xi * itd;
          si_kr = si_xi * itr;
          si_gd = ex * itd;
          if (mode == 3) {
            const T ditd = mc[MC_DSIITD * B + b], ditr = mc[MC_DSIITR * B + b], dex = mc[MC_DSIEX * B + b];
            si_dkd = si_dxi * itd + si_xi * ditd;
            si_dkr = si_dxi * itr + si_xi * ditr;
            si_dgd = dex * itd + ex * ditd;
          }
        }
      }
#pragma unroll
      for (int k = 0; k < FWD_TC; ++k) {
        int c = c0 + k;
        if (c >= Cp) break;
        int kk = par + 2 * c;            // n - m
        int n = m + kk;
        T nn1 = (T)(n * (n + 1));
        T s = sig[bt * cntmax + kk], sp = sigP[bt * cntmax + kk], tc = tcmn[bt * cntmax + kk];
        const int pc = par ? C0 + c : c;
        if (prim) {
          // primal pre-step spectra (incremental form: curr + tendency part)
          T sphi = acc[SP_PHI1][k] + acc[NSPX + SH_PHI1][k] + nn1 * acc[SP_PHI2][k];
          T sdel = acc[SP_D1][k] + acc[NSPX + SH_D1][k] + nn1 * (acc[SP_D2][k] + acc[NSPX + SH_D2][k]);
          T seta = acc[SP_E1][k] + acc[NSPX + SH_E1][k];
          if (incr) {
            sphi += acc[NSPX > SP_IPHI ? SP_IPHI : 0][k];
            sdel += acc[NSPX > SP_ID ? SP_ID : 0][k];
            seta += acc[NSPX > SP_IE ? SP_IE : 0][k];
          }
          Kin[((size_t)0 * cntmax + pc) * R + r] = seta;
          Kin[((size_t)1 * cntmax + pc) * R + r] = sdel;
          Kin[((size_t)2 * cntmax + pc) * R + r] = sphi;
          continue;
        }
        T cphi, cdel, ceta;      // spectral eta, delta (full, for the winds)
        T kphi, kdel, keta;      // what the inverse transform turns into the new Fourier carries
        T pce = (T)0, pcd = (T)0;  // primal spectral eta, delta after hyperdiffusion (tl_coef)
        if (mode == 2) {
          ceta = acc[SP_E1][k];
          cdel = acc[SP_D1][k];
          cphi = (T)0;
          kphi = cphi; kdel = cdel; keta = ceta;
        } else if (cfg.scheme == 2 && mode == 3) {
          // tangent of the implicit solve below: the tangent spectra through the
          // primal solve, plus the solve's and the exponential sigmas' parameter
          // tangents applied to the primal spectra (pass 0)
          T seta = acc[SP_E1][k] + acc[NSPX + SH_E1][k];
          T sdel = acc[SP_D1][k] + acc[NSPX + SH_D1][k] + nn1 * acc[SP_D2][k];
          T sphi = acc[SP_PHI1][k] + acc[NSPX + SH_PHI1][k];
          T Se = Kin[((size_t)0 * cntmax + pc) * R + r], Sd = Kin[((size_t)1 * cntmax + pc) * R + r];
          T Sp = Kin[((size_t)2 * cntmax + pc) * R + r];
          if (m == 0 && n == 1 && comp == 0) {
            Se += (si_gd + si_kd) * om_p;
            seta += (si_dgd + si_dkd) * om_p + (si_gd + si_kd) * om;  // om: tangent of f here
          }
          const T bq = si_xi * (nn1 * si_ia2), cq = si_xi * si_pb;
          const T ikr = (T)1 / ((T)1 + si_kr), ikd = (T)1 / ((T)1 + si_kd);
          const T Dn = ((T)1 + si_kd) + bq * cq * ikr;
          const T dnew = (Sd + bq * Sp * ikr) / Dn, pnew = (Sp - cq * dnew) * ikr, enew = Se * ikd;
          const T dbq = nn1 * (si_dxi * si_ia2 + si_xi * si_dia2), dcq = si_dxi * si_pb + si_xi * si_dpb;
          const T dikr = -ikr * ikr * si_dkr;
          const T denew = (seta - enew * si_dkd) * ikd;
          const T dnum = sdel + dbq * Sp * ikr + bq * sphi * ikr + bq * Sp * dikr;
          const T dD = si_dkd + dbq * cq * ikr + bq * dcq * ikr + bq * cq * dikr;
          const T ddnew = (dnum - dnew * dD) / Dn;
          const T dpnew = (sphi - dcq * dnew - cq * ddnew) * ikr + (Sp - cq * dnew) * dikr;
          T dsg = (T)0, dsp = (T)0;
          if (cfg.diffflag && bt < mt) {
            const size_t qs = (size_t)G.B * cntmax, qo = (size_t)(b0 + bt) * cntmax + n;
            dsg = G.nco[NC_DSIGX * qs + qo];
            dsp = G.nco[NC_DSIGPX * qs + qo];
          }
          cphi = sp * dpnew + dsp * pnew;
          cdel = s * ddnew + dsg * dnew;
          ceta = s * denew + dsg * enew;
          kphi = cphi; kdel = cdel; keta = ceta;
          pce = s * enew;
          pcd = s * dnew;
        } else if (cfg.scheme == 2) {
          // eta* , delta*, Phi* -> the implicit (delta, Phi) pair per degree,
          // eliminated for delta; then the exponential hyperdiffusion
          T seta = acc[SP_E1][k] + acc[NSPX + SH_E1][k];
          T sdel = acc[SP_D1][k] + acc[NSPX + SH_D1][k] + nn1 * acc[SP_D2][k];
          T sphi = acc[SP_PHI1][k] + acc[NSPX + SH_PHI1][k];
          if (m == 0 && n == 1 && comp == 0) {  // f_{0,1}: explicit then implicit drag toward it
            seta += si_gd * om;
            seta += si_kd * om;
          }
          T bq = si_xi * (nn1 * si_ia2), cq = si_xi * si_pb;
          T ikr = (T)1 / ((T)1 + si_kr);
          T dnew = (sdel + bq * sphi * ikr) / (((T)1 + si_kd) + bq * cq * ikr);
          T pnew = (sphi - cq * dnew) * ikr;
          T enew = seta / ((T)1 + si_kd);
          cphi = sp * pnew;
          cdel = s * dnew;
          ceta = s * enew;
          kphi = cphi; kdel = cdel; keta = ceta;
        } else {
          T sphi = acc[SP_PHI1][k] + acc[NSPX + SH_PHI1][k] + nn1 * acc[SP_PHI2][k];
          T sdel = acc[SP_D1][k] + acc[NSPX + SH_D1][k] + nn1 * (acc[SP_D2][k] + acc[NSPX + SH_D2][k]);
          T seta = acc[SP_E1][k] + acc[NSPX + SH_E1][k];
          if (incr) {
            // new = curr + Inv(dc), dc = (sigma - 1) Fwd(curr) + sigma * tendency
            T iphi = acc[NSPX > SP_IPHI ? SP_IPHI : 0][k], idel = acc[NSPX > SP_ID ? SP_ID : 0][k];
            T ieta = acc[NSPX > SP_IE ? SP_IE : 0][k];
            T sm1 = sigm1[bt * cntmax + kk], spm1 = sigPm1[bt * cntmax + kk];
            cdel = s * (idel + sdel);
            ceta = s * (ieta + seta);
            cphi = sp * (iphi + sphi);
            kphi = spm1 * iphi + sp * sphi;
            kdel = sm1 * idel + s * sdel;
            keta = sm1 * ieta + s * seta;
          } else {
            cphi = sp * sphi;
            cdel = s * sdel;
            ceta = s * seta;
            kphi = cphi; kdel = cdel; keta = ceta;
          }
          if (tl_coef && bt < mt) {
            // hyperdiffusion tangent: d(sigma) times the primal spectra
            const size_t qs = (size_t)G.B * cntmax, qo = (size_t)(b0 + bt) * cntmax + n;
            const T dsg = G.nco[NC_DSIG * qs + qo], dsp = G.nco[NC_DSIGP * qs + qo];
            const T pe = Kin[((size_t)0 * cntmax + pc) * R + r], pd = Kin[((size_t)1 * cntmax + pc) * R + r];
            const T pp = Kin[((size_t)2 * cntmax + pc) * R + r];
            cphi += dsp * pp; cdel += dsg * pd; ceta += dsg * pe;
            kphi += dsp * pp; kdel += dsg * pd; keta += dsg * pe;
            pce = s * pe;
            pcd = s * pd;
          }
        }
        // wind inversion inputs (spectral_transform.py:577-594)
        T dp = (n == 0) ? (T)0 : cdel;
        T ep = (n == 0) ? (T)0 : ceta;
        if (m == 0 && n == 1 && comp == 0) ep -= om;
        T es = ep * tc, ds = dp * tc;
        if (tl_coef && bt < mt) {  // tangent of a/(n(n+1)) times the primal (eta - f), delta
          const T dtc = G.nco[(size_t)NC_DTC * G.B * cntmax + (size_t)(b0 + bt) * cntmax + n];
          T epp = (n == 0) ? (T)0 : pce;
          if (m == 0 && n == 1 && comp == 0) epp -= om_p;
          es += epp * dtc;
          ds += ((n == 0) ? (T)0 : pcd) * dtc;
        }
        Kin[((size_t)0 * cntmax + pc) * R + r] = keta;
        Kin[((size_t)1 * cntmax + pc) * R + r] = kdel;
        Kin[((size_t)2 * cntmax + pc) * R + r] = kphi;
        // Uprep = -i m delta_s ; Vprep = -i m eta_s  (write the other component)
        T xm = (T)m;
        if (comp == 0) {
          Kin[((size_t)3 * cntmax + pc) * R + r + 1] = -xm * ds;
          Kin[((size_t)4 * cntmax + pc) * R + r + 1] = -xm * es;
        } else {
          Kin[((size_t)3 * cntmax + pc) * R + r - 1] = xm * ds;
          Kin[((size_t)4 * cntmax + pc) * R + r - 1] = xm * es;
        }
        Kin[((size_t)5 * cntmax + pc) * R + r] = es;
        Kin[((size_t)6 * cntmax + pc) * R + r] = -ds;
      }
    }
  }
  __syncthreads();
  }  // pass
  // ---- phase 4: inverse basis block for m
  if (!L.early_inv) {
    copy_basis<T>(Bi, cntmax * Jh, g.P_i + g.boff[m], g.H_i + g.boff[m], cnt * Jh);
    cp_async_wait_all();
    __syncthreads();
  }

  // ---- phase 5: inverse contraction (even/odd n-m) -> Fourier outputs in smem
  T* Out = X;  // [5][MT][J][2]
  {
    const int njt = (Jh + INV_TJ - 1) / INV_TJ;
    const int tasks = R * njt;
    const T* BP = Bi;
    const T* BH = Bi + cntmax * Jh;
    for (int task = threadIdx.x; task < tasks; task += blockDim.x) {
      int r = task % R;
      int j0 = (task / R) * INV_TJ;
      T E[NKIN][INV_TJ], O[NKIN][INV_TJ];
#pragma unroll
      for (int q = 0; q < NKIN; ++q)
#pragma unroll
        for (int k = 0; k < INV_TJ; ++k) { E[q][k] = (T)0; O[q][k] = (T)0; }
      // even n-m
      for (int c = 0; c < C0; ++c) {
        T kin[NKIN];
#pragma unroll
        for (int q = 0; q < NKIN; ++q) kin[q] = Kin[((size_t)q * cntmax + c) * R + r];
#pragma unroll
        for (int k = 0; k < INV_TJ; ++k) {
          int jp = j0 + k;
          T p = jp < Jh ? BP[c * Jh + jp] : (T)0;
          T h = jp < Jh ? BH[c * Jh + jp] : (T)0;
#pragma unroll
          for (int q = 0; q < NKIN_P; ++q) E[q][k] = fma(kin[q], p, E[q][k]);
#pragma unroll
          for (int q = NKIN_P; q < NKIN; ++q) E[q][k] = fma(kin[q], h, E[q][k]);
        }
      }
      // odd n-m
      for (int c = 0; c < C1; ++c) {
        T kin[NKIN];
#pragma unroll
        for (int q = 0; q < NKIN; ++q) kin[q] = Kin[((size_t)q * cntmax + C0 + c) * R + r];
#pragma unroll
        for (int k = 0; k < INV_TJ; ++k) {
          int jp = j0 + k;
          T p = jp < Jh ? BP[Jh * C0 + c * Jh + jp] : (T)0;
          T h = jp < Jh ? BH[Jh * C0 + c * Jh + jp] : (T)0;
#pragma unroll
          for (int q = 0; q < NKIN_P; ++q) O[q][k] = fma(kin[q], p, O[q][k]);
#pragma unroll
          for (int q = NKIN_P; q < NKIN; ++q) O[q][k] = fma(kin[q], h, O[q][k]);
        }
      }
      const int bt = r >> 1, comp = r & 1;
#pragma unroll
      for (int k = 0; k < INV_TJ; ++k) {
        int jp = j0 + k;
        if (jp >= Jh) break;
        int jn = jp, js = J - 1 - jp;
        auto put = [&](int f, int j, T v) { Out[(((size_t)f * MT + bt) * J + j) * 2 + comp] = v; };
        put(0, jn, E[0][k] + O[0][k]); put(0, js, E[0][k] - O[0][k]);
        put(1, jn, E[1][k] + O[1][k]); put(1, js, E[1][k] - O[1][k]);
        put(2, jn, E[2][k] + O[2][k]); put(2, js, E[2][k] - O[2][k]);
        put(3, jn, (E[3][k] + O[3][k]) + (E[5][k] + O[5][k]));
        put(3, js, (E[3][k] - O[3][k]) + (O[5][k] - E[5][k]));
        put(4, jn, (E[4][k] + O[4][k]) + (E[6][k] + O[6][k]));
        put(4, js, (E[4][k] - O[4][k]) + (O[6][k] - E[6][k]));
      }
    }
  }
  __syncthreads();

  // ---- phase 6: write-out and carries (coalesced along j)
  const int do_uv = (mode == 2) || (cfg.test != 1);
  for (int t = threadIdx.x; t < MT * J; t += blockDim.x) {
    int bt = t / J, j = t % J;
    if (bt >= mt || sdead[bt]) continue;
    int b = b0 + bt;
    size_t o = ((size_t)m * G.B + b) * J + j;
    auto get = [&](int f) { return mk<T2>(Out[(((size_t)f * MT + bt) * J + j) * 2], Out[(((size_t)f * MT + bt) * J + j) * 2 + 1]); };
    if (mode == 2) {
      G.four_out[F_U * FS + o] = get(3);
      G.four_out[F_V * FS + o] = get(4);
      continue;
    }
    const T2 nw[3] = {get(0), get(1), get(2)};
    write_step_point<T>(G, cfg, incr, FS, o, b, nw, do_uv != 0, get(3), get(4), mode == 3);
  }
  // residual weights of the initial condition in the physical curr / prev fields
  if (mode == 0 && m == 0 && threadIdx.x < mt && !sdead[threadIdx.x]) {
    int b = b0 + threadIdx.x;
    double wc = G.member[MS_WCURR * G.B + b], wm = G.member[MS_WMID * G.B + b];
    if (cfg.tl_filter) {
      double dwc = G.dw[b], dwm = G.dw[G.B + b];
      step_residual_weights_tl(cfg, G.par[P_ALPHA * G.B + b], G.par[P_WALPHA * G.B + b],
                               G.dpar[T_ALPHA * G.B + b], G.dpar[T_WALPHA * G.B + b], wc, wm, dwc, dwm);
      G.dw[b] = dwc;
      G.dw[G.B + b] = dwm;
    }
    step_residual_weights(cfg, G.par[P_ALPHA * G.B + b], G.par[P_WALPHA * G.B + b], wc, wm);
    G.member[MS_WMID * G.B + b] = wm;
    G.member[MS_WCURR * G.B + b] = wc;
    G.member[MS_UPDATED * G.B + b] = 1.0;
  }
}

// FP32: 128 registers with a few spills, for a second CTA per SM (M = 42, 32
// members: 36 -> 29 us)
template <typename T, bool SMALL>
__global__ void __launch_bounds__(256, sizeof(T) == 4 ? 2 : 1) k_spectral(const __grid_constant__ SpecLaunch<T> L) {
  pdl_enter();
  for_each_unit(L, [&](const SpecGroup<T>& G, int idx) { spectral_unit<T, SMALL>(L, G, idx); });
}

// ---------------------------------------------------------------------------
// Adjoint of k_spectral (modified Euler, mode 0).  Same per-m decomposition:
//   lambda of the Fourier outputs (eta, delta, Phi, U, V at column m)
//   --transposed inverse Legendre (P^T, H^T)--> lambda of the spectral inputs
//   --transposed wind inversion, n(n+1), hyperdiffusion-->
//   --transposed forward Legendre (Pw, Hw)--> lambda of the 9 combined inputs
//   --transposed combination--> lambda of the 11 Fourier state fields.
// The Phibar gradient of the combination is accumulated from the primal
// state before the step.
constexpr int NYS_P = 5;   // lambda eta, delta, Phi, U, V on P
constexpr int NYS_H = 2;   // lambda U, V on H
constexpr int NYS = NYS_P + NYS_H;
// coefficient vectors of the transposed forward contraction: 5, plus the three
// identity slots of the incremental form on the FP32 path
template <typename T> struct AdjCount { static constexpr int NK = SlotCount<T>::NP; };

template <typename T>
size_t spec_adj_smem_bytes(int M, int J, int MT) {
  int Jh = J / 2, R = 2 * MT, cnt = M + 1;
  constexpr int NK = AdjCount<T>::NK;
  size_t x = (size_t)2 * (NK + 4) * J * MT;
  size_t x2 = (size_t)NYS * 2 * Jh * R;
  if (x2 > x) x = x2;
  size_t bf = (size_t)2 * cnt * Jh;
  size_t sres = (size_t)NYS * cnt * R;
  size_t kad = (size_t)NK * cnt * R;
  size_t coef = (size_t)5 * MT * cnt;
  return (x + bf + sres + kad + coef) * sizeof(T) + 16 + (size_t)2 * MT * (J / 32) * sizeof(double);
}
template size_t spec_adj_smem_bytes<double>(int, int, int);
template size_t spec_adj_smem_bytes<float>(int, int, int);

template <typename T, bool SMALL>
__device__ __forceinline__ void spectral_adj_unit(const SpecLaunch<T>& L, const SpecGroup<T>& G, const int idx) {
  typedef typename cplx<T>::type T2;
  constexpr int NKADJ = AdjCount<T>::NK;
  constexpr int NCAD = NKADJ + 4;
  constexpr int FWD_TC = Reg<SMALL>::FWD_TC, INV_TJ = Reg<SMALL>::INV_TJ;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const StepCfg& cfg = L.cfg;
  const bool incr = SlotCount<T>::INCR && cfg.incremental;
  const Geom<T>& g = G.g;
  const int M = g.M, N = M, J = g.J, Jh = J / 2;
  const int m = idx / G.ntb;
  const int b0 = (idx % G.ntb) * G.MT;
  const int MT = G.MT;
  const int mt = min(MT, G.B - b0);
  const int R = 2 * MT;
  const int cnt = N + 1 - m, C0 = (cnt + 1) / 2, C1 = cnt / 2;
  const int cntmax = N + 1;
  const size_t FS = (size_t)(M + 1) * G.B * J;

  T* X = (T*)smem_raw;                                  // [NYS][2][Jh][R], later [NCAD][MT][J][2]
  const size_t xsz = ((size_t)2 * NCAD * J * MT > (size_t)NYS * 2 * Jh * R) ? (size_t)2 * NCAD * J * MT
                                                                            : (size_t)NYS * 2 * Jh * R;
  T* Bf = X + xsz;                                       // [2][cnt*Jh]
  T* Sres = Bf + (size_t)2 * cntmax * Jh;                // [NYS][cnt][R]
  T* Kad = Sres + (size_t)NYS * cntmax * R;              // [NKADJ][cnt][R]
  T* sig = Kad + (size_t)NKADJ * cntmax * R;
  T* sigP = sig + MT * cntmax;
  T* sigm1 = sigP + MT * cntmax;
  T* sigPm1 = sigm1 + MT * cntmax;
  T* tcmn = sigPm1 + MT * cntmax;
  // [2][MT][J/32] Phibar and taudrag gradient partials of each warp-sized run
  // of latitudes (doubles: round the address up to 16 bytes)
  double* sgrad = (double*)(((uintptr_t)(tcmn + MT * cntmax) + 15) & ~(uintptr_t)15);
  const int nws = J / 32;
  T* Bi = L.early_inv ? (T*)(((uintptr_t)(sgrad + 2 * MT * nws) + 15) & ~(uintptr_t)15) : Bf;
  copy_basis<T>(Bf, cntmax * Jh, g.P_f + g.boff[m], g.H_f + g.boff[m], cnt * Jh);
  if (L.early_inv) copy_basis<T>(Bi, cntmax * Jh, g.Pw_i + g.boff[m], g.Hw_i + g.boff[m], cnt * Jh);

  load_spec_coefs<T>(G, cfg.diffflag != 0, m, b0, mt, MT, cnt, cntmax, sig, sigP, sigm1, sigPm1, tcmn,
                     cfg.scheme == 2);
  for (int t = threadIdx.x; t < 2 * MT * nws; t += blockDim.x) sgrad[t] = 0.0;

  // ---- phase 1: symmetrised adjoints of the step outputs at column m.  The
  // semi-implicit step's new level also enters its filtered mid carry with
  // weight al (Robert-Asselin update), whose adjoint adds here.
  const T2* LY = G.lamY;  // [5][M+1][B][J]
  const bool si_ra = cfg.scheme == 2 && cfg.ra_mode == 2;
  for (int t = threadIdx.x; t < MT * Jh; t += blockDim.x) {
    int bt = t / Jh, jp = t % Jh;
    T2 ys[5], ya[5];
    if (bt < mt) {
      int b = b0 + bt;
      size_t on = ((size_t)m * G.B + b) * J + jp, os = ((size_t)m * G.B + b) * J + (J - 1 - jp);
      const T al = si_ra ? G.mco[MC_ALPHA * G.B + b] : (T)0;
#pragma unroll
      for (int f = 0; f < 5; ++f) {
        T2 u = LY[f * FS + on], v = LY[f * FS + os];
        if (si_ra && f < 3) {
          const int mf = f == 0 ? F_ETA_MID : f == 1 ? F_DELTA_MID : F_PHI_MID;
          u = cadd(u, cscale(G.lam[mf * FS + on], al));
          v = cadd(v, cscale(G.lam[mf * FS + os], al));
        }
        ys[f] = cadd(u, v);
        ya[f] = csub(u, v);
      }
    } else {
#pragma unroll
      for (int f = 0; f < 5; ++f) { ys[f] = mk<T2>(0, 0); ya[f] = ys[f]; }
    }
    auto put = [&](int q, int sa, T2 v) {
      T* base = X + (size_t)q * 2 * Jh * R;
      base[(sa * Jh + jp) * R + 2 * bt] = v.x;
      base[(sa * Jh + jp) * R + 2 * bt + 1] = v.y;
    };
#pragma unroll
    for (int f = 0; f < 5; ++f) { put(f, 0, ys[f]); put(f, 1, ya[f]); }
    put(5, 0, ys[3]); put(5, 1, ya[3]);
    put(6, 0, ys[4]); put(6, 1, ya[4]);
  }
  cp_async_wait_all();
  __syncthreads();

  // ---- phase 2: transposed inverse Legendre (contract over J/2 latitudes)
  {
    const int nt0 = (C0 + FWD_TC - 1) / FWD_TC, nt1 = (C1 + FWD_TC - 1) / FWD_TC;
    const int tasks = R * (nt0 + nt1);
    const T* BP = Bf;
    const T* BH = Bf + cntmax * Jh;
    for (int task = threadIdx.x; task < tasks; task += blockDim.x) {
      int r = task % R;
      int ct = task / R;
      int par = ct < nt0 ? 0 : 1;
      if (par) ct -= nt0;
      int Cp = par ? C1 : C0;
      int c0 = ct * FWD_TC;
      const T* bp = BP + (par ? Jh * C0 : 0);
      const T* bh = BH + (par ? Jh * C0 : 0);
      const int sP = par, sH = 1 - par;
      T acc[NYS][FWD_TC];
#pragma unroll
      for (int q = 0; q < NYS; ++q)
#pragma unroll
        for (int k = 0; k < FWD_TC; ++k) acc[q][k] = (T)0;
      for (int jp = 0; jp < Jh; ++jp) {
        T xp[NYS_P], xh[NYS_H];
#pragma unroll
        for (int q = 0; q < NYS_P; ++q) xp[q] = X[((size_t)q * 2 * Jh + sP * Jh + jp) * R + r];
#pragma unroll
        for (int q = 0; q < NYS_H; ++q) xh[q] = X[((size_t)(NYS_P + q) * 2 * Jh + sH * Jh + jp) * R + r];
        T vp[FWD_TC], vh[FWD_TC];
#pragma unroll
        for (int k = 0; k < FWD_TC; ++k) {
          int c = c0 + k;
          vp[k] = c < Cp ? bp[jp * Cp + c] : (T)0;
          vh[k] = c < Cp ? bh[jp * Cp + c] : (T)0;
        }
#pragma unroll
        for (int k = 0; k < FWD_TC; ++k) {
#pragma unroll
          for (int q = 0; q < NYS_P; ++q) acc[q][k] = fma(xp[q], vp[k], acc[q][k]);
#pragma unroll
          for (int q = 0; q < NYS_H; ++q) acc[NYS_P + q][k] = fma(xh[q], vh[k], acc[NYS_P + q][k]);
        }
      }
#pragma unroll
      for (int k = 0; k < FWD_TC; ++k) {
        int c = c0 + k;
        if (c >= Cp) break;
        int pc = par ? C0 + c : c;
#pragma unroll
        for (int q = 0; q < NYS; ++q) Sres[((size_t)q * cntmax + pc) * R + r] = acc[q][k];
      }
    }
  }
  __syncthreads();
  // ---- phase 3: transposed wind inversion, n(n+1) and hyperdiffusion
  for (int t = threadIdx.x; t < MT * cnt; t += blockDim.x) {
    int bt = t / cnt, kk = t % cnt, n = m + kk;
    int par = kk & 1, c = kk >> 1;
    int pc = par ? C0 + c : c;
    auto S = [&](int q, int comp) { return Sres[((size_t)q * cntmax + pc) * R + 2 * bt + comp]; };
    T xm = (T)m;
    T tc = tcmn[bt * cntmax + kk];
    T s = sig[bt * cntmax + kk], sp = sigP[bt * cntmax + kk];
    T nn1 = (T)(n * (n + 1));
    // lambda delta_s = (i m) lambda Uprep - lambda Hin_V ; lambda eta_s = (i m) lambda Vprep + lambda Hin_U
    T lds_r = -xm * S(3, 1) - S(6, 0), lds_i = xm * S(3, 0) - S(6, 1);
    T les_r = -xm * S(4, 1) + S(5, 0), les_i = xm * S(4, 0) + S(5, 1);
    T w = (n == 0) ? (T)0 : tc;
    T lce_r = S(0, 0) + w * les_r, lce_i = S(0, 1) + w * les_i;
    T lcd_r = S(1, 0) + w * lds_r, lcd_i = S(1, 1) + w * lds_i;
    T lcp_r = S(2, 0), lcp_i = S(2, 1);
    auto K = [&](int q, int comp, T v) { Kad[((size_t)q * cntmax + pc) * R + 2 * bt + comp] = v; };
    if (cfg.scheme == 2) {
      // transpose of the semi-implicit solve per degree (spectral_unit):
      //   dnew = (sdel + bq ikr sphi) / Dn,  pnew = (sphi - cq dnew) ikr,  enew = seta ikd,
      // then the exponential sigmas; slot map as below with PhiP2 unused
      T xi = (T)0, kd = (T)0, kr = (T)0, pbv = (T)0, ia2 = (T)0;
      if (bt < mt) {
        const T* mc = G.mco;
        const int b = b0 + bt, B = G.B;
        xi = mc[MC_SIXI * B + b];
        pbv = mc[MC_PB * B + b];
        ia2 = mc[MC_IA2 * B + b];
        if (cfg.si_relax) {
          kd = xi * mc[MC_SIITD * B + b];
          kr = xi * mc[MC_SIITR * B + b];
        }
      }
      const T bq = xi * (nn1 * ia2), cq = xi * pbv;
      const T ikr = (T)1 / ((T)1 + kr), ikd = (T)1 / ((T)1 + kd);
      const T Dn = ((T)1 + kd) + bq * cq * ikr;
      const T lpn_r = sp * lcp_r, lpn_i = sp * lcp_i;
      const T ldn_r = s * lcd_r - cq * ikr * lpn_r, ldn_i = s * lcd_i - cq * ikr * lpn_i;
      const T lsd_r = ldn_r / Dn, lsd_i = ldn_i / Dn;
      K(0, 0, ikr * lpn_r + bq * ikr * lsd_r); K(0, 1, ikr * lpn_i + bq * ikr * lsd_i);
      K(1, 0, (T)0); K(1, 1, (T)0);
      K(2, 0, lsd_r); K(2, 1, lsd_i);
      K(3, 0, nn1 * lsd_r); K(3, 1, nn1 * lsd_i);
      K(4, 0, ikd * s * lce_r); K(4, 1, ikd * s * lce_i);
    } else {
      K(0, 0, sp * lcp_r); K(0, 1, sp * lcp_i);
      K(1, 0, nn1 * sp * lcp_r); K(1, 1, nn1 * sp * lcp_i);
      K(2, 0, s * lcd_r); K(2, 1, s * lcd_i);
      K(3, 0, nn1 * s * lcd_r); K(3, 1, nn1 * s * lcd_i);
      K(4, 0, s * lce_r); K(4, 1, s * lce_i);
    }
    if (NKADJ > 5) {
      // identity slots of the incremental form: d/d Fwd(curr) of
      //   dc_f = (sigma_f - 1) Fwd(curr_f) + ...  and of the full c_eta, c_delta used for the winds
      T sm1 = sigm1[bt * cntmax + kk], spm1 = sigPm1[bt * cntmax + kk];
      T ide_r = incr ? (s * w * les_r + sm1 * S(0, 0)) : (T)0, ide_i = incr ? (s * w * les_i + sm1 * S(0, 1)) : (T)0;
      T idd_r = incr ? (s * w * lds_r + sm1 * S(1, 0)) : (T)0, idd_i = incr ? (s * w * lds_i + sm1 * S(1, 1)) : (T)0;
      T idp_r = incr ? spm1 * S(2, 0) : (T)0, idp_i = incr ? spm1 * S(2, 1) : (T)0;
      K(NKADJ > 5 ? 5 : 0, 0, idp_r); K(NKADJ > 5 ? 5 : 0, 1, idp_i);
      K(NKADJ > 6 ? 6 : 0, 0, idd_r); K(NKADJ > 6 ? 6 : 0, 1, idd_i);
      K(NKADJ > 7 ? 7 : 0, 0, ide_r); K(NKADJ > 7 ? 7 : 0, 1, ide_i);
    }
  }
  __syncthreads();
  if (!L.early_inv) {
    copy_basis<T>(Bi, cntmax * Jh, g.Pw_i + g.boff[m], g.Hw_i + g.boff[m], cnt * Jh);
    cp_async_wait_all();
    __syncthreads();
  }
  // ---- phase 4: transposed forward Legendre -> adjoints of the 9 combined inputs
  T* Cad = X;  // [NCAD][MT][J][2]
  {
    const int njt = (Jh + INV_TJ - 1) / INV_TJ;
    const int tasks = R * njt;
    const T* BP = Bi;
    const T* BH = Bi + cntmax * Jh;
    // P results: K0..K4 on Pw -> PhiP1, PhiP2, dP1, dP2, eP1 ; H results: K0, K2, K3, K4 on Hw -> PhiH1, dH1, dH2, eH1
    for (int task = threadIdx.x; task < tasks; task += blockDim.x) {
      int r = task % R;
      int j0 = (task / R) * INV_TJ;
      T E[NCAD][INV_TJ], O[NCAD][INV_TJ];
#pragma unroll
      for (int q = 0; q < NCAD; ++q)
#pragma unroll
        for (int k = 0; k < INV_TJ; ++k) { E[q][k] = (T)0; O[q][k] = (T)0; }
      auto accum = [&](T (&acc)[NCAD][INV_TJ], int par, int c) {
        int pc = par ? C0 + c : c;
        T kv[NKADJ];
#pragma unroll
        for (int q = 0; q < NKADJ; ++q) kv[q] = Kad[((size_t)q * cntmax + pc) * R + r];
#pragma unroll
        for (int k = 0; k < INV_TJ; ++k) {
          int jp = j0 + k;
          T p = jp < Jh ? BP[(par ? Jh * C0 : 0) + c * Jh + jp] : (T)0;
          T h = jp < Jh ? BH[(par ? Jh * C0 : 0) + c * Jh + jp] : (T)0;
#pragma unroll
          for (int q = 0; q < NKADJ; ++q) acc[q][k] = fma(kv[q], p, acc[q][k]);
          acc[NKADJ + 0][k] = fma(kv[0], h, acc[NKADJ + 0][k]);
          acc[NKADJ + 1][k] = fma(kv[2], h, acc[NKADJ + 1][k]);
          acc[NKADJ + 2][k] = fma(kv[3], h, acc[NKADJ + 2][k]);
          acc[NKADJ + 3][k] = fma(kv[4], h, acc[NKADJ + 3][k]);
        }
      };
      for (int c = 0; c < C0; ++c) accum(E, 0, c);
      for (int c = 0; c < C1; ++c) accum(O, 1, c);
      const int bt = r >> 1, comp = r & 1;
#pragma unroll
      for (int k = 0; k < INV_TJ; ++k) {
        int jp = j0 + k;
        if (jp >= Jh) break;
        int jn = jp, js = J - 1 - jp;
#pragma unroll
        for (int q = 0; q < NKADJ; ++q) {
          Cad[(((size_t)q * MT + bt) * J + jn) * 2 + comp] = E[q][k] + O[q][k];
          Cad[(((size_t)q * MT + bt) * J + js) * 2 + comp] = E[q][k] - O[q][k];
        }
#pragma unroll
        for (int q = NKADJ; q < NCAD; ++q) {
          Cad[(((size_t)q * MT + bt) * J + jn) * 2 + comp] = E[q][k] + O[q][k];
          Cad[(((size_t)q * MT + bt) * J + js) * 2 + comp] = O[q][k] - E[q][k];
        }
      }
    }
  }
  __syncthreads();
  // ---- phase 5: transposed combination -> adjoints of the state fields; Phibar gradient
  for (int t = threadIdx.x; t < MT * J; t += blockDim.x) {
    int bt = t / J, j = t % J;
    if (bt >= mt) continue;
    int b = b0 + bt;
    size_t o = ((size_t)m * G.B + b) * J + j;
    auto ld = [&](int q) { return mk<T2>(Cad[(((size_t)q * MT + bt) * J + j) * 2], Cad[(((size_t)q * MT + bt) * J + j) * 2 + 1]); };
    AdjPointIn<T> in;
    adj_load_point<T>(G, cfg, incr, FS, o, in);
    T gtd = (T)0;
    T gp = adj_store_point<T, NKADJ>(G, cfg, incr, FS, o, m, b, j, ld, in, gtd);
    if (G.grad) {
      // J is a multiple of 32, so a warp holds one member: reduce over the warp
      // in the compute type, accumulate the warp sums in FP64
#pragma unroll
      for (int off = 16; off > 0; off >>= 1) {
        gp += __shfl_xor_sync(0xffffffffu, gp, off);
        gtd += __shfl_xor_sync(0xffffffffu, gtd, off);
      }
      if ((threadIdx.x & 31) == 0) {
        sgrad[bt * nws + j / 32] = (double)gp;
        sgrad[(MT + bt) * nws + j / 32] = (double)gtd;
      }
    }
  }
  __syncthreads();
  if (G.grad && threadIdx.x < mt) {
    double acc = 0.0, acd = 0.0;
    for (int w = 0; w < nws; ++w) {
      acc += sgrad[threadIdx.x * nws + w];
      acd += sgrad[(MT + threadIdx.x) * nws + w];
    }
    atomicAdd(&G.grad[G_PHIBAR * G.B + b0 + threadIdx.x], acc);
    // the explicit scheme's own drag terms (modified Euler: its drag is the grid physics')
    if (cfg.scheme == 1) atomicAdd(&G.grad[G_TAUDRAG * G.B + b0 + threadIdx.x], acd);
  }
}

template <typename T, bool SMALL>
__global__ void __launch_bounds__(256) k_spectral_adj(const __grid_constant__ SpecLaunch<T> L) {
  pdl_enter();
  for_each_unit(L, [&](const SpecGroup<T>& G, int idx) { spectral_adj_unit<T, SMALL>(L, G, idx); });
}

namespace {
// CTAs of a persistent launch: every slot the kernel can keep resident, never
// more than the launch has units.
template <typename K>
int persistent_blocks(K kernel, int nunits, size_t smem) {
  static int nsm = 0;
  if (nsm == 0) {
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || nsm <= 0)
      nsm = 1;
  }
  int per_sm = 0;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, 256, smem) != cudaSuccess || per_sm < 1)
    per_sm = 1;
  return std::max(1, std::min(nunits, per_sm * nsm));
}

// Give the second basis block its own buffer where that costs no CTA per SM.
template <typename T>
SpecLaunch<T> with_early_inv(const SpecLaunch<T>& L0, size_t& smem) {
  SpecLaunch<T> L = L0;
  size_t extra = 0;
  for (int g = 0; g < L.ng; ++g)
    if (L.grp[g].B > 0) extra = std::max(extra, basis_bytes<T>(L.grp[g].g.M, L.grp[g].g.J) + 16);
  auto ctas = [](size_t n) { return (size_t)228 * 1024 / (n + 1024 + 128); };
  if (smem + extra <= (size_t)SPEC_DYN_SMEM_MAX && ctas(smem + extra) >= std::min<size_t>(ctas(smem), 2)) {
    smem += extra;
    L.early_inv = 1;
  }
  return L;
}
// CTAs of a launch: one per unit where all are resident at once (the unit counter
// would only add its round trips to L2, 4 us a launch), else persistent.
template <typename T, typename K>
int unit_blocks(SpecLaunch<T>& L, K kernel, int nunits, size_t smem) {
  if (!L.sched) return nunits;
  const int n = persistent_blocks(kernel, nunits, smem);
  if (n >= nunits) L.sched = nullptr;
  return n;
}
template <typename T>
bool small_units(const SpecLaunch<T>& L) {
  for (int g = 0; g < L.ng; ++g)
    if (L.grp[g].B > 0 && L.grp[g].MT > SMALL_MT) return false;
  return true;
}
}  // namespace

template <typename T>
cudaError_t launch_spec_adj(const SpecLaunch<T>& L0, int nblocks, size_t smem, cudaStream_t s) {
  if (nblocks <= 0) return cudaSuccess;
  SpecLaunch<T> L = with_early_inv(L0, smem);
  auto kernel = small_units(L) ? k_spectral_adj<T, true> : k_spectral_adj<T, false>;
  const int grid = unit_blocks(L, kernel, nblocks, smem);
  cudaError_t e = launch_pdl(kernel, grid, 256, smem, s, std::is_same<T, float>::value, L);
  return e != cudaSuccess ? e : cudaGetLastError();
}
template cudaError_t launch_spec_adj<float>(const SpecLaunch<float>&, int, size_t, cudaStream_t);

// Programmatic dependent launch of the FP32 step kernels, unless SWP_PDL=0.
bool pdl_enabled() {
  static const bool on = [] {
    const char* e = getenv("SWP_PDL");
    return !(e && e[0] == '0');
  }();
  return on;
}

void spec_set_attributes() {
  for (auto k : {k_spectral<double, false>, k_spectral<double, true>})
    cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, SPEC_DYN_SMEM_MAX);
  for (auto k : {k_spectral<float, false>, k_spectral<float, true>, k_spectral_adj<float, false>,
                 k_spectral_adj<float, true>})
    cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, SPEC_DYN_SMEM_MAX);
}

template <typename T>
cudaError_t launch_spec(const SpecLaunch<T>& L0, int nblocks, size_t smem, cudaStream_t s) {
  if (nblocks <= 0) return cudaSuccess;
  SpecLaunch<T> L = with_early_inv(L0, smem);
  auto kernel = small_units(L) ? k_spectral<T, true> : k_spectral<T, false>;
  const int grid = unit_blocks(L, kernel, nblocks, smem);
  cudaError_t e = launch_pdl(kernel, grid, 256, smem, s, std::is_same<T, float>::value, L);
  return e != cudaSuccess ? e : cudaGetLastError();
}
template cudaError_t launch_spec<double>(const SpecLaunch<double>&, int, size_t, cudaStream_t);
template cudaError_t launch_spec<float>(const SpecLaunch<float>&, int, size_t, cudaStream_t);

}  // namespace swp

// Building blocks of the grid kernels (grid.cu): the grid-space physics and
// its adjoint and tangent, the half-length C2R / R2C bin maps, double atomics
// and the group lookup of a launch.
#pragma once
#include <float.h>
#include "swp_internal.h"

namespace swp {

// x / pts with one reciprocal per point for all of its quotients.  FP32: x times
// the correctly rounded 1/pts (within 1 ulp of the quotient).  FP64: x inv and one
// residual correction (Markstein, IBM J. Res. Dev. 34, 1990), three instructions
// where a division takes about twelve, of the three the adjoint's point needs;
// outside the range in which the residual is exact, the division.
__device__ __forceinline__ float div_pts(float x, float inv, float) { return x * inv; }
__device__ __forceinline__ double div_pts(double x, double inv, double pts) {
  const double q = x * inv;
  const int ep = (__double2hiint(pts) >> 20) & 0x7ff, eq = (__double2hiint(q) >> 20) & 0x7ff;
  if ((unsigned)(ep - 523) <= 1000u && eq < 0x7ff) return fma(fma(-q, pts, x), inv, q);
  return x / pts;
}
__device__ __forceinline__ float recip_pts(float pts) { return __frcp_rn(pts); }
__device__ __forceinline__ double recip_pts(double pts) { return 1.0 / pts; }

template <typename T> __device__ __forceinline__ T tiny_val();
template <> __device__ __forceinline__ double tiny_val<double>() { return DBL_MIN; }
template <> __device__ __forceinline__ float tiny_val<float>() { return FLT_MIN; }

template <typename T>
__device__ __forceinline__ const GridGroup<T>& pick_ggroup(const GridLaunch<T>& L, int& idx, int block) {
  int gi = 0;
  while (gi + 1 < L.ng && block >= L.prefix[gi + 1]) ++gi;
  idx = block - L.prefix[gi];
  return L.grp[gi];
}
template <typename T>
__device__ __forceinline__ const GridGroup<T>& pick_ggroup(const GridLaunch<T>& L, int& idx) {
  return pick_ggroup(L, idx, (int)blockIdx.x);
}

// Half-length spectrum Z_k (k < L) of the C2R transform
//   x_i = Re(Y_0) + 2 Re sum_{m=1..M} Y_m e^{2 pi i m i / I},   x_{2n} + i x_{2n+1} = sum_k Z_k e^{2 pi i k n / L}
// from the truncated row y[m * ys], m = 0..M.  scale0 / scale multiply Y_0 / Y_m.
template <typename T2, typename T>
__device__ __forceinline__ T2 c2r_pre(const T2* y, int ys, int M, int L, int k, const T2* twI, T scale0, T scale) {
  T2 hk = mk<T2>(0, 0), hl = mk<T2>(0, 0);
  if (k == 0) { hk = mk<T2>(y[0].x * scale0, 0); }
  else if (k <= M) { hk = cscale(y[k * ys], scale); }
  int kl = L - k;  // partner index (k=0 -> L, which is > M)
  if (kl >= 1 && kl <= M) hl = cscale(y[kl * ys], scale);
  T2 fe = cadd(hk, cconj(hl));
  T2 fo = cmulc(csub(hk, cconj(hl)), twI[k]);  // * exp(+2 pi i k / I)
  T2 z; z.x = fe.x - fo.y; z.y = fe.y + fo.x;  // fe + i fo
  return z;
}

// Bin k (0..M) of the R2C transform from the half-length spectrum Z (after the
// forward FFT of x_{2n} + i x_{2n+1}), times `scale`.
template <typename T2, typename T>
__device__ __forceinline__ T2 r2c_post(const T2* Z, int L, int k, const T2* twI, T scale) {
  T2 zk = Z[k], zl = cconj(Z[(L - k) % L]);
  T2 e = cscale(cadd(zk, zl), (T)0.5);
  T2 d = csub(zk, zl);
  T2 o; o.x = (T)0.5 * d.y; o.y = (T)-0.5 * d.x;  // d / (2i)
  return cscale(cadd(e, cmul(o, twI[k])), scale);
}

// Extremes of doubles by integer atomics, which take one trip and no answer: above
// zero a double's bits order as its value, below in reverse.  NaN changes nothing.
__device__ __forceinline__ void atomic_min_d(double* addr, double v) {
  if (v != v) return;
  const long long k = __double_as_longlong(v + 0.0);  // -0 as 0
  if (k >= 0) atomicMin((long long*)addr, k);
  else atomicMax((unsigned long long*)addr, (unsigned long long)k);
}
__device__ __forceinline__ void atomic_max_d(double* addr, double v) {
  if (v != v) return;
  const long long k = __double_as_longlong(v + 0.0);
  if (k >= 0) atomicMax((long long*)addr, k);
  else atomicMin((unsigned long long*)addr, (unsigned long long)k);
}

// Order-preserving integers of floats and doubles.
template <typename T> struct Order;
template <> struct Order<float> {
  typedef int K;
  static __device__ __forceinline__ K flip(K b) { return b ^ ((b >> 31) & 0x7fffffff); }
  static __device__ __forceinline__ K key(float v) { return flip(__float_as_int(v)); }
  static __device__ __forceinline__ double value(K k) { return (double)__int_as_float(flip(k)); }
  static constexpr K INF_BITS = 0x7f800000;
};
template <> struct Order<double> {
  typedef long long K;
  static __device__ __forceinline__ K flip(K b) { return b ^ ((b >> 63) & 0x7fffffffffffffffll); }
  static __device__ __forceinline__ K key(double v) { return flip(__double_as_longlong(v)); }
  static __device__ __forceinline__ double value(K k) { return __longlong_as_double(flip(k)); }
  static constexpr K INF_BITS = 0x7ff0000000000000ll;
};

// The diagnostics of a step over a CTA's points: the area-weighted sum of squared
// speed, the least speed, the extremes of Phi (NaN counts for none of the three).
// All but the sum are compared as integers and the root is taken of the least
// square: an FP64 comparison is a trip through the slow pipe, and a chain of five
// shuffles and eight warps of them, retried CAS loops on the member's four words and
// a root per point made the diagnostics the larger part of a small run's step
// (M = 42, us per step without and with them: one member FP64 23.1 / 31.3, fast
// 15.3 / 24.6, 16 members fast 21.2 / 46.3; now 22.8 / 24.1, 15.2 / 18.0, 21.2 / 28.1).
template <typename T>
struct StepDiag {
  typedef typename Order<T>::K K;
  static constexpr K PINF = Order<T>::INF_BITS, NINF = ~PINF;  // the keys of +inf and -inf; NaN's are outside
  struct Block { double rms[8]; unsigned long long spin[8]; K lo[8], hi[8]; };
  double rms = 0.0;
  unsigned long long spin = 0x7ff0000000000000ull;  // bits of the least square, NaN's are above
  K lo = PINF, hi = NINF;
  __device__ __forceinline__ void speed(double aw, double s2) {
    rms += aw * s2;
    spin = min(spin, (unsigned long long)__double_as_longlong(s2));
  }
  __device__ __forceinline__ void phi(T p) {
    const K k = Order<T>::key(p);
    if (k < NINF || k > PINF) return;
    lo = min(lo, k);
    hi = max(hi, k);
  }
  // a warp's result to the block's slots (followed by a barrier)
  __device__ __forceinline__ void put(Block& s) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      rms += __shfl_down_sync(0xffffffffu, rms, o);
      spin = min(spin, __shfl_down_sync(0xffffffffu, spin, o));
      lo = min(lo, __shfl_down_sync(0xffffffffu, lo, o));
      hi = max(hi, __shfl_down_sync(0xffffffffu, hi, o));
    }
    if ((threadIdx.x & 31) == 0) {
      const int w = threadIdx.x >> 5;
      s.rms[w] = rms; s.spin[w] = spin; s.lo[w] = lo; s.hi[w] = hi;
    }
  }
  // the block's contribution to a member's row, one quantity per warp
  // (Phi's extremes only where dc is given)
  static __device__ __forceinline__ void add(const Block& s, double* dn, double* dc, int B, int b) {
    if ((threadIdx.x & 31) != 0) return;
    const int q = 7 - (threadIdx.x >> 5);
    if (q == 0) {
      double r = s.rms[0];
      for (int w = 1; w < 8; ++w) r += s.rms[w];
      atomicAdd(&dn[D_RMS2 * B + b], r);
    } else if (q == 1) {
      unsigned long long m = s.spin[0];
      for (int w = 1; w < 8; ++w) m = min(m, s.spin[w]);
      const double v = __longlong_as_double((long long)m);
      if (m < 0x7ff0000000000000ull) atomic_min_d(&dn[D_SPIN * B + b], sqrt(v));  // the least square is finite
    } else if (q == 2 && dc) {
      K m = s.lo[0];
      for (int w = 1; w < 8; ++w) m = min(m, s.lo[w]);
      atomic_min_d(&dc[D_PHIMIN * B + b], Order<T>::value(m));
    } else if (q == 3 && dc) {
      K m = s.hi[0];
      for (int w = 1; w < 8; ++w) m = max(m, s.hi[w]);
      atomic_max_d(&dc[D_PHIMAX * B + b], Order<T>::value(m));
    }
  }
};

template <typename T>
struct Physics {
  T Pb, itr, itd, DPe;
  bool nodrag, forced;
  __device__ __forceinline__ void eval(T eta, T Phi, T U, T V, T ihalf, T day_s, T* out) const {
    // ABCDE_init (initial_conditions.py:499-503)
    out[0] = U * eta; out[1] = V * eta; out[2] = U * Phi; out[3] = V * Phi;
    out[4] = (U * U + V * V) * ihalf;
    if (forced) {
      T Phieq = Pb + DPe * day_s;                        // forcing.py:55-60
      T Q = itr * (Phieq - (Phi + Pb));                  // forcing.py:94
      T Qc = Q < (T)0 ? (T)0 : Q;                        // forcing.py:133
      T pt = Phi + Pb;
      T pts = fabs(pt) > (T)0 ? pt : tiny_val<T>();     // forcing.py:139-140
      T r = div_pts(Qc, recip_pts(pts), pts);
      T Ru = -U * r, Rv = -V * r;
      out[5] = Q;
      out[6] = nodrag ? Ru : Ru - U * itd;               // forcing.py:143-153
      out[7] = nodrag ? Rv : Rv - V * itd;
    } else {
      out[5] = out[6] = out[7] = (T)0;
    }
  }
};

// Adjoint of Physics::eval.  lz = adjoints of (A, B, C, D, E, PhiF, F, G),
// lx = adjoints of (eta, Phi, U, V); gacc accumulates d/d(taurad, taudrag,
// DPhieq, Phibar).  The Q<0 clamp passes no gradient where Q<0 (the
// reference's jnp.where semantics); Phieq's Phibar cancels in Q.
template <typename T>
struct PhysicsAdj {
  T Pb, itr, itd, DPe;
  bool nodrag, forced;
  __device__ __forceinline__ void eval(T eta, T Phi, T U, T V, T ihalf, T day_s, const T* lz, T* lx,
                                       T* gacc) const {
    T lU = lz[0] * eta + lz[2] * Phi + lz[4] * (T)2 * U * ihalf;
    T lV = lz[1] * eta + lz[3] * Phi + lz[4] * (T)2 * V * ihalf;
    T leta = lz[0] * U + lz[1] * V;
    T lPhi = lz[2] * U + lz[3] * V;
    if (forced) {
      T Phieq = Pb + DPe * day_s;
      T Q = itr * (Phieq - (Phi + Pb));
      bool pos = !(Q < (T)0);
      T Qc = pos ? Q : (T)0;
      T pt = Phi + Pb;
      T pts = fabs(pt) > (T)0 ? pt : tiny_val<T>();
      const T ipts = recip_pts(pts);
      T r = div_pts(Qc, ipts, pts);
      T lF = lz[6], lG = lz[7];
      T lr = -U * lF - V * lG;
      T itdd = nodrag ? (T)0 : itd;
      lU += lF * (-r - itdd);
      lV += lG * (-r - itdd);
      T lQc = div_pts(lr, ipts, pts);
      T lpts = div_pts(-lr * r, ipts, pts);
      T lQ = lz[5] + (pos ? lQc : (T)0);
      lPhi += -itr * lQ + lpts;
      // per-thread partial sums in the compute type (two points per thread);
      // the block and global reductions run in FP64
      gacc[G_TAURAD] += lQ * (-Q * itr);
      if (!nodrag) gacc[G_TAUDRAG] += (lF * U + lG * V) * itd * itd;
      gacc[G_DPHIEQ] += lQ * itr * day_s;
      gacc[G_PHIBAR] += lpts;
    }
    lx[0] = leta; lx[1] = lPhi; lx[2] = lU; lx[3] = lV;
  }
};

// Tangent of Physics::eval (forward mode): x = (eta, Phi, U, V) with tangent
// dx, parameter tangents dp = d(taurad, taudrag, DPhieq, Phibar).  Same
// branch conventions as the adjoint: the clamp passes no tangent where Q < 0,
// Phieq's Phibar cancels in Q, taudrag = -1 has no drag term.
template <typename T>
struct PhysicsTL {
  T Pb, itr, itd, DPe;
  bool nodrag, forced;
  __device__ __forceinline__ void eval(T eta, T Phi, T U, T V, T deta, T dPhi, T dU, T dV, T ihalf, T day_s,
                                       const T* dp, T* out) const {
    out[0] = dU * eta + U * deta;
    out[1] = dV * eta + V * deta;
    out[2] = dU * Phi + U * dPhi;
    out[3] = dV * Phi + V * dPhi;
    out[4] = (T)2 * (U * dU + V * dV) * ihalf;
    if (forced) {
      T Phieq = Pb + DPe * day_s;
      T Q = itr * (Phieq - (Phi + Pb));
      // dQ = -itr dPhi - Q itr dtaurad + itr day_s dDPhieq
      T dQ = itr * (day_s * dp[G_DPHIEQ] - dPhi) - Q * itr * dp[G_TAURAD];
      bool pos = !(Q < (T)0);
      T Qc = pos ? Q : (T)0, dQc = pos ? dQ : (T)0;
      T pt = Phi + Pb;
      T pts = fabs(pt) > (T)0 ? pt : tiny_val<T>();
      const T ipts = recip_pts(pts);
      T r = div_pts(Qc, ipts, pts);
      T dr = div_pts(dQc - r * (dPhi + dp[G_PHIBAR]), ipts, pts);
      T dRu = -(dU * r + U * dr), dRv = -(dV * r + V * dr);
      out[5] = dQ;
      if (nodrag) {
        out[6] = dRu;
        out[7] = dRv;
      } else {
        // d(U / taudrag) = dU itd - U itd^2 dtaudrag
        const T ditd = itd * itd * dp[G_TAUDRAG];
        out[6] = dRu - dU * itd + U * ditd;
        out[7] = dRv - dV * itd + V * ditd;
      }
    } else {
      out[5] = out[6] = out[7] = (T)0;
    }
  }
};

}  // namespace swp

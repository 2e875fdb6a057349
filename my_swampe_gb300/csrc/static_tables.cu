// The parameter-dependent tables of the reference's Static (model.py:457-557)
// in one launch, where tensor expressions took about a hundred small ones
// (1.6 ms of a call's preparation).  One thread per entry or, for Phieq, pixel.  Parameter rows: dt, a,
// omega, g, Phibar, taurad, taudrag, DPhieq, K6, K6Phi.
#include "swp_internal.h"

namespace swp {
namespace {

__global__ void k_static_tables(const double* __restrict__ par, int n, const double* __restrict__ mu, int M, int J,
                                int I, int forced, double* __restrict__ out) {
  const int N1 = M + 1;
  const size_t nt = (size_t)n * N1, nj = (size_t)n * J, nf = (size_t)n * N1 * N1;
  const size_t total = 5 * nt + nj + n + nf;
  for (size_t u = (size_t)blockIdx.x * blockDim.x + threadIdx.x; u < total; u += (size_t)gridDim.x * blockDim.x) {
    auto P = [&](int row, size_t b) { return par[(size_t)row * n + b]; };
    size_t t = u;
    double v = 0.0;
    if (t < 5 * nt) {
      const int q = (int)(t / nt);
      t -= q * nt;
      const size_t b = t / N1;
      const double k = (double)(t % N1), dt = P(0, b), a = P(1, b);
      if (q == 0) {  // time_stepping.py:491-501
        v = k > 0.0 ? a / (k * (k + 1.0)) : a * 0.0;
      } else {  // filters.py:95-213
        const double a3 = a * a * a, K = (q & 1) ? P(8, b) : P(9, b);
        const double nc = ((k * k * k) / a3) * (((k + 1.0) * (k + 1.0) * (k + 1.0)) / a3);
        const double off = (q & 1) ? nc - 8.0 / (a3 * a3) : nc;  // eta, delta; Phi has no offset
        v = q <= 2 ? 1.0 / (1.0 + 2.0 * dt * K * off) : exp(-2.0 * dt * K * (off < 0.0 ? 0.0 : off));  // a NaN stays
      }
    } else if ((t -= 5 * nt) < nj) {  // time_stepping.py:516-522
      const size_t b = t / J;
      const double m = mu[t % J];
      v = (2.0 * P(0, b)) / (P(1, b) * (1.0 - __dmul_rn(m, m)));
    } else if ((t -= nj) < (size_t)n) {
      v = 2.0 * P(0, t) / (P(1, t) * P(1, t));
    } else if ((t -= n) < nf) {  // initial_conditions.py:295-316
      v = t % ((size_t)N1 * N1) == 1 ? P(2, t / ((size_t)N1 * N1)) / sqrt(0.375) : 0.0;
    }
    out[u] = v;
  }
  // Phieq: a thread per pixel, whose cosine and square root serve every member
  double* phieq = out + total;
  const int np = J * I;
  for (int q = blockIdx.x * blockDim.x + threadIdx.x; q < np; q += gridDim.x * blockDim.x) {
    const int i = q % I;  // forcing.py:14-62: strict dayside mask
    const double m = mu[q / I], pi = 3.141592653589793, lam = -pi + i * ((pi - (-pi)) / I);
    const bool day = forced && lam > -pi / 2.0 && lam < pi / 2.0;
    const double shape = day ? cos(lam) * sqrt(1.0 - __dmul_rn(m, m)) : 0.0;
    for (int b = 0; b < n; ++b)
      phieq[(size_t)b * np + q] = forced ? par[(size_t)4 * n + b] + (day ? __dmul_rn(par[(size_t)7 * n + b], shape) : 0.0) : 0.0;
  }
}

}  // namespace

cudaError_t launch_static_tables(const GroupGeom& gg, const double* params, int n, int forced, double* out,
                                 cudaStream_t s) {
  const size_t N1 = gg.M + 1, total = (size_t)n * (5 * N1 + gg.J + 1 + N1 * N1), pixels = (size_t)gg.J * gg.I;
  const size_t blocks = ((total > pixels ? total : pixels) + 255) / 256;
  k_static_tables<<<(int)(blocks < 152 * 8 ? blocks : 152 * 8), 256, 0, s>>>(params, n, gg.mu, gg.M, gg.J, gg.I,
                                                                            forced, out);
  return cudaGetLastError();
}

}  // namespace swp

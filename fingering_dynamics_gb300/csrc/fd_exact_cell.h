// One fluid cell of the FP64 step with fewer FP64 operations and the same
// bits, plain C++ so that it can be checked without a GPU.
//
// The FP64 pipe of sm_103a retires two results per clock and SM (an FP32 one
// 128), so the FP64 step's time is its count of FP64 operations.  Every
// rewriting below returns exactly what the reference's operand order
// (fd_physics.cuh) returns:
//   * products by 0 and +-1 of the velocity set are left out, and terms that
//     two opposite directions share up to sign are formed once (rounding to
//     nearest is symmetric);
//   * a product by a power of two is exact, so it moves into an FMA or past
//     another product: 4 E + (-4) W = 4 (E - W), 4 X + Y = fma(4, X, Y),
//     mu grad / 2, w_0 = 4 w_1 and w_5 = w_1 / 4 (true of the rounded weights);
//   * a / b for a constant b (12, 6, w_0) and for the divisors rho that several
//     quotients share, by Markstein's theorem (P. Markstein, Computation of
//     elementary functions on the IBM RISC System/6000 processor, IBM J. Res.
//     Dev. 34, 1990): with y = 1/b rounded to nearest and q within one ulp of
//     a / b, q + y (a - b q) in two FMAs is a / b rounded to nearest.
//     q = a y is that close when y's relative error is at most 2^-54 (it is
//     2^-54 for 1/12, 1/6 and 1/w_0); for rho one more correction makes it so.
// The rewritings need results and remainders that neither overflow nor lose
// bits below the normal range.  exact_cell() therefore checks the exponents of
// the quantities they act on and returns false where one is outside 2^-800 ..
// 2^800 and not zero (or not finite); the caller then evaluates the cell in
// the reference's own operand order.
#pragma once

#include <cmath>
#include <cstdint>
#include <cstring>

#ifdef __CUDACC__
#define FD_CELL __host__ __device__ __forceinline__
#else
#define FD_CELL inline
#endif

namespace fd {

struct ExactConst {
  double w0, w1;         // w_0 = 4/9, w_1 = 1/9 (w_5 = w_1 / 4)
  double y12, y6, yw0;   // 1/12, 1/6, 1/w_0
  double a, kappa;       // free-energy coefficients
  double eta_n, eta_n_M; // Eta_n, Eta_n * M
  double c_a0, c_b0, c_b18, one_third, tau_inv;
};

inline ExactConst make_exact_const(double w0, double w1, double a, double kappa, double eta_n, double eta_n_M,
                                   double c_a0, double c_b0, double c_b18, double one_third, double tau_inv) {
  return ExactConst{w0, w1, 1.0 / 12.0, 1.0 / 6.0, 1.0 / w0, a, kappa, eta_n, eta_n_M, c_a0, c_b0, c_b18, one_third, tau_inv};
}

FD_CELL double cell_fma(double a, double b, double c) {
#ifdef __CUDA_ARCH__
  return __fma_rn(a, b, c);
#else
  return std::fma(a, b, c);
#endif
}

// 1 / b rounded to nearest
FD_CELL double cell_rcp(double b) {
#ifdef __CUDA_ARCH__
  return __drcp_rn(b);
#else
  return 1.0 / b;
#endif
}

// true if v is zero or its magnitude lies in 2^-E .. 2^E (E = 800 or 100)
template <int E>
FD_CELL bool cell_in_range(double v) {
  uint64_t b;
#ifdef __CUDA_ARCH__
  b = (uint64_t)__double_as_longlong(v);
#else
  std::memcpy(&b, &v, 8);
#endif
  const uint32_t h = (uint32_t)(b >> 32) & 0x7fffffffu, l = (uint32_t)b;
  constexpr uint32_t lo = (uint32_t)(1023 - E) << 20, hi = (uint32_t)(1023 + E) << 20;
  return (h - lo) < (hi - lo) || (h | l) == 0u;
}

// a / b rounded to nearest for a constant b, y = 1 / b (see above)
FD_CELL double cell_div_const(double a, double b, double y) {
  const double q = a * y;
  return cell_fma(cell_fma(-b, q, a), y, q);
}

// a / b rounded to nearest, y = 1 / b rounded to nearest
FD_CELL double cell_div_shared(double a, double b, double y) {
  double q = a * y;
  q = cell_fma(cell_fma(-b, q, a), y, q);
  return cell_fma(cell_fma(-b, q, a), y, q);
}

// psi's derivatives of a 3x3 neighbourhood (fingering_periodic.py:214-256)
struct ExactStencil {
  double gx, gy, lap;
  bool ok;
};

FD_CELL ExactStencil exact_stencil(const ExactConst& k, double C, double E, double W, double N, double S, double NE,
                                   double NW, double SE, double SW) {
  const double nx = ((cell_fma(4.0, E - W, NE) - NW) - SW) + SE;
  const double ny = ((cell_fma(4.0, N - S, NE) + NW) - SW) - SE;
  double nl = cell_fma(4.0, N, -20.0 * C);
  nl = cell_fma(4.0, E, nl);
  nl = cell_fma(4.0, W, nl);
  nl = cell_fma(4.0, S, nl);
  nl = (((nl + NE) + NW) + SW) + SE;
  ExactStencil s;
  s.ok = cell_in_range<800>(nx) & cell_in_range<800>(ny) & cell_in_range<800>(nl);
  s.gx = cell_div_const(nx, 12.0, k.y12);
  s.gy = cell_div_const(ny, 12.0, k.y12);
  s.lap = cell_div_const(nl, 6.0, k.y6);
  return s;
}

// Macroscopic fields and collision of one fluid cell (fingering_periodic.py:
// 455-460, 470-479) from its pulled populations f, g, its psi and psi's
// derivatives.  On success f and g are the new populations; on failure (false)
// they are untouched.
FD_CELL bool exact_cell(const ExactConst& k, double psi, const ExactStencil& st, double (&f)[9], double (&g)[9]) {
  double rho = f[0];
#pragma unroll
  for (int i = 1; i < 9; ++i) rho = rho + f[i];
  const double mx = ((((f[1] - f[3]) + f[5]) - f[6]) - f[7]) + f[8];
  const double my = ((((f[2] - f[4]) + f[5]) + f[6]) - f[7]) - f[8];
  const double gx = st.gx, gy = st.gy;
  const double mu = ((k.a * psi) * (1.0 - psi * psi)) - k.kappa * st.lap;
  const double mgx = mu * gx, mgy = mu * gy;
  const double jx = cell_fma(0.5, mgx, mx), jy = cell_fma(0.5, mgy, my);
  const double y = cell_rcp(rho);
  const double ux = cell_div_shared(jx, rho, y), uy = cell_div_shared(jy, rho, y);
  const double p = k.one_third * rho + psi * mu;
  const double v1 = cell_div_shared(k.eta_n, rho, y), v2 = cell_div_shared(k.eta_n_M, rho, y);
  const double vv = v1 * v2;
  const double mv = vv / ((v1 * (1.0 - psi)) + (v2 * (1.0 + psi)));  // half of the mixed viscosity
  const double inv_t = cell_rcp(cell_fma(2.0, 3.0 * mv, 0.5));
  const double pref = cell_fma(-0.5, inv_t, 1.0);                     // 1 - 1 / (2 tau)
  const double na = rho - k.c_a0 * p, nb = psi - k.c_b0 * mu;
  const bool ok = st.ok & cell_in_range<100>(rho) & (rho != 0.0) & cell_in_range<800>(jx) & cell_in_range<800>(jy) &
                  cell_in_range<800>(k.eta_n) & cell_in_range<800>(k.eta_n_M) & cell_in_range<800>(vv) &
                  cell_in_range<800>(mgx) & cell_in_range<800>(mgy) & cell_in_range<800>(mu) & cell_in_range<800>(na) &
                  cell_in_range<800>(nb) & cell_in_range<100>(ux) & cell_in_range<100>(uy) & cell_in_range<100>(inv_t);
  if (!ok) return false;
  const double A0 = cell_div_const(na, k.w0, k.yw0), A = 3.0 * p;
  const double B0 = cell_div_const(nb, k.w0, k.yw0), B = k.c_b18 * mu;
  const double P = (mu * k.w1) * pref;  // forcing prefactor of w_1; 4 P and P / 4 are those of w_0 and w_5
  const double xx = ux * ux, yy = uy * uy;
  const double u15 = 1.5 * (xx + yy);
  // relaxation of one direction: SF = w_1's multiple of the forcing weight
#define FD_CELL_RELAX(I, WQ, AQ, BQ, Q, SF, S)                      \
  {                                                                 \
    const double q_ = (Q);                                          \
    const double fe = (WQ) * ((AQ) + rho * q_);                     \
    const double ge = (WQ) * ((BQ) + psi * q_);                     \
    f[I] = cell_fma(SF, P * (S), f[I] - inv_t * (f[I] - fe));       \
    g[I] = g[I] - k.tau_inv * (g[I] - ge);                          \
  }
  const double x3 = 3.0 * ux, y3 = 3.0 * uy;
  const double wx = x3 * gx, wy = y3 * gy;
  FD_CELL_RELAX(0, k.w0, A0, B0, -u15, 4.0, -(wx + wy));
  const double xp = (1.0 - ux) * 3.0, xm = (-1.0 - ux) * 3.0, yp = (1.0 - uy) * 3.0, ym = (-1.0 - uy) * 3.0;
  {
    const double s = 4.5 * xx, n = 9.0 * ux;
    FD_CELL_RELAX(1, k.w1, A, B, (x3 + s) - u15, 1.0, (xp + n) * gx - wy);
    FD_CELL_RELAX(3, k.w1, A, B, (s - x3) - u15, 1.0, (xm + n) * gx - wy);
  }
  {
    const double s = 4.5 * yy, n = 9.0 * uy;
    FD_CELL_RELAX(2, k.w1, A, B, (y3 + s) - u15, 1.0, (yp + n) * gy - wx);
    FD_CELL_RELAX(4, k.w1, A, B, (s - y3) - u15, 1.0, (ym + n) * gy - wx);
  }
  const double w5 = 0.25 * k.w1;
  {
    const double e = ux + uy, t = 3.0 * e, s = 4.5 * (e * e), n = 9.0 * e;
    FD_CELL_RELAX(5, w5, A, B, (t + s) - u15, 0.25, (xp + n) * gx + (yp + n) * gy);
    FD_CELL_RELAX(7, w5, A, B, (s - t) - u15, 0.25, (xm + n) * gx + (ym + n) * gy);
  }
  {
    const double e = uy - ux, t = 3.0 * e, s = 4.5 * (e * e), n = 9.0 * e;
    FD_CELL_RELAX(6, w5, A, B, (t + s) - u15, 0.25, (xm - n) * gx + (yp + n) * gy);
    FD_CELL_RELAX(8, w5, A, B, (s - t) - u15, 0.25, (xp - n) * gx + (ym + n) * gy);
  }
#undef FD_CELL_RELAX
  return true;
}

}  // namespace fd

// One fluid cell of the FP64 step with fewer FP64 operations and the same
// bits, plain C++ so that it can be checked without a GPU.
//
// The FP64 pipe of sm_103a retires two results per clock and SM (the FP32 one
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
// the reference's own operand order.  rho and 1 / tau stay within 2^+-100, psi, g
// and u within 2^+-400, so that their squares stay within 2^+-800: away from the
// interface u and g are products of rounding errors, 1e-36 and below, and with
// 2^+-100 for them too whole columns there were evaluated twice (a channel of
// 194 x 2372 ahead of the front: 311 -> 242 us per iteration over the first twenty).
#pragma once

#include <cmath>
#include <cstdint>
#include <cstring>

#ifdef __CUDACC__
#define FD_CELL __host__ __device__ __forceinline__
#define FD_CELL_CALL static __host__ __device__ __noinline__
#else
#define FD_CELL inline
#define FD_CELL_CALL inline
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

// true if v is zero or its magnitude lies in 2^-E .. 2^E
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
  return ((h - lo) < (hi - lo)) | ((h | l) == 0u);
}

FD_CELL uint64_t cell_bits(double v) {
#ifdef __CUDA_ARCH__
  return (uint64_t)__double_as_longlong(v);
#else
  uint64_t b;
  std::memcpy(&b, &v, 8);
  return b;
#endif
}
FD_CELL double cell_double(uint32_t hi, uint32_t lo) {
#ifdef __CUDA_ARCH__
  return __hiloint2double((int)hi, (int)lo);
#else
  const uint64_t b = ((uint64_t)hi << 32) | lo;
  double v;
  std::memcpy(&v, &b, 8);
  return v;
#endif
}

// a * b rounded to nearest even in integer arithmetic (the product of the two
// 53-bit significands, its top 53 bits, the rest as the rounding bits).  A zero
// operand gives a signed zero.  Operands and result must be zero or have
// exponents within +-800: `ok` is cleared where the result has not (operands
// are results that were checked before, or sums of them).
FD_CELL double cell_mul_int(double a, double b, bool& ok) {
  const uint64_t A = cell_bits(a), B = cell_bits(b);
  const uint32_t ah = (uint32_t)(A >> 32), al = (uint32_t)A, bh = (uint32_t)(B >> 32), bl = (uint32_t)B;
  const uint32_t Ah = ((ah << 11) | (al >> 21)) | 0x80000000u, Al = al << 11;
  const uint32_t Bh = ((bh << 11) | (bl >> 21)) | 0x80000000u, Bl = bl << 11;
  const uint64_t t = (uint64_t)Al * Bl;
  const uint64_t u = (uint64_t)Al * Bh + (t >> 32);
  const uint64_t v = (uint64_t)Ah * Bl + (uint32_t)u;
  const uint64_t h = (uint64_t)Ah * Bh + (u >> 32) + (v >> 32);  // significands' product / 2^64: bit 63 or 62 is set
  const uint32_t top = (uint32_t)(h >> 63), sh = 10u + top;
  const uint32_t rem = ((uint32_t)h << (32u - sh)) | (((uint32_t)v | (uint32_t)t) != 0u ? 1u : 0u);
  uint64_t m = h >> sh;
  m += (rem + ((uint32_t)m & 1u)) > 0x80000000u ? 1u : 0u;
  const uint32_t ea = ah & 0x7ff00000u, eb = bh & 0x7ff00000u;
  // the exponent field, one less because the leading bit of m adds one
  const uint32_t e = ea + eb + (top << 20) - (1024u << 20);
  const bool zero = (ea == 0u) | (eb == 0u);
  ok = ok & (zero | (e - (223u << 20) < (1600u << 20)));
  const uint32_t sign = (ah ^ bh) & 0x80000000u;
  return cell_double((zero ? 0u : (uint32_t)(m >> 32) + e) | sign, zero ? 0u : (uint32_t)m);
}

// N 2^X a rounded to nearest even in integer arithmetic (N = 3 or 9)
template <int N, int X>
FD_CELL double cell_scale_int(double a) {
  constexpr uint32_t L = N == 3 ? 1 : 3;  // floor(log2 N)
  static_assert(N == 3 || N == 9, "multipliers of the equilibria");
  const uint64_t A = cell_bits(a);
  const uint32_t ah = (uint32_t)(A >> 32);
  const uint64_t p = ((A & 0xfffffffffffffull) | 0x10000000000000ull) * (uint64_t)N;
  const uint32_t top = (uint32_t)(p >> (53 + L)), sh = L + top;
  const uint32_t rem = (uint32_t)p << (32u - sh);
  uint64_t m = p >> sh;
  m += (rem + ((uint32_t)m & 1u)) > 0x80000000u ? 1u : 0u;
  const uint32_t ea = ah & 0x7ff00000u;
  const uint32_t hi = (uint32_t)(m >> 32) + ea + ((top + L - 1u + (uint32_t)X) << 20);
  const bool zero = ea == 0u;
  return cell_double((zero ? 0u : hi) | (ah & 0x80000000u), zero ? 0u : (uint32_t)m);
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

// How many of a cell's products are formed in integer arithmetic (0: none, 58:
// all), in the order of their numbers below.  An integer product is about 40
// instructions, which the four schedulers issue in 10 clocks beside the FP64
// pipe, against the pipe's 16.  Ten iterations of 1024 x 2048: 11.7 ms with
// none, 10.0 with those of cell_relax (7), 8.4 with all; 25 of 400 x 400:
// 3.33, 2.85, 2.45 ms.
#ifndef FD_EXACT_INT_PRODUCTS
#define FD_EXACT_INT_PRODUCTS 58
#endif

// The products outside cell_relax are calls of one function: 33 copies of it took
// more instructions than the caches hold (2.8 stalls on a missing instruction per
// issue).  us per iteration at 128 threads, inlined -> called: 1024 x 2048 894 -> 844,
// 400 x 400 unchanged; those of cell_relax too: 843, but 400 x 400 97 -> 104.
struct CellProduct {
  double v;
  int ok;
};
FD_CELL_CALL CellProduct cell_mul_call(double a, double b) {
  bool ok = true;
  const double v = cell_mul_int(a, b, ok);
  return CellProduct{v, ok ? 1 : 0};
}

template <int K>
FD_CELL double cell_mul(double a, double b, bool& ok) {
  if constexpr (K >= FD_EXACT_INT_PRODUCTS) {
    return a * b;
  } else if constexpr (K < 7) {
    return cell_mul_int(a, b, ok);
  } else {
    const CellProduct r = cell_mul_call(a, b);
    ok = ok & (r.ok != 0);
    return r.v;
  }
}
template <int K, int N, int X>
FD_CELL double cell_scale(double a) {
  if constexpr (K < FD_EXACT_INT_PRODUCTS) return cell_scale_int<N, X>(a);
  else return (X < 0 ? 0.5 * N : (double)N) * a;
}

// New f (x) and g (y) of one direction: w (A + rho q), w (B + psi q) are the
// equilibria, SF P S the forcing.  f is NaN where a value left the range.  A
// function of its own on the GPU: nine copies of its integer products do not
// fit the instruction cache.
struct CellPair {
  double x, y;
};
FD_CELL_CALL CellPair cell_relax(double w, double A, double B, double rho, double psi, double q, double SF, double P,
                                 double S, double inv_t, double tau_inv, double f, double g) {
  bool ok = cell_in_range<400>(g);
  const double fe = cell_mul<0>(w, A + cell_mul<1>(rho, q, ok), ok);
  const double ge = cell_mul<2>(w, B + cell_mul<3>(psi, q, ok), ok);
  const double fn = cell_fma(SF, cell_mul<4>(P, S, ok), f - cell_mul<5>(inv_t, f - fe, ok));
  return CellPair{ok ? fn : cell_double(0x7ff80000u, 0u), g - cell_mul<6>(tau_inv, g - ge, ok)};
}

// Macroscopic fields of one fluid cell (fingering_periodic.py:470-479) from its
// density, pulled f, psi and psi's derivatives.
struct ExactMacro {
  double rho, ux, uy, p, mu, tau, psi, gx, gy;
  bool ok;  // every value in range
};

// The stored fields of a cell, for exact_collide (which checks the others): the
// ranges of exact_macros.
FD_CELL ExactMacro exact_stored(double rho, double ux, double uy, double p, double mu, double tau, double psi, double gx,
                                double gy) {
  return ExactMacro{rho, ux, uy, p, mu, tau, psi, gx, gy,
                    cell_in_range<100>(rho) && cell_in_range<400>(psi) && cell_in_range<800>(p) && cell_in_range<800>(gx) &&
                        cell_in_range<800>(gy)};
}

FD_CELL ExactMacro exact_macros(const ExactConst& k, double rho, double psi, const ExactStencil& st,
                                const double (&f)[9]) {
  ExactMacro m;
  const double mx = ((((f[1] - f[3]) + f[5]) - f[6]) - f[7]) + f[8];
  const double my = ((((f[2] - f[4]) + f[5]) + f[6]) - f[7]) - f[8];
  bool ok = st.ok & cell_in_range<100>(rho) & (rho != 0.0) & cell_in_range<400>(psi);
  const double mu = cell_mul<7>(k.a * psi, 1.0 - cell_mul<8>(psi, psi, ok), ok) - cell_mul<9>(k.kappa, st.lap, ok);
  const double mgx = cell_mul<10>(mu, st.gx, ok), mgy = cell_mul<11>(mu, st.gy, ok);
  const double jx = cell_fma(0.5, mgx, mx), jy = cell_fma(0.5, mgy, my);
  const double y = cell_rcp(rho);
  m.ux = cell_div_shared(jx, rho, y);
  m.uy = cell_div_shared(jy, rho, y);
  m.p = cell_mul<12>(k.one_third, rho, ok) + cell_mul<13>(psi, mu, ok);
  const double v1 = cell_div_shared(k.eta_n, rho, y), v2 = cell_div_shared(k.eta_n_M, rho, y);
  const double vv = cell_mul<14>(v1, v2, ok);
  // half of the mixed viscosity
  const double mv = vv / (cell_mul<15>(v1, 1.0 - psi, ok) + cell_mul<16>(v2, 1.0 + psi, ok));
  m.tau = cell_fma(2.0, 3.0 * mv, 0.5);
  m.rho = rho;
  m.mu = mu;
  m.psi = psi;
  m.gx = st.gx;
  m.gy = st.gy;
  m.ok = ok & cell_in_range<800>(jx) & cell_in_range<800>(jy) & cell_in_range<800>(k.eta_n) &
         cell_in_range<800>(k.eta_n_M) & cell_in_range<800>(vv) & cell_in_range<800>(mgx) & cell_in_range<800>(mgy);
  return m;
}

// Collision of one fluid cell (fingering_periodic.py:455-460) from its
// macroscopic fields and f; g_i comes from load_g(i) and the new populations go
// to store(i, f, g).  False: what was stored must not be used, the caller
// evaluates the cell otherwise.
template <typename LoadG, typename Store>
FD_CELL bool exact_collide(const ExactConst& k, const ExactMacro& m, const double (&f)[9], LoadG load_g, Store store) {
  const double rho = m.rho, ux = m.ux, uy = m.uy, p = m.p, mu = m.mu, psi = m.psi, gx = m.gx, gy = m.gy;
  bool ok = m.ok;
  const double inv_t = cell_rcp(m.tau);
  const double pref = cell_fma(-0.5, inv_t, 1.0);  // 1 - 1 / (2 tau)
  const double na = rho - cell_mul<17>(k.c_a0, p, ok), nb = psi - cell_mul<18>(k.c_b0, mu, ok);
  ok = ok & cell_in_range<800>(mu) & cell_in_range<800>(na) & cell_in_range<800>(nb) & cell_in_range<400>(ux) &
       cell_in_range<400>(uy) & cell_in_range<100>(inv_t);
  const double A0 = cell_div_const(na, k.w0, k.yw0), A = cell_scale<40, 3, 0>(p);
  const double B0 = cell_div_const(nb, k.w0, k.yw0), B = cell_mul<19>(k.c_b18, mu, ok);
  // forcing prefactor of w_1; 4 P and P / 4 are those of w_0 and w_5
  const double P = cell_mul<20>(cell_mul<21>(mu, k.w1, ok), pref, ok);
  const double xx = cell_mul<22>(ux, ux, ok), yy = cell_mul<23>(uy, uy, ok);
  const double u15 = cell_scale<41, 3, -1>(xx + yy);
  const double x3 = cell_scale<42, 3, 0>(ux), y3 = cell_scale<43, 3, 0>(uy);
  const double wx = cell_mul<24>(x3, gx, ok), wy = cell_mul<25>(y3, gy, ok);
  // one direction: weight, constant parts of its equilibria, q, scale of its forcing, S
  auto relax = [&](int i, double w, double Aq, double Bq, double q, double SF, double S) {
    const CellPair r = cell_relax(w, Aq, Bq, rho, psi, q, SF, P, S, inv_t, k.tau_inv, f[i], load_g(i));
    ok &= ((uint32_t)(cell_bits(r.x) >> 32) & 0x7ff00000u) != 0x7ff00000u;
    store(i, r.x, r.y);
  };
  relax(0, k.w0, A0, B0, -u15, 4.0, -(wx + wy));
  const double xp = cell_scale<44, 3, 0>(1.0 - ux), xm = cell_scale<45, 3, 0>(-1.0 - ux);
  const double yp = cell_scale<46, 3, 0>(1.0 - uy), ym = cell_scale<47, 3, 0>(-1.0 - uy);
  {
    const double s = cell_scale<48, 9, -1>(xx), n = cell_scale<49, 9, 0>(ux);
    const double S1 = cell_mul<26>(xp + n, gx, ok) - wy, S3 = cell_mul<27>(xm + n, gx, ok) - wy;
    relax(1, k.w1, A, B, (x3 + s) - u15, 1.0, S1);
    relax(3, k.w1, A, B, (s - x3) - u15, 1.0, S3);
  }
  {
    const double s = cell_scale<50, 9, -1>(yy), n = cell_scale<51, 9, 0>(uy);
    const double S2 = cell_mul<28>(yp + n, gy, ok) - wx, S4 = cell_mul<29>(ym + n, gy, ok) - wx;
    relax(2, k.w1, A, B, (y3 + s) - u15, 1.0, S2);
    relax(4, k.w1, A, B, (s - y3) - u15, 1.0, S4);
  }
  const double w5 = 0.25 * k.w1;
  {
    const double e = ux + uy, t = cell_scale<52, 3, 0>(e), s = cell_scale<53, 9, -1>(cell_mul<30>(e, e, ok));
    const double n = cell_scale<54, 9, 0>(e);
    const double S5 = cell_mul<31>(xp + n, gx, ok) + cell_mul<32>(yp + n, gy, ok);
    const double S7 = cell_mul<33>(xm + n, gx, ok) + cell_mul<34>(ym + n, gy, ok);
    relax(5, w5, A, B, (t + s) - u15, 0.25, S5);
    relax(7, w5, A, B, (s - t) - u15, 0.25, S7);
  }
  {
    const double e = uy - ux, t = cell_scale<55, 3, 0>(e), s = cell_scale<56, 9, -1>(cell_mul<35>(e, e, ok));
    const double n = cell_scale<57, 9, 0>(e);
    const double S6 = cell_mul<36>(xm - n, gx, ok) + cell_mul<37>(yp + n, gy, ok);
    const double S8 = cell_mul<38>(xp - n, gx, ok) + cell_mul<39>(ym + n, gy, ok);
    relax(6, w5, A, B, (t + s) - u15, 0.25, S6);
    relax(8, w5, A, B, (s - t) - u15, 0.25, S8);
  }
  return ok;
}

// Both, for the fused step.
template <typename LoadG, typename Store>
FD_CELL bool exact_cell(const ExactConst& k, double psi, const ExactStencil& st, const double (&f)[9], LoadG load_g,
                        Store store) {
  double rho = f[0];
#pragma unroll
  for (int i = 1; i < 9; ++i) rho = rho + f[i];
  return exact_collide(k, exact_macros(k, rho, psi, st, f), f, load_g, store);
}

}  // namespace fd

// Entering and leaving the fused mode in one kernel each.
//
// fd_enter: fd_boundary_fields, fd_collide and fd_pack of a state.  The three
// kernels read the populations twice; one pass reads them once.
//
// fd_finish: the pending part of an iteration - stream, bounce-back, Zou-He, rho,
// psi and the macroscopic fields (fingering_periodic.py:461-479) - from the
// fused state (packed or in the reference's layout) into the reference's layout
// and fields.  The seven kernels it stands for (unpack, stream, bounce-back,
// two for Zou-He, rho and psi, macroscopic fields) move the populations four
// times; here each is read once and written once: a CTA owns a tile of 32 x 4
// cells, every thread pulls its cell's populations, psi of the tile and one cell
// around it goes through shared memory, and the stencils follow after one
// barrier, as in fd_tile.cuh.  Bound by memory on large lattices, by launches on
// small ones.
//
// Built with -fmad=false: the arithmetic is the per-function kernels', bit for
// bit (fd_ref.cu).
#include "fd_exact_cell.h"
#include "fd_fused_dev.cuh"
#include "fd_host.h"
#include "fd_zouhe.cuh"

namespace fd {
namespace {

constexpr int kFinTX = 32, kFinTY = 4;

template <typename T>
struct FinFields {
  T *f, *g, *psi, *npx, *npy, *np2, *rho, *ux, *uy, *p, *mu, *mix_tau;
};

template <typename T>
FinFields<T> fin_fields(const fd_fields& a) {
  return FinFields<T>{(T*)a.f,   (T*)a.g,  (T*)a.psi, (T*)a.npx, (T*)a.npy, (T*)a.np2,
                      (T*)a.rho, (T*)a.ux, (T*)a.uy,  (T*)a.p,   (T*)a.mu,  (T*)a.mix_tau};
}

inline ExactConst fin_const(const Coef<double>& c) {
  return make_exact_const(c.w[0], c.w[1], c.a, c.kappa, c.eta_n, c.eta_n_M, c.c_a0, c.c_b0, c.c_b18, c.one_third,
                          c.tau_inv);
}

// The fused state as the per-function kernels see it: 18 planes of T, or packed
// deviations converted as fd_unpack converts them.
template <typename T>
struct RefSource {
  const T* f;
  const T* g;
  size_t P;
  __device__ __forceinline__ T load_f(int i, size_t q) const { return f[i * P + q]; }
  __device__ __forceinline__ T load_g(int i, size_t q) const { return g[i * P + q]; }
};

template <typename T, typename SF>
struct PackedSource {
  const SF* f;
  const float* g0;
  const SF* gi;
  size_t pstride;
  float inv_sf, inv_sg;
  float w[9];
  __device__ __forceinline__ T load_f(int i, size_t q) const { return (T)(to_f<SF>(f[i * pstride + q]) * inv_sf + w[i]); }
  __device__ __forceinline__ T load_g(int i, size_t q) const {
    return i == 0 ? (T)g0[q] : (T)(to_f<SF>(gi[(i - 1) * pstride + q]) * inv_sg);
  }
};

struct FinShape {
  int H, W, variant, ntx;
  size_t P;
};

// Pulled populations of one cell: stream with wrap-around, then bounce-back links
template <bool G, typename T, typename Src>
__device__ __forceinline__ void fin_pull(const Src& src, const FinShape& s, int x, int y, unsigned bits, T (&v)[9]) {
  const size_t row[3] = {(size_t)wrap(y - 1, s.H) * s.W, (size_t)y * s.W, (size_t)wrap(y + 1, s.H) * s.W};
  const int col[3] = {wrap(x - 1, s.W), x, wrap(x + 1, s.W)};
#pragma unroll
  for (int i = 0; i < 9; ++i) {
    const bool link = i > 0 && ((bits >> (i - 1)) & 1u);
    const size_t q = link ? row[1] + col[1] : row[1 - ey_of(i)] + col[1 - ex_of(i)];
    const int k = link ? opp_of(i) : i;
    v[i] = G ? src.load_g(k, q) : src.load_f(k, q);
  }
}

// psi of a lattice cell from its pulled g (which Zou-He updates)
template <typename T>
__device__ __forceinline__ T fin_psi(const Coef<T>& c, const FinShape& s, int x, int y, unsigned m, T (&g)[9]) {
  if (x == 0 || x == s.W - 1) zou_he_g(c, s.variant, s.H, s.W, x, y, g);
  return (m & SOLID) ? c.psi_wall : sum9(g);
}

template <typename T, typename Src>
__global__ void __launch_bounds__(kFinTX* kFinTY) k_finish(FinShape s, Coef<T> c, ExactConst k, Src src,
                                                            const uint16_t* __restrict__ mask,
                                                            const double* __restrict__ inlet_ux,
                                                            const T* __restrict__ side, FinFields<T> F) {
  constexpr int PW = kFinTX + 2;
  __shared__ T psi[(kFinTY + 2) * PW];
  const int t = threadIdx.x, lx = t & 31, ly = t >> 5;
  const int x0 = (int)(blockIdx.x % s.ntx) * kFinTX, y0 = (int)(blockIdx.x / s.ntx) * kFinTY;
  const int x = x0 + lx, y = y0 + ly;
  const bool in = x < s.W && y < s.H;
  const size_t q = (size_t)y * s.W + x;
  const unsigned m = in ? mask[q] : 0u;
  T f[9], g[9];
  if (in) {
    fin_pull<true>(src, s, x, y, m & 0xFFu, g);
    fin_pull<false>(src, s, x, y, m & 0xFFu, f);
  }
  // psi of the cells that no thread of the tile owns: around it, and past the lattice's last row and column
  for (int e = t; e < (kFinTY + 2) * PW; e += kFinTX * kFinTY) {
    const int px = e % PW - 1, py = e / PW - 1;
    int hx = x0 + px, hy = y0 + py;
    if (hx > s.W || hy > s.H) continue;
    if (px >= 0 && px < kFinTX && py >= 0 && py < kFinTY && hx < s.W && hy < s.H) continue;
    T v;
    if (s.variant == FD_VARIANT_WALLS && (hy < 0 || hy >= s.H)) {
      v = c.psi_wall;
    } else if (s.variant != FD_VARIANT_PERIODIC_XY && (hx < 0 || hx >= s.W)) {
      v = hx < 0 ? T(1) : T(-1);
    } else {
      hx = wrap(hx, s.W);
      hy = wrap(hy, s.H);
      const unsigned hm = mask[(size_t)hy * s.W + hx];
      T gh[9];
      if (!(hm & SOLID)) fin_pull<true>(src, s, hx, hy, hm & 0xFFu, gh);
      v = (hm & SOLID) ? c.psi_wall : fin_psi(c, s, hx, hy, hm, gh);
    }
    psi[e] = v;
  }
  const T* ps = psi + (ly + 1) * PW + lx + 1;
  if (in) psi[(ly + 1) * PW + lx + 1] = fin_psi(c, s, x, y, m, g);
  __syncthreads();
  if (!in) return;
  if ((x == 0 || x == s.W - 1) && s.variant != FD_VARIANT_PERIODIC_XY) {
    const int o = (x == 0) ? 0 : 3;
    T rho_nb = T(0);
    if (s.variant == FD_VARIANT_WALLS && x == 0 && (y == 0 || y == s.H - 1)) {
      const int yn = y == 0 ? 1 : s.H - 2;
      T fn[9];
      fin_pull<false>(src, s, 0, yn, mask[(size_t)yn * s.W] & 0xFFu, fn);
      rho_nb = inlet_rho(fn, (T)inlet_ux[yn], side[0 * s.H + yn], side[2 * s.H + yn]);
    }
    zou_he_f(c, s.variant, s.H, s.W, x, y, f, (T)inlet_ux[y], side[(o + 0) * s.H + y], side[(o + 1) * s.H + y],
             side[(o + 2) * s.H + y], rho_nb);
  }
#pragma unroll
  for (int i = 0; i < 9; ++i) {
    F.f[i * s.P + q] = f[i];
    F.g[i * s.P + q] = g[i];
  }
  const T C = ps[0], E = ps[1], Wv = ps[-1], N = ps[PW], S = ps[-PW];
  const T NE = ps[PW + 1], NW = ps[PW - 1], SE = ps[1 - PW], SW = ps[-1 - PW];
  F.psi[q] = C;
  T gx, gy, lap;
  ExactStencil st{};
  if constexpr (sizeof(T) == 8) {
    st = exact_stencil(k, C, E, Wv, N, S, NE, NW, SE, SW);
    gx = st.gx;
    gy = st.gy;
    lap = st.lap;
  }
  if (sizeof(T) == 4 || !st.ok) {
    gx = grad_x(E, Wv, NE, NW, SE, SW);
    gy = grad_y(N, S, NE, NW, SE, SW);
    lap = laplacian(C, E, Wv, N, S, NE, NW, SE, SW);
  }
  F.npx[q] = gx;
  F.npy[q] = gy;
  F.np2[q] = lap;
  if (m & SOLID) return;
  const T rho = sum9(f);
  F.rho[q] = rho;
  if constexpr (sizeof(T) == 8) {
    if (!c.body) {
      const ExactMacro e = exact_macros(k, rho, C, st, f);
      if (e.ok) {
        F.mu[q] = e.mu; F.ux[q] = e.ux; F.uy[q] = e.uy; F.p[q] = e.p; F.mix_tau[q] = e.tau;
        return;
      }
    }
  }
  const T mu = chem_pot(c, C, lap);
  F.mu[q] = mu;
  F.ux[q] = velocity_c(c, mom_x(f), mu, gx, rho, c.bx);
  F.uy[q] = velocity_c(c, mom_y(f), mu, gy, rho, c.by);
  F.p[q] = pressure_of(c, rho, C, mu);
  F.mix_tau[q] = mix_tau_of(c, rho, C);
}

template <typename T, typename Src>
int launch_finish(const fd_params& p, const uint16_t* mask, const Src& src, const void* side, const double* inlet_ux,
                  const fd_fields& out, cudaStream_t st) {
  const FinShape s{p.H, p.W, p.variant, (p.W + kFinTX - 1) / kFinTX, (size_t)p.H * p.W};
  const unsigned blocks = (unsigned)s.ntx * (unsigned)((p.H + kFinTY - 1) / kFinTY);
  ExactConst k{};
  if constexpr (sizeof(T) == 8) k = fin_const(make_coef<double>(p));
  k_finish<T, Src><<<blocks, kFinTX * kFinTY, 0, st>>>(s, make_coef<T>(p), k, src, mask, inlet_ux, (const T*)side,
                                                        fin_fields<T>(out));
  return check_launch("fd_finish");
}

template <typename T, typename SF>
int finish_packed(const fd_params& p, const uint16_t* mask, const fd_storage& st, const void* src, const void* side,
                  const double* inlet_ux, const fd_fields& out, cudaStream_t s) {
  const PackedLayout<SF> L = packed_layout<SF>(p.H, p.W);
  const DevCoef c = make_dev_coef(p, st.f_scale_log2, st.g_scale_log2);
  const char* b = (const char*)src;
  PackedSource<T, SF> ps{reinterpret_cast<const SF*>(b + L.off_f), reinterpret_cast<const float*>(b + L.off_g0),
                         reinterpret_cast<const SF*>(b + L.off_gi), L.pstride, c.inv_sf, c.inv_sg, {}};
  for (int i = 0; i < 9; ++i) ps.w[i] = c.w[i];
  return launch_finish<T>(p, mask, ps, side, inlet_ux, out, s);
}

template <typename T>
int finish_any(const fd_params& p, const uint16_t* mask, const fd_storage* st, const void* src, const void* side,
               const double* inlet_ux, const fd_fields& out, cudaStream_t s) {
  if (st == nullptr) {
    const size_t P = (size_t)p.H * p.W;
    return launch_finish<T>(p, mask, RefSource<T>{(const T*)src, (const T*)src + 9 * P, P}, side, inlet_ux, out, s);
  }
  switch (st->dtype) {
    case FD_F16: return finish_packed<T, __half>(p, mask, *st, src, side, inlet_ux, out, s);
    case FD_BF16: return finish_packed<T, __nv_bfloat16>(p, mask, *st, src, side, inlet_ux, out, s);
    default: return finish_packed<T, float>(p, mask, *st, src, side, inlet_ux, out, s);
  }
}

// ---- entering: boundary values, collision, packed copy ------------------------
// psi of (x, y) as the stencils see it (fd_ref.cu, psi_nb)
template <typename T>
__device__ __forceinline__ T enter_psi(const FinShape& s, T psi_wall, const T* __restrict__ psi,
                                       const uint16_t* __restrict__ mask, int x, int y) {
  if (y < 0 || y >= s.H) {
    if (s.variant == FD_VARIANT_WALLS) return psi_wall;
    y = wrap(y, s.H);
  }
  if (s.variant == FD_VARIANT_PERIODIC_XY) {
    x = wrap(x, s.W);
  } else {
    if (x < 0) return T(1);
    if (x >= s.W) return T(-1);
  }
  const size_t q = (size_t)y * s.W + x;
  return (mask[q] & SOLID) ? psi_wall : psi[q];
}

template <typename SF>
__global__ void __launch_bounds__(256) k_enter(FinShape s, Coef<float> c, DevCoef d, const uint16_t* __restrict__ mask,
                                               FinFields<float> F, float* __restrict__ side, size_t pstride,
                                               SF* __restrict__ pf, float* __restrict__ pg0, SF* __restrict__ pg) {
  const size_t q = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (q >= s.P) return;
  const unsigned m = mask[q];
  const int x = (int)(q % s.W), y = (int)(q / s.W);
  if (x == 0 || x == s.W - 1) {  // fd_boundary_fields
    auto nb = [&](int dx, int dy) { return enter_psi(s, c.psi_wall, F.psi, mask, x + dx, y + dy); };
    const float E = nb(1, 0), Wv = nb(-1, 0), N = nb(0, 1), S = nb(0, -1);
    const float NE = nb(1, 1), NW = nb(-1, 1), SE = nb(1, -1), SW = nb(-1, -1);
    const float gx = grad_x(E, Wv, NE, NW, SE, SW), gy = grad_y(N, S, NE, NW, SE, SW);
    const float mu = chem_pot(c, F.psi[q], F.np2[q]);
    for (int col = 0; col < 2; ++col) {
      if (x != (col ? s.W - 1 : 0)) continue;
      side[(3 * col + 0) * s.H + y] = gx;
      side[(3 * col + 1) * s.H + y] = gy;
      side[(3 * col + 2) * s.H + y] = mu;
    }
  }
  float f[9], g[9];
#pragma unroll
  for (int i = 0; i < 9; ++i) { f[i] = F.f[i * s.P + q]; g[i] = F.g[i * s.P + q]; }
  if (!(m & SOLID)) {  // fd_collide
    Macro<float> mc;
    mc.rho = F.rho[q]; mc.ux = F.ux[q]; mc.uy = F.uy[q]; mc.p = F.p[q]; mc.mu = F.mu[q];
    mc.tau_mix = F.mix_tau[q]; mc.psi = F.psi[q]; mc.gx = F.npx[q]; mc.gy = F.npy[q];
    collide(c, mc, f, g);
#pragma unroll
    for (int i = 0; i < 9; ++i) { F.f[i * s.P + q] = f[i]; F.g[i * s.P + q] = g[i]; }
  }
#pragma unroll
  for (int i = 0; i < 9; ++i) pf[i * pstride + q] = from_f<SF>((f[i] - d.w[i]) * d.sf);  // fd_pack
  pg0[q] = g[0];
#pragma unroll
  for (int i = 1; i < 9; ++i) pg[(i - 1) * pstride + q] = from_f<SF>(g[i] * d.sg);
}

template <typename SF>
int launch_enter(const fd_params& p, const uint16_t* mask, const fd_fields& fl, void* side, const fd_storage& st,
                 void* dst, cudaStream_t s) {
  const PackedLayout<SF> L = packed_layout<SF>(p.H, p.W);
  const FinShape sh{p.H, p.W, p.variant, 0, L.P};
  char* b = (char*)dst;
  k_enter<SF><<<(unsigned)((L.P + 255) / 256), 256, 0, s>>>(
      sh, make_coef<float>(p), make_dev_coef(p, st.f_scale_log2, st.g_scale_log2), mask, fin_fields<float>(fl),
      (float*)side, L.pstride, reinterpret_cast<SF*>(b + L.off_f), reinterpret_cast<float*>(b + L.off_g0),
      reinterpret_cast<SF*>(b + L.off_gi));
  return check_launch("fd_enter");
}

int check_fields(const fd_fields* a, const char* what) {
  FD_REQUIRE(a && a->f && a->g && a->psi && a->npx && a->npy && a->np2 && a->rho && a->ux && a->uy && a->p && a->mu &&
                 a->mix_tau,
             FD_ERR_ARG, "%s: NULL pointer", what);
  return FD_OK;
}

}  // namespace
}  // namespace fd

using namespace fd;

extern "C" {

int fd_enter(const fd_params* prm, const uint16_t* mask, const fd_fields* fields, void* side, const fd_storage* st,
             void* dst, void* stream) {
  if (int r = check_params(prm)) return r;
  if (int r = check_fields(fields, "fd_enter")) return r;
  FD_REQUIRE(mask && side && dst, FD_ERR_ARG, "fd_enter: NULL pointer");
  FD_REQUIRE(fd_packed_bytes(prm->H, prm->W, st) != 0, FD_ERR_ARG, "fd_enter: invalid storage");
  cudaStream_t s = as_stream(stream);
  switch (st->dtype) {
    case FD_F16: return launch_enter<__half>(*prm, mask, *fields, side, *st, dst, s);
    case FD_BF16: return launch_enter<__nv_bfloat16>(*prm, mask, *fields, side, *st, dst, s);
    default: return launch_enter<float>(*prm, mask, *fields, side, *st, dst, s);
  }
}

int fd_finish(const fd_params* prm, int dtype, const uint16_t* mask, const fd_storage* st, const void* src,
              const void* side, const double* inlet_ux, const fd_fields* out, void* stream) {
  if (int r = check_params(prm)) return r;
  FD_REQUIRE(dtype == FD_F64 || dtype == FD_F32, FD_ERR_DTYPE, "fd_finish: dtype %d not supported", dtype);
  if (int r = check_fields(out, "fd_finish")) return r;
  FD_REQUIRE(mask && src && side && inlet_ux, FD_ERR_ARG, "fd_finish: NULL pointer");
  FD_REQUIRE(src != out->f, FD_ERR_ARG, "fd_finish: source and destination must differ");
  FD_REQUIRE(st == nullptr || fd_packed_bytes(prm->H, prm->W, st) != 0, FD_ERR_ARG, "fd_finish: invalid storage");
  cudaStream_t s = as_stream(stream);
  return dtype == FD_F64 ? finish_any<double>(*prm, mask, st, src, side, inlet_ux, *out, s)
                         : finish_any<float>(*prm, mask, st, src, side, inlet_ux, *out, s);
}

}  // extern "C"

// FP64 fused step: one kernel per iteration of the reference's loop body, bit
// for bit the reference's arithmetic (the state between kernels is that of
// fd_fused.cuh).
//
// The kernel is bound by the FP64 pipe, which spends 16 clocks on a warp
// instruction whatever number of its lanes is active; so the FP64 work is done
// on full warps.  A CTA owns a tile of 32 x TY cells:
//   1. psi = sum g of the tile and one cell around it, into shared memory (g
//      is pulled from global memory: stream, bounce-back, Zou-He g), and a
//      ballot per 32 cells of the cells that need arithmetic (fluid cells, and
//      the inlet and outlet columns);
//   2. the list of those cells, compacted; the other cells, solid ones, only
//      stream, so their pulled populations are copied at once;
//   3. each thread takes cells from the list: psi stencils from shared memory,
//      f and g pulled again (g from L1 / L2), Zou-He, macroscopic fields and
//      collision (exact_cell), stores.
// A group of 32 cells is 32 / TY columns x TY rows, so the cells of the inlet or
// outlet column of a tile share a warp and the Zou-He arithmetic is issued once
// per tile, not once per row; a row of a group is at least a 32-byte sector.
//
// Measured on GB300 (1024 x 2048, porosity 0.7), per iteration: 2.3 ms with one
// thread per pair of cells in the reference's operand order (solid lanes idle,
// twelve divisions, the products by 0 and 1 evaluated); 1.05 ms with full warps
// and the rewritings of fd_exact_cell.h (369 FP64 instructions per 32 fluid
// cells, the pipe 84% busy, one issue slot in ten used); 0.89 ms with the
// products in integer arithmetic (250 FP64 instructions), 0.82 with those in
// calls and a thread per cell of a tile of 8 rows.
//
// Cells whose values leave the range that exact_cell() takes (a diverging run),
// and the body-force variant, are evaluated in the reference's operand order by
// exact_slow_cell().
#pragma once

#include "fd_exact_cell.h"
#include "fd_fused.cuh"

namespace fd {

constexpr int kExactTX = 32;
// CTAs per SM that the registers are cut for: 96 registers at 128 threads (tiles of
// 4 rows), 80 at 256 (8 rows; 128 threads x 5 845 us per iteration of 1024 x 2048,
// 128 x 4 831, 192 x 4 852, 256 x 2 903, 256 x 3 819)
constexpr int exact_min_ctas(int nt) { return nt == 128 ? 5 : 3; }

struct ExactArgs {
  FusedArgs<double> a;
  ExactConst k;
  int ntx;  // tiles per row of tiles
};

// Pulled populations of one cell: stream with wrap-around, then bounce-back links.
__device__ __forceinline__ double exact_pull_one(const double* __restrict__ planes, size_t P, int H, int W, int x,
                                                 int y, unsigned bits, int i) {
  size_t src = (size_t)i * P + (size_t)wrap(y - ey_of(i), H) * W + wrap(x - ex_of(i), W);
  if (i > 0 && ((bits >> (i - 1)) & 1u)) src = (size_t)opp_of(i) * P + (size_t)y * W + x;
  return __ldg(planes + src);
}
__device__ __forceinline__ void exact_pull(const double* __restrict__ planes, size_t P, int H, int W, int x, int y,
                                           unsigned bits, double (&v)[9]) {
#pragma unroll
  for (int i = 0; i < 9; ++i) v[i] = exact_pull_one(planes, P, H, W, x, y, bits, i);
}

__device__ __forceinline__ void exact_store(const FusedArgs<double>& a, size_t P, size_t q, const double (&f)[9],
                                            const double (&g)[9]) {
#pragma unroll
  for (int i = 0; i < 9; ++i) {
    a.dst[(size_t)i * P + q] = f[i];
    a.dst[(size_t)(9 + i) * P + q] = g[i];
  }
}

// Zou-He f of a cell of column 0 or W-1, and the boundary values of this
// iteration for the next one (fingering_periodic.py:146-149 reads the stored
// psi and laplacian); `ps`: the cell's psi in the tile, rows `pw` apart.
__device__ __forceinline__ void exact_boundary(const FusedArgs<double>& a, size_t P, int x, int y, const double* ps,
                                               int pw, double (&f)[9]) {
  const int o = (x == 0) ? 0 : 3;
  double rho_nb = 0.0;
  if (a.variant == FD_VARIANT_WALLS && x == 0 && (y == 0 || y == a.H - 1))
    rho_nb = rho_inlet_row(a, P, y == 0 ? 1 : a.H - 2);
  zou_he_f(a.c, a.variant, a.H, a.W, x, y, f, a.inlet_ux[y], a.side_in[(o + 0) * a.H + y],
           a.side_in[(o + 1) * a.H + y], a.side_in[(o + 2) * a.H + y], rho_nb);
  const double C = ps[0], E = ps[1], Wv = ps[-1], N = ps[pw], S = ps[-pw];
  const double NE = ps[pw + 1], NW = ps[pw - 1], SE = ps[1 - pw], SW = ps[-1 - pw];
  a.side_out[(o + 0) * a.H + y] = grad_x(E, Wv, NE, NW, SE, SW);
  a.side_out[(o + 1) * a.H + y] = grad_y(N, S, NE, NW, SE, SW);
  a.side_out[(o + 2) * a.H + y] = chem_pot(a.c, C, laplacian(C, E, Wv, N, S, NE, NW, SE, SW));
}

// One fluid cell in the reference's own operand order, from the pull to the store.
__device__ __noinline__ void exact_slow_cell(const FusedArgs<double>& a, int x, int y, unsigned bits, const double* ps,
                                             int pw) {
  const size_t P = (size_t)a.H * a.W;
  double f[9], g[9];
  exact_pull(a.src, P, a.H, a.W, x, y, bits, f);
  exact_pull(a.src + 9 * P, P, a.H, a.W, x, y, bits, g);
  if (x == 0 || x == a.W - 1) {
    zou_he_g(a.c, a.variant, a.H, a.W, x, y, g);
    if (a.variant != FD_VARIANT_PERIODIC_XY) exact_boundary(a, P, x, y, ps, pw, f);
  }
  const double C = ps[0], E = ps[1], Wv = ps[-1], N = ps[pw], S = ps[-pw];
  const double NE = ps[pw + 1], NW = ps[pw - 1], SE = ps[1 - pw], SW = ps[-1 - pw];
  const Macro<double> m = macros_of(a.c, f, C, grad_x(E, Wv, NE, NW, SE, SW), grad_y(N, S, NE, NW, SE, SW),
                                    laplacian(C, E, Wv, N, S, NE, NW, SE, SW));
  collide(a.c, m, f, g);
  exact_store(a, P, (size_t)y * a.W + x, f, g);
}

template <int TY, int NT>
__global__ void __launch_bounds__(NT, exact_min_ctas(NT)) k_exact_step(const __grid_constant__ ExactArgs ea) {
  constexpr int CW = 32 / TY, CHUNKS = kExactTX / CW, PW = kExactTX + 2;
  static_assert(TY * CW == 32 && CHUNKS * CW == kExactTX, "a group of 32 cells is CW columns of the tile");
  __shared__ double psi[(TY + 2) * PW];
  __shared__ double edge_g[2][TY][9];  // g of the inlet and outlet column's cells after Zou-He
  __shared__ unsigned need[CHUNKS];
  __shared__ uint16_t list[CHUNKS * 32];
  const FusedArgs<double>& a = ea.a;
  const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
  const int x0 = (int)(blockIdx.x % ea.ntx) * kExactTX, y0 = (int)(blockIdx.x / ea.ntx) * TY;
  const size_t P = (size_t)a.H * a.W;
  const bool walls = a.variant == FD_VARIANT_WALLS, xy = a.variant == FD_VARIANT_PERIODIC_XY;
  auto cell_of = [&](int e, int& lx, int& ly) {
    lx = (e >> 5) * CW + (e & (CW - 1));
    ly = (e & 31) / CW;
  };

  // 1. psi of the tile and its surroundings; which cells need arithmetic
  for (int e = t; e < (TY + 2) * PW; e += NT) {
    const int px = e % PW - 1, py = e / PW - 1;
    int x = x0 + px, y = y0 + py;
    if (x > a.W || y > a.H) continue;  // past the ghost cells of a tile that the lattice ends in
    double v;
    if (walls && (y < 0 || y >= a.H)) {
      v = a.c.psi_wall;
    } else if (!xy && (x < 0 || x >= a.W)) {
      v = x < 0 ? 1.0 : -1.0;
    } else {
      x = wrap(x, a.W);
      y = wrap(y, a.H);
      const unsigned m = a.mask[(size_t)y * a.W + x];
      const bool edge = !xy && (x == 0 || x == a.W - 1);
      if ((m & SOLID) && !edge) {
        v = a.c.psi_wall;
      } else {
        double g[9];
        exact_pull(a.src + 9 * P, P, a.H, a.W, x, y, m & 0xFFu, g);
        if (edge) {
          zou_he_g(a.c, a.variant, a.H, a.W, x, y, g);
          if (py >= 0 && py < TY && px >= 0 && px < kExactTX) {
#pragma unroll
            for (int i = 0; i < 9; ++i) edge_g[x == 0 ? 0 : 1][py][i] = g[i];
          }
        }
        v = (m & SOLID) ? a.c.psi_wall : sum9(g);
      }
    }
    psi[e] = v;
  }
  for (int c = warp; c < CHUNKS; c += NT / 32) {
    int lx, ly;
    cell_of(c * 32 + lane, lx, ly);
    const int x = x0 + lx, y = y0 + ly;
    const bool in = x < a.W && y < a.H;
    const bool take = in && ((!xy && (x == 0 || x == a.W - 1)) || !(a.mask[(size_t)y * a.W + x] & SOLID));
    const unsigned b = __ballot_sync(0xffffffffu, take);
    if (lane == 0) need[c] = b;
  }
  __syncthreads();

  // 2. the list of cells that need arithmetic; the others stream
  int total = 0;
  for (int c = 0, mine = warp; c < CHUNKS; ++c) {
    const unsigned b = need[c];
    if (c == mine) {
      mine += NT / 32;
      const int e = c * 32 + lane;
      if ((b >> lane) & 1u) {
        list[total + __popc(b & ((1u << lane) - 1u))] = (uint16_t)e;
      } else {
        int lx, ly;
        cell_of(e, lx, ly);
        const int x = x0 + lx, y = y0 + ly;
        if (x < a.W && y < a.H) {
          const size_t q = (size_t)y * a.W + x;
          const unsigned bits = a.mask[q] & 0xFFu;
          double v[9], w[9];
          exact_pull(a.src, P, a.H, a.W, x, y, bits, v);
          exact_pull(a.src + 9 * P, P, a.H, a.W, x, y, bits, w);
          exact_store(a, P, q, v, w);
        }
      }
    }
    total += __popc(b);
  }
  __syncthreads();

  // 3. the cells of the list
  for (int i = t; i < total; i += NT) {
    int lx, ly;
    cell_of(list[i], lx, ly);
    const int x = x0 + lx, y = y0 + ly;
    const size_t q = (size_t)y * a.W + x;
    const unsigned m = a.mask[q];
    const double* ps = psi + (ly + 1) * PW + lx + 1;
    if (xy) {
      exact_slow_cell(a, x, y, m & 0xFFu, ps, PW);
      continue;
    }
    const unsigned bits = m & 0xFFu;
    double f[9];
    exact_pull(a.src, P, a.H, a.W, x, y, bits, f);
    const bool edge = x == 0 || x == a.W - 1;
    if (edge) exact_boundary(a, P, x, y, ps, PW, f);
    auto load_g = [&](int i) {
      return edge ? edge_g[x == 0 ? 0 : 1][ly][i] : exact_pull_one(a.src + 9 * P, P, a.H, a.W, x, y, bits, i);
    };
    auto store = [&](int i, double fn, double gn) {
      a.dst[(size_t)i * P + q] = fn;
      a.dst[(size_t)(9 + i) * P + q] = gn;
    };
    if (m & SOLID) {  // of the inlet or outlet column
#pragma unroll
      for (int i = 0; i < 9; ++i) store(i, f[i], edge_g[x == 0 ? 0 : 1][ly][i]);
      continue;
    }
    const ExactStencil st = exact_stencil(ea.k, ps[0], ps[1], ps[-1], ps[PW], ps[-PW], ps[PW + 1], ps[PW - 1],
                                          ps[1 - PW], ps[-1 - PW]);
    if (!exact_cell(ea.k, ps[0], st, f, load_g, store)) exact_slow_cell(a, x, y, bits, ps, PW);
  }
}

template <int TY>
int launch_exact(ExactArgs& ea, const fd_params& p, double* pa, double* pb, double* sa, double* sb, int nsteps,
                 cudaStream_t st) {
  constexpr int NT = 32 * TY;  // one cell a thread
  ea.ntx = (p.W + kExactTX - 1) / kExactTX;
  const unsigned blocks = (unsigned)ea.ntx * (unsigned)((p.H + TY - 1) / TY);
  for (int s = 0; s < nsteps; ++s) {
    const bool even = (s % 2) == 0;
    ea.a.src = even ? pa : pb;
    ea.a.dst = even ? pb : pa;
    ea.a.side_in = even ? sa : sb;
    ea.a.side_out = even ? sb : sa;
    k_exact_step<TY, NT><<<blocks, NT, 0, st>>>(ea);
  }
  return cudaGetLastError() == cudaSuccess ? FD_OK : FD_ERR_CUDA;
}

}  // namespace fd

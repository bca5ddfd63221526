// Fused step, packed deviation storage, one thread per cell: the kernel of
// small lattices and of widths that are not a multiple of 8.
//
// The staged kernel (fd_fused_tma.cuh) marches down strips of rows, about a
// microsecond a row, and needs thousands of band-rows to fill the GPU; a lattice
// of 64 x 128 has four strips.  Here a CTA owns a tile of 32 x TY cells and
// nothing marches: every thread pulls the g populations of its cell (and some
// threads those of one cell around the tile) straight from global memory, psi
// goes to shared memory, and after one barrier each thread forms its stencils,
// pulls f, collides and stores.  A step's time is then one chain of mask, g and
// f loads, so the launches are made programmatic: a step's CTAs start while the
// previous step drains, load their masks, and wait for it before they touch
// the populations.
//
// Measured, us per step (the kernel before -> this one): FP32 64 x 128 27.6 -> 3.4
// and 380 x 380 15.7 -> 6.2, BF16 1021 x 1500 82 -> 41.4 (there it is bound by
// instruction issue; 47.5 with 64-bit addresses).  Tiles of 4 rows: 8 rows lose 7-11% on FP32 from 1024 x 1024
// up and gain on single sizes below (256 x 512 6.2 vs 7.0).
//
// The arithmetic and the rounding of the stores are those of the kernel that the
// width had before, bit for bit (RING: the staged kernel's, widths that are
// multiples of 8; else those of the lane-per-two-cells kernel that other widths
// ran on: FP32 reciprocals rounded to nearest, scalar collision, one random word
// per stored value), so a lattice's results do not depend on its size class.
#pragma once

#include "fd_fused_tma.cuh"
#include "fd_pdl.cuh"

namespace fd {

constexpr int kTileTX = 32;

// The elements a cell pulls from, as byte offsets of type I from the first plane
// (32-bit ones where nine planes are below 4 GB, which load and store
// instructions add to a uniform base: 64-bit address arithmetic was a fifth of
// the kernel's instructions).  Rows wrap; columns do not: what streams in across
// x = 0 and x = W - 1 is replaced by the Zou-He rules, and an element before or
// after a row lies inside the packed buffer for every direction that asks for one.
template <typename SF, typename I>
struct TilePull {
  I row[3];  // the cell's element in rows y-1, y, y+1
  __device__ __forceinline__ TilePull(int x, int y, int H, int W)
      : row{el(x, wrap(y - 1, H), W), el(x, y, W), el(x, wrap(y + 1, H), W)} {}
  static __device__ __forceinline__ I el(int x, int y, int W) { return ((I)y * (I)W + (I)x) * (I)sizeof(SF); }
  // population i streams from (x - e_x, y - e_y)
  __device__ __forceinline__ I from(int i) const { return row[1 - ey_of(i)] - (I)(ex_of(i) * (int)sizeof(SF)); }
  __device__ __forceinline__ I own() const { return row[1]; }
  __device__ __forceinline__ I pull(int i, unsigned bits, I plane) const {  // plane: bytes of one
    const bool link = i > 0 && ((bits >> (i - 1)) & 1u);
    return link ? (I)opp_of(i) * plane + own() : (I)i * plane + from(i);
  }
};

// Loads of the state go to L2 (ld.global.cg): the SM's L1 may hold lines of the
// buffer from the step before the previous one, which ran until after this
// kernel had started.
template <typename S, bool RING, bool SCALED>
__device__ __forceinline__ float tile_ld(const S* p, float scale) {
  const S v = __ldcg(p);
  if constexpr (std::is_same_v<S, float>) return v;
  else if constexpr (RING && !SCALED) return to_f<S>(v);
  else return to_f<S>(v) * scale;
}

// f of a cell: stream, then the bounce-back links (the opposite population of the same cell)
template <typename SF, bool RING, bool SCALED, typename I>
__device__ __forceinline__ void tile_pull_f(const DevArgs<SF>& a, const TilePull<SF, I>& t, unsigned bits, float (&v)[9]) {
  const I plane = (I)a.pstride_f * (I)sizeof(SF);
#pragma unroll
  for (int i = 0; i < 9; ++i)
    v[i] = tile_ld<SF, RING, SCALED>(byte_at(a.src_f, t.pull(i, bits, plane)), a.c.inv_sf);
}

template <typename SF, bool RING, bool SCALED, typename I>
__device__ __forceinline__ void tile_pull_g(const DevArgs<SF>& a, const TilePull<SF, I>& t, unsigned bits, float (&v)[9]) {
  const I plane = (I)a.pstride_f * (I)sizeof(SF);
  const SF* before = a.src_gi - a.pstride_f;  // a plane before g_1's, so that every offset is positive
  v[0] = __ldcg(byte_at(a.src_g0, t.own() * (I)(4 / sizeof(SF))));
#pragma unroll
  for (int i = 1; i < 9; ++i)
    v[i] = tile_ld<SF, RING, SCALED>(byte_at(before, t.pull(i, bits, plane)), a.c.inv_sg);
}

// psi of a lattice cell from its pulled g after Zou-He (g is updated)
template <typename SF, bool RING>
__device__ __forceinline__ float2 tile_psi(const DevArgs<SF>& a, int x, int y, unsigned m, float (&g)[9]) {
  if (x == 0 || x == a.W - 1) dev_zou_he_g(a.c, a.variant, a.H, a.W, x, y, g);
  if (m & SOLID) return make_float2(a.c.psi_wall, 0.0f);
  if constexpr (std::is_same_v<SF, float>) {
    return dev_psi_pair(g);
  } else if constexpr (RING) {
    const float2 s = __fadd2_rn(__fadd2_rn(make_float2(g[1], g[2]), make_float2(g[3], g[4])),
                                __fadd2_rn(make_float2(g[5], g[6]), make_float2(g[7], g[8])));
    return make_float2(g[0] + (s.x + s.y), 0.0f);
  } else {
    const float S = ((g[1] + g[2]) + (g[3] + g[4])) + ((g[5] + g[6]) + (g[7] + g[8]));
    return make_float2(g[0] + S, 0.0f);
  }
}

// psi of a tile and one cell around it.  FP32 storage carries psi as a pair; in
// the staged kernel's arithmetic a neighbour outside the cell's own column has
// passed through that kernel's ring, whose lo parts are scaled FP16.
template <typename SF, bool RING, int TY>
struct TilePsi {
  static constexpr int PW = kTileTX + 2;
  static constexpr bool PAIR = std::is_same_v<SF, float>;
  float hi[(TY + 2) * PW];
  float lo[PAIR ? (TY + 2) * PW : 1];
  __device__ __forceinline__ void put(int e, float2 v) {
    hi[e] = v.x;
    if constexpr (PAIR) lo[e] = v.y;
  }
  __device__ __forceinline__ float2 exact(int e) const { return make_float2(hi[e], PAIR ? lo[e] : 0.0f); }
  __device__ __forceinline__ float2 near(int e) const {
    if constexpr (PAIR && RING)
      return make_float2(hi[e], __half2float(__float2half_rn(lo[e] * kPsiLoScale)) * kPsiLoInv);
    else return exact(e);
  }
  __device__ __forceinline__ DevStencil stencil(int e) const {
    if constexpr (PAIR)
      return dev_stencil_pair(exact(e), near(e + 1), near(e - 1), exact(e + PW), exact(e - PW), near(e + PW + 1),
                              near(e + PW - 1), near(e - PW + 1), near(e - PW - 1));
    else
      return dev_stencil(hi[e], hi[e + 1], hi[e - 1], hi[e + PW], hi[e - PW], hi[e + PW + 1], hi[e + PW - 1],
                         hi[e - PW + 1], hi[e - PW - 1]);
  }
};

// Stores of one cell in the arithmetic of widths that are not a multiple of 8
template <typename SF, bool STOCH, typename I>
__device__ __forceinline__ void tile_store_scalar(const DevArgs<SF>& a, uint32_t seed, I q, const float (&f)[9],
                                                  const float (&g)[9]) {
  uint32_t rs = 0;
  if constexpr (STOCH) rs = sr_hash((uint32_t)q ^ seed);
  auto conv = [&](float v, float scale) -> SF {
    if constexpr (STOCH) {
      rs = sr_next(rs);
      return from_f_sr<SF>(v * scale, rs);
    } else if constexpr (std::is_same_v<SF, float>) {
      return v;
    } else {
      return from_f<SF>(v * scale);
    }
  };
#pragma unroll
  for (int i = 0; i < 9; ++i) *plane_el(a.dst_f, a.pstride_f, i, q) = conv(f[i], a.c.sf);
  *plane_el(a.dst_g0, 0, 0, q) = g[0];
#pragma unroll
  for (int i = 1; i < 9; ++i) *plane_el(a.dst_gi, a.pstride_f, i - 1, q) = conv(g[i], a.c.sg);
}

// rho_inlet - 1 of row yn (1 or H-2) of the walled variant's inlet column
// (fingering.py:341, 357), as inlet_corner_drho, from f pulled through L2.
template <typename SF, bool RING, bool SCALED, typename I>
__device__ __forceinline__ float tile_corner_drho(const DevArgs<SF>& a, int yn) {
  float d[9];
  tile_pull_f<SF, RING, SCALED>(a, TilePull<SF, I>(0, yn, a.H, a.W), a.mask[(size_t)yn * a.W] & 0xFFu, d);
  return dev_inlet_drho(d, (float)a.inlet_ux[yn], __ldcg(a.side_in + yn), __ldcg(a.side_in + 2 * a.H + yn));
}

// What a step of a lattice of its own knows of its state: always stepped, the launch's seed.
struct TileAlone {
  uint32_t seed;
  __device__ __forceinline__ bool stepped() const { return true; }
  __device__ __forceinline__ uint32_t step_seed() const { return seed; }
};

// Tile `tile` (of `ntx` in a row of tiles) of one lattice.  `ready` is called
// before the first access to the populations and returns the step's state.
template <typename SF, bool RING, bool SCALED, bool STOCH, int TY, typename I, typename Ready>
__device__ __forceinline__ void tile_cells_step(const DevArgs<SF>& a, int ntx, int tile, TilePsi<SF, RING, TY>& psi,
                                                Ready ready) {
  using Psi = TilePsi<SF, RING, TY>;
  constexpr int PW = Psi::PW;
  const int t = threadIdx.x, lx = t & 31, ly = t >> 5;
  const int x0 = (tile % ntx) * kTileTX, y0 = (tile / ntx) * TY;
  const int x = x0 + lx, y = y0 + ly;
  const bool walls = a.variant == FD_VARIANT_WALLS;
  const bool in = x < a.W && y < a.H;
  // the cell around the tile that this thread also does: below, above, left, right
  int hx = 0, hy = 0;
  bool halo = t < 2 * PW + 2 * TY;
  if (t < 2 * PW) {
    hx = t % PW - 1;
    hy = t < PW ? -1 : TY;
  } else if (halo) {
    hx = t < 2 * PW + TY ? -1 : kTileTX;
    hy = (t - 2 * PW) % TY;
  }
  const int he = (hy + 1) * PW + hx + 1;
  hx += x0;
  hy += y0;
  halo = halo && hx <= a.W && hy <= a.H;  // past the ghost cells of a tile that the lattice ends in
  const bool hwall = walls && (hy < 0 || hy >= a.H), hghost = hx < 0 || hx >= a.W;
  const bool hcell = halo && !hwall && !hghost;
  if (hcell) hy = wrap(hy, a.H);
  const unsigned m = in ? __ldg(a.mask + (size_t)y * a.W + x) : 0u;
  const unsigned hm = hcell ? __ldg(a.mask + (size_t)hy * a.W + hx) : 0u;
  const auto state = ready();

  float g[9], f[9];
  const TilePull<SF, I> at(x, in ? y : 0, a.H, a.W);
  if (in) {
    tile_pull_g<SF, RING, SCALED>(a, at, m & 0xFFu, g);
    tile_pull_f<SF, RING, SCALED>(a, at, m & 0xFFu, f);
  }
  if (halo) {
    float2 v = make_float2(hx < 0 ? 1.0f : -1.0f, 0.0f);
    if (hwall) {
      v.x = a.c.psi_wall;
    } else if (hcell) {
      float gh[9];
      tile_pull_g<SF, RING, SCALED>(a, TilePull<SF, I>(hx, hy, a.H, a.W), hm & 0xFFu, gh);
      v = tile_psi<SF, RING>(a, hx, hy, hm, gh);
    }
    psi.put(he, v);
  }
  const int e = (ly + 1) * PW + lx + 1;
  if (in) {
    psi.put(e, tile_psi<SF, RING>(a, x, y, m, g));
  } else if (y <= a.H && x <= a.W) {
    // a ghost cell inside the tile (the lattice ends in it): past the last column, or the row above the top
    // one (psi_wall, or row 0 of the periodic variant)
    float2 v = make_float2(-1.0f, 0.0f);
    if (y == a.H && walls) {
      v.x = a.c.psi_wall;
    } else if (y == a.H && x < a.W) {
      const unsigned gm = __ldg(a.mask + x);
      float gh[9];
      tile_pull_g<SF, RING, SCALED>(a, TilePull<SF, I>(x, 0, a.H, a.W), gm & 0xFFu, gh);
      v = tile_psi<SF, RING>(a, x, 0, gm, gh);
    }
    psi.put(e, v);
  }
  __syncthreads();
  bool bad = false;  // a fluid cell with a non-finite rho or psi
  if (in && state.stepped()) {
    const DevStencil st = psi.stencil(e);
    if (x == 0 || x == a.W - 1) {
      const int o = (x == 0) ? 0 : 3;
      float drho_nb = 0.0f;
      if (walls && x == 0 && (y == 0 || y == a.H - 1))
        drho_nb = tile_corner_drho<SF, RING, SCALED, I>(a, y == 0 ? 1 : a.H - 2);
      dev_zou_he_f(a.c, a.variant, a.H, a.W, x, y, f, (float)a.inlet_ux[y], __ldcg(a.side_in + (o + 0) * a.H + y),
                   __ldcg(a.side_in + (o + 1) * a.H + y), __ldcg(a.side_in + (o + 2) * a.H + y), drho_nb);
      a.side_out[(o + 0) * a.H + y] = st.gx;
      a.side_out[(o + 1) * a.H + y] = st.gy;
      a.side_out[(o + 2) * a.H + y] = dev_mu(a.c, st);
    }
    if (!(m & SOLID)) {
      const DevMacro mc = dev_macros<RING && !std::is_same_v<SF, float>>(a.c, f, st);
      bad = nonfinite_cell(mc.rho, mc.psi);
      if constexpr (RING) dev_collide_for<SF>(a.c, mc, f, g);
      else dev_collide(a.c, mc, f, g);
    }
    if constexpr (RING) store_cell<SF, SCALED, STOCH, I>(a, state.step_seed(), at.own() / (I)sizeof(SF), f, g);
    else tile_store_scalar<SF, STOCH, I>(a, state.step_seed(), at.own() / (I)sizeof(SF), f, g);
  }
  if (__any_sync(0xffffffffu, bad) && lx == 0) report_nonfinite(a);
}

// The previous step has ended, and the next one may start (only now: a step that
// started before the step two before it had ended could overwrite what that one reads).
__device__ __forceinline__ void tile_step_begins() {
  pdl_wait();
  pdl_launch_dependents();
}

// MINB: CTAs per SM that the registers are cut for (launch_tile)
template <typename SF, bool RING, bool SCALED, bool STOCH, int TY, typename I, int MINB>
__global__ void __launch_bounds__(32 * TY, MINB) k_tile_step(const __grid_constant__ DevArgs<SF> a, int ntx) {
  __shared__ TilePsi<SF, RING, TY> psi;
  tile_cells_step<SF, RING, SCALED, STOCH, TY, I>(a, ntx, (int)blockIdx.x, psi, [&] {
    tile_step_begins();
    return TileAlone{a.seed};
  });
}

#ifndef FD_TILE_TY
#define FD_TILE_TY 4
#endif
// Cells up to which the registers are cut for 8 CTAs per SM (more loads of a cell
// in flight), above which for 10 (more cells in flight).  us per step, 8 / 10:
// FP32 380 x 380 6.2 / 6.8, 512 x 1024 14.6 / 14.6, 768 x 1024 26.4 / 25.4, 1021 x
// 1500 49.7 / 47.6; BF16 380 x 380 6.3 / 7.0, 1021 x 1500 42.4 / 41.4.
constexpr size_t kTileFewCells = 600000;

template <typename SF, bool RING, bool SCALED, bool STOCH>
int launch_tile(const fd_params& p, const DevCoef& c, const uint16_t* mask, const double* inlet_ux, char* pa, char* pb,
                float* sa, float* sb, int nsteps, uint32_t seed, cudaStream_t st) {
  constexpr int TY = FD_TILE_TY;
  const PackedLayout<SF> L = packed_layout<SF>(p.H, p.W);
  DevArgs<SF> a{};
  a.c = c;
  a.H = p.H;
  a.W = p.W;
  a.variant = p.variant;
  a.P = L.P;
  a.pstride_f = L.pstride;
  a.mask = mask;
  a.inlet_ux = inlet_ux;
  const int ntx = (p.W + kTileTX - 1) / kTileTX;
  const unsigned blocks = (unsigned)ntx * (unsigned)((p.H + TY - 1) / TY);
  for (int s = 0; s < nsteps; ++s) {
    const bool even = s % 2 == 0;
    tma_set_step(a, even ? pa : pb, even ? pb : pa, even ? sa : sb, even ? sb : sa, seed + (uint32_t)s);
    // the first step's masks may have been written by the work just before it
    auto go = [&](auto kern) { return launch_pdl(kern, blocks, 32 * TY, 0, st, s > 0, a, ntx); };
    cudaError_t e;
    if (9 * L.pstride * sizeof(SF) >= ((size_t)1 << 32)) {
      if constexpr (RING) return FD_ERR_SHAPE;  // not reached: lattices of this size take the staged kernel
      else e = go(k_tile_step<SF, RING, SCALED, STOCH, TY, size_t, 8>);
    } else if (L.P <= kTileFewCells) {
      e = go(k_tile_step<SF, RING, SCALED, STOCH, TY, uint32_t, 8>);
    } else {
      e = go(k_tile_step<SF, RING, SCALED, STOCH, TY, uint32_t, 10>);
    }
    if (e != cudaSuccess) return FD_ERR_CUDA;
  }
  return FD_OK;
}

}  // namespace fd

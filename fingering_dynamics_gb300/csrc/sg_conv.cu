// 3x3 convolution (forward and data gradient) of the learned surrogate on tcgen05: at
// widths that are multiples of 128 (sg_conv3x3_tma, sg_conv3x3_tma_ws), described here,
// and at the others (sg_conv3x3_tc): this kernel's FLAT form and k_conv3x3_narrow below.
//
// Implicit GEMM, M = pixels, N = output channels, K = 9 x input channels.  A
// persistent CTA walks tiles of R image rows x 128 pixels x BN output channels
// (R accumulators of BN tensor-memory columns, two buffers of them):
//   warp 8  (one thread) issues the boxes.  A: per chunk of CH input channels one
//           box of the input's halo, (R + 2) rows x 130 pixels x CH channels,
//           swizzled over the pixel's 32 or 64 bytes; pixels outside the image
//           read as zero, the convolution's padding.  B: per chunk nine boxes of
//           BN output channels x CH, one per tap.  Where the weights of all chunks
//           fit beside the ring they are loaded once per CTA and stay;
//   warp 9  issues the MMAs of a stage: each tap's A operand is the window that
//           starts at row r + ky and pixel kx of the halo (the swizzle follows the
//           address, so a window may start on any pixel).  The descriptors are a
//           base and constants, in uniform registers;
//   warps 0..7 finish tile j (bias, GELU, stores) while tile j + 1 is multiplied.
// K advances 16 channels at a time, the nine taps of a slice back to back, so the
// FP32 sums run in one order whatever the chunk and tile.
//
// In a list of operations (sg_run) the barriers, the tensor memory and the tensor
// maps are set up while the previous kernel drains: it took a prediction of one image
// of 256 x 512 (23 kernels of 4 to 20 us) from 256 to 210 us (195 now).
//
// What it replaced: boxes of 8 channels (16-byte pieces, four to eight times as
// many), the weights streamed anew for every tile, two descriptors built per MMA
// by the thread that also issued the boxes.  Measured at batch 32, us, before ->
// here: 16 -> 32 (256 x 512, GELU) 271 -> 167, 32 -> 32 354 -> 181, 96 -> 32 855 ->
// 338, 32 -> 96 (no activation) 924 -> 208, 64 -> 64 (128 x 256) 250 -> 96, 192 -> 64
// 507 -> 200, 128 -> 128 (64 x 128) 207 -> 68, 384 -> 128 397 -> 151 (1538 TFLOP/s).
// The thin layers are bound by the MMAs, which take some 55 clocks however few
// columns they have (32 -> 16: 114 us, its bytes 59), with GELU also by the
// epilogue's tanhf; the wide ones by the tensor pipe.
#include "sg_conv_plan.h"
#include "sg_tc.cuh"

namespace sg {
namespace {

static_assert(kConvPixels == kTcBM, "operand rows");
constexpr int kCvEpiWarps = 8;
constexpr int kCvThreads = 32 * (kCvEpiWarps + 2);

// 32 bytes of one pixel: one store of a whole sector where the tensors are 32-byte
// aligned (`wide`), else two.  Two stores of half a sector each bound the layers
// that write much: at batch 32, us, two -> one: 64 -> 64 (128 x 256, GELU) 127 -> 96,
// 32 -> 64 113 -> 87, 32 -> 96 (256 x 512) 300 -> 208, 128 -> 128 (64 x 128) 84 -> 68.
// (12 or 16 epilogue warps instead of 8 then gain 3-8% on the two thinnest layers and
// lose 2-4% on the others.)
__device__ __forceinline__ void cv_store32(bf16* p, const uint32_t (&w)[8], bool wide) {
  if (wide) {
    asm volatile("st.global.v8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(p), "r"(w[0]), "r"(w[1]), "r"(w[2]),
                 "r"(w[3]), "r"(w[4]), "r"(w[5]), "r"(w[6]), "r"(w[7])
                 : "memory");
  } else {
    reinterpret_cast<uint4*>(p)[0] = make_uint4(w[0], w[1], w[2], w[3]);
    reinterpret_cast<uint4*>(p)[1] = make_uint4(w[4], w[5], w[6], w[7]);
  }
}

// Bias, activation and stores of 16 output channels of one pixel (element offset o).
__device__ __forceinline__ void cv_store16(const float (&v)[16], const float* sbias, int act, bool wide,
                                           bf16* __restrict__ z, bf16* __restrict__ y, size_t o) {
  uint32_t zw[8], yw[8];
#pragma unroll
  for (int k = 0; k < 8; ++k) {
    float t0 = v[2 * k] + sbias[2 * k], t1 = v[2 * k + 1] + sbias[2 * k + 1];
    const __nv_bfloat162 zp = __floats2bfloat162_rn(t0, t1);
    zw[k] = *reinterpret_cast<const uint32_t*>(&zp);
    if (act == SG_ACT_GELU) {
      t0 = gelu_f(t0);
      t1 = gelu_f(t1);
    }
    const __nv_bfloat162 yp = __floats2bfloat162_rn(t0, t1);
    yw[k] = *reinterpret_cast<const uint32_t*>(&yp);
  }
  if (z) cv_store32(z + o, zw, wide);
  if (y) cv_store32(y + o, yw, wide);
}

// FLAT: the tile of k_conv3x3_rows at widths that are not a multiple of 128 and few
// channels (sg_conv3x3_tc; 64 channels a chunk and up run on k_conv3x3_narrow).  bw
// x rows pixels of an image are the first bw of every bw + 2 operand rows, so that
// the tile's halo is still one box and every tap one window of it; the two rows
// between are not read back.  K advances chunk by chunk, the nine taps of a chunk
// back to back, 16 channels at a time within a tap, as in k_conv3x3_narrow.  With a
// box per tap the copies' 32- and 64-byte rows bound the thin layers: at 32 x 200 x
// 328, GELU, us, box per tap -> halo (the kernel fed by 16-byte copies, the
// warp-level one; at batch 8): 16 -> 32 292 -> 132, 32 -> 32 292 -> 132 (8: 102, 89 ->
// 40), 96 -> 32 697 -> 270 (257, 179 -> 77), 32 -> 16 267 -> 116.
template <int BN, int R, int CH, bool FLAT>
struct CvCfg {
  static constexpr int ROW = CH * 2;                                        // bytes of a pixel or output channel
  static constexpr int A_TX = (R + 2) * kHaloPx * ROW;
  static constexpr int A_BYTES = (A_TX + 1023) / 1024 * 1024;
  static constexpr int TAP = BN * ROW, B_BYTES = (9 * TAP + 1023) / 1024 * 1024;  // one tap's and one chunk's weights
  static constexpr int NCOL = 2 * R * BN;                                   // two accumulator buffers
  static constexpr int COLS = NCOL <= 32 ? 32 : (NCOL <= 64 ? 64 : (NCOL <= 128 ? 128 : (NCOL <= 256 ? 256 : 512)));
  static constexpr int S_MAX = 6;
  static constexpr int TAIL = (2 * S_MAX + 5) * 8 + BN * 4 + 16 + 1024;       // barriers, bias, TMEM address, alignment
  static_assert(!FLAT || R == 1, "one accumulator");
  static_assert(NCOL <= 512 && TAP % (8 * ROW) == 0, "tile");
};

struct CvShape {
  int N, H, W, Cin, Cout, act;
  int nk, S;       // chunks, ring stages
  int resident;    // the weights of all chunks stay in shared memory
  int bw, rows;    // tiles of widths that are not a multiple of 128: pixels, rows
};

template <int BN, int R, int CH, bool FLAT>
__global__ void __launch_bounds__(kCvThreads, 1) k_conv3x3_rows(const __grid_constant__ ConvMaps maps, const CvShape sh,
                                                               const float* __restrict__ bias, bf16* __restrict__ z,
                                                               bf16* __restrict__ y) {
  using C = CvCfg<BN, R, CH, FLAT>;
  extern __shared__ char smem_raw[];
  char* smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
  const int S = sh.S, nk = sh.nk, stage = C::A_BYTES + (sh.resident ? 0 : C::B_BYTES);
  char* wres = smem + S * stage;  // resident weights
  char* tail = wres + (sh.resident ? nk * C::B_BYTES : 0);
  uint64_t* full = reinterpret_cast<uint64_t*>(tail);
  uint64_t *empty = full + C::S_MAX, *accf = empty + C::S_MAX, *acce = accf + 2, *wfull = acce + 2;
  float* sbias = reinterpret_cast<float*>(wfull + 1);
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(sbias + BN);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int tw = FLAT ? sh.bw : kTcBM, rows = FLAT ? sh.rows : R, pitch = FLAT ? sh.bw + 2 : kHaloPx;
  const int tiles_x = FLAT ? (sh.W + tw - 1) / tw : sh.W / kTcBM, tiles_y = FLAT ? (sh.H + rows - 1) / rows : sh.H / R;
  const int nco = sh.Cout / BN;
  const int ntiles = sh.N * tiles_y * tiles_x * nco;
  const int mine = (int)blockIdx.x < ntiles ? (ntiles - 1 - (int)blockIdx.x) / (int)gridDim.x + 1 : 0;  // this CTA's tiles
  // the grid is a multiple of the output-channel tiles, so a CTA keeps one of them
  const int co0 = ((int)blockIdx.x % nco) * BN;

  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)),
                 "r"(C::COLS)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  if (tid == 0) {
    for (int i = 0; i < 2 * C::S_MAX + 2; ++i) mbar_init(&full[i]);
    mbar_init(wfull);
    for (int i = 0; i < 2; ++i)
      asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(&acce[i])), "n"(kCvEpiWarps) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  fd::pdl_wait();
  fd::pdl_launch_dependents();
  for (int i = tid; i < BN; i += kCvThreads) sbias[i] = bias ? __ldcg(bias + co0 + i) : 0.0f;
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = *tmem_slot;

  // tile j of this CTA -> image n, first row yy, first pixel x0
  auto tile_of = [&](int j, int& n, int& yy, int& x0) {
    const int pt = ((int)blockIdx.x + j * (int)gridDim.x) / nco, py = pt / tiles_x;
    x0 = (pt - py * tiles_x) * tw;
    n = py / tiles_y;
    yy = (py - n * tiles_y) * rows;
  };

  if (warp == kCvEpiWarps) {
    if (lane == 0 && mine > 0) {
      auto load_b = [&](char* dst, int kc, uint64_t* bar) {
#pragma unroll
        for (int tap = 0; tap < 9; ++tap) tma_load_3d(dst + tap * C::TAP, &maps.w, kc * CH, tap, co0, bar);
      };
      if (sh.resident) {
        mbar_expect_tx(wfull, (unsigned)(nk * 9 * C::TAP));
        for (int kc = 0; kc < nk; ++kc) load_b(wres + kc * C::B_BYTES, kc, wfull);
      }
      const unsigned tx = (unsigned)((FLAT ? (rows + 2) * pitch * C::ROW : C::A_TX) + (sh.resident ? 0 : 9 * C::TAP));
      int c = 0;  // chunks issued
      bool ok = true;
      for (int j = 0; j < mine && ok; ++j) {
        int n, yy, x0;
        tile_of(j, n, yy, x0);
        for (int kc = 0; kc < nk; ++kc, ++c) {
          const int st = c % S;
          if (c >= S) ok = mbar_wait_ok(&empty[st], (unsigned)(c / S - 1) & 1u, true);
          if (!ok) break;
          char* a = smem + st * stage;
          mbar_expect_tx(&full[st], tx);
          tma_load_4d(a, &maps.x, kc * CH, x0 - 1, yy - 1, n, &full[st]);
          if (!sh.resident) load_b(a + C::A_BYTES, kc, &full[st]);
        }
      }
      // everything issued has landed before the CTA gives its shared memory up
      if (sh.resident) mbar_wait_ok(wfull, 0u, false);
      for (int i = 0; i < S && i < c; ++i)
        mbar_wait_ok(&full[i], (unsigned)((c - 1 - ((c - 1 - i) % S)) / S) & 1u, false);
    }
    __syncwarp();
  } else if (warp == kCvEpiWarps + 1) {
    uint32_t leader;
    asm volatile("{\n .reg .pred p;\n elect.sync _|p, 0xffffffff;\n selp.u32 %0, 1, 0, p;\n}\n" : "=r"(leader));
    constexpr uint32_t idesc = instr_desc<kTcBM, BN>();
    const uint64_t a0 = smem_desc_sw<C::ROW>(smem_u32(smem), 16, 8 * C::ROW);
    const uint64_t w0 = smem_desc_sw<C::ROW>(smem_u32(sh.resident ? wres : smem + C::A_BYTES), 16, 8 * C::ROW);
    bool ok = mine > 0 && (!sh.resident || mbar_wait_ok(wfull, 0u, true));
    int c = 0, tiles = 0;  // chunks and whole tiles issued
    for (int j = 0; j < mine && ok; ++j) {
      const int b = j & 1;
      if (j >= 2) ok = mbar_wait_ok(&acce[b], (unsigned)((j - 2) >> 1) & 1u, true);  // tile j - 2 has been read
      const uint32_t d0 = tmem + (uint32_t)(b * R * BN);
      for (int kc = 0; kc < nk && ok; ++kc, ++c) {
        const int st = c % S;
        ok = mbar_wait_ok(&full[st], (unsigned)(c / S) & 1u, true);
        if (!ok) break;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        // an address step of 16 bytes is 1 in the descriptors' low bits
        const uint64_t as = a0 + (uint64_t)(st * stage / 16);
        const uint64_t bs = w0 + (uint64_t)((sh.resident ? kc * C::B_BYTES : st * stage) / 16);
        if (leader) {
          if constexpr (FLAT) {
#pragma unroll
            for (int tap = 0; tap < 9; ++tap) {
              const uint64_t at = as + (uint64_t)(((tap / 3) * pitch + tap % 3) * C::ROW / 16);
#pragma unroll
              for (int s = 0; s < CH / 16; ++s)
                tc_mma(d0, at + (uint64_t)(s * 2), bs + (uint64_t)((tap * C::TAP + s * 32) / 16), idesc,
                       (s > 0 || tap > 0) ? 1u : (kc > 0 ? 1u : 0u));
            }
          } else {
#pragma unroll
            for (int s = 0; s < CH / 16; ++s) {
#pragma unroll
              for (int tap = 0; tap < 9; ++tap) {
                const int ky = tap / 3, kx = tap % 3;
                const uint32_t acc = (s > 0 || tap > 0) ? 1u : (kc > 0 ? 1u : 0u);
#pragma unroll
                for (int r = 0; r < R; ++r)
                  tc_mma(d0 + (uint32_t)(r * BN), as + (uint64_t)((((r + ky) * kHaloPx + kx) * C::ROW + s * 32) / 16),
                         bs + (uint64_t)((tap * C::TAP + s * 32) / 16), idesc, acc);
              }
            }
          }
          tc_commit(&empty[st]);
          if (kc == nk - 1) tc_commit(&accf[b]);  // tile j's accumulators are complete
        }
        if (kc == nk - 1) tiles = j + 1;
        __syncwarp();
      }
    }
    // the MMAs issued have completed and their commits have arrived before tensor and shared memory are given up
    for (int i = 0; i < S && i < c; ++i)
      mbar_wait_ok(&empty[i], (unsigned)((c - 1 - ((c - 1 - i) % S)) / S) & 1u, false);
    if (!ok)  // else the epilogue warps wait for every tile
      for (int j = tiles > 2 ? tiles - 2 : 0; j < tiles; ++j) mbar_wait_ok(&accf[j & 1], (unsigned)(j >> 1) & 1u, false);
  } else {
    // epilogue: warp w reads TMEM lanes 32 q .. 32 q + 31 (pixels x0 + 32 q + lane of each row, q = w % 4) of every
    // second group of 16 columns (w / 4)
    const int q = warp & 3, h = warp >> 2;
    const bool wide = ((uintptr_t)z | (uintptr_t)y) % 32 == 0;
    const int m = q * 32 + lane, my = FLAT ? m / pitch : 0, mx = m - my * pitch;
    for (int j = 0; j < mine; ++j) {
      const int b = j & 1;
      int n, yy, x0;
      tile_of(j, n, yy, x0);
      const bool in = !FLAT || (mx < tw && my < rows && yy + my < sh.H && x0 + mx < sh.W);
      mbar_wait_ok(&accf[b], (unsigned)(j >> 1) & 1u, true);
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll 1
      for (int i = h; i < R * (BN / 16); i += 2) {
        const int r = i / (BN / 16), c0 = (i % (BN / 16)) * 16;
        float v[16];
        tmem_ld16(tmem + ((uint32_t)(q * 32) << 16) + (uint32_t)(b * R * BN + i * 16), v);
        const size_t o = (((size_t)n * sh.H + yy + r + my) * sh.W + x0 + mx) * sh.Cout + co0 + c0;
        if (in) cv_store16(v, sbias + c0, sh.act, wide, z, y, o);
      }
      // this warp's reads of buffer b are complete (tcgen05.wait::ld in tmem_ld16)
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      __syncwarp();
      if (lane == 0) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(&acce[b])) : "memory");
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == 0) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(C::COLS) : "memory");
  }
}

// ---------------------------------------------------------------------------
// Widths that are not a multiple of 128 (sg_conv3x3_tc): a tile is bw x rows pixels
// of one image, at most 128 (tile_box), and ends with the image.  A halo would not
// be evenly spaced operand rows, so a stage is one tap of a chunk of BK channels: a
// box of the tile's pixels shifted by the tap (zeros outside the image) and the
// tap's weights; operand rows past the tile hold whatever the stage held before and
// their sums are not read.  K advances chunk by chunk, the nine taps of a chunk
// back to back, 16 channels at a time within a tap, as in the kernel it replaced,
// which all threads fed by 16-byte copies: at 32 x 32 x 64, us, 128 -> 256 channels
// 247 -> 50, 256 -> 256 445 -> 71, 256 -> 128 255 -> 38 (the warp-level kernel 157,
// 283, 143); one image, 256 -> 256, 48 -> 14.5 (25); at 8 x 50 x 82, 128 -> 128 77 -> 20
// (48), 384 -> 128 189 -> 34 (118).
// Same roles as k_conv3x3_rows.
// ---------------------------------------------------------------------------
template <int BN, int BK>
struct CnCfg {
  static constexpr int ROW = BK * 2;
  static constexpr int A_BYTES = kTcBM * ROW, B_BYTES = (BN * ROW + 1023) / 1024 * 1024, STAGE = A_BYTES + B_BYTES;
  static constexpr int COLS = 2 * BN < 32 ? 32 : 2 * BN;
  static constexpr int S = 220 * 1024 / STAGE > 8 ? 8 : 220 * 1024 / STAGE;
  static constexpr int OFF_BAR = S * STAGE;
  static constexpr int SMEM = OFF_BAR + (2 * S + 4) * 8 + BN * 4 + 16 + 1024;
  static_assert(A_BYTES % 1024 == 0 && SMEM <= 227 * 1024 && COLS <= 512, "tile");
};

template <int BN, int BK>
__global__ void __launch_bounds__(kCvThreads, 1) k_conv3x3_narrow(const __grid_constant__ ConvMaps maps, const CvShape sh,
                                                                 const float* __restrict__ bias, bf16* __restrict__ z,
                                                                 bf16* __restrict__ y) {
  using C = CnCfg<BN, BK>;
  constexpr int S = C::S;
  extern __shared__ char smem_raw[];
  char* smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
  uint64_t* full = reinterpret_cast<uint64_t*>(smem + C::OFF_BAR);
  uint64_t *empty = full + S, *accf = empty + S, *acce = accf + 2;
  float* sbias = reinterpret_cast<float*>(acce + 2);
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(sbias + BN);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int bw = sh.bw, rows = sh.rows, tiles_x = (sh.W + bw - 1) / bw, tiles_y = (sh.H + rows - 1) / rows;
  const int nco = sh.Cout / BN;
  const int ntiles = sh.N * tiles_y * tiles_x * nco, nst = sh.nk * 9;  // stages of a tile
  const int mine = (int)blockIdx.x < ntiles ? (ntiles - 1 - (int)blockIdx.x) / (int)gridDim.x + 1 : 0;
  const int co0 = ((int)blockIdx.x % nco) * BN;  // the grid is a multiple of the output-channel tiles

  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)),
                 "r"(C::COLS)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  if (tid == 0) {
    for (int i = 0; i < 2 * S + 2; ++i) mbar_init(&full[i]);
    for (int i = 0; i < 2; ++i)
      asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(&acce[i])), "n"(kCvEpiWarps) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  fd::pdl_wait();
  fd::pdl_launch_dependents();
  for (int i = tid; i < BN; i += kCvThreads) sbias[i] = bias ? __ldcg(bias + co0 + i) : 0.0f;
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = *tmem_slot;
  // tile j of this CTA -> image n, first row y0, first pixel x0
  auto tile_of = [&](int j, int& n, int& y0, int& x0) {
    const int pt = ((int)blockIdx.x + j * (int)gridDim.x) / nco, py = pt / tiles_x;
    x0 = (pt - py * tiles_x) * bw;
    n = py / tiles_y;
    y0 = (py - n * tiles_y) * rows;
  };

  if (warp == kCvEpiWarps) {
    if (lane == 0 && mine > 0) {
      const uint32_t tx = (uint32_t)((bw * rows + BN) * C::ROW);
      int c = 0;
      bool ok = true;
      for (int j = 0; j < mine && ok; ++j) {
        int n, y0, x0;
        tile_of(j, n, y0, x0);
        for (int k = 0; k < nst; ++k, ++c) {
          const int st = c % S, kc = k / 9, tap = k % 9;
          if (c >= S) ok = mbar_wait_ok(&empty[st], (unsigned)(c / S - 1) & 1u, true);
          if (!ok) break;
          char* a = smem + st * C::STAGE;
          mbar_expect_tx(&full[st], tx);
          tma_load_4d(a, &maps.x, kc * BK, x0 + tap % 3 - 1, y0 + tap / 3 - 1, n, &full[st]);
          tma_load_3d(a + C::A_BYTES, &maps.w, kc * BK, tap, co0, &full[st]);
        }
      }
      for (int i = 0; i < S && i < c; ++i)
        mbar_wait_ok(&full[i], (unsigned)((c - 1 - ((c - 1 - i) % S)) / S) & 1u, false);
    }
    __syncwarp();
  } else if (warp == kCvEpiWarps + 1) {
    uint32_t leader;
    asm volatile("{\n .reg .pred p;\n elect.sync _|p, 0xffffffff;\n selp.u32 %0, 1, 0, p;\n}\n" : "=r"(leader));
    constexpr uint32_t idesc = instr_desc<kTcBM, BN>();
    const uint64_t a0 = smem_desc_sw<C::ROW>(smem_u32(smem), 16, 8 * C::ROW);
    const uint64_t w0 = smem_desc_sw<C::ROW>(smem_u32(smem + C::A_BYTES), 16, 8 * C::ROW);
    bool ok = true;
    int c = 0, tiles = 0;
    for (int j = 0; j < mine && ok; ++j) {
      const int b = j & 1;
      if (j >= 2) ok = mbar_wait_ok(&acce[b], (unsigned)((j - 2) >> 1) & 1u, true);
      for (int k = 0; k < nst && ok; ++k, ++c) {
        const int st = c % S;
        ok = mbar_wait_ok(&full[st], (unsigned)(c / S) & 1u, true);
        if (!ok) break;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const uint64_t off = (uint64_t)(st * C::STAGE / 16);
        if (leader) {
#pragma unroll
          for (int s = 0; s < BK / 16; ++s)
            tc_mma(tmem + (uint32_t)(b * BN), a0 + off + (uint64_t)(s * 2), w0 + off + (uint64_t)(s * 2), idesc,
                   s > 0 ? 1u : (k > 0 ? 1u : 0u));
          tc_commit(&empty[st]);
          if (k == nst - 1) tc_commit(&accf[b]);
        }
        if (k == nst - 1) tiles = j + 1;
        __syncwarp();
      }
    }
    for (int i = 0; i < S && i < c; ++i)
      mbar_wait_ok(&empty[i], (unsigned)((c - 1 - ((c - 1 - i) % S)) / S) & 1u, false);
    if (!ok)  // else the epilogue warps wait for every tile
      for (int j = tiles > 2 ? tiles - 2 : 0; j < tiles; ++j) mbar_wait_ok(&accf[j & 1], (unsigned)(j >> 1) & 1u, false);
  } else {
    const int q = warp & 3, h = warp >> 2;
    const bool wide = ((uintptr_t)z | (uintptr_t)y) % 32 == 0;
    const int m = q * 32 + lane, my = m / bw, mx = m - my * bw;  // pixel of the tile
    for (int j = 0; j < mine; ++j) {
      const int b = j & 1;
      int n, y0, x0;
      tile_of(j, n, y0, x0);
      mbar_wait_ok(&accf[b], (unsigned)(j >> 1) & 1u, true);
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      const int yy = y0 + my, xx = x0 + mx;
      const bool in = my < rows && yy < sh.H && xx < sh.W;
#pragma unroll 1
      for (int i = h; i < BN / 16; i += 2) {
        float v[16];
        tmem_ld16(tmem + ((uint32_t)(q * 32) << 16) + (uint32_t)(b * BN + i * 16), v);
        if (in)
          cv_store16(v, sbias + i * 16, sh.act, wide, z, y, (((size_t)n * sh.H + yy) * sh.W + xx) * sh.Cout + co0 + i * 16);
      }
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      __syncwarp();
      if (lane == 0) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(&acce[b])) : "memory");
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == 0) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(C::COLS) : "memory");
  }
}

// Tensor maps of one call: x as (C, W, H, N) with boxes of CH channels x box_w
// pixels x box_h rows, the weights [co][tap][ci] as (Cin, 9, Cout) with boxes of
// CH channels x 1 tap x BN output channels.
inline int encode_conv_maps(ConvMaps& m, const bf16* x, int N, int H, int W, int Cin, const bf16* w, int Cout,
                            int box_w, int box_h, int BN, int CH) {
  const fd::EncodeTiledFn fn = fd::encode_tiled_fn();
  FD_REQUIRE(fn != nullptr, FD_ERR_CUDA, "cuTensorMapEncodeTiled is not available from the driver");
  const CUtensorMapSwizzle sw = CH == 64 ? CU_TENSOR_MAP_SWIZZLE_128B
                                         : (CH == 32 ? CU_TENSOR_MAP_SWIZZLE_64B : CU_TENSOR_MAP_SWIZZLE_32B);
  const cuuint64_t es = 2;
  const cuuint64_t xd[4] = {(cuuint64_t)Cin, (cuuint64_t)W, (cuuint64_t)H, (cuuint64_t)N};
  const cuuint64_t xs[3] = {Cin * es, (cuuint64_t)W * Cin * es, (cuuint64_t)H * W * Cin * es};
  const cuuint32_t xb[4] = {(cuuint32_t)CH, (cuuint32_t)box_w, (cuuint32_t)box_h, 1u};
  const cuuint32_t e4[4] = {1u, 1u, 1u, 1u};
  CUresult r = fn(&m.x, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 4, const_cast<bf16*>(x), xd, xs, xb, e4,
                  CU_TENSOR_MAP_INTERLEAVE_NONE, sw, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                  CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  FD_REQUIRE(r == CUDA_SUCCESS, FD_ERR_CUDA, "sg_conv3x3_tma: input tensor map (%d)", (int)r);
  const cuuint64_t wd[3] = {(cuuint64_t)Cin, 9u, (cuuint64_t)Cout};
  const cuuint64_t ws[2] = {Cin * es, 9u * Cin * es};
  const cuuint32_t wb[3] = {(cuuint32_t)CH, 1u, (cuuint32_t)BN};
  r = fn(&m.w, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, const_cast<bf16*>(w), wd, ws, wb, e4,
         CU_TENSOR_MAP_INTERLEAVE_NONE, sw, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  FD_REQUIRE(r == CUDA_SUCCESS, FD_ERR_CUDA, "sg_conv3x3_tma: weight tensor map (%d)", (int)r);
  return FD_OK;
}

struct CvCall {
  const bf16* x;
  int N, H, W, Cin;
  const bf16* w;
  const float* b;
  int Cout, act;
  bf16 *z, *y;
  cudaStream_t s;
  int sms;
};

template <int BN, int R, int CH, bool FLAT = false>
int launch_rows(const CvCall& c, int bw = kTcBM, int rows = R) {
  using C = CvCfg<BN, R, CH, FLAT>;
  auto kern = k_conv3x3_rows<BN, R, CH, FLAT>;
  static std::atomic<unsigned long long> attr_done{0};
  if (fd::ensure_smem_attr(kern, 227 * 1024, attr_done) != cudaSuccess)
    return fd::check_launch("sg_conv3x3_tma: shared-memory attribute");
  constexpr int kRoom = 227 * 1024 - C::TAIL;
  CvShape sh{c.N, c.H, c.W, c.Cin, c.Cout, c.act, c.Cin / CH, 0, 0, bw, rows};
  const ConvRing ring = conv_ring(sh.nk, C::A_BYTES, C::B_BYTES, kRoom, C::S_MAX);
  sh.resident = ring.resident;
  sh.S = ring.stages;
  if (sh.S < 1) {
    fd::set_error("sg_conv3x3_tma: no stage fits");
    return FD_ERR_SHAPE;
  }
  const int nco = c.Cout / BN;
  const long long ntiles = (long long)c.N * ((c.H + rows - 1) / rows) * ((c.W + bw - 1) / bw) * nco;
  const long long grid = std::min<long long>(ntiles, std::max(1, c.sms / nco) * (long long)nco);
  ConvMaps maps;
  if (int r = encode_conv_maps(maps, c.x, c.N, c.H, c.W, c.Cin, c.w, c.Cout, bw + 2, rows + 2, BN, CH)) return r;
  fd::launch_pdl(kern, (unsigned)grid, kCvThreads, 227 * 1024, c.s, t_op_follows, maps, sh, c.b, c.z, c.y);
  return fd::check_launch("sg_conv3x3_tma");
}

// Rows per tile: the most of 4, 2, 1 that divide H with two buffers of R x BN
// accumulator columns in the tensor memory, and fewer where there would be less
// than two tiles per SM (a batch of one: 256 x 512 has 256 tiles of four rows).
constexpr long long kCvTiles = 2;
template <int BN, int CH>
int rows_r(const CvCall& c) {
  const long long per_row = (long long)c.N * c.H * (c.W / kTcBM) * (c.Cout / BN), want = kCvTiles * c.sms;
  if constexpr (BN <= 64) {
    if (c.H % 4 == 0 && per_row / 4 >= want) return launch_rows<BN, 4, CH>(c);
  }
  if (c.H % 2 == 0 && per_row / 2 >= want) return launch_rows<BN, 2, CH>(c);
  return launch_rows<BN, 1, CH>(c);
}

template <int CH>
int rows_n(const CvCall& c) {
  if (c.Cout % 128 == 0) return rows_r<128, CH>(c);
  if (c.Cout % 96 == 0 && c.Cout % 64 != 0) return rows_r<96, CH>(c);
  if (c.Cout % 64 == 0) return rows_r<64, CH>(c);
  if (c.Cout % 32 == 0) return rows_r<32, CH>(c);
  return rows_r<16, CH>(c);
}

template <int BN, int BK>
int launch_narrow(const CvCall& c, int bw, int rows) {
  using C = CnCfg<BN, BK>;
  auto kern = k_conv3x3_narrow<BN, BK>;
  static std::atomic<unsigned long long> attr_done{0};
  if (fd::ensure_smem_attr(kern, 227 * 1024, attr_done) != cudaSuccess)
    return fd::check_launch("sg_conv3x3_tc: shared-memory attribute");
  const int nco = c.Cout / BN;
  const CvShape sh{c.N, c.H, c.W, c.Cin, c.Cout, c.act, c.Cin / BK, C::S, 0, bw, rows};
  const long long ntiles = (long long)c.N * ((c.H + rows - 1) / rows) * ((c.W + bw - 1) / bw) * nco;
  const long long grid = std::min<long long>(ntiles, std::max(1, c.sms / nco) * (long long)nco);
  ConvMaps maps;
  if (int r = encode_conv_maps(maps, c.x, c.N, c.H, c.W, c.Cin, c.w, c.Cout, bw, rows, BN, BK)) return r;
  fd::launch_pdl(kern, (unsigned)grid, kCvThreads, 227 * 1024, c.s, t_op_follows, maps, sh, c.b, c.z, c.y);
  return fd::check_launch("sg_conv3x3_tc");
}

// Output channels per tile: 128 where the tiles still give every SM one, else 64
// (a batch of one at 32 x 64 has 16 tiles of pixels).
template <int BK>
int narrow_n(const CvCall& c) {
  int bw = 1, rows = kTcBM;
  tile_box(c.H, c.W, 0, bw, rows);
  const long long px_tiles = (long long)c.N * ((c.H + rows - 1) / rows) * ((c.W + bw - 1) / bw);
  if (c.Cout % 128 == 0 && px_tiles * (c.Cout / 128) >= c.sms) return launch_narrow<128, BK>(c, bw, rows);
  if (c.Cout % 64 == 0 && px_tiles * (c.Cout / 64) >= c.sms / 2) return launch_narrow<64, BK>(c, bw, rows);
  if (c.Cout % 32 == 0) return launch_narrow<32, BK>(c, bw, rows);
  return launch_narrow<16, BK>(c, bw, rows);
}

template <int CH>
int flat_n(const CvCall& c) {
  int bw = 1, rows = 1;
  tile_box(c.H, c.W, 2, bw, rows);
  const long long px_tiles = (long long)c.N * ((c.H + rows - 1) / rows) * ((c.W + bw - 1) / bw);
  if (c.Cout % 64 == 0 && px_tiles * (c.Cout / 64) >= c.sms / 2) return launch_rows<64, 1, CH, true>(c, bw, rows);
  if (c.Cout % 32 == 0) return launch_rows<32, 1, CH, true>(c, bw, rows);
  return launch_rows<16, 1, CH, true>(c, bw, rows);
}

int conv_rows(const void* x, int N, int H, int W, int Cin, const void* w, const float* bias, int Cout, int act, void* z,
              void* y, void* stream, const char* what) {
  FD_REQUIRE(x && w && (z || y) && N > 0 && H > 0 && W > 0, FD_ERR_ARG, "%s: bad arguments", what);
  FD_REQUIRE(W % kTcBM == 0 && Cin % 16 == 0 && Cout % 16 == 0 && Cin > 0 && Cout > 0, FD_ERR_SHAPE,
             "%s: needs W a multiple of 128 and channel counts multiples of 16 (got W=%d, %d -> %d)", what, W, Cin, Cout);
  FD_REQUIRE(act == SG_ACT_NONE || act == SG_ACT_GELU, FD_ERR_ARG, "%s: activation %d", what, act);
  FD_REQUIRE(((uintptr_t)x | (uintptr_t)w | (uintptr_t)z | (uintptr_t)y) % 16 == 0, FD_ERR_ARG,
             "%s: tensors must be 16-byte aligned", what);
  CvCall c{(const bf16*)x, N, H, W, Cin, (const bf16*)w, bias, Cout, act, (bf16*)z, (bf16*)y, fd::as_stream(stream),
           fd::sm_count()};
  return Cin % 32 == 0 ? rows_n<32>(c) : rows_n<16>(c);
}

}  // namespace

int conv_error_word(unsigned* out, bool clear) { return tc_error_word(out, clear); }

// sg_conv3x3_tc on widths that are not a multiple of 128 (arguments checked by the caller).
int conv_narrow(const void* x, int N, int H, int W, int Cin, const void* w, const float* bias, int Cout, int act, void* z,
                void* y, cudaStream_t s) {
  CvCall c{(const bf16*)x, N, H, W, Cin, (const bf16*)w, bias, Cout, act, (bf16*)z, (bf16*)y, s, fd::sm_count()};
  if (Cin % 64 == 0) return narrow_n<64>(c);
  return Cin % 32 == 0 ? flat_n<32>(c) : flat_n<16>(c);
}

}  // namespace sg

extern "C" {

int sg_conv3x3_tma(const void* x, int N, int H, int W, int Cin, const void* w, const float* bias, int Cout,
                   int act, void* z, void* y, void* stream) {
  return sg::conv_rows(x, N, H, W, Cin, w, bias, Cout, act, z, y, stream, "sg_conv3x3_tma");
}

int sg_conv3x3_tma_ws(const void* x, int N, int H, int W, int Cin, const void* w, const float* bias, int Cout,
                      int act, void* z, void* y, void* stream) {
  return sg::conv_rows(x, N, H, W, Cin, w, bias, Cout, act, z, y, stream, "sg_conv3x3_tma_ws");
}

}  // extern "C"

// Weight gradient of the learned surrogate's 3x3 convolutions on the
// fifth-generation tensor cores.
#include "sg_tc.cuh"

namespace sg {
namespace {

// ---------------------------------------------------------------------------
// Weight gradient on tcgen05 (sg_conv3x3_wgrad_tc):
//   dw[co][tap][ci] = sum_p dz[p][co] x[p + (ky-1, kx-1)][ci].
// A CTA takes one kernel row ky, a block of input and of output channels and a
// contiguous range of chunks (128 pixels of one image row).
//   * Both operands are channel-contiguous in memory, so they are MN-major: a box
//     is a chunk of pixels by CB (x, 16, 32 or 64) or up to 64 (dz) channels,
//     swizzled, 32, 64 or 128 bytes a pixel.  (Boxes of 8 channels, the layout
//     without swizzle, arrive as pieces of 16 bytes: 1048 us for 32 -> 32 channels
//     at 32 x 256 x 512, where reading x and dz once takes 79 us.)
//   * The MMA's 128 rows are (kx, input channel): the stride between blocks of CB
//     rows (LBO) is one pixel, so the blocks are the same x row shifted by kx = 0,
//     1, 2, ..; nothing is built, and thin layers do not pad the rows with
//     channels they do not have.  Blocks beyond kx = 2 are computed and ignored;
//     they read at most seven pixels past a box, inside the slot's padding, and
//     rows of an MMA do not mix.  Where the input channels fill 128 rows (PAIR),
//     two blocks of 64 channels do, with an accumulator per kx.
// Warp 0 (one thread) issues the boxes of a ring of stages, warp 1 the MMAs of a
// chunk (its descriptors are a base and constants, in uniform registers: with
// descriptors built per MMA by one thread the issue was the bound).  FP32 partials
// go to partial[split][co][tap][ci] and are added in a fixed order, and the split
// into pixel ranges depends on the shape, the device's SM count and the room that
// `partial` has, so on one device the result does not depend on scheduling.
// Measured at batch 32, us, against boxes of 8 channels with output or input
// channels alone on the rows (and against the warp-level kernel): 32 -> 32 (256 x
// 512) 133 (1048; 678), 96 -> 32 336 (1232; 1988), 64 -> 64 (128 x 256) 84 (332;
// 341), 192 -> 64 285 (818; 989), 384 -> 128 (64 x 128) 149 (416; 983) = 1553
// TFLOP/s.  Walking down a column with the three rows of x in the ring, each
// loaded once for all ky, was slower (159, 648, 147, 373, 383) while one thread
// built the descriptors; the rows come from L2 twice.
// ---------------------------------------------------------------------------
// instruction descriptor of kind::f16 with both operands MN-major (transpose bits 15 and 16)
template <int M, int N>
__device__ __forceinline__ constexpr uint32_t instr_desc_mn() {
  return instr_desc<M, N>() | (1u << 15) | (1u << 16);
}

constexpr int kWgPx = kTcBM + 8;  // pixels of an x slot: the halo's 130 and padding

template <int CB, int CIT, bool PAIR, int NB>
struct WgCfg {
  static constexpr int XROW = CB * 2, XBOX = kWgPx * XROW;               // bytes a pixel; box of one channel block
  static constexpr int XSLOT = (CIT * XBOX + 1023) / 1024 * 1024;
  static constexpr int DB = NB < 64 ? NB : 64, DROW = DB * 2, DBOX = kTcBM * DROW;
  static constexpr int DSLOT = (NB / DB) * DBOX;
  static constexpr int STAGE = XSLOT + DSLOT;
  static constexpr int STACK = PAIR ? 1 : 128 / CB;                      // kx that share an MMA
  static constexpr int MG = PAIR ? 3 : (STACK >= 3 ? 1 : 2);             // MMAs per channel block and 16 pixels
  static constexpr int NACC = (PAIR ? 1 : CIT) * MG;                     // accumulators of NB columns
  // three or four stages where two CTAs then share an SM, else up to four for one
  static constexpr int PAIRED_S = (112 * 1024) / STAGE, ONE_S = (224 * 1024) / STAGE;
  static constexpr int S = PAIRED_S >= 4 ? 4 : (PAIRED_S == 3 ? 3 : (ONE_S >= 4 ? 4 : ONE_S));
  static constexpr int OFF_BAR = S * STAGE;
  static constexpr int SMEM = OFF_BAR + (2 * S + 1) * 8 + 16 + 1024;
  static constexpr int NCOL = NACC * NB;
  static constexpr int COLS = NCOL <= 32 ? 32 : (NCOL <= 64 ? 64 : (NCOL <= 128 ? 128 : (NCOL <= 256 ? 256 : 512)));
  static constexpr uint32_t TX = (uint32_t)(CIT * kHaloPx * XROW + (NB / DB) * DBOX);
  static_assert(NCOL <= 512 && SMEM <= 227 * 1024 && (!PAIR || (CB == 64 && CIT == 2)), "tile");
  static_assert(XSLOT % 1024 == 0 && DSLOT % 1024 == 0 && XBOX % (8 * XROW) == 0, "swizzle patterns start aligned");
};

template <int CB, int CIT, bool PAIR, int NB>
__global__ void __launch_bounds__(kTcThreads, 1) k_wgrad_tc(const __grid_constant__ ConvMaps maps, int H, int W, int Cin,
                                                           int Cout, int cps, long long nchunks,
                                                           float* __restrict__ partial) {
  using C = WgCfg<CB, CIT, PAIR, NB>;
  constexpr int S = C::S;
  extern __shared__ char smem_raw[];
  char* smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
  uint64_t* full = reinterpret_cast<uint64_t*>(smem + C::OFF_BAR);
  uint64_t *empty = full + S, *done = empty + S;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(done + 1);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int ci0 = blockIdx.y * CB * CIT, co0 = blockIdx.z * NB;
  const int ky = blockIdx.x % 3, split = blockIdx.x / 3;
  const long long c0 = (long long)split * cps;
  const int nc = (int)(c0 < nchunks ? (nchunks - c0 < cps ? nchunks - c0 : cps) : 0);

  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)),
                 "r"(C::COLS)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  if (tid == 0) {
    for (int i = 0; i < 2 * S + 1; ++i) mbar_init(&full[i]);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = *tmem_slot;

  if (tid == 0 && nc > 0) {
    const int tiles_x = W / kTcBM;
    int x0 = (int)(c0 % tiles_x) * kTcBM, y = (int)((c0 / tiles_x) % H), n = (int)(c0 / tiles_x / H);
    int c = 0;
    for (bool ok = true; c < nc; ++c) {
      const int st = c % S;
      if (c >= S) ok = mbar_wait_ok(&empty[st], (unsigned)(c / S - 1) & 1u, true);
      if (!ok) break;
      char* xs = smem + st * C::STAGE;
      mbar_expect_tx(&full[st], C::TX);
#pragma unroll
      for (int b = 0; b < CIT; ++b) tma_load_4d(xs + b * C::XBOX, &maps.x, ci0 + b * CB, x0 - 1, y + ky - 1, n, &full[st]);
#pragma unroll
      for (int b = 0; b < NB / C::DB; ++b)
        tma_load_4d(xs + C::XSLOT + b * C::DBOX, &maps.w, co0 + b * C::DB, x0, y, n, &full[st]);
      x0 += kTcBM;
      if (x0 == W) {
        x0 = 0;
        if (++y == H) {
          y = 0;
          ++n;
        }
      }
    }
    // the last box of every stage has landed before the CTA gives its shared memory up
    for (int i = 0; i < S && i < c; ++i)
      mbar_wait_ok(&full[i], (unsigned)((c - 1 - ((c - 1 - i) % S)) / S) & 1u, false);
  } else if (warp == 1 && nc > 0) {
    uint32_t leader;
    asm volatile("{\n .reg .pred p;\n elect.sync _|p, 0xffffffff;\n selp.u32 %0, 1, 0, p;\n}\n" : "=r"(leader));
    constexpr uint32_t idesc = instr_desc_mn<kTcBM, NB>();
    const uint32_t base = smem_u32(smem);
    const uint64_t a0 = smem_desc_sw<C::XROW>(base, PAIR ? C::XBOX : C::XROW, 8 * C::XROW);
    const uint64_t b0 = smem_desc_sw<C::DROW>(base + C::XSLOT, C::DBOX, 8 * C::DROW);
    uint32_t acc = 0;
    for (int c = 0; c < nc; ++c) {
      const int st = c % S;
      if (!mbar_wait_ok(&full[st], (unsigned)(c / S) & 1u, true)) break;
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      // an address step of 16 bytes is 1 in the descriptors' low bits
      const uint64_t as = a0 + (uint64_t)(st * C::STAGE / 16), bs = b0 + (uint64_t)(st * C::STAGE / 16);
      if (leader) {
#pragma unroll
        for (int g = 0; g < C::NACC; ++g) {
          const int blk = PAIR ? 0 : g / C::MG, mg = PAIR ? g : g % C::MG;
#pragma unroll
          for (int k = 0; k < kTcBM / 16; ++k)
            tc_mma(tmem + (uint32_t)(g * NB), as + (uint64_t)((blk * C::XBOX + (mg * C::STACK + k * 16) * C::XROW) / 16),
                   bs + (uint64_t)(k * 16 * C::DROW / 16), idesc, k > 0 ? 1u : acc);
        }
        tc_commit(&empty[st]);
      }
      __syncwarp();
      acc = 1;
    }
    if (leader) tc_commit(done);
    __syncwarp();
    mbar_wait_ok(done, 0u, false);
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");

  // epilogue: TMEM lane = (kx block, input channel), or one of 128 input channels
  const int m = warp * 32 + lane;
  float* out = partial + (size_t)split * Cout * 9 * Cin;
#pragma unroll 1
  for (int g = 0; g < C::NACC; ++g) {
    const int blk = PAIR ? 0 : g / C::MG;
    const int kx = PAIR ? g : (g % C::MG) * C::STACK + m / CB;
    const int ci = ci0 + (PAIR ? m : blk * CB + m % CB);
#pragma unroll
    for (int cc = 0; cc < NB; cc += 16) {
      float v[16];
      tmem_ld16(tmem + ((uint32_t)(warp * 32) << 16) + (uint32_t)(g * NB + cc), v);
      if (kx < 3) {
#pragma unroll
        for (int i = 0; i < 16; ++i)
          out[((size_t)(co0 + cc + i) * 9 + ky * 3 + kx) * Cin + ci] = nc > 0 ? v[i] : 0.0f;
      }
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == 0) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(C::COLS) : "memory");
  }
}

// Sum of the splits' partials in order; sixteen loads are in flight while they are added.
__global__ void __launch_bounds__(64) k_wg_sum(const float* __restrict__ partial, int splits, size_t n,
                                               float* __restrict__ out) {
  const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const float* p = partial + i;
  float s = 0.0f;
  int k = 0;
  for (; k + 16 <= splits; k += 16, p += 16 * n) {
    float v[16];
#pragma unroll
    for (int j = 0; j < 16; ++j) v[j] = __ldg(p + j * n);
#pragma unroll
    for (int j = 0; j < 16; ++j) s += v[j];
  }
  for (; k < splits; ++k, p += n) s += __ldg(p);
  out[i] = s;
}

// Tensor map of an NHWC tensor with boxes of box_c channels x box_w pixels of one
// row, swizzled over the pixel's bytes.
inline int encode_rows_map(CUtensorMap* m, const bf16* p, int N, int H, int W, int C, int box_c, int box_w) {
  const fd::EncodeTiledFn fn = fd::encode_tiled_fn();
  FD_REQUIRE(fn != nullptr, FD_ERR_CUDA, "cuTensorMapEncodeTiled is not available from the driver");
  const cuuint64_t d[4] = {(cuuint64_t)C, (cuuint64_t)W, (cuuint64_t)H, (cuuint64_t)N};
  const cuuint64_t st[3] = {(cuuint64_t)C * 2, (cuuint64_t)W * C * 2, (cuuint64_t)H * W * C * 2};
  const cuuint32_t box[4] = {(cuuint32_t)box_c, (cuuint32_t)box_w, 1u, 1u}, e[4] = {1u, 1u, 1u, 1u};
  const CUtensorMapSwizzle sw = box_c == 64 ? CU_TENSOR_MAP_SWIZZLE_128B
                                            : (box_c == 32 ? CU_TENSOR_MAP_SWIZZLE_64B : CU_TENSOR_MAP_SWIZZLE_32B);
  const CUresult r = fn(m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 4, const_cast<bf16*>(p), d, st, box, e,
                        CU_TENSOR_MAP_INTERLEAVE_NONE, sw, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                        CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  FD_REQUIRE(r == CUDA_SUCCESS, FD_ERR_CUDA, "sg_conv3x3_wgrad_tc: tensor map (%d)", (int)r);
  return FD_OK;
}

template <int CB, int CIT, bool PAIR, int NB>
int launch_wgrad_tc(const bf16* x, const bf16* dz, int N, int H, int W, int Cin, int Cout, float* dw, float* partial,
                    size_t partial_floats, int splits, cudaStream_t s) {
  using C = WgCfg<CB, CIT, PAIR, NB>;
  auto kern = k_wgrad_tc<CB, CIT, PAIR, NB>;
  static std::atomic<unsigned long long> attr_done{0};
  if (fd::ensure_smem_attr(kern, 227 * 1024, attr_done) != cudaSuccess)
    return fd::check_launch("sg_conv3x3_wgrad_tc: shared-memory attribute");
  const long long nchunks = (long long)N * H * (W / kTcBM);
  const size_t n = (size_t)Cout * 9 * Cin;
  if (splits <= 0) {
    // The pixel ranges fix the order of every sum, so their count is a function of the shape and the device: about two
    // CTAs per SM when 128 channels of the larger count and a block of the other make a tile.  Below, it is cut to the
    // chunks and to what the buffer holds (sg_wgrad_partial_floats holds it on 152 SMs).
    const int sms = fd::sm_count();
    const int big = Cin > Cout ? Cin : Cout, small = Cin > Cout ? Cout : Cin;
    const int blk = small % 128 == 0 ? 128 : (small % 64 == 0 ? 64 : (small % 32 == 0 ? 32 : 16));
    const long long per = (long long)((big + 127) / 128) * (small / blk) * 3;
    splits = (int)std::max<long long>(1, (2LL * sms) / per);
  }
  if ((long long)splits > nchunks) splits = (int)nchunks;
  if ((size_t)splits * n > partial_floats) splits = (int)(partial_floats / n);
  FD_REQUIRE(splits >= 1, FD_ERR_ARG, "sg_conv3x3_wgrad_tc: partial buffer too small");
  const int cps = (int)((nchunks + splits - 1) / splits);
  // no more CTAs per SM than their tensor memory columns fit (512)
  int smem = C::SMEM;
  const int fit = 512 / C::COLS;
  if (kSmPerSmBytes / (smem + 1024) > fit) smem = kSmPerSmBytes / (fit + 1) - 1024 + 1;
  if (smem > 227 * 1024) smem = 227 * 1024;
  ConvMaps maps;
  if (int r = encode_rows_map(&maps.x, x, N, H, W, Cin, CB, kHaloPx)) return r;
  if (int r = encode_rows_map(&maps.w, dz, N, H, W, Cout, C::DB, kTcBM)) return r;
  dim3 grid((unsigned)(3 * splits), (unsigned)(Cin / (CB * CIT)), (unsigned)(Cout / NB));
  kern<<<grid, kTcThreads, smem, s>>>(maps, H, W, Cin, Cout, cps, nchunks, partial);
  k_wg_sum<<<(unsigned)((n + 63) / 64), 64, 0, s>>>(partial, splits, n, dw);
  return fd::check_launch("sg_conv3x3_wgrad_tc");
}

template <int CB, int CIT, bool PAIR>
int wgrad_tc_n(const bf16* x, const bf16* dz, int N, int H, int W, int Cin, int Cout, float* dw, float* partial,
               size_t pf, int splits, cudaStream_t s) {
  if constexpr (WgCfg<CB, CIT, PAIR, 16>::NACC * 128 <= 512) {
    if (Cout % 128 == 0) return launch_wgrad_tc<CB, CIT, PAIR, 128>(x, dz, N, H, W, Cin, Cout, dw, partial, pf, splits, s);
  }
  if (Cout % 64 == 0) return launch_wgrad_tc<CB, CIT, PAIR, 64>(x, dz, N, H, W, Cin, Cout, dw, partial, pf, splits, s);
  if (Cout % 32 == 0) return launch_wgrad_tc<CB, CIT, PAIR, 32>(x, dz, N, H, W, Cin, Cout, dw, partial, pf, splits, s);
  return launch_wgrad_tc<CB, CIT, PAIR, 16>(x, dz, N, H, W, Cin, Cout, dw, partial, pf, splits, s);
}

}  // namespace

int wgrad_error_word(unsigned* out, bool clear) { return tc_error_word(out, clear); }

}  // namespace sg

extern "C" {

int sg_conv3x3_wgrad_tc(const void* x, const void* dz, int N, int H, int W, int Cin, int Cout, float* dw,
                        float* partial, size_t partial_floats, int splits, void* stream) {
  FD_REQUIRE(x && dz && dw && partial && N > 0 && H > 0 && W > 0, FD_ERR_ARG, "sg_conv3x3_wgrad_tc: bad arguments");
  FD_REQUIRE(W % sg::kTcBM == 0 && Cin % 16 == 0 && Cout % 16 == 0 && Cin > 0 && Cout > 0, FD_ERR_SHAPE,
             "sg_conv3x3_wgrad_tc: needs W a multiple of 128 and channel counts multiples of 16 (got W=%d, %d -> %d)",
             W, Cin, Cout);
  FD_REQUIRE(((uintptr_t)x | (uintptr_t)dz | (uintptr_t)dw | (uintptr_t)partial) % 16 == 0, FD_ERR_ARG,
             "sg_conv3x3_wgrad_tc: tensors must be 16-byte aligned");
  using sg::bf16;
  cudaStream_t s = fd::as_stream(stream);
  const bf16 *xb = (const bf16*)x, *db = (const bf16*)dz;
  // input channels on the MMA's rows: pairs of 64, or blocks of 64, 32 or 16 beside their kx neighbours
  if (Cin % 128 == 0) return sg::wgrad_tc_n<64, 2, true>(xb, db, N, H, W, Cin, Cout, dw, partial, partial_floats, splits, s);
  if (Cin % 64 == 0) return sg::wgrad_tc_n<64, 1, false>(xb, db, N, H, W, Cin, Cout, dw, partial, partial_floats, splits, s);
  if (Cin % 96 == 0) return sg::wgrad_tc_n<32, 3, false>(xb, db, N, H, W, Cin, Cout, dw, partial, partial_floats, splits, s);
  if (Cin % 32 == 0) return sg::wgrad_tc_n<32, 1, false>(xb, db, N, H, W, Cin, Cout, dw, partial, partial_floats, splits, s);
  return sg::wgrad_tc_n<16, 1, false>(xb, db, N, H, W, Cin, Cout, dw, partial, partial_floats, splits, s);
}

}  // extern "C"

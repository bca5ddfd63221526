// What the tcgen05 kernels of the learned surrogate share: copies, mbarriers,
// matrix descriptors, MMAs and reads of tensor memory.
//
// Every mbarrier wait is bounded; a wait that gives up sets bit 0 of the unit's
// g_sg_tc_error (read by sg_tc_status) and the kernel continues without hanging;
// TMEM is always released.
#pragma once

#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>

#include "../../include/fdsurrogate.h"
#include "fd_host.h"
#include "fd_pdl.cuh"
#include "fd_tmap.h"

namespace sg {

// Whether this thread is launching the second or a later operation of a list
// (sg_run): its kernels may then start while the previous operation's drain.  An
// operation on its own starts in stream order.
extern thread_local bool t_op_follows;

namespace {

// This unit's copy of the status word: bit 0 is set when a bounded wait gave up
// (the library is built without relocatable device code; sg_tc_status combines
// the copies).
__device__ unsigned int g_sg_tc_error = 0;

inline int tc_error_word(unsigned* out, bool clear) {
  if (cudaMemcpyFromSymbol(out, g_sg_tc_error, sizeof(unsigned)) != cudaSuccess) return FD_ERR_CUDA;
  const unsigned zero = 0;
  if (clear && cudaMemcpyToSymbol(g_sg_tc_error, &zero, sizeof(unsigned)) != cudaSuccess) return FD_ERR_CUDA;
  return FD_OK;
}

using bf16 = __nv_bfloat16;
constexpr int kTcThreads = 128;
constexpr int kTcBM = 128;
constexpr unsigned kTcWaitLimit = 1u << 24;

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void cp16_l1(void* dst, const void* src, int src_bytes) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 16, %2;" ::"r"(smem_u32(dst)), "l"(src), "r"(src_bytes)
               : "memory");
}
__device__ __forceinline__ void cp16(void* dst, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_wait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

__device__ __forceinline__ void mbar_init(uint64_t* bar) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(bar)) : "memory");
}

// bounded wait for phase `parity` of an mbarrier
__device__ __forceinline__ void mbar_wait(uint64_t* bar, unsigned parity) {
  const uint32_t a = smem_u32(bar);
  for (unsigned it = 0; it < kTcWaitLimit; ++it) {
    uint32_t done;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
        : "=r"(done)
        : "r"(a), "r"(parity)
        : "memory");
    if (done) return;
  }
  atomicOr(&g_sg_tc_error, 1u);
}

// bounded wait that reports whether the phase completed.  `bail`: also give
// up once any wait of the launch has given up (the error word is set), so a
// failure common to every CTA does not cost every CTA a wait's full limit;
// the waits that drain copies and MMAs in flight before a CTA exits keep the
// full limit.
__device__ __forceinline__ bool mbar_wait_ok(uint64_t* bar, unsigned parity, bool bail) {
  const uint32_t a = smem_u32(bar);
  for (unsigned it = 0; it < kTcWaitLimit; ++it) {
    uint32_t done;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
        : "=r"(done)
        : "r"(a), "r"(parity)
        : "memory");
    if (done) return true;
    if (bail && (it & 1023u) == 1023u && *reinterpret_cast<volatile unsigned*>(&g_sg_tc_error) != 0u) return false;
  }
  atomicOr(&g_sg_tc_error, 1u);
  return false;
}

__device__ __forceinline__ void mbar_expect_tx(uint64_t* bar, unsigned bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes) : "memory");
}

// one box of a 3-D / 4-D tensor map into shared memory (128-byte aligned
// destination; the innermost coordinate times the element size a multiple of
// 16 bytes)
__device__ __forceinline__ void tma_load_3d(void* dst, const CUtensorMap* map, int c0, int c1, int c2,
                                            uint64_t* bar) {
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];" ::
          "r"(smem_u32(dst)),
      "l"(map), "r"(c0), "r"(c1), "r"(c2), "r"(smem_u32(bar))
      : "memory");
}
__device__ __forceinline__ void tma_load_4d(void* dst, const CUtensorMap* map, int c0, int c1, int c2, int c3,
                                            uint64_t* bar) {
  asm volatile(
      "cp.async.bulk.tensor.4d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4, %5}], "
      "[%6];" ::"r"(smem_u32(dst)),
      "l"(map), "r"(c0), "r"(c1), "r"(c2), "r"(c3), "r"(smem_u32(bar))
      : "memory");
}

// shared-memory matrix descriptor: canonical K-major layout, no swizzle
__device__ __forceinline__ uint64_t smem_desc(uint32_t addr, uint32_t lbo, uint32_t sbo) {
  uint64_t d = 0;
  d |= (uint64_t)((addr >> 4) & 0x3FFFu);
  d |= (uint64_t)((lbo >> 4) & 0x3FFFu) << 16;
  d |= (uint64_t)((sbo >> 4) & 0x3FFFu) << 32;
  d |= (uint64_t)1 << 46;  // descriptor version of this architecture
  return d;                // base offset 0, layout "no swizzle" (bits 61..63 = 0)
}

// instruction descriptor of kind::f16: D FP32, A and B bfloat16, both K-major
template <int M, int N>
__device__ __forceinline__ constexpr uint32_t instr_desc() {
  return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(N >> 3) << 17) | ((uint32_t)(M >> 4) << 24);
}

__device__ __forceinline__ void tc_mma(uint32_t tmem_d, uint64_t a, uint64_t b, uint32_t idesc, uint32_t acc) {
  asm volatile(
      "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"
      " tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}\n" ::"r"(tmem_d),
      "l"(a), "l"(b), "r"(idesc), "r"(acc)
      : "memory");
}

__device__ __forceinline__ void tc_commit(uint64_t* bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar))
               : "memory");
}

__device__ __forceinline__ float gelu_f(float z) {
  const float u = 0.7978845608028654f * fmaf(0.044715f * z * z, z, z);
  return 0.5f * z * (1.0f + tanhf(u));
}

// 32 lanes x 16 columns of 32-bit accumulators: thread t gets lane base+t, columns col..col+15
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, float (&v)[16]) {
  uint32_t r[16];
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
        "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr));
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
  for (int i = 0; i < 16; ++i) v[i] = __uint_as_float(r[i]);
}

// shared-memory matrix descriptor of operand rows swizzled over 32, 64 or 128 bytes
template <int ROW>
__device__ __forceinline__ uint64_t smem_desc_sw(uint32_t addr, uint32_t lbo, uint32_t sbo) {
  constexpr uint64_t layout = ROW == 128 ? 2u : (ROW == 64 ? 4u : 6u);
  return smem_desc(addr, lbo, sbo) | (layout << 61);
}

constexpr int kHaloPx = kTcBM + 2;             // pixels of a 128-pixel row with its halo
constexpr int kSmPerSmBytes = 233472;          // shared memory of an SM (228 KB), 1 KB of it reserved per CTA

struct ConvMaps {
  CUtensorMap x, w;
};

}  // namespace
}  // namespace sg

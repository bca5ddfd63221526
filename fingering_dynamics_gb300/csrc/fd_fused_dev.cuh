// What the kernels of the packed step share (the FP32 arithmetic is in
// fd_dev.cuh): their arguments, the packed layout with a storage type SF for
// the f deviations and g_1..g_8 (float, __half or __nv_bfloat16; g_0 is always
// stored in FP32), its conversions and the device status word.
//
// Packed population buffer (one per ping-pong side), planes of P = H*W
// elements, each plane starting on a 256-byte boundary:
//   9 planes SF  : (f_i - w_i) * 2^s_f            i = 0..8
//   1 plane  f32 : g_0
//   8 planes SF  : g_i * 2^s_g                    i = 1..8
#pragma once

#include <type_traits>

#include "fd_dev.cuh"

namespace fd {

inline size_t plane_bytes(size_t P, size_t elem) { return (P * elem + 255) / 256 * 256; }

// Device-side status word of the library's packed kernels:
//   bit 0 (kStatusWaitTimeout)  a bounded wait on an asynchronous copy gave up;
//   bit 1 (kStatusNonFinite)    a fused step met a non-finite density or psi in a
//                               fluid cell (numpy raises FloatingPointError there
//                               under the reference's np.seterr(all='raise'),
//                               fingering_periodic.py:496).
// The library is built without relocatable device code, so every translation
// unit that includes this header has its own copy, read and cleared through
// its own device_error_word(); fd_device_status() combines the copies.
constexpr unsigned kStatusWaitTimeout = 1u;
constexpr unsigned kStatusNonFinite = 2u;
__device__ unsigned int g_fd_device_error = 0;

namespace {
inline int device_error_word(unsigned* out, bool clear) {
  if (cudaMemcpyFromSymbol(out, g_fd_device_error, sizeof(unsigned)) != cudaSuccess) return FD_ERR_CUDA;
  if (clear) {
    const unsigned zero = 0;
    if (cudaMemcpyToSymbol(g_fd_device_error, &zero, sizeof(unsigned)) != cudaSuccess) return FD_ERR_CUDA;
  }
  return FD_OK;
}
}  // namespace

// true if rho or psi of a fluid cell is not finite (NaN or +-inf)
__device__ __forceinline__ bool nonfinite_cell(float rho, float psi) { return !(fabsf(rho) + fabsf(psi) < INFINITY); }

template <typename SF>
struct DevArgs {
  DevCoef c;
  int H, W, variant, nchunks, nstrips, R;
  size_t P, pstride_f;  // plane size and plane stride (elements of SF)
  const uint16_t* __restrict__ mask;
  const double* __restrict__ inlet_ux;
  const SF* __restrict__ src_f;
  const float* __restrict__ src_g0;
  const SF* __restrict__ src_gi;  // plane i>=1 at src_gi + (i-1)*pstride_f
  SF* __restrict__ dst_f;
  float* __restrict__ dst_g0;
  SF* __restrict__ dst_gi;
  const float* __restrict__ side_in;
  float* __restrict__ side_out;
  uint32_t seed;  // stochastic rounding: sr_hash of the step's seed
  // where a non-finite cell is reported: a batch member's status word (set to
  // 1; the batched kernel skips the member's tiles from then on), or null for
  // the unit's device status word (bit kStatusNonFinite)
  unsigned* status;
};

template <typename SF>
__device__ __forceinline__ void report_nonfinite(const DevArgs<SF>& a) {
  if (a.status) atomicOr(a.status, 1u);
  else atomicOr(&g_fd_device_error, kStatusNonFinite);
}

// ---- pack / unpack between the reference layout (18 planes of T) and the
// packed deviation layout ------------------------------------------------------
template <typename T, typename SF>
__global__ void k_pack(size_t P, size_t pstride, DevCoef c, const T* __restrict__ src, SF* __restrict__ f,
                       float* __restrict__ g0, SF* __restrict__ gi) {
  const size_t q = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (q >= P) return;
#pragma unroll
  for (int i = 0; i < 9; ++i) f[i * pstride + q] = from_f<SF>(((float)src[i * P + q] - c.w[i]) * c.sf);
  g0[q] = (float)src[9 * P + q];
#pragma unroll
  for (int i = 1; i < 9; ++i) gi[(i - 1) * pstride + q] = from_f<SF>((float)src[(9 + i) * P + q] * c.sg);
}

template <typename T, typename SF>
__global__ void k_unpack(size_t P, size_t pstride, DevCoef c, const SF* __restrict__ f, const float* __restrict__ g0,
                         const SF* __restrict__ gi, T* __restrict__ dst) {
  const size_t q = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (q >= P) return;
#pragma unroll
  for (int i = 0; i < 9; ++i) dst[i * P + q] = (T)(to_f<SF>(f[i * pstride + q]) * c.inv_sf + c.w[i]);
  dst[9 * P + q] = (T)g0[q];
#pragma unroll
  for (int i = 1; i < 9; ++i) dst[(9 + i) * P + q] = (T)(to_f<SF>(gi[(i - 1) * pstride + q]) * c.inv_sg);
}

template <typename SF>
struct PackedLayout {
  size_t P, pstride;
  size_t off_f, off_g0, off_gi, total;
};

template <typename SF>
inline PackedLayout<SF> packed_layout(int H, int W) {
  PackedLayout<SF> L;
  L.P = (size_t)H * W;
  const size_t bf = plane_bytes(L.P, sizeof(SF));
  L.pstride = bf / sizeof(SF);
  L.off_f = 0;
  L.off_g0 = 9 * bf;
  L.off_gi = L.off_g0 + plane_bytes(L.P, sizeof(float));
  L.total = L.off_gi + 8 * bf;
  return L;
}

template <typename T, typename SF>
int launch_pack(const fd_params& p, const DevCoef& c, const void* src, char* dst, cudaStream_t st) {
  const PackedLayout<SF> L = packed_layout<SF>(p.H, p.W);
  k_pack<T, SF><<<(unsigned)((L.P + 255) / 256), 256, 0, st>>>(
      L.P, L.pstride, c, (const T*)src, reinterpret_cast<SF*>(dst + L.off_f), reinterpret_cast<float*>(dst + L.off_g0),
      reinterpret_cast<SF*>(dst + L.off_gi));
  return cudaGetLastError() == cudaSuccess ? FD_OK : FD_ERR_CUDA;
}

template <typename T, typename SF>
int launch_unpack(const fd_params& p, const DevCoef& c, const char* src, void* dst, cudaStream_t st) {
  const PackedLayout<SF> L = packed_layout<SF>(p.H, p.W);
  k_unpack<T, SF><<<(unsigned)((L.P + 255) / 256), 256, 0, st>>>(
      L.P, L.pstride, c, reinterpret_cast<const SF*>(src + L.off_f), reinterpret_cast<const float*>(src + L.off_g0),
      reinterpret_cast<const SF*>(src + L.off_gi), (T*)dst);
  return cudaGetLastError() == cudaSuccess ? FD_OK : FD_ERR_CUDA;
}

}  // namespace fd

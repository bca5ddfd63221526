/* fdsurrogate.h - C ABI of the learned surrogate's CUDA kernels (libfdlbm.so).
 *
 * The reference has no learned component; nothing here replaces reference
 * code.  These are the training and inference kernels of a small convolutional
 * U-Net that advances (psi, u_x, u_y) by a fixed number of lattice steps given
 * the solid mask (the network is defined in fingering_dynamics_gb300/surrogate.py;
 * a float64 numpy restatement is the test oracle).
 *
 * Conventions: every pointer is device memory; activations are NHWC bfloat16
 * with the channel dimension innermost (P = N*H*W pixels); conv weights are
 * bfloat16 [Cout][3][3][Cin] ("same" zero padding, stride 1); channel counts
 * are multiples of 16; accumulation is FP32.  Calls are asynchronous on
 * `stream` and return FD_OK (0) or a negative fd_status (fdlbm.h), with the
 * message in fd_last_error().
 */
#ifndef FDSURROGATE_H
#define FDSURROGATE_H

#include <stddef.h>
#include <stdint.h>

#ifdef __cplusplus
extern "C" {
#endif

enum sg_act { SG_ACT_NONE = 0, SG_ACT_GELU = 1 };

/* z = conv3x3(x, w) + bias (bias may be NULL); y = act(z).  z may be NULL
 * (not stored); y may equal z when act == SG_ACT_NONE.  Implicit GEMM on the
 * tensor cores (M = P pixels, N = Cout, K = 9*Cin). */
int sg_conv3x3(const void* x, int N, int H, int W, int Cin, const void* w, const float* bias, int Cout, int act,
               void* z, void* y, void* stream);

/* sg_conv3x3 on the fifth-generation tensor cores (tcgen05.mma, operands in
 * shared memory through matrix descriptors, accumulator in tensor memory);
 * same arguments and results.  sg_tc_status reads (and optionally clears) its
 * device error word: bit 0 = an mbarrier wait gave up. */
int sg_conv3x3_tc(const void* x, int N, int H, int W, int Cin, const void* w, const float* bias, int Cout, int act,
                  void* z, void* y, void* stream);
int sg_tc_status(unsigned* out, int clear);

/* sg_conv3x3_tc as a persistent kernel fed by the tensor memory accelerator:
 * one warp loads the operands as swizzled tensor-map boxes (zero fill outside
 * the image = the padding) into a ring of stages, one issues the MMAs as each
 * lands into one of two accumulator buffers, eight finish the previous tile.
 * Same arguments and results; needs W a multiple of 128 and Cin, Cout multiples
 * of 16 (FD_ERR_SHAPE otherwise).  Its waits share sg_tc_status's error word. */
int sg_conv3x3_tma(const void* x, int N, int H, int W, int Cin, const void* w, const float* bias, int Cout, int act,
                   void* z, void* y, void* stream);

/* The same kernel under the name of what was its persistent form. */
int sg_conv3x3_tma_ws(const void* x, int N, int H, int W, int Cin, const void* w, const float* bias, int Cout,
                      int act, void* z, void* y, void* stream);

/* wt[ci][ky][kx][co] = w[co][2-ky][2-kx][ci]: the weights of the data-gradient
 * convolution (dx = sg_conv3x3(dz, wt)). */
int sg_flip_weights(const void* w, int Cin, int Cout, void* wt, void* stream);

/* dw[co][ky][kx][ci] = sum_p dz[p][co] x[p + (ky-1, kx-1)][ci] (FP32 out,
 * overwritten), split over `splits` pixel ranges whose FP32 partial sums go
 * to `partial` (splits*Cout*9*Cin floats) and are added in a fixed order:
 * the result does not depend on scheduling.  splits <= 0 picks a split. */
int sg_conv3x3_wgrad(const void* x, const void* dz, int N, int H, int W, int Cin, int Cout, float* dw,
                     float* partial, size_t partial_floats, int splits, void* stream);

/* sg_conv3x3_wgrad on the fifth-generation tensor cores: MMA rows (kx, input
 * channel), columns output channels, K = pixels; the same FP32 partials added in
 * a fixed order.  Same arguments and result; needs W a multiple of 128 and Cin,
 * Cout multiples of 16 (FD_ERR_SHAPE otherwise); splits <= 0 picks a count from
 * the shape, within what `partial` holds. */
int sg_conv3x3_wgrad_tc(const void* x, const void* dz, int N, int H, int W, int Cin, int Cout, float* dw,
                        float* partial, size_t partial_floats, int splits, void* stream);

/* Floats of `partial` that sg_conv3x3_wgrad and sg_conv3x3_wgrad_tc need with splits <= 0. */
size_t sg_wgrad_partial_floats(int N, int H, int W, int Cin, int Cout);

/* db[c] = sum_p dz[p][c] (FP32, fixed order; partial: sg_bias_partial_floats). */
int sg_bias_grad(const void* dz, size_t P, int C, float* db, float* partial, void* stream);
size_t sg_bias_partial_floats(int C);

/* dz = dy * GELU'(z) (tanh form), n elements. */
int sg_gelu_bwd(const void* dy, const void* z, size_t n, void* dz, void* stream);

/* 2x2 mean pooling of x (N,H,W,C) -> y (N,H/2,W/2,C) and its backward. */
int sg_pool2(const void* x, int N, int H, int W, int C, void* y, void* stream);
int sg_pool2_bwd(const void* dy, int N, int H, int W, int C, void* dx, void* stream);

/* Nearest 2x upsampling of x (N,h,w,C) into channels [coff, coff+C) of y
 * (N,2h,2w,Cy), and its backward (dx = sum of the 4 copies). */
int sg_up2(const void* x, int N, int h, int w, int C, void* y, int Cy, int coff, void* stream);
int sg_up2_bwd(const void* dy, int N, int h, int w, int Cy, int coff, int C, void* dx, void* stream);

/* dst[p][coff + c] = src[p][c] (c < Cs): a skip connection into a concatenation. */
int sg_copy_channels(const void* src, size_t P, int Cs, void* dst, int Cd, int coff, void* stream);

/* dst[p][c] += src[p][coff + c] (c < C): the skip connection's gradient. */
int sg_add_channels(const void* src, size_t P, int Cs, int coff, int C, void* dst, void* stream);

/* Masked MSE of prediction = x[..., 0:3] + out[..., 0:3] against target =
 * xn[..., 0:3] over pixels whose solid channel x[..., 3] is 0 (all three
 * tensors NHWC with C channels).  dout (C channels, zero beyond 3) =
 * d loss / d out; loss_partial receives per-block sums (sg_loss_blocks()
 * floats) of squared error and of fluid pixels, added by the caller. */
int sg_masked_mse(const void* x, const void* out, const void* xn, size_t P, int C, void* dout, float* loss_partial,
                  float inv_count, void* stream);
int sg_loss_blocks(void);

/* Decoupled-weight-decay Adam on FP32 master weights w (n), writing the
 * bfloat16 copy w16 (may be NULL); step >= 1. */
int sg_adamw(float* w, void* w16, const float* g, float* m, float* v, size_t n, float lr, float beta1, float beta2,
             float eps, float weight_decay, int step, void* stream);

/* sg_adamw over a HOST list of tensors in one launch. */
#define SG_ADAMW_MAX 40
typedef struct sg_adamw_item {
  float* w;
  void* w16; /* may be NULL */
  const float* g;
  float *m, *v;
  size_t n;
  float weight_decay;
} sg_adamw_item;
int sg_adamw_list(const sg_adamw_item* items, int count, float lr, float beta1, float beta2, float eps, int step,
                  void* stream);

/* sg_gelu_bwd and sg_bias_grad of a layer (N,H,W,C) in one pass, the gradient dy
 * taken from where it arises: a tensor (SG_DY_PLAIN), the backward of sg_up2
 * (SG_DY_UP: dy is (N,2H,2W,Cy), channels [coff, coff+C)), or the backward of
 * sg_pool2 plus a skip connection (SG_DY_POOL: dy is (N,H/2,W/2,C), skip
 * (N,H,W,Cy), channels [coff, coff+C)).  The same bits as the separate calls. */
enum sg_dy { SG_DY_PLAIN = 0, SG_DY_UP = 1, SG_DY_POOL = 2 };
int sg_gelu_bias_bwd(int source, const void* dy, const void* skip, int N, int H, int W, int Cy, int coff, const void* z,
                     int C, void* dz, float* db, float* partial, void* stream);

/* y (N,2h,2w,C+Cs) = [sg_up2 of x, skip]: sg_up2 and sg_copy_channels in one pass. */
int sg_up2_concat(const void* x, int N, int h, int w, int C, const void* skip, int Cs, void* y, void* stream);

/* Scales of the masked loss from the batch itself, without the host waiting:
 * *count = fluid pixels, inv[0] = 1 / (3 max(count, 1)) for sg_masked_mse_scaled
 * (sg_masked_mse with its inv_count in device memory), inv[1] the reciprocal of
 * 3 max(count, 1) in single precision (device memory). */
int sg_loss_scale(const void* x, size_t P, int C, unsigned* count, float* inv, void* stream);
int sg_masked_mse_scaled(const void* x, const void* out, const void* xn, size_t P, int C, void* dout,
                         float* loss_partial, const float* inv, void* stream);

/* y = x (NHWC, C channels) with its first three channels replaced by x + out. */
int sg_add_prediction(const void* x, const void* out, size_t P, int C, void* y, void* stream);

/* A HOST list of the calls above on one stream, in order: a network's pass in one
 * call (from Python a call of each costs more than its kernel on small batches).
 * i and p are the call's integers and pointers in their order, without the
 * stream; a weight gradient's i[5] is partial_floats and its split automatic.
 * Stops at the first call that fails and returns its status. */
enum sg_op_kind {
  SG_OP_CONV = 0,       /* sg_conv3x3:        i N H W Cin Cout act; p x w bias z y */
  SG_OP_CONV_TC = 1,    /* sg_conv3x3_tc */
  SG_OP_CONV_TMA = 2,   /* sg_conv3x3_tma */
  SG_OP_WGRAD = 3,      /* sg_conv3x3_wgrad:  i N H W Cin Cout partial_floats; p x dz dw partial */
  SG_OP_WGRAD_TC = 4,   /* sg_conv3x3_wgrad_tc */
  SG_OP_POOL = 5,       /* sg_pool2:          i N H W C; p x y */
  SG_OP_UP_CONCAT = 6,  /* sg_up2_concat:     i N h w C Cs; p x skip y */
  SG_OP_GELU_BIAS = 7,  /* sg_gelu_bias_bwd:  i source N H W Cy coff C; p dy skip z dz db partial */
  SG_OP_BIAS = 8,       /* sg_bias_grad:      i P C; p dz db partial */
  SG_OP_FLIP = 9,       /* sg_flip_weights:   i Cin Cout; p w wt */
  SG_OP_ADD_PREDICTION = 10 /* sg_add_prediction: i P C; p x out y */
};
typedef struct sg_op {
  int64_t kind;
  int64_t i[8];
  uint64_t p[7];
} sg_op;
int sg_run(const sg_op* ops, int count, void* stream);

/* The network's frame of n cells: 16 bfloat16 channels psi, u_x inv_u, u_y inv_u
 * (0 on solid cells), solid, zeros, from FP32 (f64 = 0) or FP64 fields and a byte
 * per cell.  out: 32-byte aligned. */
int sg_frame(const void* psi, const void* ux, const void* uy, const void* solid, size_t n, int f64, float inv_u,
             void* out, void* stream);

/* FP32 -> bfloat16 (round to nearest even), n elements. */
int sg_to_bf16(const float* src, size_t n, void* dst, void* stream);

#ifdef __cplusplus
}
#endif

#endif /* FDSURROGATE_H */

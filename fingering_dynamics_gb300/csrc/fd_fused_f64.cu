// FP64 fused step.  Built with -fmad=false: the per-cell arithmetic is the
// reference's operand order without contraction (fd_exact_cell.h places its
// FMAs where they change no bit), so the fused FP64 step equals the
// reference-order kernels (and the reference) bit for bit.
#include "fd_exact.cuh"
#include "fd_host.h"

namespace fd {
// R, the rows per warp that a caller may ask for, shapes the FP32 kernel only.
int fused_f64(const fd_params& p, const uint16_t* mask, const double* inlet_ux, void* pa, void* pb, void* sa, void* sb,
              int nsteps, int R, cudaStream_t st) {
  ExactArgs ea{};
  ea.a.c = make_coef<double>(p);
  ea.a.H = p.H;
  ea.a.W = p.W;
  ea.a.variant = p.variant;
  ea.a.mask = mask;
  ea.a.inlet_ux = inlet_ux;
  const Coef<double>& c = ea.a.c;
  ea.k = make_exact_const(c.w[0], c.w[1], c.a, c.kappa, c.eta_n, c.eta_n_M, c.c_a0, c.c_b0, c.c_b18, c.one_third,
                          c.tau_inv);
  // Tiles of 8 rows, one cell a thread, where they give every SM five CTAs or more
  // (three are resident); below, tiles of 4 rows.  us per iteration, 8 / 4 rows, 152 SMs:
  // 400 x 400 (650 tiles of 8 rows) 105 / 97, 1764 x 128 (884) 139 / 150, 512 x 512
  // 140 / 139, 512 x 1024 242 / 253, 1024 x 2048 819 / 895.
  const long long tiles = (long long)((p.W + kExactTX - 1) / kExactTX) * ((p.H + 7) / 8);
  if (tiles < 5 * sm_count()) return launch_exact<4>(ea, p, (double*)pa, (double*)pb, (double*)sa, (double*)sb, nsteps, st);
  return launch_exact<8>(ea, p, (double*)pa, (double*)pb, (double*)sa, (double*)sb, nsteps, st);
}
}  // namespace fd

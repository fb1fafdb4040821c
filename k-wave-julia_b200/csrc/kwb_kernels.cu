// Time-step kernels of libkwb.
//
// One time step of KWave.jl's time_step_{1,2,3}d! (KWave.jl/src/solver/first_order_steps.jl:
// 296-535) is executed as:
//
//   [k_tr_inject]                      time-reversal injection (first_order.jl:450-460, 678-689)
// (k_line_pass, k_eos_x_*, k_spec_pass: kwb_generic.cu, or for the lengths of kwb_fast.cu its register
// passes; this file holds the others and the launchers that choose)
//
//   k_line_pass(axis) for every axis   fused: d/dx_d p -> u_d update (split PML) -> u source ->
//                                      d/dx_d u_d -> rho_d update (split PML) -> p source
//                                      (first_order_steps.jl:400-428, 489-521, 586-715)
//   k_eos_x_fwd                        EOS prologue (sum rho_d, nonlinearity, c^2) + x R2C
//   k_spec_pass(y [,z])                y/z FFTs of the half spectrum, EOS multiply innermost
//   k_eos_x_inv                        x C2R -> p                  (first_order_steps.jl:214-290)
//   k_sensor_gather per sensor group   record_sensor_data!         (first_order_steps.jl:728-811)
//
// The gradient along axis d is computed on lines along d only: a full N-D rfft, a multiply by
// i k_d e^{+-i k_d d/2} and an N-D irfft (fft_utils.jl:247-303) equal the 1-D transform along
// d, because the multiplier is Hermitian (it is real at the Nyquist bin).  Two real lines are
// transformed as one complex line (a + i b) for the same reason.
#include <algorithm>
#include <map>
#include <mutex>

#include "kwb_fft.cuh"
#include "kwb_record.cuh"
#include "kwb_tiles.cuh"

namespace kwb {

// ------------------------------------------------------------------------------------------
// time reversal, sensors, control
// ------------------------------------------------------------------------------------------

__global__ void k_tr_inject(const SimDev *__restrict__ sims, long long step_s) {
  KWB_STEP_KERNEL_PROLOGUE();
  const SimDev &S = sims[0];
  const long long t = step_index(S, step_s);
  if (t >= S.Nt) return;
  const long long j = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (j >= S.n_tr) return;
  const long long col = S.Nt - 1 - t;  // tr_t = Nt - t_index + 1 (1-based)
  const float val = S.tr_sig[col * S.n_tr + j];
  const long long v = S.tr_idx[j];
  for (int d = 0; d < S.D; ++d) S.rho[d][v] = val;
}

__global__ void k_sensor_gather(const SimDev *__restrict__ sims, const GroupDev *__restrict__ gp,
                                long long step_s) {
  KWB_STEP_KERNEL_PROLOGUE();
  const SimDev &S = sims[0];
  const long long t = step_index(S, step_s);
  if (t >= S.Nt) return;
  const GroupDev &g = *gp;
  const long long j = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (j >= g.n) return;
  const long long v = g.dense ? j : g.idx[j];
  record_point(S, g, t, j, S.p[v], [&](int d) { return S.u[d][v]; });
}

__global__ void k_advance_t0(long long *t0, long long k) {
  KWB_STEP_KERNEL_PROLOGUE();
  if (threadIdx.x == 0 && blockIdx.x == 0) *t0 += k;
}

// ------------------------------------------------------------------------------------------
// launchers
// ------------------------------------------------------------------------------------------

static int cdiv(long long a, long long b) { return (int)((a + b - 1) / b); }

// The dynamic shared-memory limit of a kernel is a per-function attribute.  It is raised once to
// the device's opt-in maximum, so simulations of different sizes in one process never lower
// it under one another.
cudaError_t raise_dynamic_smem(const void *fn, size_t bytes) {
  // the limit a kernel was given, per device: later calls that fit it make no API call
  static std::mutex mu;
  static std::map<std::pair<int, const void *>, size_t> given;
  int cur = 0;
  cudaError_t e = cudaGetDevice(&cur);
  if (e != cudaSuccess) return e;
  std::lock_guard<std::mutex> lk(mu);
  const auto key = std::make_pair(cur, fn);
  auto it = given.find(key);
  if (it != given.end() && bytes <= it->second) return cudaSuccess;
  cudaFuncAttributes fa;
  e = cudaFuncGetAttributes(&fa, fn);
  if (e != cudaSuccess) return e;
  if (bytes + fa.sharedSizeBytes <= 48 * 1024) {
    given[key] = 48 * 1024 - fa.sharedSizeBytes;
    return cudaSuccess;
  }
  int optin = 0;
  e = cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, cur);
  if (e != cudaSuccess) return e;
  const size_t room = (size_t)optin > fa.sharedSizeBytes ? (size_t)optin - fa.sharedSizeBytes : 0;
  if (bytes > room) return cudaErrorInvalidValue;
  e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)room);
  if (e == cudaSuccess) given[key] = room;
  return e;
}

cudaError_t launch_line_pass(const SimDev *d_sim, const SimDev &h, int axis, int mode,
                             long long step_s, cudaStream_t st) {
  if ((h.fast & 1) && fast_size(h.N[axis]) && (axis == 0 || h.N[0] % 4 == 0)) return fast_line_pass(d_sim, h, axis, mode, step_s, st);
  return generic_line_pass(h, axis, mode, step_s, st);
}

cudaError_t launch_eos_x_fwd(const SimDev *d_sim, const SimDev &h, long long step_s,
                             cudaStream_t st) {
  if ((h.fast & 2) && h.ndim >= 2 && fast_size(h.N[0])) return fast_eos(d_sim, h, true, step_s, st);
  return generic_eos(h, true, step_s, st);
}

cudaError_t launch_eos_x_inv(const SimDev *d_sim, const SimDev &h, long long step_s,
                             cudaStream_t st) {
  if ((h.fast & 2) && h.ndim >= 2 && fast_size(h.N[0])) return fast_eos(d_sim, h, false, step_s, st);
  return generic_eos(h, false, step_s, st);
}

cudaError_t launch_spec_pass(const SimDev *d_sim, const SimDev &h, int axis, int op,
                             long long step_s, cudaStream_t st) {
  if ((h.fast & 2) && fast_size(h.N[axis])) return fast_spec(d_sim, h, axis, op, step_s, st);
  return generic_spec(h, axis, op, step_s, st);
}

cudaError_t launch_change_spectrum(const SimDev &h, long long step_s, cudaStream_t st) {
  if (h.dispersion != KWB_DISP_CHANGE) return cudaSuccess;
  SimDev c = h;  // on the in-place passes, with spec2 in the place of spec
  c.spec = h.spec2;
  cudaError_t e = generic_eos(c, true, step_s, st, true);
  for (int a = 1; a < h.ndim && e == cudaSuccess; ++a) e = generic_spec(c, a, KWB_SPEC_FWD, step_s, st);
  return e;
}

cudaError_t launch_tr_inject(const SimDev *d_sim, const SimDev &h, long long step_s,
                             cudaStream_t st) {
  if (h.n_tr <= 0) return cudaSuccess;
  kwb_launch(k_tr_inject, cdiv(h.n_tr, 256), 256, 0, st, d_sim, step_s);
  return cudaGetLastError();
}

cudaError_t launch_sensor_gather(const SimDev *d_sim, const SimDev &h, const GroupDev *d_group,
                                 long long n, long long step_s, cudaStream_t st) {
  (void)h;
  if (n <= 0) return cudaSuccess;
  kwb_launch(k_sensor_gather, cdiv(n, 256), 256, 0, st, d_sim, d_group, step_s);
  return cudaGetLastError();
}

cudaError_t prime_attributes(const SimDev &h) {
  cudaError_t e = generic_prime(h);
  if (e != cudaSuccess) return e;
  if (h.fast)
    for (int a = 0; a < h.ndim; ++a)
      if (fast_size(h.N[a]) && (e = fast_prime(h.N[a])) != cudaSuccess) return e;
  if (h.plane && (e = fast_plane_prime()) != cudaSuccess) return e;
  return cudaSuccess;
}

cudaError_t launch_advance_t0(long long *t0, long long k, cudaStream_t st) {
  kwb_launch(k_advance_t0, 1, 32, 0, st, t0, k);
  return cudaGetLastError();
}

}  // namespace kwb

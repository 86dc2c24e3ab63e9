// gg_checks.cu -- device functions of the ray path exported one by one, so
// that tests can compare them bit for bit with the oracle on identical
// inputs.  No counterpart in the reference; not used by any render.
//
// The starfield (sky.rs:26-40) hashes the f64 bits of a ray's final
// direction, so a one-ulp difference anywhere before it moves a star.  A
// full-frame comparison only shows that the two sides agree where their
// directions agree; these entries feed the device code and the oracle the
// same directions (and the same velocities for spatial_dir) instead.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>
#include <new>
#include <vector>

#include "../../include/gargantua_gpu.h"
#include "gg_device.cuh"
#include "gg_host.h"
#include "gg_mixed.cuh"
#include "gg_vjp.cuh"

namespace {

__global__ void sky_dir_kernel(const double* __restrict__ dirs, double* __restrict__ rgb,
                               uint64_t n) {
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (uint64_t)gridDim.x * blockDim.x) {
    double c[3];
    gg::procedural_sky_dir(dirs[3 * i], dirs[3 * i + 1], dirs[3 * i + 2], c);
    rgb[3 * i] = c[0];
    rgb[3 * i + 1] = c[1];
    rgb[3 * i + 2] = c[2];
  }
}

__global__ void spatial_dir_kernel(const double* __restrict__ vel, double* __restrict__ dirs,
                                   uint64_t n) {
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (uint64_t)gridDim.x * blockDim.x) {
    const double v[4] = {vel[4 * i], vel[4 * i + 1], vel[4 * i + 2], vel[4 * i + 3]};
    gg::spatial_dir(v, dirs[3 * i], dirs[3 * i + 1], dirs[3 * i + 2]);
  }
}

// 12 doubles in per point (M, a, r, theta, w[4], kb[4]); 7 out (kb . da/dr,
// da/dtheta, da/dw[4], da/da).
__global__ void kerr_vjp_kernel(const double* __restrict__ in, double* __restrict__ out,
                                uint64_t n, int form) {
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (uint64_t)gridDim.x * blockDim.x) {
    const double* q = in + 12 * i;
    const double w[4] = {q[4], q[5], q[6], q[7]};
    const double kb[4] = {q[8], q[9], q[10], q[11]};
    double Xr = 0.0, Xth = 0.0, W[4] = {0.0, 0.0, 0.0, 0.0}, ga = 0.0;
    if (form == 0)
      gg::kerr_rhs_vjp_hand(q[0], q[1], q[2], q[3], w, kb, &Xr, &Xth, W, &ga);
    else
      gg::kerr_rhs_vjp_dual(q[0], q[1], q[2], q[3], w, kb, &Xr, &Xth, W, &ga);
    double* o = out + 7 * i;
    o[0] = Xr;
    o[1] = Xth;
    o[2] = W[0];
    o[3] = W[1];
    o[4] = W[2];
    o[5] = W[3];
    o[6] = ga;
  }
}

__global__ void step_factor_kernel(const double* __restrict__ s2, double* __restrict__ out,
                                   uint64_t n) {
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (uint64_t)gridDim.x * blockDim.x)
    out[i] = gg::root10_8_over(s2[i]);
}

__global__ void rcp_kernel(const float* __restrict__ x, float* __restrict__ out, uint64_t n) {
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (uint64_t)gridDim.x * blockDim.x)
    out[i] = gg::rcp(x[i]);
}

// `attempts` attempts of every ray of a small frame from the camera, or until it
// ends: its state and step (x, v, lambda, h), and how many attempts it made, how
// many were accepted and how many were at max_step.  FORM 0: the reference's
// step, 1: full Dormand-Prince, 2: that in mixed precision (up to the FP64 band).
template <int METRIC, int FORM, bool STEADY>
__global__ void __launch_bounds__(gg::kTraceBlock)
    steps_kernel(const __grid_constant__ gg::DevParams P, uint32_t attempts, double* state,
                 uint32_t* counts) {
  __shared__ double2 k_smem[FORM == 2 ? 1 : 7][2][gg::kTraceBlock];
  __shared__ __align__(16) char m_smem[FORM == 2 ? gg::mixed_smem_bytes<gg::kTraceBlock>() : 16];
  const uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= P.n_rays) return;
  gg::Ray R;
  double u, v;
  gg::sample_uv(P, i, u, v);
  gg::init_ray(P, u, v, R);
  bool k1_valid = false, k7_pending = false, acc = false;
  uint32_t n_att = 0, n_acc = 0, n_max = 0;
  if constexpr (FORM == 2) {
    const gg::MixedSmem K = gg::MixedSmem::at(m_smem);
    gg::MixedRegs S;
    gg::mixed_load(R, i, K, S);
    for (; n_att < attempts; ++n_att) {
      const float r = K.comp(gg::kSlotXh, 1), th = K.comp(gg::kSlotXh, 2);
      if (r < P.band_r || th < P.pole_band || th > gg::kPiHi - P.pole_band) break;
      n_max += S.h == P.max_step;
      float hf = 0.0f;
      if (gg::attempt_dp45_mixed<METRIC, STEADY>(P, S, K, k1_valid, k7_pending, acc, hf) !=
          gg::kContinue)
        break;
      const float th_a = th + K.comp(gg::kSlotDx, 2);
      if (acc && !(th_a > 0.0f && th_a < gg::kPiHi)) break;
      if (acc) gg::mixed_advance(S, K, hf, k1_valid, k7_pending);
      n_acc += acc;
    }
    R = gg::mixed_fp64(K, S);
  } else {
    const gg::KStore K{k_smem};
    for (; n_att < attempts; ++n_att) {
      n_max += R.h == P.max_step;
      double h_used = 0.0;
      int res;
      if constexpr (FORM == 1) {
        gg::StepEnd end;
        res = gg::attempt_dp45_fp64<METRIC, gg::kStageArms, STEADY>(P, R, K, k1_valid, k7_pending,
                                                                    acc, h_used, end);
      } else {
        res = gg::attempt_fp64<METRIC, false, STEADY>(P, R, K, k1_valid, acc, h_used);
      }
      if (res != gg::kContinue) break;
      n_acc += acc;
    }
  }
  double* o = state + 10 * i;
#pragma unroll
  for (int c = 0; c < 4; ++c) {
    o[c] = R.x[c];
    o[4 + c] = R.v[c];
  }
  o[8] = R.lam;
  o[9] = R.h;
  counts[3 * i] = n_att;
  counts[3 * i + 1] = n_acc;
  counts[3 * i + 2] = n_max;
}

template <int METRIC, int FORM>
void launch_steps(const gg::DevParams& P, bool steady, uint32_t attempts, double* state,
                  uint32_t* counts, cudaStream_t s) {
  const unsigned blocks = (unsigned)((P.n_rays + gg::kTraceBlock - 1) / gg::kTraceBlock);
  if (steady)
    steps_kernel<METRIC, FORM, true><<<blocks, gg::kTraceBlock, 0, s>>>(P, attempts, state, counts);
  else
    steps_kernel<METRIC, FORM, false><<<blocks, gg::kTraceBlock, 0, s>>>(P, attempts, state, counts);
}

template <int METRIC>
void launch_steps_form(int form, const gg::DevParams& P, bool steady, uint32_t attempts,
                       double* state, uint32_t* counts, cudaStream_t s) {
  if (form == 0) launch_steps<METRIC, 0>(P, steady, attempts, state, counts, s);
  else if (form == 1) launch_steps<METRIC, 1>(P, steady, attempts, state, counts, s);
  else launch_steps<METRIC, 2>(P, steady, attempts, state, counts, s);
}

int launch_status() {
  const cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? GG_OK : GG_ERR_CUDA;
}

}  // namespace

extern "C" GG_API int gg_check_procedural_sky(const double* dirs_dev, double* rgb_dev, uint64_t n,
                                              void* stream) {
  if (n == 0) return GG_OK;
  if (!dirs_dev || !rgb_dev) return GG_ERR_INVALID_ARG;
  const uint64_t blocks = (n + 255) / 256;
  sky_dir_kernel<<<(unsigned)(blocks < 4096 ? blocks : 4096), 256, 0,
                   static_cast<cudaStream_t>(stream)>>>(dirs_dev, rgb_dev, n);
  return launch_status();
}

extern "C" GG_API int gg_check_spatial_dir(const double* vel_dev, double* dirs_dev, uint64_t n,
                                           void* stream) {
  if (n == 0) return GG_OK;
  if (!vel_dev || !dirs_dev) return GG_ERR_INVALID_ARG;
  const uint64_t blocks = (n + 255) / 256;
  spatial_dir_kernel<<<(unsigned)(blocks < 4096 ? blocks : 4096), 256, 0,
                       static_cast<cudaStream_t>(stream)>>>(vel_dev, dirs_dev, n);
  return launch_status();
}

extern "C" GG_API int gg_check_kerr_vjp(const double* in_dev, double* out_dev, uint64_t n,
                                        int form, void* stream) {
  if (n == 0) return GG_OK;
  if (!in_dev || !out_dev || (form != 0 && form != 1)) return GG_ERR_INVALID_ARG;
  const uint64_t blocks = (n + 127) / 128;
  kerr_vjp_kernel<<<(unsigned)(blocks < 4096 ? blocks : 4096), 128, 0,
                    static_cast<cudaStream_t>(stream)>>>(in_dev, out_dev, n, form);
  return launch_status();
}

extern "C" GG_API int gg_check_step_factor(const double* s2_dev, double* out_dev, uint64_t n,
                                           void* stream) {
  if (n == 0) return GG_OK;
  if (!s2_dev || !out_dev) return GG_ERR_INVALID_ARG;
  const uint64_t blocks = (n + 255) / 256;
  step_factor_kernel<<<(unsigned)(blocks < 4096 ? blocks : 4096), 256, 0,
                       static_cast<cudaStream_t>(stream)>>>(s2_dev, out_dev, n);
  return launch_status();
}

extern "C" GG_API int gg_check_rcp(const float* x_dev, float* out_dev, uint64_t n, void* stream) {
  if (n == 0) return GG_OK;
  if (!x_dev || !out_dev) return GG_ERR_INVALID_ARG;
  const uint64_t blocks = (n + 255) / 256;
  rcp_kernel<<<(unsigned)(blocks < 4096 ? blocks : 4096), 256, 0,
               static_cast<cudaStream_t>(stream)>>>(x_dev, out_dev, n);
  return launch_status();
}

extern "C" GG_API int gg_check_backward_windows(const uint32_t* counts, uint32_t n_keys,
                                                uint64_t most, uint64_t* windows, uint64_t cap,
                                                uint64_t* n) {
  if (!counts || !n_keys || !most || !windows || !n) return GG_ERR_INVALID_ARG;
  std::vector<uint64_t> next;
  std::vector<char> bins;
  try {
    next.resize(n_keys);
    bins.resize(gg::backward_bins_bytes(n_keys));
  } catch (const std::bad_alloc&) {
    return GG_ERR_OOM;
  }
  const gg::BackwardPlan plan = gg::backward_plan(counts, n_keys, next.data(), bins.data());
  *n = 0;
  for (uint64_t e = 0; e < plan.entries && *n < cap; ++*n) {
    const gg::BackwardWindow w = gg::backward_window(bins.data(), plan, e, most);
    const uint64_t row[6] = {w.e0, w.e1, w.g0, w.g1, w.p0, w.p1};
    std::copy(row, row + 6, windows + 6 * *n);
    if (w.e1 <= e) return GG_ERR_CUDA;  // no progress
    e = w.e1;
  }
  return GG_OK;
}

extern "C" GG_API int gg_check_steps(const gg_metric_t* metric, const gg_camera_t* camera,
                                     const gg_integrator_t* integ, uint32_t width,
                                     uint32_t height, int form, int steady, uint32_t attempts,
                                     double* state_dev, uint32_t* counts_dev, void* stream) {
  if (!state_dev || !counts_dev || form < 0 || form > 2 || attempts > (1u << 16))
    return GG_ERR_INVALID_ARG;
  gg_render_opts_t opts;
  gg_render_opts_default(&opts);
  const int v = gg::validate_render(metric, camera, nullptr, integ, &opts, width, height);
  if (v != GG_OK) return v;
  if ((uint64_t)width * height > (1u << 20)) return GG_ERR_INVALID_ARG;
  gg::DevParams P;
  gg::make_params(metric, camera, nullptr, integ, &opts, width, height, &P);
  const cudaStream_t s = static_cast<cudaStream_t>(stream);
  if (P.metric == gg::kMetricKerr)
    launch_steps_form<gg::kMetricKerr>(form, P, steady != 0, attempts, state_dev, counts_dev, s);
  else
    launch_steps_form<gg::kMetricSchwarzschild>(form, P, steady != 0, attempts, state_dev,
                                                counts_dev, s);
  return launch_status();
}

extern "C" GG_API int gg_check_trace_form(const gg_metric_t* metric, const gg_camera_t* camera,
                                          const gg_disk_t* disk, const gg_integrator_t* integ,
                                          const gg_render_opts_t* opts, uint32_t width,
                                          uint32_t height) {
  const int v = gg::validate_render(metric, camera, disk, integ, opts, width, height);
  if (v != GG_OK) return v;
  if (integ->precision != GG_PREC_FP64) return GG_ERR_UNSUPPORTED;
  gg::DevParams P;
  gg::make_params(metric, camera, disk, integ, opts, width, height, &P);
  return gg::trace_form(P);
}

// gg_trace.cu -- persistent ray-tracing kernels for sm_100a.
//
// Work decomposition.  A render is a flat queue of n = width*height*spp
// samples.  The grid is persistent (a few CTAs per SM, sized from the
// occupancy of the instantiation); each warp takes 32 sample indices from a
// global counter at a time and hands them to its lanes as they free up.
// After every `kPeriod` RK45 attempts the warp ballots which lanes finished
// and refills exactly those lanes, so a warp keeps all 32 lanes busy even
// though per-ray attempt counts differ by 100x between a ray that escapes
// directly and one that grazes the photon sphere.  Ray state stays in
// registers from the camera to the terminal surface; HBM only sees the
// finished outcome (and, for supersampling, one linear colour per sample).
#include <cuda_runtime.h>

#include <cstdint>

#include "gg_device.cuh"
#include "gg_launch.h"
#include "gg_scene.cuh"
#include "gg_trace_common.cuh"

namespace gg {

namespace {

// A ray in the FP64 pass of the mixed form goes back to the FP32 stepper
// once an accepted step leaves it this far outside the band: r beyond
// band_r + kBackMargin M and theta more than kBackPole * pole_band from
// both poles (the margin keeps rays from bouncing between the passes).
// Measured on the 1080p Kerr frame (median ms; the endpoint error and class
// agreement identical throughout): margin / pole factor 0.5 / 1.5: 27.8,
// 1 / 2: 27.6, 1 / 3: 27.7, 2 / 2: 27.1, 2 / 3: 27.2, 3 / 4: 27.4,
// 5 / 6: 27.3, 8 / 8: 27.9.  With 2 M no ray re-enters the band.
#ifndef GG_BACK_MARGIN
#define GG_BACK_MARGIN 2.0
#endif
#ifndef GG_BACK_POLE
#define GG_BACK_POLE 2.0
#endif
constexpr double kBackMargin = GG_BACK_MARGIN;
constexpr double kBackPole = GG_BACK_POLE;

// Writes a ray clear of the band to the return queue (out of line, once per
// returned ray).
__device__ __noinline__ void hand_back(const DevOutputs& O, DevControl* ctl, Ray R, uint64_t idx,
                                       uint32_t n_att, uint32_t n_acc, uint32_t scene) {
  const unsigned long long slot = atomicAdd(&ctl->returned, 1ull);
  if (slot >= O.ret_cap) {
    atomicExch(&ctl->queue_overflow, 1u);
    return;
  }
  QueuedRay& q = O.ret[slot];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    q.x[i] = R.x[i];
    q.v[i] = R.v[i];
  }
  q.h = R.h;
  q.lam = R.lam;
  q.idx = idx;
  q.n_att = n_att;
  q.n_acc = n_acc;
  q.scene = scene;
}

// Writes a ray to the group pass's queue; false (the ray stays) if it is full.
// Out of line: at most kHandLanes times per warp.
__device__ __noinline__ bool hand_to_group(const DevOutputs& O, DevControl* ctl,
                                           const ChainRay& q) {
  const unsigned long long slot = atomicAdd(&ctl->chained, 1ull);
  if (slot >= O.chain_cap) return false;
  O.chain[slot] = q;
  return true;
}

constexpr int kPendSky = 0x100;  // see `pend`

// How many rays a launch is for, which sets its register budget: many (a full
// wave of lanes several times over), few per lane, or so few that one ray's
// chain is the time -- then its stages are unrolled.
enum : int { kSizeLarge = 0, kSizeSmall = 1, kSizeChain = 2 };

// Band passes of at most this many rays take the unrolled form: about a ray a
// lane.  Rolled / unrolled, mixed form, ms (band rays): 321x181 3.43 / 2.94 (1,700),
// 500x320 4.70 / 4.18, 1100x800 12.7 / 12.2 (25,000), 1080p 24.0 / 23.7 (59,000), the near
// view at 500^2 6.07 / 5.48 (27,000), 900^2 8.36 / 8.54 (86,000), 2048^2 x 4 83.1 / 86.9.
constexpr unsigned long long kBandChainRays = 1ull << 16;

// SRC: kSrcCamera traces the render's samples from the camera; kSrcQueue
// finishes, in FP64, the rays the mixed-precision pass handed over (their
// count is read from ctl->queued, which that pass wrote before this launch);
// with P.hand_back it returns rays that leave the band to the mixed form.
// BATCH (kSrcQueue only): the rays come from a batched render; each carries
// its scene, whose parameters and outputs are in B.  SCENE (kSrcCamera, no
// thin disk): every accepted step's chord is tested against P's scene of
// objects first.  CKPT (kSrcCamera, Kerr, thin disk, full Dormand-Prince):
// the differentiable render's forward, which also stores each ray's state
// (x, v, next h) at its start and after every kCkptEvery-th accepted step it
// survives (O.ckpt) and, when it ends, its DiffRay (O.diff_rays).  GROUP
// (kSrcCamera, the reference's step): kGroupLanes lanes share a ray
// (attempt_fp64_group); the rays come from the group queue if there is one
// (O.chain), else from the camera.  Without GROUP, a warp that finds no more
// samples and has at most kHandLanes rays left hands those to that queue.
template <int METRIC, int DISK, int STEPPER, int SRC, bool BATCH, bool SCENE, bool CKPT,
          int SIZE, bool GROUP>
__global__ void __launch_bounds__(kTraceBlock,
                                  GROUP || SIZE == kSizeChain ? kTraceMinBlocksGroup
                                  : METRIC != kMetricKerr     ? kTraceMinBlocksSchw
                                  : (SRC == kSrcQueue || CKPT || SIZE == kSizeSmall)
                                      ? kTraceMinBlocksKerrChain
                                      : kTraceMinBlocksKerr)
    trace_fp64_kernel(const __grid_constant__ DevParams P, const __grid_constant__ DevOutputs O,
                      DevControl* ctl, const __grid_constant__ BatchTable B) {
  if (SRC == kSrcQueue && (ctl->queued <= kBandChainRays) != (SIZE == kSizeChain)) return;
  const unsigned lane = threadIdx.x & 31u;
  const bool from_chain = GROUP && O.chain != nullptr;
  const uint64_t n_src =
      SRC == kSrcQueue ? (ctl->queued < O.queue_cap ? ctl->queued : O.queue_cap)
      : from_chain     ? (ctl->chained < O.chain_cap ? ctl->chained : O.chain_cap)
                       : P.n_rays;
  unsigned long long* const head = SRC == kSrcQueue ? &ctl->next_queued
                                   : from_chain     ? &ctl->next_chained
                                                    : &ctl->next_ray;
  // lanes that stand for a ray in the votes (one per group), and whether this
  // one writes its ray's results
  const unsigned ray_lanes = GROUP ? kGroupLeaders : kFull;
  const bool writer = !GROUP || lane % kGroupLanes == 0;
  constexpr uint32_t chunk = GROUP ? 32 / kGroupLanes : kChunk;
  __shared__ BlockStats bs;
  __shared__ double2 k_smem[GROUP ? 1 : 7][2][kTraceBlock];  // stage derivatives, see KStore
  const KStore K{k_smem};
  // SCENE: the Cartesian image of the current position, if cart_valid
  __shared__ double cart_smem[SCENE ? 3 : 1][kTraceBlock];
  bool cart_valid = false;
  GroupRole role;
  double k1[4];  // GROUP: a(x, v) of the current state if k1_valid
  if (GROUP) role = GroupRole::at(lane);
  if (threadIdx.x < sizeof(BlockStats) / 8)
    reinterpret_cast<unsigned long long*>(&bs)[threadIdx.x] = 0ull;
  __syncthreads();
  uint32_t n_att0 = 0;  // kSrcQueue: attempts the ray had made before the hand-off

  Ray R;
  uint64_t idx = 0;
  uint32_t scene = 0;  // BATCH: the ray's scene
  bool live = false;
  uint32_t n_att = 0, n_acc = 0;
  double inten = 0.0, trans = 1.0;  // volumetric disk accumulators
  bool crossed = false;
  bool k1_valid = false;    // K(0, .) holds a(x, v) of the current state
  bool k7_pending = false;  // full DP: K(6, .) is the next k1, copy pending
  // A ray that ends is finished at the next refill, by every lane of the warp that
  // has one: its redshift, shading and encoding are nine pow() and as many
  // divisions, more than an attempt, and ran a lane at a time where the ray ended.
  // The class, with kPendSky if (inten, trans) hold where the sky is read.
  // Measured before / after, ms: Schwarzschild disk at 800x600 12.1 / 10.9, near view
  // at 1024^2 9.9 / 9.0, 256^2 thin disk 1.63 / 1.52, 1080p full Dormand-Prince 42.2 /
  // 40.2, the 512^2 forward 7.3 / 6.9, the 1080p drop-in frame 35.1 / 35.0.
  int pend = -1;
  uint32_t n_ckpt = 0;      // CKPT: checkpoints of the ray so far
  auto save_ckpt = [&]() {
    if (n_ckpt < O.ckpt_per_ray) {
      Ckpt& c = O.ckpt[idx * O.ckpt_per_ray + n_ckpt];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        c.x[i] = R.x[i];
        c.v[i] = R.v[i];
      }
      c.h = R.h;
    }
    ++n_ckpt;
  };

  uint64_t wbase = 0;
  uint32_t wcount = 0;
  bool wdone = false;
  unsigned budget_pending = 0;
  constexpr bool kHandsOver =
      STEPPER == kStepperReference && SRC == kSrcCamera && !GROUP && !CKPT && !BATCH;

  for (;;) {
    // ---- finish the rays that ended ---------------------------------------
    if (pend >= 0) {
      const DevParams& PL = BATCH ? B.scenes[scene].P : P;
      const DevOutputs& OL = BATCH ? B.scenes[scene].O : O;
      const int cls = pend & ~kPendSky;
      if (writer) {
        if (SCENE && cls == kClsScene) {
          const double rgb[3] = {cart_smem[0][threadIdx.x], cart_smem[SCENE ? 1 : 0][threadIdx.x],
                                 cart_smem[SCENE ? 2 : 0][threadIdx.x]};
          finish_scene_sample(PL, OL, idx, R, n_att, n_acc, inten, rgb);
        } else {
          double out_int = 0.0, out_temp = 0.0, sky_th = R.x[2], sky_ph = R.x[3];
          if (pend & kPendSky) {
            sky_th = inten;
            sky_ph = trans;
          }
          if (DISK == kDiskThin && cls == kClsDisk) {
            const double g = redshift_factor<METRIC>(PL, R.x[1], kHalfPi, R.v);
            const double q = PL.r_inner / R.x[1];
            const double g2 = g * g;
            out_int = (g2 * g2) * pow(q, PL.emissivity_index);
            out_temp = g * pow(q, 0.75);
          } else if (cls == kClsDisk) {
            out_int = inten;
            out_temp = PL.temperature_0;
          }
          finish_sample(PL, OL, idx, cls, R, n_att, n_acc, out_int, out_temp, crossed, sky_th,
                        sky_ph);
        }
        atomicAdd(&bs.attempts, (unsigned long long)n_att);
        atomicAdd(&bs.accepted, (unsigned long long)n_acc);
        atomicAdd(&bs.cls[cls], 1ull);
        if (SRC == kSrcQueue) atomicAdd(&bs.fp64_att, (unsigned long long)(n_att - n_att0));
      }
      if (CKPT) O.diff_rays[idx] = DiffRay{n_acc, n_ckpt, cls, 0u};
      pend = -1;
    }

    // ---- refill lanes whose ray finished ----------------------------------
    unsigned need = __ballot_sync(kFull, !live);
    if (P.attempt_budget && need && !wdone) {
      unsigned long long ab = 0;
      if (lane == 0) ab = atomicOr(&ctl->abort, 0u);
      if (__shfl_sync(kFull, ab, 0)) wdone = true;
    }
    while (need && !wdone) {
      if (wcount == 0) {
        unsigned long long b = 0;
        if (lane == 0) {
          b = atomicAdd(head, (unsigned long long)chunk);
          if (P.attempt_budget) {
            const unsigned long long used = atomicAdd(&ctl->budget_used, 0ull);
            if (used > P.attempt_budget) {
              atomicExch(&ctl->abort, 1u);
              b = n_src;  // stop taking work
            }
          }
        }
        b = __shfl_sync(kFull, b, 0);
        if (b >= n_src) {
          wdone = true;
          break;
        }
        wbase = b;
        const uint64_t left = n_src - b;
        wcount = left < chunk ? (uint32_t)left : chunk;
      }
      const unsigned nn = (unsigned)__popc(need & ray_lanes);
      const unsigned take = nn < wcount ? nn : wcount;
      const unsigned below =
          GROUP ? (1u << (lane & ~(unsigned)(kGroupLanes - 1))) - 1u : lanemask_lt();
      const unsigned rank = (unsigned)__popc(need & ray_lanes & below);
      if (!live && rank < take) {
        inten = 0.0;
        trans = 1.0;
        crossed = false;
        k1_valid = false;
        k7_pending = false;
        cart_valid = false;
        if (from_chain) {
          const ChainRay& q = O.chain[wbase + rank];
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            R.x[i] = q.x[i];
            R.v[i] = q.v[i];
            k1[i] = q.k1[i];
          }
          R.h = q.h;
          R.lam = q.lam;
          inten = q.inten;
          trans = q.trans;
          idx = q.idx;
          n_att = q.n_att;
          n_acc = q.n_acc;
          k1_valid = q.k1_valid != 0u;
          crossed = q.crossed != 0u;
        } else if (SRC == kSrcQueue) {
          const QueuedRay& q = O.queue[wbase + rank];
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            R.x[i] = q.x[i];
            R.v[i] = q.v[i];
          }
          R.h = q.h;
          R.lam = q.lam;
          idx = q.idx;
          if (BATCH) scene = q.scene;
          n_att = n_att0 = q.n_att;
          n_acc = q.n_acc;
        } else {
          idx = camera_sample(P, wbase + rank);
          R = start_sample(P, idx);
          n_att = 0;
          n_acc = 0;
          if (CKPT) {
            n_ckpt = 0;
            save_ckpt();
          }
        }
        live = true;
      }
      wbase += take;
      wcount -= take;
      need = __ballot_sync(kFull, !live);
    }
    if (kHandsOver && wdone && O.chain) {
      const unsigned left = 32u - (unsigned)__popc(need);
      if (live && left <= kHandLanes) {
        ChainRay q;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          q.x[i] = R.x[i];
          q.v[i] = R.v[i];
          q.k1[i] = K(0, i);
        }
        q.h = R.h;
        q.lam = R.lam;
        q.inten = inten;
        q.trans = trans;
        q.idx = idx;
        q.n_att = n_att;
        q.n_acc = n_acc;
        q.k1_valid = k1_valid ? 1u : 0u;
        q.crossed = crossed ? 1u : 0u;
        if (hand_to_group(O, ctl, q)) live = false;
      }
    }
    if (!__any_sync(kFull, live)) break;

    // ---- advance every live ray by up to kPeriod attempts -----------------
#pragma unroll 1
    for (int it = 0; it < (SRC == kSrcQueue ? kQueuePeriod : GROUP ? kGroupPeriod : kPeriod);
         ++it) {
      if (!live) continue;
      // this lane's scene: the batch's entry, or the render's own parameters
      const DevParams& PL = BATCH ? B.scenes[scene].P : P;
      const DevOutputs& OL = BATCH ? B.scenes[scene].O : O;
      double xb[4], vb[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        xb[i] = R.x[i];
        vb[i] = R.v[i];
      }
      const double lam_b = R.lam;
      bool acc;
      double h_used = 0.0;
      StepEnd end;
      int res;
      if (STEPPER == kStepperDP45)
        res = attempt_dp45_fp64<METRIC, SIZE == kSizeChain    ? kStageUnrolled
                                        : SRC == kSrcQueue ? kStageLooped
                                                           : kStageArms>(
            PL, R, K, k1_valid, k7_pending, acc, h_used, end);
      else if (GROUP)
        res = attempt_fp64_group<METRIC>(PL, R, role, k1, k1_valid, acc, h_used);
      else
        res = attempt_fp64<METRIC, SIZE == kSizeChain>(PL, R, K, k1_valid, acc, h_used);
      n_att += 1;
      if (acc) n_acc += 1;
      int done_cls = -1;
      // full Dormand-Prince, checkerboard sky, thin disk or none: the sky is
      // read where the ray meets the escape sphere (sky_at_cross)
      constexpr bool kSkyCross = STEPPER == kStepperDP45 && DISK != kDiskVolumetric;
      bool sky_at_cross = false;
      double sky_th = 0.0, sky_ph = 0.0;
      double scene_rgb[3];

      if (SCENE && acc) {
        // trace_ray_with_scene (tracer.rs:218-236): the chord between the
        // step's ends, in Cartesian coordinates, against the scene
        double cb[3], ca[3], dd[3];
        if (cart_valid) {  // the last step's end
#pragma unroll
          for (int i = 0; i < 3; ++i) cb[i] = cart_smem[i][threadIdx.x];
        } else {
          sph_to_cart(xb, cb);
        }
        sph_to_cart(R.x, ca);
#pragma unroll
        for (int i = 0; i < 3; ++i) cart_smem[i][threadIdx.x] = ca[i];
        cart_valid = true;
#pragma unroll
        for (int i = 0; i < 3; ++i) dd[i] = sub_rn(ca[i], cb[i]);
        if (near_scene(PL, cb, ca) && dot3_nc(dd, dd) > 0.0) {
          double t_hit;
          const int k = scene_nearest(PL, cb, dd, t_hit);
          if (k >= 0) {
            scene_shade<METRIC>(PL, k, t_hit, cb, dd, scene_rgb);
            if (DISK == kDiskVolumetric) {  // tracer.rs:293-309
              double dl[3];
              disk_color(inten, dl);
#pragma unroll
              for (int c = 0; c < 3; ++c) scene_rgb[c] = add_rn(mul_rn(scene_rgb[c], trans), dl[c]);
            }
            done_cls = kClsScene;
          }
        }
      }

      if (acc && done_cls < 0) {
        // The step's path: the reference's Euler segment (exactly linear in
        // the step fraction), or the full Dormand-Prince step's continuous
        // extension.
        double raw[4];
#pragma unroll
        for (int i = 0; i < 4; ++i)
          raw[i] = STEPPER == kStepperDP45 ? end.xraw[i] : xb[i] + h_used * vb[i];
        const bool esc = (OL.cross || (kSkyCross && PL.sky == kSkyChecker)) &&
                         xb[1] <= PL.max_radius && raw[1] > PL.max_radius;
        double d_b = 0.0, d_a = 0.0;
        bool dsk = false;
        if (DISK == kDiskThin) {
          d_b = xb[2] - kHalfPi;
          d_a = R.x[2] - kHalfPi;
          dsk = (d_b < 0.0 && d_a >= 0.0) || (d_b > 0.0 && d_a <= 0.0);
        }
        if (esc || dsk) {
          StepSpan sp;
          if (STEPPER == kStepperDP45) {
#pragma unroll
            for (int i = 0; i < 4; ++i) {
              sp.xb[i] = xb[i];
              sp.vb[i] = vb[i];
              sp.xa[i] = raw[i];
              sp.va[i] = R.v[i];
            }
            for (int l = 0; l < 7; ++l)
#pragma unroll
              for (int i = 0; i < 4; ++i) sp.k[l][i] = K(l, i);
            sp.h = h_used;
          }
          // state c where component `comp` meets `target`; returns the step
          // fraction (the reference stepper's is linear_s, on its segment)
          auto cross_at = [&](int comp, double target, double linear_s, double c[8]) {
            if (STEPPER == kStepperDP45) {
              const double s = dense_crossing(sp, comp, target, c);
              normalize_coords(c);
              return s;
            }
            segment_point(xb, vb, h_used, R.v, linear_s, c);
            return linear_s;
          };
          if (esc) {
            double c[8];
            cross_at(1, PL.max_radius, (PL.max_radius - xb[1]) / (raw[1] - xb[1]), c);
            if (OL.cross) {
              if (writer) store_cross(PL, OL, idx, c);
              crossed = true;
            }
            if (kSkyCross && PL.sky == kSkyChecker) {
              sky_at_cross = true;
              sky_th = c[2];
              sky_ph = c[3];
            }
          }
          if (dsk) {
            double c[8];
            const double s = cross_at(2, kHalfPi, d_b / (d_b - d_a), c);
            const double r_c =
                STEPPER == kStepperDP45 ? c[1] : xb[1] + s * (raw[1] - xb[1]);
            if (r_c >= PL.r_inner && r_c <= PL.r_outer) {
              c[1] = r_c;
              c[2] = kHalfPi;
#pragma unroll
              for (int i = 0; i < 4; ++i) {
                R.x[i] = c[i];
                R.v[i] = c[4 + i];
              }
              R.lam = lam_b + s * h_used;
              if (writer) store_cross(PL, OL, idx, c);
              crossed = true;
              done_cls = kClsDisk;
            }
          }
        }
        // Beyond the escape sphere the next attempt only finds r > max_radius
        // and returns Escaped; the ray ends here, counting that attempt.
        if (sky_at_cross && done_cls < 0 && n_att < PL.max_steps) {
          n_att += 1;
          done_cls = kClsEscaped;
        }
      }
      if (DISK == kDiskVolumetric && done_cls < 0) {
        // trace_ray_with_disk (tracer.rs:96-145)
        const double dlambda = fmax(R.lam - lam_b, 0.0);
        double mid[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) mid[i] = 0.5 * (xb[i] + R.x[i]);
        // Inside r_inner the distance from the axis is too, and beyond r_clear
        // either it is past r_outer or the density underflows to 0: most steps of
        // a picture need no sine here.  With this, the sine and cosine shared
        // with the redshift and (SCENE) each position's Cartesian image kept
        // for the next step: the command line's disk at 800x600 12.7 -> 12.1 ms,
        // the lensed spheres with the disk 26.3 -> 23.0.
        if (dlambda > 0.0 && mid[1] >= PL.r_inner && mid[1] <= PL.r_clear) {
          double sn, cs;
          sincos(mid[2], &sn, &cs);
          const double cap_r = mid[1] * fabs(sn);
          const double z = mid[1] * cs;
          if (!(cap_r < PL.r_inner || cap_r > PL.r_outer)) {
            const double qq = PL.r_inner / cap_r;
            const double rho = PL.density_0 * (qq * qq) *
                               exp(-z * z / (2.0 * PL.scale_height * PL.scale_height));
            if (rho > 0.0) {
              const double j = rho * rho * pow(qq, 0.75);
              double pm[4];
#pragma unroll
              for (int i = 0; i < 4; ++i) pm[i] = 0.5 * (vb[i] + R.v[i]);
              const double g = redshift_factor<METRIC>(PL, mid[1], sn, cs, pm);
              const double g2 = g * g;
              inten = inten + j * (g2 * g2) * dlambda * trans;
              trans = trans * exp(-rho * dlambda * 0.1);
              if (trans < 1e-3) {
                done_cls = kClsDisk;
              }
            }
          }
        }
        if (done_cls < 0 && res != kContinue) {
          done_cls = inten > 0.0 ? kClsDisk : res == kEscaped ? kClsEscaped : kClsHorizon;
        }
        if (done_cls < 0 && n_att >= PL.max_steps) {
          done_cls = inten > 0.0 ? kClsDisk : kClsMaxSteps;
        }
      } else if (done_cls < 0) {
        if (res == kHorizon) done_cls = kClsHorizon;
        else if (res == kEscaped) done_cls = kClsEscaped;
        else if (n_att >= PL.max_steps) done_cls = kClsMaxSteps;
      }
      // a checkpoint after every kCkptEvery-th accepted step that did not end
      // the ray at a crossing (a step that runs out of attempts still counts)
      if (CKPT && acc && (done_cls < 0 || done_cls == kClsMaxSteps) &&
          n_acc % kCkptEvery == 0)
        save_ckpt();
      if (SRC == kSrcQueue && P.hand_back && acc && done_cls < 0 &&
          R.x[1] > (double)PL.band_r + kBackMargin &&
          fmin(R.x[2], kPi - R.x[2]) > kBackPole * (double)PL.pole_band) {
        hand_back(O, ctl, R, idx, n_att, n_acc, scene);
        atomicAdd(&bs.fp64_att, (unsigned long long)(n_att - n_att0));
        live = false;
        continue;
      }
      if (done_cls >= 0) {
        pend = done_cls;
        if (SCENE && done_cls == kClsScene) {
#pragma unroll
          for (int c = 0; c < 3; ++c) cart_smem[c][threadIdx.x] = scene_rgb[c];
        }
        if (sky_at_cross && done_cls == kClsEscaped) {
          pend |= kPendSky;
          inten = sky_th;
          trans = sky_ph;
        }
        budget_pending += n_att;
        live = false;
      }
    }
    if (P.attempt_budget) {
      // account finished work; stop live rays once the budget is gone
      const unsigned long long wsum = __reduce_add_sync(kFull, budget_pending);
      budget_pending = 0;
      unsigned ab = 0;
      if (lane == 0) {
        const unsigned long long used = atomicAdd(&ctl->budget_used, wsum) + wsum;
        if (used > P.attempt_budget) atomicExch(&ctl->abort, 1u);
        ab = atomicOr(&ctl->abort, 0u);
      }
      if (__shfl_sync(kFull, ab, 0)) {
        wdone = true;
        if (live) {
          pend = kClsBudget;
          live = false;
        }
      }
    }
  }

  // ---- per-block statistics -----------------------------------------------
  __syncthreads();
  if (threadIdx.x == 0) {
    atomicAdd(&ctl->attempts, bs.attempts);
    atomicAdd(&ctl->accepted, bs.accepted);
    if (SRC == kSrcQueue && bs.fp64_att) atomicAdd(&ctl->fp64_attempts, bs.fp64_att);
#pragma unroll
    for (int k = 0; k < kNumClasses; ++k)
      if (bs.cls[k]) atomicAdd(&ctl->class_count[k], bs.cls[k]);
  }
}

// Averages the spp linear sample colours of each pixel in sample order and
// encodes sRGB (render_row, renderer.rs:326-343).
__global__ void reduce_samples_kernel(const __grid_constant__ DevParams P, const double* samples,
                                      uint8_t* rgb8) {
  const uint64_t n_pix = (uint64_t)P.width * P.rows;
  for (uint64_t p = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; p < n_pix;
       p += (uint64_t)gridDim.x * blockDim.x) {
    double acc[3] = {0.0, 0.0, 0.0};
    const double* s = samples + 3 * p * P.spp;
    for (uint32_t k = 0; k < P.spp; ++k) {
#pragma unroll
      for (int c = 0; c < 3; ++c) acc[c] = add_rn(acc[c], s[3 * k + c]);
    }
#pragma unroll
    for (int c = 0; c < 3; ++c) rgb8[3 * p + c] = encode_channel(mul_rn(acc[c], P.inv_spp));
  }
}

template <int METRIC, int DISK, int STEPPER, int SRC, bool BATCH = false, bool SCENE = false,
          bool CKPT = false, int SIZE = kSizeLarge, bool GROUP = false>
const void* trace_fn() {
  return reinterpret_cast<const void*>(
      &trace_fp64_kernel<METRIC, DISK, STEPPER, SRC, BATCH, SCENE, CKPT, SIZE, GROUP>);
}

template <int METRIC, int DISK, bool SCENE = false>
const void* group_fn() {
  return trace_fn<METRIC, DISK, kStepperReference, kSrcCamera, false, SCENE, false, kSizeLarge,
                  true>();
}

// The group kernel of a render with the reference's step.
template <int METRIC>
const void* select_group_metric(const DevParams& P) {
  if (P.scene)
    return P.disk == kDiskVolumetric ? group_fn<METRIC, kDiskVolumetric, true>()
                                     : group_fn<METRIC, kDiskNone, true>();
  return P.disk == kDiskThin         ? group_fn<METRIC, kDiskThin>()
         : P.disk == kDiskVolumetric ? group_fn<METRIC, kDiskVolumetric>()
                                     : group_fn<METRIC, kDiskNone>();
}

const void* select_group(const DevParams& P) {
  return P.metric == kMetricKerr ? select_group_metric<kMetricKerr>(P)
                                 : select_group_metric<kMetricSchwarzschild>(P);
}

// Renders of so few samples are traced by the group kernel from the camera:
// there each lane of the other kernels has at most one ray, and the time is one ray's
// chain.  The group kernel has 7,104 rays in flight, and its work per attempt is
// larger, so the line lies a little above that; with the thin disk, whose rays
// end early and unevenly, at twice as many.  Lane per ray (unrolled) / group, ms, at 64^2,
// 90^2, 100^2, 128^2 (a view from 30 M, on the equator or, with the thin disk, at 80 deg):
// Schwarzschild, no disk 0.85 / 0.76, 1.49 / 1.27, 1.09 / 1.23, 1.47 / 1.60; thin disk 0.85 / 0.65,
// 1.06 / 0.80, 1.03 / 0.82, 1.04 / 1.00 (140^2: 1.10 / 1.14); volumetric disk 1.14 / 0.97, 1.92 / 1.60,
// 1.38 / 1.60, 1.82 / 2.13; that with objects 1.45 / 1.20, 1.91 / 1.70, 1.73 / 1.97, 1.81 / 2.82.
// Kerr, no disk 1.55 / 1.40, 3.77 / 3.45, 1.52 / 1.55, 1.68 / 2.05; thin disk 1.49 / 0.82, 1.48 / 1.05,
// 1.40 / 1.10, 1.75 / 1.40 (160^2: 1.82 / 1.85); volumetric disk 2.06 / 1.78, 4.65 / 4.19, 2.02 / 2.18,
// 2.13 / 2.85; that with objects 2.48 / 2.13, 5.58 / 5.03, 2.39 / 2.70, 2.60 / 3.80.
// Where no group pass follows a lane's last rays (gg_noalloc.cu), a near-critical ray
// costs the other kernels twice as much, and the line stays at 2^14: 100^2, 110^2, 120^2,
// Kerr without a disk 1.56 / 1.58, 5.5 / 4.1, 1.96 / 1.91.
constexpr uint64_t kGroupRays = 1ull << 13, kGroupRaysFar = 1ull << 14;
bool group_render(const DevParams& P) {
  const bool far = P.disk == kDiskThin || P.no_group_pass;
  return P.stepper == kStepperReference && !P.attempt_budget &&
         P.n_rays <= (far ? kGroupRaysFar : kGroupRays);
}

// Kerr camera passes of fewer samples than this run the 4-CTA budget of the
// chain-bound passes: a few rays per lane, so the longest rays set the time.
constexpr uint64_t kSmallRender = 1ull << 20;

// With a scene: no disk or the volumetric one (the reference's
// render_with_scene and render_with_disk_and_scene).
template <int METRIC, int STEPPER, int SIZE>
const void* select_disk(const DevParams& P) {
  if (P.scene)
    return P.disk == kDiskVolumetric
               ? trace_fn<METRIC, kDiskVolumetric, STEPPER, kSrcCamera, false, true, false, SIZE>()
               : trace_fn<METRIC, kDiskNone, STEPPER, kSrcCamera, false, true, false, SIZE>();
  if (P.disk == kDiskThin)
    return trace_fn<METRIC, kDiskThin, STEPPER, kSrcCamera, false, false, false, SIZE>();
  if (P.disk == kDiskVolumetric)
    return trace_fn<METRIC, kDiskVolumetric, STEPPER, kSrcCamera, false, false, false, SIZE>();
  return trace_fn<METRIC, kDiskNone, STEPPER, kSrcCamera, false, false, false, SIZE>();
}

template <int STEPPER, int SIZE>
const void* select_metric(const DevParams& P) {
  return P.metric == kMetricKerr ? select_disk<kMetricKerr, STEPPER, SIZE>(P)
                                 : select_disk<kMetricSchwarzschild, STEPPER, SIZE>(P);
}

// Full Dormand-Prince camera passes of at most this many samples take the
// unrolled form.  Rolled / unrolled, ms, the differentiable forward: 64^2 1.83 /
// 1.52, 128^2 2.84 / 2.32, 160^2 2.26 / 1.98, 200^2 2.53 / 2.34, 230^2 2.90 /
// 2.65, 256^2 3.16 / 3.39, 512^2 7.2 / 8.5; with objects 200^2, Kerr 2.57 / 2.13,
// Schwarzschild 1.88 / 1.45, and the volumetric disk 3.13 / 2.80 and 2.32 / 1.96, which
// with objects turns at 260^2 (Kerr 4.95 / 4.57, Schwarzschild 2.68 / 2.93).
constexpr uint64_t kChainRays = 3ull << 14;
// The reference's step: up to 2^18, 2^17 with the volumetric disk, whose work at
// every step wants more warps.  One line for both metrics, where the slower one, Kerr,
// has it.  Rolled / unrolled, ms: Kerr with a thin disk at 200^2 2.43 / 2.01, 400^2
// 3.97 / 3.57, 512^2 4.29 / 4.22, 600^2 5.56 / 5.66, 700^2 6.9 / 7.4; volumetric disk 200^2 4.30 /
// 3.86, 340^2 9.77 / 9.33, 362^2 11.9 / 11.8, 450^2 13.0 / 13.6; no disk 512^2 12.0 / 11.6;
// Schwarzschild with a thin disk 512^2 3.43 / 2.91, 700^2 5.27 / 4.67, volumetric 362^2 5.16 /
// 4.86, 600^2 9.3 / 9.5.  With objects the lines are within 5 % either way: Kerr 340^2 9.43 /
// 9.46, 512^2 14.4 / 15.0, and the volumetric disk 256^2 11.6 / 11.9, 340^2 12.0 / 12.0, 362^2
// 14.5 / 15.3; Schwarzschild 512^2 7.3 / 7.1, and the volumetric disk 340^2 5.73 / 5.44, 362^2
// 6.86 / 6.92.
constexpr uint64_t kChainRaysReference = 1ull << 18, kChainRaysVolumetric = 1ull << 17;

uint64_t chain_rays(const DevParams& P) {
  return P.stepper == kStepperDP45         ? kChainRays
         : P.disk == kDiskVolumetric ? kChainRaysVolumetric
                                     : kChainRaysReference;
}

// The form of the trace kernel that a render takes.
enum TraceForm : int { kFormLarge, kFormSmall, kFormChain, kFormGroup };
TraceForm form_of(const DevParams& P) {
  if (group_render(P)) return kFormGroup;
  if (P.n_rays <= chain_rays(P)) return kFormChain;
  return P.metric == kMetricKerr && P.n_rays < kSmallRender ? kFormSmall : kFormLarge;
}

template <int STEPPER>
const void* select_size(const DevParams& P, TraceForm form) {
  if (form == kFormChain) return select_metric<STEPPER, kSizeChain>(P);
  if (form == kFormSmall) return select_disk<kMetricKerr, STEPPER, kSizeSmall>(P);
  return select_metric<STEPPER, kSizeLarge>(P);
}

const void* select_trace(const DevParams& P) {
  const TraceForm form = form_of(P);
  if (form == kFormGroup) return select_group(P);
  // gg_forward_ckpt admits only Kerr, the thin disk and the full stepper
  if (P.ckpt)
    return form == kFormChain
               ? trace_fn<kMetricKerr, kDiskThin, kStepperDP45, kSrcCamera, false, false, true,
                          kSizeChain>()
               : trace_fn<kMetricKerr, kDiskThin, kStepperDP45, kSrcCamera, false, false, true>();
  return P.stepper == kStepperDP45 ? select_size<kStepperDP45>(P, form)
                                   : select_size<kStepperReference>(P, form);
}

// The FP64 pass of the mixed form: full Dormand-Prince, thin disk or none.
template <int METRIC, bool BATCH, int SIZE>
const void* queue_fn(const DevParams& P) {
  return P.disk == kDiskThin
             ? trace_fn<METRIC, kDiskThin, kStepperDP45, kSrcQueue, BATCH, false, false, SIZE>()
             : trace_fn<METRIC, kDiskNone, kStepperDP45, kSrcQueue, BATCH, false, false, SIZE>();
}

template <bool BATCH, int SIZE>
const void* select_queue_metric(const DevParams& P) {
  return P.metric == kMetricKerr ? queue_fn<kMetricKerr, BATCH, SIZE>(P)
                                 : queue_fn<kMetricSchwarzschild, BATCH, SIZE>(P);
}

const void* select_queue_trace(const DevParams& P, bool batch, bool chain) {
  if (chain)
    return batch ? select_queue_metric<true, kSizeChain>(P)
                 : select_queue_metric<false, kSizeChain>(P);
  return batch ? select_queue_metric<true, kSizeLarge>(P)
               : select_queue_metric<false, kSizeLarge>(P);
}

}  // namespace

cudaError_t trace_occupancy(const DevParams& P, int* blocks_per_sm) {
  return cudaOccupancyMaxActiveBlocksPerMultiprocessor(blocks_per_sm, select_trace(P),
                                                       kTraceBlock, 0);
}

int trace_form(const DevParams& P) { return form_of(P); }

int chain_capacity(const DevParams& P, int grid) {
  if (P.stepper != kStepperReference || P.attempt_budget || P.no_group_pass || group_render(P))
    return 0;
  return grid * (kTraceBlock / 32) * (int)kHandLanes;
}

uint64_t trace_blocks(const DevParams& P) {
  const uint64_t per = group_render(P) ? kTraceBlock / kGroupLanes : kTraceBlock;
  return (P.n_rays + per - 1) / per;
}

cudaError_t launch_group(const DevParams& P, const DevOutputs& O, DevControl* ctl, int sms,
                         cudaStream_t stream) {
  const void* fn = select_group(P);
  int bps = 0;
  const cudaError_t e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&bps, fn, kTraceBlock, 0);
  if (e != cudaSuccess) return e;
  // a CTA takes 128 / kGroupLanes rays at a time
  const int most = (int)(O.chain_cap / (kTraceBlock / kGroupLanes)) + 1;
  int grid = sms * (bps > 0 ? bps : 1);
  if (grid > most) grid = most;
  DevParams p = P;
  DevOutputs o = O;
  BatchTable b{};
  void* args[] = {&p, &o, &ctl, &b};
  return cudaLaunchKernel(fn, dim3(grid), dim3(kTraceBlock), args, 0, stream);
}

cudaError_t launch_queue_trace(const DevParams& P, const DevOutputs& O, DevControl* ctl, int sms,
                               cudaStream_t stream, const BatchTable* batch) {
  DevParams p = P;
  DevOutputs o = O;
  BatchTable b{};
  if (batch) b = *batch;
  void* args[] = {&p, &o, &ctl, &b};
  // The queue's length is only known on the device: both forms are launched,
  // full persistent grids, and the one it is not for returns at once.
  for (int chain = 1; chain >= 0; --chain) {
    if (!chain && O.queue_cap <= kBandChainRays) break;
    const void* fn = select_queue_trace(P, batch != nullptr, chain != 0);
    int bps = 0;
    const cudaError_t q = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&bps, fn, kTraceBlock, 0);
    if (q != cudaSuccess) return q;
    const cudaError_t e = cudaLaunchKernel(fn, dim3(sms * (bps > 0 ? bps : 1)),
                                           dim3(kTraceBlock), args, 0, stream);
    if (e != cudaSuccess) return e;
  }
  return cudaSuccess;
}

cudaError_t launch_trace(const DevParams& P, const DevOutputs& O, DevControl* ctl, int grid,
                         cudaStream_t stream) {
  const void* fn = select_trace(P);
  DevParams p = P;
  DevOutputs o = O;
  BatchTable b{};
  void* args[] = {&p, &o, &ctl, &b};
  return cudaLaunchKernel(fn, dim3(grid), dim3(kTraceBlock), args, 0, stream);
}

// Between the rounds of the mixed form: the band queue's entries are all
// consumed; its count moves to the running total and it restarts empty.
__global__ void next_round_kernel(DevControl* ctl) {
  ctl->band_total += ctl->queued;
  ctl->queued = 0;
  ctl->next_queued = 0;
}

cudaError_t launch_next_round(DevControl* ctl, cudaStream_t stream) {
  next_round_kernel<<<1, 1, 0, stream>>>(ctl);
  return cudaGetLastError();
}

cudaError_t launch_reduce(const DevParams& P, const double* samples, uint8_t* rgb8, int sms,
                          cudaStream_t stream) {
  const uint64_t n_pix = (uint64_t)P.width * P.rows;
  uint64_t blocks = (n_pix + 255) / 256;
  const uint64_t cap = (uint64_t)sms * 8;
  if (blocks > cap) blocks = cap;
  if (blocks < 1) blocks = 1;
  reduce_samples_kernel<<<(unsigned)blocks, 256, 0, stream>>>(P, samples, rgb8);
  return cudaGetLastError();
}

}  // namespace gg

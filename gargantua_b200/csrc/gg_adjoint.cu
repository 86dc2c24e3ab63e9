// gg_adjoint.cu -- the differentiable render: the hand-written adjoint
// (reverse-mode) pass over the forward's checkpoints.
//
// Image: Kerr, thin disk, one sample per pixel, full Dormand-Prince stepper
// in FP64.  Each pixel's linear colour is a function of five parameters:
// spin a, camera inclination and distance (the inclined camera of
// gg_camera_inclined), disk inner radius r_in and emissivity index q.  Disk
// pixels carry I = g^4 (r_in / r_c)^q through the disk colour; sky and
// horizon pixels are piecewise constant in the parameters (zero gradient;
// their jumps across class or cell boundaries are not differentiated).
//
// Forward (gg_forward_ckpt): the FP64 trace kernel's checkpointing variant
// (trace_fp64_kernel<Kerr, thin disk, full Dormand-Prince, ..., CKPT> in
// gg_trace.cu), which also stores each ray's state (x, v, next h) at the start
// and after every kCkptEvery-th accepted step, and its DiffRay.
//
// Backward, over the disk rays with a nonzero dL/d(colour), in six launches:
//   1. a counting sort lists the rays by their number of segments, longest
//      first (backward_count / backward_scatter; the host makes the prefix
//      sums in between);
//   2. backward_replay_kernel: every segment of every listed ray is replayed
//      from its checkpoint, a lane each (the controller is deterministic, so a
//      replay takes the forward's steps), and leaves each step's start, size and
//      stage derivatives in a record;
//   3. backward_crossing_kernel: the crossing step (a ray's last) again in
//      forward-mode dual numbers over its start state (6) and the spin: stages,
//      continuous extension, the root s* (one Newton correction in dual
//      arithmetic gives ds*/dp by the implicit function theorem), the crossing
//      state, the redshift and I -- so dL/d(start state), dL/da, dL/dr_in,
//      dL/dq and dL/d(observer normalisation) in one pass;
//   4. backward_chain_kernel: the steps before it in reverse, each the
//      vector-Jacobian products of its stages' Kerr right-hand sides in r, theta,
//      the stage velocity and the spin, by a hand-written reverse pass
//      (gg_vjp.cuh), with theta reflections at the poles reversing its adjoint.
//      A lane takes a ray's last few segments one after the other;
//      of a longer ray, each earlier segment is taken by six lanes, one per
//      component of the adjoint, at the same time: they give the segment's
//      transposed Jacobian;
//   5. backward_camera_kernel: the long rays' adjoints through those Jacobians,
//      then the camera: the initial state and the observer normalisation as
//      3-direction duals in (a, inclination, r_cam), contracted with the
//      adjoint of the initial state, and the five sums.
// The adjoint of t and phi is zero throughout (neither the metric nor the colour
// depends on them), so six components are carried.  What bounds it: one ray's
// chain.  Replayed and taken back by one lane, the longest ray of the 512^2
// image (673 steps, the median being 39) took the whole 8.6 ms, its warp issuing
// every fourth cycle.  With the segments in parallel the longest chain is 32 to
// 128 steps: 8.6 ms before, 3.0 after, 128^2 2.65 / 0.75 ms (CUDA events), of which
// the 512^2 replay takes 0.9, the crossing 0.4 and the chain 1.7 ms.
// The step sizes are held fixed (the adjoint of the discrete map with the
// forward's accepted steps; their own dependence on the parameters moves the
// solution by the truncation error only).
#include <cuda_runtime.h>

#include <cstdint>

#include "gg_device.cuh"
#include "gg_dual.cuh"
#include "gg_vjp.cuh"
#include "gg_launch.h"
#include "gg_trace_common.cuh"

namespace gg {

namespace {

// a^mu of one Kerr right-hand side in dual arithmetic (no r clamp: valid
// stages have r > 0).
template <int N>
GG_DEV void kerr_rhs_dual(double M, const Dual<N>& a, const Dual<N>& r, const Dual<N>& th,
                          const Dual<N> w[4], Dual<N> acc[4]) {
  Dual<N> s, c;
  sincos(th, &s, &c);
  const KerrGeo<Dual<N>> G = kerr_geometry<Dual<N>>(Dual<N>(M), a, r, s, c);
  kerr_contract<Dual<N>>(G, w, acc);
}

// g of a Keplerian emitter at the equator (redshift_factor at theta = pi/2)
// without the observer normalisation (divide by sqrt(-g_tt) at the camera).
template <class T>
GG_DEV T redshift_eq(double M, const T& a, const T& r, const T v[4]) {
  const T gtt = -(1.0 - 2.0 * M / r);
  const T gtph = -2.0 * M * a / r;
  const T gphph = r * r + a * a + 2.0 * M * a * a / r;
  const T p_t = gtt * v[0] + gtph * v[3];
  const double sm = ::sqrt(M);
  const T omega = sm / (r * sqrt(r) + a * sm);
  const T denom = -(gtt + 2.0 * gtph * omega + gphph * omega * omega);
  const T u_t = 1.0 / sqrt(denom);
  const T u_p = omega * u_t;
  const T p_phi = gtph * v[0] + gphph * v[3];
  const T e_emit = -(p_t * u_t + p_phi * u_p);
  return -p_t / e_emit;
}

// ---- backward -----------------------------------------------------------------
// Threads per CTA of the chain kernel and CTAs per SM: 255 registers, which
// still spill a little; at 168 (5 or 6 CTAs) the 512^2 backward took 3.7 ms
// instead of 3.4.
constexpr int kChainBlock = 64, kChainMinBlocks = 4;
constexpr int kRecDoubles = 31;   // a step's record: r, theta, v, h, k_1 .. k_6
// Records of 32 items side by side, so that a warp's accesses are coalesced:
// value c of step j of item i.
GG_DEV uint64_t rec_at(uint64_t i, uint32_t j, int c) {
  return ((i / 32) * (kCkptEvery * kRecDoubles) + j * kRecDoubles + c) * 32 + i % 32;
}

// This thread's columns of the chain kernel's shared memory: a step's stage
// derivatives and its stages' products (Xr, Xth, W).
struct ChainStore {
  double2 (*k)[2][kChainBlock];  // [6]
  double2 (*x)[3][kChainBlock];  // [6]
  GG_DEV void get_k(int l, double out[4]) const {
    const double2 a = k[l][0][threadIdx.x], b = k[l][1][threadIdx.x];
    out[0] = a.x;
    out[1] = a.y;
    out[2] = b.x;
    out[3] = b.y;
  }
  GG_DEV void set_k(int l, const double in[4]) const {
    k[l][0][threadIdx.x] = make_double2(in[0], in[1]);
    k[l][1][threadIdx.x] = make_double2(in[2], in[3]);
  }
  GG_DEV void get_x(int s, double out[6]) const {
#pragma unroll
    for (int j = 0; j < 3; ++j) {
      const double2 a = x[s][j][threadIdx.x];
      out[2 * j] = a.x;
      out[2 * j + 1] = a.y;
    }
  }
  GG_DEV void set_x(int s, const double in[6]) const {
#pragma unroll
    for (int j = 0; j < 3; ++j)
      x[s][j][threadIdx.x] = make_double2(in[2 * j], in[2 * j + 1]);
  }
};

// Stage S's r, theta and velocity, and its cotangent kb = dL/dk_S from the
// step's outputs and the later stages' products.
template <int S>
GG_DEV void vjp_stage(const ChainStore& C, double r, double th, const double v[4], double h,
                      double hh, const double lx[2], const double lv[4], double& pr, double& pth,
                      double w[4], double kb[4]) {
  const double ha = h * kDP.A[S];
  pr = fma(ha, v[1], r);
  pth = fma(ha, v[2], th);
#pragma unroll
  for (int i = 0; i < 4; ++i) w[i] = v[i];
#pragma unroll
  for (int l = 0; l < S; ++l) {
    double k[4];
    C.get_k(l, k);
    const double cv = h * kDP.B[S][l];
#pragma unroll
    for (int i = 0; i < 4; ++i) w[i] = fma(cv, k[i], w[i]);
    if (l < S - 1) {
      const double cb = hh * kDP.Abar[S][l];
      pr = fma(cb, k[1], pr);
      pth = fma(cb, k[2], pth);
    }
  }
  const double cb6 = hh * kDP.Abar[6][S], cv6 = h * kDP.B[6][S];
#pragma unroll
  for (int i = 0; i < 4; ++i) kb[i] = cv6 * lv[i];
  kb[1] = fma(cb6, lx[0], kb[1]);
  kb[2] = fma(cb6, lx[1], kb[2]);
#pragma unroll
  for (int j = S + 1; j < 6; ++j) {
    double x[6];
    C.get_x(j, x);
    const double cb = hh * kDP.Abar[j][S], cv = h * kDP.B[j][S];
    kb[0] = fma(cv, x[2], kb[0]);
    kb[1] = fma(cb, x[0], fma(cv, x[3], kb[1]));
    kb[2] = fma(cb, x[1], fma(cv, x[4], kb[2]));
    kb[3] = fma(cv, x[5], kb[3]);
  }
}

// Vector-Jacobian product through one accepted full Dormand-Prince step
// (Nystrom form, attempt_dp45_fp64), its stage derivatives in C: (lx, lv) is
// dL/d(r, theta, v) at its end on entry and at its start on return; dL/da is
// accumulated into *ga.
GG_DEV void step_vjp(const DevParams& P, const ChainStore& C, double r, double th,
                     const double v[4], double h, double lx[2], double lv[4], double* ga) {
  const double hh = h * h;
  // x_new = x + h v + ..., v_new = v + ...
  double xb[2] = {lx[0], lx[1]};
  double vb[4] = {lv[0], fma(h, lx[0], lv[1]), fma(h, lx[1], lv[2]), lv[3]};
#pragma unroll 1
  for (int s = 5; s >= 0; --s) {
    double pr, pth, w[4], kb[4];
    switch (s) {
      case 0: vjp_stage<0>(C, r, th, v, h, hh, lx, lv, pr, pth, w, kb); break;
      case 1: vjp_stage<1>(C, r, th, v, h, hh, lx, lv, pr, pth, w, kb); break;
      case 2: vjp_stage<2>(C, r, th, v, h, hh, lx, lv, pr, pth, w, kb); break;
      case 3: vjp_stage<3>(C, r, th, v, h, hh, lx, lv, pr, pth, w, kb); break;
      case 4: vjp_stage<4>(C, r, th, v, h, hh, lx, lv, pr, pth, w, kb); break;
      default: vjp_stage<5>(C, r, th, v, h, hh, lx, lv, pr, pth, w, kb); break;
    }
    // k_s = f(r_s, theta_s, w_s; a), back through its Jacobian
    double x[6] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
    kerr_rhs_vjp_hand(P.mass, P.spin, pr, pth, w, kb, &x[0], &x[1], &x[2], ga);
    if (s > 0) C.set_x(s, x);
    // r_s = r + h A_s v_r + ..., w_s = v + ...
    const double ha = h * kDP.A[s];
    xb[0] += x[0];
    xb[1] += x[1];
    vb[0] += x[2];
    vb[1] += fma(ha, x[0], x[3]);
    vb[2] += fma(ha, x[1], x[4]);
    vb[3] += x[5];
  }
  lx[0] = xb[0];
  lx[1] = xb[1];
#pragma unroll
  for (int i = 0; i < 4; ++i) lv[i] = vb[i];
}

// dL/d(start state of the crossing step) and the parameter terms of the
// crossing: the step, its continuous extension and root, the redshift and the
// disk colour in 7-direction duals (r, theta, the velocity, the spin;
// nothing depends on t and phi).  dl: dL/d rgb.
// Returns false when the step does not reach the disk (no contribution).
GG_DEV bool crossing_vjp(const DevParams& P, const double xb[4], const double vb[4], double h,
                         const double dl[3], double lam[6], double* ga, double* g_rin,
                         double* g_q, double* g_sobs) {
  using D7 = Dual<7>;
  D7 x[4], v[4], k[7][4], xa[4], va[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    x[i] = D7(xb[i]);
    v[i] = D7::var(vb[i], 2 + i);
  }
  x[1].d[0] = 1.0;
  x[2].d[1] = 1.0;
  const D7 a = D7::var(P.spin, 6);
  const double hh = h * h;
  for (int s = 0; s < 7; ++s) {
    D7 px[4], w[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      px[i] = x[i] + (h * kDP.A[s]) * v[i];
      w[i] = v[i];
    }
    for (int l = 0; l < s; ++l)
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        px[i] = px[i] + (hh * kDP.Abar[s][l]) * k[l][i];
        w[i] = w[i] + (h * kDP.B[s][l]) * k[l][i];
      }
    kerr_rhs_dual<7>(P.mass, a, px[1], px[2], w, k[s]);
    if (s == 6) {
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        xa[i] = px[i];
        va[i] = w[i];
      }
    }
  }
  // continuous extension coefficients of the 8 components
  D7 y0[8], r2[8], r3[8], r4[8], r5[8];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    D7 sx(0.0), sv(0.0);
    for (int l = 0; l < 7; ++l) {
      sx = sx + kDP.Dbar[l] * k[l][i];
      sv = sv + kDP.D[l] * k[l][i];
    }
    y0[i] = x[i];
    r2[i] = xa[i] - x[i];
    r3[i] = h * v[i] - r2[i];
    r4[i] = r2[i] - h * va[i] - r3[i];
    r5[i] = hh * sx;
    y0[4 + i] = v[i];
    r2[4 + i] = va[i] - v[i];
    r3[4 + i] = h * k[0][i] - r2[4 + i];
    r4[4 + i] = r2[4 + i] - h * k[6][i] - r3[4 + i];
    r5[4 + i] = h * sv;
  }
  // the root on values (safeguarded Newton), then one Newton step in duals
  StepSpan sp;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    sp.xb[i] = xb[i];
    sp.vb[i] = vb[i];
    sp.xa[i] = xa[i].v;
    sp.va[i] = va[i].v;
  }
  for (int l = 0; l < 7; ++l)
#pragma unroll
    for (int i = 0; i < 4; ++i) sp.k[l][i] = k[l][i].v;
  sp.h = h;
  double cval[8];
  const double s0 = dense_crossing(sp, 2, kHalfPi, cval);
  auto poly = [&](int c, const D7& s) {
    const D7 t = 1.0 - s;
    return y0[c] + s * (r2[c] + t * (r3[c] + s * (r4[c] + t * r5[c])));
  };
  const D7 sd0(s0);
  const D7 f = poly(2, sd0) - kHalfPi;
  const double t0 = 1.0 - s0;
  const double fp = r2[2].v + (1.0 - 2.0 * s0) * r3[2].v + s0 * (2.0 - 3.0 * s0) * r4[2].v +
                    2.0 * s0 * t0 * (1.0 - 2.0 * s0) * r5[2].v;
  const D7 sd = sd0 - f / fp;
  const D7 rc = poly(1, sd);
  double rcv = rc.v;
  {
    double cn[8];
#pragma unroll
    for (int c = 0; c < 8; ++c) cn[c] = cval[c];
    normalize_coords(cn);
    rcv = cn[1];
  }
  if (!(rcv >= P.r_inner && rcv <= P.r_outer)) return false;
  D7 vc[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) vc[i] = poly(4 + i, sd);
  // g (observer normalisation s_obs factored out), I = g^4 (r_in / r_c)^q
  const D7 g0 = redshift_eq<D7>(P.mass, a, rc, vc);
  const D7 g = g0 / P.sqrt_neg_gtt_obs;
  const D7 g2 = g * g;
  const D7 I = (g2 * g2) * pow(P.r_inner / rc, P.emissivity_index);
  // dL/dI through the disk colour (x^0.5, x^1.2, x^2.5), x = I / (1 + I)
  const double xv = I.v / (1.0 + I.v);
  const double dx = 1.0 / ((1.0 + I.v) * (1.0 + I.v));
  const double dLdI = dx * (dl[0] * 0.5 * ::pow(xv, -0.5) + dl[1] * 1.2 * ::pow(xv, 0.2) +
                            dl[2] * 2.5 * ::pow(xv, 1.5));
#pragma unroll
  for (int j = 0; j < 6; ++j) lam[j] = dLdI * I.d[j];
  *ga += dLdI * I.d[6];
  *g_rin += dLdI * I.v * P.emissivity_index / P.r_inner;
  *g_q += dLdI * I.v * ::log(P.r_inner / rc.v);
  *g_sobs += dLdI * (-4.0 * I.v / P.sqrt_neg_gtt_obs);
  return true;
}

// The initial state and the observer normalisation as functions of (a,
// inclination, r_cam) for image-plane point (u, v): the inclined camera
// (look_at = -r_hat, up = +z) and GeodesicRay::from_camera, in duals.
GG_DEV void camera_dual(const DevParams& P, double u, double v, Dual<3> y0[8], Dual<3>* sobs) {
  using D3 = Dual<3>;
  const D3 a = D3::var(P.spin, 0), th = D3::var(P.cam_pos[2], 1), r = D3::var(P.cam_pos[1], 2);
  D3 st, ct;
  sincos(th, &st, &ct);
  const D3 fwd[3] = {-st, D3(0.0), -ct};
  // right = normalize(fwd x up), up' = normalize(right x fwd), up = +z
  D3 right[3] = {fwd[1], -fwd[0], D3(0.0)};
  const D3 rn = sqrt(right[0] * right[0] + right[1] * right[1]);
  right[0] = right[0] / rn;
  right[1] = right[1] / rn;
  D3 up2[3] = {right[1] * fwd[2] - right[2] * fwd[1], right[2] * fwd[0] - right[0] * fwd[2],
               right[0] * fwd[1] - right[1] * fwd[0]};
  const D3 un = sqrt(up2[0] * up2[0] + up2[1] * up2[1] + up2[2] * up2[2]);
#pragma unroll
  for (int i = 0; i < 3; ++i) up2[i] = up2[i] / un;
  D3 d[3];
#pragma unroll
  for (int i = 0; i < 3; ++i) d[i] = fwd[i] + (u * P.half_w) * right[i] + (v * P.half_h) * up2[i];
  const D3 dn = sqrt(d[0] * d[0] + d[1] * d[1] + d[2] * d[2]);
  // local frame at phi = 0: r_hat = (st, 0, ct), theta_hat = (ct, 0, -st), phi_hat = (0, 1, 0)
  const D3 n_r = (d[0] * st + d[2] * ct) / dn;
  const D3 n_t = (d[0] * ct - d[2] * st) / dn;
  const D3 n_p = d[1] / dn;
  // Kerr metric at the camera (kerr.rs:61-94, no g_tphi, as the reference)
  const double M = P.mass;
  const D3 sig = r * r + a * a * ct * ct;
  const D3 del = r * r - 2.0 * M * r + a * a;
  const D3 gtt = -(1.0 - 2.0 * M * r / sig);
  const D3 grr = sig / del;
  const D3 gthth = sig;
  const D3 gphph = (r * r + a * a + 2.0 * M * a * a * r * st * st / sig) * st * st;
  const D3 kr = n_r / sqrt(grr), kth = n_t / sqrt(gthth), kph = n_p / sqrt(gphph);
  const D3 sns = grr * kr * kr + gthth * kth * kth + gphph * kph * kph;
  y0[0] = D3(P.cam_pos[0]);
  y0[1] = r;
  y0[2] = th;
  y0[3] = D3(P.cam_pos[3]);
  y0[4] = sqrt(-sns / gtt);
  y0[5] = kr;
  y0[6] = kth;
  y0[7] = kph;
  *sobs = sqrt(-gtt);
}

// ---- the work list ---------------------------------------------------------------
// Listed rays of the same number of segments: the first one's place in the
// list, and the segments ("items") and parallel segments of all rays before it.
struct BackwardBin {
  uint64_t start, item, par;
  uint32_t segs, pad;
};

// A window of the list: entries [e0, e1) with items from g0 and parallel
// segments from p0, and where the kernels leave their results.
struct BackwardWork {
  const uint64_t* list;      // sample indices
  const BackwardBin* bins;   // n_bins, and one past the end with the totals
  uint32_t n_bins;
  uint32_t tail;  // segments of a ray that one lane takes in sequence
  uint64_t e0, e1, g0, g1, p0, p1;
  double* rec;  // step records of the window's items
  double* ray;  // [kRayDoubles][e1 - e0]
  double* par;  // [p1 - p0][6][7]
};
constexpr int kRayDoubles = 11;  // dL/d(r, theta, v), dL/da, dL/dr_in, dL/dq, dL/ds_obs, valid

struct BackwardEntry {
  uint64_t e, item, par;  // place in the list, its first item and parallel segment
  uint32_t segs;
};

GG_DEV uint32_t parallel_segments(const BackwardWork& W, uint32_t segs) {
  return segs > W.tail ? segs - W.tail : 0u;
}

// The last bin whose `field` is at most `at`.
template <uint64_t BackwardBin::*FIELD>
GG_DEV uint32_t find_bin(const BackwardWork& W, uint64_t at) {
  uint32_t lo = 0, hi = W.n_bins;
  while (hi - lo > 1) {
    const uint32_t mid = (lo + hi) >> 1;
    if (W.bins[mid].*FIELD <= at) lo = mid; else hi = mid;
  }
  return lo;
}

GG_DEV BackwardEntry entry_at(const BackwardWork& W, uint64_t e) {
  const BackwardBin& b = W.bins[find_bin<&BackwardBin::start>(W, e)];
  const uint64_t k = e - b.start;
  return {e, b.item + k * b.segs, b.par + k * parallel_segments(W, b.segs), b.segs};
}

GG_DEV bool backward_key(const DiffOut& D, const double* dl, uint64_t idx, uint32_t* key) {
  const DiffRay dr = D.rays[idx];
  if (dr.cls != kClsDisk || dr.n_acc == 0) return false;
  if (dl[3 * idx] == 0.0 && dl[3 * idx + 1] == 0.0 && dl[3 * idx + 2] == 0.0) return false;
  uint32_t n_ck = dr.n_ckpt < D.ckpt_per_ray ? dr.n_ckpt : D.ckpt_per_ray;
  if (n_ck == 0) n_ck = 1;
  *key = D.ckpt_per_ray - n_ck;  // more segments, smaller key
  return true;
}

// Steps of segment `seg` of a ray with n_acc accepted ones; 0 if the counts do
// not fit together (the ray then has no gradient).
GG_DEV uint32_t segment_steps(uint32_t n_acc, uint32_t segs, uint32_t seg) {
  if (seg + 1 < segs) return (uint32_t)kCkptEvery;
  const uint32_t first = seg * kCkptEvery;
  return n_acc > first && n_acc - first <= (uint32_t)kCkptEvery ? n_acc - first : 0u;
}

// Neighbouring disk rays mostly share a key: the lanes of a warp with the
// same key take their slots with one atomic (count and scatter), which keeps
// the popular bins from serialising.  The loops run the same trips on every
// lane of a block, so the warp-wide votes see all 32 lanes.
__global__ void backward_count_kernel(const __grid_constant__ DevParams P,
                                      const __grid_constant__ DiffOut D, const double* dl,
                                      uint32_t* bins) {
  const unsigned lane = threadIdx.x & 31u;
  for (uint64_t base = (uint64_t)blockIdx.x * blockDim.x; base < P.n_rays;
       base += (uint64_t)gridDim.x * blockDim.x) {
    const uint64_t idx = base + threadIdx.x;
    uint32_t k = 0;
    const bool has = idx < P.n_rays && backward_key(D, dl, idx, &k);
    const unsigned grp = __match_any_sync(kFull, has ? k : 0xffffffffu);
    if (has && lane == (unsigned)(__ffs(grp) - 1)) atomicAdd(bins + k, (uint32_t)__popc(grp));
  }
}

// `next`: per key, the next free place of the list.
__global__ void backward_scatter_kernel(const __grid_constant__ DevParams P,
                                        const __grid_constant__ DiffOut D, const double* dl,
                                        unsigned long long* next, uint64_t* list) {
  const unsigned lane = threadIdx.x & 31u;
  for (uint64_t base = (uint64_t)blockIdx.x * blockDim.x; base < P.n_rays;
       base += (uint64_t)gridDim.x * blockDim.x) {
    const uint64_t idx = base + threadIdx.x;
    uint32_t k = 0;
    const bool has = idx < P.n_rays && backward_key(D, dl, idx, &k);
    const unsigned grp = __match_any_sync(kFull, has ? k : 0xffffffffu);
    if (has) {
      const unsigned leader = (unsigned)(__ffs(grp) - 1);
      unsigned long long first = 0;
      if (lane == leader) first = atomicAdd(next + k, (unsigned long long)__popc(grp));
      first = __shfl_sync(grp, first, leader);
      list[first + (uint32_t)__popc(grp & lanemask_lt())] = idx;
    }
  }
}

// Replays the window's segments, a lane each, and records their steps (the
// size negated where the step's end was reflected at a pole).
__global__ void __launch_bounds__(kTraceBlock, kTraceMinBlocksKerrChain)
    backward_replay_kernel(const __grid_constant__ DevParams P, const __grid_constant__ DiffOut D,
                           const __grid_constant__ BackwardWork W) {
  __shared__ double2 k_smem[7][2][kTraceBlock];
  const KStore K{k_smem};
  const uint64_t g = W.g0 + (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (g >= W.g1) return;
  const BackwardBin& b = W.bins[find_bin<&BackwardBin::item>(W, g)];
  const uint64_t in_bin = g - b.item;
  const uint32_t seg = (uint32_t)(in_bin % b.segs);
  const uint64_t idx = W.list[b.start + in_bin / b.segs];
  const uint32_t steps = segment_steps(D.rays[idx].n_acc, b.segs, seg);
  const Ckpt& c0 = D.ckpt[idx * D.ckpt_per_ray + seg];
  Ray R;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    R.x[i] = c0.x[i];
    R.v[i] = c0.v[i];
  }
  R.h = c0.h;
  R.lam = 0.0;
  bool k1v = false, k7p = false;
  double* const rec = W.rec + rec_at(g - W.g0, 0, 0);
  uint32_t j = 0, tries = 0;
  while (j < steps && tries < 100000u) {
    double q[6];
    q[0] = R.x[1];
    q[1] = R.x[2];
#pragma unroll
    for (int i = 0; i < 4; ++i) q[2 + i] = R.v[i];
    bool acc;
    double h_used = 0.0;
    StepEnd end;
    attempt_dp45_fp64<kMetricKerr>(P, R, K, k1v, k7p, acc, h_used, end);
    ++tries;
    if (acc) {
      double* const o = rec + (uint64_t)j * (kRecDoubles * 32);
#pragma unroll
      for (int c = 0; c < 6; ++c) o[c * 32] = q[c];
      const bool refl = end.xraw[2] < 0.0 || end.xraw[2] > kPi;
      o[6 * 32] = refl ? -h_used : h_used;
#pragma unroll
      for (int l = 0; l < 6; ++l) {
        double k[4];
        K.get(l, k);
#pragma unroll
        for (int i = 0; i < 4; ++i) o[(7 + 4 * l + i) * 32] = k[i];
      }
      ++j;
      tries = 0;
    }
  }
}

// The crossing steps of the window's rays: the adjoint at their start and the
// direct parameter terms.
__global__ void __launch_bounds__(64)
    backward_crossing_kernel(const __grid_constant__ DevParams P, const __grid_constant__ DiffOut D,
                             const double* dl_drgb, const __grid_constant__ BackwardWork W) {
  const uint64_t n = W.e1 - W.e0, le = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (le >= n) return;
  const BackwardEntry E = entry_at(W, W.e0 + le);
  const uint64_t idx = W.list[E.e];
  const double dl[3] = {dl_drgb[3 * idx], dl_drgb[3 * idx + 1], dl_drgb[3 * idx + 2]};
  const uint32_t steps = segment_steps(D.rays[idx].n_acc, E.segs, E.segs - 1);
  double lam[6] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
  double ga = 0.0, g_rin = 0.0, g_q = 0.0, g_sobs = 0.0;
  bool ok = steps > 0;
  if (ok) {
    const double* q = W.rec + rec_at(E.item + E.segs - 1 - W.g0, steps - 1, 0);
    const double x[4] = {0.0, q[0], q[32], 0.0};
    const double v[4] = {q[64], q[96], q[128], q[160]};
    ok = crossing_vjp(P, x, v, fabs(q[192]), dl, lam, &ga, &g_rin, &g_q, &g_sobs);
  }
  const double out[kRayDoubles] = {lam[0], lam[1], lam[2], lam[3], lam[4], lam[5],
                                   ga,     g_rin,  g_q,    g_sobs, ok ? 1.0 : 0.0};
#pragma unroll
  for (int c = 0; c < kRayDoubles; ++c) W.ray[c * n + le] = out[c];
}

// Back through `steps` recorded steps of one item, the last first.
GG_DEV void chain_segment(const DevParams& P, const BackwardWork& W, const ChainStore& C,
                          uint64_t item, uint32_t steps, double lx[2], double lv[4], double* ga) {
  for (uint32_t j = steps; j-- > 0;) {
    const double* q = W.rec + rec_at(item - W.g0, j, 0);
    const double r = q[0], th = q[32], h = q[192];
    const double v[4] = {q[64], q[96], q[128], q[160]};
#pragma unroll
    for (int l = 0; l < 6; ++l) {
      double k[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) k[i] = q[(7 + 4 * l + i) * 32];
      C.set_k(l, k);
    }
    if (h < 0.0) lx[1] = -lx[1];  // theta -> -theta or 2 pi - theta
    step_vjp(P, C, r, th, v, fabs(h), lx, lv, ga);
  }
}

// Blocks below `tail_blocks` take the window's rays, a lane each, through
// their last segments; the others the parallel segments, six lanes each.
__global__ void __launch_bounds__(kChainBlock, kChainMinBlocks)
    backward_chain_kernel(const __grid_constant__ DevParams P, const __grid_constant__ DiffOut D,
                          const __grid_constant__ BackwardWork W, unsigned tail_blocks) {
  __shared__ double2 k_smem[6][2][kChainBlock];
  __shared__ double2 x_smem[6][3][kChainBlock];
  const ChainStore C{k_smem, x_smem};
  if (blockIdx.x < tail_blocks) {
    const uint64_t n = W.e1 - W.e0, le = (uint64_t)blockIdx.x * kChainBlock + threadIdx.x;
    if (le >= n || W.ray[10 * n + le] == 0.0) return;
    const BackwardEntry E = entry_at(W, W.e0 + le);
    double lx[2], lv[4], ga = W.ray[6 * n + le];
    lx[0] = W.ray[le];
    lx[1] = W.ray[n + le];
#pragma unroll
    for (int i = 0; i < 4; ++i) lv[i] = W.ray[(2 + i) * n + le];
    const uint32_t par = parallel_segments(W, E.segs);
    for (uint32_t seg = E.segs; seg-- > par;) {
      const bool last = seg + 1 == E.segs;  // its last step is the crossing
      const uint32_t steps =
          last ? segment_steps(D.rays[W.list[E.e]].n_acc, E.segs, seg) - 1 : (uint32_t)kCkptEvery;
      chain_segment(P, W, C, E.item + seg, steps, lx, lv, &ga);
    }
    W.ray[le] = lx[0];
    W.ray[n + le] = lx[1];
#pragma unroll
    for (int i = 0; i < 4; ++i) W.ray[(2 + i) * n + le] = lv[i];
    W.ray[6 * n + le] = ga;
  } else {
    const uint64_t t = (uint64_t)(blockIdx.x - tail_blocks) * kChainBlock + threadIdx.x;
    const uint64_t p = W.p0 + t / 6;
    const int c = (int)(t % 6);
    if (p >= W.p1) return;
    const BackwardBin& b = W.bins[find_bin<&BackwardBin::par>(W, p)];
    const uint32_t per = parallel_segments(W, b.segs);  // > 0 in the bin that holds p
    const uint64_t in_bin = p - b.par;
    const uint64_t item = b.item + in_bin / per * b.segs + in_bin % per;
    double lx[2] = {c == 0 ? 1.0 : 0.0, c == 1 ? 1.0 : 0.0};
    double lv[4] = {c == 2 ? 1.0 : 0.0, c == 3 ? 1.0 : 0.0, c == 4 ? 1.0 : 0.0,
                    c == 5 ? 1.0 : 0.0};
    double ga = 0.0;
    chain_segment(P, W, C, item, (uint32_t)kCkptEvery, lx, lv, &ga);
    double* o = W.par + ((p - W.p0) * 6 + c) * 7;
    o[0] = lx[0];
    o[1] = lx[1];
#pragma unroll
    for (int i = 0; i < 4; ++i) o[2 + i] = lv[i];
    o[6] = ga;
  }
}

// The adjoints of the window's rays at their camera states, through the
// parallel segments' Jacobians, then the camera; the five sums into grad5.
__global__ void __launch_bounds__(128)
    backward_camera_kernel(const __grid_constant__ DevParams P, const __grid_constant__ BackwardWork W,
                           double* grad5) {
  double acc5[5] = {0.0, 0.0, 0.0, 0.0, 0.0};
  const uint64_t n = W.e1 - W.e0;
  for (uint64_t le = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; le < n;
       le += (uint64_t)gridDim.x * blockDim.x) {
    if (W.ray[10 * n + le] == 0.0) continue;
    const BackwardEntry E = entry_at(W, W.e0 + le);
    double l[6], ga = W.ray[6 * n + le];
#pragma unroll
    for (int c = 0; c < 6; ++c) l[c] = W.ray[c * n + le];
    for (uint32_t seg = parallel_segments(W, E.segs); seg-- > 0;) {
      const double* m = W.par + (E.par + seg - W.p0) * 42;
      double t[7] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
#pragma unroll
      for (int c = 0; c < 6; ++c)
#pragma unroll
        for (int d = 0; d < 7; ++d) t[d] = fma(l[c], m[7 * c + d], t[d]);
#pragma unroll
      for (int c = 0; c < 6; ++c) l[c] = t[c];
      ga += t[6];
    }
    double u, v;
    sample_uv(P, W.list[E.e], u, v);
    Dual<3> y0[8], sobs;
    camera_dual(P, u, v, y0, &sobs);
    constexpr int kComp[6] = {1, 2, 4, 5, 6, 7};
    const double g_sobs = W.ray[9 * n + le];
    double g3[3] = {ga, 0.0, 0.0};
#pragma unroll
    for (int p = 0; p < 3; ++p) {
#pragma unroll
      for (int c = 0; c < 6; ++c) g3[p] += l[c] * y0[kComp[c]].d[p];
      g3[p] += g_sobs * sobs.d[p];
    }
    acc5[0] += g3[0];
    acc5[1] += g3[1];
    acc5[2] += g3[2];
    acc5[3] += W.ray[7 * n + le];
    acc5[4] += W.ray[8 * n + le];
  }
#pragma unroll
  for (int p = 0; p < 5; ++p) {
    double x = acc5[p];
    for (int o = 16; o > 0; o >>= 1) x += __shfl_down_sync(0xffffffffu, x, o);
    if ((threadIdx.x & 31u) == 0 && x != 0.0) atomicAdd(grad5 + p, x);
  }
}

unsigned blocks_for(uint64_t n, unsigned per) { return (unsigned)((n + per - 1) / per); }

unsigned list_grid(const DevParams& P, int sms) {
  const uint64_t need = (P.n_rays + 255) / 256, cap = (uint64_t)sms * 8;
  return (unsigned)(need < cap ? (need < 1 ? 1 : need) : cap);
}

}  // namespace

cudaError_t launch_backward_count(const DevParams& P, const DiffOut& D, const double* dl_drgb,
                                  uint32_t* bins, int sms, cudaStream_t stream) {
  const cudaError_t e =
      cudaMemsetAsync(bins, 0, sizeof(uint32_t) * (size_t)D.ckpt_per_ray, stream);
  if (e != cudaSuccess) return e;
  backward_count_kernel<<<list_grid(P, sms), 256, 0, stream>>>(P, D, dl_drgb, bins);
  return cudaGetLastError();
}

size_t backward_bins_bytes(uint32_t n_keys) { return sizeof(BackwardBin) * ((size_t)n_keys + 1); }

BackwardPlan backward_plan(const uint32_t* counts, uint32_t n_keys, uint64_t* next, void* bins) {
  auto* b = static_cast<BackwardBin*>(bins);
  BackwardPlan plan{};
  uint64_t listed = 0;
  for (uint32_t k = 0; k < n_keys; ++k) listed += counts[k];
  // An earlier segment costs six lanes' work where the ray's own lane would take
  // it in sequence: with fewer rays than lanes (37,888) the chain is what
  // counts, with more the work.  Backward ms at 1 / 2 / 3 / 4 / 5 segments in
  // sequence, by listed rays: 1,800 (64^2) 0.50 / 0.66 / 0.83 / 1.00 / 1.16, 7,000
  // (128^2) 0.76 / 0.72 / 0.89 / 1.05 / 1.22, 17,000 1.28 / 0.96 / 1.03 / 1.20 / 1.33,
  // 28,000 1.86 / 1.21 / 1.17 / 1.35 / 1.52, 44,000 2.77 / 1.75 / 1.59 / 1.63 / 1.79,
  // 112,000 (512^2) 6.40 / 3.72 / 3.16 / 3.01 / 2.96.
  plan.tail = listed <= 4096 ? 1 : listed <= 24576 ? 2 : listed <= 65536 ? 3 : 4;
  for (uint32_t k = 0; k < n_keys; ++k) {
    next[k] = plan.entries;
    if (!counts[k]) continue;
    const uint32_t segs = n_keys - k;
    b[plan.bins++] = BackwardBin{plan.entries, plan.items, plan.par, segs, 0u};
    const uint64_t par = segs > plan.tail ? segs - plan.tail : 0u;
    plan.entries += counts[k];
    plan.items += (uint64_t)counts[k] * segs;
    plan.par += (uint64_t)counts[k] * par;
  }
  b[plan.bins] = BackwardBin{plan.entries, plan.items, plan.par, 1u, 0u};
  return plan;
}

// The window that starts at entry e0 and holds at most `most` items (one entry
// at least).
BackwardWindow backward_window(const void* bins, const BackwardPlan& plan, uint64_t e0,
                               uint64_t most) {
  const auto* b = static_cast<const BackwardBin*>(bins);
  BackwardWindow w{};
  bool begun = false;
  for (uint32_t k = 0; k < plan.bins; ++k) {
    const uint64_t stop = b[k + 1].start;
    if (e0 >= stop) continue;
    const uint64_t from = e0 > b[k].start ? e0 - b[k].start : 0;
    const uint64_t par = b[k].segs > plan.tail ? b[k].segs - plan.tail : 0u;
    if (!begun) {
      w.e0 = e0;
      w.g0 = b[k].item + from * b[k].segs;
      w.p0 = b[k].par + from * par;
      w.e1 = w.e0;
      w.g1 = w.g0;
      w.p1 = w.p0;
      begun = true;
    }
    if (w.e1 > w.e0 && w.g1 - w.g0 >= most) break;  // one ray may have more than `most`
    const uint64_t have = stop - b[k].start - from, left = most - (w.g1 - w.g0);
    uint64_t take = left / b[k].segs;
    if (take > have) take = have;
    if (take == 0 && w.e1 == w.e0) take = 1;
    w.e1 += take;
    w.g1 += take * b[k].segs;
    w.p1 += take * par;
    if (take < have) break;
  }
  return w;
}

size_t backward_rec_bytes(uint64_t items) {
  return ((items + 31) / 32) * 32 * sizeof(double) * kCkptEvery * kRecDoubles;
}
size_t backward_ray_bytes(uint64_t entries, uint64_t par) {
  return sizeof(double) * (kRayDoubles * entries + 42 * par);
}

cudaError_t launch_backward_scatter(const DevParams& P, const DiffOut& D, const double* dl_drgb,
                                    uint64_t* next, uint64_t* list, int sms,
                                    cudaStream_t stream) {
  backward_scatter_kernel<<<list_grid(P, sms), 256, 0, stream>>>(
      P, D, dl_drgb, reinterpret_cast<unsigned long long*>(next), list);
  return cudaGetLastError();
}

cudaError_t launch_backward_window(const DevParams& P, const DiffOut& D, const double* dl_drgb,
                                   const uint64_t* list, const void* bins, const BackwardPlan& plan,
                                   const BackwardWindow& w, double* rec, double* ray,
                                   double* grad5, int sms, cudaStream_t stream) {
  BackwardWork W{};
  W.list = list;
  W.bins = static_cast<const BackwardBin*>(bins);
  W.n_bins = plan.bins;
  W.tail = plan.tail;
  W.e0 = w.e0;
  W.e1 = w.e1;
  W.g0 = w.g0;
  W.g1 = w.g1;
  W.p0 = w.p0;
  W.p1 = w.p1;
  W.rec = rec;
  W.ray = ray;
  W.par = ray + kRayDoubles * (w.e1 - w.e0);
  const uint64_t n = w.e1 - w.e0;
  if (n == 0) return cudaSuccess;
  backward_replay_kernel<<<blocks_for(w.g1 - w.g0, kTraceBlock), kTraceBlock, 0, stream>>>(P, D, W);
  backward_crossing_kernel<<<blocks_for(n, 64), 64, 0, stream>>>(P, D, dl_drgb, W);
  const unsigned tail = blocks_for(n, kChainBlock);
  backward_chain_kernel<<<tail + blocks_for((w.p1 - w.p0) * 6, kChainBlock), kChainBlock, 0,
                          stream>>>(P, D, W, tail);
  const unsigned cam = blocks_for(n, 128), cap = (unsigned)sms * 8;
  backward_camera_kernel<<<cam < cap ? cam : cap, 128, 0, stream>>>(P, W, grad5);
  return cudaGetLastError();
}

}  // namespace gg

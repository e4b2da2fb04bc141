// The reference-order step on four lanes per ray, for batches too small to fill the schedulers.
//
// One ray per lane, a small batch waits for its slowest ray's chain of steps, each of which issues
// 3300 instructions of one warp while the SM's other lanes idle.  Here four lanes share a ray: lane
// 0 integrates r, theta, t and phi, lane 1 p_r, lane 2 p_theta (lane 3 computes what lane 2 does).
// Every stage they exchange r, theta, p_r and p_theta; each lane evaluates the metric's denominators
// and numerators, but takes only its own components' quotients -- the three sets have one form,
//
//   lane 0   n0/X n1/X  D/Y  1/Y   n4/Z          X = Sigma Delta,     Y = Sigma,   Z = X sin^2
//   lane 1   n5/X n6/X n7/Y n8/Y   n8/Z  n9/X    X = (Sigma Delta)^2, Y = Sigma^2, Z = Y sin^2
//   lane 2  n10/X n11/X n12/Y n13/Y n14/Z m14/X  X, Y likewise,                    Z = Y sin^4
//
// -- and its own sums; sin and cos of theta come from lanes 0 and 1, sin of 2 theta from lanes 2
// and 3, by one call.  Every value is formed by the operations of RefMode<double> on the same
// operands in the same order, so the results are its results bit for bit.
// Kernel times, one lane per ray and four: 64^2 photons at rtol 1e-6 1.87-2.0 and 1.5-1.68 ms, 16^2
// 1.82 and 1.26; 80^2 at a* = 0.99, rtol 1e-8 4.28 and 3.67; 96^2 (two warps per scheduler) 1.87 and
// 1.66; 142^2, where the schedulers fill up, 2.25 and 2.91 (quad_fits).
#pragma once

#include "krr_kernels.cuh"

namespace krr {

struct Quad {
  using M = RefMode<double>;
  static constexpr unsigned FULL = 0xffffffffu;
  // Slots of a lane's own components: lane 0 {r, theta, t, phi}, lane 1 {p_r}, lanes 2 and 3 {p_theta}.
  double y[4], f[4];
  double pt, pph, h, lam, m_null, m_q;
  Refs<double> ref;
  long long attempts;
  int n_steps, n_rej, state, role, base;
  bool rejected_before;

  __device__ static double from(double x, int lane) { return __shfl_sync(FULL, x, lane); }
  // Whether all four lanes of the ray agree.
  __device__ bool group_all(bool ok) const { return ((__ballot_sync(FULL, ok) >> base) & 15u) == 15u; }

  __device__ void own(const double v[NV], double s[4]) const {
    s[0] = role == 0 ? v[CR] : role == 1 ? v[CPR] : v[CPTH];
    s[1] = role == 0 ? v[CTH] : 0.0;
    s[2] = role == 0 ? v[CT] : 0.0;
    s[3] = role == 0 ? v[CPH] : 0.0;
  }
  __device__ void all(const double s[4], double v[NV]) const {  // by all lanes of the warp
    v[CR] = from(s[0], base);
    v[CTH] = from(s[1], base);
    v[CT] = from(s[2], base);
    v[CPH] = from(s[3], base);
    v[CPR] = from(s[0], base + 1);
    v[CPTH] = from(s[0], base + 2);
  }

  __device__ void start(const Params& P, const double y0[8], double q0) {
    Ray<M> ry;
    ray_init<M>(P, y0, q0, ry);
    role = min((int)(threadIdx.x & 3u), 2);
    base = (int)(threadIdx.x & 28u);
    own(ry.y, y);
    own(ry.f, f);
    pt = ry.pt;
    pph = ry.pph;
    h = ry.h;
    lam = 0.0;
    m_null = ry.m_null;
    m_q = 0.0;
    ref = ry.ref;
    attempts = 0;
    n_steps = n_rej = 0;
    state = ry.state;
    rejected_before = false;
  }

  // The lane's components of the right-hand side at (r, th, pr, pth) into g; s, c on every lane.  False,
  // with values that must not be used, outside the branch-free range (P.div_ok holds: quad_fits).
  __device__ __forceinline__ bool rhs(const Params& P, double r, double th, double pr, double pth, double g[4], double& s,
                                      double& c) const {
    const bool near = fabs(th) < 1000.0;
    const double arg = near ? ((threadIdx.x & 2u) ? 2.0 * th : th) : 0.0;
    __builtin_assume(fabs(arg) < 2000.0);
    double sa, ca;
    sincos(arg, &sa, &ca);
    s = from(sa, base);
    c = from(ca, base);
    const double sin2th = from(sa, base + 2);
    const M::Terms t = M::terms(P, r, s, c, sin2th);
    const bool zero = role == 0, one = role == 1;
    const double X = zero ? t.sd : t.sd2, Y = zero ? t.sig : t.sig2;
    const double Z = zero ? t.sds2 : one ? t.sig2s2 : t.sig2s4;
    const double a0 = zero ? t.n0 : one ? t.n5 : t.n10, a1 = zero ? t.n1 : one ? t.n6 : t.n11;
    const double a2 = zero ? t.dlt : one ? t.n7 : t.n12, a3 = zero ? 1.0 : one ? t.n8 : t.n13;
    const double a4 = zero ? t.n4 : one ? t.n8 : t.n14, a5 = one ? t.n9 : t.m14;
    const Recip ix = recip(X), iy = recip(Y);
    const double q0 = quotient(a0, ix), q1 = quotient(a1, ix), q2 = quotient(a2, iy), q3 = quotient(a3, iy);
    const double q4 = quotient(a4, Z), q5 = quotient(a5, ix);
    const unsigned gap = min(min(fraction_gap(X), fraction_gap(Y)), fraction_gap(Z));
    const bool axis = pph == 0.0;
    const double pt2 = pt * pt, ptpph = pt * pph, pr2 = pr * pr, pth2 = pth * pth, pph2 = pph * pph;
    const double last = axis ? 0.0 : q4 + q5;
    const double fp = -0.5 * (q0 * pt2 + 2.0 * q1 * ptpph + q2 * pr2 + q3 * pth2 + last * pph2);
    g[0] = zero ? q2 * pr : fp;
    g[1] = zero ? q3 * pth : 0.0;
    g[2] = zero ? q0 * pt + q1 * pph : 0.0;
    g[3] = zero ? q1 * pt + (axis ? 0.0 : q4) * pph : 0.0;
    return near && gap != 0u && M::in_range(t);
  }

  // One step attempt (attempt<RefMode<double>, false> without the disk event), by every lane of the
  // warp; `live`: this ray is still running.
  __device__ __forceinline__ void attempt(const Params& P, bool live) {
    if (live) attempts += 1;
    if (live && attempts > P.guard) {
      state = FAILURE;
      live = false;
    }
    const double remaining = P.lambda_max - lam;
    const bool last = h >= remaining;
    const double he = last ? remaining : h;
    double acc[2], g[4], k1[2], k2[4], u[2], bs[4], es[4], yn[4];
    double r, th, pr, pth, s, c;
    bool ok = true;
    auto stage = [&]() {  // at y + he acc
      const double v0 = y[0] + he * acc[0], v1 = y[1] + he * acc[1];
      r = from(v0, base);
      th = from(v1, base);
      pr = from(v0, base + 1);
      pth = from(v0, base + 2);
      ok = rhs(P, r, th, pr, pth, g, s, c) && ok;
    };
#pragma unroll
    for (int i = 0; i < 2; ++i) acc[i] = dp::A10 * f[i];
    stage();
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      k1[i] = g[i];
      acc[i] = dp::A20 * f[i] + dp::A21 * g[i];
    }
    stage();
#pragma unroll
    for (int i = 0; i < 4; ++i) k2[i] = g[i];
#pragma unroll
    for (int i = 0; i < 2; ++i) acc[i] = dp::A30 * f[i] + dp::A31 * k1[i] + dp::A32 * g[i];
    stage();
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      acc[i] = dp::A40 * f[i] + dp::A41 * k1[i] + dp::A42 * k2[i] + dp::A43 * g[i];
      u[i] = dp::A50 * f[i] + dp::A51 * k1[i] + dp::A52 * k2[i] + dp::A53 * g[i];
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      bs[i] = dp::B0 * f[i] + dp::B2 * k2[i] + dp::B3 * g[i];
      es[i] = dp::E0 * f[i] + dp::E2 * k2[i] + dp::E3 * g[i];
    }
    stage();
#pragma unroll
    for (int i = 0; i < 2; ++i) acc[i] = u[i] + dp::A54 * g[i];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      bs[i] = bs[i] + dp::B4 * g[i];
      es[i] = es[i] + dp::E4 * g[i];
    }
    stage();
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      bs[i] = bs[i] + dp::B5 * g[i];
      es[i] = es[i] + dp::E5 * g[i];
    }
    acc[0] = bs[0];
    acc[1] = bs[1];
    stage();
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      yn[i] = y[i] + he * bs[i];
      es[i] = es[i] + dp::E6 * g[i];
    }
    // A step outside the branch-free range: over again by every lane of the ray, for all components.
    const bool straight = group_all(ok);
    if (__any_sync(FULL, live && !straight)) {
      StepStart<M> a;
      all(y, a.y);
      all(f, a.f);
      a.pt = pt;
      a.pph = pph;
      a.h = he;
      if (!straight) {
        const StepEnd<M> e = dp_stages_careful<M, false>(P, a);
        own(e.yn, yn);
        own(e.k6, g);
        own(e.esum, es);
        r = e.yn[CR];
        th = e.yn[CTH];
        pr = e.yn[CPR];
        pth = e.yn[CPTH];
        s = e.tr.s;
        c = e.tr.c;
      }
      __syncwarp();
    }
    bool fin = true;
    double q[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      fin = fin && finite_(yn[i]) && finite_(g[i]);
      const double e = he * es[i], scale = P.atol + P.rtol * py_max(fabs(y[i]), fabs(yn[i]));
      const double v = quotient_any(e, scale);
      q[i] = v * v;
    }
    fin = group_all(fin);
    const double c0 = from((q[2] + q[0]) + (q[1] + q[3]), base);
    const double c1 = from(q[0], base + 1), c2 = from(q[0], base + 2);
    const int outward = __shfl_sync(FULL, g[0] > 0.0 ? 1 : 0, base);  // dr/dlambda at the candidate
    const double en = sqrt((c0 + (c1 + c2)) / 8.0);
    if (!live) return;
    if (!fin || !finite_(en)) {
      state = FAILURE;
      return;
    }
    const bool accept = en <= 1.0;
    if (!(accept && last)) {
      h = he * step_factor<M>(en, rejected_before);
      if (h > P.h_max) h = P.h_max;
    }
    rejected_before = !accept;
    if (!accept) {
      n_rej += 1;
      if (h < P.h_min) state = FAILURE;
      return;
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      y[i] = yn[i];
      f[i] = g[i];
    }
    lam = last ? P.lambda_max : lam + he;
    n_steps += 1;
    // Carter constant and null error (the latter on lane 0, which holds the velocities).
    const double e = -pt;
    const double l2 = pph != 0.0 ? quotient_any(pph * pph, s * s) : 0.0;
    const double carter_now = pth * pth + (c * c) * (l2 - P.a2 * e * e);
    m_q = py_max(m_q, drift<M>(fabs(carter_now - ref.q0), ref.q_den));
    double total = pt * f[2];
    total = total + pr * f[0];
    total = total + pth * f[1];
    total = total + pph * f[3];
    m_null = py_max(m_null, drift<M>(fabs(0.5 * total), ref.e_den));
    if (h < P.h_min) state = FAILURE;
    else if (r < 0.0 || th < -THETA_TOL || th > PI + THETA_TOL) state = OUT_OF_DOMAIN;
    else if (pph != 0.0 && fabs(s) < AXIS_SIN_TOL) state = OUT_OF_DOMAIN;
    else if (r <= P.r_capture) state = CAPTURED;
    else if (r >= P.r_escape && outward) state = ESCAPED;
    else if (lam >= P.lambda_max || (long long)n_steps >= P.max_steps) state = MAX_AFFINE;
  }

  __device__ void store(const Outputs& o, long long n) const {
    const int lane = (int)(threadIdx.x & 3u);
    double* Y = o.Y + n * 8;
    if (lane == 1) Y[5] = y[0];
    if (lane == 2) Y[6] = y[0];
    if (lane != 0) return;
    Y[0] = y[2];
    Y[1] = y[0];
    Y[2] = y[1];
    Y[3] = y[3];
    Y[4] = pt;
    Y[7] = pph;
    o.state[n] = state;
    if (o.n_steps) o.n_steps[n] = n_steps;
    if (o.n_rej) o.n_rej[n] = n_rej;
    if (o.lam) o.lam[n] = lam;
    if (o.max_null) o.max_null[n] = m_null;
    if (o.max_e) o.max_e[n] = 0.0;
    if (o.max_lz) o.max_lz[n] = 0.0;
    if (o.max_q) o.max_q[n] = m_q;
  }
};

// One ray per four lanes (k_trace_plain's arguments; no disk event).
__global__ void __launch_bounds__(128) k_trace_quad(const __grid_constant__ Params P, const Image* __restrict__ images,
                                                    int n_images, const double* __restrict__ Y0,
                                                    const long long* __restrict__ index, long long n, Outputs o, Queue* q);

}  // namespace krr

// Device helpers shared by the engines (k_cycle, k_small, k_force, k_ens): the
// FP32 reciprocal of the mixed-precision pair terms and the closed-form
// Nose-Hoover velocity solve of both precisions.
#pragma once

#include <math.h>

// 1/x by the hardware's approximate reciprocal (PTX rcp.approx.ftz.f32, at
// most 1 ulp from the exact quotient): x = r^2 of a pair inside the cut-off,
// a normal number.  The pair terms are FP32 anyway; the IEEE-rounded
// division costs several instructions more per pair.
__device__ __forceinline__ float clmd_rcp_f32(float x) {
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}

// The cell (0 .. n - 1) of a coordinate wrapped into the box, c cells per unit
// length.  A NaN, which wrapping leaves one, would convert to the smallest
// integer: its cell is the first.  (Not max(.., 0) on the integers: built so,
// the ensemble's search lists pairs of the first two cells twice.)
__device__ __forceinline__ int clmd_cell(double x, double c, int n) {
  return min((int)fmax(x * c, 0.0), n - 1);
}

// The implicit Nose-Hoover velocity step of int-verlet-nh-mav.f:105-147 in
// closed form.  The reference's Newton sweeps stop at the
// fixed point v (1 + dth p) = V + dth a =: W, p = psi1 + (m sum v^2 - 3NkT)
// dth / Q.  With S = m sum W^2 the new PSI is therefore the root of
//   f(p) = p - psi1 - (S / (1 + dth p)^2 - 3NkT) dth / Q,
// which is increasing and concave for 1 + dth p > 0 (one root), and every
// velocity is W / (1 + dth p): one reduction instead of a reduction per
// sweep (FP64, 500 replicas 9.07 -> 6.32 ms a window; N = 5,921 on one cluster
// 6.05 -> 4.10 ms per 200 steps).  Newton's method from psi1, two or three
// steps in practice; the step limit is 1e-13 of the terms' scale (|p| + |psi1| +
// (S + 3NkT) dth/Q; rounding noise in f is a few 1e-16 of it, so a tighter limit
// can stall).  Where overlapping atoms make S huge, that scale is far above p,
// and steps from below multiply 1 + dth p by 1.5 each (some 200 for S = 1e100):
// the last one must also be 1e-8 of 1 + dth p.
// False (no convergence) if the root is not finite or the iteration does not
// settle: mixed precision then stops, as the reference's STOP; FP64 takes the
// sweeps (clmd_nh_closed).
__device__ __forceinline__ bool clmd_nh_root(double S, double psi1, double nkt3, double dth,
                                             double Q, double& p) {
  const double k0 = dth / Q;
  const double scale = fabs(psi1) + k0 * (S + fabs(nkt3));
  p = psi1;
  for (int it = 0; it < 1000; it++) {
    const double c = 1.0 / (1.0 + dth * p);
    const double f = p - psi1 - (S * c * c - nkt3) * k0;
    const double fp = 1.0 + 2.0 * S * dth * k0 * c * c * c;
    const double d = f / fp;
    p = p - d;
    if (!(fabs(d) > 1e-13 * (scale + fabs(p))) && !(dth * fabs(d) > 1e-8 * fabs(1.0 + dth * p)))
      return isfinite(p) && 1.0 + dth * p > 0.0;
  }
  return false;
}

// The reference's sweeps (int-verlet-nh-mav.f:105-147) on scalars alone: their
// iterates are vn_k = al W + be V with factors common to all atoms, so every
// sweep follows from three sums (sum W.W, W.V, V.V).
struct ClmdSweep {
  double al = 0.0, be = 1.0, p;
  __device__ __forceinline__ explicit ClmdSweep(double psi1) : p(psi1) {}
  __device__ __forceinline__ void next(double sww, double swv, double svv, double psi1, double m,
                                       double nkt3, double dt, double Q) {
    const double dth = dt / 2, dt2 = dt * dt / 2;
    const double sumv2 = al * al * sww + 2.0 * al * be * swv + be * be * svv;
    const double up = 1.0 + dth * p;
    const double draw = (up * sumv2 - (al * sww + be * swv)) * m * dt / Q;
    double delps = draw + up * ((-m * sumv2 + nkt3) * dth / Q - (psi1 - p));
    delps = delps / (-dt2 * m * sumv2 / Q - up);
    const double a1 = (1.0 - dth * delps * al) / up, b1 = -dth * delps * be / up;
    al = a1;
    be = b1;
    p += delps;
  }
};

constexpr int kNhSweeps = 1000;  // the reference's limit; more: it stops

// How many sweeps one atom needs until the relative change of each of its
// velocity components stays within 1e-10; kNhSweeps + 1 if it never does.
__device__ __forceinline__ int clmd_nh_sweeps(const double* W, const double* V, double sww,
                                              double swv, double svv, double psi1, double m,
                                              double nkt3, double dt, double Q) {
  ClmdSweep s(psi1);
  int need = 1;
  for (int k = 1; k <= kNhSweeps; k++) {
    const double al = s.al, be = s.be;
    s.next(sww, swv, svv, psi1, m, nkt3, dt, Q);
    bool moved = false;
    for (int d = 0; d < 3; d++) {
      const double nx = s.al * W[d] + s.be * V[d], vo = al * W[d] + be * V[d];
      moved |= fabs(nx - vo) > 1e-10 * fabs(nx);
    }
    if (moved) need = k + 1;
    if (!moved && k > 1) break;
  }
  return need;
}

// PSI after n sweeps
static __device__ __noinline__ double clmd_nh_swept(int n, double sww, double swv, double svv,
                                                    double psi1, double m, double nkt3,
                                                    double dt, double Q) {
  ClmdSweep s(psi1);
  for (int k = 0; k < n; k++) s.next(sww, swv, svv, psi1, m, nkt3, dt, Q);
  return s.p;
}

// Whether the closed form stands for the sweeps (FP64): a root was found from
// a PSI with 1 + dth PSI > 0.  Otherwise (a thermostat mass so small, or a PSI
// so negative, that a step turns velocities round; a NaN) the kernels take
// the sweeps themselves.
__device__ __forceinline__ bool clmd_nh_closed(bool root, double psi1, double dth) {
  return root && 1.0 + dth * psi1 > 0.0;
}

// 2D-RZ SGH kernels for sm_103a (GB300), FP64: the num_dims == 2 branches of
// Explicit-Lagrange-Kokkos/SGH_solver on quad meshes (x axial, y radial).
//
// Compiled twice, like sgh_kernels.cu: FIERRO_FMA=0 with --fmad=false (every
// operation the reference's, in its order; square roots and shared-divisor
// quotients by the correctly rounded Newton forms of sgh_common.cuh; the sign of a
// zero normal apart) and
// FIERRO_FMA=1 (contraction and reciprocal reuse allowed; the Newton square
// roots, quotients and reciprocals).
//
// One cycle is 2 + 4*rk_num_stages launches: k_dt, then per RK stage
//   k_force_rz (elements)  corner normals, area and Barlow corner areas of the
//                          stage's input quad, MARS forces with the hoop terms,
//                          hypo strength model (force_sgh.cpp:407-808)
//   k_node_rz  (nodes)     corner-force gather, velocity, boundary conditions,
//                          position, and the areal node mass of the new position
//                          (momentum.cpp:11-53, boundary.cpp:10-55,
//                          geometry.cpp:9-26, sgh_solve.cpp:496-505)
//   k_axis_rz  (boundary nodes) nodes on the axis take the largest half-mass of
//                          their off-axis edge neighbours (sgh_solve.cpp:547-578)
//   k_elem_rz  (elements)  radius-weighted energy (energy_sgh.cpp:6-55), RZ volume
//                          (geometry.cpp:369-434), density and EOS
//                          (properties.cpp:118-219), the next stage's divergence
//                          (momentum.cpp:298-378) and on the last stage the CFL
//                          step (time_integration.cpp:161-246)
// then k_end.  Nothing is accumulated with atomics.
#include <cstdint>

#include "sgh_rz.h"

#ifndef FIERRO_FMA
#error "compile with -DFIERRO_FMA=0 or -DFIERRO_FMA=1"
#endif

#if FIERRO_FMA
#define FIERRO_RZ_IMPL rz_fma_impl
#else
#define FIERRO_RZ_IMPL rz_exact_impl
#endif

namespace fierro {
namespace FIERRO_RZ_IMPL {

#include "sgh_launch.cuh"
#include "sgh_common.cuh"
#include "sgh_hex_geometry.cuh"  // mul_add, mul_mul
#include "sgh_user_mat.cuh"

constexpr int kRzBlock = 128;
constexpr int kRzNodeBlock = 256;

// The differences a quad's normals, area, volume and edge lengths are made of,
// each formed once: a sum or square of the opposite difference is its exact
// negation, which the compiler does not see.
struct RzDiffs {
  double x02, x13, y02, y13;                      // diagonals
  double x03, x23, x21, x01, y03, y23, y21, y01;  // edges
};
__device__ __forceinline__ RzDiffs rz_diffs(const double (&x)[4], const double (&y)[4]) {
  RzDiffs d;
  d.x02 = x[0] - x[2];
  d.x13 = x[1] - x[3];
  d.y02 = y[0] - y[2];
  d.y13 = y[1] - y[3];
  d.x03 = x[0] - x[3];
  d.x23 = x[2] - x[3];
  d.x21 = x[2] - x[1];
  d.x01 = x[0] - x[1];
  d.y03 = y[0] - y[3];
  d.y23 = y[2] - y[3];
  d.y21 = y[2] - y[1];
  d.y01 = y[0] - y[1];
  return d;
}

// get_bmatrix2D (geometry.cpp:315-365): outward corner normals B[l][dim];
// opposite corners' are opposite.
__device__ __forceinline__ void rz_bmatrix(const RzDiffs& d, double (&B)[4][2]) {
  B[0][0] = 0.5 * d.y13;
  B[1][0] = -0.5 * d.y02;
  B[2][0] = -B[0][0];
  B[3][0] = -B[1][0];
  B[0][1] = -0.5 * d.x13;
  B[1][1] = 0.5 * d.x02;
  B[2][1] = -B[0][1];
  B[3][1] = -B[1][1];
}

// get_area_quad (geometry.cpp:438-466)
__device__ __forceinline__ double rz_area(const RzDiffs& d) {
  return 0.5 * mul_mul(d.x02, d.y13, -d.x13, d.y02);
}

// v / 6, correctly rounded (the IEEE quotient in both modes): a quotient one
// ulp off at most and one remainder step through the rounded reciprocal
// (Markstein's theorem), 3 FP64 operations instead of a general division.
__device__ __forceinline__ double sixth(double v) {
  if (!plain_range(__double_as_longlong(v))) return lib_div(v, 6.0);
  const double r = 1.0 / 6.0, q = v * r;
  return fma(fma(-6.0, q, v), r, q);
}

// get_vol_quad (geometry.cpp:369-434): volume per radian of the revolved quad.
__device__ __forceinline__ double rz_vol(const double (&y)[4], const RzDiffs& d) {
  return sixth(mul_mul(y[2] + y[3] + y[0], mul_mul(d.y23, d.x03, -d.y03, d.x23),  //
                       y[0] + y[1] + y[2], mul_mul(d.y01, d.x21, -d.y21, d.x01)));
}

// heron (geometry.cpp:470-500)
__device__ __forceinline__ double rz_heron(double x1, double y1, double x2, double y2, double x3, double y3) {
  double S = 0.0;
  const double a = sqrt((x2 - x1) * (x2 - x1) + (y2 - y1) * (y2 - y1));
  S = S + a;
  const double b = sqrt((x3 - x2) * (x3 - x2) + (y3 - y2) * (y3 - y2));
  S = S + b;
  const double c = sqrt((x3 - x1) * (x3 - x1) + (y3 - y1) * (y3 - y1));
  S = S + c;
  S = S * 0.5;
  return sqrt(S * (S - a) * (S - b) * (S - c));
}

// get_area_weights2D (geometry.cpp:503-547): Barlow's corner areas.
__device__ __forceinline__ void rz_corner_areas(const double (&x)[4], const double (&y)[4], double (&ca)[4]) {
  double rc = 0.0, zc = 0.0;
#pragma unroll
  for (int l = 0; l < 4; ++l) {
    rc = rc + 0.25 * y[l];
    zc = zc + 0.25 * x[l];
  }
  const double A12 = rz_heron(x[0], y[0], zc, rc, x[1], y[1]);
  const double A23 = rz_heron(x[1], y[1], zc, rc, x[2], y[2]);
  const double A34 = rz_heron(x[2], y[2], zc, rc, x[3], y[3]);
  const double A41 = rz_heron(x[3], y[3], zc, rc, x[0], y[0]);
  ca[0] = (5. * A41 + 5. * A12 + A23 + A34) / 12.;
  ca[1] = (A41 + 5. * A12 + 5. * A23 + A34) / 12.;
  ca[2] = (A41 + A12 + 5. * A23 + 5. * A34) / 12.;
  ca[3] = (5. * A41 + A12 + A23 + 5. * A34) / 12.;
}

// Without stress the hoop terms are tau(1,0) A_c / r = (+0 A_c) / r and
// (tau(1,1) - tau(2,2)) A_c / r = ((0 - p) - (0 - p)) A_c / r: exactly +0.0
// whenever p and the corner area A_c are finite.  A_c is finite unless one of
// Heron's factors s - a, s - b, s - c of a centroid triangle rounds to zero or
// below.  For a triangle of area T and semi-perimeter s, each factor is at least
// T^2 / s^3 (the product of all three is T^2 / s and each is below s), while the
// computed factors carry an absolute error of about 9 eps s (sides and s to a few
// ulps each); so T > 3 sqrt(eps) s^2 ~ 3.2e-8 s^2 keeps every computed factor
// positive.  With s <= P / 2 for the L1 perimeter P, |cross| = 2T > 1e-4 P^2 is
// sufficient by more than three orders of magnitude.  That margin lets the test
// run in single precision (6 FP64 operations for the centroid's offset instead
// of 68): with the diagonals a = x2 - x0, b = x3 - x1 and m = x1 + x3 - x0 - x2
// the corners lie at (-a/2 - m/4, -b/2 + m/4, a/2 - m/4, b/2 + m/4) from the
// centroid, and rounding a, b and m to 24 bits moves a cross product by under
// 1e-6 P^2.  Quads too small (P < 1e-13) or large for float fail it.
// True for all four centroid triangles (and finite coordinates) means the corner
// areas need not be formed; otherwise they are, as the reference does.
__device__ __forceinline__ bool rz_corner_areas_finite(double x02, double x13, double y02, double y13, double m_x,
                                                       double m_y) {
  const float ax = 0.5f * f32_of(-x02), bx = 0.5f * f32_of(-x13);
  const float ay = 0.5f * f32_of(-y02), by = 0.5f * f32_of(-y13);
  const float mx = 0.25f * f32_of(m_x), my = 0.25f * f32_of(m_y);
  const float px[4] = {-ax - mx, -bx + mx, ax - mx, bx + mx};
  const float py[4] = {-ay - my, -by + my, ay - my, by + my};
  bool ok = true;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int j = (i + 1) & 3;
    const float cross = px[i] * py[j] - py[i] * px[j];
    const float P = fabsf(px[i]) + fabsf(py[i]) + fabsf(px[j]) + fabsf(py[j]) + fabsf(px[j] - px[i]) +
                    fabsf(py[j] - py[i]);
    const float far = 1e-4f * P * P;
    ok = ok && (fabsf(cross) > far) && far > 1e-30f;
  }
  return ok;
}

__device__ __forceinline__ void gather4(const int* nie, int e, int (&nid)[4]) {
  const int4 q = __ldg(reinterpret_cast<const int4*>(nie) + e);
  nid[0] = q.x;
  nid[1] = q.y;
  nid[2] = q.z;
  nid[3] = q.w;
}

// Whether the cycle runs; beside its k_dt, asked as k_dt asks it.
__device__ __forceinline__ bool force_active(const RzForceArgs& a) {
  return a.beside_dt ? !a.ctrl->stopped : a.ctrl->active != 0;
}

// The scalar steps the one-thread-per-element passes and the lane passes
// (sgh_rz_lanes.cuh) share.  den (q1 c + q2 |v - v_avg|), force_sgh.cpp:520-636:
__device__ __forceinline__ double rz_impedance(double den, double q1c, double qb, double d0, double d1) {
  return den * mul_add(q1c, qb, mode_sqrt(mul_mul(d0, d0, d1, d1)));
}
// shock detector (:653-690): the minimum over neighbours of the monotone
// r_face(div_nb) sits at the smallest (div + small > 0) or largest neighbour
// divergence, as in the 3D kernel
__device__ __forceinline__ double rz_limiter_min(const RzForceArgs& a, double div, int k0, int k1, long long kmin,
                                                 long long kmax) {
  const double D = div + a.small;
  double r_min = 1.0;
  if (k1 > k0) {
    const double dsel = okey_decode(__double_as_longlong(D) > 0 ? kmin : kmax);
    if (is_finite(D) && (__double_as_longlong(D) & kAbsMask) != 0 && is_finite(dsel)) {
      const double r_face = newton_div(0.9 * (dsel + a.small), D);
      r_min = okey(r_face) < okey(1.0) ? r_face : 1.0;
    } else {
      for (int k = k0; k < k1; ++k) {
        const double r_face = newton_div(0.9 * (a.div[__ldg(a.eie + k)] + a.small), D);
        r_min = fmin(r_face, r_min);
      }
    }
  }
  return r_min;
}
// A corner force without the terms that are zeros (:718-755): the shear stress (+0.0)
// times the other component of the inward normal and, off the axis, the hoop term.
// With them a force of -0.0 stays one on the axis alone, beside a negative normal.
__device__ __forceinline__ double rz_zero_terms(double f, double other_normal, double radius) {
  if ((__double_as_longlong(f) & kAbsMask) != 0) return f;
  const bool off_axis = __double_as_longlong(radius) > __double_as_longlong(1e-14);
  return off_axis || __double_as_longlong(other_normal) >= 0 ? 0.0 : f;
}
// Mach-number detector with the characteristic length sqrt(area) (:692-700)
__device__ __forceinline__ double rz_mach_switch(double area, double div, double sspd, double fuzz) {
  return at_most_1(newton_div(20.0 * (mode_sqrt(area) * fabs(div)), sspd + fuzz));
}
// Order key of the element CFL step (time_integration.cpp:189-228); a NaN bounds nothing.
__device__ __forceinline__ long long rz_cfl_key(double d2, double sspd, double dt_cfl, double fuzz) {
  const double dt_l = newton_div(dt_cfl * mode_sqrt(d2), sspd + fuzz);
  return (__double_as_longlong(dt_l) & kAbsMask) > 0x7FF0000000000000LL ? 0x7FFFFFFFFFFFFFFFLL : okey(dt_l);
}

// ---------------------------------------------------------------------------
// Corner forces of the quad (force_sgh.cpp:407-808).  The shock-direction and
// curl terms feed only unused values (use_shock_dir = 0, phi_curl unused) and
// are not computed.  STRENGTH: tau = stress(1) - p I and the hypo model with the
// RZ velocity gradient (momentum.cpp:151-217); otherwise stress is zero.
template <bool STRENGTH>
__global__ void __launch_bounds__(kRzBlock) k_force_rz(const RzForceArgs a) {
  previous_launch_done();
  if (!force_active(a)) return;
  const int e = blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= a.ne) return;
  const int ne = a.ne;
  int nid[4];
  gather4(a.nie, e, nid);
  double x[4], y[4], u[4], v[4];
#pragma unroll
  for (int l = 0; l < 4; ++l) {
    x[l] = a.x[nid[l]];
    y[l] = a.y[nid[l]];
    u[l] = a.u[nid[l]];
    v[l] = a.v[nid[l]];
  }
  const RzDiffs df = rz_diffs(x, y);
  double B[4][2], ca[4] = {0.0, 0.0, 0.0, 0.0};
  rz_bmatrix(df, B);
  const double area = rz_area(df);
  const double den = a.den[e], pres = a.pres[e], sspd = a.sspd[e], vol = a.vol[e], div = a.div[e];
  const bool hoop_zero = !STRENGTH && is_finite(pres) && 
      rz_corner_areas_finite(df.x02, df.x13, df.y02, df.y13, -df.x01 - df.x23, -df.y01 - df.y23);
  if (!hoop_zero) rz_corner_areas(x, y, ca);
  const int mat = a.mat[e];
  const double* q = a.qtab + 4 * mat;
  const bool compress = is_negative(div);
  const double qa = compress ? q[0] : q[1];
  const double qb = compress ? q[2] : q[3];
  // Cauchy stress (:480-493): tau(i,j) = stress(i,j), tau(i,i) -= p
  double sc[9], t[9];
#pragma unroll
  for (int k = 0; k < 9; ++k) {
    sc[k] = STRENGTH ? a.stress_cur[(size_t)k * ne + e] : 0.0;
    t[k] = sc[k];
  }
  t[0] = t[0] - pres;
  t[4] = t[4] - pres;
  t[8] = t[8] - pres;
  // average velocity (:500-512); 0.25*v is exact, so fusing equals product-then-add
  double vs0 = 0.0, vs1 = 0.0;
#pragma unroll
  for (int l = 0; l < 4; ++l) {
    vs0 = fma(0.25, u[l], vs0);
    vs1 = fma(0.25, v[l], vs1);
  }
  // MARS impedances (:520-636); |inward normal| = |B|, the same at opposite corners
  const double bn[2] = {mode_sqrt(mul_mul(B[0][0], B[0][0], B[0][1], B[0][1])),
                        mode_sqrt(mul_mul(B[1][0], B[1][0], B[1][1], B[1][1]))};
  double mu[4];
  double s0 = 0.0, s1 = 0.0, s3 = 0.0;
  const double q1c = qa * sspd;
#pragma unroll
  for (int l = 0; l < 4; ++l) {
    const double mu_term = rz_impedance(den, q1c, qb, u[l] - vs0, v[l] - vs1) * bn[l & 1];
    s0 = l ? mul_add(s0, mu_term, u[l]) : mu_term * u[l];
    s1 = l ? mul_add(s1, mu_term, v[l]) : mu_term * v[l];
    s3 = l ? s3 + mu_term : mu_term;
    mu[l] = mu_term;
  }
  s0 = from_zero(s0);
  s1 = from_zero(s1);
  double vstar0 = 0.0, vstar1 = 0.0;
  if (s3 > a.fuzz) {
#if FIERRO_FMA
    const double rs = mode_rcp(s3);
    vstar0 = s0 * rs;
    vstar1 = s1 * rs;
#else
    const Divisor ds3 = divisor(s3);  // correctly rounded quotients, one reciprocal seed
    vstar0 = quot(s0, ds3);
    vstar1 = quot(s1, ds3);
#endif
  }
  const int k0 = a.eie_start[e], k1 = a.eie_start[e + 1];
  long long kmin = 0x7FFFFFFFFFFFFFFFLL, kmax = (long long)0x8000000000000000ULL;
  for (int k = k0; k < k1; ++k) {
    const long long key = okey(a.div[__ldg(a.eie + k)]);
    kmin = key < kmin ? key : kmin;
    kmax = key > kmax ? key : kmax;
  }
  const double phi = rz_mach_switch(area, div, sspd, a.fuzz) *
                     (1.0 - at_least_0(rz_limiter_min(a, div, k0, k1, kmin, kmax)));
  // corner forces with the inward normals -B, then the hoop-stress terms (:718-755)
  const double vs[2] = {vstar0, vstar1};
#pragma unroll
  for (int l = 0; l < 4; ++l) {
    const double pm = phi * mu[l];
    const double a0 = -B[l][0], a1 = -B[l][1];
    const double vl[2] = {u[l], v[l]};
    double f[2];
    if (hoop_zero) {
      // finite normals and no shear: the products with tau's zeros are zeros, and so
      // are the hoop terms; adding those changes no more than the sign of a zero
      f[0] = rz_zero_terms(mul_mul(a0, t[0], pm, vs[0] - vl[0]), a1, y[l]);
      f[1] = rz_zero_terms(mul_mul(a1, t[4], pm, vs[1] - vl[1]), a0, y[l]);
    } else {
#pragma unroll
      for (int d = 0; d < 2; ++d) f[d] = mul_add(mul_mul(a0, t[d], a1, t[3 + d]), pm, vs[d] - vl[d]);
      const double r = y[l];
      if (r > 1e-14) {
        f[0] = f[0] + t[3] * ca[l] / r;
        f[1] = f[1] + (t[4] - t[8]) * ca[l] / r;
      }
    }
    a.force[(size_t)(l * 2 + 0) * ne + e] = f[0];
    a.force[(size_t)(l * 2 + 1) * ne + e] = f[1];
  }
  if (STRENGTH) {
    if (a.stype[mat] == 1) {
      // get_velgrad2D (momentum.cpp:151-217) with the outward normals
      double L[9];
#pragma unroll
      for (int k = 0; k < 9; ++k) L[k] = 0.0;
      const double mean_radius = vol / area;
      const double elem_vel_r = 0.25 * (v[0] + v[1] + v[2] + v[3]);
      const double inverse_area = 1.0 / area;
      L[0] = (u[0] * B[0][0] + u[1] * B[1][0] + u[2] * B[2][0] + u[3] * B[3][0]) * inverse_area;
      L[1] = (u[0] * B[0][1] + u[1] * B[1][1] + u[2] * B[2][1] + u[3] * B[3][1]) * inverse_area;
      L[3] = (v[0] * B[0][0] + v[1] * B[1][0] + v[2] * B[2][0] + v[3] * B[3][0]) * inverse_area;
      L[4] = (v[0] * B[0][1] + v[1] * B[1][1] + v[2] * B[2][1] + v[3] * B[3][1]) * inverse_area;
      L[8] = elem_vel_r / mean_radius;
      double s0v[9];
#pragma unroll
      for (int k = 0; k < 9; ++k) s0v[k] = a.stress0[(size_t)k * ne + e];
      user_strength_model(sc, s0v, L, a.statev + e, ne, mat, den, a.sie0[e], vol, a.ctrl->dt, a.rk_alpha);
#pragma unroll
      for (int k = 0; k < 9; ++k) a.stress_out[(size_t)k * ne + e] = sc[k];
    } else if (a.copy_stress) {
#pragma unroll
      for (int k = 0; k < 9; ++k) a.stress_out[(size_t)k * ne + e] = sc[k];
    }
  }
}

// ---------------------------------------------------------------------------
// Node update.  The velocity uses the areal mass the previous stage left; the
// mass of the new position replaces it at the end (the reference recomputes it
// after update_state2D, and nothing in between reads it).
__global__ void __launch_bounds__(kRzNodeBlock) k_node_rz(const RzNodeArgs a) {
  previous_launch_done();
  if (!a.ctrl->active) return;
  const int n = blockIdx.x * blockDim.x + threadIdx.x;
  if (n >= a.nn) return;
  const size_t ne = (size_t)a.ne;
  double f0 = 0.0, f1 = 0.0;
  const int c0 = a.cin_start[n], c1 = a.cin_start[n + 1];
  // four corners' ids, then their force loads, are issued together; the sums keep
  // the corner order
  for (int base = c0; base < c1; base += 4) {
    double g[4][2];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const bool in = base + k < c1;
      const int cid = in ? __ldg(a.cin + base + k) : 0;
      const size_t at = (size_t)((cid & 3) * 2) * ne + (cid >> 2);
      g[k][0] = in ? a.force[at] : 0.0;
      g[k][1] = in ? a.force[at + ne] : 0.0;
    }
#pragma unroll
    for (int k = 0; k < 4; ++k)
      if (base + k < c1) {
        f0 = k || base > c0 ? f0 + g[k][0] : g[k][0];
        f1 = k || base > c0 ? f1 + g[k][1] : g[k][1];
      }
  }
  f0 = from_zero(f0);
  f1 = from_zero(f1);
  const double adt = a.rk_alpha * a.ctrl->dt;
  const double m = a.node_mass[n];
  const double u0 = a.u0[n], v0 = a.v0[n];
#if FIERRO_FMA
  const double rm = mode_rcp(m);
  double u1 = mul_add(u0, adt * f0, rm);
  double v1 = mul_add(v0, adt * f1, rm);
#else
  const Divisor dm = divisor(m);  // correctly rounded quotients, one reciprocal seed
  double u1 = u0 + quot(adt * f0, dm);
  double v1 = v0 + quot(adt * f1, dm);
#endif
  const unsigned bc = a.bc_mask[n];
  if (bc & 1u) u1 = 0.0;
  if (bc & 2u) v1 = 0.0;
  const double hu = (u1 + u0) * 0.5, hv = (v1 + v0) * 0.5;
  const double r_in = a.yin[n];  // read before y1 is overwritten (yin == y1 after the first stage)
  a.u1[n] = u1;
  a.v1[n] = v1;
  a.hx[n] = hu;
  a.hy[n] = hv;
  a.rad[n] = r_in;
  const double x1 = mul_add(a.x0[n], adt, hu);
  const double y1 = mul_add(a.y0[n], adt, hv);
  a.x1[n] = x1;
  a.y1[n] = y1;
  double mn = 0.0;
  if (y1 > a.tiny) mn = newton_div(a.node_ext[n], y1);
  a.node_mass[n] = mn;
}

// Nodes on the axis (y < tiny) among the boundary nodes: the largest half-mass
// of their off-axis edge neighbours.  Off-axis masses are not written here.
__global__ void __launch_bounds__(kRzNodeBlock) k_axis_rz(const RzAxisArgs a) {
  previous_launch_done();
  if (!a.ctrl->active) return;
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= a.naxis) return;
  const int n = a.nodes[i];
  if (!(a.y1[n] < a.tiny)) return;
  double m = a.node_mass[n];
  for (int k = a.nin_start[i]; k < a.nin_start[i + 1]; ++k) {
    const int nb = a.nin[k];
    if (a.y1[nb] > a.tiny) m = fmax(m, a.node_mass[nb] / 2.0);
  }
  a.node_mass[n] = m;
}

// ---------------------------------------------------------------------------
template <int KIND>
__global__ void __launch_bounds__(kRzBlock) k_elem_rz(const RzElemArgs a) {
  previous_launch_done();
  const int e = blockIdx.x * blockDim.x + threadIdx.x;
  Ctrl* ctrl = a.ctrl;
  if (KIND != 2 && !ctrl->active) return;
  long long dkey = 0x7FFFFFFFFFFFFFFFLL;
  if (e < a.ne) {
    const int ne = a.ne;
    int nid[4];
    gather4(a.nie, e, nid);
    double x[4], y[4], u[4], v[4];
#pragma unroll
    for (int l = 0; l < 4; ++l) {
      x[l] = a.x[nid[l]];
      y[l] = a.y[nid[l]];
      u[l] = a.u[nid[l]];
      v[l] = a.v[nid[l]];
    }
    double sie1 = 0.0;
    if (KIND != 2) {
      // energy (energy_sgh.cpp:16-52): power = sum_c F_c r_c (v1 + v0)/2 with the
      // node radius of the stage's input state
      double power = 0.0;
#pragma unroll
      for (int l = 0; l < 4; ++l) {
        const double r = a.rad[nid[l]];
        const double F0 = a.force[(size_t)(l * 2 + 0) * ne + e] * r, h0 = a.hx[nid[l]];
        power = l ? mul_add(power, F0, h0) : F0 * h0;
        power = mul_add(power, a.force[(size_t)(l * 2 + 1) * ne + e] * r, a.hy[nid[l]]);
      }
      const double adt = a.rk_alpha * ctrl->dt;
      sie1 = mul_add(a.sie0[e], -newton_div(adt, a.mass[e]), from_zero(power));
      a.sie1[e] = sie1;
    }
    const RzDiffs df = rz_diffs(x, y);
    const double vol = (KIND == 2) ? a.vol[e] : rz_vol(y, df);
    // divergence for the next stage (momentum.cpp:298-378)
    double B[4][2];
    rz_bmatrix(df, B);
    const double area = rz_area(df);
    const Divisor da = divisor(area);  // two quotients, one reciprocal seed
    const double inverse_area = quot(1.0, da);
    const double mean_radius = quot(vol, da);
    const double elem_vel_r = 0.25 * (v[0] + v[1] + v[2] + v[3]);
    const double su = mul_add(mul_add(mul_mul(u[0], B[0][0], u[1], B[1][0]), u[2], B[2][0]), u[3], B[3][0]);
    const double sv = mul_add(mul_add(mul_mul(v[0], B[0][1], v[1], B[1][1]), v[2], B[2][1]), v[3], B[3][1]);
    const double div =
        from_zero(mul_add(mul_add(newton_div(elem_vel_r, mean_radius), sv, inverse_area), su, inverse_area));
    a.div[e] = div;
    double sspd;
    if (KIND != 2) {
      a.vol[e] = vol;
      // update_state2D (properties.cpp:140, eos.cpp:12-46)
      const double den = newton_div(a.mass[e], vol);
      const double gamma = a.gamma[e], csmin = a.csmin[e];
      const double pres = (gamma - 1.0) * sie1 * den;
      sspd = mode_sqrt(gamma * (gamma - 1.0) * sie1);
      if (sspd < csmin) sspd = csmin;
      a.den[e] = den;
      a.pres[e] = pres;
      a.sspd[e] = sspd;
      if (__double_as_longlong(vol) <= 0 || !is_finite(vol)) atomicOr(&ctrl->status, FIERRO_STATUS_BAD_VOLUME);
      if (!is_finite(sie1) || !is_finite(pres)) atomicOr(&ctrl->status, FIERRO_STATUS_BAD_STATE);
    } else {
      sspd = a.sspd[e];
    }
    if (KIND != 0) {
      // CFL step (time_integration.cpp:189-228): the six node-pair distances; the
      // minimum of the square roots is the square root of the minimum
      const double dx[6] = {df.x01, df.x02, df.x03, df.x21, df.x13, df.x23};
      const double dy[6] = {df.y01, df.y02, df.y03, df.y21, df.y13, df.y23};
      long long kd = 0x7FFFFFFFFFFFFFFFLL;  // squares are >= 0: their bits order as they do
#pragma unroll
      for (int i = 0; i < 6; ++i) {
        const long long k = __double_as_longlong(mul_mul(dx[i], dx[i], dy[i], dy[i])) & kAbsMask;
        kd = k < kd ? k : kd;
      }
      dkey = rz_cfl_key(__longlong_as_double(kd), sspd, a.dt_cfl, a.fuzz);
    }
  }
  if (KIND != 0) {
    const long long k = block_min_key(dkey);
    if (threadIdx.x == 0) a.cfl_part[blockIdx.x] = k;
  }
}

#include "sgh_rz_lanes.cuh"

__global__ void __launch_bounds__(kRzNodeBlock) k_ext_rz(int nn, const double* node_mass, const double* y,
                                                        double* ext) {
  const int n = blockIdx.x * blockDim.x + threadIdx.x;
  if (n < nn) ext[n] = node_mass[n] * y[n];
}

// Energy tallies (sgh_solve.cpp:73-101): IE = sum M e, KE = 1/2 sum m y |v|^2.
constexpr int kRzEnergyBlock = 256;
__global__ void __launch_bounds__(kRzEnergyBlock) k_energy_rz_part(const RzEnergyArgs a) {
  __shared__ double sh[2][kRzEnergyBlock];
  double ie = 0.0, ke = 0.0;
  const int stride = gridDim.x * blockDim.x;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < a.ne; i += stride) ie += a.mass[i] * a.sie[i];
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < a.nn; i += stride) {
    double k = 0;
    k += a.u[i] * a.u[i];
    k += a.v[i] * a.v[i];
    ke += a.node_mass[i] * a.y[i] * k;
  }
  sh[0][threadIdx.x] = ie;
  sh[1][threadIdx.x] = ke;
  __syncthreads();
  for (int s = kRzEnergyBlock / 2; s > 0; s >>= 1) {
    if (threadIdx.x < s) {
      sh[0][threadIdx.x] += sh[0][threadIdx.x + s];
      sh[1][threadIdx.x] += sh[1][threadIdx.x + s];
    }
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    a.part[blockIdx.x] = sh[0][0];
    a.part[gridDim.x + blockIdx.x] = sh[1][0];
  }
}

// One warp's two lanes add the blocks' partials in order, energies and kinetic
// energies in the same instructions.
__global__ void __launch_bounds__(2 * kEnergyMaxBlocks) k_energy_rz_final(const RzEnergyArgs a, int nblocks) {
  __shared__ double sh[2 * kEnergyMaxBlocks];
  if (threadIdx.x < 2 * nblocks) sh[threadIdx.x] = a.part[threadIdx.x];
  __syncthreads();
  if (threadIdx.x >= 2) return;
  const double* p = sh + threadIdx.x * nblocks;
  double t = 0.0;
  for (int b = 0; b < nblocks; ++b) t += p[b];
  a.out[threadIdx.x] = threadIdx.x ? 0.5 * t : t;
}

// ---------------------------------------------------------------------------
static unsigned blocks_for(long long n, int bs) { return (unsigned)((n + bs - 1) / bs); }

static void launch_force(const RzForceArgs& a, cudaStream_t s) {
  const int bs = small_mesh_block(a.ne, kRzBlock);
  if (a.stress_out) launch(k_force_rz<true>, blocks_for(a.ne, bs), bs, s, a);
  else if (a.lanes) launch(k_force_rz_lanes, blocks_for(4LL * a.ne, kRzLaneBlock), kRzLaneBlock, s, a);
  else launch(k_force_rz<false>, blocks_for(a.ne, bs), bs, s, a);
}
static void launch_node(const RzNodeArgs& a, cudaStream_t s) {
  const int bs = small_mesh_block(a.nn, kRzNodeBlock);
  launch(k_node_rz, blocks_for(a.nn, bs), bs, s, a);
}
static void launch_axis(const RzAxisArgs& a, cudaStream_t s) {
  const int bs = small_mesh_block(a.naxis, kRzNodeBlock);
  launch(k_axis_rz, blocks_for(a.naxis > 0 ? a.naxis : 1, bs), bs, s, a);
}
static void launch_elem(const RzElemArgs& a, int kind, cudaStream_t s) {
  if (a.lanes) {
    const unsigned g = blocks_for(4LL * a.ne, kRzLaneBlock);
    if (kind == 0) launch(k_elem_rz_lanes<0>, g, kRzLaneBlock, s, a);
    else if (kind == 1) launch(k_elem_rz_lanes<1>, g, kRzLaneBlock, s, a);
    else launch(k_elem_rz_lanes<2>, g, kRzLaneBlock, s, a);
    return;
  }
  const int bs = a.block ? a.block : kRzBlock;
  const unsigned g = blocks_for(a.ne, bs);
  if (kind == 0) launch(k_elem_rz<0>, g, bs, s, a);
  else if (kind == 1) launch(k_elem_rz<1>, g, bs, s, a);
  else launch(k_elem_rz<2>, g, bs, s, a);
}
static void launch_ext(int nn, const double* node_mass, const double* y, double* ext, cudaStream_t s) {
  k_ext_rz<<<blocks_for(nn, kRzNodeBlock), kRzNodeBlock, 0, s>>>(nn, node_mass, y, ext);
}
static void launch_energy(const RzEnergyArgs& a, cudaStream_t s) {
  const int nb = energy_blocks(a.ne, a.nn);
  k_energy_rz_part<<<nb, kRzEnergyBlock, 0, s>>>(a);
  k_energy_rz_final<<<1, 2 * kEnergyMaxBlocks, 0, s>>>(a, nb);
}

}  // namespace FIERRO_RZ_IMPL

#if FIERRO_FMA
const RzKernelSet& rz_kernels_fma() {
  static const RzKernelSet k = {rz_fma_impl::launch_force, rz_fma_impl::launch_node, rz_fma_impl::launch_axis,
                                rz_fma_impl::launch_elem, rz_fma_impl::launch_ext, rz_fma_impl::launch_energy};
  return k;
}
#else
const RzKernelSet& rz_kernels_exact() {
  static const RzKernelSet k = {rz_exact_impl::launch_force, rz_exact_impl::launch_node,
                                rz_exact_impl::launch_axis, rz_exact_impl::launch_elem,
                                rz_exact_impl::launch_ext, rz_exact_impl::launch_energy};
  return k;
}
#endif

}  // namespace fierro

// The quad passes of small 2D-RZ meshes: four lanes per element (one per corner).
// Included in sgh_rz_kernels.cu's implementation namespace; bit for bit the
// one-thread-per-element passes, in both modes.
//
// Bound, as in sgh_lanes.cuh: a warp issues one FP64 instruction every ~65 clocks,
// so a mesh that fills few warps takes as long as one thread's chain.  Here a
// lane forms its corner's terms, the sums whose order is part of the result run in
// one lane each, and independent quotients run in different lanes of the same
// instructions.
#pragma once

constexpr int kRzLaneBlock = 64;  // threads: two warps, sixteen elements

__device__ __forceinline__ double quad_lane(double v, int src) { return __shfl_sync(0xFFFFFFFFu, v, src, 4); }
__device__ __forceinline__ double quad_other(double v) { return __shfl_xor_sync(0xFFFFFFFFu, v, 1); }
__device__ __forceinline__ long long quad_min(long long k) {
  for (int o = 2; o > 0; o >>= 1) {
    const long long t = __shfl_xor_sync(0xFFFFFFFFu, k, o);
    k = t < k ? t : k;
  }
  return k;
}
__device__ __forceinline__ double flip(double v, bool neg) {
  return __hiloint2double(__double2hiint(v) ^ (neg ? (int)0x80000000 : 0), __double2loint(v));
}
// The four corners' values of one field.
__device__ __forceinline__ void quad_all(double v, double (&all)[4]) {
#pragma unroll
  for (int k = 0; k < 4; ++k) all[k] = quad_lane(v, k);
}
// What both passes start from: the diagonal a lane's normal lies along (1-3 for
// even corners, 0-2 for odd ones), both diagonals, this corner's normal and the area.
struct RzLane {
  double x13, y13, x02, y02, Bx, By, area;
};
__device__ __forceinline__ RzLane rz_lane(int l, const double (&x)[4], const double (&y)[4]) {
  const bool odd = l & 1;
  const double xd = (odd ? x[0] : x[1]) - (odd ? x[2] : x[3]), yd = (odd ? y[0] : y[1]) - (odd ? y[2] : y[3]);
  const double xo = quad_other(xd), yo = quad_other(yd);
  RzLane r;
  r.x13 = odd ? xo : xd;
  r.y13 = odd ? yo : yd;
  r.x02 = odd ? xd : xo;
  r.y02 = odd ? yd : yo;
  r.Bx = flip(0.5 * yd, l == 1 || l == 2);
  r.By = flip(0.5 * xd, l == 0 || l == 3);
  r.area = 0.5 * mul_mul(r.x02, r.y13, -r.x13, r.y02);
  return r;
}

__global__ void __launch_bounds__(kRzLaneBlock) k_force_rz_lanes(const RzForceArgs a) {
  const int t = blockIdx.x * kRzLaneBlock + threadIdx.x;
  const int l = threadIdx.x & 3, ne = a.ne;
  const bool live = (t >> 2) < ne;
  const int e = live ? t >> 2 : ne - 1;
  const int n = __ldg(a.nie + 4 * (size_t)e + l);
  const int k0 = __ldg(a.eie_start + e), k1 = __ldg(a.eie_start + e + 1);
  previous_launch_done();
  if (!force_active(a) || (t & ~31) >= 4 * ne) return;  // whole warps past the end
  const double xl = a.x[n], yl = a.y[n], ul = a.u[n], vl = a.v[n];
  const double den = a.den[e], pres = a.pres[e], sspd = a.sspd[e], div = a.div[e];
  const double* q = a.qtab + 4 * a.mat[e];
  const bool compress = is_negative(div);
  const double qa = compress ? q[0] : q[1], qb = compress ? q[2] : q[3];
  long long kmin = 0x7FFFFFFFFFFFFFFFLL, kmax = (long long)0x8000000000000000ULL;
  for (int k = k0 + l; k < k1; k += 4) {
    const long long key = okey(a.div[__ldg(a.eie + k)]);
    kmin = key < kmin ? key : kmin;
    kmax = key > kmax ? key : kmax;
  }
  __syncwarp();
  kmin = quad_min(kmin);
  kmax = ~quad_min(~kmax);
  double x[4], y[4], u[4], v[4];
  quad_all(xl, x);
  quad_all(yl, y);
  quad_all(ul, u);
  quad_all(vl, v);
  const bool odd = l & 1;
  const RzLane g = rz_lane(l, x, y);
  // the centroid's offset, x in even lanes and y in odd ones
  const double m = -((odd ? y[0] : x[0]) - (odd ? y[1] : x[1])) - ((odd ? y[2] : x[2]) - (odd ? y[3] : x[3]));
  const double mo = quad_other(m);
  const bool hoop_zero =
      is_finite(pres) && rz_corner_areas_finite(g.x02, g.x13, g.y02, g.y13, odd ? mo : m, odd ? m : mo);
  double vs = 0.0;
#pragma unroll
  for (int k = 0; k < 4; ++k) vs = fma(0.25, odd ? v[k] : u[k], vs);
  const double vs0 = quad_lane(vs, 0), vs1 = quad_lane(vs, 1);
  const double bn = mode_sqrt(mul_mul(g.Bx, g.Bx, g.By, g.By));
  const double mu = rz_impedance(den, qa * sspd, qb, ul - vs0, vl - vs1) * bn;
  __syncwarp();
  double s = 0.0;
#if FIERRO_FMA
#pragma unroll
  for (int k = 0; k < 4; ++k) s = fma(quad_lane(mu, k), l == 0 ? u[k] : l == 1 ? v[k] : 1.0, s);
#else
  const double mu_u = mu * ul, mu_v = mu * vl;
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const double p0 = quad_lane(mu_u, k), p1 = quad_lane(mu_v, k), p2 = quad_lane(mu, k);
    s = s + (l == 0 ? p0 : l == 1 ? p1 : p2);
  }
#endif
  s = from_zero(s);
  const double s3 = quad_lane(s, 2);
  double vstar = 0.0;
  if (s3 > a.fuzz) {
#if FIERRO_FMA
    vstar = s * mode_rcp(s3);
#else
    vstar = quot(s, divisor(s3));
#endif
  }
  __syncwarp();
  const double vstar0 = quad_lane(vstar, 0), vstar1 = quad_lane(vstar, 1);
  const double phi = rz_mach_switch(g.area, div, sspd, a.fuzz) * (1.0 - at_least_0(rz_limiter_min(a, div, k0, k1, kmin, kmax)));
  const double pm = phi * mu, tau = 0.0 - pres;
  double f0, f1;
  if (hoop_zero) {
    f0 = rz_zero_terms(mul_mul(-g.Bx, tau, pm, vstar0 - ul), -g.By, yl);
    f1 = rz_zero_terms(mul_mul(-g.By, tau, pm, vstar1 - vl), -g.Bx, yl);
  } else {
    double ca[4];
    rz_corner_areas(x, y, ca);
    const double cl = l == 0 ? ca[0] : l == 1 ? ca[1] : l == 2 ? ca[2] : ca[3], z = 0.0;
    f0 = mul_add(mul_mul(-g.Bx, tau, -g.By, z), pm, vstar0 - ul);
    f1 = mul_add(mul_mul(-g.Bx, z, -g.By, tau), pm, vstar1 - vl);
    if (yl > 1e-14) {
      f0 = f0 + z * cl / yl;
      f1 = f1 + (tau - tau) * cl / yl;
    }
  }
  if (!live) return;
  a.force[(size_t)(l * 2 + 0) * ne + e] = f0;
  a.force[(size_t)(l * 2 + 1) * ne + e] = f1;
}

template <int KIND>
__global__ void __launch_bounds__(kRzLaneBlock) k_elem_rz_lanes(const RzElemArgs a) {
  const int t = blockIdx.x * kRzLaneBlock + threadIdx.x;
  const int lane = threadIdx.x & 31, l = lane & 3, ne = a.ne;
  const bool live = (t >> 2) < ne;
  const int e = live ? t >> 2 : ne - 1;
  const int n = __ldg(a.nie + 4 * (size_t)e + l);
  previous_launch_done();
  if ((KIND != 2 && !a.ctrl->active) || (t & ~31) >= 4 * ne) return;
  const double xl = a.x[n], yl = a.y[n], ul = a.u[n], vl = a.v[n];
  double F0 = 0.0, F1 = 0.0, hx = 0.0, hy = 0.0;
  if (KIND != 2) {
    const double r = a.rad[n];
    F0 = a.force[(size_t)(l * 2 + 0) * ne + e] * r;
    F1 = a.force[(size_t)(l * 2 + 1) * ne + e] * r;
    hx = a.hx[n];
    hy = a.hy[n];
  }
  const double mass = KIND != 2 ? a.mass[e] : 1.0, sie0 = KIND != 2 ? a.sie0[e] : 0.0;
  const double gamma = KIND != 2 ? a.gamma[e] : 0.0, csmin = KIND != 2 ? a.csmin[e] : 0.0;
  const bool odd = l & 1;
  double x[4], y[4];
  quad_all(xl, x);
  quad_all(yl, y);
  const RzLane g = rz_lane(l, x, y);
  // the volume's two terms (geometry.cpp:369-434), the first in even lanes: nodes
  // (p, q, r) = (2, 3, 0) and (0, 1, 2)
  const double xp = odd ? x[0] : x[2], xq = odd ? x[1] : x[3], xr = odd ? x[2] : x[0];
  const double yp = odd ? y[0] : y[2], yq = odd ? y[1] : y[3], yr = odd ? y[2] : y[0];
  const double S = yp + yq + yr, T = mul_mul(yp - yq, xr - xq, -(yr - yq), xp - xq);
  const double So = quad_other(S), To = quad_other(T);
  const double vol = (KIND == 2) ? a.vol[e] : sixth(mul_mul(odd ? So : S, odd ? To : T, odd ? S : So, odd ? T : To));
  // lane 0: the u sum, 1: the v sum (divergence), 2: the power, 3: the mean radial
  // velocity, corner by corner
  double uB[4], vB[4], uu[4], vv[4], acc = 0.0, pw = 0.0;
  quad_all(g.Bx, uB);
  quad_all(g.By, vB);
  quad_all(ul, uu);
  quad_all(vl, vv);
  {
    const bool first = l == 0;
    double b[4], w[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      b[k] = l == 3 ? 1.0 : first ? uB[k] : vB[k];
      w[k] = first ? uu[k] : vv[k];
    }
    acc = mul_add(mul_add(mul_mul(w[0], b[0], w[1], b[1]), w[2], b[2]), w[3], b[3]);
    if (KIND != 2) {
#if FIERRO_FMA
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        pw = fma(quad_lane(F0, k), quad_lane(hx, k), pw);
        pw = fma(quad_lane(F1, k), quad_lane(hy, k), pw);
      }
#else
      const double P0 = F0 * hx, P1 = F1 * hy;
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        pw = pw + quad_lane(P0, k);
        pw = pw + quad_lane(P1, k);
      }
#endif
    }
  }
  const double su = quad_lane(acc, 0), sv = quad_lane(acc, 1), vr = 0.25 * quad_lane(acc, 3);
  // four quotients at once: 1 / area, vol / area, dt / mass, mass / vol
  const double adt = KIND != 2 ? a.rk_alpha * a.ctrl->dt : 0.0;
  const double num = l == 0 ? 1.0 : l == 1 ? vol : l == 2 ? adt : mass;
  const double dvs = l < 2 ? g.area : l == 2 ? mass : vol;
  const double qt = newton_div(num, dvs);
  __syncwarp();
  const double inverse_area = quad_lane(qt, 0), mean_radius = quad_lane(qt, 1);
  const double div = from_zero(mul_add(mul_add(newton_div(vr, mean_radius), sv, inverse_area), su, inverse_area));
  __syncwarp();
  double sspd;
  const bool writer = live && l == 0;
  if (KIND != 2) {
    const double sie1 = mul_add(sie0, -quad_lane(qt, 2), from_zero(pw));
    const double den = quad_lane(qt, 3);
    const double pres = (gamma - 1.0) * sie1 * den;
    sspd = mode_sqrt(gamma * (gamma - 1.0) * sie1);
    if (sspd < csmin) sspd = csmin;
    if (writer) {
      a.sie1[e] = sie1;
      a.vol[e] = vol;
      a.den[e] = den;
      a.pres[e] = pres;
      a.sspd[e] = sspd;
      if (__double_as_longlong(vol) <= 0 || !is_finite(vol)) atomicOr(&a.ctrl->status, FIERRO_STATUS_BAD_VOLUME);
      if (!is_finite(sie1) || !is_finite(pres)) atomicOr(&a.ctrl->status, FIERRO_STATUS_BAD_STATE);
    }
  } else {
    sspd = a.sspd[e];
  }
  if (writer) a.div[e] = div;
  if (KIND != 0) {
    // the six pairs: each lane its edge to the next corner, then a diagonal
    const double ex = xl - (l == 0 ? x[1] : l == 1 ? x[2] : l == 2 ? x[3] : x[0]);
    const double ey = yl - (l == 0 ? y[1] : l == 1 ? y[2] : l == 2 ? y[3] : y[0]);
    const double dx = odd ? g.x13 : g.x02, dy = odd ? g.y13 : g.y02;
    const long long k1 = __double_as_longlong(mul_mul(ex, ex, ey, ey)) & kAbsMask;
    const long long k2 = __double_as_longlong(mul_mul(dx, dx, dy, dy)) & kAbsMask;
    __syncwarp();
    const long long kd = quad_min(k1 < k2 ? k1 : k2);
    long long dkey = 0x7FFFFFFFFFFFFFFFLL;
    if (live) dkey = rz_cfl_key(__longlong_as_double(kd), sspd, a.dt_cfl, a.fuzz);
    __syncwarp();
    for (int o = 16; o > 2; o >>= 1) {
      const long long tk = __shfl_xor_sync(0xFFFFFFFFu, dkey, o);
      dkey = tk < dkey ? tk : dkey;
    }
    if (lane == 0) a.cfl_part[t >> 5] = dkey;
  }
}

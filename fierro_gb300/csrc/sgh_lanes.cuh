// The force, node and element passes of small meshes: eight lanes per element
// (one per corner), one thread per node component.  Included in sgh_kernels.cu's
// implementation namespace; the results are those of the one-thread-per-element
// passes bit for bit, in both modes.
//
// Bound: a warp issues one FP64 instruction every ~65 clocks (GB300 has half an
// FP64 lane per clock and sub-partition, whatever the number of active lanes), so
// with at most one warp per sub-partition (608) a pass takes as long as one
// thread's chain: 458 instructions for an element's exact force, 15 us, however
// few elements there are.  Eight lanes cut the chain to the ~95 instructions one
// corner and the ordered sums take, at twice the total work, which such a mesh
// does not fill the chip with: a 12^3 cycle 102 -> 40.6 us exact, 78 -> 34.3 us FMA,
// 8^3 101 -> 37.3 and 78 -> 33.1 us.  Sums whose order is part of the result run in one
// lane over the corners' products in shared memory (different lanes summing
// different quantities in the same instructions); everything else is per corner.
#pragma once

#include "sgh_lane_tables.cuh"

// ---------------------------------------------------------------------------
// STRENGTH as in force_elem: each lane reads one stress component (lane 0 the
// ninth too), the velocity gradient's nine sums run in the eight lanes (one twice),
// and lane 0 runs the model.  TAPE as there: the viscosity intermediates, stored.
template <bool STRENGTH, bool TAPE>
__global__ void __launch_bounds__(kLaneBlock) k_force_lanes(const ForceArgs a) {
  // per element: the corners' velocities and impedance terms, rows u, v, w, mu
  __shared__ double s_v[kLaneWarps][kGroups][4][9];
  const int t = blockIdx.x * kLaneBlock + threadIdx.x;
  const int lane = threadIdx.x & 31, l = lane & 7, ne = a.ne;
  const bool live = (t >> 3) < ne;
  const int e = live ? t >> 3 : ne - 1;
  double(*sv)[9] = s_v[threadIdx.x >> 5][lane >> 3];
  const int n = __ldg(a.nie + 8 * (size_t)e + l);  // the mesh does not change: before the wait
  const int k0 = __ldg(a.eie_start + e), k1 = __ldg(a.eie_start + e + 1);
  previous_launch_done();
  if (!force_active(a) || (t & ~31) >= 8 * ne) return;  // whole warps past the end
  const double vu = a.u[n], vv = a.v[n], vw = a.w[n];
  const double b0 = a.bmat[(size_t)(l * 3 + 0) * ne + e];
  const double b1 = a.bmat[(size_t)(l * 3 + 1) * ne + e];
  const double b2 = a.bmat[(size_t)(l * 3 + 2) * ne + e];
  const double den = a.den[e], pres = a.pres[e], sspd = a.sspd[e], vol = a.vol[e], div = a.div[e];
  const double* q = a.qtab + 4 * a.mat[e];
  const bool compress = is_negative(div);
  const double qa = compress ? q[0] : q[1], qb = compress ? q[2] : q[3];
  // the limiter's neighbours, eight at a time
  long long kmin = 0x7FFFFFFFFFFFFFFFLL, kmax = (long long)0x8000000000000000ULL;
  for (int k = k0 + l; k < k1; k += 8) {
    const long long key = okey(a.div[__ldg(a.eie + k)]);
    kmin = key < kmin ? key : kmin;
    kmax = key > kmax ? key : kmax;
  }
  __syncwarp();
  kmin = group_min(kmin);
  kmax = ~group_min(~kmax);
  sv[0][l] = vu;
  sv[1][l] = vv;
  sv[2][l] = vw;
  __syncwarp();
  // lane r sums component r (lane 3: mu); the others repeat lane 3
  const int r = l < 3 ? l : 3, c = l < 3 ? l : 2;
  double vs = 0.0;
#pragma unroll
  for (int k = 0; k < 8; ++k) vs = fma(0.125, sv[c][k], vs);
  const double vs0 = from_lane(vs, 0), vs1 = from_lane(vs, 1), vs2 = from_lane(vs, 2);
  const Impedance z = impedance(den, sspd, qa, qb);
  double mag_vel;
  const double mu = corner_impedance(z, vu - vs0, vv - vs1, vw - vs2, b0, b1, b2, &mag_vel);
  __syncwarp();
#if FIERRO_FMA
  sv[3][l] = mu;
  __syncwarp();
  double s = 0.0;
#pragma unroll
  for (int k = 0; k < 8; ++k) s = fma(sv[3][k], l < 3 ? sv[c][k] : 1.0, s);
#else
  sv[0][l] = mu * vu;
  sv[1][l] = mu * vv;
  sv[2][l] = mu * vw;
  sv[3][l] = mu;
  __syncwarp();
  double s = 0.0;
#pragma unroll
  for (int k = 0; k < 8; ++k) s = s + sv[r][k];
#endif
  s = from_zero(s);  // a fused sum's first product may round to -0.0
  const double s3 = from_lane(s, 3);
  // the element's quotients in different lanes of the same instructions: the
  // Riemann velocity's (0-2), the limiter's (3), the Mach switch's (4 and on)
  const double D = div + a.small;
  const double dsel = okey_decode(__double_as_longlong(D) > 0 ? kmin : kmax);
  const double c_length = pow_third(vol), mach = 20.0 * (c_length * fabs(div));
  __syncwarp();
#if FIERRO_FMA
  const double num = l < 3 ? 1.0 : l == 3 ? 0.9 * (dsel + a.small) : mach;
#else
  const double num = l < 3 ? s : l == 3 ? 0.9 * (dsel + a.small) : mach;
#endif
  const double qt = newton_div(num, l < 3 ? s3 : l == 3 ? D : sspd + a.fuzz);
  __syncwarp();
  const double vstar = !(s3 > a.fuzz) ? 0.0 : FIERRO_FMA ? s * qt : qt;
  const double vstar0 = from_lane(vstar, 0), vstar1 = from_lane(vstar, 1), vstar2 = from_lane(vstar, 2);
  const double r_min = limiter_min(a, D, dsel, from_lane(qt, 3), k0, k1);
  const double phi0 = 1.0 - at_least_0(r_min);
  const double phi = at_most_1(from_lane(qt, 4)) * phi0;
  if (TAPE) {
    const double araw = from_lane(qt, 4);
    // the neighbour whose divergence set phi0 when the limiter is active: the first
    // that attains it
    int at = 0x7FFFFFFF;
    const long long ksel = __double_as_longlong(D) > 0 ? kmin : kmax;
    if (k1 > k0 && is_finite(D) && (__double_as_longlong(D) & kAbsMask) != 0 && is_finite(dsel) && r_min < 1.0 &&
        r_min > 0.0)
      for (int k = k0 + l; k < k1; k += 8)
        if (at == 0x7FFFFFFF && okey(a.div[__ldg(a.eie + k)]) == ksel) at = k;
    __syncwarp();
    for (int o = 4; o > 0; o >>= 1) at = min(at, __shfl_xor_sync(0xFFFFFFFFu, at, o));
    if (live) {
      double* t = a.tape + e;
      t[(size_t)l * ne] = mu;
      t[(size_t)(8 + l) * ne] = mag_vel;
      const double all = l == 0 ? vstar0 : l == 1 ? vstar1 : l == 2 ? vstar2 : l == 3 ? s3 : l == 4 ? phi0 : l == 5 ? araw
                         : l == 6 ? c_length : r_min;
      t[(size_t)(16 + l) * ne] = all;
      if (l == 0) a.tape_sel[e] = at == 0x7FFFFFFF ? -1 : __ldg(a.eie + at);
    }
  }
  const double pm = phi * mu;
  if constexpr (!STRENGTH) {
    if (!live) return;
    a.force[(size_t)(l * 3 + 0) * ne + e] = mul_mul(b0, pres, pm, vstar0 - vu);
    a.force[(size_t)(l * 3 + 1) * ne + e] = mul_mul(b1, pres, pm, vstar1 - vv);
    a.force[(size_t)(l * 3 + 2) * ne + e] = mul_mul(b2, pres, pm, vstar2 - vw);
  } else {
    // per element: stress(1), then the corners' velocities and normals and L
    __shared__ double s_t[kLaneWarps][kGroups][3 * 9 + 2 * 27 + 1];
    double* st = s_t[threadIdx.x >> 5][lane >> 3];
    double *tau = st, *L = st + 9, *sb = st + 27, *sw = st + 54;
    const double mine = a.stress_cur[(size_t)l * ne + e];
    const double ninth = l == 0 ? a.stress_cur[(size_t)8 * ne + e] : 0.0;
    tau[l] = (l & 3) == 0 ? mine - pres : mine;
    if (l == 0) tau[8] = ninth - pres;
    sb[l] = b0, sb[9 + l] = b1, sb[18 + l] = b2;
    sw[l] = vu, sw[9 + l] = vv, sw[18 + l] = vw;
    __syncwarp();
    const double vs[3] = {vstar0, vstar1, vstar2}, vl[3] = {vu, vv, vw};
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      const double f = mul_add(mul_add(mul_mul(-b0, tau[d], -b1, tau[3 + d]), -b2, tau[6 + d]), pm, vs[d] - vl[d]);
      if (live) a.force[(size_t)(l * 3 + d) * ne + e] = f;
    }
    const int mat = a.mat[e];
    const bool hypo = a.stype[mat] == 1;  // the same in an element's eight lanes
    const double inverse_vol = mode_rcp(vol);
    __syncwarp();
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const int k = i == 0 ? l : 8;
      const double *x = sw + 9 * (k / 3), *y = sb + 9 * (k % 3);
      double t = mul_mul(x[0], y[0], x[1], y[1]);
#pragma unroll
      for (int m = 2; m < 8; ++m) t = mul_add(t, x[m], y[m]);
      L[k] = FX_MUL(t, inverse_vol);
    }
    __syncwarp();
    if (!live) return;
    if (hypo) {
      if (l != 0) return;
      double sc[9], s0[9], G[9];
#pragma unroll
      for (int k = 0; k < 9; ++k) {
        sc[k] = a.stress_cur[(size_t)k * ne + e];
        s0[k] = a.stress0[(size_t)k * ne + e];
        G[k] = L[k];
      }
      user_strength_model(sc, s0, G, a.statev + e, ne, mat, den, a.sie0[e], vol, a.ctrl->dt, a.rk_alpha);
#pragma unroll
      for (int k = 0; k < 9; ++k) a.stress_out[(size_t)k * ne + e] = sc[k];
    } else if (a.copy_stress) {
      a.stress_out[(size_t)l * ne + e] = mine;
      if (l == 0) a.stress_out[(size_t)8 * ne + e] = ninth;
    }
  }
}

// ---------------------------------------------------------------------------
// One component of one node per thread (blockIdx.y the component).
__global__ void __launch_bounds__(kNodeBlock) k_node_lanes(const NodeArgs a) {
  const int n = blockIdx.x * blockDim.x + threadIdx.x, d = blockIdx.y;
  const bool in = n < a.nn;
  const int c0 = in ? __ldg(a.cin_start + n) : 0, c1 = in ? __ldg(a.cin_start + n + 1) : 0;
  previous_launch_done();
  if (!in || !a.ctrl->active) return;
  const size_t ne = (size_t)a.ne;
  double f = 0.0;
  for (int base = c0; base < c1; base += 8) {
    double g[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      const int cid = base + k < c1 ? __ldg(a.cin + base + k) : 0;
      g[k] = base + k < c1 ? a.force[(size_t)((cid & 7) * 3 + d) * ne + (cid >> 3)] : 0.0;
    }
#pragma unroll
    for (int k = 0; k < 8; ++k)
      if (base + k < c1) f = f + g[k];
  }
  const double adt = a.rk_alpha * a.ctrl->dt;
  const double v0 = (d == 0 ? a.u0 : d == 1 ? a.v0 : a.w0)[n];
#if FIERRO_FMA
  const double adt_rm = adt * (a.node_rm ? a.node_rm[n] : 1.0 / a.node_mass[n]);
  double v1 = fma(adt_rm, f, v0);
#else
  double v1 = v0 + quot(adt * f, divisor(a.node_mass[n]));
#endif
  if (a.bc_mask[n] & (1u << d)) v1 = 0.0;
  const double h = (v1 + v0) * 0.5;
  (d == 0 ? a.u1 : d == 1 ? a.v1 : a.w1)[n] = v1;
  (d == 0 ? a.hx : d == 1 ? a.hy : a.hz)[n] = h;
  (d == 0 ? a.x1 : d == 1 ? a.y1 : a.z1)[n] = mul_add((d == 0 ? a.x0 : d == 1 ? a.y0 : a.z0)[n], adt, h);
}

// ---------------------------------------------------------------------------
// Element update (KIND as in elem_tile), one CFL partial per warp.  Shared memory
// per element, doubles: coordinates x, y, z by node; the 18 combos of each
// component; the ordered sums' terms -- power (24), the velocity sums (8 each),
// the volume (8) -- as products (exact) or factor pairs (FMA).
constexpr int kChain = 24 + 4 * 8;
struct LaneElem {
  double x[3][8];
  double combo[3][18];
  double pr[8][7];  // a lane's products of the first component
  double p[kChain];
#if FIERRO_FMA
  double q[kChain];
#endif
  float f[3][8];
  double pad;
};

template <int KIND>
__global__ void __launch_bounds__(kLaneBlock) k_elem_lanes(const ElemArgs a) {
  __shared__ LaneElem s_e[kLaneWarps][kGroups];
  const int t = blockIdx.x * kLaneBlock + threadIdx.x;
  const int lane = threadIdx.x & 31, l = lane & 7, ne = a.ne;
  const bool live = (t >> 3) < ne;
  const int e = live ? t >> 3 : ne - 1;
  LaneElem& s = s_e[threadIdx.x >> 5][lane >> 3];
  const int n = __ldg(a.nie + 8 * (size_t)e + l);
  previous_launch_done();
  if ((KIND != 2 && !a.ctrl->active) || (t & ~31) >= 8 * ne) return;
  const double x[3] = {a.x[n], a.y[n], a.z[n]};
  const double v[3] = {a.u[n], a.v[n], a.w[n]};
  double fc[3] = {0.0, 0.0, 0.0}, h[3] = {0.0, 0.0, 0.0};
  if (KIND != 2) {
#pragma unroll
    for (int d = 0; d < 3; ++d) fc[d] = a.force[(size_t)(l * 3 + d) * ne + e];
    h[0] = a.hx[n];
    h[1] = a.hy[n];
    h[2] = a.hz[n];
  }
  const double mass = KIND != 2 ? a.mass[e] : 1.0, sie0 = KIND != 2 ? a.sie0[e] : 0.0;
  const double gamma = KIND != 2 ? a.gamma[e] : 0.0, csmin = KIND != 2 ? a.csmin[e] : 0.0;
#pragma unroll
  for (int d = 0; d < 3; ++d) s.x[d][l] = x[d];
  __syncwarp();
  // the combos: 36 two-term and 18 four-term ones over eight lanes
#pragma unroll
  for (int i = 0; i < 5; ++i) {
    const int task = l + 8 * i;
    if (task < 36) {
      const int c = task / 12, m = task - 12 * c;
      const double* I = s.x[c == 0 ? 2 : c - 1];
      const unsigned w = (unsigned)(m < 10 ? kLane.two[0] >> (6 * m) : kLane.two[1] >> (6 * (m - 10)));
      s.combo[c][m] = I[w & 7] - I[(w >> 3) & 7];
    }
  }
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    const int task = l + 8 * i;
    if (task < 18) {
      const int c = task / 6, m = task - 6 * c;
      const double* I = s.x[c == 0 ? 2 : c - 1];
      const unsigned w = (unsigned)(m < 4 ? kLane.four[0] >> (16 * m) : kLane.four[1] >> (16 * (m - 4)));
      double v4 = flip(I[w & 7], (w >> 3) & 1);
#pragma unroll
      for (int k = 1; k < 4; ++k) v4 = v4 + flip(I[(w >> (4 * k)) & 7], (w >> (4 * k + 3)) & 1);
      s.combo[c][12 + m] = v4;
    }
  }
  __syncwarp();
  // this corner's normals
  const double twelth = 1. / 12.;
  const unsigned long long row = by_lane(l, kLane.row[0], kLane.row[1], kLane.row[2], kLane.row[3], kLane.row[4],
                                         kLane.row[5], kLane.row[6], kLane.row[7]);
  const unsigned vorder = (unsigned)by_lane(l, kLane.vol[0], kLane.vol[1], kLane.vol[2], kLane.vol[3], kLane.vol[4],
                                            kLane.vol[5], kLane.vol[6], kLane.vol[7]);
  double b[3];
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    const double* O = s.x[c == 2 ? 0 : c + 1];
    double o[6], cm[6];
#pragma unroll
    for (int k = 0; k < 6; ++k) {
      const unsigned w = (unsigned)(row >> (9 * k));
      o[k] = O[w & 7];
      cm[k] = flip(s.combo[c][(w >> 3) & 31], (w >> 8) & 1);
    }
    double sum;
    if (c == 0) {
      double pr[6];
#pragma unroll
      for (int k = 0; k < 6; ++k) s.pr[l][k] = pr[k] = FX_MUL(o[k], cm[k]);
      sum = ((((pr[0] + pr[1]) + pr[2]) + pr[3]) + pr[4]) + pr[5];
      double sv = s.pr[l][vorder & 7];
#pragma unroll
      for (int k = 1; k < 6; ++k) sv = FX_ADD(sv, s.pr[l][(vorder >> (3 * k)) & 7]);
      const int at = 48 + (int)(vorder >> 18);
      s.p[at] = FX_MUL(x[0], sv);
#if FIERRO_FMA
      s.q[at] = 1.0;
#endif
    } else {
      sum = mul_mul(o[0], cm[0], o[1], cm[1]);
#pragma unroll
      for (int k = 2; k < 6; ++k) sum = mul_add(sum, o[k], cm[k]);
    }
    b[c] = sum * twelth;
    if (live) a.bmat[(size_t)(l * 3 + c) * ne + e] = b[c];
    // terms of the velocity sums and the power, in the sums' order (the fused sums
    // begin with the second corner's product, as mul_mul does)
#if FIERRO_FMA
    const int at = 24 + 8 * c + (l < 2 ? 1 - l : l);
    s.p[at] = v[c];
    s.q[at] = b[c];
    s.p[3 * l + c] = fc[c];
    s.q[3 * l + c] = h[c];
#else
    s.p[24 + 8 * c + l] = v[c] * b[c];
    s.p[3 * l + c] = fc[c] * h[c];
#endif
  }
  __syncwarp();
  // lanes 0-2: the velocity sums; 3: the volume; 4: the power (24 terms); the rest repeat the volume
  double acc = 0.0;
  const int at = l < 3 ? 24 + 8 * l : l == 4 ? 0 : 48;
#pragma unroll
  for (int k = 0; k < 8; ++k) {
#if FIERRO_FMA
    acc = fma(s.p[at + k], s.q[at + k], acc);
#else
    acc = acc + s.p[at + k];
#endif
  }
  if (KIND != 2) {
    double pw = acc;
#pragma unroll
    for (int k = 8; k < 24; ++k) {
#if FIERRO_FMA
      pw = fma(s.p[k], s.q[k], pw);
#else
      pw = pw + s.p[k];
#endif
    }
    if (l == 4) acc = pw;
  }
  const double Sx = from_lane(acc, 0), Sy = from_lane(acc, 1), Sz = from_lane(acc, 2);
  const double vol_geo = FX_MUL(from_lane(acc, 3), twelth);
  const double power = from_zero(from_lane(acc, 4));
  const double vol = (KIND == 2) ? a.vol[e] : vol_geo;
  // three quotients at once: 1 / vol, dt / mass, mass / vol
  const double adt = KIND != 2 ? a.rk_alpha * a.ctrl->dt : 0.0;
  const double qt = newton_div(l == 0 ? 1.0 : l == 1 ? adt : mass, l == 1 ? mass : vol);
  __syncwarp();
  const double div = divergence(Sx, Sy, Sz, from_lane(qt, 0));
  double sspd;
  const bool writer = live && l == 0;
  if (KIND != 2) {
    const double sie1 = sie0 - FX_MUL(from_lane(qt, 1), power);
    const double den = from_lane(qt, 2);
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
    // the CFL length: each lane screens every eighth of the 28 pairs in single
    // precision (sgh_cfl.cuh's bound) and evaluates the ones left in FP64
    bool ok = true;
    float M = 0.0f;
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      const float im = cfl::image(x[d], ok);
      s.f[d][l] = im;
      M = fmaxf(M, fabsf(im));
    }
    __syncwarp();
    for (int o = 4; o > 0; o >>= 1) M = fmaxf(M, __shfl_xor_sync(0xFFFFFFFFu, M, o));
    const unsigned bad = __ballot_sync(0xFFFFFFFFu, !ok) >> (lane & 24) & 0xFFu;
    const bool screen = bad == 0 && M >= 9.5367431640625e-07f;
    float e2[4], e2min = 3.0e38f;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int k = l + 8 * i;
      const int pa = cfl::pair_a(k < 28 ? k : l), pb = cfl::pair_b(k < 28 ? k : l);
      const float dx = s.f[0][pb] - s.f[0][pa], dy = s.f[1][pb] - s.f[1][pa], dz = s.f[2][pb] - s.f[2][pa];
      e2[i] = (dx * dx + dy * dy) + dz * dz;
      e2min = fminf(e2min, e2[i]);
    }
    for (int o = 4; o > 0; o >>= 1) e2min = fminf(e2min, __shfl_xor_sync(0xFFFFFFFFu, e2min, o));
    const float T2 = cfl::screen_limit(e2min, M);
    unsigned mask = 0;
#pragma unroll
    for (int i = 0; i < 4; ++i)
      if (l + 8 * i < 28 && (!screen || e2[i] <= T2)) mask |= 1u << i;
    long long kd = 0x7FFFFFFFFFFFFFFFLL;
    while (mask) {
      const int k = l + 8 * (__ffs((int)mask) - 1);
      mask &= mask - 1;
      const long long key = cfl::key_of(cfl::exact_d2(s.x[0], s.x[1], s.x[2], cfl::pair_a(k), cfl::pair_b(k)));
      kd = key < kd ? key : kd;
    }
    __syncwarp();
    kd = group_min(kd);
    long long dkey = 0x7FFFFFFFFFFFFFFFLL;
    if (live) dkey = cfl_key(cfl::key_decode(kd), sspd, a.dt_cfl, a.fuzz);
    __syncwarp();
    for (int o = 16; o > 4; o >>= 1) {
      const long long tk = __shfl_xor_sync(0xFFFFFFFFu, dkey, o);
      dkey = tk < dkey ? tk : dkey;
    }
    if (lane == 0) a.cfl_part[t >> 5] = dkey;
  }
}

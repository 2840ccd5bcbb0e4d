// The reverse element and force passes of small meshes: eight lanes per element,
// for the reason sgh_lanes.cuh gives (a one-thread pass takes its 500 to 800 FP64
// instructions times 65 clocks however small the mesh).  Included in
// sgh_adjoint.cu's implementation namespace.  The element's sums are butterflies
// over its eight lanes (fixed order; the reverse arithmetic has no parity target).
#pragma once

__device__ __forceinline__ double sum8(double v) {
  for (int o = 1; o < 8; o <<= 1) v += __shfl_xor_sync(0xFFFFFFFFu, v, o);
  return v;
}

// k_adj_elem, a corner per lane: the lane's corner-normal adjoints reach the
// coordinates through the 18 shared combos of each component (sgh_lane_tables.cuh).
struct LaneAdj {
  double x[3][8], g[3][8], combo[3][18], w[3][18];
  double pad;
};
template <int KIND>
__global__ void __launch_bounds__(kLaneBlock) k_adj_elem_lanes(const AdjMesh m, const AdjBufs b, const Slot s1,
                                                                const double* __restrict__ force,
                                                                const AdjRecord* __restrict__ r, double alpha,
                                                                const double* __restrict__ sie_in,
                                                                double* __restrict__ sie_c, int assign,
                                                                double* __restrict__ part) {
  __shared__ LaneAdj s_a[kLaneWarps][kGroups];
  const int t = blockIdx.x * kLaneBlock + threadIdx.x;
  const int lane = threadIdx.x & 31, l = lane & 7, ne = m.ne;
  const bool live = (t >> 3) < ne;  // the others repeat the last element and store nothing
  const int e = live ? t >> 3 : ne - 1;
  LaneAdj& s = s_a[threadIdx.x >> 5][lane >> 3];
  const int n = __ldg(m.nie + 8 * (size_t)e + l);
  double dn = 0.0;
  for (int k = m.eie_start[e] + l; k < m.eie_start[e + 1]; k += 8) {
    const int nb = __ldg(m.eie + k);
    if (b.nbc[nb] == e) dn += b.nbv[nb];
  }
  __syncwarp();
  const double divb = b.divbar[e] + sum8(dn);
  const double vol = s1.vol[e], iv = fast_rcp(vol), sb = divb * iv;
  const double vel[3] = {s1.u[n], s1.v[n], s1.w[n]};
  const double x[3] = {s1.x[n], s1.y[n], s1.z[n]};
  double bp[3], S = 0.0;
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    const size_t idx = (size_t)(l * 3 + c) * ne + e;
    bp[c] = s1.bmat[idx];
    S = fma(vel[c], bp[c], S);
    s.g[c][l] = fma(sb, vel[c], b.bbar[idx]) * (1. / 12.);
    s.x[c][l] = x[c];
    if (live) b.cv[idx] = fma(sb, bp[c], b.cv[idx]);
  }
  const double volb = fma(-divb * sum8(S), iv * iv, b.volbar[e]);
  const double vw = (KIND == 0) ? volb : 0.0;  // dV/dx_p = B_p
  double xb[3] = {bp[0] * vw, bp[1] * vw, bp[2] * vw};
  __syncwarp();
#pragma unroll
  for (int i = 0; i < 5; ++i) {
    const int task = l + 8 * i;
    if (task < 36) {
      const int c = task / 12, k = task - 12 * c;
      const double* I = s.x[c == 0 ? 2 : c - 1];
      const unsigned w = (unsigned)(k < 10 ? kLane.two[0] >> (6 * k) : kLane.two[1] >> (6 * (k - 10)));
      s.combo[c][k] = I[w & 7] - I[(w >> 3) & 7];
      const double *O = s.x[c == 2 ? 0 : c + 1], *g = s.g[c];
      const unsigned q = (unsigned)(k < 9 ? kLane.pair2[0] >> (7 * k) : kLane.pair2[1] >> (7 * (k - 9)));
      const int p = q & 7, j = (q >> 3) & 7;
      s.w[c][k] = flip(fma(g[p], O[j], -(g[j] * O[p])), (q >> 6) & 1);
    }
  }
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    const int task = l + 8 * i;
    if (task < 18) {
      const int c = task / 6, k = task - 6 * c;
      const double* I = s.x[c == 0 ? 2 : c - 1];
      const unsigned w = (unsigned)(k < 4 ? kLane.four[0] >> (16 * k) : kLane.four[1] >> (16 * (k - 4)));
      double v4 = flip(I[w & 7], (w >> 3) & 1);
#pragma unroll
      for (int h = 1; h < 4; ++h) v4 = v4 + flip(I[(w >> (4 * h)) & 7], (w >> (4 * h + 3)) & 1);
      s.combo[c][12 + k] = v4;
      const double *O = s.x[c == 2 ? 0 : c + 1], *g = s.g[c];
      const unsigned q = (unsigned)(k < 4 ? kLane.pair4[0] >> (14 * k) : kLane.pair4[1] >> (14 * (k - 4)));
      double wk = 0.0;
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const unsigned qh = q >> (7 * h);
        const int p = qh & 7, j = (qh >> 3) & 7;
        wk += flip(fma(g[p], O[j], -(g[j] * O[p])), (qh >> 6) & 1);
      }
      s.w[c][12 + k] = wk;
    }
  }
  __syncwarp();
  const unsigned long long row = by_lane(l, kLane.row[0], kLane.row[1], kLane.row[2], kLane.row[3], kLane.row[4],
                                         kLane.row[5], kLane.row[6], kLane.row[7]);
  const unsigned long long terms = by_lane(l, kLane.terms[0], kLane.terms[1], kLane.terms[2], kLane.terms[3],
                                           kLane.terms[4], kLane.terms[5], kLane.terms[6], kLane.terms[7]);
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    double &ob = xb[c == 2 ? 0 : c + 1], &ib = xb[c == 0 ? 2 : c - 1];
#pragma unroll
    for (int k = 0; k < 6; ++k) {
      const unsigned w = (unsigned)(row >> (9 * k));
      ob = fma(-s.g[c][w & 7], flip(s.combo[c][(w >> 3) & 31], (w >> 8) & 1), ob);  // comb(j, p) = -comb(p, j)
      const unsigned q = (unsigned)(terms >> (6 * k));
      ib += flip(s.w[c][q & 31], (q >> 5) & 1);
    }
  }
  if (live)
#pragma unroll
    for (int c = 0; c < 3; ++c) b.cx[(size_t)(l * 3 + c) * ne + e] = xb[c];
  if (KIND == 0) {
    double pw = 0.0;
    pw = fma(force[(size_t)(l * 3 + 0) * ne + e], s1.hx[n],
             fma(force[(size_t)(l * 3 + 1) * ne + e], s1.hy[n], force[(size_t)(l * 3 + 2) * ne + e] * s1.hz[n]));
    const double power = sum8(pw), sieb = sie_in[e];
    const double adt = alpha * r->dt, iM = sieb * fast_rcp(m.elem_mass[e]);
    double adtb = 0.0;
    if (live && l == 0) {
      if (assign) sie_c[e] = sieb;
      else sie_c[e] += sieb;
      b.w[e] = -adt * iM;
      adtb = -power * iM;
    }
    const double total = block_sum(adtb);
    if (threadIdx.x == 0) part[blockIdx.x] = total;
  }
}

// k_adj_force, a corner per lane.
__global__ void __launch_bounds__(kLaneBlock) k_adj_force_lanes(const AdjMesh m, const AdjBufs b, const Slot s0,
                                                                const Slot s1, const double* __restrict__ force_tape,
                                                                const double* __restrict__ ft,
                                                                const int* __restrict__ fsel, double fuzz,
                                                                double small, double* __restrict__ sie_out,
                                                                int accumulate) {
  __shared__ double s_v[kLaneWarps][kGroups][3][9];
  const int th = blockIdx.x * kLaneBlock + threadIdx.x;
  const int lane = threadIdx.x & 31, l = lane & 7, ne = m.ne;
  if ((th & ~31) >= 8 * ne) return;  // whole warps past the end
  const bool live = (th >> 3) < ne;
  const int e = live ? th >> 3 : ne - 1;
  double(*sv)[9] = s_v[threadIdx.x >> 5][lane >> 3];
  const int n = __ldg(m.nie + 8 * (size_t)e + l);
  const double v[3] = {s0.u[n], s0.v[n], s0.w[n]};
  const double den = s0.den[e], pres = s0.pres[e], sspd = s0.sspd[e], vol = s0.vol[e], div = s0.div[e];
  const double* q = m.qtab + 4 * m.mat[e];
  const bool compress = div < 0;
  const double qa = compress ? q[0] : q[1], qb = compress ? q[2] : q[3];
  const double* t = ft + e;
  const double mu = t[(size_t)l * ne], mv = t[(size_t)(8 + l) * ne];
  const double vstar[3] = {t[(size_t)16 * ne], t[(size_t)17 * ne], t[(size_t)18 * ne]};
  const double s3 = t[(size_t)19 * ne], phi0 = t[(size_t)20 * ne], araw = t[(size_t)21 * ne];
  const double c_length = t[(size_t)22 * ne], r_min = t[(size_t)23 * ne];
  const int sel = fsel[e];
  const double we = b.w[e];
  const double h[3] = {s1.hx[n], s1.hy[n], s1.hz[n]};
  double B[3], F[3];
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    B[c] = s0.bmat[(size_t)(l * 3 + c) * ne + e];
    F[c] = fma(we, h[c], b.fbar[c][n]);
    sv[c][l] = v[c];
  }
  __syncwarp();
  // the average velocity in the forward's order, component c in lane c
  double va = 0.0;
#pragma unroll
  for (int k = 0; k < 8; ++k) va = fma(0.125, sv[l < 3 ? l : 2][k], va);
  const double avg[3] = {from_lane(va, 0), from_lane(va, 1), from_lane(va, 2)};
  const double alpha = fmin(1.0, araw), phi = alpha * phi0, pm = phi * mu;
  if (b.mismatch) {
    unsigned bad = 0;
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      const double f = B[c] * pres + pm * (vstar[c] - v[c]);
      bad += (__double_as_longlong(f) != __double_as_longlong(force_tape[(size_t)(l * 3 + c) * ne + e])) ? 1u : 0u;
    }
    if (bad && live) atomicAdd(b.mismatch, (unsigned long long)bad);
  }
  __syncwarp();
  // pass 1: the pressure, phi and v* adjoints, sums over the corners
  const double g = fma(F[0], vstar[0] - v[0], fma(F[1], vstar[1] - v[1], F[2] * (vstar[2] - v[2])));
  const double presb = sum8(fma(F[0], B[0], fma(F[1], B[1], F[2] * B[2])));
  const double phib = sum8(mu * g);
  double pf[3], vsb[3];
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    pf[c] = pm * F[c];
    vsb[c] = sum8(pf[c]);
  }
  const double alphab = phib * phi0, phi0b = phib * alpha;
  double divb = 0.0, sspdb = 0.0, volb = 0.0;
  if (araw < 1.0) {
    const double inv = fast_rcp(sspd + fuzz);
    const double sg = div > 0.0 ? 1.0 : (div < 0.0 ? -1.0 : 0.0);
    const double a20 = 20.0 * alphab * inv;
    divb = a20 * c_length * sg;
    sspdb = -alphab * alpha * inv;
    volb = a20 * fabs(div) * c_length * fast_rcp(3.0 * vol);
  }
  int nbc = -1;
  double nbv = 0.0;
  if (sel >= 0) {
    const double rbD = -phi0b * fast_rcp(div + small);  // phi0 = 1 - r_face
    nbv = 0.9 * rbD;
    nbc = sel;
    divb = fma(-rbD, r_min, divb);
  }
  double sb[3] = {0.0, 0.0, 0.0}, s3b = 0.0;
  if (s3 > fuzz) {
    const double is3 = fast_rcp(s3);
    sb[0] = vsb[0] * is3;
    sb[1] = vsb[1] * is3;
    sb[2] = vsb[2] * is3;
    s3b = -fma(vsb[0], vstar[0], fma(vsb[1], vstar[1], vsb[2] * vstar[2])) * is3;
  }
  // pass 2: this corner's velocity (viscous term, v*, |v - v_avg|) and |B|
  const double mub = fma(sb[0], v[0], fma(sb[1], v[1], fma(sb[2], v[2], phi * g + s3b)));
  const double qB = fma(B[0], B[0], fma(B[1], B[1], B[2] * B[2]));
  const double rB = fast_rsqrt(qB);
  const double qm = fma(qb, mv, qa * sspd);
  const double mucb = mub * (qB * rB);
  const double tb = mub * den * qm * rB;  // d mu / d B = muc B / |B|
  const double sm = mv > 0.0 ? mucb * (den * qb) * fast_rcp(mv) : 0.0;  // mv = |v - v_avg|
  __syncwarp();
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    const double sd = sm * (v[c] - avg[c]);
    const double vb = fma(mu, sb[c], sd - pf[c]);
    const double cv = fma(-0.125, sum8(sd), vb);  // the average's adjoint reaches every corner equally
    const size_t i = (size_t)(l * 3 + c) * ne + e;
    if (live) {
      b.bbar[i] = fma(tb, B[c], F[c] * pres);
      b.cv[i] = cv;
    }
  }
  double denb = sum8(mucb * qm);
  sspdb = fma(sum8(mucb) * den, qa, sspdb);
  if (!live || l != 0) return;
  double sieb = 0.0, gb = 0.0;
  eos_fold(den, s0.sie[e], m.gamma[e], m.csmin[e], presb, sspdb, sieb, denb, gb);
  volb -= denb * den * fast_rcp(vol);  // den = M / vol
  b.volbar[e] = volb;
  b.divbar[e] = divb;
  b.nbc[e] = nbc;
  b.nbv[e] = nbv;
  if (accumulate) sie_out[e] += sieb;
  else sie_out[e] = sieb;
  b.gbar[e] += gb;
}

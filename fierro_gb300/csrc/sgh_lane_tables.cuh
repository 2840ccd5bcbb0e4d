// What the lane passes share (sgh_lanes.cuh forward, sgh_adjoint_lanes.cuh
// reverse): eight lanes per element, one per corner.  Included inside each unit's
// implementation namespace.
#pragma once

// ---------------------------------------------------------------------------
// The hex cofactor tables (sgh_hex.h), rearranged per lane.  two[m] = (i, j): the
// combo I[i] - I[j]; four[m]: signed 1-based terms summed left to right; a lane's
// row: for each of its six products the O node (3 bits), the combo (5 bits: 0-11
// two-term, 12-17 four-term) and its sign (1 bit); vol: the volume's order of the
// six products (3 bits each) and the node's place in the volume's sum (3 bits).
// For the adjoint: of each combo the node pairs (p, j) that share it, with the sign
// it enters B(p) with (two-term: one pair, 7 bits; four-term: two); of each node the
// six combos it is a term of, 5 bits each, and its sign there (1 bit).
struct LaneTables {
  unsigned long long two[2], four[2], row[8];
  unsigned vol[8];
  unsigned long long pair2[2], pair4[2], terms[8];
};
constexpr LaneTables make_lane_tables() {
  LaneTables r{};
  signed char uniq[18][4] = {};
  int n2 = 0, n4 = 0;
  for (int pass = 0; pass < 2; ++pass)
    for (int p = 0; p < 8; ++p)
      for (int t = 0; t < 6; ++t) {
        const signed char* T = hex::TERMS[p][t];
        const bool is4 = T[2] != 0;
        if (is4 != (pass == 1) || hex::J[p][t] < p) continue;
        bool known = false;
        const int lo = is4 ? 12 : 0, hi = is4 ? 12 + n4 : n2;
        for (int k = lo; k < hi; ++k) {
          bool same = true, neg = true;
          for (int q = 0; q < 4; ++q) {
            if (uniq[k][q] != T[q]) same = false;
            if (uniq[k][q] != -T[q]) neg = false;
          }
          if (same || neg) known = true;
        }
        if (known) continue;
        const int at = is4 ? 12 + n4++ : n2++;
        for (int q = 0; q < 4; ++q) uniq[at][q] = T[q];
      }
  for (int k = 0; k < 12; ++k) {
    const int i = (uniq[k][0] > 0 ? uniq[k][0] : uniq[k][1]) - 1, j = -(uniq[k][0] > 0 ? uniq[k][1] : uniq[k][0]) - 1;
    r.two[k / 10] |= (unsigned long long)(i | (j << 3)) << (6 * (k % 10));
  }
  for (int k = 0; k < 6; ++k) {
    unsigned long long w = 0;
    for (int q = 0; q < 4; ++q) {
      const int v = uniq[12 + k][q];
      w |= (unsigned long long)(((v > 0 ? v : -v) - 1) | (v < 0 ? 8 : 0)) << (4 * q);
    }
    r.four[k / 4] |= w << (16 * (k % 4));
  }
  for (int p = 0; p < 8; ++p) {
    for (int t = 0; t < 6; ++t) {
      const signed char* T = hex::TERMS[p][t];
      const int lo = T[2] != 0 ? 12 : 0, hi = T[2] != 0 ? 18 : 12;
      for (int k = lo; k < hi; ++k) {
        bool same = true, neg = true;
        for (int q = 0; q < 4; ++q) {
          if (uniq[k][q] != T[q]) same = false;
          if (uniq[k][q] != -T[q]) neg = false;
        }
        // a two-term combo is kept as (positive) - (negative): -a + b is b - a
        if (same || neg) r.row[p] |= (unsigned long long)(hex::J[p][t] | (k << 3) | (neg ? 256 : 0)) << (9 * t);
      }
    }
    for (int a = 0; a < 8; ++a)
      if (hex::VI[a] == p) {
        for (int b = 0; b < 6; ++b) r.vol[p] |= (unsigned)hex::slot(p, hex::VJ[a][b]) << (3 * b);
        r.vol[p] |= (unsigned)a << 18;
      }
  }
  for (int k = 0; k < 18; ++k) {
    unsigned long long w = 0;
    int n = 0;
    for (int p = 0; p < 8; ++p)
      for (int t = 0; t < 6; ++t) {
        const int j = hex::J[p][t];
        if (j < p || (int)((r.row[p] >> (9 * t + 3)) & 31) != k) continue;
        w |= (unsigned long long)(p | (j << 3) | ((r.row[p] >> (9 * t + 8)) & 1 ? 64 : 0)) << (7 * n++);
      }
    if (k < 12) r.pair2[k / 9] |= w << (7 * (k % 9));
    else r.pair4[(k - 12) / 4] |= w << (14 * ((k - 12) % 4));
  }
  for (int p = 0; p < 8; ++p) {
    int n = 0;
    for (int k = 0; k < 18; ++k)
      for (int q = 0; q < 4; ++q) {
        // two-term combos are (positive) - (negative), four-term ones as they stand
        const int v = uniq[k][q];
        if ((v > 0 ? v : -v) != p + 1) continue;
        r.terms[p] |= (unsigned long long)(k | (v < 0 ? 32 : 0)) << (6 * n++);
      }
  }
  return r;
}
constexpr LaneTables kLane = make_lane_tables();

// One of eight constants by lane, by selects (no memory access).
__device__ __forceinline__ unsigned long long by_lane(int l, unsigned long long a, unsigned long long b,
                                                      unsigned long long c, unsigned long long d, unsigned long long e,
                                                      unsigned long long f, unsigned long long g,
                                                      unsigned long long h) {
  const unsigned long long ab = l & 1 ? b : a, cd = l & 1 ? d : c, ef = l & 1 ? f : e, gh = l & 1 ? h : g;
  const unsigned long long lo = l & 2 ? cd : ab, hi = l & 2 ? gh : ef;
  return l & 4 ? hi : lo;
}
__device__ __forceinline__ double flip(double v, unsigned neg) {
  return __hiloint2double(__double2hiint(v) ^ (int)(neg << 31), __double2loint(v));
}
// Value of the first lane of each group of eight, or of its lane `src`.
__device__ __forceinline__ double from_lane(double v, int src) { return __shfl_sync(0xFFFFFFFFu, v, src, 8); }
__device__ __forceinline__ long long group_min(long long k) {
  for (int o = 4; o > 0; o >>= 1) {
    const long long t = __shfl_xor_sync(0xFFFFFFFFu, k, o);
    k = t < k ? t : k;
  }
  return k;
}

constexpr int kLaneBlock = 64;               // threads: two warps, eight elements
constexpr int kLaneWarps = kLaneBlock / 32;
constexpr int kGroups = 4;                   // elements per warp


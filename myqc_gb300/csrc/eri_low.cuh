// eri_low.cuh -- the contracted quartets of at most 64 integrals, (ss|ss),
// (sp s|ss), (sp s|sp s), (sp sp|ss) and (sp sp|sp s), in FP64 with early
// contraction (included by eri_impl.cuh).
//
// With A and C the first centres of the two pairs, AB = B - A, CD = D - C,
// AC = A - C, beta = b/p and delta = d/q, the vectors of the McMurchie-Davidson
// formula are
//     P - A = beta AB,  P - B = (beta - 1) AB,  P - Q = AC + beta AB - delta CD,
// so a contracted integral is a polynomial in the components of AB, AC and CD,
// which all primitive quartets share, whose coefficients are sums over the
// primitive quartets of products of beta, delta, 1/p, 1/q and
//     G_m = theta alpha^m F_m(T),  m = 0 .. 3.
// Only those sums are formed per primitive quartet (1, 4, 17, 16 and 73 of them), as
// Pople and Hehre's and the PRISM schemes contract before they build angular
// momentum; the vectors enter once per contracted quartet.  alpha and theta
// depend on the two exponent sums alone and come from a table (basis.cu), the
// products of contraction coefficients, beta and H = -1/p from one record per
// primitive pair, the Boys values from boys_fine.  The factors -2 of
// R_tuv's (-2 alpha)^n are taken into H: h R_1 = H (P - Q) G1,
// h^2 R_2 = H^2 (P - Q)(P - Q) G2 - H^2 G1 / 2 on the diagonal.
//
// Bound by FP64 issue (two multiply-adds per clock and SM).  FP64 instructions
// per primitive quartet with T < 36, this scheme against every component per
// primitive quartet: (ss|ss) 17 / 42, (sp s|ss) 31 / 64, (sp s|sp s) 72 / 140,
// (sp sp|ss) 65 / 146, (sp sp|sp s) 240 (in two threads) / 750.
//
// Record of a primitive pair (PP_REC doubles; c = contraction coefficients
// times K):
//   0-2 P   3 beta   4 K   5 1e-14 / K   6 c_ss
//   7 c_ps beta   8 c_ps H   9 c_sp (beta - 1)   10 c_sp H
//   11 c_pp beta (beta - 1)   12 c_pp H   13 H
#pragma once

namespace mq {

template <int LA, int LB, int LC, int LD, int EPI>
__device__ __forceinline__ void quartet_low(const EriArgs &g, int P, int Q, size_t n, double *XXout) {
  constexpr int CP = LA + LB, CQ = LC + LD, LT = CP + CQ;
  constexpr int NA = nfun(LA), NB = nfun(LB), NC = nfun(LC), ND = nfun(LD);
  static_assert((CP <= 1 && CQ <= CP) || (CP == 2 && CQ == 0), "low-order classes");
  constexpr int NSUM = CP == 0 ? 1 : (CP == 1 ? (CQ == 0 ? 4 : 17) : 16);
  const PairTable &t = g.t;
  const int p1 = t.pp_off[P + 1], q0 = t.pp_off[Q], q1 = t.pp_off[Q + 1];
  const int npq = *t.pq_n;
  double s[NSUM];
#pragma unroll
  for (int k = 0; k < NSUM; ++k) s[k] = 0.0;
  double Px = 0, Py = 0, Pz = 0, be = 0, b[8];  // b: the record's coefficients from c_ss on
  long long kmin = 0;  // bit pattern of 1e-14 / K of the bra primitive (K >= 0: patterns order as values)
  int pid = 0;
  unsigned nprim = 0;
  // the surviving primitive quartets in one flat loop (K descends in both
  // lists: see quartet() in eri_impl.cuh), the screen as an integer comparison
  int ip = t.pp_off[P] - 1, iq = q1;
  for (;;) {
    bool next_bra = iq >= q1;
    const double2 *kr = reinterpret_cast<const double2 *>(t.rec + (size_t)PP_REC * iq);
    double2 k4;
    if (!next_bra) {
      k4 = __ldg(kr + 2);
      next_bra = __double_as_longlong(k4.x) < kmin;
    }
    if (next_bra) {
      if (++ip >= p1 || q0 >= q1) break;
      const double2 *br = reinterpret_cast<const double2 *>(t.rec + (size_t)PP_REC * ip);
      iq = q0;
      kr = reinterpret_cast<const double2 *>(t.rec + (size_t)PP_REC * iq);
      k4 = __ldg(kr + 2);
      const double2 b2 = __ldg(br + 2);
      kmin = __double_as_longlong(b2.y);
      if (__double_as_longlong(k4.x) < kmin) break;  // nor any later bra primitive
      const double2 b0 = __ldg(br), b1 = __ldg(br + 1);
      Px = b0.x, Py = b0.y, Pz = b1.x, be = b1.y;
      const double2 b3 = __ldg(br + 3);
      b[0] = b3.x, b[1] = b3.y;
      if (CP >= 1) {
        const double2 b4 = __ldg(br + 4);
        b[2] = b4.x, b[3] = b4.y;
      }
      if (CP == 2) {
        const double2 b5 = __ldg(br + 5), b6 = __ldg(br + 6);
        b[4] = b5.x, b[5] = b5.y, b[6] = b6.x, b[7] = b6.y;
      }
      pid = t.pid[ip];
    }
    const double2 k0 = __ldg(kr), k2 = __ldg(kr + 1), k6 = __ldg(kr + 3);
    const double de = k2.y;
    double2 at;  // alpha, theta
    if (npq) {
      at = __ldg(t.pq + pid * npq + t.pid[iq]);
    } else {
      const double p = t.p[ip], q = t.p[iq], rs = rsqrt(p + q), pq = p * q;
      const double pref0 = g.mode == MQ_MODE_REFERENCE ? 2.0 * 17.493419544621675 : 2.0 * 17.493418327624862;
      at = make_double2(pq * (rs * rs), pref0 * rs / pq);
    }
    const double X = Px - k0.x, Y = Py - k0.y, Z = Pz - k2.x;
    const double T = at.x * fma(X, X, fma(Y, Y, Z * Z));
    double F[LT + 1];
    if (g.mode == MQ_MODE_REFERENCE) boys_ref<3 * LT, LT>(T, g.boys, F);
    else boys_fine<LT>(T, g.boys, F);
    if constexpr (CQ == 0) {
      // the ket's only coefficient goes into theta
      const double x0 = at.y * k6.x;
      if constexpr (CP == 0) {
        s[0] = fma(b[0] * x0, F[0], s[0]);
      } else {
        const double x1 = x0 * at.x, u0 = x0 * F[0], u1 = x1 * F[1];
        s[0] = fma(b[0], u0, s[0]);
        {  // (p_i s|ss): AB, AC, CD
          const double v = b[2] * u1;
          s[1] = fma(b[1], u0, fma(be, v, s[1]));
          s[2] += v;
          s[3] = fma(de, v, s[3]);
        }
        if constexpr (CP == 2) {
          {  // (s p_j|ss)
            const double v = b[4] * u1;
            s[4] = fma(b[3], u0, fma(be, v, s[4]));
            s[5] += v;
            s[6] = fma(de, v, s[6]);
          }
          // (p_i p_j|ss)
          const double u2 = x1 * at.x * F[2];
          const double v = b[6] * u1, a = b[6] * u2 * b[7], w = be * (v + a), ad = a * de;
          s[7] = fma(b[6], u0, fma(b[7], v, s[7]));               // delta_ij
          s[8] = fma(b[5], u0, fma(be, w + fma(be, v, -v), s[8]));  // AB AB
          s[9] += w;                                              // AB AC
          s[10] += v;                                             // AB AC - AC AB
          s[11] = fma(de, w, s[11]);                              // AB CD
          s[12] = fma(de, v, s[12]);
          s[13] += a;                                             // AC AC
          s[14] += ad;                                            // AC CD
          s[15] = fma(de, ad, s[15]);                             // CD CD
        }
      }
    } else {
      const double2 k8 = __ldg(kr + 4);
      const double d0 = k6.x, c1 = k6.y, c2 = k8.x;  // d_ss, d_ps delta, d_ps H'
      const double x1 = at.y * at.x, G0 = at.y * F[0], G1 = x1 * F[1], G2 = x1 * at.x * F[2];
      {
        const double u0 = d0 * G0, v = b[2] * (d0 * G1);
        s[0] = fma(b[0], u0, s[0]);
        s[1] = fma(b[1], u0, fma(be, v, s[1]));  // (p_i s|ss): AB, AC, CD
        s[2] += v;
        s[3] = fma(de, v, s[3]);
      }
      {
        const double v = c2 * (b[0] * G1);  // (ss|p_k s): CD, AC, AB
        s[4] = fma(c1, b[0] * G0, fma(de, v, s[4]));
        s[5] += v;
        s[6] = fma(be, v, s[6]);
      }
      // (p_i s|p_k s)
      const double bc = b[2] * c2, a1 = bc * G1, a2 = bc * G2, q1k = b[1] * c2 * G1;
      const double da = de * a2, ba = be * a2;
      const double f = fma(b[2] * c1, G1, da), h = q1k + ba;
      s[7] += a1;                 // delta_ik
      s[8] += a2;                 // AC AC
      s[9] += ba;                 // AC AB
      s[10] += da;                // CD AC
      s[11] = fma(be, da, s[11]); // CD AB
      s[12] += f;                 // AC CD
      s[13] = fma(de, f, s[13]);  // CD CD
      s[14] += h;                 // AB AC
      s[15] = fma(be, h, s[15]);  // AB AB
      s[16] = fma(b[1] * c1, G0, fma(be, f, fma(de, q1k, s[16])));  // AB CD
    }
    ++iq;
    ++nprim;
  }
  // the vectors
  double acc[NA][NB][NC][ND];
  acc[0][0][0][0] = s[0];
  if constexpr (CP >= 1) {
    const double *gp = t.geom + 6 * (size_t)P, *gq = t.geom + 6 * (size_t)Q;
    double AB[3], CD[3], AC[3];
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      AB[k] = gp[3 + k];
      CD[k] = gq[3 + k];
      AC[k] = gp[k] - gq[k];
    }
#pragma unroll
    for (int i = 0; i < 3; ++i) acc[i + 1][0][0][0] = fma(AB[i], s[1], fma(AC[i], s[2], -CD[i] * s[3]));
    if constexpr (CQ == 1) {
#pragma unroll
      for (int k = 0; k < 3; ++k) acc[0][0][k + 1][0] = fma(CD[k], s[4], -fma(AC[k], s[5], AB[k] * s[6]));
#pragma unroll
      for (int k = 0; k < 3; ++k) {
        const double vab = fma(CD[k], s[16], -fma(AC[k], s[14], AB[k] * s[15]));
        const double vac = fma(CD[k], s[12], -fma(AC[k], s[8], AB[k] * s[9]));
        const double vcd = fma(AC[k], s[10], fma(AB[k], s[11], -CD[k] * s[13]));
#pragma unroll
        for (int i = 0; i < 3; ++i)
          acc[i + 1][0][k + 1][0] = fma(AB[i], vab, fma(AC[i], vac, fma(CD[i], vcd, i == k ? 0.5 * s[7] : 0.0)));
      }
    }
    if constexpr (CP == 2) {
#pragma unroll
      for (int j = 0; j < 3; ++j) acc[0][j + 1][0][0] = fma(AB[j], s[4], fma(AC[j], s[5], -CD[j] * s[6]));
#pragma unroll
      for (int j = 0; j < 3; ++j) {
        const double vab = fma(AB[j], s[8], fma(AC[j], s[9], -CD[j] * s[11]));
        const double vac = fma(AB[j], s[9] - s[10], fma(AC[j], s[13], -CD[j] * s[14]));
        const double vcd = fma(CD[j], s[15], -fma(AB[j], s[11] - s[12], AC[j] * s[14]));
#pragma unroll
        for (int i = 0; i < 3; ++i)
          acc[i + 1][j + 1][0][0] = fma(AB[i], vab, fma(AC[i], vac, fma(CD[i], vcd, i == j ? -0.5 * s[7] : 0.0)));
      }
    }
  }
  eri_epilogue<LA, LB, LC, LD, 0, NA, 0, NB, 0, NC, 0, ND, EPI>(g, P, Q, n, XXout, acc, nprim);
}

// (sp sp|sp s): 64 integrals from 73 sums, shared by two threads so that the
// sums stay in registers.  Role 1: the ket's s function (the sums of (sp sp|ss),
// k = 0) and its p functions with at most one p in the bra (those of
// (sp s|sp s), for either bra function); role 2: (p_i p_j|p_k s), which is
//     CD_k [c_ps delta] (the tensor of (p_i p_j|ss))
//   - (P - Q)_k [the same tensor one order up, without its delta_ij part]
//   + the delta_ij, delta_ik, delta_jk terms,
// so its sums are those of the tensor with the weights 1, beta and delta of
// P - Q = AC + beta AB - delta CD.
template <int ROLE, int EPI>
__device__ __forceinline__ void quartet_mid(const EriArgs &g, int P, int Q, size_t n, double *XXout) {
  constexpr int LT = 3;
  constexpr int NSUM = ROLE == 1 ? 39 : 34;
  const PairTable &t = g.t;
  const int p1 = t.pp_off[P + 1], q0 = t.pp_off[Q], q1 = t.pp_off[Q + 1];
  const int npq = *t.pq_n;
  double s[NSUM];
#pragma unroll
  for (int k = 0; k < NSUM; ++k) s[k] = 0.0;
  double Px = 0, Py = 0, Pz = 0, be = 0, b[8];
  long long kmin = 0;
  int pid = 0;
  unsigned nprim = 0;
  int ip = t.pp_off[P] - 1, iq = q1;
  for (;;) {
    bool next_bra = iq >= q1;
    const double2 *kr = reinterpret_cast<const double2 *>(t.rec + (size_t)PP_REC * iq);
    double2 k4;
    if (!next_bra) {
      k4 = __ldg(kr + 2);
      next_bra = __double_as_longlong(k4.x) < kmin;
    }
    if (next_bra) {
      if (++ip >= p1 || q0 >= q1) break;
      const double2 *br = reinterpret_cast<const double2 *>(t.rec + (size_t)PP_REC * ip);
      iq = q0;
      kr = reinterpret_cast<const double2 *>(t.rec + (size_t)PP_REC * iq);
      k4 = __ldg(kr + 2);
      const double2 b2 = __ldg(br + 2);
      kmin = __double_as_longlong(b2.y);
      if (__double_as_longlong(k4.x) < kmin) break;  // nor any later bra primitive
      const double2 b0 = __ldg(br), b1 = __ldg(br + 1), b3 = __ldg(br + 3), b4 = __ldg(br + 4), b5 = __ldg(br + 5),
                    b6 = __ldg(br + 6);
      Px = b0.x, Py = b0.y, Pz = b1.x, be = b1.y;
      b[0] = b3.x, b[1] = b3.y, b[2] = b4.x, b[3] = b4.y, b[4] = b5.x, b[5] = b5.y, b[6] = b6.x, b[7] = b6.y;
      pid = t.pid[ip];
    }
    const double2 k0 = __ldg(kr), k2 = __ldg(kr + 1), k6 = __ldg(kr + 3), k8 = __ldg(kr + 4);
    const double de = k2.y, d0 = k6.x, c1 = k6.y, c2 = k8.x;  // delta, d_ss, d_ps delta, d_ps H'
    double2 at;  // alpha, theta
    if (npq) {
      at = __ldg(t.pq + pid * npq + t.pid[iq]);
    } else {
      const double p = t.p[ip], q = t.p[iq], rs = rsqrt(p + q), pq = p * q;
      const double pref0 = g.mode == MQ_MODE_REFERENCE ? 2.0 * 17.493419544621675 : 2.0 * 17.493418327624862;
      at = make_double2(pq * (rs * rs), pref0 * rs / pq);
    }
    const double X = Px - k0.x, Y = Py - k0.y, Z = Pz - k2.x;
    const double T = at.x * fma(X, X, fma(Y, Y, Z * Z));
    double F[LT + 1];
    if (g.mode == MQ_MODE_REFERENCE) boys_ref<3 * LT, LT>(T, g.boys, F);
    else boys_fine<LT>(T, g.boys, F);
    const double x1 = at.y * at.x, x2 = x1 * at.x;
    const double G0 = at.y * F[0], G1 = x1 * F[1], G2 = x2 * F[2];
    // the tensor of (p_i p_j|ss) for (u0, u1, u2): the sums o .. o + 8 with the
    // delta_ij sum first (see quartet_low)
    auto tensor = [&](int o, double u0, double u1, double u2) {
      const double v = b[6] * u1, a = b[6] * u2 * b[7], w = be * (v + a), ad = a * de;
      s[o] = fma(b[6], u0, fma(b[7], v, s[o]));
      s[o + 1] = fma(b[5], u0, fma(be, w + fma(be, v, -v), s[o + 1]));
      s[o + 2] += w;
      s[o + 3] += v;
      s[o + 4] = fma(de, w, s[o + 4]);
      s[o + 5] = fma(de, v, s[o + 5]);
      s[o + 6] += a;
      s[o + 7] += ad;
      s[o + 8] = fma(de, ad, s[o + 8]);
    };
    if constexpr (ROLE == 1) {
      const double u0 = d0 * G0, u1 = d0 * G1, u2 = d0 * G2;
      s[0] = fma(b[0], u0, s[0]);
      {  // (ss|p_k s): CD, AC, AB
        const double v = c2 * (b[0] * G1);
        s[1] = fma(c1, b[0] * G0, fma(de, v, s[1]));
        s[2] += v;
        s[3] = fma(be, v, s[3]);
      }
#pragma unroll
      for (int f = 0; f < 2; ++f) {  // the bra function p_i s, then s p_j
        const double f1 = b[1 + 2 * f], f2 = b[2 + 2 * f];
        const int o = 4 + 13 * f;
        const double v = f2 * u1;
        s[o] = fma(f1, u0, fma(be, v, s[o]));  // (p_i s|ss): AB, AC, CD
        s[o + 1] += v;
        s[o + 2] = fma(de, v, s[o + 2]);
        const double bc = f2 * c2, a1 = bc * G1, a2 = bc * G2, q1k = f1 * c2 * G1;
        const double da = de * a2, ba = be * a2;
        const double ff = fma(f2 * c1, G1, da), h = q1k + ba;
        s[o + 3] += a1;
        s[o + 4] += a2;
        s[o + 5] += ba;
        s[o + 6] += da;
        s[o + 7] = fma(be, da, s[o + 7]);
        s[o + 8] += ff;
        s[o + 9] = fma(de, ff, s[o + 9]);
        s[o + 10] += h;
        s[o + 11] = fma(be, h, s[o + 11]);
        s[o + 12] = fma(f1 * c1, G0, fma(be, ff, fma(de, q1k, s[o + 12])));
      }
      tensor(30, u0, u1, u2);  // (p_i p_j|ss)
    } else {
      const double G3 = x2 * at.x * F[3];
      tensor(0, c1 * G0, c1 * G1, c1 * G2);  // with CD_k
      const double z0 = c2 * G1, z1 = c2 * G2, z2 = c2 * G3;
      const double v = b[6] * z1, a = b[6] * z2 * b[7], w = be * (v + a), ad = a * de, wd = w * de, vd = v * de;
      const double z = fma(be, w + fma(be, v, -v), b[5] * z0), add = ad * de;
      s[9] += z;  // AB AB, with 1, beta, delta
      s[10] = fma(be, z, s[10]);
      s[11] = fma(de, z, s[11]);
      s[12] += w;  // AB AC
      s[13] = fma(be, w, s[13]);
      s[14] += wd;  // (= AB CD with 1)
      s[15] = fma(be, wd, s[15]);
      s[16] = fma(de, wd, s[16]);
      s[17] += v;  // AB AC - AC AB
      s[18] = fma(be, v, s[18]);
      s[19] += vd;  // (= AB CD - CD AB with 1)
      s[20] = fma(be, vd, s[20]);
      s[21] = fma(de, vd, s[21]);
      s[22] += a;  // AC AC
      s[23] = fma(be, a, s[23]);
      s[24] += ad;  // (= AC CD with 1)
      s[25] = fma(be, ad, s[25]);
      s[26] += add;  // (AC CD with delta, CD CD with 1)
      s[27] = fma(be, add, s[27]);
      s[28] = fma(de, add, s[28]);
      const double B1 = b[6] * z0, A2 = v * b[7], D = B1 + A2;
      s[29] += B1;
      s[30] += A2;
      s[31] = fma(be, D, s[31]);
      s[32] = fma(de, D, s[32]);
      s[33] = fma(de, A2, s[33]);
    }
    ++iq;
    ++nprim;
  }
  const double *gp = t.geom + 6 * (size_t)P, *gq = t.geom + 6 * (size_t)Q;
  double AB[3], CD[3], AC[3];
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    AB[k] = gp[3 + k];
    CD[k] = gq[3 + k];
    AC[k] = gp[k] - gq[k];
  }
  // element (i, j) of the tensor with sums ABAB, w, v, wd, vd, a, ad, add
  auto element = [&](int i, int j, double zz, double w, double v, double wd, double vd, double a, double ad,
                     double add) {
    const double vab = fma(AB[j], zz, fma(AC[j], w, -CD[j] * wd));
    const double vac = fma(AB[j], w - v, fma(AC[j], a, -CD[j] * ad));
    const double vcd = fma(CD[j], add, -fma(AB[j], wd - vd, AC[j] * ad));
    return fma(AB[i], vab, fma(AC[i], vac, CD[i] * vcd));
  };
  double acc[4][4][4][1];
#pragma unroll
  for (int a = 0; a < 4; ++a)
#pragma unroll
    for (int bb = 0; bb < 4; ++bb)
#pragma unroll
      for (int c = 0; c < 4; ++c) acc[a][bb][c][0] = 0.0;
  if constexpr (ROLE == 1) {
    acc[0][0][0][0] = s[0];
#pragma unroll
    for (int k = 0; k < 3; ++k) acc[0][0][k + 1][0] = fma(CD[k], s[1], -fma(AC[k], s[2], AB[k] * s[3]));
#pragma unroll
    for (int f = 0; f < 2; ++f) {
      const double *q = s + 4 + 13 * f;
#pragma unroll
      for (int i = 0; i < 3; ++i) {
        const double x = fma(AB[i], q[0], fma(AC[i], q[1], -CD[i] * q[2]));
        acc[f ? 0 : i + 1][f ? i + 1 : 0][0][0] = x;
      }
#pragma unroll
      for (int k = 0; k < 3; ++k) {
        const double vab = fma(CD[k], q[12], -fma(AC[k], q[10], AB[k] * q[11]));
        const double vac = fma(CD[k], q[8], -fma(AC[k], q[4], AB[k] * q[5]));
        const double vcd = fma(AC[k], q[6], fma(AB[k], q[7], -CD[k] * q[9]));
#pragma unroll
        for (int i = 0; i < 3; ++i) {
          const double x = fma(AB[i], vab, fma(AC[i], vac, fma(CD[i], vcd, i == k ? 0.5 * q[3] : 0.0)));
          acc[f ? 0 : i + 1][f ? i + 1 : 0][k + 1][0] = x;
        }
      }
    }
#pragma unroll
    for (int i = 0; i < 3; ++i)
#pragma unroll
      for (int j = 0; j < 3; ++j)
        acc[i + 1][j + 1][0][0] = element(i, j, s[31], s[32], s[33], s[34], s[35], s[36], s[37], s[38]) -
                                  (i == j ? 0.5 * s[30] : 0.0);
  } else {
    const double sD = s[29] + s[30];
#pragma unroll
    for (int i = 0; i < 3; ++i)
#pragma unroll
      for (int j = 0; j < 3; ++j) {
        const double tk1 =
            element(i, j, s[1], s[2], s[3], s[4], s[5], s[6], s[7], s[8]) - (i == j ? 0.5 * s[0] : 0.0);
        const double m1 = element(i, j, s[9], s[12], s[17], s[14], s[19], s[22], s[24], s[26]);
        const double mb = element(i, j, s[10], s[13], s[18], s[15], s[20], s[23], s[25], s[27]);
        const double md = element(i, j, s[11], s[14], s[19], s[16], s[21], s[24], s[26], s[28]);
#pragma unroll
        for (int k = 0; k < 3; ++k) {
          double x = fma(CD[k], tk1 + md, -fma(AC[k], m1, AB[k] * mb));
          if (i == j) x = fma(0.5, fma(AC[k], sD, fma(AB[k], s[31], -CD[k] * s[32])), x);
          if (j == k) x = fma(0.5, fma(AC[i], s[30], fma(AB[i], s[31], -CD[i] * s[33])), x);
          if (i == k) x = fma(0.5, fma(AC[j], s[30], fma(AB[j], s[31] - s[29], -CD[j] * s[33])), x);
          acc[i + 1][j + 1][k + 1][0] = x;
        }
      }
  }
  eri_epilogue<1, 1, 1, 0, 0, 4, 0, 4, 0, 4, 0, 1, EPI, ROLE>(g, P, Q, n, XXout, acc, nprim);
}

}  // namespace mq

// eri_low.cuh -- the contracted quartets of at most 16 integrals, (ss|ss),
// (sp s|ss), (sp s|sp s) and (sp sp|ss), in FP64 with early contraction
// (included by eri_impl.cuh).
//
// With A and C the first centres of the two pairs, AB = B - A, CD = D - C,
// AC = A - C, beta = b/p and delta = d/q, the vectors of the McMurchie-Davidson
// formula are
//     P - A = beta AB,  P - B = (beta - 1) AB,  P - Q = AC + beta AB - delta CD,
// so a contracted integral is a polynomial in the components of AB, AC and CD,
// which all primitive quartets share, whose coefficients are sums over the
// primitive quartets of products of beta, delta, 1/p, 1/q and
//     G0 = theta F_0(T),  G1 = theta alpha F_1(T),  G2 = theta alpha^2 F_2(T).
// Only those sums are formed per primitive quartet (1, 4, 17 and 16 of them), as
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
// (sp sp|ss) 65 / 146.
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

}  // namespace mq

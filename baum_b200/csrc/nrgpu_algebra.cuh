// nrgpu_algebra.cuh -- the BSSN and Z4c right-hand sides at one point, from
// derivatives that a source provides (included by nrgpu_parts.cuh).
//
// The physics is bssn_rhs_movpunc_N (spec bssn_rhs_movpunc_N.m:218-372) and
// z4_rhs_movpunc_N (spec z4_rhs_movpunc_N.m:216-397).  The order of work is
// chosen for register pressure and operation count, not the reference's:
// each group of derivatives is consumed as soon as it is formed, a variable's
// result leaves through the sink once it is complete, and tensor products
// are contracted pairwise (the connection terms of the Ricci tensor through
// one raised index: 216 products per point instead of 540; A~ A~ and A~^ij
// through A~^i_j: 63 instead of 216).  Algebraically these are the
// reference's expressions; only the rounding differs (which the levels of a
// hierarchy of fine spacing amplify: nrgpu_fmr_create).
//
// A source S gives, at its point,
//   val(v)               the variable
//   d1(v, n1)            first-derivative numerators along x, y, z
//   jet(v, n1, n2)       the same and the second-derivative numerators
//                        (xx xy xz yy yz zz)
//   add_part(v, r)       r plus the weighted advection and dissipation
//   adv_gamma(a)         the advection of Gamma~^a alone
// and a sink E takes results: put<N>(v, r) for the variables v .. v + N - 1.

// factors that turn numerators into derivatives, the same for every point:
// formed on the host, read as constants
struct DerivScale {
  double o1[3];   // 1 / (den1 h)
  double o2[6];   // 1 / (den2 h^2) on the diagonal, o1 o1 off it
  double ooh[3];  // 1 / h
};

__host__ inline DerivScale deriv_scale(int order, double dx, double dy, double dz) {
  const double h[3] = {dx, dy, dz};
  const double e1 = order == 2 ? 2.0 : order == 4 ? 12.0 : 60.0, e2 = order == 2 ? 1.0 : order == 4 ? 12.0 : 180.0;
  DerivScale s;
  for (int a = 0; a < 3; ++a) {
    s.o1[a] = 1.0 / (e1 * h[a]);
    s.ooh[a] = 1.0 / h[a];
  }
  for (int a = 0; a < 3; ++a)
    for (int b = a; b < 3; ++b) s.o2[sy(a, b)] = a == b ? 1.0 / (e2 * h[a] * h[a]) : s.o1[a] * s.o1[b];
  return s;
}

__device__ __forceinline__ void inverse_metric(const double g[6], double gi[6]) {
  const double detg = g[0] * g[3] * g[5] + 2.0 * g[1] * g[2] * g[4] - g[0] * g[4] * g[4] -
                      g[3] * g[2] * g[2] - g[5] * g[1] * g[1];
  const double detginv = 1.0 / detg;
  gi[0] = detginv * (g[3] * g[5] - g[4] * g[4]);
  gi[1] = detginv * (g[2] * g[4] - g[1] * g[5]);
  gi[2] = detginv * (g[1] * g[4] - g[2] * g[3]);
  gi[3] = detginv * (g[0] * g[5] - g[2] * g[2]);
  gi[4] = detginv * (g[1] * g[2] - g[0] * g[4]);
  gi[5] = detginv * (g[0] * g[3] - g[1] * g[1]);
}

// t^ab s_ab of two symmetric tensors
__device__ __forceinline__ double trace6(const double gi[6], const double t[6]) {
  return gi[0] * t[0] + gi[3] * t[3] + gi[5] * t[5] + 2.0 * (gi[1] * t[1] + gi[2] * t[2] + gi[4] * t[4]);
}

// base^e with the driver's usual exponent 0 free of the power function
__device__ __forceinline__ double gauge_power(double base, double e) { return e == 0.0 ? 1.0 : pow(base, e); }

// psi^-4 of chi = psi^p: chi itself for p = -4 (and NaN for a negative chi,
// as the logarithm gives)
__device__ __forceinline__ double psi_m4(double chig, double p, double oocp) {
  if (p == -4.0) return chig < 0.0 ? nan("") : chig;
  return exp(-4.0 * (oocp * log(chig)));
}

// the connection of the conformal metric, gam[c][ab], its trace Gfg[c] and
// the Ricci tensor without its conformal-factor part
template <class S>
__device__ __forceinline__ void conformal_ricci(const S &s, const DerivScale &c, int vg, int vG, const double g[6],
                                                const double gi[6], double gam[3][6], double Gfg[3], double Rt[6]) {
  double gdo[3][6];
  {
    double w[6], dg[3][6];
#pragma unroll
    for (int a = 0; a < 3; ++a)
#pragma unroll
      for (int b = a; b < 3; ++b) w[sy(a, b)] = (a == b ? -0.5 : -1.0) * gi[sy(a, b)] * c.o2[sy(a, b)];
#pragma unroll
    for (int v = 0; v < 6; ++v) {
      double n1[3], n2[6];
      s.jet(vg + v, n1, n2);
      double t = w[0] * n2[0];
#pragma unroll
      for (int q = 1; q < 6; ++q) t += w[q] * n2[q];
      Rt[v] = t;
#pragma unroll
      for (int a = 0; a < 3; ++a) dg[a][v] = c.o1[a] * n1[a];
    }
    // gdo[c][ab] = 1/2 (d_a g_bc + d_b g_ac - d_c g_ab)
#pragma unroll
    for (int d = 0; d < 3; ++d)
#pragma unroll
      for (int a = 0; a < 3; ++a)
#pragma unroll
        for (int b = a; b < 3; ++b)
          gdo[d][sy(a, b)] = 0.5 * (dg[a][sy(b, d)] + dg[b][sy(a, d)] - dg[d][sy(a, b)]);
  }
#pragma unroll
  for (int d = 0; d < 3; ++d)
#pragma unroll
    for (int q = 0; q < 6; ++q)
      gam[d][q] = gi[sy(d, 0)] * gdo[0][q] + gi[sy(d, 1)] * gdo[1][q] + gi[sy(d, 2)] * gdo[2][q];
#pragma unroll
  for (int a = 0; a < 3; ++a) Gfg[a] = trace6(gi, gam[a]);
  // connection terms: with u[e][c] = ginv^cd gdo_l,ed the three products of
  // the spec are gam^e_ca u_b[e][c], its transpose, and gam^l_ad u_l[b][d]
#pragma unroll
  for (int l = 0; l < 3; ++l) {
    double u[3][3];
#pragma unroll
    for (int e = 0; e < 3; ++e)
#pragma unroll
      for (int d = 0; d < 3; ++d)
        u[e][d] = gi[sy(d, 0)] * gdo[l][sy(e, 0)] + gi[sy(d, 1)] * gdo[l][sy(e, 1)] + gi[sy(d, 2)] * gdo[l][sy(e, 2)];
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      double t = 0.0;
#pragma unroll
      for (int e = 0; e < 3; ++e)
#pragma unroll
        for (int d = 0; d < 3; ++d) t += gam[e][sy(d, a)] * u[e][d];
      Rt[sy(a, l)] += a == l ? 2.0 * t : t;
    }
#pragma unroll
    for (int a = 0; a < 3; ++a)
#pragma unroll
      for (int b = a; b < 3; ++b)
        Rt[sy(a, b)] += gam[l][sy(a, 0)] * u[b][0] + gam[l][sy(a, 1)] * u[b][1] + gam[l][sy(a, 2)] * u[b][2];
  }
  // 1/2 (g_ca d_b G^c + g_cb d_a G^c + G^c (gdo_abc + gdo_bac))
  {
    double low[3][3];  // [b][a] = g_ca d_b G^c + G(g)^c gdo_abc
#pragma unroll
    for (int a = 0; a < 3; ++a)
#pragma unroll
      for (int b = 0; b < 3; ++b)
        low[b][a] = Gfg[0] * gdo[a][sy(b, 0)] + Gfg[1] * gdo[a][sy(b, 1)] + Gfg[2] * gdo[a][sy(b, 2)];
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      double n1[3];
      s.d1(vG + d, n1);
#pragma unroll
      for (int b = 0; b < 3; ++b) {
        const double dG = c.o1[b] * n1[b];
#pragma unroll
        for (int a = 0; a < 3; ++a) low[b][a] += g[sy(d, a)] * dG;
      }
    }
#pragma unroll
    for (int a = 0; a < 3; ++a)
#pragma unroll
      for (int b = a; b < 3; ++b) Rt[sy(a, b)] += 0.5 * (low[b][a] + low[a][b]);
  }
}

// derivatives of chi = psi^p: df = d log psi, dchic = d chi / chi, and the
// conformal-factor part of the Ricci tensor added to Rt
template <class S>
__device__ __forceinline__ void conformal_factor(const S &s, const DerivScale &c, int vchi, double oochi, double cpp,
                                                 double oocp, const double g[6], const double gi[6],
                                                 const double gam[3][6], double df[3], double dchic[3], double Rt[6]) {
  double n1[3], n2[6], cddf[6];
  s.jet(vchi, n1, n2);
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    dchic[a] = c.o1[a] * n1[a] * oochi;
    df[a] = oocp * dchic[a];
  }
  double dfdf = 0.0;
#pragma unroll
  for (int a = 0; a < 3; ++a)
    dfdf += df[a] * (gi[sy(a, 0)] * df[0] + gi[sy(a, 1)] * df[1] + gi[sy(a, 2)] * df[2]);
  const double os = oocp * oochi;
#pragma unroll
  for (int a = 0; a < 3; ++a)
#pragma unroll
    for (int b = a; b < 3; ++b) {
      const int ab = sy(a, b);
      cddf[ab] = os * (c.o2[ab] * n2[ab]) - cpp * df[a] * df[b] -
                 (gam[0][ab] * df[0] + gam[1][ab] * df[1] + gam[2][ab] * df[2]);
    }
  const double tr = 2.0 * trace6(gi, cddf) + 4.0 * dfdf;
#pragma unroll
  for (int a = 0; a < 3; ++a)
#pragma unroll
    for (int b = a; b < 3; ++b) {
      const int ab = sy(a, b);
      Rt[ab] += 4.0 * df[a] * df[b] - 2.0 * cddf[ab] - g[ab] * tr;
    }
}

// da = d alpha, cdda = D_a D_b alpha of the physical metric
template <class S>
__device__ __forceinline__ void lapse_derivatives(const S &s, const DerivScale &c, int valpha, const double g[6],
                                                  const double gi[6], const double gam[3][6], const double df[3],
                                                  double da[3], double cdda[6]) {
  double n1[3], n2[6];
  s.jet(valpha, n1, n2);
#pragma unroll
  for (int a = 0; a < 3; ++a) da[a] = c.o1[a] * n1[a];
  double dfda = 0.0;
#pragma unroll
  for (int a = 0; a < 3; ++a)
    dfda += df[a] * (gi[sy(a, 0)] * da[0] + gi[sy(a, 1)] * da[1] + gi[sy(a, 2)] * da[2]);
#pragma unroll
  for (int a = 0; a < 3; ++a)
#pragma unroll
    for (int b = a; b < 3; ++b) {
      const int ab = sy(a, b);
      const double t = c.o2[ab] * n2[ab] - (gam[0][ab] * da[0] + gam[1][ab] * da[1] + gam[2][ab] * da[2]);
      cdda[ab] = t - 2.0 * (df[a] * da[b] + df[b] * da[a] - g[ab] * dfda);
    }
}

// AA_ab = A_ac A^c_b, Ai^ab and A_ab A^ab
__device__ __forceinline__ double curvature_products(const double A[6], const double gi[6], double AA[6],
                                                     double Ai[6]) {
  double m[3][3];  // A^a_b
#pragma unroll
  for (int a = 0; a < 3; ++a)
#pragma unroll
    for (int b = 0; b < 3; ++b) m[a][b] = gi[sy(a, 0)] * A[sy(0, b)] + gi[sy(a, 1)] * A[sy(1, b)] + gi[sy(a, 2)] * A[sy(2, b)];
#pragma unroll
  for (int a = 0; a < 3; ++a)
#pragma unroll
    for (int b = a; b < 3; ++b) {
      AA[sy(a, b)] = A[sy(a, 0)] * m[0][b] + A[sy(a, 1)] * m[1][b] + A[sy(a, 2)] * m[2][b];
      Ai[sy(a, b)] = m[a][0] * gi[sy(0, b)] + m[a][1] * gi[sy(1, b)] + m[a][2] * gi[sy(2, b)];
    }
  return trace6(gi, AA);
}

// derivatives of the shift: db[a][c] = d_a beta^c, and the second-derivative
// terms of the Gamma~ equation added to rG
template <class S>
__device__ __forceinline__ void shift_derivatives(const S &s, const DerivScale &c, int vbeta, const double gi[6],
                                                  double db[3][3], double rG[3]) {
  double w[6], divdb[3] = {0.0, 0.0, 0.0};  // divdb[b] = d_b d_a beta^a
#pragma unroll
  for (int a = 0; a < 3; ++a)
#pragma unroll
    for (int b = a; b < 3; ++b) w[sy(a, b)] = (a == b ? 1.0 : 2.0) * gi[sy(a, b)] * c.o2[sy(a, b)];
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    double n1[3], n2[6];
    s.jet(vbeta + a, n1, n2);
    double t = w[0] * n2[0];
#pragma unroll
    for (int q = 1; q < 6; ++q) t += w[q] * n2[q];
    rG[a] += t;
#pragma unroll
    for (int b = 0; b < 3; ++b) {
      db[b][a] = c.o1[b] * n1[b];
      divdb[b] += c.o2[sy(a, b)] * n2[sy(a, b)];
    }
  }
#pragma unroll
  for (int a = 0; a < 3; ++a)
    rG[a] += (1.0 / 3.0) * (gi[sy(a, 0)] * divdb[0] + gi[sy(a, 1)] * divdb[1] + gi[sy(a, 2)] * divdb[2]);
}

// r_ab += d_a beta^c t_bc + d_b beta^c t_ac - 2/3 (d_c beta^c) t_ab
__device__ __forceinline__ void add_lie(const double db[3][3], double totdiv, const double t[6], double r[6]) {
  double m[3][3];
#pragma unroll
  for (int a = 0; a < 3; ++a)
#pragma unroll
    for (int b = 0; b < 3; ++b) m[a][b] = db[a][0] * t[sy(b, 0)] + db[a][1] * t[sy(b, 1)] + db[a][2] * t[sy(b, 2)];
#pragma unroll
  for (int a = 0; a < 3; ++a)
#pragma unroll
    for (int b = a; b < 3; ++b) r[sy(a, b)] += m[a][b] + m[b][a] - t[sy(a, b)] * totdiv;
}

// ---- BSSN -------------------------------------------------------------------------
template <class S, class E>
__device__ __forceinline__ void bssn_algebra(const S &s, const DerivScale &c, const nrgpu_bssn_params &p, E &out) {
  double g[6], gi[6], gam[3][6], Gfg[3], Rt[6];
#pragma unroll
  for (int a = 0; a < 6; ++a) g[a] = s.val(G11 + a);
  inverse_metric(g, gi);
  conformal_ricci(s, c, G11, GA1, g, gi, gam, Gfg, Rt);

  const double chi = s.val(CHI), alpha = s.val(ALPHA);
  const double chig = chi < p.chiDivFloor ? p.chiDivFloor : chi;
  const double oocp = 1.0 / p.chipsipower, oochi = 1.0 / chig;
  const double psim4 = psi_m4(chig, p.chipsipower, oocp);
  double df[3], dchic[3], da[3], cdda[6];
  conformal_factor(s, c, CHI, oochi, p.chipsipower, oocp, g, gi, gam, df, dchic, Rt);
  lapse_derivatives(s, c, ALPHA, g, gi, gam, df, da, cdda);
  const double trcdda = psim4 * trace6(gi, cdda);
  const double K = s.val(KK) * p.forceKzerofactor;

  double A[6], AA[6], Ai[6], rA[6], rG[3];
#pragma unroll
  for (int a = 0; a < 6; ++a) A[a] = s.val(A11 + a);
  const double AAs = curvature_products(A, gi, AA, Ai);
  const double Rsc = AAs - 2.0 * K * K / 3.0;
  const double trf = (1.0 / 3.0) * (-trcdda + alpha * Rsc);
#pragma unroll
  for (int a = 0; a < 6; ++a)
    rA[a] = psim4 * (-cdda[a] + alpha * Rt[a]) - trf * g[a] + alpha * (K * A[a] - 2.0 * AA[a]);
  const double rK = s.add_part(KK, -trcdda + alpha * (AAs + K * K / 3.0));
  {
    const double r = rK * p.forceKzerofactor;
    out.template put<1>(KK, &r);
  }
  // Gamma~ without advection: -2 Ainv da - 2 alpha divAinv + shift terms
  {
    double dK[3];
    s.d1(KK, dK);
#pragma unroll
    for (int a = 0; a < 3; ++a) dK[a] = p.forceKzerofactor * (c.o1[a] * dK[a]);
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      double t = -trace6(Ai, gam[a]), q = 0.0;
#pragma unroll
      for (int b = 0; b < 3; ++b) {
        t += (2.0 / 3.0) * gi[sy(a, b)] * dK[b] - 6.0 * Ai[sy(a, b)] * df[b];
        q += Ai[sy(a, b)] * da[b];
      }
      rG[a] = -2.0 * q - 2.0 * alpha * t;
    }
  }
  double db[3][3];
  shift_derivatives(s, c, BETA1, gi, db, rG);
  const double divbeta = db[0][0] + db[1][1] + db[2][2], totdiv = (2.0 / 3.0) * divbeta;
#pragma unroll
  for (int a = 0; a < 3; ++a)
    rG[a] += Gfg[a] * totdiv - (Gfg[0] * db[0][a] + Gfg[1] * db[1][a] + Gfg[2] * db[2][a]);
  add_lie(db, totdiv, A, rA);
#pragma unroll
  for (int a = 0; a < 6; ++a) rA[a] = s.add_part(A11 + a, rA[a]);
  out.template put<6>(A11, rA);
  {
    double rg[6];
#pragma unroll
    for (int a = 0; a < 6; ++a) rg[a] = -2.0 * alpha * A[a];
    add_lie(db, totdiv, g, rg);
#pragma unroll
    for (int a = 0; a < 6; ++a) rg[a] = s.add_part(G11 + a, rg[a]);
    out.template put<6>(G11, rg);
    const double rchi =
        s.add_part(CHI, (p.chipsipower / 6.0) * chig * divbeta - (p.chipsipower / 6.0) * chig * alpha * K);
    out.template put<1>(CHI, &rchi);
  }

  // gauge
  const double falpha = p.oploglapse * p.lapseharmonicf +
                        (p.oploglapse2 ? p.oploglapse2 * 8.0 / (3.0 * (3.0 - alpha)) : 0.0) + p.harmoniclapse * alpha;
  const double ralpha = s.add_part(ALPHA, -falpha * alpha * K);
  out.template put<1>(ALPHA, &ralpha);
  const double betaF = p.shiftgammacoeff * gauge_power(alpha, p.shiftalphapower);
  const double bfac = p.gamma0factor + p.gamma2factor * betaF;
  const double alphaG = p.shiftgammacoeff * gauge_power(alpha, p.shiftGalphapower);
  double rb[3], rB[3];
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    const double Ba = s.val(BB1 + a), ba = s.val(BETA1 + a), Ga = s.val(GA1 + a);
    const double wG = bfac * (1.0 - p.withGadv);
    rb[a] = s.add_part(BETA1 + a, (p.gamma2factor + p.gamma0factor * betaF) * p.withB * Ba +
                                      (1.0 - p.withB) * (alphaG * Ga - p.shiftdriver * ba));
    rB[a] = s.add_part(BB1 + a, p.withB * (bfac * rG[a] - p.shiftdriver * Ba +
                                           (p.withGadv != 1.0 ? wG * s.adv_gamma(a) : 0.0)));
    rG[a] = s.add_part(GA1 + a, rG[a]);
  }
  out.template put<3>(GA1, rG);
  out.template put<3>(BETA1, rb);
  out.template put<3>(BB1, rB);
}

// ---- Z4c --------------------------------------------------------------------------
template <class S, class E>
__device__ __forceinline__ void z4_algebra(const S &s, const DerivScale &c, const nrgpu_z4_params &p, E &out) {
  double g[6], gi[6], gam[3][6], Gfg[3], Rt[6];
#pragma unroll
  for (int a = 0; a < 6; ++a) g[a] = s.val(ZG11 + a);
  inverse_metric(g, gi);
  conformal_ricci(s, c, ZG11, ZGA1, g, gi, gam, Gfg, Rt);

  const double chi = s.val(ZCHI), alpha = s.val(ZALPHA);
  const double chig = chi < p.chiDivFloor ? p.chiDivFloor : chi;
  const double oocp = 1.0 / p.chipsipower, oochi = 1.0 / chig;
  const double psim4 = psi_m4(chig, p.chipsipower, oocp);
  double df[3], dchic[3], da[3], cdda[6];
  conformal_factor(s, c, ZCHI, oochi, p.chipsipower, oocp, g, gi, gam, df, dchic, Rt);
  const double Rhat = psim4 * trace6(gi, Rt);
  lapse_derivatives(s, c, ZALPHA, g, gi, gam, df, da, cdda);
  const double trcdda = psim4 * trace6(gi, cdda);
  const double Khat = s.val(ZKHAT), Theta = s.val(ZTHETA), K = Khat + 2.0 * Theta;

  double A[6], AA[6], Ai[6], rA[6], rG[3];
#pragma unroll
  for (int a = 0; a < 6; ++a) A[a] = s.val(ZA11 + a);
  const double cAA = curvature_products(A, gi, AA, Ai);
  const double Hhat = Rhat + 2.0 * K * K / 3.0 - cAA;
  const double trf = (1.0 / 3.0) * (-trcdda + alpha * Rhat);
#pragma unroll
  for (int a = 0; a < 6; ++a)
    rA[a] = psim4 * (-cdda[a] + alpha * Rt[a]) - trf * g[a] + alpha * (K * A[a] - 2.0 * AA[a]);
  {
    const double rK =
        s.add_part(ZKHAT, -trcdda + alpha * (cAA + K * K / 3.0) + p.kappa1 * (1.0 - p.kappa2) * alpha * Theta);
    const double rT =
        s.add_part(ZTHETA, alpha * (Hhat / 2.0 - (2.0 + p.kappa2) * p.kappa1 * Theta) * p.zeroThetaRHS);
    out.template put<1>(ZKHAT, &rK);
    out.template put<1>(ZTHETA, &rT);
  }
  // Gamma~ without advection: -2 Ainv da + 2 alpha divAinv - 2 alpha kappa1 (G - G(g))
  {
    double dK[3], dT[3];
    s.d1(ZKHAT, dK);
    s.d1(ZTHETA, dT);
#pragma unroll
    for (int a = 0; a < 3; ++a) dK[a] = c.o1[a] * (2.0 * dK[a] + dT[a]);
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      double dv = trace6(Ai, gam[a]), q = 0.0;
#pragma unroll
      for (int b = 0; b < 3; ++b) {
        dv += -1.5 * Ai[sy(a, b)] * dchic[b] - (1.0 / 3.0) * gi[sy(a, b)] * dK[b];
        q += Ai[sy(a, b)] * da[b];
      }
      rG[a] = -2.0 * q + 2.0 * alpha * dv - 2.0 * alpha * p.kappa1 * (s.val(ZGA1 + a) - Gfg[a]);
    }
  }
  double db[3][3];
  shift_derivatives(s, c, ZBETA1, gi, db, rG);
  const double divbeta = db[0][0] + db[1][1] + db[2][2], totdiv = (2.0 / 3.0) * divbeta;
#pragma unroll
  for (int a = 0; a < 3; ++a)
    rG[a] += Gfg[a] * totdiv - (Gfg[0] * db[0][a] + Gfg[1] * db[1][a] + Gfg[2] * db[2][a]);
  add_lie(db, totdiv, A, rA);
#pragma unroll
  for (int a = 0; a < 6; ++a) rA[a] = s.add_part(ZA11 + a, rA[a]);
  out.template put<6>(ZA11, rA);
  {
    double rg[6];
#pragma unroll
    for (int a = 0; a < 6; ++a) rg[a] = -2.0 * alpha * A[a];
    add_lie(db, totdiv, g, rg);
#pragma unroll
    for (int a = 0; a < 6; ++a) rg[a] = s.add_part(ZG11 + a, rg[a]);
    out.template put<6>(ZG11, rg);
    const double rchi =
        s.add_part(ZCHI, (-p.chipsipower / 6.0) * chig * alpha * K + (p.chipsipower / 6.0) * chig * divbeta);
    out.template put<1>(ZCHI, &rchi);
  }

  // gauge
  const double falpha = p.oploglapse * p.lapseharmonicf +
                        (p.oploglapse2 ? p.oploglapse2 * 8.0 / (3.0 * (3.0 - alpha)) : 0.0) + p.harmoniclapse * alpha;
  const double ralpha = s.add_part(ZALPHA, -falpha * alpha * Khat);
  out.template put<1>(ZALPHA, &ralpha);
  const double betaF = p.shiftgammacoeff * gauge_power(alpha, p.shiftalphapower);
  const double bfac = p.gamma0factor + p.gamma2factor * betaF;
  const bool withB = p.withB != 0.0;
  double rb[3], rB[3];
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    const double Ba = s.val(ZBB1 + a);
    if (withB) {
      rb[a] = (p.gamma2factor + p.gamma0factor * betaF) * Ba;
      rB[a] = bfac * rG[a] - p.shiftdriver * Ba;
      if (p.withGadv != 1.0) rB[a] += bfac * (1.0 - p.withGadv) * s.adv_gamma(a);
    } else {
      rb[a] = s.val(ZGA1 + a) - p.shiftdriver * s.val(ZBETA1 + a);
      rB[a] = 0.0;
    }
    rb[a] = s.add_part(ZBETA1 + a, rb[a]);
    rB[a] = s.add_part(ZBB1 + a, rB[a]);
    rG[a] = s.add_part(ZGA1 + a, rG[a]);
  }
  out.template put<3>(ZGA1, rG);
  out.template put<3>(ZBETA1, rb);
  out.template put<3>(ZBB1, rB);
}

// factors of each variable's advection and dissipation: r_v gets
// adv[v] beta^i d_i u_v + ko[v] KO u_v
template <int NV>
struct PartScale {
  double adv[NV], ko[NV];
};

__host__ inline PartScale<NRGPU_NV> part_scale(const nrgpu_bssn_params &p) {
  PartScale<NRGPU_NV> s;
  for (int v = 0; v < NRGPU_NV; ++v) {
    s.adv[v] = v == ALPHA ? p.oplogwithshift : v >= BB1 ? p.withB * p.withBadv : v >= BETA1 ? p.withShiftadv : 1.0;
    s.ko[v] = v < ALPHA && p.order_dissipation ? p.dissfactor : 0.0;
  }
  return s;
}

__host__ inline PartScale<NRGPU_Z4_NVARS> part_scale(const nrgpu_z4_params &p) {
  PartScale<NRGPU_Z4_NVARS> s;
  for (int v = 0; v < NRGPU_Z4_NVARS; ++v) {
    s.adv[v] = v == ZTHETA ? p.zeroThetaRHS : v == ZALPHA ? p.oplogwithshift
               : v >= ZBB1 ? (p.withB != 0.0 ? p.withBadv : 0.0) : v >= ZBETA1 ? p.withShiftadv : 1.0;
    s.ko[v] = p.order_dissipation ? p.dissfactor : 0.0;
  }
  return s;
}

/*
 * The arithmetic of a geodesic's step: the finite-difference connection
 * (src/geometry.c:93-144), its contractions (push_photon, src/geodesics.c:
 * 19-49, and push_polar, src/ipolarray.c:253-289) and the step size
 * (src/model_geodesics.c:267-293).
 *
 * The connection amplifies every rounding of the metric by 1/(2 DEL) = 5e6,
 * and rays near the photon ring amplify that again, so the two kernels that
 * trace geodesics, one lane per ray (k_geodesic) and eight (k_geodesic_coop),
 * must round alike: which of them traces a pixel depends on the size of its
 * launch.  Both are built from the functions of this file, in which every
 * product and sum of the FMKS path is written as an explicitly rounded
 * operation, fused or not, so that no compiler, flag or inlining decides it.
 * (The flat metrics have the one-lane kernel only and are written plainly.)
 *
 * Included by ipg_device.cuh, after the grid's constants.
 */
#ifndef IPG_CONNECTION_CUH
#define IPG_CONNECTION_CUH

#define RN_MUL(a, b) __dmul_rn(a, b)
#define RN_ADD(a, b) __dadd_rn(a, b)
#define RN_SUB(a, b) __dsub_rn(a, b)
#define RN_FMA(a, b, c) __fma_rn(a, b, c)

/* exp(d) - 1 and sin, cos(d) for |d| < 1e-5 (Taylor; exact to rounding) */
__device__ __forceinline__ double expm_small(double d)
{
  return RN_MUL(d, RN_FMA(d, RN_FMA(d, 1. / 6., 0.5), 1.));
}
__device__ __forceinline__ void sincos_small(double d, double *s, double *c)
{
  const double d2 = RN_MUL(d, d);
  *s = RN_MUL(d, RN_FMA(-d2, 1. / 6., 1.));
  *c = RN_FMA(-0.5, d2, 1.);
}
/* sin and cos of (x + d) from those of x */
__device__ __forceinline__ void rotate(double s, double c, double sd, double cd, double *so, double *co)
{
  *so = RN_FMA(s, cd, RN_MUL(c, sd));
  *co = RN_FMA(c, cd, -RN_MUL(s, sd));
}

/* X2-dependent parts of theta(X1,X2) and its Jacobian */
struct X2P {
  double S2, C2, y, P, P1;  /* sin 2piX2, cos 2piX2, 2X2-1, q^alpha, q^(alpha-1), q = y/xt */
};

/* q^n for 0 <= n < 128 by binary powering, without branches */
__device__ __forceinline__ double ipow_int(double q, int n)
{
  double r = 1.0, b = q;
#pragma unroll
  for (int k = 0; k < 7; k++) {
    r *= (n & 1) ? b : 1.0;
    b *= b;
    n >>= 1;
  }
  return r;
}

/* q^(alpha-1) of the FMKS polar map */
__device__ __forceinline__ double fmks_pow_am1(double q)
{
  const DevGrid &G = c_grid;
  return (G.alpha_int >= 0) ? ipow_int(q, G.alpha_int) : pow(q, G.poly_alpha - 1.);
}
/* the same value, for a lone warp: the usual poly_alpha = 14 without the
 * general loop's selects (5 multiplications on the chain) */
__device__ __forceinline__ double fmks_pow_am1_lone(double q)
{
  if (c_grid.alpha_int == 13) {
    const double q2 = RN_MUL(q, q), q4 = RN_MUL(q2, q2), q8 = RN_MUL(q4, q4);
    return RN_MUL(RN_MUL(q, q4), q8);
  }
  return fmks_pow_am1(q);
}

template <bool LONE = false>
__device__ __forceinline__ void x2_parts_from(double X2, double S2, double C2, X2P *o)
{
  const DevGrid &G = c_grid;
  o->S2 = S2;
  o->C2 = C2;
  o->y = RN_FMA(2., X2, -1.);
  const double q = RN_MUL(o->y, G.inv_xt);
  o->P1 = LONE ? fmks_pow_am1_lone(q) : fmks_pow_am1(q);
  o->P = RN_MUL(o->P1, q);
}

/* theta, dtheta/dX1 (J21) and dtheta/dX2 (J22) from the parts (src/
 * coordinates.c:46-97, 263-305); E = exp(mks_smooth (startx1 - X1)).  (The
 * coefficients' point evaluation, which no second kernel has to match, has
 * its own plain form, theta_jac.) */
__device__ __forceinline__ void conn_theta(double X2, double E, const X2P &p, double *th, double *J21, double *J22)
{
  const DevGrid &G = c_grid;
  const double omh = RN_SUB(1., G.hslope), c = RN_MUL(omh, IPG_PI);
  const double poly = RN_FMA(p.P, G.inv_ap1, 1.), pny = RN_MUL(G.poly_norm, p.y);
  const double hS = RN_MUL(RN_MUL(omh, 0.5), p.S2);
  const double thG = RN_FMA(IPG_PI, X2, hS), thJ = RN_FMA(pny, poly, 0.5 * IPG_PI);
  *th = RN_FMA(E, RN_SUB(thJ, thG), thG);
  *J21 = RN_MUL(RN_MUL(-E, G.mks_smooth), RN_SUB(RN_FMA(pny, poly, RN_FMA(-IPG_PI, X2, IPG_PI * 0.5)), hS));
  const double u = RN_FMA(-c, p.C2, RN_FMA(RN_MUL(G.j22c, p.y), p.P1, RN_FMA(RN_MUL(2., G.poly_norm), poly, -IPG_PI)));
  *J22 = RN_FMA(E, u, RN_FMA(c, p.C2, IPG_PI));
}

/* g^{mu nu}, symmetric; g^03 = 0 in FMKS */
struct Gcon {
  double u00, u01, u02, u11, u12, u13, u22, u23, u33;
};

/* d_d g_{mu nu} for d = 1, 2 (the metric does not depend on X0, X3, so the
 * reference's differences in those directions are exactly zero), each as
 * 00 01 03 11 12 13 22 33 (g_02 = g_23 = 0), and g^{mu nu} at X, or half of
 * it (exact), the transport matrix's factor */
struct Conn {
  double D1[8], D2[8];
  Gcon gu;
  double r; /* r at X */
};

/* The point a connection is taken at: what the metrics at its offsets need.
 * Its g^{mu nu} is the closed form of FMKS Kerr-Schild (the reference inverts
 * gcov by LU, src/geometry.c:54-64, 252-287; both agree to rounding). */
struct ConnCentre {
  double r, E, th, s, c, rho2, irho2;
  X2P p;
};

template <bool LONE = false, bool HALF = false>
__device__ __forceinline__ void conn_centre(double r, double E, double X2, ConnCentre *o, Gcon *gu)
{
  const double a = c_grid.a, aa = RN_MUL(a, a);
  double S2, C2, J21, J22;
  sincospi(RN_MUL(2., X2), &S2, &C2);
  x2_parts_from<LONE>(X2, S2, C2, &o->p);
  conn_theta(X2, E, o->p, &o->th, &J21, &J22);
  sincos(o->th, &o->s, &o->c);
  o->r = r;
  o->E = E;
  const double s2 = RN_MUL(o->s, o->s), rho2 = RN_FMA(RN_MUL(aa, o->c), o->c, RN_MUL(r, r));
  /* one division for the four reciprocals */
  const double rJ = RN_MUL(r, J22), p2 = RN_MUL(rho2, rJ), inv = 1. / RN_MUL(p2, s2);
  const double irho2 = RN_MUL(RN_MUL(inv, rJ), s2);
  const double ir = RN_MUL(RN_MUL(RN_MUL(inv, rho2), J22), s2), iJ = RN_MUL(RN_MUL(RN_MUL(inv, rho2), r), s2);
  const double is2 = RN_MUL(inv, p2), tr = RN_MUL(RN_MUL(2., r), irho2);
  const double Delta = RN_FMA(a, a, RN_FMA(-2., r, RN_MUL(r, r)));
  const double Grr = RN_MUL(Delta, irho2), Grp = RN_MUL(a, irho2);
  const double M21 = RN_MUL(RN_MUL(-J21, ir), iJ); /* dX2/dr */
  o->rho2 = rho2;
  o->irho2 = irho2;
  Gcon &u = *gu;
  u.u00 = HALF ? RN_MUL(-0.5, RN_ADD(1., tr)) : -RN_ADD(1., tr);
  u.u01 = RN_MUL(tr, ir);
  u.u02 = RN_MUL(M21, tr);
  u.u11 = RN_MUL(RN_MUL(ir, ir), Grr);
  u.u12 = RN_MUL(RN_MUL(ir, M21), Grr);
  u.u13 = RN_MUL(ir, Grp);
  u.u22 = RN_FMA(RN_MUL(iJ, iJ), irho2, RN_MUL(RN_MUL(M21, M21), Grr));
  u.u23 = RN_MUL(M21, Grp);
  u.u33 = RN_MUL(irho2, is2);
  if (HALF) {
    u.u01 = RN_MUL(0.5, u.u01);
    u.u02 = RN_MUL(0.5, u.u02);
    u.u11 = RN_MUL(0.5, u.u11);
    u.u12 = RN_MUL(0.5, u.u12);
    u.u13 = RN_MUL(0.5, u.u13);
    u.u22 = RN_MUL(0.5, u.u22);
    u.u23 = RN_MUL(0.5, u.u23);
    u.u33 = RN_MUL(0.5, u.u33);
  }
}

/* g_{mu nu} a finite-difference offset away from the centre, at X2 = X2o with
 * the parts po, r = ro and E = Eo: sin and cos theta by their exact
 * differences, 1/rho^2 from the centre's by 1/(1+e) = 1 - e(1 - e), e ~ 1e-7
 * (the e^3 term is below rounding), which saves a division.  r^2 + a^2 cos^2
 * fuses r r at the X1 offsets and (a^2 cos) cos at the X2 offsets (x2), whose
 * r is the centre's. */
struct ConnOffset {
  double s, c, J21, J22;
};
__device__ __forceinline__ void conn_offset(const ConnCentre &c, double Eo, double X2o, const X2P &po, ConnOffset *o)
{
  double th, sd, cd;
  conn_theta(X2o, Eo, po, &th, &o->J21, &o->J22);
  sincos_small(RN_SUB(th, c.th), &sd, &cd);
  rotate(c.s, c.c, sd, cd, &o->s, &o->c);
}
__device__ __forceinline__ void conn_near(const ConnCentre &c, double ro, const ConnOffset &o, bool x2, double g[8])
{
  const double a = c_grid.a, aa = RN_MUL(a, a);
  const double s2 = RN_MUL(o.s, o.s), ac = RN_MUL(aa, o.c);
  const double rho2 = RN_FMA(x2 ? ac : ro, x2 ? o.c : ro, x2 ? RN_MUL(ro, ro) : RN_MUL(ac, o.c));
  const double e = RN_MUL(RN_SUB(rho2, c.rho2), c.irho2);
  const double t = RN_MUL(RN_MUL(2., ro), RN_MUL(c.irho2, RN_FMA(-e, RN_SUB(1., e), 1.)));
  const double t1 = RN_ADD(1., t), mas2 = RN_MUL(-a, s2), rJ1 = RN_MUL(rho2, o.J21);
  g[0] = RN_ADD(t, -1.);
  g[1] = RN_MUL(t, ro);
  g[2] = RN_MUL(mas2, t);
  g[3] = RN_FMA(rJ1, o.J21, RN_MUL(RN_MUL(t1, ro), ro));
  g[4] = RN_MUL(rJ1, o.J22);
  g[5] = RN_MUL(RN_MUL(mas2, t1), ro);
  g[6] = RN_MUL(RN_MUL(rho2, o.J22), o.J22);
  g[7] = RN_MUL(s2, RN_FMA(RN_MUL(aa, s2), t1, rho2));
}

/* (h - l) / (Xh - Xl), inv = 1 / (Xh - Xl) */
__device__ __forceinline__ double conn_diff(double h, double l, double inv) { return RN_MUL(RN_SUB(h, l), inv); }

/* r of bl_coord (src/coordinates.c:46-58) */
template <int MET>
__device__ __forceinline__ double geo_r(double X1)
{
  return (MET == IPG_MET_MINK) ? X1 : exp(X1);
}

/* the flat metrics (src/coordinates.c:180-193), diagonal; r = r(X1) */
template <int MET>
__device__ __forceinline__ void conn_flat_diag(double r, double sth, double g[8])
{
  for (int k = 0; k < 8; k++) g[k] = 0.;
  g[0] = -1.;
  g[3] = (MET == IPG_MET_MINK) ? 1. : r * r;
  g[6] = r * r;
  g[7] = r * r * sth * sth;
}
template <int MET>
__device__ void fd_connection_flat(double X1, double X2, Conn *cn)
{
  double r = geo_r<MET>(X1), s0, c0, h[8], l[8];
  sincos(X2, &s0, &c0);
  Gcon &u = cn->gu;
  u.u00 = -1.;
  u.u01 = u.u02 = u.u12 = u.u13 = u.u23 = 0.;
  u.u11 = (MET == IPG_MET_MINK) ? 1. : 1. / (r * r);
  u.u22 = 1. / (r * r);
  u.u33 = 1. / (r * r * s0 * s0);
  cn->r = r;
  double Xh = X1 + IPG_DEL, Xl = X1 - IPG_DEL;
  conn_flat_diag<MET>(geo_r<MET>(Xh), s0, h);
  conn_flat_diag<MET>(geo_r<MET>(Xl), s0, l);
  for (int k = 0; k < 8; k++) cn->D1[k] = conn_diff(h[k], l[k], 1. / (Xh - Xl));
  Xh = X2 + IPG_DEL;
  Xl = X2 - IPG_DEL;
  conn_flat_diag<MET>(r, sin(Xh), h);
  conn_flat_diag<MET>(r, sin(Xl), l);
  for (int k = 0; k < 8; k++) cn->D2[k] = conn_diff(h[k], l[k], 1. / (Xh - Xl));
}

/* The connection data at (X1, X2) on one lane.  MKS is FMKS with the jet term
 * switched off (theta = thetaG, src/coordinates.c:68-70, 278-280). */
template <int MET = IPG_MET_FMKS>
IPG_HEAVY void fd_connection(double X1, double X2, Conn *cn)
{
  if constexpr (MET == IPG_MET_MINK || MET == IPG_MET_EMINK) {
    fd_connection_flat<MET>(X1, X2, cn);
    return;
  }
  const DevGrid &G = c_grid;
  const double sm = G.mks_smooth;
  ConnCentre c;
  conn_centre(exp(X1), (MET == IPG_MET_FMKS) ? exp(RN_MUL(sm, RN_SUB(G.startx[1], X1))) : 0., X2, &c, &cn->gu);
  cn->r = c.r;
  double h[8], l[8];
  ConnOffset oh, ol;
  /* X1 +- DEL: r and E by exact offsets */
  {
    const double Xh = RN_ADD(X1, IPG_DEL), Xl = RN_SUB(X1, IPG_DEL);
    const double dh = RN_SUB(Xh, X1), dl = RN_SUB(Xl, X1); /* exact */
    const double rh = RN_FMA(c.r, expm_small(dh), c.r), rl = RN_FMA(c.r, expm_small(dl), c.r);
    const double Eh = RN_FMA(c.E, expm_small(RN_MUL(-sm, dh)), c.E), El = RN_FMA(c.E, expm_small(RN_MUL(-sm, dl)), c.E);
    conn_offset(c, Eh, X2, c.p, &oh);
    conn_offset(c, El, X2, c.p, &ol);
    conn_near(c, rh, oh, false, h);
    conn_near(c, rl, ol, false, l);
    const double inv = 1. / RN_SUB(Xh, Xl);
#pragma unroll
    for (int k = 0; k < 8; k++) cn->D1[k] = conn_diff(h[k], l[k], inv);
  }
  /* X2 +- DEL */
  {
    const double Xh = RN_ADD(X2, IPG_DEL), Xl = RN_SUB(X2, IPG_DEL);
    double sd, cd, S, C;
    X2P ph, pl;
    sincos_small(RN_MUL(2. * IPG_PI, RN_SUB(Xh, X2)), &sd, &cd);
    rotate(c.p.S2, c.p.C2, sd, cd, &S, &C);
    x2_parts_from(Xh, S, C, &ph);
    sincos_small(RN_MUL(2. * IPG_PI, RN_SUB(Xl, X2)), &sd, &cd);
    rotate(c.p.S2, c.p.C2, sd, cd, &S, &C);
    x2_parts_from(Xl, S, C, &pl);
    conn_offset(c, c.E, Xh, ph, &oh);
    conn_offset(c, c.E, Xl, pl, &ol);
    conn_near(c, c.r, oh, true, h);
    conn_near(c, c.r, ol, true, l);
    const double inv = 1. / RN_SUB(Xh, Xl);
#pragma unroll
    for (int k = 0; k < 8; k++) cn->D2[k] = conn_diff(h[k], l[k], inv);
  }
}

/* v = (partial_d g) K; SPLIT: the third product of entry 1 rounded by itself
 * (transport_matrix uses it again) */
template <bool SPLIT>
__device__ __forceinline__ void dg_dot(const double D[8], const double K[4], double v[4])
{
  v[0] = RN_FMA(D[2], K[3], RN_FMA(D[0], K[0], RN_MUL(D[1], K[1])));
  const double v1 = RN_FMA(D[1], K[0], RN_MUL(D[3], K[1]));
  v[1] = RN_FMA(D[5], K[3], SPLIT ? RN_ADD(v1, RN_MUL(D[4], K[2])) : RN_FMA(D[4], K[2], v1));
  v[2] = RN_FMA(D[4], K[1], RN_MUL(D[6], K[2]));
  v[3] = RN_FMA(D[7], K[3], RN_FMA(D[2], K[0], RN_MUL(D[5], K[1])));
}

/* Gamma^k_ij K^i K^j without the matrix (unpolarized images) */
__device__ __forceinline__ void geo_accel(const Conn &cn, const double K[4], double acc[4])
{
  double v1[4], v2[4], T[4];
  dg_dot<false>(cn.D1, K, v1);
  dg_dot<false>(cn.D2, K, v2);
  const double kv1 = RN_FMA(K[3], v1[3], RN_FMA(K[2], v1[2], RN_FMA(K[0], v1[0], RN_MUL(K[1], v1[1]))));
  const double kv2 = RN_FMA(K[3], v2[3], RN_ADD(RN_FMA(K[0], v2[0], RN_MUL(K[1], v2[1])), RN_MUL(K[2], v2[2])));
#pragma unroll
  for (int m = 0; m < 4; m++) T[m] = RN_FMA(K[1], v1[m], RN_MUL(K[2], v2[m]));
  T[1] = RN_FMA(-0.5, kv1, T[1]);
  T[2] = RN_FMA(-0.5, kv2, T[2]);
  const Gcon &u = cn.gu;
  acc[0] = RN_FMA(u.u02, T[2], RN_FMA(u.u01, T[1], RN_MUL(u.u00, T[0])));
  acc[1] = RN_FMA(u.u13, T[3], RN_FMA(u.u12, T[2], RN_FMA(u.u01, T[0], RN_MUL(u.u11, T[1]))));
  acc[2] = RN_FMA(u.u23, T[3], RN_FMA(u.u22, T[2], RN_FMA(u.u02, T[0], RN_MUL(u.u12, T[1]))));
  acc[3] = RN_FMA(u.u33, T[3], RN_FMA(u.u13, T[1], RN_MUL(u.u23, T[2])));
}

/* 2 B[m][k] = K1 d1 g_km + K2 d2 g_km + delta_k1 v1_m + delta_k2 v2_m
 * - delta_m1 v1_k - delta_m2 v2_k, with v_d = (partial_d g) K:
 * A^i_k = Gamma^i_kl K^l = g^im B[m][k] */
__device__ __forceinline__ void transport_b(const Conn &cn, const double K[4], double B[4][4])
{
  double v1[4], v2[4], d[8];
  dg_dot<false>(cn.D1, K, v1);
  dg_dot<true>(cn.D2, K, v2);
#pragma unroll
  for (int k = 0; k < 8; k++) d[k] = RN_FMA(K[1], cn.D1[k], RN_MUL(K[2], cn.D2[k]));
  B[0][0] = d[0];
  B[0][1] = RN_ADD(d[1], v1[0]);
  B[0][2] = v2[0];
  B[0][3] = d[2];
  B[1][0] = RN_SUB(d[1], v1[0]);
  B[1][1] = RN_SUB(RN_ADD(d[3], v1[1]), v1[1]);
  B[1][2] = RN_SUB(RN_ADD(d[4], v2[1]), v1[2]);
  B[1][3] = RN_SUB(d[5], v1[3]);
  B[2][0] = -v2[0];
  B[2][1] = RN_SUB(RN_ADD(d[4], v1[2]), v2[1]);
  B[2][2] = RN_SUB(RN_ADD(d[6], v2[2]), v2[2]);
  B[2][3] = -v2[3];
  B[3][0] = d[2];
  B[3][1] = RN_ADD(d[5], v1[3]);
  B[3][2] = v2[3];
  B[3][3] = d[7];
}

/* row o of A, from half of g^{mu nu} and 2 B, or from g^{mu nu} and B (the same
 * bits; one lane's step is 0.6% shorter with the latter, an eight-lane one with
 * the former); row 0 fuses its second product first */
__device__ __forceinline__ void transport_row(const Gcon &u, const double B[4][4], int o, double A[4])
{
  const double r0 = o == 0 ? u.u01 : o == 1 ? u.u01 : o == 2 ? u.u02 : 0.;
  const double r1 = o == 0 ? u.u00 : o == 1 ? u.u11 : o == 2 ? u.u12 : u.u13;
  const double r2 = o == 0 ? u.u02 : o == 1 ? u.u12 : o == 2 ? u.u22 : u.u23;
  const double r3 = o == 0 ? 0. : o == 1 ? u.u13 : o == 2 ? u.u23 : u.u33;
#pragma unroll
  for (int k = 0; k < 4; k++) {
    const double b0 = o == 0 ? B[1][k] : B[0][k], b1 = o == 0 ? B[0][k] : B[1][k];
    A[k] = RN_FMA(r3, B[3][k], RN_FMA(r2, B[2][k], RN_FMA(r0, b0, RN_MUL(r1, b1))));
  }
}
/* a row's share of Gamma^o_ij K^i K^j */
__device__ __forceinline__ double transport_accel(const double A[4], const double K[4])
{
  return RN_FMA(A[3], K[3], RN_FMA(A[2], K[2], RN_FMA(A[0], K[0], RN_MUL(A[1], K[1]))));
}

/* the whole of A on one lane, and Gamma^k_ij K^i K^j from it */
__device__ __forceinline__ void transport_matrix(const Conn &cn, const double K[4], double A[4][4])
{
  double B[4][4];
  transport_b(cn, K, B);
#pragma unroll
  for (int m = 0; m < 4; m++)
#pragma unroll
    for (int k = 0; k < 4; k++) B[m][k] = RN_MUL(0.5, B[m][k]);
#pragma unroll
  for (int i = 0; i < 4; i++) transport_row(cn.gu, B, i, A[i]);
}
__device__ __forceinline__ void accel_from_A(const double A[4][4], const double K[4], double acc[4])
{
#pragma unroll
  for (int k = 0; k < 4; k++) acc[k] = transport_accel(A[k], K);
}

/* The reference forms three step limits dlx_i = eps c_i / (|K^i| + SS) and
 * returns 1 / sum 1/(|dlx_i| + SS); with a_i = |K^i| + SS and b_i = eps c_i
 * that is dl = eps b1 b2 / (eps (a1 b2 + a2 b1) + a3 b1 b2), one division
 * instead of nine (the + SS of the inner reciprocals matters only for steps
 * near 1e-80, i.e. a ray sitting exactly on the inner or polar boundary). */
__device__ __forceinline__ double stepsize(const double X[4], const double K[4], double eps)
{
  const DevGrid &G = c_grid;
  const double SS = IPG_SMALL * IPG_SMALL;
  const double cut = 0.02;
  const double deh = fmin(fabs(RN_SUB(X[1], G.cstartx[1])), 0.1);
  const double dpole = fmin(fabs(RN_MUL(X[2], G.inv_lx2)), fabs(RN_MUL(RN_SUB(G.cstopx[2], X[2]), G.inv_lx2)));
  const double d2fac = (dpole < cut) ? RN_MUL(dpole, 1. / 3.) : fmin(RN_FMA(RN_SUB(dpole, cut), 10., cut * (1. / 3.)), 1.);
  const double a1 = RN_ADD(fabs(K[1]), SS), a2 = RN_ADD(fabs(K[2]), SS), a3 = RN_ADD(fabs(K[3]), SS);
  const double b1 = RN_MUL(eps, RN_MUL(10., deh)), b2 = RN_MUL(eps, d2fac);
  const double b12 = RN_MUL(b1, b2);
  return RN_MUL(eps, b12) / RN_FMA(a3, b12, RN_MUL(eps, RN_FMA(a1, b2, RN_MUL(a2, b1))));
}

/* out = base + h d */
__device__ __forceinline__ void geo_advance(const double base[4], double h, const double d[4], double out[4])
{
#pragma unroll
  for (int k = 0; k < 4; k++) out[k] = RN_FMA(h, d[k], base[k]);
}

#endif

/*
 * The geodesic with eight lanes per ray (k_geodesic_coop), FMKS.
 *
 * k_geodesic gives a lane a ray: a half step is ~1080 instructions at 2.8
 * cycles each for a lone warp (dependent FP64 operations of 8 cycles), 3.1 us
 * a step, so the longest rays' 5e3-16e3 steps set the time of every launch
 * that does not fill the GPU.  Here one warp integrates four rays and one
 * iteration is a whole midpoint step:
 *
 *   - Xhalf = X + h K / 2 needs the step size only, so lanes 0-3 evaluate the
 *     connection at X and lanes 4-7 the one at Xhalf in the same
 *     instructions;
 *   - the four finite-difference metrics of a connection (X1 +- DEL, X2 +-
 *     DEL) run on its four lanes: with a zero offset in one coordinate the
 *     general offset formulas reproduce that coordinate's centre values
 *     exactly, so one code path serves all four;
 *   - of the transport matrix Gamma^i_kl K^l each lane forms one row, and the
 *     rows are stored as one 128-byte line.
 *
 * Only the two contractions (with K, then with Khalf) are sequential: ~800
 * instructions a step for four rays instead of ~2160 for up to 32, so this
 * is for launches of few rays.
 *
 * The connection amplifies every rounding of the metric by 1/(2 DEL) = 5e6,
 * and rays near the photon ring amplify that again, so the records must be
 * k_geodesic's bits: the functions below are those of ipg_device.cuh
 * (theta_jac, met_from_near, gcon_from, transport_matrix, geo_accel,
 * stepsize) with their roundings spelled out, fused exactly where the
 * compiler fuses them there.
 *
 * Included by ipg_kernels.cu.
 */

#define GC_MUL(a, b) __dmul_rn(a, b)
#define GC_ADD(a, b) __dadd_rn(a, b)
#define GC_SUB(a, b) __dsub_rn(a, b)
#define GC_FMA(a, b, c) __fma_rn(a, b, c)
#define GC_LANES 8

__device__ __forceinline__ double gc_expm_small(double d)
{
  return GC_MUL(d, GC_FMA(d, GC_FMA(d, 1. / 6., 0.5), 1.));
}
__device__ __forceinline__ void gc_sincos_small(double d, double *s, double *c)
{
  const double d2 = GC_MUL(d, d);
  *s = GC_MUL(d, GC_FMA(-d2, 1. / 6., 1.));
  *c = GC_FMA(-0.5, d2, 1.);
}
/* sin and cos of (x + d) from those of x */
__device__ __forceinline__ void gc_rotate(double s, double c, double sd, double cd, double *so, double *co)
{
  *so = GC_FMA(s, cd, GC_MUL(c, sd));
  *co = GC_FMA(c, cd, -GC_MUL(s, sd));
}

/* q^(alpha - 1) as fmks_pow_am1 multiplies it up; the usual poly_alpha = 14
 * without the general loop's selects (5 multiplications on the chain) */
__device__ __forceinline__ double gc_pow_am1(double q)
{
  if (c_grid.alpha_int == 13) {
    const double q2 = GC_MUL(q, q), q4 = GC_MUL(q2, q2), q8 = GC_MUL(q4, q4);
    return GC_MUL(GC_MUL(q, q4), q8);
  }
  return fmks_pow_am1(q);
}

/* 1 / x, correctly rounded, for x within 1e-4 of 2 DEL: two Newton steps
 * from 1 / (2 DEL), the second with its exact residual (Markstein 1990,
 * theorem on correctly rounded reciprocals from an approximation within one
 * ulp) */
__device__ __forceinline__ double gc_recip_2del(double x)
{
  const double y0 = 1. / (2. * IPG_DEL);
  const double e0 = GC_FMA(-x, y0, 1.);
  const double y1 = GC_FMA(GC_FMA(e0, e0, e0), y0, y0);
  return GC_FMA(GC_FMA(-x, y1, 1.), y1, y1);
}

/* theta and its Jacobian at (X2, E) with S2, C2 = sin, cos 2 pi X2 */
__device__ __forceinline__ void gc_theta(double X2, double E, double S2, double C2, double *th, double *J21, double *J22)
{
  const DevGrid &G = c_grid;
  const double omh = GC_SUB(1., G.hslope);
  const double y = GC_FMA(2., X2, -1.), q = GC_MUL(y, G.inv_xt), P1 = gc_pow_am1(q), P = GC_MUL(P1, q);
  const double poly = GC_FMA(P, G.inv_ap1, 1.), pny = GC_MUL(G.poly_norm, y);
  const double hS = GC_MUL(GC_MUL(omh, 0.5), S2);
  const double thG = GC_FMA(IPG_PI, X2, hS), thJ = GC_FMA(pny, poly, 0.5 * IPG_PI);
  *th = GC_FMA(E, GC_SUB(thJ, thG), thG);
  *J21 = GC_MUL(GC_MUL(-E, G.mks_smooth), GC_SUB(GC_FMA(pny, poly, GC_FMA(-IPG_PI, X2, IPG_PI * 0.5)), hS));
  const double c = GC_MUL(omh, IPG_PI);
  const double u = GC_FMA(-c, C2, GC_FMA(GC_MUL(G.j22c, y), P1, GC_FMA(GC_MUL(2., G.poly_norm), poly, -IPG_PI)));
  *J22 = GC_FMA(E, u, GC_FMA(c, C2, IPG_PI));
}

struct GcPoint {
  double r;
  Gcon gu;      /* g^{mu nu}, times 1/2 (the contraction's factor; exact) */
  double D1[8]; /* partial_1 g: 00 01 03 11 12 13 22 33 */
  double D2[8];
};

/* The connection data at (X1, X2), the same point on the four lanes of a
 * half; o = lane & 3 selects the finite-difference offset.  xd: the half's
 * 16-double exchange area. */
__device__ __forceinline__ void gc_connection(double X1, double X2, int o, double *xd, GcPoint *p)
{
  const DevGrid &G = c_grid;
  const double a = G.a, sm = G.mks_smooth;
  /* centre */
  /* r = exp(X1) on the even lanes, E on the odd ones, swapped */
  const double x0 = exp((o & 1) ? GC_MUL(sm, GC_SUB(G.startx[1], X1)) : X1), x1 = __shfl_xor_sync(0xffffffffu, x0, 1);
  const double r = (o & 1) ? x1 : x0, E = (o & 1) ? x0 : x1;
  double S2, C2, th0, J21, J22, s0, c0;
  sincospi(GC_MUL(2., X2), &S2, &C2);
  gc_theta(X2, E, S2, C2, &th0, &J21, &J22);
  sincos(th0, &s0, &c0);
  p->r = r;
  const double s2 = GC_MUL(s0, s0), aa = GC_MUL(a, a);
  const double rho2 = GC_FMA(GC_MUL(aa, c0), c0, GC_MUL(r, r));
  double irho2;
  {
    const double rJ = GC_MUL(r, J22), p2 = GC_MUL(rho2, rJ), inv = 1. / GC_MUL(p2, s2);
    irho2 = GC_MUL(GC_MUL(inv, rJ), s2);
    const double ir = GC_MUL(GC_MUL(GC_MUL(inv, rho2), J22), s2), iJ = GC_MUL(GC_MUL(GC_MUL(inv, rho2), r), s2);
    const double is2 = GC_MUL(inv, p2), tr = GC_MUL(GC_MUL(2., r), irho2);
    const double Delta = GC_FMA(a, a, GC_FMA(-2., r, GC_MUL(r, r)));
    const double Grr = GC_MUL(Delta, irho2), Grp = GC_MUL(a, irho2), M21 = GC_MUL(GC_MUL(-J21, ir), iJ);
    Gcon &u = p->gu;
    u.u00 = -0.5 * GC_ADD(1., tr);
    u.u01 = 0.5 * GC_MUL(tr, ir);
    u.u02 = 0.5 * GC_MUL(M21, tr);
    u.u11 = 0.5 * GC_MUL(GC_MUL(ir, ir), Grr);
    u.u12 = 0.5 * GC_MUL(GC_MUL(ir, M21), Grr);
    u.u13 = 0.5 * GC_MUL(ir, Grp);
    u.u22 = 0.5 * GC_FMA(GC_MUL(iJ, iJ), irho2, GC_MUL(GC_MUL(M21, M21), Grr));
    u.u23 = 0.5 * GC_MUL(M21, Grp);
    u.u33 = 0.5 * GC_MUL(irho2, is2);
  }
  /* the lane's offset metric */
  const double Xc = o < 2 ? X1 : X2, Xh = GC_ADD(Xc, IPG_DEL), Xl = GC_SUB(Xc, IPG_DEL);
  const double Xo = (o & 1) ? Xl : Xh, d = GC_SUB(Xo, Xc); /* exact */
  const double d1 = o < 2 ? d : 0., d2 = o < 2 ? 0. : d;
  const double ro = GC_FMA(r, gc_expm_small(d1), r), Eo = GC_FMA(E, gc_expm_small(GC_MUL(-sm, d1)), E);
  double sd, cd, So, Co, tho, J21o, J22o, so, co;
  gc_sincos_small(GC_MUL(2. * IPG_PI, d2), &sd, &cd);
  gc_rotate(S2, C2, sd, cd, &So, &Co);
  gc_theta(o < 2 ? X2 : Xo, Eo, So, Co, &tho, &J21o, &J22o);
  gc_sincos_small(GC_SUB(tho, th0), &sd, &cd);
  gc_rotate(s0, c0, sd, cd, &so, &co);
  double g[8];
  {
    /* r^2 + a^2 cos^2: the X2 offsets share r^2 with the centre, so there the
     * compiler fuses the other product */
    const double q2 = GC_MUL(so, so), ac = GC_MUL(aa, co), rr = GC_MUL(ro, ro), acc2 = GC_MUL(ac, co);
    const double ro2 = GC_FMA(o < 2 ? ro : ac, o < 2 ? ro : co, o < 2 ? acc2 : rr);
    const double e = GC_MUL(GC_SUB(ro2, rho2), irho2);
    const double t = GC_MUL(GC_MUL(2., ro), GC_MUL(irho2, GC_FMA(-e, GC_SUB(1., e), 1.)));
    const double t1 = GC_ADD(1., t), mas2 = GC_MUL(-a, q2), rJ1 = GC_MUL(ro2, J21o);
    g[0] = GC_ADD(t, -1.);
    g[1] = GC_MUL(t, ro);
    g[2] = GC_MUL(mas2, t);
    g[3] = GC_FMA(rJ1, J21o, GC_MUL(GC_MUL(t1, ro), ro));
    g[4] = GC_MUL(rJ1, J22o);
    g[5] = GC_MUL(GC_MUL(mas2, t1), ro);
    g[6] = GC_MUL(GC_MUL(ro2, J22o), J22o);
    g[7] = GC_MUL(q2, GC_FMA(GC_MUL(aa, q2), t1, ro2));
  }
  /* (high - low) / (Xh - Xl): even lanes hold the high metric, odd the low */
  const double inv = gc_recip_2del(GC_SUB(Xh, Xl));
#pragma unroll
  for (int k = 0; k < 8; k++) {
    const double other = __shfl_xor_sync(0xffffffffu, g[k], 1);
    g[k] = GC_MUL((o & 1) ? GC_SUB(other, g[k]) : GC_SUB(g[k], other), inv);
  }
  __syncwarp(); /* the area's last reads are done */
  if (!(o & 1)) {
    double2 *w = reinterpret_cast<double2 *>(xd + (o >> 1) * 8);
#pragma unroll
    for (int k = 0; k < 4; k++) w[k] = make_double2(g[2 * k], g[2 * k + 1]);
  }
  __syncwarp();
  const double2 *w = reinterpret_cast<const double2 *>(xd);
#pragma unroll
  for (int k = 0; k < 4; k++) {
    const double2 x = w[k], y = w[4 + k];
    p->D1[2 * k] = x.x;
    p->D1[2 * k + 1] = x.y;
    p->D2[2 * k] = y.x;
    p->D2[2 * k + 1] = y.y;
  }
}

/* v = (partial_d g) K; last: the third product of entry 1 rounded by itself
 * (as the compiler leaves it where that product has other uses) */
template <bool LAST>
__device__ __forceinline__ void gc_dg_dot(const double D[8], const double K[4], double v[4])
{
  v[0] = GC_FMA(D[2], K[3], GC_FMA(D[0], K[0], GC_MUL(D[1], K[1])));
  const double v1 = GC_FMA(D[1], K[0], GC_MUL(D[3], K[1]));
  v[1] = GC_FMA(D[5], K[3], LAST ? GC_ADD(v1, GC_MUL(D[4], K[2])) : GC_FMA(D[4], K[2], v1));
  v[2] = GC_FMA(D[4], K[1], GC_MUL(D[6], K[2]));
  v[3] = GC_FMA(D[7], K[3], GC_FMA(D[2], K[0], GC_MUL(D[5], K[1])));
}

/* Row o of A^i_k = Gamma^i_kl K^l (transport_matrix), and acc = A K on every
 * lane; `from` is the half whose K is meant (the other half's lanes compute
 * values that nothing uses) */
__device__ __forceinline__ void gc_transport(const GcPoint &p, const double K[4], int o, int from, double A[4],
                                             double acc[4])
{
  double v1[4], v2[4];
  const double *D1 = p.D1, *D2 = p.D2;
  gc_dg_dot<false>(D1, K, v1);
  gc_dg_dot<true>(D2, K, v2);
  double d[8];
#pragma unroll
  for (int k = 0; k < 8; k++) d[k] = GC_FMA(K[1], D1[k], GC_MUL(K[2], D2[k]));
  /* 2 B[m][k] */
  double B[4][4];
  B[0][0] = d[0];
  B[0][1] = GC_ADD(d[1], v1[0]);
  B[0][2] = v2[0];
  B[0][3] = d[2];
  B[1][0] = GC_SUB(d[1], v1[0]);
  B[1][1] = GC_SUB(GC_ADD(d[3], v1[1]), v1[1]);
  B[1][2] = GC_SUB(GC_ADD(d[4], v2[1]), v1[2]);
  B[1][3] = GC_SUB(d[5], v1[3]);
  B[2][0] = -v2[0];
  B[2][1] = GC_SUB(GC_ADD(d[4], v1[2]), v2[1]);
  B[2][2] = GC_SUB(GC_ADD(d[6], v2[2]), v2[2]);
  B[2][3] = -v2[3];
  B[3][0] = d[2];
  B[3][1] = GC_ADD(d[5], v1[3]);
  B[3][2] = v2[3];
  B[3][3] = d[7];
  const Gcon &u = p.gu;
  /* row o of g^{mu nu}; row 0 fuses its second product first */
  const double r0 = o == 0 ? u.u01 : o == 1 ? u.u01 : o == 2 ? u.u02 : 0.;
  const double r1 = o == 0 ? u.u00 : o == 1 ? u.u11 : o == 2 ? u.u12 : u.u13;
  const double r2 = o == 0 ? u.u02 : o == 1 ? u.u12 : o == 2 ? u.u22 : u.u23;
  const double r3 = o == 0 ? 0. : o == 1 ? u.u13 : o == 2 ? u.u23 : u.u33;
#pragma unroll
  for (int k = 0; k < 4; k++) {
    const double b0 = o == 0 ? B[1][k] : B[0][k], b1 = o == 0 ? B[0][k] : B[1][k];
    A[k] = GC_FMA(r3, B[3][k], GC_FMA(r2, B[2][k], GC_FMA(r0, b0, GC_MUL(r1, b1))));
  }
  const double ai = GC_FMA(A[3], K[3], GC_FMA(A[2], K[2], GC_FMA(A[0], K[0], GC_MUL(A[1], K[1]))));
#pragma unroll
  for (int k = 0; k < 4; k++) acc[k] = __shfl_sync(0xffffffffu, ai, from * 4 + k, GC_LANES);
}

/* Gamma^k_ij K^i K^j without the matrix (geo_accel: unpolarized images) */
__device__ __forceinline__ void gc_accel(const GcPoint &p, const double K[4], int from, double acc[4])
{
  double v1[4], v2[4], T[4];
  gc_dg_dot<false>(p.D1, K, v1);
  gc_dg_dot<false>(p.D2, K, v2);
  const double kv1 = GC_FMA(K[3], v1[3], GC_FMA(K[2], v1[2], GC_FMA(K[0], v1[0], GC_MUL(K[1], v1[1]))));
  const double kv2 = GC_FMA(K[3], v2[3], GC_ADD(GC_FMA(K[0], v2[0], GC_MUL(K[1], v2[1])), GC_MUL(K[2], v2[2])));
#pragma unroll
  for (int m = 0; m < 4; m++) T[m] = GC_FMA(K[1], v1[m], GC_MUL(K[2], v2[m]));
  T[1] = GC_FMA(-0.5, kv1, T[1]);
  T[2] = GC_FMA(-0.5, kv2, T[2]);
  const Gcon &u = p.gu; /* half of g^{mu nu}: the results are doubled, exactly */
  acc[0] = 2. * GC_FMA(u.u02, T[2], GC_FMA(u.u01, T[1], GC_MUL(u.u00, T[0])));
  acc[1] = 2. * GC_FMA(u.u13, T[3], GC_FMA(u.u12, T[2], GC_FMA(u.u01, T[0], GC_MUL(u.u11, T[1]))));
  acc[2] = 2. * GC_FMA(u.u23, T[3], GC_FMA(u.u22, T[2], GC_FMA(u.u02, T[0], GC_MUL(u.u12, T[1]))));
  acc[3] = 2. * GC_FMA(u.u33, T[3], GC_FMA(u.u13, T[1], GC_MUL(u.u23, T[2])));
#pragma unroll
  for (int k = 0; k < 4; k++) acc[k] = __shfl_sync(0xffffffffu, acc[k], from * 4, GC_LANES);
}

/* stepsize with its roundings spelled out */
__device__ __forceinline__ double gc_stepsize(const double X[4], const double K[4], double eps)
{
  const DevGrid &G = c_grid;
  const double SS = IPG_SMALL * IPG_SMALL;
  const double cut = 0.02;
  const double deh = fmin(fabs(GC_SUB(X[1], G.cstartx[1])), 0.1);
  const double dpole = fmin(fabs(GC_MUL(X[2], G.inv_lx2)), fabs(GC_MUL(GC_SUB(G.cstopx[2], X[2]), G.inv_lx2)));
  const double d2fac = (dpole < cut) ? GC_MUL(dpole, 1. / 3.) : fmin(GC_FMA(GC_SUB(dpole, cut), 10., cut * (1. / 3.)), 1.);
  const double a1 = GC_ADD(fabs(K[1]), SS), a2 = GC_ADD(fabs(K[2]), SS), a3 = GC_ADD(fabs(K[3]), SS);
  const double b1 = GC_MUL(eps, GC_MUL(10., deh)), b2 = GC_MUL(eps, d2fac);
  const double b12 = GC_MUL(b1, b2);
  return GC_MUL(eps, b12) / GC_FMA(a3, b12, GC_MUL(eps, GC_FMA(a1, b2, GC_MUL(a2, b1))));
}

/* lanes without a ray run along, at a point that takes none of the slow
 * paths of the functions */
__device__ __forceinline__ void gc_park(GeoLane &L)
{
  L.X[0] = L.X[3] = 0.;
  L.X[1] = 1.;
  L.X[2] = 0.3;
  L.K[0] = L.K[1] = L.K[2] = L.K[3] = 1.;
}

/* The next ray of the queue for a group of GC_LANES lanes (geo_fetch over
 * the group: its first lane does the atomics and the stores).  Warp-wide
 * call; `need` selects the groups that take one.  Groups that find the queue
 * empty set *drained. */
template <class CS>
__device__ __forceinline__ void gc_fetch(GeoLane &L, bool need, bool *has, bool *drained, int gl,
                                         const int32_t *__restrict__ ij, const int32_t *__restrict__ list, int n_list,
                                         double *__restrict__ pool, int *__restrict__ chunk_prev,
                                         int2 *__restrict__ chunk_meta, long long n_chunks,
                                         unsigned long long *__restrict__ counters, int queue,
                                         RayRec *__restrict__ rays, int32_t *__restrict__ deferred,
                                         const int32_t *__restrict__ ray_grp)
{
  while (__any_sync(0xffffffffu, need)) {
    unsigned long long t = 0, c = 0;
    int stop = 0;
    if (need && gl == 0) {
      t = atomicAdd(&counters[queue], 1ULL);
      if (t >= (unsigned long long)n_list) stop = 1;
      if constexpr (CS::batch) {
        /* a batch's step budget: once it is spent no further ray starts */
        const unsigned long long budget = counters[CNT_BUDGET];
        if (!stop && budget && *(volatile unsigned long long *)&counters[CNT_STEPS] >= budget) {
          counters[CNT_TIMEOUT] = 1;
          stop = 1;
        }
      }
      if (!stop) {
        const int ray = list ? list[t] : (int)t;
        c = atomicAdd(&counters[CNT_POOL], 1ULL);
        if ((long long)c >= n_chunks) {
          RayRec rec = {-1, 0, IPG_RAY_POOL_FULL, 0};
          rays[ray] = rec;
          deferred[atomicAdd(&counters[CNT_DEFER], 1ULL)] = ray;
        }
      }
    }
    stop = __shfl_sync(0xffffffffu, stop, 0, GC_LANES);
    t = __shfl_sync(0xffffffffu, t, 0, GC_LANES);
    c = __shfl_sync(0xffffffffu, c, 0, GC_LANES);
    if (!need) continue;
    if (stop) {
      gc_park(L);
      *drained = true;
      need = false;
      continue;
    }
    if ((long long)c >= n_chunks) continue;
    const int ray = list ? list[t] : (int)t;
    const int grp = CS::batch ? ray_grp[ray] : 0;
    const DevCam &C = CS::get(grp);
    L.ray = ray;
    L.grp = grp;
    init_ray(C, ij[2 * ray], ij[2 * ray + 1], L.X, L.K);
#pragma unroll
    for (int k = 0; k < 4; k++) {
      L.Xh[k] = L.X[k];
      L.Kh[k] = L.K[k];
    }
    L.chunk = (int)c;
    L.prev = step_ptr(pool, L.chunk, 0);
    if (gl == 0) {
      chunk_prev[L.chunk] = -1;
      chunk_meta[L.chunk] = make_int2(ray, 0);
      store_geo(L.prev, L.X, L.K, L.Xh, L.Kh, 0., 0., C.mixed);
    }
    L.nstep = 0;
    L.h = 0.;
    L.passed = (C.Xcam[2] < 0.5) ? 1 : ((C.Xcam[2] > 0.5) ? -1 : 0);
    L.nturns = 0;
    L.X1m1 = L.X1m2 = L.X[1];
    L.X2m1 = L.X2m2 = L.X[2];
    *has = true;
    need = false;
  }
}

/* row i of A1 (which = 0) or A2 (which = 1) into a record */
template <bool MIXED>
__device__ __forceinline__ void gc_store_row(double *rec, int which, int i, const double A[4])
{
  if constexpr (MIXED)
    reinterpret_cast<float4 *>(reinterpret_cast<float *>(rec) + (which ? RECM_A2F : RECM_A1F))[i] =
        make_float4((float)A[0], (float)A[1], (float)A[2], (float)A[3]);
  else
    store4(rec + (which ? REC_A2 : REC_A1) + 4 * i, A[0], A[1], A[2], A[3]);
}

/* POL: polarized images (the transport matrices are stored), MIXED: compact
 * records; compiled apart, since every branch of the step costs a lone warp
 * some 20 cycles */
template <bool POL, bool MIXED, int TPB = 32, class CS = CamOne>
__global__ void __launch_bounds__(TPB)
    k_geodesic_coop(const int32_t *__restrict__ ij, const int32_t *__restrict__ list, int n_list,
                    double *__restrict__ pool, int *__restrict__ chunk_prev, int2 *__restrict__ chunk_meta,
                    long long n_chunks, unsigned long long *__restrict__ counters, int queue,
                    RayRec *__restrict__ rays, int32_t *__restrict__ deferred, const int32_t *__restrict__ ray_grp,
                    int warps, int *started = nullptr)
{
  /* a wide block's other warps only hold its registers */
  if ((int)(threadIdx.x >> 5) >= warps) return;
  if (started && threadIdx.x == 0) {
    *(volatile int *)(started + blockIdx.x) = 1;
    __threadfence_system();
  }
  __shared__ __align__(16) double xch[TPB / 4][18]; /* per half: D1, D2; 144-byte stride */
  const DevGrid &G = c_grid;
  const int gl = threadIdx.x % GC_LANES, half = gl >> 2, o = gl & 3;
  double *xd = xch[threadIdx.x >> 2];
  GeoLane L;
  L.ray = L.grp = L.nstep = 0;
  gc_park(L);
  bool has = false, drained = false;
#define GC_FETCH()                                                                                                 \
  gc_fetch<CS>(L, !has && !drained, &has, &drained, gl, ij, list, n_list, pool, chunk_prev, chunk_meta, n_chunks, \
               counters, queue, rays, deferred, ray_grp)
  GC_FETCH();
  while (__any_sync(0xffffffffu, has)) {
    const DevCam &C = CS::get(L.grp);
    L.h = -gc_stepsize(L.X, L.K, C.eps);
    const double hh = 0.5 * L.h;
#pragma unroll
    for (int k = 0; k < 4; k++) L.Xh[k] = GC_FMA(hh, L.K[k], L.X[k]);
    GcPoint p;
    gc_connection(half ? L.Xh[1] : L.X[1], half ? L.Xh[2] : L.X[2], o, xd, &p);
    /* stop_backward_integration, src/model_geodesics.c:218-254, and the step
     * limit of trace_geodesic's loop (:71) */
    const double r = __shfl_sync(0xffffffffu, p.r, 0, GC_LANES);
    const bool stop = (r > G.rmax_geo && L.K[1] < 0.) || r < (G.Rh + 0.0001) || !(L.nstep < C.maxnstep - 1);
    double A[4], acc[4];
    if constexpr (POL) {
      gc_transport(p, L.K, o, 0, A, acc);
      /* the walk back starts at the last point: its Gamma(X) K too; a ray
       * that ends at maxnstep or at its first point needs none */
      const bool no_A = stop && (L.nstep >= C.maxnstep - 1 || L.nstep == 0);
      if (has && half == 0 && !no_A) gc_store_row<MIXED>(L.prev, 0, o, A);
    } else {
      gc_accel(p, L.K, 0, acc);
    }
    if (has && stop) {
      if (gl == 0) {
        RayRec rec = {L.chunk, L.nstep, (L.nstep >= C.maxnstep - 1) ? IPG_RAY_MAXNSTEP : IPG_RAY_OK, 0};
        rays[L.ray] = rec;
        atomicAdd(&counters[CNT_STEPS], (unsigned long long)L.nstep);
      }
      has = false;
    }
#pragma unroll
    for (int k = 0; k < 4; k++) L.Kh[k] = GC_FMA(-hh, acc[k], L.K[k]);
    if constexpr (POL) gc_transport(p, L.Kh, o, 1, A, acc);
    else gc_accel(p, L.Kh, 1, acc);
    L.nstep += has;
#pragma unroll
    for (int k = 0; k < 4; k++) {
      const double Kn = GC_FMA(-L.h, acc[k], L.K[k]), Xn = GC_FMA(L.h, L.Kh[k], L.X[k]);
      L.K[k] = has ? Kn : L.K[k];
      L.X[k] = has ? Xn : L.X[k];
    }
    const int slot = L.nstep % IPG_CHUNK_STEPS;
    const bool grow = has && slot == 0;
    /* the rare parts of an iteration behind one vote */
    const bool rare = __any_sync(0xffffffffu, grow || (!has && !drained) || C.target_nturns >= 0);
    if (rare) {
      if (has && C.target_nturns >= 0) count_turns<IPG_MET_FMKS>(C, L);
      unsigned long long nc = 0;
      if (grow && gl == 0) {
        nc = atomicAdd(&counters[CNT_POOL], 1ULL);
        if ((long long)nc >= n_chunks) {
          RayRec rec = {L.chunk, L.nstep, IPG_RAY_POOL_FULL, 0};
          rays[L.ray] = rec;
          deferred[atomicAdd(&counters[CNT_DEFER], 1ULL)] = L.ray;
        } else {
          chunk_prev[(int)nc] = L.chunk;
          chunk_meta[(int)nc] = make_int2(L.ray, L.nstep);
        }
      }
      nc = __shfl_sync(0xffffffffu, nc, 0, GC_LANES);
      if (grow) {
        if ((long long)nc >= n_chunks) has = false;
        else L.chunk = (int)nc;
      }
    }
    if (has) {
      L.prev = step_ptr(pool, L.chunk, slot);
      const double dl = -L.h;
      const double dl_cgs = dl * G.L_unit * IPG_HPL / (IPG_ME * IPG_CL * IPG_CL);
      if (POL && half == 1) gc_store_row<MIXED>(L.prev, 1, o, A); /* Gamma(Xh_n) Kh_n */
      if (gl == 0) store_geo(L.prev, L.X, L.K, L.Xh, L.Kh, dl_cgs, (double)L.nturns, MIXED);
    }
    if (rare) GC_FETCH();
  }
#undef GC_FETCH
}

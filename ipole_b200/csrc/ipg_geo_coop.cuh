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
 * The records are k_geodesic's bits: both kernels are built from the
 * explicitly rounded functions of ipg_connection.cuh, of which each lane here
 * evaluates its share.
 *
 * Included by ipg_kernels.cu.
 */

#define GC_LANES 8

/* 1 / x, correctly rounded, for x = 2 DEL (1 + d), |d| < 2^-18.  With y0 =
 * 1 / (2 DEL) and e0 = 1 - x y0, 1 / x = y0 (1 + e0 + e0^2 + ...): y1 leaves
 * out e0^3 < 2^-54 of it and one rounding, so it is within an ulp; from there
 * one step with the exact residual 1 - x y1 rounds correctly, for every x but
 * one whose mantissa is all ones (Markstein 1990), which the interval does not
 * hold.  Xh - Xl has |d| < 2^-26 for |X| < 16 (the roundings of X +- DEL).
 * ipg__check_recip compares it with the division, which costs the polarized
 * step 0.8% more (16 rays 6.03 -> 6.07 ms). */
__device__ __forceinline__ double gc_recip_2del(double x)
{
  const double y0 = 1. / (2. * IPG_DEL);
  const double e0 = RN_FMA(-x, y0, 1.);
  const double y1 = RN_FMA(RN_FMA(e0, e0, e0), y0, y0);
  return RN_FMA(RN_FMA(-x, y1, 1.), y1, y1);
}

/* The connection at (X1, X2) (HALF: with half of g^{mu nu}), the same point on
 * the four lanes of a half; o = lane & 3 selects the finite-difference offset.
 * xd: the half's 16-double exchange area. */
template <bool HALF>
__device__ __forceinline__ void gc_connection(double X1, double X2, int o, double *xd, Conn *p)
{
  const DevGrid &G = c_grid;
  const double sm = G.mks_smooth;
  /* r = exp(X1) on the even lanes, E on the odd ones, swapped */
  const double x0 = exp((o & 1) ? RN_MUL(sm, RN_SUB(G.startx[1], X1)) : X1), x1 = __shfl_xor_sync(0xffffffffu, x0, 1);
  ConnCentre c;
  conn_centre<true, HALF>((o & 1) ? x1 : x0, (o & 1) ? x0 : x1, X2, &c, &p->gu);
  p->r = c.r;
  /* the lane's offset metric */
  const double Xc = o < 2 ? X1 : X2, Xh = RN_ADD(Xc, IPG_DEL), Xl = RN_SUB(Xc, IPG_DEL);
  const double Xo = (o & 1) ? Xl : Xh, d = RN_SUB(Xo, Xc); /* exact */
  const double d1 = o < 2 ? d : 0., d2 = o < 2 ? 0. : d;
  const double ro = RN_FMA(c.r, expm_small(d1), c.r), Eo = RN_FMA(c.E, expm_small(RN_MUL(-sm, d1)), c.E);
  const double X2o = o < 2 ? X2 : Xo;
  double sd, cd, S, C, g[8];
  sincos_small(RN_MUL(2. * IPG_PI, d2), &sd, &cd);
  rotate(c.p.S2, c.p.C2, sd, cd, &S, &C);
  X2P po;
  x2_parts_from<true>(X2o, S, C, &po);
  ConnOffset off;
  conn_offset(c, Eo, X2o, po, &off);
  conn_near(c, ro, off, o >= 2, g);
  /* (high - low) / (Xh - Xl): even lanes hold the high metric, odd the low */
  const double inv = gc_recip_2del(RN_SUB(Xh, Xl));
#pragma unroll
  for (int k = 0; k < 8; k++) {
    const double other = __shfl_xor_sync(0xffffffffu, g[k], 1);
    g[k] = RN_MUL((o & 1) ? RN_SUB(other, g[k]) : RN_SUB(g[k], other), inv); /* conn_diff */
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

/* Row o of A^i_k = Gamma^i_kl K^l, and acc = A K on every lane; `from` is the
 * half whose K is meant (the other half's lanes compute values that nothing
 * uses) */
__device__ __forceinline__ void gc_transport(const Conn &p, const double K[4], int o, int from, double A[4],
                                             double acc[4])
{
  double B[4][4];
  transport_b(p, K, B);
  transport_row(p.gu, B, o, A);
  const double ai = transport_accel(A, K);
#pragma unroll
  for (int k = 0; k < 4; k++) acc[k] = __shfl_sync(0xffffffffu, ai, from * 4 + k, GC_LANES);
}

/* Gamma^k_ij K^i K^j without the matrix (unpolarized images) */
__device__ __forceinline__ void gc_accel(const Conn &p, const double K[4], int from, double acc[4])
{
  geo_accel(p, K, acc);
#pragma unroll
  for (int k = 0; k < 4; k++) acc[k] = __shfl_sync(0xffffffffu, acc[k], from * 4, GC_LANES);
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
    L.h = -stepsize(L.X, L.K, C.eps);
    const double hh = 0.5 * L.h;
    geo_advance(L.X, hh, L.K, L.Xh);
    Conn p;
    gc_connection<POL>(half ? L.Xh[1] : L.X[1], half ? L.Xh[2] : L.X[2], o, xd, &p);
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
    geo_advance(L.K, -hh, acc, L.Kh);
    if constexpr (POL) gc_transport(p, L.Kh, o, 1, A, acc);
    else gc_accel(p, L.Kh, 1, acc);
    L.nstep += has;
    /* geo_advance of K and X, component by component: in this order, and with
     * hh once, the compiler's schedule is 0.5% (polarized) to 4% (a batch's
     * cameras) shorter than with two whole calls */
#pragma unroll
    for (int k = 0; k < 4; k++) {
      const double Kn = RN_FMA(-L.h, acc[k], L.K[k]), Xn = RN_FMA(L.h, L.Kh[k], L.X[k]);
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

/* Self-check of gc_recip_2del against the division: n arguments of each kind,
 * 0: Xh - Xl of X in -1 .. 16, 1: 2 DEL (1 + d), |d| < width, 2: the doubles
 * next to 2 DEL and to both ends of that interval */
__global__ void k_check_recip(int n, unsigned long long seed, double width, unsigned long long *bad)
{
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  unsigned long long z = (seed + i) * 0x9e3779b97f4a7c15ULL;
  z = (z ^ (z >> 30)) * 0xbf58476d1ce4e5b9ULL;
  z = (z ^ (z >> 27)) * 0x94d049bb133111ebULL;
  z ^= z >> 31;
  const double u = (double)(z >> 11) * (1. / 9007199254740992.), X = 17. * u - 1.;
  const double c = 2. * IPG_DEL * (1. + (double)(i % 3 - 1) * width * (1. - 1e-9));
  const double x[3] = {RN_SUB(RN_ADD(X, IPG_DEL), RN_SUB(X, IPG_DEL)), 2. * IPG_DEL * (1. + (2. * u - 1.) * width),
                       __longlong_as_double(__double_as_longlong(c) + (i % 3 == 1 ? i / 3 - n / 6 : i % 3 ? -(i / 3) : i / 3))};
  for (int k = 0; k < 3; k++)
    if (gc_recip_2del(x[k]) != 1. / x[k]) atomicAdd(bad + k, 1ULL);
}

extern "C" int ipg__check_recip(int device, int n, unsigned long long seed, double width, unsigned long long bad[3])
{
  if (n <= 0 || !bad || cudaSetDevice(device) != cudaSuccess) return IPG_E_ARG;
  unsigned long long *d = nullptr;
  if (cudaMalloc(&d, 3 * sizeof(*d)) != cudaSuccess) return IPG_E_CUDA;
  cudaMemset(d, 0, 3 * sizeof(*d));
  k_check_recip<<<(n + 255) / 256, 256>>>(n, seed, width, d);
  const cudaError_t e = cudaMemcpy(bad, d, 3 * sizeof(*d), cudaMemcpyDeviceToHost);
  cudaFree(d);
  return e == cudaSuccess ? IPG_OK : IPG_E_CUDA;
}

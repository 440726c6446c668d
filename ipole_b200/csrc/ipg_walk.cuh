/*
 * The transfer walk with four or more lanes per ray (k_walk).
 *
 * k_transfer gives one lane a ray: each step is then a chain of ~1080
 * dependent instructions (2.3 us for a lone ray, 3-7 us beside other work),
 * and the longest ray's 16e3 steps set the time of every image.  Here a warp
 * walks 32/G rays, G lanes each, over blocks of G consecutive records per
 * ray, in two phases:
 *
 *   A  one lane per record: everything of the step that does not depend on
 *      N - the Stokes map T, u of stokes_map (or the FP32 step's factors),
 *      the unpolarized step's p, q, the optical depths.  All its sines,
 *      exponentials and divisions run 32 records side by side, so the chain
 *      of steps does not wait for them.
 *   B  the G steps in order, each shared out over the ray's lanes: lane j
 *      (mod 4) holds column j of Re N and Im N, forms column j of A N from
 *      the record's matrices in shared memory, and swaps it for row j
 *      through shared memory (the push needs A N + (A N)^T); the Stokes
 *      projection's partial sums are swapped the same way.
 *
 * A lone ray's step is then a chain of ~45 dependent FP64 operations and
 * four exchanges.  With G = 4 a warp works on eight rays at once
 * (throughput); with G = 32 on one, 32 records per phase A (latency).
 *
 * Records arrive by one bulk copy each into the block's slots, counted on
 * the ray's mbarrier; a slot is refilled with the next block's record as
 * soon as its step is done, so only the last slot's copy can be waited for.
 * Every wait is bounded: a copy that has not landed after IPG_WALK_SPINS
 * polls sets CNT_STALL, the warp gives its copies in flight their bounded
 * wait and ends, and the host fails the call.
 *
 * The sums and products are those of xfer_push / xfer_evolve with the same
 * roundings (dot4_rn, hn_upd_r, ...), so the images are k_transfer's bits.
 *
 * Included by ipg_kernels.cu.
 */

#ifndef IPG_WALK_SPINS
#define IPG_WALK_SPINS (1u << 20)
#endif
__device__ __forceinline__ unsigned smem_u32(const void *p) { return (unsigned)__cvta_generic_to_shared(p); }

/* waits for the barrier's phase `parity` to complete; false if it did not
 * within the bound */
__device__ __forceinline__ bool walk_wait(unsigned long long *bar, unsigned parity)
{
  for (unsigned it = 0; it < IPG_WALK_SPINS; it++) {
    unsigned ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(smem_u32(bar)), "r"(parity)
        : "memory");
    if (ok) return true;
  }
  return false;
}
__device__ __forceinline__ void walk_expect(unsigned long long *bar, unsigned bytes)
{
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes) : "memory");
}
__device__ __forceinline__ void walk_copy(void *dst, const void *src, unsigned bytes, unsigned long long *bar)
{
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                   smem_u32(dst)),
               "l"(src), "r"(bytes), "r"(smem_u32(bar))
               : "memory");
}
/* orders the lanes' reads of a slot before the copy that refills it */
__device__ __forceinline__ void walk_refill_fence() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }
__device__ __forceinline__ void walk_prefetch_l2(const void *src, unsigned bytes)
{
  asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(src), "r"(bytes) : "memory");
}

/* Shared memory of a warp: per ray G record slots (the record, its factors
 * over the coefficients once these are read, and the extra factors behind
 * it), then the exchange areas of the rays.  Phase A reads one slot per lane,
 * phase B one slot per ray, both in 16-byte accesses of which a quarter-warp
 * and a ray each should hit banks of their own: in units of 16 bytes modulo 8
 * the rays' stride is odd, and the slots' stride odd, or even but not a
 * multiple of 4 where a quarter-warp holds two rays (G = 4).  (With one stride
 * for both, eight rays' reads fell into a quarter of the banks, a 5-way
 * conflict; a 160x160 image's 25 600 rays: 12.0 ms then, 10.8 now.)  The
 * exchange stride is 32 modulo 128, so that four rays' 32-byte rows do. */
template <int G, int RM>
struct WalkSm {
  static constexpr int RAYS = 32 / G;
  static constexpr int COPY = RM ? 320 : 512;
  static constexpr int FT = RM ? RECM_COEF * 8 : REC_FLAGS * 8; /* the coefficient block's 128 bytes */
  static constexpr int FX = COPY;                               /* 10 doubles: u, p, q, dtau, dtauF, dl, - */
  static constexpr int SLOT = COPY + (G == 4 ? 96 : 80);
  static constexpr int RAY = G * SLOT + 16;
  static constexpr int XCH = 544; /* A N of the half and of the full push (256 each) */
  static constexpr int BYTES = RAYS * (RAY + XCH);
  static_assert((G == 4 ? SLOT % 64 == 32 : SLOT % 32 == 16) && RAY % 32 == 16 && XCH % 128 == 32, "bank layout");
};

/* Column j of N: R[.][j] and S[.][j] (S[j][j] = 0) */
struct WalkN {
  double r[4], s[4];
};

__device__ __forceinline__ void walk_ld4(const double *p, double v[4])
{
  const double2 a = reinterpret_cast<const double2 *>(p)[0], b = reinterpret_cast<const double2 *>(p)[1];
  v[0] = a.x;
  v[1] = a.y;
  v[2] = b.x;
  v[3] = b.y;
}

/* a record's transport matrix, from its slot in shared memory */
template <int RM>
struct WalkMat {
  typedef double T;
};
template <>
struct WalkMat<1> {
  typedef float T;
};
__device__ __forceinline__ void walk_ldA(const double *A, double a[4][4])
{
#pragma unroll
  for (int i = 0; i < 4; i++) walk_ld4(A + 4 * i, a[i]);
}
__device__ __forceinline__ void walk_ldA(const double *A, float a[4][4])
{
#pragma unroll
  for (int i = 0; i < 4; i++) {
    const float4 v = reinterpret_cast<const float4 *>(A)[i];
    a[i][0] = v.x;
    a[i][1] = v.y;
    a[i][2] = v.z;
    a[i][3] = v.w;
  }
}

/* out = base - dl (A M + M A^T) for the lane's column (hn_push) */
template <class T>
__device__ __forceinline__ void walk_push(const WalkN &base, const WalkN &M, const T a[4][4], double dl, int j,
                                          double *xr, WalkN *out)
{
  double ar[4], as[4], tr[4], ts[4];
#pragma unroll
  for (int i = 0; i < 4; i++) {
    const double ai[4] = {(double)a[i][0], (double)a[i][1], (double)a[i][2], (double)a[i][3]};
    ar[i] = dot4_rn(ai, M.r);
    as[i] = dot4_rn(ai, M.s);
    xr[4 * i + j] = ar[i];
    xr[16 + 4 * i + j] = as[i];
  }
  __syncwarp();
  walk_ld4(xr + 4 * j, tr);
  walk_ld4(xr + 16 + 4 * j, ts);
#pragma unroll
  for (int i = 0; i < 4; i++) {
    out->r[i] = __fma_rn(-dl, __dadd_rn(ar[i], tr[i]), base.r[i]);
    out->s[i] = __fma_rn(-dl, __dsub_rn(as[i], ts[i]), base.s[i]);
  }
}

/* the same with hn_push_f32's FP32 increments */
template <class T>
__device__ __forceinline__ void walk_push_f32(const WalkN &base, const WalkN &M, const T a[4][4], double dl, int j,
                                              double *xr, WalkN *out)
{
  double big = fabs(j == 0 ? M.r[0] : j == 1 ? M.r[1] : j == 2 ? M.r[2] : M.r[3]);
  big = fmax(big, __shfl_xor_sync(0xffffffffu, big, 1));
  big = fmax(big, __shfl_xor_sync(0xffffffffu, big, 2));
  big = fmax(big, 1e-300);
  const int ex = pow2_exponent(big);
  const double sc = pow2(-ex), us = __dmul_rn(dl, pow2(ex));
  float r[4], s[4], ar[4], as[4];
#pragma unroll
  for (int i = 0; i < 4; i++) {
    r[i] = (float)(M.r[i] * sc);
    s[i] = (float)(M.s[i] * sc);
  }
  float *xf = reinterpret_cast<float *>(xr);
#pragma unroll
  for (int i = 0; i < 4; i++) {
    const float a0 = (float)a[i][0], a1 = (float)a[i][1], a2 = (float)a[i][2], a3 = (float)a[i][3];
    ar[i] = dot4f_rn(a0, a1, a2, a3, r[0], r[1], r[2], r[3]);
    as[i] = dot4f_rn(a0, a1, a2, a3, s[0], s[1], s[2], s[3]);
    xf[4 * i + j] = ar[i];
    xf[16 + 4 * i + j] = as[i];
  }
  __syncwarp();
  const float4 tr = *reinterpret_cast<const float4 *>(xf + 4 * j), ts = *reinterpret_cast<const float4 *>(xf + 16 + 4 * j);
  const float trv[4] = {tr.x, tr.y, tr.z, tr.w}, tsv[4] = {ts.x, ts.y, ts.z, ts.w};
#pragma unroll
  for (int i = 0; i < 4; i++) {
    out->r[i] = __fma_rn(-us, (double)(ar[i] + trv[i]), base.r[i]);
    out->s[i] = __fma_rn(-us, (double)(as[i] - tsv[i]), base.s[i]);
  }
}

/* hn_stokes over the ray's lanes: lane j forms entry j of R e1, R e2, S e1
 * and its share of the four sums, which a butterfly adds up */
__device__ __forceinline__ void walk_stokes(const WalkN &N, const double e1[4], const double e2[4], int j, double *T11,
                                            double *T22, double *T12r, double *T21i)
{
  const double re1 = dot4_rn(N.r, e1), re2 = dot4_rn(N.r, e2), se1 = -dot4_rn(N.s, e1); /* S[j][.] = -S[.][j] */
  const double e1j = j == 0 ? e1[0] : j == 1 ? e1[1] : j == 2 ? e1[2] : e1[3];
  const double e2j = j == 0 ? e2[0] : j == 1 ? e2[1] : j == 2 ? e2[2] : e2[3];
  double t[4] = {__dmul_rn(e1j, re1), __dmul_rn(e2j, re2), __dmul_rn(e1j, re2), __dmul_rn(e2j, se1)};
#pragma unroll
  for (int o = 1; o <= 2; o <<= 1)
#pragma unroll
    for (int i = 0; i < 4; i++) t[i] = __dadd_rn(t[i], __shfl_xor_sync(0xffffffffu, t[i], o));
  *T11 = t[0];
  *T22 = t[1];
  *T12r = t[2];
  *T21i = t[3];
}

/* a tetrad row of a record in shared memory, FP64 or compact */
template <int RM>
__device__ __forceinline__ void walk_row(const unsigned char *slot, int row, double v[4])
{
  if constexpr (RM) {
    const float4 f = reinterpret_cast<const float4 *>(slot + RECM_TETF * 4)[row];
    v[0] = f.x;
    v[1] = f.y;
    v[2] = f.z;
    v[3] = f.w;
  } else {
    walk_ld4(reinterpret_cast<const double *>(slot) + REC_E1COV + 4 * row, v);
  }
}

/* phase A for one record: its factors, from its coefficients, into FT / FX */
template <bool S32>
__device__ __forceinline__ void walk_factors(const double c[8], double dl, int unpol, double ji, double ki, double jf,
                                             double kf, double *ft, double *fx)
{
  double p, q, dtau;
  unpol_map(ji, ki, jf, kf, dl, &p, &q, &dtau);
  double2 *x2 = reinterpret_cast<double2 *>(fx);
  x2[2] = make_double2(p, q);
  x2[3] = make_double2(dtau, __dmul_rn(dl, fabs(c[7])));
  if (unpol) return;
  if constexpr (S32) {
    StepF32 F;
    step_f32_factors(c[0], c[1], c[2], c[3], c[4], c[5], c[6], c[7], dl, &F);
    float4 *f4 = reinterpret_cast<float4 *>(ft);
    f4[0] = make_float4(F.fc, F.fs, F.fg, F.nQ);
    f4[1] = make_float4(F.nV, F.tI, F.tQ, F.tV);
    f4[2] = make_float4(F.tP, F.itP2, F.ih, F.em);
    f4[3] = make_float4(F.ep, F.e0, F.q0, F.qm);
    f4[4] = make_float4(F.qp, F.pol ? 1.f : 0.f, 0.f, 0.f);
    double2 *d2 = reinterpret_cast<double2 *>(ft + 10);
    d2[0] = make_double2(F.jxI, F.jxQ);
    d2[1] = make_double2(F.jxV, 0.);
  } else {
    StokesMap m;
    stokes_map(c[0], c[1], c[2], c[3], c[4], c[5], c[6], c[7], dl, &m);
    double2 *t2 = reinterpret_cast<double2 *>(ft);
#pragma unroll
    for (int k = 0; k < 8; k++) t2[k] = make_double2(m.T[2 * k], m.T[2 * k + 1]);
    x2[0] = make_double2(m.u[0], m.u[1]);
    x2[1] = make_double2(m.u[2], m.u[3]);
  }
}

/* the polarized step's S before -> S after, from the factors: lane j
 * evaluates component j of the map (FP64), every lane the FP32 step */
template <bool S32>
struct WalkFac;
template <>
struct WalkFac<false> {
  double T[4], u;
  __device__ __forceinline__ void load(const double *ft, const double *fx, int j)
  {
    walk_ld4(ft + 4 * j, T);
    u = fx[j];
  }
  __device__ __forceinline__ void apply(double SI, double SQ, double SU, double SV, double *SIo, double *SQo,
                                        double *SUo, double *SVo) const
  {
    const double s = stokes_row(T, u, SI, SQ, SU, SV);
    *SIo = __shfl_sync(0xffffffffu, s, 0, 4);
    *SQo = __shfl_sync(0xffffffffu, s, 1, 4);
    *SUo = __shfl_sync(0xffffffffu, s, 2, 4);
    *SVo = __shfl_sync(0xffffffffu, s, 3, 4);
  }
};
template <>
struct WalkFac<true> {
  StepF32 F;
  __device__ __forceinline__ void load(const double *ft, const double *, int)
  {
    const float4 *f4 = reinterpret_cast<const float4 *>(ft);
    const float4 a = f4[0], b = f4[1], c = f4[2], d = f4[3], e = f4[4];
    const double2 j0 = reinterpret_cast<const double2 *>(ft + 10)[0], j1 = reinterpret_cast<const double2 *>(ft + 10)[1];
    F.fc = a.x; F.fs = a.y; F.fg = a.z; F.nQ = a.w;
    F.nV = b.x; F.tI = b.y; F.tQ = b.z; F.tV = b.w;
    F.tP = c.x; F.itP2 = c.y; F.ih = c.z; F.em = c.w;
    F.ep = d.x; F.e0 = d.y; F.q0 = d.z; F.qm = d.w;
    F.qp = e.x;
    F.pol = e.y != 0.f;
    F.jxI = j0.x;
    F.jxQ = j0.y;
    F.jxV = j1.x;
  }
  __device__ __forceinline__ void apply(double SI, double SQ, double SU, double SV, double *SIo, double *SQo,
                                        double *SUo, double *SVo) const
  {
    step_f32_apply(F, SI, SQ, SU, SV, SIo, SQo, SUo, SVo);
  }
};

/* RM: record layout (0 FP64, 1 compact); ADJ (the adjoint's forward pass,
 * FP64 records): a radiating record is left with what the adjoint reads of
 * the step that ends there: the Stokes vector before the step, the step's
 * length, and bit 256 of its flags where the step had no emission */
/* BATCH: the items of a batch wave.  Item t of the list is instance slot
 * xf_slot[t] of the trajectory xf_geo[t]; its coefficients come from the
 * instance's blocks of the side pool (IPG_BCOEF doubles per record, by a
 * second bulk copy into the factors' area, which is written once they are
 * read), the rest from the record that the instances share. */
struct WalkBatch {
  const double *side;
  int slots; /* instance slots per camera group */
  const int32_t *xf_geo, *xf_slot, *geo_grp;
  int32_t *deferred;
};
template <int G, bool S32, int RM, bool ADJ = false, bool BATCH = false>
__global__ void __launch_bounds__(32)
    k_walk(const int32_t *__restrict__ list, int n_list, const double *__restrict__ pool,
           const int *__restrict__ chunk_prev, const RayRec *__restrict__ rays, ipg_pixel_out *__restrict__ out,
           unsigned long long *__restrict__ counters, int queue, const WalkBatch B = WalkBatch())
{
  static_assert(!ADJ || (RM == 0 && !S32), "the adjoint's records are FP64");
  static_assert(G == 4 || G == 8 || G == 16 || G == 32, "lanes per ray");
  using W = WalkSm<G, RM>;
  constexpr unsigned BYTES = W::COPY + (BATCH ? IPG_BCOEF * 8 : 0); /* copied per record */
  static_assert(W::COPY + IPG_BCOEF * 8 <= W::SLOT, "the coefficient block fits the factors' area");
  constexpr int CB = IPG_CHUNK_STEPS / G; /* blocks per chunk */
  constexpr unsigned GM = G == 32 ? 0xffffffffu : (1u << (G & 31)) - 1u;
  extern __shared__ __align__(16) unsigned char wsm[];
  __shared__ __align__(8) unsigned long long wbar[W::RAYS];
  const int lane = threadIdx.x, grp = lane / G, q = lane % G, j = lane & 3;
  unsigned char *const slots = wsm + grp * W::RAY;
  double *const xch = reinterpret_cast<double *>(wsm + W::RAYS * W::RAY + grp * W::XCH);
  unsigned long long *const bar = wbar + grp;
  if (q == 0) asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(bar)) : "memory");
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  __syncwarp();
  const DevGrid &Gd = c_grid;
  const int unpol = BATCH ? c_cams[0].unpol : c_cam.unpol; /* a batch's instances share it */
  int cam = 0, kslot = 0;
  /* record r (0 .. 31) of chunk ch into slot sl of the ray */
  auto copy = [&](int sl, int ch, int r) {
    walk_copy(slots + sl * W::SLOT, step_ptr(const_cast<double *>(pool), ch, r), W::COPY, bar);
    if constexpr (BATCH)
      walk_copy(slots + sl * W::SLOT + W::FX, B.side + (((size_t)ch * IPG_CHUNK_STEPS + r) * B.slots + kslot) * IPG_BCOEF,
                IPG_BCOEF * 8, bar);
  };
  unsigned ph = 0;
  bool has = false, drained = false;
  int ray = 0, n0 = 0, blk = 0, chunk = 0, cprev = -1, flag = 0;
  unsigned long long nrad = 0;
  double dl_up = 0., nt_up = 0., js = 0., ks = 0.; /* of the record above the block; last radiating record's */
  double I = 0., tau = 0., tauF = 0.;
  WalkN N;
#pragma unroll
  for (int i = 0; i < 4; i++) N.r[i] = N.s[i] = 0.;
  while (true) {
    /* rays without work take the next one whose trajectory is complete;
     * rays that hit maxnstep get an all-zero result, deferred rays are left
     * for their next wave */
    while (__any_sync(0xffffffffu, !has && !drained)) {
      unsigned long long t = 0;
      const bool want = !has && !drained;
      if (want && q == 0) {
        bool stop = false;
        if constexpr (BATCH) {
          /* the batch's step budget: once it is spent no further item starts */
          const unsigned long long budget = counters[CNT_BUDGET];
          if (budget && *(volatile unsigned long long *)&counters[CNT_XSTEPS] +
                                *(volatile unsigned long long *)&counters[CNT_STEPS] >=
                            budget) {
            counters[CNT_TIMEOUT] = 1;
            stop = true;
          }
        }
        t = stop ? ~0ULL : atomicAdd(&counters[queue], 1ULL);
      }
      t = __shfl_sync(0xffffffffu, t, 0, G);
      if (!want) continue;
      if (t >= (unsigned long long)n_list) {
        drained = true;
        continue;
      }
      ray = list ? list[t] : (int)t;
      const int geo = BATCH ? B.xf_geo[ray] : ray;
      const RayRec rec = rays[geo];
      if (rec.status == IPG_RAY_POOL_FULL) {
        if constexpr (BATCH)
          if (q == 0) B.deferred[atomicAdd(&counters[CNT_XDEFER], 1ULL)] = ray;
        continue;
      }
      if (rec.status == IPG_RAY_MAXNSTEP) {
        if (q == 0) {
          ipg_pixel_out o;
          o.I_unpol = o.tau = o.tauF = o.I = o.Q = o.U = o.V = 0.;
          o.nstep = rec.nstep;
          o.flag = 0;
          out[ray] = o;
        }
        continue;
      }
      has = true;
      if constexpr (BATCH) {
        cam = B.geo_grp[geo];
        kslot = B.xf_slot[ray];
      }
      n0 = rec.nstep;
      blk = n0 / G;
      chunk = rec.last_chunk;
      cprev = chunk_prev[chunk];
      flag = 0;
      I = tau = tauF = 0.;
#pragma unroll
      for (int i = 0; i < 4; i++) N.r[i] = N.s[i] = 0.;
      /* the top block's records (the slots are free: the last ray's steps
       * are done, and its reads ordered by the warp's barriers) */
      const int cnt = n0 - blk * G + 1;
      if (q == 0) walk_expect(bar, cnt * BYTES);
      if (q < cnt) copy(q, chunk, (blk % CB) * G + q);
    }
    if (!__any_sync(0xffffffffu, has)) break;
    const bool ok = !has || walk_wait(bar, ph);
    if (__any_sync(0xffffffffu, !ok)) {
      /* a copy that did not land: flag it, give the other rays' copies in
       * flight their bounded wait (each lane has waited for its own ray's),
       * and end the warp */
      if (lane == 0) atomicAdd(&counters[CNT_STALL], 1ULL);
      break;
    }
    if (has) ph ^= 1;
    const DevCam &C = BATCH ? c_cams[cam] : c_cam;
    /* ---- phase A: one lane per record ---- */
    unsigned char *const my = slots + q * W::SLOT;
    const int k = blk * G + q;
    const bool top = blk == n0 / G;
    const bool valid = has && k <= n0;
    double dl = 0., nt = 0., ju = 0., ku = 0., c[8];
    int flags = 0;
#pragma unroll
    for (int i = 0; i < 8; i++) c[i] = 0.;
    if (valid) {
      const double2 *p2 = reinterpret_cast<const double2 *>(my + W::FT);
      double2 v[7];
#pragma unroll
      for (int i = 0; i < 7; i++) v[i] = p2[i];
      flags = (int)v[0].x;
      dl = v[1].y;
      nt = v[5].x;
      if constexpr (BATCH) {
        /* (left unwritten at records that do not radiate, and unused there) */
        const double2 *b2 = reinterpret_cast<const double2 *>(my + W::FX);
        v[6] = b2[4];
        v[5] = b2[4];
        v[4] = b2[3];
        v[3] = b2[2];
        v[2] = b2[1];
        ju = b2[0].x;
        ku = b2[0].y;
        c[0] = v[2].x; /* jI jQ jV aI aQ aV rQ rV */
        c[1] = v[2].y;
        c[2] = v[3].x;
        c[3] = v[3].y;
        c[4] = v[4].x;
        c[5] = v[4].y;
        c[6] = v[5].x;
        c[7] = v[5].y;
      } else {
      ju = v[0].y;
      ku = v[1].x;
      c[0] = v[2].x;
      c[1] = v[2].y;
      c[2] = v[3].x;
      c[3] = v[3].y;
      c[4] = v[4].x;
      c[5] = v[4].y;
      c[6] = v[5].y;
      c[7] = v[6].x;
      }
    }
    const bool ev_my = valid && k < n0 && (flags & 1);
    const unsigned bal = (__ballot_sync(0xffffffffu, ev_my) >> (grp * G)) & GM;
    double dl_n = __shfl_down_sync(0xffffffffu, dl, 1, G), nt_n = __shfl_down_sync(0xffffffffu, nt, 1, G);
    if (q == G - 1) {
      dl_n = dl_up;
      nt_n = nt_up;
    }
    dl_up = __shfl_sync(0xffffffffu, dl, 0, G);
    nt_up = __shfl_sync(0xffffffffu, nt, 0, G);
    /* get_jkinv at the far end of the ray (src/ipolarray.c:74), then at the
     * radiating record before this one */
    {
      const int tq = n0 % G;
      const double jt = __shfl_sync(0xffffffffu, ju, tq, G), kt = __shfl_sync(0xffffffffu, ku, tq, G);
      if (top) {
        js = jt;
        ks = kt;
      }
    }
    const unsigned above = bal & ~((2u << q) - 1u);
    const int qa = above ? __ffs(above) - 1 : 0, ql = bal ? __ffs(bal) - 1 : 0;
    const double ja = __shfl_sync(0xffffffffu, ju, qa, G), ka = __shfl_sync(0xffffffffu, ku, qa, G);
    const double jl = __shfl_sync(0xffffffffu, ju, ql, G), kl = __shfl_sync(0xffffffffu, ku, ql, G);
    const double ji = above ? ja : js, ki = above ? ka : ks;
    if (bal) {
      js = jl;
      ks = kl;
    }
    if (valid) reinterpret_cast<double *>(my + W::FX)[8] = dl;
    if (ev_my) {
      int zero_emission = (flags & 2) ? 1 : 0;
      if (C.target_nturns >= 0 && (int)nt_n != C.target_nturns) zero_emission = 1;
      if (zero_emission) c[0] = c[1] = c[2] = 0.;
      walk_factors<S32>(c, dl_n, unpol, zero_emission ? 0. : ji, ki, zero_emission ? 0. : ju, ku,
                        reinterpret_cast<double *>(my + W::FT), reinterpret_cast<double *>(my + W::FX));
      nrad++;
      if (!unpol) flag |= flags >> 2;
      if constexpr (ADJ) {
        double *w = step_ptr(const_cast<double *>(pool), chunk, k % IPG_CHUNK_STEPS);
        w[REC_FLAGS] = (double)(flags | (zero_emission ? 256 : 0));
        w[REC_ADJ_DL] = dl_n;
      }
    }
    /* the next block: its address, its byte count, the slots this block
     * leaves unused */
    const bool more = has && blk > 0;
    const int kb = blk % CB;
    const int ch = kb ? chunk : cprev, r0 = (kb ? kb - 1 : CB - 1) * G;
    if (more) {
      if (q == 0) {
        walk_expect(bar, G * BYTES);
        /* and the block after it, into L2 */
        if (CB > 1 && blk > 1 && (kb != 1 || cprev >= 0)) {
          const int ch2 = kb == 1 ? cprev : ch;
          const int b2 = kb == 1 ? CB - 1 : (kb ? kb - 2 : CB - 2);
          walk_prefetch_l2(step_ptr(const_cast<double *>(pool), ch2, b2 * G), G * IPG_STEP_DOUBLES * 8);
        }
      }
    }
    /* this lane's writes of its slot come before the copies that refill it */
    walk_refill_fence();
    __syncwarp();
    if (more && k > n0) copy(q, ch, r0 + q);
    /* which of the block's steps any ray of the warp has: records walked,
     * radiating steps, pushes */
    const unsigned mine = has ? (n0 - blk * G >= G - 1 ? GM : (2u << (n0 - blk * G)) - 1u) : 0u;
    const unsigned any_act = __reduce_or_sync(0xffffffffu, mine);
    const unsigned any_ev = __reduce_or_sync(0xffffffffu, bal);
    const unsigned any_pu = __reduce_or_sync(0xffffffffu, blk == 0 ? mine & ~1u : mine);
    /* ---- phase B: the block's steps in order ---- */
#pragma unroll 1
    for (int qq = 31 - __clz((int)any_act); qq >= 0; qq--) {
      const int kk = blk * G + qq;
      const bool act = (mine >> qq) & 1u;
      unsigned char *const sl = slots + qq * W::SLOT;
      const double *const fx = reinterpret_cast<const double *>(sl + W::FX);
      const double *const A1 = reinterpret_cast<const double *>(sl), *const A2 = A1 + (RM ? 8 : 16);
      const bool pu = act && kk >= 1;
      const double dlk = fx[8];
      typename WalkMat<RM>::T a1[4][4], a2[4][4];
      if (!unpol) walk_ldA(A1, a1);
      /* the transfer step k+1 -> k at a radiating point
       * (src/ipolarray.c:91-244): evolve_N over the ray's lanes, applied
       * where ev is set (the exchanges are warp-wide) */
      if ((any_ev >> qq) & 1u) {
        const bool ev = (bal >> qq) & 1u;
        if (ev) {
          const double2 pq = reinterpret_cast<const double2 *>(fx)[2], tt = reinterpret_cast<const double2 *>(fx)[3];
          I = __fma_rn(I, pq.x, pq.y);
          tau = __dadd_rn(tau, tt.x);
          if (!unpol) tauF = __dadd_rn(tauF, tt.y);
        }
        if (!unpol) {
          double e1[4], e2[4], a[4], b[4], T11, T22, T12r, T21i, SI, SQ, SU, SV;
          WalkFac<S32> fac;
          walk_row<RM>(sl, 0, e1);
          walk_row<RM>(sl, 1, e2);
          fac.load(reinterpret_cast<const double *>(sl + W::FT), fx, j);
          walk_row<RM>(sl, 2, a);
          walk_row<RM>(sl, 3, b);
          const double aj = j == 0 ? a[0] : j == 1 ? a[1] : j == 2 ? a[2] : a[3];
          const double bj = j == 0 ? b[0] : j == 1 ? b[1] : j == 2 ? b[2] : b[3];
          walk_stokes(N, e1, e2, j, &T11, &T22, &T12r, &T21i);
          if constexpr (ADJ) {
            if (ev && q == 0) {
              double *w = step_ptr(const_cast<double *>(pool), chunk, kk % IPG_CHUNK_STEPS);
              w[REC_ADJ_SI] = (T11 + T22) / 2;
              w[REC_ADJ_SI + 1] = (T11 - T22) / 2;
              *reinterpret_cast<double2 *>(w + REC_ADJ_SU) = make_double2(T12r, T21i);
            }
          }
          fac.apply((T11 + T22) / 2, (T11 - T22) / 2, T12r, T21i, &SI, &SQ, &SU, &SV);
          if (C.stokes_floors) stokes_floor(&SI, &SQ, &SU, &SV);
          const double d11 = (SI + SQ) - T11, d22 = (SI - SQ) - T22, dr12 = SU - T12r, di21 = SV - T21i;
          if (ev) {
#pragma unroll
            for (int i = 0; i < 4; i++) {
              N.r[i] = hn_upd_r(N.r[i], a[i], aj, b[i], bj, d11, d22, dr12);
              N.s[i] = hn_upd_s(N.s[i], a[i], aj, b[i], bj, di21);
            }
            if (isnan(N.r[0]) || isnan(SI)) flag |= 4; /* lane 0's r[0] is N^00 */
          }
        }
      }
      /* push_polar for the step k -> k-1 (src/ipolarray.c:85-89) */
      if (!unpol && ((any_pu >> qq) & 1u)) {
        const double dlfull = dlk * Gd.inv_dlfac, dlhalf = (0.5 * dlk) * Gd.inv_dlfac;
        WalkN Nh, Nn;
        walk_ldA(A2, a2);
        if constexpr (S32 && IPG_S32_PUSH) {
          walk_push_f32(N, N, a1, dlhalf, j, xch, &Nh);
          walk_push_f32(N, Nh, a2, dlfull, j, xch + 32, &Nn);
        } else {
          walk_push(N, N, a1, dlhalf, j, xch, &Nh);
          walk_push(N, Nh, a2, dlfull, j, xch + 32, &Nn);
        }
        if (pu) N = Nn;
      }
      /* the slot is free: the next block's record (the copy's writes follow
       * this warp's reads; its writes of the factors were fenced above) */
      __syncwarp();
      if (more && act && q == qq) copy(q, ch, r0 + q);
    }
    /* the end of a ray: project_N in the camera's tetrad */
    const bool fin = has && blk == 0;
    if (__any_sync(0xffffffffu, fin)) {
      double T11 = 0., T22 = 0., T12r = 0., T21i = 0.;
      walk_stokes(N, C.Ecov[1], C.Ecov[2], j, &T11, &T22, &T12r, &T21i);
      int fl = flag;
#pragma unroll
      for (int o = 1; o < G; o <<= 1) {
        /* the records' tetrad flags from every lane; the NaN flag from the
         * lanes that hold N^00 only */
        fl |= __shfl_xor_sync(0xffffffffu, fl & ~4, o);
      }
      if (fin && q == 0) {
        ipg_pixel_out o;
        if (!unpol && (tauF > 1.e100 || tauF < -1.e100 || isnan(tauF))) fl |= 2;
        xfer_output(C, I, tau, tauF, T11, T22, T12r, T21i, unpol, n0, fl, &o);
        out[ray] = o;
        if constexpr (BATCH) atomicAdd(&counters[CNT_XSTEPS], (unsigned long long)n0);
      }
      if (fin) has = false;
      __syncwarp();
    }
    if (has) {
      if (kb == 0) {
        chunk = cprev;
        cprev = chunk_prev[chunk];
      }
      blk--;
    }
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) nrad += __shfl_xor_sync(0xffffffffu, nrad, o);
  if (lane == 0 && nrad) atomicAdd(&counters[CNT_RAD], nrad);
}

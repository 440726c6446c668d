/*
 * Reverse-mode adjoint of the polarized image (ipg_adjoint): the gradient of
 * a loss of the IQUV image with respect to the fluid fields ne, Theta_e and
 * |B| of every cell (the fields the fits read, model/iharm/model.c:
 * 510-593).  No counterpart in the reference, which only renders.
 *
 * The geodesics do not depend on the fluid, so only the radiative transfer
 * is differentiated (src/ipolarray.c:59-628).  Per ray, the transfer maps
 * the coherency tensor N from the source end (N = 0 at step nstep) to the
 * camera (N_0, projected to I, Q, U, V); step n -> n-1 is
 *
 *   N_h  = N_n - dl/2 (A1 N_n + N_n A1^T)       push_polar, half step
 *   N'   = N_n - dl   (A2 N_h + N_h A2^T)       push_polar, full step
 *   N_{n-1} = evolve_N(N', coefficients of step n-1)   at radiating points
 *
 * with A1, A2 from the step records.  The adjoint walks back from the
 * camera: G_0 = dL/dN_0 from dL/dIQUV, then for n = 1 .. nstep it maps
 * G_{n-1} = dL/dN_{n-1} to G_n through the transposes of these maps, and at
 * every radiating step it turns dL/d(coefficients) into dL/d(ne, Theta_e,
 * |B|) at the point and scatter-adds that to the eight cells of the
 * trilinear gather (src/grid.c:15-44), with their weights.
 *
 *   - The forward pass (k_walk, ADJ) leaves in each radiating record the
 *     Stokes vector its step was applied to, so no N is kept or recomputed.
 *   - The walk (k_adj_walk, four or more lanes per ray) carries dL/dN and
 *     leaves dL/dS' of each radiating record's step; k_adj_scatter, one
 *     thread per record, turns it into dL/d(coefficients) and dL/d(ne,
 *     Theta_e, |B|) and scatter-adds those to the cells.
 *   - The coefficients' derivatives come from re-evaluating the fits
 *     (jar_fits) in forward-mode dual numbers along ne, Theta_e, |B|
 *     (ipg_dual.cuh), the step's from its transpose (stokes_step_vjp).
 *   - Gradients of N are kept as full-matrix gradients of its real
 *     (symmetric) and imaginary (antisymmetric) parts, upper triangles
 *     stored: every map here keeps those symmetries.
 *
 * Not differentiated: the sigma cut of ne and the Theta_e floor of the
 * host (their derivative is zero almost everywhere), the Stokes floors
 * (the call refuses stokes_floors), the unpolarized intensity.
 *
 * Included by ipg_kernels.cu.
 */

#include "ipg_step_vjp.cuh"

/* the polarized step S -> S' of evolve_N (Faraday half step, absorption and
 * emission, Faraday half step; src/ipolarray.c:390-520) in any number type */
template <class R>
__device__ __forceinline__ void stokes_step(const JarT<R> &c, double dlam, R S[4])
{
  const FaradayRotT<R> F = faraday_rot(c.rQ, c.rU, c.rV, dlam * 0.5);
  faraday_apply(F, c.rQ, c.rU, c.rV, &S[1], &S[2], &S[3]);
  absorb_emit(c, dlam, &S[0], &S[1], &S[2], &S[3]);
  faraday_apply(F, c.rQ, c.rU, c.rV, &S[1], &S[2], &S[3]);
}

/* One pass of the step in Dual<4>: directions d0..d3 among the 12 inputs
 * (S0..S3, then the eight coefficients); returns u . dS'/d(direction). */
__device__ __forceinline__ void step_vjp_pass(const double S0[4], const double cv[8], double dlam, const double u[4],
                                              int first, double out[4])
{
  Dual<4> S[4], cc[8];
#pragma unroll
  for (int k = 0; k < 4; k++) S[k] = (first == 0) ? dvar<4>(S0[k], k) : dconst<4>(S0[k]);
#pragma unroll
  for (int k = 0; k < 8; k++) {
    const int dir = 4 + k - first;
    cc[k] = (dir >= 0 && dir < 4 && first > 0) ? dvar<4>(cv[k], dir) : dconst<4>(cv[k]);
  }
  JarT<Dual<4>> c;
  c.jI = cc[0];
  c.jQ = cc[1];
  c.jU = dconst<4>(0.);
  c.jV = cc[2];
  c.aI = cc[3];
  c.aQ = cc[4];
  c.aU = dconst<4>(0.);
  c.aV = cc[5];
  c.rQ = cc[6];
  c.rU = dconst<4>(0.);
  c.rV = cc[7];
  stokes_step(c, dlam, S);
#pragma unroll
  for (int d = 0; d < 4; d++) out[d] = u[0] * S[0].d[d] + u[1] * S[1].d[d] + u[2] * S[2].d[d] + u[3] * S[3].d[d];
}

/* forward links of the chunk chains and each ray's first chunk */
__global__ void k_adj_link(const int *__restrict__ prev, const int2 *__restrict__ meta,
                           const unsigned long long *__restrict__ counters, long long n_chunks, int *__restrict__ next,
                           int *__restrict__ first)
{
  long long used = (long long)counters[CNT_POOL];
  if (used > n_chunks) used = n_chunks;
  for (long long c = blockIdx.x * (long long)blockDim.x + threadIdx.x; c < used; c += (long long)gridDim.x * blockDim.x) {
    const int p = prev[c];
    if (p >= 0) next[p] = (int)c;
    else first[meta[c].x] = (int)c;
  }
}

/* dL/d(ne, Theta_e, |B|) at the point of a radiating record from dL/d(its
 * coefficients), scattered to the eight cells of its gather */
__device__ __forceinline__ void fluid_scatter(const double *__restrict__ fields, const double *__restrict__ side,
                                              int emission_type, const double gc[8], double *__restrict__ g_ne,
                                              double *__restrict__ g_th, double *__restrict__ g_b)
{
  const int fl = (int)side[7];
  if (!(fl & 2)) return; /* outside the grid: no fluid */
  const double X1 = side[0], X2 = side[1], X3 = side[2];
  GridLoc gl;
  grid_locate(X1, X2, X3, &gl);
  double acc[10];
  gather_cells<10>(fields, gl, acc);
  const double ne = sigma_cut_ne(acc[6], acc[9]);
  if (!(ne > 0.)) return;
  const double dne = ne / acc[6]; /* 1, or the factor of the sigma cut's boundary */
  JarGeo jg;
  jg.nu = side[3];
  jg.inusq = 1. / (jg.nu * jg.nu);
  jg.sth = side[4];
  jg.cth = side[5];
  jg.theta = side[6];
  jg.along = fl & 1;
  Dual<3> Ne = dvar<3>(ne, 0), Th = dvar<3>(acc[7], 1), Bm = dvar<3>(acc[8], 2);
  Dual<3> ju, ku;
  JarT<Dual<3>> jr;
  const Dual<3> z = dconst<3>(0.);
  jr.jI = jr.jQ = jr.jU = jr.jV = jr.aI = jr.aQ = jr.aU = jr.aV = jr.rQ = jr.rU = jr.rV = z;
  jar_fits(Ne, Th, Bm, jg, 1, emission_type, &ju, &ku, &jr);
  const Dual<3> *cs[8] = {&jr.jI, &jr.jQ, &jr.jV, &jr.aI, &jr.aQ, &jr.aV, &jr.rQ, &jr.rV};
  double g[3] = {0., 0., 0.};
#pragma unroll
  for (int k = 0; k < 8; k++)
#pragma unroll
    for (int d = 0; d < 3; d++) g[d] += gc[k] * cs[k]->d[d];
  g[0] *= dne;
#pragma unroll
  for (int cc = 0; cc < 4; cc++)
#pragma unroll
    for (int kk = 0; kk < 2; kk++) {
      const long long cell = gl.cs[cc] + kk;
      const double w = gl.w[2 * cc + kk];
      if (w == 0.) continue;
      atomicAdd(g_ne + cell, w * g[0]);
      atomicAdd(g_th + cell, w * g[1]);
      atomicAdd(g_b + cell, w * g[2]);
    }
}

/* The adjoint walk, camera to source, with G lanes per ray (the layout of
 * k_walk: a warp walks 32/G rays over blocks of G records).  Step n = k + 1
 * maps dL/dN_k to dL/dN_{k+1}; record k holds its coefficients and, from the
 * forward pass, the Stokes vector it was applied to and its length:
 *
 *   u    = dL/dS' = (a G a + b G b, a G a - b G b, 2 a Re G b, 2 b Im G a)
 *   gS   = T^T u, T the step's Stokes map
 *   G   += the transpose of the projection, at gS - u
 *   G    = the two pushes of record k + 1, transposed
 *
 * Only this chain is sequential.  T comes from the coefficients and is
 * evaluated one record per lane; u is left in the record (over its A1, read
 * for the last time here), and k_adj_scatter, one thread per record, turns
 * it into the gradients of the coefficients and of the fluid.  Nothing of
 * the forward pass is recomputed.
 *
 * Bound by the chain of the longest ray (two pushes and four exchanges a
 * step, ~0.7 us) and, with G = 4, by the issue rate.  A 160x160 image
 * (25 600 rays, 3.3e7 steps): walk 97 -> 16 ms against one lane per ray with
 * N recomputed between checkpoints and the step's derivatives in the chain,
 * k_adj_scatter, which has them now, 7 -> 14 ms; a 40x40 image (G = 16):
 * walk and scatter 77 -> 7 ms.  Every wait is bounded as in k_walk. */
template <int G>
__global__ void __launch_bounds__(32)
    k_adj_walk(const int32_t *__restrict__ list, int n_list, double *__restrict__ pool, const int *__restrict__ next,
               const int *__restrict__ first, const RayRec *__restrict__ rays, const double *__restrict__ dL_dout,
               unsigned long long *__restrict__ counters, int queue)
{
  using W = WalkSm<G, 0>;
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
  const DevCam &C = c_cam;
  unsigned ph = 0;
  bool has = false, drained = false;
  int n0 = 0, blk = 0, chunk = 0, cnext = -1; /* the ray's radiating records are among 0 .. n0 - 1 */
  WalkN N;                                     /* column j of dL/dN */
#pragma unroll
  for (int i = 0; i < 4; i++) N.r[i] = N.s[i] = 0.;
  while (true) {
    while (__any_sync(0xffffffffu, !has && !drained)) {
      unsigned long long t = 0;
      const bool want = !has && !drained;
      if (want && q == 0) t = atomicAdd(&counters[queue], 1ULL);
      t = __shfl_sync(0xffffffffu, t, 0, G);
      if (!want) continue;
      if (t >= (unsigned long long)n_list) {
        drained = true;
        continue;
      }
      const int ray = list ? list[t] : (int)t;
      const RayRec rec = rays[ray];
      if (rec.status != IPG_RAY_OK || rec.nstep < 1) continue;
      has = true;
      n0 = rec.nstep;
      blk = 0;
      chunk = first[ray];
      cnext = n0 > IPG_CHUNK_STEPS ? next[chunk] : -1;
      /* G_0 from dL/d(I, Q, U, V) of project_N (src/ipolarray.c:578-598) */
      const double gI = dL_dout[4 * ray], gQ = dL_dout[4 * ray + 1], gU = dL_dout[4 * ray + 2],
                   gV = dL_dout[4 * ray + 3];
      const double gSQ = gQ * C.cproj + gU * C.sproj, gSU = -gQ * C.sproj + gU * C.cproj;
      const double *e1 = C.Ecov[1], *e2 = C.Ecov[2];
#pragma unroll
      for (int i = 0; i < 4; i++) {
        N.r[i] = hn_upd_r(0., e1[i], e1[j], e2[i], e2[j], 0.5 * (gI + gSQ), 0.5 * (gI - gSQ), 0.5 * gSU);
        N.s[i] = hn_upd_s(0., e1[i], e1[j], e2[i], e2[j], 0.5 * gV);
      }
      const int cnt = n0 < G ? n0 : G;
      const unsigned char *src = reinterpret_cast<const unsigned char *>(step_ptr(pool, chunk, 0));
      if (q == 0) walk_expect(bar, cnt * W::COPY);
      if (q < cnt) walk_copy(slots + q * W::SLOT, src + (size_t)q * IPG_STEP_DOUBLES * 8, W::COPY, bar);
    }
    if (!__any_sync(0xffffffffu, has)) break;
    const bool ok = !has || walk_wait(bar, ph);
    if (__any_sync(0xffffffffu, !ok)) {
      if (lane == 0) atomicAdd(&counters[CNT_STALL], 1ULL);
      break;
    }
    if (has) ph ^= 1;
    /* ---- one lane per record: the step's Stokes map ---- */
    unsigned char *const my = slots + q * W::SLOT;
    const int k = blk * G + q;
    bool ev_my = false;
    if (has && k < n0) {
      const double2 *p2 = reinterpret_cast<const double2 *>(my + W::FT);
      const double2 v0 = p2[0], v1 = p2[1], v3 = p2[3], v4 = p2[4], v5 = p2[5], v6 = p2[6];
      ev_my = (int)v0.x & 1;
      reinterpret_cast<double *>(my + W::FX)[8] = v1.y; /* dl of the record's pushes */
      if (ev_my) {
        StokesMap m;
        stokes_map(0., 0., 0., v3.y, v4.x, v4.y, v5.y, v6.x, v6.y, &m);
        double2 *t2 = reinterpret_cast<double2 *>(my + W::FT);
#pragma unroll
        for (int i = 0; i < 8; i++) t2[i] = make_double2(m.T[2 * i], m.T[2 * i + 1]);
      }
    }
    const unsigned bal = (__ballot_sync(0xffffffffu, ev_my) >> (grp * G)) & GM;
    /* the next block: its address and byte count */
    const int kb = blk % CB;
    const int cntn = has ? min(G, n0 - (blk + 1) * G) : 0; /* <= 0: none */
    const unsigned char *src = nullptr;
    if (cntn > 0) {
      const int ch = kb == CB - 1 ? cnext : chunk;
      src = reinterpret_cast<const unsigned char *>(step_ptr(pool, ch, ((kb + 1) % CB) * G));
      if (q == 0) {
        walk_expect(bar, cntn * W::COPY);
        /* and the block after it, into L2 */
        const int cnt2 = min(G, n0 - (blk + 2) * G);
        if (CB > 1 && cnt2 > 0)
          walk_prefetch_l2(step_ptr(pool, kb < CB - 2 ? chunk : cnext, ((kb + 2) % CB) * G), cnt2 * IPG_STEP_DOUBLES * 8);
      }
    }
    /* this lane's writes of its slot come before the copies that refill it */
    walk_refill_fence();
    __syncwarp();
    const int nmine = has ? min(G, n0 - blk * G) : 0;
    const int any_n = __reduce_max_sync(0xffffffffu, nmine);
    const unsigned any_ev = __reduce_or_sync(0xffffffffu, bal);
    /* ---- the block's records in order ---- */
#pragma unroll 1
    for (int qq = 0; qq < any_n; qq++) {
      const int kk = blk * G + qq;
      const bool act = qq < nmine;
      unsigned char *const sl = slots + qq * W::SLOT;
      /* the pushes of record kk, transposed: G_h = -dl (A2^T G + G A2),
       * G += G_h - dl/2 (A1^T G_h + G_h A1); none at record 0 */
      if (__any_sync(0xffffffffu, act && kk >= 1)) {
        const double dlk = reinterpret_cast<const double *>(sl + W::FX)[8];
        const double dlfull = dlk * Gd.inv_dlfac, dlhalf = (0.5 * dlk) * Gd.inv_dlfac;
        const double *const A1 = reinterpret_cast<const double *>(sl), *const A2 = A1 + 16;
        double a[4][4], at[4][4];
        WalkN Z, Gh, Gs;
#pragma unroll
        for (int i = 0; i < 4; i++) Z.r[i] = Z.s[i] = 0.;
        walk_ldA(A2, a);
#pragma unroll
        for (int i = 0; i < 4; i++)
#pragma unroll
          for (int l = 0; l < 4; l++) at[i][l] = a[l][i];
        walk_push(Z, N, at, dlfull, j, xch, &Gh);
        walk_ldA(A1, a);
#pragma unroll
        for (int i = 0; i < 4; i++)
#pragma unroll
          for (int l = 0; l < 4; l++) at[i][l] = a[l][i];
        walk_push(Gh, Gh, at, dlhalf, j, xch + 32, &Gs);
        if (act && kk >= 1) {
#pragma unroll
          for (int i = 0; i < 4; i++) {
            N.r[i] = __dadd_rn(N.r[i], Gs.r[i]);
            N.s[i] = __dadd_rn(N.s[i], Gs.s[i]);
          }
        }
      }
      if ((any_ev >> qq) & 1u) {
        const bool ev = (bal >> qq) & 1u;
        double e1[4], e2[4], a[4], b[4], g11, g22, h12, h21;
        walk_row<0>(sl, 2, a);
        walk_row<0>(sl, 3, b);
        walk_row<0>(sl, 0, e1);
        walk_row<0>(sl, 1, e2);
        walk_stokes(N, a, b, j, &g11, &g22, &h12, &h21);
        const double u[4] = {g11 + g22, g11 - g22, 2. * h12, 2. * h21};
        if (ev && q == 0) store4(step_ptr(pool, chunk, kk % IPG_CHUNK_STEPS) + REC_A1, u[0], u[1], u[2], u[3]);
        /* component j of T^T u, swapped over the lanes */
        const double *T = reinterpret_cast<const double *>(sl + W::FT) + j;
        const double s = dot4_rn(T[0], T[4], T[8], T[12], u[0], u[1], u[2], u[3]);
        double gS[4];
#pragma unroll
        for (int i = 0; i < 4; i++) gS[i] = __shfl_sync(0xffffffffu, s, i, 4);
        /* dL/dT: directly and through S = ((T11 + T22)/2, (T11 - T22)/2,
         * Re T12, Im T21) */
        const double d11 = 0.5 * (gS[0] + gS[1]) - g11, d22 = 0.5 * (gS[0] - gS[1]) - g22;
        const double d12 = 0.5 * (gS[2] - u[2]), d21 = 0.5 * (gS[3] - u[3]);
        const double e1j = j == 0 ? e1[0] : j == 1 ? e1[1] : j == 2 ? e1[2] : e1[3];
        const double e2j = j == 0 ? e2[0] : j == 1 ? e2[1] : j == 2 ? e2[2] : e2[3];
        if (ev) {
#pragma unroll
          for (int i = 0; i < 4; i++) {
            N.r[i] = hn_upd_r(N.r[i], e1[i], e1j, e2[i], e2j, d11, d22, d12);
            N.s[i] = hn_upd_s(N.s[i], e1[i], e1j, e2[i], e2j, d21);
          }
        }
      }
      /* the slot is free: the next block's record */
      __syncwarp();
      if (q == qq && q < cntn) walk_copy(sl, src + (size_t)q * IPG_STEP_DOUBLES * 8, W::COPY, bar);
    }
    if (has) {
      blk++;
      if (blk * G >= n0) {
        has = false;
      } else if (kb == CB - 1) {
        chunk = cnext;
        cnext = n0 > (blk / CB + 1) * IPG_CHUNK_STEPS ? next[chunk] : -1;
      }
    }
    __syncwarp();
  }
}

/* One thread per step record of the wave: dL/dS' that the walk left at each
 * radiating record (steps 0 .. nstep-1 of a traced ray) becomes the
 * gradients of the step's coefficients (stokes_step_vjp, at the S that the
 * forward pass left), then dL/d(ne, Theta_e, |B|) at its point, scattered to
 * the cells of its gather (fluid_scatter). */
#ifndef IPG_SCAT_TPB
#define IPG_SCAT_TPB 384 /* one block per SM at 168 registers */
#endif
__global__ void __launch_bounds__(IPG_SCAT_TPB, 1)
    k_adj_scatter(const double *__restrict__ pool, const int2 *__restrict__ chunk_meta,
                  const unsigned long long *__restrict__ counters, long long n_chunks,
                  const RayRec *__restrict__ rays, const double *__restrict__ adj_side,
                  const double *__restrict__ fields, double *__restrict__ g_ne, double *__restrict__ g_th,
                  double *__restrict__ g_b)
{
  const DevCam &C = c_cam;
  long long used = (long long)counters[CNT_POOL];
  if (used > n_chunks) used = n_chunks;
  const long long total = used * IPG_CHUNK_STEPS;
  for (long long t0 = blockIdx.x * (long long)blockDim.x; t0 < total; t0 += (long long)gridDim.x * blockDim.x) {
    __syncthreads(); /* the warps share their instruction fetches, as in k_coeffs */
    const long long t = t0 + threadIdx.x;
    if (t >= total) continue;
    const int c = (int)(t / IPG_CHUNK_STEPS), slot = (int)(t % IPG_CHUNK_STEPS);
    const int2 meta = chunk_meta[c];
    const RayRec rec = rays[meta.x];
    const int s = meta.y + slot;
    if (rec.status != IPG_RAY_OK || s >= rec.nstep) continue;
    const double *p = step_ptr(const_cast<double *>(pool), c, slot);
    const int flags = (int)p[REC_FLAGS];
    if (!(flags & 1)) continue;
    double gc[8];
    {
      const bool zero = flags & 256; /* a step without emission */
      const double cv[8] = {zero ? 0. : p[REC_JI], zero ? 0. : p[REC_JI + 1], zero ? 0. : p[REC_JI + 2], p[REC_JI + 3],
                            p[REC_JI + 4],         p[REC_JI + 5],             p[REC_RQ],                 p[REC_RV]};
      const double S0[4] = {p[REC_ADJ_SI], p[REC_ADJ_SI + 1], p[REC_ADJ_SU], p[REC_ADJ_SU + 1]};
      double u[4], gS[4];
      load4(p + REC_A1, u);
      stokes_step_vjp(cv, p[REC_ADJ_DL], S0, u, gS, gc);
      if (zero) gc[0] = gc[1] = gc[2] = 0.;
    }
    fluid_scatter(fields, adj_side + ((size_t)c * IPG_CHUNK_STEPS + slot) * IPG_ADJ_DOUBLES, C.emission_type, gc,
                  g_ne, g_th, g_b);
  }
}

/* Self-check of stokes_step_vjp against the forward-mode dual numbers
 * (step_vjp_pass, three passes of four directions) on seeded coefficients
 * and Stokes vectors in four regimes: 0 no polarized absorption
 * (approximate_solve), 1 no Faraday rotation, 2 both, 3 optically thin
 * steps (tau ~ 1e-7: absorb_emit's small-tau series).  err[i] = the largest
 * difference over the twelve gradients, each relative to its own size plus
 * 1e-9 of the largest gradient of its group (Stokes inputs, emissivities,
 * absorptivities, rotativities).  In regime 3 absorb_emit divides by
 * a_P^2 ~ 1e-17, and both forms carry the cancellation that follows. */
__device__ __forceinline__ double vjp_rand(unsigned long long seed, int i, int k)
{
  unsigned long long z = seed * 0x9e3779b97f4a7c15ULL + (unsigned long long)i * 0xbf58476d1ce4e5b9ULL + (unsigned)k;
  z = (z ^ (z >> 30)) * 0xbf58476d1ce4e5b9ULL;
  z = (z ^ (z >> 27)) * 0x94d049bb133111ebULL;
  z ^= z >> 31;
  return (double)(z >> 11) * (1. / 9007199254740992.); /* [0, 1) */
}

__global__ void k_check_step_vjp(int n, unsigned long long seed, double *__restrict__ err, double *__restrict__ info)
{
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const double x = pow(10., -3. + 4. * vjp_rand(seed, i, 0));
  const double aI = pow(10., -5. + 6. * vjp_rand(seed, i, 1));
  const int regime = (int)(vjp_rand(seed, i, 2) * 4.);
  double fq = 2. * vjp_rand(seed, i, 3) - 1., fv = 2. * vjp_rand(seed, i, 4) - 1.;
  const double nf = sqrt(fq * fq + fv * fv) + 1e-300;
  const double pf = 0.98 * vjp_rand(seed, i, 5); /* |a_P| < a_I */
  double aQ = regime == 0 ? 0. : aI * pf * fq / nf, aV = regime == 0 ? 0. : aI * pf * fv / nf;
  const double jI = pow(10., -3. + 4. * vjp_rand(seed, i, 6));
  const double jQ = jI * (2. * vjp_rand(seed, i, 7) - 1.) * 0.7, jV = jI * (2. * vjp_rand(seed, i, 8) - 1.) * 0.3;
  double rQ = pow(10., -4. + 6. * vjp_rand(seed, i, 9)) * (vjp_rand(seed, i, 10) < 0.5 ? -1. : 1.);
  double rV = pow(10., -4. + 6. * vjp_rand(seed, i, 11)) * (vjp_rand(seed, i, 12) < 0.5 ? -1. : 1.);
  if (regime == 1) rQ = rV = 0.;
  if (regime == 3) { /* small optical depths: the series */
    const double s = 1e-7 / (aI * x);
    aQ *= s;
    aV *= s;
  }
  const double aIx = regime == 3 ? 1e-7 / x : aI;
  const double cv[8] = {jI, jQ, jV, aIx, aQ, aV, rQ, rV};
  const double SI = pow(10., -2. + 3. * vjp_rand(seed, i, 13));
  const double S0[4] = {SI, SI * (2. * vjp_rand(seed, i, 14) - 1.) * 0.5, SI * (2. * vjp_rand(seed, i, 15) - 1.) * 0.5,
                        SI * (2. * vjp_rand(seed, i, 16) - 1.) * 0.3};
  const double u[4] = {2. * vjp_rand(seed, i, 17) - 1., 2. * vjp_rand(seed, i, 18) - 1.,
                       2. * vjp_rand(seed, i, 19) - 1., 2. * vjp_rand(seed, i, 20) - 1.};
  double gS[4], gc[8], dS[4], dA[4], dB[4];
  stokes_step_vjp(cv, x, S0, u, gS, gc);
  step_vjp_pass(S0, cv, x, u, 0, dS);
  step_vjp_pass(S0, cv, x, u, 4, dA);
  step_vjp_pass(S0, cv, x, u, 8, dB);
  const double a[12] = {gS[0], gS[1], gS[2], gS[3], gc[0], gc[1], gc[2], gc[3], gc[4], gc[5], gc[6], gc[7]};
  const double b[12] = {dS[0], dS[1], dS[2], dS[3], dA[0], dA[1], dA[2], dA[3], dB[0], dB[1], dB[2], dB[3]};
  /* each gradient against its own size and the scale of its group (the
   * Stokes inputs, the emissivities, the absorptivities, the rotativities) */
  const int grp[12] = {0, 0, 0, 0, 1, 1, 1, 2, 2, 2, 3, 3};
  double sc[4] = {0., 0., 0., 0.};
  for (int k = 0; k < 12; k++) sc[grp[k]] = fmax(sc[grp[k]], fabs(b[k]));
  double e = 0.;
  int kw = 0;
  for (int k = 0; k < 12; k++) {
    const double d = fabs(a[k] - b[k]), den = fabs(b[k]) + 1e-9 * sc[grp[k]] + 1e-300;
    const double r = (d != d) ? 1e300 : d / den;
    if (r > e) {
      e = r;
      kw = k;
    }
  }
  err[i] = e;
  /* the case itself: gradient index, both values, regime, x, the eight
   * coefficients and the Stokes vector */
  double *q = info + (size_t)i * 24;
  q[0] = kw;
  q[1] = a[kw];
  q[2] = b[kw];
  q[3] = regime;
  q[4] = x;
  for (int k = 0; k < 8; k++) q[5 + k] = cv[k];
  for (int k = 0; k < 4; k++) q[13 + k] = S0[k];
  q[17] = sc[grp[kw]];
  q[18] = u[0];
  q[19] = u[1];
  q[20] = u[2];
  q[21] = u[3];
}

extern "C" int ipg__check_step_vjp(int device, int n, unsigned long long seed, double max_err[4], double worst[96])
{
  ipg_ctx *ctx = NULL;
  if (n <= 0 || !max_err) return IPG_E_ARG;
  CK(cudaSetDevice(device));
  double *d = NULL;
  CK(cudaMalloc(&d, (size_t)n * 25 * sizeof(double)));
  k_check_step_vjp<<<(n + 127) / 128, 128>>>(n, seed, d, d + n);
  cudaError_t e = cudaGetLastError();
  std::vector<double> h((size_t)n * 25);
  if (e == cudaSuccess) e = cudaMemcpy(h.data(), d, (size_t)n * 25 * sizeof(double), cudaMemcpyDeviceToHost);
  cudaFree(d);
  if (e != cudaSuccess) return IPG_E_CUDA;
  int im[4] = {0, 0, 0, 0};
  for (int r = 0; r < 4; r++) max_err[r] = -1.;
  for (int i = 0; i < n; i++) {
    const int r = (int)h[n + (size_t)i * 24 + 3];
    if (r >= 0 && r < 4 && h[i] > max_err[r]) {
      max_err[r] = h[i];
      im[r] = i;
    }
  }
  if (worst)
    for (int r = 0; r < 4; r++)
      for (int k = 0; k < 24; k++) worst[24 * r + k] = h[n + (size_t)im[r] * 24 + k];
  return IPG_OK;
}

/* ===================================================================== */
/* host side                                                              */
/* ===================================================================== */
/* lanes per ray as in the forward walk (walk_lanes) */
template <int G>
static int launch_adj_walk_g(ipg_ctx *ctx, const int32_t *list, size_t n, double *pool, const int *next,
                             const int *first, const double *dL, unsigned long long *cnt, int queue, cudaStream_t st)
{
  const void *fn = (const void *)k_adj_walk<G>;
  const size_t sm = WalkSm<G, 0>::BYTES;
  CK(cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm));
  const int wb = grid_blocks(ctx, fn, 32, n * G, sm);
  k_adj_walk<G><<<wb, 32, sm, st>>>(list, (int)n, pool, next, first, ctx->d_rays, dL, cnt, queue);
  ctx->stats.launches++;
  CK(cudaGetLastError());
  return IPG_OK;
}
static int launch_adj_walk(ipg_ctx *ctx, const int32_t *list, size_t n, double *pool, const int *next,
                           const int *first, const double *dL, unsigned long long *cnt, int queue, cudaStream_t st)
{
  switch (walk_lanes(ctx, n)) {
    case 32: return launch_adj_walk_g<32>(ctx, list, n, pool, next, first, dL, cnt, queue, st);
    case 16: return launch_adj_walk_g<16>(ctx, list, n, pool, next, first, dL, cnt, queue, st);
    case 8: return launch_adj_walk_g<8>(ctx, list, n, pool, next, first, dL, cnt, queue, st);
    default: return launch_adj_walk_g<4>(ctx, list, n, pool, next, first, dL, cnt, queue, st);
  }
}

static int adjoint_wave(ipg_ctx *ctx, int em, const int32_t *d_ij, const int32_t *list, size_t run, bool sorted,
                        double *pool, double *side, long long n_chunks, int *next, int *first, const double *dL,
                        ipg_pixel_out *d_out, double *g, size_t ncell, int32_t *deferred)
{
  cudaStream_t st = ctx->stream;
  unsigned long long *cnt = ctx->d_cnt;
  int rc = launch_geo_wave<CamOne>(ctx, 0, 0, d_ij, list, run, sorted, pool, ctx->d_chunk_prev, ctx->d_chunk_meta,
                                   n_chunks, cnt, ctx->d_rays, deferred, nullptr, st);
  if (rc) return rc;
  CK(cudaEventRecord(ctx->ev[2], st)); /* stage boundaries, read by ipg_adjoint */
  if (em == 1) {
    int cb = grid_blocks(ctx, (const void *)k_coeffs<IPG_PLUG_IHARM, 1, true>, IPG_COEF_TPB, (size_t)n_chunks * 32);
    k_coeffs<IPG_PLUG_IHARM, 1, true><<<cb, IPG_COEF_TPB, 0, st>>>(pool, ctx->d_chunk_meta, cnt, n_chunks, ctx->d_rays,
                                                              ctx->d_fields, side);
  } else {
    int cb = grid_blocks(ctx, (const void *)k_coeffs<IPG_PLUG_IHARM, 4, true>, IPG_COEF_TPB, (size_t)n_chunks * 32);
    k_coeffs<IPG_PLUG_IHARM, 4, true><<<cb, IPG_COEF_TPB, 0, st>>>(pool, ctx->d_chunk_meta, cnt, n_chunks, ctx->d_rays,
                                                              ctx->d_fields, side);
  }
  ctx->stats.launches++;
  CK(cudaGetLastError());
  CK(cudaEventRecord(ctx->ev[3], st));
  /* the longest rays' walks with 32 lanes beside the others' (walk_head) */
  const size_t head = walk_head(ctx, list, run, sorted);
  const int32_t *tail = list ? list + head : list;
  cudaStream_t sr = st;
  if (head) {
    if ((rc = walk_fork(ctx, st, &sr))) return rc;
    rc = launch_walk<false, 0, true>(ctx, list, head, pool, ctx->d_chunk_prev, ctx->d_rays, d_out, cnt, st, CNT_NEXT_H);
    if (rc) return rc;
  }
  rc = launch_walk<false, 0, true>(ctx, tail, run - head, pool, ctx->d_chunk_prev, ctx->d_rays, d_out, cnt, sr);
  if (rc || (head && (rc = walk_join(ctx, st)))) return rc;
  CK(cudaEventRecord(ctx->ev[4], st));
  k_adj_link<<<4 * ctx->n_sm, 256, 0, st>>>(ctx->d_chunk_prev, ctx->d_chunk_meta, cnt, n_chunks, next, first);
  ctx->stats.launches++;
  CK(cudaGetLastError());
  if (head) {
    if ((rc = walk_fork(ctx, st, &sr))) return rc;
    if ((rc = launch_adj_walk(ctx, list, head, pool, next, first, dL, cnt, CNT_N + 1, st))) return rc;
  }
  rc = launch_adj_walk(ctx, tail, run - head, pool, next, first, dL, cnt, CNT_N, sr);
  if (rc || (head && (rc = walk_join(ctx, st)))) return rc;
  CK(cudaEventRecord(ctx->ev_pred[0], st));
  int sb = grid_blocks(ctx, (const void *)k_adj_scatter, IPG_SCAT_TPB, (size_t)n_chunks * IPG_CHUNK_STEPS);
  k_adj_scatter<<<sb, IPG_SCAT_TPB, 0, st>>>(pool, ctx->d_chunk_meta, cnt, n_chunks, ctx->d_rays, side, ctx->d_fields, g,
                                        g + ncell, g + 2 * ncell);
  ctx->stats.launches++;
  CK(cudaGetLastError());
  return IPG_OK;
}

/* Maps the pages of a result array (its values stay) while the GPU works:
 * freshly allocated, they are otherwise mapped one by one within the copy
 * that fills it (39 MB: 8-10 ms, of which the copy itself takes 4) */
static void touch_pages(double *p, size_t n)
{
  volatile double *q = p;
  if (!p || !n) return;
  for (size_t i = 0; i < n; i += 512) q[i] = q[i];
  q[n - 1] = q[n - 1];
}

extern "C" int ipg_adjoint(ipg_ctx *ctx, const ipg_camera *cam, const int32_t *ij, size_t n, const double *dL_dout,
                           int ckpt_interval, double *grad_ne, double *grad_thetae, double *grad_b,
                           ipg_pixel_out *out)
{
  if (!ctx || !cam || !ij || !dL_dout || n == 0 || n > 0x7fffffff) return IPG_E_ARG;
  if (!ctx->have_model) return IPG_E_STATE;
  const int K = ckpt_interval;
  if (K != 16 && K != 32 && K != 64) {
    snprintf(ctx->err, sizeof(ctx->err), "checkpoint interval %d: 16, 32 or 64", K);
    return IPG_E_ARG;
  }
  if (ctx->plug != IPG_PLUG_IHARM || cam->only_unpolarized || cam->stokes_floors ||
      (cam->emission_type != 4 && cam->emission_type != 1)) {
    snprintf(ctx->err, sizeof(ctx->err),
             "the adjoint needs an iharm dump, a polarized image, thermal emission and no Stokes floors");
    return IPG_E_ARG;
  }
  if (cam->maxnstep < 2 || cam->nx <= 0 || cam->ny <= 0) return IPG_E_ARG;
  CK(cudaSetDevice(ctx->device));
  int rc = ensure_pool(ctx);
  if (rc) return rc;
  rc = ensure_cap(ctx, n);
  if (rc) return rc;
  const size_t ncell = ctx->ncell;
  DevCam dc;
  make_devcam(cam, &dc);
  dc.mixed = 0;
  cudaStream_t st = ctx->stream;
  CK(cudaMemcpyToSymbolAsync(c_grid, &ctx->dg, sizeof(DevGrid), 0, cudaMemcpyHostToDevice, st));
  CK(cudaMemcpyToSymbolAsync(c_plug, &ctx->dp, sizeof(DevPlug), 0, cudaMemcpyHostToDevice, st));
  CK(cudaMemcpyToSymbolAsync(c_cam, &dc, sizeof(DevCam), 0, cudaMemcpyHostToDevice, st));
  CK(cudaMemcpyAsync(ctx->d_ij, ij, 2 * n * sizeof(int32_t), cudaMemcpyHostToDevice, st));
  /* the pool per chunk: 32 records and their adjoint blocks */
  const size_t rec_b = (size_t)IPG_CHUNK_STEPS * IPG_STEP_DOUBLES * sizeof(double);
  const size_t side_b = (size_t)IPG_CHUNK_STEPS * IPG_ADJ_DOUBLES * sizeof(double);
  const long long n_chunks = (long long)(((size_t)ctx->n_chunks * rec_b) / (rec_b + side_b));
  if (n_chunks < 16) return IPG_E_NOMEM;
  double *pool = ctx->d_pool;
  double *side = pool + (size_t)n_chunks * IPG_CHUNK_STEPS * IPG_STEP_DOUBLES;
  /* scratch kept in the context between calls (grow-only) */
  auto grow = [](void **ptr, size_t *cap, size_t bytes) -> cudaError_t {
    if (*cap >= bytes) return cudaSuccess;
    cudaFree(*ptr);
    *ptr = nullptr;
    *cap = 0;
    cudaError_t e = cudaMalloc(ptr, bytes);
    if (e == cudaSuccess) *cap = bytes;
    return e;
  };
#define CKA(call)                       \
  do {                                  \
    cudaError_t e_ = (call);            \
    if (e_ != cudaSuccess) {            \
      return cuda_fail(ctx, e_, #call); \
    }                                   \
  } while (0)
  CKA(grow((void **)&ctx->d_adj_dl, &ctx->adj_dl_cap, 4 * n * sizeof(double)));
  CKA(grow((void **)&ctx->d_adj_g, &ctx->adj_g_cap, 3 * ncell * sizeof(double)));
  CKA(grow((void **)&ctx->d_adj_next, &ctx->adj_next_cap, (size_t)n_chunks * sizeof(int)));
  CKA(grow((void **)&ctx->d_adj_first, &ctx->adj_first_cap, n * sizeof(int)));
  double *dL = ctx->d_adj_dl, *g = ctx->d_adj_g;
  int *next = ctx->d_adj_next, *first = ctx->d_adj_first;
  CKA(cudaMemcpyAsync(dL, dL_dout, 4 * n * sizeof(double), cudaMemcpyHostToDevice, st));
  CKA(cudaMemsetAsync(g, 0, 3 * ncell * sizeof(double), st));
  memset(&ctx->stats, 0, sizeof(ctx->stats));
  /* waves as in the image trace (unsplit, longest predicted rays first):
   * rays that find the pool full go to the next wave, after this wave's
   * adjoint is done */
  rc = sort_by_length(ctx, ctx->d_ij, n, cam);
  if (rc) return rc;
  const int32_t *list = ctx->d_sorted;
  size_t pending = n, wave = n;
  int cur = 0;
  bool touched = false;
  while (pending > 0) {
    size_t run = pending < wave ? pending : wave;
    size_t carry = pending - run;
    int32_t *nextl = ctx->d_list[cur ^ 1];
    unsigned long long h0[CNT_N + 2]; /* the wave's, and the adjoint walk's two queues */
    memset(h0, 0, sizeof(h0));
    h0[CNT_DEFER] = carry;
    CKA(cudaMemcpyAsync(ctx->d_cnt, h0, sizeof(h0), cudaMemcpyHostToDevice, st));
    if (carry) {
      if (list) CKA(cudaMemcpyAsync(nextl, list + run, carry * sizeof(int32_t), cudaMemcpyDeviceToDevice, st));
      else k_iota<<<(int)((carry + 255) / 256), 256, 0, st>>>(nextl, (int)carry, (int)run);
    }
    CKA(cudaEventRecord(ctx->ev[0], st));
    const int em = cam->emission_type;
    rc = adjoint_wave(ctx, em, ctx->d_ij, list, run, list == ctx->d_sorted, pool, side, n_chunks, next, first, dL,
                      ctx->d_out, g, ncell, nextl);
    if (rc) {
      wave_stop(ctx);
      return rc;
    }
    CKA(cudaEventRecord(ctx->ev[1], st));
    if (!touched) {
      touch_pages(grad_ne, ncell);
      touch_pages(grad_thetae, ncell);
      touch_pages(grad_b, ncell);
      touched = true;
    }
    unsigned long long h[CNT_N];
    CKA(cudaMemcpyAsync(h, ctx->d_cnt, sizeof(h), cudaMemcpyDeviceToHost, st));
    CKA(cudaStreamSynchronize(st));
    if (h[CNT_STALL]) return stall_fail(ctx);
    float ms = 0.f, t[5] = {0.f, 0.f, 0.f, 0.f, 0.f};
    cudaEventElapsedTime(&ms, ctx->ev[0], ctx->ev[1]);
    cudaEventElapsedTime(&t[0], ctx->ev[0], ctx->ev[2]);
    cudaEventElapsedTime(&t[1], ctx->ev[2], ctx->ev[3]);
    cudaEventElapsedTime(&t[2], ctx->ev[3], ctx->ev[4]);
    cudaEventElapsedTime(&t[3], ctx->ev[4], ctx->ev_pred[0]);
    cudaEventElapsedTime(&t[4], ctx->ev_pred[0], ctx->ev[1]);
    ctx->stats.wall_ms += ms;
    ctx->stats.geodesic_ms += t[0];
    ctx->stats.coeffs_ms += t[1];
    ctx->stats.transfer_ms += t[2];
    ctx->stats.adjoint_ms += t[3];
    ctx->stats.adj_scatter_ms += t[4];
    ctx->stats.ray_steps += h[CNT_STEPS];
    ctx->stats.radiating_steps += h[CNT_RAD];
    ctx->stats.waves += 1;
    size_t deferred = (size_t)h[CNT_DEFER];
    if (deferred == pending) {
      if (run == 1) {
        snprintf(ctx->err, sizeof(ctx->err), "trajectory pool too small for a single ray");
        return IPG_E_NOMEM;
      }
      wave = run / 2;
    }
    pending = deferred;
    cur ^= 1;
    list = ctx->d_list[cur];
  }
  if (grad_ne) CKA(cudaMemcpyAsync(grad_ne, g, ncell * sizeof(double), cudaMemcpyDeviceToHost, st));
  if (grad_thetae) CKA(cudaMemcpyAsync(grad_thetae, g + ncell, ncell * sizeof(double), cudaMemcpyDeviceToHost, st));
  if (grad_b) CKA(cudaMemcpyAsync(grad_b, g + 2 * ncell, ncell * sizeof(double), cudaMemcpyDeviceToHost, st));
  std::vector<ipg_pixel_out> hout(out ? 0 : n);
  ipg_pixel_out *o = out ? out : hout.data();
  CKA(cudaMemcpyAsync(o, ctx->d_out, n * sizeof(ipg_pixel_out), cudaMemcpyDeviceToHost, st));
  CKA(cudaStreamSynchronize(st));
#undef CKA
  for (size_t m = 0; m < n; m++)
    if (o[m].nstep >= cam->maxnstep - 1) {
      snprintf(ctx->err, sizeof(ctx->err), "MaxNStep exceeded in pixel %d %d", ij[2 * m], ij[2 * m + 1]);
      return IPG_E_MAXNSTEP;
    }
  return IPG_OK;
}
